"""One member on the sm_100a executor: units without bridge nodes.  Same order of events, same streams, same
refusals as with them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def trainer(tied, asynchronous, optimizer="adamw", **switches):
    from shardtrain_b200.models.qwen2 import Qwen2CausalLM, Qwen2ModelConfig
    from shardtrain_b200.runtime.engine import ShardedRuntime
    from shardtrain_b200.training.qwen2_trainer import QwenTrainer

    torch.manual_seed(0)
    cfg = Qwen2ModelConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                           num_attention_heads=2, num_key_value_heads=1, tie_word_embeddings=tied)
    model = Qwen2CausalLM(cfg, device="cuda")
    rt = ShardedRuntime(device="cuda:0", async_grad_rs=asynchronous, forward_prefetch=asynchronous,
                        backward_prefetch=asynchronous, communication_policy="stream_ordered",
                        **switches).register(model)
    return model, rt, QwenTrainer(model, rt, lr=1e-3, dtype="bf16", optimizer=optimizer, accumulation_steps=2)


@pytest.mark.parametrize("tied", [True, False])
@pytest.mark.parametrize("asynchronous", [True, False])
def test_order_and_streams_of_the_units(tied, asynchronous):
    model, rt, tr = trainer(tied, asynchronous)
    assert rt.direct
    tr.train_step(torch.randint(0, 512, (4, 130), device="cuda"))
    units = len(rt.units)
    # backward enters the units from the last to the first; a tied unit is entered first, by the head
    entered = [0, *range(units - 1, 0, -1)] if tied else list(range(units - 1, -1, -1))
    rows = rt.comm.events
    for step in range(2):
        def of(kind):
            return [r["unit_id"] for r in rows if r["event_type"] == kind and r["step_id"] == step]

        assert of("unit_forward") == list(range(units))
        assert of("unit_pre_backward") == entered
        assert of("unit_grads_ready") == list(range(units - 1, -1, -1))
        # a unit is reduced before the next one is entered
        mixed = [(r["event_type"], r["unit_id"]) for r in rows if r["step_id"] == step
                 and r["event_type"] in ("unit_pre_backward", "unit_grads_ready") and r["unit_id"]]
        assert mixed == [(kind, u) for u in range(units - 1, 0, -1)
                         for kind in ("unit_pre_backward", "unit_grads_ready")]
    streams = {r["issue_stream"] for r in rows if r["event_type"] == "unit_grads_ready"}
    assert streams == ({"fsdp_rs"} if asynchronous else {"compute"})
    assert not rt.comm.live_buffers
    rt.close()


@pytest.mark.parametrize("tied", [True, False])
def test_nothing_is_gathered_and_vectors_follow_the_optimizer(tied):
    model, rt, tr = trainer(tied, True, diagnostics_enabled=False)
    assert all(plan.gather_table.numel() == 0 for plan in rt.materializer.plans.values())
    ids = torch.randint(0, 512, (4, 130), device="cuda")
    losses = [tr.train_step(ids).loss for _ in range(4)]
    assert losses[-1] < losses[0]
    torch.cuda.synchronize()
    for unit in rt.units:
        weights = rt.materializer.plans[unit.unit_id].weights
        for handle in unit.handles:
            full = weights[handle.spec.param_id]
            shard = handle.local_shard.detach().view(full.shape)
            assert torch.equal(full, shard if full.dtype == torch.float32 else shard.bfloat16())
    rt.close()


def test_a_second_backward_is_refused():
    model, rt, tr = trainer(True, True)
    ids = torch.randint(0, 512, (2, 130), device="cuda")
    with rt.compute_context():
        rt.zero_grad()
        rt.begin_step(0)
        loss = model(ids, labels=ids).loss
        loss.backward(retain_graph=True)
        with pytest.raises(RuntimeError, match="Repeated/invalid backward"):
            loss.backward()
    torch.cuda.synchronize()
    rt.close()
