"""A single member's backward writes gradients straight into the arena: same numbers as through the
ring of slots and the reduction kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _train(tied, accum, optimizer, steps=2):
    from shardtrain_b200.models.qwen2 import Qwen2CausalLM, Qwen2ModelConfig
    from shardtrain_b200.runtime.engine import ShardedRuntime
    from shardtrain_b200.training.qwen2_trainer import QwenTrainer

    torch.manual_seed(5)
    cfg = Qwen2ModelConfig(vocab_size=520, hidden_size=256, intermediate_size=520, num_hidden_layers=2,
                           num_attention_heads=2, num_key_value_heads=1, tie_word_embeddings=tied)
    model = Qwen2CausalLM(cfg, device="cuda")
    runtime = ShardedRuntime(device="cuda:0", forward_prefetch=True, backward_prefetch=True, async_grad_rs=True,
                             communication_policy="stream_ordered", diagnostics_enabled=False).register(model)
    trainer = QwenTrainer(model, runtime, lr=1e-2 if optimizer == "sgd" else 1e-4, dtype="bf16",
                          optimizer=optimizer, accumulation_steps=accum)
    ids = torch.arange(6 * 72, device="cuda").view(6, 72) % 520      # every row of the table at most once
    losses = [trainer.train_step(ids).loss for _ in range(steps)]
    in_arena = [p.arena_slot is not None for p in runtime.materializer.plans.values()]
    state = runtime.param_arena.clone(), runtime.grad_arena.clone()
    runtime.close()
    return losses, in_arena, state


@pytest.mark.parametrize("tied", [True, False])
@pytest.mark.parametrize("accum", [1, 3])
@pytest.mark.parametrize("optimizer", ["adamw", "sgd"])
def test_same_gradients_and_weights_as_through_the_slots(monkeypatch, tied, accum, optimizer):
    from shardtrain_b200.runtime.fused import FusedExecutor

    losses, in_arena, state = _train(tied, accum, optimizer)
    assert all(in_arena)
    monkeypatch.setattr(FusedExecutor, "_gradients_in_arena", lambda self, unit, plan: False)
    want_losses, in_arena, want = _train(tied, accum, optimizer)
    assert not any(in_arena)
    for got, ref in zip(state, want):
        if tied and accum > 1:
            # (sum so far + head) + lookup instead of sum so far + (head + lookup): one rounding of
            # 2^-24 apart where a row of the table takes part in both
            assert (got - ref).norm() <= 1e-6 * ref.norm()
        else:
            assert torch.equal(got, ref)
    assert losses == pytest.approx(want_losses, rel=1e-6)
