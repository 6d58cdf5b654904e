"""Which waits a step queues depends on its switches: with the event log on every gather and reduction has its
stream and events, with it off those that launch nothing have none, and without overlap there is one stream.  All
train alike, to the bit: no token occurs twice in a micro-step, so that the embedding's atomic sums have one term
each.  The layers are wide enough that their update still runs when the next step reads the first unit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def train(tied, optimizer, diagnostics, overlap, graphs):
    from shardtrain_b200.models.qwen2 import Qwen2CausalLM, Qwen2ModelConfig
    from shardtrain_b200.runtime.engine import ShardedRuntime
    from shardtrain_b200.training.qwen2_trainer import QwenTrainer

    torch.manual_seed(1)
    vocab = 8192
    cfg = Qwen2ModelConfig(vocab_size=vocab, hidden_size=1024, intermediate_size=4096, num_hidden_layers=3,
                           num_attention_heads=8, num_key_value_heads=2, tie_word_embeddings=tied)
    model = Qwen2CausalLM(cfg, device="cuda")
    rt = ShardedRuntime(device="cuda:0", async_grad_rs=overlap, forward_prefetch=overlap, backward_prefetch=overlap,
                        communication_policy="stream_ordered" if overlap else "conservative",
                        diagnostics_enabled=diagnostics, cuda_graphs=graphs).register(model)
    tr = QwenTrainer(model, rt, lr=1e-3 if optimizer == "adamw" else 0.3, dtype="bf16", optimizer=optimizer,
                     accumulation_steps=2)
    generator = torch.Generator(device="cuda").manual_seed(2)
    losses = []
    for _ in range(4):
        ids = torch.stack([torch.randperm(vocab, generator=generator, device="cuda")[:512].view(2, 256)
                           for _ in range(2)]).view(4, 256)
        losses.append(tr.train_step(ids).loss)
    torch.cuda.synchronize()
    state = [rt.param_arena.clone(), rt.grad_arena.clone()]
    if optimizer == "adamw":
        state += [tr.optimizer.exp_avg.clone(), tr.optimizer.exp_avg_sq.clone()]
    rt.close()
    return losses, state


@pytest.mark.parametrize("tied", [True, False])
@pytest.mark.parametrize("optimizer", ["adamw", "sgd"])
def test_switches_change_no_bit(tied, optimizer):
    losses, state = train(tied, optimizer, diagnostics=True, overlap=True, graphs=False)
    assert losses[0] == losses[0] and len(set(losses)) == 4
    for diagnostics, overlap, graphs in ((False, True, False), (False, True, True), (True, True, True),
                                         (False, False, True), (True, False, False)):
        got, other = train(tied, optimizer, diagnostics, overlap, graphs)
        assert got == losses, (diagnostics, overlap, graphs)
        for a, b in zip(other, state):
            assert torch.equal(a, b), (diagnostics, overlap, graphs, (a - b).abs().max().item())
