"""A step's integers on their way to the GPU, and scoring of all places of a step against scoring of some."""
import pytest
import torch

from nanoquantization_b200.engine import LLMEngine, Sequence, StepBatch
from nanoquantization_b200.models import VemedraConfig, VemedraForCausalLM

pytestmark = pytest.mark.gpu
NAMES = ("tokens", "positions", "rows", "cu", "pos0", "ctx", "slot", "table")


@pytest.mark.parametrize("lens", [[1], [3, 1], [7, 5, 1], [1000, 37]])
def test_batches_arrive_whole_behind_a_busy_stream(lens):
    hosts = [StepBatch.host([[100 * k + b + i for i in range(n)] for b, n in enumerate(lens)], [5 * k + b for b in range(len(lens))],
                            [list(range(b, b + 80)) for b in range(len(lens))], list(range(len(lens))), 81, 16) for k in range(12)]
    torch.cuda._sleep(20_000_000)      # the copies wait in the stream while the pinned blocks are handed out again
    there = [h.to("cuda") for h in hosts]
    for h, d in zip(hosts, there):
        for name in NAMES:
            assert torch.equal(getattr(h, name), getattr(d, name).cpu()), name


def test_all_places_and_some_places_have_the_same_logits():
    cfg = {"architecture": "Vemedra", "vocab": 96, "width": 64, "canon": {"taps": 4}, "norm": {"eps": 1e-5},
           "layers": [{"type": "mingru", "mixer": {"width": 64}, "mlp": {"kind": "dense", "ff": 96, "limit": 2.0}}]}
    model = VemedraForCausalLM(VemedraConfig.from_dict(cfg), device="cuda", dtype=torch.float32)
    g = torch.Generator().manual_seed(0)
    for t in model.checkpoint_tensors().values():
        t.copy_(torch.randn(t.shape, generator=g) * 0.3)
    prompts = [torch.randint(0, 96, (n,), generator=g).tolist() for n in (40, 23)]

    def score(wanted):
        eng = LLMEngine(model, num_blocks=8, block_size=16, max_batch=2)
        return eng.extend([(Sequence(i, [], 1), p, w) for i, (p, w) in enumerate(zip(prompts, wanted))])
    every = score([range(40), range(23)])
    some = score([[3, 39, 7], range(22, -1, -2)])
    torch.testing.assert_close(some[0], every[0][[3, 39, 7]], rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(some[1], every[1][list(range(22, -1, -2))], rtol=1e-5, atol=1e-5)
    assert score([[], range(23)])[0] is None
