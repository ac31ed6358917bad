"""Whole recurrent parts in steps that are large enough for the segments and the chunks of long portions."""
import pytest
import torch

from photon_infer_b200.parts.base import LayerCache, StepContext

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _step(lens, slots=None):
    S, T = len(lens), sum(lens)
    slots = list(range(S)) if slots is None else slots
    return StepContext(num_tokens=T, num_seqs=S, dtype=torch.bfloat16, token_ids=None, positions=i32([i for n in lens for i in range(n)]),
                       token_seq=i32([s for s, n in enumerate(lens) for _ in range(n)]), cu_tokens=i32([sum(lens[:s]) for s in range(S + 1)]),
                       context_lens=i32(lens), state_slots=i32(slots), groups=[], host_query_lens=lens, host_context_lens=lens,
                       host_start_positions=[0] * S, max_query_len=max(lens), max_context_len=max(lens),
                       error_flag=torch.zeros(4, dtype=torch.int32, device=DEV), host_state_slots=slots)


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("rank", [768, 800])
def test_gated_linear_attention_takes_every_rank(rank):
    """Ranks that the long portions' own pass over the inputs has no room for take the other kernels."""
    from photon_infer_b200.kernels import ops
    from photon_infer_b200.parts.gla import GatedLinearAttention
    torch.manual_seed(rank)
    heads, dim, T = 64, 16, 130
    mixer = GatedLinearAttention(256, heads, dim, dim, 16.0, 1e-5, rank)
    assert ops.linrec_segments_supported("decay_rows", dim, [T], heads)
    mixer.load({s.name: (torch.randn(s.concrete_shape() if s.name not in ("a1", "a2") else ((rank, 256) if s.name == "a1" else (heads * dim, rank)),
                                     device=DEV) * 0.06).bfloat16() for s in mixer.tensor_specs()})
    h = torch.randn(T, 256, device=DEV).bfloat16()
    state = lambda: torch.zeros(1, heads, dim, dim, device=DEV)
    whole, parts = state(), state()
    got = mixer.forward(h, _step([T]), LayerCache(state=whole))
    want = torch.cat([mixer.forward(h[i:i + 65], _step([65]), LayerCache(state=parts)) for i in (0, 65)])
    assert _rel(got, want) < 1e-2 and _rel(whole, parts) < 1e-4       # the projections of 65 and of 130 rows round to bfloat16 once each
