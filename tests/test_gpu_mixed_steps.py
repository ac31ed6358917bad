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


@pytest.mark.parametrize("mixer,portion,others", [("delta", 520, 9), ("delta", 77, 40), ("delta", 2048, 3)])
def test_a_portion_beside_decoded_tokens(mixer, portion, others):
    """The step that continuous batching runs, at the sizes of a real layer and above the sizes from which long portions have kernels
    of their own, against 64 bits."""
    from perf import cases
    case = dict(kind="mixer", mixer=mixer, width=2048, requests=1 + others, new=1, context=512, ragged=False, dtype="bf16", portion=portion)
    got = cases.run(cases.prepare(case, 3))
    want, limit = cases.exact(case, 3), cases.tolerance(case)
    for x, y in zip(got, want):
        assert _rel(x.reshape(y.shape), y) < limit["rel"]
        short = slice(portion, None) if x.dim() == 2 and x.shape[0] == portion + others else slice(1, None)
        assert _rel(x.reshape(y.shape)[short], y[short]) < limit["rel"]


@pytest.mark.parametrize("lens", [[300, 1, 1, 64, 1], [1, 63, 1, 0, 200], [1] * 33 + [128] + [1] * 33 + [64, 65], [64], [63, 700]])
def test_delta_rule_chooses_per_request(lens, monkeypatch):
    """Requests of fewer tokens than a long portion's get the token-by-token kernel's bits whatever stands beside them, long ones the
    chunks' bits."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(len(lens))
    H, G, dim, dv, T, S = 16, 8, 128, 32, sum(lens), len(lens)
    y, ab = torch.randn(T, 2 * G * dim + H * dv, device=DEV), torch.randn(T, 2 * H, device=DEV)
    y[:, :2 * G * dim] *= dim ** -0.5
    a_log, dt_bias, start = torch.zeros(H, device=DEV), torch.full((H,), -3.0, device=DEV), torch.randn(S, H * dim * dv, device=DEV)
    cu, slots = i32([sum(lens[:s]) for s in range(S + 1)]), i32(list(range(S)))

    def run(fn):
        o, s = torch.full((T, H * dv), 7.0, device=DEV), start.clone()
        fn((y, ab, a_log, dt_bias, cu, slots, s, o))
        return o, s
    tokens = run(lambda a: ops.delta_recurrent(*a, S, G, H, dim, dv, None))
    chunks = run(lambda a: ops.delta_chunked(*a, lens, G, H, dim, dv, None))

    def both(a):
        ops.delta_chunked(*a, lens, G, H, dim, dv, None, long_from=64)
        ops.delta_recurrent(*a, S, G, H, dim, dv, None, skip_from=64)
    got = run(both)
    for s, n in enumerate(lens):
        rows, want = slice(sum(lens[:s]), sum(lens[:s + 1])), chunks if n >= 64 else tokens
        assert torch.equal(got[0][rows], want[0][rows]) and torch.equal(got[1][s], want[1][s]), (s, n)


def test_recurrent_parts_choose_per_request():
    """The rules: what a request is run by depends on its own tokens; the others of the step only say whether there is enough work."""
    from photon_infer_b200.kernels import ops
    assert ops.delta_chunked_from(128, 128, [256] + [1] * 31, 32) == ops.DELTA_CHUNKED_MIN_TOKENS
    assert ops.delta_chunked_from(128, 128, [64] + [1] * 200, 32) == 0           # the decoded tokens are no work for the chunks
    assert ops.delta_chunked_from(128, 128, [63] * 100, 32) == 0
    assert ops.delta_chunked_from(129, 128, [4096], 32) == 0 and ops.delta_chunked_from(128, 257, [4096], 32) == 0


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
