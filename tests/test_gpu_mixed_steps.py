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


@pytest.mark.parametrize("mixer,portion,others", [("delta", 520, 9), ("delta", 77, 40), ("delta", 2048, 3), ("gla", 520, 9),
                                                  ("gla", 1093, 40), ("mlstm", 520, 9), ("mlstm", 1093, 40), ("mamba2", 600, 9), ("mamba2", 1093, 40),
                                                  ("hgrn2", 800, 0), ("hgrn2", 800, 9)])
def test_a_portion_beside_decoded_tokens(mixer, portion, others):
    """The step that continuous batching runs, at the sizes of a real layer and above the sizes from which long portions have kernels
    of their own, against 64 bits."""
    from perf import cases
    from photon_infer_b200.kernels import ops
    lens, mode = [portion] + [1] * others, {"gla": "decay_rows", "mlstm": "matrix_memory", "mamba2": "state_space", "hgrn2": "forget_write"}.get(mixer)
    if mode:
        assert ops.linrec_segments_supported(mode, 128, lens, 16) == (mixer != "hgrn2" or not others)
    case = dict(kind="mixer", mixer=mixer, width=2048, requests=1 + others, new=1, context=512, ragged=False, dtype="bf16", portion=portion)
    got = cases.run(cases.prepare(case, 3))
    want, limit = cases.exact(case, 3), cases.tolerance(case)
    for x, y in zip(got, want):
        assert _rel(x.reshape(y.shape), y) < limit["rel"]
        if not others:
            continue
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


@pytest.mark.parametrize("mode", ["state_space", "matrix_memory", "forget_write", "decay_rows"])
@pytest.mark.parametrize("lens", [[300, 1, 1, 128, 1], [1, 64, 1, 0, 65], [1] * 33 + [128] + [1] * 33 + [200, 129], [128], [1, 2, 64], [127, 700]])
def test_segments_of_a_request_do_not_depend_on_the_others(mode, lens):
    """Outputs, state and divisors of every request have the bits that they have when it is alone, at any place of the step."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(len(lens))
    H, N, dv, T, S = 4, 64, 40, sum(lens), len(lens)
    memory, rows = mode == "matrix_memory", mode in ("forget_write", "decay_rows")
    g = torch.randn(T, 2 * H, device=DEV)
    x = [torch.randn(T, H * N, device=DEV), torch.rand(T, H * N, device=DEV), torch.randn(T, H * dv, device=DEV),
         torch.rand(T, H * N, device=DEV).sqrt() if mode == "decay_rows" else None, None if rows else g[:, :H], g[:, H:] if memory else None]
    p = [None if rows else torch.zeros(H, device=DEV), None if rows else torch.zeros(H, device=DEV), torch.ones(H, device=DEV) if mode == "state_space" else None]
    start, cu = torch.rand(S, H * N * dv + (H * N + H if memory else 0), device=DEV), [sum(lens[:s]) for s in range(S + 1)]

    def run(at, lens_, slots):
        o, s = torch.full((at.stop - at.start, H * dv), 7.0, device=DEV), start.clone()
        den = ops.linrec_segments(mode, *(None if t is None else t[at] for t in x), *p, 5.0 if memory else 0.0, 0.1,
                                  i32([sum(lens_[:i]) for i in range(len(lens_) + 1)]), i32(slots), s, o, lens_, H, H, N, dv, None, segment=64)
        return o, s, den
    whole = run(slice(0, T), lens, list(range(S)))
    for s, n in enumerate(lens):
        at = slice(cu[s], cu[s + 1])
        if n == 0:
            assert torch.equal(whole[1][s], start[s])
            continue
        alone = run(at, [n], [s])
        assert torch.equal(whole[0][at], alone[0]) and torch.equal(whole[1][s], alone[1][s]), (s, n)
        assert not memory or torch.equal(whole[2][at], alone[2])


def test_division_beside_a_norm_of_odd_parts(monkeypatch):
    """The matrix memory's heads of 30 numbers, whose norm does not divide: segments against token by token."""
    from photon_infer_b200.kernels import ops
    from photon_infer_b200.parts.matrix_memory import MatrixMemoryMixer
    torch.manual_seed(0)
    H, dim, dv, lens = 16, 32, 30, [500, 1, 3]
    mixer = MatrixMemoryMixer(256, H, dim, dv, 15.0, 1e-5)
    mixer.load({s.name: (1.0 + 0.1 * torch.randn(s.concrete_shape(), device=DEV) if s.init == "norm" else 0.1 * torch.randn(s.concrete_shape(), device=DEV))
                .bfloat16() for s in mixer.tensor_specs()})
    h = torch.randn(sum(lens), 256, device=DEV).bfloat16()
    outs = []
    for least in (7000, 10 ** 9):
        monkeypatch.setitem(ops.LINREC_SEGMENTS_FROM, "matrix_memory", least)
        assert ops.linrec_segments_supported("matrix_memory", dim, lens, H) == (least == 7000)
        state = torch.zeros(3, *mixer.state_spec().shape, device=DEV)
        outs.append((mixer.forward(h, _step(lens), LayerCache(state=state)), state))
    assert _rel(outs[0][0], outs[1][0]) < 2e-3 and _rel(outs[0][1], outs[1][1]) < 5e-6     # a bfloat16 product behind 32-bit sums


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
