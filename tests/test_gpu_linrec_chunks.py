"""The recurrences in chunks of 128 tokens on the tensor cores (linrec_chunks.cu) against the same recurrence token by token in 64
bits: chunks that are not full, states that are not zero, reused and negative slots, small states, decays of nearly nothing, and
values that are not finite; and an error against 64 bits that is not larger than the segments'."""
import pytest
import torch

from test_gpu_linrec_segments import _rel, _walk, i32

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MODES = ["state_space", "matrix_memory", "decay_rows"]


@pytest.fixture(autouse=True)
def any_size(monkeypatch):
    """Chunks for steps of any size and shape."""
    from photon_infer_b200.kernels import ops
    monkeypatch.setattr(ops, "LINREC_CHUNKS_FROM", dict.fromkeys(ops.LINREC_CHUNKS_FROM, 0))
    monkeypatch.setattr(ops, "linrec_chunks_faster", lambda *args: True)


def _case(mode, H, G, N, dv, lens, slots, strong, seed, poison=None, what="v"):
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(seed)
    T = sum(lens)
    rows = torch.randn(T, 3 * G * N + H * dv + 2 * H + 4 - 2 * H % 4, generator=gen)
    a0 = 3 * G * N
    b0 = a0 + H * dv
    rows[:, 2 * G * N:a0] = torch.sigmoid(rows[:, 2 * G * N:a0] + 2.0) ** (40 if strong else 1)
    if strong and mode == "decay_rows":
        rows[7, 2 * G * N] = 0.0
    p0, p1, p2 = (0.5 * torch.randn(H, generator=gen) for _ in range(3))
    p1 = p1 + ((-3.0 if strong else 3.0) if mode == "matrix_memory" else -1.0)
    p0 = p0 + (2.0 if strong and mode == "state_space" else 0.0)
    memory, per_head = mode == "matrix_memory", mode in ("matrix_memory", "state_space")
    width = H * N * dv + (H * N + H if memory else 0)
    width += 4 + -width % 4
    state = torch.randn(7, width, generator=gen)
    if poison is not None:
        first = {"q": 0, "k": G * N, "a": 2 * G * N, "v": a0, "gate_a": b0, "gate_b": b0 + H}[what]
        rows[poison[0], first + poison[1]] = poison[2]
    st, r = state.to(DEV), rows.to(DEV)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    out, err = torch.full((T, H * dv), float("nan"), device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
    cap, scale = (6.0 if memory else 0.0), N ** -0.5
    args = (r[:, :G * N], r[:, G * N:2 * G * N], r[:, a0:b0], r[:, 2 * G * N:a0] if mode == "decay_rows" else None)
    assert ops.linrec_chunks_supported(mode, N, dv, lens, H, st, *args)
    den = ops.linrec_segments(mode, *args, r[:, b0:b0 + H] if per_head else None, r[:, b0 + H:b0 + 2 * H] if memory else None,
                              p0.to(DEV) if per_head else None, p1.to(DEV) if per_head else None, p2.to(DEV) if mode == "state_space" else None,
                              cap, scale, i32(cu), i32(slots), st, out, lens, H, G, N, dv, err)
    if memory:
        out = (out.view(T, H, dv) / den.unsqueeze(-1)).view(T, H * dv)
    assert err.cpu().tolist()[0] == 0
    wants = []
    for i, L in enumerate(lens):
        x = rows[cu[i]:cu[i + 1]].double()
        heads = lambda z: z.reshape(L, G, N).repeat_interleave(H // G, dim=1)
        s0 = state[slots[i]].double() if slots[i] >= 0 else torch.zeros(width, dtype=torch.float64)
        S, n = s0[:H * N * dv].view(H, N, dv), s0[H * N * dv:H * N * dv + H * N].view(H, N) if memory else None
        m = s0[H * N * (dv + 1):H * N * (dv + 1) + H] if memory else None
        wants.append(_walk(mode, heads(x[:, :G * N]), heads(x[:, G * N:2 * G * N]), x[:, a0:b0].reshape(L, H, dv), heads(x[:, 2 * G * N:a0]),
                           x[:, b0:b0 + H], x[:, b0 + H:b0 + 2 * H], p0.double(), p1.double(), p2.double(), cap, scale, S, n, m))
    return out.cpu(), st.cpu(), state, wants, cu


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("H,G,N,dv", [(2, 2, 128, 128), (4, 2, 128, 40), (3, 3, 64, 12), (2, 1, 8, 128), (1, 1, 100, 4)])
@pytest.mark.parametrize("strong", [False, True])
def test_chunks_match_the_walk(mode, H, G, N, dv, strong):
    """The tolerances of the segments' test; ``strong``: blocks of 32 tokens whose decays multiply to less than 2^-40."""
    G = H if mode == "matrix_memory" else G
    lens, slots = [130, 64, 255, 128, 300, 97], [3, 0, 6, -1, 1, 5]
    got, after, state, wants, cu = _case(mode, H, G, N, dv, lens, slots, strong, N + dv)
    memory = mode == "matrix_memory"
    for i, (want, S, n, m) in enumerate(wants):
        assert _rel(got[cu[i]:cu[i + 1]], want) < (5e-5 if memory else 2e-5), i
        if slots[i] >= 0:
            row = after[slots[i]]
            assert _rel(row[:H * N * dv], S.flatten()) < 2e-5
            if memory:
                assert _rel(row[H * N * dv:H * N * (dv + 1)], n.flatten()) < 2e-5
                assert float((row[H * N * (dv + 1):H * N * (dv + 1) + H].double() - m).abs().max()) < 1e-5
            assert torch.equal(row[-4:], state[slots[i], -4:])
    for slot in {2, 4}:
        assert torch.equal(after[slot], state[slot])


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(mode, value):
    H, N, dv, lens, t, col = 2, 32, 16, [200, 130], 150, 3
    got, after, _, wants, cu = _case(mode, H, H, N, dv, lens, [0, 1], False, 9, poison=(t, col, value))
    clean, clean_after, _, _, _ = _case(mode, H, H, N, dv, lens, [0, 1], False, 9)
    other = [c for c in range(H * dv) if c != col]
    assert torch.equal(got[:, other], clean[:, other]) and torch.equal(got[:t, col], clean[:t, col]) and torch.equal(got[200:], clean[200:])
    assert not bool(torch.isfinite(got[t:200, col]).any())
    S = after[0, :H * N * dv].view(H, N, dv)
    assert not bool(torch.isfinite(S[0, :, col]).any()) and torch.equal(after[1], clean_after[1])
    assert torch.equal(S[:, :, 4:], clean_after[0, :H * N * dv].view(H, N, dv)[:, :, 4:])


@pytest.mark.parametrize("mode,what", [(m, w) for m in MODES for w in ("q", "k", "gate_a", "gate_b", "a")
                                        if (w != "gate_a" or m != "decay_rows") and (w != "gate_b" or m == "matrix_memory") and (w != "a" or m == "decay_rows")])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("strong", [False, True])
def test_inputs_that_are_not_finite_reach_no_earlier_token(mode, what, value, strong):
    """Queries, keys, gates and decays: other heads, the other request and earlier tokens keep their bits (blocks of row decays may take
    another form for the decay: their roundings), and what is not finite in the recurrence token by token is not finite here."""
    H, N, dv, lens, t = 2, 32, 16, [200, 130], 75
    got, after, _, wants, cu = _case(mode, H, H, N, dv, lens, [0, 1], strong, 9, poison=(t, 0, value), what=what)
    clean, clean_after, _, _, _ = _case(mode, H, H, N, dv, lens, [0, 1], strong, 9)
    assert torch.equal(got[:, dv:], clean[:, dv:]) and torch.equal(got[200:], clean[200:]) and torch.equal(after[1], clean_after[1])
    if what == "a":
        assert _rel(got[:t, :dv], clean[:t, :dv].double()) < 2e-6
    else:
        assert torch.equal(got[:t, :dv], clean[:t, :dv])
    want = wants[0][0][:, :dv]
    there = torch.isfinite(want)
    assert not bool((torch.isfinite(got[:200, :dv]) & ~there).any())
    if bool(there[t:].any()):                            # a query: its own token alone; a gate or a decay that only closes
        assert _rel(torch.where(there, got[:200, :dv], 0.0), torch.where(there, want, 0.0)) < 5e-5


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("gates", ["constant", "nearly constant", "ordinary"])
@pytest.mark.parametrize("H,N,dv,T", [(2, 64, 32, 2048), (4, 128, 128, 777)])
def test_errors_are_not_larger_than_the_segments(mode, gates, H, N, dv, T):
    """Against 64 bits, decays of nearly 1 and ordinary ones, on the same inputs; a tenth for two orders of the same roundings."""
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(len(mode) + len(gates))
    vary = {"constant": 0.0, "nearly constant": 0.01, "ordinary": 1.0}[gates]
    slow, memory = gates != "ordinary", mode == "matrix_memory"
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    full = lambda x: torch.full((H,), x, device=DEV)
    q, k, v = rand(T, H * N), rand(T, H * N), rand(T, H * dv)
    a = ga = gb = p0 = p1 = p2 = None
    if mode == "decay_rows":
        per_row = torch.rand(H * N, generator=gen).to(DEV)
        a = torch.exp(torch.nn.functional.logsigmoid((4 + 3 * per_row if slow else per_row) + vary * rand(T, H * N)) / 16)
    elif mode == "state_space":
        ga, p0, p1, p2 = -4 + vary * rand(T, H), full(-3.0 if slow else 0.0), full(0.1), full(1.0)
    else:
        both = torch.cat([0.3 * rand(T, H), (6.0 if slow else 2.0) + vary * rand(T, H)], dim=1)
        ga, gb, p0, p1 = both[:, :H], both[:, H:], full(0.0), full(0.0)
    cap, scale, size = (15.0 if memory else 0.0), N ** -0.5, H * N * dv + (H * N + H if memory else 0)
    results = []
    for way in (ops.linrec_chunks, ops.linrec_segments):
        st, out = torch.zeros(1, size + -size % 4, device=DEV), torch.empty(T, H * dv, device=DEV)
        length = {} if way is ops.linrec_chunks else {"segment": ops.linrec_segment_tokens([T], H, ops.linrec_segment_blocks(N, dv), ops.sm_count(st.device))}
        den = way(mode, q, k, v, a, ga, gb, p0, p1, p2, cap, scale, i32([0, T]), i32([0]), st, out, [T], H, H, N, dv, None, **length)
        results.append(((out.view(T, H, dv) / den.unsqueeze(-1)).view(T, H * dv) if memory else out, st))
    d = lambda x: None if x is None else x.double()
    heads = lambda x: None if x is None else x.double().view(T, H, -1)
    zero = lambda *shape: torch.zeros(*shape, dtype=torch.float64, device=DEV)
    want, S, n, m = _walk(mode, heads(q), heads(k), heads(v), heads(a), d(ga), d(gb), d(p0), d(p1), d(p2), cap, scale, zero(H, N, dv), zero(H, N), zero(H))
    errors = [(_rel(out, want), _rel(st[0, :H * N * dv], S.flatten())) for out, st in results]
    print("chunks and segments (outputs, state):", errors)
    assert errors[0][0] <= 1.1 * errors[1][0] and errors[0][1] <= 1.1 * errors[1][1], errors


@pytest.mark.parametrize("forget", [2.0, -3.0, -15.0])
def test_floors_of_the_matrix_memory_keep_their_bits(forget):
    """Small queries, so that an output is divided by exp(-m_t), and forget gates whose logarithms since the chunk's start add up to
    1,900: m_t stays as small as the input gates.  The outputs are no further from 64 bits than the walk's, or within four roundings
    (the gates, the exponential, the division, the sum)."""
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(11)
    H, N, dv, T = 2, 64, 32, 300
    rand = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)
    q, k, v = 1e-4 * rand(T, H * N), rand(T, H * N), rand(T, H * dv)
    gates = torch.cat([-3.0 + rand(T, H), forget + rand(T, H)], dim=1)
    zero, scale, width = torch.zeros(H, device=DEV), N ** -0.5, H * N * dv + H * N + 4
    outs = []
    for chunks in (True, False):
        st, out = torch.zeros(1, width, device=DEV), torch.empty(T, H * dv, device=DEV)
        args = (gates[:, :H], gates[:, H:], zero, zero, None, 15.0, scale, i32([0, T]), i32([0]), st, out)
        if chunks:
            den = ops.linrec_chunks("matrix_memory", q, k, v, None, *args, [T], H, H, N, dv, None)
            out = (out.view(T, H, dv) / den.unsqueeze(-1)).view(T, H * dv)
        else:
            ops.linrec("matrix_memory", q, k, v, *args, 1, H, H, N, dv, None)
        outs.append(out)
    heads, d = (lambda x: x.double().view(T, H, -1)), (lambda x: x.double())
    none = lambda *shape: torch.zeros(*shape, dtype=torch.float64, device=DEV)
    want, _, _, _ = _walk("matrix_memory", heads(q), heads(k), heads(v), None, d(gates[:, :H]), d(gates[:, H:]), d(zero), d(zero), None, 15.0, scale,
                          none(H, N, dv), none(H, N), none(H))
    errors = [_rel(o, want) for o in outs]
    assert errors[0] <= max(1.1 * errors[1], 2.0 ** -22), errors
