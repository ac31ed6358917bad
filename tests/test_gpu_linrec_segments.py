"""The recurrences in segments (``ops.linrec_segments``) against the same recurrence token by token in 64 bits: segments that
end inside a chunk of 16 tokens, requests with one segment beside requests with many, states that are not zero, reused
and negative slots, odd and unaligned sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _walk(mode, q, k, v, a, ga, gb, p0, p1, p2, cap, scale, S, n, m):
    """One request: tensors in 64 bits ``q, k, a [L, H, N]``, ``v [L, H, dv]``, gates ``[L, H]``."""
    out = []
    softplus, logsigmoid = torch.nn.functional.softplus, torch.nn.functional.logsigmoid
    for t in range(q.shape[0]):
        write = k[t][:, :, None] * v[t][:, None, :]
        if mode == "state_space":
            dt = softplus(ga[t] + p1)
            S = torch.exp(-torch.exp(p0) * dt)[:, None, None] * S + dt[:, None, None] * write
            out.append(torch.einsum("hnv,hn->hv", S, q[t]) * scale + p2[:, None] * v[t])
        elif mode == "matrix_memory":
            i, f = cap * torch.tanh((ga[t] + p0) / cap), logsigmoid(cap * torch.tanh((gb[t] + p1) / cap))
            new = torch.maximum(f + m, i)
            keep, take = torch.exp(f + m - new), torch.exp(i - new)
            m = new
            S = keep[:, None, None] * S + take[:, None, None] * write
            n = keep[:, None] * n + take[:, None] * k[t]
            den = torch.maximum(((n * q[t]).sum(-1) * scale).abs(), torch.exp(-m)) + 1e-6
            out.append(torch.einsum("hnv,hn->hv", S, q[t]) * scale / den[:, None])
        elif mode == "forget_write":
            S = S + k[t][:, :, None] * (v[t][:, None, :] - S)
            out.append(torch.einsum("hnv,hn->hv", S, q[t]) * scale)
        else:
            S = a[t][:, :, None] * S + write
            out.append(torch.einsum("hnv,hn->hv", S, q[t]) * scale)
    return torch.stack(out).flatten(1), S, n, m


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


@pytest.mark.parametrize("mode", ["state_space", "matrix_memory", "forget_write", "decay_rows"])
@pytest.mark.parametrize("H,G,N,dv,segment", [(2, 2, 128, 128, 16), (4, 2, 128, 40, 48), (1, 1, 16, 8, 32), (3, 3, 7, 11, 16), (2, 1, 56, 65, 64),
                                              (1, 1, 200, 17, 32), (1, 1, 256, 32, 112), (1, 1, 300, 12, 48)])
@pytest.mark.parametrize("strong", [False, True])
def test_segments_match_the_walk(mode, H, G, N, dv, segment, strong):
    """``strong``: decays so strong that a chunk's product leaves the range in which the walk is scaled by it, in some chunks."""
    from photon_infer_b200.kernels import ops
    if mode == "matrix_memory" and G != H:
        G = H
    gen = torch.Generator().manual_seed(N + dv + segment)
    lens, slots = [130, 1, 0, 16, 47, 113, 129], [3, 0, 6, -1, 1, 5, 2]
    T = sum(lens)
    rows = torch.randn(T, 3 * G * N + H * dv + 2 * H + (3 if N % 4 else 4), generator=gen)
    a0 = 3 * G * N
    rows[:, 2 * G * N:a0] = torch.sigmoid(rows[:, 2 * G * N:a0] + 2.0) ** (40 if strong else 1)      # decays
    if mode == "forget_write":
        rows[:, G * N:2 * G * N] = torch.sigmoid(rows[:, G * N:2 * G * N] * (4.0 if strong else 1.0) + (4.0 if strong else -2.0))   # write gates
    p0, p1, p2 = (0.5 * torch.randn(H, generator=gen) for _ in range(3))
    p1 = p1 + ((-3.0 if strong else 3.0) if mode == "matrix_memory" else -1.0)
    p0 = p0 + (2.0 if strong and mode == "state_space" else 0.0)
    width = H * N * dv + (H * N + H if mode == "matrix_memory" else 0) + 4
    state = torch.randn(7, width, generator=gen)
    st, r = state.to(DEV), rows.to(DEV)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    out = torch.full((T, H * dv), float("nan"), device=DEV)
    err = torch.zeros(4, dtype=torch.int32, device=DEV)
    memory, per_head = mode == "matrix_memory", mode in ("matrix_memory", "state_space")
    b0 = a0 + H * dv
    cap, scale = (6.0 if memory else 0.0), N ** -0.5
    den = ops.linrec_segments(mode, r[:, :G * N], r[:, G * N:2 * G * N], r[:, a0:b0], r[:, 2 * G * N:a0] if mode == "decay_rows" else None,
                              r[:, b0:b0 + H] if per_head else None, r[:, b0 + H:b0 + 2 * H] if memory else None,
                              p0.to(DEV) if per_head else None, p1.to(DEV) if per_head else None, p2.to(DEV) if mode == "state_space" else None,
                              cap, scale, i32(cu), i32(slots), st, out, lens, H, G, N, dv, err, segment=segment)
    if memory:
        out = (out.view(T, H, dv) / den.unsqueeze(-1)).view(T, H * dv)
    assert err.cpu().tolist()[0] == 0
    got, after = out.cpu(), st.cpu()
    seen = set()
    for i, L in enumerate(lens):
        if L == 0:
            continue
        x = rows[cu[i]:cu[i + 1]].double()
        heads = lambda z: z.reshape(L, G, N).repeat_interleave(H // G, dim=1)
        s0 = state[slots[i]].double() if slots[i] >= 0 else torch.zeros(width, dtype=torch.float64)
        S, n = s0[:H * N * dv].view(H, N, dv), s0[H * N * dv:H * N * dv + H * N].view(H, N) if memory else None
        m = s0[H * N * (dv + 1):H * N * (dv + 1) + H] if memory else None
        want, S, n, m = _walk(mode, heads(x[:, :G * N]), heads(x[:, G * N:2 * G * N]), x[:, a0:b0].reshape(L, H, dv), heads(x[:, 2 * G * N:a0]),
                              x[:, b0:b0 + H], x[:, b0 + H:b0 + 2 * H], p0.double(), p1.double(), p2.double(), cap, scale, S, n, m)
        # a state element is a sum of up to 130 terms, each a few roundings of 2^-24; the division by |n . q| adds its cancellation
        assert _rel(got[cu[i]:cu[i + 1]], want) < (5e-5 if memory else 2e-5), (i, L)
        if slots[i] >= 0:
            seen.add(slots[i])
            assert _rel(after[slots[i], :H * N * dv], S.flatten()) < 2e-5
            if memory:
                assert _rel(after[slots[i], H * N * dv:H * N * (dv + 1)], n.flatten()) < 2e-5
                assert float((after[slots[i], H * N * (dv + 1):H * N * (dv + 1) + H].double() - m).abs().max()) < 1e-5
            assert torch.equal(after[slots[i], -4:], state[slots[i], -4:])
    for slot in set(range(7)) - seen:
        assert torch.equal(after[slot], state[slot])


def test_running_maxima_far_from_zero():
    """Forget gates that close for hundreds of tokens and input gates at their bound: the scale of the state moves by hundreds of
    powers of e between segments, and nothing overflows."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(5)
    H, N, dv, L = 1, 32, 16, 300
    rows = torch.randn(L, 2 * N + dv, device=DEV)
    gi = torch.full((L, H), -20.0, device=DEV)
    gf = torch.full((L, H), -20.0, device=DEV)
    gi[100:140], gi[220:] = 20.0, 20.0
    gf[150:200] = 20.0
    z = torch.zeros(H, device=DEV)
    outs = []
    for segment in (16, 64, 304):
        st = torch.zeros(1, H * N * dv + H * N + H, device=DEV)
        o = torch.empty(L, H * dv, device=DEV)
        g = torch.cat([gi, gf], dim=1)
        den = ops.linrec_segments("matrix_memory", rows[:, :N], rows[:, N:2 * N], rows[:, 2 * N:], None, g[:, :H], g[:, H:], z, z, None, 15.0,
                                  N ** -0.5, i32([0, L]), i32([0]), st, o, [L], H, H, N, dv, None, segment=segment)
        o = o / den
        assert bool(torch.isfinite(o).all()) and bool(torch.isfinite(st).all())
        outs.append(o)
    st = torch.zeros(1, H * N * dv + H * N + H, device=DEV)
    o = torch.empty(L, H * dv, device=DEV)
    ops.linrec("matrix_memory", rows[:, :N], rows[:, N:2 * N], rows[:, 2 * N:], g[:, :H], g[:, H:], z, z, None, 15.0, N ** -0.5, i32([0, L]),
               i32([0]), st, o, 1, H, H, N, dv, None)
    for x in outs:
        assert _rel(x, o.double()) < 5e-5


@pytest.mark.parametrize("mode", ["state_space", "matrix_memory", "forget_write", "decay_rows"])
@pytest.mark.parametrize("gates", ["constant", "nearly constant", "ordinary"])
def test_slow_decays_keep_their_bits(mode, gates):
    """2,048 tokens whose decays are nearly 1 (and ordinary ones), in segments of the length that a step gets: the error against 64 bits
    is no larger than that of the walk token by token, or within two roundings of the state."""
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(len(mode) + len(gates))
    H, N, dv, T = 2, 64, 32, 2048
    vary = {"constant": 0.0, "nearly constant": 0.01, "ordinary": 1.0}[gates]
    slow = gates != "ordinary"
    rand = lambda *shape: torch.randn(*shape, generator=gen)
    q, k, v = rand(T, H * N), rand(T, H * N), rand(T, H * dv)
    per_row = torch.rand(H * N, generator=gen)
    a = ga = gb = p0 = p1 = p2 = None
    if mode == "forget_write":                                   # write gates of 1e-5 to 1e-2, or of 0.01 to 0.5
        k = (10.0 ** (-5 + 3 * per_row) if slow else 0.01 + 0.49 * per_row) * (1 + 0.5 * vary * torch.tanh(rand(T, H * N)))
    elif mode == "decay_rows":
        a = torch.exp(torch.nn.functional.logsigmoid((4 + 3 * per_row if slow else per_row) + vary * rand(T, H * N)) / 16)
    elif mode == "state_space":
        ga, p0, p1, p2 = -4 + vary * rand(T, H), torch.full((H,), -3.0 if slow else 0.0), torch.full((H,), 0.1), torch.ones(H)
    else:
        ga, gb, p0, p1 = 0.3 * rand(T, H), (6.0 if slow else 2.0) + vary * rand(T, H), torch.zeros(H), torch.tensor([0.0, 0.7])
    memory, cap, scale = mode == "matrix_memory", 15.0, N ** -0.5
    size = H * N * dv + (H * N + H if memory else 0)
    dev = lambda x: None if x is None else x.to(DEV)
    q, k, v, a, ga, gb, p0, p1, p2 = map(dev, (q, k, v, a, ga, gb, p0, p1, p2))
    if memory:
        gates_ab = torch.cat([ga, gb], dim=1)
        ga, gb = gates_ab[:, :H], gates_ab[:, H:]
    s1, o1 = torch.zeros(1, size, device=DEV), torch.empty(T, H * dv, device=DEV)
    den = ops.linrec_segments(mode, q, k, v, a, ga, gb, p0, p1, p2, cap if memory else 0.0, scale, i32([0, T]), i32([0]), s1, o1, [T], H, H, N, dv,
                              None)
    if memory:
        o1 = (o1.view(T, H, dv) / den.unsqueeze(-1)).view(T, H * dv)
    s2, o2 = torch.zeros(1, size, device=DEV), torch.empty(T, H * dv, device=DEV)
    if mode == "decay_rows":
        S, rows = torch.zeros(H, N, dv, device=DEV), []
        for t in range(T):
            S = torch.addcmul(a[t].view(H, N, 1) * S, k[t].view(H, N, 1), v[t].view(H, 1, dv))
            rows.append(torch.einsum("hnv,hn->hv", S, q[t].view(H, N)) * scale)
        s2[0], o2 = S.flatten(), torch.stack(rows).flatten(1)
    else:
        ops.linrec(mode, q, k, v, ga, gb, p0, p1, p2, cap if memory else 0.0, scale, i32([0, T]), i32([0]), s2, o2, 1, H, H, N, dv, None)
    d = lambda x: None if x is None else x.double()
    heads = lambda x: None if x is None else x.double().view(T, H, -1)
    zero = lambda *shape: torch.zeros(*shape, dtype=torch.float64, device=DEV)
    want, S, n, m = _walk(mode, heads(q), heads(k), heads(v), heads(a), d(ga), d(gb), d(p0), d(p1), d(p2), cap, scale, zero(H, N, dv), zero(H, N),
                          zero(H))
    errors = [(_rel(o, want), _rel(s[0, :H * N * dv], S.flatten())) for o, s in ((o1, s1), (o2, s2))]
    print("segments and walk (outputs, state):", errors)
    assert errors[0][1] <= max(1.1 * errors[1][1], 2.0 ** -23), errors
    assert errors[0][0] <= max(1.1 * errors[1][0], 2.0 ** -22), errors       # a sum of 64 such products behind it


@pytest.mark.parametrize("mode", [None, "silu_before", "sigmoid_after"])
@pytest.mark.parametrize("groups,gs", [(16, 128), (2, 1024), (3, 4), (1, 260), (9, 512)])
def test_norm_of_parts(mode, groups, gs):
    from photon_infer_b200.kernels import ops
    torch.manual_seed(groups + gs)
    T, W = 37, groups * gs
    x, gate, w, den = torch.randn(T, W, device=DEV), torch.randn(T, W + 8, device=DEV)[:, 4:4 + W], torch.randn(W, device=DEV), \
        torch.rand(T, groups, device=DEV) + 0.5
    for d in (None, den):
        out = torch.empty(T, W, dtype=torch.bfloat16, device=DEV)
        ops.part_rmsnorm(x, w, 1e-5, groups, out, gate=gate if mode else None, gate_mode=mode, den=d)
        y = x.double().view(T, groups, gs) / (d.double().unsqueeze(-1) if d is not None else 1.0)
        z = gate.double().view(T, groups, gs)
        y = y * (z * torch.sigmoid(z)) if mode == "silu_before" else y
        y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)).reshape(T, W) * w.double()
        y = y * torch.sigmoid(gate.double()) if mode == "sigmoid_after" else y
        assert float(((out.double() - y).abs() / (y.abs() + 1e-3)).max()) < 2.0 ** -8         # one rounding to bfloat16
