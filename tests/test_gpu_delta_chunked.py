"""The delta rule in chunks of 32 tokens (``ops.delta_chunked``) against the rule token by token in 64 bits: chunks that are
not full, requests of one token beside long ones, states that are not zero, reused and negative slots, decays of nothing and of
everything, keys that repeat; and the convolution of many tokens in front of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


@pytest.mark.parametrize("H,G,dim,dv", [(2, 1, 128, 128), (3, 3, 128, 16), (4, 2, 40, 24), (1, 1, 7, 11), (2, 2, 128, 256), (2, 1, 64, 130)])
@pytest.mark.parametrize("gates", ["mild", "strong", "none"])
def test_chunks_match_the_walk(H, G, dim, dv, gates):
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(dim + dv)
    lens, slots = [130, 1, 0, 32, 47, 97, 64], [3, 0, 6, -1, 1, 5, 2]
    T, C = sum(lens), 2 * G * dim + H * dv
    y = torch.randn(T, C, generator=gen)
    q, k = (y[:, i * G * dim:(i + 1) * G * dim].view(T, G, dim) for i in (0, 1))
    q /= q.norm(dim=-1, keepdim=True) * dim ** 0.5
    k /= k.norm(dim=-1, keepdim=True)
    k[40:60] = k[39]                                             # one key again and again
    ab = torch.randn(T, 2 * H + 1, generator=gen)
    a_log, dt_bias = 0.5 * torch.randn(H, generator=gen), torch.full((H,), -2.0)
    if gates == "strong":
        a_log, dt_bias = a_log + 3.0, dt_bias + 4.0
        ab[50, :H] = 1e6                                         # a decay of 0
        ab[:, H:2 * H] += 3.0
    if gates == "none":
        ab[:, :H], ab[:, H:2 * H] = -100.0, 100.0                # decay 1, beta 1
    width = H * dim * dv + 5
    state = torch.randn(7, width, generator=gen)
    st, yd, abd = state.to(DEV), y.to(DEV), ab.to(DEV)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    o = torch.full((T, H * dv), float("nan"), device=DEV)
    err = torch.zeros(4, dtype=torch.int32, device=DEV)
    ops.delta_chunked(yd, abd[:, :2 * H], a_log.to(DEV), dt_bias.to(DEV), i32(cu), i32(slots), st, o, lens, G, H, dim, dv, err)
    assert err.cpu().tolist()[0] == 0
    got, after, seen = o.cpu(), st.cpu(), set()
    for r, L in enumerate(lens):
        if L == 0:
            continue
        x, z = y[cu[r]:cu[r + 1]].double(), ab[cu[r]:cu[r + 1]].double()
        heads = lambda t: t.reshape(L, G, dim).repeat_interleave(H // G, dim=1)
        qq, kk, v = heads(x[:, :G * dim]), heads(x[:, G * dim:2 * G * dim]), x[:, 2 * G * dim:].reshape(L, H, dv)
        g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(z[:, :H] + dt_bias.double()))
        beta = torch.sigmoid(z[:, H:2 * H])
        S = state[slots[r], :H * dim * dv].double().view(H, dim, dv) if slots[r] >= 0 else torch.zeros(H, dim, dv, dtype=torch.float64)
        want = []
        for t in range(L):
            S = g[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, kk[t]))
            S = S + kk[t][:, :, None] * u[:, None, :]
            want.append(torch.einsum("hkv,hk->hv", S, qq[t]).flatten())
        # sums of up to 128 and 130 terms of 32-bit products, each a few roundings of 2^-24; keys that repeat cancel
        assert _rel(got[cu[r]:cu[r + 1]], torch.stack(want)) < 2e-5, (r, L)
        if slots[r] >= 0:
            seen.add(slots[r])
            assert _rel(after[slots[r], :H * dim * dv], S.flatten()) < 2e-5
            assert torch.equal(after[slots[r], -5:], state[slots[r], -5:])
    for slot in set(range(7)) - seen:
        assert torch.equal(after[slot], state[slot])


def test_chunks_are_as_exact_as_the_walk():
    """2,048 tokens at the sizes of a real layer: the error against 64 bits is no larger than the token-by-token kernel's."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(3)
    T, H, G, dim, dv = 2048, 2, 1, 128, 128
    y = torch.randn(T, 2 * G * dim + H * dv, device=DEV)
    for i in (0, 1):
        p = y[:, i * dim:(i + 1) * dim]
        p /= p.norm(dim=-1, keepdim=True) * (dim ** 0.5 if i == 0 else 1.0)
    ab = torch.randn(T, 2 * H, device=DEV)
    a_log, dt_bias = torch.tensor([0.0, 2.0], device=DEV), torch.tensor([-5.0, -3.0], device=DEV)
    args = (y, ab, a_log, dt_bias, i32([0, T]), i32([0]))
    s1, s2 = torch.zeros(1, H * dim * dv, device=DEV), torch.zeros(1, H * dim * dv, device=DEV)
    o1, o2 = torch.empty(T, H * dv, device=DEV), torch.empty(T, H * dv, device=DEV)
    ops.delta_recurrent(*args, s1, o1, 1, G, H, dim, dv, None)
    ops.delta_chunked(*args, s2, o2, [T], G, H, dim, dv, None)
    yd, abd = y.double(), ab.double()
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(abd[:, :H] + dt_bias.double()))
    beta = torch.sigmoid(abd[:, H:])
    S, want = torch.zeros(H, dim, dv, dtype=torch.float64, device=DEV), torch.empty(T, H, dv, dtype=torch.float64, device=DEV)
    for t in range(T):
        k, q = yd[t, dim:2 * dim], yd[t, :dim]
        S = g[t][:, None, None] * S
        u = beta[t][:, None] * (yd[t, 2 * dim:].view(H, dv) - torch.einsum("hkv,k->hv", S, k))
        S = S + k[None, :, None] * u[:, None, :]
        want[t] = torch.einsum("hkv,k->hv", S, q)
    e = [(_rel(o, want.flatten(1)), _rel(s[0], S.flatten())) for o, s in ((o1, s1), (o2, s2))]
    print("errors of the walk and of the chunks:", e)
    assert e[1][0] <= 1.1 * e[0][0] and e[1][1] <= 1.1 * e[0][1], e


@pytest.mark.parametrize("H,G,dim,dv", [(4, 2, 128, 128), (3, 3, 40, 24), (2, 1, 7, 33)])
def test_convolution_of_many_tokens_gives_the_bits_of_few(H, G, dim, dv):
    """Requests of 1 to 70 tokens in one step of 150 against the same requests in steps of fewer than 64 tokens."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(dim)
    lens, slots = [70, 1, 2, 0, 60, 17], [2, 0, 5, 4, -1, 1]
    T, C, off = sum(lens), 2 * G * dim + H * dv, 8
    x = torch.randn(T, C + 3, device=DEV)[:, :C]
    taps = torch.randn(C, 4, device=DEV)
    state = torch.randn(6, off + 3 * C, device=DEV)

    def run(parts):
        st, y = state.clone(), torch.empty(T, C, device=DEV)
        for part in parts:                                       # (request, first token, tokens)
            rows = [sum(lens[:r]) + a + i for r, a, n in part for i in range(n)]
            cu, seq = [0], []
            for i, (_, _, n) in enumerate(part):
                cu.append(cu[-1] + n)
                seq += [i] * n
            out = torch.empty(len(rows), C, device=DEV)
            ops.delta_conv(x[rows], taps, i32(seq), i32(cu), i32([slots[r] for r, _, _ in part]), st, off, out, len(part), G, H, dim, dv, None)
            y[rows] = out
        return y, st
    whole = run([[(r, 0, n) for r, n in enumerate(lens)]])
    cut = run([[(0, 0, 33), (1, 0, 1)], [(0, 33, 37), (2, 0, 2)], [(4, 0, 60)], [(5, 0, 17)]])
    assert torch.equal(whole[0], cut[0]) and torch.equal(whole[1], cut[1])


@pytest.mark.parametrize("what", ["key", "query", "value", "decay", "step size"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [0, 13, 31, 40, 95])
def test_what_is_not_finite_reaches_no_earlier_token(what, bad, at):
    """One number of a token is not finite: the outputs before it are those that they are without it (up to the rounding of the eight
    tokens whose sums are then plain ones), and those that are not finite are the token-by-token kernel's."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(at)
    T, H, G, dim, dv = 100, 4, 2, 128, 48
    y = torch.randn(T, 2 * G * dim + H * dv, device=DEV)
    y[:, :2 * G * dim] *= dim ** -0.5
    ab = torch.randn(T, 2 * H, device=DEV)
    a_log, dt_bias = torch.zeros(H, device=DEV), torch.full((H,), -3.0, device=DEV)
    start = torch.randn(1, H * dim * dv, device=DEV)

    def run(chunks, y, ab):
        s, o = start.clone(), torch.empty(T, H * dv, device=DEV)
        args = (y, ab, a_log, dt_bias, i32([0, T]), i32([0]), s, o)
        ops.delta_chunked(*args, [T], G, H, dim, dv, None) if chunks else ops.delta_recurrent(*args, 1, G, H, dim, dv, None)
        return o, s
    clean = run(True, y, ab)[0]
    if what in ("decay", "step size"):
        ab[at, 1 if what == "decay" else H + 1] = bad
    else:
        y[at, {"key": G * dim + 5, "query": 5, "value": 2 * G * dim + dv + 7}[what]] = bad
    (o, s), (want, after) = run(True, y, ab), run(False, y, ab)
    assert torch.equal(o[:at // 8 * 8], clean[:at // 8 * 8])
    assert at == 0 or _rel(o[:at], clean[:at].double()) < 1e-6
    assert torch.equal(torch.isfinite(o), torch.isfinite(want)) and torch.equal(torch.isfinite(s), torch.isfinite(after))
    fine = torch.isfinite(want)
    assert _rel(o[fine], want[fine].double()) < 2e-5
