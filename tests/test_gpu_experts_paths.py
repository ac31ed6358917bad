"""Routed experts: pairs that share an expert's rows in the matrix-vector products of a decode step, and the router's logits of
many tokens on the tensor cores."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("pairs", [[0], [3, 3], [2, 2, 2, 2, 2] * 3, [0, 5, 0, 1, 5, 0, 0, 0, 5, 3, 3, 0, 5, 5, 5, 5], [4] * 64,
                                   [i * 7 % 6 for i in range(64)], [i % 2 * 5 for i in range(33)], [1] * 31 + [2] + [1] * 9,
                                   [7, 0, 7, 0], [7, 0] * 12, [i % 5 for i in range(70)]])
@pytest.mark.parametrize("glu", [False, True])
def test_pairs_of_one_expert_get_the_bits_that_they_get_alone(pairs, glu):
    """Groups of one, of exactly four, of more, at the ends of the 64 pairs that are seen at once, beyond them, and ids behind the
    last expert (identity experts), whose rows stay as they are."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(len(pairs))
    E, N, K = 6, 74, 264
    w = torch.randn(E, N, K, device=DEV).bfloat16()
    x = torch.randn((len(pairs) + 1) // 2, K, device=DEV).bfloat16()
    f = torch.rand(len(pairs), device=DEV)
    ids = torch.tensor(pairs, dtype=torch.int32, device=DEV)
    cols = N // 2 if glu else N
    act = dict(glu=True, activation="silu") if glu else {}
    out = torch.full((len(pairs), cols), 9.0, device=DEV)
    ops.moe_gemv(x, 2, ids, w, out, weights=f, **act)
    for p, e in enumerate(pairs):
        one = torch.full((1, cols), 9.0, device=DEV)
        ops.moe_gemv(x[p // 2:p // 2 + 1], 1, ids[p:p + 1], w, one, weights=f[p:p + 1], **act)
        assert torch.equal(one[0], out[p]), p
        if e >= E:
            assert bool((out[p] == 9.0).all())
        elif not glu:
            want = (w[e].double() @ x[p // 2].double()) * f[p].double()
            assert float((out[p].double() - want).abs().max()) < K * 2.0 ** -24 * float((w[e].double().abs() @ x[p // 2].double().abs()).max())


@pytest.mark.parametrize("T,H,E,gate", [(64, 32, 2, False), (65, 64, 8, True), (79, 288, 16, False), (2049, 2048, 16, True), (130, 96, 33, True),
                                        (100, 160, 63, True), (100, 160, 64, True),
                                        (125001, 32, 2, False), (62507, 64, 8, True), (13889, 288, 16, False), (41669, 96, 33, True),
                                        (25011, 160, 63, True), (25003, 160, 64, True)])
@pytest.mark.parametrize("scoring", ["softmax_chosen", "softmax_all", "sigmoid", "softmax_raw"])
def test_router_of_many_tokens(T, H, E, gate, scoring):
    """The choice and the weights against 64 bits; a choice may differ only where two scores are closer than the logits' rounding
    (products of bfloat16 numbers are exact: H additions of at most 2^-23 of the sum of magnitudes)."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(T + E)
    h, wr, b = torch.randn(T, H, device=DEV).bfloat16(), (torch.randn(E, H, device=DEV) * H ** -0.5).bfloat16(), torch.randn(E, device=DEV) * 0.1
    wsg = (torch.randn(1, H, device=DEV) * H ** -0.5).bfloat16() if gate else None
    got = ops.moe_route(h, wr, b, 2, scoring, w_shared_gate=wsg)
    ids, weights, counts = got[:3]
    z = h.double() @ wr.double().t() + b.double()
    err = H * 2.0 ** -23 * (h.double().abs() @ wr.double().abs().t()).max()
    score = {"softmax_chosen": z, "softmax_all": torch.softmax(z, -1), "sigmoid": torch.sigmoid(z), "softmax_raw": torch.softmax(z, -1)}[scoring]
    top, want = torch.topk(z, 2, dim=-1)
    chosen = z.gather(1, ids.long())
    assert float((chosen - top).abs().max()) <= 2 * float(err)
    s = score.gather(1, ids.long())
    w = {"softmax_chosen": torch.softmax(s, -1), "softmax_all": s / s.sum(-1, keepdim=True), "sigmoid": s, "softmax_raw": s}[scoring]
    assert float((weights.double() - w).abs().max()) < 2e-5
    assert torch.equal(counts.cpu().long(), torch.bincount(ids.flatten().long().cpu(), minlength=E))
    if gate:
        assert float((got[3].double().flatten() - torch.sigmoid(h.double() @ wsg[0].double())).abs().max()) < 2e-5


@pytest.mark.parametrize("T,H,E,shift", [(2048, 2048, 16, 0.0), (1024, 4096, 16, 0.0), (8192, 512, 64, 0.0), (2048, 2048, 32, 0.5), (16384, 256, 8, 0.0)])
def test_router_of_many_tokens_is_as_exact_as_that_of_few(T, H, E, shift):
    """The same tokens in one step, whose logits the tensor cores form, and in steps too small for that: the error against 64 bits
    (root mean square) is no larger.  All experts are chosen, so that every logit shows in a weight."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(T + E)
    h, wr = (torch.randn(T, H, device=DEV) + shift).bfloat16(), (torch.randn(E, H, device=DEV) * H ** -0.5).bfloat16()
    b = torch.randn(E, device=DEV) * 0.1
    many = ops.moe_route(h, wr, b, E, "sigmoid")
    few = [ops.moe_route(p, wr, b, E, "sigmoid") for p in h.split(T // 2)]
    want = torch.sigmoid(h.double() @ wr.double().t() + b.double())
    error = lambda ids, weights: float((weights.double() - want.gather(1, ids.long())).pow(2).mean().sqrt())
    e = error(many[0], many[1]), error(torch.cat([f[0] for f in few]), torch.cat([f[1] for f in few]))
    print("errors of many and of few:", e)
    assert e[0] <= 1.02 * e[1], e
