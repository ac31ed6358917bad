"""Prompt portions in true 32-bit (``ops.attention_rows``) against the general kernel, whose bits they are."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n_q,n_kv", [(8, 2), (3, 1), (4, 4), (32, 1), (40, 2)])
@pytest.mark.parametrize("lens,ctx,ps", [([1], [0], 16), ([7, 8, 9], [0, 25, 31], 16), ([1, 40, 1, 33], [95, 0, 63, 32], 5), ([2] * 40, [30] * 40, 16),
                                         ([203], [64], 1), ([5, 431], [600, 0], 32)])
def test_portions_get_the_general_kernels_bits(d, n_q, n_kv, lens, ctx, ps):
    """Portions of less than a block's tokens, of exactly that many and more, at the edges of the tiles of 32 keys, many requests, a
    missing page, and numbers in the cache that no token may see."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(sum(lens) + d)
    T, S = sum(lens), len(lens)
    total = [n + c for n, c in zip(lens, ctx)]
    width = max((t + ps - 1) // ps for t in total) + 1
    pages = sum((t + ps - 1) // ps for t in total) + 3
    perm = torch.randperm(pages).tolist()
    table = torch.full((S, width), -1, dtype=torch.int32)
    kc = torch.full((pages, n_kv, ps, d), float("nan"))
    vc = torch.full((pages, n_kv, ps, d), float("nan"))
    for s, t in enumerate(total):
        for i in range((t + ps - 1) // ps):
            page = perm.pop()
            used = min(ps, t - i * ps)
            kc[page, :, :used] = torch.randn(n_kv, used, d)
            vc[page, :, :used] = torch.randn(n_kv, used, d)
            table[s, i] = page
            if i * ps <= total[s] - 1 < i * ps + used:
                vc[page, :, used - 1] = float("inf")               # only the request's last token may see it
    if ctx[-1] > ps:
        table[-1, 0] = -1                                          # a page that is not there: its keys are left out
    cu = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    seq = torch.cat([torch.full((n,), i, dtype=torch.int32) for i, n in enumerate(lens)]).to(DEV)
    pos = torch.cat([torch.arange(c, c + n, dtype=torch.int32) for n, c in zip(lens, ctx)]).to(DEV)
    q = torch.randn(T, (n_q + 2 * n_kv) * d, device=DEV)[:, :n_q * d]
    kc, vc, table = kc.to(DEV), vc.to(DEV), table.to(DEV)
    want, got = torch.full((T, n_q * d), 7.0, device=DEV), torch.full((T, n_q * d), 8.0, device=DEV)
    flags = [torch.zeros(4, dtype=torch.int32, device=DEV) for _ in range(2)]
    ops.paged_attention(q, want, kc, vc, table, seq, pos, n_q, n_kv, d, None, 1 / math.sqrt(d), flags[0])
    assert ops.attention_rows_supported(q, got, kc, vc, n_q, n_kv, d) == (n_q // n_kv <= 32)
    ops.attention_rows(q, got, kc, vc, table, cu, pos, S, n_q, n_kv, d, 1 / math.sqrt(d), flags[1])
    assert torch.equal(want.nan_to_num(5.0), got.nan_to_num(5.0))
    last = (cu[1:] - 1).long()
    rest = torch.ones(T, dtype=torch.bool, device=DEV)
    rest[last] = False
    assert bool(torch.isfinite(got[rest]).all())
    assert int(flags[0][0]) == int(flags[1][0])
