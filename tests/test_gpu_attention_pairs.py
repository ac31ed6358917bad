"""Prompt attention with two query tiles a block (attention_tc.cu, attention_tc_pairs_kernel), which long contexts with heads of more
than 64 run: against the oracle, and in every option against the kernel of one tile a block."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _force(monkeypatch, least):
    """The keys from which blocks own two tiles."""
    from photon_infer_b200.kernels import ops
    real = ops.load_module
    monkeypatch.setattr(ops, "load_module", lambda module, defines=None: real(
        module, dict(defines, AT_PAIRS_KEYS=least) if module == "attention_tc" else defines))


@pytest.mark.parametrize("n_q,n_kv,d,ps,window", [
    (4, 1, 128, 16, None), (32, 8, 128, 16, None), (6, 6, 112, 8, None), (16, 2, 128, 64, None), (4, 2, 128, 128, None),
    (6, 3, 128, 32, 70), (8, 2, 128, 16, 200), (5, 1, 96, 16, None), (7, 1, 128, 8, 33)])
def test_portions(n_q, n_kv, d, ps, window, monkeypatch):
    """Odd and even numbers of row tiles, portions from the start, in the middle and at the end, last tiles of keys that are not
    full, and requests with few rows that the kernel must leave alone."""
    from test_gpu_kernels import _tc_attention_case
    _force(monkeypatch, 0)
    lens = [200, 333, 700, 1, 90, 1100]
    steps = [(0, 200), (150, 183), (699, 1), (0, 1), (60, 30), (513, 587)]
    _tc_attention_case(n_q, n_kv, d, ps, window, lens, steps)


@pytest.mark.parametrize("spike", [0, 63, 64, 127, 128, 255, 256, 600])
def test_far_key(spike, monkeypatch):
    from test_gpu_kernels import _tc_attention_case
    _force(monkeypatch, 0)
    _tc_attention_case(4, 1, 128, 16, None, [700], [(560, 140)], seed=40 + spike, spike=spike)


@pytest.mark.parametrize("d,dv", [(112, 112), (128, 128), (128, 64)])
@pytest.mark.parametrize("window,keep,sink,cap,gate", [
    (None, 0, True, 0.0, False), (100, 5, False, 0.0, False), (100, 200, True, 0.0, True), (None, 0, False, 20.0, True)])
def test_options_match_the_kernel_of_one_tile(d, dv, window, keep, sink, cap, gate, monkeypatch):
    """Both round P to bfloat16 and the output once: they differ by two roundings of the output at most, and the running maximum
    in use may be another one."""
    from photon_infer_b200.kernels import ops
    gen = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(s, generator=gen).to(torch.bfloat16).to(DEV)
    n_q, n_kv, ps, lens = 6, 2, 16, [(0, 530), (300, 97), (1000, 300)]
    pages = sum(-(-(a + b) // ps) for a, b in lens) + 1
    kc, vc = rnd(pages, n_kv, ps, d), rnd(pages, n_kv, ps, dv)
    table, at = torch.full((len(lens), 90), -1, dtype=torch.int32), 0
    for i, (a, b) in enumerate(lens):
        n = -(-(a + b) // ps)
        table[i, :n] = torch.arange(at, at + n)
        at += n
    cu = torch.tensor([0, 530, 627, 927], dtype=torch.int32, device=DEV)
    positions = torch.cat([torch.arange(a, a + b) for a, b in lens]).to(torch.int32).to(DEV)
    q, sinks, gates = rnd(927, n_q * d), torch.randn(n_q, generator=gen).to(DEV), rnd(927, n_q * dv)
    outs = []
    for least in (0, 1 << 20):
        with monkeypatch.context() as m:
            _force(m, least)
            out, err = torch.full((927, n_q * dv), float("nan"), dtype=torch.bfloat16, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
            ops.attention_tc(q, out, kc, vc, table.to(DEV), cu, positions, 3, 530, n_q, n_kv, d, window, 1.0 / math.sqrt(d), err,
                             keep_first=keep, sink=sinks if sink else None, softcap=cap, gate=gates if gate else None, value_dim=dv)
            assert err.cpu().tolist()[0] == 0
            outs.append(out.float())
    assert not torch.isnan(outs[0]).any()
    assert float((outs[0] - outs[1]).abs().max()) <= 2.0 ** -7 * float(outs[1].abs().max())
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) <= 4e-3


@pytest.mark.parametrize("n_q,n_kv,d,dv", [(8, 2, 128, 128), (6, 2, 128, 64), (5, 1, 96, 96), (2, 2, 112, 112)])
@pytest.mark.parametrize("held,value", [(0, float("nan")), (37, float("inf")), (128, float("nan"))])
def test_values_that_are_not_finite_stay_out_of_earlier_query_tiles(n_q, n_kv, d, dv, held, value, monkeypatch):
    """A token's values reach the tokens before it no further than with one query tile a block: not the tile before, which ends
    between or at multiples of 16 keys, in the block's last tile of keys or in one before it."""
    from photon_infer_b200.kernels import ops
    _force(monkeypatch, 0)
    gen = torch.Generator().manual_seed(8)
    rnd = lambda *s: torch.randn(s, generator=gen).to(torch.bfloat16).to(DEV)
    group, ps, T = n_q // n_kv, 16, 330
    tile = 128 // group                                  # tokens of a query tile
    pages = -(-(held + T) // ps)
    q, kc, vc = rnd(T, n_q * d), rnd(pages, n_kv, ps, d), rnd(pages, n_kv, ps, dv)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)

    def run(values):
        out, err = torch.empty(T, n_q * dv, dtype=torch.bfloat16, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
        ops.attention_tc(q, out, kc, values, i32([list(range(pages))]), i32([0, T]), i32(list(range(held, held + T))), 1, T, n_q, n_kv, d, None,
                         1.0 / math.sqrt(d), err, value_dim=dv)
        assert err.cpu().tolist()[0] == 0
        return out

    clean = run(vc)
    for first in range(tile, T, 2 * tile):               # the first token that only the second tile of a block sees, and one more
        for token in {first, min(first + 5, T - 1)}:
            bad = vc.clone()
            bad[(held + token) // ps, :, (held + token) % ps] = value
            out = run(bad)
            assert torch.equal(out[:first], clean[:first]), token
            assert not bool(torch.isfinite(out[token:]).any())
