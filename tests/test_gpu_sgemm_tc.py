"""32-bit products of large weights as tensor-core products (gemm_f32_tc.cu): accuracy, the same bits for every row count, tile,
split and launch form, and what is not finite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (N, K): whole tiles; ragged tiles of features, of K and of the last group; few groups' worth of tiles; long K
SIZES = [(2048, 2048), (2050, 2052), (1030, 4100), (4160, 1020 + 8), (1024, 8192)]


def _product(x, w):
    """On the tensor cores, also weights of few columns, which ``linear`` leaves to the chain."""
    from photon_infer_b200.kernels import ops
    out = torch.empty(x.shape[0], w.shape[0], device=DEV)
    ops.sgemm_tc(x, w, out)
    return out


def _chain(x, w):
    """The product as gemm_f32.cu forms it: a chain of multiply-adds."""
    from photon_infer_b200.kernels import ops
    return torch.cat([ops.linear(x, w[i:i + 512].contiguous()) for i in range(0, w.shape[0], 512)], dim=1)


@pytest.mark.parametrize("N,K", SIZES)
def test_accuracy_and_the_same_bits_for_every_row_count(N, K):
    """Error: in a chunk of 64 the four additions of the large products are truncated, at most two units of 2^-23 each with the
    alignment inside the instruction, 8 units; up to 15 sums of chunks in a group and 7 of groups are rounded (half a unit each), 11;
    the products left out are below 1.51 units of their terms, and the truncations of the small products, twenty of two units of 2^-7 of
    the sum, below 0.32: 21 units of 2^-23 of the sum of magnitudes."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(21)
    x, w = torch.randn(513, K, device=DEV), torch.randn(N, K, device=DEV)
    out = _product(x, w)
    assert not ops.sgemm_tc_supported(w) or torch.equal(out, ops.linear(x, w))
    want = x.double() @ w.double().t()
    error = (out.double() - want).abs()
    assert bool((error <= 21 * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())).all())
    # no further from 64 bits than the chain of multiply-adds
    assert float(error.pow(2).mean()) <= float((_chain(x, w).double() - want).pow(2).mean())
    for rows in (1, 2, 15, 16, 17, 33, 64, 65, 96, 97, 200):
        assert torch.equal(_product(x[:rows], w), out[:rows]), rows
    assert torch.equal(_product(x[500:], w), out[500:])


@pytest.mark.parametrize("rows", [1, 16, 40])
def test_strided_rows_and_captured_launches(rows):
    from photon_infer_b200.kernels import ops
    torch.manual_seed(22)
    wide, w = torch.randn(rows, 2060, device=DEV), torch.randn(2048, 2052, device=DEV)
    x = wide[:, 5:2057]
    want = ops.linear(x.contiguous(), w)
    assert torch.equal(ops.linear(x, w), want)
    out = torch.zeros(rows, 2048 + 3, device=DEV)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        ops.linear(x, w, out[:, :2048])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[:, :2048], want) and float(out[:, 2048:].abs().max()) == 0.0


def test_more_rows_than_one_round_takes():
    torch.manual_seed(25)
    x, w = torch.randn(4096 + 33, 1024, device=DEV), torch.randn(4096, 1024, device=DEV)
    out = _product(x, w)
    assert torch.equal(out[4090:], _product(x[4090:], w)) and torch.equal(out[:40], _product(x[:40], w))


@pytest.mark.parametrize("N,K,tensor", [(1024, 4096, True), (2048, 2048, True), (1023, 8192, False), (1024, 4092, False), (4096, 1024, False),
                                        (8192, 2044, False)])
def test_which_weights(N, K, tensor):
    from photon_infer_b200.kernels import ops
    assert ops.sgemm_tc_supported(torch.empty(N, K, device=DEV)) == tensor


@pytest.mark.parametrize("rows", [9, 70])
def test_what_is_not_finite_is_what_the_chain_gives(rows):
    from photon_infer_b200.kernels import ops
    torch.manual_seed(23)
    x, w = torch.randn(rows, 2048, device=DEV), torch.randn(2048, 2048, device=DEV)
    x[0, 7], x[1, 9], x[2], x[3], x[4, :] = math.inf, math.nan, 3.4e38, 0.0, -math.inf
    w[11, 100], w[20] = -math.inf, 3e38
    out, want = ops.linear(x, w), _chain(x, w)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(out), finite) and not bool(finite.all())
    assert torch.equal(torch.nan_to_num(out[~finite], nan=7.0), torch.nan_to_num(want[~finite], nan=7.0))


@pytest.mark.parametrize("scale", [2.0 ** -60, 2.0 ** 60])
def test_magnitudes_far_from_one(scale):
    from photon_infer_b200.kernels import ops
    torch.manual_seed(24)
    x, w = torch.randn(20, 2048, device=DEV), torch.randn(2048, 2048, device=DEV)
    assert torch.equal(ops.linear(x * scale, w / scale), ops.linear(x, w))


@pytest.mark.parametrize("rows,one_launch", [(7, 1), (7, 0), (150, 0)])
def test_a_wait_that_runs_out_is_reported(rows, one_launch):
    """A build whose weights never come and whose waits give up after a few thousand polls: every warp gives up as a whole, the kernel
    reports PHOTON_DEV_WAIT_TIMEOUT and returns; the stock build runs right afterwards."""
    from ctypes import c_int, c_long, c_void_p
    from photon_infer_b200.csrc.build import load_module
    from photon_infer_b200.kernels import ops
    torch.manual_seed(26)
    N, K = 2048, 2048
    x, w, out = torch.randn(rows, K, device=DEV), torch.randn(N, K, device=DEV), torch.zeros(rows, N, device=DEV)
    err, scratch = torch.zeros(4, dtype=torch.int32, device=DEV), torch.empty(64 << 20, dtype=torch.uint8, device=DEV)
    f = load_module("gemm_f32_tc", {"FT_TEST_NO_LOADS": 1, "TC_WAIT_LIMIT": 4096}).photon_sgemm_tc
    f.argtypes = [c_void_p, c_long, c_void_p, c_long, c_void_p, c_long, c_int, c_int, c_int, c_int, c_void_p, c_long, c_void_p, c_void_p]
    f.restype = c_int
    assert f(x.data_ptr(), K, w.data_ptr(), K, out.data_ptr(), N, rows, N, K, one_launch, scratch.data_ptr(), scratch.numel(), err.data_ptr(),
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert err.cpu().tolist()[0] == 4
    err.zero_()
    ops.sgemm_tc(x, w, out, err)
    assert err.cpu().tolist()[0] == 0
    assert float((out.double() - x.double() @ w.double().t()).norm() / out.double().norm()) < 1e-6


@pytest.mark.parametrize("N,K", [(4095, 4096), (4096, 4096)])
def test_both_sides_of_the_line_between_one_launch_and_three(N, K):
    """The rows of a product of many: below 2^24 numbers one launch forms few rows, from there on three do."""
    from photon_infer_b200.kernels import ops
    torch.manual_seed(27)
    assert ops.SGEMM_ONE_LAUNCH_SIZE == 4096 * 4096
    x, w = torch.randn(40, K, device=DEV), torch.randn(N, K, device=DEV)
    out = ops.linear(x, w)
    for rows in (1, 3, 16):
        assert torch.equal(ops.linear(x[:rows], w), out[:rows]), rows
