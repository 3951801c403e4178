"""The general kernel where its tile and K split are chosen for the shape: every tile x split x group size against the
integer path, K ranges that end inside a block or leave CTAs of a cluster without work, and the row scatter through a split."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import w2a8_oracle as O
from slimkernels_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(built_libs):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests selected but no CUDA device is visible")


from gpu_util import DeviceProblem, random_problem, to_np  # noqa: E402


# Tolerance of the first test: fp16 rounding of the output (2^-11 of the largest value) and the accumulators' 2^22 bias, each
# of whose sums is rounded to 1/4 at most 16 groups long: 4e-3 of the largest value covers both at these depths.
@pytest.mark.parametrize("tile", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("G,K", [(128, 640), (128, 1408), (256, 1280), (384, 1152), (64, 576), (64, 1088), (32, 352), (32, 1120)])
def test_every_tile_split_and_group_size(tile, split, G, K):
    M, N = {16: 13, 32: 45, 64: 70, 128: 200, 256: 300}[tile], 200
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=tile + split + K)
    dp = DeviceProblem(x_q, xs, wp, ws, G).force(kernel=capi.KERNEL_TCGEN05, token_tile=tile, split_k=split)
    y = dp.gemm(ld_out=N + 5)
    ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
    assert np.abs(to_np(y)[:, :N] - ref).max() <= 4e-3 * max(1.0, np.abs(ref).max())
    assert torch.isnan(y[:, N:]).all() and torch.equal(dp.gemm(ld_out=N + 5)[:, :N], y[:, :N])


# Where the MMA issuers take K blocks (or groups) in turn: one block or group in all, odd numbers of either, less and more than
# the rings and accumulator buffers hold, a last block with one group.  Tolerance as above.
@pytest.mark.parametrize("tile,M", [(64, 61), (128, 128), (256, 257)])
@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("G,K", [(128, 128), (128, 256), (128, 384), (128, 896), (128, 1664), (64, 64), (64, 128), (64, 192), (64, 832),
                                 (64, 1600), (32, 32), (32, 96), (32, 288), (256, 256), (256, 768)])
def test_turns_of_the_issuers(tile, M, split, G, K):
    x_q, xs, wp, ws = random_problem(M, 130, K, G, seed=tile + split + K)
    dp = DeviceProblem(x_q, xs, wp, ws, G).force(kernel=capi.KERNEL_TCGEN05, token_tile=tile, split_k=split)
    ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
    y = dp.gemm()
    assert np.abs(to_np(y) - ref).max() <= 4e-3 * max(1.0, np.abs(ref).max())
    assert dp.plan.device_status() == 0 and torch.equal(dp.gemm(), y)


@pytest.mark.parametrize("G", [32, 64, 128, 256])
@pytest.mark.parametrize("M,N,K", [(40, 512, 4096), (96, 1024, 4096), (130, 300, 11008), (333, 1000, 4096), (512, 2048, 2048),
                                   (600, 4096, 2048)])
def test_default_launch(G, M, N, K):
    K = K // G * G
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=M + G)
    dp = DeviceProblem(x_q, xs, wp, ws, G)
    y = to_np(dp.gemm())
    ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
    assert np.abs(y - ref).max() <= 1e-2
    route = dp.plan.query_route(M)
    assert route["kernel"] in (capi.KERNEL_TCGEN05, capi.KERNEL_DIRECT)
    assert route["token_tile"] <= dp.plan.query_launch(M)["token_tile"]


def test_row_scatter_takes_the_same_launch_as_the_plain_call():
    """256 tokens on few feature tiles run with smaller token tiles or a K split: the rows dealt out are the same bits."""
    M, N, K, rows = 512, 384, 11008, 256
    x_q, xs, wp, ws = random_problem(M, N, K, 128, seed=7)
    dp = DeviceProblem(x_q, xs, wp, ws)
    assert dp.plan.query_route(M) != dp.plan.query_launch(M)
    y = dp.gemm()
    for ld in (N, N + 3):
        bufs = [torch.zeros(2 * rows, ld, dtype=torch.float16, device="cuda") for _ in range(2)]
        ptrs = (ctypes.c_void_p * 2)(*[b.data_ptr() for b in bufs])
        assert capi.load().sk_w2a8_gemm_rowscatter(dp.plan.handle, M, dp.x_q.data_ptr(), K, dp.x_scale.data_ptr(), ptrs, 2, rows,
                                                   rows, ld, dp.stream()) == capi.SK_OK
        torch.cuda.synchronize()
        assert dp.plan.device_status() == 0
        for d in range(2):
            assert torch.equal(bufs[d][rows:, :N], y[d * rows:(d + 1) * rows]) and not bufs[d][:rows].any()
            assert not bufs[d][:, N:].any()
