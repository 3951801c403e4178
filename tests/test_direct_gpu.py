"""The direct decode kernel (weights from HBM to registers to mma.sync) against exact integers and the oracle, at the edges
of its tiles: 8 tokens, 16 features per MMA, 128-feature weight tiles, K blocks cut inside by group sizes 64 and 32, fewer
K blocks than warps, ragged last tiles."""
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


@pytest.mark.parametrize("G,K", [(128, 128), (128, 640), (128, 4096), (256, 768), (384, 1152), (64, 64), (64, 192), (64, 1088),
                                 (32, 32), (32, 352), (32, 1120)])
@pytest.mark.parametrize("M,N", [(1, 5), (8, 130), (9, 64), (16, 392), (17, 128), (24, 257), (32, 1000), (33, 40), (70, 200)])
def test_exact_integers(G, K, M, N):
    """Scales 1 and 2 and small activations: every output is an integer that fp16 holds exactly, so the comparison is exact.
    Deep K has 340 activations of -1 or 1 per token, anywhere in it and some in its last group."""
    rng = np.random.default_rng(M * N + K + G)
    lim = max(1, min(127, 2048 // (6 * K)))                        # |sum| <= 6 K lim or 6 * 340, below 2048
    x_q = rng.integers(-lim, lim + 1, size=(M, K), dtype=np.int8)
    if 6 * K * lim > 2048:
        x_q[:] = 0
        for row in x_q:
            at = rng.permutation(K)[:332]
            row[at] = rng.choice([-1, 1], size=332)
            row[K - G + rng.permutation(G)[:8]] = rng.choice([-1, 1], size=8)
    wp = rng.integers(0, 256, size=(N, K // 4), dtype=np.uint8)
    ws = rng.integers(1, 3, size=(K // G, N)).astype(np.float16)
    zp = int(rng.integers(0, 4))
    dp = DeviceProblem(x_q, np.ones(M, dtype=np.float32), wp, ws, G, zp).force(kernel=capi.KERNEL_DIRECT)
    assert dp.plan.query_route(M)["kernel"] == capi.KERNEL_DIRECT
    weights = (O.unpack_matrix(wp).astype(np.int64) - zp) * ws.astype(np.int64).repeat(G, axis=0).T
    want = x_q.astype(np.int64) @ weights.T
    assert np.abs(want).max() <= 2048
    y = to_np(dp.gemm(ld_out=N + 3))
    np.testing.assert_array_equal(y[:, :N], want.astype(np.float32))
    assert np.isnan(y[:, N:]).all(), "wrote outside the N columns"


@pytest.mark.parametrize("G", [32, 64, 128, 256])
@pytest.mark.parametrize("M,N,K", [(1, 392, 4096), (13, 520, 11008), (24, 136, 2048), (32, 4096, 4096)])
def test_scales_against_the_oracle_and_repeated_launches(G, M, N, K):
    # fp32 sums of at most 344 group products and one rounding to fp16: far inside the 1e-2 of the format's own bar
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=M + G)
    dp = DeviceProblem(x_q, xs, wp, ws, G).force(kernel=capi.KERNEL_DIRECT)
    y = dp.gemm()
    ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
    assert np.abs(to_np(y) - ref).max() <= 2.0 ** -10 * max(1.0, np.abs(ref).max())      # an fp16 ulp at the largest value
    assert torch.equal(dp.gemm(), y) and torch.equal(dp.force(kernel=capi.KERNEL_DIRECT, dependent_launch=1).gemm(), y)


@pytest.mark.parametrize("G,K", [(64, 4160), (64, 11072), (32, 4128), (32, 11040), (128, 8320), (256, 8448)])
@pytest.mark.parametrize("M,N", [(1, 72), (13, 136), (24, 40), (31, 200)])
def test_deep_ragged_k_and_every_split(G, K, M, N):
    """K that ends inside a block (group sizes 64 and 32) or leaves the warps and CTAs of a split uneven shares, every ring slot
    used several times: full-range activations and random scales, the K split chosen and forced."""
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=K + M)
    ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
    bound = 2.0 ** -10 * max(1.0, np.abs(ref).max())               # an fp16 ulp at the largest value, as above
    dp = DeviceProblem(x_q, xs, wp, ws, G)
    for split in (0, 1, 2, 4, 8):
        dp.force(kernel=capi.KERNEL_DIRECT, split_k=split)
        q = dp.plan.query_route(M)
        assert q["kernel"] == capi.KERNEL_DIRECT and (q["split_k"] == split if split else q["split_k"] > 1)
        assert np.abs(to_np(dp.gemm()) - ref).max() <= bound


def test_extreme_operands_and_bf16():
    for byte, xv, zp in [(0xFF, 127, 0), (0x00, -127, 3), (0xFF, -127, 1), (0x00, 127, 2)]:
        x_q = np.full((4, 256), xv, dtype=np.int8)
        wp = np.full((72, 64), byte, dtype=np.uint8)
        ws = np.full((2, 72), 0.005, dtype=np.float16)
        xs = np.full(4, 0.01, dtype=np.float32)
        dp = DeviceProblem(x_q, xs, wp, ws, 128, zp, torch.bfloat16).force(kernel=capi.KERNEL_DIRECT)
        ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, 128, zp)
        assert np.abs(to_np(dp.gemm()) - ref).max() <= 2.0 ** -8 * np.abs(ref).max()


def test_several_destinations_and_padded_rows():
    M, N, K = 10, 136, 512
    x_q, xs, wp, ws = random_problem(M, N, K, 128, seed=5)
    dp = DeviceProblem(x_q, xs, wp, ws, ld_x=K + 48).force(kernel=capi.KERNEL_DIRECT)
    y = dp.gemm()
    bufs = [torch.full((M, N + 11), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    ptrs = (ctypes.c_void_p * 3)(*[b.data_ptr() for b in bufs])
    assert capi.load().sk_w2a8_gemm_scatter(dp.plan.handle, M, dp.x_q.data_ptr(), dp.ld_x, dp.x_scale.data_ptr(), ptrs, 3,
                                            N + 11, 7, dp.stream()) == capi.SK_OK
    torch.cuda.synchronize()
    for b in bufs:
        assert torch.equal(b[:, 7:7 + N], y) and torch.isnan(b[:, :7]).all() and torch.isnan(b[:, 7 + N:]).all()


def test_route_keeps_what_the_tensor_memory_kernels_refuse():
    x_q, xs, wp, ws = random_problem(4, 128, 256, 128, seed=1)
    dp = DeviceProblem(x_q, xs, wp, ws)
    assert dp.plan.query_route(4)["kernel"] == capi.KERNEL_DIRECT and dp.plan.query_route(4096)["kernel"] == capi.KERNEL_TCGEN05
    for forced in (capi.KERNEL_TCGEN05, capi.KERNEL_TCGEN05_DECODE):
        assert dp.force(kernel=forced).plan.query_route(4)["kernel"] == forced
    K = 67584                                                     # too deep for the running sums of the general kernel
    dp = DeviceProblem(np.zeros((300, K), np.int8), np.ones(300, np.float32), np.zeros((128, K // 4), np.uint8),
                       np.ones((K // 128, 128), np.float16)).force(kernel=capi.KERNEL_DIRECT)
    with pytest.raises(capi.SkError):
        dp.gemm()


def _captured_launches(fn):
    """(grid, block, dynamic shared memory) of the kernels that fn launches, from a captured graph."""
    from cuda.bindings import driver
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    handle = driver.CUgraph(init_value=graph.raw_cuda_graph())
    _, _, count = driver.cuGraphGetNodes(handle)
    _, nodes, count = driver.cuGraphGetNodes(handle, count)
    out = []
    for node in nodes[:count]:
        err, p = driver.cuGraphKernelNodeGetParams(node)
        assert int(err) == 0
        out.append(((p.gridDimX, p.gridDimY, p.gridDimZ), p.blockDimX, p.sharedMemBytes))
    return out


@pytest.mark.parametrize("M,N,K", [(1, 4096, 11008), (8, 4096, 4096), (16, 12288, 4096), (24, 4096, 4096), (8, 57344, 512),
                                   (16, 57344, 512)])
def test_launch_floor_probe_has_the_geometry_of_the_launch_it_stands_for(M, N, K):
    from slimkernels_b200.torch import W2A8Plan
    x_q = torch.zeros(M, K, dtype=torch.int8, device="cuda")
    xs = torch.ones(M, device="cuda")
    out = torch.empty(M, N, dtype=torch.float16, device="cuda")
    plan = W2A8Plan(torch.zeros(N, K // 4, dtype=torch.uint8, device="cuda"), torch.ones(K // 128, N, dtype=torch.float16, device="cuda"))
    assert plan.query_route(M)["kernel"] == capi.KERNEL_DIRECT
    plan.gemm(x_q, xs, out=out)
    plan.launch_floor_probe(M)
    torch.cuda.synchronize()
    assert _captured_launches(lambda: plan.launch_floor_probe(M)) == _captured_launches(lambda: plan.gemm(x_q, xs, out=out))
    with pytest.raises(RuntimeError):
        plan.launch_floor_probe(4096)
