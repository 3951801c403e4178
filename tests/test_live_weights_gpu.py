"""A plan borrows its scales (and, given tiled, its codes).  With group sizes other than 128, and from 33 tokens on, a call
reads what these buffers hold when it runs in its stream.  (Up to 32 tokens with group size 128 may use the copy of the scales
that was made with the plan.)"""
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


def _at_offset(t, halves):
    """The same scales at `halves` halves past an aligned address, with NaN in front of them and behind."""
    buf = torch.full((t.numel() + halves + 64,), float("nan"), dtype=t.dtype, device=t.device)
    view = buf[halves:halves + t.numel()].view(t.shape)
    view.copy_(t)
    return view


# rows of whole 16-byte pieces, of words, and with N odd rows that start inside one; 200 and 130 leave a feature tile ragged
@pytest.mark.parametrize("G", [32, 64, 128, 256])
@pytest.mark.parametrize("M,N", [(1, 200), (7, 130), (16, 77), (24, 393), (32, 40), (60, 200), (100, 65), (300, 264)])
@pytest.mark.parametrize("offset", [0, 2, 1])
def test_a_change_of_the_scales_is_seen(G, M, N, offset):
    K = 1280
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=M + G)
    dp = DeviceProblem(x_q, xs, wp, ws, G)
    dp.w_scale = _at_offset(dp.w_scale, offset)
    dp.plan = capi.Plan(0, N, K, G, 1, dp.w_packed.data_ptr(), dp.w_scale.data_ptr(), capi.SK_OUT_F16)
    copy = G == 128 and M <= 32
    assert (dp.plan.query_route(M)["kernel"] == capi.KERNEL_DIRECT) == (M <= 100 and (copy or offset != 1))
    for seed in (1, 2):
        if seed == 2 and not copy:
            ws = np.random.default_rng(5).uniform(0.001, 0.01, size=ws.shape).astype(np.float16)
            dp.w_scale.copy_(torch.from_numpy(ws))
        ref = O.w2a8_gemm_int_path(x_q, xs, wp, ws, G)
        # fp16 rounding of the result, and for the general kernel its sums' (see test_general_launch_gpu.py)
        assert np.abs(to_np(dp.gemm()) - ref).max() <= 4e-3 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("G", [32, 64, 256, 512])
@pytest.mark.parametrize("M", [1, 8])
def test_a_change_of_the_scales_is_seen_by_the_kernel_that_quantises(G, M):
    from slimkernels_b200.torch import W2A8Linear
    lin = W2A8Linear.from_float(torch.randn(136, 1024, device="cuda") * 0.05, G)
    x = torch.randn(M, 1024, device="cuda").half()
    plan = lin.plan()
    lin(x)
    lin.w_scale.data.mul_(2)                       # (behind autograd's version counter: the plan stays)
    assert lin.plan() is plan
    y = lin(x)
    fresh = W2A8Linear(lin.w_packed, lin.w_scale.clone(), G)
    assert torch.equal(y, fresh(x))


@pytest.mark.parametrize("G,M", [(64, 4), (32, 20), (256, 8), (128, 48), (128, 300)])
def test_a_borrowed_tiled_weight_refilled_in_stream_order(G, M):
    """The buffer is rewritten by a kernel right in front of the GEMM, again and again."""
    from slimkernels_b200.torch import W2A8Plan, repack_weight
    N, K = 520, 2048
    x_q, xs, wp, ws = random_problem(M, N, K, G, seed=G + M)
    _, _, wp2, _ = random_problem(M, N, K, G, seed=G + M + 1)
    x, s, sc = (torch.from_numpy(a).cuda() for a in (x_q, xs, ws))
    tiled = [repack_weight(torch.from_numpy(w).cuda()) for w in (wp, wp2)]
    buf = tiled[0].clone()
    plan = W2A8Plan(buf, sc, N=N, K=K, group_size=G, tiled=True)
    want = []
    for i in range(2):
        buf.copy_(tiled[i])
        torch.cuda.synchronize()
        want.append(plan.gemm(x, s))
        torch.cuda.synchronize()
    refs = [O.w2a8_gemm_int_path(x_q, xs, w, ws, G) for w in (wp, wp2)]
    for y, ref in zip(want, refs):
        assert np.abs(to_np(y) - ref).max() <= 4e-3 * max(1.0, np.abs(ref).max())
    got = []
    for i in range(40):
        buf.copy_(tiled[i % 2])
        got.append(plan.gemm(x, s))
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))
