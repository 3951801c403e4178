"""The row quantiser (a weight [N, K] in its checkpoint's own element type) against the oracle's quantise-and-pack rule:
the same bytes and fp16 scales, at the edges of its tiles (32 rows x 512 columns) and for every group size it takes."""
import numpy as np
import pytest
import torch

from oracle import w2a8_oracle as O
from slimkernels_b200 import capi

TYPES = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


def _rows(w, G, ld=None):
    N, K = w.shape
    ld = ld or K
    buf = torch.zeros(N, ld, dtype=w.dtype, device="cuda")
    buf[:, :K] = w.cuda()
    packed = torch.full((N, K // 4), 0xAA, dtype=torch.uint8, device="cuda")
    s16 = torch.full((K // G, N), float("nan"), dtype=torch.float16, device="cuda")
    rc = capi.load().sk_w2a8_quantize_weight_rows(buf.data_ptr(), TYPES[w.dtype], ld, N, K, G, packed.data_ptr(),
                                                  s16.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc, packed.cpu().numpy(), s16.cpu().numpy()


def _check(w, G, ld=None):
    rc, packed, s16 = _rows(w, G, ld)
    assert rc == capi.SK_OK
    codes, scales = O.quantize_to_uint2(np.ascontiguousarray(w.float().numpy().T), G)
    np.testing.assert_array_equal(s16.view(np.uint16), scales.astype(np.float16).view(np.uint16))
    np.testing.assert_array_equal(packed, O.pack_matrix(np.ascontiguousarray(codes.T)))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", list(TYPES))
@pytest.mark.parametrize("N,K,G", [(1, 128, 128), (31, 512, 128), (33, 640, 128), (77, 1536, 512), (64, 96, 32), (5, 48, 16),
                                   (130, 1088, 64), (32, 2048, 256)])
def test_rows_bit_exact(dtype, N, K, G):
    g = torch.Generator().manual_seed(N + K + G)
    _check((torch.randn(N, K, generator=g) * 0.05).to(dtype), G)


@pytest.mark.gpu
def test_rows_ties_floor_and_pitch():
    g = torch.Generator().manual_seed(1)
    w = torch.randn(40, 256, generator=g)
    w[0, :8] = torch.tensor([1.5, 0.5, -0.5, 0.25, -1.5, 1.0, -0.75, 1.25])
    w[0, 8:128] = 0.0                                                  # scale 1: ties at +-1/2 and 3/2
    w[1] = 0.0                                                         # the 1e-9 floor
    w[2, :128] = torch.tensor([1e-12, -1e-12, 5e-10, 1e-9] * 32)
    w[3, :128] = -w[3, :128].abs()                                     # negative maximum
    for dtype in TYPES:
        _check(w.to(dtype), 128, ld=264)


@pytest.mark.gpu
def test_rows_refuses_what_it_does_not_take_and_from_float_still_does():
    from slimkernels_b200.torch import W2A8Linear
    for G in (8, 48, 1024):
        rc, _, _ = _rows(torch.zeros(4, 3072), G)
        assert rc == capi.SK_ERR_UNAVAILABLE
    g = torch.Generator().manual_seed(2)
    for w, G in ((torch.randn(48, 384, generator=g), 96), (torch.randn(48, 512, generator=g).to(torch.float64), 128),
                 (torch.randn(512, 48, generator=g).t(), 128), (torch.randn(48, 516, generator=g)[:, 3:515].half(), 128)):
        lin = W2A8Linear.from_float(w, G)
        codes, scales = O.quantize_to_uint2(np.ascontiguousarray(w.float().numpy().T), G)
        np.testing.assert_array_equal(lin.w_packed.cpu().numpy(), O.pack_matrix(np.ascontiguousarray(codes.T)))
        np.testing.assert_array_equal(lin.w_scale.cpu().numpy(), scales.astype(np.float16))


def test_comparison_rule_equals_division():
    """code = [x >= -s/2] + [x > s/2] + [x >= t], t found by division near 1.5 s, equals clip(rint(fl(x / s)) + 1, 0, 3) on
    the floats around every threshold."""
    f = np.float32
    rng = np.random.default_rng(0)
    s = (rng.random(200000, dtype=f) * 3 + f(0.001)) * f(2.0) ** rng.integers(-28, 100, 200000).astype(f)
    near = (f(1.5) * s).view(np.int32)
    t = np.full_like(s, np.nan)
    for d in (1, 0, -1, -2):
        x = (near + d).astype(np.int32).view(f)
        t = np.where(x / s >= f(1.5), x, t)
    assert not np.isnan(t).any()
    for centre in (f(0.5) * s, f(-0.5) * s, f(1.5) * s):
        for d in range(-4, 5):
            x = (centre.view(np.int32) + d).astype(np.int32).view(f)
            want = np.clip(np.rint(x / s) + 1, 0, 3)
            got = (x >= f(-0.5) * s).astype(int) + (x > f(0.5) * s) + (x >= t)
            np.testing.assert_array_equal(got, want)
