"""W2A8Linear / W2A8LlamaMLP forward in one native call: the same bits as its pieces for every activation layout, and plans
used on other streams than the one they were made on."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(built_libs):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests selected but no CUDA device is visible")


def _linear(N, K, G=128, out_dtype=torch.float16, seed=0):
    from slimkernels_b200.torch import W2A8Linear
    g = torch.Generator(device="cuda").manual_seed(seed)
    return W2A8Linear.from_float(torch.randn(N, K, generator=g, device="cuda") * 0.05, G, out_dtype=out_dtype)


def _by_pieces(lin, x):
    from slimkernels_b200.torch import quantize_activation_int8
    x_q, x_s = quantize_activation_int8(x.reshape(-1, x.shape[-1]).to(torch.float16).contiguous())
    return lin.plan().gemm(x_q, x_s).reshape(*x.shape[:-1], lin.out_features)


@pytest.mark.parametrize("K", [128, 4096, 8320, 18432])            # 2, 4 and 8 vectors per thread, and rows read twice
@pytest.mark.parametrize("M", [1, 5, 40])
def test_bf16_activations_are_rounded_to_fp16_on_the_way_in(M, K):
    lin = _linear(136, K, out_dtype=torch.bfloat16)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    x[0, :4] = torch.tensor([1e30, -3e38, 1e-30, 6e-8])            # beyond fp16 on both sides
    torch.testing.assert_close(lin(x), _by_pieces(lin, x), rtol=0, atol=0, equal_nan=True)
    x[0, :2] = 3.0
    assert torch.equal(lin(x), _by_pieces(lin, x))


def test_layouts_and_shapes():
    lin = _linear(136, 512)
    for dtype in (torch.float16, torch.bfloat16, torch.float32):
        base = torch.randn(4, 6, 1040, device="cuda").to(dtype)
        views = [base[..., 3:515], base[..., 8:520], base[:, :, ::2][..., :512], base[0, 0, :512].expand(3, 512),
                 base[0, :, :512], base[0, 0, :512], base[:0, :, :512]]
        for x in views:
            if dtype == torch.float16 and (x.data_ptr() % 16 or (x.dim() == 2 and x.stride(0) == 0) or x.stride(-1) != 1):
                continue                                           # fp16 rows are read where they are: refused before, too
            y = lin(x)
            assert y.shape == (*x.shape[:-1], 136) and torch.equal(y, _by_pieces(lin, x))
    with pytest.raises(RuntimeError):
        lin(torch.randn(4, 256, device="cuda"))
    with pytest.raises(RuntimeError):
        lin(torch.randn(4, 512))
    with pytest.raises(RuntimeError):
        lin(torch.randn(512, 4, device="cuda").half().t())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_mlp_takes_the_same_activations(dtype):
    from slimkernels_b200.torch import W2A8LlamaMLP
    mlp = W2A8LlamaMLP(_linear(768, 256), _linear(256, 384, seed=1))
    x = torch.randn(2, 9, 256, device="cuda").to(dtype)
    want = torch.ops.slimkernels.w2a8_mlp_forward(mlp.gate_up.plan()._h, mlp.down.plan()._h, x.reshape(-1, 256).half(), 256, False)
    assert torch.equal(mlp(x), want.reshape(2, 9, 256))


def test_plan_used_on_another_stream_and_dropped_there():
    """A plan made on one stream, used at once on another, and dropped while that stream still works: its memory is not
    handed out before the stream is done with it."""
    want, x = None, torch.randn(8, 4096, device="cuda").half()
    side = torch.cuda.Stream()
    for i in range(6):
        lin = _linear(4096, 4096, seed=3)
        with torch.cuda.stream(side):
            x.record_stream(side)
            side.wait_stream(torch.cuda.default_stream())
            ys = [lin(x) for _ in range(8)]
        del lin
        junk = torch.full((8 << 20,), 0xFF, dtype=torch.uint8, device="cuda")     # takes a freed block, if there is one
        side.synchronize()
        if want is None:
            want = ys[0].clone()
        assert all(torch.equal(y, want) for y in ys)
        del junk


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_narrow_slice_of_wide_rows_is_refused(dtype):
    from slimkernels_b200.torch import W2A8LlamaMLP
    mlp = W2A8LlamaMLP(_linear(768, 256), _linear(256, 384, seed=1))
    wide = torch.randn(5, 512, device="cuda").to(dtype)
    assert mlp(wide[:, :256]).shape == (5, 256)
    for x in (wide[:, :128], wide.view(1, 5, 512)[..., :248]):
        with pytest.raises(RuntimeError):
            mlp(x)
        with pytest.raises(RuntimeError):
            mlp.gate_up(x)


@pytest.mark.parametrize("M", [4, 200])
def test_plan_made_under_a_side_stream_sees_the_default_streams_weights(M):
    """A weight is still being produced on the default stream when its first use, under a side stream, makes the plan."""
    from slimkernels_b200.torch import W2A8Plan
    N, K, G = 1000, 2048, 128
    lin = _linear(N, K, G)
    x_q = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8)
    x_s = torch.full((M,), 0.01, device="cuda")
    want = W2A8Plan(lin.w_packed, lin.w_scale, group_size=G).gemm(x_q, x_s)
    codes, scales = torch.zeros_like(lin.w_packed), torch.zeros_like(lin.w_scale)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(100_000_000)
    codes.copy_(lin.w_packed)
    scales.copy_(lin.w_scale)
    with torch.cuda.stream(side):
        y = W2A8Plan(codes, scales, group_size=G).gemm(x_q, x_s)
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def _block_state(ptr):
    """What the caching allocator says of the block that holds an address."""
    for seg in torch.cuda.memory_snapshot():
        at = seg["address"]
        for block in seg["blocks"]:
            if at <= ptr < at + block["size"]:
                return block["state"]
            at += block["size"]


def _spin(stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)                             # about 0.2 s


@pytest.mark.parametrize("made_on", ["default", "third"])
@pytest.mark.parametrize("tiled", [False, True])
@pytest.mark.parametrize("M,G", [(8, 64), (200, 128)])
def test_a_dropped_plan_keeps_its_borrowed_weights_from_being_handed_out(M, G, tiled, made_on):
    """Launches on another stream than the weights' are still waiting when plan and weights are dropped: the allocator must not
    count their memory as free."""
    from slimkernels_b200.torch import W2A8Plan, repack_weight
    N, K = 1000, 2048
    lin = _linear(N, K, G)
    codes, scales = lin.w_packed.clone(), lin.w_scale.clone()
    if tiled:
        codes = repack_weight(codes)
    x_q = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8)
    x_s = torch.full((M,), 0.01, device="cuda")
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    # either the launches are on another stream than the plan was made on, or both are on another than the weights
    with torch.cuda.stream(side if made_on == "third" else torch.cuda.default_stream()):
        plan = W2A8Plan(codes, scales, N=N, K=K, group_size=G, tiled=tiled)
    want = plan.gemm(x_q, x_s)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        plan.gemm(x_q, x_s)                                        # its result's memory serves the call below (an allocation may wait)
    torch.cuda.synchronize()
    held = [t.data_ptr() for t in ((codes, scales) if tiled else (scales,))]
    _spin(side)
    with torch.cuda.stream(side):
        y = plan.gemm(x_q, x_s)
    del plan, codes, scales
    states = [_block_state(p) for p in held]
    assert not side.query()
    assert states == ["active_pending_free"] * len(held)
    side.synchronize()
    assert torch.equal(y, want)


def test_device_status_of_a_plan_whose_stream_has_not_got_to_it():
    """The status word lies in memory that held something else, and is cleared in stream order."""
    from slimkernels_b200 import capi
    from slimkernels_b200.torch import W2A8Plan
    N, K = 1024, 2048
    lin = _linear(N, K)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        nbytes = capi.load().sk_w2a8_plan_storage_bytes(0, N, K, 128, capi.SK_WEIGHT_ROWMAJOR)
        junk = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")
        side.synchronize()
        del junk
        _spin(side)
        plan = W2A8Plan(lin.w_packed, lin.w_scale)
        assert plan.device_status() == 0


def test_dropping_a_captured_plan_waits_for_the_graphs_that_use_it():
    lin = _linear(512, 1024)
    x = torch.randn(4, 1024, device="cuda").half()
    want = lin(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin(x)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    _spin(side)
    with torch.cuda.stream(side):
        graph.replay()
    assert not side.query()
    del lin
    assert side.query() and torch.equal(y, want)


def test_shapes_a_plan_refuses_need_no_storage():
    from slimkernels_b200 import capi
    from slimkernels_b200.torch import W2A8Plan
    size = capi.load().sk_w2a8_plan_storage_bytes
    assert size(0, 128, 192, 64, capi.SK_WEIGHT_ROWMAJOR) > 0
    for K, G in ((192, 96), (192, 48), (192, 128), (192, 0), (192, -64), (0, 64)):
        assert size(0, 128, K, G, capi.SK_WEIGHT_ROWMAJOR) == 0
    with pytest.raises(RuntimeError):
        W2A8Plan(torch.zeros(128, 48, dtype=torch.uint8, device="cuda"), torch.ones(2, 128, dtype=torch.float16, device="cuda"),
                 group_size=96)


def test_plan_is_refused_under_capture():
    lin = _linear(256, 256)
    x = torch.randn(2, 256, device="cuda").half()
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(graph):
            lin(x)                                                 # the plan would be made inside the capture
    torch.cuda.synchronize()
    y = lin(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        z = lin(x)                                                 # made before (on another stream): captured
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, z)


@pytest.mark.parametrize("G", [128, 256])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 40, 256), (1, 4096, 4096), (1, 512, 8192), (2, 4096, 4096), (3, 300, 2560), (8, 136, 1024),
                                   (1, 22016, 1024), (1, 57344, 512), (1, 12288, 768), (1, 4096, 8448)])
def test_activations_quantised_inside_the_gemm(M, N, K, G, dtype):
    """Few tokens: one kernel, the same bits as the quantiser followed by the GEMM (the last size is one over its limit)."""
    lin = _linear(N, K, G, out_dtype=dtype)
    for scale in (1.0, 0.0):
        x = (torch.randn(M, K, device="cuda") * scale).to(dtype)
        if M > 1:
            x[1] = 0
        assert torch.equal(lin(x), _by_pieces(lin, x))
    wide = torch.randn(M, K + 24, device="cuda").to(dtype)[:, 16:16 + K]
    if M > 1 and wide.data_ptr() % 16 == 0:
        assert torch.equal(lin(wide), _by_pieces(lin, wide))


def test_plan_used_at_once_after_it_is_made():
    """The GEMM behind a plan's copies in the stream reads them before it waits for the kernel in front of it."""
    x = torch.randn(1, 4096, device="cuda").half()
    w = [torch.randn(1024, 4096, device="cuda").half() for _ in range(2)]
    from slimkernels_b200.torch import W2A8Linear
    want = [W2A8Linear.from_float(v, 128)(x).clone() for v in w]
    torch.cuda.synchronize()
    got = [W2A8Linear.from_float(w[i % 2], 128)(x) for i in range(60)]      # storage of dropped plans comes round again
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2])
