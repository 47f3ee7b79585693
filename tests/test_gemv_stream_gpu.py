"""Few-row products that stream bf16 or NVFP4 weights through a TMA ring (`gemv_stream`) against 32-bit math on the same values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(ext):
    from ferrite_b200.ops.cuda_ops import CudaOps
    return CudaOps(DEV)


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def reference(x, w, norm_w, eps, swiglu, rounded=0.0):
    """The product in 64 bits, and how far off each output may be. 32-bit sums: the tensor cores cut up to 2^-23 of a sum at each of K / 16 steps.
    Under a norm x (1 + w) is rounded to bf16 (`rounded`, of its size) and times 1 / rms (2^-20); then silu's exponential (2^-18)."""
    x, w = x.double(), w.double()
    off = (w.shape[1] / 16 + 1) * 2.0 ** -23 + rounded
    if norm_w is not None:
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (1 + norm_w.double())
        off += 2.0 ** -20
    y, e = x @ w.t(), off * (x.abs() @ w.abs().t())
    if not swiglu:
        return y, e
    half = y.shape[1] // 2
    gate, up = y[:, :half], y[:, half:]
    act = torch.nn.functional.silu(gate)
    return act * up, 1.1 * e[:, :half] * (up.abs() + e[:, half:]) + act.abs() * e[:, half:] + 2.0 ** -18 * (act * up).abs()


def rounding(M, norm):
    """Of x (1 + w), relative: none without a norm. bf16 holds 8 bits, so a value is off by up to 2^-8; up to four rows bring what is rounded off in
    columns of their own, which are rounded in turn."""
    return 0.0 if not norm else 2.0 ** -16 if M <= 4 else 2.0 ** -8


# rows at the edges of the 8-token tiles; outputs and K around tiles (128, 64 for SwiGLU), units (64 / 256) and runs; K of one unit; a tile
# shared by many runs and runs over many tiles
@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 9, 17, 32])
@pytest.mark.parametrize("N,K", [(1, 8), (129, 64), (127, 72), (640, 5000), (4112, 1024), (20000, 264)])
@pytest.mark.parametrize("norm,swiglu", [(False, False), (True, False), (True, True)])
def test_bf16_weights(ops, M, N, K, norm, swiglu):
    x, w = rnd(M, K, seed=M), rnd((2 if swiglu else 1) * N, K, seed=2, scale=K ** -0.5)
    nw = rnd(K, seed=3, scale=0.1) if norm else None
    want, off = reference(x, w, nw, 1e-6, swiglu, rounding(M, norm))
    y = ops._stream(x, w, None, 1.0, None, nw, 1e-6, None, 1 if swiglu else 0, N, True)
    assert ((y.double() - want).abs() <= off).all()
    if not swiglu:
        res = rnd(M, N, seed=4)
        got = ops._stream(x, w, None, 1.0, None, nw, 1e-6, res, 0, N, False)
        assert torch.equal(got, (y + res.float()).to(torch.bfloat16))
        relu2 = ops._stream(x, w, None, 1.0, None, nw, 1e-6, None, 2, N, True)
        assert torch.equal(relu2, y.clamp_min(0).square())
    assert torch.equal(y, ops._stream(x, w, None, 1.0, None, nw, 1e-6, None, 1 if swiglu else 0, N, True))
    assert ops.status() == 0 and int(ops._counters.abs().sum()) == 0


@pytest.mark.parametrize("M", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("N,K,swiglu", [(1, 256, False), (130, 512, False), (8224, 1280, False), (128, 256, True), (1536, 2048, True)])
@pytest.mark.parametrize("norm", [False, True])
def test_nvfp4_weights(ops, M, N, K, swiglu, norm):
    """Every code and scale: the unpacked weights are exact, so only x (1 + w) is rounded (not at all up to four rows)."""
    from ferrite_b200.formats import nvfp4
    rows = (2 if swiglu else 1) * N
    g = torch.Generator(device=DEV).manual_seed(K + N)
    packed = torch.randint(0, 256, (rows, K // 2), generator=g, device=DEV, dtype=torch.uint8)
    scales = torch.randint(0, 127, (rows, K // 16), generator=g, device=DEV, dtype=torch.uint8)       # 0 .. 448, subnormal ones among them
    t = nvfp4.NVFP4Tensor(packed, scales.view(torch.float8_e4m3fn), 2.0 ** -10, rows, K)
    w = t.dequantize(torch.float64)
    alpha = torch.rand(rows, generator=g, device=DEV) + 0.5
    x, nw = rnd(M, K, seed=M), rnd(K, seed=3, scale=0.1) if norm else None
    tiles = nvfp4.tile_scales_mma(t.scales).contiguous()
    for ra in (None, alpha):
        wr = w if ra is None else w / t.global_scale * ra.double()[:, None] * 2.0 ** -10
        want, off = reference(x, wr, nw, 1e-6, swiglu, rounding(M, norm))
        y = ops._stream(x, packed, tiles, t.global_scale, None if ra is None else ra * 2.0 ** -10, nw, 1e-6, None, 1 if swiglu else 0, N, True)
        assert ((y.double() - want).abs() <= off + 1e-30).all()
        assert torch.equal(y, ops._stream(x, packed, tiles, t.global_scale, None if ra is None else ra * 2.0 ** -10, nw, 1e-6, None, 1 if swiglu else 0, N, True))
    assert ops.status() == 0 and int(ops._counters.abs().sum()) == 0


@pytest.mark.parametrize("M", [1, 8])
def test_nan_scales_of_4_bit_weights(ops, M):
    """e4m3's NaN (0x7f) as a block scale makes its row's outputs NaN and no other; the largest scale (0x7e, 448) stays what it is."""
    from ferrite_b200.formats import nvfp4
    N, K = 130, 512
    g = torch.Generator(device=DEV).manual_seed(M)
    packed = torch.randint(0, 256, (N, K // 2), generator=g, device=DEV, dtype=torch.uint8)
    scales = torch.full((N, K // 16), 0x7e, device=DEV, dtype=torch.uint8)
    bad = [0, 15, 77, 129]
    for i, r in enumerate(bad):
        scales[r, i * 9] = 0x7f
    t = nvfp4.NVFP4Tensor(packed, scales.view(torch.float8_e4m3fn), 1.0, N, K)
    x = rnd(M, K, seed=M)
    y = ops._stream(x, packed, nvfp4.tile_scales_mma(t.scales).contiguous(), 1.0, None, None, 1e-6, None, 0, N, True)
    nan = torch.zeros(N, dtype=torch.bool, device=DEV)
    nan[bad] = True
    assert torch.equal(y.isnan(), nan.expand(M, N))
    w = t.dequantize(torch.float64)[~nan]
    assert ((y[:, ~nan].double() - x.double() @ w.t()).abs() <= 2 ** -19 * (x.double().abs() @ w.abs().t())).all()


def test_shapes_left_to_other_kernels(ops):
    """Refused before anything is launched: rows that are no multiple of 16 bytes, 4-bit rows that are no multiple of a unit."""
    assert ops._stream(rnd(2, 16), rnd(64, 16)[:, :16], None, 1.0, None, None, 1e-6, None, 0, 64, True) is not None
    assert ops._stream(rnd(2, 12), rnd(64, 12), None, 1.0, None, None, 1e-6, None, 0, 64, True) is None
    z = torch.zeros(64, 64, dtype=torch.uint8, device=DEV)
    assert ops._stream(rnd(2, 128), z, z, 1.0, None, None, 1e-6, None, 0, 64, True) is None
    n0 = ops.launches
    assert ops._stream(rnd(9, 12), rnd(64, 12), None, 1.0, None, rnd(12), 1e-6, None, 0, 64, True) is None            # nor the norm of more rows
    odd = rnd(64 * 64 + 1)[1:].view(64, 64)                                                                          # weights on no 16 bytes
    assert ops._stream(rnd(9, 64), odd, None, 1.0, None, rnd(64), 1e-6, None, 0, 64, True) is None
    assert ops._stream(rnd(1, 64).expand(3, 64), rnd(64, 64), None, 1.0, None, None, 1e-6, None, 0, 64, True) is None   # one row three times
    assert ops.launches == n0
    with pytest.raises(RuntimeError):
        ops.C.gemv_stream(torch.empty(2, 64, device=DEV), rnd(2, 12), rnd(64, 12), None, 1.0, None, None, None, 1e-6, 0, ops._workspace(1),
                          ops._counters, ops.status_word)


def test_records_follow_the_grid_and_not_the_outputs(ops):
    """As many rows against as wide a head as there is: what the runs leave behind fits, and the call is not left to another kernel."""
    M, N, K = 32, 262144, 512
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    y = ops._stream(x, w, None, 1.0, None, None, 1e-6, None, 0, N, True)
    assert y is not None
    for n in range(0, N, 65536):
        want = x.double() @ w[n:n + 65536].double().t()
        # 32-bit sums of products exact in 32 bits
        assert (y[:, n:n + 65536].double() - want).abs().max().item() <= 2 ** -14 * max(1.0, want.abs().max().item())
    assert ops.status() == 0 and int(ops._counters.abs().sum()) == 0
