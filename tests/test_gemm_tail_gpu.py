"""Prompt-sized GEMMs whose tile width follows the shape and whose last tiles may be cut along K, against 64-bit sums."""
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


def plain(ops, x, w, mode, res=None):
    """The same call without scratch: no pieces."""
    N = w.shape[0] // 2 if mode & 1 else w.shape[0]
    y = torch.empty(x.shape[0], (N + 7) // 8 * 8, dtype=torch.float32 if mode & 2 else torch.bfloat16, device=DEV)[:, :N]
    ops.C.gemm(y, x, w, res, mode, 1, None, None, ops.status_word)
    return y


# widths that end in every part of a tile (one column, ragged 8s, multiples of 32 and 64), one tile, several waves; pieces: K deep enough for two
# to four of them, also where the last piece is shorter (K = 4104: 65 k blocks)
@pytest.mark.parametrize("M,N,K,pieces", [(65, 1, 64, False), (128, 100, 72, False), (129, 264, 1000, False), (1531, 5120, 264, False), (2048, 2500, 512, False),
                                          (70, 1000, 8192, True), (140, 2048, 4104, True), (300, 1111, 8192, True), (1111, 5120, 8192, True)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_widths_and_pieces(ops, M, N, K, pieces, swiglu):
    x, w = rnd(M, K, seed=1), rnd((2 if swiglu else 1) * N, K, seed=2, scale=K ** -0.5)
    want = x.double() @ w.double().t()
    if swiglu:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    # 32-bit sums of products exact in 32 bits, outputs of size one; the oracle's size bounds what the activation passes on
    bound = 2 ** -14 * max(1.0, want.abs().max().item())
    y = ops.linear(x, w, swiglu=swiglu, out_f32=True)
    assert (y.double() - want).abs().max().item() <= bound
    assert torch.equal(y, ops.linear(x, w, swiglu=swiglu, out_f32=True))            # whichever piece comes last
    whole = plain(ops, x, w, 3 if swiglu else 2)
    assert (whole.double() - want).abs().max().item() <= bound
    if pieces and not swiglu:
        assert not torch.equal(y, whole)
    if not swiglu:
        res = rnd(M, N + 8 - N % 8, seed=3)[:, :N]                                  # the residual shares the output's leading dimension
        y16 = torch.empty(M, N + 8 - N % 8, dtype=torch.bfloat16, device=DEV)[:, :N]
        got = ops.linear(x, w, res=res, out=y16)
        assert torch.equal(got, (y + res.float()).to(torch.bfloat16))
        assert torch.equal(ops.linear(x, w, out_f32=True, act="relu2"), y.clamp_min(0).square())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):                                                   # every stream has scratch: the same bits
        assert torch.equal(ops.linear(x, w, swiglu=swiglu, out_f32=True), y)
    torch.cuda.synchronize()
    assert ops.status() == 0 and all(int(c.abs().sum()) == 0 for _, c in ops._tails.values())


@pytest.mark.parametrize("M", [33, 40, 64])
@pytest.mark.parametrize("N,K,width", [(1, 64, 8), (264, 1000, 264), (2500, 4104, 2504), (1111, 4104, 1111), (2048, 512, 2051)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_33_to_64_rows_on_either_side(ops, M, N, K, width, swiglu):
    """Rows that leave most of a 128-row tile empty, and (outputs `width` columns apart that are no multiple of 8) rows on the narrow side of the
    product with K splits; rows of another width next to them stay as they are."""
    x, w = rnd(M, K, seed=1), rnd((2 if swiglu else 1) * N, K, seed=2, scale=K ** -0.5)
    want = x.double() @ w.double().t()
    if swiglu:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    buf = torch.full((M, width + 8), 7.0, dtype=torch.float32, device=DEV)
    flat = buf.view(-1)[:M * width].view(M, width)
    y = ops.linear(x, w, swiglu=swiglu, out_f32=True, out=flat[:, :N])
    bound = 2 ** -14 * max(1.0, want.abs().max().item())                             # as above
    assert (y.double() - want).abs().max().item() <= bound
    assert bool((flat[:, N:] == 7).all()) and bool((buf.view(-1)[M * width:] == 7).all())
    if not swiglu:
        res = rnd(M, width, seed=3)[:, :N]
        got = ops.linear(x, w, res=res, out=torch.empty(M, width, dtype=torch.bfloat16, device=DEV)[:, :N])
        assert torch.equal(got, (y + res.float()).to(torch.bfloat16))
    assert ops.status() == 0


@pytest.mark.parametrize("M,N,K", [(33, 8224, 5120), (64, 5120, 2048), (64, 2048, 4096), (48, 24, 4096), (40, 640, 8192), (64, 1111, 1032), (50, 17408, 2048),
                                   (64, 20000, 1024), (36, 256, 16384)])
def test_sums_of_33_to_64_rows_are_as_exact_as_in_k_splits(ops, M, N, K):
    """Rows in tiles of 128 against the same rows as the narrow side of the product, K cut into splits: no further off 64 bits (5 % for the sums' chance;
    chains as long as K, or as a piece of it, are 1.5 to 2.5 times as far off)."""
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    want = x.double() @ w.double().t()
    split = ops._split_k(M, N, K)
    y = torch.empty(M, (N + 7) // 8 * 8, device=DEV)[:, :N]
    ws = (torch.empty(ops.C.gemm_workspace_bytes(M, N, split) // 4, device=DEV), torch.zeros(4096, dtype=torch.int32, device=DEV)) if split > 1 else (None, None)
    ops.C.gemm(y, x, w, None, 2, split, *ws, ops.status_word)
    off = lambda t: ((t.double() - want).norm() / want.norm()).item()
    assert off(ops.linear(x, w, out_f32=True)) <= 1.05 * off(y)
    if split <= 8:                                                                   # without scratch: as many sums as there is room for
        bare = torch.empty(M, (N + 7) // 8 * 8, device=DEV)[:, :N]
        ops.C.gemm(bare, x, w, None, 2, -1, None, None, ops.status_word)
        assert off(bare) <= 1.05 * off(y)
    assert ops.status() == 0


def test_scratch_that_is_too_small_takes_no_pieces(ops):
    """Scratch of any size may come with a call: pieces are taken where they fit it, and nothing past its end is written."""
    M, N, K = 300, 1111, 8192
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    whole, pieces = plain(ops, x, w, 2), ops.linear(x, w, out_f32=True)
    assert not torch.equal(whole, pieces)
    room, ctrs = ops.C.gemm_workspace_bytes(M, N, 1) // 4, ops.C.gemm_counters(M, N, 1)
    for n_ws, n_ctr, want in [(room, ctrs, pieces), (1024, ctrs, whole), (room, 32, whole), (1024, 1, whole)]:
        ws, cnt = torch.full((n_ws + 4096,), 7.0, device=DEV), torch.zeros(n_ctr + 4096, dtype=torch.int32, device=DEV)
        y = torch.empty(M, 1112, device=DEV)[:, :N]
        ops.C.gemm(y, x, w, None, 2, 1, ws[:n_ws], cnt[:n_ctr], ops.status_word)
        assert torch.equal(y, want) and bool((ws[n_ws:] == 7).all()) and int(cnt.abs().sum()) == 0
    with pytest.raises(RuntimeError):                                                # the K splits of few rows need theirs
        ops.C.gemm(torch.empty(48, N, device=DEV), x[:48], w, None, 2, 8, torch.empty(16, device=DEV), torch.zeros(64, dtype=torch.int32, device=DEV),
                   ops.status_word)
    assert ops.status() == 0


def test_pieces_on_many_streams_and_under_capture(ext):
    """A call's bits do not depend on the stream, on which stream came first, or on being captured; a handful of streams keep scratch."""
    from ferrite_b200.ops.cuda_ops import TAIL_STREAMS, CudaOps
    ops = CudaOps(DEV)
    M, N, K = 140, 2048, 4104
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    whole = plain(ops, x, w, 2)
    torch.cuda.synchronize()
    got = []
    for s in [torch.cuda.Stream() for _ in range(TAIL_STREAMS + 3)]:                # the main stream comes last
        with torch.cuda.stream(s):
            got += [ops.linear(x, w, out_f32=True) for _ in range(3)]
    torch.cuda.synchronize()
    y = ops.linear(x, w, out_f32=True)
    assert not torch.equal(y, whole) and all(torch.equal(g, y) for g in got) and len(ops._tails) <= TAIL_STREAMS
    held, graph = dict(ops._tails), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c = ops.linear(x, w, out_f32=True)
    for _ in range(3):
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(c, y)
    assert ops._tails.keys() == held.keys() and ops.status() == 0


@pytest.mark.parametrize("M", [33, 64])
def test_captured_products_of_up_to_64_rows_share_their_scratch(ext, M, monkeypatch):
    """What a captured step holds: outputs and kernels, no scratch and no fill of a product's own; the bits of the eager call."""
    from ferrite_b200.ops.cuda_ops import CudaOps
    ops, N, K = CudaOps(DEV), 1000, 8192
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    wq, ws = ops.quantize_weight_fp8(w)
    want = ops.linear(x, w, out_f32=True), ops.linear_fp8(x, wq, ws)
    torch.cuda.synchronize()
    graph, made = torch.cuda.CUDAGraph(), []
    zeros = torch.zeros
    with torch.cuda.graph(graph):
        monkeypatch.setattr(torch, "zeros", lambda *a, **k: made.append(a) or zeros(*a, **k))
        got = [(ops.linear(x, w, out_f32=True), ops.linear_fp8(x, wq, ws)) for _ in range(4)]
        monkeypatch.undo()
    assert not made
    for _ in range(2):
        for pair in got:
            for t in pair:
                t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for pair in got for a, b in zip(pair, want))
    assert ops.status() == 0 and int(ops._counters.count_nonzero()) == 0


@pytest.mark.parametrize("N", [24, 100])
def test_output_on_no_16_bytes(ops, N):
    M, K = 130, 256
    x, w, res = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(M, 104, seed=3)[:, :N]
    want = ops.linear(x, w, res=res, out=torch.empty(M, 104, dtype=torch.bfloat16, device=DEV)[:, :N])
    out = torch.zeros(M * 104 + 1, dtype=torch.bfloat16, device=DEV)[1:].view(M, 104)
    assert torch.equal(ops.linear(x, w, res=res, out=out[:, :N]), want) and int(out[:, N:].count_nonzero()) == 0


@pytest.mark.parametrize("M,N,K", [(129, 264, 1040), (140, 2048, 8208)])
def test_scaled_fp8(ops, M, N, K):
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    wq, ws = ops.quantize_weight_fp8(w)
    xq, xs = torch.empty(M, K, dtype=torch.uint8, device=DEV), torch.empty(M, device=DEV)
    ops.C.quant_fp8(xq, xs, x, None, 1e-6)
    f8 = lambda q: q.view(torch.float8_e4m3fn).double()
    want = f8(xq) @ f8(wq).t() * xs.double()[:, None] * ws.double()
    # tensor cores add e4m3 products in 32 bits or a little less; then one rounding to bf16
    got = ops.linear_fp8(x, wq, ws).double()
    assert ((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -9).all()


@pytest.mark.parametrize("M,N,K", [(33, 264, 1040), (48, 5120, 2048), (64, 2048, 8208), (50, 17408, 1024)])
def test_scaled_fp8_of_33_to_64_rows(ops, M, N, K):
    """e4m3 rows in tiles of 128, and as the narrow side of the product, against 64 bits."""
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    wq, ws = ops.quantize_weight_fp8(w)
    xq, xs = torch.empty(M, K, dtype=torch.uint8, device=DEV), torch.empty(M, device=DEV)
    ops.C.quant_fp8(xq, xs, x, None, 1e-6)
    f8 = lambda q: q.view(torch.float8_e4m3fn).double()
    want = f8(xq) @ f8(wq).t() * xs.double()[:, None] * ws.double()
    narrow, split = torch.empty(M, N, dtype=torch.bfloat16, device=DEV), ops._split_k(M, N, K // 2)
    ops.C.gemm_fp8(narrow, xq, wq, xs, ws, None, 0, split, *ops._gemm_scratch(M, N, split), ops.status_word)
    for got in (ops.linear_fp8(x, wq, ws), narrow):
        # tensor cores add e4m3 products in 32 bits or a little less; then one rounding to bf16
        assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -9).all()
    assert ops.status() == 0
