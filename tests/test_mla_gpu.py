"""MLA kernels on the GPU: latent-cache attention at the 671B-class head shape (latent 512 + rope 64) against the fp32
PyTorch statement, and the tiny MLA + MoE model through the engine against the CPU oracle."""
import math

import pytest
import torch

from ferrite_b200.ops.torch_ops import TorchOps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(ext):
    from ferrite_b200.ops.cuda_ops import CudaOps
    return CudaOps(DEV)


@pytest.mark.parametrize("L,R,nq", [(512, 64, 16), (64, 64, 4)])
@pytest.mark.parametrize("nsplit", [1, 4])
def test_mla_prep_and_attention(ops, L, R, nq, nsplit):
    tops = TorchOps(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(L + nsplit)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device=DEV) * sc).to(torch.bfloat16)
    dn, kvb, nslots, ctx = 128 if L == 512 else 32, 64, 2, 200
    nb = (ctx + kvb - 1) // kvb + 1
    cache_a = r(nslots * nb, kvb, L + R)
    cache_b = cache_a.clone().float()
    bt = torch.arange(nslots * nb, device=DEV, dtype=torch.int32).view(nslots, nb)
    T = 6
    q, kva = r(T, nq * (dn + R)), r(T, L + R)
    norm_w, w_uk_t = r(L, sc=0.1), r(nq, L, dn, sc=0.05)
    hr = R // 2
    inv = (1e4 ** (-torch.arange(hr, dtype=torch.float64) / hr)).float().to(DEV)
    slot = torch.tensor([0, 0, 0, 1, 1, 1], device=DEV, dtype=torch.int32)
    pos = torch.tensor([150, 151, 152, 90, 91, 92], device=DEV, dtype=torch.int32)
    qa = ops.mla_prep(q, kva, norm_w, w_uk_t, inv, slot, pos, bt, cache_a, kvb, nq, dn, L, R, 1e-6)
    qb = tops.mla_prep(q, kva, norm_w, w_uk_t, inv, slot, pos, bt, cache_b, kvb, nq, dn, L, R, 1e-6)
    assert (qa.float() - qb.float()).abs().max().item() < 3e-2 * max(1.0, qb.abs().max().item())
    assert (cache_a.float() - cache_b).abs().max().item() < 3e-2
    kvlen = (pos + 1).contiguous()
    scale = 1.0 / math.sqrt(dn + R)
    oa = ops.mla_attention(qa, cache_a, slot, kvlen, bt, kvb, nq, L, R, scale, nsplit=nsplit)
    ob = tops.mla_attention(qa, cache_a, slot, kvlen, bt, kvb, nq, L, R, scale)
    assert (oa.float() - ob.float()).abs().max().item() < 2e-2


@pytest.mark.parametrize("L,R,nq", [(512, 64, 128), (512, 64, 3), (128, 64, 5), (64, 64, 4)])
@pytest.mark.parametrize("lens,rows,nsplit", [((1, 63, 64, 65), 1, 64), ((700, 129), 3, 4), ((200,), 40, 1)])
def test_mla_attention_of_segments(ops, L, R, nq, lens, rows, nsplit):
    """Segments on the tensor-core latent kernel against the CUDA-core kernel and the fp32 statement: contexts at the edges of its 64-key
    tiles, more splits than tiles, several rows per segment, heads that leave its M tiles ragged."""
    tops = TorchOps(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(L + nq + rows)
    kvb, nb, S = 64, 12, len(lens)
    cache = torch.randn(S * nb, kvb, L + R, generator=g, device=DEV).to(torch.bfloat16)
    bt = torch.randperm(S * nb, generator=g, device=DEV).to(torch.int32).view(S, nb)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    slot = i32([s for s in range(S) for _ in range(rows)])
    kvlen = i32([max(1, n - rows + 1 + r) for n in lens for r in range(rows)])
    q = torch.randn(S * rows, nq, L + R, generator=g, device=DEV).to(torch.bfloat16)
    scale = (L + R) ** -0.5
    segs = (i32(list(range(S))), i32([s * rows for s in range(S)]), i32([rows] * S), rows)
    got = ops.mla_attention(q, cache, slot, kvlen, bt, kvb, nq, L, R, scale, nsplit=nsplit, segs=segs).float()
    want = tops.mla_attention(q, cache, slot, kvlen, bt, kvb, nq, L, R, scale).float()
    plain = ops.mla_attention(q, cache, slot, kvlen, bt, kvb, nq, L, R, scale, nsplit=nsplit).float()
    # 32-bit scores and sums, weights of 16 bits (2^-17 relative): what is left is the rounding of the bf16 result, |o| <= 4.5 here
    for o in (got, plain):
        assert (o - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
    assert ops.status() == 0


@pytest.mark.parametrize("L,nq", [(512, 128), (128, 6), (64, 8)])
@pytest.mark.parametrize("ctx,nsplit", [(1, 2), (70, 2), (2000, 16), (4000, 32), (2000, 2)])
def test_mla_softmax_weights_keep_32_bits(ops, L, nq, ctx, nsplit):
    """The 32-bit records of the key splits, merged here in 64 bits, against the plain statement in 64 bits: off by a few 2^-24, as the kernel that
    multiplies 32-bit weights on the CUDA cores is, where weights of 16 bits and sums cut at every step are several times as far off."""
    R, kvb = 64, 64
    g = torch.Generator(device=DEV).manual_seed(L + ctx)
    nb = (ctx + kvb - 1) // kvb
    cache = torch.randn(nb, kvb, L + R, generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn(1, nq, L + R, generator=g, device=DEV).to(torch.bfloat16)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    bt, scale = torch.arange(nb, dtype=torch.int32, device=DEV).view(1, nb), (L + R) ** -0.5
    keys = cache.view(-1, L + R)[:ctx].double()
    want = torch.softmax(q[0].double() @ keys.t() * scale, -1) @ keys[:, :L]

    def off(run):
        o, ml = torch.empty(nq, nsplit, L, device=DEV), torch.empty(nq, nsplit, 2, device=DEV)
        run(torch.empty(1, nq, L, dtype=torch.bfloat16, device=DEV), o, ml)
        f = torch.exp2(ml[..., 0].double() - ml[..., 0].amax(1, keepdim=True).double())
        merged = (torch.where(f[..., None] > 0, o.double(), 0.0) * f[..., None]).sum(1) / (ml[..., 1].double() * f).sum(1)[:, None]
        return ((merged - want).norm() / want.norm()).item()

    mma = lambda exact: lambda out, o, ml: ops.C.latent_mma(out, o, ml, q, cache, i32(0), i32(0), i32(1), 1, i32(ctx), bt, kvb, 0, nsplit, scale,
                                                            ops.status_word, 0, 1, exact)
    three, two = off(mma(True)), off(mma(False))
    plain = off(lambda out, o, ml: ops.C.mla_attn(out, o, ml, q, cache, i32(0), i32(ctx), bt, kvb, nq, L, R, nsplit, scale))
    # four cut steps to a sum of a score's columns and six to one of a value's keys (2^-24 of it on average each), then rounded sums
    assert max(three, plain) <= 10 * 2 ** -24, (three, two, plain)
    assert ctx == 1 or two > 3 * three, (three, two, plain)
    assert ops.status() == 0


@pytest.mark.parametrize("L,nq", [(512, 128), (512, 16), (128, 5), (64, 70)])
@pytest.mark.parametrize("first", [30, 490, 2040, 4090])
def test_mla_row_has_its_bits_in_every_step(ops, L, nq, first):
    """The engine's split counts: a row alone, in a verified segment and beside other streams, at contexts where splits become longer (512 keys,
    beyond 4096) or more (2048)."""
    from ferrite_b200.engine.executor import Executor
    from types import SimpleNamespace
    splits = lambda n: Executor.attn_splits(SimpleNamespace(ecfg=SimpleNamespace(attn_splits=0)), n)
    R, kvb, rows, lens = 64, 64, 17, [first + 17, 60, 5000]
    g = torch.Generator(device=DEV).manual_seed(L + nq + first)
    nb = (max(lens) + kvb - 1) // kvb
    cache = torch.randn(3 * nb, kvb, L + R, generator=g, device=DEV).to(torch.bfloat16)
    bt = torch.randperm(3 * nb, generator=g, device=DEV).to(torch.int32).view(3, nb)
    q = torch.randn(rows + 2, nq, L + R, generator=g, device=DEV).to(torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def step(parts):                                         # (stream, first row, rows) of each segment
        at = [r for _, r, n in parts for r in range(r, r + n)]
        own = [first + 1 + r if s == 0 else lens[s] for s, a, n in parts for r in range(a, a + n)]
        slot, row0 = [s for s, _, n in parts for _ in range(n)], [sum(n for _, _, n in parts[:i]) for i in range(len(parts))]
        segs = (i32([s for s, _, _ in parts]), i32(row0), i32([n for _, _, n in parts]), max(n for _, _, n in parts))
        return ops.mla_attention(q[at], cache, i32(slot), i32(own), bt, kvb, nq, L, R, (L + R) ** -0.5, nsplit=splits(max(own)), segs=segs, picked=True)

    whole = step([(0, 0, rows)])
    for r in range(rows):
        assert torch.equal(step([(0, r, 1)])[0], whole[r]), r
    beside = step([(1, rows, 1), (0, 0, rows), (2, rows + 1, 1)])
    assert torch.equal(beside[1:1 + rows], whole)
    assert torch.equal(step([(1, rows, 1)])[0], beside[0]) and torch.equal(step([(2, rows + 1, 1)])[0], beside[-1])
    assert ops.status() == 0


@pytest.mark.parametrize("T", [1, 6, 8, 19, 300])
@pytest.mark.parametrize("nh,N,K", [(16, 512, 128), (16, 128, 512), (4, 64, 32), (3, 40, 64)])
def test_head_linear_row_kernel_and_batched_gemm(ops, T, nh, N, K):
    """Per-head linears of the latent attention: <= 8 rows (and shapes the tensor-core tiles do not take) run the row
    kernel, more rows the batched tcgen05 GEMM; x is a strided view (the query's nope part), y a strided slice."""
    tops = TorchOps(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(T * 131 + N)
    pad = 64
    xfull = (torch.randn(T, nh, K + pad, generator=g, device=DEV)).to(torch.bfloat16)
    W = (torch.randn(nh, N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    x = xfull[:, :, :K]
    want = tops.head_linear(x, W)
    got = ops.head_linear(x, W)
    err = (got.float() - want).abs().max().item()
    assert err < 2e-2 * max(1.0, want.abs().max().item()), err
    yfull = torch.full((T, nh, N + 24), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.head_linear(x, W, out=yfull[:, :, :N])
    assert torch.equal(yfull[:, :, :N], got) and bool((yfull[:, :, N:] == 7.0).all())
    assert ops.status() == 0


@pytest.mark.parametrize("nh,N,K", [(128, 512, 128), (2, 16, 32), (3, 1, 96), (5, 100, 160), (128, 136, 256), (7, 129, 512), (2, 64, 544), (2, 64, 40)])
def test_head_linear_rows_and_ragged_widths(ops, nh, N, K):
    """Outputs that fill no tile of 16, columns that fill no slab of 128 (and too many, or no multiple of 32: the other row kernel): against 64 bits, within
    the result's rounding to bf16 and 32-bit sums; a row alone has the bits that it has among others."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    W = (torch.randn(nh, N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    x = torch.randn(8, nh, K, generator=g, device=DEV).to(torch.bfloat16)
    want = torch.einsum("thk,hnk->thn", x.double(), W.double())
    mag = torch.einsum("thk,hnk->thn", x.double().abs(), W.double().abs())
    for T in (1, 2, 3, 5, 8):
        y = torch.full((T, nh, N + 3), 7.0, device=DEV, dtype=torch.bfloat16)
        ops.C.head_linear(y[:, :, :N], x[:T], W)
        assert bool(((y[:, :, :N].double() - want[:T]).abs() <= want[:T].abs() * 2 ** -8 + mag[:T] * K * 2 ** -24).all())
        assert bool((y[:, :, N:] == 7).all())
        if T > 1:
            assert torch.equal(y[:1], first)
        first = y[:1].clone()
    assert ops.status() == 0


@pytest.mark.parametrize("nq,L,R,dn,dv", [(16, 512, 64, 128, 128), (4, 64, 64, 32, 32)])
def test_mla_expanded_prefill_matches_absorbed(ops, nq, L, R, dn, dv):
    """Prompt segments through the expanded form (kv_b GEMM over the context's latent rows, padded per-head K / V, tcgen05
    flash kernel) against the absorbed-form fp32 statement on the same latent cache: two segments, one of them continuing
    a context that is already in the cache."""
    tops = TorchOps(DEV, torch.float32)
    g = torch.Generator(device=DEV).manual_seed(nq + L)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device=DEV) * sc).to(torch.bfloat16)
    kvb, nslots, nb = 64, 2, 4
    cache = torch.zeros(nslots * nb, kvb, L + R, dtype=torch.bfloat16, device=DEV)
    bt = torch.randperm(nslots * nb, generator=g, device=DEV).to(torch.int32).view(nslots, nb)
    norm_w, w_uk_t, w_uv = r(L, sc=0.1), r(nq, L, dn, sc=dn ** -0.5), r(nq, dv, L, sc=L ** -0.5)
    kv_b = torch.cat([w_uk_t.transpose(1, 2), w_uv], 1).reshape(nq * (dn + dv), L).contiguous()
    hr = R // 2
    inv = (1e4 ** (-torch.arange(hr, dtype=torch.float64) / hr)).float().to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    # 70 earlier rows of slot 1
    ops.mla_prep(r(70, nq * (dn + R)), r(70, L + R), norm_w, w_uk_t, inv, i32([1] * 70), i32(list(range(70))), bt, cache, kvb,
                 nq, dn, L, R, 1e-6)
    segs = [(0, 0, 50), (1, 70, 90)]
    T = 140
    slot = i32([0] * 50 + [1] * 90)
    pos = i32(list(range(50)) + list(range(70, 160)))
    q, kva = r(T, nq * (dn + R)), r(T, L + R)
    qabs = ops.mla_prep(q, kva, norm_w, w_uk_t, inv, slot, pos, bt, cache, kvb, nq, dn, L, R, 1e-6)
    scale = 1.0 / math.sqrt(dn + R)
    ol = tops.mla_attention(qabs, cache, slot, (pos + 1).contiguous(), bt, kvb, nq, L, R, scale)
    want = tops.mla_out(ol, w_uv).float()
    got = ops.mla_attention_prefill(q, qabs, cache, kv_b, segs, i32([0, 50]), i32([50, 90]), i32([0, 70]), bt, kvb, nq, dn, dv,
                                    L, R).float()
    assert got.shape == want.shape
    err = (got - want).abs().max().item()
    assert err < 3e-2 * max(1.0, want.abs().max().item()), err
    assert ops.status() == 0


def test_mla_engine_prompt_chunks_gpu(ext):
    """The tiny MLA + MoE model with a 70-row prompt chunk (expanded tensor-core path), a 30-row chunk (absorbed rows) and
    decode steps against the CPU oracle."""
    from ferrite_b200.config import EngineConfig, tiny_mla
    from ferrite_b200.engine.engine import Engine
    from ferrite_b200.engine.executor import Segment
    from ferrite_b200.models.weights import init_weights
    cfg = tiny_mla()
    w = init_weights(cfg, seed=0)
    p = torch.randint(0, cfg.vocab, (110,), generator=torch.Generator().manual_seed(2)).tolist()
    ref = Engine(cfg, w, EngineConfig(n_slots=1, max_ctx=128), device="cpu")
    want, _, _ = ref.forward([Segment(0, 0, p, "all")])
    eng = Engine(cfg, w, EngineConfig(n_slots=1, max_ctx=128), device=DEV)
    a, _, _ = eng.forward([Segment(0, 0, p[:70], "all")])
    b, _, _ = eng.forward([Segment(0, 70, p[70:100], "all")])
    tail = [eng.forward([Segment(0, 100 + i, [p[100 + i]], "last")])[0].clone() for i in range(10)]
    got = torch.cat([a.clone(), b.clone()] + tail).float().cpu()
    kl = torch.nn.functional.kl_div(torch.log_softmax(got, -1), torch.log_softmax(want, -1), log_target=True,
                                    reduction="batchmean").item()
    assert kl < 2e-2, kl
    eng.check()


def test_mla_engine_gpu(ext):
    from ferrite_b200.config import EngineConfig, tiny_mla
    from ferrite_b200.engine.engine import Engine
    from ferrite_b200.engine.executor import Segment
    from ferrite_b200.models.weights import init_weights
    cfg = tiny_mla()
    w = init_weights(cfg, seed=0)
    p = torch.randint(0, cfg.vocab, (40,), generator=torch.Generator().manual_seed(1)).tolist()
    ref = Engine(cfg, w, EngineConfig(n_slots=1, max_ctx=128), device="cpu")
    want, _, _ = ref.forward([Segment(0, 0, p, "all")])
    eng = Engine(cfg, w, EngineConfig(n_slots=1, max_ctx=128), device=DEV)
    got, _, _ = eng.forward([Segment(0, 0, p[:30], "all")])
    tail = [eng.forward([Segment(0, 30 + i, [p[30 + i]], "last")])[0].clone() for i in range(10)]
    got = torch.cat([got] + tail).float().cpu()
    kl = torch.nn.functional.kl_div(torch.log_softmax(got, -1), torch.log_softmax(want, -1), log_target=True,
                                    reduction="batchmean").item()
    assert kl < 2e-2, kl


@pytest.mark.parametrize("nq,R", [(70, 64), (128, 40), (5, 2)])
def test_mla_prep_of_many_rows(ops, nq, R):
    """Rows in one call (a CTA takes up to 64 heads of many rows) have the bits of the same rows in calls of few (16 heads), in the queries' rope parts and
    in the cache, and are what 64 bits give but for the angle's and the result's roundings."""
    L, dn, kvb, rows = 64, 24, 64, 600
    g = torch.Generator(device=DEV).manual_seed(nq)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)
    q, kva, norm_w = r(rows, nq * (dn + R)), r(rows, L + R), r(L)
    inv = (1e4 ** (-torch.arange(R // 2, dtype=torch.float64) / (R // 2))).float().to(DEV)
    pos, slot = torch.arange(rows, device=DEV, dtype=torch.int32), torch.zeros(rows, device=DEV, dtype=torch.int32)
    bt = torch.arange((rows + kvb - 1) // kvb, device=DEV, dtype=torch.int32).view(1, -1)
    caches = [torch.zeros(bt.numel(), kvb, L + R, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    call = lambda a, b, cache: ops.mla_prep(q[a:b], kva[a:b], norm_w, None, inv, slot[a:b], pos[a:b], bt, cache, kvb, nq, dn, L, R, 1e-6, absorb=False)[:, :, L:]
    got = call(0, rows, caches[0])
    assert torch.equal(got, torch.cat([call(a, min(a + 90, rows), caches[1]) for a in range(0, rows, 90)]))
    assert torch.equal(caches[0], caches[1])
    turn = torch.exp(1j * pos.double()[:, None, None] * inv.double())
    v = q.double().view(rows, nq, dn + R)[:, :, dn:]
    want = torch.complex(v[..., :R // 2], v[..., R // 2:]) * turn
    want = torch.cat([want.real, want.imag], -1)
    # the angle is rounded once (2^-24 of up to 600), a result to bf16 (2^-9 of it), products and sums to 32 bits
    size = torch.cat([torch.complex(v[..., :R // 2], v[..., R // 2:]).abs()] * 2, -1)
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + (600 * 2 ** -23 + 2 ** -20) * size).all())
    assert ops.status() == 0
