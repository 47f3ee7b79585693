"""Determinism check: every kernel whose result passes through a cross-CTA (or cross-GPU) hand-off is run repeatedly on
the same inputs and must return the same bits every time.

    python -m ferrite_b200.utils.detcheck [--reps 20]

Each case is named after the entry point that it runs. Hand-offs covered: split-K partial sums of the tcgen05 GEMM (few-row "swapped" form), its
last prompt tiles cut along K, the runs of the TMA-ring row kernel (bf16 and 4-bit weights) and split K of the register-staged one, stream-K slots
of the NVFP4 few-row kernel, split-KV partials + merge of decode attention (grouped queries, rows of a verified segment, latents), the chunked Gated
DeltaNet scan (state handed from chunk to chunk), MoE pair GEMVs + fixed-order combine, prompt experts from their codes, the EXL3 cross-warp sum.
Arrival order differs from run to run; the sums are taken in a fixed order, which is what this checks. Prints one JSON line; exit code 1 if any case
changed a bit. The role of the reference's `exl3-detcheck` (`crates/fe-exl3/src/bin/exl3-detcheck.rs`),
widened to every family.
"""
from __future__ import annotations

import argparse
import copy
import json
import sys

import torch


def cases(ops, dev):
    from ..formats.exl3 import Exl3Tensor
    from ..ops.exl3_linear import Exl3Linear
    from ..ops.qweight import ExpertsFP4, quantize_weight
    from ..parallel.ep import ExpertParallel
    g = torch.Generator(device=dev).manual_seed(5)
    rnd = lambda *s, scale=1.0, dtype=torch.bfloat16: (torch.randn(*s, generator=g, device=dev) * scale).to(dtype)
    i32 = lambda *v: torch.tensor(list(v), device=dev, dtype=torch.int32)
    out = {}
    x1, x4, x48 = rnd(1, 5120), rnd(4, 5120), rnd(48, 5120)
    w = rnd(5120, 5120, scale=0.03)
    small, x4s = rnd(1000, 4096, scale=0.03), rnd(4, 4096)
    wk, xk = rnd(2048, 17408, scale=0.02), rnd(48, 17408)
    wp, xp = rnd(2048, 4104, scale=0.02), rnd(140, 4104)
    out["gemv: 1 row"] = lambda: ops.linear(x1, w)
    out["gemv_mma: 4 rows (split k)"] = lambda: ops.linear(x4s, small)
    out["gemv_stream: 4 rows (runs that share tiles)"] = lambda: ops.linear(x4, w)
    out["gemm: 48 rows, K 17408 (split k)"] = lambda: ops.linear(xk, wk)
    out["gemm: 48 rows, fp32 out (split k)"] = lambda: ops.linear(x48, w, out_f32=True)
    out["gemm: 140 rows (last tiles cut along k)"] = lambda: ops.linear(xp, wp)
    q = quantize_weight(w)
    act, rows = copy.copy(ops), copy.copy(ops)
    act.fp4_act, rows.fp4_rows = True, True
    out["gemv_nvfp4_tc: 1 row (stream-k slots)"] = lambda: act.linear(x1, q)
    out["gemv_nvfp4_tc: 4 rows"] = lambda: act.linear(x4, q)
    out["gemv_stream: 4 rows, 4-bit weights"] = lambda: rows.linear(x4, q)
    lin = Exl3Linear(Exl3Tensor.random(1024, 768, 4, seed=1), dev)
    out["exl3_gemv: 4 rows"] = lambda: lin.forward(ops, x4s[:, :1024].contiguous())
    # routed experts: pairs of few rows, prompt rows straight from 4-bit stacks
    E, H, I = 8, 512, 256
    gu, dn = rnd(E, 2 * I, H, scale=0.05), rnd(E, H, I, scale=0.05)
    pick = lambda T: torch.stack([torch.randperm(E, generator=g, device=dev)[:2] for _ in range(T)]).to(torch.int32)
    h4, id4, wt4 = rnd(4, H), pick(4), torch.rand(4, 2, generator=g, device=dev)
    out["moe_experts: 4 rows"] = lambda: ops.moe_experts(h4, id4, wt4, gu, dn, 0, E)
    stack = lambda r, c: ExpertsFP4(torch.randint(0, 256, (E, r, c // 2), generator=g, device=dev, dtype=torch.uint8),
                                    torch.randint(0, 120, (E, r, c // 16), generator=g, device=dev, dtype=torch.uint8), 2.0 ** -13)
    gu4, dn4 = stack(2 * I, H), stack(H, I)
    hp, idp, wtp = rnd(100, H), pick(100), torch.rand(100, 2, generator=g, device=dev)
    ep = ExpertParallel(None, dev, E, H, cap_rows=200)
    out["ep_moe: 100 rows, 4-bit stacks"] = lambda: ep.moe(ops, hp, idp, wtp, gu4, dn4)
    # decode attention: split-KV partials + combine
    hd, nq, nkv, kvb, ctx = 256, 8, 2, 64, 1500
    nb = (ctx + kvb - 1) // kvb + 1
    bt = torch.arange(nb, device=dev, dtype=torch.int32).view(1, nb)
    kc, vc = rnd(nb, kvb, nkv, hd), rnd(nb, kvb, nkv, hd)
    qv = rnd(1, nq * hd)
    proj = rnd(1, nq * hd * 2 + 2 * nkv * hd)
    out["attn_decode_keys: 1 row, 8 key splits"] = lambda: ops.attention(qv, proj, kc, vc, i32(0), i32(ctx), bt, kvb, nq, nkv, hd, True, nsplit=8,
                                                                  segs=(i32(0), i32(0), i32(1), 1))
    q9, p9, len9 = rnd(9, nq * hd), rnd(9, nq * hd * 2 + 2 * nkv * hd), i32(*range(ctx - 8, ctx + 1))
    out["attn_decode_keys: 9 rows, 32 key splits"] = lambda: ops.attention(q9, p9, kc, vc, i32(*[0] * 9), len9, bt, kvb, nq, nkv, hd, True, nsplit=32,
                                                                           segs=(i32(0), i32(0), i32(9), 9), picked=True)
    qm, lat = rnd(1, 16, 576), rnd(nb, kvb, 576)
    out["latent_mma: 1 row, 16 key splits"] = lambda: ops.mla_attention(qm, lat, i32(0), i32(ctx), bt, kvb, 16, 512, 64, 0.05, nsplit=16,
                                                                        segs=(i32(0), i32(0), i32(1), 1))
    # chunked Gated DeltaNet scan
    nk, nv, dk, dv, T = 4, 8, 128, 128, 300
    conv_dim = 2 * nk * dk + nv * dv
    gproj = rnd(T, conv_dim + nv * dv + 2 * nv)
    qkv = rnd(T, conv_dim)
    A_log, dtb = rnd(nv, scale=0.3, dtype=torch.float32), rnd(nv, scale=0.3, dtype=torch.float32)
    rec0, conv0 = rnd(1, nv, dk, dv, scale=0.2, dtype=torch.float32), rnd(1, 3, conv_dim)

    def gdn():
        rec, conv = rec0.clone(), conv0.clone()
        y = ops.gdn_rec(qkv, gproj, rec, conv, A_log, dtb, i32(0), i32(0), i32(T), nk, nv, dk, dv, 1e-6, commit=True, chunked=True, max_rows=T)
        return torch.cat([y.flatten().float(), rec.flatten()])
    out["gdn_chunk: 300 rows (scan)"] = gdn
    return out


def main(argv=None) -> int:
    ap = argparse.ArgumentParser()
    ap.add_argument("--reps", type=int, default=20)
    a = ap.parse_args(argv)
    from ..ops.cuda_ops import CudaOps
    dev = torch.device("cuda", 0)
    ops = CudaOps(dev)
    report, bad = {}, 0
    for name, fn in cases(ops, dev).items():
        first = fn().clone()
        torch.cuda.synchronize(dev)
        same = all(torch.equal(first, fn()) for _ in range(a.reps))
        report[name] = "same bits" if same else "CHANGED"
        bad += 0 if same else 1
    report["status_word"] = ops.status()
    print(json.dumps({"reps": a.reps, "cases": report}))
    return 1 if bad or report["status_word"] else 0


if __name__ == "__main__":
    sys.exit(main())
