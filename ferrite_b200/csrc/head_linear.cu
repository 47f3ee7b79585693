// One small linear per attention head over a few rows: y[t][h][0..N) = W[h] (N x K) . x[t][h][0..K), t < T <= 8 per
// row tile (grid.z covers more). Multi-head latent attention needs two of these per layer and step: the key
// up-projection folded into the query (N = latent width, K = head width) and the value up-projection after the
// attention (N = value width, K = latent width). One launch streams the whole [heads][N][K] stack once; the reference
// issues its per-head products from the attention kernels' prologue / epilogue (`kernels/k-ds/src/attn.rs:151-548`).
//
// CTA = (64 outputs, one head, one tile of ROWS rows), 8 warps x 8 outputs, no shared memory. A group of LPO =
// min(32, K / 8) lanes owns an output and reads its weight row with 16-byte loads (CPL = K / 8 / LPO of them per lane).
// A lane meets the same K chunks in every output, so it keeps its slice of the x rows in registers (packed bf16) for the
// whole CTA. A warp works on U outputs per lane group at a time and issues all their weight loads before it uses any.
// Sums go over the lanes of a group in a fixed xor tree: a row's bits do not depend on the other rows of the step.
#include "common.cuh"

namespace fb {

constexpr int HL_OUT = 64;
constexpr int HL_MAX_K = 1024;

template <int CPL, int ROWS, int HL_U>
__global__ void __launch_bounds__(256, 2) head_linear_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ W, int T, int N, int K,
                                                          long x_rs, long x_hs, long y_rs, long y_hs) {
  const int h = blockIdx.y, t0 = blockIdx.z * ROWS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = K / 8;
  int lpo = 1;                                        // lanes per output: the power of two that covers the chunks, at most 32
  while (lpo < 32 && lpo < chunks) lpo <<= 1;
  const int per_pass = 32 / lpo;                      // outputs a warp covers in one pass
  const int passes = (HL_OUT / 8) / per_pass > 0 ? (HL_OUT / 8) / per_pass : 1;
  const int sub = lane / lpo, l = lane % lpo;
  const int n_base = blockIdx.x * HL_OUT + warp * (HL_OUT / 8);
  const __nv_bfloat16* Wh = W + (size_t)h * N * K;
  uint4 raw[HL_U][CPL];
  auto out_of = [&](int pass) { return n_base + pass * per_pass + sub; };
  auto live = [&](int pass) { return pass < passes && pass * per_pass + sub < HL_OUT / 8 && out_of(pass) < N; };
  auto load_batch = [&](int p0) {
#pragma unroll
    for (int u = 0; u < HL_U; ++u) {
      const bool ok = live(p0 + u);
#pragma unroll
      for (int c = 0; c < CPL; ++c)
        raw[u][c] = ok && l + c * lpo < chunks ? ldg_stream(reinterpret_cast<const uint4*>(Wh + (size_t)out_of(p0 + u) * K) + l + c * lpo)
                       : make_uint4(0, 0, 0, 0);
    }
  };
  load_batch(0);
  // this lane's K chunks of the x rows: as floats while they fit the register budget (no unpacking per output), else
  // packed bf16
  constexpr bool XF = ROWS * CPL <= 8;
  uint4 xr[XF ? 1 : ROWS][XF ? 1 : CPL];
  float xf[XF ? ROWS : 1][XF ? CPL : 1][8];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const uint4 v = t0 + r < T && l + c * lpo < chunks ? *reinterpret_cast<const uint4*>(x + (size_t)(t0 + r) * x_rs + (size_t)h * x_hs + (l + c * lpo) * 8)
                                 : make_uint4(0, 0, 0, 0);
      if constexpr (XF) {
        const uint32_t v4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { xf[r][c][2 * j] = bf_lo(v4[j]); xf[r][c][2 * j + 1] = bf_hi(v4[j]); }
      } else {
        xr[r][c] = v;
      }
    }
  }
  for (int p0 = 0; p0 < passes; p0 += HL_U) {          // the same trip count for every lane: shuffles below
    if (p0 > 0) load_batch(p0);
#pragma unroll
    for (int u = 0; u < HL_U; ++u) {
      float acc[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const uint32_t w4[4] = {raw[u][c].x, raw[u][c].y, raw[u][c].z, raw[u][c].w};
        float wv[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) { wv[2 * j] = bf_lo(w4[j]); wv[2 * j + 1] = bf_hi(w4[j]); }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          float s = acc[r];
          if constexpr (XF) {
#pragma unroll
            for (int j = 0; j < 8; ++j) s = fmaf(wv[j], xf[r][c][j], s);
          } else {
            const uint32_t x4[4] = {xr[r][c].x, xr[r][c].y, xr[r][c].z, xr[r][c].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { s = fmaf(wv[2 * j], bf_lo(x4[j]), s); s = fmaf(wv[2 * j + 1], bf_hi(x4[j]), s); }
          }
          acc[r] = s;
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        for (int off = lpo >> 1; off > 0; off >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
      if (l == 0 && live(p0 + u)) {
        const int n = out_of(p0 + u);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (t0 + r < T) y[(size_t)(t0 + r) * y_rs + (size_t)h * y_hs + n] = __float2bfloat16(acc[r]);
      }
    }
  }
}

// Heads of up to 512 columns, a multiple of 32, on the tensor cores: m16n8k16 with outputs as M and the tile's rows (8) as N. A dot product does not
// care about the order of k, so lane t of the four that share a fragment row takes whole 16-byte chunks, of the weights straight from global memory:
// chunk 4 b + t of block b (32 columns) holds the lane's operands of two products. Sums of 128 columns are added in 32 bits rounded (the tensor
// cores cut). A row's bits depend on no other row. grid (groups of WARPS * tiles outputs x 16, heads, tiles of 8 rows).
// The kernel above needs four shuffles an output and row and takes 3.5 us a row at 128 heads of 512 x 128 (17 MB of weights, 2.6 us). us, it / this,
// at 1, 2, 4, 6, 8 rows: 6.8, 8.8, 14.6, 23.7, 30.2 / 3.5, 3.5, 3.6, 3.5, 3.7; 128 x 512: 7.3, 9.2, 12.5, 21.3, 27.4 / 4.6, 4.7, 4.7, 5.0, 5.1.
constexpr int HM_WARPS = 4;

template <int SLABS>
__global__ void __launch_bounds__(HM_WARPS * 32) head_mma_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* x, const __nv_bfloat16* W, int T, int N,
                                                                 int K, long x_rs, long x_hs, long y_rs, long y_hs, int tiles) {
  const int h = blockIdx.y, t0 = blockIdx.z * 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = (blockIdx.x * HM_WARPS + warp) * tiles * 16, n1 = min(N, n0 + tiles * 16);
  pdl_launch_dependents();
  {                                                   // (only L2 is asked: the kernel ahead may have written the weights)
    const char* mine = reinterpret_cast<const char*>(W + ((size_t)h * N + n0) * K);
    for (long i = lane * 128l; i < 2l * K * (n1 - n0); i += 32 * 128) prefetch_l2(mine + i);
  }
  pdl_wait();
  x = after_wait(x);
  W = after_wait(W);
  if (n0 >= N) return;
  const __nv_bfloat16* Wh = W + (size_t)h * N * K + t * 8;
  auto load = [&](uint4 (&a)[4][2], int n, int slab) {
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = slab * 128 + b * 32;
        a[b][i] = k < K && n < n1 ? ldg_stream(reinterpret_cast<const uint4*>(Wh + (size_t)min(n + g + i * 8, N - 1) * K + k)) : make_uint4(0, 0, 0, 0);
      }
  };
  uint4 a[2][4][2];
  load(a[0], n0, 0);
  uint4 xr[SLABS * 4];
#pragma unroll
  for (int b = 0; b < SLABS * 4; ++b)
    xr[b] = b * 32 < K && t0 + g < T ? *reinterpret_cast<const uint4*>(x + (size_t)(t0 + g) * x_rs + (size_t)h * x_hs + b * 32 + t * 8) : make_uint4(0, 0, 0, 0);
  auto mma = [](float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  };
  // two tiles at a time where a tile is one slab, so that the buffers' turns are known
  for (int n = n0; n < n1; n += SLABS == 1 ? 32 : 16) {
#pragma unroll
    for (int half = 0; half < (SLABS == 1 ? 2 : 1); ++half) {
      const int nn = n + half * 16;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < SLABS; ++s) {
        constexpr bool one = SLABS == 1;
        const int cur = one ? half : s & 1;
        if (s + 1 < SLABS) load(a[cur ^ 1], nn, s + 1);
        else load(a[cur ^ 1], nn + 16, 0);
        float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint4 lo = a[cur][b][0], hi = a[cur][b][1], v = xr[s * 4 + b];
          mma(c[0], lo.x, hi.x, lo.y, hi.y, v.x, v.y);
          mma(c[1], lo.z, hi.z, lo.w, hi.w, v.z, v.w);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] += c[0][e] + c[1][e];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = t0 + 2 * t + (e & 1), o = nn + g + (e >> 1) * 8;
        if (row < T && o < n1) y[(size_t)row * y_rs + (size_t)h * y_hs + o] = __float2bfloat16(sum[e]);
      }
    }
  }
}

}  // namespace fb

using namespace fb;

// x: rows of stride x_rs elements, head h at offset h * x_hs (16-byte aligned); y likewise (any element alignment).
// T > 8 runs as row tiles of 8 (grid.z).
extern "C" int fb_head_linear(void* y, const void* x, const void* W, int T, int heads, int N, int K, long x_rs, long x_hs,
                              long y_rs, long y_hs, cudaStream_t s) {
  if (T <= 0 || heads <= 0) return 0;
  if (K < 8 || K > HL_MAX_K || K % 8 || x_rs % 8 || x_hs % 8 || heads > 65535) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) return -1;
  if (K % 32 == 0 && K <= 512) {
    const int slabs = K <= 128 ? 1 : K <= 256 ? 2 : 4, z = (T + 7) / 8;
    // tiles a warp: as many as leave every SM two CTAs
    int tiles = slabs == 1 ? 2 : 1;
    while (tiles < 8 && (long)heads * z * ((N + 2 * tiles * HM_WARPS * 16 - 1) / (2 * tiles * HM_WARPS * 16)) >= 2 * 148) tiles *= 2;
    const auto kern = slabs == 1 ? head_mma_kernel<1> : slabs == 2 ? head_mma_kernel<2> : head_mma_kernel<4>;
    return (int)launch_pdl(kern, dim3((N + tiles * HM_WARPS * 16 - 1) / (tiles * HM_WARPS * 16), heads, z), dim3(HM_WARPS * 32), (size_t)0, s,
                           (__nv_bfloat16*)y, (const __nv_bfloat16*)x, (const __nv_bfloat16*)W, T, N, K, x_rs, x_hs, y_rs, y_hs, tiles);
  }
  const int rows = T >= 8 ? 8 : T > 2 ? 4 : T;        // rows per tile: 1, 2, 4 or 8
  dim3 grid((N + HL_OUT - 1) / HL_OUT, heads, (T + rows - 1) / rows);
  const int chunks = K / 8, cpl = chunks <= 32 ? 1 : chunks <= 64 ? 2 : 4;
#define FB_HL(C, R)                                                                                                      \
  head_linear_kernel<C, R, (C == 1 ? (R == 8 ? 2 : 4) : C == 2 ? (R == 8 ? 1 : 2) : 1)><<<grid, 256, 0, s>>>(                \
      (__nv_bfloat16*)y, (const __nv_bfloat16*)x, (const __nv_bfloat16*)W, T, N, K, x_rs, x_hs, y_rs, y_hs)
#define FB_HL_R(C)                                                                                                       \
  { if (rows == 1) FB_HL(C, 1); else if (rows == 2) FB_HL(C, 2); else if (rows == 4) FB_HL(C, 4); else FB_HL(C, 8); }
  if (cpl == 1) FB_HL_R(1) else if (cpl == 2) FB_HL_R(2) else if (cpl == 4) FB_HL_R(4) else return -1;
#undef FB_HL_R
#undef FB_HL
  return (int)cudaGetLastError();
}
