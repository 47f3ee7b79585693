// Few-row products y[m][n] = sum_k x[m][k] W[n][k], M <= 32, bound by streaming the weights once: bf16 or NVFP4 weights through a TMA ring
// into mma.sync fragments, with the RMSNorm of the rows in front and residual / SwiGLU / squared relu behind.
//
// What bounds such a product is how many bytes of weights are in flight, and what every launch costs before its first and after its last
// byte. So:
//   * one thread keeps a ring of 16 KB TMA loads full (about 200 KB in flight per SM in two CTAs), from before the previous kernel has ended:
//     weights do not depend on it (where they do, `fresh_w`, the launch starts behind it). Loads held in registers (the form this replaced) kept
//     64 KB in flight.
//   * the units of work (128 rows x 128 bytes of K, stream_mma.cuh) of all row tiles form one list that is cut into equal runs, one per CTA,
//     whatever N and K are.
//   * three warps bring the rows of x beside each unit, in turn, scaled by (1 + w) of the norm, and sum their squares on the way; the norm's
//     factor is a number per row that the epilogue applies. Nothing waits for a pass over whole rows.
//   * eight warps multiply, each its own 16 rows of the tile: a warp finishes its rows alone. Where a run ends inside a tile, every warp
//     leaves its sums in the workspace, and the warp that completes the tile's k adds them up in the order of the runs: results do not depend
//     on timing.
// NVFP4 weights are unpacked to bf16 in registers (stream_mma.cuh: exact), so activations keep 16 bits whatever M is. With a norm in front and
// token columns to spare the rounding of x (1 + w) to bf16 goes into columns of its own.
// SwiGLU: a tile is 64 gate and 64 up rows, a fragment's rows 0..7 the gate's and 8..15 the up's, so both meet in one thread.
//
// The tensor path is mma.sync: for bf16 the products are a tenth of the time, and fragments come out of the ring as they are. For 4-bit weights it
// is part of the bound (issue slots 72 % busy, unpacking and products in the same slots). tcgen05 could take the unpacked weights as its A operand
// from tensor memory, as the prompt attention does with its softmax weights (attn_prefill_tc.cu), and leave those slots to the unpacking: not
// built.
#include "api_ext.h"
#include "stream_mma.cuh"

namespace fb {

constexpr int GS_MATH = 8, GS_FEED = 3;               // warps that multiply / that bring x where it needs work; one more brings the weights
constexpr int GS_MAX_STAGES = 6;
constexpr size_t GS_SMEM = 112 * 1024;                // of a CTA: two are resident

struct GsArgs {
  void* y;                        // bf16 or fp32 [M][ldy]
  const __nv_bfloat16* res;       // [M][ldy] or null
  const __nv_bfloat16* x;         // [M][ldx]
  const __nv_bfloat16* norm_w;    // [K] or null
  const uint8_t* sf;              // NVFP4: scale tiles [row tile][K / 64][512]
  const float* row_alpha;         // NVFP4: tensor scale per weight row (null: w_scale)
  float w_scale, eps;
  // What a CTA leaves of a tile that it does not do alone. A run meets at most two such tiles: one that began in a run before it and one that
  // begins in it and goes on, so records and counters follow the grid and not the number of outputs.
  float* ws;                      // records [CTA][begun before, begins here][warp]: sums of the lanes, sums of squares
  int* counters;                  // [CTA in which the tile begins][warp], left zero
  int* status;
  int M, N, K;
  long ldx, ldy;
  int act, out_f32;
  int kblocks, items, stages;
  int lo_rows;                    // token columns from here on hold what bf16 rounds off x (1 + w); 0: none
};

template <int MT, bool FP4, bool DUAL, bool XT> struct Gs {
  static constexpr int THREADS = (GS_MATH + (XT ? 1 : 1 + GS_FEED)) * 32;
  static constexpr int KU = FP4 ? 256 : 64;                                     // k values of a unit
  static constexpr int SF = FP4 ? (DUAL ? 4096 : 2048) : 0;
  static constexpr int X = 8 * MT * KU * 2;
  static constexpr int STAGE = SM_TILE_BYTES + SF + X;
  static constexpr int REC = 32 * 4 * MT + 8 * MT;                              // floats of a warp's record
};

template <int MT, bool FP4, bool DUAL, bool XT>
__global__ void __launch_bounds__(Gs<MT, FP4, DUAL, XT>::THREADS, 2)
gemv_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, GsArgs a) {
  using C = Gs<MT, FP4, DUAL, XT>;
  extern __shared__ __align__(1024) unsigned char gs_smem[];
  __shared__ __align__(8) uint64_t full_bar[GS_MAX_STAGES], empty_bar[GS_MAX_STAGES];
  __shared__ __align__(8) float ssq_s[GS_MAX_STAGES][8 * MT];       // sums of squares of the rows over a unit
  __shared__ int abort_s;
  pdl_launch_dependents();
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)gs_smem + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long U = (long long)a.items * a.kblocks;
  const long long u0 = (long long)blockIdx.x * U / gridDim.x, u1 = (long long)(blockIdx.x + 1) * U / gridDim.x;
  volatile int* abort_flag = &abort_s;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int i = 0; i < a.stages; ++i) { mbar_init(&full_bar[i], XT ? 1 : 2); mbar_init(&empty_bar[i], GS_MATH); }
    fence_mbar_init();
  }
  if (!XT)                                                 // token columns without a row stay zero
    for (int s = 0; s < a.stages; ++s)
      for (int i = threadIdx.x; i < C::X / 16; i += C::THREADS)
        reinterpret_cast<uint4*>(ring + (size_t)s * C::STAGE + SM_TILE_BYTES + C::SF)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();

  if (warp == GS_MATH) {
    // ---------------- weights ----------------
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      if (XT) tma_prefetch_desc(&tmX);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      int item = (int)(u0 / a.kblocks), kb = (int)(u0 % a.kblocks);
      auto load_x = [&](int st, int k) { tma_load_2d(ring + (size_t)st * C::STAGE + SM_TILE_BYTES, &tmX, &full_bar[st], k * 64, 0); };
      for (long long u = u0; u < u1; ++u) {
        const bool first = XT && u - u0 < a.stages;        // the ring's first turn: x is not there yet
        if (XT && u - u0 == a.stages) {
          pdl_wait();
          int k = (int)(u0 % a.kblocks);
          for (int i = 0; i < a.stages; ++i, k = k + 1 == a.kblocks ? 0 : k + 1) load_x(i, k);
        }
        if (!(ok = sm_wait(&empty_bar[stage], phase ^ 1u, abort_flag))) break;
        unsigned char* st = ring + (size_t)stage * C::STAGE;
        mbar_expect_tx(&full_bar[stage], (uint32_t)(SM_TILE_BYTES + C::SF + (XT ? C::X : 0)));
        const int r0 = item * (DUAL ? 64 : 128), r1 = DUAL ? a.N + r0 : r0 + 64;
        const int col = kb * (FP4 ? 128 : 64);
        tma_load_2d(st, &tmW, &full_bar[stage], col, r0);
        tma_load_2d(st + 8192, &tmW, &full_bar[stage], col, r1);
        if (XT && !first) load_x(stage, kb);
        if (FP4) {
          const size_t kt = (size_t)(a.K / 64), at = (size_t)kb * 4;
          sm_bulk_load(st + SM_TILE_BYTES, a.sf + ((size_t)(r0 / 128) * kt + at) * 512, 2048, &full_bar[stage]);
          if (DUAL) sm_bulk_load(st + SM_TILE_BYTES + 2048, a.sf + ((size_t)(r1 / 128) * kt + at) * 512, 2048, &full_bar[stage]);
        }
        if (++stage == a.stages) { stage = 0; phase ^= 1u; }
        if (++kb == a.kblocks) { kb = 0; ++item; }
      }
      if (XT && u1 - u0 <= a.stages) {                     // all of it was the first turn
        pdl_wait();
        int k = (int)(u0 % a.kblocks);
        for (int i = 0; i < (int)(u1 - u0); ++i, k = k + 1 == a.kblocks ? 0 : k + 1) load_x(i, k);
      }
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
    }
  } else if (!XT && warp > GS_MATH) {
    // ---------------- activations that need work: norm, order of e2m1 pieces ----------------
    // The warps take the units in turn, each with the rows of its next unit in flight (one warp for all of them held the kernel back: gate|up
    // of the 27B model, one row, 56 us with three, 97 with one).
    constexpr int NC = C::KU / 8;                         // 16-byte chunks of a row in a unit
    constexpr int RP = 32 / NC;                           // rows that a warp takes at once
    constexpr int PASS = 8 * MT / RP;
    const int f = warp - GS_MATH - 1, c = lane % NC, m0 = lane / NC;
    pdl_wait();
    uint4 v[PASS], nw = make_uint4(0, 0, 0, 0);
    auto load = [&](int kb) {
      const int k = kb * C::KU + c * 8;
      if (a.norm_w && k < a.K) nw = ldg_cached(a.norm_w + k);
#pragma unroll
      for (int p = 0; p < PASS; ++p) {
        const int m = m0 + p * RP;
        v[p] = m < a.M && k < a.K ? sm_ldg(a.x + (size_t)m * a.ldx + k) : make_uint4(0, 0, 0, 0);
      }
    };
    int kb = (int)((u0 + f) % a.kblocks), stage = f % a.stages;
    uint32_t phase = (uint32_t)(f / a.stages) & 1u;
    if (u0 + f < u1) load(kb);
    for (long long u = u0 + f; u < u1; u += GS_FEED) {
      const bool ok = __all_sync(0xffffffffu, sm_wait(&empty_bar[stage], phase ^ 1u, abort_flag));
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; break; }
      const uint32_t xt = smem_u32(ring + (size_t)stage * C::STAGE + SM_TILE_BYTES + C::SF);
#pragma unroll
      for (int p = 0; p < PASS; ++p) {
        if (p * RP >= a.M) break;
        const int m = m0 + p * RP;
        float ss = 0.f;
        if (m < a.M) {
          uint4 o = v[p];
          if (a.norm_w) {
            const uint32_t xu[4] = {o.x, o.y, o.z, o.w}, wu[4] = {nw.x, nw.y, nw.z, nw.w};
            uint32_t r[4], d[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float x0 = bf_lo(xu[e]), x1 = bf_hi(xu[e]);
              ss = fmaf(x0, x0, fmaf(x1, x1, ss));
              const float y0 = x0 * (1.f + bf_lo(wu[e])), y1 = x1 * (1.f + bf_hi(wu[e]));
              r[e] = pack_bf2(y0, y1);
              d[e] = pack_bf2(y0 - bf_lo(r[e]), y1 - bf_hi(r[e]));
            }
            o = make_uint4(r[0], r[1], r[2], r[3]);
            if (a.lo_rows) {
              const uint4 e = make_uint4(d[0], d[1], d[2], d[3]);
              if (FP4) sm_sts(xt + sm_x_fp4(a.lo_rows + m, c), sm_piece(e));
              else sm_sts(xt + sm_x_bf16(a.lo_rows + m, c), e);
            }
          }
          if (FP4) sm_sts(xt + sm_x_fp4(m, c), sm_piece(o));
          else sm_sts(xt + sm_x_bf16(m, c), o);
        }
        if (a.norm_w) {                                    // the row's sum of squares over this unit
#pragma unroll
          for (int o = NC / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          if (c == 0 && m < a.M) ssq_s[stage][m] = ss;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
      kb = (kb + GS_FEED) % a.kblocks;
      if (u + GS_FEED < u1) load(kb);
      stage += GS_FEED;
      while (stage >= a.stages) { stage -= a.stages; phase ^= 1u; }
    }
  } else {
    // ---------------- products ----------------
    const int g = lane >> 2, t = lane & 3;
    const SmFactors fac = sm_factors();
    const int lo = (DUAL ? 8 : 16) * warp + sm_row(g), hi = lo + (DUAL ? 64 : 8);
    pdl_wait();
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (long long u = u0; u < u1 && ok;) {
      const int item = (int)(u / a.kblocks), kb0 = (int)(u % a.kblocks);
      const int kb1 = (int)((u1 - u) < (long long)(a.kblocks - kb0) ? kb0 + (u1 - u) : a.kblocks);
      // where the rows' scales are inside an atom of 128 rows (a SwiGLU tile is one half of it)
      const int slo = DUAL ? (item & 1) * 64 + lo : lo, shi = DUAL ? (item & 1) * 64 + hi - 64 : hi;
      const uint32_t sf_lo = (uint32_t)((slo & 31) * 16 + (slo >> 5) * 4), sf_hi = (uint32_t)((shi & 31) * 16 + (shi >> 5) * 4) + (DUAL ? 2048u : 0u);
      float part[2][MT][4], acc[MT][4];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[0][i][j] = part[1][i][j] = 0.f;
      float sq[MT][2];                                     // sums of squares of this lane's two tokens per tile
#pragma unroll
      for (int i = 0; i < MT; ++i) sq[i][0] = sq[i][1] = 0.f;
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = __all_sync(0xffffffffu, sm_wait(&full_bar[stage], phase, abort_flag));
        if (!ok) break;
        const uint32_t st = smem_u32(ring + (size_t)stage * C::STAGE), sf = st + SM_TILE_BYTES;
        sm_unit<MT, FP4, XT>(part, st, lo, hi, sf + C::SF, sf + sf_lo, sf + sf_hi, fac);
        if (!XT && a.norm_w) {
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            const float2 q = *reinterpret_cast<const float2*>(&ssq_s[stage][i * 8 + 2 * t]);
            sq[i][0] += q.x; sq[i][1] += q.y;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
        if (++stage == a.stages) { stage = 0; phase ^= 1u; }
      }
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; break; }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = part[0][i][j] + part[1][i][j];
      u += kb1 - kb0;
      bool finish = true;
      if (kb0 != 0 || kb1 != a.kblocks) {
        const long long ui0 = (long long)item * a.kblocks;
        const int c_first = (int)(((ui0 + 1) * gridDim.x - 1) / U), c_last = (int)(((ui0 + a.kblocks) * gridDim.x - 1) / U);
        auto record = [&](int cta) { return a.ws + (size_t)((cta * 2 + (cta == c_first ? 1 : 0)) * GS_MATH + warp) * C::REC; };
        float* rec = record((int)blockIdx.x);
        int* counter = a.counters + c_first * GS_MATH + warp;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          __stcg(reinterpret_cast<float4*>(rec) + i * 32 + lane, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
          if (!XT && g == 0) __stcg(reinterpret_cast<float2*>(rec + 128 * MT) + i * 4 + t, make_float2(sq[i][0], sq[i][1]));
        }
        __threadfence();
        __syncwarp();
        int old = 0;
        if (lane == 0) old = atomicAdd(counter, kb1 - kb0);
        finish = __shfl_sync(0xffffffffu, old, 0) + (kb1 - kb0) == a.kblocks;
        if (finish) {
          __threadfence();
#pragma unroll
          for (int i = 0; i < MT; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; sq[i][0] = sq[i][1] = 0.f; }
          const int ns = c_last - c_first + 1;
          constexpr int B = MT <= 2 ? 4 : 2;               // records in flight
          for (int s0 = 0; s0 < ns; s0 += B) {             // added in the order of the runs, whoever arrived last
            float4 p[B][MT];
            float2 q[B][MT];
#pragma unroll
            for (int j = 0; j < B; ++j) {
              const float* r = record(c_first + min(s0 + j, ns - 1));
#pragma unroll
              for (int i = 0; i < MT; ++i) {
                p[j][i] = __ldcg(reinterpret_cast<const float4*>(r) + i * 32 + lane);
                if (!XT) q[j][i] = __ldcg(reinterpret_cast<const float2*>(r + 128 * MT) + i * 4 + t);
              }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
              if (s0 + j < ns)
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                  acc[i][0] += p[j][i].x; acc[i][1] += p[j][i].y; acc[i][2] += p[j][i].z; acc[i][3] += p[j][i].w;
                  if (!XT) { sq[i][0] += q[j][i].x; sq[i][1] += q[j][i].y; }
                }
          }
          if (lane == 0) *counter = 0;
        }
      }
      if (!finish) continue;
      if (!XT && MT == 1 && a.lo_rows) {                          // columns 4 .. 7 are the rest of 0 .. 3
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[0][j] += __shfl_xor_sync(0xffffffffu, acc[0][j], 2);
      }
      // c0, c1: fragment row g, tokens 2t, 2t + 1; c2, c3: row g + 8
      const int n_lo = item * (DUAL ? 64 : 128) + lo, n_hi = n_lo + 8;
      float al = 1.f, ah = 1.f;
      if (FP4) {
        al = ah = a.w_scale;
        if (a.row_alpha) {
          al = n_lo < a.N ? a.row_alpha[n_lo] : 0.f;
          ah = DUAL ? (n_lo < a.N ? a.row_alpha[a.N + n_lo] : 0.f) : n_hi < a.N ? a.row_alpha[n_hi] : 0.f;
        }
        al *= SM_FP4_FACTOR; ah *= SM_FP4_FACTOR;
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int m = i * 8 + (XT ? sm_row(2 * t + e) : 2 * t + e);
          if (m >= a.M) continue;
          const float rn = !XT && a.norm_w ? rsqrtf(sq[i][e] / (float)a.K + a.eps) : 1.f;
          const float v0 = acc[i][e] * (rn * al), v1 = acc[i][2 + e] * (rn * ah);
          auto store = [&](int n, float v) {
            if (n >= a.N) return;
            const size_t at = (size_t)m * a.ldy + n;
            if (a.res) v += bf2f(a.res[at]);
            if (a.out_f32) reinterpret_cast<float*>(a.y)[at] = v;
            else reinterpret_cast<__nv_bfloat16*>(a.y)[at] = f2bf(v);
          };
          if (DUAL) {
            store(n_lo, siluf_(v0) * v1);
          } else {
            store(n_lo, epilogue_act(v0, a.act));
            store(n_hi, epilogue_act(v1, a.act));
          }
        }
    }
  }
  __syncthreads();
  if (abort_s && threadIdx.x == 0)                         // loads already issued still target this CTA's shared memory
    for (int i = 0; i < a.stages; ++i)
      for (uint32_t p = 0; p < 2; ++p) (void)mbar_wait(&full_bar[i], p, 1u << 12);
}

struct GsPlan { int grid, items, kblocks; long rec_floats; };

// How many runs the units are cut into. A run costs its share of the ring's first turn and, where it ends inside a tile, a record that another
// one reads: short runs lose. Measured (us a call in a row of calls, one row, N x K):
//   bf16   an SM's second CTA from eight units each on: 5120 x 2048 (1280 units), 296 / 160 runs 9.4 / 6.8; 8224 x 5120 (5200) 20.1 with 296;
//          at least four units: 576 x 7168 (560), 280 / 140 runs 9.6 / 7.2, 4112 x 1024 (528), 264 / 132 / 66 runs 6.5 / 6.3 / 7.1
//   e2m1   (a unit is four times the work) whole tiles where they are short, 4112 x 1024 (132), 33 / 66 runs 5.6 / 6.5; else at least two units,
//          5120 x 2048 (320), 80 / 160 runs 9.4 / 7.8
static GsPlan gs_plan(int M, int N, int K, bool fp4, bool dual, int sm_count) {
  GsPlan p;
  p.items = dual ? (N + 63) / 64 : (N + 127) / 128;
  p.kblocks = fp4 ? K / 256 : (K + 63) / 64;
  const long long U = (long long)p.items * p.kblocks;
  long long grid = U / (fp4 ? 2 : 4);
  if (grid < 1) grid = 1;
  if (!fp4 && grid > sm_count && U < 16LL * sm_count) grid = sm_count;
  if (grid > 2LL * sm_count) grid = 2LL * sm_count;
  if (fp4 && p.kblocks <= 4 && p.items <= 2 * sm_count) grid = p.items;
  // nearly as many tiles as CTAs: a whole tile each has nothing to merge
  if (p.items <= grid && (long long)p.items * 8 >= grid * 7) grid = p.items;
  p.grid = (int)grid;
  p.rec_floats = (long)p.grid * 2 * GS_MATH * (136 * ((M + 7) / 8));
  return p;
}

template <int MT, bool FP4, bool DUAL, bool XT>
static int launch_gs(GsArgs a, const GsPlan& p, const CUtensorMap& tw, const CUtensorMap& tx, bool fresh_w, cudaStream_t s) {
  using C = Gs<MT, FP4, DUAL, XT>;
  static const cudaError_t attr =
      cudaFuncSetAttribute(gemv_stream_kernel<MT, FP4, DUAL, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_SMEM);
  if (attr != cudaSuccess) return (int)attr;
  int stages = (int)((GS_SMEM - 1024) / C::STAGE);
  if (stages > GS_MAX_STAGES) stages = GS_MAX_STAGES;
  a.stages = stages;
  return (int)launch_pdl_if(!fresh_w, gemv_stream_kernel<MT, FP4, DUAL, XT>, dim3(p.grid), dim3(C::THREADS), (size_t)stages * C::STAGE + 1024, s, tw, tx, a);
}

}  // namespace fb

using namespace fb;

// Whether the kernel takes a call: 0 leaves it to other kernels (rows that lie on no 16 bytes or over one another, more rows than its token tiles,
// 4-bit rows that are no whole units). x may be null (rows that are still to be made, ldx apart).
extern "C" int fb_gemv_stream_fits(const void* x, const void* w, const void* sf, const void* norm_w, int M, int N, int K, long ldx, int mode) {
  const bool fp4 = sf != nullptr;
  if (M > (fp4 || norm_w ? 8 : 32) || K <= 0 || K % 8 || (fp4 && (K % 256 || (mode == 1 && N % 128)))) return 0;
  if (ldx % 8 || (!fp4 && !norm_w && M > 1 && ldx < K)) return 0;
  return (((uintptr_t)x | (uintptr_t)w | (uintptr_t)sf | (uintptr_t)norm_w) & 15) == 0;
}

// Floats of workspace and ints of counters that any call of up to 32 rows fits, whatever its sizes.
extern "C" long fb_gemv_stream_ws_floats(int sm_count) { return 2L * sm_count * 2 * GS_MATH * 136 * 4; }
extern "C" int fb_gemv_stream_counters(int sm_count) { return 2 * sm_count * GS_MATH; }

// Weights bf16 [N or 2N][K] (sf null; K % 8 == 0; M <= 32, with norm_w M <= 8) or e2m1 codes [..][K / 2] with scale tiles sf (K % 256 == 0,
// SwiGLU: N % 128 == 0; M <= 8). mode 1: SwiGLU over [gate rows | up rows], 2: squared relu. fresh_w: the weights were written on this stream
// just before.
extern "C" int fb_gemv_stream(void* y, const void* x, const void* w, const void* sf, float w_scale, const float* row_alpha, const void* norm_w,
                              const void* res, int M, int N, int K, long ldx, long ldy, float eps, int mode, int out_f32, float* ws,
                              long ws_floats, int* counters, int n_counters, int fresh_w, int* status, int sm_count, cudaStream_t s) {
  if (M <= 0 || N <= 0) return 0;
  const bool fp4 = sf != nullptr, dual = mode == 1;
  if (sm_count <= 0) sm_count = 148;
  if (!x || !w || !fb_gemv_stream_fits(x, w, sf, norm_w, M, N, K, ldx, mode)) return -1;
  const GsPlan p = gs_plan(M, N, K, fp4, dual, sm_count);
  if (!ws || !counters || p.rec_floats > ws_floats || p.grid > n_counters / GS_MATH) return -6;
  GsArgs a;
  a.y = y; a.res = (const __nv_bfloat16*)res; a.x = (const __nv_bfloat16*)x; a.norm_w = (const __nv_bfloat16*)norm_w; a.sf = (const uint8_t*)sf;
  a.row_alpha = row_alpha; a.w_scale = w_scale; a.eps = eps; a.ws = ws; a.counters = counters; a.status = status; a.M = M; a.N = N; a.K = K;
  a.ldx = ldx; a.ldy = ldy; a.act = mode == 2 ? ACT_RELU2 : ACT_NONE; a.out_f32 = out_f32; a.kblocks = p.kblocks; a.items = p.items;
  a.stages = 0;
  a.lo_rows = norm_w && M <= 4 ? 4 : 0;
  const int mt = (M + 7) / 8;
  CUtensorMap tw, tx;
  if (!sm_map(&tw, w, fp4, fp4 ? K / 2 : K, dual ? 2L * N : N, fp4 ? K / 2 : 2L * K, fp4 ? 128 : 64, 64)) return -12;
  if (fp4 || norm_w) {
    if (fp4) return dual ? launch_gs<1, true, true, false>(a, p, tw, tw, fresh_w, s) : launch_gs<1, true, false, false>(a, p, tw, tw, fresh_w, s);
    return dual ? launch_gs<1, false, true, false>(a, p, tw, tw, fresh_w, s) : launch_gs<1, false, false, false>(a, p, tw, tw, fresh_w, s);
  }
  if (!sm_map(&tx, x, false, K, M, 2L * (M > 1 ? ldx : K), 64, 8 * mt)) return -12;
#define FB_GS(MT) return dual ? launch_gs<MT, false, true, true>(a, p, tw, tx, fresh_w, s) : launch_gs<MT, false, false, true>(a, p, tw, tx, fresh_w, s)
  switch (mt) {
    case 1: FB_GS(1);
    case 2: FB_GS(2);
    case 3: FB_GS(3);
    default: FB_GS(4);
  }
#undef FB_GS
}
