// Gated DeltaNet, chunked scan for prompt-sized segments (same recurrence as gdn.cu, see its header):
//   S_t = g_t S_{t-1} + k_t d_t^T,   d_t = beta_t (v_t - g_t S_{t-1}^T k_t),   y_t = S_t^T q_t.
//
// Over a chunk of C = 64 rows that starts from state S_0, with c_t = sum_{i<=t} log g_i:
//   (I + A) D = diag(beta) (V - diag(e^{c}) K S_0),     A[t][i] = beta_t e^{c_t - c_i} (k_t . k_i)   (i < t)
//   Y   = diag(e^{c}) Q S_0 + P D,                      P[t][i] = e^{c_t - c_i} (q_t . k_i)          (i <= t)
//   S_C = e^{c_C} S_0 + sum_i e^{c_C - c_i} k_i d_i^T
// so the work splits in two kernels:
//   prep  (parallel over chunk x head): decays, unit lengths, T' = (I + A)^{-1} diag(beta), P                            -> scratch
//   scan  (sequential over the chunks of a segment, parallel over head x 16- or 32-column slices of the state):
//         five small matrix products per chunk, operands double-buffered through cp.async.
// State columns never interact, which is what lets the scan split the value dimension over CTAs.
// The products run on the tensor cores at the precision of 32-bit ones. k and q are bf16 rows times one number each (their lengths), which
// moves out of the products, so that these operands are exact; 32-bit operands (state, deltas, T', P) are cut into three bf16 terms of eight
// bits, and every pair of terms above 2^-24 of the leading one is multiplied: three products against k or q, six between two 32-bit operands.
// The leading terms have sums of their own, since the tensor cores cut what they add to the scale of the largest addend. Off 64 bits (relative, 2-norm;
// 16 heads, 2048 rows): y 2.0e-7, state 1.6e-7; 1111 rows 2.2e-7 and 1.5e-7; steep decays 2.1e-7 and 1.0e-7. (All in 32-bit FMA: 2.9e-7, 4.0e-7;
// 3.2e-7, 2.0e-7; 6.1e-7, 4.5e-7.)
// One layer, prep + scan, us, against both in FMA on the CUDA cores: 2048 rows of 16 heads 80 + 269 -> 26 + 81, 1500 of 32 heads 112 + 387 -> 31 + 104,
// 64 of 16 heads together 32 -> 15.
//
// Counterparts in the reference: `fe_gdn_chunk`, `fe_gdn_chunk_tc`, `fe_gdn_chunk_tc1` (`kernels/k-gdn/src/lib.rs`),
// `fx_gdn_chunk*` (`kernels/k-fnext/src/gdn.rs`); host wrapper `Gdn::run` (`crates/fe-gdn/src/lib.rs`).
#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace fb {

constexpr int GC = 64;            // rows per chunk
constexpr int GC_PREP_THREADS = 256;

__device__ __forceinline__ void gc_cp16(void* smem, const void* gmem, bool live = true) {       // zeros where not live
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gc_ldsm(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p))
               : "memory");
}
__device__ __forceinline__ void gc_ldsm_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p))
               : "memory");
}
__device__ __forceinline__ void gc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Three bf16 terms of two values, each pair packed: x = t[0] + t[1] + t[2] to 2^-24.
__device__ __forceinline__ void gc_split(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = pack_bf2(x, y);
    if (i < 2) { x -= bf_lo(t[i]); y -= bf_hi(t[i]); }
  }
}

__device__ __forceinline__ float gc_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// floats of scratch per (chunk, head): T'[C][C] | P[C][C] | rows' factors: e^{c_t} / |k_t| [C] | e^{c_t} / (|q_t| sqrt(dk)) [C] |
// e^{c_C - c_t} / |k_t| [C] | e^{c_C}, padded to 4. Above the diagonal's 16 x 16 blocks T' and P are not written.
constexpr int GC_VEC = 3 * GC + 4;
__host__ __device__ constexpr long gc_rec_floats() { return 2l * GC * GC + GC_VEC; }

// ---- prep ------------------------------------------------------------------------------------------------
// T = (I + A)^{-1} of blocks of 2 w rows from that of their halves: T21 = -T22 (A21 T11). Zeros lie above T11's and T22's diagonals; above T22's
// nothing is added, so that a row which is no number reaches no row ahead of it.
template <int w, int LDA>
__device__ __forceinline__ void gc_merge(const float* Am, float* Tm, float* Xm) {
  constexpr int PER = w * w / (GC_PREP_THREADS / (GC / 2 / w));         // elements a thread, neighbours in a row: 2 or 4
  constexpr int EACH = w * w / PER;
  const int blk = threadIdx.x / EACH, u = threadIdx.x % EACH, r0 = blk * 2 * w, r = u * PER / w, c = u * PER % w;
  using V = typename std::conditional<PER == 4, float4, float2>::type;
  // (terms from the last-th on are not added)
  auto dot = [&](const float* a, const float* b, int last, float (&acc)[PER]) {
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[e] = 0.f;
#pragma unroll 1
    for (int i0 = 0; i0 < last; i0 += 8)
#pragma unroll
      for (int i = i0; i < i0 + 8; ++i) {
        const V v = *reinterpret_cast<const V*>(b + i * LDA);
        const float x = a[i];
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[e] = i < last ? fmaf(x, reinterpret_cast<const float*>(&v)[e], acc[e]) : acc[e];
      }
  };
  float acc[PER];
  dot(Am + (r0 + w + r) * LDA + r0, Tm + r0 * LDA + r0 + c, w, acc);
#pragma unroll
  for (int e = 0; e < PER; ++e) Xm[(blk * w + r) * LDA + c + e] = acc[e];
  __syncthreads();
  dot(Tm + (r0 + w + r) * LDA + r0 + w, Xm + blk * w * LDA + c, r + 1, acc);
#pragma unroll
  for (int e = 0; e < PER; ++e) Tm[(r0 + w + r) * LDA + r0 + c + e] = -acc[e];
  __syncthreads();
}

// grid (max chunks per segment, nv, nseg); three CTAs an SM. Bound by the latency of a dozen phases between barriers. (I + A)^{-1} by blocks: four of 16 x 16 by substitution (a thread a column), then twice the blocks
// below them, -T22 (A21 T11).
template <int DK>
__global__ void __launch_bounds__(GC_PREP_THREADS)
gdn_chunk_prep_kernel(float* __restrict__ scratch, const __nv_bfloat16* qkv, const __nv_bfloat16* proj, long proj_stride,
                      const float* __restrict__ A_log, const float* __restrict__ dt_bias, const int* seg_row0, const int* seg_nrows, int nk, int nv,
                      int dv, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int LDK = DK + 8, LDA = GC + 4;
  extern __shared__ __align__(16) unsigned char sm_prep[];
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(sm_prep);      // [GC][LDK]
  __nv_bfloat16* Qs = Ks + GC * LDK;                                  // [GC][LDK]
  float* Am = reinterpret_cast<float*>(Qs + GC * LDK);                // [GC][LDA]
  float* Tm = Am + GC * LDA;                                          // [GC][LDA]
  float* Xm = reinterpret_cast<float*>(sm_prep);                      // [32][LDA], once K and Q are done with
  __shared__ float chi[GC], clo[GC], bs[GC], rk[GC], rq[GC];       // c_t / ln 2 in two parts: differences of neighbours stay exact
  const int chunk = blockIdx.x, h = blockIdx.y, seg = blockIdx.z;
  const int n = after_wait(seg_nrows)[seg], seg0 = after_wait(seg_row0)[seg];
  if (chunk * GC >= n) return;
  qkv = after_wait(qkv);
  proj = after_wait(proj);
  const int row0 = seg0 + chunk * GC;
  const int valid = min(GC, n - chunk * GC);
  const int kh = h / (nv / nk);
  const int conv_dim = 2 * nk * DK + nv * dv;
  const int q_off = kh * DK, k_off = nk * DK + kh * DK;
  const int b_off = conv_dim + nv * dv + h, a_off = b_off + nv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* gT = scratch + ((size_t)(seg0 / GC + seg + chunk) * nv + h) * gc_rec_floats();
  float* gP = gT + GC * GC;
  float* gv = gP + GC * GC;

  // decays: their logs are summed up over the rows in 64 bits (neighbours' differences count, far down a steep sum), two a lane
  float gate[2] = {0.f, 0.f}, step[2] = {0.f, 0.f};
  if (warp == 0) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int t = 2 * lane + j;
      if (t < valid) {
        const __nv_bfloat16* pr = proj + (size_t)(row0 + t) * proj_stride;
        gate[j] = bf2f(pr[b_off]);
        step[j] = bf2f(pr[a_off]);
      }
    }
  }
  // rows of k and q (zeros past the segment's end) and their lengths: 16 lanes a row
  constexpr int PR = DK / 8, PIECES = 2 * GC * PR / GC_PREP_THREADS;
  static_assert(PR == 16, "");
  uint4 raw[PIECES];
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int t = (i * GC_PREP_THREADS + tid) / PR % GC, c = tid % PR * 8;
    raw[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t < valid) raw[i] = *reinterpret_cast<const uint4*>(qkv + (size_t)(row0 + t) * conv_dim + (i >= PIECES / 2 ? q_off : k_off) + c);
  }
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int t = (i * GC_PREP_THREADS + tid) / PR % GC, c = tid % PR * 8;
    *reinterpret_cast<uint4*>((i >= PIECES / 2 ? Qs : Ks) + t * LDK + c) = raw[i];
    const uint32_t u[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) { sq = fmaf(bf_lo(u[j]), bf_lo(u[j]), sq); sq = fmaf(bf_hi(u[j]), bf_hi(u[j]), sq); }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((lane & 15) == 0) {
      if (i >= PIECES / 2) rq[t] = rsqrtf(sq + eps) * rsqrtf((float)DK);
      else rk[t] = rsqrtf(sq + eps);
    }
  }
  double c2[2] = {0.0, 0.0};
  if (warp == 0) {
    float beta[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const bool live = 2 * lane + j < valid;
      beta[j] = live ? sigmoidf_(gate[j]) : 0.f;
      if (live) c2[j] = -1.4426950408889634 * (double)(__expf(A_log[h]) * softplusf_(step[j] + dt_bias[h]));
    }
    double up = c2[0] + c2[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double below = __shfl_up_sync(0xffffffffu, up, o);
      if (lane >= o) up += below;
    }
    c2[0] = up - c2[1]; c2[1] = up;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      bs[2 * lane + j] = beta[j];
      chi[2 * lane + j] = (float)c2[j];
      clo[2 * lane + j] = (float)(c2[j] - (double)(float)c2[j]);
    }
  }
  __syncthreads();
  if (warp == 0) {
    const double cC = __shfl_sync(0xffffffffu, c2[1], 31);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int t = 2 * lane + j;
      const float e = exp2f((float)c2[j]);
      gv[t] = e * rk[t];
      gv[GC + t] = e * rq[t];
      gv[2 * GC + t] = exp2f((float)(cC - c2[j])) * rk[t];
    }
    if (lane == 0) gv[3 * GC] = exp2f((float)cC);
  }

  // k k^T (warps 0 .. 3, 16 rows each) and q k^T (4 .. 7), blocks up to the diagonal
  const int g = lane >> 2, t4 = lane & 3;
  {
    const int mt = warp & 3;
    const bool isq = warp >= 4;
    const __nv_bfloat16* A = (isq ? Qs : Ks) + (mt * 16 + (lane & 15)) * LDK + (lane >> 4) * 8;
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll 2
    for (int k = 0; k < DK; k += 16) {
      uint32_t a[4];
      gc_ldsm(a, A + k);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        if (j > 2 * mt + 1) break;
        uint32_t b[4];
        gc_ldsm(b, Ks + (j * 8 + (lane >> 4) * 8 + (lane & 7)) * LDK + k + ((lane >> 3) & 1) * 8);
        gc_mma(acc[j], a, b[0], b[1]);
        gc_mma(acc[j + 1], a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j > 2 * mt + 1) break;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = mt * 16 + g + half * 8, i = j * 8 + 2 * t4;
        float2 v;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool in = isq ? i + e <= t : i + e < t;
          const float dec = in ? gc_exp2((chi[t] - chi[i + e]) + (clo[t] - clo[i + e])) * rk[i + e] * (isq ? rq[t] : rk[t] * bs[t]) : 0.f;
          (e ? v.y : v.x) = in ? dec * acc[j][2 * half + e] : 0.f;
        }
        *reinterpret_cast<float2*>(isq ? gP + t * GC + i : Am + t * LDA + i) = v;
      }
    }
  }
  __syncthreads();
  if (tid < GC) {                          // the 16 x 16 blocks on the diagonal: column j of the block from row o
    const int o = tid & ~15, j = tid & 15;
    float x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const float* row = Am + (o + t) * LDA + o;
      float a0 = (t == j) ? 1.f : 0.f, a1 = 0.f;
#pragma unroll
      for (int i = 0; i < t; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(row + i);
        a0 = fmaf(-v.x, x[i], a0);
        if (i + 1 < t) a1 = fmaf(-v.y, x[i + 1], a1);
        if (i + 2 < t) a0 = fmaf(-v.z, x[i + 2], a0);
        if (i + 3 < t) a1 = fmaf(-v.w, x[i + 3], a1);
      }
      x[t] = a0 + a1;
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) Tm[(o + t) * LDA + o + j] = x[t];
  } else if (tid < 2 * GC) {               // and zeros beside the first and third of them
    const int r = (tid & 15) + (tid & 32), c = (tid & 16) / 2 + (tid & 32) + 16;
    *reinterpret_cast<float4*>(Tm + r * LDA + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(Tm + r * LDA + c + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  gc_merge<16, LDA>(Am, Tm, Xm);
  gc_merge<32, LDA>(Am, Tm, Xm);
  for (int i = tid; i < GC * GC / 4; i += GC_PREP_THREADS) {
    const int t = i / (GC / 4), c = i % (GC / 4) * 4;
    if (c > (t | 15)) continue;
    const float4 v = *reinterpret_cast<const float4*>(Tm + t * LDA + c);
    *reinterpret_cast<float4*>(gT + t * GC + c) = make_float4(c <= t ? v.x * bs[c] : 0.f, c + 1 <= t ? v.y * bs[c + 1] : 0.f,
                                                              c + 2 <= t ? v.z * bs[c + 2] : 0.f, c + 3 <= t ? v.w * bs[c + 3] : 0.f);
  }
}

// ---- scan ------------------------------------------------------------------------------------------------
// grid (DV / (16 MT), nv, nseg); twelve warps: four walk the chain U, D, S, four others make the outputs beside them (R while U runs, P D while S
// does), four load. Everything is held transposed: the M side of the m16n8k16 products is the slice's columns, the N side the chunk's rows (a warp has
// rows 8 w .. and 56 - 8 w .., which evens out the triangular products) or the state's (32 a warp). A warp's results then come out as
// pairs along the next product's summed index, and the state stays in the warps' registers as 32-bit sums.
// Bound by latency and shared memory: a chunk takes 4,500 cycles, of which the tensor cores need 1,700 and shared memory 2,300. (One group of
// four warps doing all of it in turn, the loads too: 6,500.)
constexpr int GC_SCAN_THREADS = 384;

template <int DK, int MT>
struct GcScan {
  static constexpr int W = 16 * MT, LDK = DK + 8, LDT = GC + 8, LDB = GC + 8, LDV = W + 8;
  static constexpr int K = 0, Q = K + GC * LDK * 2, T = Q + GC * LDK * 2, P = T + GC * LDT * 4, V = P + GC * LDT * 4, C = V + GC * LDV * 2;
  static constexpr int STAGE = C + GC_VEC * 4;
  static constexpr int S = 2 * STAGE, B = S + 3 * W * LDK * 2, D = B + 3 * W * LDB * 2, E = D + 3 * W * LDB * 2, TOTAL = E + 3 * W * LDB * 2;
};
template <int ID, int N> __device__ __forceinline__ void gc_bar() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory"); }

// Rows of the slice's columns times K or Q: x[0] leading, [1] and [2] other terms. A: three terms of [16 MT][LDK] (the state), B: [GC][LDK].
template <int DK, int MT, int LDK>
__device__ __forceinline__ void gc_rows(float (&x)[3][MT][2][4], const __nv_bfloat16* A, const __nv_bfloat16* B, int w) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 3 * MT * 2 * 4; ++i) (&x[0][0][0][0])[i] = 0.f;
  const __nv_bfloat16* b = B + ((lane >> 4 ? 7 - w : w) * 8 + (lane & 7)) * LDK + ((lane >> 3) & 1) * 8;
  const __nv_bfloat16* a = A + (lane & 15) * LDK + (lane >> 4) * 8;
#pragma unroll
  for (int k = 0; k < DK; k += 16) {
    uint32_t kb[4];
    gc_ldsm(kb, b + k);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        uint32_t f[4];
        gc_ldsm(f, a + (i * MT + m) * 16 * LDK + k);
        gc_mma(x[i][m][0], f, kb[0], kb[1]);
        gc_mma(x[i][m][1], f, kb[2], kb[3]);
      }
  }
}

// out = A M^T for the warp's two tiles of 8 rows of M (32-bit, lower triangular, [GC][LDT]; first w, then 7 - w). A: three terms of [16 MT][LDB]. The
// later tile needs 16-wide steps 0 .. 2 and for w < 2 also 3, the first 0 and for w >= 2 also 1: four fixed steps and a fifth, without branches. A tile on
// an even place ends in the middle of its last step; A's other half is zero there, since M's zeros would let no numbers through (the first row's padding of
// A holds these zeros). That takes 4 of 124 us of 1500 rows of 32 heads; multiplying 8 wide instead 26.
template <int MT, int LDT, int LDB>
__device__ __forceinline__ void gc_triangle(float (&out)[MT][2][4], const __nv_bfloat16* A, const float* M, int w) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  float x[3][3][MT][4];                    // [first, later, fifth step][sizes of products]
#pragma unroll
  for (int i = 0; i < 9 * MT * 4; ++i) (&x[0][0][0][0])[i] = 0.f;
  auto step = [&](float (&acc)[3][MT][4], const uint32_t (&a)[MT][3][4], int tile, int ks) {
    const float* row = M + (tile * 8 + g) * LDT + ks * 16 + 2 * t4;
    const float2 u = *reinterpret_cast<const float2*>(row), v = *reinterpret_cast<const float2*>(row + 8);
    uint32_t b0[3], b1[3];
    gc_split(u.x, u.y, b0);
    gc_split(v.x, v.y, b1);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      gc_mma(acc[0][m], a[m][0], b0[0], b1[0]);
      gc_mma(acc[1][m], a[m][0], b0[1], b1[1]);
      gc_mma(acc[2][m], a[m][1], b0[1], b1[1]);
      gc_mma(acc[1][m], a[m][1], b0[0], b1[0]);
      gc_mma(acc[2][m], a[m][0], b0[2], b1[2]);
      gc_mma(acc[2][m], a[m][2], b0[0], b1[0]);
    }
  };
  auto load = [&](uint32_t (&a)[MT][3][4], int ks, bool half) {
    const bool zero = half && lane >= 16;  // (the lanes that say where the other half's rows lie)
    const __nv_bfloat16* p = zero ? A + GC : A + (lane & 15) * LDB + ks * 16 + (lane >> 4) * 8;
    const int next = zero ? 0 : 16 * LDB;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i) gc_ldsm(a[m][i], p + (i * MT + m) * next);
  };
  const bool late = w < 2;
#pragma unroll
  for (int ks = 0; ks < 3; ++ks) {
    uint32_t a[MT][3][4];
    load(a, ks, ks == 2 && w == 3);
    step(x[1], a, 7 - w, ks);
    if (ks > 0) continue;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i) { a[m][i][2] = w ? a[m][i][2] : 0u; a[m][i][3] = w ? a[m][i][3] : 0u; }
    step(x[0], a, w, 0);
  }
  uint32_t a[MT][3][4];
  load(a, late ? 3 : 1, w == 1 || w == 2);
  step(x[2], a, late ? 7 - w : w, late ? 3 : 1);
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float f = x[2][0][m][e] + (x[2][1][m][e] + x[2][2][m][e]);
      out[m][0][e] = x[0][0][m][e] + (x[0][1][m][e] + x[0][2][m][e]) + (late ? 0.f : f);
      out[m][1][e] = x[1][0][m][e] + (x[1][1][m][e] + x[1][2][m][e]) + (late ? f : 0.f);
    }
}

template <int DK, int MT>
__global__ void __launch_bounds__(GC_SCAN_THREADS, 1)
gdn_chunk_scan_kernel(float* __restrict__ y, float* __restrict__ rec_state, __nv_bfloat16* __restrict__ conv_state,
                      const float* scratch, const __nv_bfloat16* qkv, const __nv_bfloat16* proj, long proj_stride, const int* seg_slot,
                      const int* seg_row0, const int* seg_nrows, int nk, int nv, int dv, int commit) {
  using L = GcScan<DK, MT>;
  constexpr int W = L::W, CK = 4, LDK = L::LDK, LDT = L::LDT, LDB = L::LDB, LDV = L::LDV;
  static_assert(DK == 128, "four warps cover the state's rows, 32 each");
  extern __shared__ __align__(16) unsigned char sm_scan[];
  __nv_bfloat16* Ss = reinterpret_cast<__nv_bfloat16*>(sm_scan + L::S);      // [3][W][LDK] state, by column
  __nv_bfloat16* Bs = reinterpret_cast<__nv_bfloat16*>(sm_scan + L::B);      // [3][W][LDB] right-hand side
  __nv_bfloat16* Ds = reinterpret_cast<__nv_bfloat16*>(sm_scan + L::D);      // [3][W][LDB] deltas
  __nv_bfloat16* Es = reinterpret_cast<__nv_bfloat16*>(sm_scan + L::E);      // [3][W][LDB] deltas times e^{c_C - c_i} / |k_i|
  const int slice = blockIdx.x, h = blockIdx.y, seg = blockIdx.z;
  const int tid = threadIdx.x, role = tid >> 7, warp = (tid >> 5) & 3, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  pdl_wait();                              // the prep kernel's records (and everything before it on the stream)
  scratch = after_wait(scratch);
  qkv = after_wait(qkv);
  const int n = after_wait(seg_nrows)[seg];
  if (n <= 0) return;
  const int row0 = after_wait(seg_row0)[seg], slot = after_wait(seg_slot)[seg];
  const int kh = h / (nv / nk);
  const int conv_dim = 2 * nk * DK + nv * dv;
  const int q_off = kh * DK, k_off = nk * DK + kh * DK, v_off = 2 * nk * DK + h * dv + slice * W;
  float* Sg = rec_state + (((size_t)slot * nv + h) * DK) * dv + slice * W;
  const int nchunks = (n + GC - 1) / GC;
  if (tid < 2) *reinterpret_cast<uint4*>((tid ? Ds : Bs) + GC) = make_uint4(0u, 0u, 0u, 0u);      // see gc_triangle

  if (role == 2) {                         // loads, a chunk ahead
    const int u = tid & 127;
    const size_t rec_stride = (size_t)nv * gc_rec_floats();
    const float* rec0 = scratch + ((size_t)(row0 / GC + seg) * nv + h) * gc_rec_floats();
    for (int ch = 0; ch < nchunks; ++ch) {
      unsigned char* st = sm_scan + (ch & 1) * L::STAGE;
      const __nv_bfloat16* src = qkv + (size_t)(row0 + ch * GC) * conv_dim;
      const int valid = min(GC, n - ch * GC);
      for (int i = u; i < GC * (DK / 8); i += 128) {
        const int t = i / (DK / 8), c = i % (DK / 8) * 8;
        const __nv_bfloat16* row = src + (size_t)(t < valid ? t : 0) * conv_dim + c;
        gc_cp16(st + L::K + (t * LDK + c) * 2, row + k_off, t < valid);
        gc_cp16(st + L::Q + (t * LDK + c) * 2, row + q_off, t < valid);
      }
      const float* rec = rec0 + (size_t)ch * rec_stride;
      for (int i = u; i < GC * (GC / 4); i += 128) {
        const int t = i / (GC / 4), c = i % (GC / 4) * 4;
        if (c > (t | 15)) continue;
        gc_cp16(st + L::T + (t * LDT + c) * 4, rec + t * GC + c);
        gc_cp16(st + L::P + (t * LDT + c) * 4, rec + GC * GC + t * GC + c);
      }
      for (int i = u; i < GC * (W / 8); i += 128) {
        const int t = i / (W / 8), c = i % (W / 8) * 8;
        gc_cp16(st + L::V + (t * LDV + c) * 2, src + (size_t)(t < valid ? t : 0) * conv_dim + v_off + c, t < valid);
      }
      if (u < GC_VEC / 4) gc_cp16(st + L::C + u * 16, rec + 2 * GC * GC + u * 4);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();                     // chunk `ch` is there; nobody reads the other stage any more
    }
    pdl_launch_dependents();
    if (commit && slice == 0) {
      // conv tail: the last CK-1 raw inputs of the channels this head owns (q/k channels: first head of the group)
      const int vh_off = 2 * nk * DK + h * dv;
      __nv_bfloat16* cst = conv_state + (size_t)slot * (CK - 1) * conv_dim;
      const bool own_qk = (h % (nv / nk)) == 0;
      const int nch = dv + (own_qk ? 2 * DK : 0);
      proj = after_wait(proj);
      for (int idx = u; idx < nch; idx += 128) {
        const int c = idx < dv ? vh_off + idx : (idx < dv + DK ? q_off + (idx - dv) : k_off + (idx - dv - DK));
        __nv_bfloat16 nw[CK - 1];
#pragma unroll
        for (int j = 0; j < CK - 1; ++j) {
          const int tt = n - (CK - 1) + j;
          nw[j] = tt >= 0 ? proj[(size_t)(row0 + tt) * proj_stride + c] : cst[(size_t)(CK - 1 + tt) * conv_dim + c];
        }
#pragma unroll
        for (int j = 0; j < CK - 1; ++j) cst[(size_t)j * conv_dim + c] = nw[j];
      }
    }
    return;
  }
  auto tile = [&](int j) { return j ? 7 - warp : warp; };
  if (role == 1) {                         // Y = e^{c} Q S0 + P D
    for (int ch = 0; ch < nchunks; ++ch) {
      const unsigned char* st = sm_scan + (ch & 1) * L::STAGE;
      const float* cs = reinterpret_cast<const float*>(st + L::C);
      const int valid = min(GC, n - ch * GC);
      __syncthreads();
      float r[3][MT][2][4], d[MT][2][4];
      gc_rows<DK, MT, LDK>(r, Ss, reinterpret_cast<const __nv_bfloat16*>(st + L::Q), warp);
      gc_bar<2, 256>();                    // the deltas are there, the state's terms free
      gc_triangle<MT, LDT, LDB>(d, Ds, reinterpret_cast<const float*>(st + L::P), warp);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = tile(j) * 8 + 2 * t4 + (e & 1);
          const float f = cs[GC + t];
          if (t < valid) {
            float* to = y + ((size_t)(row0 + ch * GC + t) * nv + h) * dv + slice * W + g + (e >> 1) * 8;
#pragma unroll
            for (int m = 0; m < MT; ++m) to[m * 16] = fmaf(f, r[0][m][j][e] + (r[1][m][j][e] + r[2][m][j][e]), d[m][j][e]);
          }
        }
    }
    return;
  }

  float S[MT][4][4];                       // [m][tile][e]: columns m 16 + g (e < 2) and + 8, state rows warp 32 + tile 8 + 2 t4 + (e & 1)
  auto sg = [&](int m, int j, int e) { return Sg + (size_t)(warp * 32 + j * 8 + 2 * t4 + (e & 1)) * dv + m * 16 + g + (e >> 1) * 8; };
  auto store_terms = [&](__nv_bfloat16* to, int ld, int m, int at, float x0, float x1, float x2, float x3) {
    uint32_t a[3], b[3];
    gc_split(x0, x1, a);
    gc_split(x2, x3, b);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      __nv_bfloat16* p = to + ((i * MT + m) * 16 + g) * ld + at;
      *reinterpret_cast<uint32_t*>(p) = a[i];
      *reinterpret_cast<uint32_t*>(p + 8 * ld) = b[i];
    }
  };
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) S[m][j][e] = *sg(m, j, e);
      store_terms(Ss, LDK, m, warp * 32 + j * 8 + 2 * t4, S[m][j][0], S[m][j][1], S[m][j][2], S[m][j][3]);
    }
  for (int ch = 0; ch < nchunks; ++ch) {
    const unsigned char* st = sm_scan + (ch & 1) * L::STAGE;
    const __nv_bfloat16* Ks = reinterpret_cast<const __nv_bfloat16*>(st + L::K);
    const __nv_bfloat16* Vs = reinterpret_cast<const __nv_bfloat16*>(st + L::V);
    const float* cs = reinterpret_cast<const float*>(st + L::C);
    __syncthreads();                       // chunk `ch` and the state's terms are there
    {                                      // B = V - e^{c} K S0
      float u[3][MT][2][4];
      gc_rows<DK, MT, LDK>(u, Ss, Ks, warp);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = tile(j) * 8 + 2 * t4;
        const float2 f = *reinterpret_cast<const float2*>(cs + t);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          float b[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            b[e] = fmaf(-(e & 1 ? f.y : f.x), u[0][m][j][e] + (u[1][m][j][e] + u[2][m][j][e]),
                        bf2f(Vs[(t + (e & 1)) * LDV + m * 16 + g + (e >> 1) * 8]));
          store_terms(Bs, LDB, m, t, b[0], b[1], b[2], b[3]);
        }
      }
    }
    gc_bar<1, 128>();
    {                                      // D = T' B
      float d[MT][2][4];
      gc_triangle<MT, LDT, LDB>(d, Bs, reinterpret_cast<const float*>(st + L::T), warp);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = tile(j) * 8 + 2 * t4;
        const float2 tail = *reinterpret_cast<const float2*>(cs + 2 * GC + t);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float(&v)[4] = d[m][j];
          store_terms(Ds, LDB, m, t, v[0], v[1], v[2], v[3]);
          store_terms(Es, LDB, m, t, v[0] * tail.x, v[1] * tail.y, v[2] * tail.x, v[3] * tail.y);
        }
      }
    }
    gc_bar<2, 256>();
    {                                      // S = e^{c_C} S0 + K^T D'
      float s[3][MT][4][4];
#pragma unroll
      for (int i = 0; i < 3 * MT * 4 * 4; ++i) (&s[0][0][0][0])[i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < GC / 16; ++ks) {
        uint32_t kb[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
          gc_ldsm_t(kb[j], Ks + (ks * 16 + (lane & 15)) * LDK + warp * 32 + j * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            uint32_t a[4];
            gc_ldsm(a, Es + ((i * MT + m) * 16 + (lane & 15)) * LDB + ks * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int j = 0; j < 4; ++j) gc_mma(s[i][m][j], a, kb[j >> 1][(j & 1) * 2], kb[j >> 1][(j & 1) * 2 + 1]);
          }
      }
      const float eC = cs[3 * GC];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int e = 0; e < 4; ++e) S[m][j][e] = fmaf(eC, S[m][j][e], s[0][m][j][e] + (s[1][m][j][e] + s[2][m][j][e]));
          store_terms(Ss, LDK, m, warp * 32 + j * 8 + 2 * t4, S[m][j][0], S[m][j][1], S[m][j][2], S[m][j][3]);
        }
    }
  }
  if (commit) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) *sg(m, j, e) = S[m][j][e];
  }
}

template <int DK, int MT>
static cudaError_t launch_scan(float* y, float* rec_state, void* conv_state, const float* scratch, const void* qkv, const void* proj,
                               long proj_stride, const int* seg_slot, const int* seg_row0, const int* seg_nrows, int nseg, int nk, int nv, int dv,
                               int commit, cudaStream_t s) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(gdn_chunk_scan_kernel<DK, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, GcScan<DK, MT>::TOTAL);
  if (attr != cudaSuccess) return attr;
  return launch_pdl(gdn_chunk_scan_kernel<DK, MT>, dim3(dv / (16 * MT), nv, nseg), dim3(GC_SCAN_THREADS), (size_t)GcScan<DK, MT>::TOTAL, s, y,
                    rec_state, (__nv_bfloat16*)conv_state, scratch, (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)proj, proj_stride, seg_slot,
                    seg_row0, seg_nrows, nk, nv, dv, commit);
}

template <int DK>
static int launch_chunk(float* y, float* rec_state, void* conv_state, float* scratch, const void* qkv, const void* proj,
                        long proj_stride, const float* A_log, const float* dt_bias, const int* seg_slot,
                        const int* seg_row0, const int* seg_nrows, int nseg, int max_rows, int nk, int nv, int dv,
                        float eps, int commit, cudaStream_t s) {
  constexpr size_t prep_smem = (size_t)2 * GC * (DK + 8) * 2 + (size_t)2 * GC * (GC + 4) * 4;
  static const cudaError_t attr = cudaFuncSetAttribute(gdn_chunk_prep_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep_smem);
  if (attr != cudaSuccess) return (int)attr;
  const int max_chunks = (max_rows + GC - 1) / GC;
  cudaError_t e = launch_pdl(gdn_chunk_prep_kernel<DK>, dim3(max_chunks, nv, nseg), dim3(GC_PREP_THREADS), prep_smem, s, scratch,
                             (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)proj, proj_stride, A_log, dt_bias, seg_row0,
                             seg_nrows, nk, nv, dv, eps);
  if (e != cudaSuccess) return (int)e;
  // An SM holds one CTA: slices of 16 columns while they fit one wave. (A chunk of slices of 32 takes 1.4 times one of 16: 98 us for 24 chunks
  // against 83 for 32.)
  const bool wide = dv % 32 == 0 && (long)(dv / 16) * nv * nseg > 148;
  return (int)(wide ? launch_scan<DK, 2> : launch_scan<DK, 1>)(y, rec_state, conv_state, scratch, qkv, proj, proj_stride, seg_slot, seg_row0, seg_nrows,
                                                               nseg, nk, nv, dv, commit, s);
}

}  // namespace fb

using namespace fb;

extern "C" long fb_gdn_chunk_scratch_bytes(int rows, int nseg, int nv, int dk) {
  return ((long)rows / GC + nseg + 1) * nv * gc_rec_floats() * (long)sizeof(float);
}

extern "C" int fb_gdn_chunk(float* y, float* rec_state, void* conv_state, float* scratch, const void* qkv,
                            const void* proj, long proj_stride, const float* A_log, const float* dt_bias,
                            const int* seg_slot, const int* seg_row0, const int* seg_nrows, int nseg, int max_rows,
                            int nk, int nv, int dk, int dv, float eps, int commit, cudaStream_t s) {
  if (nseg <= 0 || max_rows <= 0) return 0;
  if (nv % nk || dv % 16 || !scratch) return -1;
  if (dk == 128)
    return launch_chunk<128>(y, rec_state, conv_state, scratch, qkv, proj, proj_stride, A_log, dt_bias, seg_slot, seg_row0,
                             seg_nrows, nseg, max_rows, nk, nv, dv, eps, commit, s);
  return -2;
}
