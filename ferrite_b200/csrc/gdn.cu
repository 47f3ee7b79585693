// Gated DeltaNet: causal depthwise conv1d + SiLU, and the gated delta-rule recurrence
//   S = S * g;  delta = (v - S^T k) * beta;  S += k (x) delta;  y = S^T q
// with q, k L2-normalised per head (q also scaled by 1/sqrt(dk)), g = exp(-exp(A_log) * softplus(a + dt_bias)),
// beta = sigmoid(b). State S is fp32 [slot][head][dk][dv].
//
// Counterparts in the reference: `fe_gdn_conv` (`kernels/k-core/src/gdn.rs:30`), `fe_gdn_rec` / `fe_gdn_rec2`
// (`:117`, `:241`) and, through the `commit` flag and saved projections, `fe_gdn_replay` (`:260`).
// The conv kernel never writes state; the recurrence kernel (which runs after it on the stream) commits both
// the recurrent state and the conv tail, so no CTA reads state another CTA of the same launch writes.
#include "api.h"
#include "common.cuh"
#include "gdn_step.cuh"

namespace fb {

constexpr int STEP_CTAS = 148;    // SMs
constexpr int STEP_ROWS = 32;     // rows of a segment that the kernel for several rows prepares at once

__device__ __forceinline__ void st_cluster_f32(float* own, uint32_t rank, float v) {      // the same place in the shared memory of CTA `rank`
  asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %0, %1;\nst.shared::cluster.f32 [a], %2;\n}" ::"r"(smem_u32(own)), "r"(rank), "f"(v)
               : "memory");
}

// proj row layout: [q (nk*dk) | k (nk*dk) | v (nv*dv) | z (nv*dv) | b (nv) | a (nv)]
// conv_state: [slot][conv_k-1][conv_dim] bf16, oldest input first.
// grid = (ceil(conv_dim/256), row chunks of 32, segments)
__global__ void gdn_conv_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ proj,
                                long proj_stride, const __nv_bfloat16* __restrict__ conv_w,
                                const __nv_bfloat16* __restrict__ conv_state, const int* __restrict__ seg_slot,
                                const int* __restrict__ seg_row0, const int* __restrict__ seg_nrows, int conv_dim) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int CK = 4, CHUNK = 32;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int seg = blockIdx.z;
  const int n = seg_nrows[seg];
  const int r0 = blockIdx.y * CHUNK;
  if (c >= conv_dim || r0 >= n) return;
  const int row0 = seg_row0[seg];
  const int slot = seg_slot[seg];
  float w[CK];
#pragma unroll
  for (int j = 0; j < CK; ++j) w[j] = bf2f(conv_w[(size_t)c * CK + j]);
  const __nv_bfloat16* st = conv_state + (size_t)slot * (CK - 1) * conv_dim + c;
  float win[CK - 1];
#pragma unroll
  for (int j = 0; j < CK - 1; ++j) {
    int r = r0 - (CK - 1) + j;                      // time index relative to the segment start
    win[j] = r >= 0 ? bf2f(proj[(size_t)(row0 + r) * proj_stride + c]) : bf2f(st[(size_t)(CK - 1 + r) * conv_dim]);
  }
  const int rend = min(n, r0 + CHUNK);
  for (int r = r0; r < rend; ++r) {
    float x = bf2f(proj[(size_t)(row0 + r) * proj_stride + c]);
    float acc = w[0] * win[0] + w[1] * win[1] + w[2] * win[2] + w[3] * x;
    out[(size_t)(row0 + r) * conv_dim + c] = f2bf(siluf_(acc));
    win[0] = win[1]; win[1] = win[2]; win[2] = x;
  }
}

// Verify-tree form of the conv: the window of a row is its three nearest ancestors (then the slot's conv tail), found
// by walking `row_parent` (parent row inside the segment, -1 for the root row). Counterpart of the tree variant of
// `fe_gdn_conv` (`kernels/k-core/src/gdn.rs:30`). grid = (ceil(conv_dim/256), segments); never writes state.
__global__ void gdn_conv_tree_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ proj,
                                     long proj_stride, const __nv_bfloat16* __restrict__ conv_w,
                                     const __nv_bfloat16* __restrict__ conv_state, const int* __restrict__ seg_slot,
                                     const int* __restrict__ seg_row0, const int* __restrict__ seg_nrows,
                                     const int* __restrict__ row_parent, int conv_dim) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int CK = 4;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int seg = blockIdx.y;
  const int n = seg_nrows[seg];
  if (c >= conv_dim || n <= 0) return;
  const int row0 = seg_row0[seg];
  const int slot = seg_slot[seg];
  float w[CK];
#pragma unroll
  for (int j = 0; j < CK; ++j) w[j] = bf2f(conv_w[(size_t)c * CK + j]);
  const __nv_bfloat16* st = conv_state + (size_t)slot * (CK - 1) * conv_dim + c;
  for (int r = 0; r < n; ++r) {
    float acc = w[CK - 1] * bf2f(proj[(size_t)(row0 + r) * proj_stride + c]);
    int i = r;
#pragma unroll
    for (int j = CK - 2; j >= 0; --j) {
      // one step back in time: the parent row, or (past the root) one entry further into the saved tail
      i = i >= 0 ? row_parent[row0 + i] : i - 1;
      if (i >= n) i = -1;                                    // malformed parent: treat as the root's predecessor
      const float x = i >= 0 ? bf2f(proj[(size_t)(row0 + i) * proj_stride + c]) : bf2f(st[(size_t)(CK - 1 + i) * conv_dim]);
      acc = fmaf(w[j], x, acc);
    }
    out[(size_t)(row0 + r) * conv_dim + c] = f2bf(siluf_(acc));
  }
}

// Recurrence over the rows of one segment for one value head. blockDim = DV * 8; thread (col = tid % DV,
// part = tid / DV) keeps DK/8 rows of state column `col` in registers across the whole segment.
// TREE: the rows of a segment form a verify tree. A row starts from the state its parent left (`row_parent`, -1 = the
// slot's committed state); states are parked in `node_state` [row][head][DK][DV] only where `row_flags` asks for it
// (bit 0: this row's parent is not the previous row, reload; bit 1: a later row branches from this one, store). A
// thread reloads exactly the elements it stored, so no barrier is needed. Tree launches never commit. Counterpart of
// the tree variant of `fe_gdn_rec` (`kernels/k-core/src/gdn.rs:117`).
template <int DK, int DV, bool TREE>
__global__ void __launch_bounds__(DV * 8)
gdn_rec_kernel(float* __restrict__ y, float* __restrict__ rec_state, __nv_bfloat16* __restrict__ conv_state,
               const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ proj, long proj_stride,
               const float* __restrict__ A_log, const float* __restrict__ dt_bias, const int* __restrict__ seg_slot,
               const int* __restrict__ seg_row0, const int* __restrict__ seg_nrows, int nk, int nv, float eps,
               int commit, const int* __restrict__ row_parent, const int* __restrict__ row_flags,
               float* __restrict__ node_state) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PARTS = 8, RP = DK / PARTS, CK = 4;
  __shared__ float qs[DK], ks[DK], vs[DV];
  __shared__ float red1[PARTS][DV], red2[PARTS][DV];
  __shared__ float ssq[2][DK / 32];
  const int h = blockIdx.x, seg = blockIdx.y;
  const int tid = threadIdx.x, col = tid % DV, part = tid / DV;
  const int n = seg_nrows[seg];
  if (n <= 0) return;
  const int row0 = seg_row0[seg], slot = seg_slot[seg];
  const int kh = h / (nv / nk);
  const int conv_dim = 2 * nk * DK + nv * DV;
  const int q_off = kh * DK, k_off = nk * DK + kh * DK, v_off = 2 * nk * DK + h * DV;
  const int b_off = conv_dim + nv * DV + h, a_off = b_off + nv;
  float* Sg = rec_state + (((size_t)slot * nv + h) * DK) * DV;
  float S[RP];
#pragma unroll
  for (int i = 0; i < RP; ++i) S[i] = Sg[(size_t)(part * RP + i) * DV + col];
  const float expA = __expf(A_log[h]);
  const float dtb = dt_bias[h];
  const float qscale = rsqrtf((float)DK);

  for (int r = 0; r < n; ++r) {
    int flags = 0;
    if (TREE) {
      flags = row_flags[row0 + r];
      if (flags & 1) {
        const int par = row_parent[row0 + r];
        const float* src = (par < 0 || par >= r) ? Sg : node_state + (((size_t)(row0 + par) * nv + h) * DK) * DV;
#pragma unroll
        for (int i = 0; i < RP; ++i) S[i] = src[(size_t)(part * RP + i) * DV + col];
      }
    }
    const __nv_bfloat16* xr = qkv + (size_t)(row0 + r) * conv_dim;
    if (tid < DK) {
      float qv = bf2f(xr[q_off + tid]), kv = bf2f(xr[k_off + tid]);
      qs[tid] = qv; ks[tid] = kv;
      float sq = warp_sum(qv * qv), sk = warp_sum(kv * kv);
      if ((tid & 31) == 0) { ssq[0][tid >> 5] = sq; ssq[1][tid >> 5] = sk; }
    }
    if (tid < DV) vs[tid] = bf2f(xr[v_off + tid]);
    __syncthreads();
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int i = 0; i < DK / 32; ++i) { sq += ssq[0][i]; sk += ssq[1][i]; }
    const float rq = rsqrtf(sq + eps) * qscale, rk = rsqrtf(sk + eps);
    const __nv_bfloat16* pr = proj + (size_t)(row0 + r) * proj_stride;
    const float beta = sigmoidf_(bf2f(pr[b_off]));
    const float g = __expf(-expA * softplusf_(bf2f(pr[a_off]) + dtb));
    float p = 0.f;
#pragma unroll
    for (int i = 0; i < RP; ++i) p = fmaf(S[i], ks[part * RP + i], p);
    red1[part][col] = p;
    __syncthreads();
    float kvv = 0.f;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) kvv += red1[i][col];
    kvv *= g * rk;
    const float delta = (vs[col] - kvv) * beta;
    float yp = 0.f;
#pragma unroll
    for (int i = 0; i < RP; ++i) {
      S[i] = fmaf(ks[part * RP + i] * rk, delta, S[i] * g);
      yp = fmaf(S[i], qs[part * RP + i], yp);
    }
    red2[part][col] = yp;
    __syncthreads();
    if (part == 0) {
      float yy = 0.f;
#pragma unroll
      for (int i = 0; i < PARTS; ++i) yy += red2[i][col];
      y[((size_t)(row0 + r) * nv + h) * DV + col] = yy * rq;
    }
    if (TREE && (flags & 2)) {
      float* dst = node_state + (((size_t)(row0 + r) * nv + h) * DK) * DV;
#pragma unroll
      for (int i = 0; i < RP; ++i) dst[(size_t)(part * RP + i) * DV + col] = S[i];
    }
  }
  if (commit && !TREE) {
#pragma unroll
    for (int i = 0; i < RP; ++i) Sg[(size_t)(part * RP + i) * DV + col] = S[i];
    // conv tail: the last CK-1 raw inputs of the channels this head owns (q/k channels: first head of the group)
    __nv_bfloat16* st = conv_state + (size_t)slot * (CK - 1) * conv_dim;
    const bool own_qk = (h % (nv / nk)) == 0;
    const int nch = DV + (own_qk ? 2 * DK : 0);
    for (int idx = tid; idx < nch; idx += blockDim.x) {
      int c = idx < DV ? v_off + idx : (idx < DV + DK ? q_off + (idx - DV) : k_off + (idx - DV - DK));
      __nv_bfloat16 nw[CK - 1];
#pragma unroll
      for (int j = 0; j < CK - 1; ++j) {
        int t = n - (CK - 1) + j;
        nw[j] = t >= 0 ? proj[(size_t)(row0 + t) * proj_stride + c] : st[(size_t)(CK - 1 + t) * conv_dim + c];
      }
#pragma unroll
      for (int j = 0; j < CK - 1; ++j) st[(size_t)j * conv_dim + c] = nw[j];
    }
  }
}

// The decode-row fusion of the three kernels above lives in gdn_step.cuh (also used by the persistent decode-layer kernel).
// PER_SM: CTAs an SM holds. One is faster by itself (its loads stay further ahead), two once there are more CTAs than SMs.
template <int DK, int DV, int PARTS, bool CLUSTER, int PER_SM>
__global__ void __launch_bounds__(DV * PARTS, PER_SM)
gdn_step_kernel(__nv_bfloat16* __restrict__ out, float* __restrict__ rec_state, __nv_bfloat16* __restrict__ conv_state,
                const __nv_bfloat16* __restrict__ proj, long proj_stride, const __nv_bfloat16* __restrict__ conv_w,
                const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                const __nv_bfloat16* __restrict__ gnorm_w, const int* __restrict__ seg_slot,
                const int* __restrict__ seg_row0, const int* __restrict__ seg_nrows, int nk, int nv, float eps,
                int commit) {
  pdl_launch_dependents();
  pdl_wait();
  const int seg = blockIdx.y;
  gdn_step_body<DK, DV, PARTS, CLUSTER>(out, rec_state, conv_state, proj, proj_stride, conv_w, A_log, dt_bias, gnorm_w,
                                        seg_nrows[seg], seg_row0[seg], seg_slot[seg], blockIdx.x, nk, nv, eps, commit);
}

// The same for segments of more than one row, bit for bit (a row's sums run in the same order), so that a drafted row equals the decoded one.
// Bound by latency: a row needs the state that the row before it left. So:
//   * a head's columns are cut over SPLIT CTAs of one cluster, which meet once per `rb` rows, for the norm's sum over all columns;
//   * the inputs of up to `rb` rows come in together (cp.async), and what does not depend on the state (convs, unit norms, decays) is done
//     for all of them at once, by all warps, ahead of the recurrence;
//   * the recurrence has no barrier: a lane holds DK / PARTS state rows of a column, the PARTS lanes of a column pass their sums by
//     shuffles, and the next row's product with the state runs in the same pass as this row's update.
// 17 rows of 16 heads, SM cycles: inputs 1,800, convs 3,700 (SiLU divisions), norms 2,000, recurrence 7,200 (420 a row: 16-byte shared-memory
// reads of q and k at four wavefronts each), gated norm 3,400, state and tail 900.
template <int DK, int DV, int PARTS, int SPLIT>
struct GdnRows {
  static constexpr int THREADS = 512, WARPS = THREADS / 32;
  static constexpr int COLS = DV / SPLIT, RP = DK / PARTS, LC = 32 / PARTS;      // LC: lanes of a warp that share their state rows
  static constexpr int REC_WARPS = COLS / LC;
  static constexpr int LP = RP + 4, LDK = PARTS * LP;      // rows of q / k: the PARTS lanes' 16-byte reads lie on banks of their own
  static constexpr int QG = DK / 32, VG = COLS / 32, NG = DV / 32;
  static constexpr int CH = 2 * DK + COLS, RAW = CH + COLS;                      // channels convolved; inputs of a row: q | k | v | z
  static constexpr int ROW = 2 * LDK + COLS + 4 + 2 * NG;                        // floats a row of the block
  static_assert(COLS % 32 == 0 && RP % 4 == 0 && REC_WARPS >= 1 && REC_WARPS <= WARPS, "");
  static constexpr size_t smem(int rb) { return (size_t)rb * ROW * 4 + (size_t)(rb + 3) * RAW * 2 + (size_t)CH * 8; }
};

__device__ __forceinline__ void step_cp16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

// grid (nv * SPLIT, segments); a cluster holds the slices of all heads of a key head, so that the conv tail, which all of them read, is
// rewritten behind a barrier. `proj`, its rows, `conv_w` and `conv_state` lie on 16 bytes (elsewhere the kernel for single rows takes over).
template <int DK, int DV, int PARTS, int SPLIT>
__global__ void __launch_bounds__(GdnRows<DK, DV, PARTS, SPLIT>::THREADS)
gdn_rows_kernel(__nv_bfloat16* __restrict__ out, float* __restrict__ rec_state, __nv_bfloat16* __restrict__ conv_state,
                const __nv_bfloat16* proj, long proj_stride, const __nv_bfloat16* __restrict__ conv_w, const float* __restrict__ A_log,
                const float* __restrict__ dt_bias, const __nv_bfloat16* __restrict__ gnorm_w, const int* seg_slot, const int* seg_row0,
                const int* seg_nrows, int nk, int nv, float eps, int commit, int rb, int cluster) {
  using G = GdnRows<DK, DV, PARTS, SPLIT>;
  constexpr int CK = 4, RP = G::RP, COLS = G::COLS, LDK = G::LDK, NG = G::NG, VG = G::VG, LC = G::LC, CH = G::CH, RAW = G::RAW;
  extern __shared__ __align__(16) float sm_rows[];
  float* qs = sm_rows;                     // [rb][LDK]   q after conv
  float* ks = qs + rb * LDK;               // [rb][LDK]   k after conv
  float* vs = ks + rb * LDK;               // [rb][COLS]  v, then y
  float4* cf = reinterpret_cast<float4*>(vs + rb * COLS);   // [rb] decay, beta, 1 / |k|, 1 / (|q| sqrt(dk))
  float* ssn = reinterpret_cast<float*>(cf + rb);           // [2][rb][NG] sums of y^2 over 32 columns each, by parity of the block
  __nv_bfloat16* raw = reinterpret_cast<__nv_bfloat16*>(ssn + 2 * rb * NG);      // [3 + rb][RAW] inputs from three rows before the block on
  __nv_bfloat16* taps = raw + (rb + 3) * RAW;               // [CH][CK]
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int seg = blockIdx.y, h = blockIdx.x / SPLIT, slice = blockIdx.x % SPLIT, kh = h / (nv / nk);
  const int conv_dim = 2 * nk * DK + nv * DV;
  const int q_off = kh * DK, k_off = nk * DK + kh * DK, v_off = 2 * nk * DK + h * DV + slice * COLS;
  const int z_off = conv_dim + h * DV + slice * COLS;
  const int b_off = conv_dim + nv * DV + h, a_off = b_off + nv;
  auto channel = [&](int c) { return c < DK ? q_off + c : (c < 2 * DK ? k_off + c - DK : (c < CH ? v_off + c - 2 * DK : z_off + c - CH)); };
  auto at = [&](int c) { return (c / RP) * G::LP + c % RP; };          // channel c inside a row of q / k
  if (tid * 16 < CH) prefetch_l2(conv_w + (size_t)CK * channel(tid * 16));       // 16 channels a line
  pdl_wait();
  const int n = after_wait(seg_nrows)[seg], row0 = after_wait(seg_row0)[seg], slot = after_wait(seg_slot)[seg];
  proj = after_wait(proj);
  if (n <= 0) return;                      // (every CTA of the cluster)
  cluster_arrive();                        // met ahead of the first store into another CTA's shared memory: by then that CTA has to run
  const __nv_bfloat16* prow = proj + (size_t)row0 * proj_stride;
  __nv_bfloat16* st = conv_state + (size_t)slot * (CK - 1) * conv_dim;
  const bool rec = warp < G::REC_WARPS;
  const int part = lane / LC, col = warp * LC + lane % LC;
  float* Sg = rec_state + ((size_t)slot * nv + h) * DK * DV + slice * COLS;
  for (int i = tid; i < DK; i += G::THREADS) prefetch_l2(Sg + (size_t)i * DV);
  Sg += (size_t)part * RP * DV + col;
  uint64_t S[RP / 2];                      // rows 2 i, 2 i + 1

  for (int b0 = 0; b0 < n; b0 += rb) {
    const int m = min(rb, n - b0);
    for (int i = tid; i < (m + CK - 1) * (RAW / 8); i += G::THREADS) {
      const int r = i / (RAW / 8), c = i % (RAW / 8) * 8, t = b0 + r - (CK - 1);     // before the segment's first row: the slot's tail
      if (t >= 0) step_cp16(raw + r * RAW + c, prow + (size_t)t * proj_stride + channel(c));
      else if (c < CH) step_cp16(raw + r * RAW + c, st + (size_t)(CK - 1 + t) * conv_dim + channel(c));
    }
    if (b0 == 0)
      for (int i = tid; i < CH / 2; i += G::THREADS) step_cp16(taps + i * 8, conv_w + (size_t)CK * channel(2 * i));
    if (warp == G::WARPS - 1 && lane < m) {
      const __nv_bfloat16* pr = prow + (size_t)(b0 + lane) * proj_stride;
      const float beta = sigmoidf_(bf2f(pr[b_off]));
      const float g = __expf(-__expf(A_log[h]) * softplusf_(bf2f(pr[a_off]) + dt_bias[h]));
      cf[lane] = make_float4(g, beta, 0.f, 0.f);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (rec && b0 == 0) {
#pragma unroll
      for (int i = 0; i < RP / 2; ++i) S[i] = f2_pack(Sg[(size_t)(2 * i) * DV], Sg[(size_t)(2 * i + 1) * DV]);
    }
    // convs: a thread takes two channels of a row
#pragma unroll 2
    for (int i = tid; i < m * (CH / 2); i += G::THREADS) {
      const int r = i / (CH / 2), c = i % (CH / 2) * 2;
      const uint4 tp = *reinterpret_cast<const uint4*>(taps + c * CK);
      const float2 w0 = bf2f2(tp.x), w1 = bf2f2(tp.y), w2 = bf2f2(tp.z), w3 = bf2f2(tp.w);      // taps 0, 1 | 2, 3 of c, then of c + 1
      const uint32_t* x = reinterpret_cast<const uint32_t*>(raw + r * RAW + c);
      const float2 a = bf2f2(x[0]), b = bf2f2(x[RAW / 2]), d = bf2f2(x[RAW]), e = bf2f2(x[RAW / 2 * 3]);
      const float2 y = make_float2(bf2f(f2bf(siluf_(w0.x * a.x + w0.y * b.x + w1.x * d.x + w1.y * e.x))),
                                   bf2f(f2bf(siluf_(w2.x * a.y + w2.y * b.y + w3.x * d.y + w3.y * e.y))));
      *reinterpret_cast<float2*>(c < DK ? qs + r * LDK + at(c) : (c < 2 * DK ? ks + r * LDK + at(c - DK) : vs + r * COLS + c - 2 * DK)) = y;
    }
    __syncthreads();
    // unit norms: a warp per row of q or k
    for (int i = warp; i < 2 * m; i += G::WARPS) {
      const float* row = i < m ? qs + i * LDK : ks + (i - m) * LDK;
      float v[G::QG], sq = 0.f;
#pragma unroll
      for (int j = 0; j < G::QG; ++j) { v[j] = row[at(j * 32 + lane)]; v[j] = warp_sum(v[j] * v[j]); }
#pragma unroll
      for (int j = 0; j < G::QG; ++j) sq += v[j];
      if (lane == 0) {
        if (i < m) cf[i].w = rsqrtf(sq + eps) * rsqrtf((float)DK);
        else cf[i - m].z = rsqrtf(sq + eps);
      }
    }
    __syncthreads();
    if (rec) {
      float p = 0.f;
      ulonglong2 k[RP / 4];                // this row's k
#pragma unroll
      for (int i = 0; i < RP / 4; ++i) {
        k[i] = *reinterpret_cast<const ulonglong2*>(ks + part * G::LP + 4 * i);
        const float2 k0 = f2_unpack(k[i].x), k1 = f2_unpack(k[i].y), a = f2_unpack(S[2 * i]), b = f2_unpack(S[2 * i + 1]);
        p = fmaf(b.y, k1.y, fmaf(b.x, k1.x, fmaf(a.y, k0.y, fmaf(a.x, k0.x, p))));
      }
      for (int r = 0; r < m; ++r) {
        const float4 co = cf[r];
        const uint64_t g2 = f2_pack(co.x, co.x), rk2 = f2_pack(co.z, co.z);
        float u = 0.f;
#pragma unroll
        for (int i = 0; i < PARTS; ++i) u += __shfl_sync(0xffffffffu, p, i * LC + lane % LC);
        const float d = fmaf(-u, co.x * co.z, vs[r * COLS + col]) * co.y;
        const uint64_t d2 = f2_pack(d, d);
        const float* q4 = qs + r * LDK + part * G::LP;
        const float* n4 = ks + min(r + 1, m - 1) * LDK + part * G::LP;       // the next row's (the last one's sums are dropped)
        float y = 0.f;
        p = 0.f;
#pragma unroll
        for (int i = 0; i < RP / 4; ++i) {
          const float4 qq = *reinterpret_cast<const float4*>(q4 + 4 * i);
          S[2 * i] = f2_fma(f2_mul(k[i].x, rk2), d2, f2_mul(S[2 * i], g2));
          S[2 * i + 1] = f2_fma(f2_mul(k[i].y, rk2), d2, f2_mul(S[2 * i + 1], g2));
          k[i] = *reinterpret_cast<const ulonglong2*>(n4 + 4 * i);
          const float2 n0 = f2_unpack(k[i].x), n1 = f2_unpack(k[i].y), a = f2_unpack(S[2 * i]), b = f2_unpack(S[2 * i + 1]);
          y = fmaf(b.y, qq.w, fmaf(b.x, qq.z, fmaf(a.y, qq.y, fmaf(a.x, qq.x, y))));
          p = fmaf(b.y, n1.y, fmaf(b.x, n1.x, fmaf(a.y, n0.y, fmaf(a.x, n0.x, p))));
        }
        u = 0.f;
#pragma unroll
        for (int i = 0; i < PARTS; ++i) u += __shfl_sync(0xffffffffu, y, i * LC + lane % LC);
        if (part == 0) vs[r * COLS + col] = u * co.w;        // (every lane of the column has read v: the shuffles lie between)
      }
    }
    __syncthreads();
    // gated norm over all of the head's columns
    if (b0 == 0) cluster_wait();
    float* sn = ssn + ((b0 / rb) & 1) * rb * NG;
    for (int i = warp; i < m * VG; i += G::WARPS) {
      const int r = i / VG, g = i % VG;
      const float yy = vs[r * COLS + g * 32 + lane];
      const float s2 = warp_sum(yy * yy);
      if (lane < SPLIT) st_cluster_f32(sn + r * NG + slice * VG + g, (int)blockIdx.x % cluster - slice + lane, s2);
    }
    cluster_arrive();
    cluster_wait();
    for (int i = warp; i < m * VG; i += G::WARPS) {
      const int r = i / VG, c = i % VG * 32 + lane;
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < NG; ++j) ss += sn[r * NG + j];
      const float rn = rsqrtf(ss / (float)DV + eps);
      out[((size_t)(row0 + b0 + r) * nv + h) * DV + slice * COLS + c] =
          f2bf(vs[r * COLS + c] * rn * bf2f(gnorm_w[slice * COLS + c]) * siluf_(bf2f(raw[(r + CK - 1) * RAW + CH + c])));
    }
    if (b0 + rb < n) {
      __syncthreads();                     // the next block's rows take the place of these
    } else if (commit) {
      // conv tail = the last CK - 1 inputs (q / k channels: first CTA of the group writes them)
      const int lo = slice == 0 && h % (nv / nk) == 0 ? 0 : 2 * DK;
      for (int i = tid; i < (CK - 1) * (CH - lo) / 8; i += G::THREADS) {
        const int j = i / ((CH - lo) / 8), c = lo + i % ((CH - lo) / 8) * 8;
        *reinterpret_cast<uint4*>(st + (size_t)j * conv_dim + channel(c)) = *reinterpret_cast<const uint4*>(raw + (m + j) * RAW + c);
      }
    }
  }
  if (commit && rec) {
#pragma unroll
    for (int i = 0; i < RP / 2; ++i) {
      const float2 a = f2_unpack(S[i]);
      Sg[(size_t)(2 * i) * DV] = a.x;
      Sg[(size_t)(2 * i + 1) * DV] = a.y;
    }
  }
}

// q / k tails of the heads that share a key head and are no cluster, behind the kernel in which all of them read the old ones.
// grid ((2 nk dk + 255) / 256, segments)
__global__ void __launch_bounds__(256) gdn_qk_tail_kernel(__nv_bfloat16* conv_state, const __nv_bfloat16* proj, long proj_stride, const int* seg_slot,
                                                          const int* seg_row0, const int* seg_nrows, int qk, int conv_dim) {
  pdl_launch_dependents();
  pdl_wait();
  const int c = blockIdx.x * 256 + threadIdx.x, n = after_wait(seg_nrows)[blockIdx.y];
  if (c >= qk || n <= 0) return;
  gdn_qk_tail(conv_state + (size_t)after_wait(seg_slot)[blockIdx.y] * 3 * conv_dim,
              after_wait(proj) + (size_t)after_wait(seg_row0)[blockIdx.y] * proj_stride, proj_stride, n, conv_dim, c);
}

}  // namespace fb

using namespace fb;

extern "C" int fb_gdn_conv(void* out, const void* proj, long proj_stride, const void* conv_w, const void* conv_state,
                           const int* seg_slot, const int* seg_row0, const int* seg_nrows, int nseg, int max_rows,
                           int conv_dim, cudaStream_t s) {
  if (nseg <= 0 || max_rows <= 0) return 0;
  dim3 grid((conv_dim + 255) / 256, (max_rows + 31) / 32, nseg);
  launch_pdl(gdn_conv_kernel, dim3(grid), dim3(256), (size_t)(0), s, (__nv_bfloat16*)out, (const __nv_bfloat16*)proj, proj_stride,
                                       (const __nv_bfloat16*)conv_w, (const __nv_bfloat16*)conv_state, seg_slot,
                                       seg_row0, seg_nrows, conv_dim);
  return (int)cudaGetLastError();
}

extern "C" int fb_gdn_rec(float* y, float* rec_state, void* conv_state, const void* qkv, const void* proj,
                          long proj_stride, const float* A_log, const float* dt_bias, const int* seg_slot,
                          const int* seg_row0, const int* seg_nrows, int nseg, int nk, int nv, int dk, int dv,
                          float eps, int commit, cudaStream_t s) {
  if (nseg <= 0) return 0;
  if (nv % nk) return -1;
  dim3 grid(nv, nseg);
  if (dk == 128 && dv == 128)
    launch_pdl(gdn_rec_kernel<128, 128, false>, dim3(grid), dim3(1024), (size_t)(0), s, y, rec_state, (__nv_bfloat16*)conv_state, (const __nv_bfloat16*)qkv,
        (const __nv_bfloat16*)proj, proj_stride, A_log, dt_bias, seg_slot, seg_row0, seg_nrows, nk, nv, eps, commit,
        (const int*)nullptr, (const int*)nullptr, (float*)nullptr);
  else if (dk == 64 && dv == 64)
    launch_pdl(gdn_rec_kernel<64, 64, false>, dim3(grid), dim3(512), (size_t)(0), s, y, rec_state, (__nv_bfloat16*)conv_state, (const __nv_bfloat16*)qkv,
        (const __nv_bfloat16*)proj, proj_stride, A_log, dt_bias, seg_slot, seg_row0, seg_nrows, nk, nv, eps, commit,
        (const int*)nullptr, (const int*)nullptr, (float*)nullptr);
  else return -2;
  return (int)cudaGetLastError();
}

// Verify trees: conv over ancestor windows, then the recurrence from each row's parent state. `node_state` holds
// rows x nv x dk x dv floats (rows = all rows of the step); nothing is committed.
extern "C" long fb_gdn_tree_scratch_bytes(int rows, int nv, int dk, int dv) {
  return (long)rows * nv * dk * dv * (long)sizeof(float);
}

extern "C" int fb_gdn_conv_tree(void* out, const void* proj, long proj_stride, const void* conv_w, const void* conv_state,
                                const int* seg_slot, const int* seg_row0, const int* seg_nrows, const int* row_parent,
                                int nseg, int conv_dim, cudaStream_t s) {
  if (nseg <= 0) return 0;
  dim3 grid((conv_dim + 255) / 256, nseg);
  launch_pdl(gdn_conv_tree_kernel, dim3(grid), dim3(256), (size_t)(0), s, (__nv_bfloat16*)out, (const __nv_bfloat16*)proj,
             proj_stride, (const __nv_bfloat16*)conv_w, (const __nv_bfloat16*)conv_state, seg_slot, seg_row0, seg_nrows,
             row_parent, conv_dim);
  return (int)cudaGetLastError();
}

extern "C" int fb_gdn_rec_tree(float* y, float* rec_state, const void* qkv, const void* proj, long proj_stride,
                               const float* A_log, const float* dt_bias, const int* seg_slot, const int* seg_row0,
                               const int* seg_nrows, const int* row_parent, const int* row_flags, float* node_state,
                               int nseg, int nk, int nv, int dk, int dv, float eps, cudaStream_t s) {
  if (nseg <= 0) return 0;
  if (nv % nk) return -1;
  if (!row_parent || !row_flags || !node_state) return -3;
  dim3 grid(nv, nseg);
  if (dk == 128 && dv == 128)
    launch_pdl(gdn_rec_kernel<128, 128, true>, dim3(grid), dim3(1024), (size_t)(0), s, y, rec_state, (__nv_bfloat16*)nullptr,
               (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)proj, proj_stride, A_log, dt_bias, seg_slot, seg_row0, seg_nrows,
               nk, nv, eps, 0, row_parent, row_flags, node_state);
  else if (dk == 64 && dv == 64)
    launch_pdl(gdn_rec_kernel<64, 64, true>, dim3(grid), dim3(512), (size_t)(0), s, y, rec_state, (__nv_bfloat16*)nullptr,
               (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)proj, proj_stride, A_log, dt_bias, seg_slot, seg_row0, seg_nrows,
               nk, nv, eps, 0, row_parent, row_flags, node_state);
  else return -2;
  return (int)cudaGetLastError();
}

template <int DK, int DV, int PARTS, int SPLIT>
static int launch_rows(void* out, float* rec_state, void* conv_state, const void* proj, long proj_stride, const void* conv_w,
                       const float* A_log, const float* dt_bias, const void* gnorm_w, const int* seg_slot, const int* seg_row0,
                       const int* seg_nrows, int nseg, int rb, int nk, int nv, float eps, int commit, cudaStream_t s) {
  using G = GdnRows<DK, DV, PARTS, SPLIT>;
  static bool attr_done = false;
  if (!attr_done) {
    FB_CUDA_CHECK(cudaFuncSetAttribute(gdn_rows_kernel<DK, DV, PARTS, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)G::smem(STEP_ROWS)));
    attr_done = true;
  }
  const int cluster = nv / nk * SPLIT;
  return (int)launch_pdl_cluster(cluster, gdn_rows_kernel<DK, DV, PARTS, SPLIT>, dim3(nv * SPLIT, nseg), dim3(G::THREADS), G::smem(rb), s,
                                 (__nv_bfloat16*)out, rec_state, (__nv_bfloat16*)conv_state, (const __nv_bfloat16*)proj, proj_stride,
                                 (const __nv_bfloat16*)conv_w, A_log, dt_bias, (const __nv_bfloat16*)gnorm_w, seg_slot, seg_row0, seg_nrows,
                                 nk, nv, eps, commit, rb, cluster);
}

// A head in as many slices as a cluster of four holds beside the heads that share a key head (clusters of eight wait for SMs of one GPC: 17
// rows of 32 heads on 16 took 30 us instead of 13).
static int step_slices(int nk, int nv, int d) {
  const int share = nv / nk;
  return share == 1 && d == 128 ? 4 : (share <= 2 ? 2 : 1);
}

// Whether a step goes to the kernel of several rows, with heads in slices.
static bool step_sliced(int nseg, int rows, int max_rows, int nk, int nv, int d) {
  const int share = nv / nk, split = step_slices(nk, nv, d);
  if (share > 8) return false;             // (no cluster holds them)
  // The kernel of several rows pays less for a row and more for a CTA, of which it has `split` times as many, one an SM. us of a wave of CTAs: 4.5 and
  // 0.35 a row (two slices 0.5, whole heads 5.9 and 0.8), against 2.8 + 1.8 a row of the kernel for single rows; heads of 64: 4.4 + 0.27 (whole 3.9 +
  // 0.45), 1.9 + 1.2. Clusters of more than four find fewer SMs. A launch is its waves over segments of the mean length and what the longest has
  // beyond it. One launch in a row of them, us, kernel for single rows / this one, 16 heads: 2 rows 6.4 / 4.8, 17 rows 33.4 / 10.7, 32 rows 60.4 / 15.8,
  // four times 17 33.6 / 21.0; 8 segments of 2, 5, 17 rows 7.1 / 18.7, 12.6 / 23.5, 34.8 / 41.6, seven of 1 and one of 17 34.1 / 23.8; 24 of 2 22.7 / 58.5.
  // Single rows whose slices fill a wave and no more: in a row 4.6 / 4.9, 32 heads on 16 4.9 / 5.3; between the other kernels of a step, where the states
  // come from DRAM, this one is the faster all the same: 771.1 / 770.0 us a step of three such layers of 16 heads, 200.8 / 198.7 of one of 32, two streams.
  const float mean = (float)rows / nseg, rest = max(0.f, (max_rows > 0 ? min(max_rows, rows - nseg + 1) : ceilf(mean)) - mean);
  const float fix_new = d == 64 ? (split == 2 ? 4.4f : 3.9f) : split == 1 ? 5.9f : 4.5f, row_old = d == 64 ? 1.2f : 1.8f;
  const float row_new = d == 64 ? (split == 2 ? 0.27f : 0.45f) : split == 4 ? 0.35f : split == 2 ? 0.5f : 0.8f;
  const int slots = share * split <= 4 ? STEP_CTAS : 96;
  const float waves_new = (nv * split * nseg + slots - 1) / slots, waves_old = max(1.f, (float)(nv * nseg) / STEP_CTAS);
  return (rows == nseg && nv * split >= 64 && nv * split * nseg <= STEP_CTAS) ||
         waves_new * (fix_new + row_new * mean) + row_new * rest < waves_old * ((d == 64 ? 1.9f : 2.8f) + row_old * mean) + row_old * rest;
}

template <int D, int PARTS>
static int launch_step(void* out, float* rec_state, void* conv_state, const void* proj, long proj_stride, const void* conv_w,
                       const float* A_log, const float* dt_bias, const void* gnorm_w, const int* seg_slot, const int* seg_row0,
                       const int* seg_nrows, int nseg, int rows, int max_rows, int nk, int nv, float eps, int commit, cudaStream_t s) {
  const int share = nv / nk;
  const int split = step_slices(nk, nv, D), rb = max(1, min(STEP_ROWS, rows - nseg + 1));
  auto go = [&](auto kern) {
    return kern(out, rec_state, conv_state, proj, proj_stride, conv_w, A_log, dt_bias, gnorm_w, seg_slot, seg_row0, seg_nrows, nseg, rb, nk, nv,
                eps, commit, s);
  };
  const uintptr_t places = reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(conv_w) | reinterpret_cast<uintptr_t>(conv_state);
  if (step_sliced(nseg, rows, max_rows, nk, nv, D) && proj_stride % 8 == 0 && (places & 15) == 0) {
    if constexpr (D == 128)
      if (split == 4) return go(launch_rows<D, D, PARTS, 4>);
    return split == 2 ? go(launch_rows<D, D, PARTS, 2>) : go(launch_rows<D, D, PARTS, 1>);
  }
  // One row each. Heads that share a key head are a cluster (0.4 us) while clusters of their size find room at once; their q / k tail is rewritten by a
  // launch of its own (1.3 us) otherwise: 16 heads on 2, 8 streams, 9.3 as clusters, 6.5 so; 24 streams of 12 heads of 64 on 2 7.2, 5.7.
  const bool cluster = share > 1 && (share <= 4 || (share <= 8 && nv * nseg <= 96));
  const auto one = cluster ? gdn_step_kernel<D, D, PARTS, true, 1> : gdn_step_kernel<D, D, PARTS, false, 1>;
  const auto two = cluster ? gdn_step_kernel<D, D, PARTS, true, 2> : gdn_step_kernel<D, D, PARTS, false, 2>;
  const cudaError_t e = launch_pdl_cluster(cluster ? share : 1, nv * nseg > STEP_CTAS ? two : one, dim3(nv, nseg), dim3(D * PARTS), (size_t)0, s,
                                           (__nv_bfloat16*)out, rec_state, (__nv_bfloat16*)conv_state, (const __nv_bfloat16*)proj, proj_stride,
                                           (const __nv_bfloat16*)conv_w, A_log, dt_bias, (const __nv_bfloat16*)gnorm_w, seg_slot, seg_row0,
                                           seg_nrows, nk, nv, eps, commit);
  if (e != cudaSuccess || share == 1 || cluster || !commit) return (int)e;
  const int qk = 2 * nk * D;
  return (int)launch_pdl(gdn_qk_tail_kernel, dim3((qk + 255) / 256, nseg), dim3(256), (size_t)0, s, (__nv_bfloat16*)conv_state,
                         (const __nv_bfloat16*)proj, proj_stride, seg_slot, seg_row0, seg_nrows, qk, qk + nv * D);
}

extern "C" int fb_gdn_step_sliced(int nseg, int rows, int max_rows, int nk, int nv, int d) { return step_sliced(nseg, rows, max_rows, nk, nv, d); }

// `rows`: rows of the step; `max_rows`: of its longest segment, 0 where that is not known (it decides on the kernel only).
extern "C" int fb_gdn_step(void* out, float* rec_state, void* conv_state, const void* proj, long proj_stride,
                           const void* conv_w, const float* A_log, const float* dt_bias, const void* gnorm_w,
                           const int* seg_slot, const int* seg_row0, const int* seg_nrows, int nseg, int rows, int max_rows, int nk, int nv,
                           int dk, int dv, float eps, int commit, cudaStream_t s) {
  if (nseg <= 0) return 0;
  if (nv % nk) return -1;
  if (dk != dv || (dk != 128 && dk != 64)) return -2;
  return (dk == 128 ? launch_step<128, 4> : launch_step<64, 8>)(out, rec_state, conv_state, proj, proj_stride, conv_w, A_log, dt_bias, gnorm_w,
                                                                 seg_slot, seg_row0, seg_nrows, nseg, rows, max_rows, nk, nv, eps, commit, s);
}
