// Experts of prompt-sized steps straight from their NVFP4 codes: y[row] = W[expert of row] x[row] over rows sorted by expert.
//
// A prompt of 1500 tokens leaves an expert of a 512-expert layer about 29 rows: too few for 128-row tiles of the grouped tcgen05 GEMM, which
// moreover needs the whole stacks in bf16 first (written and read again: 0.9 GB of codes become 3.2 GB). Here the codes go through a TMA ring
// and are unpacked in registers into mma.sync fragments (stream_mma.cuh: exact), once for up to 32 rows of their expert.
//
// Work item = (32 rows of an expert, tile of 128 weight rows; SwiGLU: 64 gate and 64 up rows), tiles of one run of rows next to each other so
// that their x comes from L2; CTAs, two per SM, take every gridDim-th item. One thread brings a unit of weights, its scales and the rows' x
// (four boxes of 64 values); eight warps multiply, each its own 16 weight rows. x comes with every eight values in the order of the code pairs
// (0 4 1 5 2 6 3 7): the dispatch of the rows and the first product's epilogue leave them so.
//
// Bound by unpacking (about 600 issue cycles a unit and SM) and by mma.sync (270 a unit and 8 rows), which overlap in part.
// 1500 rows, 512 experts, ten each, 2048 x 512: gate and up 370 us, down 213; the grouped GEMM took 670 for each after 410 for the bf16 copy of each
// stack.
#include "api_ext.h"
#include "stream_mma.cuh"

namespace fb {

constexpr int MS_ROWS = 32, MS_MT = MS_ROWS / 8;      // rows of an item
constexpr int MS_MATH = 8, MS_THREADS = (MS_MATH + 1) * 32;
constexpr int MS_SF = 2048, MS_X = MS_ROWS * 512, MS_STAGE = SM_TILE_BYTES + MS_SF + MS_X, MS_STAGES = 3;

struct MsArgs {
  const int* tile_start;          // [experts + 1] items' runs of 32 rows before an expert
  const int* row_base;            // [experts + 1] rows before an expert
  __nv_bfloat16* y;
  long ldy;
  int experts, w_rows, N, K, tiles, kblocks, cap_rows;
  float w_scale, limit;
  int* status;
};

template <bool DUAL>
__global__ void __launch_bounds__(MS_THREADS, 2)
moe_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmX, MsArgs a) {
  extern __shared__ __align__(1024) unsigned char ms_smem[];
  __shared__ __align__(8) uint64_t full_bar[MS_STAGES], empty_bar[MS_STAGES];
  __shared__ int abort_s;
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)ms_smem + 1023) & ~(uintptr_t)1023);
  int* starts = reinterpret_cast<int*>(ring + (size_t)MS_STAGES * MS_STAGE);
  int* bases = starts + a.experts + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_s;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int i = 0; i < MS_STAGES; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], MS_MATH); }
    fence_mbar_init();
  }
  pdl_wait();
  for (int i = threadIdx.x; i <= a.experts; i += MS_THREADS) { starts[i] = a.tile_start[i]; bases[i] = a.row_base[i]; }
  __syncthreads();
  const long long total = (long long)starts[a.experts] * a.tiles;
  // item -> expert, first row, rows, first weight row of its tile
  auto item = [&](long long w, int& expert, int& row0, int& rows, int& n0) {
    const int run = (int)(w / a.tiles);
    n0 = (int)(w % a.tiles) * (DUAL ? 64 : 128);
    int lo = 0, hi = a.experts;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (starts[mid] <= run) lo = mid; else hi = mid;
    }
    expert = lo;
    row0 = bases[lo] + (run - starts[lo]) * MS_ROWS;
    rows = min(min(bases[lo + 1], a.cap_rows) - row0, MS_ROWS);
  };

  if (warp == MS_MATH) {
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmS);
      tma_prefetch_desc(&tmX);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (long long w = blockIdx.x; w < total && ok; w += gridDim.x) {
        int e, row0, rows, n0;
        item(w, e, row0, rows, n0);
        const int r0 = e * a.w_rows + n0, r1 = DUAL ? r0 + a.N : r0 + 64;
        for (int kb = 0; kb < a.kblocks; ++kb) {
          if (!(ok = sm_wait(&empty_bar[stage], phase ^ 1u, abort_flag))) break;
          unsigned char* st = ring + (size_t)stage * MS_STAGE;
          mbar_expect_tx(&full_bar[stage], (uint32_t)MS_STAGE);
          tma_load_2d(st, &tmW, &full_bar[stage], kb * 128, r0);
          tma_load_2d(st + 8192, &tmW, &full_bar[stage], kb * 128, r1);
          tma_load_2d(st + SM_TILE_BYTES, &tmS, &full_bar[stage], kb * 16, r0);
          tma_load_2d(st + SM_TILE_BYTES + MS_SF / 2, &tmS, &full_bar[stage], kb * 16, r1);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            tma_load_2d(st + SM_TILE_BYTES + MS_SF + i * (MS_ROWS * 128), &tmX, &full_bar[stage], kb * 256 + i * 64, row0);
          if (++stage == MS_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
    }
  } else {
    const int g = lane >> 2, t = lane & 3;
    const SmFactors fac = sm_factors();
    const int lo = (DUAL ? 8 : 16) * warp + sm_row(g), hi = lo + (DUAL ? 64 : 8);
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (long long w = blockIdx.x; w < total; w += gridDim.x) {
      int e, row0, rows, n0;
      item(w, e, row0, rows, n0);
      const int live = (rows + 7) / 8;
      float acc[2][MS_MT][4];
#pragma unroll
      for (int i = 0; i < MS_MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[0][i][j] = acc[1][i][j] = 0.f;
      for (int kb = 0; kb < a.kblocks; ++kb) {
        ok = __all_sync(0xffffffffu, sm_wait(&full_bar[stage], phase, abort_flag));
        if (!ok) break;
        const uint32_t st = smem_u32(ring + (size_t)stage * MS_STAGE), sf = st + SM_TILE_BYTES;
        sm_unit<MS_MT, true, true, true>(acc, st, lo, hi, sf + MS_SF, sf + (uint32_t)lo * 16, sf + (uint32_t)hi * 16, fac, live);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
        if (++stage == MS_STAGES) { stage = 0; phase ^= 1u; }
      }
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; break; }
      const int n = n0 + lo;                               // the plain form's second row is n + 8
      const float scale = a.w_scale * SM_FP4_FACTOR;
#pragma unroll
      for (int i = 0; i < MS_MT; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int m = i * 8 + sm_row4(2 * t + j);
          if (i >= live || m >= rows) continue;
          const float v0 = (acc[0][i][j] + acc[1][i][j]) * scale, v1 = (acc[0][i][2 + j] + acc[1][i][2 + j]) * scale;
          __nv_bfloat16* yr = a.y + (size_t)(row0 + m) * a.ldy;
          if (DUAL) {
            const int q = n & 7;                           // stored in the order of the code pairs
            if (n < a.N) yr[(n & ~7) | (q < 4 ? 2 * q : 2 * q - 7)] = f2bf(glu_act(v0, v1, a.limit));
          } else {
            if (n < a.N) yr[n] = f2bf(v0);
            if (n + 8 < a.N) yr[n + 8] = f2bf(v1);
          }
        }
    }
  }
  __syncthreads();
  if (abort_s && threadIdx.x == 0)                         // loads already issued still target this CTA's shared memory
    for (int i = 0; i < MS_STAGES; ++i)
      for (uint32_t p = 0; p < 2; ++p) (void)mbar_wait(&full_bar[i], p, 1u << 12);
}

template <bool DUAL>
static int launch_ms(const MsArgs& a, const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap& tx, int sm_count, cudaStream_t s) {
  const size_t smem = (size_t)MS_STAGES * MS_STAGE + 1024 + 2 * (size_t)(a.experts + 1) * sizeof(int);
  static const cudaError_t attr = cudaFuncSetAttribute(moe_stream_kernel<DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024);
  if (attr != cudaSuccess) return (int)attr;
  return (int)launch_pdl(moe_stream_kernel<DUAL>, dim3(2 * sm_count), dim3(MS_THREADS), smem, s, tw, ts, tx, a);
}

}  // namespace fb

using namespace fb;

// Rows of an item: `tile_start` counts runs of so many.
extern "C" int fb_moe_stream_rows() { return MS_ROWS; }

// Whether stacks of these sizes are taken.
extern "C" int fb_moe_stream_fits(int N, int K, int experts) { return N > 0 && K > 0 && K % 256 == 0 && N % 8 == 0 && experts > 0 && experts <= 1024; }

// x [cap_rows][K] bf16 in the order of the code pairs; codes [experts (or more)][N or 2N][K / 2], scales [..][K / 16]. mode 1: SwiGLU (with a
// limit: clamped units), y in that order too; 0: plain.
extern "C" int fb_moe_stream(void* y, const void* x, const void* codes, const void* scales, float w_scale, const int* tile_start, const int* row_base,
                             int experts, int cap_rows, int N, int K, long ldx, long ldy, int mode, float limit, int* status, int sm_count,
                             cudaStream_t s) {
  if (!fb_moe_stream_fits(N, K, experts) || ldx % 8 || cap_rows <= 0) return -1;
  if (((uintptr_t)x | (uintptr_t)codes | (uintptr_t)scales) & 15) return -1;
  const bool dual = mode == 1;
  if (sm_count <= 0) sm_count = 148;
  MsArgs a;
  a.tile_start = tile_start; a.row_base = row_base; a.y = (__nv_bfloat16*)y; a.ldy = ldy; a.experts = experts; a.w_rows = dual ? 2 * N : N; a.N = N; a.K = K;
  a.tiles = dual ? (N + 63) / 64 : (N + 127) / 128; a.kblocks = K / 256; a.cap_rows = cap_rows; a.w_scale = w_scale; a.limit = limit; a.status = status;
  const long rows = (long)experts * a.w_rows;
  CUtensorMap tw, ts, tx;
  if (!sm_map(&tw, codes, true, K / 2, rows, K / 2, 128, 64) || !sm_map(&ts, scales, true, K / 16, rows, K / 16, 16, 64) ||
      !sm_map(&tx, x, false, K, cap_rows, 2L * ldx, 64, MS_ROWS))
    return -12;
  return dual ? launch_ms<true>(a, tw, ts, tx, sm_count, s) : launch_ms<false>(a, tw, ts, tx, sm_count, s);
}
