// Experts of prompt-sized steps straight from their NVFP4 codes: y[row] = W[expert of row] x[row] over rows sorted by expert.
//
// A prompt of 1500 tokens leaves an expert of a 512-expert layer about 29 rows: too few for 128-row tiles of the grouped tcgen05 GEMM, which
// moreover needs the whole stacks in bf16 first (written and read again: 0.9 GB of codes become 3.2 GB). Here the codes go through a TMA ring
// and are unpacked in registers (stream_mma.cuh: exact) into tensor memory, as the A operand of tcgen05.mma; x is the B operand, 16 to 64 rows of one
// expert, so that a code is unpacked once for all of them.
//
// Work item = (up to 64 rows of an expert, two tiles of 128 weight rows; SwiGLU: one of gate and one of up rows); a CTA an SM takes an equal share of the
// items, side by side, so that a run of rows finds its x in L2. It walks K in units of 256: x once, then the tiles' codes, each a unit.
// Warps: 0 loads; 1 and 2 multiply, a tile each; 4 .. 7 bring finished tiles out while the next item's are summed up in the other half of
// the accumulators; 8 .. 23 unpack, eight a tile, a thread half a row of a unit. The units' block scales come straight from global memory, a unit ahead.
// Tensor memory: 2 x two accumulators of 64 columns | an operand of 128 (256 values in bf16) for either tile, handed over by halves. x comes with every
// eight values in the order of the code pairs (0 4 1 5 2 6 3 7): the dispatch of the rows and the first product's epilogue leave them so.
//
// Bound by issue slots (0.8 of them taken): unpacking a unit is some 640 of its 1,300 cycles a scheduler, waits, scales, epilogue and the issue of the
// products the rest. What it hung on before: products issued behind a branch for one lane (95 cycles each instead of 16, see tc_mma_f16_ts_if),
// unrolled code that fell out of the instruction cache, two unpacking warps a scheduler instead of four.
// 1500 rows, 512 experts, ten each, 2048 x 512, us: gate and up 174, down 105, the whole block 299; in mma.sync fragments, 32 rows an item, 367, 216,
// 624; the grouped GEMM took 670 for each after 410 for the bf16 copy of each stack.
#include "api_ext.h"
#include "stream_mma.cuh"

namespace fb {

constexpr int MS_ROWS = 64, MS_TILES = 2;             // rows and tiles of an item
constexpr int MS_THREADS = 768;
constexpr int MS_CODES = SM_TILE_BYTES, MS_CODE_STAGES = 6;             // a unit: codes of 128 rows x 256 values
constexpr int MS_X = MS_ROWS * 512, MS_X_STAGES = 3;  // four boxes of 64 values, each in halves of 32 rows
constexpr uint32_t MS_COL_A = 2 * MS_TILES * MS_ROWS;

struct MsArgs {
  const int* tile_start;          // [experts + 1] items' runs of 64 rows before an expert
  const int* row_base;            // [experts + 1] rows before an expert
  const unsigned char* scales;
  __nv_bfloat16* y;
  long ldy;
  int experts, w_rows, N, K, groups, kblocks, cap_rows;             // groups of MS_TILES tiles a run
  float w_scale, limit;
  int* status;
};

template <bool DUAL>
__global__ void __launch_bounds__(MS_THREADS, 1)
moe_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, MsArgs a) {
  extern __shared__ __align__(1024) unsigned char ms_smem[];
  __shared__ __align__(8) uint64_t c_full[MS_CODE_STAGES], c_empty[MS_CODE_STAGES], x_full[MS_X_STAGES], x_empty[MS_X_STAGES];
  __shared__ __align__(8) uint64_t a_full[4], a_empty[4], d_full[2 * MS_TILES], d_empty[2 * MS_TILES];
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;
  unsigned char* codes = reinterpret_cast<unsigned char*>(((uintptr_t)ms_smem + 1023) & ~(uintptr_t)1023);
  unsigned char* xs = codes + MS_CODE_STAGES * MS_CODES;
  int* starts = reinterpret_cast<int*>(xs + MS_X_STAGES * MS_X);
  int* bases = starts + a.experts + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_s;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int i = 0; i < MS_CODE_STAGES; ++i) { mbar_init(&c_full[i], 1); mbar_init(&c_empty[i], 8); }
    for (int i = 0; i < MS_X_STAGES; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], MS_TILES); }
    for (int i = 0; i < 4; ++i) { mbar_init(&a_full[i], 4); mbar_init(&a_empty[i], 1); }
    for (int i = 0; i < 2 * MS_TILES; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], 4); }
    fence_mbar_init();
  }
  if (warp == 3) {
    tmem_alloc(&tmem_s, 512);
    tmem_relinquish();
  }
  pdl_wait();
  for (int i = threadIdx.x; i <= a.experts; i += MS_THREADS) { starts[i] = a.tile_start[i]; bases[i] = a.row_base[i]; }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  // this CTA's items: an equal share of all, side by side
  const long long all = (long long)starts[a.experts] * a.groups;
  const long long first = all * blockIdx.x / gridDim.x, end = all * (blockIdx.x + 1) / gridDim.x;
  struct Item {
    int left, run, group, e;                               // items from here on; run of rows, group of tiles; expert
  };
  auto begin = [&]() {
    Item it;
    it.left = (int)(end - first);
    it.run = (int)(first / a.groups);
    it.group = (int)(first % a.groups);
    int lo = 0, hi = a.experts;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (starts[mid] <= it.run) lo = mid; else hi = mid;
    }
    it.e = lo;
    return it;
  };
  auto next = [&](Item& it) {
    --it.left;
    if (++it.group < a.groups) return;
    it.group = 0;
    ++it.run;
    while (it.left > 0 && starts[it.e + 1] <= it.run) ++it.e;
  };
  auto row_of = [&](const Item& it) { return bases[it.e] + (it.run - starts[it.e]) * MS_ROWS; };
  auto rows_of = [&](const Item& it) { return min(min(bases[it.e + 1], a.cap_rows) - row_of(it), MS_ROWS); };
  // first weight row of tile t (SwiGLU: tiles 0 and 1 are gate and up rows of the same units)
  auto tile_row = [&](const Item& it, int t) { return DUAL ? it.group * 128 + (t ? a.N : 0) : (it.group * MS_TILES + t) * 128; };
  bool ok = true;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      int cs = 0, x = 0;
      uint32_t cp = 0, xp = 0;
      for (Item it = begin(); it.left > 0 && ok; next(it)) {
        const int row0 = row_of(it), rows = rows_of(it);
        for (int kb = 0; kb < a.kblocks && ok; ++kb) {
          for (int t = 0; t < MS_TILES; ++t) {
            if (!(ok = sm_wait(&c_empty[cs], cp ^ 1u, abort_flag))) break;
            unsigned char* st = codes + cs * MS_CODES;
            const int r = it.e * a.w_rows + tile_row(it, t);
            mbar_expect_tx(&c_full[cs], (uint32_t)MS_CODES);
            tma_load_2d(st, &tmW, &c_full[cs], kb * 128, r);
            if (++cs == MS_CODE_STAGES) { cs = 0; cp ^= 1u; }
            if (t > 0) continue;                           // (x behind the first unit, whose unpacking takes longest)
            if (!(ok = sm_wait(&x_empty[x], xp ^ 1u, abort_flag))) break;
            const int halves = rows > 32 ? 2 : 1;
            mbar_expect_tx(&x_full[x], (uint32_t)(halves * (MS_X / 2)));
            for (int i = 0; i < 4; ++i)
              for (int h = 0; h < halves; ++h)
                tma_load_2d(xs + x * MS_X + i * (MS_ROWS * 128) + h * 4096, &tmX, &x_full[x], kb * 256 + i * 64, row0 + h * 32);
            if (++x == MS_X_STAGES) { x = 0; xp ^= 1u; }
          }
        }
      }
      if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
    }
  } else if (warp <= MS_TILES) {                           // a tile each
    const uint32_t t = warp - 1;
    int x = 0;
    uint32_t xp = 0, unit = 0, done = 0;                   // units (of this tile) and items so far
    const uint64_t xd = umma_desc_k128(smem_u32(xs));
    const bool issue = elect_one();
    for (Item it = begin(); it.left > 0 && ok; next(it), ++done) {
      const int rows = rows_of(it);
      const uint32_t idesc = umma_idesc(1, 1, 128, (uint32_t)max(16, (rows + 15) & ~15)), d = (done & 1) * MS_TILES + t;
      ok = __all_sync(0xffffffffu, sm_wait(&d_empty[d], ((done >> 1) & 1u) ^ 1u, abort_flag));
      for (int kb = 0; kb < a.kblocks && ok; ++kb, ++unit) {
        ok = __all_sync(0xffffffffu, sm_wait(&x_full[x], xp, abort_flag));
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
          if (ok) ok = __all_sync(0xffffffffu, sm_wait(&a_full[2 * t + half], unit & 1u, abort_flag));
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd = xd + (uint64_t)((x * MS_X + half * (MS_ROWS * 256)) >> 4);
          const uint32_t ad = tmem + MS_COL_A + t * 128 + half * 64;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            tc_mma_f16_ts_if(issue, tmem + d * MS_ROWS, ad + k * 8, bd + (uint64_t)((k >> 2) * (MS_ROWS * 8) + 2 * (k & 3)), idesc,
                             kb > 0 || half > 0 || k > 0);
          tc_commit_if(issue, &a_empty[2 * t + half]);
        }
        if (!ok) break;
        tc_commit_if(issue, &x_empty[x]);
        if (++x == MS_X_STAGES) { x = 0; xp ^= 1u; }
      }
      if (ok) tc_commit_if(issue, &d_full[d]);
    }
    if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
  } else if (warp >= 8) {
    const uint32_t group = warp >= 16, half = (warp >> 2) & 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t to = tmem + ((uint32_t)((warp & 3) * 32) << 16) + MS_COL_A + group * 128 + half * 64;
    const SmFactors fac = sm_factors();
    uint32_t unit = group;
    int cs = (int)group;
    uint32_t cp = 0;
    Item it = begin();
    // the row's scales: the next unit's are asked for while this one is unpacked
    auto scale_row = [&]() {
      return a.scales + min((long)it.e * a.w_rows + tile_row(it, group) + row, (long)a.experts * a.w_rows - 1) * (a.K / 16) + half * 8;
    };
    const unsigned char* sr = scale_row();
    uint2 sf = it.left > 0 ? __ldg(reinterpret_cast<const uint2*>(sr)) : make_uint2(0u, 0u);
    while (it.left > 0 && ok) {
      for (int kb = 0; kb < a.kblocks && ok; ++kb, unit += 2) {
        ok = __all_sync(0xffffffffu, sm_wait(&c_full[cs], cp, abort_flag));
        if (!ok) break;
        const uint32_t st = smem_u32(codes + cs * MS_CODES) + row * 128, flip = ((row & 7) << 4) ^ (half * 64);
        uint2 sw = sf;
        if (kb + 1 < a.kblocks) {
          sf = __ldg(reinterpret_cast<const uint2*>(sr + kb * 16 + 16));
        } else {
          next(it);
          sr = scale_row();
          if (it.left > 0) sf = __ldg(reinterpret_cast<const uint2*>(sr));
        }
        uint4 v[4];                                        // four of the row's 16-byte chunks: 32 values, 16 columns each
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) v[c] = sm_lds(st + ((c * 16) ^ flip));
        ok = __all_sync(0xffffffffu, sm_wait(&a_empty[2 * group + half], ((unit >> 1) & 1u) ^ 1u, abort_flag));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          uint32_t r[32];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t two = c ? sw.y : sw.x;
            const uint2 sc = sm_scales(j ? two >> 16 : two);
            const uint32_t word[4] = {v[c + j].x, v[c + j].y, v[c + j].z, v[c + j].w};
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              uint32_t q[4];
              sm_unpack(word[p], p < 2 ? sc.x : sc.y, fac, q);
#pragma unroll
              for (int k = 0; k < 4; ++k) r[j * 16 + p * 4 + k] = q[k];
            }
          }
          tmem_st32(to + c * 16, r);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&a_full[2 * group + half]);          // half of the unit: the products with it may begin
          mbar_arrive(&c_empty[cs]);
        }
        if ((cs += 2) >= MS_CODE_STAGES) { cs -= MS_CODE_STAGES; cp ^= 1u; }
      }
    }
    if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
  } else if (warp >= 4) {
    const uint32_t from = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int lrow = (warp & 3) * 32 + lane;
    const float scale = a.w_scale * SM_FP4_FACTOR;
    uint32_t dp = 0;
    int parity = 0;
    for (Item it = begin(); it.left > 0 && ok; next(it), parity ^= 1) {
      const int row0 = row_of(it), rows = rows_of(it);
      for (int t = 0; t < MS_TILES; t += DUAL ? 2 : 1) {
        const int d = parity * MS_TILES + t;
        ok = sm_wait(&d_full[d], (dp >> d) & 1u, abort_flag) && (!DUAL || sm_wait(&d_full[d + 1], (dp >> (d + 1)) & 1u, abort_flag));
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        dp ^= (DUAL ? 3u : 1u) << d;
        tc_fence_after();
        const int n = (DUAL ? it.group : it.group * MS_TILES + t) * 128 + lrow, q = n & 7;
        const int at = DUAL ? (n & ~7) | (q < 4 ? 2 * q : 2 * q - 7) : n;              // SwiGLU: stored in the order of the code pairs
        __nv_bfloat16* yr = a.y + (size_t)row0 * a.ldy + at;
#pragma unroll 1
        for (int h = 0; h < rows; h += 8, yr += 8 * a.ldy) {
          uint32_t v[8], u[8];
          tmem_ld8(from + d * MS_ROWS + h, v);
          if (DUAL) tmem_ld8(from + (d + 1) * MS_ROWS + h, u);
          tmem_ld_wait();
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            const float s = __uint_as_float(v[m]) * scale;
            const float o = DUAL ? glu_act(s, __uint_as_float(u[m]) * scale, a.limit) : s;
            if (h + m < rows && n < a.N) yr[m * a.ldy] = f2bf(o);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&d_empty[d]);
          if (DUAL) mbar_arrive(&d_empty[d + 1]);
        }
      }
    }
    if (!ok) { set_status(a.status, ST_MBAR_TIMEOUT); abort_s = 1; }
  }
  __syncthreads();
  if (abort_s && threadIdx.x == 0) {                       // loads already issued still target this CTA's shared memory
    for (int i = 0; i < MS_CODE_STAGES; ++i)
      for (uint32_t p = 0; p < 2; ++p) (void)mbar_wait(&c_full[i], p, 1u << 12);
    for (int i = 0; i < MS_X_STAGES; ++i)
      for (uint32_t p = 0; p < 2; ++p) (void)mbar_wait(&x_full[i], p, 1u << 12);
  }
  __syncthreads();
  if (warp == 3) tmem_dealloc(tmem, 512);
}

template <bool DUAL>
static int launch_ms(const MsArgs& a, const CUtensorMap& tw, const CUtensorMap& tx, int sm_count, cudaStream_t s) {
  constexpr size_t ring = (size_t)MS_CODE_STAGES * MS_CODES + (size_t)MS_X_STAGES * MS_X + 1024;
  static const cudaError_t attr =
      cudaFuncSetAttribute(moe_stream_kernel<DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(ring + 2 * 1025 * sizeof(int)));
  if (attr != cudaSuccess) return (int)attr;
  return (int)launch_pdl(moe_stream_kernel<DUAL>, dim3(sm_count), dim3(MS_THREADS), ring + 2 * (size_t)(a.experts + 1) * sizeof(int), s, tw, tx, a);
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
  a.tile_start = tile_start; a.row_base = row_base; a.scales = (const unsigned char*)scales; a.y = (__nv_bfloat16*)y; a.ldy = ldy; a.experts = experts; a.w_rows = dual ? 2 * N : N; a.N = N; a.K = K;
  a.groups = dual ? (N + 127) / 128 : (N + 255) / 256; a.kblocks = K / 256; a.cap_rows = cap_rows; a.w_scale = w_scale; a.limit = limit; a.status = status;
  const long rows = (long)experts * a.w_rows;
  CUtensorMap tw, tx;
  if (!sm_map(&tw, codes, true, K / 2, rows, K / 2, 128, 128) || !sm_map(&tx, x, false, K, cap_rows, 2L * ldx, 64, 32))
    return -12;
  return dual ? launch_ms<true>(a, tw, tx, sm_count, s) : launch_ms<false>(a, tw, tx, sm_count, s);
}
