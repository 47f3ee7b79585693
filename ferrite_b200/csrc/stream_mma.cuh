// Pieces of the products that stream weights through a TMA ring: into mma.sync fragments (gemv_stream.cu), or, 4-bit ones, unpacked as an operand of tcgen05
// (moe_stream.cu, which takes the unpacking, the waits and the maps from here).
//
// A unit of work is 128 weight rows x 128 bytes of K: 64 bf16 or 256 e2m1 values. TMA writes it with the 128-byte swizzle (16-byte chunk c of
// row r at c ^ (r & 7)); warp w owns 16 of the rows. A dot product does not care about the order of k, so the thread that m16n8k16 makes owner
// of k pairs takes whole 16-byte chunks of its two rows: chunk t (= lane & 3) and t + 4. Fragment row g reads tile row
// sm_row(g): eight consecutive lanes (two fragment rows, four chunks) then meet rows that differ in bit 2, whose swizzled chunks lie in
// different halves of the 128 bytes, and the 16-byte reads are free of bank conflicts.
//
// Activations of a unit sit beside it, token-major: bf16 as TMA writes them (token column g of the fragments is row sm_row(g) then), or, where
// a warp prepares them, in the order in which the fragments want them:
//   bf16  row of 8 chunks, chunk c at c ^ sm_row(token)
//   e2m1  a thread's 32-value chunk q is four pieces of 8 values (one word of codes each); piece p of chunk q is at
//         ((q >> 2) * 4 + p) * 4 + (q & 3), with bit 2 flipped for odd tokens, its values in the order 0 4 1 5 2 6 3 7: the nibbles that one
//         shift brings to the same place of both halves of a register
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace fb {

constexpr int SM_TILE_BYTES = 16384;                  // 128 rows x 128 bytes

__device__ __forceinline__ int sm_row(int g) { return ((g & 1) << 2) | ((g >> 1) & 3); }
__device__ __forceinline__ uint32_t sm_x_bf16(int token, int c) { return (uint32_t)(token * 128 + ((c ^ sm_row(token & 7)) << 4)); }
__device__ __forceinline__ uint32_t sm_x_fp4(int token, int c) {                // c = k / 8 inside the unit
  const int q = c >> 2, p = c & 3;
  return (uint32_t)(token * 512 + (((((q >> 2) * 4 + p) * 4 + (q & 3)) ^ ((token & 1) << 2)) << 4));
}
// Eight consecutive bf16 values in the order of an e2m1 piece.
__device__ __forceinline__ uint4 sm_piece(uint4 v) {
  return make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
}
__device__ __forceinline__ uint4 sm_lds(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t sm_lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sm_sts(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 sm_ldg(const void* p) {                        // rows that an earlier kernel wrote: through L2
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void sm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t sm_mul_bf2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// e2m1 to bf16 by bit placement: sign to bit 15, the three bits of exponent and fraction to bits 8..6, so that a code's value comes out times
// 2^-126 (0.5 as a subnormal). The e4m3 block scale is placed the same way (its seven bits to 10..4: times 2^-120) and brought to 2^118 by
// two exact products; code x scale, six significant bits, is exact in bf16 and holds the weight times 2^-8, which the caller makes up for.
// e4m3 has one NaN and no infinity: its bits would be 480, the next step after the largest value, 448. A factor of 1.1 x 2^112 (at a scale times
// 2^7) overflows for the one and not for the other, and adding 0 x that product turns only it into NaN. (Beside the ~40 instructions that unpack
// a scale's 16 codes these two, of the multiplier pipe, are not seen.)
constexpr float SM_FP4_FACTOR = 256.f;
__device__ __forceinline__ uint2 sm_scales(uint32_t two) {                       // two neighbouring block scales -> each in both halves
  uint32_t v = ((two & 0xffu) << 4) | ((two & 0xff00u) << 12);
  v = sm_mul_bf2(v, 0x7f007f00u);                                               // 2^127
  const uint32_t top = sm_mul_bf2(v, 0x778d778du);                              // 1.1 x 2^112
  v = sm_mul_bf2(v, 0x77007700u);                                               // 2^111
  asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(v) : "r"(top), "r"(0u));
  return make_uint2(__byte_perm(v, v, 0x1010), __byte_perm(v, v, 0x3232));
}
// Nibbles j and j + 4 of a word, j = 0 .. 3, times their scale. The product with 2^12 + 2^6 (nibble at bit 0; 2^8 + 2^2 at bit 4) writes the
// nibble twice, once for its sign and once for the rest: one instruction of the multiplier pipe instead of two of the logic pipe, which is the
// busier one. (The factors come in registers: constants would be turned back into shifts and adds.)
struct SmFactors { uint32_t at0, at4; };
__device__ __forceinline__ SmFactors sm_factors() {
  SmFactors f;
  asm volatile("mov.u32 %0, 0x1040;\n\tmov.u32 %1, 0x104;" : "=r"(f.at0), "=r"(f.at4));
  return f;
}
__device__ __forceinline__ uint32_t sm_place(uint32_t w, uint32_t mask, uint32_t factor) {
  uint32_t d;
  asm("mul.lo.u32 %0, %1, %2;" : "=r"(d) : "r"(w & mask), "r"(factor));
  return d & 0x81c081c0u;
}
__device__ __forceinline__ void sm_unpack(uint32_t w, uint32_t scale, SmFactors f, uint32_t (&r)[4]) {
  const uint32_t h = w >> 8;
  r[0] = sm_mul_bf2(sm_place(w, 0x000f000fu, f.at0), scale);
  r[1] = sm_mul_bf2(sm_place(w, 0x00f000f0u, f.at4), scale);
  r[2] = sm_mul_bf2(sm_place(h, 0x000f000fu, f.at0), scale);
  r[3] = sm_mul_bf2(sm_place(h, 0x00f000f0u, f.at4), scale);
}

// One unit for one warp: acc += the warp's 16 rows x 8 MT tokens (in two sets of sums: products into one set wait for each other).
// `tile`: the weights; `lo`, `hi`: tile rows of fragment rows g and g + 8 of this lane; `xt`: the activations, XT (bf16 weights): as TMA wrote
// them; `sf_lo`, `sf_hi` (e2m1): shared addresses of the rows' scale bytes in the first of the unit's four atoms (512 bytes: 128 rows x 4 blocks).
template <int MT, bool FP4, bool XT>
__device__ __forceinline__ void sm_unit(float (&acc)[2][MT][4], uint32_t tile, int lo, int hi, uint32_t xt, uint32_t sf_lo, uint32_t sf_hi,
                                        SmFactors f) {
  static_assert(!(FP4 && XT), "");
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = t + 4 * h;
    uint4 a = sm_lds(tile + (uint32_t)(lo * 128 + ((c ^ (lo & 7)) << 4)));
    uint4 b = sm_lds(tile + (uint32_t)(hi * 128 + ((c ^ (hi & 7)) << 4)));
    if constexpr (!FP4) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int r = mt * 8 + sm_row(g);
        const uint4 x = sm_lds(xt + (XT ? (uint32_t)(r * 128 + ((c ^ sm_row(g)) << 4)) : sm_x_bf16(mt * 8 + g, c)));
        sm_mma(acc[0][mt], a.x, b.x, a.y, b.y, x.x, x.y);
        sm_mma(acc[1][mt], a.z, b.z, a.w, b.w, x.z, x.w);
      }
    } else {
      const uint32_t off = (uint32_t)((c >> 1) * 512 + ((2 * c) & 3));
      const uint2 sa = sm_scales(sm_lds16(sf_lo + off)), sb = sm_scales(sm_lds16(sf_hi + off));
      const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        uint32_t ra[4], rb[4];
        sm_unpack(wa[p], p < 2 ? sa.x : sa.y, f, ra);
        sm_unpack(wb[p], p < 2 ? sb.x : sb.y, f, rb);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const uint4 x = sm_lds(xt + sm_x_fp4(mt * 8 + g, c * 4 + p));
          sm_mma(acc[0][mt], ra[0], rb[0], ra[1], rb[1], x.x, x.y);
          sm_mma(acc[1][mt], ra[2], rb[2], ra[3], rb[3], x.z, x.w);
        }
      }
    }
  }
}

// Waits of warps that are ahead: the thread sleeps in the barrier for up to SM_NAP ns at a time, so that what it waits for gets the issue slots.
constexpr uint32_t SM_NAP = 1000;
__device__ __forceinline__ bool sm_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t at = smem_u32(bar);
  for (uint32_t i = 0; i < FB_SPIN_LIMIT / 16; ++i) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(at), "r"(parity), "r"(SM_NAP) : "memory");
    if (ok) return true;
    if ((i & 63u) == 63u && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void sm_bulk_load(void* smem_dst, const void* gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

typedef CUresult (*EncodeTiledFnSm)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Map over [rows][cols] (bf16, or bytes): boxes of `box_cols` x box_rows, 128-byte swizzle where a box row is 128 bytes, zeros outside.
static bool sm_map(CUtensorMap* tm, const void* p, bool bytes, long cols, long rows, long row_bytes, int box_cols, int box_rows) {
  static EncodeTiledFnSm fn = [] {
    void* e = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &e, cudaEnableDefault, &qres) != cudaSuccess) return (EncodeTiledFnSm) nullptr;
    return qres == cudaDriverEntryPointSuccess ? (EncodeTiledFnSm)e : (EncodeTiledFnSm) nullptr;
  }();
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_bytes};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const bool swz = box_cols * (bytes ? 1 : 2) == 128;
  return fn && fn(tm, bytes ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swz ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace fb
