// Device pieces that the tensor-core kernels on split operands (split.cuh) share: shared-memory layouts, the MMA, TMA
// loads of both planes, and the tensor map of an operand.
#pragma once
#include "split.cuh"
#include "tc_common.cuh"

namespace octc {

constexpr int SPLIT_BK = 32;      // k-values per TMA box

// An operand stored [K, rows]: atoms of 64 rows x 32 k of 128 bytes (128-byte swizzle), groups of 8 k 1024 bytes
// apart, 16 k-values are 2048 bytes; an atom's lo lies 4096 bytes behind its hi, so atoms are 8192 bytes apart.
constexpr int SPLIT_MN_ATOM = 8192, SPLIT_MN_LO = 4096;
__device__ __forceinline__ uint64_t split_desc_mn(uint32_t addr, int k16) {
  uint64_t d = (uint64_t)(((addr + k16 * 2048) & 0x3FFFFu) >> 4);
  d |= (uint64_t)(SPLIT_MN_ATOM >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// c = f32 (1<<4); a, b = f16 (0); major bits 15 / 16; N>>3 at 17; M>>4 at 24
__host__ __device__ constexpr uint32_t split_idesc(bool a_mn, bool b_mn, int m, int n) {
  return (1u << 4) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(id), "r"(accumulate) : "memory");
}

// both planes of a box (the map's last dimension)
__device__ __forceinline__ void tma_load_planes(uint32_t dst, const CUtensorMap* map, int x, int y, int z1, int z2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z1), "r"(z2), "r"(0), "r"(bar) : "memory");
}

// dims (inner, outer, problem 1, problem 2, plane); `tile_rows` is the box's extent along the rows of an operand
// stored [rows, K] (stored [K, rows]: 64 rows a box)
inline int make_split_map(CUtensorMap* map, const OcSplitOperand& o, int rows, int K, int nb1, int nb2, int tile_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) { oc_set_last_error("split operand: cuTensorMapEncodeTiled is not available"); return OC_ERR_CUDA; }
  const cuuint64_t inner = (cuuint64_t)(o.mn_major ? rows : K), outer = (cuuint64_t)(o.mn_major ? K : rows);
  const cuuint64_t whole = outer * (cuuint64_t)o.ld * 2;
  cuuint64_t dims[5] = {inner, outer, (cuuint64_t)nb1, (cuuint64_t)nb2, (cuuint64_t)o.terms};
  cuuint64_t strides[4] = {(cuuint64_t)o.ld * 2, nb1 > 1 ? (cuuint64_t)o.stride1 * 2 : whole,
                           nb2 > 1 ? (cuuint64_t)o.stride2 * 2 : whole, o.terms > 1 ? (cuuint64_t)o.plane * 2 : whole};
  cuuint32_t box[5] = {o.mn_major ? 64u : (cuuint32_t)SPLIT_BK, o.mn_major ? (cuuint32_t)SPLIT_BK : (cuuint32_t)tile_rows,
                       1, 1, (cuuint32_t)o.terms};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<__half*>(o.planes), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, o.mn_major ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { oc_set_last_error("split operand: cuTensorMapEncodeTiled failed"); return OC_ERR_CUDA; }
  return OC_OK;
}

}  // namespace octc
