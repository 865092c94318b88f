// fp32 matrices as two fp16 planes, and products of such matrices on the tensor cores
// (split.cu, gemm_split.cu).
#pragma once
#include "common.cuh"

// A matrix is cut into 128 x 128 blocks; a block (or a row of a block) is scaled by a power of two that
// brings its largest finite entry to 2^14 .. 2^15, and every scaled entry v is kept as hi = fp16(v) and
// lo = fp16(v - hi), both rounded to nearest.  hi + lo is v to 2^-23 relative for entries within 2^-17 of
// the largest, and to 2^-40 of the largest below that.  The table of a matrix holds what undoes the
// scaling, 2^-e, per block or per row of a block.  Rows of weights are scaled each for itself: what comes
// out of one row must not depend on which others are in the call.
constexpr int OC_SPLIT_BLOCK = 128;

// scale that brings `mx` to 2^14 .. 2^15, and its inverse (both powers of two; 1 for zero and subnormal)
__device__ __forceinline__ float oc_split_scale(float mx, float& inv) {
  const int e = (int)(__float_as_uint(mx) >> 23);            // biased exponent; 0: zero or subnormal
  if (e == 0 || e == 255) { inv = 1.f; return 1.f; }
  const int k = min(141 - e, 126);                           // 14 - (e - 127), kept inside the normal range
  inv = __uint_as_float((unsigned)(127 - k) << 23);
  return __uint_as_float((unsigned)(127 + k) << 23);
}

__device__ __forceinline__ float oc_finite_abs(float v) {
  const float a = fabsf(v);
  return a <= 3.402823466e38f ? a : 0.f;
}

// hi and lo of four scaled entries
__device__ __forceinline__ void oc_split4(float4 t, uint2& hi, uint2& lo) {
  const __half2 a = __floats2half2_rn(t.x, t.y), b = __floats2half2_rn(t.z, t.w);
  const float2 fa = __half22float2(a), fb = __half22float2(b);
  const __half2 c = __floats2half2_rn(t.x - fa.x, t.y - fa.y), d = __floats2half2_rn(t.z - fb.x, t.w - fb.y);
  hi = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
  lo = make_uint2(*reinterpret_cast<const unsigned*>(&c), *reinterpret_cast<const unsigned*>(&d));
}

enum : int { OC_SPLIT_ALL = 0, OC_SPLIT_UPPER = 1, OC_SPLIT_LOWER = 2 };

// src [rows, cols] -> planes (hi, and `plane` elements behind it lo; rows ldp apart) and the table: entry
// rb * ldt + cb of block (rb, cb), or cb * ldt + row where every row has its own (per_row).
// UPPER / LOWER: entries on the other side of the diagonal count as zero whatever src holds, and of the
// blocks on that side only those are written that a 256-wide tile of the product may touch.
struct OcSplitArgs {
  const float* src; long long ld;
  const int* perm;                     // column c of the matrix is column perm[c] of src; null: c
  int rows, cols;
  __half* planes; long long plane, ldp;
  float* table; long long ldt;
  int region, per_row;
  int nb1, nb2;                        // problems of two batch dimensions, with their strides in elements
  long long src1, src2, dst1, dst2, tab1, tab2;
};
int oc_split_launch(const OcSplitArgs& a, cudaStream_t stream);

struct OcSplitOperand {
  const __half* planes; long long plane, ld;    // hi plane, distance of the lo plane, row pitch (elements)
  int mn_major;                                  // 0: stored [rows, K]; 1: stored [K, rows]
  int terms;                                     // 2; 1: there is no lo plane (A, stored [rows, K], only)
  const float* scale;                            // null: 1
  long long scale_k, scale_r;                    // table step per 128 values of k, per 128 rows
  int scale_row;                                 // A only: 1 when the table has an entry per row
  long long stride1, stride2, scale1, scale2;    // between the problems of the two batch dimensions
};

// Where a result goes on as an operand: its planes and table as oc_split_launch writes them, beside C or instead of it.
enum : int { OC_SPLIT_OUT_NONE = 0, OC_SPLIT_OUT_ROWS = 1, OC_SPLIT_OUT_BLOCKS = 2 };
struct OcSplitOut {
  int mode;                                      // none, every row of a block scaled for itself, blocks
  int only;                                      // C is scratch: nobody reads it
  __half* planes; long long plane, ld;
  float* table; long long ldt;
  long long stride1, stride2, tab1, tab2;
};

// C[M,N] = alpha * A * B^T, or C += alpha * A * B^T (add), A [M,K], B [N,K] (logical); flags as in OcGemm.
// C is written by TMA in 16-byte pieces: up to three columns behind the last one of a row are overwritten.
struct OcSplitGemm {
  OcSplitOperand A, B;
  float* C; long long ldc, strideC1, strideC2;
  int M, N, K, nb1, nb2;
  float alpha;
  int add, flags;
  OcSplitOut out;              // (not with add or lower tiles only)
};
int oc_gemm_split_launch(const OcSplitGemm& g, cudaStream_t stream);

// The split products are in use unless oc_set_gemm_engine pins the FMA engine.
bool oc_split_engine_on();
