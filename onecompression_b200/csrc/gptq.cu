// GPTQ column loop for one Linear weight, given the inverse-Hessian factor U.
//
// Follows run_gptq of the reference (onecomp/quantizer/gptq/_gptq.py:646-794) in fp32 with its
// roundings: quotients rounded like true divides (by a reciprocal and its correction where that
// provably gives the same value, by a division where not), round-half-to-even, the rank-1 update as a
// rounded product followed by a rounded subtraction (this file is compiled with -fmad=false and
// uses the _rn intrinsics besides).
//
// Rows of W are independent given U.  A block of up to 128 columns is worked off 16 columns (a
// window) at a time in registers, by one of three kernels with the same bits:
//   gptq_group_kernel   up to four full blocks in one launch, one set of 32 rows per SM at most: the windows of
//                       gptq_window_kernel, and the updates from block to block on the tensor core meanwhile
//   gptq_window_kernel  full blocks with up to two sets of 32 rows per SM: eight warps share 32 rows, one
//                       warp per window; the errors of a window go to the later warps through shared
//                       memory and named barriers
//   gptq_block_kernel   everything else: one thread owns one row, whose block lives in shared memory;
//                       in CTAs with few rows the other threads apply the updates behind the window
// The lazy-batch trailing update W[:, i2:] -= Err * U[i1:i2, i2:] is a tensor-core product of operands in two fp16
// planes each (split.cuh): U is split once per call, the column kernels leave the errors of a block of 128
// columns split, transposed, every row under a scale of its own.  2 and 3 bits, other block sizes, unaligned
// workspaces and the FMA engine take fp32 errors and oc_gemm_f32_launch.  Codes are kept
// transposed ([column][row], 16 bit) until a final pass packs them in original column order.
#include "split_tc.cuh"
#include <type_traits>

namespace {

constexpr int BLK = 128;      // maximum GPTQ block size handled by the column kernel
constexpr int SUB = 16;       // columns held in registers at a time
constexpr int WS = BLK + 4;   // shared tile row stride in floats (odd multiple of 16 bytes)
constexpr int SUPER = 4;      // blocks per far trailing update (see oc_gptq_quantize)

struct ColArgs {
  const float* Wf; long long ldw;
  int out, d, i1, count;
  const float* U; long long ldu;
  float* ErrT; long long lde;   // errors [column][row], fp32; not used when they leave as planes
  __half* errp; long long err_plane; float* err_scale;   // planes [column][row] and 2^-e per row; null: fp32
  unsigned short* codesT;
  float* scales; float* zeros;  // [G][out] fp32 (G = 1 for per-channel)
  int gs, maxq, sym;
  int mse_steps; float mse_grid, mse_norm;   // mse_steps = 0: plain min/max fit
  // batched problems (blockIdx.y): element strides between consecutive problems, 0 for one problem
  long long sW, sU, sE, sC, sS;
  long long sEp, sEs;
  int batch;
  float minus_one;               // for update4
};

// t -= e * u, product and difference rounded each for itself, two entries per instruction.  The difference is the FMA
// t + p * -1, which rounds like t - p; -1 comes in as a kernel argument, because the assembler contracts a
// packed product and sum that it can see into one FMA (other bits).  28672 rows, general kernel: 48.4 -> 44 us a block,
// bound by issue slots (0.6 instructions a cycle and scheduler with two warps on it).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void update2(float& t0, float& t1, f32x2 e2, float u0, float u1, f32x2 m2) {
  f32x2 t = pack2(t0, t1), p;
  const f32x2 u = pack2(u0, u1);
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(e2), "l"(u));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t) : "l"(p), "l"(m2), "l"(t));
  unpack2(t, t0, t1);
}

// columns c .. c + 3 of a row's errors to their planes
__device__ __forceinline__ void store_halves(__half* to, long long lde, long long plane, uint2 hi, uint2 lo) {
  const unsigned h[2] = {hi.x, hi.y}, l[2] = {lo.x, lo.y};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    to[j * lde] = __ushort_as_half((unsigned short)(h[j >> 1] >> (16 * (j & 1))));
    to[plane + j * lde] = __ushort_as_half((unsigned short)(l[j >> 1] >> (16 * (j & 1))));
  }
}
__device__ __forceinline__ void store_split4(__half* to, long long lde, long long plane, float4 v, float s) {
  uint2 hi, lo;
  oc_split4(make_float4(v.x * s, v.y * s, v.z * s, v.w * s), hi, lo);
  store_halves(to, lde, plane, hi, lo);
}

// scale / zero over the values v[0..n), reference: GPTQExcecutor.find_params
// (onecomp/quantizer/gptq/_gptq.py:886-972, perchannel=True, mse=False)
__device__ __forceinline__ void params_from_range(float& mn, float& mx, int maxq, int sym,
                                                  float& scale, float& zero) {
  // mn <= 0 <= mx on entry; on exit they hold the range the parameters were derived from
  if (sym) {
    mx = fmaxf(fabsf(mn), mx);
    if (mn < 0.f) mn = -mx;
  }
  if (mn == 0.f && mx == 0.f) { mn = -1.f; mx = 1.f; }
  scale = __fdiv_rn(__fsub_rn(mx, mn), (float)maxq);
  zero = sym ? (float)(maxq + 1) * 0.5f : rintf(__fdiv_rn(-mn, scale));
}

// |scale*(q - zero) - v|^norm for one value under candidate parameters (the error term of the
// reference's shrink search, :928-950)
__device__ __forceinline__ float mse_term(float v, float scale, float zero, float maxqf, float norm) {
  float q = __fadd_rn(rintf(__fdiv_rn(v, scale)), zero);
  q = fminf(fmaxf(q, 0.f), maxqf);
  const float dq = __fmul_rn(scale, __fsub_rn(q, zero));
  return powf(fabsf(__fsub_rn(dq, v)), norm);
}

// candidate i of the shrink search: range scaled by p = 1 - i/grid
__device__ __forceinline__ void mse_candidate(int i, float grid, float mn, float mx, int maxq, int sym,
                                              float zero_sym, float& scale1, float& zero1) {
  const float p = (float)(1.0 - (double)i / (double)grid);
  const float mn1 = __fmul_rn(p, mn), mx1 = __fmul_rn(p, mx);
  scale1 = __fdiv_rn(__fsub_rn(mx1, mn1), (float)maxq);
  zero1 = sym ? zero_sym : rintf(__fdiv_rn(-mn1, scale1));
}

// Group parameters are fitted on the block-entry values of columns col .. col+gs-1 (the
// reference, :737-745, reads the matrix, not the block copy).  Kept out of line: it runs once
// per group and would otherwise be replicated in every unrolled column step.
__device__ __noinline__ void fit_group(const float* __restrict__ src, int n, int maxq, int sym,
                                       int mse_steps, float grid, float norm, float* scale, float* zero) {
  float mn = 0.f, mx = 0.f;
  int t0 = 0;
  // eight columns at a time in flight (the extrema do not depend on the order); the values of a
  // group lie in the shared tile or in the matrix, 16-byte aligned in the usual shapes
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    float mn4[4] = {0.f, 0.f, 0.f, 0.f}, mx4[4] = {0.f, 0.f, 0.f, 0.f};
    for (; t0 + 8 <= n; t0 += 8) {
      const float4 a = *reinterpret_cast<const float4*>(src + t0), b = *reinterpret_cast<const float4*>(src + t0 + 4);
      mn4[0] = fminf(mn4[0], fminf(a.x, b.x)); mx4[0] = fmaxf(mx4[0], fmaxf(a.x, b.x));
      mn4[1] = fminf(mn4[1], fminf(a.y, b.y)); mx4[1] = fmaxf(mx4[1], fmaxf(a.y, b.y));
      mn4[2] = fminf(mn4[2], fminf(a.z, b.z)); mx4[2] = fmaxf(mx4[2], fmaxf(a.z, b.z));
      mn4[3] = fminf(mn4[3], fminf(a.w, b.w)); mx4[3] = fmaxf(mx4[3], fmaxf(a.w, b.w));
    }
    mn = fminf(fminf(mn4[0], mn4[1]), fminf(mn4[2], mn4[3]));
    mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
  }
  for (int t = t0; t < n; ++t) { const float v = src[t]; mn = fminf(mn, v); mx = fmaxf(mx, v); }
  float s, z;
  params_from_range(mn, mx, maxq, sym, s, z);
  if (mse_steps > 0) {
    float best = __int_as_float(0x7f800000), bs = s, bz = z;
    for (int i = 0; i < mse_steps; ++i) {
      float s1, z1;
      mse_candidate(i, grid, mn, mx, maxq, sym, z, s1, z1);
      float err = 0.f;
      for (int t = 0; t < n; ++t) err += mse_term(src[t], s1, z1, (float)maxq, norm);
      if (err < best) { best = err; bs = s1; bz = z1; }
    }
    s = bs; z = bz;
  }
  *scale = s; *zero = z;
}

// WARPS*32 rows per CTA; the CTA always has LOADERS threads.  The threads beyond the rows load the
// tiles, and when a CTA owns few rows (WARPS <= 2) they also take over the deferred updates: after
// each window of SUB columns the row owners publish the window's errors, the helper threads first
// bring the next window's columns up to date (the owners wait for that), then the rest of the block
// while the owners already work on the next window.  Every element still receives its updates in
// ascending order of the source column with the same two roundings each, so results do not depend
// on who applies them.
constexpr int LOADERS = 256;

__device__ __forceinline__ void apply_window(float4& t, const float* __restrict__ es, const float* __restrict__ us, f32x2 m2) {
  // es: this row's SUB errors (stride = rows of the CTA is folded in by the caller); us: U rows of the window
#pragma unroll
  for (int i = 0; i < SUB; ++i) {
    const f32x2 e2 = pack2(es[i], es[i]);
    const float4 u = *reinterpret_cast<const float4*>(us + i * BLK);
    update2(t.x, t.y, e2, u.x, u.y, m2);
    update2(t.z, t.w, e2, u.z, u.w, m2);
  }
}

// w[j] -= e * u[j] for the columns behind column i of the window (product and difference rounded)
__device__ __forceinline__ void propagate(float (&w)[SUB], int i, float e, const float* __restrict__ urow) {
  const float4* up = reinterpret_cast<const float4*>(urow);
#pragma unroll
  for (int j4 = (i + 1) / 4; j4 < SUB / 4; ++j4) {
    const float4 u = up[j4];
    if (4 * j4 + 0 > i) w[4 * j4 + 0] = __fsub_rn(w[4 * j4 + 0], __fmul_rn(e, u.x));
    if (4 * j4 + 1 > i) w[4 * j4 + 1] = __fsub_rn(w[4 * j4 + 1], __fmul_rn(e, u.y));
    if (4 * j4 + 2 > i) w[4 * j4 + 2] = __fsub_rn(w[4 * j4 + 2], __fmul_rn(e, u.z));
    if (4 * j4 + 3 > i) w[4 * j4 + 3] = __fsub_rn(w[4 * j4 + 3], __fmul_rn(e, u.w));
  }
}

// ---- the column step without divisions ------------------------------------------------------
// What bounds a block of columns is the chain from one column of a row to the next: quotient,
// rounding, quotient, update.  With two IEEE divisions and rintf it was about 440 cycles; the same
// values come out of about 15 dependent additions and multiplications:
//
//  * rint(x / scale) from t = x * (1 / scale).  t and the rounded quotient both lie within
//    3 * 2^-24 |t| of the true one, so they round to the same integer unless a half-integer is that
//    near to t.  Such a column (and any non-finite t) makes the caller repeat the window with
//    divisions.  Rounding to the nearest integer is the addition and subtraction of 1.5 * 2^23.
//  * clamp(rint + zero, 0, maxq) - zero = clamp(rint, -zero, maxq - zero): all are integers below 2^24.
//  * (x - dq) / u from the rounded reciprocal y of u: q1 = q0 + (r - q0 u) y is within one ulp of the
//    quotient, and then q1 + (r - q1 u) y is the correctly rounded quotient (P. Markstein, Computation
//    of elementary functions on the IBM RISC System/6000 processor, 1990, theorem 8.3), provided
//    nothing over- or underflows: operands outside 2^-60 .. 2^60 also go the exact way.
constexpr float SAFE_LO = 0x1p-60f, SAFE_HI = 0x1p60f;

__device__ __forceinline__ float safe_reciprocal(float u) {
  // NaN where the division-free step must not be used: it poisons the error, which is checked
  return (u >= SAFE_LO && u <= SAFE_HI) ? __frcp_rn(u) : __int_as_float(0x7fffffff);
}

// One window of SUB columns of one row; false if it has to be repeated with divisions (w is not
// changed in shared memory; codes and errors already stored are overwritten by the repetition).
template <int NROWS>
__device__ __forceinline__ bool fast_window(const float* __restrict__ wcols, const float* __restrict__ ublk,
                                            const float* __restrict__ rdiag, float scale, float zero, float maxqf,
                                            unsigned short* code_out, long long ldc, float* err_out, long long lde,
                                            bool fp32_errors, float (&er)[SUB]) {
  constexpr float RINT = 12582912.f;   // 1.5 * 2^23
  float w[SUB];
#pragma unroll
  for (int v = 0; v < SUB / 4; ++v) {
    const float4 t = *reinterpret_cast<const float4*>(wcols + 4 * v);
    w[4 * v] = t.x; w[4 * v + 1] = t.y; w[4 * v + 2] = t.z; w[4 * v + 3] = t.w;
  }
  const float rs = safe_reciprocal(scale);
  const float lo = __fsub_rn(0.f, zero), hi = __fsub_rn(maxqf, zero);
  bool bad = !(fabsf(zero) < 65536.f);
#pragma unroll
  for (int i = 0; i < SUB; ++i) {
    const float x = w[i];
    const float t = __fmul_rn(x, rs);
    const float n = __fsub_rn(__fadd_rn(t, RINT), RINT);
    bad |= !(__fmaf_rn(fabsf(t), 0x1p-21f, fabsf(__fsub_rn(t, n))) < 0.5f);
    const float level = fminf(fmaxf(n, lo), hi);
    const float r = __fsub_rn(x, __fmul_rn(scale, level));
    bad |= (__float_as_uint(r) * 2u - 1u) < (__float_as_uint(SAFE_LO) * 2u - 1u);   // tiny and not zero
    const float u = ublk[i * BLK + i], y = rdiag[i];
    const float q0 = __fmul_rn(r, y);
    const float q1 = __fmaf_rn(__fmaf_rn(-q0, u, r), y, q0);
    const float e = __fmaf_rn(__fmaf_rn(-q1, u, r), y, q1);
    bad |= !(fabsf(r) < SAFE_HI) || !(fabsf(e) < 0x1p120f);
    er[i] = e;
    code_out[i * ldc] = (unsigned short)__fadd_rn(level, zero);
    if (fp32_errors) err_out[i * lde] = e;
    propagate(w, i, e, ublk + i * BLK);
  }
  return !bad;
}

// ALIGNED: every group starts on a multiple of SUB columns (per-channel, or a group size that is
// a multiple of SUB), so the fit can only fall on the first column of a register window and the
// other fifteen unrolled column steps carry no test and no call site for it.
template <int WARPS, bool ALIGNED>
__global__ void __launch_bounds__(LOADERS) gptq_block_kernel(ColArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int NROWS = WARPS * 32;
  constexpr bool HELPERS = WARPS <= 2;
  float* Us = sm;               // [BLK][BLK], upper triangle of the diagonal block of U
  float* Ws = sm + BLK * BLK;   // [NROWS][WS], block-entry values of the rows' columns
  float* rdiag = Ws + NROWS * WS;   // [BLK] reciprocals of U's diagonal
  float* Es = rdiag + BLK;          // [2][SUB][NROWS] errors of the last two windows (helpers only)
  oc_wait_before();
  const int tid = threadIdx.x;
  const int row0 = blockIdx.x * NROWS;
  const int count = a.count, i1 = a.i1;
  {
    const long long b = blockIdx.y;      // problem of a batch
    a.Wf += b * a.sW; a.U += b * a.sU; a.ErrT += b * a.sE; a.codesT += b * a.sC;
    a.scales += b * a.sS; a.zeros += b * a.sS;
    if (a.errp) { a.errp += b * a.sEp; a.err_scale += b * a.sEs; }
  }

  // whole block, 16-byte aligned rows: vector loads (the part of U below the diagonal is never used)
  const bool vec = count == BLK && (i1 & 3) == 0 && (a.ldu & 3) == 0 && (a.ldw & 3) == 0 &&
                   ((reinterpret_cast<uintptr_t>(a.U) | reinterpret_cast<uintptr_t>(a.Wf)) & 15) == 0;
  if (vec) {
#pragma unroll
    for (int it = 0; it < BLK * BLK / 4 / LOADERS; ++it) {
      const int e = it * LOADERS + tid, i = e / (BLK / 4), j4 = e % (BLK / 4);
      *reinterpret_cast<float4*>(Us + i * BLK + 4 * j4) =
          *reinterpret_cast<const float4*>(a.U + (long long)(i1 + i) * a.ldu + i1 + 4 * j4);
    }
#pragma unroll
    for (int it = 0; it < NROWS * BLK / 4 / LOADERS; ++it) {
      const int e = it * LOADERS + tid, r = e / (BLK / 4), c4 = e % (BLK / 4);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row0 + r < a.out) v = *reinterpret_cast<const float4*>(a.Wf + (long long)(row0 + r) * a.ldw + i1 + 4 * c4);
      *reinterpret_cast<float4*>(Ws + r * WS + 4 * c4) = v;
    }
  } else {
    for (int e = tid; e < BLK * BLK; e += LOADERS) {
      const int i = e / BLK, j = e % BLK;
      Us[e] = (i < count && j < count && j >= i) ? a.U[(long long)(i1 + i) * a.ldu + i1 + j] : 0.f;
    }
    for (int e = tid; e < NROWS * BLK; e += LOADERS) {
      const int r = e / BLK, c = e % BLK;
      Ws[r * WS + c] = (row0 + r < a.out && c < count) ? a.Wf[(long long)(row0 + r) * a.ldw + i1 + c] : 0.f;
    }
  }
  if (ALIGNED) {
    __syncthreads();
    if (tid < BLK) rdiag[tid] = safe_reciprocal(Us[tid * BLK + tid]);
  }
  __syncthreads();

  const int row = row0 + tid;
  const bool owner = tid < NROWS && row < a.out;
  // helpers take the deferred updates when the block's columns come in whole groups of four
  const bool helped = HELPERS && (count & 3) == 0;
  if (!helped && !owner) return;
  float* wrow = Ws + (owner ? tid : 0) * WS;
  const float* grow = a.Wf + (long long)(owner ? row : 0) * a.ldw;  // block-entry state of the whole row
  const float maxqf = (float)a.maxq;
  const f32x2 m2 = pack2(a.minus_one, a.minus_one);
  const int gs = a.gs;
  unsigned short* code_out = a.codesT + (long long)i1 * a.out + row;   // + column * out
  float* err_out = a.ErrT + row;                                        // + column * lde
  float scale = 1.f, zero = 0.f;
  if (owner) {
    if (gs == -1) { scale = a.scales[row]; zero = a.zeros[row]; }
    else if (i1 % gs != 0) {
      // the block starts inside a group opened by an earlier block: continue with its parameters
      scale = a.scales[(long long)(i1 / gs) * a.out + row];
      zero = a.zeros[(long long)(i1 / gs) * a.out + row];
    }
  }
  // helper thread -> (row, every nsel-th group of four columns)
  constexpr int NSEL = HELPERS ? (LOADERS - NROWS) / NROWS : 1;
  const int hrow = (tid - NROWS) % NROWS, gsel = (tid - NROWS) / NROWS;
  const bool helper = helped && tid >= NROWS && gsel < NSEL;

  // parameters of the group that starts at column i1 + ci of the row
  auto open_group = [&](int ci) {
    const int col = i1 + ci, n = min(gs, a.d - col);
    // the shared tile is still pristine only at the very first column of the block
    fit_group((ci == 0 && n <= count) ? wrow : grow + col, n, a.maxq, a.sym, a.mse_steps, a.mse_grid,
              a.mse_norm, &scale, &zero);
    const long long g = col / gs;
    a.scales[g * a.out + row] = scale;
    a.zeros[g * a.out + row] = zero;
  };

  for (int cb = 0; cb < count; cb += SUB) {
    float* es_buf = Es + ((cb / SUB) & 1) * SUB * NROWS;
    if (owner) {
      float er[SUB];
      bool exact = !ALIGNED || cb + SUB > count;
      if (ALIGNED) {
        if (gs != -1 && (i1 + cb) % gs == 0) open_group(cb);
        if (!exact)
          exact = !fast_window<NROWS>(wrow + cb, Us + cb * BLK + cb, rdiag + cb, scale, zero, maxqf,
                                      code_out + (long long)cb * a.out, a.out, err_out + (long long)cb * a.lde,
                                      a.lde, a.errp == nullptr, er);
      }
      if (exact) {
        float w[SUB];
#pragma unroll
        for (int v = 0; v < SUB / 4; ++v) {
          const float4 t = *reinterpret_cast<const float4*>(wrow + cb + 4 * v);
          w[4 * v] = t.x; w[4 * v + 1] = t.y; w[4 * v + 2] = t.z; w[4 * v + 3] = t.w;
        }
#pragma unroll
        for (int i = 0; i < SUB; ++i) {
          const int ci = cb + i;
          er[i] = 0.f;
          if (ci < count) {
            if (!ALIGNED && gs != -1 && (i1 + ci) % gs == 0) open_group(ci);
            const float x = w[i];
            float q = __fadd_rn(rintf(__fdiv_rn(x, scale)), zero);
            q = fminf(fmaxf(q, 0.f), maxqf);
            const float dq = __fmul_rn(scale, __fsub_rn(q, zero));
            const float e = __fdiv_rn(__fsub_rn(x, dq), Us[ci * BLK + ci]);
            er[i] = e;
            code_out[(long long)ci * a.out] = (unsigned short)q;
            if (!a.errp) err_out[(long long)ci * a.lde] = e;
            propagate(w, i, e, Us + ci * BLK + cb);
          }
        }
      }
      if (a.errp) {
        // the columns of the tile that are done with hold their errors
#pragma unroll
        for (int v = 0; v < SUB / 4; ++v)
          *reinterpret_cast<float4*>(wrow + cb + 4 * v) = make_float4(er[4 * v], er[4 * v + 1], er[4 * v + 2], er[4 * v + 3]);
      }
      if (helped) {
#pragma unroll
        for (int i = 0; i < SUB; ++i) es_buf[i * NROWS + tid] = er[i];
      } else {
        // Later columns of the block receive this sub-block's updates now, in the
        // same order (ascending source column) and with the same two roundings each.
        for (int jc = cb + SUB; jc < count; jc += 8) {
          float4 t0 = *reinterpret_cast<const float4*>(wrow + jc);
          float4 t1 = *reinterpret_cast<const float4*>(wrow + jc + 4);
#pragma unroll
          for (int i = 0; i < SUB; ++i) {
            const f32x2 e2 = pack2(er[i], er[i]);
            const float4 u0 = *reinterpret_cast<const float4*>(Us + (cb + i) * BLK + jc);
            const float4 u1 = *reinterpret_cast<const float4*>(Us + (cb + i) * BLK + jc + 4);
            update2(t0.x, t0.y, e2, u0.x, u0.y, m2);
            update2(t0.z, t0.w, e2, u0.z, u0.w, m2);
            update2(t1.x, t1.y, e2, u1.x, u1.y, m2);
            update2(t1.z, t1.w, e2, u1.z, u1.w, m2);
          }
          *reinterpret_cast<float4*>(wrow + jc) = t0;
          *reinterpret_cast<float4*>(wrow + jc + 4) = t1;
        }
      }
    }
    if (helped) {
      if (cb + SUB >= count) break;         // the last window has nothing to its right
      __syncthreads();                      // the window's errors are published
      const int g_first = (cb + SUB) / 4, g_urgent = min(count, cb + 2 * SUB) / 4, g_end = count / 4;
      if (helper) {
        // the next window's columns first: the row owners wait for these
        for (int g = g_first; g < g_urgent; ++g) {
          if (g % NSEL != gsel) continue;
          float4 t = *reinterpret_cast<const float4*>(Ws + hrow * WS + 4 * g);
          float er[SUB];
#pragma unroll
          for (int i = 0; i < SUB; ++i) er[i] = es_buf[i * NROWS + hrow];
          apply_window(t, er, Us + cb * BLK + 4 * g, m2);
          *reinterpret_cast<float4*>(Ws + hrow * WS + 4 * g) = t;
        }
      }
      __syncthreads();                      // the next window may start
      if (helper) {
        float er[SUB];
#pragma unroll
        for (int i = 0; i < SUB; ++i) er[i] = es_buf[i * NROWS + hrow];
        for (int g = g_urgent; g < g_end; ++g) {
          if (g % NSEL != gsel) continue;
          float4 t = *reinterpret_cast<const float4*>(Ws + hrow * WS + 4 * g);
          apply_window(t, er, Us + cb * BLK + 4 * g, m2);
          *reinterpret_cast<float4*>(Ws + hrow * WS + 4 * g) = t;
        }
      }
    }
  }
  oc_let_next();
  if (a.errp && owner) {        // a full block
    float mx = 0.f;
#pragma unroll 4
    for (int c = 0; c < BLK; c += 4) {
      const float4 v = *reinterpret_cast<const float4*>(wrow + c);
      mx = fmaxf(mx, fmaxf(fmaxf(oc_finite_abs(v.x), oc_finite_abs(v.y)), fmaxf(oc_finite_abs(v.z), oc_finite_abs(v.w))));
    }
    float inv;
    const float s = oc_split_scale(mx, inv);
    a.err_scale[row] = inv;
#pragma unroll 4
    for (int c = 0; c < BLK; c += 4)
      store_split4(a.errp + (long long)c * a.lde + row, a.lde, a.err_plane, *reinterpret_cast<const float4*>(wrow + c), s);
  }
}

// ---- full blocks: one warp per window ---------------------------------------------------------
// A full block of 128 columns whose groups start on window boundaries (every block of the usual
// settings).  Eight warps share 32 rows (lane = row), warp k keeps the window of columns 16k .. 16k+15
// in registers.  The window whose turn it is produces four columns at a time and publishes their errors;
// the warps of later windows apply them while it goes on, so that at its turn a window lacks the last
// four columns only.  Group parameters are fitted on block-entry values (see fit_group), so those of
// all groups of the block are found before the chain starts; codes and errors go to global memory when
// the next window has its turn.  Every element receives its updates in ascending order of the source
// column with the two roundings of the general kernel: same bits.
//
// What bounds it is the chain over the columns.  With the general kernel, whose helper threads the row
// owners wait for after each window, a block took 20 us at 4096 rows; now 14 us.  It is for up to
// two row sets per SM: a load from shared memory delivers 32 lanes 4 bytes each a cycle, broadcast or not,
// and one entry of U per row and column is twice what the arithmetic of the updates takes, so with many
// rows the general kernel's is the better split (28672 rows: 44 us there, 73 us here with
// two rows per lane).

// one column with IEEE divisions: (error, code)
__device__ __noinline__ float2 exact_column(float x, float scale, float zero, float maxqf, float u) {
  float q = __fadd_rn(rintf(__fdiv_rn(x, scale)), zero);
  q = fminf(fmaxf(q, 0.f), maxqf);
  return make_float2(__fdiv_rn(__fsub_rn(x, __fmul_rn(scale, __fsub_rn(q, zero))), u), q);
}

constexpr int NWIN = BLK / SUB, CHUNK = 4;    // windows of a block; columns published at once

// columns 4Q .. 4Q+3 of a window: errors to `es` (32 per column) and er, codes to cd.  False if a
// column of this lane has to be repeated with divisions.
template <int Q, bool EXACT>
__device__ __forceinline__ bool produce_chunk(float (&w)[SUB], const float* __restrict__ ublk,
                                              const float* __restrict__ rdiag, float scale, float rs, float lo,
                                              float hi, float zero, float maxqf, float* es, float (&er)[SUB],
                                              float (&cd)[SUB]) {
  constexpr float RINT = 12582912.f;   // 1.5 * 2^23
  bool bad = !(fabsf(zero) < 65536.f);
#pragma unroll
  for (int c = 0; c < CHUNK; ++c) {
    const int i = Q * CHUNK + c;
    const float x = w[i], u = ublk[i * BLK + i];
    if (EXACT) {
      const float2 v = exact_column(x, scale, zero, maxqf, u);
      er[i] = v.x;
      cd[i] = v.y;
    } else {
      const float t = __fmul_rn(x, rs);
      const float n = __fsub_rn(__fadd_rn(t, RINT), RINT);
      bad |= !(__fmaf_rn(fabsf(t), 0x1p-21f, fabsf(__fsub_rn(t, n))) < 0.5f);
      const float level = fminf(fmaxf(n, lo), hi);
      const float r = __fsub_rn(x, __fmul_rn(scale, level));
      bad |= (__float_as_uint(r) * 2u - 1u) < (__float_as_uint(SAFE_LO) * 2u - 1u);   // tiny and not zero
      const float y = rdiag[i];
      const float q0 = __fmul_rn(r, y);
      const float q1 = __fmaf_rn(__fmaf_rn(-q0, u, r), y, q0);
      const float e = __fmaf_rn(__fmaf_rn(-q1, u, r), y, q1);
      bad |= !(fabsf(r) < SAFE_HI) || !(fabsf(e) < 0x1p120f);
      er[i] = e;
      cd[i] = __fadd_rn(level, zero);
    }
    propagate(w, i, er[i], ublk + i * BLK);
  }
  // (not column by column: the loads of U would have to stay behind the stores)
#pragma unroll
  for (int c = 0; c < CHUNK; ++c) es[c * 32] = er[Q * CHUNK + c];
  return !bad;
}

// The chain over the columns of a block, from the view of warp `wid`: w becomes the block-entry window with the updates
// of the earlier windows, then er and cd the errors and codes of the warp's own.
__device__ __forceinline__ void window_chain(int wid, int lane, float (&w)[SUB], const float* __restrict__ Us,
                                             const float* __restrict__ rdiag, float* Es, float scale, float zero,
                                             float maxqf, f32x2 m2, float (&er)[SUB], float (&cd)[SUB]) {
  const float rs = safe_reciprocal(scale);
  const float lo = __fsub_rn(0.f, zero), hi = __fsub_rn(maxqf, zero);

  // the windows before this warp's own: their errors, as they are published.  Named barriers 1 .. 4 stand for
  // the four chunks of a window (its producer arrives, the warps of later windows wait), barrier 5 for
  // the end of a window, behind which the next one may publish.
#pragma unroll 1
  for (int pw = 0; pw < wid; ++pw) {
    const int threads = 32 * (NWIN - pw);
#pragma unroll 1
    for (int q = 0; q < SUB / CHUNK; ++q) {
      asm volatile("bar.sync %0, %1;" ::"r"(q + 1), "r"(threads) : "memory");
      const float* es = Es + q * CHUNK * 32 + lane;
      const float* ur = Us + (pw * SUB + q * CHUNK) * BLK + wid * SUB;
#pragma unroll
      for (int c = 0; c < CHUNK; ++c) {
        const f32x2 e2 = pack2(es[c * 32], es[c * 32]);
#pragma unroll
        for (int v = 0; v < SUB / 4; ++v) {
          const float4 u = *reinterpret_cast<const float4*>(ur + c * BLK + 4 * v);
          update2(w[4 * v], w[4 * v + 1], e2, u.x, u.y, m2);
          update2(w[4 * v + 2], w[4 * v + 3], e2, u.z, u.w, m2);
        }
      }
    }
    asm volatile("bar.sync 5, %0;" ::"r"(threads - 32) : "memory");
  }

  // this warp's own window
  const float* ublk = Us + wid * SUB * BLK + wid * SUB;
  auto step = [&](auto q_const) {
    constexpr int Q = decltype(q_const)::value;
    float* es = Es + Q * CHUNK * 32 + lane;
    float entry[SUB];
#pragma unroll
    for (int m = Q * CHUNK; m < SUB; ++m) entry[m] = w[m];
    if (!produce_chunk<Q, false>(w, ublk, rdiag, scale, rs, lo, hi, zero, maxqf, es, er, cd)) {
#pragma unroll
      for (int m = Q * CHUNK; m < SUB; ++m) w[m] = entry[m];
      produce_chunk<Q, true>(w, ublk, rdiag, scale, rs, lo, hi, zero, maxqf, es, er, cd);
    }
    if (wid < NWIN - 1) {
      __syncwarp();
      asm volatile("bar.arrive %0, %1;" ::"r"(Q + 1), "r"(32 * (NWIN - wid)) : "memory");
    }
  };
  step(std::integral_constant<int, 0>{});
  step(std::integral_constant<int, 1>{});
  step(std::integral_constant<int, 2>{});
  step(std::integral_constant<int, 3>{});
}

__global__ void __launch_bounds__(256, 2) gptq_window_kernel(ColArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* Us = sm;                                // [BLK][BLK], upper triangle of the diagonal block of U
  float* rdiag = Us + BLK * BLK;                 // [BLK] reciprocals of its diagonal
  float* mm_lo = rdiag + BLK, *mm_hi = mm_lo + NWIN * 32;      // [NWIN][32] range of every window
  float* ps = mm_hi + NWIN * 32, *pz = ps + NWIN * 32;         // parameters of the groups opened by every window
  float* Es = pz + NWIN * 32;                    // [SUB][32] errors of the window whose turn it is
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int i1 = a.i1, gs = a.gs;
  oc_wait_before();
  {
    const long long b = blockIdx.y;      // problem of a batch
    a.Wf += b * a.sW; a.U += b * a.sU; a.ErrT += b * a.sE; a.codesT += b * a.sC;
    a.scales += b * a.sS; a.zeros += b * a.sS;
    if (a.errp) { a.errp += b * a.sEp; a.err_scale += b * a.sEs; }
  }
  // everything that comes from global memory is requested before anything is waited for
#pragma unroll
  for (int it = 0; it < BLK * BLK / 4 / 256; ++it) {
    const int e = it * 256 + tid, i = e / (BLK / 4), j4 = e % (BLK / 4);
    if (4 * j4 + 3 >= i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                   ::"r"((unsigned)__cvta_generic_to_shared(Us + i * BLK + 4 * j4)),
                     "l"(a.U + (long long)(i1 + i) * a.ldu + i1 + 4 * j4) : "memory");
  }
  const int row = blockIdx.x * 32 + lane;
  const bool live = row < a.out;
  const int col0 = i1 + wid * SUB;               // this warp's window
  const int g = gs == -1 ? 0 : col0 / gs, opened = gs == -1 ? -1 : g * gs;   // first column of the window's group
  const float* grow = a.Wf + (long long)(live ? row : 0) * a.ldw;
  float4 t[SUB / 4];
#pragma unroll
  for (int v = 0; v < SUB / 4; ++v)
    t[v] = live ? *reinterpret_cast<const float4*>(grow + col0 + 4 * v) : make_float4(0.f, 0.f, 0.f, 0.f);
  float udiag = 0.f;
  if (tid < BLK) udiag = a.U[(long long)(i1 + tid) * a.ldu + i1 + tid];
  float scale = 1.f, zero = 0.f;
  if (opened < i1 && live) {                     // per channel, or opened by an earlier block
    scale = a.scales[(long long)g * a.out + row];
    zero = a.zeros[(long long)g * a.out + row];
  }
  float w[SUB], mn = 0.f, mx = 0.f;
#pragma unroll
  for (int v = 0; v < SUB / 4; ++v) {
    const float4 x = t[v];
    w[4 * v] = x.x; w[4 * v + 1] = x.y; w[4 * v + 2] = x.z; w[4 * v + 3] = x.w;
    mn = fminf(mn, fminf(fminf(x.x, x.y), fminf(x.z, x.w)));
    mx = fmaxf(mx, fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)));
  }
  mm_lo[wid * 32 + lane] = mn;
  mm_hi[wid * 32 + lane] = mx;
  if (tid < BLK) rdiag[tid] = safe_reciprocal(udiag);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (a.mse_steps == 0 && gs > 0 && BLK % gs == 0 && i1 % gs == 0) {
    // whole groups in the block: every window finds its group's parameters for itself
    const int first = (opened - i1) / SUB, wins = gs / SUB;
#pragma unroll
    for (int v = 0; v < NWIN; ++v)
      if (v < wins) {
        mn = fminf(mn, mm_lo[(first + v) * 32 + lane]);
        mx = fmaxf(mx, mm_hi[(first + v) * 32 + lane]);
      }
    params_from_range(mn, mx, a.maxq, a.sym, scale, zero);
    if (opened == col0 && live) {
      a.scales[(long long)g * a.out + row] = scale;
      a.zeros[(long long)g * a.out + row] = zero;
    }
  } else {
    if (opened == col0) {                        // this window opens a group
      if (live) {
        fit_group(grow + col0, min(gs, a.d - col0), a.maxq, a.sym, a.mse_steps, a.mse_grid, a.mse_norm, &scale, &zero);
        a.scales[(long long)g * a.out + row] = scale;
        a.zeros[(long long)g * a.out + row] = zero;
      }
      ps[wid * 32 + lane] = scale;
      pz[wid * 32 + lane] = zero;
    }
    __syncthreads();
    if (opened >= i1 && opened < col0) {
      scale = ps[(opened - i1) / SUB * 32 + lane];
      zero = pz[(opened - i1) / SUB * 32 + lane];
    }
  }
  float er[SUB], cd[SUB];
  window_chain(wid, lane, w, Us, rdiag + wid * SUB, Es, scale, zero, (float)a.maxq, pack2(a.minus_one, a.minus_one), er, cd);
  if (wid == NWIN - 1) oc_let_next();
  if (live) {
    unsigned short* code_out = a.codesT + (long long)col0 * a.out + row;
#pragma unroll
    for (int i = 0; i < SUB; ++i) code_out[(long long)i * a.out] = (unsigned short)cd[i];
    if (!a.errp) {
      float* err_out = a.ErrT + (long long)(wid * SUB) * a.lde + row;
#pragma unroll
      for (int i = 0; i < SUB; ++i) err_out[(long long)i * a.lde] = er[i];
    }
  }
  if (!a.errp) return;
  // the errors of a row leave under one scale, which is known when the last window is done
  float mxe = 0.f;
#pragma unroll
  for (int i = 0; i < SUB; ++i) mxe = fmaxf(mxe, oc_finite_abs(er[i]));
  mm_hi[wid * 32 + lane] = mxe;      // (its ranges were read before the chain)
  __syncthreads();
#pragma unroll
  for (int v = 0; v < NWIN; ++v) mxe = fmaxf(mxe, mm_hi[v * 32 + lane]);
  float inv;
  const float se = oc_split_scale(mxe, inv);
  if (!live) return;
  if (wid == 0) a.err_scale[row] = inv;
#pragma unroll
  for (int i = 0; i < SUB; i += 4)
    store_split4(a.errp + (long long)(wid * SUB + i) * a.lde + row, a.lde, a.err_plane,
                 make_float4(er[i], er[i + 1], er[i + 2], er[i + 3]), se);
}

int launch_windows(const ColArgs& a, cudaStream_t stream) {
  const int smem = (BLK * BLK + BLK + (4 * NWIN + SUB) * 32) * (int)sizeof(float);
  OC_OPT_IN_SMEM(gptq_window_kernel, smem);
  OC_LAUNCH(gptq_window_kernel, dim3(oc_div_up(a.out, 32), a.batch), 256, smem, stream, a);
  return OC_OK;
}

// the blocks that gptq_window_kernel takes
bool windows_fit(const ColArgs& a) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.count == BLK && a.i1 % SUB == 0 && (a.gs == -1 || a.gs % SUB == 0) && a.ldu % 4 == 0 && a.ldw % 4 == 0 &&
         aligned(a.U) && aligned(a.Wf) && (a.batch == 1 || (a.sU % 4 == 0 && a.sW % 4 == 0));
}

// ---- up to four full blocks in one launch ---------------------------------------------------------
// The blocks of one group of the lazy-batch update, 32 rows per CTA.  Between two blocks of gptq_window_kernel lie a
// launch of the product that updates the rest of the group and the start of the next kernel, 24 us a block at 4096 rows,
// of which the chain over the columns takes 11.  Here the update of the next 128 columns is 24 MMAs whose
// operand from U has been waiting in shared memory since the chain began, and those of the columns behind run
// while the next block's chain does: 14 us a block.  Bound by that chain (152 cycles a column, 19 of 23 thousand a block).
//
// D^T = U^T Err^T: M = 128 columns of W, N = the CTA's 32 rows, K = the 128 columns just quantized, accumulated as in
// gemm_split_kernel (same terms, order and chains: same bits), one accumulator of 32 TMEM columns for every pair
// of source and target block.  A target block reads its columns of W once, subtracts the accumulators of its
// sources in order and passes the result through shared memory to the windows.
//   warps 0..7  windows; between blocks TMEM lane quarter = warp % 4, i.e. 32 columns, and half of the rows
//   warp 8      TMA of U's planes, 32 k-values of 128 columns a stage
//   warp 9      MMA
// The group parameters are fitted on whole groups inside a block (128 a multiple of the group size) or given per channel.
constexpr int GROUP_STAGES = 4, GROUP_STAGE_BYTES = 2 * octc::SPLIT_MN_ATOM;    // 128 columns of both planes
constexpr int GROUP_ERR_BYTES = 2 * 32 * BLK * 2;                               // errors of 32 rows, both planes
constexpr int GROUP_SMEM = 1024 + GROUP_STAGES * GROUP_STAGE_BYTES + GROUP_ERR_BYTES +
                           (BLK * BLK + BLK * 33 + BLK + (2 * NWIN + SUB + SUPER) * 32) * 4;
struct GroupArgs {
  ColArgs c;                     // of the first block; errors of all blocks go to its planes, 128 rows a block
  int blocks;
  const float* u_table; long long u_tab_ld, u_tab_b;   // 2^-e of U's blocks
  int store_errors;              // something lies behind the group
  int* status;
};

__device__ __forceinline__ void bar_windows() { asm volatile("bar.sync 6, 256;" ::: "memory"); }

__global__ void __launch_bounds__(320, 1)
gptq_group_kernel(const __grid_constant__ CUtensorMap map_u, const GroupArgs ga) {
  using namespace octc;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[GROUP_STAGES], bar_empty[GROUP_STAGES], bar_err[SUPER], bar_acc[SUPER * SUPER], bar_u;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag_s;
  volatile int* abort_flag = &abort_flag_s;
  ColArgs a = ga.c;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, batch = blockIdx.y;
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t stage_base = smem_u32(base);
  uint8_t* err_s = base + GROUP_STAGES * GROUP_STAGE_BYTES;    // [plane][k / 64][row][64 k], 128-byte swizzle
  float* Us = reinterpret_cast<float*>(err_s + GROUP_ERR_BYTES);   // [BLK][BLK], upper triangle of the diagonal block of U
  float* tile = Us + BLK * BLK;                                // [BLK][33] entry values of a block, column by column
  float* rdiag = tile + BLK * 33;
  float* mm_lo = rdiag + BLK, *mm_hi = mm_lo + NWIN * 32;
  float* Es = mm_hi + NWIN * 32;                               // [SUB][32]
  float* inv_s = Es + SUB * 32;                                // [SUPER][32] 2^-e of the blocks' errors

  if (tid == 0) {
    for (int s = 0; s < GROUP_STAGES; ++s) { mbar_init(smem_u32(&bar_full[s]), 1); mbar_init(smem_u32(&bar_empty[s]), 1); }
    for (int j = 0; j < SUPER; ++j) mbar_init(smem_u32(&bar_err[j]), 1);
    mbar_init(smem_u32(&bar_u), 1);
    for (int j = 0; j < SUPER * SUPER; ++j) mbar_init(smem_u32(&bar_acc[j]), 1);
    abort_flag_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (wid == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  oc_wait_before();
  // accumulator of source block j and target block t
  auto acc_at = [&](int j, int t) { return tmem_base + (uint32_t)(t * (t - 1) / 2 + j) * 32u; };

  if (wid == 8) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 1;
      bool ok = true;
      for (int j = 0; j < ga.blocks && ok; ++j)
        for (int t = j + 1; t < ga.blocks && ok; ++t)
          for (int ks = 0; ks < BLK / SPLIT_BK; ++ks) {
            ok = mbar_wait(smem_u32(&bar_empty[stage]), phase, abort_flag, ga.status, 311);
            if (!ok) break;
            const uint32_t bar = smem_u32(&bar_full[stage]), dst = stage_base + stage * GROUP_STAGE_BYTES;
            mbar_expect_tx(bar, GROUP_STAGE_BYTES);
#pragma unroll
            for (int h = 0; h < 2; ++h)
              tma_load_planes(dst + h * SPLIT_MN_ATOM, &map_u, a.i1 + t * BLK + h * 64, a.i1 + j * BLK + ks * SPLIT_BK, batch, 0, bar);
            if (++stage == GROUP_STAGES) { stage = 0; phase ^= 1; }
          }
      if (!ok) {
        // let copies already issued land before the CTA's shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { }
      }
    }
    __syncwarp();
  } else if (wid == 9) {
    if (lane == 0) {
      constexpr uint32_t ID = split_idesc(true, false, BLK, 32);
      // errors: K-major rows of 64 k (128-byte swizzle), groups of 8 rows 1024 bytes apart
      auto err_desc = [&](int plane, int k16) {
        uint64_t d = (uint64_t)(((smem_u32(err_s) + plane * 8192 + (k16 >> 2) * 4096 + (k16 & 3) * 32) & 0x3FFFFu) >> 4);
        d |= (uint64_t)1 << 16;
        d |= (uint64_t)(1024 >> 4) << 32;
        d |= 1ull << 46;
        d |= 2ull << 61;
        return d;
      };
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int j = 0; j + 1 < ga.blocks && ok; ++j) {
        ok = mbar_wait(smem_u32(&bar_err[j]), 0, abort_flag, ga.status, 312);
        tc_fence_after();
        for (int t = j + 1; t < ga.blocks && ok; ++t) {
          const uint32_t d = acc_at(j, t);
          for (int ks = 0; ks < BLK / SPLIT_BK; ++ks) {
            ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag, ga.status, 313);
            if (!ok) break;
            tc_fence_after();
            const uint32_t u_hi = stage_base + stage * GROUP_STAGE_BYTES, u_lo = u_hi + SPLIT_MN_LO;
#pragma unroll
            for (int kk = 0; kk < SPLIT_BK / 16; ++kk) {
              const uint64_t uh = split_desc_mn(u_hi, kk), ul = split_desc_mn(u_lo, kk);
              const uint64_t eh = err_desc(0, ks * 2 + kk), el = err_desc(1, ks * 2 + kk);
              umma_f16(d, ul, eh, ID, (ks > 0 || kk > 0) ? 1u : 0u);
              umma_f16(d, uh, el, ID, 1u);
              umma_f16(d, uh, eh, ID, 1u);
            }
            umma_commit(smem_u32(&bar_empty[stage]));
            if (++stage == GROUP_STAGES) { stage = 0; phase ^= 1; }
          }
          if (ok) umma_commit(smem_u32(&bar_acc[j * SUPER + t]));
        }
      }
    }
    __syncwarp();
  } else {
    {
      const long long b = batch;
      a.Wf += b * a.sW; a.U += b * a.sU; a.codesT += b * a.sC; a.scales += b * a.sS; a.zeros += b * a.sS;
      a.errp += b * a.sEp; a.err_scale += b * a.sEs;
    }
    const float* u_table = ga.u_table + (long long)batch * ga.u_tab_b;
    const int row0 = blockIdx.x * 32, row = row0 + lane, gs = a.gs;
    const bool live = row < a.out;
    const int quarter = wid & 3, half = wid >> 2;       // of the columns / rows, between blocks
    const float maxqf = (float)a.maxq;
    float scale = 1.f, zero = 0.f;
    if (gs == -1 && live) { scale = a.scales[row]; zero = a.zeros[row]; }
    float wv[16], udiag = 0.f;
    // What block i1 needs from global memory.  U's block comes in bulk copies, a row from its diagonal on each (the
    // start rounded down to 16 bytes): 16 copies of 16 bytes by every thread took 2500 cycles of the chain.
    constexpr uint32_t U_BYTES = 4 * 4 * (BLK / 4) * (BLK / 4 + 1) / 2 * 4;
    auto expect_u = [&]() { mbar_expect_tx(smem_u32(&bar_u), U_BYTES); };       // one thread, before any copy
    auto request = [&](int i1) {
      if (lane < SUB) {
        const int i = wid * SUB + lane, j = i & ~3;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(Us + i * BLK + j)), "l"(a.U + (long long)(i1 + i) * a.ldu + i1 + j), "r"((BLK - j) * 4),
                       "r"(smem_u32(&bar_u)) : "memory");
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int rr = row0 + half * 16 + r;
        wv[r] = rr < a.out ? a.Wf[(long long)rr * a.ldw + i1 + quarter * 32 + lane] : 0.f;
      }
      if (tid < BLK) udiag = a.U[(long long)(i1 + tid) * a.ldu + i1 + tid];
    };
    if (tid == 0) expect_u();
    bar_windows();
    request(a.i1);

#pragma unroll 1
    for (int t = 0; t < ga.blocks; ++t) {
      const int i1 = a.i1 + t * BLK, col0 = i1 + wid * SUB;
      // ---- entry values: W minus the updates of the group's earlier blocks, in their order
#pragma unroll 1
      for (int j = 0; j < t; ++j) {
        const float fu = u_table[(long long)(a.i1 / BLK + j) * ga.u_tab_ld + a.i1 / BLK + t];
        mbar_wait(smem_u32(&bar_acc[j * SUPER + t]), 0, abort_flag, ga.status, 314);
        tc_fence_after();
        float v[16];
        tmem_ld16(acc_at(j, t) + ((uint32_t)(quarter * 32) << 16) + half * 16, v);
#pragma unroll
        for (int r = 0; r < 16; ++r) wv[r] = fmaf(-(inv_s[j * 32 + half * 16 + r] * fu), v[r], wv[r]);
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) tile[(quarter * 32 + lane) * 33 + half * 16 + r] = wv[r];
      if (tid < BLK) rdiag[tid] = safe_reciprocal(udiag);
      mbar_wait(smem_u32(&bar_u), t & 1, abort_flag, ga.status, 316);
      bar_windows();
      float w[SUB], mn = 0.f, mx = 0.f;
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
        w[i] = tile[(wid * SUB + i) * 33 + lane];
        mn = fminf(mn, w[i]);
        mx = fmaxf(mx, w[i]);
      }
      if (gs != -1) {
        // whole groups in the block: every window finds its group's parameters for itself
        mm_lo[wid * 32 + lane] = mn;
        mm_hi[wid * 32 + lane] = mx;
        bar_windows();
        const int g = col0 / gs, opened = g * gs, first = (opened - i1) / SUB, wins = gs / SUB;
#pragma unroll
        for (int v = 0; v < NWIN; ++v)
          if (v < wins) {
            mn = fminf(mn, mm_lo[(first + v) * 32 + lane]);
            mx = fmaxf(mx, mm_hi[(first + v) * 32 + lane]);
          }
        params_from_range(mn, mx, a.maxq, a.sym, scale, zero);
        if (opened == col0 && live) {
          a.scales[(long long)g * a.out + row] = scale;
          a.zeros[(long long)g * a.out + row] = zero;
        }
      }
      float er[SUB], cd[SUB];
      window_chain(wid, lane, w, Us, rdiag + wid * SUB, Es, scale, zero, maxqf, pack2(a.minus_one, a.minus_one), er, cd);
      // ---- the errors of a row leave under one scale, which is known when the last window is done
      float mxe = 0.f;
#pragma unroll
      for (int i = 0; i < SUB; ++i) mxe = fmaxf(mxe, oc_finite_abs(er[i]));
      bar_windows();                     // (the ranges have been read by all)
      mm_hi[wid * 32 + lane] = mxe;
      const bool more = t + 1 < ga.blocks;
      if (more && tid == 0) expect_u();
      bar_windows();
      if (!more) oc_let_next();
      if (more) request(i1 + BLK);       // (nobody reads this block of U any more)
#pragma unroll
      for (int v = 0; v < NWIN; ++v) mxe = fmaxf(mxe, mm_hi[v * 32 + lane]);
      float inv;
      const float se = oc_split_scale(mxe, inv);
      uint2 hi[4], lo[4];
#pragma unroll
      for (int v = 0; v < 4; ++v)
        oc_split4(make_float4(er[4 * v] * se, er[4 * v + 1] * se, er[4 * v + 2] * se, er[4 * v + 3] * se), hi[v], lo[v]);
      if (more) {
        // (the MMAs that read the previous block's errors are done: its last target's accumulator, waited for here)
        if (t > 0) mbar_wait(smem_u32(&bar_acc[(t - 1) * SUPER + ga.blocks - 1]), 0, abort_flag, ga.status, 315);
        uint8_t* to = err_s + (wid >> 2) * 4096 + lane * 128;
        const int c = (wid & 3) * 2;
        *reinterpret_cast<uint4*>(to + ((c ^ (lane & 7)) * 16)) = make_uint4(hi[0].x, hi[0].y, hi[1].x, hi[1].y);
        *reinterpret_cast<uint4*>(to + (((c + 1) ^ (lane & 7)) * 16)) = make_uint4(hi[2].x, hi[2].y, hi[3].x, hi[3].y);
        *reinterpret_cast<uint4*>(to + 8192 + ((c ^ (lane & 7)) * 16)) = make_uint4(lo[0].x, lo[0].y, lo[1].x, lo[1].y);
        *reinterpret_cast<uint4*>(to + 8192 + (((c + 1) ^ (lane & 7)) * 16)) = make_uint4(lo[2].x, lo[2].y, lo[3].x, lo[3].y);
        if (wid == 0) inv_s[t * 32 + lane] = inv;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bar_windows();
        if (tid == 0) mbar_arrive(smem_u32(&bar_err[t]));
      }
      if (live) {
        unsigned short* code_out = a.codesT + (long long)col0 * a.out + row;
#pragma unroll
        for (int i = 0; i < SUB; ++i) code_out[(long long)i * a.out] = (unsigned short)cd[i];
        if (ga.store_errors) {
          if (wid == 0) a.err_scale[(long long)t * a.lde + row] = inv;
          __half* to = a.errp + (long long)(t * BLK + wid * SUB) * a.lde + row;
#pragma unroll
          for (int v = 0; v < 4; ++v) store_halves(to + 4 * v * a.lde, a.lde, a.err_plane, hi[v], lo[v]);
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (wid == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem_base) : "memory");
  }
}

// the groups of blocks that gptq_group_kernel takes: `blocks` full blocks from column i1 on
bool group_fits(const ColArgs& a, int sm_count) {
  return (a.gs == -1 || (a.mse_steps == 0 && a.gs % SUB == 0 && BLK % a.gs == 0)) &&
         (long long)oc_div_up(a.out, 32) * a.batch <= sm_count;
}

int launch_group(const GroupArgs& a, const CUtensorMap& map_u, cudaStream_t stream) {
  OC_OPT_IN_SMEM(gptq_group_kernel, GROUP_SMEM);
  OC_LAUNCH(gptq_group_kernel, dim3(oc_div_up(a.c.out, 32), a.c.batch), 320, GROUP_SMEM, stream, map_u, a);
  return OC_OK;
}

// ---- preparation: fp16 -> fp32, act-order gather, dead columns, per-channel parameters ----
// Wf[r][j] = dead[perm[j]] ? 0 : float(W[r][perm[j]]).  Per-channel scale / zero are fitted on
// the whole original row before dead columns are zeroed (reference :690-695).
//
// One CTA per row, bound by HBM (2 bytes in, 4 out per weight).  The row is read in order, eight
// weights a thread, and with act-order passes through shared memory (`staged`: d floats), where the
// permutation is a gather on chip instead of one 2-byte global access per weight.  28672 x 4096:
// 313 us one weight per access, 106 us now; 4096 x 14336 with act-order 204, 107 us.
__global__ void __launch_bounds__(256)
gptq_prepare_kernel(const void* __restrict__ W, int bf16, long long ldw_in, int out, int d,
                    const int* __restrict__ perm, const unsigned char* __restrict__ dead,
                    float* __restrict__ Wf, long long ldw, int per_channel, int maxq,
                    int sym, int mse_steps, float mse_grid, float mse_norm,
                    float* __restrict__ scales, float* __restrict__ zeros,
                    long long s_win, long long s_wf, long long s_par, int vec, int staged) {
  extern __shared__ __align__(16) float row_s[];
  oc_wait_before();
  oc_let_next();
  const int row = blockIdx.x;
  {
    const long long b = blockIdx.y;      // problem of a batch
    W = static_cast<const char*>(W) + b * s_win * 2;
    Wf += b * s_wf; scales += b * s_par; zeros += b * s_par;
    if (perm) perm += b * d;
    if (dead) dead += b * d;
  }
  const long long src0 = (long long)row * ldw_in;
  float* dst = Wf + (long long)row * ldw;
  float mn = 0.f, mx = 0.f;
  if (perm && !staged) {
    for (int j = threadIdx.x; j < d; j += blockDim.x) {
      const int pj = perm[j];
      const float v = oc_ld16(W, src0 + pj, bf16);
      mn = fminf(mn, v); mx = fmaxf(mx, v);
      dst[j] = (dead && dead[pj]) ? 0.f : v;
    }
  } else {
    float* to = perm ? row_s : dst;
    if (vec) {          // d, ldw_in multiples of 8, 16-byte aligned rows (dead: 8-byte)
      for (int j = threadIdx.x * 8; j < d; j += blockDim.x * 8) {
        const uint4 p = *reinterpret_cast<const uint4*>(static_cast<const char*>(W) + (src0 + j) * 2);
        const uint2 dd = dead ? *reinterpret_cast<const uint2*>(dead + j) : make_uint2(0u, 0u);
        const unsigned h[4] = {p.x, p.y, p.z, p.w}, dw[2] = {dd.x, dd.y};
        float v[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = bf16 ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&h[k]))
                                : __half22float2(*reinterpret_cast<const __half2*>(&h[k]));
          v[2 * k] = f.x; v[2 * k + 1] = f.y;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          mn = fminf(mn, v[k]); mx = fmaxf(mx, v[k]);
          if ((dw[k >> 2] >> (8 * (k & 3))) & 0xffu) v[k] = 0.f;
        }
        *reinterpret_cast<float4*>(to + j) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(to + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
      }
    } else {
      for (int j = threadIdx.x; j < d; j += blockDim.x) {
        const float v = oc_ld16(W, src0 + j, bf16);
        mn = fminf(mn, v); mx = fmaxf(mx, v);
        to[j] = (dead && dead[j]) ? 0.f : v;
      }
    }
    if (perm) {
      __syncthreads();
      if (vec && (reinterpret_cast<uintptr_t>(perm) & 15) == 0) {
        for (int j = threadIdx.x * 4; j < d; j += blockDim.x * 4) {
          const int4 q = *reinterpret_cast<const int4*>(perm + j);
          *reinterpret_cast<float4*>(dst + j) = make_float4(row_s[q.x], row_s[q.y], row_s[q.z], row_s[q.w]);
        }
      } else {
        for (int j = threadIdx.x; j < d; j += blockDim.x) dst[j] = row_s[perm[j]];
      }
    }
  }
  if (!per_channel) return;
  __shared__ float smn[32], smx[32], bc[4];
  const int nwarp = (blockDim.x + 31) / 32;
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) { smn[threadIdx.x >> 5] = mn; smx[threadIdx.x >> 5] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nwarp; ++w) { mn = fminf(mn, smn[w]); mx = fmaxf(mx, smx[w]); }
    float s, z;
    params_from_range(mn, mx, maxq, sym, s, z);
    bc[0] = mn; bc[1] = mx; bc[2] = s; bc[3] = z;
  }
  __syncthreads();
  float best_s = bc[2], best_z = bc[3];
  if (mse_steps > 0) {
    // shrink search over the whole (original) row, one block-wide error sum per candidate
    const float rmn = bc[0], rmx = bc[1], zsym = bc[3];
    float best = __int_as_float(0x7f800000);
    for (int i = 0; i < mse_steps; ++i) {
      float s1, z1;
      mse_candidate(i, mse_grid, rmn, rmx, maxq, sym, zsym, s1, z1);
      float err = 0.f;
      for (int j = threadIdx.x; j < d; j += blockDim.x)
        err += mse_term(oc_ld16(W, src0 + j, bf16), s1, z1, (float)maxq, mse_norm);
      for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
      __syncthreads();
      if ((threadIdx.x & 31) == 0) smn[threadIdx.x >> 5] = err;
      __syncthreads();
      float tot = 0.f;
      for (int w = 0; w < nwarp; ++w) tot += smn[w];
      if (tot < best) { best = tot; best_s = s1; best_z = z1; }
    }
  }
  if (threadIdx.x == 0) {
    scales[row] = best_s;
    zeros[row] = best_z;
  }
}

// ---- final pass: pack, cast, dequantize ---------------------------------------------------
// Packed layout: pack_int_weights / pack_zeros of the reference
// (onecomp/quantizer/gptq/gptq_layer.py:36-83, 129-139, 160-170).
__device__ __forceinline__ void pack3(const unsigned (&v)[32], unsigned (&w)[3]) {
  w[0] = w[1] = w[2] = 0u;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const int bit = 3 * k, wi = bit >> 5, off = bit & 31;
    w[wi] |= v[k] << off;
    if (off + 3 > 32) w[wi + 1] |= v[k] >> (32 - off);
  }
}

// Group g of problem b: scales as fp16 and fp32, raw zero points, and the packed ones, qzeros[g][w]: (zero - 1) & mask of
// rows w*f .. w*f+f-1 (3 bit: 32 rows -> 3 words).  One thread per row; the first row of a word packs it.
__global__ void params_kernel(const float* __restrict__ scales, const float* __restrict__ zeros, int out, int G,
                              long long s_par, __half* __restrict__ scales16, float* __restrict__ scales32,
                              int* __restrict__ zeros_i32, long long lds, long long s_out, int bits,
                              int* __restrict__ qzeros, long long ldz, long long s_qz) {
  oc_wait_before();
  oc_let_next();
  const int r = blockIdx.x * blockDim.x + threadIdx.x, g = blockIdx.y;
  const long long b = blockIdx.z, at = b * s_out + g * lds + r;
  if (r >= out) return;
  const float* zr = zeros + b * s_par + (long long)g * out;
  if (scales16 || scales32) {
    const float s = scales[b * s_par + (long long)g * out + r];
    if (scales16) scales16[at] = __float2half_rn(s);
    if (scales32) scales32[at] = s;
  }
  if (zeros_i32) zeros_i32[at] = (int)zr[r];
  if (!qzeros) return;
  const unsigned mask = (1u << bits) - 1u;
  int* q = qzeros + b * s_qz + g * ldz;
  if (bits == 3) {
    if (r % 32) return;
    unsigned v[32], w[3];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = (unsigned)((int)zr[r + k] - 1) & mask;
    pack3(v, w);
#pragma unroll
    for (int t = 0; t < 3; ++t) q[r / 32 * 3 + t] = (int)w[t];
  } else {
    const int f = 32 / bits;
    if (r % f) return;
    unsigned word = 0u;
    for (int k = 0; k < f; ++k) word |= ((unsigned)((int)zr[r + k] - 1) & mask) << (k * bits);
    q[r / f] = (int)word;
  }
}

// Original-order outputs in one pass over the codes: packed words, integer codes [out][d] and the
// dequantised weight  fp16( float(fp16(scale)) * (q - zero) )  (reference :153-168).
//
// Bound by HBM: 2 bytes of code in, bits / 8 + 2 out per weight.  A CTA takes 64 rows x 128 columns of
// the original order, a warp 32 of the columns, a lane two neighbouring rows: a lane sees whole packed
// words of its rows, reads the codes coalesced along the rows, and reads scale and zero point only
// where the group changes.  The row-major outputs leave through shared memory, a row segment of 128
// bytes a warp.  The codes of the two rows of a lane stay together in one register from the load to the stores:
// up to 8 bits, q | 0x6400 is fp16(1024 + q), scale * (q - zero) is exact in fp32, so one fp16 subtraction (exact) and one
// product give its rounding, and the packed words grow 16 bits a row at a time.  With the rows taken apart and
// the arithmetic in fp32 issue slots bound it: 28672 x 4096, 4 bits 215 -> 113 us;
// 4096 x 4096, 3 bits 34 -> 17 us.
constexpr int FIN_ROWS = 64, FIN_COLS = 128;
// Two neighbouring columns of a row share a 4-byte word of the tile.  Writers of a warp hold every other
// row: 65 words apart, shifted by one in the second half, all 32 fall into different banks.
constexpr int FIN_PITCH = FIN_COLS / 2 + 1, FIN_TILE = FIN_ROWS * FIN_PITCH + 1;
__device__ __forceinline__ int fin_at(int row, int col) { return row * FIN_PITCH + (row >> 5) + (col >> 1); }
struct FinishArgs {
  const unsigned short* codesT; int out, d; const int* invperm; int gs;
  const float* scales; const float* zeros;
  int* qweight; long long ldq; int* codes; long long ldc; void* what; long long ldwh; int bf16;
  int narrow;                                      // codes of at most 8 bits
  long long s_codes, s_par, s_qw, s_out, s_what;   // strides between the problems of a batch
};
// BITS 0: nothing is packed.  LOOKUP: columns are permuted, a group may change inside 32 columns, or the last 32 are fewer.
template <int BITS, bool LOOKUP>
__global__ void __launch_bounds__(128) finish_kernel(FinishArgs a) {
  extern __shared__ unsigned fin_s[];        // one tile per row-major output
  __shared__ int2 look[FIN_COLS];            // source column and group
  oc_wait_before();
  unsigned* tw = fin_s;
  unsigned* tq = fin_s + (a.what ? FIN_TILE : 0);
  {
    const long long b = blockIdx.z;
    a.codesT += b * a.s_codes; a.scales += b * a.s_par; a.zeros += b * a.s_par;
    if (a.invperm) a.invperm += b * a.d;
    if (a.qweight) a.qweight += b * a.s_qw;
    if (a.codes) a.codes += b * a.s_out;
    if (a.what) a.what = static_cast<char*>(a.what) + b * a.s_what * 2;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = blockIdx.y * FIN_ROWS, cb = blockIdx.x * FIN_COLS, c0 = cb + warp * 32;
  const int r = r0 + 2 * lane;
  const bool pair = (a.out & 1) == 0;          // two rows in one 4-byte access
  const bool one = r < a.out, two = r + 1 < a.out;
  if (LOOKUP) {
    const int c = cb + tid, j = c < a.d ? (a.invperm ? a.invperm[c] : c) : 0;
    look[tid] = make_int2(j, a.gs == -1 ? 0 : j / a.gs);
    __syncthreads();
  }
  if (c0 < a.d && one) {
    unsigned q2[32];                           // codes of both rows
    {
      const unsigned short* p = a.codesT + (long long)c0 * a.out + r;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        if (LOOKUP) p = a.codesT + (long long)look[warp * 32 + k].x * a.out + r;
        q2[k] = 0u;
        if (!LOOKUP || c0 + k < a.d) {
          if (pair) q2[k] = *reinterpret_cast<const unsigned*>(p);
          else q2[k] = (unsigned)p[0] | (two ? (unsigned)p[1] << 16 : 0u);
        }
        p += a.out;
      }
    }
    if (BITS && a.qweight) {
      constexpr int PIECES = BITS ? 2 * BITS : 1;
      constexpr unsigned MASK = BITS ? (1u << BITS) - 1u : 0u;
      unsigned piece[PIECES];                  // 16 bits of both rows' packed words each
#pragma unroll
      for (int t = 0; t < PIECES; ++t) piece[t] = 0u;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int bit = k * BITS, pi = bit >> 4, off = bit & 15, low = min(BITS, 16 - off);   // bits in the first piece
        piece[pi] |= (q2[k] & (((1u << low) - 1u) * 0x10001u)) << off;
        if (low < BITS) piece[pi + 1 < PIECES ? pi + 1 : pi] |= (q2[k] >> low) & ((MASK >> low) * 0x10001u);
      }
      const long long w0 = (long long)c0 / 32 * BITS;
      const int words = min(BITS, (int)((long long)(a.d - c0) * BITS / 32));   // d is a multiple of the pack factor
      const bool both = two && (a.ldq & 1) == 0 && (reinterpret_cast<uintptr_t>(a.qweight) & 7) == 0;
#pragma unroll
      for (int t = 0; t < BITS; ++t) {
        if (t >= words) continue;
        int* p = a.qweight + (w0 + t) * a.ldq + r;
        const int wa = (int)__byte_perm(piece[2 * t], piece[2 * t + 1 < PIECES ? 2 * t + 1 : 0], 0x5410);
        const int wb = (int)__byte_perm(piece[2 * t], piece[2 * t + 1 < PIECES ? 2 * t + 1 : 0], 0x7632);
        if (both) *reinterpret_cast<int2*>(p) = make_int2(wa, wb);
        else {
          p[0] = wa;
          if (two) p[1] = wb;
        }
      }
    }
    if (a.codes) {
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        tq[fin_at(2 * lane, warp * 32 + k)] = __byte_perm(q2[k], q2[k + 1], 0x5410);
        tq[fin_at(2 * lane + 1, warp * 32 + k)] = __byte_perm(q2[k], q2[k + 1], 0x7632);
      }
    }
    if (a.what) {
      int group = -1;
      float2 zr = make_float2(0.f, 0.f);
      __half2 s2 = __floats2half2_rn(0.f, 0.f), z2 = s2;
      auto load_group = [&](int g) {
        const float* sp = a.scales + (long long)g * a.out + r;
        const float* zp = a.zeros + (long long)g * a.out + r;
        zr = make_float2(zp[0], two ? zp[1] : 0.f);
        s2 = __floats2half2_rn(sp[0], two ? sp[1] : 0.f);
        z2 = __floats2half2_rn(1024.f + zr.x, 1024.f + zr.y);
      };
      if (!LOOKUP) load_group(a.gs == -1 ? 0 : c0 / a.gs);
      // the reference rounds to fp16 first and casts to the module's dtype afterwards
      auto each = [&](auto narrow, auto bf16) {
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          unsigned w[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (LOOKUP) {
              const int g = look[warp * 32 + k + i].y;
              if (g != group) { group = g; load_group(g); }
            }
            __half2 h;
            if (decltype(narrow)::value) {
              const unsigned v = q2[k + i] | 0x64006400u;
              h = __hmul2(s2, __hsub2(*reinterpret_cast<const __half2*>(&v), z2));
            } else {
              const float2 s = __half22float2(s2);
              h = __floats2half2_rn(__fmul_rn(s.x, __fsub_rn((float)(q2[k + i] & 0xffffu), zr.x)),
                                    __fmul_rn(s.y, __fsub_rn((float)(q2[k + i] >> 16), zr.y)));
            }
            if (decltype(bf16)::value) {
              const float2 f = __half22float2(h);
              const __nv_bfloat162 bb = __floats2bfloat162_rn(f.x, f.y);
              w[i] = *reinterpret_cast<const unsigned*>(&bb);
            } else w[i] = *reinterpret_cast<const unsigned*>(&h);
          }
          tw[fin_at(2 * lane, warp * 32 + k)] = __byte_perm(w[0], w[1], 0x5410);
          tw[fin_at(2 * lane + 1, warp * 32 + k)] = __byte_perm(w[0], w[1], 0x7632);
        }
      };
      if (BITS || a.narrow) {
        if (a.bf16) each(std::true_type{}, std::true_type{});
        else each(std::true_type{}, std::false_type{});
      } else {
        if (a.bf16) each(std::false_type{}, std::true_type{});
        else each(std::false_type{}, std::false_type{});
      }
    }
  }
  oc_let_next();
  if (!a.what && !a.codes) return;
  __syncthreads();
  const bool vec = ((a.ldwh | a.d) & 1) == 0 && (reinterpret_cast<uintptr_t>(a.what) & 3) == 0;
  const bool vec_q = ((a.ldc | a.d) & 1) == 0 && (reinterpret_cast<uintptr_t>(a.codes) & 7) == 0;
#pragma unroll 4
  for (int row = warp; row < FIN_ROWS; row += 4) {
    const int rr = r0 + row;
    if (rr >= a.out) break;
#pragma unroll
    for (int h = 0; h < FIN_COLS / 64; ++h) {
      const int k = h * 64 + 2 * lane, c = cb + k;
      if (c >= a.d) continue;
      if (a.what) {
        unsigned short* w = static_cast<unsigned short*>(a.what) + (long long)rr * a.ldwh + c;
        const unsigned v = tw[fin_at(row, k)];
        if (vec) *reinterpret_cast<unsigned*>(w) = v;
        else {
          w[0] = (unsigned short)(v & 0xffffu);
          if (c + 1 < a.d) w[1] = (unsigned short)(v >> 16);
        }
      }
      if (a.codes) {
        int* p = a.codes + (long long)rr * a.ldc + c;
        const unsigned v = tq[fin_at(row, k)];
        if (vec_q) *reinterpret_cast<int2*>(p) = make_int2((int)(v & 0xffffu), (int)(v >> 16));
        else {
          p[0] = (int)(v & 0xffffu);
          if (c + 1 < a.d) p[1] = (int)(v >> 16);
        }
      }
    }
  }
}

template <bool LOOKUP>
void (*finish_of(int bits))(FinishArgs) {
  return bits == 2 ? finish_kernel<2, LOOKUP> : bits == 3 ? finish_kernel<3, LOOKUP> : bits == 4 ? finish_kernel<4, LOOKUP>
         : bits == 8 ? finish_kernel<8, LOOKUP> : finish_kernel<0, LOOKUP>;
}
int launch_finish(const FinishArgs& a, int bits, int batch, cudaStream_t stream) {
  const dim3 grid(oc_div_up(a.d, FIN_COLS), oc_div_up(a.out, FIN_ROWS), batch);
  const int smem = ((a.what ? 1 : 0) + (a.codes ? 1 : 0)) * FIN_TILE * 4;
  const bool lookup = a.invperm || (a.gs != -1 && a.gs % 32 != 0) || a.d % 32 != 0;
  OC_LAUNCH((lookup ? finish_of<true>(bits) : finish_of<false>(bits)), grid, 128, smem, stream, a);
  return OC_OK;
}

template <int WARPS, bool ALIGNED>
int launch_block_t(const ColArgs& a, cudaStream_t stream) {
  // tiles, plus the error windows the helper threads read (only CTAs with few rows have helpers)
  const int smem = (BLK * BLK + WARPS * 32 * WS + BLK + (WARPS <= 2 ? 2 * SUB * WARPS * 32 : 0)) * (int)sizeof(float);
  OC_OPT_IN_SMEM((gptq_block_kernel<WARPS, ALIGNED>), smem);
  OC_LAUNCH((gptq_block_kernel<WARPS, ALIGNED>), dim3(oc_div_up(a.out, WARPS * 32), a.batch), LOADERS, smem, stream, a);
  return OC_OK;
}

template <int WARPS>
int launch_block(const ColArgs& a, cudaStream_t stream) {
  // group starts fall on window starts when the block starts on a multiple of SUB columns and
  // the group size is a multiple of SUB
  const bool aligned = a.gs == -1 || (a.gs % SUB == 0 && a.i1 % SUB == 0);
  return aligned ? launch_block_t<WARPS, true>(a, stream) : launch_block_t<WARPS, false>(a, stream);
}

// The fewest sets of 32 rows per CTA for which all CTAs run at once; eight where even that takes several waves.
int launch_blocks(const ColArgs& a, int sm_count, cudaStream_t stream) {
  const int sets = oc_div_up(a.out, 32);
  int per_cta = 1;
  while (per_cta < 8 && (long long)oc_div_up(sets, per_cta) * a.batch > sm_count) ++per_cta;
  switch (per_cta) {
    case 1: return launch_block<1>(a, stream);
    case 2: return launch_block<2>(a, stream);
    case 3: return launch_block<3>(a, stream);
    case 4: return launch_block<4>(a, stream);
    case 5: return launch_block<5>(a, stream);
    case 6: return launch_block<6>(a, stream);
    case 7: return launch_block<7>(a, stream);
    default: return launch_block<8>(a, stream);
  }
}

long long round4(long long x) { return (x + 3) / 4 * 4; }
long long round8(long long x) { return (x + 7) / 8 * 8; }
long long u_blocks(int d) { return (d + OC_SPLIT_BLOCK - 1) / OC_SPLIT_BLOCK; }

constexpr int PREPARE_STAGED_D = 49152;   // widest row that the act-order gather keeps in shared memory

}  // namespace

extern "C" long long oc_gptq_workspace_bytes(int out, int d, int groupsize) {
  const long long G = (groupsize == -1) ? 1 : (d + groupsize - 1) / groupsize;
  long long b = 0;
  b += (long long)out * round4(d) * 4;       // Wf
  b += (long long)SUPER * BLK * round8(out) * 4;  // errors, fp32 or as two planes
  b += SUPER * round8(out) * 4;              // their scales
  b += 4 * (long long)d * round8(d);         // planes of U
  b += round4(u_blocks(d) * u_blocks(d)) * 4;     // their scales
  b += round4((long long)d * out * 2);       // codesT
  b += 2 * G * (long long)out * 4;           // scales, zeros fp32
  return b + 256;
}

// The column loop for `batch` problems of equal shape laid out one after another (every array of
// problem b starts b times its per-problem size after problem 0).  One chain of launches serves
// all problems: the block kernel and the preparation take the problem from blockIdx.y, the
// trailing updates are batched products.
static int gptq_quantize_impl(int batch, const void* W, long long ldw_in, int out, int d, const float* U,
                              long long ldu, const int* perm, const int* invperm, const unsigned char* dead,
                              int wbits, int groupsize, int sym, int blocksize, int mse, int q_grid,
                              float q_norm, int sm_count, int* qweight, int* qzeros, __half* scales16,
                              float* scales32, int* zeros_i32, long long ld_out, int* codes, void* what,
                              long long ldwh, int w_dtype, void* workspace, long long workspace_bytes,
                              cudaStream_t stream) {
  OC_REQUIRE(w_dtype == OC_DTYPE_F16 || w_dtype == OC_DTYPE_BF16, "gptq_quantize: unknown weight dtype");
  const int bf16 = w_dtype == OC_DTYPE_BF16;
  OC_REQUIRE(W && U && workspace, "gptq_quantize: null pointer");
  OC_REQUIRE(batch >= 1 && batch <= 65535, "gptq_quantize: batch must be in 1..65535");
  OC_REQUIRE(out > 0 && d > 0 && ldw_in >= d && ldu >= d, "gptq_quantize: bad dimensions");
  OC_REQUIRE(wbits >= 1 && wbits <= 15, "gptq_quantize: wbits must be in 1..15");
  OC_REQUIRE(groupsize == -1 || groupsize >= 1, "gptq_quantize: groupsize must be -1 or >= 1");
  if (blocksize < 1 || blocksize > BLK) {
    oc_set_last_error("gptq_quantize: blocksize must be in 1..128");
    return OC_ERR_UNSUPPORTED;
  }
  if (qweight || qzeros) {
    OC_REQUIRE(wbits == 2 || wbits == 3 || wbits == 4 || wbits == 8, "gptq_quantize: packing needs wbits in {2,3,4,8}");
    const int f = (wbits == 3) ? 32 : 32 / wbits;
    if (qweight) OC_REQUIRE(d % f == 0, "gptq_quantize: in_features not divisible by the pack factor");
    if (qzeros) OC_REQUIRE(out % f == 0 && ld_out % f == 0, "gptq_quantize: out_features not divisible by the pack factor");
  }
  const long long ws_one = oc_gptq_workspace_bytes(out, d, groupsize);
  if (workspace_bytes < ws_one * batch) {
    oc_set_last_error("gptq_quantize: workspace too small");
    return OC_ERR_WORKSPACE;
  }
  if (ld_out < out) ld_out = out;
  const int G = (groupsize == -1) ? 1 : (d + groupsize - 1) / groupsize;
  const long long ldw = round4(d), lde = round8(out), ldu_p = round8(d);
  // workspace: all problems' Wf, then all ErrT, codesT, scales, zeros (each contiguous over the batch)
  const long long nWf = (long long)out * ldw, nErr = (long long)SUPER * BLK * lde;
  const long long nCodes = round4((long long)d * out * 2) / 2, nPar = (long long)G * out;
  char* ws = (char*)workspace;
  float* Wf = (float*)ws;                       ws += nWf * 4 * batch;
  float* ErrT = (float*)ws;                     ws += nErr * 4 * batch;
  float* err_scale = (float*)ws;                ws += SUPER * lde * 4 * batch;
  __half* Up = (__half*)ws;                     ws += 2 * d * ldu_p * 2 * batch;
  float* u_table = (float*)ws;                  ws += round4(u_blocks(d) * u_blocks(d)) * 4 * batch;
  unsigned short* codesT = (unsigned short*)ws; ws += nCodes * 2 * batch;
  float* scales = (float*)ws;                   ws += nPar * 4 * batch;
  float* zeros = (float*)ws;
  const int maxq = (1 << wbits) - 1;
  const long long sU = (long long)d * ldu, sWin = (long long)out * ldw_in;

  OC_REQUIRE(!mse || (q_grid >= 1 && q_norm > 0.f), "gptq_quantize: mse needs q_grid >= 1 and q_norm > 0");
  const int mse_steps = mse ? (int)(0.8 * q_grid) : 0;   // maxshrink = 0.8 as in the reference
  const bool vec = d % 8 == 0 && ldw_in % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(Wf)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(dead) & 7) == 0;
  const bool staged = perm && d <= PREPARE_STAGED_D;
  if (staged) OC_OPT_IN_SMEM(gptq_prepare_kernel, PREPARE_STAGED_D * 4);
  OC_LAUNCH(gptq_prepare_kernel, dim3(out, batch), 256, staged ? d * 4 : 0, stream,
            W, bf16, ldw_in, out, d, perm, dead, Wf, ldw, groupsize == -1 ? 1 : 0, maxq, sym, mse_steps,
            (float)q_grid, q_norm, scales, zeros, sWin, nWf, nPar, vec, staged);

  if (sm_count <= 0) sm_count = 148;
  const int warps_total = oc_div_up(out, 32) * batch;
  const int per_sm = oc_div_up(warps_total, sm_count);
  // The lazy-batch update is done at two distances.  After each block the columns up to the
  // end of its group of SUPER blocks are updated at once (they are needed next); the columns
  // beyond are updated once per group with the errors of all its blocks, which cuts the
  // read-modify-write traffic on the trailing matrix by SUPER.  Every column still receives
  // the same updates, grouped differently in the fp32 sum.
  // A group's parameters are fitted on columns that must carry every earlier update, so the
  // far update may only be postponed when no group reaches across the end of a block group.
  // Full blocks of 128 columns with something behind them leave their errors split.  Not with 2 and 3 bits: sums in another
  // order move a code where a weight lies next to the middle between two, and there one code is as much as the weight
  // itself, so these keep the products they have had (tf32 terms, the same codes as before; 4096 x 4096, 3 bits: 1.17
  // ms against 0.70; dependent launches of those products made it 1.25).
  const bool split = oc_split_engine_on() && wbits >= 4 && blocksize == BLK && d > BLK &&
                     (reinterpret_cast<uintptr_t>(workspace) & 15) == 0;
  const long long nb_u = u_blocks(d), nTab = round4(nb_u * nb_u), nErrP = SUPER * BLK * lde;
  if (split) {
    OcSplitArgs us{};
    us.src = U; us.ld = ldu; us.rows = us.cols = d; us.planes = Up; us.plane = d * ldu_p; us.ldp = ldu_p;
    us.table = u_table; us.ldt = nb_u; us.region = OC_SPLIT_UPPER;
    us.nb1 = batch; us.nb2 = 1; us.src1 = sU; us.dst1 = 2 * us.plane; us.tab1 = nTab;
    const int rc = oc_split_launch(us, stream);
    if (rc) return rc;
  }
  const bool two_level = (groupsize == -1) || ((SUPER * blocksize) % groupsize == 0);
  const int super_cols = (two_level ? SUPER : 1) * blocksize;
  // Groups of full blocks in one launch each, where every SM has one set of rows at most.
  OcSplitOperand u_op{};
  u_op.planes = Up; u_op.plane = d * ldu_p; u_op.ld = ldu_p; u_op.mn_major = 1; u_op.terms = 2; u_op.stride1 = 2 * d * ldu_p;
  u_op.scale = u_table; u_op.scale_k = nb_u; u_op.scale_r = 1; u_op.scale1 = nTab;
  auto col_args = [&](int i1, int count, float* err_rows, __half* err_planes, float* err_sc) {
    return ColArgs{Wf, ldw, out, d, i1, count, U, ldu, err_rows, lde, err_planes, nErrP, err_sc, codesT, scales, zeros,
                   groupsize, maxq, sym, mse_steps, (float)q_grid, q_norm, nWf, sU, nErr, nCodes, nPar, 2 * nErrP,
                   SUPER * lde, batch, -1.f};
  };
  GroupArgs group_args{col_args(0, BLK, ErrT, (__half*)ErrT, err_scale), 0, u_table, nb_u, nTab, 0, nullptr};
  const bool grouped = split && two_level && windows_fit(group_args.c) && group_fits(group_args.c, sm_count);
  CUtensorMap map_u;
  if (grouped) {
    OcGemmDevice dev;
    int rc = octc::make_split_map(&map_u, u_op, d, d, batch, 1, 0);
    if (!rc) rc = oc_gemm_device(dev);
    if (rc) return rc;
    group_args.status = dev.status;
  }
  // W[:, n0 .. n1) -= Err U[k0 .. k0 + k, n0 .. n1), Err the planes of the group that starts at column s0
  auto split_update = [&](int s0, int k0, int k, int n0, int n1) {
    OcSplitGemm g{};
    g.A.planes = (__half*)ErrT + (long long)(k0 - s0) * lde; g.A.plane = nErrP; g.A.ld = lde; g.A.mn_major = 1;
    g.A.terms = 2; g.A.stride1 = 2 * nErrP;
    g.A.scale = err_scale + (k0 - s0) / BLK * lde; g.A.scale_k = lde; g.A.scale_r = BLK; g.A.scale_row = 1;
    g.A.scale1 = SUPER * lde;
    g.B = u_op;
    g.B.planes += (long long)k0 * ldu_p + n0; g.B.scale += k0 / BLK * nb_u + n0 / BLK;
    g.C = Wf + n0; g.ldc = ldw; g.strideC1 = nWf;
    g.M = out; g.N = n1 - n0; g.K = k; g.nb1 = batch; g.nb2 = 1; g.alpha = -1.f; g.add = 1;
    return oc_gemm_split_launch(g, stream);
  };
  for (int i1 = 0, i2; i1 < d; i1 = i2) {
    const int s0 = (i1 / super_cols) * super_cols;          // first column of the group
    const int s1 = min(d, s0 + super_cols);                 // one past its last column
    int rc;
    if (grouped && s1 - i1 >= BLK) {                        // (i1 == s0)
      const int blocks = (s1 - s0) / BLK;
      i2 = s0 + blocks * BLK;
      group_args.c.i1 = i1; group_args.blocks = blocks; group_args.store_errors = i2 < d;
      rc = launch_group(group_args, map_u, stream);
      // a partial block behind the last group, block by block as in the other schedule
      for (int j = 0; !rc && i2 < s1 && j < blocks; ++j) rc = split_update(s0, s0 + j * BLK, BLK, i2, s1);
      if (!rc && i2 == s1 && i2 < d) rc = split_update(s0, s0, i2 - s0, i2, d);
      if (rc) return rc;
      continue;
    }
    const int count = min(blocksize, d - i1);
    i2 = i1 + count;
    float* err_rows = ErrT + (long long)(i1 - s0) * lde;
    const ColArgs a = col_args(i1, count, err_rows, split && i2 < d ? (__half*)ErrT + (long long)(i1 - s0) * lde : nullptr,
                               err_scale + (i1 - s0) / BLK * lde);
    if (per_sm <= 2 && windows_fit(a)) rc = launch_windows(a, stream);
    else rc = launch_blocks(a, sm_count, stream);
    if (rc) return rc;
    if (i2 >= d) break;
    // near: the rest of the group, behind this block; far: everything behind the group, at its end
    const bool near = i2 < s1;
    if (split) rc = near ? split_update(s0, i1, count, i2, s1) : split_update(s0, s0, s1 - s0, s1, d);
    else {
      OcGemm g{};
      g.lda = lde; g.transA = 1; g.ldb = ldu; g.transB = 0; g.ldc = ldw;
      g.M = out; g.alpha = -1.f; g.beta = 1.f; g.flags = 0;
      g.batch = batch; g.strideA = nErr; g.strideB = sU; g.strideC = nWf;
      if (near) {
        g.A = err_rows; g.K = count;
        g.B = U + (long long)i1 * ldu + i2; g.C = Wf + i2; g.N = s1 - i2;
      } else {
        g.A = ErrT; g.K = s1 - s0;
        g.B = U + (long long)s0 * ldu + s1; g.C = Wf + s1; g.N = d - s1;
      }
      rc = oc_gemm_f32_launch(g, stream);
    }
    if (rc) return rc;
  }

  const int tb = 128;
  const int f = (wbits == 3) ? 32 : ((wbits == 2 || wbits == 4 || wbits == 8) ? 32 / wbits : 1);
  const long long ldz = (wbits == 3) ? ld_out / 32 * 3 : ld_out / f;
  const long long prow = (wbits == 3) ? d / 32 * 3 : d / f;     // rows of one problem's packed weight
  if (qweight || codes || what) {
    FinishArgs f_args{codesT, out, d, invperm, groupsize, scales, zeros, qweight, ld_out, codes, d, what, ldwh, bf16,
                      maxq < 256, nCodes, nPar, prow * ld_out, (long long)out * d, (long long)out * ldwh};
    const int rc = launch_finish(f_args, qweight ? wbits : 0, batch, stream);
    if (rc) return rc;
  }
  // scales, zero points (raw and packed), all problems in one launch
  if (qzeros || scales16 || scales32 || zeros_i32)
    OC_LAUNCH(params_kernel, dim3(oc_div_up(out, tb), G, batch), tb, 0, stream, scales, zeros, out, G, nPar, scales16, scales32,
              zeros_i32, ld_out, (long long)G * ld_out, wbits, qzeros, ldz, (long long)G * ldz);
  return OC_OK;
}

// See include/onecomp_b200.h for the contracts.
extern "C" int oc_gptq_quantize(const void* W, long long ldw_in, int out, int d, const float* U,
                                long long ldu, const int* perm, const int* invperm,
                                const unsigned char* dead, int wbits, int groupsize, int sym,
                                int blocksize, int mse, int q_grid, float q_norm, int sm_count,
                                int* qweight, int* qzeros, void* scales16,
                                float* scales32, int* zeros_i32, long long ld_out, int* codes,
                                void* what, long long ldwh, int w_dtype, void* workspace,
                                long long workspace_bytes, void* stream) {
  return gptq_quantize_impl(1, W, ldw_in, out, d, U, ldu, perm, invperm, dead, wbits, groupsize, sym, blocksize,
                            mse, q_grid, q_norm, sm_count, qweight, qzeros, (__half*)scales16, scales32,
                            zeros_i32, ld_out, codes, what, ldwh, w_dtype, workspace, workspace_bytes,
                            (cudaStream_t)stream);
}

extern "C" int oc_gptq_quantize_batched(int batch, const void* W, long long ldw_in, int out, int d,
                                        const float* U, long long ldu, const int* perm, const int* invperm,
                                        const unsigned char* dead, int wbits, int groupsize, int sym,
                                        int blocksize, int mse, int q_grid, float q_norm, int sm_count,
                                        int* qweight, int* qzeros, void* scales16, float* scales32,
                                        int* zeros_i32, int* codes, void* what, int w_dtype, void* workspace,
                                        long long workspace_bytes, void* stream) {
  return gptq_quantize_impl(batch, W, ldw_in, out, d, U, ldu, perm, invperm, dead, wbits, groupsize, sym,
                            blocksize, mse, q_grid, q_norm, sm_count, qweight, qzeros, (__half*)scales16,
                            scales32, zeros_i32, out, codes, what, d, w_dtype, workspace, workspace_bytes,
                            (cudaStream_t)stream);
}
