// Inverse-Hessian factor for GPTQ: U upper triangular with U^T U = (H + damp I)^-1.
//
// Replaces the potrf + potri + potrf sequence of the reference
// (onecomp/quantizer/gptq/_gptq.py:594-643, call sites :693-706) with one
// Cholesky factorisation and one triangular inverse:
//
//   A = J (P H P^T + damp I) J      (J reverses the index order, P is the act-order permutation)
//   A = L L^T                       blocked right-looking Cholesky (two levels: 128 / 512), fp32:
//                                   diagonal block on one SM, panel solve by forward substitution
//                                   (fp32 FMAs, all SMs), updates on the tensor cores (gemm_split.cu)
//   X = L^-1                        diagonal blocks inverted in one launch, then joined level by
//                                   level (recursive blocked triangular inverse), fp32
//   U = J X J                       upper triangular, U^T U = (P H P^T + damp I)^-1
//
// because J L J is the upper factor V of H = V V^T and U = V^-1.
//
// A is equilibrated: rows and columns are multiplied by powers of two that bring its diagonal into [1, 4), and the
// columns of U are scaled back.  Nothing but exponents changes, and the entries of L are below 2 in
// magnitude, so that the panels of L can be kept as two fp16 planes (split.cuh) under one fixed scale.
#include "split.cuh"

namespace {

constexpr int NB = 128;  // panel width
constexpr int OB = 512;  // outer block of the two-level Cholesky
constexpr int BUILD_STAGED_N = 49152;   // widest row that the act-order gather keeps in shared memory

// ---- diag statistics: dead columns, damping --------------------------------
// diagv[j] = H[j,j] (1 where it is 0), dead[j], damp_out[0] = percdamp * mean(diagv)
// Batched launches: block index `b` of the batch dimension selects the problem; `sH`, `sW`, ... are
// the element strides between consecutive problems.
// equil[j] = 2^-e with (diagv[j] + shift) / 4^e in [1, 4)
__global__ void diag_stats_kernel(const float* __restrict__ H, long long ld, int n, float percdamp, float rel_shift,
                                  float* __restrict__ diagv, unsigned char* __restrict__ dead,
                                  float* __restrict__ damp_out, float* __restrict__ equil, int* __restrict__ status,
                                  long long sH, long long sW) {
  oc_wait_before();
  if (threadIdx.x == 0) status[blockIdx.x] = 0;
  {
    const long long b = blockIdx.x;
    H += b * sH; diagv += b * sW; dead += b * n; damp_out += b * 2; equil += b * sW;
  }
  __shared__ double red[32];
  __shared__ float damp_s;
  double s = 0.0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    float v = H[(long long)j * ld + j];
    const bool dd = (v == 0.f);
    if (dd) v = 1.f;
    diagv[j] = v;
    dead[j] = dd ? 1 : 0;
    s += (double)v;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (blockDim.x + 31) / 32; ++w) t += red[w];
    damp_out[0] = damp_s = percdamp * (float)(t / (double)n);
    damp_out[1] = (float)(t / (double)n);
  }
  __syncthreads();
  oc_let_next();
  const float shift = rel_shift * damp_s;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const float v = diagv[j] + shift;
    const int e = ((int)(__float_as_uint(v) >> 23) - 127) >> 1;
    const bool ok = v > 0.f && v <= 3.402823466e38f;       // (anything else ends in a bad pivot)
    equil[j] = ok ? __uint_as_float((unsigned)(127 - e) << 23) : 1.f;
  }
}

// ---- act-order: stable descending argsort by counting ranks ---------------------
// A NaN counts as +infinity: without a total order two columns would share a rank, and entries of perm,
// which every later pass uses as an index, would keep what was in memory.
__device__ __forceinline__ float rank_key(float v) { return v == v ? v : __int_as_float(0x7f800000); }
__global__ void rank_sort_kernel(const float* __restrict__ key, int n, int* __restrict__ perm, long long sW) {
  oc_wait_before();
  oc_let_next();
  key += (long long)blockIdx.y * sW;
  perm += (long long)blockIdx.y * n;
  __shared__ float tile[1024];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const float ki = (i < n) ? rank_key(key[i]) : 0.f;
  int rank = 0;
  for (int base = 0; base < n; base += 1024) {
    for (int t = threadIdx.x; t < 1024; t += blockDim.x) tile[t] = (base + t < n) ? rank_key(key[base + t]) : 0.f;
    __syncthreads();
    const int lim = min(1024, n - base);
    for (int t = 0; t < lim; ++t) {
      const float kj = tile[t];
      const int j = base + t;
      rank += (kj > ki || (kj == ki && j < i)) ? 1 : 0;
    }
    __syncthreads();
  }
  if (i < n) perm[rank] = i;
}

__global__ void iota_kernel(int* __restrict__ perm, int* __restrict__ inv, int n) {
  oc_wait_before();
  oc_let_next();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { perm[(long long)blockIdx.y * n + i] = i; inv[(long long)blockIdx.y * n + i] = i; }
}

__global__ void invert_perm_kernel(const int* __restrict__ perm, int* __restrict__ inv, int n) {
  oc_wait_before();
  oc_let_next();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  perm += (long long)blockIdx.y * n;
  inv += (long long)blockIdx.y * n;
  if (i < n) inv[perm[i]] = i;
}

// ---- A = J D (P Hfix P^T + shift I) D J, D = diag(equil) --------------------------------------
// Only what the factorisation reads: every row up to the end of its diagonal block.  One CTA per row,
// bound by HBM (4 bytes in, 2 out per entry of H with act-order, where the whole row of H passes
// through shared memory and the permutation is a gather on chip; half of that without).  One global
// access per entry before: 14336 with act-order 1042 us, 264 us now; 4096 67, 16 us.
// equil_p[j] = equil[perm[j]]: what scales the columns of U back.
__global__ void __launch_bounds__(256) build_reversed_kernel(
    const float* __restrict__ H, long long ldh, int n, const int* __restrict__ perm, int permuted,
    const float* __restrict__ diagv, const float* __restrict__ damp, float rel_shift, const float* __restrict__ equil,
    float* __restrict__ equil_p, float* __restrict__ A, long long lda, long long sH, long long sW, int vec, int staged) {
  extern __shared__ __align__(16) float row_s[];
  oc_wait_before();
  oc_let_next();
  const int i = blockIdx.x;
  {
    const long long b = blockIdx.y;
    H += b * sH; perm += b * n; diagv += b * sW; damp += b * 2; A += b * sW; equil += b * sW; equil_p += b * sW;
  }
  const int pi = permuted ? perm[n - 1 - i] : n - 1 - i;
  const float* h = H + (long long)pi * ldh;
  float* a = A + (long long)i * lda;
  const float di = equil[pi];
  const int end = min(n, (i / NB + 1) * NB);
  if (permuted && staged) {
    if (vec) {
      for (int j = threadIdx.x * 4; j < n; j += 1024) {
        const float4 v = *reinterpret_cast<const float4*>(h + j), d = *reinterpret_cast<const float4*>(equil + j);
        *reinterpret_cast<float4*>(row_s + j) = make_float4(v.x * di * d.x, v.y * di * d.y, v.z * di * d.z, v.w * di * d.w);
      }
    } else {
      for (int j = threadIdx.x; j < n; j += 256) row_s[j] = h[j] * di * equil[j];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < end; j += 256) a[j] = row_s[perm[n - 1 - j]];
  } else if (permuted) {
    for (int j = threadIdx.x; j < end; j += 256) { const int p = perm[n - 1 - j]; a[j] = h[p] * di * equil[p]; }
  } else if (vec) {           // n, ldh, lda multiples of 4, 16-byte aligned: so is `end`
    for (int j = threadIdx.x * 4; j < end; j += 1024) {
      const float4 v = *reinterpret_cast<const float4*>(h + n - 4 - j), d = *reinterpret_cast<const float4*>(equil + n - 4 - j);
      *reinterpret_cast<float4*>(a + j) = make_float4(v.w * di * d.w, v.z * di * d.z, v.y * di * d.y, v.x * di * d.x);
    }
  } else {
    for (int j = threadIdx.x; j < end; j += 256) a[j] = h[n - 1 - j] * di * equil[n - 1 - j];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a[i] = (diagv[pi] + rel_shift * damp[0]) * di * di;
    equil_p[n - 1 - i] = di;
  }
}

// ---- U = J X J D (upper part), zero below the diagonal ------------------------------------
// One CTA per row, bound by HBM (2 bytes in, 4 out per entry).  One entry per access before: 14336
// 619 us, 183 us now; 4096 50, 14 us.
__global__ void __launch_bounds__(256) reverse_upper_kernel(const float* __restrict__ X, long long ldx, int n,
                                                            const float* __restrict__ equil_p, float* __restrict__ U,
                                                            long long ldu, long long sW, long long sU, int vec,
                                                            const int* __restrict__ gemm_status, int* __restrict__ status) {
  oc_wait_before();
  oc_let_next();
  const int i = blockIdx.x;
  // an expired wait in a product makes the factor as invalid as a bad pivot does
  if (i == 0 && threadIdx.x == 0 && *gemm_status) atomicCAS(status + blockIdx.y, 0, -*gemm_status);
  const float* x = X + (long long)blockIdx.y * sW + (long long)(n - 1 - i) * ldx;
  float* u = U + (long long)blockIdx.y * sU + (long long)i * ldu;
  equil_p += (long long)blockIdx.y * sW;
  if (vec) {
    for (int j = threadIdx.x * 4; j < n; j += 1024) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j + 3 >= i) {
        const float4 t = *reinterpret_cast<const float4*>(x + n - 4 - j), d = *reinterpret_cast<const float4*>(equil_p + j);
        v.x = j >= i ? t.w * d.x : 0.f; v.y = j + 1 >= i ? t.z * d.y : 0.f; v.z = j + 2 >= i ? t.y * d.z : 0.f;
        v.w = t.x * d.w;
      }
      *reinterpret_cast<float4*>(u + j) = v;
    }
  } else {
    for (int j = threadIdx.x; j < n; j += 256) u[j] = (j >= i) ? x[n - 1 - j] * equil_p[j] : 0.f;
  }
}

// Two fp32 FMAs in one instruction, each rounded like fmaf: d = a * b + c.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// ---- one diagonal block: Cholesky of a (<=128)^2 block on one SM ----------------------------
// A block (nb x nb, lower part read) -> L written back over the lower part, L^T over the upper
// (nothing reads the upper part of a diagonal block of A as matrix data; the panel solve loads L^T
// from there).  A non-positive or non-finite pivot records (global index + 1) in *status (first one
// wins); what is computed behind it means nothing, and no kernel of the chain waits for a value.
//
// A serial chain on one SM, 16 micro-panels of eight columns.  Its core is the chain from pivot block to
// pivot block (factor 8 x 8, solve the next eight rows against it, update their own 8 x 8 block, factor
// that), about 1000 cycles a step: a ninth warp walks it alone, one step ahead.  Of the other eight, two
// threads hold a row in registers, each every other group of four columns: they solve their row against the
// published pivot block, publish the eight new columns and update the rest of the row (two columns per
// FMA instruction, fma.f32x2), beginning with the two groups that the pivot warp needs next.  The
// register file moves eight columns to the left in the update itself, so one loop body serves all
// micro-panels.  The operations on an entry are those of a column-by-column elimination, in its order.
// With 8 x 8 register blocks per thread and a single lane factoring the pivot block this took 31.5 us, with
// every thread factoring it for itself 25 us; now 17 us, about 1050 cycles a step on the pivot warp and up to
// 2000 in the first steps on the rows (an entry of L that is loaded, 4 bytes to 32 lanes a cycle, serves one row).
constexpr int LP = NB + 4;     // pitch of the published columns
constexpr int ROW_THREADS = 256;

// reads the lower part of an 8 x 8 block
__device__ __forceinline__ void load_block8(const float (*m)[8], float (&l)[8][8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 lo = *reinterpret_cast<const float4*>(&m[i][0]);
    l[i][0] = lo.x; l[i][1] = lo.y; l[i][2] = lo.z; l[i][3] = lo.w;
    if (i >= 4) {
      const float4 hi = *reinterpret_cast<const float4*>(&m[i][4]);
      l[i][4] = hi.x; l[i][5] = hi.y; l[i][6] = hi.z; l[i][7] = hi.w;
    }
  }
}

// y <- y L^-T for one row of eight entries; the diagonal of l holds the reciprocals of L's
__device__ __forceinline__ void solve_row8(float (&y)[8], const float (&l)[8][8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    y[j] *= l[j][j];
#pragma unroll
    for (int c = j + 1; c < 8; ++c) y[c] = fmaf(-y[j], l[c][j], y[c]);
  }
}

__global__ void __launch_bounds__(ROW_THREADS + 32, 1)
potrf_block_kernel(float* __restrict__ A, long long lda, int k0, int nb, int* __restrict__ status, long long sW) {
  oc_wait_before();
  A += (long long)blockIdx.x * sW;
  status += blockIdx.x;
  __shared__ __align__(16) float Lp[8 * LP + 16];  // the micro-panel's columns, [8][row]
  __shared__ __align__(16) float L8[2][8][8];      // its factored pivot block, reciprocals on the diagonal
  __shared__ __align__(16) float Qs[2][8][8];      // the next pivot rows: their entries in the micro-panel,
  __shared__ __align__(16) float Pre[2][8][8];     //   and their own block, without this micro-panel's update
  __shared__ __align__(16) float Xs[8][8], Nv[8][8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == ROW_THREADS / 32) {
    // ---- pivot warp: every lane factors the pivot block for itself ----
    __syncthreads();                               // Nv (block 0), Qs[0], Pre[0] are there
#pragma unroll 1
    for (int jb = 0; jb < NB / 8; ++jb) {
      if (jb == NB / 8 - 2) oc_let_next();
      float l[8][8];
      load_block8(Nv, l);
      int bad = 8;                                 // first column with an unusable pivot
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        // (selections, not branches: the eight columns are one stretch of code, whose instructions
        // fill the waits of the chain from pivot to pivot)
        const float p = l[jj][jj];
        const bool ok = p > 0.f && p < __int_as_float(0x7f800000);
        bad = !ok && bad == 8 ? jj : bad;
        // one approximate reciprocal square root, refined once, instead of an IEEE square
        // root followed by IEEE divisions
        float inv = rsqrtf(p);
        inv = inv * fmaf(-0.5f * p * inv, inv, 1.5f);
        l[jj][jj] = inv;
#pragma unroll
        for (int ii = jj + 1; ii < 8; ++ii) l[ii][jj] *= inv;
#pragma unroll
        for (int cc = jj + 1; cc < 8; ++cc)
#pragma unroll
          for (int ii = cc; ii < 8; ++ii) l[ii][cc] = fmaf(-l[ii][jj], l[cc][jj], l[ii][cc]);
      }
      if (bad < 8 && lane == 0) atomicCAS(status, 0, k0 + 8 * jb + bad + 1);
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          *reinterpret_cast<float4*>(&L8[jb & 1][i][0]) = make_float4(l[i][0], l[i][1], l[i][2], l[i][3]);
          if (i >= 4) *reinterpret_cast<float4*>(&L8[jb & 1][i][4]) = make_float4(l[i][4], l[i][5], l[i][6], l[i][7]);
        }
      }
      __syncthreads();                             // L8(jb) to the rows; Qs(jb), Pre(jb) from them
      if (jb == NB / 8 - 1) break;
      float x[8];
      {
        const float4 lo = *reinterpret_cast<const float4*>(&Qs[jb & 1][lane & 7][0]);
        const float4 hi = *reinterpret_cast<const float4*>(&Qs[jb & 1][lane & 7][4]);
        x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w; x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
      }
      solve_row8(x, l);
      if (lane < 8) {
        *reinterpret_cast<float4*>(&Xs[lane][0]) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(&Xs[lane][4]) = make_float4(x[4], x[5], x[6], x[7]);
      }
      __syncwarp();
      // entries (r, c) and (r + 4, c) of the next pivot block
      const int r = lane >> 3, c = lane & 7;
      float v0 = Pre[jb & 1][r][c], v1 = Pre[jb & 1][r + 4][c];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 a0 = *reinterpret_cast<const float4*>(&Xs[r][4 * h]);
        const float4 a1 = *reinterpret_cast<const float4*>(&Xs[r + 4][4 * h]);
        const float4 bc = *reinterpret_cast<const float4*>(&Xs[c][4 * h]);
        v0 = fmaf(-a0.x, bc.x, v0); v1 = fmaf(-a1.x, bc.x, v1);
        v0 = fmaf(-a0.y, bc.y, v0); v1 = fmaf(-a1.y, bc.y, v1);
        v0 = fmaf(-a0.z, bc.z, v0); v1 = fmaf(-a1.z, bc.z, v1);
        v0 = fmaf(-a0.w, bc.w, v0); v1 = fmaf(-a1.w, bc.w, v1);
      }
      Nv[r][c] = v0;
      Nv[r + 4][c] = v1;
      __syncwarp();
    }
    return;
  }

  // ---- row threads: row r, columns 8q + 4h .. 8q + 4h + 3 ----
  const int h = lane >> 4, r = warp * 16 + (lane & 15);
  float* Ab = A + (long long)k0 * lda + k0;
  float* Ar = Ab + (long long)r * lda;
  f32x2 a[32];                                 // a[2q], a[2q + 1]: group q of the remaining columns
  if (nb == NB) {
    float4 v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (8 * q + 4 * h <= r) v[q] = *reinterpret_cast<const float4*>(Ar + 8 * q + 4 * h);
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) { a[2 * q] = pack2(v[q].x, v[q].y); a[2 * q + 1] = pack2(v[q].z, v[q].w); }
  } else {                                     // rows and columns behind the block: identity
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = 8 * q + 4 * h + i;
        v[i] = (c <= r && r < nb) ? Ar[c] : (r == c ? 1.f : 0.f);
      }
      a[2 * q] = pack2(v[0], v[1]);
      a[2 * q + 1] = pack2(v[2], v[3]);
    }
  }
  auto publish = [&](float (*to)[8], f32x2 v0, f32x2 v1) {
    const float2 lo = unpack2(v0), hi = unpack2(v1);
    *reinterpret_cast<float4*>(&to[r & 7][4 * h]) = make_float4(lo.x, lo.y, hi.x, hi.y);
  };
  if (r < 8) publish(Nv, a[0], a[1]);
  else if (r < 16) {
    publish(Qs[0], a[0], a[1]);
    publish(Pre[0], a[2], a[3]);
  }
  __syncthreads();

#pragma unroll 1
  for (int jb = 0; jb < NB / 8; ++jb) {
    const int j0 = 8 * jb;
    float y[8];
    const bool live = warp * 16 + 15 >= j0;    // the same for the whole warp
    __syncthreads();                           // L8(jb) from the pivot warp; the rows' columns are up to date
    if (live) {
      float l[8][8];
      load_block8(L8[jb & 1], l);
      {
        const float2 m0 = unpack2(a[0]), m1 = unpack2(a[1]);
        const float mine[4] = {m0.x, m0.y, m1.x, m1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, mine[i], 16);
          y[i] = h ? other : mine[i];
          y[4 + i] = h ? mine[i] : other;
        }
      }
      solve_row8(y, l);
      const float4 m = h ? make_float4(y[4], y[5], y[6], y[7]) : make_float4(y[0], y[1], y[2], y[3]);
      const float mv[4] = {m.x, m.y, m.z, m.w};
      if (r >= j0 + 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) Lp[(4 * h + i) * LP + r] = mv[i];
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");     // the row threads: Lp is there
    if (live) {
      f32x2 ny[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) ny[j] = pack2(-y[j], -y[j]);
      const float* lp = Lp + j0 + 8 + 4 * h;
#pragma unroll
      for (int q = 0; q < 16; q += 2) {
        // columns up to this warp's last row, two groups in flight (the entries above the diagonal are
        // updated too: nothing reads them; a group behind the last column meets a dead register pair)
        if (jb + 1 + q <= 2 * warp + 1) {
          f32x2 v[4] = {a[2 * q + 2], a[2 * q + 3], q < 14 ? a[q < 14 ? 2 * q + 4 : 0] : 0ull,
                        q < 14 ? a[q < 14 ? 2 * q + 5 : 0] : 0ull};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 t = *reinterpret_cast<const float4*>(lp + j * LP + 8 * q);
            const float4 u = *reinterpret_cast<const float4*>(lp + j * LP + 8 * q + 8);
            v[0] = fma2(ny[j], pack2(t.x, t.y), v[0]);
            v[1] = fma2(ny[j], pack2(t.z, t.w), v[1]);
            v[2] = fma2(ny[j], pack2(u.x, u.y), v[2]);
            v[3] = fma2(ny[j], pack2(u.z, u.w), v[3]);
          }
          a[2 * q] = v[0]; a[2 * q + 1] = v[1];
          a[2 * q + 2] = v[2]; a[2 * q + 3] = v[3];
          if (q == 0 && (r >> 3) == jb + 2) {
            publish(Qs[(jb + 1) & 1], v[0], v[1]);
            publish(Pre[(jb + 1) & 1], v[2], v[3]);
          }
        }
      }
      // the new columns go to global memory while the pivot warp is at work
      const int c = j0 + 4 * h;                // columns c .. c + 3 are this thread's to store
      const float mv[4] = {h ? y[4] : y[0], h ? y[5] : y[1], h ? y[6] : y[2], h ? y[7] : y[3]};
      if (r >= j0 + 8) {
        if (nb == NB) *reinterpret_cast<float4*>(Ar + c) = make_float4(mv[0], mv[1], mv[2], mv[3]);
        else if (r < nb) {
#pragma unroll
          for (int i = 0; i < 4; ++i) Ar[c + i] = mv[i];       // c + i < r < nb
        }
        if (r < nb) {
#pragma unroll
          for (int i = 0; i < 4; ++i) Ab[(long long)(c + i) * lda + r] = mv[i];
        }
      } else if (r >= j0 && r < nb) {          // pivot rows: up to the diagonal
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c + i <= r) {
            Ar[c + i] = mv[i];
            Ab[(long long)(c + i) * lda + r] = mv[i];
          }
      }
    }
  }
}

// ---- panel solve: P <- P * L^-T for the rows below a factored diagonal block -----------------
// L = the 128 x 128 lower block at (k0, k0), P = the `rest` rows below it (same columns).  Row r of
// the result is the forward substitution y_j = (p_j - sum_{i<j} y_i L[j][i]) / L[j][j]: rows are
// independent.  Two threads per row: eight columns at a time, one sums over the even and one over the
// odd earlier columns, the pair combines with one shuffle per column and both
// finish the 8 x 8 diagonal step.  The block kernel left L^T in the upper triangle of the
// diagonal block, so the tile loads as it is (coalesced, no transposition) and the inner loop
// reads eight consecutive entries L[j0..j0+7][i] as two broadcast vector loads.  Plain fp32 FMAs.
//
// Bound by the latency of the chain over columns and by shared-memory loads (an entry of L serves one row
// of a lane).  With few rows (TR 32) every SM gets its share of them: 12 to 13 us up to 9472 rows, where
// 128 rows per CTA on a quarter of the SMs
// took 21.  With more rows two CTAs of 64 share an SM: 21 us for 9472 to 14208 rows, as before (two rows
// per thread pair, which halve the loads of L, were slower for want of warps: 25 us).  Even and odd columns
// of a row lie apart in shared memory: a thread reads four of its own at once.
constexpr int TRT = 256;                   // threads per CTA (the first 2 * TR solve, all of them load)
constexpr int LPITCH = NB + 4, YPITCH = NB + 4;
template <int TR> constexpr int TRSM_SMEM = (NB * LPITCH + TR * YPITCH + NB) * (int)sizeof(float);
// With SPLIT the solved rows leave as two fp16 planes under the fixed scale L_SCALE (the products behind the
// panel are all that reads them), without as fp32 in place.
constexpr float L_SCALE = 8192.f;          // entries of L are below 2
template <int TR, bool SPLIT>              // rows per CTA
__global__ void __launch_bounds__(TRT, 2) trsm_panel_kernel(float* __restrict__ A, long long lda, int k0, int rest,
                                                         long long sW, __half* __restrict__ planes, long long plane) {
  oc_wait_before();
  A += (long long)blockIdx.y * sW;
  if (SPLIT) planes += (long long)blockIdx.y * sW * 2;
  extern __shared__ __align__(16) float sm[];
  float* Lt = sm;                           // Lt[i * LPITCH + j] = L[j][i] for j >= i
  float* Ys = sm + NB * LPITCH;             // this CTA's rows: 64 even columns, then 64 odd ones
  float* dinv = Ys + TR * YPITCH;
  const int tid = threadIdx.x;
  const float* Lkk = A + (long long)k0 * lda + k0;
  float* P = A + (long long)(k0 + NB) * lda + k0;
  const int row0 = blockIdx.x * TR;
  const int rows = min(TR, rest - row0);
#pragma unroll
  for (int it = 0; it < NB * NB / 4 / TRT; ++it) {
    const int e = it * TRT + tid, i = e / (NB / 4), j4 = e % (NB / 4);
    const float4 v = *reinterpret_cast<const float4*>(Lkk + (long long)i * lda + 4 * j4);
    *reinterpret_cast<float4*>(Lt + i * LPITCH + 4 * j4) = v;
  }
#pragma unroll
  for (int it = 0; it < TR * NB / 4 / TRT; ++it) {
    const int e = it * TRT + tid, r = e / (NB / 4), c4 = e % (NB / 4);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) v = *reinterpret_cast<const float4*>(P + (long long)(row0 + r) * lda + 4 * c4);
    *reinterpret_cast<float2*>(Ys + r * YPITCH + 2 * c4) = make_float2(v.x, v.z);
    *reinterpret_cast<float2*>(Ys + r * YPITCH + NB / 2 + 2 * c4) = make_float2(v.y, v.w);
  }
  __syncthreads();
  if (tid < NB) dinv[tid] = 1.f / Lt[tid * LPITCH + tid];
  __syncthreads();
  if (tid < 2 * TR) {
    const int part = tid & 1;
    float* y = Ys + (tid >> 1) * YPITCH;
    for (int j0 = 0; j0 < NB; j0 += 8) {
      const float4 ev = *reinterpret_cast<const float4*>(y + j0 / 2);
      const float4 od = *reinterpret_cast<const float4*>(y + NB / 2 + j0 / 2);
      f32x2 acc2[4] = {part ? 0ull : pack2(ev.x, od.x), part ? 0ull : pack2(ev.y, od.y),
                       part ? 0ull : pack2(ev.z, od.z), part ? 0ull : pack2(ev.w, od.w)};
      const float* lt = Lt + part * LPITCH + j0;
#pragma unroll 2
      for (int i4 = 0; i4 < j0 / 2; i4 += 4) {      // this thread's columns 2 (i4 + k) + part
        const float4 yv = *reinterpret_cast<const float4*>(y + part * (NB / 2) + i4);
        float4 lv[4][2];                             // all loads of the step before its arithmetic
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          lv[k][0] = *reinterpret_cast<const float4*>(lt + 2 * (i4 + k) * LPITCH);
          lv[k][1] = *reinterpret_cast<const float4*>(lt + 2 * (i4 + k) * LPITCH + 4);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const f32x2 l[4] = {pack2(lv[k][0].x, lv[k][0].y), pack2(lv[k][0].z, lv[k][0].w),
                              pack2(lv[k][1].x, lv[k][1].y), pack2(lv[k][1].z, lv[k][1].w)};
          const float yk = k == 0 ? yv.x : k == 1 ? yv.y : k == 2 ? yv.z : yv.w;
          const f32x2 ny = pack2(-yk, -yk);
#pragma unroll
          for (int c = 0; c < 4; ++c) acc2[c] = fma2(ny, l[c], acc2[c]);
        }
      }
      float acc[8];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 v = unpack2(acc2[c]);
        acc[2 * c] = v.x + __shfl_xor_sync(0xffffffffu, v.x, 1);
        acc[2 * c + 1] = v.y + __shfl_xor_sync(0xffffffffu, v.y, 1);
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float di = dinv[j0 + c];
        const float4 l0 = *reinterpret_cast<const float4*>(Lt + (j0 + c) * LPITCH + j0);
        const float4 l1 = *reinterpret_cast<const float4*>(Lt + (j0 + c) * LPITCH + j0 + 4);
        const float lr[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
        const float yc = acc[c] * di;
        acc[c] = yc;
#pragma unroll
        for (int c2 = c + 1; c2 < 8; ++c2) acc[c2] = fmaf(-yc, lr[c2], acc[c2]);
      }
      // each partner keeps its own columns
      *reinterpret_cast<float4*>(y + part * (NB / 2) + j0 / 2) =
          part ? make_float4(acc[1], acc[3], acc[5], acc[7]) : make_float4(acc[0], acc[2], acc[4], acc[6]);
      __syncwarp();
    }
  }
  __syncthreads();
  oc_let_next();
#pragma unroll
  for (int it = 0; it < TR * NB / 4 / TRT; ++it) {
    const int e = it * TRT + tid, r = e / (NB / 4), c4 = e % (NB / 4);
    if (r < rows) {
      const float2 ev = *reinterpret_cast<const float2*>(Ys + r * YPITCH + 2 * c4);
      const float2 od = *reinterpret_cast<const float2*>(Ys + r * YPITCH + NB / 2 + 2 * c4);
      if (SPLIT) {
        uint2 hi, lo;
        oc_split4(make_float4(ev.x * L_SCALE, od.x * L_SCALE, ev.y * L_SCALE, od.y * L_SCALE), hi, lo);
        __half* to = planes + (long long)(k0 + NB + row0 + r) * lda + k0 + 4 * c4;
        *reinterpret_cast<uint2*>(to) = hi;
        *reinterpret_cast<uint2*>(to + plane) = lo;
      } else {
        *reinterpret_cast<float4*>(P + (long long)(row0 + r) * lda + 4 * c4) = make_float4(ev.x, od.x, ev.y, od.y);
      }
    }
  }
}

template <int TR, bool SPLIT>
int launch_trsm(float* A, long long ld, int k0, int rest, int batch, long long sW, __half* planes, long long plane,
                cudaStream_t stream) {
  OC_OPT_IN_SMEM((trsm_panel_kernel<TR, SPLIT>), TRSM_SMEM<TR>);
  OC_LAUNCH((trsm_panel_kernel<TR, SPLIT>), dim3(oc_div_up(rest, TR), batch), TRT, TRSM_SMEM<TR>, stream, A, ld, k0, rest, sW,
            planes, plane);
  return OC_OK;
}

// ---- inverses of all diagonal blocks of L, one CTA per block (off the critical path) ----------
// L block (nb x nb, lower) -> L^-1 written to the matching block of X (lower part; upper part
// zero).  The 8 x 8 diagonal blocks are inverted at once, then neighbouring inverted blocks are
// joined level by level (four levels, two small products each).  Bound by the latency of those products'
// loads: with 256 threads, two steps of k in flight and one entry per global access 33 us, now 23 us.
constexpr int DINV_T = 512;
constexpr int DINV_SMEM = (2 * NB * (NB + 1) + (NB / 2) * (NB / 2)) * (int)sizeof(float);
__global__ void __launch_bounds__(DINV_T) diag_inverse_kernel(const float* __restrict__ A, long long lda,
                                                           float* __restrict__ X, long long ldx, int n,
                                                           long long sW, __half* __restrict__ planes, long long plane,
                                                           float* __restrict__ table, int ldt) {
  oc_wait_before();
  A += (long long)blockIdx.y * sW;
  X += (long long)blockIdx.y * sW;
  extern __shared__ __align__(16) float sm[];
  float (*S)[NB + 1] = reinterpret_cast<float (*)[NB + 1]>(sm);                    // L
  float (*Y)[NB + 1] = reinterpret_cast<float (*)[NB + 1]>(sm + NB * (NB + 1));    // L^-1
  float* T = sm + 2 * NB * (NB + 1);                                               // [64 * 64]
  const int tid = threadIdx.x;
  const int k0 = blockIdx.x * NB, nb = min(NB, n - k0);
  const float* Ab = A + (long long)k0 * lda + k0;
  float* Xb = X + (long long)k0 * ldx + k0;
  if (nb == NB) {                                   // 16-byte accesses, all in flight at once
    float4 v[NB * NB / 4 / DINV_T];
#pragma unroll
    for (int it = 0; it < NB * NB / 4 / DINV_T; ++it) {
      const int e = it * DINV_T + tid, r = e / (NB / 4), c = e % (NB / 4) * 4;
      v[it] = c <= r ? *reinterpret_cast<const float4*>(Ab + (long long)r * lda + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int it = 0; it < NB * NB / 4 / DINV_T; ++it) {
      const int e = it * DINV_T + tid, r = e / (NB / 4), c = e % (NB / 4) * 4;
      const float x[4] = {v[it].x, v[it].y, v[it].z, v[it].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { S[r][c + i] = c + i <= r ? x[i] : 0.f; Y[r][c + i] = 0.f; }
    }
  } else {
    for (int e = tid; e < NB * NB; e += DINV_T) {
      const int r = e / NB, c = e % NB;
      S[r][c] = (r < nb && c <= r) ? Ab[(long long)r * lda + c] : ((r == c) ? 1.f : 0.f);
      Y[r][c] = 0.f;
    }
  }
  __syncthreads();
  if (tid < NB) {
    const int i0 = (tid >> 3) * 8, t = tid & 7;     // column t of the inverse of diagonal block i0
    float x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float acc = (r == t) ? 1.f : 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < r) acc = fmaf(-S[i0 + r][i0 + q], x[q], acc);
      x[r] = (r >= t) ? acc / S[i0 + r][i0 + r] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) Y[i0 + r][i0 + t] = x[r];
  }
  __syncthreads();
  for (int sz = 8; sz < NB; sz *= 2) {
    // (NB / (2 sz)) problems of sz x sz elements; a thread takes strips of four rows of one column,
    // i.e. four independent sums per pass over k
    const int strips = (NB / 8) * sz;
    const int lg = 31 - __clz(sz);
    for (int e = tid; e < strips; e += DINV_T) {       // T = L21 * X11 (X11 lower triangular)
      const int j = e & (sz - 1), i = ((e >> lg) & (sz / 4 - 1)) * 4, m = e >> (2 * lg - 2);
      const int q0 = 2 * sz * m, mid = q0 + sz;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int k = j; k < sz; ++k) {
        const float y = Y[q0 + k][q0 + j];
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) acc[ii] = fmaf(S[mid + i + ii][q0 + k], y, acc[ii]);
      }
#pragma unroll
      for (int ii = 0; ii < 4; ++ii) T[(m << (2 * lg)) + ((i + ii) << lg) + j] = acc[ii];
    }
    __syncthreads();
    for (int e = tid; e < strips; e += DINV_T) {       // X21 = -X22 * T (X22 lower triangular)
      const int j = e & (sz - 1), i = ((e >> lg) & (sz / 4 - 1)) * 4, m = e >> (2 * lg - 2);
      const int q0 = 2 * sz * m, mid = q0 + sz;
      const float* tcol = T + (m << (2 * lg)) + j;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int k = 0; k < i + 4; ++k) {              // X22[i + ii][k] = 0 for k > i + ii
        const float t = tcol[k << lg];
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) acc[ii] = fmaf(Y[mid + i + ii][mid + k], t, acc[ii]);
      }
#pragma unroll
      for (int ii = 0; ii < 4; ++ii) Y[mid + i + ii][q0 + j] = -acc[ii];
    }
    __syncthreads();
  }
  oc_let_next();
  if (nb == NB) {
#pragma unroll 4
    for (int it = 0; it < NB * NB / 4 / DINV_T; ++it) {
      const int e = it * DINV_T + tid, i = e / (NB / 4), j = e % (NB / 4) * 4;
      *reinterpret_cast<float4*>(Xb + (long long)i * ldx + j) =
          make_float4(Y[i][j], Y[i][j + 1], Y[i][j + 2], Y[i][j + 3]);   // (zero above the diagonal)
    }
  } else {
    for (int e = tid; e < nb * NB; e += DINV_T) {
      const int i = e / NB, j = e % NB;
      if (j < nb) Xb[(long long)i * ldx + j] = (j <= i) ? Y[i][j] : 0.f;
    }
  }
  // A product with the lower triangular X starts its k-range at its tile's first column; tiles are up
  // to 256 columns wide and start at even blocks, so they also read the block right of an even
  // diagonal block.  Nothing else above the diagonal blocks is ever read.
  const int width = (blockIdx.x & 1) == 0 ? min(NB, n - k0 - NB) : 0;
  if (!planes) {
    for (int e = tid; e < nb * NB; e += DINV_T)
      if (e % NB < width) Xb[(long long)(e / NB) * ldx + NB + e % NB] = 0.f;
    return;
  }
  // the products read the two planes of X (split.cuh; block scales)
  planes += (long long)blockIdx.y * sW * 2 + (long long)k0 * ldx + k0;
  table += (long long)blockIdx.y * sW + (long long)blockIdx.x * (ldt + 1);
  float mx = 0.f;
  for (int e = tid; e < NB * NB; e += DINV_T) mx = fmaxf(mx, oc_finite_abs(Y[e / NB][e % NB]));
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) T[tid >> 5] = mx;                // (the joins' scratch is free)
  __syncthreads();
  mx = 0.f;
  for (int w = 0; w < DINV_T / 32; ++w) mx = fmaxf(mx, T[w]);
  float inv;
  const float sc = oc_split_scale(mx, inv);
  if (tid == 0) {
    table[0] = inv;
    if (width > 0) table[1] = 1.f;
  }
#pragma unroll 4
  for (int e = tid; e < NB * NB / 4; e += DINV_T) {
    const int i = e / (NB / 4), j = e % (NB / 4) * 4;
    if (i >= nb) break;
    __half* to = planes + (long long)i * ldx + j;
    uint2 hi, lo;
    if (j < nb) {      // (entries behind the last column are zero, and rows are padded to groups of eight)
      oc_split4(make_float4(Y[i][j] * sc, j + 1 < nb ? Y[i][j + 1] * sc : 0.f, j + 2 < nb ? Y[i][j + 2] * sc : 0.f,
                            j + 3 < nb ? Y[i][j + 3] * sc : 0.f), hi, lo);
      *reinterpret_cast<uint2*>(to) = hi;
      *reinterpret_cast<uint2*>(to + plane) = lo;
    }
    if (j < width) {
      *reinterpret_cast<uint2*>(to + NB) = make_uint2(0u, 0u);
      *reinterpret_cast<uint2*>(to + NB + plane) = make_uint2(0u, 0u);
    }
  }
}

}  // namespace

// Workspace of one problem (floats, rows ld = round_up(n, 8) apart): A, X, T fp32; the fp16 planes of L and X (two planes
// take the room of one fp32 matrix); vectors of n; block tables of X and T.  The planes of T take A's place:
// behind the Cholesky factorisation nothing reads A.  A batch keeps the problems' workspaces one after another.
struct FactorWs {
  long long ld, mat, nblk, total;
  explicit FactorWs(int n) {
    ld = (n + 7) / 8 * 8; mat = (long long)n * ld; nblk = (n + NB - 1) / NB;
    total = (5 * mat + 3 * ld + 2 * ((nblk * nblk + 3) / 4 * 4) + 63) / 64 * 64;
  }
  float* A(float* w) const { return w; }
  float* X(float* w) const { return w + mat; }
  float* T(float* w) const { return w + 2 * mat; }
  __half* planesL(float* w) const { return reinterpret_cast<__half*>(w + 3 * mat); }
  __half* planesX(float* w) const { return reinterpret_cast<__half*>(w + 4 * mat); }
  __half* planesT(float* w) const { return reinterpret_cast<__half*>(w); }
  float* diagv(float* w) const { return w + 5 * mat; }
  float* equil(float* w) const { return w + 5 * mat + ld; }
  float* equil_p(float* w) const { return w + 5 * mat + 2 * ld; }
  float* tableX(float* w) const { return w + 5 * mat + 3 * ld; }
  float* tableT(float* w) const { return w + 5 * mat + 3 * ld + (nblk * nblk + 3) / 4 * 4; }
};
static long long factor_ws_floats(int n) { return FactorWs(n).total; }

extern "C" long long oc_hinv_workspace_bytes(int n) { return factor_ws_floats(n) * 4; }

// `count` problems of one level of the blocked inverse, for `batch` matrices: T21 = L21 X11, X21 = -X22 T21 with
// X11, X22 of s and `rows` rows, the first at row and column r0, `step` entries apart.  T and X21 (unless no level
// follows) leave as planes for the products that read them.
static int invert_level_split(const FactorWs& ws, float* w0, int s, long long r0, int rows, int count, long long step,
                              int batch, long long sW, bool more, cudaStream_t stream) {
  const long long ld = ws.ld, mid = r0 + s, at = mid * ld + r0;
  const long long nblk = ws.nblk, tab_step = 2 * (s / NB) * (nblk + 1), tab_at = mid / NB * nblk + r0 / NB;
  auto operand = [&](__half* planes, long long row, long long col, float* table) {
    OcSplitOperand o{};
    o.planes = planes + row * ld + col; o.plane = ws.mat; o.ld = ld; o.terms = 2;
    o.stride1 = step; o.stride2 = 2 * sW;
    if (table) {
      o.scale = table + row / NB * nblk + col / NB; o.scale1 = tab_step; o.scale2 = sW;
      o.scale_k = 1; o.scale_r = nblk;
    }
    return o;
  };
  auto stored_by_k = [](OcSplitOperand o) {
    o.mn_major = 1;
    const long long t = o.scale_k; o.scale_k = o.scale_r; o.scale_r = t;
    return o;
  };
  auto goes_on = [&](OcSplitGemm& g, __half* planes, float* table, int only) {
    g.out.mode = OC_SPLIT_OUT_BLOCKS; g.out.only = only;
    g.out.planes = planes + at; g.out.plane = ws.mat; g.out.ld = ld; g.out.table = table + tab_at; g.out.ldt = nblk;
    g.out.stride1 = step; g.out.stride2 = 2 * sW; g.out.tab1 = tab_step; g.out.tab2 = sW;
  };
  OcSplitGemm g{};
  g.ldc = ld; g.strideC1 = step; g.strideC2 = sW; g.nb1 = count; g.nb2 = batch; g.M = rows; g.N = s;
  g.A = operand(ws.planesL(w0), mid, r0, nullptr);
  g.B = stored_by_k(operand(ws.planesX(w0), r0, r0, ws.tableX(w0)));
  g.C = ws.T(w0) + at; g.K = s; g.alpha = 1.f / L_SCALE; g.flags = OC_GEMM_KLO_FROM_N;
  goes_on(g, ws.planesT(w0), ws.tableT(w0), 1);
  const int rc = oc_gemm_split_launch(g, stream);
  if (rc) return rc;
  g.A = operand(ws.planesX(w0), mid, mid, ws.tableX(w0));
  g.B = stored_by_k(operand(ws.planesT(w0), mid, r0, ws.tableT(w0)));
  g.C = ws.X(w0) + at; g.K = rows; g.alpha = -1.f; g.flags = OC_GEMM_KHI_FROM_M;
  if (more) goes_on(g, ws.planesX(w0), ws.tableX(w0), 0);
  else g.out = OcSplitOut{};
  return oc_gemm_split_launch(g, stream);
}

// Factorisation of `batch` matrices of equal size laid out one after another (H [batch, n, ldh],
// U [batch, n, ldu], perm / invperm / dead [batch, n], damp_out [batch, 2], status [batch]).  The
// panel chain is walked once; every launch covers all problems.
static int hinv_factor_impl(int batch, const float* H, long long ldh, int n, float percdamp, float rel_shift,
                            int actorder, int reuse_perm, float* U, long long ldu, int* perm, int* invperm,
                            unsigned char* dead, float* damp_out, int* status, void* workspace,
                            long long workspace_bytes, cudaStream_t stream) {
  OC_REQUIRE(H && U && perm && invperm && dead && damp_out && status && workspace, "hinv_factor: null pointer");
  OC_REQUIRE(n > 0 && ldh >= n && ldu >= n, "hinv_factor: bad dimensions");
  OC_REQUIRE(batch >= 1 && batch <= 65535, "hinv_factor: batch must be in 1..65535");
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  // (full panels are read and written 16 bytes at a time)
  OC_REQUIRE(n < NB || aligned(workspace), "hinv_factor: the workspace must be 16-byte aligned");
  const long long sW = factor_ws_floats(n);
  if (workspace_bytes < sW * 4 * batch) {
    oc_set_last_error("hinv_factor: workspace too small");
    return OC_ERR_WORKSPACE;
  }
  const FactorWs ws(n);
  const long long ld = ws.ld;
  const long long sH = (long long)n * ldh, sU = (long long)n * ldu;
  float* w0 = (float*)workspace;
  float *A = ws.A(w0), *X = ws.X(w0), *T = ws.T(w0);
  float *diagv = ws.diagv(w0), *equil = ws.equil(w0), *equil_p = ws.equil_p(w0);
  const bool split = oc_split_engine_on() && n > NB;     // (and then the workspace is aligned)

  OC_LAUNCH(diag_stats_kernel, batch, 1024, 0, stream, H, ldh, n, percdamp, rel_shift, diagv, dead, damp_out, equil, status,
            sH, sW);
  const int tb = 256, gb = oc_div_up(n, tb);
  if (!reuse_perm) {
    if (actorder) {
      OC_LAUNCH(rank_sort_kernel, dim3(gb, batch), tb, 0, stream, diagv, n, perm, sW);
      OC_LAUNCH(invert_perm_kernel, dim3(gb, batch), tb, 0, stream, perm, invperm, n);
    } else {
      OC_LAUNCH(iota_kernel, dim3(gb, batch), tb, 0, stream, perm, invperm, n);
    }
  }
  const bool vec_h = n % 4 == 0 && ldh % 4 == 0 && sH % 4 == 0 && aligned(H) && aligned(A);
  // (with reuse_perm the caller's perm counts, whatever actorder says)
  const int permuted = actorder || reuse_perm;
  const bool staged = permuted && n <= BUILD_STAGED_N;
  if (staged) OC_OPT_IN_SMEM(build_reversed_kernel, BUILD_STAGED_N * 4);
  OC_LAUNCH(build_reversed_kernel, dim3(n, batch), 256, staged ? n * 4 : 0, stream,
            H, ldh, n, perm, permuted, diagv, damp_out, rel_shift, equil, equil_p, A, ld, sH, sW, vec_h, staged);

  // ---- blocked right-looking Cholesky --------------------------------------------------
  OC_OPT_IN_SMEM(diag_inverse_kernel, DINV_SMEM);
  __half* Lp = ws.planesL(w0);
  // C -= P P^T for the rows of L below `r0`, columns [c0, c0 + k): lower tiles of the N columns from r0 on
  auto update = [&](int r0, int c0, int k, int M, int N) {
    if (split) {
      OcSplitGemm g{};
      g.A.planes = Lp + (long long)r0 * ld + c0; g.A.plane = ws.mat; g.A.ld = ld; g.A.terms = 2;
      g.A.stride2 = 2 * sW;
      g.B = g.A;
      g.C = A + (long long)r0 * ld + r0; g.ldc = ld; g.strideC2 = sW;
      g.M = M; g.N = N; g.K = k; g.nb1 = 1; g.nb2 = batch;
      g.alpha = -1.f / (L_SCALE * L_SCALE); g.add = 1; g.flags = OC_GEMM_SKIP_UPPER_TILES;
      return oc_gemm_split_launch(g, stream);
    }
    OcGemm g{};
    g.A = A + (long long)r0 * ld + c0; g.lda = ld; g.B = g.A; g.ldb = ld; g.transB = 1;
    g.C = A + (long long)r0 * ld + r0; g.ldc = ld;
    g.M = M; g.N = N; g.K = k; g.alpha = -1.f; g.beta = 1.f; g.flags = OC_GEMM_SKIP_UPPER_TILES;
    g.batch = batch; g.strideA = g.strideB = g.strideC = sW;
    return oc_gemm_f32_launch(g, stream);
  };
  // Two levels: inside an outer block of OB columns every 128-column panel updates only the
  // rest of that outer block (full height); the matrix behind the outer block is updated once per
  // outer block with K = OB, so it is read and written n/OB times instead of n/128 times.
  // Per panel the serial chain is: factor the diagonal block (one SM), solve the rows below it
  // against that block (all SMs, fp32 FMAs), update the rest of the outer block (tensor cores).
  for (int K0 = 0; K0 < n; K0 += OB) {
    const int kend = min(n, K0 + OB);
    for (int k0 = K0; k0 < kend; k0 += NB) {
      const int nb = min(NB, n - k0);
      OC_LAUNCH(potrf_block_kernel, batch, ROW_THREADS + 32, 0, stream, A, ld, k0, nb, status, sW);
      const int rest = n - k0 - nb;
      if (rest <= 0) break;
      OC_REQUIRE(nb == NB, "hinv_factor: a panel with rows below it is a full panel");
      // the fewer rows per CTA, the shorter its time, as long as all CTAs run at once (one or two on each
      // of a B200's 148 SMs)
      const long long row_sets = (long long)oc_div_up(rest, 32) * batch;
      const bool few = row_sets <= 2 * 148;
      const int rc_t = split ? (few ? launch_trsm<32, true>(A, ld, k0, rest, batch, sW, Lp, ws.mat, stream)
                                    : launch_trsm<64, true>(A, ld, k0, rest, batch, sW, Lp, ws.mat, stream))
                             : (few ? launch_trsm<32, false>(A, ld, k0, rest, batch, sW, nullptr, 0, stream)
                                    : launch_trsm<64, false>(A, ld, k0, rest, batch, sW, nullptr, 0, stream));
      if (rc_t) return rc_t;
      const int inner = kend - (k0 + nb);
      if (inner <= 0) continue;
      // columns [k0+nb, kend) of all rows below the panel's diagonal block
      const int rc = update(k0 + nb, k0, nb, rest, inner);
      if (rc) return rc;
    }
    const int rest2 = n - kend;
    if (rest2 <= 0) break;
    // trailing <- trailing - P * P^T with P = L[kend.., K0..kend)
    const int rc2 = update(kend, K0, kend - K0, rest2, rest2);
    if (rc2) return rc2;
  }
  // inverses of the diagonal blocks, all at once: the seeds of the blocked inverse below
  OC_LAUNCH(diag_inverse_kernel, dim3(oc_div_up(n, NB), batch), DINV_T, DINV_SMEM, stream,
            A, ld, X, ld, n, sW, split ? ws.planesX(w0) : nullptr, ws.mat, ws.tableX(w0), (int)ws.nblk);

  // ---- recursive blocked inverse of L: X holds the inverted diagonal blocks -----------------
  // The uniform problems of a level form one batched product (of both batch dimensions: problems and
  // matrices); a last problem with fewer rows has its own.
  for (long long s = NB; s < n; s *= 2) {
    const int nprob = (int)((n + 2 * s - 1) / (2 * s));
    const int nfull = (int)(n / (2 * s));
    const long long mid_last = 2 * s * nfull + s;
    // (first problem, count, rows of the lower block)
    struct Launch { int first, count, rows; };
    Launch list[2];
    int nl = 0;
    if (nfull > 0) list[nl++] = {0, nfull, (int)s};
    if (nfull < nprob && mid_last < n) list[nl++] = {nfull, 1, (int)(n - mid_last)};
    for (int li = 0; li < nl; ++li) {
      const int count = list[li].count, rows = list[li].rows;
      const long long r0 = 2 * s * list[li].first, mid = r0 + s, step = 2 * s * (ld + 1);
      if (split) {
        const int rc = invert_level_split(ws, w0, (int)s, r0, rows, count, step, batch, sW, 2 * s < n, stream);
        if (rc) return rc;
        continue;
      }
      // (the FMA engine has one batch dimension: the matrices of a batch one by one)
      for (int b = 0; b < batch; ++b) {
        float *Ab = A + b * sW, *Xb = X + b * sW, *Tb = T + b * sW;
        OcGemm g1{};  // T21 = L21 * X11   (X11 lower triangular)
        g1.A = Ab + mid * ld + r0; g1.lda = ld; g1.strideA = step;
        g1.B = Xb + r0 * ld + r0; g1.ldb = ld; g1.strideB = step;
        g1.C = Tb + mid * ld + r0; g1.ldc = ld; g1.strideC = step;
        g1.M = rows; g1.N = (int)s; g1.K = (int)s; g1.alpha = 1.f; g1.beta = 0.f;
        g1.flags = OC_GEMM_KLO_FROM_N; g1.batch = count;
        int rc = oc_gemm_f32_launch(g1, stream);
        if (rc) return rc;
        OcGemm g2{};  // X21 = -X22 * T21  (X22 lower triangular)
        g2.A = Xb + mid * ld + mid; g2.lda = ld; g2.strideA = step;
        g2.B = Tb + mid * ld + r0; g2.ldb = ld; g2.strideB = step;
        g2.C = Xb + mid * ld + r0; g2.ldc = ld; g2.strideC = step;
        g2.M = rows; g2.N = (int)s; g2.K = rows; g2.alpha = -1.f; g2.beta = 0.f;
        g2.flags = OC_GEMM_KHI_FROM_M; g2.batch = count;
        rc = oc_gemm_f32_launch(g2, stream);
        if (rc) return rc;
      }
    }
  }
  const bool vec_u = n % 4 == 0 && ldu % 4 == 0 && sU % 4 == 0 && aligned(U) && aligned(X);
  OcGemmDevice dev;
  if (const int rc = oc_gemm_device(dev)) return rc;
  OC_LAUNCH(reverse_upper_kernel, dim3(n, batch), 256, 0, stream, X, ld, n, equil_p, U, ldu, sW, sU, vec_u, dev.status, status);
  return OC_OK;
}

// See include/onecomp_b200.h for the contracts.
extern "C" int oc_hinv_factor(const float* H, long long ldh, int n, float percdamp, float rel_shift,
                              int actorder, int reuse_perm, float* U, long long ldu, int* perm,
                              int* invperm, unsigned char* dead, float* damp_out, int* status,
                              void* workspace, long long workspace_bytes, void* stream) {
  return hinv_factor_impl(1, H, ldh, n, percdamp, rel_shift, actorder, reuse_perm, U, ldu, perm, invperm, dead,
                          damp_out, status, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int oc_hinv_factor_batched(int batch, const float* H, int n, float percdamp, int actorder, float* U,
                                      int* perm, int* invperm, unsigned char* dead, float* damp_out,
                                      int* status, void* workspace, long long workspace_bytes, void* stream) {
  return hinv_factor_impl(batch, H, n, n, percdamp, 1.f, actorder, 0, U, n, perm, invperm, dead, damp_out,
                          status, workspace, workspace_bytes, (cudaStream_t)stream);
}
