// QEP weight correction  W <- fp16( W + perccorr * (W C) (H + damp I)^-1 )
// (reference: Quantizer.adjust_weight, onecomp/quantizer/_quantizer.py:362-432).
//
// The reference factors H + damp I and solves with potrf + potrs.  Here the
// inverse-Hessian factor U of the same damped matrix (U^T U = (P H P^T + damp I)^-1,
// P the act-order permutation or the identity) is already at hand for the GPTQ
// column loop, so the solve becomes two triangular products:   dW P^T = ((W C) P^T) U^T U.
// The three products run on the tensor cores with operands in two fp16 planes (split.cuh); the weight, 16 bits
// wide, needs one plane.
#include "split.cuh"

namespace {

// The elementwise passes take four columns a thread where rows are aligned (`vec`), one otherwise.
__device__ __forceinline__ float4 ld16x4(const void* p, long long i, int bf16) {
  const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const char*>(p) + i * 2);
  float2 a, b;
  if (bf16) {
    a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  } else {
    a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  }
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ float4 load_masked(const void* W, long long i, int c, const unsigned char* dead, int bf16) {
  float4 v = ld16x4(W, i, bf16);
  if (dead) {
    const unsigned m = *reinterpret_cast<const unsigned*>(dead + c);
    if (m & 0xffu) v.x = 0.f;
    if (m & 0xff00u) v.y = 0.f;
    if (m & 0xff0000u) v.z = 0.f;
    if (m & 0xff000000u) v.w = 0.f;
  }
  return v;
}

__global__ void qep_load_kernel(const void* __restrict__ W, long long ldw_in, int out, int d,
                                const unsigned char* __restrict__ dead, float* __restrict__ Wf,
                                long long ldw, int bf16, int vec) {
  const int r = blockIdx.y;
  if (vec) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (c < d) *reinterpret_cast<float4*>(Wf + (long long)r * ldw + c) = load_masked(W, (long long)r * ldw_in + c, c, dead, bf16);
    return;
  }
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d) return;
  const float v = oc_ld16(W, (long long)r * ldw_in + c, bf16);
  Wf[(long long)r * ldw + c] = (dead && dead[c]) ? 0.f : v;
}

// W with dead columns zeroed as one fp16 plane: an fp16 weight as it is; a bf16 weight with every row of 128 columns
// scaled by a power of two (table, entry chunk * out + row), which keeps its 8 bits.  One warp per row of 128.
__global__ void __launch_bounds__(256) qep_plane_kernel(const void* __restrict__ W, long long ldw_in, int out, int d,
                                                        const unsigned char* __restrict__ dead, __half* __restrict__ plane,
                                                        long long ldp, float* __restrict__ table, int bf16, int vec) {
  oc_wait_before();
  oc_let_next();
  const int lane = threadIdx.x & 31, r = blockIdx.y * 8 + (threadIdx.x >> 5), c = blockIdx.x * 128 + lane * 4;
  if (r >= out) return;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < d) {
    if (vec) {
      const float4 t = load_masked(W, (long long)r * ldw_in + c, c, dead, bf16);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < d && !(dead && dead[c + j])) v[j] = oc_ld16(W, (long long)r * ldw_in + c + j, bf16);
    }
  }
  if (bf16) {
    float mx = fmaxf(fmaxf(oc_finite_abs(v[0]), oc_finite_abs(v[1])), fmaxf(oc_finite_abs(v[2]), oc_finite_abs(v[3])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float inv;
    const float s = oc_split_scale(mx, inv);
    if (lane == 0) table[(long long)blockIdx.x * out + r] = inv;
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] *= s;
  }
  if (c >= d) return;
  const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(plane + (long long)r * ldp + c) =
      make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}

__global__ void gather_cols_kernel(const float* __restrict__ src, long long lds, int out, int d,
                                   const int* __restrict__ perm, float* __restrict__ dst, long long ldd) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= d) return;
  dst[(long long)r * ldd + i] = src[(long long)r * lds + perm[i]];
}

// W[r][perm[i]] = round16( Wz[r][perm[i]] + perccorr * T[r][i] ) in the weight's own 16-bit type, where
// Wz is W with its dead columns zeroed
__global__ void qep_store_kernel(const unsigned char* __restrict__ dead, const float* __restrict__ T,
                                 long long ldt, int out, int d, const int* __restrict__ perm,
                                 float perccorr, void* __restrict__ W, long long ldw_out, int bf16, int vec) {
  oc_wait_before();
  oc_let_next();
  const int r = blockIdx.y;
  if (vec) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (c >= d) return;
    const long long at = (long long)r * ldw_out + c;
    const float4 w = load_masked(W, at, c, dead, bf16);
    const float4 t = *reinterpret_cast<const float4*>(T + (long long)r * ldt + c);
    const float v[4] = {w.x + perccorr * t.x, w.y + perccorr * t.y, w.z + perccorr * t.z, w.w + perccorr * t.w};
    uint2 o;
    if (bf16) {
      *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(v[0], v[1]);
      *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(v[2], v[3]);
    } else {
      *reinterpret_cast<__half2*>(&o.x) = __floats2half2_rn(v[0], v[1]);
      *reinterpret_cast<__half2*>(&o.y) = __floats2half2_rn(v[2], v[3]);
    }
    *reinterpret_cast<uint2*>(static_cast<char*>(W) + at * 2) = o;
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d) return;
  const int c = perm ? perm[i] : i;
  const float wz = (dead && dead[c]) ? 0.f : oc_ld16(W, (long long)r * ldw_out + c, bf16);
  const float v = wz + perccorr * T[(long long)r * ldt + i];
  oc_st16(W, (long long)r * ldw_out + c, v, bf16);
}

long long round4(long long x) { return (x + 3) / 4 * 4; }

long long round8(long long x) { return (x + 7) / 8 * 8; }
long long blocks(long long x) { return (x + OC_SPLIT_BLOCK - 1) / OC_SPLIT_BLOCK; }

// Workspace with split operands: planes of the left operands, in turn (a product reads one and writes the other), an
// fp32 result, the planes of C (later those of U), and their tables.
struct QepWs {
  long long ld, left, right, tab_rows, tab, total;
  QepWs(int out, int d) {
    ld = round8(d);
    left = 4 * (long long)out * ld; right = 4 * (long long)d * ld;
    tab_rows = round8(blocks(d) * out) * 4; tab = round8(blocks(d) * blocks(d)) * 4;
    total = 3 * left + right + 2 * tab_rows + tab;
  }
};

// dW P^T (fp32, ws.ld apart) into the workspace; returned in `delta`
int split_products(const void* W, long long ldw_io, int out, int d, const float* C, long long ldc, const float* U,
                   long long ldu, const int* perm, const unsigned char* dead, int bf16, int vec, char* workspace,
                   float*& delta, cudaStream_t stream) {
  const QepWs ws(out, d);
  __half* Lp[2] = {(__half*)workspace, (__half*)(workspace + ws.left)};
  float* R = (float*)(workspace + 2 * ws.left);
  __half* Rp = (__half*)(workspace + 3 * ws.left);
  char* tabs = workspace + 3 * ws.left + ws.right;
  float* tabL[2] = {(float*)tabs, (float*)(tabs + ws.tab_rows)};
  float* tabR = (float*)(tabs + 2 * ws.tab_rows);
  const long long nb = blocks(d), plane_l = out * ws.ld, plane_r = d * ws.ld;
  delta = R;
  OC_LAUNCH(qep_plane_kernel, dim3((int)nb, oc_div_up(out, 8)), 256, 0, stream, W, ldw_io, out, d, dead, Lp[0], ws.ld, tabL[0], bf16, vec);
  OcSplitArgs right{};
  right.rows = right.cols = d; right.planes = Rp; right.plane = plane_r; right.ldp = ws.ld; right.table = tabR;
  right.ldt = nb; right.nb1 = right.nb2 = 1;
  right.src = C; right.ld = ldc;
  int rc = oc_split_launch(right, stream);
  if (rc) return rc;
  OcSplitGemm g{};
  g.C = R; g.ldc = ws.ld; g.M = out; g.N = d; g.K = d; g.nb1 = g.nb2 = 1; g.alpha = 1.f;
  g.A.plane = plane_l; g.A.ld = ws.ld; g.A.scale_k = out; g.A.scale_r = OC_SPLIT_BLOCK; g.A.scale_row = 1;
  g.B.planes = Rp; g.B.plane = plane_r; g.B.ld = ws.ld; g.B.terms = 2; g.B.scale = tabR;
  auto left = [&](int i) { g.A.planes = Lp[i]; g.A.scale = tabL[i]; };
  auto goes_on = [&](int i) {      // the result is the next left operand
    g.out.mode = OC_SPLIT_OUT_ROWS; g.out.only = 1; g.out.planes = Lp[i]; g.out.plane = plane_l; g.out.ld = ws.ld;
    g.out.table = tabL[i]; g.out.ldt = out;
  };
  // R = Wz C
  left(0);
  g.A.terms = 1;
  if (!bf16) g.A.scale = nullptr;
  g.B.mn_major = 1; g.B.scale_k = nb; g.B.scale_r = 1;
  if (!perm) goes_on(1);
  rc = oc_gemm_split_launch(g, stream);
  if (rc) return rc;
  if (perm) {
    OcSplitArgs s{};
    s.src = R; s.ld = ws.ld; s.perm = perm; s.rows = out; s.cols = d; s.planes = Lp[1]; s.plane = plane_l; s.ldp = ws.ld;
    s.table = tabL[1]; s.ldt = out; s.per_row = 1; s.nb1 = s.nb2 = 1;
    rc = oc_split_launch(s, stream);
    if (rc) return rc;
  }
  // T = R P^T U^T      (U upper: U[n][k] = 0 for k < n)
  right.src = U; right.ld = ldu; right.region = OC_SPLIT_UPPER;
  rc = oc_split_launch(right, stream);
  if (rc) return rc;
  left(1);
  g.A.terms = 2;
  g.B.mn_major = 0; g.B.scale_k = 1; g.B.scale_r = nb; g.flags = OC_GEMM_KLO_FROM_N;
  goes_on(0);
  rc = oc_gemm_split_launch(g, stream);
  if (rc) return rc;
  // dW P^T = T U       (U[k][n] = 0 for k > n)
  left(0);
  g.B.mn_major = 1; g.B.scale_k = nb; g.B.scale_r = 1; g.flags = OC_GEMM_KHI_FROM_N;
  g.out = OcSplitOut{};
  return oc_gemm_split_launch(g, stream);
}

}  // namespace

extern "C" long long oc_qep_workspace_bytes(int out, int d) {
  const long long plain = 3 * (long long)out * round4(d) * 4, split = QepWs(out, d).total;
  return (plain > split ? plain : split) + 256;
}

// See include/onecomp_b200.h for the contract.
extern "C" int oc_qep_adjust(void* W_, long long ldw_io, int out, int d, const float* C, long long ldc,
                             const float* U, long long ldu, const int* perm, const unsigned char* dead,
                             float perccorr, int w_dtype, void* workspace, long long workspace_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  void* W = W_;
  OC_REQUIRE(w_dtype == OC_DTYPE_F16 || w_dtype == OC_DTYPE_BF16, "qep_adjust: unknown weight dtype");
  const int bf16 = w_dtype == OC_DTYPE_BF16;
  OC_REQUIRE(W && C && U && workspace && out > 0 && d > 0, "qep_adjust: bad arguments");
  OC_REQUIRE(ldw_io >= d && ldc >= d && ldu >= d, "qep_adjust: bad leading dimension");
  OC_REQUIRE(out <= 65535, "qep_adjust: more than 65535 rows in one call");
  if (workspace_bytes < oc_qep_workspace_bytes(out, d)) {
    oc_set_last_error("qep_adjust: workspace too small");
    return OC_ERR_WORKSPACE;
  }
  const long long ld = round4(d);
  float* Wf = (float*)workspace;
  float* A = Wf + (long long)out * ld;
  float* B = A + (long long)out * ld;
  const int tb = 256;
  dim3 grid(oc_div_up(d, tb), out);
  const bool vec = d % 4 == 0 && ldw_io % 4 == 0 && (reinterpret_cast<uintptr_t>(W) & 7) == 0 &&
                   (reinterpret_cast<uintptr_t>(Wf) & 15) == 0 && (reinterpret_cast<uintptr_t>(dead) & 3) == 0;
  const dim3 grid4(oc_div_up(d, 4 * tb), out);
  if (oc_split_engine_on() && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0) {
    float* delta = nullptr;
    const bool vec_w = d % 4 == 0 && ldw_io % 4 == 0 && (reinterpret_cast<uintptr_t>(W) & 7) == 0 &&
                       (reinterpret_cast<uintptr_t>(dead) & 3) == 0;
    const int rc = split_products(W, ldw_io, out, d, C, ldc, U, ldu, perm, dead, bf16, vec_w, (char*)workspace, delta, stream);
    if (rc) return rc;
    const bool vec_st = vec_w && !perm;
    OC_LAUNCH(qep_store_kernel, vec_st ? grid4 : grid, tb, 0, stream, dead, delta, QepWs(out, d).ld, out, d, perm, perccorr, W,
              ldw_io, bf16, vec_st);
    return OC_OK;
  }
  qep_load_kernel<<<vec ? grid4 : grid, tb, 0, stream>>>(W, ldw_io, out, d, dead, Wf, ld, bf16, vec);
  OC_CHECK_LAUNCH();
  OcGemm g{};
  // A = Wf * C
  g.A = Wf; g.lda = ld; g.B = C; g.ldb = ldc; g.C = A; g.ldc = ld;
  g.M = out; g.N = d; g.K = d; g.alpha = 1.f; g.beta = 0.f; g.batch = 1;
  int rc = oc_gemm_f32_launch(g, stream);
  if (rc) return rc;
  if (perm) {   // B = A P^T
    gather_cols_kernel<<<grid, tb, 0, stream>>>(A, ld, out, d, perm, B, ld);
    OC_CHECK_LAUNCH();
    float* t = A; A = B; B = t;
  }
  // B = A * U^T      (U upper: U[n][k] = 0 for k < n)
  OcGemm t1{};
  t1.A = A; t1.lda = ld; t1.B = U; t1.ldb = ldu; t1.transB = 1; t1.C = B; t1.ldc = ld;
  t1.M = out; t1.N = d; t1.K = d; t1.alpha = 1.f; t1.beta = 0.f; t1.flags = OC_GEMM_KLO_FROM_N; t1.batch = 1;
  rc = oc_gemm_f32_launch(t1, stream);
  if (rc) return rc;
  // A = B * U        (U[k][n] = 0 for k > n)
  OcGemm t2{};
  t2.A = B; t2.lda = ld; t2.B = U; t2.ldb = ldu; t2.C = A; t2.ldc = ld;
  t2.M = out; t2.N = d; t2.K = d; t2.alpha = 1.f; t2.beta = 0.f; t2.flags = OC_GEMM_KHI_FROM_N; t2.batch = 1;
  rc = oc_gemm_f32_launch(t2, stream);
  if (rc) return rc;
  const bool vec_st = vec && !perm;
  qep_store_kernel<<<vec_st ? grid4 : grid, tb, 0, stream>>>(dead, A, ld, out, d, perm, perccorr, W, ldw_io, bf16, vec_st);
  OC_CHECK_LAUNCH();
  return OC_OK;
}
