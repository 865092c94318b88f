// Stand-alone packing, unpacking and dequantisation of the AutoGPTQ int32 layout
// (reference: onecomp/quantizer/gptq/gptq_layer.py:36-170 and
// GPTQResult.compute_dequantized_weight, onecomp/quantizer/gptq/_gptq.py:84-168).
// The column loop packs its own results; these entry points serve the callers
// that hold integer codes or a packed result already.
#include "packed_field.cuh"

namespace {

__device__ __forceinline__ void pack3(const unsigned (&v)[32], unsigned (&w)[3]) {
  w[0] = w[1] = w[2] = 0u;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const int bit = 3 * k, wi = bit >> 5, off = bit & 31;
    w[wi] |= v[k] << off;
    if (off + 3 > 32) w[wi + 1] |= v[k] >> (32 - off);
  }
}

__device__ __forceinline__ unsigned unpack3(const unsigned (&w)[3], int k) {
  const int bit = 3 * k, wi = bit >> 5, off = bit & 31;
  unsigned v = w[wi] >> off;
  if (off + 3 > 32) v |= w[wi + 1] << (32 - off);
  return v & 7u;
}

// Pack along the strided axis: word (p, c) gathers in[(p*f + k) * stride_k + c * stride_c].
// qweight: in = codes [out][d], k walks d (stride 1), c walks out (stride d)  -> [d*bits/32][out]
// qzeros : in = zeros [G][out], handled per group with k walking out          -> [G][out*bits/32]
__global__ void pack_axis_kernel(const int* __restrict__ in, long long stride_k, long long stride_c,
                                 int nk, int nc, int bits, int add, int* __restrict__ out,
                                 long long out_stride_p, long long out_stride_c) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const unsigned mask = (1u << bits) - 1u;
  const int* src = in + (long long)c * stride_c;
  if (bits == 3) {
    const long long k0 = (long long)blockIdx.y * 32;
    unsigned v[32], w[3];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = (unsigned)(src[(k0 + k) * stride_k] + add) & mask;
    pack3(v, w);
#pragma unroll
    for (int t = 0; t < 3; ++t) out[(long long)(blockIdx.y * 3 + t) * out_stride_p + (long long)c * out_stride_c] = (int)w[t];
  } else {
    const int f = 32 / bits;
    const long long k0 = (long long)blockIdx.y * f;
    unsigned word = 0u;
    for (int k = 0; k < f; ++k) word |= ((unsigned)(src[(k0 + k) * stride_k] + add) & mask) << (k * bits);
    out[(long long)blockIdx.y * out_stride_p + (long long)c * out_stride_c] = (int)word;
  }
}

__global__ void unpack_axis_kernel(const int* __restrict__ in, long long in_stride_p, long long in_stride_c,
                                   int nk, int nc, int bits, int add, int* __restrict__ out,
                                   long long stride_k, long long stride_c) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const unsigned mask = (1u << bits) - 1u;
  int* dst = out + (long long)c * stride_c;
  if (bits == 3) {
    const long long k0 = (long long)blockIdx.y * 32;
    unsigned w[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) w[t] = (unsigned)in[(long long)(blockIdx.y * 3 + t) * in_stride_p + (long long)c * in_stride_c];
#pragma unroll
    for (int k = 0; k < 32; ++k)
      if (k0 + k < nk) dst[(k0 + k) * stride_k] = (int)((unpack3(w, k) + (unsigned)add) & mask);
  } else {
    const int f = 32 / bits;
    const long long k0 = (long long)blockIdx.y * f;
    const unsigned word = (unsigned)in[(long long)blockIdx.y * in_stride_p + (long long)c * in_stride_c];
    for (int k = 0; k < f; ++k)
      if (k0 + k < nk) dst[(k0 + k) * stride_k] = (int)((((word >> (k * bits)) & mask) + (unsigned)add) & mask);
  }
}

// W^[r][c] = fp16( float(scale16[g][r]) * (q - zero) ), g = g_idx[c]; zero = (stored + 1) & mask
//
// Bound by HBM: bits / 8 bytes in and two out per weight.  A CTA makes 64 rows x 128 columns: a thread
// decodes 32 columns of one row (neighbouring lanes hold neighbouring rows, so the packed words,
// scales and zero points load coalesced; each word is read once, and scale and zero only where the
// group changes from one column to the next), and the tile leaves through shared memory in
// 256-byte row segments.  Eight columns of one group are decoded as pairs of fp16 (as in packed_linear.cu: q | 0x6400 is
// 1024 + q, the subtraction is exact and the product rounds once, the same values): in fp32, one weight
// after the other, issue slots bound it.  14336 x 4096, 4 bits: 54 -> 37 us
// of kernel time, cold L2; 4096 x 14336, 3 bits: 54 -> 37 us (act-order, column by column: 106 -> 107 us).
constexpr int DQ_ROWS = 64, DQ_COLS = 128, DQ_PITCH = DQ_COLS + 8;   // pitch: 16-byte accesses without conflicts
template <int BITS>
__global__ void __launch_bounds__(256) dequant_packed_kernel(const int* __restrict__ qweight,
                                                             const int* __restrict__ qzeros,
                                                             const __half* __restrict__ scales,
                                                             const int* __restrict__ g_idx, int out, int d,
                                                             long long ldz, __half* __restrict__ w, long long ldw) {
  constexpr unsigned MASK = (1u << BITS) - 1u;
  __shared__ __align__(16) __half tile[DQ_ROWS * DQ_PITCH];
  const int tid = threadIdx.x, lr = tid % DQ_ROWS, lc = tid / DQ_ROWS * 32;
  const int r = blockIdx.y * DQ_ROWS + lr, c0 = blockIdx.x * DQ_COLS + lc;
  if (r < out && c0 < d) {
    unsigned v[BITS];
    const long long w0 = (long long)c0 / 32 * BITS;
    const int words = min(BITS, (int)((long long)(d - c0) * BITS / 32));   // d is a multiple of the pack factor
#pragma unroll
    for (int j = 0; j < BITS; ++j) v[j] = j < words ? (unsigned)qweight[(w0 + j) * out + r] : 0u;
    int group = -1;
    float s = 0.f, z = 0.f;
    auto load_group = [&](int g) {
      if (g == group) return;
      group = g;
      s = __half2float(scales[(long long)g * out + r]);
      unsigned zq;
      if (BITS == 3) {
        const int zb = 3 * (r & 31), zw = zb >> 5, zo = zb & 31;
        const int* zr = qzeros + (long long)g * ldz + (r / 32) * 3;
        zq = (unsigned)zr[zw] >> zo;
        if (zo + 3 > 32) zq |= (unsigned)zr[zw + 1] << (32 - zo);
      } else {
        constexpr int F = 32 / (BITS == 3 ? 4 : BITS);
        zq = (unsigned)qzeros[(long long)g * ldz + r / F] >> ((r % F) * BITS);
      }
      z = (float)(((zq & MASK) + 1u) & MASK);
    };
    const bool wide_idx = (reinterpret_cast<uintptr_t>(g_idx) & 15) == 0;
#pragma unroll
    for (int k8 = 0; k8 < 4; ++k8) {
      __align__(16) __half h[8];
      const int cu = c0 + k8 * 8;
      int gi[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      bool uniform = cu + 8 <= d;
      if (g_idx) {
        if (uniform && wide_idx) {
          const int4 ga = *reinterpret_cast<const int4*>(g_idx + cu), gb = *reinterpret_cast<const int4*>(g_idx + cu + 4);
          gi[0] = ga.x; gi[1] = ga.y; gi[2] = ga.z; gi[3] = ga.w; gi[4] = gb.x; gi[5] = gb.y; gi[6] = gb.z; gi[7] = gb.w;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) gi[i] = cu + i < d ? g_idx[cu + i] : 0;
        }
#pragma unroll
        for (int i = 1; i < 8; ++i) uniform = uniform && gi[i] == gi[0];
      }
      if (uniform) {
        load_group(gi[0]);
        const int first = Field<BITS>::first(k8);
        const unsigned w2[2] = {v[first], Field<BITS>::WORDS > 1 ? v[first + 1 < BITS ? first + 1 : first] : 0u};
        const __half2 s2 = __float2half2_rn(s), z2 = __float2half2_rn(1024.f + z);
        unsigned p[4];                                 // columns (k, k + 4)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const __half2 x = __hmul2(s2, __hsub2(as_half2(Field<BITS>::pair(w2, k8, k) | 0x64006400u), z2));
          p[k] = *reinterpret_cast<const unsigned*>(&x);
        }
        *reinterpret_cast<uint4*>(h) = make_uint4(__byte_perm(p[0], p[1], 0x5410), __byte_perm(p[2], p[3], 0x5410),
                                                  __byte_perm(p[0], p[1], 0x7632), __byte_perm(p[2], p[3], 0x7632));
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int k = k8 * 8 + i, c = c0 + k, bit = k * BITS, wi = bit >> 5, off = bit & 31;
          if (c < d) {
            load_group(gi[i]);
            unsigned q = v[wi] >> off;
            if (off + BITS > 32) q |= v[wi + 1 < BITS ? wi + 1 : wi] << (32 - off);
            h[i] = __float2half_rn(s * ((float)(q & MASK) - z));
          } else {
            h[i] = __ushort_as_half(0);
          }
        }
      }
      *reinterpret_cast<uint4*>(tile + lr * DQ_PITCH + lc + k8 * 8) = *reinterpret_cast<const uint4*>(h);
    }
  }
  __syncthreads();
  const bool vec = (ldw % 8 == 0) && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
#pragma unroll
  for (int it = 0; it < DQ_ROWS * DQ_COLS / 8 / 256; ++it) {
    const int e = it * 256 + tid, row = e / (DQ_COLS / 8), c8 = e % (DQ_COLS / 8) * 8;
    const int rr = blockIdx.y * DQ_ROWS + row, c = blockIdx.x * DQ_COLS + c8;
    if (rr >= out || c >= d) continue;
    const __half* src = tile + row * DQ_PITCH + c8;
    __half* dst = w + (long long)rr * ldw + c;
    if (vec && c + 8 <= d) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
    else
      for (int i = 0; i < 8 && c + i < d; ++i) dst[i] = src[i];
  }
}

int check_bits(int bits) {
  if (bits == 2 || bits == 3 || bits == 4 || bits == 8) return OC_OK;
  oc_set_last_error("pack: wbits must be one of 2, 3, 4, 8");
  return OC_ERR_UNSUPPORTED;
}

}  // namespace

extern "C" int oc_pack_qweight(const int* codes, int out, int d, int bits, int* qweight, void* stream) {
  if (int rc = check_bits(bits)) return rc;
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(codes && qweight && out > 0 && d > 0, "pack_qweight: bad arguments");
  OC_REQUIRE(d % f == 0, "pack_qweight: in_features not divisible by the pack factor");
  pack_axis_kernel<<<dim3(oc_div_up(out, 128), d / f), 128, 0, (cudaStream_t)stream>>>(
      codes, 1, d, d, out, bits, 0, qweight, out, 1);
  OC_CHECK_LAUNCH();
  return OC_OK;
}

extern "C" int oc_unpack_qweight(const int* qweight, int out, int d, int bits, int* codes, void* stream) {
  if (int rc = check_bits(bits)) return rc;
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(codes && qweight && out > 0 && d > 0, "unpack_qweight: bad arguments");
  unpack_axis_kernel<<<dim3(oc_div_up(out, 128), oc_div_up(d, f)), 128, 0, (cudaStream_t)stream>>>(
      qweight, out, 1, d, out, bits, 0, codes, 1, d);
  OC_CHECK_LAUNCH();
  return OC_OK;
}

// zeros [G][out] raw zero points; stored value is (zero + add) & mask with add = -1 for the
// v1 checkpoint convention (pass add = 0 for values that carry the offset already).
extern "C" int oc_pack_qzeros(const int* zeros, int G, int out, int bits, int add, int* qzeros, void* stream) {
  if (int rc = check_bits(bits)) return rc;
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(zeros && qzeros && G > 0 && out > 0, "pack_qzeros: bad arguments");
  OC_REQUIRE(out % f == 0, "pack_qzeros: out_features not divisible by the pack factor");
  const long long ldz = (bits == 3) ? out / 32 * 3 : out / f;
  pack_axis_kernel<<<dim3(oc_div_up(G, 128), out / f), 128, 0, (cudaStream_t)stream>>>(
      zeros, 1, out, out, G, bits, add, qzeros, 1, ldz);
  OC_CHECK_LAUNCH();
  return OC_OK;
}

extern "C" int oc_unpack_qzeros(const int* qzeros, int G, int out, int bits, int add, int* zeros, void* stream) {
  if (int rc = check_bits(bits)) return rc;
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(zeros && qzeros && G > 0 && out > 0, "unpack_qzeros: bad arguments");
  const long long ldz = (bits == 3) ? (long long)oc_div_up(out, 32) * 3 : oc_div_up(out, f);
  unpack_axis_kernel<<<dim3(oc_div_up(G, 128), oc_div_up(out, f)), 128, 0, (cudaStream_t)stream>>>(
      qzeros, 1, ldz, out, G, bits, add, zeros, 1, out);
  OC_CHECK_LAUNCH();
  return OC_OK;
}

extern "C" int oc_dequantize_packed(const int* qweight, const int* qzeros, const void* scales16,
                                    const int* g_idx, int out, int d, int bits, void* w16,
                                    long long ldw, void* stream) {
  if (int rc = check_bits(bits)) return rc;
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(qweight && qzeros && scales16 && w16 && out > 0 && d > 0 && ldw >= d, "dequantize_packed: bad arguments");
  OC_REQUIRE(d % f == 0 && out % f == 0, "dequantize_packed: shape not divisible by the pack factor");
  const long long ldz = (bits == 3) ? out / 32 * 3 : out / f;
  OC_REQUIRE(oc_div_up(out, DQ_ROWS) <= 65535, "dequantize_packed: too many rows");
  const dim3 grid(oc_div_up(d, DQ_COLS), oc_div_up(out, DQ_ROWS));
  cudaStream_t s = (cudaStream_t)stream;
  const __half* sc = (const __half*)scales16;
  __half* w = (__half*)w16;
  switch (bits) {
    case 2: dequant_packed_kernel<2><<<grid, 256, 0, s>>>(qweight, qzeros, sc, g_idx, out, d, ldz, w, ldw); break;
    case 3: dequant_packed_kernel<3><<<grid, 256, 0, s>>>(qweight, qzeros, sc, g_idx, out, d, ldz, w, ldw); break;
    case 4: dequant_packed_kernel<4><<<grid, 256, 0, s>>>(qweight, qzeros, sc, g_idx, out, d, ldz, w, ldw); break;
    default: dequant_packed_kernel<8><<<grid, 256, 0, s>>>(qweight, qzeros, sc, g_idx, out, d, ldz, w, ldw);
  }
  OC_CHECK_LAUNCH();
  return OC_OK;
}
