// y = x W^T (+ bias) for a few tokens, W in the packed AutoGPTQ layout, decoded inside the product.
//
// The packed weight is read once (bits / 8 bytes per weight) and nothing else of that size moves;
// decoding into an fp16 matrix first writes and reads 4 more bytes per weight.
// The weights are the values of oc_dequantize_packed, bit for bit: scale * (q - z) is exact in fp32
// (11 + 9 significant bits), so the fp16 product of the fp16 scale with the exact fp16 integer q - z is
// its rounding.  Products and sums are fp32 (mma.sync m16n8k16; at these token counts the tensor
// pipe is idle, and an operand in registers saves the way through shared memory that tcgen05 needs).
//
// A warp takes 32 rows of W and a share of the columns, 32 at a time.  Lane (g, q) = (lane / 4,
// lane % 4) reads the packed words of rows 4g .. 4g+3 (one 16-byte load per word row) for columns
// 8q .. 8q+7.  The order of k inside an MMA is free as long as both operands agree: the lane's pairs
// (k, k+4) of columns are what fills its slots in the A fragment, and the matching pairs of x come out
// of one 16-byte load per token.  Rows are dealt to the two m16 tiles the same way.  The warps
// of a CTA share the rows and split the columns; their sums meet in shared memory in a fixed order.
//
// Measured, 14336 x 4096, 4 bits, cold L2: 4 tokens 20 us, 16 tokens 29.5 us, against 77 us for decoding
// and a library product (56 + 20); act-order 53 against 129 us.  4096 x 4096: 9 against 36 us.  At 16 tokens
// it still takes less than half of the other way; more tokens are left to decoding once and a GEMM on
// the tensor cores.
//
// What bounds it at 4 tokens is latency: HBM delivers 1.3 TB/s (its floor is 5 us), and the 9.3 M warp instructions
// are issued in 49 % of the cycles that an SM is active (74 % of the kernel's).  A CTA stages all group
// parameters and the groups of all columns before its first product, and a warp has eleven iterations behind a
// ring of two; the leading stalls are loads on their way (1.9 cycles per instruction) and the barrier
// behind the staging (0.8).
#include "packed_field.cuh"

namespace {

constexpr int ROWS = 32;      // rows of W per CTA

__device__ __forceinline__ void mma_f16(float (&c)[4], const __half2 (&a)[4], unsigned b0, unsigned b1) {
  const unsigned* ar = reinterpret_cast<const unsigned*>(a);
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(ar[0]), "r"(ar[1]), "r"(ar[2]), "r"(ar[3]), "r"(b0), "r"(b1));
}

// stored zero points of rows r .. r + 3 (r a multiple of 4) of group row `zrow`
template <int BITS>
__device__ __forceinline__ void load_zeros(const int* __restrict__ zrow, int r, unsigned (&z)[4]) {
  constexpr unsigned MASK = (1u << BITS) - 1u;
  unsigned v;
  if (BITS == 3) {
    const int bit = 3 * (r & 31), wi = (r >> 5) * 3 + (bit >> 5);
    const unsigned lo = (unsigned)zrow[wi], hi = (bit & 31) > 20 ? (unsigned)zrow[wi + 1] : 0u;
    v = __funnelshift_r(lo, hi, bit & 31);
  } else {
    constexpr int F = 32 / BITS;
    v = (unsigned)zrow[r / F] >> ((r % F) * BITS);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) z[i] = (((v >> (BITS * i)) & MASK) + 1u) & MASK;
}

struct LinearArgs {
  const int* qweight; const int* qzeros; const __half* scales; const int* g_idx;
  const __half* x; const __half* bias; __half* y;
  int out, d, tokens, groups;
  int staged;                // groups whose parameters lie in shared memory: all of them and one of zeros, or none
  long long ldz;
};

__device__ __forceinline__ void copy16(void* dst, const void* src, bool valid) {   // zeros where not valid
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// one warp's slot of the ring: packed words and x of one iteration (two times 32 columns)
template <int WORDS, int NT> struct __align__(16) Slot { int4 w[2][WORDS][32]; uint4 x[2][NT][32]; };

constexpr int PAR_BYTES = ROWS * 3;   // per group: 32 fp16 scales and 32 zero points of one byte
constexpr int STAGED_GROUPS = 427;    // most groups whose parameters are staged, the one of zeros included
constexpr int STAGED_BYTES = STAGED_GROUPS * PAR_BYTES;
constexpr int MAX_UNITS = 8192;       // most eight-column units (two bytes each); wider layers are refused

// NT * 8 tokens, WARPS column shares per CTA, DEPTH iterations of a warp in flight
template <int BITS, int NT, int WARPS, int DEPTH, int CTAS>
__global__ void __launch_bounds__(WARPS * 32, CTAS) packed_linear_kernel(const LinearArgs a) {
  using F = Field<BITS>;
  using S = Slot<F::WORDS, NT>;
  extern __shared__ __align__(16) unsigned char smem[];
  __half* par_s = reinterpret_cast<__half*>(smem + sizeof(S) * DEPTH * WARPS);
  unsigned char* par_z = reinterpret_cast<unsigned char*>(par_s + a.staged * ROWS);
  // group of every unit, 0xffff where its columns belong to several
  unsigned short* ugroup = reinterpret_cast<unsigned short*>(par_z + a.staged * ROWS);
  float (*part)[ROWS][NT * 8 + 1] = reinterpret_cast<float (*)[ROWS][NT * 8 + 1]>(smem);   // after the loop
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int r = blockIdx.x * ROWS + 4 * g;           // this lane's four rows
  const bool rows_ok = r < a.out;                    // out is a multiple of 4
  const int units = a.d >> 3;
  // every warp takes a contiguous share of the columns, so that a group's parameters serve several
  // iterations of one warp
  const int total = (units + 7) >> 3, per = (total + WARPS - 1) / WARPS;
  const int it0 = min(total, warp * per), n_it = min(total, it0 + per) - it0;
  S* ring = reinterpret_cast<S*>(smem) + warp * DEPTH;

  // this lane's unit of the next iteration to fetch (and, 4 further, of its second half)
  int funit = it0 * 8 + q;
  const int* wp = a.qweight + (long long)F::first(funit) * a.out + (rows_ok ? r : 0);
  const __half* xp = a.x + 8 * funit + (long long)(g < a.tokens ? g : 0) * a.d;
  const long long w_half = (long long)BITS * a.out;      // 32 columns are BITS word rows
  auto fetch = [&](bool more, S& f) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool in = more && funit + 4 * h < units;
#pragma unroll
      for (int j = 0; j < F::WORDS; ++j) {
        // (the last unit of 32 three-bit columns lies in one word)
        const bool ok = in && rows_ok && (BITS != 3 || j == 0 || q != 3);
        copy16(&f.w[h][j][lane], ok ? wp + h * w_half + (long long)j * a.out : a.qweight, ok);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const bool ok = in && n * 8 + g < a.tokens;
        copy16(&f.x[h][n][lane], ok ? xp + 32 * h + (long long)n * 8 * a.d : a.x, ok);
      }
    }
    copy_commit();
    funit += 8;
    wp += 2 * w_half;
    xp += 64;
  };
#pragma unroll
  for (int s = 0; s < DEPTH; ++s) fetch(s < n_it, ring[s]);

  // parameters of all groups for this CTA's rows, and the groups of the units
  for (int e = tid; e < a.staged * (ROWS / 4); e += WARPS * 32) {
    const int gi = e / (ROWS / 4), r4 = e % (ROWS / 4) * 4, rr = blockIdx.x * ROWS + r4;
    unsigned z[4] = {0u, 0u, 0u, 0u};
    uint2 sv = make_uint2(0u, 0u);
    if (rr < a.out && gi < a.groups) {
      sv = *reinterpret_cast<const uint2*>(a.scales + (long long)gi * a.out + rr);
      load_zeros<BITS>(a.qzeros + gi * a.ldz, rr, z);
    }
    *reinterpret_cast<uint2*>(par_s + gi * ROWS + r4) = sv;
    *reinterpret_cast<unsigned*>(par_z + gi * ROWS + r4) = z[0] | (z[1] << 8) | (z[2] << 16) | (z[3] << 24);
  }
  for (int u = tid; u < units; u += WARPS * 32) {
    int first = 0;
    bool uniform = true;
    if (a.g_idx) {
      const int4 ga = *reinterpret_cast<const int4*>(a.g_idx + 8 * u), gb = *reinterpret_cast<const int4*>(a.g_idx + 8 * u + 4);
      first = ga.x;
      uniform = ga.y == first && ga.z == first && ga.w == first && gb.x == first && gb.y == first &&
                gb.z == first && gb.w == first;
    }
    ugroup[u] = uniform ? (unsigned short)first : (unsigned short)0xffff;
  }
  __syncthreads();

  float acc[2][NT][4];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[t][n][i] = 0.f;

  int group = -1;
  __half2 s2[4], z2[4];
  auto load_group = [&](int gi) {
    unsigned z[4] = {0u, 0u, 0u, 0u};
    uint2 sv = make_uint2(0u, 0u);
    if (a.staged) {
      sv = *reinterpret_cast<const uint2*>(par_s + gi * ROWS + 4 * g);
      const unsigned zb = *reinterpret_cast<const unsigned*>(par_z + gi * ROWS + 4 * g);
#pragma unroll
      for (int i = 0; i < 4; ++i) z[i] = (zb >> (8 * i)) & 0xffu;
    } else if (rows_ok && gi < a.groups) {
      sv = *reinterpret_cast<const uint2*>(a.scales + (long long)gi * a.out + r);
      load_zeros<BITS>(a.qzeros + gi * a.ldz, r, z);
    }
    s2[0] = as_half2(__byte_perm(sv.x, 0u, 0x1010)); s2[1] = as_half2(__byte_perm(sv.x, 0u, 0x3232));
    s2[2] = as_half2(__byte_perm(sv.y, 0u, 0x1010)); s2[3] = as_half2(__byte_perm(sv.y, 0u, 0x3232));
#pragma unroll
    for (int i = 0; i < 4; ++i) z2[i] = as_half2((z[i] | (z[i] << 16)) | 0x64006400u);   // 1024 + z
  };

  S* cur = ring;
  int unit0 = it0 * 8 + q;
  for (int it = 0; it < n_it; ++it, unit0 += 8) {
    copy_wait<DEPTH - 1>();                // (every lane reads what it copied itself)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int unit = unit0 + 4 * h;
      const int4 w0 = cur->w[h][0][lane], w1 = F::WORDS > 1 ? cur->w[h][F::WORDS - 1][lane] : make_int4(0, 0, 0, 0);
      // Columns behind the last one belong to a group of their own with a scale of zero: a group of the
      // layer could make their weights infinite (scale * zero point beyond fp16), and 0 * inf a NaN.
      const int ug = unit < units ? (int)ugroup[unit] : a.groups;
      const unsigned wr[4][2] = {{(unsigned)w0.x, (unsigned)w1.x}, {(unsigned)w0.y, (unsigned)w1.y},
                                 {(unsigned)w0.z, (unsigned)w1.z}, {(unsigned)w0.w, (unsigned)w1.w}};
      __half2 v[4][4];    // [row][pair]: weights of columns (k, k + 4) of the unit
      if (ug != 0xffff) {
        if (ug != group) { group = ug; load_group(ug); }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            v[i][k] = __hmul2(s2[i], __hsub2(as_half2(F::pair(wr[i], unit, k) | 0x64006400u), z2[i]));
      } else {
        // act-order: the columns of a unit belong to different groups
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          __half2 sa[4], za[4];
          load_group(a.g_idx[8 * unit + k]);
#pragma unroll
          for (int i = 0; i < 4; ++i) { sa[i] = s2[i]; za[i] = z2[i]; }
          load_group(a.g_idx[8 * unit + k + 4]);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            v[i][k] = __hmul2(__lows2half2(sa[i], s2[i]),
                              __hsub2(as_half2(F::pair(wr[i], unit, k) | 0x64006400u), __lows2half2(za[i], z2[i])));
        }
        group = -1;
      }
      __syncwarp();
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const uint4 xv = cur->x[h][n][lane];
        const unsigned b[4] = {__byte_perm(xv.x, xv.z, 0x5410), __byte_perm(xv.x, xv.z, 0x7632),
                               __byte_perm(xv.y, xv.w, 0x5410), __byte_perm(xv.y, xv.w, 0x7632)};
#pragma unroll
        for (int t = 0; t < 2; ++t) {   // rows 4g + 2t (slot g) and 4g + 2t + 1 (slot g + 8)
          const __half2 a0[4] = {v[2 * t][0], v[2 * t + 1][0], v[2 * t][1], v[2 * t + 1][1]};
          const __half2 a1[4] = {v[2 * t][2], v[2 * t + 1][2], v[2 * t][3], v[2 * t + 1][3]};
          mma_f16(acc[t][n], a0, b[0], b[1]);
          mma_f16(acc[t][n], a1, b[2], b[3]);
        }
      }
    }
    fetch(it + DEPTH < n_it, *cur);
    cur = (cur == ring + DEPTH - 1) ? ring : cur + 1;
  }
  copy_wait<0>();
  __syncthreads();                         // the ring's memory now holds the partial sums
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) part[warp][4 * g + 2 * t + (i >> 1)][n * 8 + 2 * q + (i & 1)] = acc[t][n][i];
  __syncthreads();
  for (int e = tid; e < ROWS * NT * 8; e += WARPS * 32) {
    const int row = e % ROWS, t = e / ROWS, rr = blockIdx.x * ROWS + row;
    if (t >= a.tokens || rr >= a.out) continue;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += part[w][row][t];
    if (a.bias) s += __half2float(a.bias[rr]);
    a.y[(long long)t * a.out + rr] = __float2half_rn(s);
  }
}

template <int BITS, int NT, int WARPS, int DEPTH, int CTAS>
int launch(const LinearArgs& a, int grid, cudaStream_t stream) {
  constexpr int ring = (int)sizeof(Slot<Field<BITS>::WORDS, NT>) * DEPTH * WARPS;
  static_assert(ring >= WARPS * ROWS * (NT * 8 + 1) * 4, "the partial sums reuse the ring");
  static_assert(ring + STAGED_BYTES + 2 * MAX_UNITS <= 227 * 1024, "shared memory of one CTA");
  OC_OPT_IN_SMEM((packed_linear_kernel<BITS, NT, WARPS, DEPTH, CTAS>), ring + STAGED_BYTES + 2 * MAX_UNITS);
  packed_linear_kernel<BITS, NT, WARPS, DEPTH, CTAS>
      <<<grid, WARPS * 32, ring + a.staged * PAR_BYTES + a.d / 8 * 2, stream>>>(a);
  OC_CHECK_LAUNCH();
  return OC_OK;
}

template <int BITS>
int launch_bits(const LinearArgs& a, int sm_count, cudaStream_t stream) {
  const int grid = oc_div_up(a.out, ROWS);
  // With at most one CTA per SM the columns are split over 16 warps, with more over 6, so that several CTAs
  // share an SM: four for up to 8 tokens (one wave up to 18944 rows; 14336 rows are 448 CTAs, just over
  // three per SM), two for more tokens, whose sums take the registers (14336 rows are one and a half waves).
  const bool few = grid <= sm_count;
  if (a.tokens <= 8)
    return few ? launch<BITS, 1, 16, 2, 1>(a, grid, stream) : launch<BITS, 1, 6, 2, 4>(a, grid, stream);
  return few ? launch<BITS, 2, 16, 2, 1>(a, grid, stream) : launch<BITS, 2, 6, 2, 2>(a, grid, stream);
}

}  // namespace

// See include/onecomp_b200.h for the contract.
extern "C" int oc_packed_linear(const int* qweight, const int* qzeros, const void* scales16, const int* g_idx,
                                int out, int d, int groups, int bits, const void* x16, int tokens, const void* bias16,
                                void* y16, int sm_count, void* stream) {
  OC_REQUIRE(qweight && qzeros && scales16 && x16 && y16 && out > 0 && d > 0, "packed_linear: bad arguments");
  OC_REQUIRE(tokens >= 1 && tokens <= 16, "packed_linear: 1..16 tokens");
  OC_REQUIRE(bits == 2 || bits == 3 || bits == 4 || bits == 8, "packed_linear: wbits must be one of 2, 3, 4, 8");
  const int f = (bits == 3) ? 32 : 32 / bits;
  OC_REQUIRE(d % f == 0 && out % f == 0 && d % 8 == 0, "packed_linear: shape not divisible by the pack factor or 8");
  OC_REQUIRE(((reinterpret_cast<uintptr_t>(qweight) | reinterpret_cast<uintptr_t>(x16) |
               reinterpret_cast<uintptr_t>(g_idx)) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(scales16) & 7) == 0 && (reinterpret_cast<uintptr_t>(qzeros) & 3) == 0,
             "packed_linear: operands must be 16-byte aligned (scales 8-byte)");
  OC_REQUIRE(d / 8 <= MAX_UNITS && groups < 0xffff, "packed_linear: too many columns or groups");
  OC_REQUIRE(groups >= 1 && (groups == 1 || g_idx), "packed_linear: several groups need g_idx");
  LinearArgs a{qweight, qzeros, (const __half*)scales16, g_idx, (const __half*)x16, (const __half*)bias16,
               (__half*)y16, out, d, tokens, groups, groups < STAGED_GROUPS ? groups + 1 : 0,
               (bits == 3) ? out / 32 * 3 : out / f};
  if (sm_count <= 0) sm_count = 148;
  cudaStream_t s = (cudaStream_t)stream;
  switch (bits) {
    case 2: return launch_bits<2>(a, sm_count, s);
    case 3: return launch_bits<3>(a, sm_count, s);
    case 4: return launch_bits<4>(a, sm_count, s);
    default: return launch_bits<8>(a, sm_count, s);
  }
}
