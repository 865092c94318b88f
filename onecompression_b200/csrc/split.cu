// fp32 -> two scaled fp16 planes (see split.cuh).
#include "split.cuh"

namespace {

// One CTA per 128 x 128 block: 64 entries a thread in registers, the block's maximum through a shuffle and
// shared memory, then both planes.  Bound by HBM (4 bytes in, 4 out per entry).
constexpr int ST = 256;

template <bool VEC, bool PER_ROW>
__global__ void __launch_bounds__(ST) split_kernel(OcSplitArgs a) {
  oc_wait_before();
  const int rb = blockIdx.y, cb = blockIdx.x;
  if (a.region == OC_SPLIT_UPPER && cb < (rb & ~1)) return;
  if (a.region == OC_SPLIT_LOWER && cb > (rb | 1)) return;
  {
    const long long z1 = blockIdx.z % a.nb1, z2 = blockIdx.z / a.nb1;
    a.src += z1 * a.src1 + z2 * a.src2;
    a.planes += z1 * a.dst1 + z2 * a.dst2;
    a.table += z1 * a.tab1 + z2 * a.tab2;
  }
  __shared__ float red[ST / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = cb * 128 + lane * 4;
  float4 v[16];
  float mx[PER_ROW ? 16 : 1];
#pragma unroll
  for (int i = 0; i < (PER_ROW ? 16 : 1); ++i) mx[i] = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = rb * 128 + i * 8 + warp;
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < a.rows && c < a.cols) {
      const float* p = a.src + (long long)r * a.ld;
      if (VEC) {
        const float4 t = *reinterpret_cast<const float4*>(p + c);
        e[0] = t.x; e[1] = t.y; e[2] = t.z; e[3] = t.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (c + j < a.cols) e[j] = p[a.perm ? a.perm[c + j] : c + j];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if ((a.region == OC_SPLIT_UPPER && c + j < r) || (a.region == OC_SPLIT_LOWER && c + j > r)) e[j] = 0.f;
      mx[PER_ROW ? i : 0] = fmaxf(mx[PER_ROW ? i : 0], oc_finite_abs(e[j]));
    }
    v[i] = make_float4(e[0], e[1], e[2], e[3]);
  }
  // (a warp holds whole rows)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < (PER_ROW ? 16 : 1); ++i) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
  oc_let_next();
  float inv, s = 1.f;
  if (!PER_ROW) {
    if (lane == 0) red[warp] = mx[0];
    __syncthreads();
    float m = 0.f;
#pragma unroll
    for (int w = 0; w < ST / 32; ++w) m = fmaxf(m, red[w]);
    s = oc_split_scale(m, inv);
    if (tid == 0) a.table[rb * a.ldt + cb] = inv;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = rb * 128 + i * 8 + warp;
    if (r >= a.rows) break;
    if (PER_ROW) {
      s = oc_split_scale(mx[PER_ROW ? i : 0], inv);
      if (lane == 0) a.table[cb * a.ldt + r] = inv;
    }
    if (c >= a.cols) continue;
    uint2 hi, lo;
    oc_split4(make_float4(v[i].x * s, v[i].y * s, v[i].z * s, v[i].w * s), hi, lo);
    // (rows of the planes are padded to whole groups of eight columns)
    __half* d = a.planes + (long long)r * a.ldp + c;
    *reinterpret_cast<uint2*>(d) = hi;
    *reinterpret_cast<uint2*>(d + a.plane) = lo;
  }
}

}  // namespace

int oc_split_launch(const OcSplitArgs& a, cudaStream_t stream) {
  if (a.rows <= 0 || a.cols <= 0 || a.nb1 <= 0 || a.nb2 <= 0) return OC_OK;
  const dim3 grid(oc_div_up(a.cols, 128), oc_div_up(a.rows, 128), a.nb1 * a.nb2);
  OC_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "split: too many blocks");
  OC_REQUIRE(a.ldp % 8 == 0 && a.ldp >= a.cols, "split: bad row pitch");
  const bool vec = !a.perm && a.cols % 4 == 0 && a.ld % 4 == 0 && a.src1 % 4 == 0 && a.src2 % 4 == 0 &&
                   (reinterpret_cast<uintptr_t>(a.src) & 15) == 0;
  if (a.per_row) {
    OC_LAUNCH((vec ? split_kernel<true, true> : split_kernel<false, true>), grid, ST, 0, stream, a);
  } else {
    OC_LAUNCH((vec ? split_kernel<true, false> : split_kernel<false, false>), grid, ST, 0, stream, a);
  }
  return OC_OK;
}
