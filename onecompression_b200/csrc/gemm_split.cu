// Products of fp32 matrices that lie in memory as two scaled fp16 planes (split.cuh):
// C = alpha*A*B^T or C += alpha*A*B^T with lo*hi + hi*lo + hi*hi on tcgen05.mma.kind::f16.
//
// Against the engine that splits fp32 tiles in shared memory into tf32 terms (gemm_tc.cu): the tensor core does
// twice the products of a tf32 pass per cycle, a term is two bytes instead of four, and nothing but TMA writes
// shared memory, so that the kernel is bound by the tensor pipe instead of shared memory.  Both
// terms are rounded to nearest (11 + 11 bits, the dropped lo*lo is 2^-24 relative and has either sign).
//
// Pipeline of one persistent CTA:
//   warp 0      TMA: hi and lo planes of 32 k-values of A and B, one box each (K-major) or one per 64 columns
//   warp 1      MMA: per 16 k-values three tcgen05.mma, M=128 N=BN K=16, into one of two TMEM buffers
//   warps 4..11 drain: accumulators leave TMEM every 128 k-values, are scaled by the powers of two of the blocks
//               that were multiplied and summed in registers (the tensor core truncates when it
//               accumulates, so chains are short); at the end of a tile they leave through shared memory as TMA
//               stores (beta 0) or TMA reductions in L2 (beta 1), or split again for the next product.
// Tiles are 128 x 256 (4 stages of 48 KB) or 128 x 128 (6 stages of 32 KB).  Both cut k into the same chains on
// the same grid of 128, so a product gives the same bits with either.
// Operands may be stored [rows, K] or [K, rows]; both are native layouts.
// All mbarrier waits are bounded (tc_common.cuh).
#include "split_tc.cuh"

namespace {

using namespace octc;

constexpr int BM = 128, BK = SPLIT_BK, CHAIN_K = 128, CHAIN_STAGES = CHAIN_K / BK;
// Three warpgroups: TMA, MMA and two idle warps; eight drain warps.  They trade registers (setmaxnreg): a drain
// thread of a wide tile holds 128 sums.
constexpr int FIRST_DRAIN = 4, DRAIN_WARPS = 8, THREADS = 32 * (FIRST_DRAIN + DRAIN_WARPS);

template <int BN_, int STAGES_>
struct Shape {
  static constexpr int BN = BN_, STAGES = STAGES_;
  static constexpr int A_BYTES = BM * BK * 4, B_BYTES = BN * BK * 4;   // both planes
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int DW = BN * 4 / DRAIN_WARPS;                       // columns per drain warp
  static constexpr int SMEM_DYN = STAGES * STAGE_BYTES + 1024 + DRAIN_WARPS * 4096;
  static constexpr int TMEM_COLS = 2 * BN;
};
using Narrow = Shape<128, 6>;
using Wide = Shape<256, 4>;

struct Params {
  const float* C; long long ldc, strideC1, strideC2;
  int M, N, K, nb1, nb2;
  float alpha;
  int add;
  int flags, tiles_m, tiles_n, per_problem;
  int a_terms;
  const float *a_scale, *b_scale;
  long long a_sk, a_sr, a_s1, a_s2, b_sk, b_sr, b_s1, b_s2;
  int a_row;
  int out_mode, store_c;         // planes of the result (wide tiles only)
  float* o_table;
  long long o_ldt, o_t1, o_t2;
  int* status;
};

// K-major: a plane is ROWS rows of 64 bytes (64-byte swizzle), groups of 8 rows 512 bytes apart, 16 k-values
//   are 32 bytes.  lo lies a plane behind hi.  MN-major: see split_desc_mn.
template <bool MN>
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, int k16) {
  if (MN) return split_desc_mn(addr, k16);
  uint64_t d = (uint64_t)(((addr + k16 * 32) & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;                   // unused for swizzled K-major layouts
  d |= (uint64_t)(512 >> 4) << 32;
  d |= 1ull << 46;
  d |= 4ull << 61;
  return d;
}
template <bool MN, int ROWS> constexpr int LO_OFFSET = MN ? SPLIT_MN_LO : ROWS * 64;

template <bool MN, int ROWS>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap* map, int mn0, int k0, int z1, int z2, uint32_t bar) {
  if (MN) {
#pragma unroll
    for (int a = 0; a < ROWS / 64; ++a) tma_load_planes(dst + a * SPLIT_MN_ATOM, map, mn0 + a * 64, k0, z1, z2, bar);
  } else {
    tma_load_planes(dst, map, k0, mn0, z1, z2, bar);
  }
}

__device__ __forceinline__ void tma_store(const CUtensorMap* map, uint32_t src, int x, int y, int z1, int z2, int add) {
  if (add)
    asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                 ::"l"(map), "r"(x), "r"(y), "r"(z1), "r"(z2), "r"(src) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                 ::"l"(map), "r"(x), "r"(y), "r"(z1), "r"(z2), "r"(src) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__device__ __forceinline__ void tma_store_plane(const CUtensorMap* map, uint32_t src, int x, int y, int z1, int z2, int plane) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4, %5}], [%6];"
               ::"l"(map), "r"(x), "r"(y), "r"(z1), "r"(z2), "r"(plane), "r"(src) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// ---- the order of the tiles ---------------------------------------------------------------------
// A CTA takes one tile of every wave of gridDim.x tiles, from the front in even and from the back in odd
// waves.  Where the flags give tiles k-ranges of different length, the longest come first, so that the sums of
// the CTAs differ by less than a tile.  Tiles above the diagonal of a lower-tiles-only product are not counted.
struct Tile { int z1, z2, m0, n0, k_lo, k_hi; };

// tiles of row block `i` of a lower-tiles-only product
template <int BN>
__host__ __device__ __forceinline__ int lower_count(int i, int tiles_n) {
  const int c = (i * BM + BM - 1) / BN + 1;
  return c < tiles_n ? c : tiles_n;
}

template <int BN>
struct Walker {
  int wave = 0, z = 0, row = 0, base = 0;      // lower tiles only: the row of the last tile, tiles before it
  __device__ __forceinline__ bool next(const Params& p, Tile& t) {
    const long long total = (long long)p.per_problem * p.nb1 * p.nb2;
    const long long i = (long long)wave * gridDim.x + ((wave & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    ++wave;
    if (i >= total) return false;            // (an incomplete wave is the last one)
    locate(p, (int)i, t);
    return true;
  }
  __device__ __forceinline__ void locate(const Params& p, int item, Tile& t) {
    const int zi = item / p.per_problem, r = item - zi * p.per_problem;
    t.z1 = zi % p.nb1; t.z2 = zi / p.nb1;
    if (p.flags & OC_GEMM_SKIP_UPPER_TILES) {
      if (zi != z) { z = zi; row = 0; base = 0; }
      int cnt = lower_count<BN>(row, p.tiles_n);
      while (r >= base + cnt) { base += cnt; cnt = lower_count<BN>(++row, p.tiles_n); }
      t.m0 = row * BM; t.n0 = (r - base) * BN;
    } else if (p.flags & (OC_GEMM_KLO_FROM_N | OC_GEMM_KHI_FROM_N)) {
      const int n = r / p.tiles_m;
      t.m0 = (r - n * p.tiles_m) * BM;
      t.n0 = ((p.flags & OC_GEMM_KHI_FROM_N) ? p.tiles_n - 1 - n : n) * BN;
    } else {
      const int m = r / p.tiles_n;
      t.n0 = (r - m * p.tiles_n) * BN;
      t.m0 = ((p.flags & OC_GEMM_KHI_FROM_M) ? p.tiles_m - 1 - m : m) * BM;
    }
    t.k_lo = 0; t.k_hi = p.K;
    if (p.flags & OC_GEMM_KLO_FROM_N) t.k_lo = max(t.k_lo, t.n0);
    if (p.flags & OC_GEMM_KLO_FROM_M) t.k_lo = max(t.k_lo, t.m0);
    if (p.flags & OC_GEMM_KHI_FROM_M) t.k_hi = min(t.k_hi, t.m0 + BM);
    if (p.flags & OC_GEMM_KHI_FROM_N) t.k_hi = min(t.k_hi, t.n0 + BN);
  }
};

// the upper 128 columns of a wide tile that straddles the diagonal of a lower-tiles-only product are a tile the
// narrow shape skips: no MMA, not written
template <int BN>
__device__ __forceinline__ bool upper_half_in_use(const Params& p, const Tile& t) {
  return BN == 128 || !(p.flags & OC_GEMM_SKIP_UPPER_TILES) || t.n0 + 128 <= t.m0 + BM - 1;
}

template <bool A_MN, bool B_MN, class S>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_o, const Params p) {
  constexpr int BN = S::BN, STAGES = S::STAGES, STAGE_BYTES = S::STAGE_BYTES, A_BYTES = S::A_BYTES, DW = S::DW;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag_s;
  __shared__ float block_max[2][2][4];           // [tile & 1][half][quarter]
  volatile int* abort_flag = &abort_flag_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* stage_ptr = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t stage_base = smem_u32(stage_ptr);

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&bar_full[s]), 1); mbar_init(smem_u32(&bar_empty[s]), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(smem_u32(&bar_acc_full[b]), 1); mbar_init(smem_u32(&bar_acc_empty[b]), DRAIN_WARPS); }
    abort_flag_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid == 64) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_c) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)S::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  oc_wait_before();
  Walker<BN> walk;
  Tile t;

  if (warp < FIRST_DRAIN) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 1;
      bool ok = true;
      const uint32_t bytes = (uint32_t)(A_BYTES / 2 * p.a_terms + S::B_BYTES);
      while (ok && walk.next(p, t)) {
        for (int k0 = t.k_lo; k0 < t.k_hi; k0 += BK) {
          ok = mbar_wait(smem_u32(&bar_empty[stage]), phase, abort_flag, p.status, 301);
          if (!ok) break;
          const uint32_t bar = smem_u32(&bar_full[stage]);
          const uint32_t sa = stage_base + stage * STAGE_BYTES;
          mbar_expect_tx(bar, bytes);
          load_operand<A_MN, BM>(sa, &map_a, t.m0, k0, t.z1, t.z2, bar);
          load_operand<B_MN, BN>(sa + A_BYTES, &map_b, t.n0, k0, t.z1, t.z2, bar);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      oc_let_next();
      if (!ok) {
        // let copies already issued land before the CTA's shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t ID_FULL = split_idesc(A_MN, B_MN, BM, BN), ID_HALF = split_idesc(A_MN, B_MN, BM, 128);
      uint32_t stage = 0, phase = 0, cc = 0;
      bool ok = true;
      while (ok && walk.next(p, t)) {
        const uint32_t ID = upper_half_in_use<BN>(p, t) ? ID_FULL : ID_HALF;
        const int n_stages = max(0, (t.k_hi - t.k_lo + BK - 1) / BK);
        const int n_chunks = max(1, (n_stages + CHAIN_STAGES - 1) / CHAIN_STAGES);
        for (int ch = 0; ch < n_chunks && ok; ++ch, ++cc) {
          const uint32_t buf = cc & 1u;
          ok = mbar_wait(smem_u32(&bar_acc_empty[buf]), ((cc >> 1) & 1u) ^ 1u, abort_flag, p.status, 302);
          if (!ok) break;
          tc_fence_after();
          const int s_begin = ch * CHAIN_STAGES, s_end = min(n_stages, s_begin + CHAIN_STAGES);
          const uint32_t tmem_d = tmem_base + buf * BN;
          for (int s = s_begin; s < s_end; ++s) {
            ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag, p.status, 303);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_hi = stage_base + stage * STAGE_BYTES, a_lo = a_hi + LO_OFFSET<A_MN, BM>;
            const uint32_t b_hi = a_hi + A_BYTES, b_lo = b_hi + LO_OFFSET<B_MN, BN>;
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              const uint64_t dah = make_desc<A_MN>(a_hi, kk), dal = make_desc<A_MN>(a_lo, kk);
              const uint64_t dbh = make_desc<B_MN>(b_hi, kk), dbl = make_desc<B_MN>(b_lo, kk);
              umma_f16(tmem_d, dah, dbl, ID, (s > s_begin || kk > 0) ? 1u : 0u);
              if (p.a_terms == 2) umma_f16(tmem_d, dal, dbh, ID, 1u);
              umma_f16(tmem_d, dah, dbh, ID, 1u);
            }
            umma_commit(smem_u32(&bar_empty[stage]));
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
          if (ok) umma_commit(smem_u32(&bar_acc_full[buf]));
        }
      }
    }
    __syncwarp();
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // drain warps: TMEM lane quarter = warp % 4; a second set of four takes the upper half of the columns
    // The epilogue passes 32 x 32 slices of the tile through 4 KB of shared memory per warp.  Reading the old
    // values of C into registers instead, 16 rows at a time, kept the drain warps so long that the tensor
    // pipe ran out of buffers: 28672 x 3584 x 512 420 us, now 292 us.
    const int quarter = warp & 3, half = (warp - FIRST_DRAIN) >> 2;
    uint8_t* stg_ptr = stage_ptr + STAGES * STAGE_BYTES + (warp - FIRST_DRAIN) * 4096;
    const uint32_t stg = smem_u32(stg_ptr);
    uint32_t cc = 0;
    int tiles = 0;
    bool ok = true;
    while (walk.next(p, t)) {
      const int n_stages = max(0, (t.k_hi - t.k_lo + BK - 1) / BK);
      const int n_chunks = max(1, (n_stages + CHAIN_STAGES - 1) / CHAIN_STAGES);
      const bool in_use = half == 0 || upper_half_in_use<BN>(p, t);
      const int row0 = t.m0 + quarter * 32, col0 = t.n0 + half * DW;
      if (in_use && p.add)
        prefetch_tile<DW>(p.C + t.z1 * p.strideC1 + t.z2 * p.strideC2, p.ldc, p.M, p.N, row0, col0, lane);
      const float *sa = nullptr, *sb = nullptr;
      if (p.a_scale)
        sa = p.a_scale + t.z1 * p.a_s1 + t.z2 * p.a_s2 + (t.k_lo / 128) * p.a_sk + (t.m0 / 128) * p.a_sr +
             (p.a_row ? min(quarter * 32 + lane, p.M - 1 - t.m0) : 0);
      if (p.b_scale)      // (columns behind N have no entry)
        sb = p.b_scale + t.z1 * p.b_s1 + t.z2 * p.b_s2 + (t.k_lo / 128) * p.b_sk + (min(col0, p.N - 1) / 128) * p.b_sr;
      float acc[DW];
#pragma unroll
      for (int i = 0; i < DW; ++i) acc[i] = 0.f;
      for (int ch = 0; ch < n_chunks; ++ch, ++cc) {
        const uint32_t buf = cc & 1u;
        float fa = 1.f, fb = 1.f;
        if (n_stages > 0 && sa) fa = sa[ch * p.a_sk];
        if (n_stages > 0 && sb) fb = sb[ch * p.b_sk];
        ok = mbar_wait(smem_u32(&bar_acc_full[buf]), (cc >> 1) & 1u, abort_flag, p.status, 304);
        if (!ok) break;
        tc_fence_after();
        if (n_stages > 0 && in_use) {
          const float f = fa * fb;
          const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * BN + half * DW;
#pragma unroll
          for (int c = 0; c < DW / 32; ++c) {
            float v[32];
            tmem_ld32(taddr + c * 32, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[c * 32 + i] = fmaf(v[i], f, acc[c * 32 + i]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[buf]));
      }
      if (!ok) break;
      if (!in_use) continue;
      if (BN == 128 || p.store_c) {
#pragma unroll
        for (int c = 0; c < DW / 32; ++c) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float* v = acc + c * 32 + j * 4;
            // (16-byte chunks in the order of the 128-byte swizzle: free of bank conflicts)
            *reinterpret_cast<float4*>(stg_ptr + lane * 128 + ((j ^ (lane & 7)) * 16)) =
                make_float4(p.alpha * v[0], p.alpha * v[1], p.alpha * v[2], p.alpha * v[3]);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0 && row0 < p.M && col0 + c * 32 < p.N)
            tma_store(&map_c, stg, col0 + c * 32, row0, t.z1, t.z2, p.add);
        }
      }
      if (BN == 256 && p.out_mode) {
        // The result as the next product's operand.  A thread has one row of a block of 128 columns, the four warps of a
        // half its 128 rows.  As a pass of its own this read and wrote 8 bytes an entry: correction of 4096 x 4096
        // 858 -> 821 us.
        float mx = 0.f, inv;
#pragma unroll
        for (int i = 0; i < DW; ++i) { acc[i] *= p.alpha; mx = fmaxf(mx, oc_finite_abs(acc[i])); }
        if (p.out_mode == OC_SPLIT_OUT_BLOCKS) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          float* red = block_max[tiles & 1][half];
          if (lane == 0) red[quarter] = mx;
          asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
          mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
        }
        const float se = oc_split_scale(mx, inv);
        float* tab = p.o_table + t.z1 * p.o_t1 + t.z2 * p.o_t2;
        if (col0 < p.N) {
          if (p.out_mode == OC_SPLIT_OUT_BLOCKS) {
            if (lane == 0 && quarter == 0) tab[(long long)(t.m0 / 128) * p.o_ldt + col0 / 128] = inv;
          } else if (row0 + lane < p.M) {
            tab[(long long)(col0 / 128) * p.o_ldt + row0 + lane] = inv;
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int pl = 0; pl < 2; ++pl) {         // 32 rows x 64 columns of a plane
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float* v = acc + (DW == 128 ? c * 64 + j * 8 : 0);
              uint2 h0, l0, h1, l1;
              oc_split4(make_float4(v[0] * se, v[1] * se, v[2] * se, v[3] * se), h0, l0);
              oc_split4(make_float4(v[4] * se, v[5] * se, v[6] * se, v[7] * se), h1, l1);
              *reinterpret_cast<uint4*>(stg_ptr + lane * 128 + ((j ^ (lane & 7)) * 16)) =
                  pl ? make_uint4(l0.x, l0.y, l1.x, l1.y) : make_uint4(h0.x, h0.y, h1.x, h1.y);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && row0 < p.M && col0 + c * 64 < p.N)
              tma_store_plane(&map_o, stg, col0 + c * 64, row0, t.z1, t.z2, pl);
          }
      }
      ++tiles;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem_base), "r"((uint32_t)S::TMEM_COLS) : "memory");
  }
}

int make_map_c(CUtensorMap* map, const OcSplitGemm& g) {
  EncodeTiledFn enc = get_encode_fn();
  const cuuint64_t whole = (cuuint64_t)g.M * (cuuint64_t)g.ldc * 4;
  cuuint64_t dims[4] = {(cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.nb1, (cuuint64_t)g.nb2};
  cuuint64_t strides[3] = {(cuuint64_t)g.ldc * 4, g.nb1 > 1 ? (cuuint64_t)g.strideC1 * 4 : whole,
                           g.nb2 > 1 ? (cuuint64_t)g.strideC2 * 4 : whole};
  cuuint32_t box[4] = {32, 32, 1, 1}, estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, g.C, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { oc_set_last_error("split gemm: cuTensorMapEncodeTiled failed"); return OC_ERR_CUDA; }
  return OC_OK;
}

int make_map_out(CUtensorMap* map, const OcSplitGemm& g) {
  EncodeTiledFn enc = get_encode_fn();
  const OcSplitOut& o = g.out;
  const cuuint64_t whole = (cuuint64_t)g.M * (cuuint64_t)o.ld * 2;
  cuuint64_t dims[5] = {(cuuint64_t)g.N, (cuuint64_t)g.M, (cuuint64_t)g.nb1, (cuuint64_t)g.nb2, 2};
  cuuint64_t strides[4] = {(cuuint64_t)o.ld * 2, g.nb1 > 1 ? (cuuint64_t)o.stride1 * 2 : whole,
                           g.nb2 > 1 ? (cuuint64_t)o.stride2 * 2 : whole, (cuuint64_t)o.plane * 2};
  cuuint32_t box[5] = {64, 32, 1, 1, 1}, estr[5] = {1, 1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, o.planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { oc_set_last_error("split gemm: cuTensorMapEncodeTiled failed"); return OC_ERR_CUDA; }
  return OC_OK;
}

template <bool A_MN, bool B_MN, class S>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const CUtensorMap& mo, const Params& p, int grid, cudaStream_t s) {
  OC_OPT_IN_SMEM((gemm_split_kernel<A_MN, B_MN, S>), S::SMEM_DYN);
  OC_LAUNCH((gemm_split_kernel<A_MN, B_MN, S>), grid, THREADS, S::SMEM_DYN, s, ma, mb, mc, mo, p);
  return OC_OK;
}

template <int BN>
long long tiles_of(const OcSplitGemm& g) {
  const int tm = oc_div_up(g.M, BM), tn = oc_div_up(g.N, BN);
  if (!(g.flags & OC_GEMM_SKIP_UPPER_TILES)) return (long long)tm * tn;
  long long n = 0;
  for (int i = 0; i < tm; ++i) n += lower_count<BN>(i, tn);
  return n;
}

template <class S>
int launch_shape(const OcSplitGemm& g, const OcGemmDevice& dev, cudaStream_t stream) {
  CUtensorMap ma, mb, mc, mo;
  int rc = make_split_map(&ma, g.A, g.M, g.K, g.nb1, g.nb2, BM);
  if (rc) return rc;
  rc = make_split_map(&mb, g.B, g.N, g.K, g.nb1, g.nb2, S::BN);
  if (rc) return rc;
  rc = make_map_c(&mc, g);
  if (rc) return rc;
  mo = mc;
  if (S::BN == 256 && g.out.mode) {
    rc = make_map_out(&mo, g);
    if (rc) return rc;
  }
  Params p{};
  p.C = g.C; p.ldc = g.ldc; p.strideC1 = g.strideC1; p.strideC2 = g.strideC2;
  p.M = g.M; p.N = g.N; p.K = g.K; p.nb1 = g.nb1; p.nb2 = g.nb2;
  p.alpha = g.alpha; p.add = g.add; p.flags = g.flags;
  p.tiles_m = oc_div_up(g.M, BM); p.tiles_n = oc_div_up(g.N, S::BN);
  p.a_terms = g.A.terms;
  p.a_scale = g.A.scale; p.a_sk = g.A.scale_k; p.a_sr = g.A.scale_r; p.a_s1 = g.A.scale1; p.a_s2 = g.A.scale2;
  p.a_row = g.A.scale_row;
  p.b_scale = g.B.scale; p.b_sk = g.B.scale_k; p.b_sr = g.B.scale_r; p.b_s1 = g.B.scale1; p.b_s2 = g.B.scale2;
  p.out_mode = g.out.mode; p.store_c = !(g.out.mode && g.out.only);
  p.o_table = g.out.table; p.o_ldt = g.out.ldt; p.o_t1 = g.out.tab1; p.o_t2 = g.out.tab2;
  p.status = dev.status;
  const long long per = tiles_of<S::BN>(g), items = per * g.nb1 * g.nb2;
  OC_REQUIRE(items < (1ll << 30), "split gemm: too many tiles");
  p.per_problem = (int)per;
  const int grid = (int)(items < dev.sms ? items : dev.sms);
  if (g.A.mn_major)
    return g.B.mn_major ? launch<true, true, S>(ma, mb, mc, mo, p, grid, stream) : launch<true, false, S>(ma, mb, mc, mo, p, grid, stream);
  return g.B.mn_major ? launch<false, true, S>(ma, mb, mc, mo, p, grid, stream) : launch<false, false, S>(ma, mb, mc, mo, p, grid, stream);
}

// Time of a wide tile against a narrow one.
constexpr double WIDE_TILE_COST = 1.45;

}  // namespace

int oc_gemm_split_launch(const OcSplitGemm& g, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0 || g.nb1 <= 0 || g.nb2 <= 0) return OC_OK;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  auto fits = [&](const OcSplitOperand& o) {
    return al(o.planes) && o.ld % 8 == 0 && o.plane % 8 == 0 && o.stride1 % 8 == 0 && o.stride2 % 8 == 0;
  };
  OC_REQUIRE(g.K > 0 && fits(g.A) && fits(g.B) && g.B.terms == 2 && (g.A.terms == 2 || !g.A.mn_major), "split gemm: bad operand");
  OC_REQUIRE(al(g.C) && g.ldc % 4 == 0 && g.strideC1 % 4 == 0 && g.strideC2 % 4 == 0, "split gemm: C is not 16-byte aligned");
  OC_REQUIRE(!g.out.mode || (!g.add && !(g.flags & OC_GEMM_SKIP_UPPER_TILES) && al(g.out.planes) && g.out.ld % 8 == 0 &&
                             g.out.plane % 8 == 0 && g.out.stride1 % 8 == 0 && g.out.stride2 % 8 == 0), "split gemm: bad output");
  OcGemmDevice dev;
  int rc = oc_gemm_device(dev);
  if (rc) return rc;
  int shape = dev.tile_shape;
  if (shape == 0) {
    const long long nb = (long long)g.nb1 * g.nb2, sms = dev.sms;
    const double narrow = (double)((tiles_of<128>(g) * nb + sms - 1) / sms);
    const double wide = WIDE_TILE_COST * (double)((tiles_of<256>(g) * nb + sms - 1) / sms);
    shape = wide < narrow ? 2 : 1;
  }
  if (shape == 2) return launch_shape<Wide>(g, dev, stream);
  rc = launch_shape<Narrow>(g, dev, stream);
  if (rc || !g.out.mode) return rc;
  // (a drain thread of a narrow tile has half of a block's columns: a pass of its own)
  OcSplitArgs s{};
  s.src = g.C; s.ld = g.ldc; s.rows = g.M; s.cols = g.N; s.nb1 = g.nb1; s.nb2 = g.nb2;
  s.planes = g.out.planes; s.plane = g.out.plane; s.ldp = g.out.ld; s.table = g.out.table; s.ldt = g.out.ldt;
  s.per_row = g.out.mode == OC_SPLIT_OUT_ROWS;
  s.src1 = g.strideC1; s.src2 = g.strideC2; s.dst1 = g.out.stride1; s.dst2 = g.out.stride2; s.tab1 = g.out.tab1; s.tab2 = g.out.tab2;
  return oc_split_launch(s, stream);
}

// ---- C entry for the tests --------------------------------------------------------------------------
// C = alpha*opA(A)*opB(B) (+ C with `add`), operands as for oc_gemm_f32, both operands split first.  rows_scaled: A is scaled by rows
// (A not transposed).  workspace: oc_gemm_split_workspace_bytes, 256-byte aligned.
static long long pad8(long long x) { return (x + 7) / 8 * 8; }
static long long split_bytes(long long rows, long long cols) {
  const long long planes = 2 * rows * pad8(cols) * 2, table = (oc_div_up(cols, 128) * (rows + 128)) * 4ll;
  return (planes + 255) / 256 * 256 + (table + 255) / 256 * 256;
}
extern "C" long long oc_gemm_split_workspace_bytes(int M, int N, int K, int transA, int transB) {
  return (transA ? split_bytes(K, M) : split_bytes(M, K)) + (transB ? split_bytes(N, K) : split_bytes(K, N));
}
extern "C" int oc_gemm_split_f32(const float* A, long long lda, const float* B, long long ldb, float* C, long long ldc,
                                 int M, int N, int K, float alpha, int add, int transA, int transB, int flags,
                                 int rows_scaled, void* workspace, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  OC_REQUIRE(A && B && C && workspace && M > 0 && N > 0 && K > 0, "gemm_split: bad arguments");
  OC_REQUIRE(!(rows_scaled && transA), "gemm_split: rows of a transposed A have no scales of their own");
  char* ws = (char*)workspace;
  auto split = [&](const float* src, long long ld, int rows, int cols, int per_row, OcSplitOperand& o) {
    OcSplitArgs s{};
    s.src = src; s.ld = ld; s.rows = rows; s.cols = cols; s.nb1 = s.nb2 = 1; s.per_row = per_row;
    s.ldp = pad8(cols); s.plane = (long long)rows * s.ldp; s.planes = (__half*)ws;
    s.table = (float*)(ws + (2 * s.plane * 2 + 255) / 256 * 256);
    s.ldt = per_row ? rows : oc_div_up(cols, 128);
    ws += split_bytes(rows, cols);
    o.planes = s.planes; o.plane = s.plane; o.ld = s.ldp; o.terms = 2; o.scale = s.table; o.scale_row = per_row;
    if (per_row) { o.scale_k = s.ldt; o.scale_r = 128; }
    else if (o.mn_major) { o.scale_k = s.ldt; o.scale_r = 1; }
    else { o.scale_k = 1; o.scale_r = s.ldt; }
    return oc_split_launch(s, stream);
  };
  OcSplitGemm g{};
  g.A.mn_major = transA != 0; g.B.mn_major = transB == 0;
  int rc = transA ? split(A, lda, K, M, 0, g.A) : split(A, lda, M, K, rows_scaled, g.A);
  if (rc) return rc;
  rc = transB ? split(B, ldb, N, K, 0, g.B) : split(B, ldb, K, N, 0, g.B);
  if (rc) return rc;
  g.C = C; g.ldc = ldc; g.M = M; g.N = N; g.K = K; g.nb1 = g.nb2 = 1;
  g.alpha = alpha; g.add = add != 0; g.flags = flags;
  return oc_gemm_split_launch(g, stream);
}
