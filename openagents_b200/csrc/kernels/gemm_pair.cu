// bf16 GEMM for large products: D[M][N] = A[M][K] * B[N][K]^T (+ epilogue) on pairs of CTAs.
//
// Two CTAs of a cluster (the two SMs of a TPC) share one 256 x BN output tile (BN 256 or 128) through
// tcgen05.mma.cta_group::2: each SM loads 128 rows of A and BN / 2 rows of B, the tensor cores of both read
// both halves of B.  A K block of 64 then takes 512 cycles and 32 KB of shared-memory reads per SM, half of what
// shared memory delivers, where a 128 x 256 tile of one CTA needs 48 KB in the same time (three quarters).  The
// room that this leaves is what the epilogue needs: it goes through shared memory and leaves by TMA (a plain store, or
// a reduction that adds in L2), so that the warps issue no scattered stores and the next tile's MMAs run beside it.
//
//   warp 0      one thread per CTA: TMA loads of its half of A and B; both halves count on the first CTA's barrier
//   warp 1      first CTA, one thread: tcgen05.mma for the pair; commits release the slots of both CTAs
//   warps 2..5  epilogue of this CTA's 128 rows: tensor memory -> registers -> swizzled shared memory -> TMA
//
// Persistent: a pair walks tiles with a ring of six 32 KB stages per CTA (eight of 24 KB) and two accumulators of BN columns.  Tiles are
// walked in panels of 16 rows of tiles, so that the 74 pairs of a wave read about 16 blocks of A and 5 of B.
// Every wait is bounded and reports through `status`.
#include "gemm_pair.h"
#include "tc05.cuh"

using namespace b200;
using namespace b200::tc;

namespace {

enum { OUT_16 = 0, OUT_F32 = 1, OUT_SWIGLU = 2, OUT_COMBINE = 3 };
enum { ACT_GELU = 1, ACT_RELU2 = 3, ACT_GELU_ERF = 4 };      // as in gemm_tc05.cu

constexpr int BM = 128, BK = 64;                              // rows per CTA, K per stage
constexpr int kPanel = 16;
constexpr int kABytes = BM * BK * 2;
constexpr int kPatch = 4096;                                  // epilogue staging: 32 rows x 128 bytes, two per warp
// The grouped form gives one stage up for its list of live tiles.
constexpr int stages_of(int bn, bool grouped) { return (bn == 256 ? 6 : 8) - (grouped ? 1 : 0); }
constexpr size_t smem_bytes(int bn, bool grouped) {
  const int stages = stages_of(bn, grouped);
  return 1024 + (size_t)stages * (kABytes + bn / 2 * BK * 2) + 8 * kPatch + (grouped ? kPairLiveTiles * 4 : bn * 4) + (2 * stages + 4) * 8 + 16;
}
static_assert(smem_bytes(256, false) + 64 <= 232448 && smem_bytes(256, true) + 64 <= 232448 && smem_bytes(128, false) + 64 <= 232448 &&
              smem_bytes(128, true) + 64 <= 232448, "shared memory per CTA");

struct PairArgs {
  int M, N, K, tiles_m, tiles_n, splits, kps;
  const float* bias;
  const __nv_bfloat16* resid;
  int ldc, act, half_out, add;
  float alpha;
  int group_rows, groups;
  const int* group_counts;
  const int* meta;
  const float* gate_w;
  size_t sym_off;
  int end_barrier;
  int* status;
  SymTable sym;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address of the first CTA's copy of a shared-memory variable.
__device__ __forceinline__ uint32_t in_first_cta(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// TMA load into this CTA's shared memory that counts on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once every MMA issued so far has finished.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_add_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

struct Tile { int m0, n0, live_end, group; };      // first row of the pair's tile, first column, rows below live_end are written

template <int BN, bool GROUPED>
__device__ __forceinline__ Tile locate(const PairArgs& a, const int* live_m, int tile, int tiles_m) {
  Tile t;
  if constexpr (GROUPED) {                  // columns fastest: one expert's rows and weights at a time
    const int v = live_m[tile / a.tiles_n];
    t.m0 = v;
    t.n0 = (tile % a.tiles_n) * BN;
    t.group = v / a.group_rows;
    t.live_end = t.group * a.group_rows + min(a.group_counts[t.group], a.group_rows);
  } else {
    const int p = tile / (kPanel * a.tiles_n), r = tile - p * kPanel * a.tiles_n;
    const int rows = min(kPanel, tiles_m - p * kPanel);
    t.m0 = (p * kPanel + r % rows) * kPairRows;
    t.n0 = (r / rows) * BN;
    t.live_end = a.M;
    t.group = 0;
  }
  return t;
}

template <int BN, bool MN, int OUT, bool GROUPED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                     const __grid_constant__ PairArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int kStages = stages_of(BN, GROUPED), BNH = BN / 2, kBBytes = BNH * BK * 2;
  uint8_t* sA = smem;
  uint8_t* sB = sA + kStages * kABytes;
  uint8_t* patch_all = sB + kStages * kBBytes;
  float* s_bias = (float*)(patch_all + 8 * kPatch);
  int* live_m = (int*)s_bias;                    // grouped: first row of every tile with live rows
  uint64_t* full = (uint64_t*)(s_bias + (GROUPED ? kPairLiveTiles : BN));     // [kStages] first CTA's: both CTAs' bytes have landed
  uint64_t* empty = full + kStages;              // [kStages] this CTA's slot is free
  uint64_t* tfull = empty + kStages;             // [2] accumulator complete
  uint64_t* tempty = tfull + 2;                  // [2] first CTA's: all eight epilogue warps have read the accumulator
  uint32_t* tmem_holder = (uint32_t*)(tempty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
  __shared__ int s_n_live;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int KB = (a.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(smem_u32(full + s), 1);
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(smem_u32(tfull + s), 1);
      mbar_init(smem_u32(tempty + s), 8);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if constexpr (OUT != OUT_COMBINE) tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(2 * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                // the partner's barriers are set up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  pdl_trigger();
  pdl_wait();

  int tiles_m = a.tiles_m;
  if constexpr (GROUPED) {
    if (threadIdx.x == 0) {
      int n = 0;
      for (int g = 0; g < a.groups; g++) {
        const int cnt = min(a.group_counts[g], a.group_rows);
        for (int r = 0; r < cnt && n < kPairLiveTiles; r += kPairRows) live_m[n++] = g * a.group_rows + r;
      }
      s_n_live = n;
    }
    __syncthreads();
    tiles_m = s_n_live;
  }
  const int n_tiles = tiles_m * a.tiles_n, n_items = n_tiles * a.splits;

  if (warp == 0) {
    uint32_t s = 0, ph = 1;
    bool ok = true;
    const uint32_t full0 = in_first_cta(smem_u32(full)), empty0 = smem_u32(empty), own_full0 = smem_u32(full);
    for (int item = pair; item < n_items && ok; item += n_pairs) {
      const int sp = item / n_tiles;
      const Tile t = locate<BN, GROUPED>(a, live_m, item - sp * n_tiles, tiles_m);
      const int ar = t.m0 + (int)rank * BM;
      const int br = t.n0 + (int)rank * BNH + t.group * (GROUPED ? a.N : 0);
      const int kb0 = sp * a.kps, kb1 = min(KB, kb0 + a.kps);
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait_warp(empty0 + 8 * s, ph, abort_flag)) { ok = false; break; }
        const uint32_t bar = full0 + 8 * s, da = smem_u32(sA) + s * kABytes, db = smem_u32(sB) + s * kBBytes;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(own_full0 + 8 * s, 2 * (kABytes + kBBytes));
          if constexpr (MN) {                     // 64-column blocks of 64 k rows
#pragma unroll
            for (int h = 0; h < BM / 64; h++) tma_load_pair(da + h * 8192, &tmA, bar, ar + h * 64, kb * BK);
#pragma unroll
            for (int h = 0; h < BNH / 64; h++) tma_load_pair(db + h * 8192, &tmB, bar, br + h * 64, kb * BK);
          } else {
            tma_load_pair(da, &tmA, bar, kb * BK, ar);
            tma_load_pair(db, &tmB, bar, kb * BK, br);
          }
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // The whole warp walks the loop and one elected lane issues: the descriptors then live in uniform registers, which
      // tcgen05.mma takes its operands from.  A loop inside `if (lane == 0)` has to move each of them over per instruction.
      constexpr uint32_t idesc = idesc_bf16(2 * BM, BN) | (MN ? ((1u << 15) | (1u << 16)) : 0u);      // bits 15 / 16: A / B MN-major
      const uint64_t ad0 = MN ? smem_desc_sw128_mn(smem_u32(sA), 8192) : smem_desc_sw128(smem_u32(sA));
      const uint64_t bd0 = MN ? smem_desc_sw128_mn(smem_u32(sB), 8192) : smem_desc_sw128(smem_u32(sB));
      const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty);
      uint32_t s = 0, ph = 0, tcount = 0;
      bool ok = true;
      for (int item = pair; item < n_items && ok; item += n_pairs, tcount++) {
        const int sp = item / n_tiles;
        const int kb0 = sp * a.kps, kb1 = min(KB, kb0 + a.kps);
        const uint32_t acc = tcount & 1;
        if (!mbar_wait_warp(smem_u32(tempty + acc), ((tcount >> 1) & 1) ^ 1, abort_flag)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        uint32_t add = 0;
        for (int kb = kb0; kb < kb1; kb++) {
          if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t ad = ad0 + s * (kABytes >> 4), bd = bd0 + s * (kBBytes >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; k++)    // 16 of K: 32 bytes along K-major rows, 16 rows of 128 bytes otherwise
              umma_pair(d_tmem, ad + (MN ? 128 : 2) * k, bd + (MN ? 128 : 2) * k, idesc, k == 0 ? add : 1u);
            umma_commit_pair(empty0 + 8 * s);
          }
          __syncwarp();
          add = 1;
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
        if (elect_one()) umma_commit_pair(smem_u32(tfull + acc));      // released even after a failed wait; the flag says why
        __syncwarp();
      }
    }
  } else {
    const int q = warp & 3;                      // tensor-memory lane quarter
    const uint32_t patch = smem_u32(patch_all + q * 2 * kPatch);
    uint32_t n_out = 0;                          // patches handed to TMA so far
    uint32_t tcount = 0;
    // the patch after next may be written once the store before the last has read its own
    auto next_patch = [&]() -> uint32_t {
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      __syncwarp();
      return patch + (n_out & 1) * kPatch;
    };
    auto send = [&](int col, int row) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (OUT == OUT_F32 && a.add) tma_add_2d(&tmC, patch + (n_out & 1) * kPatch, col, row);
        else tma_store_2d(&tmC, patch + (n_out & 1) * kPatch, col, row);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      n_out++;
    };
    for (int item = pair; item < n_items; item += n_pairs, tcount++) {
      const int sp = item / n_tiles;
      const Tile t = locate<BN, GROUPED>(a, live_m, item - sp * n_tiles, tiles_m);
      const uint32_t acc = tcount & 1;
      const bool use_bias = (OUT == OUT_16 || OUT == OUT_F32) && a.bias && sp == 0;
      if (use_bias) {                            // the tile's bias values, shared by the four warps
        asm volatile("bar.sync 1, 128;" ::: "memory");
        for (int i = threadIdx.x - 64; i < BN; i += 128) s_bias[i] = t.n0 + i < a.N ? a.bias[t.n0 + i] : 0.f;
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      const int mw = t.m0 + (int)rank * BM + q * 32, m = mw + lane;      // this warp's first row, this thread's row
      const bool rows_live = mw < t.live_end;
      const bool resid = OUT == OUT_16 && a.resid && m < a.M;
      const __nv_bfloat16* rp = resid ? a.resid + (size_t)m * a.ldc + t.n0 : nullptr;
      uint4 rr[4];
      auto load_resid = [&](int c) {
        if constexpr (OUT == OUT_16) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            rr[i] = resid && t.n0 + c * 32 + i * 8 < a.N ? *(const uint4*)(rp + c * 32 + i * 8) : make_uint4(0, 0, 0, 0);
        }
      };
      if (OUT == OUT_16 && a.resid) load_resid(0);
      bool ok = mbar_wait(smem_u32(tfull + acc), (tcount >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok && !*abort_flag);
      if (!ok) continue;                         // every later wait gives up at once; the warps still meet at the barriers above
      tc_fence_after();

      uint32_t buf = 0;
      auto process = [&](int c, const uint32_t (&r)[32]) {
        const int n = t.n0 + c * 32;
        if (n >= a.N || !rows_live) return;
        if constexpr (OUT == OUT_SWIGLU) {        // 16 (gate, up) pairs; four chunks fill a patch of 64 columns
          const float w = GROUPED && a.gate_w ? a.gate_w[min(m, t.live_end - 1)] : 1.f;
          if ((c & 3) == 0) buf = next_patch();
          uint32_t o[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const float g0 = w * __uint_as_float(r[4 * j]), u0 = w * __uint_as_float(r[4 * j + 1]);
            const float g1 = w * __uint_as_float(r[4 * j + 2]), u1 = w * __uint_as_float(r[4 * j + 3]);
            o[j] = pack_bf16(silu(g0) * u0, silu(g1) * u1);
          }
#pragma unroll
          for (int h = 0; h < 2; h++)
            st_shared_v4(buf + lane * 128 + ((((c & 3) * 2 + h) ^ (lane & 7)) << 4), make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]));
          if ((c & 3) == 3 || n + 32 >= a.N) send((t.n0 >> 1) + (c >> 2) * 64, mw);
        } else if constexpr (OUT == OUT_COMBINE) {
          // transposed through the patch, so that an instruction adds four rows of 128 contiguous bytes
#pragma unroll
          for (int j = 0; j < 8; j++)
            st_shared_v4(patch + lane * 128 + ((j ^ (lane & 7)) << 4), make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
          __syncwarp();
          const int j = lane & 7;
          if (n + j * 4 < a.N) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const int row = (lane >> 3) + 4 * i, mr = mw + row;
              if (mr >= t.live_end) break;
              const float w = a.gate_w ? a.gate_w[mr] : 1.f;
              float4 o = *(const float4*)(patch_all + q * 2 * kPatch + row * 128 + ((j ^ (row & 7)) << 4));
              o.x *= w; o.y *= w; o.z *= w; o.w *= w;
              sym_red_to_f32x4(a.sym, a.meta[2 * mr], a.sym_off + ((size_t)a.meta[2 * mr + 1] * a.ldc + n + j * 4) * 4, o);
            }
          }
          __syncwarp();
        } else {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]) * a.alpha;
          if (use_bias) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 b = *(const float4*)(s_bias + c * 32 + j);
              v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
            }
          }
          if (a.act == ACT_GELU) {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = gelu_tanh(v[j]);
          } else if (a.act == ACT_GELU_ERF) {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = gelu_erf_fast(v[j]);
          } else if (a.act == ACT_RELU2) {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = v[j] > 0.f ? v[j] * v[j] : 0.f;
          }
          if constexpr (OUT == OUT_F32) {
            buf = next_patch();
#pragma unroll
            for (int j = 0; j < 8; j++)
              st_shared_v4(buf + lane * 128 + ((j ^ (lane & 7)) << 4), make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]),
                                                                                 __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3])));
            send(n, mw);
          } else {
            if (a.resid) {
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const __nv_bfloat162* p = (const __nv_bfloat162*)&rr[i];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                  const float2 f = __bfloat1622float2(p[e]);
                  v[8 * i + 2 * e] += f.x;
                  v[8 * i + 2 * e + 1] += f.y;
                }
              }
              if (c + 1 < BN / 32) load_resid(c + 1);
            }
            if ((c & 1) == 0) buf = next_patch();
#pragma unroll
            for (int h = 0; h < 4; h++) {
              uint4 o;
              if (a.half_out) {
                o = make_uint4(pack_f16(v[8 * h], v[8 * h + 1]), pack_f16(v[8 * h + 2], v[8 * h + 3]), pack_f16(v[8 * h + 4], v[8 * h + 5]),
                               pack_f16(v[8 * h + 6], v[8 * h + 7]));
              } else {
                o = make_uint4(pack_bf16(v[8 * h], v[8 * h + 1]), pack_bf16(v[8 * h + 2], v[8 * h + 3]), pack_bf16(v[8 * h + 4], v[8 * h + 5]),
                               pack_bf16(v[8 * h + 6], v[8 * h + 7]));
              }
              st_shared_v4(buf + lane * 128 + ((((c & 1) * 4 + h) ^ (lane & 7)) << 4), o);
            }
            if ((c & 1) == 1 || n + 32 >= a.N) send(t.n0 + (c >> 1) * 64, mw);
          }
        }
      };
      // two register buffers: the tensor-memory load of the next 32 columns is in flight while this chunk is finished
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      uint32_t ra[32], rb[32];
      tmem_ld32(t_addr, ra);
#pragma unroll 1
      for (int c = 0; c < BN / 32; c += 2) {
        tmem_ld_wait();
        tmem_ld32(t_addr + (uint32_t)((c + 1) * 32), rb);
        process(c, ra);
        tmem_ld_wait();
        if (c + 2 < BN / 32) {
          tmem_ld32(t_addr + (uint32_t)((c + 2) * 32), ra);
        } else {                                 // everything is in registers: the accumulator may be overwritten
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(in_first_cta(smem_u32(tempty + acc)));
        }
        process(c + 1, rb);
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                // neither CTA leaves while the other may still signal it
  __syncwarp();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BN) : "memory");
  if (threadIdx.x == 0 && *abort_flag && a.status) atomicExch(a.status, (int)B200_ERR_TIMEOUT_MMA);
  if (OUT == OUT_COMBINE && a.end_barrier) sym_kernel_end_barrier(a.sym, 0, gridDim.x);
}

int sm_pairs() {
  static int n = 0;
  if (!n) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    n = sms > 1 ? sms / 2 : 74;
  }
  return n;
}

template <int BN, bool MN, int OUT, bool GROUPED>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const PairArgs& a, int items, cudaStream_t st) {
  auto kern = gemm_pair_kernel<BN, MN, OUT, GROUPED>;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(BN, GROUPED));
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int pairs = items < sm_pairs() ? items : sm_pairs();
  return launch_pdl(kern, dim3(2 * pairs), dim3(192), smem_bytes(BN, GROUPED), st, ta, tb, tc, a);
}

}  // namespace

namespace b200 {

bool pair_takes(const PairGemm& g) {
  const bool one_out = (g.out_f32 != nullptr) + (g.out_16 != nullptr) + (g.combine ? 1 : 0) == 1;
  if (!one_out || g.M < 1 || g.N < 32 || g.K < BK) return false;
  if ((g.lda % 8) || (g.ldb % 8) || ((uintptr_t)g.A & 15) || ((uintptr_t)g.B & 15)) return false;
  if (g.out_f32 && ((g.ldc % 4) || ((uintptr_t)g.out_f32 & 15))) return false;
  if (g.out_16 && ((g.ldc % 8) || ((uintptr_t)g.out_16 & 15))) return false;
  if (((uintptr_t)g.bias & 15) || ((uintptr_t)g.resid_bf16 & 15) || (g.resid_bf16 && (!g.out_16 || g.N % 8))) return false;
  if (g.swiglu && (!g.out_16 || g.half_out || g.bias || g.resid_bf16 || g.act || (g.N % 32))) return false;
  if (g.add && !g.out_f32) return false;         // 16-bit results are stored: a split would leave its share alone
  if (g.splits > 1 && (!g.add || g.act)) return false;
  if (g.groups && (g.mn_major || (!g.swiglu && !g.combine) || g.group_rows % BM)) return false;
  return true;
}

template <int BN>
static int launch_tile(const PairGemm& g, cudaStream_t st) {
  CUtensorMap ta, tb, tc = {};
  const uint64_t b_rows = g.groups ? (uint64_t)g.groups * g.N : g.N;
  int rc = g.mn_major ? make_tmap_2d(&ta, g.A, 2, g.K, g.M, (uint64_t)g.lda * 2, BK, 64, true)
                      : make_tmap_2d(&ta, g.A, 2, g.M, g.K, (uint64_t)g.lda * 2, BM, BK, true);
  if (rc) return rc;
  rc = g.mn_major ? make_tmap_2d(&tb, g.B, 2, g.K, g.N, (uint64_t)g.ldb * 2, BK, 64, true)
                  : make_tmap_2d(&tb, g.B, 2, b_rows, g.K, (uint64_t)g.ldb * 2, BN / 2, BK, true);
  if (rc) return rc;
  if (g.out_f32) rc = make_tmap_2d(&tc, g.out_f32, 4, g.M, g.N, (uint64_t)g.ldc * 4, 32, 32, true);
  else if (g.out_16) rc = make_tmap_2d(&tc, g.out_16, 2, g.M, g.swiglu ? g.N / 2 : g.N, (uint64_t)g.ldc * 2, 32, 64, true);
  if (rc) return rc;
  PairArgs a = {};
  const int KB = (g.K + BK - 1) / BK, splits = g.splits > 1 ? g.splits : 1;
  a.M = g.M; a.N = g.N; a.K = g.K;
  a.tiles_m = (g.M + kPairRows - 1) / kPairRows;
  a.tiles_n = (g.N + BN - 1) / BN;
  a.kps = (KB + splits - 1) / splits;
  a.splits = (KB + a.kps - 1) / a.kps;           // no empty split
  a.bias = g.bias; a.resid = (const __nv_bfloat16*)g.resid_bf16; a.ldc = g.ldc; a.act = g.act; a.half_out = g.half_out; a.add = g.add;
  a.alpha = g.alpha; a.status = g.status;
  a.group_rows = g.group_rows; a.groups = g.groups; a.group_counts = g.group_counts; a.meta = g.meta; a.gate_w = g.gate_w;
  a.sym = g.sym; a.sym_off = g.sym_off; a.end_barrier = g.end_barrier;
  const int items = a.tiles_m * a.tiles_n * a.splits;
  if (g.groups) return g.combine ? launch<BN, false, OUT_COMBINE, true>(ta, tb, tc, a, items, st) : launch<BN, false, OUT_SWIGLU, true>(ta, tb, tc, a, items, st);
  if (g.swiglu) return launch<BN, false, OUT_SWIGLU, false>(ta, tb, tc, a, items, st);
  if (g.mn_major) return g.out_f32 ? launch<BN, true, OUT_F32, false>(ta, tb, tc, a, items, st) : launch<BN, true, OUT_16, false>(ta, tb, tc, a, items, st);
  return g.out_f32 ? launch<BN, false, OUT_F32, false>(ta, tb, tc, a, items, st) : launch<BN, false, OUT_16, false>(ta, tb, tc, a, items, st);
}

int launch_gemm_pair(const PairGemm& g, cudaStream_t st) {
  if (!pair_takes(g)) return B200_ERR_BAD_ARG;
  return g.tile_n == 128 ? launch_tile<128>(g, st) : launch_tile<256>(g, st);
}

}  // namespace b200

// The kernel by itself, for plain products (tests and measurements; b200_gemm_bf16 chooses it by size).  Exactly one of out_f32 and out_16.
B200_API int b200_gemm_pair(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int mn_major, float* out_f32, void* out_16,
                            int half_out, int swiglu, int add, int ldc, const float* bias, const void* resid_bf16, float alpha, int act,
                            int splits, int tile_n, int* status, cudaStream_t st) {
  PairGemm g = {};
  g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb; g.mn_major = mn_major; g.out_f32 = out_f32; g.out_16 = out_16;
  g.half_out = half_out; g.swiglu = swiglu; g.add = add; g.ldc = ldc; g.bias = bias; g.resid_bf16 = resid_bf16; g.alpha = alpha; g.act = act;
  g.splits = splits; g.tile_n = tile_n; g.status = status;
  return launch_gemm_pair(g, st);
}
