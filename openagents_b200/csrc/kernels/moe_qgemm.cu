// Grouped GEMM of a mixture-of-experts layer on MXFP4 weights, for few rows per expert (decode batches):
//     Y[t][n] (+)= sum_k X[t][k] * W[n][k]   for the rows t that each expert received.
// Such a layer reads every chosen expert's weights for a few dozen rows, so their bytes are the floor.  The grouped
// bf16 GEMM (gemm_tc05.cu) reads a bf16 expansion, 3.8 times as many; here the 4-bit blocks are expanded inside the
// pipeline, exactly (a 4-bit float times a power of two fits bf16), as qgemm_tc05.cu does for dense layers: the weight
// tile is the MMA's M operand in tensor memory, the expert's rows are its N operand (16, 32 or 64).
//
//   warp 0      TMA loads of packed tiles (128 rows x 128 bytes = 256 of K, 128-byte swizzle)
//   warp 1      one elected lane: tcgen05.mma, A from tensor memory, B from shared memory
//   warp 2      TMA loads of the expert's rows, 32 at a time
//   warps 4-19  expansion, two groups of eight that take stages in turn: a warp owns 32 weight rows (its tensor-memory lanes) and
//               128 of the 256 of K of its group's stages; the first group also runs the epilogue of item i after its first stage
//               of item i + 1
//
// Layout (pack_mxfp4_wide in torch_codecs.py): eight values to a 32-bit word, element i in half i % 2; the four values of a half
// lie so that one shift and one mask put sign and magnitude where bf16 has sign, exponent and mantissa (the
// fourth takes three).  Read as bf16 that is value * 2^-126, subnormals included, so one multiplication by the block's
// scale * 2^126 finishes a pair: 15 instructions for eight weights, where nibbles in GGUF order take 20.
// Scales [ceil(K / 256)][rows][8]: the biased exponent of that factor, 0 past the end of K.
//
// MXFP4 as the reference's model servers load it: docs/muse/muse-glimmer.md:112.
#include "../comm/sym.cuh"
#include "tc05.cuh"

using namespace b200;
using namespace b200::tc;

namespace {

constexpr int kM = 128, kN = 64, kK = 256;           // weight rows per tile, tokens per tile, K per stage
constexpr int kRaw = 6, kOps = 3;                    // packed stages; operand stages (tensor memory) and row stages (shared memory)
constexpr int kRawBytes = kM * kK / 2, kXBytes = kN * kK * 2;
constexpr int kRoles = 4, kExpWarps = 8, kThreads = 32 * (kRoles + 2 * kExpWarps);      // expansion warps of a group
constexpr int kMaxBlocks = 1024;                     // 64-row blocks with live rows
constexpr size_t kSmem = 1024 + kOps * kXBytes + kRaw * kRawBytes + kMaxBlocks * 8 + (2 * kRaw + 3 * kOps + 4) * 8 + 16;
static_assert(kSmem <= 227 * 1024, "shared memory budget");
static_assert(kRaw % 2 == 0, "a slot of the packed ring stays with one group: its parity then tells the stage (see QTraits in qgemm_tc05.cu)");

struct MoeQArgs {
  const uint2* scales;       // [ceil(K / 256)][groups * N]
  const int* counts;         // [groups] rows received
  int groups, group_rows, N, K, ldo;
  __nv_bfloat16* out;        // gate / up: [groups * group_rows][ldo], N / 2 columns of silu(gate) * up
  const int* meta;           // down: row m is token meta[2m + 1]
  const float* gate_w;       //       and is added times gate_w[m]
  float* y;                  //       into y [tokens][ldo]
  int* status;
};

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// One block of 32: four words -> sixteen bf16 pairs.
__device__ __forceinline__ void expand_mxfp4(const uint4 q, uint32_t scale, uint32_t* out) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t v = w[i];
    out[4 * i + 0] = mul_bf16x2(v & 0x81C081C0u, scale);
    out[4 * i + 1] = mul_bf16x2((v << 3) & 0x81C081C0u, scale);
    out[4 * i + 2] = mul_bf16x2((v << 6) & 0x81C081C0u, scale);
    out[4 * i + 3] = mul_bf16x2(((v >> 4) & 0x00C000C0u) | ((v >> 6) & 0x01000100u) | ((v << 2) & 0x80008000u), scale);
  }
}

template <bool DOWN>
__global__ void __launch_bounds__(kThreads, 1) moe_qgemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                                const MoeQArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sX = smem;
  uint8_t* sR = sX + kOps * kXBytes;
  int2* live = (int2*)(sR + kRaw * kRawBytes);       // (first row, live rows) of every block of 64
  uint64_t* raw_full = (uint64_t*)(live + kMaxBlocks);
  uint64_t* raw_empty = raw_full + kRaw;
  uint64_t* x_full = raw_empty + kRaw;
  uint64_t* a_full = x_full + kOps;
  uint64_t* done = a_full + kOps;                    // the stage's MMAs have finished: its row and operand slots are free
  uint64_t* tfull = done + kOps;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_holder = (uint32_t*)(tempty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);
  __shared__ int s_blocks;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_st = (a.K + kK - 1) / kK, tiles = (a.N + kM - 1) / kM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRaw; s++) {
      mbar_init(smem_u32(raw_full + s), 1);
      mbar_init(smem_u32(raw_empty + s), kExpWarps);
    }
    for (int s = 0; s < kOps; s++) {
      mbar_init(smem_u32(x_full + s), 1);
      mbar_init(smem_u32(a_full + s), kExpWarps);
      mbar_init(smem_u32(done + s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(smem_u32(tfull + s), 1);
      mbar_init(smem_u32(tempty + s), kExpWarps);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // tensor-memory columns: accumulators at +0 and +64, operand stages at +128, +256 and +384
  pdl_trigger();
  pdl_wait();                                        // the counts and rows are final
  if (warp == 2) {                                   // list the blocks: a lane per expert, places by a warp scan
    int n = 0;
    for (int g0 = 0; g0 < a.groups; g0 += 32) {
      const int g = g0 + lane, cnt = g < a.groups ? min(a.counts[g], a.group_rows) : 0, k = (cnt + kN - 1) / kN;
      int at = k;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
      }
      for (int r = 0; r < k; r++)
        if (n + at - k + r < kMaxBlocks) live[n + at - k + r] = make_int2(g * a.group_rows + r * kN, min(kN, cnt - r * kN));
      n += __shfl_sync(0xffffffffu, at, 31);
    }
    if (lane == 0) s_blocks = min(n, kMaxBlocks);
  }
  __syncthreads();
  const int n_items = s_blocks * tiles;              // columns fastest: the CTAs sweep one expert's weights at a time

  if (warp == 0) {
    uint32_t s = 0, ph = 1;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int b = item / tiles, row = live[b].x / a.group_rows * a.N + (item - b * tiles) * kM;
      for (int i = 0; i < n_st; i++) {
        if (!mbar_wait_warp(smem_u32(raw_empty + s), ph, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(smem_u32(raw_full + s), kRawBytes);
          tma_load_2d(smem_u32(sR) + s * kRawBytes, &tmW, smem_u32(raw_full + s), i * (kK / 2), row);
        }
        __syncwarp();
        if (++s == kRaw) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 2) {
    uint32_t s = 0, ph = 1;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int2 blk = live[item / tiles];
      const int boxes = blk.y > 32 ? 2 : 1;
      for (int i = 0; i < n_st; i++) {
        if (!mbar_wait_warp(smem_u32(done + s), ph, abort_flag)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(smem_u32(x_full + s), boxes * (kXBytes / 2));
          const uint32_t dst = smem_u32(sX) + s * kXBytes, bar = smem_u32(x_full + s);
          for (int h = 0; h < boxes; h++)
#pragma unroll
            for (int u = 0; u < 4; u++) tma_load_2d(dst + u * (kN * 128) + h * 4096, &tmX, bar, i * kK + u * 64, blk.x + h * 32);
        }
        __syncwarp();
        if (++s == kOps) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint64_t bd0 = smem_desc_sw128(smem_u32(sX));
    uint32_t s = 0, ph = 0, tcount = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, tcount++) {
      const int rows = live[item / tiles].y;
      const uint32_t idesc = rows <= 16 ? idesc_bf16(kM, 16) : rows <= 32 ? idesc_bf16(kM, 32) : idesc_bf16(kM, 64);
      const uint32_t acc = tcount & 1;
      if (!mbar_wait_warp(smem_u32(tempty + acc), ((tcount >> 1) & 1) ^ 1, abort_flag)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * kN;
      uint32_t add = 0;
      for (int i = 0; i < n_st; i++) {
        if (!mbar_wait_warp(smem_u32(a_full + s), ph, abort_flag) || !mbar_wait_warp(smem_u32(x_full + s), ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_tmem = tmem_base + 128 + s * 128;
        const uint64_t bd = bd0 + s * (kXBytes >> 4);
        if (elect_one()) {
#pragma unroll
          for (int m = 0; m < 16; m++)
            umma_ts(d_tmem, a_tmem + m * 8, bd + (m >> 2) * ((kN * 128) >> 4) + (m & 3) * 2, idesc, m == 0 ? add : 1u);
          umma_commit(smem_u32(done + s));
        }
        __syncwarp();
        add = 1;
        if (++s == kOps) { s = 0; ph ^= 1; }
      }
      if (elect_one()) umma_commit(smem_u32(tfull + acc));      // released even after a failed wait; the flag says why
      __syncwarp();
    }
  } else if (warp >= kRoles) {
    const int ew = warp - kRoles, q = warp & 3, half = (ew >> 2) & 1, group = ew >> 3;      // lane quarter; K blocks 2 half, 2 half + 1 of the group's stages
    const int row = q * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const int w_rows = a.groups * a.N;
    uint32_t ecount = 0;
    uint32_t g = 0, rs = 0, rph = 0, s = 0, sph = 1;      // stages so far and their slots
    bool ok = true;

    auto epilogue = [&](int item, uint32_t ec) {
      const int b = item / tiles, n = (item - b * tiles) * kM + row;
      const int2 blk = live[b];
      const uint32_t acc = ec & 1;
      bool tok = mbar_wait(smem_u32(tfull + acc), (ec >> 1) & 1, abort_flag);
      tok = __all_sync(0xffffffffu, tok && !*abort_flag);
      if (!tok) { ok = false; return; }
      tc_fence_after();
      const int t0 = half * 32;                      // this warp's 32 of the 64 rows
      if (t0 < blk.y) {
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_addr + acc * kN + (uint32_t)t0, v);
        tmem_ld_wait();
        if constexpr (!DOWN) {
          // weight rows are (gate, up) pairs in adjacent lanes; the even lane finishes the even rows, the odd lane the odd ones
          const bool odd = lane & 1;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float va = __uint_as_float(v[j]), vb = __uint_as_float(v[j + 1]);
            const float pa = __shfl_xor_sync(0xffffffffu, va, 1), pb = __shfl_xor_sync(0xffffffffu, vb, 1);
            const float gate = odd ? pb : va, up = odd ? vb : pa;
            const int t = t0 + j + (odd ? 1 : 0);
            if (n < a.N && t < blk.y) a.out[(size_t)(blk.x + t) * a.ldo + (n >> 1)] = __float2bfloat16(silu(gate) * up);
          }
        } else {
          // 4 x 4 patches transposed inside each lane quad: a lane then adds four consecutive columns of ONE row
          const int lq = lane & 3, nq = n & ~3;
#pragma unroll
          for (int k4 = 0; k4 < 8; k4++) {
            float c[4] = {__uint_as_float(v[4 * k4]), __uint_as_float(v[4 * k4 + 1]), __uint_as_float(v[4 * k4 + 2]), __uint_as_float(v[4 * k4 + 3])};
            transpose_quad(c, lq);
            const int t = t0 + 4 * k4 + lq;
            if (t >= blk.y || nq >= a.N) continue;
            const int m = blk.x + t;
            const float w = a.gate_w[m];
            asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(a.y + (size_t)a.meta[2 * m + 1] * a.ldo + nq),
                         "f"(c[0] * w), "f"(c[1] * w), "f"(c[2] * w), "f"(c[3] * w) : "memory");
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(tempty + acc));
    };

    int pending = -1;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int b = item / tiles, n = (item - b * tiles) * kM + row;
      // rows past the expert's last are the next one's and past the last expert none: they multiply by 0 and are not written
      const uint32_t* sp = (const uint32_t*)(a.scales + live[b].x / a.group_rows * a.N + n) + half;
      const size_t step = (size_t)w_rows * 2;
      const int first = (int)((g ^ group) & 1);            // this group's first stage of the item
      uint32_t sc = n < a.N && first < n_st ? sp[first * step] : 0u;
      for (int i = 0; i < n_st; i++, g++) {
        if (!((g ^ group) & 1)) {
          const uint32_t sc_next = n < a.N && i + 2 < n_st ? sp[(i + 2) * step] : 0u;      // its next stage's, latency hidden
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(raw_full + rs), rph, abort_flag));
          if (!ok) break;
          const uint8_t* tile = sR + rs * kRawBytes + row * 128;
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int kb = 2 * half + u;
            uint32_t r[32];
            expand_mxfp4(*(const uint4*)(tile + (((2 * kb) ^ (row & 7)) << 4)), ((sc >> (16 * u)) & 0xFFu) * 0x00800080u, r);
            expand_mxfp4(*(const uint4*)(tile + (((2 * kb + 1) ^ (row & 7)) << 4)), ((sc >> (16 * u + 8)) & 0xFFu) * 0x00800080u, r + 16);
            if (u == 0) {      // the first values are in registers: only now does this warp need the operand slot
              ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(done + s), sph, abort_flag));
              if (!ok) break;
              tc_fence_after();
            } else {           // everything this warp needs from the packed stage has been read
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(raw_empty + rs));
              tmem_st_wait();  // the first store must have left the registers it reads: they are reused
            }
            tmem_st32(tmem_base + lane_addr + 128 + s * 128 + kb * 32, r);
          }
          if (!ok) break;
          sc = sc_next;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(a_full + s));
          if (pending >= 0) {    // the MMA warp has a stage of the new item queued: finish the old item now
            epilogue(pending, ecount++);
            pending = -1;
          }
        }
        if (++rs == kRaw) { rs = 0; rph ^= 1; }
        if (++s == kOps) { s = 0; sph ^= 1; }
      }
      if (group == 0) {
        if (pending >= 0 && ok) epilogue(pending, ecount++);      // the new item had no stage of this group's
        pending = item;
      }
    }
    if (pending >= 0 && ok) epilogue(pending, ecount++);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
  if (threadIdx.x == 0 && *abort_flag && a.status) atomicExch(a.status, (int)B200_ERR_TIMEOUT_MMA);
}

template <bool DOWN>
int launch(const CUtensorMap& tw, const CUtensorMap& tx, const MoeQArgs& a, cudaStream_t st) {
  auto kern = moe_qgemm_kernel<DOWN>;
  static int sms = 0;
  if (!sms) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return (int)e;
    sms = n > 0 ? n : 148;
  }
  return launch_pdl(kern, dim3(sms), dim3(kThreads), kSmem, st, tw, tx, a);
}

}  // namespace

// One rank.  w [groups * N][K / 2] and scales [ceil(K / 256)][groups * N][8] as packed by pack_mxfp4_wide; x [groups * group_rows][K] bf16 holds
// the rows each expert received (counts [groups], device memory; at most live_rows in all).  Either out_bf16 (rows of w are (gate_0, up_0, gate_1, ...):
// [groups * group_rows][ldo] gets silu(gate) * up, N / 2 columns), or y: row m, times gate_w[m], is added into row meta[2m + 1] of the fp32
// tensor y [*][ldo], N columns.
B200_API int b200_moe_qgemm(const void* w, const void* scales, const void* x, int groups, int group_rows, int N, int K, const int* counts,
                            long live_rows, void* out_bf16, float* y, int ldo, const int* meta, const float* gate_w, int* status, cudaStream_t st) {
  if (groups < 1 || group_rows < kN || group_rows % kN || N < 4 || N % 4 || K < 32 || K % 32 || !w || !scales || !x || !counts) return B200_ERR_BAD_ARG;
  if (live_rows < 1 || live_rows / kN + groups > kMaxBlocks) return B200_ERR_BAD_ARG;      // every block fits the list
  if ((out_bf16 != nullptr) == (y != nullptr) || (y && (!meta || !gate_w || ldo % 4 || ((uintptr_t)y & 15))) || ((uintptr_t)scales & 7)) return B200_ERR_BAD_ARG;
  CUtensorMap tw, tx;
  int rc = make_tmap_2d(&tw, w, 1, (uint64_t)groups * N, (uint64_t)K / 2, (uint64_t)K / 2, kM, kK / 2, true);
  if (rc) return rc;
  rc = make_tmap_2d(&tx, x, 2, (uint64_t)groups * group_rows, (uint64_t)K, (uint64_t)K * 2, 32, 64, true);
  if (rc) return rc;
  MoeQArgs a = {};
  a.scales = (const uint2*)scales; a.counts = counts; a.groups = groups; a.group_rows = group_rows; a.N = N; a.K = K; a.ldo = ldo;
  a.out = (__nv_bfloat16*)out_bf16; a.meta = meta; a.gate_w = gate_w; a.y = y; a.status = status;
  return y ? launch<true>(tw, tx, a, st) : launch<false>(tw, tx, a, st);
}
