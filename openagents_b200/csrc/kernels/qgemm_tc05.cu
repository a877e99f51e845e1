// Quantized-weight GEMM for decode batches and short prompts (64 or 128 tokens per tile) on tcgen05 with the
// dequantization inside the pipeline:
//     Y[t][n] (+)= sum_k X[t][k] * W[n][k],   W in Q4_K-R or Q6_K-R (row-major packed), X bf16.
// The packed weights are read from HBM exactly once, in their 4.5- or 6.6-bit form; nothing keeps a
// bf16 copy of them.
//
// The weight tile is the MMA's M operand (128 weight rows), the tokens are its N operand, so a
// decode batch fills the 128-lane accumulator without padding.  A persistent CTA (one per SM) walks
// work items (128-row tile, K split) with a ring of stages of one superblock (256 of K) each:
//   warp 0      one thread: TMA loads of the raw packed superblocks (128 rows x 144 / 208 bytes)
//   warp 1      one thread: tcgen05.mma, TS form: the expanded weights are the A operand in TENSOR
//               MEMORY, the activations the B operand in shared memory; owns the allocation
//   warp 2      one thread: TMA loads of the activation tiles (from L2; they are a few hundred KB)
//   warps 4-19  expansion, two groups of eight that take stages in turn: a thread owns one weight row (= one
//               tensor-memory lane) and two 64-wide K blocks of its group's stages: one mask puts two adjacent 4-bit values into the mantissas of
//               a bf16 pair, one subtraction and one fma apply the sub-block scale and offset, and
//               tcgen05.st writes the 64 values where the MMA reads them, with no shared-memory round
//               trip, no swizzle arithmetic and no proxy fence.  The first group runs the
//               epilogue of item i after it has expanded its first stage of item i + 1 (two accumulators).
// What bounds it is the expansion: 2 instructions per weight on the issue slots of the SM, beside what a warp spends per stage on
// barriers, addresses and scales.  The MMAs are not in the way: 128 x 64 x 16 from tensor memory retires every 32 cycles
// (measured, one CTA per SM; 18 at N = 32), 512 a stage.  For that the warp that issues them has to walk its loop as a whole, one
// elected lane issuing: the descriptors then stay in uniform registers.  From a loop inside `if (lane == 0)` the
// same instruction went out every 85 cycles and bounded the kernel.  Measured, 28672 x 4096 Q4_K, 16 tokens, a launch in a graph:
// 34.4 us with eight expansion warps and that loop, 31.1 with the uniform one, 30.8 with sixteen warps of one K block each per
// stage, 27.9 with the two groups (half the per-stage work per weight); 20 without expanding, which is 0.5 of the copy
// bandwidth and the 1.5 waves of 224 tiles.
// Stages hand over through mbarriers; every wait is bounded and reports through `status`.
//
// Epilogues: plain store (fp32 and/or bf16), accumulation with vector `red` (K may be split; under tensor
// parallelism the row-parallel projections accumulate this rank's partial result that way and the RMSNorm
// that follows all-reduces it) and SwiGLU over interleaved (gate, up) rows.
//
// GEMM-shaped reference math: apps/openagents.com/workers/api/src/cs336-a2-benchmark-workload.ts:251-292;
// the quantized formats are the ones the reference serves (docs/muse/muse-glimmer.md:112).
#include "tc05.cuh"

using namespace b200;
using namespace b200::tc;

enum { QW_Q4KR = 0, QW_Q6KR = 1 };
enum { QEPI_STORE = 0, QEPI_ADD = 1, QEPI_SWIGLU = 2 };

struct QGemmArgs {
  const __half* w2;      // Q6_K-R: fp16 d per (row, superblock); unused for Q4_K-R
  float* out_f32;        // [T][ldo] (STORE / ADD), or null
  __nv_bfloat16* out_bf16;   // [T][ldo] (STORE) or [T][ldo] with N / 2 live columns (SWIGLU), or null
  const float* bias;     // [N] in the row order of W, or null (applied by K split 0)
  int ldo, T, N, K;
  int x_box;             // tokens of one TMA box: T rounded up to 8 (rows beyond T cost the TMA unit time; the tile's other columns are not read back)
  int epi;
  int splits, sb_per_split, n_items;
  int* status;
};

__device__ __forceinline__ uint32_t bf162_as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __nv_bfloat162 u32_as_bf162(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }

__device__ __forceinline__ float low_half(uint32_t t) { return __uint_as_float(t << 16); }
__device__ __forceinline__ float high_half(uint32_t t) { return __uint_as_float(t & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) { return bf162_as_u32(__floats2bfloat162_rn(lo, hi)); }

// Q4_K-R: one 32-element sub-block (4 words, word w = elements 8w .. 8w + 7, element i at bit
// 4 (i / 2) + 16 (i % 2)) -> 16 words of bf16 pairs.  The nibble sits in the mantissa of bf16 16.0 (one shift and
// one lop3 for two weights); (16 + q) - 24 = q - 8 is exact, and value = a * (q - 8) + c with c = 8 a - min keeps
// the constant small (the sub-block's range is roughly centred on it), so rounding a and c to bf16 costs no more
// than rounding the weight itself does.
//
// WHOLE: the weight itself in 32 bits, rounded to bf16 once: the value that dequant.cu makes, bit for bit (`scale` and `least` are the
// sub-block's 32-bit scale and min, `A2` and `C2` unused).
template <bool WHOLE>
__device__ __forceinline__ void expand_q4k(__nv_bfloat162 A2, __nv_bfloat162 C2, float scale, float least, const uint4 q, uint32_t* out) {
  const __nv_bfloat162 off = __halves2bfloat162(__float2bfloat16(WHOLE ? 16.f : 24.f), __float2bfloat16(WHOLE ? 16.f : 24.f));
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t v = w[i];
    const uint32_t t0 = ((v << 3) & 0x00780078u) | 0x41804180u;
    const uint32_t t1 = ((v >> 1) & 0x00780078u) | 0x41804180u;
    const uint32_t t2 = ((v >> 5) & 0x00780078u) | 0x41804180u;
    const uint32_t t3 = ((v >> 9) & 0x00780078u) | 0x41804180u;
    auto finish = [&](uint32_t t) {
      const __nv_bfloat162 x = __hsub2(u32_as_bf162(t), off);
      if constexpr (!WHOLE) return bf162_as_u32(__hfma2(x, A2, C2));
      const uint32_t u = bf162_as_u32(x);
      return pack2(fmaf(scale, low_half(u), -least), fmaf(scale, high_half(u), -least));
    };
    out[4 * i + 0] = finish(t0);
    out[4 * i + 1] = finish(t1);
    out[4 * i + 2] = finish(t2);
    out[4 * i + 3] = finish(t3);
  }
}

// Q6_K-R: 6-bit value = nibble | two high bits; (64 + q) - 96 = q - 32 is exact in bf16.  `s0` and `s1` are the scales of the
// sub-block's first and second 16 elements, rounded to bf16 here unless WHOLE.
template <bool WHOLE>
__device__ __forceinline__ void expand_q6k(const uint4 lo, const uint2 tw, float s0, float s1, uint32_t* out) {
  const __nv_bfloat162 sv = __floats2bfloat162_rn(s0, s1);
  const __nv_bfloat162 off = __halves2bfloat162(__float2bfloat16(96.f), __float2bfloat16(96.f));
  const uint32_t w[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t v = w[i];
    const uint32_t T = (i < 2 ? tw.x : tw.y) >> (4 * (i & 1));
    const __nv_bfloat162 S2 = i < 2 ? __halves2bfloat162(sv.x, sv.x) : __halves2bfloat162(sv.y, sv.y);
    const float scale = i < 2 ? s0 : s1;
    auto finish = [&](uint32_t q) {
      const __nv_bfloat162 x = __hsub2(u32_as_bf162((q << 1) | 0x42804280u), off);
      if constexpr (!WHOLE) return bf162_as_u32(__hmul2(x, S2));
      const uint32_t u = bf162_as_u32(x);
      return pack2(scale * low_half(u), scale * high_half(u));
    };
    const uint32_t q0 = (v & 0x000F000Fu) | ((T & 0x00030003u) << 4);
    const uint32_t q1 = ((v >> 4) & 0x000F000Fu) | (((T >> 2) & 0x00030003u) << 4);
    const uint32_t q2 = ((v >> 8) & 0x000F000Fu) | (((T >> 8) & 0x00030003u) << 4);
    const uint32_t q3 = ((v >> 12) & 0x000F000Fu) | (((T >> 10) & 0x00030003u) << 4);
    out[4 * i + 0] = finish(q0);
    out[4 * i + 1] = finish(q1);
    out[4 * i + 2] = finish(q2);
    out[4 * i + 3] = finish(q3);
  }
}

constexpr int QBM = 128, QSB = 256;                // weight rows per tile, K per stage (tokens per tile: QBN, 64 or 128)
constexpr int kRoleWarps = 4;                      // raw loads, MMA, activation loads, one idle (keeps warp % 4 = lane quarter)
constexpr int kDqWarps = 8;                        // expansion warps of a group: lane quarter = warp & 3, K half of the stage
constexpr int kDqGroups = 2;                       // groups take stages in turn
constexpr int kQThreads = 32 * (kRoleWarps + kDqGroups * kDqWarps);
// Every CTA walks the K range of its item from a different starting superblock (rotated by the CTA index): at any
// moment the SMs then read different slices of the activations, instead of all of them pulling the same few L2 lines.
__device__ __forceinline__ int rot_sb(int sb0, int sb1, int i) { const int n = sb1 - sb0; return sb0 + (i + (int)blockIdx.x) % n; }

// RS packed stages in shared memory; kAS operand stages in tensor memory and as many activation stages (four 64-wide K blocks) in
// shared memory.  Two accumulators of QBN columns and the operands of 128 fill the 512 columns.
template <int WT, int QBN> struct QTraits {
  static constexpr int RAWB = WT == QW_Q4KR ? 144 : 208;
  static constexpr int RS = WT == QW_Q4KR ? (QBN == 64 ? 6 : 5) : (QBN == 64 ? 4 : 3);
  static constexpr int kAS = QBN == 64 ? 3 : 2, kXStage = 4 * QBN * 64 * 2;
  // A group may ask for the bytes of stage g only when those of stage g - RS, in the same slot, are known to have landed: the barrier's
  // parity says no more than that.  With an even RS the group read that stage itself; else the other group did, and what this one
  // knows is that the MMAs of stage g - kAS - 2 have finished (its last wait for an operand slot), g - RS among them from RS = kAS + 3 on.  Below that it
  // waits for its operand slot first, which stands for stage g - kAS.
  static constexpr bool kSlotFirst = RS % kDqGroups != 0 && RS < kAS + 3;
  static_assert(kDqGroups == 2 && RS >= kAS, "a stage's slots are known to be free and landed");
};

template <int WT, int QBN>
__global__ void __launch_bounds__(kQThreads, 1) qgemm_kernel(const __grid_constant__ CUtensorMap tmW,
                                                             const __grid_constant__ CUtensorMap tmX, const QGemmArgs a) {
  constexpr int RAWB = QTraits<WT, QBN>::RAWB, RS = QTraits<WT, QBN>::RS, kAS = QTraits<WT, QBN>::kAS, kXStage = QTraits<WT, QBN>::kXStage;
  constexpr int RAW_BYTES = QBM * RAWB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sX = smem;                               // kAS stages of activations, 128-byte swizzle
  uint8_t* sR = sX + kAS * kXStage;                 // RS raw packed stages
  uint64_t* bars = (uint64_t*)(sR + RS * RAW_BYTES);
  uint64_t* raw_full = bars;             // [RS]  TMA bytes landed
  uint64_t* raw_empty = raw_full + RS;   // [RS]  every expansion warp has read the stage
  uint64_t* x_full = raw_empty + RS;     // [kAS]
  uint64_t* a_full = x_full + kAS;       // [kAS] every expansion warp has written its part of the operand
  uint64_t* done = a_full + kAS;         // [kAS] the stage's MMAs have finished: its activation and operand slots are free
  uint64_t* tfull = done + kAS;          // [2]   accumulator complete
  uint64_t* tempty = tfull + 2;          // [2]   accumulator read back by every epilogue warp
  uint32_t* tmem_holder = (uint32_t*)(tempty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsb_total = a.K / QSB;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RS; s++) {
      mbar_init(smem_u32(raw_full + s), 1);
      mbar_init(smem_u32(raw_empty + s), kDqWarps);
    }
    for (int s = 0; s < kAS; s++) {
      mbar_init(smem_u32(x_full + s), 1);
      mbar_init(smem_u32(a_full + s), kDqWarps);
      mbar_init(smem_u32(done + s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(smem_u32(tfull + s), 1);
      mbar_init(smem_u32(tempty + s), kDqWarps);
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
  // tensor-memory columns: accumulators at +0 and +QBN, then operand stages of 128 columns (256 of K) each
  constexpr uint32_t kOpCol = 2 * QBN;
  // More than 64 tokens: the weights that the expansion for longer prompts gives.  In 32 bits a pair takes eight instructions in place of four (an 8B prompt of
  // 128 tokens takes 4.2 ms, 4.0 with scales in two bf16 parts, 8.3 through the expansion).
  constexpr bool kWhole = QBN == 128;
  pdl_trigger();

  if (warp == 0) {
    // The weights are not written by any kernel: this thread does not wait for the kernel before this one, so the
    // first stages stream in while that kernel is still finishing.
    if (lane == 0) {
      uint32_t g = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
        const int tile = item / a.splits, sp = item - tile * a.splits;
        const int sb0 = sp * a.sb_per_split, sb1 = min(nsb_total, sb0 + a.sb_per_split);
        for (int sb = sb0; sb < sb1; sb++, g++) {
          const uint32_t s = g % RS;
          if (!mbar_wait(smem_u32(raw_empty + s), ((g / RS) & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(smem_u32(raw_full + s), RAW_BYTES);
          tma_load_2d(smem_u32(sR + s * RAW_BYTES), &tmW, smem_u32(raw_full + s), rot_sb(sb0, sb1, sb - sb0) * RAWB, tile * QBM);
        }
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      pdl_wait();
      uint32_t g = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
        const int tile = item / a.splits, sp = item - tile * a.splits;
        const int sb0 = sp * a.sb_per_split, sb1 = min(nsb_total, sb0 + a.sb_per_split);
        for (int sb = sb0; sb < sb1; sb++, g++) {
          const uint32_t s = g % kAS;
          if (!mbar_wait(smem_u32(done + s), ((g / kAS) & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(smem_u32(x_full + s), 4 * a.x_box * 128);
          const int k0 = rot_sb(sb0, sb1, sb - sb0) * QSB;
          const uint32_t dst = smem_u32(sX + s * kXStage), bar = smem_u32(x_full + s);
#pragma unroll
          for (int u = 0; u < 4; u++) tma_load_2d(dst + u * (QBN * 128), &tmX, bar, k0 + u * 64, 0);
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop and one elected lane issues: the descriptors stay in uniform registers, where tcgen05.mma
    // wants them.
    constexpr uint32_t idesc = idesc_bf16(QBM, QBN);
    const uint64_t bd0 = smem_desc_sw128(smem_u32(sX));
    const uint32_t a_full0 = smem_u32(a_full), x_full0 = smem_u32(x_full), done0 = smem_u32(done);
    uint32_t s = 0, ph = 0, tcount = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x, tcount++) {
      const int sp = item % a.splits;
      const int n_st = min(nsb_total, (sp + 1) * a.sb_per_split) - sp * a.sb_per_split;
      const uint32_t acc = tcount & 1;
      if (!mbar_wait_warp(smem_u32(tempty + acc), ((tcount >> 1) & 1) ^ 1, abort_flag)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * QBN;
      uint32_t add = 0;
      for (int i = 0; i < n_st; i++) {
        if (!mbar_wait_warp(a_full0 + 8 * s, ph, abort_flag) || !mbar_wait_warp(x_full0 + 8 * s, ph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_tmem = tmem_base + kOpCol + s * 128;
        const uint64_t bd = bd0 + s * (kXStage >> 4);
        if (elect_one()) {
#pragma unroll
          for (int m = 0; m < 16; m++)     // K block m / 4 (8 KB apart in shared memory, 32 columns apart in tensor memory), K step m % 4
            umma_ts(d_tmem, a_tmem + (m >> 2) * 32 + (m & 3) * 8, bd + (m >> 2) * ((QBN * 128) >> 4) + (m & 3) * 2, idesc, m == 0 ? add : 1u);
          umma_commit(done0 + 8 * s);
        }
        __syncwarp();
        add = 1;
        if (++s == kAS) { s = 0; ph ^= 1; }
      }
      if (elect_one()) umma_commit(smem_u32(tfull + acc));      // released even after a failed wait; the flag says why
      __syncwarp();
    }
  } else if (warp >= kRoleWarps) {
    // ---- expansion + epilogue warps
    const int dw = warp - kRoleWarps, q = warp & 3, khalf = (dw >> 2) & 1, group = dw >> 3;      // lane quarter; K blocks 2 khalf, 2 khalf + 1 of the group's stages
    const int row = q * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    uint32_t g = 0, ecount = 0;
    bool ok = true;
    bool waited = false;

    // epilogue of the item with accumulator number `ec`: this warp takes its lane quarter and half of the token columns, 32 at a time
    auto epilogue = [&](int item, uint32_t ec) {
      const int tile = item / a.splits, sp = item - tile * a.splits;
      const uint32_t acc = ec & 1;
      bool tok = mbar_wait(smem_u32(tfull + acc), (ec >> 1) & 1, abort_flag);
      tok = __all_sync(0xffffffffu, tok && !*abort_flag);
      if (!tok) { ok = false; return; }
      tc_fence_after();
      if (!waited) {                      // first global write of this thread: the kernel before this one must be complete
        pdl_wait();
        waited = true;
      }
      const int n = tile * QBM + row;
      const bool live = n < a.N;
#pragma unroll 1
      for (int t0 = khalf * (QBN / 2); t0 < (khalf + 1) * (QBN / 2) && t0 < a.T; t0 += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_base + lane_addr + acc * QBN + (uint32_t)t0, v);
        tmem_ld_wait();
        if (a.epi == QEPI_SWIGLU) {
          // rows are (gate_i, up_i) pairs in adjacent lanes; the even lane finishes the even tokens, the odd lane the odd ones
          const float b = (a.bias && live) ? a.bias[n] : 0.f;
          const bool odd = lane & 1;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float va = __uint_as_float(v[j]) + b, vb = __uint_as_float(v[j + 1]) + b;
            const float pa = __shfl_xor_sync(0xffffffffu, va, 1), pb = __shfl_xor_sync(0xffffffffu, vb, 1);
            const float gate = odd ? pb : va, up = odd ? vb : pa;
            const int t = t0 + j + (odd ? 1 : 0);
            if (live && t < a.T) a.out_bf16[(size_t)t * a.ldo + (n >> 1)] = __float2bfloat16(silu(gate) * up);
          }
        } else {
          // Transpose 4 x 4 patches inside each lane quad (four shuffles per four tokens): a lane then holds, for ONE token,
          // four consecutive output columns, so that a warp instruction moves four rows of 128 contiguous bytes: vector
          // stores, vector reductions into L2, full packets over NVLink.
          float b = 0.f;
          if (a.bias && live && sp == 0) b = a.bias[n];
          const int lq = lane & 3, nq = tile * QBM + q * 32 + (lane & ~3);      // first of this lane's four columns
          const bool quad_live = nq + 3 < a.N && (a.ldo & 3) == 0;
#pragma unroll
          for (int k4 = 0; k4 < 8; k4++) {
            float c[4] = {__uint_as_float(v[4 * k4]) + b, __uint_as_float(v[4 * k4 + 1]) + b, __uint_as_float(v[4 * k4 + 2]) + b,
                          __uint_as_float(v[4 * k4 + 3]) + b};
            transpose_quad(c, lq);
            const int t = t0 + 4 * k4 + lq;          // c[0..3] = columns nq .. nq + 3 of token t
            if (t >= a.T) continue;
            const size_t idx = (size_t)t * a.ldo + nq;
            if (quad_live) {
              const float4 o = make_float4(c[0], c[1], c[2], c[3]);
              if (a.epi == QEPI_ADD) {
                asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(a.out_f32 + idx), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
              } else {
                if (a.out_f32) *(float4*)(a.out_f32 + idx) = o;
                if (a.out_bf16) *(uint2*)(a.out_bf16 + idx) = make_uint2(pack2(o.x, o.y), pack2(o.z, o.w));
              }
            } else {
#pragma unroll
              for (int e = 0; e < 4; e++) {
                if (nq + e >= a.N) break;
                if (a.epi == QEPI_ADD) {
                  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(a.out_f32 + idx + e), "f"(c[e]) : "memory");
                } else {
                  if (a.out_f32) a.out_f32[idx + e] = c[e];
                  if (a.out_bf16) a.out_bf16[idx + e] = __float2bfloat16(c[e]);
                }
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(tempty + acc));
    };

    int pending = -1;
    for (int item = blockIdx.x; item < a.n_items && ok; item += gridDim.x) {
      const int tile = item / a.splits, sp = item - tile * a.splits;
      const int sb0 = sp * a.sb_per_split, sb1 = min(nsb_total, sb0 + a.sb_per_split);
      const int n = tile * QBM + row;
      [[maybe_unused]] float d6 = 0.f;
      if constexpr (WT == QW_Q6KR) {
        const int first = (int)((g ^ group) & 1);          // this group's first stage of the item
        d6 = n < a.N && sb0 + first < sb1 ? __half2float(a.w2[(size_t)n * nsb_total + rot_sb(sb0, sb1, first)]) : 0.f;
      }
      for (int sb = sb0; sb < sb1 && ok; sb++, g++) {
        if ((g ^ group) & 1) continue;                     // the other group's stage
        [[maybe_unused]] float d6_next = 0.f;
        if constexpr (WT == QW_Q6KR) {      // the next stage's d, fetched a stage ahead so that its latency is hidden
          if (n < a.N && sb + 2 < sb1) d6_next = __half2float(a.w2[(size_t)n * nsb_total + rot_sb(sb0, sb1, sb + 2 - sb0)]);
        }
        const uint32_t rs = g % RS, s = g % kAS;
        if constexpr (QTraits<WT, QBN>::kSlotFirst) {
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(done + s), ((g / kAS) & 1) ^ 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
        }
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(raw_full + rs), (g / RS) & 1, abort_flag));
        if (!ok) break;
        const uint8_t* rowp = sR + rs * RAW_BYTES + row * RAWB;
        [[maybe_unused]] uint4 hdr;
        [[maybe_unused]] float d4 = 0.f, dmin4 = 0.f;
        if constexpr (WT == QW_Q4KR) {
          hdr = *(const uint4*)rowp;
          const __half2 dd = *reinterpret_cast<const __half2*>(&hdr.x);
          d4 = __low2float(dd);
          dmin4 = __high2float(dd);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int kbu = 2 * khalf + u;               // K block of the stage
          uint32_t r[32];
          if constexpr (WT == QW_Q4KR) {
            // sub-blocks 2 kbu and 2 kbu + 1: their 6-bit scale and min, byte-parallel
            uint32_t S, Mn;
            if (kbu < 2) {
              S = hdr.y & 0x3F3F3F3Fu;
              Mn = hdr.z & 0x3F3F3F3Fu;
            } else {
              S = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
              Mn = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int j = 2 * kbu + h, sh = 8 * (j & 3);
              const float av = d4 * (float)((S >> sh) & 0xFFu);
              const float least = dmin4 * (float)((Mn >> sh) & 0xFFu);
              const __nv_bfloat16 ab = __float2bfloat16(av);
              const __nv_bfloat16 cb = __float2bfloat16(8.f * __bfloat162float(ab) - least);
              expand_q4k<kWhole>(__halves2bfloat162(ab, ab), __halves2bfloat162(cb, cb), av, least, *(const uint4*)(rowp + 16 + j * 16), r + 16 * h);
            }
          } else {
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int j = 2 * kbu + h;
              const uint32_t scw = *(const uint16_t*)(rowp + 192 + 2 * j);
              expand_q6k<kWhole>(*(const uint4*)(rowp + j * 16), *(const uint2*)(rowp + 128 + j * 8), d6 * (float)(int8_t)(scw & 0xFF),
                                 d6 * (float)(int8_t)(scw >> 8), r + 16 * h);
            }
          }
          if (u == 0) {      // the first values are in registers: only now does this warp need the operand slot
            if constexpr (!QTraits<WT, QBN>::kSlotFirst) {
              ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(done + s), ((g / kAS) & 1) ^ 1, abort_flag));
              if (!ok) break;
              tc_fence_after();
            }
          } else {           // everything this warp needs from the raw stage has been read
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(raw_empty + rs));
            tmem_st_wait();  // the first store must have left the registers it reads: they are reused
          }
          tmem_st32(tmem_base + lane_addr + kOpCol + s * 128 + kbu * 32, r);
        }
        if (!ok) break;
        if constexpr (WT == QW_Q6KR) d6 = d6_next;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(a_full + s));
        if (pending >= 0) {     // the MMA thread has a stage of the new item queued: finish the old item now
          epilogue(pending, ecount++);
          pending = -1;
        }
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

static int q_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

template <int WT, int QBN>
static int launch_q(const void* w, const void* x, int ldx, QGemmArgs a, cudaStream_t st) {
  constexpr int RAWB = QTraits<WT, QBN>::RAWB, RS = QTraits<WT, QBN>::RS, kAS = QTraits<WT, QBN>::kAS, kXStage = QTraits<WT, QBN>::kXStage;
  constexpr size_t smem = 1024 + kAS * (size_t)kXStage + (size_t)RS * QBM * RAWB + (2 * RS + 3 * kAS + 4) * 8 + 16;
  static_assert(smem <= 227 * 1024, "shared memory budget");
  auto kern = qgemm_kernel<WT, QBN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  a.x_box = (a.T + 7) & ~7;
  CUtensorMap tw, tx;
  const int nsb = a.K / QSB;
  // packed rows as bytes: [N][nsb * RAWB], one box = 128 rows of one superblock; rows past N read as zeros (scale 0)
  int rc = make_tmap_2d(&tw, w, 1, (uint64_t)a.N, (uint64_t)nsb * RAWB, (uint64_t)nsb * RAWB, QBM, RAWB, false);
  if (rc) return rc;
  rc = make_tmap_2d(&tx, x, 2, (uint64_t)a.T, (uint64_t)a.K, (uint64_t)ldx * 2, a.x_box, 64, true);
  if (rc) return rc;
  const int grid = a.n_items < q_sm_count() ? a.n_items : q_sm_count();
  return launch_pdl(kern, dim3(grid), dim3(kQThreads), smem, st, tw, tx, a);
}

// wt: QW_Q4KR / QW_Q6KR; `w` the row-major packed plane the mat-vec kernels read as well ([N][K / 256][144 or 208
// bytes]), `w2` the fp16 d plane of Q6_K-R.  x: bf16 [T][ldx].  Any T: tokens are taken 128 at a time.
//   QEPI_STORE  out_f32 and/or out_bf16 [T][ldo] = result (+ bias)
//   QEPI_ADD    out_f32 [T][ldo] += result (+ bias); split_k > 1 allowed (0 = choose)
//   QEPI_SWIGLU rows of W are (gate_0, up_0, gate_1, ...); out_bf16 [T][ldo] gets silu(gate) * up, N / 2 columns
B200_API int b200_qgemm(int wt, const void* w, const void* w2, int N, int K, const void* x, int ldx, int T, float* out_f32,
                        void* out_bf16, int ldo, const float* bias, int epi, int split_k, int* status, cudaStream_t st) {
  if (K % QSB || (ldx % 8) || T < 1 || N < 1 || ((uintptr_t)w & 15) || ((uintptr_t)x & 15)) return B200_ERR_BAD_ARG;
  if (wt != QW_Q4KR && wt != QW_Q6KR) return B200_ERR_BAD_ARG;
  if (wt == QW_Q6KR && !w2) return B200_ERR_BAD_ARG;
  if (epi == QEPI_SWIGLU ? (!out_bf16 || (N & 1)) : epi == QEPI_ADD ? !out_f32 : (epi != QEPI_STORE || (!out_f32 && !out_bf16)))
    return B200_ERR_BAD_ARG;
  QGemmArgs a = {};
  a.w2 = (const __half*)w2; a.bias = bias; a.ldo = ldo; a.N = N; a.K = K; a.epi = epi; a.status = status;
  const int nsb = K / QSB, tiles = (N + QBM - 1) / QBM;
  int splits = 1;
  if (epi == QEPI_ADD) {
    if (split_k > 0) splits = split_k;
    else if (tiles < q_sm_count()) {
      splits = q_sm_count() / tiles;                 // fill the GPU once ...
      while (splits > 1 && nsb / splits < 2) splits--;  // ... with at least two stages per item
    }
    if (splits > nsb) splits = nsb;
  } else if (split_k > 1) {
    return B200_ERR_BAD_ARG;
  }
  a.sb_per_split = (nsb + splits - 1) / splits;
  a.splits = (nsb + a.sb_per_split - 1) / a.sb_per_split;     // no empty split
  a.n_items = tiles * a.splits;
  // Up to 64 tokens one narrow tile; else tiles of 128, so that the expansion, which bounds the kernel, serves twice as many.
  const bool wide = T > 64;
  for (int t0 = 0; t0 < T;) {
    a.T = min(T - t0, wide ? 128 : 64);
    a.out_f32 = out_f32 ? out_f32 + (size_t)t0 * ldo : nullptr;
    a.out_bf16 = out_bf16 ? (__nv_bfloat16*)out_bf16 + (size_t)t0 * ldo : nullptr;
    const void* xs = (const __nv_bfloat16*)x + (size_t)t0 * ldx;
    const int rc = wt == QW_Q4KR ? (wide ? launch_q<QW_Q4KR, 128>(w, xs, ldx, a, st) : launch_q<QW_Q4KR, 64>(w, xs, ldx, a, st))
                                 : (wide ? launch_q<QW_Q6KR, 128>(w, xs, ldx, a, st) : launch_q<QW_Q6KR, 64>(w, xs, ldx, a, st));
    if (rc) return rc;
    t0 += a.T;
  }
  return 0;
}
