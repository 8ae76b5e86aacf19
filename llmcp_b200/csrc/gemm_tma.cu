// Prefill GEMM (M > 1) on the fifth-generation tensor cores, operands fetched by TMA.
// Q8Matmul.cpp:143-289.
//
//   y[m, n] = act( chain_kb fma(float(dot_kb[m, n]), a_scale[m, kb] * w_scale[n, kb], acc) ),
//   dot_kb = sum of 32 int8 products.
//
// The per-block f32 chain is what bounds this GEMM: it runs on the CUDA cores, once per (row,
// column, 32-block), while the tensor core needs a fraction of that time for the block's dots.
// Two operand forms are implemented on one pipeline:
//   int8: the int8 planes the GEMV streams, tcgen05.mma kind::i8 (K = 32 = one quantisation block per
//         instruction), int32 dots, convert + multiply + fma per element in the epilogue;
//   f16 : the same integers held as f16 values (every integer up to 2048 is exact in f16), kind::f16
//         with f32 accumulation: a product is an integer below 2^14, a block's sum an integer below
//         2^19, both exact in f32, so the tensor core hands back float(dot) itself, bit for bit what
//         the conversion would give, and the epilogue is multiply + fma.  The price is operand planes
//         of twice the size in HBM and on the way from L2.
// Both forms multiply and add with two-lane f32x2 instructions (same roundings, half the instructions).
//
// What bounds it: the epilogue warps, 3 (int8) or 2 (f16) instructions' worth of lanes per (row, column, block), and
// the hand-off between them and the tensor core; the tensor pipe is under 10 % busy.  Loads from tensor memory,
// conversion, scales and fmas alone take 430 cycles per 128 x 128 x 32 block on an SM (346 without the conversion);
// handing over every block by itself made it 1000.  Two blocks per hand-off, descriptors advanced by an add, one
// elected lane per role (so that the compiler knows it is one) and a persistent grid (a tile's output is stored while
// the next tile's blocks are already multiplied) bring it to 800 (bf16 outputs): 1024 x 9216 x 2560 170 -> 130 us,
// 1024 x 2560 x 4096 87 -> 84, 1024 x 32 x 2560 42 -> 22.  Tensor-memory loads in fragment shapes, which need a third of the scale
// loads, measured 160 us (16x256b, a quarter of the read rate) and 150 us (16x128b, half).
//
// One CTA per SM (two of 320 threads for TN = 64, out of step with each other) takes 128 x TN output tiles in turn,
// 576 threads:
//   warp  0     one lane issues the TMA loads (cp.async.bulk.tensor, 128-byte swizzle, no
//               multicast): per stage a box of 128 (TN) rows x 128 bytes of K of each operand (four
//               int8 or two f16 quantisation blocks) and those blocks' f32 scales of the tile's rows
//               and columns (scale planes are block-major, [K/32][rows], so a box is consecutive
//               floats per block);
//   warp  1     one lane issues the MMAs, two blocks into a tensor-memory slot (f16: two K = 16
//               instructions per block, the first overwrites, the second accumulates), and commits the slot;
//   warps 2-17  epilogue (2-9 for TN = 64): tcgen05.ld a block (thread = row, 24 or 32 columns), hand the slot back
//               after its last block's load, then the arithmetic with the scales read from shared memory.
// Hand-offs are mbarriers; every wait is bounded (spin_limit polls) and a timed-out wait raises an
// abort flag that all roles observe, so a protocol error ends the kernel with an error code instead
// of hanging it; the loader then waits (bounded) for the copies it has in flight.  Tensor memory
// (512 columns, half of it for TN = 64) is allocated by warp 0 and always released.

#include <cuda.h>
#include <cuda_fp16.h>

#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "kernels.h"
#include "tc_common.cuh"

namespace llmcp_b200 {

namespace {

using namespace tc;

constexpr int kTileM = 128;
constexpr int kEpilogueWarp0 = 2;
constexpr int kOperandBytes = kTileM * 128; // 16 KB of activations per stage: rows of 128 bytes of K
constexpr int kMaxSlots = 4, kMaxStages = 6;
constexpr int kBarrierBytes = 256;

// Tiles of 128 rows by TN columns.  F16: operands are f16 values (64 per 128-byte row = 2 quantisation blocks per
// stage); otherwise int8 (128 per row = 4 blocks per stage).  Tensor memory holds kSlots slots of kSlotBlocks blocks'
// dots each; a slot is handed over as a whole.
template <bool F16, int TN> struct Form {
  static_assert(TN == 64 || TN == 96 || TN == 128, "tile widths with a tensor-memory plan");
  static constexpr int kCtas = TN == 64 ? 2 : 1;                    // CTAs per SM
  static constexpr int kEpilogueWarps = 16 / kCtas, kThreads = 32 * (kEpilogueWarp0 + kEpilogueWarps);
  static constexpr int kTmemColumns = 512 / kCtas;
  static constexpr int kSlotBlocks = 2;
  static constexpr int kSlots = kTmemColumns / (kSlotBlocks * TN);
  static constexpr int kWarpColumns = TN * 4 / kEpilogueWarps;      // columns per epilogue warp: 24 or 32
  static constexpr int kStages = TN == 64 ? 4 : TN >= 128 ? 5 : 6;
  static constexpr int kPiece = TN == 64 ? 16 : kWarpColumns;       // columns loaded from tensor memory at a time
  static constexpr int kStageBlocks = F16 ? 2 : 4;
  static constexpr int kStageK = kStageBlocks * 32;                 // elements of K per stage
  static constexpr int kOperandBytesB = TN * 128;
  static constexpr int kScaleBytesA = kStageBlocks * kTileM * 4;    // the rows' scales of a stage
  static constexpr int kScaleBytesB = kStageBlocks * TN * 4;        // the columns' scales
  static constexpr int kCopied = kOperandBytes + kOperandBytesB + kScaleBytesA + kScaleBytesB;
  static constexpr int kStageBytes = (kCopied + 1023) / 1024 * 1024;
  static constexpr size_t kSmemBytes = 1024 + kStages * kStageBytes + kBarrierBytes;
  static_assert(kSmemBytes * kCtas <= 226 * 1024 && kSlots >= 2 && kSlots <= kMaxSlots, "plan of a CTA");
};

// kind::f16: f16 x f16 -> f32, both operands K-major, M = 128, N = TN, K = 16 per instruction.
// kind::i8: s8 x s8 -> s32, both operands K-major, M = 128, N = TN, K = 32 per instruction.
template <int TN> struct Instruction {
  static constexpr uint32_t kF16 = (1u << 4) | ((TN >> 3) << 17) | ((kTileM >> 4) << 24);
  static constexpr uint32_t kI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((TN >> 3) << 17) | ((kTileM >> 4) << 24);
};

__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accumulate, uint32_t kInstructionF16) {
  asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p; }"
               :
               : "r"(tmem), "l"(a), "l"(b), "r"(kInstructionF16), "r"(accumulate), "r"(0u)
               : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t kInstructionI8) {
  asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p; }"
               :
               : "r"(tmem), "l"(a), "l"(b), "r"(kInstructionI8), "r"(0u), "r"(0u)
               : "memory");
}

// COLUMNS consecutive 32-bit columns of this thread's lane.
template <int COLUMNS> __device__ __forceinline__ void tmem_load_columns(uint32_t taddr, uint32_t (&r)[COLUMNS]) {
  if constexpr (COLUMNS >= 32)
    tmem_issue32(taddr, *reinterpret_cast<uint32_t(*)[32]>(r));
  else
    tmem_issue16(taddr, *reinterpret_cast<uint32_t(*)[16]>(r));
  if constexpr (COLUMNS % 16 == 8)
    tmem_issue8(taddr + COLUMNS - 8, *reinterpret_cast<uint32_t(*)[8]>(r + COLUMNS - 8));
  tmem_wait_loads_into(r);
}

// c += v * (a * w), two columns at a time; every lane of the pair rounds as the scalar instructions do.
__device__ __forceinline__ void fold2(float &c0, float &c1, float v0, float v1, float a, float w0, float w1) {
  asm("{ .reg .b64 s, w, v, c; mov.b64 s, {%2, %2}; mov.b64 w, {%3, %4}; mul.rn.f32x2 s, s, w; mov.b64 v, {%5, %6};\n"
      "mov.b64 c, {%0, %1}; fma.rn.f32x2 c, v, s, c; mov.b64 {%0, %1}, c; }"
      : "+f"(c0), "+f"(c1)
      : "f"(a), "f"(w0), "f"(w1), "f"(v0), "f"(v1));
}

// mbar_wait by a whole warp: all lanes get the same answer.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, uint32_t limit) {
  return __all_sync(0xffffffffu, mbar_poll<true>(smem_u32(bar), parity)) ||
         __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, limit));
}

// A position in a ring of `size` barriers and the parity of its current phase.
struct Ring {
  int at = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next(int size) {
    if (++at == size)
      at = 0, parity ^= 1;
  }
};

struct Barriers {
  uint64_t full[kMaxStages];     // stage landed in shared memory (one arrival + the copies' bytes)
  uint64_t empty[kMaxStages];    // stage no longer needed: MMA done (1) + every epilogue warp (scales read)
  uint64_t tfull[kMaxSlots];     // the slot's dot products are in tensor memory
  uint64_t tempty[kMaxSlots];    // the slot has been read by all epilogue warps
  uint64_t done;                 // the last commit of the MMA lane has arrived (see the end of its loop)
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(Barriers) <= kBarrierBytes, "barriers");

// fault (test hook): 1 = the loader announces the first stage's bytes but never issues its copies,
// so the barrier of that stage cannot complete and every wait behind it has to run out.
template <bool F16, bool DOTS, int TN>
__global__ void __launch_bounds__(Form<F16, TN>::kThreads, Form<F16, TN>::kCtas)
gemm_q8_tma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_as, const __grid_constant__ CUtensorMap map_bs, int M, int K,
                    int N, int tiles, int m_tiles, void *__restrict__ y, int y_dtype, int activation,
                    int32_t *__restrict__ dots_out, int *__restrict__ error_out, uint32_t spin_limit, int fault) {
  using F = Form<F16, TN>;
  constexpr int kStageBlocks = F::kStageBlocks, kStages = F::kStages, kSlots = F::kSlots, kSlotBlocks = F::kSlotBlocks;
  constexpr int kEpilogueWarps = F::kEpilogueWarps;
  constexpr int kColumns = F::kWarpColumns;
  extern __shared__ uint8_t raw_smem[];
  uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
  Barriers *bars = reinterpret_cast<Barriers *>(base + kStages * F::kStageBytes);
  volatile int *abort_flag = &bars->abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = K / kBlock;
  const int iters = (nb + kStageBlocks - 1) / kStageBlocks;

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1 + kEpilogueWarps);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&bars->tfull[i], 1);
      mbar_init(&bars->tempty[i], kEpilogueWarps);
    }
    mbar_init(&bars->done, 1);
    bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                 "r"(F::kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dependency_sync(); // barriers and tensor memory are set up; the operands belong to the kernel in front

  if (warp == 0) {
    // ---- loader ---------------------------------------------------------------------------
    if (elect_one()) {
      int use = 0; // stages requested so far, over all tiles of this CTA
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % m_tiles) * kTileM, n0 = (tile / m_tiles) * TN;
        for (int it = 0; it < iters; ++it, ++use) {
          const int s = use % kStages;
          if (use >= kStages && !mbar_wait(&bars->empty[s], (use / kStages - 1) & 1, abort_flag, spin_limit)) {
            ok = false;
            break;
          }
          uint8_t *stage = base + s * F::kStageBytes;
          mbar_expect_tx(&bars->full[s], F::kCopied);
          if (fault == 1 && use == 0)
            continue;
          const int k0 = it * F::kStageK, kb0 = it * kStageBlocks;
          tma_load_2d(stage, &map_a, k0, m0, &bars->full[s]);
          tma_load_2d(stage + kOperandBytes, &map_b, k0, n0, &bars->full[s]);
          tma_load_2d(stage + kOperandBytes + F::kOperandBytesB, &map_as, m0, kb0, &bars->full[s]);
          tma_load_2d(stage + kOperandBytes + F::kOperandBytesB + F::kScaleBytesA, &map_bs, n0, kb0, &bars->full[s]);
        }
      }
      // Leaving after a failed wait: the copies already requested still write into this CTA's
      // shared memory, so each of them gets one more bounded wait before the CTA may exit.
      if (*abort_flag) {
        for (int i = max(0, use - kStages); i < use; ++i)
          if (!(fault == 1 && i == 0))
            mbar_wait_quiet(&bars->full[i % kStages], (i / kStages) & 1, spin_limit);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issue ------------------------------------------------------------------------
    if (elect_one()) {
      Ring stages, slots;
      bool ok = true, reused = false; // reused: every slot has been filled once
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        for (int it = 0; it < iters && ok; ++it) {
          ok = mbar_wait(&bars->full[stages.at], stages.parity, abort_flag, spin_limit);
          if (!ok)
            break;
          tc_fence_after();
          const uint64_t a = operand_descriptor(smem_u32(base + stages.at * F::kStageBytes));
          const uint64_t b = operand_descriptor(smem_u32(base + stages.at * F::kStageBytes) + kOperandBytes);
          const int blocks = min(kStageBlocks, nb - it * kStageBlocks);
#pragma unroll
          for (int j = 0; j < kStageBlocks; ++j) { // descriptors advance in units of 16 bytes
            if (j >= blocks)
              break;
            if (j % kSlotBlocks == 0 && reused) {
              ok = mbar_wait(&bars->tempty[slots.at], slots.parity ^ 1, abort_flag, spin_limit);
              if (!ok)
                break;
              tc_fence_after();
            }
            const uint32_t d = tmem_base + (slots.at * kSlotBlocks + j % kSlotBlocks) * TN;
            if (F16) { // two K = 16 instructions per block: the first overwrites, the second accumulates
              mma_f16(d, a + j * 4, b + j * 4, 0u, Instruction<TN>::kF16);
              mma_f16(d, a + j * 4 + 2, b + j * 4 + 2, 1u, Instruction<TN>::kF16);
            } else {
              mma_i8(d, a + j * 2, b + j * 2, Instruction<TN>::kI8);
            }
            if (j % kSlotBlocks == kSlotBlocks - 1 || j == blocks - 1) {
              mma_commit(&bars->tfull[slots.at]);
              slots.next(kSlots);
              reused = reused || slots.at == 0;
            }
          }
          if (ok)
            mma_commit(&bars->empty[stages.at]);
          stages.next(kStages);
        }
      }
      // A commit's arrival is asynchronous, and nothing else waits for the last ones on `empty`: the
      // CTA must not end (and hand its shared memory to the next CTA on this SM, possibly of another
      // kernel with its barriers elsewhere) while an arrival is still on its way.  Commits arrive in
      // order, so seeing this one means all have.
      mma_commit(&bars->done);
      mbar_wait_quiet(&bars->done, 0, spin_limit);
    }
  } else {
    // ---- epilogue ---------------------------------------------------------------------------
    const int quarter = warp & 3;                                  // tensor-memory lanes 32 * quarter .. + 31 (fixed by the warp number)
    const int column0 = ((warp - kEpilogueWarp0) >> 2) * kColumns; // this warp's columns of the tile
    const int row = quarter * 32 + lane;
    const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + column0;
    Ring stages, slots;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int gm = (tile % m_tiles) * kTileM + row, gn0 = (tile / m_tiles) * TN + column0;
      float acc[kColumns];
#pragma unroll
      for (int c = 0; c < kColumns; ++c)
        acc[c] = 0.0f;
      bool ok = true;
      for (int it = 0; it < iters; ++it) {
        // The stage's scales arrived with the operands; observing the stage's own barrier (long
        // complete by now) is what makes the copied bytes visible to these loads.
        ok = warp_wait(&bars->full[stages.at], stages.parity, abort_flag, spin_limit);
        if (!ok) // the whole warp leaves together: the tensor-memory loads below are warp-wide
          break;
        const float *scales = reinterpret_cast<const float *>(base + stages.at * F::kStageBytes + kOperandBytes + F::kOperandBytesB);
        const int blocks = min(kStageBlocks, nb - it * kStageBlocks);
#pragma unroll
        for (int j = 0; j < kStageBlocks; ++j) {
          if (j >= blocks)
            break;
          if (j % kSlotBlocks == 0) {
            ok = warp_wait(&bars->tfull[slots.at], slots.parity, abort_flag, spin_limit);
            if (!ok)
              break;
            tc_fence_after();
          }
          const float a_scale = scales[j * kTileM + row];
          const float4 *w_scale = reinterpret_cast<const float4 *>(scales + kStageBlocks * kTileM + j * TN + column0);
          constexpr int kPiece = F::kPiece;
#pragma unroll
          for (int p = 0; p < kColumns; p += kPiece) {
            uint32_t raw[kPiece];
            tmem_load_columns<kPiece>(taddr0 + (slots.at * kSlotBlocks + j % kSlotBlocks) * TN + p, raw);
            if (p + kPiece == kColumns && (j % kSlotBlocks == kSlotBlocks - 1 || j == blocks - 1)) {
              // The slot is handed back before its last columns are folded in.
              tc_fence_before();
              __syncwarp();
              if (lane == 0)
                mbar_arrive(&bars->tempty[slots.at]);
              slots.next(kSlots);
            }
#pragma unroll
            for (int g = 0; g < kPiece / 4; ++g) {
              const float4 w = w_scale[p / 4 + g];
              float v[4];
#pragma unroll
              for (int u = 0; u < 4; ++u)
                v[u] = F16 ? __uint_as_float(raw[4 * g + u]) : __int2float_rn(static_cast<int>(raw[4 * g + u]));
              fold2(acc[p + 4 * g + 0], acc[p + 4 * g + 1], v[0], v[1], a_scale, w.x, w.y);
              fold2(acc[p + 4 * g + 2], acc[p + 4 * g + 3], v[2], v[3], a_scale, w.z, w.w);
              if (DOTS && gm < M) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                  if (gn0 + p + 4 * g + u < N)
                    dots_out[(static_cast<size_t>(gm) * N + gn0 + p + 4 * g + u) * nb + it * kStageBlocks + j] =
                        F16 ? __float2int_rn(v[u]) : static_cast<int>(raw[4 * g + u]);
              }
            }
          }
        }
        if (!ok)
          break;
        __syncwarp();
        if (lane == 0) // done with this stage's scales
          mbar_arrive(&bars->empty[stages.at]);
        stages.next(kStages);
      }
      if (!ok)
        break;
      if (gm < M) {
#pragma unroll
        for (int g = 0; g < kColumns / 8; ++g) {
          const int gn = gn0 + g * 8;
          if (gn < N) { // N is a multiple of 8, so a group of eight is entirely inside or outside
            float o[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              o[u] = apply_activation(acc[g * 8 + u], activation);
            if (y_dtype == kBF16) {
              uint32_t packed[4];
#pragma unroll
              for (int u = 0; u < 4; ++u)
                packed[u] = static_cast<uint32_t>(f32_to_bf16(o[2 * u])) | (static_cast<uint32_t>(f32_to_bf16(o[2 * u + 1])) << 16);
              *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(y) + static_cast<size_t>(gm) * N + gn) =
                  make_uint4(packed[0], packed[1], packed[2], packed[3]);
            } else {
              float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(y) + static_cast<size_t>(gm) * N + gn);
              dst[0] = make_float4(o[0], o[1], o[2], o[3]);
              dst[1] = make_float4(o[4], o[5], o[6], o[7]);
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(F::kTmemColumns) : "memory");
  }
  if (tid == 0 && bars->abort_flag && error_out)
    atomicExch(error_out, 1);
}

// int8 activations and their [M][K/32] scales -> f16 values [M][K] and block-major scales
// [K/32][ld] (ld = M rounded up to 4, the row pitch a tensor map needs).
__global__ void act_to_f16_kernel(const int8_t *__restrict__ aq, const float *__restrict__ as, int64_t M, int K, int64_t ld,
                                  __half *__restrict__ ah, float *__restrict__ ast) {
  grid_dependency_sync();
  const int64_t words = M * (K / 4);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int nb = K / kBlock;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < words; i += stride) {
    const uint32_t v = reinterpret_cast<const uint32_t *>(aq)[i];
    const __half2 lo = __halves2half2(__int2half_rn(static_cast<int8_t>(v & 0xff)), __int2half_rn(static_cast<int8_t>((v >> 8) & 0xff)));
    const __half2 hi = __halves2half2(__int2half_rn(static_cast<int8_t>((v >> 16) & 0xff)), __int2half_rn(static_cast<int8_t>(v >> 24)));
    reinterpret_cast<uint2 *>(ah)[i] = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
    if (i < M * nb) { // the first M * nb threads also move one scale each
      const int64_t m = i / nb, b = i % nb;
      ast[b * ld + m] = as[i];
    }
  }
}

// The weight planes of the same form, made once at load from the int8 / f16-scale planes.
__global__ void weights_to_f16_kernel(const int8_t *__restrict__ wq, const uint16_t *__restrict__ wd, int64_t N, int K,
                                      __half *__restrict__ wh, float *__restrict__ wst) {
  grid_dependency_sync();
  const int64_t words = N * (K / 4);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int nb = K / kBlock;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < words; i += stride) {
    const uint32_t v = reinterpret_cast<const uint32_t *>(wq)[i];
    const __half2 lo = __halves2half2(__int2half_rn(static_cast<int8_t>(v & 0xff)), __int2half_rn(static_cast<int8_t>((v >> 8) & 0xff)));
    const __half2 hi = __halves2half2(__int2half_rn(static_cast<int8_t>((v >> 16) & 0xff)), __int2half_rn(static_cast<int8_t>(v >> 24)));
    reinterpret_cast<uint2 *>(wh)[i] = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
    if (i < N * nb) {
      const int64_t n = i / nb, b = i % nb;
      wst[b * N + n] = f16_bits_to_f32(wd[i]);
    }
  }
}

struct GemmCall {
  const void *a;
  const float *ast;
  int M, K;
  const void *w;
  const float *wst;
  int N;
  void *y;
  int y_dtype, activation;
  int32_t *dots_out;
  int *error_flag;
  cudaStream_t stream;
  uint32_t spin_limit;
  int fault, sm_count;
};

template <bool F16, int TN> cudaError_t launch_tile(const GemmCall &c) {
  using F = Form<F16, TN>;
  const int nb = c.K / kBlock;
  CUtensorMap map_a, map_b, map_as, map_bs;
  if (!gemm_operand_map(&map_a, c.a, c.M, c.K, F16, kTileM) || !gemm_operand_map(&map_b, c.w, c.N, c.K, F16, TN) ||
      !gemm_scale_map(&map_as, c.ast, c.M, gemm_tc16_scale_pitch(c.M), nb, F::kStageBlocks, kTileM) ||
      !gemm_scale_map(&map_bs, c.wst, c.N, c.N, nb, F::kStageBlocks, TN))
    return cudaErrorNotSupported;
  auto kernel = c.dots_out ? gemm_q8_tma_kernel<F16, true, TN> : gemm_q8_tma_kernel<F16, false, TN>;
  if (cudaError_t e = opt_in_shared_memory(reinterpret_cast<const void *>(kernel), F::kSmemBytes); e != cudaSuccess)
    return e;
  const int m_tiles = (c.M + kTileM - 1) / kTileM;
  const int64_t tiles = static_cast<int64_t>(m_tiles) * ((c.N + TN - 1) / TN);
  if (tiles >= (1 << 30))
    return cudaErrorInvalidValue;
  launch_chained(kernel, dim3(static_cast<unsigned>(std::min<int64_t>(tiles, c.sm_count * F::kCtas))), dim3(F::kThreads), F::kSmemBytes, c.stream,
                 map_a, map_b, map_as, map_bs, c.M, c.K, c.N, static_cast<int>(tiles), m_tiles, c.y, c.y_dtype, c.activation,
                 c.dots_out, c.error_flag, c.spin_limit, c.fault);
  return cudaGetLastError();
}

// Tile width for an M x N output: an SM works through ceil(tiles / SMs) tiles.  Measured per tile at K = 2560: 32.7 us
// for 128 columns, 26.7 for 96; 64-column tiles run two to an SM, 34.5 us for both or 23.7 for one alone (1024 x 8192:
// 119 us in 64 columns, 129 in 128; 1024 x 9216: 138 and 130; 517 x 8192: 88 in 64, 79 in 96).
int choose_tile(int M, int N, int sm_count) {
  if (const int forced = gemm_forced_tile())
    return forced;
  const int64_t rows = (M + kTileM - 1) / kTileM;
  auto per_sm = [&](int width) { return (rows * ((N + width - 1) / width) + sm_count - 1) / sm_count; };
  const int64_t cost128 = per_sm(128) * 327, cost96 = per_sm(96) * 267, cost64 = per_sm(64) / 2 * 345 + per_sm(64) % 2 * 237;
  return cost128 <= cost96 && cost128 <= cost64 ? 128 : cost96 <= cost64 ? 96 : 64;
}

template <bool F16> cudaError_t launch_form(const GemmCall &c) {
  switch (choose_tile(c.M, c.N, c.sm_count)) {
  case 64:
    return launch_tile<F16, 64>(c);
  case 96:
    return launch_tile<F16, 96>(c);
  default:
    return launch_tile<F16, 128>(c);
  }
}

// [rows][K/32] scales -> block-major f32 [K/32][ld]; scales are f32 (activations) or f16 bits (weights).  A CTA turns
// 32 x 32 scales through shared memory, so that reads and writes are both of whole lines (an element per thread wrote
// with a stride of a plane's row).
__global__ void __launch_bounds__(256)
scales_block_major_kernel(const void *__restrict__ scales, int scales_are_f16, int64_t rows, int nb, int64_t ld, float *__restrict__ out) {
  __shared__ float tile[32][33];
  grid_dependency_sync();
  const int64_t r0 = blockIdx.x * static_cast<int64_t>(32);
  const int b0 = blockIdx.y * 32, x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
#pragma unroll
  for (int y = y0; y < 32; y += 8)
    if (r0 + y < rows && b0 + x < nb) {
      const int64_t i = (r0 + y) * nb + b0 + x;
      tile[y][x] = scales_are_f16 ? f16_bits_to_f32(static_cast<const uint16_t *>(scales)[i]) : static_cast<const float *>(scales)[i];
    }
  __syncthreads();
#pragma unroll
  for (int y = y0; y < 32; y += 8)
    if (r0 + x < rows && b0 + y < nb)
      out[static_cast<int64_t>(b0 + y) * ld + r0 + x] = tile[x][y];
}

} // namespace

int gemm_forced_tile() {
  const char *flag = std::getenv("LLMCP_B200_GEMM_TILE");
  const int forced = flag ? std::atoi(flag) : 0;
  if (forced == 64 || forced == 96 || forced == 128)
    return forced;
  static std::once_flag told;
  if (flag && *flag)
    std::call_once(told, [flag] {
      std::fprintf(stderr, "llmcp_b200: LLMCP_B200_GEMM_TILE=%s is not a tile width (64, 96 or 128): chosen per shape\n", flag);
    });
  return 0;
}

int64_t gemm_tc16_scale_pitch(int64_t M) { return (M + 3) / 4 * 4; }

void launch_act_to_f16(const int8_t *aq, const float *as, int64_t M, int K, void *ah, float *ast, cudaStream_t stream) {
  const int64_t words = M * (K / 4);
  const int blocks = static_cast<int>(std::min<int64_t>((words + 255) / 256, 148 * 16));
  launch_chained(act_to_f16_kernel, dim3(blocks), dim3(256), 0, stream, aq, as, M, K, gemm_tc16_scale_pitch(M),
                 static_cast<__half *>(ah), ast);
}

void launch_weights_to_f16(const int8_t *wq, const uint16_t *wd, int64_t N, int K, void *wh, float *wst, cudaStream_t stream) {
  const int64_t words = N * (K / 4);
  const int blocks = static_cast<int>(std::min<int64_t>((words + 255) / 256, 148 * 16));
  launch_chained(weights_to_f16_kernel, dim3(blocks), dim3(256), 0, stream, wq, wd, N, K, static_cast<__half *>(wh), wst);
}

void launch_scales_block_major(const void *scales, int scales_are_f16, int64_t rows, int K, int64_t ld, float *out,
                               cudaStream_t stream) {
  const int nb = K / kBlock;
  launch_chained(scales_block_major_kernel, dim3(static_cast<unsigned>((rows + 31) / 32), (nb + 31) / 32), dim3(256), 0, stream, scales,
                 scales_are_f16, rows, nb, ld, out);
}

cudaError_t launch_gemm_q8_tma(int form, const void *a, const float *ast, int M, int K, const void *w, const float *wst, int N,
                               void *y, int y_dtype, int activation, int32_t *dots_out, int *error_flag, cudaStream_t stream,
                               uint32_t spin_limit, int fault) {
  if (M <= 0 || N % 8 != 0 || K % kBlock != 0)
    return cudaErrorInvalidValue;
  if (spin_limit == 0)
    spin_limit = tc::kSpinLimit<true>;
  GemmCall call = {a, ast, M, K, w, wst, N, y, y_dtype, activation, dots_out, error_flag, stream, spin_limit, fault, 148};
  int sms = 0;
  if (current_sm_count(&sms) == cudaSuccess && sms > 0)
    call.sm_count = sms;
  switch (form) {
  case kGemmF16:
  case kGemmF16Packed:
    return launch_form<true>(call);
  case kGemmI8:
    return launch_form<false>(call);
  case kGemmI8Packed:
    if (gemm_few_preferred(M, N))
      return launch_gemm_q8_few(static_cast<const int8_t *>(a), ast, false, M, K, static_cast<const int8_t *>(w), wst, N, y, y_dtype,
                                activation, dots_out, error_flag, stream, spin_limit, fault);
    return launch_form<false>(call);
  default:
    return cudaErrorInvalidValue;
  }
}

} // namespace llmcp_b200
