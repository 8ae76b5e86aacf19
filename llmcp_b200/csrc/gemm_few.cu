// Q8 projection of few rows, or of many rows by few weight rows: short prompts, a batch of sequences decoded together.
// Q8Matmul.cpp:143-289.
//
//   y[m, n] = act( chain_kb fma(float(dot_kb[m, n]), a_scale[m, kb] * w_scale[n, kb], acc) )
//
// What bounds it: the weights (36 bytes per 32 of them from HBM) and, where N is small, the rows, which every CTA
// reads again from L2.  The additions of an output element are one chain over K, so K cannot be shared out; the
// tiles are therefore made narrow (16, 32 or 64 weight rows) until there is one for nearly every SM.  A 128-row
// tcgen05 tile leaves N = 2560 on 20 SMs and hands every 32-wide block's dots from the tensor core to the epilogue
// through tensor memory and two barriers (22 to 34 us at K = 2560, 72 to 112 us at K = 9216, whatever M is).
// Here a warp's mma.sync (m16n8k32: one quantisation block per instruction) leaves the block's dots in the registers
// that scale them and blocks follow each other without a barrier.  Measured (before this kernel -> now): 32 rows 9216 x
// 2560 44 -> 15.5 us, 2560 x 9216 143 -> 22.5; 64 rows 44 -> 26 and 144 -> 34; 32 weight rows 42 -> 9.  The computing
// warps bound it (in-order issue, one or two warps per scheduler), not HBM.
//
// A producer warp keeps a ring of stages in flight by TMA (128-byte swizzle, no multicast): weight rows, activation
// rows, and the block-major scales of both, KS bytes of K per stage.  CTAs are persistent, so the ring runs on across
// output tiles.  (With cp.async issued by the computing warps their address arithmetic was half of all instructions.)
//
// Weight rows are the 16-row operand, activations the 8-column one.  Inside a block the order of the 32 products is
// free (integers), so lane t of a quad takes bytes 8t .. 8t + 7 of each row: one 8-byte load per row where the
// instruction's own order would take two 4-byte ones.  Row g of a fragment is row 2g (g < 4) or 2g - 7 of its eight:
// the four rows that a half warp reads together then lie in different swizzle phases, all 32 banks once.

#include <cuda.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "tc_common.cuh"

namespace llmcp_b200 {

namespace {

using namespace tc;

constexpr int kMaxFewStages = 8;

// WN x WM computing warps; a warp covers 16 weight rows and 8 * NT activation rows; KS bytes of K per stage.
template <int WN, int WM, int NT, int KS, int STAGES> struct Few {
  static constexpr int kRowsW = 16 * WN, kRowsA = 8 * NT * WM, kWarps = WN * WM, kThreads = 32 * (kWarps + 1);
  static constexpr int kBlocks = KS / kBlock, kBoxes = KS / 128;
  static constexpr int kBoxW = kRowsW * 128, kBoxA = kRowsA * 128; // multiples of 1024
  static constexpr int kScalesW = kBlocks * kRowsW * 4, kScalesA = kBlocks * kRowsA * 4;
  static constexpr int kCopied = kBoxes * (kBoxW + kBoxA) + kScalesW + kScalesA;
  static constexpr int kStageBytes = (kCopied + 1023) / 1024 * 1024;
  static constexpr size_t kSmemBytes = 1024 + static_cast<size_t>(STAGES) * kStageBytes;
  static_assert(STAGES <= kMaxFewStages && kSmemBytes <= 112 * 1024, "two CTAs per SM");
};

struct FewBarriers {
  uint64_t full[kMaxFewStages];  // stage landed (one arrival + the copies' bytes)
  uint64_t empty[kMaxFewStages]; // every computing warp is done with it
  int abort_flag;
};

// 16 weight rows x 8 activation rows, 32 products each; sums start at zero.
__device__ __forceinline__ void block_dots(int (&d)[4], uint2 lo, uint2 hi, uint2 b) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
               : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(b.x), "r"(b.y), "r"(0));
}

// c += float(d) * (s * w), two columns at a time; every lane of the pair rounds as the scalar instructions do.
__device__ __forceinline__ void fold2(float &c0, float &c1, int d0, int d1, float2 s, float w) {
  asm("{ .reg .b64 s, w, d, c; mov.b64 s, {%2, %3}; mov.b64 w, {%4, %4}; mul.rn.f32x2 s, s, w; mov.b64 d, {%5, %6};\n"
      "mov.b64 c, {%0, %1}; fma.rn.f32x2 c, d, s, c; mov.b64 {%0, %1}, c; }"
      : "+f"(c0), "+f"(c1)
      : "f"(s.x), "f"(s.y), "f"(w), "f"(__int2float_rn(d0)), "f"(__int2float_rn(d1)));
}

__device__ __forceinline__ float component(float4 v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// ROWS: the activations' scales come as they are quantised, [M][K/32]; otherwise block-major.
// fault (test hook): 1 = the producer announces the first stage's bytes but never issues its copies.
template <int WN, int WM, int NT, int KS, int STAGES, bool DOTS, bool ROWS>
__global__ void __launch_bounds__(Few<WN, WM, NT, KS, STAGES>::kThreads, 2)
gemm_q8_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_ws, const __grid_constant__ CUtensorMap map_as, int M, int K, int N,
                   int tiles, int m_tiles, void *__restrict__ y, int y_dtype, int activation, int32_t *__restrict__ dots_out,
                   int *__restrict__ error_out, uint32_t spin_limit, int fault) {
  using F = Few<WN, WM, NT, KS, STAGES>;
  extern __shared__ uint8_t few_raw[];
  __shared__ FewBarriers bars;
  uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(few_raw) + 1023) & ~uintptr_t(1023));
  volatile int *abort_flag = &bars.abort_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = K / kBlock, stages = (nb + F::kBlocks - 1) / F::kBlocks;
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&bars.full[i], 1);
      mbar_init(&bars.empty[i], F::kWarps);
    }
    bars.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  grid_dependency_sync();

  if (warp == F::kWarps) {
    if (lane == 0) {
      int use = 0; // stages requested so far, over all tiles of this CTA
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % m_tiles) * F::kRowsA, n0 = (tile / m_tiles) * F::kRowsW;
        for (int it = 0; it < stages; ++it, ++use) {
          const int s = use % STAGES;
          if (use >= STAGES && !mbar_wait(&bars.empty[s], (use / STAGES - 1) & 1, abort_flag, spin_limit)) {
            ok = false;
            break;
          }
          uint8_t *stage = base + s * F::kStageBytes;
          mbar_expect_tx(&bars.full[s], F::kCopied);
          if (fault == 1 && use == 0)
            continue;
          for (int b = 0; b < F::kBoxes; ++b) {
            tma_load_2d(stage + b * F::kBoxW, &map_w, it * KS + b * 128, n0, &bars.full[s]);
            tma_load_2d(stage + F::kBoxes * F::kBoxW + b * F::kBoxA, &map_a, it * KS + b * 128, m0, &bars.full[s]);
          }
          uint8_t *scales = stage + F::kBoxes * (F::kBoxW + F::kBoxA);
          tma_load_2d(scales, &map_ws, n0, it * F::kBlocks, &bars.full[s]);
          tma_load_2d(scales + F::kScalesW, &map_as, ROWS ? it * F::kBlocks : m0, ROWS ? m0 : it * F::kBlocks, &bars.full[s]);
        }
      }
      // Leaving after a failed wait: copies already requested still write into this CTA's shared memory.
      if (*abort_flag)
        for (int i = max(0, use - STAGES); i < use; ++i)
          if (!(fault == 1 && i == 0))
            mbar_wait_quiet(&bars.full[i % STAGES], (i / STAGES) & 1, spin_limit);
    }
  } else {
    const int wn = warp % WN, wm = warp / WN, g = lane >> 2, t = lane & 3;
    const int row8 = g < 4 ? 2 * g : 2 * g - 7; // this lane's row of each group of eight
    uint32_t offset[4];                         // its 8 bytes of block b inside a swizzled row of four blocks
#pragma unroll
    for (int b = 0; b < 4; ++b)
      offset[b] = row8 * 128 + (((2 * b + (t >> 1)) ^ row8) << 4) + (t & 1) * 8;
    int use = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const int m0 = (tile % m_tiles) * F::kRowsA, n0 = (tile / m_tiles) * F::kRowsW;
      float acc[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
        acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
      for (int it = 0; it < stages; ++it, ++use) {
        const int s = use % STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.full[s], (use / STAGES) & 1, abort_flag, spin_limit));
        if (!ok)
          break;
        const uint8_t *stage = base + s * F::kStageBytes;
        const uint8_t *w_rows = stage + wn * 16 * 128, *a_rows = stage + F::kBoxes * F::kBoxW + wm * 8 * NT * 128;
        const float *w_scale = reinterpret_cast<const float *>(stage + F::kBoxes * (F::kBoxW + F::kBoxA)) + wn * 16 + row8;
        // column 2t of the result is activation row 2t of the fragment's order, column 2t + 1 row 2t + 1
        const float *a_scale = reinterpret_cast<const float *>(stage + F::kBoxes * (F::kBoxW + F::kBoxA) + F::kScalesW) + wm * 8 * NT * (ROWS ? F::kBlocks : 1);
        const int c0 = t < 2 ? 4 * t : 4 * t - 7, c1 = c0 + 2;
        // The scales as they are quantised: four blocks of a row at a time where the registers allow it.
        constexpr bool kFour = ROWS && NT <= 2;
        float4 four[kFour ? NT : 1][2];
        auto fold = [&](int b) {
          if (kFour && b % 4 == 0) {
#pragma unroll
            for (int j = 0; j < (kFour ? NT : 0); ++j) {
              four[j][0] = *reinterpret_cast<const float4 *>(a_scale + (j * 8 + c0) * F::kBlocks + b);
              four[j][1] = *reinterpret_cast<const float4 *>(a_scale + (j * 8 + c1) * F::kBlocks + b);
            }
          }
          const uint8_t *w_box = w_rows + (b / 4) * F::kBoxW + offset[b % 4], *a_box = a_rows + (b / 4) * F::kBoxA + offset[b % 4];
          const uint2 lo = *reinterpret_cast<const uint2 *>(w_box);
          const uint2 hi = *reinterpret_cast<const uint2 *>(w_box + 8 * 128);
          const float w0 = w_scale[b * F::kRowsW], w1 = w_scale[b * F::kRowsW + 8];
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint2 x = *reinterpret_cast<const uint2 *>(a_box + j * 8 * 128);
            float2 sa;
            if (kFour)
              sa = make_float2(component(four[j % (kFour ? NT : 1)][0], b % 4), component(four[j % (kFour ? NT : 1)][1], b % 4));
            else if (ROWS)
              sa = make_float2(a_scale[(j * 8 + c0) * F::kBlocks + b], a_scale[(j * 8 + c1) * F::kBlocks + b]);
            else
              sa = make_float2(a_scale[b * F::kRowsA + j * 8 + c0], a_scale[b * F::kRowsA + j * 8 + c1]);
            int d[4];
            block_dots(d, lo, hi, x);
            fold2(acc[j][0], acc[j][1], d[0], d[1], sa, w0);
            fold2(acc[j][2], acc[j][3], d[2], d[3], sa, w1);
            if (DOTS) {
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int m = m0 + wm * 8 * NT + j * 8 + (u & 1 ? c1 : c0), n = n0 + wn * 16 + row8 + (u >> 1) * 8;
                if (m < M && n < N)
                  dots_out[(static_cast<int64_t>(m) * N + n) * nb + it * F::kBlocks + b] = d[u];
              }
            }
          }
        };
        const int blocks = min(F::kBlocks, nb - it * F::kBlocks);
        if (blocks == F::kBlocks) {
#pragma unroll
          for (int b = 0; b < F::kBlocks; ++b)
            fold(b);
        } else {
#pragma unroll
          for (int b = 0; b < F::kBlocks; ++b)
            if (b < blocks)
              fold(b);
        }
        __syncwarp();
        if (lane == 0)
          mbar_arrive(&bars.empty[s]);
      }
      if (!ok)
        break;
      const int c0 = t < 2 ? 4 * t : 4 * t - 7;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int m = m0 + wm * 8 * NT + j * 8 + c0 + (u & 1) * 2, n = n0 + wn * 16 + row8 + (u >> 1) * 8;
          if (m < M && n < N)
            store_from_f32(y, y_dtype, static_cast<int64_t>(m) * N + n, apply_activation(acc[j][u], activation));
        }
    }
  }
  __syncthreads();
  if (tid == 0 && bars.abort_flag && error_out)
    atomicExch(error_out, 1);
}

struct FewCall {
  const int8_t *aq;
  const float *as; // [M][K/32], or block-major
  bool rows;
  int M, K;
  const int8_t *wq;
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

template <int WN, int WM, int NT, int KS, int STAGES, bool MAY_BE_ROWS> cudaError_t launch_few(const FewCall &c) {
  using F = Few<WN, WM, NT, KS, STAGES>;
  const int nb = c.K / kBlock;
  CUtensorMap map_w, map_a, map_ws, map_as;
  if (!gemm_operand_map(&map_w, c.wq, c.N, c.K, false, F::kRowsW) || !gemm_operand_map(&map_a, c.aq, c.M, c.K, false, F::kRowsA) ||
      !gemm_scale_map(&map_ws, c.wst, c.N, c.N, nb, F::kBlocks, F::kRowsW) ||
      !(c.rows ? gemm_scale_map(&map_as, c.as, nb, nb, c.M, F::kRowsA, F::kBlocks)
               : gemm_scale_map(&map_as, c.as, c.M, gemm_tc16_scale_pitch(c.M), nb, F::kBlocks, F::kRowsA)))
    return cudaErrorNotSupported;
  auto kernel = c.dots_out ? gemm_q8_few_kernel<WN, WM, NT, KS, STAGES, true, false>
                : c.rows   ? gemm_q8_few_kernel<WN, WM, NT, KS, STAGES, false, MAY_BE_ROWS>
                           : gemm_q8_few_kernel<WN, WM, NT, KS, STAGES, false, false>;
  if (cudaError_t e = opt_in_shared_memory(reinterpret_cast<const void *>(kernel), F::kSmemBytes); e != cudaSuccess)
    return e;
  const int m_tiles = (c.M + F::kRowsA - 1) / F::kRowsA, tiles = m_tiles * ((c.N + F::kRowsW - 1) / F::kRowsW);
  launch_chained(kernel, dim3(std::min(tiles, 2 * c.sm_count)), dim3(F::kThreads), F::kSmemBytes, c.stream, map_w, map_a, map_ws,
                 map_as, c.M, c.K, c.N, tiles, m_tiles, c.y, c.y_dtype, c.activation, c.dots_out, c.error_flag, c.spin_limit, c.fault);
  return cudaGetLastError();
}

} // namespace

// Where this kernel is the faster one (64 x 64 tiles against the 128-row tiles of gemm_tma.cu, K = 2560): up to 32
// rows always (248320 weight rows: 246 us against 460); up to 64 rows until an SM has more than four tiles (9216 weight
// rows 26 us against 36; 248320: 563 against 460); beyond that while two of three SMs at most have one (128 x 2560 x 9216
// 64 us against 72, 128 x 4096 x 2560 26 against 24).
bool gemm_few_preferred(int M, int N) {
  if (gemm_forced_tile())
    return false;
  int sms = 148;
  if (current_sm_count(&sms) != cudaSuccess || sms <= 0)
    sms = 148;
  const int64_t tiles = static_cast<int64_t>((M + 63) / 64) * ((N + 63) / 64);
  return M <= 32 || (M <= 64 ? tiles <= 4 * sms : 3 * tiles <= 2 * sms);
}

// More than 32 rows: a launch less in front of every GEMM (64 sequences decoded together, 13 steps: 105 -> 98 ms).  Up to 32
// rows their copies of 32 bytes per row cost more than that launch (a 23-token prompt: 4.8 ms block-major, 5.0 so).
bool gemm_few_takes_row_scales(int M, int K, const float *as) {
  return M > 32 && K % 128 == 0 && reinterpret_cast<uintptr_t>(as) % 16 == 0;
}

cudaError_t launch_gemm_q8_few(const int8_t *aq, const float *as, bool row_scales, int M, int K, const int8_t *wq, const float *wst,
                               int N, void *y, int y_dtype, int activation, int32_t *dots_out, int *error_flag, cudaStream_t stream,
                               uint32_t spin_limit, int fault) {
  if (M <= 0 || N % 8 != 0 || K % kBlock != 0 || (row_scales && (dots_out || !gemm_few_takes_row_scales(M, K, as))))
    return cudaErrorInvalidValue;
  if (spin_limit == 0)
    spin_limit = kSpinLimit<true>;
  FewCall call = {aq, as, row_scales, M, K, wq, wst, N, y, y_dtype, activation, dots_out, error_flag, stream, spin_limit, fault, 148};
  int sms = 0;
  if (current_sm_count(&sms) == cudaSuccess && sms > 0)
    call.sm_count = sms;
  const bool narrow = M <= 32; // activation rows of a tile: 32 or 64
  const int64_t rows = narrow ? 1 : (M + 63) / 64;
  // The widest tile that still gives four of five SMs a CTA.
  const int64_t enough = call.sm_count * 4 / 5;
  if (rows * ((N + 63) / 64) >= enough)
    return narrow ? launch_few<4, 2, 2, 128, 7, false>(call) : launch_few<4, 2, 4, 128, 6, true>(call);
  if (rows * ((N + 31) / 32) >= enough)
    return narrow ? launch_few<2, 2, 2, 256, 6, false>(call) : launch_few<2, 4, 2, 256, 4, true>(call);
  return narrow ? launch_few<1, 4, 1, 256, 7, false>(call) : launch_few<1, 4, 2, 256, 4, true>(call);
}

} // namespace llmcp_b200
