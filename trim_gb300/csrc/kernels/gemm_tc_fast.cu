// Sector GEMM of the fast tensor-core modes for sm_103a: one BF16 image per
// operand tile (NS = 1) or the two 32-k halves of a TF32 tile (NS = 2), written
// by the slicing kernels (gemm_tc.cu) as exact tcgen05 shared-memory operand
// layouts, FP32 accumulation over the whole K range in k order.
//
// A 128 x 64 output tile moves 24 KB per 64 k for 256 clocks of MMA and is bound
// by what an SM takes in from L2 (34 B per clock with 8 and 16 KB copies, 69 with
// large ones; the MMAs themselves run at 2/3 rate at N = 64).  An item is
// therefore 128 x 64 w, w = 4 column tiles wherever that still gives every SM two
// items: 48 KB for 512 clocks, N = 256 MMAs at the full rate.  The accumulators
// of two items (2 x 256 TMEM columns) are in use at once, so an item's output is
// converted and stored while the next one's MMAs run.
//
// The FP64 output of a float is assembled from its bits (a cvt.f64.f32 runs on
// the FP64 pipe, two per clock and SM: 16 k clocks for a 128 x 256 tile), read in
// the 16 x 256b fragment order and stored as in gemm_tc_split.cu.
//
// CTA (576 threads, one per SM): warp 0 bulk copies (ring of four 48 KB stages:
// one A image, w B images), warp 1 MMA issue, warps 2..17 epilogue: warp v takes
// TMEM lane quadrant v & 3 and columns 16 ((v - 2) >> 2) .. +15 of each 64.
//
// Measured, against 128 x 64 tiles with one accumulator: the GEMMs of
// the iPEPS quadrant at chi = 128, D = 8 (1.4e11 flop, two launches) 0.84 -> 0.20 ms; 16384 x 4096 x 4096
// 1.50 -> 0.40 ms (1.38 PFLOP/s), 331776 x 576 x 576, bound by its 1.5 GB of FP64
// output, 1.9 -> 0.47 ms.
#include <cstdint>

#include "../engine/engine.h"
#include "sm103_ptx.cuh"
#include "tc_digits.cuh"

namespace tn {
namespace {

using namespace ptx;

constexpr int kTM = 128, kTN = 64, kTK = 64;
constexpr int kATile = kTM * kTK * 2;  // bytes of one A image
constexpr int kBTile = kTN * kTK * 2;  // bytes of one B image
constexpr int kWide = kFastWide;       // column tiles of an item, at most
constexpr int kStages = 4, kStage = kATile + kWide * kBTile;
constexpr int kEpiWarps = 16, kEpiCols = 16;
constexpr int kThreadsFast = 64 + 32 * kEpiWarps;
constexpr int kUnit = 14;  // the operands are scaled to 2^7 of their row / column

struct __align__(8) FastShared {
  uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], mma_done;
  int info[kStages];  // steps | column tiles << 3 | first << 6 | last << 7; 0: no more
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void raise_timeout(FastShared& sh, int* err) {
  sh.abort = 1;
  atomicExch(err, TN_ERR_TIMEOUT);
}

__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, FastShared* sh) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, &sh->abort));
}

// warp: 32 TMEM lanes x 16 columns in the accumulator fragment order (see
// tmem_ld32x16x2 in gemm_tc_split.cu)
__device__ __forceinline__ void tmem_ld32x16(uint32_t a, uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(a), "r"(a + (16u << 16))
      : "memory");
}

// the float with bits b times 2^q as a double, exactly where it is normal
__device__ __forceinline__ double float_bits_scaled(uint32_t b, int q) {
  const int ef = (int)((b >> 23) & 0xFFu), ed = ef + 896 + q;
  if (ef == 0 || ef == 255 || ed < 1 || ed > 2046) return scale_pow2((double)__uint_as_float(b), q);
  return __hiloint2double((int)((b & 0x80000000u) | ((uint32_t)ed << 20) | ((b >> 3) & 0xFFFFFu)), (int)(b << 29));
}

template <int NS>
__global__ void __launch_bounds__(kThreadsFast, 1) tc_gemm_fast(const TcSector* __restrict__ secs,
                                                                const int4* __restrict__ items, int nitems, int wide,
                                                                const uint8_t* __restrict__ ws,
                                                                const unsigned long long* __restrict__ ea,
                                                                const unsigned long long* __restrict__ eb,
                                                                double* __restrict__ C, double* __restrict__ part,
                                                                int* __restrict__ err) {
  extern __shared__ uint8_t dyn[];
  __shared__ FastShared sh;
  // 1024-byte aligned operand buffers (the swizzle is anchored to 1024 B)
  uint8_t* base = (uint8_t*)(((uintptr_t)dyn + 1023) & ~(uintptr_t)1023);
  // read from lane 0, so the compiler knows the warp's role to be warp-uniform
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; i++) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&sh.acc_full[i], 1);
      mbar_init(&sh.acc_empty[i], kEpiWarps);
    }
    mbar_init(&sh.mma_done, 1);
    sh.abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&sh.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------ producer: bulk copies
    if (lane == 0) {
      uint32_t n = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
        const int4 w = items[it];
        const TcSector& S = secs[w.x];
        const uint8_t* a_src = ws + S.a_img + (int64_t)w.y * S.nkt * NS * kATile;
        const uint8_t* b_src = ws + S.b_img + (int64_t)w.z * S.nkt * NS * kBTile;
        const int64_t b_step = (int64_t)S.nkt * NS * kBTile;  // from a column tile to the next
        const int kb = w.w * S.kts, ke = min(S.nkt, kb + S.kts);
        const int cols = min(wide, S.nnt - w.z);
        // rows of the images that hold data, in whole groups of 8 rows (1 KB) of
        // A and of the 16 columns of B that are stored in permuted order
        const uint32_t a_bytes = (uint32_t)((min(kTM, S.M - w.y * kTM) + 7) >> 3) * 1024;
        const uint32_t b_last = (uint32_t)((min(kTN, S.N - (w.z + cols - 1) * kTN) + 15) >> 4) * 2048;
        for (int kt = kb; kt < ke && ok; kt++) {
          for (int s = 0; s < NS; s++) {
            const int kdat = S.K - kt * kTK - (NS == 2 ? 32 * s : 0);  // k of this image with data
            if (kdat <= 0) break;
            const int steps = NS == 2 ? min(4, (kdat + 7) >> 3) : min(kTK, kdat + 15) >> 4;
            const bool last = kt == ke - 1 && (NS == 1 || s == 1 || kdat <= 32);
            const int st = n % kStages;
            if (!mbar_wait(&sh.empty[st], ((n / kStages) & 1) ^ 1, &sh.abort)) {
              ok = false;
              break;
            }
            sh.info[st] = steps | cols << 3 | (kt == kb && s == 0) << 6 | last << 7;
            uint8_t* d = base + st * kStage;
            mbar_arrive_expect_tx(&sh.full[st], a_bytes + (cols - 1) * kBTile + b_last);
            bulk_g2s(d, a_src + ((int64_t)kt * NS + s) * kATile, a_bytes, &sh.full[st]);
            for (int c = 0; c < cols; c++)
              bulk_g2s(d + kATile + c * kBTile, b_src + c * b_step + ((int64_t)kt * NS + s) * kBTile,
                       c == cols - 1 ? b_last : kBTile, &sh.full[st]);
            n++;
          }
        }
      }
      if (ok && mbar_wait(&sh.empty[n % kStages], ((n / kStages) & 1) ^ 1, &sh.abort)) {
        sh.info[n % kStages] = 0;
        mbar_arrive(&sh.full[n % kStages]);
        n++;
      } else {
        raise_timeout(sh, err);
      }
      // the copies already issued must land before the CTA's shared memory goes away
      for (int i = 0; i < kStages; i++) {
        const uint32_t uses = n / kStages + (i < (int)(n % kStages) ? 1 : 0);
        if (uses) mbar_drain(&sh.full[i], (uses - 1) & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issue
    // the whole warp runs the loop converged; one elected lane issues
    const uint32_t base_addr = smem_u32(base);
    uint32_t n = 0, tile = 0;
    bool ok = true, ready = false;
    for (;;) {
      const int st = n % kStages;
      ok = ready || warp_wait(&sh.full[st], (n / kStages) & 1, &sh);
      if (!ok) break;
      const int info = __shfl_sync(0xffffffffu, sh.info[st], 0);
      if (info == 0) break;
      const int steps = info & 7, cols = (info >> 3) & 7;
      const uint32_t buf = tile & 1;
      if (info & 64) {
        ok = warp_wait(&sh.acc_empty[buf], ((tile >> 1) & 1) ^ 1, &sh);
        if (!ok) break;
      }
      tc_fence_after();
      n++;
      // the next stage's barrier is tested before the MMAs are issued (see gemm_tc_split.cu)
      const bool next = mbar_test(&sh.full[n % kStages], (n / kStages) & 1);
      const uint32_t d = tmem + buf * kWide * kTN;
      const uint64_t ad = desc_sw128(base_addr + st * kStage), bd = desc_sw128(base_addr + st * kStage + kATile);
      const uint32_t idesc =
          (NS == 2 ? idesc_tf32_f32(kTM, kTN) : idesc_bf16_f32(kTM, kTN)) + ((uint32_t)(cols - 1) * (kTN >> 3) << 17);
      const uint32_t acc0 = (info & 64) ? 0u : 1u;
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
        // 32 bytes of each operand row per step: +2 in the address field
        if (kk < steps) {
          if constexpr (NS == 2)
            mma_tf32_elect(d, ad + 2 * kk, bd + 2 * kk, idesc, kk ? 1u : acc0);
          else
            mma_f16_elect(d, ad + 2 * kk, bd + 2 * kk, idesc, kk ? 1u : acc0);
        }
      mma_commit_elect(&sh.empty[st]);
      if (info & 128) {
        mma_commit_elect(&sh.acc_full[buf]);
        tile++;
      }
      ready = __all_sync(0xffffffffu, next);
    }
    if (!ok && lane == 0) raise_timeout(sh, err);
    // every MMA issued must complete before the tensor memory is released
    mma_commit_elect(&sh.mma_done);
    mbar_drain(&sh.mma_done, 0);
  } else {
    // ------------------------------------------------ epilogue
    const int quad = warp & 3;         // TMEM lanes 32*quad .. +31
    const int half = (warp - 2) >> 2;  // columns half * 16 .. +15 of each column tile
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16) + half * kEpiCols;
    uint32_t tile = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x, tile++) {
      const int4 w = items[it];
      const TcSector& S = secs[w.x];
      const int64_t i0 = (int64_t)w.y * kTM + quad * 32;
      const int cols = min(wide, S.nnt - w.z), rows = (int)min((int64_t)32, S.M - i0);
      const bool split = S.nsplit > 1;  // partial tiles are scaled after their sum
      // lane l: the maximum of row i0 + l, and of column l & 15 of each column tile
      const unsigned long long row_max = lane < rows ? __ldg(ea + S.ea_off + i0 + lane) : 0;
      unsigned long long col_max[kWide];
#pragma unroll
      for (int c = 0; c < kWide; c++) {
        const int64_t j = (int64_t)(w.z + c) * kTN + half * kEpiCols + (lane & 15);
        col_max[c] = c < cols && j < S.N ? __ldg(eb + S.eb_off + j) : 0;
      }
      const uint32_t buf = tile & 1;
      if (!warp_wait(&sh.acc_full[buf], (tile >> 1) & 1, &sh)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int e_row = split ? 0 : exp_of(row_max) - kUnit;
      const int r = lane >> 2, p4 = 4 * (lane & 3);
#pragma unroll
      for (int c = 0; c < kWide; c++) {
        if (c < cols) {
          uint32_t v[16];
          tmem_ld32x16(lane_addr + buf * kWide * kTN + c * kTN, v);
          if (c == cols - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
          }
          const int64_t j0 = (int64_t)(w.z + c) * kTN + half * kEpiCols;
          const int nc = (int)min((int64_t)kEpiCols, S.N - j0);
          const int e_col = split ? 0 : exp_of(col_max[c]);
          int ej[4];
#pragma unroll
          for (int q = 0; q < 4; q++) ej[q] = __shfl_sync(0xffffffffu, e_col, p4 + q);
          const int64_t ld = split ? kTN : S.N;
          // one K range of a split sector: its FP64 partial tile, [128][64]
          double* out = split ? part + S.p_off + (((int64_t)w.y * S.nnt + w.z + c) * S.nsplit + w.w) * (kTM * kTN) +
                                    quad * 32 * kTN + half * kEpiCols + p4
                              : C + S.c_off + i0 * S.N + j0 + p4;
          const bool vec = nc == kEpiCols && (((uintptr_t)out | (uintptr_t)(8 * ld)) & 31) == 0;
#pragma unroll
          for (int t = 0; t < 4; t++) {  // row r + 8 t: values 8 (t / 2) + 2 (t % 2) + {0, 1, 4, 5}
            const int e_i = __shfl_sync(0xffffffffu, e_row, r + 8 * t);
            double* crow = out + (r + 8 * t) * ld;
            const bool live = r + 8 * t < rows;
            double x[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
              x[q] = float_bits_scaled(v[8 * (t >> 1) + 2 * (t & 1) + 4 * (q >> 1) + (q & 1)], e_i + ej[q]);
            if (vec) {
              if (live) store4(crow, x);
            } else {
#pragma unroll
              for (int q = 0; q < 4; q++)
                if (live && p4 + q < nc) crow[q] = x[q];
            }
          }
        }
      }
    }
    if (!ok) raise_timeout(sh, err);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int NS>
void launch_fast(const TcSector* secs, const int4* items, int nitems, int wide, const uint8_t* ws,
                 const unsigned long long* ea, const unsigned long long* eb, double* C, double* part, int* err, int grid,
                 cudaStream_t s) {
  constexpr size_t smem = (size_t)kStages * kStage + 1024;
  static PerDevice attr;  // per instantiation
  allow_smem(attr, current_device(), tc_gemm_fast<NS>, smem);
  tc_gemm_fast<NS><<<grid, kThreadsFast, smem, s>>>(secs, items, nitems, wide, ws, ea, eb, C, part, err);
  TN_CUDA(cudaGetLastError());
}

}  // namespace

void launch_tc_gemm_fast(int ns, const TcSector* secs, const int4* items, int nitems, int wide, const uint8_t* ws,
                         const unsigned long long* ea, const unsigned long long* eb, double* C, double* part, int* err,
                         int grid, cudaStream_t s) {
  if (ns == 2)
    launch_fast<2>(secs, items, nitems, wide, ws, ea, eb, C, part, err, grid, s);
  else
    launch_fast<1>(secs, items, nitems, wide, ws, ea, eb, C, part, err, grid, s);
}

}  // namespace tn
