// Split-precision sector GEMM for sm_103a, tiled form (TN_MODE_SPLIT): the
// digit images written by tc_slices<6> (gemm_tc.cu) multiplied on the tcgen05
// tensor cores and recombined exactly.
//
// Digits: every FP64 element is rounded to 53 bits below its row's (A) or
// column's (B) power-of-two scale 2^e > max and cut into 6 balanced base-512
// digits, x = 2^(e-8) sum_s d_s 2^(-9s), |d_0| <= 256, d_1..d_5 in
// [-256, 255]: integers that FP16 holds exactly.  C = 2^(ea+eb-16)
// sum_{s+t<=5} 2^(-9(s+t)) A_s B_t: 21 digit products.
// What is left out (s + t >= 6) is five products of, on average, 2^-55.6 of the
// two maxima per k; the 34 products of 7-bit digits this replaced rounded the
// operands at 2^-50, 2^-50.8 of a maximum times the other operand.  So the error
// is below theirs while the root mean squares of a row and a column are above
// 1/18 of their scales (it is 1/9 .. 1/4 for Gaussian entries, 0.3 .. 0.6 for
// uniform ones).  With |d_0| <= 128, a bit less of each operand, it was four times
// as large, and above theirs on Gaussian entries.
// Measured (Frobenius norm, relative, against 113-bit sums; 34 products / |d_0|
// <= 128 / now): uniform entries, K = 160000 6.7e-15 / 6.1e-16 / 2.9e-16;
// Gaussian, K = 2000 3.8e-15 / 3.6e-15 / 8.7e-16, K = 160000 8.5e-15 / 1.1e-14 /
// 3.0e-15.  Where a row and a column both hold one entry near their scale and the
// rest at 1..2% of it, the error is 1.4..1.6 times that of the 34 products; four of
// the five products of level 6 would undo that, for 28 to 35% more MMA time.
// Wider digits than 7 bits are what FP32 accumulation limits: per k the digit
// products of levels 0..5 (l = s + t) sum to at most (l + 1) 2^16, so over one
// 64-k tile levels 0..3 are exact integers up to 2^24; level 4 reaches there only
// where every digit is at its largest, and rounds by one of 2^-52, level 5 at
// 2^-60.  The accumulators are therefore drained every 64-k tile, which the
// digit width pays for only if the drain runs beside the MMAs.
//
// Tensor memory is a ring of four 128-column slots, each holding two levels
// (0/1, 2/3, 4/5) of one 64-k tile at 64 columns: a tile takes three slots,
// and the epilogue warps empty them in order while the MMAs go on.  The MMAs
// of a tile run digit s of A after digit s against B digits 0..5-s: s = 0
// opens all levels, s = 1 completes levels 0/1, s = 3 levels 2/3, s = 5 levels
// 4/5.  The next tile opens its first slot while the last one drains, and
// needs the other two only after its first 128-column MMAs, so the drain of
// levels 2/3 has about 700 clocks before the tensor pipe would wait.  One MMA
// takes an A digit with 2..4 B digits (N = 64 n, the B images lie back to
// back) wherever the levels' columns are consecutive; with three slots per
// tile in a ring of four the pattern repeats every four tiles, so four tiles
// are unrolled with every column, shape, slot and accumulate flag a constant.
// That straight line is what keeps the tensor pipe fed: an issue loop that
// worked these out at run time took 125 clocks per MMA (99 of work), and so
// did the straight line until the warp's role and the tile's step count were
// read from one lane (__shfl_sync), which makes the branches warp-uniform for
// the compiler.
//
// Drain: each level converts to int32 exactly (cvt runs at full rate); per
// output a 32-bit integer sums level 0 and a 64-bit one the others, in units of
// level 4 (2^-36 of level 0; 15 issue slots per output and tile).  Together, in
// units of 2^-34 of level 0, |sum| < K 2^50.03, so they are moved to the FP64
// output every 4096 k.
//
// CTA (576 threads, one per SM, 128 x 64 output tile): warp 0 bulk copies
// (8-slot ring of 16 KB A digit tiles, 2-slot ring of 48 KB B tiles), warp 1
// MMA issue, warps 2..17 drain: warp w takes TMEM lane quadrant w & 3 and
// columns 16 ((w - 2) >> 2) .. +15 of each level.
//
// Measured (GB300, all of a call's launches): the left MERA diagram at chi = 24
// (K = 576, 6.7e11 FP64-equivalent flop) 16.0 -> 10.0 ms, the iPEPS quadrant at
// chi = 128, D = 8 (K = 4096, 1.4e11) 3.41 -> 1.83 ms, against the 34-product
// kernel.  21 products per FP64 multiply-add: 77 TFLOP/s FP64-equivalent at
// K = 4096 is 1 620 of FP16.  What bounds it, from copies with parts left out:
// 80000 x 576 over K = 576 takes 761 us, 677 without the drain's arithmetic, 596
// without the output as well (64 KB of FP64 every ninth tile, about 8 000 clocks in
// which the ring fills and the MMAs stop), 574 without loads; 4096^3 1703, 1619,
// 1607 and 1505 us.  Converting by magic-number additions instead of cvt changed
// nothing (its range check cost 10%), nor did loading A two digits at a time.
#include <cstdint>

#include "../engine/engine.h"
#include "sm103_ptx.cuh"
#include "tc_digits.cuh"

namespace tn {
namespace {

using namespace ptx;

constexpr int kTM = 128, kTN = 64, kTK = 64;
constexpr int kDigits = 6;             // levels 0..5, one per digit
constexpr int kATile = kTM * kTK * 2;  // bytes of one A digit tile
constexpr int kBTile = kTN * kTK * 2;  // bytes of one B digit tile
constexpr int kARing = 8, kBRing = 2;
constexpr int kSlots = 4, kSlotCols = 2 * kTN;  // TMEM ring: two levels per slot
constexpr int kEpiWarps = 16, kEpiCols = kTN * 4 / kEpiWarps;
constexpr int kThreadsSplit = 64 + 32 * kEpiWarps;
constexpr int kSegTiles = 64;  // 4096 k per 64-bit integer sum
constexpr int kUnit = 50;      // the sum's unit is 2^(ea + eb - 50)

struct __align__(8) SplitShared {
  uint64_t fullA[kARing], emptyA[kARing], fullB[kBRing], emptyB[kBRing];
  uint64_t fullT[kSlots], emptyT[kSlots], mma_done;
  int steps[kBRing];  // 16-k steps with data of the tile in this B slot; 0: no more tiles
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void raise_timeout(SplitShared& sh, int* err) {
  sh.abort = 1;
  atomicExch(err, TN_ERR_TIMEOUT);
}

// column of level l of a tile whose first slot is R
__host__ __device__ constexpr int level_col(int R, int l) { return ((R + (l >> 1)) & 3) * kSlotCols + (l & 1) * kTN; }
// levels l, l+1, .. in consecutive columns, up to level 5
__host__ __device__ constexpr int level_run(int R, int l) {
  int n = 1;
  while (l + n < kDigits && level_col(R, l + n) == level_col(R, l) + n * kTN) n++;
  return n;
}
// levels one MMA takes from level l on, for A digit s: s = 0 opens its first
// slot by itself, a run of five goes as 3 + 2 (4 + 1 would end in an N = 64
// MMA, bound by its operand reads: 48 clocks for 32 of work)
__host__ __device__ constexpr int level_group(int R, int s, int l) {
  const int run = level_run(R, l);
  if (s == 0 && l == 0) return 2;
  return run == 5 ? 3 : (run > 4 ? 4 : run);
}

// What the MMA warp carries along.  Tile number n = 4 q + M of the CTA takes
// TMEM slots 3 n .. 3 n + 2, A ring slots 6 n .. 6 n + 5 and B slot n, each
// modulo its ring: with M a template parameter every slot is a constant and
// every barrier's parity is a constant or a constant XOR the parity of q.
struct MmaState {
  SplitShared* sh;
  uint32_t tmem, abuf, bbuf;  // tensor memory; shared-memory addresses of the rings
  uint32_t q;                 // parity of the tile number / 4
  int nks;                    // 16-k steps of this tile that hold data
  bool a_ready, b_ready, t_ready;  // the next A digit tile / B tile / TMEM slot was seen ready
};
static_assert(kARing == 8 && kBRing == 2 && kSlots == 4 && kDigits == 6, "the ring positions below repeat every 4 tiles");

__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, SplitShared* sh) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, &sh->abort));
}

// the MMAs of A digit S into levels L..5
template <int M, int S, int L, bool FULL>
__device__ __forceinline__ bool split_groups(MmaState& st, uint64_t adesc) {
  if constexpr (L < kDigits) {
    constexpr int R = 3 * M % kSlots, n = level_group(R, S, L);
    constexpr uint32_t idesc = idesc_fp16_f32(kTM, kTN) + ((uint32_t)(n - 1) * (kTN >> 3) << 17);
    constexpr uint32_t col = level_col(R, L);
    const uint64_t bdesc = desc_sw128(st.bbuf + (M % kBRing) * kDigits * kBTile + (L - S) * kBTile);
    uint64_t* t1 = &st.sh->emptyT[(R + 1) % kSlots];  // the tile's other two slots
    uint64_t* t2 = &st.sh->emptyT[(R + 2) % kSlots];
    const uint32_t p1 = (st.q ^ ((3 * M + 1) / kSlots) ^ 1) & 1, p2 = (st.q ^ ((3 * M + 2) / kSlots) ^ 1) & 1;
    bool r1 = false, r2 = false;
#pragma unroll
    for (int kk = 0; kk < kTK / 16; kk++) {
      if (S == 0 && L == 0 && kk == 2) {
        r1 = mbar_test(t1, p1);
        r2 = mbar_test(t2, p2);
      }
      // advancing K by 16 halves = 32 bytes inside the swizzle atom: +2 in the address field
      if (FULL || kk < st.nks)
        mma_f16_elect(st.tmem + col, adesc + 2 * kk, bdesc + 2 * kk, idesc, (S > 0 || kk > 0) ? 1u : 0u);
    }
    if constexpr (S == 0 && L == 0) {
      if (!__all_sync(0xffffffffu, r1 && r2) && !(warp_wait(t1, p1, st.sh) && warp_wait(t2, p2, st.sh))) return false;
      tc_fence_after();
    }
    return split_groups<M, S, L + n, FULL>(st, adesc);
  }
  return true;
}

template <int M, int S, bool FULL>
__device__ __forceinline__ bool split_digits(MmaState& st) {
  if constexpr (S < kDigits) {
    SplitShared* sh = st.sh;
    constexpr int A = kDigits * M + S, T = 3 * M;  // A ring and TMEM ring positions
    if (!st.a_ready && !warp_wait(&sh->fullA[A % kARing], (st.q ^ (A / kARing)) & 1, sh)) return false;
    tc_fence_after();
    // 24 A slots are three rounds of the ring, 12 TMEM slots of theirs: both
    // parities advance with q
    const bool a_next = mbar_test(&sh->fullA[(A + 1) % kARing], (st.q ^ ((A + 1) / kARing)) & 1);
    bool b_next = false, t_next = false;
    if constexpr (S == kDigits - 1) {
      b_next = mbar_test(&sh->fullB[(M + 1) % kBRing], ((M + 1) / kBRing) & 1);
      t_next = mbar_test(&sh->emptyT[(T + 3) % kSlots], (st.q ^ ((T + 3) / kSlots) ^ 1) & 1);
    }
    if (!split_groups<M, S, S, FULL>(st, desc_sw128(st.abuf + (A % kARing) * kATile))) return false;
    mma_commit_elect(&sh->emptyA[A % kARing]);
    if constexpr (S & 1) mma_commit_elect(&sh->fullT[(T + (S >> 1)) % kSlots]);  // two levels complete
    st.a_ready = __all_sync(0xffffffffu, a_next);
    if constexpr (S == kDigits - 1) {
      st.b_ready = __all_sync(0xffffffffu, b_next);
      st.t_ready = __all_sync(0xffffffffu, t_next);
    }
    return split_digits<M, S + 1, FULL>(st);
  }
  return true;
}

// tile M of the four: 1 done, 0 no more tiles, -1 a wait gave up
template <int M>
__device__ __forceinline__ int split_tile(MmaState& st) {
  SplitShared* sh = st.sh;
  if (!st.b_ready && !warp_wait(&sh->fullB[M % kBRing], (M / kBRing) & 1, sh)) return -1;
  st.nks = __shfl_sync(0xffffffffu, sh->steps[M % kBRing], 0);
  if (st.nks == 0) return 0;
  if (!st.t_ready && !warp_wait(&sh->emptyT[3 * M % kSlots], (st.q ^ (3 * M / kSlots) ^ 1) & 1, sh)) return -1;
  tc_fence_after();
  if (!(st.nks == kTK / 16 ? split_digits<M, 0, true>(st) : split_digits<M, 0, false>(st))) return -1;
  mma_commit_elect(&sh->emptyB[M % kBRing]);
  return 1;
}

// warp: 32 TMEM lanes x 16 columns at a and at b, as four 16-lane x 16-column
// loads in the accumulator fragment order: with r = lane / 4 and p = lane % 4,
// value 8 h + 4 g + 2 u + i is row 16 h + 8 u + r, column 8 g + 2 p + i.  The
// data is in the registers on return.  The caller's warp_wait has brought the warp
// together (a __syncwarp here as well took 0.2 to 0.5% of the call).
__device__ __forceinline__ void tmem_ld32x16x2(uint32_t a, uint32_t b, float (&v)[16], float (&w)[16]) {
  uint32_t r[16], s[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(s[0]),
        "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]),
        "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
      : "r"(a), "r"(a + (16u << 16)), "r"(b), "r"(b + (16u << 16))
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) {
    v[i] = __uint_as_float(r[i]);
    w[i] = __uint_as_float(s[i]);
  }
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

__global__ void __launch_bounds__(kThreadsSplit, 1) tc_gemm_split(const TcSector* __restrict__ secs,
                                                                  const int4* __restrict__ items, int nitems,
                                                                  const uint8_t* __restrict__ ws,
                                                                  const unsigned long long* __restrict__ ea,
                                                                  const unsigned long long* __restrict__ eb,
                                                                  double* __restrict__ C, double* __restrict__ part,
                                                                  int* __restrict__ err) {
  extern __shared__ uint8_t dyn[];
  __shared__ SplitShared sh;
  // 1024-byte aligned operand buffers (the swizzle is anchored to 1024 B)
  uint8_t* base = (uint8_t*)(((uintptr_t)dyn + 1023) & ~(uintptr_t)1023);
  uint8_t* abuf = base;                    // kARing x 16 KB
  uint8_t* bbuf = base + kARing * kATile;  // kBRing x 6 x 8 KB
  // read from lane 0, so the compiler knows the warp's role to be warp-uniform
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kARing; i++) {
      mbar_init(&sh.fullA[i], 1);
      mbar_init(&sh.emptyA[i], 1);
    }
    for (int i = 0; i < kBRing; i++) {
      mbar_init(&sh.fullB[i], 1);
      mbar_init(&sh.emptyB[i], 1);
    }
    for (int i = 0; i < kSlots; i++) {
      mbar_init(&sh.fullT[i], 1);
      mbar_init(&sh.emptyT[i], kEpiWarps);
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
      uint32_t na = 0, nb = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
        const int4 w = items[it];
        const TcSector& S = secs[w.x];
        const uint8_t* a_src = ws + S.a_img + (int64_t)w.y * S.nkt * kDigits * kATile;
        const uint8_t* b_src = ws + S.b_img + (int64_t)w.z * S.nkt * kDigits * kBTile;
        const int kb = w.w * S.kts, ke = min(S.nkt, kb + S.kts);  // this item's K range
        // rows of the images that hold data: A's to whole groups of 8 rows (1 KB),
        // B's to the 16 columns that are stored in permuted order
        const uint32_t a_bytes = (uint32_t)((min(kTM, S.M - w.y * kTM) + 7) >> 3) * 1024;
        const uint32_t b_bytes = (uint32_t)((min(kTN, S.N - w.z * kTN) + 15) >> 4) * 2048;
        for (int kt = kb; kt < ke && ok; kt++) {
          const int sb = nb % kBRing;
          if (!mbar_wait(&sh.emptyB[sb], ((nb / kBRing) & 1) ^ 1, &sh.abort)) {
            ok = false;
            break;
          }
          sh.steps[sb] = min(kTK, S.K - kt * kTK + 15) >> 4;
          uint8_t* bd = bbuf + sb * kDigits * kBTile;
          const uint8_t* bs = b_src + (int64_t)kt * kDigits * kBTile;
          mbar_arrive_expect_tx(&sh.fullB[sb], kDigits * b_bytes);
          if (b_bytes == kBTile)
            bulk_g2s(bd, bs, kDigits * kBTile, &sh.fullB[sb]);
          else
            for (int s = 0; s < kDigits; s++) bulk_g2s(bd + s * kBTile, bs + s * kBTile, b_bytes, &sh.fullB[sb]);
          nb++;
          for (int s = 0; s < kDigits; s++) {
            const int sa = na % kARing;
            if (!mbar_wait(&sh.emptyA[sa], ((na / kARing) & 1) ^ 1, &sh.abort)) {
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&sh.fullA[sa], a_bytes);
            bulk_g2s(abuf + sa * kATile, a_src + ((int64_t)kt * kDigits + s) * kATile, a_bytes, &sh.fullA[sa]);
            na++;
          }
        }
      }
      if (ok && mbar_wait(&sh.emptyB[nb % kBRing], ((nb / kBRing) & 1) ^ 1, &sh.abort)) {
        sh.steps[nb % kBRing] = 0;
        mbar_arrive(&sh.fullB[nb % kBRing]);
        nb++;
      } else {
        raise_timeout(sh, err);
      }
      // the copies already issued must land before the CTA's shared memory goes away
      for (int i = 0; i < kARing; i++) {
        const uint32_t uses = na / kARing + (i < (int)(na % kARing) ? 1 : 0);
        if (uses) mbar_drain(&sh.fullA[i], (uses - 1) & 1);
      }
      for (int i = 0; i < kBRing; i++) {
        const uint32_t uses = nb / kBRing + (i < (int)(nb % kBRing) ? 1 : 0);
        if (uses) mbar_drain(&sh.fullB[i], (uses - 1) & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issue
    // the whole warp runs the loop converged; one elected lane issues.  The
    // tiles come from the producer (B slot by B slot), which runs ahead and so
    // hides the loads of the work list
    MmaState st;
    st.sh = &sh;
    st.tmem = tmem;
    st.abuf = smem_u32(abuf);
    st.bbuf = smem_u32(bbuf);
    st.a_ready = st.b_ready = st.t_ready = false;
    int more = 1;
    for (st.q = 0; more > 0; st.q ^= 1) {
      more = split_tile<0>(st);
      if (more > 0) more = split_tile<1>(st);
      if (more > 0) more = split_tile<2>(st);
      if (more > 0) more = split_tile<3>(st);
    }
    const bool ok = more == 0;
    if (!ok && lane == 0) raise_timeout(sh, err);
    // every MMA issued must complete before the tensor memory is released
    mma_commit_elect(&sh.mma_done);
    mbar_drain(&sh.mma_done, 0);
  } else {
    // ------------------------------------------------ epilogue
    const int quad = warp & 3;         // TMEM lanes 32*quad .. +31
    const int half = (warp - 2) >> 2;  // columns half * kEpiCols .. +kEpiCols-1 of a level
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16) + half * kEpiCols;
    uint32_t g = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
      const int4 w = items[it];
      // the next item and its sector come into L1 while this one is drained
      const int next = min(it + (int)gridDim.x, nitems - 1);
      prefetch_l1(items + next);
      const TcSector& S = secs[w.x];
      const int kb = w.w * S.kts, ke = min(S.nkt, kb + S.kts);
      const int64_t i0 = (int64_t)w.y * kTM + quad * 32, i = i0 + lane;
      const int64_t j0 = (int64_t)w.z * kTN + half * kEpiCols;  // first column of this warp
      const int nc = (int)max((int64_t)0, min((int64_t)kEpiCols, S.N - j0));
      // lane l: the maximum of row i0 + l, and of column j0 + (l & 15)
      const unsigned long long row_max = i < S.M ? __ldg(ea + S.ea_off + i) : 0;
      const unsigned long long col_max = (lane & 15) < nc ? __ldg(eb + S.eb_off + j0 + (lane & 15)) : 0;
      for (int k0 = kb; k0 < ke && ok; k0 += kSegTiles) {
        const int k1 = min(ke, k0 + kSegTiles);
        int top[kEpiCols];  // level 0, and the others in units of level 4
        long long acc[kEpiCols];
#pragma unroll
        for (int q = 0; q < kEpiCols; q++) top[q] = 0, acc[q] = 0;
        for (int kt = k0; kt < k1 && ok; kt++) {
#pragma unroll
          for (int j = 0; j < 3; j++) {
            const int slot = g % kSlots;
            if (!warp_wait(&sh.fullT[slot], (g / kSlots) & 1, &sh)) {
              ok = false;
              break;
            }
            tc_fence_after();
            float a[kEpiCols], b[kEpiCols];  // levels 2j and 2j + 1
            tmem_ld32x16x2(lane_addr + slot * kSlotCols, lane_addr + slot * kSlotCols + kTN, a, b);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.emptyT[slot]);
            g++;
#pragma unroll
            for (int q = 0; q < kEpiCols; q++) {
              if (j == 0)
                top[q] += __float2int_rn(a[q]), acc[q] += (long long)__float2int_rn(b[q]) * (1 << 27);
              else if (j == 1)
                acc[q] += (long long)__float2int_rn(a[q]) * (1 << 18) + (long long)__float2int_rn(b[q]) * (1 << 9);
              else
                acc[q] += (long long)__float2int_rn(fmaf(b[q], 0x1p-9f, a[q]));
            }
          }
          if (kt == kb) prefetch_l1(secs + __ldg(&items[next].x));
        }
        if (!ok) break;
        if (nc > 0) {
          const int e_row = exp_of(row_max) - kUnit, e_col = exp_of(col_max);
          // every scale of the warp well inside the exponent range: no output can leave it
          const bool plain = __all_sync(0xffffffffu, abs(e_row) < 400 && abs(e_col) < 400);
          // the images of B hold the columns of a group of 16 in the order that gives a
          // thread four consecutive ones: columns j0 + 4 p .. + 3 of rows r, r + 8, ..
          const int r = lane >> 2, p4 = 4 * (lane & 3);
          int ej[4];
#pragma unroll
          for (int c = 0; c < 4; c++) ej[c] = __shfl_sync(0xffffffffu, e_col, p4 + c);
          // one K range of a split sector: its FP64 partial tile, [128][64]
          double* out = S.nsplit > 1 ? part + S.p_off +
                                           (((int64_t)w.y * S.nnt + w.z) * S.nsplit + w.w) * (kTM * kTN) +
                                           quad * 32 * kTN + half * kEpiCols + p4
                                     : C + S.c_off + i0 * S.N + j0 + p4;
          const int64_t ld = S.nsplit > 1 ? kTN : S.N;
          const int rows = (int)min((int64_t)32, S.M - i0);
          const bool several = S.nsplit > 1 || ke - kb > kSegTiles;  // partial tiles or segments
          const bool wide = plain && nc == kEpiCols && ke - kb <= kSegTiles && (((uintptr_t)out | (uintptr_t)(8 * ld)) & 31) == 0;
#pragma unroll
          for (int t = 0; t < 4; t++) {  // row r + 8 t: values 8 (t / 2) + 2 (t % 2) + {0, 1, 4, 5}
            const int e_i = __shfl_sync(0xffffffffu, e_row, r + 8 * t);
            double* crow = out + (r + 8 * t) * ld;
            const bool live = r + 8 * t < rows;
            double v[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const int n = 8 * (t >> 1) + 2 * (t & 1) + 4 * (c >> 1) + (c & 1);
              const long long x = ((long long)top[n] << 34) + ((acc[n] + 2) >> 2);
              // several sums to add: without the scales, which the last addition is
              // followed by (so a result in the subnormal range is rounded once)
              const int q = several ? -kUnit : e_i + ej[c];
              v[c] = plain ? fixed_to_double_inrange(x, q) : fixed_to_double(x, q);
            }
            if (wide) {
              if (live) store4(crow, v);
            } else {
#pragma unroll
              for (int c = 0; c < 4; c++)
                if (live && p4 + c < nc) {
                  if (k0 > kb) v[c] += crow[c];  // the segments of a long K, in order
                  crow[c] = several && S.nsplit == 1 && k1 == ke ? scale_pow2(v[c], e_i + ej[c] + kUnit) : v[c];
                }
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

}  // namespace

void launch_tc_gemm_split(const TcSector* secs, const int4* items, int nitems, const uint8_t* ws,
                          const unsigned long long* ea, const unsigned long long* eb, double* C, double* part,
                          int* err, int grid, cudaStream_t s) {
  constexpr size_t smem = (size_t)kARing * kATile + (size_t)kBRing * kDigits * kBTile + 1024;
  static PerDevice attr;
  allow_smem(attr, current_device(), tc_gemm_split, smem);
  tc_gemm_split<<<grid, kThreadsSplit, smem, s>>>(secs, items, nitems, ws, ea, eb, C, part, err);
  TN_CUDA(cudaGetLastError());
}

}  // namespace tn
