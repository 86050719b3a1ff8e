// Plain FP64 grouped sector GEMM: every C_q = A_q . B_q
// of one contraction (contract's per-sector matrixMul,
// tensor-network/lib/UniTensorTools.cpp:191-203; row-major dgemm,
// numeric/lapack/lib/uni10_lapack_cpu.cpp:41-44) in one launch, a warp per work
// item.
//
// GB300's FP64 pipe takes a warp's FMA every 64 clocks per SM sub-partition
// (1.26 TFLOP/s for the chip), so what decides is how many of the 32 lanes
// carry a wanted product; loads and index arithmetic have an order of magnitude
// to spare.  A sector's outputs are therefore dealt to lanes one after another,
// (row, column) = (o / N, o % N), with no tile shape to pad to: an item is up
// to 4 slots of 32 consecutive outputs over a K range.  A lane then loads one
// element of A (its row's, a broadcast along the row's lanes) and one of B (a
// run of a row of B) per FMA, two loads where a 4-row tile column takes 1.25;
// at 16 clocks per warp FMA and SM the load pipe keeps up.  Sectors with few
// outputs deal (K range, output) pairs the same way, so 10 x 10 outputs fill
// 25 warps' lanes with 8 K ranges instead of a quarter of a 16 x 32 tile.
// Against tiles of 512 entries shaped to N (gemm_fp64.cu), lanes carrying
// products went from 0.75 to 0.97 on 1024 contractions of bonds 16..256
// (8 382 sectors, M and N about 30, K about 2 500).
//
// Measured against the tiles: that workload in one launch 8.75 -> 5.88 ms (0.755
// -> 1.12 TFLOP/s, of 1.26), 64 of its contractions 0.81 -> 0.38 ms, an iPEPS
// quadrant at chi = 64, D = 6 (sectors of 1152 x 36 .. 648 x 648 outputs) 3.19 ->
// 3.03 ms, the captured iTEBD network at chi = 512 (operands through views)
// 42.4 -> 33.7 us; one output over K = 1e6 533 -> 23 us, 8 x 1 over 1e5 89 -> 21, 2 x 2
// over 3e5 248 -> 19, 10 x 10 over 1e6 1169 -> 393, 3 x 7 over 14786 24 -> 8.6, 100 sectors of
// 281 x 1 over 55 20.5 -> 12.3.  1 500 random lists: 0.59 of the tiles' time on average.
//
// Items that share outputs (K ranges) write partial sums to a workspace; the
// last one of a group adds them in a fixed order, so the result does not depend
// on the schedule: a lane per output in range order, or the lanes along the
// ranges where outputs are few (a dot product over K = 1e6, 488 ranges).  Launched with programmatic dependent launch (pdl.cuh): the
// first item and the view tables (plan data) are read before the wait on the
// previous grid.
#include "../engine/engine.h"
#include "pdl.cuh"

namespace tn {
namespace {

constexpr int kWarps = kFlatWarps;

__device__ __forceinline__ int find_start(const int64_t* __restrict__ st, int n, int64_t v) {
  int lo = 0, hi = n - 1;  // largest i with st[i] <= v
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (st[mid] <= v)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// acc[i] += sum over k < len of pa[i][k] pb[i][k ldb[i]], k ascending
template <int R>
__device__ __forceinline__ void fma_run(double (&acc)[R], const double* const (&pa)[R], const double* (&pb)[R],
                                        const int64_t (&ldb)[R], int len) {
  constexpr int U = R == 1 ? 8 : (R == 2 ? 4 : 2);  // loads in flight: a small item is their latency
  int k = 0;
  for (; k + U <= len; k += U) {
    double a[R][U], b[R][U];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int u = 0; u < U; u++) {
        a[i][u] = __ldg(pa[i] + k + u);
        b[i][u] = __ldg(pb[i] + u * ldb[i]);
      }
#pragma unroll
    for (int i = 0; i < R; i++) pb[i] += U * ldb[i];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int i = 0; i < R; i++) acc[i] = fma(a[i][u], b[i][u], acc[i]);
  }
  for (; k < len; k++)
#pragma unroll
    for (int i = 0; i < R; i++) {
      acc[i] = fma(__ldg(pa[i] + k), __ldg(pb[i]), acc[i]);
      pb[i] += ldb[i];
    }
}

// fma_run over a long range, kFlatChain products to a sum
template <int R>
__device__ __forceinline__ void fma_long(double (&acc)[R], const double* const (&pa)[R], const double* (&pb)[R],
                                         const int64_t (&ldb)[R], int len) {
  for (int k = 0; k < len; k += kFlatChain) {
    const double* pk[R];
    double part[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      pk[i] = pa[i] + k;
      part[i] = 0.0;
    }
    fma_run<R>(part, pk, pb, ldb, min(kFlatChain, len - k));
#pragma unroll
    for (int i = 0; i < R; i++) acc[i] += part[i];
  }
}

// Operands read through views of their unpermuted source (ViewHdr): the K range
// is walked in segments (the contracted bonds' charge tuples), each a plain
// row-major view per row (column) tuple.
template <int R, bool HUGE>
__device__ __forceinline__ void view_body(const FlatItem& t, int lane, const double* __restrict__ A,
                                          const double* __restrict__ B, double* __restrict__ C,
                                          double* __restrict__ ws, const ViewHdr* __restrict__ views,
                                          const int64_t* __restrict__ pool) {
  const ViewHdr* av = t.a_vw >= 0 ? views + t.a_vw : nullptr;
  const ViewHdr* bv = t.b_vw >= 0 ? views + t.b_vw : nullptr;
  const int slice = (int)((uint32_t)t.v0 / (uint32_t)t.mn);
  int out[R], m[R], n[R], ri[R], cj[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    out[i] = t.v0 - slice * t.mn + min(lane + 32 * i, t.nv - 1);
    m[i] = (int)((uint32_t)out[i] / (uint32_t)t.N);
    n[i] = out[i] - m[i] * t.N;
    ri[i] = av ? find_start(pool + av->rs, av->nr, m[i]) : 0;
    cj[i] = bv ? find_start(pool + bv->cs, bv->nc, n[i]) : 0;
  }
  // the column tuples of a viewed A (the row tuples of a viewed B are the same)
  const int64_t* seg = av ? pool + av->cs : pool + bv->rs;
  const int nseg = av ? av->nc : bv->nr;
  const int kb = slice * t.kc, ke = min(t.K, kb + t.kc);
  double acc[R], sum[R];
#pragma unroll
  for (int i = 0; i < R; i++) acc[i] = sum[i] = 0.0;
  int s = find_start(seg, nseg, kb);
  pdl_wait();  // A, B, C and ws may be written by the previous grid
  for (int k0 = kb, chain0 = kb; k0 < ke;) {
    const int s0 = (int)seg[s], s1 = (int)min((int64_t)ke, seg[s + 1]), k1 = HUGE ? min(s1, chain0 + kFlatChain) : s1;
    const double *pa[R], *pb[R];
    int64_t ldb[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      if (av) {
        const int64_t* pr = pool + av->tab + 2 * ((int64_t)ri[i] * av->nc + s);
        pa[i] = A + pr[0] + (m[i] - pool[av->rs + ri[i]]) * pr[1] + (k0 - s0);
      } else {
        pa[i] = A + t.a_off + (int64_t)m[i] * t.K + k0;
      }
      if (bv) {
        const int64_t* pr = pool + bv->tab + 2 * ((int64_t)s * bv->nc + cj[i]);
        ldb[i] = pr[1];
        pb[i] = B + pr[0] + (n[i] - pool[bv->cs + cj[i]]) + (k0 - s0) * pr[1];
      } else {
        ldb[i] = t.N;
        pb[i] = B + t.b_off + (int64_t)k0 * t.N + n[i];
      }
    }
    fma_run<R>(acc, pa, pb, ldb, k1 - k0);
    k0 = k1;
    s += k1 == s1;
    if (HUGE && k1 == chain0 + kFlatChain) {  // short segments share a sum
#pragma unroll
      for (int i = 0; i < R; i++) {
        sum[i] += acc[i];
        acc[i] = 0.0;
      }
      chain0 = k1;
    }
  }
  if (HUGE)
#pragma unroll
    for (int i = 0; i < R; i++) acc[i] += sum[i];
#pragma unroll
  for (int i = 0; i < R; i++)
    if (lane + 32 * i < t.nv) {
      if (t.grp < 0)
        C[t.c_off + out[i]] = acc[i];
      else
        ws[t.ws_off + (int64_t)slice * t.gs + (out[i] - t.o0)] = acc[i];
    }
}

// R slots of 32 entries; UNI: all entries of the item in one K range
template <int R, bool UNI, bool HUGE>
__device__ __forceinline__ void flat_body(const FlatItem& t, int lane, const double* __restrict__ A,
                                          const double* __restrict__ B, double* __restrict__ C,
                                          double* __restrict__ ws) {
  const double *pa[R], *pb[R];
  int len[R];
  int32_t slice[R], out[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    const uint32_t v = (uint32_t)(t.v0 + min(lane + 32 * i, t.nv - 1));  // lanes past the end repeat the last entry
    slice[i] = UNI ? (int32_t)((uint32_t)t.v0 / (uint32_t)t.mn) : (int32_t)(v / (uint32_t)t.mn);
    out[i] = (int32_t)(v - (uint32_t)slice[i] * (uint32_t)t.mn);
    const uint32_t m = (uint32_t)out[i] / (uint32_t)t.N, n = (uint32_t)out[i] - m * (uint32_t)t.N;
    const int k0 = slice[i] * t.kc;
    len[i] = min(t.kc, t.K - k0);
    pa[i] = A + t.a_off + (int64_t)m * t.K + k0;
    pb[i] = B + t.b_off + (int64_t)k0 * t.N + n;
  }
  double acc[R];
#pragma unroll
  for (int i = 0; i < R; i++) acc[i] = 0.0;
  int64_t ldb[R];
#pragma unroll
  for (int i = 0; i < R; i++) ldb[i] = t.N;
  pdl_wait();  // A, B, C and ws may be written by the previous grid
  if (UNI) {
    if (HUGE)
      fma_long<R>(acc, pa, pb, ldb, len[0]);
    else
      fma_run<R>(acc, pa, pb, ldb, len[0]);
  } else {  // the last K range may be shorter
    const int kmin = min(t.kc, t.K - (int)((uint32_t)(t.v0 + t.nv - 1) / (uint32_t)t.mn) * t.kc);
    if (HUGE)
      fma_long<R>(acc, pa, pb, ldb, kmin);
    else
      fma_run<R>(acc, pa, pb, ldb, kmin);
    for (int k = kmin; k < t.kc; k++) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        if (k < len[i]) acc[i] = fma(__ldg(pa[i] + k), __ldg(pb[i]), acc[i]);
        pb[i] += t.N;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; i++)
    if (lane + 32 * i < t.nv) {
      if (t.grp < 0)
        C[t.c_off + out[i]] = acc[i];
      else
        ws[t.ws_off + (int64_t)slice[i] * t.gs + (out[i] - t.o0)] = acc[i];
    }
}

// The sums over the lanes of V values, P = V rounded up to a power of two: while
// there are several, a lane keeps half of them and gives the other half away, so
// that four values cost 6 additions, not 20 (an addition holds the FP64 pipe as
// long as an FMA).  Lane j 32 / P returns the sum of value j.
template <int V, int P>
__device__ __forceinline__ double lane_sums(const double (&x)[V], int lane) {
  double v[P];
#pragma unroll
  for (int i = 0; i < P; i++) v[i] = i < V ? x[i] : 0.0;
  int o = 16;
#pragma unroll
  for (int s = P / 2; s > 0; s >>= 1, o >>= 1) {
    const bool high = lane & o;
#pragma unroll
    for (int i = 0; i < s; i++) {
      const double give = high ? v[i] : v[i + s], keep = high ? v[i + s] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// Sectors of few columns: lanes along K (A's row and B's rows read coalesced;
// flat lanes would gather 16 or 32 rows of A per load), the lanes' sums added by
// fixed shuffles; the item's entries are nv rows, RB of them at a time where there
// are as many (one row's loads and shuffles leave the warp waiting).
template <int NN, int RB, bool LONG>
__device__ __forceinline__ void row_block(const FlatItem& t, int m, int lane, const double* __restrict__ A,
                                          const double* __restrict__ B, double* __restrict__ C,
                                          double* __restrict__ ws) {
  const double* __restrict__ a = A + t.a_off + (int64_t)m * t.K;
  const double* __restrict__ b = B + t.b_off;
  const int k0 = LONG ? t.kq * t.kc : 0, k1 = LONG ? min(t.K, k0 + t.kc) : t.K;
  constexpr int V = RB * NN, P = V <= 2 ? V : (V <= 4 ? 4 : 8);
  double acc[V];
#pragma unroll
  for (int i = 0; i < V; i++) acc[i] = 0.0;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32) {
    double bv[NN];
#pragma unroll
    for (int n = 0; n < NN; n++) bv[n] = __ldg(b + (int64_t)k * NN + n);
#pragma unroll
    for (int r = 0; r < RB; r++) {
      const double av = __ldg(a + (int64_t)r * t.K + k);
#pragma unroll
      for (int n = 0; n < NN; n++) acc[r * NN + n] = fma(av, bv[n], acc[r * NN + n]);
    }
  }
  const double s = lane_sums<V, P>(acc, lane);
  const int j = lane / (32 / P);  // the rows of the block lie one after another
  if (lane % (32 / P) == 0 && j < V) {
    if (!LONG || t.grp < 0)
      C[t.c_off + (int64_t)m * NN + j] = s;
    else
      ws[t.ws_off + (int64_t)t.kq * t.gs + (m * NN + j - t.o0)] = s;
  }
}

template <int NN, bool LONG>
__device__ __forceinline__ void row_body(const FlatItem& t, int lane, const double* __restrict__ A,
                                         const double* __restrict__ B, double* __restrict__ C,
                                         double* __restrict__ ws) {
  constexpr int RB = NN == 1 ? 4 : (NN == 2 ? 2 : 1);
  pdl_wait();
  int m = t.v0;
  const int end = t.v0 + t.nv;
  for (; m + RB <= end; m += RB) row_block<NN, RB, LONG>(t, m, lane, A, B, C, ws);
  if (RB > 1)
    for (; m < end; m++) row_block<NN, 1, LONG>(t, m, lane, A, B, C, ws);
}

template <bool LONG>
__device__ __forceinline__ void row_dispatch(const FlatItem& t, int lane, const double* __restrict__ A,
                                             const double* __restrict__ B, double* __restrict__ C,
                                             double* __restrict__ ws) {
  if (t.N == 1) return row_body<1, LONG>(t, lane, A, B, C, ws);
  if (!LONG || t.N == 2) return row_body<2, LONG>(t, lane, A, B, C, ws);
  switch (t.N) {  // small lists only (plan_fp64_flat)
    case 3: return row_body<3, LONG>(t, lane, A, B, C, ws);
    case 4: return row_body<4, LONG>(t, lane, A, B, C, ws);
    case 5: return row_body<5, LONG>(t, lane, A, B, C, ws);
    case 6: return row_body<6, LONG>(t, lane, A, B, C, ws);
    case 7: return row_body<7, LONG>(t, lane, A, B, C, ws);
    default: return row_body<8, LONG>(t, lane, A, B, C, ws);
  }
}

template <bool UNI, bool HUGE>
__device__ __forceinline__ void flat_dispatch(const FlatItem& t, int lane, const double* __restrict__ A,
                                              const double* __restrict__ B, double* __restrict__ C,
                                              double* __restrict__ ws) {
  switch ((t.nv + 31) >> 5) {
    case 1: flat_body<1, UNI, HUGE>(t, lane, A, B, C, ws); break;
    case 2: flat_body<2, UNI, HUGE>(t, lane, A, B, C, ws); break;
    case 3: flat_body<3, UNI, HUGE>(t, lane, A, B, C, ws); break;
    default: flat_body<4, UNI, HUGE>(t, lane, A, B, C, ws); break;
  }
}

template <bool HUGE>
__device__ __forceinline__ void view_dispatch(const FlatItem& t, int lane, const double* __restrict__ A,
                                              const double* __restrict__ B, double* __restrict__ C,
                                              double* __restrict__ ws, const ViewHdr* __restrict__ views,
                                              const int64_t* __restrict__ pool) {
  if (t.nv <= 32)  // the planner gives these items at most kFlatViewSlots = 2 slots
    view_body<1, HUGE>(t, lane, A, B, C, ws, views, pool);
  else
    view_body<2, HUGE>(t, lane, A, B, C, ws, views, pool);
}

// VIEWS: some item reads an operand through views (a kernel of its own: with
// its registers the plain one would hold 4 CTAs per SM instead of 5, 20% slower
// on the batched workload).  LONG: some row is cut into K ranges, some group has
// more than kFlatFewRanges, or the list leaves warps idle, so that a group's sum
// is seen (a kernel of its own too: in one, lists without such a sector ran 1%
// longer, the batched workload 5.93 -> 6.01 ms).  HUGE: a list of 6e10
// multiply-adds and up with K ranges of more than kFlatChain, which are summed
// kFlatChain products at a time: with one sum to a range the relative error of 576
// x 576 over K = 331776 was 1.2e-15 -> 1.5e-14, now 1.0e-15 in the same 203 ms (in
// the LONG instance the breaks cost 100 x 300 over 20000 4%).
template <bool VIEWS, bool LONG, bool HUGE>
__global__ void __launch_bounds__(32 * kWarps, kFlatCtasPerSm)
    gemm_fp64_flat_kernel(const FlatItem* __restrict__ items, int nitems, const double* __restrict__ A,
                          const double* __restrict__ B, double* __restrict__ C, double* __restrict__ ws,
                          int* __restrict__ counters, const ViewHdr* __restrict__ views,
                          const int64_t* __restrict__ pool) {
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // neighbouring items share operands: the warps of a CTA take them together
  for (int it = blockIdx.x * kWarps + warp; it < nitems; it += gridDim.x * kWarps) {
    const FlatItem t = items[it];
    if (t.rows) {
      row_dispatch<LONG>(t, lane, A, B, C, ws);
      if (!LONG || t.grp < 0) continue;
    } else if (VIEWS && (t.a_vw >= 0 || t.b_vw >= 0))
      view_dispatch<HUGE>(t, lane, A, B, C, ws, views, pool);
    else if (t.v0 / t.mn == (t.v0 + t.nv - 1) / t.mn)
      flat_dispatch<true, HUGE>(t, lane, A, B, C, ws);
    else
      flat_dispatch<false, HUGE>(t, lane, A, B, C, ws);
    if (t.grp >= 0) {
      __threadfence();  // this lane's partial sums are visible device-wide
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(&counters[t.grp], 1) == t.cnt - 1;
      if (__shfl_sync(0xffffffffu, last, 0)) {
        __threadfence();
        const double* p = ws + t.ws_off;
        if (!LONG || t.go > 16 || t.nsplit <= 4) {
          for (int o = lane; o < t.go; o += 32) {
            double s = 0.0;
            for (int q = 0; q < t.nsplit; q++) s += __ldcg(p + (int64_t)q * t.gs + o);
            C[t.c_off + t.o0 + o] = s;
          }
        } else {  // few outputs of many ranges: 32 / w lanes along the ranges of each
          int w = 1;
          while (w < t.go) w *= 2;
          const int o = lane & (w - 1);
          double s = 0.0;
          if (o < t.go)
#pragma unroll 8
            for (int q = lane / w; q < t.nsplit; q += 32 / w) s += __ldcg(p + (int64_t)q * t.gs + o);
          for (int d = 16; d >= w; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
          if (lane < t.go) C[t.c_off + t.o0 + lane] = s;
        }
        if (lane == 0) counters[t.grp] = 0;  // for the next launch
      }
    }
  }
}

}  // namespace

void launch_gemm_fp64_flat(const FlatItem* items, int nitems, const double* A, const double* B, double* C, double* ws,
                           int* counters, const ViewHdr* views, const int64_t* pool, int form, int grid,
                           cudaStream_t s) {
  if (nitems <= 0) return;
  auto kernel = views ? (form == kFlatHuge   ? gemm_fp64_flat_kernel<true, true, true>
                         : form == kFlatLong ? gemm_fp64_flat_kernel<true, true, false>
                                             : gemm_fp64_flat_kernel<true, false, false>)
                      : (form == kFlatHuge   ? gemm_fp64_flat_kernel<false, true, true>
                         : form == kFlatLong ? gemm_fp64_flat_kernel<false, true, false>
                                             : gemm_fp64_flat_kernel<false, false, false>);
  launch_pdl(kernel, dim3(grid), dim3(32 * kWarps), 0, s, items, nitems, A, B, C, ws, counters, views, pool);
}

}  // namespace tn
