// Operands of the tensor-core sector GEMMs for sm_103a: their row / column
// maxima and digit images in every mode, and the sum over K ranges.  The GEMMs
// are gemm_tc_split.cu (split precision) and gemm_tc_fast.cu (BF16, TF32).
//
// Split precision (TN_MODE_SPLIT): six FP16 digit images per operand tile
// (tc_digits.cuh).
// Fast BF16 (TN_MODE_FAST_BF16): one image, the BF16 rounding of each scaled
// element.
// Fast TF32 (TN_MODE_FAST_TF32, NS = 2 below): the TF32 rounding of each scaled
// element; a 64-k tile of 4-byte operands is two 128-byte swizzle atoms, stored
// as two 16 KB (A) / 8 KB (B) images (k 0..31, then 32..63).
//
// Layout: operand tiles are written as exact images of the tcgen05
// shared-memory operand layout (K-major, 128-byte swizzle), so the GEMMs move
// each with one 1-D bulk copy.  A tile: 128 rows x 64 k (16 KB per image); B
// tile: 64 columns x 64 k (8 KB per image).
#include <cuda_bf16.h>

#include <cstdint>

#include "../engine/engine.h"
#include "sm103_ptx.cuh"
#include "tc_digits.cuh"

namespace tn {
namespace {

using namespace ptx;

constexpr int kTM = 128, kTN = 64, kTK = 64;
constexpr int kATile = kTM * kTK * 2;  // bytes of one A slice tile
constexpr int kBTile = kTN * kTK * 2;  // bytes of one B slice tile

__device__ __forceinline__ int find_seg(const int64_t* __restrict__ start, int n, int64_t v) {
  int lo = 0, hi = n - 1;  // largest i with start[i] <= v
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= v)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------- exponents
// Largest |x| per row of A and per column of B, kept as IEEE bit patterns
// (for non-negative doubles the bit order is the value order).  Every operand
// tile (the same tiling as the slicing) reduces its part and merges it with a
// 64-bit atomicMax, so large-K operands spread over the whole GPU; the arrays
// are zeroed first.
__global__ void __launch_bounds__(256) tc_maxima(const TcSector* __restrict__ secs, const int64_t* __restrict__ a_ts,
                                                 const int64_t* __restrict__ b_ts, int nsec, int64_t a_tiles,
                                                 int64_t b_tiles, const double* __restrict__ A,
                                                 const double* __restrict__ B, unsigned long long* __restrict__ amax,
                                                 unsigned long long* __restrict__ bmax) {
  __shared__ unsigned long long part[4][kTN];
  if (threadIdx.x < kTN) part[0][threadIdx.x] = 0;
  __syncthreads();
  for (int64_t t = blockIdx.x; t < a_tiles + b_tiles; t += gridDim.x) {
    if (t < a_tiles) {
      const int g = find_seg(a_ts, nsec, t);
      const TcSector& S = secs[g];
      const int64_t local = t - a_ts[g];
      const int mt = (int)(local / S.nkt), kt = (int)(local % S.nkt);
      for (int r0 = 0; r0 < kTM; r0 += 32) {  // 8 lanes per row, 32 rows per pass
        const int r = r0 + (threadIdx.x >> 3), c = threadIdx.x & 7;
        const int64_t i = (int64_t)mt * kTM + r;
        unsigned long long m = 0;
        if (i < S.M) {
          const unsigned long long* src = (const unsigned long long*)(A + S.a_off + i * S.K);
          const int k0 = kt * kTK + c * 8;
#pragma unroll
          for (int q = 0; q < 8; q++)
            if (k0 + q < S.K) {
              const unsigned long long v = __ldg(src + k0 + q) & 0x7FFFFFFFFFFFFFFFull;
              m = v > m ? v : m;
            }
        }
#pragma unroll
        for (int o = 4; o; o >>= 1) {
          const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
          m = v > m ? v : m;
        }
        if (c == 0 && i < S.M && m) atomicMax(amax + S.ea_off + i, m);
      }
    } else {
      const int64_t u = t - a_tiles;
      const int g = find_seg(b_ts, nsec, u);
      const TcSector& S = secs[g];
      const int64_t local = u - b_ts[g];
      const int nt = (int)(local / S.nkt), kt = (int)(local % S.nkt);
      const int n0 = nt * kTN, k0 = kt * kTK;
      const int w = min(kTN, S.N - n0), h = min(kTK, S.K - k0);
      // flat walk of the h x w block: consecutive threads read consecutive
      // addresses even when the sector is narrower than the tile
      unsigned long long m = 0;
      int col = -1;
      for (int f = threadIdx.x; f < h * w; f += blockDim.x) {
        const int k = f / w, n = f - k * w;
        const unsigned long long v =
            __ldg((const unsigned long long*)(B + S.b_off) + (int64_t)(k0 + k) * S.N + n0 + n) & 0x7FFFFFFFFFFFFFFFull;
        if (n != col) {  // flush the running maximum of the previous column
          if (col >= 0 && m) atomicMax((unsigned long long*)&part[0][col], m);
          col = n;
          m = 0;
        }
        m = v > m ? v : m;
      }
      // part[0][n] doubles as the per-tile column maximum (zeroed below)
      if (col >= 0 && m) atomicMax((unsigned long long*)&part[0][col], m);
      __syncthreads();
      if (threadIdx.x < w && part[0][threadIdx.x]) atomicMax(bmax + S.eb_off + n0 + threadIdx.x, part[0][threadIdx.x]);
      __syncthreads();
      if (threadIdx.x < kTN) part[0][threadIdx.x] = 0;
      __syncthreads();
    }
  }
}

// 8 consecutive k (chunk c of a 64-k tile) of image row r: the NS digit
// slices (split, BF16 fast) at chunk c of every image, or (TF32, NS = 2) the
// two 16-byte halves at chunks 2 (c & 3) and 2 (c & 3) + 1 of image c >> 2
template <int NS>
__device__ __forceinline__ void store_chunk(uint8_t* img, int img_bytes, int r, int c, const double (&x)[8], int e) {
  if constexpr (NS == 2) {
    uint4 o[2];
    make_tf32(x, e, o);
    uint8_t* at = img + (int64_t)(c >> 2) * img_bytes;
    *(uint4*)(at + swz_off(r, 2 * (c & 3))) = o[0];
    *(uint4*)(at + swz_off(r, 2 * (c & 3) + 1)) = o[1];
  } else {
    uint4 o[NS];
    if constexpr (NS == 6)
      make_digits(x, e, o);
    else
      make_slices<NS>(x, e, o);
    const uint32_t off = swz_off(r, c);
#pragma unroll
    for (int s = 0; s < NS; s++) *(uint4*)(img + (int64_t)s * img_bytes + off) = o[s];
  }
}

// A tile t: (sector, mt, kt) -> NS images of 128 rows x 64 k
template <int NS>
__device__ __forceinline__ void slice_a_tile(const TcSector* __restrict__ secs, const int64_t* __restrict__ tstart,
                                             int nsec, int64_t t, const double* __restrict__ A,
                                             const unsigned long long* __restrict__ ea, uint8_t* __restrict__ ws) {
  {
    const int g = find_seg(tstart, nsec, t);
    const TcSector& S = secs[g];
    const int64_t local = t - tstart[g];
    const int mt = (int)(local / S.nkt), kt = (int)(local % S.nkt);
    uint8_t* img = ws + S.a_img + (int64_t)local * NS * kATile;
    for (int u = threadIdx.x; u < kTM * 8; u += blockDim.x) {
      const int r = u >> 3, c = u & 7;  // row within tile, 8-element chunk
      const int64_t i = (int64_t)mt * kTM + r;
      const int k0 = kt * kTK + c * 8;
      double x[8];
      int e = 0;
      if (i < S.M) {
        e = exp_of(ea[S.ea_off + i]);
        const double* src = A + S.a_off + i * S.K;
#pragma unroll
        for (int q = 0; q < 8; q++) x[q] = (k0 + q < S.K) ? __ldg(src + k0 + q) : 0.0;
      } else {
#pragma unroll
        for (int q = 0; q < 8; q++) x[q] = 0.0;
      }
      store_chunk<NS>(img, kATile, r, c, x, e);
    }
  }
}

// The column that row r of a B image holds.  The GEMMs' epilogues read their
// accumulators in the tcgen05 16 x 256b fragment order, where a thread of a
// group of four has columns 2 p, 2 p + 1, 8 + 2 p and 9 + 2 p of 16: with the
// columns in this order they are 4 p .. 4 p + 3, and it stores 32 bytes, four
// threads the 128 bytes of a row.
__device__ __forceinline__ int image_column(int r) {
  return (r & ~15) | ((r & 6) << 1) | ((r & 8) >> 2) | (r & 1);
}

// B tile t: (sector, nt, kt) -> NS images of 64 columns (rows of the image) x 64 k.
// The FP64 block is first staged in shared memory with flat coalesced loads,
// then each thread slices 8 consecutive k of one column.
template <int NS>
__device__ __forceinline__ void slice_b_tile(const TcSector* __restrict__ secs, const int64_t* __restrict__ tstart,
                                             int nsec, int64_t t, const double* __restrict__ B,
                                             const unsigned long long* __restrict__ eb, uint8_t* __restrict__ ws,
                                             double (*stage)[kTN + 1]) {
  const int g = find_seg(tstart, nsec, t);
  const TcSector& S = secs[g];
  const int64_t local = t - tstart[g];
  const int nt = (int)(local / S.nkt), kt = (int)(local % S.nkt);
  const int n0 = nt * kTN, k0 = kt * kTK;
  const int w = min(kTN, S.N - n0), h = min(kTK, S.K - k0);
  __syncthreads();  // the stage is reused tile after tile
  for (int f = threadIdx.x; f < kTK * kTN; f += blockDim.x) {
    const int k = f / kTN, n = f - k * kTN;
    stage[k][n] = 0.0;
  }
  __syncthreads();
  for (int f = threadIdx.x; f < h * w; f += blockDim.x) {
    const int k = f / w, n = f - k * w;
    stage[k][n] = __ldg(B + S.b_off + (int64_t)(k0 + k) * S.N + n0 + n);
  }
  __syncthreads();
  uint8_t* img = ws + S.b_img + (int64_t)local * NS * kBTile;
  for (int u = threadIdx.x; u < kTN * 8; u += blockDim.x) {
    const int r = u % kTN, c = u / kTN, n = image_column(r);
    int e = 0;
    if (n < w) e = exp_of(eb[S.eb_off + n0 + n]);
    double x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = stage[c * 8 + q][n];
    store_chunk<NS>(img, kBTile, r, c, x, e);
  }
}

// ---------------------------------------------------------------- one pass
// Maxima and images of an operand in one kernel: an item is 8 rows of A (a warp
// each; one row beyond kRowWarp k) or a strip of 16 columns of B, over all of
// K.  What an item holds in shared memory (74 KB, three CTAs per SM: rows of
// up to kRowKeep k per warp or 8192 per CTA, strips of up to kWideK) is read from
// memory once; longer rows are read again, through L2.  A strip of more k is
// shared by the 2 or 4 CTAs that hold it together (the rest of its k, from 2304
// on, is read again), which exchange their maxima through distributed shared
// memory; a cluster of 4 leaves few SM slots empty, one of 8 every ninth.  8192
// columns of 4096 beside 1024 rows: 225 -> 169 us against a strip per CTA (whose
// second reads no longer found 240 MB of strips in flight in L2), 1024
// contractions of bonds 16..256 1507 -> 1061 us.
// Staging is by cp.async, 16 bytes a copy where the row (the strip's rows) starts
// on 16 bytes, else 8; a thread then slices 8 consecutive k.  8 bytes are read and
// 2 bytes per digit written per element, 4.9 TB/s on 80000 rows of 400 in split
// precision, 5.6 as columns (4.2 with 8-byte copies and reads and a digit at a
// time): the instructions per element decide (107 there), not the loads' latency
// - bringing the next item into L2 ahead made it slower.  Only what the GEMM uses
// is written: no row past M or column past N (accumulator rows and columns nobody
// reads), no k past the last 16-k step.
constexpr int kStageDoubles = 9216, kRowKeep = 1024, kWideK = kSliceWideK;
// 18 doubles per 16: 16-byte reads of 8 consecutive k per lane without bank conflicts
__host__ __device__ constexpr int padded(int k) { return k + (k >> 4 << 1); }
static_assert(8 * padded(kRowKeep) <= kStageDoubles && padded(8192) <= kStageDoubles && 16 * kWideK <= kStageDoubles,
              "the staged extents fit");

struct SliceShared {
  uint32_t part[8][16];
  uint32_t peer[2][16];  // this CTA's maxima of a shared strip, for its group
  unsigned long long full[16];
};

__device__ __forceinline__ uint32_t abs_hi(double x) { return (uint32_t)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// Row i of A by the lanes id, id + n, .. of a warp (n = 32) or a CTA (n = 256).
// Only the exponent field of the maximum matters (exp_of), so the high words
// are compared; a row of zeros and subnormals takes the full patterns.
template <int NS, int n>
__device__ __forceinline__ void slice_row(const TcSector& S, int64_t i, int id, const double* __restrict__ A,
                                          unsigned long long* __restrict__ ea, uint8_t* __restrict__ ws, double* buf,
                                          SliceShared& sh) {
  constexpr int keep_k = n == 32 ? kRowKeep : 8192, half = keep_k / 2;
  auto sync = [] {
    if (n == 32)
      __syncwarp();
    else
      __syncthreads();
  };
  const double* src = A + S.a_off + i * S.K;
  const int kend = (S.K + 15) & ~15;  // the last 16-k step
  uint8_t* img = ws + S.a_img + (i / kTM) * S.nkt * NS * kATile;
  const int r = (int)(i % kTM);
  const bool keep = kend <= keep_k;
  // k0 .. k0 + len - 1 (zero past K) on their way into the buffer at `at`
  const bool wide = ((uintptr_t)src & 15) == 0;  // two doubles a copy
  auto stage = [&](int k0, int len, int at) {
    const int end = min(len, kend - k0), left = S.K - k0;
    if (wide) {
#pragma unroll 4
      for (int k = 2 * id; k < end; k += 2 * n)
        cp_async16(buf + padded(at + k), k < left ? src + k0 + k : src, k < left ? min(16, 8 * (left - k)) : 0);
    } else {
      for (int k = id; k < end; k += n)
        cp_async8(buf + padded(at + k), k < left ? src + k0 + k : src, k < left);
    }
    cp_async_commit();
  };
  auto read8 = [&](int k, double(&x)[8]) {  // k a multiple of 8
    const double2* p = (const double2*)(buf + padded(k));
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const double2 v = p[q];
      x[2 * q] = v.x, x[2 * q + 1] = v.y;
    }
  };
  uint32_t hi = 0;
  if (keep) {
    sync();  // the buffer's last contents have been read
    stage(0, keep_k, 0);
    cp_async_wait<0>();
    sync();
    for (int k = id * 8; k < kend; k += 8 * n) {
      double x[8];
      read8(k, x);
#pragma unroll
      for (int q = 0; q < 8; q++) hi = max(hi, abs_hi(x[q]));
    }
  } else {
    sync();
    stage(0, half, 0);  // the first half buffer loads while the maximum is taken
#pragma unroll 16
    for (int k = id; k < S.K; k += n) hi = max(hi, abs_hi(__ldg(src + k)));
  }
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (n > 32) {
    if ((id & 31) == 0) sh.part[id >> 5][0] = hi;
    if (id == 0) sh.full[0] = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < n / 32; w++) hi = max(hi, sh.part[w][0]);
  }
  unsigned long long m = (unsigned long long)hi << 32;
  if ((hi >> 20) == 0) {
    m = 0;
    for (int k = id; k < S.K; k += n) m = max(m, abs_bits(__ldg(src + k)));
    if (n == 32) {
#pragma unroll
      for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    } else {
      if (m) atomicMax(&sh.full[0], m);
      __syncthreads();
      m = sh.full[0];
    }
  }
  if (id == 0) ea[S.ea_off + i] = m;
  const int e = exp_of(m);
  auto slice = [&](int k0, int len, int at) {
    for (int k = id * 8; k < min(len, kend - k0); k += 8 * n) {
      double x[8];
      read8(at + k, x);
      store_chunk<NS>(img + (int64_t)((k0 + k) / kTK) * NS * kATile, kATile, r, (k / 8) % 8, x, e);
    }
  };
  if (keep) {
    slice(0, keep_k, 0);
  } else {  // half buffers in turn: one loads (from L2) while the other is sliced
    for (int k0 = 0, at = 0; k0 < kend; k0 += half, at ^= half) {
      stage(k0 + half, half, at ^ half);
      cp_async_wait<1>();
      sync();
      slice(k0, half, at);
      sync();
    }
    cp_async_wait<0>();
  }
}

// where a B image keeps column n of its 64 (image_column's inverse)
__device__ __forceinline__ int image_row(int n) {
  return (n & ~15) | ((n & 2) << 2) | ((n & 12) >> 1) | (n & 1);
}

// 16 columns of B, their k kb .. ke - 1 (multiples of 16, or the end) by this
// CTA: thread (c, g) slices of column c the groups g, g + 16, .. of 8 k.  SHARED:
// the strip's ranges are those of `group` CTAs of the cluster; they exchange
// their maxima (through buffer `par` in turn, so one barrier an item is enough).
template <int NS, bool SHARED>
__device__ __forceinline__ void slice_strip(const TcSector& S, int64_t strip, int kb, int ke, int group, int par,
                                            const double* __restrict__ B, unsigned long long* __restrict__ eb,
                                            uint8_t* __restrict__ ws, double* buf, SliceShared& sh) {
  constexpr int W = 16, kPass = 8 * 256 / W;
  const int c = threadIdx.x % W, g = threadIdx.x / W, warp = threadIdx.x >> 5;
  const int64_t n = strip * W + c;
  const int cols = n < S.N ? S.K : 0;  // k values this thread's column has
  const double* src = B + S.b_off + n;
  const int ks = SHARED ? min(ke, kb + kWideK) : ke;  // up to here it is staged
  auto at = [&](int k) { return (k - kb) * W + c; };
  auto load = [&](int k, double(&v)[8]) {
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = k + q < cols ? __ldg(src + (int64_t)(k + q) * S.N) : 0.0;
  };
  uint32_t hi = 0;
  const double* s0 = B + S.b_off + strip * W;
  if (strip * W + W <= S.N && ((uintptr_t)s0 & 15) == 0 && (S.N & 1) == 0) {  // two columns a copy
    const int p = 2 * (threadIdx.x & 7);
#pragma unroll 4
    for (int k = kb + (threadIdx.x >> 3); k < ks; k += 32)
      cp_async16(buf + (k - kb) * W + p, k < S.K ? s0 + (int64_t)k * S.N + p : s0, k < S.K ? 16 : 0);
  } else {
    for (int k = kb + g; k < ks; k += 16)
      cp_async8(buf + at(k), k < cols ? src + (int64_t)k * S.N : B + S.b_off, k < cols);
  }
  cp_async_commit();
  if (SHARED)
    for (int k = ks + g * 8; k < ke; k += 2 * kPass) {  // 16 loads in flight
      double x[8], y[8];
      load(k, x);
      load(k + kPass, y);
#pragma unroll
      for (int q = 0; q < 8; q++) hi = max(hi, max(abs_hi(x[q]), abs_hi(y[q])));
    }
  cp_async_wait<0>();
  __syncthreads();
  for (int k = kb + g * 8; k < ks; k += kPass)
#pragma unroll
    for (int q = 0; q < 8; q++) hi = max(hi, abs_hi(buf[at(k + q)]));
#pragma unroll
  for (int o = W; o < 32; o <<= 1) hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  __syncthreads();  // the previous item's maxima have been read
  if ((threadIdx.x & 31) < W) sh.part[warp][c] = hi;
  if (threadIdx.x < W) sh.full[c] = 0;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; w++) hi = max(hi, sh.part[w][c]);
  if (SHARED) {
    if (threadIdx.x < W) sh.peer[par][c] = hi;
    cluster_sync();
    const uint32_t rank = cluster_rank(), first = rank - rank % group;
    for (int p = 0; p < group; p++) hi = max(hi, ld_cluster(&sh.peer[par][c], first + p));
  }
  const bool low = (hi >> 20) == 0;  // zero or subnormal column: the full pattern decides
  if (low) {
    unsigned long long m = 0;
    for (int k = g; k < cols; k += 256 / W) m = max(m, abs_bits(__ldg(src + (int64_t)k * S.N)));
    if (m) atomicMax(&sh.full[c], m);
  }
  __syncthreads();
  const unsigned long long m = low ? sh.full[c] : (unsigned long long)hi << 32;
  if (g == 0 && n < S.N && kb == 0) eb[S.eb_off + n] = m;
  if (n >= S.N) return;
  const int e = exp_of(m);
  uint8_t* img = ws + S.b_img + (n / kTN) * S.nkt * NS * kBTile;
  const int r = image_row((int)(n % kTN));
  double x[8];
  for (int k = kb + g * 8; k < ks; k += kPass) {
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = buf[at(k + q)];
    store_chunk<NS>(img + (int64_t)(k / kTK) * NS * kBTile, kBTile, r, (k / 8) % 8, x, e);
  }
  if (SHARED) {
    load(ks + g * 8, x);
    for (int k = ks + g * 8; k < ke; k += kPass) {  // the next group loads while this one is sliced
      double y[8];
      load(k + kPass, y);
      store_chunk<NS>(img + (int64_t)(k / kTK) * NS * kBTile, kBTile, r, (k / 8) % 8, x, e);
#pragma unroll
      for (int q = 0; q < 8; q++) x[q] = y[q];
    }
  }
}

// items: the shared ones (sector, first of the strips that a cluster takes at
// once), then (sector, strip of B), or (sector, -1 - row group of A)
template <int NS, bool SHARED>
__global__ void __launch_bounds__(256, 3) tc_slice_once(const TcSector* __restrict__ secs,
                                                        const int2* __restrict__ items, int nshared, int nitems,
                                                        const double* __restrict__ A, const double* __restrict__ B,
                                                        unsigned long long* __restrict__ ea,
                                                        unsigned long long* __restrict__ eb, uint8_t* __restrict__ ws) {
  __shared__ SliceShared sh;
  extern __shared__ __align__(16) double stage[];  // kStageDoubles
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool cta = false;  // the last item used the buffer as a CTA
  int t0 = blockIdx.x;
  if (SHARED) {
    const int rank = (int)cluster_rank(), clusters = gridDim.x / kSliceCluster;
    int par = 0;
    for (int t = blockIdx.x / kSliceCluster; t < nshared; t += clusters, par ^= 1) {
      const int2 it = items[t];
      const TcSector& S = secs[it.x];
      const int kend = (S.K + 15) & ~15, group = slice_group(S.K), kper = ((kend >> 4) + group - 1) / group * 16;
      const int kb = rank % group * kper;
      __syncthreads();
      slice_strip<NS, true>(S, it.y + rank / group, kb, max(kb, min(kend, kb + kper)), group, par, B, eb, ws, stage, sh);
    }
    cta = true;
    cluster_sync();  // the peers have read this CTA's maxima
    // clusters that had one shared item less take the first of the others
    t0 = (int)((blockIdx.x + gridDim.x - nshared % clusters * kSliceCluster) % gridDim.x);
  }
  items += nshared;
  int2 next = t0 < nitems ? items[t0] : make_int2(0, 0);
  for (int t = t0; t < nitems; t += gridDim.x) {
    const int2 it = next;
    if (t + gridDim.x < nitems) next = items[t + gridDim.x];
    const TcSector& S = secs[it.x];
    if (it.y >= 0) {
      __syncthreads();
      slice_strip<NS, false>(S, it.y, 0, (S.K + 15) & ~15, 1, 0, B, eb, ws, stage, sh);
      cta = true;
    } else if (S.K > kRowWarp) {
      __syncthreads();
      slice_row<NS, 256>(S, -1 - it.y, threadIdx.x, A, ea, ws, stage, sh);
      cta = true;
    } else {
      if (cta) __syncthreads();
      cta = false;
      const int64_t i = (int64_t)(-1 - it.y) * 8 + warp;
      if (i < S.M) slice_row<NS, 32>(S, i, lane, A, ea, ws, stage + warp * padded(kRowKeep), sh);
    }
  }
}

// every A tile, then every B tile, in one launch (after tc_maxima)
template <int NS>
__global__ void __launch_bounds__(256) tc_slices(const TcSector* __restrict__ secs, const int64_t* __restrict__ a_ts,
                                                 const int64_t* __restrict__ b_ts, int nsec, int64_t a_tiles,
                                                 int64_t b_tiles, const double* __restrict__ A,
                                                 const double* __restrict__ B, const unsigned long long* __restrict__ ea,
                                                 const unsigned long long* __restrict__ eb, uint8_t* __restrict__ ws) {
  __shared__ double stage[kTK][kTN + 1];
  for (int64_t t = blockIdx.x; t < a_tiles + b_tiles; t += gridDim.x) {
    if (t < a_tiles)
      slice_a_tile<NS>(secs, a_ts, nsec, t, A, ea, ws);
    else
      slice_b_tile<NS>(secs, b_ts, nsec, t - a_tiles, B, eb, ws, stage);
  }
}

// ---------------------------------------------------------------- K ranges
// C = the sum of an output tile's partial tiles in K-range order, scaled by
// 2^(ea + eb - unit) (the split kernel's partial tiles carry no unit).  A tile is
// cut into `parts` bands of rows, an item each, as far as it takes to fill the
// chip: the ranges are summed one after another, and with few tiles (which is
// where ranges come from) a CTA per tile read up to 64 of them by itself.
// 32 tiles of 19 ranges 89 -> 13 us, 2 tiles of 53 ranges 270 -> 27.
constexpr int kReduceParts = 32;  // at most: one output per thread
__global__ void __launch_bounds__(256) tc_reduce(const TcSector* __restrict__ secs, const int4* __restrict__ ritems,
                                                 int nred, int parts, const double* __restrict__ part,
                                                 double* __restrict__ C, const unsigned long long* __restrict__ ea,
                                                 const unsigned long long* __restrict__ eb, int unit) {
  const int band = kTM * kTN / parts;
  for (int it = blockIdx.x; it < nred * parts; it += gridDim.x) {
    const int4 w = ritems[it / parts];
    const TcSector& S = secs[w.x];
    const double* p = part + S.p_off + ((int64_t)w.y * S.nnt + w.z) * S.nsplit * (kTM * kTN);
    const int e0 = it % parts * band;
    for (int e = e0 + threadIdx.x; e < e0 + band; e += 256) {
      const int64_t i = (int64_t)w.y * kTM + e / kTN, j = (int64_t)w.z * kTN + e % kTN;
      if (i >= S.M || j >= S.N) continue;
      double s = 0.0;
#pragma unroll 8
      for (int q = 0; q < S.nsplit; q++) s += __ldg(p + (int64_t)q * (kTM * kTN) + e);
      C[S.c_off + i * S.N + j] = scale_pow2(s, exp_of(ea[S.ea_off + i]) + exp_of(eb[S.eb_off + j]) - unit);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------- launchers
void launch_tc_maxima(const TcSector* secs, int nsec, const int64_t* a_ts, int64_t a_tiles, const int64_t* b_ts,
                      int64_t b_tiles, const double* A, const double* B, unsigned long long* amax,
                      unsigned long long* bmax, int64_t nmax, int num_sms, cudaStream_t s) {
  TN_CUDA(cudaMemsetAsync(amax, 0, (size_t)nmax * sizeof(unsigned long long), s));  // bmax follows amax
  int g1 = (int)std::min<int64_t>(a_tiles + b_tiles, (int64_t)num_sms * 8);
  tc_maxima<<<g1, 256, 0, s>>>(secs, a_ts, b_ts, nsec, a_tiles, b_tiles, A, B, amax, bmax);
  TN_CUDA(cudaGetLastError());
}

template <int NS>
static void launch_once(const TcSector* secs, const int2* items, int nshared, int nitems, const double* A,
                        const double* B, unsigned long long* ea, unsigned long long* eb, uint8_t* images, int num_sms,
                        cudaStream_t s) {
  constexpr int smem = kStageDoubles * (int)sizeof(double);
  if (!nshared) {
    static PerDevice attr;
    allow_smem(attr, current_device(), tc_slice_once<NS, false>, smem);
    tc_slice_once<NS, false>
        <<<std::min(nitems, num_sms * 3), 256, smem, s>>>(secs, items, 0, nitems, A, B, ea, eb, images);
    TN_CUDA(cudaGetLastError());
    return;
  }
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kSliceCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)(num_sms * 3 / kSliceCluster * kSliceCluster));
  static PerDevice fit;  // clusters the GPU holds at once
  const int resident = fit.get(current_device(), [&] {
    TN_CUDA(cudaFuncSetAttribute(tc_slice_once<NS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int n = 0;
    TN_CUDA(cudaOccupancyMaxActiveClusters(&n, tc_slice_once<NS, true>, &cfg));
    return std::max(1, n);
  });
  const int clusters = std::min(resident, std::max(nshared, (nitems + kSliceCluster - 1) / kSliceCluster));
  cfg.gridDim = dim3((unsigned)(clusters * kSliceCluster));
  TN_CUDA(cudaLaunchKernelEx(&cfg, tc_slice_once<NS, true>, secs, items, nshared, nitems, A, B, ea, eb, images));
}

void launch_tc_slice_once(int ns, const TcSector* secs, const int2* items, int nshared, int nitems, const double* A,
                          const double* B, unsigned long long* ea, unsigned long long* eb, uint8_t* images,
                          int num_sms, cudaStream_t s) {
  auto launch = ns == kSplitDigits ? launch_once<kSplitDigits> : (ns == 2 ? launch_once<2> : launch_once<1>);
  launch(secs, items, nshared, nitems, A, B, ea, eb, images, num_sms, s);
}

void launch_tc_slices(int ns, const TcSector* secs, int nsec, const int64_t* a_ts, int64_t a_tiles,
                      const int64_t* b_ts, int64_t b_tiles, const double* A, const double* B,
                      const unsigned long long* amax, const unsigned long long* bmax, uint8_t* images, int num_sms,
                      cudaStream_t s) {
  int g2 = (int)std::min<int64_t>(a_tiles + b_tiles, (int64_t)num_sms * 8);
  if (ns == kSplitDigits)
    tc_slices<kSplitDigits><<<g2, 256, 0, s>>>(secs, a_ts, b_ts, nsec, a_tiles, b_tiles, A, B, amax, bmax, images);
  else if (ns == 2)
    tc_slices<2><<<g2, 256, 0, s>>>(secs, a_ts, b_ts, nsec, a_tiles, b_tiles, A, B, amax, bmax, images);
  else
    tc_slices<1><<<g2, 256, 0, s>>>(secs, a_ts, b_ts, nsec, a_tiles, b_tiles, A, B, amax, bmax, images);
  TN_CUDA(cudaGetLastError());
}

void launch_tc_reduce(int ns, const TcSector* secs, const int4* ritems, int nred, const double* part, double* C,
                      const unsigned long long* ea, const unsigned long long* eb, int num_sms, cudaStream_t s) {
  if (nred <= 0) return;
  int parts = 1;
  while (parts < kReduceParts && (int64_t)nred * parts < 4 * num_sms) parts *= 2;
  const int grid = (int)std::min<int64_t>((int64_t)nred * parts, (int64_t)num_sms * 8);
  tc_reduce<<<grid, 256, 0, s>>>(secs, ritems, nred, parts, part, C, ea, eb, ns == kSplitDigits ? 0 : 14);
  TN_CUDA(cudaGetLastError());
}

}  // namespace tn
