// One CTA of a tensor-core kernel on the CPU, for tests of what its warps wait
// for: every thread a fiber, mbarriers, bulk copies, tcgen05 MMAs, commits and
// tensor memory emulated, copies and MMAs completing at random times and in
// the orders the hardware allows.  The kernel's own source is compiled against
// this file; only the functions made of inline PTX are replaced by the ones
// below (the test cuts them out).
//
// Reported as failures: a copy outside the given global range, off its 16-byte
// alignment or into memory it may not write; a warp-wide instruction reached by
// part of a warp; tensor memory read or freed while an MMA is outstanding; a
// CTA that ends with copies or MMAs in flight or tensor memory held.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <random>
#include <string>
#include <vector>

namespace emu {

struct Idx {
  unsigned x, y, z;
};
struct Fiber {
  ucontext_t ctx;
  std::vector<char> stack;
  Idx tid;
  bool done = false;
  std::function<bool()> blocked;  // resumed when this is false (empty: runnable)
};

inline std::mt19937 rng(1);
inline uint32_t rnd(uint32_t n) { return (uint32_t)(rng() % n); }
inline std::string failure;
inline void check(bool ok, const char* what) {
  if (!ok && failure.empty()) failure = what;
}

inline std::vector<Fiber> fibers;
inline Fiber* cur = nullptr;
inline ucontext_t main_ctx;
inline Idx bid, gdim;
inline unsigned nthreads = 0;

inline void yield() { swapcontext(&cur->ctx, &main_ctx); }
inline void block(std::function<bool()> until) {
  cur->blocked = [until] { return !until(); };
  yield();
}

// ---- memory the asynchronous engines may touch
constexpr size_t kSmem = 230 * 1024;
alignas(1024) inline uint8_t smem[kSmem + 2048];
inline uint8_t* dyn = smem + 1024 + 256;  // an unaligned dynamic base, as after static shared memory
inline size_t dyn_bytes = 0;
inline const uint8_t* gmem0 = nullptr;
inline const uint8_t* gmem1 = nullptr;

// ---- time and faults injected on the host side
inline uint64_t clock_ns = 0;
inline int hold_copy = -1, hold_mma = -1;  // the n-th copy / MMA completes late (-1: none)
inline uint64_t hold_ns = 0;

// ---- mbarriers (8 bytes each)
struct Bar {
  uint8_t count, pending;
  uint16_t phase;
  int32_t tx;
};
static_assert(sizeof(Bar) == 8, "an mbarrier is 8 bytes");
inline Bar& bar(uint64_t* p) { return *(Bar*)p; }
inline void settle(Bar& b) {
  if (b.pending == 0 && b.tx == 0) {
    b.phase++;
    b.pending = b.count;
  }
}
inline void arrive(Bar& b) {
  check(b.pending > 0, "an arrival more than the barrier's count");
  b.pending--;
  settle(b);
}
inline bool complete(uint64_t* p, uint32_t parity) { return (bar(p).phase & 1) != parity; }

// ---- asynchronous engines
struct Copy {
  uint8_t* dst;
  const uint8_t* src;
  uint32_t bytes;
  uint64_t* bar;
  uint64_t not_before;
};
inline std::vector<Copy> copies;
inline std::deque<std::function<void()>> tensor;  // MMAs and commits, in order
inline uint64_t tensor_not_before = 0;
inline int n_copies = 0, n_mmas = 0, mmas_pending = 0;
inline float tmem[128][512];
inline int tmem_cols = 0;

inline bool engines_step() {
  bool any = false;
  if (!copies.empty()) {
    const size_t i = rnd((uint32_t)copies.size());
    Copy c = copies[i];
    if (clock_ns >= c.not_before) {
      copies.erase(copies.begin() + i);
      memcpy(c.dst, c.src, c.bytes);
      bar(c.bar).tx -= (int32_t)c.bytes;
      settle(bar(c.bar));
      any = true;
    }
  }
  if (!tensor.empty() && clock_ns >= tensor_not_before && rnd(2)) {
    auto f = tensor.front();
    tensor.pop_front();
    f();
    any = true;
  }
  return any;
}

// ---- a rendezvous of the 32 lanes of a warp
struct Meet {
  int arrived = 0;
  uint64_t gen = 0;
  uint64_t in[32], out[32];
  const char* what = "";
};
inline Meet meets[32];
inline unsigned tid() { return cur->tid.x; }
inline const uint64_t* meet(const char* what, uint64_t v) {
  Meet& m = meets[tid() / 32];
  check(m.arrived == 0 || !strcmp(m.what, what), "lanes of one warp at different warp-wide instructions");
  m.what = what;
  m.in[tid() % 32] = v;
  const uint64_t g = m.gen;
  if (++m.arrived == 32) {
    memcpy(m.out, m.in, sizeof(m.out));
    m.arrived = 0;
    m.gen++;
    // an arrival of the next one waits until every lane has read this one's
  } else {
    block([&m, g] { return m.gen != g; });
  }
  return m.out;
}
inline int sync_arrived = 0;
inline uint64_t sync_gen = 0;

// Runs one CTA; "" or what went wrong.
inline std::string run_cta(unsigned threads, unsigned b, unsigned grid, const std::function<void()>& kernel) {
  static std::function<void()> body;
  body = kernel;
  failure.clear();
  bid = {b, 0, 0};
  gdim = {grid, 1, 1};
  nthreads = threads;
  copies.clear();
  tensor.clear();
  n_copies = n_mmas = mmas_pending = 0;
  tensor_not_before = 0;
  clock_ns = 0;
  tmem_cols = 0;
  sync_arrived = 0;
  for (Meet& m : meets) m = Meet();
  for (auto& row : tmem)
    for (float& x : row) x = NAN;
  memset(smem, 0xFF, sizeof(smem));  // NaNs
  fibers.resize(threads);
  for (unsigned t = 0; t < threads; t++) {
    Fiber& f = fibers[t];
    f.stack.resize(192 * 1024);
    f.tid = {t, 0, 0};
    f.done = false;
    f.blocked = nullptr;
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.data();
    f.ctx.uc_stack.ss_size = f.stack.size();
    f.ctx.uc_link = &main_ctx;
    makecontext(&f.ctx, (void (*)())(+[] {
                  body();
                  cur->done = true;
                }),
                0);
  }
  uint64_t idle = 0;
  for (;;) {
    bool left = false, any = false;
    for (const Fiber& f : fibers) left |= !f.done;
    if (!left) break;
    const unsigned w0 = rnd(threads / 32);
    for (unsigned w = 0; w < threads / 32; w++) {
      const unsigned warp = (w0 + w) % (threads / 32);
      if (rnd(3) == 0) continue;
      const unsigned l0 = rnd(32), n = rnd(4) ? 32 : 1 + rnd(32);
      for (unsigned l = 0; l < 32; l++) {
        Fiber& f = fibers[warp * 32 + (l0 + l) % 32];
        if (f.done) continue;
        if (l >= n || (f.blocked && f.blocked())) continue;
        f.blocked = nullptr;
        cur = &f;
        swapcontext(&main_ctx, &f.ctx);
        any = true;
      }
      if (rnd(2)) any |= engines_step();
    }
    any |= engines_step();
    // time passes (a millisecond a round) only while something is held back
    bool held = clock_ns < tensor_not_before;
    for (const Copy& c : copies) held |= clock_ns < c.not_before;
    if (held) clock_ns += 1000000;
    if (!failure.empty()) return failure;
    idle = any ? 0 : idle + 1;
    if (idle > 2000) return "every thread waits and nothing is in flight";
  }
  check(copies.empty(), "the CTA ended with copies in flight");
  check(mmas_pending == 0, "the CTA ended with MMAs in flight");
  check(tensor.empty(), "the CTA ended with commits in flight");
  check(tmem_cols == 0, "the CTA ended with tensor memory held");
  return failure;
}

inline float tf32_at(uint32_t desc, int r, int k) {
  const uint32_t a = (desc & 0x3FFF) << 4;
  const uint32_t base = a & ~1023u, chunk = ((a & 127) >> 4) + k / 4;
  float v;
  memcpy(&v, smem + base + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk ^ (r & 7)) << 4) + (k % 4) * 4, 4);
  return v;
}
inline float half_at(uint32_t desc, int r, int k, bool bf16) {
  const uint32_t a = (desc & 0x3FFF) << 4;
  const uint32_t base = a & ~1023u, chunk = ((a & 127) >> 4) + k / 8;
  uint16_t v;
  memcpy(&v, smem + base + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk ^ (r & 7)) << 4) + (k % 8) * 2, 2);
  if (bf16) {
    const uint32_t u = (uint32_t)v << 16;
    float f;
    memcpy(&f, &u, 4);
    return f;
  }
  __half_raw h;
  h.x = v;
  return __half2float(__half(h));
}
inline void mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool acc, bool tf32) {
  const int M = (int)((idesc >> 24) & 31) * 16, N = (int)((idesc >> 17) & 63) * 8;
  const bool bf16 = ((idesc >> 7) & 7) == 1;
  check(((idesc >> 7) & 7) == ((idesc >> 10) & 7), "A and B of different types");
  check(M == 128 && N % 16 == 0 && N >= 16 && N <= 256, "an MMA shape that does not exist");
  check(tmem_cols == 512 && (int)(d & 0xFFFF) + N <= 512, "an MMA outside the tensor memory");
  const int n = n_mmas++;
  mmas_pending++;
  if (n == hold_mma) tensor_not_before = clock_ns + hold_ns;
  tensor.push_back([=] {
    const int K = tf32 ? 8 : 16;
    static float a[128][16], b[256][16];
    for (int k = 0; k < K; k++) {
      for (int i = 0; i < M; i++) a[i][k] = tf32 ? tf32_at((uint32_t)ad, i, k) : half_at((uint32_t)ad, i, k, bf16);
      for (int j = 0; j < N; j++) b[j][k] = tf32 ? tf32_at((uint32_t)bd, j, k) : half_at((uint32_t)bd, j, k, bf16);
    }
    check(tmem_cols == 512, "an MMA after its tensor memory was freed");
    for (int i = 0; i < M; i++)
      for (int j = 0; j < N; j++) {
        float& o = tmem[i][(d & 0xFFFF) + j];
        float s = acc ? o : 0.f;
        for (int k = 0; k < K; k++) s += a[i][k] * b[j][k];
        o = s;
      }
    mmas_pending--;
  });
}
inline int elected() { return (int)meet("elect.sync", 0)[0] * 0; }  // lane 0 of the converged warp

}  // namespace emu

// ---- what CUDA C++ gives device code
#undef __shared__
#define __shared__ static
#define threadIdx (::emu::cur->tid)
#define blockIdx (::emu::bid)
#define gridDim (::emu::gdim)
#define blockDim (::emu::Idx{::emu::nthreads, 1, 1})
#define __launch_bounds__(...)
template <class T>
T __ldg(const T* p) { return *p; }
inline void __syncwarp(unsigned = 0xffffffffu) { ::emu::meet("__syncwarp", 0); }
inline int __all_sync(unsigned, int p) {
  const uint64_t* v = ::emu::meet("__all_sync", (uint64_t)(p != 0));
  int r = 1;
  for (int i = 0; i < 32; i++) r &= (int)v[i];
  return r;
}
template <class T>
T __shfl_sync(unsigned, T v, int lane) {
  uint64_t b = 0;
  memcpy(&b, &v, sizeof(T));
  const uint64_t r = ::emu::meet("__shfl_sync", b)[lane & 31];
  memcpy(&v, &r, sizeof(T));
  return v;
}
inline void __syncthreads() {
  const uint64_t g = ::emu::sync_gen;
  if (++::emu::sync_arrived == (int)::emu::nthreads) {
    ::emu::sync_arrived = 0;
    ::emu::sync_gen++;
  } else {
    ::emu::block([g] { return ::emu::sync_gen != g; });
  }
}
template <class T>
T __shfl_xor_sync(unsigned, T v, int mask) {
  uint64_t b = 0;
  memcpy(&b, &v, sizeof(T));
  const uint64_t r = ::emu::meet("__shfl_xor_sync", b)[(::emu::tid() & 31) ^ mask];
  memcpy(&v, &r, sizeof(T));
  return v;
}
inline unsigned __reduce_max_sync(unsigned, unsigned x) {
  const uint64_t* v = ::emu::meet("__reduce_max_sync", x);
  uint64_t r = 0;
  for (int i = 0; i < 32; i++) r = v[i] > r ? v[i] : r;
  return (unsigned)r;
}
inline unsigned long long atomicMax(unsigned long long* p, unsigned long long v) {
  const unsigned long long o = *p;
  *p = v > o ? v : o;
  return o;
}
inline int atomicExch(int* p, int v) {
  const int o = *p;
  *p = v;
  return o;
}
using std::max;
using std::min;
inline int __float2int_rn(float f) { return (int)nearbyintf(f); }
inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31)); }
inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {
  const uint64_t v = ((uint64_t)y << 32) | x;
  uint32_t r = 0;
  for (int i = 0; i < 4; i++) r |= (uint32_t)((v >> (8 * ((s >> (4 * i)) & 7))) & 255) << (8 * i);
  return r;
}
inline double __hiloint2double(int hi, int lo) {
  const uint64_t b = ((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo;
  double d;
  memcpy(&d, &b, 8);
  return d;
}
inline uint64_t __double_as_longlong(double d) {
  uint64_t b;
  memcpy(&b, &d, 8);
  return b;
}
inline int __double2hiint(double d) { return (int)(__double_as_longlong(d) >> 32); }
inline int __double2loint(double d) { return (int)__double_as_longlong(d); }
inline double __longlong_as_double(long long b) { return __hiloint2double((int)(b >> 32), (int)b); }
inline float __uint_as_float(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}
inline uint32_t __float_as_uint(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}
inline double __ll2double_rn(long long v) { return (double)v; }

// ---- the functions made of inline PTX
namespace tn {
namespace ptx {
inline uint32_t smem_u32(const void* p) { return (uint32_t)((const uint8_t*)p - ::emu::smem); }
inline void mbar_init(uint64_t* b, uint32_t count) { ::emu::bar(b) = ::emu::Bar{(uint8_t)count, (uint8_t)count, 0, 0}; }
inline void fence_mbar_init() {}
inline void mbar_arrive(uint64_t* b) { ::emu::arrive(::emu::bar(b)); }
inline void mbar_arrive_expect_tx(uint64_t* b, uint32_t bytes) {
  ::emu::bar(b).tx += (int32_t)bytes;
  ::emu::arrive(::emu::bar(b));
}
inline bool mbar_try_wait(uint64_t* b, uint32_t parity) {
  if (::emu::complete(b, parity)) return true;
  ::emu::yield();
  return ::emu::complete(b, parity);
}
inline bool mbar_test(uint64_t* b, uint32_t parity) { return ::emu::complete(b, parity); }
inline uint64_t globaltimer_ns() { return ::emu::clock_ns; }
inline void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  using namespace emu;
  check(((uintptr_t)dst & 15) == 0 && ((uintptr_t)src & 15) == 0 && bytes % 16 == 0 && bytes > 0, "a bulk copy off its 16-byte alignment");
  check((const uint8_t*)src >= gmem0 && (const uint8_t*)src + bytes <= gmem1, "a bulk copy outside its global memory");
  check((uint8_t*)dst >= dyn && (uint8_t*)dst + bytes <= dyn + dyn_bytes, "a bulk copy outside the shared memory");
  copies.push_back(Copy{(uint8_t*)dst, (const uint8_t*)src, bytes, b, n_copies == hold_copy ? clock_ns + hold_ns : 0});
  n_copies++;
}
// cp.async: in order per thread here; an address has to be good even where nothing is read
inline void cp_async(void* dst, const void* src, int bytes, int size) {
  using namespace emu;
  check(((uintptr_t)dst % size) == 0 && ((uintptr_t)src % size) == 0, "a cp.async off its alignment");
  check((const uint8_t*)src >= gmem0 && (const uint8_t*)src + size_t(bytes ? bytes : 8) <= gmem1, "a cp.async with a bad address");
  check((uint8_t*)dst >= dyn && (uint8_t*)dst + size <= dyn + dyn_bytes, "a cp.async outside the shared memory");
  if (!failure.empty()) return;
  memset(dst, 0, size);
  memcpy(dst, src, bytes);
}
inline void cp_async8(void* dst, const void* src, bool valid) { cp_async(dst, src, valid ? 8 : 0, 8); }
inline void cp_async16(void* dst, const void* src, int bytes) { cp_async(dst, src, bytes, 16); }
inline void cp_async_commit() {}
template <int N>
void cp_async_wait() {}
inline void cp_async_wait_all() {}
inline uint32_t cluster_rank() { return 0; }
inline void cluster_sync() {}
inline uint32_t ld_cluster(const uint32_t* p, uint32_t) { return *p; }
inline void tc_fence_before() {}
inline void tc_fence_after() {}
inline void tmem_alloc(uint32_t* dst, uint32_t n) {
  ::emu::meet("tcgen05.alloc", 0);
  if (::emu::tid() % 32 == 0) {
    ::emu::tmem_cols = (int)n;
    *dst = 0;
  }
}
inline void tmem_relinquish() { ::emu::meet("tcgen05.relinquish", 0); }
inline void tmem_dealloc(uint32_t, uint32_t n) {
  ::emu::meet("tcgen05.dealloc", 0);
  if (::emu::tid() % 32 == 0) {
    ::emu::check(::emu::mmas_pending == 0, "tensor memory freed while an MMA writes it");
    ::emu::check((int)n == ::emu::tmem_cols, "another number of columns freed than allocated");
    ::emu::tmem_cols = 0;
  }
}
inline void mma_f16_elect(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if ((int)(::emu::tid() % 32) == ::emu::elected()) ::emu::mma(d, a, b, idesc, acc != 0, false);
}
inline void mma_tf32_elect(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if ((int)(::emu::tid() % 32) == ::emu::elected()) ::emu::mma(d, a, b, idesc, acc != 0, true);
}
inline void mma_commit_elect(uint64_t* b) {
  if ((int)(::emu::tid() % 32) == ::emu::elected())
    ::emu::tensor.push_back([b] { ::emu::arrive(::emu::bar(b)); });
}
inline void store4(double* p, const double* v) {
  ::emu::check(((uintptr_t)p & 31) == 0, "a 32-byte store off its alignment");
  memcpy(p, v, 32);
}
}  // namespace ptx
namespace {
// 32 lanes x 16 columns at a, in the 16 x 256b fragment order
inline void tmem_read(uint32_t a, float* v) {
  ::emu::meet("tcgen05.ld", a);
  const int lane = (int)(::emu::tid() % 32), row0 = (int)(a >> 16), col0 = (int)(a & 0xFFFF);
  ::emu::check(row0 == 32 * (int)((::emu::tid() / 32) & 3) && col0 + 16 <= 512, "tensor memory read outside the warp's lanes");
  for (int i = 0; i < 16; i++)
    v[i] = ::emu::tmem[row0 + 16 * (i >> 3) + 8 * ((i >> 1) & 1) + (lane >> 2)][col0 + 8 * ((i >> 2) & 1) + 2 * (lane & 3) + (i & 1)];
}
inline void tmem_ld32x16x2(uint32_t a, uint32_t b, float (&v)[16], float (&w)[16]) {
  tmem_read(a, v);
  tmem_read(b, w);
}
inline void tmem_ld32x16(uint32_t a, uint32_t (&r)[16]) {
  float v[16];
  tmem_read(a, v);
  memcpy(r, v, sizeof(r));
}
inline void prefetch_l1(const void*) {}
}  // namespace
}  // namespace tn
