// The tiled tensor-core GEMMs on the CPU (cta_emulator.h): usage
//   <exe> split|bf16|tf32 M N K K-tiles-per-range wide seed [hold-copy n | hold-mma n]
// Prints "ok <error over the sum of magnitudes>" after a product (or "timeout" where a wait was
// made to give up and the kernel said so), else what went wrong.
#include "cta_emulator.h"
#include "tc_gemm_processed.h"

using namespace tn;

static int image_row_of(int n) { return (n & ~15) | ((n & 2) << 2) | ((n & 12) >> 1) | (n & 1); }

template <int NS>
static void put(uint8_t* img, int img_bytes, int r, int c, const double (&x)[8], int e) {
  if constexpr (NS == 2) {
    uint4 o[2];
    make_tf32(x, e, o);
    uint8_t* at = img + (c >> 2) * img_bytes;
    memcpy(at + swz_off(r, 2 * (c & 3)), &o[0], 16);
    memcpy(at + swz_off(r, 2 * (c & 3) + 1), &o[1], 16);
  } else {
    uint4 o[NS];
    if constexpr (NS == 6)
      make_digits(x, e, o);
    else
      make_slices<NS>(x, e, o);
    for (int s = 0; s < NS; s++) memcpy(img + s * img_bytes + swz_off(r, c), &o[s], 16);
  }
}

template <int NS>
static int run(int M, int N, int K, int kts, int wide, unsigned seed) {
  std::mt19937 g(seed);
  std::uniform_real_distribution<double> u(-1, 1);
  std::vector<double> A((size_t)M * K), B((size_t)K * N), C((size_t)M * N + 4, NAN);
  for (double& x : A) x = u(g);
  for (double& x : B) x = u(g);
  TcSector S;
  memset(&S, 0, sizeof(S));
  S.M = M, S.N = N, S.K = K;
  S.nmt = (M + 127) / 128, S.nnt = (N + 63) / 64, S.nkt = (K + 63) / 64;
  S.kts = std::min(kts, S.nkt);
  S.nsplit = (S.nkt + S.kts - 1) / S.kts;
  S.a_img = 0;
  S.b_img = (int64_t)S.nmt * S.nkt * NS * 16384;
  S.eb_off = 0;
  const size_t bytes = S.b_img + (size_t)S.nnt * S.nkt * NS * 8192;
  std::vector<uint8_t> raw(bytes + 1024, 0xFF);  // rows and columns that do not exist hold NaNs
  uint8_t* ws = (uint8_t*)(((uintptr_t)raw.data() + 1023) & ~(uintptr_t)1023);
  std::vector<unsigned long long> ea(M), eb(N);
  for (int i = 0; i < M; i++)
    for (int k = 0; k < K; k++) ea[i] = std::max<unsigned long long>(ea[i], __double_as_longlong(fabs(A[(size_t)i * K + k])));
  for (int j = 0; j < N; j++)
    for (int k = 0; k < K; k++) eb[j] = std::max<unsigned long long>(eb[j], __double_as_longlong(fabs(B[(size_t)k * N + j])));
  const int kend = (K + 15) & ~15;
  for (int k = 0; k < kend; k += 8) {
    double x[8];
    for (int i = 0; i < M; i++) {
      for (int q = 0; q < 8; q++) x[q] = k + q < K ? A[(size_t)i * K + k + q] : 0.0;
      put<NS>(ws + ((int64_t)(i / 128) * S.nkt + k / 64) * NS * 16384, 16384, i % 128, k / 8 % 8, x, exp_of(ea[i]));
    }
    for (int j = 0; j < N; j++) {
      for (int q = 0; q < 8; q++) x[q] = k + q < K ? B[(size_t)(k + q) * N + j] : 0.0;
      put<NS>(ws + S.b_img + ((int64_t)(j / 64) * S.nkt + k / 64) * NS * 8192, 8192, image_row_of(j % 64), k / 8 % 8, x, exp_of(eb[j]));
    }
  }
  std::vector<int4> items;
  for (int mt = 0; mt < S.nmt; mt++)
    for (int nt = 0; nt < S.nnt; nt += wide)
      for (int q = 0; q < S.nsplit; q++) items.push_back(make_int4(0, mt, nt, q));
  std::vector<double> praw((size_t)S.nmt * S.nnt * S.nsplit * 8192 + 4, NAN);
  double* part = (double*)(((uintptr_t)praw.data() + 31) & ~(uintptr_t)31);
  double* c = C.data();
  int err = 0;
  emu::gmem0 = ws;
  emu::gmem1 = ws + bytes;
  emu::dyn_bytes = NS == 6 ? 8 * 16384 + 2 * 6 * 8192 + 1024 : 4 * 49152 + 1024;
  emu::rng.seed(seed * 7919 + 1);
  const unsigned grid = std::min<unsigned>(2, (unsigned)items.size());
  for (unsigned b = 0; b < grid; b++) {
    const std::string why = emu::run_cta(576, b, grid, [&] {
      if constexpr (NS == 6)
        tc_gemm_split(&S, items.data(), (int)items.size(), ws, ea.data(), eb.data(), c, part, &err);
      else
        tc_gemm_fast<NS>(&S, items.data(), (int)items.size(), wide, ws, ea.data(), eb.data(), c, part, &err);
    });
    if (!why.empty()) {
      printf("%s\n", why.c_str());
      return 1;
    }
    if (err) {
      printf(err == TN_ERR_TIMEOUT ? "timeout\n" : "error %d\n", err);
      return 0;
    }
  }
  if (S.nsplit > 1)  // the sum over K ranges
    for (int i = 0; i < M; i++)
      for (int j = 0; j < N; j++) {
        double s = 0;
        for (int q = 0; q < S.nsplit; q++)
          s += part[(((int64_t)(i / 128) * S.nnt + j / 64) * S.nsplit + q) * 8192 + (i % 128) * 64 + j % 64];
        c[(size_t)i * N + j] = scale_pow2(s, exp_of(ea[i]) + exp_of(eb[j]) - (NS == 6 ? 0 : 14));
      }
  double num = 0, den = 0;
  for (int i = 0; i < M; i++)
    for (int j = 0; j < N; j++) {
      long double s = 0, a = 0;
      for (int k = 0; k < K; k++) {
        const long double p = (long double)A[(size_t)i * K + k] * B[(size_t)k * N + j];
        s += p;
        a += fabsl(p);
      }
      const double d = c[(size_t)i * N + j] - (double)s;
      num += d * d;
      den += (double)(a * a);
    }
  printf("ok %.3e\n", sqrt(num / den));
  return 0;
}

int main(int argc, char** argv) {
  const std::string mode = argv[1];
  const int M = atoi(argv[2]), N = atoi(argv[3]), K = atoi(argv[4]), kts = atoi(argv[5]), wide = atoi(argv[6]);
  const unsigned seed = (unsigned)atoi(argv[7]);
  if (argc > 9) {
    (std::string(argv[8]) == "hold-copy" ? emu::hold_copy : emu::hold_mma) = atoi(argv[9]);
    emu::hold_ns = 3200000000ull;  // past the waits' limit of 2 s
  }
  if (mode == "split") return run<6>(M, N, K, kts, wide, seed);
  if (mode == "bf16") return run<1>(M, N, K, kts, wide, seed);
  return run<2>(M, N, K, kts, wide, seed);
}
