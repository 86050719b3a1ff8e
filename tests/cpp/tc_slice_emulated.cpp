// The one-pass operand slicing on the CPU (cta_emulator.h): usage
//   <exe> M N K seed
// one sector; every copy's address is checked against the operands, the images
// against digits taken from the elements directly.  Prints "ok" or what is wrong.
#include "cta_emulator.h"
#include "tc_slice_processed.h"

using namespace tn;

int main(int, char** argv) {
  const int M = atoi(argv[1]), N = atoi(argv[2]), K = atoi(argv[3]);
  std::mt19937 g(atoi(argv[4]));
  std::uniform_real_distribution<double> u(-1, 1);
  // A, then B, in one allocation that starts far above address zero, reached
  // with absolute offsets from a null base
  std::vector<double> mem((size_t)M * K + (size_t)K * N);
  for (double& x : mem) x = u(g);
  const double *A = mem.data(), *B = A + (size_t)M * K;
  constexpr int NS = 6;
  TcSector S;
  memset(&S, 0, sizeof(S));
  S.M = M, S.N = N, S.K = K;
  S.a_off = (int64_t)((uintptr_t)A / 8), S.b_off = (int64_t)((uintptr_t)B / 8);
  S.nmt = (M + 127) / 128, S.nnt = (N + 63) / 64, S.nkt = (K + 63) / 64;
  S.b_img = (int64_t)S.nmt * S.nkt * NS * 16384;
  std::vector<uint8_t> img(S.b_img + (size_t)S.nnt * S.nkt * NS * 8192 + 16), want = img;
  std::vector<unsigned long long> ea(M), eb(N);
  std::vector<int2> items;
  for (int c = 0; c < (N + 15) / 16; c++) items.push_back(make_int2(0, c));
  for (int r = 0; r < (K > kRowWarp ? M : (M + 7) / 8); r++) items.push_back(make_int2(0, -1 - r));
  emu::gmem0 = (const uint8_t*)mem.data();
  emu::gmem1 = emu::gmem0 + mem.size() * 8;
  emu::dyn_bytes = kStageDoubles * 8;
  uint8_t* ws = (uint8_t*)(((uintptr_t)img.data() + 15) & ~(uintptr_t)15);
  for (unsigned b = 0; b < 2; b++) {
    const std::string why = emu::run_cta(256, b, 2, [&] {
      tc_slice_once<NS, false>(&S, items.data(), 0, (int)items.size(), nullptr, nullptr, ea.data(), eb.data(), ws);
    });
    if (!why.empty()) return printf("%s\n", why.c_str()), 1;
  }
  for (int side = 0; side < 2; side++)
    for (int i = 0; i < (side ? N : M); i++) {
      unsigned long long m = 0;
      auto at = [&](int k) { return side ? B[(size_t)k * N + i] : A[(size_t)i * K + k]; };
      for (int k = 0; k < K; k++) m = std::max<unsigned long long>(m, __double_as_longlong(fabs(at(k))));
      if (exp_of(m) != exp_of(side ? eb[i] : ea[i])) return printf("a maximum is wrong\n"), 1;
      for (int k0 = 0; k0 < ((K + 15) & ~15); k0 += 8) {
        double x[8];
        for (int q = 0; q < 8; q++) x[q] = k0 + q < K ? at(k0 + q) : 0.0;
        uint4 o[NS];
        make_digits(x, exp_of(m), o);
        const int rows = side ? 64 : 128, bytes = side ? 8192 : 16384, r = i % rows;
        const uint8_t* t = ws + (side ? S.b_img : 0) + ((int64_t)(i / rows) * S.nkt + k0 / 64) * NS * bytes;
        const int row = side ? (r & ~15) | ((r & 2) << 2) | ((r & 12) >> 1) | (r & 1) : r;
        for (int s = 0; s < NS; s++)
          if (memcmp(t + s * bytes + swz_off(row, k0 / 8 % 8), &o[s], 16)) return printf("an image is wrong\n"), 1;
      }
    }
  printf("ok\n");
}
