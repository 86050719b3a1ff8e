// Planning time and tiles of a permute on the host: perm_plan_check ORDER DIM...
// (dense bonds, half of them IN) prints the planning time in microseconds (the
// least of five) and the sub-block's tile.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "engine/engine.h"

using namespace tn;

int main(int argc, char** argv) {
  const std::string order = argv[1];
  const int n = (int)order.size();
  std::vector<BondSig> src(n), dst;
  std::vector<int> rsp(n);
  for (int i = 0; i < n; i++) {
    src[i].type = i < n / 2 ? 1 : -1;
    src[i].q = {Q{}};
    src[i].deg = {atoi(argv[2 + i])};
    rsp[i] = order[i] - '0';
  }
  for (int j = 0; j < n; j++) dst.push_back(src[rsp[j]].changed(j < n / 2 ? 1 : -1));
  const SectorMapP a = build_sectormap(src), b = build_sectormap(dst);
  for (int esz : {8, 16}) {
    double best = 1e30;
    PermSub p;
    for (int r = 0; r < 5; r++) {
      const auto t0 = std::chrono::steady_clock::now();
      p = build_perm_subs(*a, *b, rsp, esz).at(0);
      best = std::min(best, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count());
    }
    printf("%.1f %d %d %d %d %d %d\n", best, p.mode, p.tx, p.ty, p.tz, p.tw, p.ydim);
  }
}
