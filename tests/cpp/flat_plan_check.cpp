// The FP64 grouped GEMM's flat work list on the host: flat_plan_check SMS
// M N K [M N K ...] plans the list and walks it as the kernel does, checking
// that every product is taken once and every index lies in its range; prints
// the items, the partial sums (elements), the warp FMAs of the costliest item,
// the most ranges that one warp adds up and the most products of one sum (0 where
// the kernel breaks them off at kFlatChain).
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "engine/engine.h"

using namespace tn;

static int bad(const char* what) {
  printf("%s\n", what);
  return 1;
}

int main(int argc, char** argv) {
  std::vector<tn_sector_gemm> list;
  int64_t a = 0, b = 0, c = 0;
  for (int i = 2; i + 2 < argc; i += 3) {
    tn_sector_gemm g;
    g.M = atoll(argv[i]), g.N = atoll(argv[i + 1]), g.K = atoll(argv[i + 2]);
    g.a_off = a, g.b_off = b, g.c_off = c;
    a += g.M * g.K, b += g.K * g.N, c += g.M * g.N;
    list.push_back(g);
  }
  int64_t ws = 0, ngrp = 0, most_cost = 0, most_ranges = 0, chain = 0;
  int form = kFlatPlain;
  const std::vector<FlatItem> items = plan_fp64_flat(list, atoi(argv[1]), &ws, &ngrp, &form);
  std::map<int64_t, int64_t> k_of;  // output -> products taken
  std::vector<int> arrived(ngrp, 0), cnt(ngrp, 0);
  const bool small = c < 100000;
  std::vector<int64_t> done(small ? c : 0, 0), slot(small ? ws : 0, 0);
  for (const FlatItem& t : items) {
    if (t.nv <= 0 || t.kc <= 0) return bad("an empty item");
    if (t.rows) {
      if (t.kq < 0 || t.kq >= t.nsplit) return bad("a range outside the row");
      most_cost = std::max<int64_t>(most_cost, (int64_t)t.nv * t.N * ((std::min(t.kc, t.K - t.kq * t.kc) + 31) / 32));
    } else {
      if (t.nv > 128) return bad("more entries than slots");
      most_cost = std::max<int64_t>(most_cost, (int64_t)((t.nv + 31) / 32) * std::min(t.kc, t.K));
    }
    if (!t.rows && form != kFlatHuge) chain = std::max<int64_t>(chain, std::min(t.kc, t.K));
    if ((t.grp >= 0) != (t.nsplit > 1)) return bad("ranges without a group");
    if (t.grp >= 0) {
      if (t.grp >= ngrp) return bad("a group out of range");
      arrived[t.grp]++;
      cnt[t.grp] = t.cnt;
      most_ranges = std::max<int64_t>(most_ranges, t.nsplit);
      if (t.ws_off < 0 || t.ws_off + (int64_t)(t.nsplit - 1) * t.gs + t.go > ws) return bad("partial sums out of range");
    }
    if (!small) continue;
    for (int v = 0; v < t.nv * (t.rows ? t.N : 1); v++) {
      const int64_t q = t.rows ? t.kq : (t.v0 + v) / t.mn;
      const int64_t o = t.rows ? (int64_t)t.v0 * t.N + v : (t.v0 + v) % t.mn;
      const int64_t len = std::min<int64_t>(t.K, (q + 1) * t.kc) - q * t.kc;
      if (len <= 0) return bad("an empty range");
      if (t.c_off + o < 0 || t.c_off + o >= c) return bad("an output out of range");
      done[t.c_off + o] += len;
      if (t.grp >= 0) {
        const int64_t s = t.ws_off + q * t.gs + (o - t.o0);
        if (o < t.o0 || o >= t.o0 + t.go || slot[s]++) return bad("a partial sum written twice or outside its group");
      }
    }
  }
  for (int64_t i = 0; i < ngrp; i++)
    if (arrived[i] != cnt[i]) return bad("a group that never completes");
  if (small)
    for (const auto& g : list)
      for (int64_t o = 0; o < g.M * g.N; o++)
        if (done[g.c_off + o] != g.K) return bad("a product left out or taken twice");
  printf("ok %zu %lld %lld %lld %lld\n", items.size(), (long long)ws, (long long)most_cost, (long long)most_ranges,
         (long long)chain);
  return 0;
}
