// Grouped sector GEMM planning and dispatch.  A contraction's sector GEMMs
// (one per Qnum present in both operands, tensor-network/lib/UniTensorTools.cpp:191-203)
// become one work list of output tiles, split along K until every SM has
// work, and run in one launch (plus a deterministic split-K reduction).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>

#include "engine.h"

namespace tn {

namespace {
constexpr int kTileElems = 512;

// tile width for a sector of N columns under a policy: rule 0 takes the
// narrowest of 4, 8, 16, 32 that covers N (32 beyond).  A narrower tile than
// that gathers A from more rows per warp load (tn = 4: 8 rows, 8x the L1
// traffic of tn = 32 per FMA); the width that pads N least (N = 33 -> 4)
// measured 1.6x slower on the batched workload's wide sectors.
int tile_width(int64_t N, const Fp64Policy& pol) {
  if (pol.tn_rule == 1) return 32;
  int tn = 4;
  while (tn < 32 && tn < N) tn *= 2;
  return tn;
}

std::vector<GemmTile> plan_fp64_split(const std::vector<tn_sector_gemm>& list, int num_sms, bool allow_split,
                                      int64_t* ws_elems, const Fp64Policy& pol,
                                      const std::vector<std::pair<int, int>>* vw = nullptr) {
  // K is split so that no work item (one tile over a K range) carries much
  // more than total / (SMs x items_per_sm), with at least ~4 items per SM
  // narrow sectors read contiguously (no operand view) take warp-per-row items
  auto rowdot = [&](size_t gi) {
    const auto& g = list[gi];
    const bool plain = !vw || ((*vw)[gi].first < 0 && (*vw)[gi].second < 0);
    return plain && pol.tn_rule == 0 && g.N <= kRowDotMaxN && g.K >= 32 && g.K <= kRowDotMaxK;  // lanes along K
  };
  int64_t tiles = 0;
  double work = 0;
  for (size_t gi = 0; gi < list.size(); gi++) {
    const auto& g = list[gi];
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || rowdot(gi)) continue;
    const int tn = tile_width(g.N, pol), tm = kTileElems / tn;
    int64_t t = ((g.M + tm - 1) / tm) * ((g.N + tn - 1) / tn);
    tiles += t;
    work += (double)t * g.K;
  }
  const int64_t target_items = (int64_t)num_sms * std::max(1, pol.items_per_sm);
  const double kmax = std::max(64.0, work / (double)target_items);  // K per item
  std::vector<GemmTile> out;
  int64_t ws = 0, ngrp = 0;
  for (size_t gi = 0; gi < list.size(); gi++) {
    const auto& g = list[gi];
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) continue;
    if (g.M > INT32_MAX || g.N > INT32_MAX || g.K > INT32_MAX) fail(TN_ERR_UNSUPPORTED, "sector GEMM dimension too large");
    if (rowdot(gi)) {
      for (int64_t m0 = 0; m0 < g.M; m0 += kRowDotRows) {
        GemmTile t;
        t.a_off = g.a_off;
        t.b_off = g.b_off;
        t.c_off = g.c_off;
        t.M = (int32_t)g.M;
        t.N = (int32_t)g.N;
        t.K = (int32_t)g.K;
        t.m0 = (int32_t)m0;
        t.n0 = 0;
        t.k0 = 0;
        t.k1 = (int32_t)g.K;
        t.split = 0;
        t.nsplit = 1;
        t.tn = 1;
        t.grp = -1;
        t.a_vw = t.b_vw = -1;
        t.ws_off = -1;
        out.push_back(t);
      }
      continue;
    }
    const int tn = tile_width(g.N, pol), tm = kTileElems / tn;
    int nsplit = 1;
    if (allow_split) {
      nsplit = (int)std::ceil((double)g.K / kmax);
      if (pol.spread > 0 && tiles < (int64_t)num_sms * pol.spread)  // few tiles: spread the K loop over the chip
        nsplit = std::max<int>(nsplit, (int)std::min<int64_t>(((int64_t)num_sms * pol.spread + tiles - 1) / tiles,
                                                              (g.K + 15) / 16));
      nsplit = std::max(1, std::min(nsplit, 256));
    }
    const int kchunk = (int)((g.K + nsplit - 1) / nsplit);
    nsplit = (int)((g.K + kchunk - 1) / kchunk);
    for (int64_t m0 = 0; m0 < g.M; m0 += tm)
      for (int64_t n0 = 0; n0 < g.N; n0 += tn) {
        int64_t slot = -1;
        if (nsplit > 1) {
          slot = ws;
          ws += (int64_t)nsplit * kTileElems;
        }
        if (nsplit > 1 && ngrp >= INT32_MAX) fail(TN_ERR_UNSUPPORTED, "too many split tiles");
        for (int s = 0; s < nsplit; s++) {
          GemmTile t;
          t.a_off = g.a_off;
          t.b_off = g.b_off;
          t.c_off = g.c_off;
          t.M = (int32_t)g.M;
          t.N = (int32_t)g.N;
          t.K = (int32_t)g.K;
          t.m0 = (int32_t)m0;
          t.n0 = (int32_t)n0;
          t.k0 = s * kchunk;
          t.k1 = (int32_t)std::min<int64_t>(g.K, (int64_t)(s + 1) * kchunk);
          t.split = s;
          t.nsplit = nsplit;
          t.tn = tn;
          t.grp = nsplit > 1 ? (int32_t)ngrp : -1;
          t.a_vw = vw ? (*vw)[gi].first : -1;
          t.b_vw = vw ? (*vw)[gi].second : -1;
          t.ws_off = slot;
          out.push_back(t);
        }
        if (nsplit > 1) ngrp++;
      }
  }
  *ws_elems = ws;
  // When CTAs take several items each (more items than the launch's grid of
  // at most 16 CTAs per SM, walked with a grid stride), order the items by
  // FMA lanes (padding included) descending, each band of num_sms items
  // alternately reversed, so every CTA's k-th item comes from the same cost
  // band and the CTAs finish together (the batched workload's grouped launch:
  // 11.9 -> 8.9 ms).  With one item per CTA the order only moves CTAs between
  // SMs and is kept as planned.  The result does not depend on the order:
  // split partials have fixed slots, summed in split order.
  if ((int64_t)out.size() <= (int64_t)num_sms * 16) return out;
  auto cost = [](const GemmTile& t) {
    return t.tn == 1 ? (int64_t)kRowDotRows * t.N * ((t.K + 31) / 32 * 32) : (int64_t)kTileElems * (t.k1 - t.k0);
  };
  std::stable_sort(out.begin(), out.end(), [&](const GemmTile& a, const GemmTile& b) { return cost(a) > cost(b); });
  const size_t band = (size_t)std::max(1, num_sms);
  for (size_t b0 = band; b0 < out.size(); b0 += 2 * band)
    std::reverse(out.begin() + b0, out.begin() + std::min(out.size(), b0 + band));
  return out;
}
}  // namespace

std::vector<GemmTile> plan_fp64(const std::vector<tn_sector_gemm>& list, int num_sms, int64_t ws_cap_elems,
                                int64_t* ws_elems, const Fp64Policy& pol) {
  std::vector<GemmTile> t = plan_fp64_split(list, num_sms, true, ws_elems, pol);
  if (ws_cap_elems >= 0 && *ws_elems > ws_cap_elems) t = plan_fp64_split(list, num_sms, false, ws_elems, pol);
  return t;
}

// Flat items.  Cost is counted in warp FMAs (slots x K): an SM sub-partition
// runs one at a time, so items are cut to about a 24th of its share (at
// least 64 warp FMAs, below which an item's own latency shows; at most 4096, or
// a 768th of the share where that is more: a list of 6e10 multiply-adds and up
// would only grow, items and partial sums by gigabytes; the kernel sums such an
// item's K range kFlatChain products at a time, so that sums stay short).
// (Sixteenths were up to 7% slower, on 64 uneven contractions 404 -> 376 us, an
// iPEPS quadrant at chi = 48, D = 5 460 -> 448; 48ths up to 6% faster still on some
// lists and 2% slower on others.)
// Sectors of at least 128 outputs are cut into chunks of at most 4 slots (one
// slot while an item is small: K ranges, with their partial sums, are the
// second choice), each with its K ranges as a group; smaller ones deal all
// their (K range, output) pairs to lanes, with the number of ranges raised
// while more than 1 lane in 16 would stay empty; 256 at most, or
// 8192 partial sums (one warp adds them up).  One- and two-column sectors (a norm, an
// expectation value) take rows, lanes along K, and K ranges of a row as soon as
// one costs two items; with a whole row to a warp 1 x 1 over K = 1e6 took one warp
// 31 250 steps.  An item that reads an operand through views walks its K range in
// the views' segments, so its entries share one range.
// *form: the kernel's instance, kFlatLong for rows over a part of K, groups of more
// than kFlatFewRanges and lists that leave warps idle, kFlatHuge for those items.
constexpr double kFlatFloor = 64.0;   // warp FMAs of an item, at least
constexpr int64_t kRowRanges = 1024;  // K ranges of a row: two for every resident warp of half the chip
std::vector<FlatItem> plan_fp64_flat(const std::vector<tn_sector_gemm>& list, int num_sms, int64_t* ws_elems,
                                     int64_t* ngroups, int* form,
                                     const std::vector<std::pair<int, int>>* vw) {
  auto row_cost = [](int64_t n, int64_t k) { return n * ((k + 31) / 32 + 5); };  // warp FMAs, and 5 to sum the lanes
  auto viewed = [&](size_t gi) { return vw && ((*vw)[gi].first >= 0 || (*vw)[gi].second >= 0); };
  double total = 0, rows8 = 0;
  for (size_t gi = 0; gi < list.size(); gi++) {
    const auto& g = list[gi];
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) continue;
    const bool rows = g.K >= 32 && !viewed(gi);
    total += rows && g.N <= 2 ? (double)g.M * (double)row_cost(g.N, g.K) : std::ceil((double)g.M * g.N / 32.0) * (double)g.K;
    if (rows && g.N <= 8) rows8 += (double)g.M;
  }
  const double share = total / (4.0 * num_sms);
  const int64_t target = (int64_t)std::min(std::max(4096.0, share / 768.0), std::max(kFlatFloor, share / 24.0));
  // A list so small that items are at their least leaves warps idle and lasts as
  // long as its longest item: up to 8 columns are rows there (a lane's chain is K /
  // 32 long, not K), and no more rows to an item than leave every resident warp one.
  const bool idle = share / 24.0 < kFlatFloor;
  const int64_t warps = (int64_t)num_sms * kFlatCtasPerSm * kFlatWarps;
  const int64_t row_cols = idle && rows8 <= (double)warps ? 8 : 2;
  int64_t most_rows = idle ? std::max<int64_t>(1, (int64_t)std::ceil(rows8 / (double)warps)) : 64;
  if (most_rows > 2) most_rows = (most_rows + 3) & ~(int64_t)3;  // rows are taken four at a time
  std::vector<FlatItem> out;
  int64_t ws = 0, ngrp = 0;
  const int64_t most_plain = std::max<int64_t>(1, std::min<int64_t>(kFlatSlots, target / 256));  // slots per chunk
  for (size_t gi = 0; gi < list.size(); gi++) {
    const auto& g = list[gi];
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) continue;
    FlatItem t;
    std::memset(&t, 0, sizeof(t));
    t.a_off = g.a_off;
    t.b_off = g.b_off;
    t.c_off = g.c_off;
    t.N = (int32_t)g.N;
    t.K = (int32_t)g.K;
    t.grp = -1;
    t.nsplit = 1;
    t.a_vw = vw ? (*vw)[gi].first : -1;
    t.b_vw = vw ? (*vw)[gi].second : -1;
    if (g.N <= row_cols && g.K >= 32 && !viewed(gi)) {  // lanes along K
      t.rows = 1;
      t.mn = (int32_t)g.M;
      const int64_t row = row_cost(g.N, g.K);
      int64_t per = std::max<int64_t>(1, std::min<int64_t>(most_rows, idle ? 2 * target / row : target / row));
      if (per > 4) per &= ~(int64_t)3;
      // a row of more than two items' cost: K ranges, a multiple of the 32 lanes each
      const int64_t ns = row > 2 * target ? std::min<int64_t>((row + target - 1) / target, kRowRanges) : 1;
      t.kc = (int32_t)(ns > 1 ? (((g.K + ns - 1) / ns + 31) / 32) * 32 : g.K);
      t.nsplit = (int32_t)((g.K + t.kc - 1) / t.kc);
      for (int64_t m0 = 0; m0 < g.M; m0 += per) {
        t.v0 = (int32_t)m0;
        t.nv = (int32_t)std::min(per, g.M - m0);
        if (t.nsplit > 1) {
          t.grp = (int32_t)ngrp++;
          t.cnt = t.nsplit;
          t.o0 = (int32_t)(m0 * g.N);
          t.go = t.gs = (int32_t)(t.nv * g.N);
          t.ws_off = ws;
          ws += (int64_t)t.nsplit * t.go;
        }
        for (t.kq = 0; t.kq < t.nsplit; t.kq++) out.push_back(t);
      }
      continue;
    }
    const int64_t mn = g.M * g.N, slots = (mn + 31) / 32;
    t.mn = (int32_t)mn;
    if (mn >= 128 || viewed(gi)) {
      const int64_t most = viewed(gi) ? std::min<int64_t>(most_plain, kFlatViewSlots) : most_plain;
      const int64_t nch = (slots + most - 1) / most;
      const int64_t kc0 = std::max<int64_t>(32, target * nch / slots);
      const int64_t ns = std::max<int64_t>(1, std::min<int64_t>((g.K + kc0 / 2) / kc0, 256));
      t.kc = (int32_t)((g.K + ns - 1) / ns);
      t.nsplit = (int32_t)((g.K + t.kc - 1) / t.kc);
      for (int64_t c = 0; c < nch; c++) {
        const int64_t o0 = 32 * (slots * c / nch), o1 = std::min(mn, 32 * (slots * (c + 1) / nch));
        if (t.nsplit > 1) {
          t.grp = (int32_t)ngrp++;
          t.cnt = t.nsplit;
          t.o0 = (int32_t)o0;
          t.go = (int32_t)(o1 - o0);
          t.gs = t.go;
          t.ws_off = ws;
          ws += (int64_t)t.nsplit * t.go;
        }
        for (int q = 0; q < t.nsplit; q++) {
          t.v0 = (int32_t)(q * mn + o0);
          t.nv = (int32_t)(o1 - o0);
          out.push_back(t);
        }
      }
    } else {
      const int64_t kc0 = std::max<int64_t>(32, target);
      int64_t most = std::max<int64_t>(256, 8192 / mn);
      if (idle)  // a range's chain and the chain of sums come out alike
        most = std::min(most, std::max<int64_t>(8, (int64_t)std::sqrt((double)(g.K / slots))));
      int64_t ns = std::max<int64_t>(1, std::min((g.K + kc0 - 1) / kc0, most));
      auto waste = [&](int64_t n) { return (double)((mn * n + 31) / 32 * 32) / (double)(mn * n); };
      while (waste(ns) > 1.0625 && ns < 32 && g.K / (ns + 1) >= 32) ns++;
      t.kc = (int32_t)((g.K + ns - 1) / ns);
      t.nsplit = (int32_t)((g.K + t.kc - 1) / t.kc);
      const int64_t nv = mn * t.nsplit;
      // entries per item: as many slots as the target allows
      const int64_t per = 32 * std::max<int64_t>(1, std::min<int64_t>(kFlatSlots, target / std::max(1, (int)t.kc)));
      if (t.nsplit > 1) {
        t.grp = (int32_t)ngrp++;
        t.cnt = (int32_t)((nv + per - 1) / per);
        t.go = t.gs = (int32_t)mn;
        t.ws_off = ws;
        ws += nv;
      }
      for (int64_t v0 = 0; v0 < nv; v0 += per) {
        t.v0 = (int32_t)v0;
        t.nv = (int32_t)std::min(per, nv - v0);
        out.push_back(t);
      }
    }
  }
  *ws_elems = ws;
  *ngroups = ngrp;
  *form = (int64_t)out.size() <= warps ? kFlatLong : kFlatPlain;
  for (const auto& t : out)
    if (!t.rows && target > 4096 && t.kc > kFlatChain)
      *form = kFlatHuge;
    else if (*form == kFlatPlain && (t.nsplit > kFlatFewRanges || (t.rows && (t.nsplit > 1 || t.N > 2))))
      *form = kFlatLong;
  // the warps of a CTA take kWarps consecutive items; with more items than the
  // grid holds at once, costly ones first, in bands alternately reversed, as
  // for the tiles above
  if ((int64_t)out.size() <= warps) return out;
  auto cost = [&](const FlatItem& t) {
    return t.rows ? t.nv * row_cost(t.N, std::min(t.kc, t.K)) : (int64_t)((t.nv + 31) / 32) * std::min(t.kc, t.K);
  };
  std::stable_sort(out.begin(), out.end(), [&](const FlatItem& a, const FlatItem& b) { return cost(a) > cost(b); });
  const size_t band = (size_t)warps;
  for (size_t b0 = band; b0 < out.size(); b0 += 2 * band)
    std::reverse(out.begin() + b0, out.begin() + std::min(out.size(), b0 + band));
  return out;
}

// 32-bit entry numbers: a sector of 2^31 / 256 outputs or more takes the tiles
static bool flat_fits(const std::vector<tn_sector_gemm>& list) {
  for (const auto& g : list)
    if (g.M > 0 && g.N > 0 && g.K > 0 &&
        (g.M > INT32_MAX || g.N > INT32_MAX || g.K > INT32_MAX / 2 || (double)g.M * (double)g.N >= (double)(1 << 23)))
      return false;
  return true;
}

struct Fp64Plan {
  DevBufP flat;  // FlatItem list (then no tiles)
  int nflat = 0;
  int form = kFlatPlain;
  std::vector<tn_sector_gemm> list;
  std::vector<std::pair<int, int>> vw;  // operand view ids per sector (empty: contiguous operands)
  const void* table = nullptr;          // the view table the ids index
  Fp64Policy pol;
  DevBufP tiles;
  DevBufP counters;  // one per split group, zero between launches
  int ntiles = 0;
  int64_t ws_elems = 0;
  double flops = 0, bytes = 0;
};

static std::shared_ptr<Fp64Plan> get_fp64_plan(Ctx& ctx, const std::vector<tn_sector_gemm>& list,
                                               const Fp64Policy& pol,
                                               const std::vector<std::pair<int, int>>* vw = nullptr,
                                               const void* table = nullptr) {
  uint64_t key = hash_list(list, 64 + 16 * pol.tn_rule + pol.items_per_sm + 1024 * pol.spread + (pol.flat ? 65536 : 0));
  if (vw) {
    for (const auto& v : *vw) key = (key ^ (uint64_t)(uint32_t)v.first ^ ((uint64_t)(uint32_t)v.second << 32)) * 1099511628211ull;
    key ^= (uint64_t)(uintptr_t)table;
  }
  {
    std::lock_guard<std::mutex> lk(ctx.mu);
    auto it = ctx.gemm_cache.find(key);
    if (it != ctx.gemm_cache.end()) {
      auto P = std::static_pointer_cast<Fp64Plan>(it->second);
      const bool same_vw = vw ? (P->vw == *vw && P->table == table) : P->vw.empty();
      if (same_vw && P->pol == pol && P->list.size() == list.size() &&
          std::memcmp(P->list.data(), list.data(), list.size() * sizeof(tn_sector_gemm)) == 0) {
        ctx.keep_alive(P);
        return P;
      }
    }
  }
  auto P = std::make_shared<Fp64Plan>();
  P->list = list;
  P->pol = pol;
  if (vw) {
    P->vw = *vw;
    P->table = table;
  }
  const bool flat = pol.flat && flat_fits(list);
  int64_t ngrp = 0;
  std::vector<FlatItem> items;
  std::vector<GemmTile> tiles;
  if (flat) {
    items = plan_fp64_flat(list, ctx.num_sms, &P->ws_elems, &ngrp, &P->form, vw);
    P->nflat = (int)items.size();
  } else {
    tiles = plan_fp64_split(list, ctx.num_sms, true, &P->ws_elems, pol, vw);
    for (const auto& t : tiles) ngrp = std::max<int64_t>(ngrp, (int64_t)t.grp + 1);
  }
  P->ntiles = (int)tiles.size();
  for (const auto& g : list) {
    P->flops += 2.0 * g.M * g.N * g.K;
    P->bytes += 8.0 * (g.M * g.K + g.K * g.N + g.M * g.N);
  }
  if (ngrp > 0) {
    P->counters = std::make_shared<DevBuf>((size_t)ngrp * sizeof(int), ctx);
    TN_CUDA(cudaMemsetAsync(P->counters->ptr, 0, (size_t)ngrp * sizeof(int), ctx.stream));
  }
  if (!items.empty()) {
    P->flat = std::make_shared<DevBuf>(items.size() * sizeof(FlatItem), ctx);
    TN_CUDA(cudaMemcpyAsync(P->flat->ptr, items.data(), items.size() * sizeof(FlatItem), cudaMemcpyHostToDevice,
                            ctx.stream));
    TN_CUDA(cudaStreamSynchronize(ctx.stream));  // the host copy dies here
  }
  if (!tiles.empty()) {
    P->tiles = std::make_shared<DevBuf>(tiles.size() * sizeof(GemmTile), ctx);
    TN_CUDA(cudaMemcpyAsync(P->tiles->ptr, tiles.data(), tiles.size() * sizeof(GemmTile), cudaMemcpyHostToDevice,
                            ctx.stream));
    TN_CUDA(cudaStreamSynchronize(ctx.stream));  // the host copy dies here
  }
  std::lock_guard<std::mutex> lk(ctx.mu);
  if (ctx.gemm_cache.size() > kPlanCacheCap) ctx.gemm_cache.clear();
  ctx.gemm_cache[key] = P;
  ctx.keep_alive(P);
  return P;
}

static void launch_fp64_plan(Ctx& ctx, const Fp64Plan& P, const double* A, const double* B, double* C,
                             const ViewHdr* views = nullptr, const int64_t* pool = nullptr) {
  double* ws = nullptr;
  if (P.ws_elems > 0) ws = (double*)ctx.ensure_workspace(P.ws_elems * sizeof(double))->ptr;
  int grid = (int)std::min<int64_t>((int64_t)P.ntiles, (int64_t)ctx.num_sms * 16);
  if (P.nflat) {
    ProfScope ps(ctx, "gemm_fp64", P.bytes, P.flops);
    grid = (int)std::min<int64_t>(((int64_t)P.nflat + kFlatWarps - 1) / kFlatWarps,
                                  (int64_t)ctx.num_sms * kFlatCtasPerSm);
    launch_gemm_fp64_flat((const FlatItem*)P.flat->ptr, P.nflat, A, B, C, ws,
                          P.counters ? (int*)P.counters->ptr : nullptr, views, pool, P.form, grid, ctx.stream);
    ctx.launched();
  } else {
    // split tiles are summed by the last CTA of each group (no second launch)
    ProfScope ps(ctx, "gemm_fp64", P.bytes, P.flops);
    launch_gemm_fp64((const GemmTile*)P.tiles->ptr, P.ntiles, A, B, C, ws,
                     P.counters ? (int*)P.counters->ptr : nullptr, views, pool, grid, ctx.stream);
    ctx.launched();
  }
}

// The key of a contraction for the autotuner: its sector-size histogram
// (number of sectors per (log2 M, log2 N, log2 K) bucket), FNV-hashed.
uint64_t sector_histogram_key(const std::vector<tn_sector_gemm>& list) {
  std::map<uint32_t, int64_t> h;
  auto lg = [](int64_t v) {
    uint32_t r = 0;
    while ((int64_t(1) << (r + 1)) <= v) r++;
    return r;
  };
  for (const auto& g : list)
    if (g.M > 0 && g.N > 0 && g.K > 0) h[(lg(g.M) << 16) | (lg(g.N) << 8) | lg(g.K)]++;
  uint64_t x = 1469598103934665603ull;
  for (const auto& kv : h) {
    x = (x ^ kv.first) * 1099511628211ull;
    x = (x ^ (uint64_t)kv.second) * 1099511628211ull;
  }
  return x;
}

const std::vector<Fp64Policy>& fp64_candidates() {
  static const std::vector<Fp64Policy> c = [] {
    std::vector<Fp64Policy> v;
    v.push_back(Fp64Policy());  // flat
    for (int rule : {0, 1})
      for (int items : {2, 8, 16})
        for (int spread : {0, 1, 2, 4}) {
          Fp64Policy p;
          p.flat = false;
          p.tn_rule = rule;
          p.items_per_sm = items;
          p.spread = spread;
          v.push_back(p);
        }
    return v;
  }();
  return c;
}

// Times every candidate on this call's operands (CUDA events on the
// context's stream, outside any graph capture; three launches after a warm-up)
// and keeps the fastest for the histogram key; the caller then runs the
// winner, whose result is the one left in C.  With vw the operands are read
// through views (table = the view table, views / pool its device arrays).
static Fp64Policy tune_fp64(Ctx& ctx, uint64_t key, const std::vector<tn_sector_gemm>& list, const double* A,
                            const double* B, double* C, const std::vector<std::pair<int, int>>* vw = nullptr,
                            const void* table = nullptr, const ViewHdr* views = nullptr,
                            const int64_t* pool = nullptr) {
  cudaEvent_t e0, e1;
  TN_CUDA(cudaEventCreate(&e0));
  TN_CUDA(cudaEventCreate(&e1));
  auto time_of = [&](const Fp64Policy& pol) -> float {
    auto P = get_fp64_plan(ctx, list, pol, vw, table);
    if (!P->ntiles && !P->nflat) return -1.0f;
    launch_fp64_plan(ctx, *P, A, B, C, views, pool);  // warm the plan and the caches
    TN_CUDA(cudaEventRecord(e0, ctx.stream));
    for (int r = 0; r < 3; r++) launch_fp64_plan(ctx, *P, A, B, C, views, pool);
    TN_CUDA(cudaEventRecord(e1, ctx.stream));
    TN_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    TN_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    return ms;
  };
  // the default policy is kept unless a candidate beats it by 3 %: a
  // candidate that wins by noise would cost more than it saves
  const Fp64Policy dflt;
  Fp64Policy best = dflt;
  const float dflt_ms = time_of(dflt);
  float best_ms = dflt_ms;
  for (const auto& pol : fp64_candidates()) {
    if (pol == dflt) continue;
    const float ms = time_of(pol);
    if (ms < 0) continue;
    if (best_ms < 0 || ms < best_ms) {
      best_ms = ms;
      best = pol;
    }
  }
  if (dflt_ms >= 0 && best_ms > 0.97f * dflt_ms) best = dflt;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  ctx.tuned[key] = best;
  return best;
}

static bool capturing(Ctx& ctx) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  TN_CUDA(cudaStreamIsCapturing(ctx.stream, &st));
  return st != cudaStreamCaptureStatusNone;
}

static void run_fp64(Ctx& ctx, const std::vector<tn_sector_gemm>& list, const double* A, const double* B, double* C) {
  Fp64Policy pol;
  if (ctx.autotune) {
    const uint64_t key = sector_histogram_key(list);
    auto it = ctx.tuned.find(key);
    if (it != ctx.tuned.end()) {
      pol = it->second;
    } else if (!capturing(ctx)) {
      pol = tune_fp64(ctx, key, list, A, B, C);
    }
  }
  auto P = get_fp64_plan(ctx, list, pol);
  if (!P->ntiles && !P->nflat) return;
  launch_fp64_plan(ctx, *P, A, B, C);
}

void run_tc_gemms(Ctx& ctx, int ns, const std::vector<tn_sector_gemm>& list, const double* A, const double* B,
                  double* C);

// The forms of a tensor-core mode (static_route): a list of thin sectors alone
// goes to the FP64 kernel; a short list of short K to the fused kernel, or to the
// FP64 kernel or the tiled form where one of them was faster when first run; every
// other list is tiled, its thin sectors on the FP64 kernel.
void run_tc_fused(Ctx& ctx, int ns, const std::vector<tn_sector_gemm>& list, const double* A, const double* B,
                  double* C, const std::vector<std::pair<int, int>>* vw = nullptr, const ViewHdr* views = nullptr,
                  const int64_t* pool = nullptr, const void* table = nullptr);
int64_t fused_items(const std::vector<tn_sector_gemm>& list);

constexpr int kModeFlags = TN_MODE_TC_ONLY | TN_MODE_TC_FUSED | TN_MODE_TC_TILED;

// A sector too thin for a 128 x 64 x 16 MMA step to pay: in the tiled form
// it stays on the exact FP64 kernel (unless TN_MODE_TC_ONLY).
//
// In split precision so does one that the FP64 kernel finishes sooner, both in
// clocks of one SM as grouped launches of small sectors run: 1.6 FMAs a clock
// there, against 5200 per 64 k of an output tile (4000 more to write it) and 1.9
// per operand element to slice.  30 x 30 outputs take the tensor cores, 8 x 30
// do not: on 1024 contractions of bonds 16..256 that moves 1474 of 3007 sectors,
// 8% of the flop, and with the size limits alone the call took 12% longer.  Of
// these constants the sums over four lists (bonds 8..120 to 64..400) came out
// lowest, 1 to 4% below those with a sixth less or a third less per tile.  The
// fast modes keep the sizes alone (there a sector's precision hangs on it), and
// so does a call that asks for the tiled form.
static bool thin_sector(int mode, const tn_sector_gemm& g) {
  if (g.K < 16 || g.N < 16) return true;
  if ((mode & ~kModeFlags) != TN_MODE_SPLIT || (mode & TN_MODE_TC_TILED)) return false;
  const double m = (double)g.M, n = (double)g.N, k = (double)g.K;
  const double tiles = std::ceil(m / 128) * std::ceil(n / 64);
  return m * n * k / 1.6 < tiles * (std::ceil(k / 64) * 5200 + 4000) + 1.9 * (m + n) * k;
}

// The fused form fits a contraction of a few 128 x 64 output tiles per SM
// whose sectors all have short K (its CTAs walk K serially).
static bool fused_fits(const Ctx& ctx, const std::vector<tn_sector_gemm>& list) {
  for (const auto& g : list)
    if (g.K > 576) return false;
  return fused_items(list) <= 4 * (int64_t)ctx.num_sms;
}

static uint64_t route_key(int mode, const std::vector<tn_sector_gemm>& list) {
  return sector_histogram_key(list) ^ ((uint64_t)(mode & 0xFF) * 0x9E3779B97F4A7C15ull);
}

// the static choice before any measurement (flags force a form)
static GemmRoute static_route(const Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list) {
  const bool tc_only = (mode & TN_MODE_TC_ONLY) != 0;
  const bool want_fused = (mode & TN_MODE_TC_FUSED) != 0, want_tiled = (mode & TN_MODE_TC_TILED) != 0;
  mode &= ~kModeFlags;
  if (mode == TN_MODE_FP64) return GemmRoute::Fp64;
  if (mode != TN_MODE_SPLIT && mode != TN_MODE_FAST_BF16 && mode != TN_MODE_FAST_TF32)
    fail(TN_ERR_ARG, "unknown contraction mode");
  if (want_fused && want_tiled) fail(TN_ERR_ARG, "TN_MODE_TC_FUSED and TN_MODE_TC_TILED exclude each other");
  if (mode == TN_MODE_FAST_TF32 && want_fused)
    fail(TN_ERR_UNSUPPORTED, "the fused tensor-core form has no TF32 variant; use TN_MODE_TC_TILED");
  if (want_tiled) return GemmRoute::Tiled;
  if (want_fused) return GemmRoute::Fused;
  bool all_thin = !tc_only;
  for (const auto& g : list) all_thin = all_thin && thin_sector(mode, g);
  if (all_thin) return GemmRoute::Fp64;
  if (mode == TN_MODE_FAST_TF32) return GemmRoute::Tiled;  // TF32 runs in the tiled form only
  // one fused launch for every sector, thin ones included (they cost a CTA
  // each, side by side with the rest)
  if (fused_fits(ctx, list)) return GemmRoute::Fused;
  return GemmRoute::Tiled;
}

// digit images per 64-k operand tile: 7 slices (split, fused form), one BF16
// slice, or the two 128-byte halves of a TF32 tile
static int mode_ns(int mode) {
  const int m = mode & ~kModeFlags;
  return m == TN_MODE_SPLIT ? 7 : (m == TN_MODE_FAST_TF32 ? 2 : 1);
}

// true when the choice between the fused form and the FP64 kernel is left to
// a measurement (no flag forces a form)
static bool route_tunable(int mode, GemmRoute st) {
  return st == GemmRoute::Fused && !(mode & kModeFlags);
}

GemmRoute sector_route(const Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list) {
  const GemmRoute st = static_route(ctx, mode, list);
  if (!route_tunable(mode, st)) return st;
  auto it = ctx.route_tuned.find(route_key(mode, list));
  if (it == ctx.route_tuned.end()) return st;
  return (GemmRoute)it->second;
}

// Times the candidate forms (each writes the same output) and keeps the
// fastest for this histogram; the chosen form runs last, so the output holds
// its result.  Not measured while a graph is being captured.  The tiled form
// is a candidate only where the operands are not read through views.
template <class Fused, class Fp64, class Tiled>
static GemmRoute tune_route(Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list, Fused&& fused, Fp64&& fp64,
                            Tiled* tiled) {
  const GemmRoute st = static_route(ctx, mode, list);
  if (!route_tunable(mode, st)) return st;
  const uint64_t key = route_key(mode, list);
  auto it = ctx.route_tuned.find(key);
  if (it != ctx.route_tuned.end()) return (GemmRoute)it->second;
  if (capturing(ctx)) return st;
  cudaEvent_t e0, e1;
  TN_CUDA(cudaEventCreate(&e0));
  TN_CUDA(cudaEventCreate(&e1));
  auto time_of = [&](auto&& fn) {
    fn();  // warm-up: plans and workspace in place
    TN_CUDA(cudaEventRecord(e0, ctx.stream));
    for (int r = 0; r < 3; r++) fn();
    TN_CUDA(cudaEventRecord(e1, ctx.stream));
    TN_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    TN_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    return ms;
  };
  GemmRoute best = GemmRoute::Fused;
  float best_ms = time_of(fused);
  const float t_fp64 = time_of(fp64);
  if (t_fp64 < best_ms) {
    best = GemmRoute::Fp64;
    best_ms = t_fp64;
  }
  if (tiled && time_of(*tiled) < best_ms) best = GemmRoute::Tiled;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  ctx.route_tuned[key] = (int)best;
  // the output holds the result of the last form timed: rerun the choice
  if (best == GemmRoute::Fused) fused();
  else if (best == GemmRoute::Fp64 && tiled) fp64();
  return best;
}

bool sectors_take_views(const Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list) {
  const GemmRoute r = sector_route(ctx, mode, list);
  return r == GemmRoute::Fp64 || r == GemmRoute::Fused;
}

// The views of one contraction's two operands as one device table.  It holds
// on to both: the table is found by their addresses, which the view cache would
// otherwise give to other views once it starts over.
struct ViewTable {
  OpViewsP va, vb;
  DevBufP hdrs, pool;
  int na = 0;  // headers of the A operand come first
};

static std::shared_ptr<ViewTable> get_view_table(Ctx& ctx, const OpViewsP& va, const OpViewsP& vb) {
  const std::string key = "VT#" + std::to_string((uintptr_t)va.get()) + "#" + std::to_string((uintptr_t)vb.get());
  const uint64_t hk = std::hash<std::string>()(key);
  {
    std::lock_guard<std::mutex> lk(ctx.mu);
    auto it = ctx.gemm_cache.find(hk);
    if (it != ctx.gemm_cache.end()) {
      auto T = std::static_pointer_cast<ViewTable>(it->second);
      ctx.keep_alive(T);
      return T;
    }
  }
  auto T = std::make_shared<ViewTable>();
  T->va = va;
  T->vb = vb;
  std::vector<ViewHdr> hdrs;
  std::vector<int64_t> pool;
  if (va) {
    hdrs = va->hdrs;
    pool = va->pool;
  }
  T->na = (int)hdrs.size();
  if (vb) {
    const int64_t shift = (int64_t)pool.size();
    for (ViewHdr h : vb->hdrs) {
      h.rs += shift;
      h.cs += shift;
      h.tab += shift;
      hdrs.push_back(h);
    }
    pool.insert(pool.end(), vb->pool.begin(), vb->pool.end());
  }
  T->hdrs = std::make_shared<DevBuf>(hdrs.size() * sizeof(ViewHdr), ctx);
  T->pool = std::make_shared<DevBuf>(pool.size() * sizeof(int64_t), ctx);
  TN_CUDA(cudaMemcpyAsync(T->hdrs->ptr, hdrs.data(), hdrs.size() * sizeof(ViewHdr), cudaMemcpyHostToDevice,
                          ctx.stream));
  TN_CUDA(cudaMemcpyAsync(T->pool->ptr, pool.data(), pool.size() * sizeof(int64_t), cudaMemcpyHostToDevice,
                          ctx.stream));
  TN_CUDA(cudaStreamSynchronize(ctx.stream));  // the host copies die here
  std::lock_guard<std::mutex> lk(ctx.mu);
  ctx.gemm_cache[hk] = T;
  ctx.keep_alive(T);
  return T;
}

void run_sector_gemms_views(Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list, const double* A,
                            const double* B, double* C, const OpViewsP& va, const std::vector<int>& a_blk,
                            const OpViewsP& vb, const std::vector<int>& b_blk) {
  if (list.empty()) return;
  if (!va && !vb) {
    run_sector_gemms(ctx, mode, list, A, B, C);
    return;
  }
  if (sector_route(ctx, mode, list) == GemmRoute::Tiled)
    fail(TN_ERR_ARG, "operand views reach the FP64 and fused forms only");
  auto T = get_view_table(ctx, va, vb);
  std::vector<std::pair<int, int>> vw(list.size(), {-1, -1});
  for (size_t i = 0; i < list.size(); i++) {
    if (va) vw[i].first = va->hdr_of_block.at(a_blk.at(i));
    if (vb) vw[i].second = T->na + vb->hdr_of_block.at(b_blk.at(i));
  }
  const ViewHdr* views = (const ViewHdr*)T->hdrs->ptr;
  const int64_t* pool = (const int64_t*)T->pool->ptr;
  const int ns = mode_ns(mode);
  auto fused = [&] { run_tc_fused(ctx, ns, list, A, B, C, &vw, views, pool, T.get()); };
  auto fp64 = [&] {
    Fp64Policy pol;
    if (ctx.autotune) {  // the FP64 tile policy tuned per histogram, as run_fp64 does
      const uint64_t key = sector_histogram_key(list) ^ 0x5A17ull;  // views: a key of its own
      auto it = ctx.tuned.find(key);
      if (it != ctx.tuned.end())
        pol = it->second;
      else if (!capturing(ctx))
        pol = tune_fp64(ctx, key, list, A, B, C, &vw, T.get(), views, pool);
    }
    auto P = get_fp64_plan(ctx, list, pol, &vw, T.get());
    if (P->ntiles || P->nflat) launch_fp64_plan(ctx, *P, A, B, C, views, pool);
  };
  const bool tuned = ctx.route_tuned.count(route_key(mode, list)) > 0;
  const GemmRoute route = tune_route(ctx, mode, list, fused, fp64, (decltype(fp64)*)nullptr);
  if (!tuned && ctx.route_tuned.count(route_key(mode, list))) return;  // measured just now: C holds the result
  if (route == GemmRoute::Fused)
    fused();
  else
    fp64();
}

void run_sector_gemms(Ctx& ctx, int mode, const std::vector<tn_sector_gemm>& list, const double* A, const double* B,
                      double* C) {
  if (list.empty()) return;
  const bool tc_only = (mode & TN_MODE_TC_ONLY) != 0;
  const int ns = mode_ns(mode);
  const bool tuned = ctx.route_tuned.count(route_key(mode, list)) > 0;
  auto tiled = [&] {
    std::vector<tn_sector_gemm> tc, f64;
    for (const auto& g : list) (!tc_only && thin_sector(mode, g) ? f64 : tc).push_back(g);
    if (!f64.empty()) run_fp64(ctx, f64, A, B, C);
    if (!tc.empty()) run_tc_gemms(ctx, ns == 7 ? kSplitDigits : ns, tc, A, B, C);
  };
  const GemmRoute route = tune_route(
      ctx, mode, list, [&] { run_tc_fused(ctx, ns, list, A, B, C); }, [&] { run_fp64(ctx, list, A, B, C); }, &tiled);
  if (!tuned && ctx.route_tuned.count(route_key(mode, list))) return;  // measured just now: C holds the result
  if (route == GemmRoute::Fp64)
    run_fp64(ctx, list, A, B, C);
  else if (route == GemmRoute::Fused)
    run_tc_fused(ctx, ns, list, A, B, C);
  else
    tiled();  // thin sectors on the FP64 kernel (unless TN_MODE_TC_ONLY)
}

}  // namespace tn
