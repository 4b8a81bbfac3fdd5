// The attention work list of a step, on the host: what engine/attention_plan.py: build_plan states, number for number (the
// comparison is in the tests).  A step makes one or two such lists before it can be launched, in the search over cuts with some
// twenty sorts each, which is 0.4 to 1.5 ms of array calls in Python and 10 to 40 us here.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace ftk {
namespace {

using i64 = long long;

constexpr int kItemInts = 8;

// quotients rounded down and up, for any sign
i64 floor_div(i64 a, i64 b) { const i64 q = a / b; return q * b != a && (a < 0) != (b < 0) ? q - 1 : q; }
i64 ceil_div(i64 a, i64 b) { return -floor_div(-a, b); }
// up, of numbers of keys, tiles and pieces (32-bit divisions: the search does some thousand of them)
i64 up(i64 a, i64 b) { return ((uint32_t)a + (uint32_t)b - 1u) / (uint32_t)b; }

struct Tile { i64 seg, tok0, ntok, lo, hi; };

i64 wave_splits(const ftk_attention_plan_rules& r, i64 base_ctas, i64 slots, i64 limit, i64 span) {
  i64 best = 1;
  double best_t = 0.;
  for (i64 s = 1; s <= std::max<i64>(1, limit); ++s) {
    const double t = (double)ceil_div(base_ctas * s, slots) * (r.fixed_cost_keys + (double)span / (double)s);
    if (s == 1 || t < best_t * 0.98) { best = s; best_t = t; }
  }
  return best;
}

std::vector<i64> deal_rows(const std::vector<i64>& spans, i64 total, i64 cap) {
  const i64 n = (i64)spans.size();
  total = std::max(total, n);
  std::vector<i64> weight(n), got(n);
  std::vector<double> want(n);
  i64 whole = 0, sum = 0;
  for (i64 i = 0; i < n; ++i) whole += weight[i] = std::max<i64>(1, spans[i]);
  for (i64 i = 0; i < n; ++i) {
    want[i] = (double)(weight[i] * total) / (double)whole;
    sum += got[i] = std::max<i64>(1, std::min(cap, (i64)want[i]));
  }
  for (; sum < total; ++sum) {  // the largest remainder first, then the heavier, then the earlier
    i64 best = -1;
    for (int any = 0; any < 2 && best < 0; ++any)  // (every tile at the cap: any of them)
      for (i64 i = 0; i < n; ++i) {
        if (!any && got[i] >= cap) continue;
        if (best < 0) { best = i; continue; }
        const double x = want[i] - (double)got[i], y = want[best] - (double)got[best];
        if (x > y || (x == y && weight[i] > weight[best])) best = i;
      }
    ++got[best];
  }
  for (; sum > total; --sum) {  // the largest share too much first, then the lighter, then the later
    i64 best = -1;
    for (i64 i = 0; i < n; ++i) {
      if (got[i] <= 1) continue;
      if (best < 0) { best = i; continue; }
      const double x = (double)got[i] - want[i], y = (double)got[best] - want[best];
      if (x > y || (x == y && weight[i] <= weight[best])) best = i;
    }
    --got[best];
  }
  return got;
}

struct Planner {
  const ftk_attention_plan_rules& r;
  std::vector<Tile> tiles;
  std::vector<i64> spans, quanta, mosts, wants;
  i64 quantum = 0, target = 0;
  double fixed_keys = 0., split_keys = 0.;
  std::vector<i64> load, costs;  // (of `played`)

  explicit Planner(const ftk_attention_plan_rules& rules) : r(rules) {}

  // keys a piece, pieces of a tile that is cut into at most `count`
  void pieces(i64 i, i64 count, i64& per, i64& n) const {
    per = up(std::max<i64>(quanta[i], 1), std::max<i64>(1, std::min(count, quanta[i]))) * quantum;
    n = spans[i] > 0 ? up(spans[i], per) : 1;
  }

  // The busiest CTA's load, in keys, when the list is dealt out to and fro, longest pieces first; false: too many pieces.
  bool played(const std::vector<i64>& counts, double& t) {
    i64 cut = 0;
    costs.clear();
    for (size_t i = 0; i < spans.size(); ++i) {
      i64 per, n;
      pieces((i64)i, counts[i], per, n);
      if (n > 1) cut += n;
      const double on_top = fixed_keys + (n > 1 ? split_keys : 0.);
      const i64 whole = (i64)std::ceil(((double)per + on_top) / (double)r.key_tile);
      const i64 last = (i64)std::ceil(((double)(spans[i] - (n - 1) * per) + on_top) / (double)r.key_tile);
      costs.insert(costs.end(), (size_t)(n - 1), whole);
      costs.push_back(last);
    }
    if (cut * r.n_kv_heads > (i64)r.deal_most_pieces * target) return false;
    std::sort(costs.begin(), costs.end(), std::greater<i64>());
    const i64 all = (i64)costs.size() * r.n_kv_heads, g = std::max<i64>(1, std::min(target, all));
    if (all <= g) {  // a piece each
      t = (double)(costs[0] * r.key_tile);
      return true;
    }
    load.assign((size_t)g, 0);
    i64 at = 0, round = 0;
    for (size_t i = 0; i < costs.size(); ++i)
      for (int h = 0; h < r.n_kv_heads; ++h) {
        load[(size_t)((round & 1) ? g - 1 - at : at)] += costs[i];
        if (++at == g) { at = 0; ++round; }
      }
    t = (double)(*std::max_element(load.begin(), load.end()) * r.key_tile);
    return true;
  }

  void make_tiles(const int32_t* segments, int n_segs) {
    const i64 quantum_kept = r.key_tile ? r.key_tile : r.split_quantum;
    for (int s = 0; s < n_segs; ++s) {
      const i64 q = segments[2 * s], pos0 = (i64)segments[2 * s + 1] - q;
      for (i64 tok0 = 0; tok0 < q; tok0 += r.tokens_per_tile) {
        Tile t{s, tok0, std::min<i64>(r.tokens_per_tile, q - tok0), 0, 0};
        t.hi = pos0 + tok0 + t.ntok;
        if (r.window >= 0) {
          t.lo = std::max<i64>(0, pos0 + tok0 - r.window + 1);
          if (r.key_tile) t.lo = t.lo / r.key_tile * r.key_tile;
        }
        if (r.sparse_block > 0) {
          t.lo = 0;
          t.hi = std::min<i64>(r.sparse_topk, floor_div(pos0 + tok0, r.sparse_block) + 1) * r.sparse_block;
        }
        if (r.window >= 0 && r.keep_first) {
          t.hi -= std::max<i64>(0, t.lo / quantum_kept * quantum_kept - ceil_div(r.keep_first, quantum_kept) * quantum_kept);
          t.lo = 0;
        }
        tiles.push_back(t);
      }
    }
  }

  // How many pieces every tile is wanted in.  Returns whether shares were dealt (the slots are then numbered the same whatever they are).
  bool choose() {
    const i64 n = (i64)tiles.size();
    if (r.fixed_splits >= 0) {
      if (r.fixed_splits > 1) {
        wants = deal_rows(spans, n * r.fixed_splits, std::max(r.fixed_splits, r.max_splits));
        return true;
      }
      wants.assign((size_t)n, r.fixed_splits);
    } else if (n * r.n_kv_heads >= target) {
      i64 all = 0;
      for (i64 x : spans) all += x;
      const double piece = std::max((double)(all * r.n_kv_heads) / (double)std::max<i64>(1, target) / 2., (double)r.min_split_keys);
      const double mean = (double)all / (double)std::max<i64>(1, n);
      wants.assign((size_t)n, 1);
      for (i64 i = 0; i < n; ++i)
        if ((double)spans[i] > piece && (double)spans[i] > 2. * mean)
          wants[i] = std::max<i64>(1, std::min(mosts[i], (i64)std::ceil((double)spans[i] / piece)));
    } else {
      wants.assign((size_t)n, 1);
      i64 known_most = -1, known_span = -1, known = 1;
      for (i64 i = 0; i < n; ++i) {
        if (r.key_tile) mosts[i] = std::max<i64>(1, std::min(mosts[i], floor_div((i64)r.deal_most_pieces * target, n * r.n_kv_heads)));
        if (mosts[i] != known_most || spans[i] != known_span) {
          known = wave_splits(r, n * r.n_kv_heads, target, mosts[i], spans[i]);
          known_most = mosts[i];
          known_span = spans[i];
        }
        wants[i] = known;
      }
    }
    return false;
  }

  // The cuts with which the dealing ends soonest.
  void search(bool& have, double& best_t) {
    std::vector<i64> best = wants, counts(wants.size()), seen;
    have = played(wants, best_t);
    const i64 longest = *std::max_element(spans.begin(), spans.end());
    for (i64 k = 1; k <= r.deal_most_cuts; ++k) {
      const i64 limit = ceil_div(longest, k * quantum) * quantum;
      if (limit < r.min_split_keys) break;
      for (size_t i = 0; i < spans.size(); ++i) counts[i] = std::max<i64>(1, std::min(mosts[i], spans[i] > 0 ? up(spans[i], limit) : 0));
      if (counts == seen) continue;
      seen = counts;
      double t;
      if (!played(counts, t)) break;
      if (!have || t < best_t * 0.97) { best = counts; best_t = t; have = true; }
    }
    wants = best;
  }
};

int plan(const int32_t* segments, int n_segs, const ftk_attention_plan_rules& r, int32_t* items, int capacity, int32_t* n_slots_out,
         double* est_out) {
  Planner p(r);
  p.make_tiles(segments, n_segs);
  const i64 n = (i64)p.tiles.size();
  p.target = 2 * (i64)r.sm_count;
  p.quantum = r.key_tile ? r.key_tile : r.split_quantum;
  for (const Tile& t : p.tiles) {
    const i64 span = t.hi - t.lo;
    p.spans.push_back(span);
    p.quanta.push_back(ceil_div(span, p.quantum));
    p.mosts.push_back(std::min<i64>(r.max_splits, std::max<i64>(1, floor_div(span, r.min_split_keys))));
  }
  p.fixed_keys = r.fixed_cost_keys;
  p.split_keys = r.split_cost_keys;
  const bool priced = r.us_per_key_tile > 0. && r.key_tile;
  if (priced) {
    p.fixed_keys = r.fixed_us / r.us_per_key_tile * r.key_tile;
    p.split_keys = r.split_us / r.us_per_key_tile * r.key_tile;
  }
  const bool dealt = n > 0 && p.choose();
  bool have = false;
  double best_t = 0.;
  if (r.key_tile && r.fixed_splits < 0 && n && n * r.n_kv_heads <= (i64)r.deal_search_limit * p.target) p.search(have, best_t);
  // the list, its slots numbered tile by tile
  struct Row { i64 tile, b, e, rows, i, base; };
  std::vector<Row> list;
  i64 n_slots = 0;
  for (i64 t = 0; t < n; ++t) {
    i64 per, real;
    p.pieces(t, p.wants[t], per, real);
    const i64 rows = std::max<i64>(1, r.fixed_splits >= 0 ? p.wants[t] : real);
    const bool slotted = rows > 1 || dealt;
    for (i64 i = 0; i < rows; ++i)
      list.push_back({t, std::min(p.tiles[t].hi, p.tiles[t].lo + i * per), std::min(p.tiles[t].hi, p.tiles[t].lo + (i + 1) * per), rows,
                      i, rows > 1 ? n_slots : 0});
    if (slotted) n_slots += rows;
  }
  if (r.key_tile) std::stable_sort(list.begin(), list.end(), [](const Row& x, const Row& y) { return x.e - x.b < y.e - y.b; });
  if ((i64)list.size() <= capacity) {
    int32_t* to = items;
    for (const Row& x : list) {
      const Tile& t = p.tiles[x.tile];
      const i64 v[kItemInts] = {t.seg, t.tok0, t.ntok, x.b, x.e, x.rows, x.i, x.base};
      for (i64 y : v) *to++ = (int32_t)y;
    }
  }
  *n_slots_out = (int32_t)n_slots;
  *est_out = -1.;
  if (priced && n && r.fixed_splits < 0) {
    if (!have) have = p.played(p.wants, best_t);
    if (have) {
      double est = best_t / r.key_tile * r.us_per_key_tile + r.launch_us;
      if (n_slots) est += 4.0 + (double)(n_slots * r.n_kv_heads * std::min(r.tile_rows, 256) * 130 * 4) / 4e6;
      *est_out = est;
    }
  }
  return list.size() > 0x7fffffff ? -1 : (int)list.size();
}

}  // namespace
}  // namespace ftk

extern "C" int ftk_attention_plan(const int32_t* segments, int n_segs, const ftk_attention_plan_rules* rules, int32_t* items,
                                  int capacity, int32_t* n_slots, double* est_us) {
  if (!rules || n_segs < 0 || (n_segs > 0 && !segments) || !n_slots || !est_us || capacity < 0 || (capacity > 0 && !items)) return -1;
  const ftk_attention_plan_rules& r = *rules;
  if (r.tokens_per_tile < 1 || r.n_kv_heads < 1 || r.sm_count < 1 || r.max_splits < 1 || r.min_split_keys < 1 || r.key_tile < 0 ||
      r.split_quantum < 1 || r.keep_first < 0)
    return -1;
  try {
    return ftk::plan(segments, n_segs, r, items, capacity, n_slots, est_us);
  } catch (...) {  // (no memory)
    return -1;
  }
}
