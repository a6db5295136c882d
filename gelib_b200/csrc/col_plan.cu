// Host side of the column kernels: which calls they take, and the walk (col.h).
#include <algorithm>
#include <cstring>
#include <map>

#include "col.h"

namespace gelib_b200 {

namespace {

// Stride in floats between consecutive cells (b, g0, g1), or -1 when the view is not an arithmetic progression.
long long cell_stride(const PartView& p, const CellGrid& cg) {
  long long st = 0;
  bool any = false;
  const long long dims[3] = {cg.G1, cg.G0, cg.B}, strides[3] = {p.sg1, p.sg0, p.sb};
  long long inner = 1;
  for (int d = 0; d < 3; d++) {
    if (dims[d] == 1) continue;
    if (!any) st = strides[d];
    else if (strides[d] != st * inner) return -1;
    any = true;
    inner *= dims[d];
  }
  return any ? st : 0;
}

// How a walk is cut for the blocks that share a set of columns: into `groups` runs of pairs, or, with a cluster, by gradient
// rows ("owned"): into groups of rows, each of whose walks is cut for the blocks of a cluster.
struct Split {
  int groups, cluster;
};
constexpr Split kSplitsFwd[] = {{1, 0}, {2, 0}, {4, 0}, {8, 0}, {16, 0}, {32, 0}, {64, 0}};
constexpr Split kSplitsBwd[] = {{1, 0}, {999, 1}, {1, 2}, {1, 4}, {1, 8}, {2, 8}, {4, 8}, {8, 8}, {16, 8}, {2, 0}, {4, 0}, {8, 0}, {16, 0}};
// Words of p.tables for a walk: {first word in h_jobs, runs, blocks of a cluster, most rows that a group sums, cost of the
// longest run, cost of all}.
constexpr int kTable = 6;

struct Step {
  int m, nl, lo, hi;  // output row, output l, first and last entry of the band
};
struct Segment {
  int half, ai, bi, la, lb, mlo, kb;  // mlo, kb: first m1 and number of rows of the a block
  int sum0 = 0;                       // owned walks: where the a block's rows lie among those that the group sums
  std::vector<Step> steps;
  std::vector<const Triple*> ls;      // the triples of the pair's l group, ascending l
  int flags = 0;
  double cost = 0;
};

struct Builder {
  const std::vector<PartSig>& rs;
  bool backward, do_x, do_y, owned;
  std::vector<int2> rows;  // the stream, in order of use

  int nlp(int nl, int kb) const { return col_nl_padded(nl, kb, backward && do_x && do_y && !owned); }
  bool do_a(int half) const { return backward && (owned || (half == 0 ? do_x : do_y)); }
  bool do_b(int half) const { return backward && !owned && (half == 0 ? do_y : do_x); }
  bool need_a(int half) const { return !backward || do_b(half); }
  bool need_b(int half) const { return !backward || do_a(half); }

  // C_l[m1, m - m1], from the band table of the triple (m ascending, then m1 ascending)
  float coefficient(const Schedule& sched, const Triple& t, int m, int m1) const {
    int at = t.coff;
    for (int k = -t.l; k < m; k++) at += std::min<int>(t.l1, k + t.l2) - std::max<int>(-t.l1, k - t.l2) + 1;
    return sched.coeffs[at + m1 - std::max<int>(-t.l1, m - t.l2)];
  }

  int2 r_row(const Segment& s, const Step& st, int j) const {
    const Triple& t = *s.ls[s.ls.size() - st.nl + j];
    return make_int2(2 * kMaxParts + t.ri, (st.m + t.l) * rs[t.ri].n + t.offs);
  }
  void emit_rows(const Segment& s) {
    if ((s.flags & kColFirstOfB) && need_b(s.half))
      for (int r = 0; r <= 2 * s.lb; r++) rows.push_back(make_int2((s.half == 0 ? kMaxParts : 0) + s.bi, r));
    if (need_a(s.half))
      for (int i = 0; i < s.kb; i++) rows.push_back(make_int2((s.half == 0 ? 0 : kMaxParts) + s.ai, s.mlo + s.la + i));
    if (backward)
      for (const Step& st : s.steps)
        for (int j = 0; j < st.nl; j++) rows.push_back(r_row(s, st, j));
  }
  // int4 units of a segment in a chunk, and how many of them are address records
  int units(const Segment& s, int* recs) {
    const size_t n0 = rows.size();
    emit_rows(s);
    *recs = (int)(rows.size() - n0);
    rows.resize(n0);
    int u = 2 + ((int)s.steps.size() + 3) / 4;
    for (const Step& st : s.steps) {
      u += s.kb * ((nlp(st.nl, s.kb) + 3) / 4);
      if (!backward) *recs += st.nl;
    }
    return u + *recs;
  }
};

// Block sizes that the bodies are instantiated for (col_bwd.cuh, col_fwd.cu).
std::vector<int> a_blocks(int rows, int most) {
  std::vector<int> v;
  if (rows <= 17) {  // sizes that differ by at most one
    const int n = (rows + most - 1) / most;
    for (int k = 0; k < n; k++) v.push_back((rows + n - 1 - k) / n);
    return v;
  }
  // an a part with l > 8, on owned walks only: elevens, and what they leave in sizes of six rows and more (smaller bodies
  // only hold the output l of a part that is no larger than they are)
  static const std::vector<int> ends[11] = {{}, {6, 6}, {7, 6}, {7, 7}, {8, 7}, {8, 8}, {6}, {7}, {8}, {9}, {7, 7, 7}};
  const std::vector<int>& end = ends[rows % 11];
  v.assign(rows / 11 - (end.size() > 1 ? 1 : 0), 11);
  v.insert(v.end(), end.begin(), end.end());
  return v;
}

// The segments of a pair for one block of a rows: groups of l, pieces of m.
void pair_segments(const Builder& B, const std::vector<const Triple*>& ts, Segment s, std::vector<Segment>* out) {
  const int cap = kColChunkBytes / 16;
  for (size_t g0 = 0; g0 < ts.size(); g0 += kColMaxNl) {
    s.steps.clear();
    s.cost = 0;
    s.ls.assign(ts.begin() + g0, ts.begin() + std::min(ts.size(), g0 + kColMaxNl));
    int room = 0;
    for (int m = -s.ls.back()->l; m <= s.ls.back()->l; m++) {
      Step st{m, 0, std::max(0, m - s.lb - s.mlo), std::min(s.kb - 1, m + s.lb - s.mlo)};
      for (const Triple* t : s.ls) st.nl += t->l >= std::abs(m);
      if (st.hi < st.lo || st.nl == 0) continue;
      const int need = 1 + s.kb * ((B.nlp(st.nl, s.kb) + 3) / 4) + st.nl;
      if (need > room || s.steps.empty() || st.m != s.steps.back().m + 1) {  // a new piece
        if (!s.steps.empty()) out->push_back(s);
        s.steps.clear();
        s.cost = 0;
        room = cap - 4 - s.kb - (2 * s.lb + 1) - 1;
      }
      room -= need;
      s.cost += (st.hi - st.lo + 1) * (1.5 * st.nl + 9) + 60 + 8 * st.nl;
      s.steps.push_back(st);
    }
    if (!s.steps.empty()) out->push_back(s);
  }
}

double cost_of(const std::vector<Segment>& v) {
  double c = 0;
  for (const auto& s : v) c += s.cost;
  return c;
}

// Appends one walk to the plan (whose schedule and coefficients are there) and describes it in p.tables.
void build_walk(DevicePlan& p, const std::vector<PartSig>& xs, const std::vector<PartSig>& ys, const std::vector<PartSig>& rs,
                bool backward, bool do_x, bool do_y, const Split& split) {
  const bool owned = split.cluster > 0;
  Builder B{rs, backward, do_x, do_y, owned};
  std::map<std::pair<int, int>, std::vector<const Triple*>> pairs;
  for (const Triple& t : p.sched.triples) pairs[{t.xi, t.yi}].push_back(&t);
  for (auto& kv : pairs)
    std::sort(kv.second.begin(), kv.second.end(), [](const Triple* u, const Triple* v) { return u->l < v->l; });
  const int cap = kColChunkBytes / 16, max_block = backward ? kColBlockBwd : kColBlockFwd;
  auto segment = [&](int half, int ai, int bi) {
    Segment s;
    s.half = half;
    s.ai = ai;
    s.bi = bi;
    s.la = (half == 0 ? xs : ys)[ai].l;
    s.lb = (half == 0 ? ys : xs)[bi].l;
    return s;
  };
  auto triples = [&](int half, int ai, int bi) -> const std::vector<const Triple*>* {
    const auto it = pairs.find(half == 0 ? std::make_pair(ai, bi) : std::make_pair(bi, ai));
    return it == pairs.end() ? nullptr : &it->second;
  };

  std::vector<std::vector<Segment>> runs;
  std::vector<std::vector<int2>> sums;  // owned: per group, the gradient rows {slot, row} that its blocks sum
  // contiguous runs of about equal cost
  auto cut = [&](const std::vector<Segment>& all, int pieces) {
    const double total = cost_of(all);
    double done = 0;
    size_t next = 0;
    for (int sp = 0; sp < pieces && next < all.size(); sp++) {
      std::vector<Segment> run;
      const double until = total * (sp + 1) / pieces;
      while (next < all.size() && (run.empty() || sp + 1 == pieces || done + 0.5 * all[next].cost <= until)) {
        done += all[next].cost;
        run.push_back(all[next++]);
      }
      runs.push_back(std::move(run));
    }
  };
  if (owned) {
    // A unit: a block of rows of a part whose gradient is wanted, with every pair of that part, it as the a side.
    struct Unit { std::vector<Segment> segs; int slot, row0; double cost; };
    std::vector<Unit> units;
    for (int half = 0; half < 2; half++) {
      if (half == 0 ? !do_x : !do_y) continue;
      const auto& as = half == 0 ? xs : ys;
      const auto& bs = half == 0 ? ys : xs;
      for (int ai = 0; ai < (int)as.size(); ai++) {
        int mlo = -as[ai].l;
        for (int kb : a_blocks(2 * as[ai].l + 1, max_block)) {
          Unit u{{}, half * kMaxParts + ai, mlo + as[ai].l, 0};
          for (int bi = 0; bi < (int)bs.size(); bi++) {
            const auto* ts = triples(half, ai, bi);
            if (!ts) continue;
            Segment s = segment(half, ai, bi);
            s.mlo = mlo;
            s.kb = kb;
            pair_segments(B, *ts, s, &u.segs);
          }
          mlo += kb;
          u.cost = cost_of(u.segs);
          if (!u.segs.empty()) units.push_back(std::move(u));
        }
      }
    }
    // Groups of units, the longest unit to the group that has least so far; a group's walk is cut for the blocks of a cluster.
    std::stable_sort(units.begin(), units.end(), [](const Unit& u, const Unit& v) { return u.cost > v.cost; });
    const int most = std::min<int>(split.groups, (int)units.size());
    std::vector<std::vector<Segment>> groups(most);
    std::vector<double> load(most, 0.);
    sums.resize(most);
    for (Unit& u : units) {
      const int kb = u.segs[0].kb;
      int g = -1;
      for (int k = 0; k < (int)groups.size(); k++)
        if ((int)sums[k].size() + kb <= kColSumRows && (g < 0 || load[k] < load[g])) g = k;
      if (g < 0) {  // no group has room for its rows
        g = (int)groups.size();
        groups.emplace_back();
        load.push_back(0.);
        sums.emplace_back();
      }
      for (Segment& s : u.segs) {
        s.sum0 = (int)sums[g].size();
        groups[g].push_back(std::move(s));
      }
      for (int i = 0; i < kb; i++) sums[g].push_back(make_int2(u.slot, u.row0 + i));
      load[g] += u.cost;
    }
    for (auto& g : groups) {
      std::stable_sort(g.begin(), g.end(), [](const Segment& s, const Segment& t) {  // the rows of a b part are fetched once
        return s.half != t.half ? s.half < t.half : s.bi < t.bi;
      });
      const size_t first = runs.size();
      cut(g, split.cluster);
      runs.resize(first + split.cluster);  // fewer segments than blocks: the others only take part in the sums
    }
  } else {
    // all segments in order: half, b part, a part, block of a rows, group of l, piece of m
    std::vector<Segment> all;
    for (int half = 0; half < 2; half++) {
      const auto& as = half == 0 ? xs : ys;
      const auto& bs = half == 0 ? ys : xs;
      for (int bi = 0; bi < (int)bs.size(); bi++)
        for (int ai = 0; ai < (int)as.size(); ai++) {
          const auto* ts = triples(half, ai, bi);
          Segment s = segment(half, ai, bi);
          if (!ts || (half == 0 ? s.la > s.lb : s.la >= s.lb)) continue;
          s.mlo = -s.la;
          for (int kb : a_blocks(2 * s.la + 1, max_block)) {
            s.kb = kb;
            pair_segments(B, *ts, s, &all);
            s.mlo += kb;
          }
        }
    }
    cut(all, split.groups);
  }

  std::vector<int> split_table, chunk_table;
  int nchunks = 0, sum_rows = 0;
  double longest = 0, total = 0;
  for (size_t ri = 0; ri < runs.size(); ri++) {
    auto& run = runs[ri];
    longest = std::max(longest, cost_of(run));
    total += cost_of(run);
    auto same_b = [](const Segment& s, const Segment& t) { return s.half == t.half && s.bi == t.bi; };
    for (size_t k = 0; k < run.size(); k++) {
      Segment& s = run[k];
      if (k == 0 || !same_b(run[k - 1], s)) s.flags |= kColFirstOfB;
      if (k + 1 == run.size() || !same_b(run[k + 1], s)) s.flags |= kColLastOfB;
      if (s.half) s.flags |= kColHalf1;
      if (k + 1 == run.size()) s.flags |= kColLast;
    }
    struct Chunk { size_t from, to, row_begin; };
    std::vector<Chunk> chunks;
    B.rows.clear();
    for (size_t k = 0; k < run.size();) {
      Chunk c{k, k, B.rows.size()};
      int used = 2;
      while (k < run.size()) {
        int recs = 0;
        const int need = B.units(run[k], &recs);
        if (k > c.from && used + need > cap) break;
        used += need;
        B.emit_rows(run[k++]);
      }
      c.to = k;
      run[k - 1].flags |= kColLastOfChunk;
      // the rows requested during the chunk push the copy of the next one out of the pending groups, or it is waited for
      if ((int)(B.rows.size() - c.row_begin) < kColRing + 12) run[k - 1].flags |= kColDrain;
      chunks.push_back(c);
    }
    auto rec = [&](size_t i) {
      if (B.rows.empty()) return make_int4(2 * kMaxParts, 0, 0, 0);
      const int2 r = B.rows[std::min(i, B.rows.size() - 1)];  // past the end: the last row again, never taken
      return make_int4(r.x, r.y, 0, 0);
    };
    split_table.push_back(nchunks);
    split_table.push_back((int)chunks.size());
    split_table.push_back((int)p.h_items.size());
    for (int j = 0; j < kColRing; j++) p.h_items.push_back(rec(j));
    split_table.push_back((int)p.h_items.size());
    if (owned) {
      const auto& rows = sums[ri / split.cluster];
      sum_rows = std::max(sum_rows, (int)rows.size());
      p.h_items.push_back(make_int4((int)rows.size(), 0, 0, 0));
      for (const int2& r : rows) p.h_items.push_back(make_int4(r.x, r.y, 0, 0));
    }
    for (size_t ci = 0; ci < chunks.size(); ci++) {
      const Chunk& c = chunks[ci];
      const size_t row_end = ci + 1 < chunks.size() ? chunks[ci + 1].row_begin : B.rows.size();
      std::vector<int4> v(2);
      for (size_t i = c.row_begin; i < row_end; i++) v.push_back(rec(i + kColRing));
      const int store_at = (int)v.size();
      if (!backward)
        for (size_t q = c.from; q < c.to; q++)
          for (const Step& st : run[q].steps)
            for (int j = 0; j < st.nl; j++) {
              const int2 r = B.r_row(run[q], st, j);
              v.push_back(make_int4(r.x, r.y, 0, 0));
            }
      const int nrec = (int)v.size() - 2;
      const int seg_at = (int)v.size();
      for (size_t q = c.from; q < c.to; q++) {
        const Segment& s = run[q];
        v.push_back(make_int4(s.kb | (s.flags << 8) | ((int)s.steps.size() << 16), s.steps[0].m - s.mlo, s.mlo + s.la, s.ai));
        v.push_back(make_int4(s.bi, s.lb, s.sum0, 0));
        std::vector<int> w;
        for (const Step& st : s.steps) w.push_back(st.nl | (st.lo << 8) | (st.hi << 16));
        while (w.size() % 4) w.push_back(0);
        for (size_t i = 0; i < w.size(); i += 4) v.push_back(make_int4(w[i], w[i + 1], w[i + 2], w[i + 3]));
      }
      const int coef_at = (int)v.size();
      std::vector<float> cf;
      for (size_t q = c.from; q < c.to; q++) {
        const Segment& s = run[q];
        for (const Step& st : s.steps)
          for (int i = 0; i < s.kb; i++) {
            const int nlp = B.nlp(st.nl, s.kb);
            for (int j = 0; j < (nlp == 2 ? 2 : (nlp + 3) / 4 * 4); j++) {
              float x = 0.f;
              if (i >= st.lo && i <= st.hi && j < st.nl) {
                const Triple& t = *s.ls[s.ls.size() - st.nl + j];
                const int ma = s.mlo + i;
                x = B.coefficient(p.sched, t, st.m, s.half == 0 ? ma : st.m - ma);
              }
              cf.insert(cf.end(), nlp == 2 ? 2 : 1, x);  // two l: each twice, for the packed multiply-adds
            }
          }
      }
      for (size_t i = 0; i < cf.size(); i += 4) {
        int4 q;
        memcpy(&q, &cf[i], 16);
        v.push_back(q);
      }
      v[0] = make_int4(16 * 2, 16 * store_at, 16 * seg_at, 16 * coef_at);
      v[1] = make_int4(nrec, 0, 0, 0);
      chunk_table.push_back((int)p.h_items.size());
      chunk_table.push_back((int)v.size());
      p.h_items.insert(p.h_items.end(), v.begin(), v.end());
      nchunks++;
    }
  }
  p.tables.insert(p.tables.end(), {(int)p.h_jobs.size(), (int)runs.size(), split.cluster, sum_rows, (int)longest, (int)total});
  p.h_jobs.insert(p.h_jobs.end(), split_table.begin(), split_table.end());
  p.h_jobs.insert(p.h_jobs.end(), chunk_table.begin(), chunk_table.end());
}

// The plan of a signature: every walk that a call of it, whatever its number of cells, may take.
void build(DevicePlan& p, const std::vector<PartSig>& xs, const std::vector<PartSig>& ys, const std::vector<PartSig>& rs,
           bool diag, bool backward, bool do_x, bool do_y) {
  build_schedule(xs, ys, rs, diag, true, &p.sched);
  if (backward)
    for (const Split& sp : kSplitsBwd) build_walk(p, xs, ys, rs, true, do_x, do_y, sp);
  else
    for (const Split& sp : kSplitsFwd) build_walk(p, xs, ys, rs, false, false, false, sp);
  p.sched.coeffs.clear();  // they are in the walks
}

// The backward walk of the least estimated time, and the warps of a block for an owned one.  Fitted to 112 calls with every
// owned walk each (maxl 1 .. 8, lopsided types, 2 .. 375 warps of columns; the choice loses 2 % on average, 28 % at worst): a
// run takes 5 us and 2.5 ns per unit of its cost (2.8 with both gradients at once, which owned walks do not do), a little
// more with every other warp on the SM, and a cluster's sums a microsecond and 40 ns a row.  120 of the 148 SMs hold clusters
// of eight and 132 clusters of four; a second wave of clusters is never worth it, while blocks by themselves fill gaps.
// Measured (us, diagonal products, both gradients): maxl 8 x 4 channels, batch 16 in one piece 564, a run per block of rows
// 71, 64 runs in clusters of eight 29; x 16, batch 500 589, 298, 506; maxl 3 x 12, batch 100 35, 16, and 14 with 16 runs.
// Runs of pairs that add to the same rows (the sums' order varies) are faster where the owned walk's second combination of
// the g rows shows -- maxl 8 x 17, batch 192 55 against 171 -- and are open to calls that no kernel summed in one order.
int choose_walk(const std::vector<int>& tables, long long warps, int b_rows, bool both, bool repeatable, int pinned, int* block_warps) {
  int best = 0;
  double best_time = 1e300;
  const int walks = (int)tables.size() / kTable;
  for (int k = 0; k < walks; k++) {
    if (pinned >= 0 && k != std::min(pinned, walks - 1)) continue;
    const int* t = &tables[kTable * k];
    const int runs = t[1], cluster = t[2], slots = cluster == 0 ? 2 * b_rows : b_rows + t[3];
    if (k > 0 && cluster == 0 && repeatable && pinned < 0) continue;
    const int most = std::min(12, (kColMaxSmem - kColFixedSmem) / (256 * (kColRing + slots)));
    const int blocks = cluster <= 2 ? 148 : cluster == 4 ? 132 : 120, sets = blocks / std::min(runs, blocks);
    long long nw = std::max<long long>(2, (warps + sets - 1) / sets);
    double cost = t[4];
    if (nw > most || runs > blocks) {  // more than one wave
      if (cluster > 1 && pinned < 0) continue;
      nw = most;
      cost = std::max(cost, (double)t[5] * ((warps + nw - 1) / nw) / blocks + 0.7 * cost);
    }
    const double time = 5.2 + 0.1 * (nw - 1) + (cluster > 1 ? 1 + 0.04 * t[3] : 0) +
                        (cluster == 0 && both ? 2.8e-3 : 2.5e-3) * cost * (1 + 0.03 * (nw - 1));
    if (time < best_time) {
      best = k;
      best_time = time;
      *block_warps = cluster == 0 ? 0 : (int)nw;
    }
  }
  return best;
}

}  // namespace

bool col_fill_part(const PartView& p, const CellGrid& cg, long long extra_floats, bool rows, ColPart* out) {
  const long long cs = cell_stride(p, cg);
  const long long unit = rows ? p.sm : 2;
  if (cs < 0 || 4 * cs > 0xffffffffLL || unit < 0 || 4 * unit > 0xffffffffLL) return false;
  out->base = p.base + extra_floats;
  out->unit = (unsigned)(4 * unit);
  out->cell_stride = (unsigned)(4 * cs);
  return true;
}

// The narrow kernels' lanes are padded to a power of two of channels (cw) and they want a full chip; one column per lane does
// without what two columns share.  us, column kernel / narrow kernel, maxl x channels, cells:
//   forward, l <= 1: 1 x 12 2400 9.2 / 7.9, 24000 27 / 22; 300 cells 6.6 / 7.1.  l <= 3: 2 x 16 2400 21 / 19, 24000 90 / 63.
//     From l = 4 on padding decides: 4 x 24 12000 331 / 394, 4 x 5 19200 416 / 522, 4 x 21 2400 95 / 119, 12000 495 / 473,
//     6 x 21 909 / 1167 at 4800; without it 4 x 32 330 / 191 at 4800.
//   gradient of y, one column per lane: l <= 1 1 x 11 2400 9.3 / 11.2, 24000 41 / 30; 1 x 21 12000 43 / 29; above, padding
//     decides: 4 x 5 19200 191 / 397, 4 x 21 4800 208 / 346; 3 x 13 2400 41 / 76 but 4800 96 / 81, 4 x 31 2400 195 / 179, 12000 641 / 569.
//   gradient of y, two columns: without padding l <= 1, l >= 6 and 32 channels lose: 6 x 16 24000 2389 / 2113, 3 x 32 12000
//     286 / 265; but 2 x 16 24000 82 / 107, and with padding 6 x 24 4800 798 / 1231, 6 x 28 802 / 1258.
bool narrow_wins(bool backward, int cpl, int n, int max_la, long long cells) {
  int cw = 1;
  while (cw < n) cw *= 2;
  const long long warps = cells * cw / 32;
  const bool padded = 4 * n <= 3 * cw;
  if (!backward) return warps >= 148 * (max_la <= 1 ? 4 : 16) && !(max_la >= 4 && padded);
  if (!narrow1_enabled() || warps < 148 * 16) return false;
  return cpl == 1 ? max_la <= 1 || !padded : n == cw && (max_la <= 1 || max_la >= 6 || n == 32);
}

bool col_setup(const VecCall& c, bool backward, ColArgs* a, ColPlan* plan) {
  if (c.x.empty() || c.y.empty() || c.r.empty() || !c.dense_channels || c.sph) return false;
  if (c.x.size() > (size_t)kMaxParts || c.y.size() > (size_t)kMaxParts || c.r.size() > (size_t)kMaxParts) return false;
  const int n = c.y[0].n, nx = c.diag ? n : 1;
  for (const auto& p : c.x) if (p.n != nx || p.l > 63) return false;
  for (const auto& p : c.y) if (p.n != n || p.l > 63) return false;
  if (n < 1 || (long long)n * c.cg.ncells > 0x7fffffffLL) return false;
  const bool do_x = !c.xg.empty(), do_y = !c.yg.empty();
  if (backward && !c.diag && do_x && n > 1) return false;  // the gradient of the one channel is a sum over columns
  int max_la = 0, max_lb = 0;
  for (const auto& p : c.x)
    for (const auto& q : c.y) {
      max_la = std::max(max_la, std::min(p.l, q.l));
      max_lb = std::max(max_lb, std::max(p.l, q.l));
    }
  if (max_la > kColMaxLa || max_lb > 40) return false;
  plan->plan_others = false;
  plan->max_block = std::min(2 * max_la + 1, backward ? kColBlockBwd : kColBlockFwd);
  a->b_rows = 2 * max_lb + 1;
  for (size_t i = 0; i < c.x.size(); i++)
    if (!col_fill_part(c.x[i], c.cg, 0, true, &a->part[i])) return false;
  for (size_t i = 0; i < c.y.size(); i++)
    if (!col_fill_part(c.y[i], c.cg, 0, true, &a->part[kMaxParts + i])) return false;
  for (size_t i = 0; i < c.r.size(); i++) {
    if (c.r[i].sm != 2LL * c.r[i].n) return false;  // the walk holds offsets of dense rows
    if ((2LL * c.r[i].l + 1) * c.r[i].n > 0x7fffffffLL) return false;
    if (!col_fill_part(c.r[i], c.cg, 2LL * c.offs_extra, false, &a->part[2 * kMaxParts + i])) return false;
    a->part[2 * kMaxParts + i].unit = 8;
  }
  for (size_t i = 0; i < c.xg.size(); i++)
    if (!col_fill_part(c.xg[i], c.cg, 0, true, &a->grad[i])) return false;
  for (size_t i = 0; i < c.yg.size(); i++)
    if (!col_fill_part(c.yg[i], c.cg, 0, true, &a->grad[kMaxParts + i])) return false;
  // two columns per lane: every access is 16 bytes (8 for an operand of one channel, which both columns share)
  const bool x_shared = nx == 1 && n > 1;
  bool two = n % 2 == 0 && c.offs_extra % 2 == 0;
  for (auto* v : {&c.y, &c.r, &c.yg, x_shared ? &c.y : &c.x, x_shared ? &c.y : &c.xg})
    for (const auto& p : *v)
      if ((uintptr_t)p.base % 16 || p.sb % 4 || p.sg0 % 4 || p.sg1 % 4 || p.sm % 4) two = false;
  // two columns share the records, coefficients and control of a step; with few columns warps matter more
  const long long columns = c.cg.ncells * n;
  const int mode = col_mode();
  plan->cpl = two && (mode == kColAuto ? columns >= 64 * 148 * 4 : mode == kColTwo) ? 2 : 1;
  // Diagonal forward, where the mirrored-row kernel does not take it: with l >= 6 and full 64-channel slices diag_fwd_cell_kernel, which shares its operands between the
  // warps of a block, fits more warps on an SM (us, that kernel / this one): maxl 8 x 128 channels, batch 2048 3018 / 3820;
  // maxl 6 x 64 608 / 835, maxl 6 x 128 1208 / 1265; but maxl 5 x 128 711 / 661, maxl 8 x 48, batch 1000 821 / 652.
  if (c.diag && mode == kColAuto) {
    const int slices = (n + 63) / 64;
    if (!backward && max_la >= 6 && 8 * n >= 7 * 64 * slices) return false;
  }
  std::vector<int> key = {20 /*family*/, backward, do_x, do_y, c.diag, (int)c.x.size(), (int)c.y.size(), (int)c.r.size(), n};
  for (const auto& p : c.x) key.push_back(p.l);
  for (const auto& p : c.y) key.push_back(p.l);
  for (const auto& p : c.r) { key.push_back(p.l); key.push_back(p.n); }
  const auto xs = sig_of(c.x), ys = sig_of(c.y), rs = sig_of(c.r);
  const bool diag = c.diag;
  plan->dev = get_plan(key, [&](DevicePlan& p) { build(p, xs, ys, rs, diag, backward, do_x, do_y); });
  if (!c.diag && n > 1 && n <= 32 && mode == kColAuto) {
    // the rule reads the number of cells: another batch of the signature may go the other way
    if (narrow_wins(backward, plan->cpl, n, max_la, c.cg.ncells)) return false;
    plan->plan_others = plan->dev && plan->dev->first_use.exchange(false);
  }
  if (!plan->dev) return true;
  a->ch_stride[0] = x_shared ? 0 : 8 * plan->cpl;
  a->ch_stride[1] = a->ch_stride[2] = 8 * plan->cpl;
  a->n = (unsigned)(n / plan->cpl);
  a->nlanes = (unsigned)(c.cg.ncells * a->n);
  // With fewer warps than the chip holds, the walk is cut into runs that different blocks take: forward into runs of pairs;
  // backward by gradient rows (owned), so that every row is added to by one lane and the sums have one order, or, where they
  // need not, into runs of pairs.  Forward, us in 16 / 32 / 64 runs: maxl 8 x 16 channels, 30 cells 63 / 40 / 36, 128 cells
  // 76 / 71 / 55; maxl 6 x 33, 4 cells 28 / 18 / 19; maxl 3 x 16, 30 cells 7.9 / 7.6 / 7.8.
  const long long warps = (a->nlanes + 31) / 32;
  const std::vector<int>& tables = plan->dev->tables;
  int walk = 0;
  plan->warps = 0;
  if (!backward) {
    const int last = (int)tables.size() / kTable - 1;
    if (mode == kColAuto)
      while (walk < last && warps * kSplitsFwd[walk + 1].groups <= 148 * 12) walk++;
    else if (mode >= kColSplit)
      walk = std::min(last, mode - kColSplit);
  } else if (plan->cpl == 1 && (mode == kColAuto || mode >= kColSplit)) {
    const bool repeatable = n <= (c.diag ? 16 : 32);  // the kernels before these summed such calls in one order
    walk = choose_walk(tables, warps, a->b_rows, do_x && do_y, repeatable, mode == kColAuto ? -1 : mode - kColSplit, &plan->warps);
  }
  plan->owned = backward && tables[kTable * walk + 2] > 0;
  a->accumulate = (c.flags & GELIB_OVERWRITE) ? 0 : 1;
  a->blob = plan->dev->items;
  a->chunks = plan->dev->jobs + tables[kTable * walk];
  a->nsplits = tables[kTable * walk + 1];
  a->cluster = tables[kTable * walk + 2];
  a->sum_rows = tables[kTable * walk + 3];
  return true;
}

}  // namespace gelib_b200
