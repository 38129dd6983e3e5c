// Plane ranges of single-patch stage launches: how many planes along i a CTA
// marches through (host code, no CUDA).
#pragma once

#include <algorithm>
#include <cstddef>
#include <utility>
#include <vector>

namespace dn {

// Time of a CTA of n planes in planes of a CTA alone on its SM: n + prolog,
// times 1 + share * r while r CTAs share the SM, times edge + (1 - edge) *
// (fraction of the tile's rows inside the patch).  tail: share of a CTA's time
// by which the last ones run late.
struct RangeCost {
  int ctas_per_sm;
  double prolog, share, edge, tail;
};
constexpr RangeCost kRangeF64 = {4, 0.75, 0.2, 0.75, 0.1};    // 4 x 32 tiles
constexpr RangeCost kRangeFx32 = {2, 1.0, 0.6, 0.75, 0.1};    // 16 x 32 tiles

// A launch of column tiles tj x tk over a patch in ranges of ic planes.  CTAs
// start in launch order (k tiles, j tiles, ranges) on the SM that has room
// first; those of an SM share it evenly.
struct RangeLaunch {
  long kt, jt, chunks, ctas;
  int ni, nj, tj, ic, sms;
  RangeCost c;
  double full, late, least;

  RangeLaunch(int ni_, int nj_, int nk, int tj_, int tk, int ic_, int sms_, const RangeCost& c_)
    : kt((nk + tk - 1) / tk), jt((nj_ + tj_ - 1) / tj_), chunks((ni_ + ic_ - 1) / ic_), ctas(kt * jt * chunks), ni(ni_),
      nj(nj_), tj(tj_), ic(ic_), sms(sms_), c(c_), full(1.0 + c_.share * c_.ctas_per_sm)
  {
    late = c.tail * (ic + c.prolog) * (ctas > sms ? full : 1.0 + c.share);
    const double rows = (double)(jt - 1) + weight(jt - 1);
    least = (double)kt * rows * ((double)ni + (double)chunks * c.prolog) / ((double)sms * c.ctas_per_sm) * full;
  }
  double weight(long j) const { return c.edge + (1.0 - c.edge) * std::min<long>(tj, nj - j * tj) / tj; }
  // all SMs busy to the end, and no less than one CTA's time
  double lower_bound() const { return std::max(least, (ic + c.prolog) * (1.0 + c.share) * weight(0)) + late; }

  // its time, or `limit` where it is not below that
  double time(double limit) const
  {
    if (lower_bound() >= limit) return limit;
    // many waves: half a CTA's time for the last one
    if (ctas > 5L * sms * c.ctas_per_sm) return std::min(limit, lower_bound() + 0.5 * (ic + c.prolog));
    const auto work = [&](long cta) {
      return (std::min<long>(ic, ni - cta / (kt * jt) * ic) + c.prolog) * weight(cta / kt % jt);
    };
    // an SM's CTAs by the planes v they end at, v the planes each has advanced
    // at time `at`; the SMs in a heap by the time their next CTA ends
    struct Sm {
      double at, v, cta[4];
      int n;
    };
    struct End {
      double t;
      int sm;
      bool operator<(const End& o) const { return t < o.t || (t == o.t && sm < o.sm); }
    };
    std::vector<Sm> sm((size_t)sms, Sm{0, 0, {}, 0});
    std::vector<End> heap;
    const auto add = [&](Sm& s, double w) {
      int k = s.n++;
      for (; k > 0 && s.cta[k - 1] < s.v + w; --k) s.cta[k] = s.cta[k - 1];   // longest first
      s.cta[k] = s.v + w;
    };
    const auto end = [&](int s) {
      return End{sm[s].at + (sm[s].cta[sm[s].n - 1] - sm[s].v) * (1.0 + c.share * sm[s].n), s};
    };
    long next = 0;
    for (int o = 0; o < c.ctas_per_sm; ++o)
      for (int s = 0; s < sms && next < ctas; ++s) add(sm[s], work(next++));
    for (int s = 0; s < sms && sm[s].n; ++s) heap.push_back(end(s));
    std::make_heap(heap.begin(), heap.end(), [](const End& a, const End& b) { return b < a; });
    const auto sift = [&](End e) {   // e in the place of the first
      size_t k = 0, n = heap.size();
      for (size_t q = 1; q < n; q = 2 * k + 1) {
        if (q + 1 < n && heap[q + 1] < heap[q]) ++q;
        if (!(heap[q] < e)) break;
        heap[k] = heap[q];
        k = q;
      }
      heap[k] = e;
    };
    double t = 0;
    while (!heap.empty()) {
      Sm& s = sm[heap[0].sm];
      t = s.at = heap[0].t;
      if (t + late >= limit) return limit;
      s.v = s.cta[--s.n];
      if (next < ctas) add(s, work(next++));
      if (s.n) {
        sift(end(heap[0].sm));
      } else {
        const End e = heap.back();
        heap.pop_back();
        if (!heap.empty()) sift(e);
      }
    }
    return t + late;
  }
};

// The `count` fastest ranges, fastest first, of the shortest ranges of every
// number of CTAs along i (65535 at most: the grid's third extent), or of `every`
// range up to 64 planes; of those the count + 7 with the lowest bounds are
// simulated (1 ms, 2 ms with every range).
//
// A CTA's planes are a serial chain: short ranges give a small patch the CTAs
// to fill the GPU, long ones spend less on prologues, and the last CTAs decide
// between them.  Fitted to stage times of 284 patches of 12^3 to 256^3 cells
// (127 FP64, 157 FP32; periodic and closed) at 10 to 30 ranges each on a B200:
// of the measured ranges the choice is within 0.2 % (FP64) and 0.9 % (FP32) of
// the fastest on average, 6 % and 14 % at most.  Against the rule that launches
// once had, about four waves of at least eight planes (which ran a 32^3 patch
// on 8 CTAs: FP32 34.9 us a stage against 10.4, FP64 70.4 against 17.5), it is
// slower at four, by 2 % each (FP32 closed 45 x 198 x 167 124.8 against 121.9).
// Whole waves of equal CTAs in place of the simulation chose 121 us for FP64 97
// x 61 x 83, whose last row of tiles has one row of four, where eight planes
// take 109, and 99 against 94 for FP32 45 x 198 x 167.
inline std::vector<int> best_ranges(int ni, int nj, int nk, int tj, int tk, int sms, const RangeCost& c, size_t count,
                                    bool every = false)
{
  std::vector<RangeLaunch> launches;
  for (int chunks = 1; chunks <= std::min(ni, 65535);) {
    const int ic = (ni + chunks - 1) / chunks;
    launches.emplace_back(ni, nj, nk, tj, tk, ic, sms, c);
    if (ic == 1) break;
    chunks = (ni + ic - 2) / (ic - 1);   // the fewest with a shorter range
    for (int q = std::min(ic - 1, 64); every && q > (ni + chunks - 1) / chunks; --q)
      launches.emplace_back(ni, nj, nk, tj, tk, q, sms, c);
  }
  std::sort(launches.begin(), launches.end(),
            [](const RangeLaunch& a, const RangeLaunch& b) { return a.lower_bound() < b.lower_bound(); });
  launches.erase(launches.begin() + (long)std::min(launches.size(), 4 * count + 4), launches.end());
  std::vector<std::pair<double, int>> best;
  for (const RangeLaunch& l : launches) {
    const double limit = best.size() < count ? 1e300 : best.back().first;
    const double t = l.time(limit);
    if (t >= limit) continue;
    if (best.size() == count) best.pop_back();
    best.insert(std::upper_bound(best.begin(), best.end(), std::make_pair(t, l.ic)), {t, l.ic});
  }
  std::vector<int> out;
  for (const auto& b : best) out.push_back(b.second);
  return out;
}

} // namespace dn
