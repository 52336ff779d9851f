// Host-side check of the GEMM kernels' tile enumeration (no GPU needed): for random problems, the tiles that
// get_tile / get_pair_tile hand out must cover every (128-row block, column block) of the output exactly once, stay
// inside one row group, and report the right group.  Built and run by tests/test_tile_enumeration.py.
#include <stdio.h>
#include <stdlib.h>
#include <algorithm>
#include <vector>

#include "../../csrc/gemm_sm100.cu"

using namespace mdt;

// (defined in csrc/comm.cu, which this host program does not link)
extern "C" unsigned long long mdt_peer_wait_limit_ns(void) { return 0; }

static unsigned long long rng_state = 88172645463325252ull;
static int rnd(int n) {
  rng_state ^= rng_state << 13; rng_state ^= rng_state >> 7; rng_state ^= rng_state << 17;
  return (int)(rng_state % (unsigned long long)n);
}

template <int BN_OUT>
static int check(const GemmParams& p, bool pair, const std::vector<int>& offs) {
  const int rows = p.mode == 1 ? offs[p.G] : p.M;
  const int mb = (rows + BM - 1) / BM, nb = (p.N + BN_OUT - 1) / BN_OUT;
  const int groups = p.mode == 2 ? p.G : 1;
  std::vector<int> seen((size_t)groups * mb * nb, 0);
  int bad = 0;
  for (int t = 0;; ++t) {
    int g, m0, n0, second = 0, nkb;
    if (pair) {
      PairTile o;
      if (!get_pair_tile<BN_OUT>(p, t, o)) break;
      g = o.g; m0 = o.m0; n0 = o.n0; second = o.second_ok; nkb = o.num_kb;
    } else {
      Tile o;
      if (!get_tile<BN_OUT>(p, t, o)) break;
      g = o.g; m0 = o.m0; n0 = o.n0; nkb = o.num_kb;
    }
    if (t > 4 * (int)seen.size() + 16) { printf("enumeration does not end\n"); return 1; }
    if (m0 % BM != 0 || n0 % BN_OUT != 0 || n0 >= p.N) { ++bad; continue; }
    for (int h = 0; h < (pair ? 2 : 1); ++h) {
      const int mm = m0 + h * BM;
      if (pair && h == 1 && (!second || mm >= rows)) continue;      // idle half: nothing is stored
      if (mm >= rows) { ++bad; continue; }
      if (p.mode == 1) {
        if (!(offs[g] <= mm && mm + BM <= offs[g + 1])) ++bad;        // the block lies inside the reported group
      }
      if (p.mode == 2) {
        const int want_kb = (offs.empty() ? p.K : offs[g + 1] - offs[g]);
        if (nkb != (want_kb + BK - 1) / BK) ++bad;
      }
      seen[((size_t)(p.mode == 2 ? g : 0) * mb + mm / BM) * nb + n0 / BN_OUT] += 1;
    }
  }
  for (size_t i = 0; i < seen.size(); ++i) {
    // row-grouped problems: blocks of empty padding between groups do not exist (groups are multiples of 128 rows)
    if (seen[i] != 1) ++bad;
  }
  return bad;
}

// The work lists of all CTAs together (get_work, 128-row kernel): every k block of every tile exactly once; whole
// tiles in one piece; a shared tile's pieces come from exactly `contributors` CTAs; at most two pieces per CTA.
template <int BN_OUT>
static int check_work(const GemmParams& p, int num_ctas, const std::vector<int>& offs) {
  const int rows = p.mode == 1 ? offs[p.G] : p.M;
  const int mb = (rows + BM - 1) / BM, nb = (p.N + BN_OUT - 1) / BN_OUT;
  const int kbt = (p.K + BK - 1) / BK + (p.K_l + BK - 1) / BK;
  std::vector<int> covered((size_t)mb * nb * kbt, 0), pieces_of_tile((size_t)mb * nb, 0), claimed((size_t)mb * nb, 0);
  int bad = 0;
  for (int cta = 0; cta < num_ctas; ++cta) {
    int pieces = 0;
    for (int it = 0;; ++it) {
      Work w;
      if (!get_work<BN_OUT>(p, cta, num_ctas, it, w)) break;
      if (it > mb * nb + 4) { printf("work list does not end\n"); return 1; }
      const size_t tile = (size_t)(w.t.m0 / BM) * nb + w.t.n0 / BN_OUT;
      if (w.kb0 < 0 || w.kb1 > kbt || w.kb0 >= w.kb1) { ++bad; continue; }
      for (int kb = w.kb0; kb < w.kb1; ++kb) covered[tile * kbt + kb] += 1;
      if (w.split >= 0) {
        ++pieces;
        pieces_of_tile[tile] += 1;
        if (claimed[tile] != 0 && claimed[tile] != w.contributors) ++bad;
        claimed[tile] = w.contributors;
        if (w.split >= num_ctas) ++bad;                 // the workspace has one tile per CTA
      } else if (w.kb0 != 0 || w.kb1 != kbt) {
        ++bad;                                          // a tile that is not shared is computed whole
      }
    }
    if (pieces > 2) ++bad;
  }
  for (size_t i = 0; i < covered.size(); ++i) if (covered[i] != 1) ++bad;
  for (size_t i = 0; i < claimed.size(); ++i) if (claimed[i] != 0 && claimed[i] != pieces_of_tile[i]) ++bad;
  return bad;
}

// The transposed pair kernel (tp_work): every (32-row unit, feature tile, k block) of the rows that exist exactly once; tiles inside
// their group; the padding of a group cleared by exactly one whole column of tiles; shared tiles as above, one per pair at most.
static int check_transposed(const std::vector<int>& start, const std::vector<int>& rows, const std::vector<int>& end, int N, int f_width, int kbt, int pairs, bool split, int cap) {
  TPTable tb;
  tb.cap = cap;
  const int G = (int)rows.size(), f_tiles = (N + f_width - 1) / f_width;
  int tiles = 0;
  tb.widest = tb.units = tb.groups = 0;
  std::vector<int> order(G);
  for (int g = 0; g < G; ++g) order[g] = g;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tp_tile_rows(rows[a], cap) > tp_tile_rows(rows[b], cap); });
  for (int i = 0; i < G; ++i) {
    const int g = order[i], units = (rows[g] + TP_UNIT - 1) / TP_UNIT, nt = (units + cap - 1) / cap;
    tb.group[i] = g; tb.start[i] = start[g]; tb.rows[i] = rows[g]; tb.end[i] = end[g]; tb.tile0[i] = tiles;
    if (nt != tp_tiles_of_rows(rows[g], cap)) return 1;
    tiles += nt * f_tiles;
    tb.units += units;
    if (nt > 0) { ++tb.groups; const int w = (units + nt - 1) / nt * TP_UNIT; if (w > tb.widest) tb.widest = w; if (w != tp_tile_rows(rows[g], cap)) return 1; }
  }
  tb.tile0[G] = tiles;
  tb.row_tiles = tiles / f_tiles;
  const int top = G ? end[G - 1] : 0, units = (top + TP_UNIT - 1) / TP_UNIT + 1;
  std::vector<int> seen((size_t)units * f_tiles * kbt, 0), cleared((size_t)(top + 1) * f_tiles, 0), pieces(pairs + 1, 0), claimed(pairs + 1, 0);
  int bad = 0;
  for (int p = 0; p < pairs; ++p) {
    int shared = 0;
    for (int it = 0;; ++it) {
      TPWork w;
      if (!tp_work(&tb, G, f_tiles, f_width, kbt, split, p, pairs, it, w)) break;
      if (it > tiles + 4) { printf("work list does not end\n"); return 1; }
      const TPTile& t = w.t;
      const int n0 = tp_first(t.n);        // first accumulator; the rest is the second
      if (t.n < TP_UNIT || t.n > 32 * cap || t.n % TP_UNIT || n0 > 256 || n0 % TP_UNIT || t.n - n0 > 256 || (t.n > 256) != (t.n > n0) || t.n > tb.widest || t.f0 % f_width || t.f0 >= N || t.g >= G || t.row0 < start[t.g] ||
          (t.row0 - start[t.g]) % TP_UNIT || t.row0 - start[t.g] >= rows[t.g] || t.end != end[t.g] || w.kb0 < 0 || w.kb1 > kbt || w.kb0 >= w.kb1) { ++bad; continue; }
      for (int u = 0; u < t.n / TP_UNIT; ++u)
        for (int kb = w.kb0; kb < w.kb1; ++kb) seen[((size_t)(t.row0 / TP_UNIT + u) * f_tiles + t.f0 / f_width) * kbt + kb] += 1;
      if (w.kb0 == 0) for (int r = t.zero0; r < t.end; ++r) cleared[(size_t)r * f_tiles + t.f0 / f_width] += 1;
      if (w.split >= 0) {
        ++shared;
        if (w.split >= pairs) { ++bad; continue; }
        pieces[w.split] += 1;
        if (claimed[w.split] != 0 && claimed[w.split] != w.contributors) ++bad;
        claimed[w.split] = w.contributors;
      } else if (w.kb0 != 0 || w.kb1 != kbt) {
        ++bad;
      }
    }
    if (shared > 2) ++bad;
  }
  for (int i = 0; i <= pairs; ++i) if (pieces[i] != claimed[i]) ++bad;
  for (int g = 0; g < G; ++g) {
    const int covered = (rows[g] + TP_UNIT - 1) / TP_UNIT;
    for (int u = 0; u < (end[g] - start[g] + TP_UNIT - 1) / TP_UNIT; ++u)
      for (int f = 0; f < f_tiles; ++f)
        for (int kb = 0; kb < kbt; ++kb)
          if (seen[((size_t)(start[g] / TP_UNIT + u) * f_tiles + f) * kbt + kb] != (u < covered ? 1 : 0)) ++bad;
    for (int r = start[g]; r < end[g]; ++r)
      for (int f = 0; f < f_tiles; ++f)
        if (rows[g] > 0 && cleared[(size_t)r * f_tiles + f] != (r >= start[g] + covered * TP_UNIT ? 1 : 0)) ++bad;
  }
  return bad;
}

// The choice of tiles of up to 512 rows: for deep products that keep every pair busy; not where their number is too small.
static int check_joint() {
  auto pays = [](std::vector<int> rows, int f_tiles, int kbt) {
    TPForm one{0, 0.f, 0.f}, two{0, 0.f, 0.f};
    int units = 0;
    for (int r : rows) { units += (r + TP_UNIT - 1) / TP_UNIT; tp_add_group(one, r, 8); tp_add_group(two, r, 16); }
    return tp_joint_pays(one, two, units, f_tiles, 74, kbt, true);
  };
  int bad = 0;
  bad += !pays({211, 281, 92, 321, 302, 269, 245, 279}, 16, 224);
  bad += !pays({1901, 2461, 870, 3124, 2866, 2298, 2253, 2627}, 16, 448);
  bad += !pays({300, 300, 300, 300, 300, 300, 300, 300, 300}, 16, 64);
  bad += pays({500, 500}, 16, 224);
  bad += pays({256, 200, 31, 0}, 16, 224);
  bad += pays({0, 0}, 16, 224);
  bad += pays({1901, 2461, 870, 3124, 2866, 2298, 2253, 2627}, 16, 16);
  return bad;
}

int main() {
  int failures = check_joint(), cases = 7;
  for (int it = 0; it < 400; ++it) {
    std::vector<int> start, rows, end;
    const int G = it % 5 == 0 ? 1 : 1 + rnd(12);
    int at = 0;
    for (int g = 0; g < G; ++g) {
      const int n = rnd(4) == 0 ? 0 : 1 + rnd(rnd(3) == 0 ? 2500 : 300);
      start.push_back(at); rows.push_back(n);
      at += it % 5 == 0 ? n : (n + BM - 1) / BM * BM;                // (dense: no padding)
      end.push_back(at);
    }
    const int N = 8 * (17 + rnd(500)), kbt = 1 + rnd(40), ps[3] = {74, 66, 5};
    for (int c = 0; c < 3; ++c) {
      const int b1 = check_transposed(start, rows, end, N, 256, kbt, ps[c], it % 3 != 0, it % 2 ? 8 : 16), b2 = check_transposed(start, rows, end, N, 128, kbt, ps[c], it % 3 != 0, it % 2 ? 8 : 16);
      ++cases;
      if (b1 || b2) { ++failures; printf("transposed: G %d N %d kbt %d pairs %d: %d / %d errors\n", G, N, kbt, ps[c], b1, b2); }
    }
  }
  for (int it = 0; it < 300; ++it) {
    GemmParams p;
    memset(&p, 0, sizeof(p));
    p.mode = it % 2;
    p.N = 8 * (1 + rnd(600));
    p.K = 8 * (1 + rnd(2000));
    p.K_l = (rnd(3) == 0) ? 16 : 0;
    p.sk_ws = reinterpret_cast<float*>(0x10);           // any non-null value: only tested against NULL
    std::vector<int> offs;
    if (p.mode == 0) {
      p.M = 1 + rnd(3000); p.G = 1;
    } else {
      p.G = 1 + rnd(8);
      offs.push_back(0);
      for (int g = 0; g < p.G; ++g) offs.push_back(offs.back() + BM * rnd(6));
      p.M = offs[p.G];
      p.offsets = offs.data();
    }
    const int ctas[3] = {148, 132, 7};
    for (int c = 0; c < 3; ++c) {
      const int b1 = check_work<256>(p, ctas[c], offs), b2 = check_work<128>(p, ctas[c], offs);
      ++cases;
      if (b1 || b2) {
        ++failures;
        printf("work lists: mode %d M %d N %d K %d K_l %d G %d ctas %d: %d / %d errors\n", p.mode, p.M, p.N, p.K, p.K_l, p.G, ctas[c], b1, b2);
      }
    }
  }
  for (int it = 0; it < 400; ++it) {
    GemmParams p;
    memset(&p, 0, sizeof(p));
    p.mode = it % 3;
    p.N = 8 * (1 + rnd(200));
    p.K = 8 * (1 + rnd(300));
    p.K_l = (rnd(3) == 0) ? 16 : 0;
    std::vector<int> offs;
    if (p.mode == 0) {
      p.M = 1 + rnd(3000); p.G = 1;
    } else if (p.mode == 1) {
      p.G = 1 + rnd(8);
      offs.push_back(0);
      for (int g = 0; g < p.G; ++g) offs.push_back(offs.back() + BM * rnd(6));   // groups of 0..5 blocks
      p.M = offs[p.G];
      p.offsets = offs.data();
    } else {
      p.G = 1 + rnd(4);
      p.M = 8 * (1 + rnd(150));
      if (rnd(2)) {
        offs.push_back(0);
        for (int g = 0; g < p.G; ++g) offs.push_back(offs.back() + BM * rnd(5));
        p.offsets = offs.data();
      } else {
        p.G = 1;
      }
    }
    for (int pair = 0; pair < 2; ++pair) {
      const int b1 = check<256>(p, pair != 0, offs);
      const int b2 = check<128>(p, pair != 0, offs);
      ++cases;
      if (b1 || b2) {
        ++failures;
        printf("mode %d pair %d M %d N %d K %d G %d: %d / %d bad tiles\n", p.mode, pair, p.M, p.N, p.K, p.G, b1, b2);
      }
    }
  }
  printf("%d cases, %d failures\n", cases, failures);
  return failures ? 1 : 0;
}
