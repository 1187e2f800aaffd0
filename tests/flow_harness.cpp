// Host check of the task images of the per-subdomain triangular solve
// (pgx_flow_pack.h): walks the images as the kernel does, with every offset
// and every ordering rule checked, and compares the solution with plain
// substitution.  Built and run by tests/test_flow_pack.py.
#include <cmath>
#include <cstdio>
#include <random>
#include <string>

#include "../pargemslr_b200/csrc/pgx_flow_pack.h"

using namespace pgx;

#define REQ(x)                                                \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("FAIL %s (line %d)\n", #x, __LINE__);       \
      return false;                                           \
    }                                                         \
  } while (0)

struct Wide {  // a complex value
  double x = 0, y = 0;
  Wide() {}
  Wide(double a) : x(a) {}
  Wide& operator+=(const Wide& o) { x += o.x, y += o.y; return *this; }
  Wide operator*(const Wide& o) const { Wide r; r.x = x * o.x - y * o.y; r.y = x * o.y + y * o.x; return r; }
  Wide operator-(const Wide& o) const { Wide r; r.x = x - o.x; r.y = y - o.y; return r; }
  bool operator==(const Wide& o) const { return x == o.x && y == o.y; }
};

struct Task {  // what a task waits for: its chunk, its progress limit and its sources
  int chunk, next_chunk, lim;
  std::vector<int> src;
};

// One subdomain's pass with copies that land in any order among those in
// flight.  A copy lands only when nothing else can move (`newest`: the last
// one issued first, else any), which is as late as it can be.  Every stage
// that a barrier test lets a warp read must hold the chunk that was meant.
template <typename C>
static bool land(const std::vector<Task>& ts, const int* chunk, int nch, std::mt19937& g, bool newest) {
  constexpr int D = C::stages, W = C::W;
  const int nt = (int)ts.size();
  std::vector<int> freed(D, 0), tot(D, 0), phases(D, 0), holds(D, -1), flight;
  std::vector<char> done(nt, 0), in(W, 0);
  std::vector<int> at(W);
  for (int w = 0; w < W; w++) at[w] = w;
  int issued = 0, below = 0;  // chunks issued; every task below `below` is done
  auto full = [&](int ch) { return flow_issued((unsigned)issued, ch) && (phases[ch % D] & 1) != ((ch / D) & 1); };
  for (;;) {
    bool moved = false;
    for (; issued < nch && (issued < D || freed[issued % D] >= tot[issued % D]); issued++) {
      tot[issued % D] += chunk[4 * issued + 2];
      holds[issued % D] = -1;
      flight.push_back(issued);
      moved = true;
    }
    for (int w = 0; w < W; w++) {
      const int t = at[w];
      if (t >= nt) continue;
      const Task& k = ts[t];
      if (!in[w]) {
        if (!full(k.chunk)) continue;
        REQ(holds[k.chunk % D] == k.chunk);
        in[w] = 1;
        moved = true;
      }
      bool ready = below >= k.lim;
      for (int s : k.src) ready = ready && done[s];
      if (!ready) continue;
      done[t] = 1;
      while (below < nt && done[below]) below++;
      freed[k.chunk % D]++;
      in[w] = 0;
      at[w] += W;
      REQ((at[w] < nt ? ts[at[w]].chunk : -1) == k.next_chunk);
      if (k.next_chunk >= 0 && full(k.next_chunk)) REQ(holds[k.next_chunk % D] == k.next_chunk);
      moved = true;
    }
    if (moved) continue;
    if (flight.empty()) break;
    const size_t q = newest ? flight.size() - 1 : g() % flight.size();
    holds[flight[q] % D] = flight[q];
    phases[flight[q] % D]++;
    flight.erase(flight.begin() + (long)q);
  }
  REQ(below == nt && issued == nch);
  return true;
}

// the kernel's walk, task by task in schedule order, then the same with
// copies that land out of order
template <typename T, typename C>
static bool walk(const FlowPack<T>& p, int n, bool upper, const std::vector<int>& dom, const std::vector<T>& rhs,
                 std::vector<T>& out) {
  out.assign(n, T(0));
  std::mt19937 gl(9);
  for (int c = 0; c < p.ncomp; c++) {
    std::vector<Task> tasks;
    const int c0 = p.comp_chunk0[c], nch = p.comp_chunk0[c + 1] - c0;
    REQ((nch == 0) == (dom[c] == dom[c + 1]));
    std::vector<int> wch(C::W), woff(C::W), cnt(nch, 0), task_of_slot(n, -1);
    for (int w = 0; w < C::W; w++) {
      wch[w] = p.first[2 * (c * C::W + w)];
      woff[w] = p.first[2 * (c * C::W + w) + 1];
      REQ(wch[w] < C::stages);  // a first task's stage is in its first use
    }
    std::vector<T> ring(C::ring + 1, T(0));
    std::vector<int> owner(C::ring, -1), read_by(C::ring, -1000);  // task that solved the slot; last reader
    int rows = 0;
    for (int t = 0;; t++) {
      const int w = t % C::W, ch = wch[w], off = woff[w];
      if (ch < 0) break;
      REQ(ch < nch);
      cnt[ch]++;
      const int* m = &p.chunk[4 * (size_t)(c0 + ch)];
      REQ(m[0] >= 0 && m[1] > 0 && ((size_t)m[0] + m[1]) * 16 <= p.blob.size() && m[1] * 16 <= C::stage_bytes);
      const unsigned char* b = p.blob.data() + (size_t)m[0] * 16;
      const int lim = m[1] * 16;
      REQ(off >= 0 && off % 16 == 0 && off + 4 * kFlowHead <= lim);
      const int* h = (const int*)(b + off);
      const int nr = h[3] & 0xff, st = h[3] >> 8, g1 = h[4] & 255, g2 = (h[4] >> 8) & 255, g4 = (h[4] >> 16) & 255;
      REQ(nr >= 1 && nr <= 32 && st >= nr && st <= 32 && st % 2 == 0 && g1 <= g2 && g2 <= g4);
      REQ(h[9] == rows && h[15] == dom[c] + rows && h[15] + nr <= n);
      REQ(h[5] == std::max(0, t - C::W + 1) && h[6] == std::max(0, t - C::W / 2 + 1));
      const int idb = upper ? (4 * st + 15) / 16 * 16 + st * (int)sizeof(T) : 8 * st;
      REQ(h[0] % 16 == 0 && h[0] + idb <= lim && h[1] % 16 == 0 && h[1] + g4 * st * 8 <= lim);
      REQ(h[2] % 16 == 0 && h[2] + g4 * st * 4 * (int)sizeof(T) <= lim && h[13] % 16 == 0);
      REQ(h[13] + h[12] * st * (16 + 4 * (int)sizeof(T)) <= lim);
      // the slots cleared: nobody reads their old value any more, and their
      // rows are solved by tasks that start after this one is done
      for (int l = 0; l < nr; l++) {
        const int s = (rows + C::ahead + l) & (C::ring - 1);
        REQ(owner[s] < 0 || (read_by[s] <= t - C::W && owner[s] <= t - C::W));
        owner[s] = -1;
        read_by[s] = -1000;
      }
      tasks.push_back({ch, h[10], g2 > g1 ? h[6] : h[5], {}});
      auto source = [&](int s) {
        auto& v = tasks.back().src;
        if (std::find(v.begin(), v.end(), s) == v.end()) v.push_back(s);
      };
      std::vector<T> res(nr);
      for (int l = 0; l < nr; l++) {
        const int id = ((const int*)(b + h[0]))[l];
        REQ(id >= dom[c] && id < dom[c + 1]);
        T acc[2][4], last[2] = {T(0), T(0)}, old(0);
        for (auto& s : acc)
          for (T& v : s) v = T(0);
        const unsigned char* fv = b + h[13] + (size_t)h[12] * st * 16;
        auto fold = [&]() {  // one set of sums: a block of quads is complete
          T s0 = acc[0][0], s1 = acc[0][1];
          s0 += acc[0][2];
          s1 += acc[0][3];
          s0 += s1;
          old += s0;
          for (T& v : acc[0]) v = T(0);
        };
        for (int q = 0; q < h[12]; q++) {
          bool next = false;
          for (int u = 0; u < 4; u++) {
            const int raw = ((const int*)(b + h[13]))[(q * st + l) * 4 + u];
            next = next || (raw >= 0 && (raw & kFlowOther));
          }
          if (kFlowSets<T> == 1 && next) fold();
          for (int u = 0; u < 4; u++) {
            const int raw = ((const int*)(b + h[13]))[(q * st + l) * 4 + u], cc = raw & kFlowIndex;
            const T v = ((const T*)fv)[(q * st + l) * 4 + u];
            if (raw >= 0) {
              REQ(cc < n);
              REQ(task_of_slot[cc] >= 0 && task_of_slot[cc] + 3 * C::W <= t);
              source(task_of_slot[cc]);
              (raw & kFlowLast ? last[u / 2] : acc[kFlowSets<T> == 2 && (raw & kFlowOther) ? 1 : 0][u]) += v * out[cc];
            } else {
              REQ(v == T(0));
            }
          }
        }
        for (int q = 0; q < g4; q++) {
          const int before = q < g1 ? h[5] : q < g2 ? h[6] : t;  // sources must be earlier than this task
          if (kFlowSets<T> == 1 && q < g4 - 1 && (g4 - q) % kFlowBlock == 0 &&
              ((const unsigned short*)(b + h[1]))[(q * st + l) * 4] != C::ring)
            fold();
          for (int u = 0; u < 4; u++) {
            const int cc = ((const unsigned short*)(b + h[1]))[(q * st + l) * 4 + u];
            const T v = ((const T*)(b + h[2]))[(q * st + l) * 4 + u];
            REQ(cc <= C::ring);
            if (cc < C::ring) {
              REQ(owner[cc] >= 0 && owner[cc] < before);
              source(owner[cc]);
              read_by[cc] = t;
            } else {
              REQ(v == T(0));
            }
            (q == g4 - 1 ? last[u / 2] : acc[kFlowSets<T> == 2 ? q & 1 : 0][u]) += v * ring[cc];
          }
        }
        T p[4];
        for (int u = 0; u < 4; u++) (p[u] = acc[0][u]) += acc[1][u];
        p[0] += p[2];
        p[1] += p[3];
        p[0] += p[1];
        old += p[0];
        last[0] += last[1];
        old += last[0];
        const T s = (upper ? rhs[h[15] + l] : rhs[id]) - old;
        res[l] = upper ? s * ((const T*)(b + h[0] + (4 * st + 15) / 16 * 16))[l] : s;
      }
      for (int l = 0; l < nr; l++) {
        const int s = (rows + l) & (C::ring - 1), id = ((const int*)(b + h[0]))[l];
        const int to = upper ? id : ((const int*)(b + h[0]))[st + l];
        REQ(owner[s] == -1 && to >= 0 && to < n && task_of_slot[to] < 0);
        ring[s] = res[l];
        owner[s] = t;
        out[to] = res[l];
        task_of_slot[to] = t;
      }
      rows += nr;
      REQ(h[10] < 0 || (h[10] >= ch && h[10] - ch <= C::W));  // the stage looked at is at most W chunks on
      wch[w] = h[10];
      woff[w] = h[11];
    }
    REQ(rows == dom[c + 1] - dom[c]);
    for (int k = 0; k < nch; k++) REQ(cnt[k] == p.chunk[4 * (size_t)(c0 + k) + 2]);
    for (int k = 0; k < 3; k++)
      if (nch > 0) REQ((land<C>(tasks, &p.chunk[4 * (size_t)c0], nch, gl, k == 0)));
  }
  return true;
}

struct Tri {
  std::vector<int> rp{0}, cj;
  std::vector<double> va;
};

template <typename T, int R, typename C = FlowCfg<T, R>>
static int solve(const Tri& L, const Tri& U, const std::vector<double>& dinv, const std::vector<int>& dom, double tol,
                 std::vector<T>* keep) {
  const int n = (int)dinv.size();
  auto lv = [&](int k) { return T(L.va[k]); };
  auto uv = [&](int k) { return T(U.va[k]); };
  auto dv = [&](int i) { return T(dinv[i]); };
  FlowPack<T> pu, pl;
  if (!flow_pack<T, C>(n, U.rp.data(), U.cj.data(), uv, true, dom, &dv, nullptr, pu)) return 2;
  if (!flow_pack<T, C>(n, L.rp.data(), L.cj.data(), lv, false, dom, &dv, &pu.slot_of_row, pl)) return 2;
  std::mt19937 g(5);
  std::uniform_real_distribution<double> d(-1, 1);
  std::vector<T> b(n), y, x;
  for (auto& v : b) v = T((float)d(g));
  if (!walk<T, C>(pl, n, false, dom, b, y) || !walk<T, C>(pu, n, true, dom, y, x)) return 1;
  std::vector<T> r = b;
  for (int i = 0; i < n; i++) {
    T s(0);
    for (int k = L.rp[i]; k < L.rp[i + 1]; k++) s += lv(k) * r[L.cj[k]];
    r[i] = r[i] - s;
  }
  double num = 0, den = 1e-300;
  for (int i = n - 1; i >= 0; i--) {
    T s(0);
    for (int k = U.rp[i]; k < U.rp[i + 1]; k++) s += uv(k) * r[U.cj[k]];
    r[i] = (r[i] - s) * dv(i);
    const T e = x[i] - r[i];


    double a, q;
    if constexpr (sizeof(T) == 16) {
      a = e.x * e.x + e.y * e.y;
      q = r[i].x * r[i].x + r[i].y * r[i].y;
    } else {
      a = (double)e * e;
      q = (double)r[i] * r[i];
    }
    num += a;
    den += q;
  }
  if (!(std::sqrt(num / den) <= tol)) {
    std::printf("FAIL solution off by %g\n", std::sqrt(num / den));
    return 1;
  }
  // every lane count sums a row's entries in the same order
  if (keep) {
    if (keep->empty())
      *keep = x;
    else
      for (int i = 0; i < n; i++)
        if (!((*keep)[i] == x[i])) {
          std::printf("FAIL row %d differs between lane counts\n", i);
          return 1;
        }
  }
  return 0;
}

// a factor pair with `deg` random entries a row, at most `back` rows away, in
// every subdomain; a band of long rows if `longrow`
static void make(const std::vector<int>& dom, int deg, int back, int longrow, unsigned seed, Tri& L, Tri& U,
                 std::vector<double>& dinv) {
  std::mt19937 g(seed);
  std::uniform_real_distribution<double> d(-1, 1);
  for (size_t c = 0; c + 1 < dom.size(); c++)
    for (int i = dom[c]; i < dom[c + 1]; i++) {
      for (int up = 0; up < 2; up++) {
        Tri& M = up ? U : L;
        const int room = up ? dom[c + 1] - 1 - i : i - dom[c];
        int want = std::min(room, (int)(g() % (unsigned)(deg + 1)));
        if (longrow && i % 97 == 96) want = std::min(room, longrow);
        std::vector<int> cols;
        for (int k = 0; k < want; k++) {
          const int span = std::min(room, std::max(back, want));
          cols.push_back(up ? i + 1 + (int)(g() % (unsigned)span) : i - 1 - (int)(g() % (unsigned)span));
        }
        std::sort(cols.begin(), cols.end());
        cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
        for (int j : cols) {
          M.cj.push_back(j);
          M.va.push_back((float)(d(g) / (1 + want)));
        }
        M.rp.push_back((int)M.cj.size());
      }
      dinv.push_back((float)(1.0 + 0.2 * d(g)));
    }
}

// a factor pair on an nx x ny x nz grid: the neighbours within `reach` in every direction that come before (after) a
// row, as a factor with much fill has them
static void grid(int nx, int ny, int nz, int reach, unsigned seed, Tri& L, Tri& U, std::vector<double>& dinv) {
  std::mt19937 g(seed);
  std::uniform_real_distribution<double> d(-1, 1);
  for (int i = 0; i < nx * ny * nz; i++) {
    const int x = i % nx, y = i / nx % ny, z = i / (nx * ny);
    for (int up = 0; up < 2; up++) {
      Tri& M = up ? U : L;
      for (int c = std::max(0, z - 1); c <= std::min(nz - 1, z + 1); c++)
        for (int b = std::max(0, y - reach); b <= std::min(ny - 1, y + reach); b++)
          for (int a = std::max(0, x - reach); a <= std::min(nx - 1, x + reach); a++) {
            const int j = (c * ny + b) * nx + a;
            if (up ? j <= i : j >= i) continue;
            M.cj.push_back(j);
            M.va.push_back((float)(d(g) / 60));
          }
      M.rp.push_back((int)M.cj.size());
    }
    dinv.push_back((float)(1.0 + 0.2 * d(g)));
  }
}

// Rounding of the lower pass of 16-byte values, some 150 entries a row, against
// 80 bits: the tasks' sums and those of eight lanes (lane l adds every eighth
// entry, then pairs).  The tasks have 1.08 times the error of the lanes here;
// 1.29 times it with one set of four sums that runs through.
static bool wide_rounding() {
  Tri L, U;
  std::vector<double> dinv;
  grid(40, 40, 12, 5, 5, L, U, dinv);
  const int n = (int)dinv.size();
  std::mt19937 g(3);
  std::uniform_real_distribution<double> d(0.5, 1);
  for (double& v : L.va) v = -d(g) / 150;
  std::vector<Wide> im(L.va.size());
  for (size_t k = 0; k < im.size(); k++) {
    im[k].x = L.va[k];
    im[k].y = 0.1 * L.va[k] * d(g);
  }
  auto lv = [&](int k) { return im[k]; };
  auto uv = [&](int k) { return Wide(U.va[k]); };
  auto dv = [&](int) { return Wide(1.0); };
  FlowPack<Wide> pu, pl;
  using C = FlowCfg<Wide, 1>;
  const std::vector<int> dom = {0, n};
  REQ((flow_pack<Wide, C>(n, U.rp.data(), U.cj.data(), uv, true, dom, &dv, nullptr, pu)));
  REQ((flow_pack<Wide, C>(n, L.rp.data(), L.cj.data(), lv, false, dom, &dv, &pu.slot_of_row, pl)));
  std::vector<Wide> b(n), y;
  for (Wide& v : b) v.x = d(g), v.y = d(g);
  REQ((walk<Wide, C>(pl, n, false, dom, b, y)));
  std::vector<long double> rx(n), ry(n);
  std::vector<Wide> e(n);
  long double flow = 0, lanes = 0;
  for (int i = 0; i < n; i++) {
    long double sx = 0, sy = 0;
    Wide s[8];
    for (int k = L.rp[i]; k < L.rp[i + 1]; k++) {
      const int j = L.cj[k];
      sx += (long double)im[k].x * rx[j] - (long double)im[k].y * ry[j];
      sy += (long double)im[k].x * ry[j] + (long double)im[k].y * rx[j];
      s[(k - L.rp[i]) % 8] += im[k] * e[j];
    }
    for (int o = 4; o > 0; o /= 2)
      for (int u = 0; u < o; u++) s[u] += s[u + o];
    rx[i] = b[i].x - sx;
    ry[i] = b[i].y - sy;
    e[i] = b[i] - s[0];
    const Wide& v = y[(size_t)pu.slot_of_row[i]];
    flow += (v.x - rx[i]) * (v.x - rx[i]) + (v.y - ry[i]) * (v.y - ry[i]);
    lanes += (e[i].x - rx[i]) * (e[i].x - rx[i]) + (e[i].y - ry[i]) * (e[i].y - ry[i]);
  }
  std::printf("rounding of 16-byte sums against eight lanes: %.3f\n", (double)std::sqrt(flow / lanes));
  REQ(flow <= 1.15L * 1.15L * lanes);
  return true;
}

int main() {
  struct Case {
    std::vector<int> dom;
    int deg, back, longrow;
  };
  std::vector<Case> cases;
  for (int n : {1, 2, 31, 32, 33, 64, 95, 417, 1000}) cases.push_back({{0, n}, 4, 40, 0});  // edges of a task
  for (int n : {1, 33, 5000}) cases.push_back({{0, n}, 0, 1, 0});     // one level
  cases.push_back({{0, 700}, 1, 1, 0});                               // a chain: one row a task
  cases.push_back({{0, 40, 40, 700, 703}, 6, 60, 0});                 // an empty and a tiny subdomain
  cases.push_back({{0, 3000}, 8, 200, 90});                           // long rows
  cases.push_back({{0, 40000}, 5, 30, 0});                            // ring wraps
  cases.push_back({{0, 30000}, 6, 9000, 0});                          // operands older than the ring
  cases.push_back({{0, 30000, 60000}, 12, 2500, 0});                  // some older, some not
  int bad = 0, packed = 0;
  for (size_t q = 0; q < cases.size(); q++) {
    Tri L, U;
    std::vector<double> dinv;
    make(cases[q].dom, cases[q].deg, cases[q].back, cases[q].longrow, 7 + (unsigned)q, L, U, dinv);
    std::vector<float> kf;
    std::vector<double> kd;
    std::vector<Wide> kw;
    // sums of at most 90 products of values below one, in either order
    const int rc[] = {solve<float, 1>(L, U, dinv, cases[q].dom, 2e-6, &kf),
                      solve<float, 2>(L, U, dinv, cases[q].dom, 2e-6, &kf),
                      solve<float, 4>(L, U, dinv, cases[q].dom, 2e-6, &kf),
                      solve<double, 1>(L, U, dinv, cases[q].dom, 4e-15, &kd),
                      solve<double, 4>(L, U, dinv, cases[q].dom, 4e-15, &kd),
                      solve<Wide, 1>(L, U, dinv, cases[q].dom, 4e-15, &kw),
                      solve<Wide, 4>(L, U, dinv, cases[q].dom, 4e-15, &kw),
                      solve<float, 1, SysFlowCfg<float>>(L, U, dinv, cases[q].dom, 2e-6, nullptr),
                      solve<float, 4, FlowCfg<float, 4, true>>(L, U, dinv, cases[q].dom, 2e-6, &kf)};
    for (int r : rc) {
      bad += r == 1;
      packed += r == 0;
      if (r == 1) std::printf("case %zu\n", q);
    }
  }
  // chunks of few tasks: some 21 entries a row, under every layout
  {
    Tri L, U;
    std::vector<double> dinv;
    grid(48, 48, 16, 2, 5, L, U, dinv);
    const std::vector<int> dom = {0, (int)dinv.size()};
    const int rc[] = {solve<float, 1>(L, U, dinv, dom, 2e-6, nullptr),
                      solve<float, 4>(L, U, dinv, dom, 2e-6, nullptr),
                      solve<double, 1>(L, U, dinv, dom, 4e-15, nullptr),
                      solve<double, 4>(L, U, dinv, dom, 4e-15, nullptr),
                      solve<Wide, 1>(L, U, dinv, dom, 4e-15, nullptr),
                      solve<Wide, 4>(L, U, dinv, dom, 4e-15, nullptr),
                      solve<float, 1, FlowCfg<float, 1, true>>(L, U, dinv, dom, 2e-6, nullptr),
                      solve<double, 4, FlowCfg<double, 4, true>>(L, U, dinv, dom, 4e-15, nullptr),
                      solve<float, 1, SysFlowCfg<float>>(L, U, dinv, dom, 2e-6, nullptr),
                      solve<double, 1, SysFlowCfg<double>>(L, U, dinv, dom, 4e-15, nullptr)};
    for (const int& r : rc) {
      bad += r != 0;
      if (r) std::printf("grid: layout %d, result %d\n", (int)(&r - rc), r);
    }
  }
  if (!wide_rounding()) bad++;
  // what the kernel does not take is refused: coupled subdomains, a row that no task can hold
  {
    Tri L, U;
    std::vector<double> dinv;
    make({0, 64}, 4, 40, 0, 3, L, U, dinv);
    if (solve<float, 1>(L, U, dinv, {0, 30, 64}, 1, nullptr) != 2) bad++;
    Tri L2, U2;
    std::vector<double> d2;
    make({0, 6000}, 0, 6000, 5000, 3, L2, U2, d2);
    if (solve<double, 1>(L2, U2, d2, {0, 6000}, 1, nullptr) != 2) bad++;
  }
  // and factors of mostly far operands, where the caller sets a limit; far operands are no reason where they are few
  {
    using C = FlowCfg<float, 1>;
    FlowPack<float> o;
    auto pack = [&](int n, int deg, int back, long long most, int nsub) {
      Tri L, U;
      std::vector<double> dinv;
      std::vector<int> dom = {0};
      for (int c = 1; c <= nsub; c++) dom.push_back(n * c);
      make(dom, deg, back, 0, 11, L, U, dinv);
      auto uv = [&](int k) { return (float)U.va[k]; };
      auto dv = [&](int i) { return (float)dinv[i]; };
      return flow_pack<float, C>(n * nsub, U.rp.data(), U.cj.data(), uv, true, dom, &dv, nullptr, o, most);
    };
    if (!pack(50000, 6, 50000, LLONG_MAX, 1) || o.nfar < 75000) bad++;
    const long long far = o.nfar;
    if (pack(50000, 6, 50000, far / 2, 1) || !pack(50000, 6, 50000, 2 * far, 1)) bad++;
    if (!pack(50000, 6, 50000, 2 * far, 2)) bad++;  // the limit is a subdomain's
    if (!pack(50000, 6, 30, 0, 1)) bad++;
  }
  std::printf("%d layouts solved, %d bad\n", packed, bad);
  return bad || packed < 100;
}
