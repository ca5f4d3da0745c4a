// The step's set-up kernels from their sources, on the CPU (cuda_runtime.h beside this file).
//   setup levels <columns> <rows> <seed>   multigrid levels by a warp and by a thread per coarse row, bit for bit
//   setup inverse <n> <seed>               the coarsest level's dense inverse against long double arithmetic
//   setup mirrors <types> <seed>           the mirrors of a box whose four sides have the given types (1 wall, 2
//                                          periodic): prints their number and every one of them; CORNER_LIST
//                                          is the corners' list length
#include "cuda_runtime.h"

#include "vebi_ctx.cuh"
#undef VEBI_LAUNCH
#define VEBI_LAUNCH(x, kern, grid, block, ...) emu::run(grid, block, [&] { kern(__VA_ARGS__); })
#ifdef CORNER_LIST
#define MIR_LIST CORNER_LIST
#include "vebi_geom.cu"
#else
#include "vebi_mg.cu"
#endif

namespace vebi {
unsigned int atom_add_release(unsigned int* a, unsigned int v) { return atomicAdd(a, v); }
unsigned int ld_acquire(const unsigned int* a) {
  emu::poll();
  return *a;
}
namespace fp {
inline float rcp_start(float m) { return 1.0f / m; }
inline float rsqrt_start(float m) { return 1.0f / std::sqrt(m); }
}  // namespace fp
}  // namespace vebi

using namespace vebi;

namespace {

uint64_t state;
uint64_t next() {  // SplitMix64
  uint64_t z = (state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
double uniform() { return (double)(next() >> 11) * 0x1p-53; }

#ifndef CORNER_LIST
struct Level {
  std::vector<int> cnt, col;
  std::vector<double> val, diag, dinv;
  MgLevel l{};
  Level(int gx, int gy)
      : cnt(gx * gy, -1), col((size_t)MG_SLOTS * gx * gy, -1), val((size_t)MG_SLOTS * gx * gy, 0.0), diag(gx * gy, 0.0),
        dinv(gx * gy, 0.0) {
    l.n = gx * gy;
    l.gx = gx;
    l.gy = gy;
    l.cnt = cnt.data();
    l.col = col.data();
    l.val = val.data();
    l.diag = diag.data();
    l.dinv = dinv.data();
  }
  bool operator==(const Level& o) const {
    auto same = [](const auto& a, const auto& b) { return std::memcmp(a.data(), b.data(), a.size() * sizeof(a[0])) == 0; };
    return same(cnt, o.cnt) && same(col, o.col) && same(val, o.val) && same(diag, o.diag) && same(dinv, o.dinv);
  }
};

// a grid of cells of 0 to 40 particles, some of them empty and some with mirrors after the particles, each
// particle with pairs of (cell, value): its own cell, some of the 3x3 around it and some across the grid;
// crowded: a cell whose row takes more columns than a level holds
int levels(int gx, int gy, bool crowded) {
  Scal s[2];
  std::memset(s, 0, sizeof(s));
  const int nc = gx * gy;
  std::vector<int> start(nc), in(nc), ip, rcnt;
  std::vector<std::vector<std::pair<int, double>>> pairs;
  int n = 0;
  for (int c = 0; c < nc; ++c) in[c] = next() % 5 == 0 ? 0 : (int)(next() % (c == 0 ? 41 : 9));
  if (crowded) in[nc / 2] = 12;
  for (int c = 0; c < nc; ++c) n += in[c];
  int at = 0;
  for (int c = 0; c < nc; ++c) {
    start[c] = (int)ip.size();
    for (int k = 0; k < in[c]; ++k) {
      ip.push_back(at++);
      std::vector<std::pair<int, double>> p{{c, 4.0 + uniform()}};
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          const int x = c % gx + dx, y = c / gx + dy;
          if ((dx || dy) && x >= 0 && x < gx && y >= 0 && y < gy && next() % 3) p.push_back({x + y * gx, -uniform()});
        }
      const int far = crowded && c == nc / 2 ? 6 : (int)(next() % 2);
      for (int q = 0; q < far; ++q) p.push_back({(int)(next() % nc), -uniform()});
      if ((int)p.size() > MG_ROW_SLOTS) p.resize(MG_ROW_SLOTS);
      pairs.push_back(p);
    }
    const int mirrors = next() % 4 == 0 ? 3 : 0;
    for (int k = 0; k < mirrors; ++k) ip.push_back(n + (int)(next() % 7));
    in[c] += mirrors;
  }
  std::vector<int> ragg((size_t)MG_ROW_SLOTS * n, -1);
  std::vector<double> rval((size_t)MG_ROW_SLOTS * n, 0.0);
  rcnt.assign(n, 0);
  for (int i = 0; i < n; ++i) {
    rcnt[i] = (int)pairs[i].size();
    for (int t = 0; t < rcnt[i]; ++t) {
      ragg[(size_t)t * n + i] = pairs[i][t].first;
      rval[(size_t)t * n + i] = pairs[i][t].second;
    }
  }
  int full = 0;  // rows of more columns than a level holds
  for (int c = 0, i = 0; c < nc; ++c) {
    std::vector<char> col(nc, 0);
    for (; i < n && pairs[i][0].first == c; ++i)
      for (auto& p : pairs[i]) col[p.first] = p.first != c;
    full += std::count(col.begin(), col.end(), 1) > MG_SLOTS;
  }
  Consts c{};
  c.npfb = n;
  Dev d{};
  d.ip = ip.data();
  d.cell_start = start.data();
  d.cell_cnt = in.data();
  int bad = 0, depth = 0;
  Level T(gx, gy), W(gx, gy);
  d.s = &s[0];
  emu::run(grid_for(nc), TPB, [&] { k_mg_level1(c, d, T.l, ragg.data(), rval.data(), rcnt.data()); });
  d.s = &s[1];
  emu::run(grid_for(32ll * nc), TPB, [&] { k_mg_level1_warp(c, d, W.l, ragg.data(), rval.data(), rcnt.data()); });
  bad += !(T == W) || s[0].mg_fail != s[1].mg_fail || s[0].mg_fail != (full ? 1 : 0);
  while (T.l.n > 1 && !full) {
    const int hx = (T.l.gx + 1) / 2, hy = (T.l.gy + 1) / 2;
    Level t(hx, hy), w(hx, hy);
    emu::run(grid_for(t.l.n), TPB, [&] { k_mg_coarsen(T.l, t.l, &s[0]); });
    emu::run(grid_for(32ll * w.l.n), TPB, [&] { k_mg_coarsen_warp(T.l, w.l, &s[1]); });
    bad += !(t == w) || s[0].mg_fail != s[1].mg_fail;
    ++depth;
    if (s[0].mg_fail) break;  // a row full of columns: the solve goes on without the multigrid
    T = t;
    T.l = t.l;
    T.l.cnt = T.cnt.data();
    T.l.col = T.col.data();
    T.l.val = T.val.data();
    T.l.diag = T.diag.data();
    T.l.dinv = T.dinv.data();
  }
  std::printf("%d particles, %d levels, %d rows too full, %d differ\n", n, depth + 1, full, bad);
  return bad;
}

// a matrix whose pivots are not on its diagonal, so that rows are exchanged: a shuffled dominant one
int inverse(int n) {
  Level K(n, 1);
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = i;
  for (int i = n - 1; i > 0; --i) std::swap(perm[i], perm[next() % (i + 1)]);
  std::vector<long double> M((size_t)n * 2 * n, 0.0L);
  for (int r = 0; r < n; ++r) {
    std::vector<int> cols;
    for (int q = 0; q < n; ++q)
      if (q != r && (q == perm[r] || (next() % 4 == 0 && (int)cols.size() < MG_SLOTS - 1))) cols.push_back(q);
    K.cnt[r] = (int)cols.size();
    for (int t = 0; t < K.cnt[r]; ++t) {
      K.col[(size_t)t * n + r] = cols[t];
      K.val[(size_t)t * n + r] = uniform() - 0.5 + (cols[t] == perm[r] ? 8.0 : 0.0);
      M[(size_t)r * 2 * n + cols[t]] = K.val[(size_t)t * n + r];
    }
    K.diag[r] = uniform() - 0.5 + (perm[r] == r ? 8.0 : 0.0);
    M[(size_t)r * 2 * n + r] = K.diag[r];
    M[(size_t)r * 2 * n + n + r] = 1.0L;
  }
  std::vector<double> inv((size_t)n * n, 0.0);
  int ok = -1;
  emu::run(1, dim3(32, 32), [&] { k_mg_coarse_inverse(K.l, inv.data(), &ok, 0); });
  if (ok != 1) return 1;
  int swaps = 0;
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int r = k; r < n; ++r)
      if (std::fabs(M[(size_t)r * 2 * n + k]) > std::fabs(M[(size_t)p * 2 * n + k])) p = r;
    swaps += p != k;
    for (int q = 0; q < 2 * n; ++q) std::swap(M[(size_t)k * 2 * n + q], M[(size_t)p * 2 * n + q]);
    const long double d = M[(size_t)k * 2 * n + k];
    for (int q = 0; q < 2 * n; ++q) M[(size_t)k * 2 * n + q] /= d;
    for (int r = 0; r < n; ++r) {
      const long double f = M[(size_t)r * 2 * n + k];
      if (r != k)
        for (int q = 0; q < 2 * n; ++q) M[(size_t)r * 2 * n + q] -= f * M[(size_t)k * 2 * n + q];
    }
  }
  // a row of the shuffled matrix is 8 off its other entries' 0.5: condition number below 10, growth 1, n steps
  long double err = 0.0L, top = 0.0L;
  for (int r = 0; r < n; ++r)
    for (int q = 0; q < n; ++q) {
      err = std::max(err, std::fabs(M[(size_t)r * 2 * n + n + q] - inv[(size_t)r * n + q]));
      top = std::max(top, std::fabs(M[(size_t)r * 2 * n + n + q]));
    }
  std::printf("%d rows, %d exchanges, error %.3Lg of %.3Lg\n", n, swaps, err, top);
  return err > 10.0L * n * 0x1p-53L * top || (n > 4 && swaps == 0);
}

#else
int mirrors(const char* types) {
  Ctx x;
  Consts& c = x.c;
  std::memset(&c, 0, sizeof(c));
  c.dx = 0.05;
  c.h = 1.3 * c.dx;
  c.sup_size = 3.0 * c.h;
  c.nb = 4;
  const double node[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}}, edge[4][2] = {{1, 0}, {0, 1}, {-1, 0}, {0, -1}};
  for (int b = 0; b < 4; ++b) {
    for (int q = 0; q < 2; ++q) c.b_node[b][q] = node[b][q], c.b_edge[b][q] = edge[b][q];
    c.b_type[b] = types[b] - '0';
    c.b_pp[b] = (b + 2) % 4;
    c.b_elen[b] = 1.0;
    c.b_corner_angle[b] = 0.5 * PI;
    c.b_vel[b] = 0.1 * b;
    c.b_thermal[b] = 0.2 * b;
    c.b_rot[b][0] = c.b_rot[b][3] = 1.0;
    const int n1 = (b + 1) % 4;
    c.bl_a[b] = (float)-edge[b][1];
    c.bl_b[b] = (float)edge[b][0];
    c.bl_c[b] = (float)-(node[n1][0] * node[b][1] - node[n1][1] * node[b][0]);
  }
  c.near_band = (float)(c.sup_size + 0.1 * c.dx + 4.0e-6 * 2.0);
  c.bf[0] = 0.3;
  c.bf[1] = -1.0;
  c.Wi = 1.0;
  // 20 wall particles along the bottom and 580 in the box
  c.nbS = 20;
  c.npfb = 600;
  c.mcap = 2 * c.npfb;
  c.cap = c.npfb + c.mcap;
  Dev& d = x.d;
  Scal s;
  std::memset(&s, 0, sizeof(s));
  s.dt = 1.0e-3;
  d.s = &s;
  std::vector<double> f[8];
  for (auto& a : f) a.assign(c.cap, 0.0);
  std::vector<int> irel(c.cap, -1), vrel(c.cap, 0), blk(64), list(2 * MIR_LIST + 2);
  std::vector<uint8_t> bin(c.cap, 0);
  std::vector<unsigned> bits(8 * 32);
  d.rx = f[0].data(), d.ry = f[1].data(), d.ux = f[2].data(), d.uy = f[3].data(), d.th = f[4].data();
  d.dP_mp = f[5].data();
  d.irel = irel.data(), d.vrel = vrel.data(), d.inbin = bin.data();
  d.sel_blk = blk.data(), d.sel_bits = bits.data(), d.mir_list = list.data();
  for (int i = 0; i < c.npfb; ++i) {
    d.rx[i] = i < c.nbS ? (i + 0.5) / 20.0 : uniform();
    d.ry[i] = i < c.nbS ? 0.0 : uniform();
    d.ux[i] = uniform() - 0.5;
    d.uy[i] = uniform() - 0.5;
    d.th[i] = uniform();
  }
  x.nsm = 4;
  launch_mirrors(x);
  std::printf("%d mirrors, status %d\n", s.nmirror, s.error);
  for (int j = c.npfb; j < c.npfb + s.nmirror; ++j)
    std::printf("%d %d %a %a %a %a %a %a\n", irel[j], vrel[j], d.rx[j], d.ry[j], d.ux[j], d.uy[j], d.th[j], d.dP_mp[j]);
  std::fprintf(stderr, "%d past a wall's end, %d about a node\n", s.n_end, s.n_node);
  return s.error || s.np != c.npfb + s.nmirror;
}
#endif

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  auto arg = [&](int k) { return k < argc ? std::atoi(argv[k]) : 0; };
  state = 0x2545f4914f6cdd1dull + arg(argc - 1);
#ifdef CORNER_LIST
  if (what == "mirrors") return mirrors(argv[2]);
#else
  if (what == "levels") return levels(arg(2), arg(3), false) + levels(arg(2), arg(3), true);
  if (what == "inverse") return inverse(arg(2));
#endif
  return 2;
}
