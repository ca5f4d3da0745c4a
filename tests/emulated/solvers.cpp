// The PPE solvers whose rows are spread over all SMs, from their sources, on the CPU (cuda_runtime.h
// beside this file): what they return must not depend on which block is ahead.
//   solvers resident <rows> <SMs> <closed> <warm>   the time step's
//   solvers noalloc <rows> <SMs> <closed>           vebi_ppe_solve_noalloc, also against the kernel
//                                                   it keeps for GPUs of too few SMs
// prints the iterations and exits 0 if the blocks' two orders give the same bits.
#include "cuda_runtime.h"

#include "vebi_noalloc.cu"
#include "vebi_resident.cu"

extern "C" void vebi_set_last_error_internal(const char* msg) { std::printf("%s\n", msg); }

namespace vebi {
namespace {
thread_local double na_mat[232448 / sizeof(double)];  // a block's dynamic shared memory
}
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

uint64_t state = 0x2545f4914f6cdd1dull;
double uniform() {  // SplitMix64, [0, 1)
  uint64_t z = (state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
}

// the Laplacian of a ring with random chords and a hub (symmetric weights), and a right-hand side; closed: zero
// row sums and a mean-free right-hand side, open: every 50th row a free surface (diagonal 1e30)
struct System {
  int n, width = 0;
  std::vector<int> cnt, col;
  std::vector<double> val, diag, rhs;
  System(int n_, bool closed) : n(n_), cnt(n_, 0), diag(n_, 0.0), rhs(n_) {
    std::vector<std::vector<std::pair<int, double>>> row(n);
    auto join = [&](int a, int b) {
      if (a == b) return;
      const double w = 0.5 + uniform();
      row[a].push_back({b, -w});
      row[b].push_back({a, -w});
    };
    for (int i = 0; i < n; ++i) {
      join(i, (i + 1) % n);
      for (int k = 0; k < 3; ++k) join(i, (int)(uniform() * n));
    }
    for (int k = 0; k < 90; ++k) join(0, (int)(uniform() * n));  // more slots than the solvers keep in a row
    for (auto& r : row) width = std::max(width, (int)r.size());
    col.assign((size_t)width * n, 0);
    val.assign((size_t)width * n, 0.0);
    double mean = 0.0;
    for (int i = 0; i < n; ++i) {
      cnt[i] = (int)row[i].size();
      for (int k = 0; k < cnt[i]; ++k) {
        col[(size_t)k * n + i] = row[i][k].first;
        val[(size_t)k * n + i] = row[i][k].second;
        diag[i] -= row[i][k].second;
      }
      rhs[i] = 100.0 * (uniform() - 0.5);
      mean += rhs[i] / n;
    }
    for (int i = 0; i < n; ++i) {
      if (closed) rhs[i] -= mean;
      else if (i % 50 == 0) diag[i] = 1.0e30;
    }
  }
};

struct Result {
  std::vector<double> x;
  int iters = 0, status = 0, warnings = 0;
  double residual = 0.0;
  bool operator==(const Result& o) const {
    return iters == o.iters && status == o.status && warnings == o.warnings &&
           std::memcmp(&residual, &o.residual, 8) == 0 && std::memcmp(x.data(), o.x.data(), 8 * x.size()) == 0;
  }
};

Result resident(const System& s, bool closed, bool warm) {
  std::vector<double> pinv(s.n), sinv(s.n), part(resident_partials(s.n)), B = s.rhs;
  Result r;
  r.x.assign(s.n, 0.0);
  if (warm)
    for (int i = 0; i < s.n; ++i) r.x[i] = std::sin(0.1 * i);
  Scal sc;
  std::memset(&sc, 0, sizeof(sc));
  BiArgs a{};
  a.pinv = pinv.data();
  a.sinv = sinv.data();
  a.part = part.data();
  a.P = r.x.data();
  a.B = B.data();
  a.diag = s.diag.data();
  a.val = s.val.data();
  a.col = s.col.data();
  a.cnt = s.cnt.data();
  a.sc = &sc;
  a.stride = a.n = s.n;
  a.itermax = 60;
  a.tol = 1.0e-8;
  a.warm = warm ? 1 : 0;
  Ctx x;
  x.nsm = emu::multiprocessors;
  x.coop_blocks = 5 * x.nsm;
  if (!launch_bicgstab_resident(x, a, closed)) std::exit(2);
  r.iters = sc.ls_iters;
  r.residual = sc.ls_residual;
  r.status = sc.error;
  r.warnings = sc.warnings;
  return r;
}

Result noalloc(const System& s, bool closed, int sms) {
  emu::multiprocessors = emu::device = sms;  // a device of its own: its set-up is kept per device
  Result r;
  r.x.assign(s.n, 1.0);
  r.status = vebi_ppe_solve_noalloc(s.cnt.data(), s.col.data(), s.val.data(), s.diag.data(), s.rhs.data(), r.x.data(),
                                    s.n, s.n, closed ? 1 : 0, 1.0e-8, 60, nullptr, &r.iters, &r.residual);
  return r;
}

int compare(const char* what, const Result& a, const Result& b) {
  std::printf("%s: %d and %d iterations, residual %.3g and %.3g, status %d and %d\n", what, a.iters, b.iters,
              a.residual, b.residual, a.status, b.status);
  return a == b && a.status == 0 && a.residual <= 1.0e-8 && a.iters >= 2 ? 0 : 1;
}

}  // namespace

int main(int argc, char** argv) {
  auto arg = [&](int k) { return k < argc ? std::atoi(argv[k]) : 0; };
  const std::string what = argc > 1 ? argv[1] : "";
  const System s(arg(2), arg(4) != 0);
  emu::multiprocessors = arg(3);
  auto in_order = [&](bool fair, auto solve) {
    emu::fair = fair;
    return solve();
  };
  if (what == "resident") {
    auto solve = [&] { return resident(s, arg(4) != 0, arg(5) != 0); };
    const Result level = in_order(true, solve);
    return compare("blocks level / one ahead", level, in_order(false, solve));
  }
  if (what == "noalloc") {
    auto solve = [&] { return noalloc(s, arg(4) != 0, arg(3)); };
    const Result level = in_order(true, solve), ahead = in_order(false, solve);
    const int bad = compare("blocks level / one ahead", level, ahead);
    // one SM holds 512 rows: the persistent kernel takes a larger system there
    return bad | compare("spread / persistent", level, in_order(false, [&] { return noalloc(s, arg(4) != 0, 1); }));
  }
  return 2;
}
