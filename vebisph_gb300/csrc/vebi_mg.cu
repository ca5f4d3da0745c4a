// vebi_mg.cu -- opt-in multigrid preconditioner of the PPE BiCGSTAB (VEBI_PRECOND_MULTIGRID).
// No counterpart in the reference, which solves closed domains unpreconditioned
// (SPARSE_PBICGSTAB_nonull, linear_solver.F90:275-425, M = 1 at :318) and open domains with
// Jacobi (SPARSE_PBICGSTAB, :82-227).
//
// Hierarchy.  Level 1 aggregates the particles by the cell they sit in: the cell grid of
// cell_griddin.F90:13-24, whose cell lists the neighbour search built this step.  Each further
// level agglomerates 2x2 aggregates of the level below, until at most MG_COARSEST remain.
// Interpolation is piecewise constant, so a coarse matrix is the Galerkin product R A P: the
// sum of the couplings between two aggregates.  Coarse matrices are ELL with at most MG_SLOTS
// off-diagonal slots per row (the 3x3 neighbourhood plus partners across periodic boundaries);
// a row that needs more sets mg_fail, and that step solves without the preconditioner.
//
// V-cycle, one per preconditioning step: one damped Jacobi sweep (MG_OMEGA) from zero, the
// residual, restriction (the sum over each aggregate), the coarser levels, prolongation scaled
// by MG_GAMMA (over-correction for piecewise-constant interpolation) and, on the coarse levels,
// one post-smoothing sweep; the particle level is pre-smoothed only (two particle-level
// products per V-cycle cost more than the iterations they save).  The coarsest level takes
// MG_SWEEPS Jacobi sweeps.  Levels of at most MG_BLOCK_ROWS rows run in
// block 0 alone with block barriers: one SM's FP64 pipe takes longer over a larger level than the
// two grid barriers (1-3 us each) that the level costs on the whole grid.  Every sum runs in a fixed order.
//
// Solver.  BiCGSTAB with right preconditioning, in the persistent cooperative kernel of the
// unpreconditioned solver: the same recurrences, residual test and, for closed domains, mean
// removal.  The preconditioned directions are made mean-free, so the solution keeps the zero
// mean of the reference's iterates.  The V-cycle reads only its own rows of the vector it is
// applied to, so it needs no barrier before it.
#include "vebi_solver.cuh"

namespace vebi {

#define ELL(k, i) ((size_t)(k) * c.npfb + (i))

// ---------------------------------------------------------------- set-up (every step)
// add v to column `col` of a row's slot table of capacity CAP; false when the table is full
template <int CAP = MG_SLOTS>
__device__ __forceinline__ bool slot_add(int* tc, double* tv, int& m, int col, double v) {
  int t = 0;
  while (t < m && tc[t] != col) ++t;
  if (t == m) {
    if (m == CAP) return false;
    tc[m] = col;
    tv[m] = 0.0;
    ++m;
  }
  tv[t] += v;
  return true;
}

__device__ __forceinline__ void slot_store(const MgLevel& L, int row, const int* tc, const double* tv, int m,
                                           double dg) {
  for (int t = 0; t < m; ++t) {
    L.col[(size_t)t * L.n + row] = tc[t];
    L.val[(size_t)t * L.n + row] = tv[t];
  }
  L.cnt[row] = m;
  L.diag[row] = dg;
  L.dinv[row] = dg != 0.0 ? 1.0 / dg : 0.0;
}

// Level 1 in two passes.  Rows: one thread per PPE row sums the row by the cell of each
// column (its own cell first, with the diagonal) into MG_ROW_SLOTS (cell, value) pairs,
// [t][i] layout.  Cells: one thread per cell merges its particles' pairs in ascending particle
// order.  val32 (mixed precision) replaces the FP64 values when given.
//
// A row's columns lie in the 3x3 cells around its own, except the parents of mirrors across
// periodic boundaries.  The nine cells own + dy*ncx + dx are summed in shared memory by direct
// index (the key difference alone picks the slot: nine distinct keys, nine distinct slots);
// any other cell goes to a short searched list.  Each cell's sum runs in slot order, as a
// searched table's would; the pairs come out own cell first, then the 3x3 in key order, then
// the list.
//
// The same sums also go out by direction for the output pass of the V-cycle: rv9[k][i] for the
// eight directions q = 0..8 without the own cell (k = q, or q - 1 past it), zero where the row
// has no column, and rx[i] = (first list slot) | (pair count << 8) | (used directions << 16).
// The output pass then computes every gather address from the row's own cell, without a
// dependent load of the pair's cell.  With val32 (mixed precision) the direction values are
// FP32, rv9 read as float [8][npfb].
__global__ void __launch_bounds__(TPB) k_mg_rows(Consts c, Dev d, const float* __restrict__ val32,
                                                 int* __restrict__ ragg, double* __restrict__ rval,
                                                 int* __restrict__ rcnt, double* __restrict__ rv9,
                                                 int* __restrict__ rx) {
  __shared__ double nb9[9][TPB];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.npfb) return;
  const int own = d.cellpart[i];
  if (own < 0) {  // a binned particle belongs to no cell
    rcnt[i] = 0;
    rx[i] = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (val32) ((float*)rv9)[(size_t)k * c.npfb + i] = 0.f;
      else rv9[(size_t)k * c.npfb + i] = 0.0;
    }
    return;
  }
  double* acc = &nb9[0][threadIdx.x];  // slot q at acc[q * TPB]
#pragma unroll
  for (int q = 0; q < 9; ++q) acc[q * TPB] = 0.0;
  acc[4 * TPB] = d.ppe_diag[i];
  unsigned used = 1u << 4;
  int tc[MG_ROW_SLOTS - 9];
  double tv[MG_ROW_SLOTS - 9];
  int m = 0;
  bool ok = true;
  const int ncx = c.ncx;
  const int cnt = d.ij_count[i];
  for (int k = 0; k < cnt; ++k) {
    const int a = d.cellpart[d.ppe_col[ELL(k, i)]];
    const double v = val32 ? widen(val32[ELL(k, i)]) : d.ppe_val[ELL(k, i)];
    if (a < 0) continue;
    const int del = a - own;
    const int r = del + ncx + 1;  // row dy=-1 at 0..2, dy=0 at ncx..ncx+2, dy=+1 at 2ncx..2ncx+2
    int q = -1;
    if (r >= 0 && r <= 2) q = r;
    else if (r >= ncx && r <= ncx + 2) q = 3 + r - ncx;
    else if (r >= 2 * ncx && r <= 2 * ncx + 2) q = 6 + r - 2 * ncx;
    if (q >= 0) {
      acc[q * TPB] += v;
      used |= 1u << q;
    } else {
      ok &= slot_add<MG_ROW_SLOTS - 9>(tc, tv, m, a, v);
    }
  }
  int t = 0;
  ragg[i] = own;
  rval[i] = acc[4 * TPB];
  ++t;
  unsigned used8 = 0;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    if (q == 4) continue;
    const int k = q < 4 ? q : q - 1;
    const bool u = (used & (1u << q)) != 0;
    if (val32) ((float*)rv9)[(size_t)k * c.npfb + i] = u ? narrow(acc[q * TPB]) : 0.f;
    else rv9[(size_t)k * c.npfb + i] = u ? acc[q * TPB] : 0.0;
    if (!u) continue;
    used8 |= 1u << k;
    ragg[(size_t)t * c.npfb + i] = own + (q / 3 - 1) * ncx + (q % 3 - 1);
    rval[(size_t)t * c.npfb + i] = acc[q * TPB];
    ++t;
  }
  const int t_list = t;
  for (int e = 0; e < m; ++e, ++t) {
    ragg[(size_t)t * c.npfb + i] = tc[e];
    rval[(size_t)t * c.npfb + i] = tv[e];
  }
  rcnt[i] = t;
  rx[i] = t_list | (t << 8) | (int)(used8 << 16);
  if (!ok) d.s->mg_fail = 1;
}

__global__ void k_mg_level1(Consts c, Dev d, MgLevel L, const int* __restrict__ ragg,
                            const double* __restrict__ rval, const int* __restrict__ rcnt) {
  const int cc = blockIdx.x * blockDim.x + threadIdx.x;
  if (cc >= L.n) return;
  int tc[MG_SLOTS];
  double tv[MG_SLOTS];
  int m = 0;
  double dg = 0.0;
  bool ok = true;
  const int s0 = d.cell_start[cc], ne = d.cell_cnt[cc];
  for (int q = 0; q < ne; ++q) {
    const int i = d.ip[s0 + q];
    if (i >= c.npfb) break;  // mirrors follow the particles in a sorted cell list
    const int mi = rcnt[i];
    for (int t = 0; t < mi; ++t) {
      const int a = ragg[(size_t)t * c.npfb + i];
      const double v = rval[(size_t)t * c.npfb + i];
      if (a == cc) dg += v;
      else ok &= slot_add(tc, tv, m, a, v);
    }
  }
  slot_store(L, cc, tc, tv, m, dg);
  if (!ok) d.s->mg_fail = 1;
}

// A coarse row by a warp.  Lane m keeps the m-th column in order of first appearance and its sum,
// the last lane the row's own column (the diagonal).  The entries come in their order, up to one a
// lane: every lane marks its column's, a column without a lane takes the next one, then the lanes
// add theirs, so each sum runs in the order of the entries, as a thread's searched table adds them.
// What bounds it: ~10 instructions per entry.  A thread per row waits for each entry's loads and
// table search in turn, ~130 us for a level-1 row however few rows there are (mg_setup has both).
struct WarpRow {
  int key, m;
  double sum;
  bool ok;
  __device__ __forceinline__ explicit WarpRow(int own)
      : key((threadIdx.x & 31) == 31 ? own : -1), m(0), sum(0.0), ok(true) {}
  __device__ __forceinline__ void add(bool in, int a, double v) {
    const int lane = threadIdx.x & 31;
    unsigned mine = 0;
    for (unsigned todo = __ballot_sync(0xffffffffu, in); todo; todo &= todo - 1) {
      const int u = __ffs(todo) - 1, au = __shfl_sync(0xffffffffu, a, u);
      if (!__ballot_sync(0xffffffffu, key == au)) {
        if (m == MG_SLOTS) { ok = false; continue; }
        if (lane == m) key = au;
        ++m;
      }
      if (key == au) mine |= 1u << u;
    }
    while (__any_sync(0xffffffffu, mine != 0)) {
      const double w = __shfl_sync(0xffffffffu, v, mine ? __ffs(mine) - 1 : lane);
      if (mine) sum += w;
      mine &= mine - 1;
    }
  }
  __device__ __forceinline__ void store(const MgLevel& L, int row) const {
    const int lane = threadIdx.x & 31;
    if (lane < m) {
      L.col[(size_t)lane * L.n + row] = key;
      L.val[(size_t)lane * L.n + row] = sum;
    }
    if (lane == 0) L.cnt[row] = m;
    if (lane == 31) {
      L.diag[row] = sum;
      L.dinv[row] = sum != 0.0 ? 1.0 / sum : 0.0;
    }
  }
};
static_assert(MG_SLOTS < 32 && MG_ROW_SLOTS == 16, "a lane per column; two particles' pairs at a time");

__global__ void __launch_bounds__(TPB) k_mg_level1_warp(Consts c, Dev d, MgLevel L, const int* __restrict__ ragg,
                                                        const double* __restrict__ rval,
                                                        const int* __restrict__ rcnt) {
  const int cc = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (cc >= L.n) return;
  WarpRow R(cc);
  const int s0 = d.cell_start[cc], ne = d.cell_cnt[cc];
  for (int q0 = 0; q0 < ne; q0 += 32) {
    int id = -1, pairs = 0;  // of particle q0 + lane; mirrors follow the particles in a sorted cell list
    if (q0 + lane < ne) {
      id = d.ip[s0 + q0 + lane];
      if (id < c.npfb) pairs = rcnt[id];
    }
    const int np = __popc(__ballot_sync(0xffffffffu, q0 + lane < ne && id < c.npfb));
    const int t = lane & 15;
    auto fetch = [&](int q, int& a, double& v) {  // pair t of particles q and q + 1
      const int from = q + (lane >> 4);
      const int i = __shfl_sync(0xffffffffu, id, from & 31), n = __shfl_sync(0xffffffffu, pairs, from & 31);
      const bool in = from < np && t < n;
      a = in ? ragg[(size_t)t * c.npfb + i] : -1;
      v = in ? rval[(size_t)t * c.npfb + i] : 0.0;
      return in;
    };
    int a, a_next;
    double v, v_next;
    bool in = fetch(0, a, v);
    for (int q = 0; q < np; q += 2) {
      const bool in_next = fetch(q + 2, a_next, v_next);
      R.add(in, a, v);
      in = in_next;
      a = a_next;
      v = v_next;
    }
    if (np < 32) break;
  }
  R.store(L, cc);
  if (!R.ok && lane == 0) d.s->mg_fail = 1;
}

__global__ void __launch_bounds__(TPB) k_mg_coarsen_warp(MgLevel F, MgLevel G, Scal* s) {
  const int C = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (C >= G.n) return;
  const int X = C % G.gx, Y = C / G.gx;
  WarpRow R(C);
  int a[4];
  double v[4];
  bool in[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // a child's diagonal, then its slots
    const int fx = 2 * X + (q & 1), fy = 2 * Y + (q >> 1), f = fx + fy * F.gx;
    in[q] = fx < F.gx && fy < F.gy && lane <= F.cnt[f];
    a[q] = -1;
    v[q] = 0.0;
    if (in[q]) {
      const size_t e = (size_t)(lane - 1) * F.n + f;
      const int cf = lane ? F.col[e] : f;
      a[q] = (cf % F.gx) / 2 + ((cf / F.gx) / 2) * G.gx;
      v[q] = lane ? F.val[e] : F.diag[f];
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) R.add(in[q], a[q], v[q]);
  R.store(G, C);
  if (!R.ok && lane == 0) s->mg_fail = 1;
}

// level l+1 from level l: one thread per coarse row sums its (up to) 2x2 child rows
__global__ void k_mg_coarsen(MgLevel F, MgLevel G, Scal* s) {
  const int C = blockIdx.x * blockDim.x + threadIdx.x;
  if (C >= G.n) return;
  const int X = C % G.gx, Y = C / G.gx;
  int tc[MG_SLOTS];
  double tv[MG_SLOTS];
  int m = 0;
  double dg = 0.0;
  bool ok = true;
  for (int q = 0; q < 4; ++q) {
    const int fx = 2 * X + (q & 1), fy = 2 * Y + (q >> 1);
    if (fx >= F.gx || fy >= F.gy) continue;
    const int f = fx + fy * F.gx;
    dg += F.diag[f];
    const int cnt = F.cnt[f];
    for (int t = 0; t < cnt; ++t) {
      const int cf = F.col[(size_t)t * F.n + f];
      const int a = (cf % F.gx) / 2 + ((cf / F.gx) / 2) * G.gx;
      const double v = F.val[(size_t)t * F.n + f];
      if (a == C) dg += v;
      else ok &= slot_add(tc, tv, m, a, v);
    }
  }
  slot_store(G, C, tc, tv, m, dg);
  if (!ok) s->mg_fail = 1;
}

// The coarsest level's dense inverse, for a direct coarse solve in the V-cycle: Gauss-Jordan
// with partial pivoting in one 32 x 32 block, a warp per row of [M | I] (at most MG_COARSEST = 32
// rows).  A step changes n of the 2n columns: those of M right of the pivot, and those of I that
// belong to the pivots so far (the pivot row's other entries of I are still zero); a lane takes one.
// (At 27 to 32 rows 32 us; all 2n columns, five block barriers a step and FP64 compares took 83.)
// A closed domain's coarse matrix is singular (its rows sum to zero: the constant is in its null
// space), so it is inverted as M + alpha 1 1^T with alpha = mean |diag| / n, which moves that
// eigenvalue to mean |diag| and leaves the mean-free solution of M x = b unchanged.  *ok = 0 (a zero
// pivot, or a level too large) makes the V-cycle fall back to Jacobi sweeps.
__global__ void __launch_bounds__(1024) k_mg_coarse_inverse(MgLevel K, double* inv, int* ok, int closed) {
  __shared__ double M[MG_COARSEST][2 * MG_COARSEST + 1];
  __shared__ int orig[MG_COARSEST];  // the row of M that now is row r
  __shared__ int good;
  __shared__ double alpha_s;
  const int n = K.n, tx = threadIdx.x, r = threadIdx.y;
  if (n > MG_COARSEST || n < 1) {
    if (tx == 0 && r == 0) *ok = 0;
    return;
  }
  if (r == 0) {  // alpha from the warp of row-owners
    double ad = tx < n ? fabs(K.diag[tx]) : 0.0;
    for (int o = 16; o > 0; o >>= 1) ad += __shfl_xor_sync(0xffffffffu, ad, o);
    if (tx == 0) alpha_s = closed ? ad / ((double)n * (double)n) : 0.0;
    orig[tx] = tx;
    if (tx == 0) good = 1;
  }
  __syncthreads();
  if (r < n) {
    for (int c = tx; c < 2 * n; c += 32) M[r][c] = c < n ? alpha_s : (c - n == r ? 1.0 : 0.0);
    __syncwarp();
    const int m = K.cnt[r];  // distinct columns, none of them r
    if (tx == 31) M[r][r] += K.diag[r];
    if (tx < m) M[r][K.col[(size_t)tx * K.n + r]] += K.val[(size_t)tx * K.n + r];
  }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    auto column = [&]() { return tx < n - 1 - k ? k + 1 + tx : n + orig[tx - (n - 1 - k)]; };
    if (r == 0) {
      // argmax of |M[i][k]| over i >= k, ties to the lower row; ordered as the bits are
      long long v = -1;
      if (tx >= k && tx < n) {
        const double x = fabs(M[tx][k]);
        v = x == x ? __double_as_longlong(x) : 0;
      }
      int p = tx;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const long long v2 = __shfl_xor_sync(0xffffffffu, v, o);
        const int p2 = __shfl_xor_sync(0xffffffffu, p, o);
        if (v2 > v || (v2 == v && p2 < p)) { v = v2; p = p2; }
      }
      if (v <= 0) {
        if (tx == 0) good = 0;
      } else {
        if (p != k) {
          for (int c = tx; c < 2 * n; c += 32) { const double t = M[k][c]; M[k][c] = M[p][c]; M[p][c] = t; }
          if (tx == 0) { const int t = orig[k]; orig[k] = orig[p]; orig[p] = t; }
        }
        __syncwarp();
        if (tx < n) M[k][column()] /= M[k][k];
      }
    }
    __syncthreads();
    if (!good) break;
    if (r < n && r != k && tx < n) {
      const int c = column();
      M[r][c] = fma(-M[r][k], M[k][c], M[r][c]);
    }
    __syncthreads();
  }
  if (good && r < n)
    for (int c = tx; c < n; c += 32) inv[(size_t)r * n + c] = M[r][n + c];
  if (tx == 0 && r == 0) *ok = good;
}

// The row's A P g in direct form, vown g_own + sum_c (A P)_ic g_c, from its direction table:
// the eight neighbour cells' values and gathers are all issued at once, their addresses computed
// from the row's own cell (`own`, with g[own] = gc, vown = (A P) at the own cell); unused
// directions gather g[own] and add nothing.  The sum runs in the pair order of k_mg_rows (the
// 3x3 in key order, then the row's searched list).  Direct form, as the FP64 row product sums
// A_ik x_k: nine FMAs on the FP64 pipe (2 lanes per clock per SM here) where the difference
// form took seventeen operations.
__device__ __forceinline__ double ap_stencil(const double* __restrict__ rv9, const int* __restrict__ ragg,
                                             const double* __restrict__ rval, int rx, size_t i, size_t n,
                                             const double* g, int own, int ncx, double gc, double vown) {
  const unsigned used = ((unsigned)rx >> 16) & 0xffu;
  double v8[8], g8[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int q = k < 4 ? k : k + 1;
    const int off = (q / 3 - 1) * ncx + (q % 3 - 1);
    v8[k] = __ldg(rv9 + (size_t)k * n + i);
    g8[k] = g[(used >> k) & 1u ? own + off : own];
  }
  double ap = vown * gc;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if ((used >> k) & 1u) ap = fma(v8[k], g8[k], ap);
  const int t0 = rx & 0xff, m = (rx >> 8) & 0xff;
  for (int t = t0; t < m; ++t) {
    const size_t e = (size_t)t * n + i;
    ap = fma(__ldg(rval + e), g[__ldg(ragg + e)], ap);
  }
  return ap;
}

// ---------------------------------------------------------------- V-cycle
// the coarse levels, as the FP64 and the mixed V-cycle share them
struct MgCoarse {
  MgLevel lv[MG_MAX_LEVELS];  // finest first; a kernel parameter, so a phase does not wait for it
  int nl;              // number of coarse levels (>= 1)
  int tail;            // first level handled by block 0 alone
  const double* kinv;  // the coarsest level's dense inverse, if *kinv_ok
  const int* kinv_ok;
  float* g32;          // mixed precision: the level-1 solution rounded to FP32, else null
};

struct MgArgs {
  BiArgs b;                  // the unpreconditioned solver's arguments
  MgCoarse co;
  const int *agg, *cstart, *ccnt, *ip;  // fine aggregate (cell) of each row; cell lists
  double *z, *fr, *dinv0, *rsum;        // fine work vectors, 1/diag, row sums
  // A P by fine row (k_mg_rows): (cell, sum of the row's values in that cell) pairs, own cell
  // first, and the same by 3x3 direction with the packed word; A times the V-cycle's output
  const int *ragg, *rx;
  const double *rval, *rv9;
  int ncx;
  double* w;
};

// (A x)_c on a coarse level with x_c = xc: the diagonal, then the slots in order.  load(k)
// returns what x_k is formed from and value(load(k)) is x_k.  U slots' columns and values are
// loaded at once and then their operands, so a row waits for two round trips to memory per U
// slots, not two per slot (the grid-wide levels, whose operands come from other blocks; 4M FP64
// solve 31.4 -> 30.7 ms.  Eight slots of two operands each spill, so the upward phase takes four).
template <int U, class Load, class Value>
__device__ __forceinline__ double lv_row(const MgLevel& L, int c, double xc, Load load, Value value) {
  double y = __ldg(L.diag + c) * xc;
  const int m = __ldg(L.cnt + c);
  const int* cp = L.col + c;
  const double* vp = L.val + c;
  for (int t0 = 0; t0 < m; t0 += U) {
    int k[U];
    double v[U];
    decltype(load(0)) x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t e = (size_t)(t0 + u) * L.n;
      k[u] = t0 + u < m ? __ldg(cp + e) : c;
      v[u] = t0 + u < m ? __ldg(vp + e) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = load(k[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t0 + u < m) y = fma(v[u], value(x[u]), y);
  }
  return y;
}

// (A x)_c with x written by this block: its operands are in L1 mostly, and the plain loop has the
// fewest instructions (20k-particle mixed solve 2.01 -> 1.88 ms against the batched form)
__device__ __forceinline__ double lv_Ax(const MgLevel& L, const double* x, int c) {
  double y = __ldg(L.diag + c) * x[c];
  const int m = __ldg(L.cnt + c);
  for (int t = 0; t < m; ++t) y = fma(__ldg(L.val + (size_t)t * L.n + c), x[__ldg(L.col + (size_t)t * L.n + c)], y);
  return y;
}

__device__ __forceinline__ void lv_residual(const MgLevel& L, int i0, int st) {
  for (int c = i0; c < L.n; c += st) L.r[c] = L.b[c] - lv_Ax(L, L.x, c);
}

// restriction of F's residual into G's right-hand side, and G's first sweep from zero
__device__ __forceinline__ void lv_restrict(const MgLevel& F, const MgLevel& G, int i0, int st) {
  for (int C = i0; C < G.n; C += st) {
    const int X = C % G.gx, Y = C / G.gx;
    double b = 0.0;
    for (int q = 0; q < 4; ++q) {
      const int fx = 2 * X + (q & 1), fy = 2 * Y + (q >> 1);
      if (fx < F.gx && fy < F.gy) b += F.r[fx + fy * F.gx];
    }
    G.b[C] = b;
    G.x[C] = MG_OMEGA * __ldg(G.dinv + C) * b;
  }
}

__device__ __forceinline__ void lv_prolong(const MgLevel& F, const double* gsol, int ggx, int i0, int st) {
  for (int c = i0; c < F.n; c += st) {
    const int X = (c % F.gx) >> 1, Y = (c / F.gx) >> 1;
    F.x[c] = fma(MG_GAMMA, gsol[X + Y * ggx], F.x[c]);
  }
}

// one damped Jacobi sweep of x into r, and into x32 rounded to FP32 when given
__device__ __forceinline__ void lv_smooth(const MgLevel& L, int i0, int st, float* x32 = nullptr) {
  for (int c = i0; c < L.n; c += st) {
    const double v = fma(MG_OMEGA * __ldg(L.dinv + c), L.b[c] - lv_Ax(L, L.x, c), L.x[c]);
    L.r[c] = v;
    if (x32) x32[c] = narrow(v);
  }
}

// The grid-wide levels fuse each pair of phases, so a level costs one grid barrier on the way
// down and one on the way up; both give the same bits as the two phases in sequence.
//
// Down: F's residual and its restriction into G.  Four consecutive lanes take the four children
// of one coarse row; their residuals are summed by shuffles in child order, as lv_restrict sums
// F.r.  The loop bound is warp-uniform (the shuffles need every lane).
__device__ __forceinline__ void lv_residual_restrict(const MgLevel& F, const MgLevel& G, int i0, int st) {
  const int lane = threadIdx.x & 31;
  const int total = 4 * G.n;
  for (int t0 = i0 - lane; t0 < total; t0 += st) {
    const int t = t0 + lane;
    const int C = t >> 2, q = t & 3;
    double r = 0.0;
    int ok = 0;
    if (t < total) {
      const int X = C % G.gx, Y = C / G.gx;
      const int fx = 2 * X + (q & 1), fy = 2 * Y + (q >> 1);
      if (fx < F.gx && fy < F.gy) {
        const int f = fx + fy * F.gx;
        r = F.b[f] - lv_row<8>(F, f, F.x[f], [&](int k) { return F.x[k]; }, [](double v) { return v; });
        ok = 1;
      }
    }
    const double r1 = __shfl_down_sync(0xffffffffu, r, 1);
    const double r2 = __shfl_down_sync(0xffffffffu, r, 2);
    const double r3 = __shfl_down_sync(0xffffffffu, r, 3);
    const int okm = ok | (__shfl_down_sync(0xffffffffu, ok, 1) << 1) | (__shfl_down_sync(0xffffffffu, ok, 2) << 2) |
                    (__shfl_down_sync(0xffffffffu, ok, 3) << 3);
    if (q == 0 && t < total) {
      double b = 0.0;
      if (okm & 1) b += r;
      if (okm & 2) b += r1;
      if (okm & 4) b += r2;
      if (okm & 8) b += r3;
      G.b[C] = b;
      G.x[C] = MG_OMEGA * __ldg(G.dinv + C) * b;
    }
  }
}

// Up: prolongation of G's solution into F and F's smoothing sweep.  Each row forms the
// prolonged x of itself and of its columns from F.x and gsol (neither written in this phase) and
// writes the smoothed value into r (and x32 rounded to FP32 when given); F.x itself is left
// as it was, which nothing reads afterwards.
__device__ __forceinline__ void lv_prolong_smooth(const MgLevel& F, const double* gsol, int ggx, int i0, int st,
                                                  float* x32 = nullptr) {
  for (int c = i0; c < F.n; c += st) {
    auto load = [&](int k) {
      const int X = (k % F.gx) >> 1, Y = (k / F.gx) >> 1;
      return make_double2(gsol[X + Y * ggx], F.x[k]);
    };
    auto value = [](const double2& o) { return fma(MG_GAMMA, o.x, o.y); };
    const double xc = value(load(c));
    const double y = lv_row<4>(F, c, xc, load, value);
    const double v = fma(MG_OMEGA * __ldg(F.dinv + c), F.b[c] - y, xc);
    F.r[c] = v;
    if (x32) x32[c] = narrow(v);
  }
}

// MG_SWEEPS damped Jacobi sweeps of a level of at most 32 rows by one warp, a row a lane, with x, b
// and the row's first slots in registers: lv_smooth's sums without its loads and block barriers
// (where aggregates outside the domain leave the coarsest level without an inverse, its sweeps were
// about half of the one-block levels' 22 us a V-cycle; with the levels in the kernel's parameters and
// cell_sum, the 20k / 250k / 4M mixed solves went from 1.61 / 3.96 / 26.2 to 1.44 / 3.69 / 25.9 ms.
// All the one-block levels in registers and shared memory were slower: 1.57 / 4.03 / 28.4, as the
// call or the code around it costs the particle level's loops more registers).
constexpr int SWEEP_SLOTS = 8;
__device__ __forceinline__ void lv_sweeps(const MgLevel& L) {
  const int c = threadIdx.x & 31;
  const bool in = c < L.n;
  const int m = in ? __ldg(L.cnt + c) : 0;
  int k[SWEEP_SLOTS];
  double v[SWEEP_SLOTS];
#pragma unroll
  for (int u = 0; u < SWEEP_SLOTS; ++u) {
    k[u] = u < m ? __ldg(L.col + u * L.n + c) : c;
    v[u] = u < m ? __ldg(L.val + u * L.n + c) : 0.0;
  }
  double x = 0.0, b = 0.0, dg = 0.0, od = 0.0;
  if (in) {
    x = L.x[c];
    b = L.b[c];
    dg = __ldg(L.diag + c);
    od = MG_OMEGA * __ldg(L.dinv + c);
  }
  const int most = __reduce_max_sync(0xffffffffu, m);
#pragma unroll 1
  for (int sw = 0; sw < MG_SWEEPS; ++sw) {
    double o[SWEEP_SLOTS], y = dg * x;
#pragma unroll
    for (int u = 0; u < SWEEP_SLOTS; ++u) o[u] = __shfl_sync(0xffffffffu, x, k[u]);
#pragma unroll
    for (int u = 0; u < SWEEP_SLOTS; ++u) {
      if (u >= most) break;
      if (u < m) y = fma(v[u], o[u], y);
    }
#pragma unroll 1
    for (int u = SWEEP_SLOTS; u < most; ++u) {
      const double xo = __shfl_sync(0xffffffffu, x, u < m ? __ldg(L.col + u * L.n + c) : c);
      if (u < m) y = fma(__ldg(L.val + u * L.n + c), xo, y);
    }
    x = fma(od, b - y, x);
  }
  if (in) L.x[c] = x;
}

// the solution of level l after the upward pass: post-smoothed into r, or x on the coarsest
__device__ __forceinline__ const double* lv_sol(const MgCoarse& a, int l) {
  return l == a.nl - 1 ? a.lv[l].x : a.lv[l].r;
}

// sum of a cell's entries of r in cell-list order (mirrors, n and up, follow the particles); the
// loads of eight are in flight together
template <class T>
__device__ __forceinline__ T cell_sum(const int* __restrict__ ip, int ne, int n, const T* r) {
  T b = 0;
#pragma unroll 1
  for (int k0 = 0; k0 < ne; k0 += 8) {
    int i[8];
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) i[u] = k0 + u < ne ? __ldg(ip + k0 + u) : n;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = i[u] < n ? r[i[u]] : T(0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (i[u] >= n) return b;
      b += v[u];
    }
  }
  return b;
}

// levels tail..nl-1 by block 0 alone
__device__ __forceinline__ void mg_block_levels(const MgCoarse& a) {
  const int i0 = threadIdx.x, st = blockDim.x;
  for (int l = a.tail; l + 1 < a.nl; ++l) {
    const MgLevel F = a.lv[l], G = a.lv[l + 1];
    lv_residual(F, i0, st);
    __syncthreads();
    lv_restrict(F, G, i0, st);
    __syncthreads();
  }
  const MgLevel K = a.lv[a.nl - 1];
  if (a.kinv_ok && *a.kinv_ok) {  // direct solve with the dense inverse
    for (int r = i0; r < K.n; r += st) {
      double v = 0.0;
      for (int c = 0; c < K.n; ++c) v = fma(__ldg(a.kinv + (size_t)r * K.n + c), K.b[c], v);
      K.x[r] = v;
    }
    __syncthreads();
  } else if (K.n <= 32) {
    if (i0 < 32) lv_sweeps(K);
    __syncthreads();
  } else {
    for (int sw = 0; sw < MG_SWEEPS; ++sw) {
      lv_smooth(K, i0, st);
      __syncthreads();
      for (int c = i0; c < K.n; c += st) K.x[c] = K.r[c];
      __syncthreads();
    }
  }
  if (a.g32 && a.nl == 1) {  // level 1 is the coarsest
    for (int c = i0; c < K.n; c += st) a.g32[c] = narrow(K.x[c]);
    __syncthreads();
  }
  for (int l = a.nl - 2; l >= a.tail; --l) {
    const MgLevel F = a.lv[l];
    lv_prolong(F, lv_sol(a, l + 1), a.lv[l + 1].gx, i0, st);
    __syncthreads();
    lv_smooth(F, i0, st, l == 0 ? a.g32 : nullptr);
    __syncthreads();
  }
}

// out = M^-1 q by one V-cycle; the last loop also sums this thread's rows of out into `sum`.
// q needs only its own rows complete (the calling thread wrote them).
// q -= qshift first (the closed domain's mean removal), stored back.  As in the solvers, the
// vector passes load each row's operands one row ahead (rows_ahead).
__device__ bool mg_vcycle(const MgArgs& a, double* q, double qshift, double* out, double& sum, int tid,
                          int stride) {
  const int n = a.b.n;
  Scal* s = a.b.sc;
  double* z = a.z;
  rows_ahead(
      tid, stride, n, [&](int i) { return make_double2(q[i], a.dinv0[i]); },
      [&](int i, const double2& o) {
        const double qi = o.x - qshift;
        q[i] = qi;
        z[i] = MG_OMEGA * o.y * qi;
      });
  if (!grid_sync(s)) return false;
  for (int i = tid; i < n; i += stride) a.fr[i] = q[i] - spmv_row(a.b, z, i);
  if (!grid_sync(s)) return false;
  {  // restriction to the cells (level 1)
    const MgLevel L1 = a.co.lv[0];
    for (int cc = tid; cc < L1.n; cc += stride) {
      const int s0 = __ldg(a.cstart + cc), ne = __ldg(a.ccnt + cc);
      const double b = cell_sum(a.ip + s0, ne, n, a.fr);
      L1.b[cc] = b;
      L1.x[cc] = MG_OMEGA * __ldg(L1.dinv + cc) * b;
    }
  }
  if (!grid_sync(s)) return false;
  const MgCoarse& co = a.co;
  for (int l = 0; l < co.tail; ++l) {
    lv_residual_restrict(co.lv[l], co.lv[l + 1], tid, stride);
    if (!grid_sync(s)) return false;
  }
  if (blockIdx.x == 0) mg_block_levels(co);
  if (!grid_sync(s)) return false;
  for (int l = co.tail - 1; l >= 0; --l) {
    lv_prolong_smooth(co.lv[l], lv_sol(co, l + 1), co.lv[l + 1].gx, tid, stride);
    if (!grid_sync(s)) return false;
  }
  // prolongation to the particles (the particle level is pre-smoothed only), and
  // w = A out = A z + gamma (A P) g1 with A z = q - fr from the fine residual and (A P) g1 in
  // direct form over the row's cells (ap_stencil).
  // Software-pipelined: a row's streamed operands are loaded one pass ahead, together with the
  // gathers of the row before, so each pass waits for one round trip to memory, not two.
  const double* g1 = lv_sol(co, 0);
  double acc = 0.0;
  struct Row {
    int c, rx;
    double z, q, fr, vown;
  };
  auto load_row = [&](int i) {
    Row r;
    r.c = __ldg(a.agg + i);
    r.rx = __ldg(a.rx + i);
    r.z = z[i];
    r.q = q[i];
    r.fr = a.fr[i];
    r.vown = __ldg(a.rval + i);  // slot 0: the row's own cell
    return r;
  };
  Row cur{};
  if (tid < n) cur = load_row(tid);
  for (int i = tid; i < n; i += stride) {
    const Row r = cur;
    if (i + stride < n) cur = load_row(i + stride);
    double o = r.z;
    double w = r.q - r.fr;
    if (r.c >= 0) {
      const double gc = g1[r.c];
      o = fma(MG_GAMMA, gc, o);
      w = fma(MG_GAMMA, ap_stencil(a.rv9, a.ragg, a.rval, r.rx, i, n, g1, r.c, a.ncx, gc, r.vown), w);
    }
    out[i] = o;
    a.w[i] = w;
    acc += o;
  }
  sum = acc;
  return true;
}

// ---------------------------------------------------------------- preconditioned BiCGSTAB
template <bool NONULL>
__global__ void __launch_bounds__(TPB, 4) k_bicgstab_mg(const __grid_constant__ MgArgs m) {
  __shared__ SolverSh sh;
  const BiArgs& a = m.b;
  const int n = a.n;
  const int nb = gridDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int stride = gridDim.x * blockDim.x;
  Scal* s = a.sc;
  if (state_failed(s)) return;
  solver_begin(sh);
  const bool use_mg = *((volatile int*)&s->mg_fail) == 0;
  double* part = a.part;
  const double rinv1 = 1.0 / (1.0 + 1.0e-15);
  const double small = NONULL ? 1.0e-6 : 4.0;  // open solver: the integer expression 10-6
  double acc = 0.0;
  // out = M^-1 (q - qshift) with q -= qshift stored back (q: own rows complete), and this
  // thread's part of sum(out)
  auto precond = [&](double* q, double qshift, double* out, double& sum) -> bool {
    if (use_mg) return mg_vcycle(m, q, qshift, out, sum, tid, stride);
    sum = 0.0;
    for (int i = tid; i < n; i += stride) {
      const double qi = q[i] - qshift;
      q[i] = qi;
      const double o = NONULL ? qi * rinv1 : qi * a.rinvM[i];
      out[i] = o;
      sum += o;
    }
    return true;
  };
  for (int i = tid; i < n; i += stride) {  // 1/diag and row sums of the fine matrix
    const double dg = __ldg(a.diag + i);
    double rs = dg;
    const int cnt = __ldg(a.cnt + i);
    for (int k = 0; k < cnt; ++k) rs += __ldg(a.val + (size_t)k * a.stride + i);
    m.dinv0[i] = dg != 0.0 ? 1.0 / dg : 0.0;
    m.rsum[i] = rs;
    if (!NONULL) a.rinvM[i] = 1.0 / (dg + 1.0e-15);
  }
  if (a.warm) {  // x0 = P of the previous step
    for (int i = tid; i < n; i += stride) {
      double xi = a.P[i];
      a.x[i] = xi;
      a.pinv[i] = xi;
    }
    if (!grid_sync(s)) return;
  }
  for (int i = tid; i < n; i += stride) {
    double bi = a.B[i];
    if (a.warm) bi = bi - spmv_row(a, a.pinv, i);
    else a.x[i] = 0.0;
    a.r[i] = bi;
    a.rb[i] = bi;
    a.v[i] = 0.0;
    a.p[i] = 0.0;
    acc = fma(bi, bi, acc);
  }
  if (!grid_reduce<1>(s, acc, 0.0, part + 10 * (size_t)nb, sh, [&](double* v, int&) { sh.rho = v[0]; })) return;
  const double dn = (double)n;
  bool at_s = false;  // the solve stopped on s, not on r
  int iter = 1, warn = 0;
  bool done = false;
  while (iter <= a.itermax) {
    if (is_zero(sh.rho)) { warn |= VEBI_WARN_BICGSTAB_BREAKDOWN; done = true; break; }
    const double beta = sh.beta, omega0 = sh.omega;
    acc = 0.0;
    // the vector passes load each row's operands one row ahead (rows_ahead)
    rows_ahead(
        tid, stride, n, [&](int i) { return make_double3(a.r[i], a.v[i], a.p[i]); },
        [&](int i, const double3& o) {
          const double ni = (iter == 1) ? o.x : fma(beta, fma(-omega0, o.y, o.z), o.x);
          a.p[i] = ni;
          acc += ni;
        });
    double mean = 0.0;
    if (NONULL) {
      if (!grid_reduce<1>(s, acc, 0.0, part, sh, [=](double* v, int&) { v[0] = v[0] / dn; })) return;
      mean = sh.v[0];
    }
    // p_hat = M^-1 (p - mean), made mean-free (closed domains) through mp
    if (!precond(a.p, mean, a.pinv, acc)) return;
    if (!grid_reduce<1>(s, acc, 0.0, part + 1 * (size_t)nb, sh,
                        [=](double* v, int&) { v[0] = NONULL ? v[0] / dn : 0.0; }))
      return;
    const double mp = sh.v[0];
    // v = A (p_hat - mp) ; (r_bar, v)
    acc = 0.0;
    if (use_mg) {
      rows_ahead(
          tid, stride, n, [&](int i) { return make_double3(m.w[i], m.rsum[i], a.rb[i]); },
          [&](int i, const double3& o) {
            const double vi = fma(-mp, o.y, o.x);
            a.v[i] = vi;
            acc = fma(o.z, vi, acc);
          });
    } else {
      for (int i = tid; i < n; i += stride) {
        double vi = fma(-mp, m.rsum[i], spmv_row(a, a.pinv, i));
        a.v[i] = vi;
        acc = fma(a.rb[i], vi, acc);
      }
    }
    if (!grid_reduce<1>(s, acc, 0.0, part + 2 * (size_t)nb, sh,
                        [&](double* v, int&) { sh.alpha = sh.rho / (v[0] + 1.0e-15); }))
      return;
    const double alpha = sh.alpha;
    double a2 = 0.0;
    acc = 0.0;
    rows_ahead(
        tid, stride, n, [&](int i) { return make_double2(a.v[i], a.r[i]); },
        [&](int i, const double2& o) {
          const double si = fma(-alpha, o.x, o.y);
          a.s[i] = si;
          acc = fma(si, si, acc);
          a2 += si;
        });
    // |s|^2 against the first one (1 when small), and the mean of s
    if (!grid_reduce<2>(s, acc, a2, part + 4 * (size_t)nb, sh, [&](double* v, int& flag) {
          sh.n2 = v[0];
          if (iter == 1) sh.n2s0 = (v[0] <= small) ? 1.0 : v[0];
          flag = v[0] <= a.tol * a.tol * sh.n2s0;
          v[1] = v[1] / dn;
        }))
      return;
    const double mean_s = sh.v[1];
    if (sh.flag) {
      for (int i = tid; i < n; i += stride) a.x[i] = fma(alpha, a.pinv[i] - mp, a.x[i]);
      at_s = true;
      done = true;
      break;
    }
    if (!precond(a.s, NONULL ? mean_s : 0.0, a.sinv, acc)) return;
    if (!grid_reduce<1>(s, acc, 0.0, part + 3 * (size_t)nb, sh,
                        [=](double* v, int&) { v[0] = NONULL ? v[0] / dn : 0.0; }))
      return;
    const double ms = sh.v[0];
    // t = A (s_hat - ms) ; (t, s) ; |t|^2
    acc = 0.0;
    a2 = 0.0;
    if (use_mg) {
      rows_ahead(
          tid, stride, n, [&](int i) { return make_double3(m.w[i], m.rsum[i], a.s[i]); },
          [&](int i, const double3& o) {
            const double ti = fma(-ms, o.y, o.x);
            a.t[i] = ti;
            acc = fma(ti, o.z, acc);
            a2 = fma(ti, ti, a2);
          });
    } else {
      for (int i = tid; i < n; i += stride) {
        double ti = fma(-ms, m.rsum[i], spmv_row(a, a.sinv, i));
        a.t[i] = ti;
        acc = fma(ti, a.s[i], acc);
        a2 = fma(ti, ti, a2);
      }
    }
    if (!grid_reduce<2>(s, acc, a2, part + 6 * (size_t)nb, sh, [&](double* v, int&) {
          sh.omega = v[0] / (v[1] + 1.0e-15);
          v[2] = fma(sh.alpha, mp, sh.omega * ms);  // the two mean shifts of x folded into one
        }))
      return;
    const double alpha1 = sh.alpha, omega = sh.omega;
    acc = 0.0;
    a2 = 0.0;
    // x += alpha (p_hat - mp) + omega (s_hat - ms)
    const double xshift = sh.v[2];
    struct XRow {
      double s, p, x, t, sv, rb;
    };
    rows_ahead(
        tid, stride, n, [&](int i) { return XRow{a.sinv[i], a.pinv[i], a.x[i], a.t[i], a.s[i], a.rb[i]}; },
        [&](int i, const XRow& o) {
          a.x[i] = fma(omega, o.s, fma(alpha1, o.p, o.x - xshift));
          const double ri = fma(-omega, o.t, o.sv);
          a.r[i] = ri;
          acc = fma(ri, ri, acc);
          a2 = fma(o.rb, ri, a2);
        });
    // |r|^2 against the first one (1 when small), the new rho and the next iteration's beta
    if (!grid_reduce<2>(s, acc, a2, part + 8 * (size_t)nb, sh, [&](double* v, int& flag) {
          sh.n2 = v[0];
          if (iter == 1) sh.n2r0 = (v[0] <= small) ? 1.0 : v[0];
          flag = v[0] <= a.tol * a.tol * sh.n2r0;
          sh.beta = v[1] / (sh.rho + 1.0e-15) * sh.alpha / (sh.omega + 1.0e-15);
          sh.rho = v[1];
        }))
      return;
    if (sh.flag) { done = true; break; }
    iter = iter + 1;
  }
  if (!done) warn |= VEBI_WARN_MAXITER;
  for (int i = tid; i < n; i += stride) a.P[i] = a.x[i];
  if (tid == 0) {
    s->ls_iters = iter;
    s->ls_iters_total += iter;
    s->ls_residual = sqrt(sh.n2 / (at_s ? sh.n2s0 : sh.n2r0));
    atomicOr(&s->warnings, warn);
  }
}

// ---------------------------------------------------------------- mixed precision
// The mixed-precision solver (FP64 recurrences, FP32 difference-form SpMV) with the same
// V-cycle, whose particle level runs in FP32: the smoothing vector and the fine residual are
// FP32 and the fine products use the FP32 values in difference form.  The coarse levels are the
// FP64 ones of the FP64 solver.  The preconditioner need not be exact: its rounding changes the
// iteration count, not the residual test the solve stops on.
struct MgMxArgs {
  MxArgs b;
  MgCoarse co;
  const int *agg, *cstart, *ccnt, *ip;
  float *z, *fr, *dinv0;
  const int *ragg, *rx;  // A P by fine row, as in MgArgs, with FP32 direction values
  const double* rval;
  const float* rv9;
  int ncx;
  float* w;                // A times the V-cycle's output, FP32
  float* rs32;             // the row sums rounded to FP32
  float* q32;              // the V-cycle's input (after mean removal) rounded to FP32
  const double* diag;      // the PPE matrix's FP64 diagonal
};

// sum_k A_ik (z_col - z_i) + rowsum_i z_i in FP32 (one FP32 vector; rs32 = FP32 row sums)
__device__ __forceinline__ float spmv_diff32s(const MxArgs& a, const float* rs32, const float* z, int i) {
  const int cnt = __ldg(a.cnt + i);
  const float* vp = a.val32 + i;
  const int* cp = a.col + i;
  const long long st = a.stride;
  const float zi = __ldca(z + i);
  float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
  int k = 0;
  for (; k + 3 < cnt; k += 4) {
    const int c0 = __ldg(cp), c1 = __ldg(cp + st), c2 = __ldg(cp + 2 * st), c3 = __ldg(cp + 3 * st);
    const float v0 = __ldg(vp), v1 = __ldg(vp + st), v2 = __ldg(vp + 2 * st), v3 = __ldg(vp + 3 * st);
    b0 = fmaf(v0, __ldca(z + c0) - zi, b0);
    b1 = fmaf(v1, __ldca(z + c1) - zi, b1);
    b2 = fmaf(v2, __ldca(z + c2) - zi, b2);
    b3 = fmaf(v3, __ldca(z + c3) - zi, b3);
    cp += 4 * st;
    vp += 4 * st;
  }
  for (; k < cnt; ++k) {
    b0 = fmaf(__ldg(vp), __ldca(z + __ldg(cp)) - zi, b0);
    cp += st;
    vp += st;
  }
  return fmaf(rs32[i], zi, (b0 + b1) + (b2 + b3));
}

// The row's A P g1 in FP32: rowsum_i g_own + sum_c (A P)_ic (g_c - g_own) from the FP32 direction
// table and the FP32 level-1 solution g, in the pair order of k_mg_rows; the searched list (rare:
// periodic partners, mirror parents outside the 3x3) from the FP64 pairs rounded to FP32.
__device__ __forceinline__ float ap_stencil32(const float* __restrict__ rv9, const int* __restrict__ ragg,
                                              const double* __restrict__ rval, int rx, size_t i, size_t n,
                                              const float* g, int own, int ncx, float gc, float rs) {
  const unsigned used = ((unsigned)rx >> 16) & 0xffu;
  float v8[8], g8[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int q = k < 4 ? k : k + 1;
    const int off = (q / 3 - 1) * ncx + (q % 3 - 1);
    v8[k] = __ldg(rv9 + (size_t)k * n + i);
    g8[k] = g[(used >> k) & 1u ? own + off : own];
  }
  float ap = rs * gc;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if ((used >> k) & 1u) ap = fmaf(v8[k], g8[k] - gc, ap);
  const int t0 = rx & 0xff, m = (rx >> 8) & 0xff;
  for (int t = t0; t < m; ++t) {
    const size_t e = (size_t)t * n + i;
    ap = fmaf((float)__ldg(rval + e), g[__ldg(ragg + e)] - gc, ap);
  }
  return ap;
}

// out = M^-1 q in FP64 (the preconditioned direction), and this thread's part of sum(out).
// The vector passes load each row's operands one row ahead (rows_ahead), so a pass's loads are
// in flight before the previous row's stores: the compiler cannot move a load above a store
// to another array it may alias.
__device__ bool mg_vcycle_mixed(const MgMxArgs& a, double* q, double qshift, double* out, double& sum, int tid,
                                int stride) {
  const int n = a.b.n;
  Scal* s = a.b.sc;
  float* z = a.z;
  // q -= qshift (the closed domain's mean removal), its FP32 rounding q32, and z = omega D^-1 q
  float* q32 = a.q32;
  struct QRow {
    double q;
    float d;
  };
  rows_ahead(
      tid, stride, n, [&](int i) { return QRow{q[i], a.dinv0[i]}; },
      [&](int i, const QRow& o) {
        const double qi = o.q - qshift;
        const float fi = narrow(qi);
        q[i] = qi;
        q32[i] = fi;
        z[i] = (float)MG_OMEGA * o.d * fi;
      });
  if (!grid_sync(s)) return false;
  for (int i = tid; i < n; i += stride) a.fr[i] = q32[i] - spmv_diff32s(a.b, a.rs32, z, i);
  if (!grid_sync(s)) return false;
  {
    const MgLevel L1 = a.co.lv[0];
    for (int cc = tid; cc < L1.n; cc += stride) {
      const int s0 = __ldg(a.cstart + cc), ne = __ldg(a.ccnt + cc);
      const double b = widen(cell_sum(a.ip + s0, ne, n, a.fr));  // in FP32, as fr is
      L1.b[cc] = b;
      L1.x[cc] = MG_OMEGA * __ldg(L1.dinv + cc) * b;
    }
  }
  if (!grid_sync(s)) return false;
  const MgCoarse& co = a.co;
  for (int l = 0; l < co.tail; ++l) {
    lv_residual_restrict(co.lv[l], co.lv[l + 1], tid, stride);
    if (!grid_sync(s)) return false;
  }
  if (blockIdx.x == 0) mg_block_levels(co);
  if (!grid_sync(s)) return false;
  for (int l = co.tail - 1; l >= 0; --l) {
    lv_prolong_smooth(co.lv[l], lv_sol(co, l + 1), co.lv[l + 1].gx, tid, stride, l == 0 ? co.g32 : nullptr);
    if (!grid_sync(s)) return false;
  }
  // prolongation to the particles (pre-smoothed only) from the FP32 level-1 solution g, and
  // w = A out, both in FP32 (the precision of this solver's products): A z = q32 - fr, plus
  // gamma (A P) g in difference form with the FP32 row sums.  The output is stored as FP64 and
  // summed in FP64 (the mean removal).  This GPU issues FP64 at 1/64 of the FP32 rate, so the
  // pass keeps to FP32 arithmetic; streamed operands are loaded one pass ahead of the gathers.
  const float* g32 = co.g32;
  const float gam = (float)MG_GAMMA;
  double acc = 0.0;
  struct Row {
    int c, rx;
    float z, fr, rs, q;
  };
  auto load_row = [&](int i) {
    Row r;
    r.c = __ldg(a.agg + i);
    r.rx = __ldg(a.rx + i);
    r.z = z[i];
    r.fr = a.fr[i];
    r.rs = a.rs32[i];
    r.q = q32[i];
    return r;
  };
  Row cur{};
  if (tid < n) cur = load_row(tid);
  for (int i = tid; i < n; i += stride) {
    const Row r = cur;
    if (i + stride < n) cur = load_row(i + stride);
    float oi = r.z;
    float wi = r.q - r.fr;
    if (r.c >= 0) {
      const float gc = g32[r.c];
      oi = fmaf(gam, gc, oi);
      wi = fmaf(gam, ap_stencil32(a.rv9, a.ragg, a.rval, r.rx, i, n, g32, r.c, a.ncx, gc, r.rs), wi);
    }
    const double od = widen(oi);
    out[i] = od;
    a.w[i] = wi;
    acc += od;
  }
  sum = acc;
  return true;
}

// Blocks per SM the mixed kernel is compiled for: its register budget is 65536 / (TPB x this)
#ifndef VEBI_MIXED_MG_BLOCKS_PER_SM
#define VEBI_MIXED_MG_BLOCKS_PER_SM 4
#endif

template <bool NONULL>
__global__ void __launch_bounds__(TPB, VEBI_MIXED_MG_BLOCKS_PER_SM) k_bicgstab_mixed_mg(const __grid_constant__ MgMxArgs m) {
  __shared__ SolverSh sh;
  const MxArgs& a = m.b;
  const int n = a.n;
  const int nb = gridDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int stride = gridDim.x * blockDim.x;
  Scal* s = a.sc;
  if (state_failed(s)) return;
  solver_begin(sh);
  const bool use_mg = *((volatile int*)&s->mg_fail) == 0;
  double* part = a.part;
  const double rinv1 = 1.0 / (1.0 + 1.0e-15);
  const double small = NONULL ? 1.0e-6 : 4.0;
  double acc = 0.0;
  // out = M^-1 (q - qshift), with q -= qshift stored back; this thread's part of sum(out)
  // With the multigrid the preconditioned directions are FP64 (pi, si read as double: same
  // size as the (hi, lo) pairs the unpreconditioned products gather)
  double* const pd = reinterpret_cast<double*>(a.pi);
  double* const sd = reinterpret_cast<double*>(a.si);
  auto precond = [&](double* q, double qshift, float2* out, double& sum) -> bool {
    if (use_mg) return mg_vcycle_mixed(m, q, qshift, reinterpret_cast<double*>(out), sum, tid, stride);
    sum = 0.0;
    for (int i = tid; i < n; i += stride) {
      const double qi = q[i] - qshift;
      q[i] = qi;
      const double o = NONULL ? qi * rinv1 : qi * a.rinvM[i];
      out[i] = split2(o);
      sum += o;
    }
    return true;
  };
  for (int i = tid; i < n; i += stride) {
    // the particle level's Jacobi sweep, in FP32: 1/diag of the assembled matrix
    const float dg = narrow(__ldg(m.diag + i));
    m.dinv0[i] = dg != 0.f ? 1.0f / dg : 0.f;
    m.rs32[i] = narrow(__ldg(a.rs + i));
  }
  if (a.warm) {
    for (int i = tid; i < n; i += stride) {
      double xi = a.P[i];
      a.x[i] = xi;
      a.pi[i] = split2(xi);
    }
    if (!grid_sync(s)) return;
  }
  for (int i = tid; i < n; i += stride) {
    double bi = a.B[i];
    if (a.warm) bi = bi - spmv_diff32(a, a.pi, i);
    else a.x[i] = 0.0;
    a.r[i] = bi;
    a.rb[i] = bi;
    a.v[i] = 0.0;
    a.p[i] = 0.0;
    acc = fma(bi, bi, acc);
  }
  if (!grid_reduce<1>(s, acc, 0.0, part + 10 * (size_t)nb, sh, [&](double* v, int&) { sh.rho = v[0]; })) return;
  const double dn = (double)n;
  bool at_s = false;  // the solve stopped on s, not on r
  int iter = 1, warn = 0;
  bool done = false;
  while (iter <= a.itermax) {
    if (is_zero(sh.rho)) { warn |= VEBI_WARN_BICGSTAB_BREAKDOWN; done = true; break; }
    const double beta = sh.beta, omega0 = sh.omega;
    acc = 0.0;
    // The vector passes load each row's operands one row ahead (rows_ahead)
    rows_ahead(
        tid, stride, n, [&](int i) { return make_double3(a.r[i], a.v[i], a.p[i]); },
        [&](int i, const double3& o) {
          const double ni = (iter == 1) ? o.x : fma(beta, fma(-omega0, o.y, o.z), o.x);
          a.p[i] = ni;
          acc += ni;
        });
    double mean = 0.0;
    if (NONULL) {
      if (!grid_reduce<1>(s, acc, 0.0, part, sh, [=](double* v, int&) { v[0] = v[0] / dn; })) return;
      mean = sh.v[0];
    }
    if (!precond(a.p, mean, a.pi, acc)) return;
    if (!grid_reduce<1>(s, acc, 0.0, part + 1 * (size_t)nb, sh,
                        [=](double* v, int&) { v[0] = NONULL ? v[0] / dn : 0.0; }))
      return;
    const double mp = sh.v[0];
    acc = 0.0;
    if (use_mg) {
      rows_ahead(
          tid, stride, n, [&](int i) { return make_double3(widen(m.w[i]), __ldg(a.rs + i), a.rb[i]); },
          [&](int i, const double3& o) {
            const double vi = fma(-mp, o.y, o.x);
            a.v[i] = vi;
            acc = fma(o.z, vi, acc);
          });
    } else {
      for (int i = tid; i < n; i += stride) {
        double vi = fma(-mp, __ldg(a.rs + i), spmv_diff32(a, a.pi, i));
        a.v[i] = vi;
        acc = fma(a.rb[i], vi, acc);
      }
    }
    if (!grid_reduce<1>(s, acc, 0.0, part + 2 * (size_t)nb, sh,
                        [&](double* v, int&) { sh.alpha = sh.rho / (v[0] + 1.0e-15); }))
      return;
    const double alpha = sh.alpha;
    double a2 = 0.0;
    acc = 0.0;
    rows_ahead(
        tid, stride, n, [&](int i) { return make_double2(a.v[i], a.r[i]); },
        [&](int i, const double2& o) {
          const double si = fma(-alpha, o.x, o.y);
          a.s[i] = si;
          acc = fma(si, si, acc);
          a2 += si;
        });
    // |s|^2 against the first one (1 when small), and the mean of s
    if (!grid_reduce<2>(s, acc, a2, part + 4 * (size_t)nb, sh, [&](double* v, int& flag) {
          sh.n2 = v[0];
          if (iter == 1) sh.n2s0 = (v[0] <= small) ? 1.0 : v[0];
          flag = v[0] <= a.tol * a.tol * sh.n2s0;
          v[1] = v[1] / dn;
        }))
      return;
    const double mean_s = sh.v[1];
    if (sh.flag) {
      for (int i = tid; i < n; i += stride)
        a.x[i] = fma(alpha, (use_mg ? pd[i] : join2(a.pi[i])) - mp, a.x[i]);
      at_s = true;
      done = true;
      break;
    }
    if (!precond(a.s, NONULL ? mean_s : 0.0, a.si, acc)) return;
    if (!grid_reduce<1>(s, acc, 0.0, part + 3 * (size_t)nb, sh,
                        [=](double* v, int&) { v[0] = NONULL ? v[0] / dn : 0.0; }))
      return;
    const double ms = sh.v[0];
    acc = 0.0;
    a2 = 0.0;
    if (use_mg) {
      rows_ahead(
          tid, stride, n, [&](int i) { return make_double3(widen(m.w[i]), __ldg(a.rs + i), a.s[i]); },
          [&](int i, const double3& o) {
            const double ti = fma(-ms, o.y, o.x);
            a.t[i] = ti;
            acc = fma(ti, o.z, acc);
            a2 = fma(ti, ti, a2);
          });
    } else {
      for (int i = tid; i < n; i += stride) {
        double ti = fma(-ms, __ldg(a.rs + i), spmv_diff32(a, a.si, i));
        a.t[i] = ti;
        acc = fma(ti, a.s[i], acc);
        a2 = fma(ti, ti, a2);
      }
    }
    if (!grid_reduce<2>(s, acc, a2, part + 6 * (size_t)nb, sh, [&](double* v, int&) {
          sh.omega = v[0] / (v[1] + 1.0e-15);
          v[2] = fma(sh.alpha, mp, sh.omega * ms);  // the two mean shifts of x folded into one
        }))
      return;
    const double alpha1 = sh.alpha, omega = sh.omega;
    acc = 0.0;
    a2 = 0.0;
    // x += alpha (p_hat - mp) + omega (s_hat - ms)
    const double xshift = sh.v[2];
    struct XRow {
      double p, s, x, t, sv, rb;
    };
    auto xr_update = [&](int i, const XRow& o) {
      a.x[i] = fma(omega, o.s, fma(alpha1, o.p, o.x - xshift));
      const double ri = fma(-omega, o.t, o.sv);
      a.r[i] = ri;
      acc = fma(ri, ri, acc);
      a2 = fma(o.rb, ri, a2);
    };
    // the preconditioned directions: FP64 with the multigrid, else (hi, lo) pairs
    if (use_mg) {
      rows_ahead(
          tid, stride, n, [&](int i) { return XRow{pd[i], sd[i], a.x[i], a.t[i], a.s[i], a.rb[i]}; }, xr_update);
    } else {
      rows_ahead(
          tid, stride, n,
          [&](int i) { return XRow{join2(a.pi[i]), join2(a.si[i]), a.x[i], a.t[i], a.s[i], a.rb[i]}; }, xr_update);
    }
    // |r|^2 against the first one (1 when small), the new rho and the next iteration's beta
    if (!grid_reduce<2>(s, acc, a2, part + 8 * (size_t)nb, sh, [&](double* v, int& flag) {
          sh.n2 = v[0];
          if (iter == 1) sh.n2r0 = (v[0] <= small) ? 1.0 : v[0];
          flag = v[0] <= a.tol * a.tol * sh.n2r0;
          sh.beta = v[1] / (sh.rho + 1.0e-15) * sh.alpha / (sh.omega + 1.0e-15);
          sh.rho = v[1];
        }))
      return;
    if (sh.flag) { done = true; break; }
    iter = iter + 1;
  }
  if (!done) warn |= VEBI_WARN_MAXITER;
  for (int i = tid; i < n; i += stride) a.P[i] = a.x[i];
  if (tid == 0) {
    s->ls_iters = iter;
    s->ls_iters_total += iter;
    s->ls_residual = sqrt(sh.n2 / (at_s ? sh.n2s0 : sh.n2r0));
    atomicOr(&s->warnings, warn);
  }
}

// ---------------------------------------------------------------- host side
// co-resident blocks of the FP64 (mixed = false) or the mixed multigrid solver
int ppe_mg_blocks(int nsm, bool mixed) {
  int per = 1 << 20;
  int o[2] = {0, 0};
  if (mixed) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[0], k_bicgstab_mixed_mg<true>, TPB, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[1], k_bicgstab_mixed_mg<false>, TPB, 0);
  } else {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[0], k_bicgstab_mg<true>, TPB, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[1], k_bicgstab_mg<false>, TPB, 0);
  }
  for (int q = 0; q < 2; ++q) per = o[q] < per ? o[q] : per;
  if (per < 1) per = 1;
  return per * nsm;
}

// coarse level sizes for a gx x gy cell grid: halve until at most MG_COARSEST aggregates
std::vector<int> mg_level_dims(int gx, int gy) {
  std::vector<int> dims;
  for (int l = 0; l < MG_MAX_LEVELS; ++l) {
    dims.push_back(gx);
    dims.push_back(gy);
    if ((long long)gx * gy <= MG_COARSEST || (gx <= 1 && gy <= 1)) break;
    gx = (gx + 1) / 2;
    gy = (gy + 1) / 2;
  }
  return dims;
}

// the coarse matrices of this step, and the first level small enough for one block
static int mg_setup(Ctx& x) {
  const Consts& c = x.c;
  const int nl = (int)x.mg.size();
  const float* v32 = x.precision == VEBI_PREC_MIXED ? x.d.ppe_val32 : nullptr;
  VEBI_LAUNCH(x, k_mg_rows, grid_for(c.npfb), TPB, c, x.d, v32, x.mg_ragg, x.mg_rval, x.mg_rcnt, x.mg_rv9,
              x.mg_rx);
  // A warp per row until the GPU is full of them.  Measured, a thread / a warp per row: level 1 of
  // 1.8k / 22k / 90k / 360k rows 128 / 137 / 139 / 400 and 19 / 58 / 196 / 743 us; a coarser level of
  // 500 / 22k / 90k rows 34 / 33 / 42 and 11 / 31 / 101 us.
  const auto level1 = x.mg[0].n <= 65536 ? k_mg_level1_warp : k_mg_level1;
  VEBI_LAUNCH(x, level1, grid_for(level1 == k_mg_level1_warp ? 32ll * x.mg[0].n : x.mg[0].n), TPB, c, x.d, x.mg[0],
              x.mg_ragg, x.mg_rval, x.mg_rcnt);
  for (int l = 0; l + 1 < nl; ++l) {
    const auto coarsen = x.mg[l + 1].n <= 16384 ? k_mg_coarsen_warp : k_mg_coarsen;
    VEBI_LAUNCH(x, coarsen, grid_for(coarsen == k_mg_coarsen_warp ? 32ll * x.mg[l + 1].n : x.mg[l + 1].n), TPB, x.mg[l],
                x.mg[l + 1], x.d.s);
  }
  VEBI_LAUNCH(x, k_mg_coarse_inverse, 1, dim3(32, 32), x.mg[nl - 1], x.mg_kinv, x.mg_kinv_ok,
              c.open_domain == 0 ? 1 : 0);
  int tail = nl - 1;
  for (int l = 0; l < nl; ++l)
    if (x.mg[l].n <= x.mg_block_rows) { tail = l; break; }
  return tail;
}

static MgCoarse coarse_args(const Ctx& x, int tail, float* g32) {
  MgCoarse co{};
  co.nl = (int)x.mg.size();
  for (int l = 0; l < co.nl; ++l) co.lv[l] = x.mg[l];
  co.tail = tail;
  co.kinv = x.mg_kinv;
  co.kinv_ok = x.mg_kinv_ok;
  co.g32 = g32;
  return co;
}

void launch_ppe_mg_mixed(Ctx& x) {
  const Consts& c = x.c;
  const Dev& d = x.d;
  const int tail = mg_setup(x);
  int nblk = x.mg_blocks_mixed;
  const long long rows_per_block = (long long)TPB * (x.solver_rows_per_thread > 0 ? x.solver_rows_per_thread : 1);
  long long need = (c.npfb + rows_per_block - 1) / rows_per_block;
  if (need < nblk) nblk = (int)(need < 1 ? 1 : need);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk);
  cfg.blockDim = dim3(TPB);
  cfg.stream = x.st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MgMxArgs m{MxArgs{d.bx, d.br, d.brb, d.bv, d.bp, d.bs, d.bt, d.bM, d.partials, d.p, d.pi2, d.si2, d.ppe_B,
                    d.rowsum, d.ppe_val32, d.ppe_col, d.ij_count, d.s, (long long)c.npfb, c.npfb, c.itermax, c.tol,
                    c.warm_start},
             coarse_args(x, tail, x.mg_g32), d.cellpart, d.cell_start, d.cell_cnt, d.ip, (float*)x.mg_z, (float*)x.mg_fr,
             (float*)x.mg_dinv0, x.mg_ragg, x.mg_rx, x.mg_rval, (const float*)x.mg_rv9, c.ncx,
             (float*)x.mg_w, (float*)x.mg_rsum, x.mg_q32, d.ppe_diag};
  if (c.open_domain == 0) cudaLaunchKernelEx(&cfg, k_bicgstab_mixed_mg<true>, m);
  else cudaLaunchKernelEx(&cfg, k_bicgstab_mixed_mg<false>, m);
  x.launches++;
}

void launch_ppe_mg(Ctx& x) {
  const Consts& c = x.c;
  const Dev& d = x.d;
  const int tail = mg_setup(x);
  int nblk = x.mg_blocks;
  const long long rows_per_block = (long long)TPB * (x.solver_rows_per_thread > 0 ? x.solver_rows_per_thread : 1);
  long long need = (c.npfb + rows_per_block - 1) / rows_per_block;
  if (need < nblk) nblk = (int)(need < 1 ? 1 : need);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk);
  cfg.blockDim = dim3(TPB);
  cfg.stream = x.st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MgArgs m{BiArgs{d.bx, d.br, d.brb, d.bv, d.bp, d.bpi, d.bs, d.bsi, d.bt, d.bM, d.partials, d.p, d.ppe_B,
                  d.ppe_diag, d.ppe_val, d.ppe_col, d.ij_count, d.s, (long long)c.npfb, c.npfb, c.itermax, c.tol,
                  c.warm_start},
           coarse_args(x, tail, nullptr), d.cellpart, d.cell_start, d.cell_cnt, d.ip, x.mg_z, x.mg_fr, x.mg_dinv0,
           x.mg_rsum, x.mg_ragg, x.mg_rx, x.mg_rval, x.mg_rv9, c.ncx, x.mg_w};
  if (c.open_domain == 0) cudaLaunchKernelEx(&cfg, k_bicgstab_mg<true>, m);
  else cudaLaunchKernelEx(&cfg, k_bicgstab_mg<false>, m);
  x.launches++;
}

}  // namespace vebi

#ifdef VEBI_BARRIER_TIMESTAMPS
// diagnostic build only: the multigrid solvers' barrier timestamps (see vebi_solver.cuh)
extern "C" int vebi_barrier_timestamps_reset(void) {
  unsigned int z = 0;
  static unsigned int zb[vebi::BAR_ALL_BLOCKS];
  cudaError_t e = cudaMemcpyToSymbol(vebi::g_bar_blk_n, zb, sizeof(zb));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(vebi::g_bar_n, &z, sizeof(z));
  return (int)e;
}
// every block's arrival at BAR_ALL_N barriers from BAR_ALL_FIRST on ([q][block]), and its SM
extern "C" int vebi_barrier_arrivals_read(unsigned long long* arr, unsigned int* smid) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess)
    e = cudaMemcpyFromSymbol(arr, vebi::g_bar_all, sizeof(unsigned long long) * vebi::BAR_ALL_N * vebi::BAR_ALL_BLOCKS);
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(smid, vebi::g_bar_smid, sizeof(unsigned int) * vebi::BAR_ALL_BLOCKS);
  return (int)e;
}
extern "C" int vebi_barrier_timestamps_read(unsigned long long* ts, unsigned int* n) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(n, vebi::g_bar_n, sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(ts, vebi::g_bar_ts, sizeof(unsigned long long) * 2 * vebi::BAR_TS_MAX);
  return (int)e;
}
#endif
