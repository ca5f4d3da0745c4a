// vebi_sph.cu -- per-pair SPH operators and per-particle updates of the step.
//
//  kernel_calculation (weights, Bonet-Lok kgcm)   kernel_calculation.F90:2-75
//  locate_free_surf_part, calc_part_dist_vars,
//  smooth_normals (open domain)                   freesurf_mod.F90:17-137
//  new_fick_shift + shifting_forces               new_fick_shift.F90:15-92,117-210
//  grad_operator (u, v, theta in one pass)        gradient_calculation.F90:50-94
//  constitutive_eqn_evolve, calc_eigens,
//  f_strain_*, f_relaxation_integrate             predictor_mod.F90:141-331
//  prediction_step pair loop and updates          predictor_mod.F90:27-139
//  calc_pressure_gradient + velocity update +
//  final advection                                gradient_calculation.F90:16-48, div_free.F90:94-117
//  secondary_properties                           div_free.F90:148-192
//
// One thread per particle walks that particle's ELL row k = 0..ij_count-1 in the reference's
// order with the reference's association, so every per-particle sum is the reference's sum.
#include "vebi_ctx.cuh"
#include "vebi_lanes.cuh"

namespace vebi {

#define ELL(k, i) ((size_t)(k) * c.npfb + (i))

// ------------------------------------------------- kernel_calculation and new_fick_shift's sums
// The weights of a pair and the factor 0.25 (Wab(r/h) / Wab1)^4 of its shifting force
// (kernel_calculation.F90:22-71, new_fick_shift.F90:135-148, where the reference calls pow with
// the exponent 4.0), each operation as the reference writes it and rounds it.  Its products, quotients
// and root run beside the FP64 pipe (vebi_fp64.cuh): 25 FP64 instructions are left of 170.
struct PairTerms {
  double w1, w2, wl, fab;
};
__device__ __forceinline__ double power4(double x) {
  const double x2 = fp::mul_int(x, x);
  return fp::mul_int(x2, x2);
}
__device__ __forceinline__ double power5(double x) {
  const double x2 = fp::mul_int(x, x);
  return fp::mul_int(x2, fp::mul_int(x, x2));
}
// the spline's classes, compared as integers (qq >= 0)
__device__ __forceinline__ bool below(double qq, int k) { return fp::hi(qq) < fp::hi((double)k); }

// Wab (sphtools.F90:46-76) of qq = rad / h
__device__ __forceinline__ double spline(const Consts& c, double qq) {
  using fp::mul_int;
  double w = 0.0;
  if (below(qq, 3)) {
    w = power5(3.0 - qq);
    if (below(qq, 2)) w = w - mul_int(6.0, power5(2.0 - qq));
    if (below(qq, 1)) w = w + mul_int(15.0, power5(1.0 - qq));
    w = mul_int(c.ad_7, w);
  }
  return w;
}
// of a pair's offset
__device__ __forceinline__ double pair_spline(const Consts& c, double r1, double r2) {
  using namespace fp;
  double y;
  const double rad = root(mul_int(r1, r1) + mul_int(r2, r2), y);
  return spline(c, is_zero(rad) ? rad : quotient_near(rad, c.h, c.oneoverh, mul_int(rad, c.oneoverh)));
}

__device__ __forceinline__ PairTerms pair_terms(const Consts& c, double r1, double r2) {
  using namespace fp;
  PairTerms o;
  const double rr2 = mul_int(r1, r1) + mul_int(r2, r2);
  double y;
  const double rad = root(rr2, y);
  const double qq = mul_int(rad, c.oneoverh);
  double f = 0.0;
  if (below(qq, 3)) {  // fac (sphtools.F90:11-44)
    f = mul_int(-5.0, power4(3.0 - qq));
    if (below(qq, 2)) f = f + mul_int(30.0, power4(2.0 - qq));
    if (below(qq, 1)) f = f - mul_int(75.0, power4(1.0 - qq));
    f = mul_int(c.ad_7h, f);
  }
  double m = rad;
  if (!(__double_as_longlong(rad) > __double_as_longlong(c.eta2))) {  // particles (almost) on one another
    m = fmax(rad, c.eta2);
    y = divided(1.0, m);
  }
  const double a1 = mul_int(r1, f), a2 = mul_int(r2, f);
  // aligned particles: 0 / m is the zero itself
  const double g1 = is_zero(a1) ? a1 : quotient_near(a1, m, y, a1 * y);
  const double g2 = is_zero(a2) ? a2 : quotient_near(a2, m, y, a2 * y);
  o.w1 = mul_int(g1, c.dv);
  o.w2 = mul_int(g2, c.dv);
  const double den = rr2 + c.eta_small;
  const double num = mul_int(2.0, mul_int(r1, o.w1) + mul_int(r2, o.w2));
  const double yd = reciprocal(den);
  o.wl = quotient_near(num, den, yd, num * yd);
  const double w = spline(c, quotient_near(rad, c.h, c.oneoverh, qq));  // rad / h
  const double wn = is_zero(w) ? w : quotient_near(w, c.wab1, c.inv_wab1, mul_int(w, c.inv_wab1));
  o.fab = mul_int(0.25, power4(wn));
  return o;
}

// the slot of particle i in row j, or -1
__device__ __forceinline__ int slot_of(const Consts& c, const Dev& d, int j, int i) {
  const int cnt = d.ij_count[j];
  for (int k0 = 0; k0 < cnt; k0 += 8) {
    int l[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) l[u] = k0 + u < cnt ? d.ij_link[ELL(k0 + u, j)] : -1;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (l[u] == i) return k0 + u;
  }
  return -1;
}

// -x, a zero as it is (a pair's x - x is +0 from both sides); on the integer pipe
__device__ __forceinline__ double negated(double x) {
  int h;
  asm("xor.b32 %0, %1, 0x80000000;" : "=r"(h) : "r"(fp::hi(x)));
  return is_zero(x) ? x : fp::pack(h, fp::lo(x));
}

// The pairs' terms.  A pair's terms serve both its particles -- r_ij and w_ij change sign, wL and
// the shifting factor do not, bit for bit -- so each pair is computed once, by the particle of
// lower index (or the one that has a mirror for a neighbour), and stored in both rows; the search
// of the partner's row for the slot waits in the shadow of the arithmetic.  A pair that one
// particle alone lists (d.s->one_sided) is computed by that one.  Each lane first lists the slots
// it computes, so that all lanes of a warp compute in every round.  P lanes share a row when the
// rows alone would not fill the GPU.
// What bounds it: the issue of ~1000 integer and FP32 instructions a pair, with the FP64 pipe at 40%.
// Measured with k_weight_sums at 4M / 250k / 20k / 1.7k particles: 12.6 / 1.08 / 0.15 / 0.08 ms, where
// a kernel each for the weights and the shifting, all pairs from both sides in FP64 instructions,
// took 43.9 / 3.21 / 0.64 / 0.58.
constexpr int PAIR_SLOTS = 96;  // nplink's limit
constexpr int PAIR_TPB = 64;    // small blocks: a 20k-particle step has few of them per SM to balance

template <int P>
__global__ void __launch_bounds__(PAIR_TPB) k_pair_terms(Consts c, Dev d, double* __restrict__ fab) {
  __shared__ unsigned char list[PAIR_SLOTS / P][PAIR_TPB];
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / P;
  if (i >= c.npfb) return;
  const int cnt = d.ij_count[i];
  const bool one_sided = d.s->one_sided != 0;
  int m = 0;
#pragma unroll 4
  for (int k = tid % P; k < cnt; k += P) {
    const int j = d.ij_link[ELL(k, i)];
    if (j > i || (one_sided && slot_of(c, d, j, i) < 0)) list[m++][threadIdx.x] = (unsigned char)k;
  }
  const double xi = d.rx[i], yi = d.ry[i];
#pragma unroll 1
  for (int e = 0; e < m; ++e) {
    const size_t o = ELL(list[e][threadIdx.x], i);
    const int j = d.ij_link[o];
    const int kj = j < c.npfb ? slot_of(c, d, j, i) : -1;
    const PairTerms t = pair_terms(c, xi - d.rx[j], yi - d.ry[j]);
    d.wGx[o] = t.w1;
    d.wGy[o] = t.w2;
    d.wL[o] = t.wl;
    fab[o] = t.fab;
    if (kj >= 0) {
      const size_t q = ELL(kj, j);
      d.wGx[q] = negated(t.w1);
      d.wGy[q] = negated(t.w2);
      d.wL[q] = t.wl;
      fab[q] = t.fab;
    }
  }
}

// Shifting displacement from the concentration gradient (new_fick_shift.F90:47-92) and the shifting
// velocity; solid boundary particles get -u (div_free.F90:65-78).  The uncommon cases are calls:
// inlined, the compiler computes their divisions, roots and exponential for every particle.
static __device__ __noinline__ double speed_coefficient(const Consts& c, const Dev& d, int i, double dt) {
  double maxU = bits_to_double(d.s->maxU_bits);
  double absU = sqrt(d.ux[i] * d.ux[i] + d.uy[i] * d.uy[i]);
  double temp = (double)0.2f * exp(-absU / ((double)0.2f * maxU));
  return 4.0 * c.h * dt * (absU + temp * maxU);
}
static __device__ __noinline__ double2 along_surface(const Dev& d, int i, double D, double gx, double gy) {
  double temp = sqrt(d.surf_nx[i] * d.surf_nx[i] + d.surf_ny[i] * d.surf_ny[i]);
  double sn1 = d.surf_nx[i] / fmax(temp, (double)1e-8f);
  double sn2 = d.surf_ny[i] / fmax(temp, (double)1e-8f);
  double st1 = -sn2, st2 = sn1;
  double dCds = st1 * gx + st2 * gy;
  return make_double2(-D * dCds * st1, -D * dCds * st2);
}
__device__ __forceinline__ void shift_velocity(const Consts& c, const Dev& d, int i, double gx, double gy) {
  if (i < c.nbS) {
    d.ushx[i] = -d.ux[i];
    d.ushy[i] = -d.uy[i];
    return;
  }
  const double dt = d.s->dt;
  const double D = c.shift_coeff == 1 ? speed_coefficient(c, d, i, dt) : 0.25 * c.h * c.h;
  double2 s;
  if (c.open_domain == 1 && d.n_surf[i] == 1) s = along_surface(d, i, D, gx, gy);
  else s = make_double2(-D * gx, -D * gy);
  const double s2 = s.x * s.x + s.y * s.y;
  double y;
  const double temp = is_zero(s2) ? s2 : fp::root(s2, y);
  if (temp > 0.1 * c.h) {
    s.x = fp::divided(0.1 * c.h * s.x, temp);
    s.y = fp::divided(0.1 * c.h * s.y, temp);
  }
  y = fp::reciprocal(dt);
  d.ushx[i] = is_zero(s.x) ? s.x : fp::quotient_near(s.x, dt, y, s.x * y);
  d.ushy[i] = is_zero(s.y) ? s.y : fp::quotient_near(s.y, dt, y, s.y * y);
}

// The sums over each row in slot order: the Bonet-Lok matrix and the concentration gradient of the
// shifting; in a closed domain the shifting velocity too.  What bounds it is the FP64 pipe, ten
// instructions a pair (16 with its products, 5.8 ms at 4M; 3.7 without).  P = 4 splits a row's eight
// sums over four lanes, two each.
template <int P>
__global__ void __launch_bounds__(TPB, 4) k_weight_sums(const __grid_constant__ Consts c, const __grid_constant__ Dev d,
                                                     const double* __restrict__ fab) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / P, p = tid % P;
  const bool in = i < c.npfb;
  const int cnt = in ? d.ij_count[i] : 0;
  double k11 = 0.0, k12 = 0.0, k21 = 0.0, k22 = 0.0, f1 = 0.0, f2 = 0.0, t1 = 0.0, t2 = 0.0;
  if (P == 1) {
    const double xi = in ? d.rx[i] : 0.0, yi = in ? d.ry[i] : 0.0;
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
      const size_t o = ELL(k, i);
      const int j = d.ij_link[o];
      const double w1 = d.wGx[o], w2 = d.wGy[o], fb = fab[o];
      const double r1 = xi - d.rx[j], r2 = yi - d.ry[j];
      k11 = k11 - fp::mul_int(w1, r1);  // dv * g1 * r1
      k12 = k12 - fp::mul_int(w2, r1);
      k21 = k21 - fp::mul_int(w1, r2);
      k22 = k22 - fp::mul_int(w2, r2);
      f1 = f1 + w1;
      f2 = f2 + w2;
      t1 = t1 + fp::mul_int(w1, fb);
      t2 = t2 + fp::mul_int(w2, fb);
    }
  } else {
    // lane 0: k11, f1; 1: k12, f2; 2: k21, t1; 3: k22, t2
    const double* wp = (p & 1) ? d.wGy : d.wGx;
    const double* xp = p < 2 ? d.rx : d.ry;
    const double x0 = in ? xp[i] : 0.0;
    double ks = 0.0, fs = 0.0;
#pragma unroll 4
    for (int k = 0; k < cnt; ++k) {
      const size_t o = ELL(k, i);
      const double w = wp[o], r = x0 - xp[d.ij_link[o]];
      ks = ks - w * r;
      fs = fs + w * (p < 2 ? 1.0 : fab[o]);
    }
    const unsigned full = 0xffffffffu;
    k11 = ks;
    k12 = __shfl_down_sync(full, ks, 1);
    k21 = __shfl_down_sync(full, ks, 2);
    k22 = __shfl_down_sync(full, ks, 3);
    f1 = fs;
    f2 = __shfl_down_sync(full, fs, 1);
    t1 = __shfl_down_sync(full, fs, 2);
    t2 = __shfl_down_sync(full, fs, 3);
  }
  if (!in || p) return;
  double temp = 1.0 / ((k11 * k22 - k12 * k21) + 1.0e-15);
  d.kgcm[0][i] = temp * k22;
  d.kgcm[2][i] = -temp * k12;
  d.kgcm[1][i] = -temp * k21;
  d.kgcm[3][i] = temp * k11;
  const double gx = f1 + t1, gy = f2 + t2;
  d.gradCx[i] = gx;
  d.gradCy[i] = gy;
  if (c.open_domain == 0) shift_velocity(c, d, i, gx, gy);
}

// open domain: after the free-surface particles and their normals are known
__global__ void k_shift_open(const __grid_constant__ Consts c, const __grid_constant__ Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.npfb) shift_velocity(c, d, i, d.gradCx[i], d.gradCy[i]);
}

// ---------------------------------------------------------------------- free surface (open)
// Both kernels' pairs are evaluated beside the FP64 pipe and, on small domains, by eight lanes a row
// (vebi_lanes.cuh).  The weights' stage with them, in FP64 instructions by a thread a row / now: 2.9k
// particles (free surface, 75 columns) 0.40 / 0.10 ms, 45k 0.89 / 0.49; dam break 3.8k 0.49 / 0.13.
template <int P>
__global__ void __launch_bounds__(P == 1 ? TPB : LANES_TPB) k_part_dist_vars(Consts c, Dev d) {
  bool in;
  const int i = lane_row<P>(c.npfb, in);
  if (P == 1 && !in) return;
  const double xi = d.rx[i], yi = d.ry[i];
  double ct = 0, dr = 0, s1 = 0, s2 = 0;
  const int cnt = in ? d.ij_count[i] : 0;
  auto pair = [&](int k, auto put) {
    const int j = d.ij_link[ELL(k, i)];
    const double r1 = xi - d.rx[j], r2 = yi - d.ry[j];
    const double w1 = d.wGx[ELL(k, i)], w2 = d.wGy[ELL(k, i)];
    put(0, pair_spline(c, r1, r2));
    put(1, fp::mul_int(r1, w1) + fp::mul_int(r2, w2));
    put(2, w1);
    put(3, w2);
  };
  if constexpr (P == 1) {
#pragma unroll 1
    for (int k = 0; k < cnt; ++k)
      pair(k, [&](int e, double v) {
        if (e == 0) ct = ct + v;
        if (e == 1) dr = dr - v;
        if (e == 2) s1 = s1 - v;
        if (e == 3) s2 = s2 - v;
      });
  } else {
    double s[4];
    pair_sums64<4, 1>(
        cnt, [&](int k, double* t) { pair(k, [&](int e, double v) { t[e] = e ? -v : v; }); }, s);
    if (!in || (threadIdx.x & (P - 1))) return;
    ct = s[0], dr = s[1], s1 = s[2], s2 = s[3];
  }
  double w0 = wab(c, 0.0);
  double conc = ct * c.dv;
  conc = conc + c.dv * w0;
  d.conc[i] = conc;
  d.div_r[i] = dr;
  d.surf_nx[i] = s1 * c.h;
  d.surf_ny[i] = s2 * c.h;
  double bdr = 1.4 + 0.5 * fmax(conc - 1.0, -0.2);
  d.beta_div_r[i] = bdr;
  d.n_surf[i] = (dr > bdr) ? 0 : 1;
}

__global__ void k_nsurf_mirrors(Consts c, Dev d) {
  const int nm = d.s->nmirror;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < nm; m += gridDim.x * blockDim.x) {
    int j = c.npfb + m;
    d.n_surf[j] = d.n_surf[d.irel[j]];
  }
}

// smooth_normals (Shepard filter) + ppe_smooth; the filtered normals go to the shifting velocity's
// arrays first and are copied back after (the reference uses a temporary array too)
template <int P>
__global__ void __launch_bounds__(P == 1 ? TPB : LANES_TPB) k_smooth_normals(Consts c, Dev d) {
  bool in;
  const int i = lane_row<P>(c.npfb, in);
  if (P == 1 && !in) return;
  const double xi = d.rx[i], yi = d.ry[i];
  double a = 0, b = 0;
  const int cnt = in ? d.ij_count[i] : 0;
  auto pair = [&](int k, auto put) {
    const int j = d.ij_link[ELL(k, i)];
    if (j >= c.npfb) return;
    const double w = pair_spline(c, xi - d.rx[j], yi - d.ry[j]);
    put(0, fp::mul_int(w, d.surf_nx[j]));
    put(1, fp::mul_int(w, d.surf_ny[j]));
  };
  if constexpr (P == 1) {
#pragma unroll 1
    for (int k = 0; k < cnt; ++k)
      pair(k, [&](int e, double v) {
        if (e == 0) a = a + v;
        else b = b + v;
      });
  } else {
    double s[2];
    pair_sums64<2, 1>(
        cnt,
        [&](int k, double* t) {
          t[0] = t[1] = 0.0;
          pair(k, [&](int e, double v) { t[e] = v; });
        },
        s);
    if (!in || (threadIdx.x & (P - 1))) return;
    a = s[0], b = s[1];
  }
  double w0 = wab(c, 0.0);
  d.ushx[i] = a * c.dv + d.surf_nx[i] * w0 * c.dv;
  d.ushy[i] = b * c.dv + d.surf_ny[i] * w0 * c.dv;
  double ps = 1.0;
  double dr = d.div_r[i], bdr = d.beta_div_r[i];
  if (!(dr > 1.2 * bdr)) {
    if (d.n_surf[i] == 1) ps = 0.0;
    else ps = 0.5 * (1.0 - cos((dr - bdr) * PI / (0.2 * bdr)));
  }
  d.ppe_smooth[i] = ps;
}

__global__ void k_copy_normals(Consts c, Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.npfb) return;
  d.surf_nx[i] = d.ushx[i];
  d.surf_ny[i] = d.ushy[i];
}

// ---------------------------------------------------------------------- gradients
// The products of a pair run on the integer pipe (vebi_fp64.cuh), beside the FP64 pipe that bounds
// these kernels on large domains; on small ones they cost nothing either.  4M particles, without /
// with: gradients 5.28 / 3.24 ms, predictor 10.97 / 5.81 ms (7.31 with two blocks per SM: 82
// registers leave too few warps to cover the gathers), right-hand side 3.9 / 1.9 ms.
template <int P>
__global__ void __launch_bounds__(P == 1 ? TPB : LANES_TPB, P == 1 ? 4 : 1) k_gradients(Consts c, Dev d) {
  using fp::mul_int;
  bool in;
  const int i = lane_row<P>(c.npfb, in);
  if (P == 1 && !in) return;
  const double ui = d.ux[i], vi = d.uy[i], ti = d.th[i];
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0, a5 = 0;
  const int cnt = in ? d.ij_count[i] : 0;
  auto pair = [&](int k, auto put) {
    const int j = d.ij_link[ELL(k, i)];
    const double w1 = d.wGx[ELL(k, i)], w2 = d.wGy[ELL(k, i)];
    const double du = d.ux[j] - ui, dvv = d.uy[j] - vi, dth = d.th[j] - ti;
    put(0, mul_int(du, w1));
    put(1, mul_int(du, w2));
    put(2, mul_int(dvv, w1));
    put(3, mul_int(dvv, w2));
    put(4, mul_int(dth, w1));
    put(5, mul_int(dth, w2));
  };
  if constexpr (P == 1) {
    for (int k = 0; k < cnt; ++k)
      pair(k, [&](int e, double v) {
        if (e == 0) a0 = a0 + v;
        if (e == 1) a1 = a1 + v;
        if (e == 2) a2 = a2 + v;
        if (e == 3) a3 = a3 + v;
        if (e == 4) a4 = a4 + v;
        if (e == 5) a5 = a5 + v;
      });
  } else {
    double a[6];
    pair_sums64<6, 1>(
        cnt, [&](int k, double* t) { pair(k, [&](int e, double v) { t[e] = v; }); }, a);
    if (!in || (threadIdx.x & (P - 1))) return;
    a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3], a4 = a[4], a5 = a[5];
  }
  const double K11 = d.kgcm[0][i], K21 = d.kgcm[1][i], K12 = d.kgcm[2][i], K22 = d.kgcm[3][i];
  d.grad[0][i] = K11 * a0 + K12 * a1;
  d.grad[1][i] = K21 * a0 + K22 * a1;
  d.grad[2][i] = K11 * a2 + K12 * a3;
  d.grad[3][i] = K21 * a2 + K22 * a3;
  d.grad[4][i] = K11 * a4 + K12 * a5;
  d.grad[5][i] = K21 * a4 + K22 * a5;
}

// ---------------------------------------------------------------------- log-conformation
// What bounds it: the FP64 pipe, ~190 instructions a particle, of which two logarithms and two
// exponentials are 98.  Its ~110 products, five quotients and four roots run beside the pipe
// (vebi_fp64.cuh; all on it, it was 398 instructions and 2.98 ms at 4M, 1.59 now).
struct M2 { double a11, a12, a21, a22; };
// a call: twelve products inlined are 140 KB of code, more than the instruction cache
static __device__ __noinline__ M2 mm(M2 A, M2 B) {
  using fp::mul_int;
  return M2{mul_int(A.a11, B.a11) + mul_int(A.a12, B.a21), mul_int(A.a11, B.a12) + mul_int(A.a12, B.a22),
            mul_int(A.a21, B.a11) + mul_int(A.a22, B.a21), mul_int(A.a21, B.a12) + mul_int(A.a22, B.a22)};
}
__device__ __forceinline__ M2 tr(const M2& A) { return M2{A.a11, A.a21, A.a12, A.a22}; }

// calc_eigens (predictor_mod.F90:253-290): closed-form symmetric 2x2 eigen-decomposition
__device__ __forceinline__ void calc_eigens(const M2& A, double& L1, double& L2, M2& R) {
  using namespace fp;
  double trc = A.a11 + A.a22;
  double det = mul_int(A.a11, A.a22) - mul_int(A.a21, A.a12);
  double tmp = mul_int(mul_int(0.25, trc), trc) - det;
  // tmp <= epsilon(1d0), compared as integers (a NaN stays)
  const long long bits = __double_as_longlong(tmp);
  if (bits <= 0x3cb0000000000000ll && (bits & 0x7fffffffffffffffll) <= 0x7ff0000000000000ll) tmp = 0.0;
  double y;
  const double rt = is_zero(tmp) ? 0.0 : root(tmp, y), half = mul_int(0.5, trc);
  L1 = half + rt;
  L2 = half - rt;
  if (!is_zero(A.a21)) {
    double r11 = L1 - A.a22, r21 = A.a21;
    double nrm = root(mul_int(r11, r11) + mul_int(r21, r21), y);
    r11 = quotient(r11, nrm, y);
    r21 = quotient(r21, nrm, y);
    R = M2{r11, -r21, r21, r11};
  } else {
    L1 = A.a11;
    L2 = A.a22;
    R = M2{1.0, 0.0, 0.0, 1.0};
  }
}
// the relaxation factor exp(-(alpha_R dt / Wi)); alpha_R = 1 is the step's own (k_mirror_corners)
static __device__ __noinline__ double relaxation(double alpha_R, double dt, double Wi) {
  return exp(-(alpha_R * 1.0 * dt / Wi));
}

__global__ void k_logconf(Consts c, Dev d) {
  using fp::mul_int;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.npfb) return;
  const double dt = d.s->dt;
  // steps 1-2: A = f_strain_backward(tau) = (tau/1 + I)/1
  M2 A{d.tau[0][i] / 1.0 + 1.0, d.tau[2][i] / 1.0 + 0.0, d.tau[1][i] / 1.0 + 0.0, d.tau[3][i] / 1.0 + 1.0};
  A = M2{A.a11 / 1.0, A.a12 / 1.0, A.a21 / 1.0, A.a22 / 1.0};
  double L1, L2;
  M2 R;
  calc_eigens(A, L1, L2, R);
  const double gap = L2 - L1;
  {  // diagnostic: particles within reach of the 1/(L2 - L1 + 1e-10) pole of step 5
    const unsigned am = __activemask();
    const unsigned near = __ballot_sync(am, __double_as_longlong(fp::magnitude(gap)) < __double_as_longlong(1.0e-7));
    if ((threadIdx.x & 31) == __ffs(am) - 1 && near) {
      atomicAdd(&d.s->n_near_pole, __popc(near));
      atomicAdd(&d.s->n_near_pole_total, __popc(near));
    }
  }
  // step 3: Psi = R log(Lambda) R^T
  M2 D{log(L1), 0.0, 0.0, log(L2)};
  M2 Psi0 = mm(R, mm(D, tr(R)));
  // step 5: B and Omega from R^T grad(u) R
  M2 G{d.grad[0][i], d.grad[1][i], d.grad[2][i], d.grad[3][i]};
  M2 tm = mm(tr(R), mm(G, R));
  const double den = gap + 1e-10;
  double tmp1 = fp::quotient(mul_int(L2, tm.a12) + mul_int(L1, tm.a21), den, fp::reciprocal(fp::magnitude(den)));
  tm.a12 = 0.0;
  tm.a21 = 0.0;
  M2 B = mm(R, mm(tm, tr(R)));
  M2 W{0.0, tmp1, -tmp1, 0.0};
  M2 Om = mm(R, mm(W, tr(R)));
  // step 6: Psi += dt (2B + Omega Psi - Psi Omega)
  M2 OP = mm(Om, Psi0), PO = mm(Psi0, Om);
  M2 t6{mul_int(2.0, B.a11) + OP.a11 - PO.a11, mul_int(2.0, B.a12) + OP.a12 - PO.a12,
        mul_int(2.0, B.a21) + OP.a21 - PO.a21, mul_int(2.0, B.a22) + OP.a22 - PO.a22};
  M2 Psi{Psi0.a11 + mul_int(dt, t6.a11), Psi0.a12 + mul_int(dt, t6.a12), Psi0.a21 + mul_int(dt, t6.a21),
         Psi0.a22 + mul_int(dt, t6.a22)};
  // step 7: A = R exp(Lambda) R^T
  calc_eigens(Psi, L1, L2, R);
  L1 = exp(L1);
  L2 = exp(L2);
  M2 E2{L1, 0.0, 0.0, L2};
  A = mm(R, mm(E2, tr(R)));
  // step 8: analytic PTT relaxation with the previous trace
  double alpha_R = 1.0 + mul_int(c.eps_ptt, d.trace_conf[i] - 2.0);
  double e1 = __double_as_longlong(alpha_R) == __double_as_longlong(1.0) ? d.s->relax : relaxation(alpha_R, dt, c.Wi);
  double e2 = (1.0 - e1) / 1.0;
  const double z = mul_int(e2, 0.0);
  A = M2{mul_int(A.a11, e1) + e2 * 1.0, mul_int(A.a12, e1) + z, mul_int(A.a21, e1) + z, mul_int(A.a22, e1) + e2 * 1.0};
  // step 9
  double trc = A.a11 + A.a22;
  d.trace_conf[i] = trc;
  d.a_out[i] = trc;
  d.tau[0][i] = 1.0 * (1.0 * A.a11 - 1.0);
  d.tau[2][i] = 1.0 * (1.0 * A.a12 - 0.0);
  d.tau[1][i] = 1.0 * (1.0 * A.a21 - 0.0);
  d.tau[3][i] = 1.0 * (1.0 * A.a22 - 1.0);
}

// ---------------------------------------------------------------------- predictor
// rhs pair loop + buoyancy; u*, theta* written to the second buffers (walls copied)
template <int P>
__global__ void __launch_bounds__(P == 1 ? TPB : LANES_TPB, P == 1 ? 4 : 1) k_predictor(Consts c, Dev d) {
  using fp::mul_int;
  bool in;
  const int i = lane_row<P>(c.npfb, in);
  if (P == 1 && !in) return;
  const double ui = d.ux[i], vi = d.uy[i], ti = d.th[i];
  const double K11 = d.kgcm[0][i], K21 = d.kgcm[1][i], K12 = d.kgcm[2][i], K22 = d.kgcm[3][i];
  double Ti11 = 0, Ti21 = 0, Ti12 = 0, Ti22 = 0;
  const bool ve = c.const_mod != 1;
  if (ve) { Ti11 = d.tau[0][i]; Ti21 = d.tau[1][i]; Ti12 = d.tau[2][i]; Ti22 = d.tau[3][i]; }
  const double cs = c.coeff_solvent, cp = c.coeff_polymeric, ct = c.coeff_theta;
  double s1 = 0, s2 = 0, st = 0;
  const int cnt = in ? d.ij_count[i] : 0;
  // terms 0 and 1 of u, the polymeric and the solvent one, 2 and 3 of v, 5 of theta
  auto pair = [&](int k, auto put) {
    const int j = d.ij_link[ELL(k, i)];
    const double u1 = ui - d.ux[j], u2 = vi - d.uy[j];
    const double wl = d.wL[ELL(k, i)];
    if (ve) {
      const double w1 = d.wGx[ELL(k, i)], w2 = d.wGy[ELL(k, i)];
      const double T11 = d.tau[0][j] - Ti11, T21 = d.tau[1][j] - Ti21;
      const double T12 = d.tau[2][j] - Ti12, T22 = d.tau[3][j] - Ti22;
      const double kw1 = mul_int(K11, w1) + mul_int(K12, w2), kw2 = mul_int(K21, w1) + mul_int(K22, w2);
      const double tw1 = mul_int(T11, kw1) + mul_int(T12, kw2), tw2 = mul_int(T21, kw1) + mul_int(T22, kw2);
      put(0, mul_int(cp, tw1));
      put(1, mul_int(mul_int(cs, u1), wl));
      put(2, mul_int(cp, tw2));
      put(3, mul_int(mul_int(cs, u2), wl));
    } else {
      put(1, mul_int(mul_int(cs, u1), wl));
      put(3, mul_int(mul_int(cs, u2), wl));
    }
    put(5, mul_int(mul_int(ct, ti - d.th[j]), wl));
  };
  if constexpr (P == 1) {
    for (int k = 0; k < cnt; ++k)
      pair(k, [&](int e, double v) {
        if (e < 2) s1 = s1 + v;
        else if (e < 4) s2 = s2 + v;
        else st = st + v;
      });
  } else {
    double s[3];
    pair_sums64<3, 2>(
        cnt,
        [&](int k, double* t) {
          t[0] = t[2] = t[4] = 0.0;
          pair(k, [&](int e, double v) { t[e] = v; });
        },
        s);
    if (!in || (threadIdx.x & (P - 1))) return;
    s1 = s[0], s2 = s[1], st = s[2];
  }
  s2 = s2 + ti;  // buoyancy (predictor_mod.F90:111-119)
  const double dt = d.s->dt;
  if (i >= c.nbS) {
    d.ux2[i] = ui + s1 * dt;
    d.uy2[i] = vi + s2 * dt;
    d.th2[i] = ti + st * dt;
  } else {
    d.ux2[i] = ui;
    d.uy2[i] = vi;
    d.th2[i] = ti;
  }
}

__device__ __forceinline__ void pgrad_one(const Consts& c, const Dev& d, int i, int cnt, double a, double b, double& mu,
                                          double& mv, double& mp) {
  const double pi_ = d.p[i];
  const double K11 = d.kgcm[0][i], K21 = d.kgcm[1][i], K12 = d.kgcm[2][i], K22 = d.kgcm[3][i];
  double gx = K11 * a + K12 * b, gy = K21 * a + K22 * b;
  d.gpx[i] = gx;
  d.gpy[i] = gy;
  const double dt = d.s->dt;
  double ux = d.ux2[i], uy = d.uy2[i], x = d.rx[i], y = d.ry[i];
  if (i >= c.nbS) {
    ux = ux + dt * (c.bf[0] - gx);
    uy = uy + dt * (c.bf[1] - gy);
    if (cnt <= 3) {
      ux = d.u0x[i] + dt * c.bf[0];
      uy = d.u0y[i] + dt * c.bf[1];
    }
    if (!c.correct_velocity) {  // else k_advect_final moves the particles after the correction
      x = d.r0x[i] + 0.5 * (ux + d.u0x[i]) * dt + d.ushx[i] * dt;
      y = d.r0y[i] + 0.5 * (uy + d.u0y[i]) * dt + d.ushy[i] * dt;
    }
  }
  d.ux[i] = ux;
  d.uy[i] = uy;
  d.rx[i] = x;
  d.ry[i] = y;
  mu = fabs(ux);
  mv = fabs(uy);
  mp = fabs(pi_);
}

// ---------------------------------------------------------------------- pressure gradient
// grad P, velocity update (div_free.F90:96-101), final advection (:111-117): reads u* (ux2)
// and writes u^{n+1} and r^{n+1} in place (no kernel of this launch reads neighbours' u or r).
template <int P>
__global__ void __launch_bounds__(P == 1 ? TPB : LANES_TPB) k_pgrad_final(Consts c, Dev d) {
  bool in;
  const int i = lane_row<P>(c.npfb, in);
  double mu = -1.0, mv = -1.0, mp = -1.0;
  const int cnt = in ? d.ij_count[i] : 0;
  const double pi_ = d.p[i];
  double a = 0, b = 0;
  auto pair = [&](int k, double* t) {
    const double temp = d.p[d.ij_link[ELL(k, i)]] - pi_;
    t[0] = temp * d.wGx[ELL(k, i)];
    t[1] = temp * d.wGy[ELL(k, i)];
  };
  if constexpr (P == 1) {
    for (int k = 0; k < cnt; ++k) {
      double t[2];
      pair(k, t);
      a = a + t[0];
      b = b + t[1];
    }
  } else {
    double s[2];
    pair_sums64<2, 1>(cnt, pair, s);
    a = s[0], b = s[1];
    if (threadIdx.x & (P - 1)) in = false;  // the row's first lane has the rest
  }
  if (in) pgrad_one(c, d, i, cnt, a, b, mu, mv, mp);
  // divergence guard (opt-in) on the new velocity (false for NaN too)
  if (c.u_limit > 0.0 && in && !(mu <= c.u_limit && mv <= c.u_limit)) set_error(d.s, VEBI_ERR_DIVERGED);
  warp_max_pos(&d.s->absu_bits, mu);
  warp_max_pos(&d.s->absv_bits, mv);
  warp_max_pos(&d.s->absp_bits, mp);
}


// correct_velocity (correct_velocity.F90:13-70), behind a switch: the reference has the call
// commented out (div_free.F90:105).  Particles closer than dx to a wall (or wall-wall corner)
// mirror lose the velocity component towards it.  A circle mirror (vrelation = 999+ib) is not
// treated as a wall: the reference indexes b_type out of range there.
__global__ void k_correct_velocity(Consts c, Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.nbS || i >= c.npfb) return;
  const double xi = d.rx[i], yi = d.ry[i];
  double r_min2 = c.dx * c.dx;
  int close = -1;
  const int cnt = d.ij_count[i];
  for (int k = 0; k < cnt; ++k) {
    int j = d.ij_link[ELL(k, i)];
    if (j < c.npfb) continue;
    double a = xi - d.rx[j], b = yi - d.ry[j];
    double d2 = a * a + b * b;
    if (!(d2 < r_min2)) continue;
    int vr = d.vrel[j];
    if (vr > 0 && vr < 999 && c.b_type[vr - 1] == 1) { r_min2 = d2; close = j; }
    if (vr == -1 || vr < -2) { r_min2 = d2; close = j; }
  }
  if (close < 0) return;
  double n1 = xi - d.rx[close], n2 = yi - d.ry[close];
  double t = sqrt(n1 * n1 + n2 * n2);
  n1 = n1 / t;
  n2 = n2 / t;
  double u1 = d.ux[i] - d.ux2[close], u2 = d.uy[i] - d.uy2[close];
  double un = u1 * n1 + u2 * n2;
  if (un <= 0.0) {
    d.ux[i] = d.ux[i] - un * n1;
    d.uy[i] = d.uy[i] - un * n2;
  }
}

// final advection after correct_velocity (div_free.F90:111-117)
__global__ void k_advect_final(Consts c, Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.nbS || i >= c.npfb) return;
  const double dt = d.s->dt;
  d.rx[i] = d.r0x[i] + 0.5 * (d.ux[i] + d.u0x[i]) * dt + d.ushx[i] * dt;
  d.ry[i] = d.r0y[i] + 0.5 * (d.uy[i] + d.u0y[i]) * dt + d.ushy[i] * dt;
}

// secondary_properties: vorticity from final fluid u and mirror u* (div_free.F90:160-183)
template <typename W>
__global__ void k_secondary(Consts c, Dev d, const double* __restrict__ uxn, const double* __restrict__ uyn,
                            const double* __restrict__ uxm, const double* __restrict__ uym,
                            const W* __restrict__ wgx, const W* __restrict__ wgy) {
  __shared__ double sh[TPB / 32 + 1];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (i < c.npfb) {
    const double ui = uxn[i], vi = uyn[i];
    double vt = 0.0;
    const int cnt = d.ij_count[i];
    for (int k = 0; k < cnt; ++k) {
      int j = d.ij_link[ELL(k, i)];
      double uj = j < c.npfb ? uxn[j] : uxm[j], vj = j < c.npfb ? uyn[j] : uym[j];
      double tmp = (vi - vj) * (double)wgx[ELL(k, i)] - (ui - uj) * (double)wgy[ELL(k, i)];
      vt = vt - tmp;
    }
    d.vort[i] = vt;
    e = ui * ui + vi * vi;
  }
  double bs = block_sum<TPB>(e, sh);
  if (threadIdx.x == 0) d.partials[blockIdx.x] = bs;
}

__global__ void k_secondary_final(Consts c, Dev d, int nblk) {
  __shared__ double sh[TPB / 32 + 1];
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += d.partials[b];
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) d.s->rms_u = sqrt(s / (double)c.npfb);
}

// Force of the fluid on the circles (the cylinder's drag and lift), as the step's own pair
// terms see it: for every fluid particle, the circle mirrors' (vrelation > 999) share of the
// viscous and polymeric sums of prediction_step (predictor_mod.F90:27-139) and of the pressure
// gradient of calc_pressure_gradient (gradient_calculation.F90:16-48), times dv; the circles
// feel the opposite.  Evaluated after the step from the values those stages read: the
// start-of-step fluid velocity u0, the mirrors' creation-time velocity (ux/uy at npfb..), the
// updated tau and the new pressure.  A diagnostic of this library; the reference has none.
// A circle mirror lies at radius 2R - rad of a source at rad (inside the support band), so a
// particle that has one as a neighbour (distance <= sup) is within sup of the circle: the
// mirror stages' candidate list (every particle within sup plus a margin of a boundary, in
// ascending index) holds all of them, and the kernels walk that list alone.
// k_circle_terms: a warp per candidate, a lane per pair; then four lanes add the mirrors' terms in
// slot order, one lane for each of the viscous and pressure sums.  k_circle_force adds the candidates.
// Measured, both: 19 us at 20k particles; by one thread per candidate, pair after pair, 137.
constexpr int CF_BLOCKS = 256;

template <class W>
__global__ void __launch_bounds__(TPB) k_circle_terms(Consts c, Dev d, const W* __restrict__ wgx, const W* __restrict__ wgy,
                                                      const W* __restrict__ wl_, const W* __restrict__ k11,
                                                      const W* __restrict__ k21, const W* __restrict__ k12,
                                                      const W* __restrict__ k22) {
  __shared__ double first[TPB / 32][4][32], second[TPB / 32][4][32];  // terms of the sums s1, s2, a, b
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncand = d.s->n_cand;
  const bool ve = c.const_mod != 1;
  const double cs = c.coeff_solvent, cp = c.coeff_polymeric;
  for (int q = blockIdx.x * (TPB / 32) + w; q < ncand; q += gridDim.x * (TPB / 32)) {
    const int i = d.cand[q];
    if (i < c.nbS || i >= c.npfb || d.inbin[i]) {
      if (lane < 2) d.circle_f[2 * (size_t)q + lane] = 0.0;
      continue;
    }
    const double ui = d.u0x[i], vi = d.u0y[i], pi_ = d.p[i];
    const double K11 = (double)k11[i], K21 = (double)k21[i], K12 = (double)k12[i], K22 = (double)k22[i];
    double Ti11 = 0, Ti21 = 0, Ti12 = 0, Ti22 = 0;
    if (ve) { Ti11 = d.tau[0][i]; Ti21 = d.tau[1][i]; Ti12 = d.tau[2][i]; Ti22 = d.tau[3][i]; }
    double sum = 0.0;  // of lanes 0..3
    const int cnt = d.ij_count[i];
    for (int k0 = 0; k0 < cnt; k0 += 32) {
      const int k = k0 + lane, j = k < cnt ? d.ij_link[ELL(k, i)] : -1;
      const bool hit = j >= c.npfb && d.vrel[j] > 999;
      unsigned hits = __ballot_sync(0xffffffffu, hit);
      if (!hits) continue;
      if (hit) {
        const double w1 = (double)wgx[ELL(k, i)], w2 = (double)wgy[ELL(k, i)], wl = (double)wl_[ELL(k, i)];
        const double u1 = ui - d.ux[j], u2 = vi - d.uy[j], temp = d.p[j] - pi_;
        if (ve) {
          const double T11 = d.tau[0][j] - Ti11, T21 = d.tau[1][j] - Ti21;
          const double T12 = d.tau[2][j] - Ti12, T22 = d.tau[3][j] - Ti22;
          const double kw1 = K11 * w1 + K12 * w2, kw2 = K21 * w1 + K22 * w2;
          first[w][0][lane] = cp * (T11 * kw1 + T12 * kw2);
          first[w][1][lane] = cp * (T21 * kw1 + T22 * kw2);
        }
        second[w][0][lane] = cs * u1 * wl;
        second[w][1][lane] = cs * u2 * wl;
        second[w][2][lane] = temp * w1;
        second[w][3][lane] = temp * w2;
      }
      __syncwarp();
      if (lane < 4)
        for (; hits; hits &= hits - 1) {
          const int u = __ffs(hits) - 1;
          if (ve && lane < 2) sum = sum + first[w][lane][u];
          sum = sum + second[w][lane][u];
        }
      __syncwarp();
    }
    const double s = __shfl_sync(0xffffffffu, sum, lane & 1);
    const double a = __shfl_sync(0xffffffffu, sum, 2), b = __shfl_sync(0xffffffffu, sum, 3);
    if (lane < 2) {
      const double g = lane == 0 ? K11 * a + K12 * b : K21 * a + K22 * b;
      d.circle_f[2 * (size_t)q + lane] = c.dv * (g - s);
    }
  }
}

__global__ void __launch_bounds__(TPB) k_circle_force(Dev d) {
  __shared__ double sh[TPB / 32 + 1];
  const int ncand = d.s->n_cand;
  double fx = 0.0, fy = 0.0;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < ncand; q += gridDim.x * blockDim.x) {
    fx += d.circle_f[2 * (size_t)q];
    fy += d.circle_f[2 * (size_t)q + 1];
  }
  double bx = block_sum<TPB>(fx, sh);
  double by = block_sum<TPB>(fy, sh);
  if (threadIdx.x == 0) {
    d.partials[blockIdx.x] = bx;
    d.partials[gridDim.x + blockIdx.x] = by;
  }
}

__global__ void k_circle_force_final(Dev d, int nblk) {
  __shared__ double sh[TPB / 32 + 1];
  double sx = 0.0, sy = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    sx += d.partials[b];
    sy += d.partials[nblk + b];
  }
  sx = block_sum<TPB>(sx, sh);
  sy = block_sum<TPB>(sy, sh);
  if (threadIdx.x == 0) {
    d.s->circle_fx = sx;
    d.s->circle_fy = sy;
  }
}

void launch_prep_weights32(Ctx& x);
void launch_shift32(Ctx& x);
void launch_gradients32(Ctx& x);
void launch_predictor32(Ctx& x);
void launch_pgrad_final32(Ctx& x);

static void launch_weights(Ctx& x) {
  const Consts& c = x.c;
  double* fab = x.d.ppe_val;  // free until the PPE is assembled
  const long long n = c.npfb;
  // Lanes per row, measured with 8 / 4 / 1: 20k particles 0.15 / 0.17 / 0.44 ms, 60k 0.37 / 0.35 /
  // 0.52, 100k 0.58 / 0.53 / 0.60, 250k 1.19 / 1.23 / 1.08.
  if (n <= 40000) VEBI_LAUNCH(x, k_pair_terms<8>, grid_for(n * 8, PAIR_TPB), PAIR_TPB, c, x.d, fab);
  else if (n <= 150000) VEBI_LAUNCH(x, k_pair_terms<4>, grid_for(n * 4, PAIR_TPB), PAIR_TPB, c, x.d, fab);
  else VEBI_LAUNCH(x, k_pair_terms<1>, grid_for(n, PAIR_TPB), PAIR_TPB, c, x.d, fab);
  if (n <= 150000) VEBI_LAUNCH(x, k_weight_sums<4>, grid_for(n * 4, PAIR_TPB), PAIR_TPB, c, x.d, fab);
  else VEBI_LAUNCH(x, k_weight_sums<1>, grid_for(n), TPB, c, x.d, fab);
}

void launch_weights_surface_shift(Ctx& x) {
  const Consts& c = x.c;
  int g = grid_for(c.npfb);
  const bool mixed = x.precision == VEBI_PREC_MIXED;
  if (mixed) launch_prep_weights32(x);
  // FP64 weights: the FP64 step, and the free-surface operators and shifting of an open domain
  const bool f64 = !mixed || c.open_domain == 1;
  if (f64) launch_weights(x);
  if (c.open_domain == 1) {
    LAUNCH_ROWS(x, k_part_dist_vars, LANE_ROWS);
    VEBI_LAUNCH(x, k_nsurf_mirrors, x.gs_blocks, TPB, c, x.d);
    LAUNCH_ROWS(x, k_smooth_normals, LANE_ROWS);
    VEBI_LAUNCH(x, k_copy_normals, g, TPB, c, x.d);
  } else {
    cudaMemsetAsync(x.d.n_surf, 0, sizeof(int) * (size_t)c.cap, x.st);
  }
  stage_mark(x, 5);
  if (!f64) launch_shift32(x);
  else if (c.open_domain == 1) VEBI_LAUNCH(x, k_shift_open, g, TPB, c, x.d);
}

void launch_grad_mirrors(Ctx& x);
void launch_mirror_stress(Ctx& x);
void launch_mirror_velocities(Ctx& x);
void launch_mirror_pressure(Ctx& x);

void launch_predictor(Ctx& x) {
  const Consts& c = x.c;
  int g = grid_for(c.npfb);
  const bool mixed = x.precision == VEBI_PREC_MIXED;
  stage_mark(x, 6);
  if (mixed) launch_gradients32(x);
  else LAUNCH_ROWS(x, k_gradients, LANE_ROWS);
  launch_grad_mirrors(x);
  stage_mark(x, 7);
  if (c.const_mod != 1) {
    VEBI_LAUNCH(x, k_logconf, g, TPB, c, x.d);
    launch_mirror_stress(x);
  }
  stage_mark(x, 8);
  if (mixed) launch_predictor32(x);
  else LAUNCH_ROWS(x, k_predictor, LANE_ROWS);
  launch_mirror_velocities(x);
  // theta* replaces theta for walls and fluid; u* stays in ux2/uy2 for the PPE and the update
  cudaMemcpyAsync(x.d.th, x.d.th2, sizeof(double) * (size_t)c.npfb, cudaMemcpyDeviceToDevice, x.st);
}

void launch_final(Ctx& x, int secondary) {
  const Consts& c = x.c;
  int g = grid_for(c.npfb);
  stage_mark(x, 11);
  launch_mirror_pressure(x);
  // keep r* (fluid and mirrors) readable after the step: the update below overwrites r
  cudaMemcpyAsync(x.d.rx2, x.d.rx, sizeof(double) * (size_t)c.cap, cudaMemcpyDeviceToDevice, x.st);
  cudaMemcpyAsync(x.d.ry2, x.d.ry, sizeof(double) * (size_t)c.cap, cudaMemcpyDeviceToDevice, x.st);
  const bool mixed = x.precision == VEBI_PREC_MIXED;
  if (mixed) launch_pgrad_final32(x);
  else LAUNCH_ROWS(x, k_pgrad_final, LANE_ROWS_PGRAD);
  if (c.correct_velocity) {
    VEBI_LAUNCH(x, k_correct_velocity, g, TPB, c, x.d);
    VEBI_LAUNCH(x, k_advect_final, g, TPB, c, x.d);
  }
  if (c.ncirc > 0) {
    const int cb = 6 * x.nsm < (c.npfb + 7) / 8 ? 6 * x.nsm : (c.npfb + 7) / 8;
    if (mixed)
      VEBI_LAUNCH(x, k_circle_terms<float>, cb, TPB, c, x.d, x.d.wGx32, x.d.wGy32, x.d.wL32, x.d.kgcm32[0],
                  x.d.kgcm32[1], x.d.kgcm32[2], x.d.kgcm32[3]);
    else
      VEBI_LAUNCH(x, k_circle_terms<double>, cb, TPB, c, x.d, x.d.wGx, x.d.wGy, x.d.wL, x.d.kgcm[0], x.d.kgcm[1],
                  x.d.kgcm[2], x.d.kgcm[3]);
    VEBI_LAUNCH(x, k_circle_force, CF_BLOCKS, TPB, x.d);
    VEBI_LAUNCH(x, k_circle_force_final, 1, TPB, x.d, CF_BLOCKS);
  }
  if (secondary) {
    stage_mark(x, 13);
    if (mixed) VEBI_LAUNCH(x, k_secondary<float>, g, TPB, c, x.d, x.d.ux, x.d.uy, x.d.ux2, x.d.uy2, x.d.wGx32, x.d.wGy32);
    else VEBI_LAUNCH(x, k_secondary<double>, g, TPB, c, x.d, x.d.ux, x.d.uy, x.d.ux2, x.d.uy2, x.d.wGx, x.d.wGy);
    VEBI_LAUNCH(x, k_secondary_final, 1, TPB, c, x.d, g);
  }
}

}  // namespace vebi
