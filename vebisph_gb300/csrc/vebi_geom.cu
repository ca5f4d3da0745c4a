// vebi_geom.cu -- time step bound, advection, bin, escapees and mirror particles.
//
//  set_time_step        div_free.F90:126-146
//  advection r*=r+dt u  div_free.F90:47-53
//  put_in_bin           put_in_bin.F90:1-56
//  replace_escapees     mirror_boundaries_mod.F90:336-407
//  create_mirror_particles (+create_boundary_boxes)  mirror_boundaries_mod.F90:18-334,409-445
//  mirror_velocities    mirror_boundaries_mod.F90:509-584
//  mirror_polymeric_stress                 mirror_boundaries_mod.F90:586-653
//  grad_operator mirror transfer           gradient_calculation.F90:96-145
//
// The reference builds mirrors serially with one global counter `imp`, patch after patch,
// then corner after corner; wall-periodic corners scan the mirrors made so far.  Here every
// stage is an order-preserving stream compaction (count / scan / emit), so mirror k here is mirror k
// of the reference.
#include "vebi_ctx.cuh"

namespace vebi {

// ------------------------------------------------------------------------------- step start
__global__ void k_step_reset(Scal* s, int npfb, int nbS) {
  // a failed step (device status, or every liquid particle binned) stays recorded; later
  // steps of this state skip the PPE solve
  if (!s->first_error) {
    if (s->error) s->first_error = s->error;
    else if (npfb > nbS && s->n_inbin == npfb - nbS) s->first_error = VEBI_ERR_ALL_IN_BIN;
  }
  s->umax_bits = (unsigned long long)__double_as_longlong(1.0e-10);
  s->maxU_bits = (unsigned long long)__double_as_longlong(1.0e-10);
  s->absu_bits = s->absv_bits = s->absp_bits = 0ull;
  s->nmirror = 0;
  s->np = npfb;
  s->n_inbin = 0;
  s->n_escapees = 0;
  s->maxneigh = 0;
  s->ls_iters = 0;
  s->warnings = 0;
  s->error = 0;
  s->rhs_mean = 0.0;
  s->ls_residual = 0.0;
  s->rms_u = 0.0;
  s->bar_count = 0u;
  s->refine_iters = 0;
  s->one_sided = 0;
  s->n_end = s->n_node = 0;
  s->mg_fail = 0;
  s->n_near_pole = 0;
}

// STEP 1-2: keep r0,u0 and reduce max|u| over the fluid (set_time_step)
__global__ void k_save_umax(Consts c, Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  double um = -1.0;
  if (i < c.npfb) {
    double ux = d.ux[i], uy = d.uy[i];
    d.r0x[i] = d.rx[i];
    d.r0y[i] = d.ry[i];
    d.u0x[i] = ux;
    d.u0y[i] = uy;
    if (i >= c.nbS) {
      um = sqrt(ux * ux + uy * uy);
      // divergence guard (opt-in): a non-finite or runaway velocity fails the step
      if (c.u_limit > 0.0 && !(um <= c.u_limit)) set_error(d.s, VEBI_ERR_DIVERGED);
    }
  }
  warp_max_pos(&d.s->umax_bits, um);
}

__device__ __forceinline__ double step_dt(const Consts& c, const Scal* s) {
  double umax = bits_to_double(s->umax_bits);
  double dt_cfl = c.dt_coef_cfl * c.h / umax;
  return fmin(dt_cfl, c.dt_visc);
}

// STEP 3-4: advect, bin, replace escapees; per particle, in the reference's order
__device__ __forceinline__ double advect_bin_one(const Consts& c, const Dev& d, int i, double dt);

__global__ void k_advect_bin(Consts c, Dev d) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  Scal* s = d.s;
  const double dt = step_dt(c, s);
  if (i == 0) s->dt = dt;
  double um = -1.0;
  if (i < c.nbS) {  // walls do not move; they still enter the maximum of new_fick_shift
    um = sqrt(d.ux[i] * d.ux[i] + d.uy[i] * d.uy[i]);
  } else if (i < c.npfb) {
    um = advect_bin_one(c, d, i, dt);
  }
  warp_max_pos(&s->maxU_bits, um);
}

// one fluid particle: advection, put_in_bin, replace_escapees; returns |u| after binning
__device__ __forceinline__ double advect_bin_one(const Consts& c, const Dev& d, int i, double dt) {
  Scal* s = d.s;
  double x = d.r0x[i] + d.u0x[i] * dt;
  double y = d.r0y[i] + d.u0y[i] * dt;
  double ux = d.ux[i], uy = d.uy[i];
  // put_in_bin
  bool ib = d.inbin[i] != 0;
  if (!ib) {
    if (x < c.x_mint || x > c.x_maxt || y < c.y_mint || y > c.y_maxt) ib = true;
    if (isnan(x) || isnan(y)) ib = true;
  }
  if (ib) {
    x = 2.0 * c.x_mint - c.x_maxt;
    y = 2.0 * c.y_mint - c.y_maxt;
    ux = 0.0;
    uy = 0.0;
    atomicAdd(&s->n_inbin, 1);
    d.inbin[i] = 1;
    d.ux[i] = 0.0;
    d.uy[i] = 0.0;
  }
  // replace_escapees: circles (no bin test in the reference), then walls / periodic patches
  int nesc = 0;
  bool touched = false;
  // FP32 prefilters (margin near_band): a particle clearly away from a circle or a patch skips
  // the FP64 tests, which would find nothing to do for it
  const float band = c.near_band;
  for (int ic = 0; ic < c.ncirc; ++ic) {
    double R = c.c_radius[ic];
    {  // from the current position: an earlier circle may have moved the particle
      const float d1 = (float)x - (float)c.c_centre[ic][0], d2 = (float)y - (float)c.c_centre[ic][1];
      const float q = fmaf(d1, d1, d2 * d2), Rf = (float)fabs(R);
      if (R > 0.0 && q > (Rf + band) * (Rf + band)) continue;              // clearly outside
      if (R < 0.0 && Rf > band && q < (Rf - band) * (Rf - band)) continue;  // clearly inside
    }
    double ric1 = x - c.c_centre[ic][0], ric2 = y - c.c_centre[ic][1];
    double rad = sqrt(ric1 * ric1 + ric2 * ric2);
    if (rad < fabs(R) && R > 0.0) {
      x = x + (ric1 / rad) * 2.0 * (R - rad);
      y = y + (ric2 / rad) * 2.0 * (R - rad);
      ++nesc;
    }
    if (rad > fabs(R) && R < 0.0) {
      x = x - (ric1 / rad) * 2.0 * (rad + R);
      y = y - (ric2 / rad) * 2.0 * (rad + R);
      ++nesc;
    }
  }
  double r0x = 0.0, r0y = 0.0;
  for (int p = 0; p < c.nb; ++p) {
    if (c.b_type[p] != 1 && c.b_type[p] != 2) continue;
    if (ib) continue;
    {
      const float pf = fmaf(c.bl_a[p], (float)x, fmaf(c.bl_b[p], (float)y, c.bl_c[p]));
      if (pf > band || pf < -band) continue;  // clearly inside, or clearly beyond the support
    }
    double perp = bound_dist(c, x, y, p);
    if (perp > 0.0) continue;
    if (fabs(perp) > c.sup_size + 1.0e-10) continue;
    double n1, n2;
    bound_norm(c, p, n1, n2);
    double tmp = pos_along(c, x, y, p, perp, n1, n2);
    if (c.b_type[p] == 1) {
      if (tmp < 0.0 || tmp > 1.0) continue;
      x = x - 2.0 * perp * n1;
      y = y - 2.0 * perp * n2;
    } else {
      int pp = c.b_pp[p];
      double pn1, pn2;
      bound_norm(c, pp, pn1, pn2);
      double t1 = -1.0 * tmp * c.b_edge[pp][0] - perp * pn1;
      double t2 = -1.0 * tmp * c.b_edge[pp][1] - perp * pn2;
      x = c.b_node[pp][0] + c.b_edge[pp][0] + t1;
      y = c.b_node[pp][1] + c.b_edge[pp][1] + t2;
    }
    ++nesc;
    r0x = x - ux * dt;
    r0y = y - uy * dt;
    touched = true;
  }
  if (touched) {
    d.r0x[i] = r0x;
    d.r0y[i] = r0y;
    d.u0x[i] = ux;
    d.u0y[i] = uy;
  }
  if (nesc) atomicAdd(&s->n_escapees, nesc);
  d.rx[i] = x;
  d.ry[i] = y;
  return sqrt(ux * ux + uy * uy);
}

// ------------------------------------------------------------------------------- mirrors
enum SelKind { SEL_CIRCLES = 0, SEL_WALL, SEL_PERIODIC, SEL_CORNER_WW, SEL_CORNER_PP, SEL_CORNER_WP, SEL_CANDIDATES };

struct SelArgs {
  int kind;
  int ib;      // patch (0-based)
};

// near-patch test of create_boundary_boxes: |perp| <= sup+1e-10 and 0<=tmp<=1
__device__ __forceinline__ bool near_patch(const Consts& c, double x, double y, int ib, double& tmp,
                                           double& perp) {
  perp = bound_dist(c, x, y, ib);
  if (fabs(perp) > c.sup_size + 1.0e-10) return false;
  double n1, n2;
  bound_norm(c, ib, n1, n2);
  tmp = pos_along(c, x, y, ib, perp, n1, n2);
  if (tmp < 0.0 || tmp > 1.0) return false;
  return true;
}
__device__ __forceinline__ bool near_corner(const Consts& c, double x, double y, int ib) {
  double a = x - c.b_node[ib][0], b = y - c.b_node[ib][1];
  double dd = sqrt(a * a + b * b);
  return !(dd > c.sup_size + 1.0e-10);
}

// number of mirrors item `it` creates in this stage.  A call, for the few items that pass an FP32
// test: inlined, the compiler computes its quotients for every particle.
static __device__ __noinline__ int sel_count(const Consts& c, const Dev& d, const SelArgs& a, int it) {
  const double x = d.rx[it], y = d.ry[it];
  switch (a.kind) {
    case SEL_CIRCLES: {
      int n = 0;
      for (int ic = 0; ic < c.ncirc; ++ic) {
        double R = c.c_radius[ic];
        double cdir = R / fabs(R);
        double r1 = x - c.c_centre[ic][0], r2 = y - c.c_centre[ic][1];
        double rad = sqrt(r1 * r1 + r2 * r2);
        if (cdir > 0.0) { if (rad <= R + c.sup_size) ++n; }
        else if (cdir < 0.0) { if (rad >= fabs(R) - c.sup_size) ++n; }
      }
      return n;
    }
    case SEL_WALL: {
      double bp1, bp2;
      if (!near_patch(c, x, y, a.ib, bp1, bp2)) return 0;
      if (bp2 <= 1.0e-10) return 0;
      int ibp1 = (a.ib + 1) % c.nb;
      double mbe = c.b_elen[a.ib];
      if (c.b_corner_angle[a.ib] < 0.0) {
        double ta = 0.5 * (PI + c.b_corner_angle[a.ib]);
        if (bp2 + 0.1 * c.dx >= bp1 * tan(ta) * mbe) return 0;
      }
      if (c.b_corner_angle[ibp1] < 0.0) {
        double ta = 0.5 * (PI + c.b_corner_angle[ibp1]);
        if (bp2 >= (1.0 - bp1) * tan(ta) * mbe) return 0;
      }
      return 1;
    }
    case SEL_PERIODIC: {
      double bp1, bp2;
      if (!near_patch(c, x, y, c.b_pp[a.ib], bp1, bp2)) return 0;
      return bp2 <= 0.0 ? 0 : 1;
    }
    case SEL_CORNER_WW:
      return near_corner(c, x, y, a.ib) ? 1 : 0;
    case SEL_CORNER_PP:
      return near_corner(c, x, y, c.b_pp[a.ib]) ? 1 : 0;
    case SEL_CORNER_WP: {
      int ibm1 = (a.ib + c.nb - 1) % c.nb;
      int ibb = (c.b_type[ibm1] == 1) ? ibm1 : a.ib;
      double perp = bound_dist(c, x, y, ibb);
      if (perp > c.sup_size + 1.0e-10) return 0;
      if (perp < 1.0e-10) return 0;
      double n1, n2;
      bound_norm(c, ibb, n1, n2);
      double t = pos_along(c, x, y, ibb, perp, n1, n2);
      return ((t < 0.0 && ibb == a.ib) || (t > 1.0 && ibb == ibm1)) ? 1 : 0;
    }
  }
  return 0;
}

__device__ __forceinline__ double dPf(const Consts& c, double xk, double yk, double xi, double yi) {
  return c.bf[0] * (xk - xi) + c.bf[1] * (yk - yi);
}

// write the mirrors of item `it` starting at mirror slot `slot` (0-based mirror number)
static __device__ __noinline__ void sel_emit(const Consts& c, const Dev& d, const SelArgs& a, int it, int slot) {
  const double x = d.rx[it], y = d.ry[it];
  auto put = [&](int parent, int vrel, double mx, double my, double mu, double mv, double mth,
                 double dp) -> void {
    if (slot >= c.mcap) { set_error(d.s, VEBI_ERR_MIRROR_CAPACITY); return; }
    int k = c.npfb + slot;
    d.irel[k] = parent;
    d.vrel[k] = vrel;
    d.rx[k] = mx;
    d.ry[k] = my;
    d.ux[k] = mu;
    d.uy[k] = mv;
    d.th[k] = mth;
    d.dP_mp[k] = dp;
    d.inbin[k] = 0;
    ++slot;
  };
  switch (a.kind) {
    case SEL_CIRCLES: {
      for (int ic = 0; ic < c.ncirc; ++ic) {
        double R = c.c_radius[ic];
        double cdir = R / fabs(R);
        double r1 = x - c.c_centre[ic][0], r2 = y - c.c_centre[ic][1];
        double rad = sqrt(r1 * r1 + r2 * r2);
        bool make = false;
        double mx = 0, my = 0, Ra = 0;
        if (cdir > 0.0) {
          if (rad <= R + c.sup_size) {
            r1 = r1 / rad; r2 = r2 / rad;
            mx = x - r1 * 2.0 * (rad - R);
            my = y - r2 * 2.0 * (rad - R);
            Ra = R;
            make = true;
          }
        } else if (cdir < 0.0) {
          if (rad >= fabs(R) - c.sup_size) {
            r1 = r1 / rad; r2 = r2 / rad;
            mx = x + r1 * 2.0 * (fabs(R) - rad);
            my = y + r2 * 2.0 * (fabs(R) - rad);
            Ra = fabs(R);
            make = true;
          }
        }
        if (make) {
          double t1 = r2, t2 = -r1;
          double mu = 2.0 * c.c_vel[ic][0] + 2.0 * t1 * Ra * c.c_omega[ic] - 1.0 * d.ux[it];
          double mv = 2.0 * c.c_vel[ic][1] + 2.0 * t2 * Ra * c.c_omega[ic] - 1.0 * d.uy[it];
          double mth = 2.0 * c.c_thermal[ic] - 1.0 * d.th[it];
          put(it, 999 + ic + 1, mx, my, mu, mv, mth, dPf(c, mx, my, x, y));
        }
      }
      break;
    }
    case SEL_WALL: {
      double bp1, bp2;
      near_patch(c, x, y, a.ib, bp1, bp2);
      double n1, n2;
      bound_norm(c, a.ib, n1, n2);
      double mx = x - 2.0 * bp2 * n1, my = y - 2.0 * bp2 * n2;
      double t1 = n2, t2 = -n1;
      put(it, a.ib + 1, mx, my, 2.0 * c.b_vel[a.ib] * t1 - d.ux[it], 2.0 * c.b_vel[a.ib] * t2 - d.uy[it],
          2.0 * c.b_thermal[a.ib] - d.th[it], dPf(c, mx, my, x, y));
      break;
    }
    case SEL_PERIODIC: {
      double bp1, bp2;
      near_patch(c, x, y, c.b_pp[a.ib], bp1, bp2);
      double n1, n2;
      bound_norm(c, a.ib, n1, n2);
      double t1 = -1.0 * bp1 * c.b_edge[a.ib][0] - bp2 * n1;
      double t2 = -1.0 * bp1 * c.b_edge[a.ib][1] - bp2 * n2;
      double mx = c.b_node[a.ib][0] + c.b_edge[a.ib][0] + t1;
      double my = c.b_node[a.ib][1] + c.b_edge[a.ib][1] + t2;
      put(it, a.ib + 1, mx, my, d.ux[it], d.uy[it], d.th[it], 0.0);
      break;
    }
    case SEL_CORNER_WW: {
      int ib = a.ib, ibm1 = (ib + c.nb - 1) % c.nb;
      // `tmp` of the reference still holds the edge cross product (mirror_..:216,242)
      double tmp = c.b_edge[ibm1][0] * c.b_edge[ib][1] - c.b_edge[ibm1][1] * c.b_edge[ib][0];
      double tb1 = x - c.b_node[ib][0], tb2 = y - c.b_node[ib][1];
      double mx = x - 2.0 * tb1, my = y - 2.0 * tb2;
      double n1, n2;
      bound_norm(c, ib, n1, n2);
      double mu = 2.0 * tmp * n2 - d.ux[it];
      double mv = 2.0 * tmp * (-n1) - d.uy[it];
      bound_norm(c, ibm1, n1, n2);
      mu = mu + 2.0 * tmp * n2;
      mv = mv + 2.0 * tmp * (-n1);
      put(it, -(ib + 1), mx, my, mu, mv, d.th[it] + 2.0 * c.b_thermal[ib], dPf(c, mx, my, x, y));
      break;
    }
    case SEL_CORNER_PP: {
      int ib = a.ib, ibp = c.b_pp[ib];
      double tb1 = c.b_node[ib][0] - c.b_node[ibp][0], tb2 = c.b_node[ib][1] - c.b_node[ibp][1];
      put(it, -(ib + 1), x + tb1, y + tb2, d.ux[it], d.uy[it], d.th[it], 0.0);
      break;
    }
    case SEL_CORNER_WP: {
      int ib = a.ib, ibm1 = (ib + c.nb - 1) % c.nb;
      int ibb = (c.b_type[ibm1] == 1) ? ibm1 : ib;
      double perp = bound_dist(c, x, y, ibb);
      double n1, n2;
      bound_norm(c, ibb, n1, n2);
      double mx = x - 2.0 * perp * n1, my = y - 2.0 * perp * n2;
      double t1 = n2, t2 = -n1;
      double dp = d.dP_mp[it];
      dp = dp + (c.bf[0] * (mx - x) + c.bf[1] * (my - y));
      put(d.irel[it], -(ib + 1), mx, my, 2.0 * c.b_vel[ibb] * t1 - d.ux[it], 2.0 * c.b_vel[ibb] * t2 - d.uy[it],
          2.0 * c.b_thermal[ibb] - d.th[it], dp);
      break;
    }
  }
}

// ---- the stages.  The reference makes circle images, then patch after patch wall and periodic
// images, then corner after corner; the order of the mirrors is that of the stages and, in a
// stage, of its items.  The stages over particles up to the corners depend on the particles alone,
// so one kernel selects for all of them (a bit per particle and stage, and a count per block of
// particles), one scan places the blocks and one kernel emits, a thread per mirror.  What a corner
// needs -- the mirrors made so far past a wall's end, the particles about a node -- is a few dozen
// items however large the domain: the emitting kernel lists them and one block runs the corners.
// Measured, all of it: 0.06 to 0.08 ms a step from 1,700 to 20,000 particles, 0.26 ms at 4M; a
// count, a scan and an emission per stage (33 to 43 launches) took 0.36 to 0.72 and 0.82 ms, these
// kernels emitting from a thread per particle, its images in turn, 0.11 to 0.18 and 0.44 ms.
//
// Every FP64 test is preceded by an FP32 one with a margin of dx/10 plus 4e-6 of the box's extent,
// far above its rounding error: a wall or periodic image needs |perp| <= sup + 1e-10 to that patch's
// line, a corner image a node distance within the same bound, a circle image rad within R + sup (or
// |R| - sup).
constexpr int MIR_STAGES = VEBI_MAX_PATCHES + 2;  // circles, patches, candidates
struct MirrorPlan {
  int ns, nc;                                  // stages over particles (the candidates last), corners
  int first_plane[MIR_STAGES + 1];             // of each stage's selections (a bit per particle)
  signed char kind[MIR_STAGES], ib[MIR_STAGES];
  signed char ckind[VEBI_MAX_PATCHES], cib[VEBI_MAX_PATCHES];
};

// the candidates: every particle that any stage may select, in ascending order (k_circle_force)
struct NearTab {
  float a[VEBI_MAX_PATCHES], b[VEBI_MAX_PATCHES], c0[VEBI_MAX_PATCHES];  // perp = a x + b y + c0
  float cx[VEBI_MAX_CIRCLES], cy[VEBI_MAX_CIRCLES], lo2[VEBI_MAX_CIRCLES], hi2[VEBI_MAX_CIRCLES];
  float band;
  int np, nc;
};

__device__ void near_table(const Consts& c, NearTab& t) {
  const double m = c.near_band;
  if (threadIdx.x == 0) {
    int k = 0;
    for (int ib = 0; ib < c.nb; ++ib) {
      if (c.b_type[ib] == 0) continue;
      t.a[k] = c.bl_a[ib];
      t.b[k] = c.bl_b[ib];
      t.c0[k] = c.bl_c[ib];
      ++k;
    }
    t.np = k;
    for (int ic = 0; ic < c.ncirc; ++ic) {
      const double R = c.c_radius[ic];
      t.cx[ic] = (float)c.c_centre[ic][0];
      t.cy[ic] = (float)c.c_centre[ic][1];
      if (R > 0.0) { t.lo2[ic] = -1.0f; t.hi2[ic] = (float)((R + m) * (R + m)); }
      else { const double l = fmax(fabs(R) - m, 0.0); t.lo2[ic] = (float)(l * l); t.hi2[ic] = 3.0e38f; }
    }
    t.nc = c.ncirc;
    t.band = (float)m;
  }
  __syncthreads();
}

__device__ __forceinline__ bool near_boundary(const NearTab& t, float x, float y) {
  for (int k = 0; k < t.np; ++k)
    if (fabsf(fmaf(t.a[k], x, fmaf(t.b[k], y, t.c0[k]))) <= t.band) return true;
  for (int ic = 0; ic < t.nc; ++ic) {
    const float r1 = x - t.cx[ic], r2 = y - t.cy[ic];
    const float q = fmaf(r1, r1, r2 * r2);
    if (t.lo2[ic] < 0.0f ? q <= t.hi2[ic] : q >= t.lo2[ic]) return true;
  }
  return false;
}

// FP32 test of the stages over particles, one bit per stage
struct StageTab {
  float a[MIR_STAGES], b[MIR_STAGES], c0[MIR_STAGES];
  float band;
};
__device__ void stage_table(const Consts& c, const MirrorPlan& pl, StageTab& t) {
  const int s = threadIdx.x;
  if (s < pl.ns && (pl.kind[s] == SEL_WALL || pl.kind[s] == SEL_PERIODIC)) {
    const int ib = pl.kind[s] == SEL_PERIODIC ? c.b_pp[pl.ib[s]] : pl.ib[s];
    t.a[s] = c.bl_a[ib];
    t.b[s] = c.bl_b[ib];
    t.c0[s] = c.bl_c[ib];
  }
  t.band = c.near_band;
}
__device__ __forceinline__ unsigned stages_near(const Consts& c, const MirrorPlan& pl, const StageTab& t, int it, float x,
                                                float y) {
  unsigned m = 0;
  for (int s = 0; s < pl.ns; ++s) {
    if (pl.kind[s] == SEL_CIRCLES) {
      if (it < c.nbS) continue;
      bool near = false;
      for (int ic = 0; ic < c.ncirc; ++ic) {
        const float R = (float)c.c_radius[ic], r1 = x - (float)c.c_centre[ic][0], r2 = y - (float)c.c_centre[ic][1];
        const float q = fmaf(r1, r1, r2 * r2), e = fabsf(R) - t.band;
        near |= R > 0.0f ? q <= (R + t.band) * (R + t.band) : (e <= 0.0f || q >= e * e);
      }
      if (near) m |= 1u << s;
    } else if (pl.kind[s] != SEL_CANDIDATES && fabsf(fmaf(t.a[s], x, fmaf(t.b[s], y, t.c0[s]))) <= t.band) {
      m |= 1u << s;
    }
  }
  return m;
}

// what the corners may select, in FP32: mirrors by the line of a wall, past the end of it that is
// the corner; particles about a corner's node
__device__ __forceinline__ int corner_wall(const Consts& c, int ib) {
  const int ibm1 = (ib + c.nb - 1) % c.nb;
  return c.b_type[ibm1] == 1 ? ibm1 : ib;
}
__device__ __forceinline__ bool past_wall_end(const Consts& c, const MirrorPlan& pl, float x, float y) {
  const float slack = c.near_band - (float)c.sup_size;
  for (int q = 0; q < pl.nc; ++q) {
    if (pl.ckind[q] != SEL_CORNER_WP) continue;
    const int ib = pl.cib[q], wl = corner_wall(c, ib);
    const float perp = fmaf(c.bl_a[wl], x, fmaf(c.bl_b[wl], y, c.bl_c[wl]));
    if (!(perp >= -slack && perp <= c.near_band)) continue;
    const float len = (float)c.b_elen[wl];
    const float along = ((x - (float)c.b_node[wl][0]) * (float)c.b_edge[wl][0] +
                         (y - (float)c.b_node[wl][1]) * (float)c.b_edge[wl][1]) / len;
    if (wl == ib ? along < slack : along > len - slack) return true;
  }
  return false;
}
__device__ __forceinline__ bool by_a_node(const Consts& c, const MirrorPlan& pl, float x, float y) {
  for (int q = 0; q < pl.nc; ++q) {
    if (pl.ckind[q] == SEL_CORNER_WP) continue;
    const int k = pl.ckind[q] == SEL_CORNER_PP ? c.b_pp[pl.cib[q]] : pl.cib[q];
    const float r1 = x - (float)c.b_node[k][0], r2 = y - (float)c.b_node[k][1];
    if (fmaf(r1, r1, r2 * r2) <= c.near_band * c.near_band) return true;
  }
  return false;
}

// particles of a block: small domains take small blocks, to fill the GPU; large ones fewer of them,
// for the scan by one block (4M particles: 3,907 counts a stage)
inline int mirror_block(int n) { return n > 200000 ? 4 * TPB : TPB; }

template <int IPT>
__global__ void __launch_bounds__(TPB) k_mirror_select(const __grid_constant__ Consts c, const __grid_constant__ Dev d,
                                                       const __grid_constant__ MirrorPlan pl) {
  __shared__ int cnt[MIR_STAGES];
  __shared__ StageTab st;
  __shared__ NearTab t;
  if (threadIdx.x < MIR_STAGES) cnt[threadIdx.x] = 0;
  stage_table(c, pl, st);
  near_table(c, t);
  const int words = (c.npfb + 31) / 32;
  for (int q = 0; q < IPT; ++q) {
    const int it = (blockIdx.x * IPT + q) * TPB + threadIdx.x;
    const int word = it >> 5;
    const bool in = it < c.npfb;
    float x = 0.f, y = 0.f;
    if (in) {
      x = narrow(d.rx[it]);
      y = narrow(d.ry[it]);
    }
    const unsigned near = in ? stages_near(c, pl, st, it, x, y) : 0u;
    for (int s = 0; s < pl.ns; ++s) {
      int n = 0;
      if (pl.kind[s] == SEL_CANDIDATES) n = in && near_boundary(t, x, y) ? 1 : 0;
      else if ((near >> s) & 1u) n = sel_count(c, d, SelArgs{pl.kind[s], pl.ib[s]}, it);
      // plane e of a stage: particles with more than e images in it
      for (int e = 0; e < pl.first_plane[s + 1] - pl.first_plane[s]; ++e) {
        const unsigned b = __ballot_sync(0xffffffffu, n > e);
        if ((threadIdx.x & 31) == 0 && word < words) {
          d.sel_bits[(size_t)(pl.first_plane[s] + e) * words + word] = b;
          if (b) atomicAdd(&cnt[s], __popc(b));
        }
      }
    }
    if (in && it >= c.nbS && by_a_node(c, pl, x, y)) {
      const int k = atomicAdd(&d.s->n_node, 1);
      if (k < MIR_LIST) d.mir_list[MIR_LIST + k] = it;
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < pl.ns) d.sel_blk[threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// exclusive scan in place of the stages' block counts, stage after stage; the total after the last
// one; nmir: entries of the stages that make mirrors
__global__ void __launch_bounds__(1024) k_mirror_scan(Dev d, int n, int nmir, int mcap) {
  __shared__ int sh[32];
  int* const v = d.sel_blk;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = (n + 1023) / 1024, b0 = threadIdx.x * per, b1 = min(n, b0 + per);
  int loc = 0;
  for (int b = b0; b < b1; ++b) loc += v[b];
  int inc = loc;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) sh[w] = inc;
  __syncthreads();
  if (w == 0) {
    int u = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(0xffffffffu, u, o);
      if (lane >= o) u += z;
    }
    sh[lane] = u;
  }
  __syncthreads();
  int run = (w ? sh[w - 1] : 0) + inc - loc;
  for (int b = b0; b < b1; ++b) {
    const int u = v[b];
    v[b] = run;
    run += u;
  }
  if (threadIdx.x == 0) v[n] = sh[31];
  __syncthreads();
  if (threadIdx.x == 0) {
    const int total = nmir < n ? v[nmir] : sh[31];
    if (total > mcap) set_error(d.s, VEBI_ERR_MIRROR_CAPACITY);
    d.s->nmirror = min(total, mcap);
    d.s->n_cand = sh[31] - total;
  }
}

// Mirrors of the stages over particles, a thread per mirror (and per candidate): its stage and block
// from the scan, its particle from the block's selection bits.  So the FP64 work runs on full
// warps; a warp of 32 consecutive particles has a few that are selected, if any.  A mirror of a
// moving solid particle copies its parent's u and theta (mirror_..:191-206).
template <int IPT>
__global__ void __launch_bounds__(TPB) k_mirror_emit(const __grid_constant__ Consts c, const __grid_constant__ Dev d,
                                                     const __grid_constant__ MirrorPlan pl, int nblk) {
  constexpr int W = IPT * TPB / 32;  // words of a block's bits
  const int n = pl.ns * nblk, words = (c.npfb + 31) / 32;
  const int total = d.sel_blk[n], nmir = total - d.s->n_cand;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < total; m += gridDim.x * blockDim.x) {
    int lo = 0, hi = n;  // the last entry that starts at or before m
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (d.sel_blk[mid] <= m) lo = mid;
      else hi = mid;
    }
    const int s = lo / nblk, b = lo % nblk;
    int r = m - d.sel_blk[lo];
    const int p0 = pl.first_plane[s], np = pl.first_plane[s + 1] - p0;
    const unsigned* bits = d.sel_bits + (size_t)p0 * words + b * W;
    int word = 0;
    for (; word < W; ++word) {
      int k = 0;
      for (int e = 0; e < np; ++e) k += __popc(bits[(size_t)e * words + word]);
      if (r < k) break;
      r -= k;
    }
    int bit = 0;
    for (;; ++bit) {
      int k = 0;
      for (int e = 0; e < np; ++e) k += (bits[(size_t)e * words + word] >> bit) & 1u;
      if (r < k) break;
      r -= k;
    }
    const int it = (b * W + word) * 32 + bit;
    if (pl.kind[s] == SEL_CANDIDATES) {
      d.cand[m - nmir] = it;
      continue;
    }
    if (r) continue;  // a particle's images in one stage are emitted together
    int made = 0;
    for (int e = 0; e < np; ++e) made += (bits[(size_t)e * words + word] >> bit) & 1u;
    sel_emit(c, d, SelArgs{pl.kind[s], pl.ib[s]}, it, m);
    for (int e = m; e < m + made && e < c.mcap; ++e) {
      const int j = c.npfb + e;
      if (it < c.nbS) {
        const double u = d.ux[it], v = d.uy[it], th = d.th[it];
        if (u * u + v * v != 0.0) { d.ux[j] = u; d.uy[j] = v; }
        if (th * th != 0.0) d.th[j] = th;
      }
      if (past_wall_end(c, pl, narrow(d.rx[j]), narrow(d.ry[j]))) {
        const int k = atomicAdd(&d.s->n_end, 1);
        if (k < MIR_LIST) d.mir_list[k] = j;
      }
    }
  }
}

// ascending copy of n distinct items (each to its rank), or false when they do not fit
__device__ bool sorted_list(const int* src, int n, int* dst) {
  if (n > MIR_LIST) return false;
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int v = src[e];
    int r = 0;
    for (int k = 0; k < n; ++k) r += src[k] < v ? 1 : 0;
    dst[r] = v;
  }
  return true;
}

// The corners, one after the other, by one block: each takes its items in ascending order -- from
// the lists, or all mirrors or particles if a list overflowed -- and appends its mirrors.  Then np
// and the step's relaxation factor.
__global__ void __launch_bounds__(1024) k_mirror_corners(const __grid_constant__ Consts c, const __grid_constant__ Dev d,
                                                         const __grid_constant__ MirrorPlan pl) {
  __shared__ int ends[MIR_LIST], nodes[MIR_LIST], wsum[32];
  Scal* const s = d.s;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int imp = s->nmirror;
  int n_ends = 0, n_nodes = 0;
  bool all_ends = false, all_nodes = false;
  if (pl.nc) {
    n_ends = s->n_end;
    n_nodes = s->n_node;
    all_ends = !sorted_list(d.mir_list, n_ends, ends);
    all_nodes = !sorted_list(d.mir_list + MIR_LIST, n_nodes, nodes);
    __syncthreads();
  }
  for (int q = 0; q < pl.nc; ++q) {
    const SelArgs a{pl.ckind[q], pl.cib[q]};
    const bool wp = a.kind == SEL_CORNER_WP, all = wp ? all_ends : all_nodes;
    const int total = all ? (wp ? imp : c.npfb - c.nbS) : (wp ? n_ends : n_nodes);
    const int imp0 = imp;  // the mirrors a corner makes are not its own items
    for (int e0 = 0; e0 < total; e0 += 1024) {
      const int e = e0 + threadIdx.x;
      const int it = e >= total ? -1 : all ? (wp ? c.npfb : c.nbS) + e : wp ? ends[e] : nodes[e];
      const bool mine = it >= 0 && sel_count(c, d, a, it) != 0;
      const unsigned b = __ballot_sync(0xffffffffu, mine);
      if (lane == 0) wsum[w] = __popc(b);
      __syncthreads();
      int before = 0, made = 0;
      for (int k = 0; k < 32; ++k) {
        before += k < w ? wsum[k] : 0;
        made += wsum[k];
      }
      if (mine) sel_emit(c, d, a, it, imp + before + __popc(b & ((1u << lane) - 1u)));
      imp += made;
      __syncthreads();
    }
    if (imp > c.mcap) {
      if (threadIdx.x == 0) set_error(s, VEBI_ERR_MIRROR_CAPACITY);
      imp = c.mcap;
    }
    if (!all_ends) {  // the new mirrors are items of the corners that follow
      if (n_ends + imp - imp0 <= MIR_LIST) {
        for (int e = imp0 + threadIdx.x; e < imp; e += 1024) ends[n_ends + e - imp0] = c.npfb + e;
        n_ends += imp - imp0;
      } else {
        all_ends = true;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    s->nmirror = imp;
    s->np = c.npfb + imp;
    s->relax = exp(-(1.0 * 1.0 * s->dt / c.Wi));  // as k_logconf's with alpha_R = 1; dt may be a replayed step's
  }
}

void launch_advect_bin(Ctx& x) {
  const Consts& c = x.c;
  VEBI_LAUNCH(x, k_step_reset, 1, 1, x.d.s, c.npfb, c.nbS);
  VEBI_LAUNCH(x, k_save_umax, grid_for(c.npfb), TPB, c, x.d);
  VEBI_LAUNCH(x, k_advect_bin, grid_for(c.npfb), TPB, c, x.d);
}

// create_mirror_particles (mirror_boundaries_mod.F90:18-334)
void launch_mirrors(Ctx& x) {
  const Consts& c = x.c;
  MirrorPlan pl{};
  auto stage = [&](int kind, int ib, int planes) {
    pl.kind[pl.ns] = (signed char)kind;
    pl.ib[pl.ns] = (signed char)ib;
    pl.first_plane[pl.ns + 1] = pl.first_plane[pl.ns] + planes;
    ++pl.ns;
  };
  auto corner = [&](int kind, int ib) {
    pl.ckind[pl.nc] = (signed char)kind;
    pl.cib[pl.nc++] = (signed char)ib;
  };
  if (c.ncirc > 0) stage(SEL_CIRCLES, 0, c.ncirc);
  for (int ib = 0; ib < c.nb; ++ib) {
    if (c.b_type[ib] == 1) stage(SEL_WALL, ib, 1);
    if (c.b_type[ib] == 2) stage(SEL_PERIODIC, ib, 1);
  }
  const int made = pl.ns;
  if (c.ncirc > 0) stage(SEL_CANDIDATES, 0, 1);
  for (int ib = 0; ib < c.nb; ++ib) {
    int ibm1 = (ib + c.nb - 1) % c.nb;
    if (c.b_type[ib] == 0 || c.b_type[ibm1] == 0) continue;
    double tmp = c.b_edge[ibm1][0] * c.b_edge[ib][1] - c.b_edge[ibm1][1] * c.b_edge[ib][0];
    if (fabs(tmp) < 1e-10) continue;
    if (c.b_type[ib] == 1 && c.b_type[ibm1] == 1 && !(c.b_corner_angle[ib] <= 0.0)) corner(SEL_CORNER_WW, ib);
    if (c.b_type[ib] == 2 && c.b_type[ibm1] == 2) corner(SEL_CORNER_PP, ib);
    if (c.b_type[ib] != c.b_type[ibm1] && (c.b_type[ib] == 1 || c.b_type[ibm1] == 1)) corner(SEL_CORNER_WP, ib);
  }
  const int per = mirror_block(c.npfb), nblk = (c.npfb + per - 1) / per;
  // the emitting grid: a thread per mirror of a domain's usual number, more by striding
  const int emit = nblk < 4 * x.nsm ? (nblk < 8 ? 8 : nblk) : 4 * x.nsm;
  if (per == TPB) VEBI_LAUNCH(x, k_mirror_select<1>, nblk, TPB, c, x.d, pl);
  else VEBI_LAUNCH(x, k_mirror_select<4>, nblk, TPB, c, x.d, pl);
  VEBI_LAUNCH(x, k_mirror_scan, 1, 1024, x.d, pl.ns * nblk, made * nblk, c.mcap);
  if (per == TPB) VEBI_LAUNCH(x, k_mirror_emit<1>, emit, TPB, c, x.d, pl, nblk);
  else VEBI_LAUNCH(x, k_mirror_emit<4>, emit, TPB, c, x.d, pl, nblk);
  VEBI_LAUNCH(x, k_mirror_corners, 1, 1024, c, x.d, pl);
}

// ------------------------------------------------------------------------------- mirror fields
// mirror_velocities (mirror_boundaries_mod.F90:509-584): u* of mirrors from their parents' u*
// (the predictor's output ux2/uy2), then solid-parent copies.
__global__ void k_mirror_velocities(Consts c, Dev d) {
  const int nm = d.s->nmirror;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < nm; m += gridDim.x * blockDim.x) {
    int j = c.npfb + m, i = d.irel[j], vr = d.vrel[j];
    double ui = d.ux2[i], vi = d.uy2[i];
    double uj = d.ux[j], vj = d.uy[j];  // creation-time value (kept if no branch applies)
    if (vr > 999) {
      int ib = vr - 999 - 1;
      double r1 = 0.5 * (d.rx[i] - d.rx[j]), r2 = 0.5 * (d.ry[i] - d.ry[j]);
      double tmp = sqrt(r1 * r1 + r2 * r2);
      double t1 = r2 / tmp, t2 = -r1 / tmp;
      uj = 2.0 * c.c_vel[ib][0] + 2.0 * t1 * c.c_radius[ib] * c.c_omega[ib] - 1.0 * ui;
      vj = 2.0 * c.c_vel[ib][1] + 2.0 * t2 * c.c_radius[ib] * c.c_omega[ib] - 1.0 * vi;
    }
    if (vr > 0 && vr < 999) {
      int ib = vr - 1;
      if (abs(c.b_type[ib]) == 1) {
        double r1 = 0.5 * (d.rx[i] - d.rx[j]), r2 = 0.5 * (d.ry[i] - d.ry[j]);
        double tmp = sqrt(r1 * r1 + r2 * r2);
        double t1 = r2 / tmp, t2 = -r1 / tmp;
        uj = 2.0 * c.b_vel[ib] * t1 - ui;
        vj = 2.0 * c.b_vel[ib] * t2 - vi;
      } else if (c.b_type[ib] == 2) {
        uj = ui;
        vj = vi;
      }
    }
    if (vr < 0 && vr > -c.npfb) {
      int ib = -vr - 1, ibm1 = (ib + c.nb - 1) % c.nb;
      if (c.b_type[ib] == 1 && c.b_type[ibm1] == 1) {
        uj = ui; vj = vi;
        if (c.b_vel[ib] != 0.0) {
          double n1, n2; bound_norm(c, ib, n1, n2);
          double tmp = c.b_vel[ib];
          uj = 2.0 * tmp * n2 - ui;
          vj = 2.0 * tmp * (-n1) - vi;
        }
        if (c.b_vel[ibm1] != 0.0) {
          double n1, n2; bound_norm(c, ibm1, n1, n2);
          double tmp = c.b_vel[ibm1];
          uj = uj + 2.0 * tmp * n2;
          vj = vj + 2.0 * tmp * (-n1);
        }
      } else if (c.b_type[ib] == 2 && c.b_type[ibm1] == 2) {
        uj = ui; vj = vi;
      } else if ((c.b_type[ib] == 1 && c.b_type[ibm1] == 2) || (c.b_type[ib] == 2 && c.b_type[ibm1] == 1)) {
        double tmp = 0.0, t1 = 0.0, t2 = 0.0;
        if (c.b_vel[ib] != 0.0) {
          double n1, n2; bound_norm(c, ib, n1, n2); t1 = n2; t2 = -n1; tmp = c.b_vel[ib];
        } else if (c.b_vel[ibm1] != 0.0) {
          double n1, n2; bound_norm(c, ibm1, n1, n2); t1 = n2; t2 = -n1; tmp = c.b_vel[ibm1];
        }
        uj = 2.0 * tmp * t1 - ui;
        vj = 2.0 * tmp * t2 - vi;
      }
    }
    if (i < c.nbS) {
      double tmp = ui * ui + vi * vi;
      if (tmp != 0.0) { uj = ui; vj = vi; }
    }
    d.ux2[j] = uj;
    d.uy2[j] = vj;
  }
}

// mirror_polymeric_stress (mirror_boundaries_mod.F90:586-653)
__device__ __forceinline__ void reflect_tau(const Dev& d, int i, int j, double n1, double n2) {
  double nt1 = -n2, nt2 = n1;
  double q11 = 1.0 * n1 + 0.0 * n2, q12 = 1.0 * nt1 + 0.0 * nt2;
  double q21 = 0.0 * n1 + 1.0 * n2, q22 = 0.0 * nt1 + 1.0 * nt2;
  double T11 = d.tau[0][i], T21 = d.tau[1][i], T12 = d.tau[2][i], T22 = d.tau[3][i];
  // tmp = Q^T (T Q)
  double a11 = T11 * q11 + T12 * q21, a12 = T11 * q12 + T12 * q22;
  double a21 = T21 * q11 + T22 * q21, a22 = T21 * q12 + T22 * q22;
  double m11 = q11 * a11 + q21 * a21, m12 = q11 * a12 + q21 * a22;
  double m21 = q12 * a11 + q22 * a21, m22 = q12 * a12 + q22 * a22;
  m11 = -m11;
  m12 = -m12;
  // Q (tmp Q^T)
  double b11 = m11 * q11 + m12 * q12, b12 = m11 * q21 + m12 * q22;
  double b21 = m21 * q11 + m22 * q12, b22 = m21 * q21 + m22 * q22;
  d.tau[0][j] = q11 * b11 + q12 * b21;
  d.tau[2][j] = q11 * b12 + q12 * b22;
  d.tau[1][j] = q21 * b11 + q22 * b21;
  d.tau[3][j] = q21 * b12 + q22 * b22;
}

__global__ void k_mirror_stress(Consts c, Dev d) {
  const int nm = d.s->nmirror;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < nm; m += gridDim.x * blockDim.x) {
    int j = c.npfb + m, i = d.irel[j], vr = d.vrel[j];
    if (vr > 999) {
      double r1 = d.rx[i] - d.rx[j], r2 = d.ry[i] - d.ry[j];
      double nn = sqrt(r1 * r1 + r2 * r2);
      reflect_tau(d, i, j, r1 / nn, r2 / nn);
    }
    if (vr > 0 && vr < 999) {
      int ib = vr - 1;
      if (c.b_type[ib] == 1) {
        double r1 = d.rx[i] - d.rx[j], r2 = d.ry[i] - d.ry[j];
        double nn = sqrt(r1 * r1 + r2 * r2);
        reflect_tau(d, i, j, r1 / nn, r2 / nn);
      } else if (c.b_type[ib] == 2 || c.b_type[ib] == 4) {
        for (int q = 0; q < 4; ++q) d.tau[q][j] = d.tau[q][i];
      } else if (c.b_type[ib] == 3) {
        for (int q = 0; q < 4; ++q) d.tau[q][j] = 0.0;
      }
    }
    if (vr < 0 && vr > -c.npfb) {
      int ib = -vr - 1, ibm1 = (ib + c.nb - 1) % c.nb;
      if (c.b_type[ib] == 1 && c.b_type[ibm1] == 1) {
        for (int q = 0; q < 4; ++q) d.tau[q][j] = -d.tau[q][i];
      } else if (c.b_type[ib] == 2 && c.b_type[ibm1] == 2) {
        for (int q = 0; q < 4; ++q) d.tau[q][j] = d.tau[q][i];
      } else if ((c.b_type[ib] == 1 && c.b_type[ibm1] == 2) || (c.b_type[ib] == 2 && c.b_type[ibm1] == 1)) {
        double n1, n2;
        if (c.b_type[ib] == 1) bound_norm(c, ib, n1, n2);
        else bound_norm(c, ibm1, n1, n2);
        reflect_tau(d, i, j, n1, n2);
      }
    }
  }
}

// grad_operator mirror transfer for the three gradients (gradient_calculation.F90:96-145).
// Circle mirrors keep 0: the reference tests vrelation == 999 while circles carry 999+ib.
__global__ void k_grad_mirrors(Consts c, Dev d) {
  const int nm = d.s->nmirror;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < nm; m += gridDim.x * blockDim.x) {
    int j = c.npfb + m, i = d.irel[j], vr = d.vrel[j];
    int mode = 0;  // 0 none, 1 reflect, 2 reflect normal-zero, 3 copy, 4 negate, 5 rotate
    double r1 = 0, r2 = 0;
    if (vr > 0 && vr < 999) {
      int ib = vr - 1;
      if (c.b_type[ib] == 2) mode = 5;
      else if (c.b_type[ib] == 3) mode = 3;
      else if (c.b_type[ib] == 1) { mode = 1; r1 = d.rx[i] - d.rx[j]; r2 = d.ry[i] - d.ry[j]; }
      else if (c.b_type[ib] == 4) { mode = 2; r1 = d.rx[i] - d.rx[j]; r2 = d.ry[i] - d.ry[j]; }
    } else if (vr < 0 && vr > -c.npfb) {
      int ib = -vr - 1, ibm1 = (ib + c.nb - 1) % c.nb;
      if (c.b_type[ib] == 1 && c.b_type[ibm1] == 1) mode = 4;
      else if (c.b_type[ib] == 2 && c.b_type[ibm1] == 2) mode = 3;
      else if ((c.b_type[ib] == 1 && c.b_type[ibm1] == 2) || (c.b_type[ib] == 2 && c.b_type[ibm1] == 1)) {
        mode = 1;
        if (c.b_type[ib] == 1) { r1 = -1.0 * c.b_edge[ib][1]; r2 = c.b_edge[ib][0]; }
        else { r1 = -1.0 * c.b_edge[ibm1][1]; r2 = c.b_edge[ibm1][0]; }
      }
    }
    if (mode == 0) {  // no branch of the reference applies: the gradient stays 0
      for (int f = 0; f < 6; ++f) d.grad[f][j] = 0.0;
      continue;
    }
    for (int f = 0; f < 3; ++f) {
      double g1 = d.grad[2 * f][i], g2 = d.grad[2 * f + 1][i], o1, o2;
      if (mode == 3) { o1 = g1; o2 = g2; }
      else if (mode == 4) { o1 = -g1; o2 = -g2; }
      else if (mode == 5) {
        const double* Q = c.b_rot[vr - 1];
        o1 = Q[0] * g1 + Q[1] * g2;
        o2 = Q[2] * g1 + Q[3] * g2;
      } else {
        double nn = sqrt(r1 * r1 + r2 * r2);
        double q11 = r1 / nn, q21 = r2 / nn, q12 = -q21, q22 = q11;
        double b1 = q11 * g1 + q12 * g2, b2 = q21 * g1 + q22 * g2;
        if (mode == 2) b1 = 0.0; else b2 = -b2;
        o1 = q11 * b1 + q21 * b2;
        o2 = q12 * b1 + q22 * b2;
      }
      d.grad[2 * f][j] = o1;
      d.grad[2 * f + 1][j] = o2;
    }
  }
}

// mirror pressure P_j = P_parent + dP_mp (gradient_calculation.F90:26-30)
__global__ void k_mirror_pressure(Consts c, Dev d) {
  const int nm = d.s->nmirror;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < nm; m += gridDim.x * blockDim.x) {
    int j = c.npfb + m;
    d.p[j] = d.p[d.irel[j]] + d.dP_mp[j];
  }
}

void launch_mirror_velocities(Ctx& x) { VEBI_LAUNCH(x, k_mirror_velocities, x.gs_blocks, TPB, x.c, x.d); }
void launch_mirror_stress(Ctx& x) { VEBI_LAUNCH(x, k_mirror_stress, x.gs_blocks, TPB, x.c, x.d); }
void launch_grad_mirrors(Ctx& x) { VEBI_LAUNCH(x, k_grad_mirrors, x.gs_blocks, TPB, x.c, x.d); }
void launch_mirror_pressure(Ctx& x) { VEBI_LAUNCH(x, k_mirror_pressure, x.gs_blocks, TPB, x.c, x.d); }

}  // namespace vebi
