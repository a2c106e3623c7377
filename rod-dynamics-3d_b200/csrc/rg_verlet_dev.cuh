// rg_verlet_dev.cuh - device bodies of the velocity-Verlet step shared by the
// multi-kernel form (rg_forces.cu, rg_integrate.cu) and the persistent one
// (rg_verlet.cu): the contact force laws and the per-rod kicks and drift.
#pragma once
#include "rg_nsc_dev.cuh"

namespace rg {

__device__ inline unsigned long long pkey(int a, int b) {
  return ((unsigned long long)(unsigned)a << 32) | (unsigned long long)(unsigned)b;
}
__device__ inline int lower_bound_u64(const unsigned long long* k, int n, unsigned long long v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int m = (lo + hi) >> 1;
    if (k[m] < v) lo = m + 1;
    else hi = m;
  }
  return lo;
}

// ---- contact forces ----------------------------------------------------------
// What one contact gives: force and torque addends of both bodies, the new
// tangential-history value (touch: the entry is written), potential energy.
struct PairForce {
  d3 fa, ta, fb, tb, hist;
  double pe;
  int touch;
};
__device__ inline void store_addends(double* cf, int cc, int c, const PairForce& p) {
  cf[c] = p.fa.x; cf[cc + c] = p.fa.y; cf[2 * cc + c] = p.fa.z;
  cf[3 * cc + c] = p.ta.x; cf[4 * cc + c] = p.ta.y; cf[5 * cc + c] = p.ta.z;
  cf[6 * cc + c] = p.fb.x; cf[7 * cc + c] = p.fb.y; cf[8 * cc + c] = p.fb.z;
  cf[9 * cc + c] = p.tb.x; cf[10 * cc + c] = p.tb.y; cf[11 * cc + c] = p.tb.z;
}

// What the force laws read of the two bodies.
struct PairIn {
  d3 xa, xb, va, wa, vb, wb;
  double ra, rb, ma, mb;  // radii and masses (0: static body)
};
__device__ inline PairIn load_pair(const State& st, int a, int b) {
  return PairIn{st.x.ld(a), st.x.ld(b), st.v.ld(a), st.w.ld(a), st.v.ld(b), st.w.ld(b),
                st.r[a],    st.r[b],    st.mass[a], st.mass[b]};
}

// Soft penalty contact (SoftContactSolver::computeForces,
// src/physics/soft_contact.cpp:80-486); old: the pair's history value;
// energy: the potential energy is wanted.
__device__ inline PairForce soft_pair(const PairIn& in, const rg_config& cfg, d3 pa, d3 pb, d3 nrm, d3 sh, double dist,
                                      double hs, d3 old, bool energy) {
  const double dt = cfg.dt;
  const double K1 = 15.0 / cfg.soft_delta;
  // potentialGradient / potentialEnergy
  double grad, U;
  if (dist > hs - cfg.soft_delta) {
    double arg = K1 * (hs - dist);
    double e = exp(arg);
    double lt = log(1.0 + e);
    grad = -2.0 / (K1 * K1) * lt * e / (1.0 + e);
    double base = lt / K1;
    U = base * base;
  } else {
    grad = -2.0 * (hs - dist);
    double pen = hs - dist;
    U = pen * pen;
  }
  double fm = -cfg.soft_k_scaler * grad;
  d3 fa = nrm * (-fm);
  d3 fb = nrm * fm;
  d3 ra = pa - in.xa;
  d3 rb = pb - (in.xb + sh);
  d3 va = in.va + cross(in.wa, ra);
  d3 vb = in.vb + cross(in.wb, rb);
  d3 vrel = va - vb;
  if (cfg.soft_damping > 1e-9) {
    double vn = dot(vrel, nrm);
    d3 fd = nrm * (-cfg.soft_damping * vn);
    fa = fa + fd;
    fb = fb - fd;
  }
  d3 fra{0, 0, 0};
  int touch = 0;
  d3 nv{0, 0, 0};
  if (cfg.soft_enable_friction) {
    double fn_mag = len(fa);
    d3 vt = vrel - nrm * dot(vrel, nrm);
    double vtm = len(vt);
    if (!(vtm < 1e-10)) {
      if (cfg.soft_friction_mode == RG_FRICTION_CUNDALL) {
        d3 ft = old - vt * (cfg.soft_kt * dt);
        double ncmp = dot(ft, nrm);
        ft = ft - nrm * ncmp;
        double ftm = len(ft);
        double lim = cfg.soft_mu * fn_mag;
        if (ftm > lim) {
          if (ftm > 1e-8) ft = ft * (lim / ftm);
          else ft = mk3(0, 0, 0);
        }
        nv = ft;
        touch = 1;
        fra = ft;
      } else if (cfg.soft_friction_mode == RG_FRICTION_KARNOPP) {
        if (vtm < cfg.soft_vel_deadband) {
          const double ma = in.ma;
          const double mb = in.mb;
          double meff = 0;
          if (ma > 0 && mb > 0) meff = (ma * mb) / (ma + mb);
          else if (ma > 0) meff = ma;
          else if (mb > 0) meff = mb;
          d3 fstop = vt * (-(meff / dt));
          d3 gv{cfg.gravity[0], cfg.gravity[1], cfg.gravity[2]};
          d3 gt = gv - nrm * dot(gv, nrm);
          d3 fdrive = gt * meff;
          d3 freq = fstop - fdrive;
          double frm = len(freq);
          double maxs = cfg.soft_mu_static * fn_mag;
          if (frm <= maxs) fra = freq;
          else if (frm > 1e-12) fra = freq * (maxs / frm);
        } else {
          fra = (vt * -1.0 / vtm) * (cfg.soft_mu * fn_mag);
        }
      } else {
        double K2 = 15.0 / cfg.soft_nu;
        double gamma = vtm > cfg.soft_nu ? 1.0 : 2.0 / (1.0 + exp(-K2 * vtm)) - 1.0;
        double mu_eff = cfg.soft_mu;
        if (cfg.soft_mu_static > cfg.soft_mu)
          mu_eff = cfg.soft_mu + (cfg.soft_mu_static - cfg.soft_mu) * exp(-vtm / cfg.soft_nu);
        d3 dir = (-vt) / vtm;
        fra = dir * (mu_eff * gamma * fn_mag);
      }
    }
  }
  d3 ta = fa + fra, tb = fb - fra;
  return PairForce{ta, cross(ra, ta), tb, cross(rb, tb), nv, energy ? cfg.soft_k_scaler * U : 0.0, touch};
}

// Hertz-Mindlin contact on capsules (src/physics/hertz_mindlin.cpp:249-383);
// old: the pair's tangential spring.
struct HmConst {
  double Es, Gs, gam;
};
__device__ inline HmConst hm_const(const rg_config& cfg) {
  const double nu = cfg.hm_poisson_ratio;
  HmConst k;
  k.Es = cfg.hm_youngs_modulus / (2.0 * (1.0 - nu * nu));
  k.Gs = cfg.hm_youngs_modulus / (2.0 * (1.0 + nu));
  k.gam = 0.0;
  if (cfg.hm_restitution < 1.0) {
    double l = log(cfg.hm_restitution);
    k.gam = -l / sqrt(M_PI * M_PI + l * l);
  }
  return k;
}
__device__ inline PairForce hm_pair(const PairIn& in, const rg_config& cfg, const HmConst& k, d3 pa, d3 pb, d3 nrm,
                                    d3 sh, double dist, double hs, d3 old, bool energy) {
  const double dt = cfg.dt, Es = k.Es, Gs = k.Gs, gam = k.gam;
  const double ra_ = in.ra, rb_ = in.rb, ma = in.ma, mb = in.mb;
  double delta = hs - dist;
  double Rs = (ra_ * rb_) / (ra_ + rb_);
  double ms = (ma * mb) / (ma + mb);
  double sd = smax(delta, 0.0);
  double sqd = sqrt(sd);
  double sqR = sqrt(smax(Rs, 0.0));
  double kn = (4.0 / 3.0) * Es * sqR * sqd;
  double Fel = kn * sd * sqd;
  d3 ra = pa - in.xa;
  d3 rb = pb - (in.xb + sh);
  const d3 wa = in.wa, wb = in.wb;
  d3 va = in.va + cross(wa, ra);
  d3 vb = in.vb + cross(wb, rb);
  d3 vrel = vb - va;
  double vn = dot(vrel, nrm);
  double Cn = gam * 2.0 * sqrt(ms * kn);
  double Fn = smax(0.0, Fel + (-Cn * vn));
  d3 fn = nrm * Fn;
  d3 ft{0, 0, 0};
  d3 xi = old;
  if (cfg.hm_enable_tangential) {
    double kt = 8.0 * Gs * sqR * sqd;
    d3 vt = vrel - nrm * vn;
    xi = xi + vt * dt;
    d3 fel = xi * (-kt);
    double Ct = gam * 2.0 * sqrt(ms * kt);
    ft = fel - vt * Ct;
    double vtm = len(vt);
    double mu_eff = cfg.hm_friction;
    if (cfg.hm_friction_static > cfg.hm_friction && cfg.hm_friction_transition_vel > 0.0)
      mu_eff += (cfg.hm_friction_static - cfg.hm_friction) * exp(-vtm / cfg.hm_friction_transition_vel);
    double fnm = len(fn);
    double ftm = len(ft);
    double ftmax = mu_eff * fnm;
    if (ftm > ftmax && ftm > 1e-10) {
      ft = ft * (ftmax / ftm);
      if (kt > 1e-10) xi = ft / (-kt);
    }
  }
  d3 tra{0, 0, 0}, trb{0, 0, 0};
  if (cfg.hm_enable_rolling) {
    d3 wr = wa - wb;
    double wm = len(wr);
    if (!(wm < 1e-10)) {
      d3 wh = wr / wm;
      double trm = cfg.hm_rolling_friction * Rs * len(fn);
      d3 tr = wh * (-trm);
      tra = tr * 0.5;
      trb = tr * -0.5;
    }
  }
  d3 F = fn + ft;
  return PairForce{-F, cross(ra, -F) + tra, F, cross(rb, F) + trb, xi,
                   energy ? (8.0 / 15.0) * Es * sqrt(Rs) * pow(delta, 2.5) : 0.0, 1};
}

// Everything a team needs to step one system (device copy per system).
struct VerletView {
  NscView v;  // state, box, configuration, detector, contacts
  int *near_cnt, *near_nbr;  // near lists; null: the full lists
  double extra;              // near-list reach beyond r_a + r_b
  double delta;              // activation margin of the detection
  double* cf;                // force addends (12) and potential energy, ccap each
  unsigned long long* hkey[2];
  double* hval[2];
  long long* hframe[2];
  int hcap, hcur;
  int *touched, *touched_off, *kept, *kept_off;
  double* newval;
  int *first[2], *hidx[2], *head, *next, *ins;  // VerletTeam
  int2 *pk[2], *flat;
  int flat_cap;
  int fresh, cb;  // 1: contacts, indices and lists of buffer cb are current
};
VerletView make_verlet_view(rg_system* s);
void verlet_launch(const VerletView* views, const TeamDesc* teams, int nteams, const int* members, int grid, int nsteps,
                   cudaStream_t st);

// ---- per-rod integrators -------------------------------------------------------
// Iinv = 1/I per principal axis for a dynamic body (0 when I = 0), as the
// state's stored inverse (rg_set_bodies), recomputed here to save its load.
__device__ inline d3 ang_accel(const State& st, int i, dq q, d3 w, d3 tau) {
  const d3 I = st.I.ld(i);
  const d3 Iinv{I.x > 0.0 ? 1.0 / I.x : 0.0, I.y > 0.0 ? 1.0 / I.y : 0.0, I.z > 0.0 ? 1.0 / I.z : 0.0};
  d3 Iw_w = rot_diag_apply(q, I, w);
  d3 gyro = cross(w, Iw_w);
  return rot_diag_apply(q, Iinv, tau - gyro);
}

__device__ inline void rotate_by_omega(dq& q, d3 w, double dt) {
  double wl = len(w);
  if (wl > 1e-8) {
    double ang = wl * dt;
    d3 ax = w / wl;
    q = qnormalize(qmul(angle_axis(ang, ax), q));
  }
}

struct DriftOut {
  Seg* seg;           // segment records of the drifted positions (n)
  const double* ref;  // list reference segments (6n), or null: no check
  const double* ref2; // near-list reference segments (6n), or null
  double skin;
};
// First half kick and drift of rod i under the summed force f and torque t
// (integrateHalfPos, src/physics/integrator.cpp:113-134; wall: the soft
// cylinder wall about axis ax), its segment record and, with a list reference,
// the displacement bounds (invL: 1 / box side, 1 where there is none).
__device__ inline void drift_rod(const State& st, const Box& box, const rg_config& cfg, d3 ax, int wall, int i, d3 f,
                                 d3 t, const DriftOut& o, const double* invL, double& m, double& m2) {
  const d3 g{cfg.gravity[0], cfg.gravity[1], cfg.gravity[2]};
  const double dt = cfg.dt, hdt = 0.5 * cfg.dt;
  d3 x = st.x.ld(i);
  dq q = st.q.ld(i);
  if (st.inv_mass[i] > 0.0) {
    d3 v = st.v.ld(i), w = st.w.ld(i);
    if (wall) soft_wall_apply(cfg, ax, st.r[i], x, v, f);
    d3 al = f / st.mass[i] + g;
    d3 aa = ang_accel(st, i, q, w, t);
    v = v + al * hdt;
    w = w + aa * hdt;
    x = x + v * dt;
    wrap_pos(box, x);
    rotate_by_omega(q, w, dt);
    st.v.st(i, v);
    st.w.st(i, w);
    st.x.st(i, x);
    st.q.st(i, q);
  }
  const Seg sg = seg_of(x, q, st.h[i], st.r[i]);
  o.seg[i] = sg;
  const int n = st.n;
  auto bound = [&](const double* ref) {  // non-finite state: 1e300 forces a rebuild
    const double rf[6] = {ref[i], ref[n + i], ref[2 * n + i], ref[3 * n + i], ref[4 * n + i], ref[5 * n + i]};
    return disp_from(sg, rf, box, invL);
  };
  if (o.ref) m = fmax(m, bound(o.ref));
  if (o.ref2) m2 = fmax(m2, bound(o.ref2));
}

// Second half kick of rod i (integrateSecondHalf, integrator.cpp:136-159);
// el, ea: the damping factors.  f comes back with the wall's part.  Returns 1
// when the new velocity is not a number.
__device__ inline int kick_rod(const State& st, const rg_config& cfg, d3 ax, int wall, int i, d3& f, d3 t, double el,
                               double ea) {
  if (!(st.inv_mass[i] > 0.0)) return 0;
  const d3 g{cfg.gravity[0], cfg.gravity[1], cfg.gravity[2]};
  const double hdt = 0.5 * cfg.dt;
  dq q = st.q.ld(i);
  d3 v = st.v.ld(i), w = st.w.ld(i);
  if (wall) soft_wall_apply(cfg, ax, st.r[i], st.x.ld(i), v, f);
  d3 al = f / st.mass[i] + g;
  d3 aa = ang_accel(st, i, q, w, t);
  v = v + al * hdt;
  w = w + aa * hdt;
  if (cfg.lin_damp > 0.0) v = v * el;
  if (cfg.ang_damp > 0.0) w = w * ea;
  double wl = len(w);
  if (wl > cfg.w_max) w = w * (cfg.w_max / wl);
  st.v.st(i, v);
  st.w.st(i, w);
  return (v.x == v.x && v.y == v.y && v.z == v.z) ? 0 : 1;
}

}  // namespace rg
