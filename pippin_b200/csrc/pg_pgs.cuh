// Projected Gauss-Seidel (crates/pippin/src/solver.rs:38-289) for one env,
// run by the Newton-phase kernel of models whose solver is PGS (pgs_kernel).
//
// Rows follow the reference's order: [normal, tangent 1, tangent 2] per
// contact (every contact of the narrow phase, not only touching ones), then
// the joint-limit sides within reach, then the joint equalities.
//
// Gauss-Seidel is sequential over rows, but rows of separate islands (trees
// joined by rows) share no velocity. Two ways give the sequential sweep's
// result to the bit:
//   pgs_tile: the tile takes every row in turn, each lane forming J_r . v
//     itself and then one dof of the update, the next row's record on its way;
//   pgs_lanes: each lane sweeps islands of its own, in row order, and the tile
//     meets once a sweep for the largest change. Only the entries of the one
//     or two trees that a row touches are formed and read (PR_SPAN), the
//     others are zero; a row's numbers sit in one 128-byte line, prefetched a
//     row ahead, the tree's velocities in registers.
// A row on a lane takes longer than one on the tile, so lanes pay where no
// lane has more than half of the contacts, and there are three trees or more.
// Us a substep of 512 envs, every row on the tile with its whole J / on lanes /
// now: Ant 669 / 1196 / 616, a box 95 / 111 / 89, two stacked 631 / 1127 / 591,
// three 913 / 1476 / 881, six 5100 / 6430 / 3030, three beside one 1213 / 1612 /
// 1260, two beside two 1245 / 1069 / 1021, four apart 1197 / 255, eight 8590 /
// 965. What bounds both is the chain of one row's loads and sums after another.
#pragma once
#include "pg_newton.cuh"

namespace pg {

constexpr double PGS_MAX_BIAS_VELOCITY = 1.0;  // solver.rs:34
constexpr double PGS_TOLERANCE = 1e-5;         // solver.rs:36
constexpr double PGS_MATCH_DIST2 = 0.01 * 0.01;  // solver.rs:255
// dofs up to which a row on the tile runs over all of them: reading its span
// first costs more than the zeros up to 24 dofs (a stack of two boxes beside
// two 1.07 times as long, of three beside one 1.14), less from 36 on (0.6 to
// 0.95)
constexpr int PGS_DENSE_NV = 24;

// The dof ranges [a0, a1) and [b0, b1) a row touches (one tree, or two in
// ascending order), packed in its record's PR_SPAN.
struct Span {
  int a0, a1, b0, b1;
  __device__ bool has(int k) const { return (k >= a0 && k < a1) || (k >= b0 && k < b1); }
  __device__ static Span of(double v) {
    unsigned u = (unsigned)v;
    return Span{(int)(u & 127), (int)(u >> 7 & 127), (int)(u >> 14 & 127), (int)(u >> 21 & 127)};
  }
};
// the tree of a body's dofs, or -1
__device__ inline int body_tree(const DModel& m, int b) {
  unsigned long long mk = m.body_dofmask[b];
  return mk ? m.dof_block[__ffsll((long long)mk) - 1] : -1;
}
// of trees t1 and t2 (-1: none)
__device__ inline double pack_span(const DModel& m, int t1, int t2) {
  if (t1 == t2) t2 = -1;
  if (t1 < 0 || (t2 >= 0 && t2 < t1)) {
    int t = t1;
    t1 = t2;
    t2 = t;
  }
  unsigned u = 0;
  if (t1 >= 0) u |= (unsigned)m.block_adr[2 * t1] | (unsigned)m.block_adr[2 * t1 + 1] << 7;
  if (t2 >= 0) u |= (unsigned)m.block_adr[2 * t2] << 14 | (unsigned)m.block_adr[2 * t2 + 1] << 21;
  return (double)u;
}
__device__ __forceinline__ void prefetch_row(const double* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// f(k) for the span's dofs in ascending order
template <class F>
__device__ __forceinline__ void span_each(const Span& s, F f) {
  for (int k = s.a0; k < s.a1; k++) f(k);
  for (int k = s.b0; k < s.b1; k++) f(k);
}

// Rows of the PGS problem (solver.rs:63-163) into J (stride nv) and R
// (PR_* records). Returns the row count, capped at maxrows. SPANS: PR_SPAN is
// set and only the entries within it are written.
template <int G, bool SPANS>
__device__ int pgs_rows(const Tile<G>& T, const DModel& m, const WsLayout& w, const EnvCtx& e, int ncon,
                        const double* v, double* J, double* R, int* status) {
  int lane = T.lane(), nv = m.nv;
  const double* ws = e.ws;
  const double* prm = e.prm;
  const double* con = e.con;
  const double* cdof = ws + w.cdof;
  int ncrow = 3 * ncon;
  if (ncrow > m.maxrows) {
    *status |= ST_CAP_EXCEEDED;
    ncrow = m.maxrows / 3 * 3;
  }
  int nc = ncrow / 3;
  // contact rows: records, then one Jacobian item per (contact, dof)
  for (int c = lane; c < nc; c += G) {
    const double* r = con + C_STRIDE * c;
    int g1 = (int)r[C_G1], g2 = (int)r[C_G2];
    double mu = fmax(prm[m.p_friction + g1], prm[m.p_friction + g2]);
    double span = SPANS ? pack_span(m, body_tree(m, m.geom_body[g1]), body_tree(m, m.geom_body[g2])) : 0.0;
    for (int q = 0; q < 3; q++) {
      double* rr = R + PR_STRIDE * (3 * c + q);
      rr[PR_KIND] = q == 0 ? PK_NORMAL : PK_FRICTION;
      rr[PR_SEP] = q == 0 ? -r[C_DEPTH] : 0.0;
      rr[PR_MU] = q == 0 ? 0.0 : mu;
      rr[PR_NORMAL] = 3 * c;
      rr[PR_CONTACT] = c;
      rr[PR_INVA] = 0.0;
      rr[PR_LAMBDA] = 0.0;
      if (SPANS) rr[PR_SPAN] = span;
    }
  }
  if (SPANS) T.sync();
  const int per = SPANS ? 2 * m.maxbs : nv;  // dofs looked at a contact
  for (int it = lane; it < nc * per; it += G) {
    int c = it / per, k = it % per;
    if (SPANS) {
      Span sp = Span::of(R[PR_STRIDE * 3 * c + PR_SPAN]);
      const bool second = k >= m.maxbs;
      k = second ? sp.b0 + k - m.maxbs : sp.a0 + k;
      if (k >= (second ? sp.b1 : sp.a1)) continue;
    }
    const double* r = con + C_STRIDE * c;
    int b1 = m.geom_body[(int)r[C_G1]], b2 = m.geom_body[(int)r[C_G2]];
    V3 p = ld3(r + C_POS);
    J[(3 * c + 0) * nv + k] = pair_jac(m, cdof, b1, b2, p, ld3(r + C_NORMAL), k);
    J[(3 * c + 1) * nv + k] = pair_jac(m, cdof, b1, b2, p, ld3(r + C_T1), k);
    J[(3 * c + 2) * nv + k] = pair_jac(m, cdof, b1, b2, p, ld3(r + C_T2), k);
  }
  // joint-limit sides within reach (solver.rs:115-139)
  int nl = 0;
  for (int base = 0; base < m.njnt; base += G) {
    int j = base + lane;
    int cnt = 0, da = 0;
    double sep[2] = {0.0, 0.0};
    bool hit[2] = {false, false};
    if (j < m.njnt && m.jnt_limited[j] && (m.jnt_type[j] == JNT_HINGE || m.jnt_type[j] == JNT_SLIDE)) {
      double q = ws[w.qpos + m.jnt_qposadr[j]];
      da = m.jnt_dofadr[j];
      double reach = m.margin + 2.0 * m.timestep * fabs(v[da]);
      sep[0] = q - m.jnt_range[2 * j];
      sep[1] = m.jnt_range[2 * j + 1] - q;
      for (int t = 0; t < 2; t++) {
        hit[t] = sep[t] < reach;
        cnt += hit[t] ? 1 : 0;
      }
    }
    int tot;
    int off = T.excl_scan(cnt, &tot);
    int row = ncrow + nl + off;
    for (int t = 0; t < 2; t++) {
      if (!hit[t]) continue;
      if (row < m.maxrows) {
        double* jr = J + row * nv;
        double* rr = R + PR_STRIDE * row;
        if (SPANS) rr[PR_SPAN] = pack_span(m, m.dof_block[da], -1);
        span_each(SPANS ? Span::of(rr[PR_SPAN]) : Span{0, nv, 0, 0}, [&](int k) { jr[k] = 0.0; });
        jr[da] = t == 0 ? 1.0 : -1.0;
        rr[PR_KIND] = PK_NORMAL;
        rr[PR_SEP] = sep[t];
        rr[PR_MU] = 0.0;
        rr[PR_NORMAL] = -1.0;
        rr[PR_CONTACT] = -1.0;
        rr[PR_INVA] = 0.0;
        rr[PR_LAMBDA] = 0.0;
      }
      row++;
    }
    nl += tot;
  }
  int nineq = ncrow + nl;
  // joint equalities (solver.rs:141-162)
  for (int q = lane; q < m.neq; q += G) {
    int row = nineq + q;
    if (row >= m.maxrows) continue;
    int j1 = m.eq_j1[q], j2 = m.eq_j2[q];
    const double* c = m.eq_poly + 5 * q;
    double q1 = ws[w.qpos + m.jnt_qposadr[j1]] - m.qpos0[m.jnt_qposadr[j1]];
    double* jr = J + row * nv;
    double* rr = R + PR_STRIDE * row;
    if (SPANS) rr[PR_SPAN] = pack_span(m, m.dof_block[m.jnt_dofadr[j1]], j2 != -1 ? m.dof_block[m.jnt_dofadr[j2]] : -1);
    span_each(SPANS ? Span::of(rr[PR_SPAN]) : Span{0, nv, 0, 0}, [&](int k) { jr[k] = 0.0; });
    jr[m.jnt_dofadr[j1]] += 1.0;
    double poly = c[0];
    if (j2 != -1) {
      double x = ws[w.qpos + m.jnt_qposadr[j2]] - m.qpos0[m.jnt_qposadr[j2]];
      poly = c[0] + x * (c[1] + x * (c[2] + x * (c[3] + x * c[4])));
      jr[m.jnt_dofadr[j2]] -= c[1] + x * (2.0 * c[2] + x * (3.0 * c[3] + x * 4.0 * c[4]));
    }
    rr[PR_KIND] = PK_BILATERAL;
    rr[PR_SEP] = q1 - poly;
    rr[PR_MU] = 0.0;
    rr[PR_NORMAL] = -1.0;
    rr[PR_CONTACT] = -1.0;
    rr[PR_INVA] = 0.0;
    rr[PR_LAMBDA] = 0.0;
  }
  int nr = nineq + m.neq;
  if (nr > m.maxrows) {
    *status |= ST_CAP_EXCEEDED;
    nr = m.maxrows;
  }
  T.sync();
  return nr;
}

// x <- (L L')^-1 x for one right-hand side, by one lane, on the dofs [s0, s1)
// of a tree, with the reference's operations (math.rs:451-463: row-oriented
// forward sweep dividing by the pivot, then column-oriented backward sweep).
__device__ __forceinline__ void tree_mass_solve(int s0, int s1, int nv, const double* L, double* x) {
  for (int i = s0; i < s1; i++) x[i] = (x[i] - dot_ref(L + i * nv + s0, 1, x + s0, 1, i - s0)) / L[i * nv + i];
  for (int i = s1 - 1; i >= s0; i--) {
    x[i] /= L[i * nv + i];
    double xi = -x[i];
    for (int k = s0; k < i; k++) x[k] += xi * L[i * nv + k];
  }
}

// The warm start (solver.rs:254-289): the nearest previous contact of the same
// geom pair within 1 cm lends its impulses, the tangent ones re-projected on
// the new frame.
template <int G>
__device__ __forceinline__ void pgs_lend(const Tile<G>& T, const double* con, int nc, const double* prev, int np, double* R) {
  for (int c = T.lane(); c < nc; c += G) {
    const double* cr = con + C_STRIDE * c;
    double g1 = cr[C_G1], g2 = cr[C_G2];
    V3 pos = ld3(cr + C_POS);
    double bd = PGS_MATCH_DIST2;
    int bi = -1;
    for (int p = 0; p < np; p++) {
      const double* pr = prev + P_STRIDE * p;
      if (pr[P_G1] == g1 && pr[P_G2] == g2) {
        V3 dp = ld3(pr + P_POS) - pos;
        double d2 = dot(dp, dp);
        if (d2 < bd) {
          bd = d2;
          bi = p;
        }
      }
    }
    if (bi != -1) {
      const double* pr = prev + P_STRIDE * bi;
      V3 f = ld3(pr + P_T1) * pr[P_LAMBDA + 1] + ld3(pr + P_T2) * pr[P_LAMBDA + 2];
      R[PR_STRIDE * (3 * c) + PR_LAMBDA] = pr[P_LAMBDA];
      R[PR_STRIDE * (3 * c + 1) + PR_LAMBDA] = dot(f, ld3(cr + C_T1));
      R[PR_STRIDE * (3 * c + 2) + PR_LAMBDA] = dot(f, ld3(cr + C_T2));
    }
  }
}
// this step's contacts and impulses for the next warm start
template <int G>
__device__ __forceinline__ void pgs_keep(const Tile<G>& T, const double* con, int nc, double* prev, int32_t* prev_ncon,
                                         const double* R) {
  for (int c = T.lane(); c < nc; c += G) {
    const double* cr = con + C_STRIDE * c;
    double* pr = prev + P_STRIDE * c;
    for (int q = 0; q < 3; q++) {
      pr[P_POS + q] = cr[C_POS + q];
      pr[P_T1 + q] = cr[C_T1 + q];
      pr[P_T2 + q] = cr[C_T2 + q];
      pr[P_LAMBDA + q] = R[PR_STRIDE * (3 * c + q) + PR_LAMBDA];
    }
    pr[P_G1] = cr[C_G1];
    pr[P_G2] = cr[C_G2];
  }
  if (T.lane() == 0) *prev_ncon = nc;
  T.sync();
}

// What a row's new impulse needs besides the row (solver.rs:44-50).
struct PgsBias {
  double h, slop, rate, mass_scale, impulse_scale;
};
__device__ __forceinline__ PgsBias pgs_bias(const DModel& m) {
  double omega = 2.0 * M_PI * m.hertz;
  double a1 = 2.0 * m.dampratio + m.timestep * omega;
  double a2 = m.timestep * omega * a1;
  double a3 = 1.0 / (1.0 + a2);
  return PgsBias{m.timestep, m.slop, omega / a1, a2 * a3, a3};
}
// A row's new impulse from its J . v (solver.rs:164-215). sep(): its
// separation; bound(): mu times its contact's normal impulse.
template <class S, class B>
__device__ __forceinline__ double pgs_impulse(const PgsBias& c, int kind, double jv, double lam, double inv_a,
                                              bool use_bias, S sep, B bound) {
  if (kind == PK_NORMAL) {
    double sl = sep() + c.slop;
    double bias = 0.0, ms = 1.0, is = 0.0;
    if (sl > 0.0) {
      bias = sl / c.h;
    } else if (use_bias) {
      bias = fmax(c.rate * sl, -PGS_MAX_BIAS_VELOCITY);
      ms = c.mass_scale;
      is = c.impulse_scale;
    }
    double delta = -inv_a * ms * (jv + bias) - is * lam;
    return fmax(lam + delta, 0.0);
  }
  if (kind == PK_BILATERAL) {
    double bias = 0.0, ms = 1.0, is = 0.0;
    if (use_bias) {
      bias = fmin(fmax(c.rate * sep(), -PGS_MAX_BIAS_VELOCITY), PGS_MAX_BIAS_VELOCITY);
      ms = c.mass_scale;
      is = c.impulse_scale;
    }
    return lam - inv_a * ms * (jv + bias) - is * lam;
  }
  double b = bound();
  return fmin(fmax(lam - inv_a * jv, -b), b);
}

// The biased sweeps, vpos from v, the relaxing sweeps (solver.rs:217-251);
// sweep(use_bias) returns the largest velocity change (one call site, so that
// it is inlined). Returns their number.
template <int G, class F>
__device__ __forceinline__ int pgs_sweeps(const Tile<G>& T, const DModel& m, const double* v, double* vpos, F sweep) {
  int sweeps = 0;
  for (int phase = 0; phase < 2; phase++) {
    const bool use_bias = phase == 0;
    const int most = use_bias ? m.iterations : max(m.iterations / 3, 2);
    for (int it = 0; it < most; it++) {
      sweeps++;
      if (sweep(use_bias) < PGS_TOLERANCE) break;
    }
    T.sync();
    if (use_bias) {
      for (int k = T.lane(); k < m.nv; k += G) vpos[k] = v[k];
      T.sync();
    }
  }
  return sweeps;
}

// Every row in turn on the whole tile (see pgs_solve). SPANS: only the entries
// within a row's span are formed and read.
template <int G, bool SPANS>
__device__ __forceinline__ int pgs_tile(const Tile<G>& T, const DModel& m, const WsLayout& w, const ScrLayout& s,
                                     const EnvCtx& e, int ncon, double* v, double* vpos, const double* L,
                                     double* prev, int32_t* prev_ncon, int* nrows, int* status) {
  int lane = T.lane(), nv = m.nv;
  double* J = e.scr + s.jac;
  double* R = e.scr + s.rows;
  double* MJ = e.scr + s.mj;
  const double* con = e.con;
  int nr = pgs_rows<G, SPANS>(T, m, w, e, ncon, v, J, R, status);
  *nrows = nr;
  for (int k = lane; k < nv; k += G) vpos[k] = v[k];
  if (nr == 0) {
    if (lane == 0) *prev_ncon = 0;
    T.sync();
    return 0;
  }
  // M^-1 J_r' and 1 / (J_r M^-1 J_r') per row, one row per lane
  for (int r = lane; r < nr; r += G) {
    double* x = MJ + r * nv;
    const double* jr = J + r * nv;
    double a = 0.0;
    if (SPANS) {
      const Span sp = Span::of(R[PR_STRIDE * r + PR_SPAN]);
      span_each(sp, [&](int k) { x[k] = jr[k]; });
      tree_mass_solve(sp.a0, sp.a1, nv, L, x);
      tree_mass_solve(sp.b0, sp.b1, nv, L, x);
      span_each(sp, [&](int k) { a += jr[k] * x[k]; });
    } else {
      for (int k = 0; k < nv; k++) x[k] = jr[k];
      for (int b = 0; b < m.nblock; b++) tree_mass_solve(m.block_adr[2 * b], m.block_adr[2 * b + 1], nv, L, x);
      for (int k = 0; k < nv; k++) a += jr[k] * x[k];
    }
    R[PR_STRIDE * r + PR_INVA] = a > 1e-12 ? 1.0 / a : 0.0;
  }
  const int nc = min(ncon, nr / 3);
  pgs_lend(T, con, nc, prev, *prev_ncon, R);
  T.sync();
  for (int k = lane; k < nv; k += G) {
    double vk = v[k];
    for (int r = 0; r < nr; r++) {
      double l = R[PR_STRIDE * r + PR_LAMBDA];
      if (l != 0.0 && (!SPANS || Span::of(R[PR_STRIDE * r + PR_SPAN]).has(k))) vk += MJ[r * nv + k] * l;
    }
    v[k] = vk;
  }
  T.sync();
  const PgsBias c = pgs_bias(m);
  auto sweep = [&](bool use_bias) -> double {
    double max_dv = 0.0, normal_l = 0.0;
    // a row's record is read while the row before it works (its impulse is
    // its own; a contact's friction rows follow its normal row)
    double inv_a = R[PR_INVA], lam = R[PR_LAMBDA], kind = R[PR_KIND], sep = R[PR_SEP], mu = R[PR_MU];
    for (int r = 0; r < nr; r++) {
      double* rr = R + PR_STRIDE * r;
      const double* nx = R + PR_STRIDE * (r + 1 < nr ? r + 1 : r);
      const double n_inv_a = nx[PR_INVA], n_lam = nx[PR_LAMBDA], n_kind = nx[PR_KIND], n_sep = nx[PR_SEP], n_mu = nx[PR_MU];
      double nw = lam;
      if (inv_a != 0.0) {
        const double* jr = J + r * nv;
        double jv = 0.0;
        Span sp;
        if (SPANS) {
          sp = Span::of(rr[PR_SPAN]);
          span_each(sp, [&](int k) { jv += jr[k] * v[k]; });
        } else {
          for (int k = 0; k < nv; k++) jv += jr[k] * v[k];
        }
        nw = pgs_impulse(c, (int)kind, jv, lam, inv_a, use_bias, [&] { return sep; }, [&] { return mu * normal_l; });
        double dl = nw - lam;
        if (dl != 0.0) {
          max_dv = fmax(max_dv, fabs(dl) / inv_a);
          T.sync();  // every lane has read v and the impulses
          const double* mr = MJ + r * nv;
          if (SPANS) {
            for (int k = sp.a0 + lane; k < sp.a1; k += G) v[k] += mr[k] * dl;
            for (int k = sp.b0 + lane; k < sp.b1; k += G) v[k] += mr[k] * dl;
          } else {
            for (int k = lane; k < nv; k += G) v[k] += mr[k] * dl;
          }
          if (lane == 0) rr[PR_LAMBDA] = nw;
          T.sync();
        }
      }
      if (kind == PK_NORMAL) normal_l = nw;
      inv_a = n_inv_a;
      lam = n_lam;
      kind = n_kind;
      sep = n_sep;
      mu = n_mu;
    }
    return max_dv;
  };
  int sweeps = pgs_sweeps(T, m, v, vpos, sweep);
  pgs_keep(T, con, nc, prev, prev_ncon, R);
  return sweeps;
}

// Islands on lanes (see pgs_solve); tree: each tree's island, by its lowest
// tree; roots: the set of these.
template <int G>
__device__ __noinline__ int pgs_lanes(const Tile<G>& T, const DModel& m, const WsLayout& w, const ScrLayout& s,
                                      const EnvCtx& e, int ncon, double* v, double* vpos, const double* L,
                                      double* prev, int32_t* prev_ncon, int* nrows, int* status, const int* tree,
                                      unsigned long long roots) {
  int lane = T.lane(), nv = m.nv;
  double* J = e.scr + s.jac;
  double* R = e.scr + s.rows;
  double* MJ = e.scr + s.mj;
  const double* con = e.con;
  int nr = pgs_rows<G, true>(T, m, w, e, ncon, v, J, R, status);
  *nrows = nr;
  for (int k = lane; k < nv; k += G) vpos[k] = v[k];
  if (nr == 0) {
    if (lane == 0) *prev_ncon = 0;
    T.sync();
    return 0;
  }
  // M^-1 J_r' and 1 / (J_r M^-1 J_r') per row, one row per lane
  for (int r = lane; r < nr; r += G) {
    double* x = MJ + r * nv;
    const double* jr = J + r * nv;
    Span sp = Span::of(R[PR_STRIDE * r + PR_SPAN]);
    span_each(sp, [&](int k) { x[k] = jr[k]; });
    tree_mass_solve(sp.a0, sp.a1, nv, L, x);
    tree_mass_solve(sp.b0, sp.b1, nv, L, x);
    double a = 0.0;
    span_each(sp, [&](int k) { a += jr[k] * x[k]; });
    R[PR_STRIDE * r + PR_INVA] = a > 1e-12 ? 1.0 / a : 0.0;
  }
  const int nc = min(ncon, nr / 3);
  pgs_lend(T, con, nc, prev, *prev_ncon, R);
  // the rows of each lane's islands, in row order (an island's lane: its
  // rank among the islands, modulo the tile)
  int* mine = reinterpret_cast<int*>(e.scr + s.isl_row);  // [maxrows] lists, then [maxrows] lanes of the rows
  int* row_lane = mine + m.maxrows;
  for (int r = lane; r < nr; r += G) {
    Span sp = Span::of(R[PR_STRIDE * r + PR_SPAN]);
    const int t = sp.a1 > 0 ? tree[m.dof_block[sp.a0]] : 0;
    row_lane[r] = __popcll(roots & ((1ull << t) - 1)) % G;
  }
  T.sync();
  int count = 0;
  for (int r = 0; r < nr; r++) count += row_lane[r] == lane ? 1 : 0;
  int all;
  int first = T.excl_scan(count, &all);
  for (int r = 0, k = first; r < nr; r++)
    if (row_lane[r] == lane) mine[k++] = r;
  // rows of one tree of at most six dofs, one 128-byte line each in the order
  // of the lists: J, M^-1 J', 1 / a, impulse, sep or mu, kind (a sweep reads
  // one line a row instead of parts of seven sectors)
  constexpr int NU = 6;
  enum { L_J = 0, L_W = NU, L_INVA = 2 * NU, L_LAMBDA, L_ARG, L_KIND, L_STRIDE };
  static_assert(L_STRIDE == 16, "a line a row");
  const bool lines = nv >= L_STRIDE;  // (the island buffer, unused on this path, holds them)
  double* line = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(e.scr + s.sub_j) + 127) & ~uintptr_t(127));
  // a line's kind: the row's, plus 4 when the row goes another way
  if (lines)
    for (int x = first; x < first + count; x++) {
      const int r = mine[x];
      const double* rr = R + PR_STRIDE * r;
      const Span sp = Span::of(rr[PR_SPAN]);
      double* o = line + L_STRIDE * x;
      const int na = sp.a1 - sp.a0;
      const bool fits = sp.b1 == 0 && na <= NU;
      for (int k = 0; k < NU; k++) {
        o[L_J + k] = fits && k < na ? J[r * nv + sp.a0 + k] : 0.0;
        o[L_W + k] = fits && k < na ? MJ[r * nv + sp.a0 + k] : 0.0;
      }
      o[L_INVA] = rr[PR_INVA];
      o[L_LAMBDA] = rr[PR_LAMBDA];
      o[L_ARG] = rr[PR_KIND] == PK_FRICTION ? rr[PR_MU] : rr[PR_SEP];
      // (span start in the upper part)
      o[L_KIND] = rr[PR_KIND] + (fits ? 0.0 : 4.0) + 8.0 * sp.a0 + 1024.0 * na;
    }
  // the warm start's impulses
  for (int x = first; x < first + count; x++) {
    int r = mine[x];
    double l = R[PR_STRIDE * r + PR_LAMBDA];
    if (l != 0.0) span_each(Span::of(R[PR_STRIDE * r + PR_SPAN]), [&](int k) { v[k] += MJ[r * nv + k] * l; });
  }
  T.sync();
  const PgsBias c = pgs_bias(m);
  // one Gauss-Seidel sweep; returns the largest velocity change. The
  // velocities of the tree that the last rows touched stay in registers (u,
  // dofs [held, held + 6)), a contact's normal impulse with them; a row of two
  // trees, or of a tree of more than six dofs, goes through shared memory.
  auto sweep = [&](bool use_bias) -> double {
    double max_dv = 0.0;
    double u[NU];
    int held = -1, hold_n = 0;
    double normal_l = 0.0;
    auto drop = [&]() {
      if (held >= 0)
#pragma unroll
        for (int k = 0; k < NU; k++)
          if (k < hold_n) v[held + k] = u[k];
      held = -1;
    };
    for (int x = first; x < first + count; x++) {
      double* o = line + L_STRIDE * x;
      double inv_a, lam, arg;
      int kind, a0 = 0, na = 0, r = -1;
      Span sp{0, 0, 0, 0};
      bool fits = false;
      if (lines) {
        if (x + 1 < first + count) prefetch_row(o + L_STRIDE);
        inv_a = o[L_INVA];
        lam = o[L_LAMBDA];
        arg = o[L_ARG];
        const int code = (int)o[L_KIND];
        kind = code & 3;
        fits = !(code & 4);
        a0 = code >> 3 & 127;
        na = code >> 10;
      }
      if (!fits) {
        r = mine[x];
        const double* rr = R + PR_STRIDE * r;
        inv_a = rr[PR_INVA];
        lam = rr[PR_LAMBDA];
        sp = Span::of(rr[PR_SPAN]);
        kind = (int)rr[PR_KIND];
        arg = kind == PK_FRICTION ? rr[PR_MU] : rr[PR_SEP];
      }
      if (inv_a == 0.0) {
        if (kind == PK_NORMAL) normal_l = lam;
        continue;
      }
      // a contact's normal row stands before its friction rows in the list
      auto sep = [&] { return arg; };
      auto bound = [&] { return arg * normal_l; };
      double nw, dl;
      if (fits) {
        if (held != a0) {
          drop();
          held = a0;
          hold_n = na;
#pragma unroll
          for (int k = 0; k < NU; k++) u[k] = k < na ? v[a0 + k] : 0.0;
        }
        double jv = 0.0;
#pragma unroll
        for (int k = 0; k < NU; k++) jv += o[L_J + k] * u[k];
        nw = pgs_impulse(c, kind, jv, lam, inv_a, use_bias, sep, bound);
        dl = nw - lam;
        if (dl != 0.0) {
#pragma unroll
          for (int k = 0; k < NU; k++) u[k] += o[L_W + k] * dl;
          o[L_LAMBDA] = nw;
        }
      } else {
        drop();
        const double* jr = J + r * nv;
        const double* mr = MJ + r * nv;
        double jv = 0.0;
        span_each(sp, [&](int k) { jv += jr[k] * v[k]; });
        nw = pgs_impulse(c, kind, jv, lam, inv_a, use_bias, sep, bound);
        dl = nw - lam;
        if (dl != 0.0) {
          span_each(sp, [&](int k) { v[k] += mr[k] * dl; });
          R[PR_STRIDE * r + PR_LAMBDA] = nw;
        }
      }
      if (kind == PK_NORMAL) normal_l = nw;
      if (dl != 0.0) max_dv = fmax(max_dv, fabs(dl) / inv_a);
    }
    drop();
    return T.fmax(max_dv);
  };
  int sweeps = pgs_sweeps(T, m, v, vpos, sweep);
  if (lines)
    for (int x = first; x < first + count; x++)
      if (!((int)line[L_STRIDE * x + L_KIND] & 4)) R[PR_STRIDE * mine[x] + PR_LAMBDA] = line[L_STRIDE * x + L_LAMBDA];
  T.sync();
  pgs_keep(T, con, nc, prev, prev_ncon, R);
  return sweeps;
}

// Whether the trees' contacts spread over islands enough for a lane each: no
// lane has more than half of them. Leaves each tree's island in `tree`, named
// by its lowest tree, and the set of these in *roots.
template <int G>
__device__ __noinline__ bool pgs_spread(const Tile<G>& T, const DModel& m, const ScrLayout& s, const EnvCtx& e,
                                        int ncon, int* tree, unsigned long long* roots) {
  const int lane = T.lane(), n = ncon + m.neq;
  int* ends = reinterpret_cast<int*>(e.scr + s.isl_row);  // the two trees of each contact, then equality
  int* held = tree + m.nblock;                            // contacts of each lane
  for (int b = lane; b < m.nblock; b += G) {
    tree[b] = b;
    held[b] = 0;
  }
  for (int i = lane; i < n; i += G) {
    int a, b = -1;
    if (i < ncon) {
      a = body_tree(m, m.geom_body[(int)e.con[C_STRIDE * i + C_G1]]);
      b = body_tree(m, m.geom_body[(int)e.con[C_STRIDE * i + C_G2]]);
    } else {
      const int j2 = m.eq_j2[i - ncon];
      a = m.dof_block[m.jnt_dofadr[m.eq_j1[i - ncon]]];
      if (j2 != -1) b = m.dof_block[m.jnt_dofadr[j2]];
    }
    // (a tree that stands alone is joined to itself)
    ends[i] = (a < 0 ? max(b, 0) : a) | (b < 0 ? max(a, 0) : b) << 8;
  }
  T.sync();
  for (bool more = true; more;) {
    bool changed = false;
    for (int i = lane; i < n; i += G) {
      const int a = ends[i] & 255, b = ends[i] >> 8;
      const int ta = tree[a], tb = tree[b];
      if (ta != tb) {
        atomicMin(tree + (ta > tb ? a : b), ta < tb ? ta : tb);
        changed = true;
      }
    }
    T.sync();
    more = T.any(changed);
  }
  unsigned long long r = 0;
  for (int b = 0; b < m.nblock; b++)
    if (tree[b] == b) r |= 1ull << b;
  *roots = r;
  for (int i = lane; i < ncon; i += G) atomicAdd(held + __popcll(r & ((1ull << tree[ends[i] & 255]) - 1)) % G, 1);
  T.sync();
  int most = 0;
  for (int b = 0; b < m.nblock; b++) most = max(most, held[b]);
  return 2 * most <= ncon;
}

// The tile on a model of one tree, out of line: two tiles of a warp that take
// different branches meet again at its syncs (4096 Ant envs 1430 us a substep,
// 1780 with this inlined beside the other paths).
template <int G>
__device__ __noinline__ int pgs_tree(const Tile<G>& T, const DModel& m, const WsLayout& w, const ScrLayout& s,
                                     const EnvCtx& e, int ncon, double* v, double* vpos, const double* L,
                                     double* prev, int32_t* prev_ncon, int* nrows, int* status) {
  return pgs_tile<G, false>(T, m, w, s, e, ncon, v, vpos, L, prev, prev_ncon, nrows, status);
}

// solver.rs:63-251 and the warm start of :254-289. On entry v holds the
// unconstrained velocity qvel + h (M + hD)^-1 f; on exit v is the final
// velocity and vpos the velocity after the biased sweeps (which positions
// integrate with). L is the factor of M + hD (stride nv). prev / prev_ncon are
// the env's previous-step contacts and impulses, replaced by this step's.
// Returns the number of sweeps; *nrows gets the row count.
template <int G>
__device__ __forceinline__ int pgs_solve(const Tile<G>& T, const DModel& m, const WsLayout& w, const ScrLayout& s,
                                      const EnvCtx& e, int ncon, double* v, double* vpos, const double* L,
                                      double* prev, int32_t* prev_ncon, int* nrows, int* status) {
  int* tree = reinterpret_cast<int*>(e.ws + w.grad);  // [2 nblock] (free on this path)
  unsigned long long roots;
  if (m.nblock > 2 && ncon > 0 && pgs_spread(T, m, s, e, ncon, tree, &roots))
    return pgs_lanes(T, m, w, s, e, ncon, v, vpos, L, prev, prev_ncon, nrows, status, tree, roots);
  if (m.nblock == 1) return pgs_tree(T, m, w, s, e, ncon, v, vpos, L, prev, prev_ncon, nrows, status);
  if (m.nv > PGS_DENSE_NV)
    return pgs_tile<G, true>(T, m, w, s, e, ncon, v, vpos, L, prev, prev_ncon, nrows, status);
  return pgs_tile<G, false>(T, m, w, s, e, ncon, v, vpos, L, prev, prev_ncon, nrows, status);
}

}  // namespace pg
