// Projected Gauss-Seidel (crates/pippin/src/solver.rs:38-289) for one env,
// run by the Newton-phase kernel when the model's solver is PGS.
//
// Rows follow the reference's order: [normal, tangent 1, tangent 2] per
// contact (every contact of the narrow phase, not only touching ones), then
// the joint-limit sides within reach, then the joint equalities. A row touches
// the dofs of one or two trees: only those entries of J and M^-1 J' are formed
// and read (PR_SPAN), the others are zero.
//
// Gauss-Seidel is sequential over rows, but rows of separate islands (trees
// joined by rows) share no velocity, so each lane sweeps islands of its own, in
// row order, and the tile meets once a sweep for the largest change: the
// sequential sweep's result to the bit (a sum's terms that are left out are
// zero). With the whole tile on one row at a time (48 dofs a product, two tile
// syncs a row) 1001 envs of 8 hulls took 6.67 ms in this phase; islands side by
// side 1.43 ms, and with a row's numbers in one 128-byte line, prefetched a row
// ahead, and the tree's velocities in registers 1.17 ms (32 lanes an env, from
// a state without impulses). What bounds it now is the chain of one row's loads
// and sums after another.
#pragma once
#include "pg_newton.cuh"

namespace pg {

constexpr double PGS_MAX_BIAS_VELOCITY = 1.0;  // solver.rs:34
constexpr double PGS_TOLERANCE = 1e-5;         // solver.rs:36
constexpr double PGS_MATCH_DIST2 = 0.01 * 0.01;  // solver.rs:255

// The dof ranges [a0, a1) and [b0, b1) a row touches (one tree, or two in
// ascending order), packed in its record's PR_SPAN.
struct Span {
  int a0, a1, b0, b1;
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
// f(k) for the span's dofs in ascending order
__device__ __forceinline__ void prefetch_row(const double* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
template <class F>
__device__ __forceinline__ void span_each(const Span& s, F f) {
  for (int k = s.a0; k < s.a1; k++) f(k);
  for (int k = s.b0; k < s.b1; k++) f(k);
}

// Rows of the PGS problem (solver.rs:63-163) into J (stride nv) and R
// (PR_* records). Returns the row count, capped at maxrows.
template <int G>
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
    double span = pack_span(m, body_tree(m, m.geom_body[g1]), body_tree(m, m.geom_body[g2]));
    for (int q = 0; q < 3; q++) {
      double* rr = R + PR_STRIDE * (3 * c + q);
      rr[PR_KIND] = q == 0 ? PK_NORMAL : PK_FRICTION;
      rr[PR_SEP] = q == 0 ? -r[C_DEPTH] : 0.0;
      rr[PR_MU] = q == 0 ? 0.0 : mu;
      rr[PR_NORMAL] = 3 * c;
      rr[PR_CONTACT] = c;
      rr[PR_INVA] = 0.0;
      rr[PR_LAMBDA] = 0.0;
      rr[PR_SPAN] = span;
    }
  }
  T.sync();
  for (int it = lane; it < nc * 2 * m.maxbs; it += G) {
    int c = it / (2 * m.maxbs), o = it % (2 * m.maxbs);
    Span sp = Span::of(R[PR_STRIDE * 3 * c + PR_SPAN]);
    int k = o < m.maxbs ? sp.a0 + o : sp.b0 + o - m.maxbs;
    if (k >= (o < m.maxbs ? sp.a1 : sp.b1)) continue;
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
        rr[PR_SPAN] = pack_span(m, m.dof_block[da], -1);
        span_each(Span::of(rr[PR_SPAN]), [&](int k) { jr[k] = 0.0; });
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
    rr[PR_SPAN] = pack_span(m, m.dof_block[m.jnt_dofadr[j1]], j2 != -1 ? m.dof_block[m.jnt_dofadr[j2]] : -1);
    span_each(Span::of(rr[PR_SPAN]), [&](int k) { jr[k] = 0.0; });
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

// x <- (L L')^-1 x for one right-hand side, by one lane, on the trees of a
// span, with the reference's operations (math.rs:451-463: row-oriented forward
// sweep dividing by the pivot, then column-oriented backward sweep).
__device__ inline void lane_mass_solve(const Span& sp, int nv, const double* L, double* x) {
  for (int t = 0; t < 2; t++) {
    int s0 = t == 0 ? sp.a0 : sp.b0, s1 = t == 0 ? sp.a1 : sp.b1;
    for (int i = s0; i < s1; i++) x[i] = (x[i] - dot_ref(L + i * nv + s0, 1, x + s0, 1, i - s0)) / L[i * nv + i];
    for (int i = s1 - 1; i >= s0; i--) {
      x[i] /= L[i * nv + i];
      double xi = -x[i];
      for (int k = s0; k < i; k++) x[k] += xi * L[i * nv + k];
    }
  }
}

// solver.rs:63-251 and the warm start of :254-289. On entry v holds the
// unconstrained velocity qvel + h (M + hD)^-1 f; on exit v is the final
// velocity and vpos the velocity after the biased sweeps (which positions
// integrate with). L is the factor of M + hD (stride nv). prev / prev_ncon are
// the env's previous-step contacts and impulses, replaced by this step's.
// Returns the number of sweeps; *nrows gets the row count.
template <int G>
__device__ __noinline__ int pgs_solve(const Tile<G>& T, const DModel& m, const WsLayout& w, const ScrLayout& s,
                                      const EnvCtx& e, int ncon, double* v, double* vpos, const double* L,
                                      double* prev, int32_t* prev_ncon, int* nrows, int* status) {
  int lane = T.lane(), nv = m.nv;
  double h = m.timestep;
  double* J = e.scr + s.jac;
  double* R = e.scr + s.rows;
  double* MJ = e.scr + s.mj;
  const double* con = e.con;
  int nr = pgs_rows(T, m, w, e, ncon, v, J, R, status);
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
    lane_mass_solve(sp, nv, L, x);
    double a = 0.0;
    span_each(sp, [&](int k) { a += jr[k] * x[k]; });
    R[PR_STRIDE * r + PR_INVA] = a > 1e-12 ? 1.0 / a : 0.0;
  }
  // warm start: the nearest previous contact of the same geom pair within
  // 1 cm lends its impulses, the tangent ones re-projected on the new frame
  int np = *prev_ncon;
  int nc = min(ncon, nr / 3);
  for (int c = lane; c < nc; c += G) {
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
  // islands: trees joined by rows, each named by its lowest tree
  int* tree = reinterpret_cast<int*>(e.ws + w.grad);  // [nblock] (free on this path)
  for (int b = lane; b < m.nblock; b += G) tree[b] = b;
  T.sync();
  for (bool more = m.nblock > 1; more;) {
    bool changed = false;
    for (int r = lane; r < nr; r += G) {
      Span sp = Span::of(R[PR_STRIDE * r + PR_SPAN]);
      if (sp.b1 == 0) continue;
      int a = m.dof_block[sp.a0], b = m.dof_block[sp.b0];
      int ta = tree[a], tb = tree[b];
      if (ta != tb) {
        atomicMin(tree + (ta > tb ? a : b), ta < tb ? ta : tb);
        changed = true;
      }
    }
    T.sync();
    more = T.any(changed);
  }
  // the rows of each lane's islands, in row order (an island's lane: its
  // rank among the islands, modulo the tile)
  int* mine = reinterpret_cast<int*>(e.scr + s.isl_row);  // [maxrows] lists, then [maxrows] lanes of the rows
  int* row_lane = mine + m.maxrows;
  for (int r = lane; r < nr; r += G) {
    Span sp = Span::of(R[PR_STRIDE * r + PR_SPAN]);
    int t = sp.a1 > 0 ? tree[m.dof_block[sp.a0]] : 0, rank = 0;
    for (int b = 0; b < t; b++) rank += tree[b] == b ? 1 : 0;
    row_lane[r] = rank % G;
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
  const bool lines = m.nblock > 1 && nv >= L_STRIDE;  // (the island buffer, unused on this path, holds them)
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
  // solver.rs:44-50
  double omega = 2.0 * M_PI * m.hertz;
  double a1 = 2.0 * m.dampratio + h * omega;
  double a2 = h * omega * a1;
  double a3 = 1.0 / (1.0 + a2);
  double bias_rate = omega / a1, mass_scale = a2 * a3, impulse_scale = a3;
  // a row's new impulse from its J . v (solver.rs:164-215)
  // (arg: the row's mu or separation)
  auto impulse = [&](double arg, int kind, double jv, double lam, double inv_a, double normal, bool use_bias) {
    if (kind == PK_FRICTION) {
      double bound = arg * normal;
      return fmin(fmax(lam - inv_a * jv, -bound), bound);
    }
    double bias = 0.0, ms = 1.0, is = 0.0;
    if (kind == PK_NORMAL) {
      double sl = arg + m.slop;
      if (sl > 0.0) {
        bias = sl / h;
      } else if (use_bias) {
        bias = fmax(bias_rate * sl, -PGS_MAX_BIAS_VELOCITY);
        ms = mass_scale;
        is = impulse_scale;
      }
      double delta = -inv_a * ms * (jv + bias) - is * lam;
      return fmax(lam + delta, 0.0);
    }
    if (use_bias) {
      bias = fmin(fmax(bias_rate * arg, -PGS_MAX_BIAS_VELOCITY), PGS_MAX_BIAS_VELOCITY);
      ms = mass_scale;
      is = impulse_scale;
    }
    return lam - inv_a * ms * (jv + bias) - is * lam;
  };
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
      const double normal = kind == PK_FRICTION ? normal_l : 0.0;
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
        nw = impulse(arg, kind, jv, lam, inv_a, normal, use_bias);
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
        nw = impulse(arg, kind, jv, lam, inv_a, normal, use_bias);
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
  int sweeps = 0;
  for (int it = 0; it < m.iterations; it++) {
    sweeps++;
    if (sweep(true) < PGS_TOLERANCE) break;
  }
  T.sync();
  for (int k = lane; k < nv; k += G) vpos[k] = v[k];
  T.sync();
  int nrelax = max(m.iterations / 3, 2);
  for (int it = 0; it < nrelax; it++) {
    sweeps++;
    if (sweep(false) < PGS_TOLERANCE) break;
  }
  if (lines)
    for (int x = first; x < first + count; x++)
      if (!((int)line[L_STRIDE * x + L_KIND] & 4)) R[PR_STRIDE * mine[x] + PR_LAMBDA] = line[L_STRIDE * x + L_LAMBDA];
  T.sync();
  // this step's contacts and impulses for the next warm start
  for (int c = lane; c < nc; c += G) {
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
  if (lane == 0) *prev_ncon = nc;
  T.sync();
  return sweeps;
}

}  // namespace pg
