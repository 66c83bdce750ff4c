// The whole substep with one lane per environment, for models of at most 8
// dofs in one tree that can have no constraint rows (no limits, every pair
// masked out): control tasks and arms.
//
// A tile of 16 lanes leaves most of them idle on such trees (a chain has one
// body a level) and pays every instruction per env; here 32 envs share each
// one. 16384 cartpoles took 2927 warp instructions an env and substep, now
// 104. A call's substeps run in one launch with the state in registers and
// local arrays, so ten substeps read and write it once. M is factored last
// row first (H = L' D L) in registers with the compile-time size N, every
// index constant: rolled loops over a local array made each entry a round
// trip to L1 (50k cycles a factor of 14 rows against 6k).
//
// Measured (B200, 16384 envs, ten substeps a call): cartpole 1620 us with the
// phase kernels, 110 us; with three batches in flight 1398 against 53 us a
// batch. What bounds it: dependent FP64 instructions of one warp a
// sub-partition (about 5 cycles each) up to some 20,000 envs.
#include <cuda_runtime.h>

#include "pg_lane.cuh"

namespace pg {
namespace {

// x <- (H + diag(add))^-1 x by H = L' D L, last row first; false if a pivot
// is not positive.
template <int N>
__device__ __forceinline__ bool factor_solve(const double* H, const double (&add)[N], double (&x)[N]) {
  double h[N * (N + 1) / 2];
#pragma unroll
  for (int t = 0; t < N * (N + 1) / 2; t++) h[t] = H[t];
#pragma unroll
  for (int i = 0; i < N; i++) h[tri(i, i)] += add[i];
  bool ok = true;
#pragma unroll
  for (int k = N - 1; k >= 0; k--) {
    double d = h[tri(k, k)];
    ok = ok && d > 0.0;
    double inv = 1.0 / d;
    h[tri(k, k)] = inv;
#pragma unroll
    for (int i = k - 1; i >= 0; i--) {
      double l = h[tri(k, i)] * inv;
#pragma unroll
      for (int j = 0; j <= i; j++) h[tri(i, j)] -= l * h[tri(k, j)];
      x[i] -= l * x[k];
      h[tri(k, i)] = l;
    }
  }
#pragma unroll
  for (int k = 0; k < N; k++) {
    double xk = x[k] * h[tri(k, k)];
#pragma unroll
    for (int j = 0; j < k; j++) xk -= h[tri(k, j)] * x[j];
    x[k] = xk;
  }
  return ok;
}

template <int N>
__global__ void __launch_bounds__(32) lane_kernel(const __grid_constant__ StepArgs A, const __grid_constant__ LaneArgs P) {
  const DModel& m = A.m;
  const int nv = m.nv, nq = m.nq, nu = m.nu;
  const int lane = threadIdx.x;
  const int64_t item0 = (int64_t)blockIdx.x * P.lanes;
  const int L = A.count - item0 < P.lanes ? (int)(A.count - item0) : P.lanes;  // envs of this warp
  const bool alive = lane < L;
  const int64_t item = item0 + (alive ? lane : L - 1);  // the others repeat the last env and write nothing
  const int64_t env = A.start + item;
  // env 0's block, or the env's column of its group's copy
  const bool mixed = __any_sync(FULL, *P.mixed != 0);  // (the same for the warp: uniform to the compiler too)
  const double* pp = mixed ? P.columns + (env >> 5) * (int64_t)(m.p_qpos_reset - m.p_mass) * 32 + (env & 31) - m.p_mass * 32
                           : A.st.params;
  const int ps = mixed ? 32 : 1;
  const double h = m.timestep;

  double q[LANE_NQ], v[N], f[N], qacc[N], hd[N];
  double M[N * (N + 1) / 2], cdof[6 * N];
  double lv[(LANE_DEPTH + 1) * V_STRIDE];

  for (int k = 0; k < nq; k++) q[k] = A.st.qpos[env * nq + k];
  bool damped = false;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const bool in = k < nv;
    v[k] = in ? A.st.qvel[env * nv + k] : 0.0;
    qacc[k] = in ? A.st.qacc[env * nv + k] : 0.0;
    hd[k] = in ? pp[(m.p_damping + k) * ps] : 0.0;
    damped |= hd[k] != 0.0;
  }
  int status_all = P.sidx == 0 ? 0 : A.st.status[env];

#pragma unroll 1
  for (int sub = 0; sub < P.nsub; sub++) {
    const int sidx = P.sidx + sub;
    int status = 0;
    // ------------------------------------------------ tree walk
#pragma unroll
    for (int i = 0; i < N; i++) {
#pragma unroll
      for (int j = 0; j < i; j++) M[tri(i, j)] = 0.0;
      M[tri(i, i)] = 1.0;
      f[i] = 0.0;
    }
#pragma unroll
    for (int t = 0; t < 6 * N; t++) cdof[t] = 0.0;
    // the body walked last: its pose, velocity, acceleration, and the sums of
    // its subtree so far (the world first)
    Walk s;
    walk_world(m, s);
    Sym& I = s.I;
    Sp& fr = s.fr;
    int top = 0;
    int path[LANE_DEPTH + 1];
    path[0] = 0;
    int par = -1;
#pragma unroll 1
    for (int b = 0; b <= m.nbody; b++) {
      if (b > 0) {
        // leave the bodies whose subtrees end here: their inertia and force
        // sums are complete, which gives the rows of M and the bias force of
        // their dofs, and go to the parent's
        par = b < m.nbody ? m.body_parent[b] : 0;
        bool left = false;
#pragma unroll 1
        while (top > 0 && path[top] != par) {
          int x = path[top], i0 = m.body_dofadr[x], i1 = i0 + m.body_dofnum[x];
          unsigned chain = (unsigned)m.body_dofmask[x];
#pragma unroll 1
          for (int i = i0; i < i1; i++) {
            Sp ci = ld6(cdof + 6 * i);
            Sp fi = sym_mul(I, ci);
            M[tri(i, i)] = sp_dot(ci, fi) + m.dof_armature[i];
            f[i] = -sp_dot(ci, fr);
            double* row = M + tri(i, 0);
            unsigned below = chain & ((1u << i) - 1u);
#pragma unroll
            for (int j = 0; j < N; j++)
              if (below >> j & 1u) row[j] = sp_dot(ld6(cdof + 6 * j), fi);
          }
          top--;
          left = true;
          if (top > 0) {
            const double* u = lv + top * V_STRIDE;
            I.mass += u[V_CRB];
            I.mc = I.mc + ld3(u + V_CRB + 1);
            I.xx += u[V_CRB + 4];
            I.xy += u[V_CRB + 5];
            I.xz += u[V_CRB + 6];
            I.yy += u[V_CRB + 7];
            I.yz += u[V_CRB + 8];
            I.zz += u[V_CRB + 9];
            fr = sp_add(fr, ld6(u + V_FRC));
          }
        }
        if (b == m.nbody) break;
        double* r = lv + top * V_STRIDE;
        if (left) {
          if (top > 0) {
            s.pos = ld3(r + V_POS);
            s.quat = ld4(r + V_QUAT);
            s.mat = q_mat(s.quat);
            s.vel = ld6(r + V_VEL);
            s.acc = ld6(r + V_ACC);
          } else {
            walk_world(m, s);
          }
        } else if (top > 0) {
          st3(r + V_POS, s.pos);
          st4(r + V_QUAT, s.quat);
          st6(r + V_VEL, s.vel);
          st6(r + V_ACC, s.acc);
        }
        if (top > 0) {
          r[V_CRB] = I.mass;
          st3(r + V_CRB + 1, I.mc);
          r[V_CRB + 4] = I.xx;
          r[V_CRB + 5] = I.xy;
          r[V_CRB + 6] = I.xz;
          r[V_CRB + 7] = I.yy;
          r[V_CRB + 8] = I.yz;
          r[V_CRB + 9] = I.zz;
          st6(r + V_FRC, fr);
        }
        top++;
        path[top] = b;
        walk_body(m, P.t, b, q, v, cdof, pp, ps, s);
      }
    }
    // ------------------------------------------------ passive and actuator forces
#pragma unroll
    for (int k = 0; k < N; k++)
      if (k < nv) f[k] += A.st.applied[env * nv + k] - hd[k] * v[k];
    for (int j = 0; j < m.njnt; j++) {
      double kp = m.jnt_stiffness[j];
      int t = m.jnt_type[j];
      if (kp != 0.0 && (t == JNT_HINGE || t == JNT_SLIDE)) f[m.jnt_dofadr[j]] -= kp * (q[m.jnt_qposadr[j]] - m.jnt_springref[j]);
    }
#pragma unroll 1
    for (int u = 0; u < nu; u++) {
      double gear = m.act_gear[u];
      int a0 = m.act_moment_adr[u], an = m.act_moment_num[u];
      double ls = 0.0, vs = 0.0;
      for (int k = a0; k < a0 + an; k++) {
        int j = m.moment_jnt[k];
        ls += m.moment_coef[k] * q[m.jnt_qposadr[j]];
        vs += m.moment_coef[k] * v[m.jnt_dofadr[j]];
      }
      double c = A.ctrl_seq ? A.ctrl_seq[((size_t)item * A.nstep + sidx) * nu + u] : A.st.ctrl[env * nu + u];
      if (A.ctrl_seq && alive) A.st.ctrl[env * nu + u] = c;  // rollout leaves the last controls in place
      if (m.act_ctrllimited[u]) c = clampd(c, m.act_ctrlrange[2 * u], m.act_ctrlrange[2 * u + 1]);
      double fu = pp[(m.p_gain + u) * ps] * c + pp[(m.p_bias + 3 * u) * ps] + pp[(m.p_bias + 3 * u + 1) * ps] * (gear * ls) +
                  pp[(m.p_bias + 3 * u + 2) * ps] * (gear * vs);
      if (m.act_forcelimited[u]) fu = clampd(fu, m.act_forcerange[2 * u], m.act_forcerange[2 * u + 1]);
      for (int k = a0; k < a0 + an; k++) f[m.jnt_dofadr[m.moment_jnt[k]]] += gear * m.moment_coef[k] * fu;
    }
    // ------------------------------------------------ a0 = M^-1 f
    double a[N];
    {
      double zero[N];
#pragma unroll
      for (int i = 0; i < N; i++) {
        a[i] = f[i];
        zero[i] = 0.0;
      }
      if (!factor_solve(M, zero, a)) status |= ST_NOT_SPD;
    }
    // ------------------------------------------------ damped solve
    if (__any_sync(FULL, damped)) {
      double x[N], add[N];
#pragma unroll
      for (int i = 0; i < N; i++) {
        x[i] = f[i];
        add[i] = h * hd[i];
      }
      bool ok = factor_solve(M, add, x);
      if (damped) {
        if (!ok) status |= ST_NOT_SPD;
#pragma unroll
        for (int i = 0; i < N; i++) a[i] = x[i];
      }
    }
    // ------------------------------------------------ integration
    if (!(status & ST_NOT_SPD)) {
#pragma unroll
      for (int k = 0; k < N; k++) {
        double vk = v[k] + h * a[k];
        qacc[k] = (vk - v[k]) / h;
        v[k] = vk;
      }
#pragma unroll 1
      for (int j = 0; j < m.njnt; j++) {
        int qa = m.jnt_qposadr[j], da = m.jnt_dofadr[j];
        int type = m.jnt_type[j];
        if (type == JNT_FREE || type == JNT_BALL) {
          int o = type == JNT_FREE ? 3 : 0;
          for (int k = 0; k < o; k++) q[qa + k] += h * v[da + k];
          Q4 x{q[qa + o], q[qa + o + 1], q[qa + o + 2], q[qa + o + 3]};
          V3 w{v[da + o], v[da + o + 1], v[da + o + 2]};
          double n = norm(w);
          if (!(n * h < 1e-15)) {
            double sn, cs;
            sincos(0.5 * (n * h), &sn, &cs);
            sn /= n;
            x = unit(q_mul(x, Q4{cs, w.x * sn, w.y * sn, w.z * sn}));
          }
          q[qa + o] = x.w;
          q[qa + o + 1] = x.x;
          q[qa + o + 2] = x.y;
          q[qa + o + 3] = x.z;
        } else {
          q[qa] += h * v[da];
        }
      }
    }
    if (A.qpos_out && alive)
      for (int k = 0; k < nq; k++) A.qpos_out[((size_t)item * A.nstep + sidx) * nq + k] = q[k];
    status_all |= status;
    __syncwarp();
  }
  if (alive) {
    for (int k = 0; k < nq; k++) A.st.qpos[env * nq + k] = q[k];
#pragma unroll
    for (int k = 0; k < N; k++)
      if (k < nv) {
        A.st.qvel[env * nv + k] = v[k];
        A.st.qacc[env * nv + k] = qacc[k];
      }
    A.st.iters[env] = 0;
    A.st.ncon[env] = 0;
    A.st.nrows[env] = 0;
    A.st.status[env] = status_all;
  }
}

}  // namespace

cudaError_t launch_lane(const StepArgs& a, const LaneArgs& p, cudaStream_t s) {
  int64_t warps = ((int64_t)a.count + p.lanes - 1) / p.lanes;
  if (warps <= 0) return cudaSuccess;
  if (a.m.nv <= 4) lane_kernel<4><<<(unsigned)warps, 32, 0, s>>>(a, p);
  else lane_kernel<8><<<(unsigned)warps, 32, 0, s>>>(a, p);
  return cudaGetLastError();
}

}  // namespace pg
