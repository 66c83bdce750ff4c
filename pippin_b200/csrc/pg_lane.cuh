// Pieces shared by the one- and four-lane substeps (pg_lane.cu, pg_quad.cu).
#pragma once
#include "pg_lane.h"
#include "pg_newton.cuh"

namespace pg {

constexpr unsigned FULL = 0xffffffffu;
__device__ __forceinline__ int tri(int i, int j) { return i * (i + 1) / 2 + j; }

// level record of the tree walk
enum { V_POS = 0, V_QUAT = 3, V_VEL = 7, V_ACC = 13, V_CRB = 19, V_FRC = 29, V_STRIDE = 35 };

struct Sym {  // spatial inertia about the origin, its rotational part symmetric
  double mass;
  V3 mc;
  double xx, xy, xz, yy, yz, zz;
};
__device__ __forceinline__ Sp sym_mul(const Sym& I, const Sp& v) {
  V3 r{I.xx * v.ang.x + I.xy * v.ang.y + I.xz * v.ang.z, I.xy * v.ang.x + I.yy * v.ang.y + I.yz * v.ang.z,
       I.xz * v.ang.x + I.yz * v.ang.y + I.zz * v.ang.z};
  return Sp{r + cross(I.mc, v.lin), v.lin * I.mass - cross(I.mc, v.ang)};
}

// impedance() out of line: its powers would double these kernels' code
__device__ __noinline__ inline double row_impedance(const double* solimp, double pos) { return impedance(solimp, pos); }

__device__ __forceinline__ Q4 unit(Q4 q) {
  double n = q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z;
  if (n < 1e-30) return q_identity();
  double r = rsqrt(n);
  return Q4{q.w * r, q.x * r, q.y * r, q.z * r};
}

// The walk down the tree at one body: pose, velocity and RNE acceleration,
// then (of the body alone) spatial inertia and force.
struct Walk {
  V3 pos;
  Q4 quat;
  M3 mat;  // of quat
  Sp vel, acc;
  Sym I;
  Sp fr;
};
__device__ __forceinline__ void walk_world(const DModel& m, Walk& s) {
  s.pos = V3{0, 0, 0};
  s.quat = q_identity();
  s.mat = m3_identity();
  s.vel = sp_zero();
  s.acc = Sp{V3{0, 0, 0}, -V3{m.gravity[0], m.gravity[1], m.gravity[2]}};
}
// forward.rs:14-90, 115-164 for body b: on entry s holds its parent's pose,
// velocity and acceleration, on return its own; its dofs' axes go to cdof.
// q, v: the env's state; pp, ps: its parameter block, the distance of its entries.
__device__ __forceinline__ void walk_body(const DModel& m, const LaneModel& t, int b, const double* q, const double* v, double* cdof,
                                          const double* pp, int ps, Walk& s) {
  V3& pos = s.pos;
  Q4& quat = s.quat;
  Sp &vel = s.vel, &acc = s.acc;
  Sym& I = s.I;
  M3& xm = s.mat;
  pos = pos + mv(xm, ld3(m.body_pos + 3 * b));
  Q4 bq = ld4(m.body_quat + 4 * b);
  bool turned = false;  // mat no longer of quat
  // (a frame turned by 2e-8 or less has w == 1 all the same)
  if (bq.w != 1.0 || bq.x != 0.0 || bq.y != 0.0 || bq.z != 0.0) {
    quat = q_mul(quat, bq);
    turned = true;
  }
  int j0 = m.body_jntadr[b], j1 = j0 + m.body_jntnum[b];
#pragma unroll 1
  for (int j = j0; j < j1; j++) {
    int qa = m.jnt_qposadr[j], da = m.jnt_dofadr[j];
    int type = m.jnt_type[j];
    if (type == JNT_FREE) {
      pos = V3{q[qa], q[qa + 1], q[qa + 2]};
      quat = unit(Q4{q[qa + 3], q[qa + 4], q[qa + 5], q[qa + 6]});
      turned = true;
      M3 rm = q_mat(quat);
      for (int k = 0; k < 3; k++) {
        V3 ek{k == 0 ? 1.0 : 0.0, k == 1 ? 1.0 : 0.0, k == 2 ? 1.0 : 0.0};
        st6(cdof + 6 * (da + k), Sp{V3{0, 0, 0}, ek});
        V3 ax = col(rm, k);
        st6(cdof + 6 * (da + 3 + k), Sp{ax, cross(pos, ax)});
      }
    } else if (type == JNT_BALL) {
      V3 jp = ld3(m.jnt_pos + 3 * j);
      V3 anchor = pos + q_rot(quat, jp);
      quat = q_mul(quat, unit(Q4{q[qa], q[qa + 1], q[qa + 2], q[qa + 3]}));
      turned = true;
      M3 rm = q_mat(quat);
      pos = anchor - mv(rm, jp);
      for (int k = 0; k < 3; k++) {
        V3 ax = col(rm, k);
        st6(cdof + 6 * (da + k), Sp{ax, cross(anchor, ax)});
      }
    } else if (type == JNT_HINGE) {
      V3 jp = ld3(m.jnt_pos + 3 * j), ja = ld3(m.jnt_axis + 3 * j), ju = ld3(t.jnt_unit + 3 * j);
      double sn, cs;
      sincos(0.5 * (q[qa] - m.qpos0[qa]), &sn, &cs);
      M3 rm = turned ? q_mat(quat) : xm;
      V3 axis = mv(rm, ja);
      quat = q_mul(quat, Q4{cs, ju.x * sn, ju.y * sn, ju.z * sn});
      turned = true;
      V3 anchor = pos;
      if (jp.x != 0.0 || jp.y != 0.0 || jp.z != 0.0) {
        anchor = pos + mv(rm, jp);
        pos = anchor - q_rot(quat, jp);
      }
      st6(cdof + 6 * da, Sp{axis, cross(anchor, axis)});
    } else {
      V3 axis = q_rot(quat, ld3(m.jnt_axis + 3 * j));
      pos = pos + axis * (q[qa] - m.qpos0[qa]);
      st6(cdof + 6 * da, Sp{V3{0, 0, 0}, axis});
    }
  }
  if (turned) {
    quat = unit(quat);
    xm = q_mat(quat);
  }
  V3 ip{pp[(m.p_ipos + 3 * b) * ps], pp[(m.p_ipos + 3 * b + 1) * ps], pp[(m.p_ipos + 3 * b + 2) * ps]};
  M3 in;
#pragma unroll
  for (int t = 0; t < 9; t++) in.m[t] = pp[(m.p_inertia + 9 * b + t) * ps];
  double mass = pp[(m.p_mass + b) * ps];
  // R I R' + m (|c|^2 1 - c c'), upper triangle
  V3 c = pos + mv(xm, ip);
  M3 ri = mm(xm, in);
  auto rot = [&](int u, int w) {
    return ri.m[3 * u] * xm.m[3 * w] + ri.m[3 * u + 1] * xm.m[3 * w + 1] + ri.m[3 * u + 2] * xm.m[3 * w + 2];
  };
  I.mass = mass;
  I.mc = c * mass;
  I.xx = rot(0, 0) + (c.z * c.z + c.y * c.y) * mass;
  I.xy = rot(0, 1) - (c.x * c.y) * mass;
  I.xz = rot(0, 2) - (c.x * c.z) * mass;
  I.yy = rot(1, 1) + (c.z * c.z + c.x * c.x) * mass;
  I.yz = rot(1, 2) - (c.y * c.z) * mass;
  I.zz = rot(2, 2) + (c.y * c.y + c.x * c.x) * mass;
#pragma unroll 1
  for (int j = j0; j < j1; j++) {
    int da = m.jnt_dofadr[j], type = m.jnt_type[j];
    if (type == JNT_FREE || type == JNT_BALL) {
      int lin = type == JNT_FREE ? 3 : 0;
      int rt = type == JNT_FREE ? da + 3 : da;
      for (int k = 0; k < lin; k++) vel = sp_add(vel, sp_scale(ld6(cdof + 6 * (da + k)), v[da + k]));
      // all rotational dofs share one velocity (forward.rs:130-133)
      Sp w = sp_zero();
      for (int k = 0; k < 3; k++) {
        Sp ck = ld6(cdof + 6 * (rt + k));
        acc = sp_add(acc, sp_scale(cross_motion(vel, ck), v[rt + k]));
        w = sp_add(w, sp_scale(ck, v[rt + k]));
      }
      vel = sp_add(vel, w);
    } else {
      Sp ck = ld6(cdof + 6 * da);
      acc = sp_add(acc, sp_scale(cross_motion(vel, ck), v[da]));
      vel = sp_add(vel, sp_scale(ck, v[da]));
    }
  }
  s.fr = sp_add(sym_mul(I, acc), cross_force(vel, sym_mul(I, vel)));
}

// A geom's pose on its body and the half box around it (forward.rs:84-89, 217-232; primitives only).
__device__ __forceinline__ void geom_box(const DModel& m, int g, const Walk& s, const double* pp, V3* x, M3* gm,
                                         V3* half) {
  *x = s.pos + mv(s.mat, ld3(m.geom_pos + 3 * g));
  *gm = mm(s.mat, q_mat(ld4(m.geom_quat + 4 * g)));
  int gt = m.geom_type[g];
  V3 z{pp[m.p_size + 3 * g], pp[m.p_size + 3 * g + 1], pp[m.p_size + 3 * g + 2]};
  V3 hb = z;
  if (gt == GEOM_SPHERE) hb = V3{z.x, z.x, z.x};
  if (gt == GEOM_CAPSULE) hb = V3{z.x, z.x, z.x + z.y};
  if (gt == GEOM_CYLINDER) hb = V3{z.x, z.x, z.y};
  *half = V3{fabs(gm->m[0]) * hb.x + fabs(gm->m[1]) * hb.y + fabs(gm->m[2]) * hb.z,
             fabs(gm->m[3]) * hb.x + fabs(gm->m[4]) * hb.y + fabs(gm->m[5]) * hb.z,
             fabs(gm->m[6]) * hb.x + fabs(gm->m[7]) * hb.y + fabs(gm->m[8]) * hb.z};
}

}  // namespace pg
