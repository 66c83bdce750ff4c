// The whole substep with four lanes per environment, for models of at most
// 16 dofs in one tree whose branches are chains (Ant, legged and armed
// robots, plain chains).
//
// The three phase kernels' tiles of 16 lanes leave three lanes in four idle
// on the tree walks, hand 12 KB an env through HBM and take 10,600 warp
// instructions an Ant env-step. Here eight envs share a warp (2,500 to 4,850
// instructions an env-step, by the contacts) and nothing leaves the SM but the contacts:
//   - every lane walks the trunk, then a limb of its own, in registers;
//   - M, the dof axes and one contact's Jacobian sit in shared memory (2.3 KB
//     an env), rows of the matrix being factored in registers, cyclic over
//     the lanes, the size compiled in;
//   - a contact is its point and frame, with one D: J x and J' f cost 3 sums
//     over the dofs for its four pyramid rows, which are never formed;
//   - M (a - a0) and the rows' residuals are carried along the line search
//     instead of being formed again each iteration.
//
// What bounds it is instruction fetch and dependent-issue latency, not FP64
// (5% of that pipe): one pass runs some 100 KB of code. Two things follow. The
// eight warps of a block start each part of the substep together (a barrier),
// so that a line of code is fetched once for all of them: with blocks of 1 / 2
// / 4 / 8 warps 65536 Ant envs take 3116 / 2457 / 1821 / 1281 us. And every
// factorisation (a0, Newton, damped solve) goes through one call site.
// Twelve warps (168 registers) were no faster than eight (255), and the model
// staged in shared memory was slower than read through L1 (1260 against 1194).
//
// Measured (B200, Ant, us a call with three batches in flight; phase kernels
// before): 16384 envs, one substep 732 -> 334; 65536 envs 2502 -> 1182; 4096
// envs, four substeps, host buffers 905 -> 641; 16 envs 175 -> 152.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "pg_lane.cuh"

namespace pg {
namespace {

constexpr int QUAD_SMEM = 220 * 1024;
constexpr int QUAD_WARPS = 8;  // most warps of a block

__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(FULL, v, 1);
  return v + __shfl_xor_sync(FULL, v, 2);
}
__device__ __forceinline__ void prefetch(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ int quad_or(int v) {
  v |= __shfl_xor_sync(FULL, v, 1);
  return v | __shfl_xor_sync(FULL, v, 2);
}

// An env's shared memory (doubles): velocities, dof axes, two published rows
// (in turn with the bias forces and a vector), the actuator forces or one
// contact's Jacobian, M (packed lower rows; before it is formed the geoms'
// boxes), qpos.
template <int N>
struct QuadLayout {
  static constexpr int ROW = N + 1;  // a published row and its right-hand side
  static constexpr int V = 0, C = V + N, B = C + 6 * N, U = B + 2 * ROW, M = U + (3 * N > QUAD_NU ? 3 * N : QUAD_NU);
  __host__ __device__ static int region(int ngeom) {
    int t = N * (N + 1) / 2;
    return 6 * ngeom > t ? 6 * ngeom : t;
  }
  // 8 envs a warp at a stride of 4 modulo 16 doubles: neither a word shared
  // by an env's lanes nor four consecutive ones meet in a bank
  __host__ __device__ static int stride(int ngeom, int nq) {
    int w = M + region(ngeom) + nq;
    return w + ((4 - w % 16) + 16) % 16;
  }
};

// x <- H^-1 x, H by rows (row i = r + 4 t on lane r, h[t][j], j <= i) and x
// likewise: H = L' D L from the last rows on, two rows a step, which halves
// the chain of divisions and exchanges. A step's two lanes publish their rows
// and right-hand sides in buf; the lanes then take the later row out of the
// earlier one, so the pivots are scalar ones (one division for both). A 2 x 2 inverse in their place is not backward stable, and H's rows
// are nearly dependent wherever contacts are much stiffer than M: with
// impratio 100, or solimp up to 0.9999, it cost two digits of qacc. False if a
// pivot is not positive (the same on the env's four lanes). (Sums of products
// are written so that each product is one FMA.)
template <int N>
__device__ __forceinline__ bool quad_factor_solve(double (&h)[(N + 3) / 4][N], double (&x)[(N + 3) / 4], double* buf, int r) {
  static_assert(N % 2 == 0, "two rows a step");
  constexpr int T = (N + 3) / 4, ROW = QuadLayout<N>::ROW;
  double *r0 = buf, *r1 = buf + ROW;
  bool ok = true;
  double own[T], other[T];  // own pivot's reciprocal; the earlier row's multiple of the later
#pragma unroll
  for (int k0 = N - 2; k0 >= 0; k0 -= 2) {
    const int k1 = k0 + 1, tk = k0 / 4;
    __syncwarp();  // the last step's rows are read
    if (r == k0 % 4) {
#pragma unroll
      for (int j = 0; j <= k0; j++) r0[j] = h[tk][j];
      r0[N] = x[tk];
    }
    if (r == k1 % 4) {
#pragma unroll
      for (int j = 0; j <= k1; j++) r1[j] = h[tk][j];
      r1[N] = x[tk];
    }
    __syncwarp();
    const double d1 = r1[k1], o = r1[k0], x1 = r1[N];
    const double det = r0[k0] * d1 - o * o;
    ok = ok && d1 > 0.0 && det > 0.0;
    const double inv = 1.0 / (d1 * det);  // of both pivots, d1 and det / d1
    const double i1 = det * inv, i0 = d1 * (d1 * inv), mul = o * i1;
    const double x0 = r0[N] - mul * x1;
    if ((r & 2) == (k0 & 2)) {
      own[tk] = (r & 1) ? i1 : i0;
      other[tk] = mul;
    }
    double l0[T], l1[T];
#pragma unroll
    for (int t = 0; t < T; t++) {
      l0[t] = l1[t] = 0.0;
      if (4 * t < k0) {
        if (4 * t + 3 < k0 || 4 * t + r < k0) {
          const double a1 = r1[4 * t + r], a0 = r0[4 * t + r] - mul * a1;
          r0[4 * t + r] = a0;
          l0[t] = a0 * i0;
          l1[t] = a1 * i1;
        }
        x[t] = (x[t] - l1[t] * x1) - l0[t] * x0;
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < k0; j++) {
      const double e0 = r0[j], e1 = r1[j];
#pragma unroll
      for (int t = 0; t < T; t++)
        if (4 * t < k0 && j <= 4 * t + 3) h[t][j] = (h[t][j] - l1[t] * e1) - l0[t] * e0;
    }
  }
  // each pair of unknowns in turn, its products with the later rows summed in s
  double s[T];
#pragma unroll
  for (int t = 0; t < T; t++) s[t] = 0.0;
#pragma unroll
  for (int k0 = 0; k0 < N; k0 += 2) {
    const int tk = k0 / 4;
    double b = x[tk] - s[tk];
    double y = own[tk] * (b - other[tk] * __shfl_xor_sync(FULL, b, 1));  // (the earlier row's lane)
    const double y0 = __shfl_sync(FULL, y, k0 % 4, 4);
    if (r & 1) y = own[tk] * (b - h[tk][k0] * y0);
    if ((r & 2) == (k0 & 2)) x[tk] = y;
    const double y1 = __shfl_sync(FULL, y, k0 % 4 + 1, 4);
#pragma unroll
    for (int t = tk; t < T; t++)
      if (4 * t + r > k0 + 1) s[t] = (s[t] + h[t][k0] * y0) + h[t][k0 + 1] * y1;
  }
  __syncwarp();
  return ok;
}

// The Jacobian of a contact (record o, [field][L]) along its frame, 3 entries
// a dof in j; zero where the env does not have it.
template <int N>
__device__ __noinline__ void quad_jacobian(double* j, const double* cdof, const double* o, int L, bool has, int r) {
  V3 pt{0, 0, 0}, n{0, 0, 0}, tg{0, 0, 0}, t2{0, 0, 0};
  unsigned mk = 0;
  if (has) {
    pt = V3{o[0], o[L], o[2 * L]};
    n = V3{o[LC_N * L], o[(LC_N + 1) * L], o[(LC_N + 2) * L]};
    tg = V3{o[LC_T * L], o[(LC_T + 1) * L], o[(LC_T + 2) * L]};
    t2 = cross(n, tg);
    mk = (unsigned)(unsigned long long)o[LC_MASK * L];
  }
  __syncwarp();  // the place's last reader is done
#pragma unroll 1
  for (int k = r; k < N; k += 4) {
    V3 u = point_vel(ld6(cdof + 6 * k), pt);
    double s = (mk >> k & 1u) ? 1.0 : ((mk >> (16 + k) & 1u) ? -1.0 : 0.0);
    j[3 * k] = s * dot(n, u);
    j[3 * k + 1] = s * dot(tg, u);
    j[3 * k + 2] = s * dot(t2, u);
  }
  __syncwarp();
}

template <int N>
__global__ void __launch_bounds__(32 * QUAD_WARPS, 1) quad_kernel(const __grid_constant__ StepArgs A, const __grid_constant__ LaneArgs P) {
  extern __shared__ __align__(16) double smem[];
  using Q = QuadLayout<N>;
  constexpr int T = (N + 3) / 4;
  const DModel& m = A.m;
  const int nv = m.nv, nq = m.nq, nu = m.nu;
  const int r = threadIdx.x & 3, slot = (threadIdx.x & 31) >> 2;
  int64_t item0 = (int64_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * P.lanes;
  int L = item0 < A.count ? (int)min((int64_t)P.lanes, A.count - item0) : 0;  // envs of this warp
  const bool alive = slot < L;
  // the other slots repeat the warp's last env (a warp past the range: the
  // range's last) and write nothing
  if (L == 0) {
    item0 = A.count - 1;
    L = 1;
  }
  const int es = slot < L ? slot : L - 1;
  const int64_t item = item0 + es;
  const int64_t env = A.start + item;
  const double* pp = A.st.params + (*P.mixed ? env * m.pstride : 0);
  double* ws = smem + (size_t)(threadIdx.x >> 2) * Q::stride(m.ngeom, nq);
  double *v = ws + Q::V, *cdof = ws + Q::C, *buf = ws + Q::B, *fs = buf, *xs = buf, *U = ws + Q::U, *Ms = ws + Q::M,
         *box = Ms, *q = Ms + Q::region(m.ngeom);
  // the warp's slice of the work record: [field][env]
  double* wk = A.work + (size_t)(A.start + item0) * A.k.stride + es;
  double* con = wk + (size_t)A.k.contacts * L;
  double* gmat = wk + (size_t)A.k.geoms * L;
  double* fm = wk + (size_t)A.k.cdof * L;  // crb cdof of each dof, 6 a dof
  const double h = m.timestep;

  for (int k = r; k < nq; k += 4) q[k] = A.st.qpos[env * nq + k];
  for (int k = r; k < N; k += 4) v[k] = k < nv ? A.st.qvel[env * nv + k] : 0.0;
  for (int k = 6 * nv + r; k < 6 * N; k += 4) cdof[k] = 0.0;
  for (int k = r; k < nu; k += 4) prefetch(A.st.ctrl + env * nu + k);
  for (int k = r; k < nv; k += 4) prefetch(A.st.applied + env * nv + k);
  double hd[T], qw[T];
  unsigned chain[T];   // dofs up to i on the chain of own row i
  bool damped = false;
#pragma unroll
  for (int t = 0; t < T; t++) {
    int k = r + 4 * t;
    bool in = k < nv;
    hd[t] = in ? pp[m.p_damping + k] : 0.0;
    qw[t] = in ? A.st.qacc[env * nv + k] : 0.0;
    chain[t] = in ? (unsigned)m.body_dofmask[m.dof_body[k]] & ((2u << k) - 1u) : 0u;
    damped |= hd[t] != 0.0;
  }
  damped = quad_or(damped) != 0;
  int status_all = P.sidx == 0 ? 0 : A.st.status[env];
  int iters = 0, ncon = 0, nr = 0;
  __syncwarp();

#pragma unroll 1
  for (int sub = 0; sub < P.nsub; sub++) {
    const int sidx = P.sidx + sub;
    int status = 0;
    if (blockDim.x > 32) __syncthreads();
    // ------------------------------------------------ tree walk
    {
      double tr[LANE_DEPTH * 16], lb[LANE_DEPTH * 16];
      auto geoms = [&](int b, int g0, int step, const Walk& s) {
        if (m.npair > 0)
#pragma unroll 1
          for (int g = P.t.body_gadr[b] + g0; g < P.t.body_gadr[b + 1]; g += step) {
            V3 x, half;
            M3 gm;
            geom_box(m, g, s, pp, &x, &gm, &half);
            st3(box + 6 * g, x);
            st3(box + 6 * g + 3, half);
            if (alive)
#pragma unroll
              for (int t = 0; t < 9; t++) gmat[(size_t)(9 * g + t) * L] = gm.m[t];
          }
      };
      auto keep = [&](double* o, const Sym& I, const Sp& fr) {
        o[0] = I.mass;
        st3(o + 1, I.mc);
        o[4] = I.xx;
        o[5] = I.xy;
        o[6] = I.xz;
        o[7] = I.yy;
        o[8] = I.yz;
        o[9] = I.zz;
        st6(o + 10, fr);
      };
      auto join = [&](const double* o, Sym& I, Sp& fr) {
        I.mass += o[0];
        I.mc = I.mc + ld3(o + 1);
        I.xx += o[4];
        I.xy += o[5];
        I.xz += o[6];
        I.yy += o[7];
        I.yz += o[8];
        I.zz += o[9];
        fr = sp_add(fr, ld6(o + 10));
      };
      // a body whose subtree is summed: bias force and momentum of its dofs
      auto leave = [&](int b, const Sym& I, const Sp& fr, bool write) {
        int i0 = m.body_dofadr[b], i1 = i0 + m.body_dofnum[b];
#pragma unroll 1
        for (int i = i0; i < i1; i++) {
          Sp ci = ld6(cdof + 6 * i);
          Sp fi = sym_mul(I, ci);
          fs[i] = -sp_dot(ci, fr);
          if (write) {
            double* o = fm + (size_t)6 * i * L;
            o[0] = fi.ang.x;
            o[L] = fi.ang.y;
            o[2 * L] = fi.ang.z;
            o[3 * L] = fi.lin.x;
            o[4 * L] = fi.lin.y;
            o[5 * L] = fi.lin.z;
          }
        }
      };
      Walk s, end;
      walk_world(m, s);
      geoms(0, r, 4, s);
      Sym I{};
      Sp fr = sp_zero();
#pragma unroll 1
      for (int l0 = 0; l0 == 0 || l0 < P.t.limb_n; l0 += 4) {
        // every lane walks the trunk (the same values), then its limb
        int l = l0 + r;
        int a0 = l < P.t.limb_n ? P.t.limb_adr[l] : 0, a1 = l < P.t.limb_n ? P.t.limb_adr[l + 1] : 0;
        if (l0 > 0) s = end;
#pragma unroll 1
        for (int k = l0 > 0 ? 0 : -P.t.trunk_n; k < P.t.limb_max; k++) {
          if (l0 == 0 && k == 0 && P.t.limb_n > 4) end = s;
          if (k < 0 || a0 + k < a1) {
            int b = k < 0 ? P.t.trunk[P.t.trunk_n + k] : P.t.limb_body[a0 + k];
            walk_body(m, P.t, b, q, v, cdof, pp, 1, s);
            if (k < 0) geoms(b, r, 4, s);
            else geoms(b, 0, 1, s);
            keep(k < 0 ? tr + 16 * (P.t.trunk_n + k) : lb + 16 * k, s.I, s.fr);
          }
          __syncwarp();
        }
        Sym J{};
        Sp jr = sp_zero();
#pragma unroll 1
        for (int k = P.t.limb_max - 1; k >= 0; k--) {
          if (a0 + k < a1) {
            join(lb + 16 * k, J, jr);
            leave(P.t.limb_body[a0 + k], J, jr, alive);
          }
          __syncwarp();
        }
        double o[16];
        keep(o, J, jr);
        join(o, I, fr);
      }
      I.mass = quad_sum(I.mass);
      I.mc = V3{quad_sum(I.mc.x), quad_sum(I.mc.y), quad_sum(I.mc.z)};
      I.xx = quad_sum(I.xx);
      I.xy = quad_sum(I.xy);
      I.xz = quad_sum(I.xz);
      I.yy = quad_sum(I.yy);
      I.yz = quad_sum(I.yz);
      I.zz = quad_sum(I.zz);
      fr.ang = V3{quad_sum(fr.ang.x), quad_sum(fr.ang.y), quad_sum(fr.ang.z)};
      fr.lin = V3{quad_sum(fr.lin.x), quad_sum(fr.lin.y), quad_sum(fr.lin.z)};
#pragma unroll 1
      for (int k = P.t.trunk_n - 1; k >= 0; k--) {
        join(tr + 16 * k, I, fr);
        leave(P.t.trunk[k], I, fr, alive && r == 0);
      }
      __syncwarp();
    }
    if (blockDim.x > 32) __syncthreads();
    // ------------------------------------------------ collision
    ncon = 0;
#pragma unroll 1
    for (int p0 = 0; p0 < m.npair; p0 += 128) {
      // the lane's pairs p0 + r, p0 + r + 4, ... whose boxes meet
      unsigned mine = 0;
#pragma unroll 1
      for (int k = 0; k < 32 && p0 + 4 * k < m.npair; k++) {
        const int pr = p0 + 4 * k + r;
        bool keep = alive && pr < m.npair;
        const int pack = P.t.pair_pack[keep ? pr : 0];
        const int g1 = pack & 255, g2 = pack >> 8 & 255, ty1 = pack >> 16 & 15, ty2 = pack >> 20;
        if (ty1 != GEOM_PLANE && ty2 != GEOM_PLANE) {
          V3 c1 = ld3(box + 6 * g1), h1 = ld3(box + 6 * g1 + 3), c2 = ld3(box + 6 * g2), h2 = ld3(box + 6 * g2 + 3);
          keep = keep && !(fabs(c1.x - c2.x) > h1.x + h2.x + m.margin || fabs(c1.y - c2.y) > h1.y + h2.y + m.margin ||
                           fabs(c1.z - c2.z) > h1.z + h2.z + m.margin);
        } else if (ty1 != ty2) {
          // a plane has no box; a geom whose box lies clear of it on the
          // plane's upper side touches it nowhere (the slack covers rounding)
          const int gpl = ty1 == GEOM_PLANE ? g1 : g2, go = ty1 == GEOM_PLANE ? g2 : g1;
          const double* pm = gmat + (size_t)9 * gpl * L;
          V3 pn{pm[2 * L], pm[5 * L], pm[8 * L]};
          V3 dc = ld3(box + 6 * go) - ld3(box + 6 * gpl), hb = ld3(box + 6 * go + 3);
          double reach = fabs(pn.x) * hb.x + fabs(pn.y) * hb.y + fabs(pn.z) * hb.z;
          double dist = dot(dc, pn);
          keep = keep && !(dist > (reach + m.margin) * (1.0 + 1e-9) + 1e-9 * (1.0 + fabs(dist)));
        }
        if (keep) mine |= 1u << k;
      }
      // narrow phase: every lane takes the next of its own
      while (__any_sync(FULL, mine != 0)) {
        bool keep = mine != 0;
        const int pr = keep ? p0 + 4 * (__ffs(mine) - 1) + r : 0;
        mine &= mine - 1;
        const int pack = P.t.pair_pack[pr];
        const int g1 = pack & 255, g2 = pack >> 8 & 255, ty1 = pack >> 16 & 15, ty2 = pack >> 20;
        const bool flat = (ty1 == GEOM_PLANE) != (ty2 == GEOM_PLANE);
        const int gpl = ty1 == GEOM_PLANE ? g1 : g2, go = ty1 == GEOM_PLANE ? g2 : g1;
        Hits hits;
        hits.n = 0;
        int nh = 0;
        if (keep) {
          unsigned t1 = (unsigned)pp[m.p_contype + g1], a1 = (unsigned)pp[m.p_conaff + g1];
          unsigned t2 = (unsigned)pp[m.p_contype + g2], a2 = (unsigned)pp[m.p_conaff + g2];
          keep = (t1 & a2) != 0 || (t2 & a1) != 0;
        }
        if (keep) {
          const int to = ty1 == GEOM_PLANE ? ty2 : ty1;
          if (flat && (to == GEOM_SPHERE || to == GEOM_CAPSULE)) {
            // collision.rs:203-212 at the centre or at both ends of the axis
            const double* pm = gmat + (size_t)9 * gpl * L;
            V3 pn{pm[2 * L], pm[5 * L], pm[8 * L]};
            V3 pc = ld3(box + 6 * gpl), x = ld3(box + 6 * go);
            double rad = pp[m.p_size + 3 * go];
            V3 ax{0, 0, 0}, e{0, 0, 0};
            if (to == GEOM_CAPSULE) {
              const double* gm = gmat + (size_t)9 * go * L;
              ax = V3{gm[2 * L], gm[5 * L], gm[8 * L]};
              e = ax * pp[m.p_size + 3 * go + 1];
            }
            V3 nn = gpl == g1 ? pn : -pn;
            for (int k = 0; k < (to == GEOM_CAPSULE ? 2 : 1); k++) {
              V3 cc = k == 0 ? x - e : x + e;
              double dist = dot(cc - pc, pn);
              double depth = rad - dist;
              if (depth > -m.margin) hits.h[nh++] = Hit{cc - (pn * (dist + rad)) * 0.5, nn, ax, depth};
            }
          } else {
            auto pose = [&](int g, int ty) {
              M3 gm;
#pragma unroll
              for (int t = 0; t < 9; t++) gm.m[t] = gmat[(size_t)(9 * g + t) * L];
              return GPose{ty, ld3(box + 6 * g), gm,
                           V3{pp[m.p_size + 3 * g], pp[m.p_size + 3 * g + 1], pp[m.p_size + 3 * g + 2]}, 0};
            };
            collide_primitive(pose(g1, ty1), pose(g2, ty2), m.margin, hits);
            nh = hits.n < MAX_HITS ? hits.n : MAX_HITS;
          }
        }
        __syncwarp();
        if (!__any_sync(FULL, nh > 0)) continue;
        // the env's contacts in the lanes' order
        int inc = nh, y = __shfl_up_sync(FULL, inc, 1, 4);
        if (r >= 1) inc += y;
        y = __shfl_up_sync(FULL, inc, 2, 4);
        if (r >= 2) inc += y;
        const int at = ncon + inc - nh;
        ncon += __shfl_sync(FULL, inc, 3, 4);
        if (nh > 0) {
          int b1 = m.geom_body[g1], b2 = m.geom_body[g2];
          unsigned k1 = (unsigned)m.body_dofmask[b1], k2 = (unsigned)m.body_dofmask[b2];
          double mu = fmax(pp[m.p_friction + g1], pp[m.p_friction + g2]);
          double tran = pp[m.p_body_invw + 2 * b1] + pp[m.p_body_invw + 2 * b2];
          double dpyr = 2.0 * mu * mu * (1.0 + mu * mu) * tran / m.impratio;
#pragma unroll 1
          for (int k = 0; k < nh; k++) {
            if (at + k >= m.maxcon) {
              status |= ST_CAP_EXCEEDED;
              break;
            }
            double* o = con + (size_t)(at + k) * LC_STRIDE * L;
            const Hit& hk = hits.h[k];
            V3 tg1, tg2;
            contact_frame(hk.normal, hk.tangent, &tg1, &tg2);
            o[(LC_POS + 0) * L] = hk.pos.x;
            o[(LC_POS + 1) * L] = hk.pos.y;
            o[(LC_POS + 2) * L] = hk.pos.z;
            o[(LC_N + 0) * L] = hk.normal.x;
            o[(LC_N + 1) * L] = hk.normal.y;
            o[(LC_N + 2) * L] = hk.normal.z;
            o[(LC_T + 0) * L] = tg1.x;
            o[(LC_T + 1) * L] = tg1.y;
            o[(LC_T + 2) * L] = tg1.z;
            o[LC_MU * L] = mu;
            double D = 0.0;
            if (hk.depth > 0.0) {
              double imp = row_impedance(m.solimp, -hk.depth);
              D = 1.0 / fmax((1.0 - imp) / imp * dpyr, 1e-15);
              o[LC_OFF * L] = imp * -hk.depth;  // completed once the velocities are taken
            }
            o[LC_D * L] = D;
            o[LC_MASK * L] = (double)((k2 & ~k1) | (k1 & ~k2) << 16);
          }
        }
        __syncwarp();
      }
    }
    if (ncon > m.maxcon) ncon = m.maxcon;
    __syncwarp();
    if (blockDim.x > 32) __syncthreads();
    // ------------------------------------------------ passive and actuator forces
    for (int j = r; j < m.njnt; j += 4) {
      double kp = m.jnt_stiffness[j];
      int t = m.jnt_type[j];
      if (kp != 0.0 && (t == JNT_HINGE || t == JNT_SLIDE)) fs[m.jnt_dofadr[j]] -= kp * (q[m.jnt_qposadr[j]] - m.jnt_springref[j]);
    }
#pragma unroll 1
    for (int u = r; u < nu; u += 4) {
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
      double fu = pp[m.p_gain + u] * c + pp[m.p_bias + 3 * u] + pp[m.p_bias + 3 * u + 1] * (gear * ls) +
                  pp[m.p_bias + 3 * u + 2] * (gear * vs);
      if (m.act_forcelimited[u]) fu = clampd(fu, m.act_forcerange[2 * u], m.act_forcerange[2 * u + 1]);
      U[u] = fu;
    }
    __syncwarp();
    double f[T], a[T], mt[T], H[T][N];
#pragma unroll
    for (int t = 0; t < T; t++) {
      int k = r + 4 * t;
      f[t] = 0.0;
      if (k < nv) {
        double s = 0.0;
        for (int i = m.dofact_adr[k]; i < m.dofact_adr[k + 1]; i++) {
          int u = m.dofact_u[i];
          s += m.act_gear[u] * m.dofact_coef[i] * U[u];
        }
        f[t] = fs[k] + A.st.applied[env * nv + k] - hd[t] * v[k] + s;
      }
    }
    // ------------------------------------------------ M and a0 = M^-1 f
    {
      Sp fi[T];
#pragma unroll
      for (int t = 0; t < T; t++) {
        int k = r + 4 * t;
        const double* o = fm + (size_t)6 * (k < nv ? k : 0) * L;
        fi[t] = Sp{V3{o[0], o[L], o[2 * L]}, V3{o[3 * L], o[4 * L], o[5 * L]}};
      }
#pragma unroll
      for (int j = 0; j < N; j++) {
        Sp cj = ld6(cdof + 6 * j);
#pragma unroll
        for (int t = j / 4; t < T; t++) {
          int i = r + 4 * t;
          double e = (chain[t] >> j & 1u) ? sp_dot(cj, fi[t]) : 0.0;
          if (i == j) e += j < nv ? m.dof_armature[j] : 1.0;
          if (j <= i && i < N) Ms[tri(i, j)] = e;
        }
      }
    }
    __syncwarp();
    // ------------------------------------------------ solves
    // One loop runs every factorisation (the code of one is most of the
    // instruction cache a substep needs): a0 = M^-1 f, then with constraint
    // rows the cost gate of the warm start and the Newton iterations, then
    // the damped solve.
    enum { SOLVE_A0, GATE, NEWTON, DAMPED };
    const double tc = fmax(m.solref[0], 2.0 * h), dr = m.solref[1], dmax = m.solimp[1];
    const double rb = 2.0 / (dmax * tc), rk = 1.0 / (dmax * dmax * tc * tc * dr * dr);
    const int maxit = m.iterations > 1 ? m.iterations : 1;
    const int cmax = __reduce_max_sync(FULL, alive ? ncon : 0);
    auto contact_on = [&](int c) { return alive && c < ncon && con[((size_t)c * LC_STRIDE + LC_D) * L] != 0.0; };
    // the Jacobian of contact c along its frame, 3 entries a dof, in U (formed
    // again where another contact's stands there)
    int in_u = -1;
    auto jac_of = [&](int c, bool has) -> const double* {
      if (in_u != c) quad_jacobian<N>(U, cdof, con + (size_t)c * LC_STRIDE * L, L, has, r);
      in_u = c;
      return U;
    };
    double limD[T], limE[T], x[T];
    double scale = 0.0;
    bool run0 = false, run = false;
    unsigned prev = 0;  // own limit rows active in the previous iteration
    nr = iters = 0;
    int kind = SOLVE_A0;
#pragma unroll 1
    while (true) {
      double mp[T];
      if (kind != GATE) {
        double s[T];
        unsigned act = 0;
#pragma unroll
        for (int t = 0; t < T; t++) {
          int i = r + 4 * t;
          double add = 0.0;
          s[t] = 0.0;
          if (kind == DAMPED) add = h * hd[t];
          if (kind == NEWTON && limD[t] != 0.0 && limE[t] < 0.0) {
            s[t] = limD[t] * limE[t];
            add = fabs(limD[t]);
            act |= 1u << t;
          }
          const double* row = Ms + tri(i < N ? i : N - 1, 0);
#pragma unroll
          for (int j = 0; j < N; j++)
            if (j <= 4 * t + 3) H[t][j] = j <= i ? row[j] + (j == i ? add : 0.0) : 0.0;
        }
        if (kind == NEWTON) {
          // gradient and active set, with H = M + J_A' D J_A
          if (run) iters++;
          bool same = act == prev;
          prev = act;
#pragma unroll 1
          for (int c = 0; c < cmax; c++) {
            bool has = contact_on(c) && run0;
            const double* j = jac_of(c, contact_on(c));
            double f0 = 0, f1 = 0, f2 = 0, w00 = 0, w01 = 0, w11 = 0, w02 = 0, w22 = 0;
            unsigned bits = 0;
            unsigned long long rec = 0;
            if (has) {
              const double* o = con + (size_t)c * LC_STRIDE * L;
              double mu = o[LC_MU * L], D = o[LC_D * L];
              double e0 = o[LC_E * L], e1 = mu * o[(LC_E + 1) * L], e2 = mu * o[(LC_E + 2) * L];
              rec = (unsigned long long)o[LC_MASK * L];
              double x0 = e0 + e1, x1 = e0 - e1, x2 = e0 + e2, x3 = e0 - e2;
              double b0 = x0 < 0.0 ? D : 0.0, b1 = x1 < 0.0 ? D : 0.0, b2 = x2 < 0.0 ? D : 0.0, b3 = x3 < 0.0 ? D : 0.0;
              x0 *= b0;
              x1 *= b1;
              x2 *= b2;
              x3 *= b3;
              f0 = ((x0 + x1) + x2) + x3;
              f1 = mu * (x0 - x1);
              f2 = mu * (x2 - x3);
              w00 = ((b0 + b1) + b2) + b3;
              w01 = mu * (b0 - b1);
              w11 = mu * mu * (b0 + b1);
              w02 = mu * (b2 - b3);
              w22 = mu * mu * (b2 + b3);
              // the contact's previous set sits beside its masks
              bits = 16u | (b0 > 0.0 ? 1u : 0u) | (b1 > 0.0 ? 2u : 0u) | (b2 > 0.0 ? 4u : 0u) | (b3 > 0.0 ? 8u : 0u);
              if ((unsigned)(rec >> 32) != bits) same = false;
            }
            __syncwarp();
            if (has && r == 0)
              con[((size_t)c * LC_STRIDE + LC_MASK) * L] = (double)((rec & 0xffffffffull) | (unsigned long long)bits << 32);
            if (__any_sync(FULL, w00 != 0.0)) {
              double y0[T], y1[T], y2[T];
#pragma unroll
              for (int t = 0; t < T; t++) {
                int i = r + 4 * t < N ? r + 4 * t : N - 1;
                double j0 = j[3 * i], j1 = j[3 * i + 1], j2 = j[3 * i + 2];
                s[t] += j0 * f0 + j1 * f1 + j2 * f2;
                y0[t] = w00 * j0 + w01 * j1 + w02 * j2;
                y1[t] = w01 * j0 + w11 * j1;
                y2[t] = w02 * j0 + w22 * j2;
              }
#pragma unroll
              for (int k = 0; k < N; k++) {
                double j0 = j[3 * k], j1 = j[3 * k + 1], j2 = j[3 * k + 2];
#pragma unroll
                for (int t = k / 4; t < T; t++) H[t][k] += y0[t] * j0 + y1[t] * j1 + y2[t] * j2;
              }
            }
          }
          double gs = 0.0;
#pragma unroll
          for (int t = 0; t < T; t++) {
            if (r + 4 * t >= N) s[t] = mt[t] = 0.0;
            x[t] = -(mt[t] + s[t]);
            gs += x[t] * x[t];
          }
          gs = quad_sum(gs);
          same = quad_or(!same) == 0;
          if (run && (sqrt(gs) < m.tolerance * scale || (nr <= 128 && same && iters > 1))) run = false;
          if (!__any_sync(FULL, run)) {
            // qfrc_constraint = -J' D (J a - aref) over the active rows
            if (run0) {
#pragma unroll
              for (int t = 0; t < T; t++) f[t] -= s[t];
            }
            if (!__any_sync(FULL, damped)) break;
            kind = DAMPED;
            continue;
          }
        } else {
#pragma unroll
          for (int t = 0; t < T; t++) x[t] = f[t];
        }
        const bool ok = quad_factor_solve<N>(H, x, buf, r);
        if (kind == DAMPED) {
          if (damped) {
            if (!ok) status |= ST_NOT_SPD;
#pragma unroll
            for (int t = 0; t < T; t++) a[t] = x[t];
          }
          break;
        }
        if (kind == SOLVE_A0) {
          if (!ok) status |= ST_NOT_SPD;
          // the rows: violated limits by dof, touching contacts
          double ss = 0.0;
#pragma unroll
          for (int t = 0; t < T; t++) {
            int k = r + 4 * t;
            a[t] = x[t];
            mt[t] = 0.0;
            ss += f[t] * f[t];  // M a0 = f
            limD[t] = limE[t] = 0.0;
          }
#pragma unroll 1
          for (int k = r; k < nv; k += 4) {
            int qa = P.t.dof_limq[k];
            double lo = 0.0, hi = 0.0;
            if (qa >= 0) {
              lo = q[qa] - P.t.dof_range[2 * k];
              hi = P.t.dof_range[2 * k + 1] - q[qa];
            }
            if (lo < 0.0 || hi < 0.0) {
              double sg = lo < 0.0 ? 1.0 : -1.0, sep = lo < 0.0 ? lo : hi;
              double imp = row_impedance(m.solimp, sep);
              double D = sg / fmax((1.0 - imp) / imp * pp[m.p_dof_invw + k], 1e-15);
              double e = rb * (sg * v[k]) + rk * imp * sep;  // -aref
#pragma unroll
              for (int t = 0; t < T; t++)
                if (k == r + 4 * t) {
                  limD[t] = D;
                  limE[t] = e + sg * a[t];
                }
              nr++;
            }
          }
          nr += __shfl_xor_sync(FULL, nr, 1);
          nr += __shfl_xor_sync(FULL, nr, 2);
          scale = 1.0 + sqrt(quad_sum(ss));
          // (a contact's residual belongs to lane c mod 4, every lane reads it)
#pragma unroll 1
          for (int c = 0; c < cmax; c++) {
            bool has = contact_on(c);
            const double* j = jac_of(c, has);
            double v0 = 0, v1 = 0, v2 = 0, e0 = 0, e1 = 0, e2 = 0;
#pragma unroll
            for (int t = 0; t < T; t++) {
              int k = r + 4 * t;
              if (k < N) {
                v0 += j[3 * k] * v[k];
                v1 += j[3 * k + 1] * v[k];
                v2 += j[3 * k + 2] * v[k];
                e0 += j[3 * k] * a[t];
                e1 += j[3 * k + 1] * a[t];
                e2 += j[3 * k + 2] * a[t];
              }
            }
            e0 = quad_sum(rb * v0 + e0);
            e1 = quad_sum(rb * v1 + e1);
            e2 = quad_sum(rb * v2 + e2);
            if (has) {
              double* o = con + (size_t)c * LC_STRIDE * L;
              if (r == (c & 3)) {
                o[LC_E * L] = e0 + rk * o[LC_OFF * L];
                o[(LC_E + 1) * L] = e1;
                o[(LC_E + 2) * L] = e2;
              }
              nr += 4;
            }
          }
          __syncwarp();
          run0 = run = alive && nr > 0 && !(status & ST_NOT_SPD);
          if (!run0) {
#pragma unroll
            for (int t = 0; t < T; t++) limD[t] = 0.0;
          }
          if (__any_sync(FULL, run0)) {
            kind = A.warm_mode == WARM_REF_PREV_QACC ? GATE : NEWTON;
          } else {
            if (!__any_sync(FULL, damped)) break;
            kind = DAMPED;
          }
          continue;
        }
        if (!ok) run = false;
      } else {
#pragma unroll
        for (int t = 0; t < T; t++) x[t] = r + 4 * t < N ? qw[t] - a[t] : 0.0;
      }
      // the step x: M x, and J x of each contact
#pragma unroll
      for (int t = 0; t < T; t++) {
        mp[t] = 0.0;
        if (r + 4 * t < N) xs[r + 4 * t] = x[t];
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < N; j++) {
        double xj = xs[j];
#pragma unroll
        for (int t = 0; t < T; t++) {
          int i = r + 4 * t < N ? r + 4 * t : N - 1;
          mp[t] += Ms[i >= j ? tri(i, 0) + j : tri(j, 0) + i] * xj;
        }
      }
#pragma unroll 1
      for (int c = 0; c < cmax; c++) {
        bool has = contact_on(c) && run0;
        const double* j = jac_of(c, contact_on(c));
        double p0 = 0, p1 = 0, p2 = 0;
#pragma unroll
        for (int t = 0; t < T; t++) {
          int k = r + 4 * t;
          if (k < N) {
            p0 += j[3 * k] * x[t];
            p1 += j[3 * k + 1] * x[t];
            p2 += j[3 * k + 2] * x[t];
          }
        }
        p0 = quad_sum(p0);
        p1 = quad_sum(p1);
        p2 = quad_sum(p2);
        if (has && r == (c & 3)) {
          double* o = con + (size_t)c * LC_STRIDE * L;
          o[LC_P * L] = p0;
          o[(LC_P + 1) * L] = p1;
          o[(LC_P + 2) * L] = p2;
        }
      }
      __syncwarp();
      double mpp = 0.0, mpg = 0.0;
#pragma unroll
      for (int t = 0; t < T; t++) {
        mpp += x[t] * mp[t];
        mpg += x[t] * mt[t];
      }
      mpp = quad_sum(mpp);
      mpg = quad_sum(mpg);
      // the derivatives of the cost along x at al; in the gate, the rows'
      // costs at 0 and 1 instead
      double al = 0.0, lo = 0.0, hi = INFINITY, ltol = 0.0;
      bool ls = run;
      double c0 = 0.0;
#pragma unroll 1
      for (int it = -1; it < 50 && __any_sync(FULL, ls); it++) {
        double d1 = 0.0, d2 = 0.0;
        auto row = [&](double D, double e, double jp) {
          double y = e + al * jp;
          if (y < 0.0) {
            double dq = kind == GATE ? 0.5 * D * y : D * jp;
            d1 += dq * y;
            d2 += dq * jp;
          }
        };
#pragma unroll
        for (int t = 0; t < T; t++)
          if (limD[t] != 0.0) row(fabs(limD[t]), limE[t], limD[t] > 0.0 ? x[t] : -x[t]);
#pragma unroll 1
        for (int c = r; c < cmax; c += 4) {
          if (run && contact_on(c)) {
            const double* o = con + (size_t)c * LC_STRIDE * L;
            double D = o[LC_D * L], mu = o[LC_MU * L], e0 = o[LC_E * L], q0 = o[LC_P * L];
#pragma unroll
            for (int k = 1; k < 3; k++) {
              double e1 = mu * o[(LC_E + k) * L], q1 = mu * o[(LC_P + k) * L];
              row(D, e0 + e1, q0 + q1);
              row(D, e0 - e1, q0 - q1);
            }
          }
        }
        __syncwarp();
        d1 = quad_sum(d1);
        d2 = quad_sum(d2) + mpp;
        if (kind == GATE) {
          // the cost gate (newton.rs:238-245): the previous acceleration
          // where it is cheaper than a0, whose quadratic term is zero
          if (it < 0) {
            c0 = d1;
            al = 1.0;
          } else {
            if (!(run && d1 + 0.5 * mpp < c0)) al = 0.0;
            break;
          }
          continue;
        }
        // exact line search on the piecewise quadratic along x
        d1 += al * mpp + mpg;
        if (it < 0) {
          ltol = 1e-12 * fmax(fabs(d1), 1e-30);
          al = 1.0;
        } else if (ls) {
          if (fabs(d1) <= ltol) {
            ls = false;
          } else {
            if (d1 < 0.0) lo = al;
            else hi = al;
            double next = al - d1 / fmax(d2, 1e-30);
            if (next <= lo || next >= hi) next = isfinite(hi) ? 0.5 * (lo + hi) : 2.0 * fmax(al, lo);
            if (fabs(next - al) <= 1e-14 * fmax(fabs(al), 1.0)) ls = false;
            al = next;
          }
        }
      }
      if (run && !(kind == GATE && al == 0.0)) {
#pragma unroll
        for (int t = 0; t < T; t++) {
          a[t] = kind == GATE ? qw[t] : a[t] + al * x[t];
          mt[t] += al * mp[t];
          if (limD[t] != 0.0) limE[t] += al * (limD[t] > 0.0 ? x[t] : -x[t]);
        }
#pragma unroll 1
        for (int c = r; c < ncon; c += 4) {
          double* o = con + (size_t)c * LC_STRIDE * L;
          if (o[LC_D * L] != 0.0)
            for (int t = 0; t < 3; t++) o[(LC_E + t) * L] += al * o[(LC_P + t) * L];
        }
        if (iters >= maxit) run = false;
      }
      __syncwarp();
      kind = NEWTON;
    }
    // ------------------------------------------------ integration
    status = quad_or(status);
    const bool good = !(status & ST_NOT_SPD);
    if (good) {
#pragma unroll
      for (int t = 0; t < T; t++) {
        int k = r + 4 * t;
        if (k < nv) {
          double vk = v[k] + h * a[t];
          qw[t] = (vk - v[k]) / h;
          v[k] = vk;
        }
      }
    } else {
      iters = nr = 0;
    }
    __syncwarp();
    if (good)
#pragma unroll 1
      for (int j = r; j < m.njnt; j += 4) {
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
    __syncwarp();
    if (A.qpos_out && alive)
      for (int k = r; k < nq; k += 4) A.qpos_out[((size_t)item * A.nstep + sidx) * nq + k] = q[k];
    status_all |= status;
  }
  if (alive) {
    for (int k = r; k < nq; k += 4) A.st.qpos[env * nq + k] = q[k];
#pragma unroll
    for (int t = 0; t < T; t++) {
      int k = r + 4 * t;
      if (k < nv) {
        A.st.qvel[env * nv + k] = v[k];
        A.st.qacc[env * nv + k] = qw[t];
      }
    }
    if (r == 0) {
      A.st.iters[env] = iters;
      A.st.ncon[env] = ncon;
      A.st.nrows[env] = nr;
      A.st.status[env] = status_all;
    }
  }
}

}  // namespace

cudaError_t launch_quad(const StepArgs& a, const LaneArgs& p, cudaStream_t s) {
  int64_t warps = ((int64_t)a.count + p.lanes - 1) / p.lanes;
  if (warps <= 0) return cudaSuccess;
  auto go = [&](auto tag) {
    constexpr int N = decltype(tag)::value;
    const size_t each = (size_t)8 * QuadLayout<N>::stride(a.m.ngeom, a.m.nq) * sizeof(double);
    const int per = (int)std::min<int64_t>(std::min<int64_t>(QUAD_WARPS, QUAD_SMEM / each), (warps + p.sms - 1) / p.sms);
    size_t smem = per * each;
    cudaError_t e = cudaFuncSetAttribute(quad_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, QUAD_SMEM);
    if (e != cudaSuccess) return e;
    quad_kernel<N><<<(unsigned)((warps + per - 1) / per), 32 * per, smem, s>>>(a, p);
    return cudaGetLastError();
  };
  if (a.m.nv <= 8) return go(std::integral_constant<int, 8>{});
  if (a.m.nv <= 12) return go(std::integral_constant<int, 12>{});
  if (a.m.nv <= 14) return go(std::integral_constant<int, 14>{});
  return go(std::integral_constant<int, 16>{});
}

}  // namespace pg
