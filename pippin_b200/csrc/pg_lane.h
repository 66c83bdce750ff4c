// Launcher of the one-lane-per-env substep (pg_lane.cu).
#pragma once
#include <cuda_runtime.h>

#include "pg_kernels.h"

namespace pg {

// which substep a model's Newton steps take: the three phase kernels, one
// lane an env (no constraint rows possible), or four
enum { STEP_PHASES = 0, STEP_LANES = 1, STEP_QUADS = 2 };
// limits of the models the lane and quad kernels take (sizes of its per-lane arrays)
constexpr int LANE_NV = 8;      // dofs (lane)
constexpr int QUAD_NV = 16;     // dofs (quad)
constexpr int LANE_NQ = 24;     // positions
constexpr int LANE_GEOM = 32;   // geoms
constexpr int QUAD_NU = 32;     // actuators (quad)
constexpr int LANE_DEPTH = 8;   // tree levels below the world
// a contact in the lane's slice of the work record (doubles): point, normal,
// first tangent, friction, D (0: not touching), the constant part of its
// residual, its dof masks, residual and its change along the search direction
enum { LC_POS = 0, LC_N = 3, LC_T = 6, LC_MU = 9, LC_D = 10, LC_OFF = 11, LC_MASK = 14, LC_E = 15, LC_P = 18,
       LC_STRIDE = 21 };

// What these kernels read beside DModel: kept out of it, since the phase
// kernels' blocks each stage DModel and its arrays in shared memory.
struct LaneModel {
  // the tree as a trunk (bodies with one child each, from the root down to
  // the first that branches) and the chains that leave its end (limb_n = -1:
  // a branch branches again)
  const int* trunk;     // [trunk_n]
  const int* limb_adr;  // [limb_n + 1] into limb_body
  const int* limb_body;
  const int* body_gadr;  // [nb + 1] first geom of each body (geoms sorted by body)
  int trunk_n, limb_n, limb_max;  // limb_max: bodies of the longest limb
  const double* jnt_unit;   // jnt_axis at unit length
  const int* dof_limq;      // position address of a limited hinge or slide's dof, else -1
  const double* dof_range;  // [nv][2] its range
  const int* pair_pack;     // [npair] g1 | g2 << 8 | type1 << 16 | type2 << 20 (models of at most 256 geoms)
};

struct LaneArgs {
  LaneModel t;
  // on the device: 0 while the envs' physical parameters are all env 0's,
  // whose block every env then reads (one address for the whole warp); 1 once
  // pg_set_param has written one. Read when the kernel runs, so that a
  // captured step replays with the parameters of that time.
  const int* mixed;
  // the blocks' entries from p_mass up to p_qpos_reset, a column an env, in
  // groups of 32: what a lane reads together lies together (one lane an env)
  const double* columns;
  int lanes;           // envs a warp takes (1..32)
  int sms;             // SMs of the GPU
  int sidx, nsub;      // substeps [sidx, sidx + nsub) of the call
};

// Substeps [p.sidx, p.sidx + p.nsub) of envs [a.start, a.start + a.count), one launch.
cudaError_t launch_lane(const StepArgs& a, const LaneArgs& p, cudaStream_t s);
// The same with four lanes per env (a.m.limb_n >= 0; p.lanes at most 8).
cudaError_t launch_quad(const StepArgs& a, const LaneArgs& p, cudaStream_t s);

}  // namespace pg
