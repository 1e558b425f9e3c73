// SQP-IK on the GPU: multi-seed sequential quadratic programming IK with
// joint limits as hard bounds on the step -- the drop-in for the sqp_ik_cuda
// custom call (src/pyroffi/cuda_kernels/_sqp_ik_cuda_kernel.cu:70-460,
// handler :462-591).
//
// Per seed, max_iter iterations: residual and Jacobian of every EE; exit when
// all EEs are within (eps_pos, eps_ori); rows weighted by (pos_weight,
// ori_weight); Jacobi column scaling; H = Js^T Js + lambda I and g = Js^T f
// (FP64 in the reference); the step's box in scaled space,
// ((lower - q) s, (upper - q) s) (0 for fixed joints); the unconstrained
// Newton step by Cholesky, clamped to the box; n_inner active-set re-solves
// (joints at a bound are held there and the free ones re-solved against
// g + H p_bound); unscaling; the trust-region
// clip; a 5-point line search on the weighted error plus the collision
// penalty (first minimum); accept with lambda x0.5 / reject x3; all-time
// best tracking.
//
// The reference kernel's FK takes no mimic or topological-order arrays; the
// FK here is the general one, which agrees with it on robots without mimic
// joints whose joints are listed parent first.
//
// B200 mapping: 32 seeds of one problem per block of 128 threads, 4 lanes
// per seed.  The lanes of a seed hold the same state and compute the same
// step; they share out the FK of the line-search trials and split the
// collision penalty of each over the obstacles (robot spheres grouped by
// joint, with exact bounding-sphere culling at the margin).  Each
// solve of the step is FP32 with one conditional FP64 refinement step
// (damped_step_f32: the 6 n_ee x 6 n_ee dual system for one or two EEs, the
// normal equations for more).
#include "pk_damped_step.cuh"
#include "pk_seed_ik.cuh"

namespace pk {

constexpr int kSqpThreads = 128;
constexpr int kSqpTps = 4;

constexpr int kSqpSets = 6;  // pose sets per seed

// Weighted squared pose error.
template <int MAXEE>
__device__ __forceinline__ float sqp_weighted(const SeedIkArgs& a, const float (&r)[6 * MAXEE]) {
  float w = 0.f;
#pragma unroll
  for (int k = 0; k < 6 * MAXEE; ++k) {
    const float rw = r[k] * (k % 6 < 3 ? a.pos_weight : a.ori_weight);
    w += rw * rw;
  }
  return w;
}

// Box-constrained step of the current point (see the file comment).
template <int MAXA, int MAXEE>
__device__ __forceinline__ void sqp_direction(const SeedIkArgs& a, const SeedIkShared& sh, const PoseSlots& ps,
                                              const float (&r)[6 * MAXEE], const float (&pee)[3 * MAXEE],
                                              const float (&cfg)[MAXA], float lam, float (&delta)[MAXA]) {
  float J[6 * MAXEE][MAXA];
  seed_ik_jacobian<MAXA, MAXEE>(sh, ps, a.n_ee, pee, J);
  float fw[6 * MAXEE];
#pragma unroll
  for (int k = 0; k < 6 * MAXEE; ++k) {
    const float wk = k % 6 < 3 ? a.pos_weight : a.ori_weight;
    fw[k] = r[k] * wk;
#pragma unroll
    for (int c = 0; c < MAXA; ++c) J[k][c] *= wk;
  }
  float cs[MAXA];
#pragma unroll
  for (int c = 0; c < MAXA; ++c) {
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < 6 * MAXEE; ++k) sq += J[k][c] * J[k][c];
    cs[c] = sqrtf(sq) + 1e-8f;
  }
#pragma unroll
  for (int k = 0; k < 6 * MAXEE; ++k)
#pragma unroll
    for (int c = 0; c < MAXA; ++c) J[k][c] = J[k][c] / cs[c];
  float lb[MAXA], ub[MAXA];
  bool fr[MAXA];
  float zero[MAXA], xn[MAXA], x[MAXA];
#pragma unroll
  for (int c = 0; c < MAXA; ++c) {
    const bool fx = sh.fixed[c];
    lb[c] = fx ? 0.f : (sh.lo[c] - cfg[c]) * cs[c];
    ub[c] = fx ? 0.f : (sh.hi[c] - cfg[c]) * cs[c];
    zero[c] = 0.f;
  }
  // it = -1: the unconstrained Newton step (fixed joints masked), clamped to
  // the box; then n_inner active-set re-solves: joints at a bound stay there,
  // the rest re-solve against g + H p_bound, i.e. with the held joints as
  // fixed columns at p_bound.  One call site for all of them.
  constexpr int R = 6 * MAXEE;
  const int rows = 6 * a.n_ee;
  float p[MAXA];
  for (int it = -1; it < a.n_inner; ++it) {
    bool act[MAXA];
#pragma unroll
    for (int c = 0; c < MAXA; ++c) {
      act[c] = it < 0 ? (bool)sh.fixed[c] : (p[c] <= lb[c] + 1e-8f || p[c] >= ub[c] - 1e-8f);
      xn[c] = (it >= 0 && act[c]) ? clampf(p[c], lb[c], ub[c]) : 0.f;
      fr[c] = !act[c];
    }
    damped_step_f32<R, MAXA>(J, fw, rows, lam, zero, fr, xn, zero, x);
#pragma unroll
    for (int c = 0; c < MAXA; ++c) p[c] = act[c] ? xn[c] : clampf(x[c], lb[c], ub[c]);
  }
  float dn2 = 0.f, max_p = 0.f, max_o = 0.f;
#pragma unroll
  for (int c = 0; c < MAXA; ++c) {
    delta[c] = p[c] / cs[c];
    dn2 += delta[c] * delta[c];
  }
#pragma unroll
  for (int e = 0; e < MAXEE; ++e) {
    if (e >= a.n_ee) continue;
    max_p = fmaxf(max_p, sqrtf(r[6 * e] * r[6 * e] + r[6 * e + 1] * r[6 * e + 1] + r[6 * e + 2] * r[6 * e + 2]));
    max_o = fmaxf(max_o,
                  sqrtf(r[6 * e + 3] * r[6 * e + 3] + r[6 * e + 4] * r[6 * e + 4] + r[6 * e + 5] * r[6 * e + 5]));
  }
  float Rt;
  if (max_p > 1e-2f || max_o > 0.6f) Rt = 0.38f;
  else if (max_p > 1e-3f || max_o > 0.25f) Rt = 0.22f;
  else if (max_p > 2e-4f || max_o > 0.08f) Rt = 0.12f;
  else Rt = 0.05f;
  const float dn = sqrtf(dn2);
  if (dn > Rt) {
    const float sc = Rt / (dn + 1e-18f);
#pragma unroll
    for (int c = 0; c < MAXA; ++c) delta[c] *= sc;
  }
}

template <int MAXA, int MAXEE, int TPS>
__global__ void __launch_bounds__(kSqpThreads) sqp_kernel(SeedIkArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SeedIkShared& sh = *reinterpret_cast<SeedIkShared*>(smem_raw);
  RobotSpheresS R = seed_ik_spheres_at(smem_raw + sizeof(SeedIkShared), a.n_rs, a.m.n_joints);
  float* world = reinterpret_cast<float*>(smem_raw + seed_ik_world_offset(a));
  float* slots = reinterpret_cast<float*>(smem_raw + seed_ik_slots_offset(a));
  const int tid = threadIdx.x, n = a.m.n_act, p = blockIdx.y;
  const int G = blockDim.x / TPS, grp = tid / TPS, gl = tid % TPS;
  const unsigned gmask = ((1u << TPS) - 1u) << ((tid & 31) & ~(TPS - 1));
  ObsView ob;
  seed_ik_stage(a, sh, R, world, ob, p, 1);
  const int s = blockIdx.x * G + grp;
  if (s >= a.S) return;  // the whole seed group
  const size_t gs = (size_t)p * a.S + s;
  auto alpha_at = [](int i) { return i == 0 ? 1.f : i == 1 ? 0.5f : i == 2 ? 0.25f : i == 3 ? 0.1f : 0.025f; };
  float cfg[MAXA], best_cfg[MAXA];
#pragma unroll
  for (int c = 0; c < MAXA; ++c) cfg[c] = best_cfg[c] = c < n ? a.seeds[gs * n + c] : 0.f;
  // The seed, then per iteration the 5 line-search trials: lane gl runs the FK
  // and residual of trials gl and gl + TPS, each into a pose set of its own;
  // the lanes then split the penalty of one trial after the other.  A seed has
  // kSqpSets pose sets, five for the trials and one (`cur`) for the current
  // point, which an accepted trial's set becomes, so the current point needs no
  // FK; its penalty is the accepted trial's, carried over.  A trial whose pose
  // error alone is not below the best so far cannot win (the penalty is >= 0
  // for a weight >= 0), so its penalty is not evaluated.  One call site each of
  // FK and penalty: with a site per use the loop outgrew the instruction cache.
  // 256 problems x 32 seeds, 8 iterations: 1131 us with every lane running
  // every trial's FK and the sites apart, 883 with one site, 762 so, the same bits.
  float delta[MAXA];
#pragma unroll
  for (int c = 0; c < MAXA; ++c) delta[c] = 0.f;
  float lam = a.lambda_init, pen_cur = 0.f, best_err = 0.f, curr = 0.f;
  int it = 0, cur = 0;
  bool init = true;
  for (;;) {
    const int nt = init ? 1 : 5;
    auto set_of = [&](int k) {  // pose set of trial k (of the seed: the current point's)
      const int i = init ? cur : cur + 1 + k;
      return PoseSlots{slots + grp * kSqpSets + (i >= kSqpSets ? i - kSqpSets : i), G * kSqpSets};
    };
    float ws0 = 0.f, ws1 = 0.f;
#pragma unroll 1
    for (int rd = 0; rd * TPS < nt; ++rd) {
      const int k = rd * TPS + gl;
      if (k >= nt) continue;
      float q[MAXA];
      const float alpha = alpha_at(k);
#pragma unroll
      for (int c = 0; c < MAXA; ++c) q[c] = init ? cfg[c] : clampf(cfg[c] + alpha * delta[c], sh.lo[c], sh.hi[c]);
      const PoseSlots ps = set_of(k);
      fk_thread(sh.jt, [&](int i) { return reg_at(q, i); }, ps);
      float r[6 * MAXEE], pee[3 * MAXEE];
      seed_ik_residual<MAXEE>(sh, ps, a.n_ee, 0, r, pee);
      const float w = sqp_weighted<MAXEE>(a, r);
      if (rd == 0) ws0 = w;
      else ws1 = w;
    }
    __syncwarp(gmask);  // the lanes' pose sets are read by the whole group
    float best_a_err = 1e30f, best_a_pen = pen_cur;
    int best_ai = 0;
#pragma unroll 1
    for (int k = 0; k < nt; ++k) {
      const float wsq = __shfl_sync(gmask, k < TPS ? ws0 : ws1, k % TPS, TPS);
      if (!init && !(wsq < best_a_err) && a.collision_weight >= 0.f) continue;  // the same on the seed's lanes
      const float pen = seed_ik_penalty<TPS>(a, set_of(k), R, ob, gl, gmask);
      const float et = wsq + pen;
      if (init) {
        pen_cur = pen;
        best_err = et;
      } else if (et < best_a_err) {
        best_a_err = et;
        best_a_pen = pen;
        best_ai = k;
      }
    }
    if (!init) {
      float trial[MAXA];
      const float best_alpha = alpha_at(best_ai);
#pragma unroll
      for (int c = 0; c < MAXA; ++c) trial[c] = clampf(cfg[c] + best_alpha * delta[c], sh.lo[c], sh.hi[c]);
      if (best_a_err < curr * (1.f - 1e-4f)) {
#pragma unroll
        for (int c = 0; c < MAXA; ++c) cfg[c] = trial[c];
        pen_cur = best_a_pen;
        cur = cur + 1 + best_ai;
        if (cur >= kSqpSets) cur -= kSqpSets;
        lam = fmaxf(lam * 0.5f, 1e-10f);
      } else {
        lam = fminf(lam * 3.f, 1e6f);
      }
      if (best_a_err < best_err) {
        best_err = best_a_err;
#pragma unroll
        for (int c = 0; c < MAXA; ++c) best_cfg[c] = trial[c];
      }
      ++it;
    }
    if (it >= a.iters) break;
    init = false;
    // the current point: convergence, step
    const PoseSlots ps{slots + grp * kSqpSets + cur, G * kSqpSets};
    float r[6 * MAXEE], pee[3 * MAXEE];
    seed_ik_residual<MAXEE>(sh, ps, a.n_ee, 0, r, pee);
    bool conv = true;
#pragma unroll
    for (int e = 0; e < MAXEE; ++e) {
      if (e >= a.n_ee) continue;
      const float pn = sqrtf(r[6 * e] * r[6 * e] + r[6 * e + 1] * r[6 * e + 1] + r[6 * e + 2] * r[6 * e + 2]);
      const float on = sqrtf(r[6 * e + 3] * r[6 * e + 3] + r[6 * e + 4] * r[6 * e + 4] + r[6 * e + 5] * r[6 * e + 5]);
      if (pn >= a.eps_pos || on >= a.eps_ori) conv = false;
    }
    if (conv) break;
    curr = sqp_weighted<MAXEE>(a, r) + pen_cur;
    sqp_direction<MAXA, MAXEE>(a, sh, ps, r, pee, cfg, lam, delta);
    __syncwarp(gmask);  // every lane has read the set that a rejected trial may reuse
  }
  if (gl == 0) {
    for (int c = 0; c < n; ++c) a.out[gs * n + c] = reg_at(best_cfg, c);
    a.out_err[gs] = best_err;
  }
}

}  // namespace pk

using namespace pk;

namespace {

template <int MAXA, int MAXEE>
int launch_sqp(const SeedIkArgs& a, int threads, size_t smem, cudaStream_t st) {
  auto k = sqp_kernel<MAXA, MAXEE, kSqpTps>;
  if (int s = set_smem_limit((const void*)k, smem)) return s;
  const int G = threads / kSqpTps;
  const dim3 grid((unsigned)((a.S + G - 1) / G), (unsigned)a.P);
  k<<<grid, threads, smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "sqp_kernel launch");
}

}  // namespace

extern "C" int pk_sqp_ik_cuda(void* stream, const float* seeds, const float* twists, const float* parent_tf,
                              const int32_t* parent_idx, const int32_t* act_idx, const float* mimic_mul,
                              const float* mimic_off, const int32_t* mimic_act_idx, const int32_t* topo_inv,
                              const int32_t* target_jnts, const int32_t* ancestor_masks, const float* target_Ts,
                              const float* robot_spheres_local, const int32_t* robot_sphere_joint_idx,
                              const float* world_spheres, const float* world_capsules, const float* world_boxes,
                              const float* world_halfspaces, const float* lower, const float* upper,
                              const int32_t* fixed_mask, int64_t max_iter, int64_t n_inner_iters, float pos_weight,
                              float ori_weight, float lambda_init, float eps_pos, float eps_ori,
                              int64_t enable_collision, float collision_weight, float collision_margin, float* out,
                              float* out_err, int32_t n_problems, int32_t n_seeds, int32_t n_act, int32_t n_joints,
                              int32_t n_ee, int32_t n_robot_spheres, int32_t Ms, int32_t Mc, int32_t Mb, int32_t Mh) {
  SeedIkArgs a = seed_ik_args(seeds, twists, parent_tf, parent_idx, act_idx, mimic_mul, mimic_off, mimic_act_idx,
                              topo_inv, target_jnts, ancestor_masks, target_Ts, robot_spheres_local,
                              robot_sphere_joint_idx, world_spheres, world_capsules, world_boxes, world_halfspaces,
                              lower, upper, fixed_mask, out, out_err, n_problems, n_seeds, n_act, n_joints, n_ee,
                              n_robot_spheres, Ms, Mc, Mb, Mh);
  PK_CHECK_ARG(max_iter >= 0 && max_iter < (1LL << 31), "bad max_iter");
  PK_CHECK_ARG(n_inner_iters >= 0 && n_inner_iters < (1LL << 31), "bad n_inner_iters");
  a.iters = (int)max_iter;
  a.n_inner = (int)n_inner_iters;
  a.pos_weight = pos_weight;
  a.ori_weight = ori_weight;
  a.lambda_init = lambda_init;
  a.eps_pos = eps_pos;
  a.eps_ori = eps_ori;
  a.enable_collision = enable_collision ? 1 : 0;
  a.collision_weight = collision_weight;
  a.collision_margin = collision_margin;
  // fewer seeds per block where the pose sets of 32 (of a robot of many joints)
  // leave no room for the world and its grid
  int threads = kSqpThreads;
  {
    SeedIkArgs w = a;
    seed_ik_want(w, true);
    while (threads > 32 && n_joints > 0 && seed_ik_smem(w, threads / kSqpTps * kSqpSets) > 200 * 1024) threads >>= 1;
  }
  size_t smem = 0;
  if (int s = seed_ik_common(a, n_act, n_joints, n_ee, threads / kSqpTps * kSqpSets, &smem, true)) return s;
  if (n_problems == 0 || n_seeds == 0) return PK_OK;
  if (int s = seed_ik_check_buffers(a)) return s;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_act <= 8 && n_ee == 1) return launch_sqp<8, 1>(a, threads, smem, st);
  if (n_ee <= 2) return launch_sqp<16, 2>(a, threads, smem, st);
  return launch_sqp<16, 4>(a, threads, smem, st);
}
