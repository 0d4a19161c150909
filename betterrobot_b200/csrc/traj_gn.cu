// traj_gn.cu — batched trajectory optimisation (Gauss-Newton / LM), one CTA per
// trajectory, Newton step in nested-dissection order.
//
// Reference: solve_trajopt with knot parameterisation
// (src/better_robot/tasks/trajopt.py:84-230) flattens a (T, nq) trajectory into one
// least-squares problem and solves the dense (T*nv)^2 normal equations with a
// dense Cholesky every iteration (448 x 448 for T = 64, nv = 7).  The stack here is
//   goal  : PoseResidual at knot T-1        (TimeIndexedResidual, residuals/temporal.py:20-126)
//   start : PoseResidual at knot 0          (optional)
//   accel : (d_{s+1} - d_s)/dt^2, d_t = difference(q_t, q_{t+1}) (= q_{t+1} - q_t for q + v
//           joints)                         (AccelerationResidual, residuals/smoothness.py:98-161)
//   limits: JointPositionLimit at every knot (residuals/limits.py:56-86)
//   ref   : difference(q_ref_t, q_t)        (ReferenceTrajectoryResidual, residuals/regularization.py:133-152)
// each with a CostStack item weight.  In its J^T J + damp I every term except the
// two pose terms acts on one DOF at a time: the acceleration rows couple knots
// t, t+1, t+2 of the same DOF, limits / reference / damping are diagonal.  So H is
// nv independent scalar PENTA-diagonal T x T matrices (one per DOF) plus the dense
// nv x nv pose blocks at knots 0 and T-1.  The kernel solves it in nested-dissection
// order: the interior knots 1..T-2 of each DOF first — two threads per DOF run the
// banded L D L^T from both ends with the right-hand side and the columns that tie the
// interior to knots 0 and T-1 — leaving a 2nv x 2nv Schur complement on the
// boundary knots,
//   S = H_bb - H_bI P^-1 H_Ib,   P = blockdiag_i(P_i) the per-DOF interior bands,
// which the block factors in panels of eight columns with its right-hand side as one
// more row; the interior step follows by one more band solve.  This is the exact
// factorization of a symmetric permutation of H (no approximation): O(T nv) sequential
// work per iteration instead of the O(T nv^3) of a block-banded factorization or the
// O((T nv)^3) of the dense one.
//
// Bound by the latency of one CTA's dependent steps (a launch lasts as long as its slowest
// trajectory).  Cycles per Gauss-Newton iteration, chain of 7 at 64 knots / humanoid at 40 knots:
//   band factorization 14.7 k / 12.3 k -> 4.7 k / 5.4 k  (one multiply-add and one reciprocal between
//     pivots; the diagonal and the next row's operands loaded off the chain; no early exit, unrolled)
//   boundary factorization and substitutions 13.5 k / 187 k -> 4.8 k / 37 k  (was one column at a time,
//     three block barriers and an index decode per entry each)
//   boundary assembly 1.2 k / 13.9 k -> 2.6 k / 6.6 k  (now with the pose J^T J that the build made)
//   back substitution 7.5 k / 5.5 k -> 3.7 k / 3.2 k
//   gradient 6.5 k / 16 k -> 4.7 k / 6.2 k  (Jr^-1 series: three lanes, a column each)
//   retraction and cost 6.6 k / 68 k -> 6.3 k / 16 k  (the float64 logs and exps of a free-flyer base
//     one lane each, where every warp of a pass held a single one)
// 256 x 64-knot chain trajectories 665 -> 362 us, 33 x 40-knot humanoid ones 1,332 -> 315 us.
// Cyclic reduction of the bands (one warp per DOF, log2 levels of 2 x 2 blocks) measured slower than the
// two-ended recurrence at every size (chain, 64 knots: 148 against 127 us for six iterations).
//
// Precision: the normal matrix has condition ~1e8 (acceleration stiffness
// (w/dt^2)^2 against a 1e-6 regularisation).  A float32 factorization fails there,
// and even float32 Jacobian entries (relative error ~1e-7) move the Gauss-Newton
// step by ~1e-1 rad along the weakly constrained directions, so the whole
// trajectory solver — iterate, residuals, pose Jacobians, bands, factorization,
// solves — is float64.
//
// After the solve, the gradient of the final cost w.r.t. the goal pose (a right
// perturbation T_goal exp(eps)) is the adjoint -w_goal^2 Jl^-1(xi)^T xi of the
// goal term (envelope theorem: the other terms do not depend on the target and
// dcost/dx = 0 at the optimum); Jl^-1(xi) = Jr^-1(-xi), exact 20-term series.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/br_b200.h"
#include "br_common.cuh"
#include "br_fk.cuh"
#include "br_lie.cuh"

namespace br {

struct TrajParams {
  br_tree_t tree;
  br_traj_settings_t s;
  int32_t frame_id, T;
  int64_t n;
  const float* x0;
  const float* xref;
  const float* goal;
  const float* start;
  float* x;
  int32_t* iters;
  int32_t* status;
  float* cost;
  float* goal_grad;
};

struct TrajLayout {
  // doubles
  int x, xn, dd, dr, g, delta, bl1, bdi, Sb, sdi, sd, zb, schur, Jg, Js, rg, rs, pA, pB, red;
  int total_doubles;
  // 4-byte arrays (offsets in doubles)
  int xref, parent, jtype, idxq, idxv, dofq, heavy, cjoint, ckind, axis, place, caxis, anc, lower, upper;
  int total;
  __host__ __device__ TrajLayout(int nj, int nq, int nv, int T, bool floating) {
    int o = 0;
    auto take = [&](int n) { int r = o; o += (n + 1) & ~1; return r; };  // 16-byte aligned
    const int nb = 2 * nv;
    x = take(T * nq); xn = take(T * nq); g = take(T * nv); delta = take(T * nv);
    // knot differences difference(x_t, x_{t+1}) and difference(xref_t, x_t) of the last
    // evaluated trajectory (kManifold variant; the other subtracts inline)
    dd = take(floating ? T * nv : 0); dr = take(floating ? T * nv : 0);
    // per-DOF interior band factors (index p * nv + i, p = knot - 1): L[p][p-1] and 1 / D[p]
    // (L[p][p-2] = c^2 / D[p-2] is rebuilt from 1 / D)
    bl1 = take(T * nv); bdi = take(T * nv);
    // boundary Schur complement, packed lower, its right-hand side as row nb; 1 / pivot, pivot, solution
    Sb = take((nb + 1) * (nb + 2) / 2); sdi = take(nb); sd = take(nb); zb = take(nb);
    schur = take(5 * nv);                     // per DOF: h0' P^-1 h0, h0' P^-1 hT, hT' P^-1 hT, h0' P^-1 y, hT' P^-1 y
    Jg = take(6 * nv); Js = take(6 * nv); rg = take(8); rs = take(8);
    pA = take(16 * nj); pB = take(16 * nj);   // FK buffers of the two pose terms (goal, start)
    red = take(32);                           // per-warp partial sums of the block reductions
    total_doubles = o;
    auto take4 = [&](int n) { int r = o; o += ((n + 3) & ~3) / 2; return r; };
    xref = take4(T * nq);                     // float32, as given
    parent = take4(nj); jtype = take4(nj); idxq = take4(nj); idxv = take4(nj); dofq = take4(nv);
    heavy = take4(nj + 1);
    cjoint = take4(nv); ckind = take4(nv);
    axis = take4(4 * nj); place = take4(8 * nj); caxis = take4(4 * nv); anc = take4(8 * nj);
    lower = take4(nq); upper = take4(nq);
    total = o;
  }
};

__device__ __forceinline__ DPose ldd8(const double* p) {
  return DPose{d3(p[0], p[1], p[2]), make_double4(p[4], p[5], p[6], p[7])};
}
__device__ __forceinline__ void std8d(double* p, const DPose& P) {
  p[0] = P.t.x; p[1] = P.t.y; p[2] = P.t.z; p[3] = 0.0;
  p[4] = P.q.x; p[5] = P.q.y; p[6] = P.q.z; p[7] = P.q.w;
}

// 1 / d for d > 0 (a pivot): the hardware reciprocal estimate r (relative error below 2^-20) refined by
// one third-order step r <- r + r (e + e^2), e = 1 - d r, which leaves e^3 < 2^-60: within an ulp or two
// of 1.0 / d in three dependent operations.  Every dependent float64 operation of a recurrence costs
// about 25 cycles of its single warp's time, so the recurrences below are written to have few of them.
__device__ __forceinline__ double fast_rcp(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// packed lower-triangle index p -> (a, b), b <= a, p = a (a + 1) / 2 + b: approximate square
// root, made exact by its two integer corrections
__device__ __forceinline__ int2 tri_decode(int p) {
  int a = (int)((sqrtf(8.f * p + 1.f) - 1.f) * 0.5f);
  if ((a + 1) * (a + 2) / 2 <= p) ++a;
  if (a * (a + 1) / 2 > p) --a;
  return make_int2(a, p - a * (a + 1) / 2);
}
__device__ __forceinline__ int tri_at(int r, int c) { return r * (r + 1) / 2 + c; }  // r >= c

// Threads per trajectory (kNT): the per-DOF interior chains take two threads each (nv <= 64), the two
// pose terms one warp each, everything else strides over the block.  256 threads when an SM holds only
// one trajectory anyway (few trajectories, or a working set above half its shared memory), else 128
// (64 trajectories of 64 knots, six iterations, 256 against 128 threads: chain of 7 94 against 100 us,
// 20 DOFs 144 / 160, humanoid 250 / 280; with more trajectories than SMs two CTAs of 128 run at once).

// Threads that the terms of a block's sums are dealt to, whatever its own number.
constexpr int kSumThreads = 256;

// kManifold: the tree has joints whose configuration is not their tangent coordinates
// (free-flyer, spherical, planar, unbounded revolute): knot differences and the retraction go
// through Model.difference / Model.integrate; otherwise they are q1 - q0 and q + v.
template <bool kManifold, int kNT>
__global__ void __launch_bounds__(kNT, 256 / kNT) traj_gn_kernel(const TrajParams P) {
  extern __shared__ __align__(16) double sm[];
  const br_tree_t& tree = P.tree;
  const int nj = tree.njoints, nq = tree.nq, nv = tree.nv, T = P.T;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NT = kNT, NW = kNT / kWarp;
  const int64_t traj = blockIdx.x;
  if (traj >= P.n) return;
  const TrajLayout L(nj, nq, nv, T, kManifold);
  double* x = sm + L.x;
  double* xn = sm + L.xn;
  double* g = sm + L.g;
  double* delta = sm + L.delta;
  double* bl1 = sm + L.bl1;
  double* bdi = sm + L.bdi;
  double* Sb = sm + L.Sb;
  double* sdi = sm + L.sdi;
  double* sd = sm + L.sd;
  double* zb = sm + L.zb;
  double* schur = sm + L.schur;
  double* Jg = sm + L.Jg;
  double* Js = sm + L.Js;
  double* rg = sm + L.rg;
  double* rs = sm + L.rs;
  double* pA = sm + L.pA;
  double* pB = sm + L.pB;
  double* red = sm + L.red;
  float* xref = reinterpret_cast<float*>(sm + L.xref);
  int* parent = reinterpret_cast<int*>(sm + L.parent);
  int* jtype = reinterpret_cast<int*>(sm + L.jtype);
  int* idxq = reinterpret_cast<int*>(sm + L.idxq);
  int* idxv = reinterpret_cast<int*>(sm + L.idxv);
  int* dofq = reinterpret_cast<int*>(sm + L.dofq);  // q slot of a DOF with a position limit, else -1
  int* heavy = reinterpret_cast<int*>(sm + L.heavy);  // [0] their count, then the joints that are not q + v
  double* dd = sm + L.dd;
  double* dr = sm + L.dr;
  int* cjoint = reinterpret_cast<int*>(sm + L.cjoint);
  int* ckind = reinterpret_cast<int*>(sm + L.ckind);
  float* axis = reinterpret_cast<float*>(sm + L.axis);
  float* place = reinterpret_cast<float*>(sm + L.place);
  float* caxis = reinterpret_cast<float*>(sm + L.caxis);
  int* ancA = reinterpret_cast<int*>(sm + L.anc);
  int* ancB = ancA + 2 * nj;
  float* lower = reinterpret_cast<float*>(sm + L.lower);
  float* upper = reinterpret_cast<float*>(sm + L.upper);
  const br_traj_settings_t& S = P.s;
  const double c = (double)S.w_accel / ((double)S.dt * (double)S.dt);
  const double c2 = c * c;
  const double wl = S.w_limit, wr = S.w_ref, wg = S.w_goal, ws = S.w_start;
  const bool has_start = P.start != nullptr && S.w_start > 0.f;
  const bool has_goal = S.w_goal > 0.f;
  const int n = T * nv, nqT = T * nq, nb = 2 * nv;
  const FastDiv divv(nv > 0 ? nv : 1), divq(nq > 0 ? nq : 1);

  for (int j = tid; j < nj; j += NT) {
    parent[j] = tree.parent[j];
    jtype[j] = tree.jtype[j];
    idxq[j] = tree.idx_q[j];
    idxv[j] = tree.idx_v[j];
    for (int k = 0; k < 4; ++k) axis[4 * j + k] = tree.axis[4 * j + k];
    for (int k = 0; k < 8; ++k) place[8 * j + k] = tree.placement[8 * j + k];
  }
  for (int k = tid; k < nv; k += NT) {
    cjoint[k] = tree.col_joint[k];
    ckind[k] = tree.col_kind[k];
    for (int m = 0; m < 4; ++m) caxis[4 * k + m] = tree.col_axis[4 * k + m];
  }
  for (int i = tid; i < nq; i += NT) {
    lower[i] = tree.lower[i];
    upper[i] = tree.upper[i];
  }
  __syncthreads();
  for (int j = tid; j < nj; j += NT) {              // limits.py:36-48: nq == nv joints only
    const int jt = jtype[j];
    const bool vec = joint_is_vector(jt);
    for (int k = 0; k < joint_nv(jt); ++k) dofq[idxv[j] + k] = vec ? idxq[j] + k : -1;
  }
  if (kManifold && tid == 0) {
    int nh = 0;
    for (int j = 0; j < nj; ++j)
      if (joint_nv(jtype[j]) && !joint_is_vector(jtype[j])) heavy[++nh] = j;
    heavy[0] = nh;
  }
  const float* x0 = P.x0 + traj * (int64_t)nqT;
  const float* xr = (P.xref ? P.xref : P.x0) + traj * (int64_t)nqT;
  for (int i = tid; i < nqT; i += NT) {
    x[i] = x0[i];
    xref[i] = xr[i];
  }
  const int fpar = tree.frame_parent[P.frame_id];
  const Pose fpl = load_pose8(tree.frame_placement + 8 * P.frame_id);
  const unsigned long long sup = tree.support[fpar];
  __syncthreads();

  auto warp_sum = [&](double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  // Sum over the block; every thread gets the same value.  A trajectory's sums do not depend on the block
  // that its launch chose: terms are dealt to kSumThreads threads, of which one of a smaller block stands
  // for several (its terms in turn, Sum::add), and the warps' partials are added in the order of those.
  constexpr int kParts = kSumThreads / NT;
  struct Sum {
    double v[kParts] = {};
    int turn = 0;
    __device__ __forceinline__ void add(double x) {
      if (kParts == 1) {
        v[0] += x;
      } else {
        const double s = (turn ? v[kParts - 1] : v[0]) + x;
        if (turn) v[kParts - 1] = s;
        else v[0] = s;
        turn ^= 1;
      }
    }
    __device__ __forceinline__ void next_loop() { turn = 0; }   // every loop deals from the first thread
  };
  static_assert(kParts <= 2, "Sum::add alternates between two");
  auto block_sum = [&](const Sum& a) -> double {
    double v[kParts];
#pragma unroll
    for (int h = 0; h < kParts; ++h) v[h] = warp_sum(a.v[h]);
    __syncthreads();                                  // the previous reduction's reads are done
    if (lane == 0) {
#pragma unroll
      for (int h = 0; h < kParts; ++h) red[h * NW + warp] = v[h];
    }
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kSumThreads / kWarp; ++w) s += red[w];
    return s;
  };
  // float64 FK of knot t of trajectory `xs` by one warp (pose term h: buffers pA / pB + 8 nj h,
  // ancA / ancB + nj h); returns the world poses
  auto fk = [&](const double* xs, int t, int h) -> double* {
    const double* q = xs + t * nq;
    double* A = pA + 8 * nj * h;
    double* B = pB + 8 * nj * h;
    int* aA = ancA + nj * h;
    int* aB = ancB + nj * h;
    for (int j = lane; j < nj; j += kWarp) {
      const Pose Pj = load_pose8(place + 8 * j);
      const DPose Lj = dlocal_transform(jtype[j], DPose{d3(Pj.t.x, Pj.t.y, Pj.t.z),
                                                        make_double4(Pj.q.x, Pj.q.y, Pj.q.z, Pj.q.w)},
                                        axis + 4 * j, q + idxq[j]);
      std8d(A + 8 * j, Lj);
      aA[j] = parent[j];
    }
    __syncwarp();
    for (int r = 0; r < tree.rounds; ++r) {
      for (int j = lane; j < nj; j += kWarp) {
        const int a = aA[j];
        if (a >= 0) {
          std8d(B + 8 * j, dcompose(ldd8(A + 8 * a), ldd8(A + 8 * j)));
          aB[j] = aA[a];
        } else {
          std8d(B + 8 * j, ldd8(A + 8 * j));
          aB[j] = -1;
        }
      }
      __syncwarp();
      double* tp = A; A = B; B = tp;
      int* ta = aA; aA = aB; aB = ta;
    }
    return A;
  };
  // both pose terms at xs, warp 0 the goal (knot T-1), warp 1 the start (knot 0): xi (into
  // rg / rs); with want_J also J = Jr^-1 blockdiag(R^T,R^T) J_lwa (6 x nv, into Jg / Js).
  // A term that is not in the problem (weight 0 or no start pose) is skipped.  With `reuse`
  // the knot's FK and xi are those the last call left (the build follows the cost evaluation
  // of the same point, and nothing in between writes the pose buffers).
  auto pose_terms = [&](const double* xs, bool want_J, bool reuse) __attribute__((always_inline)) {
    if (warp < 2) {
      const int h = warp;
      const bool active = h == 0 ? has_goal : has_start;
      if (active) {
        const float* tp = (h == 0 ? P.goal : P.start) + traj * 7;   // the term's target pose
        const DPose target{d3(tp[0], tp[1], tp[2]), make_double4(tp[3], tp[4], tp[5], tp[6])};
        double* r = h == 0 ? rg : rs;
        double* J = h == 0 ? Jg : Js;
        double* pose = reuse ? ((tree.rounds & 1) ? pB : pA) + 8 * nj * h : fk(xs, h == 0 ? T - 1 : 0, h);
        const DPose Tee = dcompose(ldd8(pose + 8 * fpar), DPose{d3(fpl.t.x, fpl.t.y, fpl.t.z),
                                                                make_double4(fpl.q.x, fpl.q.y, fpl.q.z, fpl.q.w)});
        double3 v, w;
        if (reuse) {
          v = d3(r[0], r[1], r[2]);
          w = d3(r[3], r[4], r[5]);
        } else {
          dse3_log(dcompose(dinverse(target), Tee), v, w);
          if (lane == 0) { r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = w.x; r[4] = w.y; r[5] = w.z; }
        }
        if (want_J) {
          // the series' three B columns on three lanes
          DJrInv Jr;
          Jr.w = w;
          const double3 bc = djr_inv_se3_col<9>(v, w, lane < 3 ? lane : 0, Jr.b0, Jr.b1, Jr.b2);
#pragma unroll
          for (int c3 = 0; c3 < 3; ++c3) {
            Jr.B[c3] = __shfl_sync(0xffffffffu, bc.x, c3);
            Jr.B[3 + c3] = __shfl_sync(0xffffffffu, bc.y, c3);
            Jr.B[6 + c3] = __shfl_sync(0xffffffffu, bc.z, c3);
          }
          const double4 qc = dqconj(Tee.q);
          for (int k = lane; k < nv; k += kWarp) {
            double3 ol = d3(0, 0, 0), oa = d3(0, 0, 0);
            if ((sup >> cjoint[k]) & 1ull) {
              const DPose Tj = ldd8(pose + 8 * cjoint[k]);
              const double3 a = dqrot(Tj.q, d3(caxis[4 * k], caxis[4 * k + 1], caxis[4 * k + 2]));
              double3 lin, ang;
              if (ckind[k] == 0) {
                lin = dcross(a, dsub(Tee.t, Tj.t));
                ang = a;
              } else {
                lin = a;
                ang = d3(0, 0, 0);
              }
              djr_inv_apply(Jr, dqrot(qc, lin), dqrot(qc, ang), ol, oa);
            }
            J[0 * nv + k] = ol.x; J[1 * nv + k] = ol.y; J[2 * nv + k] = ol.z;
            J[3 * nv + k] = oa.x; J[4 * nv + k] = oa.y; J[5 * nv + k] = oa.z;
          }
        }
      }
    }
    // the build reads J next; a cost evaluation reads xi only after its block sum's barriers
    if (want_J) __syncthreads();
  };
  // dd[t] = difference(xs_t, xs_{t+1}) (t < T-1) and dr[t] = difference(xref_t, xs_t)
  // (model.py:176-190): free-flyer log(q_a^-1 q_b) (free_flyer.py:53-57), spherical
  // log(normalize(q_a^-1 q_b)) (spherical.py:58-62), angle differences of atan2 for the
  // unbounded revolute and planar joints (revolute.py:233-237, planar.py:70-76)
  // The joints with a log or an arctangent take one lane per (joint, pair): by (pair, joint) in joint
  // order every warp held one such lane and 31 subtractions (humanoid, 40 knots: 79 logs in 20 passes
  // of the block, 68 k cycles per cost with the retraction; now one pass).
  auto knot_differences = [&](const double* xs) {
    const int npair = 2 * T - 1, nh = heavy[0];
    for (int e = tid; e < npair * nh; e += NT) {
      const int hj = e / npair, pi = e - hj * npair, j = heavy[1 + hj];
      const int jt = jtype[j], iq = idxq[j], iv = idxv[j];
      // configurations a -> b of the pair: (x_t, x_{t+1}) or (xref_t, x_t)
      const bool ref = pi >= T - 1;
      const int t = ref ? pi - (T - 1) : pi;
      const double* qbp = xs + (ref ? t : t + 1) * nq + iq;
      const double* qap = xs + t * nq + iq;
      const float* qrp = xref + t * nq + iq;
      auto qa = [&](int k) -> double { return ref ? (double)qrp[k] : qap[k]; };
      auto qb = [&](int k) -> double { return qbp[k]; };
      double* out = (ref ? dr : dd) + t * nv;
      if (jt == BR_JOINT_FREE_FLYER || jt == BR_JOINT_SPHERICAL) {  // one log site
        const bool ff = jt == BR_JOINT_FREE_FLYER;
        const int k = ff ? 3 : 0;
        const double4 ra = make_double4(qa(k), qa(k + 1), qa(k + 2), qa(k + 3));
        const double4 rb = make_double4(qb(k), qb(k + 1), qb(k + 2), qb(k + 3));
        DPose rel{d3(0.0, 0.0, 0.0), dqmul(dqconj(ra), rb)};
        if (ff) rel.t = dqrot(dqconj(ra), dsub(d3(qb(0), qb(1), qb(2)), d3(qa(0), qa(1), qa(2))));
        else rel.q = dqnormalize(rel.q);
        double3 v, w;
        dse3_log(rel, v, w);
        if (ff) { out[iv] = v.x; out[iv + 1] = v.y; out[iv + 2] = v.z; }
        const int o = iv + k;
        out[o] = w.x; out[o + 1] = w.y; out[o + 2] = w.z;
      } else {                                                    // planar, unbounded revolute
        const int k = jt == BR_JOINT_PLANAR ? 2 : 0;
        if (k) { out[iv] = qb(0) - qa(0); out[iv + 1] = qb(1) - qa(1); }
        out[iv + k] = atan2(qb(k + 1), qb(k)) - atan2(qa(k + 1), qa(k));
      }
    }
    for (int e = tid; e < n; e += NT) {
      const int t = divv.div(e), iq = dofq[e - t * nv];
      if (iq < 0) continue;
      const double v = xs[t * nq + iq];
      if (t < T - 1) dd[e] = xs[(t + 1) * nq + iq] - v;
      dr[e] = v - (double)xref[t * nq + iq];
    }
    __syncthreads();
  };
  // xn_t = integrate(x_t, delta_t) per knot (model.py:160-174): free-flyer normalize(q . exp(v))
  // (free_flyer.py:47-51), spherical normalize(q . exp(w)) (spherical.py:52-56), unbounded
  // revolute / planar angle atan2(s, c) + v as (cos, sin) (revolute.py:223-231, planar.py:61-68)
  auto retract_knots = [&]() {
    const int nh = heavy[0];
    for (int e = tid; e < T * nh; e += NT) {
      const int hj = e / T, t = e - hj * T, j = heavy[1 + hj];
      const int jt = jtype[j], iq = idxq[j], iv = idxv[j];
      const double* q = x + t * nq;
      const double* dv = delta + t * nv;
      double* o = xn + t * nq;
      if (jt == BR_JOINT_FREE_FLYER || jt == BR_JOINT_SPHERICAL) {  // one exp site
        const bool ff = jt == BR_JOINT_FREE_FLYER;
        const int k = ff ? 3 : 0;
        const double3 v = ff ? d3(dv[iv], dv[iv + 1], dv[iv + 2]) : d3(0.0, 0.0, 0.0);
        const DPose a{ff ? d3(q[iq], q[iq + 1], q[iq + 2]) : d3(0.0, 0.0, 0.0),
                      make_double4(q[iq + k], q[iq + k + 1], q[iq + k + 2], q[iq + k + 3])};
        DPose b = dcompose(a, dse3_exp(v, d3(dv[iv + k], dv[iv + k + 1], dv[iv + k + 2])));
        b.q = dqnormalize(b.q);
        if (ff) { o[iq] = b.t.x; o[iq + 1] = b.t.y; o[iq + 2] = b.t.z; }
        o[iq + k] = b.q.x; o[iq + k + 1] = b.q.y; o[iq + k + 2] = b.q.z; o[iq + k + 3] = b.q.w;
      } else {                                                    // planar, unbounded revolute
        const int k = jt == BR_JOINT_PLANAR ? 2 : 0;
        if (k) { o[iq] = q[iq] + dv[iv]; o[iq + 1] = q[iq + 1] + dv[iv + 1]; }
        double sn, cs;
        sincos(atan2(q[iq + k + 1], q[iq + k]) + dv[iv + k], &sn, &cs);
        o[iq + k] = cs;
        o[iq + k + 1] = sn;
      }
    }
    for (int e = tid; e < n; e += NT) {
      const int t = divv.div(e), iq = dofq[e - t * nv];
      if (iq >= 0) xn[t * nq + iq] = x[t * nq + iq] + delta[e];
    }
  };
  // total cost 0.5 |r|^2 at xs (pose terms evaluated into rg / rs)
  auto cost_of = [&](const double* xs) -> double {
    Sum acc;
    pose_terms(xs, false, false);
    if (kManifold) knot_differences(xs);
    for (int e = tid; e < (T - 2) * nv; e += NT) {              // smoothness.py:118-125
      const double a = kManifold ? c * (dd[e + nv] - dd[e]) : c * (xs[e + 2 * nv] - 2.0 * xs[e + nv] + xs[e]);
      acc.add(a * a);
    }
    acc.next_loop();
    if (kManifold) {
      for (int e = tid; e < nqT; e += NT) {                     // limits.py:56-62
        const int i = divq.mod(e);
        const double lo = fmax((double)lower[i] - xs[e], 0.0), hi = fmax(xs[e] - (double)upper[i], 0.0);
        acc.add(wl * wl * (lo * lo + hi * hi));
      }
      acc.next_loop();
      for (int e = tid; e < n; e += NT) acc.add(wr * wr * dr[e] * dr[e]);   // regularization.py:143-152
    } else {                                                    // nq == nv: one pass for both
      for (int e = tid; e < n; e += NT) {
        const int i = divv.mod(e);
        const double lo = fmax((double)lower[i] - xs[e], 0.0), hi = fmax(xs[e] - (double)upper[i], 0.0);
        const double d = xs[e] - (double)xref[e];
        acc.add(wl * wl * (lo * lo + hi * hi) + wr * wr * d * d);
      }
    }
    const double knots = block_sum(acc);
    double pc = 0.0;
    for (int k = 0; k < 6; ++k) {
      if (has_goal) pc += wg * wg * rg[k] * rg[k];
      if (has_start) pc += ws * ws * rs[k] * rs[k];
    }
    return 0.5 * (knots + pc);
  };
  // pose Jacobians and g = J^T r at x; returns |g|
  auto build = [&]() -> double {
    pose_terms(x, true, true);                        // FK and xi of x from the cost evaluation of x
    Sum gg;
    for (int e = tid; e < n; e += NT) {
      const int t = divv.div(e), i = e - t * nv;
      double acc = 0.0;
      // acceleration rows s = t, t-1, t-2 with coefficients +1, -2, +1 at knot t (the
      // identity-Jacobian blocks of smoothness.py:127-142)
      auto arow = [&](int s) {
        return kManifold ? c * (dd[(s + 1) * nv + i] - dd[s * nv + i])
                         : c * (x[(s + 2) * nv + i] - 2.0 * x[(s + 1) * nv + i] + x[s * nv + i]);
      };
      if (t <= T - 3) acc += c * arow(t);
      if (t - 1 >= 0 && t - 1 <= T - 3) acc += -2.0 * c * arow(t - 1);
      if (t - 2 >= 0) acc += c * arow(t - 2);
      const int iq = kManifold ? dofq[i] : i;
      if (iq >= 0) {
        const double xq = x[t * nq + iq];
        if (xq < (double)lower[iq]) acc -= wl * wl * ((double)lower[iq] - xq);
        if (xq > (double)upper[iq]) acc += wl * wl * (xq - (double)upper[iq]);
      }
      acc += wr * wr * (kManifold ? dr[e] : x[e] - (double)xref[e]);
      if (has_goal && t == T - 1)
        for (int r = 0; r < 6; ++r) acc += wg * wg * Jg[r * nv + i] * rg[r];
      if (has_start && t == 0)
        for (int r = 0; r < 6; ++r) acc += ws * ws * Js[r * nv + i] * rs[r];
      g[e] = acc;
      gg.add(acc * acc);
    }
    return sqrt(block_sum(gg));
  };
  // bands of J^T J + damp I at x (DOF i): diagonal at knot t, H[(t+1,i),(t,i)], and
  // H[(t+2,i),(t,i)] = c2 for t <= T-3.  Acceleration row s has coefficients (1, -2, 1)
  // on knots (s, s+1, s+2), s = 0..T-3.
  auto hdiag = [&](int t, int i, double damp) -> double {
    double a = 0.0;
    if (t <= T - 3) a += 1.0;
    if (t - 1 >= 0 && t - 1 <= T - 3) a += 4.0;
    if (t - 2 >= 0) a += 1.0;
    double d = c2 * a + wr * wr + damp;
    const int iq = kManifold ? dofq[i] : i;
    if (iq >= 0) {
      const double xv = x[t * nq + iq];
      if (xv < (double)lower[iq]) d += wl * wl;
      if (xv > (double)upper[iq]) d += wl * wl;
    }
    return d;
  };
  auto hoff1 = [&](int t) -> double {
    double b = 0.0;
    if (t <= T - 3) b += -2.0;
    if (t - 1 >= 0 && t <= T - 2) b += -2.0;
    return c2 * b;
  };
  // interior columns of the boundary knots: h0 = H[(t, i), (0, i)], hT = H[(t, i), (T-1, i)]
  auto h0_at = [&](int t) -> double { return t == 1 ? hoff1(0) : (t == 2 ? c2 : 0.0); };
  auto hT_at = [&](int t) -> double { return t == T - 2 ? hoff1(T - 2) : (t == T - 3 ? c2 : 0.0); };
  // solve (J^T J + damp I) delta = -g; false when a pivot is not positive.  Interior knots 1..T-2 of
  // DOF i form the pentadiagonal P_i, with y = -g_I and the columns h0, hT that tie it to knots 0 and
  // T-1.  The boundary system is S = H_bb - H_bI P^-1 H_Ib with right-hand side -g_b - H_bI P^-1 y; its
  // inner products h^T P^-1 k are sums of z_h z_k / pivot over the elimination (z = L^-1 v).
  const int m = T - 2;
  const double h1 = -4.0 * c2;                        // H[(p+1), (p)] inside the interior

  // Twisted elimination, two threads per DOF (at least kTwistMin interior knots): thread 2i
  // takes rows 0..k-1 top-down (L D L^T), thread 2i + 1 rows m-1..k+2 bottom-up, k = m / 2, and both then
  // reduce the 2 x 2 block of rows k, k+1 from the two sides' updates.  The multipliers into the middle
  // block are kept in the free slots of rows k, k+1 (bl1), every second-neighbour multiplier is c2 times
  // a stored reciprocal pivot.  h0 is zero in the bottom rows and hT in the top rows, so a side carries
  // y and one column.  The diagonal waits in the slots of the reciprocals that replace it (bdi), written
  // by the whole block: its limit tests are not on the chain of pivots.
  const unsigned tmask = __ballot_sync(0xffffffffu, tid < 2 * nv);
  auto interior_twisted = [&](double damp) __attribute__((always_inline)) -> bool {
    const int km = m / 2;
    bool good = true;
    for (int e = tid; e < m * nv; e += NT) {
      const int p = divv.div(e);
      bdi[e] = hdiag(p + 1, e - p * nv, damp);
    }
    __syncthreads();
    if (tid < 2 * nv) {
      const int i = tid >> 1, side = tid & 1;
      // side 0: p = 0, 1, .., km-1; side 1: p = m-1, m-2, .., km+2 (the same recurrence on
      // the reversed band: diagonal, off-diagonals h1 and c2 are symmetric)
      const int p0 = side ? m - 1 : 0, dir = side ? -1 : 1, steps = side ? m - km - 2 : km;
      const int step = dir * nv;
      // row q: multiplier l1 = e / d_(q-1) with e = h1 - c2 l1_(q-1), pivot d = hd - e^2 / d_(q-1)
      // - c2^2 / d_(q-2): from one reciprocal to the next only e^2 / d_(q-1), everything else is ready
      double di1 = 0.0, di2 = 0.0, e1 = 0.0, svv = 0.0, svy = 0.0;
      double y1 = 0, y2 = 0, u1 = 0, u2 = 0;
      int o = p0 * nv + i;
      double hd = bdi[o], gy = -g[o + nv];
      double ub = -2.0 * c2, ub_n = c2;             // h0 = (-2, 1, 0, ...) c2 from the top, hT the same from the bottom
#pragma unroll 4
      for (int q = 0; q < steps; ++q) {             // a bad pivot runs on: the result is refused below
        const double hd_n = bdi[o + step], gy_n = -g[o + step + nv];  // the next row's (a middle row's after the last)
        const double l2 = c2 * di2;
        const double dp = (hd - c2 * l2) - e1 * e1 * di1;
        good = good && dp > 0.0;
        const double dip = fast_rcp(dp);
        const double l1 = e1 * di1;
        bl1[o] = l1; bdi[o] = dip;
        const double y = (gy - l2 * y2) - l1 * y1;
        const double u = (ub - l2 * u2) - l1 * u1;
        svv += u * u * dip;
        svy += u * y * dip;
        e1 = h1 - c2 * l1;
        di2 = di1; di1 = dip;
        y2 = y1; y1 = y; u2 = u1; u1 = u;
        ub = ub_n; ub_n = 0.0;
        o += step; hd = hd_n; gy = gy_n;
      }
      // this side's multipliers into the middle block: the adjacent middle row (km for the top,
      // km + 1 for the bottom) from this side's last two rows, the far middle row from its last
      const double n1 = e1 * di1, n2 = c2 * di2, f1 = c2 * di1;
      const int near = side ? km + 1 : km;
      // updates of the middle block: near diagonal, off-diagonal, far diagonal; right-hand sides
      const double a_near = n1 * e1 + n2 * c2, a_off = c2 * n1, a_far = f1 * c2;
      const double ry_near = n1 * y1 + n2 * y2, ry_far = f1 * y1;
      const double ru_near = n1 * u1 + n2 * u2, ru_far = f1 * u1;
      const double g0 = -g[(km + 1) * nv + i], g1 = -g[(km + 2) * nv + i];
      const double hd0 = bdi[km * nv + i], hd1 = bdi[(km + 1) * nv + i];
      // the other side's updates (lanes 2i, 2i + 1 of one warp)
      const double o_near = __shfl_xor_sync(tmask, a_near, 1), o_off = __shfl_xor_sync(tmask, a_off, 1),
                   o_far = __shfl_xor_sync(tmask, a_far, 1);
      const double oy_near = __shfl_xor_sync(tmask, ry_near, 1), oy_far = __shfl_xor_sync(tmask, ry_far, 1);
      const double ou_near = __shfl_xor_sync(tmask, ru_near, 1), ou_far = __shfl_xor_sync(tmask, ru_far, 1);
      const double osvv = __shfl_xor_sync(tmask, svv, 1), osvy = __shfl_xor_sync(tmask, svy, 1);
      good = __shfl_xor_sync(tmask, (int)good, 1) && good;
      bl1[near * nv + i] = n1;
      // middle block in (top, bottom) order, the same on both lanes
      const double B00 = hd0 - (side ? o_near : a_near) - (side ? a_far : o_far);
      const double B10 = h1 - a_off - o_off;
      const double B11 = hd1 - (side ? o_far : a_far) - (side ? a_near : o_near);
      const double ry0 = g0 - (side ? oy_near : ry_near) - (side ? ry_far : oy_far);
      const double ry1 = g1 - (side ? oy_far : ry_far) - (side ? ry_near : oy_near);
      // column h0 comes from the top side, hT from the bottom side
      const double ru0 = -(side ? ou_near : ru_near), ru1 = -(side ? ou_far : ru_far);
      const double rw0 = -(side ? ru_far : ou_far), rw1 = -(side ? ru_near : ou_near);
      good = good && B00 > 0.0;
      const double dk = good ? fast_rcp(B00) : 0.0;
      const double lm = B10 * dk;
      const double D1 = B11 - lm * B10;
      good = good && D1 > 0.0;
      const double dk1 = good ? fast_rcp(D1) : 0.0;
      // a^T B^-1 b = a0 b0 / B00 + (a1 - l a0)(b1 - l b0) / D1
      auto bq = [&](double a0, double a1, double b0, double b1) {
        return a0 * b0 * dk + (a1 - lm * a0) * (b1 - lm * b0) * dk1;
      };
      if (side == 0) {
        bdi[km * nv + i] = dk; bdi[(km + 1) * nv + i] = dk1;
        schur[i] = svv + bq(ru0, ru1, ru0, ru1);
        schur[nv + i] = bq(ru0, ru1, rw0, rw1);
        schur[2 * nv + i] = osvv + bq(rw0, rw1, rw0, rw1);
        schur[3 * nv + i] = svy + bq(ru0, ru1, ry0, ry1);
        schur[4 * nv + i] = osvy + bq(rw0, rw1, ry0, ry1);
      }
    }
    return good;
  };

  // Few interior knots: thread i runs DOF i's band from the top.
  constexpr int kTwistMin = 8;
  auto interior_plain = [&](double damp) __attribute__((always_inline)) -> bool {
    bool good = true;
    if (tid < nv) {
      const int i = tid;
      double d1 = 0.0, di1 = 0.0, di2 = 0.0, l1p = 0.0;
      double y1 = 0, y2 = 0, u1 = 0, u2 = 0, w1 = 0, w2 = 0;
      double suu = 0.0, suw = 0.0, sww = 0.0, suy = 0.0, swy = 0.0;
      for (int p = 0; p < m; ++p) {
        const int t = p + 1;
        const double l2 = (p >= 2) ? c2 * di2 : 0.0;
        const double l1 = (p >= 1) ? (h1 - c2 * l1p) * di1 : 0.0;
        const double dp = hdiag(t, i, damp) - l1 * l1 * d1 - l2 * c2;
        if (!(dp > 0.0)) { good = false; break; }
        const double dip = fast_rcp(dp);
        bl1[p * nv + i] = l1; bdi[p * nv + i] = dip;
        const double y = -g[t * nv + i] - l1 * y1 - l2 * y2;
        const double u = h0_at(t) - l1 * u1 - l2 * u2;
        const double w = hT_at(t) - l1 * w1 - l2 * w2;
        suu += u * u * dip; suw += u * w * dip; sww += w * w * dip;
        suy += u * y * dip; swy += w * y * dip;
        di2 = di1; di1 = dip; d1 = dp; l1p = l1;
        y2 = y1; y1 = y; u2 = u1; u1 = u; w2 = w1; w1 = w;
      }
      schur[i] = suu; schur[nv + i] = suw; schur[2 * nv + i] = sww; schur[3 * nv + i] = suy; schur[4 * nv + i] = swy;
    }
    return good;
  };

  const bool tw = m >= kTwistMin;

  auto newton_solve = [&](double damp) __attribute__((always_inline)) -> bool {
    for (int b = tid; b < nb; b += NT) sd[b] = hdiag(b < nv ? 0 : T - 1, b < nv ? b : b - nv, damp);
    const bool good = tw ? interior_twisted(damp) : interior_plain(damp);
    if (__syncthreads_or(!good)) return false;
    // boundary system, packed lower: b = i for (knot 0, DOF i), nv + i for (knot T-1, DOF i); its
    // right-hand side is row nb, so that the factorization also substitutes forward
    for (int kb = 0; kb < 2; ++kb) {                   // the two dense blocks, four rows of a warp at once
      const double* J = kb ? Jg : Js;
      const double wj = kb ? (has_goal ? wg * wg : 0.0) : (has_start ? ws * ws : 0.0);
      for (int r0 = 4 * warp; r0 < nv; r0 += 4 * NW)
        for (int ic = lane; ic < nv && ic < r0 + 4; ic += kWarp) {
          double h[4] = {0.0, 0.0, 0.0, 0.0};
          if (wj > 0.0) {
#pragma unroll
            for (int k = 0; k < 6; ++k) {
              const double jc = J[k * nv + ic] * wj;
#pragma unroll
              for (int q = 0; q < 4; ++q) h[q] += J[k * nv + (r0 + q < nv ? r0 + q : r0)] * jc;
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int ir = r0 + q;
            if (ir >= nv || ic > ir) continue;
            if (ir == ic) h[q] += sd[kb * nv + ir] - schur[2 * kb * nv + ir];
            Sb[tri_at(kb * nv + ir, kb * nv + ic)] = h[q];
          }
        }
    }
    for (int r = warp; r < nv; r += NW)                // knots 0 and T-1 meet on each DOF's own band only
      for (int ic = lane; ic < nv; ic += kWarp)        // (T = 3: acceleration row 0 couples them)
        Sb[tri_at(nv + r, ic)] = ic == r ? (T == 3 ? c2 : 0.0) - schur[nv + r] : 0.0;
    for (int cc = tid; cc < nb; cc += NT) {
      const int kc = cc >= nv, ic = cc - kc * nv;
      Sb[tri_at(nb, cc)] = -g[(kc ? T - 1 : 0) * nv + ic] - schur[(3 + kc) * nv + ic];
    }
    __syncthreads();
    // L D L^T of S in panels of kPan columns: warp 0 eliminates the panel on its first 32 rows (lane r row
    // k0 + r; every lane carries the pivots, so that one reciprocal and one multiply-add separate two of
    // them), one thread per row the rows below, and the block updates the rest of S: one entry per thread
    // while they are few, else 4 x 4 tiles (the same sums in the same order).  The panel's entries stay as L;
    // sdi 1 / pivot, sd pivot.
    constexpr int kPan = 8;
    bool pos = true;
    for (int k0 = 0; k0 < nb; k0 += kPan) {
      const int pw = nb - k0 < kPan ? nb - k0 : kPan, k1 = k0 + pw;
      if (warp == 0) {
        const int r = k0 + lane < nb ? k0 + lane : nb;
        double* row = Sb + tri_at(r, k0);
        double a[kPan], myd = 1.0, myi = 1.0;
#pragma unroll
        for (int j = 0; j < kPan; ++j) a[j] = j < pw && k0 + j <= r ? row[j] : 0.0;
        double d = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
        for (int j = 0; j < kPan; ++j) {
          if (j >= pw) break;
          pos = pos && d > 0.0;
          const double aj = a[j];
          double bj[kPan];
#pragma unroll
          for (int k = j + 1; k < kPan; ++k) bj[k] = __shfl_sync(0xffffffffu, aj, k);
          const double nd = j + 1 < kPan ? __shfl_sync(0xffffffffu, a[j + 1 < kPan ? j + 1 : 0], j + 1) : 1.0;
          const double b1 = j + 1 < kPan ? bj[j + 1 < kPan ? j + 1 : 0] : 0.0, bb = b1 * b1;
          const double ri = fast_rcp(d);
          const double lj = aj * ri;
#pragma unroll
          for (int k = j + 1; k < kPan; ++k) a[k] -= lj * bj[k];
          a[j] = lj;
          myd = lane == j ? d : myd;
          myi = lane == j ? ri : myi;
          d = nd - bb * ri;
        }
        if (lane < pw) { sd[k0 + lane] = myd; sdi[k0 + lane] = myi; }
        if (k0 + lane <= nb) {
#pragma unroll
          for (int j = 0; j < kPan; ++j)
            if (j < pw && j < lane) row[j] = a[j];
        }
      }
      if (__syncthreads_or(warp == 0 && !pos)) return false;
      if (k0 + kWarp <= nb) {
        for (int r = k0 + kWarp + tid; r <= nb; r += NT) {           // W L^T = S, stored as W / pivot
          double w[kPan];
          double* row = Sb + tri_at(r, k0);
#pragma unroll
          for (int j = 0; j < kPan; ++j) w[j] = j < pw ? row[j] : 0.0;
#pragma unroll
          for (int j = 0; j < kPan; ++j) {
            if (j < pw) {
#pragma unroll
              for (int k = j + 1; k < kPan; ++k)
                if (k < pw) w[k] -= w[j] * Sb[tri_at(k0 + k, k0 + j)];
              row[j] = w[j] * sdi[k0 + j];
            }
          }
        }
        __syncthreads();
      }
      if (k1 >= nb) break;
      // S[r][c] -= sum_j L[r][j] pivot_j L[c][j] for k1 <= c <= r <= nb, c < nb (a full panel here)
      const int nr = nb + 1 - k1, ne = nr * (nr + 1) / 2 - 1;
      if (ne <= 4 * NT) {
        for (int e = tid; e < ne; e += NT) {
          const int2 rc = tri_decode(e);
          const double *lr = Sb + tri_at(k1 + rc.x, k0), *lc = Sb + tri_at(k1 + rc.y, k0);
          double acc = 0.0;                                        // in the tiles' order
#pragma unroll
          for (int j = 0; j < kPan; ++j) acc += lr[j] * (lc[j] * sd[k0 + j]);
          Sb[tri_at(k1 + rc.x, k1 + rc.y)] -= acc;
        }
      } else {
        const int nt = (nr + 3) >> 2;
        for (int e = tid; e < nt * (nt + 1) / 2; e += NT) {
          const int2 ij = tri_decode(e);
          const int r0 = k1 + 4 * ij.x, c0 = k1 + 4 * ij.y;
          double acc[4][4];
          const double *lr[4], *lc[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {                            // rows past the last repeat it (not stored)
            lr[q] = Sb + tri_at(r0 + q < nb ? r0 + q : nb, k0);
            lc[q] = Sb + tri_at(c0 + q < nb ? c0 + q : nb, k0);
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[q][v] = 0.0;
          }
#pragma unroll 4
          for (int j = 0; j < kPan; ++j) {
            const double dj = sd[k0 + j];
            double x[4], y[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { x[q] = lr[q][j]; y[q] = lc[q][j] * dj; }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
              for (int v = 0; v < 4; ++v) acc[q][v] += x[q] * y[v];
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int r = r0 + q, cc = c0 + v;
              if (r <= nb && cc <= r && cc < nb) Sb[tri_at(r, cc)] -= acc[q][v];
            }
        }
      }
      __syncthreads();
    }
    __syncthreads();
    // row nb now holds D^-1 L^-1 b: z = L^-T of it, panel by panel from the last
    for (int e = tid; e < nb; e += NT) zb[e] = Sb[tri_at(nb, e)];
    __syncthreads();
    for (int k0 = (nb - 1) / kPan * kPan; k0 >= 0; k0 -= kPan) {
      const int pw = nb - k0 < kPan ? nb - k0 : kPan;
      if (warp == 0) {
        double v = lane < pw ? zb[k0 + lane] : 0.0, lc[kPan];
#pragma unroll
        for (int j = 1; j < kPan; ++j) lc[j] = j < pw && lane < j ? Sb[tri_at(k0 + j, k0 + lane)] : 0.0;
#pragma unroll
        for (int j = kPan - 1; j >= 1; --j) {
          const double zj = __shfl_sync(0xffffffffu, v, j);
          v -= lc[j] * zj;
        }
        if (lane < pw) zb[k0 + lane] = v;
      }
      __syncthreads();
      for (int cc = tid; cc < k0; cc += NT) {
        double v = zb[cc];
        for (int j = 0; j < pw; ++j) v -= Sb[tri_at(k0 + j, cc)] * zb[k0 + j];
        zb[cc] = v;
      }
      __syncthreads();
    }
    // interior step of DOF i: P_i d = y - h0 z(knot 0) - hT z(knot T-1)
    if (tw && tid < 2 * nv) {
      // forward into delta, then backward in place: from both ends to the middle block and back out
      const int km = m / 2;
      const int i = tid >> 1, side = tid & 1;
      const double z0 = zb[i], zT = zb[nv + i], zs = side ? zT : z0;
      if (side == 0) {
        delta[i] = z0;
        delta[(T - 1) * nv + i] = zT;
      }
      const int p0 = side ? m - 1 : 0, dir = side ? -1 : 1, steps = side ? m - km - 2 : km;
      const int step = dir * nv;
      double y1 = 0, y2 = 0, di2 = 0.0, di1 = 0.0;
      int o = p0 * nv + i;
      double l1 = bl1[o], di = bdi[o], gy = -g[o + nv];
      for (int q = 0; q < steps; ++q) {
        const double l1_n = bl1[o + step], di_n = bdi[o + step], gy_n = -g[o + step + nv];
        const double rhs = q == 0 ? gy + 2.0 * c2 * zs : q == 1 ? gy - c2 * zs : gy;
        const double y = (rhs - c2 * di2 * y2) - l1 * y1;
        delta[o + nv] = y;
        y2 = y1; y1 = y; di2 = di1; di1 = di;
        o += step; l1 = l1_n; di = di_n; gy = gy_n;
      }
      // middle block: this side's last two rows, multipliers as in the factorization
      const double n1 = bl1[(side ? km + 1 : km) * nv + i];
      const double n2 = c2 * di2, f1 = c2 * di1;
      const double r_near = n1 * y1 + n2 * y2, r_far = f1 * y1;
      const double o_near = __shfl_xor_sync(tmask, r_near, 1), o_far = __shfl_xor_sync(tmask, r_far, 1);
      const double on1 = __shfl_xor_sync(tmask, n1, 1);
      const double x0r = -g[(km + 1) * nv + i] - (side ? o_near : r_near) - (side ? r_far : o_far);
      const double x1r = -g[(km + 2) * nv + i] - (side ? o_far : r_far) - (side ? r_near : o_near);
      const double dk = bdi[km * nv + i], dk1 = bdi[(km + 1) * nv + i];
      const double lm = (h1 - c2 * n1 - c2 * on1) * dk;           // B10 / B00 (symmetric in the sides)
      const double x1 = (x1r - lm * x0r) * dk1, x0 = x0r * dk - lm * x1;
      if (side == 0) {
        delta[(km + 1) * nv + i] = x0;
        delta[(km + 2) * nv + i] = x1;
      }
      // back substitution outwards: x_p = z_p / pivot_p - (near multiplier) x_(p+dir') - c2 / pivot_p x_(p+2dir')
      double xa = side ? x1 : x0, xb = side ? x0 : x1;            // the next two rows towards the middle
      double ln = n1;                                             // the row towards the middle, relative to p
      o -= step;
      double dp = bdi[o], yp = delta[o + nv], lp = bl1[o];
      for (int q = steps - 1; q >= 0; --q) {
        const int on = q > 0 ? o - step : o;
        const double dp_n = bdi[on], yp_n = delta[on + nv], lp_n = bl1[on];
        const double y = (yp * dp - c2 * dp * xb) - ln * xa;
        delta[o + nv] = y;
        xb = xa; xa = y;
        ln = lp;
        o = on; dp = dp_n; yp = yp_n; lp = lp_n;
      }
    } else if (!tw && tid < nv) {
      const int i = tid;
      const double z0 = zb[i], zT = zb[nv + i];
      delta[i] = z0;
      delta[(T - 1) * nv + i] = zT;
      double y1 = 0, y2 = 0;
      for (int p = 0; p < m; ++p) {
        const int t = p + 1;
        const double l1 = bl1[p * nv + i], l2 = (p >= 2) ? c2 * bdi[(p - 2) * nv + i] : 0.0;
        const double y = -g[t * nv + i] - h0_at(t) * z0 - hT_at(t) * zT - l1 * y1 - l2 * y2;
        delta[t * nv + i] = y;
        y2 = y1; y1 = y;
      }
      y1 = y2 = 0;
      for (int p = m - 1; p >= 0; --p) {
        const double di = bdi[p * nv + i];
        const double l1n = (p + 1 < m) ? bl1[(p + 1) * nv + i] : 0.0;   // L[p+1][p]
        const double l2n = (p + 2 < m) ? c2 * di : 0.0;                  // L[p+2][p] = c2 / D[p]
        const double y = delta[(p + 1) * nv + i] * di - l1n * y1 - l2n * y2;
        delta[(p + 1) * nv + i] = y;
        y2 = y1; y1 = y;
      }
    }
    __syncthreads();
    return true;
  };

  // ---- GN / LM loop (gauss_newton.py:27-76, levenberg_marquardt.py:83-135) ----
  // cost_of and newton_solve have ONE call site each (they are inlined: a second one would be a second
  // copy of the code): the first pass evaluates the start, every later one a trial point, and a last
  // pass the returned x when the goal gradient is wanted and the final trial was rejected.
  const bool lm = S.optimizer == BR_OPT_LM;
  const bool want_goal = P.goal_grad && has_goal;
  double cost = 0.0, lam = lm ? (double)S.lam0 : 0.0, gnorm = 0.0;
  bool need = true, started = false, at_x = true;
  int status = BR_IK_MAXITER, flags = 0, it = 0;
  const double* xe = x;
  for (;;) {
    const double cn = cost_of(xe);
    if (!started) {
      started = true;
      cost = cn;
    } else if (at_x) {                                             // the last pass
      break;
    } else {
      ++it;
      if (!isfinite(cn)) flags |= BR_IK_FLAG_NONFINITE;
      if (!lm || cn < cost) {
        double* t = x; x = xn; xn = t;
        at_x = true;
        cost = cn;
        need = true;
        if (lm) lam = fmax(lam / S.factor, (double)S.lam_min);
        if (gnorm < S.tol) { status = BR_IK_CONVERGED; break; }
      } else {
        lam = fmin(lam * S.factor, (double)S.lam_max);
      }
    }
    if (it >= S.max_iter) {
      if (!want_goal || at_x) break;
      at_x = true;
      xe = x;
      continue;
    }
    if (need) { gnorm = build(); need = false; }
    bool ok = false;
    double extra = 0.0;
    for (int k = 0; k < 9 && !ok; ++k) {                           // retries with diagonal regularisation
      ok = newton_solve((lm ? lam : (double)S.gn_eps) + extra);
      if (!ok) flags |= BR_IK_FLAG_REGULARIZED;
      extra = k == 0 ? 1e-9 : extra * 10.0;
    }
    if (!ok) {
      for (int e = tid; e < n; e += NT) delta[e] = 0.0;
      __syncthreads();
    }
    if (kManifold) {                                               // Model.integrate per knot (trajopt.py:159-169)
      retract_knots();
    } else {
      for (int e = tid; e < n; e += NT) xn[e] = x[e] + delta[e];
    }
    __syncthreads();
    at_x = false;
    xe = xn;
  }
  __syncthreads();
  float* xo = P.x + traj * (int64_t)nqT;
  for (int e = tid; e < nqT; e += NT) xo[e] = (float)x[e];
  if (want_goal) {                                                 // rg holds the pose error of x
    if (tid == 0) {
      const double3 v = d3(rg[0], rg[1], rg[2]);
      const double3 w = d3(rg[3], rg[4], rg[5]);
      const DJrInv Jl = djr_inv_se3_rolled<20>(dscale(v, -1.0), dscale(w, -1.0));   // Jl^-1(xi) = Jr^-1(-xi)
      double3 gl, ga;
      djr_inv_T_apply(Jl, v, w, gl, ga);
      const double k = -wg * wg;
      float* o = P.goal_grad + traj * 6;
      o[0] = (float)(k * gl.x); o[1] = (float)(k * gl.y); o[2] = (float)(k * gl.z);
      o[3] = (float)(k * ga.x); o[4] = (float)(k * ga.y); o[5] = (float)(k * ga.z);
    }
  }
  if (tid == 0) {
    P.iters[traj] = it;
    P.status[traj] = status | (flags << 8);
    P.cost[traj] = (float)cost;
  }
}

}  // namespace br

using namespace br;

extern "C" int br_trajopt_solve(const br_tree_t* tree, int32_t frame_id, int64_t n_traj, int32_t knots,
                                const float* x0, const float* x_ref, const float* goal, const float* start,
                                const br_traj_settings_t* settings, float* x, int32_t* iters, int32_t* status,
                                float* cost, float* goal_grad, void* stream) {
  int st = validate_tree(tree);
  if (st) return st;
  if (!settings || n_traj < 0 || knots < 3) return BR_EINVAL;
  if (knots > BR_MAX_TRAJ_KNOTS || tree->nv > BR_MAX_TRAJ_NV) return BR_ETOOBIG;
  {
    const int ok = (1 << (BR_JOINT_TRANSLATION + 1)) - 1;        // every kind of the tree table
    if (tree->kinds == 0 || (tree->kinds & ~ok)) return BR_EINVAL;
  }
  const int manifold_kinds = (1 << BR_JOINT_FREE_FLYER) | (1 << BR_JOINT_SPHERICAL) | (1 << BR_JOINT_PLANAR) |
                             (1 << BR_JOINT_REVOLUTE_UNBOUNDED);
  if (!(tree->kinds & manifold_kinds) && tree->nq != tree->nv) return BR_EINVAL;
  if (frame_id < 0 || frame_id >= tree->nframes) return BR_EINVAL;
  if (n_traj == 0) return BR_OK;
  if (!x0 || !goal || !x || !iters || !status || !cost) return BR_EINVAL;
  if (settings->max_iter < 0 || !(settings->dt > 0.f)) return BR_EINVAL;
  TrajParams p = {};
  p.tree = *tree;
  p.s = *settings;
  p.frame_id = frame_id;
  p.T = knots;
  p.n = n_traj;
  p.x0 = x0; p.xref = x_ref; p.goal = goal; p.start = start;
  p.x = x; p.iters = iters; p.status = status; p.cost = cost; p.goal_grad = goal_grad;
  const bool floating = (tree->kinds & manifold_kinds) != 0;
  const TrajLayout L(tree->njoints, tree->nq, tree->nv, knots, floating);
  const size_t bytes = (size_t)L.total * sizeof(double);
  const DeviceInfo& dev = device_info();
  if ((int64_t)bytes > dev.max_smem_optin) return BR_ETOOBIG;
  if (n_traj > 0x7fffffff) return BR_ETOOBIG;
  const bool wide = n_traj <= dev.sms || 2 * ((int64_t)bytes + 1024) > dev.smem_per_sm;
  auto kern = floating ? (wide ? traj_gn_kernel<true, 256> : traj_gn_kernel<true, 128>)
                       : (wide ? traj_gn_kernel<false, 256> : traj_gn_kernel<false, 128>);
  static int configured[4][16] = {{0}};
  int& conf = configured[(floating ? 2 : 0) + (wide ? 1 : 0)][dev.device & 15];
  if ((int)bytes > conf) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    conf = (int)bytes;
  }
  kern<<<(unsigned)n_traj, wide ? 256 : 128, bytes, (cudaStream_t)stream>>>(p);
  return (int)cudaGetLastError();
}
