// fk_adjoint.cu — pose loss through forward kinematics and its hand-written adjoint.
//
// Loss per configuration:  L(q) = sum_f w_f |log(T_f^-1 * oMf(q))|^2
// (the reference obtains dL/dq by torch autograd through every SE3 op of
// src/better_robot/kinematics/forward.py:73-135 and lie/_torch_native_backend.py).
//
// Adjoint, one warp per configuration (two configurations per pass of the warp where their
// frames fit one lane each: the per-frame stage then runs on both at once):
//   * g_f = 2 w_f Jr^-1(xi_f)^T xi_f is dL/d(body twist of frame f), with the exact
//     SE3 Jr^-1 (closed form jr_inv_T_xi; autograd differentiates se3_log exactly);
//   * F_f = Ad(oMf^-1)^T g_f = [R g_lin; p x (R g_lin) + R g_ang] is the same
//     sensitivity as a wrench at the world origin;
//   * dL/dv_c = sum_{f : c supports f} <S_c, F_f> = <S_c, W_j> with S_c the world twist
//     of tangent column c ([o x a; a] rotation, [a; 0] translation) and W_j the summed
//     wrench of the frames that c's joint j moves — a reverse accumulation over the tree
//     without any per-joint tape;
//   * revolute / prismatic / translation: dL/dq = dL/dv; free-flyer and spherical: the
//     body twist of the joint maps to raw q = [t, quat] through R (translation) and the
//     normalisation of the quaternion ((I - u u^T)/|quat| and du -> 2 vec(u* (x) du));
//     unbounded revolute: th = atan2(s, c); planar: [x, y] through R, the angle through
//     the reference's half-angle formula (dth/dc = -1/sin th, no dependence on s).
// World joint placements are either recomputed from q (no saved state) or read
// from the forward pass (store mode, [B, njoints, 7]).
#include <cuda_runtime.h>
#include <stdint.h>

#include "br_common.cuh"
#include "br_fk.cuh"
#include "br_lie.cuh"

namespace br {

struct LossParams {
  const float* q;          // [B, nq]
  const float* targets;    // [B, nf, 7]
  const float* weights;    // [nf] or [B, nf]
  const float* grad_loss;  // [B] (backward); null: the gradient of each configuration's own loss
  const float* oMi_in;     // [B, nj, 7] (backward, store mode) or null
  float* loss;             // [B] (forward, or with the gradient when not null)
  float* oMi_out;          // [B, nj, 7] (forward, store mode) or null
  float* grad_q;           // [B, nq] (backward)
  int64_t batch;
  int32_t nf;
  int32_t weights_per_config;
  int32_t path_slots;      // lane kernel: known bound on the waiting wrenches of a path, -1 if none
  int32_t frames[BR_MAX_TARGETS];
};

struct LossLayout {
  int parent, jtype, idxq, axis, place, cjoint, ckind, caxis, fparent, fplace, fsup;
  int cta_floats;
  int in0, in1, poseT, poseQ, anc, F, W, gv, stage;
  int pair;   // configurations per pass (2 or 1)
  int inlen;  // floats of one configuration's inputs (16-byte multiple)
  int warp_floats;
  // A warp's slice with two configurations per pass above this many floats would leave one
  // 8-warp CTA per SM instead of two (the humanoid at 12 frames takes 2,644).
  static constexpr int kPairMaxWarpFloats = 3456;
  __host__ __device__ LossLayout(int nj, int nq, int nv, int nf) {
    int o = 0;
    auto take = [&](int n) { int r = o; o += round4(n); return r; };
    parent = take(nj); jtype = take(nj); idxq = take(nj); axis = take(4 * nj); place = take(8 * nj);
    cjoint = take(nv); ckind = take(nv); caxis = take(4 * nv);
    fparent = take(nf); fplace = take(8 * nf); fsup = take(2 * nf);
    cta_floats = o;
    inlen = round4(nq + 7 * nj + 7 * nf);
    // two configurations per pass when both configurations' frames fit one lane each and the
    // slice stays small enough, else one
    for (pair = 2 * nf <= 32 ? 2 : 1;; pair = 1) {
      o = 0;
      // the inputs of a pass's configurations (q, stored oMi, targets), double buffered: the
      // next pass's are copied in (cp.async) while this one is computed
      in0 = take(pair * inlen); in1 = take(pair * inlen);
      poseT = take(pair * 4 * nj); poseQ = take(pair * 4 * nj); anc = take(nj);
      F = take(pair * 8 * nf);  // world wrench per frame (f.xyz, pad, tau.xyz, pad), per configuration
      W = take(8 * nj);         // summed wrench of the frames each joint moves (same layout)
      gv = take(nv);            // dL/dv
      stage = take(nj * 7);     // oMi staging (store mode)
      warp_floats = o;
      if (pair == 1 || warp_floats <= kPairMaxWarpFloats) break;
    }
  }
};

template <bool kBackward>
__global__ void __launch_bounds__(256, 2) pose_loss_kernel(const br_tree_t tree, const LossParams p) {
  extern __shared__ __align__(16) float smem[];
  const int nj = tree.njoints, nq = tree.nq, nv = tree.nv, nf = p.nf;
  const LossLayout L(nj, nq, nv, nf);
  int* s_parent = reinterpret_cast<int*>(smem + L.parent);
  int* s_jtype = reinterpret_cast<int*>(smem + L.jtype);
  int* s_idxq = reinterpret_cast<int*>(smem + L.idxq);
  float* s_axis = smem + L.axis;
  float* s_place = smem + L.place;
  int* s_cjoint = reinterpret_cast<int*>(smem + L.cjoint);
  int* s_ckind = reinterpret_cast<int*>(smem + L.ckind);
  float* s_caxis = smem + L.caxis;
  int* s_fparent = reinterpret_cast<int*>(smem + L.fparent);
  float* s_fplace = smem + L.fplace;
  unsigned long long* s_fsup = reinterpret_cast<unsigned long long*>(smem + L.fsup);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpc = blockDim.x >> 5;
  for (int i = threadIdx.x; i < nj; i += blockDim.x) {
    s_parent[i] = tree.parent[i];
    s_jtype[i] = tree.jtype[i];
    s_idxq[i] = tree.idx_q[i];
    for (int k = 0; k < 4; ++k) s_axis[4 * i + k] = tree.axis[4 * i + k];
    for (int k = 0; k < 8; ++k) s_place[8 * i + k] = tree.placement[8 * i + k];
  }
  for (int c = threadIdx.x; c < nv; c += blockDim.x) {
    s_cjoint[c] = tree.col_joint[c];
    s_ckind[c] = tree.col_kind[c];
    for (int k = 0; k < 4; ++k) s_caxis[4 * c + k] = tree.col_axis[4 * c + k];
  }
  for (int f = threadIdx.x; f < nf; f += blockDim.x) {
    const int id = p.frames[f];
    s_fparent[f] = tree.frame_parent[id];
    for (int k = 0; k < 8; ++k) s_fplace[8 * f + k] = tree.frame_placement[8 * id + k];
  }
  __syncthreads();
  // joints that move each frame: bit j set iff joint j supports the frame's parent joint
  for (int f = threadIdx.x; f < nf; f += blockDim.x) s_fsup[f] = tree.support[s_fparent[f]];
  __syncthreads();

  float* w = smem + L.cta_floats + warp * L.warp_floats;
  int* wanc = reinterpret_cast<int*>(w + L.anc);
  float* wW = w + L.W;
  float* wg = w + L.gv;
  float* wst = w + L.stage;
  const int64_t stride = (int64_t)gridDim.x * wpc;
  const bool stored = kBackward && p.oMi_in;
  const int o_pose = nq, o_tgt = nq + (stored ? 7 * nj : 0);   // offsets in an input buffer
  // Configurations b and b + stride are taken as a pair when both fit the frame stage's lanes
  // (2 nf <= 32): their FK, per-joint and per-column stages run one after the other over the
  // whole warp, the per-frame stage (one lane per frame) over both at once.  Pose set, wrench
  // set and input buffer hp belong to configuration b + hp * stride.
  const int pair = L.pair;
  const int64_t step = stride * pair;
  // queue the copies of configuration bb's inputs into `dst` (nothing past the end of the
  // batch): 4-byte cp.async, the rows are 4-byte aligned only
  auto prefetch = [&](int64_t bb, float* dst) {
    if (bb < p.batch) {
      const float* qb = p.q + bb * nq;
      for (int i = lane; i < nq; i += kWarp) cp_async4(dst + i, qb + i);
      if (stored) {
        const float* ob = p.oMi_in + bb * (int64_t)nj * 7;
        for (int i = lane; i < nj * 7; i += kWarp) cp_async4(dst + o_pose + i, ob + i);
      }
      const float* tb = p.targets + bb * (int64_t)nf * 7;
      for (int i = lane; i < nf * 7; i += kWarp) cp_async4(dst + o_tgt + i, tb + i);
    }
  };
  float* cur = w + L.in0;                  // this pass's inputs; the other buffers: the next pass's
  float* nxt = w + L.in1;
  int64_t b = (int64_t)blockIdx.x * wpc + warp;
  for (int hp = 0; hp < pair; ++hp) prefetch(b + hp * stride, cur + hp * L.inlen);
  cp_async_commit();                       // one commit group per pass
  for (; b < p.batch; b += step) {
    __syncwarp();                          // every lane is done with the buffers refilled next
    for (int hp = 0; hp < pair; ++hp) prefetch(b + step + hp * stride, nxt + hp * L.inlen);
    cp_async_commit();
    cp_async_wait_groups<1>();             // this pass's copies (all but the newest group)
    __syncwarp();
    const float* wq0 = cur;
    { float* t = cur; cur = nxt; nxt = t; }
    const int np = (pair == 2 && b + stride < p.batch) ? 2 : 1;
    for (int hp = 0; hp < np; ++hp) {
      const int64_t bh = b + hp * stride;
      const float* wqh = wq0 + hp * L.inlen;
      float* wpT = w + L.poseT + hp * 4 * nj;
      float* wpQ = w + L.poseQ + hp * 4 * nj;
      if (stored) {
        const float* ob = wqh + o_pose;
        for (int i = lane; i < nj * 7; i += kWarp) {
          const int j = i / 7, c = i - 7 * j;
          if (c < 3) wpT[4 * j + c] = ob[i];
          else wpQ[4 * j + c - 3] = ob[i];
        }
        __syncwarp();
      } else {
        // forward kinematics by pointer jumping (see fk_jac.cu)
        for (int j = lane; j < nj; j += kWarp) {
          store_split(wpT, wpQ, j, local_transform(s_jtype[j], load_pose8(s_place + 8 * j), s_axis + 4 * j,
                                                   wqh + s_idxq[j]));
          wanc[j] = s_parent[j];
        }
        __syncwarp();
        for (int r = 0; r < tree.rounds; ++r) {
          Pose A[2], Tj[2];
          int aa[2], an[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int j = lane + kWarp * k;
            an[k] = (j < nj) ? wanc[j] : -1;
            if (an[k] >= 0) {
              A[k] = load_split(wpT, wpQ, an[k]);
              Tj[k] = load_split(wpT, wpQ, j);
              aa[k] = wanc[an[k]];
            }
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int j = lane + kWarp * k;
            if (an[k] >= 0) {
              store_split(wpT, wpQ, j, compose(A[k], Tj[k]));
              wanc[j] = aa[k];
            }
          }
          __syncwarp();
        }
        if (!kBackward && p.oMi_out) {
          for (int j = lane; j < nj; j += kWarp) store_pose7(wst + 7 * j, load_split(wpT, wpQ, j));
          __syncwarp();
          warp_copy(p.oMi_out + bh * (int64_t)nj * 7, wst, nj * 7, lane);
          __syncwarp();
        }
      }
    }
    // per-frame residual, loss and (backward) world wrench; frame f of the pair's second
    // configuration on lane nf + f
    float acc0 = 0.f, acc1 = 0.f;
    for (int i = lane; i < np * nf; i += kWarp) {
      const int hp = i >= nf ? 1 : 0;
      const int f = i - hp * nf;
      const int64_t bh = b + hp * stride;
      const Pose Tf = compose(load_split(w + L.poseT + hp * 4 * nj, w + L.poseQ + hp * 4 * nj, s_fparent[f]),
                              load_pose8(s_fplace + 8 * f));
      const float* tp = wq0 + hp * L.inlen + o_tgt + 7 * f;
      const Pose Tt{f3(tp[0], tp[1], tp[2]), make_float4(tp[3], tp[4], tp[5], tp[6])};
      float3 v, om;
      se3_log(compose(inverse(Tt), Tf), v, om);
      const float wf = __ldg(p.weights + (p.weights_per_config ? bh * nf + f : f));
      const float lf = wf * (dot(v, v) + dot(om, om));
      if (hp) acc1 += lf; else acc0 += lf;
      if (kBackward) {
        float3 gl, ga;
        jr_inv_T_xi(v, om, gl, ga);
        const float s2 = 2.f * wf;
        const float3 fw = qrot(Tf.q, scale(gl, s2));
        const float3 tau = add(cross(Tf.t, fw), qrot(Tf.q, scale(ga, s2)));
        float* wF = w + L.F + hp * 8 * nf;
        *reinterpret_cast<float4*>(wF + 8 * f) = make_float4(fw.x, fw.y, fw.z, 0.f);
        *reinterpret_cast<float4*>(wF + 8 * f + 4) = make_float4(tau.x, tau.y, tau.z, 0.f);
      }
    }
    if (!kBackward || p.loss) {
      // the second configuration's terms moved to lanes 0..nf-1 first, so that both sums
      // take the same order (that of a configuration processed alone)
      if (pair == 2) {
        const float m1 = __shfl_sync(0xffffffffu, acc1, (lane + nf) & (kWarp - 1));
        acc1 = lane + nf < kWarp ? m1 : 0.f;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        acc0 += __shfl_xor_sync(0xffffffffu, acc0, o);
        acc1 += __shfl_xor_sync(0xffffffffu, acc1, o);
      }
      if (lane == 0) {
        p.loss[b] = acc0;
        if (np == 2) p.loss[b + stride] = acc1;
      }
    }
    if (!kBackward) continue;
    __syncwarp();
    for (int hp = 0; hp < np; ++hp) {
      const int64_t bh = b + hp * stride;
      const float* wqh = wq0 + hp * L.inlen;
      const float* wF = w + L.F + hp * 8 * nf;
      const float* wpT = w + L.poseT + hp * 4 * nj;
      const float* wpQ = w + L.poseQ + hp * 4 * nj;
      // dL/dv_c = sum over the frames f that column c moves of <S_c, F_f> = <S_c, W_j>, where
      // W_j sums F_f over the frames that c's joint j moves: one sum per joint, one dot per column
      for (int j = lane; j < nj; j += kWarp) {
        float4 sf = make_float4(0.f, 0.f, 0.f, 0.f), st = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int f = 0; f < nf; ++f) {
          if ((s_fsup[f] >> j) & 1ull) {
            const float4 fw = *reinterpret_cast<const float4*>(wF + 8 * f);
            const float4 tq = *reinterpret_cast<const float4*>(wF + 8 * f + 4);
            sf.x += fw.x; sf.y += fw.y; sf.z += fw.z;
            st.x += tq.x; st.y += tq.y; st.z += tq.z;
          }
        }
        *reinterpret_cast<float4*>(wW + 8 * j) = sf;
        *reinterpret_cast<float4*>(wW + 8 * j + 4) = st;
      }
      __syncwarp();
      const float go = p.grad_loss ? __ldg(p.grad_loss + bh) : 1.f;
      for (int c = lane; c < nv; c += kWarp) {
        const int j = s_cjoint[c];
        const Pose Tj = load_split(wpT, wpQ, j);
        const float3 a = qrot(Tj.q, f3(s_caxis[4 * c], s_caxis[4 * c + 1], s_caxis[4 * c + 2]));
        const float3 m = s_ckind[c] == 0 ? cross(Tj.t, a) : a;  // linear part of the world twist
        const float3 an = s_ckind[c] == 0 ? a : f3(0.f, 0.f, 0.f);
        const float4 fw = *reinterpret_cast<const float4*>(wW + 8 * j);
        const float4 tq = *reinterpret_cast<const float4*>(wW + 8 * j + 4);
        wg[c] = (dot(m, f3(fw.x, fw.y, fw.z)) + dot(an, f3(tq.x, tq.y, tq.z))) * go;
      }
      __syncwarp();
      float* gq = p.grad_q + bh * nq;
      for (int j = lane; j < nj; j += kWarp) {
        const int jt = s_jtype[j];
        const int iq = s_idxq[j];
        if (jt == BR_JOINT_REVOLUTE || jt == BR_JOINT_PRISMATIC) {
          gq[iq] = wg[tree.idx_v[j]];
        } else if (jt == BR_JOINT_TRANSLATION) {                     // q is the body translation
          const int iv = tree.idx_v[j];
          gq[iq] = wg[iv]; gq[iq + 1] = wg[iv + 1]; gq[iq + 2] = wg[iv + 2];
        } else if (jt == BR_JOINT_REVOLUTE_UNBOUNDED) {
          // th = atan2(s, c) (revolute.py:206-211): dth/dc = -s / r^2, dth/ds = c / r^2
          const float g = wg[tree.idx_v[j]];
          const float c = wqh[iq], sn = wqh[iq + 1];
          const float r2 = fmaxf(c * c + sn * sn, 1e-30f);
          gq[iq] = -g * sn / r2;
          gq[iq + 1] = g * c / r2;
        } else if (jt == BR_JOINT_PLANAR) {
          // T = ([x, y, 0], Rz(th)) with cos(th/2) = sqrt((1+c)/2), sin(th/2) = sqrt((1-c)/2) sign(s)
          // (planar.py:20-41): body twist = (R^T [dx, dy, 0], e_z dth), dth/dc = -1 / sin(th),
          // and th does not depend on s away from s = 0
          const int iv = tree.idx_v[j];
          const float c = wqh[iq + 2], sn = wqh[iq + 3];
          const float4 hq = planar_quat(c, sn);
          const float ct = hq.w * hq.w - hq.z * hq.z, st = 2.f * hq.z * hq.w;
          const float g0 = wg[iv], g1 = wg[iv + 1], g2 = wg[iv + 2];
          gq[iq] = ct * g0 - st * g1;
          gq[iq + 1] = st * g0 + ct * g1;
          gq[iq + 2] = -g2 / st;
          gq[iq + 3] = 0.f;
        } else if (jt == BR_JOINT_FREE_FLYER || jt == BR_JOINT_SPHERICAL) {
          // free-flyer [t, quat] / spherical [quat]: the quaternion's body rotation
          const bool ff = jt == BR_JOINT_FREE_FLYER;
          const int iv = tree.idx_v[j];
          const int qo = ff ? iq + 3 : iq;                          // first quaternion slot
          const int vo = ff ? iv + 3 : iv;                          // first rotation column
          const float4 qr = make_float4(wqh[qo], wqh[qo + 1], wqh[qo + 2], wqh[qo + 3]);
          const float4 u = qnormalize(qr);
          const float n = fmaxf(sqrtf(qr.x * qr.x + qr.y * qr.y + qr.z * qr.z + qr.w * qr.w), 1e-8f);
          const float3 ga = f3(wg[vo], wg[vo + 1], wg[vo + 2]);
          // quaternion: delta_ang = 2 vec(u* (x) du), du = (I - u u^T) dquat / n
          float4 h;
          h.x = u.w * ga.x - u.z * ga.y + u.y * ga.z;
          h.y = u.z * ga.x + u.w * ga.y - u.x * ga.z;
          h.z = -u.y * ga.x + u.x * ga.y + u.w * ga.z;
          h.w = -u.x * ga.x - u.y * ga.y - u.z * ga.z;
          const float uh = u.x * h.x + u.y * h.y + u.z * h.z + u.w * h.w;
          const float s = 2.f / n;
          if (ff) {
            const float3 gt = qrot(u, f3(wg[iv], wg[iv + 1], wg[iv + 2]));  // translation: delta_lin = R^T dt
            gq[iq] = gt.x; gq[iq + 1] = gt.y; gq[iq + 2] = gt.z;
          }
          gq[qo] = s * (h.x - u.x * uh);
          gq[qo + 1] = s * (h.y - u.y * uh);
          gq[qo + 2] = s * (h.z - u.z * uh);
          gq[qo + 3] = s * (h.w - u.w * uh);
        }
      }
      __syncwarp();
    }
  }
  cp_async_wait_groups<0>();               // the (empty) last group
}

// Raw-q chain rules of the multi-slot kinds: the joint's tangent gradient to the gradient of its q
// slots, written over them (qj holds the joint's configuration on entry).
// unbounded revolute: th = atan2(s, c) (revolute.py:206-211), dth/dc = -s / r^2, dth/ds = c / r^2
__device__ __forceinline__ void unbounded_chain(float g, float* qj) {
  const float c = qj[0], sn = qj[1];
  const float r2 = fmaxf(c * c + sn * sn, 1e-30f);
  qj[0] = -g * sn / r2;
  qj[1] = g * c / r2;
}
// planar: T = ([x, y, 0], Rz(th)) with cos(th/2) = sqrt((1+c)/2), sin(th/2) = sqrt((1-c)/2) sign(s)
// (planar.py:20-41): body twist = (R^T [dx, dy, 0], e_z dth), dth/dc = -1 / sin(th), and th does
// not depend on s away from s = 0
__device__ __forceinline__ void planar_chain(float g0, float g1, float g2, float* qj) {
  const float4 hq = planar_quat(qj[2], qj[3]);
  const float ct = hq.w * hq.w - hq.z * hq.z, st = 2.f * hq.z * hq.w;
  qj[0] = ct * g0 - st * g1;
  qj[1] = st * g0 + ct * g1;
  qj[2] = -g2 / st;
  qj[3] = 0.f;
}
// quaternion slots: delta_ang = 2 vec(u* (x) du), du = (I - u u^T) dquat / n; returns the unit u
__device__ __forceinline__ float4 quat_chain(float3 ga, float* qj) {
  const float4 qr = make_float4(qj[0], qj[1], qj[2], qj[3]);
  const float4 u = qnormalize(qr);
  const float n = fmaxf(sqrtf(qr.x * qr.x + qr.y * qr.y + qr.z * qr.z + qr.w * qr.w), 1e-8f);
  float4 h;
  h.x = u.w * ga.x - u.z * ga.y + u.y * ga.z;
  h.y = u.z * ga.x + u.w * ga.y - u.x * ga.z;
  h.z = -u.y * ga.x + u.x * ga.y + u.w * ga.z;
  h.w = -u.x * ga.x - u.y * ga.y - u.z * ga.z;
  const float uh = u.x * h.x + u.y * h.y + u.z * h.z + u.w * h.w;
  const float s = 2.f / n;
  qj[0] = s * (h.x - u.x * uh);
  qj[1] = s * (h.y - u.y * uh);
  qj[2] = s * (h.z - u.z * uh);
  qj[3] = s * (h.w - u.w * uh);
  return u;
}

// ---------------------------------------------------------------------------
// One lane per configuration.
//
// A warp owns a tile of 32 consecutive configurations and walks the tree once, in depth-first
// order, the same joint on all lanes: going down it composes the world placement and evaluates
// the frames of each joint; coming back up it carries the subtree's wrench in the joint's own
// frame.  With W_j = (f, tau) the summed sensitivity to the body twist of joint j,
//   dL/dv_j = the components of W_j along j's motion subspace (tau . axis for a revolute joint:
//             no world axis or origin is needed),
//   W_parent += (R f, R tau + t x R f),  (t, R) = liMi_j.
// So the way up needs liMi_j only (rebuilt from q_j), a wrench survives in shared memory only at
// joints with frames or several children on the current path, and there is neither an idle lane
// nor a shuffle: the warp-per-configuration kernel above spends most of its instructions on
// address arithmetic, shuffles and frames on 24 of 32 lanes.  Joints that move no frame are not
// walked (their gradient is zero).  q is staged as one slab per tile and overwritten in place by
// the gradient; targets are gathered one frame ahead by cp.async.
//
// Bound by its instructions (14.9 k per 32 humanoid configurations at 12 frames, 64 % issue active at 14
// warps per SM).  Humanoid, B = 262,144: loss and gradient together 177 us against 341 us (loss) + 421 us
// (gradient from stored placements) of the warp kernel, 762 us; loss alone 108 us.  On the way there: the
// tables built by one warp with ballots instead of shared atomics (prologue 14.4 k -> 5 k cycles);
// revolute joints turned to z; half-angle sines ahead of the walk instead of on its dependent chain and
// again on the way up (212 -> 193 us); a branch-free sincos, the caller's bound on the waiting wrenches
// (11 -> 4 for the humanoid) and any warp count per CTA (12 -> 14 warps per SM, 193 -> 177 us).
// ---------------------------------------------------------------------------
struct LaneLayout {
  int rec, fid, fplace;                             // CTA tables: visit records, frames in visit order
  int cta_floats;
  int q, cs, ring, slots, saved;                    // per warp
  int warp_floats;
  int qpitch;                                       // floats per configuration row (odd: no bank conflicts)
  int rstep;                                        // floats per ring buffer: 32 targets (+ 32 weights)
  int nslots;
  // Joints whose wrench waits in shared memory on one root-to-leaf path (not the leaf): each has a
  // frame of its own or another child whose subtree has one, all different and none the leaf's, so
  // there are at most nf - 1; fewer if the caller knows better (slots >= 0).
  __host__ __device__ LaneLayout(int nj, int nq, int nf, bool grad, bool per_cfg, int given) {
    int o = 0;
    auto take = [&](int n) { int r = o; o += round4(n); return r; };
    rec = take(32 * (nj + 1)); fid = take(nf); fplace = take(20 * nf);
    cta_floats = o;
    o = 0;
    qpitch = nq | 1;
    q = take(kWarp * qpitch);
    cs = take(kWarp * qpitch);
    rstep = kWarp * (per_cfg ? 8 : 7);
    ring = take(2 * rstep);
    nslots = nf - 1 < nj - 1 ? nf - 1 : nj - 1;
    if (given >= 0 && given < nslots) nslots = given;
    if (!grad || nslots < 0) nslots = 0;
    slots = take(nslots * 6 * kWarp);
    saved = take(7 * kWarp);
    warp_floats = o;
  }
};
// A visit record (32 floats): int4 {jtype | slot << 8 | flags << 16, idx_q, parent visit, first frame |
// end << 16}, placement [t, sign of a turned axis, quaternion], rows [R | t] (12), axis (4),
// ancestors-or-self by visit (uint64), pad.  A frame's: placement (8), rows (12).
constexpr int kRecPlace = 4, kRecRows = 12, kRecAxis = 24, kRecPath = 28;

// visit flags
constexpr int kLaneStored = 1, kLaneBranch = 2, kLaneStop = 4, kLaneChain = 8, kLaneRevZ = 16, kLaneJump = 32;

// Revolute joints about +-x, +-y or +-z are walked about z: a joint's frame is turned by the constant
// Q that takes z to |axis| (a cyclic permutation of the axes: components 0 and +-1/2, no rounding of
// their own), folded into its placement, its children's and its frames'.  Returns 0 for any other
// axis or kind (Q = identity), else the axis' sign; perm: 0 z, 1 x, 2 y.
__device__ __forceinline__ float turned_axis(int jt, float4 a, int& perm) {
  perm = 0;
  if (jt != BR_JOINT_REVOLUTE) return 0.f;
  const int nz = (a.x != 0.f) + (a.y != 0.f) + (a.z != 0.f);
  const float s = a.x + a.y + a.z;
  if (nz != 1 || fabsf(s) != 1.f) return 0.f;
  perm = a.x != 0.f ? 1 : a.y != 0.f ? 2 : 0;
  return s;
}
__device__ __forceinline__ Pose turn_by(const Pose& P, int perm) {       // P * Q
  const float h = perm == 1 ? 0.5f : -0.5f;
  return perm ? Pose{P.t, qmul(P.q, make_float4(h, h, h, 0.5f))} : P;
}
__device__ __forceinline__ Pose turned_from(const Pose& P, int perm) {   // Q^-1 * P
  if (!perm) return P;
  const float h = perm == 1 ? -0.5f : 0.5f;
  const float3 t = perm == 1 ? f3(P.t.y, P.t.z, P.t.x) : f3(P.t.z, P.t.x, P.t.y);
  return Pose{t, qmul(make_float4(h, h, h, 0.5f), P.q)};
}
// rows of [R | t] of a pose, for wrenches: f' = R f, tau' = R tau + t x f'
__device__ __forceinline__ void store_rows(float* m, const Pose& P) {
  const float3 cx = qrot(P.q, f3(1.f, 0.f, 0.f)), cy = qrot(P.q, f3(0.f, 1.f, 0.f)), cz = qrot(P.q, f3(0.f, 0.f, 1.f));
  reinterpret_cast<float4*>(m)[0] = make_float4(cx.x, cy.x, cz.x, P.t.x);
  reinterpret_cast<float4*>(m)[1] = make_float4(cx.y, cy.y, cz.y, P.t.y);
  reinterpret_cast<float4*>(m)[2] = make_float4(cx.z, cy.z, cz.z, P.t.z);
}
__device__ __forceinline__ void carry_wrench(const float* m, float3& f, float3& t) {
  const float4 r0 = reinterpret_cast<const float4*>(m)[0], r1 = reinterpret_cast<const float4*>(m)[1],
               r2 = reinterpret_cast<const float4*>(m)[2];
  f = f3(dot(f3(r0.x, r0.y, r0.z), f), dot(f3(r1.x, r1.y, r1.z), f), dot(f3(r2.x, r2.y, r2.z), f));
  t = f3(dot(f3(r0.x, r0.y, r0.z), t), dot(f3(r1.x, r1.y, r1.z), t), dot(f3(r2.x, r2.y, r2.z), t));
  t = add(t, cross(f3(r0.w, r1.w, r2.w), f));
}

// Visit order of i and j in the depth-first order with children in index order: an ancestor
// first, else by the index of the children at which their paths part.
__device__ __forceinline__ bool visited_before(unsigned long long si, unsigned long long sj) {
  const unsigned long long a = si & ~sj, b = sj & ~si;
  if (a == 0ull) return true;
  if (b == 0ull) return false;
  return (a & (0ull - a)) < (b & (0ull - b));
}

template <bool kGrad>
__global__ void __launch_bounds__(256, 2) pose_loss_lanes_kernel(const br_tree_t tree, const LossParams p) {
  extern __shared__ __align__(16) float smem[];
  const int nj = tree.njoints, nq = tree.nq, nf = p.nf;
  const bool per_cfg = p.weights_per_config != 0;
  const LaneLayout L(nj, nq, nf, kGrad, per_cfg, p.path_slots);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpc = blockDim.x >> 5;
  float* rec = smem + L.rec;
  int* fid = reinterpret_cast<int*>(smem + L.fid);
  float* fplace = smem + L.fplace;
  auto meta_of = [&](int k) { return *reinterpret_cast<const int4*>(rec + 32 * k); };

  // ---- tables in visit order, by the first warp: lane owns joints lane and lane + 32 and frames
  // likewise; masks by ballot, every global load in the first two rounds ----
  // (kLanesStatic is reserved for these; as one struct the kernel took 176.6 instead of 174.6 us)
  __shared__ unsigned long long tsup[BR_MAX_JOINTS];
  __shared__ int trank[BR_MAX_JOINTS], tchild[BR_MAX_JOINTS], tperm[BR_MAX_JOINTS];
  __shared__ unsigned long long s_moves, s_need;
  __shared__ bool s_over;
  if (warp == 0) {
    constexpr unsigned kAll = 0xffffffffu;
    auto ballot64 = [&](bool lo, bool hi) {
      return (unsigned long long)__ballot_sync(kAll, lo) | ((unsigned long long)__ballot_sync(kAll, hi) << 32);
    };
    auto or64 = [&](unsigned long long v) {
      return (unsigned long long)__reduce_or_sync(kAll, (unsigned)v) |
             ((unsigned long long)__reduce_or_sync(kAll, (unsigned)(v >> 32)) << 32);
    };
    auto place8 = [](const float* g) {               // 4-byte aligned tables are accepted
      return Pose{f3(g[0], g[1], g[2]), make_float4(g[4], g[5], g[6], g[7])};
    };
    int jt[2], iq[2], par[2], fpar[2];
    Pose P[2], F[2];
    float4 ax[2];
    float sgn[2];
    bool in[2], mv[2], ord = true;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      in[h] = j < nj;
      jt[h] = in[h] ? tree.jtype[j] : BR_JOINT_FIXED;
      iq[h] = in[h] ? tree.idx_q[j] : 0;
      par[h] = in[h] ? tree.parent[j] : -1;
      ax[h] = in[h] ? make_float4(tree.axis[4 * j], tree.axis[4 * j + 1], tree.axis[4 * j + 2], 0.f)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
      if (in[h]) P[h] = place8(tree.placement + 8 * j);
      tsup[j] = in[h] ? tree.support[j] : 0ull;
      fpar[h] = j < nf ? tree.frame_parent[p.frames[j]] : 0;
      if (j < nf) F[h] = place8(tree.frame_placement + 8 * p.frames[j]);
      int perm;
      sgn[h] = turned_axis(jt[h], ax[h], perm);
      tperm[j] = perm;
      trank[j] = tchild[j] = 0;
      mv[h] = joint_nv(jt[h]) > 0;
    }
    __syncwarp();
    unsigned long long need = 0ull, framed = 0ull;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      if (j < nf) {
        need |= tsup[fpar[h]];
        framed |= 1ull << fpar[h];
      }
      if (in[h] && j > 0) ord = ord && par[h] >= 0 && ((tsup[j - 1] >> par[h]) & 1ull);
    }
    need = or64(need);
    framed = or64(framed);
    const unsigned long long moves = ballot64(mv[0], mv[1]);
    const bool ordered = __all_sync(kAll, ord);      // numbered depth first already
    bool nd[2];
    int rank[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      nd[h] = in[h] && ((need >> j) & 1ull);
      rank[h] = 0;
      if (nd[h]) {
        if (ordered) {
          rank[h] = __popcll(need & ((1ull << j) - 1ull));
        } else {
          for (int i = 0; i < nj; ++i)
            rank[h] += i != j && ((need >> i) & 1ull) && visited_before(tsup[i], tsup[j]);
        }
        trank[j] = rank[h];
        if (par[h] >= 0) atomicAdd(tchild + par[h], 1);
      }
    }
    __syncwarp();
    // several children, or frames and a child: the wrench waits in a slot
    bool st[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      st[h] = nd[h] && (tchild[j] >= 2 || (tchild[j] == 1 && ((framed >> j) & 1ull)));
    }
    const unsigned long long stored = ballot64(st[0], st[1]);
    int fr[2], fs[2] = {0, 0}, nfr[2] = {0, 0}, pos[2] = {0, 0};
    fr[0] = trank[fpar[0]];
    fr[1] = trank[fpar[1]];
    for (int g = 0; g < nf; ++g) {                   // frames of earlier visits, of this one; visit order
      const int rg = __shfl_sync(kAll, g < kWarp ? fr[0] : fr[1], g & (kWarp - 1));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        fs[h] += rg < rank[h];
        nfr[h] += rg == rank[h];
        pos[h] += rg < fr[h] || (rg == fr[h] && g < lane + kWarp * h);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      if (nd[h]) {
        const unsigned long long above = tsup[j] & ~(1ull << j);
        unsigned long long vs = 0ull;
        if (ordered && need == (nj < 64 ? (1ull << nj) - 1ull : ~0ull)) {
          vs = tsup[j];                              // visits are joints
        } else {
          for (unsigned long long m = tsup[j]; m; m &= m - 1ull) vs |= 1ull << trank[__ffsll((long long)m) - 1];
        }
        const int flags = (st[h] ? kLaneStored : 0) | (tchild[j] >= 2 ? kLaneBranch : 0) |
                          ((above & moves) == 0ull ? kLaneStop : 0) | (tchild[j] ? kLaneChain : 0) |
                          (sgn[h] != 0.f ? kLaneRevZ : 0) |
                          (par[h] >= 0 && trank[par[h]] == rank[h] - 1 ? 0 : kLaneJump);
        float* r = rec + 32 * rank[h];
        *reinterpret_cast<int4*>(r) = make_int4(jt[h] | (__popcll(above & stored) << 8) | (flags << 16), iq[h],
                                                par[h] >= 0 ? trank[par[h]] : -1, fs[h] | ((fs[h] + nfr[h]) << 16));
        const Pose Q = turned_from(turn_by(P[h], tperm[j]), par[h] >= 0 ? tperm[par[h]] : 0);
        store_pose8(r + kRecPlace, Q);
        r[kRecPlace + 3] = sgn[h];
        store_rows(r + kRecRows, Q);
        *reinterpret_cast<float4*>(r + kRecAxis) = ax[h];
        *reinterpret_cast<unsigned long long*>(r + kRecPath) = vs;
      }
      if (j < nf) {
        fid[pos[h]] = j;
        const Pose Q = turned_from(F[h], tperm[fpar[h]]);
        store_pose8(fplace + 20 * pos[h], Q);
        store_rows(fplace + 20 * pos[h] + 8, Q);
      }
    }
    // a bound given too small by the caller: no slot may lie outside the shared memory reserved
    bool over = false;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = lane + kWarp * h;
      over = over || (kGrad && st[h] && __popcll(tsup[j] & ~(1ull << j) & stored) >= L.nslots);
    }
    over = __any_sync(kAll, over);
    if (lane == 0) {
      s_need = need;
      s_moves = moves;
      s_over = over;
    }
  }
  __syncthreads();
  const unsigned long long need = s_need, moves = s_moves;
  const int nvis = __popcll(need);
  if (s_over) {                                      // refused: NaN results
    const float nan = __int_as_float(0x7fc00000);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.batch * nq; i += (int64_t)gridDim.x * blockDim.x) {
      p.grad_q[i] = nan;
      if (p.loss && i < p.batch) p.loss[i] = nan;
    }
    return;
  }

  float* w = smem + L.cta_floats + warp * L.warp_floats;
  float* wq = w + L.q;
  float* wc = w + L.cs;
  float* ring = w + L.ring;
  float* slots = w + L.slots + lane;
  float* saved = w + L.saved + lane;
  float* qrow = wq + lane * L.qpitch;
  float* crow = wc + lane * L.qpitch;
  const int nq1 = nq > 0 ? nq : 1;
  const int row0 = lane / nq1, col0 = lane - row0 * nq1, drow = kWarp / nq1, dcol = kWarp - drow * nq1;
  const int64_t ntiles = (p.batch + kWarp - 1) / kWarp;
  for (int64_t tile = (int64_t)blockIdx.x * wpc + warp; tile < ntiles; tile += (int64_t)gridDim.x * wpc) {
    const int64_t b0 = tile * kWarp;
    const int cnt = p.batch - b0 < kWarp ? (int)(p.batch - b0) : kWarp;
    const int last = cnt - 1;
    // ---- q slab and the first frames' targets ----
    if (lane >= cnt)                                // the last tile's idle lanes walk q = 0
      for (int e = 0; e < L.qpitch; ++e) qrow[e] = 0.f;
    const float* gq = p.q + b0 * nq;
    const int qn = cnt * nq;
    if (L.qpitch == nq) {                           // one contiguous slab
      const int n4 = aligned16(gq) ? qn >> 2 : 0;
      for (int e = lane; e < n4; e += kWarp) cp_async16(wq + 4 * e, gq + 4 * e);
      for (int e = 4 * n4 + lane; e < qn; e += kWarp) cp_async4(wq + e, gq + e);
    } else {                                        // padded rows: word e of the slab is row r, column c
      for (int e = lane, r = row0, c = col0; e < qn; e += kWarp) {
        cp_async4(wq + r * L.qpitch + c, gq + e);
        r += drow; c += dcol;
        if (c >= nq) { c -= nq; ++r; }
      }
    }
    int off[7];                                     // this lane's words of a frame's 32 targets
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      const int e = lane + kWarp * i, c = e / 7;
      off[i] = (c < last ? c : last) * nf * 7 + (e - 7 * c);
    }
    const float* gt = p.targets + b0 * nf * 7;
    auto fetch = [&](int fi) {
      if (fi < nf) {
        const int f = fid[fi];
        float* dst = ring + (fi & 1) * L.rstep + lane;
        const float* src = gt + 7 * f;
#pragma unroll
        for (int i = 0; i < 7; ++i) cp_async4(dst + kWarp * i, src + off[i]);
        if (per_cfg) cp_async4(dst + 7 * kWarp, p.weights + (b0 + (lane < last ? lane : last)) * nf + f);
      }
      cp_async_commit();
    };
    fetch(0);                                       // the group that also holds the q slab
    fetch(1);
    cp_async_wait_groups<1>();
    __syncwarp();
    if (kGrad) {                                    // joints that move no frame
      for (unsigned long long m = moves & ~need; m; m &= m - 1ull) {
        const int j = __ffsll((long long)m) - 1;
        const int iq = tree.idx_q[j], n = joint_nq(tree.jtype[j]);
        for (int e = 0; e < n; ++e) qrow[iq + e] = 0.f;
      }
    }
    // half-angle sine over q and cosine beside it for every joint walked about z: independent of one
    // another here, not on the dependent chain of the walk, and read again on the way up
    bool far = false;
#pragma unroll 4
    for (int k = 0; k < nvis; ++k) {
      const int4 m = meta_of(k);
      if ((m.x >> 16) & kLaneRevZ) {
        const float x = qrow[m.y];
        float sn, cs;
        sincos_half(x, sn, cs);
        far = far || fabsf(x) > kSincosHalfMax;
        qrow[m.y] = sn * rec[32 * k + kRecPlace + 3];
        crow[m.y] = cs;
      }
    }
    if (__any_sync(0xffffffffu, far)) {             // joint angles of thousands of turns
      for (int k = 0; k < nvis; ++k) {
        const int4 m = meta_of(k);
        if (!((m.x >> 16) & kLaneRevZ)) continue;   // (a fixed joint's idx_q may lie one past the row)
        const float x = gq[(lane < last ? lane : last) * nq + m.y];
        if (fabsf(x) > kSincosHalfMax) {
          float sn, cs;
          sincosf(0.5f * x, &sn, &cs);
          qrow[m.y] = sn * rec[32 * k + kRecPlace + 3];
          crow[m.y] = cs;
        }
      }
    }
    const float go = kGrad && p.grad_loss ? __ldg(p.grad_loss + b0 + (lane < last ? lane : last)) : 1.f;
    float loss = 0.f;
    Pose T;
    int saved_at = -1;
    int4 next = meta_of(0);
    for (int k = 0; k < nvis; ++k) {
      const int4 m = next;
      next = meta_of(k + 1);                        // (one record of padding after the last)
      const int flags = m.x >> 16;
      // ---- down: the world placement of visit k, from its parent's ----
      int i = k;
      if (flags & kLaneJump) {
        if (m.z >= 0 && m.z == saved_at) {          // the last branch joint passed
          T.t = f3(saved[0], saved[kWarp], saved[2 * kWarp]);
          T.q = make_float4(saved[3 * kWarp], saved[4 * kWarp], saved[5 * kWarp], saved[6 * kWarp]);
        } else {                                    // a root, or an outer branch joint: again from the root
          T.t = f3(0.f, 0.f, 0.f);
          T.q = make_float4(0.f, 0.f, 0.f, 1.f);
          i = 0;
        }
      }
#pragma unroll 1
      for (; i <= k; ++i) {
        const float* r = rec + 32 * i;
        if (i < k && !((*reinterpret_cast<const unsigned long long*>(rec + 32 * k + kRecPath) >> i) & 1ull)) continue;
        const int4 mi = i == k ? m : *reinterpret_cast<const int4*>(r);
        const float4 pt = *reinterpret_cast<const float4*>(r + kRecPlace);
        const float4 pq = *reinterpret_cast<const float4*>(r + kRecPlace + 4);
        if ((mi.x >> 16) & kLaneRevZ) {
          const float sn = qrow[mi.y], cs = crow[mi.y];
          T.t = add(T.t, qrot(T.q, f3(pt.x, pt.y, pt.z)));
          const float4 x = qmul(T.q, pq);
          T.q = make_float4(fmaf(x.x, cs, x.y * sn), fmaf(x.y, cs, -x.x * sn), fmaf(x.z, cs, x.w * sn),
                            fmaf(x.w, cs, -x.z * sn));
        } else {
          T = compose(T, local_transform(mi.x & 0xff, Pose{f3(pt.x, pt.y, pt.z), pq}, r + kRecAxis, qrow + mi.y));
        }
      }
      if (flags & kLaneBranch) {
        saved[0] = T.t.x; saved[kWarp] = T.t.y; saved[2 * kWarp] = T.t.z;
        saved[3 * kWarp] = T.q.x; saved[4 * kWarp] = T.q.y; saved[5 * kWarp] = T.q.z; saved[6 * kWarp] = T.q.w;
        saved_at = k;
      }
      // ---- the joint's frames: loss, and their wrenches in the joint's frame ----
      float3 Wf = f3(0.f, 0.f, 0.f), Wt = f3(0.f, 0.f, 0.f);
      const int f1 = m.w >> 16;
      for (int fi = m.w & 0xffff; fi < f1; ++fi) {
        cp_async_wait_groups<1>();                  // this frame's copies (all but the newest group)
        __syncwarp();
        const float* s = ring + (fi & 1) * L.rstep;
        const float* tp = s + 7 * lane;
        const Pose Tt{f3(tp[0], tp[1], tp[2]), make_float4(tp[3], tp[4], tp[5], tp[6])};
        const float wf = per_cfg ? s[7 * kWarp + lane] : __ldg(p.weights + fid[fi]);
        __syncwarp();                               // every lane has read the buffer refilled next
        fetch(fi + 2);
        const Pose Tf = compose(T, load_pose8(fplace + 20 * fi));
        // Tt^-1 * Tf
        const Pose D{qrot_inv(Tt.q, sub(Tf.t, Tt.t)), qmul(qconj(Tt.q), Tf.q)};
        float3 v, om;
        if (kGrad) {
          float3 gl, ga;
          se3_log_grad(D, v, om, gl, ga);
          const float s2 = 2.f * wf * go;
          float3 ff = scale(gl, s2), ft = scale(ga, s2);
          carry_wrench(fplace + 20 * fi + 8, ff, ft);
          Wf = add(Wf, ff);
          Wt = add(Wt, ft);
        } else {
          se3_log(D, v, om);
        }
        loss = fmaf(wf, dot(v, v) + dot(om, om), loss);
      }
      if (!kGrad) continue;
      auto slot_of = [&](int x) { return slots + ((x >> 8) & 0xff) * 6 * kWarp; };
      auto put = [&](float* s) {
        s[0] = Wf.x; s[kWarp] = Wf.y; s[2 * kWarp] = Wf.z;
        s[3 * kWarp] = Wt.x; s[4 * kWarp] = Wt.y; s[5 * kWarp] = Wt.z;
      };
      if (flags & kLaneChain) {                     // a child comes next: frames' wrench waits if there is one
        if (flags & kLaneStored) put(slot_of(m.x));
        continue;
      }
      // ---- up: from a leaf to the parent of the next visit ----
      const int up_to = k + 1 < nvis ? next.z : -1;
      int u = k;
      int4 mu = m;
      for (;;) {
        const int jt = mu.x & 0xff;
        const float* r = rec + 32 * u;
        float* gj = qrow + mu.y;
        const bool stop = (mu.x >> 16) & kLaneStop;
        if ((mu.x >> 16) & kLaneRevZ) {
          const float sn = gj[0], cs = crow[mu.y];
          gj[0] = r[kRecPlace + 3] * Wt.z;
          if (stop) break;                          // nothing above moves
          const float s1 = 2.f * sn * cs, c1 = fmaf(-2.f * sn, sn, 1.f);
          Wf = f3(fmaf(c1, Wf.x, -s1 * Wf.y), fmaf(s1, Wf.x, c1 * Wf.y), Wf.z);
          Wt = f3(fmaf(c1, Wt.x, -s1 * Wt.y), fmaf(s1, Wt.x, c1 * Wt.y), Wt.z);
          carry_wrench(r + kRecRows, Wf, Wt);
        } else {
          Pose Lu;
          if (!stop) Lu = local_transform(jt, load_pose8(r + kRecPlace), r + kRecAxis, gj);
          const float3 ax = f3(r[kRecAxis], r[kRecAxis + 1], r[kRecAxis + 2]);
          if (jt == BR_JOINT_REVOLUTE) {
            gj[0] = dot(Wt, ax);
          } else if (jt == BR_JOINT_PRISMATIC) {
            gj[0] = dot(Wf, ax);
          } else if (jt == BR_JOINT_TRANSLATION) {  // q is the body translation
            gj[0] = Wf.x; gj[1] = Wf.y; gj[2] = Wf.z;
          } else if (jt == BR_JOINT_REVOLUTE_UNBOUNDED) {
            unbounded_chain(dot(Wt, ax), gj);
          } else if (jt == BR_JOINT_PLANAR) {
            planar_chain(Wf.x, Wf.y, Wt.z, gj);
          } else if (jt == BR_JOINT_FREE_FLYER) {
            const float4 uq = quat_chain(Wt, gj + 3);
            const float3 gt3 = qrot(uq, Wf);        // translation: delta_lin = R^T dt
            gj[0] = gt3.x; gj[1] = gt3.y; gj[2] = gt3.z;
          } else if (jt == BR_JOINT_SPHERICAL) {
            quat_chain(Wt, gj);
          }
          if (stop) break;
          Wf = qrot(Lu.q, Wf);
          Wt = add(qrot(Lu.q, Wt), cross(Lu.t, Wf));
        }
        u = mu.z;
        mu = meta_of(u);
        if ((mu.x >> 16) & kLaneStored) {
          float* s = slot_of(mu.x);
          Wf = add(Wf, f3(s[0], s[kWarp], s[2 * kWarp]));
          Wt = add(Wt, f3(s[3 * kWarp], s[4 * kWarp], s[5 * kWarp]));
          if (u == up_to) {
            put(s);
            break;
          }
        }
      }
    }
    if (p.loss && lane < cnt) p.loss[b0 + lane] = loss;
    if (kGrad) {
      __syncwarp();
      float* gg = p.grad_q + b0 * nq;
      if (L.qpitch == nq) {
        const int n4 = aligned16(gg) ? qn >> 2 : 0;
        for (int e = lane; e < n4; e += kWarp)
          reinterpret_cast<float4*>(gg)[e] = reinterpret_cast<const float4*>(wq)[e];
        for (int e = 4 * n4 + lane; e < qn; e += kWarp) gg[e] = wq[e];
      } else {
        for (int e = lane, r = row0, c = col0; e < qn; e += kWarp) {
          gg[e] = wq[r * L.qpitch + c];
          r += drow; c += dcol;
          if (c >= nq) { c -= nq; ++r; }
        }
      }
    }
    cp_async_wait_groups<0>();                      // the (empty) last groups
    __syncwarp();                                   // the slab and the ring are free for the next tile
  }
}

// out[b, :] = unit[b, :] * s[b * ss]
template <bool kVec>
__global__ void __launch_bounds__(256) scale_rows_kernel(const float* __restrict__ unit, const float* __restrict__ s,
                                                         int64_t ss, int64_t rows, int nq, float* __restrict__ out) {
  const int64_t n = rows * nq;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int V = kVec ? 4 : 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i * V < n; i += stride) {
    const int64_t e = i * V;
    int64_t b = n <= 0xffffffffll ? (int64_t)((uint32_t)e / (uint32_t)nq) : e / nq;
    int c = (int)(e - b * nq);
    if (kVec && e + 4 <= n) {
      const float4 u = reinterpret_cast<const float4*>(unit)[i];
      float r[4] = {u.x, u.y, u.z, u.w};
      float sb = __ldg(s + b * ss);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (c == nq) { c = 0; sb = __ldg(s + ++b * ss); }
        r[k] *= sb;
        ++c;
      }
      reinterpret_cast<float4*>(out)[i] = make_float4(r[0], r[1], r[2], r[3]);
    } else {
      for (int64_t x = e; x < e + V && x < n; ++x) out[x] = unit[x] * __ldg(s + x / nq * ss);
    }
  }
}

// When the lane kernel is taken (else kLanesNo, and the warp-per-configuration kernel runs):
// * an SM must hold kLanesMinWarps of its warps (its shared memory grows with the frames and the tree);
// * the batch must fill it: one tile walks the whole tree serially (27 us for the humanoid at 12
//   frames, 13 us for the dual arm, 9 us for the 7-joint chain, up to ~30,000 configurations), while the
//   warp kernel's time starts at 7 us and grows with the batch (loss and gradient in one pass, humanoid:
//   12.6 us at 4,096, 21.6 at 8,192, 41 at 16,384; chain: 7.3 / 12 / 20 us at 1,300 / 4,096 / 8,192).
//   The lines cross near 200 (njoints + nf) configurations, for the loss alone too.
constexpr int kLanesMinWarps = 4, kLanesBatch = 200;
constexpr int kLanesNo = INT32_MIN;                 // neither a BR_E* code nor a cudaError_t
constexpr int kLanesStatic = 1536;                  // reserved for the lane kernel's static shared memory

template <bool kGrad>
static int launch_lanes(const br_tree_t& tree, const LossParams& p, cudaStream_t stream) {
  if (p.batch == 0) return BR_OK;
  if (p.batch < (int64_t)kLanesBatch * (tree.njoints + p.nf)) return kLanesNo;
  const LaneLayout L(tree.njoints, tree.nq, p.nf, kGrad, p.weights_per_config != 0, p.path_slots);
  const DeviceInfo& dev = device_info();
  const int64_t tiles = (p.batch + kWarp - 1) / kWarp;
  int best = 0, wpc = 0;
  for (int c = 8; c >= 1; --c) {                    // warps per CTA: the most resident warps (16 by registers)
    const int bytes = (L.cta_floats + c * L.warp_floats) * (int)sizeof(float);
    if (bytes + kLanesStatic > dev.max_smem_optin) continue;
    const int ctas = dev.smem_per_sm / (bytes + kLanesStatic + 1024);
    const int warps = ctas * c < 16 ? ctas * c : 16 / c * c;
    if (warps < kLanesMinWarps) continue;
    // few tiles: smaller CTAs, so that they spread over the SMs
    if (c > 1 && tiles < (int64_t)c * dev.sms) continue;
    if (warps > best) { best = warps; wpc = c; }
  }
  if (!wpc) return kLanesNo;
  const int bytes = (L.cta_floats + wpc * L.warp_floats) * (int)sizeof(float);
  auto kern = pose_loss_lanes_kernel<kGrad>;
  static int configured[16] = {0};
  if (bytes > configured[dev.device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    configured[dev.device & 15] = bytes;
  }
  const int64_t need = (tiles + wpc - 1) / wpc, cap = (int64_t)(best / wpc) * dev.sms;
  kern<<<(int)(need < cap ? need : cap), wpc * kWarp, bytes, stream>>>(tree, p);
  return (int)cudaGetLastError();
}

template <bool kBackward>
static int launch_loss(const br_tree_t& tree, const LossParams& p, int wpc, cudaStream_t stream) {
  if (p.batch == 0) return BR_OK;
  const LossLayout L(tree.njoints, tree.nq, tree.nv, p.nf);
  const DeviceInfo& dev = device_info();
  size_t bytes = (size_t)(L.cta_floats + wpc * L.warp_floats) * sizeof(float);
  while ((int)bytes > dev.max_smem_optin && wpc > 1) {
    wpc >>= 1;
    bytes = (size_t)(L.cta_floats + wpc * L.warp_floats) * sizeof(float);
  }
  auto kern = pose_loss_kernel<kBackward>;
  static int configured[16] = {0};
  if ((int)bytes > configured[dev.device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    configured[dev.device & 15] = (int)bytes;
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, wpc * kWarp, bytes);
  if (per_sm < 1) per_sm = 1;
  const int64_t need = (p.batch + wpc - 1) / wpc;
  const int64_t cap = (int64_t)per_sm * dev.sms;
  kern<<<(int)(need < cap ? need : cap), wpc * kWarp, bytes, stream>>>(tree, p);
  return (int)cudaGetLastError();
}

static int fill_loss(const br_tree_t* tree, LossParams& p, const int32_t* frame_ids, int32_t n_frames) {
  int st = validate_tree(tree);
  if (st) return st;
  if (n_frames < 1 || !frame_ids) return BR_EINVAL;
  if (n_frames > BR_MAX_TARGETS) return BR_ETOOBIG;
  for (int i = 0; i < n_frames; ++i) {
    if (frame_ids[i] < 0 || frame_ids[i] >= tree->nframes) return BR_EINVAL;
    p.frames[i] = frame_ids[i];
  }
  p.nf = n_frames;
  return BR_OK;
}

}  // namespace br

using namespace br;

// Joint kinds whose raw-q chain rule the backward implements: every kind of the tree table.
static bool adjoint_kinds_ok(const br_tree_t* t) {
  const int ok = (1 << (BR_JOINT_TRANSLATION + 1)) - 1;
  return t && t->kinds != 0 && (t->kinds & ~ok) == 0;
}

// Arguments of every entry point below (loss / gradient pointers are checked by each).
static int loss_args(const br_tree_t* tree, LossParams& p, const float* q, int64_t batch, const int32_t* frame_ids,
                     int32_t n_frames, const float* targets, const float* weights, int32_t weights_per_config) {
  const int st = fill_loss(tree, p, frame_ids, n_frames);
  if (st) return st;
  if (!adjoint_kinds_ok(tree)) return BR_EINVAL;
  if (batch < 0 || (batch > 0 && (!q || !targets || !weights))) return BR_EINVAL;
  p.q = q; p.targets = targets; p.weights = weights;
  p.batch = batch; p.weights_per_config = weights_per_config != 0;
  p.path_slots = -1;
  return BR_OK;
}

extern "C" int br_pose_loss(const br_tree_t* tree, const float* q, int64_t batch, const int32_t* frame_ids,
                            int32_t n_frames, const float* targets, const float* weights,
                            int32_t weights_per_config, float* loss, float* joint_pose_world, void* stream) {
  LossParams p = {};
  int st = loss_args(tree, p, q, batch, frame_ids, n_frames, targets, weights, weights_per_config);
  if (st) return st;
  if (batch > 0 && !loss) return BR_EINVAL;
  p.loss = loss; p.oMi_out = joint_pose_world;
  if (!joint_pose_world) {
    st = launch_lanes<false>(*tree, p, (cudaStream_t)stream);
    if (st != kLanesNo) return st;
  }
  return launch_loss<false>(*tree, p, 8, (cudaStream_t)stream);
}

extern "C" int br_pose_loss_backward(const br_tree_t* tree, const float* q, const float* joint_pose_world,
                                     int64_t batch, const int32_t* frame_ids, int32_t n_frames,
                                     const float* targets, const float* weights, int32_t weights_per_config,
                                     const float* grad_loss, float* grad_q, void* stream) {
  LossParams p = {};
  int st = loss_args(tree, p, q, batch, frame_ids, n_frames, targets, weights, weights_per_config);
  if (st) return st;
  if (batch > 0 && (!grad_loss || !grad_q)) return BR_EINVAL;
  p.oMi_in = joint_pose_world; p.grad_loss = grad_loss; p.grad_q = grad_q;
  if (!joint_pose_world) {
    st = launch_lanes<true>(*tree, p, (cudaStream_t)stream);
    if (st != kLanesNo) return st;
  }
  return launch_loss<true>(*tree, p, 8, (cudaStream_t)stream);
}

extern "C" int br_pose_loss_value_grad(const br_tree_t* tree, const float* q, int64_t batch,
                                       const int32_t* frame_ids, int32_t n_frames, const float* targets,
                                       const float* weights, int32_t weights_per_config, int32_t path_slots,
                                       float* loss, float* unit_grad, void* stream) {
  LossParams p = {};
  int st = loss_args(tree, p, q, batch, frame_ids, n_frames, targets, weights, weights_per_config);
  if (st) return st;
  if (batch > 0 && (!loss || !unit_grad)) return BR_EINVAL;
  p.loss = loss; p.grad_q = unit_grad; p.path_slots = path_slots;
  st = launch_lanes<true>(*tree, p, (cudaStream_t)stream);
  return st != kLanesNo ? st : launch_loss<true>(*tree, p, 8, (cudaStream_t)stream);
}

extern "C" int br_scale_rows(const float* rows, const float* scale, int64_t scale_stride, int64_t n, int32_t width,
                             float* out, void* stream) {
  if (n < 0 || width < 0) return BR_EINVAL;
  if (n == 0 || width == 0) return BR_OK;
  if (!rows || !scale || !out) return BR_EINVAL;
  if (!aligned4(rows) || !aligned4(scale) || !aligned4(out)) return BR_EALIGN;
  const bool vec = aligned16(rows) && aligned16(out);
  const int64_t threads = vec ? (n * width + 3) / 4 : n * width;
  int64_t blocks = (threads + 255) / 256;
  const int64_t cap = (int64_t)device_info().sms * 8;
  if (blocks > cap) blocks = cap;
  if (vec) scale_rows_kernel<true><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(rows, scale, scale_stride, n, width, out);
  else scale_rows_kernel<false><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(rows, scale, scale_stride, n, width, out);
  return (int)cudaGetLastError();
}
