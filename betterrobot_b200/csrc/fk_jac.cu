// fk_jac.cu — fused forward kinematics + frame Jacobians for sm_100a.
//
// Work mapping of fk_jac_kernel: one warp owns one configuration at a time (persistent grid,
// warps stride over the batch); fk_group_kernel below shares a warp between the configurations of
// a small tree.  Inside the warp:
//   * lanes load q coalesced into shared memory;
//   * lane j builds liMi_j = placement_j * T_j(q_j) for its joint(s)
//     (forward.py:110-123 evaluates the same product joint by joint);
//   * world placements oMi come from pointer jumping over the parent table:
//     T_j <- T_anc(j) * T_j, anc(j) <- anc(anc(j)), ceil(log2 depth) rounds, so a
//     tree of depth d costs log2(d) composes per lane instead of a serial walk
//     (forward.py:125-129);
//   * target (frame) placements oMf = oMi[parent] * placement (forward.py:213-216);
//   * Jacobian columns are generated directly from the column's world axis a and
//     origin o (rotation: [a x (p_f - o); a] in LOCAL_WORLD_ALIGNED, [o x a; a] in
//     WORLD; translation: [a; 0]), zero outside the target's support — the
//     O(nj * 6 * nv) per-joint parent copies of jacobian.py:45-79 never happen;
//   * every output block of the configuration (J: n_targets*6*nv floats,
//     poses: n*7 floats) is assembled in shared memory and written with one
//     cp.async.bulk store (TMA bulk copy, full 128-B lines), so HBM sees only
//     the algorithmic bytes.  A J block above 16 KB (all 32 joints of a humanoid:
//     27.6 KB) goes out in pieces of a few targets through two alternating
//     buffers, so that its size does not cap the warps per SM;
//   * in from-poses mode (compute_joint_jacobians) the next configuration's
//     placements are loaded into registers while the current one is written.
#include <cuda_runtime.h>
#include <stdint.h>

#include "br_common.cuh"
#include "br_lie.cuh"
#include "br_fk.cuh"

namespace br {

enum : uint32_t { OUT_OMI = 1u, OUT_LIMI = 2u, OUT_TPOSE = 4u, OUT_JAC = 8u };

struct FkParams {
  const float* q;        // [B, nq]           (from-q mode)
  const float* oMi_in;   // [B, nj, 7]        (from-poses mode)
  int64_t batch;
  float* oMi;            // [B, nj, 7]        or null
  float* liMi;           // [B, nj, 7]        or null
  float* tpose;          // [B, nt, 7]        or null
  float* jac;            // [B, nt, 6, nv]    or null
  int32_t nt;
  uint32_t outputs;      // OUT_* bits
  uint32_t bulk;         // OUT_* bits whose blocks are 16-byte aligned -> TMA bulk store
  int32_t chunk;         // targets per staged piece of the J block (>= nt: the whole block)
  int32_t targets[BR_MAX_TARGETS];
};

// Shared-memory layout (in floats; every region starts on a 16-byte boundary).
struct Layout {
  // CTA-wide tables
  int parent, jtype, idxq, axis, place, cjoint, caxis, tparent, tplace, support, pairoff, pairs;
  int cta_floats;
  // per-warp regions
  int q, poseT, poseQ, anc, colA, tgt, sJ, sT, sOMi, sLiMi;
  int warp_floats;
  // chunk: targets per staged piece of a configuration's J block.  chunk >= nt stages the
  // whole block in one buffer; a smaller (even) chunk stages it piece by piece in two
  // alternating buffers, so a large block (all joints of a humanoid: 27.6 KB) does not
  // limit the warps per SM.
  // per: configurations of a warp; group: the kernel that passes placements by shuffles.
  __host__ __device__ Layout(int nj, int nq, int nv, int nt, uint32_t outputs, int chunk, int per = 1, bool group = false) {
    int o = 0;
    parent = o; o += round4(nj);
    jtype = o; o += round4(nj);
    idxq = o; o += round4(nj);
    axis = o; o += 4 * nj;
    place = o; o += 8 * nj;
    cjoint = o; o += round4(nv);
    caxis = o; o += 4 * nv;                                      // column axis in the joint frame, and its kind
    tparent = o; o += round4(nt);
    tplace = o; o += 8 * nt;
    support = o; o += round4(2 * nj);                            // uint64 per joint: the joints above it, and itself
    pairoff = o; o += round4(nt);
    pairs = o; o += (outputs & OUT_JAC) ? round4(nt * nv) : 0;   // (target << 16 | joint << 8 | column) with support
    cta_floats = o;
    o = 0;
    const bool jac = (outputs & OUT_JAC) != 0;
    q = o; o += round4(per * nq);
    poseT = o; o += group && !jac ? 0 : per * 4 * nj;            // world translation (x, y, z, 0)
    poseQ = o; o += group ? 0 : 4 * nj;                          // world quaternion
    anc = o; o += group ? 0 : round4(nj);
    colA = o; o += group && !jac ? 0 : per * 4 * nv;             // world column axis, and its kind
    tgt = o; o += group && !jac ? 0 : per * 8 * nt;
    sJ = o; o += jac ? (chunk < nt ? 2 * round4(chunk * 6 * nv) : round4(per * nt * 6 * nv)) : 0;
    sT = o; o += (outputs & OUT_TPOSE) ? round4(per * nt * 7) : 0;
    sOMi = o; o += (outputs & OUT_OMI) ? round4(per * nj * 7) : 0;
    sLiMi = o; o += (outputs & OUT_LIMI) ? round4(per * nj * 7) : 0;
    warp_floats = o;
  }
};

// Four consecutive floats of a table whose alignment is not known beyond a float's.
__device__ __forceinline__ float4 load4(const float* p) { return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3)); }

// The CTA's tables, and the number of (target, column) pairs with support.  Every CTA of a wave pays for them before
// its first configuration, so nothing here waits more than once for memory: all table loads go out together
// and each warp makes the pair list's offsets for itself.  (Masks from memory one target at a time and a
// serial prefix took 5.4 us of every call's time on the humanoid, this 1.5, 3 with Jacobians.)
__device__ __forceinline__ int build_tables(const br_tree_t& tree, const FkParams& p, float* cta, const Layout& L,
                                            bool want_jac) {
  const int nj = tree.njoints, nv = tree.nv, nt = p.nt;
  int* s_parent = reinterpret_cast<int*>(cta + L.parent);
  int* s_jtype = reinterpret_cast<int*>(cta + L.jtype);
  int* s_idxq = reinterpret_cast<int*>(cta + L.idxq);
  float* s_axis = cta + L.axis;
  float* s_place = cta + L.place;
  int* s_cjoint = reinterpret_cast<int*>(cta + L.cjoint);
  float* s_caxis = cta + L.caxis;
  int* s_tparent = reinterpret_cast<int*>(cta + L.tparent);
  float* s_tplace = cta + L.tplace;
  unsigned long long* s_support = reinterpret_cast<unsigned long long*>(cta + L.support);
  int* s_pairoff = reinterpret_cast<int*>(cta + L.pairoff);
  int* s_pairs = reinterpret_cast<int*>(cta + L.pairs);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpc = blockDim.x >> 5;
  static_assert(BR_MAX_JOINTS <= 64 && BR_MAX_NV <= 64 && BR_MAX_TARGETS <= 64, "one slot of 64 per table");
  for (int u = threadIdx.x; u < 192; u += blockDim.x) {
    const int i = u & 63;
    if (u < 64) {
      if (i >= nj) continue;
      const float4 ax = load4(tree.axis + 4 * i), pa = load4(tree.placement + 8 * i), pb = load4(tree.placement + 8 * i + 4);
      s_parent[i] = tree.parent[i];
      s_support[i] = tree.support[i];
      s_jtype[i] = tree.jtype[i];
      s_idxq[i] = tree.idx_q[i];
      *reinterpret_cast<float4*>(s_axis + 4 * i) = ax;
      *reinterpret_cast<float4*>(s_place + 8 * i) = pa;
      *reinterpret_cast<float4*>(s_place + 8 * i + 4) = pb;
    } else if (u < 128) {
      if (i >= nv) continue;
      float4 ax = load4(tree.col_axis + 4 * i);
      ax.w = tree.col_kind[i] == 0 ? 0.f : 1.f;
      s_cjoint[i] = tree.col_joint[i];
      *reinterpret_cast<float4*>(s_caxis + 4 * i) = ax;
    } else {
      if (i >= nt) continue;
      const int id = p.targets[i];
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = make_float4(0.f, 0.f, 0.f, 1.f);  // a joint: identity
      int par = -id - 1;
      if (id >= 0) {
        par = tree.frame_parent[id];
        a = load4(tree.frame_placement + 8 * id);
        b = load4(tree.frame_placement + 8 * id + 4);
      }
      s_tparent[i] = par;
      *reinterpret_cast<float4*>(s_tplace + 8 * i) = a;
      *reinterpret_cast<float4*>(s_tplace + 8 * i + 4) = b;
    }
  }
  __syncthreads();
  // Columns with a non-zero Jacobian entry for each target: col_joint[c] supports the
  // target's parent joint.  The list of such (target, column) pairs is the only part of
  // the J block that depends on q; the rest is zero and is written once above.
  int npairs = 0;
  if (want_jac) {
    unsigned long long mask[2] = {0ull, 0ull};  // of targets lane and lane + 32
    int first[2] = {0, 0};                      // their pairs' places in the list
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (kWarp * k >= nt) break;
      const int t = lane + kWarp * k;
      const unsigned long long sup = t < nt ? s_support[s_tparent[t]] : 0ull;
      const uint32_t sup0 = (uint32_t)sup, sup1 = (uint32_t)(sup >> 32);
      uint32_t half[2] = {0u, 0u};  // columns 0 to 31, 32 to 63
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c1 = nv - kWarp * h < kWarp ? nv - kWarp * h : kWarp;
#pragma unroll 4
        for (int c = 0; c < c1; ++c) {
          const int j = s_cjoint[kWarp * h + c];
          half[h] |= (((j < 32 ? sup0 : sup1) >> (j & 31)) & 1u) << c;
        }
      }
      mask[k] = half[0] | (unsigned long long)half[1] << 32;
      const int n = __popcll(mask[k]);
      int upto = n;
#pragma unroll
      for (int d = 1; d < kWarp; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += v;
      }
      first[k] = npairs + upto - n;
      npairs += __shfl_sync(0xffffffffu, upto, kWarp - 1);
      if (warp == 0 && t < nt) s_pairoff[t] = first[k];
    }
    for (int t = warp; t < nt; t += wpc) {
      const unsigned long long m = __shfl_sync(0xffffffffu, t < kWarp ? mask[0] : mask[1], t & 31);
      const int f = __shfl_sync(0xffffffffu, t < kWarp ? first[0] : first[1], t & 31);
      for (int c = lane; c < nv; c += kWarp)
        if ((m >> c) & 1ull) s_pairs[f + __popcll(m & ((1ull << c) - 1ull))] = (t << 16) | (s_cjoint[c] << 8) | c;
    }
  }
  __syncthreads();
  return npairs;
}

// The six entries of J column c (of joint j) for target t, rows nv floats apart from dst: from the columns' world
// axes and kinds (wcA), the joints' origins (wpT) and the targets' records (wtgt: translation, quaternion).
template <int kRef>
__device__ __forceinline__ void jac_column(const float* wcA, const float* wpT, const float* wtgt, int t, int j, int c,
                                           float* dst, int nv) {
  const float4 a4 = *reinterpret_cast<const float4*>(wcA + 4 * c);
  const float3 a = f3(a4.x, a4.y, a4.z);
  float3 lin, ang;
  if (a4.w == 0.f) {
    const float4 o4 = *reinterpret_cast<const float4*>(wpT + 4 * j);
    const float3 o = f3(o4.x, o4.y, o4.z);
    if (kRef == BR_REF_WORLD) {
      lin = cross(o, a);                                   // hat(p_j) R S_ang  (jacobian.py:290-296)
    } else {
      const float4 pt = *reinterpret_cast<const float4*>(wtgt + 8 * t);
      lin = cross(a, sub(f3(pt.x, pt.y, pt.z), o));        // J_lin - hat(p_f) J_ang (jacobian.py:213-215)
    }
    ang = a;
  } else {
    lin = a;
    ang = f3(0.f, 0.f, 0.f);
  }
  if (kRef == BR_REF_LOCAL) {                              // R_f^T rows (jacobian.py:219-225)
    const float4 qt = *reinterpret_cast<const float4*>(wtgt + 8 * t + 4);
    lin = qrot_inv(qt, lin);
    ang = qrot_inv(qt, ang);
  }
  dst[0] = lin.x; dst[nv] = lin.y; dst[2 * nv] = lin.z;
  dst[3 * nv] = ang.x; dst[4 * nv] = ang.y; dst[5 * nv] = ang.z;
}

// a * b as compose, with the product that is rounded on its own in each quaternion component written out: left to
// the compiler it follows the surrounding code, and the kernels of this file would differ in the last bit of a
// placement (an IK problem whose target is such a placement can then take another number of iterations).
__device__ __forceinline__ Pose compose_rn(const Pose& a, const Pose& b) {
  const float4 p = a.q, q = b.q;
  Pose c;
  c.t = add(a.t, qrot(p, b.t));
  c.q.x = fmaf(-p.z, q.y, fmaf(p.y, q.z, fmaf(p.w, q.x, __fmul_rn(p.x, q.w))));
  c.q.y = fmaf(p.z, q.x, fmaf(p.y, q.w, fmaf(p.w, q.y, -__fmul_rn(p.x, q.z))));
  c.q.z = fmaf(p.z, q.w, fmaf(-p.y, q.x, fmaf(p.x, q.y, __fmul_rn(p.w, q.z))));
  c.q.w = fmaf(-p.z, q.z, fmaf(-p.y, q.y, fmaf(p.w, q.w, -__fmul_rn(p.x, q.x))));
  return c;
}

template <int kRef, bool kFromQ>
__global__ void fk_jac_kernel(const br_tree_t tree, const FkParams p) {
  extern __shared__ __align__(16) float smem[];
  const int nj = tree.njoints, nq = tree.nq, nv = tree.nv, nt = p.nt;
  const bool want_jac = (p.outputs & OUT_JAC) != 0;
  const Layout L(nj, nq, nv, nt, p.outputs, p.chunk);
  const bool chunked = want_jac && p.chunk < nt;
  float* cta = smem;
  int* s_parent = reinterpret_cast<int*>(cta + L.parent);
  int* s_jtype = reinterpret_cast<int*>(cta + L.jtype);
  int* s_idxq = reinterpret_cast<int*>(cta + L.idxq);
  float* s_axis = cta + L.axis;
  float* s_place = cta + L.place;
  int* s_cjoint = reinterpret_cast<int*>(cta + L.cjoint);
  float* s_caxis = cta + L.caxis;
  int* s_tparent = reinterpret_cast<int*>(cta + L.tparent);
  float* s_tplace = cta + L.tplace;
  int* s_pairoff = reinterpret_cast<int*>(cta + L.pairoff);
  int* s_pairs = reinterpret_cast<int*>(cta + L.pairs);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpc = blockDim.x >> 5;

  float* w = smem + L.cta_floats + warp * L.warp_floats;
  float* wq = w + L.q;
  float* wpT = w + L.poseT;
  float* wpQ = w + L.poseQ;
  int* wanc = reinterpret_cast<int*>(w + L.anc);
  float* wcA = w + L.colA;
  float* wtgt = w + L.tgt;
  float* sJ = w + L.sJ;
  float* sT = w + L.sT;
  float* sOMi = w + L.sOMi;
  float* sLiMi = w + L.sLiMi;
  const int cfl = chunked ? round4(p.chunk * 6 * nv) : 0;  // floats per chunk buffer
  if (want_jac && !chunked) {  // the chunked staging buffers are cleared before each piece
    const int n = round4(nt * 6 * nv) / 4;
    for (int i = lane; i < n; i += kWarp) reinterpret_cast<float4*>(sJ)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int64_t stride = (int64_t)gridDim.x * wpc;

  // q of the warp's next configuration is loaded into registers one iteration
  // ahead, so its global-load latency overlaps the current configuration's work
  // (nq <= BR_MAX_NQ = 128: at most 4 values per lane)
  float qn[4];
  const int64_t b0 = (int64_t)blockIdx.x * wpc + warp;
  if (kFromQ && b0 < p.batch) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane + kWarp * k;
      qn[k] = i < nq ? __ldg(p.q + b0 * nq + i) : 0.f;
    }
  }
  // likewise the next configuration's joint placements in from-poses mode
  // (nj * 7 <= BR_MAX_JOINTS * 7 = 448 floats: at most 14 values per lane)
  constexpr int kPoseRegs = (BR_MAX_JOINTS * 7 + kWarp - 1) / kWarp;
  float on[kPoseRegs];
  if (!kFromQ && b0 < p.batch) {
#pragma unroll
    for (int k = 0; k < kPoseRegs; ++k) {
      const int i = lane + kWarp * k;
      on[k] = i < nj * 7 ? __ldg(p.oMi_in + b0 * nj * 7 + i) : 0.f;
    }
  }

  const int npairs = build_tables(tree, p, cta, L, want_jac);
  const int rounds = tree.rounds;
  uint32_t gc = 0;  // staged J pieces so far: piece gc uses buffer gc & 1
  for (int64_t b = b0; b < p.batch; b += stride) {
    // ---- world joint placements --------------------------------------
    if (kFromQ) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = lane + kWarp * k;
        if (i < nq) wq[i] = qn[k];
      }
      const int64_t bn = b + stride;
      if (bn < p.batch) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = lane + kWarp * k;
          qn[k] = i < nq ? __ldg(p.q + bn * nq + i) : 0.f;
        }
      }
      __syncwarp();
      Pose T[2];
      int anc[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int j = lane + kWarp * k;
        if (j < nj) {
          T[k] = local_transform(s_jtype[j], load_pose8(s_place + 8 * j), s_axis + 4 * j, wq + s_idxq[j]);
          anc[k] = s_parent[j];
        }
      }
      if (lane == 0) bulk_wait_read_all();  // staging buffers are free again
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int j = lane + kWarp * k;
        if (j < nj) {
          store_split(wpT, wpQ, j, T[k]);
          wanc[j] = anc[k];
          if (p.outputs & OUT_LIMI) store_pose7(sLiMi + 7 * j, T[k]);
        }
      }
      __syncwarp();
      for (int r = 0; r < rounds; ++r) {
        Pose A[2];
        int aa[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int j = lane + kWarp * k;
          if (j < nj && anc[k] >= 0) {
            A[k] = load_split(wpT, wpQ, anc[k]);
            aa[k] = wanc[anc[k]];
          }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int j = lane + kWarp * k;
          if (j < nj && anc[k] >= 0) {
            T[k] = compose_rn(A[k], T[k]);
            anc[k] = aa[k];
            store_split(wpT, wpQ, j, T[k]);
            wanc[j] = anc[k];
          }
        }
        __syncwarp();
      }
      if (p.outputs & OUT_OMI) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int j = lane + kWarp * k;
          if (j < nj) store_pose7(sOMi + 7 * j, T[k]);
        }
      }
    } else {
      if (!chunked && lane == 0) bulk_wait_read_all();  // the whole-block buffer is free again
#pragma unroll
      for (int k = 0; k < kPoseRegs; ++k) {
        const int i = lane + kWarp * k;
        if (i < nj * 7) {
          const int j = i / 7, c = i - 7 * j;
          if (c < 3) wpT[4 * j + c] = on[k];
          else wpQ[4 * j + c - 3] = on[k];
        }
      }
      const int64_t bn = b + stride;
      if (bn < p.batch) {
#pragma unroll
        for (int k = 0; k < kPoseRegs; ++k) {
          const int i = lane + kWarp * k;
          on[k] = i < nj * 7 ? __ldg(p.oMi_in + bn * nj * 7 + i) : 0.f;
        }
      }
      __syncwarp();
    }

    // ---- target placements and world Jacobian columns --------------------
    for (int s = lane; s < nt; s += kWarp) {
      const Pose Tt = compose_rn(load_split(wpT, wpQ, s_tparent[s]), load_pose8(s_tplace + 8 * s));
      store_pose8(wtgt + 8 * s, Tt);
      if (p.outputs & OUT_TPOSE) store_pose7(sT + 7 * s, Tt);
    }
    if (want_jac) {
      for (int c = lane; c < nv; c += kWarp) {
        const float4 ax = *reinterpret_cast<const float4*>(s_caxis + 4 * c);
        const float3 a = qrot(*reinterpret_cast<const float4*>(wpQ + 4 * s_cjoint[c]), f3(ax.x, ax.y, ax.z));
        *reinterpret_cast<float4*>(wcA + 4 * c) = make_float4(a.x, a.y, a.z, ax.w);
      }
    }
    __syncwarp();

    auto jac_pair = [&](int s, int j, int c, float* dst) {
      jac_column<kRef>(wcA, wpT, wtgt, s, j, c, dst, nv);
    };
    if (want_jac && !chunked) {
      for (int idx = lane; idx < npairs; idx += kWarp) {
        const int pr = s_pairs[idx];
        const int s = pr >> 16, j = (pr >> 8) & 255, c = pr & 255;
        jac_pair(s, j, c, sJ + s * 6 * nv + c);
      }
    }
    if (chunked) {
      // targets [t0, t1) at a time: clear a buffer, fill the piece's (target, column) pairs,
      // store it; the other buffer's store is still reading while this one is filled
      const bool bulkJ = (p.bulk & OUT_JAC) != 0;
      float* gJ = p.jac + b * (int64_t)nt * 6 * nv;
      for (int t0 = 0; t0 < nt; t0 += p.chunk) {
        const int t1 = t0 + p.chunk < nt ? t0 + p.chunk : nt;
        float* buf = sJ + (int)(gc & 1u) * cfl;
        ++gc;
        if (bulkJ && lane == 0) bulk_wait_read<1>();         // the store two pieces back has read buf
        __syncwarp();
        for (int i = lane; i < cfl / 4; i += kWarp) reinterpret_cast<float4*>(buf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        const int e1 = t1 < nt ? s_pairoff[t1] : npairs;
        for (int idx = s_pairoff[t0] + lane; idx < e1; idx += kWarp) {
          const int pr = s_pairs[idx];
          const int s = pr >> 16, j = (pr >> 8) & 255, c = pr & 255;
          jac_pair(s, j, c, buf + (s - t0) * 6 * nv + c);
        }
        const int n = (t1 - t0) * 6 * nv;
        if (bulkJ) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_store(gJ + (int64_t)t0 * 6 * nv, buf, (uint32_t)n * 4u);
            bulk_commit();
          }
        } else {
          __syncwarp();
          warp_copy(gJ + (int64_t)t0 * 6 * nv, buf, n, lane);
        }
        __syncwarp();
      }
    }

    // ---- write the configuration's output blocks -----------------------
    fence_proxy_async_smem();
    __syncwarp();
    struct Out { uint32_t bit; float* g; const float* s; int n; };
    const Out outs[4] = {
        {OUT_JAC, p.jac ? p.jac + b * (int64_t)nt * 6 * nv : nullptr, sJ, nt * 6 * nv},
        {OUT_TPOSE, p.tpose ? p.tpose + b * (int64_t)nt * 7 : nullptr, sT, nt * 7},
        {OUT_OMI, p.oMi ? p.oMi + b * (int64_t)nj * 7 : nullptr, sOMi, nj * 7},
        {OUT_LIMI, p.liMi ? p.liMi + b * (int64_t)nj * 7 : nullptr, sLiMi, nj * 7}};
    bool issued = false;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      if (!(p.outputs & outs[o].bit) || outs[o].n == 0 || (chunked && outs[o].bit == OUT_JAC)) continue;
      if (p.bulk & outs[o].bit) {
        if (lane == 0) bulk_store(outs[o].g, outs[o].s, (uint32_t)outs[o].n * 4u);
        issued = true;
      } else {
        warp_copy(outs[o].g, outs[o].s, outs[o].n, lane);
      }
    }
    if (issued && lane == 0) bulk_commit();
    __syncwarp();
  }
  if (lane == 0) bulk_wait_read_all();  // the staging buffers outlive their stores
}

// ---------------------------------------------------------------------------
// Trees of at most 32 joints, from q: kG lanes (a power of two, at least the joints) per configuration and
// 32 / kG consecutive configurations per warp.
//
// Lane j of a configuration keeps joint j: its tables and placements stay in registers, its ancestor in every
// jumping round is known beforehand, and placements pass between lanes by shuffles, so only the outputs (and what
// a Jacobian column is made from) go through shared memory; the blocks of a warp's configurations are one
// contiguous store.  Bound by the schedulers (the work per joint), hence the lanes per configuration and, without
// Jacobians, the register limit.  Forward kinematics with all frames, against a warp per configuration
// and staged records (B = 65,536): 7-DOF arm 79 -> 35 us, dual arm 78 -> 33, humanoid 86 -> 64 (B = 16,384 24 -> 19); one
// frame's Jacobian of the arm 79 -> 36.
template <int kRef, int kG, bool kJac>
__global__ void __launch_bounds__(256, kJac ? 2 : 3) fk_group_kernel(const br_tree_t tree, const FkParams p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int kPer = kWarp / kG;
  constexpr int kQRegs = kG == kWarp ? BR_MAX_NQ / kWarp : 7;  // nq <= 7 * kG otherwise
  const int nj = tree.njoints, nq = tree.nq, nv = tree.nv, nt = p.nt;
  const Layout L(nj, nq, nv, nt, p.outputs, nt, kPer, true);
  const int lane = threadIdx.x & 31;
  const int wpc = blockDim.x >> 5;
  const int own = lane & (kG - 1), base = lane - own, sub_ = lane / kG;  // this lane in its configuration, and which
  float* w = smem + L.cta_floats + (threadIdx.x >> 5) * L.warp_floats;
  float* wq = w + L.q;
  float* wpT = w + L.poseT + sub_ * 4 * nj;
  float* wcA = w + L.colA + sub_ * 4 * nv;
  float* wtgt = w + L.tgt + sub_ * 8 * nt;
  float* sJ = w + L.sJ;
  float* sT = w + L.sT;
  float* sOMi = w + L.sOMi;
  float* sLiMi = w + L.sLiMi;
  if (kJac) {  // only the entries of the pair list are written again
    const int n = round4(kPer * nt * 6 * nv) / 4;
    for (int i = lane; i < n; i += kWarp) reinterpret_cast<float4*>(sJ)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int64_t groups = (p.batch + kPer - 1) / kPer;
  const int64_t stride = (int64_t)gridDim.x * wpc;
  int64_t g = (int64_t)blockIdx.x * wpc + (threadIdx.x >> 5);
  float qn[kQRegs];
  auto fetch = [&](int64_t gr) {  // the group's rows of q
    const int64_t b = gr * kPer;
    const int n = (p.batch - b < kPer ? (int)(p.batch - b) : kPer) * nq;
#pragma unroll
    for (int k = 0; k < kQRegs; ++k) {
      const int i = lane + kWarp * k;
      qn[k] = i < n ? __ldg(p.q + b * nq + i) : 0.f;
    }
  };
  if (g < groups) fetch(g);
  const int npairs = build_tables(tree, p, smem, L, kJac);
  const int* s_pairs = reinterpret_cast<const int*>(smem + L.pairs);
  const int* s_tparent = reinterpret_cast<const int*>(smem + L.tparent);
  const int* s_cjoint = reinterpret_cast<const int*>(smem + L.cjoint);
  const float* s_caxis = smem + L.caxis;
  const float* s_tplace = smem + L.tplace;

  const int j = own < nj ? own : nj - 1;
  const bool joint = own < nj;
  const Pose place = load_pose8(smem + L.place + 8 * j);
  float axis[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) axis[k] = smem[L.axis + 4 * j + k];
  const int jt = reinterpret_cast<const int*>(smem + L.jtype)[j];
  const int iq = reinterpret_cast<const int*>(smem + L.idxq)[j] + sub_ * nq;
  const int rounds = tree.rounds < 5 ? tree.rounds : 5;
  unsigned long long ancs = 0ull;  // lane of the ancestor in each round, 0xff: none left
  {
    int a = reinterpret_cast<const int*>(smem + L.parent)[j];
    for (int r = 0; r < 5; ++r) {
      ancs |= (unsigned long long)(a < 0 ? 0xff : base + a) << (8 * r);
      const int up = __shfl_sync(0xffffffffu, a, a < 0 ? lane : base + a);
      a = a < 0 ? -1 : up;
    }
  }
  auto from_lane = [](const Pose& P, int l) {
    Pose T;
    T.t.x = __shfl_sync(0xffffffffu, P.t.x, l);
    T.t.y = __shfl_sync(0xffffffffu, P.t.y, l);
    T.t.z = __shfl_sync(0xffffffffu, P.t.z, l);
    T.q.x = __shfl_sync(0xffffffffu, P.q.x, l);
    T.q.y = __shfl_sync(0xffffffffu, P.q.y, l);
    T.q.z = __shfl_sync(0xffffffffu, P.q.z, l);
    T.q.w = __shfl_sync(0xffffffffu, P.q.w, l);
    return T;
  };

  for (; g < groups; g += stride) {
    const int64_t b = g * kPer;
    const int cnt = p.batch - b < kPer ? (int)(p.batch - b) : kPer;
#pragma unroll
    for (int k = 0; k < kQRegs; ++k) {
      const int i = lane + kWarp * k;
      if (i < kPer * nq) wq[i] = qn[k];
    }
    if (g + stride < groups) fetch(g + stride);
    __syncwarp();
    const Pose Tl = local_transform(jt, place, axis, wq + iq);
    Pose T = Tl;
    for (int r = 0; r < rounds; ++r) {
      const int a = (int)(ancs >> (8 * r)) & 0xff;
      const Pose P = from_lane(T, a & 31);
      if (a != 0xff) T = compose_rn(P, T);
    }
    if (lane == 0) bulk_wait_read_all();  // the last group's blocks have been read out
    __syncwarp();
    if ((p.outputs & OUT_LIMI) && joint) store_pose7(sLiMi + 7 * (sub_ * nj + own), Tl);
    if ((p.outputs & OUT_OMI) && joint) store_pose7(sOMi + 7 * (sub_ * nj + own), T);
    for (int t0 = 0; t0 < nt; t0 += kG) {
      const int t = t0 + own < nt ? t0 + own : nt - 1;
      const Pose Tt = compose_rn(from_lane(T, base + s_tparent[t]), load_pose8(s_tplace + 8 * t));
      if (t0 + own < nt) {
        if (kJac) store_pose8(wtgt + 8 * t, Tt);
        if (p.outputs & OUT_TPOSE) store_pose7(sT + 7 * (sub_ * nt + t), Tt);
      }
    }
    if (kJac) {
      if (joint) *reinterpret_cast<float4*>(wpT + 4 * own) = make_float4(T.t.x, T.t.y, T.t.z, 0.f);
      for (int c0 = 0; c0 < nv; c0 += kG) {
        const int c = c0 + own < nv ? c0 + own : nv - 1;
        const int l = base + s_cjoint[c];
        float4 qc;
        qc.x = __shfl_sync(0xffffffffu, T.q.x, l);
        qc.y = __shfl_sync(0xffffffffu, T.q.y, l);
        qc.z = __shfl_sync(0xffffffffu, T.q.z, l);
        qc.w = __shfl_sync(0xffffffffu, T.q.w, l);
        const float4 ax = *reinterpret_cast<const float4*>(s_caxis + 4 * c);
        const float3 a = qrot(qc, f3(ax.x, ax.y, ax.z));
        if (c0 + own < nv) *reinterpret_cast<float4*>(wcA + 4 * c) = make_float4(a.x, a.y, a.z, ax.w);
      }
      __syncwarp();
      float* block = sJ + sub_ * nt * 6 * nv;
      for (int idx = own; idx < npairs; idx += kG) {
        const int pr = s_pairs[idx];
        const int t = pr >> 16, jc = (pr >> 8) & 255, c = pr & 255;
        jac_column<kRef>(wcA, wpT, wtgt, t, jc, c, block + t * 6 * nv + c, nv);
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    bool issued = false;
    auto put = [&](uint32_t bit, float* out, const float* s, int n) {  // n floats per configuration
      if (!(p.outputs & bit) || n == 0) return;
      float* dst = out + b * n;
      if ((p.bulk & bit) && cnt == kPer) {
        if (lane == 0) bulk_store(dst, s, (uint32_t)(kPer * n) * 4u);
        issued = true;
      } else {
        warp_copy(dst, s, cnt * n, lane);
      }
    };
    if (kJac) put(OUT_JAC, p.jac, sJ, nt * 6 * nv);
    put(OUT_TPOSE, p.tpose, sT, nt * 7);
    if (!kJac) {
      put(OUT_OMI, p.oMi, sOMi, nj * 7);
      put(OUT_LIMI, p.liMi, sLiMi, nj * 7);
    }
    if (issued && lane == 0) bulk_commit();
    __syncwarp();
  }
  if (lane == 0) bulk_wait_read_all();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
const DeviceInfo& device_info() {
  static DeviceInfo info[16];
  int dev = 0;
  cudaGetDevice(&dev);
  DeviceInfo& d = info[dev & 15];
  if (d.device != dev) {
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, dev);
    d.sms = prop.multiProcessorCount;
    d.max_smem_optin = (int)prop.sharedMemPerBlockOptin;
    d.smem_per_sm = (int)prop.sharedMemPerMultiprocessor;
    d.l2_bytes = prop.l2CacheSize;
    d.device = dev;
  }
  return d;
}

int validate_tree(const br_tree_t* t) {
  if (!t) return BR_EINVAL;
  if (t->njoints < 1 || t->nq < 0 || t->nv < 0 || t->nframes < 0 || t->rounds < 0) return BR_EINVAL;
  if (t->njoints > BR_MAX_JOINTS || t->nv > BR_MAX_NV || t->nq > BR_MAX_NQ) return BR_ETOOBIG;
  if (!t->parent || !t->jtype || !t->idx_q || !t->idx_v || !t->axis || !t->placement || !t->support) return BR_EINVAL;
  if (t->nv > 0 && (!t->col_joint || !t->col_kind || !t->col_axis)) return BR_EINVAL;
  if (t->nframes > 0 && (!t->frame_parent || !t->frame_placement)) return BR_EINVAL;
  return BR_OK;
}

static int g_warps_per_cta = 8;

// A configuration's J block above kWholeBlockBytes is staged in pieces of about
// kPieceBytes (an even number of targets, so that every piece starts and ends on a
// 16-byte boundary of a 16-byte aligned block).  Measured on all 32 joint Jacobians of the
// humanoid at B = 16,384: pieces of 2 / 4 / 8 / 14 / 18 targets (2-16 KB) took 92 / 92 / 84 /
// 92 / 108 us; the 8 KB pieces leave one 8-warp CTA per SM and fewer, larger bulk copies.
constexpr int kWholeBlockBytes = 16384, kPieceBytes = 8192;

// Launch kern over `items` pieces of work, one warp each at a time, on one wave of resident CTAs.
template <typename Kernel>
static int launch_wave(Kernel kern, int (&configured_bytes)[16], const Layout& L, int64_t items, const br_tree_t& tree,
                       const FkParams& p, cudaStream_t stream) {
  const DeviceInfo& dev = device_info();
  int wpc = g_warps_per_cta;
  size_t bytes = 0;
  for (;;) {
    bytes = (size_t)(L.cta_floats + wpc * L.warp_floats) * sizeof(float);
    if ((int)bytes <= dev.max_smem_optin || wpc == 1) break;
    wpc >>= 1;
  }
  if ((int)bytes > dev.max_smem_optin) return BR_ETOOBIG;
  const int devslot = dev.device & 15;
  if ((int)bytes > configured_bytes[devslot]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    configured_bytes[devslot] = (int)bytes;
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, wpc * kWarp, bytes);
  if (per_sm < 1) per_sm = 1;
  const int64_t need = (items + wpc - 1) / wpc;
  const int64_t cap = (int64_t)per_sm * dev.sms;
  const int grid = (int)(need < cap ? need : cap);
  kern<<<grid, wpc * kWarp, bytes, stream>>>(tree, p);
  return (int)cudaGetLastError();
}

static uint32_t bulk_bit(uint32_t bit, const float* base, int64_t floats_per_item) {
  return (base && aligned16(base) && ((floats_per_item * 4) % 16) == 0) ? bit : 0u;
}

template <int kRef, int kG, bool kJac>
static int launch_group(const br_tree_t& tree, FkParams p, cudaStream_t stream) {
  constexpr int kPer = kWarp / kG;
  const Layout L(tree.njoints, tree.nq, tree.nv, p.nt, p.outputs, p.nt, kPer, true);
  p.bulk = bulk_bit(OUT_JAC, p.jac, (int64_t)kPer * p.nt * 6 * tree.nv) | bulk_bit(OUT_TPOSE, p.tpose, (int64_t)kPer * p.nt * 7) |
           bulk_bit(OUT_OMI, p.oMi, (int64_t)kPer * tree.njoints * 7) |
           bulk_bit(OUT_LIMI, p.liMi, (int64_t)kPer * tree.njoints * 7);
  static int configured_bytes[16] = {0};
  return launch_wave(fk_group_kernel<kRef, kG, kJac>, configured_bytes, L, (p.batch + kPer - 1) / kPer, tree, p, stream);
}

// Lanes per configuration of the group kernel for this call, 0 where a warp per configuration with staged records
// runs: more than 32 joints; J blocks of a warp above kWholeBlockBytes; and, for trees that take a whole warp either
// way, Jacobians that do not fit in L2: stores to HBM bound those, and the group kernel's, issued closer together,
// drain more slowly (12 Jacobians of the humanoid, group / staged: B = 8,192 20.2 / 23.1 us, 16,384 36.7 / 36.6,
// 65,536 126 / 120).
static int group_lanes(const br_tree_t& tree, const FkParams& p) {
  if (tree.njoints > kWarp) return 0;
  const int lanes = tree.njoints <= 8 ? 8 : tree.njoints <= 16 ? 16 : 32;
  if (tree.nq > 7 * lanes && lanes < kWarp) return 0;
  if (p.outputs & OUT_JAC) {
    const int64_t block = (int64_t)p.nt * 6 * tree.nv * 4;
    if (block * (kWarp / lanes) > kWholeBlockBytes) return 0;
    if (lanes == kWarp && block * p.batch > device_info().l2_bytes) return 0;
  }
  return lanes;
}

template <int kRef, bool kFromQ>
static int launch_fk(const br_tree_t& tree, FkParams p, cudaStream_t stream) {
  if (p.batch == 0) return BR_OK;
  if (kFromQ) {
    const bool jac = (p.outputs & OUT_JAC) != 0;
    switch (group_lanes(tree, p)) {
      case 8: return jac ? launch_group<kRef, 8, true>(tree, p, stream) : launch_group<BR_REF_WORLD, 8, false>(tree, p, stream);
      case 16: return jac ? launch_group<kRef, 16, true>(tree, p, stream) : launch_group<BR_REF_WORLD, 16, false>(tree, p, stream);
      case 32: return jac ? launch_group<kRef, 32, true>(tree, p, stream) : launch_group<BR_REF_WORLD, 32, false>(tree, p, stream);
      default: break;
    }
  }
  p.chunk = p.nt;
  const int64_t jbytes = (int64_t)p.nt * 6 * tree.nv * 4;
  if ((p.outputs & OUT_JAC) && tree.nv > 0 && jbytes > kWholeBlockBytes) {
    int ch = (kPieceBytes / (6 * tree.nv * 4)) & ~1;
    p.chunk = ch < 2 ? 2 : ch;
  }
  const Layout L(tree.njoints, tree.nq, tree.nv, p.nt, p.outputs, p.chunk);
  static int configured_bytes[16] = {0};
  return launch_wave(fk_jac_kernel<kRef, kFromQ>, configured_bytes, L, p.batch, tree, p, stream);
}

template <bool kFromQ>
static int dispatch_fk(const br_tree_t& tree, const FkParams& p, int32_t reference, cudaStream_t s) {
  switch (reference) {
    case BR_REF_WORLD: return launch_fk<BR_REF_WORLD, kFromQ>(tree, p, s);
    case BR_REF_LOCAL_WORLD_ALIGNED: return launch_fk<BR_REF_LOCAL_WORLD_ALIGNED, kFromQ>(tree, p, s);
    case BR_REF_LOCAL: return launch_fk<BR_REF_LOCAL, kFromQ>(tree, p, s);
    default: return BR_EINVAL;
  }
}

static int fill_targets(const br_tree_t* tree, FkParams& p, const int32_t* targets, int32_t n) {
  if (n < 0) return BR_EINVAL;
  if (n > BR_MAX_TARGETS) return BR_ETOOBIG;
  if (n > 0 && !targets) return BR_EINVAL;
  for (int i = 0; i < n; ++i) {
    const int id = targets[i];
    if (id >= 0 ? id >= tree->nframes : (-id - 1) >= tree->njoints) return BR_EINVAL;
    p.targets[i] = id;
  }
  p.nt = n;
  return BR_OK;
}

}  // namespace br

using namespace br;

extern "C" int br_forward_kinematics(const br_tree_t* tree, const float* q, int64_t batch,
                                     float* joint_pose_world, float* joint_pose_local,
                                     const int32_t* frame_ids, int32_t n_frames, float* frame_pose_world,
                                     void* stream) {
  int st = validate_tree(tree);
  if (st) return st;
  if (batch < 0 || (batch > 0 && tree->nq > 0 && !q)) return BR_EINVAL;
  if ((q && !aligned4(q))) return BR_EALIGN;
  FkParams p = {};
  p.q = q;
  p.batch = batch;
  p.oMi = joint_pose_world;
  p.liMi = joint_pose_local;
  p.tpose = frame_pose_world;
  st = fill_targets(tree, p, frame_ids, frame_pose_world ? n_frames : 0);
  if (st) return st;
  if ((joint_pose_world && !aligned4(joint_pose_world)) || (joint_pose_local && !aligned4(joint_pose_local)) ||
      (frame_pose_world && !aligned4(frame_pose_world)))
    return BR_EALIGN;
  p.outputs = (joint_pose_world ? OUT_OMI : 0u) | (joint_pose_local ? OUT_LIMI : 0u) |
              (frame_pose_world && p.nt > 0 ? OUT_TPOSE : 0u);
  p.bulk = bulk_bit(OUT_OMI, joint_pose_world, (int64_t)tree->njoints * 7) |
           bulk_bit(OUT_LIMI, joint_pose_local, (int64_t)tree->njoints * 7) |
           bulk_bit(OUT_TPOSE, frame_pose_world, (int64_t)p.nt * 7);
  if (!p.outputs) return BR_OK;
  return dispatch_fk<true>(*tree, p, BR_REF_LOCAL_WORLD_ALIGNED, (cudaStream_t)stream);
}

extern "C" int br_frame_jacobians(const br_tree_t* tree, const float* q, int64_t batch, const int32_t* targets,
                                  int32_t n_targets, int32_t reference, float* target_pose_world,
                                  float* jacobians, void* stream) {
  int st = validate_tree(tree);
  if (st) return st;
  if (batch < 0 || (batch > 0 && ((tree->nq > 0 && !q) || !jacobians))) return BR_EINVAL;  // B = 0: empty buffers
  if (!aligned4(q) || !aligned4(jacobians) || (target_pose_world && !aligned4(target_pose_world))) return BR_EALIGN;
  FkParams p = {};
  p.q = q;
  p.batch = batch;
  p.jac = jacobians;
  p.tpose = target_pose_world;
  st = fill_targets(tree, p, targets, n_targets);
  if (st) return st;
  p.outputs = OUT_JAC | (target_pose_world ? OUT_TPOSE : 0u);
  p.bulk = bulk_bit(OUT_JAC, jacobians, (int64_t)p.nt * 6 * tree->nv) |
           bulk_bit(OUT_TPOSE, target_pose_world, (int64_t)p.nt * 7);
  return dispatch_fk<true>(*tree, p, reference, (cudaStream_t)stream);
}

extern "C" int br_frame_jacobians_from_poses(const br_tree_t* tree, const float* joint_pose_world, int64_t batch,
                                             const int32_t* targets, int32_t n_targets, int32_t reference,
                                             float* jacobians, void* stream) {
  int st = validate_tree(tree);
  if (st) return st;
  if (batch < 0 || (batch > 0 && (!joint_pose_world || !jacobians))) return BR_EINVAL;  // B = 0: empty buffers
  if (!aligned4(joint_pose_world) || !aligned4(jacobians)) return BR_EALIGN;
  FkParams p = {};
  p.oMi_in = joint_pose_world;
  p.batch = batch;
  p.jac = jacobians;
  st = fill_targets(tree, p, targets, n_targets);
  if (st) return st;
  p.outputs = OUT_JAC;
  p.bulk = bulk_bit(OUT_JAC, jacobians, (int64_t)p.nt * 6 * tree->nv);
  return dispatch_fk<false>(*tree, p, reference, (cudaStream_t)stream);
}

extern "C" const char* br_version(void) { return "br_b200 0.1 (sm_100a)"; }
