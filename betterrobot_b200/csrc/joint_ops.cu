// joint_ops.cu — batched configuration-space retraction and difference.
//
// integrate:  q' = q (+) v   (Model.integrate, src/better_robot/data_model/model.py:160-174):
//   revolute / prismatic / translation  q' = q + v       (revolute.py:46-48, translation.py:40-41)
//   free-flyer            q' = normalize(q * exp(v))     (free_flyer.py:47-51)
//   spherical             q' = normalize(q * exp(v))     (spherical.py:52-56)
//   planar, unbounded     theta' = atan2(sin, cos) + v   (planar.py:61-68, revolute.py:223-231)
// difference: v = q1 (-) q0  (Model.difference, model.py:176-190):
//   revolute / prismatic / translation  v = q1 - q0      (revolute.py:51-53)
//   free-flyer            v = log(q0^-1 * q1)            (free_flyer.py:53-57)
//   spherical             v = log(normalize(q0^-1 q1))   (spherical.py:58-62)
//   planar, unbounded     atan2(q1) - atan2(q0)          (planar.py:70-76, revolute.py:233-237)
//
// Layout: a warp owns a tile of 32 consecutive configurations.  Their rows of every
// input are one contiguous slab, copied into the warp's shared memory with 16-byte
// cp.async copies (all of a tile's copies in flight at once; pointers that are not
// 16-byte aligned are read 4 bytes at a time, kVec = false); the slots of the other kinds
// (free-flyer, spherical, planar, unbounded) are then computed one configuration per lane (the float64 exp / log runs on 32 lanes at once),
// and the output slab is written 32 consecutive floats at a time, each from the one or two
// staged floats that a table of the CTA names.  Memory bound: 4 * (nq + nv + nq) bytes per
// configuration for integrate, 4 * (nq + nq + nv) for difference.
#include <cuda_runtime.h>
#include <stdint.h>

#include "br_common.cuh"
#include "br_fk.cuh"
#include "br_lie.cuh"

namespace br {

struct JointOpParams {
  const float* a;   // q (integrate) or q0 (difference)        [B, nq]
  const float* b;   // v (integrate, [B, nv]) or q1 (difference, [B, nq])
  float* out;       // q' [B, nq] or v [B, nv]
  int64_t batch;
  int32_t n_active; // joints with nq > 0
  int32_t diff;     // 0 integrate, 1 difference
};

constexpr int kJointOpsWarps = 4;

// Floats of shared memory one warp stages: both inputs' rows of a tile.
__host__ __device__ inline int joint_ops_warp_floats(int nq, int nv, bool diff) { return 32 * (diff ? 2 * nq : nq + nv); }

__device__ __forceinline__ DPose dpose7(const float* p) {
  return DPose{d3(p[0], p[1], p[2]), make_double4(p[3], p[4], p[5], p[6])};
}

template <bool kVec>
__device__ __forceinline__ void slab_in(float* s, const float* __restrict__ g, int n, int lane) {
  int done = 0;
  if (kVec) {
    const int n4 = n >> 2;
    for (int i = lane; i < n4; i += 32) cp_async16(s + 4 * i, g + 4 * i);
    done = n4 << 2;
  }
  for (int i = done + lane; i < n; i += 32) s[i] = g[i];
}

// exp of a free-flyer's step, as dse3_exp with one sincos and one reciprocal root: with k = sin(th/2) / th,
// (1 - cos th) / th^2 = 2 k^2 and (th - sin th) / th^3 = (1 - 2 k cos(th/2)) / th^2.
__device__ __forceinline__ DPose step_exp(double3 v, double3 w) {
  const double th2 = ddot(w, w);
  double b, c, k, ch;
  if (th2 < 1e-8) {
    b = 0.5 - th2 / 24.0;
    c = 1.0 / 6.0 - th2 / 120.0;
    k = 0.5 - th2 / 48.0;
    ch = 1.0 - 0.125 * th2;
  } else {
    const double r = rsqrt(th2);
    double sh;
    sincos(0.5 * (th2 * r), &sh, &ch);
    k = sh * r;
    b = 2.0 * k * k;
    c = fma(-2.0 * k, ch, 1.0) * (r * r);
  }
  const double3 wv = dcross(w, v);
  DPose T;
  T.t = dadd(dadd(v, dscale(wv, b)), dscale(dcross(w, wv), c));
  T.q = make_double4(k * w.x, k * w.y, k * w.z, ch);
  return T;
}

constexpr uint32_t kNoTerm = 0xffffu;
// Tiles per warp of a CTA.  The hardware deals out the CTAs, so that SMs that run ahead take more (a fixed
// share per SM left them idle for a sixth of the time), and a CTA's tables are made while its first copies are in
// flight.  Measured, integrate / difference of 999,999 humanoids: 1 tile 82 / 88 us, 2 83 / 85, 4 84 / 86, one
// resident wave with all tiles 87 / 89; a copy of as many bytes takes 74.
constexpr int kTilesPerWarp = 2;

template <bool kVec, bool kDiff>
__global__ void __launch_bounds__(32 * kJointOpsWarps) joint_ops_kernel(const br_tree_t tree,
                                                                        const int32_t* __restrict__ active,
                                                                        const JointOpParams p) {
  extern __shared__ __align__(16) float slabs[];
  __shared__ int16_t vmap[BR_MAX_NQ];     // q slot -> v slot of a 1:1 joint, -1 for other slots
  __shared__ int16_t qmap[BR_MAX_NV];     // v slot -> q slot k of a 1:1 joint (k), or of the q0 slot that
                                          // holds a per-lane joint's output (-k - 1)
  __shared__ int16_t ffq[BR_MAX_JOINTS];  // q / v offsets and kind of the joints handled per lane
  __shared__ int16_t ffv[BR_MAX_JOINTS];   // (free-flyer, spherical, planar, unbounded revolute)
  __shared__ int8_t ffk[BR_MAX_JOINTS];
  __shared__ int nff;
  const int nq = tree.nq, nv = tree.nv;
  const int lb = kDiff ? nq : nv;  // floats per configuration of b
  const int lo = kDiff ? nv : nq;  // floats per configuration of out
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  float* A = slabs + 32 * lo + (size_t)(threadIdx.x >> 5) * joint_ops_warp_floats(nq, nv, kDiff);
  float* Bs = A + 32 * nq;
  const int64_t tiles = (p.batch + 31) >> 5;
  auto fetch = [&](int64_t tile) {  // the tile's rows of both inputs
    const int64_t b = tile << 5;
    const int c = p.batch - b < 32 ? (int)(p.batch - b) : 32;
    slab_in<kVec>(A, p.a + b * nq, c * nq, lane);
    slab_in<kVec>(Bs, p.b + b * lb, c * lb, lane);
  };
  // the first tile's copies run while the tables below are made
  int64_t tile = (int64_t)blockIdx.x * (kTilesPerWarp * warps) + (threadIdx.x >> 5);
  if (tile < tiles) fetch(tile);
  for (int k = threadIdx.x; k < nq; k += blockDim.x) vmap[k] = -1;
  for (int k = threadIdx.x; k < nv; k += blockDim.x) qmap[k] = -1;
  if (threadIdx.x == 0) nff = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < p.n_active; i += blockDim.x) {
    const int j = active[i];
    const int iq = tree.idx_q[j], iv = tree.idx_v[j];
    const int jt = tree.jtype[j];
    if (joint_is_vector(jt)) {
      for (int k = 0; k < joint_nv(jt); ++k) {
        vmap[iq + k] = (int16_t)(iv + k);
        qmap[iv + k] = (int16_t)(iq + k);
      }
    } else {
      for (int k = 0; k < joint_nv(jt); ++k) qmap[iv + k] = (int16_t)(-(iq + k) - 1);
      const int s = atomicAdd(&nff, 1);
      ffq[s] = (int16_t)iq;
      ffv[s] = (int16_t)iv;
      ffk[s] = (int8_t)jt;
    }
  }
  __syncthreads();
  // Output e of a tile is S[term e & 0xffff] (+ or -) S[term e >> 16] of the warp's slab S (both inputs' rows), the
  // second left out where it is kNoTerm: 32 lanes at consecutive e read consecutive banks.  (Four outputs per lane as one
  // float4, their slots found by division, took a 4-way bank conflict on every read.)
  uint32_t* term = reinterpret_cast<uint32_t*>(slabs);
  for (int e = threadIdx.x; e < 32 * lo; e += blockDim.x) {
    const int c = e / lo, k = e - c * lo;
    if (kDiff) {
      const int kq = qmap[k];
      term[e] = kq >= 0 ? (uint32_t)(32 * nq + c * nq + kq) | (uint32_t)(c * nq + kq) << 16
                        : (uint32_t)(c * nq - kq - 1) | kNoTerm << 16;
    } else {
      term[e] = (uint32_t)e | (vmap[k] >= 0 ? (uint32_t)(32 * nq + c * nv + vmap[k]) : kNoTerm) << 16;
    }
  }
  __syncthreads();
  const int n_ff = nff;
  for (int i = 0; i < kTilesPerWarp && tile < tiles; ++i, tile += warps) {
    const int64_t b0 = tile << 5;
    const int cnt = p.batch - b0 < 32 ? (int)(p.batch - b0) : 32;
    if (i > 0) fetch(tile);
    if (kVec) cp_async_wait_all();
    __syncwarp();
    if (lane < cnt) {
      for (int f = 0; f < n_ff; ++f) {
        const int iq = ffq[f], iv = ffv[f], jt = ffk[f];
        float* qa = A + lane * nq + iq;
        if (!kDiff) {
          const float* v = Bs + lane * nv + iv;
          if (jt == BR_JOINT_FREE_FLYER) {
            DPose n = dcompose(dpose7(qa), step_exp(d3(v[0], v[1], v[2]), d3(v[3], v[4], v[5])));
            n.q = dqnormalize(n.q);
            qa[0] = (float)n.t.x; qa[1] = (float)n.t.y; qa[2] = (float)n.t.z;
            qa[3] = (float)n.q.x; qa[4] = (float)n.q.y; qa[5] = (float)n.q.z; qa[6] = (float)n.q.w;
          } else if (jt == BR_JOINT_SPHERICAL) {  // normalize(q * exp(v)), spherical.py:52-56
            const double4 n = dqnormalize(dqmul(make_double4(qa[0], qa[1], qa[2], qa[3]),
                                                dse3_exp(d3(0.0, 0.0, 0.0), d3(v[0], v[1], v[2])).q));
            qa[0] = (float)n.x; qa[1] = (float)n.y; qa[2] = (float)n.z; qa[3] = (float)n.w;
          } else {                                // planar.py:61-68, revolute.py:223-231
            const int k = jt == BR_JOINT_PLANAR ? 2 : 0;
            double s, c;
            sincos(atan2((double)qa[k + 1], (double)qa[k]) + (double)v[k], &s, &c);
            if (jt == BR_JOINT_PLANAR) {
              qa[0] = qa[0] + v[0];
              qa[1] = qa[1] + v[1];
            }
            qa[k] = (float)c;
            qa[k + 1] = (float)s;
          }
        } else {
          // outputs in place of the joint's own q0 slots (each read before it is written)
          const float* qb = Bs + lane * nq + iq;
          float* o = qa;
          if (jt == BR_JOINT_FREE_FLYER) {
            double3 v, w;
            dse3_log(dcompose(dinverse(dpose7(qa)), dpose7(qb)), v, w);
            o[0] = (float)v.x; o[1] = (float)v.y; o[2] = (float)v.z;
            o[3] = (float)w.x; o[4] = (float)w.y; o[5] = (float)w.z;
          } else if (jt == BR_JOINT_SPHERICAL) {  // log(normalize(q0^-1 q1)), spherical.py:58-62
            const double3 w = dso3_log(dqnormalize(dqmul(dqconj(make_double4(qa[0], qa[1], qa[2], qa[3])),
                                                         make_double4(qb[0], qb[1], qb[2], qb[3]))));
            o[0] = (float)w.x; o[1] = (float)w.y; o[2] = (float)w.z;
          } else {                                // planar.py:70-76, revolute.py:233-237
            const int k = jt == BR_JOINT_PLANAR ? 2 : 0;
            const double dth = atan2((double)qb[k + 1], (double)qb[k]) - atan2((double)qa[k + 1], (double)qa[k]);
            if (jt == BR_JOINT_PLANAR) {
              o[0] = qb[0] - qa[0];
              o[1] = qb[1] - qa[1];
            }
            o[k] = (float)dth;
          }
        }
      }
    }
    __syncwarp();
    float* go = p.out + b0 * lo;
    const int n = cnt * lo;
#pragma unroll 4
    for (int e = lane; e < n; e += 32) {
      const uint32_t t = term[e];
      float x = A[t & 0xffffu];
      const uint32_t y = t >> 16;
      if (y != kNoTerm) x = kDiff ? x - A[y] : x + A[y];
      go[e] = x;
    }
    __syncwarp();  // the slab is free for the next tile
  }
}

// *flag = 1 if any row's quaternion norm is further than tol from 1 (a NaN norm is not).  One pass over
// four floats of each row, bound by latency: 3 us for 16,001 rows of 30 floats, where the norms, the
// comparison, the reduction and the copy of the answer as tensor operations took 16 us of the GPU and a
// round trip before the caller's own kernel could start (forward kinematics + joint Jacobians of those
// configurations: 184 -> 125 us).  The flag may be pinned host memory; it is only written on a violation.
__global__ void __launch_bounds__(256) check_quaternions_kernel(const float* __restrict__ q, int64_t rows,
                                                                int32_t row_floats, float tol, int32_t* flag) {
  bool bad = false;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < rows; b += (int64_t)gridDim.x * blockDim.x) {
    const float* p = q + b * row_floats;
    const float x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2), w = __ldg(p + 3);
    bad = bad || fabsf(sqrtf(x * x + y * y + z * z + w * w) - 1.f) > tol;
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *flag = 1;
}

}  // namespace br

using namespace br;

extern "C" int br_check_quaternions(const float* quat, int64_t rows, int32_t row_floats, int32_t tol_millionths,
                                    int32_t* flag, void* stream) {
  if (rows < 0 || row_floats < 4 || tol_millionths < 0) return BR_EINVAL;
  if (rows == 0) return BR_OK;
  if (!quat || !flag) return BR_EINVAL;
  if (!aligned4(quat) || !aligned4(flag)) return BR_EALIGN;
  int64_t blocks = (rows + 255) / 256;
  const int64_t cap = (int64_t)device_info().sms * 8;
  if (blocks > cap) blocks = cap;
  check_quaternions_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(quat, rows, row_floats,
                                                                               1e-6f * (float)tol_millionths, flag);
  return (int)cudaGetLastError();
}

extern "C" int br_configuration_op(const br_tree_t* tree, const int32_t* active_joints, int32_t n_active, int32_t op,
                                   const float* a, const float* b, int64_t batch, float* out, void* stream) {
  int st = validate_tree(tree);
  if (st) return st;
  if (op != BR_OP_INTEGRATE && op != BR_OP_DIFFERENCE) return BR_EINVAL;
  if (batch < 0 || n_active < 0 || n_active > tree->njoints) return BR_EINVAL;
  if (batch == 0 || n_active == 0) return BR_OK;
  if (!active_joints || !a || !b || !out) return BR_EINVAL;
  if (!aligned4(a) || !aligned4(b) || !aligned4(out)) return BR_EALIGN;
  JointOpParams p = {a, b, out, batch, n_active, op == BR_OP_DIFFERENCE};
  const DeviceInfo& d = device_info();
  const bool vec = aligned16(a) && aligned16(b) && aligned16(out);
  const int lo = p.diff ? tree->nv : tree->nq;
  const size_t bytes =
      (32 * (size_t)lo + (size_t)kJointOpsWarps * joint_ops_warp_floats(tree->nq, tree->nv, p.diff)) * sizeof(float);
  if ((int64_t)bytes > d.max_smem_optin) return BR_ETOOBIG;
  auto kern = p.diff ? (vec ? joint_ops_kernel<true, true> : joint_ops_kernel<false, true>)
                     : (vec ? joint_ops_kernel<true, false> : joint_ops_kernel<false, false>);
  static size_t configured[4][16] = {};
  size_t& have = configured[2 * p.diff + vec][d.device & 15];
  if (bytes > have) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    have = bytes;
  }
  const int64_t tiles = (batch + 31) / 32;
  const int64_t blocks = (tiles + kTilesPerWarp * kJointOpsWarps - 1) / (kTilesPerWarp * kJointOpsWarps);
  if (blocks > 0x7fffffff) return BR_ETOOBIG;
  kern<<<(unsigned)blocks, 32 * kJointOpsWarps, bytes, (cudaStream_t)stream>>>(*tree, active_joints, p);
  return (int)cudaGetLastError();
}
