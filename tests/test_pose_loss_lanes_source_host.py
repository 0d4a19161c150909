"""The lane-per-configuration pose-loss kernel's own source, run on the CPU between guard pages.

``cuda_on_cpu.h`` compiles the kernel with g++ (no optimisation: every load in the source is made) and
runs its CTAs fiber by fiber.  Each buffer of the call ends, then begins, at an unmapped page, so an access one
float outside it fails the test; shared memory is exactly as large as the launch makes it and starts
as NaN.  Results are compared with the float64 oracle: float32 rounding through ~40 products each way,
2e-6 of the batch's norm; a loss that is zero but for rounding (a frame that nothing moves) to 1e-11, the
square of a 1e-6 pose error over the frames' weights.
"""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from betterrobot_b200 import synthetic as syn, tree as tr
from betterrobot_b200.adjoint import path_slots
from betterrobot_b200.model import build_model
from oracle import adjoint as A, kinematics as K

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "betterrobot_b200", "csrc")
TOL, ZERO_LOSS = 2e-6, 1e-11

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")

_DRIVER = r"""
using namespace br;
extern "C" int run_lanes(const br_tree_t* tree, const float* q, int64_t B, const int* frames, int nf, const float* targets,
                         const float* weights, int per, const float* go, float* loss, float* grad, int grid, int warps,
                         int want_grad, int slots, int at_end) {
  const size_t nq = tree->nq, f = sizeof(float);
  emu::Guarded gq(q, B * nq * f, at_end), gt(targets, B * nf * 7 * f, at_end), gw(weights, (per ? B : 1) * nf * f, at_end);
  emu::Guarded gg(go, B * f, at_end), gl(nullptr, B * f, at_end), gr(nullptr, B * nq * f, at_end);
  LossParams p = {};
  p.q = (const float*)gq.data; p.targets = (const float*)gt.data; p.weights = (const float*)gw.data;
  p.weights_per_config = per; p.batch = B; p.nf = nf; p.path_slots = slots;
  p.loss = (float*)gl.data; p.grad_q = (float*)gr.data; p.grad_loss = go ? (const float*)gg.data : nullptr;
  for (int i = 0; i < nf; ++i) p.frames[i] = frames[i];
  const LaneLayout L(tree->njoints, tree->nq, nf, want_grad, per, slots);
  const size_t bytes = (size_t)(L.cta_floats + warps * L.warp_floats) * f;
  void* bad = emu::launch(grid, warps * 32, bytes, [&] {
    if (want_grad) pose_loss_lanes_kernel<true>(*tree, p);
    else pose_loss_lanes_kernel<false>(*tree, p);
  });
  memcpy(loss, gl.data, B * f);
  if (want_grad) memcpy(grad, gr.data, B * nq * f);
  return bad ? -1 : 0;
}
"""


def _between(text, a, b):
    return text[text.index(a):text.index(b, text.index(a))]


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")

    def read(name):
        text = open(os.path.join(CSRC, name)).read()
        return "\n".join(x for x in text.splitlines() if not x.startswith(("#include", "#pragma once"))) + "\n"

    src = read("fk_adjoint.cu")
    kernel = _between(src, "struct LossParams", "struct LossLayout") + \
        _between(src, "// Raw-q chain rules", "// out[b, :] = unit[b, :]")
    kernel = kernel.replace("extern __shared__ __align__(16) float smem[];", "float* smem = emu::smem;")
    cpp, so = str(d / "lanes.cpp"), str(d / "lanes.so")
    with open(cpp, "w") as f:
        f.write('#include "cuda_on_cpu.h"\n' + read("br_lie.cuh") + read("br_fk.cuh") + "namespace br {\n" + kernel +
                "}\n" + _DRIVER)
    subprocess.run(["g++", "-std=c++20", "-O0", "-U_FORTIFY_SOURCE", "-w", "-shared", "-fPIC", f"-I{HERE}",
                    f"-I{os.path.join(os.path.dirname(HERE), 'include')}", "-I/usr/local/cuda/include", cpp, "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def _ptr(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def _check(lib, build, fids, B, warps=1, grid=1, per=False, far=None, go=False, slots=True):
    m, m64 = build(torch.float32), build(torch.float64)
    dt = tr.DeviceTree(m, torch.device("cpu"))
    rng = np.random.default_rng(B)
    q = np.ascontiguousarray(syn.random_q(m64, B, 1, rev_range=2.5).float().numpy())
    if far is not None:
        q[-1, far] += 65536.0
    near = syn.noisy_start(m64, torch.from_numpy(q).double(), 0.3, 2).numpy()
    T = np.ascontiguousarray(K.frame_placements(m64, K.forward_kinematics(m64, near)[0], fids).astype(np.float32))
    w = rng.uniform(0.5, 2.0, (B, len(fids)) if per else len(fids)).astype(np.float32)
    s = rng.uniform(0.5, 2.0, B).astype(np.float32) if go else None
    f = np.array(fids, np.int32)
    want_l = A.pose_loss(m64, q.astype(float), fids, T.astype(float), w.astype(float))
    want_g = A.pose_loss_grad(m64, q.astype(float), fids, T.astype(float), w.astype(float))
    if go:
        want_g = want_g * s[:, None]
    n_slots = path_slots(dt.arrays, tuple(fids)) if slots else -1
    for at_end in (1, 0):
        for want in (1, 0):
            loss, grad = np.zeros(B, np.float32), np.zeros_like(q)
            rc = lib.run_lanes(ctypes.byref(dt.struct), _ptr(q), ctypes.c_int64(B), _ptr(f), len(fids), _ptr(T), _ptr(w),
                               int(per), _ptr(s), _ptr(loss), _ptr(grad), grid, warps, want, n_slots, at_end)
            assert rc == 0, "an access outside the call's buffers"
            assert np.abs(loss - want_l).max() <= TOL * np.abs(want_l).max() + ZERO_LOSS
            if want:
                assert np.linalg.norm(grad - want_g) <= TOL * np.linalg.norm(want_g) + ZERO_LOSS ** 0.5


def _arm_with_flange(n):
    """A serial arm of n revolute joints whose tracked frame sits on a fixed joint after the last one."""
    def build(dtype):
        rng = np.random.default_rng(n)
        joints = [{"name": f"j{i}", "kind": ("revolute_rx", "revolute_ry", "revolute_rz")[i % 3], "parent": i,
                   "origin": syn._rand_pose(rng), "lower": -3, "upper": 3, "body": f"b{i}"} for i in range(n)]
        joints.append({"name": "flange", "kind": "fixed", "parent": n, "origin": syn._rand_pose(rng), "body": "tool"})
        return build_model("arm", joints, [{"name": "tcp", "parent": n + 1, "placement": syn._rand_pose(rng)}], dtype=dtype)
    return build


@pytest.mark.parametrize("n", [2, 3, 6, 7])
@pytest.mark.parametrize("B", [32, 33, 45])
def test_far_angle_beside_a_trailing_fixed_joint(lanes, n, B):
    """Angles beyond the fast sine's range are read again from q; a flange after the last moving joint
    has no slot of q (its idx_q is nq), and nothing may be read there."""
    build = _arm_with_flange(n)
    m = build(torch.float32)
    assert int(m.idx_qs[-1]) == m.nq
    _check(lanes, build, [m.frame_id("tcp")], B, far=0)


def _spec(f):
    return lambda dtype: syn.model_from_spec(f(), dtype=dtype)


def _random_tree(seed):
    """14 joints of every axis form and several kinds, numbered in any topological order; nq from 8 to 40."""
    def build(dtype):
        rng = np.random.default_rng(seed)
        kinds = ["revolute_rx", "revolute_ry", "revolute_rz", "revolute_unaligned", "prismatic_px", "fixed", "spherical"]
        joints = []
        for i in range(14):
            rec = {"name": f"j{i}", "kind": str(rng.choice(kinds)), "parent": int(rng.integers(0, i + 1)),
                   "origin": syn._rand_pose(rng), "lower": -3, "upper": 3, "body": f"b{i}"}
            if rec["kind"] == "revolute_unaligned":
                rec["axis"] = [(0, -1, 0), (0.6, 0, 0.8), (-1, 0, 0), (0, 0, -1)][rng.integers(0, 4)]
            joints.append(rec)
        frames = [{"name": f"f{i}", "parent": int(rng.integers(0, 15)), "placement": syn._rand_pose(rng)}
                  for i in range(5)]
        return build_model("tree", joints, frames, dtype=dtype)
    return build


_MODELS = {"chain7": _spec(syn.chain_spec), "dual_arm": _spec(syn.dual_arm_spec), "humanoid": _spec(syn.humanoid_spec),
           "mixed": _spec(syn.mixed_spec)} | {f"tree{i}": _random_tree(i) for i in range(12)}


@pytest.mark.parametrize("name", sorted(_MODELS))
def test_every_access_in_bounds(lanes, name):
    """Odd and even nq (contiguous and padded rows), ragged tiles, one and two warps and CTAs, both kinds
    of weights, a known and an unknown bound on the waiting wrenches, all frames and few."""
    build = _MODELS[name]
    m = build(torch.float32)
    op = syn.op_frame_ids(m)
    _check(lanes, build, op, 33, per=True)
    _check(lanes, build, op + [m.nframes - 1], 16, go=True, slots=False)
    _check(lanes, build, [m.nframes - 1], 70, warps=2, per=True)
    _check(lanes, build, list(range(min(m.nframes, 30))), 97, grid=2, go=True)


def test_both_row_layouts_are_covered():
    parity = {_MODELS[n](torch.float32).nq % 2 for n in _MODELS if n.startswith("tree")}
    assert parity == {0, 1} and _MODELS["dual_arm"](torch.float32).nq % 2 == 0
