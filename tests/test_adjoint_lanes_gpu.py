"""GPU checks of the lane-per-configuration pose-loss kernel against the float64 oracle.

Batches are above the dispatch line (200 (njoints + n_frames) configurations takes it for every entry
point) and ragged against the 32-configuration tiles.  Tolerance, fixed beforehand: float32 rounding
through a chain of at most ~40 products per frame pose and as many on the way back; the start's
warp-per-configuration kernel is held to 1e-5 per configuration by ``test_adjoint_gpu.py`` and the same
bar holds here, per configuration, for targets 0.3 rad per joint away (no rotation near pi).
"""

import numpy as np
import pytest
import torch

from betterrobot_b200 import _lib, synthetic as syn
from betterrobot_b200.adjoint import path_slots, pose_loss
from betterrobot_b200.model import build_model
from betterrobot_b200.tree import device_tree
from oracle import adjoint as A, kinematics as K

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _axes_tree(dtype):
    """Revolute joints about every kind of axis (+-x, +-y, +-z, unaligned), numbered out of depth-first order."""
    rng = np.random.default_rng(8)
    kinds = [("revolute_rx", None), ("revolute_ry", None), ("revolute_unaligned", (0, -1, 0)), ("revolute_rz", None),
             ("revolute_unaligned", (0.6, 0, 0.8)), ("prismatic_px", None), ("revolute_unaligned", (-1, 0, 0)),
             ("spherical", None), ("revolute_unaligned", (0, 0, -1))]
    joints = []
    for i, ((k, ax), par) in enumerate(zip(kinds, [0, 1, 1, 2, 3, 4, 3, 6, 7])):
        rec = {"name": f"j{i}", "kind": k, "parent": par, "origin": syn._rand_pose(rng), "lower": -3, "upper": 3,
               "body": f"b{i}"}
        joints.append(rec | ({"axis": ax} if ax else {}))
    frames = [{"name": f"f{i}", "parent": p, "placement": syn._rand_pose(rng)} for i, p in enumerate((9, 8, 5, 3))]
    return build_model("axes", joints, frames, dtype=dtype)


MODELS = {"humanoid": lambda d: syn.model_from_spec(syn.humanoid_spec(), dtype=d),
          "dual_arm": lambda d: syn.model_from_spec(syn.dual_arm_spec(), dtype=d),
          "chain7": lambda d: syn.model_from_spec(syn.chain_spec(), dtype=d),
          "mixed": lambda d: syn.model_from_spec(syn.mixed_spec(), dtype=d), "axes": _axes_tree}


def _problem(name, B, fids=None, per_cfg=False):
    m, m64 = MODELS[name](torch.float32), MODELS[name](torch.float64)
    fids = tuple(fids or syn.op_frame_ids(m))
    q = syn.random_q(m64, B, 11, rev_range=2.5, base_translation=1.0).float()
    if name == "mixed":  # away from the planar angle's own singularity at 0 and pi
        i = int(m.idx_qs[[jm.kind for jm in m.joint_models].index("planar")]) + 2
        th = torch.rand(B, generator=torch.Generator().manual_seed(1)) * 2.0 + 0.5
        q[:, i], q[:, i + 1] = th.cos(), th.sin()
    near = syn.noisy_start(m64, q.double(), 0.3, 12).numpy()
    T = K.frame_placements(m64, K.forward_kinematics(m64, near)[0], list(fids)).astype(np.float32)
    w = np.random.default_rng(13).uniform(0.5, 2.0, (B, len(fids)) if per_cfg else len(fids)).astype(np.float32)
    q64, T64, w64 = q.double().numpy(), T.astype(float), w.astype(float)
    return (m, fids, q.cuda(), torch.from_numpy(T).cuda(), torch.from_numpy(w).cuda(),
            A.pose_loss(m64, q64, list(fids), T64, w64), A.pose_loss_grad(m64, q64, list(fids), T64, w64))


def _rel(g, ref):
    return np.linalg.norm(g - ref, axis=-1) / np.maximum(np.linalg.norm(ref, axis=-1), 1e-6 * np.abs(ref).max())


@pytest.mark.parametrize("name,B,per_cfg", [("humanoid", 8833, True), ("dual_arm", 3617, False), ("chain7", 2047, True),
                                            ("mixed", 2081, False), ("axes", 2849, True)])
def test_value_and_gradient(name, B, per_cfg):
    m, fids, q, T, w, loss, grad = _problem(name, B, per_cfg=per_cfg)
    qg = q.clone().requires_grad_(True)
    out = pose_loss(m, qg, fids, T, w)
    go = torch.linspace(0.5, 2.0, B, device="cuda")
    g, = torch.autograd.grad(out, qg, go)
    np.testing.assert_allclose(out.detach().cpu().numpy(), loss, rtol=TOL, atol=TOL * loss.max())
    assert _rel(g.cpu().double().numpy(), grad * go.cpu().double().numpy()[:, None]).max() <= TOL
    with torch.no_grad():  # the loss alone
        np.testing.assert_allclose(pose_loss(m, qg, fids, T, w).cpu().numpy(), loss, rtol=TOL, atol=TOL * loss.max())


def test_unmoved_branches_and_large_angles():
    """One tracked hand (every other branch has no gradient), angles of thousands of turns in some rows."""
    B = 6000
    m, fids, q, T, w, loss, grad = _problem("humanoid", B, fids=[MODELS["humanoid"](torch.float32).nframes - 1])
    qg = q.clone().requires_grad_(True)
    g, = torch.autograd.grad(pose_loss(m, qg, fids, T, w).sum(), qg)
    g = g.cpu().double().numpy()
    assert _rel(g, grad).max() <= TOL and (g[:, (grad == 0).all(0)] == 0).all()
    far = q.clone()
    far[::7, 10:] += 65536.0                     # a float32 angle of its own: compared at that angle
    m64 = MODELS["humanoid"](torch.float64)
    ref = A.pose_loss_grad(m64, far.double().cpu().numpy(), list(fids), T.double().cpu().numpy(),
                           w.double().cpu().numpy())
    qf = far.clone().requires_grad_(True)
    gf, = torch.autograd.grad(pose_loss(m, qf, fids, T, w).sum(), qf)
    ok = _rel(gf.cpu().double().numpy(), ref)    # rows whose rotation error lands near pi are not comparable
    assert np.quantile(ok, 0.99) <= TOL


def test_backward_entry_point_and_slot_bound():
    """``br_pose_loss_backward`` without stored placements, and a path-slot bound that is too small."""
    B = 8900
    m, fids, q, T, w, loss, grad = _problem("humanoid", B)
    dt, ids = device_tree(m, q.device), (_lib.c_int32 * len(fids))(*fids)
    go, g, out = torch.full((B,), 0.5, device="cuda"), torch.empty_like(q), torch.empty(B, device="cuda")
    s = _lib.stream_ptr()
    _lib.call("br_pose_loss_backward", dt.ptr, q.data_ptr(), None, B, ids, len(fids), T.data_ptr(), w.data_ptr(), 0,
              go.data_ptr(), g.data_ptr(), s)
    assert _rel(g.cpu().double().numpy(), 0.5 * grad).max() <= TOL
    need = path_slots(dt.arrays, fids)
    assert need >= 1
    for slots, good in ((-1, True), (need, True), (need - 1, False)):
        _lib.call("br_pose_loss_value_grad", dt.ptr, q.data_ptr(), B, ids, len(fids), T.data_ptr(), w.data_ptr(), 0,
                  slots, out.data_ptr(), g.data_ptr(), s)
        if good:
            assert _rel(g.cpu().double().numpy(), grad).max() <= TOL
        else:
            assert torch.isnan(out).all() and torch.isnan(g).all()


def test_unaligned_buffers():
    """Rows that start off a 16-byte boundary take 4-byte copies."""
    B = 2049
    m, fids, q, T, w, loss, grad = _problem("chain7", B)
    buf = torch.empty(B * m.nq + 1, device="cuda")
    qo = buf[1:].view(B, m.nq).copy_(q).requires_grad_(True)
    g, = torch.autograd.grad(pose_loss(m, qo, fids, T, w).sum(), qo)
    assert _rel(g.cpu().double().numpy(), grad).max() <= TOL
