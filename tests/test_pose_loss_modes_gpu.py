"""What the modes of the pose loss keep between forward and backward, and the entry points' stored placements.

Gradient tolerance: 1e-5 per configuration against the float64 oracle, as in ``test_adjoint_gpu.py``.
"""

import numpy as np
import pytest
import torch

from betterrobot_b200 import _lib, synthetic as syn
from betterrobot_b200.adjoint import pose_loss
from betterrobot_b200.tree import device_tree
from oracle import adjoint as A, kinematics as K

pytestmark = pytest.mark.gpu
TOL = 1e-5
SPECS = {"humanoid": syn.humanoid_spec, "dual_arm": syn.dual_arm_spec}


def _problem(robot, B, nf=None):
    m, m64 = syn.model_from_spec(SPECS[robot]()), syn.model_from_spec(SPECS[robot](), dtype=torch.float64)
    fids = syn.op_frame_ids(m)
    if nf is not None:
        fids = [(fids + list(range(m.nframes)))[i % m.nframes] for i in range(nf)]
    q = syn.random_q(m64, B, 71, rev_range=2.5, base_translation=1.0).float()
    near = syn.noisy_start(m64, q.double(), 0.3, 72).numpy()
    T = K.frame_placements(m64, K.forward_kinematics(m64, near)[0], fids).astype(np.float32)
    w = np.random.default_rng(73).uniform(0.5, 2.0, len(fids)).astype(np.float32)
    args = (q.double().numpy(), fids, T.astype(float), w.astype(float))
    return m, fids, q.cuda(), torch.from_numpy(T).cuda(), torch.from_numpy(w).cuda(), A.pose_loss(m64, *args), \
        A.pose_loss_grad(m64, *args)


def _rel(g, ref):
    return np.linalg.norm(g.cpu().double().numpy() - ref, axis=-1) / np.linalg.norm(ref, axis=-1)


@pytest.mark.parametrize("robot,B", [("humanoid", 301), ("humanoid", 9000), ("dual_arm", 4001)])
def test_recompute_keeps_no_gradient_and_returns_the_same(robot, B):
    m, fids, q, T, w, loss, grad = _problem(robot, B)
    kept, got = {}, {}
    for mode in ("store", "recompute", "auto"):
        qg = q.clone().requires_grad_(True)
        saved = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (saved.append(t), t)[1], lambda t: t):
            out = pose_loss(m, qg, fids, T, w, mode=mode)
        own = {t.data_ptr() for t in (qg, T, w)}
        kept[mode] = sum(t.numel() for t in saved if t.data_ptr() not in own)
        go = torch.linspace(0.5, 2.0, B, device="cuda")
        got[mode], = torch.autograd.grad(out, qg, go, retain_graph=True)
        again, = torch.autograd.grad(out, qg, torch.stack((go, go), 1)[:, 0])      # a strided gradient
        assert torch.equal(again, got[mode])
        assert _rel(got[mode], grad * go.cpu().double().numpy()[:, None]).max() <= TOL, mode
        np.testing.assert_allclose(out.detach().cpu().numpy(), loss, rtol=TOL)
    assert kept == {"store": B * m.nq, "recompute": 0, "auto": B * m.nq}
    assert torch.equal(got["auto"], got["store"])


def test_inputs_changed_before_the_backward_stay_an_error():
    m, fids, q, T, w, _, _ = _problem("dual_arm", 33)
    for mode in ("store", "recompute"):
        qg, Tc = q.clone().requires_grad_(True), T.clone()
        out = pose_loss(m, qg, fids, Tc, w, mode=mode).sum()
        Tc += 1.0
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            out.backward()


@pytest.mark.parametrize("robot,B,nf", [("humanoid", 37, None), ("humanoid", 9001, None), ("humanoid", 37, 20),
                                        ("dual_arm", 301, 16)])
@pytest.mark.parametrize("per_cfg", [False, True])
def test_stored_placements_of_the_entry_points(robot, B, nf, per_cfg):
    """``br_pose_loss`` writes the joint placements, ``br_pose_loss_backward`` reads them instead of q's
    kinematics: two configurations per warp pass and one (more than 16 frames), odd batches."""
    m, fids, q, T, w, loss, grad = _problem(robot, B, nf)
    if per_cfg:
        w = w.expand(B, -1).contiguous()
    dt, ids, F = device_tree(m, q.device), (_lib.c_int32 * len(fids))(*fids), len(fids)
    oMi = torch.full((B, m.njoints, 7), float("nan"), device="cuda")
    out, g = torch.empty(B, device="cuda"), torch.full_like(q, float("nan"))
    go = torch.linspace(0.5, 2.0, B, device="cuda")
    s = _lib.stream_ptr()
    _lib.call("br_pose_loss", dt.ptr, q.data_ptr(), B, ids, F, T.data_ptr(), w.data_ptr(), int(per_cfg),
              out.data_ptr(), oMi.data_ptr(), s)
    m64 = syn.model_from_spec(SPECS[robot](), dtype=torch.float64)
    ref = K.forward_kinematics(m64, q.cpu().double().numpy())[0]
    assert np.abs(oMi.cpu().double().numpy()[..., :3] - ref[..., :3]).max() <= 1e-5
    np.testing.assert_allclose(out.cpu().numpy(), loss, rtol=TOL)
    _lib.call("br_pose_loss_backward", dt.ptr, q.data_ptr(), oMi.data_ptr(), B, ids, F, T.data_ptr(), w.data_ptr(),
              int(per_cfg), go.data_ptr(), g.data_ptr(), s)
    assert _rel(g, grad * go.cpu().double().numpy()[:, None]).max() <= TOL
