"""The kernels behind ``forward_kinematics`` and ``frame_jacobians``: configurations that share a warp (8 or 16
lanes each), a configuration per warp, and Jacobians beyond L2, at the edges of a group, with every block aligned
and not.  Tolerances are those of the float32 kernels against the float64 oracle (1e-5 m and rad, 1e-4 of a
Jacobian's largest entry); between two kernels the same hold twice over."""

import numpy as np
import pytest
import torch

import betterrobot_b200 as br
from betterrobot_b200 import synthetic as syn
from oracle import kinematics as K

pytestmark = pytest.mark.gpu

SPECS = {"chain7": syn.chain_spec, "dual_arm": syn.dual_arm_spec, "humanoid": syn.humanoid_spec, "mixed": syn.mixed_spec}


def _jac_close(got, ref, factor=1.0):
    scale = np.abs(ref).max(axis=(-1, -2), keepdims=True)
    assert (np.abs(got - ref) / np.maximum(scale, 1e-12)).max() <= factor * 1e-4


@pytest.mark.parametrize("reference", ["world", "local_world_aligned", "local"])
@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 33, 4097])
@pytest.mark.parametrize("name", list(SPECS))
def test_group_edges(name, B, reference):
    m = syn.model_from_spec(SPECS[name]())
    m64 = syn.model_from_spec(SPECS[name](), dtype=torch.float64)
    q = syn.random_q(m64, B, 7 + B, rev_range=2.5).float()
    rows = np.unique(np.r_[0:min(B, 6), max(0, B - 6):B])
    ids = sorted({0, m.nframes // 2, m.nframes - 1})
    oMi, liMi = K.forward_kinematics(m64, q.double().numpy()[rows])
    data = br.forward_kinematics(m, q.cuda(), compute_frames=True)
    T, J = br.frame_jacobians(m, q.cuda(), ids, reference=reference)
    host = lambda x: x.cpu().double().numpy()[rows]  # noqa: E731
    oMf = K.frame_placements(m64, oMi)
    for got, ref in ((data.joint_pose_world, oMi), (data.joint_pose_local, liMi), (data.frame_pose_world, oMf),
                     (T, oMf[:, ids])):
        got = host(got)
        assert np.abs(got[..., :3] - ref[..., :3]).max() <= 1e-5
        assert np.minimum(np.abs(got[..., 3:] - ref[..., 3:]), np.abs(got[..., 3:] + ref[..., 3:])).max() <= 1e-5
    _jac_close(host(J), np.stack([K.frame_jacobian(m64, oMi, q.double().numpy()[rows], f, reference) for f in ids], 1))


def test_jacobians_beyond_l2():
    """The same configurations in a batch whose Jacobians exceed L2 and in one whose do not."""
    m = syn.model_from_spec(syn.humanoid_spec())
    ids = syn.op_frame_ids(m)
    B = 2 * torch.cuda.get_device_properties(0).L2_cache_size // (len(ids) * 6 * m.nv * 4)
    q = syn.random_q(m, B, 3).float().cuda()
    T, J = br.frame_jacobians(m, q, ids)
    for rows in (slice(0, 257), slice(B - 257, B)):
        t, j = br.frame_jacobians(m, q[rows], ids)
        assert (T[rows] - t).abs().max() <= 2e-5
        _jac_close(J[rows].cpu().numpy(), j.cpu().numpy(), 2.0)


@pytest.mark.parametrize("reference", ["world", "local_world_aligned", "local"])
def test_kernels_agree_to_the_bit(reference):
    """A batch whose Jacobians exceed L2 (staged records) against its rows in a small one (registers): the same
    bits, so that a problem made from a placement does not depend on the batch it was computed in."""
    m = syn.model_from_spec(syn.humanoid_spec())
    ids = syn.op_frame_ids(m)
    B = 2 * torch.cuda.get_device_properties(0).L2_cache_size // (len(ids) * 6 * m.nv * 4)
    q = syn.random_q(m, B, 4).float().cuda()
    T, J = br.frame_jacobians(m, q, ids, reference=reference)
    t, j = br.frame_jacobians(m, q[:513], ids, reference=reference)
    assert torch.equal(T[:513], t) and torch.equal(J[:513], j)
