"""The loss is the same number, to the bit, whether or not a gradient is computed with it, in every mode."""

import numpy as np
import pytest
import torch

from betterrobot_b200 import synthetic as syn
from betterrobot_b200.adjoint import pose_loss

pytestmark = pytest.mark.gpu
SPECS = {"chain7": syn.chain_spec, "humanoid": syn.humanoid_spec, "dual_arm": syn.dual_arm_spec, "mixed": syn.mixed_spec}


@pytest.mark.parametrize("robot", sorted(SPECS))
@pytest.mark.parametrize("B", [5, 300, 20_011])  # the warp kernel twice, the lane kernel
@pytest.mark.parametrize("per_cfg", [False, True])
def test_same_loss_with_and_without_gradient(robot, B, per_cfg):
    m, m64 = syn.model_from_spec(SPECS[robot]()), syn.model_from_spec(SPECS[robot](), dtype=torch.float64)
    fids = syn.op_frame_ids(m)
    q = syn.random_q(m64, B, 51, rev_range=2.5, base_translation=1.0).float().cuda()
    T = syn.random_targets(B, len(fids), 52).float().cuda()      # rotation errors up to pi
    near = B // 2                                                # and small ones
    from betterrobot_b200.kinematics import frame_jacobians
    T[:near] = frame_jacobians(m, q[:near] + 1e-4, fids, check_quaternion=False)[0]
    w = torch.from_numpy(np.random.default_rng(53).uniform(0.5, 2, (B, len(fids)) if per_cfg else len(fids))).float().cuda()
    with torch.no_grad():
        alone = pose_loss(m, q, fids, T, w)
    for mode in ("auto", "store", "recompute"):
        got = pose_loss(m, q.clone().requires_grad_(True), fids, T, w, mode=mode).detach()
        assert torch.equal(got, alone), (mode, float((got - alone).abs().max()))
