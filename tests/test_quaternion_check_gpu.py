"""The free-flyer quaternion check of the public calls: a norm off by more than 0.1 anywhere raises, as
the same comparison on float32 tensors does; whatever the strides, and call after call."""

import pytest
import torch

import betterrobot_b200 as br
from betterrobot_b200 import synthetic as syn
from betterrobot_b200.exceptions import QuaternionNormError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 31, 257, 70001])
def test_bad_row_anywhere(B):
    m = syn.model_from_spec(syn.humanoid_spec())
    q = syn.random_q(m, B, 1).float().cuda()
    br.forward_kinematics(m, q)
    for row in sorted({0, B // 2, B - 1}):
        for scale in (0.89, 1.11):
            bad = q.clone()
            bad[row, 3:7] *= scale
            with pytest.raises(QuaternionNormError):
                br.forward_kinematics(m, bad)
            with pytest.raises(QuaternionNormError):  # a strided view of the same
                br.frame_jacobians(m, torch.cat([bad, bad], -1)[:, :m.nq], [0], check_quaternion=True)
            br.forward_kinematics(m, bad, check_quaternion=False)
    fine = q.clone()
    fine[0, 3:7] *= 1.09
    br.forward_kinematics(m, fine)
    fine[0, 3] = float("nan")  # not a norm further than the tolerance
    br.forward_kinematics(m, fine)
