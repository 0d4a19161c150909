"""Frame lists that the pose loss refuses are refused alike with and without a gradient."""

import pytest
import torch

from betterrobot_b200 import synthetic as syn
from betterrobot_b200.adjoint import pose_loss
from betterrobot_b200.exceptions import KernelError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["auto", "store", "recompute"])
@pytest.mark.parametrize("ids", [(), (44,), (0, 1000), (-1,), (0,) * 65])
def test_bad_frame_lists(ids, mode):
    m = syn.model_from_spec(syn.humanoid_spec())
    assert m.nframes == 44
    q = m.q_neutral.float().repeat(3, 1).cuda()
    T, w = torch.zeros(3, len(ids), 7, device="cuda"), torch.ones(len(ids), device="cuda")
    T[..., 6] = 1.0
    with torch.no_grad(), pytest.raises(KernelError):
        pose_loss(m, q, ids, T, w, mode=mode)
    with pytest.raises(KernelError):
        pose_loss(m, q.requires_grad_(True), ids, T, w, mode=mode)
