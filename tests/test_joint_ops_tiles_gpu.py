"""``integrate`` / ``difference`` at the edges of a warp's tile (32 configurations) and a CTA's share (256), for
every joint kind, with 16-byte aligned and unaligned rows, against the float64 oracle.

The joints of one lane are computed in float64 and rounded once; the others are one float32 operation on
values below 8: an error of half a unit in the last place, 4.8e-7, and as much again for the oracle's
comparison in the rounded inputs' units.
"""

import numpy as np
import pytest
import torch

from betterrobot_b200 import configuration, synthetic as syn
from oracle import kinematics as K

pytestmark = pytest.mark.gpu

SPECS = {"chain7": syn.chain_spec, "humanoid": syn.humanoid_spec, "dual_arm": syn.dual_arm_spec,
         "mixed": syn.mixed_spec}
TOL = 1e-6


def _rows(x, aligned: bool):
    x = x.float()
    if aligned:
        return x.cuda()
    buf = torch.empty(x.numel() + 1, device="cuda")
    buf[1:] = x.reshape(-1).cuda()
    return buf[1:].view(x.shape)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("B", [1, 31, 33, 255, 256, 257, 513])
@pytest.mark.parametrize("name", list(SPECS))
def test_tile_edges(name, B, aligned):
    m = syn.model_from_spec(SPECS[name]())
    m64 = syn.model_from_spec(SPECS[name](), dtype=torch.float64)
    q = syn.random_q(m64, B, B).float()
    g = torch.Generator().manual_seed(B)
    v = torch.randn(B, m.nv, generator=g) * 10.0 ** (-6.0 * torch.rand(B, 1, generator=g))  # |v| from 1e-6 to 1
    v[0] = 0.0
    moved = configuration.integrate(m, _rows(q, aligned), _rows(v, aligned))
    ref = K.integrate(m64, q.double().numpy(), v.double().numpy())
    assert np.abs(moved.cpu().double().numpy() - ref).max() <= TOL * max(1.0, np.abs(ref).max() / 8.0)
    back = configuration.difference(m, _rows(q, aligned), _rows(moved, aligned))
    ref = K.difference(m64, q.double().numpy(), moved.cpu().double().numpy())
    assert np.abs(back.cpu().double().numpy() - ref).max() <= TOL * max(1.0, np.abs(ref).max() / 8.0)
