"""Level-schedule tables that this library did not write: refused problem by problem (status flag BADTREE,
x = x0) from what they hold, without a read past their end."""

import numpy as np
import pytest
import torch

from betterrobot_b200 import ik as bik, synthetic as syn
from betterrobot_b200.tree import TreeArrays

pytestmark = pytest.mark.gpu
BADTREE = 4  # BR_IK_FLAG_BADTREE


def _entry_words(s):
    nlev, ntask, nextra = (int(v) for v in s[:3])
    return ((5 + nlev + 3) & ~3) + 4 * ntask + 2 * nextra


def _entries_only(s):
    """The table as a library without a row section wrote it: its last word is its last contribution's."""
    old = s[:_entry_words(s) - 2].copy()
    old[2] -= 1
    return old


def _other_length(s):
    t = s.copy()
    t[_entry_words(s) - 1] += 4
    return t


def _cut_before_rows(s):
    t = s[:_entry_words(s)].copy()
    t[-1] = len(t)                                        # honest about it
    return t


@pytest.mark.parametrize("robot", ["chain7", "humanoid", "dual_arm"])
@pytest.mark.parametrize("change", [_entries_only, _other_length, _cut_before_rows])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_refused(robot, change, precision):
    spec = {"chain7": syn.chain_spec, "humanoid": syn.humanoid_spec, "dual_arm": syn.dual_arm_spec}[robot]()
    m = syn.model_from_spec(spec)
    fid, P = syn.op_frame_ids(m)[0], 40
    pk = bik.PackedIK([m], [np.full((P, 1), fid, np.int32)], [np.ones(P, np.int32)])
    q0 = m.q_neutral.float().repeat(P, 1).cuda()
    T = torch.zeros(P, 1, 7, device="cuda")
    T[..., 0], T[..., 6] = 0.2, 1.0
    pk.set_inputs([T], [q0])
    settings = bik.settings_from(bik.IKCostConfig(), bik.OptimizerConfig(max_iter=5, precision=precision))
    good = pk._trees[0].dof_sched
    table = torch.from_numpy(change(TreeArrays(m).dof_schedule()).view(np.int32)).cuda()
    pk._trees[0].dof_sched = table.data_ptr()
    pk.solve(settings)
    assert (((pk.status.cpu() >> 8) & BADTREE) != 0).all() and torch.equal(pk.q_of(0), q0)
    pk._trees[0].dof_sched = good
    pk.solve(settings)
    assert (((pk.status.cpu() >> 8) & BADTREE) == 0).all()
