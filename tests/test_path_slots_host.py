"""The bound on waiting wrenches leaves frame lists that the entry point refuses to the entry point."""

import pytest

from betterrobot_b200 import synthetic as syn
from betterrobot_b200.adjoint import path_slots
from betterrobot_b200.tree import TreeArrays


@pytest.mark.parametrize("ids", [(), (44,), (0, 1000), (-1,)])
def test_bad_frame_lists_have_no_bound(ids):
    arrays = TreeArrays(syn.model_from_spec(syn.humanoid_spec()))
    assert arrays.nf == 44 and path_slots(arrays, ids) == -1
    assert ids not in arrays.path_slots


def test_good_lists_keep_theirs():
    arrays = TreeArrays(syn.model_from_spec(syn.humanoid_spec()))
    assert path_slots(arrays, (0,)) == 0 and path_slots(arrays, tuple(range(44))) > 0
