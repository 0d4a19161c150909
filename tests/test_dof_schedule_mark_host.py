"""A table says that it has a row section, and how long it is, inside its entry section: a reader finds
out without looking past the end of a table that ends there."""

import numpy as np
import pytest

from test_dof_row_schedule_host import _rows, _trees
from test_dof_schedule_host import _contribs, _decode, _schedule, _tree

MARK = 0x5752ffff  # BR_DOF_SCHED_MARK


@pytest.mark.parametrize("name", sorted(_trees()))
def test_mark_and_length(name):
    s = _schedule(_trees()[name])
    dp = _trees()[name]
    _, _, starts, tasks, extra = _decode(s)
    assert tuple(extra[-1]) == (MARK, len(s))
    ntr = _rows(s)[4]
    starts_r, tasks_r, extra_r = _rows(s)[:3]
    end = len(s) - len(extra_r) - 4 * len(tasks_r) - (len(dp) - ntr if ntr else 0)
    assert end % 4 == 0                                     # (the row tasks start there)
    # no contribution looks like the mark, and no task reaches it
    zoff = _tree(dp)[2][len(dp)]
    assert (extra[:-1, 0] != MARK).all() and zoff + len(dp) < 0xffff
    assert all((t[2] >> 16) + (t[0] >> 16) <= len(extra) - 1 for t in tasks)
    assert sum(len(_contribs(t, extra)) for t in tasks) == len(tasks) + len(extra) - 1
