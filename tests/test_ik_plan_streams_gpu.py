"""A ``PackedIK`` plan is complete when its constructor returns, whatever stream it was built on."""

import numpy as np
import pytest
import torch

from betterrobot_b200 import synthetic as syn
from betterrobot_b200.ik import IKCostConfig, OptimizerConfig, PackedIK, settings_from

pytestmark = pytest.mark.gpu


def _plan():
    specs, n = [syn.chain_spec(), syn.humanoid_spec()], [70, 33]
    models = [syn.model_from_spec(s) for s in specs]
    fids = [np.tile(np.array(syn.op_frame_ids(m)[:2] * 2, np.int32)[:2], (k, 1)) for m, k in zip(models, n)]
    kinds = [None, ["pose", "position"]]
    return PackedIK(models, fids, [np.full(k, 2, np.int32) for k in n], target_kinds=kinds)


def _inputs(pk):
    g = torch.Generator().manual_seed(3)
    T = [torch.zeros(n, 2, 7) for n in pk.counts]
    for t in T:
        t[..., :3] = 0.3 * torch.rand(t.shape[:2] + (3,), generator=g)
        t[..., 6] = 1.0
    return [t.cuda() for t in T], [m.q_neutral.float().repeat(n, 1).cuda() for m, n in zip(pk.models, pk.counts)]


def test_built_on_a_busy_stream_solved_on_another():
    settings = settings_from(IKCostConfig(), OptimizerConfig(max_iter=8))
    ref = _plan()
    T, q0 = _inputs(ref)
    ref.set_inputs(T, q0)
    ref.solve(settings)
    torch.cuda.synchronize()
    build, solve = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(build):
        torch.cuda._sleep(200_000_000)  # ~0.1 s ahead of the upload
        pk = _plan()
    assert build.query(), "the plan was handed out before its tables had arrived"
    with torch.cuda.stream(solve):
        pk.set_inputs(T, q0)
        pk.solve(settings)
    solve.synchronize()
    for name in ("order", "items", "n_targets_t", "frames_t", "q_offset", "r_offset", "kinds", "q_rest"):
        assert torch.equal(getattr(pk, name), getattr(ref, name)), name
    assert torch.equal(pk.x, ref.x) and torch.equal(pk.verdict, ref.verdict)
    # the raw stream handle that solve() takes
    pk.x.zero_()
    torch.cuda.synchronize()
    pk.solve(settings, stream=solve.cuda_stream)
    solve.synchronize()
    assert torch.equal(pk.x, ref.x)
