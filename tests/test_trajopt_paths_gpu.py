"""GPU parity of the trajectory solver at the edges of its dispatch, against the float64 oracle.

Few interior knots (the plain band elimination, T < 10) and many (twisted), one CTA of 256 threads per
trajectory (no more trajectories than SMs, or a working set above half an SM's shared memory) and of
128, boundary systems inside one warp's rows and beyond them, every trial update path of the dense
factorization (one entry per thread, 4 x 4 tiles).  Bars as in ``test_trajopt_gpu.py``: trajectories
within 1e-4, costs within 1e-6 + 1e-4 relative, where both converged (goals 0.2 rad away: all do).
"""

import numpy as np
import pytest
import torch

from betterrobot_b200 import synthetic as syn, trajopt as btr
from oracle import kinematics as K, trajopt as ot

pytestmark = pytest.mark.gpu
SPECS = {"chain7": (syn.chain_spec, "ee"), "dual_arm": (syn.dual_arm_spec, "ee_l"),
         "floating": (syn.floating_chain_spec, "ee"), "mixed": (syn.mixed_spec, "ee"),
         "chain20": (lambda: syn.chain_spec(n=20, name="chain20"), "ee"),
         "humanoid": (syn.humanoid_spec, "track0")}


@pytest.mark.parametrize("name,T,many", [("chain7", 3, False), ("chain7", 9, True), ("chain7", 10, False),
                                         ("chain7", 33, True), ("dual_arm", 11, True), ("floating", 10, True),
                                         ("mixed", 9, False), ("chain20", 12, False), ("humanoid", 11, False)])
def test_against_oracle(name, T, many):
    spec, frame = SPECS[name][0](), SPECS[name][1]
    m, m64 = syn.model_from_spec(spec), syn.model_from_spec(spec, dtype=torch.float64)
    fid, N = m.frame_id(frame), 3
    qs, qg = syn.trajopt_endpoints(m64, N, 17, 0.2)
    qs = qs.float().double()
    pose = lambda q: K.frame_placements(m64, K.forward_kinematics(m64, q.numpy())[0], [fid])[:, 0].astype(np.float32)  # noqa: E731
    goal, start = pose(qg), pose(qs)
    X0 = np.repeat(qs.numpy()[:, None], T, 1)
    ref = ot.solve(m64, X0, fid, goal.astype(float), start.astype(float), ot.TrajSettings(max_iter=30))
    reps = -(-2 * torch.cuda.get_device_properties(0).multi_processor_count // N) if many else 1
    dev = lambda a: torch.from_numpy(np.tile(a, (reps,) + (1,) * (a.ndim - 1))).float().cuda()  # noqa: E731
    out = btr.solve_trajopt_batched(m, fid, dev(goal), dev(X0), start=dev(start), cfg=btr.TrajOptConfig(max_iter=30))
    X, cost = out.q.cpu().double().numpy(), out.cost.cpu().double().numpy()
    both = out.converged.cpu().numpy()[:N] & ref.converged
    assert both.sum() >= N - 1
    np.testing.assert_array_equal(X.reshape(reps, N, T, -1), np.broadcast_to(X[:N], (reps, N) + X.shape[1:]))
    assert np.abs(X[:N][both] - ref.X[both]).max() <= 1e-4
    np.testing.assert_allclose(cost[:N][both], ref.cost[both], rtol=1e-4, atol=1e-6)
