"""A trajectory's result does not depend, to the bit, on how many others are solved with it: alone a block
of 256 threads takes it, among more trajectories than SMs one of 128."""

import pytest
import torch

import betterrobot_b200 as br
from betterrobot_b200 import synthetic as syn, trajopt as btr

pytestmark = pytest.mark.gpu
SPECS = {"chain7": syn.chain_spec, "chain20": lambda: syn.chain_spec(n=20, name="chain20"), "dual_arm": syn.dual_arm_spec,
         "floating": syn.floating_chain_spec, "mixed": syn.mixed_spec, "humanoid": syn.humanoid_spec}


@pytest.mark.parametrize("robot,T", [("chain7", 3), ("chain7", 9), ("chain7", 10), ("chain7", 64), ("chain20", 12),
                                     ("dual_arm", 40), ("floating", 33), ("mixed", 17), ("humanoid", 8),
                                     ("humanoid", 14)])
@pytest.mark.parametrize("optimizer", ["gn", "lm"])
def test_alone_and_among_many(robot, T, optimizer):
    m, m64 = syn.model_from_spec(SPECS[robot]()), syn.model_from_spec(SPECS[robot](), dtype=torch.float64)
    fid, N = syn.op_frame_ids(m)[0], torch.cuda.get_device_properties(0).multi_processor_count + 92
    qs = syn.random_q(m64, N, 61, rev_range=1.0)
    qg = syn.noisy_start(m64, qs, 0.4, 62).float().cuda()
    qs = qs.float().cuda()
    pose = lambda q: br.forward_kinematics(m, q, compute_frames=True).frame_pose_world[:, fid].contiguous()  # noqa: E731
    goal, start = pose(qg), pose(qs)
    X0 = qs[:, None].expand(-1, T, -1).contiguous()
    cfg = btr.TrajOptConfig(max_iter=12, optimizer=optimizer)
    solve = lambda s: btr.solve_trajopt_batched(m, fid, goal[s], X0[s], start=start[s], cfg=cfg)  # noqa: E731
    many = solve(slice(0, N))
    assert bool(torch.isfinite(many.cost).all())
    for at in range(0, N, 60):
        few = solve(slice(at, at + 60))
        for name in ("iters", "status", "q", "cost", "goal_grad"):
            a, b = getattr(many, name)[at:at + 60], getattr(few, name)
            assert torch.equal(a, b), (name, at, float((a.double() - b.double()).abs().max()))
