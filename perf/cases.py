"""The work that users of ``betterrobot_b200`` have it do, as measurable cases.

Every case is one pass through public entry points on inputs made from a seed:

* ``ik_single``        one ``solve_ik`` call, the drop-in call of an interactive or control program;
* ``ik_batch``         ``solve_ik_batched`` on one robot, with its precision and robust-kernel options;
* ``ik_mix``           a kept ``PackedIK`` plan over an uneven mix of robots, re-solved with new inputs;
* ``fk_joint_jac``     ``forward_kinematics`` with frames, then ``compute_joint_jacobians`` on its result;
* ``frame_jac``        the fused ``frame_jacobians``;
* ``pose_loss``        forward and backward of the differentiable pose loss;
* ``trajopt``          ``solve_trajopt_batched``;
* ``configuration``    ``integrate`` and ``difference``;
* ``lie``              a chain of batched SE3 primitives.

Robots are the seeded synthetic ones of ``betterrobot_b200.synthetic`` (a 7-revolute chain, a
14-revolute dual arm, a 36-DOF floating-base humanoid).  The helpers below are a plain float64
torch restatement of the kinematics; inputs that need it (target poses) and the exact values come
from them and never from the kernels.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import betterrobot_b200 as br
from betterrobot_b200 import configuration, ik, lie, synthetic, trajopt
from betterrobot_b200.adjoint import pose_loss

DEV = "cuda"
SPECS = {"chain7": synthetic.chain_spec, "dual_arm": synthetic.dual_arm_spec, "humanoid": synthetic.humanoid_spec}
# frames that IK problems draw their targets from
IK_FRAMES = {
    "humanoid": [f"track{i}" for i in range(6)],
    "dual_arm": ["ee_l", "ee_r", "body_l_link5", "body_r_link5", "body_l_link3", "body_r_link3"],
    "chain7": ["ee", "body_link7", "body_link6", "body_link5", "body_link4", "body_link3"],
}


# --------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # the smallest calls: one arm, one configuration, one target, as a control loop makes them
        {"name": "frame_jac_chain7_1", "kind": "frame_jac", "robot": "chain7", "batch": 1, "reference": "local"},
        {"name": "ik_single_chain7", "kind": "ik_single", "robot": "chain7"},
        # a humanoid batch solved with the float64 normal equations (the reference's own iterates)
        {"name": "ik_humanoid_301_f64", "kind": "ik_batch", "robot": "humanoid", "batch": 301, "targets": 4,
         "precision": "f64", "kernel": "l2"},
        # the benchmark's uneven mix of robots, 1 to 6 targets each, on a kept plan
        {"name": "ik_mix_8192", "kind": "ik_mix", "batch": 8192},
        # placements, frames and all joint Jacobians of a batch, the usual call sequence
        {"name": "fk_joint_jac_humanoid_16001", "kind": "fk_joint_jac", "robot": "humanoid", "batch": 16001},
        # the benchmark's fused FK + Jacobians at twelve frames
        {"name": "frame_jac_humanoid_65536", "kind": "frame_jac", "robot": "humanoid", "batch": 65536,
         "reference": "local_world_aligned"},
        # a training step's loss and gradient: an ordinary batch, and the largest
        {"name": "pose_loss_humanoid_16384", "kind": "pose_loss", "robot": "humanoid", "batch": 16384,
         "per_config": False},
        {"name": "pose_loss_humanoid_262144", "kind": "pose_loss", "robot": "humanoid", "batch": 262144,
         "per_config": True},
        # trajectory optimisation: the benchmark's arm batch, and whole-body trajectories
        {"name": "trajopt_chain7_256x64", "kind": "trajopt", "robot": "chain7", "batch": 256, "knots": 64},
        {"name": "trajopt_humanoid_33x40", "kind": "trajopt", "robot": "humanoid", "batch": 33, "knots": 40},
        # retraction and difference of a large sample set (a filter's or a sampler's update)
        {"name": "configuration_humanoid_999999", "kind": "configuration", "robot": "humanoid", "batch": 999999},
        # relative pose errors and the step that undoes them, element by element
        {"name": "lie_chain_2m", "kind": "lie", "batch": (1 << 21) + 3},
    ]


def draw(rng) -> dict:
    """One more case of the same ranges: every kind, all robots, sizes spread over their logarithm."""
    def size(lo: int, hi: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ik_single", "ik_batch", "ik_mix", "fk_joint_jac", "frame_jac", "frame_jac", "pose_loss",
                       "pose_loss", "trajopt", "configuration", "lie"])
    robot = rng.choice(sorted(SPECS))
    if kind == "ik_single":  # one call is one size: robot, targets and limit weight vary
        return {"kind": kind, "robot": robot, "targets": rng.randint(1, 3), "limit_scale": rng.choice([0.5, 1.0, 2.0])}
    if kind == "ik_batch":
        return {"kind": kind, "robot": robot, "batch": size(2, 4096 if robot != "humanoid" else 600),
                "targets": rng.randint(1, 6), "precision": rng.choice(["f32", "f32", "f64"]),
                "kernel": rng.choice(["l2", "l2", "huber", "cauchy"])}
    if kind == "ik_mix":
        return {"kind": kind, "batch": size(16, 8192)}
    if kind == "fk_joint_jac":
        return {"kind": kind, "robot": robot, "batch": size(1, 16001)}
    if kind == "frame_jac":
        return {"kind": kind, "robot": robot, "batch": size(1, 65536),
                "reference": rng.choice(["world", "local_world_aligned", "local"])}
    if kind == "pose_loss":
        return {"kind": kind, "robot": robot, "batch": size(16, 262144), "per_config": rng.choice([False, True])}
    if kind == "trajopt":
        top = 33 if robot == "humanoid" else 256
        return {"kind": kind, "robot": robot, "batch": size(1, top), "knots": rng.randint(16, 40 if robot == "humanoid" else 64)}
    if kind == "configuration":
        return {"kind": kind, "robot": robot, "batch": size(16, 999999)}
    return {"kind": kind, "batch": size(16, (1 << 21) + 3)}


# --------------------------------------------------------------------------- plain float64 kinematics
@functools.lru_cache(maxsize=None)
def _model(robot: str):
    return synthetic.model_from_spec(SPECS[robot]())


def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def _qrot(q, p):
    u, w = q[..., :3], q[..., 3:]
    u, p = torch.broadcast_tensors(u, p)
    return p + 2.0 * torch.linalg.cross(u, torch.linalg.cross(u, p, dim=-1) + w * p, dim=-1)


def _conj(q):
    return torch.cat([-q[..., :3], q[..., 3:]], -1)


def _unit(q):
    return q / q.norm(dim=-1, keepdim=True)


def _compose(a, b):
    return a[0] + _qrot(a[1], b[0]), _qmul(a[1], b[1])


def _inverse(a):
    c = _conj(a[1])
    return -_qrot(c, a[0]), c


def _pose(t):
    return t[..., :3], t[..., 3:]


def _exp_q(w):
    th = w.norm(dim=-1, keepdim=True)
    return torch.cat([0.5 * torch.sinc(th / (2.0 * math.pi)) * w, torch.cos(0.5 * th)], -1)


def _exp(v, w):
    th2 = (w * w).sum(-1, keepdim=True)
    th = th2.clamp_min(1e-30).sqrt()
    small = th2 < 1e-4
    b = torch.where(small, 0.5 - th2 / 24 + th2 * th2 / 720, (1 - torch.cos(th)) / th2.clamp_min(1e-30))
    c = torch.where(small, 1 / 6 - th2 / 120 + th2 * th2 / 5040, (th - torch.sin(th)) / (th2 * th).clamp_min(1e-30))
    wv = torch.linalg.cross(w, v, dim=-1)
    return v + b * wv + c * torch.linalg.cross(w, wv, dim=-1), _exp_q(w)


def _log(a):
    t, q = a
    q = torch.where(q[..., 3:] < 0, -q, q)
    s2 = (q[..., :3] ** 2).sum(-1, keepdim=True)
    s = s2.clamp_min(1e-30).sqrt()
    half = torch.atan2(s, q[..., 3:])
    small = s2 < 1e-8
    w = torch.where(small, 2.0 + s2 / 3.0, 2.0 * half / s) * q[..., :3]
    th2 = (w * w).sum(-1, keepdim=True)
    c = torch.where(small, 1 / 12 + th2 / 720, (1.0 - half * q[..., 3:] / s) / (4.0 * half * half).clamp_min(1e-30))
    wt = torch.linalg.cross(w, t, dim=-1)
    return t - 0.5 * wt + c * torch.linalg.cross(w, wt, dim=-1), w


def _axis(jm, ref):
    named = {"x": (1.0, 0.0, 0.0), "y": (0.0, 1.0, 0.0), "z": (0.0, 0.0, 1.0)}
    a = named[jm.kind[-1]] if jm.kind[-1] in named else jm.axis.tolist()
    return torch.tensor(a, dtype=ref.dtype, device=ref.device)


def _fk(m, q):
    """World and parent-relative placements ``[(t, quat)]`` of every joint at ``q (B, nq)`` float64."""
    place = m.joint_placements.double().to(q.device)
    world, local = [], []
    for j, jm in enumerate(m.joint_models):
        T = tuple(x.expand(q.shape[0], -1) for x in _pose(place[j]))
        iq = m.idx_qs[j]
        if jm.kind == "free_flyer":
            T = _compose(T, (q[:, iq:iq + 3], _unit(q[:, iq + 3:iq + 7])))
        elif jm.kind.startswith("revolute"):
            h = 0.5 * q[:, iq:iq + 1]
            T = (T[0], _qmul(T[1], torch.cat([torch.sin(h) * _axis(jm, q), torch.cos(h)], -1)))
        local.append(T)
        world.append(T if m.parents[j] < 0 else _compose(world[m.parents[j]], T))
    return world, local


def _frame(m, world, f):
    place = m.frames[f].joint_placement.double().to(world[0][0].device)
    return _compose(world[m.frames[f].parent_joint], tuple(x.expand(world[0][0].shape[0], -1) for x in _pose(place)))


def _cat(poses):
    return torch.stack([torch.cat(p, -1) for p in poses], 1)


def _jacobian(m, world, joint, pose, reference, out):
    """Columns of the Jacobian of a frame at ``pose`` carried by ``joint``, into ``out (B, 6, nv)``."""
    sup = m.supports[joint]
    for j in sup:
        jm, iv = m.joint_models[j], m.idx_vs[j]
        t, q = world[j]
        eye = torch.eye(3, dtype=t.dtype, device=t.device)
        if jm.kind == "free_flyer":
            cols = [(k, eye[k], False) for k in range(3)] + [(3 + k, eye[k], True) for k in range(3)]
        elif jm.nv == 1:
            cols = [(0, _axis(jm, t), True)]
        else:
            cols = []
        for k, ax, rot in cols:
            a = _qrot(q, ax)
            lin, ang = a, torch.zeros_like(a)
            if rot:
                ang = a
                lin = (torch.linalg.cross(t, a, dim=-1) if reference == "world"
                       else torch.linalg.cross(a, pose[0] - t, dim=-1))
            if reference == "local":
                c = _conj(pose[1])
                lin, ang = _qrot(c, lin), _qrot(c, ang)
            out[:, :3, iv + k], out[:, 3:, iv + k] = lin, ang


# --------------------------------------------------------------------------- inputs
def _gen(seed: int):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, r):
    return (2.0 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) - 1.0) * r


def _normal(g, shape, s=1.0):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64) * s


def _random_q(m, n, g, base=1.0):
    """Configurations inside the limits (revolute within 2.5 rad, a free base within ``base`` m, any attitude)."""
    q = _uniform(g, (n, m.nq), 2.5)
    if m.joint_models[1].kind == "free_flyer":
        q[:, :3] *= base / 2.5
        q[:, 3:7] = _unit(_normal(g, (n, 4)))
    return q


def _moved(m, q, sigma, g):
    """``q`` moved by N(0, sigma^2) rad per joint (a third of that in metres for a free base), inside the limits."""
    d = _normal(g, q.shape, sigma)
    out = q + d
    if m.joint_models[1].kind == "free_flyer":
        out[:, :3] = q[:, :3] + d[:, :3] / 3.0
        out[:, 3:7] = _qmul(q[:, 3:7], _exp_q(d[:, 3:6]))
    lim = m.upper_pos_limit.double().to(DEV), m.lower_pos_limit.double().to(DEV)
    return torch.maximum(torch.minimum(out, lim[0]), lim[1])


def _frame_poses(m, q, ids):
    world, _ = _fk(m, q)
    return _cat([_frame(m, world, f) for f in ids])


def _op_frames(m):
    return synthetic.op_frame_ids(m)


def _ik_problems(robot, n, k, g, rng):
    """Frames ``(n, k)``, target poses at a hidden configuration, and a start 0.3 rad per joint away from it."""
    m = _model(robot)
    cand = np.array([m.frame_id(f) for f in IK_FRAMES[robot]], np.int32)
    q_star = _random_q(m, n, g, 0.5)
    q0 = _moved(m, q_star, 0.3, g)
    poses = _frame_poses(m, q_star, cand.tolist())
    pick = np.stack([rng.permutation(6)[:k] for _ in range(n)])
    at = torch.from_numpy(pick).to(DEV)
    targets = torch.gather(poses, 1, at[..., None].expand(-1, -1, 7))
    return cand[pick], targets.float().contiguous(), q0.float().contiguous()


def _ik_options(precision="f32", kernel="l2"):
    return (ik.IKCostConfig(rest_weight=1e-3, limit_weight=0.1),
            ik.OptimizerConfig(max_iter=100, lam0=1e-3, factor=10.0, tol=1e-6, precision=precision, kernel=kernel))


def prepare(case: dict, seed: int) -> dict:
    kind, g, rng = case["kind"], _gen(seed), np.random.default_rng(seed)
    s = {"kind": kind}
    if kind == "lie":
        n = case["batch"]
        a = torch.cat([_uniform(g, (n, 3), 1.0), _unit(_normal(g, (n, 4)))], -1)
        w = _unit(_normal(g, (n, 3))) * (torch.rand((n, 1), generator=g, device=DEV, dtype=torch.float64) * 2.5)
        b = torch.cat(_compose(_pose(a), _exp(_uniform(g, (n, 3), 0.5), w)), -1)
        return s | {"a": a.float(), "b": b.float()}
    if kind == "ik_mix":
        # the benchmark's shares: 40 % arms, 30 % dual arms, 30 % humanoids, 1 to 6 targets each
        n = case["batch"]
        counts = {"humanoid": n - int(round(0.4 * n)) - int(round(0.3 * n)), "dual_arm": int(round(0.3 * n)),
                  "chain7": int(round(0.4 * n))}
        made = {r: _ik_problems(r, c, 6, g, rng) for r, c in counts.items()}
        cost, opt = _ik_options()
        plan = ik.PackedIK([_model(r) for r in counts], [made[r][0] for r in counts],
                           [rng.integers(1, 7, size=c).astype(np.int32) for c in counts.values()], device=DEV)
        return s | {"plan": plan, "targets": [made[r][1] for r in counts], "q0": [made[r][2] for r in counts],
                    "settings": ik.settings_from(cost, opt)}
    m = _model(case["robot"])
    s["model"] = m
    if kind == "ik_single":
        k = case.get("targets", 1)
        frames, targets, q0 = _ik_problems(case["robot"], 1, k, g, rng)
        names = [m.frame_names[f] for f in frames[0]]
        return s | {"targets": dict(zip(names, targets[0])), "q0": q0[0],
                    "cost": ik.IKCostConfig(limit_weight=0.1 * case.get("limit_scale", 1.0))}
    if kind == "ik_batch":
        frames, targets, q0 = _ik_problems(case["robot"], case["batch"], case["targets"], g, rng)
        cost, opt = _ik_options(case["precision"], case["kernel"])
        return s | {"frames": frames, "targets": targets, "q0": q0, "cost": cost, "opt": opt}
    n = case["batch"]
    if kind == "trajopt":
        # trajectories that start at rest in one configuration, with the goal pose of one 0.15 rad per
        # joint away: an arm's point-to-point motion, a humanoid's reach (further goals make undamped
        # Gauss-Newton oscillate on some of them, and its end point is then a matter of rounding)
        f = _op_frames(m)[0]
        qs = _random_q(m, n, g, 0.5)
        qg = _moved(m, qs, 0.15, g)
        return s | {"frame": f, "goal": _frame_poses(m, qg, [f])[:, 0].float().contiguous(),
                    "start": _frame_poses(m, qs, [f])[:, 0].float().contiguous(),
                    "x0": qs.float()[:, None].expand(-1, case["knots"], -1).contiguous(),
                    "cfg": trajopt.TrajOptConfig(max_iter=30)}
    q = _random_q(m, n, g)
    s["q"] = q.float()
    if kind == "frame_jac":
        return s | {"frames": _op_frames(m), "reference": case["reference"]}
    if kind == "pose_loss":
        # tracking: targets at a configuration 0.2 rad per joint away
        ids = _op_frames(m)
        goal = torch.cat([_frame_poses(m, part, ids) for part in _moved(m, q, 0.2, g).split(32768)])
        w = 0.5 + 1.5 * torch.rand((n, len(ids)) if case["per_config"] else (len(ids),), generator=g, device=DEV)
        return s | {"q": q.float().requires_grad_(True), "frames": ids, "targets": goal.float(), "weights": w}
    if kind == "configuration":
        return s | {"v": _normal(g, (n, m.nv), 0.3).float()}
    return s


def run(s: dict):
    kind = s["kind"]
    if kind == "frame_jac":
        T, J = br.frame_jacobians(s["model"], s["q"], s["frames"], reference=s["reference"])
        return {"poses": T, "jacobians": J}
    if kind == "fk_joint_jac":
        d = br.forward_kinematics(s["model"], s["q"], compute_frames=True)
        br.compute_joint_jacobians(s["model"], d)
        return {"world": d.joint_pose_world, "local": d.joint_pose_local, "frames": d.frame_pose_world,
                "jacobians": d.joint_jacobians}
    if kind == "pose_loss":
        loss = pose_loss(s["model"], s["q"], s["frames"], s["targets"], s["weights"])
        grad, = torch.autograd.grad(loss.sum(), s["q"])
        return {"loss": loss.detach(), "grad": grad}
    if kind == "configuration":
        moved = configuration.integrate(s["model"], s["q"], s["v"])
        return {"moved": moved, "back": configuration.difference(s["model"], s["q"], moved)}
    if kind == "lie":
        rel = lie.se3_compose(lie.se3_inverse(s["a"]), s["b"])
        xi = lie.se3_log(rel)
        return {"rel": rel, "xi": xi, "again": lie.se3_compose(s["a"], lie.se3_exp(xi))}
    if kind == "ik_single":
        r = br.solve_ik(s["model"], s["targets"], initial_q=s["q0"], cost_cfg=s["cost"])
        return {"q": r.q, "residual": r.residual, "iters": r.iters, "converged": r.converged}
    if kind == "ik_batch":
        r = br.solve_ik_batched(s["model"], s["frames"], s["targets"], s["q0"], cost_cfg=s["cost"],
                                optimizer_cfg=s["opt"])
        return {"q": r.q, "cost": r.cost, "iters": r.iters, "converged": r.converged}
    if kind == "ik_mix":
        plan = s["plan"]
        plan.set_inputs(s["targets"], s["q0"])
        plan.solve(s["settings"])
        return {"q": plan.x, "cost": plan.cost, "iters": plan.iters, "status": plan.status}
    r = br.solve_trajopt_batched(s["model"], s["frame"], s["goal"], s["x0"], start=s["start"], cfg=s["cfg"])
    return {"q": r.q, "cost": r.cost, "iters": r.iters, "converged": r.converged, "goal_grad": r.goal_grad}


# --------------------------------------------------------------------------- what a pass cannot do without
def _lm_work(robot, n, k, iters):
    """Bytes and flops of ``n`` problems of ``k`` targets at ``iters`` iterations: forward kinematics,
    residuals and the tree-sparse normal equations and factorization of each."""
    m = _model(robot)
    depth = [0] * m.nv
    for j in range(m.njoints):
        for c in range(m.nvs[j]):
            depth[m.idx_vs[j] + c] = sum(m.nvs[i] for i in m.supports[j][:-1]) + c
    solve = sum(d * (d + 3) for d in depth) + 4 * sum(d + 1 for d in depth)
    col = max(depth) + 1
    per = 80 * m.njoints + k * (300 + 60 * col + 6 * col * (col + 1)) + solve
    return {"bytes": n * 4 * (2 * m.nq + 8 * k + 4), "flops": n * iters * per}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "lie":  # a, b in; rel, xi, again out
        return {"bytes": case["batch"] * 4 * (7 + 7 + 7 + 6 + 7), "flops": case["batch"] * 500}
    if kind == "ik_mix":
        n = case["batch"]
        parts = [_lm_work(r, share * n, 3.5, it) for r, share, it in
                 (("chain7", 0.4, 25), ("dual_arm", 0.3, 40), ("humanoid", 0.3, 80))]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    m = _model(case["robot"])
    if kind in ("ik_single", "ik_batch"):  # mean iteration counts of these problems, roughly
        return _lm_work(case["robot"], case.get("batch", 1), case.get("targets", 1),
                        {"chain7": 25, "dual_arm": 40, "humanoid": 80}[case["robot"]])
    n, f = case["batch"], len(_op_frames(m))
    if kind == "frame_jac":
        return {"bytes": n * 4 * (m.nq + f * 7 + f * 6 * m.nv), "flops": n * (80 * m.njoints + f * (80 + 15 * m.nv))}
    if kind == "fk_joint_jac":
        return {"bytes": n * 4 * (m.nq + 7 * (2 * m.njoints + m.nframes) + m.njoints * 6 * m.nv),
                "flops": n * (80 * (m.njoints + m.nframes) + m.njoints * 15 * m.nv)}
    if kind == "pose_loss":  # q, targets, weights in; loss and gradient out
        return {"bytes": n * 4 * (2 * m.nq + 7 * f + (f if case["per_config"] else 0) + 1),
                "flops": n * (80 * m.njoints + 450 * f + 40 * m.nv)}
    if kind == "configuration":
        return {"bytes": n * 4 * (3 * m.nq + 2 * m.nv), "flops": n * (4 * m.nv + 300)}
    t = case["knots"]  # about ten Gauss-Newton steps: bands per DOF, the dense boundary system, residuals
    per = t * m.nv * 70 + (2 * m.nv) ** 3 / 3 + 4 * (80 * m.njoints + 200 * m.nv)
    return {"bytes": n * 4 * (3 * t * m.nq + 7 * 2 + 6), "flops": n * 10 * per}


# --------------------------------------------------------------------------- exact values
def _exact_loss(m, q, ids, targets, weights):
    q = q.clone().requires_grad_(True)
    world, _ = _fk(m, q)
    loss = 0.0
    for i, f in enumerate(ids):
        v, w = _log(_compose(_inverse(_pose(targets[:, i])), _frame(m, world, f)))
        loss = loss + weights[..., i] * ((v * v).sum(-1) + (w * w).sum(-1))
    grad, = torch.autograd.grad(loss.sum(), q)
    return loss.detach(), grad


def exact(case: dict, seed: int):
    """What ``run`` returns, in float64 by plain torch; ``None`` for the iterative solvers, whose results
    are where their iteration stops."""
    kind = case["kind"]
    if kind in ("ik_single", "ik_batch", "ik_mix", "trajopt"):
        return None
    s = prepare(case, seed)
    if kind == "lie":
        a, b = _pose(s["a"].double()), _pose(s["b"].double())
        rel = _compose(_inverse(a), b)
        xi = _log(rel)
        return {"rel": torch.cat(rel, -1), "xi": torch.cat(xi, -1), "again": torch.cat(_compose(a, _exp(*xi)), -1)}
    m, q = s["model"], s["q"].detach().double()
    if kind == "pose_loss":
        w = s["weights"].double()
        parts = [_exact_loss(m, q[i:i + 16384], s["frames"], s["targets"][i:i + 16384].double(),
                             w[i:i + 16384] if w.dim() == 2 else w) for i in range(0, len(q), 16384)]
        return {"loss": torch.cat([p[0] for p in parts]), "grad": torch.cat([p[1] for p in parts])}
    if kind == "configuration":
        v = s["v"].double()
        moved, back = q.clone(), v.clone()
        free = m.joint_models[1].kind == "free_flyer"
        k, kv = (7, 6) if free else (0, 0)
        moved[:, k:] = q[:, k:] + v[:, kv:]
        if free:
            T = _compose(_pose(q[:, :7]), _exp(v[:, :3], v[:, 3:6]))
            moved[:, :3], moved[:, 3:7] = T[0], _unit(T[1])
            back[:, :3], back[:, 3:6] = _log(_compose(_inverse(_pose(q[:, :7])), _pose(moved[:, :7])))
        return {"moved": moved, "back": back}
    world, local = _fk(m, q)
    if kind == "frame_jac":
        poses = [_frame(m, world, f) for f in s["frames"]]
        J = torch.zeros(len(q), len(poses), 6, m.nv, dtype=torch.float64, device=DEV)
        for i, f in enumerate(s["frames"]):
            _jacobian(m, world, m.frames[f].parent_joint, poses[i], s["reference"], J[:, i])
        return {"poses": _cat(poses), "jacobians": J}
    J = torch.zeros(len(q), m.njoints, 6, m.nv, dtype=torch.float64, device=DEV)
    for j in range(m.njoints):
        _jacobian(m, world, j, world[j], "world", J[:, j])
    return {"world": _cat(world), "local": _cat(local),
            "frames": _cat([_frame(m, world, f) for f in range(m.nframes)]), "jacobians": J}
