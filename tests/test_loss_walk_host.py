"""The depth-first walk of the lane-per-configuration pose-loss kernel, restated on the CPU.

The restatement follows the kernel's table build (visit order from support masks, pruning to the
joints that move a frame, wrench slots) and its down / up traversal step by step, in float64.  It
must visit what it should, stay inside the slots the launch reserves (``n_frames - 1``) and give
the oracle's loss and gradient: on the synthetic robots, on random trees numbered in any
topological order, and for frame sets that leave whole branches unmoved.
"""

import numpy as np
import pytest
import torch

from betterrobot_b200 import synthetic as syn
from betterrobot_b200.model import build_model
from oracle import adjoint as A, kinematics as K, lie


def _tables(m, fids):
    sup = [sum(1 << k for k in m.supports[j]) for j in range(m.njoints)]
    fpar = [m.frames[f].parent_joint for f in fids]
    need = 0
    for p in fpar:
        need |= sup[p]
    moves = sum(1 << j for j in range(m.njoints) if m.nvs[j])
    framed = sum({1 << p for p in fpar})
    vis = [j for j in range(m.njoints) if need >> j & 1]

    def before(i, j):
        a, b = sup[i] & ~sup[j], sup[j] & ~sup[i]
        return a == 0 or (b != 0 and (a & -a) < (b & -b))

    ordered = all(m.parents[j] >= 0 and sup[j - 1] >> m.parents[j] & 1 for j in range(1, m.njoints))
    rank = {j: sum(i != j and before(i, j) for i in vis) for j in vis}
    if ordered:
        assert rank == {j: n for n, j in enumerate(vis)}
    child = {j: sum(m.parents[c] == j for c in vis) for j in vis}
    stored = sum(1 << j for j in vis if child[j] >= 2 or (child[j] == 1 and framed >> j & 1))
    order = sorted(vis, key=rank.get)
    frames = sorted(range(len(fids)), key=lambda f: (rank[fpar[f]], f))
    visits = []
    for j in order:
        above = sup[j] & ~(1 << j)
        visits.append(dict(j=j, slot=bin(above & stored).count("1"), stored=stored >> j & 1, branch=child[j] >= 2,
                           stop=(above & moves) == 0, chain=child[j] > 0,
                           parent=rank[m.parents[j]] if m.parents[j] >= 0 else -1,
                           frames=[f for f in frames if fpar[f] == j]))
    return visits


def _local(m, j, q):
    """liMi of joint j alone, through the oracle's FK of the chain's last link."""
    return K.forward_kinematics(m, q[None])[1][0, j]


def _adT(L, W):
    """Wrench of a child carried to its parent: (R f, R tau + t x R f)."""
    f, t = lie.so3_act(L[3:], W[:3]), lie.so3_act(L[3:], W[3:])
    return np.concatenate([f, t + np.cross(L[:3], f)])


def _walk(m, q, fids, targets, w):
    """(loss, dL/dv, slots used) of one configuration by the kernel's traversal."""
    visits = _tables(m, fids)
    local = K.forward_kinematics(m, q[None])[1][0]
    limit = max(0, min(len(fids) - 1, m.njoints - 1))
    slots, gv, loss = {}, np.zeros(m.nv), 0.0
    T, saved_at, saved = None, -1, None
    for k, v in enumerate(visits):
        if v["parent"] < 0:
            T = local[v["j"]]
        else:
            if v["parent"] != k - 1:
                if v["parent"] == saved_at:
                    T = saved
                else:
                    path = sorted(i for i, u in enumerate(visits) if u["j"] in m.supports[visits[v["parent"]]["j"]])
                    T = local[visits[path[0]]["j"]]
                    for i in path[1:]:
                        T = lie.se3_compose(T, local[visits[i]["j"]])
            T = lie.se3_compose(T, local[v["j"]])
        if v["branch"]:
            saved_at, saved = k, T
        W = np.zeros(6)
        for f in v["frames"]:
            P = m.frames[fids[f]].joint_placement.double().numpy()
            xi = lie.se3_log(lie.se3_compose(lie.se3_inverse(targets[f]), lie.se3_compose(T, P)))
            # body gradient 2 w Jr^-T xi by central differences of the log
            g = np.zeros(6)
            for c in range(6):
                e = np.zeros(6)
                e[c] = 1e-6
                D = lie.se3_compose(lie.se3_inverse(targets[f]), lie.se3_compose(T, P))
                hi = lie.se3_log(lie.se3_compose(D, lie.se3_exp(e)))
                lo = lie.se3_log(lie.se3_compose(D, lie.se3_exp(-e)))
                g[c] = w[f] * ((hi * hi).sum() - (lo * lo).sum()) / 2e-6
            W += _adT(P, g)
            loss += w[f] * (xi * xi).sum()
        if v["chain"]:
            if v["stored"]:
                assert v["slot"] < limit
                slots[v["slot"]] = W
            continue
        up_to = visits[k + 1]["parent"] if k + 1 < len(visits) else -1
        u = k
        while True:
            j = visits[u]["j"]
            for c in range(m.nvs[j]):
                gv[m.idx_vs[j] + c] = _column(m, j, c) @ W
            if visits[u]["stop"]:
                break
            W = _adT(local[j], W)
            u = visits[u]["parent"]
            if visits[u]["stored"]:
                assert visits[u]["slot"] < limit
                W = W + slots[visits[u]["slot"]]
                if u == up_to:
                    slots[visits[u]["slot"]] = W
                    break
    return loss, gv


def _column(m, j, c):
    """Motion subspace column c of joint j in its own frame, as (linear, angular)."""
    jm, S = m.joint_models[j], np.zeros(6)
    if jm.kind == "free_flyer":
        S[c] = 1.0
    elif jm.kind in ("spherical", "translation"):
        S[(3 if jm.kind == "spherical" else 0) + c] = 1.0
    elif jm.kind == "planar":
        S[c if c < 2 else 5] = 1.0
    else:
        from betterrobot_b200.model import joint_axis
        S[(3 if jm.kind.startswith("revolute") else 0):][:3] = joint_axis(jm)
    return S


def _random_tree(rng, n, preorder):
    """A random tree of revolute, prismatic and fixed joints; numbered depth first or in any topological order."""
    parents = [0]
    for i in range(1, n):
        if preorder:  # a joint on the previous one's path
            path, j = [], i
            while j > 0:
                path.append(j)
                j = parents[j - 1]
            parents.append(int(rng.choice(path)) if rng.random() < 0.5 else i)
        else:
            parents.append(int(rng.integers(0, i + 1)))
    joints = [{"name": f"j{i}", "kind": str(rng.choice(["revolute_rz", "revolute_rx", "prismatic_py", "fixed"])),
               "parent": p, "origin": syn._rand_pose(rng), "lower": -3, "upper": 3, "body": f"b{i}"}
              for i, p in enumerate(parents)]
    frames = [{"name": f"f{i}", "parent": int(rng.integers(0, n + 1)), "placement": syn._rand_pose(rng)}
              for i in range(int(rng.integers(1, 7)))]
    return build_model("tree", joints, frames, dtype=torch.float64)


def _check(m, fids, seed):
    rng = np.random.default_rng(seed)
    q = syn.random_q(m, 1, seed, rev_range=2.0).numpy()
    oMi, _ = K.forward_kinematics(m, syn.noisy_start(m, torch.from_numpy(q), 0.3, seed).numpy())
    targets = K.frame_placements(m, oMi, fids)
    w = rng.uniform(0.5, 2.0, size=len(fids))
    loss, gv = _walk(m, q[0], fids, targets[0], w)
    np.testing.assert_allclose(loss, A.pose_loss(m, q, fids, targets, w)[0], rtol=1e-12)
    # dL/dv by central differences through the retraction of single-DOF joints
    gq = A.pose_loss_grad(m, q, fids, targets, w)[0]
    for j in range(m.njoints):
        if m.nqs[j] == 1:
            assert abs(gv[m.idx_vs[j]] - gq[m.idx_qs[j]]) <= 1e-6 * (1.0 + np.abs(gq).max()), j


@pytest.mark.parametrize("robot", [syn.humanoid_spec, syn.dual_arm_spec, syn.chain_spec, syn.mixed_spec])
def test_robots(robot):
    m = syn.model_from_spec(robot(), dtype=torch.float64)
    _check(m, syn.op_frame_ids(m), 3)
    _check(m, [m.nframes - 1], 4)                      # one frame: every other branch unmoved
    _check(m, list(range(0, m.nframes, 3)) * 2, 5)     # body frames, each twice


@pytest.mark.parametrize("seed", range(12))
def test_random_trees(seed):
    rng = np.random.default_rng(seed)
    m = _random_tree(rng, int(rng.integers(2, 24)), seed % 2 == 0)
    _check(m, syn.op_frame_ids(m), seed)
    _check(m, list(range(m.nframes)), seed + 100)
