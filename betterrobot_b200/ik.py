"""Batched LM / Gauss-Newton IK on the sm_100a persistent kernel.

Drop-in for ``better_robot.tasks.ik`` (``src/better_robot/tasks/ik.py:37-266``):
``solve_ik(model, targets, initial_q=..., cost_cfg=..., optimizer_cfg=...)`` builds
the same cost stack — one ``PoseResidual`` per target, ``JointPositionLimit``
(item weight ``limit_weight``), ``RestResidual`` (item weight ``rest_weight``) —
and runs the same Levenberg-Marquardt loop with ``Adaptive`` damping.  Unlike
the reference it also solves whole batches, including uneven mixes of robots,
in one launch (``solve_ik_batched``, ``PackedIK``).
"""

from __future__ import annotations

import ctypes
from dataclasses import dataclass, field
from typing import Literal, Sequence

import numpy as np
import torch

from . import _lib
from ._lib import BrTree, IKBatch, IKResultBuf, IKSettings, c_int32
from .exceptions import ShapeError
from .tree import device_tree

OPT_LM, OPT_GN = 0, 1
MAX_CLASSES, MAX_TARGETS = 8, 8
SCRATCH_BYTES = 16
HOST_FILL_FLOATS = 16384


@dataclass
class IKCostConfig:
    """Weights of the built-in IK stack (``tasks/ik.py:37-48``)."""

    pos_weight: float = 1.0
    ori_weight: float = 1.0
    pose_weight: float = 1.0
    limit_weight: float = 0.1
    rest_weight: float = 0.01
    collision_margin: float = 0.02
    collision_weight: float = 1.0
    q_rest: torch.Tensor | None = None


@dataclass
class OptimizerConfig:
    """Optimizer selection (``tasks/ik.py:51-69``).

    ``lam0``/``factor`` are the ``Adaptive`` damping parameters; their defaults are
    what ``solve_ik`` effectively uses (``Adaptive()`` = 1e-4 / 2, ``tasks/ik.py:250``).
    ``lam_min``/``lam_max`` are ``Adaptive``'s clamps (``strategies/adaptive.py:19-25``).
    """

    optimizer: Literal["lm", "gn", "adam", "lbfgs", "lm_then_lbfgs"] = "lm"
    max_iter: int = 100
    jacobian_strategy: object = None
    linear_solver: Literal["cholesky", "lstsq", "cg"] = "cholesky"
    kernel: Literal["l2", "huber", "cauchy", "tukey"] = "l2"
    damping: Literal["constant", "adaptive", "trust_region"] = "adaptive"
    tol: float = 1e-6
    refine_disabled_items: tuple = ()
    lam0: float = 1e-4
    factor: float = 2.0
    lam_min: float = 1e-10
    lam_max: float = 1e8
    gn_eps: float = 1e-8
    kernel_param: float | None = None  # None: the kernel class's default (Huber 1.0, Cauchy 1.0, Tukey 4.685)
    # arithmetic of the Jacobian, J^T J, J^T r and the factorization ("f32": fastest; "f64": the
    # float64 reference's iterates); the iterate, FK, residual and cost are float64 in both
    precision: Literal["f32", "f64"] = "f32"


PRECISIONS = {"f32": 0, "f64": 1}  # BR_PREC_*


# OptimizerConfig.kernel -> BR_KERNEL_*, and the default parameter of each kernel class
# (src/better_robot/optim/kernels/huber.py, cauchy.py, tukey.py)
KERNELS = {"l2": 0, "huber": 1, "cauchy": 2, "tukey": 3}
TARGET_KINDS = {"pose": 0, "position": 1, "orientation": 2}   # BR_TARGET_*
KERNEL_DEFAULTS = {"huber": 1.0, "cauchy": 1.0, "tukey": 4.685}


@dataclass
class IKResult:
    """Return type of ``solve_ik`` (``tasks/ik.py:72-99``)."""

    q: torch.Tensor
    residual: torch.Tensor
    iters: int
    converged: bool
    model: object

    def fk(self):
        from .kinematics import forward_kinematics
        return forward_kinematics(self.model, self.q, compute_frames=True)

    def frame_pose(self, name: str) -> torch.Tensor:
        return self.fk().frame_pose_world[..., self.model.frame_id(name), :]

    def q_only(self) -> torch.Tensor:
        return self.q


@dataclass
class BatchIKResult:
    """Batched result: ``q (P, nq)`` (or a list for uneven mixes), per-problem iterations/verdicts."""

    q: object
    iters: torch.Tensor
    converged: torch.Tensor
    status: torch.Tensor
    cost: torch.Tensor
    residual: object = None


def settings_from(cost_cfg: IKCostConfig, opt: OptimizerConfig) -> IKSettings:
    if opt.optimizer not in ("lm", "gn"):
        raise NotImplementedError(f"optimizer {opt.optimizer!r}: the sm_100a path runs 'lm' and 'gn'")
    if opt.linear_solver != "cholesky":
        raise NotImplementedError("the sm_100a path solves the normal equations by Cholesky")
    if opt.damping not in ("adaptive", "constant"):
        raise NotImplementedError(f"damping {opt.damping!r} is not on the sm_100a path")
    s = IKSettings()
    s.lam0 = opt.lam0
    s.factor = 1.0 if opt.damping == "constant" else opt.factor   # Constant: lambda never changes
    s.tol = opt.tol
    s.lam_min, s.lam_max, s.gn_eps = opt.lam_min, opt.lam_max, opt.gn_eps
    s.pos_weight = cost_cfg.pos_weight * cost_cfg.pose_weight       # tasks/ik.py:193-194
    s.ori_weight = cost_cfg.ori_weight * cost_cfg.pose_weight
    s.limit_weight = cost_cfg.limit_weight
    s.rest_weight = cost_cfg.rest_weight
    s.max_iter = int(opt.max_iter)
    s.optimizer = OPT_LM if opt.optimizer == "lm" else OPT_GN
    if opt.kernel not in KERNELS:
        raise ValueError(f"Unknown kernel {opt.kernel!r}; expected one of {sorted(KERNELS)}")
    s.kernel = KERNELS[opt.kernel]
    s.kernel_param = KERNEL_DEFAULTS.get(opt.kernel, 0.0) if opt.kernel_param is None else float(opt.kernel_param)
    if opt.precision not in PRECISIONS:
        raise ValueError(f"Unknown precision {opt.precision!r}; expected 'f32' or 'f64'")
    s.precision = PRECISIONS[opt.precision]
    return s


def team_floats(model, max_targets: int, device) -> int:
    dt = device_tree(model, device)
    return int(_lib.load().br_lm_team_floats(dt.ptr, max_targets))


def default_team_size(model) -> int:
    """Lanes per problem: the kernel is built for 32-lane teams only."""
    return 32


class PackedIK:
    """An uneven batch of IK problems packed for one persistent launch.

    ``problems`` are grouped by robot (class).  For class ``c``: ``models[c]``,
    ``frame_ids[c]`` (P_c, K_c) int, ``targets[c]`` (P_c, K_c, 7) float32,
    ``q0[c]`` (P_c, nq_c) float32 and ``n_targets[c]`` (P_c,) (<= K_c).
    Device buffers are allocated once; ``set_inputs`` refreshes targets / q0 in place
    and ``solve`` launches (graph-capturable: no allocation, no host sync).
    """

    def __init__(self, models: Sequence, frame_ids: Sequence, n_targets: Sequence, q_rest: Sequence | None = None,
                 team_sizes: Sequence[int] | None = None, device="cuda", warps_per_cta: int = 4,
                 with_residual: bool = False, target_kinds: Sequence | None = None):
        self._build(models, frame_ids, n_targets, q_rest, team_sizes, device, warps_per_cta, with_residual,
                    target_kinds, True)
        # The tables hold the indices and offsets that the kernel addresses memory with, and a plan may be
        # solved on any stream: the upload, queued on the current one, is complete when the plan is handed out.
        torch.cuda.current_stream(self.device).synchronize()

    def _build(self, models, frame_ids, n_targets, q_rest, team_sizes, device, warps_per_cta, with_residual,
               target_kinds, fill: bool) -> None:
        """Lay out and upload the plan, on the current stream and without waiting for it.  ``fill``: the
        identity targets and zero start configurations of a plan that is solved before ``set_inputs``
        are written."""
        if not 1 <= len(models) <= MAX_CLASSES:
            raise ShapeError(f"1..{MAX_CLASSES} robot classes per launch, got {len(models)}")
        self.device = torch.device(device)
        if self.device.index is None:
            self.device = torch.device("cuda", torch.cuda.current_device())
        self.models = list(models)
        self.C = len(models)
        n_targets = [np.asarray(n, np.int32) for n in n_targets]
        frame_ids = [np.asarray(f, np.int32) for f in frame_ids]
        self.counts = [int(n.shape[0]) for n in n_targets]
        P = self.P = sum(self.counts)
        K = self.K = max(int(f.shape[1]) for f in frame_ids)
        if K > MAX_TARGETS:
            raise ShapeError(f"at most {MAX_TARGETS} targets per problem")
        self.team = [int(t) for t in (team_sizes or [default_team_size(m) for m in models])]
        for m, t in zip(models, self.team):
            if t != 32:
                raise ShapeError(f"team size {t}: the kernel runs one problem per 32-lane warp")
        self.trees = [device_tree(m, self.device) for m in models]
        self.warps_per_cta = warps_per_cta
        # per-problem layout: classes contiguous, in class order
        starts, q_total = [0], 0
        for n, m in zip(self.counts, models):
            starts.append(starts[-1] + n)
            q_total += n * m.nq
        self.class_start = np.array(starts[:-1])
        self.q_total = q_total
        kinds = self._kinds_of(target_kinds) if target_kinds is not None else None
        rest = [torch.as_tensor(m.q_neutral if q_rest is None or q_rest[c] is None else q_rest[c],
                                dtype=torch.float32).detach().reshape(-1, m.nq) for c, m in enumerate(models)]
        # Every table of the plan lies in one int32 array and goes up in one copy, and so do the rest
        # configurations up to 64 KB; larger ones are broadcast on the device.  (Made and copied one by one,
        # with the fills of the buffers, they took 350 of a single solve's 480 us.)
        host_rest = q_total <= HOST_FILL_FLOATS and not any(r.is_cuda for r in rest)
        self._sections, o = {}, SCRATCH_BYTES // 4
        self._sections["scratch"] = (0, o, None, (o,))
        for name, n, dtype, shape in (
                ("order", P, None, (P,)), ("items", 3 * P, None, (3 * P,)), ("n_targets_t", P, None, (P,)),
                ("frames_t", P * K, None, (P, K)), ("q_offset", 2 * P + 2, torch.int64, (P + 1,)),
                ("r_offset", 2 * P + 2, torch.int64, (P + 1,)),
                ("kinds", 0 if kinds is None else P * K, None, (P, K)),
                ("q_rest", q_total if host_rest else 0, torch.float32, (q_total,))):
            self._sections[name] = (o, n, dtype, shape)
            o += (n + 3) & ~3
        # staged in pinned memory (the allocator holds it until the copy has run); a capture refuses the copy
        # of pageable memory, whose address a replay would read
        capturing = _lib.capturing(self.device)
        staged = torch.zeros(o, dtype=torch.int32, pin_memory=not capturing)
        host = staged.numpy()

        def part(name, dtype=np.int32):
            o, n = self._sections[name][:2]
            return host[o:o + n].view(dtype)

        nt_all, fr = part("n_targets_t"), part("frames_t").reshape(P, K)
        # P + 1 offsets (the last one is the total), so a class with no problems indexes in range
        self.q_offset_np, self.r_offset_np = part("q_offset", np.int64), part("r_offset", np.int64)
        self.r_dim = np.empty(P, np.int64)
        for c, (m, n, f) in enumerate(zip(models, n_targets, frame_ids)):
            s0, s1 = starts[c], starts[c + 1]
            if n.size and (n.min() < 1 or n.max() > K):
                raise ShapeError("each problem needs 1..K targets")
            if f.size and (f.min() < 0 or f.max() >= m.nframes):
                raise ShapeError(f"class {c}: frame id out of range")
            nt_all[s0:s1] = n
            fr[s0:s1, :f.shape[1]] = f
            self.q_offset_np[s0 + 1:s1 + 1] = m.nq
            if kinds is None:
                rows = 6 * n
            else:
                rows = (np.where(kinds[s0:s1] == 0, 6, 3) * (np.arange(K)[None, :] < n[:, None])).sum(-1)
            self.r_dim[s0:s1] = rows + (2 * m.nq + m.nv)
        np.cumsum(self.q_offset_np, out=self.q_offset_np)
        np.cumsum(self.r_dim, out=self.r_offset_np[1:])
        # work items: heaviest classes first, and inside a class the problems with the fewest
        # targets first (they run the most iterations: a less constrained problem's rest term
        # settles slowly), so the longest solves start early and the launch's tail is short
        cost = [m.nv ** 2 * (1 + K) for m in models]
        order, items, slot = part("order"), part("items").reshape(P, 3), 0  # item: (slot, problems, class)
        items[:, 0] = np.arange(P, dtype=np.int32)
        items[:, 1] = 1  # one problem per 32-lane team
        for c in sorted(range(self.C), key=lambda k: -cost[k]):
            n = self.counts[c]
            order[slot:slot + n] = np.argsort(n_targets[c], kind="stable")
            order[slot:slot + n] += starts[c]
            items[slot:slot + n, 2] = c
            slot += n
        self.n_items = P
        if kinds is not None:
            part("kinds").reshape(P, K)[...] = kinds
        dev = self.device
        x0s = [int(self.q_offset_np[s]) for s in starts]
        if host_rest:
            qr = part("q_rest", np.float32)
            for c, m in enumerate(models):
                qr[x0s[c]:x0s[c + 1]].reshape(-1, m.nq)[...] = rest[c].expand(self.counts[c], m.nq).numpy()
        self._tables = staged.to(dev, non_blocking=not capturing)
        if not host_rest:
            self.q_rest = torch.empty(q_total, device=dev)
            for c, m in enumerate(models):
                self.q_rest[x0s[c]:x0s[c + 1]].view(-1, m.nq).copy_(rest[c].to(dev).expand(self.counts[c], m.nq))
        if kinds is None:
            self.kinds = None
        self.targets = torch.empty(P, K, 7, device=dev)
        self.x0 = torch.empty(q_total, device=dev)
        if fill:
            self.targets.zero_()
            self.targets[..., 6] = 1.0
            self.x0.zero_()
        self.x = torch.empty(q_total, device=dev)
        self.verdict = torch.empty(2, P, dtype=torch.int32, device=dev)  # iterations, status
        self.iters, self.status = self.verdict.unbind()
        self.cost = torch.empty(P, device=dev)
        # fixed layout per problem: target rows, 2 nq limit rows, nv rest rows (zero when unused)
        self.residual = torch.zeros(int(self.r_offset_np[-1]), device=dev) if with_residual else None
        # ctypes structs (kept alive on the object)
        self._trees = (BrTree * self.C)(*[t.struct for t in self.trees])
        self._teams = (c_int32 * self.C)(*self.team)
        base = self._tables.data_ptr()
        at = {name: base + 4 * sec[0] for name, sec in self._sections.items()}
        b = IKBatch()
        b.n_problems, b.max_targets, b.n_classes, b.n_items = P, K, self.C, self.n_items
        b.trees, b.team_size = self._trees, self._teams
        b.items, b.order = at["items"], at["order"]
        b.n_targets, b.frames = at["n_targets_t"], at["frames_t"]
        b.targets, b.q_offset = self.targets.data_ptr(), at["q_offset"]
        b.x0, b.q_rest = self.x0.data_ptr(), at["q_rest"] if host_rest else self.q_rest.data_ptr()
        b.r_offset = at["r_offset"]
        b.target_kind = at["kinds"] if kinds is not None else None
        self._batch, self._scratch = b, base
        r = IKResultBuf()
        r.x, r.iters, r.status, r.cost = self.x.data_ptr(), self.iters.data_ptr(), self.status.data_ptr(), \
            self.cost.data_ptr()
        r.residual = self.residual.data_ptr() if self.residual is not None else None
        self._result = r

    def _kinds_of(self, target_kinds):
        """Target kinds of every problem ``(P, K)``, None when all are poses."""
        kinds = np.zeros((self.P, self.K), np.int32)
        for c in range(self.C):
            if target_kinds[c] is None:
                continue
            k = np.asarray([TARGET_KINDS[x] if isinstance(x, str) else int(x)
                            for x in np.asarray(target_kinds[c]).reshape(-1)], np.int32)
            k = k.reshape(np.asarray(target_kinds[c]).shape)
            if ((k < 0) | (k > 2)).any():
                raise ShapeError("target kinds are 'pose', 'position' or 'orientation'")
            s0 = self.class_start[c]
            kinds[s0:s0 + self.counts[c], :k.shape[-1]] = np.broadcast_to(k, (self.counts[c], k.shape[-1]))
        return kinds if kinds.any() else None

    def __getattr__(self, name):
        """The device tables as tensors, views of the one buffer, made when asked for."""
        sec = self.__dict__.get("_sections", {}).get(name)
        if sec is None:
            raise AttributeError(name)
        o, n, dtype, shape = sec
        t = self._tables[o:o + n]
        t = (t if dtype is None else t.view(dtype)).view(shape)
        self.__dict__[name] = t
        return t

    def set_inputs(self, targets: Sequence, q0: Sequence) -> None:
        """Copy per-class targets (P_c, K_c, 7) and start configurations (P_c, nq_c) into the device buffers."""
        for c, m in enumerate(self.models):
            s0, n = int(self.class_start[c]), self.counts[c]
            t = torch.as_tensor(targets[c], dtype=torch.float32).detach()
            self.targets[s0:s0 + n, :t.shape[1]].copy_(t, non_blocking=True)
            o = int(self.q_offset_np[s0])
            self.x0[o:o + n * m.nq].copy_(torch.as_tensor(q0[c], dtype=torch.float32).detach().reshape(-1),
                                                 non_blocking=True)

    def solve(self, settings: IKSettings, stream: int | None = None) -> None:
        _lib.call("br_lm_solve", ctypes.byref(self._batch), ctypes.byref(settings), ctypes.byref(self._result),
                  self.warps_per_cta, self._scratch, SCRATCH_BYTES,
                  stream if stream is not None else _lib.stream_ptr(self.device))

    def capture(self, settings: IKSettings) -> "torch.cuda.CUDAGraph":
        """Capture one solve (scratch zeroing + the persistent launch) in a CUDA graph.

        Replaying the graph re-solves from the current contents of the input buffers
        (``set_inputs`` copies new targets / start configurations into them in place).
        """
        self._graph_settings = settings  # the struct must outlive the capture call
        with torch.cuda.device(self.device):
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                self.solve(settings)           # warm-up outside capture (module load, smem attribute)
            torch.cuda.current_stream().wait_stream(side)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                self.solve(settings)
        self.graph = g
        return g

    def q_of(self, c: int) -> torch.Tensor:
        s0, n, nq = int(self.class_start[c]), self.counts[c], self.models[c].nq
        o = int(self.q_offset_np[s0])
        return self.x[o:o + n * nq].view(n, nq)

    def class_slice(self, c: int) -> slice:
        s0 = int(self.class_start[c])
        return slice(s0, s0 + self.counts[c])


def solve_ik_batched(model, frame_ids, targets: torch.Tensor, initial_q: torch.Tensor, *,
                     cost_cfg: IKCostConfig | None = None, optimizer_cfg: OptimizerConfig | None = None,
                     n_targets=None, with_residual: bool = False, team_size: int | None = None,
                     warps_per_cta: int = 4, target_kinds=None) -> BatchIKResult:
    """Solve ``P`` independent problems of one robot: ``targets (P, K, 7)`` for ``frame_ids``
    (K ids shared by all problems, or ``(P, K)``), ``initial_q (P, nq)``.

    ``target_kinds`` (K names, or a ``(P, K)`` array): "pose" (``PoseResidual``, the
    default), "position" (``PositionResidual``, weight ``pos_weight * pose_weight``) or
    "orientation" (``OrientationResidual``, weight ``ori_weight * pose_weight``),
    ``src/better_robot/residuals/pose.py:58-195``.  With ``with_residual`` the stacked
    residual has 6 rows per pose target and 3 per position / orientation target.
    """
    pk, res = _solve_one_class(model, frame_ids, targets, initial_q, cost_cfg, optimizer_cfg, n_targets,
                               with_residual, team_size, warps_per_cta, target_kinds)
    return BatchIKResult(q=pk.q_of(0), iters=pk.iters, converged=(pk.status & 0xFF) == 0, status=pk.status,
                         cost=pk.cost, residual=res)


def _solve_one_class(model, frame_ids, targets, initial_q, cost_cfg=None, optimizer_cfg=None, n_targets=None,
                     with_residual=False, team_size=None, warps_per_cta=4, target_kinds=None):
    """The solved ``PackedIK`` and its stacked residual (arguments of ``solve_ik_batched``)."""
    cost_cfg = cost_cfg or IKCostConfig()
    optimizer_cfg = optimizer_cfg or OptimizerConfig()
    if initial_q.dim() != 2 or initial_q.shape[-1] != model.nq:
        raise ShapeError(f"initial_q must be (P, {model.nq}), got {tuple(initial_q.shape)}")
    _lib.require_cuda(initial_q)
    P = initial_q.shape[0]
    fr = np.asarray(frame_ids, np.int32)
    if fr.ndim == 1:
        fr = np.broadcast_to(fr, (P, fr.shape[0]))
    K = fr.shape[1]
    if targets.shape != (P, K, 7):
        raise ShapeError(f"targets must be ({P}, {K}, 7), got {tuple(targets.shape)}")
    nt = np.full(P, K, np.int32) if n_targets is None else np.asarray(n_targets, np.int32)
    qr = [cost_cfg.q_rest] if cost_cfg.q_rest is not None else None
    pk = PackedIK.__new__(PackedIK)
    pk._build([model], [fr], [nt], qr, [team_size or default_team_size(model)], initial_q.device, warps_per_cta,
              with_residual, None if target_kinds is None else [target_kinds], False)
    pk.set_inputs([targets], [initial_q])
    with _lib.on(initial_q.device):
        pk.solve(settings_from(cost_cfg, optimizer_cfg))
    res = None
    if with_residual:
        # the reference's CostStack has a limit / rest block only when its weight is > 0
        # (tasks/ik.py:200-205): drop the unused blocks of the fixed device layout
        def stack_rows(r: torch.Tensor) -> torch.Tensor:
            if cost_cfg.limit_weight > 0.0 and cost_cfg.rest_weight > 0.0:
                return r
            nt_rows = r.shape[-1] - 2 * model.nq - model.nv
            parts = [r[..., :nt_rows]]
            if cost_cfg.limit_weight > 0.0:
                parts.append(r[..., nt_rows:nt_rows + 2 * model.nq])
            if cost_cfg.rest_weight > 0.0:
                parts.append(r[..., nt_rows + 2 * model.nq:])
            return torch.cat(parts, -1) if len(parts) > 1 else parts[0]
        if P == 0:
            res = pk.residual.view(0, 0)
        else:
            res = (stack_rows(pk.residual.view(P, -1)) if (pk.r_dim == pk.r_dim[0]).all()
                   else [stack_rows(r) for r in torch.split(pk.residual, [int(d) for d in pk.r_dim])])
    return pk, res


def solve_ik(model, targets: dict, *, initial_q: torch.Tensor | None = None, cost_cfg: IKCostConfig | None = None,
             optimizer_cfg: OptimizerConfig | None = None, robot_collision=None, device=None) -> IKResult:
    """Whole-body IK for one configuration (``tasks/ik.py:150-266``); ``targets``: frame name -> (7,) pose."""
    cost_cfg = cost_cfg or IKCostConfig()
    optimizer_cfg = optimizer_cfg or OptimizerConfig()
    if initial_q is not None:
        x0 = initial_q.detach().float()
    else:
        x0 = model.q_neutral.clone().float()
    dev = x0.device if x0.is_cuda else torch.device(device or "cuda")
    x0 = x0.to(dev).reshape(1, -1)
    names = list(targets)
    if not names:
        raise ShapeError("solve_ik needs at least one target")
    fids = [model.frame_id(n) for n in names]
    T = torch.stack([torch.as_tensor(targets[n], dtype=torch.float32).reshape(7) for n in names]).to(dev)
    pk, residual = _solve_one_class(model, fids, T[None], x0, cost_cfg, optimizer_cfg, with_residual=True)
    (iters,), (status,) = pk.verdict.tolist()
    return IKResult(q=pk.x, residual=residual[0], iters=iters, converged=(status & 0xFF) == 0, model=model)
