"""FK pose loss with a hand-written adjoint behind ``torch.autograd.Function``.

``pose_loss(model, q, frame_ids, targets, weights)`` returns, per configuration,
``sum_f w_f |log(T_f^-1 * oMf(q))|^2`` — the pose residual of
``src/better_robot/residuals/pose.py:58-66`` squared and summed over frames.
In the reference its gradient comes from torch autograd through every SE3 op
of the FK loop (``src/better_robot/kinematics/forward.py:79-81`` keeps that tape
on purpose); here it is the hand-written adjoint of ``fk_adjoint.cu``.

A configuration's loss depends on its own q only, so a forward pass whose ``q`` needs a gradient can
compute the loss and each configuration's own gradient together (one walk over the tree instead of
one per pass); ``backward`` scales that gradient row by row with the incoming one.  Without a
gradient to compute, the forward evaluates the loss alone.

Modes: ``"store"`` does that, and keeps ``batch * nq`` floats for the backward; ``"recompute"`` evaluates the
loss alone, keeps nothing of its own, and walks the tree again for the gradient in the backward (for
when memory is short, or no backward may follow); ``"auto"`` is ``"store"``, the faster of the two with a
backward at every batch (humanoid, 12 frames, kernels of both passes: 34 against 50 us at B = 16,384, 194
against 320 at 262,144; forward alone 31 against 19, 176 against 103).

The loss is the same number in every mode and without a gradient.  Batches of at least 200 (joints + frames)
configurations run another kernel than smaller ones, so the same configuration in a small and in a
large batch agrees to float32 rounding, not to the bit.
"""

from __future__ import annotations

from typing import Sequence

import torch

from . import _lib
from .exceptions import ShapeError
from .kinematics import _validate_q
from .tree import device_tree

def path_slots(arrays, frame_ids: tuple) -> int:
    """Most joints on one root-to-leaf path that hold a waiting wrench in the adjoint's walk: in the tree
    pruned to the frames' ancestors, those with a child and a frame of their own or a second child.
    Kept with the tree table, per frame set; -1 (not known) for a list that the entry point refuses."""
    n = arrays.path_slots.get(frame_ids)
    if n is None:
        if not frame_ids or min(frame_ids) < 0 or max(frame_ids) >= arrays.nf:
            return -1
        framed = {int(arrays.frame_parent[f]) for f in frame_ids}
        support = [int(x) for x in arrays.support]
        need = 0
        for j in framed:
            need |= support[j]
        children = [0] * arrays.nj
        for j in range(1, arrays.nj):
            if need >> j & 1 and arrays.parent[j] >= 0:
                children[arrays.parent[j]] += 1
        stored = sum(1 << j for j in range(arrays.nj)
                     if children[j] >= 2 or (children[j] == 1 and j in framed))
        n = max(bin(support[j] & stored).count("1") for j in framed)
        if len(arrays.path_slots) >= 256:
            arrays.path_slots.clear()
        arrays.path_slots[frame_ids] = n
    return n


def _loss_only(model, q, frame_ids, targets, weights):
    loss = torch.empty(q.shape[0], device=q.device, dtype=torch.float32)
    with _lib.on(q.device):
        _lib.call("br_pose_loss", device_tree(model, q.device).ptr, q.data_ptr(), q.shape[0],
                  _lib.id_array(frame_ids), len(frame_ids), targets.data_ptr(), weights.data_ptr(),
                  int(weights.dim() == 2), loss.data_ptr(), None, _lib.stream_ptr())
    return loss


class _PoseLoss(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, targets, weights, model, frame_ids, mode):
        """``mode``: "store", "recompute", or None where no gradient can be asked for."""
        if mode != "store":
            ctx.model, ctx.frame_ids = model, frame_ids
            ctx.save_for_backward(q, targets, weights)
            return _loss_only(model, q, frame_ids, targets, weights)
        loss = torch.empty(q.shape[0], device=q.device, dtype=torch.float32)
        unit = torch.empty_like(q)
        dt = device_tree(model, q.device)
        with _lib.on(q.device):
            _lib.call("br_pose_loss_value_grad", dt.ptr, q.data_ptr(), q.shape[0], _lib.id_array(frame_ids),
                      len(frame_ids), targets.data_ptr(), weights.data_ptr(), int(weights.dim() == 2),
                      path_slots(dt.arrays, frame_ids), loss.data_ptr(), unit.data_ptr(), _lib.stream_ptr())
        # the inputs too: changing one in place before the backward stays an error
        ctx.save_for_backward(q, targets, weights, unit)
        return loss

    @staticmethod
    def backward(ctx, grad_loss):
        q, targets, weights, *stored = ctx.saved_tensors
        g = grad_loss if grad_loss.dtype == torch.float32 else grad_loss.float()
        grad_q = torch.empty_like(q)
        with _lib.on(q.device):
            if stored:
                if g.stride(0) not in (0, 1):
                    g = g.contiguous()
                _lib.call("br_scale_rows", stored[0].data_ptr(), g.data_ptr(), g.stride(0), q.shape[0], q.shape[1],
                          grad_q.data_ptr(), _lib.stream_ptr())
            else:
                g = g.contiguous()
                _lib.call("br_pose_loss_backward", device_tree(ctx.model, q.device).ptr, q.data_ptr(), None, q.shape[0],
                          _lib.id_array(ctx.frame_ids), len(ctx.frame_ids), targets.data_ptr(), weights.data_ptr(),
                          int(weights.dim() == 2), g.data_ptr(), grad_q.data_ptr(), _lib.stream_ptr())
        return grad_q, None, None, None, None, None


def pose_loss(model, q: torch.Tensor, frame_ids: Sequence[int], targets: torch.Tensor, weights: torch.Tensor,
              mode: str = "auto", check_quaternion: bool = False) -> torch.Tensor:
    """Per-configuration pose loss ``(B,)``; differentiable w.r.t. ``q`` (B, nq) float32 CUDA.

    The backward kernel maps gradients to raw q for every joint kind of the tree table
    (fixed, revolute, unbounded revolute, prismatic, free-flyer, spherical, planar,
    translation).  ``mode``: "store", "recompute" or "auto", above.
    """
    _validate_q(model, q, check_quaternion)
    if q.dim() != 2:
        raise ShapeError("pose_loss takes q of shape (B, nq)")
    frame_ids = tuple(int(f) for f in frame_ids)
    B, F = q.shape[0], len(frame_ids)
    if targets.shape != (B, F, 7):
        raise ShapeError(f"targets must be ({B}, {F}, 7), got {tuple(targets.shape)}")
    if weights.shape not in ((F,), (B, F)):
        raise ShapeError(f"weights must be ({F},) or ({B}, {F}), got {tuple(weights.shape)}")
    if mode not in ("store", "recompute", "auto"):
        raise ValueError(f"mode must be 'store', 'recompute' or 'auto', got {mode!r}")
    if not (torch.is_grad_enabled() and (q.requires_grad or targets.requires_grad or weights.requires_grad)):
        mode = None
    elif mode == "auto":
        mode = "store"
    return _PoseLoss.apply(q.contiguous(), targets.contiguous().float(), weights.contiguous().float(), model,
                           frame_ids, mode)
