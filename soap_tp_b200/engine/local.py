"""Single-GPU (grid (1, 1)) device pipeline.

With one rank the packed block-cyclic buffers ARE the dense column-major matrices, so the whole
step is a chain of this package's kernels on the caller's stream, its averages on one beside it:

    split G (both orientations)                                   largest_kernel, half_planes_kernel
    T   = X^T Q_L                (planes)                          gemm_half / split epilogue
    Y   = T^T Q_R, Adam(Y) -> U  (planes), m, v updated in place   gemm_half / Adam epilogue
    T2  = U^T Q_L^T              (planes)                          gemm_half / split epilogue
    out = T2^T Q_R^T             (row-major shard)                 gemm_half / row-major epilogue
    L   = b L + (1-b) G G^T,  R = b R + (1-b) G^T G                gemm_half / EMA epilogue, lower tiles + mirror

Every product is brought to the kernel's single form ``acc = Za^T Zb`` with K-contiguous operands
by keeping each basis in both orientations as operand planes; the planes are rebuilt only when the
basis tensor changes (refresh, initialisation, or a user writing into ``state``).  The planes are scaled fp16 pairs
(``kernels.HalfPlanes``); where a matrix has rows or columns so small beside the others that pairs would hold fewer bits of
them than tf32 values with bf16 corrections do, the rotation's kernels find that out on the device and run on such planes
instead (``csrc/gemm_half.h``, ``RangeGuard``).  With ``SOAP_TP_MIXED_CORRECTIONS=0`` every product is three tf32 MMAs.
"""
from __future__ import annotations

import functools
import math
import os
import weakref
from collections import Counter, OrderedDict
from typing import Any, Dict, MutableMapping, Optional, Tuple

import torch
from torch import Tensor

from ..profiling import GLOBAL_STAGE_TIMER as TIMER
from . import kernels as k
from . import factor

_C = k._C


_NO_OPERAND = (0, 0, 64, 0, 0)        # of an orientation that the native call does not use


class BasisPlanes:
    """Both orientations of one orthogonal basis as operand planes, tied to a tensor version."""

    def __init__(self, half: bool = True) -> None:
        self.half = half                  # scaled fp16 planes; else tf32 planes with bf16 corrections
        self.key: Optional[tuple] = None
        self.owner = None                 # weak reference to the tensor object the planes were made from
        self.plain = None                 # operand Q   (depth = rows of Q)
        self.transposed = None            # operand Q^T (depth = cols of Q)
        self.native = None                # both, and the basis itself, as the native calls take them
        self.copy: Optional[Tensor] = None    # of a basis of another type, which they mean then

    def once(self, Q: Tensor, size: int, turned: bool) -> "BasisPlanes":
        """The planes of one orientation only, for one use."""
        view = Q[:size, :size]
        self.copy = None if Q.dtype == torch.float32 else view.float()
        if self.copy is not None:
            view = self.copy
        planes = (_operand if self.half else _tf32_operand)(size, size, Q.device)
        self.plain, self.transposed = (None, planes) if turned else (planes, None)
        split(view, self.plain, self.transposed)
        if isinstance(planes, k.HalfPlanes):
            here = planes.operand()
            self.native = _C.BasisOperands(size, (_NO_OPERAND + here if turned else here + _NO_OPERAND) + (view.data_ptr(), *view.stride()))
        return self

    def refresh(self, Q: Tensor, size: int) -> None:
        key = (Q.data_ptr(), Q._version, size)
        # the planes belong to one tensor OBJECT: a new tensor at a recycled address with the same version count
        # (a freshly loaded checkpoint, a test's next case) must not be taken for the old one
        if key == self.key and self.owner is not None and self.owner() is Q:
            return
        view = Q[:size, :size]
        self.copy = None if Q.dtype == torch.float32 else view.float()
        if self.copy is not None:
            view = self.copy
        if self.plain is None or self.plain.depth != size or self.plain.device != Q.device:
            # (an address that was recycled by a tensor of another size starts over)
            make = _operand if self.half else _tf32_operand
            self.plain, self.transposed = make(size, size, Q.device), make(size, size, Q.device)
        split(view, self.plain, self.transposed)
        if isinstance(self.plain, k.HalfPlanes):
            self.native = _C.BasisOperands(size, self.plain.operand() + self.transposed.operand() + (view.data_ptr(), *view.stride()))
        self.key = (Q.data_ptr(), Q._version, size)
        self.owner = weakref.ref(Q)


class ParameterContext:
    """Per-parameter device-side caches (basis planes)."""

    def __init__(self) -> None:
        self.left = BasisPlanes()
        self.right = BasisPlanes()
        self.bytes = 0


_CONTEXTS: "OrderedDict[tuple, ParameterContext]" = OrderedDict()
_WORKSPACES: Dict[tuple, Any] = {}


# Operand planes of the eigenbases kept between steps (SOAP_TP_BASIS_CACHE_GB, default 40), counted as 12 bytes per basis
# element; fp16 pairs hold 8 (two orientations of 4), tf32 planes 16.  Beyond the limit parameters' planes are dropped (the
# most recently used first, see ``context_for``) and split again on use.
BASIS_CACHE_BYTES = int(float(os.environ.get("SOAP_TP_BASIS_CACHE_GB", "40")) * 2**30)


def context_for(state: MutableMapping[str, Any]) -> ParameterContext:
    key = (state["left_basis"].data_ptr(), state["right_basis"].data_ptr(),
           tuple(state["momentum"].shape))
    ctx = _CONTEXTS.get(key)
    if ctx is None:
        ctx = ParameterContext()
        rows, cols = state["momentum"].shape
        ctx.bytes = 12 * (rows * rows + cols * cols)
        _CONTEXTS[key] = ctx
    else:
        _CONTEXTS.move_to_end(key)
        return ctx                     # (nothing was added)
    total = sum(c.bytes for c in _CONTEXTS.values())
    if total > BASIS_CACHE_BYTES or len(_CONTEXTS) > 4096:
        # contexts of tensors that no longer exist go first; then the MOST recently used ones: an optimizer walks
        # its parameters in the same order every step, so the oldest contexts are the next to be used
        dead = [other for other, c in _CONTEXTS.items()
                if other != key and c.left.owner is not None and c.left.owner() is None]
        for other in dead + [other for other in reversed(_CONTEXTS) if other != key and other not in dead]:
            if total <= BASIS_CACHE_BYTES and len(_CONTEXTS) <= 4096:
                break
            total -= _CONTEXTS.pop(other).bytes
    return ctx


CLASSIC_TAGS = {"P", "Qtmp"}      # operands of the power iteration, which feeds the QR: always 3xTF32


def _operand(depth: int, cols: int, device, *, blocked: bool = False, terms: int = 2):
    """Uninitialised operand planes for the products of the optimizer step."""
    if k.MIXED_CORRECTIONS:
        return k.HalfPlanes.empty(depth, cols, device, blocked=blocked, terms=terms)
    return k.Planes.empty(depth, cols, device)


def _tf32_operand(depth: int, cols: int, device) -> k.Planes:
    return k.Planes.empty(depth, cols, device, mixed=k.MIXED_CORRECTIONS)


def split(source: Tensor, plain=None, turned=None) -> None:
    """Write a matrix as operand planes: ``plain`` is the operand ``source`` itself, ``turned`` its transpose."""
    if isinstance(plain if plain is not None else turned, k.HalfPlanes):
        k.half_planes(source, plain, turned)
        return
    k.split_planes_both(source, plain, turned)


def product(a, b, **epilogue) -> None:
    """``a^T b`` with a fused epilogue, by the kernel that the operands' form belongs to."""
    (k.gemm_half if isinstance(a, k.HalfPlanes) else k.gemm)(a, b, **epilogue)


def workspace_planes(tag: str, depth: int, cols: int, device, *, blocked: bool = False, terms: int = 2, slot: int = 0):
    """Scratch operand planes shared by every parameter of the same shape on ``device``.  ``blocked``: written by a
    product's epilogue; ``terms=1``: written from bf16 values; ``slot``: one more set, for steps that share launches."""
    key = (tag, depth, cols, str(device), terms, blocked, k.MIXED_CORRECTIONS and tag not in CLASSIC_TAGS, slot)
    planes = _WORKSPACES.get(key)
    if planes is None:
        planes = (k.Planes.empty(depth, cols, device) if tag in CLASSIC_TAGS
                  else _operand(depth, cols, device, blocked=blocked, terms=terms))
        _WORKSPACES[key] = planes
    return planes


def workspace_matrix(tag: str, rows: int, cols: int, device) -> Tensor:
    key = ("m", tag, rows, cols, str(device))
    matrix = _WORKSPACES.get(key)
    if matrix is None:
        matrix = torch.empty((max(1, cols), max(1, rows)), dtype=torch.float32, device=device).T
        _WORKSPACES[key] = matrix
    return matrix


def release_workspaces() -> None:
    _WORKSPACES.clear()
    _CONTEXTS.clear()


def gradient_planes(gradient: Tensor, *, plain: Optional[str] = None, turned: Optional[str] = None) -> tuple:
    """Planes of G (depth = rows) and of G^T (depth = columns) in the workspaces of these names; one term for bf16."""
    g = gradient.detach()
    if g.dtype != torch.bfloat16:
        g = g.float()
    terms = 1 if g.dtype == torch.bfloat16 else 2
    rows, cols = g.shape
    xp = workspace_planes(plain, rows, cols, g.device, terms=terms) if plain else None
    gtp = workspace_planes(turned, cols, rows, g.device, terms=terms) if turned else None
    split(g, xp, gtp)
    return xp, gtp


def tf32_workspace(tag: str, depth: int, cols: int, device, slot: int = 0) -> k.Planes:
    """Scratch planes of the tf32 form with bf16 corrections (``kernels.Planes``, mixed)."""
    key = ("tf32", tag, depth, cols, str(device), slot)
    planes = _WORKSPACES.get(key)
    if planes is None:
        planes = _WORKSPACES[key] = _tf32_operand(depth, cols, device)
    return planes


def rotate_planes(source, first, second, rows: int, cols: int, device, *, tag: str, **final) -> None:
    """``final epilogue( (source^T first)^T second )`` -- two chained GEMMs through scratch planes."""
    middle = workspace_planes(tag, source.cols, first.cols, device, blocked=True)
    product(source, first, mode=k.EPI_SPLIT, out_planes=middle)
    product(middle, second, **final)


def gram_updates(xp, gtp, state, beta: float, rows: int, cols: int, between=None) -> None:
    product(gtp, gtp, out=state["left_preconditioner"][:rows, :rows], alpha=1.0 - beta, beta=beta, symmetric=True)
    if between is not None:
        between()
    product(xp, xp, out=state["right_preconditioner"][:cols, :cols], alpha=1.0 - beta, beta=beta, symmetric=True)


def gram_updates_for_bases(gradient: Tensor, state, beta: float, rows: int, cols: int, between=None) -> None:
    """The averages of a step that derives bases from them (the first one, and those with a refresh), on tf32 planes like
    everything else that is factored.

    The QR panel kernels take the sign of a basis's last column from a rounding residue (``|x|^2 - x_1^2`` of a column of one
    element), so that column and what is expressed in it would change sign with the last bits of the averages.  These keep
    the products they have always been formed with: the same gradient and state give the same bases, not the same ones up
    to a sign."""
    gp, gtp = tf32_workspace("G", rows, cols, gradient.device), tf32_workspace("GT", cols, rows, gradient.device)
    split(gradient.detach(), gp, gtp)
    gram_updates(gp, gtp, state, beta, rows, cols, between)


class _Scratch:
    """Buffers of a rotation as the native calls take them, shared by matrices of one shape: with ``update`` those of a step's
    way back as well, with ``averages`` the planes of its Gram products.  ``slots``: which set of them, of the mixed form of the
    left basis, and of the right one's (steps that share launches, ``shared_steps``)."""

    def __init__(self, rows: int, cols: int, device, terms: int, update: bool, averages: bool, slots: tuple) -> None:
        slot, left, right = slots
        self.wide = torch.zeros(1, dtype=torch.int32, device=device)        # the decision on the range
        self.maxima = torch.empty(max(1, rows), dtype=torch.int32, device=device)
        planes = [workspace_planes("X", rows, cols, device, terms=terms, slot=slot)]
        if averages:
            planes.append(workspace_planes("GT", cols, rows, device, terms=terms, slot=slot))
        middle = workspace_planes("T", cols, rows, device, blocked=True, slot=slot)
        mixed = [tf32_workspace(tag, depth, width, device, which) for tag, depth, width, which in (
            ("G", rows, cols, slot), ("T", cols, rows, slot), ("L", rows, rows, left), ("LT", rows, rows, left),
            ("R", cols, cols, right), ("RT", cols, cols, right))]
        turned = planes[1].target() if averages else (0, 0, 64, 0, self.maxima.data_ptr())
        addresses = (planes[0].target() + turned + middle.operand() + (self.wide.data_ptr(), int(k.SPLIT_ROUND_NEAREST))
                     + tuple(value for each in mixed for value in each.mixed_target()))
        self.keep = planes + [middle] + mixed                               # (addresses alone hold nothing)
        if update:
            update_planes = workspace_planes("U", rows, cols, device, blocked=True, slot=slot)
            mixed_update = tf32_workspace("U", rows, cols, device, slot)
            addresses += update_planes.operand() + mixed_update.mixed_target()
            self.keep += [update_planes, mixed_update]
        self.native = _C.RotationScratch(rows, cols, addresses)


_FIRST = (0, 0, 0)


def _scratch(rows: int, cols: int, device, terms: int, update: bool = False, averages: bool = False, slots: tuple = _FIRST) -> _Scratch:
    key = ("scratch", rows, cols, device, terms, update, averages, slots)
    entry = _WORKSPACES.get(key)
    if entry is None:
        entry = _WORKSPACES[key] = _Scratch(rows, cols, device, terms, update, averages, slots)
    return entry


def rotate_matrix(source: Tensor, left: BasisPlanes, right: BasisPlanes, turned: bool, out: Tensor) -> None:
    """``out <- Q_l^T X Q_r`` (``turned``: ``Q_l X Q_r^T``) for an fp32 matrix; ``out`` is column-major and may be ``source``."""
    rows, cols = source.shape
    if k.MIXED_CORRECTIONS:
        if rows and cols:
            k.rotate_half(_scratch(rows, cols, source.device, 2).native, left.native, right.native, source, turned, out)
        return
    planes = workspace_planes("X", rows, cols, source.device)
    split(source, planes)
    first, second = (left.transposed, right.transposed) if turned else (left.plain, right.plain)
    rotate_planes(planes, first, second, rows, cols, source.device, tag="T", mode=k.EPI_STORE, out=out)


# SOAP_TP_OVERLAP_GRAM=0: the Gram averages run after the rotations on the same stream instead of beside them
OVERLAP_GRAM = os.environ.get("SOAP_TP_OVERLAP_GRAM", "1") != "0"
_SIDE_STREAMS: Dict[tuple, "torch.cuda.Stream"] = {}


def _side_stream(device, home: int) -> int:
    """The stream of the averages of steps on the stream ``home`` (forked from and joined to it within every step): one of its
    own for every caller's stream, so that callers do not wait for one another, and of that stream's priority."""
    if not OVERLAP_GRAM:
        return home
    stream = _SIDE_STREAMS.get((device, home))
    if stream is None:
        if len(_SIDE_STREAMS) >= 64:          # (streams that came and went; nothing is left on theirs)
            _SIDE_STREAMS.clear()
        stream = torch.cuda.Stream(device=device, priority=torch.cuda.current_stream().priority)
        _SIDE_STREAMS[(device, home)] = stream
    return stream.cuda_stream


def _native_arguments(gradient: Tensor, state, step: int, rows: int, cols: int, averages: bool, slots: tuple, *, beta, beta1, beta2,
                      eps) -> tuple:
    """An ordinary step as the native call takes it: scratch, bases, addresses and scalars; then the tensor of its result."""
    g = gradient if gradient.shape == (rows, cols) else gradient.detach().reshape(rows, cols)
    if g.dtype != torch.float32 and g.dtype != torch.bfloat16:
        g = g.detach().float()
    ctx = context_for(state)
    ctx.left.refresh(state["left_basis"], rows)
    ctx.right.refresh(state["right_basis"], cols)
    bias2 = 1.0 - beta2**step
    momentum, variance = state["momentum"], state["variance"]
    left, right = state["left_preconditioner"], state["right_preconditioner"]
    scratch = _scratch(rows, cols, g.device, 1 if g.dtype == torch.bfloat16 else 2, update=True, averages=averages, slots=slots)
    update = torch.empty((rows, cols), dtype=torch.float32, device=g.device)
    arguments = (k.strided_source(g)
                 + (momentum.data_ptr(), k._ld(momentum), variance.data_ptr(), k._ld(variance), update.data_ptr(),
                    left.data_ptr(), k._ld(left), right.data_ptr(), k._ld(right)))
    scalars = (beta, beta1, beta2, eps / math.sqrt(bias2), 1.0 / (1.0 - beta1**step), 1.0 / math.sqrt(bias2))
    # (the gradient and the planes of the bases are held until the launches are issued)
    return (scratch.native, ctx.left.native, ctx.right.native, arguments, scalars), update, (g, ctx)


def _count_launches(averages: int, planes: int = 1) -> None:
    """Of one step, or of several that share launches; ``averages``, ``planes``: the launches of their averages and of their planes."""
    for name, count in (("clear_kernel", planes), ("largest_kernel", planes), ("half_planes_kernel", planes),
                        ("gemm_half_kernel", 4 + averages)):
        k.LAUNCH_COUNTS[name] = k.LAUNCH_COUNTS.get(name, 0) + count


_WRITTEN = ("momentum", "variance", "left_preconditioner", "right_preconditioner")


def _native_step(gradient: Tensor, state, step: int, rows: int, cols: int, *, beta, beta1, beta2, eps, averages: bool) -> Tensor:
    """An ordinary step, its launches issued by one native call; without ``averages`` the rotations and Adam only."""
    call, update, held = _native_arguments(gradient, state, step, rows, cols, averages, _FIRST, beta=beta, beta1=beta1, beta2=beta2, eps=eps)
    home = k._stream()
    tail = (k.status_word(update.device).data_ptr(), home, _side_stream(update.device, home))
    if TIMER.enabled:
        for name, phase in _STEP_STAGES if averages else _STEP_STAGES[:-1]:
            with TIMER.stage(name, update.device):
                _C.steady_step(*call, phase, *tail)
    else:
        _C.steady_step(*call, _ALL_PHASES if averages else _ALL_PHASES - _C.STEP_AVERAGES, *tail)
    torch.autograd.graph.increment_version([state[name] for name in (_WRITTEN if averages else _WRITTEN[:2])])
    _count_launches((1 if _C.averages_share(rows, cols) else 2) if averages else 0)
    return update


def shares_launches(state, rows: int, cols: int, interval: int) -> bool:
    """Whether the next step of this parameter is an ordinary one whose launches it can share with other small parameters'."""
    return (k.MIXED_CORRECTIONS and not TIMER.enabled and "left_basis" in state and interval > 0 and (int(state["step"]) + 1) % interval != 0
            and _C.steady_step_shares(rows, cols))


@functools.lru_cache(maxsize=1024)
def _scratch_numbers(shapes: tuple) -> tuple:
    """Which sets of scratch matrices of these shapes take that run together (``_Scratch``, ``slots``): each has its own, those of one
    shape, and of the mixed form of bases of one size whatever the other side (workspaces of other tags or sizes are others)."""
    whole, lefts, rights, numbers = Counter(), Counter(), Counter(), []
    for rows, cols in shapes:
        numbers.append((whole[rows, cols], lefts[rows], rights[cols]))
        for count, key in ((whole, (rows, cols)), (lefts, rows), (rights, cols)):
            count[key] += 1
    return tuple(numbers)


def shared_steps(parameters, *, beta: float, beta1: float, beta2: float, eps: float) -> list:
    """Ordinary steps of several small parameters, ``(gradient, state, rows, cols)`` each, on one device; their updates.

    A product of a small matrix leaves most of the GPU idle and ends in latencies (fill, drain, epilogue, launch) that are as
    long as its work; eight of them in one launch take about as long as one (seven matrices of a decoder layer of hidden size 512:
    921 us one after another, 405 together)."""
    for _, state, rows, cols in parameters:
        _check_state(state, rows, cols)
    updates = []
    for first in range(0, len(parameters), _C.STEP_GROUP):
        some = parameters[first:first + _C.STEP_GROUP]
        calls, held = [], []
        numbers = _scratch_numbers(tuple([(rows, cols) for _, _, rows, cols in some]))
        for (gradient, state, rows, cols), slots in zip(some, numbers):
            call, update, holds = _native_arguments(gradient, state, int(state["step"]) + 1, rows, cols, True, slots, beta=beta,
                                                    beta1=beta1, beta2=beta2, eps=eps)
            calls.append(call)
            held.append(holds)
            updates.append(update)
        device, home = updates[-1].device, k._stream()
        _C.steady_steps(calls, k.status_word(device).data_ptr(), home, _side_stream(device, home))
        torch.autograd.graph.increment_version([state[name] for _, state, _, _ in some for name in _WRITTEN])
        for _, state, _, _ in some:
            state["step"] = int(state["step"]) + 1
        _count_launches(-(-2 * len(some) // _C.STEP_GROUP), len({g.dtype for g, _ in held}))
    return updates


_STEP_STAGES = (("split_gradient", _C.STEP_PLANES), ("rotate_forward+adam", _C.STEP_FORWARD),
                ("rotate_backward", _C.STEP_BACKWARD), ("gram", _C.STEP_AVERAGES))
_ALL_PHASES = sum(phase for _, phase in _STEP_STAGES)


def _tf32_step(gradient: Tensor, state, step: int, rows: int, cols: int, *, beta, beta1, beta2, eps, averages: bool) -> Tensor:
    """The same on tf32 planes, launch by launch (``SOAP_TP_MIXED_CORRECTIONS=0``)."""
    device = gradient.device
    with TIMER.stage("split_gradient", device):
        xp, gtp = gradient_planes(gradient.reshape(rows, cols), plain="X", turned="GT" if averages else None)
    ctx = context_for(state)
    ctx.left.refresh(state["left_basis"], rows)
    ctx.right.refresh(state["right_basis"], cols)
    bias2 = 1.0 - beta2**step
    adam = dict(beta1=beta1, beta2=beta2, eps=eps / math.sqrt(bias2),
                bias_correction1=1.0 - beta1**step, bias_correction2=bias2)
    up = workspace_planes("U", rows, cols, device, blocked=True)
    with TIMER.stage("rotate_forward+adam", device):
        rotate_planes(xp, ctx.left.plain, ctx.right.plain, rows, cols, device, tag="T",
                      mode=k.EPI_ADAM, out_planes=up, momentum=state["momentum"][:rows, :cols],
                      variance=state["variance"][:rows, :cols], adam=adam)
    update = torch.empty((rows, cols), dtype=torch.float32, device=device)
    with TIMER.stage("rotate_backward", device):
        rotate_planes(up, ctx.left.transposed, ctx.right.transposed, rows, cols, device, tag="T",
                      mode=k.EPI_ROW_MAJOR, out=update)
    if averages:
        with TIMER.stage("gram", device):
            gram_updates(xp, gtp, state, beta, rows, cols)
    return update


def _check_state(state: MutableMapping[str, Any], rows: int, cols: int) -> None:
    """The kernels write these buffers through raw pointers: fp32, of at least their matrix's size, column-major."""
    for name, height, width in (("momentum", rows, cols), ("variance", rows, cols), ("left_preconditioner", rows, rows),
                                ("right_preconditioner", cols, cols)):
        buffer = state[name]
        if buffer.dtype is torch.float32 and buffer.shape == (height, width) and buffer.stride() == (1, height):
            continue                      # as they are allocated
        if buffer.dtype != torch.float32:
            raise ValueError(f"state['{name}'] must use float32, got {buffer.dtype}.")
        if buffer.ndim != 2 or buffer.shape[0] < height or buffer.shape[1] < width:
            raise ValueError(f"state['{name}'] has shape {tuple(buffer.shape)}, smaller than {(height, width)}.")
        if (buffer.stride(0) != 1 and height > 1) or (buffer.stride(1) < height and width > 1):
            raise ValueError(f"state['{name}'] must be column-major, got strides {buffer.stride()}.")


def soap_step(
    gradient: Tensor,
    state: MutableMapping[str, Any],
    *,
    global_shape,
    beta: float,
    beta1: float,
    beta2: float,
    eps: float,
    interval: int,
    implementation: str,
    initializing: bool,
) -> Tensor:
    rows, cols = global_shape
    device = gradient.device
    if initializing:
        gram_updates_for_bases(gradient.reshape(rows, cols), state, beta, rows, cols)
        for side, size in (("left", rows), ("right", cols)):
            values = torch.empty(size, dtype=torch.float32, device=device)
            factor.symmetric_eigenbasis(
                state[f"{side}_preconditioner"][:size, :size], state[f"{side}_basis"][:size, :size],
                state[f"{side}_work"][:size, :size], values, implementation,
            )
        prepare_refresh(rows, cols, device)
        state["step"] = 0
        return torch.zeros((rows, cols), dtype=torch.float32, device=device)

    _check_state(state, rows, cols)
    step = int(state["step"]) + 1
    refreshing = step % interval == 0
    # (an empty matrix has nothing to rotate on pairs; the other path takes it as every product does)
    run = _native_step if k.MIXED_CORRECTIONS and rows and cols else _tf32_step
    scalars = dict(beta=beta, beta1=beta1, beta2=beta2, eps=eps)
    if not refreshing:
        update = run(gradient, state, step, rows, cols, averages=True, **scalars)
    else:
        # The averages first: the update does not depend on them, and runs beside the factorisations of the refresh, which leave most
        # of the GPU idle (chains of panels).  The left side's power iteration comes before the right side's average, so that its
        # factorisation starts earlier.
        orders = []

        def iterate(side: str, size: int) -> None:
            with TIMER.stage("refresh.power_iteration", device):
                order = estimated_order(state[f"{side}_preconditioner"], state[f"{side}_basis"], state[f"{side}_work"], size)
            orders.append((order, torch.cuda.Event()))
            orders[-1][1].record()

        with TIMER.stage("gram", device):
            gram_updates_for_bases(gradient.reshape(rows, cols), state, beta, rows, cols,
                                   None if TIMER.enabled else lambda: iterate("left", rows))
        if TIMER.enabled:
            iterate("left", rows)
        iterate("right", cols)
        update = None

        def issue_update() -> None:
            nonlocal update
            update = run(gradient, state, step, rows, cols, averages=False, **scalars)

        if TIMER.enabled:
            issue_update()                # (by itself, so that each stage's time is its own)
        with TIMER.stage("refresh", device):
            refresh(state, global_shape, orders, (lambda: None) if TIMER.enabled else issue_update)
    state["step"] = step
    return update


_WARMED: Dict[Any, bool] = {}


def warm_refresh_kernels(device, sizes=()) -> None:
    """Launch the kernels of a refresh once, on a tiny problem.

    CUDA loads a kernel's code the first time it is launched; without this the first refresh of a
    training run pays tens of milliseconds of module loading in the middle of a step.  (The tiles that products take at larger
    sizes are not among them: launching those here as well did not shorten a first refresh.)  The eigenvalue-order sort
    sizes its shared memory by length, so it is warmed at the real ``sizes``.
    """
    for size in sizes:
        if not _WARMED.get((str(torch.device(device)), "sort", size)):
            _WARMED[(str(torch.device(device)), "sort", size)] = True
            k.order_by_estimate(torch.rand((size, 2), device=device).T)
    key = str(torch.device(device))
    if _WARMED.get(key):
        return
    _WARMED[key] = True
    n = 384
    generator = torch.Generator(device=device).manual_seed(0)
    matrix = torch.randn(n, n, generator=generator, device=device).T
    out = torch.empty(n, n, device=device).T
    order = torch.randperm(n, generator=generator, device=device)
    factor_jobs = [(matrix.clone(), out, order), (matrix.clone(), torch.empty(n, n, device=device).T, None)]
    from . import qr as qr_driver

    qr_driver.householder_qr_pair(factor_jobs)
    qr_driver.householder_qr(matrix.clone(), out)      # a lone factorisation takes the forward-accumulation path
    estimated_order(matrix, out, torch.empty(n, n, device=device).T, n)
    k.gather2d(matrix, out, order, order)
    qr_driver.release_workspaces_for(n, device)


def prepare_refresh(rows: int, cols: int, device) -> None:
    """Allocate what a refresh needs at initialisation time, so that the first refresh in the middle of
    training launches kernels only."""
    from . import qr as qr_driver

    for size in {rows, cols}:
        workspace_planes("P", size, size, device)
        workspace_planes("Qtmp", size, size, device)
        qr_driver._workspace(size, device, 0)
    if rows == cols:
        qr_driver._workspace(cols, device, 1)     # the second of two concurrent factorisations
    else:
        qr_driver._workspace(rows, device, 0), qr_driver._workspace(cols, device, 1)
    for tag in ("perm", "space"):
        workspace_matrix(tag, rows, cols, device)
    if k.MIXED_CORRECTIONS and rows and cols:
        _scratch(rows, cols, device, 2)
    else:
        for tag, depth, width in (("X", rows, cols), ("T", cols, rows)):
            workspace_planes(tag, depth, width, device)
    warm_refresh_kernels(device, sizes={rows, cols})


def rotate(matrix: Tensor, Q_left: Tensor, Q_right: Tensor, global_shape, direction: str) -> Tensor:
    rows, cols = global_shape
    turned = direction != "forward"
    left, right = BasisPlanes().once(Q_left, rows, turned), BasisPlanes().once(Q_right, cols, turned)
    view = matrix[:rows, :cols]
    rotate_matrix(view, left, right, turned, view)
    return matrix


def estimated_order(P: Tensor, Q: Tensor, work: Tensor, size: int) -> Tensor:
    """``work <- P Q`` (P symmetric, so ``P^T Q``), estimates ``colsum(Q * work)``, stable descending order."""
    device = P.device
    pp = k.split_planes(P[:size, :size], out=workspace_planes("P", size, size, device))
    qp = k.split_planes(Q[:size, :size], out=workspace_planes("Qtmp", size, size, device))
    k.gemm(pp, qp, out=work[:size, :size])
    estimates = k.column_dot(Q, work, size, size)
    return k.order_by_estimate(estimates.view(1, size))


def power_iteration_qr(P: Tensor, Q: Tensor, work: Tensor, size: int) -> Tensor:
    order = estimated_order(P, Q, work, size)
    factor.householder_qr(work[:size, :size], Q[:size, :size], column_order=order)
    return order


def permute(matrix: Tensor, global_shape, row_order: Tensor, column_order: Tensor) -> Tensor:
    rows, cols = global_shape
    scratch = workspace_matrix("perm", rows, cols, matrix.device)
    view = matrix[:rows, :cols]
    k.gather2d(view, scratch, row_order, column_order)
    k.gather2d(scratch, view, None, None)
    return matrix


def refresh(state: MutableMapping[str, Any], global_shape, orders, issue_update) -> Tuple[Tensor, Tensor]:
    """QR of the power iteration's results on both sides (``orders``: the order of the columns and the event of both, per side) with
    momentum transport and variance permutation; ``issue_update`` issues the step's own update, which the momentum and variance
    come from.

    Neither it nor the momentum's way out of the old bases depends on the factorisations: at 8192 x 8192 16 of 86 ms that were
    spent before them run beside them now (a GPU-wide product delays a panel by what is left of its tiles, so 3.5 ms are gained;
    3000 x 2000 11.3 -> 10.8 ms)."""
    rows, cols = global_shape
    momentum, variance = state["momentum"], state["variance"]
    device = momentum.device
    (left_order, left_start), (right_order, right_start) = orders
    # momentum out of the old bases: Q_L M Q_R^T, in fp32 so that the way back sees the range of every row and column
    parameter_space = workspace_matrix("space", rows, cols, device)
    ctx = context_for(state)

    def beside() -> None:
        issue_update()
        ctx.left.refresh(state["left_basis"], rows)
        ctx.right.refresh(state["right_basis"], cols)
        with TIMER.stage("refresh.momentum_out", device):
            rotate_matrix(momentum[:rows, :cols], ctx.left, ctx.right, True, parameter_space)
        with TIMER.stage("refresh.permute_variance", device):
            permute(variance, global_shape, left_order, right_order)

    serial = os.environ.get("SOAP_TP_SERIAL_QR", "0") == "1"
    if serial or TIMER.enabled:
        beside()
    with TIMER.stage("refresh.qr", device):
        # the two factorisations are independent: issued on two streams they fill each other's gaps
        if serial:
            factor.householder_qr(state["left_work"][:rows, :rows], state["left_basis"][:rows, :rows], column_order=left_order)
            factor.householder_qr(state["right_work"][:cols, :cols], state["right_basis"][:cols, :cols], column_order=right_order)
        else:
            factor.householder_qr_pair([
                (state["left_work"][:rows, :rows], state["left_basis"][:rows, :rows], left_order),
                (state["right_work"][:cols, :cols], state["right_basis"][:cols, :cols], right_order)],
                None if TIMER.enabled else beside, (left_start, right_start))
    with TIMER.stage("refresh.momentum_in", device):
        ctx.left.refresh(state["left_basis"], rows)
        ctx.right.refresh(state["right_basis"], cols)
        rotate_matrix(parameter_space, ctx.left, ctx.right, False, momentum[:rows, :cols])
    return left_order, right_order
