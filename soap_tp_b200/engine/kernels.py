"""Python wrappers of the native kernels (module ``soap_tp_b200._C``).

Everything here launches this package's own sm_100a kernels on the current CUDA stream; there is
no eager-PyTorch fallback.  If the extension is missing it is built in place
(``soap_tp_b200.build_ext``); if that fails the import error propagates -- a CUDA tensor never
silently takes another path.
"""
from __future__ import annotations

import math
import os
import time
from dataclasses import dataclass, field
from typing import Dict, Optional

import torch
from torch import Tensor

try:
    from .. import _C  # type: ignore[attr-defined]
except ImportError:  # pragma: no cover - build on first use
    from .. import build_ext

    build_ext.build()
    from .. import _C  # type: ignore[attr-defined]

EPI_STORE, EPI_SPLIT, EPI_ADAM, EPI_ROW_MAJOR, EPI_PAIR_UPDATE, EPI_PUSH = 0, 1, 2, 3, 4, 5

STATUS_MESSAGES = {
    1: "GEMM consumer timed out waiting for a TMA stage",
    2: "GEMM producer timed out waiting for a free stage",
    3: "GEMM epilogue timed out waiting for the accumulator",
    4: "cross-rank barrier timed out",
    5: "bad kernel argument",
    6: "QR panel exchange between thread blocks timed out",
    7: "wait for a peer's data-ready flag timed out",
    8: "tridiagonalisation grid barrier timed out",
}

LAUNCH_COUNTS: Dict[str, int] = {}


def _count(name: str) -> None:
    LAUNCH_COUNTS[name] = LAUNCH_COUNTS.get(name, 0) + 1


def total_launches() -> int:
    """Number of kernels of this library launched by this process so far."""
    return sum(LAUNCH_COUNTS.values())


class SoapKernelError(RuntimeError):
    """A kernel of this library reported a bounded-wait timeout or a bad argument."""


class SoapCommTimeout(SoapKernelError):
    """A bounded device-side wait on a peer (barrier flag, data-ready flag) ran out."""


_STATUS: Dict[int, Tensor] = {}


def status_word(device: torch.device) -> Tensor:
    index = device.index if device.index is not None else torch.cuda.current_device()
    word = _STATUS.get(index)
    if word is None:
        word = torch.zeros(4, dtype=torch.int32, device=torch.device("cuda", index))
        _STATUS[index] = word
    return word


def _raise_for(index: int, code: int) -> None:
    kind = SoapCommTimeout if code in (4, 7) else SoapKernelError
    raise kind(f"cuda:{index}: {STATUS_MESSAGES.get(code, f'status {code}')}")


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronise and raise :class:`SoapKernelError` if any kernel gave up on a wait."""
    words = _STATUS.items() if device is None else [(device.index or 0, status_word(device))]
    for index, word in list(words):
        code = int(word[0].item())
        if code != 0:
            word.zero_()
            if index in _MONITORS:
                _MONITORS.pop(index).finish()
            _raise_for(index, code)


class _StatusMonitor:
    """Deferred read-back of one device's status word: a 4-byte copy into pinned memory per step, looked at
    one step later, so that a timed-out wait surfaces as an exception without a device synchronisation."""

    waited_seconds = 0.0      # host time spent waiting for the previous step's copy (all devices of the process)

    def __init__(self, index: int, on_device: bool = True) -> None:
        self.index = index
        self.host = torch.zeros(2, dtype=torch.int32)
        # `on_device=False` serves the host-side tests, which hand in a CPU tensor as the status word
        self.events = [torch.cuda.Event(), torch.cuda.Event()] if on_device else None
        if on_device:
            self.host = self.host.pin_memory()
        self.words = (self.host[0:1], self.host[1:2])
        self.pending = [False, False]
        self.turn = 0

    def poll(self, word: Tensor) -> None:
        previous = 1 - self.turn
        if self.pending[previous]:
            if self.events is not None:
                # recorded a whole step ago: complete unless the host runs a full step ahead of the device
                begin = time.perf_counter()
                self.events[previous].synchronize()
                _StatusMonitor.waited_seconds += time.perf_counter() - begin
            self.pending[previous] = False
            code = int(self.host[previous])
            if code != 0:
                word.zero_()
                self.pending = [False, False]
                _raise_for(self.index, code)
        if self.events is not None:
            _C.read_status(word.data_ptr(), self.words[self.turn].data_ptr(), _stream())
            self.events[self.turn].record()
        else:
            self.words[self.turn].copy_(word[:1])
        self.pending[self.turn] = True
        self.turn = previous

    def finish(self) -> None:
        """Waits for the copy in flight, on whatever stream: its pinned memory goes back to an allocator that does not know of it."""
        for event, pending in zip(self.events or (), self.pending):
            if pending:
                event.synchronize()


_MONITORS: Dict[int, _StatusMonitor] = {}


def poll_status(device: torch.device) -> None:
    """Called once per optimizer step on the step's stream.  Raises :class:`SoapKernelError` if the status
    word copied at the end of the PREVIOUS step was non-zero, then enqueues this step's copy.  A failure is
    therefore reported at most one step late and costs no synchronisation when nothing failed."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    monitor = _MONITORS.get(index)
    if monitor is None:
        monitor = _MONITORS[index] = _StatusMonitor(index)
    monitor.poll(status_word(torch.device("cuda", index)))


def mark_written(*tensors: Optional[Tensor]) -> None:
    """Bump the version counter of tensors a kernel wrote through a raw pointer, so that caches
    keyed on ``tensor._version`` (basis planes) notice the change."""
    for tensor in tensors:
        if tensor is not None:
            torch.autograd.graph.increment_version(tensor)


def _stream() -> int:
    """Handle of the current stream of the current device (every launch asks; the stream object costs 3 us to make)."""
    return _raw_stream(torch.cuda.current_device())


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", lambda index: torch.cuda.current_stream(index).cuda_stream)


def round_up(value: int, multiple: int) -> int:
    return -(-value // multiple) * multiple


# SOAP_TP_MIXED_CORRECTIONS=0 keeps every product on three tf32 MMAs per k-step.  By default the products of an ordinary
# single-GPU step, of rotations and of the one-sided step's average run on scaled fp16 pairs (``HalfPlanes``; rotations of
# matrices whose range asks for it on mixed planes); those of the multi-GPU engine, of the one-sided update and of averages that
# bases are derived from take their two correction terms as bf16 MMAs (``Planes``, mixed form); the factorisations (QR,
# eigensolvers, power iteration) always use the full 3xTF32 form.
MIXED_CORRECTIONS = os.environ.get("SOAP_TP_MIXED_CORRECTIONS", "1") != "0"


def use_cta_pairs(on: bool) -> None:
    """Large plain products (tf32 planes: at least 148 tiles of 128 x 256, each part of a split counted, no batching; fp16
    pairs: where they need fewer waves that way) run on CTA pairs (``cta_group::2``: 256 x 256 tiles, each CTA staging half of the B tile) unless
    switched off here or with ``SOAP_TP_GEMM_CTA_PAIRS=0``."""
    _C.gemm_use_cta_pairs(bool(on))


if os.environ.get("SOAP_TP_GEMM_CTA_PAIRS", "1") == "0":
    use_cta_pairs(False)


@dataclass
class Planes:
    """Operand planes of a K x cols column-major matrix ``x``.

    Classic form: ``hi = rn_tf32(x)`` and ``lo = x - hi`` in fp32; a product is three tf32 MMAs per k-step
    (``lo*hi + hi*lo + hi*hi``).  Mixed form (``hl`` present, ``lo`` absent): ``hi`` as before plus one bf16 plane
    that holds, for every 32 elements of K, the 32 values ``hb = bf16(x)`` followed by the 32 values
    ``lb = bf16(x - hi)`` (one 128-byte row per TMA box and k-block; elements past K are zero).  The two correction
    products then run as bf16 MMAs at twice the tf32 rate (their terms are 2^-11 of the main term, so bf16's 2^-9
    leaves about 2^-20), with the same bytes per element.  Both operands of a product must be of the same form.
    """

    hi: Tensor
    lo: Optional[Tensor]
    depth: int   # K: the contiguous, contracted extent
    cols: int
    ld: int
    hl: Optional[Tensor] = None
    ld16: int = 0
    # windows handed out by `sub` (a launch-heavy driver asks for the same few thousand windows at every refresh, and
    # slicing tensors is what its launching thread would otherwise spend its time on)
    _windows: Dict[tuple, "Planes"] = field(default_factory=dict, repr=False, compare=False)
    _pointers: Optional[tuple] = field(default=None, repr=False, compare=False)

    @property
    def mixed(self) -> bool:
        return self.hl is not None

    @property
    def device(self):
        return self.hi.device

    @staticmethod
    def empty(depth: int, cols: int, device, mixed: bool = False) -> "Planes":
        ld = max(4, round_up(depth, 4))
        if not mixed:
            storage = torch.empty((2, max(1, cols), ld), dtype=torch.float32, device=device)
            return Planes(storage[0], storage[1], depth, cols, ld)
        ld16 = 2 * round_up(max(1, depth), 32)
        hi = torch.empty((max(1, cols), ld), dtype=torch.float32, device=device)
        hl = torch.zeros((max(1, cols), ld16), dtype=torch.bfloat16, device=device)     # zeros: the tail past K stays zero
        return Planes(hi, None, depth, cols, ld, hl, ld16)

    def sub(self, k0: int, c0: int, depth: int, cols: int) -> "Planes":
        """Operand planes of the sub-matrix starting at row ``k0`` (a multiple of 4; of 32 for mixed planes, whose
        depth may only be shortened to a multiple of 32), column ``c0``.  Windows are cached: treat them as
        read-only descriptions of the parent's memory."""
        key = (k0, c0, depth, cols)
        window = self._windows.get(key)
        if window is not None:
            return window
        assert k0 + depth <= self.ld and c0 + cols <= self.hi.shape[0]
        if self.mixed:
            assert k0 % 32 == 0 and (k0 + depth == self.depth or depth % 32 == 0)
            window = Planes(self.hi[c0:, k0:], None, depth, cols, self.ld, self.hl[c0:, 2 * k0:], self.ld16)
        else:
            assert k0 % 4 == 0
            window = Planes(self.hi[c0:, k0:], self.lo[c0:, k0:], depth, cols, self.ld)
        if len(self._windows) < 65536:
            self._windows[key] = window
        return window

    def pointers(self) -> tuple:
        """hi, lo and pitch of classic planes for the native calls (windows are kept, so that this is looked up once for each)."""
        if self._pointers is None:
            self._pointers = (self.hi.data_ptr(), self.lo.data_ptr(), self.ld)
        return self._pointers

    def low_pointers(self) -> dict:
        """Pointer arguments of the low part for the native calls."""
        if self.mixed:
            return dict(lo=0, hl=self.hl.data_ptr(), ld16=self.ld16)
        return dict(lo=self.lo.data_ptr(), hl=0, ld16=0)

    def mixed_target(self) -> tuple:
        """Mixed planes as the native rotation takes them."""
        return (self.hi.data_ptr(), self.ld, self.hl.data_ptr(), self.ld16)

    def halves(self):
        """(hb, lb) of mixed planes as ``cols x depth`` fp32 tensors (tests)."""
        groups = self.hl[: max(1, self.cols)].view(max(1, self.cols), -1, 2, 32).float()
        hb = groups[:, :, 0, :].reshape(max(1, self.cols), -1)[: self.cols, : self.depth]
        lb = groups[:, :, 1, :].reshape(max(1, self.cols), -1)[: self.cols, : self.depth]
        return hb, lb

    def dense(self) -> Tensor:
        """The represented K x cols matrix (for tests; to bf16 accuracy of the low part for mixed planes)."""
        low = self.halves()[1] if self.mixed else self.lo[: self.cols, : self.depth]
        return (self.hi[: self.cols, : self.depth] + low).T


HALF_SCALE_BLOCK = 128      # rows of a result that share one scale per column when it becomes the next operand


@dataclass
class HalfPlanes:
    """Operand of a single-GPU product as scaled fp16 planes of a K x cols matrix (``csrc/gemm_half.h``).

    ``x = scale * (h + l)`` with ``h``, ``l`` fp16 (22 to 24 bits of x, or to 2^-39 of the largest element that shares the
    scale) and ``scale`` a power of two per K-vector (``blocked=False``: what ``half_planes`` makes, usable on either side of
    a product) or per K-vector and block of 128 (``blocked=True``: what a product's epilogue writes, usable as the first
    operand).  ``l`` is absent where the matrix comes from bf16 values, which ``h`` holds by itself down to 2^-32 of the
    largest.  Rotations (``rotate_half``, ``steady_step``) decide on the device whether that is enough.
    """

    h: Tensor
    l: Optional[Tensor]
    scale: Tensor               # (cols,) or (blocks, cols)
    depth: int
    cols: int
    ld: int
    blocked: bool
    largest: Optional[Tensor] = None      # scratch of ``half_planes``: the largest magnitude of every vector

    @staticmethod
    def empty(depth: int, cols: int, device, *, blocked: bool = False, terms: int = 2) -> "HalfPlanes":
        ld = round_up(max(1, depth), 64)
        planes = torch.empty((terms, max(1, cols), ld), dtype=torch.float16, device=device)
        blocks = -(-max(1, depth) // HALF_SCALE_BLOCK) if blocked else 1
        scale = torch.empty((blocks, max(1, cols)), dtype=torch.float32, device=device)
        largest = None if blocked else torch.empty(max(1, cols), dtype=torch.int32, device=device)
        return HalfPlanes(planes[0], planes[1] if terms == 2 else None, scale, depth, cols, ld, blocked, largest)

    @property
    def terms(self) -> int:
        return 1 if self.l is None else 2

    @property
    def device(self):
        return self.h.device

    def dense(self) -> Tensor:
        """The represented K x cols matrix in fp64 (tests)."""
        total = self.h[: self.cols, : self.depth].double()
        if self.l is not None:
            total = total + self.l[: self.cols, : self.depth].double()
        scale = self.scale.double()[:, : self.cols]
        if self.blocked:
            scale = scale.repeat_interleave(HALF_SCALE_BLOCK, dim=0)[: self.depth]
        return total.T * scale

    def target(self) -> tuple:
        return (self.h.data_ptr(), 0 if self.l is None else self.l.data_ptr(), self.ld, self.scale.data_ptr(),
                self.largest.data_ptr())

    def operand(self) -> tuple:
        return (self.h.data_ptr(), 0 if self.l is None else self.l.data_ptr(), self.ld, self.scale.data_ptr(),
                self.scale.shape[1] if self.blocked else 0)


_NO_TARGET = (0, 0, 64, 0, 0)


def half_planes(source: Tensor, plain: Optional[HalfPlanes] = None, turned: Optional[HalfPlanes] = None) -> None:
    """Write a 2-D tensor (any strides; fp32 or bf16) as scaled fp16 planes: ``plain`` is the operand ``source`` itself,
    ``turned`` its transpose.  One-term planes take bf16 sources only."""
    rows, cols = source.shape
    if source.dtype not in (torch.float32, torch.bfloat16):
        source = source.float()
    for planes, shape in ((plain, (rows, cols)), (turned, (cols, rows))):
        if planes is not None:
            assert (planes.depth, planes.cols) == shape and not planes.blocked
            assert planes.terms == 2 or source.dtype == torch.bfloat16
    _C.half_planes(source.data_ptr(), int(source.dtype == torch.bfloat16), source.stride(0), source.stride(1), rows, cols,
                   *(plain.target() if plain is not None else _NO_TARGET),
                   *(turned.target() if turned is not None else _NO_TARGET), _stream())
    _count("clear_kernel")
    _count("largest_kernel")
    _count("half_planes_kernel")


def gemm_half(a: HalfPlanes, b: HalfPlanes, *, mode: int = EPI_STORE, out: Optional[Tensor] = None,
              out_planes: Optional[HalfPlanes] = None, alpha: float = 1.0, beta: float = 0.0, symmetric: bool = False,
              momentum: Optional[Tensor] = None, variance: Optional[Tensor] = None, adam: Optional[dict] = None,
              tiles: int = 0) -> None:
    """``acc[m, n] = sum_k a[k, m] * b[k, n]`` on scaled fp16 planes, then the fused epilogue; arguments as :func:`gemm`.
    ``tiles``: 1 single CTAs, 2 CTA pairs, 0 by size."""
    assert a.depth == b.depth, (a.depth, b.depth)
    M, N, K = a.cols, b.cols, a.depth
    if M == 0 or N == 0:
        return
    c = ldc = mom = ldm = var = ldv = 0
    target = (0, 0, 64, 0, 0)
    moments = (0.0, 0.0, 0.0, 0.0, 0.0)
    if out is not None:
        c = out.data_ptr()
        ldc = (out.stride(0) if M > 1 else max(1, N)) if mode == EPI_ROW_MAJOR else _ld(out)
        assert (out.stride(1) == 1 or N == 1) if mode == EPI_ROW_MAJOR else (out.stride(0) == 1 or M == 1)
    if out_planes is not None:
        assert out_planes.blocked and out_planes.depth == M and out_planes.cols == N
        target = out_planes.operand()
    if mode == EPI_ADAM:
        mom, ldm, var, ldv = momentum.data_ptr(), _ld(momentum), variance.data_ptr(), _ld(variance)
        moments = (adam["beta1"], adam["beta2"], adam["eps"], 1.0 / adam["bias_correction1"],
                   1.0 / math.sqrt(adam["bias_correction2"]))
    _C.gemm_half(*a.operand(), *b.operand(), M, N, K, mode, int(symmetric), tiles, alpha, beta, c, ldc, *target, mom, ldm,
                 var, ldv, *moments, status_word(a.device).data_ptr(), _stream())
    mark_written(out, momentum, variance)
    _count("gemm_half_kernel")


SPLIT_ROUND_NEAREST = os.environ.get("SOAP_TP_SPLIT_NEAREST", "1") == "1"


def split_planes(source: Tensor, *, transpose: bool = False, out: Optional[Planes] = None, scale: float = 1.0,
                 nearest: Optional[bool] = None, mixed: bool = False) -> Planes:
    """Split a 2-D fp32 tensor (any strides) into operand planes (of the form of ``out``, else of ``mixed``).

    The operand is ``source`` itself (``depth = rows``) or, with ``transpose=True``, its transpose.
    """
    if source.dtype != torch.float32:
        source = source.float()
    rows, cols = source.shape
    s_i, s_j = source.stride()
    if transpose:
        rows, cols, s_i, s_j = cols, rows, s_j, s_i
    if out is None:
        out = Planes.empty(rows, cols, source.device, mixed=mixed)
    assert out.depth == rows and out.cols == cols
    low = out.low_pointers()
    _C.split_planes(source.data_ptr(), s_i, s_j, out.hi.data_ptr(), low["lo"], out.ld, rows, cols,
                    float(scale), int(SPLIT_ROUND_NEAREST if nearest is None else nearest), _stream(),
                    hl=low["hl"], ld16=low["ld16"])
    _count("split_planes_kernel")
    return out


def split_planes_both(source: Tensor, plain: Optional[Planes] = None, turned: Optional[Planes] = None) -> None:
    """Operand planes of a 2-D fp32 or bf16 tensor (any strides) and of its transpose in one pass over it."""
    if source.dtype not in (torch.float32, torch.bfloat16):
        source = source.float()
    rows, cols = source.shape
    arguments = []
    for planes, shape in ((plain, (rows, cols)), (turned, (cols, rows))):
        if planes is None:
            arguments += (0, 0, 0, 0, 0)
            continue
        assert (planes.depth, planes.cols) == shape
        low = planes.low_pointers()
        arguments += (planes.hi.data_ptr(), low["lo"], planes.ld, low["hl"], low["ld16"])
    _C.split_planes_both(source.data_ptr(), int(source.dtype == torch.bfloat16), source.stride(0), source.stride(1), rows, cols,
                         *arguments, int(SPLIT_ROUND_NEAREST), _stream())
    _count("split_planes_kernel")


def gemm(
    a: Planes,
    b: Planes,
    *,
    mode: int = EPI_STORE,
    out: Optional[Tensor] = None,
    out_ld: Optional[int] = None,
    out_planes: Optional[Planes] = None,
    alpha: float = 1.0,
    beta: float = 0.0,
    symmetric: bool = False,
    momentum: Optional[Tensor] = None,
    variance: Optional[Tensor] = None,
    adam: Optional[dict] = None,
    force_narrow: bool = False,
    k_splits: int = 1,
    split_stride: int = 0,
    batch: Optional[dict] = None,
    lower_of_grid: Optional[tuple] = None,
    push: Optional[dict] = None,
    second_exact: bool = False,
) -> None:
    """``acc[m, n] = sum_k a[k, m] * b[k, n]`` then the fused epilogue (see ``csrc/gemm.h``).

    ``out`` is a column-major ``M x N`` view for ``EPI_STORE`` (and the optional plain copy of
    ``EPI_SPLIT``/``EPI_ADAM``) or a row-major ``M x N`` tensor for ``EPI_ROW_MAJOR``.  ``EPI_PUSH`` writes no
    local output: ``push`` = ``dict(table, ld, ld16, nb, Pr, Pc, pr, pc, mixed)`` names the operand planes of the
    consuming ranks (``csrc/gemm.h``, ``kEpiPush``), which the epilogue fills through peer pointers.
    ``second_exact``: ``b`` comes from bf16 values; a product of mixed planes then leaves out the terms that are zero.
    """
    if batch is None:
        assert a.depth == b.depth, (a.depth, b.depth)
        M, N, K = a.cols, b.cols, a.depth
    else:
        M, N, K = batch["M"], batch["N"], batch["K"]   # per batch item; a and b describe the whole buffers
    if M == 0 or N == 0:
        return
    if batch is None and lower_of_grid is None and (mode == EPI_SPLIT or mode == EPI_STORE) and a.hl is None and b.hl is None and (
            out_planes is None or out_planes.hl is None):
        c_ptr = ldc = 0
        if out is not None:
            assert out.stride(0) == 1 or out.shape[0] == 1
            c_ptr, ldc = out.data_ptr(), out_ld if out_ld is not None else _ld(out)
        target = (0, 0, 0)
        if out_planes is not None:
            assert out_planes.depth == M and out_planes.cols == N
            target = out_planes.pointers()
        _C.gemm_planes((*a.pointers(), *b.pointers(), M, N, K, mode, int(symmetric), int(force_narrow), c_ptr, ldc, *target, k_splits,
                        split_stride, status_word(a.device).data_ptr(), _stream()), alpha, beta)
        mark_written(out)
        _count("gemm_tf32x3_kernel")
        return
    c_ptr, ldc = 0, 0
    if out is not None:
        c_ptr = out.data_ptr()
        if mode == EPI_ROW_MAJOR:
            assert out.stride(1) == 1 or out.shape[1] == 1
            ldc = out.stride(0) if out.shape[0] > 1 else max(1, out.shape[1])
        else:
            assert out.stride(0) == 1 or out.shape[0] == 1
            ldc = out_ld if out_ld is not None else (out.stride(1) if out.shape[1] > 1 else max(1, out.shape[0]))
    if a.mixed != b.mixed:
        raise ValueError("both operands of a product must be classic planes or both mixed planes.")
    chi = clo = ldp = 0
    mixed_arguments = {}
    if a.mixed:
        mixed_arguments.update(a_hl=a.hl.data_ptr(), lda16=a.ld16, b_hl=b.hl.data_ptr(), ldb16=b.ld16, b_exact=int(second_exact))
    if out_planes is not None:
        assert batch is not None or (out_planes.depth == M and out_planes.cols == N)
        low = out_planes.low_pointers()
        chi, clo, ldp = out_planes.hi.data_ptr(), low["lo"], out_planes.ld
        if out_planes.mixed:
            assert beta == 0.0, "mixed output planes cannot be read-modify-written"
            mixed_arguments.update(Chl=low["hl"], ldp16=low["ld16"])
    mom = var = ldm = ldv = 0
    b1 = b2 = eps = ibc1 = isbc2 = 0.0
    if mode == EPI_ADAM:
        assert momentum is not None and variance is not None and adam is not None
        mom, var = momentum.data_ptr(), variance.data_ptr()
        ldm = momentum.stride(1) if momentum.shape[1] > 1 else max(1, momentum.shape[0])
        ldv = variance.stride(1) if variance.shape[1] > 1 else max(1, variance.shape[0])
        b1, b2, eps = adam["beta1"], adam["beta2"], adam["eps"]
        ibc1, isbc2 = 1.0 / adam["bias_correction1"], 1.0 / math.sqrt(adam["bias_correction2"])
    push_arguments = {}
    if mode == EPI_PUSH:
        assert push is not None and batch is None and k_splits == 1 and not symmetric
        push_arguments = dict(push_table=push["table"].data_ptr(), push_ld=int(push["ld"]), push_ld16=int(push["ld16"]),
                              push_nb=int(push["nb"]), push_Pr=int(push["Pr"]), push_Pc=int(push["Pc"]),
                              push_pr=int(push["pr"]), push_pc=int(push["pc"]), push_mixed=int(bool(push["mixed"])))
    status = status_word(a.hi.device)
    _C.gemm_tf32x3(a.hi.data_ptr(), a.low_pointers()["lo"], a.ld, b.hi.data_ptr(), b.low_pointers()["lo"], b.ld, M, N, K,
                   mode, 2 if lower_of_grid is not None else int(symmetric), int(force_narrow), float(alpha), float(beta), c_ptr, ldc, chi, clo, ldp,
                   mom, var, ldm, ldv, b1, b2, eps, ibc1, isbc2, int(k_splits), int(split_stride), status.data_ptr(),
                   _stream(), **_batch_arguments(a, b, batch), **_triangle_arguments(lower_of_grid), **mixed_arguments,
                   **push_arguments)
    mark_written(out, momentum, variance)
    _count("gemm_tf32x3_kernel")


def _triangle_arguments(lower_of_grid: Optional[tuple]) -> dict:
    """``(block_size, pr, Pr, pc, Pc[, m0, n0])``: produce only the entries of this rank's packed block that
    lie on or below the global diagonal of a symmetric result; ``m0, n0`` is the local index of the output's
    first element when the output is a window of the packed block."""
    if lower_of_grid is None:
        return {}
    nb, pr, Pr, pc, Pc = lower_of_grid[:5]
    m0, n0 = (lower_of_grid[5], lower_of_grid[6]) if len(lower_of_grid) > 5 else (0, 0)
    return dict(tri_nb=int(nb), tri_pr=int(pr), tri_Pr=int(Pr), tri_pc=int(pc), tri_Pc=int(Pc), tri_m0=int(m0),
                tri_n0=int(n0))


def _batch_arguments(a: "Planes", b: "Planes", batch: Optional[dict]) -> dict:
    """Keyword arguments of the batched launch (see ``csrc/gemm.h``): ``a`` and ``b`` are the whole operand
    buffers, the per-item sub-blocks start at multiples of the ``*_step`` values."""
    if batch is None:
        return {}
    second = batch.get("out2_planes")
    remap = batch.get("remap")
    return dict(
        batches=int(batch["count"]), a_k_step=int(batch.get("a_k_step", 0)), a_row_step=int(batch.get("a_row_step", 0)),
        b_k_step=int(batch.get("b_k_step", 0)), b_row_step=int(batch.get("b_row_step", 0)),
        c_batch_stride=int(batch.get("c_batch_stride", 0)), a_k_total=a.depth, a_rows_total=a.cols, b_k_total=b.depth,
        b_rows_total=b.cols, remap=remap.data_ptr() if remap is not None else 0,
        C2hi=second.hi.data_ptr() if second is not None else 0, C2lo=second.lo.data_ptr() if second is not None else 0,
        ld2=second.ld if second is not None else 0, m_limit=int(batch.get("m_limit", 0)),
        o1_row_start=int(batch.get("o1_row_start", 0)))


def gemm_simt(a: Tensor, b: Tensor, out: Tensor, *, alpha: float = 1.0, beta: float = 0.0) -> Tensor:
    """``out[m, n] = alpha * sum_k a[k, m] * b[k, n] + beta * out`` in fp32 FMA (any strides)."""
    K, M = a.shape
    K2, N = b.shape
    assert K == K2 and out.shape == (M, N)
    _C.gemm_simt(a.data_ptr(), a.stride(0), a.stride(1), b.data_ptr(), b.stride(0), b.stride(1), out.data_ptr(),
                 out.stride(0), out.stride(1), M, N, K, float(alpha), float(beta), _stream())
    _count("gemm_simt_kernel")
    return out


def _ld(t: Tensor) -> int:
    return t.stride(1) if t.shape[1] > 1 else max(1, t.shape[0])


def adam_update(gradient: Tensor, momentum: Tensor, variance: Tensor, beta1: float, beta2: float, eps: float,
                bias_correction1: float, bias_correction2: float) -> Tensor:
    """Fused Adam on 2-D tensors; the result has the strides of ``variance``."""
    for t in (gradient, momentum, variance):
        if t.dtype != torch.float32 or t.ndim != 2:
            raise ValueError("adam_update on CUDA needs 2-D float32 tensors.")
    update = torch.empty_strided(variance.shape, variance.stride(), dtype=torch.float32, device=variance.device)
    rows, cols = variance.shape
    views = [gradient, momentum, variance, update]
    if not all(v.stride(0) == 1 or v.shape[0] == 1 for v in views):
        if all(v.stride(1) == 1 or v.shape[1] == 1 for v in views):
            views = [v.T for v in views]
            rows, cols = cols, rows
        else:
            raise ValueError("adam_update needs all operands column-major or all row-major.")
    g, m, v, u = views
    _C.adam_update(g.data_ptr(), _ld(g), m.data_ptr(), _ld(m), v.data_ptr(), _ld(v), u.data_ptr(), _ld(u), rows, cols,
                   beta1, beta2, eps, 1.0 / bias_correction1, 1.0 / math.sqrt(bias_correction2), _stream())
    _count("adam_kernel")
    return update


def strided_source(matrix: Tensor) -> tuple:
    """A 2-D fp32 or bf16 tensor as the native rotation takes it."""
    return (matrix.data_ptr(), int(matrix.dtype == torch.bfloat16), *matrix.stride())


def rotate_half(scratch, left, right, matrix: Tensor, turned: bool, out: Tensor) -> None:
    """``out <- Q_L^T G Q_R`` (``turned``: ``Q_L G Q_R^T``), ``out`` column-major."""
    assert out.stride(0) == 1 or out.shape[0] == 1
    _C.rotate_half(scratch, left, right, strided_source(matrix) + (int(turned), out.data_ptr(), _ld(out), status_word(out.device).data_ptr(), _stream()))
    mark_written(out)
    for name in ("clear_kernel", "largest_kernel", "half_planes_kernel", "gemm_half_kernel", "gemm_half_kernel"):
        _count(name)


_PARAMETER_TYPES = {torch.float32: 0, torch.bfloat16: 1}
_PLAIN_TENSORS = (Tensor, torch.nn.Parameter)


def _addressable(*tensors: Tensor) -> bool:
    """Whether a flat kernel of the current stream may work on these tensors through their addresses: plain, dense tensors
    (a subclass may have no storage behind its address, or a meaning of its own) of one shape on the current device."""
    index, shape = tensors[0].get_device(), tensors[0].shape
    for t in tensors:
        if (type(t) not in _PLAIN_TENSORS or t.get_device() != index or t.shape != shape or t.layout is not torch.strided
                or not t.is_contiguous() or t.is_neg()):
            return False
    return tensors[0].is_cuda and index == torch.cuda.current_device()


def apply_updates(pairs, keep: float, lr: float) -> list:
    """``p.mul_(keep); p.add_(update.to(p.dtype), alpha=-lr)`` for several ``(p, update)`` in one pass each and as few launches as
    there are parameter types, value for value; returns the pairs that the kernel does not take (nothing is done to them)."""
    jobs: Dict[int, list] = {}
    left = []
    for p, update in pairs:
        kind = _PARAMETER_TYPES.get(p.dtype)
        if kind is None or update.dtype != torch.float32 or not _addressable(p, update):
            left.append((p, update))
        else:
            jobs.setdefault(kind, []).append((p, (p.data_ptr(), update.data_ptr(), p.numel())))
    for kind, some in jobs.items():
        launches = _C.apply_updates([job for _, job in some], kind, keep, lr, _stream())
        mark_written(*(p for p, _ in some))
        LAUNCH_COUNTS["apply_updates_kernel"] = LAUNCH_COUNTS.get("apply_updates_kernel", 0) + launches
    return left


def apply_update(p: Tensor, update: Tensor, keep: float, lr: float) -> bool:
    """The same for one; ``False`` (and nothing done) for tensors that the kernel does not take."""
    return not apply_updates([(p, update)], keep, lr)


def adamw_update(p: Tensor, gradient: Tensor, exp_avg: Tensor, exp_avg_sq: Tensor, beta1: float, beta2: float, bias1: float,
                 bias2: float, eps: float, keep: float, lr: float) -> bool:
    """One AdamW step of a parameter in one pass; ``False`` for tensors that the kernel does not take."""
    kind = _PARAMETER_TYPES.get(p.dtype)
    if (kind is None or gradient.dtype != p.dtype or exp_avg.dtype != torch.float32 or exp_avg_sq.dtype != torch.float32
            or not _addressable(p, gradient, exp_avg, exp_avg_sq)):
        return False
    _C.adamw_update(p.data_ptr(), kind, gradient.data_ptr(), exp_avg.data_ptr(), exp_avg_sq.data_ptr(), p.numel(), 1.0 - beta1,
                    beta2, 1.0 - beta2, bias1, bias2, eps, keep, lr, _stream())
    mark_written(p, exp_avg, exp_avg_sq)
    _count("adamw_kernel")
    return True


def column_dot(a: Tensor, b: Tensor, rows: int, cols: int, out: Optional[Tensor] = None) -> Tensor:
    if out is None:
        out = torch.empty(cols, dtype=torch.float32, device=a.device)
    _C.column_dot(a.data_ptr(), _ld(a), b.data_ptr(), _ld(b), out.data_ptr(), rows, cols, _stream())
    _count("column_dot_kernel")
    return out


def order_by_estimate(table: Tensor) -> Tensor:
    """Stable descending order of the column sums of ``table`` (``parts x n``, any strides with unit row stride or a
    single row): the eigenvalue order of a refresh.  One launch of this library's sort kernel for ``n`` up to
    ``ORDER_MAX_LENGTH``; longer vectors use the framework's sort."""
    parts, n = table.shape
    if n > _C.ORDER_MAX_LENGTH or (parts > 1 and table.stride(0) != 1):
        return torch.argsort(table.sum(dim=0), descending=True, stable=True)
    order = torch.empty(n, dtype=torch.int64, device=table.device)
    ld = table.stride(1) if n > 1 else parts
    _C.order_by_estimate(table.data_ptr(), ld, parts, n, order.data_ptr(), _stream())
    _count("order_by_estimate_kernel")
    return order


def gather2d(src: Tensor, dst: Tensor, row_map: Optional[Tensor], col_map: Optional[Tensor]) -> Tensor:
    """``dst[i, j] = src[row_map[i], col_map[j]]`` (``None`` = identity); ``dst`` must not alias ``src``."""
    rows, cols = dst.shape
    _C.gather2d(src.data_ptr(), src.stride(0), src.stride(1), dst.data_ptr(), dst.stride(0), dst.stride(1),
                row_map.data_ptr() if row_map is not None else 0, col_map.data_ptr() if col_map is not None else 0,
                rows, cols, _stream())
    _count("gather2d_kernel")
    return dst
