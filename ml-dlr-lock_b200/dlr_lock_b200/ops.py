"""Tensor-level entry points: torch supplies device memory and the stream, the
arithmetic happens in ``libdlr_b200.so``.

Calling conventions mirrored from the reference kernels:

* ``forward_folded(x, Vp, Up)``      - this library's own layouts
  (V' (L,r,d), U' (L,d,r)).
* ``forward_xvu(x, Vs, Us)``         - the reference CUDA wrappers' convention,
  e.g. ``cooperative_forward(x, Vs, Us)`` with both stacks (L, R, D)
  (kernels/kernels/cooperative.py:41-68).
* ``dlrnet_fused(x, weights)``       - the reference Triton convention, taking
  the dict of ``pack_dlrnet_weights`` (kernels/kernels/triton_fused.py:68-92).
"""
from __future__ import annotations

import ctypes
from typing import Dict, Tuple

import torch

from . import _lib

EPS = 1e-6

class _Scratch:
    """Per (device, stream): workspace, device status word and its mirror in pinned host memory.

    A kernel writes both words, and only when a device-side wait gives up; the host looks at the mirror without a copy or a
    synchronisation.
    """

    __slots__ = ("ws", "nbytes", "ptr", "status", "status_ptr", "mirror", "word", "retired")

    def __init__(self, device: torch.device, nbytes: int):
        self.status = torch.zeros(1, dtype=torch.int32, device=device)
        self.status_ptr = self.status.data_ptr()
        self.mirror = torch.zeros(1, dtype=torch.int32).pin_memory()
        self.word = ctypes.c_int.from_address(self.mirror.data_ptr())
        _lib.check(_lib.load().dlrb200_set_status_mirror(self.status_ptr, self.mirror.data_ptr()), "dlrb200_set_status_mirror")
        _words.append((self.status, self.mirror))
        # workspaces that were outgrown: a CUDA graph captured earlier has their address in its nodes, so
        # they stay allocated for the life of the process (they are small: at most a few tens of MB)
        self.retired = []
        self.ws = None
        self.resize(device, nbytes)

    def resize(self, device: torch.device, nbytes: int):
        if self.ws is not None:
            self.retired.append(self.ws)
        self.ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
        self.nbytes = nbytes
        self.ptr = self.ws.data_ptr()


_workspaces: Dict[Tuple[int, int], _Scratch] = {}
# status words and their mirrors, kept for the life of the process: the library knows the pair by address, and a CUDA graph
# captured earlier has both in its nodes
_words: list = []
_derived: Dict[Tuple, Tuple[torch.Tensor, ...]] = {}
_MIN_WORKSPACE = 1 << 20
# the current stream of a device as an address, without building a stream object
_raw_stream = torch._C._cuda_getCurrentRawStream if hasattr(torch._C, "_cuda_getCurrentRawStream") else None


def _stream_ptr(index: int) -> int:
    return _raw_stream(index)


def _raise_status(ent: _Scratch, word: int):
    ent.word.value = 0          # a non-zero word makes later calls give up early: clear it before reporting
    ent.status.zero_()
    raise _lib.DlrB200Error(word & 0xff, f"device status: {_lib.strerror(word & 0xff)} at layer {word >> 8}")


def _workspace(index: int, stream: int, nbytes: int) -> _Scratch:
    """Scratch + status word for a (device, stream); grown on demand.

    One workspace per stream, because calls that share one must not overlap.  A workspace that is outgrown
    is kept, not freed: a CUDA graph captured while it was current still clears and uses that memory on
    every replay.  Also the lazy error check: a wait that gave up in a call before, on this stream, is
    reported here without synchronising.
    """
    ent = _workspaces.get((index, stream))
    if ent is None:
        ent = _workspaces[(index, stream)] = _Scratch(torch.device("cuda", index), max(nbytes, _MIN_WORKSPACE))
        return ent
    word = ent.word.value
    if word != 0 and not torch.cuda.is_current_stream_capturing():
        _raise_status(ent, word)
    if ent.nbytes < nbytes:
        ent.resize(torch.device("cuda", index), nbytes)
    return ent


def check_status(device=None) -> None:
    """Synchronise and raise if a bounded device-side wait gave up on `device`.

    Without this call a timeout still surfaces, one call late: the next forward on that stream looks at the
    status word first.
    """
    for (dev, _), ent in list(_workspaces.items()):
        if device is not None and torch.device(device).index not in (None, dev):
            continue
        word = int(ent.status.item())
        if word != 0:
            _raise_status(ent, word)


def _check_inputs(x, Vp, Up):
    if not (x.is_cuda and Vp.is_cuda and Up.is_cuda):
        raise ValueError("dlr_b200 runs on CUDA tensors only (there is no CPU path)")
    if not (x.dtype == Vp.dtype == Up.dtype == torch.bfloat16):
        raise TypeError("dlr_b200 takes bfloat16 activations and folded weights")
    if Vp.dim() != 3 or Up.dim() != 3:
        raise ValueError("folded weights must be V' (L,r,d) and U' (L,d,r)")
    L, r, d = Vp.shape
    if Up.shape != (L, d, r):
        raise ValueError(f"U' has shape {tuple(Up.shape)}, expected {(L, d, r)}")
    if x.shape[-1] != d:
        raise ValueError(f"last dimension of x is {x.shape[-1]}, expected d={d}")
    if not (Vp.is_contiguous() and Up.is_contiguous()):
        raise ValueError("folded weights must be contiguous")
    return L, r, d


def forward_folded(x: torch.Tensor, Vp: torch.Tensor, Up: torch.Tensor, eps: float = EPS,
                   out: torch.Tensor | None = None) -> torch.Tensor:
    """y = DLRNet(x) on folded weights; x is (..., d) bf16 on CUDA, y is a new tensor.

    Asynchronous on the current stream.  A device-side timeout is reported by
    ``check_status`` (which synchronises) or, without a synchronisation, by the
    next forward on the same stream that runs after the failed one has finished.
    """
    L, r, d = _check_inputs(x, Vp, Up)
    index = x.get_device()
    if index != torch.cuda.current_device():
        with torch.cuda.device(index):
            return forward_folded(x, Vp, Up, eps, out)
    if not x.is_contiguous():
        x = x.contiguous()
    y = torch.empty_like(x) if out is None else out.view(-1, d)
    M = x.numel() // d
    if M != 0:
        lib = _lib.load()
        need = lib.dlrb200_workspace_bytes(M, d, r, L)
        if need == 0:
            _lib.check(2, f"dlrb200_forward(M={M}, d={d}, r={r}, L={L})")
        stream = _stream_ptr(index)
        ent = _workspace(index, stream, need)
        rc = lib.dlrb200_forward(x.data_ptr(), y.data_ptr(), Vp.data_ptr(), Up.data_ptr(), M, d, r, L, eps,
                                 ent.ptr, ent.nbytes, ent.status_ptr, stream)
        if rc != 0:
            _lib.check(rc, f"dlrb200_forward(M={M}, d={d}, r={r}, L={L})")
    return y if out is None else y.view(x.shape)


def forward_host(x_host: torch.Tensor, y_host: torch.Tensor, x_dev: torch.Tensor, y_dev: torch.Tensor,
                 Vp: torch.Tensor, Up: torch.Tensor, eps: float = EPS) -> None:
    """Forward with activations in (pinned) host memory; copies ride the current stream."""
    L, r, d = Vp.shape
    M = x_host.numel() // d
    lib = _lib.load()
    with torch.cuda.device(Vp.device):
        index = Vp.get_device()
        need = lib.dlrb200_workspace_bytes(M, d, r, L)
        stream = _stream_ptr(index)
        ent = _workspace(index, stream, need)
        rc = lib.dlrb200_forward_host(x_host.data_ptr(), y_host.data_ptr(), x_dev.data_ptr(), y_dev.data_ptr(), Vp.data_ptr(),
                                      Up.data_ptr(), M, d, r, L, float(eps), ent.ptr, ent.nbytes, ent.status_ptr, stream)
        _lib.check(rc, "dlrb200_forward_host")


def query(M: int, d: int, r: int, L: int) -> _lib.Plan:
    """What ``forward_folded`` launches for a call of this shape on the current CUDA device."""
    plan = _lib.Plan()
    _lib.check(_lib.load().dlrb200_query(M, d, r, L, ctypes.byref(plan)), "dlrb200_query")
    return plan


query_call = query          # (an earlier name)


def fold_weights(V: torch.Tensor, U: torch.Tensor, gain: torch.Tensor, alpha: torch.Tensor):
    """Stacked (L,r,d)/(L,d,r)/(L,d)/(L,) parameters -> folded bf16 (V', U') on the device.

    Same rounding as the reference packer (kernels/reference.py:73-79): V, U and
    the gain are rounded to bf16 first, alpha goes through the parameter dtype to
    fp32, products are formed in fp32 and rounded once.
    """
    if not V.is_cuda:
        raise ValueError("fold_weights runs on CUDA tensors only")
    L, r, d = V.shape
    Vb = V.detach().to(torch.bfloat16).contiguous()
    Ub = U.detach().to(torch.bfloat16).contiguous()
    gb = gain.detach().to(torch.bfloat16).contiguous()
    af = alpha.detach().to(torch.float32).contiguous()
    Vp = torch.empty_like(Vb)
    Up = torch.empty_like(Ub)
    with torch.cuda.device(V.device):
        rc = _lib.load().dlrb200_fold_weights(Vb.data_ptr(), Ub.data_ptr(), gb.data_ptr(), af.data_ptr(), Vp.data_ptr(),
                                              Up.data_ptr(), d, r, L, _stream_ptr(V.get_device()))
    _lib.check(rc, "dlrb200_fold_weights")
    return Vp, Up


_MATRICES_F32, _ALPHA_F32, _ROUND_ALPHA = 1, 2, 4


def fold_layers(found, round_alpha: bool):
    """Folded stacks from unstacked parameters, as ``_host.layers`` or ``_host.state_layers`` found them: the tensors are read
    where they are.  The same values as ``fold_weights``; ``round_alpha`` rounds fp32 scales to bf16 first."""
    L, r, d, index, bf16, alpha_bf16, V, U, gain, alpha = found
    flags = (0 if bf16 else _MATRICES_F32) | (0 if alpha_bf16 else _ALPHA_F32) | (_ROUND_ALPHA if round_alpha else 0)
    device = torch.device("cuda", index)
    Vp = torch.empty((L, r, d), dtype=torch.bfloat16, device=device)
    Up = torch.empty((L, d, r), dtype=torch.bfloat16, device=device)
    with torch.cuda.device(device):
        rc = _lib.load().dlrb200_fold_layers(V, U, gain, alpha, flags, Vp.data_ptr(), Up.data_ptr(), d, r, L, _stream_ptr(index))
    _lib.check(rc, "dlrb200_fold_layers")
    return Vp, Up


def transpose_stack(src: torch.Tensor) -> torch.Tensor:
    """(L, rows, cols) bf16 -> (L, cols, rows), on the device."""
    L, rows, cols = src.shape
    src = src.contiguous()
    dst = torch.empty((L, cols, rows), dtype=src.dtype, device=src.device)
    with torch.cuda.device(src.device):
        rc = _lib.load().dlrb200_transpose_stack(src.data_ptr(), dst.data_ptr(), L, rows, cols, _stream_ptr(src.get_device()))
    _lib.check(rc, "dlrb200_transpose_stack")
    return dst


def _cached_transpose(t: torch.Tensor) -> torch.Tensor:
    key = ("T", t.data_ptr(), t._version, tuple(t.shape), t.device.index)
    hit = _derived.get(key)
    if hit is None:
        if len(_derived) > 64:
            _derived.clear()
        hit = (transpose_stack(t),)
        _derived[key] = hit
    return hit[0]


def forward_xvu(x: torch.Tensor, Vs: torch.Tensor, Us: torch.Tensor) -> torch.Tensor:
    """Reference CUDA-wrapper convention: Vs (L,R,D) and Us (L,R,D), both folded.

    Us is U'^T there; its transpose is derived on the device once per weight
    tensor and cached.  Any B >= 1 is accepted (no padding needed).
    """
    if Vs.dim() != 3 or Us.shape != Vs.shape:
        raise ValueError("expected Vs (L,R,D) and Us (L,R,D)")
    return forward_folded(x, Vs.contiguous(), _cached_transpose(Us))


def dlrnet_fused(x: torch.Tensor, weights: dict, **_ignored) -> torch.Tensor:
    """Reference Triton convention: `weights` is the dict of pack_dlrnet_weights
    with Vs (L,D,R) = V'^T and Us (L,R,D) = U'^T, premultiplied."""
    if not weights.get("premultiplied", False):
        raise ValueError("dlrnet_fused needs premultiplied weights (pack with premultiply=True)")
    return forward_folded(x, _cached_transpose(weights["Vs"]), _cached_transpose(weights["Us"]))
