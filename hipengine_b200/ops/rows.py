"""Launchers of the few-row products with quantised weights (``csrc/gemm_rows.cu``): 1..64 activation rows, written once
per product as an image of MMA fragments, times any number of weight rows streamed once."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence, Tuple

import torch

from ..core import native as N
from .kernels import EPI_GELU_MUL, EPI_SILU_MUL, DeviceWeight, GemvSegment, _check_device, _dt, _p, _stream, status_tensor

MAX_ROWS = 64
MAX_SEGMENTS = 4
QTYPES = (8, 12, 14)         # Q8_0, Q4_K, Q6_K
HALF_TILE = 64               # smallest tile: weight rows of each weight of a gate/up pair
IMAGE_UNIT = 576             # image bytes of 256 columns of a row


class _Seg(C.Structure):
    _fields_ = [("w", C.c_void_p), ("w2", C.c_void_p), ("out", C.c_void_p), ("out_stride", C.c_longlong),
                ("n_rows", C.c_int), ("qtype", C.c_int), ("epi", C.c_int), ("tile0", C.c_int)]


class _Args(C.Structure):
    _fields_ = [("seg", _Seg * MAX_SEGMENTS), ("n_seg", C.c_int), ("K", C.c_int), ("R", C.c_int),
                ("image", C.c_void_p), ("ws", C.c_void_p), ("ws_floats", C.c_longlong), ("counters", C.c_void_p),
                ("n_counters", C.c_int), ("status", C.c_void_p), ("stages", C.c_int), ("stage_bytes", C.c_int),
                ("w_bytes", C.c_int), ("tiles", C.c_int)]


_CHECKED = False


def _lib():
    global _CHECKED
    L = N.lib()
    if not _CHECKED:
        if L.he_rows_args_size() != C.sizeof(_Args):
            raise RuntimeError(f"ABI mismatch for HeRowsArgs: C={L.he_rows_args_size()} Python={C.sizeof(_Args)}")
        L.he_rows_image_bytes.restype = L.he_rows_ws_floats.restype = C.c_longlong
        _CHECKED = True
    return L


def weight_ok(w: DeviceWeight) -> bool:
    return w.qtype in QTYPES and w.n_cols % 256 == 0


class RowsSpace:
    """What the products of one stream share: the activation image and the partial tiles (named scratch of the owner)
    and the arrival counters of the tiles (zero between launches)."""

    def __init__(self, scratch, device: torch.device, max_weight_rows: int):
        self.scratch = scratch
        # tiles of a launch: at most MAX_SEGMENTS segments of the largest weight, in half tiles when they are pairs
        n = MAX_SEGMENTS * (-(-max_weight_rows // HALF_TILE))
        self.counters = torch.zeros(n, dtype=torch.int32, device=device)

    def image(self, x: torch.Tensor, norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6,
              side_w: Optional[torch.Tensor] = None, side_out: Optional[torch.Tensor] = None,
              by_row: bool = False, product: bool = True) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
        """The fragments of (RMSNorm of) the rows ``x`` [R, K] (fp32 or bf16): (for ``product``, for ``experts``), each on
        demand.  With ``side_w`` (fp32 [n, K]) the same launch also writes ``side_out`` [R, >= n] = normalised rows @
        side_w^T, all in fp32."""
        _check_device(x)
        R, K = x.shape
        assert x.stride(1) == 1
        L = _lib()
        img = rows = None
        if product:
            img = self.scratch.get("rows_image", (int(L.he_rows_image_bytes(C.c_int(R), C.c_int(K))),), torch.uint8)
        if by_row:
            rows = self.scratch.get("rows_by_row", (R * (K // 256) * IMAGE_UNIT,), torch.uint8)
        n_side = 0
        if side_w is not None:
            n_side = side_w.shape[0]
            assert side_w.dtype == side_out.dtype == torch.float32 and side_w.is_contiguous() and side_w.shape[1] == K
            assert side_out.shape[0] >= R and side_out.shape[1] >= n_side and side_out.stride(1) == 1
        N.check(L.he_rows_image(C.c_void_p(x.data_ptr()), C.c_int(_dt(x)), C.c_longlong(x.stride(0)),
                                C.c_void_p(_p(norm_w)), C.c_float(eps), C.c_int(K), C.c_int(R), C.c_void_p(_p(img)),
                                C.c_void_p(_p(rows)), C.c_void_p(_p(side_w)), C.c_int(n_side),
                                C.c_void_p(_p(side_out) if n_side else None),
                                C.c_longlong(side_out.stride(0) if n_side else 0), _stream()), "he_rows_image")
        return img, rows

    def product(self, image: torch.Tensor, R: int, K: int, segs: Sequence[GemvSegment]) -> None:
        """out (+)= rows @ W^T for every segment (see ``GemvSegment``), from the rows' image."""
        L = _lib()
        a = _Args()
        assert len(segs) <= MAX_SEGMENTS
        for s, g in zip(segs, a.seg):
            assert weight_ok(s.w) and s.w.n_cols == K, (s.w.qtype, s.w.n_cols, K)
            if s.epi in (EPI_SILU_MUL, EPI_GELU_MUL):
                assert s.w2.qtype == s.w.qtype and s.w2.n_rows == s.w.n_rows and s.w2.n_cols == K
                g.w2 = s.w2.ptr
            g.w, g.out, g.n_rows, g.qtype, g.epi = s.w.ptr, s.out.data_ptr(), s.w.n_rows, s.w.qtype, s.epi
            g.out_stride = s.out.stride(0) if s.out.dim() > 1 else s.out.numel()
        n_ws = int(L.he_rows_ws_floats(C.c_int(R), C.c_int(N.num_sms())))
        a.n_seg, a.K, a.R = len(segs), K, R
        a.image = image.data_ptr()
        a.ws, a.ws_floats = self.scratch.get("rows_ws", (n_ws,), torch.float32).data_ptr(), n_ws
        a.counters, a.n_counters = self.counters.data_ptr(), self.counters.numel()
        a.status = status_tensor(self.counters.device).data_ptr()
        N.check(L.he_rows_gemm(C.byref(a), C.c_int(N.num_sms()), _stream()), "he_rows_gemm")

    def gemm(self, x: torch.Tensor, segs: Sequence[GemvSegment], norm_w: Optional[torch.Tensor] = None,
             eps: float = 1e-6) -> None:
        self.product(self.image(x, norm_w, eps)[0], x.shape[0], x.shape[1], segs)
