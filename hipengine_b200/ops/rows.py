"""Launchers of the few-row products with quantised weights (``csrc/gemm_rows.cu``, on tcgen05 ``csrc/gemm_rows_tc.cu``): 1..64
activation rows, written once per product as an image of MMA operands, times any number of weight rows streamed once."""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import Optional, Sequence, Tuple

import torch

from ..core import native as N
from .kernels import EPI_GELU_MUL, EPI_SILU_MUL, DeviceWeight, GemvSegment, _check_device, _dt, _p, _stream, status_tensor

MAX_ROWS = 64
# Rows up to which products run on mma.sync, above them on tcgen05 (csrc/gemm_rows_tc.cu): 17408 x 5120 weights at 16 rows 22.2 us
# (Q4_K), 24.7 (Q8_0), Q6_K 5120 x 17408 24.8; at 24 rows tcgen05 takes 20.7 / 36.5 / 27.0 us, mma.sync 24.4 / 29.5 / 27.4.
MMA_ROWS = 16
MMA_ROWS_Q8 = 24             # ... of models with Q8_0 projections
MAX_SEGMENTS = 4
QTYPES = (8, 12, 14)         # Q8_0, Q4_K, Q6_K
HALF_TILE = 64               # smallest tile: weight rows of each weight of a gate/up pair
IMAGE_UNIT = 576             # image bytes of 256 columns of a row
SIDE_MAX_COLS = 25600        # widest rows that products with fp32 side weights take: two of those in shared memory


class _Seg(C.Structure):
    _fields_ = [("w", C.c_void_p), ("w2", C.c_void_p), ("out", C.c_void_p), ("out_stride", C.c_longlong),
                ("n_rows", C.c_int), ("qtype", C.c_int), ("epi", C.c_int), ("tile0", C.c_int)]


class _Args(C.Structure):
    _fields_ = [("seg", _Seg * MAX_SEGMENTS), ("n_seg", C.c_int), ("K", C.c_int), ("R", C.c_int), ("tc", C.c_int),
                ("image", C.c_void_p), ("ws", C.c_void_p), ("ws_floats", C.c_longlong), ("counters", C.c_void_p),
                ("n_counters", C.c_int), ("status", C.c_void_p), ("stages", C.c_int), ("stage_bytes", C.c_int),
                ("w_bytes", C.c_int), ("tiles", C.c_int)]


class _ExpertsArgs(C.Structure):
    _fields_ = [("image", C.c_void_p), ("jobs", C.c_void_p), ("entries", C.c_void_p), ("meta", C.c_void_p),
                ("out", C.c_void_p), ("out_stride", C.c_longlong), ("status", C.c_void_p), ("pairs_per_row", C.c_int),
                ("N", C.c_int), ("K", C.c_int), ("E", C.c_int), ("expert_rows", C.c_int), ("qtype", C.c_int),
                ("epi", C.c_int), ("stages", C.c_int), ("stage_bytes", C.c_int), ("w_bytes", C.c_int)]


@dataclass
class ExpertJobs:
    entries: torch.Tensor      # [P] pair ids sorted by expert
    list: torch.Tensor         # [bound, 4] (expert, first entry, entries, 0)
    meta: torch.Tensor         # [0]: jobs
    E: int
    cols: int
    P: int


_CHECKED = False


def _lib():
    global _CHECKED
    L = N.lib()
    if not _CHECKED:
        if L.he_rows_args_size() != C.sizeof(_Args):
            raise RuntimeError(f"ABI mismatch for HeRowsArgs: C={L.he_rows_args_size()} Python={C.sizeof(_Args)}")
        if L.he_rows_experts_args_size() != C.sizeof(_ExpertsArgs):
            raise RuntimeError("ABI mismatch for RowsExpertsArgs")
        L.he_rows_image_bytes.restype = L.he_rows_ws_floats.restype = L.he_tc_gather_bytes.restype = C.c_longlong
        _CHECKED = True
    return L


def weight_ok(w: DeviceWeight) -> bool:
    return w.qtype in QTYPES and w.n_cols % 256 == 0


class RowsSpace:
    """What the products of one stream share: the activation image and the partial tiles (named scratch of the owner)
    and the arrival counters of the tiles (zero between launches)."""

    def __init__(self, scratch, device: torch.device, max_weight_rows: int, mma_rows: int = MMA_ROWS):
        self.scratch = scratch
        self.mma_rows = mma_rows
        self._image_bytes, self._ws_floats = {}, {}      # by (rows, columns, form), by (rows, form)
        # tiles of a launch: at most MAX_SEGMENTS segments of the largest weight, in half tiles when they are pairs
        n = MAX_SEGMENTS * (-(-max_weight_rows // HALF_TILE))
        self.counters = torch.zeros(n, dtype=torch.int32, device=device)

    def image(self, x: torch.Tensor, norm_w: Optional[torch.Tensor] = None, eps: float = 1e-6,
              side_w: Optional[torch.Tensor] = None, side_out: Optional[torch.Tensor] = None,
              by_row: bool = False, product: bool = True, steady: bool = False) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
        """The fragments of (RMSNorm of) the rows ``x`` [R, K] (fp32 or bf16): (for ``product``, for ``experts``), each on
        demand.  With ``side_w`` (fp32 [n, K]) the same launch also writes ``side_out`` [R, >= n] = normalised rows @
        side_w^T, all in fp32, or nothing else; ``steady``: a row's are the same bits beside any number of others."""
        _check_device(x)
        R, K = x.shape
        assert x.stride(1) == 1
        L = _lib()
        img = rows = None
        tc = int(R > self.mma_rows)
        if product:
            size = self._image_bytes.get((R, K, tc))
            if size is None:
                size = self._image_bytes[R, K, tc] = int(L.he_rows_image_bytes(C.c_int(R), C.c_int(K), C.c_int(tc)))
            img = self.scratch.get("rows_image", (size,), torch.uint8)
        if by_row:
            rows = self.scratch.get("rows_by_row", (R * (K // 256) * IMAGE_UNIT,), torch.uint8)
        n_side = 0
        if side_w is not None:
            n_side = side_w.shape[0]
            assert side_w.dtype == side_out.dtype == torch.float32 and side_w.is_contiguous() and side_w.shape[1] == K
            assert side_out.shape[0] >= R and side_out.shape[1] >= n_side and side_out.stride(1) == 1
        N.check(L.he_rows_image(C.c_void_p(x.data_ptr()), C.c_int(_dt(x)), C.c_longlong(x.stride(0)),
                                C.c_void_p(_p(norm_w)), C.c_float(eps), C.c_int(K), C.c_int(R), C.c_void_p(_p(img)), C.c_int(tc),
                                C.c_void_p(_p(rows)), C.c_void_p(_p(side_w)), C.c_int(n_side),
                                C.c_void_p(_p(side_out) if n_side else None),
                                C.c_longlong(side_out.stride(0) if n_side else 0), C.c_int(int(steady)), _stream()), "he_rows_image")
        return img, rows

    def jobs(self, ids: torch.Tensor, E: int, cols: int) -> "ExpertJobs":
        """The (row, choice) pairs of ``ids`` [T, k] (int32) sorted by expert, cut into jobs of at most ``cols`` pairs."""
        L = _lib()
        L.he_moe_jobs_bound.restype = C.c_longlong
        P = ids.numel()
        n = int(L.he_moe_jobs_bound(C.c_longlong(P), C.c_int(E), C.c_int(cols)))
        j = ExpertJobs(self.scratch.get("moe_entries", (P,), torch.int32),
                       self.scratch.get("moe_job_list", (n, 4), torch.int32),
                       self.scratch.get("moe_job_meta", (4,), torch.int32), E, cols, P)
        assert ids.dtype == torch.int32 and ids.is_contiguous()
        N.check(L.he_moe_jobs(C.c_void_p(ids.data_ptr()), C.c_int(P), C.c_int(E), C.c_int(cols),
                              C.c_void_p(j.entries.data_ptr()), C.c_void_p(j.list.data_ptr()), C.c_int(n),
                              C.c_void_p(j.meta.data_ptr()), _stream()), "he_moe_jobs")
        return j

    def experts(self, jobs: "ExpertJobs", by_row: torch.Tensor, pairs_per_row: int, w: DeviceWeight, out: torch.Tensor,
                epi: int, w2: Optional[DeviceWeight] = None) -> None:
        """out[pair] = (row of the pair) @ W[its expert]^T for the stacked expert weights ``w`` (gate, with ``w2`` up, for
        the activation epilogues); ``by_row`` holds the image of pair // pairs_per_row."""
        L = _lib()
        assert w.n_rows % jobs.E == 0 and weight_ok(w) and out.shape[0] >= jobs.P and out.stride(1) == 1
        a = _ExpertsArgs()
        a.image, a.jobs, a.entries, a.meta = by_row.data_ptr(), jobs.list.data_ptr(), jobs.entries.data_ptr(), jobs.meta.data_ptr()
        a.out, a.out_stride, a.status = out.data_ptr(), out.stride(0), status_tensor(out.device).data_ptr()
        a.pairs_per_row, a.N, a.K, a.E = pairs_per_row, w.n_rows // jobs.E, w.n_cols, jobs.E
        a.expert_rows, a.qtype, a.epi = w.n_rows // jobs.E, w.qtype, epi
        if w2 is not None:
            assert w2.qtype == w.qtype and w2.n_rows == w.n_rows and w2.n_cols == w.n_cols
        N.check(L.he_rows_experts(C.byref(a), C.c_void_p(w.ptr), C.c_void_p(None if w2 is None else w2.ptr),
                                  C.c_int(jobs.cols), C.c_int(N.num_sms()), _stream()), "he_rows_experts")

    def gather(self, jobs: "ExpertJobs", x: torch.Tensor, pairs_per_row: int) -> torch.Tensor:
        """Images of the jobs' rows (of 64) for ``experts_tc``: row pair // pairs_per_row of ``x`` (fp32 or bf16)."""
        L = _lib()
        n, K = jobs.list.shape[0], x.shape[1]
        # (in the buffer that the grouped GEMM gathers its rows into, of the same size: an expert block takes one route or the other)
        size = int(L.he_tc_gather_bytes(C.c_longlong(n), C.c_int(K)))
        img = self.scratch.get("moe_xs", (size // 2,), torch.bfloat16).view(torch.uint8)
        assert jobs.cols == 64 and x.stride(1) == 1 and x.shape[0] * pairs_per_row >= jobs.P
        N.check(L.he_tc_gather(C.c_void_p(x.data_ptr()), C.c_int(_dt(x)), C.c_longlong(x.stride(0)), C.c_int(K),
                               C.c_void_p(jobs.list.data_ptr()), C.c_void_p(jobs.entries.data_ptr()),
                               C.c_void_p(jobs.meta.data_ptr()), C.c_int(pairs_per_row), C.c_int(n),
                               C.c_void_p(img.data_ptr()), _stream()), "he_tc_gather")
        return img

    def experts_tc(self, jobs: "ExpertJobs", image: torch.Tensor, w: DeviceWeight, out: torch.Tensor, epi: int,
                   w2: Optional[DeviceWeight] = None) -> None:
        """``experts`` for jobs of 64 rows on tcgen05, from the images of ``gather``."""
        assert jobs.cols == 64 and w.n_rows % jobs.E == 0 and weight_ok(w) and out.shape[0] >= jobs.P and out.stride(1) == 1
        a = _Args()
        g = a.seg[0]
        g.w, g.out, g.out_stride, g.n_rows, g.qtype, g.epi = w.ptr, out.data_ptr(), out.stride(0), w.n_rows // jobs.E, w.qtype, epi
        if w2 is not None:
            assert w2.qtype == w.qtype and w2.n_rows == w.n_rows and w2.n_cols == w.n_cols
            g.w2 = w2.ptr
        a.K, a.R, a.tc, a.image, a.status = w.n_cols, jobs.cols, 1, image.data_ptr(), status_tensor(out.device).data_ptr()
        N.check(_lib().he_tc_experts(C.byref(a), C.c_int(jobs.E), C.c_void_p(jobs.list.data_ptr()),
                                     C.c_void_p(jobs.entries.data_ptr()), C.c_void_p(jobs.meta.data_ptr()),
                                     C.c_int(N.num_sms()), _stream()), "he_tc_experts")

    @staticmethod
    def sum_pairs(h: torch.Tensor, y: torch.Tensor, wts: torch.Tensor, shared: Optional[torch.Tensor] = None,
                  shared_gate: Optional[torch.Tensor] = None) -> None:
        """h[t] += sum_j wts[t, j] * y[t * k + j] (+ sigmoid(shared_gate[t]) * shared[t])."""
        T, k = wts.shape
        assert h.dtype == torch.float32 and wts.is_contiguous() and wts.dtype == torch.float32
        assert shared is None or shared.dtype == torch.bfloat16
        N.check(_lib().he_moe_sum_pairs(
            C.c_void_p(h.data_ptr()), C.c_longlong(h.stride(0)), C.c_void_p(y.data_ptr()), C.c_int(_dt(y)),
            C.c_longlong(y.stride(0)), C.c_void_p(wts.data_ptr()), C.c_int(T), C.c_int(k), C.c_void_p(_p(shared)),
            C.c_longlong(0 if shared is None else shared.stride(0)), C.c_void_p(_p(shared_gate)),
            C.c_longlong(0 if shared_gate is None else shared_gate.stride(0)), C.c_int(h.shape[1]), _stream()),
            "he_moe_sum_pairs")

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
        a.n_seg, a.K, a.R, a.tc = len(segs), K, R, int(R > self.mma_rows)
        n_ws = self._ws_floats.get((R, a.tc))
        if n_ws is None:
            n_ws = self._ws_floats[R, a.tc] = int(L.he_rows_ws_floats(C.c_int(R), C.c_int(N.num_sms()), C.c_int(a.tc)))
        a.image = image.data_ptr()
        a.ws, a.ws_floats = self.scratch.get("rows_ws", (n_ws,), torch.float32).data_ptr(), n_ws
        a.counters, a.n_counters = self.counters.data_ptr(), self.counters.numel()
        a.status = status_tensor(self.counters.device).data_ptr()
        N.check(L.he_rows_gemm(C.byref(a), C.c_int(N.num_sms()), _stream()), "he_rows_gemm")

    def gemm(self, x: torch.Tensor, segs: Sequence[GemvSegment], norm_w: Optional[torch.Tensor] = None,
             eps: float = 1e-6) -> None:
        self.product(self.image(x, norm_w, eps)[0], x.shape[0], x.shape[1], segs)
