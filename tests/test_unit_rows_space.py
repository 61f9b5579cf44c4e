"""What the few-row products ask the library for (ops/rows.py), with the launches left out."""
import pytest
import torch

from hipengine_b200.core import native


class _Quiet:
    """The library without its launches."""

    def __init__(self, lib):
        self.lib, self.he_rows_image, self.he_rows_gemm = lib, lambda *a: 0, lambda *a: 0

    def __getattr__(self, name):
        return getattr(self.lib, name)


@pytest.mark.skipif(not native.lib_available(), reason="native library not built")
def test_sizes_follow_the_form_of_the_product(monkeypatch):
    """Rows that change from one form to the other get the other's image and workspace."""
    import ctypes as C
    from types import SimpleNamespace
    from hipengine_b200.ops import rows as ROWS
    lib = ROWS._lib()
    monkeypatch.setattr(ROWS, "_lib", lambda: _Quiet(lib))
    monkeypatch.setattr(ROWS, "_check_device", lambda x: None)
    monkeypatch.setattr(ROWS, "_stream", lambda: C.c_void_p(0))
    monkeypatch.setattr(ROWS, "status_tensor", lambda d: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ROWS.N, "num_sms", lambda: 148)
    asked = {}

    def get(name, shape, dtype):
        asked[name] = shape[0]
        return torch.empty(shape, dtype=dtype)

    w = SimpleNamespace(qtype=12, n_cols=512, n_rows=128, ptr=256)
    space = ROWS.RowsSpace(SimpleNamespace(get=get), torch.device("cpu"), 256)
    for R in (17, 20, 24):
        for mma_rows in (24, 16, 24):
            space.mma_rows = mma_rows
            img, _ = space.image(torch.zeros(R, 512))
            space.product(img, R, 512, [SimpleNamespace(w=w, w2=None, out=torch.zeros(R, 128), epi=0)])
            tc = C.c_int(int(R > mma_rows))
            assert asked["rows_image"] == lib.he_rows_image_bytes(C.c_int(R), C.c_int(512), tc), (R, mma_rows)
            assert asked["rows_ws"] == lib.he_rows_ws_floats(C.c_int(R), C.c_int(148), tc), (R, mma_rows)


@pytest.mark.skipif(not native.lib_available(), reason="native library not built")
@pytest.mark.parametrize("pairs,E,K", [(16384, 256, 2048), (28672, 256, 2048), (1792, 16, 512)])
def test_job_images_take_the_buffer_of_the_grouped_gemm(monkeypatch, pairs, E, K):
    """A process that runs expert prompts of both routes holds one buffer of gathered rows, no larger than the grouped GEMM's."""
    import ctypes as C
    from types import SimpleNamespace
    from hipengine_b200.ops import kernels as KN
    from hipengine_b200.ops import rows as ROWS
    lib = ROWS._lib()
    quiet = _Quiet(lib)
    quiet.he_tc_gather = lambda *a: 0
    monkeypatch.setattr(ROWS, "_lib", lambda: quiet)
    monkeypatch.setattr(ROWS, "_stream", lambda: C.c_void_p(0))
    asked = {}

    def get(name, shape, dtype):
        asked[name] = (shape[0], dtype)
        return torch.empty(shape, dtype=dtype)

    space = ROWS.RowsSpace(SimpleNamespace(get=get), torch.device("cpu"), 256)
    lib.he_moe_jobs_bound.restype = C.c_longlong
    n = int(lib.he_moe_jobs_bound(C.c_longlong(pairs), C.c_int(E), C.c_int(64)))
    jobs = ROWS.ExpertJobs(torch.zeros(1), torch.zeros(n, 4), torch.zeros(4), E, 64, pairs)
    img = space.gather(jobs, torch.zeros(pairs // 4, K, dtype=torch.bfloat16), 4)
    assert img.dtype == torch.uint8 and img.numel() == lib.he_tc_gather_bytes(C.c_longlong(n), C.c_int(K))
    assert set(asked) == {"moe_xs"} and asked["moe_xs"][1] == torch.bfloat16
    assert asked["moe_xs"][0] <= KN.moe_sorted_rows_bound(pairs, E) * K
