"""Few-row products with quantised weights (csrc/gemm_rows.cu) against 64-bit products of the dequantised blocks."""
import pytest
import torch

from hipengine_b200.quant import ggml as Q

pytestmark = pytest.mark.gpu
T = Q.GGMLType


def _weight(t, n, k, seed):
    from hipengine_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(seed)
    raw = Q.quantize(torch.randn(n, k, generator=g, device="cuda") * 0.02, t)
    return K.to_device_weight(raw, t, n, k), Q.dequantize_torch(raw, t, n, k).double()


@pytest.fixture(scope="module")
def space():
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    return RowsSpace(_Scratch(dev, canaries=True), dev, 5000)


# fp32 rows round to 11 bits: at most 2^-11 of each value, so at most that of the result where the signs are random (2.1e-4 on
# average for normal rows).  The weights are exact, but for Q6_K above eight rows: rounded to 11 bits as well, sqrt(2) of it
BOUND = {T.Q4_K: 2 ** -11, T.Q6_K: 2 ** -10.5, T.Q8_0: 2 ** -11}


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
@pytest.mark.parametrize("n,k", [(1, 256), (130, 512), (300, 768), (4999, 1280), (64, 17408)])
def test_products_match_64_bit(space, t, n, k):
    """Edges: fewer weight rows than a tile, remainders of it, one block, an odd number of blocks, tiles shared by many CTAs;
    every group of eight activation rows."""
    from hipengine_b200.ops import kernels as K
    w, wd = _weight(t, n, k, n + k)
    for R in (1, 2, 8, 9, 17, 32, 33, 41, 49, 64):
        torch.manual_seed(R)
        x = torch.randn(R, k, device="cuda") * torch.logspace(-3, 3, R, device="cuda")[:, None]
        for xx in (x, x.bfloat16()):
            out = torch.full((R, n), float("nan"), device="cuda")
            space.gemm(xx, [K.GemvSegment(w, out)])
            ref = xx.double() @ wd.t()
            err = ((out.double() - ref).norm(dim=1) / ref.norm(dim=1)).max() if n > 1 else \
                (out.double() - ref).abs().max() / (xx.double().norm(dim=1) * wd.norm()).max()
            assert err < BOUND[t], (R, xx.dtype, float(err))
        again = torch.zeros_like(out)
        space.gemm(xx, [K.GemvSegment(w, again)])
        assert torch.equal(out, again)
    K.check_status()
    assert int(space.counters.abs().sum()) == 0 and space.scratch.check_canaries() == []


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
@pytest.mark.parametrize("R", [1, 8, 9, 24, 40, 64])
def test_weights_enter_exactly(space, t, R):
    """Rows that their image holds exactly: what is left is the rounding of fp32 sums.  Scales from the type's largest to its
    smallest within a block."""
    from hipengine_b200.ops import kernels as K
    n, k = 200, 1280
    g = torch.Generator(device="cuda").manual_seed(R)
    wf = torch.randn(n, k // 16, 16, generator=g, device="cuda") * 10 ** (-4 * torch.rand(n, k // 16, 1, generator=g, device="cuda"))
    raw = Q.quantize(wf.reshape(n, k), t)
    w, wd = K.to_device_weight(raw, t, n, k), Q.dequantize_torch(raw, t, n, k).double()
    x = torch.randint(-31, 32, (R, k), generator=g, device="cuda").float()
    out = torch.zeros(R, n, device="cuda")
    space.gemm(x, [K.GemvSegment(w, out)])
    ref = x.double() @ wd.t()
    # 1280 terms in fp32: sqrt(1280) 2^-24 of the terms' norm; above eight rows Q6_K operands round to 11 bits
    assert float((out.double() - ref).norm() / ref.norm()) < (2 ** -11 if t == T.Q6_K and R > 8 else 36 * 2 ** -24)
    K.check_status()


def test_a_row_does_not_depend_on_its_neighbours(space):
    from hipengine_b200.ops import kernels as K
    w, _ = _weight(T.Q4_K, 640, 2048, 3)
    x = torch.randn(8, 2048, device="cuda")
    out = torch.zeros(8, 640, device="cuda")
    space.gemm(x, [K.GemvSegment(w, out)])
    for r in range(8):
        one = torch.zeros(1, 640, device="cuda")
        space.gemm(x[r:r + 1], [K.GemvSegment(w, one)])
        assert torch.equal(one[0], out[r])


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_a_row_beside_others(space, t):
    """A row's bits are the same for every number of rows that takes the same kernel; between kernels the sums take another
    order and Q6_K operands another rounding (11 bits above eight rows)."""
    from hipengine_b200.ops import kernels as K
    w, _ = _weight(t, 640, 2048, 3)
    x = torch.randn(64, 2048, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
    first = {}
    for R in (1, 3, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 48, 49, 64):
        out = torch.zeros(R, 640, device="cuda")
        space.gemm(x[:R], [K.GemvSegment(w, out)])
        kernel = min((R + 7) // 8, 7)
        seen = first.setdefault(kernel, out)
        n = min(R, seen.shape[0])
        assert torch.equal(out[:n], seen[:n]), R
        if R > seen.shape[0]:
            first[kernel] = out
        rel = float((out[0] - first[1][0]).norm() / first[1][0].norm())
        assert rel < (2 ** -11 if t == T.Q6_K and R > 8 else 2e-6), R


@pytest.mark.parametrize("R", [4, 16, 24, 40, 64])
@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_outliers_cost_the_other_columns_of_their_block_an_absolute_error(space, t, R):
    """One value a block a million times the others: those are fp16 subnormals under the block's power of two, off by at most
    2^-25 of it each (bf16 rows too, whose small values the image no longer holds exactly)."""
    from hipengine_b200.ops import kernels as K
    n, k = 96, 1024
    w, wd = _weight(t, n, k, 11)
    x = torch.randn(R, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)) * 1e-6
    x[:, 37::256] = torch.tensor([1.0, 1.5, -1.25, 1.75], device="cuda").repeat(R // 4)[:, None]
    for xx in (x, x.bfloat16()):
        out = torch.zeros(R, n, device="cuda")
        space.gemm(xx, [K.GemvSegment(w, out)])
        err = (out.double() - xx.double() @ wd.t()).abs()
        # the rounding of the small values, and of fp32 sums of at most 1.75 times the outliers' weights
        bound = 2 ** -25 * wd.abs().sum(1) + 2 ** -20 * 1.75 * wd[:, 37::256].abs().sum(1)
        if t == T.Q6_K and R > 8:               # weights as fp16 numbers: half of the last of 11 bits, at most 2^-11 of each
            bound = bound + 2 ** -11 * (xx.double().abs() @ wd.abs().t()).amax(0)
        assert bool((err <= bound[None]).all()), float((err / bound[None]).max())


def test_segments_pairs_norm_side_rows(space):
    """Segments of all block types in one launch; gate/up pair; adding into a strided residual; fp32 side rows."""
    from hipengine_b200.ops import kernels as K
    k = 1024
    (g, gd), (u, ud) = _weight(T.Q4_K, 200, k, 1), _weight(T.Q4_K, 200, k, 2)
    (a, ad), (b, bd) = _weight(T.Q6_K, 129, k, 3), _weight(T.Q8_0, 96, k, 4)
    side = torch.randn(97, k, device="cuda") * 0.02
    for R in (2, 7, 24, 40, 64):
        x, nw = torch.randn(R, k, device="cuda"), torch.rand(k, device="cuda") + 0.5
        act = torch.zeros(R, 208, device="cuda", dtype=torch.bfloat16)
        add = torch.ones(R, 160, device="cuda")
        pre = torch.zeros(R, 96, device="cuda")
        so = torch.full((R, 104), float("nan"), device="cuda")
        img, _ = space.image(x, nw, 1e-6, side, so)
        space.product(img, R, k, [K.GemvSegment(g, act, K.EPI_SILU_MUL, u), K.GemvSegment(a, add[:, :129], K.EPI_ADD_F32),
                                  K.GemvSegment(b, pre)])
        xn = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * nw.double()
        rel = lambda y, r: float((y.double() - r).norm() / r.norm())
        assert rel(act[:, :200], torch.nn.functional.silu(xn @ gd.t()) * (xn @ ud.t())) < 4e-3       # bf16 result
        assert rel(add[:, :129] - 1, xn @ ad.t()) < 2 ** -10.5 and bool((add[:, 129:] == 1).all())
        assert rel(pre, xn @ bd.t()) < 2 ** -10.5
        assert rel(so[:, :97], xn @ side.double().t()) < 3e-6 and bool(so[:, 97:].isnan().all())
        alone = torch.full((R, 104), float("nan"), device="cuda")
        assert space.image(x, nw, 1e-6, side, alone, product=False) == (None, None)
        assert torch.equal(alone[:, :97], so[:, :97])
    K.check_status()


@pytest.mark.parametrize("R", [7, 16, 24, 40, 64])
@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_extreme_rows(space, t, R):
    """Zero rows, large and small numbers up to the largest of all, and a NaN that stays in its own row."""
    from hipengine_b200.ops import kernels as K
    w, wd = _weight(t, 128, 512, 9)
    x = torch.randn(R, 512, device="cuda")
    x[0] = 0
    x[1] *= 1e30
    x[2] *= 1e-30
    x[3, 5] = float("nan")
    x[4, 7] = float("inf")
    x[6] *= 1e38 / x[6].abs().max()
    x[6, 300] = torch.finfo(torch.float32).max
    out = torch.zeros(R, 128, device="cuda")
    space.gemm(x, [K.GemvSegment(w, out)])
    ref = x.double() @ wd.t()
    assert bool((out[0] == 0).all()) and bool(out[3].isnan().all()) and not bool(out[4].isfinite().any())
    for r in (1, 2, *range(5, R)):
        assert float((out[r].double() - ref[r]).norm() / ref[r].norm()) < BOUND[t], r


def test_refusals(space):
    from hipengine_b200.ops import kernels as K
    w, _ = _weight(T.Q4_K, 128, 512, 9)
    with pytest.raises(RuntimeError):
        space.gemm(torch.zeros(65, 512, device="cuda"), [K.GemvSegment(w, torch.zeros(65, 128, device="cuda"))])
    with pytest.raises(RuntimeError):
        space.image(torch.zeros(2, 516, device="cuda")[:, 2:514])         # rows that are not 16-byte aligned
    from hipengine_b200.ops.rows import SIDE_MAX_COLS
    for k in (SIDE_MAX_COLS, SIDE_MAX_COLS + 256):
        z = torch.zeros(2, k, device="cuda")
        side = lambda: space.image(z[:1], torch.ones(k, device="cuda"), 1e-6, z, torch.zeros(1, 2, device="cuda"))
        if k == SIDE_MAX_COLS:
            side()
        else:
            with pytest.raises(RuntimeError):
                side()


FIRST_LAUNCHES = """
import sys, threading
sys.path.insert(0, %r)
import torch
from hipengine_b200.models.executor import _Scratch
from hipengine_b200.ops import kernels as K
from hipengine_b200.ops.rows import RowsSpace
from hipengine_b200.quant import ggml as Q
dev = torch.device("cuda", 0)
T, k, bad = Q.GGMLType, 1024, []
raw = {t: Q.quantize(torch.randn(200, k, device=dev), t) for t in (T.Q4_K, T.Q6_K, T.Q8_0)}
w = {t: (K.to_device_weight(r, t, 200, k), Q.dequantize_torch(r, t, 200, k).double()) for t, r in raw.items()}
x = torch.randint(-9, 9, (24, k), device=dev).float()
side = torch.randn(8, k, device=dev)
torch.cuda.synchronize()
gate = threading.Barrier(9)
def run(i):
    t = list(w)[i %% 3]
    space = RowsSpace(_Scratch(dev), dev, 256)
    out, so = torch.zeros(24, 200, device=dev), torch.zeros(24, 8, device=dev)
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.synchronize()
        gate.wait()
        for _ in range(5):
            img, _ = space.image(x, torch.ones(k, device=dev), 1e-6, side, so)
            space.product(img, 24, k, [K.GemvSegment(w[t][0], out)])
    torch.cuda.synchronize()
    xn = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
    ref = xn @ w[t][1].t()
    if not float((out.double() - ref).norm() / ref.norm()) < 2 ** -10:
        bad.append((i, float((out.double() - ref).norm() / ref.norm())))
threads = [threading.Thread(target=run, args=(i,)) for i in range(9)]
[t.start() for t in threads]
[t.join(120) for t in threads]
K.check_status()
print("bad", bad, "alive", sum(t.is_alive() for t in threads))
"""


def test_first_launches_from_several_threads():
    """The shared memory that the kernels ask for depends on the block type; the first launches of a process, from nine threads
    with streams of their own, do not take it from one another."""
    import subprocess
    import sys
    from pathlib import Path
    r = subprocess.run([sys.executable, "-c", FIRST_LAUNCHES % str(Path(__file__).resolve().parent.parent)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "bad [] alive 0" in r.stdout and "Error" not in r.stderr, (r.stdout, r.stderr[-2000:])


def test_models_that_the_products_cannot_take_keep_the_other_routes(monkeypatch):
    """Rows too wide for the fp32 side products, gates of which one is quantised: the executor does without."""
    from hipengine_b200.loading.synth import build_random_model
    from hipengine_b200.loading.weights import QTensor
    from hipengine_b200.models.config import TINY_HYBRID
    from hipengine_b200.models.executor import HybridExecutor
    from hipengine_b200.ops import rows as ROWS
    w = build_random_model(TINY_HYBRID, seed=0, std=0.05).to("cuda")
    toks = list(range(1, 13))
    build = lambda: HybridExecutor(w, device="cuda", max_slots=1, max_context=64)
    ex = build()
    assert ex.rows is not None and not ex.ab_q8          # one form of the gates, the one that is used
    with monkeypatch.context() as m:
        m.setattr(ROWS, "SIDE_MAX_COLS", TINY_HYBRID.hidden - 1)
        ex = build()
    assert ex.rows is None and ex.ab_q8 and bool(ex.prefill(0, toks).isfinite().all())
    name = next(n for n in w.tensors if n.endswith("ssm_beta.weight"))
    t = w.tensors[name]
    n, k = t.shape
    w.tensors[name] = QTensor(name, T.Q8_0, t.shape, Q.quantize(t.float(), T.Q8_0).reshape(n, -1))
    ex = build()
    assert ex.rows is None
