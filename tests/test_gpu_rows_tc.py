"""The two forms of the few-row products (csrc/gemm_rows.cu, csrc/gemm_rows_tc.cu) at the edges of their row ranges."""
import pytest
import torch

from hipengine_b200.quant import ggml as Q

pytestmark = pytest.mark.gpu
T = Q.GGMLType


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
@pytest.mark.parametrize("n,k", [(127, 256), (200, 11 * 256), (129, 40 * 256)])
def test_forms_agree_and_add(t, n, k):
    """Tiles with a row more or less, odd numbers of blocks (the second operand slot empty at the end), tiles that more CTAs share than
    are summed at a time; results added to a strided residual.  Rows that the image holds exactly: what is left is the order of
    fp32 sums, sqrt(k) 2^-24 of the terms' norm; Q6_K operands above eight rows round to 11 bits."""
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops import kernels as K
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device="cuda").manual_seed(n + k)
    raw = Q.quantize(torch.randn(n, k, generator=g, device="cuda") * 0.02, t)
    w, wd = K.to_device_weight(raw, t, n, k), Q.dequantize_torch(raw, t, n, k).double()
    spaces = [RowsSpace(_Scratch(dev, canaries=True), dev, 256, m) for m in (8, 24)]
    for R in (9, 16, 17, 24, 32, 33, 48, 49, 63, 64):
        x = torch.randint(-31, 32, (R, k), generator=g, device="cuda").float()
        ref = x.double() @ wd.t()
        for space in spaces:
            out = torch.full((R, n + 5), 0.5, device="cuda")
            space.gemm(x, [K.GemvSegment(w, out[:, :n], K.EPI_ADD_F32)])
            # 0.5 and the sum: another rounding each
            bound = 2 ** -11 if t == T.Q6_K else k ** 0.5 * 2 ** -24 + 2 ** -22
            err = (out[:, :n].double() - 0.5 - ref).norm() / ref.norm()
            assert float(err) < bound and bool((out[:, n:] == 0.5).all()), (R, space.mma_rows, float(err))
            again = torch.full((R, n + 5), 0.5, device="cuda")
            space.gemm(x, [K.GemvSegment(w, again[:, :n], K.EPI_ADD_F32)])
            assert torch.equal(out, again)
    K.check_status()
    for space in spaces:
        assert int(space.counters.abs().sum()) == 0 and space.scratch.check_canaries() == []


def test_steady_side_rows():
    """fp32 side rows whose sums do not depend on the rows beside: a verify chain routes like a plain step."""
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    space = RowsSpace(_Scratch(dev), dev, 256)
    g = torch.Generator(device="cuda").manual_seed(3)
    x, nw = torch.randn(8, 2304, generator=g, device="cuda"), torch.rand(2304, generator=g, device="cuda") + 0.5
    side = torch.randn(257, 2304, generator=g, device="cuda") * 0.02
    out, one = (torch.zeros(8, 264, device="cuda") for _ in range(2))
    space.image(x, nw, 1e-6, side, out, product=False, steady=True)
    for r in range(8):
        space.image(x[r:r + 1], nw, 1e-6, side, one[r:r + 1], product=False, steady=True)
    assert torch.equal(out, one)
    xn = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * nw.double()
    ref = xn @ side.double().t()
    assert float((out[:, :257].double() - ref).norm() / ref.norm()) < 3e-6 and bool((out[:, 257:] == 0).all())


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_expert_jobs(t):
    """Experts without rows, with one, with a job more or less than full; tiles with a remainder of weight rows; ids of no expert."""
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops import kernels as K
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    space = RowsSpace(_Scratch(dev, canaries=True), dev, 256)
    cols = 64
    counts, k, H, F = [0, 1, cols - 1, cols, cols + 1, 2 * cols + 3, 0, 5], 2, 512, 200
    E, P = len(counts), sum(counts) + 2
    P += P % 2
    g = torch.Generator().manual_seed(cols)
    ids = torch.tensor([e for e, c in enumerate(counts) for _ in range(c)] + [-1] * (P - sum(counts)), dtype=torch.int32)
    ids = ids[torch.randperm(P, generator=g)].reshape(-1, k).cuda()
    gd = torch.Generator(device="cuda").manual_seed(cols)
    def weight(n, kk):
        raw = Q.quantize(torch.randn(E * n, kk, generator=gd, device="cuda") * 0.05, t)
        return K.to_device_weight(raw, t, E * n, kk), Q.dequantize_torch(raw, t, E * n, kk).double().reshape(E, n, kk)
    (wg, g64), (wu, u64), (wd, d64) = weight(F, H), weight(F, H), weight(300, 256)
    x = torch.randn(P // k, H, generator=gd, device="cuda").bfloat16()
    jobs = space.jobs(ids, E, cols)
    act = torch.full((P, F), float("nan"), device="cuda", dtype=torch.bfloat16)
    space.experts_tc(jobs, space.gather(jobs, x, k), wg, act, K.EPI_SILU_MUL, wu)
    y = torch.randn(P, 256, generator=gd, device="cuda")
    down = torch.full((P, 300), float("nan"), device="cuda")
    space.experts_tc(jobs, space.gather(jobs, y, 1), wd, down, K.EPI_F32)
    flat = ids.reshape(-1).tolist()
    for p, e in enumerate(flat):
        if e < 0:
            assert bool(act[p].isnan().all()) and bool(down[p].isnan().all())
            continue
        xp, yp = x[p // k].double(), y[p].double()
        ref = torch.nn.functional.silu(g64[e] @ xp) * (u64[e] @ xp)
        assert float((act[p].double() - ref).norm() / ref.norm()) < 6e-3, (p, e)          # bf16 result
        ref = d64[e] @ yp
        # rows round to 11 bits; Q6_K operands as well
        assert float((down[p].double() - ref).norm() / ref.norm()) < (2 ** -10.5 if t == T.Q6_K else 2 ** -11), (p, e)
    K.check_status()
    assert space.scratch.check_canaries() == []


@pytest.mark.parametrize("top,small", [(10, -12), (15, -7), (15, -14), (-14, -14)])
def test_q8_scales_far_apart_within_a_block(top, small):
    """Q8_0 scales of a block up to 2^22 apart enter exactly; beyond that a small one is a multiple of 2^-32 of the power of two of the
    largest, off by at most half of it.  Rows that are zero where the scales are large show what is left of the small ones; the largest
    scale (511.75 under its power) meets -128, the largest integer."""
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops import kernels as K
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    space, n, k = RowsSpace(_Scratch(dev, canaries=True), dev, 256), 200, 1024
    g = torch.Generator(device="cuda").manual_seed(top - small)
    scale = (1 + torch.rand(n, k // 32, generator=g, device="cuda")) * 2.0 ** small
    scale[:, ::8] = (2 - 2 ** -10) * 2.0 ** top
    q = torch.randint(-128, 128, (n, k // 32, 32), generator=g, device="cuda").to(torch.int8)
    raw = torch.cat([scale.half().view(torch.uint8).view(n, k // 32, 2), q.view(torch.uint8)], 2).reshape(n, -1).contiguous()
    w, wd = K.to_device_weight(raw, T.Q8_0, n, k), Q.dequantize_torch(raw, T.Q8_0, n, k).double()
    off = (q.double().abs() * 2.0 ** (top - 33)).reshape(n, k) if top - small > 22 else torch.zeros(n, k, dtype=torch.double, device="cuda")
    for R in (8, 32, 48, 64):
        x = torch.randint(-31, 32, (R, k), generator=g, device="cuda").float()
        x.view(R, k // 32, 32)[::2, ::8] = 0
        out = torch.zeros(R, n, device="cuda")
        space.gemm(x, [K.GemvSegment(w, out)])
        ref = x.double() @ wd.t()
        # fp32 sums: of at most k terms, each a rounding of the terms' sum
        bound = x.double().abs() @ (off + k * 2 ** -24 * wd.abs()).t()
        assert bool(((out.double() - ref).abs() <= bound).all()), (R, float(((out.double() - ref).abs() / bound).max()))
        small_rows = (out.double() - ref)[::2].norm() / ref[::2].norm()
        assert top - small > 22 or float(small_rows) < k ** 0.5 * 2 ** -24, (R, float(small_rows))
    K.check_status()
    assert space.scratch.check_canaries() == []
