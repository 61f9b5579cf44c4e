"""The few-row products and expert jobs on tcgen05 (csrc/gemm_rows_tc.cu) in their steady state: CTAs of many blocks, so that stages,
operand slots and accumulators are used again and again."""
import pytest
import torch

from hipengine_b200.quant import ggml as Q

pytestmark = pytest.mark.gpu
T = Q.GGMLType


def _space():
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    return RowsSpace(_Scratch(dev, canaries=True), dev, 13000)


def _weight(t, n, k, seed, experts=1):
    from hipengine_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(seed)
    raw = Q.quantize(torch.randn(experts * n, k, generator=g, device="cuda") * 0.02, t)
    return K.to_device_weight(raw, t, experts * n, k), Q.dequantize_torch(raw, t, experts * n, k)


def _whole(R, k, seed):
    """Rows that their image holds exactly."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-31, 32, (R, k), generator=g, device="cuda").float()


def _bound(t, k):
    """fp32 sums of k terms; Q6_K operands round to 11 bits."""
    return 2 ** -11 if t == T.Q6_K else k ** 0.5 * 2 ** -24


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_many_blocks_a_cta(t):
    """12300 x 5120: 97 tiles of 20 blocks, 13 or 14 blocks for each of 148 CTAs, ranges that start and end within tiles."""
    from hipengine_b200.ops import kernels as K
    space, n, k = _space(), 12300, 5120
    w, wd = _weight(t, n, k, 1)
    for R in (25, 32, 33, 48, 49, 64):
        x = _whole(R, k, R)
        out, again = (torch.full((R, n), float("nan"), device="cuda") for _ in range(2))
        for o in (out, again):
            space.gemm(x, [K.GemvSegment(w, o)])
        ref = x.double() @ wd.t().double()
        assert float((out.double() - ref).norm() / ref.norm()) < _bound(t, k) and torch.equal(out, again), R
    K.check_status()
    assert int(space.counters.abs().sum()) == 0 and space.scratch.check_canaries() == []


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 2, 1, 0), (1, 3, 0, 2)])
def test_segments_of_several_types_within_a_cta(order):
    """Four segments, 15 or 16 blocks a CTA: the CTAs at the three boundaries go from one block type to the next (Q8_0 hands its
    operands over in four parts, the others in two)."""
    from hipengine_b200.ops import kernels as K
    space, k = _space(), 5120
    (a, ad), (b, bd), (c, cd) = _weight(T.Q8_0, 3700, k, 1), _weight(T.Q6_K, 3800, k, 2), _weight(T.Q4_K, 2900, k, 3)
    (g, gd), (u, ud) = _weight(T.Q8_0, 1800, k, 4), _weight(T.Q8_0, 1800, k, 5)
    for R in (32, 48, 64):
        x = _whole(R, k, R)
        results = []
        for _ in range(2):
            o = [torch.full((R, w.n_rows), float("nan"), device="cuda") for w in (a, b, c)]
            act = torch.full((R, 1800), float("nan"), device="cuda", dtype=torch.bfloat16)
            segs = [K.GemvSegment(a, o[0]), K.GemvSegment(b, o[1]), K.GemvSegment(c, o[2]), K.GemvSegment(g, act, K.EPI_SILU_MUL, u)]
            space.gemm(x, [segs[i] for i in order])
            results.append([*o, act])
        for t, y, wd in zip((T.Q8_0, T.Q6_K, T.Q4_K), results[0], (ad, bd, cd)):
            ref = x.double() @ wd.t().double()
            assert float((y.double() - ref).norm() / ref.norm()) < _bound(t, k), (R, t)
        ref = torch.nn.functional.silu(x.double() @ gd.t().double()) * (x.double() @ ud.t().double())
        assert float((results[0][3].double() - ref).norm() / ref.norm()) < 2 ** -8          # bf16 result
        assert all(torch.equal(p, q) for p, q in zip(*results)), R
    K.check_status()
    assert int(space.counters.abs().sum()) == 0 and space.scratch.check_canaries() == []


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
def test_several_items_a_cta(t):
    """Jobs of 64 rows: 28 x 24 gate/up items of eight blocks, 28 x 16 down items of six, three to five a CTA."""
    from hipengine_b200.ops import kernels as K
    space, cols, k, H, F = _space(), 64, 4, 2048, 1536
    counts = [0, 1, 63, 64, 65, 128, 129, 200, 3, 17, 90, 64, 140, 96, 70, 122]
    E, P = len(counts), sum(counts)
    counts[-1] += -P % k
    P += -P % k
    assert sum(-(-c // cols) for c in counts) == 28
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    flat = ids[torch.randperm(P, generator=torch.Generator().manual_seed(1))]
    ids = flat.int().reshape(-1, k).cuda()
    (wg, gd), (wu, ud), (wd, dd) = _weight(t, F, H, 1, E), _weight(t, F, H, 2, E), _weight(t, H, F, 3, E)
    x, y = _whole(P // k, H, 1), _whole(P, F, 2)
    got = []
    for _ in range(2):
        jobs = space.jobs(ids, E, cols)
        act = torch.full((P, F), float("nan"), device="cuda", dtype=torch.bfloat16)
        space.experts_tc(jobs, space.gather(jobs, x, k), wg, act, K.EPI_SILU_MUL, wu)
        down = torch.full((P, H), float("nan"), device="cuda")
        space.experts_tc(jobs, space.gather(jobs, y, 1), wd, down, K.EPI_F32)
        got.append((act, down))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    for e in range(E):
        p = (flat == e).nonzero().flatten().cuda()
        if p.numel() == 0:
            continue
        xe, of = x[p // k].double(), lambda m, n: m[e * n:(e + 1) * n].double().t()
        ref = torch.nn.functional.silu(xe @ of(gd, F)) * (xe @ of(ud, F))
        assert float((got[0][0][p].double() - ref).norm() / ref.norm()) < 2 ** -8, e        # bf16 result
        ref = y[p].double() @ of(dd, H)
        assert float((got[0][1][p].double() - ref).norm() / ref.norm()) < _bound(t, F), e
    K.check_status()
    assert space.scratch.check_canaries() == []
