"""Routed experts as jobs (csrc/moe_rows.cu): the job list, the products of the jobs and the weighted sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def space():
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops.rows import RowsSpace
    dev = torch.device("cuda", torch.cuda.current_device())
    return RowsSpace(_Scratch(dev, canaries=True), dev, 5000)


def _ids_of_counts(counts, k, seed):
    """Expert ids [T, k] in which expert e appears counts[e] times, in random order."""
    flat = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    flat = flat[torch.randperm(flat.numel(), generator=torch.Generator().manual_seed(seed))]
    return flat.to(torch.int32).reshape(-1, k).cuda()


@pytest.mark.parametrize("cols", [8, 16, 32])
@pytest.mark.parametrize("E,rows", [(3, 4), (32, 4), (33, 1), (512, 4), (512, 70)])
def test_job_list(space, cols, E, rows):
    """Every pair in one job of its expert, in ascending order, jobs full except an expert's last; ids that are no expert's
    are in no job."""
    g = torch.Generator().manual_seed(E + cols)
    ids = torch.randint(0, E, (rows * cols + 3, 5), generator=g).int()
    ids[:, 0] = E - 1                                   # one expert of several jobs
    for k, bad in ((7, -1), (11, E), (12, 0x7FFFFFFF), (30, -0x80000000)):
        ids.view(-1)[k] = bad
    j = space.jobs(ids.cuda(), E, cols)
    n, flat = int(j.meta[0]), ids.view(-1).tolist()
    entries, jobs = j.entries.cpu().tolist(), j.list[:n].cpu().tolist()
    seen, of = [], {}
    for e, first, count, _ in jobs:
        assert 1 <= count <= cols and 0 <= e < E
        assert all(flat[p] == e for p in entries[first:first + count])
        seen += entries[first:first + count]
        of.setdefault(e, []).append(count)
    assert seen == sorted((p for p, e in enumerate(flat) if 0 <= e < E), key=lambda p: (flat[p], p))
    assert all(c == cols for counts in of.values() for c in counts[:-1])
    assert space.scratch.check_canaries() == []


def _weight(t, n, k, seed):
    from hipengine_b200.ops import kernels as K
    from hipengine_b200.quant import ggml as Q
    g = torch.Generator(device="cuda").manual_seed(seed)
    raw = Q.quantize(torch.randn(n, k, generator=g, device="cuda") * 0.02, t)
    return K.to_device_weight(raw, t, n, k), Q.dequantize_torch(raw, t, n, k).double()


def _types():
    from hipengine_b200.quant.ggml import GGMLType as T
    return [T.Q4_K, T.Q6_K, T.Q8_0]


@pytest.mark.parametrize("t", _types())
def test_crowded_experts_repeat(space, t):
    """Experts of more rows than a job: the same rows fall into the short last one, whose sums take another order, every time."""
    from hipengine_b200.ops import kernels as K
    counts, n, k = [33, 48, 7, 40], 160, 768
    w, _ = _weight(t, len(counts) * n, k, 3)
    ids = _ids_of_counts(counts, 1, 0)
    x = torch.randn(ids.shape[0], k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    rows = space.image(x, by_row=True, product=False)[1]
    first = None
    for i in range(20):
        out = torch.full((ids.shape[0], n), float("nan"), device="cuda")
        space.experts(space.jobs(ids, len(counts), 32), rows, 1, w, out, K.EPI_F32)
        first = out if first is None else first
        assert torch.equal(out, first), i
    K.check_status()


@pytest.mark.parametrize("t", _types())
@pytest.mark.parametrize("cols,n", [(8, 96), (16, 130), (32, 300), (8, 512)])
def test_products_of_jobs_match_64_bit(space, t, cols, n):
    """Experts of no row, one, a job's worth, one more and several jobs; tiles that end inside an expert's rows (the box reaches
    into the next expert); token rows that two pairs share and rows of their own; rows that the image holds exactly."""
    from hipengine_b200.ops import kernels as K
    counts, k = [0, 1, cols, cols + 1, 3 * cols + 4], 768
    E = len(counts)
    (a, ad), (b, bd) = _weight(t, E * n, k, n), _weight(t, E * n, k, n + 1)
    ids = _ids_of_counts(counts, 2, cols)
    P = ids.numel()
    jobs = space.jobs(ids, E, cols)
    e = ids.view(-1).long()
    ad, bd = ad.reshape(E, n, k)[e], bd.reshape(E, n, k)[e]
    g = torch.Generator(device="cuda").manual_seed(cols)
    rel = lambda y, r: float((y.double() - r).norm(dim=1).div(r.norm(dim=1)).max())
    x = torch.randint(-31, 32, (P // 2, k), generator=g, device="cuda").float() / 16
    img = space.image(x, by_row=True, product=False)[1]
    up = lambda m: torch.einsum("pk,pnk->pn", x.double()[torch.arange(P, device="cuda") // 2], m)
    for epi, f in ((K.EPI_SILU_MUL, torch.nn.functional.silu), (K.EPI_GELU_MUL, lambda v: torch.nn.functional.gelu(v, approximate="tanh"))):
        act = torch.full((P + 1, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        space.experts(jobs, img, 2, a, act[:P, :n], epi, b)
        assert rel(act[:P, :n], f(up(ad)) * up(bd)) < 4e-3                       # bf16 result
        assert bool((act[P] == 7).all()) and bool((act[:, n:] == 7).all())
    rows = torch.randint(-31, 32, (P, k), generator=g, device="cuda").bfloat16()
    img = space.image(rows, by_row=True, product=False)[1]
    want = torch.einsum("pk,pnk->pn", rows.double(), ad)
    out = torch.full((P + 1, n + 4), 7.0, device="cuda")
    space.experts(jobs, img, 1, a, out[:P, :n], K.EPI_F32)
    # fp32 sums of 768 terms; Q6_K operands of 32-row jobs round to 11 bits
    assert rel(out[:P, :n], want) < (2 ** -11 if t == _types()[1] and cols == 32 else 28 * 2 ** -24)
    assert bool((out[P] == 7).all()) and bool((out[:, n:] == 7).all())
    half = torch.zeros(P, n, device="cuda", dtype=torch.bfloat16)
    space.experts(jobs, img, 1, a, half, K.EPI_BF16)
    assert torch.equal(half, out[:P, :n].bfloat16())
    K.check_status()
    assert space.scratch.check_canaries() == []


@pytest.mark.parametrize("T,k,n", [(1, 1, 4), (3, 8, 1028), (70, 2, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sum_of_pairs(space, T, k, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    h, y, w = rand(T, n + 4)[:, :n], rand(T * k, n).to(dtype), torch.rand(T, k, generator=g, device="cuda")
    sh, gate = rand(T, n).bfloat16(), rand(T, 3)
    want = h.double() + (w.double()[..., None] * y.double().reshape(T, k, n)).sum(1)
    for shared in (False, True):
        got = h.clone()
        space.sum_pairs(got, y, w, sh if shared else None, gate[:, 1:2] if shared else None)
        ref = want + torch.sigmoid(gate[:, 1:2].double()) * sh.double() if shared else want
        assert float((got.double() - ref).abs().max()) < 1e-5                    # fp32 sums of at most ten terms below 30


def test_sum_of_pairs_refuses_rows_that_are_not_aligned(space):
    """Rows are read four columns at once."""
    h, y, w = torch.zeros(2, 12, device="cuda"), torch.zeros(4, 12, device="cuda"), torch.zeros(2, 2, device="cuda")
    sh = torch.zeros(2, 12, device="cuda", dtype=torch.bfloat16)
    for a, b, c in ((h[:, 1:9], y[:, :8], None), (h[:, :8], y[:, 2:10], None), (h[:, :8], y.bfloat16()[:, 2:10], None),
                    (h[:, :8], y[:, :8], sh[:, 1:9])):
        with pytest.raises(RuntimeError):
            space.sum_pairs(a, b, w, c)
