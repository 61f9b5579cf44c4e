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
