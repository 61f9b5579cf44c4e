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
