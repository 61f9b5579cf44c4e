"""Quantised GEMM with several activation tiles per call: even and odd numbers of them, ragged last ones, more units than SMs."""
import pytest
import torch

from hipengine_b200.quant import ggml as Q

pytestmark = pytest.mark.gpu
T = Q.GGMLType


@pytest.mark.parametrize("t", [T.Q4_K, T.Q6_K, T.Q8_0])
@pytest.mark.parametrize("M,N,K", [(193, 130, 256), (385, 128, 512), (577, 300, 768), (777, 2432, 1280), (1000, 2560, 256),
                                   (4096, 1024, 1024), (2048, 6144, 256)])
def test_units_of_two_tiles(t, M, N, K):
    from hipengine_b200.models.executor import _Scratch
    from hipengine_b200.ops import gemm as GM
    from hipengine_b200.ops import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(M)
    raw = Q.quantize(torch.randn(N, K, generator=g, device="cuda") * 0.02, t)
    w = KK.to_device_weight(raw, t, N, K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    sc = _Scratch(torch.device("cuda", torch.cuda.current_device()), canaries=True)
    out = torch.full((M, N + 8), float("nan"), device="cuda")
    GM.gemm_quant(x, w, out[:, :N], sc)
    ref = x.double() @ Q.dequantize_torch(raw, t, N, K).bfloat16().double().t()     # the operands are the bf16 weights
    # exact products, fp32 sums of K terms: a relative error of at most sqrt(K) * 2^-24 for random signs, with room for the
    # few weights whose fp32 dequantisation rounds to the other bf16 neighbour
    assert float((out[:, :N].double() - ref).norm() / ref.norm()) < 2e-4
    assert bool(out[:, N:].isnan().all()) and sc.check_canaries() == []
    again = torch.zeros(M, N, device="cuda")
    GM.gemm_quant(x, w, again, sc)
    assert torch.equal(again, out[:, :N])
    KK.check_status()
