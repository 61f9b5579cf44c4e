"""Prompt-path kernels against the kernels or formulas that they stand in for, at their edges."""
import math

import pytest
import torch

from hipengine_b200.ref import ops as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,Hkv,pos0", [(224, 4, 2, 0), (1, 4, 2, 223), (64, 4, 2, 170), (129, 2, 1, 97),
                                          (200, 4, 1, 1000), (300, 6, 1, 64)])
def test_tensor_memory_attention_matches_64_bit(T, H, Hkv, pos0):
    """Scattered pages, ragged tiles, a context before the rows; keys past the last one hold NaN."""
    from hipengine_b200.ops import attention as A
    from hipengine_b200.ops import kernels as K
    D, last = 256, pos0 + T
    n = -(-last // 16)
    g = torch.Generator(device="cuda").manual_seed(T)
    kv = torch.randn(n + 3, 2, Hkv, 16, D, device="cuda", generator=g).bfloat16()
    pages = torch.randperm(n + 2, device="cuda", generator=g)[:n].int() + 1
    table = torch.zeros(2, n + 1, dtype=torch.int32, device="cuda")
    table[1, :n] = pages
    if last % 16:
        kv[int(pages[-1]), :, :, last % 16:] = float("nan")
    q = (3 * torch.randn(T, H, D, device="cuda", generator=g)).bfloat16()
    gate = torch.randn(T, H, D, device="cuda", generator=g).bfloat16()
    kk, vv = (kv[pages.long(), i].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :last].double() for i in (0, 1))
    s = torch.einsum("thgd,hkd->thgk", q.double().reshape(T, Hkv, H // Hkv, D), kk) / 16
    dark = torch.arange(last, device="cuda")[None] > pos0 + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgk,hkd->thgd", torch.softmax(s.masked_fill(dark[:, None, None], -math.inf), -1), vv).reshape(T, H, D)
    for gt in (None, gate):
        out = torch.zeros(T, H * D, device="cuda", dtype=torch.bfloat16)
        A.flash_prefill(q, gt, kv, table, 1, pos0, out, H, Hkv, D, 16, 1 / 16)
        want = (ref if gt is None else ref * torch.sigmoid(gt.double())).reshape(T, -1)
        # weights and outputs round to bf16 (2^-9 each)
        assert float((out.double() - want).norm() / want.norm()) < 5e-3
        assert float((out.double() - want).abs().max()) < 2e-2 * float(want.abs().max())
    K.check_status()


@pytest.mark.parametrize("lens,Hv", [([5500], 1), ([64, 1, 95], 2), ([100, 2600, 33], 2)])
def test_scan_windows_and_segments(lens, Hv):
    """More chunks than one window holds, segments of uneven length: the same recurrence as the serial kernel."""
    from hipengine_b200.ops import kernels as K
    G, S, T = 1, 128, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = R.l2norm(rand(T, G, S)) * S ** -0.5, R.l2norm(rand(T, G, S))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), rand(T, Hv * S) * 0.5], 1).contiguous()
    decay, beta = torch.exp(-0.2 * rand(T, Hv).abs()), torch.sigmoid(rand(T, Hv))
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    slot = torch.arange(len(lens), 0, -1, dtype=torch.int32, device="cuda")
    state0 = rand(len(lens) + 1, Hv, S, S) * 0.1
    outs, states = [], []
    for fn in (K.gdn_scan, K.gdn_scan_chunked):
        st, out = state0.clone(), torch.zeros(T, Hv, S, device="cuda")
        fn(qkv, decay, beta, st, start, slot, out, G, Hv)
        outs.append(out)
        states.append(st)
    assert torch.equal(states[1][0], state0[0])
    for a, b in ((outs[1], outs[0]), (states[1], states[0])):
        assert float((a - b).norm() / b.norm()) < 2e-3          # TF32 products against fp32
    st, out = state0.clone(), torch.zeros(T, Hv, S, device="cuda")
    K.gdn_scan_chunked(qkv, decay, beta, st, start, slot, out, G, Hv, write_state=False)
    assert torch.equal(st, state0) and float((out - outs[1]).norm() / outs[1].norm()) < 1e-6
