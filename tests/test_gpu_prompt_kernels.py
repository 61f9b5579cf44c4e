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


@pytest.mark.parametrize("T,pos0,size", [(777, 0, 1.0), (600, 2000, 2.0), (512, 3000, 3.0), (300, 100, 8.0)])
def test_tensor_memory_attention_loses_nothing_but_the_output_rounding(T, pos0, size):
    """Flat to peaked weights, maxima that grow a little at a time: what is left is the output's bf16."""
    from hipengine_b200.ops import attention as A
    H, G, D, last = 8, 2, 256, pos0 + T
    n = -(-last // 16)
    g = torch.Generator(device="cuda").manual_seed(T)
    kv = torch.randn(n, 2, G, 16, D, device="cuda", generator=g).bfloat16()
    q = (size * torch.randn(T, H, D, device="cuda", generator=g)).bfloat16()
    out = torch.zeros(T, H * D, device="cuda", dtype=torch.bfloat16)
    A.flash_prefill(q, None, kv, torch.arange(n, device="cuda", dtype=torch.int32)[None].contiguous(), 0, pos0, out, H, G, D, 16, 1 / 16)
    k, v = (kv[:, i].permute(1, 0, 2, 3).reshape(G, -1, D)[:, :last].double() for i in (0, 1))
    s = torch.einsum("thgd,hkd->thgk", q.double().reshape(T, G, H // G, D), k) / 16
    dark = torch.arange(last, device="cuda")[None] > pos0 + torch.arange(T, device="cuda")[:, None]
    want = torch.einsum("thgk,hkd->thgd", torch.softmax(s.masked_fill(dark[:, None, None], -math.inf), -1), v).reshape(T, -1)
    least = float((want.bfloat16().double() - want).norm())
    # scores are fp32 sums of 256 products: 2^-20 of scores up to 60 beside the output's 2^-9
    assert float((out.double() - want).norm()) < 1.01 * least


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


@pytest.mark.parametrize("lens", [[700] * 8, [64] * 40, [5200, 64, 300], [65] * 165, [2000, 100, 33]])
def test_scan_of_packed_prompts_makes_no_empty_passes(lens):
    """With the longest segment given: as many passes as it has windows, the results of the scan that was not told."""
    from hipengine_b200.ops import kernels as K
    G, Hv, S, T, n = 1, 1, 128, sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = R.l2norm(rand(T, G, S)) * S ** -0.5, R.l2norm(rand(T, G, S))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), rand(T, Hv * S) * 0.5], 1).contiguous()
    decay, beta = torch.exp(-0.2 * rand(T, Hv).abs()), torch.sigmoid(rand(T, Hv))
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    slot = torch.arange(n, dtype=torch.int32, device="cuda")
    state0 = rand(n, Hv, S, S) * 0.1
    per = max(1, 160 // n) if T // 32 + n > 160 else -(-max(lens) // 32)
    res = []
    for longest in (0, max(lens)):
        st, out = state0.clone(), torch.zeros(T, Hv, S, device="cuda")
        before = K.launch_count()
        K.gdn_scan_chunked(qkv, decay, beta, st, start, slot, out, G, Hv, longest=longest)
        res.append((st, out, K.launch_count() - before))
    assert res[1][2] == 2 * -(-(-(-max(lens) // 32)) // per) <= res[0][2]
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    st, out = state0.clone(), torch.zeros(T, Hv, S, device="cuda")
    K.gdn_scan(qkv, decay, beta, st, start, slot, out, G, Hv)
    for a, b in ((res[1][1], out), (res[1][0], st)):
        assert float((a - b).norm() / b.norm()) < 2e-3          # TF32 products against fp32


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[1], [2, 3, 40], [17, 1, 16, 100]])
def test_front_is_convolution_then_preparation(dtype, lens):
    from hipengine_b200.ops import kernels as K
    G, Hv, S, T = 2, 6, 128, sum(lens)
    C = 2 * G * S + Hv * S
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, ab = rand(T, C + 8).to(dtype)[:, :C], rand(C, 4) * 0.5, rand(T, 2 * Hv + 4)
    a, b, ssm_a, dt = ab[:, :Hv], ab[:, Hv:2 * Hv], -rand(Hv).abs(), rand(Hv)
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    slot = torch.arange(len(lens), 0, -1, dtype=torch.int32, device="cuda")
    seg = torch.repeat_interleave(torch.arange(len(lens), device="cuda", dtype=torch.int32), torch.tensor(lens, device="cuda"))
    state0 = rand(len(lens) + 1, C, 3)
    got, want = [], []
    for res, front in ((got, True), (want, False)):
        st, out = state0.clone(), torch.zeros(T, C, device="cuda")
        decay, beta = torch.zeros(T, Hv, device="cuda"), torch.zeros(T, Hv, device="cuda")
        if front:
            K.gdn_front(x, w, st, start, slot, out, a, b, ssm_a, dt, decay, beta, G, Hv)
        else:
            K.conv1d(x, w, st, start, slot, seg, out, C)
            K.gdn_prepare(out, a, b, ssm_a, dt, decay, beta, G, Hv, S)
        res += [st, out, decay, beta]
    assert torch.equal(got[0], want[0])
    for p, q in zip(got[1:], want[1:]):
        assert torch.allclose(p, q, rtol=1e-5, atol=1e-6)


def test_front_and_scan_refuse_operands_that_are_not_aligned():
    from hipengine_b200.ops import kernels as K
    G, Hv, T = 1, 1, 64
    C = 3 * 128
    z = lambda *s: torch.zeros(*s, device="cuda")
    start, slot = torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    odd = lambda *s: z(torch.Size(s).numel() + 1)[1:].view(*s)
    ab, one = z(T, Hv), z(Hv)
    for w, out in ((odd(C, 4), z(T, C)), (z(C, 4), odd(T, C))):
        with pytest.raises(RuntimeError):
            K.gdn_front(z(T, C), w, z(1, C, 3), start, slot, out, ab, ab, one, one, z(T, Hv), z(T, Hv), G, Hv)
    for qkv, ws in ((odd(T, C), None), (z(T, C), odd(K.gdn_chunk_ws_floats(T, 1, Hv)))):
        with pytest.raises(RuntimeError):
            K.gdn_scan_chunked(qkv, z(T, Hv), z(T, Hv), z(1, Hv, 128, 128), start, slot, z(T, Hv, 128), G, Hv, ws=ws)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 33])
def test_gated_norm_of_128_columns(dtype, T):
    from hipengine_b200.ops import kernels as K
    Hv = 5
    o, w = torch.randn(T, Hv, 128, device="cuda"), torch.rand(128, device="cuda") + 0.5
    z = torch.randn(T, Hv * 128 + 8, device="cuda").to(dtype)[:, :Hv * 128]
    out = torch.zeros(T, Hv * 128 + 4, device="cuda", dtype=torch.bfloat16)[:, :Hv * 128]
    K.gdn_gated_norm(o, z, w, out, Hv, 128, 1e-6)
    ref = R.gated_rmsnorm(o, w, z.float().reshape(T, Hv, 128), 1e-6).reshape(T, -1)
    assert torch.allclose(out.float(), ref, rtol=8e-3, atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gated,rope,qk_norm", [(True, 64, True), (False, 256, True), (False, 0, False), (True, 16, False)])
def test_projection_rows_match_the_per_head_kernel(dtype, gated, rope, qk_norm):
    """16 tokens and more go a token per CTA; the same rows one by one go a head per CTA."""
    from hipengine_b200.ops import kernels as K
    T, H, Hkv, D = 19, 6, 2, 256
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = (rand(T, n).to(dtype) for n in (H * D * (2 if gated else 1), Hkv * D, Hkv * D))
    qn, kn = (rand(D).abs() + 0.5, rand(D).abs() + 0.5) if qk_norm else (None, None)
    table = torch.randperm(8, device="cuda", generator=g).int().reshape(2, 4)
    slot = torch.ones(T, dtype=torch.int32, device="cuda")
    pos = torch.arange(11, 11 + T, dtype=torch.int32, device="cuda")
    res = []
    for step in (T, 1):
        qo, go = torch.zeros(T, H, D, device="cuda", dtype=torch.bfloat16), torch.zeros(T, H, D, device="cuda", dtype=torch.bfloat16)
        kv = torch.zeros(9, 2, Hkv, 16, D, device="cuda", dtype=torch.bfloat16)
        for r in range(0, T, step):
            s = slice(r, r + step)
            K.qkv_post(q[s], k[s], v[s], qn, kn, qo[s], go[s] if gated else None, kv, table, slot[s], pos[s], H, Hkv, D, 16,
                       gated, rope, 1e7, 1e-6)
        res.append((qo, go, kv))
    for a, b in zip(*res):
        assert torch.allclose(a.float(), b.float(), rtol=8e-3, atol=1e-5)      # one bf16 rounding apart at most


@pytest.mark.parametrize("K", [256, 5120, 6144, 6148, 9000])
def test_single_row_gates_in_the_decode_step(K):
    """Gates from the residual row inside the step against gates given to it: fewer columns than threads, all that a thread keeps
    in registers (6144), and what it loads in place beyond."""
    from hipengine_b200.ops import kernels as Kn
    G, Hv, S = 2, 6, 128
    C = 2 * G * S + Hv * S
    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    h, norm, gw = 3 * rand(1, K), rand(K).abs() + 0.5, rand(2 * Hv, K) * K ** -0.5
    xn = h.double() * torch.rsqrt(h.double().square().mean(-1, keepdim=True) + 1e-6) * norm.double()
    ab = (xn @ gw.double().t()).float()
    x, w, z = rand(1, C), rand(C, 4) * 0.5, rand(1, Hv * S)
    ssm_a, dt, nw, slot = -rand(Hv).abs(), rand(Hv), rand(S).abs(), torch.tensor([1], dtype=torch.int32, device="cuda")
    conv0, state0 = rand(2, C, 3), rand(2, Hv, S, S) * 0.1
    res = []
    for gates in (None, (gw, h, norm, 1e-6)):
        conv, state = conv0.clone(), state0.clone()
        qkv, decay, beta = torch.zeros(1, C, device="cuda"), torch.zeros(1, Hv, device="cuda"), torch.zeros(1, Hv, device="cuda")
        out = torch.zeros(1, Hv * S, device="cuda", dtype=torch.bfloat16)
        a, b = (ab[:, :Hv], ab[:, Hv:]) if gates is None else (None, None)
        Kn.gdn_decode(x, w, conv, a, b, ssm_a, dt, slot, qkv, decay, beta, state, z, nw, out, G, Hv, 1e-6, gates)
        res.append((decay, beta, state, conv, out.float()))
    for got, want, tol in zip(res[1], res[0], (1e-5, 1e-5, 1e-5, 0, 8e-3)):       # fp32 sums; the output is bf16
        assert torch.allclose(got, want, rtol=tol, atol=tol)
