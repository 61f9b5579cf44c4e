"""Packed batch descriptor: every field against the plain construction from lists."""
import pytest
import torch

from hipengine_b200.models.executor import make_batch


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("segments", [[], [(3, 0, [7])], [(1, 5, []), (2, 9, (4, 5, 2 ** 40))],
                                      [(0, 16, range(33)), (4, 0, torch.arange(2)), (2, 100, [9] * 7)],
                                      [(s, s * 3, [s]) for s in range(64)]])
def test_fields(device, segments):
    b = make_batch(segments, device)
    rows = [(int(t), s, p0 + j, si) for si, (s, p0, ids) in enumerate(segments) for j, t in enumerate(ids)]
    assert b.tokens.dtype == torch.int64 and b.tokens.tolist() == [r[0] for r in rows]
    starts = [0]
    for _, _, ids in segments:
        starts.append(starts[-1] + len(ids))
    for field, want in ((b.slot, [r[1] for r in rows]), (b.pos, [r[2] for r in rows]), (b.ctx_len, [r[2] + 1 for r in rows]),
                        (b.tok_seg, [r[3] for r in rows]), (b.seg_start, starts), (b.seg_slot, [s for s, _, _ in segments])):
        assert field.dtype == torch.int32 and field.tolist() == want and field.device.type == device
        assert field.is_contiguous() and field.data_ptr() % 16 == 0
    assert (b.T, b.n_seg, b.max_ctx) == (len(rows), len(segments), max([1] + [p0 + len(i) for _, p0, i in segments]))
    assert b.segs_host == [(s, p0, len(i)) for s, p0, i in segments]
