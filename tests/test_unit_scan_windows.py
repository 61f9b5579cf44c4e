"""Passes of the chunked delta-rule scan: they cover every chunk of every segment within the workspace that the caller sizes."""
import random

import pytest

from hipengine_b200.core import native

UNIT = 32 * 128 * 2 + 32 * 32 + 32        # workspace floats of a chunk and head
CHUNK = 32


@pytest.mark.skipif(not native.lib_available(), reason="native library not built")
def test_passes_cover_the_chunks_within_the_workspace():
    from hipengine_b200.ops import kernels as K
    rng = random.Random(0)
    for case in range(400):
        n = rng.choice([1, 2, 3, 8, 40, 159, 160, 161, 300])
        lens = [rng.choice([1, 31, 32, 33, 64, rng.randint(1, 6000)]) for _ in range(n)]
        if case % 3 == 0:
            lens = [lens[0]] * n
        T, longest = sum(lens), max(lens)
        units, rest = divmod(K.gdn_chunk_ws_floats(T, n, 1), UNIT)
        assert rest == 0 and units <= max(160, n)
        for given in (longest, 0):
            passes = K.gdn_chunk_windows(T, n, True, given)
            # chunks of a segment in one pass: all, or an equal share of what the workspace holds
            total = T // CHUNK + n
            per = -(-(given or T) // CHUNK) if total <= 160 else max(1, 160 // n)
            chunks = [-(-m // CHUNK) for m in lens]
            assert passes * per >= max(chunks) and (given == 0 or (passes - 1) * per < max(chunks))
            for p in range(passes):
                assert sum(max(0, min(c, (p + 1) * per) - p * per) for c in chunks) <= units
    assert K.gdn_chunk_windows(4096, 8, True, 512) == 1 and K.gdn_chunk_windows(4096, 32, True, 128) == 1
    assert K.gdn_chunk_windows(9000, 1, False, 0) == 1 and K.gdn_chunk_windows(9000, 1, True, 0) == 2
