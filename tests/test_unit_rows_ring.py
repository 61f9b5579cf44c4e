"""The ring of the few-row products on tcgen05 (csrc/gemm_rows_tc.cu): whatever the order in which its warps run, none of them
misses the phase of a barrier that it waits for."""
import ctypes as C

import pytest

from hipengine_b200.core import native
from hipengine_b200.quant.ggml import GGMLType as T

BLOCKS = 13


def _lost(stages: int, parity, shared: bool) -> bool:
    """Can the pipeline stop short of the last block, or a group take a block that has not landed?  All orders of: a producer that
    loads block j into stage j % stages, two groups of expanding warps (one of each stands for the group's last) that take blocks in turn,
    waiting for the arrival of block j with parity[j], and a summer that follows the expanded blocks and gives their stages back.
    An arrival is signalled to the group that takes the block, or (`shared`) to both, which in an odd ring have to look at each
    other's blocks then.  A barrier is the number of its completed phases; a wait for a parity passes while the last one has it."""
    passes = lambda phases, p: phases & 1 != p
    look = shared and stages % 2 == 1
    start = (0, (0, 0), 0)                                # loaded, next block of each group, summed
    todo, seen = [start], {start}
    while todo:
        loaded, at, summed = state = todo.pop()
        after = []
        s = loaded % stages
        if loaded < BLOCKS and (loaded < stages or passes((summed - s + stages - 1) // stages, loaded // stages - 1 & 1)):
            after.append((loaded + 1, at, summed))
        for g in range(2):
            j = at[g]
            if j == BLOCKS:
                continue
            phases = sum(i % stages == j % stages and (shared or i % 2 == j % 2) for i in range(loaded))
            if j % 2 == g or look:
                if not passes(phases, parity[j]):
                    continue
                if j >= loaded:
                    return True
            after.append((loaded, (j + 1, at[1]) if g == 0 else (at[0], j + 1), summed))
        if summed < BLOCKS and at[summed % 2] > summed:
            after.append((loaded, at, summed + 1))
        if not after and state != (BLOCKS, (BLOCKS, BLOCKS), BLOCKS):
            return True
        for x in after:
            if x not in seen:
                seen.add(x)
                todo.append(x)
    return False


@pytest.mark.skipif(not native.lib_available(), reason="native library not built")
def test_no_group_misses_the_arrival_of_a_block():
    per_lap = lambda n: [j // n & 1 for j in range(BLOCKS)]
    assert _lost(3, per_lap(3), True) and not _lost(4, per_lap(4), True) and _lost(3, per_lap(3), False)
    stage, parity, odd = (C.c_int * BLOCKS)(), (C.c_int * BLOCKS)(), 0
    for rows in (17, 32, 33, 48, 49, 64):
        for t in (T.Q4_K, T.Q6_K, T.Q8_0):
            stages = native.lib().he_rows_tc_walk(C.c_int(rows), C.c_int(int(t)), C.c_int(BLOCKS), stage, parity)
            assert stages >= 2 and list(stage) == [j % stages for j in range(BLOCKS)]
            assert not _lost(stages, list(parity), False), (rows, t, stages, list(parity))
            odd += stages % 2
    assert odd > 0
