"""The ring of the few-row products on tcgen05 (csrc/gemm_rows_tc.cu): whatever the order in which its warps run, none of them
misses the phase of a barrier that it waits for."""
import ctypes as C

import pytest

from hipengine_b200.core import native
from hipengine_b200.quant.ggml import GGMLType as T

BLOCKS = 9


def _lost(stages: int, arrivals: int) -> bool:
    """Can the pipeline stop short of the last block?  All orders of: a producer that loads block j into stage j % stages, two groups
    of expanding warps (one of each stands for the group's last) that take blocks in turn and, in an odd ring, look at the other
    group's too, arriving on the stage's `empty` if it counts them (`arrivals`); a summer that follows the expanded blocks.
    A barrier is the number of its completed phases; a wait for parity p passes while the last completed one has it."""
    passes = lambda phases, p: phases & 1 != p
    own = stages % 2 == 0
    start = (0, (0, 0), 0, (0,) * stages)                 # loaded, next block of each group, summed, group arrivals at `empty`
    todo, seen = [start], {start}
    while todo:
        loaded, at, summed, come = state = todo.pop()
        after = []
        full = [(loaded - s + stages - 1) // stages for s in range(stages)]
        # a stage is given back once its block is summed and, where they are counted, the other group's warps have come by
        given = [min((summed - s + stages - 1) // stages, come[s] if arrivals else BLOCKS) for s in range(stages)]
        s = loaded % stages
        if loaded < BLOCKS and (loaded < stages or passes(given[s], loaded // stages - 1 & 1)):
            after.append((loaded + 1, at, summed, come))
        for g in range(2):
            j = at[g]
            if j == BLOCKS:
                continue
            mine, s = j % 2 == g, j % stages
            if (mine or not own) and not passes(full[s], j // stages & 1):
                continue
            nxt = (j + 1, at[1]) if g == 0 else (at[0], j + 1)
            here = list(come)
            if not mine and not own:
                here[s] += 1
            after.append((loaded, nxt, summed, tuple(here)))
        if summed < BLOCKS and at[summed % 2] > summed:
            after.append((loaded, at, summed + 1, come))
        if not after and state[:3] != (BLOCKS, (BLOCKS, BLOCKS), BLOCKS):
            return True
        for x in after:
            if x not in seen:
                seen.add(x)
                todo.append(x)
    return False


@pytest.mark.skipif(not native.lib_available(), reason="native library not built")
def test_no_stage_is_loaded_again_before_both_groups_have_seen_it():
    assert _lost(3, 0) and not _lost(3, 1) and not _lost(4, 0) and not _lost(2, 0)
    odd = 0
    for rows in (17, 32, 33, 48, 49, 64):
        for t in (T.Q4_K, T.Q6_K, T.Q8_0):
            n = C.c_int(-1)
            stages = native.lib().he_rows_tc_ring(C.c_int(rows), C.c_int(int(t)), C.byref(n))
            assert stages >= 2 and not _lost(stages, n.value), (rows, t, stages, n.value)
            odd += stages % 2
    assert odd > 0
