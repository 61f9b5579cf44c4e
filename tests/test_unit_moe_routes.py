"""Routes of an expert prompt's pairs (models/moe.py): the lines lie where the routes were measured to cross, by block type."""
from types import SimpleNamespace

import pytest

from hipengine_b200.models import moe as M
from hipengine_b200.quant.ggml import GGMLType as T


def _executor(gate, up, down, experts=256, rows=True):
    types = {"gate": gate, "up": up, "down": down}
    weight = lambda i, name: SimpleNamespace(qtype=int(types[name.split("_")[1]]), n_cols=512)
    return SimpleNamespace(cfg=SimpleNamespace(n_experts=experts, hidden=2048), rows=object() if rows else None, W=weight)


@pytest.mark.parametrize("gate,down,few,tc", [(T.Q4_K, T.Q4_K, 28, 112), (T.Q4_K, T.Q6_K, 28, 112), (T.Q8_0, T.Q8_0, 32, 64),
                                              (T.Q4_K, T.Q8_0, 32, 64), (T.Q8_0, T.Q6_K, 32, 64)])
def test_lines_by_block_type(gate, down, few, tc):
    for experts in (16, 256):
        ex = _executor(gate, gate, down, experts)
        route = lambda load, more=0: M._prompt_route(ex, 0, load * experts + more, None)
        assert route(few) == "jobs" and route(few, 1) == "jobs_tc" and route(tc) == "jobs_tc" and route(tc, 1) == "grouped"


def test_what_the_jobs_cannot_take_is_grouped():
    for load in (8, 40, 100, 200):
        for ex, rng in ((_executor(T.Q4_K, T.Q4_K, T.Q6_K), (0, 128)), (_executor(T.Q4_K, T.Q4_K, T.Q6_K, rows=False), None),
                        (_executor(T.Q4_K, T.Q4_K, T.Q5_K), None), (_executor(T.Q4_K, T.Q6_K, T.Q4_K), None),
                        (_executor(T.Q4_K, T.Q4_K, T.Q4_K, experts=513), None)):
            assert M._prompt_route(ex, 0, load * ex.cfg.n_experts, rng) == "grouped"
