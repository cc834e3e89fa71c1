"""A query that stays while targets are loaded in turn: every pass runs on the
target loaded last, completely loaded."""
import numpy as np
import pytest

from hspz_b200 import EngineConfig, sequence, synth
from hspz_b200.build import build
from tests.test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build()


def _pair(seed, n):
    rng = np.random.default_rng(seed)
    targets = [synth.random_bases(rng, n), synth.random_bases(rng, n // 2)]
    query = synth.random_bases(rng, 400_000)
    for t in targets:
        synth.plant(rng, t, query, 30, 200, 3000, 0.05, 0.3)
    return targets, query


@pytest.mark.parametrize("tables", [False, True])
@pytest.mark.parametrize("seed", ["12of19", "14of22"])
def test_targets_in_turn_under_one_query(seed, tables):
    """run_pass's extra workspaces run on streams of their own, from the second
    pass on with their buffers in place: nothing of a load may still be under
    way when they start."""
    targets, query = _pair(7, 1_500_000)
    sm = EngineConfig().sub_mat
    want, host = [], []
    for t in targets:
        with engine_for(sm, seed=seed, wga_chunk=20_000) as e:
            e.set_tuning(plain_streams=1)
            e.load_target(t)
            e.swap_query_ascii(query)
            want.append(e.run_pass())
            if tables:
                host.append((*e.read_tables(), sequence.encode(t)))
    with engine_for(sm, seed=seed, wga_chunk=20_000) as e:
        e.set_tuning(plain_calls=1)  # a wave a call: all four workspaces start at once
        e.swap_query_ascii(query)
        for _ in range(2):
            for k, t in enumerate(targets):
                if tables:
                    e.load_tables(*host[k])
                else:
                    e.load_target(t)
                recs, st = e.run_pass()
                assert recs.tobytes() == want[k][0].tobytes() and recs.size > 10
                assert st == want[k][1]
