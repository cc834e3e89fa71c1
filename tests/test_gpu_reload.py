"""A query that stays while targets are loaded in turn: every pass runs on the
target loaded last, completely loaded; one that could not be loaded is no
target."""
import contextlib

import numpy as np
import pytest

from hspz_b200 import EngineConfig, sequence, synth
from hspz_b200 import _native as N
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


@contextlib.contextmanager
def device_memory_left(nbytes):
    """All of the device's free memory but nbytes is taken."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def test_a_load_or_swap_that_fails_leaves_nothing_to_run():
    rng = np.random.default_rng(3)
    targets, query = _pair(9, 600_000)
    big = synth.random_bases(rng, 30_000_000)
    sm = EngineConfig().sub_mat
    with engine_for(sm, wga_chunk=50_000) as e:
        e.load_target(targets[0])
        e.swap_query_ascii(query)
        want, st = e.run_pass()
        assert want.size > 10

        def refused():
            runs = [e.run_pass, e.run_batched, lambda: e.seed_and_filter(0, False),
                    lambda: e.generate_seeds(0, False, (0, 1000))]
            for run in runs:
                with pytest.raises(N.HzError) as ex:
                    run()
                assert ex.value.code == N.HZ_E_STATE

        # arguments that are refused leave the target that is there
        idx, pos = e.read_tables()
        with pytest.raises(N.HzError) as ex:
            e.load_tables(idx[:-1], pos, sequence.encode(targets[0]))
        assert ex.value.code == N.HZ_E_INVALID
        assert e.run_pass()[0].tobytes() == want.tobytes()
        # room for the 30 Mbp target's codes and packed copy, not for its k-mers
        with device_memory_left(160 << 20):
            with pytest.raises(N.HzError) as ex:
                e.load_target(big)
            assert ex.value.code == N.HZ_E_OOM
        refused()
        with pytest.raises(N.HzError) as ex:
            e.read_tables()
        assert ex.value.code == N.HZ_E_STATE
        e.load_target(targets[0])
        got, st2 = e.run_pass()
        assert got.tobytes() == want.tobytes() and st2 == st
        # the query store's 60 MB
        for swap in (lambda: e.swap_query_ascii(big), lambda: e.stage_queries([query, big]),
                     lambda: e.swap_query(sequence.encode(big), sequence.encode(big))):
            with device_memory_left(32 << 20):
                with pytest.raises(N.HzError) as ex:
                    swap()
                assert ex.value.code == N.HZ_E_OOM
            refused()
            e.swap_query_ascii(query)
            got, st2 = e.run_pass()
            assert got.tobytes() == want.tobytes() and st2 == st
