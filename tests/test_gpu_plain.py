"""How a plain pass's calls share waves changes no record and no count."""
import numpy as np
import pytest

from hspz_b200 import EngineConfig, synth
from hspz_b200.build import build
from tests.test_gpu_parity import engine_for, oracle_run
from tests.test_gpu_reload import device_memory_left

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build()


@pytest.mark.parametrize("kw", [dict(wga_chunk=7_000), dict(wga_chunk=9_000, max_hits=300, interval=50_000),
                                dict(wga_chunk=5_000, strand="minus", transitions=False)])
def test_calls_per_wave_and_streams(kw):
    t, q = synth.config1(seed=5, scale=0.12)
    sm = EngineConfig().sub_mat
    okw = {**kw, **({"strand": 2} if "strand" in kw else {})}
    want, st_o = oracle_run(t, q, sm, **okw)
    with engine_for(sm, **kw) as e:
        e.load_target(t)
        e.swap_query_ascii(q)
        runs = []
        # the last setting splits every wave of several calls: too many hits
        for calls, streams, cap in ((0, 4, 1 << 33), (1, 1, 1 << 33), (1, 4, 1 << 33), (3, 2, 1 << 33),
                                    (4, 4, 1 << 33), (1000, 1, 1 << 33), (1000, 4, 1 << 20)):
            e.set_tuning(plain_calls=calls, plain_streams=streams, wave_hits_cap=cap)
            got, st = e.run_pass()
            runs.append((got.tobytes(), st))
    assert want.size > 20
    for got, st in runs:
        assert got == want.tobytes()
        assert st == runs[0][1]
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert runs[0][1][k] == st_o[k], k


@pytest.mark.parametrize("streams,calls,left", [(1, 80, 40 << 20), (4, 20, 12 << 20)])
def test_waves_that_do_not_fit_run_call_by_call(streams, calls, left):
    """A wave of several calls needs 24 bytes a position, 96 MB and 24 MB here;
    where that is not to be had, its calls still fit one by one."""
    rng = np.random.default_rng(2)
    t, q = synth.random_bases(rng, 1_000_000), synth.random_bases(rng, 2_000_000)
    synth.plant(rng, t, q, 100, 200, 3000, 0.05, 0.3)
    with engine_for(EngineConfig().sub_mat, wga_chunk=50_000) as e:
        e.load_target(t)
        e.swap_query_ascii(q)
        e.set_tuning(plain_streams=streams, plain_calls=1)
        want, st = e.run_pass()
        e.set_tuning(plain_calls=calls)
        with device_memory_left(left):
            got, st2 = e.run_pass()
        assert want.size > 100
        assert got.tobytes() == want.tobytes() and st2 == st
        got, st2 = e.run_pass()
        assert got.tobytes() == want.tobytes() and st2 == st
