"""The device seed table at the edges of its sort tiles (4096 positions), of
its four-position windows and of its seed patterns, against the oracle's."""
import numpy as np
import pytest

import oracle
from hspz_b200 import EngineConfig
from hspz_b200.build import build
from tests.test_gpu_parity import engine_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build()


# 35 bases: wider than a packed window; 29 and 30: around four windows in one
WIDE = "1" + "0" * 20 + "1" + "0" * 11 + "11"
SPEC29, SPEC30 = "111" + "0" * 23 + "111", "111" + "0" * 24 + "111"


@pytest.mark.parametrize("seed,step", [("12of19", 1), ("12of19", 2), ("11011", 1), (SPEC29, 1), (SPEC30, 1), (WIDE, 1),
                                       (WIDE, 3)])
@pytest.mark.parametrize("n", [0, 17, 19, 20, 21, 39, 4096 + 18, 4096 + 19, 4097 + 19, 3 * 4096 + 37, 50_001])
def test_table_at_tile_edges(n, seed, step):
    rng = np.random.default_rng(n + step)
    alpha = np.frombuffer(b"ACGTNag&", dtype=np.uint8)
    seq = rng.choice(alpha, size=n, p=[.5, .2, .1, .1, .04, .03, .02, .01])  # skewed: buckets of many positions
    if n > 40:
        seq[n // 2:] = rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=n - n // 2)
    idx_o, pos_o = oracle.seed_table(oracle.encode(seq.tobytes()), oracle.shape(seed), step)
    with engine_for(EngineConfig().sub_mat, seed=seed, step=step) as e:
        e.load_target(seq[: n // 3])  # the second build reuses the first one's memory
        e.load_target(seq)
        idx_d, pos_d = e.read_tables()
    assert np.array_equal(idx_d, idx_o)
    assert np.array_equal(pos_d, pos_o)
