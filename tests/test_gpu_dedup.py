"""The device dedup's tile and merge edges against the host entry point."""
import ctypes as C

import numpy as np
import pytest

from hspz_b200 import Engine, EngineConfig, synth
from hspz_b200 import _native as N
from hspz_b200 import engine as E
from hspz_b200.build import build
from hspz_b200.hsp import SEGMENT_PAIR

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build()


def records(n: int, kind: str) -> np.ndarray:
    rng = np.random.default_rng(n)
    a = np.zeros(n, dtype=SEGMENT_PAIR)
    if kind == "spread":  # coordinates over all 32 bits, wrapping ends, negative scores
        for f in ("ref_start", "query_start", "len"):
            a[f] = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
        a["score"] = rng.integers(-(1 << 31), 1 << 31, n)
    else:  # few diagonals, many copies and nested segments
        a["query_start"] = rng.integers(0, 3000, n)
        a["ref_start"] = a["query_start"] + rng.integers(0, 7, n).astype(np.uint32)
        a["len"] = rng.integers(0, 200, n)
        a["score"] = rng.integers(3000, 3010, n)
    return a


@pytest.mark.parametrize("kind", ["spread", "dense"])
@pytest.mark.parametrize("n", [0, 1, 2, 31, 2047, 2048, 2049, 4096, 4097, 6145, 8193, 100_001, 262_144])
def test_noalloc_dedup_at_tile_edges(n, kind):
    import torch

    recs = records(n, kind)
    want = E.dedup_and_order(recs)
    # a 4-byte aligned buffer that is not 16-byte aligned
    d_in = torch.zeros(16 * n + 4, dtype=torch.uint8, device="cuda")
    d_in[4:] = torch.from_numpy(recs.view(np.uint8).copy()).cuda()
    d_out = torch.full((16 * n + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    d_n = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    N.check(N.lib().hz_dedup_and_order_device_noalloc(
        C.c_void_p(d_in.data_ptr() + 4), n, C.c_void_p(d_out.data_ptr()), C.c_void_p(d_n.data_ptr()),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    k = int(d_n.item())
    out = d_out.cpu().numpy()
    assert k == want.size
    assert out[:16 * k].tobytes() == want.tobytes()
    assert (out[16 * k:] == 0xAB).all()


@pytest.mark.parametrize("max_hits", [40, 16711680])
def test_batched_device_dedup_equals_host_dedup(max_hits):
    """Repeat-dense blocks: copies by the thousand, in one scope and in many."""
    rng = np.random.default_rng(8)
    fam = synth.repeat_families(rng, n_fam=6, lo=300, hi=900)
    t, q = synth.repeat_genome(rng, 120_000, fam), synth.repeat_genome(rng, 60_000, fam)
    with Engine(EngineConfig(occ_cap=30, max_hits=max_hits, wga_chunk=5000)) as e:
        e.load_target(t)
        e.stage_queries([q[:25_000], q[25_000:]])
        got, st = e.run_batched()
        e.set_tuning(device_dedup=0)
        want, st_h = e.run_batched()
    assert st["raw_hsps"] > st["hsps"] > 500  # the workload has copies to take out
    assert got.tobytes() == want.tobytes() and st == st_h
