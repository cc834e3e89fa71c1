"""The lockstep gate's own edges against the oracle: extensions that end at
the window's last cells, in later rounds, at soft-masked, N and IUPAC bases,
at sequence ends and at the cap; score matrices with and without strand
symmetry; drops that need more than one flagged group."""
import numpy as np
import pytest

from hspz_b200 import EngineConfig, synth
from hspz_b200.build import build
from tests.test_gpu_parity import engine_for, oracle_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    build()


def sequences(seed: int):
    """A pair rich in ends: many short records' worth of N, IUPAC codes,
    lowercase and planted segments of 19..400 bases, some at the ends."""
    rng = np.random.default_rng(seed)
    t, q = synth.random_bases(rng, 40_000), synth.random_bases(rng, 30_000)
    synth.plant(rng, t, q, 120, 19, 400, 0.0, 0.25)
    q[:300] = t[-300:]
    q[-250:] = t[:250]
    for s in (t, q):
        s[rng.integers(0, s.size, 60)] = ord("N")
        s[rng.integers(0, s.size, 60)] = ord("R")
        for a in rng.integers(0, s.size - 60, 40).tolist():
            s[a:a + int(rng.integers(1, 60))] |= 0x20
        s[rng.integers(0, s.size, 6)] = ord("&")
    return t, q


def matrix(kind: str, xdrop: int):
    m = EngineConfig().sub_mat if kind != "ambiguous" else None
    if m is None:
        from hspz_b200 import build_sub_mat
        return build_sub_mat("n", xdrop)
    m = list(m)
    if kind == "wide":  # a close-species score set: mismatches beyond a byte
        rows = [[90, -330, -236, -356], [-330, 100, -318, -236], [-236, -318, 100, -330], [-356, -236, -330, 90]]
        for r in range(4):
            for c in range(4):
                m[r * 8 + c] = rows[r][c]
    if kind == "widest":  # the largest cost the lockstep gate takes
        for r in range(4):
            for c in range(4):
                m[r * 8 + c] = 130 if r == c else -585
    if kind == "general":  # no two of the sixteen ACGT scores are tied by strand
        rng = np.random.default_rng(5)
        for r in range(4):
            for c in range(4):
                m[r * 8 + c] = int(rng.integers(60, 127)) if r == c else -int(rng.integers(20, 127))
    return m


@pytest.mark.parametrize("kind,xdrop,cap,sparse", [
    ("default", 910, 128, 0), ("default", 910, 128, 1), ("default", 910, 40, 0), ("default", 910, 56, 1),
    ("default", 910, 96, 0), ("default", 910, 8, 0), ("default", 910, 65528, 0), ("default", 120, 128, 0),
    ("default", 0, 128, 0), ("default", 9000, 1024, 1), ("default", 20000, 256, 0),
    ("general", 910, 128, 0), ("general", 910, 104, 1), ("general", 150, 128, 0), ("ambiguous", 910, 128, 0),
    ("wide", 910, 128, 0), ("wide", 910, 128, 1), ("wide", 910, 8, 0), ("wide", 300, 104, 0), ("wide", 20000, 1024, 1),
    ("widest", 910, 128, 0), ("widest", 25000, 512, 0), ("widest", 32637, 256, 1),
    ("ambiguous", 910, 4096, 1)])
def test_gate_edges_match_the_oracle(kind, xdrop, cap, sparse):
    t, q = sequences(xdrop + cap)
    sm = matrix(kind, xdrop)
    hspthresh = 3000 if xdrop >= 500 else 1500
    want, st_o = oracle_run(t, q, sm, xdrop=xdrop, hspthresh=hspthresh)
    with engine_for(sm, xdrop=xdrop, hspthresh=hspthresh) as e:
        e.set_tuning(gate_cap=cap, gate_sparse=sparse)
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
    assert want.size > 20
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


@pytest.mark.parametrize("seed,occ_cap,transitions", [
    ("12of19", 0, True), ("12of19", 2, True), ("12of19", 0, False), ("14of22", 1, True), ("1111", 200, True),
    ("1" * 8 + "0" + "1" * 7, 0, True)])  # 15 care positions: no per-k-mer tables
def test_sparse_setup_skips_seeds_without_hits(seed, occ_cap, transitions):
    t, q = sequences(31)
    if seed == "1111":
        t, q = t[:3000], q[:2000]
    sm = EngineConfig().sub_mat
    want, st_o = oracle_run(t, q, sm, seed=seed, occ_cap=occ_cap, transitions=transitions)
    with engine_for(sm, seed=seed, occ_cap=occ_cap, transitions=transitions) as e:
        e.set_tuning(gate_sparse=1)
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


@pytest.mark.parametrize("n", [19, 20, 40, 57, 95, 96, 97, 130])
def test_short_sequences_match_the_oracle(n):
    """Targets and queries around a window long: windows reach past both ends."""
    rng = np.random.default_rng(n)
    t = synth.random_bases(rng, n)
    q = np.concatenate([t, synth.random_bases(rng, 40), t])
    sm = EngineConfig().sub_mat
    want, st_o = oracle_run(t, q, sm, hspthresh=1000)
    with engine_for(sm, hspthresh=1000) as e:
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


@pytest.mark.parametrize("period", [1, 5, 33])
@pytest.mark.parametrize("copies", [1, 40])
def test_match_counts_of_every_segment_length(period, copies):
    """Planted segments of 40..700 cells, N and soft-masked bases `period` or
    more apart among them: the entropy's match counts at the ends of 32-base
    words and of 256-base steps, with few candidates and with several a warp."""
    rng = np.random.default_rng(period)
    t, q = [], []
    for n in list(range(40, 100)) + list(range(250, 262)) + [287, 288, 289, 511, 512, 513, 545, 700]:
        seg = synth.random_bases(rng, n)
        seg = np.where(rng.random(n) < 0.6, np.uint8(ord("A")), seg) if n % 3 else seg  # low entropy
        other = seg.copy()
        other[rng.integers(0, n, max(1, n // 30))] = ord("C")
        for at in rng.integers(0, n, n // (16 * period)).tolist():
            other[at] = seg[at] = ord("N") if at % 2 else seg[at] | 0x20
        pad = synth.random_bases(rng, 60)
        t += [seg, pad]
        q += [other, pad[::-1]]
    t, q = np.concatenate(t), np.concatenate(q * copies)
    sm = EngineConfig().sub_mat
    want, st_o = oracle_run(t, q, sm, hspthresh=1500)
    with engine_for(sm, hspthresh=1500) as e:
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
    assert want.size > 50
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("xdrop,cap,sparse,seed", [(910, 128, 0, "12of19"), (910, 56, 1, "12of19"), (0, 128, 0, "12of19"),
                                                   (20000, 256, 1, "12of19"), (910, 8, 0, "1111")])
def test_scores_of_the_whole_signed_byte(xdrop, cap, sparse, seed, alike):
    """-128 and 127 beside strands that score differently (and alike): the
    lockstep gate and the candidates' kernel take them, by half warps and
    (the short seed's candidates, more than 32768) by lanes."""
    t, q = sequences(xdrop + cap)
    if seed == "1111":
        t, q = t[:3000], q[:3000]
    m = matrix("default", xdrop)
    m[0 * 8 + 3], m[3 * 8 + 0], m[2 * 8 + 2] = -128, -128, 127  # A-T, T-A and G-G
    if alike:
        m[1 * 8 + 1] = 127  # C-C
    else:
        m[0 * 8 + 1], m[2 * 8 + 0] = -127, -128  # A-C and G-A, but not T-G and C-T
    hspthresh = 3000 if xdrop >= 500 else 1500
    want, st_o = oracle_run(t, q, m, xdrop=xdrop, hspthresh=hspthresh, seed=seed)
    with engine_for(m, xdrop=xdrop, hspthresh=hspthresh, seed=seed) as e:
        e.set_tuning(gate_cap=cap, gate_sparse=sparse)
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
        e.set_profiling(True)
        e.run_pass()
        assert "long" in e.profile()  # it follows the lockstep gate only
    assert want.size > 0
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


def test_exact_seeds_keep_no_live_mask():
    """An engine for exact seeds holds no 16-bit word per k-mer (0.5 GB for 14
    care positions), and seeds with transitions still run on it."""
    import torch

    t, q = sequences(31)
    sm = EngineConfig().sub_mat
    want, _ = oracle_run(t, q, sm, seed="14of22")
    held, got = [], []
    with engine_for(sm) as e:  # the library's own memory is in place
        e.load_target(t)
        e.swap_query_ascii(q)
        e.run_pass()
    for transitions in (True, False):
        free = torch.cuda.mem_get_info()[0]
        with engine_for(sm, seed="14of22", transitions=transitions) as e:
            e.set_tuning(gate_sparse=1)
            e.load_target(t)
            held.append(free - torch.cuda.mem_get_info()[0])
            e.swap_query_ascii(q)
            e.generate_seeds(0, False, (0, q.size - e.seed_size + 1), transitions=True)
            got.append(e.seed_and_filter(0, False))
    assert held[0] - held[1] >= 2 * 4 ** 14 - (8 << 20)
    assert got[0][0].size > 10 and want.size > 10
    assert got[0][0].tobytes() == got[1][0].tobytes() and got[0][1] == got[1][1]


@pytest.mark.parametrize("seed", ["1111", "12of19"])
def test_special_base_at_a_rounds_last_cell(seed):
    """An extension that goes on past a soft-masked base: at the last cell of a
    48-cell round, where it packs as an A and would match, while the maximum
    lies in an earlier group of the round (the eight cells before it fall by 26
    from their best).  Anchors lie at every distance from it, both ways; the
    short seed's candidates are more than 32768."""
    rng = np.random.default_rng(6)
    t, q = synth.random_bases(rng, 3000), synth.random_bases(rng, 3000)
    for i in range(10):
        at = 100 + 280 * i
        body = synth.random_bases(rng, 110)
        # outward from the body: A-T, A-A, A-G, A-C, A-A, A-G, A-A, a-A, three matches
        tail_t, tail_q = np.frombuffer(b"AAAAAAAaCCC", np.uint8), np.frombuffer(b"TAGCAGAACCC", np.uint8)
        t[at:at + 132] = np.concatenate([tail_t[::-1], body, tail_t])
        q[at + 3:at + 135] = np.concatenate([tail_q[::-1], body, tail_q])
    sm = EngineConfig().sub_mat
    want, st_o = oracle_run(t, q, sm, xdrop=3000, seed=seed)
    with engine_for(sm, xdrop=3000, seed=seed) as e:
        e.set_tuning(gate_cap=8)
        e.load_target(t)
        e.swap_query_ascii(q)
        got, st = e.run_pass()
    assert want.size >= 10
    assert got.tobytes() == want.tobytes()
    for k in ("hits", "raw_hsps", "hsps", "cells"):
        assert st[k] == st_o[k], k


def test_many_candidates_of_a_score_of_128_below_zero():
    """-128 is no signed byte's cost, and the gate takes strands that score alike
    with 16-bit ones; the candidates still go by lanes, not half a warp each
    (six times as long here), and match those of half warps."""
    rng = np.random.default_rng(12)
    t, q = synth.random_bases(rng, 1_000_000), synth.random_bases(rng, 1_000_000)
    synth.plant(rng, t, q, 40, 200, 2000, 0.1, 0.3)
    ms = []
    for score in (-127, -128):
        m = list(EngineConfig().sub_mat)
        m[0 * 8 + 3] = m[3 * 8 + 0] = score
        got = []
        with engine_for(m) as e:
            e.load_target(t)
            e.swap_query_ascii(q)
            for cap in (8, 128):  # every hit a candidate, few of them
                e.set_tuning(gate_cap=cap)
                got.append(e.run_pass())
            e.set_tuning(gate_cap=8, plain_streams=1)
            e.run_pass()
            for _ in range(5):
                e.set_profiling(True)
                e.profile_reset()
                e.run_pass()
                ms.append(e.profile()["long"][0])
                e.set_profiling(False)
        assert got[0][0].size >= 40 and got[0][0].tobytes() == got[1][0].tobytes() and got[0][1] == got[1][1]
    assert min(ms[5:]) < 2 * min(ms[:5])
