"""Batched plain realms (amca_batch_*) against the unmodified reference.

A batch runs many independent realms in one cooperative launch, teams of
blocks taking realms from a queue. Every realm's fields must be bit-exact to
its own np=1 reference run, whatever the team size and queue order:
  * the small golden decks of cases.py (digests in plain_golden.json), as
    one batch, at several team sizes, and again after the autotuner;
  * the 64 instances of the batched workload at full size (edges 32..128),
    against batched_64_golden.json made by make_golden.py --batched.
"""
import hashlib
import json
import os
import sys
import threading
import time

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLD = os.path.join(ROOT, "tests", "golden")
sys.path.insert(0, GOLD)
import cases  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = json.load(open(os.path.join(GOLD, "plain_golden.json")))


def sha(a):
    return hashlib.sha256(np.ascontiguousarray(a, dtype="<i4").tobytes()).hexdigest()


@pytest.fixture(scope="module")
def amca():
    import amca3d_gb300

    amca3d_gb300.load_library()
    return amca3d_gb300


def open_realms(amca, decks_):
    realms = []
    for c in decks_:
        r = amca.CellularAutomataRealm(c.to_yaml(), seed=c.seed)
        r.initialize()
        realms.append(r)
    return realms


def check_golden(realms, decks_, golden):
    bad = []
    for r, c in zip(realms, decks_):
        g = golden[c.name]
        st = r.stats()
        if st["step"] != g["steps"] or sha(r.field("orientation_id")) != g["orient_sha256"] \
                or sha(r.field("grain_id")) != g["grain_sha256"]:
            bad.append(c.name)
    return bad


@pytest.fixture(scope="module")
def small_batch(amca):
    decks_ = cases.small_cases()
    realms = open_realms(amca, decks_)
    yield decks_, realms
    for r in realms:
        r.close()


@pytest.mark.parametrize("team", [1, 3, 8, 32])
def test_batch_of_small_decks_matches_reference(amca, small_batch, team):
    decks_, realms = small_batch
    with amca.Batch(realms, team_size=team) as b:
        b.run()
        assert check_golden(realms, decks_, GOLDEN) == []
        st = b.stats()
        assert st["team_size"] == team and st["realms"] == len(realms) and st["runs"] == 1
        assert st["cell_updates"] == sum(r.stats()["step"] * c.n_interior for r, c in zip(realms, decks_))
        # a second run starts again from the initial state
        b.run()
        assert check_golden(realms, decks_, GOLDEN) == []


def test_batch_reads_like_single_runs(amca, small_batch):
    """After a batch run each handle's stats and fields are those of
    amca_reset + amca_run on that handle alone."""
    decks_, realms = small_batch
    with amca.Batch(realms, team_size=4) as b:
        b.run()
        got = [(r.stats(), r.field("orientation_id"), r.field("site_undercooling")) for r in realms]
    keys = ("step", "time", "dt", "liquid_cells", "grains", "orientations", "done", "captures", "nucleations")
    for r, (st, o, s) in zip(realms, got):
        r.reset()
        r.run()
        ref = r.stats()
        assert {k: st[k] for k in keys} == {k: ref[k] for k in keys}
        assert np.array_equal(o, r.field("orientation_id"))
        assert np.array_equal(s, r.field("site_undercooling"))


@pytest.mark.parametrize("layout", [((1, 4, 16), (5, 3, 2)), ((2, 64), (4, 1)), ((3,), (1,))])
def test_batch_mixed_layouts_match_reference(amca, small_batch, layout):
    """Teams of several sizes in one launch (realm r in class r mod k), and a
    single team that runs every realm in turn."""
    decks_, realms = small_batch
    sizes, teams = layout
    with amca.Batch(realms) as b:
        b.set_layout(sizes, teams, [r % len(sizes) for r in range(len(realms))])
        st = b.stats()
        assert st["grid_blocks"] == sum(s * t for s, t in zip(sizes, teams)) and st["n_classes"] == len(sizes)
        b.run()
        assert check_golden(realms, decks_, GOLDEN) == []


def test_batch_autotune_keeps_results(amca, small_batch):
    decks_, realms = small_batch
    with amca.Batch(realms) as b:
        t = b.tune(repeats=1)
        st = b.stats()
        assert t == st["team_size"] and len(st["tuned"]) >= 5 and (t == 0 or t in st["tuned"])
        assert st["mixed_ms"] > 0 or t != 0
        assert st["graph"] == 1, "the batched run is not replayed as a CUDA graph"
        b.run()
        assert check_golden(realms, decks_, GOLDEN) == []
        ts, tn, rc, qo = b.layout()
        assert sorted(qo) == list(range(len(realms))) and int((ts * tn).sum()) == b.stats()["grid_blocks"]
    # the tuned layout set on another batch of the same realms
    with amca.Batch(realms) as b2:
        b2.set_layout(ts, tn, rc, qo)
        assert [list(x) for x in b2.layout()] == [list(x) for x in (ts, tn, rc, qo)]
        b2.run()
        assert check_golden(realms, decks_, GOLDEN) == []


def test_batch_rejects_bad_handles(amca, small_batch):
    decks_, realms = small_batch
    with pytest.raises(amca.AmcaError, match="appears twice"):
        amca.Batch([realms[0], realms[1], realms[0]])
    with pytest.raises(amca.AmcaError, match="team size"):
        amca.Batch(realms[:2], team_size=100000)
    with amca.Batch(realms[:2]) as b:
        with pytest.raises(amca.AmcaError, match="more blocks"):
            b.set_layout([64], [100], [0, 0])
        with pytest.raises(amca.AmcaError, match="out of range"):
            b.set_layout([4], [2], [0, 1])
        with pytest.raises(amca.AmcaError, match="permutation"):
            b.set_layout([4], [2], [0, 0], [1, 1])


def test_batched_64_full_size_matches_reference(amca):
    """The batched workload as measured: 64 instances, edges 32..128 (about
    44M cells), one tuned, graph-replayed launch; every instance bit-exact to
    its own reference run."""
    from amca3d_gb300 import decks

    golden = json.load(open(os.path.join(GOLD, "batched_64_golden.json")))
    decks_ = decks.config_batched_64()
    realms = open_realms(amca, decks_)
    try:
        with amca.Batch(realms) as b:
            b.tune(repeats=1)
            b.run()
            assert check_golden(realms, decks_, golden) == []
            # a mixed layout: the 8 largest realms on teams of 32, the rest on 2
            big = set(np.argsort([-c.n_interior for c in decks_])[:8])
            b.set_layout([32, 2], [8, 100], [0 if r in big else 1 for r in range(len(decks_))])
            b.run()
            assert check_golden(realms, decks_, golden) == []
    finally:
        for r in realms:
            r.close()


@pytest.mark.parametrize("edge,team,count", [
    (58, 8, 3),    # 24,389 cells a block: 512 threads
    (57, 8, 3),    # 23,149: 256
    (92, 8, 2),    # 97,336: 1,024
    (46, 1, 5),    # a block of its own per realm: 1,024
    (60, 3, 120),  # 360 blocks: too many for wider ones
])
def test_batch_block_widths_give_the_same_fields(amca, edge, team, count):
    """The widths a launch's blocks can have, at the edges of the rule that picks them: every realm's fields and steps
    equal its own run's."""
    case = cases._mixed("wide", (edge, edge - 1, edge + 1), 3, 40, 200, t_dot=-200.0)
    realms = [amca.CellularAutomataRealm(case.to_yaml(), seed=3 + k % 3) for k in range(count)]
    for r in realms:
        r.initialize()
    want = []
    for r in realms[:3]:
        r.run()
        want.append((r.field("grain_id"), r.field("orientation_id"), r.stats()["step"]))
    with amca.Batch(realms, team_size=team) as b:
        b.run()
        for k in (0, 1, 2, count - 1):
            if k < count:
                g, o, n = want[k % 3] if k % 3 < len(want) else want[0]
                assert np.array_equal(realms[k].field("grain_id"), g)
                assert np.array_equal(realms[k].field("orientation_id"), o) and realms[k].stats()["step"] == n
    for r in realms:
        r.close()


@pytest.mark.parametrize("cells,team,count,width", [
    ((26, 13, 71), 1, 3, 256),    # 23,998 cells a block: below the first line
    ((30, 32, 25), 1, 3, 512),    # 24,000: on it
    ((29, 10, 331), 1, 3, 512),   # 95,990
    ((40, 48, 50), 1, 3, 1024),   # 96,000
    ((58, 57, 59), 8, 3, 512),    # 24,381 of a block of a team
    ((57, 56, 58), 8, 3, 256),    # 23,142
    ((92, 91, 93), 8, 2, 1024),   # 97,324
    ((60, 59, 61), 3, 120, 256),  # 360 blocks: too many for wider ones
])
def test_batch_launch_takes_the_width_of_its_rule(amca, cells, team, count, width):
    """The widths of blocks on both sides of each line of the rule, as the launch has them, and the fields of its first
    and last realm against their own runs."""
    case = cases._mixed("width", cells, 3, 40, 200, t_dot=-200.0)
    realms = [amca.CellularAutomataRealm(case.to_yaml(), seed=3 + k % 3) for k in range(count)]
    for r in realms:
        r.initialize()
    with amca.Batch(realms, team_size=team) as b:
        assert b.block_threads() == width
        b.run()
        assert b.block_threads() == width
        got = [(realms[k].field("grain_id"), realms[k].stats()["step"]) for k in (0, count - 1)]
        # the width follows the layout
        b.set_layout([64], [1], [0] * count)
        assert b.block_threads() == (512 if np.prod(cells) // 64 >= 24000 else 256)
    for k, (grain, step) in zip((0, count - 1), got):
        realms[k].reset()
        realms[k].run()
        assert np.array_equal(realms[k].field("grain_id"), grain) and realms[k].stats()["step"] == step
    for r in realms:
        r.close()


@pytest.mark.parametrize("cells", [(30, 32, 25), (40, 48, 50)])
def test_batch_of_wide_blocks_leaves_room_for_other_threads(amca, cells):
    """On both sides of the launch that would take nearly all of the SMs' registers: the width gives way before it does,
    and a small realm's grain field comes while the batch runs (it waited for the batch's first teams to end)."""
    case = cases._mixed("room", cells, 3, 40, 60, t_dot=-20.0)
    small = amca.CellularAutomataRealm(cases._mixed("small", (40, 40, 40), 3, 40, 60).to_yaml(), seed=3)
    small.initialize()
    small.run()
    out = small.field("grain_id")
    realms = [amca.CellularAutomataRealm(case.to_yaml(), seed=3 + k % 3) for k in range(3)]
    for r in realms:
        r.initialize()
    wide = 1024 if np.prod(cells) >= 96000 else 512
    with amca.Batch(realms, team_size=1) as b:
        assert b.block_threads() == wide
        most = 15 * (b.stats()["max_blocks"] * 256 // wide) // 16  # (512 and 1,024 threads: as many registers a thread)
    for r in realms:
        r.close()
    realms = []
    for count, width in ((most, wide), (most + 1, wide // 2)):
        while len(realms) < count:
            realms.append(amca.CellularAutomataRealm(case.to_yaml(), seed=3 + len(realms) % 3))
            realms[-1].initialize()
        with amca.Batch(realms, team_size=1) as b:
            assert b.stats()["grid_blocks"] == count and b.block_threads() == width
            b.run()
            run, wait = [], []
            for _ in range(7):
                t0 = time.perf_counter()
                th = threading.Thread(target=b.run)
                th.start()
                time.sleep(0.003)
                t1 = time.perf_counter()
                small.field("grain_id", out=out)
                wait.append(time.perf_counter() - t1)
                th.join()
                run.append(time.perf_counter() - t0)
        assert np.median(wait) < 0.1 * np.median(run), (count, wait, run)
    for r in realms + [small]:
        r.close()
