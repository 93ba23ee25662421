"""The CTA-pair product's schedule, checked on the host through the kernel library's own code.

`ferrum_gemm_pair_schedule` runs the same `PairSchedule` that the kernel's three roles walk
(producer, MMA issuer, epilogue).  For every pair it lists the segments (tile, k-blocks); here
they are put together again: every (tile, k-block) unit is computed exactly once, a pair leaves
at most one partial in each of its two workspace slots, the contributors of a shared tile are
exactly the consecutive pairs the kernel's owner formulas name, the pair that holds a shared
tile's first k-blocks meets it in its last segment (the finisher's stages lie idle then), and
the tile numbering reaches every (weight tile, token tile) once.  No GPU is needed: the
library is compiled here and only its host function is called.
"""
import ctypes
import random

import pytest


@pytest.fixture(scope="module")
def schedule():
    from ferrum_b200.ops import lib as ops
    fn = ops.lib().ferrum_gemm_pair_schedule
    fn.restype = ctypes.c_int
    out = (ctypes.c_longlong * 8)()

    def segments(M, rows, K, pairs, cluster):
        segs = []
        s = 0
        while fn(ctypes.c_int(M), ctypes.c_longlong(rows), ctypes.c_int(K), ctypes.c_int(pairs), ctypes.c_int(cluster),
                 ctypes.c_int(s), out):
            segs.append(tuple(out))
            s += 1
            assert s < 100000
        return segs
    return segments


@pytest.fixture(scope="module")
def launch():
    """(tokens per tile, token tiles, pairs that run, their segments) of a launch for so many pairs."""
    from ferrum_b200.ops import lib as ops
    fn = ops.lib().ferrum_gemm_pair_launch_schedule
    out = (ctypes.c_longlong * 11)()

    def run(M, rows, K, pairs):
        args = ctypes.c_int(M), ctypes.c_longlong(rows), ctypes.c_int(K), ctypes.c_int(pairs)
        fn(*args, ctypes.c_int(0), ctypes.c_int(0), out)
        bt, tiles_t, runs = out[8:]
        segs = {}
        for c in range(runs):
            segs[c] = []
            while fn(*args, ctypes.c_int(c), ctypes.c_int(len(segs[c])), out):
                segs[c].append(tuple(out[:8]))
                assert len(segs[c]) < 100000
        return bt, tiles_t, runs, segs
    return run


def check(schedule, M, rows, K, pairs, tiles_t=None):
    nkb = (K + 63) // 64
    tiles_n, tiles_t = (rows + 255) // 256, tiles_t or (M + 255) // 256
    done = {}
    coords = {}
    sharers = {}
    n_shared_tiles = 0
    for c in range(pairs):
        slots = set()
        segs = schedule(M, rows, K, pairs, c)
        for i, (tile, kb0, kb1, n_idx, t_idx, first, last, slot) in enumerate(segs):
            assert 0 <= kb0 < kb1 <= nkb
            assert 0 <= n_idx < tiles_n and 0 <= t_idx < tiles_t
            assert coords.setdefault(tile, (n_idx, t_idx)) == (n_idx, t_idx)
            for kb in range(kb0, kb1):
                assert (tile, kb) not in done, f"unit {(tile, kb)} computed twice (pairs {done.get((tile, kb))} and {c})"
                done[(tile, kb)] = c
            if first >= 0:                                   # a tile that pairs share
                assert first <= c <= last and last > first
                assert slot in (0, 1) and slot not in slots, "two partials in one workspace slot"
                slots.add(slot)
                sharers.setdefault(tile, (first, last, []))[2].append(c)
                assert sharers[tile][:2] == (first, last)
                if c == first:
                    assert i == len(segs) - 1, "the finisher meets its tile before its last segment"
            else:
                assert (kb0, kb1) == (0, nkb)
    assert len(done) == tiles_n * tiles_t * nkb, "units left out"
    assert len(set(coords.values())) == tiles_n * tiles_t == len(coords), "tile numbering is not one-to-one"
    for tile, (first, last, cs) in sharers.items():
        assert cs == list(range(first, last + 1)), (tile, first, last, cs)
        n_shared_tiles += 1
    return n_shared_tiles


def test_prefill_shapes(schedule):
    """The products of a Llama-3.1-8B layer at 2048 tokens on 74 pairs: whole tiles only
    (the left-over tiles are too short to be worth cutting)."""
    for rows, K in ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)):
        assert check(schedule, 2048, rows, K, 74) == 0


def test_long_tiles_are_cut(schedule):
    """Few tiles of many k-blocks are shared among the pairs; one wave too many joins the cut."""
    assert check(schedule, 512, 4096, 14336, 74) > 0          # 32 tiles of 224 k-blocks on 74 pairs
    assert check(schedule, 300, 256, 8192, 6) > 0
    assert check(schedule, 515, 640, 8192, 4) > 0             # 9 tiles on 4 pairs: the last whole wave is cut too
    assert check(schedule, 257, 256, 64 * 500, 74) > 0        # two tiles, dozens of sharers each


def test_random_shapes(schedule):
    rng = random.Random(7)
    for _ in range(300):
        M = rng.randint(129, 3000)
        rows = rng.randint(1, 40) * rng.choice((64, 200, 256))
        K = rng.choice((64, 320, 4096, 8192, 14336, 20000))
        check(schedule, M, rows, K, rng.randint(1, 74))


def check_launch(launch, M, rows, K, pairs):
    from ferrum_b200.ops import lib as ops
    bt, tiles_t, runs, segs = launch(M, rows, K, pairs)
    assert 64 <= bt <= 256 and bt % 32 == 0 and (tiles_t - 1) * bt < M <= tiles_t * bt
    assert runs == min(pairs, (rows + 255) // 256 * tiles_t * ((K + 63) // 64))
    shared = check(lambda M, rows, K, pairs, c: segs[c], M, rows, K, runs, tiles_t)
    if shared:      # the shared tiles' counters, two each, are there
        n = ctypes.c_int()
        ops.lib().ferrum_gemm_tc_workspace(ctypes.c_int(M), ctypes.c_int(rows), ctypes.c_int(K), ctypes.c_int(0), ctypes.c_int(2 * pairs), ctypes.byref(n))
        assert 2 * max(tile for s in segs.values() for tile, *_, slot in s if slot >= 0) + 1 < n.value
    return bt, shared > 0


def test_launches(launch):
    """What runs: the width of the token tiles and the cut as the launch chooses them, fewer units than pairs among them."""
    rng = random.Random(11)
    seen = set()
    for i in range(700):
        M = rng.randint(65, 512) if i % 2 else rng.randint(65, 3000)
        rows = rng.randint(1, 40) * rng.choice((64, 200, 256))
        K = rng.choice((64, 320, 4096, 8192, 14336, 20000))
        seen.add(check_launch(launch, M, rows, K, rng.randint(1, 74)))
    assert {bt for bt, _ in seen} == set(range(64, 257, 32))
    assert {bt for bt, cut in seen if cut} == set(range(64, 257, 32))       # every width also with shared tiles
    check_launch(launch, 65, 200, 64, 74)                                     # one unit
    check_launch(launch, 100, 256, 64 * 30, 74)                               # fewer k-blocks than pairs


def test_launches_of_models(launch):
    """A Llama-3.1-8B layer's products at the sizes a server meets."""
    for rows, K in ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)):
        for M in (65, 80, 128, 129, 256, 300, 391, 512, 2048):
            check_launch(launch, M, rows, K, 74)
