"""The two-ply leaf where its queue and its choice of form have their edges:
CTAs whose queued moves overflow a thread's column and the CTA's queue, partly
filled CTAs, and levels with many dead nodes around the size from which the
leaf collects the live ones.  Counts are exact: they equal the oracle's."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 218 legal moves, and a middlegame with checks and pins on every side
MANY = "R6R/3Q4/1Q4Q1/4Q3/2Q4Q/Q4Q2/pp1Q4/kBNN1KB1 w - - 0 1"
SHARP = "r3k2r/p1ppqpb1/bn2pnp1/3PN3/1p2P3/2N2Q1p/PPPBBPPP/R3K2R w KQkq - 0 1"


@pytest.fixture(scope="module")
def orc():
    import oracle
    oracle.build()
    return oracle.Oracle(1)


def _copies(pg, fen, n):
    return np.repeat(pg.boards_array([pg.board_from_fen(fen)]), n)


@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("slider", ["ks", "byte"])
@pytest.mark.parametrize("n", [1, 31, 513])
def test_leaf_queue_overflows_and_partial_ctas(pg, orc, block, slider, n):
    for fen in (MANY, SHARP):
        boards = _copies(pg, fen, n)
        # every third node one ply shallower, so that nodes of both depths share CTAs
        depths = np.where(np.arange(n) % 3 == 1, 1, 2).astype(np.uint8)
        want = {d: orc.perft(orc.fen(fen), d) for d in (1, 2)}
        got = pg.perft_batch(boards, depths, slider=slider, block_size=block, leaf_plies=2)
        assert (got == np.array([want[int(d)] for d in depths], dtype=np.uint64)).all()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, (1 << 19) + 1500])
def test_leaf_collects_live_nodes_of_a_sparse_level(pg, orc, n):
    """n white-to-move nodes of which every second one repeats another."""
    boards = pg.random_playouts(41, 400000, 2, 60)
    boards = boards[(boards["pawns"] >> np.uint64(63)) == 0]
    half = (n + 1) // 2
    base = boards[np.arange(half) % len(boards)]
    nodes = np.empty(n, dtype=boards.dtype)
    nodes[0::2], nodes[1::2] = base, base[:n // 2]
    got = pg.perft_batch(nodes, np.full(n, 2, np.uint8), use_tt="dedup")
    distinct, _ = orc.perft_batch(boards[:min(half, len(boards))], np.full(min(half, len(boards)), 2, np.uint8),
                                  os.cpu_count() or 1)
    want = distinct[np.arange(half) % len(boards)]
    assert np.array_equal(got[0::2], want)
    assert np.array_equal(got[1::2], want[:n // 2])


@pytest.mark.parametrize("n", [1, 257, 8191, 8192, 8193])
def test_counts_scan_and_plan_of_small_levels(pg, orc, n):
    """A first level of n white-to-move nodes, at the size from which counts,
    scan and plan are separate launches, with one chunk and with several."""
    boards = pg.random_playouts(43, 40000, 2, 60)
    boards = boards[(boards["pawns"] >> np.uint64(63)) == 0][:n]
    depths = np.full(n, 3, np.uint8)
    depths[::5] = 2
    want, _ = orc.perft_batch(boards, depths, os.cpu_count() or 1)
    assert np.array_equal(pg.perft_batch(boards, depths, slider="ks"), want)
    pg.shutdown()
    try:
        pg.init(hbm_budget_bytes=1 << 20)  # 65,536 nodes a level: several chunks
        assert np.array_equal(pg.perft_batch(boards, depths, slider="ks"), want)
        assert np.array_equal(pg.perft_batch(boards, depths, slider="ks", graph=True), want)
        assert np.array_equal(pg.perft_batch(boards, depths, slider="ks", graph=True), want)
    finally:
        pg.shutdown()
        pg.init()


@pytest.mark.parametrize("n", [4096, 4097, 30000])
@pytest.mark.parametrize("bad", ["board", "depth", "both"])
def test_batches_report_the_first_bad_root(pg, n, bad):
    """The host checks small batches, the device large ones: same answer."""
    boards = pg.random_playouts(47, n, 0, 40)
    depths = np.full(n, 1, np.uint8)
    moves = pg.count_moves_batch(boards)
    assert np.array_equal(pg.perft_batch(boards, depths), moves)
    spoilt, deep = boards.copy(), depths.copy()
    if bad != "depth":
        spoilt["kings"][n - 2] = 0
    if bad != "board":
        deep[n - 3] = 16
    for options in ({}, {"persistent": True}, {"use_tt": "dedup"}):
        with pytest.raises(pg.PerftError) as e:
            pg.perft_batch(spoilt, deep, **options)
        assert e.value.status == (3 if bad == "board" else 2)
        assert str(n - 2 if bad == "board" else n - 3) in str(e.value)
    if bad == "board":
        with pytest.raises(pg.PerftError) as e:
            pg.count_moves_batch(spoilt)
        assert e.value.status == 3 and str(n - 2) in str(e.value)
    assert np.array_equal(pg.perft_batch(boards, depths), moves)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 4095, 4096, 4097])
def test_small_calls_read_and_write_pinned_memory(pg, orc, n):
    """Calls of up to 4,096 roots leave their boards and find their counts in
    pinned memory: two calls with different roots, the counts cleared between."""
    for seed, persistent in ((53, False), (59, False), (61, True)):
        boards, depths = pg.random_playouts(seed, n, 0, 60, 1, 0, 2, with_depths=True)
        want, _ = orc.perft_batch(boards, depths, os.cpu_count() or 1)
        assert np.array_equal(pg.perft_batch(boards, depths, persistent=persistent), want)


# 224 legal moves: 294 of them have more children than the smallest level buffer
BEYOND = "Q6Q/3Q4/1Q4Q1/4Q3/2Q4Q/Q4Q2/pp1Q4/kBNN1KB1 w - - 0 1"


@pytest.mark.parametrize("n", [1, 2, 274, 300, 301])
@pytest.mark.parametrize("depth", [3, 4])
def test_levels_launched_before_their_size_is_known(pg, orc, n, depth):
    """Up to 300 roots have their first levels launched without waiting for each
    one's size; roots of every depth and both sides, and boards whose children do
    not fit (the call then waits level by level)."""
    want = {(f, d): orc.perft(orc.fen(f), d) for f in (MANY, BEYOND) for d in range(1, depth)}
    assert want[BEYOND, 1] * 294 > 1 << 16
    for fen in (MANY, BEYOND):
        deep = min(depth, 3) if n > 1 else depth
        boards, depths = _copies(pg, fen, n), np.full(n, deep, np.uint8)
        expect = np.full(n, orc.perft(orc.fen(fen), deep), np.uint64)
        if n > 250:
            depths[::50] = 2
            expect[::50] = want[fen, 2]
        assert np.array_equal(pg.perft_batch(boards, depths), expect)
    boards, depths = pg.random_playouts(61, n, 0, 60, 1, 0, depth, with_depths=True)
    expect, _ = orc.perft_batch(boards, depths, os.cpu_count() or 1)
    assert np.array_equal(pg.perft_batch(boards, depths), expect)


@pytest.mark.parametrize("n", [1, 4096, 4097, 4170, 4171])
def test_operator_calls_at_the_pinned_buffer_s_size(pg, orc, n):
    """Boards and results of up to 4,170 positions fit the pinned buffer."""
    boards = pg.random_playouts(71, n, 0, 60)
    want, _ = orc.perft_batch(boards, np.full(n, 1, np.uint8), os.cpu_count() or 1)
    assert np.array_equal(pg.count_moves_batch(boards).astype(np.uint64), want)
    pos = pg.board_of(boards[n // 2])
    assert len(pg.generate_moves(pos)) == len(pg.generate_boards(pos)) == want[n // 2]
    divided = pg.perft_divide(pos, 2)
    assert [m for m, _ in divided] == list(pg.generate_moves(pos))
    total, _ = orc.perft_batch(boards[n // 2:n // 2 + 1], np.full(1, 2, np.uint8), 1)
    assert sum(c for _, c in divided) == total[0]


@pytest.mark.parametrize("lo, hi", [(4, 4), (3, 5)])
def test_duplicates_within_and_across_depths(pg, orc, lo, hi):
    """The duplicate pass takes a node's depth into account where a level mixes
    depths: the same positions at several depths, and once more each."""
    boards = pg.random_playouts(73, 40, 4, 40)
    boards = np.concatenate([boards] * (2 * (hi - lo + 1)))
    depths = np.repeat(np.arange(lo, hi + 1, dtype=np.uint8), 80)
    want, _ = orc.perft_batch(boards, depths, os.cpu_count() or 1)
    for mode in ("dedup", True):
        pg.tt_clear()
        assert np.array_equal(pg.perft_batch(boards, depths, use_tt=mode, tt_bytes=1 << 28), want)
    pg.tt_clear()


@pytest.mark.parametrize("n", [1, 23, 24, 25])
def test_one_cta_steps_a_small_level(pg, orc, n):
    """Up to 24 roots, and the children of one, are counted and expanded by one
    CTA: its queue has more than one window on boards with many moves."""
    for fen in (MANY, SHARP):
        depth = 4 if n == 1 else 3
        got = pg.perft_batch(_copies(pg, fen, n), np.full(n, depth, np.uint8), slider="byte")
        assert np.array_equal(got, pg.perft_batch(_copies(pg, fen, n), np.full(n, depth, np.uint8), slider="ks"))
        assert (got == orc.perft(orc.fen(fen), depth)).all()


@pytest.mark.parametrize("slider", ["ks", "byte", "hybrid"])
@pytest.mark.parametrize("block", [128, 256, 512])
def test_sparse_leaf_at_every_block_size(pg, orc, slider, block):
    """A level in which most nodes repeat another, not a whole number of CTAs long."""
    boards = pg.random_playouts(97, 4000, 2, 60)
    boards = boards[(boards["pawns"] >> np.uint64(63)) == 0]
    n = (1 << 19) + 777
    which = (np.arange(n) // 4) % len(boards)
    got = pg.perft_batch(boards[which], np.full(n, 2, np.uint8), use_tt="dedup", slider=slider, block_size=block)
    want, _ = orc.perft_batch(boards, np.full(len(boards), 2, np.uint8), os.cpu_count() or 1)
    assert np.array_equal(got, want[which])
