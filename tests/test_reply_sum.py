"""The leaf's set-wise count of the last two plies (pg_reply.cuh), built for
the host: for every board the replies to the plain moves, summed in sets, plus
those to the remaining moves, made one by one, must equal all moves made one
by one (the general path), and on legal positions the oracle's perft(2).
The boards cover what the split decides on: playouts (checks, pins, castling,
promotions, en passant), crowded and empty arbitrary boards of every piece
mix, kings at home with every set of castling rights, and boards on which the
side not to move is already in check (no move is plain there)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, golden_npz

BOARD_DTYPE = np.dtype([(k, "<u8") for k in ("white", "pawns", "knights", "bishop_queens", "rook_queens", "kings")])


@pytest.fixture(scope="module")
def both_ways(tmp_path_factory):
    csrc = os.path.join(ROOT, "perft_gpu_gb300", "csrc")
    lib = str(tmp_path_factory.mktemp("reply") / "libreply.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC", "-I", csrc, "-o", lib,
                           os.path.join(ROOT, "tests", "reply_host.cpp"), os.path.join(csrc, "pg_tables.cpp")])
    fn = ctypes.CDLL(lib).reply_both_ways

    def call(boards):
        boards = np.ascontiguousarray(boards, dtype=BOARD_DTYPE)
        n = len(boards)
        split, made = np.zeros(n, np.uint64), np.zeros(n, np.uint64)
        moves, queued = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
        assert fn(*(ctypes.c_void_p(a.ctypes.data) if i != 1 else ctypes.c_uint32(n)
                    for i, a in enumerate((boards, boards, split, made, moves, queued)))) == 0
        return split, made, moves, queued
    return call


def _walk_boards():
    """The walk positions and the workload positions of the fixtures."""
    words = [golden_npz("walk.npz")["boards"], golden_npz("config3.npz")["boards"]]
    return np.ascontiguousarray(np.concatenate(words)).view(BOARD_DTYPE).reshape(-1)


def _arbitrary(seed, n, home):
    """n valid boards of 2..40 pieces of any kind and colour; kings anywhere or at home."""
    r = np.random.RandomState(seed)
    out = np.zeros(n, dtype=BOARD_DTYPE)
    for i in range(n):
        squares = r.permutation(64)
        if home:
            squares = np.concatenate(([4, 60], squares[(squares != 4) & (squares != 60)]))
        w, p, k = 1 << int(squares[0]), 0, (1 << int(squares[0])) | (1 << int(squares[1]))
        sets = {"knights": 0, "bishop_queens": 0, "rook_queens": 0}
        pawns_only = r.rand() < 0.3
        for q in squares[2:2 + r.randint(0, 39)]:
            bit = 1 << int(q)
            kind = 0 if pawns_only and r.rand() < 0.7 else r.randint(0, 6)
            if kind in (0, 5) and 8 <= q < 56:
                p |= bit
            elif kind in (0, 1, 5):
                sets["knights"] |= bit
            else:
                if kind != 3:
                    sets["bishop_queens"] |= bit
                if kind != 2:
                    sets["rook_queens"] |= bit
            if r.rand() < 0.5:
                w |= bit
        p |= int(r.randint(0, 16)) | (int(r.randint(0, 9)) << 4 if r.rand() < 0.3 else 0) | (int(r.randint(0, 2)) << 63)
        out[i] = (w, p, sets["knights"], sets["bishop_queens"], sets["rook_queens"], k)
    return out


def test_legal_positions_match_every_move_made_and_the_oracle(both_ways, oracle):
    boards = np.concatenate([_walk_boards(), oracle.playouts(31, 20000, 0, 150)])
    split, made, moves, queued = both_ways(boards)
    assert np.array_equal(split, made)
    want, _ = oracle.perft_batch(boards, np.full(len(boards), 2, np.uint8), os.cpu_count() or 1)
    assert np.array_equal(split, want)
    assert queued.sum() < 0.5 * moves.sum()  # most moves are counted in sets


@pytest.mark.parametrize("home", [False, True])
def test_arbitrary_boards_match_every_move_made(both_ways, home):
    boards = _arbitrary(5 + home, 15000, home)
    split, made, moves, queued = both_ways(boards)
    bad = np.nonzero(split != made)[0]
    assert len(bad) == 0, (len(bad), boards[bad[0]])
    assert (queued <= moves).all()
