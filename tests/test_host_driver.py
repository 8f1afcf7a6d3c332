"""What the host driver asks of the CUDA runtime and launches, without a GPU: the
library runs over a runtime of host memory and empty kernels (cuda_host.cpp), in
a process of its own.  Counts are all zero there; what is looked at is which
kernels a call launches, how, and on which device."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

PRELUDE = """
import ctypes, os
import numpy as np
import perft_gpu_gb300 as pg
host = ctypes.CDLL(os.environ["LD_PRELOAD"])
host.host_launches.restype = ctypes.c_char_p
launches = lambda: [l.split() for l in host.host_launches().decode().splitlines()]
pos = pg.board_from_fen("rnbqkbnr/pppppppp/8/8/8/8/PPPPPPPP/RNBQKBNR w KQkq - 0 1")
boards = lambda n: np.repeat(pg.boards_array([pos]), n)
depths = lambda n, d: np.full(n, d, np.uint8)
"""


@pytest.fixture(scope="module")
def host_run(tmp_path_factory):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        include = "/usr/local/cuda/include"
    lib = str(tmp_path_factory.mktemp("cuda_host") / "libcuda_host.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-shared", "-fPIC", "-I", include, "-o", lib,
                           os.path.join(ROOT, "tests", "cuda_host.cpp")])

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], capture_output=True, text=True, timeout=300,
                           cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT, LD_PRELOAD=lib))
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("options", ["persistent=True", "persistent=True, graph=True", "graph=True", "",
                                     "use_tt='dedup'", "slider='ks', block_size=512", "slider='byte', block_size=512"])
def test_kernels_are_set_up_again_on_another_device(host_run, options):
    """Dynamic shared memory above 48 KB is allowed for each kernel and device:
    again after the engine has moved to another one."""
    host_run("""
for device in (0, 1):
    pg.init(device=device)
    for n in (1, 300, 9000):
        pg.perft_batch(boards(n), depths(n, 3), %s)
    pg.count_moves_batch(boards(3))
    pg.generate_moves(pos)
    pg.shutdown()
    assert launches()
""" % options)


@pytest.mark.parametrize("options, threads", [("block_size=128", "128"), ("block_size=512", "512"),
                                              ("slider='byte', block_size=512", "512"), ("block_size=256", "256")])
@pytest.mark.parametrize("n", [1000, 1 << 19])
def test_leaf_runs_the_block_size_asked_for(host_run, options, threads, n):
    """Also on a level large enough for the leaf that collects its live nodes."""
    host_run("""
pg.init()
pg.perft_batch(boards(%d), depths(%d, 2), use_tt='dedup', %s)
leaves = [l[1] for l in launches() if 'k_leaf' in l[0]]
assert leaves and set(leaves) == {%r}, leaves
""" % (n, n, options, threads))


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("before", ["", "pg.perft_batch(boards(300), depths(300, 2), slider='ks', stats=pg.PgStats())"])
def test_served_waves_record_no_timing(host_run, before, persistent):
    """Whatever the call before them asked for: nobody reads a wave's times."""
    host_run("""
pg.init(slider='ks')
%s
assert bool(host.host_events()) == bool(%r)
launches()
server = pg.Server(slider='ks', persistent=%r)
assert server.wait(server.submit(pos, 2), timeout=60)[0] == 0
server.stop()
assert any('k_gather_wave' in l[0] for l in launches())
assert host.host_events() == 0
""" % (before, before, persistent))


@pytest.mark.parametrize("call", ["cli.main([fen, '4'])", "pg.perftLauncher(pos, 3)"])
def test_timed_counts_take_the_path_of_a_plain_call(host_run, call):
    """The command line and the launcher time a call; only --stats asks for the
    counters, which make it wait for every level's size and record events."""
    host_run("""
from perft_gpu_gb300 import cli
fen = 'rnbqkbnr/pppppppp/8/8/8/8/PPPPPPPP/RNBQKBNR w KQkq - 0 1'
pg.init(slider='ks')
%s
assert any('k_step' in l[0] for l in launches())
assert host.host_events() == 0
cli.main([fen, '4', '--stats', '--slider', 'ks'])
assert host.host_events() > 0
""" % call.replace("'4']", "'4', '--slider', 'ks']"))


@pytest.mark.parametrize("call", ["pg.count_moves_batch(boards(3))", "pg.count_moves_batch(boards(4170))",
                                  "pg.generate_moves(pos)", "pg.generate_boards(pos)", "pg.perft_divide(pos, 3)",
                                  "pg.perft_batch(boards(3), depths(3, 2), slider='ks')"])
def test_a_failed_call_waits_for_what_reads_its_inputs(host_run, call):
    """An error found behind a launch (here one that somebody else's call left)
    ends the call; its kernel may still run on the pinned inputs and results, which
    the next call writes."""
    host_run("""
pg.init()
launches()
host.host_error()
try:
    %s
    raise SystemExit("no error reported")
except pg.PerftError as e:
    assert e.status == 4
done = launches()
assert any(l != ["wait"] for l in done) and done[-1] == ["wait"], done
""" % call)
