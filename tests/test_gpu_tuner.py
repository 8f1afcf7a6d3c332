"""The autotuner gives up part-way: it runs inside the first call that leaves
the leaf's form to it, and a level allocation of its own that fails must not
change what that call counts.  A fresh process each, since the tuner runs once."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# the tuner's own allocations: levels 0 and 1 (depth 3), 2 (depth 4), 3 (depth 5), 4 (depth 6)
CALL = """
import sys
import numpy as np
import oracle
import perft_gpu_gb300 as pg
kind, after = sys.argv[1], int(sys.argv[2])
orc = oracle.Oracle(1)
boards, depths = orc.playouts(83, 2000, 0, 60, 1, 1, 3, with_depths=True)
black = (boards["pawns"] >> np.uint64(63)) == 1
some = np.arange(300) if kind == "mixed" else np.nonzero(black == (kind == "black"))[0][:1]
boards = boards[some]
depths = depths[some] if kind == "mixed" else np.full(1, 3, np.uint8)
pg.init()
assert pg.selftest(pg.SELFTEST_FAIL_NEXT_ALLOC | after << 8) == 0
got = pg.perft_batch(boards, depths)
assert b"buffer of" in pg.load_library().pg_last_error()  # the tuner met it, not the call
want, _ = orc.perft_batch(boards, depths, 1)
assert np.array_equal(got, want), (got, want)
assert np.array_equal(pg.perft_batch(boards, depths), want)  # tuned by now
"""


@pytest.mark.parametrize("kind", ["white", "black", "mixed"])
@pytest.mark.parametrize("after", [0, 1, 3, 4])
def test_a_call_counts_right_when_its_tuning_fails(kind, after):
    import oracle
    oracle.build()
    r = subprocess.run([sys.executable, "-c", CALL, kind, str(after)], capture_output=True, text=True, timeout=300,
                       cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stdout + r.stderr
