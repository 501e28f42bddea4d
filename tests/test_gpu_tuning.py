"""Which operators of a hierarchy have their schedule timed: all of 16384
rows and more, and from 4096 rows those of more than 4 MB of entries; the
others follow size rules (the same every time)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, raptor_b200 as rb
rb.init(0)
A = rb.par_stencil_grid(rb.laplace_stencil_27pt(), [%d] * 3)
ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
ml.precision = rb.%s
ml.setup(A)
for l in range(ml.num_levels):
    print(*ml.level_info(l))
"""


# 56^3: level 1 of 14426 rows and 799,402 entries (FP64 9.6 MB, FP32 6.4 MB);
# 36^3: of 4012 rows; 40^3: of 5315 rows and 282,000 entries (3.4 MB in FP64)
@pytest.mark.parametrize("side,prec,timed", [(56, "FP64", True), (56, "FP32", True),
                                             (40, "FP64", False), (36, "FP64", False)])
def test_small_operators_of_many_entries_are_timed(tmp_path, side, prec, timed):
    env = dict(os.environ, RAPTOR_B200_TUNE_CACHE=str(tmp_path / "tune.json"))
    r = subprocess.run([sys.executable, "-c", CODE % (side, prec)], env=env, capture_output=True, text=True,
                       timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr
    n, nnz, _ = (int(w) for w in r.stdout.splitlines()[1].split())
    v = 8 if prec == "FP64" else 4
    assert n < 16384 and timed == (n >= 4096 and nnz * (4 + v) > 4 << 20), (n, nnz)
    keys = json.load(open(tmp_path / "tune.json"))
    assert ("A:%d:%d:%d" % (n, nnz, v) in keys) == timed, sorted(keys)
