"""What the tuner takes from a CL_TUNE_CACHE file: the entries of its own kernels
and of tables with the same symmetry, not those of an earlier library's file,
whose "pairs" named other kernels.  Each case in a process of its own (the file
is read once per process).
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CHILD = r"""
import os, sys
import numpy as np
sys.path[:0] = [sys.argv[1], os.path.join(sys.argv[2], "closures-2d_b200"), os.path.join(sys.argv[2], "oracle")]
import closures_b200 as cb
from test_gpu_newton_turned import _turned
order, Q, nx = 3, 10, 124
a = _turned(order, Q, 0.3)[0] if sys.argv[3] == "turned" else cb.Angular(order, Q, 1)
cells = (nx + 4) * (nx + 4)
m = np.zeros((cells, a.n))
m[:, 0] = 1.0
ctx = cb.Context(cb.cl_grid(nx, nx, 2, 0, 0.0, 0.0, 2.0), cb.make_options(), a, np.ones(cells), np.ones(cells), m,
                 cb.isotropic_alpha(a.n, cells))
t = ctx.tune(use_cache=True)
print("RESULT", int(t["from_cache"]), t["newton_warps"], t["newton_contraction"], t["flux_contraction"])
"""


def _tune(cache, tables="own"):
    out = subprocess.run([sys.executable, "-c", CHILD, HERE, os.path.dirname(HERE), tables], check=True, timeout=300,
                         env=dict(os.environ, CL_TUNE_CACHE=str(cache)), capture_output=True, text=True).stdout
    return [l for l in out.splitlines() if l.startswith("RESULT")][0].split()[1:]


def test_entries_of_other_kernels_are_measured_again(tmp_path):
    cache = tmp_path / "cache.txt"
    cache.write_text("n10_n228_nq100_gaunt1_mt0_prec0_opt0 4 0 1\n")
    assert _tune(cache)[0] == "0"
    key = cache.read_text().splitlines()[-1].split()[0]
    cache.write_text("%s 4 0 1\n" % key)
    assert _tune(cache) == ["1", "4", "pairs", "single"]
    # tables whose pairs are other kernels: an entry of their own
    assert _tune(cache, "turned")[0] == "0"
