"""GPU: launch shapes saved by an earlier build (MGP_TUNE_CACHE).  They were searched against that
build's kernels and keep levels off the ones built in since, so they are not taken: the search
runs again.  What this build saved is taken without a search."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PKG = Path(__file__).resolve().parent.parent / "multigrid-poisson_b200"
PROG = """
import sys
sys.path.insert(0, sys.argv[1])
import mgp
s = mgp.Solver((33, 17, 17), 3, 1 / 32, (0,) * 6, mgp.FULLWEIGHTING, mgp.JACOBI, mgp.F64, 3, 1, 0.0)
r = s.autotune("Vcycle", 2)
print("searched" if r["untuned_ms"] > 0 else "taken", r["params"])
"""


def autotune(path):
    out = subprocess.run([sys.executable, "-c", PROG, str(PKG)], env=dict(os.environ, MGP_TUNE_CACHE=str(path)),
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    return out.stdout


def test_shapes_of_earlier_builds_are_searched_again(mgp_mod, gpu_ready, tmp_path):
    path = tmp_path / "tune.txt"
    first = autotune(path)
    assert first.startswith("searched")
    saved = path.read_text()
    assert autotune(path) == first.replace("searched", "taken")
    # an entry as earlier builds wrote it: the key without what tells the launch rules apart,
    # planes set on every level
    key = re.search(r"sm\d+x.*", saved.split()[0]).group(0)
    old = key + " " + " ".join(["3 3 3 1 0 0 0 0"] * 3) + "\n"
    path.write_text(old)
    assert autotune(path).startswith("searched")
    path.write_text(old + saved)
    assert autotune(path) == first.replace("searched", "taken")
