"""Split-K routes whose count does not divide the K blocks evenly: every slice of the partial sums is
written, and the residual agrees with FP64 whatever count the route table names."""

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import numpy as np
from et_b200 import CCSD, FP64, MIXED
from et_b200.synthetic import make_system
out = {}
s = make_system(9, 90, 200, seed=3)
t = None
for prec in (FP64, MIXED):
    with CCSD(9, 90, 200, precision=prec, autotune=1) as g:
        g.set_system(s.L_mo, s.h_mo, s.eps)
        if t is None:
            rng = np.random.default_rng(1)
            t = 0.05 * rng.standard_normal(g.n_amp)
        g.set_amplitudes(t)
        g.construct_omega()
        out[prec] = g.construct_omega()
print(np.linalg.norm(out[MIXED] - out[FP64]) / np.linalg.norm(out[FP64]))
"""


def _error(tune_file):
    env = dict(os.environ, CCSD_GPU_TUNE_FILE=str(tune_file))
    r = subprocess.run([sys.executable, "-c", RUN], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return float(r.stdout.split()[-1])


@pytest.mark.parametrize("pair", [0, 100])
def test_uneven_split_counts(tmp_path, pair):
    """Routes forced to counts s with (s - 1) ceil(nkt / s) >= nkt for the K blocks nkt of the shape."""
    f = tmp_path / "routes"
    assert _error(f) < 1e-4
    lines, forced = f.read_text().split("\n"), 0
    with open(f, "w") as out:
        for line in filter(None, lines):
            key, _ = line.split()
            m, n, k = (int(x) for x in key.split("/")[-1].split("x"))
            nkt = -(-k // 64)
            uneven = [s for s in range(2, min(nkt, 64)) if (s - 1) * -(-nkt // s) >= nkt]
            route = 1
            if uneven and (not pair or m >= 256):
                route, forced = pair + uneven[-1], forced + 1
            out.write(f"{key} {route}\n")
    assert forced >= 3
    assert _error(f) < 1e-4
