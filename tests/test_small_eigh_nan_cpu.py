"""The small eigensolver of the Krylov cycles on matrices with NaN entries: a comparison that is not an
order sends std::sort out of its range, so NaN eigenvalues come last. In a child process, as what
is tested for could end it."""
import subprocess
import sys

import pytest

CHILD = """
import sys
import numpy as np
import mps_gb300 as mg
n = int(sys.argv[1])
for seed in range(40):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal(n)
    bad = rng.random(n) < 0.4
    d[bad] = np.nan
    w, v = mg.small_eigh(np.diag(d))
    good = np.sort(d[~bad])
    assert np.array_equal(w[:len(good)], good), (w, good)
    assert np.isnan(w[len(good):]).all()
    assert np.array_equal(np.sort(np.abs(v).argmax(0)), np.arange(n))
    A = rng.standard_normal((n, n))
    A[0, n - 1] = A[n - 1, 0] = np.nan
    mg.small_eigh(A + A.T)
print("ok")
"""


@pytest.mark.parametrize("n", [2, 5, 16, 17, 32])
def test_nan_eigenvalues_come_last(n):
    r = subprocess.run([sys.executable, "-c", CHILD, str(n)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-800:]
