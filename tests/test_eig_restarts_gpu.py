"""Restarts of the top-r eigensolver whose Krylov blocks are numerically rank
deficient: the restart is repeated in the careful form once per solve, not every time
(SPB_TRACE_EIG prints the counts of each solve)."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys; sys.path.insert(0, sys.argv[1])
import numpy as np, symprop_b200 as sp
S = np.load(sys.argv[2])
assert sp.lib().symprop_debug_set(4, int(sys.argv[4])) == 0  # SYMPROP_DEBUG_UNSAFE_PIVOTS
np.save(sys.argv[2] + ".out.npy", sp.matrix.syevd(S, S.shape[0], int(sys.argv[3])))
"""


def solve(S, r, tmp_path, unsafe=0):
    f = str(tmp_path / "S.npy")
    np.save(f, S)
    p = subprocess.run([sys.executable, "-c", CODE, ROOT, f, str(r), str(unsafe)], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SPB_TRACE_EIG": "1"})
    assert p.returncode == 0, p.stderr
    m = re.search(r"restarts=(\d+) repeated=(\d+)", p.stderr)
    assert m, p.stderr
    return int(m[1]), int(m[2]), np.load(f + ".out.npy").reshape(S.shape[0], r)


def test_no_pivot_is_ever_safe(gpu, tmp_path):
    """Injected: every restart that does not check its pivots is refused.  The first one is
    repeated, the others run in the careful form at once, and the vectors are right."""
    A = np.random.default_rng(1).standard_normal((300, 300))
    S = A @ A.T
    restarts, repeated, V = solve(S, 8, tmp_path, unsafe=1)
    assert restarts > 2 and repeated == 1
    w = np.linalg.eigvalsh(S)[-8:]
    assert np.linalg.norm(S @ V - V * w) < 1e-9 * w[-1]  # residuals to 1e-12, values to their squares


@pytest.mark.parametrize("s,rank,r", [(300, 3, 8), (1500, 5, 16)])
def test_rank_below_the_block(gpu, tmp_path, s, rank, r):
    """Exact zeros beyond a rank below r: the Krylov space closes within a restart."""
    rng = np.random.default_rng(s)
    A = np.zeros((s, rank))
    A[:40] = rng.integers(-3, 4, (40, rank))
    restarts, repeated, V = solve(A @ A.T, r, tmp_path)
    assert restarts <= 1 and repeated <= 1
    V = V[:, r - rank:]  # ascending
    Q = np.linalg.qr(A)[0]
    assert np.linalg.norm(V - Q @ (Q.T @ V)) < 1e-10  # the leading vectors span the range
