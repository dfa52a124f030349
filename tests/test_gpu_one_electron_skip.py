"""What the one-electron kernels leave out of S, T and V, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_kernel_edges import _cgfs, _table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha,beta", [(1500.0, 1500.0), (4000.0, 30.0), (30.0, 4000.0), (1e5, 2e4)])
@pytest.mark.parametrize("l", [0, 1, 2])
def test_skipped_pairs_stay_below_the_limit(cuda, l, alpha, beta):
    """Uncontracted pairs whose product Gaussian exp(-mu R^2) goes through the limit, where the kinetic energy is
    mu (2 mu R^2 - 3) times the overlap: nothing of more than 1e-17 (times 3, the largest component factor) is left
    out.  Added to that the rounding of sums that cancel to a hundredth at worst: 1e-12 of the shells' largest."""
    from segfault_py_gb300.fock import FockBuilder
    mu = alpha * beta / (alpha + beta)
    x = np.sqrt(np.arange(20.0, 60.0, 0.5) / mu)   # mu R^2 from 20 to 60
    n = len(x) + 1
    table = _table([l] * n, [1] * n, 1, 1.0)
    table["exps"][:], table["exps"][0], table["coefs"][:] = beta, alpha, 1.0
    table["center"][:] = 0.0
    direction = np.array([0.6, 0.64, 0.48])
    table["center"][1:] = x[:, None] * direction
    xyz, Z = np.array([[0.1, -0.2, 0.3]]), np.array([1.0])
    fb = FockBuilder(table, device=cuda)
    got = [m.cpu().numpy() for m in fb.one_electron(xyz, Z)]
    fb.close()
    nc = (l + 1) * (l + 2) // 2
    for name, a, b in zip("STV", got, O.one_electron(_cgfs(table), xyz, Z)):
        a, b = (m[:nc, nc:].reshape(nc, n - 1, nc) for m in (a, b))   # the first shell with the others
        excess = np.abs(a - b) - 1e-12 * np.abs(b).max(axis=(0, 2), keepdims=True)
        assert excess.max() <= 3e-17, (name, excess.max())
