"""The eigen-solve in one CTA and in a cluster of eight (k_jacobi_svd) at the
sizes where the form or a share changes: around the one-CTA limit (32), columns
per lane (64, 128), what fits the first CTA's shared memory (114), odd sizes,
CTAs without a column, the largest -- and equal eigenvalues, ordered as a
selection sort does.  Bounds as in test_gpu_small."""
import numpy as np
import pytest

from test_gpu_small import _check, _spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 34, 41, 43, 57, 64, 65, 114, 115, 128, 129, 255, 256])
def test_sizes(engine, m):
    rng = np.random.default_rng(1000 + m)
    x = rng.standard_normal((3 * m + 2, m)) * rng.uniform(0.1, 10, m)
    _check(engine, x.T @ x)


@pytest.mark.parametrize("m", [7, 32, 40, 90])
def test_equal_eigenvalues(engine, m):
    _check(engine, np.eye(m) * 3.0)
    _check(engine, _spd(np.random.default_rng(m), m, np.repeat([5.0, 2.0, 0.0], [m // 3, m // 3, m - 2 * (m // 3)])))
