"""Matrices that are far from positive definite behind a small pivot: the entries of L would exceed every bound of
the diagonal block's fixed-point numbers.  They are refused, and what is positive definite however closely is not."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu


def _create(m):
    return cg.Likelihood(W.full_to_packed(m), None, np.zeros(len(m) * (len(m) + 1) // 2))


def _indefinite(p, b, c, scale):
    a = np.sqrt(1 - 2.0 ** -p)
    m = np.array([[1, a, b], [a, 1, c], [b, c, 1]]) * np.outer(scale, scale)
    return (m + m.T) / 2


@pytest.mark.parametrize("at", [0, 1, 59, 61, 62, 64, 100])
def test_a_small_pivot_does_not_hide_an_indefinite_matrix(at):
    """Rows at .. at + 2 of a larger identity, so that they fall into one panel of four columns, two, or two blocks.
    The smallest eigenvalues are -0.2 and below, in units of the diagonal."""
    rng = np.random.default_rng(at)
    for _ in range(40):
        scale = 10.0 ** rng.uniform(-3, 3, 3)
        m3 = _indefinite(rng.uniform(12, 36), rng.uniform(-0.5, 0.5), rng.choice([-1, 1]) * rng.uniform(0.75, 0.9), scale)
        unit = m3 / np.sqrt(np.outer(np.diag(m3), np.diag(m3)))
        assert np.linalg.eigvalsh(unit)[0] < -0.01
        m = np.eye(max(at + 3, 5))
        m[at:at + 3, at:at + 3] = m3
        with pytest.raises(cg.CGError) as e:
            _create(m).close()
        assert e.value.code == cg.CG_ERR_NOT_PD


@pytest.mark.parametrize("n", [2, 3, 7, 63, 64, 65])
def test_nearly_singular_matrices_are_accepted(n):
    """Condition numbers up to 1e12: LAPACK factors them, so does the block."""
    rng = np.random.default_rng(n)
    for _ in range(20):
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        ev = 10.0 ** np.concatenate([[0.0, -12.0], rng.uniform(-12, 0, n - 2)])
        m = (q * ev) @ q.T
        m = (m + m.T) / 2
        np.linalg.cholesky(m)
        _create(m).close()
