"""The subspace eigensolver at the edges of its one-CTA reduction: one, two and
four rows a lane (m = 32, 64, 128 real; 32, 64 complex) and the first sizes
past them, against LAPACK: eigenvalues to 1e-12 ||A||, residuals to 1e-11
||A||, vectors orthonormal to 1e-12 up to m = 64 (the wider Gram-Schmidt
groups) and 1e-11 above, on spread, repeated and graded spectra."""

import numpy as np
import pytest

from conftest import rng
from pwgpu.lib import dense_eigh

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _matrix(g, m, cpx, kind):
    lam = np.sort(g.uniform(-10.0, 300.0, m))
    if kind == "repeated":
        lam[m // 3:m // 3 + 4] = lam[m // 3]
        lam = np.sort(lam)
    elif kind == "graded":
        lam = np.geomspace(1e-9, 100.0, m)
    a = g.standard_normal((m, m)) + (1j * g.standard_normal((m, m)) if cpx else 0.0)
    q, _ = np.linalg.qr(a)
    a = (q * lam) @ q.conj().T
    return 0.5 * (a + a.conj().T)


@pytest.mark.parametrize("kind", ["spread", "repeated", "graded"])
@pytest.mark.parametrize("cpx,m", [(False, m) for m in (4, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129)]
                         + [(True, m) for m in (4, 31, 32, 33, 63, 64, 65)])
def test_edges_of_the_one_cta_reduction(cpx, m, kind):
    g = rng(100 * m + cpx)
    a = _matrix(g, m, cpx, kind) if m > 8 else _matrix(g, m, cpx, "spread")
    for nev in (m, max(1, m // 3)):
        w, z, _ = dense_eigh(a, nev)
        ref = np.linalg.eigvalsh(a)[:nev]
        scale = np.linalg.norm(a, 2)
        assert np.max(np.abs(w - ref)) <= TOL * scale
        assert np.max(np.linalg.norm(a @ z - z * w, axis=0)) <= 10 * TOL * scale
        assert np.max(np.abs(z.conj().T @ z - np.eye(nev))) <= (TOL if m <= 64 else 10 * TOL)


@pytest.mark.parametrize("cpx", [False, True])
@pytest.mark.parametrize("m", [1, 2, 5, 33, 65])
def test_diagonal_and_extreme_scales(cpx, m):
    """Every reflector the identity, and entries near the ends of the exponent range the norms can square."""
    g = rng(m)
    for scale in (1.0, 1e140, 1e-140):
        d = np.sort(g.uniform(-1.0, 1.0, m)) * scale
        a = np.diag(d).astype(np.complex128 if cpx else np.float64)
        w, z, _ = dense_eigh(a, m)
        assert np.max(np.abs(w - d)) <= TOL * np.max(np.abs(d))
        assert np.max(np.abs(z.conj().T @ z - np.eye(m))) <= 10 * TOL
