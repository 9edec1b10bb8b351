"""The fused block steps of the eigensolver (narrow blocks) against dense diagonalisation.

Block widths at the edges of the kernels: 3 columns, 32 / 33 (four and eight column tiles), 47 / 48 complex and 64 / 65
real (the widest fused block and the first that takes the library products), and row counts from fewer than a
cluster's CTAs hold to several thousand with a remainder.  nd = bands + max(2, bands // 8).  Bars as the other
eigensolver tests: eigenvalues 1e-7 Ha; residuals below the requested 1e-7 eV; |X^H X - I| 1e-11 (Cholesky-QR passes
leave 1e-12, the Ritz rotations since then a few rounding errors each)."""

import numpy as np
import pytest

from conftest import rng
from oracle import pwdft_oracle as O
from pwgpu.context import build_system
from pwgpu.crystal import KPoint, diamond_primitive, diamond_supercell, gamma_only
from pwgpu.lib import PRECISION_FP64, PRECISION_MIXED, PwGpu, PwGpuError
from pwgpu.symmetry import SymmetryInfo

pytestmark = pytest.mark.gpu

HA = 27.211386245988


def _veff(s):
    rho_g = O.density_r_to_g(s.rho_init_r, s.dims)
    _, vxc = O.lda_xc(O.add_core(s.rho_init_r, s.rho_core_r))
    return s.v_local_g + O.hartree(rho_g, s.g_squared) + O.density_r_to_g(vxc, s.dims)


def _check(s, bands):
    veff = _veff(s)
    p = s.projectors[0]
    h = O.dense_hamiltonian(s.basis.miller, s.kinetic[0], veff, s.dims, p.b, p.d_dense())
    ref = np.linalg.eigvalsh(h)[:bands]
    with PwGpu(s) as dev:
        dev.set_veff_g(veff)
        ev, psi, _, res = dev.eigensolve(bands, tol=1e-7, max_iter=400)
    assert np.max(np.abs(ev - ref)) / HA < 1e-7
    assert res < 1e-7
    assert np.max(np.abs(psi.conj().T @ psi - np.eye(bands))) < 1e-11
    assert np.max(np.linalg.norm(h @ psi - psi * ev, axis=0)) < 1e-6


@pytest.mark.parametrize("bands", [1, 7, 29, 30, 42, 43])
def test_complex_blocks(bands, si_pp):
    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 260.0, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    _check(s, bands)


@pytest.mark.parametrize("bands", [1, 20, 29, 30, 57, 58])
def test_gamma_real_blocks(bands, si_pp):
    cr = diamond_supercell("Si", 5.431, (1, 1, 1), 0.02, rng(5))
    s = build_system(cr, {"Si": si_pp}, 190.0, gamma_only(), SymmetryInfo.identity_only())
    _check(s, bands)


@pytest.mark.parametrize("ecut,bands", [(30.0, 3), (45.0, 9), (80.0, 4)])
def test_few_plane_waves(ecut, bands, si_pp):
    """Rows for one or two CTAs only, and blocks close to the whole space."""
    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, ecut, [KPoint(np.array([0.05, 0.1, -0.2]), 1.0)])
    _check(s, bands)


@pytest.mark.parametrize("gamma_complex", [True, False])
def test_failed_step_keeps_the_bands(gamma_complex, si_pp):
    """A potential beyond the range of FP32 makes H W of the mixed form non-finite: the step fails, and the bands left
    on the device are the orthonormal ones from before it."""
    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 190.0, gamma_only(), SymmetryInfo.identity_only())
    veff = np.zeros(s.n_grid, dtype=np.complex128)
    veff[0] = 1e39
    with PwGpu(s, precision=PRECISION_MIXED, gamma_complex=gamma_complex) as dev:
        dev.set_veff_g(veff)
        with pytest.raises(PwGpuError, match="non-finite"):
            dev.eigensolve(5, tol=1e-7, max_iter=4)
        psi = dev.get_bands(5)
        assert np.max(np.abs(psi.conj().T @ psi - np.eye(5))) < 1e-11
        dev.set_veff_g(_veff(s))
        dev.set_precision(PRECISION_FP64)  # H W in FP32 does not resolve residuals below ~1e-6 of max |H| ~ 190 eV
        assert dev.eigensolve(5, tol=1e-7, max_iter=400)[3] < 1e-7


@pytest.mark.parametrize("gamma,ecut,bands", [(False, 700.0, 36), (True, 350.0, 45)])
def test_wide_blocks_of_many_rows(gamma, ecut, bands, si_pp):
    """The first steps, every band active, take the library products (block_step_gains), the later ones the fused
    launches; values, directions and columns pass from one form to the other."""
    if gamma:
        cr = diamond_supercell("Si", 5.431, (1, 1, 1), 0.02, rng(5))
        s = build_system(cr, {"Si": si_pp}, ecut, gamma_only(), SymmetryInfo.identity_only())
    else:
        s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, ecut, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    m = 3 * (bands + bands // 8)
    assert m * m * (1.0 + s.n_pw / 3000.0) > (35e3 if gamma else 20e3) > (m / 3 + 10) ** 2 * (1.0 + s.n_pw / 3000.0)
    _check(s, bands)


@pytest.mark.parametrize("gamma", [True, False])
def test_long_solves_stay_orthonormal(gamma, si_pp):
    """X is rotated, not orthonormalised again, through a solve: some 20 steps at tolerance 1e-10 eV."""
    if gamma:
        cr = diamond_supercell("Si", 5.431, (1, 1, 1), 0.02, rng(5))
        s = build_system(cr, {"Si": si_pp}, 190.0, gamma_only(), SymmetryInfo.identity_only())
    else:
        s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 520.0, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    with PwGpu(s) as dev:
        dev.set_veff_g(_veff(s))
        _, psi, its, res = dev.eigensolve(3, tol=1e-10, max_iter=800)
    assert res < 1e-10 and its >= 15
    assert np.max(np.abs(psi.conj().T @ psi - np.eye(3))) < 1e-11
