"""The two-stage local pipeline of H|psi> against numpy's FFT, over every grid length it takes.

A sphere of radius m with 4 m < L on each axis fills the pruned slots of its
lengths to the edge.  Cubic grids take the square-plane kernel, the others the
one with run-time radix pairs.  A basis listed in another order, and grids
with no room for the sphere's products, take the general kernels: the same
operator to rounding.  Bounds: FP64 transforms of length <= 120 keep 2^-52
times a few stages of growth, 1e-13 of max |H psi|; FP32 ones 2^-23 times the
same, 3e-6, as the other H|psi> tests."""

import numpy as np
import pytest

from conftest import rng
from pwgpu.context import Projectors, ScfSystem
from pwgpu.crystal import Atom, Crystal, KPoint, Lattice, miller_to_idx
from pwgpu.lib import PRECISION_FP64, PRECISION_MIXED, PwGpu
from pwgpu.symmetry import SymmetryInfo

pytestmark = pytest.mark.gpu

LENGTHS = (12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 80, 81, 90, 96, 100, 108, 120)


class _Basis:
    def __init__(self, miller):
        self.miller, self.g = miller, miller.astype(np.float64)

    def __len__(self):
        return len(self.miller)


def _sphere(m, keep=1.0, order=None, seed=0):
    """Integer points of the ellipsoid with half axes m, the axis points included."""
    ax = [np.arange(-k, k + 1) for k in m]
    p = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    p = p[np.sum((p / (np.array(m) + 0.4)) ** 2, 1) <= keep]
    if order == "permuted":
        p = p[rng(seed).permutation(len(p))]
    elif order == "reversed":
        p = p[::-1]
    return np.ascontiguousarray(p, dtype=np.int32)


def _system(dims, miller):
    n = int(np.prod(dims))
    mi = miller.astype(np.int64)
    idx = miller_to_idx(dims, mi[:, 0], mi[:, 1], mi[:, 2])
    kin = 0.1 * np.sum(mi.astype(np.float64) ** 2, 1)
    proj = Projectors(np.zeros((len(miller), 0), dtype=np.complex128), [], np.array([0], dtype=np.int32))
    s = ScfSystem(Crystal(Lattice.from_rows(np.eye(3) * 2 * np.pi), [Atom("Si", (0.0, 0.0, 0.0))]), _Basis(miller),
                  dims, idx, [KPoint(np.zeros(3), 1.0)], [kin], [proj], np.zeros(n, dtype=np.complex128), np.zeros(n),
                  np.zeros(0), 4.0, (2 * np.pi) ** 3, 0.0, SymmetryInfo.identity_only(), np.zeros(0))
    return s, idx, kin


def _check(dims, miller, nb=3, seed=1):
    s, idx, kin = _system(dims, miller)
    g = rng(seed)
    v = g.uniform(-2.0, 1.0, dims)
    psi = g.standard_normal((s.n_pw, nb)) + 1j * g.standard_normal((s.n_pw, nb))
    ref = np.empty_like(psi)
    for b in range(nb):
        grid = np.zeros(int(np.prod(dims)), dtype=np.complex128)
        grid[idx] = psi[:, b]
        r = np.fft.ifftn(grid.reshape(dims), norm="forward") * v
        ref[:, b] = np.fft.fftn(r).ravel()[idx] / v.size + kin * psi[:, b]
    scale = np.max(np.abs(ref))
    with PwGpu(s) as dev:
        dev.set_veff_g(np.fft.fftn(v).ravel() / v.size)
        for precision, tol in ((PRECISION_FP64, 1e-13), (PRECISION_MIXED, 3e-6)):
            dev.set_precision(precision)
            err = np.max(np.abs(dev.apply_h(psi) - ref)) / scale
            assert err < tol, f"{dims} precision {precision}: {err:.2e}"


@pytest.mark.parametrize("L", LENGTHS)
def test_cubic_grid_matches_numpy(L):
    m = (L - 1) // 4
    _check((L, L, L), _sphere((m, m, min(m, 3))))


@pytest.mark.parametrize("dims", [(12, 120, 15), (108, 16, 36), (72, 40, 100), (25, 27, 81), (90, 96, 18), (60, 50, 48),
                                  (30, 108, 64), (45, 20, 120)])
def test_unequal_axes_match_numpy(dims):
    m = tuple((d - 1) // 4 for d in dims)
    _check(dims, _sphere(m, keep=1.0))


def test_columns_off_centre_match_numpy():
    """Columns whose points start and end anywhere (a sphere around another origin, one column empty)."""
    p = _sphere((6, 5, 8))
    c = p + np.array([0, 0, 2])
    c = c[(np.abs(c[:, 2]) <= 9) & ~((c[:, 0] == 1) & (c[:, 1] == 2))]
    _check((32, 24, 40), np.ascontiguousarray(c, dtype=np.int32))


@pytest.mark.parametrize("order", ["permuted", "reversed"])
def test_other_basis_orders_take_the_general_kernels(order):
    _check((40, 40, 40), _sphere((9, 9, 9), order=order))


@pytest.mark.parametrize("dims", [(20, 20, 20), (75, 24, 24), (24, 24, 10), (128, 20, 20)])
def test_grids_outside_the_rule_take_the_general_kernels(dims):
    """No room for the sphere's products (2 m + 1 <= L < 4 m), and lengths that are no radix pair."""
    m = (9, 9, 9) if dims == (20, 20, 20) else (5, 5, 4)
    _check(dims, _sphere(m))


def test_large_block_matches_single_bands():
    """A block wider than one chunk of planes equals its bands one by one."""
    miller = _sphere((8, 8, 8))
    s, _, _ = _system((36, 36, 36), miller)
    g = rng(5)
    psi = g.standard_normal((s.n_pw, 530)) + 1j * g.standard_normal((s.n_pw, 530))
    with PwGpu(s) as dev:
        dev.set_veff_g(np.fft.fftn(g.uniform(-1.0, 1.0, s.dims)).ravel() / s.n_grid)
        for precision in (PRECISION_FP64, PRECISION_MIXED):
            dev.set_precision(precision)
            full = dev.apply_h(psi)
            for b in (0, 255, 256, 511, 529):
                assert np.array_equal(full[:, b], dev.apply_h(psi[:, b:b + 1])[:, 0])


@pytest.mark.parametrize("dims,nb", [((18, 18, 18), 1), ((36, 36, 27), 5), ((60, 60, 16), 40), ((96, 96, 12), 3),
                                     ((24, 36, 20), 7), ((25, 25, 25), 70)])
def test_density_matches_numpy(dims, nb):
    """Square planes (band groups summed per plane) and an unequal one (the line kernels), occupations ending in zero."""
    m = tuple((d - 1) // 4 for d in dims)
    s, idx, _ = _system(dims, _sphere(m))
    g = rng(nb)
    psi = g.standard_normal((s.n_pw, nb)) + 1j * g.standard_normal((s.n_pw, nb))
    occ = np.sort(g.uniform(0.1, 2.0, nb))[::-1].copy()
    if nb > 2:
        occ[-1] = 0.0
    rho = np.zeros(dims)
    for b in range(nb):
        grid = np.zeros(int(np.prod(dims)), dtype=np.complex128)
        grid[idx] = psi[:, b]
        rho += occ[b] * np.abs(np.fft.ifftn(grid.reshape(dims), norm="forward")) ** 2
    rho *= s.n_electrons / (rho.sum() * s.omega / rho.size)
    with PwGpu(s, gamma_complex=True) as dev:
        got = dev.density(occ[None, :], [psi])
    assert np.max(np.abs(got - rho.ravel())) < 1e-13 * np.max(rho)
