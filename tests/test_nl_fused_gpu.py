"""The one-launch projector term against the dense operator: block widths around its column tiles and groups of bands (up
to two passes of column tiles a cluster), D blocks of several channels, rows staged at once and in several chunks with a
remainder, and both sides of the work limit past which the library products run; packed real against complex.
Bar: 1e-12 of max |H psi|, as the other FP64 H|psi> tests."""

import numpy as np
import pytest

from conftest import rng
from oracle import pwdft_oracle as O
from pwgpu.context import Projectors, ScfSystem, build_system
from pwgpu.crystal import Atom, Crystal, KPoint, Lattice, diamond_primitive, diamond_supercell, gamma_only, miller_to_idx
from pwgpu.lib import PwGpu
from pwgpu.symmetry import SymmetryInfo

pytestmark = pytest.mark.gpu


def _veff(s):
    rho_g = O.density_r_to_g(s.rho_init_r, s.dims)
    _, vxc = O.lda_xc(O.add_core(s.rho_init_r, s.rho_core_r))
    return s.v_local_g + O.hartree(rho_g, s.g_squared) + O.density_r_to_g(vxc, s.dims)


@pytest.mark.parametrize("nb", [1, 2, 8, 9, 31, 33, 64, 65, 150, 200, 257, 300])
def test_complex_matches_dense(nb, si_pp):
    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 260.0, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    veff = _veff(s)
    p = s.projectors[0]
    h = O.dense_hamiltonian(s.basis.miller, s.kinetic[0], veff, s.dims, p.b, p.d_dense())
    g = rng(nb)
    psi = g.standard_normal((s.n_pw, nb)) + 1j * g.standard_normal((s.n_pw, nb))
    ref = h @ psi
    with PwGpu(s) as dev:
        dev.set_veff_g(veff)
        got = dev.apply_h(psi)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-12


@pytest.mark.parametrize("nb", [1, 5, 32, 37])
def test_packed_real_matches_complex(nb, si_pp):
    cr = diamond_supercell("Si", 5.431, (1, 1, 1), 0.02, rng(5))
    s = build_system(cr, {"Si": si_pp}, 190.0, gamma_only(), SymmetryInfo.identity_only())
    veff = _veff(s)
    p = s.projectors[0]
    h = O.dense_hamiltonian(s.basis.miller, s.kinetic[0], veff, s.dims, p.b, p.d_dense())
    # packed basis: u -> psi(G) over the half sphere, first nonzero index positive
    mi = s.basis.miller.astype(int)
    where = {tuple(x): i for i, x in enumerate(mi.tolist())}
    half = [i for i, x in enumerate(mi.tolist()) if tuple(x) > (0, 0, 0)]
    n, nh = s.n_pw, len(half)
    t = np.zeros((n, n), dtype=np.complex128)
    t[where[(0, 0, 0)], 0] = 1.0
    for q, i in enumerate(half):
        j = where[tuple(-mi[i])]
        t[i, 1 + q] = t[j, 1 + q] = np.sqrt(0.5)
        t[i, 1 + nh + q], t[j, 1 + nh + q] = 1j * np.sqrt(0.5), -1j * np.sqrt(0.5)
    u = rng(nb).standard_normal((n, nb))
    ref = (t.conj().T @ (h @ (t @ u))).real
    with PwGpu(s) as dev:
        dev.set_veff_g(veff)
        got = dev.apply_h_packed(u)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-12


@pytest.mark.parametrize("nb", [3, 20, 64])
def test_dependent_calls_without_waits(nb, si_pp):
    """Each launch may begin while the one before it runs: a chain of calls, each reading the block the call before it
    wrote and overwriting the one that call read, equals the same chain with a wait after every call."""
    import torch

    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 260.0, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    g = rng(nb)
    psi = g.standard_normal((nb, s.n_pw)) + 1j * g.standard_normal((nb, s.n_pw))
    with PwGpu(s) as dev:
        dev.set_veff_g(_veff(s))
        out = []
        for wait in (True, False):
            a, b = torch.from_numpy(psi).cuda(), torch.empty((nb, s.n_pw), dtype=torch.complex128, device="cuda")
            torch.cuda.synchronize()
            for _ in range(6):
                dev.apply_h_device(a.data_ptr(), s.n_pw, nb, b.data_ptr(), s.n_pw)
                if wait:
                    torch.cuda.synchronize()
                a, b = b, a
            torch.cuda.synchronize()
            out.append(a.cpu().numpy())
    assert np.array_equal(out[0], out[1])


def test_capture_of_a_narrower_block(si_pp):
    """After one call with a wide block (library products) a narrower one, which takes the one-launch term, can be
    captured: it allocates nothing."""
    import torch

    s = build_system(diamond_primitive("Si", 5.431), {"Si": si_pp}, 260.0, [KPoint(np.array([0.11, -0.23, 0.31]), 1.0)])
    wide, nb = 6_000_000 // (s.n_pw * s.projectors[0].n_ch) + 1, 8
    g = rng(7)
    psi = torch.from_numpy(g.standard_normal((wide, s.n_pw)) + 1j * g.standard_normal((wide, s.n_pw))).cuda()
    out, ref = torch.zeros_like(psi), torch.zeros_like(psi)
    with PwGpu(s) as dev:
        dev.set_veff_g(_veff(s))
        dev.apply_h_device(psi.data_ptr(), s.n_pw, wide, ref.data_ptr(), s.n_pw)
        torch.cuda.synchronize()
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            dev.apply_h_device(psi.data_ptr(), s.n_pw, nb, out.data_ptr(), s.n_pw, stream=side.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        scale = float(ref.abs().max())
        assert float((out[:nb] - ref[:nb]).abs().max()) < 1e-12 * scale
        del graph


class _Basis:
    def __init__(self, miller):
        self.miller, self.g = miller, miller.astype(np.float64)

    def __len__(self):
        return len(self.miller)


def _sphere_system(radius, n_ch, gamma):
    """A sphere of plane waves with random projectors, B(-G) = conj B(G), and 4-channel D blocks; V_eff stays zero."""
    ax = np.arange(-radius, radius + 1)
    p = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    p = np.ascontiguousarray(p[np.sum((p / (radius + 0.4)) ** 2, 1) <= 1.0], dtype=np.int32)
    dims, mi, g = (4 * radius + 2 if radius % 2 else 4 * radius + 4,) * 3, p.astype(np.int64), rng(n_ch)
    b = g.standard_normal((len(p), n_ch)) + 1j * g.standard_normal((len(p), n_ch))
    b = (b + b[::-1].conj()) / np.sqrt(4 * len(p))  # -G is the mirrored row of the symmetric list
    d = [np.array([[2.0, 0.3, 0, 0], [0.3, -1.0, 0, 0], [0, 0, 1.5, 0], [0, 0, 0, -0.5]])] * (n_ch // 4)
    proj = Projectors(b, d, np.arange(0, n_ch + 1, 4, dtype=np.int32))
    n = int(np.prod(dims))
    atoms = [Atom("Si", (4.0 * i / n_ch, 0.0, 0.0)) for i in range(n_ch // 4)]
    k = np.zeros(3) if gamma else np.array([0.1, 0.2, 0.3])
    return ScfSystem(Crystal(Lattice.from_rows(np.eye(3) * 2 * np.pi), atoms), _Basis(p), dims,
                     miller_to_idx(dims, mi[:, 0], mi[:, 1], mi[:, 2]), [KPoint(k, 1.0)],
                     [0.1 * np.sum(mi.astype(np.float64) ** 2, 1)], [proj], np.zeros(n, dtype=np.complex128), np.zeros(n),
                     np.zeros(0), 4.0, (2 * np.pi) ** 3, 0.0, SymmetryInfo.identity_only(), np.zeros(0))


def _dense(s, psi):
    p = s.projectors[0]
    return s.kinetic[0][:, None] * psi + p.b @ (p.d_dense() @ (p.b.conj().T @ psi))


# radius 13: 10,059 rows, 629 a CTA; 16 complex (40 real) channels and 8 bands of a group do not fit at once: two chunks.
# radius 8: 2,517 rows; 40 channels: the complex work limit lies between 49 and 50 bands, the real one between 119 and 120.
@pytest.mark.parametrize("radius,n_ch,nb", [(13, 16, 1), (13, 16, 7), (13, 16, 28), (8, 40, 49), (8, 40, 50)])
def test_complex_chunks_and_work_limit(radius, n_ch, nb):
    s = _sphere_system(radius, n_ch, gamma=False)
    g = rng(nb)
    psi = g.standard_normal((s.n_pw, nb)) + 1j * g.standard_normal((s.n_pw, nb))
    ref = _dense(s, psi)
    with PwGpu(s) as dev:
        dev.set_veff_g(s.v_local_g)
        got = dev.apply_h(psi)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-12


@pytest.mark.parametrize("radius,n_ch,nb", [(13, 40, 1), (13, 40, 13), (13, 40, 28), (8, 40, 119), (8, 40, 120)])
def test_real_chunks_and_work_limit(radius, n_ch, nb):
    s = _sphere_system(radius, n_ch, gamma=True)
    n, zero = s.n_pw, s.n_pw // 2
    half = np.arange(zero + 1, n)  # first nonzero index positive, in basis order
    u = rng(nb).standard_normal((n, nb))
    c = np.sqrt(0.5) * (u[1:zero + 1] + 1j * u[zero + 1:])
    psi = np.empty((n, nb), dtype=np.complex128)
    psi[zero], psi[half], psi[zero - 1 - np.arange(zero)] = u[0], c, c.conj()
    h = _dense(s, psi)
    ref = np.concatenate([h[zero:zero + 1].real, np.sqrt(2.0) * h[half].real, np.sqrt(2.0) * h[half].imag])
    with PwGpu(s) as dev:
        dev.set_veff_g(s.v_local_g)
        got = dev.apply_h_packed(u)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-12
