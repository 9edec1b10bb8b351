"""Launches that begin beside the one before them, in every form of H|psi>: a chain of calls, each reading the block the
call before it wrote and overwriting the one that call read, equals the same chain with a wait after every call, bit for
bit.  Systems are spheres on a grid with random projectors (none, few, and more than the one-launch term takes)."""

import numpy as np
import pytest
import torch

from conftest import rng
from oracle import pwdft_oracle as O
from pwgpu.context import Projectors, ScfSystem, build_system
from pwgpu.crystal import Atom, Crystal, KPoint, Lattice, diamond_supercell, gamma_only, miller_to_idx
from pwgpu.lib import PRECISION_FP64, PRECISION_MIXED, PwGpu
from pwgpu.symmetry import SymmetryInfo

pytestmark = pytest.mark.gpu


class _Basis:
    def __init__(self, miller):
        self.miller, self.g = miller, miller.astype(np.float64)

    def __len__(self):
        return len(self.miller)


def _system(dims, n_ch, order=None):
    m = np.array([(d - 1) // 4 for d in dims])
    p = np.stack(np.meshgrid(*[np.arange(-k, k + 1) for k in m], indexing="ij"), -1).reshape(-1, 3)
    p = np.ascontiguousarray(p[np.sum((p / (m + 0.4)) ** 2, 1) <= 1.0], dtype=np.int32)
    if order == "permuted":
        p = np.ascontiguousarray(p[rng(2).permutation(len(p))])
    mi, n, g = p.astype(np.int64), int(np.prod(dims)), rng(n_ch)
    b = g.standard_normal((len(p), n_ch)) + 1j * g.standard_normal((len(p), n_ch))
    b /= np.sqrt(2 * len(p))
    proj = Projectors(b, [np.diag([2.0, -1.0, -1.0, 0.5])] * (n_ch // 4), np.arange(0, n_ch + 1, 4, dtype=np.int32))
    atoms = [Atom("Si", (i / max(1, n_ch // 4), 0.0, 0.0)) for i in range(max(1, n_ch // 4))]
    return ScfSystem(Crystal(Lattice.from_rows(np.eye(3) * 2 * np.pi), atoms), _Basis(p), dims,
                     miller_to_idx(dims, mi[:, 0], mi[:, 1], mi[:, 2]), [KPoint(np.array([0.1, 0.2, 0.3]), 1.0)],
                     [0.1 * np.sum(mi.astype(np.float64) ** 2, 1)], [proj], np.zeros(n, dtype=np.complex128), np.zeros(n),
                     np.zeros(0), 4.0, (2 * np.pi) ** 3, 0.0, SymmetryInfo.identity_only(), np.zeros(0))


def _handle(s, precision):
    dev = PwGpu(s, precision=precision)
    dev.set_veff_g(np.fft.fftn(rng(3).uniform(-2.0, 1.0, s.dims)).ravel() / s.n_grid)
    return dev


def _start(s, nb, seed):
    g = rng(seed)
    return torch.from_numpy(g.standard_normal((nb, s.n_pw)) + 1j * g.standard_normal((nb, s.n_pw))).cuda()


FORMS = {
    "square planes": ((36, 36, 36), 16, 20, None),
    "run-time radices": ((40, 36, 50), 16, 20, None),
    "no projectors": ((36, 36, 36), 0, 7, None),
    "library projector products": ((40, 40, 40), 160, 20, None),
    "line kernels": ((36, 36, 36), 16, 9, "permuted"),
    "several chunks of bands": ((24, 24, 24), 8, 600, None),
}


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
@pytest.mark.parametrize("form", list(FORMS))
def test_chain_equals_the_chain_with_waits(form, precision):
    dims, n_ch, nb, order = FORMS[form]
    s = _system(dims, n_ch, order)
    out = []
    with _handle(s, precision) as dev:
        for wait in (True, False):
            a, b = _start(s, nb, 1), torch.empty((nb, s.n_pw), dtype=torch.complex128, device="cuda")
            torch.cuda.synchronize()
            for k in range(6):
                width = nb - k if k % 2 else nb  # widths alternate
                dev.apply_h_device(a.data_ptr(), s.n_pw, width, b.data_ptr(), s.n_pw)
                if wait:
                    torch.cuda.synchronize()
                a, b = b, a
            torch.cuda.synchronize()
            out.append(a[:nb - 5].cpu().numpy())
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0], out[1])


def test_two_handles_on_two_streams():
    s1, s2 = _system((36, 36, 36), 16), _system((40, 36, 50), 24)
    with _handle(s1, PRECISION_FP64) as d1, _handle(s2, PRECISION_MIXED) as d2:
        pairs = [(d1, s1, torch.cuda.Stream()), (d2, s2, torch.cuda.Stream())]
        out = []
        for wait in (True, False):
            buf = [[_start(s, 12, 4), torch.empty((12, s.n_pw), dtype=torch.complex128, device="cuda")]
                   for _, s, _ in pairs]
            torch.cuda.synchronize()
            for _ in range(6):
                for (dev, s, st), ab in zip(pairs, buf):
                    dev.apply_h_device(ab[0].data_ptr(), s.n_pw, 12, ab[1].data_ptr(), s.n_pw, stream=st.cuda_stream)
                    if wait:
                        torch.cuda.synchronize()
                    ab.reverse()
            torch.cuda.synchronize()
            out.append([ab[0].cpu().numpy() for ab in buf])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("bands", [4, 20])
def test_packed_real_solves_repeat(bands, si_pp):
    """Unpack, local part, pack and projector term of packed real bands inside the block steps: the same bits each time."""
    cr = diamond_supercell("Si", 5.431, (1, 1, 1), 0.02, rng(5))
    s = build_system(cr, {"Si": si_pp}, 190.0, gamma_only(), SymmetryInfo.identity_only())
    rho_g = O.density_r_to_g(s.rho_init_r, s.dims)
    _, vxc = O.lda_xc(O.add_core(s.rho_init_r, s.rho_core_r))
    with PwGpu(s) as dev:
        dev.set_veff_g(s.v_local_g + O.hartree(rho_g, s.g_squared) + O.density_r_to_g(vxc, s.dims))
        ev, psi, its, _ = dev.eigensolve(bands, tol=1e-7, max_iter=400)
        for _ in range(5):
            e2, p2, i2, _ = dev.eigensolve(bands, tol=1e-7, max_iter=400)
            assert i2 == its and np.array_equal(ev, e2) and np.array_equal(psi, p2)
