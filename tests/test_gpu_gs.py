"""GPU parity of the ground-state path (real orbitals) against the oracle:
real hpsi, the CG eigensolver (with and without the low-pass
preconditioner), classical Gram-Schmidt (real, and complex as the RT path
calls it) and the subspace diagonalisation."""
import functools

import numpy as np
import pytest

import _systems as S
from oracle import Oracle
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def gs_system():
    return synth.isolated_system(num=24, no=6, natom=2, seed=41, real=True, name="gs24")


def _ctx(s):
    from salmon2_b200.rt import Context
    return Context(s)


def test_hpsi_real_parity():
    s = gs_system()
    O = Oracle(s)
    ref = O.hpsi_real(s.psi)
    ctx = _ctx(s)
    t = ctx.gs_upload(s.psi)
    h = ctx.gs_empty()
    ctx.hpsi_real(t, h)
    assert S.rel_err(ctx.gs_download(h), ref) < 1e-12


def test_gs_relayout_round_trip():
    s = gs_system()
    ctx = _ctx(s)
    assert np.array_equal(ctx.gs_download(ctx.gs_upload(s.psi)), s.psi)


@pytest.mark.parametrize("pre", ["none", "lowpass"])
def test_gscg_parity(pre):
    s = gs_system()
    O = Oracle(s)
    psi0 = O.gram_schmidt_real(s.psi)
    ref, esp_ref = O.gscg(psi0, ncg=4, precondition=(pre == "lowpass"))
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    esp = ctx.gscg(psi, ncg=4, precondition=pre)
    np.testing.assert_allclose(esp, esp_ref, rtol=1e-10, atol=1e-12)
    assert S.rel_err(ctx.gs_download(psi), ref) < 1e-9


def test_gram_schmidt_real_parity():
    s = gs_system()
    rng = np.random.default_rng(5)
    psi0 = s.psi + 0.3 * rng.standard_normal(s.psi.shape) * (s.psi != 0)
    O = Oracle(s)
    ref = O.gram_schmidt_real(psi0)
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    ctx.gram_schmidt_real(psi)
    assert S.rel_err(ctx.gs_download(psi), ref) < 1e-11


def test_subspace_diag_parity():
    s = gs_system()
    O = Oracle(s)
    psi0 = O.gram_schmidt_real(s.psi)
    ref, ev_ref = O.subspace_diag_real(psi0)
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    ev = ctx.subspace_diag_real(psi)
    np.testing.assert_allclose(ev, ev_ref, rtol=1e-10, atol=1e-12)
    got = ctx.gs_download(psi)
    # eigenvectors are defined up to sign; both sides fix the largest component positive
    assert S.rel_err(got, ref) < 1e-8


@pytest.mark.parametrize("make", [S.periodic_small, S.isolated_odd], ids=lambda f: f.__name__)
def test_gram_schmidt_complex_parity(make):
    """Complex column Gram-Schmidt (RT path, every (k, spin) group) against the
    oracle's gram_schmidt_col_complex8, on orbitals mixed to be far from
    orthonormal; the result is orthonormal in the hvol metric."""
    s = make()
    rng = np.random.default_rng(5)
    psi = s.psi.copy(order="F")
    no = s.no
    mix = np.eye(no) + 0.3 * (rng.standard_normal((no, no)) + 1j * rng.standard_normal((no, no)))
    psi = np.asfortranarray(np.einsum("xyzsok,op->xyzspk", psi, mix))
    ref = Oracle(s).gram_schmidt_complex(psi)
    ctx = _ctx(s)
    d = ctx.upload(psi)
    ctx.gram_schmidt_complex(d)
    out = ctx.download(d)
    assert S.rel_err(out, ref) < 1e-12
    sl = s.grid.interior_slices()
    for ik in range(s.nk):
        for isp in range(s.nspin):
            X = out[sl + (isp, slice(None), ik)].reshape(-1, no, order="F")
            np.testing.assert_allclose(X.conj().T @ X * s.grid.hvol, np.eye(no), atol=1e-12)


@pytest.mark.parametrize("no", [1, 2, 3, 37, 160], ids=lambda n: f"no{n}")
def test_subspace_diag_gpu_eigensolver(no):
    """The subspace Hamiltonian is diagonalised on the GPU (Householder
    reduction, accumulated reflections, implicit-shift QL).  Against numpy's
    eigvalsh of the same matrix built from the oracle's H: eigenvalues to
    1e-10, and the rotated orbitals are orthonormal and diagonalise H in the
    subspace (the residual ||H V - V Lambda|| checks of a dsyev result)."""
    s = synth.isolated_system(num=20, no=no, natom=2, seed=52 + no, real=True, name=f"gs20n{no}")
    O = Oracle(s)
    psi0 = O.gram_schmidt_real(s.psi)
    sl = s.grid.interior_slices()
    X = np.stack([psi0[sl + (0, i, 0)].ravel(order="F") for i in range(no)], axis=1)
    h = O.hpsi_real(psi0)
    HX = np.stack([h[sl + (0, i, 0)].ravel(order="F") for i in range(no)], axis=1)
    M = X.T @ HX * s.grid.hvol
    w_ref = np.linalg.eigvalsh(np.triu(M) + np.triu(M, 1).T)
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    ev = ctx.subspace_diag_real(psi)
    np.testing.assert_allclose(ev, w_ref, rtol=1e-10, atol=1e-10 * np.max(np.abs(w_ref)))
    out = ctx.gs_download(psi)
    Y = np.stack([out[sl + (0, i, 0)].ravel(order="F") for i in range(no)], axis=1)
    h2 = O.hpsi_real(out)
    HY = np.stack([h2[sl + (0, i, 0)].ravel(order="F") for i in range(no)], axis=1)
    np.testing.assert_allclose(Y.T @ Y * s.grid.hvol, np.eye(no), atol=1e-11)
    D = Y.T @ HY * s.grid.hvol
    assert np.max(np.abs(D - np.diag(w_ref))) <= 1e-9 * max(1.0, np.max(np.abs(w_ref)))


@pytest.mark.parametrize("no,dependence", [(1, 0.0), (31, 0.0), (32, 0.0), (33, 0.0), (65, 0.0), (151, 0.0), (20, 1e-3)],
                         ids=lambda v: str(v))
def test_gram_schmidt_real_all_columns_at_once(no, dependence):
    """Gram-Schmidt of all columns from one Gram matrix, at the edges of its
    32-column tiles and past the coefficients' shared-memory size, and (last
    case) orbitals so close to dependent that the column-by-column form takes
    over.  Tolerance: both forms keep rounding times the growth |T_ij| |x_i|,
    at most 100 in the one and 1 / dependence in the other, over `no` terms."""
    s = synth.isolated_system(num=(18, 17, 19), no=no, natom=1, seed=60 + no, real=True, name=f"gsall{no}")
    rng = np.random.default_rng(7)
    psi0 = s.psi + 0.2 * rng.standard_normal(s.psi.shape) * (s.psi != 0)
    if dependence:
        psi0[..., 5, 0] = psi0[..., 2, 0] + dependence * psi0[..., 5, 0]
    ref = Oracle(s).gram_schmidt_real(psi0)
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    ctx.gram_schmidt_real(psi)
    out = ctx.gs_download(psi)
    growth = 1.0 / dependence if dependence else 100.0
    assert S.rel_err(out, ref) < 4 * no * growth * 2.2e-16
    sl = s.grid.interior_slices()
    X = np.stack([out[sl + (0, i, 0)].ravel() for i in range(no)], axis=1)
    np.testing.assert_allclose(X.T @ X * s.grid.hvol, np.eye(no), atol=4 * no * growth * 2.2e-16)


@pytest.mark.parametrize("no,near", [(1, 1.0), (31, 1.0), (33, 1.0), (65, 1.0), (151, 1.0), (8, 0.05), (24, 0.1), (24, 0.015),
                                     (40, 0.03)], ids=lambda v: str(v))
def test_gram_schmidt_real_of_a_group_close_together(no, near):
    """Columns 3 to 7 within `near` of column 2 (growth 1 / near, below the limit at
    which the column form takes over), and columns far apart at the edges of the
    tiles.  Against a Householder QR, whose own error is linear in the growth: the
    coefficients from one Gram matrix lose the growth's square, 4 growth^2 2^-52 in
    a restatement in numpy; columns far apart keep 1e-14 (here ten times that)."""
    s = synth.isolated_system(num=(18, 17, 19), no=no, natom=1, seed=60 + no, real=True, name=f"gsnear{no}")
    rng = np.random.default_rng(no)
    sl = s.grid.interior_slices()
    X = rng.standard_normal((18 * 17 * 19, no))
    X /= np.linalg.norm(X, axis=0)
    if near < 1.0:
        X[:, 3:8] = X[:, 2:3] + near * X[:, 3:8]
    psi0 = np.zeros_like(s.psi)
    psi0[sl] = X.reshape((18, 17, 19, 1, no, 1), order="F")
    ctx = _ctx(s)
    psi = ctx.gs_upload(psi0)
    ctx.gram_schmidt_real(psi)
    Q = ctx.gs_download(psi)[sl].reshape(-1, no, order="F") * np.sqrt(s.grid.hvol)
    ref, r = np.linalg.qr(X)
    ref *= np.sign(np.diag(r))
    tol = 1e-13 if near == 1.0 else 16.0 * near ** -2 * 2.2e-16
    np.testing.assert_allclose(Q.T @ Q, np.eye(no), atol=tol)
    assert S.rel_err(Q, ref) < tol
    ctx.close()
