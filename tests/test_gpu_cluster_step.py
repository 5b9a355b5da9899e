"""The cluster-resident fused Taylor step of general periodic grids against the
oracle: every cluster size and the sweeps (0), extents that leave partial warps, several columns
per thread and uneven slabs, one and two spins, with and without projectors;
H psi alone, one Taylor step, and the time loop's observables."""
import functools

import numpy as np
import pytest

import _systems as S
from oracle import Oracle
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _system(num, nspin, no, nkgrid, natom):
    """Orthorhombic periodic cell with random atoms (natom = 0: no projectors)."""
    rng = np.random.default_rng(sum(num) + 7 * natom)
    nums = np.array(num)
    cell = 0.62 * nums
    grid = synth.make_grid(nums, cell / nums, periodic=True)
    rion = np.asfortranarray(rng.uniform(0.0, 1.0, (3, max(natom, 1))) * cell[:, None])
    V = synth.gaussian_potential(grid, rion, rng.uniform(-2.0, -0.5, rion.shape[1]),
                                 rng.uniform(0.8, 1.6, rion.shape[1]), cell=cell)
    pp = synth.make_pp(grid, rion, min(2.2, 0.45 * cell.min()), sigma=0.6, amp=0.4,
                       inorm=rng.choice([-1, 1], size=(rion.shape[1], 2)), cell=cell)
    vec_k, wtk = synth.mp_kpoints(nkgrid, cell)
    nk = vec_k.shape[1]
    V_local = np.asfortranarray(np.stack([V * (1.0 + 0.1 * i) for i in range(nspin)], axis=3))
    s = synth.System(grid, pp, nspin, no, nk, vec_k, np.asfortranarray(np.full((no, nk, nspin), 2.0 / nspin)), wtk,
                     V_local, rion, synth.random_orbitals(grid, rng, nspin, no, nk), int(np.prod(nums)), 1)
    return S.no_pp(s) if natom == 0 else s


CASES = [((12, 12, 12), 1, 2, 2, 8), ((5, 9, 4), 2, 2, 1, 0), ((21, 18, 15), 2, 1, 1, 3), ((24, 23, 9), 1, 2, 1, 40),
         ((32, 32, 16), 1, 1, 1, 6)]


@pytest.mark.parametrize("clusters", ["0", "1", "2", "4", "8"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_cluster_step_against_oracle(case, clusters, monkeypatch):
    from salmon2_b200.rt import Context
    monkeypatch.setenv("SB200_CLUSTER", clusters)
    s = _system(*case)
    O = Oracle(s)
    ac = np.array([0.02, -0.01, 0.03])
    O.set_vec_Ac(ac)
    zc = synth.taylor_zc(0.04)
    ctx = Context(s)
    ctx.set_vec_Ac(ac)
    a, b, w = ctx.upload(s.psi), ctx.zeros(), ctx.zeros()
    assert S.rel_err(ctx.download(ctx.hpsi(a, b)), O.hpsi(s.psi)) < 1e-12
    assert S.rel_err(ctx.download(ctx.taylor(a, b, w, zc)), O.taylor(s.psi, zc)) < 1e-12
    nt = 3
    Ac = synth.asin2cos(nt, 0.04, 0.2, 0.01, 1.0, epdir=(0.3, 0.4, 0.8))
    ref = Oracle(s).rt_run(s.psi, nt, 0.04, zc, Ac_ext=Ac, trans_longi=1)
    got = ctx.rt_propagate(ctx.upload(s.psi), b, w, nt, 0.04, zc, Ac_ext=Ac, trans_longi="lo")
    assert S.rel_err(got["curr"], ref["curr"]) < 1e-10
    assert S.rel_err(got["rbox"], ref["rbox"]) < 1e-10
    assert S.rel_err(ctx.download(got["psi"]), ref["psi"]) < 1e-11


@pytest.mark.parametrize("no", [1, 32, 34])
def test_form_chosen_by_the_orbitals_against_oracle(no):
    """24^3: one wave of clusters (1, 32 orbitals) and one orbital or two more, which
    the sweeps take; H psi alone chooses for itself."""
    from salmon2_b200.rt import Context
    s = _system((24, 24, 24), 1, no, 1, 3)
    O, ctx = Oracle(s), Context(s)
    a, b, w = ctx.upload(s.psi), ctx.zeros(), ctx.zeros()
    assert S.rel_err(ctx.download(ctx.hpsi(a, b)), O.hpsi(s.psi)) < 1e-12
    nt, zc = 2, synth.taylor_zc(0.04)
    Ac = synth.asin2cos(nt, 0.04, 0.2, 0.01, 1.0, epdir=(0.3, 0.4, 0.8))
    ref = O.rt_run(s.psi, nt, 0.04, zc, Ac_ext=Ac)
    got = ctx.rt_propagate(a, b, w, nt, 0.04, zc, Ac_ext=Ac)
    assert S.rel_err(got["curr"], ref["curr"]) < 1e-10
    assert S.rel_err(ctx.download(got["psi"]), ref["psi"]) < 1e-11
    ctx.close()
