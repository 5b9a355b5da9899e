"""A context whose grid or orbitals are set again: tables of the earlier shape are
never used with the new one, and a context set up in steps computes what a
fresh one does; a vector potential set again between replays of a caller's graph."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import _systems as S
from oracle import Oracle
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu

_dp, _ip = C.POINTER(C.c_double), C.POINTER(C.c_int)


def _set_grid(ctx, g):
    from salmon2_b200._lib import check, lib
    i3 = lambda v: (C.c_int * 3)(*[int(x) for x in v])  # noqa: E731
    maps = [np.ascontiguousarray(a, dtype=np.int32) for a in (g.idx, g.idy, g.idz)]
    lap, nab = (np.ascontiguousarray(np.asarray(a).ravel(order="F")) for a in (g.coef_lap, g.coef_nab))
    hgs = np.ascontiguousarray(g.hgs, dtype=np.float64)
    check(lib().sb200_set_grid(ctx.h, i3(g.is_), i3(g.ie), i3(g.is_array), i3(g.ie_array),
                               *[m.ctypes.data_as(_ip) for m in maps], i3(g.num), hgs.ctypes.data_as(_dp), g.hvol,
                               g.coef_lap0, lap.ctypes.data_as(_dp), nab.ctypes.data_as(_dp)))


def _set_vlocal(ctx, V):
    from salmon2_b200._lib import check, lib
    v = np.asfortranarray(V, dtype=np.float64)
    check(lib().sb200_set_vlocal(ctx.h, v.ctypes.data_as(_dp)))


def _set_orbitals(ctx, s):
    from salmon2_b200._lib import check, lib
    k, occ = np.asfortranarray(s.vec_k, dtype=np.float64), np.asfortranarray(s.rocc, dtype=np.float64)
    w = np.ascontiguousarray(s.wtk, dtype=np.float64)
    check(lib().sb200_set_orbitals(ctx.h, s.nspin, s.no, s.nk, *[a.ctypes.data_as(_dp) for a in (k, occ, w)]))
    ctx.sys, ctx.shape = s, (s.norb,) + s.grid.shape[::-1]


def _cell(num):
    cell = 0.62 * np.array(num)
    rng = np.random.default_rng(sum(num))
    grid = synth.make_grid(np.array(num), cell / np.array(num), periodic=True)
    rion = np.asfortranarray(rng.uniform(0.0, 1.0, (3, 3)) * cell[:, None])
    V = synth.gaussian_potential(grid, rion, np.full(3, -1.0), np.full(3, 1.0), cell=cell)
    pp = synth.make_pp(grid, rion, 2.2, sigma=0.6, amp=0.4, inorm=np.ones((3, 2), dtype=int), cell=cell)
    vec_k, wtk = synth.mp_kpoints(1, cell)
    return synth.System(grid, pp, 1, 2, 1, vec_k, np.full((2, 1, 1), 2.0, order="F"), wtk,
                        np.asfortranarray(V[..., None]), rion, synth.random_orbitals(grid, rng, 1, 2, 1),
                        int(np.prod(num)), 1)


def test_grid_of_as_many_points_and_other_extents():
    """12 x 24 x 12 -> 12 x 12 x 24 points: V_local and the projectors of the first
    grid are gone (H psi is refused), and right once they are set again."""
    from salmon2_b200._lib import SB200Error
    from salmon2_b200.rt import Context
    first, second = _cell((12, 24, 12)), _cell((12, 12, 24))
    ctx = Context(first)
    psi, out = ctx.upload(first.psi), ctx.zeros()
    ctx.hpsi(psi, out)
    _set_grid(ctx, second.grid)
    with pytest.raises(SB200Error):
        ctx.hpsi(psi, out)
    _set_vlocal(ctx, second.V_local)
    bare = S.no_pp(second)
    ctx.sys, ctx.shape = second, (second.norb,) + second.grid.shape[::-1]
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(second.psi), ctx.zeros())), Oracle(bare).hpsi(second.psi)) < 1e-12
    ctx.set_pp(second.pp)
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(second.psi), ctx.zeros())), Oracle(second).hpsi(second.psi)) < 1e-12
    ctx.close()


@pytest.mark.parametrize("extra", ["absorbing", "microscopic"])
def test_fields_of_the_earlier_grid(extra):
    """The absorbing boundary's plane table and the microscopic vector potential of
    a smaller grid go with it, as V_local does: H psi of the larger grid is that
    of a fresh context."""
    from salmon2_b200.rt import Context
    first, second = _cell((12, 12, 12)), _cell((12, 14, 40))
    ctx = Context(first)
    if extra == "absorbing":
        ctx.set_absorbing_boundary(w0=0.3, dr=2.0)
    else:
        ctx.set_micro_ac(0.01 * np.ones((3,) + first.grid.shape, order="F"))
    ctx.hpsi(ctx.upload(first.psi), ctx.zeros())
    _set_grid(ctx, second.grid)
    _set_vlocal(ctx, second.V_local)
    ctx.sys, ctx.shape = second, (second.norb,) + second.grid.shape[::-1]
    ctx.set_pp(second.pp)
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(second.psi), ctx.zeros())), Oracle(second).hpsi(second.psi)) < 1e-12
    if extra == "microscopic":  # a field of the new size is taken, and taken off again
        ctx.set_micro_ac(0.01 * np.ones((3,) + second.grid.shape, order="F"))
        ctx.set_micro_ac(None)
    ctx.close()


@pytest.mark.parametrize("num", [(12, 13, 14), (16, 16, 16)], ids=["cluster", "16cubed"])
def test_more_k_points_after_the_projectors(num):
    """One k-point, the projectors, then eight k-points: every phase table follows."""
    from salmon2_b200.rt import Context
    one = _cell(num)
    vec_k, wtk = synth.mp_kpoints(2, 0.62 * np.array(num))
    nk = vec_k.shape[1]
    psi = synth.random_orbitals(one.grid, np.random.default_rng(5), 1, 2, nk)
    many = dataclasses.replace(one, nk=nk, vec_k=vec_k, wtk=wtk, rocc=np.full((2, nk, 1), 2.0, order="F"), psi=psi)
    ctx = Context(one)
    _set_orbitals(ctx, many)
    O = Oracle(many)
    ac = (0.01, -0.02, 0.03)
    O.set_vec_Ac(ac)
    ctx.set_vec_Ac(ac)
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(many.psi), ctx.zeros())), O.hpsi(many.psi)) < 1e-12
    zc = synth.taylor_zc(0.03)
    got = ctx.taylor(ctx.upload(many.psi), ctx.zeros(), ctx.zeros(), zc)
    assert S.rel_err(ctx.download(got), O.taylor(many.psi, zc)) < 1e-12
    ctx.close()


def test_second_spin_after_v_local():
    """V_local of one spin, then two spins: H psi is refused until the V_local of
    both is there; back to one spin, what is there serves on."""
    from salmon2_b200._lib import SB200Error
    from salmon2_b200.rt import Context
    one = _cell((12, 11, 13))
    psi = synth.random_orbitals(one.grid, np.random.default_rng(6), 2, 2, 1)
    two = dataclasses.replace(one, nspin=2, rocc=np.full((2, 1, 2), 1.0, order="F"), psi=psi,
                              V_local=np.asfortranarray(np.concatenate([one.V_local, 1.2 * one.V_local], axis=3)))
    ctx = Context(one)
    _set_orbitals(ctx, two)
    with pytest.raises(SB200Error):
        ctx.hpsi(ctx.upload(two.psi), ctx.zeros())
    _set_vlocal(ctx, two.V_local)
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(two.psi), ctx.zeros())), Oracle(two).hpsi(two.psi)) < 1e-12
    _set_orbitals(ctx, one)
    assert S.rel_err(ctx.download(ctx.hpsi(ctx.upload(one.psi), ctx.zeros())), Oracle(one).hpsi(one.psi)) < 1e-12
    ctx.close()


def test_vector_potential_between_replays():
    """set_vec_Ac and H psi captured in a graph of the caller's: a replay takes the
    context's vector potential of that time, not the one of the capture."""
    import torch
    from salmon2_b200.rt import Context
    s = _cell((12, 13, 14))
    O, ctx, stream = Oracle(s), Context(s), torch.cuda.Stream()
    ctx.set_stream(stream)
    psi, out = ctx.upload(s.psi), ctx.zeros()
    torch.cuda.synchronize()
    ctx.set_vec_Ac((0.01, 0.0, 0.02))
    ctx.hpsi(psi, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ctx.set_vec_Ac((0.01, 0.0, 0.02))
        ctx.hpsi(psi, out)
    for ac in ((-0.03, 0.02, 0.0), (0.0, 0.05, -0.01)):
        ctx.set_vec_Ac(ac)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        O.set_vec_Ac(ac)
        assert S.rel_err(ctx.download(out), O.hpsi(s.psi)) < 1e-12
    ctx.close()
