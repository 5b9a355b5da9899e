"""Contexts of different grids side by side, as two systems in one program: what
one of them sets up or launches leaves the other's launches alone (limits of a
kernel that belong to the function, not to the context)."""
import threading

import numpy as np
import pytest

import _systems as S
from oracle import Oracle
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu


def test_cg_hartree_of_two_box_sizes():
    """The on-chip CG solve of a 60^3 grid takes less shared memory than that of
    64^3, by the same kernel: the 64^3 loop, configured first, runs as it does
    alone, bit for bit."""
    from salmon2_b200.rt import Context
    large, small = (synth.isolated_system(num=n, h_aa=0.25, no=1, natom=1, seed=n, rc_aa=0.7) for n in (64, 60))

    def configured(s):
        ctx = Context(s)
        ctx.set_hartree_cg(np.zeros(s.grid.shape, order="F"), layout=1)
        g = s.grid
        ctx.set_self_consistent(True, s.V_local[..., 0], np.diag([2.0 * np.pi / (n * h) for n, h in zip(g.shape, g.hgs)]))
        return ctx

    def loop(ctx):
        return ctx.download(ctx.rt_propagate(ctx.upload(large.psi), ctx.zeros(), ctx.zeros(), 4, 0.05,
                                             synth.taylor_zc(0.05))["psi"])

    alone = configured(large)
    ref = loop(alone)
    alone.close()
    first, second = configured(large), configured(small)
    assert np.array_equal(loop(first), ref)
    first.close()
    second.close()


def _together(jobs):
    """Every job in a host thread of its own (one context each); the first error."""
    errors = []

    def guarded(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_nonorthogonal_grids_in_two_threads():
    """H psi on two lattices whose tiles take 20 and 40 KB, each from its own
    host thread: no launch is refused and the results stay right."""
    from salmon2_b200.rt import Context
    cell = np.array([[0.60, 0.0, 0.0], [0.16, 0.57, 0.0], [-0.09, 0.19, 0.66]]).T
    systems = [synth.nonorthogonal_system(cell * np.array(n), n, nkgrid=1, no=1, seed=sum(n), natom=1)
               for n in ((8, 8, 8), (24, 24, 20))]
    ctxs = [Context(s) for s in systems]
    bufs = [(c.upload(s.psi), c.zeros()) for c, s in zip(ctxs, systems)]
    _together([lambda c=c, b=b: [c.hpsi(*b) for _ in range(3000)] for c, b in zip(ctxs, bufs)])
    for c, s, b in zip(ctxs, systems, bufs):
        assert S.rel_err(c.download(b[1]), Oracle(s).hpsi(s.psi)) < 1e-12
        c.close()


def test_periodic_hartree_in_two_threads():
    """The one-launch periodic Hartree solve of 8^3 and 24^3 grids (6 and 108 KB a
    CTA), each from its own host thread, against the oracle."""
    import oracle as OR
    from salmon2_b200.rt import Context
    rng, jobs = np.random.default_rng(4), []
    for n in (8, 24):
        s = synth.periodic_system(a=10.26, num=n, nkgrid=1, no=1, seed=n)
        brl = OR.primitive_b_orthogonal([m * h for m, h in zip(s.grid.shape, s.grid.hgs)])
        jobs.append((Context(s), rng.uniform(0.0, 0.2, s.grid.shape), brl))
    _together([lambda c=c, r=r, b=b: [c.hartree_periodic(r, b) for _ in range(800)] for c, r, b in jobs])
    for c, r, b in jobs:
        assert S.rel_err(c.hartree_periodic(r, b), OR.poisson_ft(r, b)) < 1e-12
        c.close()
