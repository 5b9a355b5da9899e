"""Contexts of different grids side by side, as two systems in one program: what
one of them sets up or launches leaves the other's launches alone (limits of a
kernel that belong to the function, not to the context)."""
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
