"""The one-sweep non-orthogonal H psi at the edges of its column tiles and z
chunks, against the oracle: rows of two tiles with a ragged last one, tiles
wider than a warp, extents of the stencil's reach (the halo wraps onto the tile
itself), z chunks of one plane to all, and two spins; H psi and one Taylor step.  1e-12
relative, as for the other sizes of this kernel."""
import numpy as np
import pytest

import _systems as S
from oracle import Oracle

pytestmark = pytest.mark.gpu

CELL = np.array([[0.60, 0.0, 0.0], [0.16, 0.57, 0.0], [-0.09, 0.19, 0.66]]).T  # per grid point


@pytest.mark.parametrize("num,no,nspin", [((65, 9, 8), 1, 1), ((9, 41, 11), 2, 1), ((8, 8, 8), 1, 2),
                                          ((24, 24, 20), 2, 2), ((33, 10, 37), 40, 1), ((12, 12, 12), 1, 1),
                                          ((13, 17, 15), 8, 1), ((20, 20, 20), 34, 1)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_tile_edges_against_oracle(num, no, nspin):
    from salmon2_b200 import synth
    from salmon2_b200.rt import Context
    s = synth.nonorthogonal_system(CELL * np.array(num), num, nkgrid=1, no=no, seed=sum(num), natom=2, nspin=nspin)
    zc = synth.taylor_zc(0.02)
    ac = (0.013, -0.021, 0.034)
    O, ctx = Oracle(s), Context(s)
    O.set_vec_Ac(ac)
    ctx.set_vec_Ac(ac)
    psi, out, work = ctx.upload(s.psi), ctx.zeros(), ctx.zeros()
    assert S.rel_err(ctx.download(ctx.hpsi(psi, out)), O.hpsi(s.psi)) < 1e-12
    assert S.rel_err(ctx.download(ctx.taylor(psi, out, work, zc)), O.taylor(s.psi, zc)) < 1e-12
    ctx.close()
