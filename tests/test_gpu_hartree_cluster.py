"""The one-launch periodic Hartree solve (a cluster of eight CTAs) against the
oracle: extents below the cluster's size and odd ones (uneven slabs and line
shares, remainders of the outputs of a thread), and both sides of the line
to the six-launch form.  1e-12 relative as for the six passes: the same sums,
the inverse passes in another order."""
import dataclasses

import numpy as np
import oracle as OR
import pytest

import _systems as S
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num", [(5, 4, 6), (8, 16, 9), (13, 21, 7), (24, 24, 24), (24, 26, 23), (26, 25, 27), (4, 5, 100)],
                         ids=lambda n: "x".join(map(str, n)))
def test_hartree_against_oracle(num):
    from salmon2_b200.rt import Context
    g = synth.make_grid(list(num), 0.6, periodic=True)
    s = dataclasses.replace(S.no_pp(S.periodic_small()), grid=g, no=1, nk=1, vec_k=np.zeros((3, 1), order="F"),
                            rocc=np.full((1, 1, 1), 2.0, order="F"), wtk=np.ones(1),
                            V_local=np.zeros(num + (1,), order="F"),
                            psi=np.zeros(g.shape_array + (1, 1, 1), dtype=np.complex128, order="F"),
                            ngrid=int(np.prod(num)))
    brl = OR.primitive_b_orthogonal([n * h for n, h in zip(g.shape, g.hgs)])
    rho = np.random.default_rng(sum(num)).uniform(0.0, 0.2, num)
    ctx = Context(s)
    assert S.rel_err(ctx.hartree_periodic(rho, brl), OR.poisson_ft(rho, brl)) < 1e-12
    ctx.close()
