"""The CG Hartree solve with every vector on chip (k_pcg_box) at the edges of
its boxes: fewer planes than the halo, uneven boxes, a row of boxes along one
axis, the largest boxes of each instantiation and a grid past them (the rows
form).  25 iterations with the threshold at zero against the oracle, 1e-10
relative as for the other sizes: the block sums are ordered differently and CG
carries those roundings forward."""
import numpy as np
import pytest

from oracle import Oracle
from salmon2_b200 import synth

pytestmark = pytest.mark.gpu


def _system(num):
    return synth.isolated_system(num=num, h_aa=0.35, no=1, natom=1, seed=sum(num), rc_aa=0.7)


@pytest.mark.parametrize("num", [(10, 9, 11), (23, 8, 31), (8, 8, 150), (53, 49, 50), (69, 70, 68), (76, 72, 74)],
                         ids=lambda n: "x".join(map(str, n)))
def test_boxes_against_oracle(num):
    from salmon2_b200.rt import Context
    import _systems as S
    s = _system(num)
    g = s.grid
    ax = [((np.arange(g.is_[d], g.ie[d] + 1) - (0.5 if g.num[d] % 2 == 0 else 0.0)) * g.hgs[d]) for d in range(3)]
    X, Y, Z = np.meshgrid(*ax, indexing="ij")
    rho = np.exp(-((X - 0.3) ** 2 + (Y + 0.2) ** 2 + (Z - 0.1) ** 2) / 1.5)
    ref, it_ref = Oracle(s).poisson_isolated_cg(rho, layout=1, threshold=0.0, maxiter=25)
    ctx = Context(s)
    got, it = ctx.hartree_isolated_cg(rho, layout=1, threshold=0.0, maxiter=25)
    assert it == it_ref == 26
    assert S.rel_err(got, ref) < 1e-10
    ctx.close()
