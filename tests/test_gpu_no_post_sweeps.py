"""V(n,0) cycles (iproln = 0): the fill after the last pre-smoothing sweep of a level is the last
one before the corrections, which read edge and corner ghosts, so it has to be the whole
fill.  Level 2 of these layouts is outside the fused coarse end and the one-launch visits."""
import numpy as np
import pytest

from tests.helpers import to_oracle_descs

pytestmark = pytest.mark.gpu

W, P = 4, 5
LAYOUTS = [
    ((2, 1, 1), (64, 48, 48), [P] * 6, 3),
    ((2, 2, 1), (48, 48, 48), [P, P, P, P, W, W], 3),
]


@pytest.mark.parametrize("nblk,n,bc,ngrid", LAYOUTS)
@pytest.mark.parametrize("irestr,iproln", [(2, 0), (1, 0), (2, 1)])
def test_fp64_solve_is_the_oracles(oracle_mod, h3d, nblk, n, bc, ngrid, irestr, iproln):
    blocks = h3d.topology.block_grid(nblk, n, bc, [1.0 / 32, 1.0 / 40, 1.0 / 36], ngrid)
    rng = np.random.default_rng(4)
    b = [rng.standard_normal((d.n[2], d.n[1], d.n[0])) for d in blocks]
    mean = sum(x.sum() for x in b) / sum(x.size for x in b)
    b = [x - mean for x in b]
    orc = oracle_mod.Oracle(to_oracle_descs(oracle_mod, blocks), ngrid, 3, irestr, iproln)
    orc.coeff()
    ref = orc.solve([np.zeros((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2)) for d in blocks], b, tol=0.0, maxcy=3)
    s = h3d.MultigridSolver(blocks, ngrid, irestr=irestr, iproln=iproln)
    host = [h3d.host_field(d) for d in blocks]
    for x, d, v in zip(host, blocks, b):
        h3d.interior(x, d)[...] = v
    p = [h3d.host_field(d) for d in blocks]
    s.newsolv_mg(p, host, tol=0.0, maxcy=3)
    for x, y, d in zip(p, ref["p"], blocks):
        assert np.array_equal(h3d.interior(x, d), y[1:-1, 1:-1, 1:-1])
    s.close()


@pytest.mark.parametrize("nblk,n,bc,ngrid", LAYOUTS)
@pytest.mark.parametrize("irestr,iproln", [(2, 0), (2, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_vcycle_is_the_levels_one_by_one(h3d, nblk, n, bc, ngrid, irestr, iproln, precision):
    """The cycle against its own entry points, ghost shell included (each shows every ghost)."""
    blocks = h3d.topology.block_grid(nblk, n, bc, [1.0 / 32] * 3, ngrid)
    rng = np.random.default_rng(6)
    shape = [(d.n[2], d.n[1], d.n[0]) for d in blocks]
    phi = [rng.standard_normal([v + 2 for v in q]) for q in shape]
    rhs = [rng.standard_normal(q) for q in shape]
    out = []
    for whole in (True, False):
        s = h3d.MultigridSolver(blocks, ngrid, precision=precision, irestr=irestr, iproln=iproln)
        for ib in range(len(blocks)):
            s.put_level(1, "phi", ib, phi[ib])
            s.put_level(1, "rhs", ib, rhs[ib])
        if whole:
            s.vcycle()
        else:
            for g in range(1, ngrid):
                s.mgrelax(g, irestr)
                s.mgrestr(g + 1)
            s.mgrelax(ngrid, irestr)
            s.mgrelax(ngrid, iproln)
            for g in range(ngrid - 1, 0, -1):
                s.mgcorr(g)
                s.mgrelax(g, iproln)
        out.append([s.get_level(1, "phi", ib) for ib in range(len(blocks))])
        s.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
