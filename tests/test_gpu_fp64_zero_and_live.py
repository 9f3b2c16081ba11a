"""FP64 solves against the level-by-level V-cycle of the entry points: the TMA sweeps
from a zero iterate (every variant that has one, chunked and ragged tiles) and the
live fills that solves use between sweeps, also after a solve that diverged and
left NaN in the ghosts of walls."""
import numpy as np
import pytest

from tests.helpers import to_oracle_descs

pytestmark = pytest.mark.gpu

W, P = 4, 5


def _pair(O, h3d, nblk, n, bc, ngrid):
    blocks = h3d.topology.block_grid(nblk, n, bc, [1.0 / 32, 1.0 / 40, 1.0 / 36], ngrid)
    s = h3d.MultigridSolver(blocks, ngrid)
    s.coeff()
    orc = O.Oracle(to_oracle_descs(O, blocks), ngrid, 3, 2, 1)
    orc.coeff()
    rng = np.random.default_rng(2)
    b = [rng.standard_normal((d.n[2], d.n[1], d.n[0])) for d in blocks]
    mean = sum(x.sum() for x in b) / sum(x.size for x in b)
    return blocks, s, orc, [x - mean for x in b]


def _solve(h3d, s, blocks, b, maxcy):
    host = [h3d.host_field(d) for d in blocks]
    for x, d, v in zip(host, blocks, b):
        h3d.interior(x, d)[...] = v
    p = [h3d.host_field(d) for d in blocks]
    info = s.newsolv_mg(p, host, tol=0.0, maxcy=maxcy)
    return p, info


@pytest.mark.parametrize("nblk,n,bc", [
    ((1, 1, 1), (32, 24, 16), [W] * 6),
    ((2, 1, 2), (48, 20, 12), [P, P, W, W, W, W]),
    ((1, 2, 1), (96, 12, 24), [W, W, P, P, P, P]),
])
def test_solve_every_variant_is_the_oracles(oracle_mod, h3d, nblk, n, bc):
    blocks, s, orc, b = _pair(oracle_mod, h3d, nblk, n, bc, 3)
    ref = orc.solve([np.zeros((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2)) for d in blocks], b, tol=0.0, maxcy=3)
    _, _, nvar = s.get_smoother(1)
    tried = 0
    for v in range(nvar):
        for zc in (5, 64):
            if not s.set_smoother(1, v, zc):
                continue
            tried += 1
            p, _ = _solve(h3d, s, blocks, b, 3)
            for x, y, d in zip(p, ref["p"], blocks):
                assert np.array_equal(h3d.interior(x, d), y[1:-1, 1:-1, 1:-1]), (v, zc)
    assert tried >= 8
    s.close()


def test_solve_after_divergence(oracle_mod, h3d):
    """NaN in b, then a clean right-hand side on the same handle; and NaN through the
    V-cycle entry point, which keeps it in every ghost."""
    blocks, s, orc, b = _pair(oracle_mod, h3d, (1, 1, 1), (16, 24, 16), [W] * 6, 3)
    ref = orc.solve([np.zeros((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2)) for d in blocks], b, tol=0.0, maxcy=2)
    bad = [x.copy() for x in b]
    bad[0][3, 4, 5] = np.nan
    for how in ("solve", "vcycle"):
        if how == "solve":
            with pytest.raises(h3d.H3DError):
                _solve(h3d, s, blocks, bad, 2)
        else:
            nz, ny, nx = s.level_dims(1, 0)
            s.put_level(1, "phi", 0, np.full((nz + 2, ny + 2, nx + 2), np.nan))
            s.put_level(1, "rhs", 0, bad[0])
            s.vcycle()
        p, _ = _solve(h3d, s, blocks, b, 2)
        assert np.array_equal(h3d.interior(p[0], blocks[0]), ref["p"][0][1:-1, 1:-1, 1:-1]), how
    s.close()


def test_solve_without_a_cycle_leaves_the_levels(oracle_mod, h3d):
    """Level iterates are cleared for the live fills before the first cycle: a solve that
    needs none changes nothing, and the cycle after it starts from what was put there."""
    blocks, s, orc, b = _pair(oracle_mod, h3d, (1, 1, 1), (16, 24, 16), [W] * 6, 3)
    nz, ny, nx = s.level_dims(1, 0)
    phi = np.random.default_rng(5).standard_normal((nz + 2, ny + 2, nx + 2))
    s.put_level(1, "phi", 0, phi)
    s.zero_field("p")
    s.zero_field("b")
    assert s.solve_resident(tol=1e-8)["outer"] == 0
    assert np.array_equal(s.get_level(1, "phi", 0), phi)
    ref = orc.solve([np.zeros((nz + 2, ny + 2, nx + 2))], b, tol=0.0, maxcy=2)
    p, _ = _solve(h3d, s, blocks, b, 2)
    assert np.array_equal(h3d.interior(p[0], blocks[0]), ref["p"][0][1:-1, 1:-1, 1:-1])
    s.close()
