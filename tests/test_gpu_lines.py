"""Line-TDMA sweeps (mg_itrsch 2) through every kernel the level can take:
whole blocks in shared memory, diagonals staged from rearranged copies, and
one thread a line in global memory.  The recurrences and their operands are the
reference's (mgsolver.for:434-549), so two sweeps are the oracle's bit for bit."""
import numpy as np
import pytest

from tests.helpers import to_oracle_descs

pytestmark = pytest.mark.gpu

W, P = 4, 5


@pytest.mark.parametrize("nblk,n,bc", [
    ((1, 1, 1), (2, 2, 2), [W] * 6),                  # whole: two cells a line
    ((2, 1, 1), (16, 16, 24), [P, P, W, W, W, W]),    # whole: the largest of the common sizes
    ((1, 2, 1), (40, 2, 34), [W, W, P, P, W, W]),     # whole: lines of two cells, more than a warp of them
    ((1, 1, 2), (32, 26, 18), [W] * 6),               # diagonals
    ((2, 1, 1), (70, 66, 4), [W, W, W, W, P, P]),     # diagonals: more than two warps of lines
    ((1, 1, 1), (4, 6, 300), [P] * 6),                # diagonals: long lines, few of them
    ((1, 1, 1), (96, 96, 4), [W] * 6),                # global: a diagonal's operands exceed shared memory
])
def test_tdma_sweeps_bitexact(oracle_mod, h3d, nblk, n, bc):
    _sweeps_bitexact(oracle_mod, h3d, h3d.topology.block_grid(nblk, n, bc, [1.0 / 32, 1.0 / 40, 1.0 / 24], 2))


def test_tdma_sweeps_uneven_blocks_bitexact(oracle_mod, h3d):
    """Blocks of different sizes in one launch: their scratch starts where the last one's ends."""
    sizes = [(40, 8, 34), (32, 26, 18), (2, 2, 2), (6, 30, 44)]
    _sweeps_bitexact(oracle_mod, h3d, h3d.topology.independent_blocks(sizes, (1.0 / 32, 1.0 / 40, 1.0 / 24), 2))


def _sweeps_bitexact(oracle_mod, h3d, blocks):
    s = h3d.MultigridSolver(blocks, 2, mg_itrsch=2)
    orc = oracle_mod.Oracle(to_oracle_descs(oracle_mod, blocks), 2, 2, 2, 1)
    orc.coeff()
    rng = np.random.default_rng(5)
    for ib, d in enumerate(blocks):
        phi = rng.standard_normal((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2))
        rhs = rng.standard_normal((d.n[2], d.n[1], d.n[0]))
        s.put_level(1, "phi", ib, phi)
        s.put_level(1, "rhs", ib, rhs)
        orc.put_phi(1, ib, phi)
        orc.put_rhs(1, ib, rhs)
    s.mgrelax(1, 2)
    orc.mgrelax(1, 2)
    for ib in range(len(blocks)):
        a, b = s.get_level(1, "phi", ib), orc.get_phi(1, ib)
        assert np.array_equal(a, b), (ib, float(np.abs(a - b).max()))
    s.close()
