"""Relaxation visits with the blocks in shared memory and their cells in registers:
levels whose fill stays inside every block (k_relax_resident) and the many-sweep
coarsest level of the cluster, against the oracle bit for bit in FP64.  Sizes: odd
extents (pairs with one cell), one to four pairs a thread, periodic blocks
(ghosts read between the sweeps), blocks that do not fit (more than four)."""
import numpy as np
import pytest

from tests.helpers import to_oracle_descs

pytestmark = pytest.mark.gpu

W, P = 4, 5


def _run(O, h3d, blocks, ngrid, g, sweeps):
    s = h3d.MultigridSolver(blocks, ngrid)
    orc = O.Oracle(to_oracle_descs(O, blocks), ngrid, 3, 2, 1)
    orc.coeff()
    rng = np.random.default_rng(7)
    for ib in range(len(blocks)):
        nz, ny, nx = s.level_dims(g, ib)
        phi, rhs = rng.standard_normal((nz + 2, ny + 2, nx + 2)), rng.standard_normal((nz, ny, nx))
        s.put_level(g, "phi", ib, phi)
        s.put_level(g, "rhs", ib, rhs)
        orc.put_phi(g, ib, phi)
        orc.put_rhs(g, ib, rhs)
    s.mgrelax(g, sweeps)
    orc.mgrelax(g, sweeps)
    for ib in range(len(blocks)):
        a, b = s.get_level(g, "phi", ib), orc.get_phi(g, ib)
        assert np.array_equal(a, b), (ib, float(np.abs(a - b).max()))
    s.close()


@pytest.mark.parametrize("sizes", [
    [(30, 26, 22), (32, 32, 32), (2, 34, 18)],   # odd coarse extents, two cells a row
    [(32, 32, 32)] * 3,                          # the largest: four pairs a thread
    [(6, 10, 64), (18, 14, 30), (22, 26, 32)],   # one and two pairs
    [(2, 64, 64), (2, 2, 1200), (32, 32, 26)],   # a row of one cell: more than four pairs, the global kernel
])
def test_block_local_visit_bitexact(oracle_mod, h3d, sizes):
    blocks = h3d.topology.independent_blocks(sizes, (1.0 / 64, 1.0 / 48, 1.0 / 80), 2)
    _run(oracle_mod, h3d, blocks, 2, 2, 3)


@pytest.mark.parametrize("bc", [[P, P, W, W, P, P], [P] * 6])
def test_periodic_block_visit_bitexact(oracle_mod, h3d, bc):
    """One block, its own periodic partner: ghosts change between the sweeps."""
    blocks = h3d.topology.block_grid((1, 1, 1), (30, 28, 32), bc, [1.0 / 32] * 3, 2)
    _run(oracle_mod, h3d, blocks, 2, 2, 4)


@pytest.mark.parametrize("nblk,n,bc", [
    ((1, 1, 1), (16, 32, 24), [W] * 6),
    ((2, 2, 1), (20, 24, 24), [P, P, W, W, W, W]),
    ((3, 1, 2), (24, 24, 56), [W] * 6),
    ((2, 1, 1), (40, 32, 32), [P, P, W, W, W, W]),  # the second level is above the size that joins two
    ((1, 1, 1), (40, 32, 32), [W] * 6),             # the same alone: 1024 threads
])
def test_cluster_many_sweeps_bitexact(oracle_mod, h3d, nblk, n, bc):
    """A V-cycle whose coarsest level takes 12 sweeps: the cluster keeps its cells in
    registers; with 4 sweeps it does not.  Both are the level-by-level cycle."""
    blocks = h3d.topology.block_grid(nblk, n, bc, [1.0 / 32] * 3, 3)
    rng = np.random.default_rng(9)
    phis = [rng.standard_normal((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2)) for d in blocks]
    rhss = [rng.standard_normal((d.n[2], d.n[1], d.n[0])) for d in blocks]
    for sweeps in (4, 12):
        s = h3d.MultigridSolver(blocks, 3, coarse_sweeps=sweeps)
        orc = oracle_mod.Oracle(to_oracle_descs(oracle_mod, blocks), 3, 3, 2, 1)
        orc.coeff()
        for ib in range(len(blocks)):
            s.put_level(1, "phi", ib, phis[ib])
            s.put_level(1, "rhs", ib, rhss[ib])
            orc.put_phi(1, ib, phis[ib])
            orc.put_rhs(1, ib, rhss[ib])
        s.vcycle()
        # mgkcyc with `sweeps` relaxations of the coarsest level
        orc.mgrelax(1, 2); orc.mgrestr(2)
        orc.mgrelax(2, 2); orc.mgrestr(3)
        orc.mgrelax(3, sweeps)
        orc.mgcorr(2); orc.mgrelax(2, 1)
        orc.mgcorr(1); orc.mgrelax(1, 1)
        for ib in range(len(blocks)):
            a, b = s.get_level(1, "phi", ib), orc.get_phi(1, ib)
            assert np.array_equal(a, b), (sweeps, ib, float(np.abs(a - b).max()))
        s.close()


@pytest.mark.parametrize("nblk", [(1, 1, 1), (2, 1, 1)])
def test_mixed_cluster_large_coarsest_level(h3d, nblk):
    """FP32 blocks of 24 x 20 x 18 over an FP64 coarsest level of 540 cells a colour (1024 threads, a
    pass a colour), swept 12 times: the cycle through the level entry points, whose FP32
    updates round in another order (2e-5: test_gpu_parity's bound for FP32 sweeps)."""
    blocks = h3d.topology.block_grid(nblk, (48, 40, 36), [W] * 6, [1.0 / 32] * 3, 3)
    rng = np.random.default_rng(10)
    phi = [rng.standard_normal((d.n[2] + 2, d.n[1] + 2, d.n[0] + 2)) for d in blocks]
    rhs = [rng.standard_normal((d.n[2], d.n[1], d.n[0])) for d in blocks]
    out = []
    for whole in (True, False):
        s = h3d.MultigridSolver(blocks, 3, precision="mixed", coarse_sweeps=12)
        for ib in range(len(blocks)):
            s.put_level(1, "phi", ib, phi[ib])
            s.put_level(1, "rhs", ib, rhs[ib])
        if whole:
            s.vcycle()
        else:
            s.mgrelax(1, 2)
            s.mgrestr(2)
            s.mgrelax(2, 2)
            s.mgrestr(3)
            s.mgrelax(3, 12)
            s.mgcorr(2)
            s.mgrelax(2, 1)
            s.mgcorr(1)
            s.mgrelax(1, 1)
        out.append([s.get_level(1, "phi", ib) for ib in range(len(blocks))])
        s.close()
    for a, b in zip(*out):
        np.testing.assert_allclose(a, b, rtol=2e-5, atol=2e-5 * np.abs(b).max())
