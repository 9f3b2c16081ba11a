"""Solves of a few thousand cells, called again and again: kernels of such sizes start before
their predecessor ends (programmatic dependent launch) and may read nothing that it
writes before they have waited for it.  The mean that remove_mean subtracts is written by
the kernel just before the one that reads it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, P = 4, 5


@pytest.mark.parametrize("nblk,n,itrsch,precision", [
    ((1, 1, 1), (16, 16, 16), 3, "mixed"),
    ((1, 1, 2), (24, 24, 32), 3, "fp64"),
    ((1, 1, 2), (24, 24, 32), 2, "fp64"),
])
def test_repeated_solves_are_the_same(h3d, nblk, n, itrsch, precision):
    blocks = h3d.topology.block_grid(nblk, n, [P, P, W, W, P, P], [1.0 / 64, 1.0 / 80, 1.0 / 72], 3)
    rng = np.random.default_rng(3)
    b = [h3d.host_field(d) for d in blocks]
    for x, d in zip(b, blocks):
        h3d.interior(x, d)[...] = rng.standard_normal((d.n[2], d.n[1], d.n[0]))
    mean = np.mean([h3d.interior(x, d).mean() for x, d in zip(b, blocks)])
    for x, d in zip(b, blocks):
        h3d.interior(x, d)[...] -= mean
    s = h3d.MultigridSolver(blocks, 3, mg_itrsch=itrsch, precision=precision)
    ref = None
    for _ in range(300):
        p = [h3d.host_field(d) for d in blocks]
        for x, d in zip(p, blocks):
            h3d.with_ghost(x, d)[...] = 0.7  # a mean for the call to remove
        s.newsolv_mg(p, b, tol=0.0, maxcy=2, remove_mean=True)
        got = np.concatenate([h3d.interior(x, d).ravel() for x, d in zip(p, blocks)])
        if ref is None:
            ref = got
            # 0.7 and its sum over n cells, each at most n roundings off
            assert abs(ref.mean()) <= 2 * ref.size * 2.0 ** -53 * (0.7 + np.abs(ref).max())
        assert np.array_equal(got, ref)
    s.close()
