"""Host fields in and out of the resident arrays (h3d_mg_upload / _download):
the contiguous route up through the staging buffer and the strided one (host
arrays that are mostly padding) move the same cells, and a download writes no
other cell of the host array."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, P = 4, 5


@pytest.mark.parametrize("pl,extra", [(1, 0), (1, 3), (2, 0), (3, 1), (3, 40)])
@pytest.mark.parametrize("field", ["p", "b", "u", "wstar", "pp"])
def test_round_trip(h3d, field, pl, extra):
    blocks = h3d.topology.block_grid((2, 1, 2), (16, 8, 12), [P, P, W, W, W, W], [1.0 / 32] * 3, 2, pl=pl)
    for d in blocks:
        for a in range(3):
            d.ttc[a] += extra
    s = h3d.MultigridSolver(blocks, 2)
    rng = np.random.default_rng(3)
    hosts = [rng.standard_normal((d.ttc[2], d.ttc[1], d.ttc[0])) for d in blocks]
    for ib, x in enumerate(hosts):
        s.upload(field, ib, x)
    for ib, (d, x) in enumerate(zip(blocks, hosts)):
        back = np.full_like(x, 7.0)
        s.download(field, ib, back)
        part = h3d.interior if field == "b" else h3d.with_ghost
        want = np.full_like(x, 7.0)
        part(want, d)[...] = part(x, d)
        assert np.array_equal(back, want), (field, pl, extra, ib)
    s.close()
