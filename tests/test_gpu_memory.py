"""Handles on a device with little memory left.  What a handle holds for speed alone (staged host
fields, the wide layout of the SIP factors, the line-TDMA's rearranged copies) is given back
when an allocation that a call needs finds none, and the call goes on with the same result.
The rest of the device is taken by plain allocations, freed at the end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, P = 4, 5
MB = 1 << 20


class _Rest:
    """All but `mb` of the free device memory."""

    def __init__(self, mb):
        import torch
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        if free < (mb + 64) * MB:
            pytest.skip("the device is in use")
        self.t = torch.empty(free - mb * MB, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch
        del self.t
        torch.cuda.empty_cache()


def _fields(blocks, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((d.ttc[2], d.ttc[1], d.ttc[0])) for d in blocks]


def _sip_run(h3d, s, blocks, b):
    for ib, d in enumerate(blocks):
        s.upload("b", ib, b[ib])
        s.upload("pp", ib, np.zeros_like(b[ib]))
    sweeps, _ = s.sipsol(3)
    out = []
    for ib, d in enumerate(blocks):
        x = np.zeros_like(b[ib])
        s.download("pp", ib, x)
        out.append(h3d.interior(x, d).copy())
    return sweeps, out


def test_sip_factors_and_staging_are_given_back(h3d):
    """Eight blocks of 64^3 cells: the wide factors take 272 MB, the plain ones 163, a field 20."""
    blocks = h3d.topology.block_grid((2, 2, 2), (64, 64, 64), [W] * 6, [1.0 / 128] * 3, 2)
    b = _fields(blocks, 2)
    with h3d.MultigridSolver(blocks, 2) as s:  # every kernel is loaded, and the result with memory to spare
        want = _sip_run(h3d, s, blocks, b)
        s.calvel(0.5)
    with h3d.MultigridSolver(blocks, 2) as s:
        s.coeff()
        with _Rest(400):  # the wide factors and what goes with them
            got = _sip_run(h3d, s, blocks, b)
            assert got[0] == want[0] and all(np.array_equal(x, y) for x, y in zip(got[1], want[1]))
            s.calvel(0.5)  # six velocity fields, 122 MB: more than is left
            got = _sip_run(h3d, s, blocks, b)  # the plain factors
            assert got[0] == want[0] and all(np.array_equal(x, y) for x, y in zip(got[1], want[1]))


def test_line_scratch_is_given_back(h3d):
    """Eight blocks of 48^3 cells with the line smoother: the rearranged copies of level 1 take 48 MB,
    six velocity fields 53."""
    blocks = h3d.topology.block_grid((2, 2, 2), (48, 48, 48), [W] * 6, [1.0 / 96] * 3, 3)
    b = _fields(blocks, 4)
    mean = np.mean([h3d.interior(x, d).mean() for x, d in zip(b, blocks)])
    b = [x - mean for x in b]

    def solve(s):
        p = [h3d.host_field(d) for d in blocks]
        s.newsolv_mg(p, b, tol=0.0, maxcy=2)
        return [h3d.interior(x, d).copy() for x, d in zip(p, blocks)]

    with h3d.MultigridSolver(blocks, 3, mg_itrsch=2) as s:
        want = solve(s)
        s.calvel(0.5)
    with h3d.MultigridSolver(blocks, 3, mg_itrsch=2) as s:
        s.coeff()
        assert all(np.array_equal(x, y) for x, y in zip(solve(s), want))
        with _Rest(24):
            s.calvel(0.5)
            assert all(np.array_equal(x, y) for x, y in zip(solve(s), want))
