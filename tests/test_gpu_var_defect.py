"""The FP64 defect with variable coefficients (L_LSM) against the oracle bit for bit: its z march
(even rows of at most 512 cells, in tiles of as many rows as 256 threads hold) and the kernel of
one warp a row that takes the other sizes, alone and after the correction p + e."""
import numpy as np
import pytest

from tests.helpers import to_host, to_oracle_descs

pytestmark = pytest.mark.gpu

W, P = 4, 5
H = (1.0 / 32, 1.0 / 40, 1.0 / 24)


def _blocks(h3d, kind):
    if kind == "uneven":  # blocks of different nx: other row tiles each
        return h3d.topology.independent_blocks([(32, 8, 8), (48, 12, 4), (6, 100, 12)], H, 2), 2
    nblk, n, bc, ngrid = {
        "long rows": ((1, 1, 1), (256, 6, 10), [W, W, P, P, W, W], 2),     # two rows a tile
        "one row": ((1, 1, 1), (512, 4, 6), [W] * 6, 1),                   # one row a tile
        "over half": ((1, 1, 1), (260, 6, 10), [W, W, P, P, W, W], 1),     # one row a tile, idle threads
        "ragged": ((1, 2, 1), (20, 30, 22), [P, P, W, W, W, W], 2),        # tiles of 25 and 5 rows
        "two cells": ((1, 1, 2), (2, 6, 8), [W] * 6, 2),
        "too long": ((1, 1, 1), (516, 4, 4), [W] * 6, 1),                  # a warp a row
        "odd": ((2, 1, 1), (7, 5, 9), [W] * 6, 1),                         # a warp a row
    }[kind]
    return h3d.topology.block_grid(nblk, n, bc, H, ngrid), ngrid


def _setup(O, h3d, kind, **opts):
    blocks, ngrid = _blocks(h3d, kind)
    rng = np.random.default_rng(8)
    canon = [(d.n[2] + 2, d.n[1] + 2, d.n[0] + 2) for d in blocks]
    dens = [rng.uniform(1.0, 50.0, q) for q in canon]
    p = [rng.standard_normal(q) for q in canon]
    b = [rng.standard_normal([v - 2 for v in q]) for q in canon]
    s = h3d.MultigridSolver(blocks, ngrid, var_coef=True, **opts)
    orc = O.Oracle(to_oracle_descs(O, blocks), ngrid, 3, 2, 1, lsm=True)
    for ib, f in enumerate(to_host(blocks, dens)):
        s.set_density(ib, f)
        orc.set_density(ib, np.ascontiguousarray(dens[ib][1:-1, 1:-1, 1:-1]))
    s.coeff()
    orc.coeff()
    return blocks, s, orc, p, b


def _host(h3d, blocks, b):
    out = [h3d.host_field(d) for d in blocks]
    for f, d, v in zip(out, blocks, b):
        h3d.interior(f, d)[...] = v
    return out


KINDS = ["long rows", "one row", "over half", "ragged", "two cells", "uneven", "too long", "odd"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", KINDS)
def test_residual_bitexact(oracle_mod, h3d, kind, precision):
    blocks, s, orc, p, b = _setup(oracle_mod, h3d, kind, precision=precision)
    r, rr, bb, rinf = orc.residual(p, b)
    for ib, (f, q) in enumerate(zip(to_host(blocks, p), _host(h3d, blocks, b))):
        s.upload("p", ib, f)
        s.upload("b", ib, q)
    got = s.residual()
    for ib, want in enumerate(r):
        if precision == "mixed":  # level 1 holds the defect rounded to FP32
            want = want.astype(np.float32).astype(np.float64)
        assert np.array_equal(s.get_level(1, "rhs", ib), want), (kind, ib)
    # sums of n squares in another order: at most n roundings apart
    n = sum(x.size for x in r)
    assert abs(got[0] - rr) <= n * 2.0 ** -52 * rr and abs(got[1] - bb) <= n * 2.0 ** -52 * bb
    assert got[2] == max(float(np.abs(x).max()) for x in r)  # the flux balance: no cell volume
    s.close()


@pytest.mark.parametrize("kind", KINDS)
def test_solve_cycles_bitexact(oracle_mod, h3d, kind):
    """Two cycles: the defect after p + e."""
    blocks, s, orc, p, b = _setup(oracle_mod, h3d, kind)
    ref = orc.solve(p, b, tol=0.0, maxcy=2)
    host = to_host(blocks, p)
    s.newsolv_mg(host, _host(h3d, blocks, b), tol=0.0, maxcy=2)
    for x, y, d in zip(host, ref["p"], blocks):
        assert np.array_equal(h3d.interior(x, d), y[1:-1, 1:-1, 1:-1]), kind
    s.close()


def test_per_block_stop_rule_is_refused(oracle_mod, h3d):
    blocks, s, _, _, b = _setup(oracle_mod, h3d, "uneven")
    with pytest.raises(h3d.H3DError) as e:
        s.newsolv_mg([h3d.host_field(d) for d in blocks], _host(h3d, blocks, b), tol=1e-8, maxcy=5, stop_rule=2)
    assert e.value.code == h3d._lib.H3D_ERR_BAD_CONFIG
    s.close()
