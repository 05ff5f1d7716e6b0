"""The coarse levels that run in one cluster launch: slab splits and edges.

Whole FP64 cycles and solves equal the oracle bit for bit where the levels are
dealt out unevenly over the blocks (more planes than blocks, a last block with
fewer, fewer planes than blocks), with odd periodic sizes and with an odd number
of sweeps; coarsest systems below, at and above the sizes its solve is written
for are checked through the direct solve."""
import numpy as np
import pytest

from nga2_b200 import problems as P

pytestmark = pytest.mark.gpu

SLABS = [((40, 24, 36), (True, False, True)),   # three planes a block, the last blocks without any
         ((24, 20, 17), (False, True, False)),  # two planes a block, the last with one
         ((64, 40, 12), (True, True, True)),    # fewer planes than blocks
         ((21, 18, 35), (True, False, True)),   # odd periodic sizes
         ((36, 32, 32), (True, True, True))]    # the largest first level


def pair(dims, per, seed=3, **kw):
    from nga2_b200.bbmg import BBMG, BBOX, FP64
    from oracle.oracle import OracleBBMG
    stc, opr = P.random_operator(*dims, per, seed=seed)
    o = OracleBBMG(*dims, *per, method=BBOX, **kw)
    o.setup(stc, opr)
    g = BBMG(*dims, *per, method=BBOX, precision=FP64, **kw)
    g.setup(stc, opr)
    return o, g


@pytest.mark.parametrize("dims,per", SLABS)
def test_slab_splits_bitexact(dims, per):
    o, g = pair(dims, per, maxit=3, rcvg=0.0)
    assert g.cluster() == (1, 16)
    b = np.random.default_rng(5).standard_normal(dims[::-1])
    b -= b.mean()
    xo, ito, ro = o.solve(b)
    xg, itg, rg, _ = g.solve(b)
    assert ito == itg and ro == rg
    assert np.array_equal(xo, xg)


@pytest.mark.parametrize("pre,post", [(1, 2), (3, 1), (0, 2)])
def test_sweep_counts_bitexact(pre, post):
    o, g = pair((20, 12, 18), (True, False, True), maxit=2, rcvg=0.0, relax_pre=pre, relax_post=post)
    b = np.random.default_rng(6).standard_normal((18, 12, 20))
    b -= b.mean()
    xo, _, ro = o.solve(b)
    xg, _, rg, _ = g.solve(b)
    assert ro == rg and np.array_equal(xo, xg)


@pytest.mark.parametrize("dims", [(2, 3, 1), (4, 4, 2), (4, 4, 4), (5, 5, 4), (8, 8, 2), (8, 6, 3), (8, 6, 6)])
def test_coarsest_solve_sizes(dims):
    """6 to 288 unknowns: registers of one and two lanes' worth, factors on and off chip."""
    o, g = pair(dims, (False, False, False), seed=9, ncell_coarsest=300)
    n = g.nlvl
    nx, ny, nz = g.level_dims(n)
    f = np.zeros((nz + 2, ny + 2, nx + 2))
    f[1:-1, 1:-1, 1:-1] = np.random.default_rng(8).standard_normal((nz, ny, nx))
    o.put(n, "f", f)
    g.put(n, "f", f)
    o.direct_solve()
    g.step("direct", n)
    assert np.array_equal(g.get(n, "v"), o.get(n, "v"))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("dims,per", SLABS)
def test_cycle_leaves_the_vectors_of_every_level(monkeypatch, dims, per, prec):
    """v, f and r of all levels after a cycle, overlap included, equal those of one launch per pass."""
    from nga2_b200.bbmg import BBMG, FP64, MIXED, PCG_BBOX
    stc, opr = P.random_operator(*dims, per, seed=3)
    rng = np.random.default_rng(4)
    f = rng.standard_normal(tuple(n + 2 for n in dims[::-1]))
    got = []
    for cells in (None, "0"):
        if cells:
            monkeypatch.setenv("BBMG_TAIL_CELLS", cells)
        h = BBMG(*dims, *per, method=PCG_BBOX, precision=MIXED if prec else FP64)
        h.setup(stc, opr)
        h.put(1, "v", np.zeros_like(f), prec)
        h.put(1, "f", f, prec)
        h.step("cycle", 1, 0, prec)
        got.append([{w: h.get(n, w, prec) for w in ("v", "f", "r")} for n in range(1, h.nlvl + 1)])
        h.close()
    for n, (a, b) in enumerate(zip(*got)):
        for w in ("v", "f", "r"):
            assert np.array_equal(a[w], b[w]), (n + 1, w)


@pytest.mark.parametrize("dims,unknowns", [((262, 2, 2), 131), ((22, 12, 4), 132), ((38, 8, 4), 152), ((34, 18, 2), 153),
                                           ((20, 16, 4), 160), ((46, 14, 2), 161), ((12, 12, 12), 216)])
def test_solves_around_the_sizes_of_the_coarsest_solve(dims, unknowns):
    """In the cluster factors on chip up to 131 unknowns, read eight columns at a time up to 160, column by column
    above; the solve as a launch of its own, on chip up to 160, at the same sizes."""
    o, g = pair(dims, (True, False, False), seed=11, maxit=2, rcvg=0.0)
    assert g.cluster() == (1, 16)
    assert int(np.prod(g.level_dims(g.nlvl))) == unknowns
    b = np.random.default_rng(12).standard_normal(dims[::-1])
    b -= b.mean()
    xo, _, ro = o.solve(b)
    xg, _, rg, _ = g.solve(b)
    assert ro == rg and np.array_equal(xo, xg)
    n = g.nlvl
    f = np.zeros(tuple(m + 2 for m in g.level_dims(n)[::-1]))
    f[1:-1, 1:-1, 1:-1] = np.random.default_rng(13).standard_normal(tuple(g.level_dims(n)[::-1]))
    o.put(n, "f", f)
    g.put(n, "f", f)
    o.direct_solve()
    g.step("direct", n)
    assert np.array_equal(g.get(n, "v"), o.get(n, "v"))


def solved(monkeypatch, dims, per, prec, env=(), seed=3, **kw):
    """Solution, iterations and residual of a solve, and the cluster that it ran in, with BBMG_* settings."""
    from nga2_b200.bbmg import BBMG, BBOX, FP64, MIXED
    with monkeypatch.context() as m:
        for k, v in dict(env).items():
            m.setenv(k, v)
        h = BBMG(*dims, *per, method=BBOX, precision=MIXED if prec else FP64, maxit=3, rcvg=0.0, **kw)
    stc, opr = P.random_operator(*dims, per, seed=seed)
    h.setup(stc, opr)
    b = np.random.default_rng(5).standard_normal(dims[::-1])
    b -= b.mean()
    x, it, r, _ = h.solve(b)
    cl = h.cluster(prec)
    h.close()
    return (x, it, r), cl


def same(a, b):
    return np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("dims,per", SLABS)
def test_cluster_of_16_and_8_blocks_and_passes_give_the_same_bits(monkeypatch, dims, per, prec):
    ref, off = solved(monkeypatch, dims, per, prec, {"BBMG_TAIL_CELLS": "0"})
    assert off == (0, 0)
    got, cl = solved(monkeypatch, dims, per, prec)
    assert cl == (1, 16)
    assert same(got, ref)
    got, (level, blocks) = solved(monkeypatch, dims, per, prec, {"BBMG_TAIL_BLOCKS": "8"})
    assert level >= 1 and blocks == 8  # slabs twice as high: not every first level fits
    assert same(got, ref)


@pytest.mark.parametrize("pre,post,direct", [(1, 2, True), (3, 1, True), (0, 3, True), (2, 2, False)])
def test_single_precision_sweep_counts_and_relaxed_coarsest_level(monkeypatch, pre, post, direct):
    kw = dict(relax_pre=pre, relax_post=post, use_direct_solve=direct)
    dims, per = (20, 12, 18), (True, False, True)  # 5 cells in x on the third level
    ref, _ = solved(monkeypatch, dims, per, 1, {"BBMG_TAIL_CELLS": "0"}, **kw)
    got, cl = solved(monkeypatch, dims, per, 1, **kw)
    assert cl == (1, 16) and same(got, ref)


@pytest.mark.parametrize("cells", [None, "0"])
@pytest.mark.parametrize("pre,post,direct", [(3, 3, True), (1, 2, True), (2, 2, False)])
def test_odd_periodic_sizes_with_three_sweeps_bitexact(monkeypatch, cells, pre, post, direct):
    """The all-even colour has cells that meet across an odd periodic wrap: it is run again after a backward
    sweep, in the cluster and pass by pass."""
    if cells:
        monkeypatch.setenv("BBMG_TAIL_CELLS", cells)
    o, g = pair((15, 12, 9), (True, False, True), maxit=2, rcvg=0.0, relax_pre=pre, relax_post=post,
                use_direct_solve=direct)
    assert g.cluster() == ((0, 0) if cells else (1, 16))
    b = np.random.default_rng(6).standard_normal((9, 12, 15))
    b -= b.mean()
    xo, _, ro = o.solve(b)
    xg, _, rg, _ = g.solve(b)
    assert ro == rg and np.array_equal(xo, xg)


@pytest.mark.parametrize("prec,level", [(0, 2), (1, 1)])
def test_first_level_that_does_not_fit_beside_the_factors(monkeypatch, prec, level):
    """33^3 in FP64 with 125 coarsest unknowns: the cluster starts a level below; in FP32 it holds the first."""
    dims, per = (33, 33, 33), (True, True, True)
    got, cl = solved(monkeypatch, dims, per, prec)
    assert cl == (level, 16)
    ref, _ = solved(monkeypatch, dims, per, prec, {"BBMG_TAIL_CELLS": "0"})
    assert same(got, ref)
