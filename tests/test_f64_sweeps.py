"""The FP64 sweeps of large fronts and roots (cluster panels, digit products on the tensor cores) at the
edges of their tiles: the root's Green's function (caroli_root_green) against a dense inverse.

A two-slice device of width W has no tree, so its root is the 2 W-orbital matrix E - H - Σ itself: the
widths put its size at the edges of a panel (32), of the operand tiles (32 columns, 128 rows) and of the
rows a cluster's CTAs take. Longer devices add fronts (the trailing form) of uneven sizes."""
import numpy as np
import pytest

import caroli_gb300
from caroli_gb300 import NestedTwoTerminal, Region, _native, square
from caroli_gb300.disorder import ScalarPotential, disordered
from systems import oracle_T

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _device(length, width, spread, seed):
    clean = square()
    region = Region.cuboid(clean.lattice, [length, width, 0])
    rng = np.random.RandomState(seed)
    # On-site energies over `spread` decades: rows and columns of very different scales.
    pot = (rng.uniform(size=length * width) - 0.5) * 10.0 ** rng.uniform(-spread, spread, length * width)
    dev = clean.with_onsite_term(ScalarPotential(pot, width, 1, 1))
    return NestedTwoTerminal.from_model(dev, clean, region, 0)


def _dense(s, sigma):
    y = s.system
    h = np.zeros((y.n, y.n), complex)
    h[np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)] = y.values[0]
    a = sigma.energy * np.eye(y.n) - h
    for blk, (sl, sr) in zip(y.blocks, sigma.blocks):
        a[np.ix_(blk.left, blk.left)] -= sl
        a[np.ix_(blk.right, blk.right)] -= sr
    return a


@pytest.mark.parametrize("length,width,spread", [
    (2, 1, 0), (2, 15, 0), (2, 16, 0), (2, 17, 0), (2, 32, 1), (2, 33, 0), (2, 63, 0), (2, 64, 2), (2, 65, 0),
    (2, 129, 1), (2, 200, 0), (2, 300, 0), (9, 40, 1), (24, 33, 0), (40, 37, 1), (30, 70, 0)])
def test_root_green_against_dense_inverse(length, width, spread):
    s = _device(length, width, spread, 100 * length + width)
    sigma = s.self_energies(0.37)
    a = _dense(s, sigma)
    blk = s.system.blocks[0]
    kept = np.concatenate([blk.left, blk.right])
    ref = np.linalg.inv(a)[np.ix_(kept, kept)]
    greens, st = s.plan().root_green([s._slot(sigma)], [0], [len(kept)])
    assert st[0] == 0
    # A backward-stable elimination of n unknowns, growth taken as n: n^2 eps cond(A) at the very most;
    # the bound below is n eps cond(A) in the 2-norm, which LAPACK's own inverse meets.
    bound = len(a) * EPS * np.linalg.cond(a)
    assert np.linalg.norm(greens[0][0] - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("length,width", [(40, 6), (40, 9), (33, 12), (50, 15), (37, 16), (64, 17), (45, 21), (70, 8)])
def test_small_fronts_against_dense_inverse(length, width):
    """Narrow devices: fronts of up to 64 variables, eight lanes per boundary row of any remainder."""
    s = _device(length, width, 1, 7 * length + width)
    sigma = s.self_energies(0.21)
    a = _dense(s, sigma)
    blk = s.system.blocks[0]
    kept = np.concatenate([blk.left, blk.right])
    ref = np.linalg.inv(a)[np.ix_(kept, kept)]
    greens, st = s.plan().root_green([s._slot(sigma)], [0], [len(kept)])
    assert st[0] == 0
    bound = len(a) * EPS * np.linalg.cond(a)  # as above
    assert np.linalg.norm(greens[0][0] - ref) <= bound * np.linalg.norm(ref)


def test_batches_fill_clusters_differently():
    """One solve takes clusters of 16 CTAs per matrix, forty take one CTA each: the sums run in the same
    order either way, so every T is the same to the last bit."""
    s = _device(36, 40, 0, 7)
    sigmas = [s.self_energies(e) for e in np.linspace(-1.1, 0.9, 40)]
    together = s.transmissions_with(sigmas)
    alone = [s.transmission_with(x) for x in sigmas]
    assert together == alone


@pytest.mark.parametrize("length,width", [(30, 40), (40, 48), (26, 56), (44, 41), (33, 57), (70, 72), (36, 90)])
def test_trailing_panels_of_many_solves(length, width):
    """Panels of every remainder (1, 8, 9, 16, 24, 25, ... columns) with the vectors of a matrix over several
    tiles: 330 solves take a CTA per 128 rows and columns, one takes a CTA per 32 of either. Bit for bit the same,
    and the one against a dense inverse."""
    s = _device(length, width, 1, length + 3 * width)
    sigmas = [s.self_energies(e) for e in np.linspace(-0.8, 0.7, 11)]
    alone = [s.transmission_with(x) for x in sigmas]
    assert s.transmissions_with(sigmas * 30) == alone * 30
    a = _dense(s, sigmas[4])
    blk = s.system.blocks[0]
    kept = np.concatenate([blk.left, blk.right])
    ref = np.linalg.inv(a)[np.ix_(kept, kept)]
    greens, st = s.plan().root_green([s._slot(sigmas[4])], [0], [len(kept)])
    assert st[0] == 0
    bound = len(a) * EPS * np.linalg.cond(a)  # as above
    assert np.linalg.norm(greens[0][0] - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("length,width,at", [(2, 10, 3), (1, 12, 3), (12, 9, 4), (30, 40, 5)])
def test_root_with_an_overflowing_square_is_singular(length, width, at):
    """A slice orbital at an energy whose square overflows: refused as a root that is not finite, as by the other paths."""
    clean = square()
    pot = np.zeros(length * width)
    pot[at] = 1e155
    dev = clean.with_onsite_term(ScalarPotential(pot, width, 1, 1))
    s = NestedTwoTerminal.from_model(dev, clean, Region.cuboid(clean.lattice, [length, width, 0]), 0)
    _, st, _ = s.solve_batch([s.self_energies(0.37)], [0])
    assert st[0] == _native.SINGULAR


def _scales(n, decades, rng):
    return 2.0 ** np.round(rng.uniform(-decades, decades, n) * np.log2(10.0))


@pytest.mark.parametrize("width", [20, 33, 64, 100, 161])
@pytest.mark.parametrize("form", ["rows", "columns", "both"])
def test_root_of_rows_and_columns_of_different_sizes(width, form):
    """Any matrix as the root of a one-slice device (H = 0, E = 0, A = -Σ): rows and columns scaled by powers of two over
    six decades either way, so that the exact inverse is that of the unscaled matrix, scaled."""
    s = _device(1, width, 0, 1)
    plan, n = s.plan(), width
    plan.upload_values(np.zeros_like(s.system.values[:1]))
    rng = np.random.RandomState(width)
    a0 = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    left = _scales(n, 6, rng) if form != "columns" else np.ones(n)
    right = _scales(n, 6, rng) if form != "rows" else np.ones(n)
    a = left[:, None] * a0 * right
    plan.upload_sigma(0, 0.0, [(np.asfortranarray(-a), np.zeros((n, n), complex))], [np.zeros((n, 1), complex)])
    greens, st = plan.root_green([0], [0], [n])
    assert st[0] == 0
    ref = np.linalg.inv(a0) / right[:, None] / left
    bound = n * EPS * np.linalg.cond(a0)  # as above, of the unscaled matrix
    assert np.linalg.norm(greens[0][0] - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("length,width,decades", [(14, 40, 3), (9, 64, 6), (24, 24, 6), (6, 90, 6)])
def test_fronts_of_rows_and_columns_of_different_sizes(length, width, decades):
    """H and Σ scaled on both sides by powers of two over decades either way (E = 0, A = D (E - H - Σ) D)."""
    s = _device(length, width, 0, 3 * length + width)
    y, plan = s.system, s.plan()
    sigma = s.self_energies(0.37)
    a0 = _dense(s, sigma)
    d = _scales(y.n, decades, np.random.RandomState(width))
    rows, cols = np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)
    blk, (sl, sr) = y.blocks[0], sigma.blocks[0]
    h = y.values[0] - np.where(rows == cols, 0.37, 0.0)
    plan.upload_values((d[rows] * h * d[cols])[None])
    scaled = [np.asfortranarray(d[o][:, None] * m * d[o]) for o, m in ((blk.left, sl), (blk.right, sr))]
    plan.upload_sigma(0, 0.0, [tuple(scaled)], [np.zeros((width, 1), complex)])
    kept = np.concatenate([blk.left, blk.right])
    greens, st = plan.root_green([0], [0], [len(kept)])
    assert st[0] == 0
    ref = np.linalg.inv(a0)[np.ix_(kept, kept)] / d[kept][:, None] / d[kept]
    bound = y.n * EPS * np.linalg.cond(a0)  # as above, of the unscaled matrix
    assert np.linalg.norm(greens[0][0] - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("model,shape,strength", [
    ("square", (60, 30), 16.0), ("square", (60, 30), 60.0), ("square", (120, 24), 8.0), ("square", (40, 60), 30.0),
    ("graphene", (60, 30), 8.0), ("graphene", (40, 40), 30.0), ("cubic", (24, 10, 10), 60.0)])
def test_transmission_of_localised_devices(model, shape, strength):
    """Strong disorder: T down to 1e-190, the product of couplings that decay over the pivots of a panel, relative to
    the oracle's FP64 elimination. (Both are eliminations of the same matrices: 1e-9 leaves them four decades past
    the 1e-13 by which such an elimination's T of these devices moves with the order of its sums.)"""
    clean = getattr(caroli_gb300, model)()
    region = Region.cuboid(clean.lattice, list(shape) + [0] * (3 - len(shape)))
    device = disordered(clean, region, [{"kind": "anderson", "strength": strength}], 3)
    s = NestedTwoTerminal.from_models([device], clean, region, 0)
    sigma = s.self_energies(0.13)
    ref = oracle_T(s, sigma)
    t = s.transmission_with(sigma)
    assert 0.0 < ref < 1e-10
    assert abs(t - ref) <= 1e-9 * ref


def test_localised_devices_in_a_batch():
    """Outputs computed again are the same whatever form the batch takes (a CTA per 128 rows and columns, or per 32)."""
    clean = square()
    region = Region.cuboid(clean.lattice, [40, 48, 0])
    device = disordered(clean, region, [{"kind": "anderson", "strength": 20.0}], 7)
    s = NestedTwoTerminal.from_models([device], clean, region, 0)
    sigmas = [s.self_energies(e) for e in np.linspace(-0.8, 0.7, 11)]
    alone = [s.transmission_with(x) for x in sigmas]
    assert s.transmissions_with(sigmas * 30) == alone * 30
