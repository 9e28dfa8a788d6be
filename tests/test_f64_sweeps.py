"""The FP64 sweeps of large fronts and roots (cluster panels, digit products on the tensor cores) at the
edges of their tiles: the root's Green's function (caroli_root_green) against a dense inverse.

A two-slice device of width W has no tree, so its root is the 2 W-orbital matrix E - H - Σ itself: the
widths put its size at the edges of a panel (32), of the operand tiles (32 columns, 128 rows) and of the
rows a cluster's CTAs take. Longer devices add fronts (the trailing form) of uneven sizes."""
import numpy as np
import pytest

from caroli_gb300 import NestedTwoTerminal, Region, _native, square
from caroli_gb300.disorder import ScalarPotential

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
