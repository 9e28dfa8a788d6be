"""The FP64 GEMMs on the tensor cores (traces, slice products, lead self-energies) at the edges of their
tiles (16 columns, 32 inner entries, 128 rows), against a dense solve in numpy.

A two-slice square device of width W has slices of W orbitals and no tree: its trace multiplies W x W
blocks, the refined solve multiplies Σ with as many columns as the right lead has open channels, and the
self-energies formed on the device are W x W x W products."""
import numpy as np
import pytest

from caroli_gb300 import NestedTwoTerminal, Precision, Region, _native, nested, square
from caroli_gb300.disorder import ScalarPotential

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _dense_transmission(s, sigma):
    y = s.system
    h = np.zeros((y.n, y.n), complex)
    h[np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)] = y.values[0]
    a = sigma.energy * np.eye(y.n) - h
    blk, (sl, sr) = y.blocks[0], sigma.blocks[0]
    a[np.ix_(blk.left, blk.left)] -= sl
    a[np.ix_(blk.right, blk.right)] -= sr
    g = np.linalg.inv(a)[np.ix_(blk.left, blk.right)]
    gl, gr = 1j * (sl - sl.conj().T), 1j * (sr - sr.conj().T)
    return np.trace(gl @ g @ gr @ g.conj().T).real, np.linalg.cond(a)


# Widths around one and two tiles of every kind; lengths 1 (one slice that is both) and 2.
@pytest.mark.parametrize("length,width", [(2, 1), (2, 15), (2, 16), (2, 17), (2, 31), (2, 32), (2, 33), (2, 64), (1, 33),
                                          (2, 96), (2, 127), (2, 128), (2, 129), (2, 161)])
def test_transmission_against_dense(length, width):
    clean = square()
    region = Region.cuboid(clean.lattice, [length, width, 0])
    pot = np.random.RandomState(width).uniform(-0.7, 0.7, length * width)
    s = NestedTwoTerminal.from_model(clean.with_onsite_term(ScalarPotential(pot, width, 1, 1)), clean, region, 0)
    sigma = s.self_energies(0.37)
    ref, cond = _dense_transmission(s, sigma)
    # n eps cond(A) for G, twice for |G|^2, against at most one per channel.
    bound = 4 * length * width * EPS * cond * width
    assert abs(s.transmission_with(sigma) - ref) <= bound
    on_device = s.self_energies_on_device(0.37)
    assert abs(s.transmission_with(on_device) - ref) <= bound
    s.plan().ctx.set_mixed_max_channels(1000)
    try:
        assert abs(s.transmission_with_precision(sigma, Precision.MIXED) - ref) <= 1e-8 + bound
        assert abs(s.transmission_with_precision(on_device, Precision.MIXED) - ref) <= 1e-8 + bound
    finally:
        s.plan().ctx.set_mixed_max_channels()


# Entries are cut to 62 bits below twice the largest of their row: with 1 the largest, steps of 2^-61.
@pytest.mark.parametrize("bits", [30, 50, 53, 56, 59, 61])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_cancelling_products(bits, sign):
    """Σ_L = Y diag(d) Y^† with Y = [[1, 1], [0, 1]] and d = (1 - i δ, -1): its first entry cancels to -i δ, all that
    Γ_L holds, so that T is proportional to what the product leaves of δ (three bits wide)."""
    clean = square()
    s = NestedTwoTerminal.from_model(clean, clean, Region.cuboid(clean.lattice, [2, 2, 0]), 0)
    plan, delta = s.plan(), sign * 5.0 * 2.0 ** -bits
    plan.lead_modes(0, 0, np.array([[1.0, 1.0], [0.0, 1.0]]), 1.0)
    plan.lead_modes(0, 1, np.eye(2), 1.0)
    d = [np.array([1.0 - 1j * delta, -1.0]), np.array([0.2 - 0.7j, 0.1 - 0.4j])]
    plan.sigma_from_modes(0, 0.3, [(d[0], d[1], np.zeros(0, np.int32), np.zeros(0))])
    y = s.system
    a = 0.3 * np.eye(y.n, dtype=complex)
    a[np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)] -= y.values[0]
    blk = y.blocks[0]
    sl, sr = np.array([[-1j * delta, -1.0], [-1.0, -1.0]]), np.diag(d[1])
    a[np.ix_(blk.left, blk.left)] -= sl
    a[np.ix_(blk.right, blk.right)] -= sr
    g = np.linalg.inv(a)[np.ix_(blk.left, blk.right)]
    gl, gr = 1j * (sl - sl.conj().T), 1j * (sr - sr.conj().T)
    ref = np.trace(gl @ g @ gr @ g.conj().T).real
    t, st, _ = plan.ctx.solve_multi([plan], [0], [0])
    assert st[0] == 0
    assert abs(t[0] - ref) <= 64 * EPS * np.linalg.cond(a) * abs(ref)


def test_wide_slices_go_block_by_block():
    """Slices whose digits would take more than the scratch for them (256 MB): the trace and the self-energies formed
    on the device in blocks, against a dense solve, and without more memory than the blocks take."""
    import torch

    width = 1900
    clean = square()
    pot = np.random.RandomState(5).uniform(-0.7, 0.7, width)
    region = Region.cuboid(clean.lattice, [1, width, 0])
    s = NestedTwoTerminal.from_model(clean.with_onsite_term(ScalarPotential(pot, width, 1, 1)), clean, region, 0)
    sigma = s.self_energies(0.37)
    ref, cond = _dense_transmission(s, sigma)
    bound = 4 * width * EPS * cond * width  # as above
    ctx = _native.Context(0)
    s._plan = None
    nested._CONTEXTS[0], kept = ctx, nested._CONTEXTS.get(0)
    try:
        slot = s._slot(sigma)
        before = torch.cuda.mem_get_info()[0]
        assert abs(s.transmission_with(sigma) - ref) <= bound
        # The root, its operands (3.3 KB per row), products of the trace and the digits of a block; 32 MB of small things.
        root = 16 * width * width
        assert before - torch.cuda.mem_get_info()[0] <= 3 * root + 3400 * width + (256 << 20) + (32 << 20)
        on_device = s.self_energies_on_device(0.37)
        assert abs(s.transmission_with(on_device) - ref) <= bound
    finally:
        nested._CONTEXTS.pop(0)
        if kept is not None:
            nested._CONTEXTS[0] = kept


@pytest.mark.parametrize("half", [1, 7, 20, 40])
@pytest.mark.parametrize("coupling", [1e-6, 1e-12, 1e-20])
def test_transmission_between_weakly_coupled_halves(half, coupling):
    """Left lead open on one half of the slice only, right lead on the other, the halves coupled by `coupling`: T (of its
    square's size) comes from entries of G far below those of the same columns that the closed half holds."""
    clean = square()
    width = 2 * half
    s = NestedTwoTerminal.from_model(clean, clean, Region.cuboid(clean.lattice, [2, width, 0]), 0)
    plan, y = s.plan(), s.system
    rows, cols = np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)
    across = np.asarray(y.cells)[np.repeat(np.arange(len(y.site_offsets)), y.site_orbitals), 1] >= half
    h = y.values[0] * np.where(across[rows] != across[cols], coupling, 1.0)
    plan.upload_values(h[None])
    blk = y.blocks[0]
    sl = np.diag(np.where(across[blk.left], 0.3, -0.5j))
    sr = np.diag(np.where(across[blk.right], -0.4j, 0.2))
    plan.upload_sigma(0, 0.31, [(np.asfortranarray(sl), np.asfortranarray(sr))], [np.zeros((width, 1), complex)])
    a = 0.31 * np.eye(y.n, dtype=complex)
    a[rows, cols] -= h
    a[np.ix_(blk.left, blk.left)] -= sl
    a[np.ix_(blk.right, blk.right)] -= sr
    # To first order in the coupling, exact to coupling^2: G_ab = G_aa H_ab G_bb of the uncoupled halves.
    i, j = np.nonzero(~across)[0], np.nonzero(across)[0]
    ga, gb = np.linalg.inv(a[np.ix_(i, i)]), np.linalg.inv(a[np.ix_(j, j)])
    g = np.zeros((y.n, y.n), complex)
    g[np.ix_(i, j)] = -ga @ a[np.ix_(i, j)] @ gb
    gl, gr = 1j * (sl - sl.conj().T), 1j * (sr - sr.conj().T)
    g = g[np.ix_(blk.left, blk.right)]
    ref = np.trace(gl @ g @ gr @ g.conj().T).real
    t, st, _ = plan.ctx.solve_multi([plan], [0], [0])
    assert st[0] == 0 and ref > 0.0
    cond = np.linalg.cond(a)
    bound = 2.0 * y.n * EPS * cond + 4.0 * (coupling * cond) ** 2  # both halves' inverses; the next order
    assert abs(t[0] - ref) <= bound * ref


@pytest.mark.parametrize("length,half", [(2, 7), (2, 40), (20, 20), (30, 12)])
@pytest.mark.parametrize("coupling", [1e-3, 1e-9, 1e-20])
def test_refined_transmission_between_weakly_coupled_halves(length, half, coupling):
    """The same device refined: the products of Σ with the solution hold both halves, and the open one's entries
    are `coupling` of the closed one's. Against the FP64 path; 1e-9 is ten times the refinement's tolerance."""
    clean = square()
    width = 2 * half
    s = NestedTwoTerminal.from_model(clean, clean, Region.cuboid(clean.lattice, [length, width, 0]), 0)
    plan, y = s.plan(), s.system
    rows, cols = np.repeat(np.arange(y.n), np.diff(y.row_ptr)), y.cols.astype(int)
    across = np.asarray(y.cells)[np.repeat(np.arange(len(y.site_offsets)), y.site_orbitals), 1] >= half
    plan.upload_values((y.values[0] * np.where(across[rows] != across[cols], coupling, 1.0))[None])
    blk = y.blocks[0]
    sl = np.diag(np.where(across[blk.left], 0.3, -0.5j))
    sr = np.diag(np.where(across[blk.right], -0.4j, 0.2))
    w = np.zeros((width, half), complex)
    w[np.nonzero(across[blk.right])[0], np.arange(half)] = np.sqrt(0.8)
    plan.upload_sigma(0, 0.31, [(np.asfortranarray(sl), np.asfortranarray(sr))], [np.asfortranarray(w)])
    ref, st, _ = plan.ctx.solve_multi([plan], [0], [0])
    assert st[0] == 0
    t, st, _ = plan.ctx.solve_multi([plan], [0], [0], Precision.MIXED)
    assert st[0] == 0
    assert abs(t[0] - ref[0]) <= 1e-9 * ref[0]
