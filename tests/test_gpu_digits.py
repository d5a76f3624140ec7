"""RLZ ring and column stages as digit-slice products: edges of their tiles against the
FP64 oracle, value ranges against the FFT kernels, and the rule that chooses them."""
import numpy as np
import pytest

import springsteel_gpu as S
from springsteel_gpu import fields
from test_gpu_parity import TOL64, _assert_parity, _run_both

pytestmark = pytest.mark.gpu


def _gp(cells, levels, nvars, **kw):
    kw.setdefault("BCB", {"default": S.DirichletBC()})
    kw.setdefault("BCT", {"default": S.NeumannBC()})
    return S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=float(cells), num_cells=cells, kMin=0.0,
                                       kMax=1000.0, kDim=levels, vars={"v%d" % i: i + 1 for i in range(nvars)}, **kw)


# rings n = 2..: one K-step (n ≤ 32) to several, quadrant rows across one 128-row tile (n = 126..130 at
# 43 cells), item counts around the groups of 8, level counts around the 32-row blocks and the 16-mode
# steps, levels not a multiple of 4 (scalar stores), a kmax that ends inside a K-step, kmax = 0
@pytest.mark.parametrize("cells,levels,nvars,kmax", [
    (1, 5, 1, -1), (4, 12, 1, -1), (11, 24, 1, -1), (12, 25, 2, -1), (43, 13, 1, -1), (6, 33, 3, -1),
    (5, 72, 1, -1), (14, 16, 1, 16), (14, 16, 1, 31), (9, 16, 2, 0)])
def test_digit_products_match_oracle(cells, levels, nvars, kmax):
    gp = _gp(cells, levels, nvars, max_wavenumber={"default": kmax})
    pts = S.getGridpoints(S.createGrid(gp))
    u = np.column_stack([fields.blob_sum(pts, seed=40 + v, nblobs=4, wmin=2.0, wmax=6.0, zmax=1000.0, noise=1e-3)
                         for v in range(nvars)])
    _, _, sg, so, pg, po = _run_both(gp, u)
    _assert_parity(sg, so, pg, po, gp, tol=TOL64)


def _round_trip(gp, u):
    g = S.createGrid(gp)
    g.set_physical(u, slot=1)
    S.spectralTransform_b(g)
    S.gridTransform_b(g)
    g.synchronize()
    out = g.get_spectral(), g.get_physical()
    g.close()
    return out


def _field(gp, seed=3):
    pts = S.getGridpoints(S.createGrid(gp))
    return np.column_stack([fields.blob_sum(pts, seed=seed + v, nblobs=3, wmin=2.0, wmax=6.0, zmax=1000.0)
                            for v in range(len(gp.vars))])


def test_digit_products_scale_exactly():
    """Every column has its own exponent, so a power of two commutes with the transforms bit for bit
    down to the edge of the normal range (2^-900) and up to large values (2^700)."""
    gp = _gp(8, 12, 2)
    u = _field(gp)
    spec, phys = _round_trip(gp, u)
    for s in (-900, 700):
        sp, ph = _round_trip(gp, np.ldexp(u, s))
        assert np.array_equal(np.ldexp(spec, s), sp)
        assert np.array_equal(np.ldexp(phys, s), ph)


def test_digit_products_of_zero_and_non_finite_fields(monkeypatch):
    gp = _gp(8, 12, 2)
    u = _field(gp)
    u[:, 1] = 0.0
    _, ph = _round_trip(gp, u)
    assert np.all(ph[:, 1, :] == 0.0) and np.all(np.isfinite(ph))
    for bad in (np.nan, np.inf):
        w = u.copy()
        w[100, 0] = bad
        _, got = _round_trip(gp, w)
        monkeypatch.setenv("SS_RING_DIGITS", "0")
        _, want = _round_trip(gp, w)
        monkeypatch.delenv("SS_RING_DIGITS")
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
        assert np.all(got[:, 1, :] == 0.0)


@pytest.mark.parametrize("cells,levels,nvars", [(7, 9, 1), (20, 18, 2)])
def test_digit_and_fft_kernels_agree(monkeypatch, cells, levels, nvars):
    gp = _gp(cells, levels, nvars)
    u = _field(gp)
    spec, phys = _round_trip(gp, u)
    monkeypatch.setenv("SS_RING_DIGITS", "0")
    spec0, phys0 = _round_trip(gp, u)
    for v in range(nvars):
        assert np.max(np.abs(spec[:, v] - spec0[:, v])) <= TOL64 * np.max(np.abs(spec0[:, v]))
        for s in range(7):
            assert np.max(np.abs(phys[:, v, s] - phys0[:, v, s])) <= TOL64 * np.max(np.abs(phys0[:, v, s]))


# forward columns: 8 levels a lane, 4, 8 or 16 lanes a column (32 and 64 levels), 16 levels a K-step,
# 32 modes a block (48 and 50 levels keep 32 and 33 modes), the last level count with six K-steps
@pytest.mark.parametrize("cells,levels,nvars", [(3, 6, 1), (5, 8, 2), (4, 31, 1), (7, 32, 1), (5, 48, 1), (4, 50, 2),
                                               (6, 64, 1), (3, 65, 1), (4, 96, 1), (3, 97, 1)])
def test_forward_columns_match_oracle(cells, levels, nvars):
    gp = _gp(cells, levels, nvars)
    pts = S.getGridpoints(S.createGrid(gp))
    u = np.column_stack([fields.blob_sum(pts, seed=60 + v, nblobs=4, wmin=2.0, wmax=6.0, zmax=1000.0, noise=1e-3)
                         for v in range(nvars)])
    _, _, sg, so, pg, po = _run_both(gp, u)
    _assert_parity(sg, so, pg, po, gp, tol=TOL64)


# binary32: the four derivatives by digit products, f and the forward transform by the FFT kernels.  Small
# grids are sent there by the override: quadrants around the blocks of 16 positions (n = 2.., 43 cells:
# n up to 130), levels not a multiple of 4, item counts around the groups of 8, columns too long for the kernel
# that reads quadrant parts (210 levels); 60 cells by the rule
@pytest.mark.parametrize("cells,levels,nvars,kmax,least", [
    (1, 5, 1, -1, "1"), (5, 13, 1, -1, "1"), (6, 33, 3, -1, "1"), (43, 16, 1, -1, "1"), (14, 16, 1, 31, "1"),
    (9, 16, 2, 0, "1"), (3, 210, 1, -1, "1"), (60, 44, 2, -1, None)])
def test_binary32_derivatives_by_digits(monkeypatch, cells, levels, nvars, kmax, least):
    gp = _gp(cells, levels, nvars, max_wavenumber={"default": kmax}, precision="f32")
    u = _field(gp)
    if least:
        monkeypatch.setenv("SS_RING_DIGITS", least)
    spec, phys = _round_trip(gp, u)
    monkeypatch.setenv("SS_RING_DIGITS", "0")
    spec0, phys0 = _round_trip(gp, u)
    assert np.array_equal(spec, spec0)
    for s in (0, 5, 6):
        assert np.array_equal(phys[:, :, s], phys0[:, :, s])
    for v in range(nvars):
        for s in (1, 2, 3, 4):
            # products: 28-bit digits; FFT: 24 bits through up to log2(4n) ≤ 10 stages
            assert np.max(np.abs(phys[:, v, s] - phys0[:, v, s])) <= 1e-5 * np.max(np.abs(phys0[:, v, s]))


def test_binary32_digits_keep_non_finite_rings(monkeypatch):
    gp = _gp(6, 12, 2, precision="f32")
    u = _field(gp)
    u[:, 1] = 0.0
    u[50, 0] = np.inf
    monkeypatch.setenv("SS_RING_DIGITS", "1")
    _, got = _round_trip(gp, u)
    monkeypatch.setenv("SS_RING_DIGITS", "0")
    _, want = _round_trip(gp, u)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.all(got[:, 1, :] == 0.0)


# ring launches: buckets joined or not, an item or an output per CTA or several items, by the number
# of (ring, item) pairs.  Each gives the same bits, so a variable's result does not depend on its company
@pytest.mark.parametrize("geometry,precision,cells,levels", [
    ("RL", "f32", 120, 0), ("RL", "f32", 300, 0), ("RL", "f64", 130, 0), ("RL", "f32", 5, 0), ("RLZ", "f32", 20, 8)])
def test_ring_launches_give_the_same_bits(geometry, precision, cells, levels):
    outs = []
    for nvars in (1, 4, 12):
        kw = dict(geometry=geometry, iMin=0.0, iMax=float(cells), num_cells=cells, precision=precision,
                  vars={"v%d" % i: i + 1 for i in range(nvars)})
        if levels:
            kw.update(kMin=0.0, kMax=1000.0, kDim=levels)
        gp = S.SpringsteelGridParameters(**kw)
        n = S.getGridpoints(S.createGrid(gp)).shape[0]
        u = np.random.default_rng(5).standard_normal((n, 12))[:, :nvars]
        outs.append(_round_trip(gp, u))
    for spec, phys in outs[1:]:
        assert np.array_equal(spec[:, 0], outs[0][0][:, 0])
        assert np.array_equal(phys[:, 0], outs[0][1][:, 0])
