"""Digit-slice products at the ends of their range: the longest rings, against the FFT kernels."""
import ctypes as C

import numpy as np
import pytest

import springsteel_gpu as S
from springsteel_gpu import abi
from test_gpu_parity import TOL64

pytestmark = pytest.mark.gpu


def digit_stages(g):
    out = C.c_int32()
    assert S.load_library().ss_grid_digits(g.handle, C.byref(out)) == abi.SS_OK
    return out.value


def _inverse(gp, fill):
    g = S.createGrid(gp)
    spec = np.full((g.dims["n_spectral"], g.dims["nvars"]), fill)
    g.set_spectral(spec)
    S.gridTransform_b(g)
    out, on = g.get_physical(), digit_stages(g)
    g.close()
    return out, on


@pytest.mark.parametrize("cells", [241, 242, 300])
def test_longest_rings_keep_their_sign(monkeypatch, cells):
    """Equal real and imaginary parts at every wavenumber: the largest point of a ring is 1.27·n times the
    column's scale (n = 3·cells + 1; 724 and 727 at the line where the parts are stored halved)."""
    gp = S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=float(cells), num_cells=cells, kMin=0.0, kMax=1.0,
                                     kDim=3, vars={"u": 1})
    got, on = _inverse(gp, 1.0 - 2.0 ** -20)
    assert on == 15
    monkeypatch.setenv("SS_RING_DIGITS", "0")
    want, on = _inverse(gp, 1.0 - 2.0 ** -20)
    assert on == 0
    for s in range(7):
        assert np.max(np.abs(got[:, 0, s] - want[:, 0, s])) <= TOL64 * np.max(np.abs(want[:, 0, s]))


@pytest.mark.parametrize("first,second", [(32, 12), (48, 20), (12, 32)])
def test_grids_of_other_level_counts_share_the_column_kernels(first, second):
    """Creating a grid of fewer levels leaves the shared memory of the earlier grid's kernels alone."""
    def grid(levels):
        return S.createGrid(S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=6.0, num_cells=6, kMin=0.0,
                                                        kMax=10.0, kDim=levels, vars={"u": 1}))

    def transform(g):
        g.set_physical(np.random.default_rng(2).standard_normal((g.dims["n_physical"], 1)), slot=1)
        S.spectralTransform_b(g)
        S.gridTransform_b(g)
        return g.get_spectral(), g.get_physical()

    a = grid(first)
    assert digit_stages(a) == 15
    want = transform(a)
    b = grid(second)
    transform(b)
    got = transform(a)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    a.close(), b.close()
