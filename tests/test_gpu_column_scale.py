"""Column derivatives by digit products: as right as their own terms allow, whatever the modes that they
do not see (a column's mean) or hardly see (the low modes of a smooth column), against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
import springsteel_gpu as S
from test_gpu_digit_range import digit_stages
from test_gpu_parity import TOL64

pytestmark = pytest.mark.gpu

CELLS = 5


def _gp(levels, bc="natural"):
    end = {"natural": S.CHEB_R0, "dirichlet": S.DirichletBC(), "neumann": S.NeumannBC()}[bc]
    return S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=float(CELLS), num_cells=CELLS, kMin=0.0,
                                       kMax=10.0, kDim=levels, vars={"u": 1}, BCB={"default": end}, BCT={"default": end})


def _inverse(gp, weights):
    """Slots f, ∂z, ∂zz of a spectral array of random entries times a weight per Chebyshev mode."""
    g, o = S.createGrid(gp), O.OracleGrid(gp.to_abi())
    assert digit_stages(g) & 8
    bk = g.dims["b_kDim"]
    spec = np.random.default_rng(11).standard_normal(g.spectral_shape[0]).reshape(bk, -1)
    spec = np.asfortranarray((spec * weights(np.arange(bk))[:, None]).reshape(-1, 1))
    g.set_spectral(spec)
    S.gridTransform_b(g)
    got, want = g.get_physical(), o.grid_transform(spec)
    g.close()
    return got[:, 0, [0, 5, 6]], want[:, 0, [0, 5, 6]]


def _check(got, want):
    for s in range(3):
        assert np.max(np.abs(got[:, s] - want[:, s])) <= TOL64 * np.max(np.abs(want[:, s])), s


# natural ends: the derivatives of mode 0 (and the second one of mode 1) are zero, and no rounding of it is theirs
@pytest.mark.parametrize("levels", [12, 32, 40])
@pytest.mark.parametrize("mean", [1e3, 1e6, 1e9])
def test_derivatives_do_not_see_the_mean(levels, mean):
    _check(*_inverse(_gp(levels), lambda k: np.where(k == 0, mean, 1.0)))
    _check(*_inverse(_gp(levels), lambda k: np.where(k < 2, mean, 1.0)))


# coefficients that fall faster than the derivatives' weights grow, and as fast as those of ∂zz
@pytest.mark.parametrize("bc", ["natural", "dirichlet", "neumann"])
@pytest.mark.parametrize("levels", [12, 32, 48])
def test_derivatives_of_smooth_columns(levels, bc):
    _check(*_inverse(_gp(levels, bc), lambda k: 4.0 ** -k))
    _check(*_inverse(_gp(levels, bc), lambda k: (1.0 + k) ** -4.0))


def test_a_mode_that_is_not_finite_reaches_the_derivatives():
    got, _ = _inverse(_gp(12), lambda k: np.where(k == 0, np.nan, 1.0))
    assert np.all(np.isnan(got))
