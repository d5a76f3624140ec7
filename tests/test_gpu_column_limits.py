"""The edges of the column products: which stages of a grid run as such, and their results there against the
FP64 oracle."""
import numpy as np
import pytest

import oracle as O
import springsteel_gpu as S
from test_gpu_digit_range import digit_stages
from test_gpu_parity import TOL64

pytestmark = pytest.mark.gpu

FWD, INV = 4, 8  # SS_DIGITS_CHEB_FWD, SS_DIGITS_CHEB_INV
BOTH = FWD | INV


# levels and modes around a K-step of 16, a matrix block of 32 and 8 levels a lane (four lanes a column up to
# 32 levels, eight above); the last shapes that the shared memory holds, and the next
@pytest.mark.parametrize("levels,modes,stages", [
    (16, 16, BOTH), (17, 16, BOTH), (17, 17, BOTH), (32, 32, BOTH), (33, 32, BOTH), (33, 33, BOTH), (48, 33, BOTH),
    (48, 39, BOTH), (48, 40, FWD), (49, 32, BOTH), (49, 33, INV),
    (64, 32, BOTH), (64, 39, INV), (65, 32, INV), (96, 32, INV),
    (97, 32, 0), (160, 16, INV), (161, 16, 0)])
def test_shapes_of_the_column_products(levels, modes, stages):
    """Each direction on its own data: a derivative of the other's rounding would be the square of the mode
    number times larger, whichever kernel serves (near as many modes as levels: 10^-12 of ∂z)."""
    gp = S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=4.0, num_cells=4, kMin=0.0, kMax=1000.0, kDim=levels,
                                     b_kDim=modes, vars={"u": 1, "v": 2}, BCB={"default": S.DirichletBC(), "v": S.CHEB_R0},
                                     BCT={"default": S.NeumannBC()})
    g, o = S.createGrid(gp), O.OracleGrid(gp.to_abi())
    assert digit_stages(g) & BOTH == stages
    rng = np.random.default_rng(9)
    u = rng.standard_normal((g.dims["n_physical"], 2))
    phys = np.zeros(o.physical_shape, order="F")
    phys[:, :, 0] = u
    g.set_physical(u, slot=1)
    S.spectralTransform_b(g)
    spec = np.asfortranarray(rng.standard_normal(g.spectral_shape))
    got, want = [g.get_spectral()], [o.spectral_transform(phys)]
    g.set_spectral(spec)
    S.gridTransform_b(g)
    got.append(g.get_physical()), want.append(o.grid_transform(spec))
    g.close()
    for a, b in zip(got, want):
        for v in range(2):
            x, y = a[:, v].reshape(len(a), -1), b[:, v].reshape(len(b), -1)
            assert np.all(np.max(np.abs(x - y), axis=0) <= TOL64 * np.max(np.abs(y), axis=0))
