"""Forward Chebyshev columns of binary32 and double-float grids (folded straight from
global memory) against the FP64 oracle, at the edges of the fold."""
import numpy as np
import pytest

import oracle as O
import springsteel_gpu as S
from springsteel_gpu import fields
from test_gpu_parity import TOL_FAST

pytestmark = pytest.mark.gpu


# a warp folds 8 point pairs of 4 columns, a thread 8 (4) pairs at a time: pairs around 8, 16, 32 and 64,
# an odd level count (its middle point counts once); 1 to 12 rings leave a ragged block of 64 columns
@pytest.mark.parametrize("precision", ["f32", "f64_fast"])
@pytest.mark.parametrize("cells,levels", [(1, 5), (2, 15), (3, 16), (2, 17), (4, 31), (2, 33), (1, 64), (2, 65), (1, 130)])
def test_forward_columns_match_oracle(precision, cells, levels):
    gp = S.SpringsteelGridParameters(geometry="RLZ", iMin=0.0, iMax=float(cells), num_cells=cells, kMin=0.0, kMax=1000.0,
                                     kDim=levels, vars={"a": 1, "b": 2}, precision=precision,
                                     BCB={"default": S.DirichletBC()}, BCT={"default": S.NeumannBC()})
    g = S.createGrid(gp)
    pts = S.getGridpoints(g)
    u = np.column_stack([fields.blob_sum(pts, seed=70 + v, nblobs=4, wmin=1.0, wmax=4.0, zmax=1000.0, noise=1e-2)
                         for v in range(2)])
    if precision == "f32":
        u = u.astype(np.float32).astype(np.float64)
    g.set_physical(u, slot=1)
    S.spectralTransform_b(g)
    got = g.get_spectral()
    o = O.OracleGrid(gp.to_abi())
    ph = np.zeros(o.physical_shape, order="F")
    ph[:, :, 0] = u
    want = o.spectral_transform(ph)
    # binary32: levels / 2 sums of the fold, about 10 FFT stages, 12 taps and their roundings, the largest
    # coefficient down to 1/16 of the field
    tol = 16 * (levels / 2 + 24) * 2.0 ** -24 if precision == "f32" else TOL_FAST
    for v in range(2):
        assert np.max(np.abs(got[:, v] - want[:, v])) <= tol * np.max(np.abs(want[:, v]))
