"""SAtransform! + SI in shared memory (32 slots per CTA): slot counts around the CTA, every Γ fold,
short splines, and the binary32 grids' FP64 solve, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
import springsteel_gpu as S
from test_gpu_parity import SLOT_DERIV, TOL64, _assert_parity, _run_both

pytestmark = pytest.mark.gpu

# boundary pairs that cover both fold forms on both ends, three-rank ends and no fold
BCS = [(S.NaturalBC(), S.NaturalBC()), (S.DirichletBC(), S.NeumannBC()), (S.CauchyBC(0.0, 0.0), S.AntisymmetricBC()),
       (S.ZerosBC(), S.SecondDerivativeBC()), (S.RobinBC(1.0, 0.5), S.ZerosBC())]


def _field(g, seed):
    rng = np.random.default_rng(seed)
    p = S.getGridpoints(g)
    return (np.exp(-((p[:, 0] - 0.4 * p[:, 0].max()) / 3.0) ** 2) * (1 + 0.3 * np.cos(p[:, 1]) + 0.2 * np.sin(2 * p[:, 1]))
            + 0.01 * rng.normal(size=p.shape[0]))


# slots 1 + 6·cells: 7 (cells 1), 31 (5), 37 (6), 61 (10), 67 (11); 16 rows and fewer
@pytest.mark.parametrize("bc", range(len(BCS)))
@pytest.mark.parametrize("cells", [4, 5, 6, 10, 11])
def test_band_solve_matches_oracle(cells, bc):
    left, right = BCS[bc]
    gp = S.SpringsteelGridParameters(geometry="RL", iMin=0.0, iMax=float(cells), num_cells=cells, vars={"u": 1},
                                     BCL={"default": left}, BCR={"default": right})
    u = _field(S.createGrid(gp), bc)
    _, _, sg, so, pg, po = _run_both(gp, u[:, None])
    _assert_parity(sg, so, pg, po, gp, tol=TOL64)


@pytest.mark.parametrize("bc", range(len(BCS)))
def test_band_solve_binary32_rounds_the_exact_solution(bc):
    """The oracle solves the binary32 grid's own spectral array in FP64; f, ∂r, ∂rr then differ by the
    binary32 rounding of a and of the ring sums alone: 2^-24 of each slot's scale, times the few dozen
    roundings of a ring (f) and times 4/DX per radial derivative of the 4-tap windows."""
    left, right = BCS[bc]
    cells = 9
    gp = S.SpringsteelGridParameters(geometry="RL", iMin=0.0, iMax=float(cells), num_cells=cells, vars={"u": 1},
                                     BCL={"default": left}, BCR={"default": right}, precision="f32")
    g, o = S.createGrid(gp), O.OracleGrid(gp.to_abi())
    g.set_physical(_field(g, 7 + bc)[:, None].astype(np.float32), slot=1)
    S.spectralTransform_b(g)
    spec = g.get_spectral()
    S.gridTransform_b(g)
    got, want = g.get_physical(), o.grid_transform(np.asfortranarray(spec))
    fmax = np.max(np.abs(want[:, 0, 0]))
    for s, (way, order) in enumerate(SLOT_DERIV[:3]):
        scale = max(np.max(np.abs(want[:, 0, s])), fmax)
        assert np.max(np.abs(got[:, 0, s] - want[:, 0, s])) <= 2.0 ** -24 * 32 * 4 ** order * scale, (s, way)


def test_band_solve_reads_the_r3x_background():
    gp = S.SpringsteelGridParameters(geometry="RL", iMin=0.0, iMax=12.0, num_cells=12, vars={"u": 1},
                                     BCL={"default": S.FixedBC()}, BCR={"default": S.NaturalBC()})
    g = S.createGrid(gp)
    b, blocks = g.dims["b_iDim"], g.dims["n_blocks"]
    rng = np.random.default_rng(5)
    ah = []
    for blk in (0, 1, blocks - 1):
        a = np.zeros(b)
        a[:3] = rng.normal(size=3)
        ah.append((0, blk, a))
    u = _field(g, 3)
    _, _, sg, so, pg, po = _run_both(gp, u[:, None], ahats=ah)
    _assert_parity(sg, so, pg, po, gp, tol=TOL64)
