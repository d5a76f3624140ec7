"""Binary32 grids' SAtransform! at any unit of length, along a slot of many decades, and at the
ends of the type's range, against the FP64 oracle (which solves the grid's own spectral array)."""
import numpy as np
import pytest

import oracle as O
import springsteel_gpu as S

pytestmark = pytest.mark.gpu

CELLS = 40


def _grid(dx, bc="natural"):
    end = {"natural": S.NaturalBC(), "dirichlet": S.DirichletBC(), "robin": S.RobinBC(1.0, 0.5 * dx)}[bc]
    return S.SpringsteelGridParameters(geometry="RL", iMin=0.0, iMax=CELLS * dx, num_cells=CELLS, vars={"u": 1},
                                       BCL={"default": end}, BCR={"default": end}, precision="f32",
                                       max_wavenumber={"default": 0})


def _rings(gp, spec):
    """f, ∂r, ∂rr of an axisymmetric field: one value a ring, from the GPU and from the oracle."""
    g, o = S.createGrid(gp), O.OracleGrid(gp.to_abi())
    g.set_spectral(spec)
    S.gridTransform_b(g)
    got, want = g.get_physical(), o.grid_transform(np.asfortranarray(spec))
    g.close()
    first = np.cumsum([0] + [4 + 4 * r for r in range(1, 3 * CELLS)])
    return got[first, 0, :3], want[first, 0, :3]


def _spectrum(gp, b):
    g = S.createGrid(gp)
    spec = np.zeros(g.spectral_shape)
    spec[: len(b), 0] = np.asarray(b, dtype=np.float32)  # wavenumber 0
    g.close()
    return spec


# the rounding of x to binary32 and of the four taps of f, ∂r, ∂rr: a few 2^-24 of x (up to 8 times f),
# and 4 times as much, in units of DX, for every derivative
TOL = 2.0 ** -24 * 32


@pytest.mark.parametrize("bc", ["natural", "dirichlet", "robin"])
@pytest.mark.parametrize("dx", [1e-6, 1e-3, 1.0, 1e4, 1e8, 1e12])
def test_solution_does_not_depend_on_the_unit_of_length(dx, bc):
    gp = _grid(dx, bc)
    got, want = _rings(gp, _spectrum(gp, dx * np.random.default_rng(3).standard_normal(CELLS + 3)))
    for d in range(3):
        assert np.max(np.abs(got[:, d] - want[:, d])) * dx ** d <= TOL * 4 ** d * np.max(np.abs(want[:, 0]))


# b falls by half a row, 2^-42 over the slot; the solution at a ring hangs on the rows around it
def test_far_field_keeps_its_bits():
    gp = _grid(1.0)
    got, want = _rings(gp, _spectrum(gp, 0.5 ** np.arange(CELLS + 3) * (1 + 0.3 * np.cos(np.arange(CELLS + 3)))))
    local = np.array([np.max(np.abs(want[max(0, r - 6): r + 7, 0])) for r in range(len(want))])
    for d in range(3):
        assert np.all(np.abs(got[:, d] - want[:, d]) <= TOL * 4 ** d * local)


# near the smallest normal numbers (entries below them lose bits to the type's spacing alone) and far above one
@pytest.mark.parametrize("scale", [2.0 ** -120, 2.0 ** -60, 2.0 ** 60])
def test_range_of_the_type(scale):
    gp = _grid(1.0)
    b = np.random.default_rng(4).standard_normal(CELLS + 3)
    b[5:9] = 0.0
    b[12] = -2.0 ** -140 / scale if scale < 1.0 else 0.0
    got, want = _rings(gp, _spectrum(gp, scale * b))
    for d in range(2):
        tol = TOL * 4 ** d * np.max(np.abs(want[:, 0])) + 8 * 2.0 ** -149
        assert np.max(np.abs(got[:, d] - want[:, d])) <= tol
