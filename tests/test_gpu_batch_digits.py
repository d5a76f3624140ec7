"""Fused batches of FP64 RL grids whose rings run as digit products: a few launches for all of them, and
bit for bit what each grid's own calls give."""
import numpy as np
import pytest

import springsteel_gpu as S
from test_gpu_digit_range import digit_stages

pytestmark = pytest.mark.gpu


def _grid(cells, nvars, precision="f64", levels=0, kmax=-1):
    kw = dict(kMin=0.0, kMax=10.0, kDim=levels) if levels else {}
    return S.createGrid(S.SpringsteelGridParameters(
        geometry="RLZ" if levels else "RL", iMin=0.0, iMax=float(cells), num_cells=cells, precision=precision,
        vars={"v%d" % i: i + 1 for i in range(nvars)}, max_wavenumber={"default": kmax}, **kw))


def _run(grids, order=None, fused=True):
    """(own calls, batch) of every grid."""
    fields = [np.random.default_rng(i).standard_normal((g.dims["n_physical"], g.dims["nvars"])) for i, g in enumerate(grids)]
    own = []
    for g, u in zip(grids, fields):
        g.set_physical(u, slot=1)
        S.spectralTransform_b(g)
        S.gridTransform_b(g)
        own.append((g.get_spectral(), g.get_physical()))
    batch = S.Batch([grids[i] for i in order] if order else grids, autotune=False, fused=fused)
    launches = batch.fused_launches(3)
    got = []
    for use_graph in (False, True):
        for g, u in zip(grids, fields):
            g.set_physical(u, slot=1)
            g.synchronize()
        batch.run(what=3, use_graph=use_graph)
        batch.synchronize()
        got.append([(g.get_spectral(), g.get_physical()) for g in grids])
    batch.close()
    for run in got:
        for (s0, p0), (s1, p1) in zip(own, run):
            assert np.array_equal(s0, s1) and np.array_equal(p0, p1)
    return launches


# one ring tile to several (43 cells: quadrants of up to 130 rows), items over one group of 8 and one column
# tile (13 and 33 variables), one K-step to many; every launch once, whatever the number of grids
@pytest.mark.parametrize("shapes", [[(10, 1)] * 16, [(1, 1), (2, 3), (24, 1)], [(43, 1), (12, 13), (6, 33), (80, 2)]])
def test_small_grids_share_their_launches(shapes):
    grids = [_grid(c, v) for c, v in shapes]
    assert all(digit_stages(g) for g in grids)
    # digits 3 + 3, SB projection, spline solve (a launch per class of shared memory, at most two here)
    assert 0 < _run(grids) <= 9


def test_beside_grids_of_other_kinds():
    grids = [_grid(20, 2), _grid(125, 1), _grid(20, 2, "f32"), _grid(6, 1, levels=8), _grid(14, 1, kmax=5),
             _grid(10, 1, "f64_fast")]
    assert [bool(digit_stages(g)) for g in grids] == [True, False, False, True, True, False]
    assert _run(grids) > 0


@pytest.mark.parametrize("fused", [True, False])
def test_a_grid_listed_twice(fused):
    """Once a run, like any other: two streams of one grid would share its digit buffers."""
    _run([_grid(10, 1), _grid(16, 2), _grid(5, 1, levels=12)], order=[0, 1, 2, 0, 2], fused=fused)
