"""The matrix digits that grids of the same rings share: held once, until the last such grid goes."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import springsteel_gpu as S
from test_gpu_digit_range import digit_stages

pytestmark = pytest.mark.gpu


def _grid(cells, nvars=1, kmax=-1, levels=0):
    kw = dict(kMin=0.0, kMax=10.0, kDim=levels) if levels else {}
    g = S.createGrid(S.SpringsteelGridParameters(
        geometry="RLZ" if levels else "RL", iMin=0.0, iMax=float(cells), num_cells=cells,
        vars={"v%d" % i: i + 1 for i in range(nvars)}, max_wavenumber={"default": kmax}, **kw))
    assert digit_stages(g)
    return g


def _transform(g):
    g.set_physical(np.random.default_rng(5).standard_normal((g.dims["n_physical"], g.dims["nvars"])), slot=1)
    S.spectralTransform_b(g)
    S.gridTransform_b(g)
    return g.get_spectral(), g.get_physical()


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_memory_of_further_grids():
    before = _free()
    first = _grid(100)
    tables = before - _free()
    assert tables > 600e6  # two directions of 0.3 GB
    others = [_grid(100) for _ in range(4)]
    assert before - _free() < tables + 4 * 200e6
    for g in [first] + others:
        g.close()
    assert before - _free() < 64e6


# same rings, whatever the variables and levels; a cap of the wavenumbers is another matrix
@pytest.mark.parametrize("other", [dict(), dict(nvars=3), dict(kmax=9), dict(levels=12)])
def test_results_outlive_the_grid_that_built_them(other):
    first = _grid(20)
    want = _transform(first)
    second = _grid(20, **other)
    alone = _transform(second)
    first.close()
    third = _grid(20)
    for (s0, p0), (s1, p1) in ((alone, _transform(second)), (want, _transform(third))):
        assert np.array_equal(s0, s1) and np.array_equal(p0, p1)
    second.close(), third.close()


def test_threads_create_and_destroy_them():
    want = _transform(_grid(30))

    def work(i):
        g = _grid(30 if i % 2 else 17)
        out = _transform(g)
        g.close()
        return out

    with ThreadPoolExecutor(6) as pool:
        for i, (s, p) in enumerate(pool.map(work, range(24))):
            if i % 2:
                assert np.array_equal(s, want[0]) and np.array_equal(p, want[1])
