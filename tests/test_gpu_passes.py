"""Launch-by-launch passes: operands outside the range of the straight-line divisions
(each path against itself on scaled data), and the norm reduction beside the next
iteration."""
import numpy as np
import pytest

from conftest import make_case
from supersonicflowsolver_b200 import meshgen
from supersonicflowsolver_b200.psst import Grid, Solver

pytestmark = pytest.mark.gpu


def solve(tmp_path, m, scale, resident, n, **ckw):
    path, d, name = make_case(tmp_path, m, max_iter=n, mach=2.5, p=101325.0 * scale, **ckw)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = 64, 1
    s = Solver(g, sc)
    s.use_wavefront(resident)
    s.set_state(prim)
    linf, l2 = s.explicit_solve(n)
    out = s.get_state(with_w=True) + (linf, l2, s.get("dt"))
    nv = g.nvol
    s.close()
    return nv, out


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("ckw", [dict(flux=3, order=2, limiter=4, lc=1), dict(flux=2, order=1, lc=2), dict(flux=1, order=1, lc=1)],
                         ids=["hllc", "hll", "ausm"])
@pytest.mark.parametrize("e", [-80, -420, 90])
def test_scaled_pressure_scales_every_result_exactly(tmp_path, resident, dim, ckw, e):
    """Pressure times a power of two: density, momentum, energy and residuals scale by it, and
    temperature, velocity and time step stay -- in every bit, since the equations are
    homogeneous and no intermediate under- or overflows. 2^-80 takes the fluxes and 2^-420 also the
    RK update out of the straight-line operations' range (pressures 2^-60.., states 2^-400..)."""
    m = meshgen.wedge2d(24, 9, 12.0) if dim == 2 else meshgen.wedge3d(4, 3, 2, 12.0, tets=True)
    k = 2.0 ** e
    nv, a = solve(tmp_path, m, 1.0, resident, 5, **ckw)
    _, b = solve(tmp_path, m, k, resident, 5, **ckw)
    assert np.array_equal(a[0][:nv] * k, b[0][:nv])
    assert np.array_equal(a[0][nv:], b[0][nv:])
    for i in (1, 2, 3):
        assert np.array_equal(np.asarray(a[i]) * k, np.asarray(b[i])), i
    assert np.array_equal(a[4], b[4])
    assert np.abs(a[2]).max() > 0


@pytest.mark.parametrize("bits", [32, 64])
def test_norms_of_a_block_equal_those_of_single_iterations(tmp_path, bits):
    """72000 tets, so that the norm reduction runs on its own stream without a graph too."""
    m = meshgen.wedge3d(40, 20, 15, 12.0, tets=True)
    path, d, name = make_case(tmp_path, m, max_iter=4, mach=2.5, flux=3, order=2, limiter=5, lc=1)
    g = Grid.read_fluent(path)
    sc, prim = g.read_case(d, name)
    sc.precision, sc.lc1_mode = bits, 1
    rows = []
    for graphs in (True, False):
        for block in (4, 1):
            s = Solver(g, sc)
            s.use_graphs(graphs)
            s.set_state(prim)
            got = [s.explicit_solve(block) for _ in range(4 // block)]
            rows.append(np.concatenate([np.concatenate([a, b], axis=1) for a, b in got]))
            s.close()
    assert np.isfinite(rows[0]).all() and (rows[0][:, :5] > 0).any()
    for r in rows[1:]:
        assert np.array_equal(rows[0], r)
