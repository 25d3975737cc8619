"""Which solve a projection over terrain takes (GPU): the fast one while r . z0 stays below 1e-9, else the one in a fixed
order of operations, from the start again.

Tolerances. Both solves stop at 1e-6 of the first residual. Below the watch's 1e-9 rounding has not come to decide the
iterations: they stop after the same number, their FP64 pressures agree to 1e-9 of its norm and their FP32 winds to a
rounding each (6e-8). A solve that starts again is the ordered one's, bit for bit.
"""
import numpy as np
import pytest

from meteolab_gb300.grid import GridOptions, create_grid

pytestmark = pytest.mark.gpu
FAST, ORDERED = 1, 2


@pytest.fixture(scope="module")
def ctx():
    from meteolab_gb300 import build
    build.build()
    from meteolab_gb300.runtime import Context
    c = Context()
    yield c
    c.close()


def _case(ctx, shape, kind, height):
    from meteolab_gb300.runtime import MaskedProjection, terrain_heights
    nx, ny, nz = shape
    g = create_grid(GridOptions(nx, ny, nz, nx * 1200.0, ny * 1125.0, 18_900.0, 100.0))
    h = terrain_heights({"kind": kind, "height": height, "width": 5}, g)
    rho = 1.2 * np.exp(-np.asarray(g.zs) / 9000)
    rng = np.random.default_rng(nx)
    u = (10 + rng.normal(0, 2, g.n)).astype(np.float32)
    v, w = (rng.normal(0, s, g.n).astype(np.float32) for s in (2, 1))
    return MaskedProjection(ctx, g, rho, h), g, (u, v, w)


def _project(m, g, winds, force=0):
    out = [a.copy() for a in winds] + [np.zeros(g.layer * (g.nz - 1))]
    m.debug_route(force)
    m.project(*out[:3], 3.0, out[3])
    return out, m.debug_route(), m.iterations


def _rel(a, b):
    return np.linalg.norm(a.astype(float) - b) / np.linalg.norm(b.astype(float))


# the routes as measured: what sends a solve to the ordered one is a column whose open share of a cell layer is small, by
# where the ground happens to lie between the nodes, not the slope
@pytest.mark.parametrize("shape,kind,height,route", [((17, 13, 21), "hill", .4, FAST), ((32, 24, 30), "hill", .4, FAST),
                                                     ((40, 32, 33), "plateau", 1.0, FAST), ((16, 12, 20), "hill", .4, ORDERED),
                                                     ((30, 7, 25), "hill", 1.0, ORDERED), ((23, 24, 32), "plateau", 1.0, ORDERED)])
def test_the_ground_decides_which_solve_a_projection_takes(ctx, shape, kind, height, route):
    m, g, winds = _case(ctx, shape, kind, height)
    _, took, iterations = _project(m, g, winds)
    m.close()
    assert took == route and iterations > 1


def test_the_fast_solve_is_kept_only_where_the_two_agree(ctx):
    rng = np.random.default_rng(77)
    taken = {FAST: 0, ORDERED: 0}
    for _ in range(24):
        shape = tuple(int(k) for k in rng.integers((8, 6, 12), (48, 40, 51)))
        kind = ("hill", "ridge", "schar", "plateau")[rng.integers(4)]
        m, g, winds = _case(ctx, shape, kind, float(np.exp(rng.uniform(np.log(.1), np.log(2)))))
        got, route, n = _project(m, g, winds)
        ordered, _, k = _project(m, g, winds, ORDERED)
        m.close()
        taken[route] += 1
        if route == ORDERED:
            assert n == k and all(np.array_equal(a, b) for a, b in zip(got, ordered)), (shape, kind)
        else:
            assert n == k and _rel(got[3], ordered[3]) < 1e-9, (shape, kind)
            assert all(_rel(a, b) < 6e-8 for a, b in zip(got[:3], ordered[:3])), (shape, kind)
    assert taken[FAST] > 3 and taken[ORDERED] > 3, taken
