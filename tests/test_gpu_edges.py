"""The kernels' edges (GPU): odd and prime transform lengths, the smallest and ragged grids, columns cut into slabs of
levels, node and sum chunks with remainders, the batch a run is in, and steep ground.

Tolerances. Two device results of the same run have to be the same bits. Against the FP64 oracle one step keeps the 1e-5
of the parity tests (FP32 storage and stencils). The FP64 field solves keep their own tests' bounds: transforms of length
n round to some log2(n) ulps and the column solves amplify that by their condition, below 1e-10 of the largest value; the
faces' conjugate gradients stop at 1e-10 of the right-hand side, so two of them agree to 1e-8; the projection's stop at
1e-6, so its fields agree to 1e-5.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))
import electric as E  # noqa: E402
import pyoracle as O  # noqa: E402
from parity import developed_state, field_errors, threads  # noqa: E402
from meteolab_gb300.grid import GridOptions, create_grid  # noqa: E402
from meteolab_gb300.scenarios import CARRIED, baseline_run  # noqa: E402

pytestmark = pytest.mark.gpu
DT = 3.0


@pytest.fixture(scope="module")
def ctx():
    from meteolab_gb300 import build
    build.build()
    from meteolab_gb300.runtime import Context
    c = Context()
    yield c
    c.close()


def _grid(nx, ny, nz):
    return create_grid(GridOptions(nx, ny, nz, nx * 1200.0, ny * 1125.0, 18_900.0, 100.0))


def _small_storm(nx, ny, nz, steps=60):
    return developed_state(baseline_run(_grid(nx, ny, nz), seed=nx + nz, bubble=4.0), steps)


# nx, ny: prime and composite transform lengths, single columns; nz: level counts about the slabs' eight levels, the
# sedimentation's eight slices and its four-level remainder, the sweeps' blocks of eight levels (nz and nz - 1 of them)
@pytest.mark.parametrize("shape", [(16, 12, 8), (17, 13, 9), (24, 10, 17), (31, 5, 16), (20, 18, 33), (45, 36, 24), (41, 33, 25)])
def test_a_step_on_ragged_grids_matches_the_oracle(ctx, shape):
    spec = _small_storm(*shape)
    o = O.OracleModel(spec, fp64=True, threads=threads())
    o.step(DT, 1)
    r = ctx.create(spec)
    r.step(1)
    errs = field_errors(r.read(), o.fields())
    r.retire()
    assert max(errs.values()) < 1e-5, errs


@pytest.mark.parametrize("shape", [(40, 32, 50), (17, 13, 16), (24, 20, 25), (33, 9, 128)])
def test_a_run_alone_and_in_batches_of_any_size_gives_the_same_bits(ctx, shape):
    """Alone its columns are cut into slabs and its pointwise items are small; batches of growing size cut them less and
    less, until they take whole columns."""
    specs = [baseline_run(_grid(*shape), seed=s, bubble=3.0) for s in (1, 2)]
    alone = ctx.create(specs[0])
    alone.step(3)
    want = alone.read()
    for count in (2, 9, 40):
        runs = [ctx.create(specs[k % 2]) for k in range(count)]
        ctx.batch_step(runs, 3)
        got = runs[(count - 1) // 2 * 2].read()
        assert all(np.array_equal(got[k], want[k]) for k in CARRIED), count
        for r in runs:
            r.retire()
    alone.retire()


@pytest.mark.parametrize("count,groups", [(4, 4), (9, 2)])
def test_pipelined_groups_give_the_bits_of_one_batch(ctx, count, groups):
    """The groups of the host round trips count one another's work when their items are made."""
    specs = [baseline_run(_grid(40, 32, 50), seed=20 + k, bubble=3.0) for k in range(count)]
    a, b = [ctx.create(s) for s in specs], [ctx.create(s) for s in specs]
    got = np.empty(sum(s.grid.n for s in specs) * len(CARRIED), np.float32)
    ctx.read_packed(a, got)
    want = got.copy()
    ctx.batch_round_trips(a, got, steps=2, groups=groups)
    for _ in range(2):
        ctx.write_packed(b, want)
        ctx.batch_step(b, 1)
        ctx.read_packed(b, want)
    assert np.array_equal(got, want)
    for r in a + b:
        r.retire()


# lengths of every radix and of primes, even and odd, of one point, and past one block's threads
@pytest.mark.parametrize("shape", [(1, 1, 4), (2, 3, 5), (8, 9, 6), (11, 13, 10), (25, 49, 7), (127, 2, 6), (3, 101, 5), (60, 84, 12), (300, 1, 4)])
def test_electric_potential_of_any_transform_length(ctx, shape):
    from meteolab_gb300.runtime import ElectricSolver
    nx, ny, nz = shape
    grid = create_grid(GridOptions(nx, ny, nz, nx * 900.0, ny * 1000.0, 4000.0, None))
    rho = np.random.default_rng(nx * 100 + ny).standard_normal(grid.n) * 1e-9
    s = ElectricSolver(ctx, grid)
    got, want = s.solve(rho), E.solve(grid, rho)
    s.close()
    assert np.max(np.abs(got - want)) <= 1e-10 * np.max(np.abs(want))


def _rel(a, b):
    return np.linalg.norm(np.asarray(a, float) - b) / max(np.linalg.norm(b), 1e-30)


# gentle ground takes the fast solves, a plateau's edge the ones in the reference's order of operations; odd and prime sides
@pytest.mark.parametrize("shape,kind,height", [((16, 12, 20), "hill", .4), ((17, 13, 21), "hill", .4), ((30, 7, 25), "hill", 1.0),
                                               ((23, 24, 32), "plateau", 1.0), ((40, 32, 33), "plateau", 1.0)])
def test_projection_and_faces_over_gentle_and_steep_ground(ctx, shape, kind, height):
    """The hill against the oracle. Over the plateau's edge the last bit decides the iterations, so there the projection is
    held to what it promises: the residual, and the divergence it leaves (the FP32 fields' rounding, below 1e-5)."""
    from meteolab_gb300.runtime import MaskedProjection, TerrainFaces, terrain_heights
    g = _grid(*shape)
    h = terrain_heights({"kind": kind, "height": height, "width": 5}, g)
    rho = 1.2 * np.exp(-np.asarray(g.zs) / 9000)
    rng = np.random.default_rng(shape[0])
    u = (10 + rng.normal(0, 2, g.n)).astype(np.float32)
    v, w = (rng.normal(0, s, g.n).astype(np.float32) for s in (2, 1))
    p0 = np.zeros(g.layer * (g.nz - 1))
    m = MaskedProjection(ctx, g, rho, h)
    got = [u.copy(), v.copy(), w.copy(), p0.copy()]
    m.project(*got[:3], DT, got[3])
    masked = [u.copy(), v.copy(), w.copy()]
    m.mask(*masked)
    before, after = (np.linalg.norm(m.divergence(*a)) for a in (masked, got[:3]))
    assert m.residual <= 1e-6 and after < 1e-5 * before
    if kind == "hill":
        for a, b in zip(got, O.masked_project(g, rho, h, u, v, w, DT, p0)[:4]):
            assert _rel(a, b) < 1e-5
    m.close()
    f = TerrainFaces(ctx, g, rho, h)
    mine, ref = f.set_velocity_masked(u, v, w), O.masked_faces(g, rho, h, u, v, w)
    f.close()
    for a, b in zip(mine[:3], ref[:3]):
        assert _rel(a, b) < 1e-8
