"""The masked projection's per-cell code compiled for the host: what it reads, and the quotient its ordered solve takes from
reciprocals."""
import ctypes as C

import numpy as np
import pytest

from test_block_schedules import _compile, _excerpt

DP = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def code(tmp_path_factory):
    flux = _excerpt("sg_masked.cu", "// The column fluxes of the node winds", "// What the iterations here take")
    quotient = _excerpt("sg_masked_ordered.cu", "__device__ __forceinline__ double quotient", "__device__ __forceinline__ double warp_sum")
    return _compile(tmp_path_factory.mktemp("terrain"), "terrain_code", {"masked_flux.inc": flux, "quotient.inc": quotient})


def test_winds_under_the_ground_stay_out_of_the_divergence(code):
    """A column without an open share of a cell layer takes no part in it (divergencePart, src/core/terrain.ts:240-264: the
    nodes there are not read), whatever the wind arrays hold there."""
    nx, ny, nz = 9, 7, 6
    layer, nc = nx * ny, nz - 1
    rng = np.random.default_rng(2)
    ground = rng.integers(0, 3, layer)  # shut cell layers of each column
    k = np.arange(nc)[:, None]
    A = np.where(k >= ground, rng.uniform(.1, .3, (nc, layer)), 0.)
    B = np.where(k >= ground, rng.uniform(.1, .3, (nc, layer)), 0.)
    A[k == ground] = 0  # the ground node is solid
    u, v, w = rng.standard_normal((3, nz, layer)).astype(np.float32)
    rho4, idz = rng.uniform(.2, .3, nz), rng.uniform(1e-3, 2e-3, nz)
    open_ = (B > 0).reshape(nc, ny, nx)
    dropped = np.ascontiguousarray(~(open_ | np.roll(open_, -1, 2) | np.roll(open_, -1, 1) | np.roll(open_, (-1, -1), (1, 2))), dtype=np.uint8)

    def divergence(u, v):
        out = np.zeros((nc, layer))
        f = lambda a: np.ascontiguousarray(a).ctypes.data_as(C.POINTER(C.c_float))  # noqa: E731
        d = lambda a: np.ascontiguousarray(a).ctypes.data_as(DP)  # noqa: E731
        code.tc_divergence(nx, ny, nz, C.c_double(1000), C.c_double(900), f(u), f(v), f(w), dropped.ctypes.data_as(C.POINTER(C.c_uint8)), d(A), d(B),
                           d(rho4), d(idz), d(out))
        return out

    buried = np.arange(nz)[:, None] < ground  # read by no open share
    want = divergence(np.where(buried, 0, u).astype(np.float32), np.where(buried, 0, v).astype(np.float32))
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    for junk in (np.nan, np.inf, 7e8):
        got = divergence(np.where(buried, junk, u).astype(np.float32), np.where(buried, junk, v).astype(np.float32))
        assert np.array_equal(got, want), junk


def test_quotients_from_reciprocals_are_the_division_to_the_last_bit(code):
    """x / d from 1 / d (Markstein 1990): the last bit of a division, over spacings, pivots and mode values of any size
    the solve meets, over quotients next to a half of the last place, and over divisors whose reciprocal rounds the worst
    (all bits set, and powers of two)."""
    rng = np.random.default_rng(11)
    n = 2_000_000
    x = rng.standard_normal(n) * 10.0 ** rng.uniform(-60, 60, n)
    d = rng.standard_normal(n) * 10.0 ** rng.uniform(-60, 60, n)
    third = n // 3
    # x the rounded product of d and a short number and its neighbours: quotients a hair off a double, or off a midpoint of two
    y = np.round(rng.uniform(1, 2, third) * 2.0 ** 26) / 2.0 ** 26 + rng.integers(-2, 3, third) * 2.0 ** -53
    x[:third] = np.nextafter(d[:third] * y, np.where(rng.random(third) < .5, np.inf, -np.inf))
    ones = np.ldexp(2 - 2.0 ** -52, rng.integers(-100, 100, third))
    d[third:2 * third] = np.where(rng.random(third) < .5, ones, np.ldexp(1.0, rng.integers(-100, 100, third)))
    edge = [(0., 3.), (-0., 3.), (1., 3.), (np.pi, -7.), (1., 2 - 2.0 ** -52), (2 - 2.0 ** -52, 1 + 2.0 ** -52)]
    x[-len(edge):], d[-len(edge):] = zip(*edge)
    dp = lambda a: a.ctypes.data_as(DP)  # noqa: E731
    assert code.tc_quotients(dp(x), dp(d), n, 0) == 0
    d[d > 0] *= -1
    assert code.tc_quotients(dp(x), dp(d), n, 1) == 0
