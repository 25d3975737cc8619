"""The barriers of kernels whose warps share state, on the CPU: the kernels' text, cut out of its file, runs block by block
with any warp ahead of the others (tests/native/block_emulator.h). A result that depends on the order of the warps is a
missing barrier; on a GPU it would be a result that seldom repeats. Every comparison is of bits: the same operations on the
same values in every schedule."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "meteolab_gb300", "csrc")
from test_device_code_on_cpu import _cuda_include  # noqa: E402


def _excerpt(name, start, end):
    """The text of a source file from the line that begins with `start` up to the one that begins with `end`."""
    src = open(os.path.join(CSRC, name)).read()
    a = src.index("\n" + start) + 1
    return src[a:src.index("\n" + end, a) + 1]


def _compile(tmp, main, excerpts, **defines):
    for name, text in excerpts.items():
        (tmp / name).write_text(text)
    lib = tmp / (main + ".so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fno-ipa-reference", "-fPIC", "-shared", "-w", "-I", _cuda_include(),
                    "-I", os.path.join(HERE, "..", "include"), "-I", str(tmp), "-o", str(lib), os.path.join(HERE, "native", main + ".cpp")], check=True)
    return C.CDLL(str(lib))


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.fixture(scope="module")
def transport(tmp_path_factory):
    text = _excerpt("sg_transport.cu", "constexpr int TMAXC", "// MINB:")
    return _compile(tmp_path_factory.mktemp("transport"), "transport_block", {"transport_item.inc": text})


# kind 0 WENO, 1 dynamics; ragged tiles (13 x 11 columns on 8 x 8), slabs of five and six levels, the least the plan cuts,
# and of one
@pytest.mark.parametrize("kind,G,ew", [(1, 4, 0), (0, 3, 1), (0, 3, 0), (0, 1, 0)])
@pytest.mark.parametrize("nz,slabs", [(11, 2), (15, 3), (9, 9)])
def test_slabs_of_levels_give_the_whole_columns_bits_whichever_warp_is_ahead(transport, kind, G, ew, nz, slabs):
    nx, ny, fields = 13, 11, 13
    rng = np.random.default_rng(nz)
    n = nx * ny * nz
    start = rng.standard_normal(3 * fields * n).astype(np.float32)
    faces = rng.standard_normal(4 * n).astype(np.float32)
    lv = rng.uniform(.5, 1.5, 64 * nz).astype(np.float32)
    threads = 64 + (64 if ew else 0)

    def stage(slabs, order, late=0):
        fld = start.copy()
        assert transport.tb_transport(kind, G, ew, 8, 8, nx, ny, nz, slabs, order, late, 64 | 1, 1, 1, _fp(fld), _fp(faces), _fp(lv)) == 0
        return fld

    want = stage(1, 0)
    assert np.isfinite(want).all() and not np.array_equal(want, start)
    for order in range(2 + threads // 32):
        assert np.array_equal(stage(1, order), want), order
        assert np.array_equal(stage(slabs, order), want), order
        assert np.array_equal(stage(slabs, order, late=1), want), order


MAX_CHANNEL = 3000
GROW_WARPS = 4


def _growth(tmp, front):
    """The channel's growth with `front` links of its front in shared memory."""
    helpers = _excerpt("sg_lightning.cu", "constexpr double EPS0", "// Block sum in a fixed order")
    grow = _excerpt("sg_lightning.cu", "// The state record in shared memory", "// deposit() (:352-381)")
    for old, new in (("constexpr int FRONT = 5120", f"constexpr int FRONT = {front}"), ("extern __shared__ double fsm[];", "double* fsm = dynamic_shared.data();")):
        assert grow.count(old) == 1
        grow = grow.replace(old, new)
    return _compile(tmp, "lightning_block", {"lightning_helpers.inc": helpers, "lightning_grow.inc": grow})


@pytest.fixture(scope="module")
def growth(tmp_path_factory):
    return _growth(tmp_path_factory.mktemp("growth"), 5120)


def _flash(lib, seed, order, stages=3):
    """A flash in a storm of two charge layers, clear air around its cloud; later stages on a weakened, disturbed field."""
    nx, ny, nz = 14, 12, 16
    rng = np.random.default_rng(seed)
    zs = np.cumsum(rng.uniform(300, 500, nz)) - 300
    air = 1.2 * np.exp(-zs / 9000)
    z, y, x = np.meshgrid(zs / zs[-1], np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij")
    inside = np.exp(-((x - .5) ** 2 + (y - .5) ** 2) / .08)
    base = 4e8 * inside * np.sin(2 * np.pi * z) * (1 + .2 * rng.standard_normal((nz, ny, nx)))
    base[0] = base[-1] = 0
    phi = np.ascontiguousarray([base * f + 1e6 * rng.standard_normal(base.shape) * (z > 0) for f in np.linspace(1, .7, stages)])
    rho = np.where(inside > .15, 1e-9 * np.sin(2 * np.pi * z), 0.)
    cloudy = np.where(inside > .3, 1e-3, 0.).astype(np.float32)
    start = int(np.ravel_multi_index((nz // 4, ny // 2, nx // 2), (nz, ny, nx)))
    out, state = np.zeros(2 * MAX_CHANNEL, np.int32), np.zeros(7)
    dp = C.POINTER(C.c_double)
    lib.lb_flash.argtypes = [C.c_int] * 3 + [C.c_double] * 2 + [dp] * 4 + [C.POINTER(C.c_float), C.c_int, C.c_int, C.c_uint, C.c_int, C.POINTER(C.c_int), dp]
    d = lambda a: np.ascontiguousarray(a, float).ctypes.data_as(dp)  # noqa: E731
    largest = lib.lb_flash(nx, ny, nz, 1000., 900., d(zs), d(air), d(rho), d(phi), _fp(cloudy), stages, start, 1000 + seed, order,
                           out.ctypes.data_as(C.POINTER(C.c_int)), d(state))
    return largest, out, state


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_a_channel_grows_the_same_whichever_warp_is_ahead(growth, seed):
    largest, nodes, state = _flash(growth, seed, 0)
    assert largest > 128 and state[0] > 40, (largest, state)  # a front of several links a thread, a channel of many picks
    for order in range(1, 2 + GROW_WARPS):
        got = _flash(growth, seed, order)
        assert got[0] == largest and np.array_equal(got[1], nodes) and np.array_equal(got[2], state), order


@pytest.mark.parametrize("front", [64, 200])
def test_a_front_longer_than_shared_memory_grows_the_same_channel(growth, tmp_path, front):
    """Links past the front's part in shared memory live in the run's buffers: the same picks and the same channel."""
    lib = _growth(tmp_path, front)
    for seed in (1, 2, 3):
        largest, nodes, state = _flash(growth, seed, 0)
        assert largest > front
        for order in (0, 1, 3):
            got = _flash(lib, seed, order)
            assert got[0] == largest and np.array_equal(got[1], nodes) and np.array_equal(got[2], state), (seed, order)


def test_the_mean_potential_is_the_division_to_the_last_bit(growth):
    """Sums of any size over every count a channel may have, and sums next to those whose means are next to a midpoint."""
    rng = np.random.default_rng(5)
    n = 900 * MAX_CHANNEL
    sums = rng.standard_normal(n) * 10.0 ** rng.uniform(-30, 30, n)
    count = np.arange(n) % MAX_CHANNEL + 1
    half = n // 2
    mean = np.ldexp(np.round(np.ldexp(rng.uniform(1, 2, half), 52)) + .5, -52 + rng.integers(-40, 40, half))
    sums[:half] = np.nextafter(mean * count[:half], np.where(rng.random(half) < .5, np.inf, -np.inf))
    growth.lb_means.argtypes = [C.POINTER(C.c_double), C.c_int]
    assert growth.lb_means(sums.ctypes.data_as(C.POINTER(C.c_double)), n) == 0
