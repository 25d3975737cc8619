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

    def stage(slabs, order):
        fld = start.copy()
        assert transport.tb_transport(kind, G, ew, 8, 8, nx, ny, nz, slabs, order, 64 | 1, 1, 1, _fp(fld), _fp(faces), _fp(lv)) == 0
        return fld

    want = stage(1, 0)
    assert np.isfinite(want).all() and not np.array_equal(want, start)
    for order in range(2 + threads // 32):
        assert np.array_equal(stage(1, order), want), order
        assert np.array_equal(stage(slabs, order), want), order
