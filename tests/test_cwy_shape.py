"""The rows of an Arnoldi solve in one launch over blocks, warps and lanes
(cwy_shape.h), for every number of blocks a GPU may leave it."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "psfun_gb300" / "csrc"


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("shape")
    (d / "s.cpp").write_text(
        '#include "cwy_shape.h"\n'
        'extern "C" int max_rt() { return psf::kCwyMaxRt; }\n'
        'extern "C" void shape(long long n, int g, int* o) {\n'
        '  const psf::CwyShape s = psf::cwy_shape(n, g);\n'
        '  o[0] = s.G; o[1] = s.chunk; o[2] = s.rt; o[3] = s.threads;\n}\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(d / "s.so"), str(d / "s.cpp")],
                   check=True)
    lib = C.CDLL(str(d / "s.so"))

    def f(n, g):
        o = (C.c_int * 4)()
        lib.shape(C.c_longlong(n), g, o)
        return tuple(o)

    f.max_rt = lib.max_rt()
    return f


@pytest.mark.parametrize("blocks", [1, 2, 56, 116, 132, 136, 148, 152, 160])
def test_rows_are_covered(shape, blocks):
    for n in (1, 2, 63, 64, 65, 640, 641, 10000, 86387, 97281, 4096 * 127 + 1, 506881, 522240, 522241, 524287):
        G, chunk, rt, threads = shape(n, blocks)
        if G == 0:
            assert n > blocks * shape.max_rt * 640 - 2 * blocks
            continue
        assert 1 <= G <= blocks and 1 <= rt <= shape.max_rt and 32 <= threads <= 640
        assert (G - 1) * chunk < n <= G * chunk and chunk % 2 == 0
        groups = -(-chunk // (32 * rt))  # of 32 rt rows, a warp each
        assert groups * 32 * rt >= chunk and groups <= threads // 32
