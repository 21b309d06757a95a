"""Fused or tiled step of 1D batches (csrc/tile_plan.h lines_on_the_tiled_path), on the host: a function of the
batch's sizes and the device, not of the memory that is free, on either side of every line of it."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
GB = 1 << 30


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tile") / "libtile.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-w",
                    "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(HERE, "tile_harness.cpp"), "-o", so], check=True)
    return C.CDLL(so)


# precision, rule, sites of a line, components, chains, imaginary times -> tiled
@pytest.mark.parametrize("fp64,ref,ln,nc,chains,nt,tiled", [
    (1, 1, 64, 4, 40, 64, 1), (1, 1, 64, 4, 8, 64, 0), (1, 1, 256, 4, 120, 100, 1), (1, 1, 128, 4, 120, 100, 0),
    (1, 0, 64, 3, 40, 64, 1), (1, 0, 256, 3, 40, 64, 0), (0, 1, 64, 4, 3, 32, 1), (0, 1, 256, 4, 1, 32, 0),
    (0, 0, 64, 3, 120, 100, 1), (0, 0, 64, 3, 40, 64, 0), (0, 0, 256, 3, 256, 128, 0),
    # one chain of a field of more than a 64th of the memory: fused, but for the reference model at FP64
    (0, 1, 256, 4, 1, 400000, 1), (0, 1, 256, 4, 1, 800000, 0), (0, 1, 256, 4, 2, 800000, 1), (1, 1, 256, 4, 1, 800000, 1),
    (1, 0, 64, 3, 1, 2000000, 0), (1, 0, 64, 3, 1, 1000000, 1)])
def test_path_of_a_batch(lib, fp64, ref, ln, nc, chains, nt, tiled):
    assert lib.line_path(fp64, ref, ln, nc, chains, nt, C.c_longlong(277 * GB)) == tiled

