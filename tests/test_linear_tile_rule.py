"""The rule that names the tile of a linear of many rows, asked on the host for 148 SMs: which cases of the GPU tests reach which tile, and the switch that keeps pairs out."""
import ctypes as C
import os
import subprocess
import sys

import pytest

import test_linear_many_rows_gpu as many
import test_linear_pair_widths_gpu as widths


@pytest.fixture(scope="module")
def tile(pkg):
    f = C.CDLL(pkg.lib_path())["_ZN4b20011linear_tileEiiibbi"]
    f.restype, f.argtypes = C.c_int, [C.c_int] * 3 + [C.c_bool] * 2 + [C.c_int]
    return lambda M, N, K, gated, f32: f(M, N, K, gated, f32, 148)


def cases(test):
    return [m.args[1] for m in test.pytestmark if m.name == "parametrize" and m.args[0].startswith("M,N,K")][0]


def test_the_gpu_tests_reach_every_tile(tile):
    plain = {tile(*c[:3], False, f32) for c in cases(many.test_plain) for f32 in (False, True)} | {tile(*c[:3], False, c[3]) for c in cases(widths.test_plain)}
    gated = {tile(*c[:3], True, f32) for c in cases(many.test_gated) for f32 in (False, True)} | {tile(*c[:3], True, c[3]) for c in cases(widths.test_gated)}
    assert plain == {64, 128, 256, -128, -160, -192, -224, -256}
    assert gated == {256, -128, -160, -192, -224, -256}


def test_narrow_outputs_stay_on_one_cta(tile):
    assert all(tile(M, N, K, False, f32) > 0 for M in (257, 1000, 5000) for N in (24, 100, 255) for K in (64, 4096) for f32 in (False, True))


def test_the_switch_keeps_pairs_out(tile):
    shapes = [(M, N, K, g) for M in (300, 1522, 8192) for N in (1024, 2048, 12288) for K in (1024, 4096) for g in (False, True)]
    assert any(tile(*s, False) < 0 for s in shapes)
    code = ("import ctypes as C, sys\nf = C.CDLL(sys.argv[1])['_ZN4b20011linear_tileEiiibbi']\nf.argtypes = [C.c_int] * 3 + [C.c_bool] * 2 + [C.c_int]\n"
            "assert all(f(*s, False, 148) > 0 for s in %r)" % (shapes,))
    lib = sys.modules["llm_inference_b200"].lib_path()
    subprocess.run([sys.executable, "-c", code, lib], check=True, env=dict(os.environ, B200_GEMM_PAIR="0"))


@pytest.mark.parametrize("M,N,K,gated,want", [
    (4096, 4096, 11008, False, -256), (6000, 4096, 4096, False, -256), (4096, 2048, 8192, False, -256), (2048, 4096, 11008, False, -256), (8192, 11008, 4096, True, -256),   # at the power limit
    (2048, 12288, 4096, False, -224), (3000, 2048, 5504, False, -192), (1522, 2048, 8192, False, -192), (1024, 1024, 1024, False, 64),                                      # 8 % cheaper, or too short for it
    (4096, 1000, 1032, False, -256), (8192, 1000, 1032, False, -256), (4096, 1024, 1024, False, 256), (3000, 264, 136, False, 64)])                                          # rows that end inside 64 columns
def test_beyond_the_fitted_sizes(tile, M, N, K, gated, want):
    assert tile(M, N, K, gated, False) == want
