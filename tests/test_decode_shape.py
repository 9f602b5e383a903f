"""The shapes of the per-pair kernels' launches, and what the context's settings do to it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("shape") / "decode_shape_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "moe4all_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "decode_shape_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.fixture(scope="module")
def shape(exe):
    def run(ne, nff, sh_ff, rows, used, warps, chunks, q5k=False):
        args = [exe, ne, nff, sh_ff, rows, used, 176 if q5k else 144, int(q5k), 148, warps, chunks]
        return tuple(int(v) for v in subprocess.run([str(a) for a in args], check=True, capture_output=True, text=True).stdout.split())

    return run


# one-wave shape 16 x 2: 16 CTAs per 512-wide expert; 148 SMs, so five rows of nine experts are the first past four waves
@pytest.mark.parametrize("warps,chunks", [(0, 0), (0, 4), (4, 0)])
@pytest.mark.parametrize("ne", [2048, 3072])
def test_zero_keeps_the_one_wave_shape(shape, warps, chunks, ne):
    assert shape(ne, 512, 512, 5, 8, warps, chunks) == (16, 2, 5 * 9 * 16)


@pytest.mark.parametrize("warps,chunks", [(4, 4), (8, 4), (16, 1)])
def test_named_shape(shape, warps, chunks):
    assert shape(2048, 512, 512, 5, 8, warps, chunks) == (warps, chunks, 5 * 9 * 512 // (warps * chunks))


def test_named_shape_that_does_not_fit(shape):
    # four warps do not stage 3072 activations, three do not divide 512 rows: 8 x 2 and 4 x 2, as on grids of two to four waves
    assert shape(3072, 512, 512, 5, 8, 4, 4) == (8, 2, 5 * 9 * 32)
    assert shape(2048, 512, 512, 5, 8, 3, 4) == (4, 2, 5 * 9 * 64)


@pytest.mark.parametrize("setting", [(4, 4), (0, 0), (16, 2)])
def test_up_to_four_waves_the_setting_is_not_read(shape, setting):
    assert shape(2048, 512, 512, 4, 8, *setting) == (4, 2, 4 * 9 * 64)  # 576 CTAs of 16 x 2: 3.9 waves
    assert shape(2048, 512, 512, 2, 8, *setting) == (8, 2, 2 * 9 * 32)  # 1.9
    assert shape(2048, 512, 512, 1, 8, *setting) == (16, 2, 9 * 16)     # one
    assert shape(1024, 256, 0, 1, 4, *setting) == (16, 1, 4 * 16)       # half of one
    assert shape(1024, 256, 0, 1, 4, *setting, q5k=True) == (16, 2, 4 * 8)


# the count of warps that a sweep of the launches found best or next to it, and the one before it in brackets
@pytest.mark.parametrize("ctas,tasks,fit,q4k,want", [
    (160, 14, 2, 0, 14), (480, 14, 2, 0, 14),                        # two CTAs of 114 KB to an SM (24)
    (1024, 14, 5, 1, 7), (1536, 16, 4, 1, 8), (1280, 14, 2, 1, 12),  # past four waves, light tasks (12); two CTAs
    (1280, 14, 2, 0, 12), (888, 16, 2, 0, 12),                       # heavy ones
    (512, 16, 3, 1, 16),                                             # two CTAs take as many waves as three (8)
    (384, 18, 4, 0, 12), (384, 18, 4, 1, 12), (512, 18, 4, 1, 9), (128, 16, 2, 0, 20), (448, 18, 1, 0, 24), (4096, 18, 4, 0, 9)])
def test_down_warps(exe, ctas, tasks, fit, q4k, want):
    out = subprocess.run([exe] + [str(v) for v in (ctas, tasks, fit, q4k, 148, 12)], check=True, capture_output=True, text=True).stdout
    assert int(out) == want


@pytest.mark.parametrize("cap", [0, 1, 5, 12, 24])
def test_down_warps_within_a_launch(exe, cap):
    for ctas in (1, 149, 300, 600, 5000):
        for tasks in (1, 2, 7, 14, 18, 66):
            for fit in (1, 2, 3, 6):
                n = int(subprocess.run([exe] + [str(v) for v in (ctas, tasks, fit, tasks % 2, 148, cap)], check=True, capture_output=True, text=True).stdout)
                assert 1 <= n <= 24
