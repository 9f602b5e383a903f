"""The shape of a per-pair gate/up launch, and what the context's settings do to it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("shape") / "decode_shape_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "moe4all_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "decode_shape_check.cpp"), "-o", exe], check=True)

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
