"""The weight-gradient kernels by themselves (kernels/wgrad_check.cu), on grids
that fill no tile, chunk or segment."""

import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def check(tmp_path_factory, cuda):
    exe = tmp_path_factory.mktemp("wgrad") / "wgrad_check"
    subprocess.run([NVCC, "-std=c++20", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{ROOT / 'include'}", f"-I{ROOT / 'stable-fluids_b200' / 'csrc'}",
                    str(ROOT / "tests" / "kernels" / "wgrad_check.cu"), "-o", str(exe), "-ldl"], check=True, capture_output=True)

    def run(mode):
        r = subprocess.run([str(exe), mode], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout.splitlines()

    return run


def _differing(lines, layers):
    mine = [l for l in lines if l.split()[1].endswith(layers)]
    assert len(mine) >= 12
    return [l for l in mine if not l.endswith(" 0 differ")]


@pytest.mark.gpu
@pytest.mark.parametrize("layers", [("->16",), ("->32", "->64")], ids=["16 channels", "32 and 64 channels"])
def test_whole_numbers_sum_exactly(layers, check):
    assert _differing(check("exact"), layers) == []


@pytest.mark.gpu
def test_an_infinity_beside_a_segment(check):
    """16 channels: an infinity in the gradient is in the sums it belongs to and in
    no other; the zeros that stand for what is outside a segment must not meet it."""
    assert _differing(check("inf"), ("->16",)) == []


@pytest.mark.gpu
def test_an_infinity_at_the_last_column(check):
    """32 and 64 channels: an infinity among the activations beside voxels that a
    tile has past the grid, and in the gradient."""
    assert _differing(check("inf"), ("->32", "->64")) == []


@pytest.mark.gpu
def test_bias_sums_are_rounded_to_nearest(check):
    """64 x 32 x 64 voxels of positive gradients over twelve octaves. A lane adds at
    most 7 tiles x 16 rows x 8 values one after the other (32 channels: 74 CTAs
    for 256 tiles, half the rows a warp; 64: 37 CTAs, all rows), each
    rounded to nearest: an error of 0.29 ulp, independent, so that the largest of
    a layer's relative errors stays below 1e-6 (over 100 chains a sum, standard
    deviation some 1e-7). Sums rounded towards zero fall short by 5e-6 with 64
    channels. The chain kernel (16) adds 1640 values a lane in 10 chains."""
    worst = {int(l.split()[0]): float(l.split()[1]) for l in check("bias")}
    assert set(worst) == {16, 32, 64}
    assert all(e <= 1e-6 for e in worst.values()), worst
