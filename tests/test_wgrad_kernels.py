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
