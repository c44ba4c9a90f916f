"""A cell's index has 32 bits: grids of 2^32 cells and more are refused as out
of memory, which they are on a device of 180 GB, even where the memory could be
had (a CUDA runtime without a GPU, fake_cuda.py, hands out any amount)."""

import pytest

from tests import fake_cuda


@pytest.mark.parametrize("storage", ["STORAGE_FP32", "STORAGE_BF16"])
@pytest.mark.parametrize("n,fits", [((2048, 2048, 1024), False), ((65536, 65536, 1), False), ((2147483647, 2147483647, 2147483647), False), ((2048, 2048, 1023), True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_cells_are_counted_in_32_bits(n, fits, storage, sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    o = sf.default_options(lib)
    o.storage = getattr(sf, storage)
    rc, ctx = fake_cuda.create(sf, lib, n, o)
    assert rc == (sf.RESULT_OK if fits else sf.RESULT_OUT_OF_MEMORY)
    assert bool(ctx.value) == fits
    lib.stable_fluids_destroy_context_cuda(ctx)
