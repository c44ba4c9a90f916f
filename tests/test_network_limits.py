"""The network's kernels count voxels in 32 bits: a grid beyond that is refused
as out of memory, which it is on any device, before anything is launched (a
CUDA runtime without a GPU, fake_cuda.py, would hand out the memory)."""

import ctypes

import pytest

from tests import fake_cuda


@pytest.mark.parametrize("n", [(2048, 1024, 1024), (65536, 65536, 4)], ids=lambda n: "x".join(map(str, n)))
def test_grids_beyond_32_bits_are_refused(n, sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    net, p = ctypes.c_void_p(), ctypes.c_void_p(4096)
    assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
    before = lib.fake_executed()
    assert lib.stable_fluids_b200_network_gradients(net, p, p, p, *n, 1.0, None, None, None) == sf.RESULT_OUT_OF_MEMORY
    assert lib.stable_fluids_b200_network_predict(net, p, p, *n, 1.0, p, None) == sf.RESULT_OUT_OF_MEMORY
    assert lib.fake_executed() == before
    lib.stable_fluids_b200_network_destroy(net)
