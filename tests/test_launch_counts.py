"""The launch counts that the library reports are the launches it makes,
counted by a CUDA runtime without a GPU (fake_cuda.py)."""

import ctypes

import pytest

from tests import fake_cuda

N = (32, 24, 20)


def _counts(sf, lib, options, n=N, network=False):
    """(kernels_per_step, kernels in the step graph)"""
    rc, ctx = fake_cuda.create(sf, lib, n, options)
    assert rc == sf.RESULT_OK
    net = ctypes.c_void_p()
    if network:
        assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
        assert lib.stable_fluids_b200_attach_network(ctx, net) == sf.RESULT_OK
    info = sf.B200StepInfo()
    lib.stable_fluids_b200_get_step_info(ctx, ctypes.byref(info))
    before = lib.fake_executed()
    assert lib.stable_fluids_step_cuda(ctx) == sf.RESULT_OK
    executed = lib.fake_executed() - before
    lib.stable_fluids_destroy_context_cuda(ctx)
    if network:
        lib.stable_fluids_b200_network_destroy(net)
    return info.kernels_per_step, executed


@pytest.mark.parametrize("storage", ["STORAGE_FP32", "STORAGE_BF16"])
@pytest.mark.parametrize("per_pass", [0, 1, 2])
@pytest.mark.parametrize("scheme", ["SCHEME_RBGS", "SCHEME_JACOBI"])
@pytest.mark.parametrize("n", [N, (31, 24, 20), (104, 80, 66), (1040, 6, 4)], ids=lambda n: "x".join(map(str, n)))
def test_step_counts(n, scheme, per_pass, storage, sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    o = sf.default_options(lib)
    o.scheme, o.iterations_per_pass, o.storage, o.compute_residual = getattr(sf, scheme), per_pass, getattr(sf, storage), 1
    told, made = _counts(sf, lib, o, n)
    assert told == made


@pytest.mark.parametrize("coarse", [0, 1])
def test_learned_step_counts(coarse, sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    o = sf.default_options(lib)
    o.warm_start, o.warm_start_coarsening = sf.WARM_START_LEARNED, coarse
    told, made = _counts(sf, lib, o, (32, 24, 16), network=True)
    assert told == made
