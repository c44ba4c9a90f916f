"""The network's buffers are cleared before the first pass on them starts,
whichever stream it runs on: nothing is launched on a stream of the caller's
while work on the default stream is under way (a CUDA runtime without a GPU,
fake_cuda.py, keeps the account)."""

import ctypes

from tests import fake_cuda


def test_first_pass_on_a_stream_of_the_callers(sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    stream, net = ctypes.c_void_p(), ctypes.c_void_p()
    assert lib.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
    assert lib.fake_unordered() == 0
    for n in ((16, 12, 8), (8, 8, 12)):
        field = (ctypes.c_float * (n[0] * n[1] * n[2]))()
        assert lib.stable_fluids_b200_network_predict(net, field, None, *n, 1.0, field, stream) == sf.RESULT_OK
        assert lib.stable_fluids_b200_network_gradients(net, field, field, field, *n, 1.0, None, None, stream) == sf.RESULT_OK
        assert lib.fake_unordered() == 0
    lib.stable_fluids_b200_network_destroy(net)


def test_first_step_of_a_learned_context(sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    net = ctypes.c_void_p()
    assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
    o = sf.default_options(lib)
    o.warm_start = sf.WARM_START_LEARNED
    rc, ctx = fake_cuda.create(sf, lib, (16, 12, 8), o)
    assert rc == sf.RESULT_OK
    assert lib.stable_fluids_b200_attach_network(ctx, net) == sf.RESULT_OK
    assert lib.stable_fluids_step_cuda(ctx) == sf.RESULT_OK
    assert lib.fake_unordered() == 0
    lib.stable_fluids_destroy_context_cuda(ctx)
    lib.stable_fluids_b200_network_destroy(net)
