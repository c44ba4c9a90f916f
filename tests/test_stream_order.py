"""What the network does on the default stream is in order with the passes on
the caller's streams, which do not wait for it: its buffers are cleared before
the first pass on them, and parameters are read and set when no step of the
optimizer is under way (a CUDA runtime without a GPU, fake_cuda.py, keeps the
account)."""

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


def test_parameters_after_a_training_step(sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    stream, net, count = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_uint64()
    assert lib.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
    lib.stable_fluids_b200_network_parameters(net, ctypes.byref(count), None)
    values = (ctypes.c_float * count.value)()
    n = (16, 12, 8)
    field = (ctypes.c_float * (n[0] * n[1] * n[2]))()
    for use in (lib.stable_fluids_b200_network_set_parameters, lambda h, v: lib.stable_fluids_b200_network_parameters(h, None, v)):
        assert lib.stable_fluids_b200_network_train_step(net, field, field, field, *n, 1.0, 1e-3, None, stream) == sf.RESULT_OK
        assert use(net, values) == sf.RESULT_OK
        assert lib.fake_unordered() == 0
    lib.stable_fluids_b200_network_destroy(net)
