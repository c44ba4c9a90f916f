"""A kernel whose bounded wait gives up sets an error word; the call that waits
for its results reports it. The word is set here on its way to the host (the
CUDA runtime without a GPU of fake_cuda.py), no kernel fails."""

import ctypes

from tests import fake_cuda

STATS_BYTES, STATS_ERROR = 72, 64  # sf_types.h: DeviceStats, its error word
LOSS_BYTES, LOSS_ERROR = 16, 8  # the loss sum and the network's error word


def test_step_stats_report_a_failed_wait(sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    rc, ctx = fake_cuda.create(sf, lib, (32, 24, 20))
    assert rc == sf.RESULT_OK
    stats = sf.B200StepStats()

    def step():
        assert lib.stable_fluids_step_cuda(ctx) == sf.RESULT_OK
        return lib.stable_fluids_b200_get_step_stats(ctx, ctypes.byref(stats))

    assert step() == sf.RESULT_OK and stats.pressure_iterations == 6
    lib.fake_patch_copies(STATS_BYTES, STATS_ERROR, 1)
    assert step() == sf.RESULT_BACKEND_FAILURE
    lib.fake_patch_copies(0, 0, 0)
    assert step() == sf.RESULT_OK
    lib.stable_fluids_destroy_context_cuda(ctx)


def test_gradients_report_a_failed_wait(sf, tmp_path):
    lib = fake_cuda.load(sf, tmp_path)
    n = (16, 12, 8)
    field = (ctypes.c_float * (n[0] * n[1] * n[2]))()
    net, loss = ctypes.c_void_p(), ctypes.c_double(-1.0)
    assert lib.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
    adam = lib.fake_executed_of(b"k_adam")

    def train():
        return lib.stable_fluids_b200_network_train_step(net, field, field, field, *n, 1.0, 1e-3, ctypes.byref(loss), None)

    lib.fake_patch_copies(LOSS_BYTES, LOSS_ERROR, 2)
    assert lib.stable_fluids_b200_network_gradients(net, field, field, field, *n, 1.0, ctypes.byref(loss), None, None) == sf.RESULT_BACKEND_FAILURE
    assert train() == sf.RESULT_BACKEND_FAILURE
    assert loss.value == -1.0 and lib.fake_executed_of(b"k_adam") == adam  # the parameters stay
    lib.fake_patch_copies(0, 0, 0)
    assert train() == sf.RESULT_OK
    assert loss.value == 0.0 and lib.fake_executed_of(b"k_adam") > adam
    lib.stable_fluids_b200_network_destroy(net)
