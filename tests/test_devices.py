"""Kernel attributes belong to a device: a program that uses the library on one
GPU and then on another gets the same on both. The devices are those of a CUDA
runtime without a GPU (fake_cuda.py), which refuses a launch that asks for more
shared memory or a larger cluster than its device has allowed for the kernel."""

import ctypes

import pytest

from tests import fake_cuda


@pytest.fixture
def fake(sf, tmp_path):
    return fake_cuda.load(sf, tmp_path)


def _step(sf, fake, n, scheme):
    o = sf.default_options(fake)
    o.scheme = scheme
    rc, ctx = fake_cuda.create(sf, fake, n, o)
    assert rc == sf.RESULT_OK
    info = sf.B200StepInfo()
    fake.stable_fluids_b200_get_step_info(ctx, info)
    assert fake.stable_fluids_step_cuda(ctx) == sf.RESULT_OK
    fake.stable_fluids_destroy_context_cuda(ctx)
    return info.kernels_per_step


@pytest.mark.parametrize("scheme", ["SCHEME_RBGS", "SCHEME_JACOBI"])
@pytest.mark.parametrize("n", [(32, 32, 32), (48, 40, 33)], ids=lambda n: "x".join(map(str, n)))
def test_small_contexts_on_a_second_device(n, scheme, sf, fake):
    counts = []
    for device in (0, 1, 0, 2):
        fake.fake_set_device(device)
        counts.append(_step(sf, fake, n, getattr(sf, scheme)))
    fake.fake_set_device(0)
    assert fake.fake_refused() == 0
    assert counts == counts[:1] * 4 and counts[0] <= 11  # the resident solves on each


def test_a_refused_cluster_launch_takes_the_sweeps(sf, fake):
    """Where the device says that a cluster fits and then does not take it, the
    solve runs as launches of one sweep."""
    fake.fake_take_clusters(0)
    assert _step(sf, fake, (40, 32, 24), sf.SCHEME_RBGS) > 11
    fake.fake_take_clusters(1)
    assert _step(sf, fake, (40, 32, 24), sf.SCHEME_RBGS) <= 11


def test_gradients_on_a_second_device(sf, fake):
    n = (16, 12, 8)
    field = (ctypes.c_float * (n[0] * n[1] * n[2]))()
    executed = []
    for device in (0, 1):
        fake.fake_set_device(device)
        net = ctypes.c_void_p()
        assert fake.stable_fluids_b200_network_create(1, ctypes.byref(net)) == sf.RESULT_OK
        before = fake.fake_executed()
        assert fake.stable_fluids_b200_network_gradients(net, field, field, field, *n, 1.0, None, None, None) == sf.RESULT_OK
        executed.append(fake.fake_executed() - before)
        fake.stable_fluids_b200_network_destroy(net)
    fake.fake_set_device(0)
    assert fake.fake_refused() == 0
    assert executed[0] == executed[1] > 0


@pytest.mark.parametrize("n", [(128, 24, 16), (72, 24, 16)], ids=["wavefront passes", "TMA passes"])
def test_blocked_passes_on_a_second_device(n, sf, fake):
    o = sf.default_options(fake)
    o.iterations_per_pass = 2
    for device in (0, 1):
        fake.fake_set_device(device)
        rc, ctx = fake_cuda.create(sf, fake, n, o)
        assert rc == sf.RESULT_OK
        fake.stable_fluids_destroy_context_cuda(ctx)
    fake.fake_set_device(0)
    assert fake.fake_refused() == 0
