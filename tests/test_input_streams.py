"""A field given as a device tensor is read on the simulation's stream: it has
to wait for the stream that the program computed it on. Checked without a
device, with stand-ins for torch's streams and tensors."""

import types


class Stream:
    def __init__(self):
        self.waited_for = []

    def wait_stream(self, other):
        self.waited_for.append(other)


class Tensor:
    device, dtype = "cuda:0", "float32"

    def is_contiguous(self):
        return True

    def numel(self):
        return 24

    def data_ptr(self):
        return 4096


def test_device_tensors_are_waited_for(sf):
    current = Stream()
    sim = object.__new__(sf.Simulation)
    sim._torch = types.SimpleNamespace(Tensor=Tensor, float32="float32", cuda=types.SimpleNamespace(current_stream=lambda device: current))
    sim.device, sim.cells, sim.stream, sim._keep = "cuda:0", 24, Stream(), []
    sim.lib = types.SimpleNamespace(stable_fluids_update_scalar_field_cuda=lambda *a: 0, stable_fluids_update_vector_field_cuda=lambda *a: 0, stable_fluids_destroy_context_cuda=lambda *a: 0)
    sim.ctx = None
    sim.set_scalar(1, Tensor())
    assert sim.stream.waited_for == [current]
    sim.set_vector(1, Tensor(), None, Tensor())
    assert sim.stream.waited_for == [current] * 3
    assert len(sim._keep) == 3
