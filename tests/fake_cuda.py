"""The library's host code over a CUDA runtime without a GPU
(fakes/cudart.cpp), for tests of what it asks of the runtime. Kernels do
nothing there; memory is host memory, and a tensor or array on the host serves
where a device pointer is wanted."""

import ctypes
import functools
import pathlib
import shutil
import subprocess
import tempfile

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
PACKAGE = ROOT / "stable-fluids_b200"
CUDA = pathlib.Path("/usr/local/cuda")


@functools.lru_cache(maxsize=None)
def build():
    if not (shutil.which("nvcc") or (CUDA / "bin" / "nvcc").exists()):
        pytest.skip("no CUDA toolkit")
    subprocess.run(["make", "-s", "-j4", "-C", str(PACKAGE)], check=True, capture_output=True)
    sources = [*(PACKAGE / "csrc").glob("*.cu"), *(PACKAGE / "csrc").glob("*.cpp")]
    objects = [str(PACKAGE / "_build" / f"{p.stem}.o") for p in sorted(sources)]
    folder = tempfile.TemporaryDirectory(prefix="fake-cuda-")
    so = pathlib.Path(folder.name) / "libstable-fluids-fake.so"
    subprocess.run(["g++", "-std=c++20", "-O1", "-shared", "-fPIC", f"-I{CUDA / 'include'}", str(ROOT / "tests" / "fakes" / "cudart.cpp"), *objects, "-o", str(so), "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-ldl"], check=True)
    return so, folder


def load(sf, out):
    """The library on the fake runtime, as a process of its own would see it
    (nothing looked up yet); its fake_* functions are the tests' handles."""
    so, _ = build()
    lib = sf.load_library(shutil.copy(so, out))
    lib.fake_set_device.argtypes = [ctypes.c_int]
    lib.fake_executed_of.argtypes = [ctypes.c_char_p]
    lib.fake_patch_copies.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_uint]
    return lib


def create(sf, lib, n, options=None, iterations=(4, 6), scalars=1, walls=None):
    """A context of a plume on grid n; (result, handle)."""
    flow, scalar = walls if walls is not None else sf.scenes.stam_walls()
    cfg = sf.scenes.make_config(n, 1.0 / n[0], 0.1, 1e-4, *iterations, flow)
    s = (sf.ScalarFieldDesc * max(1, scalars))(*[sf.ScalarFieldDesc(diffusion=1e-5, dissipation=0.0, initial_value=0.0, boundary=scalar)] * scalars)
    v = (sf.VectorFieldDesc * 1)(sf.VectorFieldDesc(usage=sf.VECTOR_FIELD_FORCE, initial_value_x=0.0, initial_value_y=0.0, initial_value_z=0.0))
    desc = sf.ContextCreateDesc(config=cfg, stream=None, scalar_fields=ctypes.cast(s, ctypes.POINTER(sf.ScalarFieldDesc)), scalar_field_count=scalars, vector_fields=ctypes.cast(v, ctypes.POINTER(sf.VectorFieldDesc)), vector_field_count=1)
    ctx = ctypes.c_void_p()
    handles = (ctypes.c_uint32 * max(1, scalars))()
    rc = lib.stable_fluids_b200_create_context(ctypes.byref(desc), ctypes.byref(options) if options is not None else None, ctypes.byref(ctx), handles, scalars, (ctypes.c_uint32 * 1)(), 1)
    return rc, ctx
