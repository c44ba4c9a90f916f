"""Whole solves held in a cluster's shared memory (sf_resident.cu), at the edges
of their shapes: rows of less than one float4 of a colour, odd rows, blocks of
one row, grids that need one CTA and grids that need sixteen, every kind of
face and periodic axes. The reference is the CPU oracle: its FP32 arithmetic is
the library's, so red-black results are bit-equal; Jacobi's are the oracle's
to one rounding a sweep. The update's division is checked on the CPU."""

import ctypes
import subprocess

import numpy as np
import pytest

from tests.golden import cases as C

GRIDS = [(1, 6, 4), (2, 2, 2), (5, 4, 6), (8, 2, 2), (17, 9, 14), (33, 18, 12), (12, 30, 22), (64, 64, 64), (100, 36, 44), (181, 47, 29), (256, 12, 10), (7, 100, 2)]


def _scene(sf, n, walls):
    sc = sf.scenes
    if walls == "mixed":
        flow = sc.flow_boundary([sf.FLOW_NO_SLIP_WALL, sf.FLOW_OUTFLOW, sf.FLOW_NO_SLIP_WALL, sf.FLOW_FREE_SLIP_WALL, sf.FLOW_PERIODIC, sf.FLOW_PERIODIC],
                                velocities=[(0, 0, 0), (0, 0, 0), (0.02, 0, -0.01), (0, 0, 0), (0, 0, 0), (0, 0, 0)], pressures=[0, 0.25, 0, 0, 0, 0])
        scalar = sc.scalar_boundary([sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_PERIODIC, sf.SCALAR_PERIODIC], values=[0.25, 0, 0.5, 0, 0, 0])
        w = (flow, scalar)
    else:
        w = sc.stam_walls() if walls == "stam" else sc.benchmark_walls()
    nx, ny, nz = n
    return sc.plume("resident", n, dissipation=0.3, diffuse_iterations=4, pressure_iterations=6, sources=[(nx / 2, 1 + min(ny, 8) / 2, nz / 2, 2.0, 10.0, 6.0)], walls=w, velocity_seed=3, steps=2)


@pytest.mark.gpu
@pytest.mark.parametrize("walls", ["stam", "benchmark", "mixed"])
@pytest.mark.parametrize("n", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_resident_solves_match_oracle(n, walls, sf, lib, orc, cuda):
    if (walls == "benchmark" and (n[0] % 2 or n[2] % 2)) or (walls == "mixed" and n[2] % 2):
        pytest.skip("an odd periodic side has no red-black colouring")
    scene = _scene(sf, n, walls)
    case = C.Case("resident", scene.config, scene.scalars, scene.vectors, scene.steps)
    for scheme in (sf.SCHEME_RBGS, sf.SCHEME_JACOBI):
        o = sf.default_options(lib)
        o.scheme = scheme
        sim = sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib, options=o)
        sf.scenes.run(sim, scene)
        got = C.collect_outputs(sim, sf, case)
        if scheme == sf.SCHEME_RBGS:  # every solve of the step one launch (Jacobi keeps two iterates: the two largest grids do not fit)
            assert sim.info().kernels_per_step <= 11
        sim.close()
        ref = orc.Oracle(scene.config, scene.scalars, scene.vectors, precision=32, scheme=scheme)
        sf.scenes.run(ref, scene)
        want = C.collect_oracle(ref, orc, case)
        for k in want:
            if scheme == sf.SCHEME_RBGS:
                assert np.array_equal(np.asarray(got[k], np.float32), np.asarray(want[k], np.float32)), k
            else:
                assert C.max_rel_err(got[k], want[k], 1e-3) <= 1e-5, k


@pytest.mark.gpu
def test_resident_solve_of_a_diverged_field(sf, lib, orc, cuda):
    """Infinities and NaN stay where a half-sweep carries them: the cells that
    are not finite are the oracle's."""
    scene = _scene(sf, (32, 24, 20), "stam")
    rng = np.random.default_rng(0)
    b = rng.standard_normal((20, 24, 32)).astype(np.float32)
    b[3, 4, 5], b[10, 11, 12] = np.inf, np.nan
    got = []
    for make in (lambda: sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib), lambda: orc.Oracle(scene.config, scene.scalars, scene.vectors, precision=32)):
        s = make()
        s.set_scalar(1, b)
        s.step(1)
        got.append(s.fetch(sf.VIEW_SCALAR_FIELD_DATA, 1) if hasattr(s, "ctx") else s.get(orc.SCALAR, 1))
        s.close()
    assert np.array_equal(np.isfinite(got[0]), np.isfinite(got[1]))
    m = np.isfinite(got[0])
    assert m.any() and not m.all() and np.array_equal(got[0][m], got[1][m])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(32, 24, 20), (104, 80, 66)], ids=["resident", "split layout"])
def test_quotients_over_the_whole_range(n, sf, lib, orc, cuda):
    """The FP32 quotient and the FP64 one behind it meet in one row: values from
    the subnormals to the largest, zeros, infinities and NaN, bit for bit the
    oracle's wherever that is finite."""
    scene = _scene(sf, n, "stam")
    rng = np.random.default_rng(1)
    shape = n[::-1]
    exponent = rng.integers(-149, 127, (shape[0], shape[1] // 4, 1)).repeat(4, axis=1)
    b = np.ldexp(rng.standard_normal(shape), exponent).astype(np.float32)
    b[: shape[0] // 4][rng.random((shape[0] // 4,) + shape[1:]) < 0.7] = 0
    b[-2, 3, 5], b[-3, 11, 12] = np.inf, np.nan
    got = []
    for make in (lambda: sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib), lambda: orc.Oracle(scene.config, scene.scalars, scene.vectors, precision=32)):
        s = make()
        s.set_scalar(1, b)
        s.step(1)
        got.append(s.fetch(sf.VIEW_SCALAR_FIELD_DATA, 1) if hasattr(s, "ctx") else s.get(orc.SCALAR, 1))
        s.close()
    m = np.isfinite(got[1])
    assert m.any() and not m.all() and np.array_equal(np.isfinite(got[0]), m)
    assert np.array_equal(got[0][m], got[1][m])


def test_one_correction_divides_by_six(tmp_path):
    """RN32(n / 6) by one correction of n RN32(1 / 6), two for other divisors,
    for every significand of n (both parities of the exponent)."""
    src = tmp_path / "division.c"
    src.write_text("""
#include <math.h>
#include <stdint.h>
#include <string.h>
long wrong(float d, int corrections) {
    const float y = (float)(1.0 / (double)d);
    long bad = 0;
    for (uint32_t m = 0; m < (1u << 24); ++m) {
        uint32_t u = (127u << 23) + m;
        float n;
        memcpy(&n, &u, 4);
        float q = n * y;
        for (int k = 0; k < corrections; ++k) q = fmaf(fmaf(-q, d, n), y, q);
        bad += q != n / d;
    }
    return bad;
}
""")
    so = tmp_path / "division.so"
    subprocess.run(["g++", "-x", "c", "-O2", "-march=x86-64-v3", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(src), "-lm"], check=True)
    lib = ctypes.CDLL(str(so))
    lib.wrong.argtypes, lib.wrong.restype = [ctypes.c_float, ctypes.c_int], ctypes.c_long
    assert lib.wrong(6.0, 1) == 0
    for d in (1.0006, 1.06, 1.5, 1.9999999, 3.22, 4.9, 7.3, 96.7):
        assert lib.wrong(d, 2) == 0, d
