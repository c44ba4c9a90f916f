"""The forms a solve takes by default (iterations_per_pass = 0) against one
launch per sweep or per colour on the interleaved field (iterations_per_pass
= 1), bit for bit, with the launch count telling which form ran:

- the colour-split layout, on grids a cluster's shared memory does not take
  (rows beyond 1024 cells, or more cells than it holds), at the edges of its
  shapes: colour rows of one float4, rows beyond a thread block, odd y and z,
  periodic axes down to two planes, every kind of face;
- solves resident in a cluster, in the forms whose bits are compared nowhere
  else: Jacobi sweeps, and BF16 storage with rows that are no whole number of
  float4s."""

import numpy as np
import pytest

from tests.golden import cases as C

DIFFUSE, PRESSURE = 4, 6
SOLVES = 5  # three velocity components, the pressure, the scalar


def _walls(sf, kind):
    sc = sf.scenes
    if kind == "stam":
        return sc.stam_walls()
    if kind == "benchmark":
        return sc.benchmark_walls()
    if kind == "periodic":
        return sc.flow_boundary([sf.FLOW_PERIODIC] * 6), sc.scalar_boundary([sf.SCALAR_PERIODIC] * 6)
    if kind == "periodic_y":  # moving x wall, outflow at a pressure, fixed scalars
        flow = [sf.FLOW_NO_SLIP_WALL, sf.FLOW_OUTFLOW, sf.FLOW_PERIODIC, sf.FLOW_PERIODIC, sf.FLOW_FREE_SLIP_WALL, sf.FLOW_NO_SLIP_WALL]
        scalar = [sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_PERIODIC, sf.SCALAR_PERIODIC, sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE]
        vel = [(0, 0.03, -0.01), (0, 0, 0), (0, 0, 0), (0, 0, 0), (0, 0, 0), (0.02, 0.01, 0)]
        return sc.flow_boundary(flow, vel, [0, 0.25, 0, 0, 0, 0]), sc.scalar_boundary(scalar, [0.25, 0, 0, 0, 0, 0.5])
    if kind == "mixed":  # no periodic axis; both ends of every axis differ
        flow = [sf.FLOW_OUTFLOW, sf.FLOW_NO_SLIP_WALL, sf.FLOW_NO_SLIP_WALL, sf.FLOW_OUTFLOW, sf.FLOW_OUTFLOW, sf.FLOW_FREE_SLIP_WALL]
        scalar = [sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE, sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX]
        vel = [(0, 0, 0), (0, -0.02, 0.01), (0.02, 0, -0.01), (0, 0, 0), (0, 0, 0), (0.01, 0.01, 0.01)]
        return sc.flow_boundary(flow, vel, [-0.1, 0, 0, 0.25, 0.125, 0]), sc.scalar_boundary(scalar, [0, 0.5, 0.25, 0, 0.75, 0])
    raise KeyError(kind)


def _scene(sf, n, walls):
    nx, ny, nz = n
    source = (nx / 2, 1 + min(ny, 8) / 2, nz / 2, 4.0, 10.0, 6.0)
    return sf.scenes.plume("default", n, dissipation=0.3, diffuse_iterations=DIFFUSE, pressure_iterations=PRESSURE, sources=[source], walls=_walls(sf, walls), velocity_seed=3, steps=2)


def _run(sf, lib, scene, per_pass, scheme, storage):
    o = sf.default_options(lib)
    o.scheme, o.storage, o.iterations_per_pass = scheme, storage, per_pass
    sim = sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib, options=o)
    sf.scenes.run(sim, scene)
    out = C.collect_outputs(sim, sf, C.Case(scene.name, scene.config, scene.scalars, scene.vectors, scene.steps))
    kernels = sim.info().kernels_per_step
    sim.close()
    return out, kernels


def _assert_same(got, want):
    for k in want:
        assert np.isfinite(want[k]).all() and np.abs(want[k]).max() > 0, k
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k


SPLIT = [
    ((8, 300, 240), "stam"), ((8, 300, 240), "mixed"), ((8, 300, 240), "periodic"),
    ((104, 80, 66), "benchmark"), ((104, 80, 66), "mixed"), ((104, 80, 66), "periodic_y"), ((104, 80, 66), "periodic"),
    ((16, 16400, 2), "periodic"), ((16, 16400, 2), "periodic_y"),
    ((1032, 2, 2), "periodic"), ((1032, 2, 2), "stam"), ((2048, 7, 5), "mixed"), ((1040, 7, 6), "benchmark"), ((1040, 6, 5), "periodic_y"), ((1040, 31, 1), "stam"),
]


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("n,walls", SPLIT, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_split_layout_matches_colour_launches(n, walls, storage, sf, lib, cuda):
    scene = _scene(sf, n, walls)
    bf16 = sf.STORAGE_BF16 if storage == "bf16" else sf.STORAGE_FP32
    split, kernels = _run(sf, lib, scene, 0, sf.SCHEME_RBGS, bf16)
    colours, colour_kernels = _run(sf, lib, scene, 1, sf.SCHEME_RBGS, bf16)
    # the split layout ran: a launch per colour, and two layout passes a solve
    # (the scalar's last one replaces the pass that scales it)
    assert kernels >= 2 * (4 * DIFFUSE + PRESSURE)
    assert kernels == colour_kernels + 2 * SOLVES - 1
    _assert_same(split, colours)


@pytest.mark.gpu
@pytest.mark.parametrize("n,walls", [((1040, 6, 4), "stam"), ((1040, 6, 4), "benchmark"), ((1040, 6, 4), "periodic"), ((1040, 6, 5), "periodic_y"), ((1040, 7, 5), "mixed"), ((104, 80, 66), "mixed")],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_split_layout_matches_oracle(n, walls, sf, lib, orc, cuda):
    scene = _scene(sf, n, walls)
    got, kernels = _run(sf, lib, scene, 0, sf.SCHEME_RBGS, sf.STORAGE_FP32)
    assert kernels >= 2 * (4 * DIFFUSE + PRESSURE)
    ref = orc.Oracle(scene.config, scene.scalars, scene.vectors, precision=32)
    sf.scenes.run(ref, scene)
    want = C.collect_oracle(ref, orc, C.Case(scene.name, scene.config, scene.scalars, scene.vectors, scene.steps))
    for k in want:
        assert np.array_equal(np.asarray(got[k], np.float32), np.asarray(want[k], np.float32)), k


RESIDENT = [((5, 4, 6), "mixed"), ((17, 9, 14), "mixed"), ((12, 30, 22), "benchmark"), ((33, 18, 12), "periodic_y"), ((32, 32, 32), "periodic"), ((30, 26, 40), "periodic"), ((100, 36, 44), "stam"), ((64, 40, 48), "mixed"), ((256, 12, 10), "benchmark")]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["jacobi-fp32", "jacobi-bf16", "rbgs-fp32", "rbgs-bf16"])
@pytest.mark.parametrize("n,walls", RESIDENT, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_resident_solves_match_sweeps(n, walls, form, sf, lib, cuda):
    scene = _scene(sf, n, walls)
    scheme = sf.SCHEME_JACOBI if form.startswith("jacobi") else sf.SCHEME_RBGS
    storage = sf.STORAGE_BF16 if form.endswith("bf16") else sf.STORAGE_FP32
    resident, kernels = _run(sf, lib, scene, 0, scheme, storage)
    sweeps, sweep_kernels = _run(sf, lib, scene, 1, scheme, storage)
    # the resident form ran: three launches for the five solves
    assert sweep_kernels - kernels >= 4 * DIFFUSE + PRESSURE - 3
    _assert_same(resident, sweeps)


@pytest.mark.gpu
@pytest.mark.parametrize("start", ["previous", "tolerance", "learned"])
@pytest.mark.parametrize("scheme", ["SCHEME_RBGS", "SCHEME_JACOBI"])
@pytest.mark.parametrize("n,walls", [((24, 20, 16), "stam"), ((28, 36, 20), "mixed"), ((20, 12, 8), "periodic"), ((34, 17, 12), "periodic_z"), ((31, 18, 14), "periodic_y")],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_resident_solves_from_other_starts(n, walls, scheme, start, sf, lib, cuda):
    """The pressure from the previous step's, in the intervals of a solve to a
    tolerance, and on both candidates of a learned start."""
    if start == "learned" and any(k % 4 for k in n):
        pytest.skip("the network takes grids of multiples of four")
    if walls == "periodic_z":
        sc = sf.scenes
        flow = [sf.FLOW_NO_SLIP_WALL, sf.FLOW_OUTFLOW, sf.FLOW_FREE_SLIP_WALL, sf.FLOW_NO_SLIP_WALL, sf.FLOW_PERIODIC, sf.FLOW_PERIODIC]
        scalar = [sf.SCALAR_FIXED_VALUE, sf.SCALAR_ZERO_FLUX, sf.SCALAR_ZERO_FLUX, sf.SCALAR_FIXED_VALUE, sf.SCALAR_PERIODIC, sf.SCALAR_PERIODIC]
        scene = _scene(sf, n, "stam")
        scene = sf.scenes.plume("default", n, diffuse_iterations=DIFFUSE, pressure_iterations=PRESSURE, sources=scene.meta["sources"], velocity_seed=3, steps=3,
                                walls=(sc.flow_boundary(flow, [(0, 0.03, -0.01)] + [(0, 0, 0)] * 5, [0, 0.25, 0, 0, 0, 0]), sc.scalar_boundary(scalar, [0.25, 0, 0, 0.5, 0, 0])))
    else:
        scene = _scene(sf, n, walls)
    got = []
    for per_pass in (0, 1):
        o = sf.default_options(lib)
        o.scheme, o.iterations_per_pass, o.compute_residual = getattr(sf, scheme), per_pass, 1
        o.warm_start = sf.WARM_START_LEARNED if start == "learned" else sf.WARM_START_PREVIOUS
        o.warm_start_trial_iterations = 3
        if start == "tolerance":
            o.residual_tolerance, o.residual_check_interval, o.max_pressure_iterations = 1e-4, 6, 60
        sim = sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib, options=o)
        if start == "learned":
            with sf.WarmStartNetwork(seed=3, lib=lib) as net:
                net.attach(sim)
                sf.scenes.run(sim, scene)
                out = C.collect_outputs(sim, sf, C.Case(scene.name, scene.config, scene.scalars, scene.vectors, scene.steps))
                stats = sim.stats()
                sf.WarmStartNetwork.detach(sim)
        else:
            sf.scenes.run(sim, scene)
            out = C.collect_outputs(sim, sf, C.Case(scene.name, scene.config, scene.scalars, scene.vectors, scene.steps))
            stats = sim.stats()
        got.append((out, stats, sim.info().kernels_per_step))
        sim.close()
    (a, sa, ka), (b, sb, kb) = got
    _assert_same(a, b)
    assert (sa.pressure_iterations, sa.hit_cap, sa.used_fallback) == (sb.pressure_iterations, sb.hit_cap, sb.used_fallback)
    # FP64 sums of squares of at most 20160 cells, in the order of their atomics
    assert abs(sa.rel_residual - sb.rel_residual) <= 20160 * 2.0**-53 * sb.rel_residual
    assert ka < kb
