"""BF16 storage in the vectorised stencils, at the edges of their shapes: one
group of four a row, rows that are no multiple of four (the general kernel),
rows beyond a warp, planes beyond a z chunk."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("periodic_z", [False, True])
@pytest.mark.parametrize("n", [(4, 6, 5), (6, 5, 4), (36, 7, 10), (140, 18, 33), (96, 80, 70)], ids=lambda n: "x".join(map(str, n)))
def test_divergence_and_magnitude_of_bf16_velocity(n, periodic_z, sf, lib, cuda):
    """Both are formed in FP32 from the stored values: four roundings for the
    divergence of terms below 2 max|u| / 2h each, four for the magnitude."""
    sc = sf.scenes
    wall, per = sf.FLOW_NO_SLIP_WALL, sf.FLOW_PERIODIC
    flow = sc.flow_boundary([wall] * 4 + [per if periodic_z else wall] * 2, velocities=[(0, 0, 0)] * 6, pressures=[0] * 6)
    sper = sf.SCALAR_PERIODIC if periodic_z else sf.SCALAR_ZERO_FLUX
    scalar = sc.scalar_boundary([sf.SCALAR_ZERO_FLUX] * 4 + [sper] * 2, values=[0] * 6)
    scene = sc.plume("bf16", n, diffuse_iterations=2, pressure_iterations=4, walls=(flow, scalar), velocity_seed=5, steps=1)
    o = sf.default_options(lib)
    o.storage = sf.STORAGE_BF16
    sim = sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib, options=o)
    sf.scenes.run(sim, scene)
    u = np.stack(sim.fetch(sf.VIEW_FLOW_VELOCITY)).astype(np.float64)
    div, mag = sim.fetch(sf.VIEW_FLOW_DIVERGENCE), sim.fetch(sf.VIEW_FLOW_VELOCITY_MAGNITUDE)
    h = scene.config.cell_size
    sim.close()

    def central(c, axis, wrap):
        lo, hi = np.roll(c, 1, axis), np.roll(c, -1, axis)
        if not wrap:  # the wall value is zero: the ghost mirrors the face cell
            first, last = [slice(None)] * 3, [slice(None)] * 3
            first[axis], last[axis] = 0, -1
            lo[tuple(first)], hi[tuple(last)] = -c[tuple(first)], -c[tuple(last)]
        return (hi - lo) / (2 * h)

    want = central(u[0], 2, False) + central(u[1], 1, False) + central(u[2], 0, periodic_z)
    top = np.abs(u).max()
    assert top > 0
    assert np.abs(div - want).max() <= 3 * 4 * 2.0**-24 * 2 * top / (2 * h)
    assert np.abs(mag - np.sqrt((u**2).sum(0))).max() <= 4 * 2.0**-24 * np.sqrt(3) * top


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(104, 80, 66), (8, 300, 240)], ids=lambda n: "x".join(map(str, n)))
def test_bf16_half_sweeps_over_the_whole_range(n, sf, lib, cuda):
    """The split layout's packed sums and quotients give the colour launches'
    bits (iterations_per_pass 1) from the subnormals to the largest values,
    zeros and infinities among them."""
    rng = np.random.default_rng(2)
    shape = n[::-1]
    exponent = rng.integers(-133, 126, (shape[0], shape[1] // 4, 1)).repeat(4, axis=1)
    with np.errstate(over="ignore"):
        b = np.ldexp(rng.standard_normal(shape), exponent).astype(np.float32)
    b[: shape[0] // 4][rng.random((shape[0] // 4,) + shape[1:]) < 0.7] = 0
    b[-2, 3, 5] = np.inf
    scene = sf.scenes.plume("bf16", n, diffuse_iterations=3, pressure_iterations=2, walls=sf.scenes.stam_walls(), velocity_seed=3, steps=1)
    got = []
    for per_pass in (0, 1):
        o = sf.default_options(lib)
        o.storage, o.iterations_per_pass = sf.STORAGE_BF16, per_pass
        sim = sf.Simulation(scene.config, scene.scalars, scene.vectors, lib=lib, options=o)
        sim.set_scalar(1, b)
        sim.step(1)
        got.append([sim.fetch(sf.VIEW_SCALAR_FIELD_DATA, 1), *sim.fetch(sf.VIEW_FLOW_VELOCITY)])
        sim.close()
    for a, c in zip(*got):
        m = np.isfinite(c)
        assert m.any() and np.array_equal(np.isfinite(a), m) and np.array_equal(a[m], c[m])
    assert not np.isfinite(got[0][0]).all()
