"""The all-FP64 simulation against the FP64 oracle, where the two must agree to
FP64 rounding: cell sizes that are and are not powers of two (the reference's
1/dx is an FP32 number, so that dx (1/dx) differs from 1 by up to 6e-8 on the
latter).

Tolerance: the two differ by the order of the grid sums and by contraction, some
1e-15 relative an operation.  A substep forms the stress from strains of 1e-3,
so that the 2e-16 of F = 1 + strain is 2e-13 of it, and 40 substeps add up 40 such
velocity changes: 1e-11 relative to the largest velocity."""

import numpy as np
import pytest

import molla_b200 as m
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DT = float(np.float32(1e-4))  # the oracle's scene holds dt in FP32


def config(grid, rheology, n):
    return m.MpmConfig(grid_size=grid, cell_size=1.0 / grid, grid_origin=(0.0, 0.0, 0.0), gravity_y=-9.8, youngs=5.0e5, poisson=0.2,
                       friction_angle=0.0, boundary_friction=0.2, particle_mass=2.0e-3, particle_volume=1.0e-6, max_particles=n,
                       rheology=rheology)


def run_both(engine, cfg, pts, substeps, dt=DT):
    sim = m.MpmSimulation64(engine, cfg)
    sim.set_particles(pts)
    sim.set_materials([cfg.rheology], np.zeros(len(pts), np.uint32))
    sim.step_n(dt, substeps)
    got = sim.read_state()
    faulted = sim.read_active_grid_status().numerical_fault
    sim.close()
    st = O.cast_state(O.init_state(pts.astype(np.float32), mass=cfg.particle_mass, volume=cfg.particle_volume), np.float64)
    O.step(O.make_scene(cfg, [cfg.rheology], dt, svd_tol=1e-14, svd_sweeps=30), st, substeps, precision="f64")
    return got, faulted, st


@pytest.mark.parametrize("rheology", ["Viscous", "Snow"])
@pytest.mark.parametrize("grid", [24, 32, 48, 70])
def test_all_fp64_matches_oracle_on_any_cell_size(engine, grid, rheology):
    n = 20_000
    cfg = config(grid, getattr(m.MpmRheology, rheology)(), n)
    lo, hi = [0.3, 2.0 / grid, 0.3], [0.6, 0.3, 0.6]  # on the floor, so that it is strained from the first substep on
    pts = np.random.default_rng(grid).uniform(lo, hi, size=(n, 3)).astype(np.float32).astype(np.float64)
    (pos, vel, F), faulted, st = run_both(engine, cfg, pts, 40)
    assert not faulted
    assert np.abs(st["F"] - np.eye(3).reshape(-1)).max() > 1e-4  # the stress acts
    assert np.abs(vel - st["vel"]).max() < 1e-11 * np.abs(st["vel"]).max()
    assert np.abs(pos - st["pos"]).max() < 1e-12


def test_new_particles_after_a_fault_see_no_old_velocity(engine):
    """A call whose gravity times dt overflows leaves infinite grid velocities and
    faults; a new particle half-way between nodes has a stencil node of weight zero
    that nothing is deposited to, with such a velocity on it."""
    cfg = config(32, m.MpmRheology.Viscous(), 4096)
    sim = m.MpmSimulation64(engine, cfg)
    sim.set_particles(np.random.default_rng(0).uniform(0.25, 0.5, size=(4096, 3)))
    sim.step_n(1.7e308, 1)
    assert sim.read_active_grid_status().numerical_fault
    x = np.array([[10.5 / 32, 12.5 / 32, 11.5 / 32]])
    sim.set_particles(x)
    sim.step_n(1e-4, 1)
    assert not sim.read_active_grid_status().numerical_fault
    pos, vel, _ = sim.read_state()
    gy = float(np.float32(-9.8))
    assert np.abs(vel - [[0.0, gy * 1e-4, 0.0]]).max() < 1e-15 and np.abs(pos - x - vel * 1e-4).max() < 1e-15
    sim.close()


@pytest.mark.parametrize("dt", [1e-4, 1e14, 1e26, 1e30])
def test_blown_up_deformation_is_clamped(engine, dt):
    """One substep of a huge dt deforms the particles whose stencil reaches the floor
    by -g dt^2 / dx along y (1e30, 1e54, 1e62): that value comes out at its clamp, 20,
    as the oracle's does (the other directions are rounding noise there).  1e-4
    reaches no clamp and is compared whole."""
    n = 4096
    dt = float(np.float32(dt))
    cfg = config(32, m.MpmRheology.Viscous(), n)
    lo, hi = [0.3, 2.0 / 32, 0.3], [0.6, 0.2, 0.6]
    pts = np.random.default_rng(3).uniform(lo, hi, size=(n, 3)).astype(np.float32).astype(np.float64)
    (_, _, F), faulted, st = run_both(engine, cfg, pts, 1, dt=dt)
    assert not faulted
    if dt < 1.0:
        assert np.abs(F - st["F"]).max() < 1e-12
        return
    floor = pts[:, 1] < 2.49 / 32
    for f in (F, st["F"]):
        assert np.abs(np.asarray(f)[floor, 4] + 20.0).max() < 1e-6


def test_overflowing_deformation_faults(engine):
    """F of 1e182, whose F^T F is not finite, faults."""
    cfg = config(32, m.MpmRheology.Viscous(), 64)
    sim = m.MpmSimulation64(engine, cfg)
    sim.set_particles(np.random.default_rng(4).uniform([0.3, 2.0 / 32, 0.3], [0.4, 0.1, 0.4], size=(64, 3)))
    sim.step_n(1e90, 1)
    assert sim.read_active_grid_status().numerical_fault
    sim.close()
