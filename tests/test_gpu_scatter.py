"""The scatter's edges against the oracle: item sizes around the CTA's rounds
and the record stage, particles that left their tile's own cells since the
regrouping (margin cells) or the 8^3 block (direct deposits), and grids whose
dx is not a power of two, where a position within rounding of a cell face must
be regrouped under the same cell it is deposited from (the fixed-order P2G
stops with a fault bit otherwise).

Tolerance: one node sums the FP32 contributions of at most 27 cells of
particles; n terms of one sign differ by at most n ulps from the oracle's sum,
so mass is compared at n * 2^-23 relative to the largest node."""

import numpy as np
import pytest

import molla_b200 as m
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def config(grid, n, dx=None):
    return m.MpmConfig(grid_size=grid, cell_size=dx or 1.0 / grid, grid_origin=(0.0, 0.0, 0.0), gravity_y=-9.8, youngs=1.0e4, poisson=0.2,
                       friction_angle=0.0, boundary_friction=0.0, particle_mass=2.0e-3, particle_volume=1.0e-6, max_particles=max(n, 1),
                       rheology=m.MpmRheology.Viscous())


@pytest.mark.parametrize("n", [1, 31, 191, 192, 193, 639, 640, 641, 1500])
def test_item_sizes_match_oracle_grid(engine, n):
    cfg = config(16, n)
    rng = np.random.default_rng(n)
    pts = rng.uniform(0.5 + 0.51 / 16, 0.5 + 4.49 / 16, size=(n, 3)).astype(np.float32)  # base cells of one tile
    vel = rng.uniform(-0.5, 0.5, size=(n, 3)).astype(np.float32)
    sim = m.MpmSimulation.new(engine, cfg)
    sim.set_particles(pts, vel)
    sim.step(1e-4)
    gm, gp = sim.read_grid_mass_momentum()
    st = O.init_state(pts, vel, mass=cfg.particle_mass, volume=cfg.particle_volume)
    om, op = O.step(O.make_scene(cfg, [cfg.rheology], 1e-4), st, 1, want_grid=True)
    total = n * cfg.particle_mass
    assert abs(gm.astype(np.float64).sum() / total - 1.0) < 1e-5
    want = (vel.astype(np.float64) * cfg.particle_mass).sum(0)
    assert np.abs(gp.reshape(-1, 3).astype(np.float64).sum(0) - want).max() < 1e-5 * total
    om, op = np.asarray(om).reshape(-1), np.asarray(op).reshape(-1)
    assert np.abs(gm - om).max() <= max(n, 8) * 2.0 ** -23 * om.max()
    assert np.abs(gp - op).max() <= max(n, 8) * 2.0 ** -23 * max(om.max(), np.abs(op).max())
    sim.close()


@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("speed", [2.0, 40.0])
def test_moved_particles_still_deposit(engine, speed, fused, monkeypatch):
    """Without a regrouping for 20 substeps particles end up in margin cells
    (2 m/s: 0.6 cells) or outside their tile's block (40 m/s: 13 cells); deposited
    by the separate scatter and by the fused kernel."""
    monkeypatch.setenv("MOLLA_MPM_FUSED", fused)
    cfg = config(64, 20_000)
    cfg.gravity_y = 0.0
    rng = np.random.default_rng(3)
    pts = rng.uniform(0.3, 0.45, size=(20_000, 3)).astype(np.float32)
    vel = np.tile(np.array([[speed, 0.25 * speed, 0.1 * speed]], np.float32), (len(pts), 1))
    sim = m.MpmSimulation.new(engine, cfg)
    sim.set_particles(pts, vel)
    sim.set_sort_interval(1000)
    sim.step_n(2.5e-4, 20)
    t = sim.conservation_totals()
    assert not sim.read_active_grid_status().faulted()
    np.testing.assert_allclose(t[0], t[4], rtol=1e-5)
    np.testing.assert_allclose(t[1:4], t[5:8], rtol=1e-4, atol=1e-4 * abs(t[5]))
    sim.close()


@pytest.mark.parametrize("grid", [49, 98, 100])
def test_fixed_order_on_any_grid(engine, grid):
    n = 60_000
    cfg = config(grid, n)
    cfg.youngs, cfg.rheology = 6.0e4, m.MpmRheology.Sand(0.5)
    rng = np.random.default_rng(grid)
    pts = rng.uniform(0.3, 0.6, size=(n, 3)).astype(np.float32)
    vel = rng.uniform(-0.3, 0.3, size=(n, 3)).astype(np.float32)
    sim = m.MpmSimulation.new(engine, cfg)
    sim.set_particles(pts, vel)
    sim.prepare_particle_tile_ordering(n)
    sim.set_particle_tile_ordering(True)
    sim.prepare_deterministic_p2g()
    sim.set_deterministic_p2g(True)
    sim.step_n(2e-5, 60)
    s = sim.read_active_grid_status()
    assert s.fault_bits == 0 and s.completed_substeps == 60
    sim.close()
