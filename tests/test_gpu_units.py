"""The gather's units and the grid update's block lists at their edges: tiles of
particle counts around the rounds of a warp and the ends of units, at each unit
size the group's particle count picks; grids below, at and off the 8^3 velocity
box, against the oracle; sparse storage whose particles leave the block of their
tile; and faults all over a scene.

Tolerances: one substep in FP32, |dx| <= 1e-6 and |dv| <= 1e-5 max(1, |v|) (see
test_gpu_parity)."""

import numpy as np
import pytest

import molla_b200 as m
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def config(grid, n, svd=0):
    return m.MpmConfig(grid_size=grid, cell_size=1.0 / grid, grid_origin=(0.0, 0.0, 0.0), gravity_y=-9.8, youngs=1.0e4, poisson=0.2,
                       friction_angle=0.0, boundary_friction=0.2, particle_mass=2.0e-3, particle_volume=1.0e-6, max_particles=max(n, 1),
                       rheology=m.MpmRheology.Snow(), svd_precision=svd)


@pytest.mark.parametrize("svd", [0, 1])
@pytest.mark.parametrize("grid,n", [(5, 40), (7, 33), (8, 32), (9, 65), (33, 31), (33, 1), (64, 20_001), (65, 96)])
def test_units_match_oracle(engine, grid, n, svd):
    cfg = config(grid, n, svd)
    rng = np.random.default_rng(grid * 1000 + n)
    pts = rng.uniform(2.2 / grid, 1.0 - 3.2 / grid, size=(n, 3)).astype(np.float32) if grid > 8 else \
        rng.uniform(2.0 / grid, (grid - 2.9) / grid, size=(n, 3)).astype(np.float32)
    vel = rng.uniform(-0.5, 0.5, size=(n, 3)).astype(np.float32)
    sim = m.MpmSimulation.new(engine, cfg)
    sim.set_particles(pts, vel)
    st = O.init_state(pts, vel, mass=cfg.particle_mass, volume=cfg.particle_volume)
    sc = O.make_scene(cfg, [cfg.rheology], 1e-4)
    sim.step(1e-4)
    O.step(sc, st, 1, precision="f32_svd64" if svd else "f32")
    assert not sim.read_active_grid_status().faulted()
    assert np.abs(sim.read_positions() - st["pos"]).max() <= 1e-6
    v = sim.read_velocities()
    assert (np.abs(v - st["vel"]) / np.maximum(np.abs(st["vel"]), 1.0)).max() <= 1e-5
    sim.close()


@pytest.mark.parametrize("beside,unit", [(0, 32), (250_000, 64), (4_000_000, 128), (24_000_000, 640)])
def test_unit_sizes_and_remainders(engine, beside, unit):
    """One substep of tiles of 1 to 1,300 particles, in units of each size: the
    unit grows with the group's particles (64 from 189,441 on, a twelfth of the
    particles per resident warp above, at most 640), so a scene beside sets it."""
    counts = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 639, 640, 641, 673, 1281, 1300]
    grid, dt = 64, 1e-3
    rng = np.random.default_rng(unit)
    pts = []
    for k, c in enumerate(counts):  # base cells of every other tile: nothing is shared
        tile = np.array([2 + 2 * (k % 5), 2 + 2 * (k // 5), 6])
        pts.append((4 * tile + 0.51 + 3.97 * rng.random((c, 3))) / grid)
    pts = np.concatenate(pts).astype(np.float32)[rng.permutation(sum(counts))]
    cfg = config(grid, len(pts))
    cfg.gravity_y = -500.0
    g = m.MpmGroup(engine, 2, len(pts) + beside, grid ** 3 + 256 ** 3 + 1024)
    sid = g.add_scene(cfg, [cfg.rheology], pts, np.zeros(len(pts), np.uint32), dt)
    if beside:
        other = config(256, beside)
        g.add_scene(other, [other.rheology], rng.random((beside, 3), np.float32) * np.float32(0.8) + np.float32(0.1),
                    np.zeros(beside, np.uint32), 1e-5)
    g.step(1)
    got = g.read_positions(sid)
    assert not g.read_status(sid).faulted()
    g.close()
    st = O.init_state(pts, mass=cfg.particle_mass, volume=cfg.particle_volume)
    O.step(O.make_scene(cfg, [cfg.rheology], dt), st, 1, precision="f32")
    assert np.abs(st["pos"] - pts)[:, 1].min() > 4e-4  # every particle falls
    assert np.abs(got - st["pos"]).max() <= 1e-6


@pytest.mark.parametrize("speed", [0.5, 30.0])
def test_sparse_marks_follow_moving_particles(engine, speed):
    """No regrouping for 24 substeps: at 30 m/s the stencils leave the 27 tiles
    around the unit's (11 cells); dense and sparse storage agree."""
    n = 5_000
    rng = np.random.default_rng(7)
    pts = rng.uniform(0.2, 0.35, size=(n, 3)).astype(np.float32)
    vel = np.tile(np.array([[speed, 0.3 * speed, 0.2 * speed]], np.float32), (n, 1))
    out = []
    for cap in (None, 3000):
        cfg = config(64, n)
        cfg.gravity_y = 0.0
        sim = m.MpmSimulation(engine, cfg, cap)
        sim.set_particles(pts, vel)
        sim.set_sort_interval(1000)
        sim.step_n(2.5e-4, 24)
        assert not sim.read_active_grid_status().faulted()
        out.append((sim.read_positions(), sim.conservation_totals()))
        sim.close()
    assert np.abs(out[0][0] - out[1][0]).max() < 1e-5
    np.testing.assert_allclose(out[0][1][0], out[1][1][0], rtol=1e-6)


@pytest.mark.parametrize("n", [500, 30_000])
def test_all_fp64_positions_off_the_grid(engine, n):
    """The all-FP64 path's cell lists against the oracle, a few particles' stencils
    reaching over the grid's edge (deposited node by node)."""
    cfg = config(24, n)
    rng = np.random.default_rng(n)
    pts = rng.uniform(0.2, 0.8, size=(n, 3))
    pts[:5] = rng.uniform(-0.02, 0.0, size=(5, 3))
    sim = m.MpmSimulation64(engine, cfg)
    sim.set_particles(pts.astype(np.float32))
    sim.set_materials([cfg.rheology], np.zeros(n, np.uint32))
    dt = float(np.float32(1e-4))
    sim.step_n(dt, 3)
    sim.step_n(dt, 2)
    pos, vel, F = sim.read_state()
    st = O.cast_state(O.init_state(pts.astype(np.float32), mass=cfg.particle_mass, volume=cfg.particle_volume), np.float64)
    O.step(O.make_scene(cfg, [cfg.rheology], dt, svd_tol=1e-14, svd_sweeps=30), st, 5, precision="f64")
    assert np.abs(pos - st["pos"]).max() < 1e-9
    assert np.abs(vel - st["vel"]).max() < 1e-7
    assert np.abs(F - st["F"]).max() < 1e-8
    sim.close()


@pytest.mark.parametrize("value", [np.nan, 1.0e30])
def test_faults_all_over_a_large_scene(engine, value):
    """Particles with a bad F all over a scene of more than 65,536 particles, whose
    gather runs by warps on their own: some latch the fault (not finite: in the
    call's record pass; out of the SVD's range: in the gather) while others of the
    same launch find it latched.  The call ends and the scene stands still."""
    n = 100_000
    cfg = config(48, n)
    rng = np.random.default_rng(5)
    sim = m.MpmSimulation.new(engine, cfg)
    sim.set_particles(rng.uniform(0.2, 0.7, size=(n, 3)).astype(np.float32))
    sim.step_n(1e-4, 2)
    C0, F0, jp0 = sim.read_particle_state()
    F = F0.copy()
    F[rng.choice(n, 3000, replace=False), 4] = value
    sim.write_particle_state(F=F)
    sim.step_n(1e-4, 3)
    s = sim.read_active_grid_status()
    assert s.numerical_fault and s.completed_substeps <= 3
    before = (sim.read_positions(), sim.read_velocities(), *sim.read_particle_state())
    sim.step_n(1e-4, 3)
    after = (sim.read_positions(), sim.read_velocities(), *sim.read_particle_state())
    for a, b in zip(before, after):
        assert np.array_equal(a, b, equal_nan=True)
    sim.write_particle_state(C_=C0, F=F0, jp=jp0)
    sim.reset_active_grid()
    sim.step_n(1e-4, 3)
    assert not sim.read_active_grid_status().faulted()
    sim.close()
