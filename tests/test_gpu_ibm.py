"""Immersed-boundary step for spheres on the GPU against the FP64 oracle.

Tolerances (FP32 Eulerian fields and interpolation vs FP64, <= 60 steps):
  sphere position   |dx| <= 2e-6 + 1e-3 * |x - x0|  (lattice units; sphere radius >= 3)
  sphere velocity   |dv| <= 2e-3 * max|v| + 1e-9 (and the same for the rotation)
  fluid velocity    relative L2 <= 5e-3, max abs <= 5e-6 (settling flows are
                    ~1e-4, so FP32 rounding of rho*u weighs in)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make_case(vlbm, oracle, q, builder, size, spheres, ibm_kw, cfg_kw):
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, **cfg_kw)
    ib = vlbm.IbmConfig.default(**ibm_kw)
    m = vlbm.build_node_map(builder, nx, ny, nz)
    sim = vlbm.Simulation(cfg, node_map=m)
    sp = [vlbm.Sphere(**s) for s in spheres]
    sim.add_spheres(ib, sp)
    o = oracle.OracleIbm(cfg, m, ib, sp)
    return sim, o, sp


CLOSED = dict(max_iterations=3, gx=0.0, gy=0.0, gz=-2e-5, wall_x=1, wall_y=1, wall_z=1,
              particle_young=1e5, wall_young=1e5, pp_friction=0.3, pw_friction=0.3)

CASES = [
    ("settling_pair_closed_box_q19", 19, 3, (20, 20, 28),
     [dict(diameter=8, cx=9.5, cy=9.7, cz=14.2, density=1.5, movable=1),
      dict(diameter=8, cx=10.1, cy=10.3, cz=5.0, density=1.5, movable=1)],
     CLOSED, dict(tau=0.8), 40),
    ("bingham_channel_periodic_xz_q19", 19, 1, (24, 20, 24),
     [dict(diameter=8, cx=1.5, cy=9.0, cz=12.0, vx=0.01, wz=0.002, density=1.5, movable=1)],
     dict(max_iterations=1, gx=0.0, gy=-1e-5, gz=0.0),
     dict(rheology=1, eta_p=0.1, yield_stress=1e-6, fx=2e-5), 30),
    ("contacts_pair_and_wall_q27", 27, 3, (24, 20, 24),
     [dict(diameter=8, cx=8.0, cy=10.0, cz=12.0, vx=0.02, density=1.5, movable=1),
      dict(diameter=8, cx=15.9, cy=10.2, cz=12.1, vx=-0.02, density=1.5, movable=1),
      dict(diameter=8, cx=12.0, cy=10.0, cz=3.95, vz=-0.01, wx=0.01, density=1.5, movable=1)],
     dict(CLOSED, max_iterations=2, particle_young=0.5, wall_young=100.0), dict(tau=0.7), 25),
    ("fixed_sphere_in_flow_q19", 19, 1, (24, 16, 16),
     [dict(diameter=6, cx=12.0, cy=8.0, cz=8.0, density=1.0, movable=0)],
     dict(max_iterations=2), dict(tau=0.8, fx=1e-5), 60),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_ibm_step_matches_oracle(vlbm, oracle, case):
    name, q, builder, size, spheres, ibm_kw, cfg_kw, steps = case
    sim, o, sp = make_case(vlbm, oracle, q, builder, size, spheres, ibm_kw, cfg_kw)
    x0 = np.array([[s.cx, s.cy, s.cz] for s in sp])
    sim.step(steps)
    sim.sync()
    o.step(steps)
    pg = sim.particles(len(sp))
    po = o.particles()
    pos = np.array([list(p.pos) for p in pg])
    vel = np.array([list(p.vel) for p in pg])
    w = np.array([list(p.w) for p in pg])
    assert np.all(np.abs(pos - po["pos"]) <= 2e-6 + 1e-3 * np.abs(po["pos"] - x0)), (name, pos - po["pos"])
    vscale = max(np.abs(po["vel"]).max(), 1e-12)
    assert np.abs(vel - po["vel"]).max() <= 2e-3 * vscale + 1e-9, (name, vel - po["vel"])
    wscale = max(np.abs(po["w"]).max(), 1e-12)
    assert np.abs(w - po["w"]).max() <= 2e-3 * wscale + 1e-9, (name, w - po["w"])
    mg, mo = sim.macroscopics(), o.macroscopics()
    ug = np.stack([mg["ux"], mg["uy"], mg["uz"]]).astype(np.float64)
    uo = np.stack([mo["ux"], mo["uy"], mo["uz"]])
    rel = np.linalg.norm(ug - uo) / np.linalg.norm(uo)
    assert rel <= 5e-3, (name, rel)
    assert np.abs(ug - uo).max() <= 5e-6, (name, np.abs(ug - uo).max())
    nodes_g, _ = sim.lagrangian_nodes()
    assert np.abs(nodes_g - o.nodes()).max() <= 1e-6 + 1e-3 * np.abs(po["pos"] - x0).max()


def test_sphere_mesh_matches_reference_mesher(vlbm, oracle):
    cfg = vlbm.Config.default(nx=24, ny=24, nz=24)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_CLOSED_BOX)
    c = (11.3, 12.0, 12.7)
    sim.add_spheres(vlbm.IbmConfig.default(), [vlbm.Sphere(diameter=16, cx=c[0], cy=c[1], cz=c[2], density=1.5,
                                                           movable=1)])
    assert sim.info().n_lagrangian_nodes == 608
    pos, _ = sim.lagrangian_nodes()
    xyz, S = oracle.sphere_mesh(16.0)
    np.testing.assert_allclose(pos, xyz + np.array(c)[:, None], atol=1e-12)
    p = sim.particles(1)[0]
    assert p.n_nodes == 608 and abs(p.volume - 4 / 3 * np.pi * 512) < 1e-9


def test_ibm_forces_exported(vlbm):
    cfg = vlbm.Config.default(nx=16, ny=16, nz=16, tau=0.8)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_CLOSED_BOX)
    sim.add_spheres(vlbm.IbmConfig.default(**CLOSED),
                    [vlbm.Sphere(diameter=6, cx=8, cy=8, cz=8, vx=0.01, density=1.5, movable=1)])
    sim.step(3)
    f = sim.forces()
    assert np.count_nonzero(f[0]) > 50           # spread force only around the sphere
    assert np.abs(f[0]).max() > 0
    far = f[:, 0:2, :, :]
    assert np.count_nonzero(far) == 0


def test_ibm_reset_is_reproducible(vlbm):
    cfg = vlbm.Config.default(nx=16, ny=16, nz=16, tau=0.8)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_CLOSED_BOX)
    sim.add_spheres(vlbm.IbmConfig.default(**CLOSED),
                    [vlbm.Sphere(diameter=6, cx=8, cy=8, cz=9, density=1.5, movable=1)])
    out = []
    for _ in range(2):
        sim.init_equilibrium(1.0, 0, 0, 0)
        sim.step(10)
        out.append(np.array(list(sim.particles(1)[0].pos)))
    assert np.allclose(out[0], out[1], atol=1e-9, rtol=0)  # float atomics in the spread


def test_ibm_step_bit_reproducible(vlbm):
    """Two runs of the same sphere case give identical fields and particles:
    spread forces are summed in fixed point and sphere forces in a fixed order."""
    name, q, builder, size, spheres, ibm_kw, cfg_kw, steps = CASES[2]
    out = []
    for _ in range(2):
        nx, ny, nz = size
        cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, **cfg_kw)
        sim = vlbm.Simulation(cfg, builder=builder)
        sim.add_spheres(vlbm.IbmConfig.default(**ibm_kw), [vlbm.Sphere(**s) for s in spheres])
        sim.step(steps)
        sim.sync()
        m = sim.macroscopics()
        parts = sim.particles(len(spheres))
        out.append((np.stack([m["rho"], m["ux"], m["uy"], m["uz"]]),
                    np.array([list(p.pos) + list(p.vel) + list(p.w) for p in parts])))
        sim.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("diameter,center,walls", [
    (1.5, (7.9, 8.2, 8.4), 1),      # few nodes: part-filled groups of lanes, one CTA
    (3.0, (0.4, 8.1, 9.0), 0),      # stencils across a periodic face
    (3.0, (0.4, 8.1, 15.7), 0),     # stencils across two periodic faces
    (7.0, (8.3, 3.6, 8.0), 1),      # stencils cut by a wall
    (9.0, (8.1, 8.0, 7.8), 0),      # several CTAs per sphere, the last one part-filled
])
def test_ibm_node_counts_match_oracle(vlbm, oracle, diameter, center, walls):
    w = dict(wall_x=walls, wall_y=1, wall_z=walls)
    sim, o, sp = make_case(vlbm, oracle, 19, 3 if walls else 1, (16, 17, 18),
                           [dict(diameter=diameter, cx=center[0], cy=center[1], cz=center[2], vx=0.01, wz=0.003,
                                 density=2.0, movable=1)],
                           dict(max_iterations=2, gx=0.0, gy=0.0, gz=-1e-5, **w), dict(tau=0.8))
    sim.step(6)
    o.step(6)
    pg, po = sim.particles(1)[0], o.particles()
    assert np.abs(np.array(list(pg.vel)) - po["vel"][0]).max() <= 2e-3 * np.abs(po["vel"]).max()
    assert np.abs(np.array(list(pg.w)) - po["w"][0]).max() <= 2e-3 * np.abs(po["w"]).max() + 1e-9
    mg, mo = sim.macroscopics(), o.macroscopics()
    for k in ("ux", "uy", "uz"):
        assert np.abs(mg[k] - mo[k]).max() <= 5e-6, k


def test_checkpoint_image_keeps_ibm_macroscopics_as_planes(vlbm):
    cfg = vlbm.Config.default(nx=16, ny=18, nz=20, tau=0.8)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_CLOSED_BOX)
    sim.add_spheres(vlbm.IbmConfig.default(**CLOSED),
                    [vlbm.Sphere(diameter=6, cx=8, cy=8, cz=9, vx=0.01, density=1.5, movable=1)])
    sim.step(1)
    image = sim.checkpoint().tobytes()
    off = int(np.frombuffer(image, np.uint32, 1, 12)[0])   # header_bytes
    regions = {}
    while off < len(image) - 8:
        rid, _ = np.frombuffer(image, np.uint32, 2, off)
        size = int(np.frombuffer(image, np.uint64, 1, off + 8)[0])
        regions[int(rid)] = image[off + 16:off + 16 + size]
        off += 16 + size
    planes = np.frombuffer(regions[112], np.float32).reshape(4, 20, 18, 16)
    box = planes[0] != 0
    assert 100 < box.sum() < box.size
    m = sim.macroscopics()
    for k, name in enumerate(("rho", "ux", "uy", "uz")):
        np.testing.assert_array_equal(planes[k][box], m[name][box])


@pytest.mark.parametrize("diameter,iterations", [(3.0, 1), (8.0, 2), (11.0, 1)])
def test_reading_nodes_between_steps_changes_nothing(vlbm, diameter, iterations):
    """A step leaves its node movement to the next step's boxes; a reader takes
    it at once, and the run goes on bit for bit as if nothing had been read."""
    def make():
        cfg = vlbm.Config.default(nx=24, ny=22, nz=20, tau=0.7, fx=1e-5)
        sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_PLATES_Y)
        sim.add_spheres(vlbm.IbmConfig.default(max_iterations=iterations),
                        [vlbm.Sphere(diameter=diameter, cx=1.5, cy=10.5, cz=9.0, vx=-0.02, wy=0.01, density=2.0,
                                     movable=1),
                         vlbm.Sphere(diameter=4.0, cx=14.0, cy=11.0, cz=10.0, vz=0.01, density=2.0, movable=1)])
        return sim
    a, b = make(), make()
    a.step(7)
    for k in range(7):
        b.step(1)
        if k % 2 == 0:
            b.lagrangian_nodes()
            b.lagrangian_nodes()
        if k == 3:
            c = make()
            c.restore(b.checkpoint())
            b = c
    for x, y in zip(a.lagrangian_nodes(), b.lagrangian_nodes()):
        np.testing.assert_array_equal(x, y)
    ma, mb = a.macroscopics(), b.macroscopics()
    for k in ma:
        np.testing.assert_array_equal(ma[k], mb[k])
    for p, q in zip(a.particles(2), b.particles(2)):
        assert list(p.pos) == list(q.pos) and list(p.vel) == list(q.vel) and list(p.w) == list(q.w)


@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("size", [(32, 20, 24), (20, 20, 24), (20, 20, 23)], ids=lambda s: "x".join(map(str, s)))
def test_ibm_macroscopics_are_those_of_the_populations(vlbm, oracle, q, storage, size):
    """rho and u of the sphere boxes come from the IBM step's own read of single
    nodes (natural layout, node pairs, blocked pairs).  With the force that it
    spread, they are the moments of the populations: rho = sum f, rho u = sum c f
    + F / 2.  The spheres cross the plane where the pairs' lanes change (NZ / 2),
    the periodic z seam and an x face.  Sums of Q values below 0.4 in FP32 and
    one quotient: below 1e-6."""
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, storage=storage, tau=0.8, fx=1e-4,
                              layout=vlbm.LAYOUT_NATURAL if nz % 2 else vlbm.LAYOUT_ZPAIR)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_PLATES_Y)
    assert sim.info().layout == (0 if nz % 2 else 2 if nx % 32 == 0 else 1)
    rng = np.random.default_rng(2)
    sim.set_populations((sim.populations() * (1 + 0.02 * rng.standard_normal((q, nz, ny, nx)))).astype(np.float32))
    sim.add_spheres(vlbm.IbmConfig.default(max_iterations=2, gx=0.0, gy=0.0, gz=-1e-5),
                    [vlbm.Sphere(diameter=6.0, cx=8.2, cy=9.6, cz=nz / 2, vx=0.01, density=1.5, movable=1),
                     vlbm.Sphere(diameter=5.0, cx=0.7, cy=9.4, cz=nz - 0.6, vz=0.01, density=1.5, movable=1)])
    c = np.array(oracle.velocities(q), dtype=np.float64)
    for step in (1, 2, 3):
        sim.step(1)
        m, f, force = sim.macroscopics(), sim.populations().astype(np.float64), sim.forces().astype(np.float64)
        assert np.count_nonzero(force[2]) > 200          # the spread force reaches the nodes around both spheres
        rho = f.sum(0)
        assert np.abs(m["rho"] - rho).max() <= 1e-6, step
        for a, name in enumerate(("ux", "uy", "uz")):
            u = (np.tensordot(c[:, a], f, 1) + 0.5 * force[a]) / rho
            assert np.abs(m[name] - u).max() <= 1e-6, (step, name)
    sim.close()
