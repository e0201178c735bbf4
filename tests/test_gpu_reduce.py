"""FP64 global mass/momentum reduction (vlbm_moments_sum) against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,builder,size,steps", [
    (19, 1, (33, 17, 9), 40),      # node count not a multiple of the chunk
    (27, 3, (16, 16, 20), 25),
    (19, 6, (64, 64, 8), 11),      # several reduction blocks, odd parity
])
def test_moments_sum_matches_oracle(vlbm, oracle, q, builder, size, steps):
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, tau=0.8, fx=1e-4, fz=-3e-5,
                              ux_bc=[0, 0.05])
    m = vlbm.build_node_map(builder, nx, ny, nz)
    sim = vlbm.Simulation(cfg, node_map=m)
    sim.step(steps)
    got = sim.moments_sum()
    o = oracle.Oracle(cfg, m)
    o.step(steps)
    mo = o.macroscopics()
    ref = np.array([mo["rho"].sum(), (mo["rho"] * mo["ux"]).sum(), (mo["rho"] * mo["uy"]).sum(),
                    (mo["rho"] * mo["uz"]).sum()])
    n = nx * ny * nz
    assert abs(got[0] - ref[0]) <= 5e-6 * n
    assert np.all(np.abs(got[1:] - ref[1:]) <= 2e-6 * n)
    # repeated calls are bit-identical (fixed partition and order)
    assert np.array_equal(sim.moments_sum(), got)


@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("size", [(32, 9, 6), (32, 7, 2), (20, 9, 6), (20, 7, 2)], ids=lambda s: "x".join(map(str, s)))
def test_moments_sum_of_paired_layouts_equals_natural(vlbm, q, storage, size):
    """The same stored values summed from a z-paired state (blocked pairs where
    NX is a multiple of 32) and from the natural layout, after both parities:
    the same nodes in the same order, so the same bits."""
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, storage=storage, tau=0.8, fx=1e-4, fz=-3e-5,
                              layout=vlbm.LAYOUT_ZPAIR)
    sim = vlbm.Simulation(cfg, builder=vlbm.BUILDER_PLATES_Y)
    assert sim.info().layout == (2 if nx % 32 == 0 else 1)
    rng = np.random.default_rng(5)
    f = sim.populations() * (1 + 0.03 * rng.standard_normal((q, nz, ny, nx)))
    sim.set_populations(f.astype(np.float32))
    for steps in (0, 1, 1):
        sim.step(steps)
        paired = sim.moments_sum()
        pops = sim.populations().astype(np.float64)
        assert abs(paired[0] - pops.sum()) <= 1e-6 * pops.sum()
        sim.set_layout(vlbm.LAYOUT_NATURAL)
        natural = sim.moments_sum()
        sim.set_layout(vlbm.LAYOUT_ZPAIR)
        np.testing.assert_array_equal(paired, natural)
    sim.close()
