"""Read-outs of z-paired states (k_macro2, k_get_pops2) against the one-node
read-outs of the same stored values in the natural layout."""
import numpy as np
import pytest

vlbm = pytest.importorskip("vlbm")
pytestmark = pytest.mark.gpu

# (nx, ny, nz): blocked pairs (NX % 32 == 0) and plain ones, one and two planes
# of pairs (both seams in one plane at NZ = 2), part-filled last blocks
SIZES = [(32, 3, 2), (33, 5, 4), (64, 7, 6), (31, 9, 2)]
CASES = [(19, vlbm.NEWTONIAN, vlbm.STORE_F32), (19, vlbm.BINGHAM, vlbm.STORE_F16),
         (27, vlbm.POWERLAW, vlbm.STORE_BF16), (27, vlbm.BINGHAM, vlbm.STORE_F32),
         (19, vlbm.POWERLAW, vlbm.STORE_F16)]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("q,rheo,st", CASES)
@pytest.mark.parametrize("builder", [vlbm.BUILDER_PERIODIC, vlbm.BUILDER_PLATES_Y, vlbm.BUILDER_CIRCULAR_DUCT])
def test_paired_readout_equals_natural(size, q, rheo, st, builder):
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, rheology=rheo, storage=st, fx=1e-5, fz=-2e-6,
                              eta_p=0.1, yield_stress=1e-6, n_index=0.8, k_consistency=0.05,
                              layout=vlbm.LAYOUT_ZPAIR)
    sim = vlbm.Simulation(cfg, builder=builder)
    rng = np.random.default_rng(3)
    w = np.concatenate([[1 / 3], np.full(6, 1 / 18), np.full(12, 1 / 36)]) if q == 19 else \
        np.concatenate([[8 / 27], np.full(6, 2 / 27), np.full(12, 1 / 54), np.full(8, 1 / 216)])
    f = w[:, None, None, None] * (1 + 0.02 * rng.standard_normal((q, nz, ny, nx)))
    sim.set_populations(f.astype(np.float32))
    for steps in (0, 1, 1):   # initial state, then both parities of the in-place scheme
        sim.step(steps)
        pair, pops = sim.macroscopics(), sim.populations()
        sim.set_layout(vlbm.LAYOUT_NATURAL)
        nat, pops_n = sim.macroscopics(), sim.populations()
        sim.set_layout(vlbm.LAYOUT_ZPAIR)
        # the interpolated rule is the only one with products: its sums may contract differently
        assert np.abs(pops - pops_n).max() <= (2e-7 if builder == vlbm.BUILDER_CIRCULAR_DUCT else 0.0)
        # the same operations in both read-outs, so the same bits; after the interpolated rule, sums of Q
        # deviations |g| <= 0.1 w and one reciprocal: 27 * 2^-24 * 0.1 and a few ulp of 1
        for k in pair:
            if builder != vlbm.BUILDER_CIRCULAR_DUCT:
                np.testing.assert_array_equal(pair[k], nat[k], err_msg=k)
            else:
                # omega follows the stress, whose 1e-7 is 1e-4 of the 1e-3 that these populations have
                tol = 1e-3 * np.abs(nat[k]) + 1e-4 if k == "omega" else 1e-6
                assert np.all(np.abs(pair[k] - nat[k]) <= tol), k
    sim.close()
