"""The half-storage collision against the FP64 oracle, one step of each parity.

The oracle starts each step from the populations that the GPU holds, so a
stored population differs by the rounding of its own store only: stochastic,
unbiased and below one unit in the last place of the stored deviation (2^-10 of
its value for FP16, 2^-7 for BF16), plus FP32 arithmetic on values below 0.4 (a
few 2^-24 of it: 2e-7).  Its mean over the lattice is tighter by the square
root of the node count, which is what shows a constant, a sign or a force term
that is off by a little.
"""
import numpy as np
import pytest

vlbm = pytest.importorskip("vlbm")
pytestmark = pytest.mark.gpu

# (nx, ny, nz): one node per thread; node pairs; node pairs in blocks of 32
SIZES = [(16, 12, 11), (16, 12, 12), (32, 12, 10)]
F32_ERR = 2e-7
DIGITS = {vlbm.STORE_F16: 10, vlbm.STORE_BF16: 7}


def start(q, shape, oracle):
    """Populations off equilibrium by a few per cent, with flow in all directions."""
    rng = np.random.default_rng(11)
    w = np.array([oracle.weight(q, i) for i in range(q)])
    c = np.array(oracle.velocities(q))
    u = np.array([0.03, -0.02, 0.04])
    f = w * (1 + 3 * c @ u + 4.5 * (c @ u) ** 2 - 1.5 * u @ u)
    return (f[:, None, None, None] * (1 + 0.03 * rng.standard_normal((q,) + shape))).astype(np.float32)


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [vlbm.STORE_F16, vlbm.STORE_BF16])
@pytest.mark.parametrize("rheo", [vlbm.NEWTONIAN, vlbm.BINGHAM])
@pytest.mark.parametrize("op", [vlbm.OP_REGULARIZED, vlbm.OP_BGK])
@pytest.mark.parametrize("q", [19, 27])
def test_half_step_matches_oracle(oracle, q, op, rheo, storage, size):
    check_steps(oracle, q, op, rheo, storage, size)


# the last lattice whose blocks are all resident at once (148 x 3 blocks of 256), and the first that is not
@pytest.mark.parametrize("size", [(32, 32, 111), (41, 25, 111)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [vlbm.STORE_F16, vlbm.STORE_BF16])
@pytest.mark.parametrize("rheo", [vlbm.NEWTONIAN, vlbm.BINGHAM])
@pytest.mark.parametrize("op", [vlbm.OP_REGULARIZED, vlbm.OP_BGK])
def test_half_step_matches_oracle_around_one_wave(oracle, op, rheo, storage, size):
    check_steps(oracle, 27, op, rheo, storage, size)


def check_steps(oracle, q, op, rheo, storage, size):
    nx, ny, nz = size
    cfg = vlbm.Config.default(nx=nx, ny=ny, nz=nz, vel_set=q, collision=op, rheology=rheo, storage=storage, tau=0.8,
                              eta_p=0.08, yield_stress=2e-4, fx=4e-3, fy=-3e-3, fz=5e-3)
    node_map = vlbm.build_node_map(vlbm.BUILDER_PLATES_Y, nx, ny, nz)
    sim = vlbm.Simulation(cfg, node_map=node_map)
    assert sim.info().layout == (0 if nz % 2 else 2 if nx % 32 == 0 else 1)
    sim.set_populations(start(q, (nz, ny, nx), oracle))
    rest = np.array([oracle.weight(q, i) for i in range(q)])[:, None, None, None]
    for parity in (0, 1):
        assert sim.aa_parity() == parity
        o = oracle.Oracle(cfg, node_map)
        o.set_populations(sim.populations().astype(np.float64))
        sim.step(1)
        o.step(1)
        want = o.populations()
        o.close()
        off = sim.populations() - want
        ulp = np.abs(want - rest) * 2.0 ** -DIGITS[storage]
        assert np.all(np.abs(off) <= ulp + F32_ERR), (parity, np.max(np.abs(off) - ulp))
        # a rounding of a value d is off by at most its ulp, with a variance of at most ulp^2 / 4
        off, ulp = off[:, :, 1:-1, :].reshape(q, -1), ulp[:, :, 1:-1, :].reshape(q, -1)
        sigma = 0.5 * np.sqrt((ulp ** 2).sum(1)) / ulp.shape[1]
        bias = np.abs(off.mean(1))
        assert np.all(bias <= 5 * sigma + 2e-8), (parity, bias / sigma)
    sim.close()
