"""The packed FP32 sweeps where they can go wrong: the particle counts where
the lanes per particle change, lists of any length in their octets (empty, one
entry, odd, full octets), both pair forms with and without noise, and pairs of
two boundary particles (counted, not listed for the force)."""
import numpy as np
import pytest

from mcf_gb300 import SDPD, configs
from mcf_gb300.params import PRECISION_FP32_MIXED, PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

# bars of the FP32-mixed path: density relative, acceleration of its pair scale
DENSITY, FORCE = 2e-6, 1e-4


def _compare(w):
    from oracle.oracle import Oracle
    g, o = SDPD(w.params), Oracle(w.params)
    for s in (g, o):
        s.upload(w.x, w.v, w.m, w.id)
        s.marching_init_force(0)
    a, b = g.download("rho", "f"), o.download("rho", "f")
    assert np.abs(a["rho"] / b["rho"] - 1.0).max() <= DENSITY
    scale = o.force_scale()[:, None] + np.abs(b["f"])
    assert (np.abs(a["f"] - b["f"]) <= FORCE * scale).all()


@pytest.mark.parametrize("side", [22, 23, 42, 43])
def test_lanes_3d(side):
    # 10,648 / 12,167 and 74,088 / 79,507 particles
    _compare(configs.c2_fluctuating_3d(n_side=side, precision=PRECISION_FP32_MIXED))


@pytest.mark.parametrize("side", [141, 142])
def test_lanes_2d(side):
    # 19,881 / 20,164 particles
    w = configs.c1_poiseuille_2d(n_side=side, precision=PRECISION_FP32_MIXED)
    rng = np.random.default_rng(side)
    w.x = w.x + rng.uniform(-0.05, 0.05, w.x.shape) / side
    _compare(w)


@pytest.mark.parametrize("noise", [False, True])
@pytest.mark.parametrize("form", [3, 4])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 10, 17, 33])
def test_list_lengths(n, dim, form, noise):
    # n particles within the cut-off of one another: lists of n - 1 entries
    rng = np.random.default_rng(100 * n + form)
    L = 12.0
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0, c=10.0, eta=1.0, dt=1e-4, rhs_force_type=form,
                    kt=1e-3 if noise else 0.0, Brownian=int(noise),
                    precision=PRECISION_FP32_MIXED)
    x = rng.uniform(5.0, 6.6, (n, dim))
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    w = configs.Workload("cluster", p, x, rng.normal(0.0, 0.1, (n, dim)), np.ones(n), ids, 1e-4, 1)
    _compare(w)


@pytest.mark.parametrize("side", [16, 30])
def test_walls_and_pair_count(side):
    # walls: the pair count is the FP64 path's (wall-wall pairs included)
    pairs = []
    for precision in (PRECISION_FP32_MIXED, PRECISION_FP64):
        w = configs.c3_poiseuille_3d(n_side=side, precision=precision)
        rng = np.random.default_rng(side)
        fluid = w.id[:, 1] == 0
        w.x[fluid] += rng.uniform(-0.05, 0.05, (int(fluid.sum()), 3))
        # off the lattice's exact cut-off distances, where FP32 may differ
        w.x[~fluid] += rng.uniform(-0.01, 0.01, (int((~fluid).sum()), 3)) * [1, 0, 1]
        g = SDPD(w.params)
        g.upload(w.x, w.v, w.m, w.id)
        g.marching_init_force(0)
        pairs.append(g.info()["num_pairs"])
    # FP32 separations may take a pair at the cut-off the other way
    assert abs(pairs[0] - pairs[1]) <= 1e-6 * pairs[1] + 2


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 575])
def test_last_block_of_an_oldroyd_b_system(n, precision):
    # several lanes per particle: the last block's idle lanes, the epilogues
    # run by the block's first threads (velocity, conformation tensor, stress)
    from oracle.oracle import Oracle
    w = configs.c5_oldroyd_b_2d(n_side=24)
    w.params.stress_tensor = 1
    w.params.precision, w.params.Brownian, w.params.kt = precision, 0, 0.0
    rng = np.random.default_rng(n)
    w.x = w.x + rng.uniform(-0.2, 0.2, w.x.shape)
    w.v = rng.normal(0, 1e-2, w.v.shape)
    g, o = SDPD(w.params), Oracle(w.params)
    for s in (g, o):
        s.upload(w.x[:n], w.v[:n], w.m[:n], w.id[:n])
        s.marching_init_force(0)
    fp64 = precision == PRECISION_FP64
    a, b = g.download("rho", "f", "s"), o.download("rho", "f", "s")
    assert np.abs(a["rho"] / b["rho"] - 1.0).max() <= (1e-12 if fp64 else DENSITY)
    bar = 1e-12 if fp64 else FORCE
    scale = o.force_scale()[:, None]
    assert (np.abs(a["f"] - b["f"]) <= bar * (scale + np.abs(b["f"]))).all()
    # s_i sums r (x) a / 2 over pairs within the cut-off
    assert np.abs(a["s"] - b["s"]).max() <= bar * w.params.cut_off * scale.max()
    for s in (g, o):
        s.marching_integrate_VV(1, w.dt)
    a, b = g.download("v", "ct"), o.download("v", "ct")
    assert np.abs(a["v"] - b["v"]).max() <= bar * (np.abs(b["v"]).max() + w.dt * scale.max())
    dev = np.abs(b["ct"] - np.array([1.0, 0, 0, 1.0])).max()
    assert np.abs(a["ct"] - b["ct"]).max() <= (1e-12 if fp64 else 1e-3 * dev + 1e-9)
