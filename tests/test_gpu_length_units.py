"""One fluid in units of length a million times apart: what pads a partial octet
of a list or a last lone pair stays outside the support whatever the unit."""
import numpy as np
import pytest

from mcf_gb300 import SDPD, configs
from mcf_gb300.params import PRECISION_FP32_MIXED, PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

# the bars of the FP32-mixed path: density relative, acceleration of its pair scale
DENSITY, FORCE = 2e-6, 1e-4


def _compare(p, x, v, m):
    from oracle.oracle import Oracle
    ids = np.stack([np.arange(1, len(x) + 1), np.zeros(len(x))], axis=1).astype(np.int32)
    fp64 = p.precision == PRECISION_FP64
    g, o = SDPD(p), Oracle(p)
    for s in (g, o):
        s.upload(x, v, m, ids)
        s.marching_init_force(0)
    a, b = g.download("rho", "f"), o.download("rho", "f")
    assert np.abs(a["rho"] / b["rho"] - 1.0).max() <= (1e-12 if fp64 else DENSITY)
    scale = o.force_scale()[:, None] + np.abs(b["f"])
    assert (np.abs(a["f"] - b["f"]) <= (1e-12 if fp64 else FORCE) * scale).all()
    if fp64:
        return
    # the list of a step of its own and the kept one hold the same pairs
    pairs = g.info()["num_pairs"]
    kept = p.copy()
    kept.reserved[1] = 1
    h = SDPD(kept)
    h.upload(x, 0.0 * v, m, ids)
    h.marching_init_force(0)
    h.run_vv(0, 1, 1e-12 * p.dt)
    assert h.info()["num_pairs"] == pairs


# time goes with the length, so velocities, pressures over density and kT keep
# their values; mass is left alone (densities go with 1 / length^dim)
@pytest.mark.parametrize("unit", [2.0 ** 20, 2.0 ** -18])
@pytest.mark.parametrize("form,kernel", [(3, 1), (4, 1), (3, 2)])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [2, 3, 10])
def test_list_lengths(gpu_lib, n, dim, form, kernel, unit):
    rng = np.random.default_rng(10 * n + form)
    L = 12.0 * unit
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0 * unit, c=1.0, eta=unit ** (1 - dim),
                    rho=unit ** -dim, rho_ref=unit ** -dim, dt=1e-4 * unit, rhs_force_type=form,
                    kernel_type=kernel, precision=PRECISION_FP32_MIXED)
    x = rng.uniform(5.0, 6.6, (n, dim)) * unit
    _compare(p, x, rng.normal(0.0, 0.1, (n, dim)), np.ones(n))


@pytest.mark.parametrize("side,precision", [(13, PRECISION_FP32_MIXED), (23, PRECISION_FP32_MIXED),
                                            (43, PRECISION_FP32_MIXED), (13, PRECISION_FP64)])
def test_many_particles(gpu_lib, side, precision):
    # FP32: 16, 4 lanes and one a particle, partial octets everywhere
    unit = 2.0 ** 20
    w = configs.c2_fluctuating_3d(n_side=side)
    rng = np.random.default_rng(side)
    L = side * unit
    p = make_params(num_dim=3, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0 * unit, c=1.0, eta=unit ** -2,
                    rho=unit ** -3, rho_ref=unit ** -3, dt=1e-4 * unit, precision=precision)
    x = (w.x + rng.uniform(-0.2, 0.2, w.x.shape)) % side * unit
    _compare(p, x, rng.normal(0.0, 0.1, x.shape), np.ones(len(x)))
