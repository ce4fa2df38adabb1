"""The candidate scan and the FP64 density's lanes per particle where they can
go wrong: cells around 32 particles (the scan's chunk), crowded and empty
cells, more chunks than the scan notes at once, and the particle counts where
the lanes per particle change."""
import numpy as np
import pytest

from mcf_gb300 import SDPD, configs
from mcf_gb300.params import PRECISION_FP32_MIXED, PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu


def _brute(x, L, rc):
    """Number density (quintic, 64 bits) and directed pair count, all pairs."""
    dim = x.shape[1]
    h = rc / 3.0
    coef = 7.0 / (478.0 * np.pi * h * h) if dim == 2 else 3.0 / (359.0 * np.pi * h ** 3)
    rho = np.full(len(x), 66.0 * coef)
    pairs = 0
    for i in range(len(x)):
        d = x - x[i]
        d -= L * np.round(d / L)
        r = np.sqrt((d * d).sum(1))
        r[i] = rc
        s = r[r < rc] / h
        pairs += len(s)
        p5 = lambda a: np.clip(a - s, 0.0, None) ** 5  # noqa: E731
        rho[i] += coef * (p5(3.0) - 6.0 * p5(2.0) + 15.0 * p5(1.0)).sum()
    return rho, pairs


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("crowd", [1, 31, 32, 33, 64, 200])
def test_crowded_cells(dim, crowd, precision):
    rng = np.random.default_rng(crowd)
    L, rc = 12.5, 3.0
    # `crowd` particles in each of two neighbouring cells (one at the box's
    # corner, so that images are met), a few everywhere else
    x = np.concatenate([rng.uniform(0.05, 3.0, (crowd, dim)),
                        np.r_[3.2, 0.05, 0.05][:dim] + rng.uniform(0.0, 2.8, (crowd, dim)),
                        rng.uniform(0.0, L, (40, dim))])
    n = len(x)
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=rc, c=10.0, eta=1.0, dt=1e-4, precision=precision)
    p.reserved[0] = 512
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    g = SDPD(p)
    g.upload(x, np.zeros_like(x), np.ones(n), ids)
    g.technique_build_list(False)
    g.particles_compute_density()
    rho, pairs = _brute(x, L, rc)
    err = np.abs(g.download("rho")["rho"] / rho - 1.0).max()
    # 64 bits: a sum of up to 440 terms of one sign, each within ~10 roundings
    # (density bar of the FP64 path); FP32: bar of the FP32-mixed density
    assert err <= (1e-12 if precision == PRECISION_FP64 else 2e-6)
    if precision == PRECISION_FP64:
        assert g.info()["num_pairs"] == pairs


@pytest.mark.parametrize("side", [22, 23, 36, 37])
def test_lanes_per_particle_thresholds(side):
    # 10,648 and 12,167, 46,656 and 50,653 particles: 8, 4, 4, 1 lanes each
    from oracle.oracle import Oracle
    w = configs.c2_fluctuating_3d(n_side=side)
    g, o = SDPD(w.params), Oracle(w.params)
    for s in (g, o):
        s.upload(w.x, w.v, w.m, w.id)
        s.technique_build_list(False)
        s.particles_compute_density()
    a, b = g.download("rho")["rho"], o.download("rho")["rho"]
    assert np.abs(a / b - 1.0).max() <= 1e-12
