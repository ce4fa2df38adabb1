"""FP32 lists of more entries with a boundary particle than 15 bits count: a
fluid particle among 34,200 wall particles, all within its reach."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import (BC_PERIODIC, BC_WALL_SOLID, PRECISION_FP32_MIXED, PRECISION_FP64,
                              make_params)

pytestmark = pytest.mark.gpu

PER_CELL = 1800  # of at most 2,048


@pytest.mark.parametrize("reuse", [0, 1])
@pytest.mark.parametrize("form", [2, 3])
def test_many_boundary_partners(gpu_lib, form, reuse):
    rng = np.random.default_rng(form)
    L, rc = 12.0, 3.0  # 27 cells of side 4; the fluid particle at the centre of the middle one
    parts = [np.full((1, 3), 6.0)]
    for c in np.ndindex(3, 3, 3):
        c = np.array(c) - 1
        turns = np.abs(c).sum()
        if turns > 2:
            continue  # the corner cells are out of reach
        u = rng.uniform(0.0, 1.0, (PER_CELL, 3))
        depth = 0.1 if turns == 2 else 0.6
        away = np.where(c != 0, c * (2.001 + depth * u), 0.6 * (u - 0.5))
        parts.append(6.0 + away)
    x = np.concatenate(parts)
    n = len(x)
    r = np.sqrt(((x[1:] - x[0]) ** 2).sum(1))
    assert n - 1 > 32768 and r.max() < 2.999
    ids = np.stack([np.arange(1, n + 1), np.full(n, -3)], axis=1).astype(np.int32)
    ids[0, 1] = 0
    v = np.zeros((n, 3))
    v[0] = [0.3, -0.2, 0.1]
    out = []
    for precision in (PRECISION_FP32_MIXED, PRECISION_FP64):
        p = make_params(num_dim=3, bcdef=[BC_PERIODIC] * 2 + [BC_WALL_SOLID] * 2 + [BC_PERIODIC] * 2,
                        min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                        max_phys_t=[L] * 3, cut_off=rc, c=1.0, eta=1.0, dt=1e-12,
                        rhs_force_type=form, precision=precision)
        p.reserved[0], p.reserved[1] = 36000, reuse
        g = SDPD(p)
        g.upload(x, v, np.ones(n), ids)
        g.marching_init_force(0)
        if reuse:
            g.run_vv(0, 1, 1e-12)
        out.append((g.download("rho", "f"), g.info()["num_pairs"], g.info()["max_neigh"]))
        del g
    (a, pairs_a, most_a), (b, pairs_b, most_b) = out
    assert most_a == most_b == n - 1
    # FP32 separations may take a pair at the cut-off the other way
    assert abs(pairs_a - pairs_b) <= 1e-5 * pairs_b
    # number density of the fluid particle in 64 bits (bar of the FP32-mixed density)
    h = rc / 3.0
    coef = 3.0 / (359.0 * np.pi * h ** 3)
    s = r / h
    q = lambda a, e: np.clip(a - s, 0.0, None) ** e  # noqa: E731
    rho = 66.0 * coef + coef * (q(3, 5) - 6.0 * q(2, 5) + 15.0 * q(1, 5)).sum()
    assert abs(a["rho"][0] / rho - 1.0) <= 2e-6 and abs(b["rho"][0] / rho - 1.0) <= 1e-12
    # its acceleration against the FP64 path, bar on the sum of the pair terms' sizes: both
    # pressures are the fluid's, a wall particle's density 1, |v_ij| at most 1.5 |v|
    gw = coef / h * (5.0 * q(3, 4) - 30.0 * q(2, 4) + 75.0 * q(1, 4))
    press = rho - 1.0
    inv = 1.0 / rho
    scale = ((press * (inv ** 2 + 1.0)) * gw + 3.0 * (inv + 1.0) ** 2 * gw / r).sum()
    assert np.abs(a["f"][0] - b["f"][0]).max() <= 1e-4 * scale
