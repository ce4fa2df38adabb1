"""Repulsion of colloids far outside the box (they have left it through an open
face): the test for partners in reach has room for their coordinates' rounding."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import (BC_FREESPACE, BC_PERIODIC, PRECISION_FP32_MIXED, PRECISION_FP64,
                              ColloidDynamics, ColloidParams, make_params)
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("law", [1, 2])
@pytest.mark.parametrize("where", [6.0, -3e3, 1e6, 3e7])
def test_repulsion_far_from_the_box(gpu_lib, where, law, precision):
    L = 12.0
    p = make_params(num_dim=3, bcdef=[BC_FREESPACE] * 2 + [BC_PERIODIC] * 4, min_phys=[0.0] * 3,
                    max_phys=[L] * 3, min_phys_t=[0.0] * 3, max_phys_t=[L] * 3, cut_off=3.0,
                    c=10.0, eta=1.0, dt=1e-4, precision=precision)
    hn = 1e-3
    cp = ColloidParams(num_colloid=24, noslip_type=2, translate=1, rotate=1, cc_repul_type=law,
                       dout=0.05, cc_repul_F0=10.0, cc_repul_cut_off=hn, cc_repul_cut_on=0.1 * hn)
    # pairs along x with gaps across the repulsion's range, the pairs out of each other's reach
    rng = np.random.default_rng(int(abs(where)))
    radius = rng.uniform(0.3, 0.5, 24)
    x = np.full((24, 3), 6.0)
    x[0::2, 0] = where + 50.0 * np.arange(12) + rng.uniform(0.0, 1.0, 12)
    x[1::2, 0] = x[0::2, 0] + radius[0::2] + radius[1::2] + hn * np.linspace(0.2, 4.8, 12)
    cd = ColloidDynamics()
    cd.integrate_AB, cd.sub_time_step = 1, 1
    # each has one boundary particle, at its centre
    ids = np.stack([np.arange(1, 25), np.arange(1, 25)], axis=1).astype(np.int32)
    got = []
    for h in (SDPD(p), Oracle(p)):
        h.upload(x, np.zeros((24, 3)), np.ones(24), ids)
        h.set_colloids(cp, x, np.zeros((24, 3)), np.zeros((24, 3)), radius)
        h.set_colloid_dynamics(cd, np.ones(24), np.ones((24, 3)))
        h.marching_init_force(0)
        got.append(h.colloid_state()["f"][0])
    a, b = got
    # the same FP64 operations in the same order but for exp's last bit
    assert (np.abs(b[:, 0]) > 1e-3).sum() >= (4 if law == 1 else 20)
    assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
