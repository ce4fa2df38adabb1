"""Time steps at the ends of FP64's range: the half kick's dt / 2 is 0.5 dt."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import PRECISION_FP32_MIXED, PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

TINY = np.finfo(np.float64).tiny


@pytest.mark.parametrize("reuse", [0, 1])
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dt", [TINY, 2 * TINY, 2.0 ** 1000, np.inf])
def test_kick_of_a_lone_particle(gpu_lib, dt, precision, reuse):
    dim = 3
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[12.0] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[12.0] * 3, cut_off=3.0, c=10.0, eta=1.0, dt=1e-4,
                    body_force_type=1, body_force=[2.0, 0.0, 0.0], precision=precision)
    p.reserved[1] = reuse
    g = SDPD(p)
    g.upload(np.full((1, dim), 6.0), np.zeros((1, dim)), np.ones(1), np.array([[1, 0]], np.int32))
    g.marching_init_force(0)
    # a_x = 2 throughout: two half kicks of (0.5 2) dt
    g.run_vv(0, 1, dt)
    v = g.download("v")["v"][0]
    with np.errstate(over="ignore", invalid="ignore"):
        kick = (0.5 * 2.0) * dt
        assert v[0] == kick + kick
        # none along the other axes: 0 dt
        rest = np.float64(0.0) * dt
        assert np.array_equal(v[1:], np.full(dim - 1, rest + rest), equal_nan=True)
