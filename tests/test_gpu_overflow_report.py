"""What an overflowing list reports: the candidates of the fullest particle and
the capacity of the list they did not fit in, of a step's own list and of the
one kept between steps, in single steps and replayed ones."""
import re

import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.mcfg import MCFGError
from mcf_gb300.params import MCFG_EOVERFLOW, PRECISION_FP32_MIXED, PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

CROWD = 20  # particles of each of two tight clusters


def _handle(dim, precision, capacity, reuse, apart):
    L = 10.0  # 3 cells of 3.33: a skin of 0.33 beyond the cut-off of 3
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0, c=1.0, eta=1.0, dt=1e-9, precision=precision)
    p.reserved[0], p.reserved[1] = capacity, int(reuse)
    rng = np.random.default_rng(dim)
    x = 5.0 + rng.uniform(-0.03, 0.03, (2 * CROWD, dim))
    x[CROWD:, 0] += apart
    n = len(x)
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    g = SDPD(p)
    g.upload(x, np.zeros_like(x), np.ones(n), ids)
    return g


def _reported(e):
    assert e.value.code == MCFG_EOVERFLOW
    return [int(q) for q in re.search(r"has (\d+) candidates.*capacity (\d+)", str(e.value)).groups()]


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
def test_own_list(gpu_lib, dim, precision):
    g = _handle(dim, precision, 16, False, 1.0)
    with pytest.raises(MCFGError) as e:
        g.marching_init_force(0)
    assert _reported(e) == [2 * CROWD - 1, 16]
    assert g.info()["max_neigh"] == 2 * CROWD - 1


@pytest.mark.parametrize("steps", [1, 2, 9])
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
def test_kept_list(gpu_lib, dim, precision, steps):
    # the clusters meet within the skin only: each step's pairs fit
    g = _handle(dim, precision, CROWD, True, 3.15)
    g.marching_init_force(0)
    assert g.info()["max_neigh"] == CROWD - 1
    with pytest.raises(MCFGError) as e:
        g.run_vv(0, steps, 1e-9)
    kept, capacity = _reported(e)
    assert kept == 2 * CROWD - 1 and CROWD < capacity < kept
    # the cut list is not stepped on with: it is made, and reported, again
    with pytest.raises(MCFGError) as e:
        g.run_vv(0, steps, 1e-9)
    assert _reported(e) == [kept, capacity]
    # room for them: no error
    roomy = _handle(dim, precision, 4 * CROWD, True, 3.15)
    roomy.marching_init_force(0)
    roomy.run_vv(0, steps, 1e-9)
    assert roomy.info()["max_neigh"] == CROWD - 1
