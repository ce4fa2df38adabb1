"""When the kept candidate list is made again: at the first step in which a
particle has moved more than half the skin, decided as FP64 positions decide it,
for particles in the mesh and for those that have left it through an open face."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import (BC_FREESPACE, BC_PERIODIC, PRECISION_FP32_MIXED, PRECISION_FP64,
                              make_params)

pytestmark = pytest.mark.gpu

STEPS = 4  # half a skin is reached at the end of the fourth


@pytest.mark.parametrize("replayed", [False, True])
@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("where", [4.3, 4000.3, -70000.7])
@pytest.mark.parametrize("beyond", [-1e-9, 1e-9])
def test_rebuild_at_half_the_skin(gpu_lib, beyond, where, dim, precision, replayed):
    L = 12.0
    bc = [BC_PERIODIC] * 6
    if not 0.0 <= where < L:
        bc[0] = bc[1] = BC_FREESPACE
    p = make_params(num_dim=dim, bcdef=bc, min_phys=[0.0] * 3, max_phys=[L] * 3,
                    min_phys_t=[0.0] * 3, max_phys_t=[L] * 3, cut_off=3.0, c=10.0, eta=1.0,
                    dt=1e-2, precision=precision)
    p.reserved[1] = 1
    g = SDPD(p)
    dt = 1e-2
    # one particle that flies freely, one at rest out of its reach
    x = np.full((2, dim), 1.0)
    x[0, 0], x[0, 1] = where, 7.1
    v = np.zeros((2, dim))
    ids = np.array([[1, 0], [2, 0]], np.int32)
    g.upload(x, v, np.ones(2), ids)
    half = 0.5 * g.info()["skin"]
    assert half > 0.4
    v[0, 0] = half * (1.0 + beyond) / STEPS / dt
    # the additions' rounding leaves the displacement on its side of the bound
    assert STEPS * np.spacing(abs(where) + 1.0) < 0.5 * abs(beyond) * half
    g.upload(x, v, np.ones(2), ids)
    g.marching_init_force(0)
    g.run_vv(0, 1, dt)  # makes the first list
    done = [g.info()["list_rebuilds"]]
    for count in ([STEPS - 1, 1, 1] if not replayed else [STEPS, 1]):
        g.run_vv(1, count, dt)
        done.append(g.info()["list_rebuilds"])
    last = [0, 0, 1, 1] if beyond > 0.0 else [0, 0, 0, 1]
    if replayed:
        last = [last[0], last[2], last[3]]
    assert [d - done[0] for d in done] == last
