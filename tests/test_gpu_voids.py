"""FP64 forces beside empty cells (a droplet, slabs with a void between them, a
few particles in an empty box), where the symmetric sweep's warps share a cell:
a cell without particles hands its neighbours the zeros that its warps agreed on,
not what an earlier block left in shared memory."""
import numpy as np
import pytest

from mcf_gb300 import SDPD, configs
from mcf_gb300.params import PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

SIDE = 30.0  # 9 cells a side: 81 in 2D, 729 in 3D


def _places(shape, dim, rng):
    grid = np.stack(np.meshgrid(*[np.arange(SIDE) + 0.5] * dim, indexing="ij"), -1).reshape(-1, dim)
    if shape == "droplet":
        x = grid[((grid - SIDE / 2) ** 2).sum(1) < 49.0]
    elif shape == "slabs":
        x = grid[(grid[:, 0] < 4.0) | ((grid[:, 0] > 14.0) & (grid[:, 0] < 17.0))]
    else:
        x = rng.uniform(0.0, SIDE, (60, dim))
    return x + rng.uniform(-0.2, 0.2, x.shape)


@pytest.mark.parametrize("form", [1, 3, 4])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shape", ["droplet", "slabs", "scattered"])
def test_forces_beside_voids(gpu_lib, shape, dim, form):
    from oracle.oracle import Oracle
    rng = np.random.default_rng(dim + form)
    x = _places(shape, dim, rng) % SIDE
    n = len(x)
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[SIDE] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[SIDE] * 3, cut_off=3.0, c=10.0, eta=1.0, dt=1e-4,
                    precision=PRECISION_FP64, rhs_force_type=form,
                    rhs_density_type=1 if form == 1 else 2)
    v = rng.normal(0.0, 0.1, (n, dim))
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    o = Oracle(p)
    o.upload(x, v, np.ones(n), ids)
    o.marching_init_force(0)
    ref = o.download("f")["f"]
    # the FP64 path's acceleration bar, with its floor of 1e-6 of the median scale
    scale = o.force_scale()
    scale = np.maximum(scale, 1e-6 * np.median(scale))[:, None] + np.abs(ref)
    g = SDPD(p)
    g.upload(x, v, np.ones(n), ids)
    # a full box of its own leaves its sums in the shared memory between calls
    w = configs.c2_fluctuating_3d(n_side=24)
    full = SDPD(w.params)
    full.upload(w.x, w.v, w.m, w.id)
    got = []
    for _ in range(5):
        full.marching_init_force(0)
        g.marching_init_force(0)
        got.append(g.download("f")["f"])
        assert (np.abs(got[-1] - ref) <= 1e-12 * scale).all()
    assert all(np.array_equal(f, got[0]) for f in got)
