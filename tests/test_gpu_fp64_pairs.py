"""FP64 pair arithmetic at the places where it can go wrong: the ends of the
quintic's intervals (s = r/h at 1, 2, 3 and beside them), the inner interval
where its powers cancel, and coincident particles."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.mcfg import MCFGError
from mcf_gb300.params import PRECISION_FP64, make_params

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
AT = [0.25, 0.7, 1.0, 1.5, 2.0, 2.6, 3.0]
BESIDE = [np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), np.nextafter(2.0, 0.0),
          np.nextafter(2.0, 3.0), np.nextafter(3.0, 0.0), 2.999]


def _pair(dim, sep, **kw):
    L = 12.0
    p = make_params(num_dim=dim, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0, c=10.0, eta=1.0, dt=1e-4,
                    precision=PRECISION_FP64, **kw)
    x = np.full((2, dim), 4.0)
    x[1, 0] += sep  # 4 + sep keeps sep's bits but the last two: the reference takes the difference
    v = np.zeros((2, dim))
    v[0, :] = [0.3, -0.2, 0.1][:dim]
    ids = np.array([[1, 0], [2, 0]], np.int32)
    return p, x, v, np.ones(2), ids


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("sep", AT + BESIDE)
def test_pair_against_the_oracle(dim, sep, kernel):
    from oracle.oracle import Oracle
    p, x, v, m, ids = _pair(dim, sep, kernel_type=kernel)
    got = []
    for side in (SDPD(p), Oracle(p)):
        side.upload(x, v, m, ids)
        side.marching_init_force(0)
        got.append(side.download("rho", "f"))
    a, b = got
    # W: at most 6 roundings a side, each against at most W(0) = rho's self term
    assert np.abs(a["rho"] / b["rho"] - 1.0).max() <= 16 * EPS
    # W': the oracle's truncated powers cancel by the ratio of their sum of
    # magnitudes to the value (quintic); the rest of the pair term has about
    # 20 roundings a side and no cancellation (rho is far from rho_ref)
    s = x[1, 0] - x[0, 0]
    terms = np.array([5, -30, 75]) * np.clip(np.array([3, 2, 1]) - s, 0.0, None) ** 4
    ratio = np.abs(terms).sum() / abs(terms.sum()) if kernel == 1 and s < 3.0 else 1.0
    tol = EPS * (64 + 8 * ratio)
    assert np.abs(a["f"] - b["f"]).max() <= tol * np.abs(b["f"]).max()


@pytest.mark.parametrize("dim", [2, 3])
def test_coincident_particles(dim):
    p, x, v, m, ids = _pair(dim, 0.0)
    g = SDPD(p)
    g.upload(x, v, m, ids)
    g.technique_build_list(False)
    g.particles_compute_density()
    coef = 7.0 / (478.0 * np.pi) if dim == 2 else 3.0 / (359.0 * np.pi)
    assert np.abs(g.download("rho")["rho"] / (2 * 66.0 * coef) - 1.0).max() <= 16 * EPS
    with pytest.raises(MCFGError, match="non-finite"):
        g.marching_init_force(0)


def _forces(p, x, v, m, ids):
    from oracle.oracle import Oracle
    g, o = SDPD(p), Oracle(p)
    for side in (g, o):
        side.upload(x, v, m, ids)
        side.marching_init_force(0)
    a, b = g.download("f")["f"], o.download("f")["f"]
    # the FP64 path's acceleration bar, with its floor of 1e-6 of the median scale
    scale = o.force_scale()
    scale = np.maximum(scale, 1e-6 * np.median(scale))[:, None] + np.abs(b)
    assert (np.abs(a - b) <= 1e-12 * scale).all()


@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("crowd", [1, 32, 33, 64, 65, 150])
def test_symmetric_sweep_crowded_cells(crowd, dim, form):
    # partner sums in shared or global memory, more than one chunk of owners
    rng = np.random.default_rng(crowd)
    p, _, _, _, _ = _pair(dim, 1.0, rhs_force_type=form, rhs_density_type=1 if form == 1 else 2)
    p.reserved[0] = 512
    x = np.concatenate([rng.uniform(0.05, 2.9, (crowd, dim)),
                        np.r_[3.1, 0.05, 0.05][:dim] + rng.uniform(0.0, 2.8, (crowd, dim)),
                        rng.uniform(0.0, 12.0, (40, dim))])
    n = len(x)
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    _forces(p, x, rng.normal(0.0, 0.1, (n, dim)), np.ones(n), ids)


@pytest.mark.parametrize("side", [55, 58])
def test_symmetric_sweep_shared_cells_threshold(side):
    # 5,832 and 6,859 cells: a cell to a block, a cell to a warp
    from mcf_gb300 import configs
    w = configs.c2_fluctuating_3d(n_side=side)
    w.params.Brownian, w.params.kt = 0, 0.0
    _forces(w.params, w.x, w.v, w.m, w.id)
