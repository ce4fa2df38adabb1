"""A particle at -0 where a face of the box lies at 0: on the face, as at +0."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import (BC_FREESPACE, BC_PERIODIC, PRECISION_FP32_MIXED, PRECISION_FP64,
                              make_params)

pytestmark = pytest.mark.gpu

L = 12.0


def _handle(dim, low, face, precision, reuse, zero):
    p = make_params(num_dim=dim, bcdef=[face] * 2 + [BC_PERIODIC] * 4, min_phys=[low] * 3,
                    max_phys=[low + L] * 3, min_phys_t=[low] * 3, max_phys_t=[low + L] * 3,
                    cut_off=3.0, c=10.0, eta=1.0, dt=1e-4, precision=precision)
    p.reserved[1] = int(reuse)
    x = np.full((3, dim), low + 0.5 * L)
    x[0, 0] = zero
    x[1, 0] = low + 1.0  # beside the lower face
    x[2, 0] = low + L - 1.0
    ids = np.stack([np.arange(1, 4), np.zeros(3)], axis=1).astype(np.int32)
    g = SDPD(p)
    g.upload(x, np.zeros((3, dim)), np.ones(3), ids)
    return g


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("low", [0.0, -L])
def test_wrap(gpu_lib, low, dim, precision):
    got = []
    for zero in (-0.0, 0.0):
        g = _handle(dim, low, BC_PERIODIC, precision, False, zero)
        g.particles_adjust_particles()
        got.append(g.download("x")["x"])
        assert got[-1][0, 0] == (0.0 if low == 0.0 else -L)
    assert np.array_equal(*got)
    if low == 0.0:
        # within the box: left as it is
        assert np.signbit(got[0][0, 0]) and not np.signbit(got[1][0, 0])


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("face", [BC_PERIODIC, BC_FREESPACE])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("low", [0.0, -L])
def test_cell_and_density(gpu_lib, low, dim, face, precision):
    # on an open upper face: outside the mesh, with neither cell nor neighbours
    got = []
    for zero in (-0.0, 0.0):
        g = _handle(dim, low, face, precision, False, zero)
        if face == BC_PERIODIC:
            g.particles_adjust_particles()
        g.technique_build_list(False)
        g.particles_compute_density()
        got.append((g.info()["num_outside"], _bits(g.download("rho")["rho"])))
        assert got[-1][0] == (1 if face == BC_FREESPACE and low < 0.0 else 0)
    assert np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP32_MIXED])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("low", [0.0, -L])
def test_position_kept_with_the_list(gpu_lib, low, dim, precision):
    # with the list kept, a position handed over is wrapped on its way back
    got = []
    for zero in (-0.0, 0.0):
        g = _handle(dim, low, BC_PERIODIC, precision, True, 0.1 if low == 0.0 else -0.1)
        g.marching_init_force(0)
        g.run_vv(0, 3, 1e-12)
        x = g.download("x")["x"]
        x[0, 0] = zero
        g.update_state(x=x)
        got.append(g.download("x")["x"])
        assert got[-1][0, 0] == (0.0 if low == 0.0 else -L)
    assert np.array_equal(*got)
