"""Mass densities (sum of m W) in units where a particle's mass is near the
smallest number that FP32 holds, and the densities are not."""
import numpy as np
import pytest

from mcf_gb300 import SDPD
from mcf_gb300.params import PRECISION_FP32_MIXED, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass", [2.0 ** -122, 1.0])
@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("n", [9, 25000, 80000])
def test_mass_density(gpu_lib, n, kernel, mass):
    # particles per unit volume as in a lattice of spacing `unit`
    from oracle.oracle import Oracle
    unit = 2.0 ** -36
    rng = np.random.default_rng(n)
    side = max(12.0, n ** (1.0 / 3.0))
    L = side * unit
    p = make_params(num_dim=3, min_phys=[0.0] * 3, max_phys=[L] * 3, min_phys_t=[0.0] * 3,
                    max_phys_t=[L] * 3, cut_off=3.0 * unit, dt=1e-4, kernel_type=kernel,
                    rhs_density_type=1, rhs_force_type=1, precision=PRECISION_FP32_MIXED)
    x = rng.uniform(0.0, L, (n, 3))
    ids = np.stack([np.arange(1, n + 1), np.zeros(n)], axis=1).astype(np.int32)
    m = mass * rng.uniform(1.0, 2.0, n)
    rho = []
    for s in (SDPD(p), Oracle(p)):
        s.upload(x, np.zeros((n, 3)), m, ids)
        s.technique_build_list(False)
        s.particles_compute_density()
        rho.append(s.download("rho")["rho"])
    # the density bar of the FP32-mixed path
    assert np.abs(rho[0] / rho[1] - 1.0).max() <= 2e-6
