"""The l_max 6 descriptor with two lanes per radial index (n_max <= 8) against
the FP64 oracle: both stream widths (n_max <= 4 and above), odd n_max (the last
column of the two-column epilogue), one to four species, with and without
cross terms, centres with enough pairs that a stream's sums are written out
between batches, and the coefficients that the derivatives start from."""
import numpy as np
import pytest

from oracle.soap_oracle import OracleSOAP, rel_l2
from cusoap_b200 import workloads as W

pytestmark = pytest.mark.gpu

DESC_TOL = 1e-5   # the float32 path's bars against float64
DERIV_TOL = 1e-4


@pytest.mark.parametrize("n_max", [1, 4, 5, 7, 8])
@pytest.mark.parametrize("n_species,crossover,average", [(1, True, "off"), (2, False, "off"), (4, True, "off"),
                                                         (3, True, "cc")])
def test_two_lanes_per_radial_index(n_max, n_species, crossover, average):
    from cusoap_b200 import SOAP
    species = [1, 6, 7, 8][:n_species]
    P = dict(species=species, r_cut=6.0, n_max=n_max, l_max=6, sigma=0.5, crossover=crossover, average=average)
    s, o = SOAP(**P), OracleSOAP(**P)
    pos = W.water_cluster(5, 5, 5, seed=3)["positions"]
    Z = np.asarray(species)[np.random.default_rng(n_max).integers(0, n_species, len(pos))]
    centres = [0, 7, 62, 187, 188, 374]
    got = s.create({"positions": pos, "atomic_numbers": Z}, centers=centres).cpu().numpy().reshape(len(centres), -1)
    want = np.asarray(o.create(pos, Z, centers=centres)).reshape(len(centres), -1)
    for a, b in zip(got, want):
        assert rel_l2(a, b) < DESC_TOL


def test_jacobian_from_its_coefficients():
    from cusoap_b200 import SOAP
    P = dict(species=[1, 8], r_cut=4.0, n_max=7, l_max=6, sigma=0.5)
    s, o = SOAP(**P), OracleSOAP(**P)
    sysd = W.water_cluster(3, 3, 3, seed=5)
    J = s.derivatives(sysd, centers=[13, 40], return_descriptor=False).cpu().numpy()
    ref, _ = o.derivatives(sysd["positions"], sysd["atomic_numbers"], centers=[13, 40])
    assert rel_l2(J, ref) < DERIV_TOL
