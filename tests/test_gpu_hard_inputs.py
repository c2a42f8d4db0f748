"""Inputs at the edge of what a call accepts: coordinates that are not numbers,
cells without a volume, buffers of the least alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _soap(periodic=False, **over):
    from cusoap_b200 import SOAP
    return SOAP(**{**dict(species=[1, 8], r_cut=4.0, n_max=3, l_max=2, sigma=0.3, periodic=periodic), **over})


def _atoms(n, seed, offset=0.0):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, (n / 0.05) ** (1.0 / 3.0), (n, 3)) + offset, rng.choice(np.array([1, 8]), n)


@pytest.mark.parametrize("at", [0, 77, 200])
def test_atom_without_a_position(at):
    """A NaN coordinate leaves the rows of the other atoms of an open structure as they are."""
    soap = _soap()
    pos, Z = _atoms(200, 8, offset=-40.0)
    want = soap.create({"positions": pos, "atomic_numbers": Z})
    got = soap.create({"positions": np.insert(pos, at, [np.nan, 1.0, 2.0], 0), "atomic_numbers": np.insert(Z, at, 1)})
    assert torch.equal(got[torch.arange(201, device="cuda") != at], want)
