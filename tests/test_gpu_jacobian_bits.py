"""Derivatives with fixed centres keep their values bit by bit: an FP32 value that is also
returned as float64 (dtype="float64").  Open structures: a row has one edge, so nothing
depends on how a centre's edges are split into tasks.  Values by digest."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIGESTS = {
    (2, 0, "off"): "5db7f0c9da6338f7", (2, 0, "cc"): "6bfe978cc415ff6c",
    (2, 1, "off"): "6128a5ef1ccb84c6", (2, 1, "cc"): "eb5be6dd0ddf3662",
    (2, 2, "off"): "9674289fbdafa741", (2, 2, "cc"): "255df3bea9c0871b",
    (2, 3, "off"): "ffd510cd3ec49e36", (2, 3, "cc"): "a60873f76963dd1f",
    (2, 4, "off"): "cd073d1d18aa71d1", (2, 4, "cc"): "2c0c86087c23c6fd",
    (2, 5, "off"): "7402773b712b626f", (2, 5, "cc"): "53d6bc8cb9ff6e5d",
    (2, 6, "off"): "4666200ead56eb1d", (2, 6, "cc"): "e46f13fc60abd23e",
    (2, 7, "off"): "b2f12f8b0d690b7e", (2, 7, "cc"): "334b1ac11a7fa705",
    (2, 8, "off"): "bfb6b480d2d0219a", (2, 8, "cc"): "b94fdf51d1496ee0",
    (2, 9, "off"): "992d6489ab00b3cd", (2, 9, "cc"): "bdb13f795b780672",
    (2, 10, "off"): "4f9ed748f59be48f", (2, 10, "cc"): "b21a873f085e509a",
    (2, 11, "off"): "c938c6c03eae2a19", (2, 11, "cc"): "535157c404823a4f",
    (2, 12, "off"): "b58f2b2f77e7fd67", (2, 12, "cc"): "cdcc8344f3d2b62f",
    (8, 6, "off"): "a6b447a86244b5db", (10, 9, "off"): "40e014c50915b084",
    (7, 3, "off"): "ef1ba7514813ec4f",
}

CASES = [(2, l, average) for l in range(13) for average in ("off", "cc")] + [(8, 6, "off"), (10, 9, "off"), (7, 3, "off")]


def digest(n_max, l_max, average):
    from cusoap_b200 import SOAP
    rng = np.random.default_rng(n_max + l_max)
    s = {"positions": rng.uniform(0.0, 9.0, (60, 3)), "atomic_numbers": rng.choice(np.array([1, 8]), 60)}
    soap = SOAP(species=[1, 8], r_cut=3.0, n_max=n_max, l_max=l_max, sigma=0.4, average=average, dtype="float64")
    J = soap.derivatives(s, centers=list(range(0, 60, 3)), return_descriptor=False)
    return hashlib.sha256((J.cpu().numpy() + 0.0).tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("case", CASES)
def test_derivatives(case):
    assert digest(*case) == DIGESTS[case]
