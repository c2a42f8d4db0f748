"""The power spectrum is p[(j n), (j' n'), l] = sqrt(8 pi^2 / (2 l + 1)) sum_m c[j n lm] c[j' n' lm], with the
sum in FP32 FMAs over m in order: a descriptor asked for as float64 keeps these values."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _in_order(c, N, L, crossover):
    """(C, S, N, K) float32 coefficients -> (C, F), one rounding a product (a product of two FP32
    values is exact in float64)."""
    S, out = c.shape[1], []
    pref = torch.tensor([8.0], dtype=torch.float32, device=c.device) * float(np.float32(math.pi ** 2))
    for j in range(S):
        for jd in range(j, S if crossover else j + 1):
            n, nd = torch.meshgrid(torch.arange(N), torch.arange(N), indexing="ij")
            keep = (n <= nd).reshape(-1) if j == jd else torch.ones(N * N, dtype=torch.bool)
            n, nd = n.reshape(-1)[keep].to(c.device), nd.reshape(-1)[keep].to(c.device)
            for l in range(L + 1):
                acc = torch.zeros((c.shape[0], len(n)), dtype=torch.float32, device=c.device)
                for k in range(l * l, (l + 1) ** 2):
                    acc = (c[:, j, n, k].double() * c[:, jd, nd, k].double() + acc.double()).float()
                out.append(acc * torch.sqrt(pref / (2.0 * l + 1.0)))
    return torch.cat(out, 1)


# every l_max of the radial-index lanes with both stream widths, and the lanes grouped by l
@pytest.mark.parametrize("n_max,l_max", [(n, l) for l in range(7) for n in (3, 8)] + [(10, 3), (8, 7), (10, 9), (8, 12)])
def test_sum_over_m(n_max, l_max):
    from cusoap_b200 import SOAP, _lib
    from cusoap_b200.soap import _Batch, _Pairs
    rng = np.random.default_rng(n_max + l_max)
    s = {"positions": rng.uniform(0.0, 8.0, (40, 3)), "atomic_numbers": rng.choice(np.array([1, 8]), 40)}
    for crossover in (True, False):
        soap = SOAP(species=[1, 8], r_cut=4.0, n_max=n_max, l_max=l_max, sigma=0.4, crossover=crossover, dtype="float64")
        batch = _Batch(soap, [s], [None])
        _, c = soap._run_descriptor(batch, _Pairs(soap, batch, _lib.NL_CREATE), _lib.OUT_PS, want_coeff=True)
        want = _in_order(c.reshape(40, 2, n_max, (l_max + 1) ** 2), n_max, l_max, crossover)
        assert torch.equal(soap.create(s), want.double())
