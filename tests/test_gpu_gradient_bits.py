"""Position gradients keep their values bit by bit.

The gradient with respect to float64 positions is a float64 tensor of FP32
sums, so a change in the order of those sums is a change of the result.  Three
things fix it: the pair lists and their order; the coefficients (radial and
harmonic values, the order of the sum over neighbours), read here through
average="cc"; and the edge kernel.  For the last, the energy of one centre
reaches an atom through at most two edges (cells wider than the cutoff), whose
atomic sum does not depend on their order, and other centres add exact zeros.
So each has one value, compared by digest."""
import hashlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# values of FP64 bins and distance tests, and of scalar FMAs in the order of the neighbours and of
# the radial indices
PAIRS = {
    ("open", 14.0, 260, 2, 3.0): "d67b087785677a3d65162e38b84089dc",
    ("open", 14.0, 260, 2, 6.0): "352cf1d3ae7b52a92e8f15cda9b8e1b5",
    ("open", 5.0, 9, 4, 3.0): "447c2bcf3311c391a805806b6213a177",
    ("open", 5.0, 9, 4, 6.0): "f1833d9654ce85ec3c1a9f7401edf038",
    ("cubic", 4.5, 11, 4, 3.0): "5f85438a00bf7f6c4d5aa8d41e60ff11",
    ("cubic", 4.5, 11, 4, 6.0): "d1a7a97a77bf9b2555ffc8a0885104f0",
    ("cubic", 15.0, 300, 2, 3.0): "372598eaf57f5b01de0d40ebce356a0b",
    ("cubic", 15.0, 300, 2, 6.0): "fd3ad787ea2572689469ae8b655bb142",
    ("thin", 7.0, 40, 2, 3.0): "b906198a68cdb3de2f140078b17f1ee5",
    ("thin", 7.0, 40, 2, 6.0): "394e1fa54a6d9a1312dc4c1337d35359",
    ("triclinic", 6.0, 21, 2, 3.0): "d63d80bd3b0a5369731af4720dc7d66a",
    ("triclinic", 6.0, 21, 2, 6.0): "3f97027b3989590dda11b215f74e0683",
    ("triclinic", 16.0, 330, 4, 3.0): "069d0b2037a3d9ae8882b54caae2d508",
    ("triclinic", 16.0, 330, 4, 6.0): "1aa0101ec645095e4bd6445435b44c69",
    ("slab", 12.0, 150, 3, 3.0): "8b1417e9a2456a36e8aa58ac604bf0d0",
    ("slab", 12.0, 150, 3, 6.0): "0a40912671618706edacae3b1509cf77",
}


def _digest(t):
    v = t.detach().cpu().numpy()
    return hashlib.sha256((v + np.zeros((), v.dtype)).tobytes()).hexdigest()[:16]  # (+ 0: one zero)


def _structure(kind, side, n, n_species):
    """n atoms; a quarter of them on a lattice of the box's bins, where a rounding decides the bin."""
    rng = np.random.default_rng([n, len(kind), int(10 * side)])
    frac = rng.uniform(0.0, 1.0, (n, 3))
    frac[::4] = np.round(frac[::4] * 8) / 8
    cell = {"open": np.eye(3), "cubic": np.eye(3), "slab": np.diag([1.0, 0.9, 1.2]), "thin": np.diag([0.3, 1.4, 2.0]),
            "triclinic": np.array([[1.0, 0.0, 0.0], [0.2, 0.97, 0.0], [0.1, -0.15, 0.95]])}[kind] * side
    s = {"positions": frac @ cell, "atomic_numbers": rng.choice(np.array([1, 6, 7, 8][:n_species]), n)}
    if kind != "open":
        s.update(cell=cell, pbc=[True, True, kind != "slab"])
    return s


def _soap(kind, n_species, **basis):
    from cusoap_b200 import SOAP
    return SOAP(species=[1, 6, 7, 8][:n_species], periodic=kind != "open", **basis)


# open boxes of several and of less than one cutoff, cells of many images (also by x alone), wide
# ones, an open axis; every l_max of the radial-index lanes with both stream widths, and beyond
C_STRUCTURES = [("open", 14.0, 260, 2), ("open", 5.0, 9, 4), ("cubic", 4.5, 11, 4), ("cubic", 15.0, 300, 2),
                ("thin", 7.0, 40, 2), ("triclinic", 6.0, 21, 2), ("triclinic", 16.0, 330, 4), ("slab", 12.0, 150, 3)]


def pairs(structure, r_cut):
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    kind, _, _, ns = structure
    soap = _soap(kind, ns, r_cut=r_cut, n_max=2, l_max=1, sigma=0.4)
    p = _Pairs(soap, _Batch(soap, [_structure(*structure)], [None]), _lib.NL_ALL)
    return _digest(p.pair_off) + _digest(p.pairs.view(torch.int32))


@pytest.mark.parametrize("r_cut", [3.0, 6.0])
@pytest.mark.parametrize("structure", C_STRUCTURES)
def test_pair_lists(structure, r_cut):
    assert pairs(structure, r_cut) == PAIRS[structure + (r_cut,)]
