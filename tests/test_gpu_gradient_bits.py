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
    ("triclinic", 16.0, 330, 4, 6.0): "1aa0101ec645095e90c372a3f72a376a",
    ("slab", 12.0, 150, 3, 3.0): "8b1417e9a2456a36e8aa58ac604bf0d0",
    ("slab", 12.0, 150, 3, 6.0): "0a40912671618706edacae3b1509cf77",
}
COEFFICIENTS = {
    ("open", 14.0, 260, 2, 4, 0): "ae9d6416e85553d3", ("open", 14.0, 260, 2, 8, 1): "fab634dc0752b73c",
    ("open", 14.0, 260, 2, 3, 2): "e6a0840a7efca690", ("open", 14.0, 260, 2, 4, 3): "a24cb3a7ec66c1a4",
    ("open", 14.0, 260, 2, 8, 4): "e69bf4e45fbaee18", ("open", 14.0, 260, 2, 7, 5): "00a004a01588bea3",
    ("open", 14.0, 260, 2, 8, 6): "576874da62956518", ("open", 14.0, 260, 2, 2, 6): "d90adcbd9fbd6e24",
    ("open", 14.0, 260, 2, 10, 4): "02ddea5f327a89bd", ("open", 14.0, 260, 2, 8, 8): "ab830cc19375b6c7",
    ("open", 5.0, 9, 4, 4, 0): "a3f24c8de86ff91c", ("open", 5.0, 9, 4, 8, 1): "9d83066bb015c6b4",
    ("open", 5.0, 9, 4, 3, 2): "dc827ffa84584bfb", ("open", 5.0, 9, 4, 4, 3): "84e1a1ecce37a342",
    ("open", 5.0, 9, 4, 8, 4): "a6f387f6c3c39596", ("open", 5.0, 9, 4, 7, 5): "6d37cff72f4f9d07",
    ("open", 5.0, 9, 4, 8, 6): "6a3c9a8963cb51ab", ("open", 5.0, 9, 4, 2, 6): "a038cec30acb5ea7",
    ("open", 5.0, 9, 4, 10, 4): "045a6f90b10ec5f4", ("open", 5.0, 9, 4, 8, 8): "b1aabe7de014665a",
    ("cubic", 4.5, 11, 4, 4, 0): "67733d6b497a9e83", ("cubic", 4.5, 11, 4, 8, 1): "0e2888a0a4aa341f",
    ("cubic", 4.5, 11, 4, 3, 2): "9dd299974689dbe9", ("cubic", 4.5, 11, 4, 4, 3): "ca009219b359311f",
    ("cubic", 4.5, 11, 4, 8, 4): "4460289e32826ca0", ("cubic", 4.5, 11, 4, 7, 5): "9e739ff933e72414",
    ("cubic", 4.5, 11, 4, 8, 6): "68dcd04bafd2df79", ("cubic", 4.5, 11, 4, 2, 6): "0c1f22a132aa489a",
    ("cubic", 4.5, 11, 4, 10, 4): "e90d76c787a941e0", ("cubic", 4.5, 11, 4, 8, 8): "82c5ec77d2f5fa32",
    ("cubic", 15.0, 300, 2, 4, 0): "f9f0ff141617e1ce", ("cubic", 15.0, 300, 2, 8, 1): "10e129186acfe562",
    ("cubic", 15.0, 300, 2, 3, 2): "99606ce9bc6575ca", ("cubic", 15.0, 300, 2, 4, 3): "0cb7b88397c21d6b",
    ("cubic", 15.0, 300, 2, 8, 4): "0eba5a046266e2f3", ("cubic", 15.0, 300, 2, 7, 5): "d77bb4bba924c9a9",
    ("cubic", 15.0, 300, 2, 8, 6): "e994b7061c75097a", ("cubic", 15.0, 300, 2, 2, 6): "cd2c65b7873b2cda",
    ("cubic", 15.0, 300, 2, 10, 4): "fdd678fe5463ae2e", ("cubic", 15.0, 300, 2, 8, 8): "28d543763998c535",
    ("thin", 7.0, 40, 2, 4, 0): "2f2dfc574a1d614f", ("thin", 7.0, 40, 2, 8, 1): "eee7548ec658cacf",
    ("thin", 7.0, 40, 2, 3, 2): "e2eddd5abade0789", ("thin", 7.0, 40, 2, 4, 3): "71e769e3b5c685bf",
    ("thin", 7.0, 40, 2, 8, 4): "130d4be81714ce09", ("thin", 7.0, 40, 2, 7, 5): "e1fa9ec942794a42",
    ("thin", 7.0, 40, 2, 8, 6): "d4846c47a354f85d", ("thin", 7.0, 40, 2, 2, 6): "91f925a2d4e227ae",
    ("thin", 7.0, 40, 2, 10, 4): "e7e166542f6e0de3", ("thin", 7.0, 40, 2, 8, 8): "d4df1e2b45ed9e60",
    ("triclinic", 6.0, 21, 2, 4, 0): "1737714268557601", ("triclinic", 6.0, 21, 2, 8, 1): "774244156029f3c8",
    ("triclinic", 6.0, 21, 2, 3, 2): "02194f37cb1d7627", ("triclinic", 6.0, 21, 2, 4, 3): "264613f3eb224b61",
    ("triclinic", 6.0, 21, 2, 8, 4): "5cc9b80bdd9cc9a5", ("triclinic", 6.0, 21, 2, 7, 5): "e06e9b75f3e890aa",
    ("triclinic", 6.0, 21, 2, 8, 6): "ea8472c426c5e7db", ("triclinic", 6.0, 21, 2, 2, 6): "7cb25e7230ae1b33",
    ("triclinic", 6.0, 21, 2, 10, 4): "7e62261c0ff65a17", ("triclinic", 6.0, 21, 2, 8, 8): "7b6fde5b6ebb26a8",
    ("triclinic", 16.0, 330, 4, 4, 0): "f60af04bb369840d", ("triclinic", 16.0, 330, 4, 8, 1): "e9c0c314480df32e",
    ("triclinic", 16.0, 330, 4, 3, 2): "cf817cc653457566", ("triclinic", 16.0, 330, 4, 4, 3): "87be270f1af210bf",
    ("triclinic", 16.0, 330, 4, 8, 4): "12e5af0b07320696", ("triclinic", 16.0, 330, 4, 7, 5): "cd74a5cd2ec73a5a",
    ("triclinic", 16.0, 330, 4, 8, 6): "fbad6e62d3391de6", ("triclinic", 16.0, 330, 4, 2, 6): "d9c0f21b7794dfba",
    ("triclinic", 16.0, 330, 4, 10, 4): "7b68df470ebd620d", ("triclinic", 16.0, 330, 4, 8, 8): "0a458a2f4c4c7c9d",
    ("slab", 12.0, 150, 3, 4, 0): "f5de31adc52f1cce", ("slab", 12.0, 150, 3, 8, 1): "0836b7d570e65b4f",
    ("slab", 12.0, 150, 3, 3, 2): "4ddd82ec6229f191", ("slab", 12.0, 150, 3, 4, 3): "99c6563be0587636",
    ("slab", 12.0, 150, 3, 8, 4): "f4f068b62a70d534", ("slab", 12.0, 150, 3, 7, 5): "d9b3e2a01711e082",
    ("slab", 12.0, 150, 3, 8, 6): "54b9699fa995686d", ("slab", 12.0, 150, 3, 2, 6): "ce1afbeb42808416",
    ("slab", 12.0, 150, 3, 10, 4): "18362965da9ddd29", ("slab", 12.0, 150, 3, 8, 8): "19e3079dbdce3d21",
}
GRADIENTS = {
    ("open", 7.0, 45, 2, 8, 6): "0e4c131121a1829b", ("open", 7.0, 45, 2, 8, 3): "6fecf0c5a716f983",
    ("open", 7.0, 45, 2, 8, 1): "6c7e3c4069012cac", ("open", 7.0, 45, 2, 4, 3): "b554970a29a1fc8c",
    ("open", 7.0, 45, 2, 7, 4): "6aa82edc58c8b95d", ("open", 7.0, 45, 2, 1, 2): "059dbd5a5c45c8c4",
    ("open", 7.0, 45, 2, 6, 6): "3feb0586d616894f", ("open", 7.0, 45, 2, 8, 9): "aab829f2d81072e0",
    ("open", 7.0, 45, 2, 5, 8): "6eea00807697286a", ("open", 7.0, 45, 2, 10, 9): "b45c2ec9678715c1",
    ("open", 7.0, 45, 2, 8, 12): "36e4467c4017f36b",
    ("cubic", 8.4, 60, 3, 8, 6): "00069470f4ac900a", ("cubic", 8.4, 60, 3, 8, 3): "5df8b18a0e890450",
    ("cubic", 8.4, 60, 3, 8, 1): "d41d9fbce057bafd", ("cubic", 8.4, 60, 3, 4, 3): "dde284545268f745",
    ("cubic", 8.4, 60, 3, 7, 4): "b6fe14a5e932f517", ("cubic", 8.4, 60, 3, 1, 2): "088b698ba9018f3e",
    ("cubic", 8.4, 60, 3, 6, 6): "0920ace064257b20", ("cubic", 8.4, 60, 3, 8, 9): "3c677abdc6240923",
    ("cubic", 8.4, 60, 3, 5, 8): "f83a647a24d35920", ("cubic", 8.4, 60, 3, 10, 9): "1fbe41256e57b421",
    ("cubic", 8.4, 60, 3, 8, 12): "0aa5298a40b7a876",
    ("triclinic", 9.0, 75, 2, 8, 6): "9738954def761f57", ("triclinic", 9.0, 75, 2, 8, 3): "870d8a42bf2a0c98",
    ("triclinic", 9.0, 75, 2, 8, 1): "d4afcd04f4d325bd", ("triclinic", 9.0, 75, 2, 4, 3): "84b58eb2e22c5736",
    ("triclinic", 9.0, 75, 2, 7, 4): "a181dc909a36420e", ("triclinic", 9.0, 75, 2, 1, 2): "5aa3d09443a8a481",
    ("triclinic", 9.0, 75, 2, 6, 6): "88bd991a25990ea6", ("triclinic", 9.0, 75, 2, 8, 9): "4c4c76c07d0acd43",
    ("triclinic", 9.0, 75, 2, 5, 8): "b53cd7eff6912d30", ("triclinic", 9.0, 75, 2, 10, 9): "4e44535bea287642",
    ("triclinic", 9.0, 75, 2, 8, 12): "bb1507c5e4d59103",
    ("slab", 9.6, 60, 2, 8, 6): "3c1e4d5e756b17b1", ("slab", 9.6, 60, 2, 8, 3): "cd19ad4867cb0973",
    ("slab", 9.6, 60, 2, 8, 1): "3df4eebeb5f7bba3", ("slab", 9.6, 60, 2, 4, 3): "259a63cd04e5a67a",
    ("slab", 9.6, 60, 2, 7, 4): "ee2ab37b8929cfcd", ("slab", 9.6, 60, 2, 1, 2): "cea884d9f5cea66c",
    ("slab", 9.6, 60, 2, 6, 6): "cc35ba3141689072", ("slab", 9.6, 60, 2, 8, 9): "a1b2648f4f94acbe",
    ("slab", 9.6, 60, 2, 5, 8): "72232f60c063be68", ("slab", 9.6, 60, 2, 10, 9): "7506b0d9b5c8265a",
    ("slab", 9.6, 60, 2, 8, 12): "5449e267224e6d63",
}


def _digest(t):
    v = t.detach().cpu().numpy()
    return hashlib.sha256((v + np.zeros((), v.dtype)).tobytes()).hexdigest()[:16]  # (+ 0: one zero)


def _at(frac, cell):
    """frac @ cell without a library's choice of FMAs."""
    return frac[:, :1] * cell[0] + frac[:, 1:2] * cell[1] + frac[:, 2:] * cell[2]


def _structure(kind, side, n, n_species):
    """n atoms; a quarter of them on a lattice of the box's bins, where a rounding decides the bin."""
    rng = np.random.default_rng([n, len(kind), int(10 * side)])
    frac = rng.uniform(0.0, 1.0, (n, 3))
    frac[::4] = np.round(frac[::4] * 8) / 8
    cell = {"open": np.eye(3), "cubic": np.eye(3), "slab": np.diag([1.0, 0.9, 1.2]), "thin": np.diag([0.3, 1.4, 2.0]),
            "triclinic": np.array([[1.0, 0.0, 0.0], [0.2, 0.97, 0.0], [0.1, -0.15, 0.95]])}[kind] * side
    s = {"positions": _at(frac, cell), "atomic_numbers": rng.choice(np.array([1, 6, 7, 8][:n_species]), n)}
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
C_BASES = [(4, 0), (8, 1), (3, 2), (4, 3), (8, 4), (7, 5), (8, 6), (2, 6), (10, 4), (8, 8)]
# (cells at least twice the 4.1 A cutoff wide)
G_STRUCTURES = [("open", 7.0, 45, 2), ("cubic", 8.4, 60, 3), ("triclinic", 9.0, 75, 2), ("slab", 9.6, 60, 2)]
G_BASES = [(8, 6), (8, 3), (8, 1), (4, 3), (7, 4), (1, 2), (6, 6), (8, 9), (5, 8), (10, 9), (8, 12)]


def pairs(structure, r_cut):
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    kind, _, _, ns = structure
    soap = _soap(kind, ns, r_cut=r_cut, n_max=2, l_max=1, sigma=0.4)
    p = _Pairs(soap, _Batch(soap, [_structure(*structure)], [None]), _lib.NL_ALL)
    return _digest(p.pair_off) + _digest(p.pairs.view(torch.int32))


def coefficients(structure, basis):
    kind, _, _, ns = structure
    soap = _soap(kind, ns, r_cut=6.0, n_max=basis[0], l_max=basis[1], sigma=0.4, average="cc")
    return _digest(soap.create(_structure(*structure)))


def gradients(structure, basis):
    kind, _, n, ns = structure
    soap = _soap(kind, ns, r_cut=3.0, n_max=basis[0], l_max=basis[1], sigma=0.3)
    s = _structure(*structure)
    w = torch.as_tensor(np.random.default_rng(3).standard_normal(soap.get_number_of_features()), dtype=torch.float32,
                        device="cuda")
    out = []
    for c in (0, n // 2, n - 1):
        pos = torch.as_tensor(s["positions"], device="cuda").requires_grad_(True)
        (soap.create(dict(s, positions=pos))[c] @ w).backward()
        out.append(pos.grad)
    return _digest(torch.stack(out))


@pytest.mark.parametrize("r_cut", [3.0, 6.0])
@pytest.mark.parametrize("structure", C_STRUCTURES)
def test_pair_lists(structure, r_cut):
    assert pairs(structure, r_cut) == PAIRS[structure + (r_cut,)]


@pytest.mark.parametrize("basis", C_BASES)
@pytest.mark.parametrize("structure", C_STRUCTURES)
def test_coefficients(structure, basis):
    assert coefficients(structure, basis) == COEFFICIENTS[structure + basis]


@pytest.mark.parametrize("basis", G_BASES)
@pytest.mark.parametrize("structure", G_STRUCTURES)
def test_gradient_of_one_centre(structure, basis):
    assert gradients(structure, basis) == GRADIENTS[structure + basis]


def _radius(v, order):
    """FP32 radius of FP32 vectors, squares added in an order, by FMAs (exact products in float64)."""
    f = lambda x: x.astype(np.float32).astype(np.float64)  # noqa: E731
    x, y, z = (v[:, order.index(k)].astype(np.float64) for k in "abc")
    return np.sqrt(f(z * z + f(y * y + f(x * x))).astype(np.float32))


def test_pairs_at_segment_edges():
    """Pairs whose segment depends on the rounding of their radius: that of z z + (x x + y y)."""
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    soap = _soap("open", 1, r_cut=6.0, n_max=4, l_max=3, sigma=0.4)
    h, nseg = soap._basis.seg_width, int(soap._basis.n_seg)
    rng = np.random.default_rng(2)
    v = rng.standard_normal((40000, 3))
    v *= (rng.integers(1, nseg, (40000, 1)) * h) / np.linalg.norm(v, axis=1, keepdims=True)
    v = v.astype(np.float32)
    seg = lambda order: np.minimum((_radius(v, order) * np.float32(1.0 / h)).astype(np.int64), nseg - 1)  # noqa: E731
    edge = (seg("bac") != seg("abc")) | (seg("bac") != seg("cba"))
    v = v[edge & (np.linalg.norm(v, axis=1) < 0.99 * soap._cutoff)][:300]
    assert len(v) == 300
    pos = np.concatenate([np.zeros((1, 3)), v.astype(np.float64)])
    batch = _Batch(soap, [{"positions": pos, "atomic_numbers": np.ones(301, int)}], [[0]])
    p = _Pairs(soap, batch, _lib.NL_ALL)
    got = p.pairs[:p.total].cpu().numpy()
    assert p.total == 301
    r = _radius(got[:, :3], "bac")
    assert (np.diff(np.minimum((r * np.float32(1.0 / h)).astype(np.int64), nseg - 1)) >= 0).all()


# by shape of the cell: 12 cells each
SITES = {"rotated": "f096e2f68e70664b", "skewed": "8817e01d8cbd18b8", "both": "e08721337261f0da"}


def sites(shape):
    """Pair lists of atoms on lattice sites, where a rounding decides the bin and the image."""
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    soap = _soap("cubic", 1, r_cut=4.0, n_max=2, l_max=1, sigma=0.3)
    out = []
    for i in range(12):
        rng = np.random.default_rng([i, len(shape)])
        cell = np.diag(rng.uniform(3.0, 14.0, 3))
        if shape != "rotated":
            cell[1] += rng.uniform(-0.5, 0.5) * cell[0]
            cell[2] += rng.uniform(-0.5, 0.5) * cell[0] + rng.uniform(-0.5, 0.5) * np.array([0.0, cell[1, 1], 0.0])
        if shape != "skewed":  # (to 20 bits behind the point, whatever the library's last bits)
            cell = np.round(_at(cell, np.linalg.qr(rng.standard_normal((3, 3)))[0]) * 2.0 ** 20) / 2.0 ** 20
        pos = _at(rng.integers(0, 24, (40, 3)) / 24.0 + rng.integers(-1, 2, (40, 3)), cell)
        p = _Pairs(soap, _Batch(soap, [{"positions": pos, "atomic_numbers": np.ones(40, int), "cell": cell,
                                        "pbc": [True, True, i % 4 > 0]}], [None]), _lib.NL_ALL)
        out += [_digest(p.pair_off), _digest(p.pairs[:p.total].view(torch.int32))]
    return hashlib.sha256("".join(out).encode()).hexdigest()[:16]


@pytest.mark.parametrize("shape", ["rotated", "skewed", "both"])
def test_lattice_sites(shape):
    assert sites(shape) == SITES[shape]
