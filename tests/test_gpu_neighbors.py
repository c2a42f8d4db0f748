"""Neighbour lists against a brute-force float64 distance test on the device:
every centre's pair set, the offsets and the {total, largest, flags} summary."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _soap(periodic, r_cut=4.0):
    from cusoap_b200 import SOAP
    return SOAP(species=[1, 8], r_cut=r_cut, n_max=2, l_max=1, sigma=0.3, periodic=periodic)


def _lattice(kind):
    """Cells of every enumeration: diagonal, sheared both ways, and with an open axis."""
    return {"cubic": np.eye(3), "flat": np.diag([1.9, 1.1, 0.5]),
            "sheared": np.array([[1.0, 0.0, 0.0], [0.7, 0.8, 0.0], [-0.5, 0.4, 0.9]]),
            "rotated": np.array([[0.6, 0.8, 0.0], [-0.8, 0.6, 0.1], [0.0, 0.1, 1.0]])}[kind]


def _system(n, periodic, rng, density=0.05):
    side = (n / density) ** (1.0 / 3.0)
    s = {"positions": rng.uniform(0.0, side, (n, 3)) + (0.0 if periodic else -3.0 * side),
         "atomic_numbers": rng.choice(np.array([1, 8]), n)}
    if periodic:
        s.update(cell=np.eye(3) * side, pbc=[True, True, True])
    return s


def _brute(soap, s):
    """(centre, atom, x, y, z) of every pair of one structure, r = 0 own edges included."""
    pos = torch.as_tensor(s["positions"], device="cuda")
    shifts = torch.zeros((1, 3), dtype=torch.float64, device="cuda")
    if "cell" in s:  # the image offsets of the atoms as given: |n_i| <= ceil(cutoff / width_i) on periodic axes
        width = 1.0 / np.linalg.norm(np.linalg.inv(s["cell"]), axis=0)
        g = [torch.arange(-k, k + 1, dtype=torch.float64, device="cuda")
             for k in (int(np.ceil(soap._cutoff / w)) if p else 0 for w, p in zip(width, s["pbc"]))]
        shifts = torch.cartesian_prod(*g) @ torch.as_tensor(s["cell"], device="cuda")
    img = (pos[None] + shifts[:, None]).reshape(-1, 3)
    rows = []
    step = max(1, (1 << 25) // img.shape[0])
    for a in range(0, pos.shape[0], step):
        d = img[None] - pos[a:a + step, None]
        i, j = ((d * d).sum(-1) <= soap._cutoff ** 2).nonzero(as_tuple=True)
        rows.append(torch.cat([(i + a)[:, None].double(), (j % pos.shape[0])[:, None].double(), d[i, j]], 1))
    return torch.cat(rows).cpu().numpy()


def _check(soap, systems):
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    batch = _Batch(soap, systems, [None] * len(systems))
    pairs = _Pairs(soap, batch, _lib.NL_ALL)
    off = pairs.pair_off.cpu().numpy()
    p = pairs.pairs.cpu().numpy()
    word = p[:, 3].copy().view(np.int32)
    a0 = 0
    for s in systems:
        n = len(s["atomic_numbers"])
        want = _brute(soap, s)
        counts = np.bincount(want[:, 0].astype(int), minlength=n)
        assert np.array_equal(np.diff(off[a0:a0 + n + 1]), counts)
        rows = slice(off[a0], off[a0 + n])
        got = np.concatenate([np.repeat(np.arange(n), counts)[:, None], (word[rows] & ((1 << 27) - 1))[:, None] - a0,
                              p[rows, :3]], 1)
        # same pairs: vectors differ by FP32 rounding (2^-24 of up to the cutoff, 5 A) and by the order of
        # the float64 operations at coordinates of up to 300 A (about 1e-13 A)
        key = lambda v: v[np.lexsort(np.concatenate([np.round(v[:, 2:], 3).T[::-1], v[:, 1::-1].T]))]  # noqa: E731
        g, w = key(got), key(want)
        assert np.array_equal(g[:, :2], w[:, :2])
        assert np.abs(g[:, 2:] - w[:, 2:]).max() < 2e-3 if len(w) else True
        # rounding to 1e-3 can order two images of one atom differently; their sums agree
        assert np.abs(g[:, 2:].sum(0) - w[:, 2:].sum(0)).max() <= 1e-6 * max(1, len(w))
        a0 += n
    assert pairs.total == off[-1]
    assert pairs.max_pairs == (np.diff(off).max() if len(off) > 1 else 0)
    # the two-call form gives the same offsets and summary
    lib = _lib.load()
    off2 = torch.empty_like(pairs.pair_off)
    stats = torch.empty(3, dtype=torch.int64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    args = (ctypes.byref(soap._basis), ctypes.byref(batch.cs), ctypes.byref(batch.cc))
    _lib.check(lib.soapb_neighbors_count(*args, _lib.NL_ALL, pairs.work.data_ptr(), pairs.work.numel(),
                                         off2.data_ptr(), st))
    _lib.check(lib.soapb_neighbors_stats(*args, pairs.work.data_ptr(), off2.data_ptr(), stats.data_ptr(), st))
    assert torch.equal(off2, pairs.pair_off)
    assert stats.tolist() == [pairs.total, pairs.max_pairs, 0]


# one CTA, the edges of its 512 threads, clusters of 2, 4 and 8 CTAs, the last size whose offsets
# the count's last block scans (8192), the last one built in a single launch (16384), and beyond
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("n", [1, 2, 33, 511, 513, 1025, 2050, 4097, 8192, 8193, 16384, 16385])
def test_lists_match_brute_force(n, periodic):
    _check(_soap(periodic), [_system(n, periodic, np.random.default_rng(n))])


@pytest.mark.parametrize("periodic", [False, True])
def test_batch_of_uneven_structures(periodic):
    rng = np.random.default_rng(5)
    _check(_soap(periodic), [_system(n, periodic, rng) for n in (1, 700, 2, 40, 1500, 3)])


def test_coincident_and_clustered_atoms():
    """One bin that holds most atoms, two atoms at one point, far outliers."""
    rng = np.random.default_rng(6)
    pos = np.concatenate([rng.uniform(0, 0.5, (600, 3)), [[0.1, 0.1, 0.1], [0.1, 0.1, 0.1]],
                          [[5e4, 0, 0], [0, -3e4, 2e4]]])
    _check(_soap(False), [{"positions": pos, "atomic_numbers": np.ones(len(pos), np.int64)}])


@pytest.mark.parametrize("wrapped", [True, False])
@pytest.mark.parametrize("pbc", [[True, True, True], [True, False, True], [False, True, False]])
@pytest.mark.parametrize("kind", ["cubic", "flat", "sheared", "rotated"])
@pytest.mark.parametrize("n", [2, 9, 150, 1200])
def test_frames_and_images(n, kind, pbc, wrapped):
    """Cells much smaller than the cutoff to several times it; positions in the
    cell and up to two cells outside (the image set is that of the atoms as given)."""
    rng = np.random.default_rng(n + len(kind))
    cell = _lattice(kind)
    cell = cell * (n / 0.06 / abs(np.linalg.det(cell))) ** (1.0 / 3.0)
    frac = rng.uniform(0.0, 1.0, (n, 3))
    if not wrapped:
        frac += rng.integers(-2, 3, (n, 3))
    _check(_soap(True), [{"positions": frac @ cell, "atomic_numbers": rng.choice(np.array([1, 8]), n),
                          "cell": cell, "pbc": pbc}])


@pytest.mark.parametrize("n,side", [(700, 9.0), (1000, 9.5), (2000, 10.0), (60, 1.2)])
def test_dense_centres(n, side):
    """More pairs per centre than the fill stages, and a cell whose shifts do not fit its packed form."""
    rng = np.random.default_rng(n)
    s = {"positions": rng.uniform(0.0, side, (n, 3)), "atomic_numbers": rng.choice(np.array([1, 8]), n)}
    if n == 60:
        s = {"positions": rng.uniform(0.0, 0.5, (2, 3)), "atomic_numbers": np.array([1, 8]),
             "cell": np.diag([0.5, 2.0, 5.0]), "pbc": [True] * 3}
    _check(_soap(n == 60, r_cut=5.0), [s])
