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


FLAT = {"no third vector": np.diag([9.0, 8.0, 0.0]), "no cell": np.zeros((3, 3)),
        "in a plane": np.array([[9.0, 0.0, 0.0], [0.0, 8.0, 0.0], [9.0, 8.0, 0.0]])}


@pytest.mark.parametrize("n", [1, 60, 17000])  # (the last one builds its lists in separate launches)
@pytest.mark.parametrize("pbc", [[True, True, True], [True, True, False], [False, False, True]])
@pytest.mark.parametrize("cell", FLAT)
def test_cell_without_a_volume(cell, pbc, n):
    soap = _soap(True)
    pos, Z = _atoms(n, 3)
    flat = {"positions": pos, "atomic_numbers": Z, "cell": FLAT[cell], "pbc": pbc}
    with pytest.raises(ValueError, match="singular cell"):
        soap.create(flat)
    if n == 60:
        good = dict(flat, cell=np.eye(3) * 11.0)
        want = soap.create(good)
        with pytest.raises(ValueError, match="singular cell"):
            soap.create([good, flat, good])
        with pytest.raises(ValueError, match="singular cell"):
            soap.derivatives(flat, centers=[0])
        assert torch.equal(soap.create(good), want)
        # not periodic: the cell is not read
        assert soap.create(dict(flat, pbc=[False] * 3)).shape == want.shape


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("n", [1, 60, 17000])
def test_cell_not_of_numbers(n, value):
    """No atom has a place in such a cell."""
    pos, Z = _atoms(n, 3)
    cell = np.eye(3) * 11.0
    cell[1, 1] = value
    with pytest.raises(ValueError, match="outside its periodic cell"):
        _soap(True).create({"positions": pos, "atomic_numbers": Z, "cell": cell, "pbc": [True] * 3})


@pytest.mark.parametrize("at", [0, 31, 32, 511, 512, 699])
def test_one_cell_without_a_volume_among_many(at):
    """The flag of every structure of a batch is seen, whichever thread block finds it."""
    soap = _soap(True)
    systems = [{"positions": np.ones((1, 3)), "atomic_numbers": [1], "cell": np.eye(3) * 9.0, "pbc": [True] * 3}
               for _ in range(700)]
    systems[at] = dict(systems[at], cell=np.diag([9.0, 0.0, 9.0]))
    for _ in range(20):
        with pytest.raises(ValueError, match="singular cell"):
            soap.create(systems)


@pytest.mark.parametrize("cell,pbc", [(np.diag([0.006, 9.0, 8.0]), [True] * 3),
                                      (np.diag([9.0, 8.0, 0.003]), [True] * 3),
                                      (np.array([[9.0, 0.0, 0.0], [5.0, 0.008, 0.0], [0.0, 2.0, 9.0]]), [True] * 3),
                                      (np.diag([8.0, 0.004, 9.0]), [False, True, False])])
def test_thin_cells(cell, pbc):
    """More images along an axis than a 10-bit shift holds."""
    from test_gpu_neighbors import _check
    rng = np.random.default_rng(9)
    _check(_soap(True, n_max=2, l_max=1),
           [{"positions": rng.uniform(0.0, 1.0, (3, 3)) @ cell, "atomic_numbers": np.array([1, 8, 1]), "cell": cell,
             "pbc": pbc}])


def test_cell_without_a_volume_by_rounding():
    """Vectors in a plane up to rounding: as many images as no list can hold."""
    pos, Z = _atoms(20, 3)
    cell = np.array([[3.0, 0.1, 0.7], [0.3, 2.9, 0.2], [0.0, 0.0, 0.0]])
    cell[2] = 0.1 * cell[0] + 0.7 * cell[1]
    assert abs(np.linalg.det(cell)) < 1e-12
    with pytest.raises(ValueError, match="singular cell"):
        _soap(True).create({"positions": pos, "atomic_numbers": Z, "cell": cell, "pbc": [True] * 3})


def test_jacobian_workspace_of_eight_byte_alignment():
    """The library's Jacobian in a workspace that starts 8 bytes behind a 256-byte boundary."""
    import ctypes
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    soap = _soap()
    pos, Z = _atoms(60, 4)
    s = {"positions": pos, "atomic_numbers": Z}
    want, _ = soap.derivatives(s)
    batch = _Batch(soap, [s], [None])
    pairs = _Pairs(soap, batch, _lib.NL_ALL)
    _, coeff = soap._run_descriptor(batch, pairs, _lib.OUT_PS, want_coeff=True)
    lib, need = _lib.load(), ctypes.c_int64(0)
    _lib.check(lib.soapb_jacobian_workspace(ctypes.byref(soap._basis), 60, pairs.total, 60, 0, ctypes.byref(need)))
    work = torch.empty(need.value + 256, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(want)
    status = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    _lib.check(lib.soapb_jacobian(ctypes.byref(soap._basis), 60, pairs.pair_off.data_ptr(), pairs.pairs.data_ptr(),
                                  pairs.total, coeff.data_ptr(), batch.centre_atom.data_ptr(), 60,
                                  batch.centre_attach.data_ptr(), 0, pairs.max_pairs, _lib.OUT_PS, out.data_ptr(),
                                  work.data_ptr() + 8, need.value, status.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out, want)


def _edge_cells():
    """Cells a whole number of quarter cutoffs wide between their faces, rectangular, skewed and
    rotated: lattice vectors at exactly the cutoff, atoms on the edges of bins."""
    out = []
    for i in range(60):
        rng = np.random.default_rng(i)
        quarters = rng.integers(1, 12, 3).astype(float)
        skew = np.eye(3)
        if i % 3:
            skew[1, 0], skew[2, 0], skew[2, 1] = rng.uniform(-0.5, 0.5, 3)
        turn = np.linalg.qr(rng.standard_normal((3, 3)))[0] if i % 3 == 2 else np.eye(3)
        n = 1 + i % 9
        out.append((quarters, skew, turn, rng.integers(0, 12, (n, 3)) / 12.0, rng.choice(np.array([1, 8]), n)))
    return out


def test_pairs_at_the_cutoff(monkeypatch):
    """The fill finds the pairs that the count found, also where a rounding decides; all pairs nearer
    than the cutoff and none beyond it, up to that rounding."""
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    soap = _soap(True, n_max=1, l_max=0)
    rc, empty = soap._cutoff, torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (
        lambda t: t.fill_(float("nan")) if t.is_floating_point() and t.is_cuda else t)(empty(*a, **k)))
    lists = []
    for quarters, skew, turn, frac, Z in _edge_cells():
        cell = np.diag(quarters * rc / 4) @ skew @ turn
        batch = _Batch(soap, [{"positions": frac @ cell, "atomic_numbers": Z, "cell": cell, "pbc": [True] * 3}], [None])
        p = _Pairs(soap, batch, _lib.NL_ALL)
        lists.append((cell, frac @ cell, p.pair_off.tolist(), p.pairs[:p.total].cpu().numpy()))
    monkeypatch.undo()
    for cell, pos, off, pairs in lists:
        assert np.isfinite(pairs[:, :3]).all()
        perp = 1.0 / np.linalg.norm(np.linalg.inv(cell), axis=0)
        reps = [np.arange(-k, k + 1) for k in np.ceil(rc / perp).astype(int) + 1]
        shifts = np.stack(np.meshgrid(*reps, indexing="ij"), -1).reshape(-1, 3) @ cell
        for c in range(len(pos)):
            r = np.linalg.norm((pos[None] - pos[c]) + shifts[:, None], axis=2).reshape(-1)
            got = np.sort(np.linalg.norm(pairs[off[c]:off[c + 1], :3].astype(np.float64), axis=1))
            near, far = np.sort(r[r < rc * (1 - 1e-12)]), np.sum(r <= rc * (1 + 1e-12))
            assert len(near) <= len(got) <= far
            assert np.abs(got[:len(near)] - near).max(initial=0.0) < 1e-5
            assert np.abs(got[len(near):] - rc).max(initial=0.0) < 1e-5
