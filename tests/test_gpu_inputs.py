"""The host path of a call: index centres from host and device positions,
species numbers, positions left as they are, threads sharing an object."""
import threading

import numpy as np
import pytest
import torch

from cusoap_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _soap(**over):
    from cusoap_b200 import SOAP
    return SOAP(**{**W.CONFIGS["cluster192"], **over})


@pytest.mark.parametrize("device_positions", [False, True])
@pytest.mark.parametrize("centres", [[0], [80, 3, 3, 17], range(5, 9), np.array([1, 2]), [-1, 4], []])
def test_index_centres(centres, device_positions):
    """Rows of index centres are those of the same Cartesian centres and, for
    indices from 0, those of every atom as a centre (same pair lists)."""
    s = W.water_cluster(3, 3, 3, seed=1)
    soap = _soap()
    sysd = dict(s, positions=torch.as_tensor(s["positions"], device="cuda")) if device_positions else s
    got = soap.create(sysd, centers=centres)
    idx = [int(c) for c in centres]
    assert got.shape[0] == len(idx)
    every = soap.create(s)
    for row, i in zip(got, idx):
        if i >= 0:
            assert torch.equal(row, every[i])
        else:  # counted from the end, without the atom's own Gaussian: no counterpart among the atoms' rows
            assert not torch.equal(row, every[i])
    if idx and min(idx) >= 0:
        mixed = soap.create(sysd, centers=idx + [s["positions"][idx[0]].tolist()])  # one Cartesian centre: the general path
        assert torch.equal(mixed[:-1], got) and torch.equal(mixed[-1], got[0])
        lists = soap.create_flat([sysd, sysd], centers=[idx, None])[0]
        assert torch.equal(lists[:len(idx)], got) and torch.equal(lists[len(idx):], every)


@pytest.mark.parametrize("device_positions", [False, True])
@pytest.mark.parametrize("bad", [81, -82])
def test_index_out_of_range(bad, device_positions):
    s = W.water_cluster(3, 3, 3, seed=1)
    if device_positions:
        s = dict(s, positions=torch.as_tensor(s["positions"], device="cuda"))
    with pytest.raises(IndexError):
        _soap().create(s, centers=[0, bad])


@pytest.mark.parametrize("numbers", [(1, 8), (3, 2000), (-7, 5)])
def test_species_numbers(numbers):
    s = W.water_cluster(2, 2, 2, seed=1)
    ref = _soap().create(s)
    Z = np.where(s["atomic_numbers"] == 1, numbers[0], numbers[1])
    assert torch.equal(_soap(species=list(numbers)).create(dict(s, atomic_numbers=Z)), ref)
    with pytest.raises(ValueError, match="not in species list"):
        _soap(species=list(numbers)).create(dict(s, atomic_numbers=np.where(Z == numbers[0], 999, Z)))


def test_positions_are_not_written():
    """The caller's device positions are read in place; a plan has its own."""
    s = W.water_cluster(3, 3, 3, seed=2)
    pos = torch.as_tensor(s["positions"], device="cuda")
    keep = pos.clone()
    soap = _soap()
    out = soap.create(dict(s, positions=pos))
    plan = soap.batch([dict(s, positions=pos)])
    moved = plan.create(pos + 0.1).clone()
    assert torch.equal(pos, keep)
    # strided and float32 positions take a copy
    wide = torch.zeros((len(pos), 5), dtype=torch.float64, device="cuda")
    wide[:, 1:4] = pos
    assert torch.equal(soap.create(dict(s, positions=wide[:, 1:4])), out)
    p32 = pos.float()
    assert torch.equal(soap.create(dict(s, positions=p32)), soap.create(dict(s, positions=p32.double())))
    assert torch.equal(plan.create(pos), out) and moved.shape == out.shape


def test_threads_share_an_object():
    """Calls of several threads on one object (default stream) do not mix
    their staging or summary buffers: structures of different sizes."""
    soap = _soap()
    systems = [W.water_cluster(2, 2, k, seed=k) for k in (1, 2, 3, 4)]
    want = [soap.create(s) for s in systems]
    wrong = []

    def work(i):
        for _ in range(20):
            if not torch.equal(soap.create(systems[i]), want[i]):
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
