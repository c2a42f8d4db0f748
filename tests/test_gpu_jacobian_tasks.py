"""The Jacobian's compute tasks: whole rows in batches of staged entries, rows
with more entries than a batch (images of a tiny cell), and the row of a centre
that moves with its atom."""
import numpy as np
import pytest
import torch

from cusoap_b200 import workloads as W
from oracle.soap_oracle import OracleSOAP, rel_l2

pytestmark = pytest.mark.gpu

# FP32 values (2^-24 relative each) summed over at most some hundred edges, relative to the block
TOL = 1e-5

BASES = [dict(r_cut=5.0, n_max=4, l_max=3, sigma=0.5), dict(r_cut=4.0, n_max=3, l_max=2, sigma=0.5),
         dict(r_cut=4.0, n_max=8, l_max=6, sigma=0.5), dict(r_cut=3.0, n_max=10, l_max=9, sigma=0.5)]


def _soap(**kw):
    from cusoap_b200 import SOAP
    return SOAP(species=[1, 8], **kw)


@pytest.mark.parametrize("average", ["off", "cc"])
@pytest.mark.parametrize("basis", BASES)
def test_fixed_centres_vs_oracle(basis, average):
    s = W.water_cluster(3, 3, 3, seed=4)
    centres, include = [0, 40, 80], [0, 3, 4, 40, 41, 77, 80]
    J = _soap(average=average, **basis).derivatives(s, centers=centres, include=include, return_descriptor=False)
    Jo, _ = OracleSOAP(species=[1, 8], average=average, **basis).derivatives(
        s["positions"], s["atomic_numbers"], centers=centres, include=include)
    for k in range(3):
        assert rel_l2(J[k].cpu().numpy(), Jo[k]) < TOL


def _structure(kind):
    if kind == "cluster":
        return W.water_cluster(4, 4, 4, seed=2)
    if kind == "tiny":  # every atom of the cell many times within the cutoff
        return {"positions": np.array([[0.0, 0.0, 0.0], [1.1, 0.9, 1.3], [0.2, 1.9, 0.4]]),
                "atomic_numbers": np.array([8, 1, 1]), "pbc": [True] * 3,
                "cell": np.array([[2.9, 0.0, 0.0], [0.3, 3.0, 0.0], [0.1, -0.2, 3.1]])}
    return W.water_box(20, 8.5, seed=3)


@pytest.mark.parametrize("average", ["off", "cc"])
@pytest.mark.parametrize("kind", ["cluster", "tiny", "box"])
@pytest.mark.parametrize("basis", BASES)
def test_moving_centres(basis, kind, average):
    """With attached centres the rows of a centre sum to zero, the other rows
    are those of fixed centres, and an excluded centre atom leaves them so."""
    s = _structure(kind)
    soap = _soap(average=average, periodic=kind != "cluster", **basis)
    n = len(s["atomic_numbers"])
    centres = [0, 1, n - 1]
    Ja = soap.derivatives(s, centers=centres, attach=True, return_descriptor=False).double()
    Jf = soap.derivatives(s, centers=centres, return_descriptor=False).double()
    inc = [i for i in range(n) if i != 1]
    Jx = soap.derivatives(s, centers=centres, include=inc, attach=True, return_descriptor=False).double()
    for k, c in enumerate(centres):
        scale = Ja[k].abs().sum(0).norm()
        assert Ja[k].sum(0).norm() <= TOL * scale
        rest = [i for i in range(n) if i != c]
        assert (Ja[k, rest] - Jf[k, rest]).norm() <= TOL * Jf[k, rest].norm()
        keep = [i for i in inc if i != c]
        assert (Jx[k, [inc.index(i) for i in keep]] - Ja[k, keep]).norm() <= TOL * Ja[k, keep].norm()
    # the centre whose atom is left out has no centre row; the others keep theirs
    assert (Jx[0, 0] - Ja[0, 0]).norm() <= TOL * Ja[0, 0].norm()
    assert torch.isfinite(Jx).all()


@pytest.mark.parametrize("n_max,l_max,n_species", [(1, 0, 1), (1, 1, 2), (1, 2, 2), (1, 0, 2), (3, 2, 2), (2, 1, 2)])
def test_zero_rows_of_any_length(monkeypatch, n_max, l_max, n_species):
    """Runs of zero rows that start and end anywhere within 16 bytes: every element is written."""
    s = W.water_cluster(1, 1, 9, seed=6)
    if n_species == 1:
        s = dict(s, atomic_numbers=np.ones(len(s["atomic_numbers"]), int))
    basis = dict(species=[1, 8][:n_species], r_cut=2.5, n_max=n_max, l_max=l_max, sigma=0.3)
    n = len(s["atomic_numbers"])
    centres, include = [0, 7, n - 1], [i for i in range(n) if i % 7 != 3]
    from cusoap_b200 import SOAP
    soap, empty = SOAP(**basis), torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (lambda t: t.fill_(float("nan")) if t.is_floating_point() else t)(
        empty(*a, **k)))
    J = soap.derivatives(s, centers=centres, include=include, return_descriptor=False)
    monkeypatch.undo()
    Jo, _ = OracleSOAP(**basis).derivatives(s["positions"], s["atomic_numbers"], centers=centres, include=include)
    J, far = J.cpu().numpy(), (np.asarray(Jo) == 0.0).all((2, 3))
    assert far.any(1).all() and not far.all(1).any()
    assert (J[far] == 0.0).all()
    for k in range(3):
        assert rel_l2(J[k], Jo[k]) < TOL


@pytest.mark.parametrize("average", ["off", "cc"])
@pytest.mark.parametrize("n_max,l_max", [(3, 0), (2, 1), (4, 2), (4, 3), (4, 4), (2, 4)])
def test_many_centres_of_few_features(n_max, l_max, average):
    """More centres than three blocks on every SM take: the blocks of centres evaluated alone."""
    s = W.water_cluster(5, 5, 8, seed=8)
    soap = _soap(r_cut=2.5, n_max=n_max, l_max=l_max, sigma=0.3, average=average)
    assert len(s["atomic_numbers"]) == 600
    for attach in (False, True):
        J = soap.derivatives(s, attach=attach, return_descriptor=False)
        pick = list(range(0, 600, 37))
        few = soap.derivatives(s, centers=pick, attach=attach, return_descriptor=False)
        assert torch.equal(J[pick] == 0.0, few == 0.0)
        assert (J[pick].double() - few.double()).norm() <= TOL * few.double().norm()
