"""Calls of several threads and streams on one object."""
import threading

import numpy as np
import pytest
import torch

from cusoap_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _soap(**over):
    from cusoap_b200 import SOAP
    return SOAP(**{**dict(species=[1, 8], r_cut=2.5, n_max=2, l_max=1, sigma=0.3), **over})


def _run(work, n):
    errors = []

    def guarded(i):
        try:
            work(i)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(i,)) for i in range(n)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    if errors:
        raise errors[0]


@pytest.mark.parametrize("own_stream", [False, True])
def test_work_queues(own_stream):
    """More centres than resident warps: the descriptor and the adjoint take them from a queue."""
    soap = _soap()
    systems = [W.water_cluster(17, 17, 17 + k, seed=k) for k in range(3)]
    pos = [torch.as_tensor(s["positions"], device="cuda") for s in systems]
    w = torch.linspace(-1.0, 1.0, soap.get_number_of_features(), device="cuda")

    def step(i):
        p = pos[i].clone().requires_grad_(True)
        D = soap.create(dict(systems[i], positions=p))
        (D @ w).sum().backward()
        return D.detach(), p.grad

    want = [step(i) for i in range(3)]
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.current_stream()):
            for _ in range(12):
                D, g = step(i)
                assert torch.equal(D, want[i][0])
                # FP32 atomic sums of about 40 edges in another order
                assert float((g - want[i][1]).norm() / want[i][1].norm()) < 2e-6

    _run(work, 3)


class _Emptied(list):
    """A pool whose last buffer another thread takes between a look at it and the pop."""

    def __bool__(self):
        return True

    def __len__(self):
        return 1

    def pop(self, *a):
        raise IndexError("pop from empty list")


def test_pool_emptied_by_another_thread():
    soap, s = _soap(), W.water_cluster(2, 2, 2, seed=1)
    want = soap.create(s)
    soap._stage_pool, soap._stats_pool = _Emptied(), _Emptied()
    assert torch.equal(soap.create(s), want)


def test_topology_of_an_upload_that_waits():
    """Arrays whose copy still waits on one stream are not used on another, and their staging buffer
    is not given out again, whoever waits for what."""
    from cusoap_b200 import _lib
    from cusoap_b200.soap import _Batch, _Pairs
    soap, s = _soap(), W.water_cluster(3, 3, 3, seed=1)
    want = _soap().create(s)
    sysd = dict(s, positions=torch.as_tensor(s["positions"], device="cuda"))
    torch.cuda.synchronize()
    first, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(200_000_000)
        batch = _Batch(soap, [sysd], [None])
    assert soap._topology is None and not soap._stage_pool
    with torch.cuda.stream(other):
        assert torch.equal(soap.create(sysd), want)
    assert len(soap._stage_pool) == 1 and soap._topology["dev"] is not batch._dev
    with torch.cuda.stream(first):
        pairs = _Pairs(soap, batch, _lib.NL_CREATE)
        assert torch.equal(soap._run_descriptor(batch, pairs, _lib.OUT_PS)[0], want)
    assert len({p.data_ptr() for p in soap._stage_pool}) == len(soap._stage_pool) == 2
    with torch.cuda.stream(other):  # the arrays of the first stream's upload, complete by now
        assert torch.equal(soap.create(sysd), want)


def test_lists_of_systems():
    """Every call splits its output by its own counts."""
    soap = _soap()
    lists = [[W.water_cluster(1, 1, k + i, seed=k) for k in range(1, 4 + i)] for i in range(4)]
    want = [soap.create(v) for v in lists]

    def work(i):
        for _ in range(40):
            got = soap.create(lists[i])
            assert len(got) == len(want[i]) and all(torch.equal(a, b) for a, b in zip(got, want[i]))
            flat, off = soap.create_flat(lists[i])
            assert np.diff(off.numpy()).tolist() == [len(w) for w in want[i]]
            assert torch.equal(flat, torch.cat(want[i]))

    _run(work, 4)


class _Late:
    """A graph whose replay waits on the device for about 50 ms first."""

    def __init__(self, graph):
        self.graph = graph

    def replay(self):
        torch.cuda._sleep(100_000_000)
        self.graph.replay()


@pytest.mark.parametrize("late", ["g_desc", "g_bwd"])
def test_plan_on_another_stream(late):
    """A call of a plan on another stream than the last waits for that one's graphs."""
    soap, s = _soap(), W.water_cluster(4, 4, 4, seed=1)
    plan = soap.batch([s])
    pos = torch.as_tensor(s["positions"], device="cuda")
    moved = pos + 0.05 * torch.sin(torch.arange(pos.numel(), device="cuda").reshape(pos.shape))
    w = torch.linspace(-1.0, 1.0, soap.get_number_of_features(), device="cuda").expand(len(pos), -1)
    want = plan.create(moved).clone()
    first, other = torch.cuda.Stream(), torch.cuda.Stream()
    setattr(plan, late, _Late(getattr(plan, late)))
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(first):
        plan.create(pos)
        if late == "g_bwd":
            plan.forces_from(w)
        done.record()
    with torch.cuda.stream(other):
        got = plan.create(moved)  # returns when its pair lists are there
        assert done.query()
        assert torch.equal(got, want)


def test_plan_is_made_anew_when_its_graphs_are_done():
    soap, s = _soap(), W.water_cluster(4, 4, 4, seed=1)
    plan = soap.batch([s], headroom=1.0)
    pos = torch.as_tensor(s["positions"], device="cuda")
    plan.g_desc = _Late(plan.g_desc)
    build, done = plan._build, torch.cuda.Event()

    def checked(capacity):
        assert plan.finished.query()
        done.record()
        build(capacity)

    plan._build = checked
    with torch.cuda.stream(torch.cuda.Stream()):
        got = plan.create(pos * 0.5)
        assert done.query() and torch.equal(got, soap.create(dict(s, positions=pos * 0.5)))
