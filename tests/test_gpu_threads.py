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
