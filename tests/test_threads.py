"""Plans of different sizes prepared from several threads: a launch's
shared-memory limit is the kernel's, not the last caller's."""
import threading

import numpy as np
import pytest

import geosgs
from geosgs import ensemble

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def run(jobs, turns):
    """Every job `turns` times in a thread of its own; the exceptions."""
    errors = []
    start = threading.Barrier(len(jobs))

    def work(job):
        try:
            start.wait(60)
            for _ in range(turns):
                job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def plan(k, nvars):
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=k, precision="fp64")
    model = geosgs.ExponentialVariogram(range=6.0, sill=1.0, nugget=0.1)
    p, keep = geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid((12, 11)), None, method)
    plan = geosgs.Plan(p, keep)
    if nvars > 1:
        plan.set_multivariate(np.zeros(nvars), (np.eye(nvars) + 0.1)[None])
    return plan


@pytest.mark.parametrize("sizes", [((4, 2), (32, 2), (9, 3), (8, 8)), ((20, 1), (64, 1), (40, 1), (33, 1))])
def test_plans_of_different_sizes(geosgs_lib, sizes):
    plans = [plan(k, nvars) for k, nvars in sizes]
    assert run([p.prepare for p in plans], 400) == []
    for p in plans:
        p.close()


def test_quantiles_of_different_lengths(geosgs_lib):
    rows = [torch.randn(64, r, dtype=torch.float64, device="cuda") for r in (40, 1024, 500, 130)]
    torch.cuda.synchronize()
    jobs = [lambda v=v: ensemble.quantile(v, v.shape[1], [0.5], v.shape[1]) for v in rows]
    assert run(jobs, 400) == []
    torch.cuda.synchronize()
