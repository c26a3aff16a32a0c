"""GMRES solves of different restart lengths on two handles, two host threads and two streams: each
gives the bits and the residual of the same solve run alone. (A shared-memory limit that one
solve sets for its own restart length must not take away the other's.)"""
import threading

import pytest

from plugin_navierstokes_gb300 import mesh
from test_gpu_gmres import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restarts", [(30, 10), (64, 8)])
def test_two_threads_with_their_own_restart_lengths(cuda, restarts):
    import torch

    jobs = []
    for m in restarts:
        d, vals, A, _, _ = system("quad", 9, "f64")
        rhs = torch.from_numpy(2 * mesh.uniform(7, A.shape[0]) - 1).to(cuda)
        jobs.append(dict(m=m, d=d, vals=vals, rhs=rhs, stream=torch.cuda.Stream()))
    torch.cuda.synchronize()

    def solve(j):
        x = torch.empty_like(j["rhs"])
        with torch.cuda.stream(j["stream"]):
            r = j["d"].linear_solve(j["vals"], j["rhs"], x, lin_rtol=1e-13, lin_max_iter=40, linear_solver="gmres", gmres_restart=j["m"],
                                    stream=j["stream"], raise_on_error=False)
        j["stream"].synchronize()
        return x, r

    for j in jobs:
        j["alone"] = solve(j)
    wrong = []

    def work(j):
        torch.cuda.set_device(cuda)
        for k in range(150):
            x, r = solve(j)
            if r != j["alone"][1] or not torch.equal(x, j["alone"][0]):
                wrong.append((j["m"], k, r, j["d"].last_error()))
                return

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
