"""Contexts of different meshes beside each other: the one-launch solve's kernel is one
function of the process, launched with another amount of shared memory by every
mesh, so a small mesh's solve must not refuse a large one's. 150^2 and 180^2 Q1
need more than the 48 KiB that a kernel may ask for by default, 20^2 Q1 less."""
import threading

import numpy as np
import pytest

from helpers import setup_case, tgv
from lbfem_gpu import make_params

pytestmark = pytest.mark.gpu

PRM = dict(cg_tolerance=1e-10)


def _solver(n, streaming="tg2"):
    import lbfem_gpu

    tc, m = tgv(n)
    return setup_case(lbfem_gpu.Solver, tc, m, make_params("bardow", "cg", streaming=streaming, **PRM),
                      m.time_step(0.3), tc.relaxation_time())


@pytest.mark.parametrize("streaming", ["tg2", "tg3-split"])
def test_threads_with_meshes_of_different_sizes(gpu_lib, streaming):
    """Host threads with a context each that create, step, solve and drop, one of them on a
    large mesh: no call fails, and each result is that of the same call alone, bitwise."""
    import torch

    kw = {} if streaming == "tg2" else {"e": (1.0, 0.0), "tg3_coefficient": 1e-6}
    errors, large_done = [], threading.Event()

    def once(n, rhs, x, solves):
        h = _solver(n, streaming)
        h.step(3)
        for _ in range(solves):
            x.zero_()
            torch.cuda.current_stream().synchronize()
            h.mass_solve_dev(x.data_ptr(), rhs.data_ptr(), **kw)
        out = h.get_populations(), x.cpu().numpy()
        h.close()
        return out

    def data(n):
        r = torch.from_numpy(np.random.default_rng(n).standard_normal((n + 1) ** 2)).cuda()
        return r, torch.zeros_like(r)

    alone = {n: once(n, *data(n), 1) for n in (180, 20)}

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                rhs, x = data(n)
                for k in range(4) if n == 180 else iter(lambda: large_done.is_set(), True):
                    out = once(n, rhs, x, 1000 if n == 180 else 200)
                    for a, b in zip(out, alone[n]):
                        assert np.array_equal(a, b)
        except BaseException as e:  # noqa: BLE001
            errors.append((n, e))
        finally:
            if n == 180:
                large_done.set()

    threads = [threading.Thread(target=work, args=(n,)) for n in (180, 20, 20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_batch_of_large_and_small_fp64_instances(gpu_lib):
    """One batch graph with FP64 instances of several sizes (recorded largest first): every
    instance ends where its own steps take it, bitwise."""
    import lbfem_gpu

    sizes = (20, 180, 9, 150)
    batched, single = [_solver(n) for n in sizes], [_solver(n) for n in sizes]
    b = lbfem_gpu.Batch(batched)
    b.step(4)
    b.step(3)
    b.close()
    for hb, hs in zip(batched, single):
        hs.step(7)
        assert np.array_equal(hb.get_populations(), hs.get_populations())
