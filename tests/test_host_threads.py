"""The host phases on the library's kept worker threads: several callers at once, a caller after the
workers have gone, and a forked child (which inherits none of them) get what one caller gets."""
import concurrent.futures as cf
import os
import time

import numpy as np
import pytest

import fem_2d_gb300 as fg
from fem_2d_gb300 import configs


def _results(seed):
    dom = fg.Domain.from_mesh(configs.build_mesh(configs.full_scale(seed=seed, nx=9, ny=6, rounds=2, fraction=0.4)))
    plan = fg.factor_plan(dom)
    return [*fg.domain_pattern(dom), *(plan[k] for k in sorted(plan))]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b)) and len(a) == len(b)


@pytest.mark.parametrize("callers", [2, 12])
def test_concurrent_callers(callers):
    alone = [_results(s) for s in range(3)]
    with cf.ThreadPoolExecutor(callers) as ex:
        for k, got in enumerate(ex.map(lambda k: _results(k % 3), range(2 * callers))):
            assert _same(got, alone[k % 3])
    time.sleep(0.5)   # the idle workers end after 0.2 s
    assert _same(_results(1), alone[1])


def test_forked_child():
    alone = _results(0)
    pid = os.fork()
    if pid == 0:
        ok = False
        try:
            ok = _same(_results(0), alone)
        finally:
            os._exit(0 if ok else 1)
    assert os.waitpid(pid, 0)[1] == 0
    assert _same(_results(0), alone)
