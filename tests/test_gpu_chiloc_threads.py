"""chi~_loc called by two threads, each with a context of its own, on sectors whose
launches need very different amounts of shared memory (tables in shared memory
against tables in global memory): a kernel's shared-memory limit belongs to the
process, so one call must not take it away between another's setting and launch."""
import threading

import numpy as np
import pytest

from ed_solver_b200 import edk

pytestmark = pytest.mark.gpu

N = 4000


def test_two_threads_with_unequal_sectors():
    w = 1j * np.pi / 10.0 * np.array([(1, 3, 5)])
    fails, outs = [], [[], []]

    def work(i, n):
        try:
            rng = np.random.default_rng(i)
            E, M = [np.array([0.2])] + [None] * 10, [None] * 14       # one state, n in the sector above it
            E[2], M[1] = np.sort(rng.uniform(-1, 1, n)), rng.standard_normal((n, 1))
            c = edk.Context(0)
            for _ in range(N):
                outs[i].append(edk.chiloc(c, E, M, w, 10.0, 3.0, -1.0, 1, 0, 0, ops=(1,))[0][0])
            c.close()
        except Exception as e:
            fails.append(e)

    threads = [threading.Thread(target=work, args=(i, n)) for i, n in enumerate((36, 40))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fails, fails
    assert all(len(o) == N and len(set(o)) == 1 for o in outs)
