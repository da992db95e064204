"""GPU: force fields of different sizes in two host threads.

Their kernels' limits on dynamic shared memory are the process's; the Hessian products of
C20H42 (55 KB) and of C4H10 (51 KB) exceed the default limit, each by another amount, and
so do the gradients of C172H346 (plain 50 KB) and of C190H382 (52 KB). Every call of either thread
must succeed and give its own force field's result, bit for bit."""
import threading

import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q

pytestmark = pytest.mark.gpu


def race(fields, call, reps):
    rng = np.random.default_rng(0)
    x = [f.xyz[None] + rng.normal(0, 0.02, (2,) + f.xyz.shape) for f, _ in fields]
    want = [call(g, a) for (_, g), a in zip(fields, x)]
    bad = []

    def work(i):
        try:
            for _ in range(reps):
                got = call(fields[i][1], x[i])
                if not all(np.array_equal(u, v) for u, v in zip(got, want[i])):
                    bad.append((i, "differs"))
        except Exception as e:  # noqa: BLE001
            bad.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(fields))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


@pytest.mark.parametrize("sizes,call,reps", [
    ((20, 4), lambda g, x: g.hvp(x, np.ones_like(x)), 60),
    ((172, 190), lambda g, x: g.egrad(x, "fp64"), 8)])
def test_two_threads(require_gpu, sizes, call, reps):
    ffs = [Q.alkane(nc=n) for n in sizes]
    fields = [(f, QMDFFForceField(f)) for f in ffs]
    race(fields, call, reps)
    for _, g in fields:
        g.close()
