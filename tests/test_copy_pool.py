"""Host-buffer calls of several plans share the process's copy threads: calls on different plans
from different threads at once, plans made and closed in between, every product
against the oracle."""
import threading

import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import random_q, uniform_below

pytestmark = pytest.mark.gpu


def test_plans_on_several_threads_share_the_pool(cuda):
    rng = np.random.default_rng(77)
    work = []
    for n in (256, 4096, 16384, 32768):
        q = random_q(rng, 868)
        a, b = uniform_below(rng, q, n, 14), uniform_below(rng, q, n, 14)
        work.append((n, q, a, b, oracle.rns_multiply(a, b, q)))
    errors = []

    def caller(n, q, a, b, want, reps):
        try:
            for _ in range(reps):
                with polymul.Plan(n, q, coef_limbs=14) as p:  # the pool outlives each plan while any other holds it
                    for _ in range(3):
                        if not (p.multiply_host(a, b) == want).all():
                            errors.append((n, "wrong product"))
        except Exception as e:  # noqa: BLE001
            errors.append((n, repr(e)))

    threads = [threading.Thread(target=caller, args=(*w, 4)) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
        assert not t.is_alive()
    assert not errors
    # after the last plan the pool is gone; the next call makes a new one
    n, q, a, b, want = work[1]
    caller(n, q, a, b, want, 2)
    assert not errors
