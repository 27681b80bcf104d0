"""Mode changes of a server under load: each waits for the batched calls that run, and every request
is solved in one of the modes that were set."""
import threading

import numpy as np
import pytest

from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu


def test_mode_changes_under_load(bph):
    g = (40, 30, 64, 1.0 / 36.0, 2, 16)
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=140 + i)) for i in range(4)]
    s = bph.PotentialSolver(*g)
    want = []
    for r in rhos:  # what the modes converge to, and the drop-in sequence approaches
        one = bph.PotentialSolver(*g)
        want.append(one.solve_converged(r, 10, True, 1e-12, 60)[0])
        one.close()
    server = bph.Server(s, max_clients=4)
    clients = [server.open_client() for _ in rhos]
    done, errors = threading.Event(), []

    def client(i):
        try:
            last = None
            while not done.is_set():
                last, _ = server.wait(server.submit(clients[i], rhos[i]), timeout=60.0)
            # the density stands still: every mode's potential is near the converged one, and a last
            # converged request is at it
            assert rel_l2(last, want[i]) <= 0.1
        except Exception as err:  # reported by the main thread
            errors.append(err)

    threads = [threading.Thread(target=client, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for k in range(30):
        server.set_converged(nsteps=(0, 10, 6)[k % 3], tol=1e-11, max_cycles=40, mixed=k % 2 == 1)
    server.set_converged(nsteps=10, tol=1e-12, max_cycles=60)
    done.set()
    for t in threads:
        t.join(timeout=60.0)
        assert not t.is_alive()
    assert not errors, errors
    for i, r in enumerate(rhos):
        pot, _ = server.wait(server.submit(clients[i], r), timeout=60.0)
        assert rel_l2(pot, want[i]) <= 1e-9
    server.close()
    s.close()
