"""Contexts of their own on several host threads (GPU): a context is one
thread's, the process's are many."""
import threading

import numpy as np
import pytest

from portal_gb300 import synth

pytestmark = pytest.mark.gpu


def test_images_of_several_contexts_at_once(built_lib):
    """Three threads image different lines again and again: each gets
    what it gets alone."""
    import portal_gb300 as pg

    mol = synth.linear_rotor(5)
    cloud = synth.power_law_sphere(1500, 3, mol, t_law="loglinear", b_random=0.3)
    rc = synth.RunConfig(nth=4, nph=4, nvel=8, kmax=2, n_depth=500, gvec=synth.gauge_vector(3))

    def context(k):
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(cloud)
        c.radiation_field(rc)
        c.solve_se(rc.kmax)
        return c, lambda: c.image([1 + k], [2 + k], 0.4, 0.3, 8, 150.0, 0.0, 6, 0.5)[0]

    jobs = [context(k) for k in range(3)]
    want = [f() for _, f in jobs]
    wrong = [0] * len(jobs)

    def loop(k):
        for _ in range(60):
            wrong[k] += not np.array_equal(jobs[k][1](), want[k], equal_nan=True)

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, _ in jobs:
        c.close()
    assert wrong == [0] * len(jobs)


def test_node_loops_of_several_contexts_at_once(built_lib):
    """Node loops of different sizes on the same kernels: equal bits to each
    alone."""
    import portal_gb300 as pg

    def context(k):
        mol = synth.linear_rotor(4 + 5 * k)
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(synth.power_law_sphere(300 + 200 * k, k, mol, t_law="loglinear", b_random=0.3))
        rc = synth.RunConfig(nth=6, nph=6, nvel=8 + 12 * k, kmax=2 + 2 * k, n_depth=500, gvec=synth.gauge_vector(3))
        return c, lambda: c.radiation_field_split(rc)[:4] + c.solve_se(rc.kmax)

    jobs = [context(k) for k in range(3)]
    want = [f() for _, f in jobs]
    wrong = [0] * len(jobs)

    def loop(k):
        for _ in range(40):
            wrong[k] += not all(np.array_equal(a, b) for a, b in zip(jobs[k][1](), want[k]))

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, _ in jobs:
        c.close()
    assert wrong == [0] * len(jobs)
