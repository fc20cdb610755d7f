"""What the library's host code does when a call of the CUDA runtime fails.

Runs on the CPU: tests/fake_cudart.cpp stands in for the runtime (preloaded in
a process of its own), kernels do nothing, and the failure is the error code
that the stand-in returns."""
import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PREAMBLE = """
import ctypes as C, os, re
import numpy as np
import portal_gb300 as pg
from portal_gb300 import synth

fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_log.restype = fake.fake_live_bytes.restype = C.c_size_t
UNLIMITED = 2**64 - 1

def memory(single=UNLIMITED, total=UNLIMITED):
    fake.fake_memory(C.c_size_t(single), C.c_size_t(total))

def live():
    return fake.fake_live_bytes()

def log(clear=True):
    n = fake.fake_log(None, C.c_size_t(0))
    b = C.create_string_buffer(n + 1)
    fake.fake_log(b, C.c_size_t(n + 1))
    if clear:
        fake.fake_log_clear()
    return b.value.decode().splitlines()

def fails(code, f, *a, **k):
    try:
        f(*a, **k)
    except pg.PortalError as e:
        assert e.code == code, e
        return
    raise AssertionError("the call succeeded")

CUDA_ERR, STATE, DEPTH, NOMEM = -1, -3, -4, -6

def model(points=600, levels=4, seed=1):
    mol = synth.linear_rotor(levels)
    c = pg.Context(0)
    c.set_molecule(mol)
    c.set_cloud(synth.power_law_sphere(points, seed, mol))
    return c

def run(nth=6, nvel=8, kmax=2, n_depth=32):
    return synth.RunConfig(nth=nth, nph=nth, nvel=nvel, kmax=kmax, n_depth=n_depth, gvec=synth.gauge_vector(3))
"""


@pytest.fixture(scope="session")
def fake_cuda(built_lib, tmp_path_factory):
    from portal_gb300 import build
    inc = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-fPIC", "-shared", "-I", inc,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o", so], check=True)

    def script(body, **env):
        r = subprocess.run([sys.executable, "-c", PREAMBLE + textwrap.dedent(body)], cwd=ROOT, text=True,
                           capture_output=True, timeout=120,
                           env={**os.environ, "PYTHONPATH": ROOT, "LD_PRELOAD": so, "OMP_NUM_THREADS": "2", **env})
        assert r.returncode == 0, r.stdout + r.stderr
    return script


def test_failed_allocation_does_not_fail_the_next_call(fake_cuda):
    fake_cuda("""
        c = model()
        memory(single=14399)            # J0 takes 8 x 3 x 600 bytes
        fails(NOMEM, c.radiation_field, run())
        memory()
        c.radiation_field(run())
        memory(single=1 << 20)          # the FP64 matrices of the solve
        fails(NOMEM, c.solve_se, 2)
        memory()
        c.solve_se(2)
    """)


@pytest.mark.parametrize("nth,nvel", [(10, 8), (6, 60), (10, 60)])
def test_failed_call_does_not_keep_tables_it_replaced(fake_cuda, nth, nvel):
    """More angles or channels, then no memory for the split field: the tables
    are new and empty by then, so the next call uploads its own again."""
    fake_cuda(f"""
        c = model()
        c.radiation_field(run())
        dirs, channels = [l for l in log() if l.startswith("h2d")][-2:]
        memory(single=14399)            # J_eff takes 8 x 3 x 600 bytes
        fails(NOMEM, c.radiation_field_split, run({nth}, {nvel}))
        memory()
        log()
        c.radiation_field(run())
        sent = log()
        assert {nth} == 6 or dirs in sent, sent
        assert {nvel} == 8 or channels in sent, sent
    """)


def test_failed_solve_does_not_keep_a_program_it_replaced(fake_cuda):
    """Memory for the larger program's integers, not for its coefficients: the
    smaller one is uploaded again."""
    fake_cuda("""
        c, other = model(), model()
        sizes = []
        for ctx, kmax in ((other, 6), (c, 2)):
            ctx.radiation_field(run(kmax=kmax))
            log()
            ctx.solve_se(kmax)
            sizes.append([int(l.split()[1]) for l in log() if l.startswith("h2d")])
        (big_i, big_d), (small_i, small_d) = sizes
        memory(total=live() + big_i + big_d - small_i - small_d - 1)
        fails(NOMEM, c.solve_se, 6)
        memory()
        log()
        c.solve_se(2)
        assert [int(l.split()[1]) for l in log() if l.startswith("h2d")] == [small_i, small_d]
    """)


def test_failed_star_call_does_not_keep_items_it_replaced(fake_cuda):
    """A larger cloud whose star-mode items do not fit, then the first cloud
    again: its items are uploaded again."""
    fake_cuda("""
        star = (5000.0, 1e9, (0.0, 0.0, 0.0))
        mol = synth.linear_rotor(4)
        small, large = (synth.power_law_sphere(n, 1, mol) for n in (600, 900))
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(large)
        c.set_star(star)
        c.set_star(None)
        c.radiation_field(run())
        c.set_cloud(small)
        c.set_star(star)
        log()
        c.radiation_field(run())
        assert "h2d 4800" in [l.split(" stream")[0] for l in log()]
        c.set_star(None)
        c.set_cloud(large)
        c.set_star(star)
        memory(single=7199)
        fails(NOMEM, c.radiation_field, run())
        memory()
        c.set_cloud(small)
        log()
        c.radiation_field(run())
        assert "h2d 4800" in [l.split(" stream")[0] for l in log()]
    """)


def test_failed_batch_does_not_keep_a_workspace_it_freed(fake_cuda):
    """A network wider than the whole-network kernels: a batch that does not
    fit, then the earlier one, whose workspace is allocated again."""
    fake_cuda("""
        with pg.MLP(4, 300, 1, 3) as net:
            X, T = np.zeros((4096, 4)), np.zeros((4096, 3))
            net.gradients(X[:32], T[:32])
            memory(single=1 << 20)
            fails(NOMEM, net.gradients, X, T)
            memory()
            log()
            net.gradients(X[:32], T[:32])
            assert any(l.startswith("malloc") for l in log())
    """)


def test_star_mask_that_does_not_fit(fake_cuda):
    """No memory for the mask: set_star leaves the context as it was, a new
    cloud in star mode is refused as a whole."""
    fake_cuda("""
        star = (5000.0, 1e9, (0.0, 0.0, 0.0))
        mol = synth.linear_rotor(4)
        small, large = (synth.power_law_sphere(n, 1, mol) for n in (600, 900))
        c = model()
        memory(single=4799)
        fails(NOMEM, c.set_star, star)
        memory()
        c.radiation_field(run())        # without a star
        c.set_cloud(large)
        c.set_cloud(small)
        c.set_star(star)
        log()
        c.set_star(None)
        c.set_cloud(large)
        staging = [int(l.split()[1]) for l in log() if l.startswith("malloc")][-1]
        c.set_cloud(small)
        c.set_star(star)
        memory(total=live() + staging + 2399)
        fails(NOMEM, c.set_cloud, large)
        memory()
        fails(STATE, c.radiation_field, run())
    """)


def test_only_populations_of_a_solve_are_used(fake_cuda):
    """An image without pol_pops after an iteration that solved nothing, and
    after a solve for a smaller cloud or molecule, is refused."""
    fake_cuda("""
        def image(c):
            return c.image([1], [2], 0.3, 0.2, 4, 300.0, 0.0, 4, 0.4)
        c = model()
        memory(single=14399)            # J0 takes 8 x 3 x 600 bytes
        fails(NOMEM, c.lambda_iterate, run())
        memory()
        fails(STATE, image, c)
        c.radiation_field(run())
        fails(STATE, c.results)
        c.solve_se(2)
        image(c)
        c.results()
        mol = synth.linear_rotor(4)
        c.set_cloud(synth.power_law_sphere(900, 1, mol))
        fails(STATE, image, c)
        c.set_cloud(synth.power_law_sphere(600, 1, mol))
        image(c)
        c.lambda_iterate(run(), max_iter=1)
        image(c)
    """)


def test_field_that_a_failed_call_cleared_is_not_used(fake_cuda):
    """No memory for the walks: the field of the call before is gone by then."""
    fake_cuda("""
        c = model()
        c.radiation_field(run())
        c.solve_se(2)
        memory(single=1 << 20)
        fails(NOMEM, c.radiation_field, run(n_depth=3200))
        memory()
        fails(STATE, c.solve_se, 2)
        fails(STATE, c.results)
        c.radiation_field(run())
        c.solve_se(2)
    """)


def test_prepared_batch_runs_after_smaller_calls(fake_cuda):
    """A prepared batch's launches are not refused because a smaller batch, or a
    star-mode call, has used the same kernels since."""
    fake_cuda("""
        rc = run(nvel=64, kmax=6)
        large, small, star = model(600, 20), model(600, 14), model(600, 3)
        star.set_star((5000.0, 1e9, (0.0, 0.0, 0.0)))
        with pg.Batch(0) as a, pg.Batch(0) as b:
            a.add(large)
            a.prepare(rc)
            b.add(small)
            b.prepare(rc)
            star.radiation_field(rc)
            star.solve_se(6)
            log()
            a.run(use_graph=False)
            b.run(use_graph=False)
        launched = [l.split()[1] for l in log() if l.startswith("launch")]
        assert sum("k_radiation_field" in l for l in launched) == 2
        assert sum("k_solve_se" in l for l in launched) == 2
    """)


def test_shared_memory_limits_are_not_lowered(fake_cuda):
    """A kernel's limit is one value in every call: what one thread has set for
    its launch, another thread's call for a smaller one leaves."""
    fake_cuda("""
        for levels in (4, 14, 20):
            c = model(600, levels)
            for nvel in (8, 40, 64):
                for kmax in (2, 6):
                    c.radiation_field(run(nvel=nvel))
                    c.radiation_field_split(run(nvel=nvel))
                    c.solve_se(kmax)
        for shape in ((4, 32, 2, 3), (8, 256, 3, 40), (8, 200, 1, 250), (4, 300, 1, 3)):
            with pg.MLP(*shape) as net:
                X, T = np.zeros((70, shape[0])), np.zeros((70, shape[3]))
                net.gradients(X, T)
                net.predict(X)
        seen = {}
        for l in log():
            if l.startswith("limit"):
                seen.setdefault(l.split()[1], set()).add(int(l.split()[2]))
        assert len(seen) > 10
        assert all(len(v) == 1 for v in seen.values()), seen
    """)


def test_scratch_of_ray_items_refuses_no_call(fake_cuda):
    """Items of rays (small clouds) need a scratch for the rays' sums that whole
    nodes do not: where it does not fit the call runs whole nodes, and what it
    holds does not keep the walks or the solve after it from fitting."""
    fake_cuda("""
        def kernels():
            return [l.split()[1] for l in log() if l.startswith("launch")]
        c = model()
        c.radiation_field(run())
        walk = max(int(l.split()[1]) for l in log(False) if l.startswith("malloc"))
        assert any("k_rf_finish" in k for k in kernels())
        # the sums (540 kB) do not fit
        c = model()
        memory(total=live() + walk + 200000)
        c.radiation_field(run())
        k = kernels()
        assert any("k_radiation_field" in x for x in k) and not any("k_rf_finish" in x for x in k)
        memory()
        c.radiation_field(run())
        assert any("k_rf_finish" in x for x in kernels())
        # kept sums in the way of a solve, and of a walk of twice the cells
        model_2 = model()
        model_2.radiation_field(run())
        used = live()
        model_2.solve_se(2)
        solve = live() - used
        c.close()
        model_2.close()
        c = model()
        c.radiation_field(run())
        memory(total=live() + solve - 300000)
        c.solve_se(2)
        memory()
        c.radiation_field(run())
        memory(total=live() + walk - 300000)
        log()
        c.radiation_field(run(n_depth=64))
        assert max(int(l.split()[1]) for l in log() if l.startswith("free")) == walk
        assert live() > 2 * walk
        memory()
        # not held above 1 GB
        mol = synth.linear_rotor(20)
        c.set_molecule(mol)
        c.set_cloud(synth.power_law_sphere(14000, 1, mol))
        log()
        before = live()
        rc = run(nth=40)
        c.radiation_field(rc)
        sums = max(int(l.split()[1]) for l in log(False) if l.startswith("malloc"))
        assert sums > 1 << 30 and any("k_rf_finish" in x for x in kernels())
        assert live() < before + sums
    """)


def test_failed_copy_does_not_fail_the_next_call(fake_cuda):
    fake_cuda("""
        c = model()
        fake.fake_refuse_d2h(1)
        fails(CUDA_ERR, c.radiation_field, run())
        c.radiation_field(run())
        with pg.MLP(4, 32, 1, 3) as net, pg.Batch(0) as b:
            X = np.zeros((16, 4))
            fake.fake_refuse_d2h(1)
            fails(CUDA_ERR, net.predict, X)
            net.predict(X)
            b.add(c)
            b.prepare(run())
            fake.fake_refuse_d2h(1)
            fails(CUDA_ERR, b.run)
            b.run()
            c.radiation_field(run())
    """)


def test_failed_call_leaves_the_result_arrays(fake_cuda):
    """A copy to the host that fails: the caller's arrays keep what they held
    (large enough for their pages to be mapped ahead of the copies)."""
    fake_cuda("""
        mol = synth.linear_rotor(5)
        N = 4096
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(synth.power_law_sphere(N, 1, mol))
        rc = run()
        g = np.ascontiguousarray(rc.gvec)
        L = pg.lib()
        a = [np.full((N, 4), 0.1) for _ in range(4)]
        P = pg._p
        fake.fake_refuse_d2h(1)
        assert L.portal_radiation_field_split(c._h, rc.nth, rc.nph, rc.nvel, P(g), rc.dx, rc.n_depth, P(a[0]), P(a[1]),
                                              P(a[2]), P(a[3]), None, None) == CUDA_ERR
        assert all((x == 0.1).all() for x in a)
        c.radiation_field(rc)
        pops = np.full((10, N), 0.1)
        rates = np.full((10, 3, N), 0.1)
        fake.fake_refuse_d2h(1)
        assert L.portal_solve_se(c._h, 2, None, None, P(pops), P(rates), None, None) == CUDA_ERR
        assert (pops == 0.1).all() and (rates == 0.1).all()
        c.radiation_field(rc)
        c.solve_se(2)
        out = np.full((8, 1, 41, 31, 31), 0.1, dtype=np.float32)
        l1, l2 = np.array([1], dtype=np.int32), np.array([2], dtype=np.int32)
        fake.fake_refuse_d2h(1)
        ptrs = [out[q].ctypes.data_as(pg.P_F) for q in range(8)]
        assert L.portal_image(c._h, None, 1, P(l1, pg.P_I), P(l2, pg.P_I), 0.3, 0.2, 20, 300.0, 0.0, 15, 0.4, 0.15, 1e-4,
                              1000, *ptrs, None) == CUDA_ERR
        assert (out == np.float32(0.1)).all()
    """)


def test_result_in_the_place_of_an_input(fake_cuda):
    """Pinned memory, where the upload is still on its way when the kernel has
    been launched: JJ_20 in the array of J2 leaves the J2 that is solved for."""
    fake_cuda("""
        mol = synth.linear_rotor(5)
        cloud = synth.power_law_sphere(2048, 1, mol)
        c = pg.Context(0)
        c.set_molecule(mol)
        c.set_cloud(cloud)
        c.radiation_field(run())
        c.solve_se(2)
        rng = np.random.default_rng(1)
        J0, J2 = rng.random((2048, 4)) + 1.0, rng.random((2048, 4)) + 1.0
        keep = J2.copy()
        pops = np.zeros((10, 2048))
        rates = np.zeros((10, 3, 2048))
        P = pg._p
        fake.fake_deferred(1)
        assert pg.lib().portal_solve_se(c._h, 2, P(J0), P(J2), P(pops), P(rates), P(J2), None) == 0
        fake.fake_deferred(0)
        _, sent, _ = c.results(pops=False)
        np.testing.assert_array_equal(sent, keep)
    """)


def test_batch_times_no_launch_twice(fake_cuda):
    """Line groups of 5 and of 10 are one launch with dust or five lines at most."""
    fake_cuda("""
        def candidates(levels, dust=False):
            mol = synth.linear_rotor(levels)
            cloud = synth.power_law_sphere(600, 1, mol)
            if dust:
                cloud.dust_p = cloud.h2_dens * synth.F4(2.32e-27) / 100.0
            c = pg.Context(0)
            c.set_molecule(mol)
            c.set_cloud(cloud)
            with pg.Batch(0) as b:
                b.add(c)
                b.prepare(run())
                rows = b.config()[1]
            fake.fake_log_clear()
            return [int(r[0]) for r in rows]
        assert candidates(4)[:2] == [5, 2]            # the second row is the solve's
        assert candidates(12, dust=True)[:2] == [5, 2]
        assert candidates(12)[:3] == [5, 10, 2]
    """)


def test_batch_waits_for_its_models(fake_cuda):
    """A model's call that fails after its first launch (no memory for the walks)
    leaves kernels on its stream: the batch's own launches come after them,
    also where the model's tables are kept from before."""
    fake_cuda("""
        c = model()
        with pg.Batch(0) as b:
            b.add(c)
            b.prepare(run())
            memory(single=300 << 20)
            log()
            fails(NOMEM, c.radiation_field, run(n_depth=3200000))
            launches = [l for l in log() if l.startswith("launch")]
            memory()
            stream = launches[-1].split("stream ")[1]
            b.prepare(run())
            ops = [l for l in log() if l.startswith(("launch", "sync"))]
            first = next(i for i, l in enumerate(ops) if l.startswith("launch"))
            assert "sync stream " + stream in ops[:first]
            assert not ops[first].endswith("stream " + stream)
    """)


def test_batch_too_large_for_the_whole_network_kernels(fake_cuda):
    """Their buffers take more memory a row than the layers' one by one: where
    they do not fit, the call runs layer by layer, and the weights it leaves
    are the ones that are packed for the next."""
    fake_cuda("""
        def kernels():
            return [l.split()[1] for l in log() if l.startswith("launch")]
        with pg.MLP(8, 256, 16, 40) as net:
            X, T = np.zeros((20000, 8)), np.zeros((20000, 40))
            rows = 4 * (16 * 256 + 40)
            memory(single=int(20000 * 2.6 * rows))     # whole network 3 x, layers 2.1 x
            net.gradients(X, T)
            assert any("k_gemm_tc" in k for k in kernels())
            net.train(X, T, 1, 20000, 1e-3)
            assert any("k_adam" in k for k in kernels())
            memory()
            net.train(X, T, 1, 20000, 1e-3)
            k = kernels()
            assert any("k_mlp_rows" in x for x in k) and any("k_pack_weights" in x for x in k)
    """)


def test_training_rows_are_not_held_above_the_bound(fake_cuda):
    fake_cuda("""
        with pg.MLP(8, 16, 1, 200) as net:
            X, T = np.zeros((1400000, 8), dtype=np.float32), np.zeros((1400000, 200), dtype=np.float32)
            net.train(X[:1000], T[:1000], 1, 1000, 1e-3)
            held = live()
            net.train(X[:1000], T[:1000], 1, 1000, 1e-3)
            assert live() == held
            net.train(X, T, 1, 1000, 1e-3)      # 1.16 GB
            assert live() <= held
    """)


def test_set_cloud_makes_no_more_calls_than_the_cloud_needs(fake_cuda):
    """The walk tables come with the cloud's: one upload for both offsets, their
    padding written by the kernel that fills them."""
    fake_cuda("""
        mol = synth.linear_rotor(4)
        c = pg.Context(0)
        c.set_molecule(mol)
        cloud = synth.power_law_sphere(600, 1, mol)
        c.set_cloud(cloud)
        log()
        c.set_cloud(cloud)
        calls = [l.split()[0] for l in log()]
        assert calls.count("h2d") == 13 and calls.count("launch") == 2 and calls.count("memset") == 0, calls
    """)
