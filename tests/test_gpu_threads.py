"""GPU: handles on threads of their own, with anatomies of different extent, so
that the same kernels are launched with different amounts of shared memory at
once: no launch fails or takes another path for it, and every result is the
one the handle gives alone."""
import threading

import numpy as np
import pytest

from gliomauq_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu
LIK = (0.0025, 1.0, 0.7, 0.25, 0.09)


def _side_by_side(calls):
    """Each of the calls over and over on a thread of its own; the lists of their
    results, an exception in place of a result that failed."""
    outs = [[] for _ in calls]
    start = threading.Barrier(len(calls))

    def work(call, out):
        start.wait()
        for _ in range(40):
            try:
                out.append(call())
            except _lib.GbgError as e:
                out.append(e)

    ts = [threading.Thread(target=work, args=a) for a in zip(calls, outs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return outs


def _anatomies(n):
    """Every cell tissue; three planes of it; an ellipsoid."""
    full = np.full((2, n, n, n), 0.5)
    thin = np.zeros((2, n, n, n))
    thin[:, n // 2 - 2:n // 2 + 3] = 0.5
    an = S.make_anatomy(n, seed=2)
    return [full, thin, (an.p_w, an.p_g)]


def _check(calls):
    alone = [c() for c in calls]
    for k, out in enumerate(_side_by_side(calls)):
        for r in out:
            assert not isinstance(r, Exception), (k, r)
            for x, y in zip(r, alone[k]):
                assert np.array_equal(x, y), k


@pytest.mark.parametrize("n,graphs", [(32, False), (64, False), (64, True), (128, False)])
def test_batched_solves(gbg, n, graphs):
    c = 0.5 * (n - 1)
    dt = S.reference_dt(n, 0.0013, n * 0.1)[0]
    smp = [(0.0013, 0.05 + 0.01 * i, c + 0.2 * i, c, c, 5 * dt) for i in range(6)]
    hs = [_lib.Handle(n, "f32", max_samples=6) for _ in range(3)]
    try:
        for h, a in zip(hs, _anatomies(n)):
            h.set_anatomy(*a)
            h.set_batch_graphs(graphs)
        _check([lambda h=h, k=k: h.batch_solve(smp[:k], n * 0.1, with_loglik=False, want_phi=True)["phi"]
                for h, k in zip(hs, (6, 2, 4))])
    finally:
        for h in hs:
            h.close()


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
def test_exact_steps_in_one_launch(gbg, prec):
    sizes = (8, 24, 48)
    hs = [_lib.Handle(n, prec) for n in sizes]
    phi = [np.random.default_rng(n).uniform(0, 1, (n, n, n)).astype(np.float32).astype(float) for n in sizes]

    def call(h, p):
        h.set_phi(p)
        before = h.launch_count()
        h.rd_step(0.1 / h.n ** 2, 0.01 / h.n ** 2, 0.05, 0.6, 9)
        return h.get_phi(), h.launch_count() - before

    try:
        for h in hs:
            h.set_anatomy(np.full((h.n,) * 3, 0.6), np.full((h.n,) * 3, 0.3))
        for h, p in zip(hs, phi):
            call(h, p)  # the tables and the list
        _check([lambda h=h, p=p: call(h, p) for h, p in zip(hs, phi)])
    finally:
        for h in hs:
            h.close()


def test_gradients_at_128(gbg):
    n, c = 128, 63.5
    hs = [_lib.Handle(n, "f32", max_samples=2) for _ in range(2)]
    smp = [(0.0013, 0.05, c, c, c, 3.0)]
    try:
        for h, a in zip(hs, _anatomies(n)[1:]):
            h.set_anatomy(*a)
            an = S.make_anatomy(n, seed=2)
            obs = S.make_observations(np.clip(S.gaussian_ic(an, c, c, c, peak=0.9, sigma=4.0), 0, 1), an, seed=3,
                                      centre_xyz=(c, c, c), radius_vox=20.0)
            h.set_observations(obs.pet, obs.t1, obs.t2, obs.points, LIK)
        calls = [lambda h=h: h.adjoint_grad(smp, -1.0, n * 0.1) for h in hs]
        alone = [f() for f in calls]
        for k, out in enumerate(_side_by_side(calls)):
            for r in out:
                assert not isinstance(r, Exception), (k, r)
                assert np.array_equal(r[0], alone[k][0])
                # the sensitivities' FP64 atomics add in any order
                assert np.allclose(r[1], alone[k][1], rtol=1e-9, atol=1e-12 * np.abs(alone[k][1]).max())
    finally:
        for h in hs:
            h.close()
