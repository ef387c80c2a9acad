"""GPU: the resident-anatomy population kernel (the batched solver's default)
against the dense register kernel, bit for bit, at the edges of its division
of work: sample counts around a team's lanes, anatomies with no live cell, one
live plane, every cell live (the most units a CTA can own; stencils across
every periodic face) and scattered tissue (short runs of planes)."""
import numpy as np
import pytest

from gliomauq_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu


def _tissue(kind, n, rng):
    if kind == "ellipsoid":
        an = S.make_anatomy(n, seed=2)
        return an.p_w, an.p_g
    t = np.zeros((n, n, n))
    if kind == "full":
        t[:] = 1.0
    elif kind == "one plane":
        t[5:8] = 1.0  # live: plane 6, in every row
    elif kind == "scattered":
        t[rng.random((n, n, n)) < 0.93] = 1.0
        t[:, ::7] = 0.0
    w = rng.random((n, n, n))
    return t * w, t * (1.0 - w)


@pytest.mark.parametrize("n", [32, 64, 128])
@pytest.mark.parametrize("kind,count", [("ellipsoid", 1), ("ellipsoid", 9), ("ellipsoid", 75), ("full", 3), ("full", 17),
                                        ("one plane", 5), ("scattered", 10), ("none", 2)])
def test_resident_kernel_equals_dense(gbg, n, kind, count):
    rng = np.random.default_rng(n + count)
    pw, pg = _tissue(kind, n, rng)
    dt = S.reference_dt(n, 0.0013, n * 0.1)[0]
    smp = [(0.0013 * rng.uniform(0.3, 1.5), rng.uniform(0.01, 0.2), *rng.uniform(0, n - 1, 3), dt * rng.uniform(-1, 30))
           for _ in range(count)]
    with _lib.Handle(n, "f32", max_samples=count) as h:
        h.set_anatomy(pw, pg)
        names = [h.population_variant_name(i) for i in range(len(h.population_variants()))]
        dense = [i for i, nm in enumerate(names) if nm.startswith("k_population8<")][0]
        assert names[0].endswith("resident")
        for sigma, dt0 in ((1.0, 0.0), (0.3 * n, -0.75)):
            out = []
            for v in (dense, 0):
                h.set_population_variant(v)
                out.append(h.batch_solve(smp, n * 0.1, ic_sigma=sigma, with_loglik=False, want_phi=True, dt0=dt0))
                cells = h.last_population_cells()
                assert 0 <= cells <= int(np.sum(out[-1]["nsteps"])) * n ** 3
            assert np.array_equal(out[0]["nsteps"], out[1]["nsteps"])
            for j in range(count):
                assert np.array_equal(out[0]["phi"][j], out[1]["phi"][j]), (sigma, j)


@pytest.mark.parametrize("n", [32, 64, 128])
@pytest.mark.parametrize("steps", [(4,), (5,), (3, 4, 6), (25,)])
def test_single_solve_equals_the_dense_kernel(gbg, n, steps):
    """gbg_rd_step on the resident kernel takes any state (values outside the
    tissue and beyond [0, 1] too) to the dense kernel's bits."""
    an = S.make_anatomy(n, seed=6)
    phi = np.random.default_rng(n).uniform(-0.2, 1.2, (n, n, n))
    D = 0.1 / n ** 2
    outs = []
    for variant in (0, 1):
        with _lib.Handle(n, "f32", max_samples=1) as h:
            h.set_anatomy(an.p_w, an.p_g)
            h.set_population_variant(variant)
            h.set_phi(phi)
            for k in steps:
                h.rd_step(D, 0.1 * D, 0.05, 0.6, k)
            outs.append(h.get_phi())
    assert np.array_equal(outs[0], outs[1])
    assert outs[0].max() > 0


@pytest.mark.parametrize("kind", ["ellipsoid", "full", "scattered"])
def test_few_samples_at_32_equal_the_same_samples_among_others(gbg, kind):
    """A few samples at 32^3 run on a cluster of CTAs each; the bits are those of
    the same samples in a larger call, for one sample up to more than there are
    clusters for."""
    rng = np.random.default_rng(8)
    pw, pg = _tissue(kind, 32, rng)
    dt = S.reference_dt(32, 0.0013, 3.2)[0]
    smp = [(0.0013 * rng.uniform(0.3, 1.5), rng.uniform(0.01, 0.2), *rng.uniform(8, 24, 3), dt * rng.uniform(0, 40))
           for _ in range(24)]
    with _lib.Handle(32, "f32", max_samples=24) as h:
        h.set_anatomy(pw, pg)
        whole = h.batch_solve(smp, 3.2, with_loglik=False, want_phi=True)["phi"]
        for a, b in ((0, 1), (1, 3), (3, 9), (9, 16), (16, 24)):
            part = h.batch_solve(smp[a:b], 3.2, with_loglik=False, want_phi=True)["phi"]
            assert np.array_equal(part, whole[a:b])


@pytest.mark.parametrize("n", [32, 64, 128])
def test_negative_step_coefficients_equal_the_dense_kernel(gbg, n):
    """On the scaled time grid a strongly negative rho makes the step, and so the
    coefficient of the full steps, negative, with a last (here the only) step of
    the whole time: a sample like any other."""
    an = S.make_anatomy(n, seed=2)
    c = 0.5 * (n - 1)
    smp = [(0.0013, -3.0, c, c + 0.4, c - 0.3, 0.8), (0.0013, 0.05, c, c, c, 4.0), (0.0009, -2.0, c + 1, c, c, 0.5)]
    with _lib.Handle(n, "f32", max_samples=len(smp)) as h:
        h.set_anatomy(an.p_w, an.p_g)
        names = [h.population_variant_name(i) for i in range(len(h.population_variants()))]
        out = []
        for v in ([i for i, nm in enumerate(names) if nm.startswith("k_population8<")][0], 0):
            h.set_population_variant(v)
            out.append(h.batch_solve(smp, n * 0.1, with_loglik=False, want_phi=True, dt0=-0.75))
    assert list(out[0]["nsteps"]) == list(out[1]["nsteps"]) and out[0]["nsteps"][0] == 1
    for j in range(len(smp)):
        assert out[0]["phi"][j].max() > 0
        assert np.array_equal(out[0]["phi"][j], out[1]["phi"][j]), j
