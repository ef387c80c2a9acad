"""GPU: the CUDA step through the C ABI against the reference (golden
fixtures) and the oracle. Exact modes must be bit-identical; the fast FP32
path must stay within the stated error of the FP64 reference."""
import hashlib

import numpy as np
import pytest

from gliomauq_gb300 import _lib, synthetic as S
from helpers import boundary_layer, golden_json, golden_npz, rel_l2

pytestmark = pytest.mark.gpu

# Fast FP32 path: relative L2 error of the final density against the FP64
# reference after a full config-1 solve (64^3, 237 steps).
F32_REL_L2_TOL = 1e-5


def _sha(a):
    return hashlib.sha256(np.ascontiguousarray(a, dtype="<f8").tobytes()).hexdigest()


@pytest.mark.parametrize("k", [1, 10, 60])
@pytest.mark.parametrize("prec,variant", [("f64", "f64"), ("f32ref", "f32")])
def test_exact_modes_bitwise_vs_reference_golden(gbg, prec, variant, k):
    d = golden_npz("rd32.npz")
    with _lib.Handle(32, prec) as h:
        h.set_anatomy(d["p_w"], d["p_g"])
        h.set_phi(d["phi0"])
        h.rd_step(float(d[f"Dw_{variant}"]), float(d[f"Dg_{variant}"]), float(d["rho"]),
                  float(d[f"dt_{variant}"]), k)
        out = h.get_phi()
    assert np.array_equal(out, d[f"phi_{variant}_{k}"].astype(np.float64))


@pytest.mark.parametrize("prec,variant", [("f64", "f64"), ("f32ref", "f32")])
def test_config1_full_run_bitwise(gbg, prec, variant):
    meta = golden_json("c1_64.json")
    a = golden_npz("anatomy64.npz")
    with _lib.Handle(64, prec) as h:
        h.set_anatomy(a["p_w"], a["p_g"])
        h.set_phi(a["phi0"])
        ns, dt = h.run(meta["Dw_file"], meta["rho"], meta["tend"], meta["L"])
        out = h.get_phi()
    assert ns == meta[variant]["steps"] and dt == meta[variant]["dt"]
    assert _sha(out) == meta[variant]["sha256"]


def test_fast_f32_error_against_fp64_reference(gbg, oracle_lib):
    meta = golden_json("c1_64.json")
    a = golden_npz("anatomy64.npz")
    with _lib.Handle(64, "f32") as h:
        h.set_anatomy(a["p_w"], a["p_g"])
        h.set_phi(a["phi0"])
        ns, dt = h.run(meta["Dw_file"], meta["rho"], meta["tend"], meta["L"])
        out = h.get_phi()
    assert ns == 237 and dt == meta["f64"]["dt"]
    dt64, dw, dg = S.reference_dt(64, meta["Dw_file"], meta["L"])
    ref = oracle_lib.rd_solve(a["p_w"], a["p_g"], a["phi0"], dw, dg, meta["rho"], dt64, ns)
    assert _sha(ref) == meta["f64"]["sha256"]
    err = rel_l2(out, ref)
    print(f"fast f32 vs FP64 reference, config 1: rel L2 = {err:.3e}")
    assert err <= F32_REL_L2_TOL
    brain = (a["p_w"].astype(np.float64) + a["p_g"]) > 0
    assert np.all(out[boundary_layer(brain)] == 0.0) and np.all(out[~brain] == 0.0)


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
@pytest.mark.parametrize("seed", [0, 1])
def test_exact_modes_vs_live_oracle_random(gbg, oracle_lib, prec, seed):
    """Random anatomy (including non-tissue holes), random densities with values
    below 0 and above 1, odd grid size: bitwise equal to the oracle."""
    rng = np.random.default_rng(seed)
    n = 24 + 3 * seed
    pw = rng.random((n, n, n)) * (rng.random((n, n, n)) > 0.15)
    pg = (1 - pw) * (rng.random((n, n, n)) > 0.1)
    phi = rng.uniform(-0.2, 1.2, size=(n, n, n))
    if prec == "f32ref":
        pw, pg, phi = (x.astype(np.float32).astype(np.float64) for x in (pw, pg, phi))
    Dw, Dg, rho, dt = 2.1e-4, 2.1e-5, 0.08, 0.5 * (1 / n) ** 2 / (6 * 2.1e-4)
    with _lib.Handle(n, prec) as h:
        h.set_anatomy(pw, pg)
        h.set_phi(phi)
        h.rd_step(Dw, Dg, rho, dt, 7)
        out = h.get_phi()
    ref = oracle_lib.rd_solve(pw, pg, phi, Dw, Dg, rho, dt, 7, prec=prec)
    assert np.array_equal(out, ref.astype(np.float64))


@pytest.mark.parametrize("prec", ["f64", "f32ref", "f32"])
def test_zero_state_stays_zero_and_full_tissue(gbg, prec):
    n = 32
    with _lib.Handle(n, prec) as h:
        h.set_anatomy(np.full((n,) * 3, 0.6), np.full((n,) * 3, 0.4))
        h.set_phi(np.zeros((n,) * 3))
        h.rd_step(1e-4, 1e-5, 0.1, 1.0, 3)
        assert np.all(h.get_phi() == 0.0)
        # uniform density in an all-tissue periodic box follows the logistic ODE
        h.set_phi(np.full((n,) * 3, 0.25))
        h.rd_step(1e-4, 1e-5, 0.1, 1.0, 1)
        u = h.get_phi()
    exp = 0.25 + 1.0 * 0.1 * 0.25 * 0.75
    assert np.allclose(u, exp, rtol=1e-6)


def test_errors_are_reported(gbg):
    with _lib.Handle(32, "f64") as h:
        with pytest.raises(_lib.GbgError) as e:
            h.rd_step(1e-4, 1e-5, 0.1, 1.0, 1)  # before anatomy/phi
        assert e.value.status == -5
        with pytest.raises(_lib.GbgError) as e:
            h.set_anatomy(np.full((32,) * 3, np.nan), np.zeros((32,) * 3))
        assert e.value.status == -4
        with pytest.raises(ValueError):
            h.set_phi(np.zeros(10))
    with pytest.raises(_lib.GbgError) as e:
        _lib.Handle(2, "f64")
    assert e.value.status == -1


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
@pytest.mark.parametrize("kind,n", [("ellipsoid", 37), ("scattered", 20), ("full", 24), ("grey", 21), ("none", 16), ("one", 17)])
def test_exact_steps_over_the_live_cells_equal_oracle(gbg, oracle_lib, prec, kind, n):
    """From the third step on the exact modes compute the cells of a list only:
    dead cells (a NaN face) leave it, cells with a zero face (p_g only and Dg =
    0) stay on it with the doubling. Split over calls, after a new density and
    with new diffusivities; bit for bit the oracle's steps over every cell."""
    rng = np.random.default_rng(n)
    if kind == "ellipsoid":
        an = S.make_anatomy(n, seed=2)
        pw, pg = an.p_w, an.p_g
    else:
        t = {"scattered": (rng.random((n, n, n)) < 0.9), "full": np.ones((n, n, n)), "grey": rng.random((n, n, n)) < 0.97,
             "none": np.zeros((n, n, n)), "one": np.zeros((n, n, n))}[kind].astype(float)
        if kind == "one":
            t[5:8, 5:8, 5:8] = 1
        w = (rng.random((n, n, n)) < 0.5) * 1.0 if kind == "grey" else rng.random((n, n, n))
        pw, pg = t * w, t * (1.0 - w)
    f32 = prec == "f32ref"
    with _lib.Handle(n, prec) as h:
        h.set_anatomy(pw, pg)
        for Dw_file, ratio in ((0.0013, 0.1), (0.0009, 0.0 if kind == "grey" else 0.1)):
            dt, dw, dg = S.reference_dt(n, Dw_file, n * 0.1, f32=f32)
            dg = dg if ratio else 0.0
            phi = np.where(pw + pg > 0, rng.random((n, n, n)) ** 8, 0.0)
            phi[0, 0, 0] = 0.5  # tissue or not
            if f32:
                phi = phi.astype(np.float32).astype(np.float64)
            h.set_phi(phi)
            done = 0
            for steps in (1, 1, 1, 4, 9):
                h.rd_step(dw, dg, 0.025, dt, steps)
                done += steps
                ref = oracle_lib.rd_solve(pw, pg, phi, dw, dg, 0.025, dt, done, "f32ref" if f32 else "f64")
                assert np.array_equal(h.get_phi(), ref.astype(np.float64)), (Dw_file, done)


@pytest.mark.parametrize("precision", ["f64", "f32ref"])
@pytest.mark.parametrize("n,dense", [(5, True), (16, False), (40, True), (64, False), (100, True)])
def test_exact_steps_in_one_call_equal_single_steps(gbg, precision, n, dense):
    """Many exact steps in one call run in one launch whose CTAs meet between
    steps: the bits of the same steps in calls of their own, with fewer
    cells than CTAs, tissue up to the periodic faces (dense), more cells than
    the CTAs' shared memory holds, and an even and an odd number of steps."""
    rng = np.random.default_rng(n)
    if dense:
        pw, pg = rng.uniform(0.05, 1.0, (2, n, n, n))
    else:
        an = S.make_anatomy(n, seed=3)
        pw, pg = an.p_w, an.p_g
    phi = rng.uniform(0.0, 1.0, (n, n, n)) * (pw + pg > 0)
    D = 0.1 / n ** 2
    with _lib.Handle(n, precision) as h:
        h.set_anatomy(pw, pg)
        outs = []
        for calls in ((1,) * 13, (13,), (2, 4, 7), (6, 1, 6)):
            h.set_phi(phi)
            for k in calls:
                h.rd_step(D, 0.1 * D, 0.05, 0.6, k)
            outs.append(h.get_phi())
    assert outs[0].max() > 0
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
@pytest.mark.parametrize("calls", [(1, 1, 1, 1, 3), (9,), (2, 5)])
def test_exact_steps_from_densities_below_zero_with_decay(gbg, oracle_lib, prec, calls):
    """A first step from densities below 0 with a negative rho leaves positive
    values in cells without tissue, which the second one clears: neither the
    cells of the list nor those off it may keep them, bit for bit the oracle's
    steps over every cell, also with a rho of the other sign afterwards."""
    n, f32 = 14, prec == "f32ref"
    rng = np.random.default_rng(3)
    t = (rng.random((n, n, n)) < 0.85).astype(float)
    w = rng.random((n, n, n))
    pw, pg = t * w, t * (1.0 - w)
    phi = rng.uniform(-3.0, 1.0, (n, n, n))
    dt, dw, dg = S.reference_dt(n, 0.0013, n * 0.1, f32=f32)
    rho = -0.5 / dt
    if f32:
        phi = phi.astype(np.float32).astype(np.float64)
        rho = float(np.float32(rho))
    ref = phi
    with _lib.Handle(n, prec) as h:
        h.set_anatomy(pw, pg)
        h.set_phi(phi)
        for k in calls:
            h.rd_step(dw, dg, rho, dt, k)
            ref = oracle_lib.rd_solve(pw, pg, ref, dw, dg, rho, dt, k, prec).astype(np.float64)
            assert np.array_equal(h.get_phi(), ref), k
            rho = -rho
    assert ref.max() > 0


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
@pytest.mark.parametrize("n", [13, 48])
def test_exact_steps_with_other_coefficients_in_each_call(gbg, oracle_lib, prec, n):
    """Whether a call makes the list depends on the steps ahead of it, on those
    taken and on the grid (from 200,000 cell-steps, two at 48^3, or five steps on):
    calls of one to eight steps, some with the coefficients of the one before."""
    rng = np.random.default_rng(n)
    t = (rng.random((n, n, n)) < 0.9).astype(float)
    w = rng.random((n, n, n))
    pw, pg = t * w, t * (1.0 - w)
    phi = rng.uniform(0.0, 1.0, (n, n, n)).astype(np.float32).astype(np.float64)
    with _lib.Handle(n, prec) as h:
        h.set_anatomy(pw, pg)
        h.set_phi(phi)
        ref = phi
        for k, scale in ((1, 1.0), (2, 0.9), (2, 0.9), (1, 0.9), (1, 0.9), (3, 1.0), (4, 0.8), (1, 0.8), (5, 0.9), (6, 1.0), (8, 0.7)):
            dt, dw, dg = S.reference_dt(n, 0.0013, n * 0.1, f32=prec == "f32ref")
            dw = float(np.float32(dw * scale)) if prec == "f32ref" else dw * scale
            h.rd_step(dw, dg, 0.025, dt, k)
            ref = oracle_lib.rd_solve(pw, pg, ref, dw, dg, 0.025, dt, k, prec).astype(np.float64)
            assert np.array_equal(h.get_phi(), ref), (k, scale)
