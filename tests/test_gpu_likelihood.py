"""GPU: the log-likelihood kernels through the C ABI against the reference's
`likelihood` program (golden, printed to six decimals) and the oracle."""
import numpy as np
import pytest

from gliomauq_gb300 import _lib
from helpers import golden_json, golden_npz

pytestmark = pytest.mark.gpu

# double accumulation in a fixed tree order against the reference's long
# double running sum
REL_TOL = 1e-11


@pytest.mark.parametrize("mode", ["sel", "all"])
def test_loglik_vs_reference_program(gbg, mode):
    d = golden_npz("lik32.npz")
    ref = golden_json("lik32.json")
    with _lib.Handle(32, "f64") as h:
        h.set_phi(d["model"])
        h.set_observations(d["pet"], d["t1"], d["t2"], d["points"], ref["params"],
                           step_pet=ref["step_pet"], step_ti=ref["step_ti"],
                           selective=(mode == "sel"))
        r = h.loglik()
    exp = ref[mode]
    assert r["n_pet"] == exp["n_pet"]
    for k in ("l_pet", "l_t1", "l_t2"):
        assert abs(r[k] - exp[k]) <= 1e-6, k
    assert abs(-r["total"] - exp["minus_loglik"]) <= 1e-6


@pytest.mark.parametrize("prec", ["f64", "f32ref", "f32"])
@pytest.mark.parametrize("selective", [True, False])
def test_loglik_vs_oracle(gbg, oracle_lib, prec, selective):
    d = golden_npz("lik32.npz")
    ref = golden_json("lik32.json")
    model = d["model"]
    if prec != "f64":
        model = model.astype(np.float32).astype(np.float64)
    with _lib.Handle(32, prec) as h:
        h.set_phi(model)
        h.set_observations(d["pet"], d["t1"], d["t2"], d["points"], ref["params"], step_pet=3,
                           step_ti=2, selective=selective)
        r = h.loglik()
    o = oracle_lib.loglik(model, d["pet"], d["t1"], d["t2"], d["points"], ref["params"],
                          step_pet=3, step_ti=2, selective=selective)
    assert r["n_pet"] == o["n_pet"]
    for k in ("l_pet", "l_t1", "l_t2", "total"):
        assert abs(r[k] - o[k]) <= REL_TOL * max(1.0, abs(o[k])), (k, r[k], o[k])


def test_loglik_edge_cases(gbg, oracle_lib):
    n = 32
    rng = np.random.default_rng(5)
    model = rng.random((n, n, n))
    pet = np.zeros((n, n, n))  # no PET voxel: N = 0, PET term 0
    t1 = (rng.random((n, n, n)) > 0.5).astype(float)
    t2 = np.ones((n, n, n))
    model[0, 0, 0] = 0.7  # u == uc: sgn = 0, alpha = 0.5
    params = (0.0025, 1.0, 0.7, 0.25, 0.09)
    pts = np.array([[0, 0, 0], [2, 4, 6], [31, 31, 31]], dtype=float)
    with _lib.Handle(n, "f64") as h:
        h.set_phi(model)
        h.set_observations(pet, t1, t2, pts, params, step_pet=3, step_ti=1, selective=True)
        r = h.loglik()
        with pytest.raises(_lib.GbgError):
            h.set_observations(pet, t1, t2, np.array([[40.0, 0, 0]]), params)
    o = oracle_lib.loglik(model, pet, t1, t2, pts, params, step_pet=3, step_ti=1, selective=True)
    assert r["n_pet"] == 0 and r["l_pet"] == 0.0
    for k in ("l_t1", "l_t2", "total"):
        assert abs(r[k] - o[k]) <= REL_TOL * max(1.0, abs(o[k]))


@pytest.mark.parametrize("n_pet,n_ti", [(1, 1), (255, 257), (256, 2049), (2047, 256), (2049, 2048), (6000, 1)])
def test_loglik_at_the_edges_of_the_clusters(gbg, oracle_lib, n_pet, n_ti):
    """Lists that end inside, at and behind a run of 256 entries and a chunk of
    eight runs, one longer than the other (the double sums' order differs from
    the oracle's: REL_TOL)."""
    n = 32
    rng = np.random.default_rng(n_pet)
    model = rng.random((n, n, n))
    pet = np.zeros(n ** 3)
    pet[rng.choice(n ** 3, n_pet, replace=False)] = rng.uniform(0.1, 1.0, n_pet)
    pet = pet.reshape(n, n, n)
    t1, t2 = ((rng.random((n, n, n)) > 0.5).astype(float) for _ in range(2))
    c = rng.choice(n ** 3, n_ti, replace=False)
    pts = np.stack([c % n, c // n % n, c // n ** 2], axis=1).astype(float)
    params = (0.0025, 1.0, 0.7, 0.25, 0.09)
    with _lib.Handle(n, "f64") as h:
        h.set_phi(model)
        h.set_observations(pet, t1, t2, pts, params, step_pet=1, step_ti=1, selective=True)
        assert h.observation_counts() == (n_pet, n_ti)
        r = h.loglik()
    o = oracle_lib.loglik(model, pet, t1, t2, pts, params, step_pet=1, step_ti=1, selective=True)
    assert r["n_pet"] == o["n_pet"] == n_pet
    for k in ("l_pet", "l_t1", "l_t2", "total"):
        assert abs(r[k] - o[k]) <= REL_TOL * max(1.0, abs(o[k])), (k, r[k], o[k])


@pytest.mark.parametrize("n_pet,n_ti", [(200, 100), (2049, 300), (100, 1900)])
def test_loglik_of_many_fields_is_each_fields_own(gbg, n_pet, n_ti):
    """Few chunks of entries are reduced by clusters, many (over six per SM: 912 on
    a GB300) by a CTA each, in the same order: counts around the change, bit for
    bit the fields one by one."""
    n = 32
    rng = np.random.default_rng(n_ti)
    pet = np.zeros(n ** 3)
    pet[rng.choice(n ** 3, n_pet, replace=False)] = rng.uniform(0.1, 1.0, n_pet)
    t1, t2 = ((rng.random((n, n, n)) > 0.5).astype(float) for _ in range(2))
    c = rng.choice(n ** 3, n_ti, replace=False)
    pts = np.stack([c % n, c // n % n, c // n ** 2], axis=1).astype(float)
    chunks = -(-max(n_pet, n_ti) // 2048)
    with _lib.Handle(n, "f32") as h:
        h.set_anatomy(np.full((n, n, n), 0.5), np.full((n, n, n), 0.4))
        h.set_observations(pet.reshape(n, n, n), t1, t2, pts, (0.0025, 1.0, 0.7, 0.25, 0.09), step_pet=1, step_ti=1, selective=True)
        h.affine_set(rng.random((n, n, n)), rng.standard_normal((2, n, n, n)))
        d = rng.uniform(-1, 1, (2000 // chunks, 2))
        whole = h.affine_loglik(d)
        for count in (911 // chunks, 912 // chunks, 913 // chunks + 1):
            assert np.array_equal(h.affine_loglik(d[:count]), whole[:count]), count
        assert np.array_equal(np.concatenate([h.affine_loglik(x) for x in d[:40]]), whole[:40])
