"""GPU: exact steps captured from the handle's stream into a caller's CUDA
graph. A replay takes the steps from whatever density it finds, and calls
outside the graph, before and after the capture and its replays, take theirs:
bit for bit the oracle's steps on the uniform grid, and on the block grid those
of calls one by one."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from gliomauq_gb300 import _lib, synthetic as S
from helpers import golden_npz

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _capture(stream):
    """A graph of what the body enqueues on the handle's stream, and its replay."""
    torch = pytest.importorskip("torch")
    s = torch.cuda.ExternalStream(stream)
    g = torch.cuda.CUDAGraph()

    def replay():
        with torch.cuda.stream(s):
            g.replay()

    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        try:
            yield replay
        finally:
            g.capture_end()


def _problem(prec, n=18):
    rng = np.random.default_rng(4)
    t = (rng.random((n, n, n)) < 0.9).astype(float)
    w = rng.random((n, n, n))
    fields = rng.uniform(0.0, 1.0, (3, n, n, n))  # off the tissue too
    if prec == "f32ref":
        fields = fields.astype(np.float32).astype(np.float64)
    dt, dw, dg = S.reference_dt(n, 0.0013, n * 0.1, f32=prec == "f32ref")
    return t * w, t * (1.0 - w), fields, (dw, dg, 0.03125, dt)


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
@pytest.mark.parametrize("before,captured", [(2, 4), (2, 2), (8, 6)])
def test_replays_step_the_density_they_find(gbg, oracle_lib, prec, before, captured):
    pw, pg, (a, b, c), co = _problem(prec)

    def ref(phi, k):
        return oracle_lib.rd_solve(pw, pg, phi, *co, k, prec).astype(np.float64)

    with _lib.Handle(pw.shape[0], prec) as h:
        h.set_anatomy(pw, pg)
        h.set_phi(a)
        h.rd_step(*co, before)
        with _capture(h.stream()) as replay:
            h.rd_step(*co, captured)
        for phi in (b, c):
            h.set_phi(phi)
            replay()
            assert np.array_equal(h.get_phi(), ref(phi, captured))
            replay()
            assert np.array_equal(h.get_phi(), ref(phi, 2 * captured))
            h.rd_step(*co, 5)
            assert np.array_equal(h.get_phi(), ref(phi, 2 * captured + 5))


def _block_grid_replays(prec):
    """The grid after a graph of four steps has run on a new density, and after two
    more replays and steps between them; and the same by calls."""
    d = golden_npz("amr64_f32.npz")
    co = tuple(float(np.float32(v)) for v in (2e-4, 2e-5, 0.2)) + (0.5,)
    rng = np.random.default_rng(2)
    a, b = rng.uniform(0.0, 1.0, (2,) + d["phi"].shape).astype(np.float32).astype(np.float64)
    tabs = (d["ghost_start"], d["ghost_src_block"], d["ghost_src_cell"].astype(np.int32), d["ghost_w"].astype(np.float64))
    outs = []
    for graph in (False, True):
        with _lib.AmrHandle(64, prec) as h:
            h.set_grid(d["blocks"], d["p_w"], d["p_g"], a)
            h.set_ghosts(*tabs)
            h.step(*co, 4)
            if graph:
                stream = C.c_void_p()
                _lib.check(h.lib.gbg_stream(h._h, C.byref(stream)))
                with _capture(stream.value) as run:
                    h.step(*co, 4)
            h.set_grid(d["blocks"], d["p_w"], d["p_g"], b)
            if not graph:
                h.set_ghosts(*tabs)
                run = lambda: h.step(*co, 4)
            run()
            outs.append([h.get_phi()])
            h.set_ghosts(*tabs)
            h.step(*co, 2)
            run()
            run()
            outs[-1].append(h.get_phi())
    return outs


@pytest.mark.parametrize("prec", ["f64", "f32ref", "f32"])
def test_replays_on_the_block_grid(gbg, prec):
    calls, graph = _block_grid_replays(prec)
    for x, y in zip(calls, graph):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", ["f64", "f32ref"])
def test_a_capture_that_never_runs_changes_nothing(gbg, oracle_lib, prec):
    """The list a captured call makes is made when its graph runs; calls that
    follow do not wait for that."""
    pw, pg, (a, b, _), co = _problem(prec)
    with _lib.Handle(pw.shape[0], prec) as h:
        h.set_anatomy(pw, pg)
        h.set_phi(a)
        h.rd_step(*co, 1)
        with _capture(h.stream()):
            h.rd_step(*co, 6)
        h.set_phi(b)
        h.rd_step(*co, 9)
        assert np.array_equal(h.get_phi(), oracle_lib.rd_solve(pw, pg, b, *co, 9, prec).astype(np.float64))
