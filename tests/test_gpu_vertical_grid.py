"""Grids stretched in z only (xi_y, xi_z, eta_x and eta_z zero in every cell, as
every grid built from a run directory is) take streaming kernels that neither
load these four fields nor form their terms.  The terms are exact zeros, so
the results are the general kernels' bit for bit: one cell of the padding
column, outside every stencil that reaches the interior's output, made nonzero
sends the same model through the general kernels."""
import numpy as np
import pytest

from test_gpu_batch import _scaled, _synthetic
from test_gpu_step_forms import PREC, _wave

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")

# field, cell: a corner of the padded grid, whose coefficients no point reads
CORNER = (slice(None), 0, 0, 0)


def _vertical(shape, precision, general):
    nx, ny, nz, npml = shape
    sc = _synthetic(nx, ny, nz, npml, seed=nx)
    if precision != "fp32":
        sc = _scaled(sc)
    c = sc["cjm"].reshape(13, nz + 6, ny + 6, nx + 6)
    for f in (1, 2, 3, 5):
        c[f] = 0.0
    if general:
        c[general][CORNER[1:]] = 0.25
    return sc


def _run(shape, precision, form, general, steps=9):
    nx, ny, nz, npml = shape
    sc = _vertical(shape, precision, general)
    d = cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, steps, PREC[precision],
                        cgfdm.KERNEL_STREAM)
    with cgfdm.Simulation(d) as sim:
        sim.set_tile_rows(form)
        sim.set_model(sc["cjm"], sc["rdz"])
        sim.set_state(0, W=_wave(nx, ny, nz, 3, precision != "fp32"))
        sim.set_timing(True)  # counts the bytes of the form that ran
        sim.run(steps)
        st = sim.get_state()
        return st, sim.kernel_stats()["stream_bytes"]


@pytest.mark.parametrize("form", [16, 8, 64])
@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape,general", [((200, 41, 29, 6), 1), ((131, 24, 40, 9), 2),
                                           ((64, 33, 21, 0), 3), ((71, 17, 30, 5), 5)])
def test_vertical_grid_is_bitwise_the_general_form(gpu_available, shape, general, precision, form):
    if form == 64 and precision == "fp32":
        pytest.skip("the paired form is for 16-bit storage")
    got, b_vert = _run(shape, precision, form, 0)
    ref, b_gen = _run(shape, precision, form, general)
    assert b_vert < b_gen  # both forms were exercised
    for key in ("W", "t", "aux"):
        assert np.isfinite(ref[key]).all()
        assert np.array_equal(got[key], ref[key]), key
    assert np.abs(ref["W"]).max() > 0


def test_a_new_model_replaces_captured_steps(gpu_available):
    """A model that is not vertical, set after steps were captured for one that
    is (alone and in a batch): the next steps run the general form."""
    shape = (71, 45, 30, 5)
    nx, ny, nz, npml = shape
    a, b = _vertical(shape, "fp32", 0), _synthetic(nx, ny, nz, npml, seed=3)
    out = []
    for mode in ("eager", "graph", "batch"):
        d = cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, 48, cgfdm.FP32, cgfdm.KERNEL_STREAM)
        with cgfdm.Simulation(d) as sim:
            sim.set_tile_rows(16)
            sim.set_graph(mode == "graph")
            batch = cgfdm.Batch([sim], graph=True) if mode == "batch" else None
            run = batch.run if batch else sim.run
            sim.set_model(a["cjm"], a["rdz"])
            sim.set_state(0, W=_wave(nx, ny, nz, 3, False))
            run(20)  # every phase captured, some replayed
            sim.set_model(b["cjm"], b["rdz"])
            run(20)
            out.append(sim.wavefield())
            if batch:
                batch.close()
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
