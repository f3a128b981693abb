"""A whole step of the fast path against the same step made stage by stage,
and the free-surface kernel on grids where a PML slab reaches it.

In a whole step (cgfdm_run) stage 2 forms the RK accumulator t from the
stage inputs; cgfdm_stage updates t in every stage as the reference does.
Both are the same sums in another order: in FP32 they agree to a few units
of rounding (2^-24 relative per operation, about ten of them; bar 1e-6), in
16-bit storage t and each stage output are rounded to the format (unit
roundoff 2^-11 FP16, 2^-8 BF16), t up to three times on one side: bar four
units."""
import numpy as np
import pytest

from test_gpu_batch import _scaled, _synthetic

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")

FB0 = (-1, -1, -1)  # signs of step 0, flipped after every stage
BAR = {"fp32": 1e-6, "fp16": 4 * 2.0 ** -11, "bf16": 4 * 2.0 ** -8}
PREC = {"fp32": cgfdm.FP32, "fp16": cgfdm.FP16, "bf16": cgfdm.BF16}


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _wave(nx, ny, nz, seed, scaled):
    rng = np.random.default_rng(seed)
    W = np.zeros((9, nz + 6, ny + 6, nx + 6), np.float32)
    amp = np.array([0.1] * 3 + [1e6] * 6, np.float32)
    if scaled:
        amp *= np.array([5e3] * 3 + [1e-6] * 6, np.float32)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    for v in range(9):
        k = 2 * np.pi / rng.uniform(9, 25, 3)
        p = rng.uniform(0, 6, 3)
        W[v, 3:-3, 3:-3, 3:-3] = amp[v] * np.sin(k[0] * z + p[0]) * np.sin(
            k[1] * y + p[1]) * np.sin(k[2] * x + p[2])
    return W


@pytest.mark.parametrize("form", [16, 8, 64])
@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape", [(70, 21, 25, 5), (200, 33, 19, 0)])
def test_whole_step_matches_its_stages(gpu_available, shape, precision, form):
    if form == 64 and precision == "fp32":
        pytest.skip("the paired form is for 16-bit storage")
    nx, ny, nz, npml = shape
    sc = _synthetic(nx, ny, nz, npml, seed=11)
    if precision != "fp32":
        sc = _scaled(sc)
    W = _wave(nx, ny, nz, 3, precision != "fp32")
    out = []
    for whole in (True, False):
        d = cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, 2, PREC[precision],
                            cgfdm.KERNEL_STREAM)
        with cgfdm.Simulation(d) as sim:
            sim.set_tile_rows(form)
            sim.set_model(sc["cjm"], sc["rdz"])
            sim.set_state(0, W=W)
            if whole:
                sim.run(1)
            else:
                for irk in range(4):
                    sim.stage(irk, [f * (-1 if irk % 2 else 1) for f in FB0])
            out.append(sim.get_state())
    for key in ("W", "t"):
        a, b = (s[key].reshape(9, -1) for s in out)
        for v in range(9):
            assert np.isfinite(a[v]).all()
            assert rel_l2(a[v], b[v]) <= BAR[precision], (key, v, rel_l2(a[v], b[v]))
    # the auxiliaries stay in FP32; in 16-bit storage they see the rounded stage inputs
    if npml:
        assert rel_l2(out[0]["aux"], out[1]["aux"]) <= BAR[precision]


@pytest.mark.parametrize("shape", [(33, 17, 6, 5), (65, 9, 4, 4), (32, 8, 5, 0), (31, 7, 9, 3),
                                   (20, 41, 30, 10)])
def test_surface_layers_with_every_slab(gpu_available, shape):
    """Partial tiles, corners of x and y slabs, and a bottom slab that reaches
    the three free-surface layers: against the exact-order kernel, 8 steps."""
    nx, ny, nz, npml = shape
    sc = _synthetic(nx, ny, nz, npml, seed=5)
    W = _wave(nx, ny, nz, 4, False)
    out = []
    for kern in (cgfdm.KERNEL_EXACT, cgfdm.KERNEL_STREAM):
        d = cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, 8, cgfdm.FP32, kern)
        with cgfdm.Simulation(d) as sim:
            sim.set_model(sc["cjm"], sc["rdz"])
            sim.set_state(0, W=W)
            sim.run(8)
            out.append((sim.wavefield().reshape(9, -1), sim.pgv()))
    assert np.isfinite(out[1][0]).all()
    for v in range(9):
        assert rel_l2(out[1][0][v], out[0][0][v]) <= 1e-5
    assert rel_l2(out[1][1], out[0][1]) <= 1e-5
