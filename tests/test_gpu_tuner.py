"""What the autotuner times.  The kernels that a run launches are taken from
the profiler's record of it."""
import re
from collections import Counter

import numpy as np
import pytest

from test_gpu_batch import _scaled, _synthetic

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")


def stage_classes(run):
    """Launches of the streaming kernels during run(), by stage class: 4, 5, 6
    and 3 are the stages 0 to 3 of a whole step."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    if not any("stage_surface_kernel" in n for n in names):
        pytest.skip("the profiler records no kernels here")
    out = Counter()
    for n in names:
        m = re.search(r"stage_(stream|pair)_kernel<(.*?)>\(", n)
        if m:
            args = [a.strip() for a in m.group(2).split(",")]
            out[int(args[-2])] += 1  # <..., RK, VT>
    return out


@pytest.mark.parametrize("precision,dims", [("fp32", (140, 44, 41, 6)), ("fp16", (204, 44, 41, 6))])
def test_every_timed_stage_class_is_a_candidate_s(gpu_available, precision, dims):
    """Stages 0, 1 and 2 of a whole step are kernels of their own: the tuner
    times each of them with every candidate, and the results are those of a
    handle that does not tune."""
    nx, ny, nz, npml = dims
    sc = _synthetic(nx, ny, nz, npml, seed=8)
    if precision == "fp16":
        sc = _scaled(sc)
    prec = cgfdm.FP32 if precision == "fp32" else cgfdm.FP16
    waves = []
    for form in (0, 8):
        d = cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, 6, prec, cgfdm.KERNEL_STREAM)
        with cgfdm.Simulation(d) as sim:
            sim.set_tile_rows(form)
            sim.set_model(sc["cjm"], sc["rdz"])
            sim.set_point_source(*sc["src"], 6.0)

            def one():
                sim.run(1)
                sim.synchronize()

            first = stage_classes(one)
            step = stage_classes(one)
            if form == 0:
                timed = {c: first[c] - step[c] for c in (4, 5, 6, 3)}
                assert timed[4] == timed[5] == timed[6], timed
                assert timed[4] >= 6 * 2  # six candidates, interior and PML launches
                assert timed[3] == 0
            else:
                assert first == step
            sim.run(4)
            waves.append(sim.wavefield())
    assert np.abs(waves[0]).max() > 0
    assert np.array_equal(waves[0], waves[1])
