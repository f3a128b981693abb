"""What an autotuner choice is kept under: a model of the other kind of grid
(stretched in z only or general) runs other kernels and is tuned by itself,
also on a handle or in a batch that has run before, and an entry of a tuning
file that was made for earlier kernels is not taken."""
import json

import pytest

from test_gpu_batch import _synthetic

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")


def _models(nx, ny, nz, npml):
    general = _synthetic(nx, ny, nz, npml, seed=2)
    vertical = _synthetic(nx, ny, nz, npml, seed=2)
    c = vertical["cjm"].reshape(13, -1)
    for f in (1, 2, 3, 5):
        c[f] = 0.0
    return vertical, general


def _sim(nx, ny, nz, npml):
    return cgfdm.Simulation(cgfdm.make_desc(nx, ny, nz, npml, 100.0, 0.008, 20, cgfdm.FP32,
                                            cgfdm.KERNEL_AUTO))


@pytest.mark.parametrize("batch", [False, True])
def test_each_kind_of_grid_is_tuned_by_itself(gpu_available, tmp_path, monkeypatch, batch):
    cache = tmp_path / "tune.json"
    monkeypatch.setenv("CGFDM_TUNE_CACHE", str(cache))
    dims = (98 + batch, 81, 31, 6)
    vertical, general = _models(*dims)
    with _sim(*dims) as sim:
        b = cgfdm.Batch([sim]) if batch else None
        seen = []
        for sc in (vertical, general, vertical):
            sim.set_model(sc["cjm"], sc["rdz"])
            (b or sim).run(1)
            sim.synchronize()
            seen.append(json.loads(cache.read_text()))
        if b:
            b.close()
    assert [len(s) for s in seen] == [1, 2, 2]
    assert sorted(k.split("|")[-1] for k in seen[1]) == ["general", "vertical"]


def test_a_form_that_the_caller_fixed_stays(gpu_available):
    dims = (100, 81, 31, 6)
    vertical, general = _models(*dims)
    with _sim(*dims) as sim:
        sim.set_tile_rows(16)
        sim.set_chunk(9)
        for sc in (vertical, general):
            sim.set_model(sc["cjm"], sc["rdz"])
            sim.run(1)
            assert sim.tuning() == (16, 9)


def test_an_entry_for_earlier_kernels_is_not_taken(gpu_available, tmp_path, monkeypatch):
    import torch

    prop = torch.cuda.get_device_properties(0)
    cache = tmp_path / "tune.json"
    dims = (101, 81, 31, 6)
    old = "%s|sm%d|precision0|%dx%dx%d|npml%d|chunk-1|batch0" % (
        (prop.name, prop.multi_processor_count) + dims)
    cache.write_text(json.dumps({old: [16, 64, 0]}))
    monkeypatch.setenv("CGFDM_TUNE_CACHE", str(cache))
    sc = _models(*dims)[1]
    with _sim(*dims) as sim:
        sim.set_model(sc["cjm"], sc["rdz"])
        sim.run(1)
        assert sim.tuning3()[2] == 1  # the entry asks for the exact-order surface kernel
    now = json.loads(cache.read_text())
    assert len(now) == 2 and now[old] == [16, 64, 0]  # other keys' entries are kept
