"""What went wrong in one call does not reach the next: the no-allocation
stage after its shared scratch was left with work queues that are not empty,
and a handle that goes on after a bounded wait expired."""
import ctypes

import numpy as np
import pytest

from test_gpu_batch import SHAPES, _scaled, _sim, _synthetic

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")
from cgfdm import _lib  # noqa: E402


def _stale_queues(stream, kind=2):
    _lib.check(_lib.lib().cgfdm_stage_noalloc_inject_fault(kind, stream))


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_noalloc_stage_after_stale_work_queues(gpu_available, precision):
    import torch

    nx, ny, nz, npml = 131, 45, 40, 6  # interior and PML launches in both precisions
    sc = _synthetic(nx, ny, nz, npml, seed=3)
    if precision == "fp16":
        sc = _scaled(sc)
    ebytes, dtype = (4, torch.float32) if precision == "fp32" else (2, torch.float16)
    dev = torch.device("cuda", 0)
    L = cgfdm.hbm_layout(nx, ny, nz, ebytes)

    def buffer(nf, src=None):
        b = torch.zeros(nf * L["fs"], dtype=dtype, device=dev)
        if src is not None:
            v = b.view(nf, L["fs"])[:, :L["nz_"] * L["plane"]].view(nf, L["nz_"], L["ny_"], L["px"])
            v[..., L["xoff"]:L["xoff"] + L["nx_"]] = src
        return b

    g = torch.Generator(device=dev).manual_seed(1)
    W = torch.zeros(9, nz + 6, ny + 6, nx + 6, device=dev)
    W[:, 3:-3, 3:-3, 3:-3] = torch.randn(9, nz, ny, nx, generator=g, device=dev)
    w = buffer(9, W)
    cjm = buffer(13, torch.from_numpy(sc["cjm"]).to(dev).view(13, nz + 6, ny + 6, nx + 6))
    rdz = torch.from_numpy(sc["rdz"]).to(dev)
    naux = 9 * npml * (2 * ny * nz + 2 * nx * nz + nx * ny)
    aux = torch.randn(naux, generator=g, device=dev)
    out = []
    stream = torch.cuda.current_stream(dev).cuda_stream
    for stale in (False, True):
        w_out, t, a_out, a_t = buffer(9), buffer(9), torch.zeros_like(aux), torch.zeros_like(aux)
        b = _lib.StageBuffers(nx=nx, ny=ny, nz=nz, npml=npml, dh=100.0, dt=0.008,
                              precision=cgfdm.FP32 if precision == "fp32" else cgfdm.FP16, irk=0,
                              fb1=1, fb2=-1, fb3=1, w_in=w.data_ptr(), w_out=w_out.data_ptr(),
                              w_m=w.data_ptr(), t=t.data_ptr(), cjm=cjm.data_ptr(),
                              rdz=rdz.data_ptr(), aux_in=aux.data_ptr(), aux_out=a_out.data_ptr(),
                              aux_m=aux.data_ptr(), aux_t=a_t.data_ptr())
        if stale:
            _stale_queues(stream)
        cgfdm.stage_noalloc(b, stream, wait=True)
        out.append((w_out, t, a_out, a_t))
    assert all(torch.isfinite(x).all() for x in out[0])
    assert (out[0][0] != 0).sum() > 0.99 * 9 * nx * ny * nz  # no item was skipped there
    for x, y in zip(*out):
        assert torch.equal(x, y)


def test_unknown_noalloc_fault_is_refused():
    assert _lib.lib().cgfdm_stage_noalloc_inject_fault(1, ctypes.c_void_p(None)) == 1


def test_a_handle_goes_on_after_an_expired_wait(gpu_available):
    """The launch whose wait expired leaves its work queues empty as every
    launch does: the same handle, set back to a step before it, matches an
    undisturbed run bit for bit."""
    sc = _synthetic(*SHAPES[0], seed=9)
    with _sim(sc) as ref:
        ref.run(6)
        want = ref.wavefield(), ref.stations(), ref.pgv()
    with _sim(sc) as s:
        s.run(2)
        saved = s.checkpoint()
        s.inject_fault(1)
        s.run(1)
        with pytest.raises(cgfdm.CgfdmError) as e:
            s.synchronize()
        assert e.value.code == 303
        s.restore(saved)
        s.run(4)
        for a, b in zip((s.wavefield(), s.stations(), s.pgv()), want):
            np.testing.assert_array_equal(a, b)
