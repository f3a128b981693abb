"""cgfdm_device_bytes against what a handle takes from the device, its kept
read-back buffers included.  The grid is flat, so that the surface maps weigh:
the free-surface staging alone is 75 MB.  Each of the handle's about fifteen
allocations may be rounded up to 2 MB."""
import pytest

pytestmark = pytest.mark.gpu
cgfdm = pytest.importorskip("cgfdm")


def _held(nx, ny):
    import torch

    d = cgfdm.make_desc(nx, ny, 4, 0, 100.0, 0.008, 2, cgfdm.FP16, cgfdm.KERNEL_STREAM)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    with cgfdm.Simulation(d) as sim:
        sim.set_tile_rows(8)
        sim.run(1)
        sim.free_surface()
        sim.pgv()
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info(0)[0], cgfdm.device_bytes(d)


def test_device_bytes_covers_what_a_handle_holds(gpu_available):
    _held(40, 40)  # loads the kernels, which stay on the device
    held, said = _held(2500, 2500)
    assert said <= held + (1 << 20)
    assert held <= said + (40 << 20), (held, said)
