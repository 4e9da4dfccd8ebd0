"""Memory that a context holds: what it does not read it does not allocate,
and what a solve needs it gives back.

512,000 atoms, sp3d5s* with spin and recomputed blocks: 295 bytes of device
memory an atom (neighbours 16, on-site records 256, sites, types, surface flags,
the recompute order and the reduction scratch), 315 with the work order of the
stored blocks.  Bar: 304, room for four 2 MB mappings.
"""
import pytest

from nemo3d_b200 import materials, workloads

pytestmark = pytest.mark.gpu

MATS = [materials.MATERIALS["GaAs_spds"], materials.MATERIALS["InAs_spds"]]


def test_recomputed_blocks_need_no_work_order():
    import torch
    from nemo3d_b200.tbgpu import Hamiltonian
    st = workloads.gaas_cube(40)
    small = Hamiltonian(workloads.gaas_cube(4), "sp3d5s*_so", MATS, recompute=True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g = Hamiltonian(st, "sp3d5s*_so", MATS, recompute=True)
    torch.cuda.synchronize()
    held = (before - torch.cuda.mem_get_info()[0]) / g.natoms
    g.close()
    small.close()
    print("bytes an atom", held)
    assert g.natoms == 512000 and held <= 304.0


def _address_space():
    """Bytes of the process's mappings (VmSize)."""
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) * 1024 for line in f if line.startswith("VmSize"))


def test_large_iteration_limits_hold_no_pinned_memory():
    """A solve copies alpha and beta into pinned memory of 80 bytes per
    iteration allowed: 160 MB at a limit of two million.  The context keeps at
    most 4 MB of it (bar: 64 MB more address space than after a solve with a
    small limit; a context that is closed again has run the large one before,
    so that the process has its thread arenas and the device pool)."""
    from nemo3d_b200.tbgpu import Hamiltonian
    first, g = (Hamiltonian(workloads.gaas_cube(6), "sp3d5s*_so", MATS) for _ in range(2))
    r0 = workloads.random_start(g.n, seed=0)
    kw = dict(ConvCheckStartIter=100, ConvCheckSkipRate=50, requested1=1, requested2=0,
              emin1=-100.0, emax1=100.0, emin2=200.0, emax2=201.0, tolerance=1e-2)
    first.eigensolve_lanczos(r0, imax=2_000_000, **kw)
    first.close()
    small = g.eigensolve_lanczos(r0, imax=2000, **kw)
    before = _address_space()
    large = g.eigensolve_lanczos(r0, imax=2_000_000, **kw)
    held = _address_space() - before
    print("iterations", small["iterations"], large["iterations"], "held MB", held / 2**20)
    assert large["iterations"] == small["iterations"] < 2000
    assert (large["values"] == small["values"]).all()
    assert held <= 64 << 20
    again = g.eigensolve_lanczos(r0, imax=2000, **kw)
    assert (again["values"] == small["values"]).all()
