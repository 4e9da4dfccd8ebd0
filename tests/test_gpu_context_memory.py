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
