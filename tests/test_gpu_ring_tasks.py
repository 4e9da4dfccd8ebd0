"""The ring kernel on both sides of the sizes where its tasks change from 8 to
16 and from 16 to 32 atoms.

Periodic alloys of a given count of atoms; the limits are those of 148 SMs:
4,736 atoms (four tasks of 8 a SM), 18,944 and 28,416 (8 and 12 tasks of 16).
Bars: against the oracle, 45e-12 of max|H| for double vectors, for
float vectors 90 * 2^-24 of the largest absolute row sum (45 terms of entries
up to 1, two roundings each); the fused dot of the allocation-free product
within 1e-12 of the sum of its terms' magnitudes.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from nemo3d_b200 import materials, workloads

pytestmark = pytest.mark.gpu

CELLS = {"4736": (4, 4, 37), "4752": (3, 3, 66), "18944": (8, 8, 37), "18960": (5, 6, 79),
         "28416": (8, 12, 37), "28424": (11, 17, 19)}


def _alloy(cells):
    rng = np.random.default_rng(3)
    t = np.empty(cells + (8,), np.uint8)
    t[..., :4] = np.where(rng.random(cells + (4,)) < 0.5, materials.SPECIES["In"],
                          materials.SPECIES["Ga"])
    t[..., 4:] = materials.SPECIES["As"]
    a = workloads.A_GAAS
    return workloads.Structure(*cells, (a, a, a), (True,) * 3, t,
                               rng.normal(0, 0.004, t.shape + (3,)))


def _pair(name, model, **opts):
    import torch
    from nemo3d_b200.tbgpu import Hamiltonian
    fam = "sps" if model.startswith("sp3s*") else "spds"
    mats = [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]
    st = _alloy(CELLS[name])
    o = oracle.OracleHamiltonian(st, *materials.BAND_MODELS[model], mats)
    if opts.get("ham_bits") == 32:
        o.onsite = o.onsite.astype(np.float32).astype(np.float64)
        o.blocks = o.blocks.astype(np.float32).astype(np.float64)
    g = Hamiltonian(st, model, mats, **opts)
    g.set_stream(torch.cuda.current_stream().cuda_stream)
    assert g.natoms == int(name)
    return g, o, max(np.abs(o.onsite).max(), np.abs(o.blocks).max())


@pytest.mark.parametrize("name", list(CELLS))
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
@pytest.mark.parametrize("kvec", [None, (0.31, -0.17, 0.23)])
def test_double_products(name, model, kvec):
    import torch
    from nemo3d_b200 import tbgpu
    g, o, scale = _pair(name, model)
    if kvec:
        g.set_bloch_k(kvec)
        o.kvec = np.asarray(kvec, np.float64)
    x = np.random.default_rng(6).uniform(-1, 1, 2 * g.n)
    xd = torch.from_numpy(x).cuda()
    yd, dot = torch.full_like(xd, float("nan")), torch.zeros(1, dtype=torch.float64, device="cuda")
    g.hx_dev(xd.data_ptr(), yd.data_ptr(), 0.7)
    y = yd.cpu().numpy()
    assert np.abs(y - o.hx(x, 0.7)).max() <= 45e-12 * scale
    f = tbgpu._lib().tbgpu_hx_dot_noalloc  # the fused dot
    f.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    yd.fill_(float("nan"))
    assert f(g._ctx, 0.7, xd.data_ptr(), yd.data_ptr(), dot.data_ptr()) == 0
    assert np.array_equal(yd.cpu().numpy(), y)
    assert abs(dot.item() - float(x @ y)) <= 1e-12 * float(np.abs(x) @ np.abs(y))


@pytest.mark.parametrize("name", list(CELLS))
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
def test_float_products(name, model):
    import torch
    g, o, _ = _pair(name, model, ham_bits=32, lanczos_bits=32)
    x = np.random.default_rng(7).uniform(-1, 1, 2 * g.n).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    yd = torch.full_like(xd, float("nan"))
    g.hx_dev_f32(xd.data_ptr(), yd.data_ptr(), 0.7)
    err = np.abs(yd.cpu().numpy() - o.hx(x.astype(np.float64), 0.7)).max()
    rows = _abs_row_sum(o)
    assert err <= 90 * 2.0 ** -24 * rows, (err, rows)


def _abs_row_sum(o):
    """At least the largest absolute row sum of H: an on-site row and the rows
    of four bond blocks."""
    blk = np.abs(o.blocks).reshape(-1, o.norb, o.norb)
    ons = np.abs(o.onsite).reshape(o.natoms, o.nb, -1).sum(-1).max()
    return ons + 4 * max(blk.sum(1).max(), blk.sum(2).max())


@pytest.mark.parametrize("model", ["sp3s*", "sp3d5s*_so"])
def test_few_atoms_in_a_wide_flat_grid(model):
    """90,000 pencils, atoms in 60 of them at two corners: the work order's
    counts per pencil need more scratch than the products' reductions."""
    from nemo3d_b200.tbgpu import Hamiltonian
    st = _alloy((300, 300, 1))
    keep = np.zeros(st.types.shape, bool)
    keep[:6, :5] = keep[-5:, -6:] = True
    st.types[~keep] = 0
    st = workloads.Structure(300, 300, 1, st.lattice, (False,) * 3, st.types, st.dsp)
    fam = "sps" if model.startswith("sp3s*") else "spds"
    mats = [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]
    g = Hamiltonian(st, model, mats)
    o = oracle.OracleHamiltonian(st, *materials.BAND_MODELS[model], mats)
    assert 300 < g.natoms == o.natoms <= 480
    scale = max(np.abs(o.onsite).max(), np.abs(o.blocks).max())
    x = np.random.default_rng(6).uniform(-1, 1, 2 * g.n)
    assert np.abs(g.matvect_mult(x, 0.7) - o.hx(x, 0.7)).max() <= 45e-12 * scale
