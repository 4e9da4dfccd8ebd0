"""The ring kernel (default H*x) against kernels and arithmetic that are not
its own.

* Products: the oracle and variants 1 (lane gather) and 6 (pencil layout) on
  domes with surfaces, a periodic supercell and an alloy dot; the numbers 2 to
  5, which select the ring kernel too, give its results bit for bit.  Bars:
  45e-12 of max|H| in double; float vectors 8 * 2^-24 of max|y| (45 terms of
  both signs: 7 roundings in root mean square, of terms below max|y|; measured
  1.3 to 2.8, the pencil kernel 3.9 to 6.5).
* Lanczos values on variants 0, 1 and 6: within 1e-9 eV.
* The mixed recurrence against the same steps in numpy with the vectors rounded
  to float: alpha and beta of six steps within 1e-5 of max|H| (a step's product
  and update are a few 1e-7 off, and each step carries the earlier ones on by a
  factor of a few).  A step that loses the last entry of an odd vector is 1e-3
  of max|H| off and more.
* Infinities and NaN in x reach the atom, its neighbours and nothing else,
  beside missing bonds and vacancies as well, and the same rows as with the
  lane-gather kernel.
* Batched solves of dots smaller than a task, whose tasks hold atoms of several
  dots of which some have converged: each dot's values as when solved alone.
"""
import numpy as np
import pytest

import oracle
from nemo3d_b200 import materials, workloads

pytestmark = pytest.mark.gpu


def _alloy(nx, ny, nz, seed, vacancies=0.0, periodic=False):
    rng = np.random.default_rng(seed)
    t = np.empty((nx, ny, nz, 8), np.uint8)
    t[..., :4] = np.where(rng.random((nx, ny, nz, 4)) < 0.5, materials.SPECIES["In"],
                          materials.SPECIES["Ga"])
    t[..., 4:] = materials.SPECIES["As"]
    if vacancies:
        t[rng.random(t.shape) < vacancies] = 0
    a = workloads.A_GAAS
    return workloads.Structure(nx, ny, nz, (a, a, a), (periodic,) * 3, t,
                               rng.normal(0, 0.004, t.shape + (3,)))


STRUCTURES = {
    "dome_7x6x5": lambda: workloads.dome_in_box(cells=(7, 6, 5), base_nm=2.4, height_nm=1.0,
                                                wl_z_nm=1.2, sigma_frac=0.02, seed=3),
    "dome_20x18x13": lambda: workloads.dome_in_box(cells=(20, 18, 13), base_nm=7.0,
                                                   height_nm=2.0, wl_z_nm=1.5,
                                                   sigma_frac=0.02, seed=4),
    "periodic_3x4x3": lambda: _alloy(3, 4, 3, 5, periodic=True),
    "alloy_dot": lambda: workloads.alloy_dot(6000, 0.3, seed=2),
    "vacancies_5x3x7": lambda: _alloy(5, 3, 7, 3, vacancies=0.25),
}


def _pair(st, model, **opts):
    import torch
    from nemo3d_b200.tbgpu import Hamiltonian
    fam = "sps" if model.startswith("sp3s*") else "spds"
    mats = [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]
    o = oracle.OracleHamiltonian(st, *materials.BAND_MODELS[model], mats)
    if opts.get("ham_bits") == 32:
        o.onsite = o.onsite.astype(np.float32).astype(np.float64)
        o.blocks = o.blocks.astype(np.float32).astype(np.float64)
    g = Hamiltonian(st, model, mats, **opts)
    g.set_stream(torch.cuda.current_stream().cuda_stream)
    return g, o, max(np.abs(o.onsite).max(), np.abs(o.blocks).max())


@pytest.mark.parametrize("name", list(STRUCTURES))
@pytest.mark.parametrize("model", ["sp3d5s*", "sp3d5s*_so"])
@pytest.mark.parametrize("bits", [64, 32])
def test_products_of_every_kernel(name, model, bits):
    g, o, scale = _pair(STRUCTURES[name](), model, ham_bits=bits)
    x = np.random.default_rng(17).uniform(-1, 1, 2 * g.n)
    want = o.hx(x, 0.9)
    y = {}
    for v in (0, 1, 2, 3, 4, 5, 6):
        g.set_spmv_variant(v)
        y[v] = g.matvect_mult(x, 0.9)
        assert np.abs(y[v] - want).max() <= 45e-12 * scale, v
    for v in (2, 3, 4, 5):
        np.testing.assert_array_equal(y[v], y[0])
    assert not np.array_equal(y[1], y[0]) and not np.array_equal(y[6], y[0])  # other kernels


@pytest.mark.parametrize("name", list(STRUCTURES))
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
def test_float_products_of_every_kernel(name, model):
    import torch
    g, o, _ = _pair(STRUCTURES[name](), model, ham_bits=32, lanczos_bits=32)
    x = np.random.default_rng(7).uniform(-1, 1, 2 * g.n).astype(np.float32)
    want = o.hx(x.astype(np.float64), 0.3)
    xd = torch.from_numpy(x).cuda()
    for v in (0, 6) if model.startswith("sp3d5") else (0,):
        g.set_spmv_variant(v)
        yd = torch.full_like(xd, float("nan"))
        g.hx_dev_f32(xd.data_ptr(), yd.data_ptr(), 0.3)
        err = np.abs(yd.cpu().numpy() - want).max() / np.abs(want).max()
        print(name, model, v, "error in 2^-24", err * 2.0 ** 24)
        assert err <= 8 * 2.0 ** -24, (v, err)


def test_lanczos_values_of_every_kernel():
    st = workloads.dome_in_box(cells=(8, 8, 6), base_nm=3.0, height_nm=1.2, wl_z_nm=1.2,
                               sigma_frac=0.01, seed=2)
    g, _, _ = _pair(st, "sp3d5s*_so")
    r0 = workloads.random_start(g.n, seed=0)
    kw = dict(imax=3000, requested1=3, requested2=3, emin1=-0.6, emax1=0.3, emin2=0.8,
              emax2=2.4, tolerance=1e-7)
    values = {}
    for v in (0, 1, 6):
        g.set_spmv_variant(v)
        values[v] = g.eigensolve_lanczos(r0, **kw)["values"]
        assert len(values[v]) >= 2
    for v in (1, 6):  # a borderline check may accept a value more or less
        few, many = sorted((values[0], values[v]), key=len)
        assert len(many) - len(few) <= 2
        assert all(np.abs(many - e).min() < 1e-9 for e in few), v


@pytest.mark.parametrize("name", ["vacancies_5x3x7", "dome_7x6x5"])
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
def test_mixed_recurrence_matches_numpy(name, model):
    import torch
    its = 6
    g, o, scale = _pair(STRUCTURES[name](), model, ham_bits=32, lanczos_bits=32)
    start = np.random.default_rng(9).uniform(-1, 1, 2 * g.n)
    r0 = torch.from_numpy(start.copy()).cuda()
    g.eigensolve_lanczos_dev(r0.data_ptr(), imax=its + 1, emin1=1.0, emax1=1.1, emin2=1.4,
                             emax2=1.5)
    alpha, beta = g.tridiagonal(its + 1)

    def run(lose_last):
        f32 = lambda v: v.astype(np.float32).astype(np.float64)  # noqa: E731
        r, before, a_ref, b_ref = f32(start / np.linalg.norm(start)), None, [], []
        norm, norm_before = np.linalg.norm(r), 0.0
        for _ in range(its):
            u = f32(r / norm)
            w = f32(o.hx(u, 0.0))
            a = float(w @ u)
            nxt = w - a * r / norm
            if before is not None:
                nxt = nxt - norm * before / norm_before
            nxt = f32(nxt)
            if lose_last:
                nxt[-2:] = 0.0
            before, norm_before, r, norm = r, norm, nxt, np.linalg.norm(nxt)
            a_ref.append(a)
            b_ref.append(norm)
        return np.array(a_ref), np.array(b_ref)

    assert len(alpha) == its
    a_ref, b_ref = run(False)
    off = max(np.abs(alpha - a_ref).max(), np.abs(beta[:its] - b_ref).max())
    print(name, model, g.n, "off by", off / scale, "of max|H|")
    assert off <= 1e-5 * scale, off
    a_bad, b_bad = run(True)  # the mistake is in the oracle's steps: the bar sees it
    assert max(np.abs(alpha - a_bad).max(), np.abs(beta[:its] - b_bad).max()) > 1e-5 * scale


@pytest.mark.parametrize("name", ["dome_7x6x5", "vacancies_5x3x7"])
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("single", [False, True])
def test_non_finite_entries_stay_with_their_neighbours(name, model, value, single):
    """One entry of the first, the last and a middle atom at a time; the first
    atom's data are what lanes without an atom or a bond point at."""
    import torch
    opts = dict(ham_bits=32, lanczos_bits=32) if single else {}
    g, _, _ = _pair(STRUCTURES[name](), model, **opts)
    _, nbr, _ = g.export_pattern()
    nbr = nbr.reshape(-1, 4)
    dt = np.float32 if single else np.float64
    x = np.random.default_rng(3).uniform(-1, 1, 2 * g.n).astype(dt)
    call = g.hx_dev_f32 if single else g.hx_dev

    def product(v):
        xd = torch.from_numpy(v).cuda()
        yd = torch.full_like(xd, 7.0)
        call(xd.data_ptr(), yd.data_ptr(), 0.2)
        return yd.cpu().numpy().reshape(g.natoms, -1)

    clean = product(x)
    assert np.isfinite(clean).all()
    per = 2 * g.n // g.natoms
    for atom in (0, g.natoms // 2, g.natoms - 1):
        bad = x.copy()
        bad[atom * per + 4] = value  # the third orbital's real part
        y = product(bad)
        near = np.zeros(g.natoms, bool)
        near[atom] = True
        near[nbr[atom][nbr[atom] >= 0]] = True
        assert not np.isfinite(y[near]).all(axis=1).any()
        np.testing.assert_array_equal(y[~near], clean[~near])
        if not single and model.startswith("sp3d5"):
            g.set_spmv_variant(1)
            other = product(bad)
            g.set_spmv_variant(0)
            np.testing.assert_array_equal(np.isfinite(y), np.isfinite(other))


@pytest.mark.parametrize("p", [3, 4])
def test_non_finite_entries_in_a_block(p):
    """... and stay in their column of a block product."""
    import torch
    g, _, _ = _pair(STRUCTURES["vacancies_5x3x7"](), "sp3d5s*_so")
    x = np.random.default_rng(3).uniform(-1, 1, (p, 2 * g.n))

    def product(v):
        xd = torch.from_numpy(v).cuda()
        yd = torch.full_like(xd, 7.0)
        g.hx_block_dev(p, xd.data_ptr(), yd.data_ptr(), 0.2)
        return yd.cpu().numpy()

    clean = product(x)
    bad = x.copy()
    bad[1, 4] = np.nan
    y = product(bad)
    keep = [v for v in range(p) if v != 1]
    np.testing.assert_array_equal(y[keep], clean[keep])
    assert np.isnan(y[1]).any() and (y[1] == clean[1]).sum() > g.n


@pytest.mark.parametrize("model", ["sp3s*", "sp3s*_so", "sp3d5s*", "sp3d5s*_so"])
def test_batch_of_dots_smaller_than_a_task(model):
    from nemo3d_b200.tbgpu import Hamiltonian
    fam = "sps" if model.startswith("sp3s*") else "spds"
    mats = [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]
    dots = [workloads.alloy_dot(n, 0.6, seed=i) for i, n in enumerate((30, 200, 60, 500, 40))]
    packed, cells = workloads.pack_dots(dots)
    gb = Hamiltonian(packed, model, mats)
    singles = [Hamiltonian(d, model, mats) for d in dots]
    starts = [workloads.random_start(g.n, seed=10 + i) for i, g in enumerate(singles)]
    kw = dict(ConvCheckStartIter=40, ConvCheckSkipRate=20, imax=2000, requested1=1, requested2=1,
              tolerance=1e-7)
    res = gb.eigensolve_lanczos_batched(np.concatenate(starts), cells, -0.8, 0.4, 1.0, 3.5, **kw)
    print(model, res["iterations"])
    assert len(set(res["iterations"].tolist())) > 1  # some dots are done before others
    for d, (g, r0) in enumerate(zip(singles, starts)):
        alone = g.eigensolve_lanczos(r0, emin1=-0.8, emax1=0.4, emin2=1.0, emax2=3.5, **kw)
        few, many = sorted((res["values"][d], alone["values"]), key=len)
        assert len(few) >= 1
        assert all(np.abs(many - e).min() < 1e-7 for e in few), d
