"""The ring kernel (default H*x, block product, float product) where it can go
wrong: tasks that fill only partly, structures smaller than one task, missing
neighbours, vacancies, vectors that start off a 128-byte line, block widths
whose lanes do not fill a warp.

Bars: against the oracle within 45e-12 of max|H| for double vectors (the bar
of every double H*x test); for float vectors within 48 * 2^-24 * 45 max|H|
(45 terms of at most max|H| each, one rounding each and three more for the
scale and the shift, entries up to 1); columns of the block product equal to
the single product bit for bit.
"""
import numpy as np
import pytest

import oracle
from nemo3d_b200 import materials, workloads

pytestmark = pytest.mark.gpu

A = workloads.A_GAAS


def _alloy(nx, ny, nz, seed, vacancies=0.0, periodic=False):
    rng = np.random.default_rng(seed)
    t = np.zeros((nx, ny, nz, 8), np.uint8)
    t[..., :4] = np.where(rng.random((nx, ny, nz, 4)) < 0.5, materials.SPECIES["In"],
                          materials.SPECIES["Ga"])
    t[..., 4:] = materials.SPECIES["As"]
    if vacancies:
        t[rng.random(t.shape) < vacancies] = 0
    dsp = rng.normal(0, 0.004, (nx, ny, nz, 8, 3))
    return workloads.Structure(nx, ny, nz, (A, A, A), (periodic,) * 3, t, dsp)


STRUCTURES = {
    "1x1x1": lambda: _alloy(1, 1, 1, 1),                    # less than one task
    "1x2x3": lambda: _alloy(1, 2, 3, 2),                    # 24 + 24 atoms
    "5x3x7_vacancies": lambda: _alloy(5, 3, 7, 3, 0.25),    # unequal kinds, remainders
    "17x9x11": lambda: _alloy(17, 9, 11, 4),                # several rounds of the grid
    "3x3x3_periodic": lambda: _alloy(3, 3, 3, 5, periodic=True),
}


def _pair(name, model, **opts):
    from nemo3d_b200.tbgpu import Hamiltonian
    fam = "sps" if model.startswith("sp3s*") else "spds"
    mats = [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]
    st = STRUCTURES[name]()
    norb, nspin = materials.BAND_MODELS[model]
    o = oracle.OracleHamiltonian(st, norb, nspin, mats)
    if opts.get("ham_bits") == 32:
        o.onsite = o.onsite.astype(np.float32).astype(np.float64)
        o.blocks = o.blocks.astype(np.float32).astype(np.float64)
    scale = max(np.abs(o.onsite).max(), np.abs(o.blocks).max())
    return Hamiltonian(st, model, mats, **opts), o, scale


@pytest.mark.parametrize("name", list(STRUCTURES))
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
@pytest.mark.parametrize("bits", [64, 32])
def test_ring_hx_matches_oracle(name, model, bits):
    g, o, scale = _pair(name, model, ham_bits=bits)
    x = np.random.default_rng(6).uniform(-1, 1, 2 * g.n)
    assert np.abs(g.matvect_mult(x, 0.7) - o.hx(x, 0.7)).max() <= 45e-12 * scale


@pytest.mark.parametrize("name", list(STRUCTURES))
@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
def test_ring_float_vectors_match_oracle(name, model):
    import torch
    g, o, scale = _pair(name, model, ham_bits=32, lanczos_bits=32)
    x = np.random.default_rng(7).uniform(-1, 1, 2 * g.n).astype(np.float32)
    xd, yd = torch.from_numpy(x).cuda(), torch.empty(2 * g.n, dtype=torch.float32, device="cuda")
    g.hx_dev_f32(xd.data_ptr(), yd.data_ptr(), 0.7)
    torch.cuda.synchronize()
    err = np.abs(yd.cpu().numpy() - o.hx(x.astype(np.float64), 0.7)).max()
    assert err <= 48 * 2.0 ** -24 * 45 * scale, err


@pytest.mark.parametrize("name", ["1x1x1", "5x3x7_vacancies", "17x9x11"])
@pytest.mark.parametrize("model", ["sp3d5s*_so", "sp3d5s*"])
@pytest.mark.parametrize("p", [2, 3, 4, 5, 6, 7, 8])
def test_ring_block_columns_equal_single_products(name, model, p):
    import torch
    g, _, _ = _pair(name, model)
    n2 = 2 * g.n
    x = torch.rand(p * n2, dtype=torch.float64, device="cuda") * 2 - 1
    y, one = torch.full_like(x, float("nan")), torch.empty_like(x)
    g.hx_block_dev(p, x.data_ptr(), y.data_ptr(), 0.4)
    for v in range(p):
        g.hx_dev(x.data_ptr() + v * n2 * 8, one.data_ptr() + v * n2 * 8, 0.4)
    torch.cuda.synchronize()
    assert torch.equal(y, one)


@pytest.mark.parametrize("model", ["sp3d5s*_so", "sp3s*"])
@pytest.mark.parametrize("off", [2, 4, 6, 14])
def test_ring_vectors_off_a_line(model, off):
    """Vectors that start 16, 32, 48 or 112 bytes past an aligned address."""
    import torch
    g, o, scale = _pair("5x3x7_vacancies", model)
    n2 = 2 * g.n
    x = torch.zeros(n2 + off, dtype=torch.float64, device="cuda")
    x[off:] = torch.rand(n2, dtype=torch.float64, device="cuda") * 2 - 1
    y = torch.full((n2 + off + 16,), 7.0, dtype=torch.float64, device="cuda")
    g.hx_dev(x.data_ptr() + 8 * off, y.data_ptr() + 8 * off, 0.1)
    torch.cuda.synchronize()
    yo = o.hx(x[off:].cpu().numpy(), 0.1)
    assert np.abs(y[off:off + n2].cpu().numpy() - yo).max() <= 45e-12 * scale
    assert bool((y[:off] == 7.0).all()) and bool((y[off + n2:] == 7.0).all())


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("name", ["1x1x1", "17x9x11"])
def test_order_of_overlapped_launches(name, captured):
    """Products whose starts overlap the kernels before them, between copies,
    elementwise kernels and a second stream's work: bit for bit what the same
    calls give with a synchronisation after each one."""
    import torch
    from nemo3d_b200.tbgpu import Hamiltonian
    mats = [materials.MATERIALS["GaAs_spds"], materials.MATERIALS["InAs_spds"]]
    H = Hamiltonian(STRUCTURES[name](), "sp3d5s*_so", mats)
    x = torch.from_numpy(np.random.default_rng(7).uniform(-1, 1, 2 * H.n)).cuda()
    bufs = [torch.zeros_like(x) for _ in range(4)]
    side = torch.cuda.Stream()

    def work(sync):
        main, wait = torch.cuda.current_stream(), torch.cuda.synchronize if sync else lambda: None
        a, b, c, d = bufs
        a.copy_(x); wait()
        for k in range(6):
            H.hx_dev(a.data_ptr(), b.data_ptr(), 0.1 * k); wait()   # reads a, writes b
            H.hx_dev(b.data_ptr(), a.data_ptr(), 0.2); wait()       # reads b, overwrites a
            side.wait_stream(main)
            with torch.cuda.stream(side):
                c.copy_(a); c.mul_(0.25)
            H.hx_dev(a.data_ptr(), d.data_ptr(), 0.3); wait()
            main.wait_stream(side); wait()
            H.hx_dev(c.data_ptr(), b.data_ptr(), 0.4); wait()       # behind a join
            b.add_(d); wait()
            H.hx_dev(b.data_ptr(), a.data_ptr(), 0.5); wait()       # behind another kernel
            a.mul_(2.0 ** -8); wait()

    H.set_stream(torch.cuda.current_stream().cuda_stream)
    work(True)
    want = [t.clone() for t in bufs]
    assert torch.isfinite(want[0]).all() and want[0].abs().max() > 0
    for t in bufs:
        t.zero_()
    run = torch.cuda.Stream()
    run.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(run):
        H.set_stream(run.cuda_stream)
        if captured:
            work(False)
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=run):
                work(False)
            for t in bufs:
                t.zero_()
            graph.replay()
            graph.replay()
        else:
            work(False)
    torch.cuda.synchronize()
    for got, w in zip(bufs, want):
        assert torch.equal(got, w)


@pytest.mark.parametrize("name", ["1x1x1", "5x3x7_vacancies", "17x9x11"])
@pytest.mark.parametrize("model", ["sp3d5s*_so", "sp3s*"])
@pytest.mark.parametrize("bits", [64, 32])
def test_recurrence_matches_oracle(name, model, bits):
    """alpha and beta of six Lanczos steps (product, update, overlapped
    launches; vectors of odd and even lengths, fewer entries than threads)
    against the same steps on the oracle's product.  Each step adds at most
    one product's error (the bars above) to the vector, and the vector of the
    step before enters once more, so seven bars a step are allowed."""
    import torch
    its = 6
    opts = dict(ham_bits=32, lanczos_bits=32) if bits == 32 else {}
    g, o, scale = _pair(name, model, **opts)
    rng = np.random.default_rng(9)
    r = rng.uniform(-1, 1, 2 * g.n)
    r0 = torch.from_numpy(r.copy()).cuda()
    g.eigensolve_lanczos_dev(r0.data_ptr(), imax=its + 1, emin1=1.0, emax1=1.1, emin2=1.4,
                             emax2=1.5)
    alpha, beta = g.tridiagonal(its + 1)
    r /= np.linalg.norm(r)
    prev, bprev, a_ref, b_ref = np.zeros_like(r), 0.0, [], []
    for _ in range(its):
        w = o.hx(r, 0.0)
        a = float(w @ r)
        w = w - a * r - bprev * prev
        b = float(np.linalg.norm(w))
        prev, bprev, r = r, b, w / b
        a_ref.append(a)
        b_ref.append(b)
    bar = 45e-12 * scale if bits == 64 else 48 * 2.0 ** -24 * 45 * scale
    assert len(alpha) == its
    assert np.abs(alpha - a_ref).max() <= 7 * its * bar
    assert np.abs(beta[:its] - b_ref).max() <= 7 * its * bar
