"""Products whose time must not exceed that of a product that does more.

A time of one shape is compared with the time of another on the same GPU in
the same process, so the bars hold on any clock: a block of p vectors takes no
longer than a block of 8 on the same structure (1.35 times allowed; measured
0.75 to 1.13, and 1.6 to 2.4 with the staging that took line after line of a
flat count for p = 3, 5, 6 and 7).
"""
import numpy as np
import pytest

from nemo3d_b200 import materials, workloads

pytestmark = pytest.mark.gpu


def _ham(cells, model, **opts):
    """An InGaAs alloy cube of `cells`^3 conventional cells, on torch's stream."""
    import torch
    from nemo3d_b200.tbgpu import Hamiltonian
    fam = "sps" if model.startswith("sp3s*") else "spds"
    rng = np.random.default_rng(3)
    t = np.empty((cells,) * 3 + (8,), np.uint8)
    t[..., :4] = np.where(rng.random((cells,) * 3 + (4,)) < 0.5, materials.SPECIES["In"],
                          materials.SPECIES["Ga"])
    t[..., 4:] = materials.SPECIES["As"]
    st = workloads.Structure(cells, cells, cells, (workloads.A_GAAS,) * 3, (False,) * 3, t,
                             rng.normal(0, 0.004, t.shape + (3,)))
    g = Hamiltonian(st, model, [materials.MATERIALS["GaAs_" + fam],
                                materials.MATERIALS["InAs_" + fam]], **opts)
    g.set_stream(torch.cuda.current_stream().cuda_stream)
    return g


def _time(fn, calls=200, rounds=7):
    """us per call: the shortest of a few rounds of calls in a row."""
    import torch
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = float("inf")
    for _ in range(rounds):
        a.record()
        for _ in range(calls):
            fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / calls)
    return best


@pytest.mark.parametrize("model", ["sp3d5s*_so", "sp3d5s*"])
def test_narrow_blocks_take_no_longer_than_wide_ones(model):
    import torch
    g = _ham(6, model)
    x = torch.rand(8 * 2 * g.n, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    t = {p: _time(lambda: g.hx_block_dev(p, x.data_ptr(), y.data_ptr(), 0.3))
         for p in range(2, 9)}
    print(model, {p: round(v, 2) for p, v in t.items()})
    assert max(t.values()) <= 1.35 * t[8], t


@pytest.mark.parametrize("store,single", [(64, False), (32, False), (32, True)])
def test_spinless_product_takes_no_longer_than_the_spin_model(store, single):
    """216 atoms, sp3s* without and with spin, 5 and 10 entries an atom: the
    same (1.12 times allowed; measured 0.78 to 0.83, and 1.24 to 1.28 with tasks
    of 32 atoms whatever the size)."""
    import torch
    opts = dict(ham_bits=store, **(dict(lanczos_bits=32) if single else {}))
    t = {}
    for model in ("sp3s*", "sp3s*_so"):
        g = _ham(3, model, **opts)
        x = torch.rand(2 * g.n, dtype=torch.float32 if single else torch.float64, device="cuda")
        y = torch.empty_like(x)
        call = g.hx_dev_f32 if single else g.hx_dev
        t[model] = _time(lambda: call(x.data_ptr(), y.data_ptr(), 0.3))
    print(store, single, {m: round(v, 2) for m, v in t.items()})
    assert t["sp3s*"] <= 1.12 * t["sp3s*_so"], t


@pytest.mark.parametrize("model", list(materials.BAND_MODELS))
def test_product_with_dot_takes_less_than_two_products(model):
    """216 atoms: the allocation-free product with its dot (one reduction more
    than the product) against 1.8 products; measured 1.46 to 1.57, and 2.0 to
    2.5 with the counter cleared by a memset."""
    import ctypes as C
    import torch
    from nemo3d_b200 import tbgpu
    f = tbgpu._lib().tbgpu_hx_dot_noalloc
    f.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    g = _ham(3, model)
    x = torch.rand(2 * g.n, dtype=torch.float64, device="cuda")
    y, dot = torch.empty_like(x), torch.zeros(1, dtype=torch.float64, device="cuda")
    one = _time(lambda: g.hx_dev(x.data_ptr(), y.data_ptr(), 0.3))
    both = _time(lambda: f(g._ctx, 0.3, x.data_ptr(), y.data_ptr(), dot.data_ptr()))
    print(model, round(one, 2), round(both, 2))
    assert both <= 1.8 * one, (one, both)


@pytest.mark.parametrize("cells", [1, 6])
def test_product_with_dot_in_a_row_and_captured(cells):
    """Calls in a row, each on the result of the one before, and the same calls
    replayed from a graph: dots and vectors as with a synchronisation after
    every call."""
    import ctypes as C
    import torch
    from nemo3d_b200 import tbgpu
    f = tbgpu._lib().tbgpu_hx_dot_noalloc
    f.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p]
    f.restype = C.c_int
    g = _ham(cells, "sp3d5s*_so")
    x = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, 2 * g.n)).cuda()
    a, b = x.clone(), torch.zeros_like(x)
    dots = torch.zeros(8, dtype=torch.float64, device="cuda")

    def work(sync):
        a.copy_(x)
        for k in range(8):
            src, dst = (a, b) if k % 2 == 0 else (b, a)
            assert f(g._ctx, 0.1 * k, src.data_ptr(), dst.data_ptr(),
                     dots.data_ptr() + 8 * k) == 0
            if sync:
                torch.cuda.synchronize()

    work(True)
    want = [t.clone() for t in (a, b, dots)]
    assert dots.abs().min() > 0
    run = torch.cuda.Stream()
    run.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(run):
        g.set_stream(run.cuda_stream)
        dots.zero_()
        work(False)
        torch.cuda.synchronize()
        assert all(torch.equal(t, w) for t, w in zip((a, b, dots), want))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=run):
            work(False)
        dots.zero_()
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(t, w) for t, w in zip((a, b, dots), want))
