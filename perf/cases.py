"""What this package's users have it do, as cases that can be timed.

A user builds a structure's tight-binding Hamiltonian once and then applies it
thousands of times: H*x on device vectors (``hx_dev``, the product of every
double-precision Lanczos solve), the mixed-precision product on complex-float
vectors over the float store (``hx_dev_f32``; with variant 5 the kernel of the
mixed solves that regenerate their eigenvectors), the block product of the
block Lanczos solver (``hx_block_dev``), and Lanczos runs
(``eigensolve_lanczos_dev`` with ``tridiagonal``).  The listed cases cover the
band models, the closed, periodic and packed structures, single, double and
block vectors, and sizes from the 4096-atom cube of the tests to the
two-million-atom dot of the benchmark; ``draw`` gives further cases of the
same ranges.

``exact`` computes the same results with plain torch in 64 bits: the
Slater-Koster blocks from rotated orbitals (amplitudes of every orbital along
the bond's own axes) rather than from the tabulated polynomials.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from nemo3d_b200 import materials, workloads
from nemo3d_b200.tbgpu import Hamiltonian

SHIFT = 1.246          # mid-gap of the benchmark's dot (eV)
BLOCH = (0.31, -0.17, 0.23)
ALLOY = 0.35           # In fraction of the periodic alloy and the packed dots


def listed():
    return [
        # the smallest call: one product on the 8x8x8-cell cube of the tests,
        # where latency and launches count
        dict(name="hx64-cube8", op="hx", model="sp3d5s*_so", shape="dome", nx=8, ny=8, nz=8),
        # an ordinary dot, its Hamiltonian about as large as the L2 cache
        dict(name="hx64-dome66k", op="hx", model="sp3d5s*_so", shape="dome", nx=23, ny=21, nz=17),
        # the spinless model on a ragged box
        dict(name="hx64-nospin197k", op="hx", model="sp3d5s*", shape="dome", nx=37, ny=29, nz=23),
        # the benchmark's double-precision dot
        dict(name="hx64-dome1M", op="hx", model="sp3d5s*_so", shape="dome", nx=58, ny=58, nz=38),
        # a periodic alloy away from the Gamma point (a band-structure sweep)
        dict(name="hx64-bloch", op="hx", model="sp3d5s*_so", shape="periodic", nx=20, ny=20, nz=20),
        # many 5-orbital dots packed in one structure (the batched solve)
        dict(name="hx64-dots", op="hx", model="sp3s*_so", shape="dots", ndots=48, atoms=9000),
        # the mixed-precision product on a ragged dot and on the benchmark's, and
        # the kernel of the mixed solve with regenerated eigenvectors
        dict(name="hx32-dome127k", op="hx32", model="sp3d5s*_so", shape="dome", nx=31, ny=27, nz=19),
        dict(name="hx32-dot2M", op="hx32", model="sp3d5s*_so", shape="dome", nx=72, ny=72, nz=48),
        dict(name="hx32-lane381k", op="hx32", model="sp3d5s*_so", shape="dome", nx=42, ny=42, nz=27, variant=5),
        # the block Lanczos solver's product, four and eight vectors at once
        dict(name="block4-dome381k", op="block", model="sp3d5s*_so", shape="dome", nx=42, ny=42, nz=27, p=4),
        dict(name="block8-dome66k", op="block", model="sp3d5s*_so", shape="dome", nx=23, ny=21, nz=17, p=8),
        # a whole call: a Lanczos run and the tridiagonal matrix it builds
        # (spectral bounds, densities of states)
        dict(name="lanczos64-dome45k", op="lanczos", model="sp3d5s*_so", shape="dome", nx=20, ny=20, nz=14, its=96),
    ]


def _box(rng, lo, hi):
    """Box of about exp(uniform(log lo, log hi)) cells, sides of any parity."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = cells ** (1.0 / 3.0)
    nx = max(3, round(a * rng.uniform(0.75, 1.3)))
    ny = max(3, round(a * rng.uniform(0.75, 1.3)))
    return nx, ny, max(3, int(cells / (nx * ny)))


def draw(rng):
    op = rng.choice(["hx", "hx", "hx", "hx32", "hx32", "block", "lanczos"])
    if op == "hx":
        kind = rng.choice(["dome", "dome", "nospin", "periodic", "dots"])
        if kind == "dots":
            return dict(op=op, model=rng.choice(["sp3s*_so", "sp3s*"]), shape="dots",
                        ndots=rng.randint(3, 60), atoms=rng.randint(1000, 12000))
        if kind == "periodic":
            nx, ny, nz = _box(rng, 100, 12000)
            return dict(op=op, model=rng.choice(["sp3d5s*_so", "sp3d5s*"]), shape="periodic",
                        nx=nx, ny=ny, nz=nz)
        nx, ny, nz = _box(rng, 300, 110000)
        return dict(op=op, model="sp3d5s*" if kind == "nospin" else "sp3d5s*_so", shape="dome",
                    nx=nx, ny=ny, nz=nz)
    if op == "hx32":
        nx, ny, nz = _box(rng, 300, 200000)
        return dict(op=op, model=rng.choice(["sp3d5s*_so", "sp3d5s*_so", "sp3d5s*"]),
                    shape="dome", nx=nx, ny=ny, nz=nz, variant=rng.choice([0, 0, 5]))
    if op == "block":
        p = rng.randint(2, 8)
        nx, ny, nz = _box(rng, 300, 100000 // p)
        return dict(op=op, model=rng.choice(["sp3d5s*_so", "sp3d5s*"]), shape="dome",
                    nx=nx, ny=ny, nz=nz, p=p)
    nx, ny, nz = _box(rng, 2000, 30000)
    return dict(op=op, model="sp3d5s*_so", shape="dome", nx=nx, ny=ny, nz=nz,
                its=rng.randint(24, 96))


def _structure(case, seed):
    if case["shape"] == "dots":
        rng = np.random.default_rng(case["atoms"])   # one set of sizes, other alloys by seed
        sizes = rng.integers(int(0.7 * case["atoms"]), int(1.3 * case["atoms"]) + 1, case["ndots"])
        dots = [workloads.alloy_dot(int(n), ALLOY, seed=int(seed) + 7919 * i)
                for i, n in enumerate(sizes)]
        return workloads.pack_dots(dots)[0]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    a = workloads.A_GAAS
    if case["shape"] == "periodic":
        rng = np.random.default_rng(seed)
        t = np.empty((nx, ny, nz, 8), np.uint8)
        t[..., :4] = np.where(rng.random((nx, ny, nz, 4)) < ALLOY, materials.SPECIES["In"],
                              materials.SPECIES["Ga"])
        t[..., 4:] = materials.SPECIES["As"]
        return workloads.Structure(nx, ny, nz, (a, a, a), (True, True, True), t,
                                   rng.normal(0.0, 0.0015, (nx, ny, nz, 8, 3)))
    return workloads.dome_in_box(cells=(nx, ny, nz), base_nm=0.6 * min(nx, ny) * a,
                                 height_nm=0.25 * nz * a, sigma_frac=0.005, seed=seed)


def _sets(case):
    fam = "sps" if case["model"].startswith("sp3s*") else "spds"
    return [materials.MATERIALS["GaAs_" + fam], materials.MATERIALS["InAs_" + fam]]


def _vector(case, n, seed):
    """Start vectors: real and imaginary parts uniform in [-1, 1]."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    dt = torch.float32 if case["op"] == "hx32" else torch.float64
    return torch.rand(case.get("p", 1) * 2 * n, dtype=dt, device="cuda", generator=g) * 2 - 1


def prepare(case, seed):
    single = case["op"] == "hx32"
    opts = dict(ham_bits=32, lanczos_bits=32) if single else {}
    H = Hamiltonian(_structure(case, seed), case["model"], _sets(case), **opts)
    H.set_stream(torch.cuda.current_stream().cuda_stream)
    if case["shape"] == "periodic":
        H.set_bloch_k(BLOCH)
    if case.get("variant"):
        H.set_spmv_variant(case["variant"])
    x = _vector(case, H.n, seed)
    return dict(case=case, H=H, x=x, y=None if case["op"] == "lanczos" else torch.empty_like(x))


def run(state):
    case, H, x, y = state["case"], state["H"], state["x"], state["y"]
    if case["op"] == "hx":
        H.hx_dev(x.data_ptr(), y.data_ptr(), SHIFT)
    elif case["op"] == "hx32":
        H.hx_dev_f32(x.data_ptr(), y.data_ptr(), SHIFT)
    elif case["op"] == "block":
        H.hx_block_dev(case["p"], x.data_ptr(), y.data_ptr(), SHIFT)
    else:
        res = H.eigensolve_lanczos_dev(x.data_ptr(), imax=case["its"] + 1, emin1=1.0, emax1=1.1,
                                       emin2=1.4, emax2=1.5)
        alpha, beta = H.tridiagonal(case["its"] + 1)
        return dict(values=res["values"], alpha=alpha, beta=beta)
    return y


def _size(case):
    if case["shape"] == "dots":
        return float(case["ndots"] * case["atoms"])
    return 8.0 * case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Each bond block and on-site record once, every vector once."""
    atoms = _size(case)
    norb, nspin = materials.BAND_MODELS[case["model"]]
    nb = norb * nspin
    single = case["op"] == "hx32"
    real = 4 if single else 8
    ham = atoms * (2 * norb * norb * real + nb * real + 2 * 4)   # two bonds per atom
    vec = atoms * nb * 2 * real
    flops = atoms * 4 * norb * norb * nspin * 4
    p, its = case.get("p", 1), case.get("its", 1)
    if case["op"] == "lanczos":
        return dict(bytes=its * (ham + 3 * vec), flops=its * (flops + 20 * atoms * nb))
    return dict(bytes=ham + 2 * p * vec, flops=p * flops)


# ---- the same results by plain torch in 64 bits -----------------------------

# neighbours of each cation site of the conventional cell: (cell step, anion
# site), and the anion's own slot order for its dangling bonds
_BONDS = [[((0, 0, 0), 4), ((1, 0, 1), 7), ((1, 1, 0), 6), ((0, 1, 1), 5)],
          [((0, 0, 0), 5), ((0, 0, 0), 4), ((1, 0, 0), 6), ((1, 0, 0), 7)],
          [((0, 0, 0), 4), ((0, 0, 0), 6), ((0, 0, 1), 5), ((0, 0, 1), 7)],
          [((0, 0, 0), 4), ((0, 0, 0), 7), ((0, 1, 0), 5), ((0, 1, 0), 6)]]
_HYBRID = np.array([[1, 1, 1], [-1, -1, 1], [1, -1, -1], [-1, 1, -1]]) * 0.25
_KIND = [0, 1, 2, 2, 2, 3, 3, 3, 3, 3]      # s*, s, p, d
_ANG = [0, 0, 1, 1, 1, 2, 2, 2, 2, 2]
# two-centre integrals (anion kind, cation kind) -> sigma, pi, delta entries
_INT = {(0, 0): (11,), (0, 1): (12,), (0, 2): (16,), (0, 3): (20,),
        (1, 0): (13,), (1, 1): (10,), (1, 2): (14,), (1, 3): (18,),
        (2, 0): (17,), (2, 1): (15,), (2, 2): (22, 23), (2, 3): (24, 26),
        (3, 0): (21,), (3, 1): (19,), (3, 2): (25, 27), (3, 3): (28, 29, 30)}
# Harrison exponent of each integral, strain-correction coefficient per kinds
_ETA = {10: 2, 11: 1, 12: 0, 13: 0, 14: 3, 15: 3, 16: 7, 17: 7, 18: 6, 19: 6, 20: 14, 21: 14,
        22: 4, 23: 5, 24: 8, 25: 8, 26: 9, 27: 9, 28: 11, 29: 12, 30: 13}
_COEF = [[18, 19, 23, 27], [20, 17, 21, 25], [24, 22, 29, 30], [28, 26, 31, 32]]
_EN = [[4, 0, 1, 6], [5, 2, 3, 7]]           # on-site energy: anion, cation, by kind
_R3 = 1.73205080757                          # the reference program's sqrt(3)


def _parameters(mat):
    """[35] two-centre and on-site parameters and [33] strain parameters."""
    pv, st = list(mat["pv"]), list(mat["strain"])
    p = [0.0] * 35
    if mat["family"] == "sp3s*":
        p[:6] = pv[:6]
        p[8], p[9] = pv[13] / 3, pv[14] / 3
        p[10], p[14], p[15] = pv[6] / 4, pv[9] * 3 ** 0.5 / 4, pv[10] * 3 ** 0.5 / 4
        p[16], p[17] = pv[11] * 3 ** 0.5 / 4, pv[12] * 3 ** 0.5 / 4
        p[22], p[23] = (pv[7] + 2 * pv[8]) / 4, (pv[7] - pv[8]) / 4
        p[31] = mat["a0"]
    else:
        p[:] = pv
    kinds = (0, 1, 2) if mat["family"] == "sp3s*" else (0, 1, 2, 3)
    for k in kinds:
        p[_EN[0][k]] += mat["ev_offset"] - st[16]
        p[_EN[1][k]] += mat["ev_offset"] - st[15]
    return p, st


def _amplitudes(d, norb):
    """Of each orbital on the bond's own axes: sigma [B, norb], pi and delta
    [B, norb, 2]; a d orbital is the quadratic form r^T Q r."""
    B = d.shape[0]
    ax = torch.zeros_like(d)
    ax.scatter_(1, d.abs().argmin(1, keepdim=True), 1.0)
    e1 = torch.linalg.cross(d, ax)
    e1 = e1 / e1.norm(dim=1, keepdim=True)
    e2 = torch.linalg.cross(d, e1)
    sig = torch.zeros(B, norb, dtype=d.dtype, device=d.device)
    pi = torch.zeros(B, norb, 2, dtype=d.dtype, device=d.device)
    de = torch.zeros_like(pi)
    sig[:, 0] = sig[:, 1] = 1.0
    sig[:, 2:5] = d
    pi[:, 2:5, 0], pi[:, 2:5, 1] = e1, e2
    if norb == 10:
        Q = torch.zeros(5, 3, 3, dtype=d.dtype, device=d.device)
        for o, (u, v) in enumerate(((0, 1), (1, 2), (2, 0))):
            Q[o, u, v] = Q[o, v, u] = 0.5 * _R3
        Q[3, 0, 0], Q[3, 1, 1] = 0.5 * _R3, -0.5 * _R3
        Q[4] = torch.diag(torch.tensor([-0.5, -0.5, 1.0], dtype=d.dtype, device=d.device))
        form = lambda u, v: torch.einsum("oij,bi,bj->bo", Q, u, v)  # noqa: E731
        sig[:, 5:] = form(d, d)
        pi[:, 5:, 0], pi[:, 5:, 1] = form(d, e1) * (2 / _R3), form(d, e2) * (2 / _R3)
        de[:, 5:, 0] = (form(e1, e1) - form(e2, e2)) / _R3
        de[:, 5:, 1] = form(e1, e2) * (2 / _R3)
    return sig, pi, de


def _blocks(d, V, norb):
    """[B, cation orbital, anion orbital] from cosines (anion to cation) and
    the integrals V[k] of every bond."""
    sig, pi, de = _amplitudes(d, norb)
    out = torch.zeros(d.shape[0], norb, norb, dtype=d.dtype, device=d.device)
    for a in range(norb):
        for c in range(norb):
            idx = _INT[(_KIND[a], _KIND[c])]
            e = V[idx[0]] * sig[:, a] * sig[:, c]
            if len(idx) > 1:
                e = e + V[idx[1]] * (pi[:, a] * pi[:, c]).sum(1)
            if len(idx) > 2:
                e = e + V[idx[2]] * (de[:, a] * de[:, c]).sum(1)
            if _ANG[a] > _ANG[c] and (_ANG[a] + _ANG[c]) % 2:
                e = -e
            out[:, c, a] = e
    return out


class _Exact:
    """H*x of a case's structure by plain torch in 64 bits, on the GPU."""

    def __init__(self, case, seed):
        st, dev, f8 = _structure(case, seed), "cuda", torch.float64
        self.norb, self.nspin = materials.BAND_MODELS[case["model"]]
        norb = self.norb
        dims = (st.nx, st.ny, st.nz)
        per = [bool(v) for v in st.periodic]
        kvec = BLOCH if case["shape"] == "periodic" else None
        types = torch.from_numpy(st.types.reshape(-1).astype(np.int64)).to(dev)
        dsp = None if st.dsp is None else torch.from_numpy(st.dsp.reshape(-1, 3)).to(dev)
        lat = torch.tensor(st.lattice, dtype=f8, device=dev)
        site = torch.from_numpy(workloads.SITE_POS).to(dev)
        ijk = torch.stack(torch.meshgrid(*[torch.arange(n, device=dev) for n in dims],
                                         indexing="ij"), -1).reshape(-1, 3)
        # every bond of the grid: cation site, anion site, slots, image crossed
        bonds = []
        for m in range(4):
            for n, (step, an) in enumerate(_BONDS[m]):
                to = ijk + torch.tensor(step, device=dev)
                wrap = torch.zeros_like(to)
                ok = torch.ones(len(to), dtype=torch.bool, device=dev)
                for k in range(3):
                    over = to[:, k] >= dims[k]
                    if per[k]:
                        wrap[:, k] = over.long()
                        to[:, k] = torch.where(over, to[:, k] - dims[k], to[:, k])
                    else:
                        ok &= ~over
                cell = torch.arange(len(to), device=dev)
                sc = cell * 8 + m
                sa = ((to[:, 0] * dims[1] + to[:, 1]) * dims[2] + to[:, 2]).clamp(
                    max=len(cell) - 1) * 8 + an
                ok &= (types[sc] > 0) & (types[sa] > 0)
                vec = torch.tensor(step, dtype=f8, device=dev) + site[an] - site[m]
                bonds.append((sc[ok], sa[ok], wrap[ok], vec))
        # atoms: sites with a bond that crosses no periodic image, in site order
        keep = torch.zeros(len(types), dtype=torch.bool, device=dev)
        for sc, sa, wrap, _ in bonds:
            inside = (wrap == 0).all(1)
            keep[sc[inside]] = True
            keep[sa[inside]] = True
        index = torch.cumsum(keep.long(), 0) - 1
        self.n_atoms = int(keep.sum())
        A = self.n_atoms
        self.atom_site = torch.nonzero(keep).reshape(-1)
        cnt = torch.zeros(A, dtype=f8, device=dev)
        E = torch.zeros(A, 10, dtype=f8, device=dev)
        shift = torch.zeros(A, dtype=f8, device=dev)
        corr = torch.zeros(A, norb, dtype=f8, device=dev)
        have = torch.zeros(A, 4, dtype=torch.bool, device=dev)  # hybrids that are bonded
        sign = torch.ones(A, dtype=f8, device=dev)
        sets = {}
        for mat in _sets(case):
            sets[materials.SPECIES[mat["cation"]]] = _parameters(mat)
        self.bonds = []
        for sc, sa, wrap, vec in bonds:
            both = keep[sc] & keep[sa]
            sc, sa, wrap = sc[both], sa[both], wrap[both]
            if not len(sc):
                continue
            v = lat * vec
            v = v.expand(len(sc), 3) if dsp is None else v + dsp[sa] - dsp[sc]
            r = v.norm(dim=1)
            d, d0 = -v / r[:, None], -(vec / vec.norm()).expand(len(sc), 3)
            ic, ia = index[sc], index[sa]
            blk = torch.empty(len(sc), norb, norb, dtype=f8, device=dev)
            for sp in torch.unique(types[sc]).tolist():
                P, S = sets[sp]
                sel = torch.nonzero(types[sc] == sp).reshape(-1)
                ratio = 0.25 * _R3 * P[31] / r[sel]
                V = {k: P[k] * ratio ** S[_ETA[k]] for k in _ETA}
                b = _blocks(d[sel], V, norb)
                b0 = _blocks(d0[:1], {k: torch.tensor([P[k]], dtype=f8, device=dev) for k in _ETA}, norb)
                blk[sel] = b
                w = torch.tensor([[S[_COEF[_KIND[a]][_KIND[c]]]
                                   / (P[_EN[0][_KIND[a]]] + P[_EN[1][_KIND[c]]])
                                   for a in range(norb)] for c in range(norb)], dtype=f8, device=dev)
                e = (b0 ** 2 - b ** 2) * (S[10] * w)
                corr.index_add_(0, ic[sel], e.sum(2))
                corr.index_add_(0, ia[sel], e.sum(1))
                for at, sh in ((ic[sel], S[15]), (ia[sel], S[16])):
                    E.index_add_(0, at, torch.tensor(P[:10], dtype=f8, device=dev).expand(len(at), 10))
                    shift.index_add_(0, at, torch.full((len(at),), sh, dtype=f8, device=dev))
                    cnt.index_add_(0, at, torch.ones(len(at), dtype=f8, device=dev))
            for at, dirs in ((ic, vec), (ia, -vec)):
                dots = dirs.cpu().numpy() @ _HYBRID.T
                have[at, int(np.argmax(np.abs(dots) >= 0.15))] = True
            phase = None
            if kvec is not None:
                w = wrap.double() @ torch.tensor(kvec, dtype=f8, device=dev)
                ph = -math.pi * (w - 2 * torch.trunc(0.5 * w))
                phase = torch.polar(torch.ones_like(ph), -ph)
            self.bonds.append((ic, ia, blk, phase))
        cat = (self.atom_site & 7) < 4
        # which side of its hybrids an atom's bonds lie on: the last slot's bond
        last = {0: _BONDS[0][3], 1: _BONDS[1][3], 2: _BONDS[2][3], 3: _BONDS[3][3]}
        for m in range(8):
            if m < 4:
                step, an = last[m]
                w = np.array(step) + workloads.SITE_POS[an] - workloads.SITE_POS[m]
            else:  # the last slot of an anion points along the opposite of a cation bond
                c, s = {4: (3, (0, 0, 0)), 5: (0, (0, -1, -1)), 6: (0, (-1, -1, 0)),
                        7: (0, (-1, 0, -1))}[m]
                w = np.array(s) + workloads.SITE_POS[c] - workloads.SITE_POS[m]
            dots = _HYBRID @ w
            first = int(np.argmax(np.abs(dots) >= 0.15))
            sign[(self.atom_site & 7) == m] = 1.0 if dots[first] > 0 else -1.0
        E, shift = E / cnt[:, None], shift / cnt
        on = torch.where(cat[:, None], E[:, _EN[1]], E[:, _EN[0]])[:, [_KIND[o] for o in range(norb)]]
        v = torch.where(have, 0.0, 0.25 * 30.0).to(f8)
        v = torch.where((cnt < 4)[:, None], v, torch.zeros_like(v))
        v0, v1 = v.sum(1), v[:, 0] - v[:, 1] + v[:, 2] - v[:, 3]
        v2, v3 = v[:, 0] - v[:, 1] - v[:, 2] + v[:, 3], v[:, 0] + v[:, 1] - v[:, 2] - v[:, 3]
        on[:, 1:5] += v0[:, None]
        on += shift[:, None] + corr
        K = torch.zeros(A, norb, norb, dtype=f8, device=dev)
        K.diagonal(dim1=1, dim2=2).copy_(on)
        for (i, j), val in {(1, 2): sign * v1, (1, 3): sign * v2, (1, 4): sign * v3,
                            (2, 3): v3, (2, 4): v2, (3, 4): v1}.items():
            K[:, i, j] = K[:, j, i] = val
        self.onsite = K
        self.lam = torch.where(cat, E[:, 9], E[:, 8])

    def hx(self, x, shift):
        """x: complex128 [atoms, nspin, norb]."""
        cplx = torch.view_as_real(x)                       # [A, s, o, 2]
        y = torch.einsum("aij,asjr->asir", self.onsite, cplx)
        if self.nspin == 2:
            U, D, L = x[:, 0], x[:, 1], self.lam
            so = torch.zeros_like(x)
            so[:, 0, 2] = -1j * L * U[:, 3] + L * D[:, 4]
            so[:, 0, 3] = 1j * L * U[:, 2] - 1j * L * D[:, 4]
            so[:, 0, 4] = -L * D[:, 2] + 1j * L * D[:, 3]
            so[:, 1, 2] = 1j * L * D[:, 3] - L * U[:, 4]
            so[:, 1, 3] = -1j * L * D[:, 2] - 1j * L * U[:, 4]
            so[:, 1, 4] = L * U[:, 2] + 1j * L * U[:, 3]
            y = y + torch.view_as_real(so)
        for ic, ia, blk, ph in self.bonds:
            xa, xc = x[ia], x[ic]
            if ph is not None:
                xa, xc = xa * ph[:, None, None], xc * ph.conj()[:, None, None]
            y.index_add_(0, ic, torch.einsum("bca,bsar->bscr", blk, torch.view_as_real(xa)))
            y.index_add_(0, ia, torch.einsum("bca,bscr->bsar", blk, torch.view_as_real(xc)))
        return torch.view_as_complex(y.contiguous()) - shift * x


def exact(case, seed):
    X = _Exact(case, seed)
    n = X.n_atoms * X.norb * X.nspin
    x = _vector(case, n, seed).double()
    xs = torch.view_as_complex(x.reshape(case.get("p", 1), X.n_atoms, X.nspin, X.norb, 2))
    if case["op"] != "lanczos":
        return torch.cat([torch.view_as_real(X.hx(v, SHIFT)).reshape(-1) for v in xs])
    q = xs[0] / xs[0].abs().square().sum().sqrt()
    prev, b, alpha, beta = torch.zeros_like(q), 0.0, [], []
    for _ in range(case["its"]):
        w = X.hx(q, 0.0)
        a = torch.vdot(q.reshape(-1), w.reshape(-1)).real
        w = w - a * q - b * prev
        b = w.abs().square().sum().sqrt()
        prev, q = q, w / b
        alpha.append(a)
        beta.append(b)
    return dict(values=None, alpha=torch.stack(alpha).cpu(), beta=torch.stack(beta).cpu())
