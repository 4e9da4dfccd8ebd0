// Zincblende topology on the GPU: which sites hold atoms, the atom numbering,
// the four-neighbour table and the surface flags.
//
// Restates, for a dense cell grid:
//   remove_few_bonded_atoms(0)          nemo3d/src/base/geo_struct.c:1527-1579
//   get_total_hamiltonian_dimension_and_offsets
//                                       nemo3d/src/base/ham3d_final.c:547-568
//   FindSurfaceAtoms (bit 0, isOnSurface) nemo3d/src/base/geo_struct.c:1374-1463
// Atoms are numbered in site order (cell-major, k fastest, then in-cell site),
// which is the reference's vector layout.
#include <algorithm>

#include <cub/block/block_scan.cuh>
#include <cub/device/device_scan.cuh>

#include "tbgpu_internal.cuh"
#include "zincblende.cuh"

namespace tbgpu {

struct Grid {
  int nx, ny, nz, px, py, pz;
};

// neighbour site of site s along slot n; -1 outside a closed boundary.
// *wrapped is set when a periodic image is crossed; w (optional) receives the
// image crossed along each axis (-1, 0, +1).
__device__ __forceinline__ long nbr_site(const Grid g, long s, int n, bool *wrapped,
                                         int *w = nullptr) {
  const int m = int(s & 7);
  long cell = s >> 3;
  int k = int(cell % g.nz);
  int j = int((cell / g.nz) % g.ny);
  int i = int(cell / ((long)g.nz * g.ny));
  int c[3] = {i + c_nnmap[m][n][0], j + c_nnmap[m][n][1], k + c_nnmap[m][n][2]};
  const int dim[3] = {g.nx, g.ny, g.nz};
  const int per[3] = {g.px, g.py, g.pz};
  *wrapped = false;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (w) w[d] = 0;
    if (c[d] < 0 || c[d] >= dim[d]) {
      if (!per[d]) return -1;
      *wrapped = true;
      if (w) w[d] = c[d] < 0 ? -1 : 1;
      c[d] = (c[d] + dim[d]) % dim[d];
    }
  }
  return ((((long)c[0] * g.ny + c[1]) * g.nz + c[2]) << 3) + c_nnmap[m][n][3];
}

// 1 for a site that holds an atom bonded to at least one in-domain atom
// (periodic images are not counted here, as in remove_few_bonded_atoms).
__global__ void k_mark(Grid g, long nsites, const unsigned char *type, int *flag) {
  long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= nsites) return;
  int f = 0;
  if (type[s]) {
    for (int n = 0; n < 4; n++) {
      bool w;
      long t = nbr_site(g, s, n, &w);
      if (t >= 0 && !w && type[t]) { f = 1; break; }
    }
  }
  flag[s] = f;
}

__global__ void k_finalize(Grid g, long nsites, const int *flag, const int *index,
                           int *site_index, int *atom_site, int4 *nbr,
                           unsigned char *site_m, unsigned char *surface) {
  long s = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (s >= nsites) return;
  if (!flag[s]) {
    site_index[s] = -1;
    return;
  }
  const int a = index[s];
  site_index[s] = a;
  atom_site[a] = int(s);
  site_m[a] = (unsigned char)(s & 7);
  int b[4], cnt = 0;
  for (int n = 0; n < 4; n++) {
    bool w;
    long t = nbr_site(g, s, n, &w);
    b[n] = (t >= 0 && flag[t]) ? index[t] : -1;
    cnt += b[n] >= 0;
  }
  nbr[a] = make_int4(b[0], b[1], b[2], b[3]);
  surface[a] = (unsigned char)(cnt != 4);
}

// Phase of H[a][b] for every bond: the conjugate of the Bloch factor of the
// periodic image crossed from a to b, exp(i*ph) with ph = -pi*(w.k -
// 2*int(0.5*w.k)) (geo_struct::phasePeriodic, nemo3d/src/base/geo_struct.h:
// 811-826, applied in Hmult_stored.c:386-437); 1 inside the domain.
__global__ void k_phase(Grid g, long natoms, const int *atom_site, const int4 *nbr,
                        double k0, double k1, double k2, double2 *phase, unsigned char *wrap) {
  long a = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (a >= natoms) return;
  const long s = atom_site[a];
  const int4 v = nbr[a];
  const int b[4] = {v.x, v.y, v.z, v.w};
  bool any = false;
  for (int n = 0; n < 4; n++) {
    double2 p = make_double2(1.0, 0.0);
    bool wrapped;
    int w[3];
    nbr_site(g, s, n, &wrapped, w);
    if (b[n] >= 0 && wrapped) {
      double ph = w[0] * k0 + w[1] * k1 + w[2] * k2;
      ph = -M_PI * (ph - 2 * (int)(0.5 * ph));
      double sn, cs;
      sincos(ph, &sn, &cs);
      p = make_double2(cs, -sn);
      any = true;
    }
    phase[a * 4 + n] = p;
  }
  wrap[a] = any;
}

int build_phases(Ctx &c) {
  if (!c.d_phase) TB_CUDA(cudaMalloc(&c.d_phase, sizeof(double2) * 4 * c.natoms));
  if (!c.d_wrap) TB_CUDA(cudaMalloc(&c.d_wrap, c.natoms));
  Grid g{c.nx, c.ny, c.nz, c.periodic[0], c.periodic[1], c.periodic[2]};
  const int threads = 256;
  const unsigned blocks = unsigned((c.natoms + threads - 1) / threads);
  k_phase<<<blocks, threads, 0, c.stream>>>(g, c.natoms, c.d_atom_site, c.d_nbr, c.kvec[0],
                                            c.kvec[1], c.kvec[2], c.d_phase, c.d_wrap);
  TB_CUDA(cudaGetLastError());
  return TBGPU_OK;
}

// Work order of the H*x kernels.  Atoms are numbered in site order, so the
// atoms of a k-pencil of cells (i, j, 0..nz-1) are one contiguous run.
// Visiting pencils j-block by j-block (kPencilBlock pencils wide, i slower
// than j inside a block) keeps the atoms that share a bond, and with it the x
// segments and bond blocks read twice, within a few thousand atoms of each
// other in processing order, so the second read hits L2; in plain atom order
// the i-direction neighbours are a whole y-z plane apart.
constexpr int kPencilBlock = 8;

// The order of the ring kernel (spmv_ring.cu): all cations, then all anions,
// each kind in the pencil order above; beside each atom its bonds, four times
// the neighbour for a cation, the block its neighbour stores the bond in
// (neighbour * 4 + slot) for an anion, -1 for none.  Built on the device in
// three launches without a wait: the host reads the count of cations where it
// reads the build's status.  Only a stored Hamiltonian has the order, behind
// its blocks: 20 bytes an atom in an allocation of their own are a further
// mapping of device memory (building 65,688 atoms: 3.1 against 2.75 ms).

// first atom on a site not below s (atoms are numbered in site order)
__device__ __forceinline__ int first_atom(int natoms, const int *__restrict__ atom_site, long s) {
  int lo = 0, hi = natoms;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(atom_site + mid) < s) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// cations[p] and anions[p] (COUNT), or the pencil's entries from at[0][p] and
// at[1][p] (plus the number of cations); one warp per pencil, per sites each
template <bool COUNT>
__global__ void k_kind_order(int natoms, int npen, long per, const int *__restrict__ atom_site,
                             const unsigned char *__restrict__ site_m,
                             const int4 *__restrict__ nbr, const int *__restrict__ at,
                             const int *__restrict__ ncations, int *__restrict__ cations,
                             int *__restrict__ anions, int *__restrict__ order,
                             int4 *__restrict__ bonds) {
  const int p = int(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (p >= npen) return;
  const int lane = threadIdx.x & 31;
  const unsigned before = (1u << lane) - 1u;
  const int start = first_atom(natoms, atom_site, p * per);
  const int end = first_atom(natoms, atom_site, (p + 1) * per);
  int nc = COUNT ? 0 : at[p], na = COUNT ? 0 : at[npen + p] + *ncations;
  for (int a0 = start; a0 < end; a0 += 32) {
    const int a = a0 + lane;
    const bool in = a < end;
    const int m = in ? site_m[a] : 0;
    const unsigned cat = __ballot_sync(0xffffffffu, in && m < 4);
    const unsigned an = __ballot_sync(0xffffffffu, in && m >= 4);
    if (!COUNT && in) {
      const int to = m < 4 ? nc + __popc(cat & before) : na + __popc(an & before);
      const int4 v = nbr[a];
      auto bond = [&](int b, int n) { return b < 0 ? -1 : b * 4 + (m < 4 ? 0 : c_rev_slot[m][n]); };
      order[to] = a;
      bonds[to] = make_int4(bond(v.x, 0), bond(v.y, 1), bond(v.z, 2), bond(v.w, 3));
    }
    nc += __popc(cat);
    na += __popc(an);
  }
  if (COUNT && lane == 0) {
    cations[p] = nc;
    anions[p] = na;
  }
}

// at[0][p], at[1][p]: cations and anions of the pencils visited before p;
// ncations: all of them.  One block.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads)
    k_kind_scan(int nx, int ny, const int *__restrict__ cations, const int *__restrict__ anions,
                int *__restrict__ at, int *__restrict__ ncations) {
  using Scan = cub::BlockScan<int, kScanThreads>;
  __shared__ typename Scan::TempStorage tmp;
  const int npen = nx * ny, full = ny / kPencilBlock * kPencilBlock;
  int nc = 0, na = 0;
  for (int v0 = 0; v0 < npen; v0 += kScanThreads) {
    const int v = v0 + int(threadIdx.x);
    int p = 0, cat = 0, an = 0;
    if (v < npen) {  // the v-th pencil visited: j-blocks, i, j within the block
      const bool whole = v < full * nx;
      const int w = whole ? kPencilBlock : ny - full, r = whole ? v % (w * nx) : v - full * nx;
      const int jb = whole ? v / (w * nx) * kPencilBlock : full;
      p = r / w * ny + jb + r % w;
      cat = cations[p];
      an = anions[p];
    }
    int c0, a0, ct, t;
    Scan(tmp).ExclusiveSum(cat, c0, ct);
    __syncthreads();
    Scan(tmp).ExclusiveSum(an, a0, t);
    __syncthreads();
    if (v < npen) {
      at[p] = nc + c0;
      at[npen + p] = na + a0;
    }
    nc += ct;
    na += t;
  }
  if (threadIdx.x == 0) *ncations = nc;
}

// into room (natoms * kOrderBytes, 16-byte aligned) behind the stored blocks;
// *ncations (device) receives the count of cations.  The counts per pencil are
// kept in the reduction scratch meanwhile: a stream-ordered allocation would
// map memory again, which the pool has given back in the waits before.
int build_work_order(Ctx &c, void *room, int *ncations) {
  const int na = int(c.natoms), npen = c.nx * c.ny;
  const long per = long(c.nz) * 8;
  c.d_bonds = static_cast<int4 *>(room);
  c.d_order = reinterpret_cast<int *>(c.d_bonds + na);
  const int rc = ensure_partials(c, std::max(partials_of_build(c), 2 * npen));
  if (rc) return rc;
  int *tmp = reinterpret_cast<int *>(c.d_partial);  // at[2 npen], cations[npen], anions[npen]
  int *cations = tmp + 2 * size_t(npen), *anions = cations + npen;
  const unsigned wb = unsigned((npen + 7) / 8);
  k_kind_order<true><<<wb, 256, 0, c.stream>>>(na, npen, per, c.d_atom_site, c.d_site_m, c.d_nbr,
                                               nullptr, nullptr, cations, anions, nullptr,
                                               nullptr);
  k_kind_scan<<<1, kScanThreads, 0, c.stream>>>(c.nx, c.ny, cations, anions, tmp, ncations);
  k_kind_order<false><<<wb, 256, 0, c.stream>>>(na, npen, per, c.d_atom_site, c.d_site_m, c.d_nbr,
                                                tmp, ncations, nullptr, nullptr, c.d_order,
                                                c.d_bonds);
  TB_CUDA(cudaGetLastError());
  return TBGPU_OK;
}

int build_topology(Ctx &c) {
  Grid g{c.nx, c.ny, c.nz, c.periodic[0], c.periodic[1], c.periodic[2]};
  const long ns = c.nsites;
  int *flag = nullptr, *index = nullptr;
  void *tmp = nullptr;
  size_t tmp_bytes = 0;
  const int threads = 256;
  const unsigned blocks = unsigned((ns + threads - 1) / threads);
  int rc = TBGPU_OK;
  if (cudaMallocAsync(&flag, sizeof(int) * (ns + 1), c.stream) != cudaSuccess ||
      cudaMallocAsync(&index, sizeof(int) * (ns + 1), c.stream) != cudaSuccess)
    return set_error(TBGPU_E_NOMEM);
  TB_CUDA(cudaMemsetAsync(flag + ns, 0, sizeof(int), c.stream));
  k_mark<<<blocks, threads, 0, c.stream>>>(g, ns, c.d_type, flag);
  TB_CUDA(cudaGetLastError());
  // exclusive scan over ns+1 entries: index[ns] is the atom count
  cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, flag, index, ns + 1, c.stream);
  TB_CUDA(cudaMallocAsync(&tmp, tmp_bytes, c.stream));
  TB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, flag, index, ns + 1, c.stream));
  int natoms = 0;
  TB_CUDA(cudaMemcpyAsync(&natoms, index + ns, sizeof(int), cudaMemcpyDeviceToHost,
                          c.stream));
  TB_CUDA(cudaStreamSynchronize(c.stream));
  c.natoms = natoms;
  if (natoms <= 0) rc = set_error(TBGPU_E_ARG);
  if (rc == TBGPU_OK) {
    TB_CUDA(cudaMalloc(&c.d_site_index, sizeof(int) * ns));
    TB_CUDA(cudaMalloc(&c.d_atom_site, sizeof(int) * natoms));
    TB_CUDA(cudaMalloc(&c.d_nbr, sizeof(int4) * natoms));
    TB_CUDA(cudaMalloc(&c.d_site_m, natoms));
    TB_CUDA(cudaMalloc(&c.d_surface, natoms));
    k_finalize<<<blocks, threads, 0, c.stream>>>(g, ns, flag, index, c.d_site_index,
                                                 c.d_atom_site, c.d_nbr, c.d_site_m,
                                                 c.d_surface);
    TB_CUDA(cudaGetLastError());
  }
  cudaFreeAsync(tmp, c.stream);
  cudaFreeAsync(flag, c.stream);
  cudaFreeAsync(index, c.stream);
  return rc;
}

}  // namespace tbgpu
