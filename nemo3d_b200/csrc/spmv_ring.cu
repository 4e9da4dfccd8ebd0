// H*x, the block product and the regenerating product of the eigenvector
// pass over the stored Hamiltonian: one lane per (atom, vector, spin), the
// operands staged through shared memory one bond at a time.
//
// Restates Hv_stored_20_Hzb (nemo3d/src/base/Hmult_stored.c:176-607) with the
// Lanczos alpha dot of eigen/src/lanczos.c:679-707 fused, and the block
// product matmat_mult (nemo3d/src/base/h_cmat_mult.c:21).
//
//  * A task is 32 / (vectors * spins * H) atoms of one kind (all cations or
//    all anions; 8 or 16 for 32 on small structures, see run_one), one lane per atom,
//    vector and spin (H = 2 lanes for single double vectors of the 10-orbital
//    models, see ring_split).  A cation
//    lane streams the rows of its block against its neighbour's x segment; an
//    anion lane streams the rows of the block its cation neighbour stores and
//    scales each by that neighbour's x entry (the transposed product).  A lane
//    uses a block element it loads for one complex FMA, and the lanes of an
//    atom load it together (one broadcast address).
//  * Tasks are run by pairs of warps.  The producer copies the blocks and the
//    neighbour x segments of one bond n = 0..3 of the task's atoms into a slot
//    of the pair's ring: the blocks by bulk copies (TMA, one request a block),
//    the vectors by 16-byte cp.async, eight lanes to a 128-byte line, so that
//    both units carry half of the staging.  The consumer waits on the slot's
//    barrier, multiplies and hands the slot back.  Every wait is bounded
//    (TBGPU_E_TIMEOUT in the status word; both warps leave their loops after
//    their copies landed or a second bounded wait).  The atom pitches are odd
//    multiples of 16 bytes, so the row loads have no bank conflicts.
//  * The task's own segments (and, for the regenerating product, the r before
//    them) and on-site records arrive in a slot of their own while the bonds
//    compute; the results take the own segments' place and leave by bulk
//    stores (single vectors) or as whole lines.
//
// What bounds it (10 orbitals, spin, double, 1.02M atoms): about 120 cycles an
// atom and SM, where HBM alone (2504 bytes at 6.5 TB/s) would take 115 at full
// clock, the TMA unit 67, the load/store unit 70 and the consumers 98.  Long
// runs of it sit at the 1000 W power limit (SM clock 1.5 GHz).  With every
// copy by cp.async the load/store unit carried 140 cycles and was the bound.
// The kernels this one replaced: lane per orbital row with x read by
// broadcast, 201 wavefronts an atom (0.81 against 0.53 ms in back-to-back
// passes); lane per (atom, spin) with rows straight from global memory, one
// tag lookup per lane and load (float, 381k atoms: 0.181 against 0.118 ms);
// lane-gather, 5-orbital dots, 0.43M atoms: 0.200 against 0.104 ms; a staged
// block product of 8 vectors, 66k atoms: 0.296 against 0.177 ms.
//
// Every column of a launch computes as a one-vector launch would, operation
// for operation, so regenerated recurrences are bit-identical to the first
// pass.  UPD fuses the Lanczos three-term update into the epilogue.
//
// PHASE (Bloch phases): tasks with an atom that has a bond across the
// periodic boundary (wrap[a], set with the phases) rotate the neighbours' x.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "lane_math.cuh"
#include "launch.cuh"
#include "lanczos_step.cuh"
#include "reduce.cuh"
#include "stage.cuh"
#include "tbgpu_internal.cuh"
#include "zincblende.cuh"

namespace tbgpu {

namespace {

using namespace stage;
using namespace lanemath;

// asynchronous copy of CH bytes into shared memory, zeros where ok is false
template <int CH, bool ZERO>
__device__ __forceinline__ void cpa(uint32_t dst, uintptr_t src, bool ok) {
  if constexpr (CH == 16 && !ZERO)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else if constexpr (CH == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                 "r"(ok ? 16 : 0)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(CH),
                 "r"(ok ? CH : 0)
                 : "memory");
}

// Line pc of a segment of N chunks of CH bytes at src: lane `sub` of eight
// has chunk 8 pc + sub - off, off = the MASK bits of the first chunk's place
// in its 128-byte line, so that the eight lanes move one line (only the first
// and last lines need a test).  f(byte offset in the segment) for a lane's
// chunk.
template <int N, int CH, int MASK, typename F>
__device__ __forceinline__ void line_chunk(uintptr_t src, int sub, int pc, F &&f) {
  const int c0 = sub * CH - (MASK ? int(src & uintptr_t(MASK * 16)) : 0);  // bytes
  if ((MASK == 0 || pc > 0 || c0 >= 0) && (pc * 8 + 7 < N || pc * 8 * CH + c0 < N * CH))
    f(pc * 8 * CH + c0);
}

template <typename VT, int P>
struct RingCols {
  const VT *x[P];        // input vectors (the r's; q = r * scale)
  VT *y[P];              // output: (H - shift) q, or with UPD the next r
  const VT *rp[P];       // UPD: the r before x (null: none)
  int it[P];             // scale = 1 / bet[it]; UPD: alpha[it], bet[it-1]
};

__host__ __device__ constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }

// Lanes that share the orbitals of one atom, vector and spin: two for single
// double vectors of the 10-orbital models, whose 16-atom slots (18.7 KB) would
// leave room for only 3 or 4 consumers per SM, one per scheduler (0.70 against
// 0.61 ms at 1.02M atoms).  Lane h of them owns orbitals 4h..4h+3 and 8+h
// (16-byte pairs of a block row, then one more).
__host__ __device__ constexpr int ring_split(int norb, int p, int vector_bytes) {
  return norb == 10 && p == 1 && vector_bytes == 16 ? 2 : 1;
}

// Slots per ring: a task's own data travel with its bond kSlots.  With three,
// fewer pairs fit (7 for 8 in double): 0.533 against 0.512 ms at 1.02M atoms,
// float 0.315 against 0.279.
constexpr int kSlots = 2;

// Shared-memory geometry of a configuration (bytes), tasks of TA atoms at most
template <int NORB, int NSPIN, int P, typename HT, typename VT, bool UPD, int TA>
struct RingShape {
  static constexpr int NB = NORB * NSPIN;
  static constexpr int H = ring_split(NORB, P, int(sizeof(VT)));
  static constexpr int NO = NORB / H;                 // orbitals per lane
  static constexpr int LPA = P * NSPIN * H;           // lanes per atom
  static constexpr int APW = 32 / LPA < TA ? 32 / LPA : TA;  // atoms per task
  static constexpr int BLKB = NORB * NORB * int(sizeof(HT));
  // a block's 16-byte chunks (a block of the 5-orbital models may start
  // inside one), and their odd pitch
  static constexpr int BCH = BLKB % 16 ? cdiv(BLKB + 16 - (BLKB % 8 ? 4 : 8), 16) : BLKB / 16;
  static constexpr int BPITCH = (BCH | 1) * 16;
  static constexpr int BMASK = BCH == 50 ? 6 : BCH == 25 ? 7 : BCH == 13 ? 3 : 1;
  static constexpr int BPC = cdiv(BCH + BMASK, 8);    // line pieces per block
  // Atoms of a task whose block comes by a bulk copy, one request of the TMA
  // unit (about 17 cycles for 800 bytes, 12 for 400, as many for 200); the
  // rest come by lines through the load/store unit, which also carries the
  // vectors.  Small blocks of single vectors leave it four atoms' a task, a
  // quarter of 16 or an eighth of 32 (2M-atom float dot 0.50 against 0.53 ms,
  // 5-orbital dots 104 against 111 us); 800-byte blocks none (half of them by
  // lines: 0.48 against 0.44 ms, 1.02M).
  static constexpr int BULK = BLKB >= 800 || P > 1 || APW < 16 ? APW : APW - 4;
  // a vector segment: NSPIN parts of SEG bytes
  static constexpr int SEG = NORB * int(sizeof(VT));
  static constexpr int XB = NSPIN * SEG;
  static constexpr int XCH_B = XB % 16 ? 8 : 16;      // bytes per chunk
  static constexpr int XCH = XB / XCH_B;
  // pitch of a spin part: eight lanes (a quarter warp's 16-byte loads) reading
  // eight segments of 160 bytes need an odd pitch, four (H = 2) do not
  static constexpr int SP = SEG == 160 && H == 1 ? 176 : SEG;
  static constexpr int XP = cdiv(NSPIN * SP, 16) * 16;
  static constexpr int XMASK = XCH_B == 8 ? 0 : XCH == 20 ? 4 : XCH == 10 ? 6 : 3;
  static constexpr int XPC = cdiv(XCH + XMASK, 8);
  static constexpr int ONS = onsite_len(NB);
  static constexpr int RCH = ONS * int(sizeof(HT)) / 16;
  static constexpr int RPITCH = RCH * 16 + 16;
  static constexpr int SLOT = APW * (BPITCH + P * XP);
  static constexpr int OWN = APW * P * XP;
  static constexpr int PREV = UPD ? OWN : 0;
  static constexpr int TASK = OWN + PREV + APW * RPITCH;
  // of a warp pair: the ring, the task's own data, two barriers per slot
  __host__ __device__ static constexpr int pair_bytes() {
    return cdiv(kSlots * SLOT + TASK + 16 * kSlots, 128) * 128;
  }
};

// The lines of NSEG segments, NPC each, eight lanes (group ag) per segment:
// line(get(s, u), s, pc) with u the group's count of segments so far.  get may
// shuffle, so all lanes call it.  pc is a compile-time constant in every call,
// so only a segment's first and last lines are tested, and a segment is looked
// up once.  (With the groups taking line after line of one flat count where
// NSEG is no multiple of four, a division, a lookup and both tests went with
// every line: blocks of 5 vectors, 140k atoms, 264 against 154 us without spin
// and 419 against 241 with it, where a block of 8 takes 198 and 320.)
template <int NSEG, int NPC, typename G, typename F>
__device__ __forceinline__ void for_lines(int ag, G &&get, F &&line) {
#pragma unroll
  for (int u = 0; u < cdiv(NSEG, 4); u++) {
    const int s = ag + 4 * u;
    const bool in = NSEG % 4 == 0 || s < NSEG;
    const auto v = get(in ? s : NSEG - 1, u);
    if (in) {
#pragma unroll
      for (int pc = 0; pc < NPC; pc++) line(v, s, pc);
    }
  }
}

template <typename T>
__device__ __forceinline__ void lds_rows2(const double *p, T (&r)[20]) {
#pragma unroll
  for (int k = 0; k < 10; k++) {
    const double2 v = reinterpret_cast<const double2 *>(p)[k];
    r[2 * k] = T(v.x);
    r[2 * k + 1] = T(v.y);
  }
}
template <typename T>
__device__ __forceinline__ void lds_rows2(const float *p, T (&r)[20]) {
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const float4 v = reinterpret_cast<const float4 *>(p)[k];
    r[4 * k] = T(v.x);
    r[4 * k + 1] = T(v.y);
    r[4 * k + 2] = T(v.z);
    r[4 * k + 3] = T(v.w);
  }
}
// one block row, or the five elements 4h..4h+3, 8+h of it (p at element 4h
// or at 8 + h: even elements start on 2-element boundaries)
template <typename T>
__device__ __forceinline__ void lds_pairs(const double *p, T *r, int n) {
#pragma unroll
  for (int k = 0; k < n; k++) {
    const double2 v = reinterpret_cast<const double2 *>(p)[k];
    r[2 * k] = T(v.x);
    r[2 * k + 1] = T(v.y);
  }
}
template <typename T>
__device__ __forceinline__ void lds_pairs(const float *p, T *r, int n) {
#pragma unroll
  for (int k = 0; k < n; k++) {
    const float2 v = reinterpret_cast<const float2 *>(p)[k];
    r[2 * k] = T(v.x);
    r[2 * k + 1] = T(v.y);
  }
}
template <int N>
__device__ __forceinline__ void lds_seg(const double2 *p, double2 (&v)[N]) {
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = p[k];
}
template <int N>
__device__ __forceinline__ void lds_seg(const float2 *p, float2 (&v)[N]) {
  if constexpr (N % 2 == 0) {
#pragma unroll
    for (int k = 0; k < N / 2; k++) {
      const float4 t = reinterpret_cast<const float4 *>(p)[k];
      v[2 * k] = make_float2(t.x, t.y);
      v[2 * k + 1] = make_float2(t.z, t.w);
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = p[k];
  }
}
template <int N>
__device__ __forceinline__ void sts_seg(double2 *p, const double2 (&v)[N]) {
#pragma unroll
  for (int k = 0; k < N; k++) p[k] = v[k];
}
template <int N>
__device__ __forceinline__ void sts_seg(float2 *p, const float2 (&v)[N]) {
  if constexpr (N % 2 == 0) {
#pragma unroll
    for (int k = 0; k < N / 2; k++)
      reinterpret_cast<float4 *>(p)[k] = make_float4(v[2 * k].x, v[2 * k].y, v[2 * k + 1].x, v[2 * k + 1].y);
  } else {
#pragma unroll
    for (int k = 0; k < N; k++) p[k] = v[k];
  }
}

// The atoms of a task that a lane issues copies for (U of them: those of its
// group of eight lanes, or lane l < atoms per task holds atom l and the
// lanes shuffle) and their bonds from the next one on: four times the
// neighbour for a cation, the neighbour's block for an anion, -1 for none
template <int U>
struct TaskMeta {
  int a[U];
  int v[U][4];
};

template <int NORB, int NSPIN, int P, typename HT, typename VT, bool DOT, bool UPD, bool PHASE,
          int TA, int PAIRS>
__global__ void __launch_bounds__(PAIRS * 64, 1)
    k_hx_ring(int ncat, int nan, const int *__restrict__ order, const int4 *__restrict__ bonds,
              const HT *__restrict__ onsite, const HT *__restrict__ blocks,
              const __grid_constant__ RingCols<VT, P> A, const double *bet, const double *alpha,
              double shift_d, double *partial, unsigned int *counter, double *alpha_out,
              int alpha_idx, const double2 *phase, const unsigned char *wrap,
              const unsigned char *skip, int *status) {
  using S = RingShape<NORB, NSPIN, P, HT, VT, UPD, TA>;
  using RT = typename RealOf<VT>::T;
  constexpr int NB = S::NB, APW = S::APW, LPA = S::LPA, H = S::H, NO = S::NO;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pair = warp < PAIRS ? warp : warp - PAIRS;
  const int ag = lane >> 3, sub = lane & 7;
  const bool live = lane < APW * LPA;
  const int al = live ? lane / LPA : APW - 1;          // this lane's atom of the task,
  const int h = H > 1 ? (lane % LPA) / (P * NSPIN) : 0;     // part of the orbitals,
  const int col = (lane % (P * NSPIN)) / NSPIN, sp = lane % NSPIN;  // vector and spin
  unsigned char *wbase = smem + pair * S::pair_bytes();
  unsigned char *own_p = wbase + kSlots * S::SLOT;
  // per slot: full (the 32 producer lanes' copies and the bulk copies landed),
  // empty (consumed)
  const uint32_t bars = smem_addr(wbase) + S::pair_bytes() - 16 * kSlots;
  if (warp < PAIRS && lane == 0) {
#pragma unroll
    for (int k = 0; k < kSlots; k++) {
      mbar_init(bars + 16 * k, 33);
      mbar_init(bars + 16 * k + 8, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  wait_for_previous();

  // The tasks in sequence: cations 0, anions 0, cations 1, ...  Round t of the
  // grid takes the next of them for each of its nw warp pairs, and every pair
  // alternates between the kinds (with an even nw its place in the round
  // moves on by one each time): both kinds advance through the structure
  // together, and the blocks an anion task reads were read by cation tasks
  // shortly before.  With a kind per pair the faster kind runs ahead and the
  // blocks leave L2 in between (2M-atom float dot: 0.77 against 0.56 ms).
  const int nw = int(gridDim.x) * PAIRS;
  const int tasks = 2 * cdiv(max(ncat, nan), APW);
  int place = pair * int(gridDim.x) + int(blockIdx.x);
  auto advance = [&](int q) {  // the task of the pair's next round
    if (nw & 1) return q + nw;
    const bool over = ++place == nw;
    if (over) place = 0;
    return q + nw + (over ? 1 - nw : 1);
  };
  // first atom of task q in the order, and one past its kind's last
  auto first = [&](int q) { return (q & 1 ? ncat : 0) + (q >> 1) * APW; };
  auto last = [&](int q) { return q & 1 ? ncat + nan : ncat; };
  // the atom of this lane's results (-1: none)
  auto lane_atom = [&](int q) {
    const int j = first(q) + al;
    return q < tasks && live && j < last(q) ? __ldg(order + j) : -1;
  };
  auto lane_skip = [&](int a) { return skip && a >= 0 ? int(skip[a]) : 0; };
  // a task without atoms, or whose atoms are all left out, is neither staged
  // nor computed
  auto runs = [&](int a, int left) { return __any_sync(0xffffffffu, a >= 0 && !left) != 0; };
  double dot = 0.0;
  bool late = false;  // a bounded wait ran out

  if (warp >= PAIRS) {
    // ---- producer: copies the pair's bonds in order, kSlots ahead -----------
    constexpr bool DIRECT = P == 1 && APW <= 16;
    constexpr int U = DIRECT ? APW / 4 : 1;
    auto load_meta = [&](int q) {
      TaskMeta<U> M;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int l = DIRECT ? ag + 4 * u : lane;
        const int j = first(q) + l;
        const bool in = q < tasks && l < APW && j < last(q);
        M.a[u] = in ? __ldg(order + j) : 0;
        const int4 w = in ? __ldg(bonds + j) : make_int4(-1, -1, -1, -1);
        M.v[u][0] = w.x; M.v[u][1] = w.y; M.v[u][2] = w.z; M.v[u][3] = w.w;
      }
      return M;
    };
    // atom s of the task: the group's own register, or shuffled
    auto of_atom = [&](const int (&r)[U], int s, int u) {
      return DIRECT ? r[DIRECT ? u : 0] : __shfl_sync(0xffffffffu, r[0], s);
    };
    auto copy_seg = [&](uintptr_t src, uint32_t dst, int pc, bool ok) {
      line_chunk<S::XCH, S::XCH_B, S::XMASK>(src, sub, pc, [&](int o) {
        cpa<S::XCH_B, true>(dst + o + (S::SP > S::SEG && o >= S::SEG ? S::SP - S::SEG : 0), src + o, ok);
      });
    };
    const uint32_t ring = smem_addr(wbase), own = smem_addr(own_p);
    uint32_t slot = 0, phase_bit = 1;  // the first pass over the slots finds them empty
    int q = place, q1 = advance(q);
    TaskMeta<U> cur = load_meta(q);
    int la = lane_atom(q), la1 = lane_atom(q1);
    int left = lane_skip(la);
    auto issue_own = [&]() {
      for_lines<APW * P, S::XPC>(
          ag, [&](int s, int u) { return long(of_atom(cur.a, s / P, u)) * S::XB; },
          [&](long o, int s, int pc) {
            const int v = P == 1 ? 0 : s % P;
            copy_seg(reinterpret_cast<uintptr_t>(A.x[v]) + o, own + s * S::XP, pc, true);
            if (UPD) {
              const VT *rp = A.rp[v] ? A.rp[v] : A.x[v];
              copy_seg(reinterpret_cast<uintptr_t>(rp) + o, own + S::OWN + s * S::XP, pc,
                       A.rp[v] != nullptr);
            }
          });
      for_lines<APW, cdiv(S::RCH, 8)>(
          ag,
          [&](int s, int u) {
            return reinterpret_cast<uintptr_t>(onsite) + long(of_atom(cur.a, s, u)) * (S::RCH * 16);
          },
          [&](uintptr_t src, int s, int pc) {
            line_chunk<S::RCH, 16, 0>(src, sub, pc, [&](int o) {
              cpa<16, false>(own + S::OWN + S::PREV + s * S::RPITCH + o, src + o, true);
            });
          });
    };
    while (q < tasks && !late) {
      const bool cat = !(q & 1), run = runs(la, left);
      const int q2 = advance(q1);
      const TaskMeta<U> nxt = load_meta(q1);
      const int la2 = lane_atom(q2), left1 = lane_skip(la1);
      if (run) {
#pragma unroll 1
        for (int n = 0; n < 4; n++) {
          const uint32_t full = bars + 16 * slot, dst = ring + slot * S::SLOT;
          if (!mbar_wait(full + 8, phase_bit)) late = true;
          if (__any_sync(0xffffffffu, late)) {
            late = true;
            break;
          }
          if (lane == 0) mbar_expect_tx(full, uint32_t(S::BULK * S::BCH * 16));
          __syncwarp();
          // bond 0 of the task is consumed, so the task before it has left
          // the own slot: this task's own data, covered by this bond's barrier
          if (n == kSlots) issue_own();
          int v[U], id[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            v[u] = cur.v[u][0];
            cur.v[u][0] = cur.v[u][1];
            cur.v[u][1] = cur.v[u][2];
            cur.v[u][2] = cur.v[u][3];
            // a cation's own block; for a missing bond the (zeroed) one of the atom
            id[u] = cat || v[u] < 0 ? cur.a[u] * 4 + n : v[u];
          }
          // the blocks: one bulk copy per atom for the first BULK, the rest by lines
          {
            int mine = id[0];
#pragma unroll
            for (int u = 1; u < U; u++) mine = sub == u ? id[u] : mine;
            const int s = DIRECT ? ag + 4 * sub : lane;
            if (DIRECT ? sub < S::BULK / 4 : lane < S::BULK) {
              uintptr_t src = reinterpret_cast<uintptr_t>(blocks) + long(mine) * S::BLKB;
              if (S::BLKB % 16) src &= ~uintptr_t(15);
              bulk_g2s(dst + s * S::BPITCH, reinterpret_cast<const void *>(src), S::BCH * 16, full);
            }
          }
          if constexpr (S::BULK < APW) {
#pragma unroll
            for (int u = S::BULK / 4; u < APW / 4; u++) {
              const int s = ag + 4 * u;
              uintptr_t src = reinterpret_cast<uintptr_t>(blocks) + long(of_atom(id, s, u)) * S::BLKB;
              if (S::BLKB % 16) src &= ~uintptr_t(15);
#pragma unroll
              for (int pc = 0; pc < S::BPC; pc++)
                line_chunk<S::BCH, 16, S::BMASK>(src, sub, pc, [&](int o) {
                  cpa<16, false>(dst + s * S::BPITCH + o, src + o, true);
                });
            }
          }
          struct Src { uintptr_t p; bool ok; };
          for_lines<APW * P, S::XPC>(
              ag,
              [&](int s, int u) {
                const int w = of_atom(v, s / P, u);
                const VT *x = A.x[P == 1 ? 0 : s % P];
                return Src{reinterpret_cast<uintptr_t>(x) + long(max(w, 0) >> 2) * S::XB, w >= 0};
              },
              [&](Src t, int s, int pc) { copy_seg(t.p, dst + APW * S::BPITCH + s * S::XP, pc, t.ok); });
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
          if (++slot == kSlots) {
            slot = 0;
            phase_bit ^= 1;
          }
        }
      }
      q = q1;
      q1 = q2;
      cur = nxt;
      la = la1;
      la1 = la2;
      left = left1;
    }
    cp_wait<0>();
    if (late)  // once more, bounded, for the bulk copies in flight
      for (uint32_t k = 0; k < kSlots; k++)
        mbar_wait(bars + 16 * k, k < slot ? phase_bit ^ 1 : phase_bit);
  } else {
    // ---- consumer --------------------------------------------------------------
    auto orb = [&](int j) { return H == 1 ? j : j < 4 ? 4 * h + j : 8 + h; };
    const int it = A.it[col];
    const RT scale = RT(bet ? 1.0 / bet[it] : 1.0);
    const RT shift = RT(shift_d);
    double al_u = 0.0, bp_u = 0.0, iq_u = 0.0, ip_u = 0.0;
    if (UPD) {  // as k_update: alpha[it], bet[it], bet[it-1]
      al_u = alpha[it];
      bp_u = bet[it];
      iq_u = 1.0 / bp_u;
      ip_u = it > 0 ? 1.0 / bet[it - 1] : 0.0;
    }
    auto lane_rot = [&](int a) { return PHASE && a >= 0 ? int(wrap[a]) : 0; };
    auto lane_bonds = [&](int q) {  // 5-orbital models: where the blocks start
      const int j = first(q) + al;
      return S::BLKB % 16 && q < tasks && live && j < last(q) ? __ldg(bonds + j)
                                                              : make_int4(-1, -1, -1, -1);
    };
    uint32_t slot = 0, phase_bit = 0;
    int q = place, q1 = advance(q);
    int la = lane_atom(q), la1 = lane_atom(q1);
    int left = lane_skip(la), rotl = lane_rot(la);
    int4 lb = lane_bonds(q);
    const int seg = (al * P + col) * S::XP + sp * S::SP;  // this lane's segment
    // Double vectors without a split: 40 registers of sums, as many of a whole
    // x segment and of two block rows leave none to load ahead, so the x
    // entries are read as they are used and the next ten block elements while
    // the last ten are multiplied (block of 4 at 381k atoms 0.54 against 0.57
    // ms, of 8 at 66k 0.177 against 0.188)
    constexpr bool PIPE = NORB == 10 && H == 1 && sizeof(VT) == 16;
    static_assert(!(PHASE && (PIPE || sizeof(VT) == 8)), "Bloch phases: single double vectors");
    constexpr bool BULK_OUT = P == 1 && S::XP == S::XB;
    while (q < tasks && !late) {
      const bool cat = !(q & 1), run = runs(la, left);
      const int q2 = advance(q1);
      const int la2 = lane_atom(q2), left1 = lane_skip(la1), rotl1 = lane_rot(la1);
      const int4 lb1 = lane_bonds(q1);
      if (run) {
        VT acc[NO];
#pragma unroll
        for (int i = 0; i < NO; i++) acc[i].x = acc[i].y = RT(0);
        bool rot = false;
        if (PHASE) rot = __any_sync(0xffffffffu, rotl);
#pragma unroll 1
        for (int n = 0; n < 4; n++) {
          const uint32_t full = bars + 16 * slot;
          if (!mbar_wait(full, phase_bit)) late = true;
          if (__any_sync(0xffffffffu, late)) {
            late = true;
            break;
          }
          const unsigned char *st = wbase + slot * S::SLOT;
          const HT *bk = reinterpret_cast<const HT *>(st + al * S::BPITCH);
          if (S::BLKB % 16) {  // where the block starts in its first chunk
            const int w = n == 0 ? lb.x : n == 1 ? lb.y : n == 2 ? lb.z : lb.w;
            const int id = cat || w < 0 ? max(la, 0) * 4 + n : w;
            bk += (unsigned(id) * unsigned(S::BLKB) & 15u) / unsigned(sizeof(HT));
          }
          const VT *xp = reinterpret_cast<const VT *>(st + APW * S::BPITCH + seg);
          constexpr bool FLOAT = sizeof(VT) == 8;
          VT xn[PIPE || FLOAT ? 1 : NORB];
          if constexpr (!PIPE && !FLOAT) lds_seg(xp, xn);
          if (PHASE && rot) {
            const double2 ph = phase[long(max(la, 0)) * 4 + n];
#pragma unroll
            for (int k = 0; k < NORB; k++) {
              const VT u = xn[k];
              xn[k].x = RT(ph.x) * u.x - RT(ph.y) * u.y;
              xn[k].y = RT(ph.x) * u.y + RT(ph.y) * u.x;
            }
          }
          // cation: y_a[i] += sum_k B_n[i][k] x_nb[k]; anion: y_a[k] += sum_i
          // B[i][k] x_nb[i], B the block its cation neighbour stores
          if constexpr (PIPE) {
            RT r[2][10];
            VT xs[2][2];
            if (cat) {
              // step (k, half): five rows of a column pair
              auto load = [&](int t, RT (&b)[10], VT (&x2)[2]) {
                const int k = t & ~1, i0 = t & 1 ? 5 : 0;
#pragma unroll
                for (int j = 0; j < 5; j++) {
                  RT v[2];
                  lds_pairs(bk + (i0 + j) * NORB + k, v, 1);
                  b[2 * j] = v[0];
                  b[2 * j + 1] = v[1];
                }
                if (!(t & 1)) {
                  x2[0] = xp[k];
                  x2[1] = xp[k + 1];
                }
              };
              load(0, r[0], xs[0]);
#pragma unroll
              for (int t = 0; t < 10; t++) {
                if (t < 9) load(t + 1, r[(t + 1) & 1], xs[((t + 1) >> 1) & 1]);
                const VT(&x2)[2] = xs[(t >> 1) & 1];
                const int i0 = t & 1 ? 5 : 0;
#pragma unroll
                for (int j = 0; j < 5; j++) cfma(acc[i0 + j], r[t & 1][2 * j], x2[0]);
#pragma unroll
                for (int j = 0; j < 5; j++) cfma(acc[i0 + j], r[t & 1][2 * j + 1], x2[1]);
              }
            } else {
              lds_pairs(bk, r[0], 5);
              xs[0][0] = xp[0];
#pragma unroll
              for (int i = 0; i < NORB; i++) {
                if (i < NORB - 1) {
                  lds_pairs(bk + (i + 1) * NORB, r[(i + 1) & 1], 5);
                  xs[(i + 1) & 1][0] = xp[i + 1];
                }
#pragma unroll
                for (int k = 0; k < NORB; k++) cfma(acc[k], r[i & 1][k], xs[i & 1][0]);
              }
            }
          } else if constexpr (H == 2) {
            if (cat) {
#pragma unroll
              for (int k = 0; k < NORB; k += 2) {  // two columns of the lane's five rows
                RT r[NO][2];
#pragma unroll
                for (int j = 0; j < NO; j++) lds_pairs(bk + orb(j) * NORB + k, r[j], 1);
#pragma unroll
                for (int j = 0; j < NO; j++) cfma(acc[j], r[j][0], xn[k]);
#pragma unroll
                for (int j = 0; j < NO; j++) cfma(acc[j], r[j][1], xn[k + 1]);
              }
            } else {
#pragma unroll
              for (int i = 0; i < NORB; i++) {
                RT r[4];
                lds_pairs(bk + i * NORB + 4 * h, r, 2);
                const RT r4 = RT(bk[i * NORB + 8 + h]);
#pragma unroll
                for (int j = 0; j < 4; j++) cfma(acc[j], r[j], xn[i]);
                cfma(acc[4], r4, xn[i]);
              }
            }
          } else if constexpr (FLOAT) {
            // Float sums: each bond's NORB terms by themselves, then added to
            // the bonds before them.  One chain of 40 terms is 7.8e-8 off the
            // 64-bit result (127k atoms, sp3d5s*), the sums by bond 6.3e-8.
            auto rows2 = [&](int i, RT (&r)[2 * NORB]) {
              if constexpr (NORB == 10) {
                lds_rows2(bk + i * NORB, r);
              } else {
#pragma unroll
                for (int k = 0; k < 2 * NORB; k++) r[k] = i * NORB + k < NORB * NORB ? RT(bk[i * NORB + k]) : RT(0);
              }
            };
            auto first_term = [](RT m, VT x) { return VT{m * x.x, m * x.y}; };
            if (cat) {
              VT xv[NORB];
              lds_seg(xp, xv);
#pragma unroll
              for (int i = 0; i < NORB; i += 2) {
                RT r[2 * NORB];
                rows2(i, r);
                VT t0 = first_term(r[0], xv[0]), t1 = first_term(r[NORB], xv[0]);
#pragma unroll
                for (int k = 1; k < NORB; k++) {
                  cfma(t0, r[k], xv[k]);
                  cfma(t1, r[NORB + k], xv[k]);
                }
                acc[i].x += t0.x;
                acc[i].y += t0.y;
                if (i + 1 < NORB) {
                  acc[i + 1].x += t1.x;
                  acc[i + 1].y += t1.y;
                }
              }
            } else {
              VT t[NORB];
#pragma unroll
              for (int i = 0; i < NORB; i += 2) {
                RT r[2 * NORB];
                rows2(i, r);
                VT x2[2];
                if constexpr (NORB == 10) {
                  lds_seg(xp + i, x2);
                } else {
                  x2[0] = xp[i];
                  if (i + 1 < NORB) x2[1] = xp[i + 1];
                }
#pragma unroll
                for (int k = 0; k < NORB; k++) {
                  if (i == 0) t[k] = first_term(r[k], x2[0]);
                  else cfma(t[k], r[k], x2[0]);
                  if (i + 1 < NORB) cfma(t[k], r[NORB + k], x2[1]);
                }
              }
#pragma unroll
              for (int k = 0; k < NORB; k++) {
                acc[k].x += t[k].x;
                acc[k].y += t[k].y;
              }
            }
          } else {
            static_assert(NORB == 5, "10 orbitals: the branches above");
            if (cat) {
#pragma unroll
              for (int i = 0; i < NORB; i++)
#pragma unroll
                for (int k = 0; k < NORB; k++) cfma(acc[i], RT(bk[i * NORB + k]), xn[k]);
            } else {
#pragma unroll
              for (int i = 0; i < NORB; i++)
#pragma unroll
                for (int k = 0; k < NORB; k++) cfma(acc[k], RT(bk[i * NORB + k]), xn[i]);
            }
          }
          // (bond 0 also hands the own slot on: its results have left)
          if (BULK_OUT && n == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();  // every lane has read the slot
          if (lane == 0) mbar_arrive(full + 8);
          if (++slot == kSlots) {
            slot = 0;
            phase_bit ^= 1;
          }
        }
        if (late) break;
        // own data: copied before bond kSlots of the task and so covered by its
        // full barrier
        const VT *xo_p = reinterpret_cast<const VT *>(own_p + seg);
        const VT *ot_p = reinterpret_cast<const VT *>(own_p + (al * P + col) * S::XP + (NSPIN - 1 - sp) * S::SP);
        const HT *rec = reinterpret_cast<const HT *>(own_p + S::OWN + S::PREV + al * S::RPITCH);
        VT xo[NO];
        if constexpr (H == 1) {
          lds_seg(xo_p, xo);
        } else {
#pragma unroll
          for (int j = 0; j < NO; j++) xo[j] = xo_p[orb(j)];
        }
#pragma unroll
        for (int j = 0; j < NO; j++) cfma(acc[j], RT(rec[sp * NORB + orb(j)]), xo[j]);
        if (rec[NB + 1] != HT(0)) {  // dangling-bond sp3 couplings (orbitals 1..4)
          const RT sx = RT(rec[NB + 2]), sy = RT(rec[NB + 3]), sz = RT(rec[NB + 4]);
          const RT cxy = RT(rec[NB + 5]), cxz = RT(rec[NB + 6]), cyz = RT(rec[NB + 7]);
          const VT x1 = xo_p[1], x2 = xo_p[2], x3 = xo_p[3], x4 = xo_p[4];
          if (h == 0) {
            cfma(acc[1], sx, x2); cfma(acc[1], sy, x3); cfma(acc[1], sz, x4);
            cfma(acc[2], sx, x1); cfma(acc[2], cxy, x3); cfma(acc[2], cxz, x4);
            cfma(acc[3], sy, x1); cfma(acc[3], cxy, x2); cfma(acc[3], cyz, x4);
          }
          if (H == 1 || h == 1) {
            VT &a4 = acc[H == 1 ? 4 : 0];
            cfma(a4, sz, x1); cfma(a4, cxz, x2); cfma(a4, cyz, x3);
          }
        }
        if (NSPIN == 2) {  // on-site spin-orbit (mb_ham_spds_so.h): p orbitals 2..4
          const RT L = RT(rec[NB]), Lu = sp ? -L : L;
          if (h == 0) {
            const VT o4 = ot_p[4];
            cfma_im(acc[2], -Lu, xo[3]); cfma(acc[2], Lu, o4);
            cfma_im(acc[3], Lu, xo[2]);  cfma_im(acc[3], -L, o4);
          }
          if (H == 1 || h == 1) {
            VT &a4 = acc[H == 1 ? 4 : 0];
            cfma(a4, -Lu, ot_p[2]); cfma_im(a4, L, ot_p[3]);
          }
        }
        const bool valid = la >= 0 && !left;
        const VT *rp_p = reinterpret_cast<const VT *>(own_p + S::OWN + seg);
        double d = 0.0;
#pragma unroll
        for (int j = 0; j < NO; j++) {  // w = scale * acc - shift * (scale * x)
          VT u, w;
          u.x = mul_rn(scale, xo[j].x);
          u.y = mul_rn(scale, xo[j].y);
          w.x = fma_rn(scale, acc[j].x, -mul_rn(shift, u.x));
          w.y = fma_rn(scale, acc[j].y, -mul_rn(shift, u.y));
          if (DOT) d += double(u.x) * double(w.x) + double(u.y) * double(w.y);
          if constexpr (UPD) {
            const VT rpv = rp_p[orb(j)];
            const double2 r = lanczos_update_entry(
                make_double2(double(w.x), double(w.y)),
                make_double2(double(xo[j].x), double(xo[j].y)),
                make_double2(double(rpv.x), double(rpv.y)), al_u, bp_u, iq_u, ip_u);
            w.x = RT(r.x);
            w.y = RT(r.y);
          }
          acc[j] = w;
        }
        if (DOT && valid) dot += d;
        __syncwarp();  // the atom's other lanes have read their entries
        if (live) {  // the results take the own segments' place and leave as whole lines
          VT *w = const_cast<VT *>(xo_p);
          if constexpr (H == 1) {
            sts_seg(w, acc);
          } else {
#pragma unroll
            for (int j = 0; j < NO; j++) w[orb(j)] = acc[j];
          }
        }
        if constexpr (BULK_OUT) {
          // whole segments by bulk stores: one per four atoms that follow one
          // another in memory, else one per atom
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          const int lead = (al & ~3) * LPA;  // the four atoms' first lane
          const int a0 = __shfl_sync(0xffffffffu, la, lead);
          const unsigned in_run = __ballot_sync(0xffffffffu, valid && la == a0 + (al & 3));
          constexpr unsigned FOUR = 4 * LPA == 32 ? ~0u : (1u << (4 * LPA % 32)) - 1u;
          const bool whole = APW % 4 == 0 && ((in_run >> lead) & FOUR) == FOUR;
          if (whole ? lane == lead : valid && lane == al * LPA) {
            const uintptr_t dst = reinterpret_cast<uintptr_t>(A.y[0]) + long(la) * S::XB;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                         "r"(smem_addr(own_p) + al * S::XP), "r"(whole ? 4 * S::XB : S::XB)
                         : "memory");
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        } else {
          __syncwarp();
          for_lines<APW * P, S::XPC>(
              ag, [&](int s, int) { return __shfl_sync(0xffffffffu, valid ? la : -1, (s / P) * LPA); },
              [&](int a, int s, int pc) {
                const uintptr_t dst =
                    reinterpret_cast<uintptr_t>(A.y[P == 1 ? 0 : s % P]) + long(max(a, 0)) * S::XB;
                line_chunk<S::XCH, S::XCH_B, S::XMASK>(dst, sub, pc, [&](int o) {
                  const unsigned char *src =
                      own_p + s * S::XP + o + (S::SP > S::SEG && o >= S::SEG ? S::SP - S::SEG : 0);
                  if (a < 0) return;
                  if constexpr (S::XCH_B == 16)
                    *reinterpret_cast<float4 *>(dst + o) = *reinterpret_cast<const float4 *>(src);
                  else
                    *reinterpret_cast<float2 *>(dst + o) = *reinterpret_cast<const float2 *>(src);
                });
              });
        }
        // (the own slot is free once bond 0 of the next task is arrived on)
      }
      q = q1;
      q1 = q2;
      la = la1;
      la1 = la2;
      lb = lb1;
      left = left1;
      rotl = rotl1;
    }
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (late && lane == 0 && status) atomicExch(status, TBGPU_E_TIMEOUT);
  if (DOT) grid_reduce<PAIRS * 64>(dot, partial, counter, alpha_out, alpha_idx, false);
}

constexpr int kMaxSmem = 227 * 1024;
// Warp pairs per SM: as many as shared memory holds, at most 12; the
// 10-orbital double products take at most eight, which leaves them the 128
// registers a thread they need (nine: 0.63 against 0.53 ms at 1.02M atoms,
// block of 4 at 381k 0.73 against 0.55).
template <class S>
constexpr int ring_pairs(bool wide) {
  const int w = kMaxSmem / S::pair_bytes(), most = wide ? 8 : 12;
  return w > most ? most : w;
}

struct RingLaunch {
  const double *bet, *alpha;
  double shift;
  double *partial;  // null: the context's
  unsigned int *counter;
  int cap;
  double *alpha_out;
  int aidx;
};

template <int NORB, int NSPIN, int P, typename HT, typename VT, bool DOT, bool UPD, bool PHASE,
          int TA = 32>
int run_ring(Ctx &c, const RingCols<VT, P> &A, RingLaunch L, cudaStream_t s) {
  using S = RingShape<NORB, NSPIN, P, HT, VT, UPD, TA>;
  constexpr int PAIRS = ring_pairs<S>(NORB == 10 && sizeof(VT) == 16);
  constexpr int smem = PAIRS * S::pair_bytes();
  static_assert(PAIRS >= 1, "a task does not fit shared memory");
  const auto kernel = k_hx_ring<NORB, NSPIN, P, HT, VT, DOT, UPD, PHASE, TA, PAIRS>;
  static std::atomic<unsigned long long> attr_done{0};
  if (ensure_smem_attr(attr_done, c.device, kernel, smem)) return TBGPU_E_CUDA;
  const int ncat = int(c.ncations), nan = int(c.natoms - c.ncations);
  const int tasks = 2 * cdiv(std::max(ncat, nan), S::APW);
  const unsigned grid = unsigned(std::min(tasks, c.sms));
  if (DOT && !L.partial) {
    int rc = ensure_partials(c, int(grid));
    if (rc) return rc;
    L.partial = c.d_partial;
    L.counter = c.d_counter;
  } else if (DOT && int(grid) > L.cap) {
    return set_error(TBGPU_E_ARG);
  }
  launch_overlapped(kernel, grid, PAIRS * 64, smem, s, ncat, nan, c.d_order, c.d_bonds,
                    ham_onsite<HT>(c), ham_blocks<HT>(c), A, L.bet, L.alpha, L.shift, L.partial,
                    L.counter, L.alpha_out, L.aidx, c.d_phase, c.d_wrap, c.d_skip, c.d_status);
  TB_CUDA(cudaGetLastError());
  return TBGPU_OK;
}

template <int NORB, int NSPIN, typename HT, typename VT, int TA>
int run_tasks(Ctx &c, const VT *x, VT *y, int it, const RingLaunch &L, cudaStream_t s) {
  RingCols<VT, 1> A{};
  A.x[0] = x;
  A.y[0] = y;
  A.it[0] = it;
  if constexpr (sizeof(VT) == sizeof(double2)) {
    if (c.bloch)
      return L.alpha_out ? run_ring<NORB, NSPIN, 1, HT, VT, true, false, true, TA>(c, A, L, s)
                         : run_ring<NORB, NSPIN, 1, HT, VT, false, false, true, TA>(c, A, L, s);
  }
  return L.alpha_out ? run_ring<NORB, NSPIN, 1, HT, VT, true, false, false, TA>(c, A, L, s)
                     : run_ring<NORB, NSPIN, 1, HT, VT, false, false, false, TA>(c, A, L, s);
}

// One vector.  A product with fewer tasks than warp pairs takes as long as one
// task, whose producer copies for every atom the task has room for: 8 or 16
// with several lanes an atom, 32 with one (5 orbitals or float vectors, no
// spin).  Those 32 make way for tasks of
//  * 8 atoms while the SMs get at most four of them (216 atoms, sp3s*: 4.9 us,
//    5.7 with 16, 7.4 with 32; float sp3d5s* 5.4, 6.3 and 7.2.  At 5,832 and
//    8,000 atoms float sp3d5s* is at 6.0 to 6.4 with either, so the line is
//    where each scheduler has one pair),
//  * 16 atoms while the warp pairs get at most one (the 10-orbital models:
//    eight a SM).  17,576 atoms, sp3s*: 6.7 us, 7.9 with 32; float sp3d5s* 7.6
//    against 8.1.  Past the line the second round costs more than it saves:
//    32,768 atoms, sp3s*, 10.7 against 8.8; float sp3d5s*, 27,000, 9.2 against
//    8.8.
// Results are the same bit for bit, only the fused dot sums in another order.
template <int NORB, int NSPIN, typename HT, typename VT>
int run_one(Ctx &c, const VT *x, VT *y, int it, const RingLaunch &L, cudaStream_t s) {
  if constexpr (RingShape<NORB, NSPIN, 1, HT, VT, false, 32>::APW == 32) {
    const int kind = int(std::max(c.ncations, c.natoms - c.ncations));
    auto per_sm = [&](int atoms, int tasks) { return 2 * cdiv(kind, atoms) <= tasks * c.sms; };
    if (per_sm(8, 4)) return run_tasks<NORB, NSPIN, HT, VT, 8>(c, x, y, it, L, s);
    if (per_sm(16, NORB == 5 ? 12 : 8))
      return run_tasks<NORB, NSPIN, HT, VT, 16>(c, x, y, it, L, s);
  }
  return run_tasks<NORB, NSPIN, HT, VT, 32>(c, x, y, it, L, s);
}

template <typename HT, typename VT>
int run_model(Ctx &c, const VT *x, VT *y, int it, const RingLaunch &L, cudaStream_t s) {
  if (c.norb == 10 && c.nspin == 2) return run_one<10, 2, HT, VT>(c, x, y, it, L, s);
  if (c.norb == 10 && c.nspin == 1) return run_one<10, 1, HT, VT>(c, x, y, it, L, s);
  if (c.norb == 5 && c.nspin == 2) return run_one<5, 2, HT, VT>(c, x, y, it, L, s);
  if (c.norb == 5 && c.nspin == 1) return run_one<5, 1, HT, VT>(c, x, y, it, L, s);
  return set_error(TBGPU_E_UNSUPPORTED);
}

template <int NSPIN, int P>
int run_block_p(Ctx &c, const double *x, long xs, double *y, long ys, double shift,
                cudaStream_t s) {
  RingCols<double2, P> A{};
  for (int v = 0; v < P; v++) {
    A.x[v] = reinterpret_cast<const double2 *>(x + v * xs);
    A.y[v] = reinterpret_cast<double2 *>(y + v * ys);
  }
  const RingLaunch L{nullptr, nullptr, shift, nullptr, nullptr, 0, nullptr, 0};
  return run_ring<10, NSPIN, P, double, double2, false, false, false>(c, A, L, s);
}

template <int NSPIN>
int run_block(Ctx &c, int p, const double *x, long xs, double *y, long ys, double shift,
              cudaStream_t s) {
  switch (p) {
    case 2: return run_block_p<NSPIN, 2>(c, x, xs, y, ys, shift, s);
    case 3: return run_block_p<NSPIN, 3>(c, x, xs, y, ys, shift, s);
    case 4: return run_block_p<NSPIN, 4>(c, x, xs, y, ys, shift, s);
    case 5: return run_block_p<NSPIN, 5>(c, x, xs, y, ys, shift, s);
    case 6: return run_block_p<NSPIN, 6>(c, x, xs, y, ys, shift, s);
    case 7: return run_block_p<NSPIN, 7>(c, x, xs, y, ys, shift, s);
    case 8: return run_block_p<NSPIN, 8>(c, x, xs, y, ys, shift, s);
  }
  return set_error(TBGPU_E_ARG);
}

}  // namespace

int launch_spmv_ring(Ctx &c, const double *x, double *y, double shift, const double *xnorm,
                     int xidx, double *alpha_out, int aidx, cudaStream_t s) {
  const RingLaunch L{xnorm, nullptr, shift, nullptr, nullptr, 0, alpha_out, aidx};
  const double2 *X = reinterpret_cast<const double2 *>(x);
  double2 *Y = reinterpret_cast<double2 *>(y);
  return c.ham_fp32 ? run_model<float>(c, X, Y, xidx, L, s) : run_model<double>(c, X, Y, xidx, L, s);
}

int launch_spmv_ring_f32(Ctx &c, const float *x, float *y, double shift, const double *xnorm,
                         int xidx, double *alpha_out, int aidx, cudaStream_t s) {
  const RingLaunch L{xnorm, nullptr, shift, nullptr, nullptr, 0, alpha_out, aidx};
  return run_model<float>(c, reinterpret_cast<const float2 *>(x), reinterpret_cast<float2 *>(y),
                          xidx, L, s);
}

// The same with the alpha dot reduced through caller-provided scratch:
// partial[cap] doubles and a zeroed counter.  Allocates nothing.
int launch_spmv_ring_scratch(Ctx &c, const double *x, double *y, double shift, double *partial,
                             unsigned int *counter, int cap, double *dot_out, cudaStream_t s) {
  const RingLaunch L{nullptr, nullptr, shift, partial, counter, cap, dot_out, 0};
  const double2 *X = reinterpret_cast<const double2 *>(x);
  double2 *Y = reinterpret_cast<double2 *>(y);
  return c.ham_fp32 ? run_model<float>(c, X, Y, 0, L, s) : run_model<double>(c, X, Y, 0, L, s);
}

bool lane_supported(const Ctx &c) { return c.norb == 10 && !c.bloch && !c.recompute; }

// Regeneration of p Lanczos segments in one pass (p <= lane_max_cols): column j
// takes r = x[j] at iteration it[j] (q = r / bet[it]) and r_prev = rp[j]
// (null at it = 0) and writes the next r, exactly as one product followed by
// k_update would.
template <typename VT>
int launch_lane_regen(Ctx &c, int p, const VT *const *x, VT *const *y, const VT *const *rp,
                      const int *it, const double *bet, const double *alpha, cudaStream_t s) {
  constexpr bool F32 = sizeof(VT) == sizeof(float2);
  if (!lane_supported(c) || p < 1 || p > lane_max_cols(F32)) return set_error(TBGPU_E_UNSUPPORTED);
  if (F32 && !c.ham_fp32) return set_error(TBGPU_E_UNSUPPORTED);
  const RingLaunch L{bet, alpha, 0.0, nullptr, nullptr, 0, nullptr, 0};
  auto run = [&](auto cols) -> int {
    constexpr int P = decltype(cols)::value;
    RingCols<VT, P> A{};
    for (int j = 0; j < P; j++) {
      A.x[j] = x[j];
      A.y[j] = y[j];
      A.rp[j] = rp[j];
      A.it[j] = it[j];
    }
    if (c.ham_fp32)
      return c.nspin == 2 ? run_ring<10, 2, P, float, VT, false, true, false>(c, A, L, s)
                          : run_ring<10, 1, P, float, VT, false, true, false>(c, A, L, s);
    if constexpr (!F32)
      return c.nspin == 2 ? run_ring<10, 2, P, double, VT, false, true, false>(c, A, L, s)
                          : run_ring<10, 1, P, double, VT, false, true, false>(c, A, L, s);
    return set_error(TBGPU_E_UNSUPPORTED);
  };
  if (p == 1) return run(std::integral_constant<int, 1>());
  if (p == 2) return run(std::integral_constant<int, 2>());
  if constexpr (F32) {
    if (p == 3) return run(std::integral_constant<int, 3>());
    return run(std::integral_constant<int, 4>());
  }
  return set_error(TBGPU_E_UNSUPPORTED);
}

template int launch_lane_regen<double2>(Ctx &, int, const double2 *const *, double2 *const *,
                                        const double2 *const *, const int *, const double *,
                                        const double *, cudaStream_t);
template int launch_lane_regen<float2>(Ctx &, int, const float2 *const *, float2 *const *,
                                       const float2 *const *, const int *, const double *,
                                       const double *, cudaStream_t);

// y + v*ystride = (H - shift)(x + v*xstride), v < p (p <= 8; strides in
// doubles).  One launch for the 10-orbital models with the double-precision
// store at the Gamma point and p >= 2 (variant 1 aside), one H*x launch per
// vector otherwise.
int launch_spmm(Ctx &c, int p, const double *x, long xstride, double *y, long ystride,
                double shift, cudaStream_t s) {
  if (p < 1 || p > 8) return set_error(TBGPU_E_ARG);
  if (p >= 2 && c.norb == 10 && !c.bloch && !c.ham_fp32 && !c.recompute && c.spmv_variant != 1)
    return c.nspin == 2 ? run_block<2>(c, p, x, xstride, y, ystride, shift, s)
                        : run_block<1>(c, p, x, xstride, y, ystride, shift, s);
  for (int v = 0; v < p; v++) {
    int rc = launch_spmv(c, x + v * xstride, y + v * ystride, shift, nullptr, 0, nullptr, 0, s);
    if (rc) return rc;
  }
  return TBGPU_OK;
}

}  // namespace tbgpu

extern "C" int tbgpu_hx_block_dev(tbgpu_ctx *ctx, int p, double shift, const double *x_dev,
                                  double *y_dev) {
  using namespace tbgpu;
  if (!ctx || !x_dev || !y_dev || p < 1 || p > 8 || misaligned16(x_dev) || misaligned16(y_dev))
    return set_error(TBGPU_E_ARG);
  Ctx &c = *reinterpret_cast<Ctx *>(ctx);
  if (!c.built) return set_error(TBGPU_E_STATE);
  set_error(TBGPU_OK);
  const long n = 2 * c.natoms * c.nb;  // doubles per vector
  return launch_spmm(c, p, x_dev, n, y_dev, n, shift, c.stream);
}
