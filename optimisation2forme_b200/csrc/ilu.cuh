// Block ILU(0) preconditioner of the adjoint operator A = J^T, for the
// preconditioned BiCGSTAB (no reference counterpart: the reference runs
// BiCGSTAB with the identity preconditioner, src/shape_optimization.cpp:699,
// which on realistic meshes needs 10^4-10^5 iterations).  The preconditioner
// changes only the convergence path: the solution is the same J^T lambda = b
// at the same true-residual tolerance.
//
// A in block form (4x4 blocks, one row per cell).  From the matrix-free
// product (src/shape_optimization.cpp:433-482), with B_{c,e} the flux
// Jacobian block of edge e on cell c's side and s = -1 for the left cell,
// +1 for the right cell of e:
//   A_cc = sum_e (s_c L_e / V_c) B_{c,e}^T
//   A_co = (s_o L_e / V_o) B_{c,e}^T      (o: the other cell of e)
// Rows are stored as 5 blocks: [0] the diagonal, [1..4] the neighbours in the
// cell's slot order (ilu.nbr[k][c], -1 when absent).
//
// Factorization (IKJ form, rows in a reverse Cuthill-McKee order, each level
// of the dependency DAG processed by one launch): for row i and its lower
// neighbours k in increasing order, L_ik = A_ik D_k^{-1}, then
// A_ij -= L_ik U_kj for every block j of row k above k that row i also holds;
// finally D_i^{-1} is stored.  Solves: forward y_i = r_i - sum_{k<i} L_ik y_k,
// backward z_i = D_i^{-1} (y_i - sum_{j>i} U_ij z_j).
#pragma once

#include "kernels.cuh"
#include "sweep_plan.hpp"

namespace o2f {

// Assemble the block rows of A from the Jacobian blocks of k_jt_blocks.
__global__ void __launch_bounds__(kBlock) k_ilu_assemble(int64_t nc, const int32_t* __restrict__ jslot, Geom<double> g,
                                                         const int2* __restrict__ ec,
                                                         const uint8_t* __restrict__ ebc,
                                                         const double* __restrict__ blk, double shift,
                                                         IluDev ilu) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  double* row = ilu.A + c * 80;
  double diag[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) diag[i] = 0.0;
  const double Vc = g.cgeom[c].c;
  for (int k = 0; k < 4; ++k) {
    double* nb = row + 16 * (1 + k);
#pragma unroll
    for (int i = 0; i < 16; ++i) nb[i] = 0.0;
    const int s = jslot[(int64_t)k * nc + c];
    if (s < 0) continue;
    const int e = s >> 1;
    const bool left = (s & 1) == 0;
    const double L = g.egeom[e].c;
    const double* B = blk + (int64_t)e * 32 + (left ? 0 : 16);
    const double sc = (left ? -1.0 : 1.0) * L / Vc;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) diag[r * 4 + q] += sc * B[q * 4 + r];  // B^T
    if (ebc[e] != 0) continue;
    const int2 cc = ec[e];
    const int o = left ? cc.y : cc.x;
    const double so = (left ? 1.0 : -1.0) * L / g.cgeom[o].c;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) nb[r * 4 + q] = so * B[q * 4 + r];
  }
  if (shift > 0.0) {  // pseudo-time shift: s times the block's max row sum
    double nrm = 0.0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      nrm = fmax(nrm, fabs(diag[r * 4]) + fabs(diag[r * 4 + 1]) + fabs(diag[r * 4 + 2]) + fabs(diag[r * 4 + 3]));
#pragma unroll
    for (int r = 0; r < 4; ++r) diag[r * 5] += (diag[r * 5] < 0.0 ? -shift : shift) * nrm;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) row[i] = diag[i];
}

// One level of the factorization.  Sixteen lanes solve a row, one matrix
// element each: a level is bound by the latency of its rows, and with a
// thread per row that was a chain of some 700 FP64 operations through local
// memory.  What a solve costs besides its iterations, most of it here: 75k
// rows 16 -> 4.1 ms, and 2.8 with the levels overlapped as below; 300k rows
// 36 -> 9.1 -> 5.8.  Every element sees the operations of Gauss-Jordan
// elimination with partial pivoting, and of the block products, in the same
// order.
constexpr int kFactorBlock = 128;
constexpr int kFactorRows = kFactorBlock / 16;

__device__ __forceinline__ double lane16(double v, int src) { return __shfl_sync(0xffffffffu, v, src, 16); }
__device__ __forceinline__ int lane16(int v, int src) { return __shfl_sync(0xffffffffu, v, src, 16); }

// Element (r, q) of the inverse of the block whose element (r, q) is a; false
// for a singular block (the inverse is then the identity).
__device__ __forceinline__ bool mat4_inv16(double a, int r, int q, double& inv) {
  const double one = r == q ? 1.0 : 0.0;
  inv = one;
  bool regular = true;
  for (int col = 0; col < 4; ++col) {
    int piv = col;
    double best = fabs(lane16(a, col * 5));
    for (int k = col + 1; k < 4; ++k) {
      const double v = fabs(lane16(a, k * 4 + col));
      if (v > best) {
        best = v;
        piv = k;
      }
    }
    if (!(best > 0.0)) regular = false;
    // rows col and piv change places
    const int from = (r == col ? piv : r == piv ? col : r) * 4 + q;
    a = lane16(a, from);
    inv = lane16(inv, from);
    const double d = 1.0 / lane16(a, col * 5);
    if (r == col) {
      a *= d;
      inv *= d;
    }
    const double f = lane16(a, r * 4 + col), pa = lane16(a, col * 4 + q), pi = lane16(inv, col * 4 + q);
    if (r != col && f != 0.0) {
      a -= f * pa;
      inv -= f * pi;
    }
  }
  if (!regular) inv = one;
  return regular;
}

// A level may start while the one before it runs (all launches but the
// first): it then loads its own rows, which no other level writes, and waits
// for that level's results.  It lets its successor start after that wait, so
// that the assembled rows are complete when any level reads them.
__global__ void __launch_bounds__(kFactorBlock) k_ilu_factor(const int32_t* __restrict__ cells, int n, IluDev ilu,
                                                             int* status) {
  const int t = (blockIdx.x * kFactorBlock + threadIdx.x) >> 4;
  const int e = threadIdx.x & 15, r = e >> 2, q = e & 3;
  const bool mine = t < n;
  const int64_t nc = ilu.nc;
  const int i = mine ? cells[t] : 0;
  double* row = ilu.A + (int64_t)i * 80;
  const int pi = mine ? ilu.pos[i] : 0;
  // lane 4 k + m: neighbour m of neighbour k
  const int nk = mine ? ilu.nbr[(int64_t)r * nc + i] : -1;
  const int pk_e = nk >= 0 ? ilu.pos[nk] : -1;
  const int j_e = nk >= 0 ? ilu.nbr[(int64_t)q * nc + nk] : -1;
  const int pj_e = j_e >= 0 ? ilu.pos[j_e] : -1;
  double blk[5];
#pragma unroll
  for (int b = 0; b < 5; ++b) blk[b] = mine ? row[16 * b + e] : 0.0;
  int nb[4], pk[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    nb[k] = lane16(nk, 4 * k);
    pk[k] = lane16(pk_e, 4 * k);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (nk >= 0 && pk_e < pi) {  // one line a block: the factors this row will read
    asm volatile("prefetch.global.L1 [%0];" ::"l"(ilu.A + (int64_t)nk * 80 + 16 * (1 + q)));
    if (q == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(ilu.Dinv + (int64_t)nk * 16));
  }
  // lower neighbours in increasing ILU position (equal ones in slot order)
  int last = -1, last_slot = -1;
  for (int a = 0; a < 4; ++a) {
    int slot = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool low = nb[k] >= 0 && pk[k] < pi && (pk[k] > last || (pk[k] == last && k > last_slot));
      if (low && (slot < 0 || pk[k] < pk[slot < 0 ? 0 : slot])) slot = k;
    }
    const bool on = slot >= 0;
    if (!__any_sync(0xffffffffu, on)) break;
    int kc = 0, pks = 0;
    double aik = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (slot == k) {
        kc = nb[k];
        pks = pk[k];
        aik = blk[1 + k];
      }
    if (on) {
      last = pks;
      last_slot = slot;
    }
    // L = A_ik D_k^{-1}
    const double* D = ilu.Dinv + (int64_t)(on ? kc : i) * 16 + q;
    const double L = lane16(aik, 4 * r) * (on ? D[0] : 0.0) + lane16(aik, 4 * r + 1) * (on ? D[4] : 0.0) +
                     lane16(aik, 4 * r + 2) * (on ? D[8] : 0.0) + lane16(aik, 4 * r + 3) * (on ? D[12] : 0.0);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (slot == k) blk[1 + k] = L;
    const double l0 = lane16(L, 4 * r), l1 = lane16(L, 4 * r + 1), l2 = lane16(L, 4 * r + 2), l3 = lane16(L, 4 * r + 3);
    // subtract L_ik U_kj for the upper blocks j of row k held by row i
    const double* rowk = ilu.A + (int64_t)(on ? kc : i) * 80;
    for (int m = 0; m < 4; ++m) {
      const int j = lane16(j_e, 4 * (on ? slot : 0) + m), pj = lane16(pj_e, 4 * (on ? slot : 0) + m);
      int dst = -1;
      if (on && j >= 0 && pj > pks) {
        if (j == i) {
          dst = 0;
        } else {
#pragma unroll
          for (int s = 0; s < 4; ++s)
            if (nb[s] == j) dst = 1 + s;
        }
      }
      if (dst < 0) continue;
      const double* U = rowk + 16 * (1 + m) + q;
      const double prod = l0 * U[0] + l1 * U[4] + l2 * U[8] + l3 * U[12];
#pragma unroll
      for (int b = 0; b < 5; ++b)
        if (dst == b) blk[b] -= prod;
    }
  }
  double inv;
  const bool regular = mat4_inv16(blk[0], r, q, inv);
  if (!mine) return;
#pragma unroll
  for (int b = 0; b < 5; ++b) row[16 * b + e] = blk[b];
  ilu.Dinv[(int64_t)i * 16 + e] = inv;
  if (!regular && e == 0) atomicExch(status, 1);
}

// Sync-free triangular sweeps (one launch per triangle).  Rows are processed
// in a level order of the triangle's dependency graph (ilu.sweep: forward
// levels, then backward levels), a topological order, so the rows of one
// 32-row chunk are mostly independent.  Warps take chunks from a counter
// (see k_ilu_sweep for why the waits cannot deadlock).
//
// The solved values are their own ready signals: every output slot holds
// the sentinel bit pattern kSweepEmpty until its row writes the solution,
// and a waiting row polls the 8-byte words of its dependencies' slots
// (relaxed loads at GPU scope, single-copy atomic per word) until none is
// the sentinel, so a level costs one L2 round trip and no fence.  The
// forward sweep writes into ilu.tmp and resets the backward sweep's output
// to the sentinel; the backward sweep reads ilu.tmp and resets it after
// reading, so both buffers are empty again for the next application.  A
// computed NaN is stored as the canonical NaN, never as the sentinel.
//
// Waits are bounded: past ilu.spin_limit polls (default kSweepSpinLimit) the
// warp records sync->err and stops waiting, and every other waiting row
// gives up once it sees the error; the host turns it into an error status.
constexpr int kSweepBlock = 128;
constexpr long long kSweepSpinLimit = 1ll << 22;
constexpr unsigned long long kSweepEmpty = 0x7ff4f11ed5eed000ull;  // a NaN no arithmetic produces

__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const void* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed_u64(void* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long sweep_bits(double x) {
  return x != x ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(x);
}

__device__ __forceinline__ void store_empty(Vec4<double>* p) {
  unsigned long long* q = reinterpret_cast<unsigned long long*>(p);
#pragma unroll
  for (int k = 0; k < 4; ++k) st_relaxed_u64(q + k, kSweepEmpty);
}

// Fill a sweep buffer with the sentinel (set-up of ilu.tmp).
__global__ void k_ilu_empty(int64_t n, Vec4<double>* y) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) store_empty(y + i);
}

// kForward: tmp_i = r_i - sum_{k lower} L_ik tmp_k; z_i <- empty.
// backward: z_i = D_i^{-1} (tmp_i - sum_{j upper} U_ij z_j); tmp_i <- empty.
// A small grid of persistent warps (ilu_sweep_blocks): each warp claims the
// next 32-row chunk, solves it, and claims again, so only the warps near the
// front of the dependency levels poll -- a launch of one warp per chunk kept
// thousands of warps polling and saturated the load path.  Claims are in
// order and a warp claims again only after finishing its chunk, so every
// claimed chunk belongs to a running warp and the earliest unfinished row
// has its dependencies done: no deadlock for any grid size.  The last warp
// to leave resets the counters for the next launch (all its claims, failing
// ones included, come before it leaves).
template <bool kForward>
__global__ void __launch_bounds__(kSweepBlock) k_ilu_sweep(int n, IluDev ilu, const Vec4<double>* r,
                                                           Vec4<double>* z, const int* gate) {
  if (gated(gate)) return;
  constexpr unsigned int kFull = 0xffffffffu;
  SweepSync* sync = ilu.sync + (kForward ? 0 : 1);
  Vec4<double>* out = kForward ? ilu.tmp : z;  // slots this sweep fills (empty on entry)
  const int lane = threadIdx.x & 31;
  const unsigned int nchunks = (unsigned int)(n + 31) / 32u;
  const unsigned int nwarps = gridDim.x * (unsigned int)(kSweepBlock / 32);
  const int64_t nc = ilu.nc;
  while (true) {
    unsigned int chunk = 0;
    if (lane == 0) chunk = atomicAdd(&sync->claim, 1u);
    chunk = __shfl_sync(kFull, chunk, 0);
    if (chunk >= nchunks) break;
    const int p = (int)chunk * 32 + lane;
    const bool active = p < n;
    int i = 0, dep[4], ndep = 0, slot[4];
    Vec4<double> own{};
    if (active) {
      i = ilu.sweep[kForward ? p : (int64_t)n + p];
      const int pi = ilu.pos[i];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int o = ilu.nbr[k * nc + i];
        if (o < 0) continue;
        const int po = ilu.pos[o];
        if (kForward ? po < pi : po > pi) {
          dep[ndep] = o;
          slot[ndep] = k;
          ++ndep;
        }
      }
      // The row's blocks (and D^-1 backward) do not depend on the waits:
      // bring them towards L1 first.
      const char* rowp = reinterpret_cast<const char*>(ilu.A + (int64_t)i * 80);
#pragma unroll
      for (int b = 0; b < 5; ++b) prefetch_l1(rowp + 128 * b);
      if (!kForward) prefetch_l1(ilu.Dinv + (int64_t)i * 16);
      if (kForward) {
        own = r[i];
        store_empty(z + i);  // the backward sweep's slot
      } else {
        const double2* t = reinterpret_cast<const double2*>(ilu.tmp + i);
        const double2 a = __ldcg(t), b = __ldcg(t + 1);
        own = Vec4<double>{a.x, a.y, b.x, b.y};
        store_empty(ilu.tmp + i);  // empty again for the next forward sweep
      }
    }
    bool done = !active;
    long long spins = 0;
    while (__any_sync(kFull, !done)) {
      if (done) continue;
      // the last word first (cheap while waiting), then all four
      bool ready = true;
      for (int d = 0; d < ndep; ++d)
        if (ld_relaxed_u64(reinterpret_cast<const unsigned long long*>(out + dep[d]) + 3) == kSweepEmpty)
          ready = false;
      unsigned long long w[4][4];
      if (ready) {
        for (int d = 0; d < ndep; ++d) {
          const unsigned long long* q = reinterpret_cast<const unsigned long long*>(out + dep[d]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            w[d][k] = ld_relaxed_u64(q + k);
            if (w[d][k] == kSweepEmpty) ready = false;
          }
        }
      }
      if (ready) {
        const double* row = ilu.A + (int64_t)i * 80;
        Vec4<double> acc = own;
        for (int d = 0; d < ndep; ++d) {
          const double* Bk = row + 16 * (1 + slot[d]);
          const Vec4<double> v{__longlong_as_double((long long)w[d][0]), __longlong_as_double((long long)w[d][1]),
                               __longlong_as_double((long long)w[d][2]), __longlong_as_double((long long)w[d][3])};
          acc.a -= Bk[0] * v.a + Bk[1] * v.b + Bk[2] * v.c + Bk[3] * v.d;
          acc.b -= Bk[4] * v.a + Bk[5] * v.b + Bk[6] * v.c + Bk[7] * v.d;
          acc.c -= Bk[8] * v.a + Bk[9] * v.b + Bk[10] * v.c + Bk[11] * v.d;
          acc.d -= Bk[12] * v.a + Bk[13] * v.b + Bk[14] * v.c + Bk[15] * v.d;
        }
        if (!kForward) {
          const double* D = ilu.Dinv + (int64_t)i * 16;
          Vec4<double> o4;
          o4.a = D[0] * acc.a + D[1] * acc.b + D[2] * acc.c + D[3] * acc.d;
          o4.b = D[4] * acc.a + D[5] * acc.b + D[6] * acc.c + D[7] * acc.d;
          o4.c = D[8] * acc.a + D[9] * acc.b + D[10] * acc.c + D[11] * acc.d;
          o4.d = D[12] * acc.a + D[13] * acc.b + D[14] * acc.c + D[15] * acc.d;
          acc = o4;
        }
        if (!kForward || i != ilu.stall_row) {
          unsigned long long* q = reinterpret_cast<unsigned long long*>(out + i);
          st_relaxed_u64(q, sweep_bits(acc.a));
          st_relaxed_u64(q + 1, sweep_bits(acc.b));
          st_relaxed_u64(q + 2, sweep_bits(acc.c));
          st_relaxed_u64(q + 3, sweep_bits(acc.d));
        }
        done = true;
      } else {
        __nanosleep(32);
        if ((++spins & 63) == 0) {
          if (spins > ilu.spin_limit) {
            atomicExch(&sync->err, 1);
            done = true;
          } else if (*reinterpret_cast<volatile int*>(&sync->err)) {
            done = true;
          }
        }
      }
    }
  }
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    const unsigned int f = atomicAdd(&sync->done, 1u);  // warps that have left
    if (f == nwarps - 1) {
      sync->claim = 0;
      sync->done = 0;
      __threadfence();
    }
  }
}

// One cluster of thread blocks solves a whole triangle, level after level
// (sweep_plan.hpp: the levels, the rows of each block, and where each solved
// value goes).  What bounds a sweep is the latency of a level -- about 500 of
// them for 75k rows, each a dot of a few dozen terms -- so a level's path has
// nothing on it but operand read, dot, and the way of the value to the rows
// that need it:
//   * a solved value is stored straight into the operand slots of the rows
//     that need it, in the shared memory of their blocks, by st.async, whose
//     bytes count on the barrier of the level that waits for them: no fence,
//     no barrier over the cluster per level (only one every kSweepSkew / 2
//     levels, arrived at that long before it is waited for, which bounds how
//     far blocks run apart and so makes slots and barriers reusable);
//   * factor blocks, D^-1 (backward), own values and records of the next
//     kStageRing levels are copied into shared memory by warps of their own,
//     one per slot of the ring (bulk copies, contiguous in sweep order; to
//     start a level's takes a thread 1,000 cycles), and are in a row's
//     registers, with the addresses it stores to, before the level begins:
//     two sets of warps take turns, so that a set has two levels for that.
// Four lanes solve a row (one component each), eight warps the kSweepChunks
// chunks of a block.  The arithmetic of a row (dependencies in slot order)
// is that of k_ilu_sweep: both give the same bits.
// Measured on B200, ms per adjoint iteration (four sweeps) alone: 0.97 at
// 74,528 rows, 1.96 at 300,300, against 3.93 and 13.1 for one block walking
// plain levels behind a block barrier and 5.2 and 11.6 for k_ilu_sweep, 1.09
// and 2.31 with one set of warps and one staging warp per chunk.  About 900
// cycles a level, of them 550 (forward) to 800 (backward) from the barrier to
// the stores; a warp's two levels are filled by 135 cycles of the cluster
// barrier, 250 of waiting, 650 of loading the next row.  Slower, and not kept: a
// cluster barrier with release per level (3.0 ms at 74,528 rows: the release
// waits for the level's global stores, 1,400 cycles), operand slots that are
// polled for a sentinel instead of barriers that are waited on (1.27 ms),
// 16-byte instead of 8-byte stores per lane (1.18 against 1.13 ms), plain
// shared stores and an arrival per warp for values that stay in the block
// (1.01 against 0.96 ms), four copies started by one instruction (1.45
// against 1.17 ms).
constexpr int kSweepWarps = 4 * kSweepChunks;  // of a level
constexpr int kStageRing = 4;  // levels staged at once
constexpr int kSweepThreads = 32 * (2 * kSweepWarps + kStageRing + 2);
constexpr int kSweepWindow = 2048;  // operand slots (32 B each)
static_assert(kSweepWindow == kSweepSlots && (kSweepSlots & (kSweepSlots - 1)) == 0, "operand slots");
constexpr int kStageSlots = 3;      // dependencies whose blocks are staged (the third where a row of the chunk has one)
constexpr int kStageChunkDoubles = kStageSlots * 512;
constexpr int kStageChunksFwd = 2;
constexpr int kStageChunksBwd = 2;
static_assert(kStageChunksFwd == kSweepChunks && kStageChunksBwd == kSweepChunks, "every chunk of a block is staged");
constexpr int kStageBwdD = kStageChunksBwd * kStageChunkDoubles;  // offset of the staged D^-1, doubles
constexpr int kStageDoubles = kStageBwdD + kStageChunksBwd * 512;  // blocks (and D^-1) of one level
constexpr int kStageOwn = kSweepChunks * 128;  // own values of one level, doubles
constexpr int kRecChunkBytes = 32 * kSweepRec * 4;
constexpr int kL2Lead = 16;         // levels between the L2 prefetch of a level's blocks and its use
constexpr int kSweepBlockBytes = kStageRing * kStageDoubles * 8;
constexpr int kSweepOwnBytes = kStageRing * kStageOwn * 8;
constexpr int kSweepRecBytes = kStageRing * kSweepChunks * kRecChunkBytes;
// operand slots, blocks, own values + records + mbarriers + chunk counts + the mark of a wait that ran out
constexpr size_t kSweepSmem = sizeof(Vec4<double>) * kSweepWindow + 4 * kStageDoubles * sizeof(double) + 20692;
static_assert(kSweepSmem == 32 * kSweepWindow + kSweepBlockBytes + kSweepOwnBytes + kSweepRecBytes +
                                8 * (kSweepBars + 2 * kStageRing) + 4 * kStageRing + 4,
              "shared memory of a sweep block");
static_assert(kSweepSmem <= 227 * 1024, "block sweep shared memory above the per-block limit");
static_assert(kStageBwdD + kStageChunksBwd * 512 <= kStageDoubles, "backward staging overflows its buffer");
constexpr int kSweepWaitLimit = 1 << 20;  // polls of an mbarrier (up to 1 us each) before the sweep gives up

// Factor blocks in sweep order, repacked after every factorization: dependency
// d of position p of direction dir at pack[dir] + (p >> 5) * 2048 + d * 512 +
// sweep_pack_place(p & 31, .), D^-1 of backward position p at packD +
// (p >> 5) * 512 + the same.  One thread per two consecutive doubles written.
__global__ void __launch_bounds__(256) k_ilu_pack(IluDev ilu) {
  const int64_t nf = (int64_t)ilu.cl_chunks[0] * 1024, nb = (int64_t)ilu.cl_chunks[1] * 1024,
                nd = (int64_t)ilu.cl_chunks[1] * 256;
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf + nb + nd) return;
  const int kind = t < nf ? 0 : t < nf + nb ? 1 : 2;
  t -= kind == 0 ? 0 : kind == 1 ? nf : nf + nb;
  const int per = kind == 2 ? 256 : 1024;
  const int64_t chunk = t / per;
  const int d = (int)(t % per) >> 8, in = (int)(t & 255);
  const int half = in >> 7, q = (in >> 2) & 31, c = in & 3;
  const int32_t* rec = ilu.cl_rec[kind == 0 ? 0 : 1] + (chunk * 32 + q) * kSweepRec;
  const int row = rec[0];
  if (row < 0) return;
  const double* src;
  double* dst;
  if (kind == 2) {
    src = ilu.Dinv + (int64_t)row * 16;
    dst = ilu.packD + chunk * 512;
  } else {
    if (d >= rec[1]) return;
    const int slot = (int)(((unsigned int)rec[9] >> (8 * d)) & 0xff);
    src = ilu.A + (int64_t)row * 80 + 16 * (1 + slot);
    dst = ilu.pack[kind] + chunk * 2048 + d * 512;
  }
  *reinterpret_cast<double2*>(dst + sweep_pack_place(q, 4 * c + 2 * half)) =
      *reinterpret_cast<const double2*>(src + 4 * c + 2 * half);
}

__device__ __forceinline__ uint32_t sweep_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bulk prefetch of [p, p + bytes) into L2 (a hint: no data is returned and
// no completion is awaited); p 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Whether the phase has completed; sleeps up to a microsecond for it.  Acquire
// at cluster scope: the values it counts come from other blocks (st.async).
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(1000)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase of an mbarrier.  When one has run out (bad), the
// warp waits no more, and the block's other warps give up at their next wait
// that is not over at once (quit).
struct SweepWaits {
  int limit;           // polls
  volatile int* quit;  // in shared memory
  bool bad;
  __device__ __forceinline__ void operator()(uint32_t bar, uint32_t parity) {
    if (bad || bar_try(bar, parity)) return;
    for (int i = 0; i < limit && !*quit; ++i)
      if (bar_try(bar, parity)) return;
    bad = true;
    *quit = 1;
    __threadfence_block();  // before the next cluster barrier
  }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// r (in forward sweep order, ilu.own_f) -> ilu.own_b (kForward), ilu.own_b ->
// z (backward).  Grid: one cluster.  Every wait on an mbarrier is bounded
// (ilu.spin_limit).  A warp whose wait runs out waits on none any more, uses
// nothing it waited for, tells nobody that it has read a staged slot (which is
// then never filled again under a warp that still reads it), sends no values,
// and still takes part in every cluster barrier; warps that need what it held
// back run out too.  At the end it records sync->err, and the sweeps after
// that return at once (their input is void).
template <bool kForward>
__global__ void __launch_bounds__(kSweepThreads, 1) k_ilu_sweep_cluster(IluDev ilu, Vec4<double>* z, const int* gate) {
  if ((int)gated(gate) | ilu.sync[0].err | ilu.sync[1].err) return;  // (loaded side by side)
  constexpr int kDir = kForward ? 0 : 1;
  extern __shared__ __align__(128) unsigned char sweep_sm[];
  double* s_blk = reinterpret_cast<double*>(sweep_sm);
  double* s_own = reinterpret_cast<double*>(sweep_sm + kSweepBlockBytes);
  unsigned char* s_op = sweep_sm + kSweepBlockBytes + kSweepOwnBytes;
  unsigned char* s_rec = s_op + 32 * kSweepWindow;
  const uint32_t bar_op = sweep_smem(s_rec + kSweepRecBytes);  // values of a level
  const uint32_t bar_full = bar_op + 8 * kSweepBars;           // staged copies of a level
  const uint32_t bar_empty = bar_full + 8 * kStageRing;        // its last reader
  int* s_cnt = reinterpret_cast<int*>(s_rec + kSweepRecBytes + 8 * (kSweepBars + 2 * kStageRing));
  int* s_quit = s_cnt + kStageRing;
  const int nlev = ilu.cl_nlev[kDir];
  const int C = (int)gridDim.x, rank = (int)blockIdx.x;
  const int4* __restrict__ info = reinterpret_cast<const int4*>(ilu.cl_info[kDir]) + rank;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kSweepBars; ++i) bar_init(bar_op + 8u * i, 1);
    for (int i = 0; i < kStageRing; ++i) {
      bar_init(bar_full + 8u * i, 1);
      bar_init(bar_empty + 8u * i, kSweepWarps);
    }
    *s_quit = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // all blocks run, their mbarriers are set up
  SweepWaits wait{(int)(ilu.spin_limit < kSweepWaitLimit ? ilu.spin_limit : kSweepWaitLimit), s_quit, false};
  const bool& bad = wait.bad;
  int staged = -1;  // the level that the thread's copies were started for last
  // Before level 4 i a warp arrives for the i-th time, once all have arrived
  // for the (i-1)-th: at level l every level up to l - kSweepSkew has been
  // left.  (Relaxed: what a warp read of those levels it has used by then.)
  auto keep_together = [&](int l) {
    if (l % (kSweepSkew / 2)) return;
    __syncwarp();
    if (l > 0) cluster_wait();
    cluster_arrive();
  };

  // Helper warps: one per staging slot, whose first thread starts the slot's
  // copies (they take it longer than a level), one that sets what each level's
  // barrier waits for, one that requests blocks into L2.
  if (warp >= 2 * kSweepWarps) {
    const int32_t* __restrict__ rec = ilu.cl_rec[kDir];
    const double* __restrict__ pack = ilu.pack[kDir];
    const double* own = reinterpret_cast<const double*>(kForward ? ilu.own_f : ilu.own_b);
    const int slot = warp - 2 * kSweepWarps;
    auto info_of = [&](int l) { return l < nlev ? info[(int64_t)l * C] : make_int4(0, -1, 0, 0); };
    if (slot < kStageRing) {
      const uint32_t bar = bar_full + 8u * slot;
      auto stage = [&](int l, const int4& in) {
        if (in.y < 0) return;
        staged = l;
        s_cnt[slot] = in.y;
        uint32_t bytes = 0;
        for (int j = 0; j < in.y; ++j)
          bytes += 1024 + kRecChunkBytes + (kForward ? 0 : 4096) + (in.z >> j & 1 ? 3 : 2) * 4096;
        bar_expect(bar, bytes);
        const uint32_t dst = sweep_smem(s_blk + slot * kStageDoubles);
        for (int j = 0; j < in.y; ++j) {
          const int64_t k = in.x + (int64_t)j * C;
          bulk_copy(dst + (uint32_t)j * kStageChunkDoubles * 8, pack + k * 2048, (in.z >> j & 1 ? 3 : 2) * 4096, bar);
          if (!kForward) bulk_copy(dst + (uint32_t)(kStageBwdD + j * 512) * 8, ilu.packD + k * 512, 4096, bar);
          bulk_copy(sweep_smem(s_rec) + (uint32_t)(slot * kSweepChunks + j) * kRecChunkBytes,
                    rec + k * 32 * kSweepRec, kRecChunkBytes, bar);
          bulk_copy(sweep_smem(s_own + slot * kStageOwn + j * 128), own + k * 128, 1024, bar);
        }
      };
      int4 next{};
      if (lane == 0) {
        stage(slot, info_of(slot));
        next = info_of(slot + kStageRing);
      }
      for (int l = slot; l - slot < nlev; l += kStageRing) {
        keep_together(l - slot);
        if (lane == 0 && l < nlev) {
          const int4 in = next;
          next = info_of(l + 2 * kStageRing);
          wait(bar_empty + 8u * slot, (l / kStageRing) & 1);
          if (!bad) stage(l + kStageRing, in);
        }
      }
    } else {
      // A level's barrier is set kSweepNear levels ahead: by then every warp
      // has left the level that used it last (kSweepSkew levels back), so a
      // phase that has nothing to wait for cannot pass one that is waited on.
      // (And that level's phase is over then, unless a warp gave up on it: it
      // marked that before it came to the cluster barrier.  A phase must not be
      // set twice.)
      const bool arms = slot == kStageRing;
      const int kLead = arms ? kSweepNear : kL2Lead;
      auto work = [&](int l, const int4& in) {
        if (in.y < 0) return;
        if (arms) {
          if (lane == 0) bar_expect(bar_op + 8u * (l % kSweepBars), (uint32_t)in.w);
        } else if (lane < 2 * kSweepChunks && (lane >> 1) < in.y && !(kForward && (lane & 1))) {
          const int64_t k = in.x + (int64_t)(lane >> 1) * C;
          prefetch_l2_bulk(lane & 1 ? ilu.packD + k * 512 : pack + k * 2048, lane & 1 ? 4096 : 8192);
        }
      };
      // entries of 32 levels, one a lane, and the 32 after them
      int4 now = info_of(lane), then = info_of(32 + lane);
      auto entry = [&](int l) {
        if (l && l % 32 == 0) {
          now = then;
          then = info_of(l + 32 + lane);
        }
        return make_int4(__shfl_sync(0xffffffffu, now.x, l % 32), __shfl_sync(0xffffffffu, now.y, l % 32),
                         __shfl_sync(0xffffffffu, now.z, l % 32), __shfl_sync(0xffffffffu, now.w, l % 32));
      };
      for (int l = 0; l < kLead; ++l) work(l, entry(l));
      for (int l = 0; l < nlev; ++l) {
        keep_together(l);
        const int4 in = entry(l + kLead);
        if (arms) {
          if (l % (kSweepSkew / 2) == 0 && *wait.quit) wait.bad = true;
        } else {
          wait(bar_op + 8u * (l % kSweepBars), (l / kSweepBars) & 1);
          wait.bad = __any_sync(0xffffffffu, bad);
        }
        if (!bad) work(l + kLead, in);
      }
    }
  } else {
    const int set = warp / kSweepWarps, j = (warp >> 2) % kSweepChunks;
    const int q = (warp & 3) * 8 + (lane >> 2), c = lane & 3;
    const uint32_t op_base = sweep_smem(s_op);
    // a row's operands that do not depend on the levels before, in registers,
    // and every address its solve needs
    double2 b[3][2], dv[2];
    double ow = 0.0;
    int4 r0;
    bool row = false;
    uint32_t x0 = 0, x1 = 0, va[4], ba[4];  // operand slots; where the value goes and its barrier (0: nowhere)
    double* to = nullptr;
    auto load_row = [&](int l) {
      const int slot = l % kStageRing;
      wait(bar_full + 8u * slot, (l / kStageRing) & 1);
      const double* s = s_blk + slot * kStageDoubles + (q * 4 + c) * 2;
      const unsigned char* r = s_rec + (slot * kSweepChunks + j) * kRecChunkBytes + q * (kSweepRec * 4);
      const int cnt = s_cnt[slot];
      r0 = *reinterpret_cast<const int4*>(r);
      const int4 tgt = *reinterpret_cast<const int4*>(r + 16);
      const int posb = kForward ? *reinterpret_cast<const int*>(r + 32) : 0;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        b[d][0] = *reinterpret_cast<const double2*>(s + j * kStageChunkDoubles + d * 512);
        b[d][1] = *reinterpret_cast<const double2*>(s + j * kStageChunkDoubles + d * 512 + 256);
      }
      ow = s_own[slot * kStageOwn + j * 128 + q * 4 + c];
      if (!kForward) {
        dv[0] = *reinterpret_cast<const double2*>(s + kStageBwdD + j * 512);
        dv[1] = *reinterpret_cast<const double2*>(s + kStageBwdD + j * 512 + 256);
      }
      row = !bad && j < cnt && r0.x >= 0;  // after a wait that ran out nothing is taken for a record
      x0 = op_base + ((uint32_t)r0.z & (kSweepSlots - 1)) * 32;
      x1 = op_base + ((uint32_t)r0.z >> 16 & (kSweepSlots - 1)) * 32;
      const int tg[4] = {tgt.x, tgt.y, tgt.z, tgt.w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const bool on = row && tg[t] >= 0 && (!kForward || r0.x != ilu.stall_row);
        uint32_t base;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base) : "r"(op_base), "r"(on ? tg[t] >> 16 : rank));
        va[t] = on ? base + (uint32_t)(tg[t] & 0xfff) * 32 + (uint32_t)c * 8 : 0;
        ba[t] = base + (bar_op - op_base) + (uint32_t)(tg[t] >> 12 & 15) * 8;
      }
      if (r0.y > 2) {  // rare on triangles
        b[2][0] = *reinterpret_cast<const double2*>(s + j * kStageChunkDoubles + 1024);
        b[2][1] = *reinterpret_cast<const double2*>(s + j * kStageChunkDoubles + 1024 + 256);
      }
      to = !row       ? nullptr
           : kForward ? reinterpret_cast<double*>(ilu.own_b) + (int64_t)posb * 4 + c
                      : reinterpret_cast<double*>(z) + (int64_t)r0.x * 4 + c;
      __syncwarp();
      if (lane == 0 && !bad) bar_arrive(bar_empty + 8u * slot);
    };
    if (set < nlev) load_row(set);
    for (int pair = 0; pair < nlev; pair += 2) {
      const int l = pair + set;
      keep_together(pair);
      if (l >= nlev) break;  // pair was the last level
      double acc = ow;
      wait(bar_op + 8u * (l % kSweepBars), (l / kSweepBars) & 1);
      const int nd = row ? r0.y : 0;
      // both usual operands at once, whether the row has them or not
      auto operand = [&](uint32_t a, double2& x, double2& y) {
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x.x), "=d"(x.y) : "r"(a) : "memory");
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(y.x), "=d"(y.y) : "r"(a + 16) : "memory");
      };
      double2 x, y, xx, yy;
      operand(x0, x, y);
      operand(x1, xx, yy);
      const double s0 = b[0][0].x * x.x + b[0][0].y * x.y + b[0][1].x * y.x + b[0][1].y * y.y;
      const double s1 = b[1][0].x * xx.x + b[1][0].y * xx.y + b[1][1].x * yy.x + b[1][1].y * yy.y;
      if (nd > 0) acc -= s0;
      if (nd > 1) acc -= s1;
      if (nd > 2) {
        operand(op_base + ((uint32_t)r0.w & (kSweepSlots - 1)) * 32, x, y);
        acc -= b[2][0].x * x.x + b[2][0].y * x.y + b[2][1].x * y.x + b[2][1].y * y.y;
        if (nd > 3) {  // quadrilaterals, at the end of an elimination front
          const int64_t k = info[(int64_t)l * C].x + (int64_t)j * C;
          const double* g = ilu.pack[kDir] + k * 2048 + 1536 + (q * 4 + c) * 2;
          const double2 gx = *reinterpret_cast<const double2*>(g), gy = *reinterpret_cast<const double2*>(g + 256);
          operand(op_base + ((uint32_t)r0.w >> 16 & (kSweepSlots - 1)) * 32, x, y);
          acc -= gx.x * x.x + gx.y * x.y + gy.x * y.x + gy.y * y.y;
        }
      }
      if (!kForward) {
        const int g = lane & ~3;
        __syncwarp();
        const double a0 = __shfl_sync(0xffffffffu, acc, g), a1 = __shfl_sync(0xffffffffu, acc, g + 1),
                     a2 = __shfl_sync(0xffffffffu, acc, g + 2), a3 = __shfl_sync(0xffffffffu, acc, g + 3);
        acc = dv[0].x * a0 + dv[0].y * a1 + dv[1].x * a2 + dv[1].y * a3;
      }
      if (!bad) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (va[t] == 0) break;  // the record's targets come first
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(va[t]),
                       "l"(__double_as_longlong(acc)), "r"(ba[t])
                       : "memory");
        }
      }
      double* const out = bad ? nullptr : to;
      if (l + 2 < nlev) load_row(l + 2);
      if (out) *out = acc;
    }
  }
  __syncwarp();
  cluster_wait();
  cluster_arrive();
  cluster_wait();  // no block leaves while another may still write into it
  // What is on its way into this block's shared memory ends before the block:
  // its own copies, which a warp that gave up did not wait for, and values of
  // other blocks, all sent by now, that no warp waited for (a store to
  // another SM takes microseconds: a millisecond).
  if (staged >= 0) {
    for (int i = 0; i < kSweepWaitLimit; ++i)
      if (bar_try(bar_full + 8u * (staged % kStageRing), (staged / kStageRing) & 1)) break;
  }
  if (bad) {
    atomicExch(&ilu.sync[kDir].err, 1);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
}

// Blocks of one sweep launch: enough warps to cover several dependency
// levels ahead of the front, few enough that waiting warps do not crowd the
// load path, and that the sweeps of other contexts can run beside them.
inline int ilu_sweep_blocks(int n) {
  const int chunks = (n + 31) / 32;
  const int blocks = (chunks + kSweepBlock / 32 - 1) / (kSweepBlock / 32);
  return blocks < 64 ? blocks : 64;
}

}  // namespace o2f
