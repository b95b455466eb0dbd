// The f(A)b engine's persistent kernel.
//
// One cooperative launch runs a contiguous subset of the phases
//   LANCZOS -> TRISOLVE -> COEF -> APPLY -> UPDATE_* -> DEFLATE
// with bounded grid barriers (GridBar) between passes.  The grid is sized so
// that every block is co-resident (cudaLaunchCooperativeKernel checks it).
//
// HBM layout (n rows, R right-hand sides, interleaved so that one gather of
// x[c] fetches all R values of a column with one vector load):
//   A            SELL-32: slice_off[nslices+1] (int64), col/val per slot,
//                slot = slice*32 + lane, slice-column-major (coalesced);
//                optional perm[slot] -> row (sigma-sorted slices)
//   U, Usol, X,
//   update, S    [n][R] FP64
//   V            [m][n][R] BT (FP64, or FP32 in the mixed engine)
//   W0/W1        [n][R] BT   Lanczos work vector (ping-pong between steps)
//   H0/H1        [n][R] HT   Horner / lift ping-pong (FP64 or float-float)
//   P            [d+1][n][R] HT   lifted polynomial terms V c_i
//   aabb         (m+1) x 2R column-major: alpha_r in column r, beta_r in R+r
//   Yr, Yi       m x (R C) column-major (column r*C + j), as the reference
//   coef         [R][d+1][m] FP64, coef_ff the float-float copy
//   hpart, hblk  (Gram-Schmidt only) per-block partial dots [2][m+8][R][G]
//                and each block's totals [G][m+1][R]
#pragma once
#include "dia_slices.cuh"
#include "fab_common.cuh"

namespace gm {

constexpr int kResThreads = 640;   // largest block of the resident entry points

enum Phase : int {
  PH_LANCZOS = 1, PH_TRISOLVE = 2, PH_COEF = 4, PH_APPLY = 8,
  PH_UPDATE_FKPP = 16, PH_UPDATE_FHN = 32, PH_DEFLATE = 64,
  PH_APPLY_SET = 128,  // apply writes X = lift (fused solve) instead of X += lift
  PH_MPK = 256,        // compile-time only: entry points with matrix-powers Horner passes
  PH_REORTH = 512,     // compile-time only: entry points with Gram-Schmidt reorthogonalisation
  PH_RESIDENT = 1024   // compile-time only: entry points whose Lanczos phase keeps the problem on chip
};

struct KParams {
  long long n, nslices;
  int m, d, C, k;
  int phases;
  int G;
  const long long* slice_off;
  const int* col;
  const void* val;
  const int* perm;
  const float* dlo;     // mixed: per-slot-row diagonal compensation (slot order), or null
  const double* gamma;
  const double* gs_re;
  const double* gs_im;
  const double* wts;
  const double* shifts;
  const double* flam;
  const double* Q;
  const double* mass;
  double dt, aode, bode, code, vrest, vamp, vpeak, c1ion;
  double bd_tol;
  double* U;
  double* Usol;
  double* upd;
  double* X;
  double* S;
  double* ode;
  void* V;
  void* W0;
  void* W1;
  void* H0;
  void* H1;
  void* P;
  double* aabb;
  double* Yr;
  double* Yi;
  double* coef;
  float2* coef_ff;
  double* tri;
  double* Z;
  double* part;     // [2R + k R][G]
  unsigned* bar;    // 64-bit barrier arrival counters: [0,1] whole grid, [2+2p, 3+2p] group p
  const int* blk_slice;       // [G+1] slice range owned by each block
  const int* dep_ptr;         // [G+1] neighbour list of each block
  const int* dep_idx;
  unsigned long long* prog;   // [G] pass progress flags
  unsigned long long epoch;   // launch counter
  int dep_mode;               // 1: neighbour waits between SpMV passes, 0: grid barriers
  int nprob;                  // independent problems in this launch (0 or 1: one problem)
  const int* blk_prob;        // [G] problem of each block
  const int* prob_blk0;       // [nprob+1] first block of each problem
  const long long* prob_row0; // [nprob+1] first row of each problem
  int stage_cap;              // >0: stage each slice's column indices in shared memory by TMA
  int pf_vals;                // >0: L2 bulk prefetch of the next slice's values (bytes per value)
  // Diagonal slices: per slice (first entry / 32, entries per row | pattern <<
  // 16; pattern -1: an ordinary slice), the patterns' offsets from the row
  // [pattern][dia_len] by problem (dia_pat0), and per problem 32 * its first
  // slice - its first row
  const int2* dia_meta;
  const int* dia_off;
  const int* dia_pat0;
  const int* dia_shift;
  int dia_len;
  // Two Horner levels per pass (matrix powers): per block, the rows its rows
  // reference outside its own range (halo), the SELL column indices in block-
  // local numbering (own rows first, then the halo), and the offset of the
  // local vector in dynamic shared memory.  Enabled only without a row perm.
  int mpk;
  long long su_off;
  const long long* halo_ptr;  // [G + 1]
  const int* halo_rows;
  const int* lcol;            // per SELL slot
  // Gram-Schmidt reorthogonalisation of each Lanczos vector against the
  // stored basis: 0 = none (the reference's recurrence), 1 = CGS, 2 = CGS2
  int reorth;
  double* hpart;    // [2][m + 8][R][G] per-block partial dots
  double* hblk;     // [G][m + 1][R] each block's totals
  // Resident Lanczos phase (fab_resident.cuh): per SELL slot entry the column
  // in block-local numbering (own slots, then the halo of halo_ptr/halo_rows),
  // per slot whether another block references the row, the tagged words of
  // exchanged rows [2][n][R] and of block partials [2][G][kRedStride], the
  // offset of the state in dynamic shared memory and its capacities (entries, vector
  // elements per right-hand side)
  const unsigned short* res_col;
  const unsigned char* res_exp;
  ulonglong2* res_words;
  ulonglong2* res_red;
  ulonglong2* res_slice;     // mixed: sums of slices for other blocks' groups, [nslices][kRedStride]
  int res_off, res_ent, res_vec;
  int* status;
  int* meff;        // [R]
  unsigned long long timeout_ns;
};

// ------------------------------------------------------------------ helpers
// Thread coordinates, recomputed from the special registers on use rather
// than held in registers across the passes (the kernel is register-bound).
struct Ctx {
  int G;
  __device__ explicit Ctx(int G_) : G(G_) {}
  __device__ __forceinline__ int b() const { return blockIdx.x; }
  __device__ __forceinline__ int tid() const { return threadIdx.x; }
  __device__ __forceinline__ int nt() const { return blockDim.x; }
  __device__ __forceinline__ int lane() const { return threadIdx.x & 31; }
  __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
  __device__ __forceinline__ int nw() const { return blockDim.x >> 5; }
  __device__ __forceinline__ long long gw() const { return (long long)blockIdx.x * nw() + warp(); }
  __device__ __forceinline__ long long tw() const { return (long long)G * nw(); }
  __device__ __forceinline__ long long gt() const { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }
  __device__ __forceinline__ long long tt() const { return (long long)G * blockDim.x; }
};

__device__ __forceinline__ DepSync make_dep(const KParams& kp) {
  return DepSync{kp.prog, kp.dep_ptr, kp.dep_idx, kp.status, kp.epoch << 20, kp.timeout_ns};
}

// Orders consecutive SpMV passes: after pass pc (published), the next
// gathering pass waits for the neighbours' pass pc (or a grid barrier).  One
// PassSync lives for the whole launch and is shared by all phases, so pass
// numbers keep increasing across phases: a phase that restarted at 0 would
// find its waits already satisfied by flags published earlier in the launch.
struct PassSync {
  int mode;
  int p;        // problem (group) whose barrier orders the passes without waits
  unsigned pc;
  __device__ void done(const KParams& kp) {
    ++pc;
    if (mode) make_dep(kp).publish(pc);
  }
  __device__ bool before_next(const KParams& kp);
};

// Arrival counter of problem group p's barrier (words 2 + 2p, 3 + 2p of
// kp.bar), or of the whole grid's (words 0, 1) for p = -1.
__device__ __forceinline__ unsigned long long* bar_word(const KParams& kp, int p) {
  return reinterpret_cast<unsigned long long*>(kp.bar + 2 + 2 * p);
}

// The block's problem group.  A launch can carry several independent
// problems (a batch); each owns a contiguous range of blocks, rows and SELL
// slices, its own barrier and its own reductions.  One problem is the
// single-group case.
struct Grp {
  int p, gb, Gp, bl;
  __device__ Grp(const KParams& kp, const Ctx& c) {
    if (kp.nprob > 0) {
      p = kp.blk_prob[c.b()];
      gb = kp.prob_blk0[p];
      Gp = kp.prob_blk0[p + 1] - gb;
    } else {
      p = 0; gb = 0; Gp = c.G;
    }
    bl = c.b() - gb;
  }
  // rows of this problem and the group-strided row loop (recomputed on use)
  __device__ __forceinline__ long long r0(const KParams& kp) const { return kp.nprob > 0 ? kp.prob_row0[p] : 0; }
  __device__ __forceinline__ long long r1(const KParams& kp) const { return kp.nprob > 0 ? kp.prob_row0[p + 1] : kp.n; }
  __device__ __forceinline__ long long gt(const KParams& kp) const {
    return r0(kp) + (long long)bl * blockDim.x + threadIdx.x;
  }
  __device__ __forceinline__ long long tt() const { return (long long)Gp * blockDim.x; }
  // barrier over this group's blocks (words 2 + 2p, 3 + 2p of kp.bar)
  __device__ GridBar bar(const KParams& kp) const {
    return GridBar{bar_word(kp, p), kp.status, (unsigned)Gp, kp.timeout_ns};
  }
};

__device__ __forceinline__ GridBar group_bar(const KParams& kp, int p) {
  const unsigned Gp = kp.nprob > 0 ? (unsigned)(kp.prob_blk0[p + 1] - kp.prob_blk0[p]) : (unsigned)kp.G;
  return GridBar{bar_word(kp, p), kp.status, Gp, kp.timeout_ns};
}

__device__ __forceinline__ bool PassSync::before_next(const KParams& kp) {
  return mode ? make_dep(kp).wait(pc) : group_bar(kp, p).sync();
}

// Row of SELL slot (slice s, lane); -1 for padding.
__device__ __forceinline__ long long slot_row(const KParams& kp, long long s, int lane) {
  long long slot = s * 32 + lane;
  if (kp.perm) return kp.perm[slot];
  return slot < kp.n ? slot : -1;
}

// acc[r] = sum_j A(row, col_j) x[col_j][r] over the slice row of this lane.
// What the SpMV needs is loads in flight per SM, and resident warps supply
// them more cheaply than several entries per lane, each of which keeps a
// column index, a value and R gathered entries live: every right-hand-side
// count runs its kernels at the residency below with one entry per step.
//   R = 1: three 512-thread blocks per SM (GM_MINB1, 40 registers, no spills);
//          against two blocks, ms a solve: 160^3 mixed 8.72 vs 9.57, disks of
//          degree 8 FP64 500k nodes 9.78 vs 10.67, 1M 17.0 vs 18.5 (160^3 FP64 12.3
//          vs 12.0); a mixed engine's matrix held in L2 is the exception
//          (PolMixedL2).  The matrix-powers and Gram-Schmidt entry points, whose
//          passes hold more state, stay at two blocks (GM_MINB1X): the 250k-node
//          adjoint 288 vs 325 ms per gradient with three.
//   R = 2: two blocks per SM (GM_MINB, 64 registers); against two / three
//          entries, disks of degree 8, us per step: mixed 200k nodes 77 vs 87 /
//          88, 500k 118 vs 137 / 142, 1M 240 vs 326 / 295; FP64 500k 169 vs 184 /
//          185, 1M 322 vs 388 / 398.  Three blocks: 300k mixed 97 vs 84, FP64 128
//          vs 114.
//   R = 4: two blocks per SM (GM_MINB4); against one block with three entries
//          at 128 registers (1M-node FE disk: mixed 40.0 vs 48.7 ms per launch,
//          FP64 58.6 vs 64.9 ms).  The mixed policy's Lanczos entry points run
//          three blocks (GM_MINB4M): 1M-node disk 39.0 vs 40.5 ms, 64-problem
//          batch 19.0 vs 20.3 ms, where FP64 at three blocks is slower (63.1 vs
//          58.8 ms).
// One entry per step over a slice row: column index, value, gather, product.
// The column source (shared-memory stage or global memory) is fixed for the
// whole row, addresses advance by a slot column (32 entries) per step, and the
// mixed engine's diagonal compensation (entry 0 is the diagonal) is peeled
// out of the loop: the kernel is issue-bound, and these are the per-entry
// instructions that are not the product itself.
template <class Pol, int R, class XT, bool kStaged>
__device__ __forceinline__ void row_entries1(const int* __restrict__ cp, const typename Pol::VT* __restrict__ vp,
                                             int len, const XT* __restrict__ x, float dl,
                                             typename Pol::AT (&acc)[R]) {
  if (len <= 0) return;
  XT xv[R];
  int cc = kStaged ? cp[0] : __ldg(cp);
  typename Pol::VT a = ld_val(vp);
  VecIO<R>::ld(x + (long long)cc * R, xv);
  if constexpr (Pol::kMixed) {
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], dl, xv[r]);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], a, xv[r]);
  for (int jj = 1; jj < len; ++jj) {
    cp += 32;
    vp += 32;
    cc = kStaged ? cp[0] : __ldg(cp);
    a = ld_val(vp);
    VecIO<R>::ld(x + (long long)cc * R, xv);
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], a, xv[r]);
  }
}

// Entries of a diagonal slice row: the row's vector entries at fixed offsets,
// so index and gather are not a chain of two loads and neighbouring lanes read
// neighbouring entries.  DiaWidth entries are loaded before their products: six
// with one right-hand side (160^3 mixed 86.4 us per step with three, 84.8 with
// two, 82.1 with six), else one (one / two / three or four: 500^2 FP64 with two
// right-hand sides and degree 3 41.5 / 52.2 / 47.2 us, 400^2 mixed with two 16.7 /
// 17.0 / 17.1, 24 grids mixed with four 54.9 / 55.8 / 56.7).
// Against column indices, per step: 160^3 mixed 96.6 -> 82.1 us, 500^2 mixed
// with four right-hand sides 62 -> 38, 24 grids up to 512^2 67 -> 61, 117^3
// FP64 61.3 -> 57.3 (bound by FP64 issue), 700^2 FP64 28.4 -> 27.3.  The
// entries keep the row's order, with a zero value where a row lacks an offset
// that its slice has.
template <class Pol, int R>
struct DiaWidth {
  static constexpr int value = R == 1 ? 6 : 1;
};
template <class Pol, int R, class XT>
__device__ __forceinline__ void row_dia(const int* of, const typename Pol::VT* __restrict__ vp, int len,
                                        const XT* __restrict__ xr, float dl, typename Pol::AT (&acc)[R]) {
  constexpr int U = DiaWidth<Pol, R>::value;
  if constexpr (Pol::kMixed) {
    // entry 0 is the diagonal (see spmv_slot); dl is zero without compensation
    XT xv[R];
    VecIO<R>::ld(xr + of[0] * R, xv);
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], dl, xv[r]);
  }
  int jj = 0;
  for (; jj + U <= len; jj += U) {
    typename Pol::VT a[U];
    XT xv[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ld_val(vp + (jj + u) * 32);
      VecIO<R>::ld(xr + of[jj + u] * R, xv[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], a[u], xv[u][r]);
  }
  for (; U > 1 && jj < len; ++jj) {
    XT xv[R];
    const typename Pol::VT a = ld_val(vp + jj * 32);
    VecIO<R>::ld(xr + of[jj] * R, xv);
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], a, xv[r]);
  }
}

// The offsets of the patterns of the block's problem and its row shift, in
// shared memory.
__device__ __forceinline__ int* dia_table() {
  __shared__ int s_dia[kDiaTable + 1];
  return s_dia;
}

template <class Pol, int R, class XT>
__device__ __forceinline__ void spmv_slot(const KParams& kp, long long s, int lane, const XT* __restrict__ x,
                                          typename Pol::AT (&acc)[R], const int* scol = nullptr,
                                          const int* colarr = nullptr) {
  using VT = typename Pol::VT;
  const long long base = kp.slice_off[s];
  const int len = (int)((kp.slice_off[s + 1] - base) >> 5);
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = Pol::zero();
  // Mixed engine: diagonal compensation of the FP32-stored values, c_r x_r.
  // The engine stores every row's diagonal entry first (slice column 0); pad
  // lanes carry dl = 0.
  float dl = 0.f;
  if constexpr (Pol::kMixed) {
    if (kp.dlo) dl = __ldg(kp.dlo + s * 32 + lane);
  }
  const VT* vp = reinterpret_cast<const VT*>(kp.val) + base + lane;
  if (scol)
    row_entries1<Pol, R, XT, true>(scol + lane, vp, len, x, dl, acc);
  else
    row_entries1<Pol, R, XT, false>((colarr ? colarr : kp.col) + base + lane, vp, len, x, dl, acc);
}

// A Horner / lift buffer entry as the policy's accumulator.
template <class Pol> __device__ __forceinline__ typename Pol::AT h_load_at(const typename Pol::HT& h) {
  if constexpr (Pol::kMixed) {
    return {h.x, h.y};
  } else {
    return h;
  }
}

// Per-warp double-buffered staging of SELL column indices.  Lane 0 issues a
// TMA bulk copy of the next slice's column block (128 bytes per slice column,
// contiguous in the SELL layout) into shared memory while the warp computes
// the current slice, so a slice costs one global round trip (values and x
// gathers together) instead of two.  Dynamic shared memory holds, per warp,
// two mbarriers and two stages of stage_cap * 32 ints.
// After a timed-out wait, how long a warp still waits for its TMA copy in
// flight before leaving (independent of the configured wait limit, which
// may be short): a copy completes in microseconds unless the GPU is failing.
constexpr unsigned long long kDrainNs = 2000000000ull;

struct ColStage {
  unsigned st;   // bit k: parity of stage k's next completion; bit 2 + k: stage k holds a copy
  int cap;

  // stage k's mbarrier and buffer for this warp, derived from the warp index
  __device__ __forceinline__ static unsigned char* base() {
    extern __shared__ __align__(128) unsigned char dsm[];
    return dsm;
  }
  __device__ __forceinline__ unsigned long long* bar(int k) const {
    return reinterpret_cast<unsigned long long*>(base()) + 2 * (threadIdx.x >> 5) + k;
  }
  __device__ __forceinline__ int* buf(int k) const {
    int* bufs = reinterpret_cast<int*>(base() + 16 * (blockDim.x >> 5));
    return bufs + (long long)(2 * (threadIdx.x >> 5) + k) * cap * 32;
  }

  __device__ void init(const KParams& kp, const Ctx& c) {
    cap = kp.stage_cap;
    st = 0u;
    if (cap <= 0) return;
    if (c.lane() == 0) {
      mbar_init(bar(0), 1);
      mbar_init(bar(1), 1);
      mbar_init_fence();
    }
    __syncwarp();
  }

  // Per warp: the vector whose slice rows the current pass's row epilogue
  // reads and the gathers of x do not bring into cache (set by lane 0 at the
  // start of a pass, read by lane 0 when it issues a slice), or null.  Kept
  // in shared memory rather than a register: the SpMV loop is register-bound.
  __device__ __forceinline__ static const void** row_pf_slot() {
    __shared__ const void* s_row_pf[32];
    return s_row_pf + (threadIdx.x >> 5);
  }

  // stage k <- columns of slice s (lane 0 issues; warp-uniform bookkeeping).
  // With RowB > 0 (bytes per row of the epilogue's vector) and a vector set
  // in row_pf_slot(), that vector's 32 rows of the slice are prefetched into
  // L2 with the values, so the epilogue's load after the slice's SpMV is an
  // L2 hit instead of a full HBM round trip.  Rows of a slice are
  // consecutive only without a row perm.
  template <unsigned RowB = 0>
  __device__ void issue(const KParams& kp, int k, long long s, int lane) {
    if (cap <= 0) return;
    const long long base = kp.slice_off[s];
    const int len = (int)((kp.slice_off[s + 1] - base) >> 5);
    if (len <= 0 || len > cap) return;
    if (lane == 0) {
      unsigned long long* b = bar(k);
      const unsigned bytes = 128u * (unsigned)len;
      mbar_arrive_expect_tx(b, bytes);
      tma_bulk_g2s(buf(k), kp.col + base, bytes, b);
      // the slice's values, which the warp reads right after the columns,
      // start their way from HBM into L2 now
      if (kp.pf_vals) {
        tma_bulk_prefetch_l2(static_cast<const unsigned char*>(kp.val) + base * kp.pf_vals,
                             (unsigned)kp.pf_vals * 32u * (unsigned)len);
        if constexpr (RowB > 0) {
          const void* rp = *row_pf_slot();
          if (rp && !kp.perm) {
            // rows s*32 .. min(s*32 + 32, n) of an n-row buffer: the start is
            // a multiple of 32 rows (aligned), the length rounded down to
            // whole 16-byte units
            const long long r0 = s * 32;
            const long long nr = kp.n - r0 < 32 ? kp.n - r0 : 32;
            const unsigned pb = nr > 0 ? (unsigned)(nr * RowB) & ~15u : 0u;
            if (pb > 0) tma_bulk_prefetch_l2(static_cast<const unsigned char*>(rp) + r0 * RowB, pb);
          }
        }
      }
    }
    st |= 4u << k;
  }

  // Waits for stage k; returns its buffer, or nullptr when the slice is read
  // from global memory (not staged) or the wait ran out (status recorded).
  __device__ const int* ready(const KParams& kp, int k, int lane) {
    if (!(st & (4u << k))) return nullptr;
    unsigned long long* b = bar(k);
    const unsigned par = (st >> k) & 1u;
    unsigned long long start = 0;
    bool timed_out = false;
    while (!mbar_try_wait(b, par)) {
      const unsigned long long now = global_timer_ns();
      if (start == 0) {
        start = now;
      } else if (!timed_out && now - start > kp.timeout_ns) {
        if (lane == 0) atomicCAS(kp.status, 0, (int)ST_TIMEOUT);
        timed_out = true;
        start = now;  // keep waiting a bounded time for the copy in flight
      } else if (timed_out && now - start > kDrainNs) {
        break;
      }
    }
    st ^= 1u << k;
    st &= ~(4u << k);
    return timed_out ? nullptr : buf(k);
  }

  // all lanes are done reading stage k before a later copy overwrites it
  __device__ void release() {
    if (cap <= 0) return;
    fence_proxy_async_smem();
    __syncwarp();
  }
};

// One SpMV pass over the block's slices: z = A x for the slice rows, then
// epi(row, z) for the row epilogue (row -1: padding).  rowpf: the [n][R] storage-precision
// vector the epilogue reads at the slice rows and that the gathers of x do
// not bring into cache (prefetched one slice ahead with the values when the
// matrix streams from HBM), or null.
template <class Pol, int R, class XT, class Epi>
__device__ __forceinline__ bool spmv_pass(const KParams& kp, const Ctx& c, ColStage& cs, const XT* x, Epi&& epi,
                                          PassSync* wait = nullptr, const typename Pol::BT* rowpf = nullptr) {
  using AT = typename Pol::AT;
  // (one and two right-hand sides: with four, the 1M-node FE disk's mixed
  // launch measured 2.5% slower with the row prefetch, 3D 256^3 mixed with one
  // right-hand side 2% faster)
  constexpr unsigned kRowB = R <= 2 ? (unsigned)(R * sizeof(typename Pol::BT)) : 0u;
  const long long sb = kp.blk_slice[c.b()], se = kp.blk_slice[c.b() + 1];
  long long s = sb + c.warp();
  if constexpr (Pol::kDia) {
    // no stages: the slice's place and pattern one slice ahead, and with a
    // matrix streamed from HBM the bulk prefetch of its values and of the
    // epilogue's rows
    using VT = typename Pol::VT;
    const int* const tab = dia_table();
    int2 mt = s < se ? __ldg(kp.dia_meta + s) : make_int2(0, 0);
    if (wait && !wait->before_next(kp)) return false;
    for (; s < se; s += c.nw()) {
      const long long sn = s + c.nw();
      const int2 mn = sn < se ? __ldg(kp.dia_meta + sn) : make_int2(0, 0);
      if (kp.pf_vals && sn < se && c.lane() == 0) {
        tma_bulk_prefetch_l2(static_cast<const unsigned char*>(kp.val) + (long long)mn.x * 32 * kp.pf_vals,
                             (unsigned)kp.pf_vals * 32u * (unsigned)(mn.y & 0xffff));
        if (kRowB > 0 && rowpf && tab[kDiaTable] == 0 && (mn.y >> 16) >= 0)
          tma_bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(rowpf) + sn * 32 * kRowB, 32u * kRowB);
      }
      const int len = mt.y & 0xffff, pat = mt.y >> 16;
      const VT* vp = reinterpret_cast<const VT*>(kp.val) + (long long)mt.x * 32 + c.lane();
      float dl = 0.f;
      if constexpr (Pol::kMixed) {
        if (kp.dlo) dl = __ldg(kp.dlo + s * 32 + c.lane());
      }
      AT z[R];
#pragma unroll
      for (int r = 0; r < R; ++r) z[r] = Pol::zero();
      long long row;
      if (pat >= 0) {
        row = s * 32 + c.lane() - tab[kDiaTable];
        row_dia<Pol, R, XT>(tab + pat * kp.dia_len, vp, len, x + row * R, dl, z);
      } else {
        row = slot_row(kp, s, c.lane());
        row_entries1<Pol, R, XT, false>(kp.col + (long long)mt.x * 32 + c.lane(), vp, len, x, dl, z);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) z[r] = Pol::norm(z[r]);
      epi(row, z);
      mt = mn;
    }
    return true;
  }
  if (kRowB > 0 && c.lane() == 0) *ColStage::row_pf_slot() = rowpf;
  if (s < se) cs.issue<kRowB>(kp, 0, s, c.lane());
  // the ordering wait on the previous pass comes after the first column copy
  // is issued: the matrix does not depend on it, so the copy overlaps the wait
  if (wait && !wait->before_next(kp)) {
    if (s < se) cs.ready(kp, 0, c.lane());   // bounded drain of the copy in flight
    return false;
  }
  int k = 0;
  for (; s < se; s += c.nw(), k ^= 1) {
    const long long sn = s + c.nw();
    if (sn < se) cs.issue<kRowB>(kp, k ^ 1, sn, c.lane());
    const int* scol = cs.ready(kp, k, c.lane());
    AT z[R];
    spmv_slot<Pol, R, XT>(kp, s, c.lane(), x, z, scol);
#pragma unroll
    for (int r = 0; r < R; ++r) z[r] = Pol::norm(z[r]);
    epi(slot_row(kp, s, c.lane()), z);
    cs.release();
  }
  return true;
}

// The same products by (row, right-hand side): lane l of a warp takes row
// l / R of the unit's 32 / R rows and right-hand side l % R, so a slice is R
// units of work.  For the FP64 engine's Horner passes, which sum nothing over
// the block: a lane holds one accumulator instead of R, which leaves registers
// for four gathers in flight (by rows one at a time), and a
// block of few slices waits less for the warps that have one slice more.  The
// FP64 pipe does the same number of warp instructions either way.
// Disks of degree 8, us per step by rows / split: R = 2 200k nodes 95.1 / 93.1,
// 300k 113.9 / 116.4, 500k 180.7 / 171.1; R = 4 100k 123.1 / 111.7, 300k 216.3 /
// 194.1, 500k 343.9 / 311.2, 700k 464 / 434.  With more slices per warp the
// staged columns and prefetched values of the other pass win (1M, 6.4 slices,
// R = 4: 655 / 680), hence kSplitSlices.  The mixed
// engine is bound by FP32 issue and loses by the extra index loads (300k, R =
// 4: 136 / 168); the apply's passes gain nothing (300k 539 / 540).
// epi(e, r, z): element e = row R + r.
template <int N> struct IntC { static constexpr int value = N; };
constexpr int kSplitSlices = 5;   // slices per warp up to which it is taken
template <class Pol, int R>
__device__ __forceinline__ bool split_rows(const KParams& kp, const Ctx& c) {
  if constexpr (R == 1 || Pol::kDia || Pol::kMixed) return false;
  return kp.blk_slice[c.b() + 1] - kp.blk_slice[c.b()] <= kSplitSlices * c.nw();
}
template <class Pol, int R, class XT, class Epi>
__device__ __forceinline__ bool spmv_pass_split(const KParams& kp, const Ctx& c, const XT* __restrict__ x, Epi&& epi,
                                                PassSync* wait = nullptr) {
  using AT = typename Pol::AT;
  using VT = typename Pol::VT;
  const int sb = kp.blk_slice[c.b()], nu = (kp.blk_slice[c.b() + 1] - sb) * R;
  if (wait && !wait->before_next(kp)) return false;
  for (int u = c.warp(); u < nu; u += c.nw()) {
    const long long s = sb + u / R;
    const int sl = (u % R) * (32 / R) + c.lane() / R, r = c.lane() % R;
    const long long base = kp.slice_off[s];
    const int len = (int)((kp.slice_off[s + 1] - base) >> 5);
    const int* cp = kp.col + base + sl;
    const VT* vp = reinterpret_cast<const VT*>(kp.val) + base + sl;
    AT z = Pol::zero();
    int jj = 0;
    auto chunk = [&](auto width) {
      constexpr int U = decltype(width)::value;
      VT a[U];
      XT xv[U][1];
      int cc[U];
#pragma unroll
      for (int v = 0; v < U; ++v) { cc[v] = __ldg(cp + (jj + v) * 32); a[v] = ld_val(vp + (jj + v) * 32); }
#pragma unroll
      for (int v = 0; v < U; ++v) VecIO<1>::ld(x + (long long)cc[v] * R + r, xv[v]);
#pragma unroll
      for (int v = 0; v < U; ++v) z = Pol::acc(z, a[v], xv[v][0]);
      jj += U;
    };
    while (jj + 4 <= len) chunk(IntC<4>{});
    if (jj + 2 <= len) chunk(IntC<2>{});
    if (jj < len) chunk(IntC<1>{});
    const long long row = slot_row(kp, s, sl);
    if (row >= 0) epi(row * R + r, r, Pol::norm(z));
  }
  return true;
}

// One row of A x read through the SELL layout without a row perm (row r is
// lane r % 32 of slice r / 32): the halo rows of a matrix-powers pass.
template <class Pol, int R, class XT>
__device__ __forceinline__ void row_spmv(const KParams& kp, long long r, const XT* __restrict__ x,
                                         typename Pol::AT (&acc)[R]) {
  using VT = typename Pol::VT;
  const long long s = r >> 5;
  const int l = (int)(r & 31);
  const long long base = kp.slice_off[s];
  const int len = (int)((kp.slice_off[s + 1] - base) >> 5);
  const VT* vp = reinterpret_cast<const VT*>(kp.val) + base + l;
  const int* cp = kp.col + base + l;
#pragma unroll
  for (int q = 0; q < R; ++q) acc[q] = Pol::zero();
  float dl = 0.f;
  if constexpr (Pol::kMixed) {
    if (kp.dlo) dl = __ldg(kp.dlo + s * 32 + l);
  }
  for (int jj = 0; jj < len; ++jj) {
    const int cc = __ldg(cp + (long long)jj * 32);
    const VT a = __ldg(vp + (long long)jj * 32);
    XT xv[R];
    VecIO<R>::ld(x + (long long)cc * R, xv);
    if constexpr (Pol::kMixed) {
      if (jj == 0) {
#pragma unroll
        for (int q = 0; q < R; ++q) acc[q] = Pol::acc(acc[q], dl, xv[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) acc[q] = Pol::acc(acc[q], a, xv[q]);
  }
#pragma unroll
  for (int q = 0; q < R; ++q) acc[q] = Pol::norm(acc[q]);
}

// Two Horner levels in one pass (matrix powers):
//   level 1  u1 = A hin + g1 w   on the block's rows and its halo rows,
//            kept in shared memory in block-local numbering;
//   level 2  hout = A u1 + g2 w  on the block's rows, A read with local
//            column indices against the shared-memory vector.
// The ordering wait before it covers two hops of the row graph (the halo
// rows' neighbours), as every wait does when these passes are enabled.
template <class Pol, int R>
__device__ __forceinline__ bool horner_pair(const KParams& kp, const Ctx& c, ColStage& cs, PassSync& ps,
                            const typename Pol::HT* hin, typename Pol::HT* hout, const typename Pol::BT* w,
                            const typename Pol::ST (&g1)[R], const typename Pol::ST (&g2)[R]) {
  using BT = typename Pol::BT;
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  extern __shared__ __align__(128) unsigned char dsm[];
  HT* const su = reinterpret_cast<HT*>(dsm + kp.su_off);
  const long long sb = kp.blk_slice[c.b()], se = kp.blk_slice[c.b() + 1];
  const long long rb0 = sb * 32;
  const long long nown = (se * 32 < kp.n ? se * 32 : kp.n) - rb0;
  // level 1, own rows (the usual pass, results to shared memory)
  const bool ok = spmv_pass<Pol, R, HT>(kp, c, cs, hin, [&](long long row, AT (&z)[R]) {
    if (row < 0) return;
    BT sv[R];
    VecIO<R>::ld(w + row * R, sv);
    HT u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(z[r], g1[r], sv[r]));
    VecIO<R>::st(su + (row - rb0) * R, u);
  }, &ps);
  if (!ok) return false;
  // level 1, halo rows
  const long long h0 = kp.halo_ptr[c.b()], h1 = kp.halo_ptr[c.b() + 1];
  for (long long k = h0 + c.tid(); k < h1; k += c.nt()) {
    const long long r = kp.halo_rows[k];
    AT z[R];
    row_spmv<Pol, R, HT>(kp, r, hin, z);
    BT sv[R];
    VecIO<R>::ld(w + r * R, sv);
    HT u[R];
#pragma unroll
    for (int q = 0; q < R; ++q) u[q] = Pol::to_h(Pol::add_mul(z[q], g1[q], sv[q]));
    VecIO<R>::st(su + (nown + (k - h0)) * R, u);
  }
  __syncthreads();
  // level 2, own rows from the shared-memory vector: its gathers have
  // shared-memory latency, so one entry at a time (few live registers)
  using VT = typename Pol::VT;
  for (long long s = sb + c.warp(); s < se; s += c.nw()) {
    const long long base = kp.slice_off[s];
    const int len = (int)((kp.slice_off[s + 1] - base) >> 5);
    const int* lp = kp.lcol + base + c.lane();
    const VT* vp = reinterpret_cast<const VT*>(kp.val) + base + c.lane();
    AT z[R];
#pragma unroll
    for (int r = 0; r < R; ++r) z[r] = Pol::zero();
    float dl = 0.f;
    if constexpr (Pol::kMixed) {
      if (kp.dlo) dl = __ldg(kp.dlo + s * 32 + c.lane());
    }
    for (int jj = 0; jj < len; ++jj) {
      const int lc = __ldg(lp + (long long)jj * 32);
      const VT a = __ldg(vp + (long long)jj * 32);
      HT xv[R];
      VecIO<R>::ld(su + (long long)lc * R, xv);
      if constexpr (Pol::kMixed) {
        if (jj == 0) {
#pragma unroll
          for (int r = 0; r < R; ++r) z[r] = Pol::acc(z[r], dl, xv[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) z[r] = Pol::acc(z[r], a, xv[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) z[r] = Pol::norm(z[r]);
    const long long row = s * 32 + c.lane();
    if (row >= kp.n) continue;
    BT sv[R];
    VecIO<R>::ld(w + row * R, sv);
    HT u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(z[r], g2[r], sv[r]));
    VecIO<R>::st(hout + row * R, u);
  }
  return true;
}

// ------------------------------------------------------------------ LANCZOS
// build_subspace.cu:5-89 with the three-term recurrence as two grid passes
// per step (A: SpMV + beta_j v_{j-1} + alpha partials; B: w -= alpha v_j +
// beta partials), plus d Horner passes for the polynomial preconditioner.
// v_{j+1} = w (1/beta_{j+1}) is formed on the fly in the next step's first
// pass, which also stores it in V.
// Block-uniform Lanczos scalars live in shared memory, not registers: with R
// right-hand sides they would otherwise occupy ~10R registers across every
// SpMV pass and push the passes into local-memory spills.
#ifndef GM_MAX_DEG
#define GM_MAX_DEG 32
#endif
template <class Pol, int R>
struct LanczosScalars {
  double beta[R], rbeta[R], rbp[R], alpha[R], bound[R];
  int broken[R];
  typename Pol::ST sc[R], rb[R], bj[R], al[R];
  typename Pol::ST gr[GM_MAX_DEG + 1][R];   // gamma_h rbeta_j of the current step
  double gam[GM_MAX_DEG + 1];
};

// Where a problem's alpha, beta and m_eff go; lead: the one thread that writes.
struct LanczosOut {
  double* aab;
  int* meff;
  bool lead;
};

// The scalars of right-hand side r, each function by one full warp: different
// lanes form the products and conversions at once, since an FP64 instruction
// takes 64 cycles of issue for one lane as for 32.
//
// alpha_j = w^T v_j = rbeta_j (w^T w_j); pass B subtracts alpha_j rbeta_j w_j.
template <class Pol, int R>
__device__ __forceinline__ void step_alpha(LanczosScalars<Pol, R>& sh, int r, double tot) {
  const double al = tot * sh.rbeta[r];
  const typename Pol::ST q = Pol::scalar(al * sh.rbeta[r]);
  if ((threadIdx.x & 31) == 0) {
    sh.alpha[r] = al;
    sh.al[r] = q;
  }
}
// Off the critical path, after step_alpha: alpha's store and the bound of the
// breakdown test, bd_tol (|alpha_j| + beta_j).
template <class Pol, int R>
__device__ __forceinline__ void step_bound(LanczosScalars<Pol, R>& sh, const KParams& kp, const LanczosOut& out, int r,
                                           int j) {
  const double al = sh.alpha[r];
  if (out.lead) out.aab[j + (long long)(kp.m + 1) * r] = sh.broken[r] ? 0.0 : al;
  if ((threadIdx.x & 31) == 0) {
    sh.bound[r] = kp.bd_tol * (fabs(al) + (j > 0 ? sh.beta[r] : 0.0));
    if (out.lead && !(al == al)) atomicCAS(kp.status, 0, (int)ST_NONFINITE);
  }
  __syncwarp();
}
// From tot = beta^2: the end of step j, or beta_0 = ||U_r|| for j < 0.
template <class Pol, int R>
__device__ __forceinline__ void step_beta(LanczosScalars<Pol, R>& sh, const KParams& kp, const LanczosOut& out, int r,
                                          double tot, int j) {
  const int lane = threadIdx.x & 31, m = kp.m, d = kp.d;
  const int hi = __double2hiint(tot);
  const bool normal = hi >= 0x00100000 && hi < 0x7ff00000;
  double rb, bn;
  if (normal && !Pol::kMixed) {
    // sqrt(tot) and its reciprocal by Newton's iteration from the FP32
    // instruction, y = 1/sqrt(t) with an error of about 2^-22 (t: tot scaled by an
    // even power of two into [1, 4)): twice b + (t - b^2) y / 2, then y (1 + h + h^2)
    // with h = 1 - b y; eight FP64 instructions.  (The mixed engine keeps the
    // bits of the square root and the division.)  The reciprocal is that of the
    // rounded b, as a division gives it: with rsqrt(tot) itself, beta_j v_j missed
    // w_j by 0.49 of 2^-53 root mean square instead of 0.40, and solutions that
    // Lanczos rounding decides lost as much (45^3, m = 60, 250 right-hand sides:
    // 1.0e-12 against 8.2e-13); rsqrt and the corrections after it took 64 x 64
    // 434 us, this 432.
    const int ex = (((hi >> 20) - 1023) & ~1) * 0x100000;
    const int lo = __double2loint(tot);
    const double t = __hiloint2double(hi - ex, lo);
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(yf) : "f"(__int_as_float(((hi - ex - 0x38000000) << 3) | (int)((unsigned)lo >> 29))));
    const int yb = __float_as_int(yf), yh = (yb >> 3) + 0x38000000;
    const double y = __hiloint2double(yh, yb << 29), half_y = __hiloint2double(yh - 0x100000, yb << 29);
    double b = t * y;
    b = fma(fma(-b, b, t), half_y, b);
    b = fma(fma(-b, b, t), half_y, b);
    const double h = fma(-b, y, 1.0);
    const double r = fma(y, fma(h, h, h), y);
    bn = __hiloint2double(__double2hiint(b) + ex / 2, __double2loint(b));
    rb = __hiloint2double(__double2hiint(r) - ex / 2, __double2loint(r));
  } else {
    bn = sqrt(tot);
    rb = 1.0 / bn;
  }
  const int was = j < 0 ? 0 : sh.broken[r];
  int broken = was;
  if (j < 0) {
    broken = !normal && !(bn > 0.0);
  } else if (!broken && j + 1 < m) {
    // positive numbers compare like their bits
    const bool down = normal ? __double_as_longlong(bn) <= __double_as_longlong(sh.bound[r]) : !(bn > sh.bound[r]);
    if (down) {
      broken = 1;
      if (out.lead) out.meff[r] = j + 1;
    }
  }
  const double rb_old = j < 0 ? 0.0 : sh.rbeta[r];
  if (out.lead) {
    out.aab[(j + 1) + (long long)(m + 1) * (R + r)] = was ? 0.0 : bn;
    if (j < 0) out.meff[r] = broken ? 0 : m;
    if (!normal && (!(bn == bn) || isinf(bn))) atomicCAS(kp.status, 0, (int)ST_NONFINITE);
  }
  const double be = broken && j >= 0 ? 0.0 : bn;
  if (broken) rb = 0.0;
  __syncwarp();   // every lane has read the old values
  if (lane == 0) {
    sh.broken[r] = broken;
    sh.rbp[r] = rb_old;
    sh.beta[r] = be;
    sh.rbeta[r] = rb;
  }
  // lane 0: rbeta, lane 1: beta_j rbeta_{j-1}, lane 2 + h: gamma_h rbeta
  const double f = lane == 0 ? 1.0 : lane == 1 ? rb_old : lane - 2 <= d ? sh.gam[lane - 2] : 0.0;
  const typename Pol::ST q = Pol::scalar((lane == 1 ? be : rb) * f);
  if (lane == 0) sh.rb[r] = q;
  if (lane == 1) sh.bj[r] = q;
  if (lane == 2) sh.sc[r] = q;
  if (lane > 2 && lane - 2 <= d) sh.gr[lane - 2][r] = q;
  for (int h = 30 + lane; h <= d; h += 32) sh.gr[h][r] = Pol::scalar(sh.gam[h] * rb);
}

// Sum of p[r] over the problem's blocks, then fin(r, total) with one full warp
// per right-hand side; also the problem's grid barrier.  The tree is fixed:
// the 32 lanes of a warp, the warps of a block, then each lane's blocks in
// order and the lanes.  With one or two right-hand sides the lanes' trees run
// from shared memory, eight lanes to a warp's sum (six FP64 additions in a
// quarter of the warps instead of five in all of them: with 48 warps per SM
// 2.2 us of issue), and so do the totals, whose loads are then one round trip.
// Ends with a block barrier; false when a wait failed.
template <int R>
struct ReduceBuf {
  static constexpr bool kStage = R <= 2;
  static constexpr int kCap = 512;
  double v[kStage ? R : 1][kStage ? kCap : 1];
  double w[32][R];
  int ok;
};
template <int R, class Fin>
__device__ __forceinline__ bool reduce_blocks(ReduceBuf<R>& buf, const KParams& kp, const Ctx& c, const Grp& g,
                                              double (&p)[R], double* part, Fin&& fin) {
  constexpr bool kStage = ReduceBuf<R>::kStage;
  constexpr int kCap = ReduceBuf<R>::kCap;
  auto& s_v = buf.v;
  auto& s_w = buf.w;
  const int lane = c.lane(), warp = c.warp(), nw = c.nw(), G = kp.G;
  if constexpr (kStage) {
#pragma unroll
    for (int r = 0; r < R; ++r) s_v[r][c.tid()] = p[r];
    __syncthreads();
    for (int item = c.tid() >> 3; item < ((R * nw + 3) & ~3); item += c.nt() >> 3) {
      const int it = item < R * nw ? item : R * nw - 1;   // whole warps for the shuffles
      const int r = it / nw, w = it - r * nw, i = lane & 7;
      const double* v = s_v[r] + w * 32 + i;
      double t = (v[0] + v[16]) + (v[8] + v[24]);
      t += __shfl_xor_sync(0xffffffffu, t, 4);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      if (i == 0) s_w[w][r] = t;
    }
  } else {
    const double s = warp_sum_packed<R>(p);
    if ((lane & (32 / R - 1)) == 0) s_w[warp][packed_index<R>(lane)] = s;
  }
  __syncthreads();
  if (warp == 0) {
    double t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = lane < nw ? s_w[lane][r] : 0.0;
    const double q = warp_sum_packed<R>(t);
    if ((lane & (32 / R - 1)) == 0) part[(long long)packed_index<R>(lane) * G + c.b()] = q;
    __syncwarp();
    if (lane == 0) buf.ok = g.bar(kp).arrive_and_wait();
  }
  __syncthreads();
  if (!buf.ok) return false;
  const double* pg = part + g.gb;
  const bool staged = kStage && g.Gp <= kCap;
  if constexpr (kStage) {
    if (staged) {
      for (int b = c.tid(); b < g.Gp; b += c.nt())
#pragma unroll
        for (int r = 0; r < R; ++r) s_v[r][b] = pg[(long long)r * G + b];
      __syncthreads();
    }
  }
  for (int r = warp; r < R; r += nw) {
    double t = 0.0;
    const double* v = pg + (long long)r * G;
    if constexpr (kStage) {
      if (staged) v = s_v[r];
    }
    for (int b = lane; b < g.Gp; b += 32) t += v[b];
    fin(r, warp_sum(t));
  }
  __syncthreads();
  return true;
}

// The per-block Gram-Schmidt coefficient x as the policy's scalar: FP64, or
// the float-float pair stored in the same 8 bytes.
template <class Pol>
__device__ __forceinline__ typename Pol::ST reorth_scalar(const double* hb, int x) {
  if constexpr (Pol::kMixed) {
    const float2 f = reinterpret_cast<const float2*>(hb)[x];
    return ff{f.x, f.y};
  } else {
    return hb[x];
  }
}

// Classical Gram-Schmidt of the step's work vector w (unrounded, in Hw)
// against the stored basis V_0..V_j, kp.reorth times (1 = CGS, 2 = CGS2):
//   h_t = V_t^T w  (t = 0..j; per-block partials, then every block totals the
//                  group's partials in one fixed order: deterministic)
//   w  <- w - sum_t h_t V_t
// The dots run over tiles of TT basis vectors so that each V_t is read once
// per dot pass with TT*R accumulators per thread.  Between passes w stays in
// the accumulator precision in Hw; the last correction rounds it to storage
// once (Wout) and accumulates ||w||^2 into bpa.  Consecutive passes use
// alternate halves of hpart, so a block that runs ahead cannot overwrite
// partials another block is still summing.
template <class Pol, int R>
__device__ bool reorth_step(const KParams& kp, const Ctx& c, const Grp& g, int j, typename Pol::HT* Hw,
                            typename Pol::BT* Wout, typename Pol::AT (&bpa)[R]) {
  using BT = typename Pol::BT;
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  constexpr int TT = 8 / R;
  const long long n = kp.n;
  const BT* const V = reinterpret_cast<const BT*>(kp.V);
  const int G = kp.G;
  double* const hb = kp.hblk + (long long)c.b() * (kp.m + 1) * R;   // this block's totals [t][r]
  for (int q = 0; q < kp.reorth; ++q) {
    double* const hp = kp.hpart + (long long)(q & 1) * (kp.m + TT) * R * G;   // [t][r][G]
    for (int t0 = 0; t0 <= j; t0 += TT) {
      AT acc[TT][R];
#pragma unroll
      for (int u = 0; u < TT; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[u][r] = Pol::zero();
      if (t0 + TT <= j + 1) {
        // a whole tile: its loads before its products (with a guard per vector
        // the compiler ordered them either way, 117^3 275 or 337 us per step
        // from one build to the next)
        for (long long i = g.gt(kp); i < g.r1(kp); i += g.tt()) {
          HT wh[R];
          VecIO<R>::ld(Hw + i * R, wh);
          BT v[TT][R];
#pragma unroll
          for (int u = 0; u < TT; ++u) VecIO<R>::ld(V + ((long long)(t0 + u) * n + i) * R, v[u]);
#pragma unroll
          for (int u = 0; u < TT; ++u)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[u][r] = Pol::dot(acc[u][r], h_load_at<Pol>(wh[r]), v[u][r]);
        }
      } else {
        for (long long i = g.gt(kp); i < g.r1(kp); i += g.tt()) {
          HT wh[R];
          VecIO<R>::ld(Hw + i * R, wh);
#pragma unroll
          for (int u = 0; u < TT; ++u) {
            if (t0 + u <= j) {
              BT v[R];
              VecIO<R>::ld(V + ((long long)(t0 + u) * n + i) * R, v);
#pragma unroll
              for (int r = 0; r < R; ++r) acc[u][r] = Pol::dot(acc[u][r], h_load_at<Pol>(wh[r]), v[r]);
            }
          }
        }
      }
      double a[TT * R];
#pragma unroll
      for (int u = 0; u < TT; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) a[u * R + r] = Pol::to_d(acc[u][r]);
      block_sum_store<TT * R>(a, hp + (long long)t0 * R * G + c.b(), G);
    }
    if (!group_bar(kp, g.p).sync()) return false;
    for (int x = c.warp(); x < (j + 1) * R; x += c.nw()) {
      const double* pp = hp + (long long)x * G + g.gb;
      double t = 0.0;
      for (int b = c.lane(); b < g.Gp; b += 32) t += pp[b];
      t = warp_sum(t);
      if (c.lane() == 0) {
        // the correction's scalar, once per block: float-float for the
        // mixed engine (no double conversions per element)
        if constexpr (Pol::kMixed) {
          const ff hv = ff_from_double(t);
          reinterpret_cast<float2*>(hb)[x] = make_float2(hv.hi, hv.lo);
        } else {
          hb[x] = t;
        }
      }
    }
    __syncthreads();
    const bool last = q + 1 == kp.reorth;
    for (long long i = g.gt(kp); i < g.r1(kp); i += g.tt()) {
      HT wh[R];
      VecIO<R>::ld(Hw + i * R, wh);
      AT w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) w[r] = h_load_at<Pol>(wh[r]);
      // TT basis entries loaded before they are used: TT loads in flight per row
      int t = 0;
      for (; t + TT <= j + 1; t += TT) {
        BT v[TT][R];
#pragma unroll
        for (int u = 0; u < TT; ++u) VecIO<R>::ld(V + ((long long)(t + u) * n + i) * R, v[u]);
#pragma unroll
        for (int u = 0; u < TT; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r) w[r] = Pol::sub_mul(w[r], reorth_scalar<Pol>(hb, (t + u) * R + r), v[u][r]);
      }
      for (; t <= j; ++t) {
        BT v[R];
        VecIO<R>::ld(V + ((long long)t * n + i) * R, v);
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = Pol::sub_mul(w[r], reorth_scalar<Pol>(hb, t * R + r), v[r]);
      }
      if (last) {
        BT wb[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          wb[r] = Pol::to_b(w[r]);
          bpa[r] = Pol::dot_self(bpa[r], w[r]);
        }
        VecIO<R>::st(Wout + i * R, wb);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) wh[r] = Pol::to_h(w[r]);
        VecIO<R>::st(Hw + i * R, wh);
      }
    }
    __syncthreads();
  }
  return true;
}

template <class Pol, int R, bool MPK, bool RO>
__device__ bool phase_lanczos(const KParams& kp, const Ctx& c, const Grp& g, PassSync& ps, ColStage& cs) {
  using BT = typename Pol::BT;
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  const long long n = kp.n;
  const int m = kp.m, d = kp.d, G = kp.G;
  const LanczosOut out{kp.aabb + (long long)(m + 1) * 2 * R * g.p, kp.meff + (long long)R * g.p,
                       g.bl == 0 && c.lane() == 0};   // this problem's
  const double* const gam = kp.gamma + (long long)(d + 1) * g.p;
  BT* V = reinterpret_cast<BT*>(kp.V);
  BT* const W0 = reinterpret_cast<BT*>(kp.W0);
  BT* const W1 = reinterpret_cast<BT*>(kp.W1);
  HT* const H0 = reinterpret_cast<HT*>(kp.H0);
  HT* const H1 = reinterpret_cast<HT*>(kp.H1);
  double* part_a = kp.part;
  double* part_b = kp.part + (long long)R * G;
  __shared__ LanczosScalars<Pol, R> sh;
  __shared__ ReduceBuf<R> buf;

  // prologue: W1 = U (storage precision), beta_0 = ||U_r||
  {
    double bp[R];
#pragma unroll
    for (int r = 0; r < R; ++r) bp[r] = 0.0;
    for (long long i = g.gt(kp); i < g.r1(kp); i += g.tt()) {
      double u[R];
      VecIO<R>::ld(kp.U + i * R, u);
      BT wb[R];
#pragma unroll
      for (int r = 0; r < R; ++r) { bp[r] = fma(u[r], u[r], bp[r]); wb[r] = (BT)u[r]; }
      VecIO<R>::st(W1 + i * R, wb);
    }
    if (c.tid() <= d) sh.gam[c.tid()] = gam[c.tid()];   // (read after reduce_blocks' barriers)
    if (!reduce_blocks<R>(buf, kp, c, g, bp, part_b, [&](int r, double t) { step_beta<Pol, R>(sh, kp, out, r, t, -1); }))
      return false;
  }
  // Inside the recurrence the Lanczos vector is v_j = rbeta_j w_j, formed
  // from the stored work vector w_j (src) in the accumulator precision in
  // every pass, so the polynomial's terms all act on the same vector: its
  // monomial terms cancel strongly, and mixing w_j-based and separately
  // rounded v_j terms would turn the storage rounding into an error of
  // p(B) v_j.  The rounded v_j is stored in V for the apply only.  v_{j-1}
  // is rbeta_{j-1} w_{j-1}, read from the work buffer this step overwrites.
  const BT* src = W1;
  for (int j = 0; j < m; ++j) {
    BT* Vj = V + (long long)j * n * R;
    BT* Wout = (j & 1) ? W1 : W0;
    // w = B v_j - beta_j v_{j-1} goes to the Horner buffer the last pass does
    // not read, in the accumulator precision; pass B subtracts alpha_j v_j and
    // rounds once to storage (rounding before the subtraction would make the
    // storage error relative to |w| instead of to beta_{j+1} << |w|).
    HT* Hw = (d & 1) ? H0 : H1;
    AT apa[R];
#pragma unroll
    for (int r = 0; r < R; ++r) apa[r] = Pol::zero();
    if (d == 0) {
      spmv_pass<Pol, R, BT>(kp, c, cs, src, [&](long long row, AT (&z)[R]) {
        if (row < 0) return;
        BT sv[R], v[R];
        VecIO<R>::ld(src + row * R, sv);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = Pol::scale_to_b(sv[r], sh.rb[r]);
        VecIO<R>::st(Vj + row * R, v);
        AT w[R];
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = Pol::mul(z[r], sh.sc[r]);
        if (j > 0) {
          BT wp[R];
          VecIO<R>::ld(Wout + row * R, wp);   // w_{j-1}
#pragma unroll
          for (int r = 0; r < R; ++r) w[r] = Pol::sub_mul(w[r], sh.bj[r], wp[r]);
        }
        HT wh[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { wh[r] = Pol::to_h(w[r]); apa[r] = Pol::dot(apa[r], w[r], sv[r]); }
        VecIO<R>::st(Hw + row * R, wh);
      }, nullptr, j > 0 ? Wout : nullptr);
    } else {
      // Horner pass 1: u = gamma_1 v_j + A (gamma_0 v_j); stores v_j
      const bool split = split_rows<Pol, R>(kp, c);
      if (split) {
        spmv_pass_split<Pol, R, BT>(kp, c, src, [&](long long e, int r, AT z) {
          BT sv[1], v[1];
          VecIO<1>::ld(src + e, sv);
          v[0] = Pol::scale_to_b(sv[0], sh.rb[r]);
          VecIO<1>::st(Vj + e, v);
          HT u[1];
          u[0] = Pol::to_h(Pol::add_mul(Pol::mul(z, sh.sc[r]), sh.gr[1][r], sv[0]));
          VecIO<1>::st(H1 + e, u);
        });
      } else {
        spmv_pass<Pol, R, BT>(kp, c, cs, src, [&](long long row, AT (&z)[R]) {
          if (row < 0) return;
          BT sv[R], v[R];
          VecIO<R>::ld(src + row * R, sv);
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = Pol::scale_to_b(sv[r], sh.rb[r]);
          VecIO<R>::st(Vj + row * R, v);
          HT u[R];
#pragma unroll
          for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(Pol::mul(z[r], sh.sc[r]), sh.gr[1][r], sv[r]));
          VecIO<R>::st(H1 + row * R, u);
        });
      }
      ps.done(kp);
      const HT* hin;
      if constexpr (MPK) {
        // Horner levels 2..d, pairs in one pass each, then single passes.
        // Pass k (0-based, after pass 1) reads H1 when k is even, H0 when odd,
        // and writes the other buffer.
        int k = 0, h = 2;
        for (; h + 1 <= d; h += 2, ++k) {
          if (!horner_pair<Pol, R>(kp, c, cs, ps, (k & 1) ? H0 : H1, (k & 1) ? H1 : H0, src, sh.gr[h],
                                   sh.gr[h + 1]))
            return false;
          ps.done(kp);
        }
        for (; h <= d; ++h, ++k) {
          HT* hout = (k & 1) ? H1 : H0;
          const bool ok = spmv_pass<Pol, R, HT>(kp, c, cs, (k & 1) ? H0 : H1, [&](long long row, AT (&z)[R]) {
            if (row < 0) return;
            BT sv[R];
            VecIO<R>::ld(src + row * R, sv);
            HT u[R];
#pragma unroll
            for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(z[r], sh.gr[h][r], sv[r]));
            VecIO<R>::st(hout + row * R, u);
          }, &ps);
          if (!ok) return false;
          ps.done(kp);
        }
        hin = (k & 1) ? H0 : H1;
        Hw = (k & 1) ? H1 : H0;   // w goes to the buffer the final pass does not read
      } else {
        for (int h = 2; h <= d; ++h) {
          const HT* hin_h = (h & 1) ? H0 : H1;
          HT* hout = (h & 1) ? H1 : H0;
          const bool ok = split ? spmv_pass_split<Pol, R, HT>(kp, c, hin_h, [&](long long e, int r, AT z) {
            BT sv[1];
            VecIO<1>::ld(src + e, sv);
            HT u[1];
            u[0] = Pol::to_h(Pol::add_mul(z, sh.gr[h][r], sv[0]));
            VecIO<1>::st(hout + e, u);
          }, &ps) : spmv_pass<Pol, R, HT>(kp, c, cs, hin_h, [&](long long row, AT (&z)[R]) {
            if (row < 0) return;
            BT sv[R];
            VecIO<R>::ld(src + row * R, sv);
            HT u[R];
#pragma unroll
            for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(z[r], sh.gr[h][r], sv[r]));
            VecIO<R>::st(hout + row * R, u);
          }, &ps, src);
          if (!ok) return false;
          ps.done(kp);
        }
        hin = (d & 1) ? H1 : H0;
      }
      // final pass: w = A u - beta_j v_{j-1}
      const bool ok = spmv_pass<Pol, R, HT>(kp, c, cs, hin, [&](long long row, AT (&z)[R]) {
        if (row < 0) return;
        BT sv[R];
        VecIO<R>::ld(src + row * R, sv);
        AT w[R];
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = z[r];
        if (j > 0) {
          BT wp[R];
          VecIO<R>::ld(Wout + row * R, wp);   // w_{j-1}
#pragma unroll
          for (int r = 0; r < R; ++r) w[r] = Pol::sub_mul(w[r], sh.bj[r], wp[r]);
        }
        HT wh[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { wh[r] = Pol::to_h(w[r]); apa[r] = Pol::dot(apa[r], w[r], sv[r]); }
        VecIO<R>::st(Hw + row * R, wh);
      }, &ps, j > 0 ? Wout : src);
      if (!ok) return false;
    }
    {
      double ap[R];
#pragma unroll
      for (int r = 0; r < R; ++r) ap[r] = Pol::to_d(apa[r]);
      ps.done(kp);
      if (!reduce_blocks<R>(buf, kp, c, g, ap, part_a, [&](int r, double t) { step_alpha<Pol, R>(sh, r, t); })) return false;
      for (int r = c.warp(); r < R; r += c.nw()) step_bound<Pol, R>(sh, kp, out, r, j);
    }
    // pass B: w -= alpha_j v_j; beta_{j+1} = ||w||  (after the optional
    // Gram-Schmidt against V_0..V_j)
    {
      AT bpa[R];
#pragma unroll
      for (int r = 0; r < R; ++r) bpa[r] = Pol::zero();
      const bool ro = RO && kp.reorth > 0;
      long long i = g.gt(kp);
      if (!ro) {
        // a pure stream (16-32 bytes per row): PB rows per thread per
        // iteration with all their loads issued before any store, so each
        // thread keeps PB rows in flight; rows and the ||w||^2 terms in the
        // same order as the one-row loop below (bit-identical sums)
        constexpr int PB = R == 1 ? 4 : (R == 2 ? 2 : 1);
        const long long i1 = g.r1(kp), step = g.tt();
        for (; PB > 1 && i + (PB - 1) * step < i1; i += PB * step) {
          HT wh[PB][R];
          BT v[PB][R];
#pragma unroll
          for (int u = 0; u < PB; ++u) {
            VecIO<R>::ld(Hw + (i + u * step) * R, wh[u]);
            VecIO<R>::ld(src + (i + u * step) * R, v[u]);
          }
#pragma unroll
          for (int u = 0; u < PB; ++u) {
            BT wb[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              AT w = Pol::sub_mul(h_load_at<Pol>(wh[u][r]), sh.al[r], v[u][r]);
              wb[r] = Pol::to_b(w);
              bpa[r] = Pol::dot_self(bpa[r], w);
            }
            VecIO<R>::st(Wout + (i + u * step) * R, wb);
          }
        }
      }
      for (; i < g.r1(kp); i += g.tt()) {
        HT wh[R];
        BT wb[R], v[R];
        VecIO<R>::ld(Hw + i * R, wh);
        VecIO<R>::ld(src + i * R, v);   // w_j
        if (ro) {
#pragma unroll
          for (int r = 0; r < R; ++r) wh[r] = Pol::to_h(Pol::sub_mul(h_load_at<Pol>(wh[r]), sh.al[r], v[r]));
          VecIO<R>::st(Hw + i * R, wh);
          continue;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          AT w = Pol::sub_mul(h_load_at<Pol>(wh[r]), sh.al[r], v[r]);
          wb[r] = Pol::to_b(w);
          bpa[r] = Pol::dot_self(bpa[r], w);
        }
        VecIO<R>::st(Wout + i * R, wb);
      }
      if constexpr (RO) {
        if (ro && !reorth_step<Pol, R>(kp, c, g, j, Hw, Wout, bpa)) return false;
      }
      double bp[R];
#pragma unroll
      for (int r = 0; r < R; ++r) bp[r] = Pol::to_d(bpa[r]);
      if (!reduce_blocks<R>(buf, kp, c, g, bp, part_b, [&](int r, double t) { step_beta<Pol, R>(sh, kp, out, r, t, j); }))
        return false;
    }
    src = Wout;
    bool all = true;
#pragma unroll
    for (int r = 0; r < R; ++r) all = all && sh.broken[r];
    if (all) break;
  }
  return true;
}

// ------------------------------------------------------------------ solves
// copyforsolve + linsyssolve + copyafter (lanczos_impl.cu:292-406,
// lin_sys_solves.cu:8-19): system (r, j) has diagonal alpha_r - shift,
// off-diagonals beta_r[1..meff-1] and right-hand side -beta0_r w_{r,j} e1.
// Because the right-hand side is a multiple of e1, the solution needs no
// back substitution of a general right-hand side: with the bottom-up Schur
// complements g_q = (alpha_q - s_q) - beta_{q+1} (beta_{q+1} / g_{q+1}), the
// solution is y_0 = rhs / g_0 and y_q = -beta_q y_{q-1} / g_q.
// The recurrence is serial in q; neighbouring lanes take neighbouring contour
// nodes of the same alpha/beta, complex FP64.
// Scaling: 1/g is formed from g scaled by the power of two that brings its
// larger component into [1, 2) (pair_recip), and the Schur update multiplies
// beta by (beta / g) instead of forming beta^2, so entries of T up to ~1e300
// and down to ~1e-300 neither overflow nor underflow.
//
// What bounds it: FP64 issue.  A warp's FP64 instruction holds its scheduler
// for 64 cycles on GB300 whatever its active lanes and whether or not it
// depends on the one before, so the time of a system is its FP64 instruction
// count per entry.  Hence:
//   - two lanes per system, one for the real and one for the imaginary part:
//     one instruction does both parts of every complex operation;
//   - FP64 engine: one cubic Newton reciprocal and scaling by powers of two on
//     the integer pipe instead of the two divisions of Smith's formula, and a
//     top-down sweep that multiplies by t_q = beta_q / g_q, which the bottom-up
//     sweep has formed anyway;
//   - mixed engine: Smith's formula (R. L. Smith, "Algorithm 116: Complex
//     division", CACM 5(8), 1962) on the larger and smaller component instead
//     of on both sides of a branch, operation for operation what one thread
//     per system computed.  In a time loop X becomes the next U, and FP32
//     storage turns a last-bit change of U into changes of 1e-8, so the mixed
//     engine's results keep their bits;
//   - alpha, beta, shifts and t_q are loaded kTriU entries ahead (two: the
//     engine's kernels have 40 to 64 registers; m = 453 345 us, four 387 us);
//   - the warps' systems are spread over the blocks, one warp per SM first.
// Against one thread per system with Smith's formula on both sides of a branch:
// FP64 m = 60 120 -> 55 us, m = 200 378 -> 147; mixed m = 453 1010 -> 450.
constexpr int kTriU = 2;

// x * 2^(-k) by exponent arithmetic: exact while x and the result are normal
// numbers, 0 below that (the callers' results stay below the largest number).
__device__ __forceinline__ double scale_exp2(double x, int k) {
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7ff;
  return ex > max(k, 0) ? __hiloint2double(hi - (k << 20), __double2loint(x)) : 0.0;
}

// This lane's component of 1/(a + ib), g being this lane's component (even
// lanes a, odd lanes b), by Smith's formula, which never forms |g|^2: with x the
// larger and y the smaller component, t = y / x and v = 1 / (x + y t), 1/g is
// (v, -t v) for a larger real part and (t v, -v) otherwise.  Called by whole
// warps, as pair_recip is.
__device__ __forceinline__ double pair_recip_smith(double g) {
  const double o = __shfl_xor_sync(0xffffffffu, g, 1);
  const bool im = threadIdx.x & 1;
  const double a = im ? o : g, b = im ? g : o;
  const bool real_big = (__double_as_longlong(a) & 0x7fffffffffffffffll) >= (__double_as_longlong(b) & 0x7fffffffffffffffll);
  const double x = real_big ? a : b, y = real_big ? b : a;
  const double t = y / x;
  const double v = 1.0 / fma(y, t, x);
  const double tv = t * v;
  return im ? (real_big ? -tv : -v) : (real_big ? v : tv);
}

// The same in the FP64 engine.  g is scaled by 2^-e, e the exponent of its
// larger component, so that |g|^2 lies in [1, 8).  From r, the FP32 reciprocal of
// |g|^2 with an error of about 2^-22, one cubically convergent Newton step gives
// x r (1 + h + h^2), h = 1 - |g|^2 r, an error of 2^-66 before rounding.  h and the
// product keep the exact x r = p + e: without it (|g|^2 and its reciprocal
// rounded, two instructions of eight less) the root mean square of the relative
// error is 0.83 to 0.85 of 2^-53 and the solutions' error 1.06 times that with
// Smith's formula, which has 0.59 to 0.65; this has 0.44 to 0.48, and the
// solutions 0.98 times (nine operators, 60 right-hand sides each).  The
// conversions to and from FP32 move bits (truncating): m = 450 357 -> 338 us,
// which is what the shorter form took.
// The scaling drops subnormal components: where those may be more
// than 2^-63 of |g| or |1/g|, and for 0, Inf and NaN, the pair takes Smith's
// formula, which the whole warp then runs (every shuffle names all lanes).
__device__ __forceinline__ double pair_recip(double x) {
  const unsigned full = 0xffffffffu;
  const bool im = threadIdx.x & 1;
  const int ex = (__double2hiint(x) >> 20) & 0x7ff, eo = __shfl_xor_sync(full, ex, 1);
  const int em = max(ex, eo), k = em - 1023;
  const double xs = scale_exp2(x, k);
  // (roundings spelled out: both lanes must form the same r, and a contracted
  // sum would count e twice)
  const int hi = __double2hiint(xs) & 0x7fffffff;
  const float xf = hi >= 0x38100000 ? __int_as_float(((hi - 0x38000000) << 3) | (int)((unsigned)__double2loint(xs) >> 29)) : 0.f;
  const float sq = __fmul_rn(xf, xf);
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__fadd_rn(sq, __shfl_xor_sync(full, sq, 1))));
  const int rb = __float_as_int(rf);
  const double r = __hiloint2double((rb >> 3) + 0x38000000, rb << 29);
  const double p = __dmul_rn(xs, r), e = fma(xs, r, -p);
  // the lane of the larger component starts at 1, the other at 0
  const double f = fma(-xs, e, fma(-xs, p, ex > eo || (ex == eo && !im) ? 1.0 : 0.0));
  const double h = __dadd_rn(f, __shfl_xor_sync(full, f, 1));
  const double q = scale_exp2(fma(xs, r, __dmul_rn(p, fma(h, h, h))), k);
  double y = im ? -q : q;
  const bool out = em < 64 || em > 1980;
  if (__any_sync(full, out)) {
    const double z = pair_recip_smith(x);
    if (out) y = z;
  }
  return y;
}

template <int R, bool kSmith>
__device__ void phase_trisolve(const KParams& kp, const Ctx& c) {
  const int m = kp.m, C = kp.C;
  const int np = kp.nprob > 0 ? kp.nprob : 1;
  const long long nsys = (long long)np * R * C;
  const unsigned full = 0xffffffffu;
  const bool im = threadIdx.x & 1;
  // warp w of block b takes systems 16 (w G + b) + lane / 2; lanes past the
  // last system repeat it without storing, so that every shuffle is full
  for (long long s0 = 16LL * ((long long)c.warp() * c.G + c.b()); s0 < nsys; s0 += c.tt() / 2) {
    const long long sl = s0 + (c.lane() >> 1);
    const bool act = sl < nsys;
    const long long sys = act ? sl : nsys - 1;
    // sys = (p R + r) C + j for problem p, right-hand side r, node j
    const long long rr = sys / C;
    const int j = (int)(sys % C);
    const long long p = rr / R;
    const int r = (int)(rr % R);
    const int me = kp.meff[rr];
    int mew = me;   // the warp's largest m_eff: its loops' common length
    for (int o = 16; o > 0; o >>= 1) mew = max(mew, __shfl_xor_sync(full, mew, o));
    const double* __restrict__ al = kp.aabb + (long long)(m + 1) * (2 * R * p + r);
    const double* __restrict__ be = kp.aabb + (long long)(m + 1) * (2 * R * p + R + r);
    const double* __restrict__ sh = kp.shifts + 2LL * m * sys + (im ? 1 : 0);
    // kept per entry, (re, im): 1/g_q, or in the FP64 engine beta_q / g_q for q >= 1
    double* ts = kp.tri + 4LL * m * sys;
    double* __restrict__ y = (im ? kp.Yi : kp.Yr) + (long long)m * sys;
    double t = 0.0, bn = 0.0;   // t_{q+1} = beta_{q+1} / g_{q+1} (Smith: 1/g_{q+1}) and beta_{q+1}
    double la[kTriU], lb[kTriU], ls[kTriU];
    auto load = [&](int q0) {
#pragma unroll
      for (int u = 0; u < kTriU; ++u) {
        const int q = q0 - u;
        const bool in = q >= 0 && q < me;
        la[u] = in && !im ? al[q] : 0.0;
        lb[u] = in ? be[q] : 0.0;
        ls[u] = in ? sh[2 * q] : -1.0;
      }
    };
    load(mew - 1);
    for (int q0 = mew - 1; q0 >= 0; q0 -= kTriU) {
      double ca[kTriU], cb[kTriU];
#pragma unroll
      for (int u = 0; u < kTriU; ++u) { ca[u] = la[u] - ls[u]; cb[u] = lb[u]; }
      load(q0 - kTriU);
#pragma unroll
      for (int u = 0; u < kTriU; ++u) {
        const int q = q0 - u;
        if (q < 0) break;
        // Schur complement: beta^2 / g_{q+1} as beta (beta / g_{q+1})
        const double g = fma(-bn, kSmith ? bn * t : t, ca[u]);
        const double ig = kSmith ? pair_recip_smith(g) : pair_recip(g);
        if (q < me) {
          bn = cb[u];
          t = !kSmith && q > 0 ? bn * ig : ig;
          if (act) ts[2 * q + (im ? 1 : 0)] = t;
        }
      }
    }
    // y_0 = rhs / g_0, rhs = -(beta0 w); y_q = -(beta_q / g_q) y_{q-1}
    double yo = 0.0;
    {
      const double b0 = be[0];
      const double xr = -(b0 * kp.wts[2LL * C * rr + j]), xi = -(b0 * kp.wts[2LL * C * rr + C + j]);
      const double to = __shfl_xor_sync(full, t, 1);
      // re: xr tr - xi ti; im: xr ti + xi tr
      const double q1 = xi * to;
      if (me > 0) yo = fma(xr, t, im ? q1 : -q1);
      if (act && me > 0) y[0] = yo;
    }
    __syncwarp();   // ts written by the pair's other lane
    const double2* tv = reinterpret_cast<const double2*>(ts);
    double2 lt[kTriU];
    double lq[kTriU];   // Smith: beta_q
    auto load_t = [&](int q0) {
#pragma unroll
      for (int u = 0; u < kTriU; ++u)
        if (q0 + u < me) {
          lt[u] = tv[q0 + u];
          if (kSmith) lq[u] = be[q0 + u];
        }
    };
    load_t(1);
    for (int q0 = 1; q0 < mew; q0 += kTriU) {
      double2 ct[kTriU];
      double cq[kTriU];
#pragma unroll
      for (int u = 0; u < kTriU; ++u) { ct[u] = lt[u]; cq[u] = lq[u]; }
      load_t(q0 + kTriU);
#pragma unroll
      for (int u = 0; u < kTriU; ++u) {
        const int q = q0 + u;
        if (q >= mew) break;
        if constexpr (kSmith) {
          // (tr, ti) = -beta_q y_{q-1}; re: tr gr - ti gi; im: ti gr + tr gi
          const double po = -cq[u] * yo, q1 = __shfl_xor_sync(full, po, 1) * ct[u].y;
          yo = fma(po, ct[u].x, im ? q1 : -q1);
        } else {
          // re: ty yi - tx yr; im: -ty yr - tx yi
          const double other = __shfl_xor_sync(full, yo, 1);
          yo = fma(im ? -ct[u].y : ct[u].y, other, -(ct[u].x * yo));
        }
        if (act && q < me) y[q] = yo;
      }
    }
    if (act)
      for (int q = me; q < m; ++q) y[q] = 0.0;
  }
}

// coef[r][i][q] = sum_j Im(gs(i, j) y_{r, j}[q]) = sum_j gs_re y_im + gs_im y_re:
// the m-vectors that collapse apply_V.cu's 2C per-node passes into one lift.
template <int R>
__device__ void phase_coef(const KParams& kp, const Ctx& c) {
  const int m = kp.m, C = kp.C, d1 = kp.d + 1;
  const int np = kp.nprob > 0 ? kp.nprob : 1;
  const long long total = (long long)np * R * d1 * m;
  // (warps spread over the blocks: FP64 issue is per scheduler)
  for (long long t = 32LL * ((long long)c.warp() * c.G + c.b()) + c.lane(); t < total; t += c.tt()) {
    // t = (rr d1 + i) m + q with rr = p R + r
    const int q = (int)(t % m);
    const int i = (int)((t / m) % d1);
    const long long rr = t / ((long long)m * d1);
    const long long p = rr / R;
    const double* gr = kp.gs_re + (long long)d1 * C * p;
    const double* gi = kp.gs_im + (long long)d1 * C * p;
    double acc = 0.0;
#pragma unroll 8
    for (int j = 0; j < C; ++j) {
      const long long col = rr * C + j;
      acc = fma(gr[i + (long long)d1 * j], kp.Yi[col * m + q], acc);
      acc = fma(gi[i + (long long)d1 * j], kp.Yr[col * m + q], acc);
    }
    kp.coef[t] = acc;
    const float h = (float)acc;
    kp.coef_ff[t] = make_float2(h, (float)(acc - (double)h));
  }
}

// ------------------------------------------------------------------ APPLY
// X_r += sum_i A^(d-i) V_r c_{r,i}: one lift pass P_i = V c_i, then d Horner
// passes X = A X + P_i.
//
// The lift is row-local: the general path runs it as a kernel of its own
// (k_lift, a thread per row and chunk of polynomial terms, no grid barrier, its
// own registers), the resident entry points as part of theirs.  It streams
// V; a load per Krylov vector and row in series left it latency-bound at a
// third to a half of the memory rate, so QU vectors are loaded before their
// products.  Measured, the whole apply: 300k-node disk mixed, degree 8, four
// right-hand sides 1427 -> 667 us; 160^3 mixed without a polynomial, m = 100,
// 626 -> 411; 117^3 FP64 225 -> 172; batch of 24 211 -> 178.  Three terms per
// pass over V and exact counts: wider chunks cost more in registers than they
// save in reads, and a guard per term computes the absent ones (117^3: 1616 us
// with nine guarded terms).
constexpr int kLiftTerms = 3;                                             // polynomial terms per pass over V
template <int R> struct LiftWidth { static constexpr int value = R == 1 ? 8 : 4; };   // Krylov vectors in flight

// acc[ii][r] = sum_q c_{r, i0 + ii}[q] V_q[i][r] over the first mv vectors, q
// ascending.
template <class Pol, int R, int IC>
__device__ __forceinline__ void lift_row(const KParams& kp, int p, long long i, int i0, int mv,
                                         typename Pol::AT (&acc)[IC][R]) {
  using BT = typename Pol::BT;
  constexpr int QU = LiftWidth<R>::value;
  const int m = kp.m, d1 = kp.d + 1;
  const BT* v0 = reinterpret_cast<const BT*>(kp.V) + i * R;
  const long long step = kp.n * R, c0 = (long long)R * p * d1 + i0;
#pragma unroll
  for (int ii = 0; ii < IC; ++ii)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[ii][r] = Pol::zero();
  auto add = [&](int q, const BT (&v)[R]) {
#pragma unroll
    for (int ii = 0; ii < IC; ++ii) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const long long ci = (c0 + (long long)r * d1 + ii) * m + q;
        if constexpr (Pol::kMixed) {
          const float2 cf = kp.coef_ff[ci];
          acc[ii][r] = Pol::add(acc[ii][r], ff_mulf(ff{cf.x, cf.y}, v[r]));
        } else {
          acc[ii][r] = fma((double)v[r], kp.coef[ci], acc[ii][r]);
        }
      }
    }
  };
  int q = 0;
  for (; q + QU <= mv; q += QU) {
    BT v[QU][R];
#pragma unroll
    for (int u = 0; u < QU; ++u) VecIO<R>::ld(v0 + (q + u) * step, v[u]);
#pragma unroll
    for (int u = 0; u < QU; ++u) add(q + u, v[u]);
  }
  for (; q < mv; ++q) {
    BT v[R];
    VecIO<R>::ld(v0 + q * step, v);
    add(q, v);
  }
}

// The lift's result for row i: P terms i0.., or without a polynomial X and S.
template <class Pol, int R, int IC>
__device__ __forceinline__ void lift_store(const KParams& kp, long long i, int i0, bool overwrite,
                                           const typename Pol::AT (&acc)[IC][R]) {
  using HT = typename Pol::HT;
  if (kp.d == 0) {
    double x[R], u[R], s[R];
    if (overwrite) {
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = 0.0;
    } else {
      VecIO<R>::ld(kp.X + i * R, x);
    }
    VecIO<R>::ld(kp.upd + i * R, u);
#pragma unroll
    for (int r = 0; r < R; ++r) { x[r] += Pol::to_d(acc[0][r]); s[r] = x[r] + u[r]; }
    VecIO<R>::st(kp.X + i * R, x);
    VecIO<R>::st(kp.S + i * R, s);
    return;
  }
  HT* P = reinterpret_cast<HT*>(kp.P);
#pragma unroll
  for (int ii = 0; ii < IC; ++ii) {
    HT hv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) hv[r] = Pol::to_h(acc[ii][r]);
    VecIO<R>::st(P + ((long long)(i0 + ii) * kp.n + i) * R, hv);
  }
}

// Chunk y of the d + 1 terms: whole chunks of kLiftTerms, then single terms.
__host__ __device__ inline int lift_chunks(int d) { return (d + 1) / kLiftTerms + (d + 1) % kLiftTerms; }
template <class Pol, int R>
__device__ __forceinline__ void lift_chunk(const KParams& kp, int p, long long i, int y, int mv, bool overwrite) {
  const int full = (kp.d + 1) / kLiftTerms;
  if (y < full) {
    typename Pol::AT acc[kLiftTerms][R];
    lift_row<Pol, R, kLiftTerms>(kp, p, i, y * kLiftTerms, mv, acc);
    lift_store<Pol, R, kLiftTerms>(kp, i, y * kLiftTerms, overwrite, acc);
  } else {
    typename Pol::AT acc[1][R];
    const int i0 = full * kLiftTerms + (y - full);
    lift_row<Pol, R, 1>(kp, p, i, i0, mv, acc);
    lift_store<Pol, R, 1>(kp, i, i0, overwrite, acc);
  }
}

// 256 / 128 / 64 threads: 16,384 rows at m = 200 take 56 / 33 / 46 us (at 256
// they fill 64 of 152 SMs); the large cases agree within 3 %.
constexpr int kLiftBlock = 128;
template <class Pol, int R>
__global__ void __launch_bounds__(kLiftBlock) k_lift(KParams kp) {
  if (*(volatile int*)kp.status != 0) return;
  const long long i = (long long)blockIdx.x * kLiftBlock + threadIdx.x;
  if (i >= kp.n) return;
  int p = 0;   // the row's problem
  if (kp.nprob > 1) {
    int hi = kp.nprob;
    while (hi - p > 1) {
      const int mid = (p + hi) >> 1;
      if (kp.prob_row0[mid] <= i) p = mid; else hi = mid;
    }
  }
  lift_chunk<Pol, R>(kp, p, i, (int)blockIdx.y, kp.m, (kp.phases & PH_APPLY_SET) != 0);
}

template <class Pol, int R, bool kLift>
__device__ bool phase_apply(const KParams& kp, const Ctx& c, const Grp& g, bool overwrite, PassSync& ps,
                            ColStage& cs) {
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  const long long n = kp.n;
  const int d = kp.d;
  HT* P = reinterpret_cast<HT*>(kp.P);
  HT* const H0 = reinterpret_cast<HT*>(kp.H0);
  HT* const H1 = reinterpret_cast<HT*>(kp.H1);
  if constexpr (kLift) {
    // (the vectors past m_eff of every column stay out: see clear_unwritten)
    int mv = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) mv = max(mv, kp.meff[R * g.p + r]);
    const long long sb = kp.blk_slice[c.b()], se = kp.blk_slice[c.b() + 1];
    for (long long s = sb + c.warp(); s < se; s += c.nw()) {
      const long long i = slot_row(kp, s, c.lane());
      if (i < 0) continue;
      for (int y = 0; y < lift_chunks(d); ++y) lift_chunk<Pol, R>(kp, g.p, i, y, mv, overwrite);
    }
    if (d == 0) return true;
    ps.done(kp);
  }
  for (int h = 1; h <= d; ++h) {
    const HT* hin = h == 1 ? P : ((h & 1) ? H0 : H1);
    HT* hout = (h & 1) ? H1 : H0;
    const HT* Ph = P + (long long)h * n * R;
    const bool ok = spmv_pass<Pol, R, HT>(kp, c, cs, hin, [&](long long row, AT (&z)[R]) {
      if (row < 0) return;
      HT p[R];
      VecIO<R>::ld(Ph + row * R, p);
      AT x[R];
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = Pol::add(z[r], h_load_at<Pol>(p[r]));
      if (h < d) {
        HT hv[R];
#pragma unroll
        for (int r = 0; r < R; ++r) hv[r] = Pol::to_h(x[r]);
        VecIO<R>::st(hout + row * R, hv);
      } else {
        double xo[R], u[R], so[R];
        if (overwrite) {
#pragma unroll
          for (int r = 0; r < R; ++r) xo[r] = 0.0;
        } else {
          VecIO<R>::ld(kp.X + row * R, xo);
        }
        VecIO<R>::ld(kp.upd + row * R, u);
#pragma unroll
        for (int r = 0; r < R; ++r) { xo[r] += Pol::to_d(x[r]); so[r] = xo[r] + u[r]; }
        VecIO<R>::st(kp.X + row * R, xo);
        VecIO<R>::st(kp.S + row * R, so);
      }
    }, kLift || h > 1 ? &ps : nullptr);
    if (!ok) return false;
    if (h < d) ps.done(kp);
  }
  return true;
}

// ------------------------------------------------------------------ UPDATE + DEFLATE
// Pass 1 (optional time step, update_U.cu:8-16 / update_U_monodomain.cu:8-22)
// then Z = Q^T Usol; pass 2: U = Usol - Q Z, update = Q (flam o Z), X = 0
// (lanczos_impl.cu:84-89, update_U.cu:26-38).
template <int R, bool kOrdered>
__device__ bool phase_deflate(const KParams& kp, const Ctx& c, int mode) {
  const long long n = kp.n;
  const int k = kp.k, G = kp.G;
  GridBar bar{bar_word(kp, -1), kp.status, (unsigned)G, kp.timeout_ns};
  double* part_z = kp.part + 2LL * R * G;
  constexpr int KC = 4;
  if (mode != 0 && R == 2) {
    for (long long i = c.gt(); i < n; i += c.tt()) {
      const double* x = kp.X + i * 2;
      const double* up = kp.upd + i * 2;
      double u = ((x[0] + x[1]) + up[0]) + up[1];
      double g;
      if (mode == 1) {
        u = u * (double)(u >= 0.0);
        const double uo = u / kp.mass[i];
        g = kp.mass[i] * uo * (1.0 - uo);
        g = g * kp.dt;
      } else {
        const double p1 = u * (kp.dt * kp.aode);
        const double p2 = kp.ode[i] * (kp.dt * kp.bode);
        const double o = kp.ode[i] + ((p1 + p2) + kp.code);
        kp.ode[i] = o;
        double srcv = ((u - kp.vrest) * u) * (u - kp.vpeak);
        srcv = srcv * ((kp.c1ion / kp.vamp) / kp.vamp);
        g = (srcv - o) * kp.dt;
      }
      kp.Usol[i * 2] = u;
      kp.Usol[i * 2 + 1] = g;
    }
  }
  if (k > 0) {
    for (int e0 = 0; e0 < k; e0 += KC) {
      double zp[KC * R];
#pragma unroll
      for (int t = 0; t < KC * R; ++t) zp[t] = 0.0;
      for (long long i = c.gt(); i < n; i += c.tt()) {
        double u[R];
        VecIO<R>::ld(kp.Usol + i * R, u);
#pragma unroll
        for (int ee = 0; ee < KC; ++ee) {
          if (e0 + ee < k) {
            const double q = kp.Q[(long long)(e0 + ee) * n + i];
#pragma unroll
            for (int r = 0; r < R; ++r) zp[ee * R + r] = fma(q, u[r], zp[ee * R + r]);
          }
        }
      }
      block_sum_store<KC * R>(zp, part_z + (long long)e0 * R * G + c.b(), G);
    }
    if (!bar.sync()) return false;
    // every block totals the k*R entries in the same fixed order
    __shared__ double s_z[256];
    const int kr = k * R;
    for (int t0 = 0; t0 < kr; t0 += 256) {
      if constexpr (kOrdered) {
        // the mixed engine's U keeps its bits (see phase_trisolve): one thread
        // per entry adds the blocks in order, 16 loads ahead of the additions
        for (int t = t0 + c.tid(); t < kr && t < t0 + 256; t += c.nt()) {
          double acc = 0.0;
          const double* p = part_z + (long long)t * G;
          int b = 0;
          for (; b + 16 <= G; b += 16) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = p[b + u];
#pragma unroll
            for (int u = 0; u < 16; ++u) acc += v[u];
          }
          for (; b < G; ++b) acc += p[b];
          s_z[t - t0] = acc;
          if (c.b() == 0) kp.Z[t] = acc;
        }
      } else {
        // one warp per entry, lanes over the blocks' partials (one thread per
        // entry, all G of them in series: 256^2 with 10 modes 35 us a launch,
        // now 27)
        for (int t = t0 + c.warp(); t < kr && t < t0 + 256; t += c.nw()) {
          const double* p = part_z + (long long)t * G;
          double acc = 0.0;
          for (int b = c.lane(); b < G; b += 32) acc += p[b];
          acc = warp_sum(acc);
          if (c.lane() == 0) {
            s_z[t - t0] = acc;
            if (c.b() == 0) kp.Z[t] = acc;
          }
        }
      }
      __syncthreads();
      // pass 2 over this chunk of Z entries (rows by thread stride)
      const int e_lo = t0 / R, e_hi = min(k, (t0 + 256) / R);
      for (long long i = c.gt(); i < n; i += c.tt()) {
        double u[R], up[R];
        if (t0 == 0) {
          VecIO<R>::ld(kp.Usol + i * R, u);
#pragma unroll
          for (int r = 0; r < R; ++r) up[r] = 0.0;
        } else {
          VecIO<R>::ld(kp.U + i * R, u);
          VecIO<R>::ld(kp.upd + i * R, up);
        }
        double qz[R];
#pragma unroll
        for (int r = 0; r < R; ++r) qz[r] = 0.0;
        for (int e = e_lo; e < e_hi; ++e) {
          const double q = kp.Q[(long long)e * n + i];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double z = s_z[e * R + r - t0];
            qz[r] = fma(q, z, qz[r]);
            up[r] = fma(q, kp.flam[e + (long long)k * r] * z, up[r]);
          }
        }
        double x0[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { u[r] = u[r] - qz[r]; x0[r] = 0.0; }
        VecIO<R>::st(kp.U + i * R, u);
        VecIO<R>::st(kp.upd + i * R, up);
        VecIO<R>::st(kp.X + i * R, x0);
      }
      __syncthreads();
    }
  } else {
    for (long long i = c.gt(); i < n; i += c.tt()) {
      double u[R], z0[R];
      VecIO<R>::ld(kp.Usol + i * R, u);
#pragma unroll
      for (int r = 0; r < R; ++r) z0[r] = 0.0;
      VecIO<R>::st(kp.U + i * R, u);
      VecIO<R>::st(kp.upd + i * R, z0);
      VecIO<R>::st(kp.X + i * R, z0);
    }
  }
  return true;
}

}  // namespace gm

#include "fab_resident.cuh"

namespace gm {

// ------------------------------------------------------------------ kernel
// Phase groups compiled as separate entry points.
constexpr int KG_LANCZOS = PH_LANCZOS;
constexpr int KG_SOLVE = PH_TRISOLVE | PH_COEF;
constexpr int KG_APPLY = PH_APPLY | PH_APPLY_SET;
constexpr int KG_DEFLATE = PH_DEFLATE | PH_UPDATE_FKPP | PH_UPDATE_FHN;

// Block size of the shifted solves' entry point: few warps per SM, each with
// registers for the entries loaded ahead (at 40 they spilled).
constexpr int kSolveThreads = 128;

// Zeros in the Krylov vectors that a build left unwritten because every column
// of a problem broke down.  The lift reads all m, and what they held before
// (fresh memory, or NaN of a failed build) would come through its zero
// coefficients.  It is done here, where nothing is tight: an end to the lift's
// loop at m_eff cost the batch of 24 1 %, and these lines after the Lanczos loop
// made one of its entry points spill.  (In the resident one-launch solve it is
// the other way round: 64 x 64 takes 432 us with the loop's end at m_eff and 446
// with these lines.)
template <class Pol, int R>
__device__ void clear_unwritten(const KParams& kp, const Ctx& c) {
  using BT = typename Pol::BT;
  const int m = kp.m, np = kp.nprob > 0 ? kp.nprob : 1;
  auto written = [&](int p) {
    int mv = 0;
    for (int r = 0; r < R; ++r) mv = max(mv, kp.meff[R * p + r]);
    return mv;
  };
  bool any = false;
  for (int p = c.tid(); p < np; p += c.nt()) any = any || written(p) < m;
  if (!__syncthreads_or(any)) return;
  BT* const V = reinterpret_cast<BT*>(kp.V);
  BT z[R];
#pragma unroll
  for (int r = 0; r < R; ++r) z[r] = (BT)0;
  for (int p = 0; p < np; ++p) {
    const long long r0 = kp.nprob > 0 ? kp.prob_row0[p] : 0, r1 = kp.nprob > 0 ? kp.prob_row0[p + 1] : kp.n;
    for (int q = written(p); q < m; ++q)
      for (long long i = r0 + c.gt(); i < r1; i += c.tt()) VecIO<R>::st(V + ((long long)q * kp.n + i) * R, z);
  }
}

// The shifted solves or the coefficients, one of them per launch; the latter
// always comes between a build and its apply.  Its grid is
// sized by the SMs and not by the partition, so nothing here may look up the
// tables that hold an entry per block of the partition.
template <class Pol, int R>
__global__ void __launch_bounds__(kSolveThreads, 3) k_solve(KParams kp) {
  if (*(volatile int*)kp.status != 0) return;
  const Ctx c(kp.G);
  if (kp.phases & PH_TRISOLVE) phase_trisolve<R, Pol::kMixed>(kp, c);
  if (kp.phases & PH_COEF) {
    clear_unwritten<Pol, R>(kp, c);
    phase_coef<R>(kp, c);
  }
}

// PH is the compile-time set of phases this entry point can run (the runtime
// mask kp.phases selects among them); specialising on it lets the compiler
// size registers per phase group.
#ifndef GM_MINB
#define GM_MINB 2
#endif
#ifndef GM_MAXT
#define GM_MAXT 512
#endif
static_assert(GM_MAXT <= ReduceBuf<1>::kCap, "a block's sums are staged in kCap words");
template <class Pol, int R, int PH>
#ifndef GM_MINB4
#define GM_MINB4 2   // resident 512-thread blocks per SM for four right-hand sides
#endif
#ifndef GM_MINB4M
#define GM_MINB4M 3   // four right-hand sides, mixed precision, Lanczos entry points
#endif
#ifndef GM_MINB1
#define GM_MINB1 3   // and for one right-hand side
#endif
#ifndef GM_MINB1X
#define GM_MINB1X 2   // one right-hand side, matrix-powers or Gram-Schmidt entry points
#endif
#ifndef GM_MINB1L2
#define GM_MINB1L2 2   // one right-hand side, mixed, matrix held in the L2 window (PolMixedL2)
#endif
__global__ void __launch_bounds__((PH & PH_RESIDENT) ? kResThreads : GM_MAXT, ((PH & PH_RESIDENT) ? 1 : R >= 4 ? ((Pol::kMixed && !(PH & (PH_MPK | PH_REORTH))) ? GM_MINB4M : GM_MINB4)
                                            : (R == 1 ? ((PH & (PH_MPK | PH_REORTH)) ? GM_MINB1X
                                                                                     : (Pol::kL2 ? GM_MINB1L2 : GM_MINB1))
                                                      : GM_MINB))) fab_kernel(KParams kp) {
  const Ctx c(kp.G);
  if (*(volatile int*)kp.status != 0) return;
  const int ph = kp.phases & PH;
  const Grp g(kp, c);
  PassSync ps{kp.dep_mode, g.p, 0u};
  ColStage cs;
  if constexpr (Pol::kDia) {
    int* const tab = dia_table();
    const int p0 = kp.dia_pat0[g.p], pn = kp.dia_pat0[g.p + 1] - p0;
    for (int t = c.tid(); t < pn * kp.dia_len; t += c.nt()) tab[t] = kp.dia_off[p0 * kp.dia_len + t];
    if (c.tid() == 0) tab[kDiaTable] = kp.dia_shift[g.p];
    __syncthreads();
  } else if (PH & (PH_LANCZOS | PH_APPLY)) {
    cs.init(kp, c);
  }
  bool first = true;
  auto sep = [&]() -> bool {
    if (first) { first = false; return true; }
    return GridBar{bar_word(kp, -1), kp.status, (unsigned)kp.G, kp.timeout_ns}.sync();
  };
  if ((PH & PH_LANCZOS) && (ph & PH_LANCZOS)) {
    if (!sep()) return;
    if constexpr ((PH & PH_RESIDENT) != 0) {
      if (!phase_lanczos_resident<Pol, R>(kp, c)) return;
    } else {
      if (!phase_lanczos<Pol, R, (PH & PH_MPK) != 0, (PH & PH_REORTH) != 0>(kp, c, g, ps, cs)) return;
    }
  }
  if ((PH & PH_TRISOLVE) && (ph & PH_TRISOLVE)) {
    if (!sep()) return;
    // A build that met a non-finite value has recorded it before its barrier:
    // the handle's results stay as they were.  (Launched by themselves, the
    // phases after the build find the status where they start.)
    if (__syncthreads_or(c.tid() == 0 && *(volatile int*)kp.status != 0)) return;
    phase_trisolve<R, Pol::kMixed>(kp, c);
  }
  if ((PH & PH_COEF) && (ph & PH_COEF)) {
    if (!sep()) return;
    phase_coef<R>(kp, c);
  }
  if ((PH & PH_APPLY) && (ph & PH_APPLY)) {
    if (!sep()) return;
    if (!phase_apply<Pol, R, (PH & PH_RESIDENT) != 0>(kp, c, g, (ph & PH_APPLY_SET) != 0, ps, cs)) return;
  }
  if (PH & (PH_DEFLATE | PH_UPDATE_FKPP | PH_UPDATE_FHN)) {
    const int upd_mode = (ph & PH_UPDATE_FKPP) ? 1 : ((ph & PH_UPDATE_FHN) ? 2 : 0);
    if ((ph & PH_DEFLATE) || upd_mode) {
      if (!sep()) return;
      if (!phase_deflate<R, Pol::kMixed>(kp, c, upd_mode)) return;
    }
  }
}

}  // namespace gm
