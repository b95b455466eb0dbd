// The Lanczos phase of problems with at most one SELL slice per warp on one
// block per SM (16 slices per SM: 77,824 rows on 152 SMs).  The block's share
// of the matrix stays in shared memory for the whole launch, each thread keeps
// its row of w_j, w_{j-1} and the step's result in registers, and blocks
// exchange only the rows that another block references.
//
// What bounds it: round trips through L2 and FP64 issue.  A step at these
// sizes computes for about a microsecond; the general phase spends 12 to 20 us
// on it, in chains of L2 round trips (slice offsets, column copy, one gather
// per entry, row operands; the barrier's fence, atomic, poll, fence and status
// read; the partials).  Here a pass costs one:
//   - an exported vector entry travels as a 16-byte word (value, tag), written
//     and read by single 128-bit relaxed accesses, so the word that arrives is
//     its own flag: no fence, no flag, no L1 invalidation;
//   - the block partials of alpha and beta travel the same way, and every
//     block sums all of them in one fixed order (identical bits everywhere);
//   - the halo of the next step's vector is read while one warp per right-hand
//     side waits for beta.
// A warp's FP64 instruction holds its scheduler for 64 cycles whatever its
// active lanes, so in the FP64 engine the sums run on the integer pipe
// (warp_fixed_sum), beta and 1/beta come from one FP32 reciprocal square root,
// and the scalars of a step are formed by different lanes at once.
//
// The mixed engine stores its Lanczos vectors in FP32, and a last-bit change of
// alpha or beta flips roundings there that a long recurrence amplifies to
// 1e-8.  It therefore keeps the general path's sums bit for bit: the same two
// groupings of slices into blocks of 16 warps (alpha by the balanced partition
// that also owns the rows, beta by rows) and the same trees.  A slice whose
// beta belongs to another block's group sends its sum there, as a word.
//
// Exchange k of a launch uses half k & 1 of the word buffer and tag
// (epoch << 32) + k.  A block writes exchange k + 2 only after it has read
// exchange k + 1 of every block that reads its rows, and such a block posted
// k + 1 after it had read k (the host makes "reads from" symmetric: a block
// that is read one way reads a row of its reader): no word is overwritten
// unread.  The words of alpha and
// beta alternate too: a block posts its next alpha after the beta that every
// other block posted after it had read the last alpha.
//
// Included by fab_kernel.cuh.
#pragma once

namespace gm {

__device__ __forceinline__ void st_word(ulonglong2* p, unsigned long long data, unsigned long long tag) {
  asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}"
               ::"l"(p), "l"(data), "l"(tag) : "memory");
}
__device__ __forceinline__ void ld_word(const ulonglong2* p, unsigned long long& data, unsigned long long& tag) {
  asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}"
               : "=l"(data), "=l"(tag) : "l"(p) : "memory");
}

// Waits, within the launch's limit, until *p carries tag.  False when the
// limit has passed (recorded) or another block has recorded an error.  No
// backoff: sleeping 50 ns between reads cost 256^2 8.6 -> 12.3 us per step.
__device__ __forceinline__ bool poll_word(const KParams& kp, const ulonglong2* p, unsigned long long tag,
                                          unsigned long long& data) {
  unsigned long long t, start = 0;
  ld_word(p, data, t);
  unsigned spins = 0;
  while (t != tag) {
    if ((++spins & 7u) == 0u) {
      const unsigned long long now = global_timer_ns();
      if (start == 0) {
        start = now;
      } else if (now - start > kp.timeout_ns) {
        atomicCAS(kp.status, 0, (int)ST_TIMEOUT);
        return false;
      }
      if ((spins & 63u) == 0u && *(volatile int*)kp.status != 0) return false;
    }
    ld_word(p, data, t);
  }
  return true;
}

__device__ __forceinline__ unsigned long long to_bits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ unsigned long long to_bits(float x) { return (unsigned long long)__float_as_uint(x); }
__device__ __forceinline__ unsigned long long to_bits(float2 x) {
  return (unsigned long long)__float_as_uint(x.x) | ((unsigned long long)__float_as_uint(x.y) << 32);
}
__device__ __forceinline__ void from_bits(unsigned long long b, double& x) { x = __longlong_as_double((long long)b); }
__device__ __forceinline__ void from_bits(unsigned long long b, float& x) { x = __uint_as_float((unsigned)b); }
__device__ __forceinline__ void from_bits(unsigned long long b, float2& x) {
  x = make_float2(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

// Exponent (biased as FP64's), sign and 53-bit mantissa: x = +-q 2^(e - 1075).
__device__ __forceinline__ long long fixed_parts(double x, int& e, bool& neg) {
  const int hi = __double2hiint(x), f = (hi >> 20) & 0x7ff;
  e = max(f, 1);
  neg = hi < 0;
  return ((long long)((hi & 0xfffff) | (f > 0 ? 0x100000 : 0)) << 32) | (unsigned)__double2loint(x);
}

// Sum of N numbers per lane over the warp, the same in all lanes, on the
// integer pipe: every mantissa is shifted to the largest exponent present (55
// or 57 bits below its leading bit, rounded), the integers are added exactly
// and the total is rounded to FP64 once.  A shuffle tree of FP64 additions
// takes 64 cycles of issue and two shuffles per stage, 575 cycles against
// about 200, and rounds at every stage.  Inf, NaN and totals outside the
// normal range take the FP64 tree.
template <int N>
__device__ __forceinline__ double warp_fixed_sum(const double (&x)[N]) {
  constexpr unsigned full = 0xffffffffu;
  constexpr int kUp = N == 1 ? 4 : 2;   // N 2^kUp 2^53 2^5 <= 2^63
  static_assert(N <= 8, "headroom");
  int e[N], em = 0;
  bool neg[N];
  long long q[N];
#pragma unroll
  for (int u = 0; u < N; ++u) {
    q[u] = fixed_parts(x[u], e[u], neg[u]);
    em = max(em, e[u]);
  }
  const int E = (int)__reduce_max_sync(full, (unsigned)em);
  long long a = 0;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int sh = min(E - e[u], 62);
    const long long w = ((q[u] << kUp) + ((1ll << sh) >> 1)) >> sh;
    a += neg[u] ? -w : w;
  }
  const unsigned lo = __reduce_add_sync(full, (unsigned)(a & 0x3ffffff));
  const unsigned mid = __reduce_add_sync(full, (unsigned)((a >> 26) & 0x3ffffff));
  const int top = __reduce_add_sync(full, (int)(a >> 52));
  const long long t = ((long long)top << 52) + ((long long)mid << 26) + (long long)lo;
  const unsigned long long v = t < 0 ? 0ull - (unsigned long long)t : (unsigned long long)t;
  if (v == 0 && E < 0x7ff) return 0.0;
  const int lz = __clzll((long long)v);
  const int be = (63 - lz) + E - 52 - kUp;   // biased exponent of the leading bit
  if (E == 0x7ff || be < 1 || be > 0x7fe) {
    double s = x[0];
#pragma unroll
    for (int u = 1; u < N; ++u) s += x[u];
    return warp_sum(s);
  }
  const unsigned long long nm = v << lz;
  unsigned long long mant = nm >> 11;   // 53 bits with the leading one; round half to even
  const unsigned rem = (unsigned)(nm & 0x7ff);
  mant += rem > 0x400u || (rem == 0x400u && (mant & 1ull)) ? 1ull : 0ull;
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + mant;
  return __longlong_as_double((long long)(bits | (t < 0 ? 0x8000000000000000ull : 0ull)));
}
__device__ __forceinline__ double warp_fixed_sum(double x) {
  const double v[1] = {x};
  return warp_fixed_sum<1>(v);
}

// Words of one block's partials to the next block's: each block writes a
// 128-byte line of its own.  Packed, eight blocks write a line that every
// block polls: 9,800 cycles per reduction over 147 blocks (5,300 over 32)
// against 3,900 (1,900).
constexpr int kRedStride = 8;

// The block's resident state: shared memory (after the column stages, at
// kp.res_off) and this thread's place in it.  Thread t owns slot t of the
// block (warp w holds slice blk_slice[b] + w); local indices are the block's
// own slots, then its halo.
template <class Pol, int R>
struct Resident {
  using VT = typename Pol::VT;
  using BT = typename Pol::BT;
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  const VT* v;               // this lane's first entry
  const unsigned short* ci;  // and its local column index
  unsigned char* x0;         // vectors by exchange parity: own slots, then halo
  double* red;               // [R][32] warps' sums
  unsigned char* chain;      // mixed: rows of slices 16.. of the alpha group, 128 R (AT, BT)
  int sb, ns;                // first slice of the block and their number
  int len;                   // entries of the slice row (0: no slice)
  long long row;             // global row, -1 for padding
  float dl;                  // mixed: diagonal compensation
  bool exported;             // another block references this row
  long long h0;              // halo list of the block
  int nh;
  unsigned long long base, k;   // tag base, current exchange

  __device__ __forceinline__ ulonglong2* words(const KParams& kp) const {
    return kp.res_words + (long long)(k & 1) * kp.n * R;
  }
  __device__ __forceinline__ unsigned char* buf(const KParams& kp) const {
    return x0 + (int)(k & 1) * (kp.res_vec * R * 8);
  }

  __device__ void init(const KParams& kp) {
    extern __shared__ __align__(128) unsigned char dsm[];
    unsigned char* p = dsm + kp.res_off;
    const int nt = blockDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    sb = kp.blk_slice[blockIdx.x];
    const int se = kp.blk_slice[blockIdx.x + 1];
    ns = se - sb;
    const long long e0 = kp.slice_off[sb];
    const int ne = (int)(kp.slice_off[se] - e0);
    VT* sv = reinterpret_cast<VT*>(p);
    p += kp.res_ent * sizeof(VT);
    unsigned short* sc = reinterpret_cast<unsigned short*>(p);
    p += kp.res_ent * sizeof(unsigned short);
    x0 = p;
    p += 2 * (kp.res_vec * R * 8);
    red = reinterpret_cast<double*>(p);
    chain = p + 32 * R * sizeof(double);
    const VT* gv = reinterpret_cast<const VT*>(kp.val) + e0;
    for (int i = tid; i < ne; i += nt) {
      sv[i] = gv[i];
      sc[i] = kp.res_col[e0 + i];
    }
    const long long s = sb + warp;
    const bool act = warp < ns;
    const int o = act ? (int)(kp.slice_off[s] - e0) : 0;
    len = act ? (int)(kp.slice_off[s + 1] - kp.slice_off[s]) >> 5 : 0;
    v = sv + o + lane;
    ci = sc + o + lane;
    row = act && s * 32 + lane < kp.n ? s * 32 + lane : -1;
    dl = 0.f;
    if (Pol::kMixed && act && kp.dlo) dl = kp.dlo[s * 32 + lane];
    exported = row >= 0 && kp.res_exp[row] != 0;
    h0 = kp.halo_ptr[blockIdx.x];
    nh = (int)(kp.halo_ptr[blockIdx.x + 1] - h0);
    // padding slots are referenced by padding entries: finite from the start
    for (int q = 0; q < 2; ++q)
      for (int r = 0; r < R; ++r) reinterpret_cast<double*>(x0)[(q * kp.res_vec + tid) * R + r] = 0.0;
    base = kp.epoch << 32;
    k = 0;
    __syncthreads();
  }

  // Posts this thread's row of the next exchange: into the block's vector and,
  // where another block reads it, as words.
  template <class XT>
  __device__ __forceinline__ void post(const KParams& kp, const XT (&x)[R]) {
    ++k;
    if (row < 0) return;
    VecIO<R>::st(reinterpret_cast<XT*>(buf(kp)) + threadIdx.x * R, x);
    if (exported) {
      ulonglong2* w = words(kp) + row * R;
#pragma unroll
      for (int r = 0; r < R; ++r) st_word(w + r, to_bits(x[r]), base + k);
    }
  }

  // Reads the halo of the current exchange with threads t0, t0 + step, ...
  template <class XT>
  __device__ __forceinline__ bool halo(const KParams& kp, int t0, int step) const {
    XT* x = reinterpret_cast<XT*>(buf(kp)) + (long long)blockDim.x * R;
    const ulonglong2* w = words(kp);
    bool ok = true;
    for (int t = t0; t < nh * R && ok; t += step) {
      const int i = t / R, r = t - i * R;
      unsigned long long d;
      ok = poll_word(kp, w + (long long)__ldg(kp.halo_rows + h0 + i) * R + r, base + k, d);
      if (ok) from_bits(d, x[t]);
    }
    return ok;
  }

  // The row's sum over the stored entries, in the general path's order.
  template <class XT>
  __device__ __forceinline__ void spmv(const KParams& kp, AT (&acc)[R]) const {
    const XT* x = reinterpret_cast<const XT*>(buf(kp));
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::zero();
    if (Pol::kMixed && len > 0) {
      XT xv[R];
      VecIO<R>::ld(x + (int)ci[0] * R, xv);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], dl, xv[r]);
    }
#pragma unroll 4
    for (int jj = 0; jj < len; ++jj) {
      XT xv[R];
      const VT a = v[jj * 32];
      VecIO<R>::ld(x + (int)ci[jj * 32] * R, xv);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = Pol::acc(acc[r], a, xv[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Pol::norm(acc[r]);
  }

  __device__ __forceinline__ static double part_double(double x) { return x; }
  __device__ __forceinline__ static double part_double(ff x) { return ff_to_double(x); }

  // Sums part[r] over all blocks and calls fin(r, total) with one full warp
  // per right-hand side (pre(r) while the others' words are under way); the
  // other warps run other() meanwhile.  half: 0 alpha, 1 beta.  Ends with a
  // block barrier; false when a wait failed.
  template <class PT, class Pre, class Fin, class Other>
  __device__ __forceinline__ bool reduce(const KParams& kp, const Ctx& c, const PT (&part)[R], int half,
                                         unsigned long long tag, Pre&& pre, Fin&& fin, Other&& other) const {
    bool ok = true;
    // Mixed: red[r][q] is the sum of the general path's warp q of this block:
    // for alpha the block's own slices (a second round already added), for beta
    // slice 16 b + q, which another block may hold.
    const int slice = sb + c.warp(), first = 16 * c.b();
    const bool act = c.warp() < ns;
    if constexpr (Pol::kMixed) {
      double v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = part_double(part[r]);
      const double s = warp_sum_packed<R>(v);
      if (act && (c.lane() & (32 / R - 1)) == 0) {
        const int r = packed_index<R>(c.lane());
        if (half == 0) {
          if (c.warp() < 16) red[r * 32 + c.warp()] = s;
        } else if ((slice >> 4) == c.b()) {
          red[r * 32 + (slice & 15)] = s;
        } else {
          st_word(kp.res_slice + slice * kRedStride + r, to_bits(s), tag);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double s = warp_fixed_sum(part[r]);
        if (c.lane() == 0) red[r * 32 + c.warp()] = s;
      }
    }
    __syncthreads();
    for (int r = c.warp(); r < R; r += c.nw()) {
      double s;
      if constexpr (Pol::kMixed) {
        const int count = half ? (int)min(16ll, kp.nslices - first) : min(ns, 16);
        double x = 0.0;
        if (c.lane() < count) {
          const int q = first + c.lane();
          if (half && (q < sb || q >= sb + ns)) {
            unsigned long long d = 0ull;
            ok = poll_word(kp, kp.res_slice + q * kRedStride + r, tag, d);
            x = __longlong_as_double((long long)d);
          } else {
            x = red[r * 32 + c.lane()];
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        s = warp_sum(x);
      } else {
        s = warp_fixed_sum(c.lane() < c.nw() ? red[r * 32 + c.lane()] : 0.0);
      }
      ulonglong2* w = kp.res_red + half * c.G * kRedStride + r;
      if (c.lane() == 0) st_word(w + c.b() * kRedStride, to_bits(s), tag);
      pre(r);
      double t = 0.0;   // mixed: this lane's blocks in order
      for (int b0 = 0; b0 < c.G && ok; b0 += 32 * 5) {
        // five words in flight per lane
        unsigned long long d[5], g[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) {
          const int b = b0 + 32 * u + c.lane();
          d[u] = 0ull;
          g[u] = tag;
          if (b < c.G) ld_word(w + b * kRedStride, d[u], g[u]);
        }
        double x[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) {
          if (g[u] != tag && ok) ok = poll_word(kp, w + (b0 + 32 * u + c.lane()) * kRedStride, tag, d[u]);
          x[u] = __longlong_as_double((long long)d[u]);
        }
        ok = __all_sync(0xffffffffu, ok);
        if constexpr (Pol::kMixed) {
#pragma unroll
          for (int u = 0; u < 5; ++u)
            if (b0 + 32 * u + c.lane() < c.G) t += x[u];
        } else {
          const double q = warp_fixed_sum<5>(x);
          t = b0 == 0 ? q : t + q;
        }
      }
      if (!ok) break;
      fin(r, Pol::kMixed ? warp_sum(t) : t);
    }
    if (ok) ok = other();
    return !__syncthreads_or(!ok);
  }
};

// build_subspace.cu:5-89 as phase_lanczos, with the same operations per row in
// the same order.
template <class Pol, int R>
__device__ bool phase_lanczos_resident(const KParams& kp, const Ctx& c) {
  using BT = typename Pol::BT;
  using HT = typename Pol::HT;
  using AT = typename Pol::AT;
  const long long n = kp.n;
  const int m = kp.m, d = kp.d;
  __shared__ LanczosScalars<Pol, R> sh;
  Resident<Pol, R> rs;
  rs.init(kp);
  BT* const V = reinterpret_cast<BT*>(kp.V);
  const LanczosOut out{kp.aabb, kp.meff, c.b() == 0 && c.lane() == 0};
  // (a block of one slice has 32 threads, a polynomial up to 33 coefficients)
  for (int i = c.tid(); i <= d; i += c.nt()) sh.gam[i] = kp.gamma[i];
  auto read_halo = [&]() -> bool {
    const int w0 = c.nw() > R ? R : 0;   // the warps that do not reduce, or all
    if (c.warp() < w0) return true;
    return rs.template halo<BT>(kp, c.tid() - 32 * w0, c.nt() - 32 * w0);
  };

  BT sv[R], wp[R];   // w_j and w_{j-1}
  {
    double u[R], p[R];
#pragma unroll
    for (int r = 0; r < R; ++r) { u[r] = 0.0; wp[r] = (BT)0; }
    if (rs.row >= 0) VecIO<R>::ld(kp.U + rs.row * R, u);
#pragma unroll
    for (int r = 0; r < R; ++r) { sv[r] = (BT)u[r]; p[r] = u[r] * u[r]; }
    rs.post(kp, sv);
    if (!rs.reduce(kp, c, p, 1, rs.base + 1, [](int) {},
                   [&](int r, double t) { step_beta<Pol, R>(sh, kp, out, r, t, -1); }, read_halo))
      return false;
  }
  for (int j = 0; j < m; ++j) {
    AT w[R];
    rs.template spmv<BT>(kp, w);
    if (rs.row >= 0) {
      BT v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = Pol::scale_to_b(sv[r], sh.rb[r]);
      VecIO<R>::st(V + ((long long)j * n + rs.row) * R, v);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = Pol::mul(w[r], sh.sc[r]);
    // Horner passes 1..d: u = gamma_h v_j + A u
    for (int h = 1; h <= d; ++h) {
      HT u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = Pol::to_h(Pol::add_mul(w[r], sh.gr[h][r], sv[r]));
      rs.post(kp, u);
      if (__syncthreads_or(!rs.template halo<HT>(kp, c.tid(), c.nt()))) return false;
      rs.template spmv<HT>(kp, w);
    }
    AT p[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (j > 0) w[r] = Pol::sub_mul(w[r], sh.bj[r], wp[r]);
      p[r] = rs.row >= 0 ? Pol::dot(Pol::zero(), w[r], sv[r]) : Pol::zero();
    }
    if constexpr (Pol::kMixed) {
      // the general path's warps take slices 16.. of a block as a second round,
      // accumulated onto their first
      if (rs.ns > 16) {
        AT* const cw = reinterpret_cast<AT*>(rs.chain);
        BT* const cv = reinterpret_cast<BT*>(cw + 128 * R);
        const int q = (c.warp() - 16) * 32 + c.lane();
        if (c.warp() >= 16) {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            cw[q * R + r] = rs.row >= 0 ? w[r] : Pol::zero();
            cv[q * R + r] = rs.row >= 0 ? sv[r] : (BT)0;
          }
        }
        __syncthreads();
        if (c.warp() + 16 < rs.ns) {
#pragma unroll
          for (int r = 0; r < R; ++r) p[r] = Pol::dot(p[r], cw[c.tid() * R + r], cv[c.tid() * R + r]);
        }
      }
    }
    if (!rs.reduce(kp, c, p, 0, rs.base + 2 + 2 * (unsigned long long)j, [](int) {},
                   [&](int r, double t) { step_alpha<Pol, R>(sh, r, t); }, []() { return true; }))
      return false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const AT x = Pol::sub_mul(w[r], sh.al[r], sv[r]);
      wp[r] = sv[r];
      sv[r] = Pol::to_b(x);
      p[r] = rs.row >= 0 ? Pol::dot_self(Pol::zero(), x) : Pol::zero();
    }
    rs.post(kp, sv);
    if (!rs.reduce(kp, c, p, 1, rs.base + 3 + 2 * (unsigned long long)j, [&](int r) { step_bound<Pol, R>(sh, kp, out, r, j); },
                   [&](int r, double t) { step_beta<Pol, R>(sh, kp, out, r, t, j); }, read_halo))
      return false;
    bool all = true;
#pragma unroll
    for (int r = 0; r < R; ++r) all = all && sh.broken[r];
    if (all) break;
  }
  return true;
}

}  // namespace gm
