// Host side of the diagonal slices: which slices of a matrix are diagonals.
#pragma once

#include <algorithm>
#include <vector>

namespace gm {

// Ints of the kernels' table of patterns: patterns per problem times kLen.
constexpr int kDiaTable = 512;

// Diagonal slices.  A full slice is one when the union of its rows' offsets
// (column minus row) is no longer than its longest row and every entry a row
// lacks would still fall inside its problem: the slice then stores the union,
// with zeros, and its columns follow from the row.  The entries keep the rows'
// (ascending) order, the diagonal first where diag_first asks for it, and the
// slice its length, so neither the sums nor the partition change.  Offsets are
// at most reach: the kernels multiply them by the number of right-hand sides in
// 32 bits (in 64 the four-column FP64 kernel spills: 500^2 2,306 -> 2,354 us).
struct DiaSlices {
  static constexpr int kLen = 16;                      // offsets per pattern, at most
  std::vector<int> off;                                // [pattern][kLen], problem after problem
  std::vector<int> len;                                // [pattern]
  std::vector<int> pat0;                               // [problem + 1] its first pattern
  std::vector<short> pat;                              // [slice] within its problem, -1: ordinary
  long long count = 0;
};
template <class Csr>
DiaSlices find_dia(const Csr& A, const std::vector<long long>& prow0, const std::vector<long long>& pslice0,
                   bool diag_first, int reach) {
  DiaSlices D;
  const int np = (int)prow0.size() - 1;
  D.pat.assign(pslice0[np], -1);
  const int max_pat = kDiaTable / DiaSlices::kLen;
  D.pat0.assign(1, 0);
  for (int p = 0; p < np; ++p) {
    const int base = D.pat0[p];
    int last = -1;
    for (long long s = pslice0[p]; s < pslice0[p + 1]; ++s) {
      const long long r0 = prow0[p] + 32 * (s - pslice0[p]);
      if (r0 + 32 > prow0[p + 1]) continue;
      int u[DiaSlices::kLen], nu = 0, longest = 0;
      bool ok = true;
      if (diag_first) u[nu++] = 0;
      for (long long r = r0; r < r0 + 32 && ok; ++r) {
        longest = std::max<int>(longest, (int)std::min<long long>(A.ptr[r + 1] - A.ptr[r], 1000));
        if (A.ptr[r + 1] - A.ptr[r] == nu) {
          // most rows have the offsets of the one before
          const int* c = A.col.data() + A.ptr[r];
          int q = 0;
          while (q < nu && c[q] - (int)r == u[q]) ++q;
          if (q == nu) continue;
        }
        int at = 0;
        long long before = -1;
        bool has_diag = false;
        for (long long t = A.ptr[r]; t < A.ptr[r + 1] && ok; ++t) {
          const int o = A.col[t] - (int)r;
          ok = A.col[t] > before;
          before = A.col[t];
          has_diag = has_diag || o == 0;
          while (at < nu && u[at] < o) ++at;
          if (at < nu && u[at] == o) continue;
          if (nu == DiaSlices::kLen) { ok = false; break; }
          for (int q = nu; q > at; --q) u[q] = u[q - 1];
          u[at] = o;
          ++nu;
        }
        if (diag_first && !has_diag) ok = false;   // (its explicit zero diagonal comes first)
      }
      if (!ok || nu == 0 || nu > longest) continue;
      // every offset of every row inside the problem
      if (r0 + u[0] < prow0[p] || r0 + 31 + u[nu - 1] >= prow0[p + 1]) continue;
      if (u[0] < -reach || u[nu - 1] > reach) continue;
      if (diag_first) {
        int z = 0;
        while (u[z] != 0) ++z;
        for (; z > 0; --z) u[z] = u[z - 1];
        u[0] = 0;
      }
      auto same = [&](int q) { return D.len[q] == nu && std::equal(u, u + nu, D.off.begin() + q * DiaSlices::kLen); };
      int id = last >= 0 && same(last) ? last : -1;
      for (int q = base; id < 0 && q < (int)D.len.size(); ++q)
        if (same(q)) id = q;
      if (id < 0) {
        if ((int)D.len.size() - base == max_pat) continue;
        id = (int)D.len.size();
        D.len.push_back(nu);
        D.off.insert(D.off.end(), u, u + nu);
        D.off.resize((size_t)(id + 1) * DiaSlices::kLen, 0);
      }
      D.pat[s] = (short)(id - base);
      last = id;
      ++D.count;
    }
    D.pat0.push_back((int)D.len.size());
  }
  return D;
}

}  // namespace gm
