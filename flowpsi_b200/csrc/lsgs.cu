// lsgs.cu -- line symmetric Gauss-Seidel (linearSolverLSGS.loci) on the GPU.
//
// Lines are solved as batched block-tridiagonal systems (block Thomas
// algorithm, one thread per line, 32 lines per group stored position-major
// so that the group's threads read coalesced rows).  Lines are coloured so
// that the lines of one colour are independent; a sweep runs the colours in
// order (forward) and in reverse (backward).  The iteration is the
// reference's solve loop (linearSolverLSGS.loci:1692-1954):
//   * start: every line solved with its own right-hand side B (:1708-1728);
//   * per iteration: forward sweep, backward sweep, relaxation
//     X = w X + (1-w) X_t with X_t the iterate before the backward line solve
//     (:1868-1874), residual ||X - X_t||, w *= 1/rel when rel > 1 (:1935),
//     stop on the absolute or relative tolerance (:1944-1947).
// The stopping test runs on the device (no host round trip per iteration);
// once it fires, the remaining launches of the solve return at entry.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "fpsi_internal.h"
#include "kernels.cuh"
#include "line_quotient.cuh"
#include "pdl.cuh"

namespace fpsi {

// ---------------------------------------------------------------------------
// host: lines, colours, groups, roles of the cell's faces
// ---------------------------------------------------------------------------
namespace {

// default lines: link cells that are mutually among each other's two
// strongest couplings, measured geometrically by area / centre distance,
// keeping a second link only when it is within a factor 25 of the first
// (the test of linearSolverLSGS.loci:620).
std::vector<std::vector<int32_t>> default_lines(const HostMesh& H) {
  const int64_t nc = H.nc;
  std::vector<std::array<int32_t, 2>> best(nc, {-1, -1});
  std::vector<std::array<double, 2>> bw(nc, {0.0, 0.0});
  for (int64_t c = 0; c < nc; ++c) {
    for (int32_t e = H.cf_off[c]; e < H.cf_off[c + 1]; ++e) {
      const int64_t f = H.cf[e] >> 1;
      if (H.cr[f] < 0) continue;
      const int32_t o = (H.cf[e] & 1) ? H.cl[f] : H.cr[f];
      double d2 = 0;
      for (int k = 0; k < 3; ++k) {
        const double d = H.rL[3 * f + k] - H.rR[3 * f + k];
        d2 += d * d;
      }
      const double w = H.area[f] / std::sqrt(d2);
      if (w > bw[c][0]) {
        bw[c][1] = bw[c][0], best[c][1] = best[c][0];
        bw[c][0] = w, best[c][0] = o;
      } else if (w > bw[c][1]) {
        bw[c][1] = w, best[c][1] = o;
      }
    }
    if (best[c][1] >= 0 && bw[c][1] * 25.0 <= bw[c][0]) best[c][1] = -1;
  }
  auto mutual = [&](int32_t a, int32_t b) {
    return best[b][0] == a || best[b][1] == a;
  };
  std::vector<std::array<int32_t, 2>> link(nc, {-1, -1});
  for (int64_t c = 0; c < nc; ++c)
    for (int s = 0; s < 2; ++s) {
      const int32_t o = best[c][s];
      if (o >= 0 && mutual(int32_t(c), o)) link[c][s] = o;
    }
  std::vector<char> seen(nc, 0);
  std::vector<std::vector<int32_t>> lines;
  auto degree = [&](int64_t c) { return (link[c][0] >= 0) + (link[c][1] >= 0); };
  // paths from their ends first, then what is left (cycles) cut anywhere
  for (int pass = 0; pass < 2; ++pass)
    for (int64_t s0 = 0; s0 < nc; ++s0) {
      if (seen[s0] || (pass == 0 && degree(s0) > 1)) continue;
      std::vector<int32_t> L;
      int32_t prev = -1, cur = int32_t(s0);
      while (cur >= 0 && !seen[cur]) {
        seen[cur] = 1;
        L.push_back(cur);
        int32_t nxt = -1;
        for (int s = 0; s < 2; ++s)
          if (link[cur][s] >= 0 && link[cur][s] != prev && !seen[link[cur][s]]) {
            nxt = link[cur][s];
            break;
          }
        prev = cur;
        cur = nxt;
      }
      lines.push_back(std::move(L));
    }
  return lines;
}

}  // namespace

int build_lines(fpsi_ctx* x, const std::vector<std::vector<int32_t>>* given) {
  const HostMesh& H = x->H;
  LineLayout& Y = x->LY;
  const int64_t nc = H.nc;
  std::vector<std::vector<int32_t>> lines = given ? *given : default_lines(H);
  // cells not covered become single-cell lines
  std::vector<int32_t> line_of(nc, -1), pos(nc, -1);
  for (size_t l = 0; l < lines.size(); ++l)
    for (size_t p = 0; p < lines[l].size(); ++p) {
      const int32_t c = lines[l][p];
      if (c < 0 || c >= nc || line_of[c] >= 0) {
        set_error("lines: cell %d missing or repeated", c);
        return FPSI_E_INVALID;
      }
      line_of[c] = int32_t(l), pos[c] = int32_t(p);
    }
  for (int64_t c = 0; c < nc; ++c)
    if (line_of[c] < 0) {
      line_of[c] = int32_t(lines.size()), pos[c] = 0;
      lines.push_back({int32_t(c)});
    }
  const int64_t nl = int64_t(lines.size());
  // consecutive cells of a line must share an interior face
  auto coupled = [&](int32_t a, int32_t b) {
    for (int32_t e = H.cf_off[a]; e < H.cf_off[a + 1]; ++e) {
      const int64_t f = H.cf[e] >> 1;
      if (H.cr[f] < 0) continue;
      if (((H.cf[e] & 1) ? H.cl[f] : H.cr[f]) == b) return true;
    }
    return false;
  };
  for (const auto& L : lines)
    for (size_t p = 1; p < L.size(); ++p)
      if (!coupled(L[p - 1], L[p])) {
        set_error("lines: consecutive cells %d and %d share no face", L[p - 1], L[p]);
        return FPSI_E_INVALID;
      }
  // greedy colouring of the line graph in line order
  std::vector<int32_t> lcol(nl, -1);
  std::vector<int64_t> mark;
  int ncol = 0;
  for (int64_t l = 0; l < nl; ++l) {
    for (int32_t c : lines[l])
      for (int32_t e = H.cf_off[c]; e < H.cf_off[c + 1]; ++e) {
        const int64_t f = H.cf[e] >> 1;
        if (H.cr[f] < 0) continue;
        const int32_t o = (H.cf[e] & 1) ? H.cl[f] : H.cr[f];
        const int32_t ol = line_of[o];
        if (ol == l || lcol[ol] < 0) continue;
        if (lcol[ol] >= int32_t(mark.size())) mark.resize(lcol[ol] + 1, -1);
        mark[lcol[ol]] = l;
      }
    int k = 0;
    while (k < int(mark.size()) && mark[k] == l) ++k;
    lcol[l] = k;
    ncol = std::max(ncol, k + 1);
  }
  // groups of 32 lines per colour, lines ordered by their first cell
  Y = LineLayout();
  Y.nlines = nl;
  Y.ncolours = ncol;
  Y.col_goff.assign(ncol + 1, 0);
  Y.t_of.assign(nc, -1);
  Y.line_of = line_of;
  Y.line_colour = lcol;
  int64_t row = 0;
  for (int k = 0; k < ncol; ++k) {
    std::vector<int32_t> ls;
    for (int64_t l = 0; l < nl; ++l)
      if (lcol[l] == k) ls.push_back(int32_t(l));
    std::sort(ls.begin(), ls.end(), [&](int32_t a, int32_t b) { return lines[a][0] < lines[b][0]; });
    Y.col_goff[k] = Y.ngroups;
    for (size_t g0 = 0; g0 < ls.size(); g0 += 32) {
      int32_t glen = 0;
      for (size_t j = g0; j < std::min(ls.size(), g0 + 32); ++j)
        glen = std::max<int32_t>(glen, int32_t(lines[ls[j]].size()));
      Y.grp_row0.push_back(row);
      Y.grp_len.push_back(glen);
      for (int lane = 0; lane < 32; ++lane) {
        const size_t j = g0 + lane;
        if (j >= ls.size()) {
          Y.lane_len.push_back(0);
          continue;
        }
        const auto& L = lines[ls[j]];
        Y.lane_len.push_back(int32_t(L.size()));
        for (size_t p = 0; p < L.size(); ++p) Y.t_of[L[p]] = int32_t((row + p) * 32 + lane);
      }
      row += glen;
      Y.ngroups++;
    }
  }
  Y.col_goff[ncol] = Y.ngroups;
  Y.nrows = row;
  for (int32_t n : Y.grp_len) Y.max_len = std::max(Y.max_len, n);
  if (row * 32 >= (int64_t(1) << 31)) {
    set_error("lines: padded size too large");
    return FPSI_E_INVALID;
  }
  Y.c_of_t.assign(size_t(row * 32), -1);
  for (int64_t c = 0; c < nc; ++c) Y.c_of_t[Y.t_of[c]] = int32_t(c);
  // roles of the cell's faces and outer slots
  Y.role.assign(H.cf.size(), 0);
  int mout = 0;
  std::vector<int32_t> nout(nc, 0);
  for (int64_t c = 0; c < nc; ++c) {
    const auto& L = lines[line_of[c]];
    const int32_t p = pos[c];
    const int32_t prv = p > 0 ? L[p - 1] : -1;
    const int32_t nxt = p + 1 < int32_t(L.size()) ? L[p + 1] : -1;
    bool hp = false, hn = false;
    for (int32_t e = H.cf_off[c]; e < H.cf_off[c + 1]; ++e) {
      const int64_t f = H.cf[e] >> 1;
      if (H.cr[f] < 0) continue;
      const int32_t o = (H.cf[e] & 1) ? H.cl[f] : H.cr[f];
      if (o == prv && !hp) {
        Y.role[e] = 1, hp = true;
      } else if (o == nxt && !hn) {
        Y.role[e] = 2, hn = true;
      } else {
        if (nout[c] > 120) {
          set_error("lines: cell %lld has too many outer couplings", (long long)c);
          return FPSI_E_INVALID;
        }
        Y.role[e] = int8_t(3 + nout[c]++);
      }
    }
    mout = std::max(mout, nout[c]);
  }
  Y.mout = std::max(mout, 1);
  Y.onbr.assign(size_t(row) * Y.mout * 32, -1);
  for (int64_t c = 0; c < nc; ++c) {
    const int64_t t = Y.t_of[c], r = t / 32, lane = t % 32;
    for (int32_t e = H.cf_off[c]; e < H.cf_off[c + 1]; ++e) {
      if (Y.role[e] < 3) continue;
      const int64_t f = H.cf[e] >> 1;
      const int32_t o = (H.cf[e] & 1) ? H.cl[f] : H.cr[f];
      Y.onbr[(r * Y.mout + (Y.role[e] - 3)) * 32 + lane] = Y.t_of[o];
    }
  }
  Y.built = true;
  return FPSI_OK;
}

// ---------------------------------------------------------------------------
// device
// ---------------------------------------------------------------------------
namespace dev {

struct LineView {
  const int32_t* t_of;       // RCM cell -> t
  const int8_t* role;        // per cf entry
  const int32_t* onbr;       // [(row*mout+s)*32+lane]
  const int32_t* lane_len;   // [g*32+lane]
  const int64_t* grp_row0;
  int mout;
};

struct LsgsCtl {
  double w, zero, resid;
  int32_t iter, done;
};

// A group row's blocks (D, L, U): entries 0..23 as six quads, [quad][32
// lanes][4], then entry 24 [32 lanes]: a lane moves a block in seven accesses,
// each contiguous over the warp.
template <class T>
struct alignas(4 * sizeof(T) < 16 ? 4 * sizeof(T) : 16) Quad {
  T v[4];
};
template <class T>
__device__ __forceinline__ void block_load(const T* row, int lane, T* b) {
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const Quad<T> w = *reinterpret_cast<const Quad<T>*>(row + (q * 32 + lane) * 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[4 * q + i] = w.v[i];
  }
  b[24] = row[24 * 32 + lane];
}
template <class T>
__device__ __forceinline__ void block_store(T* row, int lane, const T* b) {
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    Quad<T> w;
#pragma unroll
    for (int i = 0; i < 4; ++i) w.v[i] = b[4 * q + i];
    *reinterpret_cast<Quad<T>*>(row + (q * 32 + lane) * 4) = w;
  }
  row[24 * 32 + lane] = b[24];
}

// A row of lD: the block, then (once factored) the reciprocals of its five
// pivots, [5][32 lanes]; NaN for a pivot outside the range in which
// quotient() is exact.
constexpr int DROW = 30 * 32;

// Gather the line-ordered system: raw diagonal block, in-line couplings
// (row p to p-1 in L, to p+1 in U), outer couplings and B.  The coupling of
// row c to neighbour n through face f is fjm_f when c = cl(f), -fjp_f when
// c = cr(f) (solverLinearSystem.loci:57-77).  One thread per line slot t,
// so that the 32 lanes of a row store 32 consecutive words of every stream.
//
// What is not written here has to stay as alloc_lsgs cleared it.  The line
// solves walk a group's rows for all 32 lanes and have no test at a line's
// ends: U of a line's last row, which they multiply with the zero that starts
// the back substitution, must be zero (and so finite), L of a first row is
// copied along; D, L and U of padding rows are computed on, with the results
// dropped.  Nothing else may use these arrays.  The first coupling of a slot
// without any (lF) is read ahead and dropped, whatever it holds.
template <class TB, class TD>
__global__ void k_lsgs_scatter(int64_t nt, const int32_t* __restrict__ c_of_t,
                               const int32_t* __restrict__ cf_off, const int32_t* __restrict__ cf,
                               LineView V, const TB* D, const TB* fjp,
                               const TB* fjm, const double* src,
                               TD* __restrict__ lD, TB* __restrict__ lL, TB* __restrict__ lU,
                               TB* __restrict__ lF, TB* __restrict__ lB) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (t >= nt) return;
  const int64_t c = c_of_t[t];
  if (c < 0) return;
  const int64_t r = t >> 5, lane = t & 31;
  TD d[25];
#pragma unroll
  for (int e = 0; e < 25; ++e) d[e] = TD(D[25 * c + e]);
  block_store<TD>(lD + r * DROW, int(lane), d);
#pragma unroll
  for (int k = 0; k < 5; ++k) lB[(r * 5 + k) * 32 + lane] = TB(src[5 * c + k]);
  for (int32_t e = cf_off[c]; e < cf_off[c + 1]; ++e) {
    const int ro = V.role[e];
    if (ro == 0) continue;
    const int32_t ent = cf[e];
    const int64_t f = ent >> 1;
    const bool neg = ent & 1;
    const TB* A = neg ? fjp + 25 * f : fjm + 25 * f;
    TB b[25];
#pragma unroll
    for (int k = 0; k < 25; ++k) b[k] = neg ? TB(-A[k]) : A[k];
    if (ro < 3) {
      block_store<TB>((ro == 1 ? lL : lU) + r * 25 * 32, int(lane), b);
    } else {
      TB* o = lF + (r * V.mout + (ro - 3)) * 25 * 32 + lane;
#pragma unroll
      for (int k = 0; k < 25; ++k) o[k * 32] = b[k];
    }
  }
}

// 5x5 LU without pivoting (decompose_lu of linearSolverLSGS.loci:1474) and
// its solve, on a block held in registers
template <class T>
__device__ __forceinline__ bool lu5_nopiv(T* A) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const T d = A[5 * k + k];
    if (d == T(0)) ok = false;
#pragma unroll
    for (int i = k + 1; i < 5; ++i) {
      A[5 * i + k] /= d;
#pragma unroll
      for (int j = k + 1; j < 5; ++j) A[5 * i + j] -= A[5 * i + k] * A[5 * k + j];
    }
  }
  return ok;
}
template <class T, class TV>
__device__ __forceinline__ void lu5_nopiv_solve(const T* A, TV* y) {
#pragma unroll
  for (int i = 1; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < i; ++j) y[i] -= TV(A[5 * i + j]) * y[j];
#pragma unroll
  for (int i = 4; i >= 0; --i) {
#pragma unroll
    for (int j = i + 1; j < 5; ++j) y[i] -= TV(A[5 * i + j]) * y[j];
    y[i] /= TV(A[5 * i + i]);
  }
}

// lu5_nopiv_solve with the pivots' reciprocals r[5]; key: of the dividends
template <class T>
__device__ __forceinline__ void lu5_recip_solve(const T* A, const T* r, T* y, uint32_t& key) {
#pragma unroll
  for (int i = 1; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < i; ++j) y[i] -= A[5 * i + j] * y[j];
#pragma unroll
  for (int i = 4; i >= 0; --i) {
#pragma unroll
    for (int j = i + 1; j < 5; ++j) y[i] -= A[5 * i + j] * y[j];
    key = key_min(key, y[i]);
    y[i] = quotient<T>(y[i], A[6 * i], r[i]);
  }
}

// lu5_nopiv that also gives the pivots' reciprocals r[5] (NaN outside the
// range of quotient()); key: of the dividends
template <class T>
__device__ __forceinline__ void lu5_nopiv_recip(T* A, T* r, uint32_t& key) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const T d = A[6 * k];
    r[k] = pivot_ok(d) ? T(1) / d : T(nanf(""));
#pragma unroll
    for (int i = k + 1; i < 5; ++i) {
      key = key_min(key, A[5 * i + k]);
      A[5 * i + k] = quotient<T>(A[5 * i + k], d, r[k]);
#pragma unroll
      for (int j = k + 1; j < 5; ++j) A[5 * i + j] -= A[5 * i + k] * A[5 * k + j];
    }
  }
}

// block Thomas preprocessing (preprocessLine, linearSolverLSGS.loci:1465-1495):
// D'_0 = D_0, D'_p = D_p - L_p D'_{p-1}^{-1} U_{p-1}; each D' factored in
// place.  As in the reference the Schur product is formed with real_fj
// (TB) intermediates.
//
// A serial chain per line with less than a warp per SM, so a row's
// instructions set it, and most of them were its 40 divisions.  Five remain
// (the pivots' reciprocals, which the solves need as well); the others are
// quotient()s.  A row whose operands leave their range, or that comes out
// not finite, is done again with divisions.  262,144 cells in rows of 64:
// 134 -> 70 us MIXED; 24,576 cells in rows of 32: 114 -> 78 us REF, 109 -> 84 us
// FP64 (whose next row's blocks do not fit beside this one's).  The FP64 forms
// spend 2 to 15 us of 84 to 226 on telling the smallest subnormal dividends from
// zero (line_quotient.cuh).
template <class TB, class TD>
__global__ void k_lsgs_prep(int64_t ngroups, LineView V, TD* __restrict__ lD,
                            const TB* lL, const TB* lU,
                            int32_t* __restrict__ err) {
  const int64_t gl = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (gl >= ngroups * 32) return;
  const int64_t g = gl >> 5, lane = gl & 31;
  const int len = V.lane_len[gl];
  const int64_t r0 = V.grp_row0[g];
  TD prev[25], rp[5];  // the row before: its factors and their pivots' reciprocals
  constexpr bool AHEAD = sizeof(TD) == 4;  // the next row's blocks fit in registers
  struct Blocks {
    TD D[25];
    TB L[25], U[25];
  } nx;
  auto load = [&](int p, Blocks& w) {
    const int64_t r = r0 + p;
    block_load<TD>(lD + r * DROW, int(lane), w.D);
    if (p > 0) {
      block_load<TB>(lL + r * 25 * 32, int(lane), w.L);
      block_load<TB>(lU + (r - 1) * 25 * 32, int(lane), w.U);
    }
  };
  // row p from its blocks; whether the result stands
  auto row = [&](int p, Blocks& w, bool exact, TD* rn) {
    TD* Dp = w.D;
    uint32_t key = ~0u;
    TD chk = TD(0);  // stays 0 while everything is finite
    if (p > 0) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        TD v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) v[k] = TD(w.U[5 * k + j]);
        if (exact)
          lu5_nopiv_solve<TD, TD>(prev, v);
        else
          lu5_recip_solve<TD>(prev, rp, v, key);
        TB tt[5], z[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) chk += v[k] * TD(0), tt[k] = TB(v[k]), z[k] = TB(0);
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
          for (int m = 0; m < 5; ++m) z[k] += w.L[5 * k + m] * tt[m];
#pragma unroll
        for (int k = 0; k < 5; ++k) Dp[5 * k + j] -= TD(z[k]);
      }
    }
    if (exact) {
      if (!lu5_nopiv<TD>(Dp)) atomicOr(err, 2);
#pragma unroll
      for (int k = 0; k < 5; ++k) rn[k] = pivot_ok(Dp[6 * k]) ? TD(1) / Dp[6 * k] : TD(nanf(""));
      return true;
    }
    lu5_nopiv_recip<TD>(Dp, rn, key);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = k + 1; i < 5; ++i) chk += Dp[5 * i + k] * TD(0);
    // the last pivot divides nothing in its own row but must not be zero
    return chk == TD(0) && !tiny<TD>(key) && Dp[24] != TD(0);
  };
  if (AHEAD && len > 0) load(0, nx);
  for (int p = 0; p < len; ++p) {
    const int64_t r = r0 + p;
    Blocks w;
    if (AHEAD) {
      w = nx;
      if (p + 1 < len) load(p + 1, nx);
    } else {
      load(p, w);
    }
    TD rn[5];
    if (!row(p, w, false, rn)) {
      load(p, w);  // its own block is still the raw one
      row(p, w, true, rn);
    }
    block_store<TD>(lD + r * DROW, int(lane), w.D);
#pragma unroll
    for (int k = 0; k < 5; ++k) lD[r * DROW + (25 + k) * 32 + lane] = rn[k];
#pragma unroll
    for (int e = 0; e < 25; ++e) prev[e] = w.D[e];
#pragma unroll
    for (int k = 0; k < 5; ++k) rp[k] = rn[k];
  }
}

// right-hand side of the rows of one colour: B - sum_outer F x_outer; xt (may
// be null) keeps the rows' own iterate for the relaxation, before the line
// solve that follows overwrites it
// The system is complete before a solve's first launch, so B, the neighbour
// ids and the first coupling are read before the wait for the line solve
// whose iterate the rows take.
template <class TB, class TX>
__global__ void k_lsgs_rhs(int64_t row_begin, int64_t nrows, LineView V, const TB* lF, const TB* lB, const TX* x,
                           TX* rhs, TX* xt, const LsgsCtl* ctl) {
  pdl_trigger();
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nrows * 32) return;
  const int64_t r = row_begin + (i >> 5), lane = i & 31;
  const int32_t* on = V.onbr + r * V.mout * 32 + lane;
  const TB* F = lF + r * V.mout * 25 * 32 + lane;
  TX b[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) b[k] = TX(__ldcs(lB + (r * 5 + k) * 32 + lane));
  int32_t o = on[0];
  TB f[25];
#pragma unroll
  for (int k = 0; k < 25; ++k) f[k] = __ldcs(F + k * 32);
  pdl_wait();
  if (ctl->done) return;
  if (xt) {
    const int64_t t = r * 32 + lane;
#pragma unroll
    for (int k = 0; k < 5; ++k) xt[5 * t + k] = x[5 * t + k];
  }
  for (int s = 0; s < V.mout && o >= 0; ++s) {
    const int32_t onext = s + 1 < V.mout ? on[(s + 1) * 32] : -1;
    TX xo[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xo[k] = x[5 * int64_t(o) + k];
    if (s > 0) {
#pragma unroll
      for (int k = 0; k < 25; ++k) f[k] = __ldcs(F + (s * 25 + k) * 32);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
      for (int j = 0; j < 5; ++j) b[k] -= TX(f[5 * k + j]) * xo[j];
    o = onext;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) rhs[(r * 5 + k) * 32 + lane] = b[k];
}

// ---- bulk-copy pipeline (TMA engine, no multicast) -------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

constexpr int THOMAS_STAGES = 4;  // most stages in flight per group
constexpr size_t THOMAS_SMEM_MAX = 227 * 1024;  // what a CTA may have
constexpr int THOMAS_THREADS = 64;

// a stage holds `rows` consecutive rows of a group
template <class TB, class TD, class TX>
struct ThomasStage {
  static constexpr int rows = sizeof(TD) == 4 ? 4 : 2;
  static constexpr uint32_t d_row = DROW * sizeof(TD);
  static constexpr uint32_t m_row = 25 * 32 * sizeof(TB);  // L (forward) or U (backward)
  static constexpr uint32_t b_row = 5 * 32 * (sizeof(TX) > sizeof(TB) ? sizeof(TX) : sizeof(TB));
  static constexpr uint32_t m_off = rows * d_row, b_off = m_off + rows * m_row;
  static constexpr uint32_t bytes = b_off + rows * b_row;  // multiple of 16
};
// shared memory: nst stages, their full and empty barriers, an abort flag
// and the forward results of `rows` rows
template <class TB, class TD, class TX>
constexpr size_t thomas_smem_bytes(int nst, int64_t rows) {
  return size_t(nst) * ThomasStage<TB, TD, TX>::bytes + 16 * nst + 16 + size_t(rows) * 5 * 32 * sizeof(TX);
}

// block Thomas solve of the lines of groups [g0, g0+ng) (lineSolve,
// linearSolverLSGS.loci:1523-1572), one CTA per group of 32 lines, one line
// per lane of its first warp.  use_B: right-hand side B (start).
//
// The 5x5 recurrence along a line is a serial chain: with 4,096 lines there
// is less than one walking warp per SM and nothing hides what it waits for.
// So the walking warp does the arithmetic alone: a second warp feeds it
// (the rows of a group are contiguous, [row][block][32 lanes], and arrive as
// bulk copies of a stage's rows, full/empty barriers), each row's blocks are
// requested from shared memory before the row before is done, and the
// forward results stay in shared memory (YS; lines too long for it keep them
// in the spent right-hand-side rows).  Divisions are quotient()s; a chunk of
// rows whose operands leave its range is done again with divisions.  An LSGS
// iteration of 131,072 cells (64 rows, four solves with their right-hand
// sides, MIXED) went from 397 to 174 us: a row's step from 0.66 to 0.21 us,
// against about 0.1 us of its dependent FMAs (the iteration is 156 us with the
// launches overlapped; 154 where each lane decided on its wait alone).  Every
// wait is bounded and its outcome the warp's; one that gives up sets bit 4 of
// err and the abort flag, and the copies in flight land before the CTA ends.
template <class TB, class TD, class TX, bool YS>
__global__ void __launch_bounds__(THOMAS_THREADS)
k_lsgs_thomas(int nst, int64_t g0, LineView V, const TD* lD, const TB* lL,
              const TB* lU, TX* rhs, const TB* lB, int use_B, TX* x,
              const LsgsCtl* ctl, int32_t* __restrict__ err) {
  using S = ThomasStage<TB, TD, TX>;
  constexpr int R = S::rows;
  static_assert(R % 2 == 0, "register sets alternate by row");
  pdl_trigger();
  pdl_wait();
  if (ctl && ctl->done) return;
  extern __shared__ __align__(128) unsigned char th_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(th_smem + size_t(nst) * S::bytes);
  uint64_t* empty = full + nst;
  volatile int* dead = reinterpret_cast<volatile int*>(empty + nst);
  TX* ysm = reinterpret_cast<TX*>(th_smem + size_t(nst) * S::bytes + 16 * nst + 16);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t g = g0 + blockIdx.x;
  const int len = V.lane_len[g * 32 + lane];
  const int glen = __reduce_max_sync(0xffffffffu, len);
  const int nch = (glen + R - 1) / R;  // stages' worth of rows: chunk c holds rows R c ..
  const int64_t r0 = V.grp_row0[g];
  if (threadIdx.x == 0) {
    for (int s = 0; s < nst; ++s) mbar_init(full + s), mbar_init(empty + s);
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 24); ++it) {
      if (mbar_try_wait(bar, parity)) return true;
      if (*dead) break;
    }
    return false;
  };

  if (warp == 1) {
    // the chunks forward (D'_{p-1}, L_p and the right-hand side of each row
    // p), then backward (D'_p and U_p)
    if (lane == 0) {
      int q = 0, s = 0;
      uint32_t round = 0;  // uses of each stage before this one
      for (; q < 2 * nch; ++q) {
        if (round > 0 && !wait(empty + s, (round - 1) & 1)) break;
        unsigned char* st = th_smem + size_t(s) * S::bytes;
        const int c = q < nch ? q : 2 * nch - 1 - q;
        const int64_t r = r0 + int64_t(R) * c;
        const uint32_t n = uint32_t(min(R, glen - R * c));
        if (q < nch) {
          const uint32_t first = c == 0 ? 1 : 0;  // row 0 has no D' before it
          const uint32_t bb = 5 * 32 * uint32_t(use_B ? sizeof(TB) : sizeof(TX));
          mbar_expect_tx(full + s, (n - first) * S::d_row + n * (S::m_row + bb));
          if (n > first) bulk_g2s(st + first * S::d_row, lD + (r - 1 + first) * DROW, (n - first) * S::d_row, full + s);
          bulk_g2s(st + S::m_off, lL + r * 25 * 32, n * S::m_row, full + s);
          bulk_g2s(st + S::b_off, use_B ? (const void*)(lB + r * 5 * 32) : (const void*)(rhs + r * 5 * 32), n * bb,
                   full + s);
        } else {
          mbar_expect_tx(full + s, n * (S::d_row + S::m_row));
          bulk_g2s(st, lD + r * DROW, n * S::d_row, full + s);
          bulk_g2s(st + S::m_off, lU + r * 25 * 32, n * S::m_row, full + s);
        }
        if (++s == nst) s = 0, ++round;
      }
      if (q < 2 * nch) {
        atomicOr(err, 4);
        *dead = 1;
      }
      // the last use of every stage has landed before the CTA may end
      for (int k = q > nst ? q - nst : 0; k < q; ++k)
        for (uint32_t it = 0; it < (1u << 24) && !mbar_try_wait(full + k % nst, (k / nst) & 1); ++it) {
        }
    }
    return;
  }

  // the walking warp goes on or gives up as one: the votes and barriers of its
  // loops need every lane
  auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
  static_assert(sizeof(TD) == sizeof(TX), "the factors and the iterate have one type");
  // register sets: the next row's blocks beside this one's, except where both
  // are FP64 (they would spill)
  constexpr int NS = sizeof(TB) == 8 ? 1 : 2;
  bool ok = true;
  TD D[NS][25], RD[NS][5];  // factors and their pivots' reciprocals
  TB M[NS][25];
  TX B[NS][5];
  int s = 0;  // the stage being read
  uint32_t parity = 0;
  uint32_t key = ~0u;  // of the chunk's dividends
  // row j of the stage's chunk (row p of the group) into register set k
  auto fetch = [&](int j, int p, int k, bool fwd) {
    k %= NS;
    const unsigned char* st = th_smem + size_t(s) * S::bytes;
    const TD* sd = reinterpret_cast<const TD*>(st + j * S::d_row);
    block_load<TD>(sd, lane, D[k]);
#pragma unroll
    for (int e = 0; e < 5; ++e) RD[k][e] = sd[(25 + e) * 32 + lane];
    block_load<TB>(reinterpret_cast<const TB*>(st + S::m_off + j * S::m_row), lane, M[k]);
    if (!fwd) {
#pragma unroll
      for (int e = 0; e < 5; ++e) B[k][e] = YS ? ysm[(p * 5 + e) * 32 + lane] : rhs[((r0 + p) * 5 + e) * 32 + lane];
    } else if (use_B) {
      const TB* sb = reinterpret_cast<const TB*>(st + S::b_off) + j * 5 * 32 + lane;
#pragma unroll
      for (int e = 0; e < 5; ++e) B[k][e] = TX(sb[e * 32]);
    } else {
      const TX* sb = reinterpret_cast<const TX*>(st + S::b_off) + j * 5 * 32 + lane;
#pragma unroll
      for (int e = 0; e < 5; ++e) B[k][e] = sb[e * 32];
    }
  };
  // on to the next chunk's stage; release: hands one back
  auto advance = [&]() {
    if (++s == nst) s = 0, parity ^= 1;
    ok = wait_all(full + s, parity) && ok;
  };
  auto release = [&](int st) {
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + st);
  };
  // D'^{-1} v; a lane past its line's end computes on padding and keeps
  // neither the result nor the key
  auto solve = [&](int k, bool live, bool exact, TX* v) {
    if (exact) {
      lu5_nopiv_solve<TD, TX>(D[k], v);
    } else {
      uint32_t kk = ~0u;
      lu5_recip_solve<TX>(D[k], RD[k], v, kk);
      if (live) key = min(key, kk);
    }
  };
  // forward elimination: y_p = rhs_p - L_p D'_{p-1}^{-1} y_{p-1}
  TX y[5] = {TX(0), TX(0), TX(0), TX(0), TX(0)};
  auto fwd_row = [&](int p, int k, bool first, bool exact) {
    k %= NS;
    const bool live = p < len;
    TX yn[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) yn[e] = B[k][e];
    if (!first) {
      TX v[5];
#pragma unroll
      for (int e = 0; e < 5; ++e) v[e] = y[e];
      solve(k, live, exact, v);
#pragma unroll
      for (int e = 0; e < 5; ++e)
#pragma unroll
        for (int j = 0; j < 5; ++j) yn[e] -= TX(M[k][5 * e + j]) * v[j];
    }
#pragma unroll
    for (int e = 0; e < 5; ++e) {
      y[e] = live ? yn[e] : y[e];
      if (YS)
        ysm[(p * 5 + e) * 32 + lane] = yn[e];
      else
        rhs[((r0 + p) * 5 + e) * 32 + lane] = yn[e];
    }
  };
  // back substitution: x_p = D'_p^{-1} (y_p - U_p x_{p+1}); a line's last
  // row has U = 0 and comes before any x of its line (xn = 0)
  TX xn[5] = {TX(0), TX(0), TX(0), TX(0), TX(0)};
  auto bwd_row = [&](int p, int k, bool exact) {
    k %= NS;
    const bool live = p < len;
    TX v[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) v[e] = B[k][e];
#pragma unroll
    for (int e = 0; e < 5; ++e)
#pragma unroll
      for (int j = 0; j < 5; ++j) v[e] -= TX(M[k][5 * e + j]) * xn[j];
    solve(k, live, exact, v);
    TX* xo = x + 5 * ((r0 + p) * 32 + lane);
#pragma unroll
    for (int e = 0; e < 5; ++e) {
      xn[e] = live ? v[e] : xn[e];
      if (live) xo[e] = v[e];
    }
  };
  // whether a chunk has to be done again with divisions: a dividend too
  // small, a pivot out of range or an overflow (v: the chunk's last row)
  auto inexact = [&](const TX* v) {
    const TX sum = ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
    const bool again = tiny<TX>(key) || sum != sum;
    key = ~0u;
    return __any_sync(0xffffffffu, again);
  };
  // n rows of chunk c, forward or backward; next: another chunk follows in
  // the same direction, whose stage is waited for before this chunk's last
  // row.  On entry the first row's blocks are in registers (NS == 2).
  auto chunk = [&](int c, auto full_chunk, auto forward, bool next) {
    constexpr bool FULL = decltype(full_chunk)::value, FWD = decltype(forward)::value;
    const int n = FULL ? R : glen - R * c;
    TX v0[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) v0[e] = FWD ? y[e] : xn[e];
    const int sc = s;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int j = FWD ? i : R - 1 - i, p = R * c + j;
      if (!FULL && j >= n) continue;
      if (NS == 1) fetch(j, p, 0, FWD);
      if (i + 1 < R && (FULL || !FWD || j + 1 < n)) {
        if (NS == 2) fetch(FWD ? j + 1 : j - 1, FWD ? p + 1 : p - 1, (j + 1) & 1, FWD);
      } else if (next) {
        advance();
        if (NS == 2) fetch(FWD ? 0 : R - 1, FWD ? p + 1 : p - 1, (j + 1) & 1, FWD);
      }
      if (FWD)
        fwd_row(p, j & 1, j == 0 && c == 0, false);
      else
        bwd_row(p, j & 1, false);
    }
    if (inexact(FWD ? y : xn)) {
      const int sn = s;
      s = sc;
#pragma unroll
      for (int e = 0; e < 5; ++e) (FWD ? y : xn)[e] = v0[e];
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const int j = FWD ? i : n - 1 - i, p = R * c + j;
        fetch(j, p, 0, FWD);
        if (FWD)
          fwd_row(p, 0, p == 0, true);
        else
          bwd_row(p, 0, true);
      }
      s = sn;
      key = ~0u;
      // the next row's blocks again, overwritten by the second pass
      if (NS == 2 && next) fetch(FWD ? 0 : R - 1, FWD ? R * c + R : R * c - 1, FWD ? 0 : 1, FWD);
    }
    release(sc);
  };
  using yes = std::true_type;
  using no = std::false_type;
  if (nch > 0) {
    const int nfull = glen / R;
    ok = wait_all(full, 0);
    if (NS == 2) fetch(0, 0, 0, true);
    for (int c = 0; c < nfull && ok; ++c) chunk(c, yes{}, yes{}, c + 1 < nch);
    if (nfull < nch && ok) chunk(nfull, no{}, yes{}, false);
    if (ok) advance();
    if (NS == 2 && ok) {
      if ((glen - 1) & 1)
        fetch((glen - 1) % R, glen - 1, 1, false);
      else
        fetch((glen - 1) % R, glen - 1, 0, false);
    }
    if (nfull < nch && ok) chunk(nfull, no{}, no{}, nfull > 0);
    for (int c = nfull - 1; c >= 0 && ok; --c) chunk(c, yes{}, no{}, c > 0);
  }
  if (!ok) {
    atomicOr(err, 4);
    *dead = 1;
  }
}

constexpr int RELAX_THREADS = 256;

// X = w X + (1-w) X_t and the block partial of ||X - X_t||^2 (:1868-1874)
template <class TX>
__global__ void __launch_bounds__(RELAX_THREADS)
k_lsgs_relax(int64_t nt, TX* x, const TX* xt,
             const LsgsCtl* ctl, double* part) {
  pdl_trigger();
  pdl_wait();
  if (ctl->done) return;
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const double w = ctl->w;
  double s = 0;
  if (t < nt) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const TX xo = xt[5 * t + k];
      const TX xv = TX(w * double(x[5 * t + k]) + (1.0 - w) * double(xo));
      x[5 * t + k] = xv;
      const double d = double(xv) - double(xo);
      s += d * d;
    }
  }
  __shared__ double sh[RELAX_THREADS];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = RELAX_THREADS / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// residual, adaptive relaxation and stopping test (:1923-1947)
__global__ void k_lsgs_control(const double* part, int nblk, double abs_tol,
                               double rel_tol, LsgsCtl* ctl) {
  pdl_trigger();
  pdl_wait();
  if (ctl->done) return;
  __shared__ double sh[RELAX_THREADS];
  double s = 0;
  for (int i = threadIdx.x; i < nblk; i += RELAX_THREADS) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = RELAX_THREADS / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double resid = sqrt(sh[0]);
    if (ctl->iter == 0) ctl->zero = fmax(resid, 1e-16);
    const double rel = resid / ctl->zero;
    if (rel > 1.0) ctl->w *= 1.0 / rel;
    ctl->resid = resid;
    ctl->iter += 1;
    if (resid < abs_tol || rel < rel_tol) ctl->done = 1;
  }
}

__global__ void k_lsgs_init(LsgsCtl* ctl, double w) {
  ctl->w = w;
  ctl->zero = 1.0;
  ctl->resid = 0.0;
  ctl->iter = 0;
  ctl->done = 0;
}

}  // namespace dev

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
namespace {
inline unsigned nblocks(int64_t n, int t) { return unsigned((n + t - 1) / t); }

dev::LineView line_view(const fpsi_ctx* x) {
  dev::LineView V;
  V.t_of = x->d_lt;
  V.role = x->d_lrole;
  V.onbr = x->d_lonbr;
  V.lane_len = x->d_llen;
  V.grp_row0 = x->d_lrow0;
  V.mout = x->LY.mout;
  return V;
}
}  // namespace

template <class TB, class TD, class TX>
static int lsgs_assemble_t(fpsi_ctx* x) {
  const LineLayout& Y = x->LY;
  const dev::LineView V = line_view(x);
  prof_begin(x, "lsgs_scatter");
  launch_chain(x, dev::k_lsgs_scatter<TB, TD>, nblocks(Y.nrows * 32, 128), 128, 0,
      Y.nrows * 32, x->d_lct, x->d_cf_off, x->d_cf, V, (const TB*)x->d_D, (const TB*)x->d_fjp,
      (const TB*)x->d_fjm, x->d_src, (TD*)x->d_lD, (TB*)x->d_lL, (TB*)x->d_lU, (TB*)x->d_lF,
      (TB*)x->d_lB);
  prof_end(x);
  prof_begin(x, "lsgs_prep");
  launch_chain(x, dev::k_lsgs_prep<TB, TD>, nblocks(Y.ngroups * 32, 64), 64, 0,
      Y.ngroups, V, (TD*)x->d_lD, (const TB*)x->d_lL, (const TB*)x->d_lU, x->d_err);
  prof_end(x);
  FPSI_CUDA_TRY(cudaGetLastError());
  return FPSI_OK;
}

int lsgs_assemble(fpsi_ctx* x) {
  switch (x->P.precision) {
    case FPSI_PREC_FP64:
      return lsgs_assemble_t<double, double, double>(x);
    case FPSI_PREC_MIXED:
      return lsgs_assemble_t<float, float, float>(x);
    default:
      return lsgs_assemble_t<float, double, double>(x);
  }
}

// The line solves of ng groups from g0.  Stages per group: what half an SM's
// shared memory holds beside the longest line's forward results (two CTAs
// per SM), or the whole of it where the groups do not fill the SMs twice
// anyway or half holds fewer than two; lines too long for that keep their
// forward results in memory.
template <class TB, class TD, class TX>
static int launch_thomas(fpsi_ctx* x, int64_t g0, int64_t ng, bool use_B, const dev::LsgsCtl* ctl) {
  auto stages = [&](size_t smem, int64_t ylen) {
    int n = 0;
    while (n < dev::THOMAS_STAGES && dev::thomas_smem_bytes<TB, TD, TX>(n + 1, ylen) <= smem) ++n;
    return n;
  };
  const size_t half = dev::THOMAS_SMEM_MAX / 2 - 1024, whole = dev::THOMAS_SMEM_MAX;
  int64_t ylen = x->LY.max_len;
  int nst = stages(half, ylen);
  if (nst < 2 || ng <= x->nsm) nst = stages(whole, ylen);
  if (nst < 2) {
    ylen = 0;
    nst = stages(half, ylen);
  }
  auto k = ylen > 0 ? dev::k_lsgs_thomas<TB, TD, TX, true> : dev::k_lsgs_thomas<TB, TD, TX, false>;
  const size_t smem = dev::thomas_smem_bytes<TB, TD, TX>(nst, ylen);
  prof_begin(x, "lsgs_thomas");
  launch_chain(x, k, ng, dev::THOMAS_THREADS, smem, nst, g0, line_view(x), (const TD*)x->d_lD, (const TB*)x->d_lL, (const TB*)x->d_lU, (TX*)x->d_lrhs,
      (const TB*)x->d_lB, use_B, (TX*)x->d_lx, ctl, x->d_err);
  prof_end(x);
  return FPSI_OK;
}

template <class TB, class TD, class TX>
static int lsgs_solve_t(fpsi_ctx* x, bool jacobi_start) {
  const LineLayout& Y = x->LY;
  cudaStream_t s = x->stream;
  const dev::LineView V = line_view(x);
  dev::LsgsCtl* ctl = (dev::LsgsCtl*)x->d_lctl;
  const int64_t nt = Y.nrows * 32;
  TX* X = (TX*)x->d_lx;
  TX* XT = (TX*)x->d_lxt;
  // A limit, the same for every context and thread: one that followed the
  // launch's own size could be lowered by another's between here and there.
  for (auto k : {dev::k_lsgs_thomas<TB, TD, TX, true>, dev::k_lsgs_thomas<TB, TD, TX, false>})
    FPSI_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dev::THOMAS_SMEM_MAX)));
  // in full: the launches behind it read the system before their waits
  dev::k_lsgs_init<<<1, 1, 0, s>>>(ctl, x->P.lsgs_relaxation);
  int rc;
  if (jacobi_start && (rc = launch_thomas<TB, TD, TX>(x, 0, Y.ngroups, true, nullptr))) return rc;
  const int K = Y.ncolours;
  const int nblk = int(nblocks(nt, dev::RELAX_THREADS));
  for (int it = 0; it < x->P.lsgs_max_iter; ++it) {
    for (int pass = 0; pass < 2; ++pass)
      for (int kk = 0; kk < K; ++kk) {
        const int k = pass == 0 ? kk : K - 1 - kk;
        const int64_t g0 = Y.col_goff[k], ng = Y.col_goff[k + 1] - g0;
        if (ng == 0) continue;
        const int64_t rb = Y.grp_row0[g0];
        const int64_t re = Y.grp_row0[g0 + ng - 1] + Y.grp_len[g0 + ng - 1];
        prof_begin(x, "lsgs_rhs");
        launch_chain(x, dev::k_lsgs_rhs<TB, TX>, nblocks((re - rb) * 32, 128), 128, 0,
            rb, re - rb, V, (const TB*)x->d_lF, (const TB*)x->d_lB, X, (TX*)x->d_lrhs,
            pass == 1 ? XT : nullptr, ctl);
        prof_end(x);
        if ((rc = launch_thomas<TB, TD, TX>(x, g0, ng, false, ctl))) return rc;
      }
    prof_begin(x, "lsgs_relax");
    launch_chain(x, dev::k_lsgs_relax<TX>, nblk, dev::RELAX_THREADS, 0, nt, X, XT, ctl, x->d_lpart);
    launch_chain(x, dev::k_lsgs_control, 1, dev::RELAX_THREADS, 0, x->d_lpart, nblk, x->P.lsgs_abs_tol,
                                                         x->P.lsgs_rel_tol, ctl);
    prof_end(x);
  }
  FPSI_CUDA_TRY(cudaGetLastError());
  return FPSI_OK;
}

int lsgs_solve(fpsi_ctx* x, bool jacobi_start) {
  switch (x->P.precision) {
    case FPSI_PREC_FP64:
      return lsgs_solve_t<double, double, double>(x, jacobi_start);
    case FPSI_PREC_MIXED:
      return lsgs_solve_t<float, float, float>(x, jacobi_start);
    default:
      return lsgs_solve_t<float, double, double>(x, jacobi_start);
  }
}

}  // namespace fpsi
