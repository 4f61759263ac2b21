// Set-up and answers of many LPs (members) on the device: the scaled costs,
// bounds and sides of every member, the norms its decisions need, its starting
// point, and at the end its point in its own units.
//
// The arithmetic is the host's (src/pdhg/pdhg.cpp:424-481, 506-545, 571-587),
// operation for operation: element-wise expressions in the same order, sums in
// index order (pdhg_ordered.cuh), so every value is bit-identical.  On the
// host these passes, the zero-filled vectors they wrote and the pageable
// copies of those were 40 of the 66 ms of set-up of 296 members of
// 1,692 x 3,528.
//
// Members' arrays are concatenated; member b has columns [coff[b], coff[b+1])
// and rows [roff[b], roff[b+1]).  Members of one operator (op_stride 0) share
// its scaling factors R and Cs, else every member has its own range of them.
#pragma once

#include <cstdint>

#include "pdhg_kernels.cuh"
#include "pdhg_ordered.cuh"

namespace b2p {

// Raw arrays as the caller gave them, concatenated; all on the device.
struct MemberData {
  const int32_t *coff, *roff;                     // members + 1
  const double *cost, *lower, *upper, *rl, *ru;   // raw
  const double *R, *Cs;                           // scaling factors
  int32_t shared;                                 // one operator: R and Cs of member 0 serve all
  int32_t rescale;                                // objective and bounds rescaled
};

// Sums per member: ||c||^2, ||sides||^2, then both of the scaled LP before its
// rescaling, then both after it.
enum MemberSum : int { MS_C = 0, MS_B = 1, MS_SC = 2, MS_SB = 3, MS_RC = 4, MS_RB = 5, kMemberSums = 6 };

__device__ __forceinline__ bool member_finite(double v) { return v < 1e20 && v > -1e20; }

__device__ __forceinline__ double member_gamma(const MemberData& d, const double* sums) {
  return d.rescale ? __dadd_rn(1.0, __dsqrt_rn(sums[MS_SC])) : 1.0;
}
__device__ __forceinline__ double member_beta(const MemberData& d, const double* sums) {
  return d.rescale ? __dadd_rn(1.0, __dsqrt_rn(sums[MS_SB])) : 1.0;
}

// Blocks of a member along the grid's y dimension, which holds 65,535: enough
// for one thread per element of a member of 16.7 M, whose threads take several
// beyond that.
constexpr int64_t kMemberMaxBlocks = 65535;
inline unsigned member_grid_y(int64_t elements) {
  const int64_t blocks = (elements + kBlock - 1) / kBlock;
  return static_cast<unsigned>(blocks < 1 ? 1 : blocks < kMemberMaxBlocks ? blocks : kMemberMaxBlocks);
}
__device__ __forceinline__ int64_t member_first() {
  return static_cast<int64_t>(blockIdx.y) * kBlock + threadIdx.x;
}
__device__ __forceinline__ int64_t member_stride() { return static_cast<int64_t>(gridDim.y) * kBlock; }

__device__ __forceinline__ double add_in_order(double t, const double* term, int count) {
#pragma unroll 16
  for (int i = 0; i < count; ++i) t = __dadd_rn(t, term[i]);
  return t;
}

// The squares of the finite sides, lower then upper of every row, an upper one
// that equals the lower left out (an absent term adds +0 to a sum that is
// never negative).
__device__ __forceinline__ double side_term(double lo, double up, int64_t i) {
  const bool upper = i & 1;
  const double v = upper ? up : lo;
  const bool in = member_finite(v) && (!upper || up != lo);
  return in ? __dmul_rn(v, v) : 0.0;
}

// grid = (members, 4): sum q of member b.
__global__ void __launch_bounds__(kOrderedThreads) k_member_raw_sums(MemberData d, double* __restrict__ sums) {
  const int b = blockIdx.x, q = blockIdx.y;
  const int32_t c0 = d.coff[b], n = d.coff[b + 1] - c0, r0 = d.roff[b], m = d.roff[b + 1] - r0;
  const double* Cs = d.Cs + (d.shared ? 0 : c0);
  const double* R = d.R + (d.shared ? 0 : r0);
  double s;
  if (q == MS_C || q == MS_SC) {
    s = ordered_sum(
        n,
        [&](int64_t j) {
          const double t = q == MS_C ? d.cost[c0 + j] : __dmul_rn(d.cost[c0 + j], Cs[j]);
          return __dmul_rn(t, t);
        },
        add_in_order);
  } else {
    s = ordered_sum(
        2 * static_cast<int64_t>(m),
        [&](int64_t t) {
          const int64_t i = t >> 1;
          const double lo = d.rl[r0 + i], up = d.ru[r0 + i];
          if (q == MS_B) return side_term(lo, up, t);
          // the scaled sides, chosen by the raw ones
          const double v = (t & 1) ? up : lo;
          const bool in = member_finite(v) && (!(t & 1) || up != lo);
          const double w = __dmul_rn(v, R[i]);
          return in ? __dmul_rn(w, w) : 0.0;
        },
        add_in_order);
  }
  if (threadIdx.x == 0) sums[static_cast<int64_t>(b) * kMemberSums + q] = s;
}

// grid = (members, blocks of columns): scaled costs and bounds, x = proj(0),
// the check's column factors.
__global__ void __launch_bounds__(kBlock) k_member_columns(MemberData d, const double* __restrict__ sums,
                                                           double* __restrict__ c, double* __restrict__ lo,
                                                           double* __restrict__ up, double* __restrict__ x,
                                                           double* __restrict__ cfac) {
  const int b = blockIdx.x;
  const int32_t c0 = d.coff[b], n = d.coff[b + 1] - c0;
  const double* sb = sums + static_cast<int64_t>(b) * kMemberSums;
  const double gamma = member_gamma(d, sb), beta = member_beta(d, sb);
  for (int64_t j = member_first(); j < n; j += member_stride()) {
    const double s = d.Cs[(d.shared ? 0 : c0) + j];
    const int64_t t = c0 + j;
    const double l = d.lower[t], u = d.upper[t];
    cfac[t] = __ddiv_rn(gamma, s);
    c[t] = __ddiv_rn(__dmul_rn(d.cost[t], s), gamma);
    const double lv = member_finite(l) ? __ddiv_rn(__ddiv_rn(l, s), beta) : -INFINITY;
    const double uv = member_finite(u) ? __ddiv_rn(__ddiv_rn(u, s), beta) : INFINITY;
    lo[t] = lv;
    up[t] = uv;
    double v = (0.0 < lv) ? lv : 0.0;
    v = (uv < v) ? uv : v;
    x[t] = v;
  }
}

// grid = (members, blocks of rows): scaled sides, the check's row factors.
__global__ void __launch_bounds__(kBlock) k_member_rows(MemberData d, const double* __restrict__ sums,
                                                        double* __restrict__ rl, double* __restrict__ ru,
                                                        double* __restrict__ rfac) {
  const int b = blockIdx.x;
  const int32_t r0 = d.roff[b], m = d.roff[b + 1] - r0;
  const double beta = member_beta(d, sums + static_cast<int64_t>(b) * kMemberSums);
  for (int64_t i = member_first(); i < m; i += member_stride()) {
    const double s = d.R[(d.shared ? 0 : r0) + i];
    const int64_t t = r0 + i;
    const double l = d.rl[t], u = d.ru[t];
    rfac[t] = __ddiv_rn(beta, s);
    rl[t] = member_finite(l) ? __ddiv_rn(__dmul_rn(l, s), beta) : -INFINITY;
    ru[t] = member_finite(u) ? __ddiv_rn(__dmul_rn(u, s), beta) : INFINITY;
  }
}

// grid = (members, 2): the norms of the scaled LP.
__global__ void __launch_bounds__(kOrderedThreads) k_member_scaled_sums(MemberData d, const double* __restrict__ c,
                                                                        const double* __restrict__ rl,
                                                                        const double* __restrict__ ru,
                                                                        double* __restrict__ sums) {
  const int b = blockIdx.x, q = MS_RC + blockIdx.y;
  const int32_t c0 = d.coff[b], n = d.coff[b + 1] - c0, r0 = d.roff[b], m = d.roff[b + 1] - r0;
  const double s = q == MS_RC ? ordered_sum(
                                    n, [&](int64_t j) { return __dmul_rn(c[c0 + j], c[c0 + j]); }, add_in_order)
                              : ordered_sum(
                                    2 * static_cast<int64_t>(m),
                                    [&](int64_t t) { return side_term(rl[r0 + (t >> 1)], ru[r0 + (t >> 1)], t); },
                                    add_in_order);
  if (threadIdx.x == 0) sums[static_cast<int64_t>(b) * kMemberSums + q] = s;
}

// y = M x member by member, every member with the same M (rows x cols).
__global__ void __launch_bounds__(kBlock) k_member_spmv(int64_t total, int32_t rows, int32_t cols, CsrView M,
                                                        const double* __restrict__ x, double* __restrict__ y) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (t >= total) return;
  const int64_t b = t / rows;
  y[t] = row_dot(M, x + b * cols, t - b * rows, 1, 0);
}

// grid = (members from `first`, blocks of elements): x = x+ Cs beta and
// y = y+ R gamma.
__global__ void __launch_bounds__(kBlock) k_member_answers(MemberData d, int32_t first, const double* __restrict__ sums,
                                                           const double* __restrict__ xp,
                                                           const double* __restrict__ yp, double* __restrict__ x,
                                                           double* __restrict__ y) {
  const int b = first + blockIdx.x;
  const int32_t c0 = d.coff[b], n = d.coff[b + 1] - c0, r0 = d.roff[b], m = d.roff[b + 1] - r0;
  const double* sb = sums + static_cast<int64_t>(b) * kMemberSums;
  const double gamma = member_gamma(d, sb), beta = member_beta(d, sb);
  for (int64_t i = member_first(); i < (n > m ? n : m); i += member_stride()) {
    if (i < n) x[c0 + i] = __dmul_rn(__dmul_rn(xp[c0 + i], d.Cs[(d.shared ? 0 : c0) + i]), beta);
    if (i < m) y[r0 + i] = __dmul_rn(__dmul_rn(yp[r0 + i], d.R[(d.shared ? 0 : r0) + i]), gamma);
  }
}

}  // namespace b2p
