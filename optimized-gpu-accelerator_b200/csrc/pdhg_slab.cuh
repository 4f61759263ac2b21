// The CTA form's slab kernel: one LP per thread-block cluster of C blocks
// (C = 1, 2, 4 or 8), its operators in their shared memory.
//
// The general kernel (pdhg_cta.cuh) runs an LP on one SM; where the operators
// do not fit beside the vectors it reads them from L2 every iteration (360 KB
// for the 1,692 x 3,528 refinery), and a batch of few such LPs leaves most SMs
// idle.  Here
//   - the rows of A and of A^T, in order of length (stable, so that runs stay
//     together), are cut into slices of 32, and slice s belongs to block s mod
//     C of the cluster, to one of its warps (unsorted, a slice's longest row
//     pads the others by a third: 235 KB a block at C = 2 for that refinery,
//     194 KB sorted);
//   - a slice lies in its block's shared memory column by column (entry q of
//     its 32 rows together: one wavefront per 16-bit index load, two per
//     value load), built once per run;
//   - x+ and y, which every row gathers from, are whole in every block's
//     shared memory: a row's owner stores its entry to all C of them
//     (distributed shared memory), and two cluster barriers separate the
//     phases of an iteration;
//   - what only the owner touches (x, x0, y0, A x, A x0) stays in its
//     registers; costs, bounds and sides come from L1 / L2, asked for before
//     the row's sum.
// Every row is summed left to right with separately rounded products and sums
// and every element updated by run_lp's expressions; at a check the owners
// store their elements' terms, and every block adds them in the CTA form's one
// order (kSumThreads) and makes the decisions itself (with rank 0's reading of
// the stop flag): answers are the other variants' bit for bit.
//
// Measured on 30 members of 1,692 x 3,528 (us per iteration): general kernel
// 9.9; here 3.7 on clusters of 4 blocks of 512 threads, 5.6 on 2 blocks of
// 512.  (Blocks of 1,024 threads with two slices a warp hold what 512 with four
// do, and took 5.9 on 2.)  With members enough to keep every SM busy anyway
// (296 of them) a cluster of 2 takes as long per member and SM as the general
// kernel, so it serves batches whose clusters need no more blocks than there
// are SMs.
#pragma once

#include <cstdint>
#include <vector>

#include "pdhg_cta.cuh"

namespace b2p {

// Rows of an operator (row pointers ptr[0..rows]) in decreasing order of
// length, stable.
inline void slab_order(const int32_t* ptr, int32_t rows, int32_t* order) {
  int32_t most = 0;
  for (int32_t r = 0; r < rows; ++r) most = ptr[r + 1] - ptr[r] > most ? ptr[r + 1] - ptr[r] : most;
  std::vector<int32_t> at(static_cast<size_t>(most) + 2, 0);  // first place of each length, longest first
  for (int32_t r = 0; r < rows; ++r) ++at[most - (ptr[r + 1] - ptr[r]) + 1];
  for (size_t i = 1; i < at.size(); ++i) at[i] += at[i - 1];
  for (int32_t r = 0; r < rows; ++r) order[at[most - (ptr[r + 1] - ptr[r])]++] = r;
}

// Largest entries (32 x width summed over its slices) any block of a cluster
// of C holds: the first one's, whose slices are the longest of each round.
inline int64_t slab_entries(const int32_t* ptr, int32_t rows, const int32_t* order, int C) {
  int64_t e = 0;
  for (int64_t s = 0; s * 32 < rows; s += C) e += 32 * static_cast<int64_t>(ptr[order[s * 32] + 1] - ptr[order[s * 32]]);
  return e;
}

// Dynamic shared memory of one block: the gathered vectors, then both
// operators' values, then their indices.
__host__ __device__ inline int64_t slab_smem_bytes(int64_t m, int64_t n, int64_t a_entries, int64_t t_entries,
                                                   int esize) {
  const int64_t vec = (esize * (n + m) + 7) / 8 * 8;
  return vec + (esize * (a_entries + t_entries) + 7) / 8 * 8 + 2 * (a_entries + t_entries);
}

namespace slab {

// passes of a block of NT threads over the virtual threads of a check's sums
template <int NT>
constexpr int kSumPasses = (cta::kSumThreads + NT - 1) / NT;

__device__ __forceinline__ void barrier(int C) {
  if (C == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

__device__ __forceinline__ void store_peer(uint32_t at, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ void store_peer(uint32_t at, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
// v to the same place of every block of the cluster.
template <class T>
__device__ __forceinline__ void publish(T* local, T v, int C, int rank) {
  *local = v;
  const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(local));
  for (int r = 0; r < C; ++r) {
    if (r == rank) continue;
    uint32_t peer;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(r));
    store_peer(peer, v);
  }
}

// A thread's row of an operator: its slice starts at `base`, it has `len`
// entries.
struct Row {
  int base, len;
};

template <class T>
__device__ __forceinline__ double row_sum(const Row& r, const uint16_t* __restrict__ idx, const T* __restrict__ val,
                                          const T* __restrict__ v) {
  double s = 0.0;
  int p = r.base;
#pragma unroll 4
  for (int q = 0; q < r.len; ++q, p += 32)
    s = __dadd_rn(s, __dmul_rn(static_cast<double>(val[p]), static_cast<double>(v[idx[p]])));
  return s;
}

// The slices of one operator into shared memory: ptr / gidx / gval are the
// LP's rows in the concatenated CSR, `shift` what its indices carry, own[r]
// this thread's row of its slice r (-1: none), placed in rows[r].
template <int NT, int R, class T>
__device__ __forceinline__ void place(const int32_t* __restrict__ ptr, const int32_t* __restrict__ gidx,
                                      const T* __restrict__ gval, int shift, const int (&own)[R], T* val, uint16_t* idx,
                                      int* widths /* R * NT / 32 */, Row (&rows)[R]) {
  constexpr int W = NT / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int beg[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    beg[r] = 0;
    rows[r].len = 0;
    if (own[r] >= 0) {
      beg[r] = ptr[own[r]];
      rows[r].len = ptr[own[r] + 1] - beg[r];
    }
    const int w = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(rows[r].len));
    if (lane == 0) widths[warp + r * W] = 32 * w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0;
    for (int s = 0; s < R * W; ++s) {
      const int w = widths[s];
      widths[s] = at;
      at += w;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    rows[r].base = widths[warp + r * W] + lane;
    for (int q = 0; q < rows[r].len; ++q) {
      val[rows[r].base + 32 * q] = gval[beg[r] + q];
      idx[rows[r].base + 32 * q] = static_cast<uint16_t>(gidx[beg[r] + q] - shift);
    }
  }
  __syncthreads();
}

// The terms of one element into the cluster's scratch: the row sums' (q < 5)
// or the column sums'.
__device__ __forceinline__ void store_terms(const double (&s)[kNumSums], int first, double* scratch, int64_t stride,
                                            int64_t at) {
#pragma unroll
  for (int q = 0; q < kRowSums; ++q) __stcg(scratch + q * stride + at, s[first + q]);
}

// All terms stored: every block adds them up and decides (every thread of
// every block).  entry: only the termination test, on the starting point.
// Out of line: its sums live here, not in the iteration loop's registers.
template <int NT>
__device__ __noinline__ void cluster_decide(cta::Shared& sh, int32_t* stop, const CtaArgs& a, const CtaLp& L, int C,
                                               int rank, int64_t it, bool entry) {
  if (rank == 0 && threadIdx.x == 0) {
    const int32_t v = a.stop ? *a.stop : 0;
    *stop = v;
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(stop));
    for (int r = 1; r < C; ++r) {
      uint32_t peer;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(r));
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer), "r"(v) : "memory");
    }
  }
  __threadfence();
  barrier(C);
  for (int pass = 0; pass < kSumPasses<NT>; ++pass) {
    double s[kNumSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int v = threadIdx.x + pass * NT;
    for (int i = v; i < L.m; i += cta::kSumThreads)
#pragma unroll
      for (int q = 0; q < kRowSums; ++q) s[q] += __ldcg(a.row_terms + q * a.rows_total + L.roff + i);
    for (int j = v; j < L.n; j += cta::kSumThreads)
#pragma unroll
      for (int q = 0; q < kRowSums; ++q) s[kRowSums + q] += __ldcg(a.col_terms + q * a.cols_total + L.coff + j);
    if (v < cta::kSumThreads) cta::pass_sums<NT>(s, sh, pass);
  }
  if (entry) {
    cta::entry_decide(sh, a, L);
    return;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    cta::total_sums(sh);
    if (threadIdx.x == 0) {
      sh.ctl.stop = *stop;
      cta::decide(sh.ctl, sh.tot, L.scale_obj, L.rhsnorm, L.cnorm, L.eta, it, a.tol, a.check_every, a.stall_checks);
    }
  }
  __syncthreads();
}

}  // namespace slab

// RC / RR: slices of columns / rows per warp.
template <int NT, int RC, int RR, class T>
__global__ void __launch_bounds__(NT, 1) k_lp_slab(const __grid_constant__ CtaArgs a, int C) {
  constexpr int W = NT / 32;
  extern __shared__ __align__(16) unsigned char cta_smem[];
  __shared__ cta::Shared sh;
  __shared__ int32_t stop_sh;
  __shared__ int widths[(RC > RR ? RC : RR) * W];
  __shared__ double s_lam[2];
  const int lp = a.order[blockIdx.x / C], rank = blockIdx.x % C;
  const CtaLp L = a.lps[lp];
  const int m = L.m, n = L.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const CtaState<T> g = cta_state(a, static_cast<T*>(nullptr));
  T* xp = reinterpret_cast<T*>(cta_smem);
  T* y = xp + n;  // y; y+ at a check iteration
  T* tval = reinterpret_cast<T*>(cta_smem + (sizeof(T) * (static_cast<size_t>(n) + m) + 7) / 8 * 8);
  const double* __restrict__ cost = a.c + L.coff;
  const double* __restrict__ lo = a.lo + L.coff;
  const double* __restrict__ up = a.up + L.coff;
  const double* __restrict__ rl = a.rl + L.roff;
  const double* __restrict__ ru = a.ru + L.roff;

  // owned column / row of slice r: place (slice * C + rank) * 32 + lane in the
  // order by length; -1 past the end
  int col[RC], row[RR];
  slab::Row tr[RC], ar[RR];
#pragma unroll
  for (int r = 0; r < RC; ++r) {
    const int at = ((warp + r * W) * C + rank) * 32 + lane;
    col[r] = at < n ? a.slab_cols[L.tptr_off + at] : -1;
  }
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    const int at = ((warp + r * W) * C + rank) * 32 + lane;
    row[r] = at < m ? a.slab_rows[L.aptr_off + at] : -1;
  }
  // the operators' values, then their indices: entries of this block's slices
  const int32_t* tp = a.AT.ptr + L.tptr_off;
  const int32_t* ap = a.A.ptr + L.aptr_off;
  int te = 0, ae = 0;
#pragma unroll
  for (int r = 0; r < RC; ++r)
    te += 32 * __reduce_max_sync(0xffffffffu, col[r] >= 0 ? static_cast<unsigned>(tp[col[r] + 1] - tp[col[r]]) : 0u);
#pragma unroll
  for (int r = 0; r < RR; ++r)
    ae += 32 * __reduce_max_sync(0xffffffffu, row[r] >= 0 ? static_cast<unsigned>(ap[row[r] + 1] - ap[row[r]]) : 0u);
  __shared__ int placed[2][W];
  if (lane == 0) {
    placed[0][warp] = te;
    placed[1][warp] = ae;
  }
  __syncthreads();
  int t_entries = 0, a_entries = 0;
  for (int w = 0; w < W; ++w) {
    t_entries += placed[0][w];
    a_entries += placed[1][w];
  }
  T* aval = tval + t_entries;
  uint16_t* tidx = reinterpret_cast<uint16_t*>(reinterpret_cast<unsigned char*>(tval) +
                                               (sizeof(T) * (static_cast<size_t>(t_entries) + a_entries) + 7) / 8 * 8);
  uint16_t* aidx = tidx + t_entries;
  slab::place<NT, RC, T>(tp, a.AT.idx, g.Tv, L.tshift, col, tval, tidx, widths, tr);
  slab::place<NT, RR, T>(ap, a.A.idx, g.Av, L.ashift, row, aval, aidx, widths, ar);

  T x[RC], x0[RC], y0[RR], ax[RR], ax0[RR], yold[RR], axpr[RR];
#pragma unroll
  for (int r = 0; r < RC; ++r) {
    const int j = col[r];
    x[r] = x0[r] = j >= 0 ? static_cast<T>(a.xinit[L.coff + j]) : T(0);
  }
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    const int i = row[r];
    y0[r] = i >= 0 ? static_cast<T>(a.yinit[L.roff + i]) : T(0);
    ax[r] = ax0[r] = i >= 0 ? static_cast<T>(a.axinit[L.roff + i]) : T(0);
    yold[r] = axpr[r] = T(0);
  }
  for (int i = tid; i < m; i += NT) y[i] = static_cast<T>(a.yinit[L.roff + i]);
  if (tid == 0) cta::init_ctl(sh.ctl, L);
  slab::barrier(C);  // every block runs, and is set up, before the first store to its shared memory

  const double rho = a.rho;
  const int cE = a.check_every;
  double tau = sh.ctl.tau, sigma = sh.ctl.sigma;
  int64_t restartAt = L.it0, it = L.it0;
  if (a.entry_check) {
    // the starting point measured as it is (x+ = x, y+ = y, A x+ = A x)
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int i = row[r];
      if (i >= 0) {
        double s[kNumSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        const double yv = static_cast<double>(y0[r]);
        cta::row_check(s, static_cast<double>(ax[r]), rl[i], ru[i], a.rfac[L.roff + i], yv, yv, yv);
        slab::store_terms(s, 0, a.row_terms, a.rows_total, L.roff + i);
        axpr[r] = ax[r];
        a.yp[L.roff + i] = yv;
      }
    }
#pragma unroll
    for (int r = 0; r < RC; ++r) {
      const int j = col[r];
      if (j >= 0) {
        double s[kNumSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        const double xv = static_cast<double>(x[r]);
        cta::col_check(s, slab::row_sum(tr[r], tidx, tval, y), cost[j], lo[j], up[j], a.cfac[L.coff + j], xv, xv, xv);
        slab::store_terms(s, kRowSums, a.col_terms, a.cols_total, L.coff + j);
        xp[j] = x[r];
      }
    }
    slab::cluster_decide<NT>(sh, &stop_sh, a, L, C, rank, it, true);
    if (sh.ctl.status) it = L.it0 - 1;  // reported as the check iteration that produced the point
  }
  // lambda of the next iteration is one thread's division during this one
  const bool lam_maker = tid == NT - 32;
  while (!sh.ctl.status && it < a.max_it) {
    const int Lint = static_cast<int>((a.max_it - it) < cE ? (a.max_it - it) : cE);
    if (lam_maker) s_lam[0] = cta::lambda_at(it - restartAt);
    __syncthreads();
    for (int l = 0; l < Lint; ++l) {
      const bool halpern = l != Lint - 1;
      const double lam = s_lam[l & 1];
      if (lam_maker && halpern) s_lam[(l + 1) & 1] = cta::lambda_at(it + l + 1 - restartAt);
      // x+ = proj(x - tau (c - A^T y)), Halpern step of x
#pragma unroll
      for (int r = 0; r < RC; ++r) {
        const int j = col[r];
        if (j >= 0) {
          const double cj = __ldg(cost + j), lj = __ldg(lo + j), uj = __ldg(up + j);
          const double aty = slab::row_sum(tr[r], tidx, tval, y);
          const double xv = static_cast<double>(x[r]);
          double v = __dsub_rn(xv, __dmul_rn(tau, __dsub_rn(cj, aty)));
          v = (v < lj) ? lj : v;
          v = (uj < v) ? uj : v;
          slab::publish(xp + j, static_cast<T>(v), C, rank);
          if (halpern) x[r] = static_cast<T>(halpern_step(xv, v, static_cast<double>(x0[r]), lam, rho));
        }
      }
      slab::barrier(C);
      // A x+, y+ = v + sigma proj(-v / sigma), Halpern steps of y and A x
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        const int i = row[r];
        if (i >= 0) {
          const double li = __ldg(rl + i), ui = __ldg(ru + i);
          const double yv = static_cast<double>(y[i]);
          const double axpv = slab::row_sum(ar[r], aidx, aval, xp);
          const double axv = static_cast<double>(ax[r]);
          const double v = __dsub_rn(yv, __dmul_rn(sigma, __dsub_rn(__dmul_rn(2.0, axpv), axv)));
          double w = __ddiv_rn(-v, sigma);
          w = (w < li) ? li : w;
          w = (ui < w) ? ui : w;
          const double ypv = __dadd_rn(v, __dmul_rn(sigma, w));
          if (halpern) {
            slab::publish(y + i, static_cast<T>(halpern_step(yv, ypv, static_cast<double>(y0[r]), lam, rho)), C, rank);
            ax[r] = static_cast<T>(halpern_step(axv, axpv, static_cast<double>(ax0[r]), lam, rho));
          } else {
            // y+ takes y's place for the check; y itself stays with its owner
            axpr[r] = static_cast<T>(axpv);
            yold[r] = static_cast<T>(yv);
            slab::publish(y + i, static_cast<T>(ypv), C, rank);
          }
        }
      }
      slab::barrier(C);
    }
    // ---- check at iteration it + Lint - 1
    const double lam = s_lam[(Lint - 1) & 1];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int i = row[r];
      if (i >= 0) {
        double s[kNumSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        const double yv = static_cast<double>(y[i]);
        cta::row_check(s, static_cast<double>(axpr[r]), rl[i], ru[i], a.rfac[L.roff + i], yv,
                       static_cast<double>(yold[r]), static_cast<double>(y0[r]));
        slab::store_terms(s, 0, a.row_terms, a.rows_total, L.roff + i);
        a.yp[L.roff + i] = yv;
      }
    }
#pragma unroll
    for (int r = 0; r < RC; ++r) {
      const int j = col[r];
      if (j >= 0) {
        double s[kNumSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        const double atyp = slab::row_sum(tr[r], tidx, tval, y);
        cta::col_check(s, atyp, cost[j], lo[j], up[j], a.cfac[L.coff + j], static_cast<double>(xp[j]),
                       static_cast<double>(x[r]), static_cast<double>(x0[r]));
        slab::store_terms(s, kRowSums, a.col_terms, a.cols_total, L.coff + j);
      }
    }
    it += Lint - 1;
    slab::cluster_decide<NT>(sh, &stop_sh, a, L, C, rank, it, false);
    if (sh.ctl.status) break;
    // the deferred Halpern step of that iteration, or the restart in its place
    const bool restart = sh.ctl.restart;
    if (restart) {
      tau = sh.ctl.tau;
      sigma = sh.ctl.sigma;
      restartAt = sh.ctl.restart_at;
    }
#pragma unroll
    for (int r = 0; r < RC; ++r) {
      const int j = col[r];
      if (j >= 0) {
        if (restart)
          x[r] = x0[r] = xp[j];
        else
          x[r] = static_cast<T>(halpern_step(static_cast<double>(x[r]), static_cast<double>(xp[j]),
                                             static_cast<double>(x0[r]), lam, rho));
      }
    }
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int i = row[r];
      if (i >= 0) {
        const T yp = y[i];
        if (restart) {
          y0[r] = yp;
          ax[r] = ax0[r] = axpr[r];
        } else {
          slab::publish(y + i, static_cast<T>(halpern_step(static_cast<double>(yold[r]), static_cast<double>(yp),
                                                           static_cast<double>(y0[r]), lam, rho)),
                        C, rank);
          ax[r] = static_cast<T>(halpern_step(static_cast<double>(ax[r]), static_cast<double>(axpr[r]),
                                              static_cast<double>(ax0[r]), lam, rho));
        }
      }
    }
    slab::barrier(C);
    ++it;
  }
  // results: x+ to the engine's FP64 arrays (y+ went there at the last check),
  // the scalars to out[lp]
#pragma unroll
  for (int r = 0; r < RC; ++r) {
    const int j = col[r];
    if (j >= 0) a.xp[L.coff + j] = static_cast<double>(xp[j]);
  }
  if (rank == 0) cta::write_out(a, sh.ctl, lp, it);
  slab::barrier(C);  // no block leaves while another may still store to it
}

}  // namespace b2p
