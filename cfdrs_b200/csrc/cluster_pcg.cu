// Whole-solve PCG for small systems in one thread-block cluster: the plain CG
// and Jacobi-PCG of krylov::cg[_preconditioned] (krylov.rs:318-360, with
// DiagJacobi) in FP64, for systems whose rows fit the shared memory of a
// cluster of up to 16 CTAs (the 2-D 128^2 pressure Poisson system of 16 384
// unknowns among them).
//
// A multi-kernel PCG iteration on such a system is bound by launch and
// grid-reduction latency (about 19 us per iteration at 128^2: three to four
// kernels on data that sits in L2). Here one launch runs the whole solve, and an
// iteration is bound by two cluster barriers (450 cycles each with release and
// acquire), one remote gather (325 cycles) and the two reductions' shuffles:
//  - A thread owns R rows: x, r, p, q and D^-1 of those rows, and up to two
//    rows a thread the first entries of the matrix, stay in registers; z = D^-1 r
//    and p are also in shared memory, where the other rows read them.
//  - The SpMV forms another CTA's new direction itself, z_j + beta p_j from that
//    CTA's z and old p (two buffers of p in turn), so p needs no barrier of its
//    own; the same operations as the owner's, so the same bits. Only lanes whose
//    entry is another CTA's take the cluster path (a predicate on the load): its
//    throughput is low even for a CTA's own memory (SpMV phase 1600 -> 1190
//    cycles at 128^2).
//  - A row's five entries are read without branches (slots past its end take a
//    zero entry, value 0 times a vector slot that stays 0, so that no vector entry
//    reaches a row without its column), so all of its gathers are in flight together.
//  - Behind a reduction's barrier one warp fetches the CTAs' partials (one
//    remote load) and hands the totals to the others; pushing them to every CTA
//    before the barrier made the barrier wait for the stores (3.65 against 3.08
//    us an iteration).
// Every CTA sums all partials in the same order, so every CTA holds the same
// value and takes the same branch. The barriers are the hardware cluster
// barrier; control flow is uniform across the cluster, so no CTA can wait for
// one that has left. Measured, Jacobi-CG to 1e-10, device time before (three
// barriers an iteration, vectors in shared memory, entry-by-entry gathers of p)
// and now: 64^2 0.99 -> 0.53 ms, 128^2 2.03 -> 1.30 ms, 181^2 3.74 -> 2.43 ms,
// 200 x 170 4.92 -> 2.96 ms.
//
// Recurrence and termination are pcg_loop's: r0 = b - A x0, threshold
// max(tol, rtol ||r0||), InitialResidual / Breakdown on the initial residual;
// per iteration q = A p, NonPositiveCurvature when p.q <= 0, alpha = rho / p.q,
// x += alpha p, r -= alpha q, Breakdown / Converged / MaxIterations on ||r||,
// rho' = r.z (z = D^-1 r, or r), Breakdown when rho' is 0 or not finite,
// beta = rho' / rho, p = z + beta p. The row sums run in CSR order as the
// one-thread-per-row pipelines do; the dot products sum per-CTA partials in a
// different tree than the grid reductions, so iterates agree with the
// multi-kernel solve to rounding.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace cfd {
namespace {

constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClMaxCtas = 16;
constexpr int kClMaxRows = 8;  // rows per thread
constexpr int kClU = 5;        // entries of a row read together (a five-point row)
constexpr int kClMaxFar = 1500;  // scattered entries of other CTAs (cluster_pcg_solve)

struct ClusterArgs {
  const int* __restrict__ rp;  // global CSR (int32)
  const int* __restrict__ col;
  const double* __restrict__ val;
  const double* __restrict__ jinv;  // nullptr: no preconditioner
  const double* __restrict__ b;
  double* __restrict__ x;
  DevState* st;
  int n, rpc, nnz_cap;  // rows, rows per CTA, nonzeros per CTA at most
};

struct ClusterLayout {
  size_t val, ent, rpl, z, p, bytes;
};

__host__ __device__ inline size_t cl_round16(size_t b) { return (b + 15) / 16 * 16; }

__host__ __device__ inline ClusterLayout cluster_layout(int rpc, int nnz_cap) {
  ClusterLayout L;
  L.val = 0;  // nnz_cap values and a zero entry
  L.ent = cl_round16((size_t)(nnz_cap + 1) * 8);
  L.rpl = L.ent + cl_round16((size_t)(nnz_cap + 1) * 4);
  L.z = L.rpl + cl_round16((size_t)(rpc + 1) * 4);
  L.p = L.z + cl_round16((size_t)rpc * 8);
  L.bytes = L.p + 2 * cl_round16((size_t)(rpc + 1) * 8);  // two buffers, each with a slot that stays zero
  return L;
}

__device__ __forceinline__ uint32_t cl_map(uint32_t a, uint32_t rank) {
  uint32_t d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}
// A load of the cluster's shared memory (volatile keeps it between the barriers
// that order it) only where `on` (a predicate, not a branch), else v as it is: the
// cluster path is slow even for a CTA's own memory, so only lanes whose entry is
// another CTA's take it.
__device__ __forceinline__ void cl_ld_if(double& v, uint32_t a, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.shared::cluster.f64 %0, [%1];\n}\n"
               : "+d"(v)
               : "r"(a), "r"((int)on));
}

template <int R>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_pcg(ClusterArgs A) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int ncta = (int)cluster.num_blocks();
  extern __shared__ __align__(16) unsigned char sm[];
  const ClusterLayout L = cluster_layout(A.rpc, A.nnz_cap);
  double* sval = reinterpret_cast<double*>(sm + L.val);
  int* sent = reinterpret_cast<int*>(sm + L.ent);  // owner << 16 | local index
  int* srp = reinterpret_cast<int*>(sm + L.rpl);
  double* sz = reinterpret_cast<double*>(sm + L.z);
  const uint32_t psz = (uint32_t)cl_round16((size_t)(A.rpc + 1) * 8);  // bytes of a p buffer
  auto sp = [&](int buf) { return reinterpret_cast<double*>(sm + L.p + (buf ? psz : 0u)); };
  __shared__ double part[2][2];  // [slot][value]: this CTA's partial sums
  __shared__ double bcast[2];
  __shared__ double red[2][kClWarps];
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  const uint32_t pbase = (uint32_t)__cvta_generic_to_shared(&part[0][0]);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  const int r0 = rank * A.rpc;
  const int nrow = max(0, min(A.rpc, A.n - r0));
  const int k0 = nrow > 0 ? A.rp[r0] : 0;
  const int nnz = nrow > 0 ? A.rp[r0 + nrow] - k0 : 0;
  for (int i = tid; i <= nrow; i += kClThreads) srp[i] = nrow > 0 ? A.rp[r0 + i] - k0 : 0;
  for (int e = tid; e < nnz; e += kClThreads) {
    const int c = A.col[k0 + e];
    const int owner = c / A.rpc;
    sent[e] = (owner << 16) | (c - owner * A.rpc);
    sval[e] = A.val[k0 + e];
  }
  if (tid == 0) {  // the zero entry
    sent[A.nnz_cap] = (rank << 16) | A.rpc;
    sval[A.nnz_cap] = 0.0;
    sp(0)[A.rpc] = sp(1)[A.rpc] = 0.0;
  }
  double x[R], r[R], p[R], q[R], jv[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int i = tid + u * kClThreads;
    const bool live = i < nrow;
    x[u] = live ? A.x[r0 + i] : 0.0;
    jv[u] = live ? (A.jinv ? A.jinv[r0 + i] : 1.0) : 0.0;
    r[u] = p[u] = q[u] = 0.0;
    if (i < A.rpc) {
      sz[i] = x[u];
      sp(0)[i] = 0.0;
      sp(1)[i] = x[u];
    }
  }
  cluster_barrier();  // every CTA's x staged (in z and the second p buffer)

  // Up to two rows a thread keep their first kClU entries in registers: read
  // from shared memory every iteration they bound the SpMV (12 of 20 bytes an
  // entry at 128 bytes a cycle).
  constexpr bool kKeep = R <= 2;
  // rows side by side, so that their gathers overlap, where the registers allow it
  constexpr int G = R == 2 || R == 4 ? 2 : 1;
  struct Entries {
    int c[kClU];
    double v[kClU];
  };
  auto entries = [&](Entries& E, int k, int ke) {
#pragma unroll
    for (int w = 0; w < kClU; ++w) {
      const int e = k + w < ke ? k + w : A.nnz_cap;
      E.c[w] = sent[e];
      E.v[w] = sval[e];
    }
  };
  auto bounds = [&](int u, int& k, int& ke) {
    const int i = min(tid + u * kClThreads, nrow);  // row nrow: empty
    k = srp[i];
    ke = srp[min(i + 1, nrow)];
  };
  Entries kept[kKeep ? R : 1];
  int kbeg[kKeep ? R : 1], kend[kKeep ? R : 1];
  if constexpr (kKeep) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
      bounds(u, kbeg[u], kend[u]);
      entries(kept[u], kbeg[u], kend[u]);
    }
  }
  // sum_j a_ij p_j over the thread's rows, p the new direction: this CTA's own
  // from its p buffer (complete in the CTA), another CTA's formed here from
  // that CTA's z and old p
  auto row_sums = [&](int buf, double beta, double (&out)[R]) {
    const uint32_t zb = base + (uint32_t)L.z;
    const uint32_t dold = (uint32_t)(L.p - L.z) + (buf ? psz : 0u);
    const double* pn = sp(buf ^ 1);
#pragma unroll
    for (int u0 = 0; u0 < R; u0 += G) {
      Entries E[G];
      int k[G], ke[G];
      double s[G];
      bool more = false;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if constexpr (kKeep) {
          E[g] = kept[u0 + g];
          k[g] = kbeg[u0 + g];
          ke[g] = kend[u0 + g];
        } else {
          bounds(u0 + g, k[g], ke[g]);
          entries(E[g], k[g], ke[g]);
        }
        s[g] = 0.0;
        more |= k[g] < ke[g];
      }
      while (more) {
        bool own = true;
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int w = 0; w < kClU; ++w) own &= (E[g].c[w] >> 16) == rank;
        double x[G][kClU];
        if (__all_sync(__activemask(), own)) {
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int w = 0; w < kClU; ++w) x[g][w] = pn[E[g].c[w] & 0xffff];
        } else {
          double pv[G][kClU];
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int w = 0; w < kClU; ++w) {
              const int c = E[g].c[w], owner = c >> 16;
              const bool far = owner != rank;
              const uint32_t at = cl_map(zb + 8u * (uint32_t)(c & 0xffff), (uint32_t)owner);
              x[g][w] = pn[far ? 0 : c & 0xffff];
              pv[g][w] = 0.0;
              cl_ld_if(x[g][w], at, far);
              cl_ld_if(pv[g][w], at + dold, far);
            }
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int w = 0; w < kClU; ++w) x[g][w] = fma(beta, pv[g][w], x[g][w]);
        }
        more = false;
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
          for (int w = 0; w < kClU; ++w) s[g] = fma(E[g].v[w], x[g][w], s[g]);
          k[g] += kClU;
          more |= k[g] < ke[g];
        }
        if (more) {
#pragma unroll
          for (int g = 0; g < G; ++g) entries(E[g], k[g], ke[g]);
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) out[u0 + g] = s[g];
    }
  };
  // Sums over the cluster: each CTA leaves its partials in a slot of its own, and
  // behind one barrier a warp of every CTA fetches all of them and folds them in the
  // same butterfly, so all hold the same bits. Two slots in turn: a CTA writes one
  // again only after a barrier that the others pass behind their reads of it.
  int slot = 0;
  auto totals = [&](double a, double b2, double& ta, double& tb) {
    // both sums folded at once: the lower half-warp takes a, the upper b2
    const bool up = lane >= 16;
    auto fold = [&](double t) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      return t;
    };
    const double got = __shfl_xor_sync(0xffffffffu, up ? a : b2, 16);
    double t = fold((up ? b2 : a) + got);
    if ((lane & 15) == 0) red[up][warp] = t;
    __syncthreads();
    if (warp == 0) {
      t = fold(red[up][lane & 15]);
      if ((lane & 15) == 0) part[slot][up] = t;
    }
    cluster_barrier();
    if (warp == 0) {
      t = 0.0;
      cl_ld_if(t, cl_map(pbase + (uint32_t)(slot * 2 + up) * 8u, (uint32_t)(lane & 15)), (lane & 15) < ncta);
      t = fold(t);
      if ((lane & 15) == 0) bcast[up] = t;
    }
    __syncthreads();
    ta = bcast[0];
    tb = bcast[1];
    slot ^= 1;
  };
  static_assert(kClWarps == 16 && kClMaxCtas == 16, "the folds take 16 partials");

  // r0 = b - A x0, z0 = D^-1 r0, rho = r0.z0 (x was staged in z and the
  // second p buffer, the old p in the first is zero)
  double arr = 0.0, arz = 0.0;
  row_sums(0, 0.0, q);
  cluster_barrier();  // x gathered by every CTA before z takes its place
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int i = tid + u * kClThreads;
    if (i < nrow) {
      r[u] = A.b[r0 + i] - q[u];
      const double zi = r[u] * jv[u];
      sz[i] = zi;
      arr += r[u] * r[u];
      arz += r[u] * zi;
    }
  }
  double rr, rho;
  totals(arr, arz, rr, rho);
  const double rnorm0 = sqrt(rr);
  const double thr = fmax(A.st->tol_abs, A.st->tol_rel * rnorm0);
  const int max_iter = A.st->max_iter;
  int iter = 0, term = CFD_TERM_MAX_ITERATIONS;
  double rn = rnorm0, beta = 0.0;
  if (!isfinite(rnorm0)) {
    term = CFD_TERM_BREAKDOWN;
  } else if (rnorm0 <= thr) {
    term = CFD_TERM_INITIAL_RESIDUAL;
  } else {
    for (int buf = 0;; buf ^= 1) {
      // p = z + beta p into the other buffer, q = A p
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int i = tid + u * kClThreads;
        p[u] = fma(beta, p[u], r[u] * jv[u]);
        if (i < nrow) sp(buf ^ 1)[i] = p[u];
      }
      __syncthreads();
      row_sums(buf, beta, q);
      double apq = 0.0;
#pragma unroll
      for (int u = 0; u < R; ++u)
        if (tid + u * kClThreads < nrow) apq += p[u] * q[u];
      double pq, unused;
      totals(apq, 0.0, pq, unused);
      if (!(pq > 0.0)) {
        term = CFD_TERM_NON_POSITIVE_CURVATURE;
        break;
      }
      const double alpha = rho / pq;
      arr = 0.0;
      arz = 0.0;
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int i = tid + u * kClThreads;
        if (i < nrow) {
          x[u] = x[u] + alpha * p[u];
          r[u] = r[u] - alpha * q[u];
          const double zi = r[u] * jv[u];
          sz[i] = zi;
          arr += r[u] * r[u];
          arz += r[u] * zi;
        }
      }
      double rz;
      totals(arr, arz, rr, rz);
      ++iter;
      beta = rz / rho;
      rho = rz;
      rn = sqrt(rr);
      if (!isfinite(rn)) {
        term = CFD_TERM_BREAKDOWN;
        break;
      }
      if (rn <= thr) {
        term = CFD_TERM_CONVERGED;
        break;
      }
      if (iter >= max_iter) {
        term = CFD_TERM_MAX_ITERATIONS;
        break;
      }
      if (rz == 0.0 || !isfinite(rz)) {
        term = CFD_TERM_BREAKDOWN;
        break;
      }
    }
  }
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int i = tid + u * kClThreads;
    if (i < nrow) A.x[r0 + i] = x[u];
  }
  if (rank == 0 && tid == 0) {
    DevState* st = A.st;
    st->rnorm0 = rnorm0;
    st->threshold = thr;
    st->rnorm = rn;
    st->rr = rn * rn;
    st->iter = iter;
    st->term = term;
    st->done = 1;
  }
  cluster_barrier();  // no CTA leaves while its shared memory may still be read
}

template <int R>
cfd_status cl_launch(cfd_context* ctx, const ClusterArgs& args, int ncta, size_t bytes, bool* launched) {
  auto kern = k_cluster_pcg<R>;
  CFD_TRY(allow_dynamic_smem(kern, ctx->device));
  if (ncta > 8) CFD_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfgl = {};
  cfgl.gridDim = dim3(ncta);
  cfgl.blockDim = dim3(kClThreads);
  cfgl.dynamicSmemBytes = bytes;
  cfgl.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfgl.attrs = attr;
  cfgl.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfgl) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return CFD_OK;
  }
  CFD_TRY_CUDA(cudaLaunchKernelEx(&cfgl, kern, args));
  ctx->stats.launches++;
  *launched = true;
  return CFD_OK;
}

}  // namespace

int64_t scattered_far(const HostCsr& h, int rpc) {
  int64_t cap = 0;
  for (int64_t r = 0; r < h.nrows; r += rpc) {
    const int64_t e = std::min<int64_t>(r + rpc, h.nrows);
    int64_t far = 0;
    for (int64_t i = r; i < e; ++i) {
      const int64_t k0 = h.rp[i], k1 = h.rp[i + 1], up = i > r ? k0 - h.rp[i - 1] : 0;
      if (k0 == k1 || (h.ci[k0] >= r && h.ci[k1 - 1] < e)) continue;  // columns ascend: a row of the block's own
      for (int64_t k = k0; k < k1; ++k)
        if (h.ci[k] < r || h.ci[k] >= e)
          far += k - k0 >= up || h.ci[k - up] + 1 != h.ci[k];
    }
    cap = std::max(cap, far);
  }
  return cap;
}

// The cluster solve applies when the system's rows, split over at most 16
// CTAs, fit their shared memory and registers, and no CTA gathers more than
// kClMaxFar scattered entries from others; *ok = false otherwise (nothing
// launched). What bounds it beyond that is the throughput of remote loads, two an
// entry (about 4.5 ns each where the columns are scattered; a stencil's
// neighbouring rows share theirs), where the grid form stays at 6 to 8 us an
// iteration. Us an iteration in a cluster / on the grid / multi-kernel:
//    1031 scattered entries (1000 rows)   5.7 / 6.7 / 12.9
//    1458 ( 300 rows)                     5.5 / 7.2 / 16.3
//    1563 (2000 rows)                     7.6 / 6.7 / 13.3
//    4794 (8000 rows)                    27.3 / 7.8 / 15.4
//   27-point 16^3 (4232, most of them in runs)  5.8 / 7.3 / 21.3
cfd_status cluster_pcg_solve(cfd_context* ctx, cfd_csr* a, const double* jinv, const double* b, double* x, DevState* st,
                             bool* ok) {
  *ok = false;
  const HostCsr& h = a->host;
  const DevMat& m = a->dev;
  const int64_t n = m.nrows;
  if (n <= 0 || n > (int64_t)kClMaxCtas * kClThreads * kClMaxRows || m.nrows != m.ncols) return CFD_OK;
  int max_smem = 0;
  CFD_TRY_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const size_t budget = (size_t)max_smem - 2048;  // static shared arrays
  // one row per thread where the cluster allows it, more rows per thread at 16 CTAs
  int first = 2;
  while (first < kClMaxCtas && (n + first - 1) / first > kClThreads) first *= 2;
  for (int ncta = first; ncta <= kClMaxCtas; ncta *= 2) {
    const int rpc = (int)((n + ncta - 1) / ncta);
    if (rpc > kClThreads * kClMaxRows) continue;
    int64_t nnz_cap = 0;
    for (int64_t r = 0; r < n; r += rpc) nnz_cap = std::max(nnz_cap, h.rp[std::min<int64_t>(r + rpc, n)] - h.rp[r]);
    const ClusterLayout L = cluster_layout(rpc, (int)std::min<int64_t>(nnz_cap, 1 << 24));
    if (L.bytes > budget) continue;
    if (cluster_scattered(a, 0, rpc) > kClMaxFar) return CFD_OK;
    ClusterArgs args{m.rp, m.col, m.v64, jinv, b, x, st, (int)n, rpc, (int)nnz_cap};
    const int rows = (rpc + kClThreads - 1) / kClThreads;
    if (rows <= 1)
      CFD_TRY(cl_launch<1>(ctx, args, ncta, L.bytes, ok));
    else if (rows <= 2)
      CFD_TRY(cl_launch<2>(ctx, args, ncta, L.bytes, ok));
    else if (rows <= 4)
      CFD_TRY(cl_launch<4>(ctx, args, ncta, L.bytes, ok));
    else if (rows <= 5)
      CFD_TRY(cl_launch<5>(ctx, args, ncta, L.bytes, ok));
    else
      CFD_TRY(cl_launch<8>(ctx, args, ncta, L.bytes, ok));
    if (*ok) return CFD_OK;
  }
  return CFD_OK;
}

}  // namespace cfd
