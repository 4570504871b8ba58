// CG and Jacobi-PCG (krylov::cg[_preconditioned], krylov.rs:318-360, with
// DiagJacobi) in FP64 for systems beyond one cluster whose rows fit the shared
// memory and registers of the whole GPU (five-point systems to about 380 000
// rows): one cooperative grid of one CTA per SM iterates on data that never
// leaves the SMs but for the vectors other CTAs read.
//
// What bounds it: the multi-kernel iteration is three launches (update 6.6 us,
// SpMV with its reduction 5.3 us, direction 2.4 us at 123 300 rows) on data that
// sits in L2. Here an iteration is bound by two grid-wide reductions and one
// exchange of boundary entries, each a store to L2 and the others' polls of it.
// No fence is on that path: a double travels as NCCL's LL protocol sends data, in
// two 8-byte words of 32 data and 32 flag bits (the number of the reduction or
// iteration), each stored and loaded as one 64-bit access, so a reader that sees
// a word's flag has its data. (With fences around flags and sums read apart the same
// kernel took 15 us an iteration, more than the three launches' 13.) Measured,
// five-point Jacobi-CG to 1e-10, before (multi-kernel) and now: 256 x 256 10.6
// -> 5.4 ms, 411 x 300 18.6 -> 8.8 ms, 600 x 620 46.4 -> 20.1 ms. Half the CTAs
// (fewer polls, more rows each): 5.0, 9.4 ms and no room for the third.
//
// A thread owns R rows: x, r, p, q, D^-1, and up to two rows a thread the first
// entries of the matrix, in registers. Shared memory holds the matrix rows and
// the direction p of the CTA's rows and of its boundary: one slot per entry that
// lies in another CTA's rows. Owners publish z = D^-1 r; a boundary slot's new
// direction is z_j + beta p_j formed where it is used, the same operations as
// the owner's, so p itself never travels. A z is published over the last one
// only after a reduction every reader has contributed to behind its read. Every
// CTA sums all partial sums in the same order, so all hold the same bits and
// take the same branches.
//
// The launch is cooperative (all CTAs resident). Every wait is bounded: one that
// runs out sets the context's error word and the CTA leaves; the others' waits
// then run out too. A launch runs at most kGpIters iterations and the host
// launches again until the state is done; x, r, p, the published z and the
// scalars are in global memory between launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "internal.h"
#include "kernels.cuh"

namespace cfd {
namespace {

constexpr int kGpThreads = 512;
constexpr int kGpWarps = kGpThreads / 32;
constexpr int kGpU = 5;          // entries of a row read together (a five-point row)
constexpr int kGpIters = 160;    // iterations of one launch at most
constexpr int kGpMaxGrid = 160;  // CTAs whose sums one round of five warps reads
constexpr unsigned kGpSpin = 1u << 21;  // polls of a word, an L2 round trip each: about a second

struct GridArgs {
  const int* __restrict__ rp;
  const int* __restrict__ col;
  const double* __restrict__ val;
  const double* __restrict__ jinv;  // nullptr: no preconditioner
  const double* __restrict__ b;
  double* x;
  double* r;    // residual and direction between launches
  double* p;
  ulonglong2* z;     // published D^-1 r of all rows
  ulonglong2* sums;  // published partial sums: two buffers of two per CTA
  DevState* st;
  int* err;
  int n, rpc, nnz_cap, far_cap, first;
  unsigned spin;  // polls of a word before a wait gives up (LIMIT only)
};

struct GridLayout {
  size_t val, ent, rpl, far, p, bytes;
};
__host__ __device__ inline size_t gp_round16(size_t b) { return (b + 15) / 16 * 16; }
__host__ __device__ inline GridLayout grid_layout(int rpc, int nnz_cap, int far_cap) {
  GridLayout L;
  L.val = 0;  // nnz_cap values and a zero entry
  L.ent = gp_round16((size_t)(nnz_cap + 1) * 8);
  L.rpl = L.ent + gp_round16((size_t)(nnz_cap + 1) * 4);
  L.far = L.rpl + gp_round16((size_t)(rpc + 1) * 4);
  L.p = L.far + gp_round16((size_t)far_cap * 4);
  L.bytes = L.p + gp_round16((size_t)(rpc + far_cap + 1) * 8);  // and a slot that stays zero
  return L;
}

// A double as two 8-byte words, each 32 bits of it (low) and the flag (high). The
// elements of the vector access are 64 bits wide: PTX makes no promise for a word
// made of two 32-bit elements.
__device__ __forceinline__ void gp_publish(ulonglong2* to, double v, unsigned flag) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v), f = (unsigned long long)flag << 32;
  asm volatile("st.volatile.global.v2.b64 [%0], {%1, %2};" ::"l"(to), "l"((bits & 0xffffffffull) | f),
               "l"((bits >> 32) | f)
               : "memory");
}
__device__ __forceinline__ bool gp_read(const ulonglong2* from, unsigned flag, double& v) {
  unsigned long long a, b;
  asm volatile("ld.volatile.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(from) : "memory");
  v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
  return (unsigned)(a >> 32) == flag && (unsigned)(b >> 32) == flag;
}
// Polls until the flag is there; false when the wait runs out.
__device__ __forceinline__ bool gp_wait(const ulonglong2* from, unsigned flag, double& v, unsigned spin) {
  for (unsigned tries = 0; tries < spin; ++tries)
    if (gp_read(from, flag, v)) return true;
  return false;
}

// LIMIT: the self test's form, whose waits give up after A.spin polls. The solve's
// bound is a constant: as an argument it made the polls slower (411 x 300 8.5 -> 10.9
// ms).
template <int R, bool LIMIT = false>
__global__ void __launch_bounds__(kGpThreads, 1) k_grid_pcg(GridArgs A) {
  const unsigned spin = LIMIT ? A.spin : kGpSpin;
  if (!A.first && A.st->done) return;  // the same in every CTA: written by an earlier launch
  extern __shared__ __align__(16) unsigned char sm[];
  const GridLayout L = grid_layout(A.rpc, A.nnz_cap, A.far_cap);
  double* sval = reinterpret_cast<double*>(sm + L.val);
  int* sent = reinterpret_cast<int*>(sm + L.ent);  // local row, or rows + boundary slot
  int* srp = reinterpret_cast<int*>(sm + L.rpl);
  int* sfar = reinterpret_cast<int*>(sm + L.far);  // row of a boundary slot
  double* sp = reinterpret_cast<double*>(sm + L.p);
  __shared__ int s_far;
  __shared__ double red[2][kGpWarps];
  __shared__ double red2[2][kGpMaxGrid / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ncta = (int)gridDim.x;
  const int r0 = blockIdx.x * A.rpc;
  const int nrow = max(0, min(A.rpc, A.n - r0));
  const int k0 = nrow > 0 ? A.rp[r0] : 0;
  const int nnz = nrow > 0 ? A.rp[r0 + nrow] - k0 : 0;
  if (tid == 0) s_far = 0;
  __syncthreads();
  for (int i = tid; i <= nrow; i += kGpThreads) srp[i] = nrow > 0 ? A.rp[r0 + i] - k0 : 0;
  for (int e = tid; e < nnz; e += kGpThreads) {
    const int c = A.col[k0 + e];
    int slot = c - r0;
    if (c < r0 || c >= r0 + nrow) {
      const int f = min(atomicAdd(&s_far, 1), A.far_cap - 1);  // the host sized far_cap to the count
      sfar[f] = c;
      slot = nrow + f;
    }
    sent[e] = slot;
    sval[e] = A.val[k0 + e];
  }
  if (tid == 0) {  // the zero entry: a slot that stays zero, times 0
    sent[A.nnz_cap] = A.rpc + A.far_cap;
    sval[A.nnz_cap] = 0.0;
    sp[A.rpc + A.far_cap] = 0.0;
  }
  const int iter0 = A.first ? 0 : A.st->iter;
  double x[R], r[R], p[R], q[R], jv[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int i = tid + u * kGpThreads;
    const bool live = i < nrow;
    x[u] = live ? A.x[r0 + i] : 0.0;
    jv[u] = live ? (A.jinv ? A.jinv[r0 + i] : 1.0) : 0.0;
    r[u] = p[u] = q[u] = 0.0;
    if (live && !A.first) {
      r[u] = A.r[r0 + i];
      p[u] = A.p[r0 + i];
    }
    if (live) sp[i] = x[u];
  }
  __syncthreads();
  const int nfar = min(s_far, A.far_cap);
  // a boundary slot starts as x (for the first residual) or its row's direction
  for (int f = tid; f < nfar; f += kGpThreads) sp[nrow + f] = A.first ? A.x[sfar[f]] : A.p[sfar[f]];
  __syncthreads();

  // Up to two rows a thread keep their first kGpU entries in registers.
  constexpr bool kKeep = R <= 2;
  constexpr int G = R == 2 || R == 4 ? 2 : 1;  // rows side by side, so that their gathers overlap
  struct Entries {
    int c[kGpU];
    double v[kGpU];
  };
  auto entries = [&](Entries& E, int k, int ke) {
#pragma unroll
    for (int w = 0; w < kGpU; ++w) {
      const int e = k + w < ke ? k + w : A.nnz_cap;
      E.c[w] = sent[e];
      E.v[w] = sval[e];
    }
  };
  auto bounds = [&](int u, int& k, int& ke) {
    const int i = min(tid + u * kGpThreads, nrow);  // row nrow: empty
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
  // sum_j a_ij p_j over the thread's rows, p in shared memory
  auto row_sums = [&](double (&out)[R]) {
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
        double y[G][kGpU];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int w = 0; w < kGpU; ++w) y[g][w] = sp[E[g].c[w]];
        more = false;
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
          for (int w = 0; w < kGpU; ++w) s[g] = fma(E[g].v[w], y[g][w], s[g]);
          k[g] += kGpU;
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
  // Grid-wide sums of a and (two) b2, reduction number `epoch`, rising by one.
  // False when a wait ran out. The two sums are polled one after the other: the
  // polls of all CTAs load L2, and polling both at once, or with pauses between
  // polls, cost 7.9 against 6.4 us an iteration at 411 x 300.
  const bool up = lane >= 16;
  auto fold = [&](double t) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  };
  auto half = [&](double a, double b2) {  // lower half-warp a, upper b2, each summed over the warp
    const double got = __shfl_xor_sync(0xffffffffu, up ? a : b2, 16);
    return fold((up ? b2 : a) + got);
  };
  auto totals = [&](unsigned epoch, bool two, double a, double b2, double& ta, double& tb) -> bool {
    ulonglong2* sums = A.sums + (size_t)(epoch & 1u) * 2 * kGpMaxGrid;
    double t = half(a, b2);
    if ((lane & 15) == 0) red[up][warp] = t;
    __syncthreads();
    if (warp == 0) {
      t = fold(red[up][lane & 15]);
      if ((lane & 15) == 0 && (two || !up)) gp_publish(sums + 2 * blockIdx.x + (up ? 1 : 0), t, epoch);
    }
    double va = 0.0, vb = 0.0;
    int bad = 0;
    if (tid < ncta) {
      bad = !gp_wait(sums + 2 * tid, epoch, va, spin);
      if (two && !bad) bad = !gp_wait(sums + 2 * tid + 1, epoch, vb, spin);
      if (bad) atomicExch(A.err, 1);
    }
    if (warp < kGpMaxGrid / 32) {
      t = half(va, vb);
      if ((lane & 15) == 0) red2[up][warp] = t;
    }
    if (__syncthreads_or(bad)) return false;
    ta = tb = 0.0;
#pragma unroll
    for (int w = 0; w < kGpMaxGrid / 32; ++w) {
      ta += red2[0][w];
      tb += red2[1][w];
    }
    return true;
  };
  static_assert(kGpWarps == 16 && kGpMaxGrid <= kGpThreads && kGpMaxGrid % 32 == 0, "the folds take 16 partials");

  double rr, rho, rn0, rn, thr, beta;
  int iter = iter0, term = CFD_TERM_MAX_ITERATIONS;
  const int max_iter = A.st->max_iter;
  bool done = false;
  if (A.first) {
    // r0 = b - A x0, z0 = D^-1 r0, rho = r0.z0
    row_sums(q);
    double arr = 0.0, arz = 0.0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = tid + u * kGpThreads;
      if (i < nrow) {
        r[u] = A.b[r0 + i] - q[u];
        const double zi = r[u] * jv[u];
        gp_publish(A.z + r0 + i, zi, 1u);
        arr += r[u] * r[u];
        arz += r[u] * zi;
      }
    }
    if (!totals(1u, true, arr, arz, rr, rho)) return;
    rn0 = rn = sqrt(rr);
    thr = fmax(A.st->tol_abs, A.st->tol_rel * rn0);
    beta = 0.0;
    for (int f = tid; f < nfar; f += kGpThreads) sp[nrow + f] = 0.0;  // no direction yet
    if (!isfinite(rn0)) {
      term = CFD_TERM_BREAKDOWN;
      done = true;
    } else if (rn0 <= thr) {
      term = CFD_TERM_INITIAL_RESIDUAL;
      done = true;
    }
  } else {
    rho = A.st->rho;
    beta = A.st->beta;
    rn0 = A.st->rnorm0;
    rn = A.st->rnorm;
    thr = A.st->threshold;
  }
  while (!done && iter < iter0 + kGpIters) {
    // p = z + beta p, the boundary's from the owners' z; q = A p
    int bad = 0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = tid + u * kGpThreads;
      p[u] = fma(beta, p[u], r[u] * jv[u]);
      if (i < nrow) sp[i] = p[u];
    }
    for (int f = tid; f < nfar; f += kGpThreads) {
      double zf;
      if (!gp_wait(A.z + sfar[f], (unsigned)iter + 1u, zf, spin)) bad = 1;
      sp[nrow + f] = fma(beta, sp[nrow + f], zf);
    }
    if (bad) atomicExch(A.err, 1);
    if (__syncthreads_or(bad)) return;
    row_sums(q);
    double apq = 0.0;
#pragma unroll
    for (int u = 0; u < R; ++u)
      if (tid + u * kGpThreads < nrow) apq += p[u] * q[u];
    double pq, unused;
    if (!totals(2u * (unsigned)iter + 2u, false, apq, 0.0, pq, unused)) return;
    if (!(pq > 0.0)) {
      term = CFD_TERM_NON_POSITIVE_CURVATURE;
      done = true;
      break;
    }
    const double alpha = rho / pq;
    double arr = 0.0, arz = 0.0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = tid + u * kGpThreads;
      if (i < nrow) {
        x[u] = x[u] + alpha * p[u];
        r[u] = r[u] - alpha * q[u];
        const double zi = r[u] * jv[u];
        gp_publish(A.z + r0 + i, zi, (unsigned)iter + 2u);
        arr += r[u] * r[u];
        arz += r[u] * zi;
      }
    }
    double rz;
    if (!totals(2u * (unsigned)iter + 3u, true, arr, arz, rr, rz)) return;
    ++iter;
    beta = rz / rho;
    rho = rz;
    rn = sqrt(rr);
    if (!isfinite(rn)) {
      term = CFD_TERM_BREAKDOWN;
      done = true;
    } else if (rn <= thr) {
      term = CFD_TERM_CONVERGED;
      done = true;
    } else if (iter >= max_iter) {
      term = CFD_TERM_MAX_ITERATIONS;
      done = true;
    } else if (rz == 0.0 || !isfinite(rz)) {
      term = CFD_TERM_BREAKDOWN;
      done = true;
    }
  }
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int i = tid + u * kGpThreads;
    if (i < nrow) {
      A.x[r0 + i] = x[u];
      A.r[r0 + i] = r[u];
      A.p[r0 + i] = p[u];
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    // every CTA read the state before its first reduction, which this CTA has passed
    DevState* st = A.st;
    st->rho = rho;
    st->beta = beta;
    st->rnorm0 = rn0;
    st->threshold = thr;
    st->rnorm = rn;
    st->rr = rn * rn;
    st->iter = iter;
    st->term = term;
    st->done = done ? 1 : 0;
  }
}

template <int R, bool LIMIT = false>
cfd_status gp_launch(cfd_context* ctx, GridArgs& A, int grid, size_t bytes, bool probe, bool* fits) {
  auto kern = k_grid_pcg<R, LIMIT>;
  if (probe) {  // once a solve, before its launches
    CFD_TRY(allow_dynamic_smem(kern, ctx->device));
    int occ = 0;
    CFD_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kGpThreads, bytes));
    *fits = occ >= 1;
    return CFD_OK;
  }
  void* args[] = {&A};
  CFD_TRY_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kGpThreads), args, bytes, ctx->stream));
  ctx->stats.launches++;
  return CFD_OK;
}

cfd_status gp_launch_rows(cfd_context* ctx, GridArgs& A, int rows, int grid, size_t bytes, bool probe, bool* fits) {
  if (rows <= 1) return gp_launch<1>(ctx, A, grid, bytes, probe, fits);
  if (rows <= 2) return gp_launch<2>(ctx, A, grid, bytes, probe, fits);
  if (rows <= 3) return gp_launch<3>(ctx, A, grid, bytes, probe, fits);
  if (rows <= 4) return gp_launch<4>(ctx, A, grid, bytes, probe, fits);
  if (rows <= 5) return gp_launch<5>(ctx, A, grid, bytes, probe, fits);
  return gp_launch<8>(ctx, A, grid, bytes, probe, fits);
}

// Entries of the fullest block of rpc rows that lie outside that block's rows.
int64_t gp_far_cap(const HostCsr& h, int rpc) {
  int64_t cap = 0;
  for (int64_t r = 0; r < h.nrows; r += rpc) {
    const int64_t e = std::min<int64_t>(r + rpc, h.nrows);
    int64_t far = 0;
    for (int64_t k = h.rp[r]; k < h.rp[e]; ++k) far += h.ci[k] < r || h.ci[k] >= e;
    cap = std::max(cap, far);
  }
  return cap;
}

}  // namespace

// The grid CG applies when the rows, split over the GPU's SMs, and their
// boundaries fit their shared memory and eight rows a thread; *ok = false
// otherwise (nothing launched).
cfd_status grid_pcg_solve(cfd_context* ctx, cfd_csr* a, const double* jinv, const double* b, double* x, DevState* st,
                          DevState* host_st, bool* ok) {
  *ok = false;
  const HostCsr& h = a->host;
  const DevMat& m = a->dev;
  const int64_t n = m.nrows;
  const int grid = std::min(ctx->num_sms, kGpMaxGrid);
  if (n <= 0 || n > (int64_t)grid * kGpThreads * 8 || m.nrows != m.ncols) return CFD_OK;
  int max_smem = 0, coop = 0;
  CFD_TRY_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  CFD_TRY_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
  if (!coop) return CFD_OK;
  const int rpc = (int)((n + grid - 1) / grid);
  int64_t nnz_cap = 0;
  for (int64_t r = 0; r < n; r += rpc) nnz_cap = std::max(nnz_cap, h.rp[std::min<int64_t>(r + rpc, n)] - h.rp[r]);
  const size_t budget = (size_t)max_smem - 2048;  // static shared arrays
  if (nnz_cap > (int64_t)budget / 12) return CFD_OK;
  // the boundary's size follows from the pattern, which a matrix keeps for life
  if (a->grid_far < 0) a->grid_far = gp_far_cap(h, rpc);
  if (a->grid_far > (int64_t)budget / 12) return CFD_OK;
  const int far_cap = std::max(1, (int)a->grid_far);
  const GridLayout L = grid_layout(rpc, (int)nnz_cap, far_cap);
  if (L.bytes > budget) return CFD_OK;
  const int rows = (rpc + kGpThreads - 1) / kGpThreads;
  GridArgs A{m.rp, m.col, m.v64, jinv, b, x, nullptr, nullptr, nullptr, nullptr, st, ctx->err, (int)n, rpc,
             (int)nnz_cap, far_cap, 1, 0};
  bool fits = false;
  CFD_TRY(gp_launch_rows(ctx, A, rows, grid, L.bytes, true, &fits));
  if (!fits) return CFD_OK;
  // published sums and z (zeroed: no flag set), r, p
  const size_t words = 4 * (size_t)kGpMaxGrid + (size_t)n;
  ulonglong2* ws = nullptr;
  if (cudaMallocAsync((void**)&ws, words * sizeof(ulonglong2) + 2 * (size_t)n * sizeof(double), ctx->stream) !=
      cudaSuccess) {
    cudaGetLastError();
    return CFD_OK;  // the multi-kernel solve reports an allocation that fails there too
  }
  A.sums = ws;
  A.z = ws + 4 * (size_t)kGpMaxGrid;
  A.r = reinterpret_cast<double*>(ws + words);
  A.p = A.r + n;
  cfd_status s = CFD_OK;
  cudaError_t e = cudaMemsetAsync(ws, 0, words * sizeof(ulonglong2), ctx->stream);
  // two launches between looks at the state: one that finds the solve done returns at once
  while (e == cudaSuccess && s == CFD_OK) {
    for (int k = 0; k < 2 && s == CFD_OK; ++k) {
      s = gp_launch_rows(ctx, A, rows, grid, L.bytes, false, &fits);
      A.first = 0;
    }
    if (s != CFD_OK) break;
    e = cudaMemcpyAsync(host_st, st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_err, ctx->err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess || host_st->done || *ctx->h_err != 0) break;
  }
  if (e != cudaSuccess) {
    set_error("grid CG: %s", cudaGetErrorString(e));
    s = CFD_ERR_CUDA;
  }
  cudaFreeAsync(ws, ctx->stream);
  CFD_TRY(s);
  CFD_TRY(check_device_flag(ctx));  // a wait that ran out
  *ok = true;
  return CFD_OK;
}

}  // namespace cfd

// The grid CG's own wait on a flag that nothing sets: a launch that goes on from a
// state whose directions were never published, with a small bound.
cfd_status cfd_selftest_grid_wait_timeout(cfd_context* ctx, int32_t tries) {
  using namespace cfd;
  if (!ctx || tries < 1) {
    set_error("cfd_selftest_grid_wait_timeout: null context or tries < 1");
    return CFD_ERR_CONFIG;
  }
  return guarded("cfd_selftest_grid_wait_timeout", [&]() -> cfd_status {
    std::lock_guard<std::mutex> g(ctx->mu);
    CFD_TRY_CUDA(cudaSetDevice(ctx->device));
    const int grid = std::min(ctx->num_sms, kGpMaxGrid), rpc = 4, n = rpc * grid, nnz = 3 * n - 2;
    std::vector<int> rp(n + 1, 0), col;
    for (int i = 0; i < n; ++i) {
      for (int j = std::max(0, i - 1); j <= std::min(n - 1, i + 1); ++j) col.push_back(j);
      rp[i + 1] = (int)col.size();
    }
    // zeroed: vectors and values, published words (no flag set), the state (not done, iteration 0)
    const size_t words = 4 * (size_t)kGpMaxGrid + (size_t)n;
    const size_t bytes = words * sizeof(ulonglong2) + ((size_t)nnz + 5 * (size_t)n) * sizeof(double) + sizeof(DevState);
    char* ws = nullptr;
    int *drp = nullptr, *dcol = nullptr;
    auto run = [&]() -> cfd_status {
      CFD_TRY_CUDA(cudaMalloc((void**)&ws, bytes));
      CFD_TRY_CUDA(cudaMalloc((void**)&drp, rp.size() * sizeof(int)));
      CFD_TRY_CUDA(cudaMalloc((void**)&dcol, col.size() * sizeof(int)));
      CFD_TRY_CUDA(cudaMemsetAsync(ws, 0, bytes, ctx->stream));
      CFD_TRY_CUDA(cudaMemcpyAsync(drp, rp.data(), rp.size() * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
      CFD_TRY_CUDA(cudaMemcpyAsync(dcol, col.data(), col.size() * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
      GridArgs A{};
      A.sums = reinterpret_cast<ulonglong2*>(ws);
      A.z = A.sums + 4 * (size_t)kGpMaxGrid;
      double* v = reinterpret_cast<double*>(ws + words * sizeof(ulonglong2));
      A.val = v;
      A.b = v + nnz;
      A.x = v + nnz + n;
      A.r = v + nnz + 2 * n;
      A.p = v + nnz + 3 * n;
      A.st = reinterpret_cast<DevState*>(v + nnz + 5 * (size_t)n);
      A.rp = drp;
      A.col = dcol;
      A.err = ctx->err;
      A.n = n;
      A.rpc = rpc;
      A.nnz_cap = 3 * rpc;
      A.far_cap = 2;
      A.first = 0;
      A.spin = (unsigned)tries;
      const GridLayout L = grid_layout(rpc, A.nnz_cap, A.far_cap);
      bool fits = false;
      CFD_TRY((gp_launch<1, true>(ctx, A, grid, L.bytes, true, &fits)));
      CFD_TRY((gp_launch<1, true>(ctx, A, grid, L.bytes, false, &fits)));
      return check_device_flag(ctx);
    };
    const cfd_status s = run();
    cudaFree(ws);
    cudaFree(drp);
    cudaFree(dcol);
    return s;
  });
}
