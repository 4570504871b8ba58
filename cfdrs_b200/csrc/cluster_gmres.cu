// Whole-solve GMRES(m) for small systems in one thread-block cluster: the
// restarted, right-preconditioned GMRES of krylov::gmres[_preconditioned]
// (krylov.rs:150-246) in FP64, with no preconditioner, Jacobi, or the whole
// AMG V-cycle (amg.rs:423-503), for systems whose matrix and hierarchy fit the
// shared memory of a cluster of up to 16 CTAs. The 2-D pressure correction
// (GMRES(30) with AMG below 10 000 rows, correction.rs:40-168) is the caller
// this is for.
//
// What bounds it: nothing but latency. One Arnoldi step of that caller is a
// V(2,2)-cycle over five or six levels, an SpMV and three reductions, 53
// dependent passes over a few hundred kilobytes. As kernels each pass costs 4
// us (launch, descriptor, staging and gather latencies); here a pass is a
// cluster barrier (450 cycles with release and acquire), shared-memory matrix
// reads made before that barrier, and one gather from the owner's shared memory
// (325 cycles when remote). Measured, GMRES(30) with the pressure AMG to 1e-10:
// 47 x 35 cells 18.0 -> 2.8 ms, 101 x 98 cells 65 -> 13 ms.
//
// Layout: the rows of every level are split over the CTAs in equal blocks. A
// CTA keeps its rows of A, R and P (values, columns as owner << 12 | index) and
// its slices of the level vectors in shared memory; gathered entries of other
// CTAs are read through distributed shared memory. From the first level of at
// most kTailRows rows down, the cycle is one fixed linear map of that level's
// right-hand side: at the start every CTA runs it on its share of the unit
// vectors (its own copy of those small levels, CTA barriers only) and the rest
// of the solve applies the resulting dense matrix, one pass instead of 16 to 20.
// The Krylov basis stays in shared memory where it fits, else in global memory:
// a CTA only ever reads the rows it wrote. A dot product is a per-warp partial
// pushed to every CTA's shared memory, one cluster barrier, and every CTA
// summing the partials in rank order, so all CTAs hold the same bits, apply the
// same Givens rotations and take the same branches. The barriers are the
// hardware cluster barrier and control flow is uniform across the cluster.
//
// The sweeps, residuals and transfers are the V-cycle's operations with another
// summation order in the rows (several threads a row), and the dot products use
// another summation tree than k_mdot, so iterates agree with the multi-kernel
// solve to rounding.
//
// A launch runs at most kGcStepsPerLaunch Arnoldi steps (whole cycles) and the
// host launches again until the state is done, so no launch is unbounded.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "amg_device.h"
#include "internal.h"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace cfd {
namespace {

constexpr int kGcThreads = 640;
constexpr int kGcWarps = kGcThreads / 32;
constexpr int kGcMaxCtas = 16;
constexpr int kGcMaxLevels = 10;
constexpr int kGcMaxRestart = 64;
constexpr int kTailRows = 128;          // levels up to this size are applied as one dense matrix
constexpr int kGcRowsPerCta = 64;     // smallest block worth another CTA
constexpr int kGcIdxBits = 12;          // local index bits of a packed column
constexpr int kGcMaxDense = 512;        // rows of a dense coarsest solve at most
constexpr int kGcStepsPerLaunch = 4096;
constexpr int kGcMaxPhases = 128;
constexpr int kGcMaxFar = 14000;        // scattered entries of other CTAs (cluster_gmres_solve)

enum { kGcNone = 0, kGcJacobi = 1, kGcAmg = 2 };

// One matrix in a CTA's shared memory: byte offsets of the row offsets
// (uint16, rows per CTA + 1), packed columns (uint16) and values, and its
// global CSR. Rows are split like the vectors of row partition rpc_r, columns
// name entries of partition rpc_c.
struct GcMat {
  const int* __restrict__ rp;
  const int* __restrict__ col;
  const double* __restrict__ val;
  int n, rpc_r, rpc_c;
  int solo;  // every CTA holds all rows and gathers from itself
  int o_rp, o_col, o_val;
  int zero, tl;  // index of an entry with value 0; log2 of the threads on a row
};

// One level: A (and R to the next level, P from it), vector offsets.
struct GcLevel {
  GcMat A, R, P;
  const double* __restrict__ diag;
  int n, rpc;
  int o_b, o_xa, o_xb, o_r, o_d;  // o_d: 1 / a_ii, NaN where the smoother skips the row
};

// One pass of the V-cycle over the rows of a level. The V-cycle is a list of
// these, built on the host, so that every pass runs the same few hundred
// instructions: written out level by level the code outgrew the instruction
// cache and a pass took 3000 cycles.
//   kGcSmooth0   out = w b rd
//   kGcSweep     out = old + w (b - s) rd
//   kGcResidual  out = b - s
//   kGcRestrict  out = s and the level's first sweep (or 0) in out2
//   kGcProlong   out = old + s
//   kGcDense     out = D b, D the coarsest inverse (global memory)
//   kGcTail      out = D b, D the tail's matrix (shared memory)
// s = sum_j a_ij x_j over the row of the pass's matrix, 1 << tl threads a row.
// Offsets are bytes of shared memory; `rows` holds the level's rows, and the
// CTA's own once loaded; `zero` is the index of the matrix's zero entry.
enum { kGcSmooth0 = 0, kGcSweep, kGcResidual, kGcRestrict, kGcProlong, kGcDense, kGcTail };
struct __align__(16) GcPhase {
  int type, zero_start, rows, o_rp;
  int o_col, o_val, o_x, o_out;
  int o_b, o_rd, o_out2, o_old;
  int rpc, zero, tl, cols;
};

struct GcArgs {
  GcLevel lev[kGcMaxLevels];   // split levels; the last of them may be the tail's finest
  GcLevel solo[kGcMaxLevels];  // the tail's levels, whole in every CTA
  GcMat M;  // the operator of the solve (the hierarchy has its own copy)
  const double* __restrict__ jinv;
  const double* __restrict__ inv;  // dense inverse of the coarsest operator or nullptr
  const double* __restrict__ b;
  const GcPhase* __restrict__ program;
  double* x;
  double* rg;    // residual, kept between launches
  double* V;     // (m + 1) x n basis
  double* H;     // m columns of m + 1 (rank 0's copy)
  DevState* st;
  double omega;
  int levels, solo_levels, m, resume;
  int phases, solo_phases, o_z, o_solo_z;  // o_z: where the V-cycle leaves its result
  int o_tail;                              // the tail's matrix, this CTA's rows
  int n, rpc;
  int o_w, o_part, o_h, o_cs, o_sn, o_g, o_y, o_stage, o_prog;
  int o_v, smem_bytes;  // o_v: the basis in shared memory, or -1 (global memory)
};

__device__ __forceinline__ uint32_t gc_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t gc_map(uint32_t a, uint32_t rank) {
  uint32_t d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}
// Loads and stores of the cluster's shared memory. Volatile keeps them between
// the barriers that order them; consecutive loads still overlap.
__device__ __forceinline__ double gc_ld(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
// This CTA's own shared memory by 32-bit address (a generic load costs more).
__device__ __forceinline__ double gc_own(uint32_t a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void gc_put(uint32_t a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ int gc_u16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void gc_st(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

struct GcCta {
  unsigned char* sm;
  uint32_t base;  // shared address of sm
  int rank, ncta;
  __device__ double* d(int off) const { return reinterpret_cast<double*>(sm + off); }
};

__device__ __forceinline__ int gc_rows(int n, int rpc, int rank) { return max(0, min(rpc, n - rank * rpc)); }

// This CTA's rows of a matrix into shared memory.
__device__ void gc_stage(const GcMat& A, const GcCta& C) {
  const int rank = A.solo ? 0 : C.rank;
  const int r0 = rank * A.rpc_r, nr = gc_rows(A.n, A.rpc_r, rank);
  if (nr <= 0) return;
  const int k0 = A.rp[r0], nnz = A.rp[r0 + nr] - k0;
  uint16_t* rp = reinterpret_cast<uint16_t*>(C.sm + A.o_rp);
  uint16_t* cl = reinterpret_cast<uint16_t*>(C.sm + A.o_col);
  double* v = C.d(A.o_val);
  for (int i = threadIdx.x; i <= nr; i += kGcThreads) rp[i] = (uint16_t)(A.rp[r0 + i] - k0);
  for (int e = threadIdx.x; e < nnz; e += kGcThreads) {
    const int c = A.col[k0 + e], o = c / A.rpc_c;
    cl[e] = (uint16_t)(((A.solo ? C.rank : o) << kGcIdxBits) | (c - o * A.rpc_c));
    v[e] = A.val[k0 + e];
  }
  if (threadIdx.x == 0) {
    cl[A.zero] = (uint16_t)((C.rank << kGcIdxBits) | A.rpc_c);  // the slot behind this CTA's slice: stays zero
    v[A.zero] = 0.0;
  }
}
// 1 / a_ii of a level's rows in this CTA.
__device__ void gc_stage_diag(const GcLevel& L, bool solo, const GcCta& C) {
  const int rank = solo ? 0 : C.rank, q0 = rank * L.rpc, nq = gc_rows(L.n, L.rpc, rank);
  for (int i = threadIdx.x; i < nq; i += kGcThreads) {
    const double d = L.diag[q0 + i];
    C.d(L.o_d)[i] = diag_ok<double>(d) ? 1.0 / d : CUDART_NAN;
  }
}

// A row's entries ka, ka + step, ... below ke of a matrix, U at a time: values
// and the gathered entries' cluster addresses. Slots past the end take the
// matrix's zero entry, so the loads carry no branches and overlap; it names a slot
// of the vector that stays zero, so no vector entry reaches a row without its column.
constexpr int kGcU = 5;  // a five-point row in one batch
struct GcBatch {
  double v[kGcU];
  uint32_t at[kGcU];
};
__device__ __forceinline__ void gc_fetch(GcBatch& B, uint32_t base, int o_col, int o_val, int o_x, int k, int ke,
                                         int step, int zero) {
  constexpr uint32_t kIdx = (1u << kGcIdxBits) - 1u;
  const uint32_t cb = base + (uint32_t)o_col, vb = base + (uint32_t)o_val, xb = base + (uint32_t)o_x;
  int e[kGcU];
  uint32_t c[kGcU];
#pragma unroll
  for (int u = 0; u < kGcU; ++u) e[u] = k + u * step < ke ? k + u * step : zero;
#pragma unroll
  for (int u = 0; u < kGcU; ++u) c[u] = (uint32_t)gc_u16(cb + 2u * (uint32_t)e[u]);
#pragma unroll
  for (int u = 0; u < kGcU; ++u) B.v[u] = gc_own(vb + 8u * (uint32_t)e[u]);
#pragma unroll
  for (int u = 0; u < kGcU; ++u) B.at[u] = gc_map(xb + 8u * (c[u] & kIdx), c[u] >> kGcIdxBits);
}
__device__ __forceinline__ double gc_gather(const GcBatch& B, double s) {
  double x[kGcU];
#pragma unroll
  for (int u = 0; u < kGcU; ++u) x[u] = gc_ld(B.at[u]);
#pragma unroll
  for (int u = 0; u < kGcU; ++u) s = fma(B.v[u], x[u], s);
  return s;
}

// f(i, row sum) for this CTA's nr rows of a matrix.
template <class F>
__device__ __forceinline__ void gc_spmv(const GcMat& M, uint32_t base, int nr, int o_x, F f) {
  const int tl = M.tl, step = 1 << tl, part = threadIdx.x & (step - 1);
  const int live = (nr + (32 >> tl) - 1) & ~((32 >> tl) - 1);  // whole warps
  for (int r = threadIdx.x >> tl; r < live; r += kGcThreads >> tl) {
    const uint32_t ra = base + (uint32_t)M.o_rp + 2u * (uint32_t)min(r, nr - 1);
    const int ke = gc_u16(ra + 2u);
    double s = 0.0;
    for (int k = gc_u16(ra) + part; k < ke; k += kGcU * step) {
      GcBatch B;
      gc_fetch(B, base, M.o_col, M.o_val, o_x, k, ke, step, M.zero);
      s = gc_gather(B, s);
    }
    for (int o = step >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (part == 0 && r < nr) f(r, s);
  }
}

// First sweep from zero, w b / a_ii with the stored 1 / a_ii (NaN where the
// smoother skips the row, smooth0_value).
__device__ __forceinline__ double gc_smooth0(double b, double rd, double omega) {
  return rd == rd ? omega * (b * rd) : 0.0;
}

// Runs a program's passes. Before the barrier that a pass's gathers wait for,
// every thread already holds its row's matrix entries and gather addresses, so
// behind the barrier are one gather, the sum and the update. solo: all CTAs run
// the program on their own copies (CTA barriers).
__device__ __noinline__ void gc_run(const GcPhase* __restrict__ prog, int phases, uint32_t base, int rank, int solo,
                                    double omega, const double* __restrict__ inv, double* stage) {
  GcPhase P = prog[0];
  GcBatch B;
  int k = 0, ke = 0;  // this thread's first entry and its row's end
  auto fetch = [&]() {
    if (P.type > kGcSmooth0 && P.type < kGcDense && P.rows > 0) {
      const int i = min((int)threadIdx.x >> P.tl, P.rows - 1);
      const uint32_t ra = base + (uint32_t)P.o_rp + 2u * (uint32_t)i;
      k = gc_u16(ra) + ((int)threadIdx.x & ((1 << P.tl) - 1));
      ke = gc_u16(ra + 2u);
      gc_fetch(B, base, P.o_col, P.o_val, P.o_x, k, ke, 1 << P.tl, P.zero);
    }
  };
  fetch();
  for (int q = 0; q < phases; ++q) {
    if (P.type < kGcDense) {
      const int tl = P.tl, step = 1 << tl, part = threadIdx.x & (step - 1);
      const int live = (P.rows + (32 >> tl) - 1) & ~((32 >> tl) - 1);  // whole warps
      for (int r = threadIdx.x >> tl; r < live; r += kGcThreads >> tl) {
        const int i = min(r, P.rows - 1);
        const uint32_t at = 8u * (uint32_t)i + base;
        double s = 0.0;
        if (P.type != kGcSmooth0) {
          if (r != (int)threadIdx.x >> tl) {  // a further row of this thread
            const uint32_t ra = base + (uint32_t)P.o_rp + 2u * (uint32_t)i;
            k = gc_u16(ra) + part;
            ke = gc_u16(ra + 2u);
            gc_fetch(B, base, P.o_col, P.o_val, P.o_x, k, ke, step, P.zero);
          }
          s = gc_gather(B, s);
          for (k += kGcU * step; k < ke; k += kGcU * step) {
            gc_fetch(B, base, P.o_col, P.o_val, P.o_x, k, ke, step, P.zero);
            s = gc_gather(B, s);
          }
          for (int o = step >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        const double b = gc_own(at + (uint32_t)P.o_b), rd = gc_own(at + (uint32_t)P.o_rd);
        const double old = gc_own(at + (uint32_t)P.o_old);
        double out;
        if (P.type == kGcSweep) {
          out = rd == rd ? fma(omega, (b - s) * rd, old) : old;
        } else if (P.type == kGcResidual) {
          out = b - s;
        } else if (P.type == kGcProlong) {
          out = old + s;
        } else {
          out = P.zero_start ? 0.0 : gc_smooth0(P.type == kGcRestrict ? s : b, rd, omega);
          if (P.type == kGcRestrict) {
            if (part == 0 && r < P.rows) gc_put(at + (uint32_t)P.o_out2, out);
            out = s;
          }
        }
        if (part == 0 && r < P.rows) gc_put(at + (uint32_t)P.o_out, out);
      }
    } else {
      // dense: the right-hand side of all rows staged, one warp per row
      for (int c = threadIdx.x; c < P.cols; c += kGcThreads) {
        const int o = c / P.rpc;
        stage[c] = gc_ld(gc_map(base + (uint32_t)P.o_b + 8u * (uint32_t)(c - o * P.rpc), (uint32_t)(solo ? rank : o)));
      }
      __syncthreads();
      for (int i = threadIdx.x >> 5; i < P.rows; i += kGcWarps) {
        double s = 0.0;
        if (P.type == kGcTail) {
          for (int c = threadIdx.x & 31; c < P.cols; c += 32)
            s = fma(gc_own(base + (uint32_t)P.o_val + 8u * (uint32_t)(i * P.cols + c)), stage[c], s);
        } else {
          const double* a = inv + (size_t)((solo ? 0 : rank) * P.rpc + i) * P.cols;
          for (int c = threadIdx.x & 31; c < P.cols; c += 32) s += a[c] * stage[c];
        }
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) gc_put(base + (uint32_t)P.o_out + 8u * (uint32_t)i, s);
      }
    }
    const bool more = q + 1 < phases;
    if (solo) {
      __syncthreads();
      if (more) {
        P = prog[q + 1];
        fetch();
      }
    } else {
      cluster_arrive();
      if (more) {
        P = prog[q + 1];
        fetch();
      }
      cluster_wait();
    }
  }
}

template <int PRE>
__global__ void __launch_bounds__(kGcThreads, 1) k_cluster_gmres(const __grid_constant__ GcArgs A) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char gc_sm[];
  GcCta C;
  C.sm = gc_sm;
  C.base = gc_addr(gc_sm);
  C.rank = (int)cluster.block_rank();
  C.ncta = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = A.n, m = A.m, r0 = C.rank * A.rpc, nr = gc_rows(n, A.rpc, C.rank);
  double* w = C.d(A.o_w);
  double *h = C.d(A.o_h), *h2 = h + (m + 1), *hr = h2 + (m + 1), *cs = C.d(A.o_cs), *sn = C.d(A.o_sn), *g = C.d(A.o_g), *yv = C.d(A.o_y);
  // this CTA's rows of the basis: only it reads them
  double* V = A.o_v >= 0 ? C.d(A.o_v) : A.V + r0;
  const size_t ldv = A.o_v >= 0 ? (size_t)A.rpc : (size_t)n;
  const int o_x0 = A.lev[0].o_xa;  // gather buffer of level-0 vectors outside the V-cycle

  for (int q = tid; q < A.smem_bytes / 16; q += kGcThreads) reinterpret_cast<int4*>(gc_sm)[q] = make_int4(0, 0, 0, 0);
  __syncthreads();
  gc_stage(A.M, C);
  if (PRE == kGcAmg) {
    for (int q = tid; q < A.phases + A.solo_phases; q += kGcThreads) {
      GcPhase p = A.program[q];
      p.rows = gc_rows(p.rows, p.rpc, q < A.phases ? C.rank : 0);
      reinterpret_cast<GcPhase*>(gc_sm + A.o_prog)[q] = p;
    }
    for (int l = 0; l < A.levels; ++l) {
      if (A.lev[l].A.rp) gc_stage(A.lev[l].A, C);
      if (l + 1 < A.levels) {
        gc_stage(A.lev[l].R, C);
        gc_stage(A.lev[l].P, C);
      }
      gc_stage_diag(A.lev[l], false, C);
    }
    for (int l = 0; l < A.solo_levels; ++l) {
      gc_stage(A.solo[l].A, C);
      if (l + 1 < A.solo_levels) {
        gc_stage(A.solo[l].R, C);
        gc_stage(A.solo[l].P, C);
      }
      gc_stage_diag(A.solo[l], true, C);
    }
    cluster_barrier();
    // the tail's matrix: the tail's cycle on this CTA's share of the unit
    // vectors, each column's entries sent to the CTAs that own their rows
    if (A.solo_levels > 0) {
      const GcLevel &T = A.lev[A.levels - 1], &S = A.solo[0];
      for (int j = C.rank; j < T.n; j += C.ncta) {
        __syncthreads();
        for (int i = tid; i < T.n; i += kGcThreads) C.d(S.o_b)[i] = i == j ? 1.0 : 0.0;
        __syncthreads();
        gc_run(reinterpret_cast<const GcPhase*>(gc_sm + A.o_prog) + A.phases, A.solo_phases, C.base, C.rank, 1,
               A.omega, A.inv, C.d(A.o_stage));
        for (int i = tid; i < T.n; i += kGcThreads) {
          const int o = i / T.rpc;
          gc_st(gc_map(C.base + (uint32_t)A.o_tail + 8u * (uint32_t)((i - o * T.rpc) * T.n + j), (uint32_t)o),
                C.d(A.o_solo_z)[i]);
        }
      }
    }
  }

  // Sums over the cluster of nv products V_k . u (u: this CTA's rows), result
  // in out[0..nv) of every CTA. Partials alternate between two slots, so a
  // CTA's pushes never reach a slot another is still reading.
  int slot = 0;
  auto dots = [&](int nv, const double* u, double* out) {
    const uint32_t po = (uint32_t)A.o_part + 8u * (uint32_t)(slot * (m + 1) * kGcMaxCtas);
    for (int k = warp; k < nv; k += kGcWarps) {
      const double* vk = V + (size_t)k * ldv;
      double s = 0.0;
      // every load of a 640-row block in flight at once: from global memory the
      // pass is one latency (the L1 does not survive the cluster barriers)
      for (int i0 = lane; i0 < nr; i0 += kGcThreads) {
        double x[kGcThreads / 32];
#pragma unroll
        for (int q = 0; q < kGcThreads / 32; ++q) x[q] = i0 + 32 * q < nr ? vk[i0 + 32 * q] : 0.0;
#pragma unroll
        for (int q = 0; q < kGcThreads / 32; ++q)
          if (i0 + 32 * q < nr) s += x[q] * u[i0 + 32 * q];
      }
      s = __shfl_sync(0xffffffffu, warp_sum(s), 0);
      if (lane < C.ncta) gc_st(gc_map(C.base + po + 8u * (uint32_t)(k * kGcMaxCtas + C.rank), (uint32_t)lane), s);
    }
    cluster_barrier();
    const double* p = C.d((int)po);
    if (tid < nv) {
      double s = 0.0;
      for (int c = 0; c < C.ncta; ++c) s += p[tid * kGcMaxCtas + c];
      out[tid] = s;
    }
    slot ^= 1;
    __syncthreads();
  };
  // ||u||^2 over the cluster in every thread.
  auto norm2 = [&](const double* u) -> double {
    const uint32_t po = (uint32_t)A.o_part + 8u * (uint32_t)(slot * (m + 1) * kGcMaxCtas);
    __shared__ double red[kGcWarps];
    double s = 0.0;
    for (int i = tid; i < nr; i += kGcThreads) s += u[i] * u[i];
    s = warp_sum(s);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (warp == 0) {
      double t = lane < kGcWarps ? red[lane] : 0.0;
      t = __shfl_sync(0xffffffffu, warp_sum(t), 0);
      if (lane < C.ncta) gc_st(gc_map(C.base + po + 8u * (uint32_t)C.rank, (uint32_t)lane), t);
    }
    cluster_barrier();
    const double* p = C.d((int)po);
    double t = 0.0;
    for (int c = 0; c < C.ncta; ++c) t += p[c];
    slot ^= 1;
    return t;
  };
  // w = b - A x for the x in global memory (own rows gathered through o_x0).
  auto residual = [&]() {
    for (int i = tid; i < nr; i += kGcThreads) C.d(o_x0)[i] = A.x[r0 + i];
    cluster_barrier();
    gc_spmv(A.M, C.base, nr, o_x0, [&](int i, double s) { w[i] = A.b[r0 + i] - s; });
    __syncthreads();
  };
  // z = M^-1 u in shared memory of every CTA's rows; returns its offset.
  const GcPhase* prog = reinterpret_cast<const GcPhase*>(gc_sm + A.o_prog);
  // (the V-cycle's program names w as its right-hand side)
  auto precond = [&](const double* u) -> int {
    if constexpr (PRE == kGcAmg) {
      gc_run(prog, A.phases, C.base, C.rank, 0, A.omega, A.inv, C.d(A.o_stage));
      return A.o_z;
    } else {
      for (int i = tid; i < nr; i += kGcThreads) C.d(o_x0)[i] = PRE == kGcJacobi ? u[i] * A.jinv[r0 + i] : u[i];
      cluster_barrier();
      return o_x0;
    }
  };

  // start (EpiResidual MODE 1) or the state of the previous launch
  double rn, rn0, thr;
  int iter, term;
  const int max_iter = A.st->max_iter;
  bool done = false;
  cluster_barrier();  // matrices and diagonals staged, every CTA running
  if (!A.resume) {
    residual();
    rn0 = rn = sqrt(norm2(w));
    thr = fmax(A.st->tol_abs, A.st->tol_rel * rn0);
    iter = 0;
    term = CFD_TERM_MAX_ITERATIONS;
    if (!isfinite(rn)) {
      term = CFD_TERM_BREAKDOWN;
      done = true;
    } else if (rn <= thr) {
      term = CFD_TERM_INITIAL_RESIDUAL;
      done = true;
    }
  } else {
    for (int i = tid; i < nr; i += kGcThreads) w[i] = A.rg[r0 + i];
    rn0 = A.st->rnorm0;
    rn = A.st->rnorm;
    thr = A.st->threshold;
    iter = A.st->iter;
    term = A.st->term;
    __syncthreads();
  }

  for (int steps = 0; !done && steps < kGcStepsPerLaunch; steps += m) {
    // cycle start: beta = ||r||, v_0 = r / beta
    const double beta = sqrt(norm2(w));
    if (tid < m + 1) g[tid] = tid == 0 ? beta : 0.0;
    for (int i = tid; i < nr; i += kGcThreads) {
      const double v = beta != 0.0 ? w[i] / beta : w[i];
      w[i] = v;
      V[i] = v;
    }
    __syncthreads();
    int cols = 0;
    for (int j = 0; j < m; ++j) {
      const int z = precond(w);
      gc_spmv(A.M, C.base, nr, z, [&](int i, double s) { w[i] = s; });
      __syncthreads();
      double* hp = h;
      for (int pass = 0; pass < 2; ++pass, hp = h2) {
        dots(j + 1, w, hp);
        for (int i = tid; i < nr; i += kGcThreads) {
          const double* vi = V + i;
          double s = 0.0;
#pragma unroll 8
          for (int k = 0; k <= j; ++k) s += hp[k] * vi[k * ldv];
          w[i] = w[i] - s;
        }
        __syncthreads();
      }
      const double hn = sqrt(norm2(w));
      if (hn != 0.0) {
        double* vn = V + (j + 1) * ldv;
        for (int i = tid; i < nr; i += kGcThreads) {
          const double v = w[i] / hn;
          w[i] = v;
          vn[i] = v;
        }
      }
      // Givens rotations (k_gmres_rot), the same bits in every CTA
      if (tid == 0) {
        double* __restrict__ out = hr;
        const double *__restrict__ ha = h, *__restrict__ hb = h2, *__restrict__ cr = cs, *__restrict__ sr = sn;
        double c = ha[0] + hb[0];
#pragma unroll 4
        for (int q = 0; q < j; ++q) {
          const double nx = ha[q + 1] + hb[q + 1], cq = cr[q], sq = sr[q];
          out[q] = cq * c + sq * nx;
          c = -sq * c + cq * nx;
        }
        const double d = hypot(c, hn);
        cs[j] = d > 0.0 ? c / d : 1.0;
        sn[j] = d > 0.0 ? hn / d : 0.0;
        out[j] = d;
        g[j + 1] = -sn[j] * g[j];
        g[j] = cs[j] * g[j];
      }
      __syncthreads();
      if (C.rank == 0)
        for (int q = tid; q <= j; q += kGcThreads) A.H[(size_t)j * (m + 1) + q] = hr[q];
      ++iter;
      rn = fabs(g[j + 1]);
      cols = j + 1;
      if (!isfinite(rn)) {
        term = CFD_TERM_BREAKDOWN;
        done = true;
        break;
      }
      if (rn <= thr || iter >= max_iter || hn == 0.0) break;
    }
    if (done) break;
    // least squares in CTA 0, its solution to every CTA (k_gmres_lsq)
    __syncthreads();
    if (C.rank == 0 && warp == 0) {
      for (int q = cols - 1; q >= 0; --q) {
        double s = 0.0;
        for (int l = q + 1 + lane; l < cols; l += 32) s += A.H[(size_t)l * (m + 1) + q] * yv[l];
        s = __shfl_sync(0xffffffffu, warp_sum(s), 0);
        const double dqq = A.H[(size_t)q * (m + 1) + q];
        const double y = dqq != 0.0 ? (g[q] - s) / dqq : 0.0;
        if (lane < C.ncta) gc_st(gc_map(C.base + (uint32_t)A.o_y + 8u * (uint32_t)q, (uint32_t)lane), y);
        __syncwarp();
      }
    }
    cluster_barrier();
    // x += M^-1 (V y); r = b - A x; the true residual decides (k_gmres_check)
    for (int i = tid; i < nr; i += kGcThreads) {
      const double* vi = V + i;
      double s = 0.0;
#pragma unroll 8
      for (int k = 0; k < cols; ++k) s += yv[k] * vi[k * ldv];
      w[i] = s;
    }
    __syncthreads();
    const int z = precond(w);
    for (int i = tid; i < nr; i += kGcThreads) A.x[r0 + i] = A.x[r0 + i] + C.d(z)[i];
    cluster_barrier();  // z read before the residual's gather buffer is written
    residual();
    rn = sqrt(norm2(w));
    if (!isfinite(rn)) {
      term = CFD_TERM_BREAKDOWN;
      done = true;
    } else if (rn <= thr) {
      term = CFD_TERM_CONVERGED;
      done = true;
    } else if (iter >= max_iter) {
      term = CFD_TERM_MAX_ITERATIONS;
      done = true;
    }
  }
  for (int i = tid; i < nr; i += kGcThreads) A.rg[r0 + i] = w[i];
  if (C.rank == 0 && tid == 0) {
    DevState* st = A.st;
    st->rnorm0 = rn0;
    st->threshold = thr;
    st->rnorm = rn;
    st->rr = rn * rn;
    st->iter = iter;
    st->term = term;
    st->done = done ? 1 : 0;
  }
  cluster_barrier();  // no CTA leaves while its shared memory may still be read
}

size_t gc_round16(size_t b) { return (b + 15) / 16 * 16; }

// Largest number of nonzeros any of the ncta row blocks of rpc rows holds.
int64_t gc_nnz_cap(const HostCsr& h, int rpc) {
  int64_t cap = 0;
  for (int64_t r = 0; r < h.nrows; r += rpc) cap = std::max(cap, h.rp[std::min<int64_t>(r + rpc, h.nrows)] - h.rp[r]);
  return cap;
}

// The per-CTA shared-memory layout for ncta CTAs; 0 bytes when the packed
// columns or row offsets cannot express the system.
size_t gc_layout(GcArgs& A, const HostCsr& op, const cfd_amg* amg, int pre, int ncta) {
  size_t at = 0;
  bool ok = true;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += gc_round16(bytes);
    return (int)o;
  };
  auto split = [&](int64_t n) {
    const int64_t rpc = (n + ncta - 1) / ncta;
    if (rpc >= (1 << kGcIdxBits)) ok = false;
    return (int)rpc;
  };
  auto mat = [&](GcMat& M, const HostCsr& h, int rpc_r, int rpc_c, bool solo, const GcMat* pattern) {
    const int64_t cap = gc_nnz_cap(h, rpc_r) + 1;  // and a zero entry
    if (cap >= 65536) ok = false;
    M.solo = solo;
    M.zero = (int)cap - 1;
    // as many threads on a row as the CTA has to spare, at most one per entry
    M.tl = 0;
    while (M.tl < 3 && (rpc_r << (M.tl + 1)) <= kGcThreads && ((int64_t)h.nrows << (M.tl + 1)) <= h.nnz()) ++M.tl;
    M.n = (int)h.nrows;
    M.rpc_r = rpc_r;
    M.rpc_c = rpc_c;
    M.o_val = take((size_t)cap * 8);
    M.o_col = pattern ? pattern->o_col : take((size_t)cap * 2);
    M.o_rp = pattern ? pattern->o_rp : take((size_t)(rpc_r + 1) * 2);
  };
  A.n = (int)op.nrows;
  A.rpc = split(op.nrows);
  if (!ok) return 0;
  // the hierarchy's finest operator usually has the solve's pattern: its
  // columns and row offsets are then stored once
  const bool same = pre == kGcAmg && amg->host[0].A.rp == op.rp && amg->host[0].A.ci == op.ci;
  mat(A.M, op, A.rpc, A.rpc, false, nullptr);
  A.o_w = take((size_t)A.rpc * 8);
  if (pre == kGcAmg) {
    for (int l = 0; l < A.levels; ++l) {
      A.lev[l].n = (int)amg->host[l].A.nrows;
      A.lev[l].rpc = split(A.lev[l].n);
    }
    const int t = A.levels - 1;
    for (int l = 0; l < A.levels; ++l) {
      GcLevel& L = A.lev[l];
      const size_t vb = (size_t)(L.rpc + 1) * 8;  // and a zero behind the slice
      L.o_xa = take(vb);
      L.o_b = l == 0 ? A.o_w : take(vb);
      L.o_d = take(vb);
      if (l < t) {
        mat(L.R, amg->host[l].R, A.lev[l + 1].rpc, L.rpc, false, nullptr);
        mat(L.P, amg->host[l].P, L.rpc, A.lev[l + 1].rpc, false, nullptr);
      }
      if (l < t || A.solo_levels == 0) {
        mat(L.A, amg->host[l].A, L.rpc, L.rpc, false, l == 0 && same ? &A.M : nullptr);
        L.o_xb = take(vb);
        L.o_r = take(vb);
      }
    }
    for (int l = 0; l < A.solo_levels; ++l) {
      GcLevel& L = A.solo[l];
      const HostLevel& H = amg->host[t + l];
      L.n = L.rpc = (int)H.A.nrows;
      const size_t vb = (size_t)(L.n + 1) * 8;
      mat(L.A, H.A, L.n, L.n, true, nullptr);
      if (l + 1 < A.solo_levels) {
        const int nc = (int)amg->host[t + l + 1].A.nrows;
        mat(L.R, H.R, nc, L.n, true, nullptr);
        mat(L.P, H.P, L.n, nc, true, nullptr);
      }
      L.o_b = take(vb);
      L.o_xa = take(vb);
      L.o_xb = take(vb);
      L.o_r = take(vb);
      L.o_d = take(vb);
    }
    if (A.solo_levels > 0) A.o_tail = take((size_t)A.lev[t].rpc * A.lev[t].n * 8);
    A.o_prog = take((size_t)(A.phases + A.solo_phases) * sizeof(GcPhase));
    A.o_stage = take((size_t)A.lev[t].n * 8);
  } else {
    A.lev[0].o_xa = take((size_t)(A.rpc + 1) * 8);
  }
  const size_t mv = (size_t)(A.m + 1) * 8;
  A.o_part = take(2 * mv * kGcMaxCtas);
  A.o_h = take(3 * mv);
  A.o_cs = take(mv);
  A.o_sn = take(mv);
  A.o_g = take(mv);
  A.o_y = take(mv);
  return ok ? at : 0;
}

// Appends the passes of one V-cycle from zero (amg.rs:423-503) over levels
// lev[0..levels); coarse: how the last of them is solved (kGcSweep, kGcDense or
// kGcTail). Returns where the result is left.
int gc_program(const GcLevel* lev, int levels, int coarse, int o_tail, const cfd_amg_config& c,
               std::vector<GcPhase>& prog) {
  const int last = levels - 1, sweeps = std::max(0, (int)c.coarse_sweeps);
  auto add = [&](int type, const GcLevel& L, const GcMat* M, int o_x, int o_out, bool zero = false, int o_out2 = 0) {
    GcPhase p{};
    p.type = type;
    p.zero_start = zero;
    p.rows = p.cols = L.n;
    p.rpc = L.rpc;
    if (M) {
      p.o_rp = M->o_rp;
      p.o_col = M->o_col;
      p.o_val = M->o_val;
      p.zero = M->zero;
      p.tl = M->tl;
    }
    if (type == kGcTail) p.o_val = o_tail;
    p.o_old = type == kGcProlong ? o_out : o_x;
    p.o_x = o_x;
    p.o_out = o_out;
    p.o_b = L.o_b;
    p.o_rd = L.o_d;
    p.o_out2 = o_out2;
    prog.push_back(p);
  };
  auto smooth = [&](const GcLevel& L, int& x, int count) {
    for (int s = 0; s < count; ++s) {
      const int y = x == L.o_xa ? L.o_xb : L.o_xa;
      add(kGcSweep, L, &L.A, x, y);
      x = y;
    }
  };
  std::vector<int> at(levels);  // the iterate of each level
  for (int l = 0; l < last; ++l) {
    const GcLevel &L = lev[l], &N = lev[l + 1];
    int x = L.o_xa;
    if (l == 0) add(kGcSmooth0, L, nullptr, x, x, c.pre_smooth < 1);
    smooth(L, x, c.pre_smooth - 1);
    add(kGcResidual, L, &L.A, x, L.o_r);
    at[l] = x;
    const bool zero = l + 1 == last ? (coarse != kGcSweep || sweeps < 1) : c.pre_smooth < 1;
    add(kGcRestrict, N, &L.R, L.o_r, N.o_b, zero, N.o_xa);
  }
  const GcLevel& L = lev[last];
  int e = L.o_xa;
  // a single level: this pass is also the barrier before its right-hand side is gathered
  if (last == 0) add(kGcSmooth0, L, nullptr, e, e, coarse != kGcSweep || sweeps < 1);
  if (coarse == kGcSweep)
    smooth(L, e, sweeps - 1);
  else
    add(coarse, L, nullptr, 0, e);
  for (int l = last - 1; l >= 0; --l) {
    int x = at[l];
    add(kGcProlong, lev[l], &lev[l].P, e, x);
    smooth(lev[l], x, c.post_smooth);
    e = x;
  }
  return e;
}

// Both programs of a laid-out hierarchy: the cycle's, then the tail's.
void gc_programs(GcArgs& A, const cfd_amg_config& c, std::vector<GcPhase>& prog) {
  prog.clear();
  const int coarse = A.inv ? kGcDense : kGcSweep;
  A.o_z = gc_program(A.lev, A.levels, A.solo_levels > 0 ? kGcTail : coarse, A.o_tail, c, prog);
  A.phases = (int)prog.size();
  if (A.solo_levels > 0) A.o_solo_z = gc_program(A.solo, A.solo_levels, coarse, 0, c, prog);
  A.solo_phases = (int)prog.size() - A.phases;
}

template <int PRE>
cfd_status gc_launch(cfd_context* ctx, const GcArgs& A, int ncta, size_t smem, bool probe, bool* fits) {
  auto kern = k_cluster_gmres<PRE>;
  if (probe) {  // once a solve, before its launches
    CFD_TRY(allow_dynamic_smem(kern, ctx->device));
    if (ncta > 8) CFD_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncta);
  cfg.blockDim = dim3(kGcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (probe) {
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    *fits = clusters >= 1;
    return CFD_OK;
  }
  CFD_TRY_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
  ctx->stats.launches++;
  return CFD_OK;
}

cfd_status gc_launch_pre(cfd_context* ctx, int pre, const GcArgs& A, int ncta, size_t smem, bool probe, bool* fits) {
  if (pre == kGcAmg) return gc_launch<kGcAmg>(ctx, A, ncta, smem, probe, fits);
  if (pre == kGcJacobi) return gc_launch<kGcJacobi>(ctx, A, ncta, smem, probe, fits);
  return gc_launch<kGcNone>(ctx, A, ncta, smem, probe, fits);
}

}  // namespace

// The cluster GMRES applies when the operator (and with AMG the hierarchy)
// split over at most 16 CTAs fits their shared memory; *ok = false otherwise
// (nothing launched). x holds the initial guess and takes the solution; the
// state takes the outcome. m: the restart width (a power of two).
// Without a V-cycle a step is one SpMV, bound by its remote gathers where the columns
// are scattered over the CTAs: such a system goes to the separate kernels beyond
// kGcMaxFar entries of other CTAs in a block. A GMRES(8) of 16 steps, here / separate
// kernels, ms: 0.82 / 0.92 at 12300 entries, 0.84 / 0.86 and 0.88 / 0.90 at 13800 and
// 14200, 0.98 / 0.91 at 14800, 1.14 / 0.92 at 17200. With the V-cycle, some fifty
// launches a step, the cluster was ahead wherever the hierarchy fits (1.13x at least).
// What bounds the size otherwise is capacity: five-point systems of 48400 rows, the
// largest that fit, 0.46 / 0.86 ms, tridiagonal ones of 65000 0.58 / 0.85.
cfd_status cluster_gmres_solve(cfd_context* ctx, cfd_csr* a, cfd_amg* amg, int precond, int m, const double* b,
                               double* x, DevState* st, DevState* host_st, bool* ok) {
  *ok = false;
  const int64_t n = a->dev.nrows;
  if (n <= 0 || m > kGcMaxRestart || n >= ((int64_t)kGcMaxCtas << kGcIdxBits)) return CFD_OK;
  const int pre = precond == CFD_PRECOND_AMG ? kGcAmg : (precond == CFD_PRECOND_JACOBI ? kGcJacobi : kGcNone);
  GcArgs A;
  std::memset(&A, 0, sizeof(A));
  A.m = m;
  if (pre == kGcAmg) {
    const size_t nl = amg->host.size();
    if (nl < 1 || nl > (size_t)kGcMaxLevels || amg->dev.size() != nl) return CFD_OK;
    if (amg->cfg.coarse_solve == CFD_COARSE_DENSE && amg->coarse_inv) {
      if (amg->coarse_n > kGcMaxDense) return CFD_OK;
      A.inv = amg->coarse_inv;
    }
  }
  std::vector<GcPhase> prog;
  if (pre == kGcAmg) {
    const int nl = (int)amg->host.size();
    int t = 0;
    while (t < nl && amg->host[t].A.nrows > kTailRows) ++t;
    A.levels = std::min(nl, t + 1);
    A.solo_levels = nl - t;
    gc_programs(A, amg->cfg, prog);  // their lengths do not depend on the layout
    if (prog.size() > (size_t)kGcMaxPhases) return CFD_OK;
  } else {
    A.levels = 1;
  }
  int max_smem = 0;
  CFD_TRY_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const size_t budget = (size_t)max_smem - 1024;  // static shared arrays
  int ncta = 1;
  size_t smem = 0;
  while (ncta < kGcMaxCtas && n > (int64_t)ncta * kGcRowsPerCta) ncta *= 2;
  for (; ncta <= kGcMaxCtas; ncta *= 2) {
    smem = gc_layout(A, a->host, amg, pre, ncta);
    if (smem == 0 || smem > budget) continue;
    bool fits = false;
    CFD_TRY(gc_launch_pre(ctx, pre, A, ncta, smem, true, &fits));
    if (fits) break;
  }
  if (ncta > kGcMaxCtas) return CFD_OK;
  if (pre != kGcAmg && cluster_scattered(a, 1, A.rpc) > kGcMaxFar) return CFD_OK;
  const size_t basis = gc_round16((size_t)(m + 1) * A.rpc * 8);
  A.o_v = -1;
  if (smem + basis <= budget) {
    A.o_v = (int)smem;
    smem += basis;
  }
  A.smem_bytes = (int)smem;
  auto dev = [](GcMat& M, const DevMat& d) {
    M.rp = d.rp;
    M.col = d.col;
    M.val = d.v64;
  };
  dev(A.M, a->dev);
  if (pre == kGcAmg) {
    for (int l = 0; l < A.levels; ++l) {
      if (l + 1 < A.levels || A.solo_levels == 0) dev(A.lev[l].A, amg->dev[l].A);
      if (l + 1 < A.levels) {
        dev(A.lev[l].R, amg->dev[l].R);
        dev(A.lev[l].P, amg->dev[l].P);
      }
      A.lev[l].diag = amg->dev[l].d64;
    }
    for (int l = 0; l < A.solo_levels; ++l) {
      const DevLevel& D = amg->dev[A.levels - 1 + l];
      dev(A.solo[l].A, D.A);
      if (l + 1 < A.solo_levels) {
        dev(A.solo[l].R, D.R);
        dev(A.solo[l].P, D.P);
      }
      A.solo[l].diag = D.d64;
    }
    A.omega = amg->cfg.relaxation;
    gc_programs(A, amg->cfg, prog);
  }
  A.jinv = a->jinv64;
  A.b = b;
  A.x = x;
  A.st = st;
  double* ws = nullptr;
  const size_t prog_elems = prog.size() * sizeof(GcPhase) / sizeof(double);
  const size_t ws_elems = prog_elems + (size_t)(m + 2) * n + (size_t)m * (m + 1);
  if (cudaMallocAsync((void**)&ws, ws_elems * sizeof(double), ctx->stream) != cudaSuccess) {
    cudaGetLastError();
    set_error("GMRES workspace allocation failed (%lld unknowns, restart %d)", (long long)n, m);
    return CFD_ERR_ALLOC;
  }
  A.program = reinterpret_cast<const GcPhase*>(ws);
  A.V = ws + prog_elems;
  A.rg = A.V + (size_t)(m + 1) * n;
  A.H = A.rg + n;
  cfd_status s = CFD_OK;
  if (prog_elems > 0 && cudaMemcpyAsync(ws, prog.data(), prog.size() * sizeof(GcPhase), cudaMemcpyHostToDevice,
                                        ctx->stream) != cudaSuccess) {
    set_error("cluster GMRES: upload of the V-cycle's passes failed");
    s = CFD_ERR_CUDA;
  }
  int64_t cycles = 0;
  while (s == CFD_OK && !host_st->done) {
    bool unused = false;
    s = gc_launch_pre(ctx, pre, A, ncta, smem, false, &unused);
    if (s != CFD_OK) break;
    cudaError_t e = cudaMemcpyAsync(host_st, st, sizeof(DevState), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
      set_error("cluster GMRES: %s", cudaGetErrorString(e));
      s = CFD_ERR_CUDA;
      break;
    }
    A.resume = 1;
    cycles += kGcStepsPerLaunch / m;
    if (!host_st->done && cycles > (int64_t)host_st->max_iter + 2) {
      set_error("GMRES did not terminate within its iteration budget");
      s = CFD_ERR_TIMEOUT;
    }
  }
  cudaFreeAsync(ws, ctx->stream);
  if (s == CFD_OK) *ok = true;
  return s;
}

}  // namespace cfd
