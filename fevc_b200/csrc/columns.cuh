// Blocked PCG with one thread block per column, for Laplacians whose vectors
// fit one SM's shared memory.
//
// The columns of a block of right-hand sides are independent, so a small
// problem needs no grid-wide barrier: each block holds its column's direction
// p, residual r, solution x and the segment products in shared memory, reads
// the matrix from L1 / L2, and iterates on block barriers alone until its own
// column has converged.  The cooperative kernels (persistent.cuh, flex.cuh)
// pay three to five grid barriers and as many grid-wide reductions an
// iteration, about 9 us of their 15 us on a 1,000-vertex firm graph.
//
// What it costs is the matrix once per column: 12 bytes an entry through one
// SM's L2 port.  Rule of use (column_form, engine.cu): whenever p and the
// segment products fit, about 11,000 vertices; there an iteration reads
// 2 MB an SM and still takes less than the cooperative kernel's.
//
// All storage is FP64, for every precision option: FP32 storage halves bytes
// of device memory, and here the vectors do not leave the SM.  Jacobi, or the
// degree-1 stage z = wa r + ws (A (ws r)) (flex.cuh) when POLY.
#pragma once

#include "persistent.cuh"

namespace fevcb {

constexpr int COL_MAX_THREADS = 1024;
constexpr int COL_LANES = 8;  // lanes of a segment: up to four of its <= 32 entries each
constexpr size_t COL_SMEM = 225 * 1024;  // dynamic shared memory of a block, at most

struct ColumnPcg {
  uint32_t n, nseg;
  int K;  // columns of the block (the stride of b and x)
  const uint32_t* seg_begin;
  const uint32_t* seg_end;
  const uint32_t* row_first;
  const uint32_t* col;
  const double* val;
  const double* diag;
  const double* dinv;
  const double* wa;  // POLY: per-vertex weights
  const double* ws;
  const double* b;  // n x K right-hand sides, uncentred
  double* x;        // n x K solutions
  double* rx;       // 2 x K x n: r and x of every column when they stay in device memory
  PcgState s;
  int ncols, fresh, max_iters;
  int resident;  // r and x in shared memory
  double tol;
};

// Shared memory of a block: p, the segment products, with POLY the weighted
// residual, and r and x when they fit (resident).  0: the problem is too large.
inline size_t column_smem(uint32_t n, uint32_t nseg, bool poly, bool* resident) {
  const size_t must = (size_t(n) * (poly ? 2 : 1) + nseg) * sizeof(double);
  const size_t all = must + 2 * size_t(n) * sizeof(double);
  *resident = all <= COL_SMEM;
  return *resident ? all : must <= COL_SMEM ? must : 0;
}

inline int column_threads(uint32_t nseg) { return nseg <= 128 ? 256 : nseg <= 512 ? 512 : COL_MAX_THREADS; }

namespace column {

// Sum M values over the block in a fixed order; every thread gets the totals.
// buf alternates between two buffers so one barrier a reduction is enough.
template <int M>
__device__ __forceinline__ void block_sum(double (&v)[M], double (*buf)[2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll
  for (int m = 0; m < M; ++m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[m] += __shfl_xor_sync(0xffffffffu, v[m], o);
    if (lane == 0) buf[warp][m] = v[m];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < M; ++m) {
    double t = lane < warps ? buf[lane][m] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    v[m] = t;
  }
}

// seg[s] = sum of the segment's entries times y, COL_LANES lanes a segment;
// the next segment's range is loaded while the current entries are in flight
__device__ __forceinline__ void products(const ColumnPcg& a, const double* y, double* seg) {
  const int sub = threadIdx.x % COL_LANES;
  const uint32_t groups = blockDim.x / COL_LANES;
  const uint32_t rounds = (a.nseg + groups - 1) / groups;
  uint32_t sg = threadIdx.x / COL_LANES, b = 0, e = 0;
  if (sg < a.nseg) {
    b = __ldg(a.seg_begin + sg);
    e = __ldg(a.seg_end + sg);
  }
  for (uint32_t k = 0; k < rounds; ++k) {
    const uint32_t next = sg + groups;
    uint32_t nb = 0, ne = 0;
    if (next < a.nseg) {
      nb = __ldg(a.seg_begin + next);
      ne = __ldg(a.seg_end + next);
    }
    uint32_t j[4];
    double w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = b + sub + uint32_t(u) * COL_LANES;
      j[u] = i < e ? __ldg(a.col + i) : 0;
      w[u] = i < e ? __ldg(a.val + i) : 0.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) acc += w[u] * y[j[u]];
#pragma unroll
    for (int o = COL_LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sub == 0 && sg < a.nseg) seg[sg] = acc;
    sg = next;
    b = nb;
    e = ne;
  }
}

// The row's segment products in order, four partial sums for a hub's many.
__device__ __forceinline__ double row_sum(const double* seg, uint32_t s0, uint32_t s1) {
  double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
  uint32_t s = s0;
  for (; s + 4 <= s1; s += 4) {
    t0 += seg[s];
    t1 += seg[s + 1];
    t2 += seg[s + 2];
    t3 += seg[s + 3];
  }
  for (; s < s1; ++s) t0 += seg[s];
  return (t0 + t1) + (t2 + t3);
}

}  // namespace column

template <bool POLY>
__global__ void __launch_bounds__(COL_MAX_THREADS, 1) k_pcg_columns(ColumnPcg a) {
  extern __shared__ double sh[];
  __shared__ double red[2][COL_MAX_THREADS / 32][2];
  const int j = blockIdx.x;
  const uint32_t n = a.n;
  double* p = sh;
  double* seg = p + n;
  double* t = seg + a.nseg;  // POLY: ws .* r
  double* r = a.resident ? t + (POLY ? n : 0) : a.rx + size_t(j) * n;
  double* x = a.resident ? r + n : a.rx + size_t(a.K + j) * n;
  int flip = 0;
  auto sum2 = [&](double& u, double& v) {
    double w[2] = {u, v};
    column::block_sum<2>(w, red[flip]);
    flip ^= 1;
    u = w[0];
    v = w[1];
  };
  // ---- start: the column's mean and norm (fresh), r = (b - mean) - L x
  double mean, tol2;
  int active, iters = 0;
  if (a.fresh) {
    double s1 = 0.0, s2 = 0.0;
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) {
      const double bv = a.b[size_t(v) * a.K + j];
      r[v] = bv;
      x[v] = 0.0;
      s1 += bv;
      s2 += bv * bv;
    }
    sum2(s1, s2);
    mean = s1 / double(n);
    const double bb = fmax(s2 - double(n) * mean * mean, 0.0);
    tol2 = a.tol * a.tol * bb;
    active = j < a.ncols && bb > 0.0 ? 1 : 0;
    if (threadIdx.x == 0) {
      a.s.mean[j] = mean;
      a.s.bb[j] = bb;
      a.s.tol2[j] = tol2;
      a.s.rr[j] = bb;
    }
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) r[v] -= mean;
  } else {
    mean = a.s.mean[j];
    tol2 = a.s.tol2[j];
    active = a.s.active[j];
    iters = a.s.iters[j];
    if (active == 0) return;  // x stays as the last launch left it
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) {
      const double xv = a.x[size_t(v) * a.K + j];
      x[v] = xv;
      p[v] = xv;
    }
    __syncthreads();
    column::products(a, p, seg);
    __syncthreads();
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x)
      r[v] = (a.b[size_t(v) * a.K + j] - mean) -
             (a.diag[v] * x[v] - column::row_sum(seg, a.row_first[v], a.row_first[v + 1]));
    __syncthreads();
  }
  // z of the current residual into seg[row_first] (POLY) and r.z; with Jacobi
  // z = dinv r is formed where it is used
  auto precondition = [&]() {
    double rz = 0.0, none = 0.0;
    if constexpr (POLY) {
      for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) t[v] = a.ws[v] * r[v];
      __syncthreads();
      column::products(a, t, seg);
      __syncthreads();
      for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) {
        const uint32_t s0 = a.row_first[v], s1 = a.row_first[v + 1];
        const double z = a.wa[v] * r[v] + a.ws[v] * column::row_sum(seg, s0, s1);
        rz += r[v] * z;
        t[v] = z;  // only this thread reads t[v] again
      }
    } else {
      for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) rz += r[v] * (a.dinv[v] * r[v]);
    }
    sum2(rz, none);
    return rz;
  };
  double rz = 0.0, rr_out = -1.0;
  if (active == 1) {
    rz = precondition();
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) p[v] = POLY ? t[v] : a.dinv[v] * r[v];
    __syncthreads();
  }
  for (int it = 0; active == 1 && it < a.max_iters; ++it) {
    // ---- q = L p and p.q; q is kept in the row's first segment slot
    column::products(a, p, seg);
    __syncthreads();
    double pq = 0.0, none = 0.0;
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) {
      const uint32_t s0 = a.row_first[v], s1 = a.row_first[v + 1];
      const double pv = p[v], q = a.diag[v] * pv - column::row_sum(seg, s0, s1);
      pq += pv * q;
      if (s0 < s1) seg[s0] = q;
    }
    sum2(pq, none);
    if (!(pq > 0.0) || !isfinite(pq)) {
      active = 2;  // nonpositive curvature
      break;
    }
    const double alpha = rz / pq;
    // ---- x += alpha p, r -= alpha q; r.r (and Jacobi's r.z)
    double rr = 0.0, rzn = 0.0;
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) {
      const uint32_t s0 = a.row_first[v], s1 = a.row_first[v + 1];
      const double pv = p[v], q = s0 < s1 ? seg[s0] : a.diag[v] * pv;
      const double rv = r[v] - alpha * q;
      x[v] += alpha * pv;
      r[v] = rv;
      rr += rv * rv;
      if (!POLY) rzn += rv * (a.dinv[v] * rv);
    }
    sum2(rr, rzn);
    ++iters;
    rr_out = rr;
    if (rr <= tol2) {
      active = 0;
      break;
    }
    if constexpr (POLY) rzn = precondition();
    const double beta = rzn / rz;
    rz = rzn;
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x)
      p[v] = (POLY ? t[v] : a.dinv[v] * r[v]) + beta * p[v];
    __syncthreads();
  }
  for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) a.x[size_t(v) * a.K + j] = x[v];
  if (threadIdx.x == 0) {
    a.s.active[j] = active;
    a.s.iters[j] = iters;
    if (rr_out >= 0.0) a.s.rr[j] = rr_out;
  }
}

}  // namespace fevcb
