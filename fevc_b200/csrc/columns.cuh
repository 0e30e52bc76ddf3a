// Blocked PCG with one thread block per column, for Laplacians small enough
// that a column's vectors live in one SM.
//
// The columns of a block of right-hand sides are independent, so a small
// problem needs no grid-wide barrier: each block iterates its own column on
// block barriers alone until that column has converged.  A thread owns one or
// two vertices and keeps their r, x, q and diagonal in registers; the
// direction p, the segment products and, up to about 1,150 vertices of a firm
// graph, the matrix (FP64 values, 16-bit columns: 10 bytes an entry) sit in
// shared memory, so an iteration touches no memory off the SM.  Beyond that
// the matrix streams from L2, 12 bytes an entry and column.
//
// What bounds it is latency: four block barriers, two block sums and the
// dependent shared-memory loads of a segment.  The cooperative kernels
// (persistent.cuh, flex.cuh) pay three to five grid barriers and as many
// grid-wide reductions an iteration, about 9 us of their 17 us on a
// 1,000-vertex firm graph.  A 64-column solve of about 20 Jacobi iterations,
// cooperative against this form: 148 vertices 315 / 45 us, 991 332 / 137 us,
// 1,391 340 / 220 us, 1,988 350 / 310 us.  Beyond 2,048 vertices the matrix,
// read once per column instead of once per block, costs more than the barriers
// (2,479 vertices 362 / 417 us, 9,929 583 / 1,717 us), and below them so do
// many entries: column_limit.
//
// A finished column's active flag is 0, one at the iteration limit 1, one that
// met a nonpositive curvature 2; the host counts them (no grid-wide counter).
//
// All storage is FP64, for every precision option: FP32 storage halves bytes
// of device memory, and here the vectors do not leave the SM.  Jacobi, or the
// degree-1 stage z = wa r + ws (A (ws r)) (flex.cuh) when POLY.
#pragma once

#include "persistent.cuh"

namespace fevcb {

constexpr int COL_MAX_THREADS = 1024;
constexpr uint32_t COL_MAX_VERTICES = 2 * COL_MAX_THREADS;
constexpr int COL_LANES = 8;  // lanes of a segment: up to four of its <= 32 entries each
constexpr size_t COL_SMEM = 225 * 1024;  // dynamic shared memory of a block, at most

struct ColumnPcg {
  uint32_t n, nseg, nnz;
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
  PcgState s;
  int ncols, fresh, max_iters;
  double tol;
};

// Shared memory of a block: p, the segment products, with POLY the weighted
// residual, and the matrix when it fits (MAT): values, 16-bit columns and the
// segments' first entries.  0: the problem is too large for a block.
inline size_t column_smem(uint32_t n, uint32_t nseg, size_t nnz, bool poly, bool* mat) {
  const size_t vec = (size_t(n) * (poly ? 2 : 1) + nseg) * sizeof(double);
  const size_t all = vec + nnz * (sizeof(double) + sizeof(uint16_t)) + (size_t(nseg) + 1) * sizeof(uint32_t) + 16;
  *mat = all <= COL_SMEM;
  return n > COL_MAX_VERTICES ? 0 : *mat ? all : vec <= COL_SMEM ? vec : 0;
}

// Rule of use: entries + 16 vertices of the Laplacian, at most this for a block
// of K columns.  A column's iteration takes 1.5 us, 0.27 us per 1,000 entries
// and 3 us per 1,000 vertices on its SM, whatever K; a cooperative iteration is
// mostly barriers, moves little with the entries and has a dearer start (more
// of it in a dense graph's few iterations: the vertices' weight).  Solves of
// panels with 12 to 1,000 workers a firm, cooperative / this form in us, each
// line's entries on both sides of its limit (thousands):
//   K = 1      104 321 / 295 (1,000 vertices), 103 345 / 379 (1,900)
//   K = 2      61 255 / 209 (1,000),           84 292 / 346 (1,500)
//   K = 8      35 224 / 180 (1,000),           46 245 / 278 (1,500)
//   K = 16     29 308 / 299 (1,839),           61 187 / 229 (1,000)
//   K = 32     20 214 / 146 (997),             23 247 / 258 (1,449)   FP64 Jacobi
//              35 226 / 192 (1,000),           46 258 / 293 (1,500)   k_pcg_flex
//   K = 64     46 294 / 281 (1,500),           56 298 / 332 (1,897)   FP64 Jacobi
//              61 320 / 250 (1,000),           56 316 / 350 (1,897)   k_pcg_flex
// A graph of 1,900 firms and 326,000 entries is where it costs most to miss:
// 296 / 862 us at K = 64, 216 / 858 at K = 8.
constexpr size_t column_limit(int K, bool flex) {
  return K == 1 ? 125000 : K == 2 ? 90000 : K <= 16 ? 62000 : K == 32 ? (flex ? 62000 : 46000) : 80000;
}

// Whether the column form takes a block of K columns; flex: the cooperative
// alternative is k_pcg_flex (flex.cuh), poly: the degree-1 stage.
inline bool column_rule(int K, uint32_t n, uint32_t nseg, size_t nnz, bool flex, bool poly) {
  bool mat;
  return nnz + 16 * size_t(n) <= column_limit(K, flex) && column_smem(n, nseg, nnz, poly, &mat) > 0;
}

inline int column_threads(uint32_t n) { return n <= 64 ? 256 : n <= 256 ? 512 : COL_MAX_THREADS; }

namespace column {

// Sum two values over the block in a fixed order; every thread gets the
// totals.  The caller alternates between two buffers, so one barrier is
// enough.  The half-warps each carry one of the values after the first
// exchange: 22 shuffles a warp instead of 40 (a shuffle of a 1,024-thread
// block is 32 issue slots, as much as a barrier).
__device__ __forceinline__ void block_sum(double& u, double& v, double (*buf)[COL_MAX_THREADS / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, half = lane >> 4;
  // lanes 0-15 collect u, lanes 16-31 collect v
  double w = (half ? v : u) + __shfl_xor_sync(0xffffffffu, half ? u : v, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if ((lane & 15) == 0) buf[half][warp] = w;
  __syncthreads();
  const int k = lane & 15;
  w = (k < warps ? buf[half][k] : 0.0) + (k + 16 < warps ? buf[half][k + 16] : 0.0);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  u = __shfl_sync(0xffffffffu, w, 0);
  v = __shfl_sync(0xffffffffu, w, 16);
}

// The matrix as the product pass reads it.
struct Matrix {
  const double* val;      // shared (MAT) or global
  const uint16_t* col16;  // MAT
  const uint32_t* first;  // MAT: first entry of every segment (nseg + 1)
};

// seg[s] = sum of the segment's entries times y, COL_LANES lanes a segment.
// From global memory the next segment's entries are loaded while the current
// ones are summed, and the range of the one after.
template <bool MAT>
__device__ __forceinline__ void products(const ColumnPcg& a, const Matrix& m, const double* y, double* seg) {
  const uint32_t sub = threadIdx.x % COL_LANES, groups = blockDim.x / COL_LANES;
  const uint32_t rounds = (a.nseg + groups - 1) / groups;
  uint32_t sg = threadIdx.x / COL_LANES;
  auto reduce = [&](double acc) {
#pragma unroll
    for (int o = COL_LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sub == 0 && sg < a.nseg) seg[sg] = acc;
  };
  if constexpr (MAT) {
    for (uint32_t k = 0; k < rounds; ++k, sg += groups) {
      const bool on = sg < a.nseg;
      const uint32_t b = on ? m.first[sg] : 0, e = on ? m.first[sg + 1] : 0;
      double acc = 0.0;
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t i = b + sub + u * COL_LANES;
        if (i < e) acc += m.val[i] * y[m.col16[i]];
      }
      reduce(acc);
    }
  } else {
    auto range = [&](uint32_t s, uint32_t& b, uint32_t& e) {
      b = e = 0;
      if (s < a.nseg) {
        b = __ldg(a.seg_begin + s);
        e = __ldg(a.seg_end + s);
      }
    };
    auto load = [&](uint32_t b, uint32_t e, uint32_t (&j)[4], double (&w)[4]) {
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t i = b + sub + u * COL_LANES;
        j[u] = i < e ? __ldg(a.col + i) : 0;
        w[u] = i < e ? __ldg(a.val + i) : 0.0;
      }
    };
    uint32_t b, e, j[4];
    double w[4];
    range(sg, b, e);
    load(b, e, j, w);
    range(sg + groups, b, e);
    for (uint32_t k = 0; k < rounds; ++k, sg += groups) {
      uint32_t nj[4];
      double nw[4];
      load(b, e, nj, nw);
      range(sg + 2 * groups, b, e);
      double acc = 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc += w[u] * y[j[u]];
        w[u] = nw[u];
        j[u] = nj[u];
      }
      reduce(acc);
    }
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

// RPT: vertices a thread owns (threadIdx.x, threadIdx.x + blockDim.x).
template <bool POLY, int RPT, bool MAT>
__global__ void __launch_bounds__(COL_MAX_THREADS, 1) k_pcg_columns(ColumnPcg a) {
  extern __shared__ double sh[];
  __shared__ double red[2][2][COL_MAX_THREADS / 32];
  const int j = blockIdx.x;
  const uint32_t n = a.n;
  double* p = sh;
  double* seg = p + n;
  double* t = seg + a.nseg;  // POLY: ws .* r
  column::Matrix m{};
  if constexpr (MAT) {
    double* val = t + (POLY ? n : 0);
    uint32_t* first = reinterpret_cast<uint32_t*>(val + a.nnz);
    uint16_t* col = reinterpret_cast<uint16_t*>(first + a.nseg + 1);
    for (uint32_t i = threadIdx.x; i < a.nnz; i += blockDim.x) {
      val[i] = a.val[i];
      col[i] = uint16_t(a.col[i]);
    }
    for (uint32_t i = threadIdx.x; i <= a.nseg; i += blockDim.x) first[i] = i < a.nseg ? a.seg_begin[i] : a.nnz;
    m.val = val;
    m.col16 = col;
    m.first = first;
  }
  int flip = 0;
  auto sum2 = [&](double& u, double& v) {
    column::block_sum(u, v, red[flip]);
    flip ^= 1;
  };
  // ---- own vertices
  bool own[RPT];
  uint32_t s0[RPT], s1[RPT];
  double d[RPT], wa[RPT], ws[RPT], r[RPT], x[RPT], z[RPT];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const uint32_t v = threadIdx.x + uint32_t(k) * blockDim.x;
    own[k] = v < n;
    s0[k] = own[k] ? a.row_first[v] : 0;
    s1[k] = own[k] ? a.row_first[v + 1] : 0;
    d[k] = own[k] ? a.diag[v] : 0.0;
    wa[k] = !own[k] ? 0.0 : POLY ? a.wa[v] : a.dinv[v];  // Jacobi: the inverse diagonal
    ws[k] = own[k] && POLY ? a.ws[v] : 0.0;
    r[k] = own[k] ? a.b[size_t(v) * a.K + j] : 0.0;
    x[k] = 0.0;
  }
  auto vertex = [&](int k) { return threadIdx.x + uint32_t(k) * blockDim.x; };
  // ---- start: the column's mean and norm (fresh), r = (b - mean) - L x
  double mean, tol2;
  int active, iters = 0;
  if (a.fresh) {
    double sum = 0.0, sq = 0.0;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      sum += r[k];
      sq += r[k] * r[k];
    }
    sum2(sum, sq);
    mean = sum / double(n);
    const double bb = fmax(sq - double(n) * mean * mean, 0.0);
    tol2 = a.tol * a.tol * bb;
    active = j < a.ncols && bb > 0.0 ? 1 : 0;
    if (threadIdx.x == 0) {
      a.s.mean[j] = mean;
      a.s.bb[j] = bb;
      a.s.tol2[j] = tol2;
      a.s.rr[j] = bb;
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k) r[k] = own[k] ? r[k] - mean : 0.0;
  } else {
    mean = a.s.mean[j];
    tol2 = a.s.tol2[j];
    active = a.s.active[j];
    iters = a.s.iters[j];
    if (active == 0) return;  // x stays as the last launch left it
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (own[k]) p[vertex(k)] = x[k] = a.x[size_t(vertex(k)) * a.K + j];
    __syncthreads();
    column::products<MAT>(a, m, p, seg);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (own[k]) r[k] = (r[k] - mean) - (d[k] * x[k] - column::row_sum(seg, s0[k], s1[k]));
  }
  // z = M r of the own vertices and r.z (Jacobi: over the values in hand)
  auto precondition = [&](double& rz) {
    rz = 0.0;
    if constexpr (POLY) {
#pragma unroll
      for (int k = 0; k < RPT; ++k)
        if (own[k]) t[vertex(k)] = ws[k] * r[k];
      __syncthreads();
      column::products<MAT>(a, m, t, seg);
      __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      z[k] = wa[k] * r[k];
      if (POLY && own[k]) z[k] += ws[k] * column::row_sum(seg, s0[k], s1[k]);
      rz += r[k] * z[k];
    }
  };
  double rz = 0.0, none = 0.0, rr_out = -1.0;
  __syncthreads();  // the matrix is in place; the restart's products have been read
  if (active == 1) {
    precondition(rz);
    sum2(rz, none);
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (own[k]) p[vertex(k)] = z[k];
    __syncthreads();
  }
  for (int it = 0; active == 1 && it < a.max_iters; ++it) {
    // ---- q = L p and p.q
    column::products<MAT>(a, m, p, seg);
    __syncthreads();
    double pq = 0.0, q[RPT], pv[RPT];
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      pv[k] = own[k] ? p[vertex(k)] : 0.0;
      q[k] = own[k] ? d[k] * pv[k] - column::row_sum(seg, s0[k], s1[k]) : 0.0;
      pq += pv[k] * q[k];
    }
    none = 0.0;
    sum2(pq, none);
    if (!(pq > 0.0) || !isfinite(pq)) {
      active = 2;  // nonpositive curvature
      break;
    }
    const double alpha = rz / pq;
    // ---- x += alpha p, r -= alpha q; r.r and (Jacobi) r.z
    double rr = 0.0, rzn = 0.0;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      x[k] += alpha * pv[k];
      r[k] -= alpha * q[k];
      rr += r[k] * r[k];
    }
    if (!POLY) precondition(rzn);
    sum2(rr, rzn);
    ++iters;
    rr_out = rr;
    if (rr <= tol2) {
      active = 0;
      break;
    }
    if constexpr (POLY) {
      precondition(rzn);
      none = 0.0;
      sum2(rzn, none);
    }
    const double beta = rzn / rz;
    rz = rzn;
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (own[k]) p[vertex(k)] = z[k] + beta * pv[k];
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < RPT; ++k)
    if (own[k]) a.x[size_t(vertex(k)) * a.K + j] = x[k];
  if (threadIdx.x == 0) {
    a.s.active[j] = active;
    a.s.iters[j] = iters;
    if (rr_out >= 0.0) a.s.rr[j] = rr_out;
  }
}

// Launch the variant for the problem's size on K columns.
inline void launch_pcg_columns(const ColumnPcg& a, bool poly, cudaStream_t s) {
  bool mat = false;
  const size_t smem = column_smem(a.n, a.nseg, a.nnz, poly, &mat);
  const int threads = column_threads(a.n);
  const bool two = a.n > uint32_t(threads);
  auto go = [&](auto kernel) {
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(COL_SMEM)));
    kernel<<<a.K, threads, smem, s>>>(a);
  };
  if (poly) {
    if (two) mat ? go(k_pcg_columns<true, 2, true>) : go(k_pcg_columns<true, 2, false>);
    else mat ? go(k_pcg_columns<true, 1, true>) : go(k_pcg_columns<true, 1, false>);
  } else {
    if (two) mat ? go(k_pcg_columns<false, 2, true>) : go(k_pcg_columns<false, 2, false>);
    else mat ? go(k_pcg_columns<false, 1, true>) : go(k_pcg_columns<false, 1, false>);
  }
  CK_LAUNCH();
}

}  // namespace fevcb
