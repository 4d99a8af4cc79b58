// Coarse correction of the gradient-corrected COCG (AFEM_PRECOND_HYBRID).
//
// Smoothing on the edges and on the gradients (the polynomials of afem_solver.cu's smoothed iteration)
// removes the error that varies from edge to edge; what is left is smooth, and its reduction would take
// as many iterations as the mesh is cells wide.  Following Hiptmair and Xu (SIAM J.
// Numer. Anal. 45, 2007) the smooth part of an edge field is represented by
// nodal functions: the gradient of a scalar potential and a vector field whose
// three components are taken one by one,
//
//     z += sum_{c=0..3} Q_c B_c Q_c^T r,   Q_0 = G T,  Q_k = Pi_k T,
//
// with G the edge-node incidence, (Pi_k v)_e = (x_head - x_tail)_k (v_head +
// v_tail) / 2 and T the trilinear interpolation from a tensor-product grid
// about twice as coarse as the mesh (its planes are quantiles of the node
// coordinates, so a graded mesh gets a graded grid and an unstructured one
// planes where its nodes are).  B_c is one symmetric V-cycle on the Galerkin
// matrices Q_c^T A Q_c, kept as pairs (K, M) like the edge matrix, over grids
// halved per axis; its smoother is l1-Jacobi, D = sum_j |K_ij| + i omega
// sum_j |M_ij|, which needs no estimate of the largest eigenvalue on stretched
// cells.  Everything is complex symmetric, so COCG applies as before.
// Measured to 1e-10 on a B200 in FP64, the colour sweeps alone against sweeps and correction against the
// smoothed iteration with it: 461, 59, 69 iterations and 361, 70, 49 ms on 48x48x32 cells (8 systems), about
// 850, 65, 70 and 1,290, 151, 103 ms on 88x88x56 (one system), 110, 43, 50 and 30, 16, 3.3 ms on 12x12x9.
//
// The four components and the systems are independent below the restriction,
// so the lower levels of the V-cycle run as one block per (component, system)
// with its vectors in shared memory and no grid-wide step at all; only levels
// of more than COARSE_TAIL nodes take launches of their own.
#include <algorithm>
#include <cmath>

#include "afem_coarse.cuh"
#include "afem_hybrid.h"

namespace afem {

namespace {

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ int pk(int i, int j, int k) { return i | (j << 10) | (k << 20); }

// ------------------------------------------------------------------ pattern (once per mesh)
__global__ void k_edge_vec(const double* __restrict__ xyz, const int32_t* __restrict__ line, int n,
                           double* __restrict__ te) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const double* a = xyz + 3L * (line[2L * e] - 1);
  const double* b = xyz + 3L * (line[2L * e + 1] - 1);
  for (int d = 0; d < 3; ++d) te[3L * e + d] = b[d] - a[d];
}

__device__ __forceinline__ int find_plane(const double* __restrict__ p, int n, double x) {
  int lo = 0, hi = n - 1;  // p[lo] <= x < p[hi] as far as x lies inside
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (p[m] <= x) lo = m;
    else hi = m;
  }
  return lo;
}

// Cell of each mesh node in its mesh's level-1 grid and its position there; counts the supports.
// planes: the meshes' x, y and z planes one after another, from pofs[mesh].
__global__ void k_node_cells(const double* __restrict__ xyz, int node, const uint8_t* __restrict__ seg,
                             const CoarseGrid* __restrict__ grids, const double* __restrict__ planes,
                             const int32_t* __restrict__ pofs, int32_t* __restrict__ corner,
                             double* __restrict__ frac, int32_t* __restrict__ cnt) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= node) return;
  const int sg = seg ? seg[a] : 0;
  const CoarseGrid g = grids[(long)sg * COARSE_LEVELS];
  const int np[3] = {g.nx, g.ny, g.nz};
  const double* p = planes + pofs[sg];
  int ijk[3];
  double f[3];
  for (int d = 0; d < 3; ++d) {
    const double x = xyz[3L * a + d];
    const int i = find_plane(p, np[d], x);
    double t = (x - p[i]) / (p[i + 1] - p[i]);
    t = t > 0.0 ? (t < 1.0 ? t : 1.0) : 0.0;
    ijk[d] = i;
    f[d] = t;
    frac[3L * a + d] = t;
    p += np[d];
  }
  corner[a] = pk(ijk[0], ijk[1], ijk[2]);
  const int base = g.off + ijk[0] + g.nx * (ijk[1] + g.ny * ijk[2]);
  for (int q = 0; q < 8; ++q) {
    const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
    if ((dx ? f[0] : 1 - f[0]) * (dy ? f[1] : 1 - f[1]) * (dz ? f[2] : 1 - f[2]) != 0.0)
      atomicAdd(cnt + base + dx + g.nx * (dy + g.ny * dz), 1);
  }
}

__global__ void k_support_max(int n1, const int32_t* __restrict__ cnt, int* __restrict__ most) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = __reduce_max_sync(0xffffffffu, c < n1 ? cnt[c] : 0);
  if ((threadIdx.x & 31) == 0) atomicMax(most, v);
}

__global__ void k_support_fill(int node, const uint8_t* __restrict__ seg, const CoarseGrid* __restrict__ grids,
                               const int32_t* __restrict__ corner, const double* __restrict__ frac,
                               const int32_t* __restrict__ lptr, int32_t* __restrict__ cur,
                               int32_t* __restrict__ lidx) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= node) return;
  const CoarseGrid g = grids[(long)(seg ? seg[a] : 0) * COARSE_LEVELS];
  const int c = corner[a];
  const double fx = frac[3L * a], fy = frac[3L * a + 1], fz = frac[3L * a + 2];
  const int base = g.off + (c & 1023) + g.nx * (((c >> 10) & 1023) + g.ny * (c >> 20));
  for (int q = 0; q < 8; ++q) {
    const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
    if ((dx ? fx : 1 - fx) * (dy ? fy : 1 - fy) * (dz ? fz : 1 - fz) != 0.0) {
      const int ci = base + dx + g.nx * (dy + g.ny * dz);
      lidx[lptr[ci] + atomicAdd(cur + ci, 1)] = a;
    }
  }
}

// The atomics above fill a support in any order: sorted ascending, sums over it have one order
// (insertion sort: ~27 nodes on a box mesh).
__global__ void k_support_sort(int n1, const int32_t* __restrict__ lptr, int32_t* __restrict__ lidx) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n1) return;
  const int b = lptr[c], e = lptr[c + 1];
  for (int i = b + 1; i < e; ++i) {
    const int v = lidx[i];
    int j = i;
    for (; j > b && lidx[j - 1] > v; --j) lidx[j] = lidx[j - 1];
    lidx[j] = v;
  }
}

__global__ void k_cseg(int nseg, const CoarseGrid* __restrict__ grids, int n1, uint8_t* __restrict__ cseg) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n1) return;
  int s = 0;
  while (s + 1 < nseg && c >= grids[(long)(s + 1) * COARSE_LEVELS].off) ++s;
  cseg[c] = (uint8_t)s;
}

// ------------------------------------------------------------------ values (once per assembly)
// A node with a Dirichlet edge takes no part in the correction: its interpolation is zero.
__global__ void k_free_cells(int node, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nlist,
                             const uint8_t* __restrict__ bc, const uint8_t* __restrict__ seg,
                             const CoarseGrid* __restrict__ grids, const int32_t* __restrict__ corner,
                             int32_t* __restrict__ cell) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= node) return;
  bool fixed = false;
  for (int q = nptr[a]; q < nptr[a + 1]; ++q) fixed |= bc[nlist[q] >> 1] != 0;
  const CoarseGrid g = grids[(long)(seg ? seg[a] : 0) * COARSE_LEVELS];
  const int c = corner[a];
  cell[a] = fixed ? -1 : g.off + (c & 1023) + g.nx * (((c >> 10) & 1023) + g.ny * (c >> 20));
}

// trilinear weight of grid node (i, j, k) at a position in the cell with lowest corner c
__device__ __forceinline__ double corner_weight(int i, int j, int k, int c, double fx, double fy, double fz) {
  const int dx = i - (c & 1023), dy = j - ((c >> 10) & 1023), dz = k - (c >> 20);
  const double wx = dx == 0 ? 1.0 - fx : (dx == 1 ? fx : 0.0);
  const double wy = dy == 0 ? 1.0 - fy : (dy == 1 ? fy : 0.0);
  const double wz = dz == 0 ? 1.0 - fz : (dz == 1 ? fz : 0.0);
  return wx * wy * wz;
}

__global__ void k_support_weights(int n1, const uint8_t* __restrict__ cseg, const CoarseGrid* __restrict__ grids,
                                  const int32_t* __restrict__ lptr, const int32_t* __restrict__ lidx,
                                  const int32_t* __restrict__ corner, const double* __restrict__ frac,
                                  const int32_t* __restrict__ cell, double* __restrict__ lw) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n1) return;
  const CoarseGrid g = grids[(long)cseg[c] * COARSE_LEVELS];
  const int l = c - g.off, i = l % g.nx, j = (l / g.nx) % g.ny, k = l / (g.nx * g.ny);
  for (int p = lptr[c]; p < lptr[c + 1]; ++p) {
    const int a = lidx[p];
    lw[p] = cell[a] < 0 ? 0.0
                        : corner_weight(i, j, k, corner[a], frac[3L * a], frac[3L * a + 1], frac[3L * a + 2]);
  }
}

// One component's row from the warp's slots (lane < 27), with the row sums of |K| and |M|; a dead
// row (zero diagonal) gets zero sums.
__device__ __forceinline__ void store_row(double2 v, int lane, int c, const CoarseGrid& g, int l,
                                          double2* __restrict__ km, double2* __restrict__ l1) {
  if (lane < 27) km[108L * g.off + (long)(c * 27 + lane) * g.n + l] = v;
  double sk = lane < 27 ? fabs(v.x) : 0.0, sm = lane < 27 ? fabs(v.y) : 0.0;
  for (int m = 16; m > 0; m >>= 1) {
    sk += __shfl_xor_sync(0xffffffffu, sk, m);
    sm += __shfl_xor_sync(0xffffffffu, sm, m);
  }
  const double dk = __shfl_sync(0xffffffffu, v.x, 13), dm = __shfl_sync(0xffffffffu, v.y, 13);
  if (lane == 0) l1[4L * (g.off + l) + c] = (dk == 0.0 && dm == 0.0) ? make_double2(0.0, 0.0) : make_double2(sk, sm);
}

// Level 1: T^T N_c T.  A block of four warps per grid node, a lane per slot; the warps take the
// support's mesh nodes in turn.  The entries of a mesh node's row are fetched by 32 lanes at once and
// handed round through shared memory, so a row costs one load latency and not one per entry (a lane
// per slot reading entry by entry took 2.8 ms on 88x88x56 cells and 0.22 ms on 12x12x9).
constexpr int GM_WARPS = 4;
struct MeshEntry {  // a nodal row's entry: its column's place in the grid and the four components
  double fx, fy, fz;
  int corner, pad;
  double2 v[4];
};
__global__ void __launch_bounds__(32 * GM_WARPS)
    k_galerkin_mesh(const uint8_t* __restrict__ cseg, const CoarseGrid* __restrict__ grids,
                    const int32_t* __restrict__ lptr, const int32_t* __restrict__ lidx,
                    const double* __restrict__ lw, const int32_t* __restrict__ corner,
                    const double* __restrict__ frac, const int32_t* __restrict__ cell,
                    const int32_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                    const double2* __restrict__ n0, const double2* __restrict__ n3, double2* __restrict__ km,
                    double2* __restrict__ l1) {
  __shared__ MeshEntry ent[GM_WARPS][32];
  __shared__ double2 sum[GM_WARPS][4][32];
  const int c = blockIdx.x, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const CoarseGrid g = grids[(long)cseg[c] * COARSE_LEVELS];
  const int l = c - g.off;
  const int i = l % g.nx + lane % 3 - 1, j = (l / g.nx) % g.ny + (lane / 3) % 3 - 1,
            k = l / (g.nx * g.ny) + lane / 9 - 1;
  double2 acc[4] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
  for (int p = lptr[c] + w; p < lptr[c + 1]; p += GM_WARPS) {
    const double wa = lw[p];
    if (wa == 0.0) continue;
    const int a = lidx[p], r1 = rowptr[a + 1];
    for (int q0 = rowptr[a]; q0 < r1; q0 += 32) {
      const int q = q0 + lane;
      bool take = false;
      MeshEntry x;
      if (q < r1) {
        const int b = col[q];
        take = cell[b] >= 0;
        x.corner = corner[b];
        x.fx = frac[3L * b]; x.fy = frac[3L * b + 1]; x.fz = frac[3L * b + 2];
        x.v[0] = n0[q];
        for (int m = 0; m < 3; ++m) x.v[m + 1] = n3[3L * q + m];
      }
      const unsigned have = __ballot_sync(0xffffffffu, take);
      if (take) ent[w][__popc(have & ((1u << lane) - 1))] = x;
      __syncwarp();
      const int cnt = __popc(have);
      for (int e = 0; e < cnt; ++e) {
        const MeshEntry& y = ent[w][e];
        const double wt = wa * corner_weight(i, j, k, y.corner, y.fx, y.fy, y.fz);
        if (wt != 0.0)
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            acc[m].x += wt * y.v[m].x;
            acc[m].y += wt * y.v[m].y;
          }
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) sum[w][m][lane] = acc[m];
  __syncthreads();
  // warp m adds component m
  double2 v = sum[0][w][lane];
  for (int u = 1; u < GM_WARPS; ++u) {
    v.x += sum[u][w][lane].x;
    v.y += sum[u][w][lane].y;
  }
  store_row(v, lane, w, g, l, km, l1);
}

// Level l + 1 from level l of each mesh that has both: P^T A P with P the product of three axis
// interpolations, applied axis by axis.  A block per node of the next level, a warp per component: the
// up to 27 x 27 entries around the node go to shared memory (one latency), then the axes are
// contracted one after another, 9 terms a value (a lane per slot reading the 729 entries in turn
// took 0.3 to 0.5 ms a level whatever its size).
__global__ void __launch_bounds__(128)
    k_galerkin_grid(const CoarseGrid* __restrict__ grids, const int32_t* __restrict__ levels, int lev,
                    const double* __restrict__ axw, double2* __restrict__ km, double2* __restrict__ l1) {
  __shared__ double W[3][27];          // [axis][fine plane ii][fine slot s][coarse slot S]
  __shared__ double2 E[4][27 * 9];     // fine entries of three x planes at a time, then the y stage
  __shared__ double2 X[4][27 * 9];     // after the x axis: [kk][jj][sz][sy][SX]
  const int sg = blockIdx.y;
  if (lev + 1 >= levels[sg]) return;
  const CoarseGrid f = grids[(long)sg * COARSE_LEVELS + lev], g = grids[(long)sg * COARSE_LEVELS + lev + 1];
  const int l = blockIdx.x, c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (l >= g.n) return;
  const int N[3] = {g.nx, g.ny, g.nz}, n[3] = {f.nx, f.ny, f.nz}, wo[3] = {f.wx, f.wy, f.wz};
  const int I[3] = {l % g.nx, (l / g.nx) % g.ny, l / (g.nx * g.ny)};
  int lo[3], cnt[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const bool h = (f.halved >> d) & 1;
    lo[d] = h ? max(0, 2 * I[d] - 1) : I[d];
    cnt[d] = (h ? min(n[d] - 1, 2 * I[d] + 1) : I[d]) - lo[d] + 1;
  }
  if (threadIdx.x < 81) {
    const int d = threadIdx.x / 27, ii = threadIdx.x % 27 / 9, s = threadIdx.x % 9 / 3 - 1, S = threadIdx.x % 3 - 1;
    const bool h = (f.halved >> d) & 1;
    const int i = lo[d] + ii, b = i + s;
    double w = 0.0;
    if (ii < cnt[d] && b >= 0 && b < n[d])
      w = axis_weight(i, I[d], h, N[d], axw[wo[d] + i]) * axis_weight(b, I[d] + S, h, N[d], axw[wo[d] + b]);
    W[d][threadIdx.x % 27] = w;
  }
  __syncthreads();
  const double2* A = km + 108L * f.off + (long)c * 27 * f.n;
  // x axis, three fine planes kk in turn: E[ii][jj][slot] (9 x 27 entries), X[kk][jj][sz][sy][SX]
  for (int kk = 0; kk < 3; ++kk) {
    for (int q = lane; q < 243; q += 32) {
      const int ii = q % 3, jj = q / 3 % 3, s = q / 9;
      double2 v = make_double2(0.0, 0.0);
      if (ii < cnt[0] && jj < cnt[1] && kk < cnt[2])
        v = A[(long)s * f.n + (lo[0] + ii) + f.nx * ((lo[1] + jj) + f.ny * (lo[2] + kk))];
      E[c][q] = v;
    }
    __syncwarp();
    for (int q = lane; q < 81; q += 32) {  // q = SX + 3 (sy + 3 (sz + 3 jj))
      const int SX = q % 3, sy = q / 3 % 3, sz = q / 9 % 3, jj = q / 27;
      double2 v = make_double2(0.0, 0.0);
#pragma unroll
      for (int ii = 0; ii < 3; ++ii)
#pragma unroll
        for (int sx = 0; sx < 3; ++sx) {
          const double w = W[0][ii * 9 + sx * 3 + SX];
          const double2 e = E[c][ii + 3 * jj + 9 * (sx + 3 * sy + 9 * sz)];
          v.x += w * e.x;
          v.y += w * e.y;
        }
      X[c][q + 81 * kk] = v;
    }
    __syncwarp();
  }
  // y axis: Y[kk][sz][SY][SX] in E
  for (int q = lane; q < 81; q += 32) {  // q = SX + 3 (SY + 3 (sz + 3 kk))
    const int SX = q % 3, SY = q / 3 % 3, sz = q / 9 % 3, kk = q / 27;
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int jj = 0; jj < 3; ++jj)
#pragma unroll
      for (int sy = 0; sy < 3; ++sy) {
        const double w = W[1][jj * 9 + sy * 3 + SY];
        const double2 e = X[c][SX + 3 * (sy + 3 * (sz + 3 * jj)) + 81 * kk];
        v.x += w * e.x;
        v.y += w * e.y;
      }
    E[c][q] = v;
  }
  __syncwarp();
  double2 v = make_double2(0.0, 0.0);
  if (lane < 27) {
    const int SZ = lane / 9;
#pragma unroll
    for (int kk = 0; kk < 3; ++kk)
#pragma unroll
      for (int sz = 0; sz < 3; ++sz) {
        const double w = W[2][kk * 9 + sz * 3 + SZ];
        const double2 e = E[c][lane % 9 + 9 * (sz + 3 * kk)];
        v.x += w * e.x;
        v.y += w * e.y;
      }
  }
  store_row(v, lane, c, g, l, km, l1);
}

__global__ void k_to_float(const double2* __restrict__ in, float2* __restrict__ out, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = make_float2((float)in[i].x, (float)in[i].y);
}

// ------------------------------------------------------------------ application
// The steps as launches (the grids are small where they matter: see COARSE_TAIL).
template <class T, int NS>
__global__ void __launch_bounds__(256)
    k_grid_restrict(int n1, const int32_t* __restrict__ lptr, const int32_t* __restrict__ lidx,
                    const double* __restrict__ lw, const typename CV<T>::V* __restrict__ t,
                    const double2* __restrict__ l1, const double* __restrict__ omega,
                    typename CV<T>::V* __restrict__ R, typename CV<T>::V* __restrict__ Z,
                    const int* __restrict__ done) {
  if (*done) return;
  grid_restrict<T, NS>(n1, lptr, lidx, lw, t, l1, omega, R, Z, blockIdx.x, gridDim.x);
}

template <class T, int NS, int STEP>
__global__ void __launch_bounds__(256)
    k_grid_step(const CoarseGrid f, const CoarseGrid g, const typename CV<T>::V* __restrict__ km,
                const double2* __restrict__ l1, const double* __restrict__ axw, const double* __restrict__ omega,
                typename CV<T>::V* __restrict__ R, typename CV<T>::V* __restrict__ Z, typename CV<T>::V* __restrict__ O,
                const int* __restrict__ done, double2* __restrict__ rho, RedSet red) {
  if (*done) return;
  double v[1][2];
  grid_step<T, NS, STEP>(f, g, km, l1, axw, omega, R, Z, O, v, blockIdx.x, gridDim.x);
  if constexpr (STEP == 3) {
    if (!rho) return;
    // the grid's stride is a multiple of 32, so a lane keeps its system
    __shared__ double2 sums[RED_SYS], buf[8 * NS];
    block_pair<NS, 1, NS>(v, threadIdx.x % NS, true, red, blockIdx.x, buf);
    if (reduce_blocks(red, blockIdx.x, gridDim.x, NS, sums) && threadIdx.x < NS) {
      rho[threadIdx.x] = sums[threadIdx.x];
      for (int c = 1; c < 4; ++c) rho[c * RED_SYS + threadIdx.x] = make_double2(0.0, 0.0);
    }
  }
}

template <class T, int NS, bool SEG>
__global__ void __launch_bounds__(TAIL_THREADS)
    k_grid_tail(const CoarseGrid* __restrict__ grids, const int32_t* __restrict__ levels, int top, int vals,
                const typename CV<T>::V* __restrict__ km, const double2* __restrict__ l1,
                const double* __restrict__ axw, const double* __restrict__ omega,
                const typename CV<T>::V* __restrict__ R, typename CV<T>::V* __restrict__ O,
                const int32_t* __restrict__ lptr, const int32_t* __restrict__ lidx, const double* __restrict__ lw,
                const typename CV<T>::V* __restrict__ t, const int* __restrict__ done, double2* __restrict__ rho) {
  if (*done) return;
  extern __shared__ double2 tail_smem[];
  grid_tail<T, NS, SEG>(blockIdx.x, blockIdx.y, reinterpret_cast<typename CV<T>::V*>(tail_smem), grids, levels, top,
                        vals, km, l1, axw, omega, R, O, lptr, lidx, lw, t, rho);
}

// ------------------------------------------------------------------ host: grids of one mesh
// Planes of one axis: about m slabs holding equal shares of the nodes, ends at the extent.  The
// coordinates are binned (a node layer of a box mesh falls into one bin, whose smallest coordinate
// stands for it), so a plane passes through the nodes of a layered mesh.
void axis_planes(const double* xyz, int a0, int a1, int d, int m, std::vector<double>& out) {
  constexpr int BINS = 8192;
  double lo = xyz[3L * a0 + d], hi = lo;
  for (int a = a0; a < a1; ++a) {
    lo = std::min(lo, xyz[3L * a + d]);
    hi = std::max(hi, xyz[3L * a + d]);
  }
  out.clear();
  out.push_back(lo);
  if (m > 1 && hi > lo) {
    std::vector<int> cnt(BINS, 0);
    std::vector<double> low(BINS, hi);
    const double sc = BINS / (hi - lo);
    for (int a = a0; a < a1; ++a) {
      const double x = xyz[3L * a + d];
      const int b = std::min(BINS - 1, std::max(0, (int)((x - lo) * sc)));
      cnt[b] += 1;
      low[b] = std::min(low[b], x);
    }
    const double share = (double)(a1 - a0) / m;
    // a slab's upper plane is the first layer at which the nodes below and on it exceed its share
    long cum = 0;
    int j = 1;
    for (int b = 0; b < BINS && j < m; ++b) {
      if (!cnt[b]) continue;
      cum += cnt[b];
      if ((double)cum > j * share + 0.5) {
        if (low[b] > out.back() && low[b] < hi) out.push_back(low[b]);
        while (j < m && (double)cum > j * share + 0.5) ++j;
      }
    }
  }
  out.push_back(hi);
}

}  // namespace

size_t coarse_bytes(const HybridState* h, int ns, int pb) {
  const CoarseState* co = h->co;
  return (size_t)2 * pb * ns * 3 * 4 * (size_t)co->ntot;
}

// The grids of every mesh and the mesh nodes' places in them.  Slabs per axis: half the node
// layers, estimated from the mean edge extent along the axis (over the edges that have one), scaled
// down together where the product would exceed an eighth of the nodes (unstructured meshes).
void coarse_pattern(afem_ctx* c) {
  HybridState* h = c->hyb;
  if (!h->co) h->co = new CoarseState();
  CoarseState* co = h->co;
  cudaStream_t s = c->stream;
  const int node = c->node, nline = c->nline, nseg = std::max(1, c->nseg);
  co->on = false;
  co->values_gen = -1;
  co->nseg = nseg;
  std::vector<double> xyz(3L * node);
  std::vector<int32_t> ln(2L * nline);
  c->xyz.download(xyz.data(), xyz.size(), s);
  c->line.download(ln.data(), ln.size(), s);
  AFEM_CUDA(cudaStreamSynchronize(s));
  co->grids.assign((size_t)nseg * COARSE_LEVELS, CoarseGrid());
  co->levels.assign(nseg, 0);
  std::vector<std::vector<double>> pls[3];
  std::vector<double> planes;
  std::vector<int32_t> pofs(nseg);
  for (int d = 0; d < 3; ++d) pls[d].resize(nseg);
  int e0 = 0, off = 0;
  for (int sg = 0; sg < nseg; ++sg) {
    const int a0 = c->nseg > 0 ? c->seg_node_ptr[sg] : 0, a1 = c->nseg > 0 ? c->seg_node_ptr[sg + 1] : node;
    const int e1 = c->nseg > 0 ? c->seg_row_ptr[sg + 1] : nline;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, sum[3] = {0.0, 0.0, 0.0}, cells[3];
    double prod = 1.0;
    long cnt[3] = {0, 0, 0};
    for (int a = a0; a < a1; ++a)
      for (int d = 0; d < 3; ++d) {
        lo[d] = std::min(lo[d], xyz[3L * a + d]);
        hi[d] = std::max(hi[d], xyz[3L * a + d]);
      }
    for (int d = 0; d < 3; ++d)  // a flat or unreadable mesh: no correction
      if (!(hi[d] - lo[d] > 0.0) || !std::isfinite(hi[d] - lo[d])) return;
    for (int e = e0; e < e1; ++e) {
      const double* p = xyz.data() + 3L * (ln[2L * e] - 1);
      const double* q = xyz.data() + 3L * (ln[2L * e + 1] - 1);
      for (int d = 0; d < 3; ++d) {
        const double t = std::fabs(q[d] - p[d]);
        if (t > 1e-9 * (hi[d] - lo[d])) { sum[d] += t; cnt[d] += 1; }
      }
    }
    for (int d = 0; d < 3; ++d) {
      if (!cnt[d] || !std::isfinite(sum[d])) return;
      cells[d] = std::max(1.0, 0.5 * (hi[d] - lo[d]) * cnt[d] / sum[d]);
      prod *= cells[d];
    }
    e0 = e1;
    if (a1 - a0 < COARSE_MIN_NODES && nseg == 1) return;
    double scale = prod > (a1 - a0) / 8.0 ? std::cbrt((a1 - a0) / 8.0 / prod) : 1.0;
    CoarseGrid* G = co->grids.data() + (size_t)sg * COARSE_LEVELS;
    for (;;) {  // packed batches: the whole cycle of a mesh has to fit one block
      long n1 = 1;
      for (int d = 0; d < 3; ++d) {
        const int m = std::min(256, std::max(1, (int)std::lround(cells[d] * scale)));
        axis_planes(xyz.data(), a0, a1, d, m, pls[d][sg]);
        n1 *= (long)pls[d][sg].size();
      }
      if (nseg == 1 || n1 * 4.6 < TAIL_VALS || scale < 1e-3) break;
      scale *= 0.9;
    }
    pofs[sg] = (int)planes.size();
    for (int d = 0; d < 3; ++d) planes.insert(planes.end(), pls[d][sg].begin(), pls[d][sg].end());
    G[0].nx = (int)pls[0][sg].size();
    G[0].ny = (int)pls[1][sg].size();
    G[0].nz = (int)pls[2][sg].size();
    G[0].n = G[0].nx * G[0].ny * G[0].nz;
    G[0].off = off;
    off += G[0].n;
    co->levels[sg] = 1;
  }
  co->n1 = off;
  co->nlev = 1;
  std::vector<double> axw;
  for (int sg = 0; sg < nseg; ++sg) {
    CoarseGrid* G = co->grids.data() + (size_t)sg * COARSE_LEVELS;
    int l = 0;
    for (; l + 1 < COARSE_LEVELS && G[l].n > COARSE_STOP && std::max(G[l].nx, std::max(G[l].ny, G[l].nz)) > 3; ++l) {
      int* nc[3] = {&G[l + 1].nx, &G[l + 1].ny, &G[l + 1].nz};
      int* wo[3] = {&G[l].wx, &G[l].wy, &G[l].wz};
      for (int d = 0; d < 3; ++d) {
        std::vector<double>& p = pls[d][sg];
        const bool half = p.size() > 3;
        std::vector<double> q;
        if (half) {
          G[l].halved |= 1 << d;
          for (size_t i = 0; i + 1 < p.size(); i += 2) q.push_back(p[i]);
          q.push_back(p.back());
        } else {
          q = p;
        }
        *wo[d] = (int)axw.size();
        for (size_t i = 0; i < p.size(); ++i) {
          const size_t ci = std::min(half ? i / 2 : i, q.size() - 2);
          axw.push_back((p[i] - q[ci]) / (q[ci + 1] - q[ci]));
        }
        *nc[d] = (int)q.size();
        p = q;
      }
      G[l + 1].n = G[l + 1].nx * G[l + 1].ny * G[l + 1].nz;
      G[l + 1].off = off;
      off += G[l + 1].n;
    }
    co->levels[sg] = l + 1;
    co->nlev = std::max(co->nlev, l + 1);
  }
  co->ntot = off;
  co->tail = 0;
  if (nseg == 1)
    while (co->grids[co->tail].n > COARSE_TAIL && co->tail + 1 < co->levels[0]) ++co->tail;
  co->tail_vals = 0;
  for (int sg = 0; sg < nseg; ++sg) {
    const CoarseGrid* G = co->grids.data() + (size_t)sg * COARSE_LEVELS;
    size_t v = G[co->tail].n, ax = 0, all;
    for (int l = co->tail; l < co->levels[sg]; ++l) {
      v += 3 * (size_t)G[l].n;
      ax += G[l].nx + G[l].ny + G[l].nz;
    }
    if (v > TAIL_VALS || ax > TAIL_AXIS) return;  // (a grid of hundreds of planes on one axis)
    all = v;
    for (int l = co->tail; l < co->levels[sg]; ++l) all += 27 * (size_t)G[l].n;
    co->tail_vals = std::max(co->tail_vals, all);
  }
  if (axw.empty()) axw.push_back(0.0);
  co->d_grids.upload(co->grids.data(), co->grids.size(), s);
  co->d_levels.upload(co->levels.data(), co->levels.size(), s);
  co->planes.upload(planes.data(), planes.size(), s);
  co->axw.upload(axw.data(), axw.size(), s);
  DBuf<int32_t> dpofs, cnt, dmost;
  dpofs.upload(pofs.data(), pofs.size(), s);
  co->corner.alloc(node);
  co->frac.alloc(3L * node);
  co->cell.alloc(node);
  co->te.alloc(3L * nline);
  co->cseg.alloc(co->n1);
  cnt.alloc(co->n1);
  cnt.zero(s);
  const uint8_t* seg = c->nseg > 0 ? h->seg.p : nullptr;
  k_edge_vec<<<nblk(nline, 256), 256, 0, s>>>(c->xyz.p, c->line.p, nline, co->te.p);
  count_launch();
  k_node_cells<<<nblk(node, 256), 256, 0, s>>>(c->xyz.p, node, seg, co->d_grids.p, co->planes.p, dpofs.p,
                                               co->corner.p, co->frac.p, cnt.p);
  count_launch();
  k_cseg<<<nblk(co->n1, 256), 256, 0, s>>>(nseg, co->d_grids.p, co->n1, co->cseg.p);
  count_launch();
  int most = 0;
  dmost.upload(&most, 1, s);
  k_support_max<<<nblk(co->n1, 256), 256, 0, s>>>(co->n1, cnt.p, dmost.p);
  count_launch();
  dmost.download(&most, 1, s);
  AFEM_CUDA(cudaStreamSynchronize(s));  // (the host vectors above may go out of scope, too)
  if (most > COARSE_CROWD) return;
  long total = 0;
  co->lptr.alloc(co->n1 + 1);
  exclusive_scan(cnt.p, co->lptr.p, co->n1, s, &total);
  co->lidx.alloc(std::max(1L, total));
  co->lw.alloc(std::max(1L, total));
  cnt.zero(s);
  k_support_fill<<<nblk(node, 256), 256, 0, s>>>(node, seg, co->d_grids.p, co->corner.p, co->frac.p, co->lptr.p,
                                                 cnt.p, co->lidx.p);
  count_launch();
  k_support_sort<<<nblk(co->n1, 128), 128, 0, s>>>(co->n1, co->lptr.p, co->lidx.p);
  count_launch();
  co->n3.alloc(3 * h->nnz);
  co->km.alloc(108L * co->ntot);
  co->l1.alloc(4L * co->ntot);
  AFEM_CUDA(cudaStreamSynchronize(s));  // the host vectors above go out of scope
  co->on = true;
}

void coarse_values(afem_ctx* c) {
  HybridState* h = c->hyb;
  CoarseState* co = h->co;
  if (!co || !co->on || co->values_gen == c->assemble_gen) return;
  cudaStream_t s = c->stream;
  const int node = c->node;
  const uint8_t* seg = c->nseg > 0 ? h->seg.p : nullptr;
  k_free_cells<<<nblk(node, 256), 256, 0, s>>>(node, h->nptr.p, h->nlist.p, c->bc.p, seg, co->d_grids.p, co->corner.p,
                                               co->cell.p);
  count_launch();
  k_support_weights<<<nblk(co->n1, 128), 128, 0, s>>>(co->n1, co->cseg.p, co->d_grids.p, co->lptr.p, co->lidx.p,
                                                      co->corner.p, co->frac.p, co->cell.p, co->lw.p);
  count_launch();
  k_galerkin_mesh<<<co->n1, 32 * GM_WARPS, 0, s>>>(co->cseg.p, co->d_grids.p, co->lptr.p, co->lidx.p,
                                                          co->lw.p, co->corner.p, co->frac.p, co->cell.p, h->rowptr.p,
                                                          h->col.p, h->km.p, co->n3.p, co->km.p, co->l1.p);
  count_launch();
  for (int l = 0; l + 1 < co->nlev; ++l) {
    int nmax = 1;
    for (int sg = 0; sg < co->nseg; ++sg)
      if (l + 1 < co->levels[sg]) nmax = std::max(nmax, co->grids[(size_t)sg * COARSE_LEVELS + l + 1].n);
    k_galerkin_grid<<<dim3(nmax, co->nseg), 128, 0, s>>>(co->d_grids.p, co->d_levels.p, l, co->axw.p,
                                                                          co->km.p, co->l1.p);
    count_launch();
  }
  co->kmf_valid = false;
  co->values_gen = c->assemble_gen;
}

// FP32 copy of the Galerkin matrices (outside any graph capture)
void coarse_float(afem_ctx* c) {
  CoarseState* co = c->hyb->co;
  if (!co || !co->on || co->kmf_valid) return;
  co->kmf.alloc(co->km.n);
  k_to_float<<<c->num_sms * 8, 256, 0, c->stream>>>(co->km.p, co->kmf.p, (long)co->km.n);
  count_launch();
  co->kmf_valid = true;
}

void coarse_destroy(HybridState* h) {
  delete h->co;
  h->co = nullptr;
}

template <class PT, int NS, bool SEG>
const void* coarse_cycle(afem_ctx* c, const CoarseArgs& a) {
  using V = typename CV<PT>::V;
  CoarseState* co = c->hyb->co;
  cudaStream_t s = c->stream;
  const size_t vec = (size_t)4 * NS * co->ntot;
  V* R = static_cast<V*>(a.buf);
  V* Z = R + vec;
  V* O = Z + vec;
  const V* t = static_cast<const V*>(a.t);
  const V* km;
  if constexpr (sizeof(PT) == 8) km = co->km.p;
  else km = co->kmf.p;
  const unsigned wide = c->num_sms * 8;
  if (co->tail > 0) {
    k_grid_restrict<PT, NS><<<std::min(wide, nblk(4L * co->n1 * NS, 256)), 256, 0, s>>>(
        co->n1, co->lptr.p, co->lidx.p, co->lw.p, t, co->l1.p, a.omega, R, Z, a.done);
    count_launch();
  }
  auto step = [&](auto tag, int l, int nodes, double2* rho) {
    constexpr int ST = decltype(tag)::value;
    const unsigned g = std::min(nblk(4L * nodes * NS, 256), std::min(wide, (unsigned)a.red.rows));
    k_grid_step<PT, NS, ST><<<g, 256, 0, s>>>(co->grids[l], co->grids[l + 1], km, co->l1.p, co->axw.p, a.omega, R, Z,
                                              O, a.done, rho, a.red);
    count_launch();
  };
  if constexpr (!SEG)
    for (int l = 0; l < co->tail; ++l) {
      step(std::integral_constant<int, 0>(), l, co->grids[l].n, nullptr);
      step(std::integral_constant<int, 1>(), l, co->grids[l + 1].n, nullptr);
    }
  const size_t smem = std::min(TAIL_BYTES, sizeof(V) * co->tail_vals);
  auto tail = k_grid_tail<PT, NS, SEG>;
  allow_shared(tail, TAIL_BYTES);
  tail<<<dim3(4, SEG ? co->nseg : NS), TAIL_THREADS, smem, s>>>(
      co->d_grids.p, co->d_levels.p, co->tail, (int)(smem / sizeof(V)), km, co->l1.p, co->axw.p, a.omega, R, O, co->lptr.p, co->lidx.p,
      co->lw.p, t, a.done, co->tail == 0 ? a.rho : nullptr);
  count_launch();
  if constexpr (!SEG)
    for (int l = co->tail - 1; l >= 0; --l) {
      step(std::integral_constant<int, 2>(), l, co->grids[l].n, nullptr);
      step(std::integral_constant<int, 3>(), l, co->grids[l].n, l == 0 ? a.rho : nullptr);
    }
  return O;
}

#define AFEM_COARSE(NS, SEG)                                                                 \
  template const void* coarse_cycle<double, NS, SEG>(afem_ctx*, const CoarseArgs&);          \
  template const void* coarse_cycle<float, NS, SEG>(afem_ctx*, const CoarseArgs&);
AFEM_COARSE(1, false)
AFEM_COARSE(2, false)
AFEM_COARSE(4, false)
AFEM_COARSE(8, false)
AFEM_COARSE(16, false)
AFEM_COARSE(1, true)
#undef AFEM_COARSE

}  // namespace afem
