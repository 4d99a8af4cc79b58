// Device code of the coarse correction's cycle (see afem_coarse.cu), shared by its own launches and the
// one-launch iteration of small systems.
#pragma once

#include "afem_hybrid.h"

namespace afem {

constexpr int COARSE_TAIL = 600;      // nodes of the first level the one-block cycle takes
constexpr int COARSE_STOP = 300;      // a grid of at most this many nodes is the coarsest
constexpr int COARSE_SWEEPS = 4;      // smoothing sweeps on the coarsest grid
constexpr int TAIL_THREADS = 512;
constexpr size_t TAIL_BYTES = 212 << 10;  // its shared memory (vectors, and the matrices that fit)
constexpr size_t TAIL_VALS = TAIL_BYTES / 16;
constexpr int TAIL_AXIS = 1024;       // axis weights of its levels
constexpr int COARSE_MIN_NODES = 64;  // smaller meshes keep the SSOR corrections alone
// Mesh nodes in the support of one grid node up to which the correction is taken (36 at most on box
// meshes).  Where a mesh is refined around a few points, its nodes crowd into few cells of a tensor
// grid: a step waits for one thread's support, and the correction leaves what varies inside the cell.
// Solves of 8 systems with the correction / by the colour sweeps alone, by the largest support: 734 125 /
// 187 ms, 1,240 123 / 125, 1,306 80 / 93, 1,968 153 / 126, 2,271 262 / 201, 7,059 3,466 / 834.
constexpr int COARSE_CROWD = 1500;

template <class T>
struct CV;
template <>
struct CV<double> {
  using V = double2;
};
template <>
struct CV<float> {
  using V = float2;
};

// weight of plane I of the next level at plane i of this one
__device__ __forceinline__ double axis_weight(int i, int I, bool halved, int nc, double w) {
  const int ci = min(halved ? i >> 1 : i, nc - 2);
  return I == ci ? 1.0 - w : (I == ci + 1 ? w : 0.0);
}

// D^-1 v with D the l1 row sums (0 on a dead row)
template <class T>
__device__ __forceinline__ typename CV<T>::V l1_solve(double2 d, double om, typename CV<T>::V v) {
  typename CV<T>::V o;
  const double k = d.x, m = om * d.y, s = k * k + m * m;
  const double inv = s > 0.0 ? 1.0 / s : 0.0;
  const T ix = (T)(k * inv), iy = (T)(-m * inv);
  o.x = ix * v.x - iy * v.y;
  o.y = ix * v.y + iy * v.x;
  return o;
}

// (T^T t) of level-1 node c, component cc, system s; t [mesh node][4][system].  Over the support's
// nodes p0 + q, p0 + q + G, ...: G lanes may share a support.
template <class T, int NS, int G>
__device__ __forceinline__ typename CV<T>::V mesh_down(int c, int cc, int s, int q, const int32_t* __restrict__ lptr,
                                                       const int32_t* __restrict__ lidx,
                                                       const double* __restrict__ lw,
                                                       const typename CV<T>::V* __restrict__ t) {
  typename CV<T>::V acc;
  acc.x = 0; acc.y = 0;
  const int p1 = __ldg(lptr + c + 1);
#pragma unroll 4
  for (int p = __ldg(lptr + c) + q; p < p1; p += G) {
    const T w = (T)__ldg(lw + p);
    const typename CV<T>::V v = t[((long)__ldg(lidx + p) * 4 + cc) * NS + s];
    acc.x += w * v.x;
    acc.y += w * v.y;
  }
  return acc;
}

template <class T>
__device__ __forceinline__ typename CV<T>::V cm(typename CV<T>::V a, typename CV<T>::V b) {
  typename CV<T>::V o;
  o.x = a.x * b.x - a.y * b.y;
  o.y = a.x * b.y + a.y * b.x;
  return o;
}

// R = T^T t at level 1 and Z = D^-1 R
template <class T, int NS>
__device__ __forceinline__ void grid_restrict(int n1, const int32_t* lptr, const int32_t* lidx, const double* lw,
                                              const typename CV<T>::V* t, const double2* l1, const double* omega,
                                              typename CV<T>::V* R, typename CV<T>::V* Z, int bid, int nb) {
  const long total = (long)n1 * 4 * NS;
  for (long i = bid * (long)blockDim.x + threadIdx.x; i < total; i += (long)nb * blockDim.x) {
    const int s = (int)(i % NS), cc = (int)(i / NS) & 3, c = (int)(i / (4 * NS));
    const double2 d = l1[4L * c + cc];
    typename CV<T>::V v = mesh_down<T, NS, 1>(c, cc, s, 0, lptr, lidx, lw, t);
    if (d.x == 0.0 && d.y == 0.0) { v.x = 0; v.y = 0; }
    R[i] = v;
    Z[i] = l1_solve<T>(d, omega[s], v);
  }
}

// (A v) at a node for one component and system: a = the component's first slot at the node, as =
// the stride between slots; v the vector at the node's own entry, vs its stride between nodes.  Slots
// outside the grid hold zeros, so they may be multiplied with any value (the node's own): no
// branches, and three entries are in flight together (nine cost registers and so resident warps).
template <class T>
__device__ __forceinline__ typename CV<T>::V grid_row(const CoarseGrid& g, int l, double om,
                                                      const typename CV<T>::V* __restrict__ a, long as,
                                                      const typename CV<T>::V* v, long vs) {
  const int i = l % g.nx, jk = l / g.nx, j = jk % g.ny, k = jk / g.ny;
  const bool x0 = i > 0, x1 = i + 1 < g.nx, y0 = j > 0, y1 = j + 1 < g.ny, z0 = k > 0, z1 = k + 1 < g.nz;
  T t1x = 0, t1y = 0, t2x = 0, t2y = 0;
#pragma unroll
  for (int b = 0; b < 27; b += 3) {
    typename CV<T>::V m[3], w[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int s = b + q, di = s % 3 - 1, dj = s / 3 % 3 - 1, dk = s / 9 - 1;
      const bool ok = (dk < 0 ? z0 : (dk > 0 ? z1 : true)) && (dj < 0 ? y0 : (dj > 0 ? y1 : true)) &&
                      (di < 0 ? x0 : (di > 0 ? x1 : true));
      m[q] = a[(long)s * as];
      w[q] = v[ok ? (long)(di + g.nx * (dj + g.ny * dk)) * vs : 0L];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      t1x += m[q].x * w[q].x; t1y += m[q].x * w[q].y;
      t2x += m[q].y * w[q].x; t2y += m[q].y * w[q].y;
    }
  }
  typename CV<T>::V o;
  o.x = t1x - (T)om * t2y;
  o.y = t1y + (T)om * t2x;
  return o;
}

// (P^T v) at node l of the next level g; v on level f
template <class T>
__device__ __forceinline__ typename CV<T>::V grid_down(const CoarseGrid& f, const CoarseGrid& g, int l,
                                                       const double* axw, const typename CV<T>::V* v,
                                                       long vs) {
  const bool hx = f.halved & 1, hy = f.halved & 2, hz = f.halved & 4;
  const int I = l % g.nx, J = (l / g.nx) % g.ny, K = l / (g.nx * g.ny);
  const int i0 = hx ? max(0, 2 * I - 1) : I, i1 = hx ? min(f.nx - 1, 2 * I + 1) : I;
  const int j0 = hy ? max(0, 2 * J - 1) : J, j1 = hy ? min(f.ny - 1, 2 * J + 1) : J;
  const int k0 = hz ? max(0, 2 * K - 1) : K, k1 = hz ? min(f.nz - 1, 2 * K + 1) : K;
  typename CV<T>::V o;
  o.x = 0; o.y = 0;
  for (int k = k0; k <= k1; ++k) {
    const double wk = axis_weight(k, K, hz, g.nz, axw[f.wz + k]);
    for (int j = j0; j <= j1; ++j) {
      const double wj = wk * axis_weight(j, J, hy, g.ny, axw[f.wy + j]);
      for (int i = i0; i <= i1; ++i) {
        const T w = (T)(wj * axis_weight(i, I, hx, g.nx, axw[f.wx + i]));
        const typename CV<T>::V x = v[(long)(i + f.nx * (j + f.ny * k)) * vs];
        o.x += w * x.x;
        o.y += w * x.y;
      }
    }
  }
  return o;
}

// (P v) at node l of level f; v on the next level g
template <class T>
__device__ __forceinline__ typename CV<T>::V grid_up(const CoarseGrid& f, const CoarseGrid& g, int l,
                                                     const double* axw, const typename CV<T>::V* v,
                                                     long vs) {
  const int i = l % f.nx, j = (l / f.nx) % f.ny, k = l / (f.nx * f.ny);
  const int I = min((f.halved & 1) ? i >> 1 : i, g.nx - 2), J = min((f.halved & 2) ? j >> 1 : j, g.ny - 2),
            K = min((f.halved & 4) ? k >> 1 : k, g.nz - 2);
  const double fx = axw[f.wx + i], fy = axw[f.wy + j], fz = axw[f.wz + k];
  typename CV<T>::V o;
  o.x = 0; o.y = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
    const double wd = (dx ? fx : 1.0 - fx) * (dy ? fy : 1.0 - fy) * (dz ? fz : 1.0 - fz);
    if (wd == 0.0) continue;
    const T w = (T)wd;
    const typename CV<T>::V x = v[(long)(I + dx + g.nx * (J + dy + g.ny * (K + dz))) * vs];
    o.x += w * x.x;
    o.y += w * x.y;
  }
  return o;
}

// Levels too large for one block: the steps of the V-cycle over (node, component, system),
// systems fastest, by nb blocks.  STEP 0: O = R - A Z (pre-smoothed residual); 1: R, Z of the next
// level g from O; 2: Z += P O_g; 3: O = Z + D^-1 (R - A Z), with the thread's part of R^T O.
template <class T, int NS, int STEP>
__device__ __forceinline__ void grid_step(const CoarseGrid& f, const CoarseGrid& g, const typename CV<T>::V* km,
                                          const double2* l1, const double* axw, const double* omega,
                                          typename CV<T>::V* R, typename CV<T>::V* Z, typename CV<T>::V* O,
                                          double (&rho)[1][2], int bid, int nb) {
  constexpr long VS = 4L * NS;
  const CoarseGrid& w = STEP == 1 ? g : f;
  const long total = (long)w.n * VS, fo = f.off * VS, go = g.off * VS;
  double px = 0.0, py = 0.0;
  for (long i = bid * (long)blockDim.x + threadIdx.x; i < total; i += (long)nb * blockDim.x) {
    const int s = (int)(i % NS), c = (int)(i / NS) & 3, l = (int)(i / VS);
    const long in = i % VS;  // component and system
    if constexpr (STEP == 0) {
      const typename CV<T>::V a = grid_row<T>(f, l, omega[s], km + 108L * f.off + (long)c * 27 * f.n + l, f.n,
                                              Z + fo + i, VS);
      typename CV<T>::V v = R[fo + i];
      v.x -= a.x; v.y -= a.y;
      O[fo + i] = v;
    } else if constexpr (STEP == 1) {
      const double2 d = l1[4L * (g.off + l) + c];
      typename CV<T>::V v = grid_down<T>(f, g, l, axw, O + fo + in, VS);
      if (d.x == 0.0 && d.y == 0.0) { v.x = 0; v.y = 0; }
      R[go + i] = v;
      Z[go + i] = l1_solve<T>(d, omega[s], v);
    } else if constexpr (STEP == 2) {
      const double2 d = l1[4L * (f.off + l) + c];
      if (d.x == 0.0 && d.y == 0.0) continue;
      const typename CV<T>::V u = grid_up<T>(f, g, l, axw, O + go + in, VS);
      typename CV<T>::V z = Z[fo + i];
      z.x += u.x; z.y += u.y;
      Z[fo + i] = z;
    } else {
      const typename CV<T>::V a = grid_row<T>(f, l, omega[s], km + 108L * f.off + (long)c * 27 * f.n + l, f.n,
                                              Z + fo + i, VS);
      const typename CV<T>::V r = R[fo + i];
      typename CV<T>::V z = Z[fo + i], e;
      e.x = r.x - a.x; e.y = r.y - a.y;
      e = l1_solve<T>(l1[4L * (f.off + l) + c], omega[s], e);
      z.x += e.x; z.y += e.y;
      O[fo + i] = z;
      px += (double)r.x * (double)z.x - (double)r.y * (double)z.y;
      py += (double)r.x * (double)z.y + (double)r.y * (double)z.x;
    }
  }
  rho[0][0] = px;
  rho[0][1] = py;
}

// Half of grid_row's sum for the one-block cycle, where two lanes share a node: slots q, q + 2, ...
// with the slots' node offsets `off` and the node's valid slots `ok` (bit per slot).
template <class T>
__device__ __forceinline__ void grid_half(int q, unsigned ok, const int* off, const typename CV<T>::V* __restrict__ a,
                                          int as, const typename CV<T>::V* v, T (&t)[4]) {
#pragma unroll
  for (int b = 0; b < 14; b += 7) {
    typename CV<T>::V m[7], w[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      const int s = min(q + 2 * (b + j), 26);
      const bool in = q + 2 * (b + j) < 27 && ((ok >> s) & 1);
      m[j] = a[(long)s * as];
      w[j] = v[in ? off[s] : 0];
      if (!in) m[j].x = m[j].y = 0;
    }
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      t[0] += m[j].x * w[j].x; t[1] += m[j].x * w[j].y;
      t[2] += m[j].y * w[j].x; t[3] += m[j].y * w[j].y;
    }
  }
}

// Valid slots of node (i, j, k): bit (di+1) + 3 (dj+1) + 9 (dk+1)
__device__ __forceinline__ unsigned grid_mask(const CoarseGrid& g, int l) {
  const int i = l % g.nx, jk = l / g.nx, j = jk % g.ny, k = jk / g.ny;
  unsigned m = 0x7ffffffu;
  if (i == 0) m &= ~0x1249249u;                 // di = -1: bits 0, 3, 6, ...
  if (i + 1 == g.nx) m &= ~(0x1249249u << 2);   // di = +1
  if (j == 0) m &= ~0x01c0e07u;                 // dj = -1: bits 0..2, 9..11, 18..20
  if (j + 1 == g.ny) m &= ~(0x01c0e07u << 6);   // dj = +1
  if (k == 0) m &= ~0x1ffu;                     // dk = -1
  if (k + 1 == g.nz) m &= ~(0x1ffu << 18);      // dk = +1
  return m;
}

template <class T>
__device__ __forceinline__ void copy_async(typename CV<T>::V* dst, const typename CV<T>::V* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

// The V-cycle from level `top` down, one block of TAIL_THREADS per (component, system) -- in a packed
// batch per (component, mesh) -- with `vals` values of shared memory at sh: the levels' R, Z and D^-1 and
// one scratch vector, then the matrices that fit.
// Starts from R of the top level, or (top = 0) from the mesh nodes' t, and writes the top level's O;
// rho (top = 0): the component's share of rho of its system.
// A step is one load latency long, so what bounds it is how many dependent loads it makes: the
// matrices of the lower levels that fit are copied to shared memory while the restriction runs, the
// inverse diagonals are formed once, the axis weights sit in shared memory, and the larger levels' rows
// come seven entries at a time on two lanes a node.  49.6 -> 21 us a cycle on 12x12x9 cells (one 245-node grid,
// whose four sweeps replaced two more levels).
template <class T, int NS, bool SEG>
__device__ __forceinline__ void grid_tail(int comp, int by, typename CV<T>::V* sh, const CoarseGrid* grids,
                                          const int32_t* levels, int top, int vals, const typename CV<T>::V* km,
                                          const double2* l1, const double* axw, const double* omega,
                                          const typename CV<T>::V* R, typename CV<T>::V* O, const int32_t* lptr,
                                          const int32_t* lidx, const double* lw, const typename CV<T>::V* t,
                                          double2* rho) {
  using V = typename CV<T>::V;
  __shared__ CoarseGrid gs[COARSE_LEVELS];
  __shared__ int so[COARSE_LEVELS], mo[COARSE_LEVELS];  // a level's vectors; its matrix (-1: in global memory)
  __shared__ int scratch, off[COARSE_LEVELS][27];
  __shared__ double aw[TAIL_AXIS];
  const int sg = SEG ? by : 0, s = SEG ? 0 : by;
  const double om = omega[by];
  const int nl = levels[sg];
  if (threadIdx.x < nl) gs[threadIdx.x] = grids[(long)sg * COARSE_LEVELS + threadIdx.x];
  __syncthreads();
  for (int u = threadIdx.x; u < nl * 27; u += TAIL_THREADS) {
    const int q = u % 27;
    off[u / 27][q] = q % 3 - 1 + gs[u / 27].nx * (q / 3 % 3 - 1 + gs[u / 27].ny * (q / 9 - 1));
  }
  const int aw0 = gs[top].wx;  // the axis weights of a mesh's levels are consecutive
  if (threadIdx.x == 0) {      // a level: R, Z, D^-1; then the scratch; then matrices from the coarsest up
    int o = 0;
    for (int l = top; l < nl; ++l) { so[l] = o; o += 3 * gs[l].n; }
    scratch = o;
    o += gs[top].n;
    for (int l = nl - 1; l >= top; --l) {
      mo[l] = -1;
      if (o + 27 * gs[l].n <= vals && (l == nl - 1 || mo[l + 1] >= 0)) { mo[l] = o; o += 27 * gs[l].n; }
    }
  }
  __syncthreads();
  for (int l = top; l < nl; ++l) {
    if (mo[l] < 0) continue;
    const V* src = km + 108L * gs[l].off + (long)comp * 27 * gs[l].n;
    for (int i = threadIdx.x; i < 27 * gs[l].n; i += TAIL_THREADS) copy_async<T>(sh + mo[l] + i, src + i);
  }
  if (nl - 1 > top) {
    const CoarseGrid& g = gs[nl - 2];
    for (int i = threadIdx.x; i < g.wz + g.nz - aw0; i += TAIL_THREADS) aw[i] = axw[aw0 + i];
  }
  V* tmp = sh + scratch;
  const double* ax = aw - aw0;
  constexpr long VS = 4L * NS;
  V one;
  one.x = 1; one.y = 0;
  for (int l = top; l < nl; ++l) {
    const CoarseGrid& g = gs[l];
    V* r = sh + so[l];
    for (int i = threadIdx.x; i < g.n; i += TAIL_THREADS) {
      const V d = l1_solve<T>(l1[4L * (g.off + i) + comp], om, one);
      r[2 * g.n + i] = d;
    }
  }
  __syncthreads();
  {
    const CoarseGrid& g = gs[top];
    V* r = sh + so[top];
    V* z = r + g.n;
    const V* d = z + g.n;
    if (top) {
      for (int i = threadIdx.x; i < g.n; i += TAIL_THREADS) {
        r[i] = R[((long)(g.off + i) * 4 + comp) * NS + s];
        z[i] = cm<T>(d[i], r[i]);
      }
    } else {  // four lanes share a support
      const int n4 = (4 * g.n + TAIL_THREADS - 1) / TAIL_THREADS * TAIL_THREADS;
      for (int u = threadIdx.x; u < n4; u += TAIL_THREADS) {
        const int i = u >> 2;
        V v;
        v.x = 0; v.y = 0;
        if (i < g.n) v = mesh_down<T, NS, 4>(g.off + i, comp, s, u & 3, lptr, lidx, lw, t);
#pragma unroll
        for (int m = 1; m < 4; m <<= 1) {
          v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
          v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
        }
        if (i < g.n && (u & 3) == 0) {
          if (d[i].x == 0 && d[i].y == 0) { v.x = 0; v.y = 0; }
          r[i] = v;
          z[i] = cm<T>(d[i], v);
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // f(i, (A z)_i) for every node of level l, two lanes a node
  auto product = [&](int l, const V* z, auto f) {
    const CoarseGrid& g = gs[l];
    const V* a = mo[l] >= 0 ? sh + mo[l] : km + 108L * g.off + (long)comp * 27 * g.n;
    const int n2 = (2 * g.n + TAIL_THREADS - 1) / TAIL_THREADS * TAIL_THREADS;
    for (int u = threadIdx.x; u < n2; u += TAIL_THREADS) {
      const int i = min(u >> 1, g.n - 1);
      T t[4] = {0, 0, 0, 0};
      grid_half<T>(u & 1, grid_mask(g, i), off[l], a + i, g.n, z + i, t);
#pragma unroll
      for (int m = 0; m < 4; ++m) t[m] += __shfl_xor_sync(0xffffffffu, t[m], 1);
      if ((u & 1) == 0 && (u >> 1) < g.n) {
        V o;
        o.x = t[0] - (T)om * t[3];
        o.y = t[1] + (T)om * t[2];
        f(i, o);
      }
    }
  };
  const V* zc = nullptr;  // the solution of the level below
  for (int l = top; l < nl; ++l) {  // down: the residual of z = D^-1 r to the next level
    const CoarseGrid& g = gs[l];
    V* r = sh + so[l];
    V* z = r + g.n;
    const V* d = z + g.n;
    if (l + 1 == nl) {
      V* from = z;
      V* to = tmp;
      for (int k = 1; k < COARSE_SWEEPS; ++k) {
        product(l, from, [&](int i, V a) {
          V e = r[i];
          e.x -= a.x; e.y -= a.y;
          e = cm<T>(d[i], e);
          e.x += from[i].x; e.y += from[i].y;
          to[i] = e;
        });
        __syncthreads();
        V* u = from;
        from = to;
        to = u;
      }
      zc = from;
      break;
    }
    product(l, z, [&](int i, V a) {
      V e = r[i];
      e.x -= a.x; e.y -= a.y;
      tmp[i] = e;
    });
    __syncthreads();
    const CoarseGrid& n = gs[l + 1];
    V* rn = sh + so[l + 1];
    for (int i = threadIdx.x; i < n.n; i += TAIL_THREADS) {
      V v = grid_down<T>(g, n, i, ax, tmp, 1);
      const V dn = rn[2 * n.n + i];
      if (dn.x == 0 && dn.y == 0) { v.x = 0; v.y = 0; }
      rn[i] = v;
      rn[n.n + i] = cm<T>(dn, v);
    }
    __syncthreads();
  }
  for (int l = nl - 2; l >= top; --l) {  // up: z += P z_next, then one sweep
    const CoarseGrid& g = gs[l];
    V* r = sh + so[l];
    V* z = r + g.n;
    const V* d = z + g.n;
    for (int i = threadIdx.x; i < g.n; i += TAIL_THREADS) {
      if (d[i].x == 0 && d[i].y == 0) continue;
      const V u = grid_up<T>(g, gs[l + 1], i, ax, zc, 1);
      z[i].x += u.x; z[i].y += u.y;
    }
    __syncthreads();
    product(l, z, [&](int i, V a) {
      V e = r[i];
      e.x -= a.x; e.y -= a.y;
      e = cm<T>(d[i], e);
      e.x += z[i].x; e.y += z[i].y;
      tmp[i] = e;
    });
    __syncthreads();
    zc = tmp;
  }
  const CoarseGrid& g = gs[top];
  const V* r = sh + so[top];
  double px = 0.0, py = 0.0;
  for (int i = threadIdx.x; i < g.n; i += TAIL_THREADS) {
    const V z = zc[i];
    O[((long)(g.off + i) * 4 + comp) * NS + s] = z;
    px += (double)r[i].x * (double)z.x - (double)r[i].y * (double)z.y;
    py += (double)r[i].x * (double)z.y + (double)r[i].y * (double)z.x;
  }
  if (!rho) return;
  __shared__ double red[TAIL_THREADS / 32][2];
  for (int m = 16; m > 0; m >>= 1) {
    px += __shfl_xor_sync(0xffffffffu, px, m);
    py += __shfl_xor_sync(0xffffffffu, py, m);
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5][0] = px; red[threadIdx.x >> 5][1] = py; }
  __syncthreads();
  if (threadIdx.x == 0) {
    px = py = 0.0;
    for (int b = 0; b < TAIL_THREADS / 32; ++b) { px += red[b][0]; py += red[b][1]; }
    rho[comp * RED_SYS + by] = make_double2(px, py);
  }
}

}  // namespace afem
