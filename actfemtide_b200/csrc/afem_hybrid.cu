// Gradient-space (nodal) correction for COCG: the set-up half.
//
// The curl-curl operator vanishes on discrete gradients, so in the resistive
// air (sigma = 1e-8 S/m) the edge system has eigenvalues ~1e-12 of the rest
// along the gradients of nodal functions; SSOR on the edges does not reach
// them and COCG stagnates.  The hybrid preconditioner of Hiptmair (SIAM J.
// Numer. Anal. 36, 1998) adds a correction in that subspace:
//
//     z = SSOR_edge(r) + G SSOR_node(G^T r),   A_G = G^T A G,
//
// with G the edge-node incidence (G x)_e = x_n2(e) - x_n1(e) over the edges
// that are not Dirichlet.  A_G is formed here as a Galerkin product of the
// assembled edge matrix, split like A: A_G(omega) = K_G + i omega M_G, one
// (K_G, M_G) pair per nodal entry.  Its pattern is the node graph of the mesh
// (two nodes of one tetrahedron share an edge), so row a holds a and the far
// ends of a's edges.  The nodal SSOR runs multicoloured like the edge one.
#include <algorithm>

#include "afem_hybrid.h"

namespace afem {

namespace {

constexpr int NODE_EDGE_MAX = 128;  // edges meeting at one node

// The node graph from the edges.  bad[0..2]: the first edge with a bad node id, the first node with too
// many edges, the first with a repeated one.
__global__ void k_node_degree(const int32_t* __restrict__ line, int nline, int node, int32_t* __restrict__ deg,
                              int32_t* __restrict__ bad) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nline) return;
  const int a = line[2L * e] - 1, b = line[2L * e + 1] - 1;
  if (a < 0 || a >= node || b < 0 || b >= node || a == b) {
    atomicMin(bad, e);
    return;
  }
  atomicAdd(deg + a, 1);
  atomicAdd(deg + b, 1);
}

__global__ void k_check_degree(const int32_t* __restrict__ deg, int node, int32_t* __restrict__ bad) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < node && deg[a] > NODE_EDGE_MAX) atomicMin(bad + 1, a);
}

__global__ void k_node_fill(const int32_t* __restrict__ line, int nline, const int32_t* __restrict__ nptr,
                            int32_t* __restrict__ cur, int32_t* __restrict__ nlist) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nline) return;
  const int a = line[2L * e] - 1, b = line[2L * e + 1] - 1;
  nlist[nptr[a] + atomicAdd(cur + a, 1)] = (e << 1) | 1;
  nlist[nptr[b] + atomicAdd(cur + b, 1)] = e << 1;
}

// Sorts a node's edges (the atomics above leave any order) and writes its row, a thread per node: an
// insertion sort of ~14 entries.
__global__ void k_node_rows(const int32_t* __restrict__ line, int node, const int32_t* __restrict__ nptr,
                            int32_t* __restrict__ nlist, int32_t* __restrict__ rowptr, int32_t* __restrict__ col,
                            int32_t* __restrict__ diagpos, int32_t* __restrict__ bad) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a > node) return;
  const int b = nptr[a];
  rowptr[a] = a + b;  // a row holds the node and its edges' far ends
  if (a == node) return;
  const int e = nptr[a + 1];
  for (int i = b + 1; i < e; ++i) {
    const int v = nlist[i];
    int j = i;
    for (; j > b && nlist[j - 1] > v; --j) nlist[j] = nlist[j - 1];
    nlist[j] = v;
  }
  int32_t* row = col + a + b;
  int len = 0;
  for (int i = b - 1; i < e; ++i) {
    const int v = i < b ? a : ((nlist[i] & 1) ? line[2L * (nlist[i] >> 1) + 1] : line[2L * (nlist[i] >> 1)]) - 1;
    int j = len++;
    for (; j > 0 && row[j - 1] > v; --j) row[j] = row[j - 1];
    row[j] = v;
  }
  for (int k = 0; k < len; ++k) {
    if (k && row[k] == row[k - 1]) atomicMin(bad + 2, a);
    if (row[k] == a) diagpos[a] = a + b + k;
  }
}

// Nodal matrices on the node graph: A_G = G^T P (K, M) P G, and with VEC the vector components'
// Pi_k^T P (K, M) P Pi_k (n3[3 * entry + k]).  Half a warp per row, a lane per entry, so an entry stays
// in registers over the row's edges; an edge's matrix row is fetched by the lanes at once and handed
// round through shared memory (one load latency per edge and not per entry: two kernels that read
// entry by entry took 5.1 + 7.5 ms on 88x88x56 cells, 0.46 + 0.11 ms on 12x12x9).  The sums run over
// the edges and their entries in order.
struct EdgeEntry {
  int head, tail;  // 1-based node ids, 0: a Dirichlet edge
  double2 v;
  double tx, ty, tz;
};
template <bool VEC>
__global__ void __launch_bounds__(256)
    k_node_values(const int32_t* __restrict__ line, const uint8_t* __restrict__ bc, int node,
                  const int32_t* __restrict__ nptr, const int32_t* __restrict__ nlist,
                  const int32_t* __restrict__ erow, const int32_t* __restrict__ ecol,
                  const double2* __restrict__ ekm, const double* __restrict__ te, const int32_t* __restrict__ rowptr,
                  const int32_t* __restrict__ col, double2* __restrict__ km, double2* __restrict__ n3,
                  uint8_t* __restrict__ live) {
  __shared__ EdgeEntry ent[16][16];
  const int hw = threadIdx.x >> 4, lane = threadIdx.x & 15;
  const unsigned mask = 0xffffu << (threadIdx.x & 16);
  const long a = blockIdx.x * 16L + hw;
  if (a >= node) return;
  const int r0 = rowptr[a], r1 = rowptr[a + 1], i0 = nptr[a], i1 = nptr[a + 1];
  bool any = false;
  for (int q0 = r0; q0 < r1; q0 += 16) {
    const int q = q0 + lane, b = q < r1 ? col[q] + 1 : -1;
    double2 s0 = make_double2(0.0, 0.0), s1 = s0, s2 = s0, s3 = s0;
    for (int i = i0; i < i1; ++i) {
      const int el = nlist[i], e = el >> 1;
      if (bc[e]) continue;
      any = true;
      const double ga = (el & 1) ? -1.0 : 1.0;
      double ex = 0.0, ey = 0.0, ez = 0.0;
      if constexpr (VEC) {
        ex = 0.25 * te[3L * e];
        ey = 0.25 * te[3L * e + 1];
        ez = 0.25 * te[3L * e + 2];
      }
      const int k1 = erow[e + 1];
      for (int k0 = erow[e]; k0 < k1; k0 += 16) {
        const int k = k0 + lane;
        if (k < k1) {
          const int f = ecol[k];
          EdgeEntry x;
          const bool free = !bc[f];
          x.tail = free ? line[2L * f] : 0;
          x.head = free ? line[2L * f + 1] : 0;
          x.v = ekm[k];
          if constexpr (VEC) {
            x.tx = te[3L * f];
            x.ty = te[3L * f + 1];
            x.tz = te[3L * f + 2];
          }
          ent[hw][lane] = x;
        }
        __syncwarp(mask);
        const int cnt = min(16, k1 - k0);
        for (int m = 0; m < cnt; ++m) {
          const EdgeEntry& y = ent[hw][m];
          const bool h = y.head == b, t = y.tail == b;
          if (h || t) {
            const double2 v = y.v;
            const double g = h ? ga : -ga;
            s0.x += g * v.x; s0.y += g * v.y;
            if constexpr (VEC) {
              const double wx = ex * y.tx, wy = ey * y.ty, wz = ez * y.tz;
              s1.x += wx * v.x; s1.y += wx * v.y;
              s2.x += wy * v.x; s2.y += wy * v.y;
              s3.x += wz * v.x; s3.y += wz * v.y;
            }
          }
        }
        __syncwarp(mask);
      }
    }
    if (q < r1) {
      km[q] = s0;
      if constexpr (VEC) {
        n3[3L * q] = s1;
        n3[3L * q + 1] = s2;
        n3[3L * q + 2] = s3;
      }
    }
  }
  if (lane == 0) live[a] = any ? 1 : 0;
}

__global__ void k_gather_km(const double2* __restrict__ km, const int32_t* __restrict__ src, long cnt,
                            double2* __restrict__ out) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < cnt) out[k] = km[src[k]];
}

__global__ void k_node_seg(const int32_t* __restrict__ ptr, int nseg, int node, uint8_t* __restrict__ seg) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= node) return;
  int k = 0;
  while (k + 1 < nseg && a >= ptr[k + 1]) ++k;
  seg[a] = (uint8_t)k;
}

inline unsigned nblk(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void hybrid_prepare(afem_ctx* c, bool coarse, bool colours) {
  AFEM_REQUIRE(c->node > 0 && c->nline > 0 && c->line.p, AFEM_ESTATE,
               "hybrid preconditioner: needs the mesh (not available for a system loaded in split layout)");
  AFEM_REQUIRE(c->assembled, AFEM_ESTATE, "hybrid preconditioner: assemble first");
  if (!c->hyb) c->hyb = new HybridState();
  HybridState* h = c->hyb;
  cudaStream_t s = c->stream;
  const int node = c->node;
  if (h->node != node || h->nline != c->nline || !h->pattern_ready) {
    h->node = node;
    h->nline = c->nline;
    // The node graph, once per mesh: incident edges per node in ascending edge order
    // (edge << 1 | 1 at the tail line(1,e), edge << 1 at the head), rows = the node and the far
    // ends of its edges, ascending.
    const int nline = c->nline;
    const long nnz = node + 2L * nline;
    DBuf<int32_t> deg, bad;
    deg.alloc(node);
    deg.zero(s);
    const int32_t none[3] = {INT32_MAX, INT32_MAX, INT32_MAX};
    int32_t found[3];
    bad.upload(none, 3, s);
    k_node_degree<<<nblk(nline, 256), 256, 0, s>>>(c->line.p, nline, node, deg.p, bad.p);
    count_launch();
    k_check_degree<<<nblk(node, 256), 256, 0, s>>>(deg.p, node, bad.p);
    count_launch();
    bad.download(found, 3, s);
    AFEM_CUDA(cudaStreamSynchronize(s));
    AFEM_REQUIRE(found[0] == INT32_MAX, AFEM_EINVAL,
                 "hybrid preconditioner: edge " + std::to_string(found[0] + 1L) + " has a bad node id");
    AFEM_REQUIRE(found[1] == INT32_MAX, AFEM_EPATTERN,
                 "hybrid preconditioner: more than 128 edges meet at node " + std::to_string(found[1] + 1L));
    h->nptr.alloc(node + 1);
    exclusive_scan(deg.p, h->nptr.p, node, s, nullptr);
    h->nlist.alloc(2L * nline);
    h->rowptr.alloc(node + 1);
    h->col.alloc(nnz);
    h->diagpos.alloc(node);
    deg.zero(s);
    k_node_fill<<<nblk(nline, 256), 256, 0, s>>>(c->line.p, nline, h->nptr.p, deg.p, h->nlist.p);
    count_launch();
    k_node_rows<<<nblk(node + 1, 128), 128, 0, s>>>(c->line.p, node, h->nptr.p, h->nlist.p, h->rowptr.p, h->col.p,
                                                    h->diagpos.p, bad.p);
    count_launch();
    bad.download(found, 3, s);
    AFEM_CUDA(cudaStreamSynchronize(s));
    AFEM_REQUIRE(found[2] == INT32_MAX, AFEM_EPATTERN,
                 "hybrid preconditioner: repeated edge at node " + std::to_string(found[2] + 1L));
    h->nnz = nnz;
    h->km.alloc(nnz);
    h->live.alloc(node);
    h->pattern_ready = true;
    h->values_gen = -1;
    h->coarse_ready = h->colours_ready = false;
  }
  if (c->nseg > 0 && (int)h->seg_nseg != c->nseg) {
    DBuf<int32_t> ptr;
    ptr.upload(c->seg_node_ptr.data(), c->nseg + 1, s);
    h->seg.alloc(node);
    k_node_seg<<<nblk(node, 256), 256, 0, s>>>(ptr.p, c->nseg, node, h->seg.p);
    count_launch();
    AFEM_CUDA(cudaStreamSynchronize(s));
    h->seg_nseg = c->nseg;
    h->coarse_ready = false;
  }
  if (coarse && !h->coarse_ready) {
    coarse_pattern(c);
    h->coarse_ready = true;
  }
  const bool vec = coarse && h->co->on && h->co->values_gen != c->assemble_gen;
  if (h->values_gen != c->assemble_gen || vec) {
    auto k = vec ? k_node_values<true> : k_node_values<false>;
    k<<<nblk(node, 16), 256, 0, s>>>(c->line.p, c->bc.p, node, h->nptr.p, h->nlist.p, c->rowptr.p, c->col.p, c->km.p,
                                     vec ? h->co->te.p : nullptr, h->rowptr.p, h->col.p, h->km.p,
                                     vec ? h->co->n3.p : nullptr, h->live.p);
    count_launch();
    h->values_gen = c->assemble_gen;
    h->splitf_valid = false;
  }
  if (vec) coarse_values(c);
  if (colours && !h->colours_ready) {
    std::vector<int32_t> rp(node + 1), cl(h->nnz);
    h->rowptr.download(rp.data(), rp.size(), s);
    h->col.download(cl.data(), cl.size(), s);
    AFEM_CUDA(cudaStreamSynchronize(s));
    std::vector<int32_t> pm(node), cptr(256);
    std::vector<uint8_t> color(node);
    // multicolour order of the node graph (host greedy colouring, as for the edges)
    const int nc = compute_coloring(node, rp.data(), cl.data(), color.data(), pm.data(), cptr.data(), 255);
    AFEM_REQUIRE(nc > 0, AFEM_EPATTERN, "hybrid preconditioner: more than 255 colours in the node graph");
    h->ncolors = nc;
    h->color.upload(color.data(), node, s);
    h->perm.upload(pm.data(), node, s);
    h->cptr.upload(cptr.data(), nc + 1, s);
    // colour-ordered split rows of the node graph, built on the device like the edges'
    split_rows_device(c, h->rowptr.p, h->col.p, h->diagpos.p, h->color.p, h->perm.p, node, h->lptr, h->lcol, h->lsrc,
                      h->uptr, h->ucol, h->usrc, nullptr);
    h->lkm.alloc(h->lcol.n);
    h->ukm.alloc(h->ucol.n);
    AFEM_CUDA(cudaStreamSynchronize(s));
    h->colours_ready = true;
    h->split_gen = -1;
  }
  if (colours && h->split_gen != c->assemble_gen) {
    if (h->lcol.n) {
      k_gather_km<<<nblk((long)h->lcol.n, 256), 256, 0, s>>>(h->km.p, h->lsrc.p, (long)h->lcol.n, h->lkm.p);
      count_launch();
    }
    if (h->ucol.n) {
      k_gather_km<<<nblk((long)h->ucol.n, 256), 256, 0, s>>>(h->km.p, h->usrc.p, (long)h->ucol.n, h->ukm.p);
      count_launch();
    }
    h->split_gen = c->assemble_gen;
    h->splitf_valid = false;
  }
  AFEM_CUDA(cudaStreamSynchronize(s));
}

void hybrid_invalidate(afem_ctx* c) {
  if (c->hyb) {
    c->hyb->pattern_ready = false;
    c->hyb->seg_nseg = 0;
  }
}

void hybrid_destroy(afem_ctx* c) {
  if (c->hyb) coarse_destroy(c->hyb);
  delete c->hyb;
  c->hyb = nullptr;
}

// Host only: the nodal matrix of the last preparation, for tests.
void hybrid_export(afem_ctx* c, int* node, long* nnz, int32_t* rowptr, int32_t* col, double* km) {
  hybrid_prepare(c, false, false);
  HybridState* h = c->hyb;
  if (node) *node = h->node;
  if (nnz) *nnz = h->nnz;
  cudaStream_t s = c->stream;
  if (rowptr) h->rowptr.download(rowptr, h->node + 1, s);
  if (col) h->col.download(col, h->nnz, s);
  if (km) h->km.download(reinterpret_cast<double2*>(km), h->nnz, s);
  AFEM_CUDA(cudaStreamSynchronize(s));
}

}  // namespace afem
