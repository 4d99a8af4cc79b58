// Gradient-space (nodal) correction of the COCG preconditioner: device state.
#pragma once

#include "afem_internal.h"
#include "afem_reduce.cuh"

namespace afem {

struct CoarseState;

struct HybridState {
  int node = 0, nline = 0;
  long nnz = 0;
  bool pattern_ready = false;
  bool colours_ready = false;   // the multicolour order and its split rows
  long split_gen = -1;          // assembly generation of lkm / ukm
  bool coarse_ready = false;    // co was set up for this mesh (it may have found no hierarchy)
  long values_gen = -1;         // assembly generation the values belong to
  DBuf<int32_t> nptr, nlist;    // node -> incident edges (edge << 1 | tail flag), ascending
  DBuf<int32_t> rowptr, col;    // nodal pattern (node graph), columns ascending
  DBuf<int32_t> diagpos;
  DBuf<double2> km;             // (K_G, M_G) per nodal entry
  DBuf<uint8_t> live;           // 1 when the node has a non-Dirichlet edge
  DBuf<uint8_t> color;          // nodal multicolour order
  DBuf<int32_t> perm, cptr;
  int ncolors = 0;
  // rows in colour order, split into earlier-colour (l*) and later-colour (u*) parts;
  // *src = index of the entry in the nodal CSR, *km the values (FP64, FP32 copies)
  DBuf<int32_t> lptr, lcol, lsrc, uptr, ucol, usrc;
  DBuf<double2> lkm, ukm;
  DBuf<float2> lkmf, ukmf;
  bool splitf_valid = false;    // lkmf, ukmf match lkm, ukm
  DBuf<uint8_t> seg;            // packed batches: mesh of each node
  int seg_nseg = 0;
  CoarseState* co = nullptr;    // coarse correction (owned; afem_coarse.cu)
};

// One tensor-product grid of the coarse correction (a level of one mesh's hierarchy).
// Nodes are numbered x fastest; the grid's nodes, matrix entries and axis weights sit at
// the given offsets of the pools in CoarseState.  A node (i, j, k) has up to 27 neighbours,
// slot (di+1) + 3 (dj+1) + 9 (dk+1).
struct CoarseGrid {
  int off = 0, n = 0;           // nodes: pool index off .. off + n
  int nx = 0, ny = 0, nz = 0;
  int halved = 0;               // bit d: axis d is halved towards the next level
  int wx = 0, wy = 0, wz = 0;   // axis pool: weight of the upper coarse plane at each plane
};
constexpr int COARSE_LEVELS = 9;

// Coarse correction of the gradient-corrected SSOR: see afem_coarse.cu.
struct CoarseState {
  bool on = false;              // the mesh has a hierarchy (false: too few nodes for one)
  long values_gen = -1;         // assembly generation of the values
  int nseg = 0;                 // meshes (1, or the packed batch's)
  int nlev = 0;                 // levels of the deepest mesh
  int n1 = 0, ntot = 0;         // level-1 nodes and nodes of all levels, all meshes
  int tail = 0;                 // first level that the one-block V-cycle takes
  size_t tail_vals = 0;         // its shared values per block (largest mesh)
  std::vector<CoarseGrid> grids;    // [mesh * COARSE_LEVELS + level]
  std::vector<int32_t> levels;      // levels of each mesh
  DBuf<CoarseGrid> d_grids;
  DBuf<int32_t> d_levels;
  DBuf<double> planes, axw;     // level-1 plane coordinates; axis weights of every grid
  DBuf<int32_t> corner;         // mesh node -> packed (i, j, k) of its level-1 cell
  DBuf<double> frac;            // mesh node -> position in the cell, 3 values
  DBuf<int32_t> cell;           // mesh node -> pool index of the cell's lowest corner, -1: Dirichlet node
  DBuf<int32_t> lptr, lidx;     // level-1 node -> mesh nodes in its support, ascending
  DBuf<double> lw;              // their weights (0 for Dirichlet nodes)
  DBuf<uint8_t> cseg;           // level-1 node -> mesh
  DBuf<double> te;              // edge vectors x_head - x_tail, 3 values per edge
  DBuf<double2> n3;             // nodal matrices of the vector components, 3 per nodal entry
  DBuf<double2> km;             // (K, M) of every grid, [27 grid.off * 4 + (comp * 27 + slot) * n + node]
  DBuf<float2> kmf;             // FP32 copy
  bool kmf_valid = false;
  DBuf<double2> l1;             // (sum |K|, sum |M|) of each row, [(off + node) * 4 + comp]; 0: dead row
};

// node graph (once per mesh) and A_G (once per assembly); coarse: also the coarse correction;
// colours: also the colouring and the colour-ordered rows of the nodal sweeps
void hybrid_prepare(afem_ctx* c, bool coarse, bool colours);
void hybrid_invalidate(afem_ctx* c);  // the mesh changed
void hybrid_destroy(afem_ctx* c);
void hybrid_export(afem_ctx* c, int* node, long* nnz, int32_t* rowptr, int32_t* col, double* km);


// afem_coarse.cu
void coarse_pattern(afem_ctx* c);     // grids, supports and interpolation, once per mesh
void coarse_values(afem_ctx* c);      // Galerkin matrices, once per assembly
void coarse_float(afem_ctx* c);      // their FP32 copy
void coarse_destroy(HybridState* h);
// Bytes of the work vectors of one solve (pb: bytes of a preconditioner real, ns systems per row)
size_t coarse_bytes(const HybridState* h, int ns, int pb);
struct CoarseArgs {
  const void* t;        // mesh nodes' right-hand sides (G^T r, Pi_k^T r) [node][4][system]
  void* buf;            // coarse_bytes
  const double* omega;  // per system
  const int* done;      // the batch has finished: every kernel returns
  double2* rho;         // the correction's share of rho, 4 rows of RED_SYS values (to be added up)
  RedSet red;           // block sums
};
// The V-cycle of every component and system; returns the level-1 values [grid node][4][system].
template <class PT, int NS, bool SEG>
const void* coarse_cycle(afem_ctx* c, const CoarseArgs& a);

}  // namespace afem
