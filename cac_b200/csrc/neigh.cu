// Periodic wrap, cell binning and neighbour-list construction.
//
// Lists hold, for every i-site (atoms, then the 8 Gauss points of each
// element), the atoms and element lattice sites within cutneigh = cut + skin,
// with the periodic image of each neighbour.  Membership is decided in the
// reference's FP64 arithmetic, so the sets equal the reference's bit for bit:
//   atom j:           rsq of xi - (xj + s*L)          (npair_half_bin_newton.cpp:116-120)
//   lattice site j:   xi - sum_k N_k (xnode_k + s*L)  subtracted node by node
//                                                     (npair_half_bin_newton.cpp:194-200)
// with products and differences rounded separately (no FMA).
//
// Candidates come from two periodic cell grids instead of the reference's
// bin/stencil/sub-element walk: atoms from a grid of cell >= cutneigh with a
// 3x3x3 stencil (atoms: one block per chunk of 32 cell-sorted atoms, the
// atoms as lanes sharing broadcast candidate loads; Gauss points: one warp
// each, the lanes over the candidates), element sites
// from a grid over element centres of cell >= cutneigh + (centre-to-node
// radius + affine deviation), and for each candidate element only the lattice
// sites whose affine position can lie within cutneigh (a box in lattice-index
// space).  Both prunings are exact supersets, so they change cost, not
// membership.
//
// Full lists are written in their final form: an entry packs the neighbour's
// pair-table index (atoms by list slot) with its image; a site's entries
// inside the inner radius at build time fill its list from row 0 up, the
// others from row cap-1 down, so no pass reorders them.  Element-site entries
// are first written as (item, lattice site) along their query's own row (the
// pair-table index of a lattice site is known only once every list has marked
// the sites it uses) and converted by k_remap_sites.  Half lists (read only by the list download)
// are written as raw entries and compacted by k_remap.
//
// Storage rules (the reference's, restated):
//   full  (npair_full_bin.cpp:23-358): every neighbour except the site itself.
//   half  (npair_half_bin_newton.cpp:25-392): an atom keeps atom j when j's
//         reference bin is in its upper half stencil, or in the same bin when j
//         is owned and later in order, or a ghost "above and to the right";
//         it keeps every lattice site.  A Gauss point keeps no atoms, every
//         non-Gauss lattice site, and a Gauss site once: owned (element i < j,
//         or same element and igcell < jgcell) or ghost with its element
//         centre above and to the right.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <tuple>
#include <type_traits>

#include "ctx.cuh"
#include "device.cuh"

namespace cacb200 {

namespace {

// Marks of an element's lattice sites: a byte each while lists are built, then
// one bit each in words of 32 with the pair-table rank of the word's first.
constexpr int MARK_WORDS = (NU + 31) / 32, MARKS = 32 * MARK_WORDS;

constexpr int KIND_SITE = 1 << 30;  // build-time entry flag: lattice site (gid = e*729+u)

// Replica lookup.  A single system uses OneRep (its descriptor is a kernel
// argument); a batch uses ManyRep (descriptor table plus per-site, per-element
// and per-cell replica indices).  The kernels are written once for both.
struct OneRep {
  Rep r;
  static constexpr bool many = false;
  __device__ __forceinline__ Rep site(int) const { return r; }
  __device__ __forceinline__ Rep elem(int) const { return r; }
  __device__ __forceinline__ Rep acell(int) const { return r; }
  __device__ __forceinline__ int elem_id(int) const { return 0; }
};
struct ManyRep {
  const Rep *reps;
  const int *site_rep, *elem_rep, *acell_rep;
  static constexpr bool many = true;
  __device__ __forceinline__ Rep site(int i) const { return reps[site_rep[i]]; }
  __device__ __forceinline__ Rep elem(int e) const { return reps[elem_rep[e]]; }
  __device__ __forceinline__ Rep acell(int c) const { return reps[acell_rep[c]]; }
  __device__ __forceinline__ int elem_id(int e) const { return elem_rep[e]; }
};

// ------------------------------------------------------------------ pbc

__device__ __forceinline__ int grid_cell(const Grid &g, const BoxD &b, const double *w) {
  int c[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    int v = (int)((w[d] - b.lo[d]) * g.inv[d]);
    c[d] = min(max(v, 0), g.nc[d] - 1);
  }
  return (c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0];
}

__device__ __forceinline__ void wrap_cell(int v, int nc, int &cell, int &W) {
  W = 0;
  while (v < 0) {
    v += nc;
    W--;
  }
  while (v >= nc) {
    v -= nc;
    W++;
  }
  cell = v;
}

// What a rebuild starts from, cleared by its first kernel.
struct BuildStart {
  double4 *xbuild;      // the wrapped positions the lists are built from (null: only wrap)
  float *disp;
  int *inner_ok;        // [nrep]
  int inner;            // the prefix is usable (its margin is not zero)
  unsigned *dmax;       // [nrep]
  int *overflow, *nact, *nwork, *sm_counter;
  int nrep, nsm;
  int *key, *place, *count;   // per atom: its cell and its place among the cell's arrivals; atoms per cell
};

// Domain::pbc for owned atoms (domain.cpp:562-630), and the clearing of the
// rebuild's flags and counters (one launch instead of a dozen small ones,
// which a small system would wait for one by one).
template <class RP>
__global__ void k_pbc_atoms(double4 *xs, int na, RP P, BuildStart S) {
  behind_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (S.xbuild) {
    if (i < S.nrep) {
      S.inner_ok[i] = S.inner;
      S.dmax[i] = 0u;
    }
    if (i < S.nsm) S.sm_counter[i] = 0;
    if (i < 4) S.overflow[i] = 0;
    if (i < 2) S.overflow[8 + i] = 0;
    if (i == 0) {
      *S.nact = 0;
      *S.nwork = 0;
    }
  }
  if (i >= na) return;
  const BoxD b = P.site(i).b;
  double4 p = xs[i];
  double *q = &p.x;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double x = q[d];
    if (x < b.lo[d]) x += b.L[d];
    if (x >= b.hi[d]) {
      x -= b.L[d];
      x = fmax(x, b.lo[d]);
    }
    q[d] = x;
  }
  xs[i] = p;
  if (S.xbuild) {
    S.xbuild[i] = p;
    S.disp[i] = 0.0f;
    const Rep r = P.site(i);
    const int c = r.abase + grid_cell(r.ag, r.b, q);
    S.key[i] = c;
    S.place[i] = atomicAdd(S.count + c, 1);
  }
}

// Element centre (ElementVecCAC::update_center_coord, element_vec_cac.cpp:3740-3765),
// Domain::pbc for elements (domain.cpp:645-720 with update_node_coord,
// element_vec_cac.cpp:3772-3785), then the geometry used by the candidate
// search: affine frame n0 + i a + j b + k c of the lattice sites, its inverse,
// the largest deviation of the trilinear nodes from that frame, and the
// centre-to-node radius.
//   eframe[e*EFR + 0..2]  n0
//   eframe[e*EFR + 3..11] rows of the inverse frame matrix
//   eframe[e*EFR + 12]    dmax
//   eframe[e*EFR + 13..21] frame vectors a, b, c (one lattice step each)
//   eframe[e*EFR + 22..24] norms of the inverse frame's rows (lattice steps
//                         per unit length along each index)
constexpr int EFR = 28;

template <class RP>
__global__ void k_elem_geom(double *nodex, int ne, RP P, double4 *ecenter, double *eframe,
                            unsigned long long *reach_bits, int *grew, double *nodex_build, float *edisp, int *key,
                            int *place, int *count) {
  behind_previous();
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  double reach = 0.0;
  if (e < ne) {
    const Rep rp = P.elem(e);
    const BoxD b = rp.b;
    double *nx = nodex + (size_t)e * 24;
    double c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double s = 0.0;
      for (int k = 0; k < NPE; k++) s = __dadd_rn(s, nx[3 * k + d]);
      c[d] = s / NPE / 1;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      bool moved = false;
      if (c[d] < b.lo[d]) {
        c[d] += b.L[d];
        moved = true;
      }
      if (c[d] >= b.hi[d]) {
        c[d] -= b.L[d];
        c[d] = fmax(c[d], b.lo[d]);
        moved = true;
      }
      if (moved) {
        double s = 0.0;
        for (int k = 0; k < NPE; k++) s = __dadd_rn(s, nx[3 * k + d]);
        double sh = c[d] - s / NPE / 1;
        for (int k = 0; k < NPE; k++) nx[3 * k + d] += sh;
      }
    }
    double R = 0.0;
    for (int k = 0; k < NPE; k++) {
      double dx = nx[3 * k] - c[0], dy = nx[3 * k + 1] - c[1], dz = nx[3 * k + 2] - c[2];
      R = fmax(R, sqrt(dx * dx + dy * dy + dz * dz));
    }
    double n0[3], A[3][3];  // columns a, b, c
#pragma unroll
    for (int d = 0; d < 3; d++) {
      n0[d] = nx[d];
      A[d][0] = (nx[3 * 1 + d] - n0[d]) / (NC - 1);
      A[d][1] = (nx[3 * 3 + d] - n0[d]) / (NC - 1);
      A[d][2] = (nx[3 * 4 + d] - n0[d]) / (NC - 1);
    }
    double dmax = 0.0;
    for (int k = 0; k < NPE; k++) {
      double dev2 = 0.0;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        double aff = n0[d] + (NC - 1) * (node_xi(k) * A[d][0] + node_eta(k) * A[d][1] +
                                         node_zeta(k) * A[d][2]);
        double t = nx[3 * k + d] - aff;
        dev2 += t * t;
      }
      dmax = fmax(dmax, sqrt(dev2));
    }
    // inverse of the 3x3 frame
    double det = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) -
                 A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
                 A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
    double id = 1.0 / det;
    double inv[3][3];
    inv[0][0] = (A[1][1] * A[2][2] - A[1][2] * A[2][1]) * id;
    inv[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * id;
    inv[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * id;
    inv[1][0] = (A[1][2] * A[2][0] - A[1][0] * A[2][2]) * id;
    inv[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * id;
    inv[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * id;
    inv[2][0] = (A[1][0] * A[2][1] - A[1][1] * A[2][0]) * id;
    inv[2][1] = (A[0][1] * A[2][0] - A[0][0] * A[2][1]) * id;
    inv[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * id;
    double *fr = eframe + (size_t)e * EFR;
    fr[0] = n0[0];
    fr[1] = n0[1];
    fr[2] = n0[2];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int q = 0; q < 3; q++) fr[3 + 3 * r + q] = inv[r][q];
#pragma unroll
    for (int r = 0; r < 3; r++)
      fr[22 + r] = sqrt(inv[r][0] * inv[r][0] + inv[r][1] * inv[r][1] + inv[r][2] * inv[r][2]);
    fr[12] = dmax;
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
      for (int d = 0; d < 3; d++) fr[13 + 3 * q + d] = A[d][q];
    ecenter[e] = make_double4(c[0], c[1], c[2], R);
    if (nodex_build) {   // the nodes the lists are built from
      for (int k = 0; k < 24; k++) nodex_build[(size_t)e * 24 + k] = nx[k];
      edisp[e] = 0.0f;
      const int k = rp.ebase + grid_cell(rp.eg, b, c);
      key[e] = k;
      place[e] = atomicAdd(count + k, 1);
    }
    reach = R + dmax;
    if (!(reach <= rp.reach_budget)) atomicExch(grew, 1);
    // per-replica maximum (non-negative doubles order like their bit patterns)
    if (RP::many) atomicMax(reach_bits + P.elem_id(e), (unsigned long long)__double_as_longlong(reach));
  }
  if (!RP::many) {
    for (int o = 16; o > 0; o >>= 1) reach = fmax(reach, __shfl_down_sync(0xffffffffu, reach, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reach_bits, (unsigned long long)__double_as_longlong(reach));
  }
}

// ---------------------------------------------------------------- binning

// Binning is a counting sort: the kernels above count the arrivals of each
// cell, a scan turns the counts into the cells' first places, each atom (and
// element) is put at its cell's first place plus its order of arrival, and
// there takes the place that its index has among the cell's members, so the
// order is that of a stable sort by cell whatever the order of arrival was.
// Few launches (a radix sort takes about a dozen for atoms and elements, which
// is what small systems waited for), and no keys to move.

// Exclusive scan of the atom cells' counts and of the element cells', each
// with its total behind (one block; larger grids use CUB).
constexpr int SCAN_CELLS = 16384;
__global__ void __launch_bounds__(1024) k_scan_cells(const int *count, int na_cell, int ne_cell, int *astart, int *estart) {
  behind_previous();
  __shared__ int warp_sum[32];
  __shared__ int carry, atoms;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = na_cell + ne_cell;
  if (threadIdx.x == 0) carry = 0;
  if (threadIdx.x == 0 && na_cell == 0) atoms = 0;
  for (int base = 0; base < n; base += 4096) {
    const int i0 = base + 4 * threadIdx.x;
    int v[4], sum = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      v[u] = i0 + u < n ? count[i0 + u] : 0;
      sum += v[u];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();   // the last round's warp_sum and carry have been read
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; w++) before += warp_sum[w];
    int at = before + incl - sum;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u;
      if (i < na_cell) astart[i] = at;
      else if (i < n) estart[i - na_cell] = at;
      at += v[u];
      if (i == na_cell - 1) atoms = at;
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + incl;
  }
  __syncthreads();
  // element places count from their own zero
  const int a = atoms;
  for (int i = threadIdx.x; i < ne_cell; i += 1024) estart[i] -= a;
  if (threadIdx.x == 0) {
    astart[na_cell] = a;
    estart[ne_cell] = carry - a;
  }
}

// near[c]: some cell of the 27-cell block around cell c (a single system's
// grid, periodic) holds an entry (element grid: an element; atom grid: an
// atom)
__device__ __forceinline__ void near_cell(int c, const int *start, const Grid &g, unsigned char *near) {
  const int cx = c % g.nc[0], cy = (c / g.nc[0]) % g.nc[1], cz = c / (g.nc[0] * g.nc[1]);
  bool any = false;
  for (int oz = -1; oz <= 1 && !any; oz++)
    for (int oy = -1; oy <= 1 && !any; oy++)
      for (int ox = -1; ox <= 1 && !any; ox++) {
        const int x = (cx + ox + g.nc[0]) % g.nc[0], y = (cy + oy + g.nc[1]) % g.nc[1],
                  z = (cz + oz + g.nc[2]) % g.nc[2];
        const int k = (z * g.nc[1] + y) * g.nc[0] + x;
        any = start[k + 1] > start[k];
      }
  near[c] = any ? 1 : 0;
}

struct BinArgs {
  const int *akey, *aplace, *astart, *ekey, *eplace, *estart;
  int *aorder, *eorder;             // members of each cell in order of arrival
  int na, ne;
  unsigned char *anear, *enear;     // single systems with elements (else null)
  Grid ag, eg;
  float reach;                      // cutneigh
  int *bad_image;                   // flag (null while half lists are built)
};

// Atoms and elements to their cells; the cells' near flags.
__global__ void k_scatter(BinArgs B) {
  behind_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.na) {
    B.aorder[B.astart[B.akey[i]] + B.aplace[i]] = i;
    return;
  }
  i -= B.na;
  if (i < B.ne) {
    B.eorder[B.estart[B.ekey[i]] + B.eplace[i]] = i;
    return;
  }
  i -= B.ne;
  if (!B.enear) return;
  if (i < B.eg.ncell) {
    near_cell(i, B.estart, B.eg, B.enear);
    return;
  }
  i -= B.eg.ncell;
  if (i < B.ag.ncell) near_cell(i, B.astart, B.ag, B.anear);
}

// The place of member i of a cell: its first place plus the members of
// smaller index.
__device__ __forceinline__ int cell_place(const int *start, const int *order, int cell, int i) {
  const int beg = start[cell], end = start[cell + 1];
  int r = 0;
  for (int k = beg; k < end; k++) r += order[k] < i;
  return beg + r;
}

// Fixed-point copy of a wrapped atom position for the screen of the atom build: quanta of
// 2^-20 A from the box corner, modulo 2^32 (4096 A).  The differences of
// positions less than 2048 A apart are exact integers whatever the size of the
// box; the build takes no positions together that could be further apart
// (PART_SPAN; WIDE_CELL where the cells themselves are that large).  An atom
// further than WIDE_CELL (or a box length) outside the box gets FAR_ATOM and is
// nobody's neighbour (but see refuse_far_images).
constexpr int FAR_ATOM = 0x80000000;
// A chunk's atoms are taken together over at most PART_SPAN A of their row of
// cells.  With the cells to either side, each up to WIDE_CELL A wide, a
// position lies within 1000 + 3 x 256 A of the part's first cell and of every
// other one of the part: well inside 2048.
constexpr double PART_SPAN = 1000.0, WIDE_CELL = 256.0;
constexpr float QUANTUM = 1.0f / 1048576.0f;
__device__ __forceinline__ int fix20(double x) { return (int)(unsigned)(unsigned long long)__double2ll_rn(x * 1048576.0); }

// What the element walk reads of an element, in FP32: its centre from the box
// corner with the reach of its sites (radius + deviation from affine); the rows
// of its inverse frame (position from the centre -> lattice indices) with the
// centre's own indices; and the rows' norms with the deviation from affine.
// Rounding is at most a few 2^-24 of the box, which the walk allows for
// (it only has to find every site; the sites are tested for themselves).
struct ElemBox {
  float4 centre, row[3], norm;
};

// An atom that is outside the box after the wrap (positions given boxes away,
// or a run that has blown up): is another one within reach under an image that
// no list entry can hold?  Then the build is refused.  The screen of the atom
// build knows the images of atoms inside the box only.
template <class RP>
__device__ void refuse_far_images(const BinArgs &B, const RP &P, const double4 *xs, int i) {
  const Rep r = P.site(i);
  const double4 p = xs[i];
  const double px[3] = {p.x, p.y, p.z};
  int c = B.akey[i] - r.abase, at[3], t[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    at[d] = c % r.ag.nc[d];
    c /= r.ag.nc[d];
    t[d] = -(int)floor((px[d] - r.b.lo[d]) / r.b.L[d]);
  }
#pragma unroll 1
  for (int k = 0; k < 27; k++) {
    const int o[3] = {k % 3 - 1, k / 3 % 3 - 1, k / 9 - 1};
    int cell[3], W[3];
    float q[3];
    bool held = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      wrap_cell(at[d] + o[d], r.ag.nc[d], cell[d], W[d]);
      held = held && abs(W[d] - t[d]) <= 1;
    }
    if (held) continue;
    const int m = r.abase + (cell[2] * r.ag.nc[1] + cell[1]) * r.ag.nc[0] + cell[0];
#pragma unroll 1
    for (int u = B.astart[m]; u < B.astart[m + 1]; u++) {
      if (*(volatile int *)B.bad_image) return;
      const double4 x = xs[B.aorder[u]];
      q[0] = (float)(px[0] - (x.x + W[0] * r.b.L[0]));
      q[1] = (float)(px[1] - (x.y + W[1] * r.b.L[1]));
      q[2] = (float)(px[2] - (x.z + W[2] * r.b.L[2]));
      if (B.aorder[u] != i && q[0] * q[0] + q[1] * q[1] + q[2] * q[2] <= B.reach * B.reach) *B.bad_image = 1;
    }
  }
}

// The sorted atoms: positions (w = atom index), the fixed-point copies of the
// screen (x, y, z parts na apart), slots and cells; and the sorted elements
// with their boxes.
template <class RP>
__global__ void __launch_bounds__(256, RP::many ? 6 : 8)
    k_place(BinArgs B, RP P, const double4 *xs, double4 *out, int *fixed, int *slot_atom, int *atom_slot, int *slot_cell,
            const double4 *ecenter, const double *eframe, int *elems, ElemBox *boxes) {
  behind_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B.na) {
    const int cell = B.akey[i], k = cell_place(B.astart, B.aorder, cell, i);
    slot_atom[k] = i;
    atom_slot[i] = k;
    slot_cell[k] = cell;
    double4 p = xs[i];
    const BoxD b = P.site(i).b;
    const double q[3] = {p.x, p.y, p.z};
    int f[3];
    bool near = true, in = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      in = in && q[d] >= b.lo[d] && q[d] < b.hi[d];
      const double m = fmin(b.L[d], WIDE_CELL);
      near = near && q[d] >= b.lo[d] - m && q[d] <= b.hi[d] + m;
      f[d] = fix20(q[d] - b.lo[d]);
    }
    if (f[0] == FAR_ATOM) f[0]++;
    fixed[k] = near ? f[0] : FAR_ATOM;
    fixed[k + (size_t)B.na] = f[1];
    fixed[k + 2 * (size_t)B.na] = f[2];
    p.w = __longlong_as_double((long long)i);
    out[k] = p;
    if (!in && B.bad_image) refuse_far_images(B, P, xs, i);
    return;
  }
  i -= B.na;
  if (i >= B.ne) return;
  const int k = cell_place(B.estart, B.eorder, B.ekey[i], i);
  elems[k] = i;
  const double4 c = ecenter[i];
  const double *fr = eframe + (size_t)i * EFR;
  const BoxD b = P.elem(i).b;
  ElemBox &o = boxes[k];
  o.centre = make_float4((float)(c.x - b.lo[0]), (float)(c.y - b.lo[1]), (float)(c.z - b.lo[2]),
                         __double2float_ru(c.w + fr[12]));
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const double a0 = fr[3 + 3 * r], a1 = fr[4 + 3 * r], a2 = fr[5 + 3 * r];
    o.row[r] = make_float4((float)a0, (float)a1, (float)a2,
                           (float)(a0 * (c.x - fr[0]) + a1 * (c.y - fr[1]) + a2 * (c.z - fr[2])));
  }
  o.norm = make_float4(__double2float_ru(fr[22]), __double2float_ru(fr[23]), __double2float_ru(fr[24]),
                       __double2float_ru(fr[12]));
}

// -------------------------------------------------------------- the build

struct BuildArgs {
  const double4 *xs;          // atom positions (first na entries)
  const double *nodex;
  const double4 *ecenter;
  const double *eframe;
  const int *acell_start;
  const double4 *acell_pos;
  const int *acell_x, *acell_y, *acell_z;   // wrapped positions in fixed point (fix20)
  const int *acell_of;        // [na] cell of each sorted atom (list slot)
  const int *ecell_start;
  const unsigned char *ecell_near;   // single systems: element cell has an element in its 27-cell block (else null)
  const unsigned char *acell_near;   // single systems: atom cell has an atom in its 27-cell block (else null)
  const int *ecell_elems;
  const ElemBox *ecell_box;      // the sorted elements, as the element walk reads them
  const int *atom_of_slot;    // list slot (cell-sorted position) -> atom index
  unsigned char *site_flag;   // [ne * MARKS] marks the lattice sites some full list references
  int na, ne, nsi, cap;
  RefBins rb;                 // single systems only (half lists)
  double cutneigh, cutneighsq;
  double cutforcesq;          // pairs inside the inner radius (force cutoff + margin) at build time go first
  int want_half;
  int wide;                   // cells wider than WIDE_CELL: no fixed-point screen of atoms
  int *nbr_full;              // final full-list entries (atoms; element sites after k_remap_sites)
  int *num_in;                // per slot: entries in the front segment
  int2 *site_from;            // per slot: front / back rows before the element-site entries
  int *num_full;
  int *raw_sites;             // element-site entries before conversion (k_remap_sites), `cap` per query
  int *raw_half, *num_half;
  unsigned char *img_half;
  int *overflow;              // [0] flag, [1] max count, [2] bad image
};

__device__ __forceinline__ int ref_bin1(const RefBins &rb, int d, double x) {
  int ix;
  if (x >= rb.hi[d]) ix = (int)((x - rb.hi[d]) * rb.inv[d]) + rb.nbin[d];
  else if (x >= rb.lo[d]) {
    ix = (int)((x - rb.lo[d]) * rb.inv[d]);
    ix = min(ix, rb.nbin[d] - 1);
  } else ix = (int)((x - rb.lo[d]) * rb.inv[d]) - 1;
  return ix;
}

// >0: q's reference bin is in p's upper half stencil; 0: same bin; <0 otherwise
__device__ __forceinline__ int ref_bin_order(const RefBins &rb, const double *p, const double *q) {
#pragma unroll
  for (int d = 2; d >= 0; d--) {
    int a = ref_bin1(rb, d, p[d]), c = ref_bin1(rb, d, q[d]);
    if (c != a) return c > a ? 1 : -1;
  }
  return 0;
}

__device__ __forceinline__ bool above_right(const double *q, const double *p) {
  if (q[2] < p[2]) return false;
  if (q[2] == p[2]) {
    if (q[1] < p[1]) return false;
    if (q[1] == p[1] && q[0] < p[0]) return false;
  }
  return true;
}

__device__ __forceinline__ double rsq_rn(double dx, double dy, double dz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Stores one entry; the image byte carries IN_CUT when the pair lies inside
// the force cutoff at build time (the compaction puts those entries first).
constexpr unsigned char IN_CUT = 0x80;
__device__ __forceinline__ void emit(const BuildArgs &A, int i, int &n, int *raw, unsigned char *img,
                                     int val, int code) {
  if (n < A.cap) {
    raw[(size_t)n * A.nsi + i] = val;
    img[(size_t)n * A.nsi + i] = (unsigned char)code;
  }
  n++;
}

// One query point (an i-site) of the build.
struct Query {
  Rep r;          // its replica
  int i;          // site-table index (atoms: input order)
  int slot;       // list slot: atoms in cell-sorted order, then Gauss points
  bool iatom;
  int ie, ig, iu;
  double xi[3];   // raw position
  double wi[3];   // wrapped into the box: wi = xi + ti L
  int ti[3];
};

template <class RP>
__device__ __forceinline__ void make_query(const BuildArgs &A, const RP &P, int i, Query &q) {
  q.r = P.site(i);
  q.i = i;
  q.slot = i;
  q.iatom = i < A.na;
  q.ie = q.ig = q.iu = -1;
  if (q.iatom) {
    double4 p = A.xs[i];
    q.xi[0] = p.x;
    q.xi[1] = p.y;
    q.xi[2] = p.z;
  } else {
    q.ie = (i - A.na) / NG;
    q.ig = (i - A.na) % NG;
    q.iu = gauss_site(q.ig);
    const double *nx = A.nodex + (size_t)q.ie * 24 + 3 * gauss_node(q.ig);
    q.xi[0] = nx[0];
    q.xi[1] = nx[1];
    q.xi[2] = nx[2];
  }
  const BoxD &b = q.r.b;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double f = floor((q.xi[d] - b.lo[d]) / b.L[d]);
    q.ti[d] = -(int)f;
    q.wi[d] = q.xi[d] - f * b.L[d];
    if (q.wi[d] >= b.hi[d]) {
      q.wi[d] -= b.L[d];
      q.ti[d] -= 1;
    }
    if (q.wi[d] < b.lo[d]) {
      q.wi[d] += b.L[d];
      q.ti[d] += 1;
    }
  }
}

// A candidate atom j seen in a cell with wrap count W: exact test and storage
// rules (atoms are inside the box after pbc, so their own wrap is zero).
// Full-list entries go to `full(j, code)`; half-list entries are stored here.
template <class FullSink>
__device__ __forceinline__ void try_atom(const BuildArgs &A, const Query &q, int j, const int W[3], int &nh,
                                         FullSink &&full) {
  int s[3] = {W[0] - q.ti[0], W[1] - q.ti[1], W[2] - q.ti[2]};
  bool zero = (s[0] == 0 && s[1] == 0 && s[2] == 0);
  if (q.iatom && j == q.i && zero) return;
  double4 xj = A.xs[j];
  double qq[3] = {xj.x, xj.y, xj.z};
  if (!zero) {
    qq[0] = s[0] ? __dadd_rn(qq[0], s[0] * q.r.b.L[0]) : qq[0];
    qq[1] = s[1] ? __dadd_rn(qq[1], s[1] * q.r.b.L[1]) : qq[1];
    qq[2] = s[2] ? __dadd_rn(qq[2], s[2] * q.r.b.L[2]) : qq[2];
  }
  double rsq = rsq_rn(__dsub_rn(q.xi[0], qq[0]), __dsub_rn(q.xi[1], qq[1]), __dsub_rn(q.xi[2], qq[2]));
  if (!(rsq <= A.cutneighsq)) return;
  // a neighbour beyond the first periodic image cannot be stored (the box is
  // shorter than twice the cutoff)
  if (s[0] < -1 || s[0] > 1 || s[1] < -1 || s[1] > 1 || s[2] < -1 || s[2] > 1) {
    atomicExch(&A.overflow[2], 1);
    return;
  }
  int code = img_code(s[0], s[1], s[2]) | (rsq < A.cutforcesq ? IN_CUT : 0);
  full(j, code);
  if (A.want_half && q.iatom) {
    int ord = ref_bin_order(A.rb, q.xi, qq);
    bool keep = ord > 0 || (ord == 0 && (zero ? (j > q.i) : above_right(qq, q.xi)));
    if (keep) emit(A, q.slot, nh, A.raw_half, A.img_half, j, code);
  }
}

// Element lattice sites are found in two phases.  Phase A (one thread per
// query) walks the element cells around the query and, for every element
// whose site box in lattice-index space is not empty, writes a work item:
// the element, the periodic image and the box.  Phase B (one warp per query)
// tests the sites of each item with the lanes splitting the box, emitting in
// box order, so the list is the one a serial walk would write.

// work item: x = element | (image + 4 per dimension, 3 bits each) << 21,
// y = box lo/hi in lattice indices (4 bits each)
__device__ __forceinline__ int2 pack_item(int e, const int s[3], const int lo[3], const int hi[3]) {
  int x = e | ((s[0] + 4) << 21) | ((s[1] + 4) << 24) | ((s[2] + 4) << 27);
  int y = lo[0] | (lo[1] << 4) | (lo[2] << 8) | (hi[0] << 12) | (hi[1] << 16) | (hi[2] << 20);
  return make_int2(x, y);
}
__device__ __forceinline__ void unpack_item(int2 it, int &e, int s[3], int lo[3], int hi[3]) {
  e = it.x & ((1 << 21) - 1);
  s[0] = ((it.x >> 21) & 7) - 4;
  s[1] = ((it.x >> 24) & 7) - 4;
  s[2] = ((it.x >> 27) & 7) - 4;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    lo[d] = (it.y >> (4 * d)) & 15;
    hi[d] = (it.y >> (12 + 4 * d)) & 15;
  }
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Phase A for the Q queries of a warp (32 / Q lanes each, all with the query):
// those of one replica within two cells of one another are taken together.
// The lanes walk the cells around all of them, 32 at a time, and keep the
// elements that can reach the queries' bounding box (the candidate sphere, then
// the lattice-index box); each query tests the few that are left.  A query's
// items are those of the 27 cells around it in the order of the cells (x
// fastest) and of the elements in each, whatever queries it shares the walk
// with.  Returns the number of items of the lane's query; at most cap are stored.
// All in FP32 from the box corner, with the roundings allowed for: an item too
// many costs a few site tests and changes no list.
constexpr int NEAR = 64;
struct NearStage {
  float4 centre[NEAR];    // of the image in the box the queries are wrapped into; w: reach of the sites
  int kk[NEAR];           // place among the sorted elements
  int w[NEAR];            // the cell's image + 1 per dimension, 2 bits each
  int2 item[8][32];       // accepted items until their places are known (Q = 8)
};
template <int Q>
__device__ int element_items(const BuildArgs &A, const Query &q, int rep, bool live, int2 *out, int cap,
                             NearStage &st) {
  constexpr int S = 32 / Q;
  static_assert(Q == 32 || Q == 8, "st.item's rows");
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const Grid &eg = q.r.eg;
  float lo[3], hi[3];
  int ci[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double r = fmax(q.wi[d] - q.r.b.lo[d], 0.0);
    lo[d] = __double2float_rd(r);
    hi[d] = __double2float_ru(r);
    ci[d] = min(max((int)((q.wi[d] - q.r.b.lo[d]) * eg.inv[d]), 0), eg.nc[d] - 1);
  }
  // no element in the 27 cells around: nothing to walk
  if (A.ecell_near && !A.ecell_near[q.r.ebase + (ci[2] * eg.nc[1] + ci[1]) * eg.nc[0] + ci[0]]) live = false;
  int n = 0;
  for (unsigned todo = __ballot_sync(full, live); todo;) {
    const int lead = __ffs(todo) - 1;
    const int lead_rep = __shfl_sync(full, rep, lead);
    bool in = ((todo >> lane) & 1u) && rep == lead_rep;
    int c0[3], nc[3], nr[3], ebase = __shfl_sync(full, q.r.ebase, lead);
    float blo[3], bhi[3], L[3];   // positions from the box corner
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float far = fabsf(lo[d] - __shfl_sync(full, lo[d], lead)) * (float)eg.inv[d];
      in = in && far <= 2.0f;
    }
    in = in || lane / S == lead / S;
    todo &= ~__ballot_sync(full, in);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      blo[d] = __int_as_float(__reduce_min_sync(full, in ? __float_as_int(lo[d]) : 0x7fffffff));
      bhi[d] = __int_as_float(__reduce_max_sync(full, in ? __float_as_int(hi[d]) : 0));
      c0[d] = __reduce_min_sync(full, in ? ci[d] : 0x7fffffff) - 1;
      nr[d] = __reduce_max_sync(full, in ? ci[d] : 0) + 2 - c0[d];
      nc[d] = __shfl_sync(full, eg.nc[d], lead);
      L[d] = __shfl_sync(full, (float)q.r.b.L[d], lead);
    }
    // roundings of the positions (each at most 2^-23 of the box)
    const float slack = 1e-6f * (L[0] + L[1] + L[2]) + 1e-4f;
    int m = 0;
    auto flush = [&] {
      __syncwarp();
      for (int b = 0; b < m; b += 32) {
        const int mm = min(32, m - b);
        unsigned acc = 0;
        for (int j = lane % S; j < mm; j += S) {
          const float4 ce = st.centre[b + j];
          const float dx = lo[0] - ce.x, dy = lo[1] - ce.y, dz = lo[2] - ce.z, R = ce.w + (float)A.cutneigh + slack;
          if (in && dx * dx + dy * dy + dz * dz <= R * R) acc |= 1u << j;
        }
        unsigned ok = 0;
        for (; acc; acc &= acc - 1) {
          // the box of the sites whose affine position can lie within cutneigh +
          // the element's deviation from affine
          const int j = __ffs(acc) - 1, w = st.w[b + j], kk = st.kk[b + j];
          const float4 ce = st.centre[b + j], norm = A.ecell_box[kk].norm;
          const float dx = lo[0] - ce.x, dy = lo[1] - ce.y, dz = lo[2] - ce.z;
          const float n3[3] = {norm.x, norm.y, norm.z}, far = (float)A.cutneigh + norm.w + slack;
          int blo3[3], bhi3[3];
          bool some = true;
#pragma unroll
          for (int r = 0; r < 3; r++) {
            const float4 row = A.ecell_box[kk].row[r];
            const float idx = row.x * dx + row.y * dy + row.z * dz + row.w, rho = far * n3[r] + 1e-4f;
            blo3[r] = max(0, (int)ceilf(idx - rho));
            bhi3[r] = min(NC - 1, (int)floorf(idx + rho));
            some = some && blo3[r] <= bhi3[r];
          }
          const int s[3] = {(w & 3) - 1 - q.ti[0], ((w >> 2) & 3) - 1 - q.ti[1], (w >> 4) - 1 - q.ti[2]};
          // a box shorter than the candidate sphere's diameter shows an element
          // under two images; images beyond +-2 cannot be encoded (and are far
          // beyond any cutoff in such a box)
          if (some && (s[0] < -3 || s[0] > 3 || s[1] < -3 || s[1] > 3 || s[2] < -3 || s[2] > 3)) {
            atomicExch(&A.overflow[2], 1);
            some = false;
          }
          if (some) {
            const int2 item = pack_item(A.ecell_elems[kk], s, blo3, bhi3);
            if (S > 1) {
              st.item[lane / S][j] = item;
              ok |= 1u << j;
            } else {
              if (n < cap) out[n] = item;
              n++;
            }
          }
        }
        if (S > 1) {
          unsigned all = ok;
          __syncwarp();
#pragma unroll
          for (int o = 1; o < S; o <<= 1) all |= __shfl_xor_sync(full, all, o);
          for (; ok; ok &= ok - 1) {
            const int j = __ffs(ok) - 1, at = n + __popc(all & ((1u << j) - 1u));
            if (at < cap) out[at] = st.item[lane / S][j];
          }
          n += __popc(all);
        }
      }
      m = 0;
      __syncwarp();
    };
    // elements of a cell this far from the bounding box are out of reach
    const float reach = __shfl_sync(full, (float)q.r.reach_budget, lead) + (float)A.cutneigh + 0.01f + slack;
    float size[3];
#pragma unroll
    for (int d = 0; d < 3; d++) size[d] = L[d] / (float)nc[d];
    const int cells = nr[0] * nr[1] * nr[2];
    for (int b = 0; b < cells; b += 32) {
      const int c = b + lane;
      int end = 0, incl = 0, w = 0;
      if (c < cells) {
        const int y = c / nr[0], z = y / nr[1];
        const int o[3] = {c0[0] + c - y * nr[0], c0[1] + y - z * nr[1], c0[2] + z};
        int cc[3], W[3];
        float d2 = 0.0f;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          wrap_cell(o[d], nc[d], cc[d], W[d]);
          const float g = fmaxf(0.0f, fmaxf((float)o[d] * size[d] - bhi[d], blo[d] - (float)(o[d] + 1) * size[d]));
          d2 += g * g;
        }
        if (d2 <= reach * reach) {
          const int cell = ebase + (cc[2] * nc[1] + cc[1]) * nc[0] + cc[0];
          w = (W[0] + 1) | (W[1] + 1) << 2 | (W[2] + 1) << 4;
          end = A.ecell_start[cell + 1];
          incl = end - A.ecell_start[cell];
        }
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(full, incl, 31);
      int k0 = 0;
      do {
        const int k = k0 + lane;
        int o = 0;   // the lane whose cell holds the k-th element
#pragma unroll
        for (int step = 16; step; step >>= 1)
          if (__shfl_sync(full, incl, o + step - 1) <= k) o += step;
        const int kk = __shfl_sync(full, end, o) - (__shfl_sync(full, incl, o) - k);
        const int ow = __shfl_sync(full, w, o);
        bool pass = false;
        float4 ce = make_float4(0, 0, 0, 0);
        if (k < total) {
          ce = A.ecell_box[kk].centre;
          ce.x += ((ow & 3) - 1) * L[0];
          ce.y += (((ow >> 2) & 3) - 1) * L[1];
          ce.z += ((ow >> 4) - 1) * L[2];
          const float R = ce.w + (float)A.cutneigh + slack;
          const float dx = fmaxf(0.0f, fmaxf(blo[0] - ce.x, ce.x - bhi[0]));
          const float dy = fmaxf(0.0f, fmaxf(blo[1] - ce.y, ce.y - bhi[1]));
          const float dz = fmaxf(0.0f, fmaxf(blo[2] - ce.z, ce.z - bhi[2]));
          pass = dx * dx + dy * dy + dz * dz <= R * R;
          if (pass) {
            // the same in the element's own directions: the lattice indices of
            // the bounding box' centre, and how far its sides carry them
            const float4 norm = A.ecell_box[kk].norm;
            const float n3[3] = {norm.x, norm.y, norm.z}, far = (float)A.cutneigh + norm.w + slack;
            const float x = 0.5f * (blo[0] + bhi[0]) - ce.x, y = 0.5f * (blo[1] + bhi[1]) - ce.y,
                        z = 0.5f * (blo[2] + bhi[2]) - ce.z;
            const float hx = 0.5f * (bhi[0] - blo[0]), hy = 0.5f * (bhi[1] - blo[1]), hz = 0.5f * (bhi[2] - blo[2]);
#pragma unroll
            for (int r = 0; r < 3; r++) {
              const float4 row = A.ecell_box[kk].row[r];
              const float idx = row.x * x + row.y * y + row.z * z + row.w;
              const float rho = far * n3[r] + 1e-4f + fabsf(row.x) * hx + fabsf(row.y) * hy + fabsf(row.z) * hz;
              if (idx + rho < 0.0f || idx - rho > NC - 1) pass = false;
            }
          }
        }
        const unsigned acc = __ballot_sync(full, pass);
        if (pass) {
          const int at = m + __popc(acc & lanemask_lt());
          st.centre[at] = ce;
          st.kk[at] = kk;
          st.w[at] = ow;
        }
        m += __popc(acc);
        k0 += 32;
        if (m > NEAR - 32 || (b + 32 >= cells && k0 >= total)) flush();
      } while (k0 < total);
    }
  }
  return n;
}

// Warp-wide emission: the lanes' accepted candidates are stored in lane
// order after the entries already written, so a warp walking candidates in
// chunks of 32 writes exactly the order of a serial walk.  Every lane keeps
// the same count n.
__device__ __forceinline__ void warp_emit(const BuildArgs &A, int slot, int &n, int *raw, unsigned char *img,
                                          bool pass, int val, int code) {
  const unsigned m = __ballot_sync(0xffffffffu, pass);
  if (pass) {
    const int at = n + __popc(m & lanemask_lt());
    if (at < A.cap) {
      raw[(size_t)at * A.nsi + slot] = val;
      img[(size_t)at * A.nsi + slot] = (unsigned char)code;
    }
  }
  n += __popc(m);
}

// The same for full lists: accepted entries go to the front segment (inside
// the inner radius) or the back segment, each in lane order.  Rows outside
// [0, cap) are not written (the count still grows and flags the overflow).
__device__ __forceinline__ void warp_emit_full(const BuildArgs &A, int slot, int &nin, int &nout, bool pass,
                                               bool incut, int val) {
  const unsigned mi = __ballot_sync(0xffffffffu, pass && incut);
  const unsigned mo = __ballot_sync(0xffffffffu, pass && !incut);
  if (pass) {
    const int row = incut ? nin + __popc(mi & lanemask_lt()) : A.cap - 1 - (nout + __popc(mo & lanemask_lt()));
    if (row >= 0 && row < A.cap) A.nbr_full[(size_t)row * A.nsi + slot] = val;
  }
  nin += __popc(mi);
  nout += __popc(mo);
}

// Phase B for one query: its items in groups of up to 16.  The warp stages each
// item in its shared scratch as the element's trilinear map of the lattice
// indices, relative to the query, in FP32: position = sum over subsets of (a,
// bb, cc) of coefficient x product, the coefficients formed in FP64 by
// differences of the nodes along each direction.  The coordinates are at most
// a few element radii long, so the FP32 distance decides all but the sites
// within about 1e-3 A of the cutoff; those take the reference's exact FP64
// distance.
// An item's box is loose (a sphere in skewed indices: about one site in
// fifteen is a neighbour), so the lanes first take its rows (a, bb), along
// which the position is linear in cc: the cc within reach solve a quadratic.
// The rows' sites go to a queue in (item, a, bb, cc) order -- the order of a
// serial walk -- and are tested and stored 32 at a time.
// An entry is left as (item << 10) | lattice site in the query's own row of
// raw_sites (front segment entries from its start, back ones from its end), so
// a warp's stores are consecutive; scattered into the transposed lists they
// took a memory sector each.  Bound by instruction issue (61 - 68 % of its
// slots).  Measured against every site of the box in FP64, node by node, per
// build: Gauss points of 20,000 elements (with their atoms) 479 -> 326 us, of
// 100,000 with 4.18 M atoms 2696 -> 1604 us, 180 elements 68 -> 38 us; atoms of
// 64 replicas of 1.44 M atoms 1832 -> 1592 us.
constexpr int ITEM_GROUP = 16;   // items staged at a time (a query has a few)
struct ItemStage {
  float4 map[ITEM_GROUP][3][2];   // per component: coefficients of 1, a, bb, a bb; cc, a cc, bb cc, a bb cc
  float lim[ITEM_GROUP][2];       // squares of cutneigh + margin, cutneigh - margin
  int mg[ITEM_GROUP];             // ceil(2^16 / n) of the box's y extent (division by multiply-shift)
  int2 item[ITEM_GROUP];          // the group's items
  int queue[31 + 32 * NC];        // sites to test: item << 12 | a << 8 | bb << 4 | cc
};

// The reference's distance test of lattice site u of element e under image s.
__device__ __forceinline__ bool site_exact(const BuildArgs &A, const Query &q, int e, const int s[3], int u,
                                           bool &inside) {
  const double *nx = A.nodex + (size_t)e * 24;
  double d[3] = {q.xi[0], q.xi[1], q.xi[2]};
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    const double N = shape_val(u, k);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double g = s[c] ? __dadd_rn(nx[3 * k + c], s[c] * q.r.b.L[c]) : nx[3 * k + c];
      d[c] = __dsub_rn(d[c], __dmul_rn(N, g));
    }
  }
  const double rsq = rsq_rn(d[0], d[1], d[2]);
  inside = rsq < A.cutforcesq;
  return rsq <= A.cutneighsq;
}

__device__ void items_warp(const BuildArgs &A, const Query &q, const int2 *items, int n, ItemStage &st, int *raw,
                           int &nin, int &nout, int &nh) {
  const int lane = threadIdx.x & 31;
  int rin = 0, rout = 0;   // element sites of each segment so far
  const float in2 = (float)A.cutforcesq;
  for (int g0 = 0; g0 < n; g0 += ITEM_GROUP) {
    const int ng = min(ITEM_GROUP, n - g0);
    __syncwarp();
    int nrows = 0;
    if (lane < ng) {
      const int2 it = items[g0 + lane];
      st.item[lane] = it;
      int e, sv[3], lo[3], hi[3];
      unpack_item(it, e, sv, lo, hi);
      const int n1s = hi[1] - lo[1] + 1;
      nrows = (hi[0] - lo[0] + 1) * n1s;
      st.mg[lane] = (65536 + n1s - 1) / n1s;
      // every coordinate and coefficient is shorter than four times the reach
      // below; 16 roundings of 2^-24 of that are 4e-6 of it, the margin five
      // times as much
      const float reach = (float)(A.cutneigh + 2.0 * (A.ecenter[e].w + A.eframe[(size_t)e * EFR + 12]));
      const float pre = (float)A.cutneigh + 2e-5f * reach, sure = (float)A.cutneigh - 2e-5f * reach;
      // In an element large against the cutoff that margin no longer covers the
      // rounding of the rows' discriminants (some 1e-6 reach^2 against 4e-5
      // cutneigh reach, in units of the squared step), nor, from 250 A on, the
      // prefix rule's allowance of 1e-3 A that of the segments (4e-6 reach):
      // there no row is cut short, and every site near enough is decided exactly.
      const bool long_rows = reach > 40.0f * (float)A.cutneigh;
      st.lim[lane][0] = long_rows ? 3e38f : pre * pre;
      st.lim[lane][1] = sure > 0.0f && !long_rows && reach <= 250.0f ? sure * sure : 0.0f;
    }
    __syncwarp();
    // the maps, four items at a time: lane 8 i + p takes the node at corner p =
    // xi + 2 eta + 4 zeta of item i, then each direction's far nodes become
    // steps from the near ones
    for (int m0 = 0; m0 < ng; m0 += 4) {
      const int m = min(m0 + (lane >> 3), ng - 1), p = lane & 7;
      int e, sv[3], lo[3], hi[3];
      unpack_item(st.item[m], e, sv, lo, hi);
      const double *nx = A.nodex + (size_t)e * 24 + 3 * corner_node(p & 1, (p >> 1) & 1, p >> 2);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        double v = nx[c] + sv[c] * q.r.b.L[c] - q.xi[c];
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1) {
          const double w = __shfl_xor_sync(0xffffffffu, v, bit);
          if (p & bit) v = (v - w) * (1.0 / (NC - 1));
        }
        reinterpret_cast<float *>(st.map[m])[8 * c + p] = (float)v;   // (lanes past the last item repeat it)
      }
    }
    __syncwarp();
    // a row's position at cc = 0 and its step along cc
    auto row_map = [&](int m, int a, int bb, float low[3], float up[3]) {
      const float fa = (float)a, fb = (float)bb;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float4 p = st.map[m][c][0], r = st.map[m][c][1];
        low[c] = __fmaf_rn(__fmaf_rn(p.w, fa, p.z), fb, __fmaf_rn(p.y, fa, p.x));
        up[c] = __fmaf_rn(__fmaf_rn(r.w, fa, r.z), fb, __fmaf_rn(r.y, fa, r.x));
      }
    };
    // test and store one queued site per lane
    auto test = [&](bool active, int site) {
      bool full = false, inside = false, half = false;
      const int m = site >> 12, a = (site >> 8) & 15, bb = (site >> 4) & 15, cc = site & 15;
      const int u = (a * NC + bb) * NC + cc;
      int e = 0, code = 0;
      if (active) {
        float low[3], up[3];
        row_map(m, a, bb, low, up);
        const float fc = (float)cc;
        const float dx = __fmaf_rn(up[0], fc, low[0]), dy = __fmaf_rn(up[1], fc, low[1]), dz = __fmaf_rn(up[2], fc, low[2]);
        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        const int2 it = st.item[m];
        e = it.x & ((1 << 21) - 1);
        full = r2 <= st.lim[m][0];
        // not the query's own site (same element, zero image)
        if (full && !q.iatom && u == q.iu) full = !(e == q.ie && (it.x >> 21) == ((4 << 6) | (4 << 3) | 4));
        if (full) {
          const int sv[3] = {((it.x >> 21) & 7) - 4, ((it.x >> 24) & 7) - 4, ((it.x >> 27) & 7) - 4};
          inside = r2 < in2;
          if (!(r2 < st.lim[m][1])) full = site_exact(A, q, e, sv, u, inside);
          if (full && (sv[0] < -1 || sv[0] > 1 || sv[1] < -1 || sv[1] > 1 || sv[2] < -1 || sv[2] > 1)) {
            atomicExch(&A.overflow[2], 1);
            full = false;
          }
          if (full) {
            code = img_code(sv[0], sv[1], sv[2]);
            const int jg = site_gauss(u);
            if (jg < 0) A.site_flag[(size_t)e * MARKS + u] = 1;   // to be interpolated
            half = true;
            if (A.want_half && !q.iatom && jg >= 0) {
              if (code == IMG_ZERO) {
                half = (q.ie < e) || (q.ie == e && q.ig < jg);
              } else {
                const double4 ce = A.ecenter[e], ci = A.ecenter[q.ie];
                const double sL[3] = {sv[0] * q.r.b.L[0], sv[1] * q.r.b.L[1], sv[2] * q.r.b.L[2]};
                double qcen[3] = {sv[0] ? __dadd_rn(ce.x, sL[0]) : ce.x, sv[1] ? __dadd_rn(ce.y, sL[1]) : ce.y,
                                  sv[2] ? __dadd_rn(ce.z, sL[2]) : ce.z};
                double icen[3] = {ci.x, ci.y, ci.z};
                half = above_right(qcen, icen);
              }
            }
          }
        }
      }
      // the warp's entries of each segment, in lane order
      const unsigned mi = __ballot_sync(0xffffffffu, full && inside), mo = __ballot_sync(0xffffffffu, full && !inside);
      if (full) {
        const int k = inside ? rin + __popc(mi & lanemask_lt()) : A.cap - 1 - (rout + __popc(mo & lanemask_lt()));
        if (k >= 0 && k < A.cap) raw[k] = ((g0 + m) << 10) | u;
      }
      rin += __popc(mi);
      rout += __popc(mo);
      if (A.want_half)
        warp_emit(A, q.slot, nh, A.raw_half, A.img_half, half, KIND_SITE | (e * NU + u), code);
    };
    // exclusive prefix of the items' row counts
    int incl = nrows;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int excl = incl - nrows;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int qn = 0;   // queued sites (warp-uniform)
    for (int base = 0; base < total; base += 32) {
      const int f = base + lane;
      // item of flattened row f: the last lane m < ng with excl[m] <= f
      int m = 0;
#pragma unroll
      for (int step = ITEM_GROUP / 2; step > 0; step >>= 1) {
        const int cand = m + step;
        const int v = __shfl_sync(0xffffffffu, excl, cand & 31);
        if (cand < ng && v <= f) m = cand;
      }
      const int t = f - __shfl_sync(0xffffffffu, excl, m);
      int c0 = 0, cnt = 0, place = 0;
      if (f < total) {
        const int y = st.item[m].y;
        const int lo1 = (y >> 4) & 15, lo2 = (y >> 8) & 15, hi2 = (y >> 20) & 15, n1 = ((y >> 16) & 15) - lo1 + 1;
        // (a, bb) of the t-th row of the box; the multiply-shift quotient is
        // exact for t < 81 and extents <= 9
        const int qa = (t * st.mg[m]) >> 16, a = (y & 15) + qa, bb = lo1 + t - qa * n1;
        float low[3], up[3];
        row_map(m, a, bb, low, up);
        // |low + cc up|^2 <= lim: the exact neighbours lie well inside (lim
        // holds the margin, or is without bound), so rounding here loses none
        const float A2 = up[0] * up[0] + up[1] * up[1] + up[2] * up[2];
        const float B = low[0] * up[0] + low[1] * up[1] + low[2] * up[2];
        const float C = low[0] * low[0] + low[1] * low[1] + low[2] * low[2] - st.lim[m][0];
        int c1 = hi2;
        c0 = lo2;
        if (A2 > 1e-6f) {
          const float disc = B * B - A2 * C, inv = 1.0f / A2;
          if (disc >= 0.0f) {
            const float w = sqrtf(disc) * inv, mid = -B * inv;
            c0 = max(c0, (int)ceilf(fmaxf(mid - w - 1e-2f, -1.0f)));
            c1 = min(c1, (int)floorf(fminf(mid + w + 1e-2f, 16.0f)));
          } else if (disc < 0.0f) {
            c1 = -1;
          }
        }
        cnt = max(c1 - c0 + 1, 0);
        place = (m << 12) | (a << 8) | (bb << 4);
      }
      int at = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
      }
      const int add = __shfl_sync(0xffffffffu, at, 31);
      at += qn - cnt;
      for (int k = 0; k < cnt; k++) st.queue[at + k] = place | (c0 + k);
      qn += add;
      __syncwarp();
      int done = 0;
      for (; qn - done >= 32; done += 32) test(true, st.queue[done + lane]);
      if (done) {
        // the rest to the front
        const int rest = lane < qn - done ? st.queue[done + lane] : 0;
        __syncwarp();
        if (lane < qn - done) st.queue[lane] = rest;
        qn -= done;
        __syncwarp();
      }
    }
    if (qn > 0) test(lane < qn, lane < qn ? st.queue[lane] : 0);
  }
  nin += rin;
  nout += rout;
}

// An atom candidate j of a Gauss point seen in a cell with wrap count W:
// the exact distance test; code gets the image and the in-cutoff mark
// (Gauss points keep no atoms in half lists).
__device__ __forceinline__ bool gauss_atom_test(const BuildArgs &A, const Query &q, int j, const int W[3],
                                                int &code) {
  int s[3] = {W[0] - q.ti[0], W[1] - q.ti[1], W[2] - q.ti[2]};
  double4 xj = A.xs[j];
  double qq[3] = {xj.x, xj.y, xj.z};
  qq[0] = s[0] ? __dadd_rn(qq[0], s[0] * q.r.b.L[0]) : qq[0];
  qq[1] = s[1] ? __dadd_rn(qq[1], s[1] * q.r.b.L[1]) : qq[1];
  qq[2] = s[2] ? __dadd_rn(qq[2], s[2] * q.r.b.L[2]) : qq[2];
  double rsq = rsq_rn(__dsub_rn(q.xi[0], qq[0]), __dsub_rn(q.xi[1], qq[1]), __dsub_rn(q.xi[2], qq[2]));
  if (!(rsq <= A.cutneighsq)) return false;
  if (s[0] < -1 || s[0] > 1 || s[1] < -1 || s[1] > 1 || s[2] < -1 || s[2] > 1) {
    atomicExch(&A.overflow[2], 1);
    return false;
  }
  code = img_code(s[0], s[1], s[2]) | (rsq < A.cutforcesq ? IN_CUT : 0);
  return true;
}

__device__ __forceinline__ void finish_counts(const BuildArgs &A, int i, int nin, int nout, int nh) {
  A.num_full[i] = nin + nout;
  A.num_in[i] = nin;
  if (A.want_half) A.num_half[i] = nh;
  int m = max(nin + nout, nh);
  if (m > A.cap) {
    atomicExch(&A.overflow[0], 1);
    atomicMax(&A.overflow[1], m);
  }
}

// Two FP32 values in one 64-bit register and the packed operations on them
// (sm_100: one instruction for two lanes' worth of arithmetic, each half
// rounded as the scalar operation rounds it).
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2_pack(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// mask << 2 with the sign bits of the halves of v below, the first half first
__device__ __forceinline__ unsigned f2_signs(unsigned mask, F2 v) {
  unsigned lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return __funnelshift_l(hi, __funnelshift_l(lo, mask, 1), 1);
}

// Atoms, atom neighbours: one block per chunk of 32 consecutive sorted atoms
// (list slots), the atoms as lanes.  Cells (>= cutneigh) are sorted x
// fastest, so a chunk lies in one row of cells, or in two at a row's end
// (then the warps take the two parts in turn); where atoms are so few that a
// chunk spans more than PART_SPAN of its row, in as many parts as that takes.
// For each of the 9 rows around the part's row the candidates are the cells from one left of the part's
// first cell to one right of its last, as at most three runs of consecutive
// cells under one image (the left and right wraps and the middle).  A lane
// meets the cells of its own 27-cell block in the order a walk of that block
// alone would take (ascending x in each row) and the others only beyond its
// reach, so its list is the same entry for entry.
//
// The kernel is bound by instruction issue, so the work is cut in three.
// Gather: the lanes take one candidate each, 32 consecutive ones of a run at a
// time, and keep those within reach of the box around the part's atoms (about
// 490 of 850): position relative to the part's first cell under the run's
// image, as floats, and list entry, in shared memory.  These coordinates are
// a few cells long, so FP32 decides all but the few candidates within 1e-4 A
// or so of the cutoff.
// Screen: over each word of 32 kept candidates every lane forms, without a
// branch, three bit masks (first candidate in the top bit): within cutneigh +
// margin, within cutneigh - margin, within the inner radius, from broadcast
// 128-bit loads and packed FP32 arithmetic, about 8 instructions a candidate.
// Bits between the first two masks take the exact FP64 test at once.  The
// masks replace the word's coordinates.
// Write-out: each lane pops its masks' bits in order, all lanes their n-th
// entry together: the lanes' list slots are consecutive, so each row of the
// (transposed) list is one coalesced store.
constexpr int SMALL_CHUNKS = 8;   // chunks per SM below which a chunk takes four warps
template <int NW, class RP>
__device__ __forceinline__ void build_atoms_chunk(const BuildArgs &A, const RP &P, const int chunk) {
  // words of kept candidates between two write-outs: 16 are usual; with four
  // warps, as many as the words of candidates taken at a time
  constexpr int MAXW = NW == 1 ? 20 : 32;
  __shared__ float4 kx4[MAXW][8], ky4[MAXW][8], kz4[MAXW][8];   // kept candidates' coordinates, then the masks
  __shared__ int entry[MAXW * 32];                              // (list slot << IMG_BITS) | image code
  __shared__ unsigned kept[NW > 1 ? MAXW : 1];
  __shared__ int self_at[32], back[32];
  unsigned *const m_acc = reinterpret_cast<unsigned *>(kx4), *const m_in = reinterpret_cast<unsigned *>(ky4);
  const int lane = threadIdx.x & 31, warp = NW > 1 ? (int)threadIdx.x >> 5 : 0;
  auto sync = [] {
    if (NW > 1) __syncthreads();
    else __syncwarp();
  };
  const int h = chunk * 32 + lane;
  const bool mine = h < A.na;
  const int key = mine ? A.acell_of[h] : -1;
  Query q;
  int3 qh = make_int3(FAR_ATOM, 0, 0);
  if (mine) {
    make_query(A, P, (int)__double_as_longlong(A.acell_pos[h].w), q);
    q.slot = h;
    qh = make_int3(A.acell_x[h], A.acell_y[h], A.acell_z[h]);
  } else {
    q.ti[0] = q.ti[1] = q.ti[2] = 0;
  }
  const bool unwrapped = (q.ti[0] | q.ti[1] | q.ti[2]) == 0;
  // the chunk's parts, one row of cells each, lowest lanes first
  unsigned todo = __ballot_sync(0xffffffffu, mine);
  while (todo) {
    const int lkey = __shfl_sync(0xffffffffu, key, __ffs(todo) - 1);
    const Rep R = P.acell(lkey);
    const int nc0 = R.ag.nc[0], nc1 = R.ag.nc[1], nc2 = R.ag.nc[2];
    const int row = (lkey - R.abase) / nc0;   // cz * nc1 + cy of the part
    const int hx = key - R.abase - row * nc0;
    // no further along the row than PART_SPAN from its first atom's cell
    const int hx0 = lkey - R.abase - row * nc0;
    const bool active = mine && ((todo >> lane) & 1u) && hx >= 0 && hx < nc0 && (hx - hx0) <= PART_SPAN * R.ag.inv[0];
    todo &= ~__ballot_sync(0xffffffffu, active);
    const int hy = row % nc1, hz = row / nc1;
    // unwrapped x range of the candidate cells
    const int xlo = __reduce_min_sync(0xffffffffu, active ? hx : 0x7fffffff) - 1;
    const int xhi = __reduce_max_sync(0xffffffffu, active ? hx : -1) + 1;
    // positions relative to the corner of the part's first cell
    const unsigned ox = fix20((xlo + 1) / R.ag.inv[0]), oy = fix20(hy / R.ag.inv[1]), oz = fix20(hz / R.ag.inv[2]);
    const unsigned Lx = fix20(R.b.L[0]), Ly = fix20(R.b.L[1]), Lz = fix20(R.b.L[2]);
    const bool near = active && qh.x != FAR_ATOM;
    const int ix = (int)(qh.x - ox), iy = (int)(qh.y - oy), iz = (int)(qh.z - oz);
    const float wx = near ? (float)ix * QUANTUM : 1e18f, wy = (float)iy * QUANTUM, wz = (float)iz * QUANTUM;
    const F2 wx2 = f2_pack(wx, wx), wy2 = f2_pack(wy, wy), wz2 = f2_pack(wz, wz);
    // the box around the part's atoms
    auto box_lo = [&](int v) { return (float)__reduce_min_sync(0xffffffffu, near ? v : 0x7fffffff) * QUANTUM; };
    auto box_hi = [&](int v) { return (float)__reduce_max_sync(0xffffffffu, near ? v : (int)0x80000000) * QUANTUM; };
    const float bx0 = box_lo(ix), by0 = box_lo(iy), bz0 = box_lo(iz), bx1 = box_hi(ix), by1 = box_hi(iy), bz1 = box_hi(iz);
    // FP32 screen: a separation carries at most 1.5 quanta of each component,
    // the rounding of two coordinates no longer than the part's span, and its
    // own: together under 6e-6 A + 3e-7 span; the margin is over six times that
    const float span = (float)((xhi - xlo + 1) / R.ag.inv[0] + 3.0 / R.ag.inv[1] + 3.0 / R.ag.inv[2]);
    const float margin = 1e-4f + 2e-6f * span;
    const float pre = (float)A.cutneigh + margin, sure = (float)A.cutneigh - margin;
    const float pre2 = __uint_as_float(__float_as_uint(pre * pre) + 1u);   // r2 <= pre^2 as r2 < pre2
    const float sure2 = sure > 0.0f ? sure * sure : 0.0f, in2 = (float)A.cutforcesq;
    const float reach2 = (pre + margin) * (pre + margin);
    const F2 lim_pre = f2_pack(pre2, pre2), lim_sure = f2_pack(sure2, sure2), lim_in = f2_pack(in2, in2);

    // the part's runs, one per lane (9 rows x 3): unwrapped x in [xlo, -1]
    // (the cell nc0 - 1 one image left), [0, nc0 - 1], [nc0, xhi] (the cell 0
    // one image right), each in words of 32 candidates
    int beg = 0, end = 0, rn = 0, rcode = 0;
    if (lane < 27) {
      const int run = lane % 3 - 1, ry = lane / 3;
      int cy, Wy, cz, Wz;
      wrap_cell(hz + ry / 3 - 1, nc2, cz, Wz);
      wrap_cell(hy + ry % 3 - 1, nc1, cy, Wy);
      const int u0 = run < 0 ? xlo : (run == 0 ? max(xlo, 0) : max(xlo, nc0));
      const int u1 = run < 0 ? min(xhi, -1) : (run == 0 ? min(xhi, nc0 - 1) : xhi);
      if (u0 <= u1) {
        const int rowbase = R.abase + (cz * nc1 + cy) * nc0 - run * nc0;
        beg = A.acell_start[rowbase + u0];
        end = A.acell_start[rowbase + u1 + 1];
        rn = (end - beg + 31) >> 5;
        rcode = img_code(run, Wy, Wz);
      }
    }
    int off = rn;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += v;
    }
    const int nraw = __shfl_sync(0xffffffffu, off, 31);
    // this lane's candidate of raw word r: list slot (-1 past the run's end) and image code
    auto candidate = [&](int r, int &code) {
      const int m = __popc(__ballot_sync(0xffffffffu, off <= r));   // the word's run
      const int first = __shfl_sync(0xffffffffu, beg, m) + 32 * (r - __shfl_sync(0xffffffffu, off - rn, m));
      code = __shfl_sync(0xffffffffu, rcode, m);
      const int k = first + lane;
      return k < __shfl_sync(0xffffffffu, end, m) ? k : -1;
    };
    auto fetch = [&](int k) {
      return k >= 0 ? make_int3(A.acell_x[k], A.acell_y[k], A.acell_z[k]) : make_int3(FAR_ATOM, 0, 0);
    };
    // its coordinates under the run's image, and whether they are in reach
    auto place = [&](const int3 c, int code, float &x, float &y, float &z) {
      unsigned ux = c.x, uy = c.y, uz = c.z;
      if (code != IMG_ZERO) {
        int W0, W1, W2;
        img_decode(code, W0, W1, W2);
        ux += W0 * Lx;
        uy += W1 * Ly;
        uz += W2 * Lz;
      }
      x = (float)(int)(ux - ox) * QUANTUM;
      y = (float)(int)(uy - oy) * QUANTUM;
      z = (float)(int)(uz - oz) * QUANTUM;
      const float dx = fmaxf(fmaxf(bx0 - x, x - bx1), 0.0f), dy = fmaxf(fmaxf(by0 - y, y - by1), 0.0f),
                  dz = fmaxf(fmaxf(bz0 - z, z - bz1), 0.0f);
      return c.x != FAR_ATOM && (A.wide || dx * dx + dy * dy + dz * dz <= reach2);
    };
    auto keep = [&](unsigned m, int at, int k, int code, float x, float y, float z) {
      at += __popc(m & lanemask_lt());
      reinterpret_cast<float *>(kx4)[at] = x;
      reinterpret_cast<float *>(ky4)[at] = y;
      reinterpret_cast<float *>(kz4)[at] = z;
      entry[at] = (k << IMG_BITS) | code;
      if (code == IMG_ZERO && (unsigned)(k - chunk * 32) < 32u) self_at[k - chunk * 32] = at;
    };

    int nin = 0, nout = 0, nh = 0;
    int r = 0;
    int code1 = 0, k1 = -1;
    int3 c1 = make_int3(FAR_ATOM, 0, 0);
    if (NW == 1) {
      k1 = candidate(0, code1);
      c1 = fetch(k1);
    }
    while (r < nraw) {
      sync();
      if (warp == 0) self_at[lane] = -1;
      sync();
      int n = 0;   // candidates kept
      if (NW == 1) {
        // the next word's candidates are on their way while one is placed
        while (r < nraw && n + 32 <= MAXW * 32) {
          const int k = k1, code = code1;
          const int3 c = c1;
          if (++r < nraw) {
            k1 = candidate(r, code1);
            c1 = fetch(k1);
          }
          float x, y, z;
          const bool ok = place(c, code, x, y, z);
          const unsigned m = __ballot_sync(0xffffffffu, ok);
          if (ok) keep(m, n, k, code, x, y, z);
          n += __popc(m);
        }
      } else {
        const int r1 = min(nraw, r + MAXW);
        for (int u = r + warp; u < r1; u += NW) {
          int code;
          float x, y, z;
          const int k = candidate(u, code);
          const unsigned m = __ballot_sync(0xffffffffu, place(fetch(k), code, x, y, z));
          if (lane == 0) kept[u - r] = m;
        }
        __syncthreads();
        int at = lane < r1 - r ? __popc(kept[lane]) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, at, o);
          if (lane >= o) at += v;
        }
        n = __shfl_sync(0xffffffffu, at, 31);
        for (int u = r + warp; u < r1; u += NW) {
          int code;
          float x, y, z;
          const int k = candidate(u, code);
          const unsigned m = kept[u - r];
          const int a0 = u > r ? __shfl_sync(0xffffffffu, at, (u - r - 1) & 31) : 0;
          place(fetch(k), code, x, y, z);
          if ((m >> lane) & 1u) keep(m, a0, k, code, x, y, z);
        }
        r = r1;
      }
      sync();
      const int nw = (n + 31) >> 5;
      for (int w = warp; w < nw; w += NW) {
        // the distance in explicitly rounded operations (packed ones round as
        // the scalar ones): the in-cutoff mark decides an entry's list segment,
        // so every kernel that builds these lists must round it the same way
        unsigned mp = 0, ms = 0, mi = 0;
#pragma unroll
        for (int g = 0; g < 8; g++) {
          const float4 x = kx4[w][g], y = ky4[w][g], z = kz4[w][g];
          const F2 ex = f2_sub(wx2, f2_pack(x.x, x.y)), fx = f2_sub(wx2, f2_pack(x.z, x.w));
          const F2 ey = f2_sub(wy2, f2_pack(y.x, y.y)), fy = f2_sub(wy2, f2_pack(y.z, y.w));
          const F2 ez = f2_sub(wz2, f2_pack(z.x, z.y)), fz = f2_sub(wz2, f2_pack(z.z, z.w));
          const F2 r2 = f2_fma(ez, ez, f2_fma(ey, ey, f2_mul(ex, ex)));
          const F2 s2 = f2_fma(fz, fz, f2_fma(fy, fy, f2_mul(fx, fx)));
          mp = f2_signs(f2_signs(mp, f2_sub(r2, lim_pre)), f2_sub(s2, lim_pre));
          ms = f2_signs(f2_signs(ms, f2_sub(r2, lim_sure)), f2_sub(s2, lim_sure));
          mi = f2_signs(f2_signs(mi, f2_sub(r2, lim_in)), f2_sub(s2, lim_in));
        }
        const int nv = n - 32 * w;
        unsigned valid = near ? (nv < 32 ? 0xffffffffu << (32 - nv) : 0xffffffffu) : 0u;
        // its own place under its own image (an atom of the box: image zero)
        const int self = self_at[lane];
        if (unwrapped && self >= 0 && (self >> 5) == w) valid &= ~(0x80000000u >> (self & 31));
        mp &= valid;
        unsigned acc = ms & mp, in = mi & acc, band = mp & ~acc;
        if (A.want_half || A.wide || !unwrapped) {
          // half lists, and atoms outside the box, take every candidate
          // through the exact test, in order (in wide cells even those that
          // the screen drops)
          band = A.wide ? valid : mp;
          acc = in = 0;
        }
        while (band) {
          const int at = __clz(band);
          const unsigned bit = 0x80000000u >> at;
          band &= ~bit;
          const int e = entry[32 * w + at];
          int W[3];
          img_decode(e & ((1 << IMG_BITS) - 1), W[0], W[1], W[2]);
          try_atom(A, q, (int)__double_as_longlong(A.acell_pos[e >> IMG_BITS].w), W, nh, [&](int, int cd) {
            acc |= bit;
            if (cd & IN_CUT) in |= bit;
          });
        }
        __syncwarp();
        m_acc[32 * w + lane] = acc;
        m_in[32 * w + lane] = in;
      }
      sync();
      // write-out of one segment: front entries to rows n.., back ones from
      // row cap - 1 down
      auto write = [&](const bool front, int &n) {
        auto mask = [&](int w) { return front ? m_in[32 * w + lane] : m_acc[32 * w + lane] & ~m_in[32 * w + lane]; };
        unsigned some = 0;   // the lane's words with entries, first word in the top bit
        for (int w = 0; w < nw; w++)
          if (mask(w)) some |= 0x80000000u >> w;
        int w = 0;
        unsigned bits = 0;
        while (__any_sync(0xffffffffu, (some | bits) != 0)) {
          if (!bits && some) {
            w = __clz(some);
            some &= ~(0x80000000u >> w);
            bits = mask(w);
          }
          if (bits) {
            const int at = __clz(bits);
            bits &= ~(0x80000000u >> at);
            int e = entry[32 * w + at];
            if (!unwrapped) {
              int W0, W1, W2;
              img_decode(e & ((1 << IMG_BITS) - 1), W0, W1, W2);
              e = (e & ~((1 << IMG_BITS) - 1)) | img_code(W0 - q.ti[0], W1 - q.ti[1], W2 - q.ti[2]);
            }
            if (n < A.cap) A.nbr_full[(size_t)(front ? n : A.cap - 1 - n) * A.nsi + h] = e;
            n++;
          }
        }
      };
      if (NW == 1) {
        write(true, nin);
        write(false, nout);
      } else if (warp == 0) {
        write(true, nin);
      } else if (warp == 1) {
        write(false, nout);
      }
    }
    if (NW > 1) {
      if (warp == 1) back[lane] = nout;
      __syncthreads();
      nout = back[lane];
    }
    if (warp == 0 && active) {
      A.site_from[h] = make_int2(nin, nout);
      finish_counts(A, h, nin, nout, nh);
    }
  }
}

// Large systems: one warp per chunk.  Small ones (below SMALL_CHUNKS per SM),
// whose chunks would leave most of the chip idle: the chunk's words over four
// warps and the two segments' write-outs over two.  Measured per build against
// one warp walking its chunk candidate by candidate (42 instructions a
// candidate, entries staged in shared memory): 4.18 M atoms 6.05 -> 2.02 ms,
// 1.05 M 1.56 -> 0.54 ms, 272 k 474 -> 177 us, 4,374 atoms (four warps)
// 183 -> 47 us, 64 replicas of 1.44 M atoms 1.37 -> 0.51 ms.
template <int NW, class RP>
__global__ void __launch_bounds__(32 * NW) k_build_atoms(BuildArgs A, RP P) {
  build_atoms_chunk<NW>(A, P, blockIdx.x);
}

// Single systems: persistent warps taking the chunks in SM-local runs (one
// chunk per run, sm_run in device.cuh), so that the warps resident on one SM
// walk neighbouring cells and share their candidates in L1.  The same lists.
__global__ void __launch_bounds__(32) k_build_atoms_sm(BuildArgs A, OneRep P, int nchunk, int *cnt, int nsm) {
  __shared__ int v;
  if (threadIdx.x == 0) v = sm_id() % nsm;
  for (;;) {
    const int chunk = sm_run(cnt, nsm, nchunk, v);
    if (chunk < 0) return;
    build_atoms_chunk<1>(A, P, chunk);
  }
}

// Phase A over every list slot: the element walk of each atom and Gauss
// point; atoms with at least one item go on the work list of phase B (its
// order does not matter: an atom's entries depend on that atom alone).
// The Gauss points go first, a warp for each element's eight (their walk is the
// longest, and the atoms' fill in behind it), then the atoms, Q to a warp: 32
// of the sorted ones, in a small system 8 (below EIGHT_QUERY_SITES a warp's
// serial chain of loads is what the kernel takes: 6 k sites 20.5 us against
// 22.9, while at 80 k to 88 k sites 32 are the faster by a fifth).
// A query alone walked 27 cells, about 130 elements, in FP64, and its warp took
// 6,700 instructions in one long chain.  Measured per build, before and after:
// 1,554 queries 29 -> 16 us, 83,550 88 -> 31 us, 93,000 (FIRE) 145 -> 40 us,
// 313,120 142 -> 53 us, 4.98 M 1024 -> 571 us, 64 replicas with 1.72 M
// 828 -> 343 us.  Groups of queries within one cell, half of one or a quarter
// instead of two: 5 M queries 1074, 1692 and 2662 us against 858 (each group
// walks the cells again).  Registers: 8 blocks an SM at Q = 32 (96 -> 64
// registers; 694 -> 571 us at 5 M), 5 at Q = 8, where more only spills.
constexpr int EIGHT_QUERY_SITES = 30000;
template <int Q, class RP>
__device__ __forceinline__ void elem_items_queries(const BuildArgs &A, const RP &P, int first, int end, int2 *items,
                                                   int *nitems, int icap, int *work, int *nwork, NearStage &st) {
  constexpr int S = 32 / Q;
  const int lane = threadIdx.x & 31, place = first + lane / S;
  const bool live = place < end;
  const int t = live ? place : end - 1;
  const int i = t < A.na ? A.atom_of_slot[t] : t;
  Query q;
  make_query(A, P, i, q);
  q.slot = t;
  int rep = 0;
  if constexpr (RP::many) rep = P.site_rep[i];
  const int n = element_items<Q>(A, q, rep, live, items + (size_t)t * icap, icap, st);
  const bool one = live && lane % S == 0;
  if (one) {
    nitems[t] = n;
    if (n > icap) {
      atomicExch(&A.overflow[8], 1);
      atomicMax(&A.overflow[9], n);
    }
  }
  const bool listed = one && t < A.na && n > 0;
  const unsigned m = __ballot_sync(0xffffffffu, listed);
  int at = 0;
  if (m && lane == 0) at = atomicAdd(nwork, __popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (listed) work[at + __popc(m & lanemask_lt())] = t;
}

template <int Q, class RP>
__global__ void __launch_bounds__(128, Q == 32 ? 8 : 5) k_elem_items(BuildArgs A, RP P, int2 *items, int *nitems, int icap, int *work,
                                                    int *nwork) {
  __shared__ NearStage stage[4];
  NearStage &st = stage[threadIdx.x >> 5];
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w < A.ne)
    elem_items_queries<8>(A, P, A.na + NG * w, A.nsi, items, nitems, icap, work, nwork, st);
  else if (Q * (w - A.ne) < A.na)   // whole warps
    elem_items_queries<Q>(A, P, Q * (w - A.ne), A.na, items, nitems, icap, work, nwork, st);
}

// Phase B for atoms: one warp per listed atom, its element sites appended
// after its atom neighbours.
template <class RP>
__global__ void __launch_bounds__(128, 7) k_build_atom_sites(BuildArgs A, RP P, const int2 *items, const int *nitems,
                                                          int icap, const int *work, const int *nwork) {
  __shared__ ItemStage stage[4];
  ItemStage &st = stage[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  // the next query's place, atom and counts are on their way while one is
  // worked on (a chain of loads as long as a query's own work)
  const int nw = *nwork, step = (gridDim.x * blockDim.x) >> 5;
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int h = w < nw ? work[w] : 0, h1 = w + step < nw ? work[w + step] : 0;
  int i = A.atom_of_slot[h], ni = nitems[h], fin = A.num_in[h], num = A.num_full[h];
  for (; w < nw; w += step) {
    Query q;
    make_query(A, P, i, q);
    q.slot = h;
    int nin = fin, nout = num - fin, nh = A.want_half ? A.num_half[h] : 0;
    const int here = h, n = min(ni, icap);
    h = h1;
    h1 = w + 2 * step < nw ? work[w + 2 * step] : 0;
    i = A.atom_of_slot[h];
    ni = nitems[h];
    fin = A.num_in[h];
    num = A.num_full[h];
    items_warp(A, q, items + (size_t)here * icap, n, st, A.raw_sites + ((size_t)NG * A.ne + w) * A.cap, nin, nout, nh);
    if (lane == 0) finish_counts(A, here, nin, nout, nh);
    __syncwarp();
  }
}

// Phase B for Gauss points: one warp each; atoms from the 27 surrounding atom
// cells (full list only), 32 candidates at a time, then the element sites.
template <class RP>
__global__ void __launch_bounds__(128, 7) k_build_gauss(BuildArgs A, RP P, const int2 *items, const int *nitems,
                                                     int icap) {
  __shared__ ItemStage stage[4];
  ItemStage &st = stage[threadIdx.x >> 5];
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= NG * A.ne) return;   // whole warps
  Query q;
  make_query(A, P, A.na + t, q);
  const Grid &ag = q.r.ag;
  int nin = 0, nout = 0, nh = 0;
  if (A.na > 0) {
    const double pre = (A.cutneigh + 1e-6) * (A.cutneigh + 1e-6);
    int ci[3];
#pragma unroll
    for (int d = 0; d < 3; d++)
      ci[d] = min(max((int)((q.wi[d] - q.r.b.lo[d]) * ag.inv[d]), 0), ag.nc[d] - 1);
    // no atom in the 27 cells around (most Gauss points of an element
    // region): no atom candidates, the walk below would find none
    const bool atoms_near = !A.acell_near || A.acell_near[q.r.abase + (ci[2] * ag.nc[1] + ci[1]) * ag.nc[0] + ci[0]];
    if (atoms_near)
    for (int oz = -1; oz <= 1; oz++) {
      int cz, Wz;
      wrap_cell(ci[2] + oz, ag.nc[2], cz, Wz);
      for (int oy = -1; oy <= 1; oy++) {
        int cy, Wy;
        wrap_cell(ci[1] + oy, ag.nc[1], cy, Wy);
        for (int ox = -1; ox <= 1; ox++) {
          int cx, Wx;
          wrap_cell(ci[0] + ox, ag.nc[0], cx, Wx);
          int cell = q.r.abase + (cz * ag.nc[1] + cy) * ag.nc[0] + cx;
          int W[3] = {Wx, Wy, Wz};
          double sh[3] = {Wx * q.r.b.L[0], Wy * q.r.b.L[1], Wz * q.r.b.L[2]};
          int beg = A.acell_start[cell], end = A.acell_start[cell + 1];
          for (int base = beg; base < end; base += 32) {
            const int k = base + lane;
            bool pass = false;
            int j = 0, code = 0;
            if (k < end) {
              double4 pj = A.acell_pos[k];
              double ex = q.wi[0] - (pj.x + sh[0]), ey = q.wi[1] - (pj.y + sh[1]), ez = q.wi[2] - (pj.z + sh[2]);
              if (ex * ex + ey * ey + ez * ez <= pre) {
                j = (int)__double_as_longlong(pj.w);
                pass = gauss_atom_test(A, q, j, W, code);
              }
            }
            // the atom's list slot is its sorted position k
            warp_emit_full(A, q.slot, nin, nout, pass, (code & IN_CUT) != 0,
                           (k << IMG_BITS) | (code & (IN_CUT - 1)));
          }
        }
      }
    }
  }
  const int slot = A.na + t;
  if (lane == 0) A.site_from[slot] = make_int2(nin, nout);
  items_warp(A, q, items + (size_t)slot * icap, min(nitems[slot], icap), st, A.raw_sites + (size_t)t * A.cap, nin, nout,
             nh);
  if (lane == 0) finish_counts(A, q.slot, nin, nout, nh);
}

// ------------------------------------------------------------- compaction

// The table of marked sites, one warp per element: its marks become words of
// bits, each with the rank of its first site, and its sites get consecutive
// ranks.  Elements take their ranges from a counter, a block at a time, so
// their order in the table may differ from one rebuild to the next; nothing
// depends on it.
__global__ void __launch_bounds__(256) k_act_table(const unsigned char *flag, int ne, int nsi, uint2 *words, int *act_gid,
                                                   int *nact, int *too_many) {
  __shared__ int total[8], base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * 8 + warp;
  unsigned word = 0;
  if (e < ne) {
    const unsigned char *f = flag + (size_t)e * MARKS;
#pragma unroll
    for (int w = 0; w < MARK_WORDS; w++) {
      const unsigned b = __ballot_sync(0xffffffffu, f[32 * w + lane] != 0);
      if (lane == w) word = b;
    }
  }
  int incl = __popc(word);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) total[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int w = 0; w < 8; w++) {
      const int t = total[w];
      total[w] = n;
      n += t;
    }
    base = atomicAdd(nact, n);
    if ((long)nsi + base + n >= (1L << (31 - IMG_BITS))) *too_many = 1;
  }
  __syncthreads();
  if (e >= ne) return;
  const int first = base + total[warp] + incl - __popc(word);
  if (lane < MARK_WORDS) words[(size_t)e * MARK_WORDS + lane] = make_uint2(word, first);
#pragma unroll 1
  for (int w = 0; w < MARK_WORDS; w++) {
    const unsigned b = __shfl_sync(0xffffffffu, word, w);
    const int r = __shfl_sync(0xffffffffu, first, w);
    if ((b >> lane) & 1u) act_gid[r + __popc(b & lanemask_lt())] = e * NU + 32 * w + lane;
  }
}

// Pair-table index of lattice site u of element e (Gauss points at their fixed
// place, the other sites by rank among the marked ones).
__device__ __forceinline__ int site_index(int e, int u, const uint2 *words, int na, int ne) {
  const int g = site_gauss(u);
  if (g >= 0) return na + NG * e + g;
  const uint2 w = words[(size_t)e * MARK_WORDS + (u >> 5)];
  return na + NG * ne + (int)w.y + __popc(w.x & ((1u << (u & 31)) - 1u));
}

// Packs each entry of a half list as (pair-table index << 5 | image code): atoms
// by their list slot (the pair table holds atoms in cell-sorted order), element
// sites after them as in the site table.  Entries inside the inner radius (the
// force cutoff plus a margin) at build time go first, each group in build order.
__global__ void k_remap(const int *raw, const unsigned char *img, const int *num, int nsi, int cap,
                        const uint2 *words, const int *atom_slot, int na, int ne, int *out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsi) return;
  int n = min(num[i], cap);
  int nin = 0;
  for (int k = 0; k < n; k++) nin += (img[(size_t)k * nsi + i] & IN_CUT) != 0;
  int a = 0, b = nin;   // next in-cutoff and next other position
  for (int k = 0; k < n; k++) {
    size_t o = (size_t)k * nsi + i;
    unsigned char im = img[o];
    int v = raw[o];
    int sidx;
    if (v & KIND_SITE) {
      const int gid = v & ~KIND_SITE;
      sidx = site_index(gid / NU, gid % NU, words, na, ne);
    } else {
      sidx = atom_slot[v];
    }
    const int w = (im & IN_CUT) ? a++ : b++;
    out[(size_t)w * nsi + i] = (sidx << IMG_BITS) | (im & (IN_CUT - 1));
  }
}

// Element-site entries into the full lists: from (item, lattice site) in the
// queries' own rows to pair-table indices in the transposed lists (rows
// site_from.x .. num_in - 1 of the front segment, cap - back .. cap - 1 -
// site_from.y of the back one).  Only Gauss points and the atoms of the work
// list have any.  A block takes 32 of them at a time and turns their entries
// through shared memory, so that it reads along a query's row and writes along
// the lists' rows (neighbouring queries are mostly neighbouring list slots).
// With the site table: 522 us for 100,000 elements with 4.18 M atoms, 542 us
// for 64 replicas of 1.44 M atoms (385 and 304 us where a query's entries stood
// in the lists' rows from the start, whose scattered stores cost the kernels
// before it more).
__global__ void __launch_bounds__(256) k_remap_sites(const int *raw, const int2 *items, int icap, const int *num,
                                                     const int *num_in, const int2 *site_from, int nsi, int cap,
                                                     const uint2 *words, int na, int ne, const int *work,
                                                     const int *nwork, int *out) {
  __shared__ int tile[32][33];
  __shared__ int slot[32], from[2][32], count[2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = NG * ne + *nwork;
  for (int d0 = blockIdx.x * 32; d0 < n; d0 += gridDim.x * 32) {
    __syncthreads();
    if (warp == 0) {
      const int d = d0 + lane;
      int i = -1, nf = 0, nb = 0;
      int2 f = make_int2(0, 0);
      if (d < n) {
        i = d < NG * ne ? na + d : work[d - NG * ne];
        const int nin = num_in[i], nback = num[i] - nin;
        f = site_from[i];
        if (nin + nback <= cap) {   // else an overflow: the build is repeated
          nf = nin - f.x;
          nb = nback - f.y;
        }
      }
      slot[lane] = i;
      from[0][lane] = f.x;
      from[1][lane] = f.y;
      count[0][lane] = nf;
      count[1][lane] = nb;
    }
    __syncthreads();
#pragma unroll 1
    for (int seg = 0; seg < 2; seg++) {
      const int c = count[seg][lane], f = from[seg][lane];
      const int most = __reduce_max_sync(0xffffffffu, c);
      for (int k0 = 0; k0 < most; k0 += 32) {
        // each query's entries k0 .. k0 + 31 of the segment, a query at a time
        // (four of them per warp, their loads side by side)
        int e[4], el[4], code[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int s = warp + 8 * u, k = k0 + lane;
          e[u] = k < count[seg][s] ? raw[(size_t)(d0 + s) * cap + (seg ? cap - 1 - k : k)] : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int2 it = e[u] >= 0 ? items[(size_t)slot[warp + 8 * u] * icap + (e[u] >> 10)] : make_int2(0, 0);
          int sv[3], bl[3], bh[3];
          unpack_item(it, el[u], sv, bl, bh);
          code[u] = img_code(sv[0], sv[1], sv[2]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          tile[lane][warp + 8 * u] =
              e[u] >= 0 ? (site_index(el[u], e[u] & 1023, words, na, ne) << IMG_BITS) | code[u] : -1;
        __syncthreads();
        for (int k = warp; k < min(32, most - k0); k += 8) {
          const int v = tile[k][lane], row = seg ? cap - 1 - (f + k0 + k) : f + k0 + k;
          if (v >= 0) out[(size_t)row * nsi + slot[lane]] = v;
        }
        __syncthreads();
      }
    }
  }
}

inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

// Reference atom bins of a single system (nbin_standard.cpp:84-128),
// orthogonal box: used only by the half-list storage rule.
void setup_ref_bins(Ctx &c) {
  double binsize_optimal = 0.5 * c.cutneigh;
  double binsizeinv = 1.0 / binsize_optimal;
  for (int d = 0; d < 3; d++) {
    double bbox = c.boxhi[d] - c.boxlo[d];
    c.rbins.lo[d] = c.boxlo[d];
    c.rbins.hi[d] = c.boxhi[d];
    int nb = (int)(bbox * binsizeinv);
    if (nb == 0) nb = 1;
    c.rbins.nbin[d] = nb;
    double bs = bbox / nb;
    c.rbins.inv[d] = 1.0 / bs;
  }
}

// Candidate grids of one replica: atoms in cells >= cutneigh, element
// centres in cells >= cutneigh + element reach.
void setup_grids(const Ctx &c, Rep &r, bool has_elements) {
  for (int d = 0; d < 3; d++) {
    double L = r.b.L[d];
    int na_c = (int)(L / c.cutneigh);
    if (na_c < 1) throw Error(CACB200_EINVAL, "box shorter than the neighbour cutoff");
    r.ag.nc[d] = na_c;
    r.ag.inv[d] = na_c / L;
    double reach = c.cutneigh + r.reach_budget + 1e-6;
    if (has_elements && L < reach)
      throw Error(CACB200_EINVAL, "box shorter than the cutoff plus the element radius in dimension " +
                                      std::to_string(d));
    int ne_c = std::max(1, (int)(L / reach));
    r.eg.nc[d] = ne_c;
    r.eg.inv[d] = ne_c / L;
  }
  r.ag.ncell = r.ag.nc[0] * r.ag.nc[1] * r.ag.nc[2];
  r.eg.ncell = r.eg.nc[0] * r.eg.nc[1] * r.eg.nc[2];
}

// Launch a rebuild kernel for a single system or a batch.
template <class F>
void with_reps(const Ctx &c, F &&f) {
  if (c.nrep == 1) {
    OneRep P{c.rep_h[0]};
    f(P);
  } else {
    ManyRep P{c.rep_d.p, c.site_rep.p, c.elem_rep.p, c.acell_rep.p};
    f(P);
  }
}

}  // namespace

// Capacity plan: sizes every buffer of a rebuild for the current system (site
// table for the worst case of every lattice site active, candidate grids with
// room for elements to grow, list slots of `cap` per site), so that rebuilds
// afterwards neither allocate nor synchronise and can be queued or captured
// in a CUDA graph.  Synchronises once to read the element radii.
void neigh_plan(Ctx &c, bool want_half) {
  c.check_system();
  if (c.pp.style == CACB200_PAIR_NONE) throw Error(CACB200_ESTATE, "no pair style set");
  if (want_half && c.nrep > 1) throw Error(CACB200_EINVAL, "half lists are built for single systems only");
  double cutoff = std::sqrt(c.pp.cut * c.pp.cut);
  c.cutneigh = cutoff + c.skin;
  c.cutneighsq = c.cutneigh * c.cutneigh;
  c.ecenter.reserve(std::max(c.ne, 1));
  c.eframe.reserve((size_t)std::max(c.ne, 1) * EFR);
  c.overflow.reserve(16);
  c.dev_nact.reserve(1);
  c.inner_margin = c.inner_margin_set >= 0.0 ? c.inner_margin_set : 0.5 * c.skin;
  c.inner_ok.reserve(c.nrep);
  c.disp.reserve(std::max(c.na, 1));
  c.edisp.reserve(std::max(c.ne, 1));
  c.dmax.reserve(c.nrep);
  c.xbuild.reserve(std::max(c.na, 1));
  c.nodex_build.reserve(24 * (size_t)std::max(c.ne, 1));
  c.num_in.reserve(std::max(c.nsite_i(), 1));
  c.reach_bits.reserve(c.nrep);
  c.rep_d.reserve(c.nrep);
  c.sm_counter.reserve(2 * c.num_sms);
  CACB200_CUDA(cudaMemsetAsync(c.overflow.p, 0, 16 * sizeof(int), c.stream));
  CACB200_CUDA(cudaMemsetAsync(c.dev_nact.p, 0, sizeof(int), c.stream));
  CACB200_CUDA(cudaMemsetAsync(c.reach_bits.p, 0, sizeof(unsigned long long) * c.nrep, c.stream));
  // element geometry with no reach limit, to measure each replica's radius
  for (Rep &r : c.rep_h) r.reach_budget = 1e300;
  stream_copy(c, c.rep_d.p, c.rep_h.data(), sizeof(Rep) * c.nrep, cudaMemcpyHostToDevice);
  std::vector<unsigned long long> bits(c.nrep, 0);
  if (c.ne) {
    with_reps(c, [&](auto P) {
      if (c.na) k_pbc_atoms<<<nblk(c.na, 256), 256, 0, c.stream>>>(c.xs.p, c.na, P, BuildStart{});
      k_elem_geom<<<nblk(c.ne, 64), 64, 0, c.stream>>>(c.nodex.p, c.ne, P, c.ecenter.p, c.eframe.p,
                                                       c.reach_bits.p, c.overflow.p + 3, nullptr, nullptr, nullptr,
                                                       nullptr, nullptr);
    });
    stream_copy(c, bits.data(), c.reach_bits.p, sizeof(unsigned long long) * c.nrep, cudaMemcpyDeviceToHost);
  }
  int abase = 0, ebase = 0;
  for (int r = 0; r < c.nrep; r++) {
    Rep &R = c.rep_h[r];
    double ereach = 0.0;
    std::memcpy(&ereach, &bits[r], sizeof(double));
    if (!(ereach < 1e30)) throw Error(CACB200_EUNSTABLE, "non-finite element geometry");
    // elements may grow by 20 % (and 2 A) before the grid is planned again,
    // as far as the box allows
    R.reach_budget = 0.0;
    if (c.rep_ne[r]) {
      double room = std::min(R.b.L[0], std::min(R.b.L[1], R.b.L[2])) - c.cutneigh - 2e-6;
      R.reach_budget = std::max(ereach, std::min(std::max(1.2 * ereach, ereach + 2.0), room));
    }
    setup_grids(c, R, c.rep_ne[r] > 0);
    // fixed-point frame of the mixed form: quantum 2^-26 A, box length in
    // quanta modulo 2^32 (pair separations are taken modulo 2^32 as well)
    for (int d = 0; d < 3; d++) {
      R.qscale[d] = std::ldexp(1.0, 26);
      R.Lq[d] = (int)(uint32_t)(uint64_t)std::llrint(R.b.L[d] * R.qscale[d]);
    }
    R.abase = abase;
    R.ebase = ebase;
    abase += R.ag.ncell;
    ebase += R.eg.ncell;
  }
  stream_copy(c, c.rep_d.p, c.rep_h.data(), sizeof(Rep) * c.nrep, cudaMemcpyHostToDevice);
  c.agrid.ncell = abase;
  c.egrid.ncell = ebase;
  if (c.nrep > 1) {
    std::vector<int> cr(abase);
    for (int r = 0; r < c.nrep; r++)
      std::fill(cr.begin() + c.rep_h[r].abase, cr.begin() + c.rep_h[r].abase + c.rep_h[r].ag.ncell, r);
    c.acell_rep.reserve(abase);
    stream_copy(c, c.acell_rep.p, cr.data(), sizeof(int) * abase, cudaMemcpyHostToDevice);
  } else {
    setup_ref_bins(c);
  }

  const int nsi = c.nsite_i();
  const size_t ngid = (size_t)c.ne * NU;
  int nmax = std::max(std::max(c.na, c.ne), 1);
  c.atom_key.reserve(std::max(c.na, 1));
  c.atom_place.reserve(std::max(c.na, 1));
  c.atom_order.reserve(std::max(c.na, 1));
  c.elem_key.reserve(std::max(c.ne, 1));
  c.elem_place.reserve(std::max(c.ne, 1));
  c.elem_order.reserve(std::max(c.ne, 1));
  c.cell_count.reserve((size_t)c.agrid.ncell + c.egrid.ncell + 2);
  c.slot_atom.reserve(nmax);
  c.atom_slot.reserve(std::max(c.na, 1));
  c.xss.reserve(std::max(c.xs.n, (size_t)1));
  c.acell_start.reserve(c.agrid.ncell + 1);
  c.acell_pos.reserve(std::max(c.na, 1));
  c.acell_fix.reserve(3 * (size_t)std::max(c.na, 1));
  c.acell_of.reserve(std::max(c.na, 1));
  c.ecell_start.reserve(c.egrid.ncell + 1);
  c.ecell_near.reserve(c.egrid.ncell + 1);
  c.acell_near.reserve(c.agrid.ncell + 1);
  c.ecell_elems.reserve(std::max(c.ne, 1));
  c.ecell_box.reserve(sizeof(ElemBox) * std::max(c.ne, 1));
  size_t slots = (size_t)c.cap * std::max(nsi, 1);
  c.raw_sites.reserve(slots);
  c.num_full.reserve(std::max(nsi, 1));
  c.site_from.reserve(std::max(nsi, 1));
  c.nbr_full.reserve(slots);
  if (want_half) {
    c.raw_half.reserve(slots);
    c.img_half.reserve(slots);
    c.num_half.reserve(std::max(nsi, 1));
    c.nbr_half.reserve(slots);
  }
  c.items.reserve((size_t)std::max(nsi, 1) * c.item_cap);
  c.nitems.reserve(std::max(nsi, 1));
  c.atom_work.reserve(std::max(c.na, 1));
  c.atom_nwork.reserve(1);
  c.site_flag.reserve((size_t)std::max(c.ne, 1) * MARKS);
  c.site_words.reserve((size_t)std::max(c.ne, 1) * MARK_WORDS);
  c.act_gid.reserve(std::max<size_t>(ngid, 1));
  // site table for every lattice site active, keeping the atom positions
  size_t ns_cap = (size_t)nsi + ngid;
  if (ns_cap > c.xs.n) {
    double4 *np_ = nullptr;
    if (cudaMalloc(&np_, ns_cap * sizeof(double4)) != cudaSuccess) {
      cudaGetLastError();
      throw Error(CACB200_ENOMEM, "site table allocation failed");
    }
    if (c.na)
      CACB200_CUDA(cudaMemcpyAsync(np_, c.xs.p, sizeof(double4) * c.na, cudaMemcpyDeviceToDevice, c.stream));
    CACB200_CUDA(cudaStreamSynchronize(c.stream));
    cudaFree(c.xs.p);
    c.xs.p = np_;
    c.xs.n = ns_cap;
  }
  c.ns_cap = ns_cap;
  // CUB temporary storage of the cell scans
  size_t need = 0, bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, c.cell_count.p, c.acell_start.p, c.agrid.ncell + 1, c.stream);
  need = bytes;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, c.cell_count.p, c.ecell_start.p, c.egrid.ncell + 1, c.stream);
  need = std::max(need, bytes);
  c.cub_tmp.reserve(std::max<size_t>(need, 1));
  c.cub_bytes = need;
  c.plan_half = want_half;
  c.planned = true;
  const long gen_before = c.gen;
  c.gen++;
  if (c.box_replan) {
    // only the box moved (fix deform): the block sizes chosen for this
    // system stay valid
    if (c.tune_gen == gen_before) c.tune_gen = c.gen;
    c.box_replan = false;
  }
  c.plan_na = c.na;
  c.plan_ne = c.ne;
}

// Queue a rebuild: pbc, element geometry, binning, candidate search, storage
// rules, compaction of the referenced lattice sites and packing of the list
// entries.  Nothing here allocates or waits for the device; problems are
// reported in the flag words (list overflow, distant image, element grown past
// the grid plan) for neigh_check.
void neigh_build_async(Ctx &c, bool want_half) {
  if (!c.planned || c.plan_na != c.na || c.plan_ne != c.ne || (want_half && !c.plan_half))
    throw Error(CACB200_ESTATE, "rebuild without a capacity plan");
  const int nsi = c.nsite_i();
  with_reps(c, [&](auto P) {
    using RP = decltype(P);
    {
      KernelTimer t(c, "pbc_geom");
      // the positions these lists are built from are kept for the displacement
      // test of the inner prefix, which is usable until a site has moved far
      const BuildStart S{c.xbuild.p, c.disp.p,       c.inner_ok.p, inner_limit(c) > 0.0 ? 1 : 0, c.dmax.p,
                         c.overflow.p, c.dev_nact.p, c.atom_nwork.p, c.sm_counter.p,
                         c.nrep,       c.num_sms,    c.atom_key.p,     c.atom_place.p, c.cell_count.p};
      // counts of the atom cells, one more, then of the element cells and one
      // more (the single-block scan needs no gap: its element counts follow)
      const bool small = c.agrid.ncell + (c.ne ? c.egrid.ncell : 0) <= SCAN_CELLS;
      int *const ecount = c.cell_count.p + c.agrid.ncell + (small ? 0 : 1);
      CACB200_CUDA(cudaMemsetAsync(c.cell_count.p, 0, sizeof(int) * ((size_t)c.agrid.ncell + c.egrid.ncell + 2),
                                   c.stream));
      const int n = std::max(std::max(c.na, c.nrep), c.num_sms);
      k_pbc_atoms<<<nblk(n, 256), 256, 0, c.stream>>>(c.xs.p, c.na, P, S);
      if (c.ne)
        launch_behind(c, nblk(c.ne, 64), 64, 0, k_elem_geom<RP>, c.nodex.p, c.ne, P, c.ecenter.p, c.eframe.p,
                      c.reach_bits.p, c.overflow.p + 3, c.nodex_build.p, c.edisp.p, c.elem_key.p, c.elem_place.p,
                      ecount);
    }
    {
      KernelTimer t(c, "bin");
      const int nac = c.agrid.ncell, nec = c.ne ? c.egrid.ncell : 0;
      if (nac + nec <= SCAN_CELLS) {
        launch_behind(c, 1, 1024, 0, k_scan_cells, c.cell_count.p, nac, nec, c.acell_start.p, c.ecell_start.p);
      } else {
        size_t bytes = c.cub_bytes;
        CACB200_CUDA(cub::DeviceScan::ExclusiveSum(c.cub_tmp.p, bytes, c.cell_count.p, c.acell_start.p, nac + 1, c.stream));
        if (c.ne)
          CACB200_CUDA(cub::DeviceScan::ExclusiveSum(c.cub_tmp.p, bytes, c.cell_count.p + nac + 1, c.ecell_start.p,
                                                     nec + 1, c.stream));
      }
      const bool near = c.nrep == 1 && c.ne;
      const BinArgs B{c.atom_key.p,  c.atom_place.p, c.acell_start.p, c.elem_key.p, c.elem_place.p,
                      c.ecell_start.p, c.atom_order.p, c.elem_order.p, c.na,         c.ne,
                      near ? c.acell_near.p : nullptr, near ? c.ecell_near.p : nullptr,
                      c.rep_h[0].ag, c.rep_h[0].eg, (float)c.cutneigh, want_half ? nullptr : c.overflow.p + 2};
      const long n = (long)c.na + c.ne, cells = near ? (long)c.rep_h[0].ag.ncell + c.rep_h[0].eg.ncell : 0;
      if (n + cells) launch_behind(c, nblk(n + cells, 256), 256, 0, k_scatter, B);
      if (n)
        launch_behind(c, nblk(n, 256), 256, 0, k_place<RP>, B, P, c.xs.p, c.acell_pos.p, c.acell_fix.p, c.slot_atom.p,
                      c.atom_slot.p, c.acell_of.p, c.ecenter.p, c.eframe.p, c.ecell_elems.p,
                      (ElemBox *)c.ecell_box.p);
    }
    BuildArgs A;
    A.xs = c.xs.p;
    A.nodex = c.nodex.p;
    A.ecenter = c.ecenter.p;
    A.eframe = c.eframe.p;
    A.acell_start = c.acell_start.p;
    A.acell_pos = c.acell_pos.p;
    A.acell_x = c.acell_fix.p;
    A.acell_y = A.acell_x + c.na;
    A.acell_z = A.acell_y + c.na;
    A.acell_of = c.acell_of.p;
    A.ecell_start = c.ecell_start.p;
    A.ecell_near = (c.nrep == 1 && c.ne) ? c.ecell_near.p : nullptr;
    A.acell_near = (c.nrep == 1 && c.na && c.ne) ? c.acell_near.p : nullptr;
    A.ecell_elems = c.ecell_elems.p;
    A.ecell_box = (const ElemBox *)c.ecell_box.p;
    A.atom_of_slot = c.slot_atom.p;
    A.site_flag = c.site_flag.p;
    if (c.ne) CACB200_CUDA(cudaMemsetAsync(c.site_flag.p, 0, (size_t)c.ne * MARKS, c.stream));
    A.na = c.na;
    A.ne = c.ne;
    A.nsi = nsi;
    A.cap = c.cap;
    A.rb = c.rbins;
    A.cutneigh = c.cutneigh;
    A.cutneighsq = c.cutneighsq;
    A.cutforcesq = (c.pp.cut + c.inner_margin) * (c.pp.cut + c.inner_margin);
    A.want_half = want_half ? 1 : 0;
    A.wide = 0;
    for (const Rep &R : c.rep_h)
      for (int d = 0; d < 3; d++)
        if (R.ag.inv[d] * WIDE_CELL < 1.0) A.wide = 1;
    A.nbr_full = c.nbr_full.p;
    A.num_in = c.num_in.p;
    A.site_from = c.site_from.p;
    A.raw_sites = c.raw_sites.p;
    A.num_full = c.num_full.p;
    A.raw_half = want_half ? c.raw_half.p : nullptr;
    A.num_half = want_half ? c.num_half.p : nullptr;
    A.img_half = want_half ? c.img_half.p : nullptr;
    A.overflow = c.overflow.p;
    // The atom-atom lists need no element work: they run on the context
    // stream while the side stream does phase A for every slot and then the
    // Gauss-point lists (disjoint slots); the atoms' element sites follow the
    // atom-atom lists once phase A is done.  Timed one kernel at a time when
    // profiling.
    const bool split = c.na && c.ne && !c.prof.enabled;
    cudaStream_t es = split ? c.side : c.stream;
    if (split) {
      CACB200_CUDA(cudaEventRecord(c.fork_ev, c.stream));
      CACB200_CUDA(cudaStreamWaitEvent(c.side, c.fork_ev, 0));
    }
    if (c.ne) {
      {
        KernelTimer t(c, "build_items");
        if (nsi < EIGHT_QUERY_SITES)
          k_elem_items<8><<<nblk(32L * (c.ne + nblk(c.na, 8)), 128), 128, 0, es>>>(
              A, P, c.items.p, c.nitems.p, c.item_cap, c.atom_work.p, c.atom_nwork.p);
        else
          k_elem_items<32><<<nblk(32L * (c.ne + nblk(c.na, 32)), 128), 128, 0, es>>>(
              A, P, c.items.p, c.nitems.p, c.item_cap, c.atom_work.p, c.atom_nwork.p);
      }
      if (split) CACB200_CUDA(cudaEventRecord(c.items_ev, c.side));
      {
        KernelTimer t(c, "build_gauss");
        k_build_gauss<<<nblk(32L * NG * c.ne, 128), 128, 0, es>>>(A, P, c.items.p, c.nitems.p, c.item_cap);
      }
      if (split) CACB200_CUDA(cudaEventRecord(c.join_ev, c.side));
    }
    if (c.na) {
      KernelTimer t(c, "build_atoms");
      const int nchunk = (c.na + 31) / 32;
      bool done = false;
      if (!want_half && nchunk < SMALL_CHUNKS * c.num_sms) {   // half lists are stored in order by one warp
        k_build_atoms<4><<<nchunk, 128, 0, c.stream>>>(A, P);
        done = true;
      }
      if constexpr (std::is_same_v<decltype(P), OneRep>) {
        if (!done && c.work_queue) {
          static const int per_sm = [] {
            int b = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_build_atoms_sm, 32, 0);
            return b > 0 ? b : 1;
          }();
          k_build_atoms_sm<<<per_sm * c.num_sms, 32, 0, c.stream>>>(A, P, nchunk, c.sm_counter.p, c.num_sms);
          done = true;
        }
      }
      if (!done) k_build_atoms<1><<<nchunk, 32, 0, c.stream>>>(A, P);
    }
    if (c.na && c.ne) {
      if (split) CACB200_CUDA(cudaStreamWaitEvent(c.stream, c.items_ev, 0));
      KernelTimer t(c, "build_atom_sites");
      // the warps stride over the work list: one wave of resident blocks
      static const int per_sm = [] {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_build_atom_sites<decltype(P)>, 128, 0);
        return b > 0 ? b : 1;
      }();
      const int grid = (int)std::min<long>(stride_grid(32L * c.na, 128), (long)per_sm * c.num_sms);
      k_build_atom_sites<<<grid, 128, 0, c.stream>>>(A, P, c.items.p, c.nitems.p, c.item_cap, c.atom_work.p,
                                                     c.atom_nwork.p);
    }
    if (split) CACB200_CUDA(cudaStreamWaitEvent(c.stream, c.join_ev, 0));
  });
  {
    KernelTimer t(c, "compact");
    if (c.ne) {
      k_act_table<<<nblk(c.ne, 8), 256, 0, c.stream>>>(c.site_flag.p, c.ne, nsi, c.site_words.p, c.act_gid.p,
                                                       c.dev_nact.p, c.overflow.p + 7);
      const int grid = (int)std::min<long>(nblk((long)NG * c.ne + c.na, 32), (long)8 * c.num_sms);
      // (a plain launch: blocks that wait for k_act_table's to end keep its
      // last ones out; 12 replicas 3.09 ms a run plainly, 3.17 ms so)
      k_remap_sites<<<grid, 256, 0, c.stream>>>(c.raw_sites.p, c.items.p, c.item_cap, c.num_full.p, c.num_in.p,
                                                c.site_from.p, nsi, c.cap, c.site_words.p, c.na, c.ne,
                                                c.atom_work.p, c.atom_nwork.p, c.nbr_full.p);
    }
    if (want_half)
      k_remap<<<nblk(nsi, 256), 256, 0, c.stream>>>(c.raw_half.p, c.img_half.p, c.num_half.p, nsi, c.cap,
                                                     c.site_words.p, c.atom_slot.p, c.na, c.ne, c.nbr_half.p);
  }
  c.have_half = want_half;
  c.lists_valid = true;
  c.nact_known = false;
  c.build_count++;
  CACB200_CUDA(cudaGetLastError());
}

// Read the rebuild's flag words (synchronises).  Returns 0 when the lists are
// good, 1 when a capacity must grow (the plan was updated: rebuild again).
int neigh_check(Ctx &c) {
  int ov[16];
  stream_copy(c, ov, c.overflow.p, sizeof(ov), cudaMemcpyDeviceToHost);
  if (ov[2]) throw Error(CACB200_EINVAL, "neighbour image beyond the first periodic image (box too small)");
  if (ov[6]) throw Error(CACB200_EUNSTABLE, "a site position is not finite or absurdly far from the box (unstable run)");
  if (ov[7]) throw Error(CACB200_EOVERFLOW, "more referenced sites than 26-bit list entries can address");
  int again = 0;
  if (ov[0]) {
    c.cap = ((ov[1] + 31) / 32) * 32;
    again = 1;
  }
  if (ov[3]) again = 1;   // an element outgrew the candidate grid
  if (ov[8]) {            // a query met more element boxes than its item slots
    c.item_cap = ((ov[9] + 15) / 16) * 16;
    again = 1;
  }
  if (again) {
    c.lists_valid = false;
    neigh_plan(c, c.plan_half);
  }
  return again;
}

// Synchronous rebuild with retries (API calls, setup, tests).
void neigh_build(Ctx &c, bool want_half) {
  c.check_system();
  if (!c.planned || c.plan_na != c.na || c.plan_ne != c.ne || (want_half && !c.plan_half))
    neigh_plan(c, want_half || c.plan_half);
  for (int attempt = 0; attempt < 4; attempt++) {
    neigh_build_async(c, want_half);
    if (!neigh_check(c)) {
      note_build_box(c);
      return;
    }
  }
  throw Error(CACB200_EOVERFLOW, "neighbour list capacity could not be settled");
}

int device_nact(Ctx &c) {
  if (!c.nact_known) {
    int n = 0;
    if (c.ne) stream_copy(c, &n, c.dev_nact.p, sizeof(int), cudaMemcpyDeviceToHost);
    c.nact = n;
    c.nact_known = true;
  }
  return c.nact;
}

void neigh_download(Ctx &c, bool half, int64_t *offset, int8_t *kind, int32_t *idx, int32_t *site,
                    int8_t *img, int64_t *nentries) {
  if (!c.lists_valid || (half && !c.have_half)) throw Error(CACB200_ESTATE, "list not built");
  const int nsi = c.nsite_i();
  std::vector<int> num_slot(nsi), num(nsi), slot_of(nsi), nin_slot(nsi, 0);
  std::vector<int> ent((size_t)c.cap * nsi);
  std::vector<int> atom_of(std::max(c.na, 1));
  device_nact(c);
  std::vector<int> act(std::max(c.nact, 1));
  CACB200_CUDA(cudaStreamSynchronize(c.stream));
  stream_copy(c, num_slot.data(), half ? c.num_half.p : c.num_full.p, sizeof(int) * nsi,
                          cudaMemcpyDeviceToHost);
  if (!half) stream_copy(c, nin_slot.data(), c.num_in.p, sizeof(int) * nsi, cudaMemcpyDeviceToHost);
  if (c.na) stream_copy(c, atom_of.data(), c.slot_atom.p, sizeof(int) * c.na, cudaMemcpyDeviceToHost);
  for (int k = 0; k < nsi; k++) slot_of[k] = k;
  for (int h = 0; h < c.na; h++) slot_of[atom_of[h]] = h;
  for (int i = 0; i < nsi; i++) num[i] = num_slot[slot_of[i]];
  stream_copy(c, ent.data(), half ? c.nbr_half.p : c.nbr_full.p, sizeof(int) * ent.size(),
                          cudaMemcpyDeviceToHost);
  if (c.nact)
    stream_copy(c, act.data(), c.act_gid.p, sizeof(int) * c.nact, cudaMemcpyDeviceToHost);
  int64_t total = 0;
  for (int i = 0; i < nsi; i++) total += num[i];
  *nentries = total;
  if (!offset) return;
  int64_t pos = 0;
  std::vector<std::tuple<int, int, int, int, int, int>> row;
  for (int i = 0; i < nsi; i++) {
    offset[i] = pos;
    row.clear();
    const int sl = slot_of[i], nin = half ? num[i] : nin_slot[sl];
    for (int k = 0; k < num[i]; k++) {
      // full lists: the front segment, then the back one from row cap - 1 down
      const int r = k < nin ? k : c.cap - 1 - (k - nin);
      int v = ent[(size_t)r * nsi + sl];
      int sidx = v >> IMG_BITS, code = v & ((1 << IMG_BITS) - 1);
      int sx, sy, sz;
      img_decode(code, sx, sy, sz);
      int kd, id, st;
      if (sidx < c.na) {   // atoms are stored by list slot
        kd = 0;
        id = atom_of[sidx];
        st = -1;
      } else if (sidx < c.na + NG * c.ne) {
        kd = 1;
        id = (sidx - c.na) / NG;
        st = gauss_site((sidx - c.na) % NG);
      } else {
        int gid = act[sidx - c.na - NG * c.ne];
        kd = 1;
        id = gid / NU;
        st = gid % NU;
      }
      row.emplace_back(kd, id, st, sx, sy, sz);
    }
    std::sort(row.begin(), row.end());
    for (auto &t : row) {
      kind[pos] = (int8_t)std::get<0>(t);
      idx[pos] = std::get<1>(t);
      site[pos] = std::get<2>(t);
      img[3 * pos] = (int8_t)std::get<3>(t);
      img[3 * pos + 1] = (int8_t)std::get<4>(t);
      img[3 * pos + 2] = (int8_t)std::get<5>(t);
      pos++;
    }
  }
  offset[nsi] = pos;
}

}  // namespace cacb200
