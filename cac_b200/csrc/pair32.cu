// Mixed-precision pair kernels: FP32 distances and force arithmetic on
// fixed-point positions, FP64 everywhere else.
//
// Every site of the site table gets, each step, a 32-bit fixed-point copy of
// its FP64 position relative to the box corner, q = rint((x - lo) 2^26) taken
// modulo 2^32.  A pair's separation is then
//     x_i - (x_j + s L) = (q_i - q_j - s Lq) 2^-26   (mod 2^32 quanta),
// an exact integer difference in wrap-around 32-bit arithmetic, which is the
// true difference whenever that is shorter than 2^31 quanta = 32 A (pairs are
// within the neighbour cutoff), rounded once to FP32: no FP32 sum ever
// carries a box-sized coordinate, and the quantum (1.5e-8 A) does not depend
// on the box size.  A site's record is 16 bytes, (qx, qy, qz, F'), so one
// 128-bit load brings everything a pair needs from its neighbour.
//
// What stays FP64 (as the mixed form specifies): positions and velocities and
// their integration, element interpolation, nodal assembly over Gauss points,
// and the global energy/virial reductions (per-block partials in FP64).
// Per-site sums of pair terms are FP32.  EAM terms are cubics in r^2 fitted to
// the FP64 splines where these are smooth (Eam32), else FP32 copies of the
// splines' coefficients.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctx.cuh"
#include "device.cuh"

namespace cacb200 {

namespace {

inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

// Fixed-point frame of a single system; batches read each replica's from its
// descriptor.
struct FixGrid {
  double lo[3];
  double scale[3];
  int Lq[3];
  const Rep *reps;          // batches (null for one system)
  const int *site_rep;      // [nsite_i]
  const int *elem_rep;      // [ne]
  const int *act_gid;       // active lattice sites -> element * 729 + site
  const int *slot_atom;     // list slot -> atom
  int na, nsi;
};

// Fixed-point record of pair-table entry k at FP64 position (px, py, pz),
// in the frame of its replica; w (F') is written later in the step.
__device__ __forceinline__ void pack_pos(double px, double py, double pz, int k, const FixGrid &G, int4 *pos,
                                         int *bad) {
  double q[3] = {px, py, pz};
  double lo[3] = {G.lo[0], G.lo[1], G.lo[2]};
  double sc[3] = {G.scale[0], G.scale[1], G.scale[2]};
  if (G.reps) {
    int r = k < G.na ? G.site_rep[G.slot_atom[k]]
                     : (k < G.nsi ? G.site_rep[k] : G.elem_rep[G.act_gid[k - G.nsi] / NU]);
    const Rep *R = G.reps + r;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = R->b.lo[d];
      sc[d] = R->qscale[d];
    }
  }
  int o[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double rel = (q[d] - lo[d]) * sc[d];
    // positions further than 2^62 quanta (~7e10 A) from the box, or not
    // finite, only come from a run that has blown up
    if (!(rel > -4.6e18 && rel < 4.6e18)) {
      atomicExch(bad, 1);
      rel = 0.0;
    }
    o[d] = (int)(unsigned)(unsigned long long)__double2ll_rn(rel);   // modulo 2^32
  }
  pos[k] = make_int4(o[0], o[1], o[2], 0);
}

// The mixed form's pair table in one pass: the slot-ordered atoms, the Gauss
// points and the interpolated active lattice sites (the positions of
// k_pair_table, integrate.cu, in the same FP64 operations) written straight
// as fixed-point records, with no FP64 copy in between.
__global__ void k_pair_table32(const double4 *xs, const int *slot_atom, const double *nodex, int na, int ne,
                               const int *act_gid, const int *nact_dev, FixGrid G, int4 *pos, int *bad) {
  behind_previous();
  const int ngp = NG * ne;
  const int n = na + ngp + *nact_dev;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    if (t < na) {
      const double4 p = xs[slot_atom[t]];
      pack_pos(p.x, p.y, p.z, t, G, pos, bad);
      continue;
    }
    const int s = t - na;
    if (s < ngp) {
      const int e = s / NG, g = s % NG;
      const double *nx = nodex + (size_t)e * 24 + 3 * gauss_node(g);
      pack_pos(nx[0], nx[1], nx[2], t, G, pos, bad);
      continue;
    }
    const int gid = act_gid[s - ngp];
    const int e = gid / NU, u = gid % NU;
    const double *nx = nodex + (size_t)e * 24;
    double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll
    for (int m = 0; m < NPE; m++) {
      const double N = shape_val(u, m);
      x += N * nx[3 * m];
      y += N * nx[3 * m + 1];
      z += N * nx[3 * m + 2];
    }
    pack_pos(x, y, z, t, G, pos, bad);
  }
}

// Positions are in quanta of 2^-26 A in every replica; separations stay in
// quanta through the pair arithmetic (scaling by a power of two is exact) and
// the sums are scaled once per site.
constexpr float QUANTUM = 1.0f / 67108864.0f;

struct Args32 {
  const int4 *pos;
  const int *nbr;          // lists and counts indexed by list slot
  const int *num;
  const int *num_in;                // inner prefix length of each list ...
  PrefixRule prefix;                // ... and the rule for walking the rest
  const int *slot_atom;    // list slot -> atom (slots past the atoms are Gauss points)
  int na, ne, nsi;
  int cap;                 // list rows: the rest of a list fills its last rows
  FixGrid G;
  double *f, *gaussf;
  double *eatom, *vatom, *enode, *vnode;
  double *partial;
  int eflag, vflag;
  double escale_node, vscale_node;
};

__device__ __forceinline__ int site_of_slot(const Args32 &A, int t) { return t < A.na ? A.slot_atom[t] : t; }

// Walks n entries of a list: each lane takes four at a time, the next four
// entries loaded ahead and the four records issued back to back before any is
// used.  Entries past the end are walked as pairs too far apart to count.
// f(partial, dx, dy, dz, rsq, w): the separation from the neighbour and its
// square, in quanta; w = F' of the neighbour.
template <int G, class F>
__device__ __forceinline__ void walk32(const Args32 &A, int t, int i, const int4 &oi, const int *nb, int n, F &&f) {
  const size_t step = (size_t)G * A.nsi;
  const int *p = nb + (size_t)(threadIdx.x % G) * A.nsi;
  int v[4];
  auto load = [&](int left) {   // entries this lane still has
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = u < left ? __ldcs(p + u * step) : (t << IMG_BITS) | IMG_ZERO;
    p += 4 * step;
  };
  int left = (n - (int)(threadIdx.x % G) + G - 1) / G;
  load(left);
  for (; left > 0; left -= 4) {
    int4 o[4];
#pragma unroll
    for (int u = 0; u < 4; u++) o[u] = A.pos[v[u] >> IMG_BITS];
    // images: shift the neighbour by s L, s in {-1, 0, 1}, modulo 2^32
    if (((v[0] ^ IMG_ZERO) | (v[1] ^ IMG_ZERO) | (v[2] ^ IMG_ZERO) | (v[3] ^ IMG_ZERO)) & ((1 << IMG_BITS) - 1)) {
      const int *Lq = A.G.reps ? A.G.reps[A.G.site_rep[i]].Lq : A.G.Lq;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        int sx, sy, sz;
        img_decode(v[u] & ((1 << IMG_BITS) - 1), sx, sy, sz);
        o[u].x += sx * Lq[0];
        o[u].y += sy * Lq[1];
        o[u].z += sz * Lq[2];
      }
    }
    const int now = left;
    load(left - 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const float dx = (float)(int)((unsigned)oi.x - (unsigned)o[u].x), dy = (float)(int)((unsigned)oi.y - (unsigned)o[u].y),
                  dz = (float)(int)((unsigned)oi.z - (unsigned)o[u].z);
      float rsq = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
      if (u && u >= now) rsq = 1e30f;
      f(u % (4 / G), dx, dy, dz, rsq, __int_as_float(o[u].w));
    }
  }
}

// A site's list: the inner prefix on its own, then the rest unless the
// prefix still holds every pair of the site inside the cutoff (walk_rest,
// device.cuh; an entry's partial depends on its place in a walk, so the
// prefix is always walked alone).
template <int G, class F>
__device__ __forceinline__ void for_each32(const Args32 &A, int t, int i, const int4 &oi, F &&f) {
  const int n_in = A.num_in[t], n = A.num[t];
  const int *nb = A.nbr + t;
  const bool rest = n > n_in && walk_rest(A.prefix, i, A.G.reps ? A.G.site_rep[i] : 0);
#pragma unroll 1
  for (int seg = 0; seg < (rest ? 2 : 1); seg++)
    walk32<G>(A, t, i, oi, seg ? nb + (size_t)(A.cap - (n - n_in)) * A.nsi : nb, seg ? n - n_in : n_in, f);
}

// Writes force (and per-site energy / virial) of i-site i and adds its global
// energy / virial to red.
template <bool EV>
__device__ __forceinline__ void finish32(const Args32 &A, int i, const float fi[3], float esum, const float vsum[6],
                                         double eextra_site, double eextra_global, double red[7]) {
  const bool atom = i < A.na;
  int e = 0, g = 0, node = 0;
  double *fo;
  if (atom) {
    fo = A.f + 3 * (size_t)i;
  } else {
    e = (i - A.na) / NG;
    g = (i - A.na) % NG;
    node = gauss_node(g);
    fo = A.gaussf + (size_t)e * 24 + 3 * g;
  }
  fo[0] = fi[0];
  fo[1] = fi[1];
  fo[2] = fi[2];
  if (EV) {
    const double es = atom ? 0.5 : A.escale_node, vs = atom ? 0.5 : A.vscale_node;
    if (A.eflag & CACB200_ENERGY_GLOBAL) red[0] += es * (double)esum + eextra_global;
    if (A.vflag & CACB200_VIRIAL_GLOBAL)
#pragma unroll
      for (int k = 0; k < 6; k++) red[1 + k] += vs * (double)vsum[k];
    if (A.eflag & CACB200_ENERGY_ATOM) {
      const double v = 0.5 * (double)esum + eextra_site;
      if (atom) A.eatom[i] = v;
      else A.enode[(size_t)e * 8 + node] = v;
    }
    if (A.vflag & CACB200_VIRIAL_ATOM) {
      double *vo = atom ? A.vatom + 6 * (size_t)i : A.vnode + 48 * (size_t)e + 6 * node;
#pragma unroll
      for (int k = 0; k < 6; k++) vo[k] = 0.5 * (double)vsum[k];
    }
  }
}

// Per-site sums of a force pass.
template <int G, bool EV>
struct ForceSums {
  Sum4<float, G> f[3], e[1], v[EV ? 6 : 1];
  __device__ __forceinline__ void add(int part, float dx, float dy, float dz, float fpair) {
    f[0].a[part] = __fmaf_rn(dx, fpair, f[0].a[part]);
    f[1].a[part] = __fmaf_rn(dy, fpair, f[1].a[part]);
    f[2].a[part] = __fmaf_rn(dz, fpair, f[2].a[part]);
  }
  __device__ __forceinline__ void add_ev(int part, float dx, float dy, float dz, float fpair, float phi) {
    e[0].a[part] = __fadd_rn(e[0].a[part], phi);
    const float a[6] = {dx * dx, dy * dy, dz * dz, dx * dy, dx * dz, dy * dz};
#pragma unroll
    for (int k = 0; k < 6; k++) v[k].a[part] = __fmaf_rn(a[k], fpair, v[k].a[part]);
  }
  // totals in A, eV; fscale: of separation times fpair, the force's unit
  __device__ __forceinline__ void totals(float fscale, float fi[3], float &esum, float vsum[6]) const {
#pragma unroll
    for (int d = 0; d < 3; d++) fi[d] = f[d].total() * fscale;
    if constexpr (EV) {
      esum = e[0].total();
#pragma unroll
      for (int k = 0; k < 6; k++) vsum[k] = v[k].total() * (fscale * QUANTUM);
    }
  }
};

// ---------------------------------------------------------------------- LJ

struct Lj32 {
  float cutsq, lj1, lj2, lj3, lj4, offset;
};

// The LJ pass takes one lane a site, with one running sum per component in the
// order of the list and separations in A, and leaves the contraction of the
// pair's expressions to the compiler.  In a crystal at rest the forces are what
// the rounding of these sums leaves, and a relaxation carries it on: with four
// lanes and four partial sums a site, which took 27.6 us at 84 k sites, the node
// forces after 18 iterations from 0 K were off by 7e-5 from those of this
// order, as far as either is from 64 bits.  Entries are loaded ahead of
// their use: 34.4 -> 32.9 us at 84 k sites, 191 -> 179 at 0.78 M, 531 -> 503 at
// 2.3 M (eight entries at a time instead of four: 34.6 at 84 k).
__device__ __forceinline__ void sep_lj(const Args32 &A, const int Lq[3], const int4 &oi, int v, float &dx, float &dy,
                                       float &dz) {
  const int code = v & ((1 << IMG_BITS) - 1);
  const int4 oj = A.pos[v >> IMG_BITS];
  int s[3] = {0, 0, 0};
  if (code != IMG_ZERO) img_decode(code, s[0], s[1], s[2]);
  // s in {-1, 0, 1}, modulo 2^32
  dx = (float)(int)((unsigned)oi.x - (unsigned)oj.x - (unsigned)s[0] * (unsigned)Lq[0]) * QUANTUM;
  dy = (float)(int)((unsigned)oi.y - (unsigned)oj.y - (unsigned)s[1] * (unsigned)Lq[1]) * QUANTUM;
  dz = (float)(int)((unsigned)oi.z - (unsigned)oj.z - (unsigned)s[2] * (unsigned)Lq[2]) * QUANTUM;
}

// Four entries at a time, the next four loaded ahead and the records issued
// back to back before any is used.
template <class F>
__device__ __forceinline__ void walk_lj(const Args32 &A, int t, const int Lq[3], const int4 &oi, const int *nb, int n,
                                        F &&f) {
  int v[4];
  auto load = [&](int left) {
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = u < left ? __ldcs(nb + (size_t)u * A.nsi) : (t << IMG_BITS) | IMG_ZERO;
    nb += (size_t)4 * A.nsi;
  };
  load(n);
  for (int left = n; left > 0; left -= 4) {
    float d[4][3];
#pragma unroll
    for (int u = 0; u < 4; u++) sep_lj(A, Lq, oi, v[u], d[u][0], d[u][1], d[u][2]);
    load(left - 4);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (u < left) f(d[u][0], d[u][1], d[u][2]);
  }
}

template <bool EV>
__global__ void __launch_bounds__(128, EV ? 4 : 8) k_lj32(Args32 A, Lj32 P) {
  behind_previous();
  double red[7] = {0, 0, 0, 0, 0, 0, 0};
  const int t = blockIdx.x * blockDim.x + threadIdx.x;   // list slot
  if (t < A.nsi) {
    const int i = site_of_slot(A, t);           // site-table index
    float fi[3] = {0, 0, 0}, esum = 0.f, vsum[6] = {0, 0, 0, 0, 0, 0};
    const int4 oi = A.pos[t];
    const int rep = A.G.reps ? A.G.site_rep[i] : 0;
    int Lq[3];
#pragma unroll
    for (int d = 0; d < 3; d++) Lq[d] = A.G.reps ? A.G.reps[rep].Lq[d] : A.G.Lq[d];
    const int n_in = A.num_in[t], n = A.num[t];
    const int *nb = A.nbr + t;
    const bool rest = n > n_in && walk_rest(A.prefix, i, rep);
#pragma unroll 1
    for (int seg = 0; seg < (rest ? 2 : 1); seg++)
      walk_lj(A, t, Lq, oi, seg ? nb + (size_t)(A.cap - (n - n_in)) * A.nsi : nb, seg ? n - n_in : n_in,
              [&](float dx, float dy, float dz) {
                float rsq = dx * dx + dy * dy + dz * dz;
                if (rsq < P.cutsq) {
                  float r2inv = 1.0f / rsq;
                  float r6inv = r2inv * r2inv * r2inv;
                  float fpair = r6inv * (P.lj1 * r6inv - P.lj2) * r2inv;
                  fi[0] += dx * fpair;
                  fi[1] += dy * fpair;
                  fi[2] += dz * fpair;
                  if (EV) {
                    esum += r6inv * (P.lj3 * r6inv - P.lj4) - P.offset;
                    vsum[0] += dx * dx * fpair;
                    vsum[1] += dy * dy * fpair;
                    vsum[2] += dz * dz * fpair;
                    vsum[3] += dx * dy * fpair;
                    vsum[4] += dx * dz * fpair;
                    vsum[5] += dy * dz * fpair;
                  }
                }
              });
    finish32<EV>(A, i, fi, esum, vsum, 0.0, 0.0, red);
  }
  if (EV) block_reduce_store<7>(red, A.partial);
}

// --------------------------------------------------------------------- EAM

// rz: per r-knot m the rhor value coefficients at [2m] and the z2r ones at
// [2m+1], one 32-byte record; derivatives as in the FP64 kernels.
//
// Beside them the smooth part of the same splines as functions of s = r^2,
// which a pair needs no square root for: the density rho, and the two terms
// of the force over r, rho'/r and phi'/r, and for tallies phi, each a cubic in s
// on intervals of equal width (eam_fast_tables: fitted to the splines to 2e-8 of
// their local size, a third of an FP32 rounding, and phi to 4e-8, or not used).  Their records, 16 bytes
// per function, cover the intervals [lo, lo + cnt) and are few enough to be
// held in shared memory `copies` times over, lane l reading copy l % copies:
// with eight copies a warp's gather has no bank conflict, and L1 keeps the
// site records.  Pairs beyond the cutoff read a record of zeros, so no branch
// parts them from the others; pairs inside it but outside the intervals (too
// close, or within the last knots of the splines) take the splines themselves.
// The passes are bound by the L1 data pipe (ncu: 80 and 86 % of its peak while
// active; a gather of 32 site records takes about 13 of its cycles, a 16-byte
// spline record from global memory as many, from eight copies in shared memory
// four; with four copies the force pass is 17 % slower).  4.98 M sites: density
// 1.047 -> 0.73 ms, force 1.170 -> 0.88 ms; 313 k: 91 -> 60 and 96 -> 70 us.
// Other tables, 1.21 M sites: 7 A cutoff (482 records) density 647 -> 434 us, force
// 723 -> 603; without a fit (1,000 knots, 5.5 A; this launch shape with the
// splines from memory) 335 -> 286 and 376 -> 351.
// With tallies: 313 k sites 123 -> 96 us, 1.21 M 417 -> 310 us (133 and 489 us
// where phi was read from the splines beside the records).
constexpr int FAST_INTERVALS[] = {192, 256, 384, 512}, FAST_COPIES = 8;
constexpr size_t FAST_BYTES = sizeof(float4) * (512 + 1) * FAST_COPIES;   // the most that one function takes
struct Eam32 {
  const float4 *rz, *frho_val, *frho_der;
  float rdr, rdrho, rhomax, cutforcesq;      // cutforcesq in square quanta
  int nr, nrho;
  const float4 *fast;                        // [4][cnt + 1]: rho, rho'/r, phi'/r, phi
  float inv_ds;                              // intervals per square quantum
  int base, cnt, copies;                     // base: bits of 2^23 + the first interval
};

// The record of s = rsq among the fast ones and the place p in its interval;
// the last record, T.cnt, holds zeros: any s outside the intervals.
// floor(rsq * inv_ds) + 2^23 is formed in one rounded operation, exactly.
__device__ __forceinline__ unsigned fast_interval(const Eam32 &T, float rsq, float &p) {
  const float x = __fmaf_rd(rsq, T.inv_ds, 8388608.0f);
  p = __fmaf_rn(rsq, T.inv_ds, 8388608.0f - x);
  return min((unsigned)(__float_as_int(x) - T.base), (unsigned)T.cnt);
}

// n functions' records into the block's shared memory, `copies` times.
__device__ __forceinline__ void load_fast(const Eam32 &T, const float4 *from, int n, float4 *tab) {
  for (int k = threadIdx.x; k < n * (T.cnt + 1) * T.copies; k += blockDim.x) tab[k] = __ldg(from + k / T.copies);
  __syncthreads();
}

__device__ __forceinline__ float cubic(const float4 &c, float p) {
  return __fmaf_rn(__fmaf_rn(__fmaf_rn(c.x, p, c.y), p, c.z), p, c.w);
}

__device__ __forceinline__ float fp32_of(const Eam32 &T, float rho, float *phi) {
  float p = rho * T.rdrho + 1.0f;
  int m = (int)p;
  m = max(1, min(m, T.nrho - 1));
  p -= (float)m;
  p = fminf(p, 1.0f);
  float4 d = T.frho_der[m];
  float fp = (d.x * p + d.y) * p + d.z;
  if (phi) {
    float4 v = T.frho_val[m];
    float e = ((v.x * p + v.y) * p + v.z) * p + v.w;
    if (rho > T.rhomax) e += fp * (rho - T.rhomax);
    *phi = e;
  }
  return fp;
}

// The knot of distance r and the place in its interval.
__device__ __forceinline__ int r_knot(const Eam32 &T, float r, float &p) {
  p = __fmaf_rn(r, T.rdr, 1.0f);
  int m = (int)p;
  m = max(1, min(m, T.nr - 1));
  p = fminf(__fadd_rn(p, -(float)m), 1.0f);
  return m;
}

// rho'/r and phi'/r from the splines, and phi itself.
__device__ __forceinline__ void spline_force(const Eam32 &T, float rsq, float &g, float &h, float &phi) {
  const float s = __fmul_rn(rsq, QUANTUM * QUANTUM);
  const float recip = rsqrtf(s), r = __fmul_rn(s, recip);
  float p;
  const int m = r_knot(T, r, p);
  float4 rv, zv;
  ldg256(T.rz + 2 * m, rv, zv);
  const float rhop = __fmul_rn(__fmaf_rn(__fmaf_rn(3.0f * rv.x, p, 2.0f * rv.y), p, rv.z), T.rdr);
  const float z2p = __fmul_rn(__fmaf_rn(__fmaf_rn(3.0f * zv.x, p, 2.0f * zv.y), p, zv.z), T.rdr);
  phi = __fmul_rn(cubic(zv, p), recip);
  g = __fmul_rn(rhop, recip);
  h = __fmul_rn(__fmaf_rn(z2p, recip, -__fmul_rn(phi, recip)), recip);
}

// Density pass: rho at each i-site, then F' into its record (and F into
// phi_site for energies).
template <int G, bool FAST>
__global__ void __launch_bounds__(512, 2) k_eam_rho32(Args32 A, Eam32 T, double *rho_out, double *phi_site,
                                                      int4 *pos_w) {
  extern __shared__ float4 tab[];
  if (FAST) load_fast(T, T.fast, 1, tab);   // (constants: loaded while the kernel before ends)
  behind_previous();
  const float4 *mine = tab + threadIdx.x % T.copies;
  for_each_slot<G>(A.nsi, [&](int t, bool valid) {
    const int i = valid ? site_of_slot(A, t) : 0;           // site-table index
    Sum4<float, G> sum;
    if (valid) {
      const int4 oi = A.pos[t];
      for_each32<G>(A, t, i, oi, [&](int part, float, float, float, float rsq, float) {
        float p, v = 0.0f;
        bool spline = rsq < T.cutforcesq;
        if (FAST) {
          const unsigned m = fast_interval(T, rsq, p);
          v = cubic(mine[m * T.copies], p);
          spline = spline && m == T.cnt;
        }
        if (spline) {
          const int k = r_knot(T, __fsqrt_rn(__fmul_rn(rsq, QUANTUM * QUANTUM)), p);
          v = cubic(__ldg(T.rz + 2 * k), p);
        }
        sum.a[part] = __fadd_rn(sum.a[part], v);
      });
    }
    const float rho = sum.total();
    if (!valid || threadIdx.x % G) return;
    int slot = i;
    if (i >= A.na) {
      int e = (i - A.na) / NG, g = (i - A.na) % NG;
      slot = A.na + 8 * e + gauss_node(g);
    }
    rho_out[slot] = rho;
    float phi = 0.f;
    const float fp = fp32_of(T, rho, A.eflag ? &phi : nullptr);
    pos_w[t].w = __float_as_int(fp);
    if (A.eflag) phi_site[i] = phi;
  });
}

__global__ void k_eam_site_fp32(int4 *pos, const int *act_gid, const int *nact_dev, int base, int na,
                                const double *rho, Eam32 T) {
  behind_previous();
  const int nact = *nact_dev;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nact; k += gridDim.x * blockDim.x) {
    int gid = act_gid[k];
    int e = gid / NU, u = gid % NU;
    const double *rn = rho + na + 8 * (size_t)e;
    double r = 0.0;
#pragma unroll
    for (int n = 0; n < NPE; n++) r += shape_val(u, n) * rn[n];
    pos[base + k].w = __float_as_int(fp32_of(T, (float)r, nullptr));
  }
}

// Force pass.  A pair's force is -((F'_i + F'_j) rho'/r + phi'/r) d.
template <int G, bool FAST, bool EV>
__global__ void __launch_bounds__(512, EV ? 1 : 2) k_eam_force32(Args32 A, Eam32 T, const double *phi_site) {
  extern __shared__ float4 tab[];
  if (FAST) load_fast(T, T.fast + T.cnt + 1, EV ? 3 : 2, tab);
  behind_previous();
  const float4 *mine = tab + threadIdx.x % T.copies;
  const int second = (T.cnt + 1) * T.copies;
  double red[7] = {0, 0, 0, 0, 0, 0, 0};
  for_each_slot<G>(A.nsi, [&](int t, bool valid) {
    const int i = valid ? site_of_slot(A, t) : 0;           // site-table index
    ForceSums<G, EV> S;
    if (valid) {
      const int4 oi = A.pos[t];
      const float fpi = __int_as_float(oi.w);
      for_each32<G>(A, t, i, oi, [&](int part, float dx, float dy, float dz, float rsq, float fpj) {
        float p, g = 0.0f, h = 0.0f, phi = 0.0f;
        bool spline = rsq < T.cutforcesq;
        if (FAST) {
          const unsigned m = fast_interval(T, rsq, p);
          g = cubic(mine[m * T.copies], p);
          h = cubic(mine[m * T.copies + second], p);
          if (EV) phi = cubic(mine[m * T.copies + 2 * second], p);
          spline = spline && m == T.cnt;
        }
        if (spline) spline_force(T, rsq, g, h, phi);
        const float pull = __fmaf_rn(__fadd_rn(fpi, fpj), g, h);
        S.add(part, dx, dy, dz, pull);
        if (EV) S.add_ev(part, dx, dy, dz, pull, phi);
      });
    }
    float fi[3], esum = 0.0f, vsum[6];
    S.totals(-QUANTUM, fi, esum, vsum);
    if (!valid || threadIdx.x % G) return;
    double eemb_site = 0.0, eemb_global = 0.0;
    if (EV && A.eflag) {
      eemb_site = phi_site[i];
      eemb_global = i < A.na ? eemb_site : eemb_site * A.escale_node * 2.0;
    }
    finish32<EV>(A, i, fi, esum, vsum, eemb_site, eemb_global, red);
  });
  if (EV) block_reduce_store<7>(red, A.partial);
}

__global__ void k_reduce_partials32(const double *partial, int nblocks, double *out) {
  int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k >= 7) return;
  double s = 0.0;
  for (int b = lane; b < nblocks; b += 32) s += partial[b * 7 + k];
  s = warp_sum(s);
  if (lane == 0) out[k] = s;
}

FixGrid make_fix_grid(const Ctx &c) {
  FixGrid G;
  const Rep &r0 = c.rep_h[0];
  for (int d = 0; d < 3; d++) {
    G.lo[d] = r0.b.lo[d];
    G.scale[d] = r0.qscale[d];
    G.Lq[d] = r0.Lq[d];
  }
  G.reps = c.nrep > 1 ? c.rep_d.p : nullptr;
  G.site_rep = c.site_rep.p;
  G.elem_rep = c.elem_rep.p;
  G.act_gid = c.act_gid.p;
  G.slot_atom = c.slot_atom.p;
  G.na = c.na;
  G.nsi = c.nsite_i();
  return G;
}

// The splines as the host evaluates them: value and derivative at r.
struct HostSpline {
  const std::vector<double4> &rz;
  int which, nr;
  double rdr;
  void at(double r, double &v, double &d) const {
    double p = r * rdr + 1.0;
    const int m = std::max(1, std::min((int)p, nr - 1));
    p = std::min(p - m, 1.0);
    const double4 c = rz[2 * (size_t)m + which];
    v = ((c.x * p + c.y) * p + c.z) * p + c.w;
    d = ((3.0 * c.x * p + 2.0 * c.y) * p + c.z) * rdr;
  }
};

// i-sites from which a site takes one lane, and two: below, one lane per site
// leaves too few warps to hide the gathers' latency; above, more lanes per
// site read more list rows per load.  Density pass in us with 1 / 2 / 4 lanes
// (measured before the fast records, which shifted all alike): 6 k sites
// 29 / 19 / 15, 84 k 33 / 33 / 31, 313 k 91 / 83 / 88, 1.21 M 268 / 275 / 311.
constexpr int ONE_LANE_SITES = 600000, TWO_LANE_SITES = 100000;

// The functions of s = r^2 that the passes need (three for the forces, and
// phi for tallies), as cubics on n equal intervals of [0, top^2], each the
// interpolant at the interval's four Chebyshev nodes.  An interval is good when
// every function's cubic stays within 2e-8 (phi: 4e-8) of the spline, relative
// to its largest value within 0.5 A.  Returns the first interval from which all
// are good (n: none).
int fit_fast(const HostSpline &rho, const HostSpline &z, double top, int n, float &inv_ds, std::vector<float4> rec[4]) {
  // pairs at the top or beyond fall past the last interval
  inv_ds = (float)((double)n / (double)(float)(top * top));
  while ((double)inv_ds * (double)(float)(top * top) < n) inv_ds = std::nextafter(inv_ds, 1e30f);
  const double ds = 1.0 / (double)inv_ds;
  auto eval = [&](double s, double out[4]) {
    const double r = std::sqrt(s);
    double dr, zv, dz;
    rho.at(r, out[0], dr);
    z.at(r, zv, dz);
    out[1] = dr / r;
    out[2] = (dz - zv / r) / s;
    out[3] = zv / r;
  };
  double node[4], inv[4][4];
  for (int k = 0; k < 4; k++) node[k] = 0.5 - 0.5 * std::cos((2 * k + 1) * 3.14159265358979323846 / 8.0);
  // Lagrange basis polynomials' coefficients
  for (int k = 0; k < 4; k++) {
    double c[4] = {1, 0, 0, 0};
    int deg = 0;
    for (int j = 0; j < 4; j++) {
      if (j == k) continue;
      const double q = 1.0 / (node[k] - node[j]);
      double e[4] = {0, 0, 0, 0};
      for (int d = 0; d <= deg; d++) {
        e[d + 1] += c[d] * q;
        e[d] -= c[d] * node[j] * q;
      }
      deg++;
      std::copy(e, e + 4, c);
    }
    std::copy(c, c + 4, inv[k]);
  }
  constexpr int TEST = 12;
  std::vector<double> err[4], val[4], mid(n);
  for (int q = 0; q < 4; q++) {
    rec[q].resize(n);
    err[q].assign(n, 0.0);
    val[q].assign(n, 0.0);
  }
  for (int m = 0; m < n; m++) {
    mid[m] = std::sqrt((m + 0.5) * ds);
    double c[4][4] = {};
    for (int k = 0; k < 4; k++) {
      double v[4];
      eval((m + node[k]) * ds, v);
      for (int q = 0; q < 4; q++)
        for (int d = 0; d < 4; d++) c[q][d] += v[q] * inv[k][d];
    }
    for (int u = 0; u <= TEST; u++) {
      const double p = (double)u / TEST;
      double v[4];
      eval(std::max((m + p) * ds, 1e-6 * ds), v);
      for (int q = 0; q < 4; q++) {
        const double a = ((c[q][3] * p + c[q][2]) * p + c[q][1]) * p + c[q][0];
        err[q][m] = std::max(err[q][m], std::fabs(a - v[q]));
        val[q][m] = std::max(val[q][m], std::fabs(v[q]));
      }
    }
    for (int q = 0; q < 4; q++)
      rec[q][m] = make_float4((float)c[q][3], (float)c[q][2], (float)c[q][1], (float)c[q][0]);
  }
  for (int m = n - 1; m >= 0; m--)
    for (int q = 0; q < 4; q++) {
      double size = 0.0;
      for (int j = m; j >= 0 && mid[m] - mid[j] <= 0.5; j--) size = std::max(size, val[q][j]);
      for (int j = m; j < n && mid[j] - mid[m] <= 0.5; j++) size = std::max(size, val[q][j]);
      if (!(err[q][m] <= (q < 3 ? 2e-8 : 4e-8) * size)) return m + 1;
    }
  return 0;
}

// Fast records of the context's splines: the fewest intervals that are good
// from 0.4 of the cutoff on (closer pairs are rare), up to the cutoff or, as
// the splines' slopes at the last knots are cruder, up to four knots before
// it.  Tables that no fit follows (noisy ones) have none.
void eam_fast_tables(Ctx &c, const std::vector<double4> &rz) {
  c.fast_cnt = 0;
  const HostSpline rho{rz, 0, c.pp.nr, c.pp.rdr}, z{rz, 1, c.pp.nr, c.pp.rdr};
  std::vector<float4> rec[4];
  for (int n : FAST_INTERVALS)
    for (double top : {c.pp.cut, c.pp.cut - 4.0 * c.pp.dr}) {
      if (!(top > 0.5 * c.pp.cut)) continue;
      float inv_ds;
      const int lo = fit_fast(rho, z, top, n, inv_ds, rec);
      if (!(std::sqrt(lo / (double)inv_ds) <= 0.4 * c.pp.cut)) continue;
      c.fast_lo = lo;
      c.fast_cnt = n - lo;
      c.fast_inv_ds = inv_ds;
      std::vector<float4> out;
      for (int q = 0; q < 4; q++) {
        out.insert(out.end(), rec[q].begin() + lo, rec[q].end());
        out.push_back(make_float4(0.0f, 0.0f, 0.0f, 0.0f));
      }
      c.fast32.reserve(out.size());
      stream_copy(c, c.fast32.p, out.data(), sizeof(float4) * out.size(), cudaMemcpyHostToDevice);
      return;
    }
}

// The limit on a kernel's shared memory belongs to the kernel on the device,
// which every context of the process launches: it is the most that any table
// can need, so no context lowers what another is about to launch with.
void allow_fast_records() {
  auto one = [](auto kernel, size_t bytes) {
    CACB200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  };
  auto allow = [&](size_t bytes, auto... kernels) { (one(kernels, bytes), ...); };
  allow(FAST_BYTES, k_eam_rho32<1, true>, k_eam_rho32<2, true>, k_eam_rho32<4, true>);
  allow(2 * FAST_BYTES, k_eam_force32<1, true, false>, k_eam_force32<2, true, false>, k_eam_force32<4, true, false>);
  allow(3 * FAST_BYTES, k_eam_force32<1, true, true>, k_eam_force32<2, true, true>, k_eam_force32<4, true, true>);
}

}  // namespace

void pair_table_mixed(Ctx &c) {
  const long ns = (long)c.nsite_i() + (long)c.ne * NU;   // capacity: every lattice site active
  c.pos32.reserve(std::max(ns, 1L));
  c.overflow.reserve(16);
  FixGrid G = make_fix_grid(c);
  // 64 blocks per SM: the item loop's loads are in flight across more
  // threads than stride_grid's 16 blocks give (0.193 -> 0.181 ms on config 3)
  launch_behind(c, std::min(nblk(ns, 256), 148 * 64), 256, 0, k_pair_table32, c.xs.p, c.slot_atom.p, c.nodex.p,
                c.na, c.ne, c.act_gid.p, c.dev_nact.p, G, c.pos32.p, c.overflow.p + 6);
}

void mixed_tables(Ctx &c) {
  auto conv = [&](DBuf<double4> &src, DBuf<float4> &dst, int n) {
    std::vector<double4> h(n + 1);
    stream_copy(c, h.data(), src.p, sizeof(double4) * (n + 1), cudaMemcpyDeviceToHost);
    std::vector<float4> g(n + 1);
    for (int m = 0; m <= n; m++) g[m] = make_float4((float)h[m].x, (float)h[m].y, (float)h[m].z, (float)h[m].w);
    dst.reserve(n + 1);
    stream_copy(c, dst.p, g.data(), sizeof(float4) * (n + 1), cudaMemcpyHostToDevice);
    return h;
  };
  eam_fast_tables(c, conv(c.rz, c.rz32, 2 * c.pp.nr + 1));
  if (c.fast_cnt) allow_fast_records();
  conv(c.frho_val, c.frho_val32, c.pp.nrho);
  conv(c.frho_der, c.frho_der32, c.pp.nrho);
}

void pair_compute_mixed(Ctx &c, int eflag, int vflag) {
  const int nsi = c.nsite_i();
  FixGrid G = make_fix_grid(c);
  Args32 A;
  A.pos = c.pos32.p;
  A.nbr = c.nbr_full.p;
  A.num = c.num_full.p;
  A.num_in = c.num_in.p;
  A.prefix = prefix_rule(c);
  A.slot_atom = c.slot_atom.p;
  A.na = c.na;
  A.ne = c.ne;
  A.nsi = nsi;
  A.cap = c.cap;
  A.G = G;
  A.f = c.f.p;
  A.gaussf = c.gaussf.p;
  if (eflag & CACB200_ENERGY_ATOM) {
    c.eatom.reserve(std::max(c.na, 1));
    c.enode.reserve(std::max(c.ne * 8, 1));
  }
  if (vflag & CACB200_VIRIAL_ATOM) {
    c.vatom.reserve(std::max(c.na * 6, 1));
    c.vnode.reserve(std::max(c.ne * 48, 1));
  }
  A.eatom = c.eatom.p;
  A.enode = c.enode.p;
  A.vatom = c.vatom.p;
  A.vnode = c.vnode.p;
  c.partial.reserve((size_t)std::max(c.num_sms * 8, nblk(nsi, 128)) * 7);
  c.ev_out.reserve(7);
  A.partial = c.partial.p;
  A.eflag = eflag;
  A.vflag = vflag;
  double nodal_weight = (double)NU / (double)NPE;
  A.vscale_node = nodal_weight / 2.0;
  A.escale_node = nodal_weight / 2.0;
  if (c.pp.style == CACB200_PAIR_EAM && c.nodal_energy_weight >= 0.0) A.escale_node = c.nodal_energy_weight / 2.0;
  c.escale_node_last = A.escale_node;
  const bool ev = eflag || vflag;
  // lanes per site by the size (results do not depend on it)
  const int lanes = nsi >= ONE_LANE_SITES ? 1 : nsi >= TWO_LANE_SITES ? 2 : 4;
  auto by_lanes = [&](auto &&launch) {
    if (lanes == 1) launch(std::integral_constant<int, 1>());
    else if (lanes == 2) launch(std::integral_constant<int, 2>());
    else launch(std::integral_constant<int, 4>());
  };
  int grid_ev = 1;
  if (c.pp.style == CACB200_PAIR_LJ) {
    Lj32 P{(float)(c.pp.cut * c.pp.cut), (float)c.pp.lj1, (float)c.pp.lj2, (float)c.pp.lj3, (float)c.pp.lj4,
           (float)c.pp.offset};
    KernelTimer t(c, "pair_lj32");
    grid_ev = std::max(nblk(nsi, 128), 1);
    if (ev) launch_behind(c, grid_ev, 128, 0, k_lj32<true>, A, P);
    else launch_behind(c, grid_ev, 128, 0, k_lj32<false>, A, P);
  } else {
    if (!c.have_mixed_tables) {
      mixed_tables(c);
      c.have_mixed_tables = true;
    }
    Eam32 Tb;
    Tb.rz = c.rz32.p;
    Tb.frho_val = c.frho_val32.p;
    Tb.frho_der = c.frho_der32.p;
    Tb.rdr = (float)c.pp.rdr;
    Tb.rdrho = (float)c.pp.rdrho;
    Tb.rhomax = (float)c.pp.rhomax;
    Tb.cutforcesq = (float)(c.pp.cut * c.pp.cut * std::ldexp(1.0, 52));
    Tb.nr = c.pp.nr;
    Tb.nrho = c.pp.nrho;
    Tb.fast = c.fast32.p;
    Tb.inv_ds = std::ldexp(c.fast_inv_ds, -52);
    Tb.base = 0x4b000000 + c.fast_lo;
    Tb.cnt = c.fast_cnt;
    c.rho.reserve(std::max(c.na + 8 * c.ne, 1));
    c.phi_site.reserve(std::max(nsi, 1));
    // resident blocks stride over the list slots, so the records are loaded
    // once per block; small systems take small blocks and one copy
    const long threads = (long)nsi * lanes;
    const bool small = threads < (long)c.num_sms * 512;
    const int tb = small ? 128 : 512;
    Tb.copies = small ? 1 : FAST_COPIES;
    const int need = std::max(nblk(threads, tb), 1);
    const int grid = c.work_queue && !small ? std::min(need, 2 * c.num_sms) : need;
    grid_ev = std::min(need, small ? c.num_sms * 8 : c.num_sms);
    c.tb_rho32 = c.tb_force32 = tb;
    if (c.nrep > 1)
      for (int &k : c.work_tile) k = c.work_queue && !small ? tb : 0;
    const bool fast = c.fast_cnt > 0;
    const size_t rec = fast ? sizeof(float4) * (size_t)(c.fast_cnt + 1) * Tb.copies : 0;
    auto go = [&](auto kernel, int blocks, size_t bytes, auto... args) {
      launch_behind(c, blocks, tb, bytes, kernel, A, Tb, args...);
    };
    {
      KernelTimer t(c, "eam_rho32");
      by_lanes([&](auto g) {
        constexpr int GL = decltype(g)::value;
        if (fast) go(k_eam_rho32<GL, true>, grid, rec, c.rho.p, c.phi_site.p, c.pos32.p);
        else go(k_eam_rho32<GL, false>, grid, 0, c.rho.p, c.phi_site.p, c.pos32.p);
      });
    }
    if (c.ne) {
      KernelTimer t(c, "eam_site_fp32");
      launch_behind(
          c, stride_grid((long)c.ne * NU, 256), 256, 0, k_eam_site_fp32, c.pos32.p, c.act_gid.p, c.dev_nact.p, c.na + NG * c.ne, c.na, c.rho.p, Tb);
    }
    {
      KernelTimer t(c, "eam_force32");
      by_lanes([&](auto g) {
        constexpr int GL = decltype(g)::value;
        if (ev && fast) go(k_eam_force32<GL, true, true>, grid_ev, 3 * rec, c.phi_site.p);
        else if (ev) go(k_eam_force32<GL, false, true>, grid_ev, 0, c.phi_site.p);
        else if (fast) go(k_eam_force32<GL, true, false>, grid, 2 * rec, c.phi_site.p);
        else go(k_eam_force32<GL, false, false>, grid, 0, c.phi_site.p);
      });
    }
  }
  if (ev) {
    k_reduce_partials32<<<1, 256, 0, c.stream>>>(c.partial.p, grid_ev, c.ev_out.p);
    c.have_peratom_e = (eflag & CACB200_ENERGY_ATOM) != 0;
    c.have_peratom_v = (vflag & CACB200_VIRIAL_ATOM) != 0;
    c.ev_pending = true;
    if (eflag & CACB200_ENERGY_GLOBAL) c.tally_step_e = c.step;
    if (vflag & CACB200_VIRIAL_GLOBAL) c.tally_step_v = c.step;
    if (eflag & CACB200_ENERGY_ATOM) c.tally_step_ae = c.step;
    if (vflag & CACB200_VIRIAL_ATOM) c.tally_step_av = c.step;
  }
  CACB200_CUDA(cudaGetLastError());
}

}  // namespace cacb200
