// Pair kernels: LJ 12-6 and two-pass EAM over the full neighbour list.
//
// Each i-site (atom or Gauss point) gathers over its own full list, so every
// force, density and per-site energy is written once by one thread with no
// atomics; the totals equal the reference's half-list sums with reactions
// (pair_lj_cut.cpp:227-417, pair_eam.cpp:618-1031) up to summation order:
//   * an atom's force is the sum over every neighbour; a Gauss point's force
//     likewise (its atom neighbours are the reactions the reference applies
//     from atom lists);
//   * the global energy and virial are sum_i scale_i * sum_j term_ij with
//     scale 1/2 for atoms and nodal_weight/2 for node Gauss points (the
//     reference's iescale + jescale split over the two ends of a pair);
//   * per-site energy and virial are half of each pair term (Pair::ev_tally,
//     pair.cpp:428-482).
// EAM evaluates F'(rho) once per site (atoms and nodes from their own
// density, interpolated lattice sites from shape-weighted nodal density)
// instead of once per pair, and keeps it in the w slot of the site table so
// one 32-byte load brings a neighbour's position and F'.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctx.cuh"
#include "device.cuh"

namespace cacb200 {

namespace {

inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

struct PairArgs {
  const double4 *xs;                // pair table (list-slot order; w = F')
  const int *nbr;                   // lists and counts indexed by list slot
  const int *num;
  const int *num_in;                // inner prefix length of each list ...
  PrefixRule prefix;                // ... and the rule for walking the rest
  const int *slot_atom;             // list slot -> atom (slots past the atoms are Gauss points)
  int na, ne, nsi;
  int cap;                          // list rows: the rest of a list fills its last rows
  double L[3];                      // box of a single system
  const Rep *reps;                  // batches: replica descriptors ...
  const int *site_rep;              // ... and the replica of each i-site (null for one system)
  double *f, *gaussf;
  double *eatom, *vatom, *enode, *vnode;
  double *partial;
  int eflag, vflag;
  double escale_node, vscale_node;  // global scales of a node Gauss point
};

__device__ __forceinline__ int site_of_slot(const PairArgs &A, int t) { return t < A.na ? A.slot_atom[t] : t; }

// The FP64 pair arithmetic in explicitly rounded and explicitly fused
// operations: every kernel that inlines it (grid and SM-local launches, with
// and without tallies) rounds alike, where the compiler would contract each
// copy its own way.
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }

// Walks n entries of a list: each lane takes four at a time, the next four
// entries loaded ahead and the four records issued back to back before any is
// used.  Entries past the end are walked as pairs too far apart to count.
// List entries are read once per pass: they are loaded as streaming
// (evict-first) so that L1 keeps the neighbour positions and spline records,
// which are reused.  f(partial, record, apart): the neighbour's record under
// its image; apart: past the end.
template <int G, class F>
__device__ __forceinline__ void walk(const PairArgs &A, int t, int i, const int *nb, int n, F &&f) {
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
    double4 o[4];
#pragma unroll
    for (int u = 0; u < 4; u++) o[u] = ld256(A.xs + (v[u] >> IMG_BITS));
    if (((v[0] ^ IMG_ZERO) | (v[1] ^ IMG_ZERO) | (v[2] ^ IMG_ZERO) | (v[3] ^ IMG_ZERO)) & ((1 << IMG_BITS) - 1)) {
      // images: an entry's image (0, 0, 0) leaves its position as it is
      const double *L = A.site_rep ? A.reps[A.site_rep[i]].b.L : A.L;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        int sx, sy, sz;
        img_decode(v[u] & ((1 << IMG_BITS) - 1), sx, sy, sz);
        if (sx) o[u].x = radd(o[u].x, rmul((double)sx, L[0]));
        if (sy) o[u].y = radd(o[u].y, rmul((double)sy, L[1]));
        if (sz) o[u].z = radd(o[u].z, rmul((double)sz, L[2]));
      }
    }
    const int now = left;
    load(left - 4);
#pragma unroll
    for (int u = 0; u < 4; u++) f(u % (4 / G), o[u], u && u >= now);
  }
}

// A site's list in two walks: the inner prefix (entries within the cutoff
// plus a margin at the build, the list's first rows), then, unless the
// site's displacement since the build and the largest one cannot close the
// margin (walk_rest, device.cuh), the rest (the list's last rows).  An entry's
// partial sum depends on its place in the walk, so the prefix is always walked
// on its own: the sums are the same whether the rest is walked or not.  The
// rule's flag and largest displacement belong to the site's replica (one hot
// replica of a batch does not end the shortcut for the others); one copy of
// the walk serves both segments.
template <int G, class F>
__device__ __forceinline__ void walk_list(const PairArgs &A, int t, int i, F &&f) {
  const int n_in = A.num_in[t], n = A.num[t];
  const int *nb = A.nbr + t;
  const bool rest = n > n_in && walk_rest(A.prefix, i, A.site_rep ? A.site_rep[i] : 0);
#pragma unroll 1
  for (int seg = 0; seg < (rest ? 2 : 1); seg++)
    walk<G>(A, t, i, seg ? nb + (size_t)(A.cap - (n - n_in)) * A.nsi : nb, seg ? n - n_in : n_in, f);
}

// Writes force (and per-site energy / virial) of i-site i and adds its global
// energy / virial to red.
template <bool EV>
__device__ __forceinline__ void finish_site(const PairArgs &A, int i, const double fi[3], double esum,
                                            const double vsum[6], double eextra_site, double eextra_global,
                                            double red[7]) {
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
    if (A.eflag & CACB200_ENERGY_GLOBAL) red[0] += es * esum + eextra_global;
    if (A.vflag & CACB200_VIRIAL_GLOBAL)
#pragma unroll
      for (int k = 0; k < 6; k++) red[1 + k] += vs * vsum[k];
    if (A.eflag & CACB200_ENERGY_ATOM) {
      const double ev = 0.5 * esum + eextra_site;
      if (atom) A.eatom[i] = ev;
      else A.enode[(size_t)e * 8 + node] = ev;
    }
    if (A.vflag & CACB200_VIRIAL_ATOM) {
      double *vo = atom ? A.vatom + 6 * (size_t)i : A.vnode + 48 * (size_t)e + 6 * node;
#pragma unroll
      for (int k = 0; k < 6; k++) vo[k] = 0.5 * vsum[k];
    }
  }
}

// Per-site sums of a force pass; fpair and the separation as in the pair terms.
template <int G, bool EV>
struct ForceSums {
  Sum4<double, G> f[3], e[1], v[EV ? 6 : 1];
  __device__ __forceinline__ void add(int part, double dx, double dy, double dz, double fpair) {
    f[0].a[part] = fma(dx, fpair, f[0].a[part]);
    f[1].a[part] = fma(dy, fpair, f[1].a[part]);
    f[2].a[part] = fma(dz, fpair, f[2].a[part]);
  }
  __device__ __forceinline__ void add_ev(int part, double dx, double dy, double dz, double fpair, double phi,
                                         int eflag, int vflag) {
    if (eflag) e[0].a[part] = radd(e[0].a[part], phi);
    if (vflag) {
      v[0].a[part] = fma(rmul(dx, dx), fpair, v[0].a[part]);
      v[1].a[part] = fma(rmul(dy, dy), fpair, v[1].a[part]);
      v[2].a[part] = fma(rmul(dz, dz), fpair, v[2].a[part]);
      v[3].a[part] = fma(rmul(dx, dy), fpair, v[3].a[part]);
      v[4].a[part] = fma(rmul(dx, dz), fpair, v[4].a[part]);
      v[5].a[part] = fma(rmul(dy, dz), fpair, v[5].a[part]);
    }
  }
  __device__ __forceinline__ void totals(double fi[3], double &esum, double vsum[6]) const {
#pragma unroll
    for (int d = 0; d < 3; d++) fi[d] = f[d].total();
    if constexpr (EV) {
      esum = e[0].total();
#pragma unroll
      for (int k = 0; k < 6; k++) vsum[k] = v[k].total();
    }
  }
};

// ------------------------------------------------------------------- LJ

struct LjParams {
  double cutsq, lj1, lj2, lj3, lj4, offset;
};

template <int G, bool EV>
__global__ void __launch_bounds__(128, EV ? 4 : 6) k_lj(PairArgs A, LjParams P) {
  behind_previous();
  double red[7] = {0, 0, 0, 0, 0, 0, 0};
  for_each_slot<G>(A.nsi, [&](int t, bool valid) {
    const int i = valid ? site_of_slot(A, t) : 0;           // site-table index
    ForceSums<G, EV> S;
    if (valid) {
      const double4 xi = A.xs[t];
      walk_list<G>(A, t, i, [&](int part, const double4 &xj, bool apart) {
        const double dx = rsub(xi.x, xj.x), dy = rsub(xi.y, xj.y), dz = rsub(xi.z, xj.z);
        const double rsq = fma(dz, dz, fma(dy, dy, rmul(dx, dx)));
        if (rsq < P.cutsq && !apart) {
          const double r2inv = 1.0 / rsq;
          const double r6inv = rmul(rmul(r2inv, r2inv), r2inv);
          const double fpair = rmul(rmul(r6inv, fma(P.lj1, r6inv, -P.lj2)), r2inv);
          S.add(part, dx, dy, dz, fpair);
          if (EV) S.add_ev(part, dx, dy, dz, fpair, fma(r6inv, fma(P.lj3, r6inv, -P.lj4), -P.offset), A.eflag, A.vflag);
        }
      });
    }
    double fi[3], esum = 0.0, vsum[6];
    S.totals(fi, esum, vsum);
    if (valid && threadIdx.x % G == 0) finish_site<EV>(A, i, fi, esum, vsum, 0.0, 0.0, red);
  });
  if (EV) block_reduce_store<7>(red, A.partial);
}

// ------------------------------------------------------------------ EAM

// r-dependent splines as one 64-byte record per knot m: rz[2m] the rhor value
// coefficients (S3, S4, S5, S6 of PairEAM::interpolate), rz[2m+1] those of
// z2r.  A pair reads the record once; the derivative coefficients are the
// reference's (S0, S1, S2) = (3 S3, 2 S4, S5) / dr (pair_eam.cpp:612-614),
// applied as ((3 S3 p + 2 S4) p + S5) * (1/dr).
struct EamTables {
  const double4 *rz, *frho_val, *frho_der;
  double rdr, rdrho, rhomax, cutforcesq;
  int nr, nrho;
};

// Distance and its reciprocal from the square: rsqrt carries at most one ulp,
// as the reciprocal of a rounded square root does, and one step of Newton's
// method takes r = rsq / sqrt(rsq) to within rounding of the square root.
// Sites on one another (the square's high word is 0 below 2e-314) are 0 apart
// (0 x inf would be no number), with an infinite reciprocal.
__device__ __forceinline__ double distance(double rsq, double &recip) {
  recip = rsqrt(rsq);
  const double r = rmul(rsq, recip);
  return __double2hiint(rsq) ? fma(fma(-r, r, rsq), rmul(0.5, recip), r) : 0.0;
}

// The knot of distance r and the place p in its interval, as the reference's
// m = int(r / dr + 1), limited to 1 .. nr - 1, and p = min(r / dr + 1 - m, 1): the
// truncation is a fused operation rounded down at 2^52.
__device__ __forceinline__ int r_knot(const EamTables &T, double r, double &p) {
  const double x = __fma_rd(r, T.rdr, 4503599627370497.0);   // 2^52 + 1
  int m = max(__double2loint(x), 1);
  p = fma(r, T.rdr, rsub(4503599627370497.0, x));
  if (m >= T.nr) {
    m = T.nr - 1;
    p = 1.0;
  }
  return m;
}

// A cubic's value and derivative (Horner's scheme and its derivative's).
__device__ __forceinline__ double cubic(const double4 &c, double p) { return fma(fma(fma(c.x, p, c.y), p, c.z), p, c.w); }
__device__ __forceinline__ double cubic_slope(const double4 &c, double p) {
  const double b = fma(c.x, p, c.y);
  return fma(fma(c.x, p, b), p, fma(b, p, c.z));
}

// F'(rho) and F(rho) on the frho spline row (PairEAM::compute_fp,
// pair_eam.cpp:1160-1169; the energy read on the same row, i.e. the
// reference with its coefficient pointer returned to the caller)
__device__ __forceinline__ double eam_fp(const EamTables &T, double rho, double *phi) {
  double p = radd(rmul(rho, T.rdrho), 1.0);
  int m = (int)p;
  m = max(1, min(m, T.nrho - 1));
  p = rsub(p, (double)m);
  p = fmin(p, 1.0);
  double4 d = T.frho_der[m];
  double fp = radd(rmul(radd(rmul(d.x, p), d.y), p), d.z);
  if (phi) {
    double4 v = T.frho_val[m];
    double e = radd(rmul(radd(rmul(radd(rmul(v.x, p), v.y), p), v.z), p), v.w);
    if (rho > T.rhomax) e = radd(e, rmul(fp, rsub(rho, T.rhomax)));
    *phi = e;
  }
  return fp;
}

// pass 1: density at atoms and node Gauss points (pair_eam.cpp:707-812), then
// F' at the site itself into xs[i].w (pair_eam.cpp:819-833 for atoms; for a
// node the reference's rhoi = noderho at :901-903).
template <int G>
__device__ __forceinline__ void rho_slot(const PairArgs &A, const EamTables &T, int t, bool valid, double *rho_out,
                                         double *phi_site) {
  const int i = valid ? site_of_slot(A, t) : 0;           // site-table index
  Sum4<double, G> sum;
  if (valid) {
    const double4 xi = A.xs[t];
    walk_list<G>(A, t, i, [&](int part, const double4 &xj, bool apart) {
      const double dx = rsub(xi.x, xj.x), dy = rsub(xi.y, xj.y), dz = rsub(xi.z, xj.z);
      const double rsq = fma(dz, dz, fma(dy, dy, rmul(dx, dx)));
      if (rsq < T.cutforcesq && !apart) {
        double recip, p;
        const int m = r_knot(T, distance(rsq, recip), p);
        sum.a[part] = radd(sum.a[part], cubic(ldg256(T.rz + 2 * m), p));
      }
    });
  }
  const double rho = sum.total();
  if (!valid || threadIdx.x % G) return;
  int slot = i;
  if (i >= A.na) {
    int e = (i - A.na) / NG, g = (i - A.na) % NG;
    slot = A.na + 8 * e + gauss_node(g);
  }
  rho_out[slot] = rho;
  double phi = 0.0;
  double fp = eam_fp(T, rho, A.eflag ? &phi : nullptr);
  ((double *)A.xs)[4 * (size_t)t + 3] = fp;
  if (A.eflag) phi_site[i] = phi;
}

template <int TB, int G>
__global__ void __launch_bounds__(TB, 1024 / TB) k_eam_rho(PairArgs A, EamTables T, double *rho_out,
                                                       double *phi_site) {
  behind_previous();
  for_each_slot<G>(A.nsi, [&](int t, bool valid) { rho_slot<G>(A, T, t, valid, rho_out, phi_site); });
}

// Both passes are bound by the L1 data pipe (ncu, 313 k sites: force pass 84 %
// of its peak while active, FP64 pipe 24 %, density pass 77 % and 20 %): each
// neighbour's 32-byte record and each in-cutoff pair's 64-byte spline record is
// a scattered read.  Fused operations and one rsqrt in place of a root and a
// division halve the FP64 work (1.21 M sites: density 410 -> 397 us, force 581
// -> 570; with tallies 747 -> 658; 6 k sites, four lanes a site, 43 -> 15 and
// 45 -> 17).  Sharing a spline record's two halves between neighbouring lanes
// was slower (641 us: the exchanges cost more than the reads).
//
// Single systems: the force-only passes over SM-local runs of list slots
// (sm_run, device.cuh); each slot is computed by the same function as in the
// grid launch, so the results are the grid launch's bit for bit.
template <int TB, int G>
__global__ void __launch_bounds__(TB, 1024 / TB) k_eam_rho_sm(PairArgs A, EamTables T, double *rho_out,
                                                          double *phi_site, int *cnt, int nsm) {
  behind_previous();
  __shared__ int v;
  if (threadIdx.x == 0) v = sm_id() % nsm;
  const int nrun = (A.nsi + TB / G - 1) / (TB / G);
  for (;;) {
    const int r = sm_run(cnt, nsm, nrun, v);
    if (r < 0) return;
    const int t = r * (TB / G) + (int)threadIdx.x / G;
    rho_slot<G>(A, T, t, t < A.nsi, rho_out, phi_site);
  }
}

// F' at interpolated lattice sites from shape-weighted nodal density
// (pair_eam.cpp:957-969)
__global__ void k_eam_site_fp(double4 *xs, const int *act_gid, const int *nact_dev, int base, int na,
                              const double *rho, EamTables T) {
  behind_previous();
  const int nact = *nact_dev;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nact; k += gridDim.x * blockDim.x) {
    int gid = act_gid[k];
    int e = gid / NU, u = gid % NU;
    const double *rn = rho + na + 8 * (size_t)e;
    double r = 0.0;
#pragma unroll
    for (int n = 0; n < NPE; n++) r = radd(r, rmul(shape_val(u, n), rn[n]));
    xs[base + k].w = eam_fp(T, r, nullptr);
  }
}

// pass 2: forces (pair_eam.cpp:845-1028)
template <int G, bool EV>
__device__ __forceinline__ void force_slot(const PairArgs &A, const EamTables &T, int t, bool valid,
                                           const double *phi_site, double red[7]) {
  const int i = valid ? site_of_slot(A, t) : 0;           // site-table index
  ForceSums<G, EV> S;
  if (valid) {
    const double4 xi = A.xs[t];
    const double fpi = xi.w;
    walk_list<G>(A, t, i, [&](int part, const double4 &xj, bool apart) {
      const double dx = rsub(xi.x, xj.x), dy = rsub(xi.y, xj.y), dz = rsub(xi.z, xj.z);
      const double rsq = fma(dz, dz, fma(dy, dy, rmul(dx, dx)));
      if (rsq < T.cutforcesq && !apart) {
        double recip, p;
        const int m = r_knot(T, distance(rsq, recip), p);
        const double4 rv = ldg256(T.rz + 2 * m), zv = ldg256(T.rz + 2 * m + 1);
        const double rhop = rmul(cubic_slope(rv, p), T.rdr);
        const double phi = rmul(cubic(zv, p), recip);
        const double phip = rmul(fma(cubic_slope(zv, p), T.rdr, -phi), recip);
        const double fpair = -rmul(fma(radd(fpi, xj.w), rhop, phip), recip);
        S.add(part, dx, dy, dz, fpair);
        if (EV) S.add_ev(part, dx, dy, dz, fpair, phi, A.eflag, A.vflag);
      }
    });
  }
  double fi[3], esum = 0.0, vsum[6];
  S.totals(fi, esum, vsum);
  if (!valid || threadIdx.x % G) return;
  double eemb_site = 0.0, eemb_global = 0.0;
  if (EV && A.eflag) {
    eemb_site = phi_site[i];
    eemb_global = i < A.na ? eemb_site : eemb_site * A.escale_node * 2.0;
  }
  finish_site<EV>(A, i, fi, esum, vsum, eemb_site, eemb_global, red);
}

template <int TB, int G, bool EV>
__global__ void __launch_bounds__(TB, (EV ? 512 : 768) / TB) k_eam_force(PairArgs A, EamTables T,
                                                                       const double *phi_site) {
  behind_previous();
  double red[7] = {0, 0, 0, 0, 0, 0, 0};
  for_each_slot<G>(A.nsi, [&](int t, bool valid) { force_slot<G, EV>(A, T, t, valid, phi_site, red); });
  if (EV) block_reduce_store<7>(red, A.partial);
}

template <int TB, int G>
__global__ void __launch_bounds__(TB, 640 / TB) k_eam_force_sm(PairArgs A, EamTables T, const double *phi_site,
                                                           int *cnt, int nsm) {
  behind_previous();
  __shared__ int v;
  if (threadIdx.x == 0) v = sm_id() % nsm;
  const int nrun = (A.nsi + TB / G - 1) / (TB / G);
  for (;;) {
    const int r = sm_run(cnt, nsm, nrun, v);
    if (r < 0) return;
    const int t = r * (TB / G) + (int)threadIdx.x / G;
    force_slot<G, false>(A, T, t, t < A.nsi, phi_site, nullptr);
  }
}

__global__ void k_reduce_partials(const double *partial, int nblocks, double *out) {
  // one warp per component, fixed order
  int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k >= 7) return;
  double s = 0.0;
  for (int b = lane; b < nblocks; b += 32) s += partial[b * 7 + k];
  s = warp_sum(s);
  if (lane == 0) out[k] = s;
}

// ---------------------------------------------------------- spline tables

// PairEAM::interpolate (pair_eam.cpp:580-616): 7 coefficients per knot m = 1..n
void spline7(int n, double delta, const std::vector<double> &f1, std::vector<double> &sp) {
  sp.assign((size_t)(n + 1) * 7, 0.0);
  auto S = [&](int m, int c) -> double & { return sp[(size_t)m * 7 + c]; };
  for (int m = 1; m <= n; m++) S(m, 6) = f1[m];
  S(1, 5) = S(2, 6) - S(1, 6);
  S(2, 5) = 0.5 * (S(3, 6) - S(1, 6));
  S(n - 1, 5) = 0.5 * (S(n, 6) - S(n - 2, 6));
  S(n, 5) = S(n, 6) - S(n - 1, 6);
  for (int m = 3; m <= n - 2; m++)
    S(m, 5) = ((S(m - 2, 6) - S(m + 2, 6)) + 8.0 * (S(m + 1, 6) - S(m - 1, 6))) / 12.0;
  for (int m = 1; m <= n - 1; m++) {
    S(m, 4) = 3.0 * (S(m + 1, 6) - S(m, 6)) - 2.0 * S(m, 5) - S(m + 1, 5);
    S(m, 3) = S(m, 5) + S(m + 1, 5) - 2.0 * (S(m + 1, 6) - S(m, 6));
  }
  S(n, 4) = 0.0;
  S(n, 3) = 0.0;
  for (int m = 1; m <= n; m++) {
    S(m, 2) = S(m, 5) / delta;
    S(m, 1) = 2.0 * S(m, 4) / delta;
    S(m, 0) = 3.0 * S(m, 3) / delta;
  }
}

void upload_split(Ctx &c, const std::vector<double> &sp, int n, DBuf<double4> &val, DBuf<double4> &der) {
  std::vector<double4> hv(n + 1), hd(n + 1);
  for (int m = 0; m <= n; m++) {
    const double *r = &sp[(size_t)m * 7];
    hv[m] = make_double4(r[3], r[4], r[5], r[6]);
    hd[m] = make_double4(r[0], r[1], r[2], 0.0);
  }
  val.reserve(n + 1);
  der.reserve(n + 1);
  stream_copy(c, val.p, hv.data(), sizeof(double4) * (n + 1), cudaMemcpyHostToDevice);
  stream_copy(c, der.p, hd.data(), sizeof(double4) * (n + 1), cudaMemcpyHostToDevice);
}

}  // namespace

void eam_tables(Ctx &c, const double *frho, const double *rhor, const double *z2r) {
  PairParams &p = c.pp;
  std::vector<double> a(p.nrho + 1, 0.0), b(p.nr + 1, 0.0), z(p.nr + 1, 0.0), sp;
  for (int m = 1; m <= p.nrho; m++) a[m] = frho[m - 1];
  for (int m = 1; m <= p.nr; m++) {
    b[m] = rhor[m - 1];
    z[m] = z2r[m - 1];
  }
  c.have_mixed_tables = false;
  spline7(p.nrho, p.drho, a, sp);
  upload_split(c, sp, p.nrho, c.frho_val, c.frho_der);
  spline7(p.nr, p.dr, b, sp);
  std::vector<double4> rz((size_t)2 * (p.nr + 1));
  for (int m = 0; m <= p.nr; m++) {
    const double *r = &sp[(size_t)m * 7];
    rz[2 * m] = make_double4(r[3], r[4], r[5], r[6]);
  }
  spline7(p.nr, p.dr, z, sp);
  for (int m = 0; m <= p.nr; m++) {
    const double *r = &sp[(size_t)m * 7];
    rz[2 * m + 1] = make_double4(r[3], r[4], r[5], r[6]);
  }
  // a block of 2 MiB of its own: sharing one with the tables of F, 640 KB into
  // it, cost 3 % of both passes at 1.21 M sites (force 572 -> 589 us, density
  // 396 -> 407)
  c.rz.reserve(std::max(rz.size(), (size_t)(2 << 20) / sizeof(double4)));
  stream_copy(c, c.rz.p, rz.data(), sizeof(double4) * rz.size(), cudaMemcpyHostToDevice);
}

// i-sites from which a site takes two lanes, and below which four (the sums
// do not depend on it).  us with 1 / 2 / 4 lanes a site before the walk loaded
// ahead: LJ pass 6 k sites 34 / 21 / 17, 84 k 42 / 40 / 39, 313 k 119 / 105 /
// 118, 1.21 M 356 / 354 / 423; EAM force pass 45 / 31 / 22, 68 / 63 / 61,
// 178 / 174 / 182, 578 / 574 / 616.
constexpr int TWO_LANE_SITES = 100000;

// Block size of the force-only pair passes of batches, chosen per context by
// timing 64, 128 and 256 threads (best of three launches each; 128 unless
// another is at least 3 % faster) on the context's own lists the first time
// they run (results do not depend on the choice; the passes are idempotent, so
// the trial launches change nothing).  Not during stream capture: there the
// default stays.
template <int G>
void launch_rho(const Ctx &c, int tb, int nsi, const PairArgs &A, const EamTables &T, double *rho, double *phi) {
  const int nb = std::max(nblk((long)nsi * G, tb), 1);
  const auto kernel = tb == 64 ? k_eam_rho<64, G> : tb == 256 ? k_eam_rho<256, G> : k_eam_rho<128, G>;
  launch_behind(c, nb, tb, 0, kernel, A, T, rho, phi);
}
template <int G>
void launch_force(const Ctx &c, int tb, int nsi, const PairArgs &A, const EamTables &T, const double *phi) {
  const int nb = std::max(nblk((long)nsi * G, tb), 1);
  const auto kernel = tb == 64    ? k_eam_force<64, G, false>
                      : tb == 256 ? k_eam_force<256, G, false>
                                  : k_eam_force<128, G, false>;
  launch_behind(c, nb, tb, 0, kernel, A, T, phi);
}

template <class F>
float time_launch(cudaStream_t st, F &&launch) {
  cudaEvent_t a, b;
  CACB200_CUDA(cudaEventCreate(&a));
  CACB200_CUDA(cudaEventCreate(&b));
  float best = 1e30f;
  for (int rep = 0; rep < 3; rep++) {
    CACB200_CUDA(cudaEventRecord(a, st));
    launch();
    CACB200_CUDA(cudaEventRecord(b, st));
    CACB200_CUDA(cudaEventSynchronize(b));
    float ms = 0.f;
    CACB200_CUDA(cudaEventElapsedTime(&ms, a, b));
    best = std::min(best, ms);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return best;
}

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CACB200_CUDA(cudaStreamIsCapturing(st, &cs));
  return cs != cudaStreamCaptureStatusNone;
}

void pair_compute(Ctx &c, int eflag, int vflag) {
  c.check_system();
  if (!c.lists_valid) throw Error(CACB200_ESTATE, "neighbour lists not built");
  if (c.precision == CACB200_MIXED) {
    pair_compute_mixed(c, eflag, vflag);
    return;
  }
  const int nsi = c.nsite_i();
  const int T = 128;
  const int lanes = nsi >= TWO_LANE_SITES ? 2 : 4;
  auto by_lanes = [&](auto &&launch) {
    if (lanes == 2) launch(std::integral_constant<int, 2>());
    else launch(std::integral_constant<int, 4>());
  };
  const int nb = std::max(nblk((long)nsi * lanes, T), 1);
  const int nb_ev = std::min(nb, 4 * c.num_sms);   // with tallies: resident blocks, one partial each
  PairArgs A;
  A.xs = c.xss.p;
  A.nbr = c.nbr_full.p;
  A.num = c.num_full.p;
  A.num_in = c.num_in.p;
  A.prefix = prefix_rule(c);
  A.slot_atom = c.slot_atom.p;
  A.na = c.na;
  A.ne = c.ne;
  A.nsi = nsi;
  A.cap = c.cap;
  for (int d = 0; d < 3; d++) A.L[d] = c.prd[d];
  A.reps = c.rep_d.p;
  A.site_rep = c.nrep > 1 ? c.site_rep.p : nullptr;
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
  c.partial.reserve((size_t)nb_ev * 7);
  c.ev_out.reserve(7);
  A.partial = c.partial.p;
  A.eflag = eflag;
  A.vflag = vflag;
  double nodal_weight = (double)NU / (double)NPE;   // element_vec_cac.cpp:1732
  A.vscale_node = nodal_weight / 2.0;
  A.escale_node = nodal_weight / 2.0;
  if (c.pp.style == CACB200_PAIR_EAM && c.nodal_energy_weight >= 0.0)
    A.escale_node = c.nodal_energy_weight / 2.0;
  c.escale_node_last = A.escale_node;

  if (c.pp.style == CACB200_PAIR_LJ) {
    LjParams P{c.pp.cut * c.pp.cut, c.pp.lj1, c.pp.lj2, c.pp.lj3, c.pp.lj4, c.pp.offset};
    KernelTimer t(c, "pair_lj");
    by_lanes([&](auto g) {
      constexpr int G = decltype(g)::value;
      if (eflag || vflag) launch_behind(c, nb_ev, T, 0, k_lj<G, true>, A, P);
      else launch_behind(c, nb, T, 0, k_lj<G, false>, A, P);
    });
  } else if (c.pp.style == CACB200_PAIR_EAM) {
    EamTables Tb;
    Tb.rz = c.rz.p;
    Tb.frho_val = c.frho_val.p;
    Tb.frho_der = c.frho_der.p;
    Tb.rdr = c.pp.rdr;
    Tb.rdrho = c.pp.rdrho;
    Tb.rhomax = c.pp.rhomax;
    Tb.cutforcesq = c.pp.cut * c.pp.cut;
    Tb.nr = c.pp.nr;
    Tb.nrho = c.pp.nrho;
    c.rho.reserve(std::max(c.na + 8 * c.ne, 1));
    c.phi_site.reserve(std::max(nsi, 1));
    const bool many = c.nrep > 1;
    auto site_fp = [&] {
      if (c.ne)
        launch_behind(
            c, stride_grid((long)c.ne * NU, 256), 256, 0, k_eam_site_fp, c.xss.p, c.act_gid.p, c.dev_nact.p, c.na + NG * c.ne, c.na, c.rho.p, Tb);
    };
    auto rho = [&](int tb) {
      by_lanes([&](auto g) { launch_rho<decltype(g)::value>(c, tb, nsi, A, Tb, c.rho.p, c.phi_site.p); });
    };
    auto force = [&](int tb) {
      by_lanes([&](auto g) { launch_force<decltype(g)::value>(c, tb, nsi, A, Tb, c.phi_site.p); });
    };
    // single systems of more than a wave of blocks: the force-only passes
    // over SM-local runs
    const bool smq = !many && c.work_queue && lanes == 2;
    c.sm_counter.reserve(2 * c.num_sms);
    auto resident = [](auto kernel) {
      int b = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, 128, 0);
      return b > 0 ? b : 1;
    };
    static const int per_sm_rho = resident(k_eam_rho_sm<128, 2>), per_sm_force = resident(k_eam_force_sm<128, 2>);
    auto rho_s = [&] {
      CACB200_CUDA(cudaMemsetAsync(c.sm_counter.p, 0, sizeof(int) * c.num_sms, c.stream));
      k_eam_rho_sm<128, 2><<<per_sm_rho * c.num_sms, 128, 0, c.stream>>>(
          A, Tb, c.rho.p, c.phi_site.p, c.sm_counter.p, c.num_sms);
    };
    auto force_s = [&] {
      CACB200_CUDA(cudaMemsetAsync(c.sm_counter.p + c.num_sms, 0, sizeof(int) * c.num_sms, c.stream));
      k_eam_force_sm<128, 2><<<per_sm_force * c.num_sms, 128, 0, c.stream>>>(
          A, Tb, c.phi_site.p, c.sm_counter.p + c.num_sms, c.num_sms);
    };
    if (many && c.tune_gen != c.gen && !eflag && !vflag && !capturing(c.stream)) {
      // another size replaces 128 only when it is at least 3 % faster
      const int cand[3] = {128, 64, 256};
      float best = 1e30f;
      for (int tb : cand) {
        float ms = time_launch(c.stream, [&] { rho(tb); });
        if (tb == 128 || ms < 0.97f * best) best = ms, c.tb_rho = tb;
      }
      rho(c.tb_rho);
      site_fp();
      best = 1e30f;
      for (int tb : cand) {
        float ms = time_launch(c.stream, [&] { force(tb); });
        if (tb == 128 || ms < 0.97f * best) best = ms, c.tb_force = tb;
      }
      c.tune_gen = c.gen;
    }
    {
      KernelTimer t(c, "eam_rho");
      if (smq) rho_s();
      else rho(c.tb_rho);
    }
    {
      KernelTimer t(c, "eam_site_fp");
      site_fp();
    }
    {
      KernelTimer t(c, "eam_force");
      if (eflag || vflag) {
        by_lanes([&](auto g) {
          launch_behind(c, nb_ev, T, 0, k_eam_force<128, decltype(g)::value, true>, A, Tb, c.phi_site.p);
        });
      } else if (smq) {
        force_s();
      } else {
        force(c.tb_force);
      }
    }
  } else {
    throw Error(CACB200_ESTATE, "no pair style set");
  }
  if (eflag || vflag) {
    k_reduce_partials<<<1, 256, 0, c.stream>>>(c.partial.p, nb_ev, c.ev_out.p);
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
