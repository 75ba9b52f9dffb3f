// Device-resident views of a GCMC system and of one chain's mutable state, plus the
// block-level building blocks shared by the plain (one launch per trial) kernels and the
// persistent batched kernel.
//
// HBM layout (per system, immutable): framework atoms as double4 {x,y,z,q} in condensed
// order + int type; voxel lists (CSR, ascending atom index); erc/vvv tables (mxgrid+1 doubles
// per row); k-vector table packed (l | (m+128)<<8 | (n+128)<<16) + akk (double).
// Per chain (mutable): S(k) as double2 {Re, Im}; guest sites as double4 {x,y,z,q} + int type,
// one contiguous segment per guest species, molecules in the reference's order.
#pragma once
#include <cuda_runtime.h>

#include "fmc_common.h"

namespace fmc {

struct DevSystem {
  CellGeom cell;
  int nf;
  const double4* fw;
  const int* fw_type;
  int nvox[3];
  const int* vox_off;
  const int* vox_atoms;
  const unsigned short* vox_atoms16;  // the same lists as 16-bit indices (null when nf > 65535)
  const double4* vox_xyzq;            // the same lists with each entry's atom inlined, and
  const unsigned char* vox_type;      // its type (coalesced one-hop reads)
  double rcut2, rdr_e, rdr_v;
  const double* erc;
  const double* vvv;
  // {erc, vvv} of one table row interleaved, row 0 holding {erc, 0} for pairs without a vdW
  // table; null when the two tables have different spacings (rvdw other than rcut)
  const double2* pair_tab;
  int tab_stride;
  int ntypes;
  const int* pair_row;
  int K;
  int kmax[3];
  const int* kpack;
  const struct KOctet* koct;  // the k-vectors by (l, |m|) and pairs of |n|
  int noct;
  const double* akk;
  double recip_pref;
};

// The k-vectors (l, +-m, +-n) of two |n|: table indices in the order (+m,+n), (+m,-n), (-m,+n), (-m,-n)
// of n[0], then of n[1]; -1 where the half space or the cut-off leaves one out.
struct KOctet {
  int k[8];
  short l, m, n[2];
};

constexpr int kMaxPassSites = 2 * kMaxGuestSites;

// Guest-site segments of one chain as seen by one launch (counts passed by value).
struct GuestView {
  const double4* site;
  const int* type;
  int nseg;
  int seg_off[kMaxGuestTypes];
  int seg_len[kMaxGuestTypes];  // sites currently present
};

FMC_HD int kpack(int l, int m, int n) { return l | ((m + 128) << 8) | ((n + 128) << 16); }
FMC_HD void kunpack(int p, int& l, int& m, int& n) {
  l = p & 0xff;
  m = ((p >> 8) & 0xff) - 128;
  n = ((p >> 16) & 0xff) - 128;
}

#if defined(__CUDACC__)

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.y * b.x + b.y * a.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - b.y * a.x);
}

// e^{i 2 pi j s} for j = 0..kmax by the recurrence of ewald.f:118-137 into tab[0..kmax].
__device__ __forceinline__ void axis_phases(double s, int kmax, double2* tab) {
  double sn, cs;
  sincos(2.0 * kPi * s, &sn, &cs);
  tab[0] = make_double2(1.0, 0.0);
  double2 p = make_double2(cs, sn);
  if (kmax >= 1) tab[1] = p;
#pragma unroll 1
  for (int j = 2; j <= kmax; j++) {
    p = make_double2(p.x * cs - p.y * sn, p.y * cs + p.x * sn);
    tab[j] = p;
  }
}

// sqrt(x) for x >= 0 without a branch, within an ulp or rounded correctly: the hardware's estimate of
// 1/sqrt(x), refined.  The added 1e-300 leaves every x above 1e-284 as it is and keeps x = 0 finite.
__device__ __forceinline__ double rsqrt_estimate(double& x) {
  double y;
  x += 1e-300;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double sqrt_approx(double x) {
  const double y = rsqrt_estimate(x);
  return sqrt_refine(x, y);
}
__device__ __forceinline__ double sqrt_exact(double x) {
  const double y = rsqrt_estimate(x);
  return sqrt_rounded(x, y);
}

// Fractional coordinates s = rcell . r as in ewald.f:106-108.
FMC_HD void frac_coords(const CellGeom& c, double x, double y, double z, double* s) {
  const double* r = c.rh;
  s[0] = r[0] * x + r[3] * y + r[6] * z;
  s[1] = r[1] * x + r[4] * y + r[7] * z;
  s[2] = r[2] * x + r[5] * y + r[8] * z;
}

// ------------------------------------------------------------------ pairs without branches
// How pairs are imaged and tabulated, each compiled by itself: orthorhombic cells (imcon 1, 2) and
// parallelepipeds (3) whose erc and vvv share one spacing, and everything else (half-shift cells, slabs,
// rvdw other than rcut) reading the boundary condition from the cell.
enum PairKind : int { kPairOrtho = 0, kPairTriclinic = 1, kPairGeneral = 2 };

FMC_HD int pair_kind(const DevSystem& S) {
  return !S.pair_tab || S.cell.imcon > 3 ? kPairGeneral : (S.cell.imcon == 3 ? kPairTriclinic : kPairOrtho);
}

constexpr double kMagic = 6755399441055744.0;  // 1.5 x 2^52: adding it rounds to an integer

// x - nint(x) (halves away from zero) by the rounding of an addition.
__device__ __forceinline__ double nint_rest(double x) {
  const double f = x - ((x + kMagic) - kMagic);
  return fabs(f) == 0.5 ? copysign(0.5, -x) : f;
}

// The reference's image of a separation (images, utility_pack.f:1138-1349).
template <int KIND>
__device__ __forceinline__ void image(const CellGeom& c, double& dx, double& dy, double& dz) {
  if (KIND == kPairOrtho) {
    // nint by the rounding of an addition: a tie picks either image, at the same distance; imcon 1
    // takes the first edge for every axis
    const int iy = c.imcon == 1 ? 0 : 1, iz = c.imcon == 1 ? 0 : 2;
    dx = fma(-c.h[0], fma(c.inv[0], dx, kMagic) - kMagic, dx);
    dy = fma(-c.h[4 * iy], fma(c.inv[iy], dy, kMagic) - kMagic, dy);
    dz = fma(-c.h[4 * iz], fma(c.inv[iz], dz, kMagic) - kMagic, dz);
  } else if (KIND == kPairTriclinic) {
    const double *r = c.rh, *h = c.h;
    const double fx = nint_rest(r[0] * dx + r[3] * dy + r[6] * dz);
    const double fy = nint_rest(r[1] * dx + r[4] * dy + r[7] * dz);
    const double fz = nint_rest(r[2] * dx + r[5] * dy + r[8] * dz);
    dx = h[0] * fx + h[3] * fy + h[6] * fz;
    dy = h[1] * fx + h[4] * fy + h[7] * fz;
    dz = h[2] * fx + h[5] * fy + h[8] * fz;
  } else {
    min_image(c, dx, dy, dz);
  }
}

template <int KIND>
__device__ __forceinline__ double image_dist2(const CellGeom& c, double dx, double dy, double dz) {
  image<KIND>(c, dx, dy, dz);
  return fma(dx, dx, fma(dy, dy, dz * dz));
}

// Adds a pair's table energies: v1 += cq erc(r), v2 += sg vvv(r) with r^2 = rs <= rcut^2 and the row that
// begins at `off` (0: none; row 0 of the interleaved table holds no vdW).
template <int KIND>
__device__ __forceinline__ void pair_table(const DevSystem& S, double rs, double cq, int off, double sg, double& v1,
                                           double& v2) {
  const double r = sqrt_approx(rs);
  const double x = __dmul_rn(r, S.rdr_e);
  const double f = (x - 0.5) + kMagic;  // floor(x) but for integers, where either interval agrees
  const int l = __double2loint(f);
  const double p = x - (f - kMagic), pm = p - 1.0, hp = 0.5 * p;
  if (KIND != kPairGeneral) {
    const double2* tb = S.pair_tab + (off + l);
    const double2 a0 = tb[0], a1 = tb[1], a2 = tb[2];
    const double e1 = fma(a1.x - a0.x, p, a0.x), e2 = fma(a2.x - a1.x, pm, a1.x);
    const double w1 = fma(a1.y - a0.y, p, a0.y), w2 = fma(a2.y - a1.y, pm, a1.y);
    v1 = fma(fma(e2 - e1, hp, e1), cq, v1);
    v2 = fma(fma(w2 - w1, hp, w1), sg, v2);
  } else {
    v1 = fma(interp3(S.erc, r, S.rdr_e), cq, v1);
    if (off) v2 = fma(interp3(S.vvv + off, r, S.rdr_v), sg, v2);
  }
}

// The voxel of n that t falls into; t below 1, or no number, is voxel 0 (converting it to an int first would
// give the host any value).
FMC_HD int voxel_index(double t, int n) { return t >= 1.0 ? (t < (double)n ? (int)t : n - 1) : 0; }

// Voxel of a position (wrapped into the cell; a slab's z clamped to its layers, whose lowest and
// highest hold no atom).
FMC_HD int voxel_of(const DevSystem& S, double x, double y, double z) {
  double s[3];
  if (S.cell.imcon == 6) {
    const CellGeom& c = S.cell;
    s[0] = c.slab[0] * x + c.slab[2] * y;
    s[1] = c.slab[1] * x + c.slab[3] * y;
    const int v0 = voxel_index((s[0] - floor(s[0])) * S.nvox[0], S.nvox[0]);
    const int v1 = voxel_index((s[1] - floor(s[1])) * S.nvox[1], S.nvox[1]);
    return (v0 * S.nvox[1] + v1) * S.nvox[2] + voxel_index((z - c.zlo) * c.rdz, S.nvox[2]);
  }
  frac_coords(S.cell, x, y, z, s);
  int v[3];
  for (int a = 0; a < 3; a++) v[a] = voxel_index((s[a] - floor(s[a])) * S.nvox[a], S.nvox[a]);
  return (v[0] * S.nvox[1] + v[1]) * S.nvox[2] + v[2];
}

// A guest-site update accepted on the host and not yet written to the device arrays (an
// insert appends a molecule to its species' segment, a delete removes one and shifts the rest
// down, a displacement overwrites one).  The next trial pass reads the guest sites as if the
// update were written (GuestView indices are those after it) and writes it once every block of
// that pass has read them.
constexpr int kMaxPendSites = 8;
struct PendingCommit {
  int op;       // 0: none; kInsert, kDelete, kDisplace
  int seg;      // species segment index (-1: none)
  int lo;       // first site of the molecule (insert: the segment's end before the insert)
  int ns;       // sites per molecule
  int seg_end;  // end of the segment before the update
  double4 site[kMaxPendSites];
  int type[kMaxPendSites];
};

// The guest site j of segment sg as if the pending update were written.
__device__ __forceinline__ void guest_site(const GuestView& G, const PendingCommit& P, int sg, int j, double4& a,
                                           int& t) {
  if (sg == P.seg && j >= P.lo) {
    if (P.op == kDelete) {  // the sites after the removed molecule, one molecule on
      j += P.ns;
    } else if (j < P.lo + P.ns) {  // the inserted or displaced molecule
      a = P.site[j - P.lo];
      t = P.type[j - P.lo];
      return;
    }
  }
  a = G.site[j];
  t = G.type[j];
}

// The plain path's pairs keep one arithmetic, every bit of it: what a site's sum rounds off decides a move that leaves
// its molecule in place (an angle drawn as exactly zero, any rotation of a single site), and so where a seeded
// host loop goes from there, whether it runs in the library or calls the drop-in routines.  So the root is rounded
// correctly and the roundings are written out; the images' products are fused as the compiler does.  A plain move
// takes as long as with image_dist2 and pair_table (10.1 us, 424 atoms).
template <int KIND>
__device__ __forceinline__ double plain_dist2(const CellGeom& c, double dx, double dy, double dz) {
  image<KIND>(c, dx, dy, dz);
  return fma(dz, dz, fma(dy, dy, __dmul_rn(dx, dx)));
}

__device__ __forceinline__ double plain_interp(double v0, double v1, double v2, double p) {
  const double t1 = fma(v1 - v0, p, v0), t2 = fma(v2 - v1, p - 1.0, v1);
  return fma(__dmul_rn(t2 - t1, p), 0.5, t1);
}

// Adds a pair's table energies: ec += cq erc(r), ev += vvv(r), with rs and off as in pair_table.
template <int KIND>
__device__ __forceinline__ void plain_table(const DevSystem& S, double rs, double cq, int off, double& ec, double& ev) {
  const double r = sqrt_exact(rs), x = __dmul_rn(r, S.rdr_e);
  const double f = (x - 0.5) + kMagic;  // floor(x) but for integers
  const int l = __double2loint(f);
  const double p = x - (f - kMagic);
  if (KIND != kPairGeneral) {
    const double2* tb = S.pair_tab + (off + l);
    const double2 a0 = tb[0], a1 = tb[1], a2 = tb[2];
    ec = fma(plain_interp(a0.x, a1.x, a2.x, p), cq, ec);
    ev = ev + plain_interp(a0.y, a1.y, a2.y, p);
  } else {
    const double* te = S.erc + l;
    ec = fma(plain_interp(te[0], te[1], te[2], p), cq, ec);
    if (off) {
      const double xv = __dmul_rn(r, S.rdr_v);
      const int lv = (int)xv;
      const double* tv = S.vvv + (off + lv);
      ev = ev + plain_interp(tv[0], tv[1], tv[2], xv - (double)lv);
    }
  }
}

// A thread's share of the pairs of one site with n candidates: two candidates in flight, distances
// first, then the tables, without a branch between (a lane whose candidate is missing or beyond the
// cut-off reads row 0 at the cut-off and adds zero).  fetch(i, atom, type) gives candidate i, leaving
// type at -1 for one to skip; prow: the table row's offset for each type, there once every thread has
// called ready(), which happens after the first candidates are on their way.
template <int KIND, class Fetch, class Ready>
__device__ __forceinline__ void pair_sum(const DevSystem& S, const int* prow, double px, double py, double pz,
                                         double chgea, int n, int tid, int nthr, Fetch fetch, Ready ready, double& ec,
                                         double& ev) {
  constexpr int U = 2;
  bool first = true;
  int base = tid;
  do {
    double4 a[U];
    int t[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      a[u] = make_double4(0.0, 0.0, 0.0, 0.0);
      t[u] = -1;
      if (base + u * nthr < n) fetch(base + u * nthr, a[u], t[u]);
    }
    if (first) ready();
    first = false;
    double rs[U], cq[U];
    int off[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const double rsq = plain_dist2<KIND>(S.cell, px - a[u].x, py - a[u].y, pz - a[u].z);
      const bool in = t[u] >= 0 && rsq < S.rcut2;
      const double qq = chgea * a[u].w;
      rs[u] = in ? rsq : S.rcut2;
      cq[u] = in && fabs(qq) > 1e-10 ? qq : 0.0;  // ewald2 skips smaller products
      off[u] = in ? prow[t[u]] : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) plain_table<KIND>(S, rs[u], cq[u], off[u], ec, ev);
    base += U * nthr;
  } while (base < n);
}

// A thread's share of one site's real-space energy against the framework (the voxel list of vl entries
// from vb) and the guest sites outside [ex_lo, ex_hi).
template <int KIND, class Ready>
__device__ __forceinline__ void site_pairs(const DevSystem& S, const GuestView& G, const PendingCommit& P,
                                           const int* prow, double px, double py, double pz, double q, int vb, int vl,
                                           int ex_lo, int ex_hi, int tid, int nthr, Ready ready, double& ec_fw,
                                           double& ev_fw, double& ec_g, double& ev_g) {
  const double chgea = q * kR4pie0;
  pair_sum<KIND>(S, prow, px, py, pz, chgea, vl, tid, nthr,
                 [&](int i, double4& a, int& t) {
                   a = S.vox_xyzq[vb + i];
                   t = S.vox_type[vb + i];
                 },
                 ready, ec_fw, ev_fw);
  for (int sg = 0; sg < G.nseg; sg++) {
    const int lo = G.seg_off[sg];
    pair_sum<KIND>(S, prow, px, py, pz, chgea, G.seg_len[sg], tid, nthr,
                   [&](int i, double4& a, int& t) {
                     if (lo + i < ex_lo || lo + i >= ex_hi) guest_site(G, P, sg, lo + i, a, t);
                   },
                   [] {}, ec_g, ev_g);
  }
}

// Deterministic block sum of NV values per thread (fixed shuffle tree + fixed warp order).
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* red /* >= 32*NV */) {
#pragma unroll
  for (int k = 0; k < NV; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) red[w * NV + k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double s = 0.0;
      for (int i = 0; i < nw; i++) s += red[i * NV + k];
      v[k] = s;
    }
  }
}

#endif  // __CUDACC__

}  // namespace fmc
