// force.cu -- contact forces and integration, FP64 (K3, K4, K5).
//
// Replaces CALC_FORCE_DEM (model/des/calc_force_dem.f:18-544) with CFRELVEL
// (model/des/cfrelvel.f:54-77), the wall contacts of
// CALC_DEM_FORCE_WITH_WALL_STL (model/des/calc_collision_wall_mod.f:180-629,
// GET/UPDATE/REMOVE_COLLISION 651-792, CFRELVEL_WALL 806-847,
// ClosestPtPointTriangle in stl_functions_des_mod.f:25-160), and
// CFUPDATEOLD + CFNEWVALUES (cfupdateold.f:33-41, cfnewvalues.f:669-812).
//
// The reference loops over owners LL and scatters each pair's force into
// FC(LL) and FC(I).  Here each pair is evaluated once (k_pairs, a lane per
// pair that may be in contact), which updates its tangential history in place and writes the
// terms of both particles into a contact record; then one thread per
// particle gathers (k_gather): walls first, then the records of the pairs
// it appears in as neighbour I owned by lower-index particles (ascending
// owner, from the transpose), its own row, then the remaining incoming
// pairs.  That is exactly the order in which the serial reference adds into
// FC(me)/TOW(me), so every particle's force is bit-identical to the serial
// reference without atomics.
//
// This file is compiled with -fmad=false: every FP64 expression rounds as
// the Fortran does (gfortran emits no FMA without -march).  sqrt and '/' are
// IEEE round-to-nearest in CUDA, as they are on the host; quotients by one
// divisor share its reciprocal and round the same (quotient()).
#include "dem_internal.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace demb {

struct PState {  // one particle's gathered state
  double x[3], v[3], w[3];
  double r, m;
  int ph;
};

// Contact part of one CC iteration of CALC_FORCE_DEM (calc_force_dem.f:
// 273-363) with CFRELVEL (cfrelvel.f:54-77) for owner L and neighbour I in
// contact; dist = x_I - x_L and d2 = |dist|^2 come from the apart test.
template <int COLL>
__device__ __forceinline__ void contact_force(const DevParams& p, const PState& L, const PState& I,
                                              const double dist[3], double d2, const double pin[3],
                                              double pout[3], PairRec& o) {
  const double rl = L.r, ri = I.r;
  const double r_lm = rl + ri;
  const double dmag = sqrt(d2);
  double nrm[3], dcl, half;
  contact_quotients(dist, dmag, rl, ri, nrm, dcl, half);
  const double overlap_n = r_lm - dmag;
  // CFRELVEL
  double vrel[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) vrel[c] = L.v[c] - I.v[c];
  const double dci = dmag - dcl;
  double osum[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) osum[c] = L.w[c] * dcl + I.w[c] * dci;
  double vrot[3];
  cross3(osum, nrm, vrot);
#pragma unroll
  for (int c = 0; c < 3; ++c) vrel[c] = vrel[c] + vrot[c];
  const double vrn = dot3(vrel, nrm);
  double vt[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) vt[c] = vrel[c] - vrn * nrm[c];
  const int ix = L.ph * MAXP + I.ph;
  const double rad_eff = (rl * ri) / (rl + ri);
  const double m_eff = (L.m * I.m) / (L.m + I.m);
  double kn, kt, etan, etat;
  if (COLL == DEM_COLL_HERTZ) {
    double so = sqrt(overlap_n);
    kn = p.hkn[ix] * so * sqrt(rad_eff);
    kt = p.hkt[ix] * so * sqrt(rad_eff);
    so = sqrt(so);
    etan = p.etan[ix] * so * sqrt(p.hkn[ix] * sqrt(rad_eff) * m_eff);
    etat = p.etat[ix] * so * sqrt(p.hkt[ix] * sqrt(rad_eff) * m_eff);
  } else {
    kn = p.kn; kt = p.kt;
    etan = p.etan[ix] * sqrt(m_eff);
    etat = p.etat[ix] * sqrt(m_eff);
  }
  double fn[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) fn[c] = -(kn * overlap_n * nrm[c] + etan * vrn * nrm[c]);
  double ot[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) ot[c] = p.dt * vt[c] + pin[c];
  const double mag = sqrt(dot3(ot, ot));
  double ft[3];
  if (mag > 0.0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) ft[c] = -kt * ot[c] - etat * vt[c];
    const double ftmd = sqrt(dot3(ft, ft));
    const double fnmd = p.mew * sqrt(dot3(fn, fn));
    if (ftmd > fnmd) {
      double tg[3];
      div3(ot, mag, tg);
#pragma unroll
      for (int c = 0; c < 3; ++c) ft[c] = -fnmd * tg[c];
#pragma unroll
      for (int c = 0; c < 3; ++c) ot[c] = (fnmd / kt) * tg[c];
    }
  } else {
    ft[0] = ft[1] = ft[2] = 0.0;
  }
  pout[0] = ot[0]; pout[1] = ot[1]; pout[2] = ot[2];
  o.dcl2 = dmag / 2.0 + half;
  o.dci2 = dmag - o.dcl2;
  cross3(nrm, ft, o.tf);
#pragma unroll
  for (int c = 0; c < 3; ++c) o.fc[c] = 0.0 + fn[c] + ft[c];
  o.kn = kn;
  o.ov = overlap_n;
}

// ---------------------------------------------------------------------------
// Walls

struct WallCtx {
  const double* __restrict__ vertex;   // [f][v][c]
  const double* __restrict__ norm_face;// [f][c]
  const int8_t* __restrict__ ignore_edge; // [f][4]
  const int* __restrict__ fbin_start;
  const FacetBinEntry* __restrict__ fbin;
  const int* __restrict__ dg_pijk;
  int* __restrict__ wall_fid;          // [i][cmax]
  double* __restrict__ wall_pft;       // [i][cmax][3]
  int nf;
};

__device__ __forceinline__ void closest_pt(const DevParams& p, const WallCtx& w, int f, const double pp[3],
                                           double cpt[3], bool& poe, int& edge) {
  poe = false; edge = 0;
  const double* V = w.vertex + 9 * (size_t)f;
  double a[3], b[3], c[3], ab[3], ac[3], ap[3], bp[3], cp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) { a[k] = V[k]; b[k] = V[3 + k]; c[k] = V[6 + k]; }
#pragma unroll
  for (int k = 0; k < 3; ++k) { ab[k] = b[k] - a[k]; ac[k] = c[k] - a[k]; ap[k] = pp[k] - a[k]; }
  const double d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  const int8_t* ig = w.ignore_edge + 4 * (size_t)f;
  if (d1 < 0.0 && d2 < 0.0) {
    for (int k = 0; k < 3; ++k) cpt[k] = a[k];
    poe = true; if (ig[1]) cpt[0] = UNDEFINED_D; edge = 1; return;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) bp[k] = pp[k] - b[k];
  const double d3 = dot3(ab, bp), d4 = dot3(ac, bp);
  if (d3 > 0.0 && d4 < d3) {
    for (int k = 0; k < 3; ++k) cpt[k] = b[k];
    poe = true; if (ig[1]) cpt[0] = UNDEFINED_D; edge = 1; return;
  }
  const double vc = d1 * d4 - d3 * d2;
  if (vc < 0.0 && d1 > 0.0 && d3 < 0.0) {
    const double v = d1 / (d1 - d3);
    for (int k = 0; k < 3; ++k) cpt[k] = a[k] + v * ab[k];
    poe = true; if (ig[1]) cpt[0] = UNDEFINED_D; edge = 1; return;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) cp[k] = pp[k] - c[k];
  const double d5 = dot3(ab, cp), d6 = dot3(ac, cp);
  if (d6 > 0.0 && d5 < d6) {
    for (int k = 0; k < 3; ++k) cpt[k] = c[k];
    poe = true; if (ig[2]) cpt[0] = UNDEFINED_D; edge = 2; return;
  }
  const double vb = d5 * d2 - d1 * d6;
  if (vb < 0.0 && d2 > 0.0 && d6 < 0.0) {
    const double ww = d2 / (d2 - d6);
    for (int k = 0; k < 3; ++k) cpt[k] = a[k] + ww * ac[k];
    poe = true; if (ig[2]) cpt[0] = UNDEFINED_D; edge = 2; return;
  }
  const double va = d3 * d6 - d5 * d4;
  if (va < 0.0 && (d4 - d3) > 0.0 && (d5 - d6) > 0.0) {
    const double ww = (d4 - d3) / ((d4 - d3) + (d5 - d6));
    for (int k = 0; k < 3; ++k) cpt[k] = b[k] + ww * (c[k] - b[k]);
    poe = true; if (ig[3]) cpt[0] = UNDEFINED_D; edge = 3; return;
  }
  const double denom = 1.0 / (va + vb + vc);
  const double v = vb * denom, ww = vc * denom;
  for (int k = 0; k < 3; ++k) cpt[k] = a[k] + ab[k] * v + ac[k] * ww;
  if (p.no_k) cpt[2] = pp[2];
}

__device__ __forceinline__ void remove_collision(const DevParams& p, const WallCtx& w, int me, int f) {
  int* fid = w.wall_fid + (size_t)me * p.cmax;
  for (int s = 0; s < p.cmax; ++s) if (fid[s] == f) { fid[s] = -1; return; }
}

// returns slot index, or -1 on overflow
__device__ __forceinline__ int get_collision(const DevParams& p, const WallCtx& w, int me, int f, int cell,
                                             double out[3]) {
  int* fid = w.wall_fid + (size_t)me * p.cmax;
  double* wp = w.wall_pft + (size_t)me * p.cmax * 3;
  int free_index = -1;
  for (int s = 0; s < p.cmax; ++s) {
    int v = fid[s];
    if (f == v) { out[0] = wp[3 * s]; out[1] = wp[3 * s + 1]; out[2] = wp[3 * s + 2]; return s; }
    else if (v == -1) free_index = s;
  }
  if (free_index == -1) {
    for (int s = 0; s < p.cmax && free_index == -1; ++s) {
      bool in_cell = false;
      for (int q = w.fbin_start[cell]; q < w.fbin_start[cell + 1]; ++q)
        if (fid[s] == w.fbin[q].id) { in_cell = true; break; }
      if (!in_cell) free_index = s;
    }
  }
  if (free_index == -1) return -1;
  fid[free_index] = f;
  wp[3 * free_index] = 0.0; wp[3 * free_index + 1] = 0.0; wp[3 * free_index + 2] = 0.0;
  out[0] = out[1] = out[2] = 0.0;
  return free_index;
}

// The wall contacts of one particle in a cell with facets, by a group of
// WALL_LANES lanes (mask gm, lane gl of the group).  A cell of a triangulated
// wall holds tens of facets and a particle touches one or two of them, so the
// lanes test the cell's facets side by side (extent, plane and closest point:
// a chain of loads and FP64 arithmetic each) and the few that matter are then
// taken in the facets' order, as the reference's loop does: the history slots
// (GET/REMOVE_COLLISION choose and free slots in that order) and the sums of
// the force and torque terms.  `live` says whether any history slot may be in
// use; when none is, no slot is searched for the facets it does not touch
// (REMOVE_COLLISION would find nothing).  The particle's velocity, spin, mass
// and phase are read by the lanes in contact only.  f and t are the same in
// every lane; returns the number of contacts.
// Five hoppers of 160,000 spheres in all (a triangulated cone, 128 facets):
// 143 us per step with a thread per particle, of it 99 us this, and 68 us so.
constexpr int WALL_LANES = 8;
template <int COLL>
__device__ int wall_contacts(const DevParams& p, const WallCtx& w, int me, const double x[3], double r, bool live,
                             unsigned gm, int gl, const double4* __restrict__ vel4,
                             const double4* __restrict__ omg4, const uint8_t* __restrict__ phase, double f[3],
                             double t[3], unsigned& eflags) {
  const int cell = p.cell_off + w.dg_pijk[me] - 1;
  const int fs = w.fbin_start[cell], fe = w.fbin_start[cell + 1];
  const int g0 = __ffs(gm) - 1;  // the group's first lane in the warp
  const double radsq = r * r;
  int nwc = 0;
  for (int q0 = fs; q0 < fe; q0 += WALL_LANES) {
    const int q = q0 + gl;
    enum { NONE, MISS, HIT };
    int what = NONE, nf = -1;
    double dist[3] = {0.0, 0.0, 0.0}, distsq = 0.0;
    if (q < fe) {
      const FacetBinEntry e = w.fbin[q];
      nf = e.id;
      what = MISS;
      const double xd = x[e.dir];
      if (!(e.mn > xd + r) && !(e.mx < xd - r)) {
        const double* V = w.vertex + 9 * (size_t)nf;
        const double* N = w.norm_face + 3 * (size_t)nf;
        double d1[3] = {V[0] - x[0], V[1] - x[1], V[2] - x[2]};
        double nn[3] = {N[0], N[1], N[2]};
        const double line_t = dot3(d1, nn);
        if (!(line_t <= -1.0001 * r)) {
          double cpt[3]; bool poe; int edge;
          closest_pt(p, w, nf, x, cpt, poe, edge);
#pragma unroll
          for (int c = 0; c < 3; ++c) dist[c] = cpt[c] - x[c];
          distsq = dot3(dist, dist);
          if (!(distsq >= radsq - SMALL_NUMBER))
            what = (poe && w.ignore_edge[4 * (size_t)nf + edge]) ? NONE : HIT;
        }
      }
    }
    const unsigned hits = (__ballot_sync(gm, what == HIT) & gm) >> g0;
    unsigned gone = 0;  // facets not touched that a history slot still holds
    if (live) {
      bool held = false;
      if (what == MISS) {
        const int* fid = w.wall_fid + (size_t)me * p.cmax;
        for (int s = 0; s < p.cmax; ++s) held = held || fid[s] == nf;
      }
      gone = (__ballot_sync(gm, held) & gm) >> g0;
    }
    int slot = -1;
    double hist[3] = {0.0, 0.0, 0.0};
    for (unsigned todo = hits | gone; todo; todo &= todo - 1u) {
      if (gl == __ffs(todo) - 1) {
        if (what == HIT) slot = get_collision(p, w, me, nf, cell, hist);
        else remove_collision(p, w, me, nf);
      }
      __syncwarp(gm);  // the next facet sees the slots as this one left them
    }
    if (!hits) continue;
    double fn[3] = {0.0, 0.0, 0.0}, ft[3] = {0.0, 0.0, 0.0}, tq[3] = {0.0, 0.0, 0.0}, rl[3] = {0.0, 0.0, 0.0};
    int terms = 0;  // 1: force and torque, 2: rolling friction too
    if (what == HIT && slot < 0) eflags |= EF_WALL_SLOTS;
    if (slot >= 0) {
      const double4 vb = vel4[me], wb = omg4[me];
      const double sv[3] = {vb.x, vb.y, vb.z}, sw[3] = {wb.x, wb.y, wb.z}, m = vb.w;
      const int ph = phase[me];
      const double distmod = sqrt(distsq);
      double nrm[3] = {dist[0], dist[1], dist[2]};
      if (distsq > 0) div3(dist, distmod, nrm);
      const double overlap_n = r - distmod;
      double wxn[3]; cross3(sw, nrm, wxn);
      double vrel[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) { vrel[c] = sv[c] + distmod * wxn[c]; vrel[c] = vrel[c] - (0.0 + 0.0); }
      const double vrn = dot3(vrel, nrm);
      double vt[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) vt[c] = vrel[c] - vrn * nrm[c];
      double kn_w, kt_w, etan_w, etat_w;
      if (COLL == DEM_COLL_HERTZ) {
        double so = 0.0;
        if (overlap_n > 0) so = sqrt(overlap_n);
        kn_w = p.hkwn[ph] * so * sqrt(r);
        kt_w = p.hkwt[ph] * so * sqrt(r);
        etan_w = p.etanw[ph] * sqrt(so) * sqrt(p.hkwn[ph] * sqrt(r) * m);
        etat_w = p.etatw[ph] * sqrt(so) * sqrt(p.hkwt[ph] * sqrt(r) * m);
      } else {
        kn_w = p.kn_w; kt_w = p.kt_w;
        etan_w = p.etanw[ph] * sqrt(m);
        etat_w = p.etatw[ph] * sqrt(m);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) fn[c] = -(kn_w * overlap_n * nrm[c] + etan_w * vrn * nrm[c]);
      double ot[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) ot[c] = p.dt * vt[c] + hist[c];
      const double mag = sqrt(dot3(ot, ot));
      if (mag > 0.0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) ft[c] = -kt_w * ot[c] - etat_w * vt[c];
        const double ftmd = sqrt(dot3(ft, ft));
        const double fnmd = p.mew_w * sqrt(dot3(fn, fn));
        if (ftmd > fnmd) {
          double tg[3];
          div3(ot, mag, tg);
#pragma unroll
          for (int c = 0; c < 3; ++c) ft[c] = -fnmd * tg[c];
#pragma unroll
          for (int c = 0; c < 3; ++c) ot[c] = (fnmd / kt_w) * tg[c];
        }
      }
      double* wp = w.wall_pft + ((size_t)me * p.cmax + slot) * 3;  // UPDATE_COLLISION
      wp[0] = ot[0]; wp[1] = ot[1]; wp[2] = ot[2];
      double nxf[3]; cross3(nrm, ft, nxf);
#pragma unroll
      for (int c = 0; c < 3; ++c) tq[c] = distmod * nxf[c];
      terms = 1;
      if (p.mew_rw > 0.0) {
        const double om = sqrt(dot3(sw, sw));
        if (om > 0.0) {
          terms = 2;
#pragma unroll
          for (int c = 0; c < 3; ++c) rl[c] = p.mew_rw * (2.0 * r) * kn_w * overlap_n * sw[c];
          div3(rl, om, rl);
#pragma unroll
          for (int c = 0; c < 3; ++c) rl[c] = -rl[c];
        }
      }
    }
    for (unsigned todo = hits; todo; todo &= todo - 1u) {
      const int b = g0 + __ffs(todo) - 1;
      const int have = __shfl_sync(gm, terms, b);
      if (!have) continue;
      ++nwc;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double a = __shfl_sync(gm, fn[c], b), d = __shfl_sync(gm, ft[c], b), e = __shfl_sync(gm, tq[c], b);
        f[c] = f[c] + a + d;
        t[c] = t[c] + e;
      }
      if (have == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) t[c] = t[c] + __shfl_sync(gm, rl[c], b);
      }
    }
  }
  return nwc;
}

// ---------------------------------------------------------------------------
// Squared distance from x to the closest point of triangle (a, b, c): the
// Voronoi-region walk over vertices, edges and face (C. Ericson, Real-Time
// Collision Detection, 2005, section 5.1.5), with no edge or vertex left out.
__device__ __forceinline__ double tri_dist2(const double* __restrict__ V, const double x[3]) {
  double a[3], ab[3], ac[3], ap[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) { a[k] = V[k]; ab[k] = V[3 + k] - a[k]; ac[k] = V[6 + k] - a[k]; ap[k] = x[k] - a[k]; }
  const double d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  double q[3];
  auto at = [&](double u, double v) {
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = a[k] + u * ab[k] + v * ac[k];
  };
  if (d1 <= 0.0 && d2 <= 0.0) { at(0.0, 0.0); goto done; }
  {
    double bp[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) bp[k] = ap[k] - ab[k];
    const double d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3 >= 0.0 && d4 <= d3) { at(1.0, 0.0); goto done; }
    const double vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) { at(d1 / (d1 - d3), 0.0); goto done; }
    double cp[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) cp[k] = ap[k] - ac[k];
    const double d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) { at(0.0, 1.0); goto done; }
    const double vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) { at(0.0, d2 / (d2 - d6)); goto done; }
    const double va = d3 * d6 - d5 * d4;
    if (va <= 0.0 && (d4 - d3) >= 0.0 && (d5 - d6) >= 0.0) {
      const double w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
      at(1.0 - w, w);
      goto done;
    }
    const double den = 1.0 / (va + vb + vc);
    at(vb * den, vc * den);
  }
done:
  double d[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) d[k] = x[k] - q[k];
  return dot3(d, d);
}

// Clearance of every NORMAL particle in a DES cell with facets from those
// facets at a build (valid while the particle stays in that cell: the
// per-step placement of a periodic system sets it to -1, unknown, when the
// particle changes cell): min over the cell's facets of |x - closest point| - r,
// less a margin of 1e-6 r for the rounding of the closest point, rounded
// down to float.  A particle whose clearance exceeds the displacement bound
// since the build touches none of them (the reference's contact test is
// |x - c|^2 < r^2 - SMALL_NUMBER), so with no history it has no wall work.
template <bool B>
__global__ void k_wall_gaps(DevParams p0, BatchView bv, WallCtx w, const double4* __restrict__ pos4,
                            const int8_t* __restrict__ state, const uint8_t* __restrict__ wall_cand,
                            float* __restrict__ wgap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p0.n) return;
  // a particle that is not NORMAL now may become so before the next build
  // (ENTERING, EXITING): clearance unknown, its walls are checked
  if (state[i] != DEM_STATE_NORMAL) { wgap[i] = -1.0f; return; }
  // no facets in its cell: none to touch while it stays there (a move to
  // another cell before the next build clears the screen, see dg_place users)
  if (!wall_cand[i]) { wgap[i] = FLT_MAX; return; }
  const DevParams& p = sysp<B>(p0, bv, i);
  const int cell = p.cell_off + w.dg_pijk[i] - 1;
  const double4 a = pos4[i];
  const double x[3] = {a.x, a.y, a.z};
  double dmin2 = HUGE_VAL;
  for (int q = w.fbin_start[cell]; q < w.fbin_start[cell + 1]; ++q)
    dmin2 = fmin(dmin2, tri_dist2(w.vertex + 9 * (size_t)w.fbin[q].id, x));
  wgap[i] = __double2float_rd(sqrt(dmin2) - a.w - 1e-6 * a.w);
}

// Kernel 1: wall contacts.  A block screens blockDim.x * J particles for those
// with wall work this step -- NORMAL particles whose DES cell holds facets and
// whose clearance at the last build does not exceed the displacement bound
// since, and NORMAL particles whose history slots may be in use -- into a list
// in shared memory, and its groups of WALL_LANES lanes take the listed
// particles.  A particle's wall force and torque, the first terms of FC/TOW in
// the reference's order (CALC_DEM_FORCE_WITH_WALL_STL runs before the pair
// loop, calc_force_dem.f:113), go to wf; they depend on that particle alone,
// so the order of the list does not matter.  With J = 4 a thread's four flags
// arrive in one 32-bit load per array and its clearances in one float4.
constexpr int WALL_T = 256;
__device__ __forceinline__ unsigned wall_need(unsigned st, unsigned live, unsigned cand, float gap, double bound) {
  return (st == (unsigned)(uint8_t)DEM_STATE_NORMAL && (live || (cand && !((double)gap > bound)))) ? 1u : 0u;
}
struct WallArgs {
  WallCtx w;
  int n;       // particles
  int blocks;  // blocks that do the wall work
  const float* __restrict__ wgap;
  uint8_t* __restrict__ live;
  const uint8_t* __restrict__ cand;
  double* __restrict__ wf;
  uint8_t* __restrict__ hit;
};
template <int COLL, bool B, int J>
__device__ __forceinline__ void wall_block(const DevParams& p0, const BatchView& bv, const WallArgs& wa, int block,
                                           double bound, const int8_t* __restrict__ state,
                                           const double4* __restrict__ pos4, const double4* __restrict__ vel4,
                                           const double4* __restrict__ omg4, const uint8_t* __restrict__ phase,
                                           ContactCount* __restrict__ count, DevErr* __restrict__ err) {
  static_assert(J == 1 || J == 4, "one particle per thread, or four");
  const WallCtx& w = wa.w;
  const int n = wa.n;
  const float* __restrict__ wgap = wa.wgap;
  uint8_t* __restrict__ wall_live = wa.live;
  const uint8_t* __restrict__ wall_cand = wa.cand;
  __shared__ int s_list[WALL_T * J];
  __shared__ int s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const int i0 = J * (block * (int)blockDim.x + (int)threadIdx.x);
  unsigned need = 0;  // bit j: particle i0+j has wall work
  if (J == 4 && i0 + 3 < n) {  // the arrays are separate allocations: 256-byte aligned
    const uint32_t st = *reinterpret_cast<const uint32_t*>(state + i0);
    const uint32_t lv = *reinterpret_cast<const uint32_t*>(wall_live + i0);
    const uint32_t cd = *reinterpret_cast<const uint32_t*>(wall_cand + i0);
    const float4 g = *reinterpret_cast<const float4*>(wgap + i0);
    need = wall_need(st & 255u, lv & 255u, cd & 255u, g.x, bound) |
           (wall_need((st >> 8) & 255u, (lv >> 8) & 255u, (cd >> 8) & 255u, g.y, bound) << 1) |
           (wall_need((st >> 16) & 255u, (lv >> 16) & 255u, (cd >> 16) & 255u, g.z, bound) << 2) |
           (wall_need(st >> 24, lv >> 24, cd >> 24, g.w, bound) << 3);
  } else {
#pragma unroll
    for (int j = 0; j < J; ++j)
      if (i0 + j < n)
        need |= wall_need((uint8_t)state[i0 + j], wall_live[i0 + j], wall_cand[i0 + j], wgap[i0 + j], bound) << j;
  }
  const int lane = threadIdx.x & 31;
  const int mine = __popc(need);
  int incl = mine;  // inclusive scan of the counts over the warp
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int base = 0;
  if (lane == 31 && incl) base = atomicAdd(&s_n, incl);
  base = __shfl_sync(0xffffffffu, base, 31);
  int at = base + incl - mine;
  for (int j = 0; j < J; ++j)
    if ((need >> j) & 1u) s_list[at++] = i0 + j;
  __syncthreads();
  const int nw = s_n;
  unsigned long long nwc = 0;
  unsigned eflags = 0;
  const int gl = lane & (WALL_LANES - 1);
  const unsigned gm = ((1u << WALL_LANES) - 1u) << (lane & ~(WALL_LANES - 1));
  for (int k = threadIdx.x / WALL_LANES; k < nw; k += blockDim.x / WALL_LANES) {
    const int me = s_list[k];
    const DevParams& p = sysp<B>(p0, bv, me);
    if (!wall_cand[me]) {
      // no facet near: clear the history once (calc_collision_wall_mod.f:194-198)
      int* fid = w.wall_fid + (size_t)me * p.cmax;
      double* wp = w.wall_pft + (size_t)me * p.cmax * 3;
      for (int s = gl; s < p.cmax; s += WALL_LANES) fid[s] = -1;
      for (int s = gl; s < 3 * p.cmax; s += WALL_LANES) wp[s] = 0.0;
      if (gl == 0) wall_live[me] = 0;
      continue;
    }
    const double4 a = pos4[me];
    const double x[3] = {a.x, a.y, a.z};
    double f[3] = {0.0, 0.0, 0.0}, t[3] = {0.0, 0.0, 0.0};
    const bool live = wall_live[me] != 0;
    const int hit = wall_contacts<COLL>(p, w, me, x, a.w, live, gm, gl, vel4, omg4, phase, f, t, eflags);
    if (gl == 0) {
      nwc += hit;
      bool used = hit > 0;
      if (!hit && live) {
        const int* fid = w.wall_fid + (size_t)me * p.cmax;
        for (int s = 0; s < p.cmax; ++s) used = used || fid[s] != -1;
      }
      if (used != live) wall_live[me] = used ? 1 : 0;
      if (hit) {
        // the gather reads the wall terms only for particles marked here
        double* o = wa.wf + 6 * (size_t)me;
        o[0] = f[0]; o[1] = f[1]; o[2] = f[2]; o[3] = t[0]; o[4] = t[1]; o[5] = t[2];
        wa.hit[me] = 1;
      }
    }
  }
  __syncwarp();
  for (int o = 16; o > 0; o >>= 1) {
    nwc += __shfl_down_sync(0xffffffffu, nwc, o);
    eflags |= __shfl_down_sync(0xffffffffu, eflags, o);
  }
  if (lane == 0) {
    if (nwc) atomicAdd(&count->walls, nwc);
    if (eflags) atomicOr(&err->flags, eflags);
  }
}

template <int COLL, bool B, int J>
__global__ void __launch_bounds__(WALL_T)
k_walls(DevParams p0, BatchView bv, WallArgs wa, const double* __restrict__ skin,
        const unsigned* __restrict__ pending, const int8_t* __restrict__ state, const double4* __restrict__ pos4,
        const double4* __restrict__ vel4, const double4* __restrict__ omg4, const uint8_t* __restrict__ phase,
        ContactCount* __restrict__ count, DevErr* __restrict__ err) {
  wall_block<COLL, B, J>(p0, bv, wa, blockIdx.x, displacement_bound(skin, pending), state, pos4, vel4, omg4, phase,
                         count, err);
}

// Kernel 2 (per pair): one CC iteration of CALC_FORCE_DEM, evaluated once
// per pair.  A warp takes a window of WIN_PAIRS pairs, queues those that may
// be in contact (screen_window) and gives each lane one of the queue.  The
// apart test needs only the two positions; velocities, spins and masses are
// gathered only for pairs in contact.  The tangential history PFT is updated
// in place (only this kernel reads it).  pflag keeps, per pair, PF_CONTACT
// (in contact at this pass) and PF_HIST (history nonzero), so a pair that
// stays apart with a zero history costs no history traffic; in_flag keeps the
// neighbour's view of PF_CONTACT in transpose order.  The contact terms go to
// a record that both particles read back in kernel 3, and both particles of a
// contact are marked in `touched`.
// Bound by latency and by the accesses the L1 takes in, not by DRAM (a fifth of
// its throughput).  The 1,000,000-sphere bed with 1.67 M of its 4.4 M pairs in contact:
// 248 us with four pairs per thread (12 of 32 lanes in contact at a time) and
// records written 8 bytes at a time, 156 us with full warps and 32-byte
// accesses, 141 us with the loads in three dependent rounds instead of five
// and the quotients side by side.
// With JW > 0 the first wa.blocks blocks do the wall work instead (JW
// particles per thread): it reads the same state and writes disjoint arrays,
// and in one launch the two run side by side with no second stream to fork
// and join.
template <int COLL, bool B, int JW>
__global__ void __launch_bounds__(256, 2)
k_pairs(DevParams p0, BatchView bv, WallArgs wa, const int* __restrict__ d_np, long long cap, const int* __restrict__ owner,
        const int* __restrict__ nbrs, const int* __restrict__ in_pos, const double4* __restrict__ pos4,
        const double4* __restrict__ vel4, const double4* __restrict__ omg4, const int8_t* __restrict__ state,
        const uint8_t* __restrict__ phase, double* __restrict__ pft, uint8_t* __restrict__ pflag,
        uint8_t* __restrict__ in_flag, uint8_t* __restrict__ touched, const float* __restrict__ pgap,
        const double* __restrict__ skin, const unsigned* __restrict__ pending, RecStore rec,
        ContactCount* __restrict__ count, DevErr* __restrict__ err) {
  __shared__ WinQueue s_queue[256 / 32];
  const int z = pdl_wait();
  pdl_next();
  const double bound = displacement_bound(skin + z, pending + z);
  int block = blockIdx.x + z, blocks = gridDim.x;
  if (JW) {
    if (block < wa.blocks) {
      wall_block<COLL, B, JW ? JW : 1>(p0, bv, wa, block, bound, state, pos4, vel4, omg4, phase, count, err);
      return;
    }
    block -= wa.blocks;
    blocks -= wa.blocks;
  }
  // persistent grid-stride loop over the device-side pair count (the grid
  // size does not depend on the list, so the launch can live in a graph)
  const long long np = min((long long)d_np[z], cap);
  const float reach = __double2float_ru(2.0 * bound);
  unsigned long long ncont = 0;
  unsigned eflags = 0;
  WinQueue* queue = &s_queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)WIN_PAIRS * ((blocks * (int)blockDim.x) >> 5);
  for (long long w0 = (long long)WIN_PAIRS * ((block * (int)blockDim.x + (int)threadIdx.x) >> 5) + z; w0 < np; w0 += stride) {
    const int nq = screen_window(w0, np, pflag, in_flag, in_pos, pgap, owner, nbrs, reach, queue);
    for (int k = lane; k < nq; k += 32) {
      const int e = queue->e[k];
      const long long cc = w0 + (e & (WIN_PAIRS - 1));
      const uint8_t f0 = (uint8_t)(e >> 7);
      const int2 who = queue->who[k];
      const int ll = who.x, i = who.y;
      uint8_t f = f0 & PF_HIST;  // NONEXISTENT partner or zero distance: history kept
      // the states and the positions in one round of loads (any slot's
      // position can be read; it is used only for existing particles), with
      // the history and, for a contact of the last pass, which is nearly always
      // one of this, the motion (1 % of a step of the beds)
      const double4 a = ld32(pos4 + ll), b = ld32(pos4 + i);
      const int8_t sl = state[ll], si = state[i];
      double pin[3] = {0.0, 0.0, 0.0};
      if (f0 & PF_HIST) { pin[0] = pft[cc]; pin[1] = pft[cap + cc]; pin[2] = pft[2 * cap + cc]; }
      const bool was = f0 & PF_CONTACT;
      double4 va, vb, wa, wb;
      if (was) { va = ld32(vel4 + ll); vb = ld32(vel4 + i); wa = ld32(omg4 + ll); wb = ld32(omg4 + i); }
      if (si != DEM_STATE_NONEXISTENT && sl != DEM_STATE_NONEXISTENT) {
        const DevParams& p = sysp<B>(p0, bv, ll);
        PState L, I;
        L.x[0] = a.x; L.x[1] = a.y; L.x[2] = a.z; L.r = a.w;
        I.x[0] = b.x; I.x[1] = b.y; I.x[2] = b.z; I.r = b.w;
        const double r_lm = L.r + I.r;
        double dist[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double pj = I.x[c];
          double s = periodic_shift(p, c, pj - L.x[c]);
          if (s != 0.0) pj = pj + s;
          dist[c] = pj - L.x[c];
        }
        const double d2 = dot3(dist, dist);
        if (d2 > (r_lm - SMALL_NUMBER) * (r_lm - SMALL_NUMBER)) {
          if (f0 & PF_HIST) { pft[cc] = 0.0; pft[cap + cc] = 0.0; pft[2 * cap + cc] = 0.0; }
          f = 0;
        } else if (d2 == 0.0) {
          eflags |= EF_ZERO_DIST;
          err->zero_a = ll; err->zero_b = i;
        } else {
          if (!was) { va = ld32(vel4 + ll); vb = ld32(vel4 + i); wa = ld32(omg4 + ll); wb = ld32(omg4 + i); }
          L.v[0] = va.x; L.v[1] = va.y; L.v[2] = va.z; L.m = va.w;
          I.v[0] = vb.x; I.v[1] = vb.y; I.v[2] = vb.z; I.m = vb.w;
          L.w[0] = wa.x; L.w[1] = wa.y; L.w[2] = wa.z;
          I.w[0] = wb.x; I.w[1] = wb.y; I.w[2] = wb.z;
          // one solids phase: no phase to look up
          L.ph = p.nph > 1 ? phase[ll] : 0;
          I.ph = p.nph > 1 ? phase[i] : 0;
          double pout[3];
          PairRec r;
          contact_force<COLL>(p, L, I, dist, d2, pin, pout, r);
          pft[cc] = pout[0]; pft[cap + cc] = pout[1]; pft[2 * cap + cc] = pout[2];
          st32(rec.main + 2 * cc, r.fc[0], r.fc[1], r.fc[2], r.tf[0]);
          st32(rec.main + 2 * cc + 1, r.tf[1], r.tf[2], r.dcl2, r.dci2);
          if (p.mew_r > 0.0) rec.roll[cc] = make_double2(r.kn, r.ov);
          touched[ll] = 1;
          touched[i] = 1;
          f = PF_CONTACT | ((pout[0] != 0.0 || pout[1] != 0.0 || pout[2] != 0.0) ? PF_HIST : 0);
          ++ncont;
        }
      }
      if (f != f0) {
        pflag[cc] = f;
        if ((f ^ f0) & PF_CONTACT) in_flag[in_pos[cc]] = f & PF_CONTACT;
      }
    }
    __syncwarp();  // the queue is read before the next window fills it
  }
  for (int o = 16; o > 0; o >>= 1) {
    ncont += __shfl_down_sync(0xffffffffu, ncont, o);
    eflags |= __shfl_down_sync(0xffffffffu, eflags, o);
  }
  if (lane == 0) {
    if (ncont) atomicAdd(&count->pairs, ncont);
    if (eflags) atomicOr(&err->flags, eflags);
  }
}

// Rolling-friction torque of one particle in a pair (calc_force_dem.f:491-506):
// -MEW_R*(2*R)*KN_DES*OVERLAP_N*OMEGA/|OMEGA|, evaluated left to right; om is
// |OMEGA| and its reciprocal, the same for all of the particle's contacts.
__device__ __forceinline__ void add_rolling(const DevParams& p, double r, const double w[3], double2 om,
                                            const PairRec& q, double t[3]) {
  const double a = p.mew_r * (2.0 * r) * q.kn * q.ov;
  const double aw[3] = {a * w[0], a * w[1], a * w[2]};
  double d[3];
  div3(aw, om.x, om.y, d);
#pragma unroll
  for (int c = 0; c < 3; ++c) t[c] = t[c] + -d[c];
}

// One pair's terms on one of its particles: the owner adds +FC and DCL2*TF,
// the neighbour -FC and DCI2*TF (calc_force_dem.f:466-506).
template <bool NBR>
__device__ __forceinline__ void add_pair_terms(const DevParams& p, const PairRec& o, bool roll, double r,
                                               const double w[3], double2 om, double f[3], double t[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) f[c] = NBR ? f[c] - o.fc[c] : f[c] + o.fc[c];
#pragma unroll
  for (int c = 0; c < 3; ++c) t[c] = t[c] + (NBR ? o.dci2 : o.dcl2) * o.tf[c];
  if (roll && om.x > 0.0) add_rolling(p, r, w, om, o, t);
}

__device__ __forceinline__ PairRec load_record(const RecStore& rec, int cc, bool roll) {
  PairRec r;
  const double4 a = ld32(rec.main + 2 * (size_t)cc), b = ld32(rec.main + 2 * (size_t)cc + 1);
  r.fc[0] = a.x; r.fc[1] = a.y; r.fc[2] = a.z;
  r.tf[0] = a.w; r.tf[1] = b.x; r.tf[2] = b.y;
  r.dcl2 = b.z; r.dci2 = b.w;
  r.kn = 0.0; r.ov = 0.0;
  if (roll) { const double2 q = rec.roll[cc]; r.kn = q.x; r.ov = q.y; }
  return r;
}

// The records of the contacts among the entries [q, e) of the particle's
// incoming list (NBR, pair indices in in_pair) or its own row, in order, 32
// entries at a time: the contact flags, which lie in the entries' order, are
// read as words, then the flagged records, each issued before the previous
// one is added.
template <bool NBR>
__device__ __forceinline__ void add_range(const DevParams& p, int q, int e, const uint8_t* __restrict__ flags,
                                          const int2* __restrict__ in_pair, const RecStore& rec, bool roll, double r,
                                          const double w[3], double2 om, double f[3], double t[3]) {
  for (int base = q; base < e; base += 32) {
    unsigned mask = contact_mask(flags, base, min(32, e - base));
    if (!mask) continue;
    auto pair = [&](int k) { return NBR ? in_pair[base + k].y : base + k; };
    PairRec cur = load_record(rec, pair(__ffs(mask) - 1), roll);
    mask &= mask - 1u;
    while (true) {
      const bool more = mask != 0u;
      PairRec nxt;
      if (more) {
        nxt = load_record(rec, pair(__ffs(mask) - 1), roll);
        mask &= mask - 1u;
      }
      add_pair_terms<NBR>(p, cur, roll, r, w, om, f, t);
      if (!more) break;
      cur = nxt;
    }
  }
}

// Kernel 3 (per particle): sums FC/TOW in the serial reference's order --
// wall terms, pairs owned by lower-index particles (ascending owner), the
// particle's own row, pairs owned by higher-index particles (in_mid is the
// first of them; a NORMAL particle has none) -- and either stores them
// (MODE 0) or integrates them in place of CFNEWVALUES (MODE 1 = Euler, MODE
// 2 = Adams-Bashforth).
// Same bed: 179 us with records read 8 bytes at a time and each incoming
// pair's flag looked up at random, 134 us now.  Bound by latency at the
// 24 warps its 80 registers allow (12 % of a step slower at 16 warps and no
// spills, 18 % at 32 and 90 bytes spilled; staged through shared memory 15 to 20
// %, the L1 it takes being worth more).
template <int MODE, bool B>
__global__ void __launch_bounds__(256, 3)
k_gather(DevParams p0, BatchView bv, const double4* __restrict__ pos_c, const double4* __restrict__ vel_c,
         const double4* __restrict__ omg_c, double4* __restrict__ pos_n, double4* __restrict__ vel_n,
         double4* __restrict__ omg_n, const int8_t* __restrict__ state, const double* __restrict__ wf,
         const int* __restrict__ row_end, const int* __restrict__ in_start, const int* __restrict__ in_mid,
         const int2* __restrict__ in_pair, const uint8_t* __restrict__ pflag, const uint8_t* __restrict__ in_flag,
         uint8_t* __restrict__ touched, uint8_t* __restrict__ wall_hit, RecStore rec,
         double* __restrict__ fc, double* __restrict__ tow, double* __restrict__ acc_old,
         double* __restrict__ rot_acc_old, unsigned* __restrict__ vslot,
         CellOut cells, StepEnd end) {
  const int z = pdl_wait();
  pdl_next();
  if (MODE != 0) end_step(end);
  const int me = blockIdx.x * blockDim.x + threadIdx.x + z;
  if (me >= p0.n) return;
  const DevParams& p = sysp<B>(p0, bv, me);
  const int8_t st = state[me];
  // the contacts of this pass; a particle in none has no terms to add (the
  // bounds of its lists are loaded all the same, beside the mark, which takes
  // a round of loads out of the others' chain: 342 to 334 us per step of the
  // bed, 57.5 to 56.1 us of a gas of 200,003)
  const bool wh = wall_hit[me] != 0, ph = touched[me] != 0;
  const int is = in_start[me], ie = in_start[me + 1], mid = in_mid[me];
  const int rs = row_end[me ? me - 1 : 0], re = row_end[me];
  if (wh) wall_hit[me] = 0;
  if (ph) touched[me] = 0;
  // no torque and Euler: the spin stays (OMEGA_NEW = OMEGA_NEW + 0), so it
  // is neither read nor written (the spin array is updated in place)
  const bool keep_w = MODE == 1 && !wh && !ph;
  const double4 W = keep_w ? make_double4(0.0, 0.0, 0.0, 0.0) : omg_c[me];
  const double w[3] = {W.x, W.y, W.z};
  double f[3] = {0.0, 0.0, 0.0}, t[3] = {0.0, 0.0, 0.0};
  if (wh && st == DEM_STATE_NORMAL) {
    const double* o = wf + 6 * (size_t)me;
    f[0] = o[0]; f[1] = o[1]; f[2] = o[2]; t[0] = o[3]; t[1] = o[4]; t[2] = o[5];
  }
  if (st != DEM_STATE_NONEXISTENT && ph) {
    const bool roll = p.mew_r > 0.0;
    const double r = pos_c[me].w;
    double2 om = make_double2(0.0, 0.0);
    if (roll) { om.x = sqrt(dot3(w, w)); om.y = 1.0 / om.x; }
    add_range<true>(p, is, mid, in_flag, in_pair, rec, roll, r, w, om, f, t);
    add_range<false>(p, me ? rs : 0, re, pflag, nullptr, rec, roll, r, w, om, f, t);
    if (mid < ie) add_range<true>(p, mid, ie, in_flag, in_pair, rec, roll, r, w, om, f, t);
  }
  const double4 X = pos_c[me], V = vel_c[me];
  const double x[3] = {X.x, X.y, X.z}, v[3] = {V.x, V.y, V.z};
  finish_particle<MODE>(p, me, st, x, v, w, X.w, V.w, W.w, f, t, pos_n, vel_n, omg_n, fc, tow, acc_old,
                        rot_acc_old, vslot, cells, keep_w);
}

// CFUPDATEOLD + CFNEWVALUES from FC/TOW, in place; zeroes FC/TOW.
template <int INTG, bool B>
__global__ void k_integrate(DevParams p0, BatchView bv, double4* __restrict__ pos4, double4* __restrict__ vel4,
                            double4* __restrict__ omg4, const int8_t* __restrict__ state,
                            double* __restrict__ fc, double* __restrict__ tow,
                            double* __restrict__ acc_old, double* __restrict__ rot_acc_old,
                            unsigned* __restrict__ vslot) {
  const int me = blockIdx.x * blockDim.x + threadIdx.x;
  if (me >= p0.n) return;
  const DevParams& p = sysp<B>(p0, bv, me);
  const size_t n = (size_t)p.n;
  const double4 X = pos4[me], V = vel4[me], W = omg4[me];
  const double x[3] = {X.x, X.y, X.z}, v[3] = {V.x, V.y, V.z}, w[3] = {W.x, W.y, W.z};
  double f[3], t[3];
  for (int c = 0; c < 3; ++c) {
    f[c] = fc[c * n + me]; t[c] = tow[c * n + me];
    fc[c * n + me] = 0.0; tow[c * n + me] = 0.0;
  }
  finish_particle<INTG == DEM_INTG_AB2 ? 2 : 1>(p, me, state[me], x, v, w, X.w, V.w, W.w, f, t, pos4, vel4, omg4,
                                                fc, tow, acc_old, rot_acc_old, vslot);
}

static WallCtx wall_ctx(dem_handle* h) {
  WallCtx w;
  w.vertex = h->vertex; w.norm_face = h->norm_face; w.ignore_edge = h->ignore_edge;
  w.fbin_start = h->fbin_start; w.fbin = h->fbin; w.dg_pijk = h->dg_pijk;
  w.wall_fid = h->wall_fid; w.wall_pft = h->wall_pft; w.nf = h->nf;
  return w;
}

// Particles screened per thread: one while that fills the device once (more
// blocks then share the listed particles), four past it, where the screening
// of the others is what the kernel does.
static bool wall_single(const dem_handle* h) { return h->nl() <= h->n_sm * 2 * WALL_T; }
static WallArgs wall_args(dem_handle* h, int threads) {
  const int per = threads * (wall_single(h) ? 1 : 4);
  WallArgs a;
  a.w = wall_ctx(h);
  a.n = h->nl();
  a.blocks = (h->nl() + per - 1) / per;
  a.wgap = h->wgap; a.live = h->wall_live; a.cand = h->wall_cand;
  a.wf = h->wf; a.hit = h->wall_hit;
  return a;
}

template <int COLL, bool B>
static void launch_walls_t(dem_handle* h) {
  const int c = h->cur;
  const WallArgs wa = wall_args(h, WALL_T);
  auto go = [&](auto kernel) {
    kernel<<<wa.blocks, WALL_T, 0, h->stream>>>(h->dp, h->bview(), wa, h->skin, h->vslot_pending(), h->state,
                                                h->pos4[c], h->vel4[c], h->omg4[c], h->phase, &h->derr->count[c],
                                                h->derr);
  };
  if (wall_single(h)) go(k_walls<COLL, B, 1>);
  else go(k_walls<COLL, B, 4>);
  DEM_LAUNCH(h);
}

template <int COLL, bool B>
static void launch_pairs_t(dem_handle* h, bool walls) {
  const int c = h->cur;
  const dem_handle::Shape sh = h->pair_shape(false);
  const int T = sh.threads;
  const WallArgs wa = wall_args(h, T);
  auto go = [&](auto kernel) {
    launch_pdl(h, kernel, (unsigned)(sh.blocks + (walls ? wa.blocks : 0)), T, h->dp, h->bview(), wa,
               h->d_np, h->pair_cap, h->pair_owner, h->nbrs[h->rb], h->in_pos, h->pos4[c], h->vel4[c], h->omg4[c],
               h->state, h->phase, h->pft[h->pcur], h->pflag(), h->in_flag, h->touched, h->pgap, h->skin,
               h->vslot_pending(), h->recs(), &h->derr->count[c], h->derr);
  };
  if (!walls) go(k_pairs<COLL, B, 0>);
  else if (wall_single(h)) go(k_pairs<COLL, B, 1>);
  else go(k_pairs<COLL, B, 4>);
}

template <int MODE, bool B>
static void launch_gather_t(dem_handle* h) {
  const int T = h->gather_block(false), G = (h->nl() + T - 1) / T;
  const int c = h->cur;
  launch_pdl(h, k_gather<MODE, B>, G, T, h->dp, h->bview(), h->pos4[c], h->vel4[c], h->omg4[c], h->pos4[1 - c],
             h->vel4[1 - c], h->omg4[1 - c], h->state, h->wf, h->row_end[h->rb], h->in_start, h->in_mid, h->in_pair,
             h->pflag(), h->in_flag, h->touched, h->wall_hit, h->recs(), h->fc, h->tow, h->acc_old, h->rot_acc_old,
             h->vslot_note(), gather_cells<MODE, B>(h), step_end(h));
}

void launch_wall_gaps(dem_handle* h) {
  if (h->nf <= 0) return;
  const int T = 256, G = (h->nl() + T - 1) / T;
  if (h->batch())
    k_wall_gaps<true><<<G, T, 0, h->stream>>>(h->dp, h->bview(), wall_ctx(h), h->pos4[h->cur], h->state,
                                              h->wall_cand, h->wgap);
  else
    k_wall_gaps<false><<<G, T, 0, h->stream>>>(h->dp, h->bview(), wall_ctx(h), h->pos4[h->cur], h->state,
                                               h->wall_cand, h->wgap);
  DEM_LAUNCH(h);
}

static void launch_walls(dem_handle* h) {
  if (h->nf <= 0) return;
  const bool hz = h->dp.coll == DEM_COLL_HERTZ;
  if (h->batch()) hz ? launch_walls_t<DEM_COLL_HERTZ, true>(h) : launch_walls_t<DEM_COLL_LSD, true>(h);
  else hz ? launch_walls_t<DEM_COLL_HERTZ, false>(h) : launch_walls_t<DEM_COLL_LSD, false>(h);
}

template <bool B>
static void launch_pairs_fp64(dem_handle* h, bool walls) {
  if (h->dp.coll == DEM_COLL_HERTZ) launch_pairs_t<DEM_COLL_HERTZ, B>(h, walls);
  else launch_pairs_t<DEM_COLL_LSD, B>(h, walls);
}

template <bool B>
static void launch_gather_fp64(dem_handle* h, int mode) {
  if (mode == 0) launch_gather_t<0, B>(h);
  else if (mode == 1) launch_gather_t<1, B>(h);
  else launch_gather_t<2, B>(h);
}

// The wall work and the pairs are one launch (launch_force_kernels).
bool walls_with_pairs(const dem_handle* h, bool split) { return h->nf > 0 && !split && !h->prof; }

// The two timed parts of the force step for the autotuner.
void launch_pairs_only(dem_handle* h, bool walls) {
  if (h->dp.prec == DEM_PREC_SPLIT) {
    // no gather in between that would clear the slip list
    cudaMemsetAsync(&h->slipfix->count, 0, sizeof(unsigned), h->stream);
    launch_pairs_split(h);
  }
  else if (h->batch()) launch_pairs_fp64<true>(h, walls);
  else launch_pairs_fp64<false>(h, walls);
}

void launch_gather_only(dem_handle* h) {
  if (h->dp.prec == DEM_PREC_SPLIT) launch_gather_split(h, 0);
  else if (h->batch()) launch_gather_fp64<true>(h, 0);
  else launch_gather_fp64<false>(h, 0);
}

// Contact forces of the current state.  mode: 0 = into FC/TOW, 1/2 = fused
// Euler/AB2 integration into the other state buffer.  The collision model,
// integrator and force precision are common to all systems of a batch.
static void launch_force_kernels(dem_handle* h, int mode, bool split) {
  // The wall work and the pair kernel read the same state and write disjoint
  // arrays (walls: wall_hit, wf and the wall histories; pairs: the pair
  // histories, flags, records and touched marks).  In FP64 they are one
  // launch; the split pair kernel is built with other arithmetic options and
  // half the registers, so its wall work runs on the side stream beside it and
  // the gather waits for both (in a captured step, two branches of the
  // graph).  With the parts of the step timed (profiling), they run one after
  // the other.
  const bool walls = h->nf > 0, merged = walls_with_pairs(h, split);
  const bool side = walls && split && h->side_stream && !h->prof;
  if (side) {
    cudaEventRecord(h->ev_fork, h->stream);
    cudaStreamWaitEvent(h->side_stream, h->ev_fork, 0);
    cudaStream_t main = h->stream;
    h->stream = h->side_stream;
    launch_walls(h);
    h->stream = main;
    cudaEventRecord(h->ev_join, h->side_stream);
  } else if (!merged) {
    ProfScope ps(h, DEM_PROF_WALLS);
    launch_walls(h);
  }
  {
    ProfScope ps(h, DEM_PROF_PAIRS);
    if (split) launch_pairs_split(h);
    else if (h->batch()) launch_pairs_fp64<true>(h, merged);
    else launch_pairs_fp64<false>(h, merged);
  }
  if (side) {
    cudaStreamWaitEvent(h->stream, h->ev_join, 0);
    h->joined = true;
  }
  ProfScope ps(h, DEM_PROF_GATHER);
  if (split) launch_gather_split(h, mode);
  else if (h->batch()) launch_gather_fp64<true>(h, mode);
  else launch_gather_fp64<false>(h, mode);
}

// The noted displacements join the bound since the last build: the pending
// set first, then the moves noted since (an upload's, or an integration
// outside the gather).
__global__ void k_skin(double* __restrict__ skin, unsigned* __restrict__ pending, unsigned* __restrict__ noted,
                       CandState* __restrict__ cand) {
  add_displacement(skin, cand, pending);
  add_displacement(skin, cand, noted);
}

void clear_counts(dem_handle* h) {
  cudaMemsetAsync(h->derr->count, 0, sizeof h->derr->count, h->stream);
  h->joined = true;
  h->count_dirty = false;
}

__global__ void k_set_skin(double* __restrict__ skin, double v) { skin[0] = v; }

void launch_skin(dem_handle* h) {
  k_skin<<<1, 32, 0, h->stream>>>(h->skin, h->vslot_pending(), h->vslot_note(), h->cand);
  DEM_LAUNCH(h);
}

void skin_unknown(dem_handle* h) {
  k_set_skin<<<1, 1, 0, h->stream>>>(h->skin, HUGE_VAL);
  DEM_LAUNCH(h);
  // positions (or walls) changed from outside: the candidate list starts over
  if (h->cand) cudaMemsetAsync(&h->cand->have, 0, sizeof(int), h->stream);
}

int run_force(dem_handle* h, bool fused) {
  ProfScope ps(h, DEM_PROF_FORCE);
  h->dp.first_pass = h->first_pass ? 1 : 0;
  const int mode = !fused ? 0 : (h->dp.intg == DEM_INTG_AB2 ? 2 : 1);
  // the counts of this pass start at zero: the last integrating gather
  // cleared them, or a pass that did not integrate has left its own
  if (!fused || h->count_dirty) clear_counts(h);
  launch_force_kernels(h, mode, h->dp.prec == DEM_PREC_SPLIT);
  h->count_set = h->cur;
  h->count_dirty = !fused;
  if (int rc = check_cuda(h, cudaGetLastError(), "force kernels")) return rc;
  if (fused) { h->cur = 1 - h->cur; h->first_pass = false; }
  return 0;
}

// The force pass of a step that the caller ends: forces into FC/TOW, then a
// kernel that integrates them into the other state buffer with end_step
// (the coupled step, whose drag comes in between).
int run_force_open(dem_handle* h) {
  ProfScope ps(h, DEM_PROF_FORCE);
  h->dp.first_pass = h->first_pass ? 1 : 0;
  if (h->count_dirty) clear_counts(h);
  launch_force_kernels(h, 0, h->dp.prec == DEM_PREC_SPLIT);
  h->count_set = h->cur;
  return check_cuda(h, cudaGetLastError(), "force kernels");
}

// Per-step force error of the split path: both paths evaluate FC for the
// current state (the wall and pair histories are restored between and after
// them); returns max|F_split - F_fp64| over all components divided by
// max|F_fp64|.
int run_split_force_error(dem_handle* h, double* rel_err) {
  if (!h->have_state || !h->have_pairs) return set_err(h, DEM_ERR_STATE, "state or pair list missing");
  const size_t n = h->n, cm = h->dp.cmax, P = (size_t)host_pairs(h);
  const size_t b_fid = sizeof(int) * cm * n, b_pft = sizeof(double) * 3 * cm * n;
  const size_t b_hist = sizeof(double) * P;  // of one component's plane
  // both passes start from the same wall and pair histories (each pass
  // updates them in place)
  char* snap = (char*)stage_buffer(h, b_fid + b_pft + n + 3 * b_hist + 2 * P + 64);
  if (!snap) return set_err(h, DEM_ERR_CUDA, "cudaMalloc stage");
  char* s_live = snap + b_fid + b_pft;
  char* s_hist = s_live + n;
  char* s_flag = s_hist + 3 * b_hist;
  char* s_inflag = s_flag + P;
  auto save = [&]() {
    cudaMemcpyAsync(snap, h->wall_fid, b_fid, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(snap + b_fid, h->wall_pft, b_pft, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(s_live, h->wall_live, n, cudaMemcpyDeviceToDevice, h->stream);
    if (P) {
      for (int c = 0; c < 3; ++c)
        cudaMemcpyAsync(s_hist + c * b_hist, h->pft[h->pcur] + c * h->pair_cap, b_hist, cudaMemcpyDeviceToDevice, h->stream);
      cudaMemcpyAsync(s_flag, h->pflag(), P, cudaMemcpyDeviceToDevice, h->stream);
      cudaMemcpyAsync(s_inflag, h->in_flag, P, cudaMemcpyDeviceToDevice, h->stream);
    }
  };
  auto restore = [&]() {
    cudaMemcpyAsync(h->wall_fid, snap, b_fid, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(h->wall_pft, snap + b_fid, b_pft, cudaMemcpyDeviceToDevice, h->stream);
    cudaMemcpyAsync(h->wall_live, s_live, n, cudaMemcpyDeviceToDevice, h->stream);
    if (P) {
      for (int c = 0; c < 3; ++c)
        cudaMemcpyAsync(h->pft[h->pcur] + c * h->pair_cap, s_hist + c * b_hist, b_hist, cudaMemcpyDeviceToDevice, h->stream);
      cudaMemcpyAsync(h->pflag(), s_flag, P, cudaMemcpyDeviceToDevice, h->stream);
      cudaMemcpyAsync(h->in_flag, s_inflag, P, cudaMemcpyDeviceToDevice, h->stream);
    }
  };
  std::vector<double> f64(3 * n), f32(3 * n);
  h->dp.first_pass = 0;
  save();
  launch_force_kernels(h, 0, false);
  cudaMemcpyAsync(f64.data(), h->fc, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, h->stream);
  restore();
  clear_counts(h);
  launch_force_kernels(h, 0, true);
  h->count_set = h->cur;  // the second pass is the last force evaluation
  h->count_dirty = true;
  cudaMemcpyAsync(f32.data(), h->fc, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, h->stream);
  restore();
  if (int rc = check_cuda(h, cudaStreamSynchronize(h->stream), "force error")) return rc;
  double dmax = 0.0, fmax = 0.0;
  for (size_t k = 0; k < 3 * n; ++k) {
    dmax = std::max(dmax, std::fabs(f32[k] - f64[k]));
    fmax = std::max(fmax, std::fabs(f64[k]));
  }
  *rel_err = fmax > 0.0 ? dmax / fmax : dmax;
  return fetch_errors(h);
}

template <int INTG, bool B>
static void launch_integrate_t(dem_handle* h) {
  const int T = 256, G = (h->nl() + T - 1) / T;
  const int c = h->cur;
  k_integrate<INTG, B><<<G, T, 0, h->stream>>>(h->dp, h->bview(), h->pos4[c], h->vel4[c], h->omg4[c], h->state,
                                               h->fc, h->tow, h->acc_old, h->rot_acc_old, h->vslot_note());
  DEM_LAUNCH(h);
}

int run_cfnewvalues(dem_handle* h) {
  ProfScope ps(h, DEM_PROF_INTEGRATE);
  h->dp.first_pass = h->first_pass ? 1 : 0;
  const bool ab2 = h->dp.intg == DEM_INTG_AB2;
  if (h->batch()) ab2 ? launch_integrate_t<DEM_INTG_AB2, true>(h) : launch_integrate_t<DEM_INTG_EULER, true>(h);
  else ab2 ? launch_integrate_t<DEM_INTG_AB2, false>(h) : launch_integrate_t<DEM_INTG_EULER, false>(h);
  launch_skin(h);
  h->first_pass = false;
  return check_cuda(h, cudaGetLastError(), "k_integrate");
}

}  // namespace demb
