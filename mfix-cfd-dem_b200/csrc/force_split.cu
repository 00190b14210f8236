// force_split.cu -- split-precision contact forces (FP32 forces, FP64
// history and integration).
//
// Same contact law as the FP64 path (calc_force_dem.f:204-506 with
// CFRELVEL, cfrelvel.f:54-77) with this split of the arithmetic:
//   FP64  the displacement x_I - x_L and the velocity difference v_L - v_I
//         (differences of large, nearly equal numbers), the squared
//         distance and R_LM^2 - |x_I - x_L|^2 (the overlap is this over
//         R_LM + |x_I - x_L|, so no FP64 square root is needed), the
//         tangential-overlap history update PFT + DT*V_t and its Coulomb
//         rescaling, and the integration (CFNEWVALUES);
//   FP32  the unit normal, relative velocity at the contact point, spring and
//         damping coefficients, normal/tangential forces, torque arms and
//         rolling friction; per-particle sums use compensated (Neumaier)
//         FP32 accumulation.
//
// Structure: the pair kernel evaluates every contact once (a lane per pair
// that may be in contact, queued from windows of the half list) and writes each particle's terms
// as a 32-byte FP32 record: the owner's at the pair index (rec_own, in row
// order) and the neighbour's at the pair's slot of the neighbour's incoming
// list (rec_in[in_pos[cc]], the transpose order).  The neighbour-side writes
// are scattered but never waited on; the per-particle kernel then reads its
// own row and its incoming list as two contiguous ranges, with no random
// load.  Contact flags: PF_CONTACT of pflag for the owner's records (row
// order), and in_flag (transpose order) for the neighbour's, written only
// when a pair's contact state changes.  Wall terms come from the FP64 wall
// kernel (force.cu).  The sum order differs from the serial reference;
// split results are compared with the FP64 path by the stated force
// tolerance, not bit for bit.
//
// This file is compiled with FMA contraction and fast single-precision
// square roots and divisions.
#include "dem_internal.cuh"

namespace demb {

struct Comp3 {  // Neumaier-compensated FP32 sum of a 3-vector
  float s[3], c[3];
  __device__ void zero() { for (int k = 0; k < 3; ++k) { s[k] = 0.f; c[k] = 0.f; } }
  __device__ __forceinline__ void add(int k, float x) {
    const float t = s[k] + x;
    if (fabsf(s[k]) >= fabsf(x)) c[k] += (s[k] - t) + x;
    else c[k] += (x - t) + s[k];
    s[k] = t;
  }
  __device__ __forceinline__ double value(int k) const { return (double)s[k] + (double)c[k]; }
};

// The pair force of one contact with L the owner and I the neighbour (the
// split arithmetic above): the force on L (fc; I receives -fc), the torque
// vector n x Ft with the two lever arms, KN and the overlap (rolling
// friction), and the new history ot.  dist = x_I - x_L, d2 = |dist|^2 and
// ovd = R_LM^2 - d2 come from the contact test in FP64.
struct PairTerms {
  float fc[3], tf[3], dcl2, dci2, kn, ov;
  bool near;  // the FP32 onset-of-slip test lies within 1e-4 of its threshold
};

// x_I - x_L of the nearest image and its square.
__device__ __forceinline__ double separation(const DevParams& p, const double4& a, const double4& b, double dist[3]) {
  const double xl[3] = {a.x, a.y, a.z}, xi[3] = {b.x, b.y, b.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double pj = xi[c];
    const double s = periodic_shift(p, c, pj - xl[c]);
    if (s != 0.0) pj = pj + s;
    dist[c] = pj - xl[c];
  }
  return dist[0] * dist[0] + dist[1] * dist[1] + dist[2] * dist[2];
}

// The onset-of-slip test of calc_force_dem.f:330-337 in FP64, evaluated as
// the FP64 kernels do (contact_force), for owner state (xl, vl, wl) and
// neighbour state (xi, vi, wi) with dist = x_I - x_L and history pin.  The
// friction law turns the tangential force at the onset of slip (below it
// -KT*OVERLAP_T - ETAT*VREL_T, above it MEW*|FN| along OVERLAP_T), so a
// contact whose FP32 test lies within the FP32 error of the threshold takes
// its branch from this test (k_slip_fix).
template <int COLL>
__device__ __forceinline__ bool slip_fp64(const DevParams& p, const double4& xl, const double4& vl,
                                          const double4& wl, const double4& xi, const double4& vi,
                                          const double4& wi, int ix, const double dist[3], double d2,
                                          const double pin[3]) {
  const double rl = xl.w, ri = xi.w;
  const double dmag = sqrt(d2);
  const double nrm[3] = {dist[0] / dmag, dist[1] / dmag, dist[2] / dmag};
  const double overlap_n = (rl + ri) - dmag;
  const double dcl = (dmag * dmag + rl * rl - ri * ri) / (2.0 * dmag);
  const double dci = dmag - dcl;
  const double osum[3] = {wl.x * dcl + wi.x * dci, wl.y * dcl + wi.y * dci, wl.z * dcl + wi.z * dci};
  const double vrel[3] = {vl.x - vi.x + (osum[1] * nrm[2] - osum[2] * nrm[1]),
                          vl.y - vi.y + (osum[2] * nrm[0] - osum[0] * nrm[2]),
                          vl.z - vi.z + (osum[0] * nrm[1] - osum[1] * nrm[0])};
  const double vrn = vrel[0] * nrm[0] + vrel[1] * nrm[1] + vrel[2] * nrm[2];
  const double vt[3] = {vrel[0] - vrn * nrm[0], vrel[1] - vrn * nrm[1], vrel[2] - vrn * nrm[2]};
  const double rad_eff = (rl * ri) / (rl + ri);
  const double m_eff = (vl.w * vi.w) / (vl.w + vi.w);
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
  double fn2 = 0.0, ft2 = 0.0, ot2 = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double fn = -(kn * overlap_n * nrm[c] + etan * vrn * nrm[c]);
    const double ot = p.dt * vt[c] + pin[c];
    const double ft = -kt * ot - etat * vt[c];
    fn2 += fn * fn;
    ot2 += ot * ot;
    ft2 += ft * ft;
  }
  if (!(ot2 > 0.0)) return false;
  return sqrt(ft2) > p.mew * sqrt(fn2);
}

// FIX false: the pair kernel's evaluation, the onset of slip decided in
// FP32 and o.near set near its threshold; FIX true: the same evaluation
// with the onset of slip decided by slip_fp64 (k_slip_fix).
template <int COLL, bool FIX>
__device__ __forceinline__ void split_contact(const DevParams& p, const double4& xl, const double4& vl,
                                              const double4& wl, int phl, const double4& xi, const double4& vi,
                                              const double4& wi, int phi, const double dist[3], double d2,
                                              double ovd, const double pin[3], double ot[3], PairTerms& o) {
  const float rl = (float)xl.w, ri = (float)xi.w;
  const float d2f = (float)d2;
  const float inv = rsqrtf(d2f);
  const float dmag = d2f * inv;
  const float ov = (float)ovd / ((rl + ri) + dmag);
  const float nrm[3] = {(float)dist[0] * inv, (float)dist[1] * inv, (float)dist[2] * inv};
  float vrel[3] = {(float)(vl.x - vi.x), (float)(vl.y - vi.y), (float)(vl.z - vi.z)};
  const float dcl = 0.5f * dmag + (rl - ri) * (rl + ri) * (0.5f * inv);
  const float dci = dmag - dcl;
  const float osum[3] = {(float)wl.x * dcl + (float)wi.x * dci, (float)wl.y * dcl + (float)wi.y * dci,
                         (float)wl.z * dcl + (float)wi.z * dci};
  vrel[0] += osum[1] * nrm[2] - osum[2] * nrm[1];
  vrel[1] += osum[2] * nrm[0] - osum[0] * nrm[2];
  vrel[2] += osum[0] * nrm[1] - osum[1] * nrm[0];
  const float vrn = vrel[0] * nrm[0] + vrel[1] * nrm[1] + vrel[2] * nrm[2];
  const float vt[3] = {vrel[0] - vrn * nrm[0], vrel[1] - vrn * nrm[1], vrel[2] - vrn * nrm[2]};
  const int ix = phl * MAXP + phi;
  const float rad_eff = (rl * ri) / (rl + ri);
  const float ml = (float)vl.w, mi = (float)vi.w;
  const float m_eff = (ml * mi) / (ml + mi);
  float kn, kt, etan, etat;
  if (COLL == DEM_COLL_HERTZ) {
    // KN = HERT_KN*sqrt(ov)*sqrt(R_eff) = HERT_KN*q with q = sqrt(ov*R_eff);
    // ETA_N = DES_ETAN*ov^(1/4)*sqrt(HERT_KN*sqrt(R_eff)*M_eff)
    //       = DES_ETAN*sqrt(HERT_KN)*sqrt(q*M_eff), and the same for t
    const float q = sqrtf(ov * rad_eff);
    const float sqm = sqrtf(q * m_eff);
    kn = p.hkn32[ix] * q;
    kt = p.hkt32[ix] * q;
    etan = p.etan_sq32[ix] * sqm;
    etat = p.etat_sq32[ix] * sqm;
  } else {
    kn = p.kn32; kt = p.kt32;
    const float sm = sqrtf(m_eff);
    etan = p.etan32[ix] * sm;
    etat = p.etat32[ix] * sm;
  }
  float fn[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) fn[c] = -(kn * ov + etan * vrn) * nrm[c];
  // tangential history in FP64: PFT + DT*V_t
#pragma unroll
  for (int c = 0; c < 3; ++c) ot[c] = p.dt * (double)vt[c] + pin[c];
  const float o32[3] = {(float)ot[0], (float)ot[1], (float)ot[2]};
  const float mag2 = o32[0] * o32[0] + o32[1] * o32[1] + o32[2] * o32[2];
  float ft[3] = {0.f, 0.f, 0.f};
  o.near = false;
  if (mag2 > 0.f) {
#pragma unroll
    for (int c = 0; c < 3; ++c) ft[c] = -kt * o32[c] - etat * vt[c];
    const float ft2 = ft[0] * ft[0] + ft[1] * ft[1] + ft[2] * ft[2];
    const float fn2 = fn[0] * fn[0] + fn[1] * fn[1] + fn[2] * fn[2];
    // |Ft| > MEW*|Fn|, compared squared
    const float thr = p.mew32 * p.mew32 * fn2;
    bool slip;
    if (FIX) {
      slip = slip_fp64<COLL>(p, xl, vl, wl, xi, vi, wi, ix, dist, d2, pin);
    } else {
      slip = ft2 > thr;
      o.near = fabsf(ft2 - thr) <= 1e-4f * thr;
    }
    if (slip) {
      // Coulomb slip: Ft = -MEW*|Fn| t, history (MEW*|Fn|/KT) t, t = ot/|ot|
      const float fnmd = p.mew32 * sqrtf(fn2);
      const float im = rsqrtf(mag2);
#pragma unroll
      for (int c = 0; c < 3; ++c) ft[c] = -fnmd * (o32[c] * im);
      const double sc = (double)(fnmd / kt * im);
#pragma unroll
      for (int c = 0; c < 3; ++c) ot[c] = sc * ot[c];
    }
  }
  o.dcl2 = dcl;
  o.dci2 = dci;
  o.tf[0] = nrm[1] * ft[2] - nrm[2] * ft[1];
  o.tf[1] = nrm[2] * ft[0] - nrm[0] * ft[2];
  o.tf[2] = nrm[0] * ft[1] - nrm[1] * ft[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) o.fc[c] = fn[c] + ft[c];
  o.kn = kn;
  o.ov = ov;
}

// One particle's terms of a contact: (force, KN*OVERLAP) and (torque, 0),
// 32 aligned bytes read and written with one instruction.
struct __align__(32) Rec32 {
  float4 a, b;
};
__device__ __forceinline__ Rec32 ld_rec(const Rec32* p) {
  Rec32 r;
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w)
      : "l"(p));
  return r;
}
__device__ __forceinline__ void st_rec(Rec32* p, const float4& a, const float4& b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
               "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

// The owner's record of a contact at its pair index, the neighbour's at its
// incoming slot.
__device__ __forceinline__ void put_records(const PairTerms& o, long long cc, const int* __restrict__ in_pos,
                                            Rec32* __restrict__ rec_own, Rec32* __restrict__ rec_in) {
  const float rol = o.kn * o.ov;
  st_rec(rec_own + cc, make_float4(o.fc[0], o.fc[1], o.fc[2], rol),
         make_float4(o.dcl2 * o.tf[0], o.dcl2 * o.tf[1], o.dcl2 * o.tf[2], 0.f));
  st_rec(rec_in + in_pos[cc], make_float4(-o.fc[0], -o.fc[1], -o.fc[2], rol),
         make_float4(o.dci2 * o.tf[0], o.dci2 * o.tf[1], o.dci2 * o.tf[2], 0.f));
}

// Kernel 1 (per pair): one CC iteration of CALC_FORCE_DEM, evaluated once.
// A warp takes a window of WIN_PAIRS pairs, queues those that may be in
// contact (screen_window) and gives each lane one of the queue.
// The bed of 1,000,000 spheres (1.67 M contacts of 4.4 M pairs): 160 us with
// four pairs per thread, 107 us so.
template <int COLL, bool B>
__global__ void __launch_bounds__(256, 4)
k_pairs_split(DevParams p0, BatchView bv, const int* __restrict__ d_np, long long cap, const int* __restrict__ owner,
              const int* __restrict__ nbrs, const int* __restrict__ in_pos, const double4* __restrict__ pos4,
              const double4* __restrict__ vel4, const double4* __restrict__ omg4, const int8_t* __restrict__ state,
              const uint8_t* __restrict__ phase, double* __restrict__ pft, uint8_t* __restrict__ pflag,
              uint8_t* __restrict__ in_flag, uint8_t* __restrict__ touched, const float* __restrict__ pgap,
              const double* __restrict__ skin, const unsigned* __restrict__ pending, Rec32* __restrict__ rec_own,
              Rec32* __restrict__ rec_in,
              SlipFix* __restrict__ fix, ContactCount* __restrict__ count, DevErr* __restrict__ err) {
  __shared__ WinQueue s_queue[256 / 32];
  const int z = pdl_wait();
  pdl_next();
  const long long np = min((long long)d_np[z], cap);
  // the bound in FP32, rounded up: a pair is skipped only when its gap
  // (rounded down at the build) exceeds it
  const float reach = __double2float_ru(2.0 * displacement_bound(skin + z, pending + z));
  unsigned long long ncont = 0;
  unsigned eflags = 0;
  WinQueue* queue = &s_queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)WIN_PAIRS * ((gridDim.x * blockDim.x) >> 5);
  for (long long w0 = (long long)WIN_PAIRS * ((int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) + z); w0 < np; w0 += stride) {
    const int nq = screen_window(w0, np, pflag, in_flag, in_pos, pgap, owner, nbrs, reach, queue);
    for (int k = lane; k < nq; k += 32) {
      const int e = queue->e[k];
      const long long cc = w0 + (e & (WIN_PAIRS - 1));
      const uint8_t f0 = (uint8_t)(e >> 7);
      const int2 who = queue->who[k];
      const int ll = who.x, i = who.y;
      uint8_t f = f0 & PF_HIST;  // NONEXISTENT partner or zero distance: history kept
      {
        // the states, the positions and the history in one round of loads (any
        // slot's position can be read; it is used only for existing particles);
        // the motion too would spill registers here
        const double4 a = ld32(pos4 + ll), b = ld32(pos4 + i);
        const int8_t sl = state[ll], si = state[i];
        double pin[3] = {0.0, 0.0, 0.0};
        if (f0 & PF_HIST) { pin[0] = pft[cc]; pin[1] = pft[cap + cc]; pin[2] = pft[2 * cap + cc]; }
        if (si != DEM_STATE_NONEXISTENT && sl != DEM_STATE_NONEXISTENT) {
          const DevParams& p = sysp<B>(p0, bv, ll);
          double dist[3];
          const double d2 = separation(p, a, b, dist);
          const double r_lm = a.w + b.w;
          if (d2 > (r_lm - SMALL_NUMBER) * (r_lm - SMALL_NUMBER)) {
            if (f0 & PF_HIST) { pft[cc] = 0.0; pft[cap + cc] = 0.0; pft[2 * cap + cc] = 0.0; }
            f = 0;
          } else if (d2 == 0.0) {
            eflags |= EF_ZERO_DIST;
            err->zero_a = ll; err->zero_b = i;
          } else {
            const double4 va = ld32(vel4 + ll), vb = ld32(vel4 + i), wa = ld32(omg4 + ll), wb = ld32(omg4 + i);
            double ot[3];
            PairTerms o;
            // one solids phase: no phase to look up
            const int phl = p.nph > 1 ? phase[ll] : 0, phi = p.nph > 1 ? phase[i] : 0;
            split_contact<COLL, false>(p, a, va, wa, phl, b, vb, wb, phi, dist, d2, r_lm * r_lm - d2, pin, ot, o);
            // near the onset of slip k_slip_fix evaluates the contact again,
            // from the history as it was (left in place here)
            bool deferred = false;
            if (o.near) {
              const unsigned t = atomicAdd(&fix->count, 1u);
              if (t < (unsigned)SLIP_FIX_CAP) {
                fix->pair[t] = 2 * cc + ((f0 & PF_HIST) ? 1 : 0);
                deferred = true;
              }
            }
            if (!deferred) { pft[cc] = ot[0]; pft[cap + cc] = ot[1]; pft[2 * cap + cc] = ot[2]; }
            put_records(o, cc, in_pos, rec_own, rec_in);
            touched[ll] = 1;
            touched[i] = 1;
            f = PF_CONTACT | ((ot[0] != 0.0 || ot[1] != 0.0 || ot[2] != 0.0) ? PF_HIST : 0);
            ++ncont;
          }
        }
      }
      if (f != f0) {
        pflag[cc] = f;
        // the neighbour's view of the contact, in transpose order
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

constexpr int FIX_T = 32, FIX_BLOCKS = 64;

// The contacts k_pairs_split left near the onset of slip, evaluated again
// with the onset decided in FP64 (slip_fp64): history, flag and both
// records rewritten.  Their history is still the one the pair kernel read.
// A few contacts each, all blocks' chains of loads and FP64 arithmetic side by
// side: one block of 128 threads took 6-12 us behind every pair pass, and a
// step of the bed of 1,000,000 spheres 278 us, 264 us so.  The gather clears
// the count for the next pass.
template <int COLL, bool B>
__global__ void __launch_bounds__(FIX_T)
k_slip_fix(DevParams p0, BatchView bv, const SlipFix* __restrict__ fix, const int* __restrict__ owner,
           const int* __restrict__ nbrs, const int* __restrict__ in_pos, const double4* __restrict__ pos4,
           const double4* __restrict__ vel4, const double4* __restrict__ omg4, const uint8_t* __restrict__ phase,
           double* __restrict__ pft, long long cap, uint8_t* __restrict__ pflag, Rec32* __restrict__ rec_own,
           Rec32* __restrict__ rec_in) {
  const int z = pdl_wait();
  pdl_next();
  const unsigned n = min(fix[z].count, (unsigned)SLIP_FIX_CAP);
  for (unsigned t = blockIdx.x * FIX_T + threadIdx.x; t < n; t += FIX_BLOCKS * FIX_T) {
    const long long code = fix->pair[t];
    const long long cc = code >> 1;
    const int ll = owner[cc], i = nbrs[cc];
    const DevParams& p = sysp<B>(p0, bv, ll);
    const double4 a = pos4[ll], b = pos4[i];
    double dist[3];
    const double d2 = separation(p, a, b, dist);
    const double r_lm = a.w + b.w;
    const double4 va = vel4[ll], vb = vel4[i], wa = omg4[ll], wb = omg4[i];
    double pin[3] = {0.0, 0.0, 0.0};
    if (code & 1) { pin[0] = pft[cc]; pin[1] = pft[cap + cc]; pin[2] = pft[2 * cap + cc]; }
    const int phl = p.nph > 1 ? phase[ll] : 0, phi = p.nph > 1 ? phase[i] : 0;
    double ot[3];
    PairTerms o;
    split_contact<COLL, true>(p, a, va, wa, phl, b, vb, wb, phi, dist, d2, r_lm * r_lm - d2, pin, ot, o);
    pft[cc] = ot[0]; pft[cap + cc] = ot[1]; pft[2 * cap + cc] = ot[2];
    put_records(o, cc, in_pos, rec_own, rec_in);
    pflag[cc] = PF_CONTACT | ((ot[0] != 0.0 || ot[1] != 0.0 || ot[2] != 0.0) ? PF_HIST : 0);
  }
}

// Compensated sums of a particle's records.
struct SplitSums {
  Comp3 F, T;
  float rs, rc;  // KN*OVERLAP
  __device__ __forceinline__ void zero() { F.zero(); T.zero(); rs = 0.f; rc = 0.f; }
  __device__ __forceinline__ void add(const float4& a, const float4& b) {
    F.add(0, a.x); F.add(1, a.y); F.add(2, a.z);
    T.add(0, b.x); T.add(1, b.y); T.add(2, b.z);
    const float x = a.w, t = rs + x;
    if (fabsf(rs) >= fabsf(x)) rc += (rs - t) + x;
    else rc += (x - t) + rs;
    rs = t;
  }
};

// The records of one contiguous range [a, e) whose flag bytes say contact,
// lane by lane: a window of up to 32 at a time, the window's flags first, then
// the flagged records, each issued before the previous one is added.
__device__ __forceinline__ void add_range(int a, int e, const uint8_t* __restrict__ flags,
                                          const Rec32* __restrict__ rec, SplitSums& S) {
  for (int base = a; base < e; base += 32) {
    unsigned mask = contact_mask(flags, base, min(32, e - base));
    if (!mask) continue;
    Rec32 cur = ld_rec(rec + base + __ffs(mask) - 1);
    mask &= mask - 1u;
    while (true) {
      const bool more = mask != 0u;
      Rec32 nxt;
      if (more) {
        nxt = ld_rec(rec + base + __ffs(mask) - 1);
        mask &= mask - 1u;
      }
      S.add(cur.a, cur.b);
      if (!more) break;
      cur = nxt;
    }
  }
}

// The records of a warp's 32 particles.  Summed lane by lane a warp takes as
// many turns, each a load, as its busiest lane has contacts, two to three
// times the average; so the lanes first list what they have to add in shared
// memory, in particle order, the warp copies the records of SPLIT_CHUNK entries
// there at once, a record per lane and turn, all of them in flight together,
// and each lane adds its own from shared memory: its incoming ones, then its
// row's.  Entries: a pair index for the particle's
// own row, ~slot for an incoming pair.  Records lie side by side: 48 bytes
// apart fewer lanes would meet in a bank, but the L1 gets what shared memory
// leaves, and the bed of 1,000,000 spheres takes 260 us per step so, 264 us the
// other way.  Chunks of 96 or 64 entries take second turns (3 to 5 % slower).
constexpr int SPLIT_T = dem_handle::SPLIT_GATHER_MAX;
constexpr int SPLIT_CHUNK = 128;
struct SplitShared {
  int entry[SPLIT_CHUNK];
  float4 rec[SPLIT_CHUNK][2];
};
__device__ __forceinline__ void add_terms(SplitShared& sh, unsigned in, unsigned own, int is, int rs,
                                          const Rec32* __restrict__ rec_own, const Rec32* __restrict__ rec_in,
                                          SplitSums& S) {
  const int lane = threadIdx.x & 31;
  int left = __popc(in) + __popc(own), incl = left;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  int at = incl - left;  // place of the lane's next entry
  for (int c0 = 0; c0 < total; c0 += SPLIT_CHUNK) {
    const int n = min(SPLIT_CHUNK, total - c0);
    const int first = at - c0;
    int mine = 0;  // the lane's entries in this chunk
    while (left && at < c0 + SPLIT_CHUNK) {
      int e;
      if (in) { e = ~(is + __ffs(in) - 1); in &= in - 1u; }
      else { e = rs + __ffs(own) - 1; own &= own - 1u; }
      sh.entry[at - c0] = e;
      ++at; --left; ++mine;
    }
    __syncwarp();
    for (int e = lane; e < n; e += 32) {
      const int d = sh.entry[e];
      const Rec32* q = d < 0 ? rec_in + ~d : rec_own + d;
      copy16(&sh.rec[e][0], &q->a);
      copy16(&sh.rec[e][1], &q->b);
    }
    copy_wait();
    __syncwarp();
    for (int k = 0; k < mine; ++k) S.add(sh.rec[first + k][0], sh.rec[first + k][1]);
    __syncwarp();  // the chunk is read before the next one is written
  }
}

// Kernel 2 (per particle): wall terms (k_walls), the particle's incoming
// records (transpose order) and its own row's -- only for particles the
// pair kernel marked as in some contact --, compensated FP32 sums, the
// rolling-friction torque -MEW_R*(2R)*sum(KN*OVERLAP_N)*OMEGA/|OMEGA|, and
// the integration (MODE 1 Euler, 2 Adams-Bashforth) or FC/TOW (MODE 0).
// Same bed: 113 us with two 16-byte loads per record lane by lane, 85 us
// staged in shared memory with the quotients side by side; the staging alone is
// 1 % of a step there, and 4 % in a batch of 16 columns of 600,000 spheres,
// whose contacts are spread less evenly.
template <int MODE, bool B>
__global__ void __launch_bounds__(SPLIT_T)
k_gather_split(DevParams p0, BatchView bv, const double4* __restrict__ pos_c, const double4* __restrict__ vel_c,
               const double4* __restrict__ omg_c, double4* __restrict__ pos_n, double4* __restrict__ vel_n,
               double4* __restrict__ omg_n, const int8_t* __restrict__ state, const double* __restrict__ wf,
               uint8_t* __restrict__ wall_hit, uint8_t* __restrict__ touched, const int* __restrict__ row_end,
               const int* __restrict__ in_start, const uint8_t* __restrict__ pflag, const uint8_t* __restrict__ in_flag,
               const Rec32* __restrict__ rec_own, const Rec32* __restrict__ rec_in, double* __restrict__ fc,
               double* __restrict__ tow, double* __restrict__ acc_old, double* __restrict__ rot_acc_old,
               unsigned* __restrict__ vslot, CellOut cells, StepEnd end, SlipFix* __restrict__ fix) {
  __shared__ SplitShared s_sh[SPLIT_T / 32];
  const int z = pdl_wait();
  pdl_next();
  if (MODE != 0) end_step(end);
  if (blockIdx.x == 0 && threadIdx.x == 0) fix->count = 0;
  const int at = blockIdx.x * blockDim.x + threadIdx.x + z;
  const bool mine = at < p0.n;
  const int me = mine ? at : p0.n - 1;  // the lanes past the end help with the warp's records only
  prefetch_l2(pos_c + me);
  prefetch_l2(vel_c + me);
  const int8_t st = state[me];
  // the sums first, the particle's own state and wall terms after them (few
  // registers live across the record loops)
  SplitSums S;
  S.zero();
  // a particle in no contact of this pass has no record to add
  const bool ph = mine && touched[me] != 0, wh = mine && wall_hit[me] != 0;
  if (ph) touched[me] = 0;
  // no torque and Euler: the spin stays (OMEGA_NEW = OMEGA_NEW + 0), so it
  // is neither read nor written (the spin array is updated in place)
  const bool keep_w = MODE == 1 && !wh && !ph;
  const bool sum = st != DEM_STATE_NONEXISTENT && ph;
  if (__any_sync(0xffffffffu, sum)) {
    int is = 0, ie = 0, rs = 0, re = 0;
    if (sum) { is = in_start[me]; ie = in_start[me + 1]; rs = me ? row_end[me - 1] : 0; re = row_end[me]; }
    if (__any_sync(0xffffffffu, ie - is > 32 || re - rs > 32)) {
      // a list longer than the masks: lane by lane
      add_range(is, ie, in_flag, rec_in, S);
      add_range(rs, re, pflag, rec_own, S);
    } else {
      const unsigned in = sum ? contact_mask(in_flag, is, ie - is) : 0u;
      const unsigned own = sum ? contact_mask(pflag, rs, re - rs) : 0u;
      add_terms(s_sh[threadIdx.x >> 5], in, own, is, rs, rec_own, rec_in, S);
    }
  }
  if (!mine) return;
  const DevParams& p = sysp<B>(p0, bv, me);
  const double4 X = pos_c[me], V = vel_c[me], W = keep_w ? make_double4(0.0, 0.0, 0.0, 0.0) : omg_c[me];
  double f0[3] = {0.0, 0.0, 0.0}, t0[3] = {0.0, 0.0, 0.0};
  if (wh) {
    wall_hit[me] = 0;
    if (st == DEM_STATE_NORMAL) {
      const double* o = wf + 6 * (size_t)me;
      f0[0] = o[0]; f0[1] = o[1]; f0[2] = o[2]; t0[0] = o[3]; t0[1] = o[4]; t0[2] = o[5];
    }
  }
  double f[3], t[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) { f[c] = f0[c] + S.F.value(c); t[c] = t0[c] + S.T.value(c); }
  if (p.mew_r > 0.0) {
    const float w32[3] = {(float)W.x, (float)W.y, (float)W.z};
    const float om = sqrtf(w32[0] * w32[0] + w32[1] * w32[1] + w32[2] * w32[2]);
    if (om > 0.f) {
      const double sc = -(p.mew_r * (2.0 * X.w) * ((double)S.rs + (double)S.rc)) / (double)om;
#pragma unroll
      for (int c = 0; c < 3; ++c) t[c] += sc * (double)w32[c];
    }
  }
  const double x[3] = {X.x, X.y, X.z}, v[3] = {V.x, V.y, V.z}, w[3] = {W.x, W.y, W.z};
  finish_particle<MODE>(p, me, st, x, v, w, X.w, V.w, W.w, f, t, pos_n, vel_n, omg_n, fc, tow, acc_old,
                        rot_acc_old, vslot, cells, keep_w);
}

// The split records live in the handle's record array: the owner records
// in its first 32*cap bytes, the neighbour records in the next 32*cap (the
// array holds 80*cap bytes, the FP64 record size).
static Rec32* rec_own_of(dem_handle* h) { return reinterpret_cast<Rec32*>(h->prec); }
static Rec32* rec_in_of(dem_handle* h) { return reinterpret_cast<Rec32*>(h->prec) + h->pair_cap; }
static_assert(2 * sizeof(Rec32) <= sizeof(PairRec) && sizeof(PairRec) == 80, "split records fit the record array");

template <int COLL, bool B>
static void launch_pairs_split_t(dem_handle* h) {
  const int c = h->cur;
  const dem_handle::Shape sh = h->pair_shape(true);
  launch_pdl(h, k_pairs_split<COLL, B>, (unsigned)sh.blocks, sh.threads, h->dp, h->bview(), h->d_np,
             h->pair_cap, h->pair_owner, h->nbrs[h->rb], h->in_pos, h->pos4[c], h->vel4[c], h->omg4[c], h->state,
             h->phase, h->pft[h->pcur], h->pflag(), h->in_flag, h->touched, h->pgap, h->skin, h->vslot_pending(),
             rec_own_of(h), rec_in_of(h), h->slipfix, &h->derr->count[c], h->derr);
  launch_pdl(h, k_slip_fix<COLL, B>, FIX_BLOCKS, FIX_T, h->dp, h->bview(), h->slipfix, h->pair_owner, h->nbrs[h->rb], h->in_pos,
             h->pos4[c], h->vel4[c], h->omg4[c], h->phase, h->pft[h->pcur], h->pair_cap, h->pflag(), rec_own_of(h),
             rec_in_of(h));
}

void launch_pairs_split(dem_handle* h) {
  const bool hz = h->dp.coll == DEM_COLL_HERTZ;
  if (h->batch()) hz ? launch_pairs_split_t<DEM_COLL_HERTZ, true>(h) : launch_pairs_split_t<DEM_COLL_LSD, true>(h);
  else hz ? launch_pairs_split_t<DEM_COLL_HERTZ, false>(h) : launch_pairs_split_t<DEM_COLL_LSD, false>(h);
}

template <int MODE, bool B>
static void launch_gather_split_t(dem_handle* h) {
  const int T = h->gather_block(true), G = (h->nl() + T - 1) / T;
  const int c = h->cur;
  launch_pdl(h, k_gather_split<MODE, B>, G, T, h->dp, h->bview(), h->pos4[c], h->vel4[c], h->omg4[c], h->pos4[1 - c],
             h->vel4[1 - c], h->omg4[1 - c], h->state, h->wf, h->wall_hit, h->touched, h->row_end[h->rb], h->in_start,
             h->pflag(), h->in_flag, rec_own_of(h), rec_in_of(h), h->fc, h->tow, h->acc_old, h->rot_acc_old,
             h->vslot_note(), gather_cells<MODE, B>(h), step_end(h), h->slipfix);
}

void launch_gather_split(dem_handle* h, int mode) {
  const bool bt = h->batch();
  if (mode == 0) bt ? launch_gather_split_t<0, true>(h) : launch_gather_split_t<0, false>(h);
  else if (mode == 1) bt ? launch_gather_split_t<1, true>(h) : launch_gather_split_t<1, false>(h);
  else bt ? launch_gather_split_t<2, true>(h) : launch_gather_split_t<2, false>(h);
}

}  // namespace demb
