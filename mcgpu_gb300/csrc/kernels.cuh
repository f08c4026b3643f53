// kernels.cuh -- the group-level pieces shared by every kernel: staging of
// the moved molecule, the cutoff screen, the per-warp neighbour rings, the
// pair batches (FP32 pair terms with FP64 per-neighbour sums, or FP64 pair
// terms), reductions and the commit.
#pragma once

#include "device.cuh"

namespace mcgpu {

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Primary position wrapped into [0, L) (FP32), for the screen.
__device__ __forceinline__ float4 wrap_pos(double x, double y, double z, const ChainHdr& H) {
  // x / L through the header's 2^32 / L (FP64 divisions are slow; a quotient at
  // an integer may round to either side of it, which moves the position by an
  // edge: the screen's minimum image does not see it)
  double wx = x - H.L[0] * floor(x * (H.fxinv[0] * 0x1p-32));
  double wy = y - H.L[1] * floor(y * (H.fxinv[1] * 0x1p-32));
  double wz = z - H.L[2] * floor(z * (H.fxinv[2] * 0x1p-32));
  return make_float4((float)wx, (float)wy, (float)wz, 0.f);
}

// Anchor position in 32-bit fixed point of the box edge (wraps mod 2^32).
__device__ __forceinline__ uint4 fixpos(double x, double y, double z, const ChainHdr& H) {
  return make_uint4((unsigned)(unsigned long long)__double2ll_rn(x * H.fxinv[0]),
                    (unsigned)(unsigned long long)__double2ll_rn(y * H.fxinv[1]),
                    (unsigned)(unsigned long long)__double2ll_rn(z * H.fxinv[2]), 0u);
}

// Minimum-image anchor difference b - a in Angstrom (FP32).
__device__ __forceinline__ float3 fixdiff(uint4 b, uint4 a, const ChainHdr& H) {
  return make_float3((float)(int)(b.x - a.x) * H.fxs[0], (float)(int)(b.y - a.y) * H.fxs[1],
                     (float)(int)(b.z - a.z) * H.fxs[2]);
}

// The same difference as a double-float (hi + lo), exact to ~1e-14 A: the
// fixed-point difference is split into a high part with its low 8 bits
// cleared (exact in FP32) and the rest, each scaled by L/2^32 held as
// fxs + fxs_lo, with the rounding of the main product recovered by an FMA.
__device__ __forceinline__ void fixdiff_ff(uint4 b, uint4 a, const ChainHdr& H, float3& hi,
                                           float3& lo) {
  const int d[3] = {(int)(b.x - a.x), (int)(b.y - a.y), (int)(b.z - a.z)};
  float h[3], l[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int dh = d[k] & ~0xFF;
    const float fh = (float)dh, fl = (float)(d[k] - dh);
    const float p = fh * H.fxs[k];
    const float e = fmaf(fh, H.fxs[k], -p);
    const float t = fmaf(fh, H.fxs_lo[k], fmaf(fl, H.fxs[k], e));
    h[k] = p + t;
    l[k] = t - (h[k] - p);
  }
  hi = make_float3(h[0], h[1], h[2]);
  lo = make_float3(l[0], l[1], l[2]);
}

// True when an atom pair of these two molecules may need its own periodic
// image (|D| + radii reaches half a box edge in some dimension).
__device__ __forceinline__ bool needs_wrap(float3 D, float rr, const ChainHdr& H) {
  return fabsf(D.x) + rr > 0.5f * H.Lf[0] - 1e-3f || fabsf(D.y) + rr > 0.5f * H.Lf[1] - 1e-3f ||
         fabsf(D.z) + rr > 0.5f * H.Lf[2] - 1e-3f;
}

// The reference's cutoff test for one primary pair, FP64, same rounding
// (SimulationStep.cpp:325-326 with :332-342 and :377-385).
__device__ __forceinline__ bool in_range64(double x1, double y1, double z1, int p2,
                                           const Pool& P, const ChainHdr& H) {
  double dx = make_periodic(P.x[p2] - x1, H.L[0]);
  double dy = make_periodic(P.y[p2] - y1, H.L[1]);
  double dz = make_periodic(P.z[p2] - z1, H.L[2]);
  double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return r2 <= __dmul_rn(H.cutoff, H.cutoff);
}

__device__ __forceinline__ float r2_screen(float4 a, float4 b, const ChainHdr& H) {
  float dx = wrapf(b.x - a.x, H.Lf[0]);
  float dy = wrapf(b.y - a.y, H.Lf[1]);
  float dz = wrapf(b.z - a.z, H.Lf[2]);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// ---- staging ------------------------------------------------------------

// misc[] slots of the staged molecule's FP32 radius and net charge factor
// (float bits: no FP64 on the step's path).
enum : int { kMiscRad = 21, kMiscQm = 22 };

// Lanes of ONE warp stage molecule m: its current placement ("old") and, if
// p is non-null, the proposed placement ("new") computed as
// SimCalcs::intermolecularMove does (SimulationStep.cpp:544-565): every
// non-vertex atom rotated about the vertex and translated, the vertex
// translated, then the molecule wrapped by its first primary atom
// (keepMoleculeInBox, :710-729).  Results go to shared memory; scalars to
// misc.  The caller synchronises the group afterwards.  NL 16: each half of the
// warp stages a molecule of its own (m, p, s and lane 0-15 are the half's; both
// or neither have a move).
template <int NL = 32>
__device__ inline void stage(const Pool& P, const ChainHdr& H, int m, const Proposal* p,
                      const GroupSmem& s, int lane) {
  const int a0 = P.mstart[m];
  const int lw = P.mlen[m];
  const int len = lw & 255;
  const int2 pi = P.mpi[m];
  for (int i = lane; i < len; i += NL) {
    int a = a0 + i;
    s.ox[i] = P.x[a]; s.oy[i] = P.y[a]; s.oz[i] = P.z[a];
    const double2 bl = P.blend ? P.blend[a] : blend64(P.sig[a], P.eps[a]);
    s.sd[i] = bl.x; s.ed[i] = bl.y; s.qd[i] = P.q[a];
    const float4 o = P.aoff[a];
    const float2 q = P.aeq[a];
    s.o_old[i] = o;
    s.l_old[i] = P.aofl[a];
    s.eq[i] = make_float4(q.x, q.y, fmaf(o.x, o.x, fmaf(o.y, o.y, o.z * o.z)), 0.f);
  }
  // net FP32 charge factor of the molecule (sum over lanes, fixed order)
  float qsum = 0.f;
  for (int i = lane; i < len; i += NL) qsum += P.aeq[a0 + i].y;
  for (int off = NL / 2; off > 0; off >>= 1) qsum += __shfl_xor_sync(~0u, qsum, off);
  for (int k = lane; k < pi.y; k += NL) {
    s.p_old[k] = P.ppos[pi.x + k];
    s.pa[k] = P.pidx[pi.x + k] - a0;
  }
  uint4 fo = P.mfix[m];
  if (lane == 0) {
    s.misc[0] = m; s.misc[1] = a0; s.misc[2] = len; s.misc[3] = pi.y;
    s.misc[4] = lw >> 8; s.misc[5] = p ? 3 : 1; s.misc[6] = p ? p->vertex : -1;
    s.misc[8] = (int)fo.x; s.misc[9] = (int)fo.y; s.misc[10] = (int)fo.z;
    s.misc[kMiscRad] = __float_as_int(P.mrad[m]);
    s.misc[kMiscQm] = __float_as_int(qsum);
  }
  if (!p) return;
  // lane k forms the cosine and sine of the k-th Euler angle
  double rc = 1.0, rs = 0.0;
  if (p->trig) {
    rc = lane == 0 ? p->cs[0] : lane == 1 ? p->cs[1] : p->cs[2];
    rs = lane == 0 ? p->sn[0] : lane == 1 ? p->sn[1] : p->sn[2];
  } else if (lane < 3) {
    sincos(__dmul_rn(lane == 0 ? p->r0 : lane == 1 ? p->r1 : p->r2, 3.14159265358979) / 180.0, &rs,
           &rc);
  }
  Rot R;
  R.cx = __shfl_sync(~0u, rc, 0, NL); R.sx = __shfl_sync(~0u, rs, 0, NL);
  R.cy = __shfl_sync(~0u, rc, 1, NL); R.sy = __shfl_sync(~0u, rs, 1, NL);
  R.cz = __shfl_sync(~0u, rc, 2, NL); R.sz = __shfl_sync(~0u, rs, 2, NL);
  __syncwarp();
  const int v = p->vertex;
  const double px = s.ox[v], py = s.oy[v], pz = s.oz[v];
  for (int i = lane; i < len; i += NL) {
    double x, y, z;
    if (i == v) {
      x = __dadd_rn(px, p->dx); y = __dadd_rn(py, p->dy); z = __dadd_rn(pz, p->dz);
    } else {
      double vx = __dadd_rn(s.ox[i], -px), vy = __dadd_rn(s.oy[i], -py), vz = __dadd_rn(s.oz[i], -pz);
      rot_apply(R, vx, vy, vz);
      x = __dadd_rn(__dadd_rn(vx, px), p->dx);
      y = __dadd_rn(__dadd_rn(vy, py), p->dy);
      z = __dadd_rn(__dadd_rn(vz, pz), p->dz);
    }
    s.nx[i] = x; s.ny[i] = y; s.nz[i] = z;
  }
  __syncwarp();
  const int an = s.pa[0];
  double ax = s.nx[an], ay = s.ny[an], az = s.nz[an];
  double shx = 0, shy = 0, shz = 0;
  if (ax < 0) shx = H.L[0]; else if (ax > H.L[0]) shx = -H.L[0];
  if (ay < 0) shy = H.L[1]; else if (ay > H.L[1]) shy = -H.L[1];
  if (az < 0) shz = H.L[2]; else if (az > H.L[2]) shz = -H.L[2];
  if (shx != 0) ax = __dadd_rn(ax, shx);
  if (shy != 0) ay = __dadd_rn(ay, shy);
  if (shz != 0) az = __dadd_rn(az, shz);
  __syncwarp();
  for (int i = lane; i < len; i += NL) {
    double x = s.nx[i], y = s.ny[i], z = s.nz[i];
    if (shx != 0) x = __dadd_rn(x, shx);
    if (shy != 0) y = __dadd_rn(y, shy);
    if (shz != 0) z = __dadd_rn(z, shz);
    s.nx[i] = x; s.ny[i] = y; s.nz[i] = z;
    const double vx = x - ax, vy = y - ay, vz = z - az;
    const float4 o = make_float4((float)vx, (float)vy, (float)vz, s.o_old[i].w);
    s.o_new[i] = o;
    s.l_new[i] = make_float4((float)(vx - (double)o.x), (float)(vy - (double)o.y),
                             (float)(vz - (double)o.z), 0.f);
    s.eq[i].w = fmaf(o.x, o.x, fmaf(o.y, o.y, o.z * o.z));
  }
  __syncwarp();
  for (int k = lane; k < pi.y; k += NL) {
    int q = s.pa[k];
    s.p_new[k] = wrap_pos(s.nx[q], s.ny[q], s.nz[q], H);
  }
  if (lane == 0) {
    uint4 fn = fixpos(ax, ay, az, H);
    s.misc[12] = (int)fn.x; s.misc[13] = (int)fn.y; s.misc[14] = (int)fn.z;
  }
}

__device__ __forceinline__ MovedInfo load_moved(const GroupSmem& s) {
  MovedInfo mi;
  mi.mol = s.misc[0]; mi.atom0 = s.misc[1]; mi.len = s.misc[2]; mi.npidx = s.misc[3];
  mi.act = s.misc[4]; mi.states = s.misc[5]; mi.vertex = s.misc[6]; mi.pad = 0;
  mi.fx_old = make_uint4((unsigned)s.misc[8], (unsigned)s.misc[9], (unsigned)s.misc[10], 0u);
  mi.fx_new = make_uint4((unsigned)s.misc[12], (unsigned)s.misc[13], (unsigned)s.misc[14], 0u);
  mi.rad = __int_as_float(s.misc[kMiscRad]);
  mi.qm = __int_as_float(s.misc[kMiscQm]);
  return mi;
}

// ---- screen ---------------------------------------------------------------

// FP32 screen with FP64 re-test inside the guard band (plain path: FP64
// positions from the master rows).
__device__ __forceinline__ int screen_mixed(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                            const MovedInfo& mi, int j) {
  const int2 pj = P.mpi[j];
  int f = 0;
  for (int k2 = 0; k2 < pj.y; k2++) {
    const float4 q = P.ppos[pj.x + k2];
    for (int k1 = 0; k1 < mi.npidx; k1++) {
      if ((mi.states & 1) && !(f & kInOld)) {
        float r2 = r2_screen(s.p_old[k1], q, H);
        if (r2 <= H.cut2_lo) {
          f |= kInOld;
        } else if (r2 <= H.cut2_hi) {
          int pa = s.pa[k1];
          if (in_range64(s.ox[pa], s.oy[pa], s.oz[pa], P.pidx[pj.x + k2], P, H)) f |= kInOld;
        }
      }
      if ((mi.states & 2) && !(f & kInNew)) {
        float r2 = r2_screen(s.p_new[k1], q, H);
        if (r2 <= H.cut2_lo) {
          f |= kInNew;
        } else if (r2 <= H.cut2_hi) {
          int pa = s.pa[k1];
          if (in_range64(s.nx[pa], s.ny[pa], s.nz[pa], P.pidx[pj.x + k2], P, H)) f |= kInNew;
        }
      }
    }
  }
  return f;
}

// ---- pair batches -----------------------------------------------------------

// Per-thread double-float accumulators of one evaluation.
struct AccFF {
  float oh, ol, nh, nl, ab;
  long long np;
};

// Displacement of a pair, atom b of the neighbour minus atom a of the moved
// molecule, both anchor-relative to the moved molecule's anchor.  PRECISE
// adds the low parts (bl: of b = D + o_b; la, with LO: of a's offset -- the
// chain state's offsets have none) so the only rounding left is the final
// one at the displacement's own magnitude.
template <bool PRECISE, bool LO>
__device__ __forceinline__ float3 pair_disp(float3 bh, float3 bl, float4 a, const float4* lo,
                                            int i) {
  if (PRECISE && !LO)
    return make_float3((bh.x - a.x) + bl.x, (bh.y - a.y) + bl.y, (bh.z - a.z) + bl.z);
  const float4 la = PRECISE ? lo[i] : a;
  if (PRECISE)
    return make_float3((bh.x - a.x) + (bl.x - la.x), (bh.y - a.y) + (bl.y - la.y),
                       (bh.z - a.z) + (bl.z - la.z));
  return make_float3(bh.x - a.x, bh.y - a.y, bh.z - a.z);
}

// Sum over the moved molecule's atoms a of the FP32 pair terms with one
// neighbour atom b, per-pair periodic image (entries whose atom pairs may
// straddle half a box edge).  abs accumulates |LJ| + |Coulomb|.
//
// NLEN > 0 fixes the moved molecule's length (at most 4) at compile time:
// the loop unrolls so its independent pair terms interleave, and bit i of
// ljmask clear means the LJ term of moved atom i is exactly zero (a sigma or
// epsilon product of zero) and is not evaluated.  NLEN == 0 (any length up
// to 64) ignores ljmask.  Neither changes a bit of the sum.
template <bool PRECISE, bool LO, int NLEN = 0>
__device__ __forceinline__ float sum_moved32_wrap(const float4* o, const float4* lo,
                                                  const float4* eq, int len, float3 bh, float3 bl,
                                                  float sb, float2 qb, const ChainHdr& H,
                                                  float& abs, unsigned ljmask = ~0u) {
  float acc = 0.f;
  auto term = [&](int i) {
    const float4 ea = eq[i];
    const float4 a = o[i];
    const float3 d = pair_disp<PRECISE, LO>(bh, bl, a, lo, i);
    const float dx = wrapf(d.x, H.Lf[0]);
    const float dy = wrapf(d.y, H.Lf[1]);
    const float dz = wrapf(d.z, H.Lf[2]);
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float ir = rsqrt_nr(r2);
    const float lj = (NLEN == 0 || ((ljmask >> i) & 1u)) ? lj32(rcp_nr(r2), a.w, sb, ea.x, qb.x)
                                                         : 0.f;
    const float cl = (ea.y * qb.y) * ir;
    const bool ok = r2 > 0.f;
    acc += ok ? lj + cl : 0.f;
    abs += ok ? fabsf(lj) + fabsf(cl) : 0.f;
  };
  if (NLEN > 0) {
#pragma unroll
    for (int i = 0; i < (NLEN > 0 ? NLEN : 1); i++) term(i);
  } else {
    for (int i = 0; i < len; i++) term(i);
  }
  return acc;
}

// The same sum for an entry whose pairs all use the anchors' image, with
// the Coulomb part written for neutral molecules: with R = |b - anchor_m|,
//   sum_a q_a / r_ab = sum_a q_a (1/r_ab - 1/R) + Q_m / R,
//   1/r - 1/R = (R^2 - r^2) / (r R (r + R)),  R^2 - r^2 = 2 b.o_a - |o_a|^2,
// so every Coulomb term is O(|o_a| / R) smaller than q_a q_b / r and carries
// proportionally less FP32 rounding.  A coincident pair (r = 0) is skipped
// as the reference skips it (BruteForceStep.cpp:68-69).  use_new selects the
// |o_a|^2 of the placement (eq.z old, eq.w new).
template <bool PRECISE, bool LO, int NLEN = 0>
__device__ __forceinline__ float sum_moved32_cf(const float4* o, const float4* lo,
                                                const float4* eq, int len, bool use_new,
                                                float3 bh, float3 bl, float sb, float2 qb,
                                                float qm, float& abs, unsigned ljmask = ~0u) {
  const float R2 = fmaf(bh.x, bh.x, fmaf(bh.y, bh.y, bh.z * bh.z));
  const float iR = rsqrt_nr(R2);
  const float R = R2 * iR;
  const float tx = bh.x + bh.x, ty = bh.y + bh.y, tz = bh.z + bh.z;
  float lj_acc = 0.f, phi = 0.f, lj_abs = 0.f, c_abs = 0.f;
  auto term = [&](int i) {
    const float4 a = o[i];
    const float4 ea = eq[i];
    const float3 d = pair_disp<PRECISE, LO>(bh, bl, a, lo, i);
    const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
    const float ir = rsqrt_nr(r2);
    const float lj = (NLEN == 0 || ((ljmask >> i) & 1u)) ? lj32(rcp_nr(r2), a.w, sb, ea.x, qb.x)
                                                         : 0.f;
    const float num = fmaf(tx, a.x, fmaf(ty, a.y, fmaf(tz, a.z, -(use_new ? ea.w : ea.z))));
    const float w = ir * rcp_approx(fmaf(r2, ir, R));
    const bool ok = r2 > 0.f;
    const float c = ok ? (ea.y * num) * w : -ea.y;
    lj_acc += ok ? lj : 0.f;
    lj_abs += ok ? fabsf(lj) : 0.f;
    phi += c;
    c_abs += fabsf(c);
  };
  if (NLEN > 0) {
#pragma unroll
    for (int i = 0; i < (NLEN > 0 ? NLEN : 1); i++) term(i);
  } else {
    for (int i = 0; i < len; i++) term(i);
  }
  const float f = qb.y * iR;
  abs += lj_abs + fabsf(f) * (c_abs + fabsf(qm));
  return fmaf(f, phi + qm, lj_acc);
}

// Pair batch of `count` ring entries from `head`, teams of T lanes (T a
// power of two <= 32): the team forms the entry's anchor differences
// (fixed point -> FP32, or double-float when PRECISE) and image flags, lane
// tl takes neighbour atoms tl, tl+T, ... against every atom of the moved
// molecule, and the team's FP32 partial of the entry is added in
// double-float to the team leader's accumulators.  (Chains of several species.)
template <bool PRECISE>
__device__ __forceinline__ void batch_ff(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                         const MovedInfo& mi, const int* rj, int head, int count,
                                         int lane, int T, AccFF& acc) {
  const int tm = lane / T, tl = lane - tm * T, nteams = 32 / T;
  for (int e0 = 0; e0 < count; e0 += nteams) {
    const int e = e0 + tm;
    int f = 0, b0 = 0, lenj = 0, actj = 0;
    float3 Do = make_float3(0.f, 0.f, 0.f), Dn = Do, Dol = Do, Dnl = Do;
    if (e < count) {
      const int jf = rj[(head + e) & (kRing - 1)];
      const int j = jf >> 4;
      f = jf & 15;
      float mrj;
      b0 = P.mstart[j];
      const int lw = P.mlen[j];
      lenj = lw & 255;
      actj = lw >> 8;
      mrj = P.mrad[j];
      const uint4 fj = P.mfix[j];
      const float rr = mi.rad + mrj;
      if (f & kInOld) {
        if (PRECISE) fixdiff_ff(fj, mi.fx_old, H, Do, Dol); else Do = fixdiff(fj, mi.fx_old, H);
        if (needs_wrap(Do, rr, H)) f |= kWrapOld;
      }
      if (f & kInNew) {
        if (PRECISE) fixdiff_ff(fj, mi.fx_new, H, Dn, Dnl); else Dn = fixdiff(fj, mi.fx_new, H);
        if (needs_wrap(Dn, rr, H)) f |= kWrapNew;
      }
    }
    float so = 0.f, sn = 0.f, sa = 0.f;
    for (int b = b0 + tl; b < b0 + lenj; b += T) {
      const float4 ob = P.aoff[b];
      const float2 qb = P.aeq[b];
      if (f & kInOld) {
        float3 bh = make_float3(Do.x + ob.x, Do.y + ob.y, Do.z + ob.z), bl = Dol;
        if (PRECISE) {
          // two-sum of D + o_b per axis, then the low parts
          const float ex = (Do.x - (bh.x - (bh.x - Do.x))) + (ob.x - (bh.x - Do.x));
          const float ey = (Do.y - (bh.y - (bh.y - Do.y))) + (ob.y - (bh.y - Do.y));
          const float ez = (Do.z - (bh.z - (bh.z - Do.z))) + (ob.z - (bh.z - Do.z));
          bl = make_float3(ex + Dol.x, ey + Dol.y, ez + Dol.z);
        }
        so += (f & kWrapOld)
                  ? sum_moved32_wrap<PRECISE, false>(s.o_old, nullptr, s.eq, mi.len, bh, bl, ob.w, qb, H, sa)
                  : sum_moved32_cf<PRECISE, false>(s.o_old, nullptr, s.eq, mi.len, false, bh, bl, ob.w, qb,
                                            mi.qm, sa);
      }
      if (f & kInNew) {
        float3 bh = make_float3(Dn.x + ob.x, Dn.y + ob.y, Dn.z + ob.z), bl = Dnl;
        if (PRECISE) {
          const float ex = (Dn.x - (bh.x - (bh.x - Dn.x))) + (ob.x - (bh.x - Dn.x));
          const float ey = (Dn.y - (bh.y - (bh.y - Dn.y))) + (ob.y - (bh.y - Dn.y));
          const float ez = (Dn.z - (bh.z - (bh.z - Dn.z))) + (ob.z - (bh.z - Dn.z));
          bl = make_float3(ex + Dnl.x, ey + Dnl.y, ez + Dnl.z);
        }
        sn += (f & kWrapNew)
                  ? sum_moved32_wrap<PRECISE, false>(s.o_new, nullptr, s.eq, mi.len, bh, bl, ob.w, qb, H, sa)
                  : sum_moved32_cf<PRECISE, false>(s.o_new, nullptr, s.eq, mi.len, true, bh, bl, ob.w, qb,
                                            mi.qm, sa);
      }
    }
    for (int off = T >> 1; off > 0; off >>= 1) {
      so += __shfl_xor_sync(~0u, so, off);
      sn += __shfl_xor_sync(~0u, sn, off);
      sa += __shfl_xor_sync(~0u, sa, off);
    }
    if (tl == 0 && f) {
      if (f & kInOld) {
        ff_add(acc.oh, acc.ol, so);
        acc.np += (long long)mi.act * actj;
      }
      if (f & kInNew) {
        ff_add(acc.nh, acc.nl, sn);
        acc.np += (long long)mi.act * actj;
      }
      acc.ab += sa;
    }
  }
}

// batch_ff for a uniform chain of molecules of N (1 to 3) atoms, one lane per (entry,
// placement): a batch of at most 16 entries takes one round of N^2 pair terms (a
// warp's share of the in-range neighbours is about 15 to 20, so a lane per
// entry left half the lanes idle for twice the time).  Rows and factors follow
// from the neighbour's index, and the rows are requested together (one
// round trip to L2).  ljmask bits 4k + i: the LJ term of neighbour atom k with
// moved atom i is not exactly zero (the same in every lane).  Each placement's
// sum is batch_ff's bit for bit.
template <int N>
__device__ __forceinline__ void batch_un(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                         const MovedInfo& mi, const int* rj, int head, int count,
                                         int lane, AccFF& acc, unsigned ljmask) {
  const int atom0 = H.atom0, mol0 = H.mol0;
  const float sx = H.fxs[0], sy = H.fxs[1], sz = H.fxs[2];
  const float Lx = H.Lf[0], Ly = H.Lf[1], Lz = H.Lf[2];
  const float rr = mi.rad + H.umrad;
  const int pairs = mi.act * H.uact;
#pragma unroll 1
  for (int base = 0; base < 2 * count; base += 32) {
    const int it = base + lane;
    const bool p = it >= count;
    if (it >= 2 * count) continue;   // lanes are independent: no shuffles below
    const int jf = rj[(head + (p ? it - count : it)) & (kRing - 1)];
    if (!(jf & (p ? kInNew : kInOld))) continue;
    const int j = jf >> 4;
    const int b0 = atom0 + (j - mol0) * N;
    const uint4 fj = P.mfix[j];
    float4 ob[N];
#pragma unroll
    for (int k = 0; k < N; k++) ob[k] = P.aoff[b0 + k];
    const float4* o = p ? s.o_new : s.o_old;
    const uint4 fm = p ? mi.fx_new : mi.fx_old;
    const float3 D = make_float3((float)(int)(fj.x - fm.x) * sx, (float)(int)(fj.y - fm.y) * sy,
                                 (float)(int)(fj.z - fm.z) * sz);
    // some pair may need its own periodic image (needs_wrap)
    const bool wrap = fabsf(D.x) + rr > 0.5f * Lx - 1e-3f ||
                      fabsf(D.y) + rr > 0.5f * Ly - 1e-3f || fabsf(D.z) + rr > 0.5f * Lz - 1e-3f;
    float sp = 0.f, sa = 0.f;
    if (wrap) {
#pragma unroll 1
      for (int k = 0; k < N; k++) {
        float4 b = ob[0];
#pragma unroll
        for (int c = 1; c < N; c++)
          if (k == c) b = ob[c];
        sp += sum_moved32_wrap<false, false, N>(o, nullptr, s.eq, N,
                                                make_float3(D.x + b.x, D.y + b.y, D.z + b.z),
                                                make_float3(0.f, 0.f, 0.f), b.w, s.teq[k], H, sa,
                                                (ljmask >> (4 * k)) & 15u);
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < N; k++) {
        float4 b = ob[0];
#pragma unroll
        for (int c = 1; c < N; c++)
          if (k == c) b = ob[c];
        sp += sum_moved32_cf<false, false, N>(o, nullptr, s.eq, N, p,
                                              make_float3(D.x + b.x, D.y + b.y, D.z + b.z),
                                              make_float3(0.f, 0.f, 0.f), b.w, s.teq[k], mi.qm,
                                              sa, (ljmask >> (4 * k)) & 15u);
      }
    }
    if (p)
      ff_add(acc.nh, acc.nl, sp);
    else
      ff_add(acc.oh, acc.ol, sp);
    acc.ab += sa;
    acc.np += pairs;
  }
}

// FP32 pair terms of atom k (of row b, factors qb) of molecule j with the moved
// molecule's old (p false) or new placement; abs grows by their magnitudes.
template <bool PRECISE>
__device__ __forceinline__ float uniform_item(const Pool& P, const ChainHdr& H,
                                              const GroupSmem& s, const MovedInfo& mi, int j,
                                              int k, bool p, float& abs) {
  const uint4 fj = P.mfix[j];
  const float4 b = P.aoff[H.atom0 + (j - H.mol0) * H.ulen + k];
  const float2 qb = s.teq[k];
  const uint4 fm = p ? mi.fx_new : mi.fx_old;
  float3 D, bl = make_float3(0.f, 0.f, 0.f);
  if (PRECISE) fixdiff_ff(fj, fm, H, D, bl); else D = fixdiff(fj, fm, H);
  const float3 bh = make_float3(D.x + b.x, D.y + b.y, D.z + b.z);
  if (PRECISE) {
    // two-sum of D + o_b per axis, then the low part
    bl.x += (D.x - (bh.x - (bh.x - D.x))) + (b.x - (bh.x - D.x));
    bl.y += (D.y - (bh.y - (bh.y - D.y))) + (b.y - (bh.y - D.y));
    bl.z += (D.z - (bh.z - (bh.z - D.z))) + (b.z - (bh.z - D.z));
  }
  const float4* o = p ? s.o_new : s.o_old;
  return needs_wrap(D, mi.rad + H.umrad, H)
             ? sum_moved32_wrap<PRECISE, false>(o, nullptr, s.eq, mi.len, bh, bl, b.w, qb, H, abs)
             : sum_moved32_cf<PRECISE, false>(o, nullptr, s.eq, mi.len, p, bh, bl, b.w, qb, mi.qm,
                                              abs);
}

// This thread's items (tid, tid + nthreads, ...) of a uniform chain's `count`
// entries that entry(e) gives (called by every lane of the warp): one atom of
// the neighbour against one placement of the moved molecule.  Rows and factors
// follow from the neighbour's index.  Where the length is a power of two, teams of
// T lanes take a (placement, entry) each, as batch_ff does, and sum its atoms as
// that does, so that the two paths' energies agree to double-float where a start
// of overlapping molecules (1e9 kcal/mol) leaves FP32 rounding in the running
// energy (atoms added in double-float one by one: 1.80 ms instead of 1.90 per 1,024
// steps of 4,000 16-atom molecules, the energies 1e-8 of the start's apart); else
// items run atom by atom and placement by placement over full warps, each added in
// double-float (teams would idle 7 lanes of 16 on 9 atoms).
template <bool PRECISE, class Entry>
__device__ __forceinline__ void uniform_items(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                              const MovedInfo& mi, int count, int tid,
                                              int nthreads, int T, AccFF& acc, Entry entry) {
  const int ulen = H.ulen, units = 2 * count, items = units * ulen;
  const int lane = tid & 31;
  if (T > 1 && (ulen & (ulen - 1)) == 0) {
    const int tl = lane & (T - 1);
    for (int first = (tid & ~31) / T; first < units; first += nthreads / T) {
      const int u = first + lane / T;
      const bool in = u < units, p = u >= count;
      const int jf = entry(!in ? 0 : p ? u - count : u);
      const bool on = in && (jf & (p ? kInNew : kInOld));
      float sp = 0.f, sa = 0.f;
      if (on)
        for (int k = tl; k < ulen; k += T)
          sp += uniform_item<PRECISE>(P, H, s, mi, jf >> 4, k, p, sa);
      for (int off = T >> 1; off > 0; off >>= 1) sp += __shfl_xor_sync(~0u, sp, off);
      if (on && tl == 0) {
        if (p)
          ff_add(acc.nh, acc.nl, sp);
        else
          ff_add(acc.oh, acc.ol, sp);
      }
      acc.ab += sa;
    }
    return;
  }
  for (int base = tid & ~31; base < items; base += nthreads) {
    const int it = base + lane;
    const int k = it / units, u = it - k * units;
    const bool p = u >= count;
    const int jf = entry(p ? u - count : u);
    if (it >= items || !(jf & (p ? kInNew : kInOld))) continue;
    float sa = 0.f;
    const float sp = uniform_item<PRECISE>(P, H, s, mi, jf >> 4, k, p, sa);
    if (p)
      ff_add(acc.nh, acc.nl, sp);
    else
      ff_add(acc.oh, acc.ol, sp);
    acc.ab += sa;
  }
}

// ---- FP64 pair batches -------------------------------------------------------
//
// GB300 issues FP64 at 1/64 of the FP32 rate: one warp instruction per 16
// cycles on an SM whatever its active lanes, so an FP64 batch is bound by its
// count of FP64 warp instructions.  Hence
//   * the items of a batch (placement, neighbour atom) fill the lanes of the
//     warp without gaps (a team of lanes per neighbour left 1 of 4 lanes idle
//     on 3-site and 7 of 16 on 9-site molecules);
//   * no FP64 comparison on a pair's path: the image, r = 0 and skipped-site
//     tests read the operands' high words on the integer pipe;
//   * the LJ term is formed only where its sigma and epsilon products are not
//     zero (water: 1 pair of 9), and r^2 by fused multiply-adds.
// 16 FP64 instructions a Coulomb pair and 23 with LJ.

// sigma factor of a skipped site (blend64).
__device__ __forceinline__ bool blend_skipped(double sa) {
  return __double2hiint(sa) == (int)0xBFF00000;
}
__device__ __forceinline__ bool bits_nonzero(double v) {
  return (__double2hiint(v) | __double2loint(v)) != 0;
}
__device__ __forceinline__ int hi_abs(double v) { return __double2hiint(v) & 0x7fffffff; }

// make_periodic with its comparisons on the high words; half = the high word
// of L / 2 (equal high words take the FP64 comparisons).
__device__ __forceinline__ double image64(double d, double L, int half) {
  const int h = hi_abs(d);
  if (h < half) return d;
  if (h > half && half >= 0) return __dadd_rn(d, copysign(L, -d));
  return make_periodic(d, L);
}

// Sum over the atoms of one molecule (rows xs, ys, zs) of the FP64 pair terms
// with atom b of another: the reference's minimum image of every pair and its
// rule for skipped sites (BruteForceStep.cpp:61-76).  b is shifted once to
// its image nearest the molecule's first atom; a pair that still lies beyond
// half an edge (molecules straddling it, or rows outside the box) takes the
// reference's own image from the unshifted rows.
// (sb, eb): b's factors (blend64), qb its charge; sd, ed, qd the molecule's.
//
// The twelfth power multiplies a relative error of sigma_ab / r by twelve, so
// sigma_ab^2 is the product of the sigmas themselves (from the atoms' square roots the
// terms were 1.0e-15 off on average over 1,000 close pairs; 7.1e-16 this way, and
// 8.1e-16 by the reference's square root and division).  FINE corrects 1/r^2 = (1/r)^2
// once by its own residual (5.3e-16): two more instructions on the longest chain, which
// cost the chains' steps up to 17 % and the static sums, bound by the pipe, 5 %.
//
// With VOTE the rare image and the LJ term stand behind votes of the lanes that
// enter together, so those lanes must hold rows of the same length with the same
// sites skipped: a lane that leaves the loop, or passes over a site, is waited for
// by the others.  Lanes on unlike molecules take VOTE false, the same terms in the
// same order behind branches of their own.
template <bool VOTE = true, bool FINE = false>
__device__ __forceinline__ double pair_sum64(const double* xs, const double* ys, const double* zs,
                                             const double* sd, const double* ed, const double* qd,
                                             int len, double xb, double yb, double zb, double sb,
                                             double eb, double qb, double Lx, double Ly,
                                             double Lz) {
  if (blend_skipped(sb)) return 0.0;
  const int hx = __double2hiint(0.5 * Lx), hy = __double2hiint(0.5 * Ly),
            hz = __double2hiint(0.5 * Lz);
  const double tx = xb - xs[0], ty = yb - ys[0], tz = zb - zs[0];
  const double bx = hi_abs(tx) >= hx ? xb - copysign(Lx, tx) : xb;
  const double by = hi_abs(ty) >= hy ? yb - copysign(Ly, ty) : yb;
  const double bz = hi_abs(tz) >= hz ? zb - copysign(Lz, tz) : zb;
  const bool lj_b = bits_nonzero(sb) && bits_nonzero(eb);
  const unsigned am = VOTE ? __activemask() : 0u;
  double cl = 0.0, lj = 0.0;   // sums without b's charge and epsilon, which come last
#pragma unroll 3
  for (int i = 0; i < len; i++) {
    const double sa = sd[i], ea = ed[i];
    if (blend_skipped(sa)) continue;
    double dx = bx - xs[i], dy = by - ys[i], dz = bz - zs[i];
    const bool far = hi_abs(dx) >= hx || hi_abs(dy) >= hy || hi_abs(dz) >= hz;
    if (VOTE ? __any_sync(am, far) != 0 : far) {
      if (VOTE) __syncwarp(am);
      if (far) {
        dx = image64(xb - xs[i], Lx, hx);
        dy = image64(yb - ys[i], Ly, hy);
        dz = image64(zb - zs[i], Lz, hz);
      }
      if (VOTE) __syncwarp(am);
    }
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const bool apart = bits_nonzero(r2);  // coincident: skipped (BruteForceStep.cpp:68-69)
    const double ri = rsqrt(r2);
    cl = fma(apart ? qd[i] : 0.0, apart ? ri : 0.0, cl);
    const bool near = apart && lj_b && bits_nonzero(sa) && bits_nonzero(ea);
    if (VOTE ? __any_sync(am, near) != 0 : near) {
      if (VOTE) __syncwarp(am);
      const double i2 = ri * ri;
      double t2 = (sa * sb) * i2;
      if (FINE) t2 = fma(t2, fma(-r2, i2, 1.0), t2);
      const double s6 = t2 * t2 * t2;
      if (near) lj = fma(ea, fma(s6, s6, -s6), lj);
      if (VOTE) __syncwarp(am);
    }
  }
  return fma(cl, qb * kCoulomb, lj * (4.0 * eb));
}

// FP64 pair batch of `count` (1..32) ring entries from `head`: the items
// (placement, entry, neighbour atom) are dealt to the lanes in order, old
// placements first.  A uniform chain's items run atom by atom over the
// entries, so the lanes of a round share the neighbour atom's kind and agree
// on the LJ term; else an item's entry is found in the prefix sums of the
// entries' lengths.  atom(j, b, x, y, z) gives the FP64 position of atom b of
// neighbour j.
template <class AtomPos>
__device__ __forceinline__ void batch_items64(const Pool& P, const ChainHdr& H,
                                              const GroupSmem& s, const MovedInfo& mi,
                                              const int* rj, int head, int count, int lane,
                                              double& eo, double& en, long long& np,
                                              AtomPos atom) {
  const int two = mi.states == 3 ? 2 : 1;
  int pref = 0, total;
  const bool uni = H.uniform != 0;
  if (uni) {
    total = count * H.ulen;
    if (lane < count) {
      const int f = rj[(head + lane) & (kRing - 1)] & 15;
      np += (long long)__popc(f & (kInOld | kInNew)) * (mi.act * H.uact);
    }
  } else {
    int len = 0;
    if (lane < count) {
      const int jf = rj[(head + lane) & (kRing - 1)];
      const int lw = P.mlen[jf >> 4];
      len = lw & 255;
      np += (long long)__popc(jf & (kInOld | kInNew)) * (mi.act * (lw >> 8));
    }
    pref = len;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(~0u, pref, off);
      if (lane >= off) pref += v;
    }
    total = __shfl_sync(~0u, pref, 31);
    pref -= len;
  }
  const int items = total * two;
  for (int base = 0; base < items; base += 32) {
    const int it = base + lane;
    const bool second = it >= total;
    const int local = second ? it - total : it;
    int e, k;
    if (uni) {
      k = local / count;
      e = local - k * count;
    } else {
      e = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int at = e + step;
        const int v = __shfl_sync(~0u, pref, at & 31);
        if (at < count && v <= local) e = at;
      }
      k = local - __shfl_sync(~0u, pref, e);
    }
    if (it >= items) continue;
    const int jf = rj[(head + e) & (kRing - 1)];
    const bool use_new = second || mi.states == 2;
    if (!(jf & (use_new ? kInNew : kInOld))) continue;
    const int j = jf >> 4;
    const int b = (uni ? H.atom0 + (j - H.mol0) * H.ulen : P.mstart[j]) + k;
    double xb, yb, zb;
    atom(j, b, xb, yb, zb);
    const double2 bl = P.blend ? P.blend[b] : blend64(P.sig[b], P.eps[b]);
    const double v = pair_sum64(use_new ? s.nx : s.ox, use_new ? s.ny : s.oy,
                                      use_new ? s.nz : s.oz, s.sd, s.ed, s.qd, mi.len, xb, yb,
                                      zb, bl.x, bl.y, P.q[b], H.L[0], H.L[1], H.L[2]);
    if (use_new) en += v; else eo += v;
  }
}

// The batch on the master rows (plain path).
__device__ __forceinline__ void batch_f64(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                          const MovedInfo& mi, const int* rj, int head, int count,
                                          int lane, double& eo, double& en, long long& np) {
  batch_items64(P, H, s, mi, rj, head, count, lane, eo, en, np,
                [&](int, int b, double& x, double& y, double& z) {
                  x = P.x[b];
                  y = P.y[b];
                  z = P.z[b];
                });
}

// FP32 pair terms of atom b of molecule j with the moved molecule's old (p false)
// or new placement (offsets with their low parts).
template <bool PRECISE>
__device__ __forceinline__ float pair_item32(const Pool& P, const ChainHdr& H,
                                             const GroupSmem& s, const MovedInfo& mi, int j,
                                             int b, bool p) {
  const uint4 fj = P.mfix[j];
  const float4 ob = P.aoff[b];
  const float2 qb = P.aeq[b];
  float4 obl = make_float4(0.f, 0.f, 0.f, 0.f);
  if (PRECISE) obl = P.aofl[b];
  // mrad, not the header's radius: a flexible molecule's changes
  const float rr = mi.rad + P.mrad[j];
  const uint4 fm = p ? mi.fx_new : mi.fx_old;
  float3 D, bl = make_float3(0.f, 0.f, 0.f);
  if (PRECISE) fixdiff_ff(fj, fm, H, D, bl); else D = fixdiff(fj, fm, H);
  const float3 bh = make_float3(D.x + ob.x, D.y + ob.y, D.z + ob.z);
  if (PRECISE) {
    // two-sum of D + o_b per axis, then the low parts
    const float ex = (D.x - (bh.x - (bh.x - D.x))) + (ob.x - (bh.x - D.x));
    const float ey = (D.y - (bh.y - (bh.y - D.y))) + (ob.y - (bh.y - D.y));
    const float ez = (D.z - (bh.z - (bh.z - D.z))) + (ob.z - (bh.z - D.z));
    bl = make_float3(ex + (bl.x + obl.x), ey + (bl.y + obl.y), ez + (bl.z + obl.z));
  }
  float sa = 0.f;
  return needs_wrap(D, rr, H)
          ? sum_moved32_wrap<PRECISE, true>(p ? s.o_new : s.o_old, p ? s.l_new : s.l_old, s.eq,
                                            mi.len, bh, bl, ob.w, qb, H, sa)
          : sum_moved32_cf<PRECISE, true>(p ? s.o_new : s.o_old, p ? s.l_new : s.l_old, s.eq,
                                          mi.len, p, bh, bl, ob.w, qb, mi.qm, sa);
}

// FP32 pair batch of `count` (1..32) ring entries from `head` on the plain path
// (offsets with their low parts), the items (placement, entry, neighbour atom)
// dealt to the lanes as batch_items64 deals them; each item's sum over the
// moved molecule's atoms is added in double-float.  Molecules of many atoms go
// entry by entry: the lanes of a round then agree on the per-pair image of an entry
// (atom by atom they took both forms of the sum where some entries straddle half an
// edge: the system energy of 16 molecules of 64 atoms 143 us, 83 entry by entry).
constexpr int kItemsByEntry = 16;
template <bool PRECISE>
__device__ __forceinline__ void batch_items32(const Pool& P, const ChainHdr& H,
                                              const GroupSmem& s, const MovedInfo& mi,
                                              const int* rj, int head, int count, int lane,
                                              AccFF& acc) {
  const int two = mi.states == 3 ? 2 : 1;
  int pref = 0, total;
  const bool uni = H.uniform != 0;
  if (uni) {
    total = count * H.ulen;
    if (lane < count)
      acc.np += (long long)__popc(rj[(head + lane) & (kRing - 1)] & (kInOld | kInNew)) *
                (mi.act * H.uact);
  } else {
    int len = 0;
    if (lane < count) {
      const int jf = rj[(head + lane) & (kRing - 1)];
      const int lw = P.mlen[jf >> 4];
      len = lw & 255;
      acc.np += (long long)__popc(jf & (kInOld | kInNew)) * (mi.act * (lw >> 8));
    }
    pref = len;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(~0u, pref, off);
      if (lane >= off) pref += v;
    }
    total = __shfl_sync(~0u, pref, 31);
    pref -= len;
  }
  const int items = total * two;
  for (int base = 0; base < items; base += 32) {
    const int it = base + lane;
    const bool p = it >= total || mi.states == 2;
    const int local = it >= total ? it - total : it;
    int e, k;
    if (uni && H.ulen >= kItemsByEntry) {
      e = local / H.ulen;
      k = local - e * H.ulen;
    } else if (uni) {
      k = local / count;
      e = local - k * count;
    } else {
      e = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int at = e + step;
        const int v = __shfl_sync(~0u, pref, at & 31);
        if (at < count && v <= local) e = at;
      }
      k = local - __shfl_sync(~0u, pref, e);
    }
    if (it >= items) continue;
    const int jf = rj[(head + e) & (kRing - 1)];
    if (!(jf & (p ? kInNew : kInOld))) continue;
    const int j = jf >> 4;
    const int b = (uni ? H.atom0 + (j - H.mol0) * H.ulen : P.mstart[j]) + k;
    const float sp = pair_item32<PRECISE>(P, H, s, mi, j, b, p);
    if (p)
      ff_add(acc.nh, acc.nl, sp);
    else
      ff_add(acc.oh, acc.ol, sp);
  }
}

// Warp w of nw screens its share of candidates [c_begin, c_end) in rounds of 32,
// appends hits to its ring rj and evaluates them in batches of 32.  DEALT: the
// warps of a whole grid, each with every nw-th candidate (neighbours in space
// are neighbours in index on a lattice start or in a file: of 128 warps with
// 32 consecutive candidates a few had all of a molecule's neighbours); the warps
// of one CTA take 32 consecutive ones in turn, one load each.  FP32 pairs
// accumulate in double-float and are added to the FP64 sums at the end.
template <bool F64, bool DEALT>
__device__ inline void warp_eval(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                 const MovedInfo& mi, int c_begin, int c_end, int w, int nw,
                                 int* rj, int lane, double& eo, double& en, long long& np) {
  int head = 0, tail = 0;
  const unsigned lt = lanemask_lt();
  AccFF acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0};
  for (int base = c_begin + (DEALT ? w : w * 32); base < c_end; base += nw * 32) {
    const int j = base + (DEALT ? lane * nw : lane);
    int f = 0;
    // the FP32 screen with the FP64 re-test inside its guard band gives the
    // FP64 test's in-range set exactly, for FP64 and FP32 pair terms alike
    if (j < c_end && j != mi.mol) f = screen_mixed(P, H, s, mi, j);
    const unsigned bal = __ballot_sync(~0u, f != 0);
    if (f) rj[(tail + __popc(bal & lt)) & (kRing - 1)] = (j << 4) | f;
    tail += __popc(bal);
    const bool last = base + nw * 32 >= c_end;
    while (tail - head >= 32 || (last && tail > head)) {
      const int count = min(32, tail - head);
      __syncwarp();
      if (F64)
        batch_f64(P, H, s, mi, rj, head, count, lane, eo, en, np);
      else if (H.precise)
        batch_items32<true>(P, H, s, mi, rj, head, count, lane, acc);
      else
        batch_items32<false>(P, H, s, mi, rj, head, count, lane, acc);
      head += count;
      __syncwarp();
    }
  }
  if (!F64) {
    eo += (double)acc.oh + (double)acc.ol;
    en += (double)acc.nh + (double)acc.nl;
    np += acc.np;
  }
}

// Warp sum of 64-bit counts (each below 2^48), in every lane: two integer
// reductions of 24-bit halves.
__device__ __forceinline__ long long warp_count(long long c) {
  const unsigned lo = __reduce_add_sync(~0u, (unsigned)(c & 0xffffff));
  const unsigned hi = __reduce_add_sync(~0u, (unsigned)(c >> 24));
  return ((long long)hi << 24) + (long long)lo;
}

// Group-wide deterministic sum of (a, b, c), the same in every thread.  The
// two halves of a warp take one sum each after the first exchange, and the
// warps' values are added by a second butterfly over the lanes: 10 FP64
// instructions a warp (adding the warps one by one in every thread took 15 +
// 3 per warp, and FP64 issues once in 16 cycles per SM).  At most 16 warps.
// Two calls must be separated by a group barrier (the scratch is reused).
__device__ __forceinline__ void group_reduce(const Group& g, const GroupSmem& s, double& a,
                                             double& b, long long& c, int par = 0) {
  const int lane = g.tid & 31, half = lane >> 4, k = lane & 15;
  double x = (half ? b : a) + __shfl_xor_sync(~0u, half ? a : b, 16);
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(~0u, x, off);
  const long long n = warp_count(c);
  const int nw = g.nwarps();
  double* red = s.red + par * 3 * nw;   // buffer `par` of two
  long long* redl = s.redl + par * nw;
  if (k == 0) red[half * nw + g.warp()] = x;
  if (lane == 0) redl[g.warp()] = n;
  g.sync();
  x = k < nw ? red[half * nw + k] : 0.0;
  c = (half == 0 && k < nw) ? redl[k] : 0;
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(~0u, x, off);
  a = __shfl_sync(~0u, x, 0);
  b = __shfl_sync(~0u, x, 16);
  c = warp_count(c);
}

// Writes the staged new placement of the moved molecule to the pool
// (master rows and mirrors); lanes of one warp.
__device__ __forceinline__ void commit(const Pool& P, const GroupSmem& s, const MovedInfo& mi,
                                       int lane) {
  for (int i = lane; i < mi.len; i += 32) {
    const int a = mi.atom0 + i;
    P.x[a] = s.nx[i];
    P.y[a] = s.ny[i];
    P.z[a] = s.nz[i];
    P.aoff[a] = s.o_new[i];
    P.aofl[a] = s.l_new[i];
  }
  const int2 pi = P.mpi[mi.mol];
  for (int k = lane; k < mi.npidx; k += 32) P.ppos[pi.x + k] = s.p_new[k];
  if (lane == 0) P.mfix[mi.mol] = mi.fx_new;
}

// Recomputes molecule m's mirrors (offsets, screen positions, fixed-point
// anchor) from its master rows; lanes [lane, nl).
__device__ __forceinline__ void refresh_molecule(const Pool& P, const ChainHdr& H, int m, int lane,
                                                 int nl) {
  const int a0 = P.mstart[m], len = P.mlen[m] & 255;
  const int2 pi = P.mpi[m];
  const int an = P.pidx[pi.x];
  const double ax = P.x[an], ay = P.y[an], az = P.z[an];
  for (int i = lane; i < len; i += nl) {
    const int a = a0 + i;
    const float w = P.aoff[a].w;
    const double vx = P.x[a] - ax, vy = P.y[a] - ay, vz = P.z[a] - az;
    const float4 o = make_float4((float)vx, (float)vy, (float)vz, w);
    P.aoff[a] = o;
    P.aofl[a] = make_float4((float)(vx - (double)o.x), (float)(vy - (double)o.y),
                            (float)(vz - (double)o.z), 0.f);
  }
  for (int k = lane; k < pi.y; k += nl) {
    const int q = P.pidx[pi.x + k];
    P.ppos[pi.x + k] = wrap_pos(P.x[q], P.y[q], P.z[q], H);
  }
  if (lane == 0) P.mfix[m] = fixpos(ax, ay, az, H);
}

}  // namespace mcgpu
