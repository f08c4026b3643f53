// chain.cuh -- the device-resident chain step: FP32 moves on the fixed-point
// + FP32-offset state (move_f32.cuh), screen and pair batches accumulated in
// double-float, decision in FP32 outside a guard band and in FP64 pairs
// inside it.  FP64 instructions are confined to a handful per step.
#pragma once

#include "kernels.cuh"
#include "move_f32.cuh"

namespace mcgpu {

// FP64 position of a chain atom: anchor (fixed point) + FP32 offset, each
// step rounded once (the CPU mirror computes the same two roundings).
__device__ __forceinline__ double chain_coord(unsigned A, float o, double L) {
  return __dadd_rn(__dmul_rn((double)A, L * 2.3283064365386963e-10), (double)o);
}

__device__ __forceinline__ double3 chain_pos3(uint4 A, float4 o, const ChainHdr& H) {
  return make_double3(chain_coord(A.x, o.x, H.L[0]), chain_coord(A.y, o.y, H.L[1]),
                      chain_coord(A.z, o.z, H.L[2]));
}

// The reference's cutoff test (SimulationStep.cpp:325-326, :332-342,
// :377-385) between FP64 positions.
__device__ __forceinline__ bool in_range_pos64(double3 p1, double3 p2, const ChainHdr& H) {
  const double dx = make_periodic(p2.x - p1.x, H.L[0]);
  const double dy = make_periodic(p2.y - p1.y, H.L[1]);
  const double dz = make_periodic(p2.z - p1.z, H.L[2]);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return r2 <= __dmul_rn(H.cutoff, H.cutoff);
}

// Screen position (FP32, wrapped into [0, L)) of an atom at anchor A with
// FP32 offset o.
__device__ __forceinline__ float4 chain_screen_pos(uint4 A, float4 o, const ChainHdr& H) {
  const unsigned x = A.x + (unsigned)fixstep(o.x, H.fxinvf[0]);
  const unsigned y = A.y + (unsigned)fixstep(o.y, H.fxinvf[1]);
  const unsigned z = A.z + (unsigned)fixstep(o.z, H.fxinvf[2]);
  return make_float4(__uint2float_rn(x) * H.fxs[0], __uint2float_rn(y) * H.fxs[1],
                     __uint2float_rn(z) * H.fxs[2], 0.f);
}

// misc[] slots written by stage_chain beyond load_moved's: new quaternion,
// acceptance uniform, "trial placement within skin/2 of the Verlet build"
// flag
enum : int { kMiscQn = 16, kMiscU = 20, kMiscNlTrial = 24 };

// One warp stages the proposed FP32 move `mv` of a chain molecule into
// slot s: old and new offsets (o_old, o_new), pair factors and |o|^2 (eq),
// screen positions of the primaries (p_old, p_new), old and new fixed-point
// anchors, the new quaternion.  No FP64.  It reads the molecule's rows
// only, so a move staged ahead stays valid until a commit of that molecule.
__device__ inline void stage_chain(const Pool& P, const ChainHdr& H, const MoveF& mv,
                                   const StageSlot& s, const float4* pcache, int lane) {
  const int m = H.mol0 + mv.mol;
  int a0, lw;
  int2 pi;
  if (H.uniform) {
    a0 = H.atom0 + mv.mol * H.ulen;
    lw = H.ulen | (H.uact << 8);
    pi = make_int2(H.pidx0 + mv.mol, 1);
  } else {
    a0 = P.mstart[m];
    lw = P.mlen[m];
    pi = P.mpi[m];
  }
  const int len = lw & 255;
  const float4 q4 = P.mq[m];
  const uint4 A = P.mfix[m];
  QuatF q;
  q.w = q4.x; q.x = q4.y; q.y = q4.z; q.z = q4.w;
  const QuatF qn = qnormalise(qmul(mv.qd, q));
  float R[9];
  qmatrix(qn, R);
  // anchor displacement from the vertex: o_v - R' t_v + d
  const float4 ov = P.aoff[a0 + mv.vertex];
  const float4 tv = P.atpl[a0 + mv.vertex];
  const float3 onv = mvec(R, tv.x, tv.y, tv.z);
  const float dlx = __fadd_rn(__fsub_rn(ov.x, onv.x), mv.dx);
  const float dly = __fadd_rn(__fsub_rn(ov.y, onv.y), mv.dy);
  const float dlz = __fadd_rn(__fsub_rn(ov.z, onv.z), mv.dz);
  uint4 An;
  An.x = A.x + (unsigned)fixstep(dlx, H.fxinvf[0]);
  An.y = A.y + (unsigned)fixstep(dly, H.fxinvf[1]);
  An.z = A.z + (unsigned)fixstep(dlz, H.fxinvf[2]);
  An.w = 0u;
  float qsum = 0.f;
  for (int i = lane; i < len; i += 32) {
    const int a = a0 + i;
    const float4 o = P.aoff[a];
    const float4 t = P.atpl[a];
    const float2 qe = P.aeq[a];
    const float3 on = mvec(R, t.x, t.y, t.z);
    s.o_old[i] = o;
    s.o_new[i] = make_float4(on.x, on.y, on.z, o.w);
    s.eq[i] = make_float4(qe.x, qe.y, fmaf(o.x, o.x, fmaf(o.y, o.y, o.z * o.z)),
                          fmaf(on.x, on.x, fmaf(on.y, on.y, on.z * on.z)));
    qsum += qe.y;
  }
  for (int off = 16; off > 0; off >>= 1) qsum += __shfl_xor_sync(~0u, qsum, off);
  __syncwarp();
  bool near = true;
  for (int k = lane; k < pi.y; k += 32) {
    const int slot = H.uniform ? H.uprim : P.pidx[pi.x + k] - a0;
    s.pa[k] = slot;
    s.p_old[k] = (k == 0 && pcache) ? pcache[m - H.mol0] : P.ppos[pi.x + k];
    const float4 pn = chain_screen_pos(An, s.o_new[slot], H);
    s.p_new[k] = pn;
    if (H.nl_on) near = near && r2_screen(pn, P.pbuild[pi.x + k], H) <= H.nl_half2;
  }
  near = __all_sync(~0u, near);
  if (lane == 0) {
    s.misc[0] = m; s.misc[1] = a0; s.misc[2] = len; s.misc[3] = pi.y;
    s.misc[4] = lw >> 8; s.misc[5] = 3; s.misc[6] = mv.vertex;
    s.misc[8] = (int)A.x; s.misc[9] = (int)A.y; s.misc[10] = (int)A.z;
    s.misc[12] = (int)An.x; s.misc[13] = (int)An.y; s.misc[14] = (int)An.z;
    s.misc[kMiscQn] = __float_as_int(qn.w); s.misc[kMiscQn + 1] = __float_as_int(qn.x);
    s.misc[kMiscQn + 2] = __float_as_int(qn.y); s.misc[kMiscQn + 3] = __float_as_int(qn.z);
    s.misc[kMiscU] = __float_as_int(mv.u);
    s.misc[kMiscNlTrial] = near ? 1 : 0;
    s.misc[kMiscRad] = __float_as_int(H.uniform ? H.umrad : P.mrad[m]);
    s.misc[kMiscQm] = __float_as_int(qsum);
  }
}

// Screen of candidate j against the staged molecule (both placements):
// FP32 distance of the screen positions, decided outright outside the
// guard band around rc^2 and by the reference's FP64 test inside it.  No
// global load outside the guard band (the positions come from the shared-
// memory cache); the entry's anchor differences are formed in the batch.
__device__ __forceinline__ int screen_chain(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                            const MovedInfo& mi, int j, float4 q0) {
  const int2 pj = H.simple_prim ? make_int2(H.pidx0 + (j - H.mol0), 1) : P.mpi[j];
  int f = 0;
  for (int k2 = 0; k2 < pj.y; k2++) {
    const float4 q = (k2 == 0) ? q0 : P.ppos[pj.x + k2];
    for (int k1 = 0; k1 < mi.npidx; k1++) {
      const float ro = r2_screen(s.p_old[k1], q, H);
      const float rn = r2_screen(s.p_new[k1], q, H);
      if (!(f & kInOld)) {
        if (ro <= H.cut2_lo) {
          f |= kInOld;
        } else if (ro <= H.cut2_hi) {
          const int p2 = P.pidx[pj.x + k2];
          const double3 a = chain_pos3(mi.fx_old, s.o_old[s.pa[k1]], H);
          const double3 b = chain_pos3(P.mfix[j], P.aoff[p2], H);
          if (in_range_pos64(a, b, H)) f |= kInOld;
        }
      }
      if (!(f & kInNew)) {
        if (rn <= H.cut2_lo) {
          f |= kInNew;
        } else if (rn <= H.cut2_hi) {
          const int p2 = P.pidx[pj.x + k2];
          const double3 a = chain_pos3(mi.fx_new, s.o_new[s.pa[k1]], H);
          const double3 b = chain_pos3(P.mfix[j], P.aoff[p2], H);
          if (in_range_pos64(a, b, H)) f |= kInNew;
        }
      }
    }
  }
  return f;
}

// Bits 4k + i: the LJ term between atoms i and k of a uniform chain's
// molecules (at most 4 atoms) is not exactly zero (sigma and epsilon
// products both nonzero in FP32).  The same for every lane.
__device__ __forceinline__ unsigned uniform_lj_mask(const Pool& P, const ChainHdr& H,
                                                    const float2* teq) {
  unsigned m = 0;
  if (!H.uniform || H.ulen > 4) return ~0u;
  for (int k = 0; k < H.ulen; k++)
    for (int i = 0; i < H.ulen; i++) {
      const float sk = P.aoff[H.atom0 + k].w, si = P.aoff[H.atom0 + i].w;
      if (si * sk != 0.f && teq[i].x * teq[k].x != 0.f) m |= 1u << (4 * k + i);
    }
  return m;
}

// The group evaluates both placements of the staged move over chain candidates
// [c_begin, c_end) -- or, with a Verlet list, the molecules cand[c_begin ..
// c_end).  Every warp screens its share in rounds of 32 (screen positions from
// the shared-memory cache when given) into its ring.  A chain of one species
// then shares the in-range neighbours of all warps out to the threads of the
// first `workers` warps as items (one more barrier): every warp waited for the
// one with most (4,000 16-atom molecules on 16 warps: 45 neighbours, 3 +- 2 a
// warp, 29,000 cycles a step).  Other chains evaluate their own rings in
// batches of 32, T lanes per neighbour molecule -- and so do chains of molecules of
// up to 3 sites, a lane per placement: there the extra barrier costs what the
// balance gains or more (512 water chains: 14.2 ms either way on 256 threads, 14.0
// against 16.5 on 160; 1,024 chains of 32 atoms, 64 steps on 64 threads 0.41 and 0.55;
// with lists on five warps the atoms would gain 6 % by sharing).
__device__ inline void group_eval_chain(const Pool& P, const ChainHdr& H, const Group& g,
                                        const GroupSmem& s, const MovedInfo& mi,
                                        const float4* pcache, int c_begin, int c_end, int workers,
                                        int T, AccFF& acc, const int* cand = nullptr) {
  const int lane = g.tid & 31, w = g.warp(), nw = g.nwarps();
  int* rj = s.lj + w * kRing;
  int head = 0, tail = 0;
  const unsigned lt = lanemask_lt();
  // all molecules: warp w screens blocks of 32 consecutive indices; a list
  // (short, in cell order): warp w takes every nw-th entry, so every warp
  // gets its share of the in-range neighbours
  const int rounds = cand ? (c_end - c_begin + 32 * nw - 1) / (32 * nw) : 0;
  const bool precise = H.precise != 0;
  const bool own = H.uniform && !precise && H.ulen <= 3;
  // (one warp has nobody to share with: where its teams, of one lane for 4 sites, would
  // be batch_ff's it takes that, both placements of a neighbour at once: 200 steps of 64
  // 64-atom molecules 66.8 ms, 77.4 by items; 256 chains of 64 4-site ones, 64 steps
  // 0.82 and 0.98)
  const bool teams = (H.ulen & (H.ulen - 1)) == 0;
  const bool shared = H.uniform && !own && !(nw == 1 && teams);
  const unsigned ljmask = H.ljmask;
  // one primary each (the common chain): the moved molecule's two placements
  // and the screen's constants in registers -- the header is global memory,
  // and the ring's stores would have it read again every round
  const bool single = H.simple_prim && mi.npidx == 1;
  const float Lx = H.Lf[0], Ly = H.Lf[1], Lz = H.Lf[2], lo = H.cut2_lo, hi = H.cut2_hi;
  const float4 po = s.p_old[0], pn = s.p_new[0];
  const int mol0 = H.mol0, pidx0 = H.pidx0;
  for (int it = 0;;) {
    // rounds of the screen until they end or the ring holds a batch (a shared
    // one waits for the other warps' with up to 32 entries)
    bool more = false;
    for (;; it++) {
      int idx;
      if (cand) {
        if (it >= rounds) break;
        idx = c_begin + (it * 32 + lane) * nw + w;
      } else {
        const int base = c_begin + w * 32 + it * nw * 32;
        if (base >= c_end) break;
        idx = base + lane;
      }
      if (tail - head > (shared ? 32 : 31)) {
        more = true;
        break;
      }
      const int j = (cand && idx < c_end) ? cand[idx] : idx;
      int f = 0;
      if (idx < c_end && j != mi.mol) {
        if (single) {
          const float4 q0 = pcache ? pcache[j - mol0] : P.ppos[pidx0 + (j - mol0)];
          const float ox = wrapf(q0.x - po.x, Lx), oy = wrapf(q0.y - po.y, Ly),
                      oz = wrapf(q0.z - po.z, Lz);
          const float nx = wrapf(q0.x - pn.x, Lx), ny = wrapf(q0.y - pn.y, Ly),
                      nz = wrapf(q0.z - pn.z, Lz);
          const float ro = fmaf(ox, ox, fmaf(oy, oy, oz * oz));
          const float rn = fmaf(nx, nx, fmaf(ny, ny, nz * nz));
          f = (ro <= lo ? kInOld : 0) | (rn <= lo ? kInNew : 0);
          if ((ro > lo && ro <= hi) || (rn > lo && rn <= hi))
            f = screen_chain(P, H, s, mi, j, q0);   // inside the guard band
        } else {
          const float4 q0 = pcache ? pcache[j - mol0]
                                   : P.ppos[H.simple_prim ? pidx0 + (j - mol0) : P.mpi[j].x];
          f = screen_chain(P, H, s, mi, j, q0);
        }
      }
      const unsigned bal = __ballot_sync(~0u, f != 0);
      if (f) rj[(tail + __popc(bal & lt)) & (kRing - 1)] = (j << 4) | f;
      tail += __popc(bal);
      if (shared) acc.np += __popc(f);
    }
    __syncwarp();
    if (!shared) {
      const int count = min(32, tail - head);
      if (count > 0) {
        if (own && H.ulen == 3)
          batch_un<3>(P, H, s, mi, rj, head, count, lane, acc, ljmask);
        else if (own && H.ulen == 1)
          batch_un<1>(P, H, s, mi, rj, head, count, lane, acc, ljmask);
        else if (own && H.ulen == 2)
          batch_un<2>(P, H, s, mi, rj, head, count, lane, acc, ljmask);
        else if (precise)
          batch_ff<true>(P, H, s, mi, rj, head, count, lane, T, acc);
        else
          batch_ff<false>(P, H, s, mi, rj, head, count, lane, T, acc);
        head += count;
      }
      __syncwarp();
      if (!more && tail == head) return;
      continue;
    }
    // entry e of the items: in the ring of the last warp q with pref <= e
    // (lane q of every warp holds q's ring head and pref, the entries before)
    int count = 32, tid = lane, threads = 32;
    const int k = lane & 15;
    int pref = k <= w ? 0 : 0x40000000, hd = head;   // this warp's own ring
    if (!more) {
      acc.np *= mi.act * H.uact;
      if (lane == 0) {
        s.hits[w] = tail - head;
        s.hits[16 + w] = head;
      }
      g.sync();
      if (w >= workers) return;
      const int cnt = k < nw ? s.hits[k] : 0;
      hd = s.hits[16 + k];
      pref = cnt;
#pragma unroll
      for (int off = 1; off < 16; off <<= 1) {
        const int v = __shfl_up_sync(~0u, pref, off, 16);
        if (k >= off) pref += v;
      }
      count = __shfl_sync(~0u, pref, 15);
      pref -= cnt;
      tid = g.tid;
      threads = 32 * workers;
    }
    auto entry = [&](int e) {
      int q = 0;
#pragma unroll
      for (int step = 8; step > 0; step >>= 1) {
        const int v = __shfl_sync(~0u, pref, q + step);
        if (q + step < nw && v <= e) q += step;
      }
      const int at = __shfl_sync(~0u, hd, q) + e - __shfl_sync(~0u, pref, q);
      return s.lj[q * kRing + (at & (kRing - 1))];
    };
    if (precise)
      uniform_items<true>(P, H, s, mi, count, tid, threads, T, acc, entry);
    else
      uniform_items<false>(P, H, s, mi, count, tid, threads, T, acc, entry);
    if (!more) return;
    head += 32;
    __syncwarp();
  }
}

// Group-wide deterministic double-float sum, the same in every thread.  After
// the first exchange the lower half of a warp carries the old placement's sum
// and the upper half the new one's, and the warps' values are added by a
// second butterfly over the lanes: a third of the instructions of reducing
// both sums in every lane and adding the warps one by one (a step of the 512
// water chains spent 1,250 of its 12,500 warp instructions there).
__device__ __forceinline__ void group_reduce_ff(const Group& g, const GroupSmem& s, AccFF& a,
                                                int par = 0) {
  const int lane = g.tid & 31, half = lane >> 4, k = lane & 15;
  float h = half ? a.nh : a.oh, l = half ? a.nl : a.ol;
  {
    const float oh = __shfl_xor_sync(~0u, half ? a.oh : a.nh, 16);
    const float ol = __shfl_xor_sync(~0u, half ? a.ol : a.nl, 16);
    ff_add2(h, l, oh, ol);
  }
  float ab = a.ab + __shfl_xor_sync(~0u, a.ab, 16);
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) {
    const float oh = __shfl_xor_sync(~0u, h, off), ol = __shfl_xor_sync(~0u, l, off);
    ff_add2(h, l, oh, ol);
    ab += __shfl_xor_sync(~0u, ab, off);
  }
  const long long n = warp_count(a.np);
  const int nw = g.nwarps();
  // buffer `par` of two; 5 floats per warp fit the 3 doubles reserved per warp
  float* red = (float*)(s.red + par * 3 * nw);
  long long* redl = s.redl + par * nw;
  if (k == 0) {
    red[5 * g.warp() + 2 * half] = h;
    red[5 * g.warp() + 2 * half + 1] = l;
  }
  if (lane == 0) {
    red[5 * g.warp() + 4] = ab;
    redl[g.warp()] = n;
  }
  g.sync();
  const bool on = k < nw;
  h = on ? red[5 * k + 2 * half] : 0.f;
  l = on ? red[5 * k + 2 * half + 1] : 0.f;
  ab = on ? red[5 * k + 4] : 0.f;
  a.np = warp_count(on && half == 0 ? redl[k] : 0);
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) {
    const float oh = __shfl_xor_sync(~0u, h, off), ol = __shfl_xor_sync(~0u, l, off);
    ff_add2(h, l, oh, ol);
    ab += __shfl_xor_sync(~0u, ab, off);
  }
  a.oh = __shfl_sync(~0u, h, 0);
  a.ol = __shfl_sync(~0u, l, 0);
  a.nh = __shfl_sync(~0u, h, 16);
  a.nl = __shfl_sync(~0u, l, 16);
  a.ab = ab;
}

// FP64 re-take of a step near the decision threshold: FP64 pair terms
// (pair_sum64, BruteForceStep.cpp:48-79) on the FP64 positions of the chain
// state (anchor + offset).  Warp 0 first writes the moved molecule's old
// and new FP64 coordinates and its FP64 parameters to shared memory; the
// caller synchronises.
__device__ inline void stage_chain_f64(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                       const MovedInfo& mi, int lane) {
  for (int i = lane; i < mi.len; i += 32) {
    const int a0 = mi.atom0 + i;
    const double2 bl = P.blend ? P.blend[a0] : blend64(P.sig[a0], P.eps[a0]);
    s.sd[i] = bl.x;
    s.ed[i] = bl.y;
    s.qd[i] = P.q[mi.atom0 + i];
    const double3 a = chain_pos3(mi.fx_old, s.o_old[i], H);
    const double3 b = chain_pos3(mi.fx_new, s.o_new[i], H);
    s.ox[i] = a.x; s.oy[i] = a.y; s.oz[i] = a.z;
    s.nx[i] = b.x; s.ny[i] = b.y; s.nz[i] = b.z;
  }
}

__device__ __forceinline__ void batch_chain64(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                              const MovedInfo& mi, const int* rj, int head,
                                              int count, int lane, double& eo, double& en,
                                              long long& np) {
  batch_items64(P, H, s, mi, rj, head, count, lane, eo, en, np,
                [&](int j, int b, double& x, double& y, double& z) {
                  const double3 p = chain_pos3(P.mfix[j], P.aoff[b], H);
                  x = p.x;
                  y = p.y;
                  z = p.z;
                });
}

// The FP64 re-take's screen: the reference's test for every primary pair
// on the chain state's FP64 positions.
//
// With a Verlet list (cand non-null), the molecules cand[c_begin .. c_end),
// every nw-th entry per warp as in group_eval_chain.
__device__ inline void warp_eval_chain64(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                  const MovedInfo& mi, const float4* pcache, int c_begin,
                                  int c_end, int w, int nw, int lane, double& eo,
                                  double& en, long long& np, const int* cand = nullptr) {
  int* rj = s.lj + w * kRing;
  int head = 0, tail = 0;
  const unsigned lt = lanemask_lt();
  const int rounds = cand ? (c_end - c_begin + 32 * nw - 1) / (32 * nw) : 0;
  for (int it = 0;; it++) {
    int idx;
    if (cand) {
      if (it >= rounds) break;
      idx = c_begin + (it * 32 + lane) * nw + w;
    } else {
      const int base = c_begin + w * 32 + it * nw * 32;
      if (base >= c_end) break;
      idx = base + lane;
    }
    const int j = (cand && idx < c_end) ? cand[idx] : idx;
    int f = 0;
    // the step's own screen: FP32 outside the guard band, the FP64 test on
    // these same FP64 positions inside it -- the FP64 in-range set exactly,
    // without an FP64 distance for every candidate
    if (idx < c_end && j != mi.mol) {
      float4 q0;
      if (pcache)
        q0 = pcache[j - H.mol0];
      else if (H.simple_prim)
        q0 = P.ppos[H.pidx0 + (j - H.mol0)];
      else
        q0 = P.ppos[P.mpi[j].x];
      f = screen_chain(P, H, s, mi, j, q0);
    }
    const unsigned bal = __ballot_sync(~0u, f != 0);
    if (f) rj[(tail + __popc(bal & lt)) & (kRing - 1)] = (j << 4) | f;
    tail += __popc(bal);
    if (tail - head >= 32) {
      __syncwarp();
      batch_chain64(P, H, s, mi, rj, head, 32, lane, eo, en, np);
      head += 32;
      __syncwarp();
    }
  }
  __syncwarp();
  if (tail > head) batch_chain64(P, H, s, mi, rj, head, tail - head, lane, eo, en, np);
  __syncwarp();
}

// Commit of an accepted chain move: offsets, quaternion, anchor, screen
// positions (and the shared-memory screen cache).
__device__ __forceinline__ void commit_chain(const Pool& P, const ChainHdr& H, const GroupSmem& s,
                                             const MovedInfo& mi, float4* pcache, int lane) {
  for (int i = lane; i < mi.len; i += 32) P.aoff[mi.atom0 + i] = s.o_new[i];
  const int2 pi = H.uniform ? make_int2(H.pidx0 + (mi.mol - H.mol0), 1) : P.mpi[mi.mol];
  for (int k = lane; k < mi.npidx; k += 32) P.ppos[pi.x + k] = s.p_new[k];
  if (lane == 0) {
    P.mfix[mi.mol] = mi.fx_new;
    P.mq[mi.mol] = make_float4(__int_as_float(s.misc[kMiscQn]), __int_as_float(s.misc[kMiscQn + 1]),
                               __int_as_float(s.misc[kMiscQn + 2]),
                               __int_as_float(s.misc[kMiscQn + 3]));
    if (pcache) pcache[mi.mol - H.mol0] = s.p_new[0];
  }
}

}  // namespace mcgpu
