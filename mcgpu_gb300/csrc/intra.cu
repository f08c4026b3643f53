// intra.cu -- flexible molecules on the plain path: the reference's
// intramolecular energy, bond stretch and angle expansion
// (src/Metropolis/SimulationStep.cpp:80-315), which it compiles but calls
// only with ENABLE_INTRA true (SimulationStep.h:15).
//
// A stage is one CTA on one molecule (a molecule has at most 64 atoms): the
// ops of the stage run in order in the first warp, each as a scalar set-up (the
// bond's unit vector or the plane normal) and one update per atom; then the
// molecule's mirrors and radius, and the intramolecular energy.  The union-
// find the reference runs on every call depends only on the bonds, so its
// partitions are computed once on the host at upload.  Coordinates follow
// the reference's FP64 operations one for one with explicit round-to-nearest
// intrinsics (no contraction) and the host's C-library cosines and sines, so
// they are the reference's bit for bit; the energies are FP64 sums in a
// different order (equal to the reference's within FP64 rounding).
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "intra.h"
#include "kernels.cuh"

namespace mcgpu {

namespace {

constexpr int kIntraThreads = 128;

// The SimCalcs pair terms of the intramolecular energy (SimulationStep.cpp:
// 344-375): blending by sqrt|a b| (sites with negative sigma or epsilon take
// part), no cutoff, zero at r = 0.  1/r from one FP64 rsqrt (a few ulps from
// the reference's sqrt and divisions, which cost many FP64 passes on this
// part); sigma^2 = |s_i s_j| and 4 eps = 4 sqrt|e_i e_j|, the root as the
// product of the atoms' own (the blending rows) where neither is negative.
__device__ __forceinline__ double intra_pair(const Pool& P, int i, int j, const ChainHdr& H) {
  const double dx = make_periodic(__dsub_rn(P.x[j], P.x[i]), H.L[0]);
  const double dy = make_periodic(__dsub_rn(P.y[j], P.y[i]), H.L[1]);
  const double dz = make_periodic(__dsub_rn(P.z[j], P.z[i]), H.L[2]);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  if (r2 == 0.0) return 0.0;
  const double ri = rsqrt(r2);
  const double ss = fabs(P.sig[i] * P.sig[j]);
  const double2 bi = P.blend[i], bj = P.blend[j];
  double ee = bi.y * bj.y;
  if (blend_skipped(bi.x) || blend_skipped(bj.x)) ee = sqrt(fabs(P.eps[i] * P.eps[j]));
  const double s2 = ss * (ri * ri);
  const double s6 = s2 * s2 * s2;
  const double lj = 4.0 * ee * (s6 * s6 - s6);
  return lj + P.q[i] * P.q[j] * 332.06 * ri;
}

// Block-wide deterministic sum (every thread gets it; at most 32 warps).  Warps
// from `active` on hold zeros and add nothing.  FP64 issues once in 16 cycles
// per SM, so the instructions of idle warps count: three values summed in every
// lane of eight warps took 312 of them, this takes 5 per active warp and 5 per
// warp.
__device__ __forceinline__ double block_sum(double a, int active, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (w < active)
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(~0u, a, off);
  __syncthreads();
  if (lane == 0) red[w] = a;
  __syncthreads();
  const int n = min(active, nw);
  a = lane < n ? red[lane] : 0.0;
  for (int off = 16; off > 0; off >>= 1)
    if (off < n) a += __shfl_xor_sync(~0u, a, off);
  return __shfl_sync(~0u, a, 0);
}

// SimCalcs::calcIntraMolecularEnergy (SimulationStep.cpp:80-129) of box
// molecule mol (pool molecule m), all threads of the block.
__device__ double intra_energy(const Pool& P, const IntraRows& R, const ChainHdr& H, int mol,
                               double* red) {
  const int m = H.mol0 + mol;
  const int tid = threadIdx.x, nt = blockDim.x;
  double sum = 0.0;
  int items = 0;
  if (R.flex_angles) {
    const int s = R.m_astart[mol], e = s + R.m_acount[mol];
    items = max(items, e - s);
    for (int k = s + tid; k < e; k += nt)
      if (R.a_var[k]) {
        const double d = R.a_eq[k] - R.a_size[k];
        sum += R.a_k[k] * d * d;
      }
  }
  if (R.flex_bonds) {
    const int s = R.m_bstart[mol], e = s + R.m_bcount[mol];
    items = max(items, e - s);
    for (int k = s + tid; k < e; k += nt)
      if (R.b_var[k]) {
        const double d = R.b_eq[k] - R.b_len[k];
        sum += R.b_k[k] * d * d;
      }
  }
  if (R.flex_bonds || R.flex_angles) {
    const int a0 = P.mstart[m], len = P.mlen[m] & 255;
    const int ty = R.m_type[mol], n = R.t_natom[ty];
    const unsigned char* code = R.code + R.t_off[ty];
    items = max(items, len * len);
    for (int q = tid; q < len * len; q += nt) {
      const int i = q / len, j = q - i * len;
      if (j <= i) continue;
      const int c = (i < n && j < n) ? code[i * n + j] : 2;
      if (c == 0) continue;
      const double e = intra_pair(P, a0 + i, a0 + j, H);
      sum += c == 1 ? 0.5 * e : e;
    }
  }
  return block_sum(sum, (items + 31) / 32, red);
}

// The molecule's mirrors after its atoms moved, and its radius (max
// distance of an atom from the first primary atom, with the margin the
// upload gives it): the FP32 pair paths decide per-pair images from it.
__device__ void refresh_flexible(const Pool& P, const ChainHdr& H, int m, double* red) {
  refresh_molecule(P, H, m, threadIdx.x, blockDim.x);
  const int a0 = P.mstart[m], len = P.mlen[m] & 255;
  const int an = P.pidx[P.mpi[m].x];
  double r = 0.0;
  for (int i = threadIdx.x; i < len; i += blockDim.x) {
    const double dx = P.x[a0 + i] - P.x[an], dy = P.y[a0 + i] - P.y[an],
                 dz = P.z[a0 + i] - P.z[an];
    r = fmax(r, sqrt(dx * dx + dy * dy + dz * dz));
  }
  // (only the warps that hold atoms)
  const int w = threadIdx.x >> 5, nw = min((int)blockDim.x >> 5, (len + 31) / 32);
  if (w < nw)
    for (int off = 16; off > 0; off >>= 1) r = fmax(r, __shfl_xor_sync(~0u, r, off));
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && w < nw) red[w] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 0; k < nw; k++) r = fmax(r, red[k]);
    P.mrad[m] = (float)(r * (1 + 1e-6) + 1e-4);
  }
}

__global__ void __launch_bounds__(kIntraThreads) k_intra_energy(Pool P, IntraRows R, int chain,
                                                                int mol, double* out) {
  __shared__ double red[3 * (kIntraThreads / 32)];
  const ChainHdr& H = P.hdr[chain];
  const double e = intra_energy(P, R, H, mol, red);
  if (threadIdx.x == 0) out[0] = e;
}

// One warp per molecule: a molecule's pairs are a few rounds of 32, and the
// block sum costs FP64 instructions in every warp.
__global__ void __launch_bounds__(32) k_intra_add(Pool P, IntraRows R, double* emol) {
  __shared__ double red[3];
  const ChainHdr& H = P.hdr[0];
  const int mol = blockIdx.x;
  const double e = intra_energy(P, R, H, mol, red);
  if (threadIdx.x == 0) emol[H.mol0 + mol] += e;
}

__global__ void __launch_bounds__(32) k_intra_add_boxes(const LoopTask* tasks) {
  __shared__ double red[3];
  const LoopTask& T = tasks[blockIdx.y];
  const int mol = blockIdx.x;
  if (!T.intra || mol >= T.n_mol) return;
  const double e = intra_energy(T.P, T.R, T.P.hdr[0], mol, red);
  if (threadIdx.x == 0) T.emol[mol] += e;
}

// Rows of one stage's ops in shared memory.
struct OpRows {
  double x[kMaxA], y[kMaxA], z[kMaxA];   // the molecule's coordinates
  double mx[kLoopSel], my[kLoopSel], mz[kLoopSel];  // a middle atom of another molecule
  int part[kLoopSel], e1[kLoopSel], e2[kLoopSel], mid[kLoopSel];  // local atoms; mid -1: mx..mz
  double v[9];
  int moved;
};

// n ops of one stage in order, SimCalcs::stretchBond (kind 0,
// SimulationStep.cpp:257-315) or SimCalcs::expandAngle (kind 1, :148-239) of
// entries idx[] of box molecule mol; trig[4 q ..]: the cosine and sine of the
// first and of the second group's angle.  Every thread of the block calls it;
// the first warp works, with the ops' rows and the coordinates in shared memory
// (an op is a chain of FP64 steps, and each followed three dependent loads and
// stood between two block barriers; 304 flexible boxes, 192 steps: 44.9 ms then,
// 42.4 this way).  Returns whether any op changed anything
// (a bond in a ring, an angle whose ends share a component do not).
__device__ bool apply_ops(const Pool& P, const IntraRows& R, const ChainHdr& H, int mol, int kind,
                          int n, const int* idx, const double* amt, const double* trig,
                          OpRows& W) {
  const int a0 = P.mstart[H.mol0 + mol], len = P.mlen[H.mol0 + mol] & 255;
  const int tid = threadIdx.x;
  if (tid < 32) {
    bool any = false;
    for (int q = tid; q < n; q += 32) {
      const int k = (kind == 0 ? R.m_bstart : R.m_astart)[mol] + idx[q];
      const int off = (kind == 0 ? R.b_part : R.a_part)[k];
      W.part[q] = off;
      any = any || off >= 0;
      const int base = a0 - H.atom0;
      W.e1[q] = (kind == 0 ? R.b_a1 : R.a_a1)[k] - base;
      W.e2[q] = (kind == 0 ? R.b_a2 : R.a_a2)[k] - base;
      if (kind == 1) {
        const int md = R.a_mid[k] - base;
        const bool in = md >= 0 && md < len;
        W.mid[q] = in ? md : -1;
        if (!in) {
          W.mx[q] = P.x[a0 + md];
          W.my[q] = P.y[a0 + md];
          W.mz[q] = P.z[a0 + md];
        }
      }
      // lengths and sizes: exact sums of the drawn amounts
      double* row = (kind == 0 ? R.b_len : R.a_size) + k;
      if (off >= 0) *row = __dadd_rn(*row, amt[q]);
    }
    for (int i = tid; i < len; i += 32) {
      W.x[i] = P.x[a0 + i];
      W.y[i] = P.y[a0 + i];
      W.z[i] = P.z[a0 + i];
    }
    any = __any_sync(~0u, any);
    if (tid == 0) W.moved = any;
    __syncwarp();
    for (int q = 0; q < n; q++) {
      const int off = W.part[q];
      if (off < 0) continue;   // the reference returns before moving
      const int e1 = W.e1[q], e2 = W.e2[q];
      if (kind == 0) {
        if (tid < 3) {
          // lanes 0-2 each form the whole vector and its length (same values)
          // and divide their own component: one division's latency, not
          // three.  (v / d) / 2 == (v / d) * 0.5 exactly.
          const double vx = __dsub_rn(W.x[e2], W.x[e1]);
          const double vy = __dsub_rn(W.y[e2], W.y[e1]);
          const double vz = __dsub_rn(W.z[e2], W.z[e1]);
          double d = __dadd_rn(0.0, __dmul_rn(vx, vx));
          d = __dadd_rn(d, __dmul_rn(vy, vy));
          d = __dadd_rn(d, __dmul_rn(vz, vz));
          d = __dsqrt_rn(d);
          const double vc = tid == 0 ? vx : (tid == 1 ? vy : vz);
          W.v[tid] = __dmul_rn(__dmul_rn(__ddiv_rn(vc, d), 0.5), amt[q]);
        }
        __syncwarp();
        for (int i = tid; i < len; i += 32) {
          const double sx = W.v[0], sy = W.v[1], sz = W.v[2];
          if (R.part[off + i] == 1) {
            W.x[i] = __dadd_rn(W.x[i], sx);
            W.y[i] = __dadd_rn(W.y[i], sy);
            W.z[i] = __dadd_rn(W.z[i], sz);
          } else {
            W.x[i] = __dsub_rn(W.x[i], sx);
            W.y[i] = __dsub_rn(W.y[i], sy);
            W.z[i] = __dsub_rn(W.z[i], sz);
          }
        }
        __syncwarp();
        continue;
      }
      if (tid < 3) {
        // lanes 0-2: the same normal and length, one component's division each
        const int md = W.mid[q];
        const double m0 = md >= 0 ? W.x[md] : W.mx[q], m1 = md >= 0 ? W.y[md] : W.my[q],
                     m2 = md >= 0 ? W.z[md] : W.mz[q];
        const double p0 = __dsub_rn(m0, W.x[e1]), p1 = __dsub_rn(m1, W.y[e1]),
                     p2 = __dsub_rn(m2, W.z[e1]);
        const double q0 = __dsub_rn(m0, W.x[e2]), q1 = __dsub_rn(m1, W.y[e2]),
                     q2 = __dsub_rn(m2, W.z[e2]);
        const double n0 = __dsub_rn(__dmul_rn(p1, q2), __dmul_rn(q1, p2));
        const double n1 = __dsub_rn(__dmul_rn(q0, p2), __dmul_rn(p0, q2));
        const double n2 = __dsub_rn(__dmul_rn(p0, q1), __dmul_rn(q0, p1));
        double nl = __dadd_rn(0.0, __dmul_rn(n0, n0));
        nl = __dadd_rn(nl, __dmul_rn(n1, n1));
        nl = __dadd_rn(nl, __dmul_rn(n2, n2));
        nl = __dsqrt_rn(nl);
        const double nc = tid == 0 ? n0 : (tid == 1 ? n1 : n2);
        W.v[tid] = __ddiv_rn(nc, nl);
        W.v[3 + tid] = tid == 0 ? m0 : (tid == 1 ? m1 : m2);
      }
      __syncwarp();
      for (int i = tid; i < len; i += 32) {
        const int lab = R.part[off + i];
        if (lab) {
          const double cs = trig[4 * q + (lab == 1 ? 0 : 2)];
          const double sn = trig[4 * q + (lab == 1 ? 1 : 3)];
          const double omc = __dsub_rn(1.0, cs);
          const double u0 = W.v[0], u1 = W.v[1], u2 = W.v[2];
          const double t0 = __dsub_rn(W.x[i], W.v[3]), t1 = __dsub_rn(W.y[i], W.v[4]),
                       t2 = __dsub_rn(W.z[i], W.v[5]);
          double dot = __dadd_rn(0.0, __dmul_rn(t0, u0));
          dot = __dadd_rn(dot, __dmul_rn(t1, u1));
          dot = __dadd_rn(dot, __dmul_rn(t2, u2));
          const double k0 = __dsub_rn(__dmul_rn(u1, t2), __dmul_rn(t1, u2));
          const double k1 = __dsub_rn(__dmul_rn(t0, u2), __dmul_rn(u0, t2));
          const double k2 = __dsub_rn(__dmul_rn(u0, t1), __dmul_rn(t0, u1));
          const double r0 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(u0, dot), omc),
                                                __dmul_rn(t0, cs)), __dmul_rn(k0, sn));
          const double r1 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(u1, dot), omc),
                                                __dmul_rn(t1, cs)), __dmul_rn(k1, sn));
          const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(u2, dot), omc),
                                                __dmul_rn(t2, cs)), __dmul_rn(k2, sn));
          W.x[i] = __dadd_rn(r0, W.v[3]);
          W.y[i] = __dadd_rn(r1, W.v[4]);
          W.z[i] = __dadd_rn(r2, W.v[5]);
        }
      }
      __syncwarp();
    }
    if (any)
      for (int i = tid; i < len; i += 32) {
        P.x[a0 + i] = W.x[i];
        P.y[a0 + i] = W.y[i];
        P.z[a0 + i] = W.z[i];
      }
  }
  __syncthreads();
  return W.moved != 0;
}

// SimCalcs::saveBonds / saveAngles (SimulationStep.cpp:678-701), all threads.
__device__ void save_rows(const IntraRows& R, int mol) {
  for (int k = R.m_bstart[mol] + threadIdx.x; k < R.m_bstart[mol] + R.m_bcount[mol];
       k += blockDim.x)
    R.b_len_rb[k] = R.b_len[k];
  for (int k = R.m_astart[mol] + threadIdx.x; k < R.m_astart[mol] + R.m_acount[mol];
       k += blockDim.x)
    R.a_size_rb[k] = R.a_size[k];
}

// Rollback with the ENABLE_INTRA branch (SimulationStep.cpp:731-775):
// coordinates from the rollback copy, angle sizes and bond lengths from
// theirs, then the mirrors; all threads.
__device__ void rollback_rows(const Pool& P, const IntraRows& R, const ChainHdr& H, int chain,
                              int mol, double* red) {
  const int m = H.mol0 + mol;
  const int a0 = P.mstart[m], len = P.mlen[m] & 255;
  const double* rb = P.rb + (size_t)chain * 3 * H.max_len;
  for (int i = threadIdx.x; i < len; i += blockDim.x) {
    P.x[a0 + i] = rb[i];
    P.y[a0 + i] = rb[H.max_len + i];
    P.z[a0 + i] = rb[2 * H.max_len + i];
  }
  for (int k = R.m_astart[mol] + threadIdx.x; k < R.m_astart[mol] + R.m_acount[mol];
       k += blockDim.x)
    R.a_size[k] = R.a_size_rb[k];
  for (int k = R.m_bstart[mol] + threadIdx.x; k < R.m_bstart[mol] + R.m_bcount[mol];
       k += blockDim.x)
    R.b_len[k] = R.b_len_rb[k];
  __syncthreads();
  refresh_flexible(P, H, m, red);
}

__global__ void __launch_bounds__(kIntraThreads) k_intra_ops(Pool P, IntraRows R, int chain,
                                                             IntraOps ops, double* out) {
  __shared__ double red[3 * (kIntraThreads / 32)];
  __shared__ OpRows W;
  __shared__ int idx[kIntraOps];
  __shared__ double amt[kIntraOps], trig[4 * kIntraOps];
  const ChainHdr& H = P.hdr[chain];
  const int mol = ops.mol, m = H.mol0 + mol;
  const int tid = threadIdx.x;
  if (ops.flags & kIntraSave) save_rows(R, mol);
  __syncthreads();
  if (ops.flags & kIntraEnergyBefore) {
    const double e = intra_energy(P, R, H, mol, red);
    if (tid == 0) out[0] = e;
  }
  if (tid < ops.n) {
    idx[tid] = ops.idx[tid];
    amt[tid] = ops.amt[tid];
    trig[4 * tid] = ops.c1[tid];
    trig[4 * tid + 1] = ops.s1[tid];
    trig[4 * tid + 2] = ops.c2[tid];
    trig[4 * tid + 3] = ops.s2[tid];
  }
  __syncthreads();
  if (apply_ops(P, R, H, mol, ops.kind, ops.n, idx, amt, trig, W)) {
    refresh_flexible(P, H, m, red);
    __syncthreads();
  }
  if (ops.flags & kIntraEnergyAfter) {
    const double e = intra_energy(P, R, H, mol, red);
    if (tid == 0) out[1] = e;
  }
}

__global__ void __launch_bounds__(kIntraThreads) k_intra_rollback(Pool P, IntraRows R, int chain,
                                                                  int mol) {
  __shared__ double red[3 * (kIntraThreads / 32)];
  rollback_rows(P, R, P.hdr[chain], chain, mol, red);
}

// ---- the reference's loop on the device ----------------------------------------

constexpr int kLoopThreads = 256;
constexpr int kLoopDrawCap = 1 << 20;

// randomReal (MathLibrary.cpp:31-33) of a number of the restated C-library
// stream, operation by operation.
__device__ __forceinline__ double real_of(int32_t v, double start, double end) {
  return __dadd_rn(__dmul_rn(__dsub_rn(end, start), crand_unit(v)), start);
}
__device__ __forceinline__ double loop_real(CRand& g, double start, double end) {
  return real_of(crand_next(g), start, end);
}

// acceptMove (SimulationStep.cpp:794-803): no draw for a decrease.
__device__ __forceinline__ bool loop_accept(CRand& g, double de, double kT) {
  if (de < 0) return true;
  return exp(-(de) / kT) >= loop_real(g, 0.0, 1.0);
}

// Scratch of cta_eval: per warp the in-range candidates of a segment, their atoms'
// items, and (mixed lengths) each entry's first item.
constexpr int kLoopWarps = kLoopThreads / 32;
struct EvalRows {
  int ent[kLoopWarps], tot[kLoopWarps];
  int first[kLoopWarps * kRing];
};

// The staged molecule's pair energies with all others, one share per thread of
// the kLoopThreads of grp (group_reduce adds them).  The warps screen 64
// candidates each, then all items (placement, entry, neighbour atom) of the
// segment are dealt over the CTA's lanes: with each warp evaluating its own hits
// a warp's last round was part full and the warps' counts differed (FP64 issues a
// warp instruction in 16 cycles however few lanes work).  Where the items leave
// warps idle the moved molecule's atoms are dealt too (FP64 pairs; the FP32 items
// factor the whole molecule's charge).  256 waters, FP64: 24.4 us a step with the
// warps' own hits, 22.8 pooled; 304 flexible boxes (192 steps) 42.4 and 40.7 ms.
template <bool F64>
__device__ void cta_eval(const Pool& P, const ChainHdr& H, const Group& grp, const GroupSmem& s,
                         const MovedInfo& mi, EvalRows& E, double& eo, double& en,
                         long long& np) {
  const int lane = grp.tid & 31, w = grp.warp();
  const unsigned lt = lanemask_lt();
  const bool uni = H.uniform != 0;
  const int two = mi.states == 3 ? 2 : 1;
  const int c_end = H.mol0 + H.n_mol;
  int* rj = s.lj + w * kRing;
  AccFF acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0};
  for (int base = H.mol0; base < c_end; base += kLoopWarps * kRing) {
    if (base > H.mol0) grp.sync();   // the last segment's entries are read
    int cnt = 0, tot = 0;
#pragma unroll
    for (int r = 0; r < kRing / 32; r++) {
      const int j0 = base + (r * kLoopWarps + w) * 32;
      if (j0 >= c_end) break;
      const int j = j0 + lane;
      int f = 0;
      // the FP32 screen with the FP64 re-test inside its guard band gives the
      // FP64 test's in-range set exactly, for FP64 and FP32 pair terms alike
      if (j < c_end && j != mi.mol) f = screen_mixed(P, H, s, mi, j);
      const unsigned bal = __ballot_sync(~0u, f != 0);
      const int at = cnt + __popc(bal & lt);
      if (f) rj[at] = (j << 4) | f;
      cnt += __popc(bal);
      const int hits = __popc(f & (kInOld | kInNew));
      if (uni) {
        np += (long long)hits * (mi.act * H.uact);
        continue;
      }
      const int lw = f ? P.mlen[j] : 0;
      np += (long long)hits * (mi.act * (lw >> 8));
      int pre = lw & 255;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(~0u, pre, off);
        if (lane >= off) pre += v;
      }
      if (f) E.first[w * kRing + at] = tot + pre - (lw & 255);
      tot += __shfl_sync(~0u, pre, 31);
    }
    if (lane == 0) {
      E.ent[w] = cnt;
      E.tot[w] = tot;
    }
    grp.sync();
    int entries = 0, total = 0;
#pragma unroll
    for (int v = 0; v < kLoopWarps; v++) {
      entries += E.ent[v];
      total += E.tot[v];
    }
    if (uni) total = entries * H.ulen;
    const int items = total * two;
    // a part takes whole warps: pair_sum64's votes need the lanes of a warp on the
    // same atoms
    const int span = (items + 31) & ~31;
    const int parts = F64 && items > 0 ? max(1, min(mi.len, kLoopThreads / span)) : 1;
    for (int it = grp.tid; it < span * parts; it += kLoopThreads) {
      const int part = it / span;
      int local = it - part * span;
      if (local >= items) continue;
      const bool use_new = local >= total || mi.states == 2;
      if (local >= total) local -= total;
      // item -> (warp's ring, entry, atom): all entries' first atoms, then their
      // second ones in a uniform box; entry by entry with mixed lengths
      int k = 0, at = local, v = 0;
      if (uni) {
        k = local / entries;
        at = local - k * entries;
      }
      while (v < kLoopWarps - 1 && at >= (uni ? E.ent[v] : E.tot[v])) {
        at -= uni ? E.ent[v] : E.tot[v];
        v++;
      }
      if (!uni) {
        const int n_e = E.ent[v];
        int e = 0;
#pragma unroll
        for (int step = kRing / 2; step > 0; step >>= 1)
          if (e + step < n_e && E.first[v * kRing + e + step] <= at) e += step;
        k = at - E.first[v * kRing + e];
        at = e;
      }
      const int jf = s.lj[v * kRing + at];
      if (!(jf & (use_new ? kInNew : kInOld))) continue;
      const int j = jf >> 4;
      const int b = (uni ? H.atom0 + (j - H.mol0) * H.ulen : P.mstart[j]) + k;
      if (F64) {
        const int i0 = part * mi.len / parts, n_i = (part + 1) * mi.len / parts - i0;
        const double2 bl = P.blend[b];
        const double e = pair_sum64(
            (use_new ? s.nx : s.ox) + i0, (use_new ? s.ny : s.oy) + i0,
            (use_new ? s.nz : s.oz) + i0, s.sd + i0, s.ed + i0, s.qd + i0, n_i, P.x[b], P.y[b],
            P.z[b], bl.x, bl.y, P.q[b], H.L[0], H.L[1], H.L[2]);
        if (use_new) en += e; else eo += e;
      } else {
        const float e = H.precise ? pair_item32<true>(P, H, s, mi, j, b, use_new)
                                  : pair_item32<false>(P, H, s, mi, j, b, use_new);
        if (use_new)
          ff_add(acc.nh, acc.nl, e);
        else
          ff_add(acc.oh, acc.ol, e);
      }
    }
  }
  if (!F64) {
    eo += (double)acc.oh + (double)acc.ol;
    en += (double)acc.nh + (double)acc.nl;
  }
}

// The first warp: the draws of one stage of intramolecularMove (kind 0 bonds,
// :589-609; kind 1 angles, :621-640): how many, which (a std::set's distinct
// draws in ascending order), an amount each; the variable entries go to
// sel / amt, and for angles the cosines and sines of their two groups to trig.
// Lane 0 takes the numbers; the amounts, variable flags and sines are formed
// side by side (one after another in lane 0 they took 15,000 cycles a stage,
// most of them sines).  Returns the count the counters take, or -1 when the set
// did not fill within the draw cap; every lane gets it and *n_sel.
__device__ int loop_draw_stage(CRand& g, const IntraRows& R, int mol, int kind, double delta,
                               int max_moves, int* sel, double* amt, double* trig, int32_t* raw,
                               int* n_sel) {
  const int lane = threadIdx.x & 31;
  const int count = kind == 0 ? R.m_bcount[mol] : R.m_acount[mol];
  const int start = kind == 0 ? R.m_bstart[mol] : R.m_astart[mol];
  const int* var = kind == 0 ? R.b_var : R.a_var;
  int n = count;
  if (lane == 0) {
    if (n > 3) n = min((int)loop_real(g, 2, count), max_moves);
    int have = 0, draws = 0;
    while (have < n) {
      if (++draws > kLoopDrawCap) {
        n = -1;
        break;
      }
      const int v = min((int)loop_real(g, 0, count), count - 1);
      int pos = 0;
      while (pos < have && sel[pos] < v) pos++;
      if (pos < have && sel[pos] == v) continue;
      for (int k = have; k > pos; k--) sel[k] = sel[k - 1];
      sel[pos] = v;
      have++;
    }
    for (int k = 0; k < n; k++) raw[k] = crand_next(g);
  }
  n = __shfl_sync(~0u, n, 0);
  __syncwarp();
  if (n < 0) return n;
  // 0.25 + (0.75 / n) * intraScaleFactor, rounded step by step as the host does
  const double scale = __dadd_rn(0.25, __dmul_rn(__ddiv_rn(0.75, (double)n), 0.625));
  int ns = 0;
  for (int k0 = 0; k0 < n; k0 += 32) {
    const int k = k0 + lane;
    int e = 0;
    bool on = false;
    double d = 0.0;
    if (k < n) {
      e = sel[k];
      on = var[start + e] != 0;
      d = __dmul_rn(scale, real_of(raw[k], -delta, delta));
    }
    const unsigned bal = __ballot_sync(~0u, on);
    __syncwarp();
    if (on) {
      const int at = ns + __popc(bal & lanemask_lt());   // at <= k: entries not read yet
      sel[at] = e;
      amt[at] = d;
    }
    ns += __popc(bal);
    __syncwarp();
  }
  if (kind == 1) {
    const double deg2rad = 3.14159256358979323846264 / 180.0;   // expandAngle's constant
    for (int q = lane; q < 2 * ns; q += 32) {
      const double a = amt[q >> 1];
      sincos(__dmul_rn(a, (q & 1) ? deg2rad : -deg2rad), &trig[2 * q + 1], &trig[2 * q]);
    }
  }
  *n_sel = ns;
  __syncwarp();
  return n;
}

// The loop of a box with the intramolecular term and moves, one CTA a box.
template <bool F64>
__global__ void __launch_bounds__(kLoopThreads) k_plain_steps(const LoopTask* tasks, int n_steps,
                                                              SmemShape shape) {
  extern __shared__ __align__(16) char smem[];
  __shared__ LoopTask task;
  if (threadIdx.x == 0) task = tasks[blockIdx.x];
  __syncthreads();
  if (!task.intra) return;   // k_plain_rigid's
  const Pool& P = task.P;
  const IntraRows& R = task.R;
  PlainLoop* L = task.L;
  __shared__ PlainLoop st;
  __shared__ Proposal prop;
  __shared__ int32_t raw[kLoopSel];
  __shared__ double red[3 * (kLoopThreads / 32)];
  __shared__ OpRows W;
  __shared__ EvalRows E;
  __shared__ int sel[kLoopSel];
  __shared__ double amt[kLoopSel], trig[4 * kLoopSel];
  __shared__ int n_sel, flag, stop;
  const ChainHdr& H = P.hdr[0];
  Group grp{(int)threadIdx.x, (int)blockDim.x, 1};
  GroupSmem s = shape.carve(smem);
  const int tid = threadIdx.x, lane = tid & 31, w = grp.warp();
  const int n = H.n_mol;
  const double kT = H.kT, max_t = H.max_t, max_r = H.max_r;
  if (tid == 0) {
    st = *L;
    stop = 0;
  }
  __syncthreads();
  for (int k = 0; k < n_steps; k++) {
    if (w == 0) {
      // chooseMolecule and the seven intermolecularMove draws
      // (SimulationStep.cpp:25-27, 527-535), clamped as the host loop clamps:
      // lane 0 takes the numbers, lane k forms the k-th real
      if (lane == 0)
        for (int q = 0; q < 8; q++) raw[q] = crand_next(st.rng);
      __syncwarp();
      const int32_t v = raw[lane & 7];
      const int mol = min((int)real_of(raw[0], 0, n), n - 1);
      const int len = P.mlen[H.mol0 + mol] & 255;
      const double top = lane < 5 ? max_t : max_r;
      const double x = lane == 1 ? real_of(v, 0, len) : real_of(v, -top, top);
      if (lane == 0) {
        prop.mol = mol;
        prop.trig = 0;
      }
      if (lane == 1) prop.vertex = min((int)x, len - 1);
      if (lane == 2) prop.dx = x;
      if (lane == 3) prop.dy = x;
      if (lane == 4) prop.dz = x;
      if (lane == 5) prop.r0 = x;
      if (lane == 6) prop.r1 = x;
      if (lane == 7) prop.r2 = x;
    }
    __syncthreads();
    const int mol = prop.mol, m = H.mol0 + mol;
    double eo = 0.0, en = 0.0;
    long long np = 0;
    const double ei_old = intra_energy(P, R, H, mol, red);
    if (w == 0) stage(P, H, m, nullptr, s, lane);
    grp.sync();
    {
      const MovedInfo mi = load_moved(s);
      cta_eval<F64>(P, H, grp, s, mi, E, eo, en, np);
      group_reduce(grp, s, eo, en, np);
    }
    const double e_old = eo + ei_old;
    long long pairs = np;
    __syncthreads();
    // the rigid move: rollback copy, move, wrap, commit
    if (w == 0) {
      stage(P, H, m, &prop, s, lane);
      __syncwarp();
      const MovedInfo mi = load_moved(s);
      double* rb = P.rb;
      for (int i = lane; i < mi.len; i += 32) {
        rb[i] = s.ox[i];
        rb[H.max_len + i] = s.oy[i];
        rb[2 * H.max_len + i] = s.oz[i];
      }
      commit(P, s, mi, lane);
    }
    __syncthreads();
    // SimCalcs::intramolecularMove (SimulationStep.cpp:568-675)
    save_rows(R, mol);
    const double bond_delta = st.max_bond_delta, angle_delta = st.max_angle_delta;
    __syncthreads();
    double cur = 0.0;
    bool have_cur = false;
    for (int kind = 0; kind < 2; kind++) {
      if (kind == 0 ? !R.flex_bonds : !R.flex_angles) continue;
      if (w == 0) {
        int ns = 0;
        const int cnt = loop_draw_stage(st.rng, R, mol, kind, kind == 0 ? bond_delta : angle_delta,
                                        st.max_intra_moves, sel, amt, trig, raw, &ns);
        if (lane == 0) {
          if (cnt < 0) {
            st.error = 1;
            stop = 1;
          } else if (kind == 0) {
            st.bond_moves += cnt;
          } else {
            st.angle_moves += cnt;
          }
          flag = cnt;
          n_sel = ns;
        }
      }
      __syncthreads();
      if (stop) break;
      const int cnt = flag;
      const double e0 = have_cur ? cur : intra_energy(P, R, H, mol, red);
      if (apply_ops(P, R, H, mol, kind, n_sel, sel, amt, trig, W)) {
        refresh_flexible(P, H, m, red);
        __syncthreads();
      }
      const double e1 = intra_energy(P, R, H, mol, red);
      if (tid == 0 && loop_accept(st.rng, e1 - e0, kT)) {
        if (kind == 0)
          st.bond_accepted += cnt;
        else
          st.angle_accepted += cnt;
      }
      cur = e1;
      have_cur = true;
      __syncthreads();
    }
    if (stop) break;
    if (tid == 0 && st.step != 0 && (st.step % 1000) == 0) {
      // width tuning (:656-674); the angle test reads the entry width
      const double bond_ratio = (double)st.bond_accepted / st.bond_moves;
      const double angle_ratio = (double)st.angle_accepted / st.angle_moves;
      double diff = bond_ratio - 0.4;
      if (fabs(diff) > 0.0001)
        st.max_bond_delta = __dadd_rn(st.max_bond_delta, __dmul_rn(st.max_bond_delta, diff));
      diff = angle_ratio - 0.4;
      if (fabs(angle_delta) > 0.0001)
        st.max_angle_delta = __dadd_rn(st.max_angle_delta, __dmul_rn(st.max_angle_delta, diff));
      st.bond_accepted = st.bond_moves = 0;
      st.angle_accepted = st.angle_moves = 0;
    }
    // the new energy: the intramolecular part is the last stage's (the same
    // coordinates and rows), else computed here
    const double ei_new = have_cur ? cur : intra_energy(P, R, H, mol, red);
    if (w == 0) stage(P, H, m, nullptr, s, lane);
    grp.sync();
    eo = en = 0.0;
    np = 0;
    {
      const MovedInfo mi = load_moved(s);
      cta_eval<F64>(P, H, grp, s, mi, E, eo, en, np);
      group_reduce(grp, s, eo, en, np);
    }
    if (tid == 0) {
      const double de = (eo + ei_new) - e_old;
      flag = loop_accept(st.rng, de, kT);
      st.pairs += pairs + np;
      if (flag) {
        st.energy += de;
        st.accepted++;
      } else {
        st.rejected++;
      }
      st.step++;
    }
    __syncthreads();
    if (!flag) rollback_rows(P, R, H, 0, mol, red);
    __syncthreads();
  }
  if (tid == 0) *L = st;
}

// chooseMolecule and the seven intermolecularMove draws (SimulationStep.cpp:25-27,
// 527-535) of words v0 (the first) and v (word lane & 7), clamped as the host loop
// clamps; lane k of NL forms the k-th real.
__device__ __forceinline__ void loop_propose(const Pool& P, const ChainHdr& H, int32_t v0,
                                             int32_t v, int lane, Proposal& prop) {
  const int n = H.n_mol;
  const int mol = min((int)real_of(v0, 0, n), n - 1);
  const int len = P.mlen[H.mol0 + mol] & 255;
  const double top = lane < 5 ? H.max_t : H.max_r;
  const double x = lane == 1 ? real_of(v, 0, len) : real_of(v, -top, top);
  if (lane == 0) {
    prop.mol = mol;
    prop.trig = 0;
  }
  if (lane == 1) prop.vertex = min((int)x, len - 1);
  if (lane == 2) prop.dx = x;
  if (lane == 3) prop.dy = x;
  if (lane == 4) prop.dz = x;
  if (lane == 5) prop.r0 = x;
  if (lane == 6) prop.r1 = x;
  if (lane == 7) prop.r2 = x;
}

// The generator as its last words: word k of the stream (the state's own 31
// first) in slot k mod 64.  One warp makes nine words at a time:
// x[k] = x[k-3] + x[k-31] is three interleaved running sums.
constexpr int kWords = 64;
__device__ __forceinline__ void words_next(uint32_t* ring, int& made, int lane) {
  uint32_t v = ring[(made + lane - 31) & (kWords - 1)];
  if (lane < 3) v += ring[(made + lane - 3) & (kWords - 1)];
  const uint32_t a = __shfl_up_sync(~0u, v, 3);
  if (lane >= 3) v += a;
  const uint32_t b = __shfl_up_sync(~0u, v, 6);
  if (lane >= 6) v += b;
  __syncwarp();
  if (lane < 9) ring[(made + lane) & (kWords - 1)] = v;
  made += 9;
  __syncwarp();
}

// The loop of a rigid box, one CTA a box: eight warps evaluate the staged move,
// and a ninth meanwhile draws and stages the next one.  Whether the acceptance
// takes a number is not known yet, so its halves stage the two moves that can
// follow, from the next word and the one after it; the step's end picks one.
// (A move of the molecule that was just moved is staged again.)  Draws and staging
// are FP64 chains of one warp: with the other warps waiting for them a step of
// 256 waters took 22.8 us, this way 16.9.
constexpr int kRigidThreads = kLoopThreads + 32;

template <bool F64>
__global__ void __launch_bounds__(kRigidThreads, 2) k_plain_rigid(const LoopTask* tasks, int n_steps,
                                                               SmemShape shape) {
  extern __shared__ __align__(16) char smem[];
  __shared__ LoopTask task;
  __shared__ Proposal prop[2];
  __shared__ EvalRows E;
  __shared__ uint32_t ring[kWords];
  __shared__ int dec[2];   // of even and odd steps; bit 0: accepted, bit 1: a word taken
  if (threadIdx.x == 0) task = tasks[blockIdx.x];
  __syncthreads();
  if (task.intra) return;   // k_plain_steps'
  const Pool& P = task.P;
  PlainLoop* L = task.L;
  const ChainHdr& H = P.hdr[0];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int half = lane >> 4, hl = lane & 15;
  const bool helper = w == kLoopWarps;
  Group grp{tid, kLoopThreads, 1};
  const int slot_bytes = shape.bytes();
  const double kT = H.kT;
  double energy = L->energy;
  long long accepted = 0, pairs = 0;
  if (tid < 31) ring[tid] = (uint32_t)L->rng.r[(L->rng.f + tid) % 31];
  __syncthreads();
  // pos: the words consumed up to the step's own draws; made: the words there are
  int pos = 31, made = 31, cur = 0;
  // the moves drawn from word `from` (first half) and the one after it into slots
  // s0 and s0 + 1 mod 3
  auto prepare = [&](int from, int s0) {
    while (made < from + 10) words_next(ring, made, lane);
    const int at = from + half;
    loop_propose(P, H, (int32_t)(ring[at & (kWords - 1)] >> 1),
                 (int32_t)(ring[(at + (hl & 7)) & (kWords - 1)] >> 1), hl, prop[half]);
    __syncwarp();
    const GroupSmem t = shape.carve(smem + ((s0 + half) % 3) * slot_bytes);
    stage<16>(P, H, H.mol0 + prop[half].mol, &prop[half], t, hl);
  };
  if (helper) prepare(pos, 0);
  pos += 8;
  __syncthreads();
  for (int k = 0; k < n_steps; k++) {
    const GroupSmem s = shape.carve(smem + cur * slot_bytes);
    const MovedInfo mi = load_moved(s);
    const int ahead = (cur + 1) % 3;
    if (helper) {
      if (k + 1 < n_steps) prepare(pos, ahead);
    } else {
      double eo = 0.0, en = 0.0;
      long long np = 0;
      cta_eval<F64>(P, H, grp, s, mi, E, eo, en, np);
      group_reduce(grp, s, eo, en, np);
      if (tid == 0) {
        // acceptMove (SimulationStep.cpp:794-803): no draw for a decrease
        const double de = en - eo;
        const bool draw = !(de < 0);
        const bool acc =
            !draw || exp(-(de) / kT) >= real_of((int32_t)(ring[pos & (kWords - 1)] >> 1), 0.0, 1.0);
        pairs += np;
        if (acc) {
          energy += de;
          accepted++;
        }
        dec[k & 1] = (acc ? 1 : 0) | (draw ? 2 : 0);
      }
    }
    __syncthreads();
    const int d = dec[k & 1], took = d >> 1;
    pos += took;
    cur = (ahead + took) % 3;
    if (d & 1) {
      // (read before the barrier: the helper's next draws come after it)
      const bool again = k + 1 < n_steps && H.mol0 + prop[took].mol == mi.mol;
      if (w == 0) commit(P, s, mi, lane);
      __syncthreads();
      if (again) {
        if (helper)
          stage<16>(P, H, mi.mol, &prop[took], shape.carve(smem + ((ahead + half) % 3) * slot_bytes),
                    hl);
        __syncthreads();
      }
    }
    if (k + 1 < n_steps) pos += 8;
  }
  // the generator's state after pos words: its last 31, the oldest next
  if (tid < 31) L->rng.r[tid] = (int32_t)ring[(pos - 31 + tid) & (kWords - 1)];
  if (tid == 0) {
    L->rng.f = 0;
    L->rng.b = 28;
    L->energy = energy;
    L->accepted += accepted;
    L->rejected += n_steps - accepted;
    L->pairs += pairs;
  }
}

// Union-find over local atom indexes (the partition is all that is used).
int uf_find(std::vector<int>& p, int a) {
  while (p[a] != a) {
    p[a] = p[p[a]];
    a = p[a];
  }
  return a;
}

}  // namespace

IntraHost::~IntraHost() {
  for (void* p : allocs)
    if (p) cudaFree(p);
  if (hout) cudaFreeHost(hout);
}

int intra_upload(mcgpu_ctx* ctx, int n_mol, int n_atom, const int* mol_start, const int* mol_len,
                 const mcgpu_topology_desc* t, std::unique_ptr<IntraHost>* out) {
  if (!t) return set_err(ctx, MCGPU_ERR_INVALID, "null topology");
  const int nb = t->n_bond, na = t->n_angle, nt = t->n_type;
  if (nb < 0 || na < 0 || nt < 0) return set_err(ctx, MCGPU_ERR_INVALID, "negative topology size");
  if ((nb && (!t->bond_a1 || !t->bond_a2 || !t->bond_var || !t->bond_k || !t->bond_eq ||
              !t->bond_len)) ||
      (na && (!t->angle_a1 || !t->angle_a2 || !t->angle_mid || !t->angle_var || !t->angle_k ||
              !t->angle_eq || !t->angle_size)) ||
      !t->mol_bond_start || !t->mol_bond_count || !t->mol_angle_start || !t->mol_angle_count ||
      !t->mol_type || (nt && !t->type_natom))
    return set_err(ctx, MCGPU_ERR_INVALID, "null topology row");
  if (t->max_intra_moves < 0)
    return set_err(ctx, MCGPU_ERR_INVALID, "negative max_intra_moves");
  std::vector<int> t_off(std::max(nt, 1), 0);
  long long codes = 0;
  for (int k = 0; k < nt; k++) {
    if (t->type_natom[k] < 0 || t->type_natom[k] > MCGPU_MAX_MOL_ATOMS)
      return set_err(ctx, MCGPU_ERR_INVALID, "type %d: %d atoms", k, t->type_natom[k]);
    t_off[k] = (int)codes;
    codes += (long long)t->type_natom[k] * t->type_natom[k];
  }
  if (codes && !t->pair_code) return set_err(ctx, MCGPU_ERR_INVALID, "null pair codes");
  auto I = std::make_unique<IntraHost>();
  I->n_bond = nb;
  I->n_angle = na;
  I->n_type = nt;
  I->max_intra_moves = t->max_intra_moves;
  I->max_bond_delta = t->max_bond_delta;
  I->max_angle_delta = t->max_angle_delta;
  I->step = t->step_num;
  I->bstart.assign(t->mol_bond_start, t->mol_bond_start + n_mol);
  I->bcount.assign(t->mol_bond_count, t->mol_bond_count + n_mol);
  I->astart.assign(t->mol_angle_start, t->mol_angle_start + n_mol);
  I->acount.assign(t->mol_angle_count, t->mol_angle_count + n_mol);
  I->bvar.assign(t->bond_var, t->bond_var + nb);
  I->avar.assign(t->angle_var, t->angle_var + na);
  for (int k = 0; k < nb; k++) I->flex_bonds |= t->bond_var[k] != 0;
  for (int k = 0; k < na; k++) I->flex_angles |= t->angle_var[k] != 0;
  // partitions, checked indexes
  std::vector<int> b_part(std::max(nb, 1), -1), a_part(std::max(na, 1), -1);
  std::vector<unsigned char> part;
  std::vector<int> p;
  for (int m = 0; m < n_mol; m++) {
    const int s = mol_start[m], len = mol_len[m];
    const int bs = I->bstart[m], bc = I->bcount[m], as = I->astart[m], ac = I->acount[m];
    if (bs < 0 || bc < 0 || bs + bc > nb || as < 0 || ac < 0 || as + ac > na)
      return set_err(ctx, MCGPU_ERR_INVALID, "molecule %d: bond or angle range outside the rows",
                     m);
    if (t->mol_type[m] < 0 || t->mol_type[m] >= nt)
      return set_err(ctx, MCGPU_ERR_INVALID, "molecule %d: type %d out of [0,%d)", m,
                     t->mol_type[m], nt);
    auto inside = [&](int a) { return a >= s && a < s + len; };
    for (int k = bs; k < bs + bc; k++)
      if (!inside(t->bond_a1[k]) || !inside(t->bond_a2[k]))
        return set_err(ctx, MCGPU_ERR_INVALID, "bond %d: atoms %d-%d outside molecule %d", k,
                       t->bond_a1[k], t->bond_a2[k], m);
    for (int k = as; k < as + ac; k++) {
      if (!inside(t->angle_a1[k]) || !inside(t->angle_a2[k]))
        return set_err(ctx, MCGPU_ERR_INVALID, "angle %d: ends %d, %d outside molecule %d", k,
                       t->angle_a1[k], t->angle_a2[k], m);
      if (t->angle_mid[k] < 0 || t->angle_mid[k] >= n_atom)
        return set_err(ctx, MCGPU_ERR_INVALID, "angle %d: middle atom %d out of [0,%d)", k,
                       t->angle_mid[k], n_atom);
    }
    for (int k = bs; k < bs + bc; k++) {
      p.resize(len);
      for (int i = 0; i < len; i++) p[i] = i;
      for (int o = bs; o < bs + bc; o++) {
        if (o == k) continue;
        int r1 = uf_find(p, t->bond_a1[o] - s), r2 = uf_find(p, t->bond_a2[o] - s);
        if (r1 != r2) p[r1] = r2;
      }
      const int side1 = uf_find(p, t->bond_a1[k] - s), side2 = uf_find(p, t->bond_a2[k] - s);
      if (side1 == side2) continue;
      b_part[k] = (int)part.size();
      for (int i = 0; i < len; i++) part.push_back(uf_find(p, i) == side2 ? 1 : 0);
    }
    for (int k = as; k < as + ac; k++) {
      const int mid = t->angle_mid[k];
      p.resize(len);
      for (int i = 0; i < len; i++) p[i] = i;
      for (int o = bs; o < bs + bc; o++) {
        if (t->bond_a1[o] == mid || t->bond_a2[o] == mid) continue;
        int r1 = uf_find(p, t->bond_a1[o] - s), r2 = uf_find(p, t->bond_a2[o] - s);
        if (r1 != r2) p[r1] = r2;
      }
      const int g1 = uf_find(p, t->angle_a1[k] - s), g2 = uf_find(p, t->angle_a2[k] - s);
      if (g1 == g2) continue;
      a_part[k] = (int)part.size();
      for (int i = 0; i < len; i++) {
        const int g = uf_find(p, i);
        part.push_back(g == g1 ? 1 : (g == g2 ? 2 : 0));
      }
    }
  }
  cudaError_t e = cudaSuccess;
  auto up = [&](auto* src, size_t n) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(src)>>;
    T* d = dalloc<T>(n, &e);
    I->allocs.push_back(d);
    if (e == cudaSuccess && n) e = cudaMemcpy(d, src, n * sizeof(T), cudaMemcpyHostToDevice);
    return d;
  };
  IntraRows& R = I->R;
  R.n_bond = nb;
  R.n_angle = na;
  R.flex_bonds = I->flex_bonds;
  R.flex_angles = I->flex_angles;
  R.b_a1 = up(t->bond_a1, nb);
  R.b_a2 = up(t->bond_a2, nb);
  R.b_var = up(t->bond_var, nb);
  R.b_part = up(b_part.data(), nb);
  R.b_k = up(t->bond_k, nb);
  R.b_eq = up(t->bond_eq, nb);
  R.b_len = up(t->bond_len, nb);
  R.b_len_rb = up(t->bond_len, nb);
  R.a_a1 = up(t->angle_a1, na);
  R.a_a2 = up(t->angle_a2, na);
  R.a_mid = up(t->angle_mid, na);
  R.a_var = up(t->angle_var, na);
  R.a_part = up(a_part.data(), na);
  R.a_k = up(t->angle_k, na);
  R.a_eq = up(t->angle_eq, na);
  R.a_size = up(t->angle_size, na);
  R.a_size_rb = up(t->angle_size, na);
  R.m_bstart = up(t->mol_bond_start, n_mol);
  R.m_bcount = up(t->mol_bond_count, n_mol);
  R.m_astart = up(t->mol_angle_start, n_mol);
  R.m_acount = up(t->mol_angle_count, n_mol);
  R.m_type = up(t->mol_type, n_mol);
  R.t_natom = up(t->type_natom, nt);
  R.t_off = up(t_off.data(), nt);
  R.code = up(t->pair_code, (size_t)codes);
  R.part = up(part.data(), part.size());
  I->dout = dalloc<double>(2, &e);
  I->allocs.push_back(I->dout);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&I->hout, 2 * sizeof(double));
  if (e != cudaSuccess)
    return set_err(ctx, MCGPU_ERR_NOMEM, "topology upload failed: %s", cudaGetErrorString(e));
  *out = std::move(I);
  return MCGPU_OK;
}

cudaError_t launch_intra_energy(const Pool& P, const IntraRows& R, int chain, int mol,
                                double* out, cudaStream_t st) {
  k_intra_energy<<<1, kIntraThreads, 0, st>>>(P, R, chain, mol, out);
  return cudaGetLastError();
}

cudaError_t launch_intra_ops(const Pool& P, const IntraRows& R, int chain, const IntraOps& ops,
                             double* out, cudaStream_t st) {
  k_intra_ops<<<1, kIntraThreads, 0, st>>>(P, R, chain, ops, out);
  return cudaGetLastError();
}

cudaError_t launch_intra_rollback(const Pool& P, const IntraRows& R, int chain, int mol,
                                  cudaStream_t st) {
  k_intra_rollback<<<1, kIntraThreads, 0, st>>>(P, R, chain, mol);
  return cudaGetLastError();
}

cudaError_t launch_plain_steps(bool f64, bool flexible, const LoopTask* tasks, int n_tasks,
                               int n_steps, SmemShape sh, cudaStream_t st) {
  if (n_tasks <= 0) return cudaSuccess;
  // three staged moves in the rigid loop
  const int bytes = flexible ? sh.bytes() : 3 * sh.bytes();
  const int threads = flexible ? kLoopThreads : kRigidThreads;
  const auto kernel = flexible ? (f64 ? k_plain_steps<true> : k_plain_steps<false>)
                               : (f64 ? k_plain_rigid<true> : k_plain_rigid<false>);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  kernel<<<n_tasks, threads, bytes, st>>>(tasks, n_steps, sh);
  return cudaGetLastError();
}

cudaError_t launch_intra_add(const Pool& P, const IntraRows& R, int n_mol, double* emol,
                             cudaStream_t st) {
  if (n_mol <= 0) return cudaSuccess;
  k_intra_add<<<n_mol, 32, 0, st>>>(P, R, emol);
  return cudaGetLastError();
}

cudaError_t launch_intra_add_boxes(const LoopTask* tasks, int n_tasks, int max_mol,
                                   cudaStream_t st) {
  k_intra_add_boxes<<<dim3(max_mol, n_tasks), 32, 0, st>>>(tasks);
  return cudaGetLastError();
}

}  // namespace mcgpu
