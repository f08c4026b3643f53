// kernels.cu -- __global__ kernels of the trial-move energy path.
//
//   k_refresh_mirrors      FP32 mirrors from the FP64 master rows (upload)
//   k_mol_energy<F64>      calcMolecularEnergyContribution over a candidate
//                          range, many CTAs, deterministic last-CTA sum
//   k_move_energies<F64>   old energy + move + new energy in one launch
//   k_change_molecule      the move alone (saves the rollback copy)
//   k_rollback             restores the rollback copy
//   k_pair_sums64          E(m, j>m) of groups of molecules, FP64 pairs
//   k_pair_sums32          E(m, j>m) per molecule, FP32 pairs
//   k_chain_sums           per-chain ordered sum of the above
//   k_box_energies         the same for many boxes, into their loop states
//   k_chain_steps          persistent Metropolis steps of many chains:
//                          Philox proposal, staging, screen, pairs, FP64
//                          dE, decision and commit without leaving the GPU
#include "chain.cuh"
#include "host.h"
#include "intra.h"
#include "pairsum.cuh"

namespace mcgpu {

// ---- mirrors ---------------------------------------------------------------

__global__ void k_refresh_mirrors(Pool P, const int* mol_chain, int m_begin, int m_end) {
  const int m = m_begin + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= m_end) return;
  refresh_molecule(P, P.hdr[mol_chain[m]], m, threadIdx.x & 31, 32);
}

// The FP64 pair terms' per-atom blending factors (blend64).
__global__ void k_blend_rows(Pool P, int n_atom) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < n_atom) P.blend[a] = blend64(P.sig[a], P.eps[a]);
}

// ---- deterministic last-CTA sum ------------------------------------------

// Thread 0 of a CTA: publishes its writes and reports whether this CTA is
// the last of the grid to arrive (it then owns the ordered final sum).
__device__ bool arrive_last(unsigned* counter) {
  __threadfence();
  unsigned t = atomicAdd(counter, 1u);
  return t == gridDim.x - 1;
}

// ---- plain contract ---------------------------------------------------------

// Publishes a plain kernel's results to the host: `out` and `done` lie in pinned
// host memory, and the host polls `done` for the call's number.
__device__ __forceinline__ void host_done(unsigned* done, unsigned call) {
  if (done) {
    __threadfence_system();
    *(volatile unsigned*)done = call;
  }
}

// Sum of the grid's partials p[0], p[stride], ... by one warp, every lane: lane
// l adds every 32nd, then a butterfly (one after another by one thread, each an
// L2 round trip, they took 22 of the 39 us of a 32-CTA launch).
__device__ __forceinline__ double sum_partials(const double* p, int stride, int lane) {
  double v = 0.0;
  for (unsigned b = lane; b < gridDim.x; b += 32) v += __ldcg(p + (size_t)b * stride);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(~0u, v, off);
  return v;
}

// Energy of molecule `curr` against chain-local candidates [start, n_mol)
// (BruteForceCalcs::calcMolecularEnergyContribution, BruteForceStep.cpp:
// 15-46).  The candidates are dealt over the warps of the grid.
template <bool F64>
__global__ void __launch_bounds__(F64 ? 256 : kPlainThreads, F64 ? 0 : 1)
    k_mol_energy(Pool P, int chain, int curr, int start, SmemShape shape, double* partials,
                 unsigned* counter, double* out, long long* pairs, unsigned* done, unsigned call) {
  extern __shared__ __align__(16) char smem[];
  const ChainHdr& H = P.hdr[chain];
  Group g{(int)threadIdx.x, (int)blockDim.x, 1};
  GroupSmem s = shape.carve(smem);
  const int lane = threadIdx.x & 31, w = g.warp(), nw = g.nwarps();
  const int m = H.mol0 + curr;
  if (w == 0) stage(P, H, m, nullptr, s, lane);
  g.sync();
  const MovedInfo mi = load_moved(s);
  double eo = 0.0, en = 0.0;
  long long np = 0;
  warp_eval<F64, true>(P, H, s, mi, H.mol0 + start, H.mol0 + H.n_mol, (int)blockIdx.x * nw + w,
                 (int)gridDim.x * nw, s.lj + w * kRing, lane, eo, en, np);
  group_reduce(g, s, eo, en, np);
  __shared__ int last;
  if (threadIdx.x == 0) {
    if (pairs) atomicAdd((unsigned long long*)pairs, (unsigned long long)np);
    partials[blockIdx.x] = eo;
    last = arrive_last(counter) ? 1 : 0;
  }
  __syncthreads();
  if (!last || w != 0) return;
  __threadfence();
  const double sum = sum_partials(partials, 1, lane);
  if (lane == 0) {
    out[0] = sum;
    *counter = 0;
    host_done(done, call);
  }
}

// Old energy, the move, and new energy of molecule `mol` in one launch
// (Simulation.cpp:244-250).  Every CTA stages the same proposed placement;
// the CTA that finishes last saves the rollback copy and commits.
template <bool F64>
__global__ void __launch_bounds__(F64 ? 256 : kPlainThreads, F64 ? 0 : 1)
    k_move_energies(Pool P, int chain, int mol, Proposal prop, SmemShape shape, double* partials,
                    unsigned* counter, double* out, long long* pairs, unsigned* done,
                    unsigned call) {
  extern __shared__ __align__(16) char smem[];
  const ChainHdr& H = P.hdr[chain];
  Group g{(int)threadIdx.x, (int)blockDim.x, 1};
  GroupSmem s = shape.carve(smem);
  const int lane = threadIdx.x & 31, w = g.warp(), nw = g.nwarps();
  const int m = H.mol0 + mol;
  if (w == 0) stage(P, H, m, &prop, s, lane);
  g.sync();
  const MovedInfo mi = load_moved(s);
  double eo = 0.0, en = 0.0;
  long long np = 0;
  warp_eval<F64, true>(P, H, s, mi, H.mol0, H.mol0 + H.n_mol, (int)blockIdx.x * nw + w,
                 (int)gridDim.x * nw, s.lj + w * kRing, lane, eo, en, np);
  group_reduce(g, s, eo, en, np);
  __shared__ int last;
  if (threadIdx.x == 0) {
    if (pairs) atomicAdd((unsigned long long*)pairs, (unsigned long long)np);
    partials[2 * blockIdx.x] = eo;
    partials[2 * blockIdx.x + 1] = en;
    last = arrive_last(counter) ? 1 : 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (w == 0) {
    double* rb = P.rb + (size_t)chain * 3 * H.max_len;
    for (int i = lane; i < mi.len; i += 32) {
      rb[i] = s.ox[i];
      rb[H.max_len + i] = s.oy[i];
      rb[2 * H.max_len + i] = s.oz[i];
    }
    commit(P, s, mi, lane);
    const double so = sum_partials(partials, 2, lane), sn = sum_partials(partials + 1, 2, lane);
    if (lane == 0) {
      out[0] = so;
      out[1] = sn;
      *counter = 0;
      host_done(done, call);
    }
  }
}

// The move alone (SimCalcs::intermolecularMove with supplied draws).
__global__ void k_change_molecule(Pool P, int chain, int mol, Proposal prop, SmemShape shape) {
  extern __shared__ __align__(16) char smem[];
  const ChainHdr& H = P.hdr[chain];
  GroupSmem s = shape.carve(smem);
  const int lane = threadIdx.x & 31;
  stage(P, H, H.mol0 + mol, &prop, s, lane);
  __syncwarp();
  const MovedInfo mi = load_moved(s);
  double* rb = P.rb + (size_t)chain * 3 * H.max_len;
  for (int i = lane; i < mi.len; i += 32) {
    rb[i] = s.ox[i];
    rb[H.max_len + i] = s.oy[i];
    rb[2 * H.max_len + i] = s.oz[i];
  }
  commit(P, s, mi, lane);
}

// SimCalcs::rollback (SimulationStep.cpp:731-749) plus the mirrors.
__global__ void k_rollback(Pool P, int chain, int mol) {
  const ChainHdr& H = P.hdr[chain];
  const int m = H.mol0 + mol;
  const int a0 = P.mstart[m], len = P.mlen[m] & 255;
  const double* rb = P.rb + (size_t)chain * 3 * H.max_len;
  const int lane = threadIdx.x & 31;
  for (int i = lane; i < len; i += 32) {
    P.x[a0 + i] = rb[i];
    P.y[a0 + i] = rb[H.max_len + i];
    P.z[a0 + i] = rb[2 * H.max_len + i];
  }
  __syncwarp();
  refresh_molecule(P, H, m, lane, 32);
}

// The pool of a launch: P0, or with tasks that of box blockIdx.y, copied to
// shared memory by the whole block.
__device__ __forceinline__ void load_pool(Pool& SP, const Pool& P0, const LoopTask* tasks) {
  static_assert(sizeof(Pool) % 4 == 0, "Pool words");
  if (tasks) {
    const int* src = (const int*)&tasks[blockIdx.y].P;
    for (int i = threadIdx.x; i < (int)(sizeof(Pool) / 4); i += blockDim.x) ((int*)&SP)[i] = src[i];
  } else if (threadIdx.x == 0) {
    SP = P0;
  }
  __syncthreads();
}

// The pool's rows as ps_items reads them.
struct PoolRows {
  const Pool& P;
  __device__ __forceinline__ int len(int j) const { return P.mlen[j] & 255; }
  __device__ __forceinline__ int start(int j) const { return P.mstart[j]; }
  __device__ __forceinline__ void atom(int b, double& x, double& y, double& z, double& sb,
                                       double& eb, double& qb) const {
    x = P.x[b];
    y = P.y[b];
    z = P.z[b];
    const double2 bl = P.blend ? P.blend[b] : blend64(P.sig[b], P.eps[b]);
    sb = bl.x;
    eb = bl.y;
    qb = P.q[b];
  }
};

// E(m, j > m) of SimulationStep::calcSystemEnergy (SimulationStep.cpp:47-48)
// with FP64 pairs, groups of ps_group consecutive molecules of a chain:
// emol[first molecule] holds the sum over the group's molecules, the others 0.
// A CTA takes the groups that start among its `span` molecules (at most the
// smallest chain's group, so that a CTA has one to take or, in a larger chain,
// none).  The in-range set is the
// FP64 test's (the FP32 screen decides outside its guard band).  32,768
// waters (rc 12 A, 35.6 M pairs): 1.84 ms, bound by the issue of the N^2 / 2
// screen beside the FP64 pipe (58 % busy); 5.84 ms with a CTA per molecule.
__global__ void __launch_bounds__(kPsThreads, 4)
    k_pair_sums64(Pool P0, const LoopTask* tasks, const int* mol_chain, int n_mol, int span, int per,
                  double* emol) {
  __shared__ Pool SP;
  __shared__ PsGroup G;
  __shared__ float4 pp[kPsGroup][kMaxP];
  __shared__ int pslot[kPsGroup][kMaxP], pnum[kPsGroup];
  load_pool(SP, P0, tasks);
  const Pool& P = SP;
  if (tasks) {
    n_mol = tasks[blockIdx.y].n_mol;
    span = ps_group(n_mol, per);
    emol = tasks[blockIdx.y].emol;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  int m0 = (int)blockIdx.x * span;
  const int mg = min(m0 + span, n_mol);
  while (m0 < mg) {
    const int c = tasks ? 0 : mol_chain[m0];
    const ChainHdr& H = P.hdr[c];
    const int group = ps_group(H.n_mol, per), off = (m0 - H.mol0) % group;
    const int m1 = min(m0 - off + group, H.mol0 + H.n_mol), n = m1 - m0;
    if (off > 0) {   // inside a group that starts before this CTA's molecules
      m0 = m1;
      continue;
    }
    for (int g = 0; g < n; g++) {
      const int m = m0 + g, a0 = P.mstart[m], len = P.mlen[m] & 255;
      const int2 pi = P.mpi[m];
      for (int i = threadIdx.x; i < len; i += kPsThreads) {
        const int o = g * kPsPitch + i;
        PoolRows{P}.atom(a0 + i, G.x[o], G.y[o], G.z[o], G.sd[o], G.ed[o], G.qd[o]);
      }
      for (int k = threadIdx.x; k < pi.y; k += kPsThreads) {
        pp[g][k] = P.ppos[pi.x + k];
        pslot[g][k] = g * kPsPitch + P.pidx[pi.x + k] - a0;
      }
      if (threadIdx.x == 0) {
        G.len[g] = len;
        pnum[g] = pi.y;
      }
    }
    __syncthreads();
    const bool alike = ps_alike(G, n);
    int* rj = G.ring[w];
    int head = 0, tail = 0;
    double acc = 0.0;
    const int end = H.mol0 + H.n_mol;
    const bool simple = H.simple_prim != 0;
    // the screen's constants in registers (the header is global memory, and
    // the ring's stores would have it read again for every test)
    const float Lx = H.Lf[0], Ly = H.Lf[1], Lz = H.Lf[2], lo = H.cut2_lo, hi = H.cut2_hi;
    for (int base = m0 + 1 + w * 32; base < end; base += kPsThreads) {
      const int j = base + lane;
      int2 pj = make_int2(0, 0);
      float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < end) {
        pj = simple ? make_int2(H.pidx0 + (j - H.mol0), 1) : P.mpi[j];
        q0 = P.ppos[pj.x];
      }
      for (int g = 0; g < n; g++) {
        bool in = false;
        if (simple) {
          // one primary each: a straight line (r2_screen's arithmetic)
          const float4 a = pp[g][0];
          const float dx = wrapf(q0.x - a.x, Lx), dy = wrapf(q0.y - a.y, Ly),
                      dz = wrapf(q0.z - a.z, Lz);
          const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
          const bool mine = j > m0 + g && j < end;
          in = mine && r2 <= lo;
          if (mine && !in && r2 <= hi) {
            const int o = pslot[g][0];
            in = in_range64(G.x[o], G.y[o], G.z[o], P.pidx[pj.x], P, H);
          }
        } else if (j > m0 + g)
          for (int k2 = 0; k2 < pj.y && !in; k2++) {
            const float4 q = k2 == 0 ? q0 : P.ppos[pj.x + k2];
            for (int k1 = 0; k1 < pnum[g] && !in; k1++) {
              const float r2 = r2_screen(pp[g][k1], q, H);
              if (r2 <= H.cut2_lo) {
                in = true;
              } else if (r2 <= H.cut2_hi) {
                const int o = pslot[g][k1];
                in = in_range64(G.x[o], G.y[o], G.z[o], P.pidx[pj.x + k2], P, H);
              }
            }
          }
        const unsigned bal = __ballot_sync(~0u, in);
        if (bal == 0) continue;
        if (in) rj[(tail + __popc(bal & lt)) & (kRing - 1)] = (j << 3) | g;
        tail += __popc(bal);
        if (tail - head >= 32) {
          __syncwarp();
          acc += ps_items<false>(G, PoolRows{P}, rj, head, 32, lane, alike, H.L[0], H.L[1], H.L[2]);
          head += 32;
          __syncwarp();
        }
      }
    }
    __syncwarp();
    if (tail > head)
      acc += ps_items<false>(G, PoolRows{P}, rj, head, tail - head, lane, alike, H.L[0], H.L[1],
                            H.L[2]);
    const double sum = ps_block_sum(G, acc);
    if ((int)threadIdx.x < n) emol[m0 + threadIdx.x] = threadIdx.x == 0 ? sum : 0.0;
    m0 = m1;
    __syncthreads();   // the next chain's molecules overwrite the stage
  }
}

// The same with FP32 pairs, one molecule m = m_begin + blockIdx.x per CTA.
__global__ void __launch_bounds__(kPlainThreads, 1)
    k_pair_sums32(Pool P0, const LoopTask* tasks, const int* mol_chain, int m_begin,
                  SmemShape shape, double* emol) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Pool SP;
  load_pool(SP, P0, tasks);
  const Pool& P = SP;
  const int m = m_begin + blockIdx.x;
  if (tasks) {
    if (m >= tasks[blockIdx.y].n_mol) return;
    emol = tasks[blockIdx.y].emol;
  }
  const ChainHdr& H = P.hdr[tasks ? 0 : mol_chain[m]];
  Group g{(int)threadIdx.x, (int)blockDim.x, 1};
  GroupSmem s = shape.carve(smem);
  const int lane = threadIdx.x & 31, w = g.warp(), nw = g.nwarps();
  if (w == 0) stage(P, H, m, nullptr, s, lane);
  g.sync();
  const MovedInfo mi = load_moved(s);
  double eo = 0.0, en = 0.0;
  long long np = 0;
  warp_eval<false, false>(P, H, s, mi, m + 1, H.mol0 + H.n_mol, w, nw, s.lj + w * kRing, lane, eo, en,
                   np);
  group_reduce(g, s, eo, en, np);
  if (threadIdx.x == 0) emol[m] = eo;
}

// Ordered sum of n terms: thread t adds every blockDim-th term from t, then
// a fixed tree; the total in thread 0 (one CTA of at most 256 threads).
__device__ __forceinline__ double ordered_sum(const double* v, int n, double* red) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += v[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int off = blockDim.x >> 1; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  return red[0];
}

// Ordered per-chain sum of emol; one CTA per chain.
__global__ void k_chain_sums(Pool P, const double* emol, double* out) {
  __shared__ double red[256];
  const ChainHdr& H = P.hdr[blockIdx.x];
  const double e = ordered_sum(emol + H.mol0, H.n_mol, red);
  if (threadIdx.x == 0) out[blockIdx.x] = e;
}

// The boxes' system energies from their emol rows, as the start of their
// loops; one CTA per box.
__global__ void k_box_energies(const LoopTask* tasks) {
  __shared__ double red[256];
  const LoopTask& T = tasks[blockIdx.x];
  const double e = ordered_sum(T.emol, T.n_mol, red);
  if (threadIdx.x == 0) {
    T.L->energy = e;
    T.L->energy0 = e;
  }
}

// Sets every chain's running energy from out[] (the start of a run).
__global__ void k_set_energy(Pool P, const double* e) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < P.n_chains) P.hdr[c].energy = e[c];
}

// ---- device-resident Metropolis -------------------------------------------

// Puts every molecule of the pool in the device-resident chain state:
// anchor = its first primary atom in fixed point, offsets = FP32 (atom -
// anchor), template = offsets, quaternion = identity; then snaps the FP64
// rows to that state (x = anchor + offset, each moved by < 1e-7 A) so both
// descriptions agree exactly.  One warp per molecule.
__global__ void k_chain_init(Pool P, const int* mol_chain, int m_begin, int m_end) {
  const int m = m_begin + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= m_end) return;
  const ChainHdr& H = P.hdr[mol_chain[m]];
  const int lane = threadIdx.x & 31;
  const int a0 = P.mstart[m], len = P.mlen[m] & 255;
  const int2 pi = P.mpi[m];
  const int an = P.pidx[pi.x];
  const double ax = P.x[an], ay = P.y[an], az = P.z[an];
  const uint4 A = fixpos(ax, ay, az, H);
  __syncwarp();
  for (int i = lane; i < len; i += 32) {
    const int a = a0 + i;
    const float w = P.aoff[a].w;
    const float4 o = make_float4((float)(P.x[a] - ax), (float)(P.y[a] - ay), (float)(P.z[a] - az), w);
    P.aoff[a] = o;
    P.aofl[a] = make_float4(0.f, 0.f, 0.f, 0.f);
    P.atpl[a] = make_float4(o.x, o.y, o.z, 0.f);
  }
  __syncwarp();
  for (int i = lane; i < len; i += 32) {
    const int a = a0 + i;
    const double3 x = chain_pos3(A, P.aoff[a], H);
    P.x[a] = x.x;
    P.y[a] = x.y;
    P.z[a] = x.z;
  }
  __syncwarp();
  for (int k = lane; k < pi.y; k += 32) {
    const int q = P.pidx[pi.x + k];
    P.ppos[pi.x + k] = wrap_pos(P.x[q], P.y[q], P.z[q], H);
  }
  if (lane == 0) {
    P.mfix[m] = A;
    P.mq[m] = make_float4(1.f, 0.f, 0.f, 0.f);
  }
}

// FP64 rows of every atom from the chain state (for downloads, FP64
// recomputes and the plain entry points).  One thread per atom.
__global__ void k_chain_export(Pool P, const int* mol_chain, const int* atom_mol, int a_begin,
                               int a_end) {
  const int a = a_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= a_end) return;
  const int m = atom_mol[a];
  const ChainHdr& H = P.hdr[mol_chain[m]];
  const double3 x = chain_pos3(P.mfix[m], P.aoff[a], H);
  P.x[a] = x.x;
  P.y[a] = x.y;
  P.z[a] = x.z;
}

// The chain task with the most work left: warp 0 of a group looks through
// sched (entry k: steps task k has taken, kChainBusy while a group runs it)
// for the free task of the largest remaining steps x cost and claims it; -1
// when every task is finished or running (each running task's group takes the
// next one itself, so this group is not needed any more).  sizes: the tasks'
// molecule counts, in one row so that a look through 512 tasks is 16
// coalesced loads (from the chain headers it took 12 us).  Each group sees the
// costs a few per cent apart from what the others see, or groups that look at
// the same time would all reach for the same task.
constexpr unsigned kChainBusy = 0x80000000u;

__device__ __forceinline__ int claim_chain(const int* sizes, unsigned* sched, int n_tasks,
                                           int n_steps, int group, bool start, int lane,
                                           int* done) {
  // at the start of a launch group k takes task k, so that the groups do not
  // all reach for the same one
  if (start && group < n_tasks) {
    int won = 0;
    if (lane == 0) won = atomicCAS(sched + group, 0u, kChainBusy) == 0u;
    if (__shfl_sync(~0u, won, 0)) {
      *done = 0;
      return group;
    }
  }
  for (;;) {
    float best = 0.f;
    int at = -1;
    unsigned seen = 0;
    for (int k = lane; k < n_tasks; k += 32) {
      const unsigned v = *(volatile unsigned*)(sched + k);
      if ((v & kChainBusy) || (int)v >= n_steps) continue;
      // a step costs a fixed latency and its screen: about 4,096 molecules' worth
      const unsigned mix = ((unsigned)k * 2654435761u) ^ ((unsigned)group * 2246822519u);
      const float key = (float)(n_steps - (int)v) * (float)(4096 + sizes[k]) *
                        (1.f + 1.4e-11f * (float)mix);
      if (key > best) {
        best = key;
        at = k;
        seen = v;
      }
    }
    float top = best;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(~0u, top, off));
    if (top == 0.f) return -1;
    const int src = __ffs(__ballot_sync(~0u, best == top)) - 1;
    int won = 0;
    if (lane == src) won = atomicCAS(sched + at, seen, seen | kChainBusy) == seen;
    if (__shfl_sync(~0u, won, src)) {
      __threadfence();   // the rows the last group to run the task wrote
      *done = (int)__shfl_sync(~0u, seen, src);
      return __shfl_sync(~0u, at, src);
    }
  }
}

// Persistent kernel: groups of `gwarps` warps take chain tasks (task k runs
// chain order[k]) for `seg` steps at a time, the one with the most work left
// first (or, in_order, the next one for all its steps), until each has taken
// n_steps; sched: n_tasks zeroed words.  With a
// task per group for all its steps, 512 chains of uneven size on 456 groups
// left the chip half idle in a second wave of 56 (SMs busy 77 % of a launch).
// A task stays on one group at a time, and its steps on the
// chain state.  A step: every warp screens its share of the candidates
// against the move staged in FP32 during the previous step and evaluates
// the in-range ones (FP32 pair terms, double-float sums); the last warp then
// stages the next move into the next of three shared-memory slots; one
// group reduction (the step's barrier) gives every thread E_old, E_new.
// Outside a guard band around the acceptance threshold the decision
// (dE < 0, else exp(-dE/kT) >= u, SimulationStep.cpp:794-803) is taken in
// FP32; inside it the group re-evaluates both placements with FP64 pairs and
// decides on that.  Every warp takes the decision and writes the accepted
// placement itself and goes on to the next step; warp 0 keeps the running
// energy and the counters.  With cache_n > 0 each group keeps its chain's
// primary screen positions in shared memory.  If trace != nullptr, step st
// of chain c is recorded at trace[c * trace_stride + trace_off + st].  The
// staging warp draws the moves of 32 steps at once (one per lane) into
// shared memory; when a commit moves the molecule of the move staged next,
// warp 0 stages it again (one more barrier).  lanes_cap > 0 caps the lanes
// per neighbour molecule of every chain.
__device__ __forceinline__ void chain_steps(Pool P, const ChainLaunch& A, char* smem) {
  const int n_steps = A.n_steps, seg = A.seg, n_tasks = A.n_tasks, gwarps = A.gwarps;
  const SmemShape shape = A.shape;
  mcgpu_trace* trace = A.trace;
  const int gsize = gwarps * 32;
  const int gid = threadIdx.x / gsize;
  Group g{(int)threadIdx.x - gid * gsize, gsize, 1 + gid};
  GroupSmem s = shape.carve(smem + gid * shape.bytes());
  const int lane = threadIdx.x & 31, w = g.warp(), nw = g.nwarps();
  const int group = blockIdx.x * ((int)blockDim.x / gsize) + gid;
  bool start = true;
  int task = -1, base = 0;
  for (;;) {
    if (A.in_order && task >= 0 && base + seg < n_steps) {
      base += seg;
    } else {
      if (w == 0) {
        int taken = 0, t = -1;
        if (A.in_order) {
          // sched's first word counts the tasks taken
          if (lane == 0) t = (int)atomicAdd(A.sched, 1u);
          t = __shfl_sync(~0u, t, 0);
          if (t >= n_tasks) t = -1;
        } else {
          t = claim_chain(A.sizes, A.sched, n_tasks, n_steps, group, start, lane, &taken);
          start = false;
        }
        if (lane == 0) {
          s.misc[31] = t;
          s.misc[30] = taken;
        }
      }
      g.sync();
      task = s.misc[31];
      base = s.misc[30];
      if (task < 0) break;
    }
    const int c = A.order[task];
    ChainHdr* Hp = P.hdr + c;
    const ChainHdr& H = *Hp;
    float4* pcache = (s.pc && H.simple_prim && H.n_mol <= shape.cache_n) ? s.pc : nullptr;
    if (pcache)
      for (int i = g.tid; i < H.n_mol; i += gsize) pcache[i] = P.ppos[H.pidx0 + i];
    if (H.uniform)
      for (int i = g.tid; i < H.ulen; i += gsize) s.teq[i] = P.aeq[H.atom0 + i];
    g.sync();
    // the chain's LJ mask, read by the pair batches after the next barrier
    // (kept in the header rather than in a register across the step loop)
    if (g.tid == 0) Hp->ljmask = uniform_lj_mask(P, H, s.teq);
    int full_scans = 0;
    // the accepted dE of this task and their FP32 error bounds, each summed
    // in double-float (FP64 costs 64 FP32 issue slots on GB300); both join
    // the FP64 header values once, at the task's end
    float de_h = 0.f, de_l = 0.f, err_h = 0.f, err_l = 0.f;
    long long acc_n = 0, npairs = 0;
    int ties = 0;
    const unsigned long long step0 = H.step;
    // the Verlet list stays valid while no accepted molecule has moved beyond
    // skin/2 of the build (every thread keeps the same flag)
    bool nl_ok = H.nl_on && H.nl_valid;
    // lanes per neighbour molecule: the cap, else one lane for a chain of
    // one species of at most 4 atoms (the single-lane pair batch), else the
    // power of two at or above its largest molecule
    const int T = A.lanes_cap > 0 ? min(A.lanes_cap, H.tpm)
                                : ((H.uniform && H.ulen <= 4 && !H.precise) ? 1 : H.tpm);
    MoveF* props = (MoveF*)s.props;
    int my_steps = min(seg, n_steps - base);
    if (H.step_limit > 0)
      my_steps = (int)max(0LL, min((long long)my_steps, H.step_limit - (long long)step0));
    // step st's move is staged in slot st % 3 (the last warp stages step
    // st + 1 during step st; slot (st + 2) % 3 = (st - 1) % 3 is rewritten
    // only after every warp has passed step st's reduction barrier, so no
    // warp still commits from it)
    const int sb = shape.ahead_bytes();
    auto slot = [&](int k) { return shape.ahead_slot(s.ahead + k * sb); };
    // moves are drawn 32 steps at a time (one per lane) by the staging warp
    auto draw32 = [&](int st0) {
      if (st0 + lane < my_steps)
        props[lane] = draw_move_f32(H.seed, H.chain_id, step0 + st0 + lane, H.n_mol,
                                    P.mlen + H.mol0, (float)H.max_t, (float)H.max_r, H.rot_mode);
      __syncwarp();
    };
    // the last warp stages the next move while the others take the items (it
    // takes its share of them in groups of fewer than four warps)
    const int workers = nw >= 4 ? nw - 1 : nw;
    if (w == 0 && my_steps > 0) {
      draw32(0);
      stage_chain(P, H, props[0], slot(0), pcache, lane);
    }
    g.sync();
    for (int st = 0; st < my_steps; st++) {
      const int k = st % 3, kn = k == 2 ? 0 : k + 1;
      const GroupSmem ss = with_slot(s, slot(k));
      const MovedInfo mi = load_moved(ss);
      const float u = __int_as_float(ss.misc[kMiscU]);
      // Verlet list while it is valid and the trial placement stays within
      // skin/2 of the build; the full scan otherwise (same in-range set)
      const int trial_near = ss.misc[kMiscNlTrial];
      const bool use_list = nl_ok && trial_near;
      AccFF acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0};
      // FP64-pair chains skip the FP32 evaluation: every step is taken by
      // the FP64 path below
      const bool f64all = H.fp64_pairs != 0;
      if (f64all) {
      } else if (use_list)
        group_eval_chain(P, H, g, ss, mi, pcache, 0, P.nl_cnt[mi.mol], workers, T, acc,
                        P.nl + (size_t)mi.mol * P.nl_stride);
      else
        group_eval_chain(P, H, g, ss, mi, pcache, H.mol0, H.mol0 + H.n_mol, workers, T, acc);
      // the last warp (with the fewest screen blocks) stages the next move
      // while the others finish their share
      if (w == nw - 1 && st + 1 < my_steps) {
        if (((st + 1) & 31) == 0) draw32(st + 1);
        stage_chain(P, H, props[(st + 1) & 31], slot(kn), pcache, lane);
      }
      // the step's one barrier; every thread ends with the same totals
      group_reduce_ff(g, ss, acc, st & 1);
      // FP32 decision unless the FP32 dE is within its rounding bound of the
      // threshold; the bound covers the pair terms' rounding (kTieRel of the
      // sum of magnitudes) and the FP32 difference of the two totals.
      const float de_f = __fadd_rn(__fsub_rn(acc.nh, acc.oh), __fsub_rn(acc.nl, acc.ol));
      const float bound = (float)kTieRel * acc.ab + 2.4e-7f * (fabsf(acc.nh) + fabsf(acc.oh)) + 1e-9f;
      const float pf = expf(-fmaxf(de_f, 0.f) * H.kTinvf);
      const int tie = f64all ||
                      ((de_f >= -bound) && (fabsf(pf - u) <= pf * (1.5f * bound * H.kTinvf) + 1e-6f));
      double e_old = 0.0, e_new = 0.0;
      int ok;
      if (tie) {
        if (w == 0) stage_chain_f64(P, H, ss, mi, lane);
        g.sync();
        double eo = 0.0, en = 0.0;
        long long np2 = 0;
        if (use_list)
          warp_eval_chain64(P, H, ss, mi, pcache, 0, P.nl_cnt[mi.mol], w, nw, lane, eo, en, np2,
                            P.nl + (size_t)mi.mol * P.nl_stride);
        else
          warp_eval_chain64(P, H, ss, mi, pcache, H.mol0, H.mol0 + H.n_mol, w, nw, lane, eo,
                            en, np2);
        group_reduce(g, ss, eo, en, np2, st & 1);
        e_old = eo;
        e_new = en;
        if (f64all) acc.np = np2;   // (a re-take's pairs are counted already)
        const double d64 = e_new - e_old;
        ok = (d64 < 0) || (exp(-d64 / H.kT) >= (double)u);
      } else {
        ok = (de_f < 0.f) || (pf >= u);
      }
      // every warp takes the same decision and writes the same new placement,
      // so each sees it in its next screen without waiting for the others
      if (ok) commit_chain(P, H, ss, mi, pcache, lane);
      __syncwarp();
      if (ok && !trial_near) nl_ok = false;
      if (w == 0 && lane == 0) {
        if (ok) {
          if (tie) {
            const double d64 = e_new - e_old;
            const float dh = (float)d64;
            ff_add2(de_h, de_l, dh, (float)(d64 - (double)dh));
            ff_add(err_h, err_l, 1e-12f * acc.ab);
          } else {
            ff_add2(de_h, de_l, acc.nh, acc.nl);
            ff_add2(de_h, de_l, -acc.oh, -acc.ol);
            ff_add(err_h, err_l, bound);
          }
          acc_n++;
        }
        if (H.nl_on && !use_list) full_scans++;
        npairs += acc.np;
        ties += tie;
        if (trace) {
          if (!tie) {
            e_old = (double)acc.oh + (double)acc.ol;
            e_new = (double)acc.nh + (double)acc.nl;
          }
          const double de = e_new - e_old;
          mcgpu_trace t;
          t.mol = mi.mol - H.mol0;
          t.accepted = ok;
          t.e_old = e_old;
          t.e_new = e_new;
          t.de = de;
          t.u = (double)u;
          t.fp64 = tie;
          t.pad0 = 0;
          trace[(size_t)c * A.trace_stride + A.trace_off + base + st] = t;
        }
      }
      // the next move was staged from rows this commit changes only if it
      // moves the same molecule (read from its slot: the staging warp may
      // already be drawing over props): warp 0 stages it again, all warps
      // wait (the condition is the same in every thread)
      if (st + 1 < my_steps && ok && slot(kn).misc[0] == mi.mol) {
        if (w == 0) stage_chain(P, H, props[(st + 1) & 31], slot(kn), pcache, lane);
        g.sync();
      }
    }
    if (g.tid == 0) {
      Hp->energy = H.energy + ((double)de_h + (double)de_l);
      Hp->run_err += (double)err_h + (double)err_l;
      Hp->step = step0 + my_steps;
      Hp->accepted += acc_n;
      Hp->pairs += npairs;
      Hp->ties += ties;
      if (H.nl_on) {
        Hp->nl_valid = nl_ok ? 1 : 0;
        Hp->nl_full += full_scans;
      }
    }
    g.sync();
    // give the task back: every thread's writes, then the steps taken
    if (!A.in_order && g.tid == 0) {
      __threadfence();
      atomicExch(A.sched + task, (unsigned)min(base + seg, n_steps));
    }
  }
}

__global__ void __launch_bounds__(256, 2) k_chain_steps(Pool P, ChainLaunch A) {
  extern __shared__ __align__(16) char smem[];
  chain_steps(P, A, smem);
}

// The same for one group of up to 16 warps per CTA (a single large chain:
// more warps per step, one CTA per SM).
__global__ void __launch_bounds__(512, 1) k_chain_steps_wide(Pool P, ChainLaunch A) {
  extern __shared__ __align__(16) char smem[];
  chain_steps(P, A, smem);
}

// ---- host launchers (template kernels are instantiated here) --------------

cudaError_t launch_mol_energy(bool f64, int grid, SmemShape sh, cudaStream_t st,
                              Pool P, int chain, int curr, int start, double* partials,
                              unsigned* counter, double* out, long long* pairs, unsigned* done,
                              unsigned call) {
  if (f64)
    k_mol_energy<true><<<grid, kPlainThreads, sh.bytes(), st>>>(P, chain, curr, start, sh, partials,
                                                          counter, out, pairs, done, call);
  else
    k_mol_energy<false><<<grid, kPlainThreads, sh.bytes(), st>>>(P, chain, curr, start, sh, partials,
                                                           counter, out, pairs, done, call);
  return cudaGetLastError();
}

cudaError_t launch_move_energies(bool f64, int grid, SmemShape sh, cudaStream_t st,
                                 Pool P, int chain, int mol, Proposal prop, double* partials,
                                 unsigned* counter, double* out, long long* pairs, unsigned* done,
                                 unsigned call) {
  if (f64)
    k_move_energies<true><<<grid, kPlainThreads, sh.bytes(), st>>>(P, chain, mol, prop, sh, partials,
                                                             counter, out, pairs, done, call);
  else
    k_move_energies<false><<<grid, kPlainThreads, sh.bytes(), st>>>(P, chain, mol, prop, sh, partials,
                                                              counter, out, pairs, done, call);
  return cudaGetLastError();
}

int pair_sum_groups(int n_mol) {
  const int group = ps_group(n_mol, kPsPerBox);
  return (n_mol + group - 1) / group;
}

cudaError_t launch_mol_pair_sums(bool f64, int n_mol, int min_chain, bool batch, SmemShape sh,
                                 cudaStream_t st, const Pool& P, const int* mol_chain,
                                 double* emol) {
  if (f64) {
    const int per = batch ? kPsPerBatch : kPsPerBox, span = ps_group(min_chain, per);
    k_pair_sums64<<<(n_mol + span - 1) / span, kPsThreads, 0, st>>>(P, nullptr, mol_chain, n_mol,
                                                                    span, per, emol);
  } else {
    k_pair_sums32<<<n_mol, kPlainThreads, sh.bytes(), st>>>(P, nullptr, mol_chain, 0, sh, emol);
  }
  return cudaGetLastError();
}

cudaError_t launch_box_energies(bool f64, const LoopTask* tasks, int n_tasks, int max_mol,
                                int max_groups, bool intra, SmemShape sh, cudaStream_t st) {
  // grid.y holds at most 65,535 boxes
  for (int t0 = 0; t0 < n_tasks; t0 += 65535) {
    const int nt = n_tasks - t0 < 65535 ? n_tasks - t0 : 65535;
    const LoopTask* T = tasks + t0;
    if (f64) {
      k_pair_sums64<<<dim3(max_groups, nt), kPsThreads, 0, st>>>(Pool{}, T, nullptr, 0, 0,
                                                                 kPsPerBox, nullptr);
    } else {
      k_pair_sums32<<<dim3(max_mol, nt), kPlainThreads, sh.bytes(), st>>>(Pool{}, T, nullptr, 0,
                                                                           sh, nullptr);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && intra) e = launch_intra_add_boxes(T, nt, max_mol, st);
    if (e != cudaSuccess) return e;
    k_box_energies<<<nt, 256, 0, st>>>(T);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace mcgpu
