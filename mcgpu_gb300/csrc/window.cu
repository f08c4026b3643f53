// window.cu -- one chain advanced in windows of K consecutive steps by a
// thread-block cluster of K CTAs (K = 2, 4, 8 or 16), one step of each
// window per CTA.
//
// The reference's loop (Simulation.cpp:219-264) is sequential: step s + 1
// sees the state step s left.  Its moves here come from counter-based draws
// (step index -> move), so the K moves of a window are known before any of
// them is decided.  Every CTA stages all K moves; CTA r evaluates step
// s0 + r against the state at the window's start (FP32 pair terms, the FP64
// re-take inside the guard band -- the one-group kernel's step) and stores
// what it found in every CTA's shared memory (distributed shared memory).
// Every CTA then takes the decisions in step order.  Step j's result stands
// unless an earlier accepted step i of the window moved the same molecule,
// or moved a molecule whose primaries, before or after step i, come within
// the screen's outer guard radius of step j's molecule at either of its
// placements (the screen of step j could have seen that move).  Such a step
// is staged again if needed and re-evaluated on the current state by every
// CTA alike.
//
// The decisions of a window are taken side by side: lane j of every warp
// decides step j on its record, warp j has found the steps step j depends on
// (once the moves are staged, before the evaluation), and the first step that
// depends on an accepted one is a vote away.  The steps before it stand and
// are committed by one warp each.  Walking the steps one by one, every warp
// committing each, took 2 to 2.5 us a step and most of a window: 28 us per
// window of 8 on 32,768 waters where a step's evaluation takes 10.
//
// Decisions, coordinates and counters are therefore those of the one-group
// kernel on the same draws; the FP32 pair sums are its own up to their order (it
// evaluates with one warp less on chains whose items the warps share, the last
// one staging the next move).
//
// Memory: every CTA writes every accepted placement (the same values), and
// a CTA reads the pool only after its own writes of every earlier step.  A
// CTA that runs ahead could only harm a slower one by committing a later
// step while the slower one still reads the state for an earlier step;
// that happens only during a re-evaluation, and a re-evaluated step ends
// with a cluster-wide wait before anyone commits it.  The waits are counts
// stored into every CTA's shared memory (after a release fence) and polled
// in the CTA's own (then an acquire fence), one lane per CTA of the cluster,
// with a time limit: on expiry the chain's error word is set
// and the CTA leaves its loop, so a fault in this protocol ends the launch
// with an error status instead of a stalled GPU.  The only hardware cluster
// barriers are at entry (before any remote store) and at exit (no CTA
// leaves while another may still store into its shared memory); every
// thread passes each of them once.
#include "chain.cuh"
#include "host.h"

namespace mcgpu {

namespace {

// What a CTA found for its step of the window (and what a re-evaluation
// finds): the FP32 totals in double-float, the sum of magnitudes, the
// pairs counted, and the FP64 totals when the decision is taken on them.
struct __align__(16) WinRec {
  float oh, ol, nh, nl, ab;
  int tie;
  long long np;
  double eo, en;
};
static_assert(sizeof(WinRec) == 48, "WinRec layout");

// Wait limit of a cluster-wide wait (ns of the global timer): far above any
// legitimate wait (a step's evaluation, milliseconds at most).
constexpr unsigned long long kWinWaitNs = 4000000000ull;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ unsigned cluster_size() {
  unsigned n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}

// Hardware cluster barrier (entry and exit only).
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Address of p (this CTA's shared memory) in CTA `rank`'s shared memory.
__device__ __forceinline__ unsigned remote_addr(const void* p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(a)
               : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}

__device__ __forceinline__ void st_remote_u64(unsigned a, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

__device__ __forceinline__ void st_remote_relaxed(unsigned a, unsigned v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned ld_relaxed_cluster(unsigned a) {
  unsigned v;
  asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void fence_cluster() {
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
}

// Shared memory of the window protocol, after the group's own.
struct WinSmem {
  WinRec* rec;        // [2][K]: the records of the window (two windows in rotation)
  unsigned* flag;     // [K]: barrier count CTA q reached, stored by CTA q
  unsigned* ok;       // [2]: outcome of this CTA's last waits
  unsigned* dep;      // [K]: steps of the window step j depends on: the same
                      // molecule (bits 16 + i) or one in range (bits i)
  char* slots;        // [2][K] staging slots (two windows in rotation)
};

__host__ __device__ inline int win_extra_bytes(const SmemShape& sh, int K) {
  return SmemShape::align16(2 * K * (int)sizeof(WinRec)) + 2 * SmemShape::align16(K * 4) + 16 +
         2 * K * sh.ahead_bytes();
}

// Cluster-wide wait number n, lane q of warp 0 serving CTA q: it stores
// rec (if any) into slot rec_at of CTA q's records, fences (release), stores
// the count n into this CTA's flag slot in CTA q, then polls CTA q's slot of
// this CTA's flag row until it reaches n or the limit passes, and fences
// (acquire).  The CTA barrier after it carries what the lanes acquired to
// every thread.  The outcome is the same in every thread of the CTA.
__device__ bool win_wait(const Group& g, const WinSmem& ws, unsigned K, unsigned rank, unsigned n,
                         const WinRec* rec, int rec_at) {
  if (g.tid < 32) {
    const unsigned q = g.tid;
    bool ok = true;
    if (q < K) {
      if (rec) {
        const unsigned a = remote_addr(ws.rec + rec_at, q);
        const unsigned long long* w = (const unsigned long long*)rec;
        for (int k = 0; k < (int)(sizeof(WinRec) / 8); k++) st_remote_u64(a + 8 * k, w[k]);
      }
      fence_cluster();
      st_remote_relaxed(remote_addr(ws.flag + rank, q), n);
      const unsigned a = remote_addr(ws.flag + q, rank);
      const unsigned long long t0 = global_ns();
      unsigned it = 0;
      while (ld_relaxed_cluster(a) < n) {
        if ((++it & 63) == 0 && global_ns() - t0 > kWinWaitNs) {
          ok = false;
          break;
        }
      }
      fence_cluster();
    }
    ok = __all_sync(~0u, ok);
    if (g.tid == 0) ws.ok[n & 1] = ok ? 1u : 0u;
  }
  g.sync();
  return ws.ok[n & 1] != 0;
}

// Whether step i (slot a), once accepted, has moved a molecule that step j's
// screen (slot b) could see: a primary pair within the guard band's outer
// radius for any of the four placement pairs, with the screen's own FP32
// distance (same operands, same order).  One thread.
__device__ bool window_near(const StageSlot& a, const StageSlot& b, const ChainHdr& H) {
  const int na = a.misc[3], nb = b.misc[3];
  for (int ka = 0; ka < na; ka++) {
    const float4 ao = a.p_old[ka], an = a.p_new[ka];
    for (int kb = 0; kb < nb; kb++) {
      const float4 bo = b.p_old[kb], bn = b.p_new[kb];
      if (r2_screen(bo, ao, H) <= H.cut2_hi || r2_screen(bn, ao, H) <= H.cut2_hi ||
          r2_screen(bo, an, H) <= H.cut2_hi || r2_screen(bn, an, H) <= H.cut2_hi)
        return true;
    }
  }
  return false;
}

// The decision on a record: on the FP64 totals where it holds them, else on
// the FP32 ones; bound gets the rounding bound of the FP32 difference.
__device__ __forceinline__ bool window_accept(const WinRec& x, float u, const ChainHdr& H,
                                              float& bound) {
  const float de_f = __fadd_rn(__fsub_rn(x.nh, x.oh), __fsub_rn(x.nl, x.ol));
  bound = (float)kTieRel * x.ab + 2.4e-7f * (fabsf(x.nh) + fabsf(x.oh)) + 1e-9f;
  if (x.tie) {
    const double d64 = x.en - x.eo;
    return (d64 < 0) || (exp(-d64 / H.kT) >= (double)u);
  }
  const float pf = expf(-fmaxf(de_f, 0.f) * H.kTinvf);
  return (de_f < 0.f) || (pf >= u);
}

// The one-group kernel's step evaluation (chain_steps in kernels.cu): FP32
// pair terms over the candidates (the Verlet list when use_list), the FP32
// decision's guard band, and inside it -- or for FP64-pair chains -- both
// placements again with FP64 pairs.  nred counts the group reductions (their
// scratch alternates between two buffers).
__device__ void window_eval(const Pool& P, const ChainHdr& H, const Group& g, const GroupSmem& ss,
                            const MovedInfo& mi, const float4* pcache, bool use_list, int T,
                            float u, int& nred, WinRec& x) {
  const int lane = g.tid & 31, w = g.warp(), nw = g.nwarps();
  AccFF acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0};
  const bool f64all = H.fp64_pairs != 0;
  if (f64all) {
  } else if (use_list) {
    group_eval_chain(P, H, g, ss, mi, pcache, 0, P.nl_cnt[mi.mol], nw, T, acc,
                     P.nl + (size_t)mi.mol * P.nl_stride);
  } else {
    group_eval_chain(P, H, g, ss, mi, pcache, H.mol0, H.mol0 + H.n_mol, nw, T, acc);
  }
  group_reduce_ff(g, ss, acc, nred++ & 1);
  const float de_f = __fadd_rn(__fsub_rn(acc.nh, acc.oh), __fsub_rn(acc.nl, acc.ol));
  const float bound = (float)kTieRel * acc.ab + 2.4e-7f * (fabsf(acc.nh) + fabsf(acc.oh)) + 1e-9f;
  const float pf = expf(-fmaxf(de_f, 0.f) * H.kTinvf);
  const int tie = f64all ||
                  ((de_f >= -bound) && (fabsf(pf - u) <= pf * (1.5f * bound * H.kTinvf) + 1e-6f));
  x.oh = acc.oh;
  x.ol = acc.ol;
  x.nh = acc.nh;
  x.nl = acc.nl;
  x.ab = acc.ab;
  x.np = acc.np;
  x.tie = tie;
  x.eo = 0.0;
  x.en = 0.0;
  if (tie) {
    if (w == 0) stage_chain_f64(P, H, ss, mi, lane);
    g.sync();
    double eo = 0.0, en = 0.0;
    long long np2 = 0;
    if (use_list)
      warp_eval_chain64(P, H, ss, mi, pcache, 0, P.nl_cnt[mi.mol], w, nw, lane, eo, en, np2,
                        P.nl + (size_t)mi.mol * P.nl_stride);
    else
      warp_eval_chain64(P, H, ss, mi, pcache, H.mol0, H.mol0 + H.n_mol, w, nw, lane, eo, en, np2);
    group_reduce(g, ss, eo, en, np2, nred++ & 1);
    x.eo = eo;
    x.en = en;
    if (f64all) x.np = np2;   // (a re-take's pairs are counted already)
  }
}

}  // namespace

// One cluster of K CTAs per chain task (task k runs chain order[k]; cluster
// c takes tasks c, c + clusters, ...), one group of all the CTA's warps per
// CTA; n_steps steps per chain in windows of K.  trace, trace_off,
// trace_stride and lanes_cap as in chain_steps.
//
// kMaxThreads 512 has 128 registers a thread and spills; 256, for CTAs of up to eight
// warps, takes the 214 it wants: windows of 4 steps on 64 molecules of 3 and 64 atoms
// 15.1 ms for 200 steps and 10.7, on 256 9-atom molecules 0.86 and 0.74.
template <int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_chain_window(Pool P, int n_steps, const int* order, int n_tasks, SmemShape shape,
                   mcgpu_trace* trace, int trace_off, int trace_stride, int lanes_cap,
                   bool count_redo) {
  extern __shared__ __align__(16) char smem[];
  const unsigned K = cluster_size(), rank = cluster_rank();
  const int n_cl = (int)(gridDim.x / K), cid = (int)(blockIdx.x / K);
  const Group g{(int)threadIdx.x, (int)blockDim.x, 1};
  GroupSmem s = shape.carve(smem);
  WinSmem ws;
  {
    char* p = smem + shape.bytes();
    ws.rec = (WinRec*)p;
    p += SmemShape::align16(2 * K * (int)sizeof(WinRec));
    ws.flag = (unsigned*)p;
    p += SmemShape::align16(K * 4);
    ws.ok = (unsigned*)p;
    p += 16;
    ws.dep = (unsigned*)p;
    p += SmemShape::align16(K * 4);
    ws.slots = p;
  }
  const int sbytes = shape.ahead_bytes();
  auto slot = [&](int par, int j) { return shape.ahead_slot(ws.slots + (par * (int)K + j) * sbytes); };
  const int lane = threadIdx.x & 31, w = g.warp(), nw = g.nwarps();
  for (int q = g.tid; q < (int)K; q += g.nthreads) ws.flag[q] = 0u;
  cluster_barrier();
  unsigned nbar = 0;
  bool alive = true;
  for (int task = cid; task < n_tasks && alive; task += n_cl) {
    const int c = order[task];
    ChainHdr* Hp = P.hdr + c;
    const ChainHdr& H = *Hp;
    float4* pcache = (s.pc && H.simple_prim && H.n_mol <= shape.cache_n) ? s.pc : nullptr;
    if (pcache)
      for (int i = g.tid; i < H.n_mol; i += g.nthreads) pcache[i] = P.ppos[H.pidx0 + i];
    if (H.uniform)
      for (int i = g.tid; i < H.ulen; i += g.nthreads) s.teq[i] = P.aeq[H.atom0 + i];
    g.sync();
    if (g.tid == 0) Hp->ljmask = uniform_lj_mask(P, H, s.teq);  // the same value in every CTA
    // warp 0 of the first CTA keeps the chain's sums and counters, one step
    // of the window per lane
    const bool lead = rank == 0 && w == 0;
    int full_scans = 0, ties = 0, redo = 0;
    float de_h = 0.f, de_l = 0.f, err_h = 0.f, err_l = 0.f;
    long long acc_n = 0, npairs = 0;
    const unsigned long long step0 = H.step;
    bool nl_ok = H.nl_on && H.nl_valid;
    const int T = lanes_cap > 0 ? min(lanes_cap, H.tpm)
                                : ((H.uniform && H.ulen <= 4 && !H.precise) ? 1 : H.tpm);
    MoveF* props = (MoveF*)s.props;
    int my_steps = n_steps;
    if (H.step_limit > 0)
      my_steps = (int)max(0LL, min((long long)n_steps, H.step_limit - (long long)step0));
    int nred = 0;
    for (int s0 = 0; s0 < my_steps; s0 += (int)K) {
      const int nst = min((int)K, my_steps - s0), par = (s0 / (int)K) & 1;
      WinRec* recs = ws.rec + par * (int)K;
      // draws 32 steps at a time (K divides 32, so a window never straddles)
      if ((s0 & 31) == 0) {
        if (w == 0) {
          if (s0 + lane < my_steps)
            props[lane] = draw_move_f32(H.seed, H.chain_id, step0 + s0 + lane, H.n_mol,
                                        P.mlen + H.mol0, (float)H.max_t, (float)H.max_r,
                                        H.rot_mode);
          __syncwarp();
        }
        g.sync();
      }
      // warp j stages step s0 + j, then finds the steps it depends on
      if (w < nst) stage_chain(P, H, props[(s0 + w) & 31], slot(par, w), pcache, lane);
      g.sync();
      if (w < nst) {
        bool same = false, near = false;
        if (lane < w) {
          const StageSlot ti = slot(par, lane), tj = slot(par, w);
          same = ti.misc[0] == tj.misc[0];
          near = same || window_near(ti, tj, H);
        }
        const unsigned d = __ballot_sync(~0u, near) | (__ballot_sync(~0u, same) << 16);
        if (lane == 0) ws.dep[w] = d;
      }
      const bool nl_ok0 = nl_ok;
      WinRec x = {};
      if ((int)rank < nst) {
        const GroupSmem ss = with_slot(s, slot(par, rank));
        const MovedInfo mi = load_moved(ss);
        window_eval(P, H, g, ss, mi, pcache, nl_ok0 && ss.misc[kMiscNlTrial] != 0, T,
                    __int_as_float(ss.misc[kMiscU]), nred, x);
      }
      if (!win_wait(g, ws, K, rank, ++nbar, &x, par * (int)K + (int)rank)) {
        alive = false;
        break;
      }
      // lane j: step j's decision on its record, dependences, and whether its
      // trial placement leaves the Verlet list valid
      unsigned dep = 0;
      bool ok = false, trial_near = true, listed = false;
      if (lane < nst) {
        const StageSlot tj = slot(par, lane);
        float bound;
        ok = window_accept(recs[lane], __int_as_float(tj.misc[kMiscU]), H, bound);
        trial_near = tj.misc[kMiscNlTrial] != 0;
        listed = nl_ok0 && trial_near;
        dep = ws.dep[lane];
      }
      unsigned okm = __ballot_sync(~0u, ok);
      for (int cur = 0;;) {
        // the first undecided step that depends on an accepted earlier one
        const unsigned conf = __ballot_sync(
            ~0u, lane >= cur && lane < nst && (dep & okm & ((1u << lane) - 1u)) != 0);
        const int jx = conf ? __ffs(conf) - 1 : nst;
        // the steps before it stand: warp j commits step j if accepted
        if (w >= cur && w < jx && ((okm >> w) & 1u)) {
          const GroupSmem ss = with_slot(s, slot(par, w));
          commit_chain(P, H, ss, load_moved(ss), pcache, lane);
        }
        if (__any_sync(~0u, lane >= cur && lane < jx && ok && !trial_near)) nl_ok = false;
        if (jx == nst) break;
        g.sync();  // the commits, before the state is read again
        const StageSlot tj = slot(par, jx);
        const GroupSmem ss = with_slot(s, tj);
        const unsigned dj = __shfl_sync(~0u, dep, jx);
        if ((dj >> 16) & okm & ((1u << jx) - 1u)) {
          // staged from rows an earlier step of the window changed: stage it
          // again, and look which later steps its new placements reach
          if (w == 0) stage_chain(P, H, props[(s0 + jx) & 31], tj, pcache, lane);
          g.sync();
          if (lane > jx && lane < nst) {
            const StageSlot tk = slot(par, lane);
            const bool near = tk.misc[0] == tj.misc[0] || window_near(tj, tk, H);
            dep = (dep & ~(1u << jx)) | ((near ? 1u : 0u) << jx);
          }
        }
        const bool near_j = ss.misc[kMiscNlTrial] != 0;
        const bool listed_j = nl_ok && near_j;
        const float uj = __int_as_float(ss.misc[kMiscU]);
        WinRec xj;
        window_eval(P, H, g, ss, load_moved(ss), pcache, listed_j, T, uj, nred, xj);
        // nobody commits step j (or a later one) while a CTA still reads the
        // state for it
        if (!win_wait(g, ws, K, rank, ++nbar, nullptr, 0)) {
          alive = false;
          break;
        }
        float bound;
        const bool okj = window_accept(xj, uj, H, bound);
        okm = (okm & ~(1u << jx)) | ((okj ? 1u : 0u) << jx);
        if (lane == jx) {
          ok = okj;
          trial_near = near_j;
          listed = listed_j;
          if (lead) recs[jx] = xj;
        }
        if (okj && w == jx) commit_chain(P, H, ss, load_moved(ss), pcache, lane);
        if (okj && !near_j) nl_ok = false;
        redo++;
        cur = jx + 1;
      }
      if (!alive) break;
      if (lead) {
        __syncwarp();
        float vh = 0.f, vl = 0.f, ve = 0.f;
        long long np = 0;
        int tie = 0;
        if (lane < nst) {
          const WinRec r = recs[lane];
          tie = r.tie;
          np = r.np;
          if (ok) {
            if (r.tie) {
              const double d64 = r.en - r.eo;
              vh = (float)d64;
              vl = (float)(d64 - (double)vh);
              ve = 1e-12f * r.ab;
            } else {
              vh = r.nh;
              vl = r.nl;
              ff_add2(vh, vl, -r.oh, -r.ol);
              ve = (float)kTieRel * r.ab + 2.4e-7f * (fabsf(r.nh) + fabsf(r.oh)) + 1e-9f;
            }
          }
          if (trace) {
            const StageSlot tj = slot(par, lane);
            double e_old = r.eo, e_new = r.en;
            if (!r.tie) {
              e_old = (double)r.oh + (double)r.ol;
              e_new = (double)r.nh + (double)r.nl;
            }
            mcgpu_trace t;
            t.mol = tj.misc[0] - H.mol0;
            t.accepted = ok ? 1 : 0;
            t.e_old = e_old;
            t.e_new = e_new;
            t.de = e_new - e_old;
            t.u = (double)__int_as_float(tj.misc[kMiscU]);
            t.fp64 = r.tie;
            t.pad0 = 0;
            trace[(size_t)c * trace_stride + trace_off + s0 + lane] = t;
          }
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) {
          const float oh = __shfl_xor_sync(~0u, vh, off), ol = __shfl_xor_sync(~0u, vl, off);
          ff_add2(vh, vl, oh, ol);
          ve += __shfl_xor_sync(~0u, ve, off);
        }
        ff_add2(de_h, de_l, vh, vl);   // lane 0's is the window's
        ff_add(err_h, err_l, ve);
        acc_n += __popc(okm);
        npairs += warp_count(np);
        ties += __popc(__ballot_sync(~0u, tie != 0));
        full_scans += __popc(__ballot_sync(~0u, H.nl_on && lane < nst && !listed));
      }
      g.sync();  // the commits, before the next moves are staged
    }
    if (!alive) {
      if (g.tid == 0) Hp->error = kErrWindowSync;
      break;
    }
    if (lead && lane == 0) {
      Hp->energy = H.energy + ((double)de_h + (double)de_l);
      Hp->run_err += (double)err_h + (double)err_l;
      Hp->step = step0 + my_steps;
      Hp->accepted += acc_n;
      Hp->pairs += npairs;
      Hp->ties += ties;
      if (count_redo) Hp->win_redo += redo;
      if (H.nl_on) {
        Hp->nl_valid = nl_ok ? 1 : 0;
        Hp->nl_full += full_scans;
      }
    }
    g.sync();
  }
  cluster_barrier();
}

int window_smem_bytes(const SmemShape& sh, int K) { return sh.bytes() + win_extra_bytes(sh, K); }

cudaError_t window_init() {
  for (const auto kernel : {k_chain_window<512>, k_chain_window<256>}) {
    const cudaError_t e = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindowSmemMax);
    if (e != cudaSuccess) return e;
    // clusters of 16 CTAs are beyond the portable size of 8; where the device
    // refuses them, window_max_clusters reports none and the setters refuse
    // the window
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
        cudaSuccess)
      cudaGetLastError();
  }
  return cudaSuccess;
}

using WindowKernel = decltype(&k_chain_window<512>);

// Launch configuration of n_clusters clusters of K CTAs; at holds its one attribute.
static cudaLaunchConfig_t window_config(int K, int n_clusters, int threads, int smem,
                                        cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(K * n_clusters, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = K;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

static int active_clusters(WindowKernel kernel, int K, int threads, int smem) {
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = window_config(K, 1, threads, smem, &at);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int window_max_clusters(int K, int threads, int smem) {
  return active_clusters(k_chain_window<512>, K, threads, smem);
}

cudaError_t launch_chain_window(int K, int n_clusters, int threads, int smem, cudaStream_t st,
                                const Pool& P, int n_steps, const int* order, int n_tasks,
                                SmemShape sh, mcgpu_trace* trace, int trace_off, int trace_stride,
                                int lanes_cap, bool count_redo) {
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = window_config(K, n_clusters, threads, smem, &at);
  cfg.stream = st;
  // the kernel of more registers where all clusters are resident with it too (37
  // clusters of 4 are not: one more wave, 1.15 ms against 1.28)
  const bool few = threads <= 256 &&
                   active_clusters(k_chain_window<256>, K, threads, smem) >= n_clusters;
  return cudaLaunchKernelEx(&cfg, few ? k_chain_window<256> : k_chain_window<512>, P, n_steps,
                            order, n_tasks, sh, trace, trace_off, trace_stride, lanes_cap,
                            count_redo);
}

}  // namespace mcgpu
