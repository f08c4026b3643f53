// nlist.cu -- Verlet neighbour lists of device-resident chains, built on the
// GPU from a cell list.
//
// A chain's list of molecule i holds every molecule j whose anchor (first
// primary atom) was within r_list = rc + skin + 2 prad of i's anchor at the
// build, prad the largest primary-to-anchor distance of the chain.  While
// every primary of every molecule stays within skin/2 of its position at
// the build, any molecule pair with a primary pair inside rc is in the list,
// so the chain kernel screens the list instead of all molecules and finds
// the same in-range set (the screen itself is unchanged).  The kernel checks
// the trial placement against skin/2 (full scan for that step if it is
// farther) and marks the list stale when such a placement is accepted; the
// rebuild below runs between launches for stale chains only.
//
// Cells: ncell[k] = floor(L_k / r_list) per edge (at least 1, at most the
// chain's allocated cells); molecule m is in cell floor(A_k * ncell[k] /
// 2^32) of its fixed-point anchor A, exact and wrap-free.  Each cell's
// members are sorted by index and each list is written cell by cell in a
// fixed stencil order, so the lists (and the pair summation order that
// follows them) are deterministic.
//
// Two launches: the cells of a chain by one CTA, the lists by CTAs of a cell's
// members.  They run before every step launch and find nothing to do nine
// times in ten, and then they are two empty launches (as seven kernels they
// cost 18 us beside the 120 us of a 64-step launch).
#include "chain.cuh"

namespace mcgpu {

__device__ __forceinline__ bool nl_rebuilding(const ChainHdr& H) { return H.nl_on && !H.nl_valid; }

__device__ __forceinline__ int cell_of(unsigned a, int n) {
  return (int)(((unsigned long long)a * (unsigned)n) >> 32);
}

constexpr int kNlCellThreads = 1024;
constexpr int kNlSortMax = 256;   // members of a cell sorted in shared memory

// The cells of a stale chain (blockIdx.x): grid from its current box, members
// counted, scanned, scattered, and each cell's sorted by index -- a warp per
// cell writes each member at its rank.  One CTA: 32,768 waters in 343 cells
// take the time of a few step launches, once per rebuild.
__global__ void __launch_bounds__(kNlCellThreads) k_nl_cells(Pool P) {
  ChainHdr& H = P.hdr[blockIdx.x];
  if (!nl_rebuilding(H)) return;
  __shared__ int nc[3];
  __shared__ int tot[kNlCellThreads / 32];
  __shared__ int buf[kNlCellThreads / 32][kNlSortMax];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) {
    for (int k = 0; k < 3; k++) nc[k] = max(1, (int)floor(H.L[k] / (double)H.nl_rlist));
    // fewer, larger cells if the grid outgrew its allocation (box growth)
    while (nc[0] * nc[1] * nc[2] > H.cell_cap) {
      int kmax = 0;
      for (int k = 1; k < 3; k++)
        if (nc[k] > nc[kmax]) kmax = k;
      nc[kmax]--;
    }
    for (int k = 0; k < 3; k++) H.ncell[k] = nc[k];
  }
  __syncthreads();
  const int n0 = nc[0], n1 = nc[1], n2 = nc[2], n = n0 * n1 * n2;
  const int m0 = H.mol0, m1 = H.mol0 + H.n_mol, c0 = H.cell0;
  for (int i = tid; i < n; i += kNlCellThreads) P.cell_cnt[c0 + i] = 0;
  __syncthreads();
  for (int m = m0 + tid; m < m1; m += kNlCellThreads) {
    const uint4 A = P.mfix[m];
    const int cell = c0 + (cell_of(A.x, n0) * n1 + cell_of(A.y, n1)) * n2 + cell_of(A.z, n2);
    P.mcell[m] = cell;
    atomicAdd(&P.cell_cnt[cell], 1);
  }
  __syncthreads();
  // exclusive scan into cell_start (pool positions from the chain's first
  // molecule), 1,024 cells a pass; the counters are reset for the scatter
  int run = m0;
  for (int i0 = 0; i0 < n; i0 += kNlCellThreads) {
    const int i = i0 + tid;
    const int v = i < n ? __ldcg(P.cell_cnt + c0 + i) : 0;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(~0u, incl, off);
      if (lane >= off) incl += u;
    }
    if (lane == 31) tot[w] = incl;
    __syncthreads();
    if (w == 0) {
      int t = tot[lane];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int u = __shfl_up_sync(~0u, t, off);
        if (lane >= off) t += u;
      }
      tot[lane] = t;
    }
    __syncthreads();
    if (i < n) {
      P.cell_start[c0 + i] = run + (w > 0 ? tot[w - 1] : 0) + incl - v;
      P.cell_cnt[c0 + i] = 0;
    }
    run += tot[kNlCellThreads / 32 - 1];
    __syncthreads();
  }
  for (int m = m0 + tid; m < m1; m += kNlCellThreads) {
    const int cell = P.mcell[m];
    const int pos = atomicAdd(&P.cell_cnt[cell], 1);
    P.cell_mol[P.cell_start[cell] + pos] = m;
  }
  __syncthreads();
  for (int i = w; i < n; i += kNlCellThreads / 32) {
    int* v = P.cell_mol + P.cell_start[c0 + i];
    const int cnt = __ldcg(P.cell_cnt + c0 + i);
    if (cnt <= kNlSortMax) {
      for (int k = lane; k < cnt; k += 32) buf[w][k] = v[k];
      __syncwarp();
      for (int k = lane; k < cnt; k += 32) {
        const int key = buf[w][k];
        int rank = 0;
        for (int q = 0; q < cnt; q++) rank += buf[w][q] < key;
        v[rank] = key;
      }
      __syncwarp();
    } else if (lane == 0) {
      // a cell of a box of few cells: in place
      for (int a = 1; a < cnt; a++) {
        const int key = v[a];
        int b = a - 1;
        while (b >= 0 && v[b] > key) {
          v[b + 1] = v[b];
          b--;
        }
        v[b + 1] = key;
      }
    }
  }
}

// Cells of the stencil along one edge: c-1, c, c+1 (periodic) when the edge
// has at least 3 cells, else every cell once.
__device__ __forceinline__ int stencil(int c, int n, int* out) {
  if (n >= 3) {
    out[0] = (c + n - 1) % n;
    out[1] = c;
    out[2] = (c + 1) % n;
    return 3;
  }
  for (int k = 0; k < n; k++) out[k] = k;
  return n;
}

// The lists of a stale chain (blockIdx.y), a quarter of a cell's members at a
// time (gridDim.x CTAs stride over the quarters): the screen positions of the stencil cells' members
// go to shared memory in chunks, in cell and member order, and each warp
// appends the near ones to its molecules' lists in that order (a warp per
// molecule that followed cell_mol -> mpi -> ppos for each of its 2,200
// candidates took 440 us for 32,768 waters).  Also the build positions of the
// members' primaries.  The last CTA of the chain marks its lists valid; a
// chain with a list beyond its row drops its lists (full scans stay exact).
constexpr int kNlThreads = 256;
constexpr int kNlChunk = 1536;
constexpr int kNlSlices = 4;

__global__ void __launch_bounds__(kNlThreads) k_nl_build(Pool P) {
  ChainHdr& H = P.hdr[blockIdx.y];
  if (!nl_rebuilding(H)) return;
  __shared__ float4 pos[kNlChunk];
  __shared__ int mol[kNlChunk];
  __shared__ int start[27], pref[28];
  __shared__ int n_cells;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int n0 = H.ncell[0], n1 = H.ncell[1], n2 = H.ncell[2];
  for (int item = blockIdx.x; item < n0 * n1 * n2 * kNlSlices; item += gridDim.x) {
    const int local = item / kNlSlices, slice = item - local * kNlSlices;
    const int cell = H.cell0 + local;
    const int cnt = P.cell_cnt[cell], first = P.cell_start[cell];
    const int per = (cnt + kNlSlices - 1) / kNlSlices;
    const int i0 = min(cnt, slice * per), i1 = min(cnt, i0 + per);
    if (i0 < i1) {
      __syncthreads();   // the last item's stencil is read no more
      if (w == 0) {
        const int cz = local % n2, cy = (local / n2) % n1, cx = local / (n1 * n2);
        int sx[3], sy[3], sz[3];
        const int nx = stencil(cx, n0, sx), ny = stencil(cy, n1, sy), nz = stencil(cz, n2, sz);
        const int n = nx * ny * nz;
        int st = 0, c = 0;
        if (lane < n) {
          const int a = lane / (ny * nz), b = (lane / nz) % ny, d = lane % nz;
          const int q = H.cell0 + (sx[a] * n1 + sy[b]) * n2 + sz[d];
          st = P.cell_start[q];
          c = P.cell_cnt[q];
        }
        int incl = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int u = __shfl_up_sync(~0u, incl, off);
          if (lane >= off) incl += u;
        }
        if (lane < n) {
          start[lane] = st;
          pref[lane] = incl - c;
        }
        if (lane == n - 1) {
          pref[n] = incl;
          n_cells = n;
        }
      }
      __syncthreads();
      const int total = pref[n_cells];
      const bool simple = H.simple_prim != 0;
      const float Lx = H.Lf[0], Ly = H.Lf[1], Lz = H.Lf[2], nl_r2 = H.nl_r2;
      const unsigned lt = lanemask_lt();
      bool over = false;
      for (int c0 = 0; c0 < total; c0 += kNlChunk) {
        const int c1 = min(total, c0 + kNlChunk);
        int k = 0;
        for (int t = c0 + tid; t < c1; t += kNlThreads) {
          while (pref[k + 1] <= t) k++;
          const int j = P.cell_mol[start[k] + (t - pref[k])];
          mol[t - c0] = j;
          pos[t - c0] = P.ppos[simple ? H.pidx0 + (j - H.mol0) : P.mpi[j].x];
        }
        __syncthreads();
        for (int i = i0 + w; i < i1; i += kNlThreads / 32) {
          const int m = P.cell_mol[first + i];
          const int2 pi = P.mpi[m];
          if (c0 == 0)
            for (int q = lane; q < pi.y; q += 32) P.pbuild[pi.x + q] = P.ppos[pi.x + q];
          const float4 am = P.ppos[pi.x];
          int* out = P.nl + (size_t)m * P.nl_stride;
          int cnt_m = c0 == 0 ? 0 : P.nl_cnt[m];
          for (int base = 0; base < c1 - c0; base += 32) {
            const int t = base + lane;
            bool in = false;
            int j = -1;
            if (t < c1 - c0) {
              j = mol[t];
              const float4 q = pos[t];
              const float dx = wrapf(q.x - am.x, Lx), dy = wrapf(q.y - am.y, Ly),
                          dz = wrapf(q.z - am.z, Lz);
              in = j != m && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= nl_r2;
            }
            const unsigned bal = __ballot_sync(~0u, in);
            if (in) {
              const int at = cnt_m + __popc(bal & lt);
              if (at < P.nl_stride) out[at] = j;
              else over = true;
            }
            cnt_m += __popc(bal);
          }
          __syncwarp();
          if (lane == 0) P.nl_cnt[m] = min(cnt_m, P.nl_stride);
          __syncwarp();
        }
        __syncthreads();
      }
      if (__any_sync(~0u, over) && lane == 0) atomicAdd(&H.nl_overflow, 1);
    }
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    // nl_done counts the chain's CTAs of this launch
    if (atomicAdd(&H.nl_done, 1) == (int)gridDim.x - 1) {
      __threadfence();
      H.nl_done = 0;
      if (*(volatile int*)&H.nl_overflow) {
        H.nl_on = 0;
      } else {
        H.nl_builds++;
        H.nl_valid = 1;
      }
    }
  }
}

// Per-chain list configuration (host-computed), applied to the headers.
__global__ void k_nl_config(Pool P, const NlCfg* cfg) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= P.n_chains) return;
  ChainHdr& H = P.hdr[c];
  const NlCfg f = cfg[c];
  H.nl_on = f.on;
  H.nl_valid = 0;
  H.nl_overflow = 0;
  H.cell0 = f.cell0;
  H.cell_cap = f.cell_cap;
  H.nl_r2 = f.r2;
  H.nl_half2 = f.half2;
  H.nl_rlist = f.rlist;
}

cudaError_t launch_nl_rebuild(Pool P, int max_cells, int sm_count, cudaStream_t st) {
  const int nc = P.n_chains;
  k_nl_cells<<<nc, kNlCellThreads, 0, st>>>(P);
  // six CTAs an SM in all, no more than a chain has work for
  int gx = sm_count * 6 / nc;
  gx = gx < 1 ? 1 : gx > max_cells * kNlSlices ? max_cells * kNlSlices : gx;
  // grid.y holds at most 65,535 chains
  for (int c0 = 0; c0 < nc; c0 += 65535) {
    Pool Q = P;
    Q.hdr += c0;
    k_nl_build<<<dim3(gx, nc - c0 < 65535 ? nc - c0 : 65535), kNlThreads, 0, st>>>(Q);
  }
  return cudaGetLastError();
}

}  // namespace mcgpu
