// static_energy.cu -- mcgpu_system_energy_static: the FP64 system energy
// (SimulationStep::calcSystemEnergy's pairs and in-range test; the pair terms, as
// exact as the reference's, from 1/r of an FP64 rsqrt: pair_sum64) over SimBox rows
// that the CALLER already holds in device memory, without allocating anything.
//
// Who needs it: programs that cannot call cudaMalloc for this library --
// an OpenACC or OpenMP-offload build that keeps its SimBox rows in its own
// device data region (as MCGPU's -p build does through acc_copyin), or an
// application whose device memory is owned by another allocator (a
// framework's caching allocator, a fixed arena of a long-running service)
// and forbids allocations from third-party code.  They pass device pointers
// to their rows and to one output double; the partial energies live in a fixed
// file-scope device array instead of a cudaMalloc'd buffer.
//
// Limits and sharing: at most kStaticMaxMol molecules per call (larger boxes
// are rejected with MCGPU_ERR_UNSUPPORTED).  Every GPU that loads the
// library holds the array (kStaticMaxMol doubles, 256 KiB) until the process
// exits.  All calls on a device share it and it keeps the last call's
// contents; each entry a call reads was written earlier in that same call,
// so nothing needs clearing, but calls that overlap on the GPU (different
// streams, no ordering) race on it.  The first call on each device looks up
// the array's device address (cudaGetSymbolAddress) with that device
// current and caches it; make that first call before any stream capture.
// The cache is keyed on the current context's id: after a device reset or a
// new primary context the next call looks the address up again (that call
// is then a first call, with the same rule on capture).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <mutex>

#include "pairsum.cuh"
#include "static_scratch_cache.h"

namespace mcgpu {
void note_process_error(const char* msg);  // abi.cu: text for mcgpu_last_error(NULL)
}

namespace {
constexpr int kStaticMaxMol = 32768;
constexpr int kMaxDevices = 64;
}  // namespace

// The scratch: one partial sum of E(m, j > m) per CTA (at most one per
// molecule of the box), one copy per device, never cleared (every entry a
// call reads, it wrote first).
static __device__ __align__(256) double g_static_emol[kStaticMaxMol];

namespace {

struct Rows {
  const double *x, *y, *z, *sig, *eps, *q;
  const int *mstart, *mlen, *mps, *mpc, *pidx;
  int n_mol, n_atom, n_pidx;
  double L[3], cutoff;
};

// SimCalcs::calcAtomDistSquared (SimulationStep.cpp:332-342), a2 - a1.
__device__ __forceinline__ double dist2(const Rows& r, int a1, int a2) {
  const double dx = mcgpu::make_periodic(r.x[a2] - r.x[a1], r.L[0]);
  const double dy = mcgpu::make_periodic(r.y[a2] - r.y[a1], r.L[1]);
  const double dz = mcgpu::make_periodic(r.z[a2] - r.z[a1], r.L[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Row ranges of molecule m inside the arrays.  A molecule without primary
// indexes (pc == 0) is valid: moleculesInRange is false for it
// (SimulationStep.cpp:317-330), so it contributes nothing.
__device__ __forceinline__ bool valid_mol(const Rows& r, int m) {
  const int s = r.mstart[m], n = r.mlen[m], ps = r.mps[m], pc = r.mpc[m];
  return s >= 0 && n >= 1 && s + n <= r.n_atom && ps >= 0 && pc >= 0 && ps + pc <= r.n_pidx;
}

// The caller's rows as ps_items reads them: sigma as it is, sqrt(eps), -1 for
// a skipped site (a negative sigma or epsilon, BruteForceStep.cpp:64-65).
struct StaticRows {
  const Rows& r;
  __device__ __forceinline__ int len(int j) const { return r.mlen[j]; }
  __device__ __forceinline__ int start(int j) const { return r.mstart[j]; }
  __device__ __forceinline__ void atom(int b, double& x, double& y, double& z, double& sb,
                                       double& eb, double& qb) const {
    x = r.x[b];
    y = r.y[b];
    z = r.z[b];
    const double sg = r.sig[b], ep = r.eps[b];
    const bool real = sg >= 0 && ep >= 0;
    sb = real ? sg : -1.0;
    eb = real && mcgpu::bits_nonzero(ep) ? sqrt(ep) : 0.0;
    qb = r.q[b];
  }
};

// FP32 primary screen of the rows: distances decided outright below lo and
// above hi (squared), by the FP64 test between; rows farther than `far` from
// the origin along an axis always by the FP64 test.
struct StaticScreen {
  float L[3], lo, hi, far;
};

// Minimum-image distance squared as makePeriodic's single shift gives it.
__device__ __forceinline__ float screen2(float3 a, float3 b, const float* L) {
  float d[3] = {fabsf(b.x - a.x), fabsf(b.y - a.y), fabsf(b.z - a.z)};
#pragma unroll
  for (int k = 0; k < 3; k++) d[k] = d[k] > 0.5f * L[k] ? fabsf(d[k] - L[k]) : d[k];
  return fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2]));
}

// E(m, j > m) of the molecules [blockIdx.x * group, ...) of a CTA into
// emol[blockIdx.x]: the reference's primary-pair cutoff
// (SimulationStep.cpp:317-330; FP32 outside the guard band) and FP64 pair
// terms (BruteForceStep.cpp:48-79, SimulationStep.cpp:344-375), as pairsum.cuh
// describes; molecules of more than kMaxA atoms pass by in chunks of their
// atoms.  A molecule with out-of-range rows makes the partial NaN instead of
// reading past them.  1,999 molecules of 16 atoms (rc 12 A, 11.5 M pairs):
// 0.60 ms, the FP64 pipe 78 % busy; 12.0 ms when each thread took a whole in-range candidate, its square root
// and division per pair included.
__global__ void __launch_bounds__(mcgpu::kPsThreads, 4)
    k_static_pair_sums(Rows r, StaticScreen sc, int group, double* emol) {
  using namespace mcgpu;
  __shared__ PsGroup G;
  __shared__ int ms[kPsGroup], ml[kPsGroup], p0[kPsGroup], pc[kPsGroup], pa[kPsGroup];
  __shared__ float3 pf[kPsGroup];
  __shared__ int near[kPsGroup];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  const int m0 = (int)blockIdx.x * group, n = min(group, r.n_mol - m0);
  bool bad = false;
  if ((int)threadIdx.x < n) {
    const int g = threadIdx.x, m = m0 + g;
    const bool ok = valid_mol(r, m);
    bad = !ok;
    ms[g] = ok ? r.mstart[m] : 0;
    ml[g] = ok ? r.mlen[m] : 0;
    p0[g] = ok ? r.mps[m] : 0;
    pc[g] = ok ? r.mpc[m] : 0;
    const int a = pc[g] > 0 ? r.pidx[p0[g]] : -1;
    pa[g] = a;
    float3 f = make_float3(0.f, 0.f, 0.f);
    bool nr = false;
    if (a >= 0 && a < r.n_atom) {
      f = make_float3((float)r.x[a], (float)r.y[a], (float)r.z[a]);
      nr = fabsf(f.x) <= sc.far && fabsf(f.y) <= sc.far && fabsf(f.z) <= sc.far;
    }
    pf[g] = f;
    near[g] = nr;
  }
  __syncthreads();
  int longest = 0;
  for (int g = 0; g < n; g++) longest = max(longest, ml[g]);
  const double rc2 = __dmul_rn(r.cutoff, r.cutoff);
  int* rj = G.ring[w];
  double acc = 0.0;
  for (int c0 = 0; c0 < longest; c0 += kMaxA) {
    for (int g = 0; g < n; g++) {
      const int len = max(0, min(kMaxA, ml[g] - c0));
      for (int i = threadIdx.x; i < len; i += kPsThreads) {
        const int o = g * kPsPitch + i;
        StaticRows{r}.atom(ms[g] + c0 + i, G.x[o], G.y[o], G.z[o], G.sd[o], G.ed[o], G.qd[o]);
      }
      if (threadIdx.x == 0) G.len[g] = len;
    }
    __syncthreads();
    const bool alike = ps_alike(G, n);
    int head = 0, tail = 0;
    for (int base = m0 + 1 + w * 32; base < r.n_mol; base += kPsThreads) {
      const int j = base + lane;
      int q0 = 0, qc = 0, qa = -1;
      float3 f = make_float3(0.f, 0.f, 0.f);
      bool nr = false;
      if (j < r.n_mol) {
        if (valid_mol(r, j)) {
          q0 = r.mps[j];
          qc = r.mpc[j];
          qa = qc > 0 ? r.pidx[q0] : -1;
          if (qa >= 0 && qa < r.n_atom) {
            f = make_float3((float)r.x[qa], (float)r.y[qa], (float)r.z[qa]);
            nr = fabsf(f.x) <= sc.far && fabsf(f.y) <= sc.far && fabsf(f.z) <= sc.far;
          }
        } else {
          bad = true;
        }
      }
      for (int g = 0; g < n; g++) {
        bool in = false;
        if (j > m0 + g && G.len[g] > 0)
          for (int k1 = 0; k1 < pc[g] && !in; k1++)
            for (int k2 = 0; k2 < qc && !in; k2++) {
              const int a1 = k1 == 0 ? pa[g] : r.pidx[p0[g] + k1];
              const int a2 = k2 == 0 ? qa : r.pidx[q0 + k2];
              if (a1 < 0 || a1 >= r.n_atom || a2 < 0 || a2 >= r.n_atom) {
                bad = true;
                break;
              }
              bool exact = true;
              if (k1 == 0 && k2 == 0 && nr && near[g]) {
                const float r2 = screen2(pf[g], f, sc.L);
                in = r2 <= sc.lo;
                exact = !in && r2 <= sc.hi;
              }
              if (exact) in = dist2(r, a1, a2) <= rc2;
            }
        const unsigned bal = __ballot_sync(~0u, in);
        if (bal == 0) continue;
        if (in) rj[(tail + __popc(bal & lt)) & (kRing - 1)] = (j << 3) | g;
        tail += __popc(bal);
        if (tail - head >= 32) {
          __syncwarp();
          acc += ps_items<true>(G, StaticRows{r}, rj, head, 32, lane, alike, r.L[0], r.L[1],
                                 r.L[2]);
          head += 32;
          __syncwarp();
        }
      }
    }
    __syncwarp();
    if (tail > head)
      acc += ps_items<true>(G, StaticRows{r}, rj, head, tail - head, lane, alike, r.L[0], r.L[1],
                             r.L[2]);
    __syncthreads();   // the next atoms overwrite the stage
  }
  const double sum = ps_block_sum(G, bad ? __longlong_as_double(0x7ff8000000000000LL) : acc);
  if (threadIdx.x == 0) emol[blockIdx.x] = sum;
}

// Ordered sum of the partials into *out (thread t adds every blockDim-th
// term from t, then a fixed tree).
__global__ void k_static_sum(const double* emol, int n, double* out) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += emol[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int off = blockDim.x >> 1; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

mcgpu::ScratchAddressCache<kMaxDevices> g_emol_cache;  // device address of the scratch

int fail(int code, const char* msg) {
  mcgpu::note_process_error(msg);
  return code;
}

// Id of the calling thread's current context (0 if none or unknown), through
// the driver's cuCtxGetCurrent / cuCtxGetId fetched from the runtime (no link
// against the driver library).
typedef int (*PfnCtxGetCurrent)(void**);
typedef int (*PfnCtxGetId)(void*, unsigned long long*);

unsigned long long current_context_id() {
  static std::once_flag once;
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_current = (PfnCtxGetCurrent)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_id = (PfnCtxGetId)f;
  });
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx) return 0;
  if (get_id(ctx, &id) != 0) return 0;
  return id;
}

}  // namespace

extern "C" int mcgpu_system_energy_static(const mcgpu_box_desc* rows, double* out, void* stream) {
  if (!rows || !out) return fail(MCGPU_ERR_INVALID, "null argument");
  if (rows->n_mol <= 0 || rows->n_atom <= 0 || rows->n_pidx <= 0)
    return fail(MCGPU_ERR_INVALID, "empty box");
  if (rows->n_mol > kStaticMaxMol)
    return fail(MCGPU_ERR_UNSUPPORTED,
                "mcgpu_system_energy_static: more than 32768 molecules (its fixed scratch holds "
                "one partial per molecule); use mcgpu_system_energy");
  if (!rows->x || !rows->y || !rows->z || !rows->sigma || !rows->epsilon || !rows->charge ||
      !rows->mol_start || !rows->mol_len || !rows->mol_pidx_start || !rows->mol_pidx_count ||
      !rows->pidx)
    return fail(MCGPU_ERR_INVALID, "null row pointer");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(MCGPU_ERR_CUDA, "no current CUDA device");
  double* emol = (double*)g_emol_cache.get(
      dev, current_context_id(),
      [](void** p) { return cudaGetSymbolAddress(p, g_static_emol) == cudaSuccess; },
      [] { return current_context_id(); });
  if (!emol) return fail(MCGPU_ERR_CUDA, "cudaGetSymbolAddress of the static scratch failed");
  Rows r;
  r.x = rows->x; r.y = rows->y; r.z = rows->z;
  r.sig = rows->sigma; r.eps = rows->epsilon; r.q = rows->charge;
  r.mstart = rows->mol_start; r.mlen = rows->mol_len;
  r.mps = rows->mol_pidx_start; r.mpc = rows->mol_pidx_count; r.pidx = rows->pidx;
  r.n_mol = rows->n_mol; r.n_atom = rows->n_atom; r.n_pidx = rows->n_pidx;
  for (int k = 0; k < 3; k++) r.L[k] = rows->size[k];
  r.cutoff = rows->cutoff;
  cudaStream_t st = (cudaStream_t)stream;
  // An error the caller's own code left pending stays the caller's: it is
  // neither cleared nor reported as this call's.
  const cudaError_t prior = cudaPeekAtLastError();
  auto launch_error = [prior]() {
    const cudaError_t e = prior == cudaSuccess ? cudaGetLastError() : cudaPeekAtLastError();
    return e == prior ? cudaSuccess : e;
  };
  // FP32 coordinates within 2 edges of the origin carry at most 2 L 2^-24
  // each; with the difference's and the image's rounding at most 10 L 2^-24
  // along an axis; the band around rc^2 is four times what that makes of r^2
  StaticScreen sc;
  double Lmax = 0;
  for (int k = 0; k < 3; k++) {
    sc.L[k] = (float)r.L[k];
    Lmax = std::fmax(Lmax, std::fabs(r.L[k]));
  }
  const double err = 10.0 * std::ldexp(Lmax, -24);
  const double band = 4.0 * (2.0 * 1.7320508075688772 * std::fabs(r.cutoff) * err + 3.0 * err * err +
                             4.0 * std::ldexp(r.cutoff * r.cutoff, -24)) + 1e-6;
  sc.lo = (float)(r.cutoff * r.cutoff - band);
  sc.hi = (float)(r.cutoff * r.cutoff + band);
  sc.far = (float)(2.0 * Lmax);
  const int group = mcgpu::ps_group(r.n_mol, mcgpu::kPsPerBox), grid = (r.n_mol + group - 1) / group;
  k_static_pair_sums<<<grid, mcgpu::kPsThreads, 0, st>>>(r, sc, group, emol);
  cudaError_t e = launch_error();
  if (e == cudaSuccess) {
    k_static_sum<<<1, 256, 0, st>>>(emol, grid, out);
    e = launch_error();
  }
  if (e != cudaSuccess) {
    static thread_local char msg[256];
    snprintf(msg, sizeof(msg), "mcgpu_system_energy_static: launch failed: %s",
             cudaGetErrorString(e));
    return fail(MCGPU_ERR_CUDA, msg);
  }
  return MCGPU_OK;
}
