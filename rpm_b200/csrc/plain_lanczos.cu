// FP64 Lanczos with two classical Gram-Schmidt passes
// (rpm_statevector_engine.py:651-688), one launch per basis.
//
// The per-iteration launch sequence spent its time in launches, in last-block
// sums and in kernels of a few blocks (the full system: 170 us per vector at
// 24 basis vectors on average, of which 46 us at the HBM rate).  Here the
// blocks of one cooperative launch (one per SM, fewer for small states) own
// the nuclear indices [g0, g0 + ng) with all four electron components for the
// whole build:
//   * the block's slice of w lives in shared memory, and the slices of the
//     first basis vectors as far as shared memory goes (all of them up to
//     about 14,000 components, 7 of 40 for the full system's 221,184); the
//     others are the block's own and come from L1/L2;
//   * iteration j: w <- H v_j by the direct H psi on the unscaled previous w
//     (v_j = w / beta is formed and stored on the way), h = V^H w over
//     v_0 .. v_j (alpha_j = Re h_j), barrier; w -= V h and again h = V^H w,
//     barrier; w -= V h, |w|^2, barrier.
// The first projection contains alpha_j v_j and beta_(j-1) v_(j-1), so the
// three-term subtraction and the first Gram-Schmidt pass are one; the second
// pass restores orthogonality to rounding as in the reference ("twice is
// enough").  Sums are deterministic: warp butterflies, the four electron
// components in order, blocks in lane-strided order.  Every block reads the
// partials of all blocks after a barrier (no last block), and the barriers
// have a time limit, after which the launch sets `timeout` and ends.
#include <algorithm>
#include <mutex>
#include <vector>

#include "hpsi.cuh"
#include "hpsi_direct.cuh"
#include "krylov.cuh"
#include "plain_lanczos.cuh"
#include "ptx.cuh"

namespace rpm {
namespace {

using direct::HRec;
using direct::Tables;

constexpr int kPT = 512;                    // threads per block
constexpr int kPW = kPT / 32;
constexpr int kMinGroups = 128;             // nuclear indices per block before a second block is used
constexpr size_t kDynamicLimit = 208 * 1024;  // dynamic shared memory beside about 14 KB static

struct PlainBasis {
  const CubeView<double2>* view;
  direct::Args<double2> tables;
  const double2* state;
  double2* basis;
  long long n;
  int groups, gpb, m, kc, tabs, lrecs;  // kc: basis slices in shared memory
  double tol;
  double *alpha, *beta;
  double2* wbuf[2];
  double2* part;  // two regions of RPM_MAX_KRYLOV x gridDim.x partial sums
  LanczosScalars* sc;
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// All blocks of the (cooperative) launch; false after the time limit.
__device__ bool grid_barrier(LanczosScalars* sc, unsigned target) {
  __shared__ int ok;
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&sc->barrier, 1u);
    const long long t0 = clock64();
    ok = 1;
    for (int spin = 0; ld_acquire(&sc->barrier) < target; ++spin) {
      if ((spin & 63) == 63 &&
          (*reinterpret_cast<volatile int*>(&sc->timeout) || clock64() - t0 > ptx::kWaitCycles)) {
        atomicExch(&sc->timeout, 1);
        ok = 0;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// h[k] = sum over blocks of part[k * G + block], k < count.
__device__ __forceinline__ void gather(const double2* part, int count, double2* h) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
  for (int k = warp; k < count; k += kPW) {
    double2 s = make_double2(0.0, 0.0);
    for (int b = lane; b < G; b += 32) s = cadd(s, __ldcg(part + (size_t)k * G + b));
    s.x = warp_sum(s.x);
    s.y = warp_sum(s.y);
    if (lane == 0) h[k] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kPT, 1) k_plain_basis(const PlainBasis p) {
  __shared__ Tables tb;
  __shared__ double2 red[RPM_MAX_KRYLOV][4];
  __shared__ double2 h[RPM_MAX_KRYLOV];
  __shared__ double2 scratch[kPW];
  __shared__ double2 tot[1];
  extern __shared__ __align__(16) unsigned char raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
  const int g0 = blockIdx.x * p.gpb, ng = min(p.gpb, p.groups - g0);
  const long long q = p.groups;
  const int hr = p.view->half_r;
  const int l0 = g0 / hr;
  double2* tab = reinterpret_cast<double2*>(raw);
  HRec* lrec = reinterpret_cast<HRec*>(tab + p.tabs);
  HRec* rrec = lrec + p.lrecs;
  double2* w = reinterpret_cast<double2*>(rrec + hr);  // [e][gpb]
  double2* vc = w + 4 * p.gpb;                         // [k][e][gpb]
  direct::load_tables(p.tables, tb, tab);
  {
    const double2* ls = reinterpret_cast<const double2*>(static_cast<const HRec*>(p.view->lrec) + l0);
    const double2* rs = static_cast<const double2*>(p.view->rrec);
    constexpr int U = sizeof(HRec) / sizeof(double2);
    const int nl = min(p.lrecs, p.view->half_l - l0);
    for (int k = tid; k < nl * U; k += kPT) reinterpret_cast<double2*>(lrec)[k] = ls[k];
    for (int k = tid; k < hr * U; k += kPT) reinterpret_cast<double2*>(rrec)[k] = rs[k];
  }
  unsigned gen = 0;
  bool alive = true;
  // partial sums of this block -> totals of all blocks, in h[0, count); false: a barrier gave up
  auto reduce_all = [&](int count) {
    if (!grid_barrier(p.sc, (gen + 1) * (unsigned)G)) return false;
    gather(p.part + (size_t)(gen & 1) * RPM_MAX_KRYLOV * G, count, h);
    ++gen;
    return true;
  };
  auto region = [&]() { return p.part + (size_t)(gen & 1) * RPM_MAX_KRYLOV * G; };
  // |w|^2 of the block's slice as the only partial
  auto put_norm = [&](double nn) {
    double2 acc[1] = {make_double2(nn, 0.0)};
    block_sum2<1>(acc, scratch, tot);
    if (tid == 0) region()[blockIdx.x] = tot[0];
  };
  // partials <v_k, w> for k0 <= k <= k1 (slot k - k0): one warp per vector and electron component
  auto put_dots = [&](int k0, int k1) {
    __syncthreads();
    for (int u = warp; u < 4 * (k1 - k0 + 1); u += kPW) {
      const int k = k0 + (u >> 2), e = u & 3;
      const double2* we = w + e * p.gpb;
      double2 a0 = make_double2(0.0, 0.0), a1 = a0;
      auto run = [&](const double2* v) {
        int gl = lane;
#pragma unroll 2
        for (; gl + 32 < ng; gl += 64) {
          a0 = cfma_conj(v[gl], we[gl], a0);
          a1 = cfma_conj(v[gl + 32], we[gl + 32], a1);
        }
        if (gl < ng) a0 = cfma_conj(v[gl], we[gl], a0);
      };
      if (k < p.kc) run(vc + ((size_t)k * 4 + e) * p.gpb);
      else run(p.basis + (size_t)k * p.n + e * q + g0);
      a0 = cadd(a0, a1);
      a0.x = warp_sum(a0.x);
      a0.y = warp_sum(a0.y);
      if (lane == 0) red[k - k0][e] = a0;
    }
    __syncthreads();
    if (tid <= k1 - k0)
      region()[(size_t)tid * G + blockIdx.x] = cadd(cadd(red[tid][0], red[tid][1]), cadd(red[tid][2], red[tid][3]));
  };
  // w -= sum_{k <= j} h_k v_k; returns this thread's |w|^2
  auto axpy = [&](int j, double2* store) {
    double nn = 0.0;
    for (int gl = tid; gl < ng; gl += kPT) {
      double2 s[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = make_double2(0.0, 0.0);
      const int ks = min(p.kc, j + 1);
      const double2* v = vc + gl;
      for (int k = 0; k < ks; ++k, v += 4 * p.gpb)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = cfma(v[e * p.gpb], h[k], s[e]);
      const double2* b = p.basis + (size_t)ks * p.n + g0 + gl;
#pragma unroll 4
      for (int k = ks; k <= j; ++k, b += p.n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = cfma(b[e * q], h[k], s[e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        double2 x = w[e * p.gpb + gl];
        x.x -= s[e].x;
        x.y -= s[e].y;
        w[e * p.gpb + gl] = x;
        if (store) store[g0 + gl + e * q] = x;
        nn = fma(x.x, x.x, fma(x.y, x.y, nn));
      }
    }
    return nn;
  };

  double nn = 0.0;
  for (int gl = tid; gl < ng; gl += kPT)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double2 x = p.state[g0 + gl + e * q];
      w[e * p.gpb + gl] = x;
      nn = fma(x.x, x.x, fma(x.y, x.y, nn));
    }
  put_norm(nn);
  alive = reduce_all(1);
  double size = sqrt(h[0].x);  // ||state||, then beta_{j-1}
  if (alive) {
    const bool zero = !(size > 0.0);
    if (blockIdx.x == 0 && tid == 0) {
      p.sc->norm = size;
      p.sc->stop = zero ? -1 : 0;
    }
    alive = !zero;
  }
  for (int j = 0; alive && j < p.m; ++j) {
    const double inv = 1.0 / size;
    const double2* src = (j == 0 ? p.state : p.wbuf[(j - 1) & 1]) + g0;
    double2* vj = p.basis + (size_t)j * p.n + g0;
    for (int gl = tid; gl < ng; gl += kPT) {
      const int l = (g0 + gl) / hr, r = g0 + gl - l * hr;
      double2 x[4], o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = w[e * p.gpb + gl];
      direct::apply_group(
          tb, tab, lrec[l - l0], rrec[r], x,
          [&](int delta, double2(&y)[4]) {
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = src[e * q + gl + delta];
          },
          o);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double2 v = make_double2(x[e].x * inv, x[e].y * inv);
        vj[e * q + gl] = v;
        if (j < p.kc) vc[((size_t)j * 4 + e) * p.gpb + gl] = v;
        w[e * p.gpb + gl] = make_double2(o[e].x * inv, o[e].y * inv);
      }
    }
    const bool last = j == p.m - 1;
    put_dots(last ? j : 0, j);
    if (!(alive = reduce_all(last ? 1 : j + 1))) break;
    if (blockIdx.x == 0 && tid == 0) p.alpha[j] = h[last ? 0 : j].x;
    if (last) break;
    axpy(j, nullptr);
    put_dots(0, j);
    if (!(alive = reduce_all(j + 1))) break;
    put_norm(axpy(j, p.wbuf[j & 1]));
    if (!(alive = reduce_all(1))) break;
    size = sqrt(h[0].x);
    if (blockIdx.x == 0 && tid == 0) {
      p.beta[j] = size;
      if (size <= p.tol) p.sc->stop = j + 1;
    }
    if (size <= p.tol) break;
    __syncthreads();  // h is read by every thread before the next gather
  }
  // the barrier counter is back at zero for the next launch
  __syncthreads();
  if (tid == 0 && G > 1) {
    __threadfence();
    if (atomicAdd(&p.sc->exits, 1u) == (unsigned)G - 1) {
      p.sc->exits = 0;
      p.sc->barrier = 0;
    }
  }
}

}  // namespace

bool launch_plain_basis(rpm_system* sys, const double2* state, int m, double tol, double2* basis, double* alpha,
                        double* beta, LanczosScalars* sc, cudaStream_t stream) {
  if (!direct_usable(sys)) return false;
  PlainBasis p{};
  p.groups = (int)(sys->n / 4);
  // one block per SM, but no block under kMinGroups nuclear indices: a grid
  // barrier costs about as much as 128 indices' work per stage
  const int want = std::max(1, std::min(sm_count(), p.groups / kMinGroups));
  p.gpb = (p.groups + want - 1) / want;
  const int G = (p.groups + p.gpb - 1) / p.gpb;
  p.tabs = sys->cube_l.ntab + sys->cube_r.ntab;
  p.lrecs = std::min(sys->half_l, (p.gpb - 1) / sys->half_r + 2);
  const size_t fixed = sizeof(double2) * (size_t)p.tabs + sizeof(HRec) * (size_t)(p.lrecs + sys->half_r) +
                       sizeof(double2) * 4 * (size_t)p.gpb;
  if (fixed > kDynamicLimit) return false;
  p.kc = (int)std::min<size_t>((size_t)m, (kDynamicLimit - fixed) / (sizeof(double2) * 4 * (size_t)p.gpb));
  const size_t smem = fixed + sizeof(double2) * 4 * (size_t)p.gpb * p.kc;
  {
    static std::mutex mu;
    static std::vector<int> done;  // devices with the attribute set
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(mu);
    if (std::find(done.begin(), done.end(), dev) == done.end()) {
      check_cuda(cudaFuncSetAttribute(k_plain_basis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynamicLimit),
                 "plain basis smem attr");
      done.push_back(dev);
    }
  }
  p.view = sys->cube64_dev;
  p.tables = direct::make_args(sys->cube64, sys->cube64_dev);
  p.state = state;
  p.basis = basis;
  p.n = sys->n;
  p.m = m;
  p.tol = tol;
  p.alpha = alpha;
  p.beta = beta;
  auto* wb = static_cast<double2*>(system_scratch(sys, SLOT_WORK, sizeof(double2) * 2 * (size_t)sys->n));
  p.wbuf[0] = wb;
  p.wbuf[1] = wb + sys->n;
  p.part = static_cast<double2*>(system_scratch(sys, SLOT_REDUCE, sizeof(double2) * 2 * RPM_MAX_KRYLOV * (size_t)G));
  p.sc = sc;
  if (G == 1) {
    k_plain_basis<<<1, kPT, smem, stream>>>(p);
    check_launch("k_plain_basis");
  } else {
    void* args[] = {&p};
    check_cuda(cudaLaunchCooperativeKernel(k_plain_basis, dim3(G), dim3(kPT), args, smem, stream), "k_plain_basis");
  }
  return true;
}

}  // namespace rpm
