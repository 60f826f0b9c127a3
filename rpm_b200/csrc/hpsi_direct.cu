// Direct FP64 H psi (see hpsi_direct.cuh): one launch, no scratch.
#include "hpsi_direct.cuh"

namespace rpm {
namespace {

// Bound by the load / store pipe (61 % of its wavefronts at 28 % occupancy, FP64
// pipe 32 %, DRAM 6 %: ncu, 8 vectors of 221,184).  Six blocks of 128 threads
// per SM (80 registers): 181 us for 32 vectors, against 187 us at 92
// registers and 202 us at 64, which spills.
constexpr int kDirectThreads = 128;

__global__ void __launch_bounds__(kDirectThreads, 6) k_hpsi_direct(const CubeView<double2>* __restrict__ view,
                                                               const double2* __restrict__ in,
                                                               double2* __restrict__ out, int groups, long long ld,
                                                               const double* __restrict__ scale) {
  using namespace direct;
  __shared__ Tables tb;
  extern __shared__ double2 tab[];
  load_tables(view, tb, tab);
  __syncthreads();
  const int g = blockIdx.x * kDirectThreads + threadIdx.x;
  if (g >= groups) return;
  const int hr = view->half_r;
  const int l = g / hr, r = g - l * hr;
  const HRec lr = static_cast<const HRec*>(view->lrec)[l];
  const HRec rr = static_cast<const HRec*>(view->rrec)[r];
  const double2* v = in + (long long)blockIdx.y * ld + g;
  const long long q = groups;
  double2 x[4], o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] = v[e * q];
  apply_group(
      tb, tab, lr, rr, x,
      [&](int delta, double2(&y)[4]) {
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = v[e * q + delta];
      },
      o);
  const double s = scale ? *scale : 1.0;
  double2* w = out + (long long)blockIdx.y * ld + g;
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e * q] = make_double2(s * o[e].x, s * o[e].y);
}

}  // namespace

bool direct_usable(const rpm_system* sys) { return sys->cube && sys->cube64.lrec && sys->cube64.rrec; }

void launch_direct(rpm_system* sys, const double2* in, double2* out, int batch, long long ld, const double* scale_dev,
                   cudaStream_t stream) {
  const int groups = (int)(sys->n / 4);
  const size_t smem = sizeof(double2) * (size_t)(sys->cube_l.ntab + sys->cube_r.ntab);
  k_hpsi_direct<<<dim3((groups + kDirectThreads - 1) / kDirectThreads, batch), kDirectThreads, smem, stream>>>(
      sys->cube64_dev, in, out, groups, ld, scale_dev);
  check_launch("k_hpsi_direct");
}

}  // namespace rpm
