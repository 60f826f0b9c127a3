// Direct FP64 H psi (see hpsi_direct.cuh): one launch, no scratch.
#include "hpsi_direct.cuh"

namespace rpm {
namespace {

// Bound by the load / store pipe (61 % of its wavefronts at 28 % occupancy, FP64
// pipe 32 %, DRAM 6 %: ncu, 8 vectors of 221,184).  Six blocks of 128 threads
// per SM (80 registers): 173 us for 32 vectors; before the tables came by
// argument 181, against 187 us at 92 registers and 202 us at 64, which spills.
constexpr int kDirectThreads = 128;

__global__ void __launch_bounds__(kDirectThreads, 6) k_hpsi_direct(const direct::Args<double2> a,
                                                               const double2* __restrict__ in,
                                                               double2* __restrict__ out, int groups, long long ld,
                                                               const double* __restrict__ scale) {
  using namespace direct;
  __shared__ Tables tb;
  extern __shared__ double2 tab[];
  const int g = blockIdx.x * kDirectThreads + threadIdx.x;
  const int l = g / a.hr, r = g - l * a.hr;
  load_tables(a, tb, tab);
  if (g >= groups) return;
  const long long q = groups;
  const double s = scale ? *scale : 1.0;
  const HRec lr = static_cast<const HRec*>(a.lrec)[l];
  const HRec rr = static_cast<const HRec*>(a.rrec)[r];
  const double2* v = in + (long long)blockIdx.y * ld + g;
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
  const int gx = (groups + kDirectThreads - 1) / kDirectThreads;
  k_hpsi_direct<<<dim3(gx, batch), kDirectThreads, smem, stream>>>(
      direct::make_args(sys->cube64, sys->cube64_dev), in, out, groups, ld, scale_dev);
  check_launch("k_hpsi_direct");
}

}  // namespace rpm
