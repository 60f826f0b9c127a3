// Direct FP64 H psi (see hpsi_direct.cuh): one launch, no scratch.
#include "hpsi_direct.cuh"

namespace rpm {
namespace {

// Bound by the load / store pipe (61 % of its wavefronts at 28 % occupancy, FP64
// pipe 32 %, DRAM 6 %: ncu, 8 vectors of 221,184).  Six blocks of 128 threads
// per SM (80 registers): 171 us for 32 vectors; before the tables came by
// argument 181, against 187 us at 92 registers and 202 us at 64, which spills.
constexpr int kDirectThreads = 128;
constexpr int kPairBlocks = 296;

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


// Two vectors per thread: partner arithmetic and coefficients, half of the load
// / store pipe's work on the right radical (its lanes' digits differ), serve
// both.  The order of additions is the one-vector kernel's, a sum per radical:
// a vector's result does not depend on its neighbours.  Four blocks per SM (128
// registers): 221,184 x 2, 8, 32 12.9, 38.0, 142 us, against 14.1, 46.5, 171 by
// single vectors.  One sum for both radicals fits five blocks (131 us for 32)
// but rounds 7 to 13 % more.
__global__ void __launch_bounds__(kDirectThreads, 4) k_hpsi_direct2(const direct::Args<double2> a,
                                                               const double2* __restrict__ in,
                                                               double2* __restrict__ out, int groups, int batch,
                                                               long long ld, const double* __restrict__ scale) {
  using namespace direct;
  __shared__ Tables tb;
  extern __shared__ double2 tab[];
  const int g = blockIdx.x * kDirectThreads + threadIdx.x;
  const int l = g / a.hr, r = g - l * a.hr;
  load_tables(a, tb, tab);
  if (g >= groups) return;
  const long long q = groups;
  // the last vector of an odd batch is read twice and written once
  const int b0 = 2 * blockIdx.y, count = min(2, batch - b0);
  const long long second = count == 2 ? ld : 0;
  const HRec lr = static_cast<const HRec*>(a.lrec)[l];
  const HRec* rrp = static_cast<const HRec*>(a.rrec) + r;
  const unsigned long long rdig = rrp->digits;
  const double2* v = in + (long long)b0 * ld + g;
  // a sum per radical, added to the local part in apply_group's order
  double2 acc[2][2][4];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[side][i][e] = make_double2(0.0, 0.0);
    const unsigned long long digits = side ? rdig : lr.digits;
    const int np = tb.np[side];
    for (int p = 0; p < np; ++p) {
      const int4 raw = *reinterpret_cast<const int4*>(&tb.part[side][p]);
      Partner t;
      memcpy(&t, &raw, sizeof(t));
      const int m = (int)(digits >> t.shift) & 15;
      int mp = m + t.t;
      if (mp >= t.d) mp -= t.d;
      const double2* cf = tab + t.offx + m * 2 * t.d + mp;
      const int d = t.d, delta = (mp - m) * t.stride;
      const double2 c00 = cf[0], c01 = cf[d], c10 = cf[2 * d * d], c11 = cf[2 * d * d + d];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        double2 y[4];
        double2(&o)[4] = acc[side][i];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = v[i * second + e * q + delta];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int i0 = side ? 2 * s : s, i1 = side ? 2 * s + 1 : 2 + s;
          o[i0] = cfma(c01, y[i1], cfma(c00, y[i0], o[i0]));
          o[i1] = cfma(c11, y[i1], cfma(c10, y[i0], o[i1]));
        }
      }
    }
  }
  const HRec rr = *rrp;
  const double s = scale ? *scale : 1.0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    double2 x[4], z[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = v[i * second + e * q];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const double dg = lr.d[b] + rr.d[c];
        double2 u = make_double2(dg * x[2 * b + c].x, dg * x[2 * b + c].y);
        u = cfma(lr.f[b], x[2 * (1 - b) + c], u);
        z[2 * b + c] = cfma(rr.f[c], x[2 * b + 1 - c], u);
      }
    if (tb.has_pair) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < 4; ++c) z[e] = cfma(tb.pair[4 * e + c], x[c], z[e]);
    }
    if (i >= count) break;
    double2* w = out + (long long)(b0 + i) * ld + g;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double2 t = cadd(cadd(z[e], acc[0][i][e]), acc[1][i][e]);
      w[e * q] = make_double2(s * t.x, s * t.y);
    }
  }
}

}  // namespace

bool direct_usable(const rpm_system* sys) { return sys->cube && sys->cube64.lrec && sys->cube64.rrec; }

void launch_direct(rpm_system* sys, const double2* in, double2* out, int batch, long long ld, const double* scale_dev,
                   cudaStream_t stream) {
  const int groups = (int)(sys->n / 4);
  const size_t smem = sizeof(double2) * (size_t)(sys->cube_l.ntab + sys->cube_r.ntab);
  const int gx = (groups + kDirectThreads - 1) / kDirectThreads;
  // Pairs where they still make two blocks per SM.  Pairs against single
  // vectors, us: 3,456 x 64 7.7 / 8.0, x 128 11.1 / 13.0; 13,824 x 9 7.8 / 7.6,
  // x 16 9.1 / 8.8, x 22 (the line) 10.3 / 10.8, x 32 11.0 / 12.3; 55,296 x 4
  // 9.7 / 9.6, x 6 11.4 / 11.7, x 7 11.7 / 12.9; 221,184 x 2 12.9 / 14.1, x 4
  // 22.7 / 25.1, x 5 31.3 / 31.2, x 17 83 / 94; three vectors waste a quarter
  // of the work: 21.3 / 20.8.
  if (batch != 3 && (long long)gx * (batch / 2) >= kPairBlocks) {
    k_hpsi_direct2<<<dim3(gx, (batch + 1) / 2), kDirectThreads, smem, stream>>>(
        direct::make_args(sys->cube64, sys->cube64_dev), in, out, groups, batch, ld, scale_dev);
    check_launch("k_hpsi_direct2");
    return;
  }
  k_hpsi_direct<<<dim3(gx, batch), kDirectThreads, smem, stream>>>(
      direct::make_args(sys->cube64, sys->cube64_dev), in, out, groups, ld, scale_dev);
  check_launch("k_hpsi_direct");
}

}  // namespace rpm
