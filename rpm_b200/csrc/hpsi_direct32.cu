// Direct complex64 H psi for rpm_hpsi: one launch, no scratch.
//
// As the complex128 direct form (hpsi_direct.cuh), with two neighbouring right
// indices per thread: the fastest right nucleus is a spin-1/2, so its partner
// is in registers, a 16-byte load brings both values of any other partner, and
// every coefficient serves eight outputs.  The two shape-specialised passes
// that the batched propagation uses (their order of additions is part of its
// results) move a partial result through memory and take two launches, the
// second behind the first.  Two passes -> this kernel, microseconds:
//   864 x 64           13.2 ->   4.9
//   13,824 x 1          9.3 ->   6.3
//   55,296 x 8         13.6 ->   9.1
//   221,184 x 1, 4, 8  21.9, 22.2, 33.5 -> 8.3, 13.5, 23.2
//   221,184 x 48        146 -> 112
// Bound by the load/store unit (each component is read once per partner, from
// L1 and L2).  Six blocks of 128 threads per SM: 129 us before the tables came
// by argument; then at five 136 us, at four 145, at seven 133, at eight 138; 64
// threads 139, 256 threads 131.
#include "hpsi_direct.cuh"

#include <cstring>

namespace rpm {
namespace direct {

struct HRec32 {
  float d[2];
  float2 f[2];
  unsigned long long digits;
};

}  // namespace direct

namespace {

using direct::HRec32;
using direct::kMaxPartners;
using direct::Partner;

constexpr int kThreads32 = 128;
// Two vectors per thread share coefficients and partner arithmetic, where they
// still make 2.5 blocks per SM.  Pairs against single vectors, us: 13,824 x 32
// 9.5 / 9.2; 55,296 x 8 10.3 / 9.2, x 32 22.2 / 22.7; 221,184 x 2 10.9 / 9.8,
// x 4 (432 blocks) 13.5 / 14.2, x 17 46.0 / 46.6, x 48 112.6 / 122.4.  Four
// blocks per SM (three 122 us, five spill).
constexpr int kPairBlocks32 = 370;

using direct::Args;
using Tables32 = direct::TablesOf<float2>;  // the right partners without the fastest nucleus's

template <int NV, int RES>
__global__ void __launch_bounds__(kThreads32, RES) k_hpsi_direct32(const Args<float2> ar,
                                                                const float2* __restrict__ in,
                                                                float2* __restrict__ out, int pairs, int batch,
                                                                long long ld, int off_fast) {
  __shared__ Tables32 tb;
  extern __shared__ float2 tab32[];
  const int idx = blockIdx.x * kThreads32 + threadIdx.x;
  const int hr2 = ar.hr / 2;
  const int l = idx / hr2, r = 2 * (idx - l * hr2);
  load_tables(ar, tb, tab32);
  if (idx >= pairs) return;
  const float2* fast = tab32 + off_fast;  // block of the fastest right nucleus, (e, m) x (e', m')
  const long long q = 2LL * pairs;
  const HRec32 lr = static_cast<const HRec32*>(ar.lrec)[l];
  const HRec32* rp = static_cast<const HRec32*>(ar.rrec) + r;
  const unsigned long long rdigits = rp[0].digits;
  // the last vector of an odd batch is read twice and written once
  const int b0 = NV * blockIdx.y, count = min(NV, batch - b0);
  const long long second = count == 2 ? ld : 0;
  const float2* v = in + (long long)b0 * ld + 2LL * idx;
  auto load = [&](long long delta, float2 (&y)[4][2]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 u = *reinterpret_cast<const float4*>(v + e * q + delta);
      y[e][0] = make_float2(u.x, u.y);
      y[e][1] = make_float2(u.z, u.w);
    }
  };
  // o: left radical; w: right radical; z (last, its registers are free until
  // then): diagonal, left flip, pair operator.  Three short sums round less
  // than one: 1.05e-7 of the norm at 221,184 against 1.26e-7 by two passes.
  float2 o[NV][4][2], w[NV][4][2];
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int i = 0; i < 2; ++i) o[k][e][i] = w[k][e][i] = czero<float2>();
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const unsigned long long digits = side ? rdigits : lr.digits;
    const int np = tb.np[side];
#pragma unroll 2
    for (int p = 0; p < np; ++p) {
      const int4 raw = *reinterpret_cast<const int4*>(&tb.part[side][p]);
      Partner pt;
      memcpy(&pt, &raw, sizeof(pt));
      const int m = (int)(digits >> pt.shift) & 15;
      int mp = m + pt.t;
      if (mp >= pt.d) mp -= pt.d;
      const float2* cf = tab32 + pt.offx + m * 2 * pt.d + mp;
      const int d = pt.d;
      const float2 c00 = cf[0], c01 = cf[d], c10 = cf[2 * d * d], c11 = cf[2 * d * d + d];
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        float2(&acc)[4][2] = side ? w[k] : o[k];
        float2 y[4][2];
        load(k * second + (mp - m) * pt.stride, y);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int i0 = side ? 2 * s : s, i1 = side ? 2 * s + 1 : 2 + s;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            acc[i0][i] = cfma(c01, y[i1][i], cfma(c00, y[i0][i], acc[i0][i]));
            acc[i1][i] = cfma(c11, y[i1][i], cfma(c10, y[i0][i], acc[i1][i]));
          }
        }
      }
    }
  }
  const HRec32 r0 = rp[0], r1 = rp[1];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (k >= count) break;
    float2 x[4][2], z[4][2];
    load(k * second, x);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const HRec32& rr = i ? r1 : r0;
          const float dg = lr.d[a] + rr.d[b];
          const float2 xe = x[2 * a + b][i];
          float2 t = make_float2(dg * xe.x, dg * xe.y);
          z[2 * a + b][i] = cfma(lr.f[a], x[2 * (1 - a) + b][i], t);
          // the electron flip and the fastest nucleus belong to the right radical
          t = cfma(rr.f[b], x[2 * a + 1 - b][i], w[k][2 * a + b][i]);
          t = cfma(fast[(2 * b + i) * 4 + 1 - i], x[2 * a][1 - i], t);
          w[k][2 * a + b][i] = cfma(fast[(2 * b + i) * 4 + 2 + 1 - i], x[2 * a + 1][1 - i], t);
        }
    if (tb.has_pair) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 p = tb.pair[4 * e + c];
#pragma unroll
          for (int i = 0; i < 2; ++i) z[e][i] = cfma(p, x[c][i], z[e][i]);
        }
    }
    float2* dst = out + (long long)(b0 + k) * ld + 2LL * idx;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 u[2];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        u[i] = make_float2(z[e][i].x + (o[k][e][i].x + w[k][e][i].x), z[e][i].y + (o[k][e][i].y + w[k][e][i].y));
      *reinterpret_cast<float4*>(dst + e * q) = make_float4(u[0].x, u[0].y, u[1].x, u[1].y);
    }
  }
}

}  // namespace

bool direct32_usable(const rpm_system* sys, const float2* in, const float2* out, long long ld) {
  const auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  return sys->cube && sys->cube32.lrec && sys->cube32.rrec && ld % 2 == 0 && aligned(in) && aligned(out);
}

void launch_direct32(rpm_system* sys, const float2* in, float2* out, int batch, long long ld, cudaStream_t stream) {
  const int pairs = (int)(sys->n / 8);
  const size_t smem = sizeof(float2) * (size_t)(sys->cube_l.ntab + sys->cube_r.ntab);
  const int gx = (pairs + kThreads32 - 1) / kThreads32;
  const CubeSide& cr = sys->cube_r;
  const bool two = batch != 3 && (long long)gx * (batch / 2) >= kPairBlocks32;
  auto* kern = two ? k_hpsi_direct32<2, 4> : k_hpsi_direct32<1, 6>;
  kern<<<dim3(gx, two ? (batch + 1) / 2 : batch), kThreads32, smem, stream>>>(
      direct::make_args(sys->cube32, sys->cube32_dev), in, out, pairs, batch, ld,
      sys->cube_l.ntab + cr.offX[cr.K - 1]);
  check_launch("k_hpsi_direct32");
}

// Records of one radical from its complex128 table (sums in FP64, rounded once).
std::vector<unsigned char> direct32_records(const CubeSide& side, const std::vector<cd>& tab) {
  std::vector<unsigned char> out(sizeof(HRec32) * (size_t)side.half);
  for (int g = 0; g < side.half; ++g) {
    double d[2] = {tab[0].real(), tab[1].real()};
    cd f[2] = {tab[2], tab[3]};
    HRec32 r{};
    for (int k = 0; k < side.K; ++k) {
      const int m = (g / side.gs[k]) % side.dim[k];
      r.digits |= (unsigned long long)m << (4 * k);
      for (int e = 0; e < 2; ++e) {
        d[e] += tab[side.offD[k] + e * side.dim[k] + m].real();
        f[e] += tab[side.offF[k] + e * side.dim[k] + m];
      }
    }
    for (int e = 0; e < 2; ++e) {
      r.d[e] = (float)d[e];
      r.f[e] = make_float2((float)f[e].real(), (float)f[e].imag());
    }
    memcpy(out.data() + sizeof(HRec32) * (size_t)g, &r, sizeof(r));
  }
  return out;
}

}  // namespace rpm
