// Device pieces of the direct H psi: one thread applies the whole Hamiltonian
// to the four electron-pair components of one nuclear index (l, r), reading
// its partners straight from the state.  Shared by the stand-alone kernel
// (hpsi_direct.cu) and the plain Lanczos kernel (plain_lanczos.cu).
//
// Systems: cube form (every radical term on {e}, {n_k} or {e, n_k}) in the
// standard layout psi[eA][eB][l][r] (rpm_statevector_engine.py:367-469), any
// spins.  Per radical group index a record holds the diagonal and electron-flip
// coefficients merged over the electron-only term and every nucleus, and the
// nuclear digits; a partner is one other value of one digit, with the 2 x 2
// electron block X_k[(e, m), (e', m')] of the cube table.
#pragma once

#include "common.cuh"
#include "hpsi.cuh"

namespace rpm {
namespace direct {

// Per group index of one radical (64 bytes; digits: four bits per nucleus).
struct HRec {
  double d[2];
  double2 f[2];
  unsigned long long digits, pad;
};

constexpr int kMaxPartners = 64;   // sum of (dimension - 1) over a radical's nuclei
constexpr int kMaxDigit = 16;      // largest nuclear dimension (four bits)
constexpr int kMaxTables = 1024;   // coefficients of both radicals staged in shared memory

// Partner t = 1 .. d - 1 of one nucleus: its value is (m + t) mod d.  One
// 16-byte shared-memory read: the load / store pipe is what bounds the kernel.
struct __align__(16) Partner {
  unsigned char shift, t, d, pad;
  int stride, offx, pad2;
};

struct Tables {
  int np[2];
  Partner part[2][kMaxPartners];
  double2 pair[16];
  int has_pair;
};

// Fills `tb` and stages both coefficient tables (left first) into `tab`;
// every thread of the block takes part, a barrier has to follow.
__device__ __forceinline__ void load_tables(const CubeView<double2>* view, Tables& tb, double2* tab) {
  const int nl = view->L.ntab;
  for (int k = threadIdx.x; k < nl; k += blockDim.x) tab[k] = view->tabL[k];
  for (int k = threadIdx.x; k < view->R.ntab; k += blockDim.x) tab[nl + k] = view->tabR[k];
  for (int k = threadIdx.x; k < 2 * kCubeMaxDigits; k += blockDim.x) {
    const int side = k / kCubeMaxDigits, q = k % kCubeMaxDigits;
    const CubeSide& s = side ? view->R : view->L;
    // nuclei without transitions (a quadrupole system's spin-1/2 ones) have no partners
    const unsigned moves = side ? view->moves_r : view->moves_l;
    if (q < s.K) {
      int at = 0;
      for (int p = 0; p < q; ++p) at += (moves >> p) & 1u ? s.dim[p] - 1 : 0;
      const int d = (moves >> q) & 1u ? s.dim[q] : 1;
      for (int t = 1; t < d; ++t)
        tb.part[side][at + t - 1] =
            Partner{(unsigned char)(4 * q), (unsigned char)t, (unsigned char)d, 0,
                    s.gs[q] * (side ? 1 : view->half_r), s.offX[q] + (side ? nl : 0), 0};
      if (q == s.K - 1) tb.np[side] = at + d - 1;
    }
  }
  if (threadIdx.x < 16) tb.pair[threadIdx.x] = view->pair[threadIdx.x];
  if (threadIdx.x == 0) {
    bool any = false;
    for (int k = 0; k < 16; ++k) any = any || view->pair[k].x != 0.0 || view->pair[k].y != 0.0;
    tb.has_pair = any ? 1 : 0;
  }
}

// out[2 eA + eB] = (H x)[eA, eB, l, r]; x: the thread's own components,
// load(delta, y): the four components of the nuclear index `delta` away.
template <class Load>
__device__ __forceinline__ void apply_group(const Tables& tb, const double2* tab, const HRec& lr, const HRec& rr,
                                            const double2 (&x)[4], Load load, double2 (&out)[4]) {
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const double dg = lr.d[a] + rr.d[b];
      double2 o = make_double2(dg * x[2 * a + b].x, dg * x[2 * a + b].y);
      o = cfma(lr.f[a], x[2 * (1 - a) + b], o);
      out[2 * a + b] = cfma(rr.f[b], x[2 * a + 1 - b], o);
    }
  if (tb.has_pair) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int c = 0; c < 4; ++c) out[e] = cfma(tb.pair[4 * e + c], x[c], out[e]);
  }
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const unsigned long long digits = side ? rr.digits : lr.digits;
    const int np = tb.np[side];
    // partner p + 1 is on its way while partner p is applied
    double2 y[4];
    auto fetch = [&](int p, double2 (&v)[4], const double2*& cf, int& d) {
      const int4 raw = *reinterpret_cast<const int4*>(&tb.part[side][p]);
      Partner q;
      memcpy(&q, &raw, sizeof(q));
      const int m = (int)(digits >> q.shift) & 15;
      int mp = m + q.t;
      if (mp >= q.d) mp -= q.d;
      cf = tab + q.offx + m * 2 * q.d + mp;
      d = q.d;
      load((mp - m) * q.stride, v);
    };
    // the radical's sum on its own: shorter rounding chains
    double2 acc[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] = make_double2(0.0, 0.0);
    const double2* cf = nullptr;
    int d = 0;
    if (np > 0) fetch(0, y, cf, d);
    for (int p = 0; p < np; ++p) {
      double2 z[4];
      const double2* cn = nullptr;
      int dn = 0;
      if (p + 1 < np) fetch(p + 1, z, cn, dn);
      const double2 c00 = cf[0], c01 = cf[d], c10 = cf[2 * d * d], c11 = cf[2 * d * d + d];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        // left: (eA, s) pairs; right: (s, eB) pairs
        const int i0 = side ? 2 * s : s, i1 = side ? 2 * s + 1 : 2 + s;
        acc[i0] = cfma(c01, y[i1], cfma(c00, y[i0], acc[i0]));
        acc[i1] = cfma(c11, y[i1], cfma(c10, y[i0], acc[i1]));
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) y[c] = z[c];
      cf = cn;
      d = dn;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) out[c] = cadd(out[c], acc[c]);
  }
}

}  // namespace direct

// Whether the direct FP64 H psi covers a system (standard layout, limits above).
bool direct_usable(const rpm_system* sys);
// out = H (in * scale) for `batch` vectors of one such system (scale_dev:
// null for 1).  No scratch.
void launch_direct(rpm_system* sys, const double2* in, double2* out, int batch, long long ld, const double* scale_dev,
                   cudaStream_t stream);
// The complex64 form (hpsi_direct32.cu): the same layout with a spin-1/2 as
// fastest right nucleus, 16-byte aligned pointers and an even stride.
bool direct32_usable(const rpm_system* sys, const float2* in, const float2* out, long long ld);
void launch_direct32(rpm_system* sys, const float2* in, float2* out, int batch, long long ld, cudaStream_t stream);
std::vector<unsigned char> direct32_records(const CubeSide& side, const std::vector<cd>& tab);

}  // namespace rpm
