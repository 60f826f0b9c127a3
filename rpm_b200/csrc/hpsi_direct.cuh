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

template <class T>
struct TablesOf {
  int np[2];
  int has_pair, pad;
  Partner part[2][kMaxPartners];
  T pair[16];
};
using Tables = TablesOf<double2>;

// What a launch passes beside the device view, so that a block's first loads do
// not wait for one another.  Through the view (its sizes, then its pointers,
// then the tables; the partner lists built by each block) the direct H psi took
// 5.0 us at 864 x 64, 11.9 at 221,184 x 1, 183 at 221,184 x 32, now 4.1, 10.8
// and 173; staging the tables once for several vectors instead (a loop over the
// batch in each block) spills at 80 registers: 187 us.
template <class T>
struct Args {
  const CubeView<T>* view;
  const T *tab_l, *tab_r;
  const Partner* parts;
  const void *lrec, *rrec;
  int ntl, ntr, hr, np[2];
};

template <class T>
inline Args<T> make_args(const CubeView<T>& host, const CubeView<T>* dev) {
  return Args<T>{dev,       host.tabL,   host.tabR,   static_cast<const Partner*>(host.parts), host.lrec, host.rrec,
                 host.L.ntab, host.R.ntab, host.half_r, {host.parts_n[0], host.parts_n[1]}};
}

// Partner lists of both radicals ([2][kMaxPartners]); nuclei without
// transitions (a quadrupole system's spin-1/2 ones) have none.
inline std::vector<Partner> partner_lists(const CubeSide& l, const CubeSide& r, int half_r, unsigned moves_l,
                                          unsigned moves_r, int (&np)[2]) {
  std::vector<Partner> out(2 * kMaxPartners);
  for (int side = 0; side < 2; ++side) {
    const CubeSide& s = side ? r : l;
    int at = 0;
    for (int q = 0; q < s.K; ++q) {
      if (!(((side ? moves_r : moves_l) >> q) & 1u)) continue;
      for (int t = 1; t < s.dim[q]; ++t)
        out[side * kMaxPartners + at++] =
            Partner{(unsigned char)(4 * q), (unsigned char)t, (unsigned char)s.dim[q], 0,
                    s.gs[q] * (side ? 1 : half_r), s.offX[q] + (side ? l.ntab : 0), 0};
    }
    np[side] = at;
  }
  return out;
}

// Fills `tb` and stages both coefficient tables (left first) into `tab`; every
// thread of the block takes part.  Ends with a barrier.
template <class T>
__device__ __forceinline__ void load_tables(const Args<T>& a, TablesOf<T>& tb, T* tab) {
  for (int k = threadIdx.x; k < a.ntl; k += blockDim.x) tab[k] = a.tab_l[k];
  for (int k = threadIdx.x; k < a.ntr; k += blockDim.x) tab[a.ntl + k] = a.tab_r[k];
#pragma unroll
  for (int side = 0; side < 2; ++side)
    for (int k = threadIdx.x; k < a.np[side]; k += blockDim.x)
      reinterpret_cast<int4*>(tb.part[side])[k] = reinterpret_cast<const int4*>(a.parts + side * kMaxPartners)[k];
  bool any = false;
  if (threadIdx.x < 16) {
    const T p = a.view->pair[threadIdx.x];
    tb.pair[threadIdx.x] = p;
    any = p.x != 0 || p.y != 0;
  }
  if (threadIdx.x < 2) tb.np[threadIdx.x] = threadIdx.x ? a.np[1] : a.np[0];
  const int has = __syncthreads_or(any);
  if (threadIdx.x == 0) tb.has_pair = has;
  __syncthreads();
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
