// Lifetime sums of the factorized exact oracle (rpm_quantum_needle_reproduction.py:
// 172-240) from the radicals' eigensystems, all orientations of a call together:
//
//   k_spin_ops      S_p in the eigenbasis, p = x, y, z, of both radicals;
//   k_bin_lines9    the nine (p, q) transition spectra of both radicals;
//   k_fft_columns   forward FFT of the 18 rows, the bits from 11 up
//                   (decimation in frequency: no reordering pass);
//   k_convolve      per tile of 2,048 elements: the low bits of both radicals'
//                   rows, their products summed over the nine pairs, the low
//                   bits of the inverse transform (decimation in time, which
//                   takes the order that the forward one leaves);
//   k_fft_columns   inverse, the bits from 11 up;
//   k_yield_sums    sum of conv x 1 and conv x k / (k - i w).
//
// What this replaces per orientation: seven small launches per spin operator,
// three per pair and radical, one memory pass per FFT bit, a reordering and a
// copy per FFT, nine for the products, five per lifetime (about 190 launches
// and three synchronisations, 1.3 ms an orientation at 72 x 48 dimensions).
#include <algorithm>
#include <vector>

#include "common.cuh"

namespace rpm {
namespace {

constexpr int kTileBits = 11, kTile = 1 << kTileBits;  // 32 KB of one row
constexpr int kColBits = 8, kCols = 8;                 // a column pass: 256 x 8 elements
constexpr int kPairs = 9;
constexpr int kSumBlocks = 64;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void caddmul(double2& s, double2 a, double2 b) {  // s += a b
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

struct Radical {
  int d;
  const double* lam;   // [batch][d]
  const double2* v;    // [batch][d][d]
  double2* ops;        // [batch][3][d][d]
};
struct Orientation {
  long long half[2];
  int logn;            // FFT length 2^logn
};

// V^H (S_p (x) 1) V, 16 x 16 tiles; grid (tiles, tiles, 2 batch).  With V_e the
// rows of electron value e: S_x = (V0^H V1 + V1^H V0) / 2, S_y = -i (V0^H V1 -
// V1^H V0) / 2, S_z = (V0^H V0 - V1^H V1) / 2.
__global__ void __launch_bounds__(256) k_spin_ops(Radical ra, Radical rb, int batch) {
  __shared__ double2 a0[16][17], a1[16][17], b0[16][17], b1[16][17];
  const int second = blockIdx.z >= (unsigned)batch;
  const Radical& r = second ? rb : ra;
  const int b = blockIdx.z - (second ? batch : 0), d = r.d, nuc = d / 2;
  const int i0 = blockIdx.y * 16, j0 = blockIdx.x * 16;
  if (i0 >= d || j0 >= d) return;
  const double2* v = r.v + (size_t)b * d * d;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const double2 zero = make_double2(0.0, 0.0);
  double2 m01 = zero, m10 = zero, mz = zero;
  for (int n0 = 0; n0 < nuc; n0 += 16) {
    const int n = n0 + ty;
    const double2 *up = v + (size_t)n * d, *dn = up + (size_t)nuc * d;
    const bool in = n < nuc, ii = in && i0 + tx < d, jj = in && j0 + tx < d;
    a0[ty][tx] = ii ? up[i0 + tx] : zero;
    a1[ty][tx] = ii ? dn[i0 + tx] : zero;
    b0[ty][tx] = jj ? up[j0 + tx] : zero;
    b1[ty][tx] = jj ? dn[j0 + tx] : zero;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const double2 c0 = cconj(a0[q][ty]), c1 = cconj(a1[q][ty]);
      caddmul(m01, c0, b1[q][tx]);
      caddmul(m10, c1, b0[q][tx]);
      caddmul(mz, c0, b0[q][tx]);
      caddmul(mz, make_double2(-c1.x, -c1.y), b1[q][tx]);
    }
    __syncthreads();
  }
  const int i = i0 + ty, j = j0 + tx;
  if (i >= d || j >= d) return;
  const size_t dd = (size_t)d * d;
  double2* o = r.ops + 3 * (size_t)b * dd + (size_t)i * d + j;
  o[0] = make_double2(0.5 * (m01.x + m10.x), 0.5 * (m01.y + m10.y));
  o[dd] = make_double2(0.5 * (m01.y - m10.y), -0.5 * (m01.x - m10.x));
  o[2 * dd] = make_double2(0.5 * mz.x, 0.5 * mz.y);
}

// Line (i, j) of a radical: frequency lam[i] - lam[j], weight S_p[i][j] S_q[j][i]
// / (nuclear dimension), shared out linearly between two bins of row 3 p + q.
// One thread per line and all nine rows: the bin is found once and each operator
// element read once.  grid (lines, batch, radical).  FP64 atomics (the order of
// additions is not fixed: results agree to rounding).
__global__ void __launch_bounds__(256) k_bin_lines9(Radical ra, Radical rb, double delta,
                                                   const Orientation* __restrict__ os, double2* __restrict__ rows,
                                                   long long ld, int* __restrict__ bad) {
  const Radical& r = blockIdx.z ? rb : ra;
  const int d = r.d;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)d * d) return;
  const int b = blockIdx.y;
  const long long half = os[b].half[blockIdx.z];
  const int i = (int)(idx / d), j = (int)(idx - (long long)i * d);
  const double* lam = r.lam + (size_t)b * d;
  const double pos = (lam[i] - lam[j]) / delta + (double)half;
  const double fl = floor(pos);
  if (!(fl >= 0.0 && fl < (double)(2 * half))) {  // before the conversion: infinite and NaN positions too
    atomicExch(bad, 1);
    return;
  }
  const long long lower = (long long)fl;
  const double frac = pos - fl;
  const size_t dd = (size_t)d * d;
  const double2* ops = r.ops + 3 * (size_t)b * dd;
  const double scale = 1.0 / (double)(d / 2);
  double2 sij[3], sji[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    sij[p] = ops[p * dd + (size_t)i * d + j];
    sji[p] = ops[p * dd + (size_t)j * d + i];
  }
  double2* g = rows + ((size_t)b * 2 + blockIdx.z) * kPairs * ld + lower;
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double2 c = cmul(sij[p], sji[q]);
      const double cx = c.x * scale, cy = c.y * scale;
      double2* row = g + (size_t)(3 * p + q) * ld;
      atomicAdd(&row[0].x, cx * (1.0 - frac));
      atomicAdd(&row[0].y, cy * (1.0 - frac));
      atomicAdd(&row[1].x, cx * frac);
      atomicAdd(&row[1].y, cy * frac);
    }
}

// tw[t] = exp(i pi t / count), t < count.
__global__ void k_twiddles(double2* tw, long long count) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < count;
       t += (long long)gridDim.x * blockDim.x) {
    double s, c;
    sincospi((double)t / (double)count, &s, &c);
    tw[t] = make_double2(c, s);
  }
}

// The butterflies of index bits [lo, hi) of a row, hi - lo <= 8, lo >= 11: a
// CTA takes 2^(hi - lo) x 8 elements (128-byte pieces) through shared memory.
// Forward: decimation in frequency, bits from the top; inverse: decimation in
// time, from the bottom.  grid (tiles of the longest row, rows, batch).
// Bound by memory: one read and one write of the rows for up to eight bits.
template <bool FWD>
__global__ void __launch_bounds__(256) k_fft_columns(double2* __restrict__ rows, long long ld, int nrows, int pass,
                                                    const Orientation* __restrict__ os,
                                                    const double2* __restrict__ tw, int logtw) {
  __shared__ double2 x[(1 << kColBits) * kCols];
  const int b = blockIdx.z, logn = os[b].logn, lo = kTileBits + pass * kColBits;
  if (lo >= logn) return;
  const int bits = min(kColBits, logn - lo), r = 1 << bits;
  const long long tiles = (1LL << (logn - bits)) / kCols;
  if (blockIdx.x >= tiles) return;
  // element (k, c) of the tile: base + (k << lo) + c
  const long long col = (long long)blockIdx.x * kCols;
  const long long low = col & ((1LL << lo) - 1);
  double2* g = rows + ((size_t)b * nrows + blockIdx.y) * ld + ((col >> lo) << (lo + bits)) + low;
  for (int t = threadIdx.x; t < r * kCols; t += blockDim.x) x[t] = g[((long long)(t / kCols) << lo) + t % kCols];
  for (int s = 0; s < bits; ++s) {
    const int hb = FWD ? bits - 1 - s : s, half = 1 << hb;
    __syncthreads();
    for (int t = threadIdx.x; t < r / 2 * kCols; t += blockDim.x) {
      const int c = t % kCols, j = t / kCols, pos = j & (half - 1), k = ((j >> hb) << (hb + 1)) + pos;
      double2 w = tw[(((long long)pos << lo) + low + c) << (logtw - lo - hb)];
      if (FWD) w.y = -w.y;
      double2 &u = x[k * kCols + c], &v = x[(k + half) * kCols + c];
      const double2 a = u, z = FWD ? v : cmul(w, v);
      u = make_double2(a.x + z.x, a.y + z.y);
      const double2 m = make_double2(a.x - z.x, a.y - z.y);
      v = FWD ? cmul(w, m) : m;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < r * kCols; t += blockDim.x) g[((long long)(t / kCols) << lo) + t % kCols] = x[t];
}

// Tile of 2^bits consecutive elements in shared memory, its `bits` low bits.
template <bool FWD>
__device__ __forceinline__ void tile_bits(double2* x, int bits, const double2* tw) {  // tw[t] = exp(i pi t / 2^10)
  for (int s = 0; s < bits; ++s) {
    const int hb = FWD ? bits - 1 - s : s, half = 1 << hb;
    __syncthreads();
    for (int j = threadIdx.x; j < 1 << (bits - 1); j += blockDim.x) {
      const int pos = j & (half - 1), k = ((j >> hb) << (hb + 1)) + pos;
      double2 w = tw[pos << (kTileBits - 1 - hb)];
      if (FWD) w.y = -w.y;
      double2 &u = x[k], &v = x[k + half];
      const double2 a = u, z = FWD ? v : cmul(w, v);
      u = make_double2(a.x + z.x, a.y + z.y);
      const double2 m = make_double2(a.x - z.x, a.y - z.y);
      v = FWD ? cmul(w, m) : m;
    }
  }
  __syncthreads();
}

constexpr int kConvThreads = 512;
constexpr size_t kConvSmem = sizeof(double2) * (2 * kTile + kTile / 2);

// grid (tiles of the longest row, batch).
__global__ void __launch_bounds__(kConvThreads) k_convolve(const double2* __restrict__ rows, long long ld,
                                                          double2* __restrict__ conv,
                                                          const Orientation* __restrict__ os,
                                                          const double2* __restrict__ tw, int logtw) {
  extern __shared__ double2 conv_smem[];
  double2 *xa = conv_smem, *xb = xa + kTile, *ts = xb + kTile;
  const int b = blockIdx.y, logn = os[b].logn, bits = min(kTileBits, logn), n = 1 << bits;
  const long long base = (long long)blockIdx.x << kTileBits;
  if (base >= 1LL << logn) return;
  // logtw >= 10 by construction
  for (int t = threadIdx.x; t < kTile / 2; t += blockDim.x) ts[t] = tw[(long long)t << (logtw - (kTileBits - 1))];
  double2 acc[kTile / kConvThreads];
#pragma unroll
  for (int k = 0; k < kTile / kConvThreads; ++k) acc[k] = make_double2(0.0, 0.0);
  for (int pq = 0; pq < kPairs; ++pq) {
    const double2* ga = rows + ((size_t)b * 2 * kPairs + pq) * ld + base;
    const double2* gb = ga + (size_t)kPairs * ld;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
      xa[t] = ga[t];
      xb[t] = gb[t];
    }
    for (int s = 0; s < bits; ++s) {  // tile_bits<true> of both, one barrier per bit
      const int hb = bits - 1 - s, half = 1 << hb;
      __syncthreads();
      for (int j = threadIdx.x; j < n / 2; j += blockDim.x) {
        const int pos = j & (half - 1), k = ((j >> hb) << (hb + 1)) + pos;
        const double2 w = cconj(ts[pos << (kTileBits - 1 - hb)]);
        const double2 ua = xa[k], va = xa[k + half], ub = xb[k], vb = xb[k + half];
        xa[k] = make_double2(ua.x + va.x, ua.y + va.y);
        xa[k + half] = cmul(w, make_double2(ua.x - va.x, ua.y - va.y));
        xb[k] = make_double2(ub.x + vb.x, ub.y + vb.y);
        xb[k + half] = cmul(w, make_double2(ub.x - vb.x, ub.y - vb.y));
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kTile / kConvThreads; ++k) {
      const int t = threadIdx.x + k * kConvThreads;
      if (t < n) {
        const double2 p = cmul(xa[t], xb[t]);
        acc[k] = make_double2(acc[k].x + p.x, acc[k].y + p.y);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < kTile / kConvThreads; ++k) {
    const int t = threadIdx.x + k * kConvThreads;
    if (t < n) xa[t] = acc[k];
  }
  tile_bits<false>(xa, bits, ts);
  double2* out = conv + (size_t)b * ld + base;
  for (int t = threadIdx.x; t < n; t += blockDim.x) out[t] = xa[t];
}

// part[b][block][0] = sum Re conv, [1 + t] = sum Re (conv k / (k - i w)) =
// sum (cx - x cy) / (1 + x^2), x = w / k; grid (kSumBlocks, batch).
__global__ void __launch_bounds__(256) k_yield_sums(const double2* __restrict__ conv, long long ld, double delta,
                                                   const Orientation* __restrict__ os,
                                                   const double* __restrict__ rates, int nlife,
                                                   double* __restrict__ part) {
  __shared__ double red[8];
  const int b = blockIdx.y;
  const long long centre = os[b].half[0] + os[b].half[1], count = 2 * centre + 1;
  const double inv = 1.0 / (double)(1LL << os[b].logn);
  const double2* c = conv + (size_t)b * ld;
  for (int t = -1; t < nlife; ++t) {
    const double k = t < 0 ? 0.0 : rates[t];
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x) {
      const double2 x = c[i];
      if (t < 0) {
        s += x.x * inv;
      } else {
        const double w = (double)(i - centre) * delta / k;
        s += (x.x - w * x.y) * inv / fma(w, w, 1.0);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double tot = 0.0;
      for (int w = 0; w < 8; ++w) tot += red[w];
      part[((size_t)b * kSumBlocks + blockIdx.x) * (nlife + 1) + t + 1] = tot;
    }
  }
}

__global__ void k_yield_total(const double* __restrict__ part, int values, double* __restrict__ out, int total) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int b = idx / values, t = idx - b * values;
  double s = 0.25;
  for (int k = 0; k < kSumBlocks; ++k) s += part[((size_t)b * kSumBlocks + k) * values + t];
  out[idx] = s;
}

struct Plan {
  long long nmax, bytes;
  int logmax;
  std::vector<Orientation> os;
  size_t ops_a, ops_b, rows, conv, tw, part, rates, orient;  // byte offsets
};

Plan make_plan(int da, int db, int batch, const long long* half_a, const long long* half_b, int nlife) {
  if (da < 2 || db < 2 || da % 2 || db % 2 || batch < 1 || batch > 32767 || nlife < 1 || !half_a || !half_b)
    fail(RPM_E_INVALID, "factorized yields: bad arguments");
  Plan p;
  p.logmax = kTileBits;
  for (int b = 0; b < batch; ++b) {
    Orientation o;
    o.half[0] = half_a[b];
    o.half[1] = half_b[b];
    if (o.half[0] < 1 || o.half[1] < 1 || o.half[0] > (1LL << 28) || o.half[1] > (1LL << 28))
      fail(RPM_E_INVALID, "factorized yields: grid half widths must be 1..2^28");
    const long long len = 2 * (o.half[0] + o.half[1]) + 1;
    o.logn = 1;
    while ((1LL << o.logn) < len) ++o.logn;
    p.logmax = std::max(p.logmax, o.logn);
    p.os.push_back(o);
  }
  p.nmax = 1LL << p.logmax;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t q = at;
    at += (bytes + 255) / 256 * 256;
    return q;
  };
  p.ops_a = take(sizeof(double2) * 3 * (size_t)batch * da * da);
  p.ops_b = take(sizeof(double2) * 3 * (size_t)batch * db * db);
  p.rows = take(sizeof(double2) * 2 * kPairs * (size_t)batch * p.nmax);
  p.conv = take(sizeof(double2) * (size_t)batch * p.nmax);
  p.tw = take(sizeof(double2) * (size_t)p.nmax / 2);
  p.part = take(sizeof(double) * (size_t)batch * kSumBlocks * (nlife + 1));
  p.rates = take(sizeof(double) * nlife);
  p.orient = take(sizeof(Orientation) * batch);
  p.bytes = (long long)at + 256;
  return p;
}

}  // namespace
}  // namespace rpm

using namespace rpm;

extern "C" {

int rpm_factorized_workspace(int da, int db, int batch, const long long* half_a, const long long* half_b, int nlife,
                             long long* bytes) {
  return guarded([&] {
    if (!bytes) fail(RPM_E_INVALID, "NULL pointer");
    *bytes = make_plan(da, db, batch, half_a, half_b, nlife).bytes;
  });
}

int rpm_factorized_yields(int da, int db, int batch, const double* lam_a_dev, const void* va_dev,
                          const double* lam_b_dev, const void* vb_dev, double delta, const long long* half_a,
                          const long long* half_b, const double* lifetimes, int nlife, double* out_dev, int* bad_dev,
                          void* work_dev, cudaStream_t stream) {
  return guarded([&] {
    if (!lam_a_dev || !va_dev || !lam_b_dev || !vb_dev || !lifetimes || !out_dev || !bad_dev || !work_dev)
      fail(RPM_E_INVALID, "NULL pointer");
    if (!(delta > 0.0)) fail(RPM_E_INVALID, "factorized yields: delta must be positive");
    const Plan p = make_plan(da, db, batch, half_a, half_b, nlife);
    char* w = reinterpret_cast<char*>(((uintptr_t)work_dev + 255) / 256 * 256);
    Radical ra{da, lam_a_dev, static_cast<const double2*>(va_dev), reinterpret_cast<double2*>(w + p.ops_a)};
    Radical rb{db, lam_b_dev, static_cast<const double2*>(vb_dev), reinterpret_cast<double2*>(w + p.ops_b)};
    auto* rows = reinterpret_cast<double2*>(w + p.rows);
    auto* conv = reinterpret_cast<double2*>(w + p.conv);
    auto* tw = reinterpret_cast<double2*>(w + p.tw);
    auto* part = reinterpret_cast<double*>(w + p.part);
    auto* rates = reinterpret_cast<double*>(w + p.rates);
    auto* os = reinterpret_cast<Orientation*>(w + p.orient);
    std::vector<double> k(nlife);
    for (int t = 0; t < nlife; ++t) k[t] = 1.0 / lifetimes[t];
    // pageable sources: the calls return once the host data are staged
    check_cuda(cudaMemcpyAsync(rates, k.data(), sizeof(double) * nlife, cudaMemcpyHostToDevice, stream), "rates");
    check_cuda(cudaMemcpyAsync(os, p.os.data(), sizeof(Orientation) * batch, cudaMemcpyHostToDevice, stream), "grids");
    check_cuda(cudaMemsetAsync(rows, 0, sizeof(double2) * 2 * kPairs * (size_t)batch * p.nmax, stream), "spectra");
    const int dmax = std::max(da, db), logtw = p.logmax - 1;
    k_twiddles<<<(unsigned)std::min<long long>((p.nmax / 2 + 255) / 256, 4096), 256, 0, stream>>>(tw, p.nmax / 2);
    const int t16 = (dmax + 15) / 16;
    k_spin_ops<<<dim3(t16, t16, 2 * batch), 256, 0, stream>>>(ra, rb, batch);
    k_bin_lines9<<<dim3((unsigned)(((long long)dmax * dmax + 255) / 256), batch, 2), 256, 0, stream>>>(
        ra, rb, delta, os, rows, p.nmax, bad_dev);
    const int passes = (p.logmax - kTileBits + kColBits - 1) / kColBits;
    // tiles of a column pass: elements / 2,048, or more where the top pass has fewer than eight bits
    auto col_tiles = [&](int pass) {
      long long most = 1;
      for (const Orientation& o : p.os) {
        const int lo = kTileBits + pass * kColBits;
        if (lo < o.logn) most = std::max(most, (1LL << (o.logn - std::min(kColBits, o.logn - lo))) / kCols);
      }
      return (unsigned)most;
    };
    for (int pass = passes - 1; pass >= 0; --pass)
      k_fft_columns<true><<<dim3(col_tiles(pass), 2 * kPairs, batch), 256, 0, stream>>>(rows, p.nmax, 2 * kPairs, pass,
                                                                                       os, tw, logtw);
    check_cuda(cudaFuncSetAttribute(k_convolve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kConvSmem),
               "convolve shared memory");
    k_convolve<<<dim3((unsigned)(p.nmax >> kTileBits), batch), kConvThreads, kConvSmem, stream>>>(rows, p.nmax, conv,
                                                                                                  os, tw, logtw);
    for (int pass = 0; pass < passes; ++pass)
      k_fft_columns<false><<<dim3(col_tiles(pass), 1, batch), 256, 0, stream>>>(conv, p.nmax, 1, pass, os, tw, logtw);
    k_yield_sums<<<dim3(kSumBlocks, batch), 256, 0, stream>>>(conv, p.nmax, delta, os, rates, nlife, part);
    const int total = batch * (nlife + 1);
    k_yield_total<<<(total + 127) / 128, 128, 0, stream>>>(part, nlife + 1, out_dev, total);
    check_launch("factorized yields");
  });
}

}  // extern "C"
