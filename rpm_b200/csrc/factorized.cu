// Kernels of the factorized exact oracle (rpm_quantum_needle_reproduction.py:
// 93-240): batched Hermitian eigen-decompositions of the radical
// Hamiltonians (FAD 576, TrpH 384 dimensions; one matrix per field
// orientation), complex products A^H B and FFTs.  All FP64.  The binned
// spectra, their convolution and the lifetime sums are in factorized_yields.cu.
//
// Eigen-decomposition; both radicals' matrices share each launch:
//   k_he_tridiag  Householder reduction Q^H A Q = T with a real symmetric
//                 tridiagonal T (the reflectors of LAPACK's zlarfg / zhetd2,
//                 lower form: H = I - tau v v^H, v[0] = 1, H^H [a; x] = [b; 0]
//                 with b real), the full trailing matrix updated by the
//                 Hermitian rank-2 update; one CTA per matrix;
//   k_he_tridiag_eig  implicit symmetric tridiagonal QR with Wilkinson shifts
//                 with the eigenvectors of T;
//   k_he_back     V = Q Z, the reflectors applied to Z in reverse order, two
//                 columns per warp.
// Eigenvalues come out in QR order and are sorted ascending with their
// vectors (k_he_sort), as LAPACK returns them.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "common.cuh"
#include "ptx.cuh"

namespace rpm {
namespace {

constexpr int kHeThreads = 1024;
constexpr int kHeMaxN = 1024;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

__device__ __forceinline__ double warp_reduce(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One size's share of a call; two radicals' matrices run in the same launches.
struct HePart {
  int n = 0;
  double2 *a = nullptr, *v = nullptr, *tau = nullptr, *house = nullptr;
  double *w = nullptr, *d = nullptr, *e = nullptr, *z = nullptr;
  int *perm = nullptr, *status = nullptr;
  int rows = 0;  // eigenvector rows per CTA of k_he_tridiag_eig
};
struct HePair {
  HePart part[2];
  int batch;
  __device__ const HePart& of(int item, int* b) const {
    const int second = item >= batch;
    *b = item - (second ? batch : 0);
    return part[second];
  }
};

constexpr int kHeSmem = 200 * 1024;    // rows of eigenvectors
constexpr int kHeReduceSmem = 224 * 1024;
// the reduction's vectors and the whole matrix
__host__ __device__ constexpr size_t tridiag_smem(int n) { return sizeof(double2) * ((size_t)n * n + 3 * (size_t)n); }
__host__ __device__ constexpr bool tridiag_in_smem(int n) { return tridiag_smem(n) <= kHeReduceSmem; }

// 0.5 (A + A^H) in place.
__global__ void __launch_bounds__(256) k_he_symmetrise(HePair p) {
  int b;
  const HePart& h = p.of(blockIdx.y, &b);
  const int n = h.n;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)n * n) return;
  const int i = (int)(idx / n), j = (int)(idx - (long long)i * n);
  if (i > j) return;
  double2* a = h.a + (size_t)b * n * n;
  const double2 x = a[(size_t)i * n + j], y = a[(size_t)j * n + i];
  const double2 m = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
  a[(size_t)i * n + j] = m;
  a[(size_t)j * n + i] = cconj(m);
}

// Householder reduction of matrix b: a (n x n, row-major, overwritten), d, e
// (n, n - 1 real), house (n x n: row k holds v_k, v_k[j] for j > k, v_k[k+1]
// = 1), tau (n - 1 complex).  Bound by the barriers and latencies of its n - 1
// serial steps.  A matrix that fits is worked on in shared memory (n <= 118),
// rows go to warps, one warp makes the reflector alone, and every warp forms
// w^H v for itself: four barriers a step.  6 x 72 and 6 x 48 took 313 + 172 us
// from global memory with eleven barriers a step, one size after the other; 290 us
// together with eleven barriers and the matrix in shared memory, 244 us now; 192,
// 288, 384 dimensions (in global memory) 2.4, 6.7, 14.2 -> 2.1, 6.3, 13.3 ms.
__global__ void __launch_bounds__(kHeThreads) k_he_tridiag(HePair p) {
  __shared__ double2 s_tau;
  extern __shared__ double2 he_smem[];
  int b;
  const HePart& h = p.of(blockIdx.x, &b);
  const int n = h.n;
  const size_t nn = (size_t)n * n;
  double2 *v = he_smem, *w = v + n, *u = w + n;  // u = w + alpha v
  double2* a = h.a + b * nn;
  double* d = h.d + (size_t)b * n;
  double* e = h.e + (size_t)b * n;
  double2* house = h.house + b * nn;
  double2* tau = h.tau + (size_t)b * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (tridiag_in_smem(n)) {
    double2* own = u + n;
    for (int k = threadIdx.x; k < (int)nn; k += blockDim.x) own[k] = a[k];
    a = own;
    __syncthreads();
  }
  for (int k = 0; k + 1 < n; ++k) {
    const int m = n - k - 1;  // trailing size
    if (warp == 0) {
      // x = A[k+1:, k] = conj(A[k, k+1:]) (A Hermitian, full storage)
      const double2* row = a + (size_t)k * n + k + 1;
      double part = 0.0;
      for (int j = 1 + lane; j < m; j += 32) {
        const double2 x = row[j];
        part += x.x * x.x + x.y * x.y;
      }
      const double xnorm2 = warp_reduce(part);
      const double2 alpha = cconj(row[0]);
      double2 t = make_double2(0.0, 0.0), scale = t;
      double beta = alpha.x;
      if (!(xnorm2 == 0.0 && alpha.y == 0.0)) {
        beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2), alpha.x);
        t = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
        // 1 / (alpha - beta)
        const double2 den = make_double2(alpha.x - beta, alpha.y);
        const double dd = den.x * den.x + den.y * den.y;
        scale = make_double2(den.x / dd, -den.y / dd);
      }
      for (int j = lane; j < m; j += 32) {
        const double2 vj = j > 0 ? cmul(cconj(row[j]), scale) : make_double2(1.0, 0.0);
        v[j] = vj;
        house[(size_t)k * n + k + 1 + j] = vj;
      }
      if (lane == 0) {
        s_tau = t;
        tau[k] = t;
        d[k] = a[(size_t)k * n + k].x;
        e[k] = beta;
      }
    }
    __syncthreads();
    const double2 t = s_tau;
    if (t.x != 0.0 || t.y != 0.0) {
      // w = tau A22 v, one warp per row (lanes over the row's columns)
      for (int i = warp; i < m; i += nw) {
        const double2* row = a + (size_t)(k + 1 + i) * n + k + 1;
        double sx = 0.0, sy = 0.0;
        for (int j = lane; j < m; j += 32) {
          const double2 q = cmul(row[j], v[j]);
          sx += q.x;
          sy += q.y;
        }
        sx = warp_reduce(sx);
        sy = warp_reduce(sy);
        if (lane == 0) w[i] = cmul(t, make_double2(sx, sy));
      }
      __syncthreads();
      // alpha = -1/2 tau (w^H v), by every warp that has columns; u = w + alpha v
      if (warp * 32 < m) {
        double wx = 0.0, wy = 0.0;
        for (int j = lane; j < m; j += 32) {
          const double2 q = cmul(cconj(w[j]), v[j]);
          wx += q.x;
          wy += q.y;
        }
        wx = warp_reduce(wx);
        wy = warp_reduce(wy);
        const double2 al = cmul(make_double2(-0.5 * t.x, -0.5 * t.y), make_double2(wx, wy));
        for (int j = threadIdx.x; j < m; j += blockDim.x) {
          const double2 q = cmul(al, v[j]);
          u[j] = make_double2(w[j].x + q.x, w[j].y + q.y);
        }
      }
      __syncthreads();
      // A22 -= v u^H + u v^H (full storage)
      for (int i = warp; i < m; i += nw) {
        double2* row = a + (size_t)(k + 1 + i) * n + k + 1;
        const double2 vi = v[i], ui = u[i];
        for (int j = lane; j < m; j += 32) {
          const double2 q = cmul(vi, cconj(u[j])), r = cmul(ui, cconj(v[j]));
          const double2 x = row[j];
          row[j] = make_double2(x.x - q.x - r.x, x.y - q.y - r.y);
        }
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) d[n - 1] = a[(size_t)(n - 1) * n + n - 1].x;
}

// Eigenvalues and eigenvectors of the tridiagonal T of matrix b (implicit
// symmetric QR with Wilkinson shifts, Golub & Van Loan, section 8.3): z (n x n,
// row i = component i), eigenvalues into d (QR order), status[b] raised when it
// does not converge.
//
// Bound by the serial chase of the bulge (n^2 rotations or so, each a chain of
// dependent FP64 operations).  Warp 0 chases and does nothing else: it leaves
// the rotations, 64 at a time, in a ring of slots that row warps work off, one
// eigenvector-matrix row per lane in shared memory, by columns.  Where the rows
// of a matrix do not fit, several CTAs each take a part of them and repeat the
// same chase.  A rotation takes no branch and loads the next one's operands
// before it stores: 275 cycles with the sweep's share of deflation and shift,
// 490 with its first and last iteration and its fallback treated apart.
// 6 x 72 and 6 x 48 dimensions, one size after the other with the rows in
// global memory behind each sweep: 3,600 + 1,560 us; now 770 us together.
// 192, 288, 384 dimensions: 30, 87, 170 -> 5.2, 10.3, 18 ms.
constexpr int kEigSlots = 8, kEigChunk = 64, kEigPad = 5;
constexpr int kEigFirst = 1, kEigLast = 2, kEigEnd = 4;
struct EigRing {
  double2 rot[kEigSlots][kEigChunk];
  int k0[kEigSlots], count[kEigSlots], flags[kEigSlots];
  unsigned long long full[kEigSlots], empty[kEigSlots];
};

// d, e: one entry of padding before e and two behind each
__device__ __forceinline__ void eig_chase(int n, double* d, double* e, EigRing& ring, int* status) {
  const int lane = threadIdx.x & 31;
  unsigned it = 0;  // slots filled (lane 0)
  int hi = n - 1;   // off-diagonal entries from hi on are zero
  auto slot_free = [&] {
    return it < kEigSlots || ptx::mbar_wait(&ring.empty[it % kEigSlots], (it / kEigSlots - 1) & 1u, status);
  };
  for (int sweeps = 0;; ++sweeps) {
    // deflation, from the top: the last unreduced block is [p, q]
    int q = 0, p = 0;
    for (int base = (hi - 1) & ~31; base >= 0; base -= 32) {
      const int i = base + lane;
      bool nz = false;
      if (i < hi) {
        const double ei = e[i];
        if (fabs(ei) <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1])) || fabs(ei) < DBL_MIN) e[i] = 0.0;
        else nz = true;
      }
      const unsigned m = __ballot_sync(0xffffffffu, nz);
      unsigned zero = ~m;
      if (q == 0) {
        if (!m) continue;
        const int top = 31 - __clz(m);
        q = base + top + 1;
        zero &= (1u << top) - 1u;
      }
      if (zero) {
        p = base + 32 - __clz(zero);
        break;
      }
    }
    __syncwarp();
    hi = q;
    int ok = 1;
    if (q == 0 || sweeps >= 40 * n) {
      if (lane == 0) {
        if (q != 0) atomicExch(status, 1);
        slot_free();
        ring.flags[it % kEigSlots] = kEigEnd;
        ptx::mbar_arrive(&ring.full[it % kEigSlots]);
      }
      return;
    }
    if (lane == 0) {
      const double delta = 0.5 * (d[q - 1] - d[q]);
      const double eq = e[q - 1];
      const double mu = d[q] - eq * eq / (delta + copysign(hypot(delta, eq), delta));
      double a = d[p], bb = e[p];  // d[k] and e[k] as the previous rotation left them
      double x = a - mu, y = bb;
      double cc = d[p + 1], en = e[p + 1];  // e[q] = 0, the padding behind it is never used
      for (int k0 = p; k0 < q; k0 += kEigChunk) {
        ok = slot_free() ? 1 : 0;
        if (!ok) break;
        const int slot = it % kEigSlots, k1 = min(q, k0 + kEigChunk);
        double2* rot = ring.rot[slot];
        for (int k = k0; k < k1; ++k) {
          // the next rotation's operands, ahead of this one's stores
          const double cn = d[k + 2], en2 = e[k + 2];
          // [d_k e_k; e_k d_k+1] turned by (c, s) = (x, y) / r: the sums over x
          // and y are formed beside 1 / r, not behind c and s
          const double xx = x * x, yy = y * y, xy = x * y;
          const double rr = xx + yy;
          const double nk = fma(xx, a, fma(2.0 * xy, bb, yy * cc));
          const double nk1 = fma(yy, a, fma(-2.0 * xy, bb, xx * cc));
          const double ne = fma(xy, cc - a, (xx - yy) * bb);
          const double inv = rsqrt(rr), inv2 = inv * inv;
          double ek = ne * inv2, dk1 = nk1 * inv2, dk = nk * inv2, c = x * inv, sn = y * inv, r = rr * inv;
          if (__builtin_expect(!(rr > 1e-150 && rr < 1e150), 0)) {
            r = hypot(x, y);
            c = r > 0.0 ? x / r : 1.0;
            sn = r > 0.0 ? y / r : 0.0;
            ek = c * sn * (cc - a) + (c * c - sn * sn) * bb;
            dk1 = sn * sn * a - 2.0 * c * sn * bb + c * c * cc;
            dk = c * c * a + 2.0 * c * sn * bb + sn * sn * cc;
          }
          x = ek;
          y = sn * en;
          bb = c * en;
          a = dk1;
          e[k - 1] = r;  // e[p - 1]: put back below
          d[k] = dk;
          e[k + 1] = bb;
          rot[k - k0] = make_double2(c, sn);
          cc = cn;
          en = en2;
        }
        ring.k0[slot] = k0;
        ring.count[slot] = k1 - k0;
        ring.flags[slot] = (k0 == p ? kEigFirst : 0) | (k1 == q ? kEigLast : 0);
        ptx::mbar_arrive(&ring.full[slot]);
        ++it;
      }
      d[q] = a;
      e[q - 1] = x;
      e[p - 1] = 0.0;
    }
    __syncwarp();
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return;  // status is raised: the row warps' waits end on it
  }
}

// One row per lane (row < 0: none); z[k * ld + row].
__device__ __forceinline__ void eig_rows(double* z, int ld, int row, EigRing& ring, int* status) {
  const int lane = threadIdx.x & 31;
  double zk = 0.0;
  for (unsigned it = 0;; ++it) {
    const int slot = it % kEigSlots;
    int ok = 1;
    if (lane == 0) ok = ptx::mbar_wait(&ring.full[slot], (it / kEigSlots) & 1u, status) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return;
    const int flags = ring.flags[slot];
    if (flags & kEigEnd) return;
    if (row >= 0) {
      const int count = ring.count[slot];
      const double2* rot = ring.rot[slot];
      double* zr = z + row + (size_t)ring.k0[slot] * ld;
      if (flags & kEigFirst) zk = zr[0];
      int k = 0;
      for (; k + 4 <= count; k += 4) {  // four rotations' operands ahead of their use
        double2 cs[4];
        double zn[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          cs[u] = rot[k + u];
          zn[u] = zr[(k + u + 1) * ld];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          zr[(k + u) * ld] = cs[u].x * zk + cs[u].y * zn[u];
          zk = -cs[u].y * zk + cs[u].x * zn[u];
        }
      }
      for (; k < count; ++k) {
        const double2 cs = rot[k];
        const double zn = zr[(k + 1) * ld];
        zr[k * ld] = cs.x * zk + cs.y * zn;
        zk = -cs.y * zk + cs.x * zn;
      }
      if (flags & kEigLast) zr[count * ld] = zk;
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&ring.empty[slot]);
  }
}

__global__ void __launch_bounds__(1024) k_he_tridiag_eig(HePair p) {
  __shared__ EigRing ring;
  extern __shared__ double eig_smem[];
  int b;
  const HePart& h = p.of(blockIdx.y, &b);
  const int n = h.n, ld = h.rows, row0 = blockIdx.x * ld;
  if (row0 >= n) return;
  const int rows = min(ld, n - row0);
  double* ds = eig_smem;
  double* es = ds + n + 3;  // es[-1] .. es[n + 1], ds[0] .. ds[n + 1]
  double* z = es + n + 2;
  double* d = h.d + (size_t)b * n;
  const double* e = h.e + (size_t)b * n;
  int* status = h.status + b;
  const int row_warps = (rows + 31) / 32, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < n + 2; i += blockDim.x) {
    ds[i] = i < n ? d[i] : 0.0;
    es[i] = i + 1 < n ? e[i] : 0.0;
  }
  for (int k = threadIdx.x; k < n * ld; k += blockDim.x) z[k] = k / ld == row0 + k % ld ? 1.0 : 0.0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kEigSlots; ++s) {
      ptx::mbar_init(&ring.full[s], 1);
      ptx::mbar_init(&ring.empty[s], row_warps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) {
    eig_chase(n, ds, es, ring, status);
  } else if (warp <= row_warps) {
    const int row = (warp - 1) * 32 + (threadIdx.x & 31);
    eig_rows(z, ld, row < rows ? row : -1, ring, status);
  }
  __syncthreads();
  double* zo = h.z + (size_t)b * n * n + (size_t)row0 * n;
  for (int k = threadIdx.x; k < rows * n; k += blockDim.x) zo[k] = z[(k % n) * ld + k / n];
  // d is read by every CTA of the matrix: the values go out through w
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n; i += blockDim.x) h.w[(size_t)b * n + i] = ds[i];
}

// Ascending order of the eigenvalues: perm[r] = index of the r-th smallest
// (ties by index, NaN behind the numbers, so that perm is a permutation whatever
// the matrix held), sorted values into w (which holds them in QR order).
__global__ void __launch_bounds__(256) k_he_sort(HePair p) {
  __shared__ double d[kHeMaxN];
  int b;
  const HePart& h = p.of(blockIdx.x, &b);
  const int n = h.n;
  int* perm = h.perm + (size_t)b * n;
  double* w = h.w + (size_t)b * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = w[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double x = d[i];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double y = d[j];
      const bool same = y == x || (isnan(x) && isnan(y));
      r += (same ? j < i : y < x || isnan(x)) ? 1 : 0;
    }
    perm[r] = i;
    w[r] = x;
  }
}

// V = Q Z[:, perm]: the reflectors H_k = I - tau_k v_k v_k^H applied for
// k = n-2 .. 0, two columns per warp in shared memory, so that a step's sum
// needs no block barrier: 125 + 62 us for 6 x 72 and 6 x 48 dimensions with
// eight warps per column, now 78 us together.
constexpr int kBackWarps = 4, kBackCols = 2;
__global__ void __launch_bounds__(32 * kBackWarps) k_he_back(HePair p) {
  extern __shared__ double2 he_smem[];
  int b;
  const HePart& h = p.of(blockIdx.y, &b);
  const int n = h.n;
  const size_t nn = (size_t)n * n;
  const double* z = h.z + b * nn;
  const int* perm = h.perm + (size_t)b * n;
  const double2* house = h.house + b * nn;
  const double2* tau = h.tau + (size_t)b * n;
  double2* v = h.v + b * nn;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * kBackWarps + warp) * kBackCols;
  if (c0 >= n) return;
  const int nc = min(kBackCols, n - c0);
  double2* x0 = he_smem + (size_t)warp * kBackCols * n;
  double2* x1 = x0 + n;
  const int s0 = perm[c0], s1 = perm[c0 + nc - 1];  // nc = 1: the same column twice
  for (int i = lane; i < n; i += 32) {
    x0[i] = make_double2(z[(size_t)i * n + s0], 0.0);
    x1[i] = make_double2(z[(size_t)i * n + s1], 0.0);
  }
  for (int k = n - 2; k >= 0; --k) {
    const double2 t = tau[k];
    if (t.x == 0.0 && t.y == 0.0) continue;  // H_k = I
    const double2* hv = house + (size_t)k * n;
    double2 a0 = make_double2(0.0, 0.0), a1 = a0;
    __syncwarp();
    for (int i = k + 1 + lane; i < n; i += 32) {
      const double2 u = cconj(hv[i]);
      const double2 p0 = cmul(u, x0[i]), p1 = cmul(u, x1[i]);
      a0 = make_double2(a0.x + p0.x, a0.y + p0.y);
      a1 = make_double2(a1.x + p1.x, a1.y + p1.y);
    }
    a0 = cmul(t, make_double2(warp_reduce(a0.x), warp_reduce(a0.y)));
    a1 = cmul(t, make_double2(warp_reduce(a1.x), warp_reduce(a1.y)));
    for (int i = k + 1 + lane; i < n; i += 32) {
      const double2 u = hv[i];
      const double2 p0 = cmul(u, a0), p1 = cmul(u, a1);
      x0[i] = make_double2(x0[i].x - p0.x, x0[i].y - p0.y);
      x1[i] = make_double2(x1[i].x - p1.x, x1[i].y - p1.y);
    }
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    v[(size_t)i * n + c0] = x0[i];
    if (nc == 2) v[(size_t)i * n + c0 + 1] = x1[i];
  }
}

// C = A^H B for square n x n complex matrices (row-major), 16 x 16 tiles;
// grid (tiles, tiles, batch).
__global__ void __launch_bounds__(256) k_zgemm_hn(const double2* a_all, const double2* b_all, double2* c_all,
                                                 int n) {
  __shared__ double2 at[16][17], bt[16][17];
  const size_t nn = (size_t)n * n;
  const double2* a = a_all + blockIdx.z * nn;
  const double2* b = b_all + blockIdx.z * nn;
  double2* c = c_all + blockIdx.z * nn;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i = blockIdx.y * 16 + ty, j = blockIdx.x * 16 + tx;
  double2 acc = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < n; k0 += 16) {
    // at[kk][ii] = A[k0 + kk][i0 + ii], bt[kk][jj] = B[k0 + kk][j0 + jj]
    const int kk = ty, ii = tx;
    const int ka = k0 + kk;
    at[kk][ii] = (ka < n && blockIdx.y * 16 + ii < n) ? a[(size_t)ka * n + blockIdx.y * 16 + ii] : make_double2(0.0, 0.0);
    bt[kk][ii] = (ka < n && blockIdx.x * 16 + ii < n) ? b[(size_t)ka * n + blockIdx.x * 16 + ii] : make_double2(0.0, 0.0);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const double2 x = cconj(at[q][ty]), y = bt[q][tx];
      acc.x = fma(x.x, y.x, fma(-x.y, y.y, acc.x));
      acc.y = fma(x.x, y.y, fma(x.y, y.x, acc.y));
    }
    __syncthreads();
  }
  if (i < n && j < n) c[(size_t)i * n + j] = acc;
}

// Radix-2 FFT (power-of-two n, batch of rows): bit-reversal permutation, then
// log2 n butterfly passes in place; sign -1 forward, +1 inverse (unscaled).
__global__ void k_fft_bitrev(const double2* in, double2* out, int n, int logn, long long total) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const long long row = t / n;
    const int i = (int)(t - row * n);
    const int r = (int)(__brev((unsigned)i) >> (32 - logn));
    out[row * n + r] = in[t];
  }
}
__global__ void k_fft_pass(double2* x, int n, int half, double sign, long long total_half) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total_half;
       t += (long long)gridDim.x * blockDim.x) {
    const long long row = t / (n / 2);
    const int j = (int)(t - row * (n / 2));
    const int pos = j % half, grp = j / half;
    const long long i0 = row * n + (long long)grp * 2 * half + pos, i1 = i0 + half;
    double s, c;
    sincospi(sign * (double)pos / (double)half, &s, &c);
    const double2 u = x[i0], v = x[i1];
    const double2 w = make_double2(c * v.x - s * v.y, c * v.y + s * v.x);
    x[i0] = make_double2(u.x + w.x, u.y + w.y);
    x[i1] = make_double2(u.x - w.x, u.y - w.y);
  }
}
// acc += x * y (element-wise), or x *= scale
__global__ void k_fft_mac(double2* acc, const double2* x, const double2* y, long long total) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const double2 p = cmul(x[t], y[t]);
    acc[t] = make_double2(acc[t].x + p.x, acc[t].y + p.y);
  }
}

int grid_for(long long work) { return (int)std::max(1LL, std::min((work + 255) / 256, 65535LL * 4)); }

// A kernel's limit is the most that any size needs, whatever the call's own
// sizes: calls of other threads may stand between this and their launches.
template <class K>
void set_smem(K kern, size_t bytes) {
  check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), "eigh shared memory");
}

long long eigh_bytes(int n, int batch) {
  const long long nn = (long long)n * n;
  // d, e, perm (as double), tau (2 doubles), status; house (complex) and z (real)
  return (long long)batch * ((3 * n + 2 * n + 1) * 8 + nn * 16 + nn * 8) + 7 * 256;  // + alignment of 7 parts
}

char* eigh_part(HePart& h, int n, int batch, void* a, double* w, void* v, char* p) {
  const long long nn = (long long)n * n;
  auto take = [&](long long bytes) {
    char* q = p;
    p += (bytes + 255) / 256 * 256;
    return q;
  };
  h.n = n;
  h.a = static_cast<double2*>(a);
  h.w = w;
  h.v = static_cast<double2*>(v);
  h.d = reinterpret_cast<double*>(take((long long)batch * n * 8));
  h.e = reinterpret_cast<double*>(take((long long)batch * n * 8));
  h.perm = reinterpret_cast<int*>(take((long long)batch * n * 8));
  h.tau = reinterpret_cast<double2*>(take((long long)batch * n * 16));
  h.status = reinterpret_cast<int*>(take((long long)batch * 8));
  h.house = reinterpret_cast<double2*>(take((long long)batch * nn * 16));
  h.z = reinterpret_cast<double*>(take((long long)batch * nn * 8));
  // as many rows per CTA as fit beside d and e (n = 1024: 22)
  h.rows = std::min({n, 31 * 32, (kHeSmem / 8 - 2 * n - kEigPad) / n});
  return p;
}

// `parts` sizes of `batch` matrices each.
void eigh_run(HePair& p, int parts, bool symmetrise, cudaStream_t stream) {
  int nmax = 0, row_blocks = 1, row_threads = 0;
  size_t eig_smem = 0, red_smem = 0;
  for (int k = 0; k < parts; ++k) {
    const HePart& h = p.part[k];
    nmax = std::max(nmax, h.n);
    row_blocks = std::max(row_blocks, (h.n + h.rows - 1) / h.rows);
    row_threads = std::max(row_threads, (h.rows + 31) / 32 * 32);
    eig_smem = std::max(eig_smem, sizeof(double) * (size_t)(2 * h.n + kEigPad + h.n * h.rows));
    red_smem = std::max(red_smem, tridiag_in_smem(h.n) ? tridiag_smem(h.n) : sizeof(double2) * 3 * (size_t)h.n);
    check_cuda(cudaMemsetAsync(h.status, 0, sizeof(int) * p.batch, stream), "eigh status");
  }
  const int items = p.batch * parts;
  if (symmetrise)
    k_he_symmetrise<<<dim3((unsigned)(((long long)nmax * nmax + 255) / 256), items), 256, 0, stream>>>(p);
  auto back_bytes = [](int n) { return sizeof(double2) * (size_t)kBackWarps * kBackCols * n; };
  const size_t back_smem = back_bytes(nmax);
  set_smem(k_he_tridiag, kHeReduceSmem);
  set_smem(k_he_tridiag_eig, kHeSmem);
  set_smem(k_he_back, back_bytes(kHeMaxN));
  k_he_tridiag<<<items, kHeThreads, red_smem, stream>>>(p);
  k_he_tridiag_eig<<<dim3(row_blocks, items), 32 + row_threads, eig_smem, stream>>>(p);
  k_he_sort<<<items, 256, 0, stream>>>(p);
  const int per = kBackWarps * kBackCols;
  k_he_back<<<dim3((nmax + per - 1) / per, items), 32 * kBackWarps, back_smem, stream>>>(p);
  check_launch("eigh");
  std::vector<int> st((size_t)items);
  for (int k = 0; k < parts; ++k)
    check_cuda(cudaMemcpyAsync(st.data() + (size_t)k * p.batch, p.part[k].status, sizeof(int) * p.batch,
                               cudaMemcpyDeviceToHost, stream), "eigh status");
  check_cuda(cudaStreamSynchronize(stream), "eigh sync");
  for (int s : st)
    if (s) fail(RPM_E_NUMERIC, "eigh: the tridiagonal QR did not converge");
}

}  // namespace
}  // namespace rpm

using namespace rpm;

extern "C" {

int rpm_he_eigh_workspace(int n, int batch, long long* bytes) {
  return guarded([&] {
    if (n < 2 || n > kHeMaxN || batch < 1 || !bytes) fail(RPM_E_INVALID, "eigh: need 2 <= n <= 1024, batch >= 1");
    *bytes = eigh_bytes(n, batch);
  });
}

int rpm_he_eigh(int n, int batch, void* a_dev, double* w_dev, void* v_dev, void* work_dev, cudaStream_t stream) {
  return guarded([&] {
    long long need = 0;
    if (rpm_he_eigh_workspace(n, batch, &need) != RPM_OK) fail(RPM_E_INVALID, "eigh: bad sizes");
    if (!a_dev || !w_dev || !v_dev || !work_dev) fail(RPM_E_INVALID, "eigh: null pointer");
    HePair p;
    p.batch = batch;
    eigh_part(p.part[0], n, batch, a_dev, w_dev, v_dev, static_cast<char*>(work_dev));
    eigh_run(p, 1, false, stream);
  });
}

int rpm_he_eigh_pair(int na, int nb, int batch, void* a_dev, void* b_dev, double* wa_dev, double* wb_dev, void* va_dev,
                     void* vb_dev, void* work_dev, cudaStream_t stream) {
  return guarded([&] {
    long long need = 0;
    if (rpm_he_eigh_workspace(na, batch, &need) != RPM_OK || rpm_he_eigh_workspace(nb, batch, &need) != RPM_OK ||
        batch > 32767)
      fail(RPM_E_INVALID, "eigh: bad sizes");
    if (!a_dev || !b_dev || !wa_dev || !wb_dev || !va_dev || !vb_dev || !work_dev)
      fail(RPM_E_INVALID, "eigh: null pointer");
    HePair p;
    p.batch = batch;
    char* rest = eigh_part(p.part[0], na, batch, a_dev, wa_dev, va_dev, static_cast<char*>(work_dev));
    eigh_part(p.part[1], nb, batch, b_dev, wb_dev, vb_dev, rest);
    eigh_run(p, 2, true, stream);
  });
}

int rpm_zgemm_hn(int n, int batch, const void* a_dev, const void* b_dev, void* c_dev, cudaStream_t stream) {
  return guarded([&] {
    if (n < 1 || batch < 1 || !a_dev || !b_dev || !c_dev) fail(RPM_E_INVALID, "zgemm_hn: bad arguments");
    const int t = (n + 15) / 16;
    k_zgemm_hn<<<dim3(t, t, batch), 256, 0, stream>>>(static_cast<const double2*>(a_dev),
                                                      static_cast<const double2*>(b_dev), static_cast<double2*>(c_dev),
                                                      n);
    check_launch("zgemm_hn");
  });
}

int rpm_fft_pow2(int n, int batch, void* data_dev, void* scratch_dev, int inverse, cudaStream_t stream) {
  return guarded([&] {
    if (n < 2 || (n & (n - 1)) || batch < 1 || !data_dev || !scratch_dev)
      fail(RPM_E_INVALID, "fft: n must be a power of two >= 2");
    int logn = 0;
    while ((1 << logn) < n) ++logn;
    const long long total = (long long)n * batch;
    double2* x = static_cast<double2*>(data_dev);
    double2* s = static_cast<double2*>(scratch_dev);
    k_fft_bitrev<<<grid_for(total), 256, 0, stream>>>(x, s, n, logn, total);
    for (int half = 1; half < n; half *= 2)
      k_fft_pass<<<grid_for(total / 2), 256, 0, stream>>>(s, n, half, inverse ? 1.0 : -1.0, total / 2);
    check_cuda(cudaMemcpyAsync(x, s, sizeof(double2) * total, cudaMemcpyDeviceToDevice, stream), "fft copy");
    check_launch("fft");
  });
}

int rpm_spectrum_mac(long long count, void* acc_dev, const void* x_dev, const void* y_dev, cudaStream_t stream) {
  return guarded([&] {
    if (count < 1 || !acc_dev || !x_dev || !y_dev) fail(RPM_E_INVALID, "spectrum_mac: bad arguments");
    k_fft_mac<<<grid_for(count), 256, 0, stream>>>(static_cast<double2*>(acc_dev), static_cast<const double2*>(x_dev),
                                                   static_cast<const double2*>(y_dev), count);
    check_launch("spectrum_mac");
  });
}

}  // extern "C"
