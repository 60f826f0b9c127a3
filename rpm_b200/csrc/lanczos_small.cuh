// Lanczos iterations of a whole Krylov step in one block per trajectory, for
// small states on the general cube kernels (included by batched.cu).
//
// The launch sequence per iteration (cube_pass_l, cube_pass_r, k_b_update) is
// latency: 64 states of 96 components took 20 us per iteration for 0.2 us of
// arithmetic.  Here v_{j-1}, v_j, the partial and w stay in shared memory for
// all m iterations and only the finished basis vectors are written out.
// Nothing changes in the numbers: the element arithmetic is the passes'
// (cube_apply), and the sums of alpha_j and beta_j run in the order of the
// launches they replace, because their last bits decide FP32 roundings and
// step sizes later on:
//   * alpha_j: pass R's tiles of `tl` rows are virtual blocks of 256 threads;
//     a virtual block with at most 32 tasks is a segment of a warp (the other
//     lanes and warps of the real block only add zeros), its warps are summed
//     in order, then the tiles in order;
//   * beta_j: k_b_update's mapping of 256 threads to 2,048 components.
namespace rpm {
namespace small {

constexpr int kMaxN = 4096;     // components (four vectors of 32 KB)
constexpr int kThreads = 256;   // the virtual blocks' and k_b_update's block size
constexpr int kWarps = kThreads / 32;
static_assert(kThreads == kEwThreads, "beta_j's sum uses k_b_update's thread mapping");

__host__ __device__ inline int align16b(int bytes) { return (bytes + 15) & ~15; }

struct Shape {
  int nl, nr, tab_cap, no_l, no_r, tl;
  __host__ __device__ int blocks() const { return (nl + tl - 1) / tl; }
  __host__ __device__ size_t smem() const {
    const int n = nl * nr;
    return 2 * (size_t)align16b(tab_cap * (int)sizeof(float2)) + align16b((no_l + no_r) * (int)sizeof(OuterRec<float2>)) +
           align16b((nl + nr) * 4) + 4 * (size_t)align16b(n * (int)sizeof(float2)) +
           sizeof(double) * (size_t)blocks() * (kWarps + 1);
  }
};

template <int NIL, int NIR>
__global__ void __launch_bounds__(kThreads) k_b_lanczos_small(BatchDev B, const CubeView<float2>* __restrict__ views,
                                                              const int* __restrict__ sys_of, int b0, Shape sh) {
  using A = CubeArith<float2>;
  constexpr int CL = 1 << NIL, CR = 1 << NIR;
  const int b = b0 + blockIdx.x;
  TrajState& s = B.st[b];
  if (s.skip) return;
  const CubeView<float2>* view = views + sys_of[b];
  __shared__ CubeSide L, R;
  __shared__ float2 pair[16];
  __shared__ double red[32];
  __shared__ double s_alpha, s_scale;
  __shared__ int s_stop;
  extern __shared__ __align__(16) unsigned char raw[];
  const int n = sh.nl * sh.nr, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* pos = raw;
  auto take = [&](int bytes) {
    unsigned char* at = pos;
    pos += align16b(bytes);
    return at;
  };
  float2* tabl = reinterpret_cast<float2*>(take(sh.tab_cap * (int)sizeof(float2)));
  float2* tabr = reinterpret_cast<float2*>(take(sh.tab_cap * (int)sizeof(float2)));
  OuterRec<float2>* otl = reinterpret_cast<OuterRec<float2>*>(take((sh.no_l + sh.no_r) * (int)sizeof(OuterRec<float2>)));
  OuterRec<float2>* otr = otl + sh.no_l;
  int* offl = reinterpret_cast<int*>(take((sh.nl + sh.nr) * 4));
  int* offr = offl + sh.nl;
  float2* x = reinterpret_cast<float2*>(take(n * (int)sizeof(float2)));   // V_j as the last update left it, then v_j
  float2* w = reinterpret_cast<float2*>(take(n * (int)sizeof(float2)));   // H v_j, then the next V_{j+1}
  float2* vp = reinterpret_cast<float2*>(take(n * (int)sizeof(float2)));  // v_{j-1}
  float2* y = reinterpret_cast<float2*>(take(n * (int)sizeof(float2)));   // pass L's partial
  double* part = reinterpret_cast<double*>(pos);                          // [virtual block][virtual warp]
  double* tile = part + sh.blocks() * kWarps;                             // [virtual block]

  if (tid < 16) pair[tid] = view->pair[tid];
  for (int k = tid; k < sh.nl; k += kThreads) offl[k] = view->offl[k];
  for (int k = tid; k < sh.nr; k += kThreads) offr[k] = view->offr[k];
  load_side(view->L, view->tabL, L, tabl);
  load_side(view->R, view->tabR, R, tabr);
  float2* base = B.V + (size_t)b * (B.m + 1) * B.ld;
  for (int k = tid; k < n; k += kThreads) x[k] = base[k];
  if (tid == 0) {
    s_scale = s.scale;
    s_stop = 0;
  }
  __syncthreads();
  build_outer<float2, NIL>(L, tabl, otl, sh.no_l);
  build_outer<float2, NIR>(R, tabr, otr, sh.no_r);
  __syncthreads();
  const InnerConst<float2, NIL> icl(L, tabl);
  const InnerConst<float2, NIR> icr(R, tabr);
  const int half_l = sh.nl / 2, half_r = sh.nr / 2;
  const int no_l = half_l >> NIL, no_r = half_r >> NIR;
  const int el = offl[half_l] - offl[0], er = offr[half_r] - offr[0];
  // virtual blocks of pass R: `tasks` cubes each, packed 32 / seg to a warp when they fit
  const int tasks = sh.tl * no_r;
  int seg = 1;
  while (seg < 32 && seg < tasks) seg <<= 1;
  const int vwarps = (min(tasks, kThreads) + 31) / 32, vblocks = sh.blocks();
  const int packed = 32 / seg;
  const int units = vwarps == 1 ? (vblocks + packed - 1) / packed : vblocks * vwarps;
  const int m = B.m, mcap = s.mcap;
  double beta_prev = 0.0;
  for (int j = 0; j < m; ++j) {
    const bool last = j == m - 1;
    const float sf = (float)s_scale;
    // pass L: L psi + the pair operator
    for (int t = tid; t < sh.nr * no_l; t += kThreads) {
      const int c = t % sh.nr, o = t / sh.nr;
      const int h = c >= half_r ? 1 : 0, col = offr[c];
      const OuterRec<float2> rec = otl[o];
      float dout[2];
      float2 fout[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        dout[e] = rec.d[e] + A::re(pair[(e * 2 + h) * 4 + e * 2 + h]);
        fout[e] = A::add(rec.f[e], pair[(e * 2 + h) * 4 + (1 - e) * 2 + h]);
      }
      float2 xv[2][CL], acc[2][CL];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int i = 0; i < CL; ++i) {
          xv[e][i] = x[offl[o * CL + i] + e * el + col];
          acc[e][i] = czero<float2>();
        }
      cube_apply<float2, NIL>(L, tabl, icl, rec, dout, fout, xv, acc,
                              [&](int e, int i, int delta) { return x[offl[(o + delta) * CL + i] + e * el + col]; });
      const int flip = offr[h ? c - half_r : c + half_r];
#pragma unroll
      for (int ep = 0; ep < 2; ++ep) {
        const float2 p0 = pair[(0 * 2 + h) * 4 + ep * 2 + (1 - h)];
        const float2 p1 = pair[(1 * 2 + h) * 4 + ep * 2 + (1 - h)];
#pragma unroll
        for (int i = 0; i < CL; ++i) {
          const float2 z = x[offl[o * CL + i] + ep * el + flip];
          acc[0][i] = A::mac(p0, z, z, acc[0][i]);
          acc[1][i] = A::mac(p1, z, z, acc[1][i]);
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int i = 0; i < CL; ++i) {
          float2 v = acc[e][i];
          v.x *= sf;
          v.y *= sf;
          y[offl[o * CL + i] + e * el + col] = v;
        }
    }
    __syncthreads();
    // pass R: adds psi R^T, and the tiles' shares of <V_j, w>
    for (int u = warp; u < units; u += kWarps) {
      const int vb = vwarps == 1 ? u * packed + lane / seg : u / vwarps;
      const int vw = vwarps == 1 ? 0 : u % vwarps;
      const int t0 = vwarps == 1 ? lane % seg : vw * 32 + lane;
      const int l0 = vb * sh.tl;
      const int mine = vb < vblocks ? min(sh.tl, sh.nl - l0) * no_r : 0;
      double dot = 0.0;
      for (int t = t0; t < mine; t += kThreads) {
        const int o = t % no_r, row = offl[l0 + t / no_r];
        const OuterRec<float2> rec = otr[o];
        const float dout[2] = {rec.d[0], rec.d[1]};
        const float2 fout[2] = {rec.f[0], rec.f[1]};
        float2 xv[2][CR], acc[2][CR];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < CR; ++i) {
            xv[e][i] = x[row + offr[o * CR + i] + e * er];
            acc[e][i] = czero<float2>();
          }
        cube_apply<float2, NIR>(R, tabr, icr, rec, dout, fout, xv, acc,
                                [&](int e, int i, int delta) { return x[row + offr[(o + delta) * CR + i] + e * er]; });
        float prt = 0;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < CR; ++i) {
            const int at = row + offr[o * CR + i] + e * er;
            const float2 p = y[at];
            float2 v;
            v.x = fma(sf, acc[e][i].x, p.x);
            v.y = fma(sf, acc[e][i].y, p.y);
            w[at] = v;
            const float2 xe = x[at];
            prt = fma(xe.x, v.x, fma(xe.y, v.y, prt));
          }
        dot += (double)prt * (double)sf;
      }
      for (int o = seg / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (vb < vblocks && (vwarps == 1 ? lane % seg == 0 : lane == 0)) part[vb * kWarps + vw] = dot;
    }
    __syncthreads();
    for (int k = tid; k < vblocks; k += kThreads) {
      double t = 0.0;
      for (int v = 0; v < vwarps; ++v) t += part[k * kWarps + v];
      tile[k] = t;
    }
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int k = 0; k < vblocks; ++k) t += tile[k];
      s_alpha = t;
      s.alpha[j] = t;
    }
    __syncthreads();
    // v_j = scale V_j;  w -= alpha_j v_j + beta_{j-1} v_{j-1};  |w|^2
    const float a = (float)s_alpha, bp = j > 0 ? (float)beta_prev : 0.0f;
    float2* vj = base + (size_t)j * B.ld;
    double tot = 0.0;
    for (int c0 = 0; c0 < n; c0 += kEwChunk) {
      double nn = 0.0;
      const int end = min(n, c0 + kEwChunk);
      for (int i = c0 + tid; i < end; i += kThreads) {
        float2 v = x[i];
        v.x *= sf;
        v.y *= sf;
        x[i] = v;
        vj[i] = v;
        if (!last) {
          float2 z = w[i];
          z.x = fmaf(-a, v.x, z.x);
          z.y = fmaf(-a, v.y, z.y);
          if (j > 0) {
            const float2 u = vp[i];
            z.x = fmaf(-bp, u.x, z.x);
            z.y = fmaf(-bp, u.y, z.y);
          }
          w[i] = z;
          nn = fma((double)z.x, (double)z.x, fma((double)z.y, (double)z.y, nn));
        }
      }
      if (!last) tot += block_sum(nn, red);
    }
    if (last) break;
    const double bj = sqrt(tot);
    if (tid == 0) {
      s.beta[j] = bj;
      s_scale = bj > 0.0 ? 1.0 / bj : 0.0;
      s.scale = s_scale;
      const double ref = fabs(s_alpha) + (j > 0 ? beta_prev : 0.0);
      if (j + 1 >= mcap) {  // this trajectory's Krylov cap: its basis ends here
        s.skip = 1;
        s.msize = mcap;
        s_stop = 1;
      } else if (!(bj > B.breakdown_rel * ref)) {
        s.stop = 1;
        s.skip = 1;
        s.msize = j + 1;
        s_stop = 1;
      }
    }
    __syncthreads();
    if (s_stop) break;
    beta_prev = bj;
    float2* old = vp;  // (v_{j-1}, v_j, w) -> (v_j, V_{j+1}, free)
    vp = x;
    x = w;
    w = old;
  }
}

// Shape of a group's launches; false when the kernel does not cover it.
inline bool shape_of(const CubePlan& p, int batch, Shape& sh) {
  if ((long long)p.nl * p.nr > kMaxN) return false;
  sh.nl = p.nl;
  sh.nr = p.nr;
  sh.tab_cap = p.tab_cap;
  sh.no_l = p.ni_l >= 2 ? p.n_outer_l2 : p.n_outer_l1;
  sh.no_r = p.ni_r >= 2 ? p.n_outer_r2 : p.n_outer_r1;
  sh.tl = cube_rows_c64(p, batch);
  return sh.tl > 0 && sh.smem() <= 200 * 1024;
}

// Kernel for a plan's inner digits.
using Kernel = void (*)(BatchDev, const CubeView<float2>*, const int*, int, Shape);
inline Kernel pick(const CubePlan& p) {
  if (p.ni_l >= 2) return p.ni_r >= 2 ? k_b_lanczos_small<2, 2> : k_b_lanczos_small<2, 1>;
  return p.ni_r >= 2 ? k_b_lanczos_small<1, 2> : k_b_lanczos_small<1, 1>;
}

// Before any capture: the shared-memory limit of the plan's kernel.
inline void prepare(const CubePlan& p) {
  check_cuda(cudaFuncSetAttribute(pick(p), cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024),
             "small Lanczos attr");
}

inline void launch(const BatchDev& B, const CubeView<float2>* views, const int* sys_of, int b0, int nb,
                   const CubePlan& p, const Shape& sh, cudaStream_t st) {
  pick(p)<<<nb, kThreads, sh.smem(), st>>>(B, views, sys_of, b0, sh);
  check_launch("k_b_lanczos_small");
}

}  // namespace small
}  // namespace rpm
