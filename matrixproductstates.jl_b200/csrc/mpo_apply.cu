// Small-K contraction with one local MPO tensor:
//     Out[x, m, y] = alpha * sum_k In[x, k, y] * Op[k, m] + beta * Out[x, m, y]
// with k = (k1, k2) and m = (m1, m2) split indices addressed by element strides.
//
// This is the second GEMM of prod_AOR (src/mps_base.jl:15-17) and of prod_AOL
// (src/mps_base.jl:34-37), with the reference's permutedims copies folded into the
// strides, and the site contraction of apply_site_MPOtoMPS (src/MatrixProductStates.jl:126-133).
// K = w*d and M = w*d are small (<= 64), so the whole Op sits in shared memory beside the In of the
// CTA's columns (a column: 32 consecutive x of one y), which is read once and before any Out is
// written (Out may be In).
//
// What bounds it: memory traffic for large sites, the chain launch -> load -> product -> store for
// small ones.  A thread has 8 loads in flight, In is staged along whichever index is contiguous (34
// elements between k), and no index needs an integer division.  The
// warps of a CTA are G groups of MQ outputs m times CW columns, so that narrow X fill it too.
// B200, against one thread per 8 outputs of 64 to 256 x of one y per CTA, with divisions per element
// (cold caches): X = Y = 512, K = M of 25 to 32 176 -> 130 us (the tensor path alone needs 58);
// 128 x 128 19.5 -> 14.9; 256 x 256 in 8 copies, K = M of 9 to 14 53.8 -> 36; 32 x 32 8.5 -> 4.3.
#include "common.cuh"

#include <algorithm>

namespace mpsb {
namespace {

constexpr int LDI = 34;   // elements between the k of a staged column (2 modulo 8: no bank conflicts of fragments)
constexpr int LOADS = 8;  // loads of a thread in flight

// n / d for n d < 2^32
struct Div {
  unsigned d, mul;
  explicit Div(int x) : d((unsigned)x), mul((unsigned)(((1ull << 32) + d - 1) / d)) {}
  __device__ __forceinline__ unsigned operator()(unsigned n) const { return d == 1 ? n : __umulhi(n, mul); }
};

struct MpoParams {
  MpoApply a;
  int64_t op_k1, op_k2, op_m1, op_m2;
  int ncols, nxb;   // columns; columns of one y
  int G;            // warps of one column
  int Mp;           // elements between the k of Op in shared memory, at least M rounded up to MQ (or 8)
  Div div_k, div_k1, div_m1;
};

// MQ: outputs m of a warp, 2 or 4 with an x per lane, or MQ_MMA as fragments of the FP64 tensor path
constexpr int MQ_MMA = 16;
template <int MQ, bool K1FAST>
__global__ void __launch_bounds__(256) mpo_apply_kernel(const __grid_constant__ MpoParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const MpoApply& a = P.a;
  constexpr bool MMA = MQ == MQ_MMA;
  const int K = a.K1 * a.K2, M = a.M1 * a.M2, Mp = P.Mp, G = P.G;
  const int Kp = MMA ? (K + 7) / 8 * 8 : K;
  cd* opS = reinterpret_cast<cd*>(smem_raw);   // [k][m], zero for m >= M and k >= K
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int cl = warp / G, g = warp - cl * G;
  const int64_t bz = blockIdx.y;
  const int CW = blockDim.x / 32 / G;
  const int n = 32 * K, step = 32 * G;
  cd* inS = opS + Kp * Mp + cl * Kp * LDI;   // [k][x], zero for k >= K
  const int col = blockIdx.x * CW + cl;
  const bool live = col < P.ncols;
  const int y = col / P.nxb, x0 = (col - y * P.nxb) * 32;
  const cd* in = a.in + bz * a.in_b + (int64_t)y * a.in_y;
  // element e of the column: lane = x and e / 32 = k, or k1 fastest, then x, then k2
  auto element = [&](int e, int& k, int& x) -> const cd* {
    if (K1FAST) {
      const int t = (int)P.div_k1((unsigned)e), k1 = e - t * a.K1, k2 = t / 32;
      x = t % 32;
      k = k1 + a.K1 * k2;
      return in + (int64_t)(x0 + x) * a.in_x + k1 + k2 * a.in_k2;
    }
    k = e / 32;
    x = lane;
    const int k2 = (int)P.div_k1((unsigned)k), k1 = k - k2 * a.K1;
    return in + (int64_t)(x0 + x) * a.in_x + k1 * a.in_k1 + k2 * a.in_k2;
  };
  cd v[LOADS];
  auto load = [&](int e0) {
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const int e = e0 + q * step;
      v[q] = cmk(0.0, 0.0);
      if (live && e < n) {
        int k, x;
        const cd* p = element(e, k, x);
        if (x0 + x < a.X) v[q] = *p;
      }
    }
  };
  auto store = [&](int e0) {
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const int e = e0 + q * step;
      if (e < n) {
        int k, x;
        element(e, k, x);
        inS[k * LDI + x] = v[q];
      }
    }
  };
  load(32 * g + lane);   // in flight while Op comes in
  const cd* op = a.op + bz * a.op_b;
  for (int e0 = threadIdx.x; e0 < K * Mp; e0 += LOADS * blockDim.x) {
    cd o[LOADS];
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const int e = e0 + q * blockDim.x;
      const int m = (int)P.div_k((unsigned)e), k = e - m * K;   // k fastest
      const int k2 = (int)P.div_k1((unsigned)k), k1 = k - k2 * a.K1;
      const int m2 = (int)P.div_m1((unsigned)m), m1 = m - m2 * a.M1;
      o[q] = cmk(0.0, 0.0);
      if (m < M) o[q] = op[k1 * P.op_k1 + k2 * P.op_k2 + m1 * P.op_m1 + m2 * P.op_m2];
    }
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const int e = e0 + q * blockDim.x;
      const int m = (int)P.div_k((unsigned)e), k = e - m * K;
      if (m < Mp) opS[k * Mp + m] = o[q];
    }
  }
  if (MMA && Kp > K) {
    for (int e = K * Mp + threadIdx.x; e < Kp * Mp; e += blockDim.x) opS[e] = cmk(0.0, 0.0);
    for (int k = K + g; k < Kp; k += G) inS[k * LDI + lane] = cmk(0.0, 0.0);
  }
  const bool use_beta = (a.beta.x != 0.0) || (a.beta.y != 0.0);
  auto put = [&](cd* o, cd acc) {
    cd r = cmul(a.alpha, acc);
    if (use_beta) r = cadd(r, cmul(a.beta, *o));
    *o = r;
  };
  auto product_mma = [&](cd* out) {
    const int fg = lane / 4, ft = lane % 4;
    for (int mb = g * MQ; mb < M; mb += MQ * G) {
      const bool two = mb + 8 < M;   // m tiles of this group
      double re[2][2][4], im[2][2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) re[i][j][e] = im[i][j][e] = 0.0;
      for (int k0 = 0; k0 < Kp; k0 += 8) {
        double br[2][2], bi[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const cd o = opS[(k0 + ft + 4 * e) * Mp + mb + 8 * (two ? j : 0) + fg];
            br[j][e] = o.x; bi[j][e] = o.y;
          }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          double ar[4], ai[4], nai[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const cd u = inS[(k0 + ft + 4 * (e >> 1)) * LDI + 16 * i + fg + 8 * (e & 1)];
            ar[e] = u.x; ai[e] = u.y; nai[e] = -u.y;
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (j == 1 && !two) break;
            dmma16(re[i][j], ar, br[j]);
            dmma16(im[i][j], ar, bi[j]);
            dmma16(re[i][j], nai, bi[j]);
            dmma16(im[i][j], ai, br[j]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int m = mb + 8 * j + 2 * ft + c;
          const int m2 = (int)P.div_m1((unsigned)m), m1 = m - m2 * a.M1;
          cd* om = out + m1 * a.out_m1 + m2 * a.out_m2;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int x = x0 + fg + 8 * i;
            if (m < M && x < a.X)
              put(om + (int64_t)x * a.out_x, cmk(re[i / 2][j][c + 2 * (i % 2)], im[i / 2][j][c + 2 * (i % 2)]));
          }
        }
    }
  };
  auto product_lanes = [&](cd* out) {
    for (int mb = g * MQ; mb < M; mb += MQ * G) {
      cd acc[MQ];
#pragma unroll
      for (int q = 0; q < MQ; ++q) acc[q] = cmk(0.0, 0.0);
#pragma unroll 4
      for (int k = 0; k < K; ++k) {
        const cd u = inS[k * LDI + lane];
#pragma unroll
        for (int q = 0; q < MQ; ++q) cfma(acc[q], u, opS[k * Mp + mb + q]);
      }
#pragma unroll
      for (int q = 0; q < MQ; ++q) {
        const int m = mb + q;
        const int m2 = (int)P.div_m1((unsigned)m), m1 = m - m2 * a.M1;
        if (m < M && x0 + lane < a.X) put(out + (int64_t)(x0 + lane) * a.out_x + m1 * a.out_m1 + m2 * a.out_m2, acc[q]);
      }
    }
  };
  for (int e0 = 32 * g + lane; e0 < n; e0 += LOADS * step) {
    if (e0 >= LOADS * step) load(e0);
    store(e0);
  }
  __syncthreads();
  if (!live) return;
  cd* out = a.out + bz * a.out_b + (int64_t)y * a.out_y;
  if constexpr (MMA) product_mma(out);
  else product_lanes(out);
}

template <int MQ>
auto pick(bool k1_fast) {
  return k1_fast ? mpo_apply_kernel<MQ, true> : mpo_apply_kernel<MQ, false>;
}

}  // namespace

int mpo_apply_launch_strided(const MpoApply& a, int64_t op_k1, int64_t op_k2, int64_t op_m1,
                             int64_t op_m2, cudaStream_t s) {
  if (a.X <= 0 || a.Y <= 0) return MPSB_OK;
  const int K = a.K1 * a.K2, M = a.M1 * a.M2;
  if (K <= 0 || M <= 0) return MPSB_ERR_DIMENSION;
  if ((size_t)K * (M + 64) * sizeof(cd) > 200 * 1024) return MPSB_ERR_UNSUPPORTED;
  if (a.Y > 65535 || a.batch < 1 || a.batch > 65535) return MPSB_ERR_UNSUPPORTED;
  const int nxb = (a.X + 31) / 32;
  if ((int64_t)nxb * a.Y >= (int64_t(1) << 31)) return MPSB_ERR_UNSUPPORTED;
  const int ncols = nxb * a.Y;
  // The tensor path from a warp per SM on (the rule looks at one problem, so a batch computes each
  // problem as a batch of one does); below it and for a small K, which would be mostly padding, as
  // many outputs per lane as leave every SM 8 warps: short warps count there, as the K products of an
  // output are a chain.  (X = Y = 512 as above: 130 us on the tensor path, 150 with 8 outputs per
  // lane, whose reads of Op from shared memory take the time.  One CTA per resident slot that loops
  // over columns, to read Op once: 158, as its loads and products no longer overlap another CTA's.)
  int MQ = K >= 8 && M >= 8 && (int64_t)ncols * ((M + MQ_MMA - 1) / MQ_MMA) >= 148 ? MQ_MMA : 4;
  int Kp = (K + 7) / 8 * 8, Mp = (M + 7) / 8 * 8 + 2;
  if (MQ == MQ_MMA && (size_t)Kp * (Mp + LDI) * sizeof(cd) > 200 * 1024) MQ = 4;
  if (MQ == 4 && (int64_t)ncols * a.batch * ((M + 3) / 4) < 148 * 8) MQ = 2;
  int G = 1;
  while (G < 8 && G * MQ < M) G *= 2;
  if (MQ != MQ_MMA) {
    Kp = K;
    Mp = (M + MQ - 1) / MQ * MQ;
  }
  // columns per CTA: what 8 warps take, fewer while the CTA would hold more than 64 KB
  int CW = 8 / G;
  auto bytes = [&](int cw) { return (size_t)Kp * (Mp + cw * LDI) * sizeof(cd); };
  while (CW > 1 && (bytes(CW) > 64 * 1024 || ncols <= CW / 2)) CW /= 2;
  const bool k1_fast = a.in_k1 == 1 && a.in_x != 1;
  auto fn = MQ == MQ_MMA ? pick<MQ_MMA>(k1_fast) : MQ == 4 ? pick<4>(k1_fast) : pick<2>(k1_fast);
  MPSB_TRY(ensure_kernel_attrs((const void*)fn, 200 * 1024));
  const MpoParams P{a, op_k1, op_k2, op_m1, op_m2, ncols, nxb, G, Mp, Div(K), Div(a.K1), Div(a.M1)};
  fn<<<dim3((unsigned)((ncols + CW - 1) / CW), (unsigned)a.batch), 32 * G * CW, bytes(CW), s>>>(P);
  MPSB_CUDA_TRY(cudaGetLastError());
  return MPSB_OK;
}

int mpo_apply_launch(const MpoApply& a, cudaStream_t s) {
  // dense column-major Op[k, m] with ld = K
  const int K = a.K1 * a.K2;
  return mpo_apply_launch_strided(a, 1, a.K1, K, (int64_t)K * a.M1, s);
}

}  // namespace mpsb
