// Complex128 strided GEMM for the environment / effective-operator contractions.
//
// Every contraction of src/mps_base.jl (prod_AOR GEMM1, prod_LR!, update_re!, update_le!,
// update_renv!, update_lenv!, ...) is a zgemm on reshaped views; here each view is an
// (m, k[, batch]) element-stride triple, so reference transposes ('), (.') and the
// reshape/permutedims chains cost no copies.
//
// Tiling (FP64 tensor path, DMMA): a 32 x 32 complex C tile per 256-thread CTA, as blocks of 16x8 by
// mma.sync.m16n8k8.f64 -- four real products per complex k8 step (Re += Ar Br - Ai Bi,
// Im += Ar Bi + Ai Br) -- with every fragment element loaded as one 16-byte (re, im) pair from
// shared memory.  Two groups of 2 x 2 warps take one k8 step each of every 16-deep stage (so a CTA
// alone on its SM still has two warps per scheduler to hide the fragment loads) and their partial
// tiles are added at the end.  Stages come through a four-deep ring of tiled TMA copies (mbarrier
// byte counts, zero fill outside the matrix) into 128-byte rows of eight elements, 128-byte swizzle;
// a quarter warp's eight 16-byte fragment loads then fall into eight distinct bank groups, for
// either contiguous index.  Problems with few tiles also split K over the CTAs of a thread-block
// cluster, which sum their partial tiles over distributed shared memory.  All sums run in a fixed
// order, so results are bitwise reproducible run to run, and no partial goes through global memory.
// One launch takes up to four problems -- each to its own C, or all into one C, as one long K -- of any
// shapes, layouts and conjugations: a sweep's contractions at one site are many and small, and as
// launches of their own they leave the chip idle and cost 3-5 us each.
//
// What bounds it: the FP64 tensor pipe (64 FMA a clock and SM) on large problems, 33 of 36.8 TFLOP/s;
// a stage's latency (1475 clocks against 1024 of tensor work) where a CTA has its SM alone.  Tiles of
// 64 x 64 were slower at every size measured (fewer CTAs to overlap, and one tile of K = 64 is 8.5 us
// of one SM); copies by the threads' cp.async ran at 12-18 B a clock and SM, 1.3-2 us a stage.
// Against that form with 64 x 64 tiles and split-K partials through global memory (B200): 512 x 2048 x
// 4096 (A along K) 1439 -> 1030 us, 2048 x 512 x 512 178 -> 139, 512 x 512 x 2048 227 -> 156, 128 x 512 x
// 1024 36.6 -> 26.7.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "tma.cuh"
#include "workspace.cuh"

namespace cg = cooperative_groups;

namespace mpsb {

namespace {

constexpr int T = 32, BK = 16, NT = 256, STAGES = 4, SPLIT_MAX = 16;
constexpr int LDS = T + 2, LDP = T + 1;              // row pitch of a copied stage, column pitch of a partial tile
constexpr int OPERAND = T * BK;                      // elements of one operand's TMA stage
constexpr int STAGE = 2 * BK * LDS;                  // elements of a copied stage (A then B)
constexpr int PART = T * LDP;                        // elements of a partial tile
constexpr int CP_STAGES = 3;
constexpr size_t SMEM_TMA = (size_t)STAGES * 2 * OPERAND * sizeof(cd) + 1024 + STAGES * sizeof(uint64_t);
constexpr size_t SMEM_COPY = (size_t)CP_STAGES * STAGE * sizeof(cd);
constexpr int WAIT_LIMIT = 1 << 20;
static_assert(2 * PART <= CP_STAGES * STAGE && 2 * PART <= STAGES * 2 * OPERAND, "the partial tiles reuse the stages");

// One problem as the kernels see it.
struct Prob {
  int M, N, KT;          // KT: stages
  int kt_per_split;      // (of the whole sum when the problems share C)
  int a_free, b_free;    // the operand's contiguous index is its free one
  unsigned a_conj, b_conj;   // sign bit to flip in the imaginary parts' high words
  int a_batch, b_batch;      // the operand has copies of its own
  cd* C;
  int64_t c_m, c_n, c_b;
  cd alpha, beta;
};
struct TmaParams {
  CUtensorMap ma[GEMM_GROUP], mb[GEMM_GROUP];
  Prob p[GEMM_GROUP];
  int n;           // problems
  int* err;        // device error word (may be null)
};
struct CopyParams {
  Gemm g;
  Prob p;
};

// The sum of the groups' (and, over the cluster, the splits') partial tiles, C = alpha sum + beta C.
// Accumulator (j, e): row wm + 8(e/2) + fg, column wn + 8j + 2ft + e%2 of the group's partial tile.
__device__ __forceinline__ void finish_tile(const Prob& p, cd* smem, const double (&cr)[2][4], const double (&ci)[2][4],
                                            int m0, int n0, int copy) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, split = blockIdx.y, splits = gridDim.y;
  const int wm = (warp & 1) * 16, wn = ((warp >> 1) & 1) * 16, fg = lane >> 2, ft = lane & 3;
  cd* part = smem + (warp >> 2) * PART;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      part[(wn + 8 * j + 2 * ft + (e & 1)) * LDP + wm + 8 * (e >> 1) + fg] = cmk(cr[j][e], ci[j][e]);
  cg::cluster_group cluster = cg::this_cluster();
  if (splits > 1) cluster.sync();
  else __syncthreads();
  // rank r sums columns r, r + splits, ... of the tile over the ranks' groups in order
  cd* C = p.C + (int64_t)copy * p.c_b;
  const cd alpha = p.alpha, beta = p.beta;
  const bool use_beta = (beta.x != 0.0) || (beta.y != 0.0);
  const int m = tid % T;
  if (m0 + m < p.M) {
    for (int n = split + splits * (tid / T); n < T && n0 + n < p.N; n += splits * (NT / T)) {
      cd* src = &smem[n * LDP + m];
      cd v;
      if (splits > 1) {
        v = cmk(0.0, 0.0);
#pragma unroll 4
        for (int q = 0; q < splits; ++q) {
          const cd* rs = cluster.map_shared_rank(src, q);
          v = cadd(v, cadd(rs[0], rs[PART]));
        }
      } else {
        v = cadd(src[0], src[PART]);
      }
      cd* c = C + (int64_t)(m0 + m) * p.c_m + (int64_t)(n0 + n) * p.c_n;
      v = cmul(alpha, v);
      if (use_beta) v = cadd(v, cmul(beta, *c));
      *c = v;
    }
  }
  if (splits > 1) cluster.sync();   // no CTA leaves while a peer reads its partials
}

// One complex k8 step of a warp's 16 x 16 block.  Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br, term-major
// so one accumulator's two products sit four issues apart.
__device__ __forceinline__ void mma_k8(double (&cr)[2][4], double (&ci)[2][4], const cd (&a)[4], const cd (&b)[2][2],
                                       unsigned conjA, unsigned conjB) {
  auto flip = [](double x, unsigned bit) { return __hiloint2double((int)((unsigned)__double2hiint(x) ^ bit), __double2loint(x)); };
  double ar[4], ai[4], nai[4], br[2][2], bi[2][2];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    ar[e] = a[e].x;
    ai[e] = flip(a[e].y, conjA);
    nai[e] = flip(a[e].y, conjA ^ 0x80000000u);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      br[j][e] = b[j][e].x;
      bi[j][e] = flip(b[j][e].y, conjB);
    }
#pragma unroll
  for (int j = 0; j < 2; ++j) dmma16(cr[j], ar, br[j]);
#pragma unroll
  for (int j = 0; j < 2; ++j) dmma16(ci[j], ar, bi[j]);
#pragma unroll
  for (int j = 0; j < 2; ++j) dmma16(cr[j], nai, bi[j]);
#pragma unroll
  for (int j = 0; j < 2; ++j) dmma16(ci[j], ai, br[j]);
}

__device__ __forceinline__ uint32_t su32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {   // bounded
  for (int it = 0; it < WAIT_LIMIT; ++it) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}

// An operand's 32 x 16 stage: free index contiguous -- four boxes of 8 (free) x 16 (k), box g at g * 2 KB,
// a row per k; k contiguous -- two boxes of 8 (k) x 32 (free), box h at h * 4 KB, a row per free
// index.  Chunk c of row r sits at c ^ (r mod 8).
__device__ __forceinline__ void tma_stage(bool free_contig, uint32_t dst, const CUtensorMap* map, uint32_t bar, int f0, int k0,
                                          int b) {
  const int y = free_contig ? k0 : f0, x = 2 * (free_contig ? f0 : k0);
  const uint32_t step = free_contig ? 2048 : 4096;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q < 2 || free_contig) asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::
                     "r"(dst + q * step), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x + 16 * q), "r"(y), "r"(b) : "memory");
}

// blockIdx: x the tile, y the split (a cluster), z copy * n + problem, or the copy when the problems share C.
// LAYOUT: bit 0 a_free, bit 1 b_free of every problem; ANY: the problems differ (the layout is then read per
// stage, 5 % slower).
constexpr int ANY = 4;
template <int LAYOUT, bool SUM>
__global__ void __launch_bounds__(NT, 3) zgemm_tma_kernel(const __grid_constant__ TmaParams P) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t OP_BYTES = OPERAND * sizeof(cd);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gz = SUM || P.n == 1 ? 0 : blockIdx.z % P.n, copy = SUM || P.n == 1 ? blockIdx.z : blockIdx.z / P.n;
  const Prob& p = P.p[gz];
  const int tiles_m = (p.M + T - 1) / T;
  if ((int)blockIdx.x >= tiles_m * ((p.N + T - 1) / T)) return;   // a smaller problem of the launch (the whole cluster)
  const int m0 = (blockIdx.x % tiles_m) * T, n0 = (blockIdx.x / tiles_m) * T;
  // stages kt0 .. kt0 + nkt - 1 of the problem, or of the problems' stages one after the other
  int KT = p.KT;
  if (SUM)
    for (int q = 1; q < P.n; ++q) KT += P.p[q].KT;
  const int kt0 = blockIdx.y * p.kt_per_split, nkt = max(0, min(KT, kt0 + p.kt_per_split) - kt0);
  int g0 = gz, l0 = kt0;   // problem and its stage of this CTA's first stage
  if (SUM)
    while (g0 + 1 < P.n && l0 >= P.p[g0].KT) l0 -= P.p[g0++].KT;
  const uint32_t ring32 = su32(ring), bars = ring32 + STAGES * 2 * OP_BYTES;
  auto a_free = [](const Prob& q) { return LAYOUT == ANY ? q.a_free != 0 : (LAYOUT & 1) != 0; };
  auto b_free = [](const Prob& q) { return LAYOUT == ANY ? q.b_free != 0 : (LAYOUT & 2) != 0; };

  int ig = g0, il = l0, it = 0;   // thread 0: the next stage to load
  auto issue = [&]() {
    const Prob& q = SUM ? P.p[ig] : p;
    const uint32_t bar = bars + 8 * (it % STAGES), dst = ring32 + (it % STAGES) * 2 * OP_BYTES;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2 * OP_BYTES) : "memory");
    tma_stage(a_free(q), dst, &P.ma[SUM ? ig : gz], bar, m0, il * BK, q.a_batch ? copy : 0);
    tma_stage(b_free(q), dst + OP_BYTES, &P.mb[SUM ? ig : gz], bar, n0, il * BK, q.b_batch ? copy : 0);
    ++it;
    ++il;
    if (SUM && il >= q.KT) { il = 0; ++ig; }
  };
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int t = 0; t < STAGES - 1 && t < nkt; ++t) issue();
  }
  __syncthreads();

  // this warp's fragments: k index t <-> row 2 t of its half stage, t + 4 <-> 2 t + 1
  const int grp = warp >> 2, wm = (warp & 1) * 16, wn = ((warp >> 1) & 1) * 16, fg = lane >> 2, ft = lane & 3;
  uint32_t oa[2], ob[2], fa, fb;   // of k rows 2 ft and 2 ft + 1; to 8 free indices on
  unsigned sa_conj, sb_conj;
  auto layout = [&](const Prob& q) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t k = 8 * grp + 2 * ft + h, c = (uint32_t)((2 * ft + h) ^ fg) << 4;
      oa[h] = c + (a_free(q) ? (wm >> 3) * 2048 + k * 128 : grp * 4096 + (wm + fg) * 128);
      ob[h] = c + (b_free(q) ? (wn >> 3) * 2048 + k * 128 : grp * 4096 + (wn + fg) * 128);
    }
    fa = a_free(q) ? 2048 : 8 * 128;
    fb = b_free(q) ? 2048 : 8 * 128;
    sa_conj = q.a_conj;
    sb_conj = q.b_conj;
  };
  layout(P.p[g0]);
  int cg_ = g0, cl = l0;   // problem and its stage being computed
  double cr[2][4], ci[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) cr[j][e] = ci[j][e] = 0.0;
  bool failed = false;
#pragma unroll 1
  for (int t = 0; t < nkt; ++t) {
    if (!failed && !bar_wait(bars + 8 * (t % STAGES), (uint32_t)(t / STAGES) & 1)) {
      failed = true;
      if (P.err) atomicOr(P.err, 8);
    }
    __syncthreads();   // every warp is done with the slot of stage t - 1
    if (tid == 0 && t + STAGES - 1 < nkt && !failed) issue();
    if (SUM) {
      if (cl >= P.p[cg_].KT) {
        cl = 0;
        layout(P.p[++cg_]);
      }
      ++cl;
    }
    const unsigned char* sa = ring + (t % STAGES) * 2 * OP_BYTES;
    const unsigned char* sb = sa + OP_BYTES;
    cd a[4], b[2][2];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = *reinterpret_cast<const cd*>(sa + oa[e >> 1] + (e & 1) * fa);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) b[j][e] = *reinterpret_cast<const cd*>(sb + ob[e] + j * fb);
    mma_k8(cr, ci, a, b, sa_conj, sb_conj);
  }
  if (failed && tid == 0) {   // the copies in flight land (or the bound ends) before the CTA goes away
    for (int t = max(0, it - STAGES); t < it; ++t) bar_wait(bars + 8 * (t % STAGES), (uint32_t)(t / STAGES) & 1);
  }
  __syncthreads();   // every warp is done with the stages
  finish_tile(p, reinterpret_cast<cd*>(ring), cr, ci, m0, n0, copy);
}

// The same tile with stages copied by the threads, for operands that a tensor map does not describe
// (neither index contiguous, or a stride outside its range).
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// One operand's stages (T x 16, stored [k][free]), zero outside the matrix: this thread's two elements
// of a stage are p and p + di, and p moves by dk per stage.
struct Stream {
  const cd* base;
  const cd* p;
  int64_t di, dk;
  unsigned dst;   // byte offset in the stage
  int k;          // this thread's k in a stage
  bool in;        // its free index is inside
  __device__ Stream(const cd* b, int64_t s_free, int64_t s_k, int f0, int extent, int k0, int tid) : base(b) {
    const int f = tid % T;
    k = tid / T;
    p = b + (int64_t)(f0 + f) * s_free + (int64_t)(k0 + k) * s_k;
    di = (NT / T) * s_k;
    dk = BK * s_k;
    dst = (unsigned)((k * LDS + f) * sizeof(cd));
    in = f0 + f < extent;
  }
  __device__ __forceinline__ void load(unsigned st, int krem) {   // krem: the matrix's k extent from this stage on
#pragma unroll
    for (int i = 0; i < T * BK / NT; ++i) {
      const bool ok = in && k + i * (NT / T) < krem;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(st + dst + i * (unsigned)((NT / T) * LDS * sizeof(cd))),
                   "l"(ok ? p + i * di : base), "r"(ok ? 16 : 0));
    }
    p += dk;
  }
};

__global__ void __launch_bounds__(NT, 3) zgemm_copy_kernel(CopyParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* smem = reinterpret_cast<cd*>(smem_raw);
  const Gemm& g = P.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles_m = (g.M + T - 1) / T;
  const int m0 = (blockIdx.x % tiles_m) * T, n0 = (blockIdx.x / tiles_m) * T;
  const int kt0 = blockIdx.y * P.p.kt_per_split, nkt = max(0, min(P.p.KT, kt0 + P.p.kt_per_split) - kt0);
  const int krem = g.K - kt0 * BK;
  const int k8 = 8 * (warp >> 2);                              // this group's half of a stage
  const int wm = (warp & 1) * 16, wn = ((warp >> 1) & 1) * 16, fg = lane >> 2, ft = lane & 3;
  double cr[2][4], ci[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) cr[j][e] = ci[j][e] = 0.0;

  Stream sa(g.A + (int64_t)blockIdx.z * g.a_b, g.a_m, g.a_k, m0, g.M, kt0 * BK, tid);
  Stream sb(g.B + (int64_t)blockIdx.z * g.b_b, g.b_n, g.b_k, n0, g.N, kt0 * BK, tid);
  auto refill = [&](int t) {
    if (t < nkt) {
      const unsigned st = su32(smem + (t % CP_STAGES) * STAGE);
      sa.load(st, krem - t * BK);
      sb.load(st + (unsigned)(BK * LDS * sizeof(cd)), krem - t * BK);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int t = 0; t < CP_STAGES - 1; ++t) refill(t);
#pragma unroll 1
  for (int t = 0; t < nkt; ++t) {
    cp_async_wait<CP_STAGES - 2>();
    __syncthreads();
    refill(t + CP_STAGES - 1);   // the slot consumed in the last iteration
    const cd* As = smem + (t % CP_STAGES) * STAGE + (k8 + ft) * LDS + wm + fg;
    const cd* Bs = smem + (t % CP_STAGES) * STAGE + BK * LDS + (k8 + ft) * LDS + wn + fg;
    cd a[4], b[2][2];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = As[4 * (e >> 1) * LDS + 8 * (e & 1)];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) b[j][e] = Bs[4 * e * LDS + 8 * j];
    mma_k8(cr, ci, a, b, P.p.a_conj, P.p.b_conj);
  }
  cp_async_wait<0>();
  __syncthreads();   // every warp is done with the stages
  finish_tile(P.p, smem, cr, ci, m0, n0, blockIdx.z);
}

__global__ void scale_c_kernel(Gemm g) {
  // K == 0: C = beta * C
  const int64_t MN = (int64_t)g.M * g.N, total = MN * g.batch;
  const bool use_beta = (g.beta.x != 0.0) || (g.beta.y != 0.0);
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t b = idx / MN, r = idx % MN;
    int m = (int)(r % g.M), n = (int)(r / g.M);
    cd* c = g.C + b * g.c_b + (int64_t)m * g.c_m + (int64_t)n * g.c_n;
    *c = use_beta ? cmul(g.beta, *c) : cmk(0.0, 0.0);
  }
}

// The tensor map of an operand (free x K, copies s_b apart), as doubles: the contiguous index (two
// doubles an element), the other one, the copy.  False when a map does not describe it.
bool operand_map(CUtensorMap* map, const cd* p, int64_t extent, int64_t s_free, int64_t K, int64_t s_k, int batch, int64_t s_b,
                 bool* free_contig) {
  // an index of extent 1 is contiguous whatever its stride
  *free_contig = s_free == 1 || (extent == 1 && s_k != 1);
  if (!*free_contig && s_k != 1 && K != 1) return false;
  const int64_t n0 = *free_contig ? extent : K, n1 = *free_contig ? K : extent;
  int64_t s1 = *free_contig ? s_k : s_free;
  if (n1 == 1) s1 = n0;
  if (s_b == 0) { batch = 1; s_b = 1; }
  const int64_t most = (int64_t)1 << 35;   // strides below 2^40 bytes, extents below 2^32
  if (s1 < 1 || s1 >= most || s_b < 1 || s_b >= most || (reinterpret_cast<uintptr_t>(p) & 15)) return false;
  cuuint64_t dims[3] = {(cuuint64_t)(2 * n0), (cuuint64_t)n1, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)s1 * sizeof(cd), (cuuint64_t)s_b * sizeof(cd)};
  cuuint32_t box[3] = {16, (cuuint32_t)(*free_contig ? BK : T), 1}, estr[3] = {1, 1, 1};
  const auto encode = tensor_map_encoder();
  return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<cd*>(p), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// K splits for `tiles` tiles of KT stages.  Measured on a B200: a stage takes 1475 clocks in a CTA alone
// on its SM and 1090 (the FP64 tensor pipe's rate) beside others; a CTA costs 3000 clocks around its
// stages, 5000 with the cluster's sum, about half of it hidden behind its SM's other CTAs.  E.g. 128 x
// 512 x 1024 (64 tiles): 51.2 / 28.8 / 26.7 / 32.9 us at 1 / 2 / 4 / 8 splits; 512 x 1024 x 128 (512
// tiles) 30.4 / 32.5 / 42.2.
int choose_splits(double tiles, int KT) {
  int best = 1;
  double tbest = 1e300;
  for (int s = 1; s <= SPLIT_MAX && (s == 1 || KT >= 2 * s); ++s) {
    const double w = std::ceil(tiles * s / 148.0), stages = (KT + s - 1) / s;
    const double ov = s > 1 ? 5000.0 : 3000.0;
    const double t = w <= 1.0 ? stages * 1475.0 + ov : w * stages * 1090.0 + ov * (1.0 + 0.5 * (w - 1.0));
    if (t < tbest) { tbest = t; best = s; }
  }
  return best;
}

}  // namespace

static Prob prob_of(const Gemm& g) {
  Prob p = {};
  p.M = g.M; p.N = g.N; p.KT = (g.K + BK - 1) / BK;
  p.a_conj = g.conjA ? 0x80000000u : 0u; p.b_conj = g.conjB ? 0x80000000u : 0u;
  p.a_batch = g.a_b != 0; p.b_batch = g.b_b != 0;
  p.C = g.C; p.c_m = g.c_m; p.c_n = g.c_n; p.c_b = g.c_b;
  p.alpha = g.alpha; p.beta = g.beta;
  return p;
}

static int tiles_of(const Gemm& g) { return ((g.M + T - 1) / T) * ((g.N + T - 1) / T); }

static int launch(const void* fn, void* params, size_t smem, int tiles, int splits, int z, cudaStream_t s) {
  MPSB_TRY(ensure_kernel_attrs(fn, (int)smem, true));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, splits, z);
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = splits;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  void* args[1] = {params};
  MPSB_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, args));
  return MPSB_OK;
}

int gemm_launch(const Gemm& g, Workspace* ws, cudaStream_t s) { return gemm_group_launch(&g, 1, false, ws, s); }

int gemm_group_launch(const Gemm* g, int n, bool sum, Workspace* ws, cudaStream_t s) {
  if (n < 1 || n > GEMM_GROUP) return MPSB_ERR_INVALID_ARG;
  for (int q = 0; q < n; ++q) {
    if (g[q].M < 0 || g[q].N < 0 || g[q].K < 0 || g[q].batch < 1) return MPSB_ERR_DIMENSION;
    if ((int64_t)g[q].batch * n > 65535) return n > 1 ? MPSB_ERR_INVALID_ARG : MPSB_ERR_UNSUPPORTED;
  }
  // a problem without a product, or with an operand that a tensor map does not describe, goes alone
  TmaParams P = {};
  bool tma = true;
  for (int q = 0; q < n && tma; ++q) {
    const Gemm& x = g[q];
    bool af, bf;
    tma = x.M > 0 && x.N > 0 && x.K > 0 && x.batch == g[0].batch &&
          operand_map(&P.ma[q], x.A, x.M, x.a_m, x.K, x.a_k, x.batch, x.a_b, &af) &&
          operand_map(&P.mb[q], x.B, x.N, x.b_n, x.K, x.b_k, x.batch, x.b_b, &bf);
    if (!tma) break;
    P.p[q] = prob_of(x);
    P.p[q].a_free = af;
    P.p[q].b_free = bf;
  }
  if (!tma && n > 1) {
    for (int q = 0; q < n; ++q) {
      Gemm x = g[q];
      if (sum && q > 0) x.beta = cmk(1.0, 0.0);
      MPSB_TRY(gemm_group_launch(&x, 1, false, ws, s));
    }
    return MPSB_OK;
  }
  if (g[0].M == 0 || g[0].N == 0) return MPSB_OK;
  count_launch(ws);
  if (g[0].K == 0) {
    int64_t total = (int64_t)g[0].M * g[0].N * g[0].batch;
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 8);
    scale_c_kernel<<<blocks, 256, 0, s>>>(g[0]);
    MPSB_CUDA_TRY(cudaGetLastError());
    return MPSB_OK;
  }
  // K splits: the launch's tiles, and the longest K (the whole sum's when the problems share C).  In
  // batched mode the partition must not depend on the number of copies: it is that of four, the usual
  // bucket's order (the copies fill the chip, so splitting for one only adds sums).  Without a
  // workspace (ws == nullptr) K is not split.
  int tiles = 0, all = 0, KT = 0;
  for (int q = 0; q < n; ++q) {
    const int kt = (g[q].K + BK - 1) / BK;
    tiles = std::max(tiles, tiles_of(g[q]));
    all = sum ? tiles : all + tiles_of(g[q]);
    KT = sum ? KT + kt : std::max(KT, kt);
  }
  int splits = ws ? choose_splits((double)all * (ws->per_problem ? 4 : g[0].batch), KT) : 1;
  splits = (KT + (KT + splits - 1) / splits - 1) / ((KT + splits - 1) / splits);
  auto per_split = [&](int kt) { return (kt + splits - 1) / splits; };
  if (!tma) {
    CopyParams Q;
    Q.g = g[0];
    Q.p = prob_of(g[0]);
    Q.p.kt_per_split = per_split(KT);
    return launch((const void*)zgemm_copy_kernel, &Q, SMEM_COPY, tiles, splits, g[0].batch, s);
  }
  P.n = n;
  P.err = ws ? ws->err : nullptr;
  for (int q = 0; q < n; ++q) P.p[q].kt_per_split = per_split(sum ? KT : P.p[q].KT);
  int layout = P.p[0].a_free + 2 * P.p[0].b_free;
  for (int q = 1; q < n; ++q)
    if (P.p[q].a_free + 2 * P.p[q].b_free != layout) layout = ANY;
  static const void* const kernels[2][5] = {
      {(const void*)zgemm_tma_kernel<0, false>, (const void*)zgemm_tma_kernel<1, false>, (const void*)zgemm_tma_kernel<2, false>,
       (const void*)zgemm_tma_kernel<3, false>, (const void*)zgemm_tma_kernel<ANY, false>},
      {(const void*)zgemm_tma_kernel<0, true>, (const void*)zgemm_tma_kernel<1, true>, (const void*)zgemm_tma_kernel<2, true>,
       (const void*)zgemm_tma_kernel<3, true>, (const void*)zgemm_tma_kernel<ANY, true>}};
  return launch(kernels[sum && n > 1][layout], &P, SMEM_TMA, tiles, splits, sum ? g[0].batch : g[0].batch * n, s);
}

}  // namespace mpsb
