// scal_prod / scal_prod_no_conj (src/MatrixProductStates.jl:345-379) of a product MPS (every bond 1, the
// form of a measurement functional: the trace, a local population, a correlation) with an MPS: the
// whole chain of vector-matrix products
//     v'[b] = sum_{a, s} v[a] f_k[s] B_k[a, s, b]
// in one launch of one thread-block cluster.
//
// Site k is a matrix-vector product with u = v (x) f over rows r = (a, s), the fastest index of B_k, so
// a CTA's slice of columns b is one contiguous block of the slab.  Those blocks do not depend on v:
// thread 0 streams the CTA's blocks of all sites through a ring of bulk copies, sites ahead of the
// arithmetic.  A warp's lanes take a column's rows (up to eight warps share a column when a ring slot
// holds few), the CTA's part of v' goes to every CTA by remote stores, and one cluster barrier ends
// the site.
//
// What bounds it: a site's chain u -> sums -> remote stores -> cluster barrier, about 3 us; the 1 MB of
// a chi = 128, d = 4 site passes underneath.  40 sites at chi = 128, d = 4, read-back included: 143 us
// against 495 us for two GEMM launches per site (M or N = 1).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "misc.cuh"

namespace cg = cooperative_groups;

namespace mpsb {
namespace {

constexpr int NT = 256, NW = NT / 32, C = 16, NSLOT = 4;
constexpr int ROWS = 2048;            // elements of a ring slot; rows of a site at most
constexpr int CHI = 512, SITES = 256, FUN = 1024;   // bond, chain and functional entries at most
constexpr int WAIT_LIMIT = 1 << 20;

struct ChainParams {
  const cd* f;    // [na][d]
  const cd* B;
  cd* out;
  int* err;
  int na, d, conj;
  int dims[SITES + 1];
};

struct Smem {
  cd ring[NSLOT][ROWS];
  cd u[ROWS];
  cd v[2][CHI];
  cd f[FUN];
  cd part[CHI / C][NW];
  uint64_t full[NSLOT];
};

__device__ __forceinline__ uint32_t su32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__global__ void __launch_bounds__(NT, 1) chain_kernel(const __grid_constant__ ChainParams P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster.block_rank();
  const int na = P.na, d = P.d;

  // this CTA's columns of site k, and the columns of one ring slot
  auto first = [&](int k) { const int n = P.dims[k + 1]; return min(n, rank * ((n + C - 1) / C)); };
  auto last = [&](int k) { const int n = P.dims[k + 1]; return min(n, (rank + 1) * ((n + C - 1) / C)); };
  auto rows = [&](int k) { return P.dims[k] * d; };

  // thread 0: the next block of columns into ring slot `issued % NSLOT`
  int pk = 0, pcol = first(0), issued = 0;
  int64_t poff = 0;
  auto issue = [&]() {
    while (pk < na && pcol >= last(pk)) {
      poff += (int64_t)rows(pk) * P.dims[pk + 1];
      if (++pk < na) pcol = first(pk);
    }
    if (pk == na) return;
    const int L = rows(pk), n = min(ROWS / L, last(pk) - pcol);
    const uint32_t bar = su32(&S.full[issued % NSLOT]), bytes = (uint32_t)(n * L * sizeof(cd));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                     "r"(su32(S.ring[issued % NSLOT])), "l"(P.B + poff + (int64_t)pcol * L), "r"(bytes), "r"(bar) : "memory");
    pcol += n;
    ++issued;
  };
  if (tid == 0) {
    for (int i = 0; i < NSLOT; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&S.full[i])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int i = 0; i < NSLOT; ++i) issue();
    S.v[0][0] = cmk(1.0, 0.0);
  }
  for (int i = tid; i < na * d; i += NT) {
    const cd x = P.f[i];
    S.f[i] = P.conj ? cconj(x) : x;
  }
  cluster.sync();

  int used = 0;   // ring slots consumed
  bool failed = false;
  for (int k = 0; k < na; ++k) {
    const int L = rows(k), chiL = P.dims[k], c0 = first(k), c1 = last(k), per = ROWS / L;
    if (c1 > c0) {
      const cd* v = S.v[k & 1];
      for (int a = tid; a < chiL; a += NT) {
        const cd x = v[a];
        for (int s = 0; s < d; ++s) S.u[s * chiL + a] = cmul(x, S.f[k * d + s]);
      }
      __syncthreads();
    }
    // warps per column: all eight when a slot holds one, one when it holds eight or more
    const int lw = per >= 8 ? 0 : (per >= 4 ? 1 : (per >= 2 ? 2 : 3)), wpc = 1 << lw, wsub = warp & (wpc - 1);
    for (int col = c0; col < c1; col += per, ++used) {
      const int n = min(per, c1 - col);
      const uint32_t bar = su32(&S.full[used % NSLOT]);
      for (int it = 0; !failed; ++it) {   // bounded
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(bar), "r"((uint32_t)(used / NSLOT) & 1) : "memory");
        if (ok) break;
        if (it >= WAIT_LIMIT) {
          failed = true;
          if (P.err) atomicOr(P.err, 8);
        }
      }
      for (int j = warp >> lw; j < n; j += NW >> lw) {
        const cd* b = S.ring[used % NSLOT] + j * L;
        cd s0 = cmk(0.0, 0.0), s1 = cmk(0.0, 0.0);
        int r = wsub * 32 + lane;
        for (; r + 32 * wpc < L; r += 64 * wpc) {
          cfma(s0, S.u[r], b[r]);
          cfma(s1, S.u[r + 32 * wpc], b[r + 32 * wpc]);
        }
        if (r < L) cfma(s0, S.u[r], b[r]);
        cd s = cadd(s0, s1);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          s.x += __shfl_xor_sync(0xffffffffu, s.x, off);
          s.y += __shfl_xor_sync(0xffffffffu, s.y, off);
        }
        if (lane == 0) S.part[col - c0 + j][wsub] = s;
      }
      __syncthreads();   // the slot is consumed
      if (tid == 0 && !failed) issue();
    }
    // this CTA's entries of v' to every CTA
    const int nb = c1 - c0;
    {
      const int q = tid / (NT / C);   // sixteen threads per rank
      for (int j = tid % (NT / C); j < nb; j += NT / C) {
        cd s = S.part[j][0];
        for (int w = 1; w < wpc; ++w) s = cadd(s, S.part[j][w]);
        *cluster.map_shared_rank(&S.v[(k + 1) & 1][c0 + j], q) = s;
        if (k == na - 1 && q == 0) *P.out = s;   // the last bond is 1
      }
    }
    cluster.sync();
  }
  if (failed && tid == 0)   // let the copies in flight land (bounded) before the CTA goes away
    for (int i = 0; i < WAIT_LIMIT && i >= 0; ++i) __nanosleep(1);
}

}  // namespace

// Whether chain_product takes these bonds.
bool chain_supported(int na, int d, const int64_t* dims) {
  if (na < 1 || na > SITES || d < 1 || (int64_t)na * d > FUN || dims[na] != 1) return false;
  for (int k = 0; k <= na; ++k)
    if (dims[k] < 1 || dims[k] > CHI) return false;
  for (int k = 0; k < na; ++k)
    if (dims[k] * d > ROWS) return false;
  return true;
}

// *out (device) = sum over all indices of f (conjugated when conj) times the MPS in slab B
int chain_product(const cd* f, const cd* B, int na, int d, const int64_t* dims, bool conj, cd* out, int* err,
                  cudaStream_t s) {
  ChainParams P;
  P.f = f; P.B = B; P.out = out; P.err = err;
  P.na = na; P.d = d; P.conj = conj;
  for (int k = 0; k <= na; ++k) P.dims[k] = (int)dims[k];
  MPSB_TRY(ensure_kernel_attrs((const void*)chain_kernel, (int)sizeof(Smem), true));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C, 1, 1);
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = sizeof(Smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MPSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, chain_kernel, P));
  return MPSB_OK;
}

}  // namespace mpsb
