// scal_prod / scal_prod_no_conj (src/MatrixProductStates.jl:345-379) of a product MPS (every bond 1, the
// form of a measurement functional: the trace, a local population, a correlation) with an MPS: the
// whole chain of vector-matrix products
//     v'[b] = sum_{a, s} v[a] f_k[s] B_k[a, s, b]
// in one launch of one thread-block cluster.
//
// Site k is a matrix-vector product with u = v (x) f over rows r = (a, s), the fastest index of B_k, so
// a CTA's slice of columns b is one contiguous block of the slab.  Those blocks do not depend on v:
// thread 0 streams the CTA's blocks of all sites through a ring of bulk copies, sites ahead of the
// arithmetic.  A warp takes a column and pushes its entry of v' to every CTA with st.async, counted on
// the receiver's mbarrier, which is the site's only synchronisation between CTAs; sites whose blocks
// take more than half of the ring go slot by slot (up to eight warps share a column there).
//
// What bounds it: a site's chain u -> sums -> exchange, about 2.2 us; the 1 MB of a chi = 128, d = 4 site
// passes underneath.  40 sites at chi = 128, d = 4, read-back included: 105 us, against 143 with a
// cluster barrier per site and the slots one by one, and 495 for two GEMM launches per site (M or
// N = 1).
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
  uint64_t full[NSLOT], vfull[2];
};

__device__ __forceinline__ uint32_t su32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint32_t mapa(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void expect(uint64_t* m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(m)), "r"(bytes) : "memory");
}
// bounded
__device__ __forceinline__ void wait(uint64_t* m, uint32_t parity, bool& failed, int* err) {
  for (int it = 0; !failed; ++it) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(su32(m)), "r"(parity) : "memory");
    if (ok) return;
    if (it >= WAIT_LIMIT) {
      failed = true;
      if (err) atomicOr(err, 8);
    }
  }
}

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
    expect(&S.full[issued % NSLOT], bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                     "r"(su32(S.ring[issued % NSLOT])), "l"(P.B + poff + (int64_t)pcol * L), "r"(bytes), "r"(bar) : "memory");
    pcol += n;
    ++issued;
  };
  if (tid == 0) {
    for (int i = 0; i < NSLOT; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&S.full[i])) : "memory");
    for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&S.vfull[i])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int j = 1; j <= 2 && j < na; ++j) expect(&S.vfull[j & 1], (uint32_t)(P.dims[j] * sizeof(cd)));
    for (int i = 0; i < NSLOT; ++i) issue();
    S.v[0][0] = cmk(1.0, 0.0);
  }
  for (int i = tid; i < na * d; i += NT) {
    const cd x = P.f[i];
    S.f[i] = P.conj ? cconj(x) : x;
  }
  cluster.sync();

  // An entry of v_{k+1} to rank q (the last bond is 1 and goes out).  A peer's v_{k+2} overwrites v_k
  // after it has all of v_{k+1}, so after this CTA has read v_k, and u and the ring of site k.
  auto push = [&](int k, int col, cd x, int q) {
    if (k + 1 == na) {
      if (q == 0) *P.out = x;
      return;
    }
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::
                     "r"(mapa(su32(&S.v[(k + 1) & 1][col]), q)), "l"(__double_as_longlong(x.x)), "l"(__double_as_longlong(x.y)),
                     "r"(mapa(su32(&S.vfull[(k + 1) & 1]), q)) : "memory");
  };
  int used = 0, owed = 0;   // ring slots consumed; of these not yet refilled
  bool failed = false;
  for (int k = 0; k < na; ++k) {
    const int L = rows(k), chiL = P.dims[k], c0 = first(k), nb = last(k) - c0, per = ROWS / L;
    if (k > 0) wait(&S.vfull[k & 1], (uint32_t)((k - 1) >> 1) & 1, failed, P.err);
    if (nb > 0) {
      const cd* v = S.v[k & 1];
      for (int a = tid; a < chiL; a += NT) {
        const cd x = v[a];
        for (int s = 0; s < d; ++s) S.u[s * chiL + a] = cmul(x, S.f[k * d + s]);
      }
    }
    __syncthreads();
    if (tid == 0 && !failed) {
      if (k > 0 && k + 2 < na) expect(&S.vfull[k & 1], (uint32_t)(P.dims[k + 2] * sizeof(cd)));
      for (int i = 0; i < owed; ++i) issue();
    }
    owed = 0;
    const int slots = (nb + per - 1) / per;
    auto dot = [&](const cd* b, int r, int step) {   // this warp's part of a column: rows r, r + step, ...
      cd s0 = cmk(0.0, 0.0), s1 = cmk(0.0, 0.0);
      for (; r + step < L; r += 2 * step) {
        cfma(s0, S.u[r], b[r]);
        cfma(s1, S.u[r + step], b[r + step]);
      }
      if (r < L) cfma(s0, S.u[r], b[r]);
      cd s = cadd(s0, s1);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, off);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, off);
      }
      return s;
    };
    if (slots <= NSLOT / 2) {
      // a warp per column, which pushes it; the slots are refilled at the next site
      for (int j = warp; j < nb; j += NW) {
        const int sl = used + j / per;
        wait(&S.full[sl % NSLOT], (uint32_t)(sl / NSLOT) & 1, failed, P.err);
        const cd s = dot(S.ring[sl % NSLOT] + (j % per) * L, lane, 32);
        if (lane < C) push(k, c0 + j, s, lane);
      }
      used += slots;
      owed = slots;
    } else {
      // slot by slot, each refilled when it is consumed; warps per column: all eight when a slot holds
      // one, one when it holds eight or more
      const int lw = per >= 8 ? 0 : (per >= 4 ? 1 : (per >= 2 ? 2 : 3)), wpc = 1 << lw, wsub = warp & (wpc - 1);
      for (int col = 0; col < nb; col += per, ++used) {
        const int n = min(per, nb - col);
        wait(&S.full[used % NSLOT], (uint32_t)(used / NSLOT) & 1, failed, P.err);
        for (int j = warp >> lw; j < n; j += NW >> lw) {
          const cd s = dot(S.ring[used % NSLOT] + j * L, wsub * 32 + lane, 32 * wpc);
          if (lane == 0) S.part[col + j][wsub] = s;
        }
        __syncthreads();   // the slot is consumed
        if (tid == 0 && !failed) issue();
      }
      for (int j = tid % (NT / C); j < nb; j += NT / C) {   // sixteen threads per rank
        cd s = S.part[j][0];
        for (int w = 1; w < wpc; ++w) s = cadd(s, S.part[j][w]);
        push(k, c0 + j, s, tid / (NT / C));
      }
    }
  }
  cluster.sync();
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
