// Householder QR with the LAPACK zgeqrf + zungqr conventions (the routines qrq! calls,
// src/orthonormalisation.jl:180-184), Q (and optionally R) of an m x n complex matrix, m >= n.
//
// Reflector convention (zlarfg): for column j with alpha = A[j,j] and x = A[j+1:m, j],
//   if x == 0 and Im(alpha) == 0:  tau = 0 (H = I, R[j,j] = alpha)
//   else beta = -copysign(|(alpha, x)|, Re alpha), tau = (beta - alpha)/beta,
//        v = [1; x/(alpha - beta)], R[j,j] = beta (real)
// H(j)^H = I - conj(tau) v v^H is applied to the trailing columns (zgeqr2), and
// Q = H(1)...H(n) [I; 0] (zungqr).  Only the span of Q carries physics in the sweeps; the
// sign / phase rule above is what must match LAPACK, and it also fixes the "junk" columns of
// zero-padded (rank-deficient) sites.
//
// Range: the sums behind |x|, v^H a and V^H x are taken on x scaled by 2^-e, e the binary
// exponent of the largest |Re|, |Im| of x when that lies outside [2^-256, 2^257) and 0 inside
// (each CTA its own e; the partials are brought to the largest e on combination), and the
// reflector is formed on (alpha, x) scaled by 2^-E, E the larger of that exponent and alpha's
// (taken the same way).  Inside the range nothing is scaled: the instruction stream is the
// plain formula's.  Outside it the scalings are exact powers of two, so columns whose norm is
// near or below sqrt(DBL_MIN) (amplitudes of 1e-150 and smaller occur in the sweeps from
// product states) get the reflector zlarfg's safe-minimum rescaling gives them instead of an
// overflow.  Not covered: an unscaled column's products with entries below 2^-766 of another
// column underflow (LAPACK's normalised v keeps them), i.e. spreads of more than ~1e-230
// between the columns of one matrix lose those small columns' directions.
//
// B200 mapping: one thread-block cluster per matrix, rows split over its C CTAs (32*RPL
// rows each; the whole matrix lives in distributed shared memory).  Blocked right-looking
// algorithm with panels of NB columns.  Every exchange between CTAs is a *push*: the
// producer writes its values straight into each consumer's shared memory with st.async,
// whose completion is counted in bytes on the consumer's mbarrier; the consumer waits on
// its own mbarrier (bounded) and then reads only local shared memory.
//   * column j: the panel sits in the registers of four warps, four columns each (lane = row).
//     Each forms conj(x)^T a for its columns over the CTA's rows and pushes the sums to all C CTAs;
//     after the exchange each sums the ranks, forms the reflector for itself, updates its columns and
//     the next column x.  The exchange is the only synchronisation of a column step: a hand-over
//     between warps through shared memory costs 160 clocks, an exchange between CTAs about 400, the
//     reflector about 200 (FP64 latency 8 clocks, a shuffle 24), so the redundant arithmetic is cheaper.
//   * the compact-WY factor T of a panel is built by a ninth warp, a column behind.
//   * block reflectors: partials of V^H A on the FP64 tensor path, pushed to the owner of each column
//     slice, reduced there in a fixed order with T (or T^H) applied, the slice pushed to every CTA,
//     then A -= V W on the tensor path.  (Bulk copies in place of the pushes need a proxy fence per
//     exchange, which took 1000 clocks.)
//   * Q = H(1)...H(n) [I; 0] is formed in place in shared memory by applying the panels' block
//     reflectors backwards to E (zungqr), so the matrix is read once and Q written once.
// Reductions run in a fixed order, so every CTA and warp computes bit-identical reflectors and
// results are reproducible run to run.  Each wait gives up after a bounded number of polls,
// records the timeout in the error word and lets the kernel run to completion.
//
// Shapes beyond one cluster (for example 2048 x 512) are factored in outer panels of up to 64
// columns by the same kernel, with the trailing updates and Q as GEMMs (qr_blocked).
//
// What bounds it: the chain of column steps (512 x 128: 2260 clocks a step at 16 CTAs -- sums over the
// rows 600, exchange 730, sum over the ranks 330, reflector 380, update 270 -- 55 % of the time; fewer
// at fewer CTAs, 1300 at one), then the products, which run at the FP64 tensor rate of the cluster's
// SMs.  One row per lane and many CTAs beat more rows per lane (512 x 128 at 1 / 2 / 4 rows: 254 / 324
// / 491 us) because the products scale with the CTAs.
// Against the form with a reflector warp behind block barriers, Q as GEMMs over a back substitution
// and outer panels of 16 columns (B200, Q only): 64 x 32 108.7 -> 45.6 us, 512 x 128 394 -> 235,
// 512 x 256 818 -> 590, 2048 x 512 3990 -> 2090.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "workspace.cuh"

namespace cg = cooperative_groups;

namespace mpsb {
namespace {

constexpr int NB = 16;                 // panel width
constexpr int CW = 4, NWP = NB / CW;   // panel columns per warp, warps that hold the panel
constexpr int NWM = 8;                 // warps of the block reflectors' products
constexpr int NT = 32 * (NWM + 1);     // and the warp that builds T
constexpr int CMAX = 16;
constexpr size_t SMEM_LIMIT = 227 * 1024;
constexpr int WAIT_LIMIT = 1 << 20;
constexpr int LDT = NB + 1, LDW = NB + 1;   // leading dimensions of T, the gathered W
enum { MB_COL = 0, MB_RS = 2, MB_AG, MB_COUNT };
constexpr int BAR_PANEL = 1, BAR_END = 2;   // named barriers: a step (C == 1), a panel's end

// Slots of the ranks' partial sums in a column's exchange: a power of two, the unused ones zero, so
// that a lane's sum over its half needs no tests (against sums tested per rank and column: 64 x 32
// 49.7 -> 47.6 us, 162 x 81 145.9 -> 142.0, 512 x 128 237.9 -> 235.1).
__host__ __device__ constexpr int rank_slots(int C) { return C <= 2 ? 2 : (C <= 4 ? 4 : (C <= 8 ? 8 : 16)); }

struct QrParams {
  QrProblem p;
  // form_q: Q goes to p.Q and T is scratch, [batch][npanels][NB][NB].  Otherwise the explicit unit
  // lower trapezoidal reflectors go to V (leading dimension v_ld) and the compact-WY factor of the
  // whole matrix to T (n x n, leading dimension t_ld).
  int form_q;
  cd* V;
  int64_t v_ld, v_b;
  cd* T;
  int64_t t_ld, t_b;
  int C, npanels, ldS, nc, ksc;   // nc: columns per exchange of a block reflector, ksc = ceil(nc / C)
  // shared-memory offsets (complex elements) and the byte offset of the mbarriers
  int o_S, o_V, o_col, o_rcol, o_rrs, o_w2s, o_rag, o_T, o_cst, o_tst, o_mbar;
};

// ---- PTX helpers -------------------------------------------------------------------
__device__ __forceinline__ uint32_t su32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16-byte remote store into CTA-rank-mapped shared memory, completion counted on its mbarrier
__device__ __forceinline__ void st_async(uint32_t raddr, cd v, uint32_t rmbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];"
               ::"r"(raddr), "d"(v.x), "d"(v.y), "r"(rmbar) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
// whether the phase of the given parity has completed, after a hardware-bounded suspension
__device__ __forceinline__ bool mbar_test(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
  return ok != 0;
}
template <int ID, int THREADS>
__device__ __forceinline__ void bar_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
// Bounded wait of one warp on the phase of the given parity.
__device__ __forceinline__ void warp_wait(uint32_t mbar, uint32_t parity, bool& failed, int* err) {
  int it = 0;
  while (!failed && !mbar_test(mbar, parity)) {
    if (++it >= WAIT_LIMIT) {
      failed = true;
      if (err) atomicOr(err, 1);
    }
  }
  __syncwarp();
}
// Bounded wait of the whole CTA on the phase of the given parity.  Only thread 0 polls --
// polling warps would compete with the computing warps for the shared-memory pipe -- and the
// block barrier then publishes the completion (and the pushed data) to every thread.  A
// timeout is recorded in the error word and later waits are skipped.
__device__ __forceinline__ void cta_wait(uint32_t mbar, uint32_t parity, bool& failed, int* err) {
  if (threadIdx.x == 0 && !failed) {
    int it = 0;
    while (!mbar_test(mbar, parity)) {
      if (++it >= WAIT_LIMIT) {
        failed = true;
        if (err) atomicOr(err, 1);
        break;
      }
    }
  }
  __syncthreads();
}

// The exponent slot of a rank's column message: no nonzero entry below the diagonal.
constexpr int ESENT = -100000;

// 2^k for -1022 <= k <= 1023, written into the exponent field
__device__ __forceinline__ double pow2i(int k) { return __hiloint2double((k + 1023) << 20, 0); }
// 2^k for k <= 0; 0 below the normal range (a contribution 2^-1022 times smaller than the rest)
__device__ __forceinline__ double pow2neg(int k) { return k >= -1022 ? pow2i(k) : 0.0; }
// binary exponent (clamped to [-1022, 1022]) of a nonnegative double from its high word;
// high word 0 (|v| < 2^-1042) is the caller's "zero"
__device__ __forceinline__ int expo_hi(unsigned hi) {
  const int b = (int)((hi >> 20) & 0x7ffu);
  return min(max(b, 1) - 1023, 1022);
}
__device__ __forceinline__ cd cscal(cd v, double f) { return cmk(v.x * f, v.y * f); }

// Half-width of the binary-exponent window [2^-SWIN, 2^(SWIN+1)) inside which nothing is scaled.
constexpr int SWIN = 256;

// A CTA whose partials are those of x 2^-e sends its |x|^2 partial (real) in the imaginary
// part and a quiet NaN carrying SCODE + e in the real part, so the unscaled combination of the
// ranks is NaN exactly when some rank scaled.
constexpr long long SCODE = 4096;
__device__ __forceinline__ double scale_nan(int e) {
  return __longlong_as_double(0x7ff8000000000000ll | (unsigned long long)(SCODE + e));
}
__device__ __forceinline__ int scale_of_nan(double v) { return (int)((__double_as_longlong(v) & 0xffffll) - SCODE); }

// The reflector when x == 0, some rank scaled its partials or alpha lies outside the window (rare:
// kept out of line so the common path's instructions stay the plain formula's).  Lane c < pw
// of a warp gets s = its combined partial at the scale 2^-E (lane jl: |x|^2 at 2^-2E), and
// every lane tau, beta, rs = 1/(alpha - beta) at 2^-E, and fE = 2^-E.  Returned by value, so
// the caller's variables stay in registers on the common path.
struct Reflector {
  cd s, tau, rs;
  double beta_x, beta_y, ib, fE;
};
__device__ __noinline__ Reflector reflector_scaled(const cd* rb, int C, int lane, int jl, int pw, cd alpha) {
  Reflector o;
  int e[CMAX];
  int ex = ESENT;
#pragma unroll
  for (int q = 0; q < CMAX; ++q) {
    e[q] = ESENT;
    if (q < C) {
      const cd pq = rb[q * NB + jl];
      e[q] = pq.x != pq.x ? scale_of_nan(pq.x) : (pq.x != 0.0 ? 0 : ESENT);
    }
    ex = max(ex, e[q]);
  }
  cd v = cmk(0.0, 0.0);
  if (lane < pw) {
    const int mult = lane == jl ? 2 : 1;
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      if (q >= C || e[q] == ESENT) continue;
      cd pq = rb[q * NB + lane];
      if (lane == jl) pq = cmk(pq.x != pq.x ? pq.y : pq.x, 0.0);
      v = cadd(v, cscal(pq, pow2neg(mult * (e[q] - ex))));
    }
  }
  const double xn2x = __shfl_sync(0xffffffffu, v.x, jl);   // |x|^2 2^-2ex
  const unsigned ha = (unsigned)__double2hiint(fmax(fabs(alpha.x), fabs(alpha.y)));
  o.fE = 1.0;
  o.s = v;
  o.tau = cmk(0.0, 0.0); o.rs = cmk(1.0, 0.0); o.ib = 0.0;
  o.beta_x = alpha.x; o.beta_y = alpha.y;
  if (ex == ESENT && (alpha.y == 0.0 || ha == 0u)) return o;   // x == 0 and a real (or negligible) pivot: H = I
  int ea = expo_hi(ha);
  ea = (ha == 0u) ? ESENT : (ea >= -SWIN && ea <= SWIN ? 0 : ea);
  const int E = max(ex, ea);
  o.fE = pow2i(-E);
  const cd as = cscal(alpha, o.fE);
  const double xn2 = (ex == ESENT) ? 0.0 : xn2x * pow2neg(2 * (ex - E));
  const double nrm = sqrt(as.x * as.x + as.y * as.y + xn2);
  const double b = -copysign(nrm, alpha.x);
  const double dr = as.x - b;
  o.ib = 1.0 / b;
  const double id = 1.0 / (dr * dr + as.y * as.y);
  o.tau = cmk((b - as.x) * o.ib, -as.y * o.ib);
  o.beta_x = b * pow2i(E);
  o.beta_y = 0.0;
  o.rs = cmk(dr * id, -as.y * id);
  o.s = (ex == ESENT) ? cmk(0.0, 0.0) : cscal(v, pow2neg(ex - E));
  return o;
}

__device__ __forceinline__ cd shfl(cd v, int src) {
  return cmk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

__device__ __forceinline__ double rsqrt_seed(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return y;
}
__device__ __forceinline__ double rcp_seed(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return y;
}

// The reflector of (alpha, x) with xn2 = |x|^2 (NaN: some rank scaled its partials), when xn2 and
// alpha lie inside the window -- tested on the high words, beside the formula: 0 < xn2 < 2^1023 and
// |Re alpha|, |Im alpha| < 2^SWIN; returns false otherwise.
//   tau = (beta - alpha)/beta, rs = 1/(alpha - beta) = conj(alpha - beta)/|alpha - beta|^2 with
//   |alpha - beta|^2 = |alpha|^2 + beta^2 + 2 |Re alpha| |beta|, ib = 1/beta
// (beta carries the opposite sign of Re alpha, so nothing cancels).  It sits on the critical path of
// every column, so |beta| = sqrt(n2), 1/|beta| and the reciprocal come from the hardware's 20-bit
// seeds, the second taken from the first's unrefined value, and one third-order Newton-Raphson
// (Householder) step each: errors below 2^-55 before the last rounding.
__device__ __forceinline__ bool reflector(cd alpha, double xn2, Reflector& o) {
  const unsigned hn = (unsigned)__double2hiint(xn2);
  const unsigned ha = max((unsigned)__double2hiint(alpha.x) & 0x7fffffffu, (unsigned)__double2hiint(alpha.y) & 0x7fffffffu);
  const bool in = hn - 0x00100000u < 0x7fe00000u - 0x00100000u && ha < (unsigned)(1023 + SWIN) << 20;
  const double a2 = fma(alpha.x, alpha.x, alpha.y * alpha.y), ax2 = 2.0 * fabs(alpha.x);
  const double n2 = a2 + xn2, s2 = a2 + n2;
  const double y0 = rsqrt_seed(n2), n0 = n2 * y0;
  const double z0 = rcp_seed(fma(ax2, n0, s2));
  const double r = fma(-n0, y0, 1.0), p = fma(r, 0.375, 0.5);
  const double y = fma(y0 * r, p, y0), nrm = fma(n0 * r, p, n0);
  const double e = fma(-fma(ax2, nrm, s2), z0, 1.0);
  const double z = fma(z0, fma(e, e, e), z0);
  o.ib = -copysign(y, alpha.x);
  o.beta_x = -copysign(nrm, alpha.x);
  o.beta_y = 0.0;
  o.tau = cmk(fma(-alpha.x, o.ib, 1.0), -alpha.y * o.ib);
  o.rs = cmk((alpha.x - o.beta_x) * z, -alpha.y * z);
  return in;
}
// a - f v
__device__ __forceinline__ cd cfms(cd a, cd f, cd v) {
  return cmk(fma(f.y, v.y, fma(-f.x, v.x, a.x)), fma(-f.y, v.x, fma(-f.x, v.y, a.y)));
}

template <int RPL, bool SOLO>   // SOLO: a cluster of one CTA
__global__ void __launch_bounds__(NT, 1) qr_kernel(QrParams P) {
  constexpr int ROWS = 32 * RPL, LDV = ROWS + 1;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* sm = reinterpret_cast<cd*>(smem_raw);
  const int C = P.C, ldS = P.ldS, ksc = P.ksc;
  const int m = P.p.m, n = P.p.n;
  const int crank = (int)cluster.block_rank();
  const int prob = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = crank * ROWS;
  int* err = P.p.err;

  cd* S = sm + P.o_S;
  cd* Vs = sm + P.o_V;
  cd* colbuf = sm + P.o_col;
  cd* rcol = sm + P.o_rcol;
  const int CP = rank_slots(C), rbuf = (CP + 1) * NB;
  cd* rrs = sm + P.o_rrs;
  cd* w2s = sm + P.o_w2s;
  cd* rag = sm + P.o_rag;
  cd* Ts = sm + P.o_T;
  cd* cst = sm + P.o_cst;
  cd* tst = sm + P.o_tst;
  cd* pst = tst + NB * NB;
  uint64_t* mb = reinterpret_cast<uint64_t*>(smem_raw + P.o_mbar);
  const uint32_t mb_rs = su32(&mb[MB_RS]), mb_ag = su32(&mb[MB_AG]), rrs32 = su32(rrs), rag32 = su32(rag);
  uint32_t ph_rs = 0, ph_ag = 0;
  bool failed = false;
  cd* Tg = P.T + (int64_t)prob * P.t_b;

  if (tid == 0) {
    for (int k = 0; k < 2; ++k) mbar_init(su32(&mb[MB_COL + k]), NWP + 1);
    mbar_init(mb_rs, 1);
    mbar_init(mb_ag, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  {  // ---- load this CTA's rows, along whichever index is contiguous in X
    const cd* X = P.p.X + (int64_t)prob * P.p.x_b;
    if (P.p.x_c == 1 && P.p.x_r != 1) {
      for (int e = tid; e < ROWS * n; e += NT) {
        const int cc = e % n, rr = e / n, g = row0 + rr;
        S[cc * ldS + rr] = (g < m) ? X[(int64_t)g * P.p.x_r + cc] : cmk(0.0, 0.0);
      }
    } else {
      for (int e = tid; e < ROWS * n; e += NT) {
        const int rr = e % ROWS, cc = e / ROWS, g = row0 + rr;
        S[cc * ldS + rr] = (g < m) ? X[(int64_t)g * P.p.x_r + (int64_t)cc * P.p.x_c] : cmk(0.0, 0.0);
      }
    }
    if (!P.form_q && crank == 0)
      for (int e = tid; e < n * n; e += NT) Tg[(e % n) + (int64_t)(e / n) * P.t_ld] = cmk(0.0, 0.0);
  }
  for (int e = tid; e < 2 * rbuf; e += NT) rcol[e] = cmk(0.0, 0.0);   // the slots of ranks >= C stay zero
  cluster.sync();   // mbarriers initialised cluster-wide before any push

  // Columns kk in [0, ncols) -- columns 0 .. nprev-1 of the matrix, then cbase, cbase + 1, ... --
  // get W = op(T) V^H A for the panel in Vs (rows >= p0, width pw), gathered in every CTA's rag, and
  // all but the first nprev of them A -= V W.  op(T) = T^H in the factorisation, T for Q.
  auto apply = [&](int p0, int pw, int nprev, int cbase, int ncols, bool factor) {
    const int fg = lane >> 2, ft = lane & 3;
    auto colp = [&](int kk) { return S + (kk < nprev ? kk : cbase + kk - nprev) * ldS; };
    for (int c0 = 0; c0 < ncols; c0 += P.nc) {
      const int ncc = min(P.nc, ncols - c0);
      const int KS = (ncc + C - 1) / C, k0 = crank * KS, ks = max(0, min(ncc, k0 + KS) - k0);
      const int ntile = (ncc + 7) / 8, inv = (65536 + KS - 1) / KS;   // kk * inv >> 16 == kk / KS for kk < 256
      const bool active = row0 + ROWS > p0;
      if (warp < NWM) {
        // partials over this CTA's rows: 16 x 8 tiles, two per warp in flight
        for (int t = warp; t < ntile; t += 2 * NWM) {
          double re[2][4], im[2][4];
          const bool two = t + NWM < ntile;
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) re[u][e] = im[u][e] = 0.0;
          if (active) {
            const cd* B0 = colp(c0 + min(8 * t + fg, ncc - 1));
            const cd* B1 = colp(c0 + min(8 * (t + NWM) + fg, ncc - 1));
#pragma unroll 2
            for (int r = 0; r < ROWS; r += 8) {
              // k index t <-> row 2t, t + 4 <-> row 2t + 1: odd leading dimensions then give the
              // eight 16-byte loads of a quarter warp distinct banks
              const int ra = r + 2 * ft;
              double vr[4], vi[4], nvi[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const cd v = Vs[(fg + 8 * (e & 1)) * LDV + ra + (e >> 1)];
                vr[e] = v.x; vi[e] = v.y; nvi[e] = -v.y;
              }
              const cd b00 = B0[ra], b01 = B0[ra + 1], b10 = B1[ra], b11 = B1[ra + 1];
              const double br[2][2] = {{b00.x, b01.x}, {b10.x, b11.x}}, bi[2][2] = {{b00.y, b01.y}, {b10.y, b11.y}};
#pragma unroll
              for (int u = 0; u < 2; ++u)
                if (u == 0 || two) {
                  dmma16(re[u], vr, br[u]);
                  dmma16(im[u], vr, bi[u]);
                  dmma16(re[u], vi, bi[u]);
                  dmma16(im[u], nvi, br[u]);
                }
            }
          }
          // pushed from the fragments: a store is four runs of eight entries of a column
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int kk = 8 * (t + u * NWM) + 2 * ft + c;
              if ((u == 0 || two) && kk < ncc) {
                const int so = kk * inv >> 16;   // its owner, kk / KS
                const uint32_t dst = mapa(rrs32, so) + (uint32_t)(((crank * ksc + kk - so * KS) * NB + fg) * sizeof(cd));
                const uint32_t bar = mapa(mb_rs, so);
                st_async(dst, cmk(re[u][c], im[u][c]), bar);
                st_async(dst + 8 * (uint32_t)sizeof(cd), cmk(re[u][2 + c], im[u][2 + c]), bar);
              }
            }
        }
      }
      if (ks > 0) {
        if (tid == 0) mbar_expect(mb_rs, (uint32_t)(C * NB * ks * sizeof(cd)));
        cta_wait(mb_rs, ph_rs, failed, err);
        ph_rs ^= 1;
      } else {
        __syncthreads();
      }
      // the ranks' sum and op(T) W on my slice (zero beyond the panel width: V and T are), a warp per
      // column: a lane has entry i, half of the ranks, half of the products and half of the pushes
      if (tid == 0) mbar_expect(mb_ag, (uint32_t)(ncc * NB * sizeof(cd)));
      for (int kk = warp; kk < ks; kk += NWM + 1) {
        const int i = lane & 15, h = lane >> 4;
        const cd* src = rrs + kk * NB + i;
        const int rs = ksc * NB;
        cd w = cmk(0.0, 0.0), w1 = cmk(0.0, 0.0);
#pragma unroll 2
        for (int q = h; q < C; q += 4) {
          w = cadd(w, src[q * rs]);
          if (q + 2 < C) w1 = cadd(w1, src[(q + 2) * rs]);
        }
        w = cadd(w, w1);
        w.x += __shfl_xor_sync(0xffffffffu, w.x, 16);
        w.y += __shfl_xor_sync(0xffffffffu, w.y, 16);
        cd* wc = w2s + kk * NB;
        if (h == 0) wc[i] = w;
        __syncwarp();
        const cd* t = (factor ? Ts + LDT * i : Ts + i);
        const int ts = factor ? 1 : LDT;
        cd s0 = cmk(0.0, 0.0), s1 = cmk(0.0, 0.0);
#pragma unroll
        for (int i2 = 8 * h; i2 < 8 * h + 8; i2 += 2) {
          cd t0 = t[i2 * ts], t1 = t[(i2 + 1) * ts];
          if (factor) { t0.y = -t0.y; t1.y = -t1.y; }
          cfma(s0, t0, wc[i2]);
          cfma(s1, t1, wc[i2 + 1]);
        }
        s0 = cadd(s0, s1);
        s0.x += __shfl_xor_sync(0xffffffffu, s0.x, 16);
        s0.y += __shfl_xor_sync(0xffffffffu, s0.y, 16);
        const uint32_t off = (uint32_t)(((k0 + kk) * LDW + i) * sizeof(cd));
#pragma unroll 2
        for (int q = h; q < C; q += 2) st_async(mapa(rag32, q) + off, s0, mapa(mb_ag, q));
      }
      cta_wait(mb_ag, ph_ag, failed, err);
      ph_ag ^= 1;
      if (factor && !P.form_q && crank == 0 && c0 < nprev) {
        // T[0:p0, panel] = -T[0:p0, 0:p0] (V_c^H V_p T_p), the bracket being the gathered W's ^H
        const int kmax = min(nprev, c0 + ncc);   // the first nprev columns come in one chunk
        for (int e = tid; e < kmax * pw; e += NT) {
          const int i = e % kmax, jj = e / kmax;
          cd s = cmk(0.0, 0.0);
          for (int c = i; c < kmax; ++c) cfma_cj(s, rag[c * LDW + jj], Tg[i + (int64_t)c * P.t_ld]);
          Tg[i + (int64_t)(p0 + jj) * P.t_ld] = cmk(-s.x, -s.y);
        }
      }
      if (active && warp < NWM) {
        for (int t = warp; t < ntile; t += NWM) {
          if (c0 + 8 * t + 7 < nprev) continue;
          double wr[2][2], wi[2][2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int i = 8 * h + ft + 4 * e;
              const cd w = rag[min(8 * t + fg, ncc - 1) * LDW + i];
              wr[h][e] = w.x; wi[h][e] = w.y;
            }
          const int ka = 8 * t + 2 * ft;
          cd* C0 = colp(c0 + min(ka, ncc - 1));
          cd* C1 = colp(c0 + min(ka + 1, ncc - 1));
          const bool ok0 = ka < ncc && c0 + ka >= nprev, ok1 = ka + 1 < ncc && c0 + ka + 1 >= nprev;
#pragma unroll 2
          for (int rb = 0; rb < ROWS; rb += 16) {
            if (row0 + rb + 16 <= p0) continue;
            double re[4], im[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const cd c = ((e & 1) ? C1 : C0)[rb + fg + 8 * (e >> 1)];
              re[e] = c.x; im[e] = c.y;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              double nvr[4], vi[4], nvi[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const cd v = Vs[(8 * h + ft + 4 * (e >> 1)) * LDV + rb + fg + 8 * (e & 1)];
                nvr[e] = -v.x; vi[e] = v.y; nvi[e] = -v.y;
              }
              dmma16(re, nvr, wr[h]);
              dmma16(im, nvr, wi[h]);
              dmma16(re, vi, wi[h]);
              dmma16(im, nvi, wr[h]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if ((e & 1) ? ok1 : ok0) ((e & 1) ? C1 : C0)[rb + fg + 8 * (e >> 1)] = cmk(re[e], im[e]);
          }
        }
      }
      __syncthreads();
    }
  };

  // ================================ factorisation ================================
  // Two buffers of the exchange suffice: another CTA pushes step j + 2 after its exchange of step
  // j + 1, so after every panel warp here pushed step j + 1, which each does when it has read step j.
  int step = 0;   // column steps so far: buffers step & 1, phase parity (step / 2) & 1
  const int pr = lane & 7, pc = CW * warp + (lane >> 3);   // this lane pushes column pc to ranks pr, pr + 8
  const bool push0 = pr < C, push1 = pr + 8 < C;
  uint32_t rd0, rd1, rm0, rm1;   // where: slot pc of this rank's row, and the exchange's mbarriers
  {
    const uint32_t slot = su32(rcol) + (uint32_t)(pc * sizeof(cd)), m0 = su32(&mb[MB_COL]);
    rd0 = mapa(slot, push0 ? pr : 0); rm0 = mapa(m0, push0 ? pr : 0);
    rd1 = mapa(slot, push1 ? pr + 8 : 0); rm1 = mapa(m0, push1 ? pr + 8 : 0);
  }
  const uint32_t off_sum = (uint32_t)(crank * NB * sizeof(cd)), off_piv = (uint32_t)(CP * NB * sizeof(cd));
  if (warp == NWM && lane == 0)   // the T warp's arrivals for the first two steps
    for (int k = 0; k < 2; ++k) mbar_arrive(su32(&mb[MB_COL + k]));
  for (int pi = 0; pi < P.npanels; ++pi) {
    const int p0 = pi * NB;
    const int pw = min(NB, n - p0);
    if (warp < NWP) {
      const int cf = CW * warp;   // first column
      cd a[CW][RPL], x[RPL];
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const int r = lane + 32 * q;
        x[q] = S[p0 * ldS + r];
#pragma unroll
        for (int k = 0; k < CW; ++k) a[k][q] = cf + k < pw ? S[(p0 + cf + k) * ldS + r] : cmk(0.0, 0.0);
        if (warp == 0) colbuf[ROWS + r] = a[1][q];   // column 1 for the step that follows column 0
      }
      for (int jl = 0; jl < pw; ++jl, ++step) {
        const int j = p0 + jl, buf = step & 1;
        cd* cs = cst + buf * 2 * NB;   // C == 1: the sums; the pivot row's entries in its owner
        const uint32_t mbc = su32(&mb[MB_COL + buf]);
        const int jr = j - row0;
        const bool owner = jr >= 0 && jr < ROWS;
#pragma unroll
        for (int q = 0; q < RPL; ++q)
          if (lane + 32 * q == jr) {
#pragma unroll
            for (int k = 0; k < CW; ++k) cs[NB + cf + k] = a[k][q];
          }
        __syncwarp();   // the pivot row's entries; and this warp's hand-over of column jl + 1, ordered by
        if (!SOLO && lane == 0) {   // its arrival
          if (warp == 0) mbar_expect(mbc, (uint32_t)((C + 1) * NB * sizeof(cd)));
          else mbar_arrive(mbc);
        }
        const uint32_t ob = (uint32_t)(buf * rbuf * sizeof(cd)), om = 8 * buf;
        if (!SOLO && owner) {   // the pivot row is known before the sums: its flight is hidden
          const cd piv = cs[NB + pc];
          if (push0) st_async(rd0 + ob + off_piv, piv, rm0 + om);
          if (push1) st_async(rd1 + ob + off_piv, piv, rm1 + om);
        }
        // -- partial sums of conj(x) a over this CTA's rows g > j (x zero elsewhere)
#pragma unroll
        for (int q = 0; q < RPL; ++q)
          if (row0 + lane + 32 * q <= j) x[q] = cmk(0.0, 0.0);
        // the largest |Re|, |Im| of x over this CTA's rows, by the high words (every warp finds the same)
        unsigned hx = 0;
#pragma unroll
        for (int q = 0; q < RPL; ++q)
          hx = max(hx, max((unsigned)__double2hiint(x[q].x) & 0x7fffffffu, (unsigned)__double2hiint(x[q].y) & 0x7fffffffu));
        const unsigned hb = __reduce_max_sync(0xffffffffu, hx);
        // the scale 2^-e of this CTA's sums: none when x is 0 (or below 2^-1042) or its largest entry
        // lies inside the window; else e is that entry's binary exponent, and the sums are redone on
        // x 2^-e (a second round of the loop, so the rare case adds no code to the common one)
        cd sum;
        bool scaled = false;
        cd xs[RPL];
#pragma unroll
        for (int q = 0; q < RPL; ++q) xs[q] = x[q];
#pragma unroll 1
        for (;;) {
          cd sk[CW];
#pragma unroll
          for (int k = 0; k < CW; ++k) {
            sk[k] = cmk(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < RPL; ++q) cfma_cj(sk[k], xs[q], a[k][q]);
          }
          // lanes 8 k .. 8 k + 7 end with the sum of column cf + k
          const bool lo = (lane & 16) == 0, lo2 = (lane & 8) == 0;
          cd u0 = lo ? sk[0] : sk[2], u1 = lo ? sk[1] : sk[3];
          const cd g0 = lo ? sk[2] : sk[0], g1 = lo ? sk[3] : sk[1];
          u0.x += __shfl_xor_sync(0xffffffffu, g0.x, 16);
          u0.y += __shfl_xor_sync(0xffffffffu, g0.y, 16);
          u1.x += __shfl_xor_sync(0xffffffffu, g1.x, 16);
          u1.y += __shfl_xor_sync(0xffffffffu, g1.y, 16);
          sum = lo2 ? u0 : u1;
          const cd give = lo2 ? u1 : u0;
          sum.x += __shfl_xor_sync(0xffffffffu, give.x, 8);
          sum.y += __shfl_xor_sync(0xffffffffu, give.y, 8);
#pragma unroll
          for (int off = 4; off > 0; off >>= 1) {
            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, off);
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, off);
          }
          if (scaled || hb == 0u || hb - ((unsigned)(1023 - SWIN) << 20) < (unsigned)(2 * SWIN + 1) << 20) break;
          scaled = true;
          const double f = pow2i(-expo_hi(hb));
#pragma unroll
          for (int q = 0; q < RPL; ++q) {
            xs[q] = cscal(x[q], f);
#pragma unroll
            for (int k = 0; k < CW; ++k)   // column j's own copy, overwritten below, gives |x 2^-e|^2
              if (cf + k == jl && row0 + lane + 32 * q > j) a[k][q] = xs[q];
          }
        }
        if (scaled && pc == jl) sum = cmk(scale_nan(expo_hi(hb)), sum.x);
        // -- the exchange: every CTA gets all ranks' sums and the pivot row
        const int c = lane & 15;
        const bool keeps = warp == (((jl >> 2) + 2) & 3);   // writes what T needs
        const cd* rb = SOLO ? cs : rcol + buf * rbuf;
        const cd* pv = SOLO ? cs + NB : rb + CP * NB;   // the pivot row's entries
        cd rv, s;
        if (!SOLO) {
          if (push0) st_async(rd0 + ob + off_sum, sum, rm0 + om);
          if (push1) st_async(rd1 + ob + off_sum, sum, rm1 + om);
          warp_wait(mbc, (uint32_t)(step >> 1) & 1, failed, err);
          // lane c sums one half of the slots of column c, lane c + 16 the other
          const cd* rp = rb + (lane >> 4) * (CP / 2) * NB + c;
          rv = pv[c];
          s = rp[0];
          if (CP == 16) {
            cd p[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) p[q] = rp[q * NB];
            s = cadd(cadd(cadd(p[0], p[4]), cadd(p[2], p[6])), cadd(cadd(p[1], p[5]), cadd(p[3], p[7])));
          } else if (CP == 8) {
            s = cadd(cadd(s, rp[2 * NB]), cadd(rp[NB], rp[3 * NB]));
          } else if (CP == 4) {
            s = cadd(s, rp[NB]);
          }
          s.x += __shfl_xor_sync(0xffffffffu, s.x, 16);
          s.y += __shfl_xor_sync(0xffffffffu, s.y, 16);
        } else {
          if (pr == 0) cs[pc] = sum;
          bar_sync<BAR_PANEL, 32 * (NWP + 1)>();
          s = cs[c];
          rv = pv[c];
        }
        // -- the reflector, formed by every warp from the same sums
        cd nx[RPL];   // column jl + 1 as updated by the reflectors before this one
#pragma unroll
        for (int q = 0; q < RPL; ++q) nx[q] = colbuf[((jl + 1) & 1) * ROWS + lane + 32 * q];
        // this warp's columns' sums and pivot entries, and the next column's, in every lane: read
        // back from shared memory while the reflector's chain runs (4 rows per lane: after it, as the
        // registers do not suffice)
        cd* sb = rag + NB * warp;
        if (lane < NB) sb[lane] = s;
        __syncwarp();
        const int jn = min(jl + 1, NB - 1);
        cd sk[CW], rk[CW], sn, rn;
        auto fetch = [&] {
          sn = sb[jn];
          rn = pv[jn];
#pragma unroll
          for (int k = 0; k < CW; ++k) { sk[k] = sb[cf + k]; rk[k] = pv[cf + k]; }
        };
        if (RPL < 4) fetch();
        const cd alpha = pv[jl];
        const double xn2 = __shfl_sync(0xffffffffu, s.x, jl);
        Reflector o;
        const bool plain = reflector(alpha, xn2, o);
        if (__builtin_expect(!plain, 0)) {
          o = reflector_scaled(rb, C, c, jl, pw, alpha);
          s = o.s;
          __syncwarp();
          if (lane < NB) sb[lane] = s;
          __syncwarp();
          if (RPL < 4) fetch();
#pragma unroll
          for (int q = 0; q < RPL; ++q) {   // v = rs x 2^-E; column j is kept as v itself
            x[q] = cscal(x[q], o.fE);
#pragma unroll
            for (int k = 0; k < CW; ++k)
              if (cf + k == jl && row0 + lane + 32 * q > j) a[k][q] = cmul(o.rs, x[q]);
          }
        }
        // right of the pivot: a_c -= f_c v with f_c = conj(tau) (a_c[j] + conj(rs) x^H a_c) =
        // conj(tau) a_c[j] - (x^H a_c)/beta and v = rs x, 1 at the pivot
        auto factor = [&](cd r, cd t) {
          return cmk(fma(o.tau.x, r.x, fma(o.tau.y, r.y, -o.ib * t.x)), fma(o.tau.x, r.y, fma(-o.tau.y, r.x, -o.ib * t.y)));
        };
        if (o.tau.x != 0.0 || o.tau.y != 0.0) {   // else H = I
          if (RPL == 4) fetch();
          const cd fn = factor(rn, sn);
          cd fk[CW];
#pragma unroll
          for (int k = 0; k < CW; ++k) fk[k] = cf + k > jl ? factor(rk[k], sk[k]) : cmk(0.0, 0.0);
#pragma unroll
          for (int q = 0; q < RPL; ++q) {
            const cd v = row0 + lane + 32 * q == j ? cmk(1.0, 0.0) : cmul(o.rs, x[q]);
            x[q] = cfms(nx[q], fn, v);
#pragma unroll
            for (int k = 0; k < CW; ++k) a[k][q] = cfms(a[k][q], fk[k], v);
          }
        } else {
#pragma unroll
          for (int q = 0; q < RPL; ++q) x[q] = nx[q];
        }
        if (keeps) {   // for T (see below) and the panel's end
          if (lane <= jl) tst[jl * NB + lane] = lane == jl ? o.tau : cadd(rv, cmul(cconj(o.rs), s));
          if (lane == 16) pst[jl] = plain ? o.rs : cmk(1.0, 0.0);
          if (lane == 17) pst[NB + jl] = cmk(o.beta_x, o.beta_y);
        }
#pragma unroll
        for (int k = 0; k < CW; ++k)
          if (cf + k == jl + 2) {
#pragma unroll
            for (int q = 0; q < RPL; ++q) colbuf[(jl & 1) * ROWS + lane + 32 * q] = a[k][q];
          }
      }
      // the panel back to shared memory, and its reflectors explicitly (unit lower trapezoidal): column
      // c holds x below the pivot, v = pst[c] x (pst = 1 where v was kept)
      bar_sync<BAR_END, 32 * (NWP + 1)>();
#pragma unroll
      for (int k = 0; k < CW; ++k) {
        const int cc = cf + k;
        const cd sc = pst[cc], beta = pst[NB + cc];
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          const int r = lane + 32 * q, g = row0 + r;
          const cd v = cmul(sc, a[k][q]);
          if (cc < pw) S[(p0 + cc) * ldS + r] = g < p0 + cc ? a[k][q] : (g == p0 + cc ? beta : v);
          Vs[cc * LDV + r] = (cc >= pw || g < p0 + cc) ? cmk(0.0, 0.0) : (g == p0 + cc ? cmk(1.0, 0.0) : v);
        }
      }
    } else if (warp == NWM) {
      // T (compact WY, zlarft forward/columnwise), each column while the panel warps are at the next:
      // T[0:jl, jl] = -tau_jl T[0:jl, 0:jl] t_jl with t_c = conj(pst[c] (a_c[j] + conj(rs) x^H x_c)),
      // the bracket kept in tst; zero outside the panel width.  Lane i and i + 16 have row i, half of
      // the sum each.
      const int i = lane & 15, h = lane >> 4;
      if (SOLO) bar_sync<BAR_PANEL, 32 * (NWP + 1)>();
      for (int jl = 0; jl < NB; ++jl) {
        // step jl's values are in place once every panel warp is at step jl + 1 or at the panel's end
        if (jl + 1 < pw) {
          if (SOLO) bar_sync<BAR_PANEL, 32 * (NWP + 1)>();
          else warp_wait(su32(&mb[MB_COL + ((step + 1) & 1)]), (uint32_t)((step + 1) >> 1) & 1, failed, err);
        } else if (jl + 1 == pw) {
          bar_sync<BAR_END, 32 * (NWP + 1)>();
        }
        cd acc = cmk(0.0, 0.0), tau = cmk(0.0, 0.0);
        if (jl < pw) {
          tau = tst[jl * NB + jl];
          for (int c = h; c < jl; c += 2) cfma(acc, Ts[i + LDT * c], cconj(cmul(pst[c], tst[jl * NB + c])));   // T[i, c] = 0 for c < i
        }
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
        const cd t = i == jl ? tau : (i < jl ? cmul(cmk(-tau.x, -tau.y), acc) : cmk(0.0, 0.0));
        __syncwarp();
        if (h == 0) {
          Ts[i + LDT * jl] = t;
          if (crank == 0 && i < pw && jl < pw) {
            if (P.form_q) Tg[(int64_t)pi * NB * NB + i + NB * jl] = t;
            else Tg[p0 + i + (int64_t)(p0 + jl) * P.t_ld] = t;
          }
        }
        __syncwarp();
        if (jl < pw) {   // its arrival for step + 2: the exchanges stay within two steps of this warp
          if (!SOLO && lane == 0) mbar_arrive(su32(&mb[MB_COL + (step & 1)]));
          ++step;
        }
      }
    } else {
      step += pw;
    }
    __syncthreads();
    const int nprev = P.form_q ? 0 : p0, nt = n - p0 - pw;
    if (nprev + nt > 0) apply(p0, pw, nprev, p0 + pw, nprev + nt, true);
  }
  __syncthreads();

  // ---- optional R (rows < n)
  if (P.p.R) {
    cd* Rout = P.p.R + (int64_t)prob * P.p.r_b;
    for (int e = tid; e < ROWS * n; e += NT) {
      const int rr = e % ROWS, k = e / ROWS, g = row0 + rr;
      if (g >= n) continue;
      Rout[(int64_t)g * P.p.r_r + (int64_t)k * P.p.r_c] = (k >= g) ? S[k * ldS + rr] : cmk(0.0, 0.0);
    }
  }
  if (!P.form_q) {
    cd* V = P.V + (int64_t)prob * P.v_b;
    for (int e = tid; e < ROWS * n; e += NT) {
      const int rr = e % ROWS, cc = e / ROWS, g = row0 + rr;
      if (g < m) V[g + (int64_t)cc * P.v_ld] = g < cc ? cmk(0.0, 0.0) : (g == cc ? cmk(1.0, 0.0) : S[cc * ldS + rr]);
    }
    cluster.sync();   // no CTA leaves while a peer may still address its shared memory
    return;
  }
  cluster.sync();   // rank 0's T of every panel

  // ================================ Q = H(1) ... H(n) E ================================
  cd tp = cmk(0.0, 0.0);   // an entry of the panel's T (zero outside its width)
  if (tid < NB * NB) {
    const int pw = n - (P.npanels - 1) * NB;
    if (tid % NB < pw && tid / NB < pw) tp = __ldcg(&Tg[(int64_t)(P.npanels - 1) * NB * NB + tid]);
  }
  for (int pi = P.npanels - 1; pi >= 0; --pi) {
    const int p0 = pi * NB, pw = min(NB, n - p0);
    // the panel's reflectors to Vs, its columns of E to S (the later columns hold Q so far)
    for (int e = tid; e < ROWS * NB; e += NT) {
      const int rr = e % ROWS, i = e / ROWS, g = row0 + rr;
      cd* a = S + (p0 + i) * ldS + rr;
      Vs[i * LDV + rr] = (i >= pw || g < p0 + i) ? cmk(0.0, 0.0) : (g == p0 + i ? cmk(1.0, 0.0) : *a);
      if (i < pw) *a = cmk(g == p0 + i ? 1.0 : 0.0, 0.0);
    }
    if (tid < NB * NB) Ts[tid % NB + LDT * (tid / NB)] = tp;
    if (tid < NB * NB && pi > 0) tp = __ldcg(&Tg[(int64_t)(pi - 1) * NB * NB + tid]);   // in flight during this panel
    __syncthreads();
    apply(p0, pw, 0, p0, n - p0, false);
  }
  {
    cd* Q = P.p.Q + (int64_t)prob * P.p.q_b;
    if (P.p.q_c == 1 && P.p.q_r != 1) {
      for (int e = tid; e < ROWS * n; e += NT) {
        const int cc = e % n, rr = e / n, g = row0 + rr;
        if (g < m) Q[(int64_t)g * P.p.q_r + cc] = S[cc * ldS + rr];
      }
    } else {
      for (int e = tid; e < ROWS * n; e += NT) {
        const int rr = e % ROWS, cc = e / ROWS, g = row0 + rr;
        if (g < m) Q[(int64_t)g * P.p.q_r + (int64_t)cc * P.p.q_c] = S[cc * ldS + rr];
      }
    }
  }
  cluster.sync();   // no CTA leaves while a peer may still address its shared memory
}

typedef void (*QrKernel)(QrParams);

QrKernel kernel_for(int rpl, int C) {
  switch (rpl) {
    case 1: return C == 1 ? qr_kernel<1, true> : qr_kernel<1, false>;
    case 2: return C == 1 ? qr_kernel<2, true> : qr_kernel<2, false>;
    case 4: return C == 1 ? qr_kernel<4, true> : qr_kernel<4, false>;
    default: return nullptr;
  }
}

size_t layout(QrParams& P, int n, int C, int rows, int nc) {
  P.C = C;
  P.npanels = (n + NB - 1) / NB;
  P.ldS = rows + 1;
  P.nc = nc;
  P.ksc = (nc + C - 1) / C;
  int o = 0;
  P.o_S = o;     o += P.ldS * n;
  P.o_V = o;     o += (rows + 1) * NB;
  P.o_col = o;   o += 2 * rows;
  P.o_rcol = o;  o += 2 * (rank_slots(C) + 1) * NB;
  P.o_rrs = o;   o += C * P.ksc * NB;
  P.o_rag = o;   o += nc * LDW;
  P.o_T = o;     o += NB * LDT;
  P.o_cst = P.o_w2s = o;   o += std::max(4, P.ksc) * NB;   // column steps / block reflectors
  P.o_tst = o;   o += NB * NB + 2 * NB;   // and per column the factor of x to v, and beta
  P.o_mbar = o * (int)sizeof(cd);
  return (size_t)P.o_mbar + MB_COUNT * sizeof(uint64_t);
}

struct Choice {
  int C = 0, rpl = 0, nc = 0;
  size_t smem = 0;
};

// Cluster of C = ceil(m / (32 rpl)) CTAs, at most 16: prefer 1 row per lane, then 2, then 4, since the
// products scale with the CTAs -- except 33 to 64 rows of up to 32 columns, where two rows per lane in
// one CTA save the exchanges (48 x 24: 40.6 -> 39.4 us, 64 x 32: 47.6 -> 45.6; but 64 x 64: 98.8 ->
// 100.9, 128 x 32 in two CTAs: 47.7 -> 53.8, 200 x 100: 177 -> 216).  The
// widest column chunk of the block reflectors that fits, in steps of 8 (512 x 256, one width against
// the next: 88 columns 635 us, 64 columns 675, as a chunk costs about 3500 clocks of exchanges
// whatever its width).  An outer panel of the blocked form
// (panel) keeps the columns beside an inner panel in one chunk, since its T needs them.
bool choose(int m, int n, Choice& ch, bool panel = false) {
  QrParams P;
  const int nc_max = panel ? std::max(8, (n - NB + 7) / 8 * 8) : std::min(256, (n + 7) / 8 * 8);
  const int nc_min = panel ? nc_max : 8;
  for (int rpl : {1, 2, 4}) {
    if (rpl == 1 && m > 32 && m <= 64 && n <= 32) continue;
    const int rows = 32 * rpl;
    const int C = (m + rows - 1) / rows;
    if (C > CMAX) continue;
    for (int nc = nc_max; nc >= nc_min; nc -= 8) {
      const size_t b = layout(P, n, C, rows, nc);
      if (b <= SMEM_LIMIT) {
        ch.C = C; ch.rpl = rpl; ch.nc = nc; ch.smem = b;
        return true;
      }
    }
  }
  return false;
}

// Strided m x n matrix fill for every problem of a batch: COPY dst = src, UPPER dst = triu(src),
// IDENT dst = [I; 0], CTRANS_UPPER dst = triu(src^H).
enum { MAT_COPY = 0, MAT_UPPER, MAT_IDENT, MAT_CTRANS_UPPER };
__global__ void mat_kernel(int mode, int m, int n, const cd* __restrict__ src, int64_t sr, int64_t sc, int64_t sb, cd* dst,
                           int64_t dr, int64_t dc, int64_t db) {
  const int64_t total = (int64_t)m * n;
  src += blockIdx.y * sb;
  dst += blockIdx.y * db;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(e % m), k = (int)(e / m);
    cd v;
    if (mode == MAT_IDENT) v = cmk(g == k ? 1.0 : 0.0, 0.0);
    else if (mode >= MAT_UPPER && k < g) v = cmk(0.0, 0.0);
    else if (mode == MAT_CTRANS_UPPER) v = cconj(src[k * sr + g * sc]);
    else v = src[g * sr + k * sc];
    dst[g * dr + k * dc] = v;
  }
}

int mat_launch(int mode, int m, int n, int batch, const cd* src, int64_t sr, int64_t sc, int64_t sb, cd* dst, int64_t dr,
               int64_t dc, int64_t db, Workspace* ws, cudaStream_t s) {
  count_launch(ws);
  const int64_t total = (int64_t)m * n;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 8);
  mat_kernel<<<dim3(blocks, batch), 256, 0, s>>>(mode, m, n, src, sr, sc, sb, dst, dr, dc, db);
  MPSB_CUDA_TRY(cudaGetLastError());
  return MPSB_OK;
}

// The cluster kernel on every problem of p.
int launch_cluster(QrParams& P, const Choice& ch, cudaStream_t s) {
  layout(P, P.p.n, ch.C, 32 * ch.rpl, ch.nc);
  QrKernel fn = kernel_for(ch.rpl, ch.C);
  if (!fn) return MPSB_ERR_UNSUPPORTED;
  MPSB_TRY(ensure_kernel_attrs((const void*)fn, (int)SMEM_LIMIT, true));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ch.C, P.p.batch, 1);
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = ch.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ch.C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MPSB_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, P));
  return MPSB_OK;
}

// Blocked QR for matrices beyond the cluster's shared memory (for example 2048 x 512): the working
// matrix is p.Q (X copied in unless they coincide); every outer panel of up to BP columns is
// factored by the cluster kernel (its R rows written back in place, its reflectors and T kept), the
// trailing columns get A -= V (T^H (V^H A)) by three tensor-core GEMMs, and Q is formed from all
// reflectors.  BP = 64: the widest panel whose 2048 rows fit 16 CTAs' shared memory; the GEMMs'
// K = 64 then reads and writes the trailing columns n/64 times.
constexpr int BP = 64;

// The look-ahead lane of the blocked QR: created by the first (eager) call of a workspace.
int qr_side_lane(Workspace* ws) {
  if (ws->qr_side) return MPSB_OK;
  if (ws->capturing) {
    set_last_message("QR look-ahead lane first needed during graph capture");
    return MPSB_ERR_UNSUPPORTED;
  }
  MPSB_CUDA_TRY(cudaStreamCreateWithFlags(&ws->qr_side, cudaStreamNonBlocking));
  for (cudaEvent_t& e : ws->qr_ev) MPSB_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  ws->qr_side_ws = new Workspace();
  return MPSB_OK;
}

// The widest outer panel that fits one cluster at every row count of the factorisation (0: none).
int panel_width(int m, int n) {
  for (int w : {BP, 32, 16}) {
    w = std::min(w, n);
    bool ok = true;
    Choice ch;
    for (int p0 = 0; p0 < n && ok; p0 += w) ok = choose(m - p0, std::min(w, n - p0), ch, true);
    if (ok) return w;
  }
  return 0;
}

// Right-looking blocked QR with look-ahead: outer panel pi's block reflector I - V T V^H is applied
// to the next panel's columns on the main stream, which then factors that panel at once, while the
// same update of the columns after it runs on the look-ahead lane -- so the latency-bound panel
// factorisations overlap the trailing GEMMs.  Every column still gets the panels' updates in panel
// order (the main stream waits for the lane's update of panel pi-1 before it applies panel pi to the
// next panel), so the result is the unblocked order's.
int qr_blocked(const QrProblem& p, Workspace* ws, cudaStream_t s) {
  const int m = p.m, n = p.n, B = p.batch, bp = panel_width(m, n), npan = (n + bp - 1) / bp;
  const int64_t qr_ = p.q_r, qc = p.q_c;
  // scratch per problem: V [n][m], T [npan][bp][bp], G, M and B [n][n], W and W2 [n][bp] (the
  // lane's trailing update), Wn and W2n [bp][bp] (the next panel's update)
  const int64_t nV = (int64_t)m * n, nT = (int64_t)npan * bp * bp, nG = (int64_t)n * n, nW = (int64_t)n * bp,
                nWn = (int64_t)bp * bp;
  MPSB_TRY(devbuf_ensure(ws, ws->qr, (size_t)B * (nV + nT + 3 * nG + 2 * nW + 2 * nWn) * sizeof(cd)));
  MPSB_TRY(qr_side_lane(ws));
  Workspace* sw = ws->qr_side_ws;
  sw->capturing = ws->capturing;
  sw->per_problem = ws->per_problem;
  sw->err = ws->err;
  cudaStream_t ls = ws->qr_side;
  cudaEvent_t ev_v = ws->qr_ev[0], ev_t = ws->qr_ev[1];
  cd* Vb = static_cast<cd*>(ws->qr.p);
  cd* Tb = Vb + B * nV;
  cd* Gb = Tb + B * nT;
  cd* Mb = Gb + B * nG;
  cd* Bb = Mb + B * nG;
  cd* Wb = Bb + B * nG;
  cd* W2 = Wb + B * nW;
  cd* Wn = W2 + B * nW;
  cd* W2n = Wn + B * nWn;
  cd* A = p.Q;
  if (p.X != p.Q || p.x_r != qr_ || p.x_c != qc || p.x_b != p.q_b)
    MPSB_TRY(mat_launch(MAT_COPY, m, n, B, p.X, p.x_r, p.x_c, p.x_b, A, qr_, qc, p.q_b, ws, s));
  MPSB_CUDA_TRY(cudaMemsetAsync(Vb, 0, (size_t)B * nV * sizeof(cd), s));
  const cd one = cmk(1.0, 0.0), zero = cmk(0.0, 0.0), mone = cmk(-1.0, 0.0);

  // factor panel pi (its columns have every earlier panel's update)
  auto factor = [&](int pi) -> int {
    const int p0 = pi * bp, pw = std::min(bp, n - p0), mp = m - p0;
    Choice ch;
    if (!choose(mp, pw, ch, true)) {
      set_last_message("QR panel of %d x %d does not fit the cluster kernel", mp, pw);
      return MPSB_ERR_UNSUPPORTED;
    }
    QrParams P = {};
    P.p = p;
    P.p.m = mp; P.p.n = pw;
    P.p.X = A + p0 * qr_ + p0 * qc; P.p.x_r = qr_; P.p.x_c = qc; P.p.x_b = p.q_b;
    P.p.Q = nullptr;
    P.p.R = A + p0 * qr_ + p0 * qc; P.p.r_r = qr_; P.p.r_c = qc; P.p.r_b = p.q_b;   // R rows back in place
    P.form_q = 0;
    P.V = Vb + p0 + (int64_t)p0 * m; P.v_ld = m; P.v_b = nV;
    P.T = Tb + (int64_t)pi * bp * bp; P.t_ld = bp; P.t_b = nT;
    count_launch(ws);
    return launch_cluster(P, ch, s);
  };
  auto gemm = [&](int M, int N, int K, const cd* Ap, int64_t am, int64_t ak, int64_t ab, bool ca, const cd* Bp, int64_t bk,
                  int64_t bn, int64_t bb, cd* Cp, int64_t cm, int64_t cn, int64_t cb, cd alpha, cd beta, Workspace* w,
                  cudaStream_t st) -> int {
    Gemm g;
    g.M = M; g.N = N; g.K = K; g.batch = B;
    g.A = Ap; g.a_m = am; g.a_k = ak; g.a_b = ab; g.conjA = ca;
    g.B = Bp; g.b_k = bk; g.b_n = bn; g.b_b = bb;
    g.C = Cp; g.c_m = cm; g.c_n = cn; g.c_b = cb;
    g.alpha = alpha; g.beta = beta;
    return gemm_launch(g, w, st);
  };
  // columns c0 .. c0 + nc - 1 of A <- (I - V T V^H)^H applied by panel pi, on stream st
  auto update = [&](int pi, int c0, int nc, cd* W, cd* Wt, int64_t wb, Workspace* w, cudaStream_t st) -> int {
    const int p0 = pi * bp, pw = std::min(bp, n - p0), mp = m - p0;
    const cd* V = Vb + p0 + (int64_t)p0 * m;   // rows p0.., leading dimension m
    cd* At = A + p0 * qr_ + (int64_t)c0 * qc;
    MPSB_TRY(gemm(pw, nc, mp, V, m, 1, nV, true, At, qr_, qc, p.q_b, W, 1, bp, wb, one, zero, w, st));    // V^H A
    MPSB_TRY(gemm(pw, nc, pw, Tb + (int64_t)pi * bp * bp, bp, 1, nT, true, W, 1, bp, wb, Wt, 1, bp, wb, one, zero, w, st));
    return gemm(mp, nc, pw, V, 1, m, nV, false, Wt, 1, bp, wb, At, qr_, qc, p.q_b, mone, one, w, st);     // A -= V Wt
  };

  MPSB_TRY(factor(0));
  bool lane_pending = false;   // the lane holds an update the main stream has not waited for
  for (int pi = 0; pi + 1 < npan; ++pi) {
    const int c1 = (pi + 1) * bp, nnext = std::min(bp, n - c1);
    const int c2 = c1 + nnext, nrest = n - c2;
    // the next panel's columns have panel pi-1's update only once the lane's update is done
    if (lane_pending) {
      MPSB_CUDA_TRY(cudaStreamWaitEvent(s, ev_t, 0));
      lane_pending = false;
    }
    int st = MPSB_OK;
    if (nrest > 0) {   // V_pi and T_pi are final on the main stream: fork the trailing update
      MPSB_CUDA_TRY(cudaEventRecord(ev_v, s));
      MPSB_CUDA_TRY(cudaStreamWaitEvent(ls, ev_v, 0));
      st = update(pi, c2, nrest, Wb, W2, nW, sw, ls);
      MPSB_CUDA_TRY(cudaEventRecord(ev_t, ls));   // recorded on failure too, so the join below holds
      lane_pending = true;
    }
    if (st == MPSB_OK) st = update(pi, c1, nnext, Wn, W2n, nWn, ws, s);
    if (st == MPSB_OK) st = factor(pi + 1);
    if (st != MPSB_OK) {   // never leave the lane forked
      cudaStreamWaitEvent(s, ev_t, 0);
      return st;
    }
  }
  if (lane_pending) MPSB_CUDA_TRY(cudaStreamWaitEvent(s, ev_t, 0));   // join the lane
  ws->launches += sw->launches;
  sw->launches = 0;
  if (p.R) MPSB_TRY(mat_launch(MAT_UPPER, n, n, B, A, qr_, qc, p.q_b, p.R, p.r_r, p.r_c, p.r_b, ws, s));
  MPSB_TRY(mat_launch(MAT_IDENT, m, n, B, A, 0, 0, 0, A, qr_, qc, p.q_b, ws, s));

  // Q = E - V M, M = T V1^H by back substitution over the outer panels: T^{-1} = diag(1/tau) +
  // striu(V^H V) is block upper triangular with the panels' T_p inverted on its diagonal, so with
  // G = V^H V and B = V1^H (upper triangular)  M_p = T_p (B_p - sum_{q > p} G_pq M_q), p = last .. 0
  // (no division; zero rows for tau = 0 reflectors).
  MPSB_TRY(gemm(n, n, m, Vb, m, 1, nV, true, Vb, 1, m, nV, Gb, 1, n, nG, one, zero, ws, s));
  MPSB_TRY(mat_launch(MAT_CTRANS_UPPER, n, n, B, Vb, 1, m, nV, Bb, 1, n, nG, ws, s));
  MPSB_CUDA_TRY(cudaMemsetAsync(Mb, 0, (size_t)B * nG * sizeof(cd), s));
  for (int pi = npan - 1; pi >= 0; --pi) {
    const int p0 = pi * bp, pw = std::min(bp, n - p0), kb = p0 + pw, nt = n - kb;
    if (nt > 0)
      MPSB_TRY(gemm(pw, nt, nt, Gb + p0 + (int64_t)kb * n, 1, n, nG, false, Mb + kb + (int64_t)kb * n, 1, n, nG,
                    Bb + p0 + (int64_t)kb * n, 1, n, nG, mone, one, ws, s));
    MPSB_TRY(gemm(pw, pw + nt, pw, Tb + (int64_t)pi * bp * bp, 1, bp, nT, false, Bb + p0 + (int64_t)p0 * n, 1, n, nG,
                  Mb + p0 + (int64_t)p0 * n, 1, n, nG, one, zero, ws, s));
  }
  return gemm(m, n, n, Vb, 1, m, nV, false, Mb, 1, n, nG, A, qr_, qc, p.q_b, mone, one, ws, s);
}

}  // namespace

bool qr_supported(int m, int n) {
  Choice ch;
  return m >= n && n >= 1 && n <= 512 && (choose(m, n, ch) || panel_width(m, n) > 0);
}

int qr_launch(const QrProblem& p, Workspace* ws, cudaStream_t s) {
  if (p.m < p.n || p.n < 1 || p.batch < 1) return MPSB_ERR_DIMENSION;
  if (p.batch > 65535) return MPSB_ERR_UNSUPPORTED;
  if (!ws) return MPSB_ERR_INVALID_ARG;
  const int m = p.m, n = p.n;
  if (!qr_supported(m, n)) {
    set_last_message("QR of a %d x %d matrix (batch %d) is beyond the supported shapes", m, n, p.batch);
    return MPSB_ERR_UNSUPPORTED;
  }
  Choice ch;
  if (!choose(m, n, ch)) return qr_blocked(p, ws, s);
  const int64_t nT = (int64_t)((n + NB - 1) / NB) * NB * NB;
  MPSB_TRY(devbuf_ensure(ws, ws->qr, (size_t)p.batch * nT * sizeof(cd)));
  QrParams P = {};
  P.p = p;
  P.form_q = 1;
  P.T = static_cast<cd*>(ws->qr.p);
  P.t_b = nT;
  return launch_cluster(P, ch, s);
}

}  // namespace mpsb
