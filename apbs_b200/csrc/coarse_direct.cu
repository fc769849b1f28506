// Direct solve of the FP64 coarsest level (LPBE) by its planes.
//
// Stands in for the reference's banded Cholesky (Vdpbfa/Vdpbsl,
// src/pmgc/mlinpckd.c:57-83, 194-233) where the level has too many unknowns
// for a sequential band factor: B x = b, B the reference's band matrix as a
// 27-point operator (k_band_restencil).  In the order of its planes B is block
// tridiagonal, with a nine-point coupling between successive planes.  Planes
// are eliminated from both ends towards the middle one:
//   S_k = B_kk - B_kp D_p B_pk,  D_k = S_k^-1   (p the plane before k),
// and the middle plane takes both sides.  A solve goes the same way with
// vectors and back out again:
//   z_k = D_k (b_k - B_kp z_p),  x_k = z_k - D_k B_kn x_n  (n the plane after),
// so its chain is as long as the level has planes, whatever their size, each
// link one dense product that all the side's CTAs share.  The inverses D_k are
// made once per operator.
//
// Measured: one solve of a 27^3 level 126 us, where the refinement kernel
// (k_coarse_exact), which is left for planes that do not fit, takes 2.8 ms; 11^3
// 25 us against 0.88 ms.  The factors take 6.7 ms at 27^3, 1.7 ms at 19^3 and
// 0.52 ms at 11^3, once per operator.
#include <algorithm>
#include <mutex>

#include "coarse_direct.cuh"
#include "mg_kernels.cuh"
#include "mixed.cuh"
#include "quotients.cuh"
#include "solver_internal.cuh"

namespace pmgb {

namespace {

constexpr int kRows = 16;            // rows of a plane's matrix per CTA, and of a pivot block
constexpr int kFactorUpdate = 384;   // threads that update rows; the rest inverts pivot blocks
constexpr int kFactorThreads = kFactorUpdate + kRows * kRows;
constexpr int kSolveThreads = 32 * kRows;  // a warp per row
constexpr int kPlanesMax = 64;
constexpr long long kWaitNs = 200LL * 1000 * 1000;  // 200 ms per wait

struct Args {
  Grid g;
  int p, pp, ez, mid;   // unknowns of a plane, the same in whole blocks, planes, the middle one
  const double* op[14];
  double* D;            // [ez][pp][pp]
  double* pan;          // [2][pp][pp]: rows of each pivot block before its step
  double* piv;          // [2][pp / 16][16][16]: inverted pivot blocks
  unsigned* flag;       // [0, 1] panels published per side, [2, 3] CTAs through a plane
  int* info;            // set where a pivot is not positive
  int* err;             // waits that ran out
  const double* b;
  double* x;
  unsigned long long* mail;  // [2 passes][ez][pp][2]: values with their launch's tag
  unsigned* counters;        // launches of each CTA
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A bounded wait: `there()` until it holds, or 200 ms went by here, or another
// wait ran out.
template <class F>
__device__ __forceinline__ void wait_for(int* err, volatile int* failed, F there) {
  unsigned long long t0 = 0;
  for (int spins = 1; !there(); spins++) {
    if ((spins & 63) != 0) continue;
    if (*failed || *(volatile int*)err) {
      *failed = 1;
      return;
    }
    const unsigned long long t = now_ns();
    if (t0 == 0) t0 = t;
    if ((long long)(t - t0) > kWaitNs) {
      *failed = 1;
      atomicAdd(err, 1);
      return;
    }
  }
}
__device__ __forceinline__ unsigned acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// -B(a, a + (dx, dy, dz)) for interior a, dz = +-1; 0 where the neighbour is
// not an interior point
__device__ __forceinline__ double coupling(const Args& A, int i, int j, int k, int dx, int dy,
                                           int dz) {
  const int ni = i + dx, nj = j + dy;
  if (ni < 1 || nj < 1 || ni > A.g.nx - 2 || nj > A.g.ny - 2) return 0.0;
  if (dz < 0) {  // stored at the neighbour, pointing back up
    i = ni;
    j = nj;
    k -= 1;
    dx = -dx;
    dy = -dy;
  }
  const int code = dy == 0 ? (dx == 0 ? UC : (dx > 0 ? UE : UW))
                           : (dx == 0 ? (dy > 0 ? UN : US)
                                      : (dy > 0 ? (dx > 0 ? UNE : UNW) : (dx > 0 ? USE : USW)));
  return A.op[code][A.g.idx(i, j, k)];
}

// B(a, c) within plane k, a = (i, j), c = (ci, cj)
__device__ __forceinline__ double in_plane(const Args& A, int i, int j, int ci, int cj, int k) {
  const int dx = ci - i, dy = cj - j;
  if (dx < -1 || dx > 1 || dy < -1 || dy > 1) return 0.0;
  if (dx == 0 && dy == 0) return A.op[OC][A.g.idx(i, j, k)];
  if (dy == 0) return -A.op[OE][A.g.idx(dx > 0 ? i : ci, j, k)];
  if (dx == 0) return -A.op[ON][A.g.idx(i, dy > 0 ? j : cj, k)];
  // a diagonal neighbour: stored at the lower row's point, to the east or west
  if (dy > 0) return -A.op[dx > 0 ? ONE : ONW][A.g.idx(i, j, k)];
  return -A.op[dx < 0 ? ONE : ONW][A.g.idx(ci, cj, k)];
}

// The inverses D_k.  One CTA per 16 rows of a plane's matrix and side, its rows
// in shared memory; Gauss-Jordan by pivot blocks of 16 (B is positive
// definite).  The CTA of block s publishes its rows and the inverted block, and
// every CTA subtracts their product with its own 16 x 16 block from its rows:
// bounded by those FP64 products (16 x 16 per column and step) and by the chain
// from one block to the next, which is why the next block's owner brings that
// block up to date first and inverts it while its other threads update the rest.
__global__ void __launch_bounds__(kFactorThreads, 1) k_direct_factor(Args A) {
  extern __shared__ double sm[];
  const int pp = A.pp, G = pp / kRows;
  double* S = sm;                 // [16][pp]
  double* T = S + kRows * pp;     // [16][pp]
  __shared__ double P[kRows * kRows], L[kRows * kRows], M[2][kRows * kRows];
  __shared__ volatile int failed;
  const int tid = threadIdx.x;
  const int side = blockIdx.x / G, cta = blockIdx.x - side * G, r0 = cta * kRows;
  const int ex = A.g.nx - 2;
  double* pan = A.pan + (size_t)side * pp * pp;
  double* piv = A.piv + (size_t)side * pp * kRows;
  unsigned* shown = A.flag + side;
  unsigned* through = A.flag + 2 + side;
  if (tid == 0) failed = 0;
  __syncthreads();
  // inverts the block in M[0] (threads kFactorUpdate and up) into piv[s]
  auto invert = [&](int s) {
    const int e = tid - kFactorUpdate, r = e / kRows, c = e - r * kRows;
    for (int q = 0; q < kRows; q++) {
      const double* m = M[q & 1];
      const double d = m[q * kRows + q];
      const double y = reciprocal(d);
      const double row = m[q * kRows + c], col = m[r * kRows + q];
      double v;
      if (r == q) v = c == q ? y : row * y;
      else if (c == q) v = -col * y;
      else v = fma(-col * y, row, m[e]);
      if (e == 0 && !(d > 0.0)) A.info[0] = 1;
      M[(q + 1) & 1][e] = v;
      asm volatile("bar.sync 1, %0;" ::"n"(kRows * kRows) : "memory");
    }
    __stcg(piv + (size_t)s * kRows * kRows + e, M[kRows & 1][e]);
  };
  const int nplanes = side == 0 ? A.mid + 1 : A.ez - 1 - A.mid;
  for (int t = 0; t < nplanes; t++) {
    const int k = side == 0 ? t : A.ez - 1 - t;  // plane k is at kk = k + 1 of the grid
    // S = B_kk - sum over the planes before of B_kp D_p B_pk, this CTA's rows
    for (int e = tid; e < kRows * pp; e += kFactorThreads) {
      const int r = r0 + e / pp, c = e % pp;
      double v = r == c ? 1.0 : 0.0;  // rows beyond the plane: the identity
      if (r < A.p && c < A.p)
        v = in_plane(A, 1 + r % ex, 1 + r / ex, 1 + c % ex, 1 + c / ex, k + 1);
      S[e] = v;
    }
    for (int from = 0; from < 2; from++) {
      const int dz = from == 0 ? -1 : 1, kp = k + dz;
      // the middle plane follows both sides, any other its own side's last
      const bool used = k == A.mid ? (from == 0 ? kp >= 0 : kp < A.ez)
                                   : (t > 0 && from == (side == 0 ? 0 : 1));
      if (!used) continue;
      const unsigned need = (unsigned)(G * (k == A.mid && from == 1 ? A.ez - 1 - A.mid : t));
      if (tid == 0)
        wait_for(A.err, &failed,
                 [&] { return acquire(A.flag + 2 + (k == A.mid ? from : side)) >= need; });
      __syncthreads();
      const double* D = A.D + (size_t)kp * pp * pp;
      // T = C D, C the (negated) coupling of this CTA's rows with plane kp
      for (int c = tid; c < pp; c += kFactorThreads)
        for (int rr = 0; rr < kRows; rr++) {
          const int r = r0 + rr;
          double v = 0.0;
          if (r < A.p && c < A.p) {
            const int i = 1 + r % ex, j = 1 + r / ex;
            for (int dy = -1; dy <= 1; dy++)
              for (int dx = -1; dx <= 1; dx++) {
                const double u = coupling(A, i, j, k + 1, dx, dy, dz);
                if (u != 0.0) v = fma(u, __ldcg(D + (size_t)(r + dy * ex + dx) * pp + c), v);
              }
          }
          T[rr * pp + c] = v;
        }
      __syncthreads();
      for (int c = tid; c < A.p; c += kFactorThreads) {
        const int ci = 1 + c % ex, cj = 1 + c / ex;
        for (int dy = -1; dy <= 1; dy++)
          for (int dx = -1; dx <= 1; dx++) {
            const double u = coupling(A, ci, cj, k + 1, dx, dy, dz);
            if (u == 0.0) continue;
            const double* Tc = T + c + dy * ex + dx;
            for (int rr = 0; rr < kRows; rr++)
              S[rr * pp + c] = fma(-u, Tc[rr * pp], S[rr * pp + c]);
          }
      }
      __syncthreads();
    }
    __syncthreads();
    if (cta == 0) {  // the first pivot block
      if (tid >= kFactorUpdate) {
        const int e = tid - kFactorUpdate;
        M[0][e] = S[(e / kRows) * pp + e % kRows];
        asm volatile("bar.sync 1, %0;" ::"n"(kRows * kRows) : "memory");
        invert(0);
      } else {
        for (int e = tid; e < kRows * pp; e += kFactorUpdate) __stcg(pan + e, S[e]);
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) atomicAdd(shown, 1u);
    }
    for (int s = 0; s < G; s++) {
      const unsigned want = (unsigned)(t * G + s + 1);
      if (tid == 0) wait_for(A.err, &failed, [&] { return acquire(shown) >= want; });
      __syncthreads();
      const double* panel = pan + (size_t)s * kRows * pp;
      const int c0 = s * kRows, c1 = c0 + kRows;  // the pivot's columns, the next one's
      const bool own = cta == s, next = cta == s + 1;
      if (tid < kRows * kRows) P[tid] = __ldcg(piv + (size_t)s * kRows * kRows + tid);
      __syncthreads();
      if (tid < kRows * kRows) {
        const int r = tid / kRows, c = tid - r * kRows;
        double v = 0.0;
        for (int q = 0; q < kRows; q++) v = fma(S[r * pp + c0 + q], P[q * kRows + c], v);
        L[tid] = own ? -P[tid] : v;
      }
      __syncthreads();
      if (next) {
        if (tid >= kFactorUpdate) {
          const int e = tid - kFactorUpdate, r = e / kRows, c = c1 + e % kRows;
          double v = S[r * pp + c];
          for (int q = 0; q < kRows; q++)
            v = fma(-L[r * kRows + q], __ldcg(panel + (size_t)q * pp + c), v);
          M[0][e] = v;
        }
        __syncthreads();
      }
      if (tid < kFactorUpdate) {
        double* out = next ? pan + (size_t)c1 * pp : nullptr;
        for (int c = tid; c < pp; c += kFactorUpdate) {
          if (c >= c0 && c < c1) {
            for (int r = 0; r < kRows; r++) {
              const double v = -L[r * kRows + c - c0];
              S[r * pp + c] = v;
              if (out) __stcg(out + (size_t)r * pp + c, v);
            }
            continue;
          }
          double w[kRows];
#pragma unroll
          for (int q = 0; q < kRows; q++) w[q] = __ldcg(panel + (size_t)q * pp + c);
#pragma unroll 4
          for (int r = 0; r < kRows; r++) {
            double v = own ? 0.0 : S[r * pp + c];
#pragma unroll
            for (int q = 0; q < kRows; q++) v = fma(-L[r * kRows + q], w[q], v);
            S[r * pp + c] = v;
            if (out) __stcg(out + (size_t)r * pp + c, v);
          }
        }
      } else if (next) {
        invert(s + 1);
      }
      if (next) __threadfence();
      __syncthreads();
      if (next && tid == 0) atomicAdd(shown, 1u);
    }
    double* D = A.D + (size_t)k * pp * pp + (size_t)r0 * pp;
    for (int e = tid; e < kRows * pp; e += kFactorThreads) __stcg(D + e, S[e]);
    __threadfence();
    __syncthreads();
    if (tid == 0) atomicAdd(through, 1u);
  }
}

// One solve.  CTA c of a side has rows 16 c .. 16 c + 15 of every plane of its
// side, a warp each; the rows of D_k come by bulk copy two planes ahead.  A
// plane's values go to all CTAs as tagged words that validate themselves (the
// readers poll the values, there is no barrier).  Bounded by that hand-over and
// by reading every D_k twice.
__global__ void __launch_bounds__(kSolveThreads, 1) k_direct_solve(Args A) {
  extern __shared__ __align__(128) double sm[];
  const int pp = A.pp, G = pp / kRows, slab = kRows * pp;
  double* rows = sm;               // [2][16][pp]
  double* v = rows + 2 * slab;     // [pp] the last plane's values
  double* y = v + pp;              // [pp] the product's vector
  double* zown = y + pp;           // [kPlanesMax][16] this CTA's z
  __shared__ unsigned long long full[2];
  __shared__ unsigned tag_sh;
  __shared__ volatile int failed;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int side = blockIdx.x / G, r0 = (blockIdx.x - side * G) * kRows;
  const int ex = A.g.nx - 2;
  const int nout = side == 0 ? A.mid : A.ez - 1 - A.mid;  // planes of this side
  const int nsteps = 2 * nout + (side == 0 ? 1 : 0);
  auto plane_of = [&](int i) -> int {  // inwards, the middle one (side 0), outwards
    if (side == 0) return i <= nout ? i : 2 * nout - i;
    return i < nout ? A.ez - 1 - i : A.mid + 1 + (i - nout);
  };
  const unsigned bar0 = (unsigned)__cvta_generic_to_shared(&full[0]);
  auto copy_rows = [&](int i) {
    const unsigned bar = bar0 + 8u * (i & 1), bytes = (unsigned)slab * 8u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"((unsigned)__cvta_generic_to_shared(rows + (i & 1) * slab)),
        "l"(A.D + (size_t)plane_of(i) * pp * pp + (size_t)r0 * pp), "r"(bytes), "r"(bar)
        : "memory");
  };
  if (tid == 0) {
    failed = 0;
    tag_sh = A.counters[blockIdx.x] + 1u;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  for (int e = A.p + tid; e < pp; e += kSolveThreads) y[e] = 0.0;
  __syncthreads();
  if (tid == 0)
    for (int i = 0; i < 2 && i < nsteps; i++) copy_rows(i);
  const unsigned tag = tag_sh;
  const unsigned long long hi = (unsigned long long)tag << 32;
  // the values of plane k in pass `pass` into v
  auto receive = [&](int pass, int k) {
    for (int r = tid; r < A.p; r += kSolveThreads) {
      const unsigned long long* slot = A.mail + 2 * (((size_t)pass * A.ez + k) * pp + r);
      unsigned long long w0 = 0, w1 = 0;
      wait_for(A.err, &failed, [&] {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(w0), "=l"(w1)
                     : "l"(slot));
        return (unsigned)(w0 >> 32) == tag && (unsigned)(w1 >> 32) == tag;
      });
      v[r] = __longlong_as_double((long long)((w1 << 32) | (unsigned)w0));
    }
  };
  // sum of couplings of point r of plane k with plane k + dz times v
  auto spread = [&](int r, int k, int dz, const double* cf) -> double {
    double t = 0.0;
#pragma unroll
    for (int n = 0; n < 9; n++) {
      const double u = cf[n];
      if (u != 0.0) t = fma(u, v[r + (n / 3 - 1) * ex + n % 3 - 1], t);
    }
    return t;
  };
  for (int i = 0; i < nsteps; i++) {
    const int k = plane_of(i);
    const bool out = i > nout || (side == 1 && i >= nout);  // outwards: from x of the next plane
    const bool middle = side == 0 && i == nout;
    // the plane whose values this one takes
    const int from = (side == 0) != out ? -1 : 1;
    const bool has = out || (middle ? A.mid > 0 : i > 0);
    constexpr int kPer = 2;  // points of a plane per thread (1024 at most)
    double cf[kPer][9], acc[kPer];
#pragma unroll
    for (int n = 0; n < kPer; n++) {
      const int r = tid + n * kSolveThreads;
      acc[n] = 0.0;
      if (r >= A.p) continue;
      const int pi = 1 + r % ex, pj = 1 + r / ex;
      if (!out) acc[n] = __ldg(A.b + A.g.idx(pi, pj, k + 1));
      if (has)
#pragma unroll
        for (int d = 0; d < 9; d++)
          cf[n][d] = coupling(A, pi, pj, k + 1, d % 3 - 1, d / 3 - 1, from);
    }
    if (has) {
      receive(out ? 1 : 0, k + from);
      __syncthreads();
#pragma unroll
      for (int n = 0; n < kPer; n++) {
        const int r = tid + n * kSolveThreads;
        if (r < A.p) acc[n] += spread(r, k, from, cf[n]);
      }
    }
    if (middle && A.mid + 1 < A.ez) {  // the other side's last plane too
      __syncthreads();
#pragma unroll
      for (int n = 0; n < kPer; n++) {
        const int r = tid + n * kSolveThreads;
        if (r >= A.p) continue;
#pragma unroll
        for (int d = 0; d < 9; d++)
          cf[n][d] = coupling(A, 1 + r % ex, 1 + r / ex, k + 1, d % 3 - 1, d / 3 - 1, 1);
      }
      receive(0, A.mid + 1);
      __syncthreads();
#pragma unroll
      for (int n = 0; n < kPer; n++) {
        const int r = tid + n * kSolveThreads;
        if (r < A.p) acc[n] += spread(r, k, 1, cf[n]);
      }
    }
#pragma unroll
    for (int n = 0; n < kPer; n++) {
      const int r = tid + n * kSolveThreads;
      if (r < A.p) y[r] = acc[n];
    }
    __syncthreads();
    // row r0 + wid of D_k times y
    {
      // (a copy always arrives, and must have before the CTA ends: this wait does
      // not give up with the others)
      const unsigned bar = bar0 + 8u * (i & 1), parity = (unsigned)(i >> 1) & 1u;
      for (int n = 0; n < (1 << 22); n++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred q;\n mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 q, [%1], "
            "%2;\n selp.u32 %0, 1, 0, q;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) break;
      }
    }
    const double2* row = reinterpret_cast<const double2*>(rows + (i & 1) * slab + wid * pp);
    const double2* yv = reinterpret_cast<const double2*>(y);
    double s0 = 0.0, s1 = 0.0;
    for (int c = lane; c < pp / 2; c += 32) {
      const double2 a = row[c], w = yv[c];
      s0 = fma(a.x, w.x, s0);
      s1 = fma(a.y, w.y, s1);
    }
    double s = s0 + s1;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int r = r0 + wid;
    if (lane == 0 && r < A.p) {
      if (out) s += zown[(k < A.mid ? k : A.ez - 1 - k) * kRows + wid];
      const bool final_x = out || middle;
      const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
      unsigned long long* slot = A.mail + 2 * (((size_t)(final_x ? 1 : 0) * A.ez + k) * pp + r);
      asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot),
                   "l"((bits & 0xffffffffull) | hi), "l"((bits >> 32) | hi)
                   : "memory");
      if (final_x) A.x[A.g.idx(1 + r % ex, 1 + r / ex, k + 1)] = s;
      else zown[i * kRows + wid] = s;
    }
    __syncthreads();  // v, y and this step's rows are free
    if (tid == 0 && i + 2 < nsteps) copy_rows(i + 2);
  }
  if (tid == 0) A.counters[blockIdx.x] = tag;
}

constexpr size_t factor_smem(int pp) { return 2 * (size_t)kRows * pp * sizeof(double); }
constexpr size_t solve_smem(int pp) {
  return (2 * (size_t)kRows * pp + 2 * (size_t)pp + kPlanesMax * kRows) * sizeof(double);
}
// The largest plane: its slabs (two in the solve) and the static arrays in a
// CTA's 227 KB of shared memory.
constexpr int kPlaneMax = 816;
static_assert(factor_smem(kPlaneMax) + 16384 <= 232448 && solve_smem(kPlaneMax) + 1024 <= 232448 &&
                  solve_smem(kPlaneMax + kRows) + 1024 > 232448 && kPlaneMax <= 2 * kSolveThreads,
              "kPlaneMax");

// Unknowns of a plane in whole blocks, 0 where the level does not fit.
int direct_blocks(Grid g) {
  const int p = (g.nx - 2) * (g.ny - 2), ez = g.nz - 2;
  const int pp = (p + kRows - 1) / kRows * kRows;
  return ez <= kPlanesMax && pp <= kPlaneMax ? pp : 0;
}

// The kernels' limits of dynamic shared memory belong to the process, not to a
// calculation: set once per device, to what the largest plane takes.  (A
// calculation that set its own would lower the limit under one with larger
// planes, whose next launches were refused.)
bool direct_smem_ready(int dev) {
  static std::once_flag once[16];
  static bool ok[16];
  if (dev < 0 || dev >= 16) return false;
  std::call_once(once[dev], [dev] {
    ok[dev] = cudaFuncSetAttribute(k_direct_factor, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)factor_smem(kPlaneMax)) == cudaSuccess &&
              cudaFuncSetAttribute(k_direct_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)solve_smem(kPlaneMax)) == cudaSuccess;
  });
  return ok[dev];
}

// The quotients of quotients.cuh beside the division's, for the test.
__global__ void k_quotients(int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = a[i] / b[i];
  out[n + i] = div_by(a[i], b[i], div_factor(b[i]));
  out[2 * n + i] = reciprocal(b[i]);
}

}  // namespace

struct DirectState {
  Grid g;
  int pp;
  double* op[14];
  double *D, *pan, *piv;
  unsigned long long* mail;
  unsigned* words;  // [0, 4) flags, then the counters of the solve's CTAs
  int* info;        // [0] pivot, [1] wrap
};

size_t direct_bytes(Grid g) {
  const size_t pp = (size_t)direct_blocks(g), ez = g.nz - 2;
  if (pp == 0) return 0;
  return pp * pp * (ez + 2) * sizeof(double) + 2 * pp * kRows * sizeof(double) +
         14 * g.n() * sizeof(double) + 4 * ez * pp * sizeof(unsigned long long);
}

void direct_destroy(DirectState* d) {
  if (!d) return;
  for (double* p : d->op) cudaFree(p);
  cudaFree(d->D);
  cudaFree(d->pan);
  cudaFree(d->piv);
  cudaFree(d->mail);
  cudaFree(d->words);
  cudaFree(d->info);
  delete d;
}

static int direct_alloc(pmgb_solver* s, Grid g, int pp) {
  int dev = 0, sms = 0, coop = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  const int ctas = 2 * (pp / kRows);
  if (!coop || ctas > sms) return 0;
  if (!direct_smem_ready(dev) ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_direct_factor, kFactorThreads,
                                                    factor_smem(pp)) != cudaSuccess ||
      per * sms < ctas ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_direct_solve, kSolveThreads,
                                                    solve_smem(pp)) != cudaSuccess ||
      per * sms < ctas) {
    cudaGetLastError();
    return 0;
  }
  DirectState* d = new DirectState();
  s->direct = d;
  d->g = g;
  d->pp = pp;
  const size_t ez = g.nz - 2, n2 = (size_t)pp * pp;
  int ok = 1;
  for (int c = 0; c < 14; c++)
    ok &= cudaMalloc((void**)&d->op[c], g.n() * sizeof(double)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->D, ez * n2 * sizeof(double)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->pan, 2 * n2 * sizeof(double)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->piv, 2 * (size_t)pp * kRows * sizeof(double)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->mail, 4 * ez * pp * sizeof(unsigned long long)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->words, (4 + ctas) * sizeof(unsigned)) == cudaSuccess;
  ok &= cudaMalloc((void**)&d->info, 2 * sizeof(int)) == cudaSuccess;
  if (ok) {
    // tag 0 is no launch's
    ok &= cudaMemsetAsync(d->mail, 0, 4 * ez * pp * sizeof(unsigned long long), s->stream) ==
          cudaSuccess;
    ok &= cudaMemsetAsync(d->words, 0, (4 + ctas) * sizeof(unsigned), s->stream) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    direct_destroy(d);
    s->direct = nullptr;
    return 0;
  }
  return 1;
}

static Args direct_args(pmgb_solver* s) {
  const DirectState* d = s->direct;
  Args A;
  A.g = d->g;
  A.p = (d->g.nx - 2) * (d->g.ny - 2);
  A.pp = d->pp;
  A.ez = d->g.nz - 2;
  A.mid = A.ez / 2;
  for (int c = 0; c < 14; c++) A.op[c] = d->op[c];
  A.D = d->D;
  A.pan = d->pan;
  A.piv = d->piv;
  A.flag = d->words;
  A.info = d->info;
  A.err = reinterpret_cast<int*>(s->d_wave) + kWaveDirectErr;
  A.b = nullptr;
  A.x = nullptr;
  A.mail = d->mail;
  A.counters = d->words + 4;
  return A;
}

int direct_prepare(pmgb_solver* s) {
  const Level& C = s->lev[s->nlev - 1];
  const int pp = direct_blocks(C.g);
  if (pp == 0) return 0;
  if (!s->direct && !direct_alloc(s, C.g, pp)) return 0;
  DirectState* d = s->direct;
  cudaStream_t st = s->stream;
  for (int c = 0; c < 14; c++)
    PMGB_CUDA_OK(cudaMemsetAsync(d->op[c], 0, C.g.n() * sizeof(double), st));
  PMGB_CUDA_OK(cudaMemsetAsync(d->info, 0, 2 * sizeof(int), st));
  PMGB_CUDA_OK(cudaMemsetAsync(d->words, 0, 4 * sizeof(unsigned), st));
  launch_band_restencil(st, C.g, C.ops(), d->op, d->info + 1);
  Args A = direct_args(s);
  void* args[] = {&A};
  if (cudaLaunchCooperativeKernel((void*)k_direct_factor, dim3(2 * (pp / kRows)),
                                  dim3(kFactorThreads), args, factor_smem(pp),
                                  st) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  note_launches(2);
  s->wave_used = 1;  // the solve's waits are looked at where the wavefronts' are
  int info[2] = {0, 0}, nerr = 0;
  PMGB_CUDA_OK(cudaMemcpyAsync(info, d->info, sizeof(info), cudaMemcpyDeviceToHost, st));
  PMGB_CUDA_OK(cudaMemcpyAsync(&nerr, A.err, sizeof(int), cudaMemcpyDeviceToHost, st));
  PMGB_CUDA_OK(cudaStreamSynchronize(st));
  if (nerr) {  // the factors are not whole: no later solve may take them
    PMGB_CUDA_OK(cudaMemsetAsync(A.err, 0, sizeof(int), st));
    set_error("%d bounded device waits ran out (factor of the direct coarse solve)", nerr);
    return -1;
  }
  // a pivot that is not positive, or a band entry that is no grid neighbour's:
  // the band factor decides
  return info[0] == 0 && info[1] == 0;
}

int launch_direct_solve(pmgb_solver* s, cudaStream_t st, const double* b, double* x) {
  Args A = direct_args(s);
  A.b = b;
  A.x = x;
  void* args[] = {&A};
  if (cudaLaunchCooperativeKernel((void*)k_direct_solve, dim3(2 * (A.pp / kRows)),
                                  dim3(kSolveThreads), args, solve_smem(A.pp),
                                  st) != cudaSuccess) {
    set_error("direct coarse solve launch: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
  }
  return 1;
}

}  // namespace pmgb

// Testing hook: a / b by division and by div_by, and reciprocal(b), of n pairs; out
// has 3 n values.
extern "C" int pmgb_debug_quotients(int n, const double* a, const double* b, double* out) {
  using namespace pmgb;
  if (n < 1 || n > (1 << 24) || !a || !b || !out) {
    set_error("pmgb_debug_quotients: bad arguments");
    return 0;
  }
  const size_t bytes = (size_t)n * sizeof(double);
  double* d = nullptr;
  PMGB_CUDA_OK(cudaMalloc((void**)&d, 5 * bytes));
  cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  k_quotients<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
  note_launches(1);
  const cudaError_t e = cudaMemcpy(out, d + 2 * (size_t)n, 3 * bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  PMGB_CUDA_OK(e);
  return 1;
}
