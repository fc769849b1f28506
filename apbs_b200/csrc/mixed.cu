// Mixed-precision PMG: FP32 V-cycles inside an FP64 refinement loop.
//
// The outer loop is the reference's own stopping rule in FP64: the fine
// residual r = f - (A + cc) x, its 1-norm against ||f||_1 (Vmvcs,
// src/pmgc/mgcsd.c:140, 540-562), and the FP64 correction x += e.  Each
// correction e solves A e = r approximately with one V-cycle run entirely in
// FP32 on an FP32 copy of the operator hierarchy.  Differences from the FP64
// V-cycle (they change rounding, not the fixed point of the outer loop):
//   * 27-point levels are smoothed by 8-colour Gauss-Seidel (colours
//     (i&1, j&1, k&1) have no 27-point neighbours in common), fully parallel,
//     instead of the lexicographic red-black order the FP64 path reproduces;
//   * the hierarchy is coarsened (Galerkin, trilinear P) below the
//     reference's coarsest level until at most 512 unknowns remain, and that
//     level is solved exactly with the dense FP64 inverse of (A_c + diag cc_c)
//     (Gauss-Jordan, recomputed whenever cc changes).
// For NPBE the Newton iteration (newtond.c:162-548) is unchanged and in FP64;
// only its inner linear solves use FP32 V-cycles.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "gs7_rb.cuh"
#include "mixed.cuh"
#include "solver_internal.cuh"

namespace cg = cooperative_groups;

namespace pmgb {

namespace {

struct MLevel {
  Grid g;
  int nop;
  float* op[14];
  double* op64[14];  // FP64 operator (owned only on levels below the FP64 hierarchy)
  int own64;
  double* cc64;      // FP64 Helmholtz term of this level (owned on extra levels)
  float* cc;
  float* w0;
  float* x;
  float* x2;         // Chebyshev smoothing: second iterate (zero boundary) and direction
  float* d;
  Op ops64() const {
    Op o;
    for (int c = 0; c < 14; c++) o.c[c] = (c < nop) ? op64[c] : nullptr;
    o.nop = nop;
    return o;
  }
};

struct OpF {
  const float* c[14];
  int nop;
};

}  // namespace

// a divisor as quotient takes it (m 0: 1)
struct Quot {
  unsigned m, shift;
};

// one level of the FP32 hierarchy as seen by the tail kernel
struct TLev {
  Grid g;
  Quot dx, dy;       // div_const of nx - 2 and ny - 2: interior_at
  const float* op[14];
  const float* cc;
  float* w0;
  float* x;
  float* x2;
  float* d;
  const float* lam;  // Gershgorin bound of D^-1 A of this level
};

struct MixedState {
  int nlev;
  MLevel lev[16];
  float* r;      // fine-sized FP32 scratch
  float* w2;     // fine-sized FP32 scratch
  float* xs;     // second fine FP32 iterate of the single-pass sweep (zero boundary)
  float* d32;    // fine-level oC + cc in FP32, 1 on the boundary (single-pass sweep)
  double* dense;  // coarsest dense factor (n x n)
  double* dvec;   // coarsest rhs / solution in FP64
  int nd;
  int* dinfo;
  cudaGraphExec_t exec[2];
  long long kernels[2];
  int cc_ready;
  int info_pending;  // dense factor status not read yet (read with the next residual)
  int lo;             // lowest level with FP32 storage (0, or the FP64 coarsest)
  int zero_cc;        // levels >= lo carry no Helmholtz term (band operator)
  int* d_flag;        // device flag of the band restencil check
  int stale;          // FP64 operators rebuilt since the FP32 copies were made
  int tail_first;     // first level run by the cluster tail kernel (0: none)
  int tail_cluster;
  TLev* d_tlev;       // device copies of the level descriptors
  float* lam;         // per level: Gershgorin bound of D^-1 (A + cc) (Chebyshev smoothing)
  // the dense coarsest inverse runs on the solver's side stream: forked after
  // the coarsest Helmholtz term is in place, done when dense_ev completes
  cudaEvent_t dense_fork, dense_ev;
};

namespace {

#define CKM(call)                                                                      \
  do {                                                                                 \
    cudaError_t e__ = (call);                                                          \
    if (e__ != cudaSuccess) {                                                          \
      set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e__));  \
      return 0;                                                                        \
    }                                                                                  \
  } while (0)

OpF opf(const MLevel& L) {
  OpF o;
  for (int c = 0; c < 14; c++) o.c[c] = (c < L.nop) ? L.op[c] : nullptr;
  o.nop = L.nop;
  return o;
}

// ---------------------------------------------------------------------------
// conversions
// ---------------------------------------------------------------------------
// Many conversions in one launch: segment i converts a[i][0..n_i) into b[i].
constexpr int kConvSegs = 32;
struct ConvBatch {
  const double* a[kConvSegs];
  float* b[kConvSegs];
  unsigned long long off[kConvSegs + 1];  // running sums of the lengths
  int nseg;
};

__global__ void k_to_f32_batch(ConvBatch c) {
  const unsigned long long tot = c.off[c.nseg];
  int seg = 0;
  for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       q < tot; q += (unsigned long long)gridDim.x * blockDim.x) {
    while (q >= c.off[seg + 1]) seg++;  // q only grows along a thread's loop
    const unsigned long long e = q - c.off[seg];
    c.b[seg][e] = (float)c.a[seg][e];
  }
}

// Collects conversions and issues them kConvSegs at a time.
struct ConvQueue {
  cudaStream_t st;
  ConvBatch c{};
  explicit ConvQueue(cudaStream_t s) : st(s) {}
  void add(const double* a, float* b, size_t n) {
    if (n == 0) return;
    if (c.nseg == kConvSegs) flush();
    c.a[c.nseg] = a;
    c.b[c.nseg] = b;
    c.off[c.nseg + 1] = c.off[c.nseg] + n;
    c.nseg++;
  }
  void flush() {
    if (c.nseg == 0) return;
    k_to_f32_batch<<<blocks_for((size_t)c.off[c.nseg]), kThreads, 0, st>>>(c);
    note_launches(1);
    c = ConvBatch{};
  }
};

// ---------------------------------------------------------------------------
// FP32 stencils
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T nb27g(const T* const* c, Grid g, const T* x, size_t id) {
  const size_t sy = g.nx, sz = (size_t)g.nx * g.ny;
  T t = c[ON][id] * x[id + sy] + c[ON][id - sy] * x[id - sy] + c[OE][id] * x[id + 1] +
            c[OE][id - 1] * x[id - 1];
  t += c[ONE][id] * x[id + sy + 1] + c[ONW][id] * x[id + sy - 1] +
       c[ONW][id - sy + 1] * x[id - sy + 1] + c[ONE][id - sy - 1] * x[id - sy - 1];
  t += c[UC][id] * x[id + sz] + c[UN][id] * x[id + sz + sy] + c[US][id] * x[id + sz - sy] +
       c[UE][id] * x[id + sz + 1] + c[UW][id] * x[id + sz - 1];
  t += c[UNE][id] * x[id + sz + sy + 1] + c[UNW][id] * x[id + sz + sy - 1] +
       c[USE][id] * x[id + sz - sy + 1] + c[USW][id] * x[id + sz - sy - 1];
  t += c[UC][id - sz] * x[id - sz] + c[US][id - sz + sy] * x[id - sz + sy] +
       c[UN][id - sz - sy] * x[id - sz - sy] + c[UW][id - sz + 1] * x[id - sz + 1] +
       c[UE][id - sz - 1] * x[id - sz - 1];
  t += c[USW][id - sz + sy + 1] * x[id - sz + sy + 1] +
       c[USE][id - sz + sy - 1] * x[id - sz + sy - 1] +
       c[UNW][id - sz - sy + 1] * x[id - sz - sy + 1] +
       c[UNE][id - sz - sy - 1] * x[id - sz - sy - 1];
  return t;
}

__device__ __forceinline__ float nb27(const OpF& o, Grid g, const float* x, size_t id) {
  return nb27g<float>(o.c, g, x, id);
}

// ---------------------------------------------------------------------------
// Chebyshev smoothing of the FP32 27-point levels (an option of the mixed
// path's inner V-cycle, which is this project's own preconditioner; the
// FP64 stopping test decides convergence).  Jacobi-preconditioned
// Chebyshev iteration on the interval [b/16, b] of D^-1 (A + cc), b the
// Gershgorin bound max_i sum_j |a_ij| / a_ii of the level, in the three-term
// form of Adams, Brezina, Hu and Tuminaro (J. Comput. Phys. 188, 2003):
//   r_i = (f - (A + cc) x_i) / a_ii,
//   d_0 = r_0 / theta,  d_i = rho_i rho_{i-1} d_{i-1} + (2 rho_i / delta) r_i,
//   x_{i+1} = x_i + d_i,
// theta = (b + a)/2, delta = (b - a)/2, rho_0 = delta/theta,
// rho_i = 1/(2 theta/delta - rho_{i-1}).  Every step updates all points
// at once (one launch, or one barrier in the cluster tail) where the 8-colour
// Gauss-Seidel needs eight.  x_i and x_{i+1} alternate between two buffers.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cheb_coef(float b, int i, float& alpha, float& beta) {
  const float a = b * (1.0f / 16.0f);
  const float theta = 0.5f * (b + a), delta = 0.5f * (b - a);
  const float sigma = theta / delta;
  float rho = 1.0f / sigma, rho_prev = 0.0f;
  for (int s = 1; s <= i; s++) {
    rho_prev = rho;
    rho = 1.0f / (2.0f * sigma - rho_prev);
  }
  alpha = (i == 0) ? 0.0f : rho * rho_prev;
  beta = (i == 0) ? 1.0f / theta : 2.0f * rho / delta;
}

__device__ __forceinline__ void cheb_point(const OpF& o, Grid g, const float* cc, const float* f,
                                           const float* xin, float* xout, float* d, size_t id,
                                           float alpha, float beta) {
  const float dg = o.c[OC][id] + cc[id];
  const float xv = xin[id];
  const float r = (f[id] + nb27(o, g, xin, id) - dg * xv) / dg;
  const float dn = alpha * d[id] + beta * r;
  d[id] = dn;
  xout[id] = xv + dn;
}

__global__ void k_cheb_step(Grid g, OpF o, const float* __restrict__ cc,
                            const float* __restrict__ f, const float* __restrict__ xin,
                            float* __restrict__ xout, float* __restrict__ d,
                            const float* __restrict__ lam, int i) {
  float alpha, beta;
  cheb_coef(*lam, i, alpha, beta);
  const int ex = g.nx - 2, ey = g.ny - 2;
  const size_t nint = (size_t)ex * ey * (g.nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i0, j0, k0;
    interior_ijk(q, g.nx, g.ny, i0, j0, k0);
    cheb_point(o, g, cc, f, xin, xout, d, g.idx(i0, j0, k0), alpha, beta);
  }
}

// Gershgorin bound of D^-1 (A + cc) over the interior rows of a 27-point
// level (cc NULL: without the Helmholtz term), as a float maximum (positive
// floats order like their bit patterns)
__global__ void k_gersh(Grid g, OpF o, const float* __restrict__ cc, float* out) {
  const int ex = g.nx - 2, ey = g.ny - 2;
  const size_t nint = (size_t)ex * ey * (g.nz - 2);
  const size_t sy = g.nx, sz = (size_t)g.nx * g.ny;
  float mx = 0.0f;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, g.nx, g.ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    const float* const* c = o.c;
    float s = fabsf(c[ON][id]) + fabsf(c[ON][id - sy]) + fabsf(c[OE][id]) + fabsf(c[OE][id - 1]) +
              fabsf(c[ONE][id]) + fabsf(c[ONW][id]) + fabsf(c[ONW][id - sy + 1]) +
              fabsf(c[ONE][id - sy - 1]) + fabsf(c[UC][id]) + fabsf(c[UN][id]) +
              fabsf(c[US][id]) + fabsf(c[UE][id]) + fabsf(c[UW][id]) + fabsf(c[UNE][id]) +
              fabsf(c[UNW][id]) + fabsf(c[USE][id]) + fabsf(c[USW][id]) +
              fabsf(c[UC][id - sz]) + fabsf(c[US][id - sz + sy]) + fabsf(c[UN][id - sz - sy]) +
              fabsf(c[UW][id - sz + 1]) + fabsf(c[UE][id - sz - 1]) +
              fabsf(c[USW][id - sz + sy + 1]) + fabsf(c[USE][id - sz + sy - 1]) +
              fabsf(c[UNW][id - sz - sy + 1]) + fabsf(c[UNE][id - sz - sy - 1]);
    const float dg = c[OC][id] + (cc ? cc[id] : 0.0f);
    if (dg > 0.0f) mx = fmaxf(mx, 1.0f + s / dg);
  }
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(out), __float_as_int(mx));
}

__device__ __forceinline__ float nb7(const OpF& o, Grid g, const float* x, size_t id) {
  const size_t sy = g.nx, sz = (size_t)g.nx * g.ny;
  return o.c[ON][id] * x[id + sy] + o.c[ON][id - sy] * x[id - sy] + o.c[OE][id] * x[id + 1] +
         o.c[OE][id - 1] * x[id - 1] + o.c[UC][id - sz] * x[id - sz] + o.c[UC][id] * x[id + sz];
}

__global__ void k_gs7_f32(Grid g, OpF o, const float* __restrict__ D,
                          const float* __restrict__ fc, float* x, int parity) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int hr = (nx - 1) / 2;
  const size_t nslots = (size_t)hr * (ny - 2) * (nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nslots;
       q += (size_t)gridDim.x * blockDim.x) {
    int m, j, k;
    split3(q, hr, ny - 2, m, j, k);
    j += 1;
    k += 1;
    const int i = 1 + (((1 + j + k) & 1) != parity) + 2 * m;
    if (i > nx - 2) continue;
    const size_t id = g.idx(i, j, k);
    x[id] = (fc[id] + nb7(o, g, x, id)) / D[id];
  }
}

// The first colour pass from x = 0: f / D at the points of the colour, 0 at the
// others, so neither x nor the couplings are read and x needs no clearing before.
__global__ void k_gs7_f32_first(Grid g, const float* __restrict__ D, const float* __restrict__ fc,
                                float* __restrict__ x, int parity) {
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, g.nx, g.ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    x[id] = ((i + j + k) & 1) == parity ? fc[id] / D[id] : 0.f;
  }
}

// r = f - (A + cc) x on interior points of a 7-point level, D = oC + cc
__global__ void k_resid7_f32(Grid g, OpF o, const float* __restrict__ D,
                             const float* __restrict__ fc, const float* __restrict__ x, float* r) {
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, g.nx, g.ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    r[id] = fc[id] + nb7(o, g, x, id) - D[id] * x[id];
  }
}

// r = f - (A + cc) x on interior points of a 27-point level
__global__ void k_resid_f32(Grid g, OpF o, const float* __restrict__ cc,
                            const float* __restrict__ fc, const float* __restrict__ x, float* r) {
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, g.nx, g.ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    r[id] = fc[id] + nb27(o, g, x, id) - (o.c[OC][id] + cc[id]) * x[id];
  }
}

// 8-colour Gauss-Seidel on a 27-point level: colour c = (i&1)|(j&1)<<1|(k&1)<<2.
// One cluster runs nsweep sweeps (colour order ascending, or descending when
// reverse) with a cluster barrier between colours.
template <int CLUSTER>
__global__ void k_gs27_mc_cluster(Grid g, OpF o, const float* __restrict__ cc,
                                  const float* __restrict__ fc, float* x, int nsweep,
                                  int reverse) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  unsigned rank = 0;
  if (CLUSTER > 1) rank = cg::this_cluster().block_rank();
  const int gtid = rank * blockDim.x + threadIdx.x;
  const int nthr = CLUSTER * blockDim.x;
  const int hx = (nx - 1) / 2, hy = (ny - 1) / 2, hz = (nz - 1) / 2;  // slots per axis
  for (int sw = 0; sw < nsweep; sw++) {
    for (int cc8 = 0; cc8 < 8; cc8++) {
      const int c = reverse ? 7 - cc8 : cc8;
      const int pi = c & 1, pj = (c >> 1) & 1, pk = (c >> 2) & 1;
      const int tot = hx * hy * hz;
      for (int t = gtid; t < tot; t += nthr) {
        const int mi = t % hx, mj = (t / hx) % hy, mk = t / (hx * hy);
        // interior index with parity: i = 1 + ((1 + p) & 1) ... first interior
        // index of parity p is 1 if p == 1 else 2
        const int i = (pi ? 1 : 2) + 2 * mi;
        const int j = (pj ? 1 : 2) + 2 * mj;
        const int k = (pk ? 1 : 2) + 2 * mk;
        if (i > nx - 2 || j > ny - 2 || k > nz - 2) continue;
        const size_t id = g.idx(i, j, k);
        x[id] = (fc[id] + nb27(o, g, x, id)) / (o.c[OC][id] + cc[id]);
      }
      if (CLUSTER > 1) cg::this_cluster().sync();
      else __syncthreads();
    }
  }
}

// one colour over the whole grid (large levels)
__global__ void k_gs27_mc_colour(Grid g, OpF o, const float* __restrict__ cc,
                                 const float* __restrict__ fc, float* x, int c) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int hx = (nx - 1) / 2, hy = (ny - 1) / 2, hz = (nz - 1) / 2;
  const int pi = c & 1, pj = (c >> 1) & 1, pk = (c >> 2) & 1;
  const size_t tot = (size_t)hx * hy * hz;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot;
       t += (size_t)gridDim.x * blockDim.x) {
    const int mi = (int)(t % hx), mj = (int)((t / hx) % hy), mk = (int)(t / ((size_t)hx * hy));
    const int i = (pi ? 1 : 2) + 2 * mi;
    const int j = (pj ? 1 : 2) + 2 * mj;
    const int k = (pk ? 1 : 2) + 2 * mk;
    if (i > nx - 2 || j > ny - 2 || k > nz - 2) continue;
    const size_t id = g.idx(i, j, k);
    x[id] = (fc[id] + nb27(o, g, x, id)) / (o.c[OC][id] + cc[id]);
  }
}

// all colours of nsweep sweeps on a large level in one cooperative launch,
// a grid-wide barrier between colours (the updates of k_gs27_mc_colour)
__global__ void __launch_bounds__(256) k_gs27_mc_coop(Grid g, OpF o, const float* __restrict__ cc,
                                                     const float* __restrict__ fc, float* x,
                                                     int nsweep, int reverse) {
  cg::grid_group grid = cg::this_grid();
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int hx = (nx - 1) / 2, hy = (ny - 1) / 2, hz = (nz - 1) / 2;
  const size_t tot = (size_t)hx * hy * hz;
  const size_t gtid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t nthr = (size_t)gridDim.x * blockDim.x;
  for (int sw = 0; sw < nsweep; sw++)
    for (int c8 = 0; c8 < 8; c8++) {
      const int c = reverse ? 7 - c8 : c8;
      const int pi = c & 1, pj = (c >> 1) & 1, pk = (c >> 2) & 1;
      for (size_t t = gtid; t < tot; t += nthr) {
        const int mi = (int)(t % hx), mj = (int)((t / hx) % hy), mk = (int)(t / ((size_t)hx * hy));
        const int i = (pi ? 1 : 2) + 2 * mi;
        const int j = (pj ? 1 : 2) + 2 * mj;
        const int k = (pk ? 1 : 2) + 2 * mk;
        if (i > nx - 2 || j > ny - 2 || k > nz - 2) continue;
        const size_t id = g.idx(i, j, k);
        x[id] = (fc[id] + nb27(o, g, x, id)) / (o.c[OC][id] + cc[id]);
      }
      grid.sync();
    }
}

// The restriction of xin to level C's right-hand side w0 (0 on the boundary).  With
// x2 given also the first Chebyshev step from x = 0, r = w0 / a_ii, d = x2 = r / theta
// (k_cheb_step over zeros, without the pass over the couplings); without, x (if given)
// is set to 0.
__global__ void k_restrict_f32(Grid gf, const float* __restrict__ xin, Grid gc, float* w0,
                               const float* __restrict__ oc, const float* __restrict__ cc,
                               const float* __restrict__ lam, float* x, float* x2, float* d) {
  const int cx = gc.nx, cy = gc.ny, cz = gc.nz;
  const size_t n = gc.n();
  float alpha, beta = 0.f;
  if (x2) cheb_coef(*lam, 0, alpha, beta);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    split3(q, cx, cy, i, j, k);
    if (!x2 && x) x[q] = 0.f;
    if (i == 0 || j == 0 || k == 0 || i == cx - 1 || j == cy - 1 || k == cz - 1) {
      w0[q] = 0.f;
      continue;
    }
    const int ii = 2 * i, jj = 2 * j, kk = 2 * k;
    float acc = 0.f;
#pragma unroll
    for (int dz = -1; dz <= 1; dz++)
#pragma unroll
      for (int dy = -1; dy <= 1; dy++)
#pragma unroll
        for (int dx = -1; dx <= 1; dx++) {
          const float w = 1.f / (float)(1 << (abs(dx) + abs(dy) + abs(dz)));
          acc += w * xin[gf.idx(ii + dx, jj + dy, kk + dz)];
        }
    w0[q] = acc;
    if (x2) {
      const float dn = beta * (acc / (oc[q] + cc[q]));
      d[q] = dn;
      x2[q] = dn;
    }
  }
}

// One thread per coarse cell (ii..ii+1, jj..jj+1, kk..kk+1): its eight corner
// values, read once, give the interpolated correction of the up to eight fine
// interior points 2ii+oi, 2jj+oj, 2kk+ok of the cell, each summed over the
// corners it uses in the order of the per-point loop (c, then b, then a, from
// 0), so the result is the per-point kernel's bit for bit with an eighth of
// its loads and index arithmetic.
__global__ void k_interp_axpy_f32(Grid gc, const float* __restrict__ xc, Grid gf, float* xf,
                                  const double* num, const double* den) {
  const float xdamp = (float)(num[0] / den[0]);
  const int cx = gc.nx - 1, cy = gc.ny - 1, cz = gc.nz - 1;
  const size_t ncell = (size_t)cx * cy * cz;
  const size_t sy = gc.nx, sz = (size_t)gc.nx * gc.ny;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < ncell;
       q += (size_t)gridDim.x * blockDim.x) {
    int ii, jj, kk;
    split3(q, cx, cy, ii, jj, kk);
    const size_t c0 = gc.idx(ii, jj, kk);
    const float x000 = xc[c0], x100 = xc[c0 + 1], x010 = xc[c0 + sy], x110 = xc[c0 + sy + 1];
    const float x001 = xc[c0 + sz], x101 = xc[c0 + sz + 1], x011 = xc[c0 + sz + sy];
    const float x111 = xc[c0 + sz + sy + 1];
#pragma unroll
    for (int ok = 0; ok < 2; ok++) {
      const int k = 2 * kk + ok;
      if (k < 1 || k > gf.nz - 2) continue;
#pragma unroll
      for (int oj = 0; oj < 2; oj++) {
        const int j = 2 * jj + oj;
        if (j < 1 || j > gf.ny - 2) continue;
#pragma unroll
        for (int oi = 0; oi < 2; oi++) {
          const int i = 2 * ii + oi;
          if (i < 1 || i > gf.nx - 2) continue;
          float w = 0.f;
          w += x000;
          if (oi) w += x100;
          if (oj) {
            w += x010;
            if (oi) w += x110;
          }
          if (ok) {
            w += x001;
            if (oi) w += x101;
            if (oj) {
              w += x011;
              if (oi) w += x111;
            }
          }
          w *= 1.f / (float)(1 << (oi + oj + ok));
          xf[gf.idx(i, j, k)] += xdamp * w;
        }
      }
    }
  }
}

// dot product of FP32 vectors on interior points, FP64 accumulation
__global__ void k_sum_parts(const double* __restrict__ part, int n, double* out) {
  __shared__ double sh[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
  const double t = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) out[0] = t;
}

// The two sums of the interpolation damping on a coarse level, x.w0 and
// x.((A + cc) x), in one pass over x: FP32 products (A + cc) x, FP64 sums,
// partials per block (at most 1184 blocks) summed by the block that finishes
// last (a ticket on *done, which it resets).
__global__ void k_damp_dots(Grid g, OpF o, const float* __restrict__ cc,
                            const float* __restrict__ x, const float* __restrict__ w0,
                            double* part_num, double* part_den, unsigned* done, double* num,
                            double* den) {
  __shared__ double sh[32];
  __shared__ bool last;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const size_t nint = (size_t)(nx - 2) * (ny - 2) * (nz - 2);
  double an = 0.0, ad = 0.0;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, nx, ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    const float nb = (o.nop == 4) ? nb7(o, g, x, id) : nb27(o, g, x, id);
    const float xv = x[id];
    const float ax = (o.c[OC][id] + cc[id]) * xv - nb;
    an += (double)xv * (double)w0[id];
    ad += (double)xv * (double)ax;
  }
  const double tn = block_sum<256>(an, sh);
  const double td = block_sum<256>(ad, sh);
  if (threadIdx.x == 0) {
    part_num[blockIdx.x] = tn;
    part_den[blockIdx.x] = td;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (!last) return;
  // the block that finishes last adds the partials in block order, as
  // the separate two-block sum did: the same sums whichever block that is
  __threadfence();
  double bn = 0.0, bd = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    bn += __ldcg(part_num + i);
    bd += __ldcg(part_den + i);
  }
  const double sn = block_sum<256>(bn, sh);
  const double sd = block_sum<256>(bd, sh);
  if (threadIdx.x == 0) {
    num[0] = sn;
    den[0] = sd;
    *done = 0u;
  }
}

void damp_dots(cudaStream_t s, Grid g, OpF o, const float* cc, const float* x, const float* w0,
               double* part, unsigned* done, double* num, double* den) {
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  // a point per thread while the partials' room lasts: with four, levels of 33^3 and
  // below had a block on fewer than half of the SMs (levels of 65^3 and 33^3 on
  // average 15.9 -> 9.5 us)
  const int nb = (int)std::min<size_t>((nint + 255) / 256, 1184);
  k_damp_dots<<<nb, 256, 0, s>>>(g, o, cc, x, w0, part, part + 2368, done, num, den);
}

// FP64 fine residual r = f - (A + cc) x written as the FP32 V-cycle rhs,
// with its FP64 1-norm (partials per block)
__global__ void k_resid64_to32(Grid g, Op op, const double* __restrict__ cc,
                               const double* __restrict__ fc, const double* __restrict__ x,
                               float* r32, double* part) {
  __shared__ double sh[32];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const size_t nint = (size_t)(nx - 2) * (ny - 2) * (nz - 2);
  const size_t sy = nx, sz = (size_t)nx * ny;
  double acc = 0.0;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, nx, ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    const double r = fc[id] + op.c[ON][id] * x[id + sy] + op.c[ON][id - sy] * x[id - sy] +
                     op.c[OE][id] * x[id + 1] + op.c[OE][id - 1] * x[id - 1] +
                     op.c[UC][id - sz] * x[id - sz] + op.c[UC][id] * x[id + sz] -
                     (op.c[OC][id] + cc[id]) * x[id];
    r32[id] = (float)r;
    acc += fabs(r);
  }
  const double t = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// x += e on interior points (FP64 accumulation of the FP32 correction)
__global__ void k_add_corr(Grid g, const float* __restrict__ e, double* x) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const size_t nint = (size_t)(nx - 2) * (ny - 2) * (nz - 2);
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nint;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_ijk(q, nx, ny, i, j, k);
    const size_t id = g.idx(i, j, k);
    x[id] += (double)e[id];
  }
}

// ---------------------------------------------------------------------------
// coarsest level: dense FP64 Cholesky of (A_c + diag cc) over interior points
// ---------------------------------------------------------------------------
__global__ void k_dense_build(Grid g, Op op, const double* __restrict__ cc, double* M, int n) {
  const int nx = g.nx, ny = g.ny;
  const int ex = nx - 2, ey = ny - 2;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * n; t += gridDim.x * blockDim.x) {
    const int r = t / n, c = t % n;
    const int ri = 1 + r % ex, rj = 1 + (r / ex) % ey, rk = 1 + r / (ex * ey);
    const int ci = 1 + c % ex, cj = 1 + (c / ex) % ey, ck = 1 + c / (ex * ey);
    const int dx = ci - ri, dy = cj - rj, dz = ck - rk;
    double v = 0.0;
    if (abs(dx) <= 1 && abs(dy) <= 1 && abs(dz) <= 1) {
      if (dx == 0 && dy == 0 && dz == 0) {
        v = op.c[OC][g.idx(ri, rj, rk)] + cc[g.idx(ri, rj, rk)];
      } else {
        int si = ri, sj = rj, sk = rk, ax = dx, ay = dy, az = dz;
        if (az < 0 || (az == 0 && ay < 0) || (az == 0 && ay == 0 && ax < 0)) {
          si = ci; sj = cj; sk = ck; ax = -ax; ay = -ay; az = -az;
        }
        int code;
        if (az == 0) code = (ay == 0) ? OE : (ax == 0) ? ON : (ax > 0 ? ONE : ONW);
        else if (ax == 0 && ay == 0) code = UC;
        else if (ay == 0) code = (ax > 0) ? UE : UW;
        else if (ax == 0) code = (ay > 0) ? UN : US;
        else if (ay > 0) code = (ax > 0) ? UNE : UNW;
        else code = (ax > 0) ? USE : USW;
        v = (code < op.nop) ? -op.c[code][g.idx(si, sj, sk)] : 0.0;
      }
    }
    M[t] = v;
  }
}

// Inverse of the SPD coarsest matrix by Gauss-Jordan elimination (no
// pivoting needed for SPD) in one cluster of CL CTAs (CL = 1: one CTA).  CTA
// `rank` keeps rows rank*rows_per .. +rows_per of M in shared memory; thread
// (g, c) updates column c of the CTA's rows g, g+G, ... (G = blockDim / n row
// groups).  The pivot row p is read from a double-buffered slot every CTA
// holds: during step p the owner of row p+1 updates that row and stores the
// result into every CTA's other slot, so one cluster barrier per pivot
// suffices.  Each element sees the same operations as in a one-CTA
// Gauss-Jordan sweep: A[r][c] -= A[r][p] A[p][c] / piv off row and column p,
// column p becomes -A[r][p] / piv, row p A[p][c] / piv, the pivot 1/piv.
// M is replaced by its inverse; info = first non-positive pivot + 1, else 0.
template <int CL>
__global__ void __launch_bounds__(1024) k_dense_inverse(double* M, int n, int rows_per,
                                                        int* info) {
  extern __shared__ double sm[];
  double* A = sm;                          // [rows_per][n]
  double* pb = A + (size_t)rows_per * n;   // [2][n] pivot rows
  double* colp = pb + 2 * (size_t)n;       // [rows_per] column p before the step
  const int rank = (CL > 1) ? (int)cg::this_cluster().block_rank() : 0;
  auto csync = [&]() {
    if (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  const int r0 = rank * rows_per;
  const int nr = max(0, min(rows_per, n - r0));
  const int G = max(1, (int)blockDim.x / n);
  const int c = threadIdx.x % n, grp = threadIdx.x / n;
  const bool active = grp < G && (int)threadIdx.x < G * n;
  for (int t = threadIdx.x; t < nr * n; t += blockDim.x) A[t] = M[(size_t)r0 * n + t];
  csync();  // every CTA runs and holds its rows before any slot is written
  if (r0 == 0 && nr > 0)  // the owner of row 0 publishes it
    for (int t = threadIdx.x; t < n; t += blockDim.x)
      for (int q = 0; q < CL; q++) {
        double* dst = (CL > 1) ? cg::this_cluster().map_shared_rank(pb, q) : pb;
        dst[t] = A[t];
      }
  csync();
  int bad = 0;
  for (int p = 0; p < n; p++) {
    const double* rowp = pb + (size_t)(p & 1) * n;
    const double piv = rowp[p];
    if (!(piv > 0.0)) {  // every thread of every CTA reads the same value
      bad = p + 1;
      break;
    }
    const double ipiv = 1.0 / piv;
    for (int r = threadIdx.x; r < nr; r += blockDim.x) colp[r] = A[(size_t)r * n + p];
    __syncthreads();
    if (active) {
      const double rc = rowp[c];
      double* nextslot = pb + (size_t)((p + 1) & 1) * n;
      for (int r = grp; r < nr; r += G) {
        const int gr = r0 + r;
        double v;
        if (gr == p) v = (c == p) ? ipiv : rc * ipiv;
        else if (c == p) v = -colp[r] * ipiv;
        else v = A[(size_t)r * n + c] - colp[r] * rc * ipiv;
        A[(size_t)r * n + c] = v;
        if (gr == p + 1)
          for (int q = 0; q < CL; q++) {
            double* dst = (CL > 1) ? cg::this_cluster().map_shared_rank(nextslot, q) : nextslot;
            dst[c] = v;
          }
      }
    }
    csync();  // row p+1 is published and column p read everywhere
  }
  for (int t = threadIdx.x; t < nr * n; t += blockDim.x) M[(size_t)r0 * n + t] = A[t];
  if (rank == 0 && threadIdx.x == 0) info[0] = bad;
  if (CL > 1) cg::this_cluster().sync();  // no CTA exits while a slot write may target it
}

// x = M^{-1} b on the coarsest level (FP32 in/out, FP64 product).
__global__ void k_dense_apply(Grid g, const double* __restrict__ Minv, int n,
                              const float* __restrict__ rhs, float* x) {
  extern __shared__ double b[];
  const int nx = g.nx, ny = g.ny;
  const int ex = nx - 2, ey = ny - 2;
  for (int q = threadIdx.x; q < n; q += blockDim.x)
    b[q] = (double)rhs[g.idx(1 + q % ex, 1 + (q / ex) % ey, 1 + q / (ex * ey))];
  for (size_t q = threadIdx.x; q < g.n(); q += blockDim.x) x[q] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int r = wid; r < n; r += nw) {
    double t = 0.0;
    for (int c = lane; c < n; c += 32) t += Minv[(size_t)r * n + c] * b[c];
    t = warp_sum(t);
    if (lane == 0) x[g.idx(1 + r % ex, 1 + (r / ex) % ey, 1 + r / (ex * ey))] = (float)t;
  }
}

// ---------------------------------------------------------------------------
// Coarse-level tail of the FP32 V-cycle in one cluster kernel: from level
// `first` (restricting the residual of level first-1) down to the coarsest
// level, the dense coarsest solve, and back up to level `first` (8-colour
// smoothing, operator-weighted interpolation with the Hackbusch-Reusken
// damping of Vmvcs, src/pmgc/mgcsd.c:450-500).  A cluster barrier separates
// dependent steps; sums use distributed shared memory in rank order, so all
// CTAs agree on every damping factor.  It ends by writing the damping sums
// of the first -> first-1 correction for the caller.
// ---------------------------------------------------------------------------

struct TailArgs {
  const TLev* lev;      // device array indexed by level
  int first, last;      // tail levels; last is the coarsest
  Grid gprev;           // grid of level first-1
  const float* rprev;   // residual of level first-1
  float* r;             // residual scratch (>= level first size)
  const double* minv;   // dense inverse on the coarsest level
  int nd;
  double* xnum;         // damping sums of the first -> first-1 correction
  double* xden;
  int nsweep;           // 8-colour sweeps before and after each coarse correction
  int cheb = 0;         // > 0: Chebyshev smoothing of this (even) degree instead
};

__device__ __forceinline__ float nb27t(const TLev& L, const float* x, size_t id) {
  OpF o;
#pragma unroll
  for (int c = 0; c < 14; c++) o.c[c] = L.op[c];
  o.nop = 14;
  return nb27(o, L.g, x, id);
}

// q / d for 0 <= q < 2^31 (T. Granlund, P. Montgomery, PLDI 1994): with l =
// ceil(log2 d) and m = ceil(2^(31 + l) / d) < 2^32, q m / 2^(31 + l) exceeds q / d by
// less than 1 / d, as q (m d - 2^(31 + l)) < 2^31 2^l (tests/test_long_axes.py).
inline Quot div_const(int d) {
  int l = 0;
  while ((1ll << l) < d) l++;
  if (l == 0) return Quot{0u, 0u};
  return Quot{(unsigned)(((1ull << (31 + l)) + d - 1) / d), (unsigned)(l - 1)};
}
__device__ __forceinline__ int quotient(int q, Quot c) {
  return c.m ? (int)(__umulhi((unsigned)q, c.m) >> c.shift) : q;
}
// Interior point q of a level as a flat index.
__device__ __forceinline__ int interior_at(Grid g, Quot dx, Quot dy, int q) {
  const int ex = g.nx - 2, ey = g.ny - 2;
  const int t = quotient(q, dx), k = quotient(t, dy);
  return ((k + 1) * g.ny + t - k * ey + 1) * g.nx + q - t * ex + 1;
}

// A thread's number among those of the cluster, in two orders: CTA by CTA, and
// warp by warp round the CTAs.  A level with fewer points than threads goes by
// the second, which spreads it over all the cluster's SMs (17^3: 16 instead of 7;
// a pass is bounded by what one SM's load pipe takes in).
struct TailTid {
  int block, round, n;
  __device__ __forceinline__ int first(int points) const { return points < n ? round : block; }
};
template <int CLUSTER>
__device__ __forceinline__ TailTid tail_tid() {
  TailTid t;
  const int rank = CLUSTER > 1 ? (int)cg::this_cluster().block_rank() : 0;
  t.block = rank * blockDim.x + threadIdx.x;
  t.round = (int)(((threadIdx.x >> 5) * CLUSTER + rank) * 32 + (threadIdx.x & 31));
  t.n = CLUSTER * blockDim.x;
  return t;
}

// The thread's points below n, U at a time: value(id) of all of them (id the flat
// index at(q), or -1: none), then the stores.  The loads of U points
// are in flight together; a thread's next point would otherwise wait for the
// stores of the one before, which the compiler must take for its inputs.
template <int U, class At, class Value, class Store>
__device__ __forceinline__ void for_points(int n, TailTid tid, At at, Value value, Store store) {
  const int nthr = tid.n;
  for (int q0 = tid.first(n); q0 < n; q0 += U * nthr) {
    int id[U];
    decltype(value(0)) v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int q = q0 + u * nthr;
      id[u] = q < n ? at(q) : -1;
      if (id[u] >= 0) v[u] = value(id[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (id[u] >= 0) store(id[u], v[u]);
  }
}

template <int CLUSTER>
__device__ __forceinline__ void tail_sync() {
  if (CLUSTER > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// Sum of two values over the cluster, the same result in every thread.  Each CTA
// stores its partial sums into every CTA's slots ahead of the barrier, so after it
// they are read locally, in rank order.  slots: [2 phases][CLUSTER][2].  A CTA may
// store into another's shared memory only once that one is known to run: every
// kernel passes a tail_sync before its first sum (tests/test_cluster_first_push.py).
template <int CLUSTER>
__device__ void tail_sum2(double& a, double& b, double* sh, double* slots, int& phase) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sh[2 * wid] = a;
    sh[2 * wid + 1] = b;
  }
  __syncthreads();
  double* mine = slots + 2 * CLUSTER * phase;
  if (threadIdx.x < CLUSTER) {
    double sa = 0.0, sb = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      sa += sh[2 * w];
      sb += sh[2 * w + 1];
    }
    if (CLUSTER > 1) {
      cg::cluster_group cl = cg::this_cluster();
      const int rank = (int)cl.block_rank();
      double* to = cl.map_shared_rank(mine, (int)threadIdx.x) + 2 * rank;
      to[0] = sa;
      to[1] = sb;
    } else {
      mine[0] = sa;
      mine[1] = sb;
    }
  }
  tail_sync<CLUSTER>();
  double ta = 0.0, tb = 0.0;
#pragma unroll
  for (int rk = 0; rk < CLUSTER; rk++) {
    ta += mine[2 * rk];
    tb += mine[2 * rk + 1];
  }
  a = ta;
  b = tb;
  phase ^= 1;
}

template <int CLUSTER>
__device__ void tail_smooth(const TLev& L, int reverse, TailTid tid, int nsweep) {
  const Grid g = L.g;
  const int hx = (g.nx - 1) / 2, hy = (g.ny - 1) / 2, hz = (g.nz - 1) / 2;
  const int tot = hx * hy * hz;
  for (int sw = 0; sw < nsweep; sw++)
    for (int c8 = 0; c8 < 8; c8++) {
      const int c = reverse ? 7 - c8 : c8;
      const int pi = c & 1, pj = (c >> 1) & 1, pk = (c >> 2) & 1;
      for (int t = tid.first(tot); t < tot; t += tid.n) {
        const int mi = t % hx, mj = (t / hx) % hy, mk = t / (hx * hy);
        const int i = (pi ? 1 : 2) + 2 * mi, j = (pj ? 1 : 2) + 2 * mj, k = (pk ? 1 : 2) + 2 * mk;
        if (i > g.nx - 2 || j > g.ny - 2 || k > g.nz - 2) continue;
        const size_t id = g.idx(i, j, k);
        L.x[id] = (L.w0[id] + nb27t(L, L.x, id)) / (L.op[OC][id] + L.cc[id]);
      }
      tail_sync<CLUSTER>();
    }
}

// Chebyshev steps first .. K-1 on level L inside the cluster (K even: the result
// ends in L.x)
template <int CLUSTER>
__device__ void tail_cheb(const TLev& L, TailTid tid, int K, int first) {
  const Grid g = L.g;
  const Quot dx = L.dx, dy = L.dy;
  OpF o;
#pragma unroll
  for (int c = 0; c < 14; c++) o.c[c] = L.op[c];
  o.nop = 14;
  const int nint = (g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  const float b = *L.lam;
  const float *cc = L.cc, *f = L.w0;
  float* d = L.d;
  for (int i = first; i < K; i++) {
    float alpha, beta;
    cheb_coef(b, i, alpha, beta);
    const float* xin = (i & 1) ? L.x2 : L.x;
    float* xout = (i & 1) ? L.x : L.x2;
    for_points<2>(
        nint, tid, [&](int q) { return interior_at(g, dx, dy, q); },
        [&](int id) {
          const float dg = o.c[OC][id] + cc[id];
          const float xv = xin[id];
          const float r = (f[id] + nb27(o, g, xin, id) - dg * xv) / dg;
          const float dn = alpha * d[id] + beta * r;
          return make_float2(dn, xv + dn);
        },
        [&](int id, float2 v) {
          d[id] = v.x;
          xout[id] = v.y;
        });
    tail_sync<CLUSTER>();
  }
}

// Restriction src (grid gs) -> level L's w0 (all points, boundary 0).  cheb0: also
// the first Chebyshev step from x = 0, which needs no neighbour -- r = f / a_ii,
// d = x2 = r / theta (the step the loop of tail_cheb would take over zeros);
// otherwise x = 0.
__device__ void tail_restrict(Grid gs, const float* src, const TLev& L, bool cheb0,
                              TailTid tid) {
  const Grid gc = L.g;
  const int n = (int)gc.n();
  const float *oc = L.op[OC], *cc = L.cc;
  float *w0 = L.w0, *x = L.x, *x2 = L.x2, *d = L.d;
  float alpha, beta = 0.f;
  if (cheb0) cheb_coef(*L.lam, 0, alpha, beta);
  for (int q = tid.first(n); q < n; q += tid.n) {
    const int i = q % gc.nx, j = (q / gc.nx) % gc.ny, k = q / (gc.nx * gc.ny);
    if (!cheb0) x[q] = 0.f;
    if (i == 0 || j == 0 || k == 0 || i == gc.nx - 1 || j == gc.ny - 1 || k == gc.nz - 1) {
      w0[q] = 0.f;
      continue;
    }
    const int ii = 2 * i, jj = 2 * j, kk = 2 * k;
    float acc = 0.f;
#pragma unroll
    for (int dz = -1; dz <= 1; dz++)
#pragma unroll
      for (int dy = -1; dy <= 1; dy++)
#pragma unroll
        for (int dx = -1; dx <= 1; dx++) {
          const float w = 1.f / (float)(1 << (abs(dx) + abs(dy) + abs(dz)));
          acc += w * src[gs.idx(ii + dx, jj + dy, kk + dz)];
        }
    w0[q] = acc;
    if (cheb0) {
      const float dn = beta * (acc / (oc[q] + cc[q]));
      d[q] = dn;
      x2[q] = dn;
    }
  }
}

// damping sums <x, w0> and <x, (A + cc) x> on level L
template <int CLUSTER>
__device__ void tail_damp(const TLev& L, TailTid tid, double* sh, double* slots,
                          int& phase, double& num, double& den) {
  const Grid g = L.g;
  const Quot dx = L.dx, dy = L.dy;
  OpF o;
#pragma unroll
  for (int c = 0; c < 14; c++) o.c[c] = L.op[c];
  o.nop = 14;
  const int nint = (g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  const float *cc = L.cc, *x = L.x, *w0 = L.w0;
  double a = 0.0, b = 0.0;
  for_points<2>(
      nint, tid, [&](int q) { return interior_at(g, dx, dy, q); },
      [&](int id) {
        const float xv = x[id];
        return make_float2(w0[id], (o.c[OC][id] + cc[id]) * xv - nb27(o, g, x, id));
      },
      [&](int id, float2 v) {
        const float xv = x[id];
        a += (double)xv * (double)v.x;
        b += (double)xv * (double)v.y;
      });
  tail_sum2<CLUSTER>(a, b, sh, slots, phase);
  num = a;
  den = b;
}

// xf += xdamp * (trilinear interpolation of xc) on the interior of gf
__device__ void tail_interp(Grid gc, const float* xc, Grid gf, Quot dx, Quot dy, float* xf,
                            float xdamp, TailTid tid) {
  const int ex = gf.nx - 2, ey = gf.ny - 2, nint = ex * ey * (gf.nz - 2);
  struct Corrected {
    int id;
    float x;
  };
  for_points<2>(
      nint, tid, [](int q) { return q; },
      [&](int q) {
        const int t = quotient(q, dx), k = quotient(t, dy) + 1;
        const int i = q - t * ex + 1, j = t - (k - 1) * ey + 1;
        const int ii = i >> 1, jj = j >> 1, kk = k >> 1;
        const int oi = i & 1, oj = j & 1, ok = k & 1;
        float w = 0.f;
        for (int c = 0; c <= ok; c++)
          for (int b = 0; b <= oj; b++)
            for (int a = 0; a <= oi; a++) w += xc[gc.idx(ii + a, jj + b, kk + c)];
        w *= 1.f / (float)(1 << (oi + oj + ok));
        const int id = (k * gf.ny + j) * gf.nx + i;
        return Corrected{id, xf[id] + xdamp * w};
      },
      [&](int, Corrected v) { xf[v.id] = v.x; });
}

// The level table in shared memory (kTailLevels at most): the pointers of a pass
// are then one shared load away, not one through an L1 that the barrier cleared.
constexpr int kTailLevels = 16;
__device__ __forceinline__ void tail_levels(TailArgs& A, TLev* sh) {
  static_assert(sizeof(TLev) % 4 == 0 && sizeof(TailArgs) % 4 == 0, "copied by words");
  const int words = (int)sizeof(TLev) / 4 * (A.last + 1);
  for (int t = threadIdx.x; t < words; t += blockDim.x)
    reinterpret_cast<unsigned*>(sh)[t] = reinterpret_cast<const unsigned*>(A.lev)[t];
  A.lev = sh;
  __syncthreads();
}

// One V-cycle from level A.first down to the dense level and back.  With
// rhs_given the right-hand side of level first is already in its w0;
// otherwise it is restricted from the residual of level first-1.
template <int CLUSTER>
__device__ void tail_cycle(const TailArgs& A, bool rhs_given, TailTid tid, double* sh,
                           double* slots, int& phase) {
  // down
  for (int l = A.first; l <= A.last; l++) {
    const TLev& L = A.lev[l];
    const bool cheb0 = A.cheb > 0 && l != A.last && !(l == A.first && rhs_given);
    if (l == A.first && rhs_given) {
      const int n = (int)L.g.n();
      for (int q = tid.first(n); q < n; q += tid.n) L.x[q] = 0.f;
    } else if (l == A.first) {
      tail_restrict(A.gprev, A.rprev, L, cheb0, tid);
    } else {
      tail_restrict(A.lev[l - 1].g, A.r, L, cheb0, tid);
    }
    tail_sync<CLUSTER>();
    if (l != A.last) {
      if (A.cheb > 0) tail_cheb<CLUSTER>(L, tid, A.cheb, cheb0 ? 1 : 0);
      else tail_smooth<CLUSTER>(L, 0, tid, A.nsweep);
      const Grid g = L.g;
      const Quot dx = L.dx, dy = L.dy;
      const int nint = (g.nx - 2) * (g.ny - 2) * (g.nz - 2);
      OpF o;
#pragma unroll
      for (int c = 0; c < 14; c++) o.c[c] = L.op[c];
      o.nop = 14;
      const float *cc = L.cc, *x = L.x, *w0 = L.w0;
      float* r = A.r;
      for_points<2>(
          nint, tid, [&](int q) { return interior_at(g, dx, dy, q); },
          [&](int id) { return w0[id] + nb27(o, g, x, id) - (o.c[OC][id] + cc[id]) * x[id]; },
          [&](int id, float v) { r[id] = v; });
      tail_sync<CLUSTER>();
    }
  }
  // coarsest: x = Minv * w0 (one warp per row)
  {
    const TLev& L = A.lev[A.last];
    const Grid g = L.g;
    const int ex = g.nx - 2, ey = g.ny - 2;
    const int lane = threadIdx.x & 31;
    const int gw = tid.round >> 5, nw = tid.n >> 5;
    for (int row = gw; row < A.nd; row += nw) {
      double t = 0.0;
      for (int c = lane; c < A.nd; c += 32)
        t += A.minv[(size_t)row * A.nd + c] *
             (double)L.w0[g.idx(1 + c % ex, 1 + (c / ex) % ey, 1 + c / (ex * ey))];
      t = warp_sum(t);
      if (lane == 0) L.x[g.idx(1 + row % ex, 1 + (row / ex) % ey, 1 + row / (ex * ey))] = (float)t;
    }
    tail_sync<CLUSTER>();
  }
  // up
  for (int l = A.last - 1; l >= A.first; l--) {
    const TLev& C = A.lev[l + 1];
    const TLev& P = A.lev[l];
    double num, den;
    tail_damp<CLUSTER>(C, tid, sh, slots, phase, num, den);
    const float xdamp = (float)(num / den);
    tail_interp(C.g, C.x, P.g, P.dx, P.dy, P.x, xdamp, tid);
    tail_sync<CLUSTER>();
    if (A.cheb > 0) tail_cheb<CLUSTER>(P, tid, A.cheb, 0);
    else tail_smooth<CLUSTER>(P, 1, tid, A.nsweep);
  }
}

// The tail of one V-cycle.  Latency bounds it: a pass is a barrier (0.5 to 1.8 us
// with the memory it orders) and a chain of L2 reads, on levels of a few thousand
// points that give each thread one or none.  So a step's barriers were merged (the
// first Chebyshev step goes with the restriction, the damping sums are pushed to
// every CTA), the level table sits in shared memory, the loads of two points are in
// flight together and small levels are spread over all the SMs: 33^3 grid (levels
// 17^3 to 5^3) 58 -> 39 us, 49^3 77 -> 53, 225^3 91 -> 62, bitwise the same cycle.
template <int CLUSTER>
__global__ void __launch_bounds__(512) k_vcycle_tail(TailArgs A) {
  __shared__ double sh[64];
  __shared__ double slots[4 * CLUSTER];
  __shared__ TLev levels[kTailLevels];
  tail_levels(A, levels);
  const TailTid tid = tail_tid<CLUSTER>();
  int phase = 0;
  tail_cycle<CLUSTER>(A, false, tid, sh, slots, phase);
  // damping sums for the first -> first-1 correction (done by the caller)
  double num, den;
  tail_damp<CLUSTER>(A.lev[A.first], tid, sh, slots, phase, num, den);
  if (tid.block == 0) {
    A.xnum[0] = num;
    A.xden[0] = den;
  }
  // no CTA may exit while another can still read its shared memory
  tail_sync<CLUSTER>();
}

// The reference's coarsest band matrix (Vbuildband1_27,
// src/pmgc/buildBd.c:183-306) written back as a symmetric 27-point operator
// B: diagonal oC without the Helmholtz term, and each of the 13 couplings a
// band column q = (i,j,k) stores with the row q + off becomes the coupling
// of (i,j,k) with its geometric neighbour at that offset.  Several of those
// values come from the coefficient of a different pair (the band's
// diagonal couplings), so B is not A_c; it is what the reference factors and
// solves.  A nonzero value whose band row is not the geometric neighbour (an
// offset that wraps across the grid edge) cannot be expressed this way and
// raises *wrap.
struct OpW {
  double* c[14];
};

__global__ void k_band_restencil(Grid g, Op a, OpW b, int* wrap) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int ex = nx - 2, exy = (nx - 2) * (ny - 2);
  const int nint = exy * (nz - 2);
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nint; q += gridDim.x * blockDim.x) {
    const int i = 1 + q % ex, j = 1 + (q / ex) % (ny - 2), k = 1 + q / exy;
    const double* const* c = a.c;
    b.c[OC][g.idx(i, j, k)] = c[OC][g.idx(i, j, k)];
    // (band offset, value, geometric displacement, target array, target point)
    auto put = [&](int off, double v, int di, int dj, int dk, int arr, int ti, int tj, int tk) {
      const int pi = i + di, pj = j + dj, pk = k + dk;
      if (pi >= 1 && pi <= nx - 2 && pj >= 1 && pj <= ny - 2 && pk >= 1 && pk <= nz - 2) {
        b.c[arr][g.idx(ti, tj, tk)] = v;
      } else if (v != 0.0 && q + off >= 0) {
        atomicOr(wrap, 1);
      }
    };
    put(-1, c[OE][g.idx(i - 1, j, k)], -1, 0, 0, OE, i - 1, j, k);
    put(-ex, c[ON][g.idx(i, j - 1, k)], 0, -1, 0, ON, i, j - 1, k);
    put(-ex + 1, c[ONE][g.idx(i, j - 1, k)], 1, -1, 0, ONW, i + 1, j - 1, k);
    put(-ex - 1, c[ONW][g.idx(i, j - 1, k)], -1, -1, 0, ONE, i - 1, j - 1, k);
    put(-exy, c[UC][g.idx(i, j, k - 1)], 0, 0, -1, UC, i, j, k - 1);
    put(-exy + 1, c[UE][g.idx(i, j, k - 1)], 1, 0, -1, UW, i + 1, j, k - 1);
    put(-exy - 1, c[UW][g.idx(i, j, k - 1)], -1, 0, -1, UE, i - 1, j, k - 1);
    put(-exy + ex, c[UN][g.idx(i, j, k - 1)], 0, 1, -1, US, i, j + 1, k - 1);
    put(-exy - ex, c[US][g.idx(i, j, k - 1)], 0, -1, -1, UN, i, j - 1, k - 1);
    put(-exy + ex + 1, c[UNE][g.idx(i, j, k - 1)], 1, 1, -1, USW, i + 1, j + 1, k - 1);
    put(-exy + ex - 1, c[UNW][g.idx(i, j, k - 1)], -1, 1, -1, USE, i - 1, j + 1, k - 1);
    put(-exy - ex + 1, c[USE][g.idx(i, j, k - 1)], 1, -1, -1, UNW, i + 1, j - 1, k - 1);
    put(-exy - ex - 1, c[USW][g.idx(i, j, k - 1)], -1, -1, -1, UNE, i - 1, j - 1, k - 1);
  }
}

// ---------------------------------------------------------------------------
// Exact-to-round-off solve of the FP64 coarsest level (FP64 path, LPBE):
// B x = b, B the reference's band matrix as a 27-point operator
// (k_band_restencil), by FP64 iterative refinement, each correction one FP32
// V-cycle over Galerkin levels of B below (tail_cycle with the residual as
// its right-hand side), until ||b - B x||_2 <= rtol ||b||_2.  It stands in
// for the reference's banded Cholesky (Vdpbfa/Vdpbsl, src/pmgc/mlinpckd.c),
// whose factorisation and substitution are sequential in the number of
// unknowns; any solve of B exact to round-off gives the V-cycle the same
// coarse-grid correction.
// ---------------------------------------------------------------------------
struct ExactArgs {
  TailArgs T;        // FP32 hierarchy; T.first is the FP64 coarsest level
  Grid g;            // grid of the FP64 coarsest level
  const double* op[14];
  const double* cc;
  const double* b;
  double* x;
  double* r;         // FP64 residual scratch of the level's size
  int maxit;
  double rtol;
  int* iters;        // refinement steps taken
};

template <int CLUSTER>
__global__ void __launch_bounds__(512) k_coarse_exact(ExactArgs E) {
  __shared__ double sh[64];
  __shared__ double slots[4 * CLUSTER];
  __shared__ TLev levels[kTailLevels];
  tail_levels(E.T, levels);
  const TailTid tid = tail_tid<CLUSTER>();
  int phase = 0;
  const Grid g = E.g;
  const int ex = g.nx - 2, ey = g.ny - 2, nint = ex * ey * (g.nz - 2);
  const int n = (int)g.n();
  const TLev& L = E.T.lev[E.T.first];
  for (int q = tid.first(n); q < n; q += tid.n) E.x[q] = 0.0;
  tail_sync<CLUSTER>();
  double bn = 0.0;
  int it = 0;
  for (;; it++) {
    double rr = 0.0, unused = 0.0;
    for (int q = tid.first(nint); q < nint; q += tid.n) {
      const size_t id = g.idx(1 + q % ex, 1 + (q / ex) % ey, 1 + q / (ex * ey));
      const double v = E.b[id] + nb27g<double>(E.op, g, E.x, id) -
                       (E.op[OC][id] + E.cc[id]) * E.x[id];
      E.r[id] = v;
      rr += v * v;
    }
    tail_sum2<CLUSTER>(rr, unused, sh, slots, phase);  // every CTA sees the same sum
    const double rn = sqrt(rr);
    if (it == 0) bn = rn;
    if (bn == 0.0 || rn <= E.rtol * bn || it >= E.maxit) break;
    for (int q = tid.first(n); q < n; q += tid.n) {
      const int i = q % g.nx, j = (q / g.nx) % g.ny, k = q / (g.nx * g.ny);
      const bool bd = (i == 0 || j == 0 || k == 0 || i == g.nx - 1 || j == g.ny - 1 ||
                       k == g.nz - 1);
      L.w0[q] = bd ? 0.f : (float)E.r[q];
    }
    tail_sync<CLUSTER>();
    tail_cycle<CLUSTER>(E.T, true, tid, sh, slots, phase);
    for (int q = tid.first(nint); q < nint; q += tid.n) {
      const size_t id = g.idx(1 + q % ex, 1 + (q / ex) % ey, 1 + q / (ex * ey));
      E.x[id] += (double)L.x[id];
    }
    tail_sync<CLUSTER>();
  }
  if (tid.block == 0) E.iters[0] = it;
  // no CTA may exit while another can still read its shared memory
  tail_sync<CLUSTER>();
}

// ---------------------------------------------------------------------------
// Batched solves: one persistent kernel for many mixed-precision LPBE
// calculations.  The descriptors of all calculations (their FP64 fine-level
// arrays and their FP32 level tables) are packed in one device array; each
// thread-block cluster takes one calculation and runs its whole refinement
// loop without returning to the host: the FP64 residual of Vmvcs's stopping
// test (src/pmgc/mgcsd.c:312-330, 1-norms), then per correction one FP32
// V-cycle -- 7-point red-black GS on the fine level, the one-cluster tail of
// levels 1 .. coarsest (tail_cycle), the Hackbusch-Reusken damping of the
// level-1 correction, interpolation and post-smoothing -- and the FP64
// accumulation.  It is the sequence of the per-launch mixed V-cycle graph, so
// calculations of uneven grid sizes share one launch and overlap on the SMs.
// ---------------------------------------------------------------------------
struct BatchItem {
  TailArgs T;             // FP32 levels 1 .. coarsest (T.first = 1)
  Grid g;                 // fine grid
  Quot dx, dy, dh;        // div_const of nx - 2, ny - 2 and the points of a colour in a row
  const double* op[4];    // FP64 fine operator: oC oE oN uC
  const double* cc;
  const double* fc;
  double* x;              // FP64 potential (interior; boundary zero)
  const float* op32[4];   // FP32 fine operator
  const float* cc32;
  float* w0;              // FP32 fine right-hand side (the FP64 residual)
  float* e;               // FP32 fine correction
  float* r;               // FP32 fine residual (T.rprev)
  double errtol;
  int itmax;
  int nlog;
  int fine_sweeps;        // red-black sweeps before and after the coarse correction
  double* out;            // [0] corrections, [1] final relative residual, [2..] log
};

// one colour of the FP32 fine-level red-black GS (the update of k_gs7_f32); from
// x = 0 (zero: the first colour of the first sweep) the neighbours are not read,
// and the other colour is set to 0
template <int CLUSTER>
__device__ void batch_gs7(const BatchItem& B, Quot dh, Quot dy, int parity, bool zero,
                          TailTid tid) {
  const Grid g = B.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int sy = nx, sz = nx * ny;
  const int hr = (nx - 1) / 2, ey = ny - 2;
  const int nslots = hr * ey * (nz - 2);
  const float *oC = B.op32[OC], *oN = B.op32[ON], *oE = B.op32[OE], *uC = B.op32[UC];
  const float *cc = B.cc32, *w0 = B.w0;
  float* x = B.e;
  for_points<4>(
      nslots, tid,
      [&](int q) {
        const int t = quotient(q, dh), k = quotient(t, dy) + 1;
        const int m = q - t * hr, j = t - (k - 1) * ey + 1;
        const int off = ((1 + j + k) & 1) != parity;
        const int i = 1 + off + 2 * m;
        if (zero) x[(k * ny + j) * nx + 2 - off + 2 * m] = 0.f;  // a boundary's 0 stays 0
        return i > nx - 2 ? -1 : (k * ny + j) * nx + i;
      },
      [&](int id) {
        float nb = 0.f;
        if (!zero)
          nb = oN[id] * x[id + sy] + oN[id - sy] * x[id - sy] + oE[id] * x[id + 1] +
               oE[id - 1] * x[id - 1] + uC[id - sz] * x[id - sz] + uC[id] * x[id + sz];
        return (w0[id] + nb) / (oC[id] + cc[id]);
      },
      [&](int id, float v) { x[id] = v; });
  tail_sync<CLUSTER>();
}

// Bounded by the L2's rate to the SMs of one cluster at 65^3 and by latency at 33^3.
// First colour from zero without reading the neighbours, points by multiplication
// instead of division, four points' loads in flight, and the tail above: a batch of
// five each of 33^3, 49^3 and 65^3 11.8 -> 10.6 ms, the same bits.
template <int CLUSTER>
__global__ void __launch_bounds__(512) k_batch_solve(const BatchItem* __restrict__ items) {
  __shared__ double sh[64];
  __shared__ double slots[4 * CLUSTER];
  __shared__ TLev levels[kTailLevels];
  __shared__ __align__(16) unsigned item[sizeof(BatchItem) / 4];
  for (int t = threadIdx.x; t < (int)sizeof(BatchItem) / 4; t += blockDim.x)
    item[t] = reinterpret_cast<const unsigned*>(items + blockIdx.x / CLUSTER)[t];
  __syncthreads();
  const BatchItem& B = *reinterpret_cast<const BatchItem*>(item);
  TailArgs T = B.T;
  tail_levels(T, levels);
  tail_sync<CLUSTER>();  // every CTA runs before the first sum stores into its slots
  const TailTid tid = tail_tid<CLUSTER>();
  int phase = 0;
  const Grid g = B.g;
  const int nx = g.nx, ny = g.ny;
  const int ex = nx - 2, ey = ny - 2, nint = ex * ey * (g.nz - 2);
  const int n = (int)g.n();
  const int sy = nx, sz = nx * ny;
  const Quot dx = B.dx, dy = B.dy;
  auto interior = [&](int q) { return interior_at(g, dx, dy, q); };

  // x = 0; ||f||_1 (Vxnrm1 on the interior)
  double fs = 0.0, u2 = 0.0;
  for (int q = tid.first(n); q < n; q += tid.n) B.x[q] = 0.0;
  for (int q = tid.first(nint); q < nint; q += tid.n) fs += fabs(B.fc[interior(q)]);
  tail_sum2<CLUSTER>(fs, u2, sh, slots, phase);
  const double rsden = (fs == 0.0) ? 1.0 : fs;
  // FP64 residual r = f - (A + cc) x -> FP32 right-hand side, and ||r||_1
  auto residual = [&]() {
    double acc = 0.0, unused = 0.0;
    const double *oC = B.op[OC], *oN = B.op[ON], *oE = B.op[OE], *uC = B.op[UC];
    const double *x = B.x, *f = B.fc, *cc = B.cc;
    float* w0 = B.w0;
    for_points<2>(
        nint, tid, interior,
        [&](int id) {
          return f[id] + oN[id] * x[id + sy] + oN[id - sy] * x[id - sy] + oE[id] * x[id + 1] +
                 oE[id - 1] * x[id - 1] + uC[id - sz] * x[id - sz] + uC[id] * x[id + sz] -
                 (oC[id] + cc[id]) * x[id];
        },
        [&](int id, double r) {
          w0[id] = (float)r;
          acc += fabs(r);
        });
    tail_sum2<CLUSTER>(acc, unused, sh, slots, phase);
    return acc;
  };
  double rs = residual();
  if (tid.block == 0 && B.nlog > 0) B.out[2] = rs / rsden;
  int it = 0;
  while (it < B.itmax && rs / rsden > B.errtol) {
    // FP32 V-cycle on A e = w0
    for (int sw = 0; sw < B.fine_sweeps; sw++) {
      batch_gs7<CLUSTER>(B, B.dh, dy, 1, sw == 0, tid);
      batch_gs7<CLUSTER>(B, B.dh, dy, 0, false, tid);
    }
    {
      const float *oC = B.op32[OC], *oN = B.op32[ON], *oE = B.op32[OE], *uC = B.op32[UC];
      const float *x = B.e, *w0 = B.w0, *cc = B.cc32;
      float* r = B.r;
      for_points<4>(
          nint, tid, interior,
          [&](int id) {
            const float nb = oN[id] * x[id + sy] + oN[id - sy] * x[id - sy] + oE[id] * x[id + 1] +
                             oE[id - 1] * x[id - 1] + uC[id - sz] * x[id - sz] +
                             uC[id] * x[id + sz];
            return w0[id] + nb - (oC[id] + cc[id]) * x[id];
          },
          [&](int id, float v) { r[id] = v; });
    }
    tail_sync<CLUSTER>();
    tail_cycle<CLUSTER>(T, false, tid, sh, slots, phase);
    const TLev& C = T.lev[1];
    double num, den;
    tail_damp<CLUSTER>(C, tid, sh, slots, phase, num, den);
    const float xdamp = (float)(num / den);
    tail_interp(C.g, C.x, g, dx, dy, B.e, xdamp, tid);
    tail_sync<CLUSTER>();
    for (int sw = 0; sw < B.fine_sweeps; sw++) {
      batch_gs7<CLUSTER>(B, B.dh, dy, 0, false, tid);
      batch_gs7<CLUSTER>(B, B.dh, dy, 1, false, tid);
    }
    {
      double* x = B.x;
      const float* e = B.e;
      for_points<4>(
          nint, tid, interior, [&](int id) { return x[id] + (double)e[id]; },
          [&](int id, double v) { x[id] = v; });
    }
    tail_sync<CLUSTER>();
    rs = residual();
    it++;
    if (tid.block == 0 && it < B.nlog) B.out[2 + it] = rs / rsden;
    if (!(rs == rs)) break;  // non-finite: reported by the host
  }
  if (tid.block == 0) {
    B.out[0] = (double)it;
    B.out[1] = rs / rsden;
  }
  // no CTA may exit while another can still read its shared memory
  tail_sync<CLUSTER>();
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
int mc_cluster_size(Grid g) {
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  if (nint > 200000) return 0;  // grid-wide colour launches
  if (nint > 20000) return 8;
  if (nint > 2000) return 2;
  return 1;
}

int gs27_mc(cudaStream_t s, const MLevel& L, float* x, int nsweep, int reverse, long long& k,
            int cooperative) {
  const int cl = mc_cluster_size(L.g);
  const OpF o = opf(L);
  if (cl == 0 && cooperative) {
    static const int coop_grid = [] {
      int dev = 0, nsm = 0, per = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_gs27_mc_coop, 256, 0);
      return nsm * (per < 1 ? 1 : per);
    }();
    Grid g = L.g;
    const float* cc = L.cc;
    const float* fc = L.w0;
    void* args[] = {&g, (void*)&o, &cc, &fc, &x, &nsweep, &reverse};
    const cudaError_t e = cudaLaunchCooperativeKernel((void*)k_gs27_mc_coop, dim3(coop_grid),
                                                      dim3(256), args, 0, s);
    k++;
    if (e != cudaSuccess) {
      set_error("gs27 multicolour cooperative launch: %s", cudaGetErrorString(e));
      return 0;
    }
    return 1;
  }
  if (cl == 0) {
    const size_t tot = (size_t)((L.g.nx - 1) / 2) * ((L.g.ny - 1) / 2) * ((L.g.nz - 1) / 2);
    for (int sw = 0; sw < nsweep; sw++)
      for (int c8 = 0; c8 < 8; c8++) {
        k_gs27_mc_colour<<<blocks_for(tot), kThreads, 0, s>>>(L.g, o, L.cc, L.w0, x,
                                                               reverse ? 7 - c8 : c8);
        k++;
      }
    return 1;
  }
  if (cl == 1) {
    k_gs27_mc_cluster<1><<<1, 512, 0, s>>>(L.g, o, L.cc, L.w0, x, nsweep, reverse);
    k++;
    return 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl, 1, 1);
  cfg.blockDim = dim3(1024, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = (cl == 8) ? cudaLaunchKernelEx(&cfg, k_gs27_mc_cluster<8>, L.g, o,
                                                 (const float*)L.cc, (const float*)L.w0, x,
                                                 nsweep, reverse)
                            : cudaLaunchKernelEx(&cfg, k_gs27_mc_cluster<2>, L.g, o,
                                                 (const float*)L.cc, (const float*)L.w0, x,
                                                 nsweep, reverse);
  k++;
  if (e != cudaSuccess) {
    set_error("gs27 multicolour launch: %s", cudaGetErrorString(e));
    return 0;
  }
  return 1;
}

// FP32 single-pass sweep arguments for the fine level (xin, xout set by the caller)
Gs7Rb<float> rb_f32(const MLevel& F, const float* d32, const int* tune) {
  Gs7Rb<float> a;
  a.oE = F.op[OE]; a.oN = F.op[ON]; a.uC = F.op[UC];
  a.D = d32; a.f = F.w0;
  a.nx = F.g.nx; a.S = F.g.nx * F.g.ny; a.nz = F.g.nz;
  a.kchunk = tune[6];  // 0: sized to the resident CTA slots
  a.xin = nullptr; a.xout = nullptr;
  return a;
}

// The fine-level FP32 smoothing: tune[11] red-black sweeps, from x = 0 (zero) or
// from x, then (r given) the residual.  Memory bounds a colour pass, the L2's up to
// 129^3 and HBM above, so the first pass from zero only writes and the diagonal is
// one array (oC + cc, as the single-pass sweep has it); an LPBE solve of 65^3 1.30 ->
// 1.22 ms, the same bits.  Every sweep is two colour passes; for tune[5] == 2 those
// after one from zero take a single pass out of place (x -> xs -> x ...; after an odd
// count xs is copied back).  Alone the single pass is the faster one on large grids
// (161^3 36.9 us against 41.5), in a solve it is not: an LPBE solve of 161^3 4.24 ms
// against 4.11 in colours, 193^3 6.43 and 6.43, 225^3 10.77 and 10.85, 257^3 15.8 and
// 15.5.  k counts the kernels launched.
bool gs7_f32_single(Grid g, const int* tune) {
  return tune[5] == 2 && (g.nx & 1) && (g.ny & 1);
}

cudaError_t gs7_f32(cudaStream_t st, const MLevel& F, float* x, float* r, int first_parity,
                    float* xs, const float* d32, bool zero, const int* tune, long long& k) {
  const int nsweep = tune[11];
  const size_t fint = (size_t)(F.g.nx - 2) * (F.g.ny - 2) * (F.g.nz - 2);
  const OpF fo = opf(F);
  const size_t nslots = (size_t)((F.g.nx - 1) / 2) * (F.g.ny - 2) * (F.g.nz - 2);
  cudaError_t e = cudaSuccess;
  auto colour = [&](int c) {
    k_gs7_f32<<<blocks_for(nslots), kThreads, 0, st>>>(F.g, fo, d32, F.w0, x, c);
    k++;
  };
  int sw = 0;
  if (zero && nsweep > 0) {
    k_gs7_f32_first<<<blocks_for(fint), kThreads, 0, st>>>(F.g, d32, F.w0, x, first_parity);
    k++;
    colour(1 - first_parity);
    sw = 1;
  } else if (zero) {
    e = cudaMemsetAsync(x, 0, F.g.n() * sizeof(float), st);
  }
  if (gs7_f32_single(F.g, tune)) {
    Gs7Rb<float> a = rb_f32(F, d32, tune);
    float *xin = x, *xout = xs;
    for (; sw < nsweep && e == cudaSuccess; sw++) {
      a.xin = xin;
      a.xout = xout;
      e = launch_gs7_rb<float>(st, a, first_parity, tune[12]);
      k++;
      std::swap(xin, xout);
    }
    if (e == cudaSuccess && xin != x)
      e = cudaMemcpyAsync(x, xs, F.g.n() * sizeof(float), cudaMemcpyDeviceToDevice, st);
  } else {
    for (; sw < nsweep; sw++) {
      colour(first_parity);
      colour(1 - first_parity);
    }
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (r && e == cudaSuccess) {
    k_resid7_f32<<<blocks_for(fint), kThreads, 0, st>>>(F.g, fo, d32, F.w0, x, r);
    k++;
    e = cudaGetLastError();
  }
  return e;
}

// FP32 D = oC + cc inside, 1 on the boundary
__global__ void k_diag_f32(Grid g, const float* __restrict__ oC, const float* __restrict__ cc,
                           float* D) {
  const size_t n = g.n();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
       q += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    split3(q, g.nx, g.ny, i, j, k);
    const bool inner = i > 0 && i < g.nx - 1 && j > 0 && j < g.ny - 1 && k > 0 && k < g.nz - 1;
    D[q] = inner ? oC[q] + cc[q] : 1.0f;
  }
}

int falloc(float** p, size_t n) {
  if (n == 0) n = 1;
  if (cudaMalloc((void**)p, n * sizeof(float)) != cudaSuccess) {
    set_error("cudaMalloc(%zu floats) failed", n);
    *p = nullptr;
    return 0;
  }
  cudaMemset(*p, 0, n * sizeof(float));
  return 1;
}

int dalloc64(double** p, size_t n) {
  if (n == 0) n = 1;
  if (cudaMalloc((void**)p, n * sizeof(double)) != cudaSuccess) {
    set_error("cudaMalloc(%zu doubles) failed", n);
    *p = nullptr;
    return 0;
  }
  cudaMemset(*p, 0, n * sizeof(double));
  return 1;
}

}  // namespace

void mixed_mark_stale(MixedState* m) {
  if (m) m->stale = 1;
}

void mixed_destroy(MixedState* m) {
  if (!m) return;
  for (int e = 0; e < 2; e++)
    if (m->exec[e]) cudaGraphExecDestroy(m->exec[e]);
  for (int l = 0; l < m->nlev; l++) {
    MLevel& L = m->lev[l];
    for (int c = 0; c < 14; c++) {
      if (L.op[c]) cudaFree(L.op[c]);
      if (L.own64 && L.op64[c]) cudaFree(L.op64[c]);
    }
    if (L.own64 && L.cc64) cudaFree(L.cc64);
    if (L.cc) cudaFree(L.cc);
    if (L.w0) cudaFree(L.w0);
    if (L.x) cudaFree(L.x);
    if (L.x2) cudaFree(L.x2);
    if (L.d) cudaFree(L.d);
  }
  if (m->lam) cudaFree(m->lam);
  if (m->r) cudaFree(m->r);
  if (m->w2) cudaFree(m->w2);
  if (m->xs) cudaFree(m->xs);
  if (m->d32) cudaFree(m->d32);
  if (m->dense) cudaFree(m->dense);
  if (m->dvec) cudaFree(m->dvec);
  if (m->dinfo) cudaFree(m->dinfo);
  if (m->d_tlev) cudaFree(m->d_tlev);
  if (m->d_flag) cudaFree(m->d_flag);
  if (m->dense_fork) cudaEventDestroy(m->dense_fork);
  if (m->dense_ev) cudaEventDestroy(m->dense_ev);
  delete m;
}

namespace {

// Build the FP32 hierarchy from the FP64 one (plus extra Galerkin levels).
int mixed_setup_from(pmgb_solver* s, int lo) {
  if (s->mixed) return 1;
  MixedState* m = new MixedState();
  memset(m, 0, sizeof(*m));
  s->mixed = m;
  m->lo = lo;
  cudaStream_t st = s->stream;
  CKM(cudaEventCreateWithFlags(&m->dense_fork, cudaEventDisableTiming));
  CKM(cudaEventCreateWithFlags(&m->dense_ev, cudaEventDisableTiming));

  // levels shared with the FP64 hierarchy
  int nl = 0;
  m->zero_cc = (lo > 0);
  for (int l = 0; l < s->nlev; l++, nl++) {
    MLevel& L = m->lev[l];
    L.g = s->lev[l].g;
    L.nop = s->lev[l].nop;
    if (lo > 0 && l == lo) {
      // exact coarse solve of the FP64 path: the reference's band matrix
      // written as a 27-point operator (k_band_restencil), without cc
      L.own64 = 1;
      for (int c = 0; c < L.nop; c++)
        if (!dalloc64(&L.op64[c], L.g.n())) return 0;
      if (!dalloc64(&L.cc64, L.g.n())) return 0;
    } else {
      for (int c = 0; c < L.nop; c++) L.op64[c] = s->lev[l].op[c];
      L.own64 = 0;
      L.cc64 = nullptr;
    }
  }
  if (lo > 0) CKM(cudaMalloc(&m->d_flag, sizeof(int)));
  // extra coarse levels until <= 512 interior unknowns or the grid cannot
  // be coarsened exactly
  while (nl < 16) {
    const Grid g = m->lev[nl - 1].g;
    const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
    if (nint <= 512) break;
    if ((g.nx - 1) % 2 || (g.ny - 1) % 2 || (g.nz - 1) % 2) break;
    const Grid c{(g.nx - 1) / 2 + 1, (g.ny - 1) / 2 + 1, (g.nz - 1) / 2 + 1};
    if (c.nx < 3 || c.ny < 3 || c.nz < 3) break;
    MLevel& L = m->lev[nl];
    L.g = c;
    L.nop = 14;
    L.own64 = 1;
    for (int q = 0; q < 14; q++)
      if (!dalloc64(&L.op64[q], c.n())) return 0;
    if (!dalloc64(&L.cc64, c.n())) return 0;
    nl++;
  }
  m->nlev = nl;
  // operator pointers of the extra levels join the solver's device table
  for (int l = s->nlev; l < nl; l++)
    CKM(cudaMemcpy(s->d_opptrs + 14 * l, m->lev[l].op64, sizeof(double*) * 14,
                   cudaMemcpyHostToDevice));
  // FP32 storage (filled by mixed_refresh)
  for (int l = lo; l < nl; l++) {
    MLevel& L = m->lev[l];
    const size_t n = L.g.n();
    for (int c = 0; c < L.nop; c++)
      if (!falloc(&L.op[c], n)) return 0;
    if (!falloc(&L.cc, n) || !falloc(&L.w0, n) || !falloc(&L.x, n)) return 0;
    if (l >= 1 && L.nop == 14 && (!falloc(&L.x2, n) || !falloc(&L.d, n))) return 0;
  }
  if (!falloc(&m->lam, 16)) return 0;
  m->stale = 1;
  const size_t nscr = m->lev[lo].g.n();
  if (!falloc(&m->r, nscr) || !falloc(&m->w2, nscr)) return 0;
  if (lo == 0 && (!falloc(&m->xs, nscr) || !falloc(&m->d32, nscr))) return 0;
  const Grid gc = m->lev[nl - 1].g;
  m->nd = (gc.nx - 2) * (gc.ny - 2) * (gc.nz - 2);
  if (m->nd > 4096) {
    set_error("mixed: coarsest level too large (%d unknowns)", m->nd);
    return 0;
  }
  if (!dalloc64(&m->dense, (size_t)m->nd * m->nd) || !dalloc64(&m->dvec, m->nd)) return 0;
  CKM(cudaMalloc(&m->dinfo, sizeof(int) * 4));
  // Levels small enough for one cluster run in the tail kernel: 16 SMs take a pass
  // over 33^3 points at about 8 us (their share of the L2's bandwidth bounds it),
  // a launch on all SMs at 3 us, while 25^3 and below take 2 to 3 us in the cluster
  // with the barrier.  Limit 70000 -> 20000: LPBE solves of 65^3 1.43 -> 1.30 ms,
  // 129^3 3.06 -> 2.90, NPBE 161^3 8.11 -> 7.52.
  // The exact coarse solve of the FP64 path always runs its levels in one
  // cluster; the mixed V-cycle does from the first level under the limit
  m->tail_first = (lo > 0) ? lo : 0;
  for (int l = 1; lo == 0 && l < nl; l++) {
    const Grid g = m->lev[l].g;
    if ((size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2) <= (size_t)s->tune[8]) {
      m->tail_first = l;
      break;
    }
  }
  {
    std::vector<TLev> tl(nl);
    for (int l = 0; l < nl; l++) {
      tl[l].g = m->lev[l].g;
      tl[l].dx = div_const(m->lev[l].g.nx - 2);
      tl[l].dy = div_const(m->lev[l].g.ny - 2);
      for (int c = 0; c < 14; c++) tl[l].op[c] = m->lev[l].op[c];
      tl[l].cc = m->lev[l].cc;
      tl[l].w0 = m->lev[l].w0;
      tl[l].x = m->lev[l].x;
      tl[l].x2 = m->lev[l].x2;
      tl[l].d = m->lev[l].d;
      tl[l].lam = m->lam + l;
    }
    CKM(cudaMalloc(&m->d_tlev, sizeof(TLev) * nl));
    CKM(cudaMemcpy(m->d_tlev, tl.data(), sizeof(TLev) * nl, cudaMemcpyHostToDevice));
    m->tail_cluster = 16;
    if (cudaFuncSetAttribute(k_vcycle_tail<16>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess ||
        cudaFuncSetAttribute(k_coarse_exact<16>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess) {
      cudaGetLastError();
      m->tail_cluster = 8;
    } else {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16, 1, 1);
      cfg.blockDim = dim3(512, 1, 1);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 16;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int ncl = 0, ncl2 = 0;
      if (cudaOccupancyMaxActiveClusters(&ncl, k_vcycle_tail<16>, &cfg) != cudaSuccess || ncl < 1 ||
          cudaOccupancyMaxActiveClusters(&ncl2, k_coarse_exact<16>, &cfg) != cudaSuccess ||
          ncl2 < 1) {
        cudaGetLastError();
        m->tail_cluster = 8;
      }
    }
  }
  CKM(cudaStreamSynchronize(st));
  return 1;
}

int mixed_setup(pmgb_solver* s) { return mixed_setup_from(s, 0); }

// Galerkin operators of the extra levels and the FP32 copies of every
// level's operator, after each rebuild of the FP64 hierarchy.
int mixed_refresh(pmgb_solver* s) {
  MixedState* m = s->mixed;
  if (!m->stale) return 1;
  cudaStream_t st = s->stream;
  for (int l = s->nlev; l < m->nlev; l++) {
    launch_galerkin(st, m->lev[l - 1].g, m->lev[l - 1].ops64(), m->lev[l].g,
                    s->d_opptrs + 14 * l);
    note_launches(1);
  }
  ConvQueue conv(st);
  for (int l = m->lo; l < m->nlev; l++) {
    MLevel& L = m->lev[l];
    for (int c = 0; c < L.nop; c++) conv.add(L.op64[c], L.op[c], L.g.n());
  }
  conv.flush();
  for (int l = m->lo; l < m->nlev; l++) {
    MLevel& L = m->lev[l];
    if (l >= 1 && L.nop == 14 && L.x2) {
      // the Chebyshev interval of this level: the Gershgorin bound of
      // D^-1 A without the Helmholtz term, which stays an upper bound for
      // every cc >= 0 (the linear term and c'(u) of the Newton steps), so
      // the bound follows operator rebuilds only
      CKM(cudaMemsetAsync(m->lam + l, 0, sizeof(float), st));
      const size_t nint = (size_t)(L.g.nx - 2) * (L.g.ny - 2) * (L.g.nz - 2);
      k_gersh<<<blocks_for(nint), kThreads, 0, st>>>(L.g, opf(L), nullptr, m->lam + l);
      note_launches(1);
    }
  }
  CKM(cudaGetLastError());
  m->stale = 0;
  m->cc_ready = 0;
  return 1;
}

// Helmholtz term on every mixed level from the fine FP64 term cc0:
// restrict through the FP64 levels (where not already present) and convert.
constexpr size_t kDenseSmemMax = 200 * 1024;

// The dense inverse on the smallest cluster whose row blocks fit one CTA's
// shared memory (rows, two pivot rows and a column).
template <int CL>
static cudaError_t dense_inverse_cl(cudaStream_t st, double* M, int n, int rows_per,
                                    size_t smem, int* info) {
  static const cudaError_t attr = [] {
    cudaError_t e = cudaFuncSetAttribute(k_dense_inverse<CL>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kDenseSmemMax);
    if (e == cudaSuccess && CL > 8)
      e = cudaFuncSetAttribute(k_dense_inverse<CL>,
                               cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  if (CL == 1) {
    k_dense_inverse<1><<<1, 1024, smem, st>>>(M, n, rows_per, info);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, 1, 1);
  cfg.blockDim = dim3(1024, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_dense_inverse<CL>, M, n, rows_per, info);
}

static int launch_dense_inverse(cudaStream_t st, double* M, int n, int* info) {
  for (int cl = 1; cl <= 16; cl *= 2) {
    const int rows_per = (n + cl - 1) / cl;
    const size_t smem = ((size_t)rows_per * n + 2 * (size_t)n + rows_per) * sizeof(double);
    if (smem > kDenseSmemMax) continue;
    cudaError_t e;
    switch (cl) {
      case 1: e = dense_inverse_cl<1>(st, M, n, rows_per, smem, info); break;
      case 2: e = dense_inverse_cl<2>(st, M, n, rows_per, smem, info); break;
      case 4: e = dense_inverse_cl<4>(st, M, n, rows_per, smem, info); break;
      case 8: e = dense_inverse_cl<8>(st, M, n, rows_per, smem, info); break;
      default: e = dense_inverse_cl<16>(st, M, n, rows_per, smem, info); break;
    }
    return e == cudaSuccess;
  }
  return 0;
}

int mixed_set_cc(pmgb_solver* s, int newton, int defer_check = 0) {
  MixedState* m = s->mixed;
  cudaStream_t st = s->stream;
  // the previous dense inverse reads the coarsest term rewritten below
  CKM(cudaStreamWaitEvent(st, m->dense_ev, 0));
  ConvQueue conv(st);
  for (int l = 0; l < m->nlev; l++) {
    MLevel& L = m->lev[l];
    const double* src;
    if (m->zero_cc) {
      // band operator below the FP64 hierarchy: no Helmholtz term anywhere
      if (l < m->lo) continue;
      CKM(cudaMemsetAsync(L.cc, 0, L.g.n() * sizeof(float), st));
      src = L.cc64;  // allocated zero and never written
    } else if (l < s->nlev) {
      src = newton ? s->lev[l].cp : s->lev[l].cc;
    } else {
      const double* prev = (l - 1 < s->nlev) ? (newton ? s->lev[l - 1].cp : s->lev[l - 1].cc)
                                             : m->lev[l - 1].cc64;
      launch_restrict(st, m->lev[l - 1].g, prev, L.g, L.cc64);
      note_launches(1);
      src = L.cc64;
    }
    if (l >= m->lo && !m->zero_cc) conv.add(src, L.cc, L.g.n());
    if (l == m->nlev - 1) {
      // dense inverse of (A_c + cc) on the coarsest level, on the side stream:
      // the V-cycle's finer levels run meanwhile and its coarsest solve waits
      // for dense_ev
      const int nd = m->nd;
      CKM(cudaEventRecord(m->dense_fork, st));
      CKM(cudaStreamWaitEvent(s->side, m->dense_fork, 0));
      k_dense_build<<<blocks_for((size_t)nd * nd), kThreads, 0, s->side>>>(
          L.g, L.ops64(), src, m->dense, nd);
      const int ok = launch_dense_inverse(s->side, m->dense, nd, m->dinfo);
      CKM(cudaEventRecord(m->dense_ev, s->side));
      if (!ok) {
        set_error("mixed: dense coarsest inverse launch failed (%d unknowns)", nd);
        return 0;
      }
      note_launches(2);
    }
  }
  // the FP32 Helmholtz terms of all levels in one launch
  conv.flush();
  MLevel& F = m->lev[0];
  if (m->d32) {
    // the fine level's divisor, one array for the sweeps and the residual to read
    k_diag_f32<<<blocks_for(F.g.n()), kThreads, 0, st>>>(F.g, F.op[OC], F.cc, m->d32);
    note_launches(1);
  }
  m->cc_ready = 1;
  if (defer_check) {
    // the caller's next read of the residual also reads the factor's status
    m->info_pending = 1;
    return 1;
  }
  CKM(cudaStreamWaitEvent(st, m->dense_ev, 0));
  int info = 0;
  CKM(cudaMemcpyAsync(&info, m->dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
  CKM(cudaStreamSynchronize(st));
  if (info != 0) {
    set_error("mixed: coarsest operator not positive definite (pivot %d)", info);
    return 0;
  }
  return 1;
}

// Chebyshev degree of the 27-point FP32 levels (PMGB_TUNE_MIXED_CHEBYSHEV,
// rounded up to even), 0 for the 8-colour Gauss-Seidel
int cheb_degree(const int* tune) {
  const int k = tune[PMGB_TUNE_MIXED_CHEBYSHEV];
  return k <= 0 ? 0 : (k + 1) & ~1;
}

// smoothing of a 27-point FP32 level outside the tail: K Chebyshev steps
// (one launch each) or the 8-colour Gauss-Seidel
int smooth27(cudaStream_t st, MLevel& L, MixedState* m, int l, int first, int reverse,
             long long& k, const int* tune) {
  const int K = cheb_degree(tune);
  if (K == 0 || !L.x2) return gs27_mc(st, L, L.x, tune[10], reverse, k, tune[9]);
  const size_t nint = (size_t)(L.g.nx - 2) * (L.g.ny - 2) * (L.g.nz - 2);
  const OpF o = opf(L);
  for (int i = first; i < K; i++) {
    k_cheb_step<<<blocks_for(nint), kThreads, 0, st>>>(L.g, o, L.cc, L.w0, (i & 1) ? L.x2 : L.x,
                                                       (i & 1) ? L.x : L.x2, L.d, m->lam + l, i);
    k++;
  }
  CKM(cudaGetLastError());
  return 1;
}

int launch_tail(pmgb_solver* s, cudaStream_t st) {
  MixedState* m = s->mixed;
  const int nl = m->nlev, tf = m->tail_first;
  TailArgs A;
  A.lev = m->d_tlev;
  A.first = tf;
  A.last = nl - 1;
  A.gprev = m->lev[tf - 1].g;
  A.rprev = m->r;
  A.r = m->w2;
  A.minv = m->dense;
  A.nd = m->nd;
  A.nsweep = s->tune[10];
  A.cheb = cheb_degree(s->tune);
  A.xnum = s->scal + S_XNUM_L + ((tf - 1) & 15);
  A.xden = s->scal + S_XDEN_L + ((tf - 1) & 15);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(m->tail_cluster, 1, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = m->tail_cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = (m->tail_cluster == 16) ? cudaLaunchKernelEx(&cfg, k_vcycle_tail<16>, A)
                                          : cudaLaunchKernelEx(&cfg, k_vcycle_tail<8>, A);
  if (e != cudaSuccess) {
    set_error("tail kernel launch: %s", cudaGetErrorString(e));
    return 0;
  }
  return 1;
}

// One FP32 V-cycle on A e = w0 (fine rhs already in lev[0].w0), e -> lev[0].x,
// then x64 += e, the FP64 residual of (fc64, cc64, x64) into lev[0].w0 and its
// 1-norm into scal[S_RSNRM].
int mixed_cycle_body(pmgb_solver* s, const double* cc64, const double* fc64, double* x64,
                     long long& k) {
  MixedState* m = s->mixed;
  cudaStream_t st = s->stream;
  const int nl = m->nlev;
  MLevel& F = m->lev[0];
  const OpF fo = opf(F);
  const size_t fint = (size_t)(F.g.nx - 2) * (F.g.ny - 2) * (F.g.nz - 2);
  if (gs7_f32(st, F, F.x, m->r, 1, m->xs, m->d32, true, s->tune, k) != cudaSuccess) {
    set_error("FP32 fine smoother launch failed");
    return 0;
  }
  const int tf = m->tail_first > 0 ? m->tail_first : nl;
  for (int l = 1; l < tf; l++) {
    MLevel& C = m->lev[l];
    const bool last = l == nl - 1;
    const bool cheb0 = !last && cheb_degree(s->tune) > 0 && C.x2;
    k_restrict_f32<<<blocks_for(C.g.n()), kThreads, 0, st>>>(
        m->lev[l - 1].g, m->r, C.g, C.w0, C.op[OC], C.cc, m->lam + l, last ? nullptr : C.x,
        cheb0 ? C.x2 : nullptr, C.d);
    k++;
    if (!last) {
      if (!smooth27(st, C, m, l, cheb0 ? 1 : 0, 0, k, s->tune)) return 0;
      const size_t cint = (size_t)(C.g.nx - 2) * (C.g.ny - 2) * (C.g.nz - 2);
      k_resid_f32<<<blocks_for(cint), kThreads, 0, st>>>(C.g, opf(C), C.cc, C.w0, C.x, m->r);
      k++;
    }
  }
  // the coarsest solve reads the dense inverse made on the side stream
  CKM(cudaStreamWaitEvent(st, m->dense_ev, cudaEventWaitExternal));
  if (m->tail_first > 0) {
    if (!launch_tail(s, st)) return 0;
    k++;
  } else {
    MLevel& C = m->lev[nl - 1];
    k_dense_apply<<<1, 512, m->nd * sizeof(double), st>>>(C.g, m->dense, m->nd, C.w0, C.x);
    k++;
  }
  const int upstart = (m->tail_first > 0) ? tf - 1 : nl - 2;
  for (int l = upstart; l >= 0; l--) {
    MLevel& C = m->lev[l + 1];
    MLevel& P = m->lev[l];
    if (l + 1 != tf || m->tail_first == 0) {
      damp_dots(st, C.g, opf(C), C.cc, C.x, C.w0, s->part, s->d_wave + kWaveMixedDampTicket,
                s->scal + S_XNUM_L + (l & 15),
                s->scal + S_XDEN_L + (l & 15));
      k += 1;
    }
    k_interp_axpy_f32<<<blocks_for((size_t)(C.g.nx - 1) * (C.g.ny - 1) * (C.g.nz - 1)),
                        kThreads, 0, st>>>(
        C.g, C.x, P.g, P.x, s->scal + S_XNUM_L + (l & 15), s->scal + S_XDEN_L + (l & 15));
    k += 1;
    if (l == 0) {
      if (gs7_f32(st, F, F.x, nullptr, 0, m->xs, m->d32, false, s->tune, k) != cudaSuccess) {
        set_error("FP32 fine smoother launch failed");
        return 0;
      }
    } else {
      if (!smooth27(st, P, m, l, 0, 1, k, s->tune)) return 0;
    }
  }
  // x64 += e ; r = f - (A + cc) x64 (FP64) -> FP32 rhs ; ||r||_1
  k_add_corr<<<blocks_for(fint), kThreads, 0, st>>>(F.g, F.x, x64);
  const int nb = (int)reduce_parts(fint);
  k_resid64_to32<<<nb, 256, 0, st>>>(F.g, s->lev[0].ops(), cc64, fc64, x64, F.w0, s->part);
  k_sum_parts<<<1, 256, 0, st>>>(s->part, nb, s->scal + S_RSNRM);
  k += 3;
  return 1;
}

int read_scal(pmgb_solver* s, int slot, double* v) {
  CKM(cudaMemcpyAsync(v, s->scal + slot, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  MixedState* m = s->mixed;
  int info = 0;
  const int check = m && m->info_pending;
  if (check) {
    CKM(cudaStreamWaitEvent(s->stream, m->dense_ev, 0));
    CKM(cudaMemcpyAsync(&info, m->dinfo, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  }
  CKM(cudaStreamSynchronize(s->stream));
  if (check) {
    m->info_pending = 0;
    if (info != 0) {
      set_error("mixed: coarsest operator not positive definite (pivot %d)", info);
      return 0;
    }
  }
  return 1;
}

// Refinement loop on (A + cc) x = f, all FP64 vectors on the fine level:
// stop when ||f - (A+cc)x||_1 / rsden <= errtol (rsden = ||f||_1, or 1 for
// the Newton inner solve, istop0, which starts from x64 = 0).
int refine(pmgb_solver* s, int newton, const double* cc64, const double* fc64, double* x64,
           double errtol, int itmax, int istop0, int* iters_out) {
  MixedState* m = s->mixed;
  cudaStream_t st = s->stream;
  const Grid g = s->g;
  const size_t fint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  const int nb = (int)reduce_parts(fint);
  if (istop0) {
    // the Newton inner solve starts from x64 = 0, where the residual is f
    // itself (f + 0 - 0): its FP32 copy is the V-cycle's rhs, and its norm
    // is not needed
    ConvQueue conv(st);
    conv.add(fc64, m->lev[0].w0, g.n());
    conv.flush();
  } else {
    // initial residual (x64 as given) -> FP32 rhs and its norm
    k_resid64_to32<<<nb, 256, 0, st>>>(g, s->lev[0].ops(), cc64, fc64, x64, m->lev[0].w0,
                                       s->part);
    k_sum_parts<<<1, 256, 0, st>>>(s->part, nb, s->scal + S_RSNRM);
    note_launches(2);
  }
  double rsden = 1.0, rsnrm = 0.0;
  if (!istop0) {
    launch_nrm1(st, g, fc64, s->part + 2368, s->scal + S_RSDEN);
    note_launches(2);
    if (!read_scal(s, S_RSDEN, &rsden)) return 0;
    if (rsden == 0.0) rsden = 1.0;
    if (!read_scal(s, S_RSNRM, &rsnrm)) return 0;
  }
  // the Newton inner solve logs 1 and always runs a cycle: its initial
  // residual norm is not needed on the host
  s->reslog.push_back(istop0 ? 1.0 : rsnrm / rsden);
  if (!m->exec[newton]) {
    cudaGraph_t graph;
    long long k = 0;
    CKM(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const int ok = mixed_cycle_body(s, cc64, fc64, x64, k);
    cudaError_t e = cudaStreamEndCapture(st, &graph);
    if (!ok) return 0;
    if (e != cudaSuccess) {
      set_error("mixed graph capture: %s", cudaGetErrorString(e));
      return 0;
    }
    CKM(cudaGraphInstantiate(&m->exec[newton], graph, 0));
    cudaGraphDestroy(graph);
    m->kernels[newton] = k;
  }
  int iters = 0;
  do {
    CKM(cudaGraphLaunch(m->exec[newton], st));
    note_launches(m->kernels[newton]);
    if (!read_scal(s, S_RSNRM, &rsnrm)) return 0;
    iters++;
    s->st.vcycles++;
    s->reslog.push_back(rsnrm / rsden);
    if (!(rsnrm == rsnrm)) {
      set_error("mixed: non-finite residual");
      return 0;
    }
  } while (iters < itmax && (rsnrm / rsden) > errtol);
  s->st.refinements += iters;
  s->st.rel_residual = rsnrm / rsden;
  *iters_out = iters;
  return 1;
}

}  // namespace

// Inner solve of one Newton step (called by the Newton driver in solver.cu
// with s->lev[*].cp and .rhs in place): xt = 0 and refine until
// ||rhs - J xt||_1 <= errtol_s.
int mixed_newton_inner(pmgb_solver* s, double errtol_s) {
  if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
  if (!mixed_set_cc(s, 1, 1)) return 0;
  Level& F = s->lev[0];
  CKM(cudaMemsetAsync(F.xt, 0, s->n * sizeof(double), s->stream));
  int it = 0;
  return refine(s, 1, F.cp, F.rhs, F.xt, errtol_s, 1000, 1, &it);
}

int mixed_fine_single(const pmgb_solver* s) { return gs7_f32_single(s->g, s->tune); }

// One FP32 fine-level half-sweep for kernel timing; 5 FP32 arrays read and
// x read/written: 12 B per point per half-sweep.
int mixed_time_gs7(pmgb_solver* s, int parity, double* bytes) {
  if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
  MixedState* m = s->mixed;
  MLevel& F = m->lev[0];
  const size_t nslots = (size_t)((F.g.nx - 1) / 2) * (F.g.ny - 2) * (F.g.nz - 2);
  k_gs7_f32<<<blocks_for(nslots), kThreads, 0, s->stream>>>(F.g, opf(F), m->d32, F.w0, F.x,
                                                            parity);
  *bytes = 12.0 * (double)(F.g.nx - 2) * (F.g.ny - 2) * (F.g.nz - 2);
  return 1;
}

// One FP32 single-pass sweep for kernel timing: 28 B per point per sweep
// (6 FP32 arrays read, x read and written once).  mixed_prepare_sweep makes
// the divisor first.
int mixed_prepare_sweep(pmgb_solver* s) {
  if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
  MixedState* m = s->mixed;
  MLevel& F = m->lev[0];
  if (!m->d32) {
    set_error("pmgb_time_kernel: no FP32 fine sweep in this calculation");
    return 0;
  }
  k_diag_f32<<<blocks_for(F.g.n()), kThreads, 0, s->stream>>>(F.g, F.op[OC], F.cc, m->d32);
  CKM(cudaGetLastError());
  return 1;
}

int mixed_time_gs7_sweep(pmgb_solver* s, double* bytes) {
  MixedState* m = s->mixed;
  MLevel& F = m->lev[0];
  Gs7Rb<float> a = rb_f32(F, m->d32, s->tune);
  a.xin = F.x; a.xout = m->xs;
  const cudaError_t e = launch_gs7_rb<float>(s->stream, a, 1, s->tune[12]);
  if (e != cudaSuccess) {
    set_error("FP32 sweep launch failed");
    return 0;
  }
  *bytes = 28.0 * (double)(F.g.nx - 2) * (F.g.ny - 2) * (F.g.nz - 2);
  return 1;
}

// The coarse tail alone, for kernel timing.  Algorithmic bytes per tail
// level above the coarsest: 2+2 FP32 27-point sweeps, the residual and the
// damping pass read 14 coefficients + cc + f + x (72 B per point each) and
// the interpolation writes x: 6 x 72 + 8 = 440 B per interior point.
int mixed_time_tail(pmgb_solver* s, double* bytes) {
  if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
  MixedState* m = s->mixed;
  if (m->lo != 0 || m->tail_first <= 0) {
    set_error("pmgb_time_kernel: no mixed-precision tail levels in this calculation");
    return 0;
  }
  if (!launch_tail(s, s->stream)) return 0;
  double b = 0.0;
  for (int l = m->tail_first; l < m->nlev - 1; l++) {
    const Grid g = m->lev[l].g;
    b += 440.0 * (double)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  }
  b += 8.0 * (double)m->nd * m->nd;
  *bytes = b;
  return 1;
}

void launch_band_restencil(cudaStream_t st, Grid g, Op op, double* const* b, int* wrap) {
  OpW w;
  for (int c = 0; c < 14; c++) w.c[c] = b[c];
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  k_band_restencil<<<blocks_for(nint), kThreads, 0, st>>>(g, op, w, wrap);
}

// FP64 path, LPBE: prepare the exact coarse solve of the FP64 coarsest level
// (FP32 Galerkin levels below it and the dense inverse at the bottom).
// Returns 1 when it is available, 0 when the band solve must be used.
int coarse_exact_prepare(pmgb_solver* s) {
  const int lo = s->nlev - 1;
  if (!s->mixed) {
    if (!mixed_setup_from(s, lo)) {
      // e.g. a coarsest level that cannot be coarsened further: fall back
      if (s->mixed) {
        mixed_destroy(s->mixed);
        s->mixed = nullptr;
      }
      cudaGetLastError();
      return 0;
    }
  }
  MixedState* m = s->mixed;
  if (m->lo != lo || m->nlev <= lo + 1) return 0;
  // B, the operator the reference's band solve inverts
  cudaStream_t st = s->stream;
  MLevel& L = m->lev[lo];
  const Grid g = L.g;
  for (int c = 0; c < 14; c++) CKM(cudaMemsetAsync(L.op64[c], 0, g.n() * sizeof(double), st));
  CKM(cudaMemsetAsync(m->d_flag, 0, sizeof(int), st));
  launch_band_restencil(st, g, s->lev[lo].ops(), L.op64, m->d_flag);
  note_launches(1);
  int wrap = 0;
  CKM(cudaMemcpyAsync(&wrap, m->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  CKM(cudaStreamSynchronize(st));
  if (wrap) return 0;  // keep the band factorisation
  m->stale = 1;
  if (!mixed_refresh(s)) return 0;
  if (!mixed_set_cc(s, 0)) return 0;
  return 1;
}

int launch_coarse_exact(pmgb_solver* s, cudaStream_t st, const double* cc, const double* b,
                        double* x) {
  MixedState* m = s->mixed;
  const int lo = m->lo;
  ExactArgs E;
  E.T.lev = m->d_tlev;
  E.T.first = lo;
  E.T.last = m->nlev - 1;
  E.T.gprev = m->lev[lo].g;
  E.T.rprev = nullptr;
  E.T.r = m->w2;
  E.T.minv = m->dense;
  E.T.nd = m->nd;
  E.T.nsweep = 2;
  E.T.xnum = s->scal + S_TMP;
  E.T.xden = s->scal + S_TMP;
  E.g = s->lev[lo].g;
  for (int c = 0; c < 14; c++) E.op[c] = m->lev[lo].op64[c];
  E.cc = m->lev[lo].cc64;  // the band matrix has no Helmholtz term
  (void)cc;
  E.b = b;
  E.x = x;
  E.r = s->w3;
  E.maxit = 40;
  E.rtol = 1.0e-12;
  E.iters = s->d_iters + 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(m->tail_cluster, 1, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = m->tail_cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = (m->tail_cluster == 16) ? cudaLaunchKernelEx(&cfg, k_coarse_exact<16>, E)
                                          : cudaLaunchKernelEx(&cfg, k_coarse_exact<8>, E);
  if (e != cudaSuccess) {
    set_error("exact coarse solve launch: %s", cudaGetErrorString(e));
    return 0;
  }
  return 1;
}

int mixed_solve(pmgb_solver* s, double errtol, int itmax) {
  if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
  CKM(cudaMemsetAsync(s->lev[0].x, 0, s->n * sizeof(double), s->stream));
  if (!s->p.nonlin) {
    if (!s->mixed->cc_ready && !mixed_set_cc(s, 0)) return 0;
    int it = 0;
    Level& F = s->lev[0];
    return refine(s, 0, F.cc, F.fc, F.x, errtol, itmax, 0, &it);
  }
  return newton_driver(s, errtol, itmax, 1);
}

}  // namespace pmgb

// ---------------------------------------------------------------------------
// Batched solve entry point
// ---------------------------------------------------------------------------
// largest level 1 (interior points) the batched kernel takes into its cluster
constexpr int kBatchTailMax = 70000;

extern "C" int pmgb_batch_solve(pmgb_solver* const* solvers, int n, void* cuda_stream) {
  using namespace pmgb;
  if (!solvers || n < 1) {
    set_error("pmgb_batch_solve: no calculations");
    return 0;
  }
  int dev = -1;
  CKM(cudaGetDevice(&dev));
  for (int b = 0; b < n; b++) {
    pmgb_solver* s = solvers[b];
    if (!s || !s->filled || s->precision != PMGB_MIXED || s->p.nonlin || s->device != dev) {
      set_error("pmgb_batch_solve: calculation %d is not a filled mixed-precision LPBE "
                "calculation on the current device", b);
      return 0;
    }
  }
  // operators, FP32 hierarchies and coarsest inverses, per calculation
  int cl = 16;
  for (int b = 0; b < n; b++) {
    pmgb_solver* s = solvers[b];
    if (!s->built && !solver_build(s)) return 0;
    if (!mixed_setup(s) || !mixed_refresh(s)) return 0;
    if (!s->mixed->cc_ready && !mixed_set_cc(s, 0)) return 0;
    // the persistent kernel runs every level from 1 down in its cluster, whatever
    // level the calculation's own V-cycle begins its tail at
    const Grid g1 = s->nlev > 1 ? s->lev[1].g : s->g;
    const size_t n1 = (size_t)(g1.nx - 2) * (g1.ny - 2) * (g1.nz - 2);
    if (s->nlev < 2 ||
        n1 > (size_t)std::max(kBatchTailMax, s->tune[PMGB_TUNE_TAIL_MAX_POINTS])) {
      set_error("pmgb_batch_solve: calculation %d (%dx%dx%d) is too large for one cluster "
                "(its level 1 exceeds the tail limit)", b, s->p.nx, s->p.ny, s->p.nz);
      return 0;
    }
    cl = std::min(cl, s->mixed->tail_cluster);
  }
  static const int cl16_ok = [] {
    if (cudaFuncSetAttribute(k_batch_solve<16>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16, 1, 1);
    cfg.blockDim = dim3(512, 1, 1);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int ncl = 0;
    if (cudaOccupancyMaxActiveClusters(&ncl, k_batch_solve<16>, &cfg) != cudaSuccess || ncl < 1) {
      cudaGetLastError();
      return 0;
    }
    return 1;
  }();
  if (!cl16_ok) cl = 8;
  cudaStream_t st = cuda_stream ? (cudaStream_t)cuda_stream : solvers[0]->stream;
  for (int b = 0; b < n; b++) CKM(cudaStreamSynchronize(solvers[b]->stream));
  // the packed descriptor table
  const int nlog = 64;
  std::vector<BatchItem> items(n);
  BatchItem* d_items = nullptr;
  double* d_out = nullptr;
  CKM(cudaMallocAsync((void**)&d_items, sizeof(BatchItem) * n, st));
  CKM(cudaMallocAsync((void**)&d_out, sizeof(double) * (2 + nlog) * n, st));
  for (int b = 0; b < n; b++) {
    pmgb_solver* s = solvers[b];
    MixedState* m = s->mixed;
    BatchItem& B = items[b];
    B.T.lev = m->d_tlev;
    B.T.first = 1;
    B.T.last = m->nlev - 1;
    B.T.gprev = m->lev[0].g;
    B.T.rprev = m->r;
    B.T.r = m->w2;
    B.T.minv = m->dense;
    B.T.nd = m->nd;
    B.T.nsweep = s->tune[10];
    B.T.cheb = cheb_degree(s->tune);  // the same smoothing as the calculation's own V-cycle
    B.fine_sweeps = s->tune[11];
    B.T.xnum = s->scal + S_TMP;
    B.T.xden = s->scal + S_TMP;
    B.g = s->g;
    B.dx = div_const(s->g.nx - 2);
    B.dy = div_const(s->g.ny - 2);
    B.dh = div_const((s->g.nx - 1) / 2);
    for (int c = 0; c < 4; c++) {
      B.op[c] = s->lev[0].op[c];
      B.op32[c] = m->lev[0].op[c];
    }
    B.cc = s->lev[0].cc;
    B.fc = s->lev[0].fc;
    B.x = s->lev[0].x;
    B.cc32 = m->lev[0].cc;
    B.w0 = m->lev[0].w0;
    B.e = m->lev[0].x;
    B.r = m->r;
    B.errtol = (s->p.etol > 0.0) ? s->p.etol : 1.0e-6;
    B.itmax = (s->p.itmax > 0) ? s->p.itmax : 200;
    B.nlog = nlog;
    B.out = d_out + (size_t)(2 + nlog) * b;
  }
  CKM(cudaMemcpyAsync(d_items, items.data(), sizeof(BatchItem) * n, cudaMemcpyHostToDevice, st));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * n, 1, 1);
  cfg.blockDim = dim3(512, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = (cl == 16) ? cudaLaunchKernelEx(&cfg, k_batch_solve<16>, (const BatchItem*)d_items)
                             : cudaLaunchKernelEx(&cfg, k_batch_solve<8>, (const BatchItem*)d_items);
  if (e != cudaSuccess) {
    set_error("pmgb_batch_solve: launch: %s", cudaGetErrorString(e));
    cudaFreeAsync(d_items, st);
    cudaFreeAsync(d_out, st);
    return 0;
  }
  note_launches(1);
  std::vector<double> out((size_t)(2 + nlog) * n);
  CKM(cudaMemcpyAsync(out.data(), d_out, sizeof(double) * out.size(), cudaMemcpyDeviceToHost, st));
  // Dirichlet values back on the boundary (VfboundPMG, mgdrvd.c:557)
  for (int b = 0; b < n; b++) {
    pmgb_solver* s = solvers[b];
    launch_fbound(st, s->g, s->lev[0].x, s->gx, s->gy, s->gz);
  }
  note_launches(n);
  cudaFreeAsync(d_items, st);
  cudaFreeAsync(d_out, st);
  CKM(cudaStreamSynchronize(st));
  CKM(cudaGetLastError());
  int ok = 1;
  for (int b = 0; b < n; b++) {
    pmgb_solver* s = solvers[b];
    const double* o = out.data() + (size_t)(2 + nlog) * b;
    const int iters = (int)o[0];
    s->reslog.clear();
    for (int i = 0; i <= iters && i < nlog; i++) s->reslog.push_back(o[2 + i]);
    s->st.vcycles = iters;
    s->st.refinements = iters;
    s->st.newton_iters = 0;
    s->st.rel_residual = o[1];
    s->st.converged = (o[1] <= ((s->p.etol > 0.0) ? s->p.etol : 1.0e-6)) ? 1 : 0;
    s->st.coarse_method = 2;
    s->st.t_setup_ms = 0.0;
    s->st.t_solve_ms = 0.0;
    if (!(o[1] == o[1])) {
      set_error("pmgb_batch_solve: non-finite residual in calculation %d", b);
      ok = 0;
      continue;
    }
    s->solved = 1;
  }
  return ok;
}
