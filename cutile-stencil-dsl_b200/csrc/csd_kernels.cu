// Fixed (non-generated) kernels of libcsd: the standalone boundary fill.
//
// apply_boundary fills the halo of one array dimension by dimension, in
// order, like the reference's per-dimension slab copies
// (reference/stencil_ref.py:102-201, target_to_python.py:199-297), so corner
// cells end up with the composition of the per-dimension rules.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/csd.h"

extern "C" int csd_internal_fail(int code, const char* msg);
extern "C" unsigned long long csd_internal_ctx_id(void);

namespace {

// Source index along one dimension of a halo cell (the interior cell whose
// value it takes); interior indices map to themselves.
template <typename I>
__device__ __forceinline__ I fill_src(I i, I nd, I h, int bc) {
  if (i >= h && i < nd - h) return i;
  const bool high = i >= nd - h;
  const I k = high ? i - (nd - h) : i;  // layer 0 .. h-1
  if (bc == CSD_BC_NEUMANN) return high ? nd - h - 1 : h;
  if (bc == CSD_BC_PERIODIC) return high ? h + k : nd - 2 * h + k;
  return high ? nd - h - 1 - k : 2 * h - 1 - k;  // reflecting
}

// Fill every halo cell of a (d0, d1, d2) array in one launch.  The halo is
// enumerated as three disjoint boxes (dim-0 halo layers over the whole
// cross-section; dim-1 layers over the dim-0 interior; dim-2 layers over
// the dim-0 and dim-1 interior), and each cell maps every out-of-interior
// dimension to its source independently.  That equals the dimension-by-
// dimension slab copies of the reference fill (corners take the value of
// the mirrored interior corner) for all four conditions.  `I` is unsigned for
// arrays under 2^31 cells: decoding a cell takes two or four divisions, which
// in 64 bits were most of the kernel's time (periodic, 300 x 320 x 340 FP64,
// halo (1, 1, 16): 26 -> 19 us).
template <typename T, typename I>
__global__ void fill_halo_kernel(T* u, I d0, I d1, I d2, I h0, I h1, I h2, int bc, T value) {
  const I i0 = d0 - 2 * h0, i1 = d1 - 2 * h1;
  const I na = 2 * h0 * d1 * d2;
  const I nb = i0 * 2 * h1 * d2;
  const I nc = i0 * i1 * 2 * h2;
  const I total = na + nb + nc;
  const I step = (I)gridDim.x * blockDim.x;
  for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += step) {
    I a, b, c;
    if (e < na) {
      c = e % d2;
      const I t = e / d2;
      b = t % d1;
      const I l = t / d1;  // 0 .. 2h0-1
      a = l < h0 ? l : d0 - 2 * h0 + l;
    } else if (e < na + nb) {
      const I f = e - na;
      c = f % d2;
      const I t = f / d2;
      const I l = t % (2 * h1);
      a = h0 + t / (2 * h1);
      b = l < h1 ? l : d1 - 2 * h1 + l;
    } else {
      const I f = e - na - nb;
      const I l = f % (2 * h2);
      const I t = f / (2 * h2);
      b = h1 + t % i1;
      a = h0 + t / i1;
      c = l < h2 ? l : d2 - 2 * h2 + l;
    }
    const I dst = (a * d1 + b) * d2 + c;
    if (bc == CSD_BC_DIRICHLET) {
      u[dst] = value;
    } else {
      u[dst] = u[(fill_src(a, d0, h0, bc) * d1 + fill_src(b, d1, h1, bc)) * d2 +
                 fill_src(c, d2, h2, bc)];
    }
  }
}

template <typename T>
int apply_boundary_t(const csd_field* f, const int* halo, int bc, double value, cudaStream_t s) {
  long long n[3] = {1, 1, 1};
  int h3[3] = {0, 0, 0};
  const int off = 3 - f->ndim;
  for (int i = 0; i < f->ndim; ++i) {
    n[off + i] = f->shape[i];
    h3[off + i] = halo[i];
  }
  long long cells = 0, inner = 1;
  for (int d = 0; d < 3; ++d) {
    if (h3[d] < 0 || n[d] - 2LL * h3[d] < 1)
      return csd_internal_fail(CSD_EINVAL, "halo leaves no interior");
    if (h3[d] > 0 && bc != CSD_BC_DIRICHLET && n[d] - 2 * h3[d] < h3[d])
      return csd_internal_fail(CSD_EINVAL, "boundary fill needs an interior at least as wide as the halo");
    inner *= n[d] - 2LL * h3[d];
  }
  cells = n[0] * n[1] * n[2] - inner;
  if (cells == 0) return CSD_OK;
  long long blocks = (cells + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  T* u = reinterpret_cast<T*>(f->ptr);
  if (n[0] * n[1] * n[2] < (1ll << 31))
    fill_halo_kernel<T, unsigned><<<(int)blocks, 256, 0, s>>>(
        u, (unsigned)n[0], (unsigned)n[1], (unsigned)n[2], (unsigned)h3[0], (unsigned)h3[1],
        (unsigned)h3[2], bc, (T)value);
  else
    fill_halo_kernel<T, long long><<<(int)blocks, 256, 0, s>>>(u, n[0], n[1], n[2], h3[0], h3[1],
                                                               h3[2], bc, (T)value);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
  return CSD_OK;
}

}  // namespace

// The fill and reduction kernels index packed (C-contiguous) arrays.
static bool packed(const csd_field* f) {
  long long expect = 1;
  for (int i = f->ndim - 1; i >= 0; --i) {
    if (f->shape[i] != 1 && f->strides[i] != expect) return false;
    expect *= f->shape[i];
  }
  return true;
}

extern "C" int csd_apply_boundary(const csd_field* f, const int* halo, int bc, double value,
                                  void* stream) {
  if (!f || !halo || !f->ptr) return csd_internal_fail(CSD_EINVAL, "null argument");
  if (f->ndim < 1 || f->ndim > 3) return csd_internal_fail(CSD_EINVAL, "ndim must be 1-3");
  if (!packed(f)) return csd_internal_fail(CSD_EINVAL, "boundary fill needs a C-contiguous field");
  if (bc < CSD_BC_DIRICHLET || bc > CSD_BC_REFLECTING)
    return csd_internal_fail(CSD_EINVAL, "unknown boundary condition");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (f->dtype == CSD_DTYPE_F64) return apply_boundary_t<double>(f, halo, bc, value, s);
  if (f->dtype == CSD_DTYPE_F32) return apply_boundary_t<float>(f, halo, bc, value, s);
  return csd_internal_fail(CSD_EINVAL, "unsupported dtype");
}

// ---------------------------------------------------------------------------
// Bricked layout conversions
//
// A bricked array holds a (n0, n1, n2) array (1-3 dims, leading dims 1) as
// bricks of B^nd elements, bricks in row-major order over the brick grid
// (ceil(n / B) per dim) and each brick row-major inside: the reference's
// to_bricks reshape/transpose (multigpu_emitter.py:370-408), padded cells
// zero.  A warp takes a segment of one array row: its brick offset is worked
// out once, lanes run along X, and an element costs shifts and adds.  Bound by
// HBM: 300 x 320 x 370 FP64, B = 8, 284 MB each way: to_bricks 221 -> 107 us,
// from_bricks 177 -> 110 (one thread per element, with 64-bit divisions).
// ---------------------------------------------------------------------------
namespace {

constexpr int BRICK_SEG = 1024;   // elements of a row segment
constexpr int BRICK_SHORT = 64;   // longest row that is walked by elements

// TO: flat -> bricked over the padded rows (zeros past the array); else
// bricked -> flat over the array's rows.  r0 x r1 rows of r2 elements are
// walked; `I` counts their segments.
template <typename T, typename I, bool TO>
__global__ void __launch_bounds__(256) brick_rows_kernel(const T* __restrict__ src,
                                                         T* __restrict__ dst, long long n0,
                                                         long long n1, long long n2, I r0, I r1,
                                                         long long r2, int nd, int s,
                                                         long long nb1, long long nb2) {
  const long long m = (1ll << s) - 1;
  const I nseg = (I)((r2 + BRICK_SEG - 1) / BRICK_SEG);
  const I units = r0 * r1 * nseg;
  const int lane = threadIdx.x & 31;
  const I warps = (I)gridDim.x * (blockDim.x >> 5);
  for (I u = (I)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < units; u += warps) {
    const I row = u / nseg;
    const long long x0 = (long long)(u - row * nseg) * BRICK_SEG;
    const long long z = (long long)(row / r1), y = (long long)(row % r1);
    // element x of the row is at brow + ((x >> s) << (nd s)) + (x & m)
    long long brow = 0;
    if (nd == 3)
      brow = ((((z >> s) * nb1 + (y >> s)) * nb2) << (3 * s)) + ((z & m) << (2 * s)) +
             ((y & m) << s);
    else if (nd == 2)
      brow = (((y >> s) * nb2) << (2 * s)) + ((y & m) << s);
    const long long frow = (z * n1 + y) * n2;
    const bool in = z < n0 && y < n1;
    const int n = (int)min((long long)BRICK_SEG, r2 - x0);
    for (int k = lane; k < n; k += 128) {
      T v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long x = x0 + k + 32 * q;
        v[q] = T(0);
        if (k + 32 * q < n) {
          if (TO) {
            if (in && x < n2) v[q] = src[frow + x];
          } else {
            v[q] = src[brow + ((x >> s) << (nd * s)) + (x & m)];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long long x = x0 + k + 32 * q;
        if (k + 32 * q < n) {
          if (TO)
            dst[brow + ((x >> s) << (nd * s)) + (x & m)] = v[q];
          else
            dst[frow + x] = v[q];
        }
      }
    }
  }
}

// The same for rows up to BRICK_SHORT, which leave most of a warp's loads
// empty: a thread per element, `total` of them, in 32-bit arithmetic.  FP64,
// B = 8, to_bricks by elements / by rows: 400 x 500 x 8 8 / 41 us, x 32 23 /
// 49, x 64 46 / 55, x 96 67 / 65; 128 x 256 x 12 4 / 10.
template <typename T, typename I, bool TO>
__global__ void __launch_bounds__(256) brick_elems_kernel(const T* __restrict__ src,
                                                          T* __restrict__ dst, I n0, I n1, I n2,
                                                          I r1, I r2, I total, int nd, int s,
                                                          I nb1, I nb2) {
  const I m = ((I)1 << s) - 1;
  const I step = (I)gridDim.x * blockDim.x;
  for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += step) {
    const I row = e / r2, x = e - row * r2;
    const I z = row / r1, y = row - z * r1;
    I b = x;
    if (nd == 3)
      b = ((((z >> s) * nb1 + (y >> s)) * nb2 + (x >> s)) << (3 * s)) + ((z & m) << (2 * s)) +
          ((y & m) << s) + (x & m);
    else if (nd == 2)
      b = (((y >> s) * nb2 + (x >> s)) << (2 * s)) + ((y & m) << s) + (x & m);
    const I f = (z * n1 + y) * n2 + x;
    if (TO)
      dst[b] = z < n0 && y < n1 && x < n2 ? src[f] : T(0);
    else
      dst[f] = src[b];
  }
}

template <typename T, bool TO>
void launch_brick_rows(const void* src, void* dst, const long long n[3], const long long nb[3],
                       int nd, int s, cudaStream_t st) {
  long long r[3], padded = 1;   // rows walked; cells of the bricked buffer
  for (int i = 0; i < 3; ++i) {
    const long long whole = i >= 3 - nd ? nb[i] << s : n[i];
    r[i] = TO ? whole : n[i];
    padded *= whole;
  }
  const T* from = static_cast<const T*>(src);
  T* to = static_cast<T*>(dst);
  const long long total = r[0] * r[1] * r[2];
  if (r[2] <= BRICK_SHORT && padded < (1ll << 30)) {
    long long eblocks = (total + 255) / 256;
    if (eblocks > 148 * 32) eblocks = 148 * 32;
    brick_elems_kernel<T, unsigned, TO><<<(int)eblocks, 256, 0, st>>>(
        from, to, (unsigned)n[0], (unsigned)n[1], (unsigned)n[2], (unsigned)r[1], (unsigned)r[2],
        (unsigned)total, nd, s, (unsigned)nb[1], (unsigned)nb[2]);
    return;
  }
  const long long units = r[0] * r[1] * ((r[2] + BRICK_SEG - 1) / BRICK_SEG);
  long long blocks = (units + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (units < (1ll << 30))
    brick_rows_kernel<T, unsigned, TO><<<(int)blocks, 256, 0, st>>>(
        from, to, n[0], n[1], n[2], (unsigned)r[0], (unsigned)r[1], r[2], nd, s, nb[1], nb[2]);
  else
    brick_rows_kernel<T, unsigned long long, TO><<<(int)blocks, 256, 0, st>>>(
        from, to, n[0], n[1], n[2], (unsigned long long)r[0], (unsigned long long)r[1], r[2], nd,
        s, nb[1], nb[2]);
}

// (n0, n1, n2) view, bricked dimensionality and brick-grid extents of a field
int brick_geometry(const csd_field* f, int brick, long long n[3], long long nb[3], int* nd,
                   int* s) {
  if (!f || !f->ptr) return csd_internal_fail(CSD_EINVAL, "null field");
  if (f->ndim < 1 || f->ndim > 3) return csd_internal_fail(CSD_EINVAL, "ndim must be 1-3");
  if (brick < 2 || brick > 1024 || (brick & (brick - 1)))
    return csd_internal_fail(CSD_EINVAL, "brick size must be a power of two in [2, 1024]");
  if (!packed(f)) return csd_internal_fail(CSD_EINVAL, "the flat array must be C-contiguous");
  *nd = f->ndim;
  *s = 0;
  while ((1 << *s) < brick) ++*s;
  const int off = 3 - f->ndim;
  for (int i = 0; i < 3; ++i) n[i] = 1;
  for (int i = 0; i < f->ndim; ++i) n[off + i] = f->shape[i];
  for (int i = 0; i < 3; ++i) nb[i] = (i < off) ? 1 : (n[i] + brick - 1) / brick;
  return CSD_OK;
}

}  // namespace

extern "C" long long csd_bricked_elems(const long long* shape, int ndim, int brick) {
  if (!shape || ndim < 1 || ndim > 3 || brick < 1) return -1;
  long long e = 1;
  for (int i = 0; i < ndim; ++i) e *= ((shape[i] + brick - 1) / brick) * brick;
  return e;
}

extern "C" int csd_to_bricks(const csd_field* flat, int brick, void* bricked, void* stream) {
  long long n[3], nb[3];
  int nd = 0, s = 0;
  int rc = brick_geometry(flat, brick, n, nb, &nd, &s);
  if (rc) return rc;
  if (!bricked) return csd_internal_fail(CSD_EINVAL, "null bricked buffer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (flat->dtype == CSD_DTYPE_F64)
    launch_brick_rows<double, true>(flat->ptr, bricked, n, nb, nd, s, st);
  else if (flat->dtype == CSD_DTYPE_F32)
    launch_brick_rows<float, true>(flat->ptr, bricked, n, nb, nd, s, st);
  else
    return csd_internal_fail(CSD_EINVAL, "unsupported dtype");
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CSD_OK : csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
}

extern "C" int csd_from_bricks(const void* bricked, int brick, const csd_field* flat, void* stream) {
  long long n[3], nb[3];
  int nd = 0, s = 0;
  int rc = brick_geometry(flat, brick, n, nb, &nd, &s);
  if (rc) return rc;
  if (!bricked) return csd_internal_fail(CSD_EINVAL, "null bricked buffer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (flat->dtype == CSD_DTYPE_F64)
    launch_brick_rows<double, false>(bricked, flat->ptr, n, nb, nd, s, st);
  else if (flat->dtype == CSD_DTYPE_F32)
    launch_brick_rows<float, false>(bricked, flat->ptr, n, nb, nd, s, st);
  else
    return csd_internal_fail(CSD_EINVAL, "unsupported dtype");
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CSD_OK : csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// FP64 reductions over the interior of a field (mass, energy, residual, max)
//
// Deterministic: interior rows are cut into segments of RED_SEG elements, and
// pass 1 gives CTA c of C the segments [c*S/C, (c+1)*S/C), its warps taking
// them in turn.  A lane adds its elements in RED_ACC independent sums in a
// fixed order, and a fixed-shape tree combines lanes and warps.  Every sum
// carries the rounding errors of its additions (Knuth's two-sum) beside it, so
// the result is the exact sum of the FP64 terms but for its last rounding, in
// nearly all cases; a CTA hands both words on in two of the `nblocks` partials
// (C = nblocks / 2; a single CTA rounds into one).  Pass 2 (one CTA) combines
// them the same way.  The result depends on nblocks, never on scheduling.
// Bound by HBM: RED_ILP loads per lane and 32 warps per SM keep enough of them
// in flight, and the seven additions per element stay behind them (sum of a
// 300 x 320 x 340 FP64 interior, 261 MB: 60 us, the difference of two
// 99; with a row at a time per CTA of 256 threads 388 and 449; a 1-D row,
// formerly one CTA's, 2^24 FP64: 10.9 ms -> 36 us).
// ---------------------------------------------------------------------------
namespace {

constexpr int RED_THREADS = 1024, RED_THREADS2 = 256;   // pass 1, pass 2
constexpr int RED_ILP = 8, RED_ACC = 4;   // loads in flight, sums per lane
constexpr int RED_SEG = 1024;   // elements of a row segment

template <int OP>
constexpr bool kRedMax = OP == CSD_RED_MAXABS || OP == CSD_RED_DIFF_MAXABS;

// A sum and the rounding errors made in it (maxima: the value alone).
struct RedSum {
  double v, err;
};

template <int OP>
__device__ __forceinline__ RedSum red_add(RedSum a, double b) {
  if (kRedMax<OP>) return {(a.v != a.v || a.v > b) ? a.v : b, 0.0};
  const double s = __dadd_rn(a.v, b);
  const double t = __dsub_rn(s, a.v);
  return {s, __dadd_rn(a.err, __dadd_rn(__dsub_rn(a.v, __dsub_rn(s, t)), __dsub_rn(b, t)))};
}
template <int OP>
__device__ __forceinline__ RedSum red_combine(RedSum a, RedSum b) {
  RedSum s = red_add<OP>(a, b.v);
  if (!kRedMax<OP>) s.err = __dadd_rn(s.err, b.err);
  return s;
}
// The sum with its errors added back; an infinity or NaN (whose errors mean
// nothing) as it is.
template <int OP>
__device__ __forceinline__ double red_value_of(RedSum a) {
  return kRedMax<OP> || !isfinite(a.v) ? a.v : __dadd_rn(a.v, a.err);
}

template <int OP, int THREADS>
__device__ __forceinline__ RedSum red_block(RedSum v, RedSum* sh) {
  // fixed-shape tree: warp shuffles, then the warp totals in order
  for (int o = 16; o > 0; o >>= 1) {
    const RedSum w = {__shfl_down_sync(0xffffffffu, v.v, o), __shfl_down_sync(0xffffffffu, v.err, o)};
    v = red_combine<OP>(v, w);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  RedSum t = {0.0, 0.0};
  if (threadIdx.x == 0) {
    t = sh[0];
    for (int w = 1; w < THREADS / 32; ++w) t = red_combine<OP>(t, sh[w]);
  }
  return t;
}

// The reduced term of one element.
template <int OP>
__device__ __forceinline__ double red_term(double va, double vb) {
  if (OP == CSD_RED_SUM) return va;
  if (OP == CSD_RED_SUMSQ) return __dmul_rn(va, va);
  if (OP == CSD_RED_MAXABS) return fabs(va);
  const double d = __dsub_rn(va, vb);
  return OP == CSD_RED_DIFF_SUMSQ ? __dmul_rn(d, d) : fabs(d);
}

template <typename T, int OP>
__global__ void __launch_bounds__(RED_THREADS, 1) reduce_pass1(const T* a, const T* b,
                                                               long long d0, long long d1,
                                                               long long d2, int h0, int h1,
                                                               int h2, double* partials,
                                                               int pairs) {
  __shared__ RedSum sh[RED_THREADS / 32];
  constexpr bool kDiff = OP == CSD_RED_DIFF_SUMSQ || OP == CSD_RED_DIFF_MAXABS;
  const long long ny = d1 - 2 * h1, nx = d2 - 2 * h2;
  const long long nseg = (nx + RED_SEG - 1) / RED_SEG;
  const long long segs = (d0 - 2 * h0) * ny * nseg;
  const long long s0 = segs * blockIdx.x / gridDim.x, s1 = segs * (blockIdx.x + 1) / gridDim.x;
  const int lane = threadIdx.x & 31;
  constexpr int NW = RED_THREADS / 32;
  // (z, y, seg) of the warp's first segment and the step to its next one
  long long i = s0 + (threadIdx.x >> 5);
  long long seg = i % nseg, z = i / nseg / ny, y = i / nseg % ny;
  const long long dseg = NW % nseg, dz = NW / nseg / ny, dy = NW / nseg % ny;
  RedSum acc[RED_ACC];
#pragma unroll
  for (int k = 0; k < RED_ACC; ++k) acc[k] = {0.0, 0.0};
  for (; i < s1; i += NW) {
    const long long base = ((z + h0) * d1 + y + h1) * d2 + h2 + seg * RED_SEG;
    const int n = (int)min((long long)RED_SEG, nx - seg * RED_SEG);
    const T* pa = a + base;
    const T* pb = kDiff ? b + base : nullptr;
    int x = lane;
    for (; x + 32 * (RED_ILP - 1) < n; x += 32 * RED_ILP) {
      T va[RED_ILP], vb[RED_ILP];
#pragma unroll
      for (int k = 0; k < RED_ILP; ++k) {
        va[k] = pa[x + 32 * k];
        vb[k] = kDiff ? pb[x + 32 * k] : T(0);
      }
#pragma unroll
      for (int k = 0; k < RED_ILP; ++k)
        acc[k % RED_ACC] =
            red_add<OP>(acc[k % RED_ACC], red_term<OP>((double)va[k], (double)vb[k]));
    }
#pragma unroll
    for (int k = 0; k < RED_ILP; ++k)
      if (x + 32 * k < n)
        acc[k % RED_ACC] = red_add<OP>(
            acc[k % RED_ACC],
            red_term<OP>((double)pa[x + 32 * k], kDiff ? (double)pb[x + 32 * k] : 0.0));
    seg += dseg;
    y += dy;
    z += dz;
    if (seg >= nseg) {
      seg -= nseg;
      ++y;
    }
    if (y >= ny) {
      y -= ny;
      ++z;
    }
  }
#pragma unroll
  for (int w = RED_ACC / 2; w > 0; w >>= 1)
#pragma unroll
    for (int k = 0; k < w; ++k) acc[k] = red_combine<OP>(acc[k], acc[k + w]);
  const RedSum t = red_block<OP, RED_THREADS>(acc[0], sh);
  if (threadIdx.x == 0) {
    if (pairs) {
      partials[2 * blockIdx.x] = t.v;
      partials[2 * blockIdx.x + 1] = t.err;
    } else {
      partials[blockIdx.x] = red_value_of<OP>(t);
    }
  }
}

template <int OP>
__global__ void __launch_bounds__(RED_THREADS2) reduce_pass2(const double* partials, int n,
                                                             int pairs, double* result) {
  __shared__ RedSum sh[RED_THREADS2 / 32];
  RedSum acc = {0.0, 0.0};
  for (int i = threadIdx.x; i < n; i += RED_THREADS2) {
    const RedSum p = {pairs ? partials[2 * i] : partials[i], pairs ? partials[2 * i + 1] : 0.0};
    acc = red_combine<OP>(acc, p);
  }
  const RedSum t = red_block<OP, RED_THREADS2>(acc, sh);
  if (threadIdx.x == 0) *result = red_value_of<OP>(t);
}

template <typename T, int OP>
int reduce_t(const csd_field* a, const csd_field* b, const long long d[3], const int h[3],
             double* partials, int nblocks, double* result, cudaStream_t s) {
  const T* pa = reinterpret_cast<const T*>(a->ptr);
  const T* pb = b ? reinterpret_cast<const T*>(b->ptr) : nullptr;
  const int pairs = nblocks >= 2, ctas = pairs ? nblocks / 2 : nblocks;
  reduce_pass1<T, OP><<<ctas, RED_THREADS, 0, s>>>(pa, pb, d[0], d[1], d[2], h[0], h[1], h[2],
                                                   partials, pairs);
  reduce_pass2<OP><<<1, RED_THREADS2, 0, s>>>(partials, ctas, pairs, result);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CSD_OK : csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
}

template <typename T>
int reduce_dispatch(int op, const csd_field* a, const csd_field* b, const long long d[3],
                    const int h[3], double* partials, int nblocks, double* result,
                    cudaStream_t s) {
  switch (op) {
    case CSD_RED_SUM: return reduce_t<T, CSD_RED_SUM>(a, b, d, h, partials, nblocks, result, s);
    case CSD_RED_SUMSQ: return reduce_t<T, CSD_RED_SUMSQ>(a, b, d, h, partials, nblocks, result, s);
    case CSD_RED_MAXABS: return reduce_t<T, CSD_RED_MAXABS>(a, b, d, h, partials, nblocks, result, s);
    case CSD_RED_DIFF_SUMSQ:
      return reduce_t<T, CSD_RED_DIFF_SUMSQ>(a, b, d, h, partials, nblocks, result, s);
    case CSD_RED_DIFF_MAXABS:
      return reduce_t<T, CSD_RED_DIFF_MAXABS>(a, b, d, h, partials, nblocks, result, s);
  }
  return csd_internal_fail(CSD_EINVAL, "unknown reduction");
}

}  // namespace

extern "C" int csd_reduce(const csd_field* a, const csd_field* b, const int* halo, int op,
                          double* partials, int nblocks, double* result, void* stream) {
  if (!a || !a->ptr || !halo || !partials || !result || nblocks < 1)
    return csd_internal_fail(CSD_EINVAL, "null argument or nblocks < 1");
  if (a->ndim < 1 || a->ndim > 3) return csd_internal_fail(CSD_EINVAL, "ndim must be 1-3");
  if (!packed(a)) return csd_internal_fail(CSD_EINVAL, "reductions need C-contiguous fields");
  const bool diff = (op == CSD_RED_DIFF_SUMSQ || op == CSD_RED_DIFF_MAXABS);
  if (diff) {
    if (!b || !b->ptr || b->dtype != a->dtype || b->ndim != a->ndim)
      return csd_internal_fail(CSD_EINVAL, "difference reductions need a second field like the first");
    if (!packed(b)) return csd_internal_fail(CSD_EINVAL, "reductions need C-contiguous fields");
    for (int i = 0; i < a->ndim; ++i)
      if (b->shape[i] != a->shape[i]) return csd_internal_fail(CSD_EINVAL, "field shapes differ");
  }
  long long d[3] = {1, 1, 1};
  int h[3] = {0, 0, 0};
  const int off = 3 - a->ndim;
  for (int i = 0; i < a->ndim; ++i) {
    d[off + i] = a->shape[i];
    h[off + i] = halo[i];
    if (d[off + i] - 2 * h[off + i] < 1) return csd_internal_fail(CSD_EINVAL, "empty interior");
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a->dtype == CSD_DTYPE_F64)
    return reduce_dispatch<double>(op, a, diff ? b : nullptr, d, h, partials, nblocks, result, s);
  if (a->dtype == CSD_DTYPE_F32)
    return reduce_dispatch<float>(op, a, diff ? b : nullptr, d, h, partials, nblocks, result, s);
  return csd_internal_fail(CSD_EINVAL, "unsupported dtype");
}

// ---------------------------------------------------------------------------
// Allocation-free reduction entry point.
//
// For callers that must not allocate device memory themselves: a host
// process whose device memory is entirely owned by another allocator (a
// framework's caching pool, a fixed up-front reservation), or a loop that
// cannot afford cudaMalloc's implicit device synchronisation between steps.
// They cannot provide the `partials` scratch csd_reduce needs, so this
// variant keeps its per-block partials in a file-scope device array of fixed
// size, which every device holds from the moment the library's kernels load
// until the process exits.
// ---------------------------------------------------------------------------
#include <mutex>

namespace {

// One partial per block of pass 1 (8 KB).  Shared by every call: pass 1
// overwrites each of the `nblocks` entries it uses before pass 2 reads them,
// so nothing has to be cleared between calls, but two calls that run at the
// same time on the GPU (different streams) race on these entries.
static __device__ __align__(256) double g_noalloc_partials[CSD_NOALLOC_MAX_BLOCKS];

// Device address of g_noalloc_partials per device ordinal (the host-side
// name is only a stand-in for the symbol, never a device pointer), with the id
// of the context it was looked up in: after cudaDeviceReset the device gets a
// new context, the old address is void, and the next call looks it up again.
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {nullptr};
unsigned long long g_noalloc_ctx[64] = {0};

int noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return csd_internal_fail(CSD_ENODEV, cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return csd_internal_fail(CSD_EINVAL, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  const unsigned long long ctx = csd_internal_ctx_id();
  if (!g_noalloc_ptr[dev] || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (e != cudaSuccess)
      return csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<double*>(p);
    g_noalloc_ctx[dev] = csd_internal_ctx_id();  // the lookup may have created the context
  }
  *out = g_noalloc_ptr[dev];
  return CSD_OK;
}

}  // namespace

extern "C" int csd_reduce_noalloc(const csd_field* a, const csd_field* b, const int* halo, int op,
                                  int nblocks, double* result, void* stream) {
  if (nblocks < 1 || nblocks > CSD_NOALLOC_MAX_BLOCKS)
    return csd_internal_fail(CSD_EINVAL,
                             "csd_reduce_noalloc: nblocks must be 1..1024 (the static scratch "
                             "holds 1024 partials)");
  if (!a || !a->ptr || !halo || !result)
    return csd_internal_fail(CSD_EINVAL, "csd_reduce_noalloc: null argument");
  double* partials = nullptr;
  int rc = noalloc_scratch(&partials);
  if (rc) return rc;
  return csd_reduce(a, b, halo, op, partials, nblocks, result, stream);
}

// ---------------------------------------------------------------------------
// CFL time-step control for batched solvers: dt[i] = cfl * scale[i] / smax[i]
// (smax = the per-grid maximum signal speed from a max-reduction launch),
// then smax[i] = 0 so the next reduction starts afresh.  One thread per grid.
// ---------------------------------------------------------------------------
namespace {
__global__ void cfl_update_kernel(int n, double* smax, const double* scale, double cfl,
                                  double dt_max, double* dt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double s = smax[i];
  double v = (s > 0.0) ? __ddiv_rn(__dmul_rn(cfl, scale[i]), s) : dt_max;
  if (v > dt_max) v = dt_max;
  dt[i] = v;
  smax[i] = 0.0;
}
}  // namespace

extern "C" int csd_cfl_update(int n, double* smax, const double* scale, double cfl, double dt_max,
                              double* dt, void* stream) {
  if (n < 1 || !smax || !scale || !dt) return csd_internal_fail(CSD_EINVAL, "bad cfl arguments");
  cfl_update_kernel<<<(n + 127) / 128, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      n, smax, scale, cfl, dt_max, dt);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CSD_OK : csd_internal_fail(CSD_ELAUNCH, cudaGetErrorString(e));
}
