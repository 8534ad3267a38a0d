/* Energy-grid construction and tricubic lookup.
 *
 * Build: MakeGrid (src/grids.c:431-690) with the per-point derivatives of
 * CalculateDerivativesAtPositionVDW (src/framework_hessian.c:63-109) and the
 * LJ branch of PotentialThirdDerivative (src/potentials.c:10959-10990),
 * computed in FP64 and stored as FP32 like the reference. One thread per grid
 * point; a block covers a 4x8x8 tile and stages, chunk by chunk, only the
 * images of framework atoms within cutoff + tile radius of the tile centre in
 * shared memory, so each thread visits ~1/7 of the framework at 0.1 A spacing
 * and forms no minimum image.
 *
 * Device layout is point-major: grid[((i*(ny+1) + j)*(nz+1) + k)*8 + m], so
 * the 8 values of a corner are one 32-byte sector and a lookup gathers eight
 * sectors (the reference's file is plane-major; the Python side converts).
 *
 * Lookup: InterpolateVDWGrid (src/grids.c:979-1077). The reference forms the
 * 64 tricubic coefficients with the Lekien-Marsden matrix and evaluates the
 * polynomial; the same interpolant is evaluated here as the tensor product of
 * 1D cubic Hermite bases over the stored value and derivatives (FP64 math on
 * the FP32 data, as in the reference).
 */
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>

#include "rgpu_device.cuh"
#include "rgpu_engine.h"
#include "rgpu_grid.cuh"

#define GRID_TX 4
#define GRID_TY 8
#define GRID_TZ 8
#define GRID_THREADS (GRID_TX * GRID_TY * GRID_TZ)

struct GridParams {
  int npts[3];
  double size[3], shift[3], delta[3];
  RgpuLJ lj[RGPU_MAX_FWTYPES];
};

#define GRID_STAGE (2 * GRID_THREADS)   /* staged images of one round of atoms */

/* 1/x by two Newton iterations from the hardware's approximation (relative
 * error 2^-20 or better, squared by each); below 1e-60, where a grid point
 * sits on an atom, by the division */
__device__ __forceinline__ double grid_reciprocal(double x)
{
  if (x < 1e-60) return 1.0 / x;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

/* Staged images: position and framework charge (Coulomb) or LJ shift, and
 * the LJ parameters 4 eps, sigma^2 */
struct GridStage {
  double4 xyz[GRID_STAGE];
  double2 lj[GRID_STAGE];
  int wcount[GRID_THREADS / 32];
};

/* Stages the images of atoms base .. base + GRID_THREADS within reach of the
 * tile about (cx, cy, cz), those numbered s0 .. s0 + GRID_STAGE in thread
 * order; returns how many there are in all. Contains a block barrier; the
 * caller puts one before the stage is read. */
template <bool COUL, bool IMAGES>
__device__ __forceinline__ int grid_stage(const RgpuSys &S, const GridParams &gp, GridStage &st, int base, int s0,
                                          double cx, double cy, double cz, double rcut2)
{
  const int a = base + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  /* this thread's atom: the images within reach, as a mask over the 8
   * choices of nearest or next image along the cell vectors */
  unsigned keep = 0;
  double4 f = make_double4(0, 0, 0, 0);
  double d[3] = {0, 0, 0}, step[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (a < S.nfw) {
    f = S.fw64[a];
    if (!IMAGES) {
      keep = 1;
    } else {
      const double c[3] = {cx - f.x, cy - f.y, cz - f.z};
      if (!S.triclinic) {
#pragma unroll
        for (int r = 0; r < 3; r++) {
          d[r] = c[r] - S.box[r] * rgpu_round(c[r] * S.inv_box[r]);
          step[r][r] = d[r] > 0.0 ? -S.box[r] : S.box[r];
        }
      } else {
        double t[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
          const double u = S.hinv[3 * r] * c[0] + S.hinv[3 * r + 1] * c[1] + S.hinv[3 * r + 2] * c[2];
          t[r] = u - rgpu_round(u);
        }
#pragma unroll
        for (int r = 0; r < 3; r++) {
          d[r] = S.hm[3 * r] * t[0] + S.hm[3 * r + 1] * t[1] + S.hm[3 * r + 2] * t[2];
#pragma unroll
          for (int q = 0; q < 3; q++) step[q][r] = t[q] > 0.0 ? -S.hm[3 * r + q] : S.hm[3 * r + q];
        }
      }
#pragma unroll
      for (int m = 0; m < 8; m++) {
        double r2 = 0.0;
#pragma unroll
        for (int r = 0; r < 3; r++) {
          const double v = d[r] + (m & 1 ? step[0][r] : 0.0) + (m & 2 ? step[1][r] : 0.0) + (m & 4 ? step[2][r] : 0.0);
          r2 += v * v;
        }
        if (r2 < rcut2) keep |= 1u << m;
      }
    }
  }
  const int mine = __popc(keep);
  int incl = mine;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int y = __shfl_up_sync(RGPU_FULL, incl, s);
    if (lane >= s) incl += y;
  }
  if (lane == 31) st.wcount[w] = incl;
  __syncthreads();
  int pos = incl - mine - s0, nsel = 0;
#pragma unroll
  for (int q = 0; q < GRID_THREADS / 32; q++) {
    if (q < w) pos += st.wcount[q];
    nsel += st.wcount[q];
  }
  if (keep) {
    int seg = 0;
    while (seg + 1 < S.nseg && a >= S.seg_start[seg + 1]) seg++;
    const double2 lj = make_double2(gp.lj[seg].eps4, gp.lj[seg].sig2);
    const double v = COUL ? f.w : gp.lj[seg].shift;
    for (unsigned m = keep; m; m &= m - 1, pos++) {
      if (pos < 0 || pos >= GRID_STAGE) continue;
      const int c = __ffs(m) - 1;
      double4 g = make_double4(f.x, f.y, f.z, v);
      if (IMAGES) {
        g.x = cx - (d[0] + (c & 1 ? step[0][0] : 0.0) + (c & 2 ? step[1][0] : 0.0) + (c & 4 ? step[2][0] : 0.0));
        g.y = cy - (d[1] + (c & 1 ? step[0][1] : 0.0) + (c & 2 ? step[1][1] : 0.0) + (c & 4 ? step[2][1] : 0.0));
        g.z = cz - (d[2] + (c & 1 ? step[0][2] : 0.0) + (c & 2 ? step[1][2] : 0.0) + (c & 4 ? step[2][2] : 0.0));
      }
      st.xyz[pos] = g;
      if (!COUL) st.lj[pos] = lj;
    }
  }
  return nsel;
}

/* COUL = false: the LJ grid of one probe pseudo-atom (gp.lj by framework
 * segment). COUL = true: the real-space Ewald (Coulomb) grid of a unit probe
 * charge, CalculateDerivativesAtPositionReal (src/framework_hessian.c:111-180)
 * with the framework charges, capped where the value exceeds the overlap
 * criterion or a framework atom is closer than 1 A (src/grids.c:656-668).
 *
 * The kernel is bound by FP64 instructions, one (point, staged image) pair at a
 * time, so a pair is kept short: the images are staged about the tile's centre
 * (no rounding to the nearest image per pair), LJ has one reciprocal by
 * Newton's iteration, the Coulomb term one rsqrt and one exponential, which
 * its erfc = exp(-x^2) erfcx(x) shares. 64 and 80 registers keep 32 and 24
 * warps on an SM; with the compiler's choice (94, 116) there were 16 and the
 * dependent FP64 instructions left the pipe half idle. 102^3 points over 4096
 * atoms in a 40 A cell, LJ: 2.27 ms, 12.9 TFLOP/s at 60 FLOP a pair inside the
 * cut-off (5.77 ms with a rounding per pair and axis and four divisions; 3.06
 * at 94 registers). 78^3 points over 1536 atoms, Coulomb: 4.01 ms (6.77; 4.71).
 * IMAGES: every image of an atom within reach of the tile is, along each cell
 * vector, its nearest to the tile's centre or the next one
 * (cutoff + tile radius below every perpendicular width); all of those within
 * reach are staged, and at most one of an atom's is inside the cut-off of a
 * point, because the widths are at least twice the cut-off. Otherwise (grids
 * coarser than about 2 A) the atoms are staged as they are and each pair takes
 * its minimum image. */
template <bool COUL, bool IMAGES>
__global__ void __launch_bounds__(GRID_THREADS, COUL ? 3 : 4) k_grid_build(const RgpuSys *sysp, GridParams gp, float *grid)
{
  __shared__ GridStage st;
  const RgpuSys &S = *sysp;
  const int nx = gp.npts[0] + 1, ny = gp.npts[1] + 1, nz = gp.npts[2] + 1;
  const int tilesz = (nz + GRID_TZ - 1) / GRID_TZ, tilesy = (ny + GRID_TY - 1) / GRID_TY;
  int b = blockIdx.x;
  const int tk = b % tilesz; b /= tilesz;
  const int tj = b % tilesy; b /= tilesy;
  const int ti = b;
  const int lk = threadIdx.x % GRID_TZ, lj = (threadIdx.x / GRID_TZ) % GRID_TY, li = threadIdx.x / (GRID_TZ * GRID_TY);
  const int i = ti * GRID_TX + li, j = tj * GRID_TY + lj, k = tk * GRID_TZ + lk;
  const bool valid = i < nx && j < ny && k < nz;
  const double px = i * gp.size[0] / gp.npts[0] + gp.shift[0];
  const double py = j * gp.size[1] / gp.npts[1] + gp.shift[1];
  const double pz = k * gp.size[2] / gp.npts[2] + gp.shift[2];
  /* tile centre and radius for culling */
  const double cx = (ti * GRID_TX + 0.5 * (GRID_TX - 1)) * gp.size[0] / gp.npts[0] + gp.shift[0];
  const double cy = (tj * GRID_TY + 0.5 * (GRID_TY - 1)) * gp.size[1] / gp.npts[1] + gp.shift[1];
  const double cz = (tk * GRID_TZ + 0.5 * (GRID_TZ - 1)) * gp.size[2] / gp.npts[2] + gp.shift[2];
  const double hx = 0.5 * (GRID_TX - 1) * gp.delta[0], hy = 0.5 * (GRID_TY - 1) * gp.delta[1],
               hz = 0.5 * (GRID_TZ - 1) * gp.delta[2];
  const double rcut = sqrt(S.rc2) + sqrt(hx * hx + hy * hy + hz * hz) + 1e-6;
  const double rc2 = S.rc2;
  double o[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  double rmin2 = 1e300;
  const double alpha = S.alpha, a2 = alpha * alpha, two_a_sqrtpi = 2.0 * alpha / sqrt(M_PI), coulomb = S.coulomb;
  const int nfw = S.nfw;
  int s0 = 0;
  for (int base = 0; base < nfw;) {
    const int nsel = grid_stage<COUL, IMAGES>(S, gp, st, base, s0, cx, cy, cz, rcut * rcut);
    __syncthreads();
    const int n = min(nsel - s0, GRID_STAGE);
    for (int q = 0; valid && q < n; q++) {
      const double4 g = st.xyz[q];
      double dx = px - g.x, dy = py - g.y, dz = pz - g.z;
      if (!IMAGES) {
        if (S.triclinic) {
          rgpu_min_image_tri(S, dx, dy, dz);
        } else {
          dx -= S.box[0] * rgpu_round(dx * S.inv_box[0]);
          dy -= S.box[1] * rgpu_round(dy * S.inv_box[1]);
          dz -= S.box[2] * rgpu_round(dz * S.inv_box[2]);
        }
      }
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 < rc2) {
        double U, DF, DDF, DDDF;
        if (COUL) {
          /* f(r) = K q erfc(a r) / r; DF = f'/r, DDF = (f'' - f'/r)/r^2,
           * DDDF = the r-part of the mixed third derivative */
          rmin2 = fmin(rmin2, r2);
          const double ri = rsqrt(r2), r = r2 * ri, ri2 = ri * ri, ar2 = a2 * r2;
          const double x2 = exp(-ar2), e = x2 * erfcx(alpha * r), gr = two_a_sqrtpi * r * x2;
          const double c1 = coulomb * g.w * ri, c3 = c1 * ri2, c5 = c3 * ri2;
          U = c1 * e;
          DF = -c3 * (gr + e);
          DDF = c5 * (gr * (3.0 + 2.0 * ar2) + 3.0 * e);
          DDDF = -c5 * ri2 * (gr * (15.0 + ar2 * (10.0 + 4.0 * ar2)) + 15.0 * e);
        } else {
          const double2 P = st.lj[q];
          const double i2 = grid_reciprocal(r2), i4 = i2 * i2;
          double r3 = P.y * i2;
          r3 = r3 * r3 * r3;
          const double v = P.x * r3;
          U = v * (r3 - 1.0) - g.w;
          DF = v * i2 * (6.0 - 12.0 * r3);
          DDF = v * i4 * (168.0 * r3 - 48.0);
          DDDF = v * (i4 * i4) * (480.0 - 2688.0 * r3);
        }
        const double xy = dx * dy;
        o[0] += U;
        o[1] += dx * DF;
        o[2] += dy * DF;
        o[3] += dz * DF;
        o[4] += DDF * xy;
        o[5] += DDF * (dx * dz);
        o[6] += DDF * (dy * dz);
        o[7] += DDDF * (xy * dz);
      }
    }
    __syncthreads();
    /* as a rule one pass a round; more where it has more images than the stage holds */
    s0 += GRID_STAGE;
    if (s0 >= nsel) {
      s0 = 0;
      base += GRID_THREADS;
    }
  }
  if (!valid) return;
  /* cap, src/grids.c:546-563 (Coulomb: also within 1 A of an atom, :656-668) */
  if (o[0] > S.overlap || (COUL && rmin2 < 1.0)) {
    o[0] = 2.0 * S.overlap;
    for (int c = 1; c <= 3; c++) {
      if (o[c] > S.overlap) o[c] = S.overlap;
      if (o[c] < -S.overlap) o[c] = -S.overlap;
    }
    o[4] = o[5] = o[6] = o[7] = 0.0;
  }
  const double dx = gp.delta[0], dy = gp.delta[1], dz = gp.delta[2];
  float4 v0 = make_float4((float)o[0], (float)o[1] * (float)dx, (float)o[2] * (float)dy, (float)o[3] * (float)dz);
  float4 v1 = make_float4((float)o[4] * (float)(dx * dy), (float)o[5] * (float)(dx * dz),
                          (float)o[6] * (float)(dy * dz), (float)o[7] * (float)(dx * dy * dz));
  float4 *dst = (float4 *)(grid + (((size_t)i * ny + j) * nz + k) * 8);
  dst[0] = v0;
  dst[1] = v1;
}

/* lj[s]: LJ parameters of the probe pseudo-atom with framework segment s;
 * nullptr: the Coulomb grid of a unit probe charge. reach: the box's smallest
 * perpendicular width less the cut-off, the largest tile radius for which
 * atoms are staged as images. */
cudaError_t rgpu_grid_build_launch(const RgpuSys *d_sys, const RgpuLJ *lj, double reach, const int npts[3],
                                   const double size[3], const double shift[3], float *d_grid, cudaStream_t st)
{
  GridParams gp = {};
  for (int c = 0; c < 3; c++) {
    gp.npts[c] = npts[c];
    gp.size[c] = size[c];
    gp.shift[c] = shift[c];
    gp.delta[c] = size[c] / (double)npts[c];
  }
  for (int s = 0; lj && s < RGPU_MAX_FWTYPES; s++) gp.lj[s] = lj[s];
  const int nx = npts[0] + 1, ny = npts[1] + 1, nz = npts[2] + 1;
  const long long blocks = (long long)((nx + GRID_TX - 1) / GRID_TX) * ((ny + GRID_TY - 1) / GRID_TY) *
                           ((nz + GRID_TZ - 1) / GRID_TZ);
  if (blocks > 2147483647LL) return cudaErrorInvalidValue;
  const double h[3] = {0.5 * (GRID_TX - 1) * gp.delta[0], 0.5 * (GRID_TY - 1) * gp.delta[1],
                       0.5 * (GRID_TZ - 1) * gp.delta[2]};
  const bool images = sqrt(h[0] * h[0] + h[1] * h[1] + h[2] * h[2]) < reach - 1e-3;
  if (lj) {
    if (images) k_grid_build<false, true><<<(unsigned)blocks, GRID_THREADS, 0, st>>>(d_sys, gp, d_grid);
    else k_grid_build<false, false><<<(unsigned)blocks, GRID_THREADS, 0, st>>>(d_sys, gp, d_grid);
  } else {
    if (images) k_grid_build<true, true><<<(unsigned)blocks, GRID_THREADS, 0, st>>>(d_sys, gp, d_grid);
    else k_grid_build<true, false><<<(unsigned)blocks, GRID_THREADS, 0, st>>>(d_sys, gp, d_grid);
  }
  return cudaGetLastError();
}

/* One thread per point. The block's positions come through shared memory, so
 * that they are read once, in order, also from mapped host memory, where the
 * kernel is bound by the 32 bytes a point that cross PCIe (else by the eight
 * 32-byte corners). */
#define INTERP_THREADS 256

__global__ void __launch_bounds__(INTERP_THREADS) k_grid_interp(const float *grid, RgpuGridGeom ip, int n, const double *xyz,
                                                              double *out)
{
  __shared__ double sx[3 * INTERP_THREADS];
  const int base = blockIdx.x * INTERP_THREADS, m = min(n - base, INTERP_THREADS);
  for (int i = threadIdx.x; i < 3 * m; i += INTERP_THREADS) sx[i] = xyz[3 * (size_t)base + i];
  __syncthreads();
  const int q = threadIdx.x;
  if (q < m) {
    const double p[3] = {sx[3 * q], sx[3 * q + 1], sx[3 * q + 2]};
    out[base + q] = rgpu_grid_value(grid, ip, p);
  }
}

cudaError_t rgpu_grid_interp_launch(const float *d_grid, const int npts[3], const double size[3],
                                    const double shift[3], const double cell[3], int n, const double *d_xyz,
                                    double *d_out, cudaStream_t st)
{
  RgpuGridGeom ip;
  memset(&ip, 0, sizeof ip);   /* a rectangular cell (tri = 0) */
  for (int c = 0; c < 3; c++) {
    ip.npts[c] = npts[c];
    ip.size[c] = size[c];
    ip.shift[c] = shift[c];
    ip.cell[c] = cell[c];
    ip.icell[c] = 1.0 / cell[c];
    ip.isize[c] = 1.0 / size[c];
  }
  if (n <= 0) return cudaSuccess;
  k_grid_interp<<<(n + INTERP_THREADS - 1) / INTERP_THREADS, INTERP_THREADS, 0, st>>>(d_grid, ip, n, d_xyz, d_out);
  return cudaGetLastError();
}

/* Grid files store the 8 values as planes ([m][i][j][k], src/grids.c:734-738);
 * the device layout is point-major (8 floats per point). One thread per
 * point: the plane reads (or writes) of neighbouring threads are contiguous,
 * and the point's 8 floats move as two 16-byte words. */
__global__ void k_grid_planes_to_points(const float *__restrict__ planes, long long npt, float *__restrict__ points)
{
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npt; p += (long long)gridDim.x * blockDim.x) {
    float v[8];
#pragma unroll
    for (int m = 0; m < 8; m++) v[m] = planes[m * npt + p];
    float4 *dst = (float4 *)(points + 8 * p);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

__global__ void k_grid_points_to_planes(const float *__restrict__ points, long long npt, float *__restrict__ planes)
{
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npt; p += (long long)gridDim.x * blockDim.x) {
    const float4 *src = (const float4 *)(points + 8 * p);
    const float4 a = src[0], b = src[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int m = 0; m < 8; m++) planes[m * npt + p] = v[m];
  }
}

static unsigned transpose_blocks(long long npt)
{
  /* at most 8 CTAs of 256 per SM-count multiple: 148 SMs x 8 */
  const long long want = (npt + 255) / 256;
  return (unsigned)std::min<long long>(want, 148LL * 8);
}

cudaError_t rgpu_grid_planes_to_points_launch(const float *d_planes, long long npt, float *d_points, cudaStream_t st)
{
  if (npt <= 0) return cudaSuccess;
  k_grid_planes_to_points<<<transpose_blocks(npt), 256, 0, st>>>(d_planes, npt, d_points);
  return cudaGetLastError();
}

cudaError_t rgpu_grid_points_to_planes_launch(const float *d_points, long long npt, float *d_planes, cudaStream_t st)
{
  if (npt <= 0) return cudaSuccess;
  k_grid_points_to_planes<<<transpose_blocks(npt), 256, 0, st>>>(d_points, npt, d_planes);
  return cudaGetLastError();
}
