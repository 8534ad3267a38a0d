/* Kernels of the per-call entry points (the reference's energy routines one
 * call at a time): bead energies.
 *
 * A call is small (1 to 64 positions against one box), so its time is a
 * launch, a wait and the longest chain of dependent work of one warp. The
 * kernels therefore spread one call over as many SMs as it has work for and
 * take their inputs as kernel parameters instead of through device copies.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "rgpu_device.cuh"
#include "rgpu_engine.h"
#include "rgpu_grid.cuh"

namespace cg = cooperative_groups;

#define POINT_WARPS 8          /* warps of a CTA of the FP64 kernel */
#define POINT_CLUSTER 8        /* largest cluster of CTAs of one position */
#define POINT_MIXED_WARPS 8    /* warps the mixed kernel's chunks are cut for */

/* Loads a descriptor copy into shared memory. */
__device__ __forceinline__ void load_sys(RgpuSys *dst, const RgpuSys *src)
{
  const uint32_t *s = (const uint32_t *)src;
  uint32_t *d = (uint32_t *)dst;
  for (int i = threadIdx.x; i < (int)(sizeof(RgpuSys) / 4); i += blockDim.x) d[i] = s[i];
  __syncthreads();
}

/* The framework terms of a bead from the energy grids (GRID framework
 * model): lanes 0..7 of warp 0 return them, the other lanes take part in the
 * shuffles. */
__device__ __forceinline__ void grid_terms(const RgpuSys &S, const BeadPos &b, int lane, double &g, double &gq)
{
  const double x[3] = {b.x, b.y, b.z};
  g = rgpu_grid_value8(S.grid[b.atom], S.grid_geom, x, lane & 7, lane < 8);
  gq = 0.0;
  if (S.use_coul_grid) {
    const double q = S.mol_q[b.atom];
    gq = q * rgpu_grid_value8(S.coul_grid, S.coul_geom, x, lane & 7, lane < 8 && q != 0.0, false);
  }
}

/* Energies of P bead positions (P <= RGPU_MAX_POS), given as FP64 xyz with
 * the molecule-atom index of each bead, FP64. out[p*4 + k], ov[p] (both in
 * mapped host memory).
 *
 * fw_grid (the GRID framework model, with the system's grids set): the
 * framework VDW energy of a bead is its atom's energy-grid value and the
 * framework real-space charge energy its charge times the Coulomb-grid value
 * (zero without a Coulomb grid: an uncharged molecule), with no framework
 * pairs, as CalculateFrameworkVDWEnergyAtPosition and
 * CalculateFrameworkChargeEnergyAtPosition do when the model is GRID
 * (src/framework_energy.c:73-77, :195-198) and the move differences
 * (:4893-4894, :5437-5438). A grid value sets no overlap flag: the
 * reference's grid branches set none.
 *
 * One cluster per position: its CTAs' warps share the framework tiles and
 * the adsorbate records evenly (contiguous ranges of the bit-reversed tile
 * order, each a sample of the whole cell), each warp runs the tile walk of
 * unit_tiles_fp64, and the sums meet in the first CTA's shared memory in rank
 * and warp order. What bounds it is the chain of one warp (descriptor load,
 * cull, two or three tile passes, one queue evaluation), not arithmetic.
 * Measured, whole call from Python: 20 positions in a 1536-atom CO2 box 34 us,
 * 139 us with one CTA of 8 warps walking all atoms of all positions; one
 * position in 3456 uncharged atoms 29 us (46 us). */
__global__ void __launch_bounds__(32 * POINT_WARPS) k_points_fp64(const RgpuSys *sysp, const AdsRec64 *ads, int nads,
                                                                 const __grid_constant__ RgpuPoints in, int pair_check,
                                                                 int fw_grid, double *out, int *ov)
{
  __shared__ RgpuSys S;
  __shared__ BeadPos b;
  __shared__ int queue[POINT_WARPS * 64];
  __shared__ double red[POINT_WARPS][4];
  __shared__ int rov[POINT_WARPS];
  __shared__ double part[POINT_CLUSTER][4];   /* the CTAs' sums (first CTA) */
  __shared__ int pov[POINT_CLUSTER];
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  cl.barrier_arrive();                        /* every CTA runs before the remote stores below */
  const int p = blockIdx.x / csize, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  load_sys(&S, sysp);
  if (threadIdx.x == 0) bead_set(b, S, in.xyz[p][0], in.xyz[p][1], in.xyz[p][2], in.atom[p], in.excl[p]);
  __syncthreads();
  const bool check = p < pair_check, grids = fw_grid && S.use_grid;
  double e[4] = {0.0, 0.0, 0.0, 0.0};
  int o = 0, nin = 0, nch = 0, nvis = 0;
  const int gw = rank * POINT_WARPS + w, ngw = csize * POINT_WARPS;
  if (!grids) {
    const int t0 = S.ntile * gw / ngw, t1 = S.ntile * (gw + 1) / ngw;   /* ntile <= 2^20 */
    if (S.triclinic)
      unit_tiles_fp64<true>(S, S.fw32, S.fw64t, S.tiles, t0, t1, b, check, e[0], e[1], o, nin, nch, nvis, queue + 64 * w);
    else
      unit_tiles_fp64<false>(S, S.fw32, S.fw64t, S.tiles, t0, t1, b, check, e[0], e[1], o, nin, nch, nvis, queue + 64 * w);
  }
  /* adsorbate atoms, 32 at a time, from the last warp down: the first ones
   * have the longer shares where the tiles do not divide evenly */
  for (int j = 32 * (ngw - 1 - gw); j < nads; j += 32 * ngw) {
    const int hi = min(j + 32, nads);
    if (S.triclinic) unit_ads_fp64<true>(S, ads, b, j, hi, b.excl, check, e[2], e[3], o, nin, nch, nvis);
    else unit_ads_fp64<false>(S, ads, b, j, hi, b.excl, check, e[2], e[3], o, nin, nch, nvis);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) e[k] = warp_sum(e[k]);
  o = warp_or(o);
  if (lane == 0) {
    for (int k = 0; k < 4; k++) red[w][k] = e[k];
    rov[w] = o;
  }
  double g = 0.0, gq = 0.0;
  if (grids && rank == 0 && w == 0) grid_terms(S, b, lane, g, gq);
  __syncthreads();
  cl.barrier_wait();
  if (w == 0) {
    /* lane k < 4: this CTA's sum of term k, to the first CTA */
    if (lane < 4) {
      double t = 0.0;
      for (int q = 0; q < POINT_WARPS; q++) t += red[q][lane];
      *cl.map_shared_rank(&part[rank][lane], 0) = t;
    }
    const int any = warp_or(lane < POINT_WARPS ? rov[lane] : 0);
    if (lane == 0) *cl.map_shared_rank(&pov[rank], 0) = any;
  }
  cl.sync();
  if (rank == 0 && threadIdx.x < 4) {
    double t = 0.0;
    for (int q = 0; q < csize; q++) t += part[q][threadIdx.x];
    if (grids && threadIdx.x < 2) t = threadIdx.x ? gq : g;
    out[4 * p + threadIdx.x] = t;
    if (threadIdx.x == 0) {
      int any = 0;
      for (int q = 0; q < csize; q++) any |= pov[q];
      ov[p] = any;
    }
  }
}

/* As k_points_fp64 on the mixed path: one CTA per position and one warp per
 * unit of eval_plan's cut for POINT_MIXED_WARPS warps (framework chunks, then
 * adsorbate chunks), so that each FP32 sum runs over the same pairs in the
 * same order whatever the number of positions a call shares the GPU with.
 * Bound by the one warp that walks all tiles of a position when a call has
 * five positions or more. 64 positions in 4096 atoms: 48 us a call (137 us
 * with all units on one CTA). */
__global__ void __launch_bounds__(64 * POINT_MIXED_WARPS) k_points_mixed(const RgpuSys *sysp, const int4 *ads, int nads,
                                                                        const __grid_constant__ RgpuPoints in,
                                                                        EvalPlan pl, int pair_check, int fw_grid,
                                                                        double *out, int *ov)
{
  __shared__ RgpuSys S;
  __shared__ BeadPos b;
  __shared__ float qr2[2 * POINT_MIXED_WARPS * 64], qq[2 * POINT_MIXED_WARPS * 64];
  __shared__ int qt[2 * POINT_MIXED_WARPS * 64];
  __shared__ double red[2 * POINT_MIXED_WARPS][2];
  __shared__ int rov[2 * POINT_MIXED_WARPS];
  const int p = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, per = pl.cf + pl.ca;
  load_sys(&S, sysp);
  if (threadIdx.x == 0) bead_set(b, S, in.xyz[p][0], in.xyz[p][1], in.xyz[p][2], in.atom[p], in.excl[p]);
  __syncthreads();
  const bool check = p < pair_check;
  if (w < per) {
    float av = 0.0f, ac = 0.0f;
    int o = 0, nin = 0, nch = 0, nvis = 0;
    float *r2 = qr2 + 64 * w, *q = qq + 64 * w;
    int *t = qt + 64 * w;
    if (w < pl.cf) {
      const int lo = (int)((unsigned)(S.ntile * w) / (unsigned)pl.cf);
      const int hi = (int)((unsigned)(S.ntile * (w + 1)) / (unsigned)pl.cf);
      if (S.triclinic)
        unit_tiles_mixed<true>(S, S.fw32, S.tiles, lo, hi, b, check, av, ac, o, nin, nch, nvis, r2, q, t);
      else
        unit_tiles_mixed<false>(S, S.fw32, S.tiles, lo, hi, b, check, av, ac, o, nin, nch, nvis, r2, q, t);
    } else {
      const int c = w - pl.cf;
      const int lo = (int)((unsigned)(nads * c) / (unsigned)pl.ca), hi = (int)((unsigned)(nads * (c + 1)) / (unsigned)pl.ca);
      if (S.triclinic) unit_ads_mixed<true>(S, ads, b, lo, hi, b.excl, check, av, ac, o, nin, nch, nvis, r2, q, t);
      else unit_ads_mixed<false>(S, ads, b, lo, hi, b.excl, check, av, ac, o, nin, nch, nvis, r2, q, t);
    }
    const double ev = (double)warp_sum(av), eq = (double)warp_sum(ac);
    o = warp_or(o);
    if (lane == 0) {
      red[w][0] = ev;
      red[w][1] = eq;
      rov[w] = o;
    }
  }
  double g = 0.0, gq = 0.0;
  if (fw_grid && S.use_grid && w == 0) grid_terms(S, b, lane, g, gq);
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[4] = {0.0, 0.0, 0.0, 0.0};
    int any = 0;
    for (int c = 0; c < per; c++) {
      const int k = c < pl.cf ? 0 : 2;
      r[k] += red[c][0];
      r[k + 1] += red[c][1];
      any |= rov[c];
    }
    if (fw_grid && S.use_grid) {
      r[0] = g;
      r[1] = gq;
    }
    for (int k = 0; k < 4; k++) out[4 * p + k] = r[k];
    ov[p] = any;
  }
}

/* ntile: the system's framework tiles (0 with the GRID framework model) */
cudaError_t rgpu_points_launch(int mixed, const RgpuSys *d_sys, const void *d_ads, int nads, const RgpuPoints &in, int P,
                               int ntile, int pair_check, int fw_grid, double *d_out, int *d_ov, cudaStream_t st)
{
  if (P < 1 || P > RGPU_MAX_POS) return cudaErrorInvalidValue;
  if (mixed) {
    EvalPlan pl = eval_plan(P, ntile, nads, POINT_MIXED_WARPS, 8 * RGPU_MAX_POS, 2);
    const int per = pl.cf + pl.ca;
    k_points_mixed<<<P, 32 * (per > 1 ? per : 1), 0, st>>>(d_sys, (const int4 *)d_ads, nads, in, pl, pair_check, fw_grid,
                                                         d_out, d_ov);
    return cudaGetLastError();
  }
  /* CTAs per position: as many (1, 2, 4 or 8, the portable cluster size) as
   * keep every CTA on an SM of its own (148 SMs), but none without a tile for
   * every second warp or adsorbate atoms of its own: below that a CTA only
   * adds to the cluster's barriers */
  int c = POINT_CLUSTER;
  while (c > 1 && (c * P > 148 || (16 * (c - 1) >= ntile && 32 * POINT_WARPS * (c - 1) >= nads))) c >>= 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(P * c), 1, 1);
  cfg.blockDim = dim3(32 * POINT_WARPS, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_points_fp64, d_sys, (const AdsRec64 *)d_ads, nads, in, pair_check, fw_grid, d_out,
                            d_ov);
}
