/* Kernels of the per-call entry points (the reference's energy routines one
 * call at a time): bead energies, total energies, structure factors, the Ewald
 * Fourier difference and its acceptance, adsorbate records.
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
 * Measured, whole call from Python: 20 positions in a 1536-atom CO2 box 25 us
 * (the kernel 13.8, cold, under the profiler; 140 us a call with one CTA of 8
 * warps walking all atoms of all positions); one position in 3456 uncharged
 * atoms 20 us (kernel 9.0; 47 us). */
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

/* As k_points_fp64 on the mixed path, whose FP32 sums run over the same pairs in
 * the same order whatever the number of positions a call shares the GPU with:
 * the units of eval_plan's cut for POINT_MIXED_WARPS warps (framework chunks,
 * then adsorbate chunks), one warp's sum each. One CTA per position.
 * k_points_mixed gives each unit a warp; it serves calls of up to four
 * positions, whose framework is cut into chunks. From five positions on a
 * position's framework is one unit (k_points_mixed_long). */
__global__ void __launch_bounds__(64 * POINT_MIXED_WARPS) k_points_mixed(const RgpuSys *sysp, const int4 *ads, int nads,
                                                                        const __grid_constant__ RgpuPoints in,
                                                                        EvalPlan pl, int pair_check, int fw_grid,
                                                                        double *out, int *ov)
{
  __shared__ RgpuSys S;
  __shared__ BeadPos b;
  __shared__ __align__(8) float queue[2 * POINT_MIXED_WARPS * RGPU_QUEUE_FLOATS];
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
    float *mem = queue + RGPU_QUEUE_FLOATS * w;
    if (w < pl.cf) {
      const int lo = (int)((unsigned)(S.ntile * w) / (unsigned)pl.cf);
      const int hi = (int)((unsigned)(S.ntile * (w + 1)) / (unsigned)pl.cf);
      if (S.triclinic)
        unit_tiles_mixed<true>(S, S.fw32, S.tiles, lo, hi, b, check, av, ac, o, nin, nch, nvis, mem);
      else
        unit_tiles_mixed<false>(S, S.fw32, S.tiles, lo, hi, b, check, av, ac, o, nin, nch, nvis, mem);
    } else {
      const int c = w - pl.cf;
      const int lo = (int)((unsigned)(nads * c) / (unsigned)pl.ca), hi = (int)((unsigned)(nads * (c + 1)) / (unsigned)pl.ca);
      if (S.triclinic) unit_ads_mixed<true>(S, ads, b, lo, hi, b.excl, check, av, ac, o, nin, nch, nvis, mem);
      else unit_ads_mixed<false>(S, ads, b, lo, hi, b.excl, check, av, ac, o, nin, nch, nvis, mem);
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

/* One framework unit per position, its pairs in the order of one warp's queue
 * (ascending tiles and atoms; pair j is added by lane j mod 32) but found and
 * formed by all warps: each culls and tests an eighth of the tiles into a list
 * of its own, all threads form the lists' pair terms into one sequence, and
 * one warp adds that up. A ninth warp takes the adsorbates meanwhile. A
 * list that overflows sends the position through one warp's queue. Bound by the
 * chain of steps. 64 positions in 4096 atoms: 27 us a call from Python (the
 * kernel 17.4, cold, under the profiler), 40 us with one warp walking all tiles
 * of a position. */
#define LONG_WARPS 8
#define LONG_LIST 256          /* pairs of one warp; an eighth of a 12 A sphere's atoms at 0.09 / A^3 is 81 */

struct LongSmem {
  RgpuSys S;
  BeadPos b;
  float2 list[LONG_WARPS][LONG_LIST];   /* {r2, charge} */
  unsigned char type[LONG_WARPS][LONG_LIST];
  float2 term[LONG_WARPS * LONG_LIST];  /* {LJ, charge} of the sequence */
  __align__(8) float queue[2 * RGPU_QUEUE_FLOATS];
  int count[LONG_WARPS], ov[LONG_WARPS + 1];
  double red[2][2];
};

template <bool TRI>
__device__ __forceinline__ int long_list(const RgpuSys &S, int t0, int t1, const BeadPos &b, float2 *list,
                                         unsigned char *type)
{
  const int lane = threadIdx.x & 31, half = lane >> 4, hl = lane & 15;
  const unsigned below = (1u << lane) - 1u;
  const float rc2 = S.rc2f;
  int n = 0;
  for (int tb = t0; tb < t1; tb += 32) {
    bool vis = false;
    int tn = 0;
    if (tb + lane < t1) {
      const TileRec tr = S.tiles[tb + lane];
      tn = tr.c.w;
      vis = tile_visible<TRI>(S, tr, b, rc2);
    }
    unsigned m = __ballot_sync(RGPU_FULL, vis);
    while (m) {
      const unsigned mm = m & (m - (unsigned)half);
      m &= m - 1;
      m &= m - 1;
      const int mine = __ffs(mm) - 1;
      const int nt = __shfl_sync(RGPU_FULL, tn, mine & 31);
      const bool live = mine >= 0 && hl < nt;
      int4 f = make_int4(0, 0, 0, 0);
      if (live) f = S.fw32[(size_t)(tb + mine) * RGPU_TILE + hl];
      float dx, dy, dz;
      if (!TRI) {
        dx = __int2float_rn(f.x - b.xi) * S.fix_scale[0];
        dy = __int2float_rn(f.y - b.yi) * S.fix_scale[1];
        dz = __int2float_rn(f.z - b.zi) * S.fix_scale[2];
      } else {
        rgpu_fix_to_cart_tri(S, f.x - b.xi, f.y - b.yi, f.z - b.zi, dx, dy, dz);
      }
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const bool in = live && r2 < rc2;
      const unsigned bal = __ballot_sync(RGPU_FULL, in);
      const int p = n + __popc(bal & below);
      if (in && p < LONG_LIST) {
        list[p] = make_float2(r2, __int_as_float(f.w));
        type[p] = (unsigned char)(f.z & 3);
      }
      n += __popc(bal);
    }
  }
  return n;
}

__global__ void __launch_bounds__(32 * (LONG_WARPS + 1)) k_points_mixed_long(const RgpuSys *sysp, const int4 *ads, int nads,
                                                                            const __grid_constant__ RgpuPoints in,
                                                                            int pair_check, double *out, int *ov)
{
  __shared__ LongSmem sm;
  const RgpuSys &S = sm.S;
  const int p = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  load_sys(&sm.S, sysp);
  if (threadIdx.x == 0) bead_set(sm.b, S, in.xyz[p][0], in.xyz[p][1], in.xyz[p][2], in.atom[p], in.excl[p]);
  __syncthreads();
  const BeadPos &b = sm.b;
  const bool check = p < pair_check;
  float av = 0.0f, ac = 0.0f;
  int o = 0, nin = 0, nch = 0, nvis = 0;
  if (w < LONG_WARPS) {
    const int t0 = S.ntile * w / LONG_WARPS, t1 = S.ntile * (w + 1) / LONG_WARPS;
    const int n = S.triclinic ? long_list<true>(S, t0, t1, b, sm.list[w], sm.type[w])
                              : long_list<false>(S, t0, t1, b, sm.list[w], sm.type[w]);
    if (lane == 0) sm.count[w] = n;
  } else if (nads > 0) {
    float *mem = sm.queue + RGPU_QUEUE_FLOATS;
    if (S.triclinic) unit_ads_mixed<true>(S, ads, b, 0, nads, b.excl, check, av, ac, o, nin, nch, nvis, mem);
    else unit_ads_mixed<false>(S, ads, b, 0, nads, b.excl, check, av, ac, o, nin, nch, nvis, mem);
  }
  __syncthreads();
  int n = 0, most = 0;
  for (int q = 0; q < LONG_WARPS; q++) {
    n += sm.count[q];
    most = max(most, sm.count[q]);
  }
  const bool listed = most <= LONG_LIST;
  if (listed && w < LONG_WARPS) {
    const RgpuLJf *P = S.ljf_bf[b.atom];
    const float qa = S.mol_qf[b.atom] * S.coulombf, alpha = S.alphaf, thr = (float)S.overlap;
    const bool charged = S.fw_charged && qa != 0.0f;
    for (int j = threadIdx.x; j < n; j += 32 * LONG_WARPS) {
      int q = 0, i = j;
      while (i >= sm.count[q]) i -= sm.count[q++];
      const float2 e = sm.list[q][i];
      float u = 0.0f, uc = 0.0f;
      pair_mixed_queued(P, e.x, e.y, charged, qa, alpha, check, thr, u, uc, o, nch, sm.type[q][i]);
      sm.term[j] = make_float2(u, uc);
    }
  }
  if (listed) __syncthreads();
  if (w == 0) {
    if (listed) {
#pragma unroll 4
      for (int j = lane; j < n; j += 32) {
        const float2 t = sm.term[j];
        av += t.x;
        ac += t.y;
      }
    } else if (S.triclinic) {
      unit_tiles_mixed<true>(S, S.fw32, S.tiles, 0, S.ntile, b, check, av, ac, o, nin, nch, nvis, sm.queue);
    } else {
      unit_tiles_mixed<false>(S, S.fw32, S.tiles, 0, S.ntile, b, check, av, ac, o, nin, nch, nvis, sm.queue);
    }
  }
  o = warp_or(o);
  if (lane == 0) sm.ov[w] = o;
  if (w == 0 || w == LONG_WARPS) {
    const double ev = (double)warp_sum(av), eq = (double)warp_sum(ac);
    if (lane == 0) {
      sm.red[w != 0][0] = ev;
      sm.red[w != 0][1] = eq;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int any = 0;
    for (int q = 0; q <= LONG_WARPS; q++) any |= sm.ov[q];
    for (int k = 0; k < 4; k++) out[4 * p + k] = sm.red[k >> 1][k & 1];
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
    /* one framework unit a position and a tile for every warp: from 300 to 4096
     * atoms 23 to 27 us a call of 8 to 64 positions, 25 to 40 with a warp per unit */
    if (pl.cf == 1 && pl.ca <= 1 && ntile >= LONG_WARPS) {
      k_points_mixed_long<<<P, 32 * (LONG_WARPS + 1), 0, st>>>(d_sys, (const int4 *)d_ads, nads, in, pair_check, d_out, d_ov);
      return cudaGetLastError();
    }
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

/* ------------------------------------------------------------------------ */
/* Pair sums of a whole configuration, FP64: over all adsorbate atoms as
 * positions (their own molecule left out), and the intramolecular exclusion
 * energy of every molecule (the sum K qa qb erf(alpha r)/r over its charged
 * pairs, src/ewald.c:7312-7330). CTA c leaves {host VDW, host real, adsorbate
 * VDW, adsorbate real, exclusion} of its atoms and molecules in out[5 c ..]
 * (mapped host memory). Each CTA takes every gridDim-th atom, a warp per
 * quarter of the framework tiles and of the adsorbate records, so that a
 * loaded box fills the GPU in one launch. 408 atoms in 4096: 22.9 us under the
 * profiler, cold, a warp's chain of tile passes with the FP64 pipe 15 % busy (4.5
 * ms in seven launches of one CTA before). */
#define TOTAL_WARPS 4

__global__ void __launch_bounds__(32 * TOTAL_WARPS) k_total_pairs(const RgpuSys *sysp, const AdsRec64 *ads, int nads,
                                                                 int fw_grid, double *out)
{
  __shared__ RgpuSys S;
  __shared__ BeadPos b;
  __shared__ int queue[TOTAL_WARPS * 64];
  __shared__ double red[TOTAL_WARPS][5];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  load_sys(&S, sysp);
  const bool grids = fw_grid && S.use_grid;
  const int t0 = S.ntile * w / TOTAL_WARPS, t1 = S.ntile * (w + 1) / TOTAL_WARPS;
  double e[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  int o = 0, nin = 0, nch = 0, nvis = 0;
  for (int p = blockIdx.x; p < nads; p += gridDim.x) {
    if (threadIdx.x == 0) {
      const AdsRec64 r = ads[p];
      bead_set(b, S, r.x, r.y, r.z, (int)(r.tag & 15), (int)(r.tag >> 4));
    }
    __syncthreads();
    if (!grids) {
      if (S.triclinic)
        unit_tiles_fp64<true>(S, S.fw32, S.fw64t, S.tiles, t0, t1, b, false, e[0], e[1], o, nin, nch, nvis, queue + 64 * w);
      else
        unit_tiles_fp64<false>(S, S.fw32, S.fw64t, S.tiles, t0, t1, b, false, e[0], e[1], o, nin, nch, nvis, queue + 64 * w);
    } else if (w == 0) {
      double g, gq;
      grid_terms(S, b, lane, g, gq);
      if (lane == 0) {
        e[0] += g;
        e[1] += gq;
      }
    }
    const int lo = nads * w / TOTAL_WARPS, hi = nads * (w + 1) / TOTAL_WARPS;
    if (S.triclinic) unit_ads_fp64<true>(S, ads, b, lo, hi, b.excl, false, e[2], e[3], o, nin, nch, nvis);
    else unit_ads_fp64<false>(S, ads, b, lo, hi, b.excl, false, e[2], e[3], o, nin, nch, nvis);
    __syncthreads();
  }
  if (S.ewald && S.mol_charged)
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m * S.natom < nads; m += gridDim.x * blockDim.x) {
      const AdsRec64 *x = ads + m * S.natom;
      for (int i = 0; i < S.natom - 1; i++)
        for (int j = i + 1; j < S.natom; j++) {
          const double qq = S.mol_q[i] * S.mol_q[j];
          if (qq == 0.0) continue;
          const double dx = x[i].x - x[j].x, dy = x[i].y - x[j].y, dz = x[i].z - x[j].z;
          const double r = sqrt(dx * dx + dy * dy + dz * dz);
          e[4] += S.coulomb * qq * erf(S.alpha * r) / r;
        }
    }
#pragma unroll
  for (int k = 0; k < 5; k++) e[k] = warp_sum(e[k]);
  if (lane == 0)
    for (int k = 0; k < 5; k++) red[w][k] = e[k];
  __syncthreads();
  if (threadIdx.x < 5) {
    double t = 0.0;
    for (int q = 0; q < TOTAL_WARPS; q++) t += red[q][threadIdx.x];
    out[5 * blockIdx.x + threadIdx.x] = t;
  }
}

cudaError_t rgpu_total_pairs_launch(const RgpuSys *d_sys, const void *d_ads, int nads, int fw_grid, double *d_out,
                                    int *ctas, cudaStream_t st)
{
  *ctas = nads < RGPU_TOTAL_CTAS ? nads : RGPU_TOTAL_CTAS;
  if (nads <= 0) return cudaSuccess;
  k_total_pairs<<<*ctas, 32 * TOTAL_WARPS, 0, st>>>(d_sys, (const AdsRec64 *)d_ads, nads, fw_grid, d_out);
  return cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Structure factors S(k) = sum_i q_i exp(i k.r_i), FP64.
 *
 * One thread per wave vector. exp(i k.r) is the product of one phase per axis:
 * a CTA tabulates exp(2 pi i n f) of its atoms' fractional coordinates f for
 * n = 0 .. kmax, SK_ATOMS atoms at a time, so a (wave vector, atom) pair costs
 * three shared-memory reads and 10 FMAs instead of a sincospi. The atoms are
 * cut into SK_PARTS parts (every SK_PARTS-th table of atoms), which the CTAs of a
 * cluster share; S(k) is the sum of the parts' sums in order, so it has the
 * same bits however many CTAs a kernel gives to it.
 * Bound by latency (the table and its barriers, one atom after the other): the
 * FP64 pipe is 13 to 19 % busy. Measured under the profiler, cold: 408 atoms,
 * about 2600 wave vectors 15.6 us, the 4096 charges of a framework 94 us, once
 * a system (103 us and more with one sincospi per pair and one thread looping
 * over all atoms). */
#define SK_THREADS 256
#define SK_ATOMS 16
#define SK_KMAX 20             /* rgpu_system_create's limit on kmax */
#define SK_PARTS 8             /* the largest cluster */

struct SkSmem {
  double2 tab[SK_ATOMS][3][SK_KMAX + 1];
  double q[SK_ATOMS];
  union {
    double2 part[SK_PARTS][SK_THREADS];       /* the parts' sums (first CTA) */
    double red[72];
  };
};

static_assert(sizeof(SkSmem) <= 48 * 1024, "more than a launch's default shared memory");

/* exp(2 pi i n f) for n < 0 is the conjugate */
__device__ __forceinline__ double2 sk_phase(const double2 *t, int n)
{
  const double2 v = t[n < 0 ? -n : n];
  return make_double2(v.x, n < 0 ? -v.y : v.y);
}

/* Sum for wave vector kv (live: this thread has one) over part `part` of n
 * atoms at xyz with charges q (by atom) or S.mol_q (by atom of the molecule). All
 * threads call. */
__device__ __forceinline__ double2 sk_sum(const RgpuSys &S, SkSmem &sm, const double *xyz, const double *q, int n, int part,
                                          char4 kv, bool live)
{
  const int km = max(S.kmax[0], max(S.kmax[1], S.kmax[2])) + 1, na = S.natom;
  double re = 0.0, im = 0.0;
  for (int base = SK_ATOMS * part; base < n; base += SK_ATOMS * SK_PARTS) {
    const int m = min(SK_ATOMS, n - base);
    for (int e = threadIdx.x; e < m * 3 * km; e += SK_THREADS) {
      const int h = e % km, sa = e / km, axis = sa % 3, a = sa / 3;
      const double *x = xyz + 3 * (base + a);
      const double f = S.triclinic ? rgpu_frac(S, axis, x[0], x[1], x[2]) : x[axis] * S.inv_box[axis];
      double sn, cs;
      sincospi(2.0 * (h * f), &sn, &cs);
      sm.tab[a][axis][h] = make_double2(cs, sn);
    }
    for (int a = threadIdx.x; a < m; a += SK_THREADS) sm.q[a] = q ? q[base + a] : S.mol_q[(base + a) % na];
    __syncthreads();
    if (live)
      for (int a = 0; a < m; a++) {
        const double2 x = sk_phase(sm.tab[a][0], kv.x), y = sk_phase(sm.tab[a][1], kv.y), z = sk_phase(sm.tab[a][2], kv.z);
        const double xr = x.x * y.x - x.y * y.y, xi = x.x * y.y + x.y * y.x, qa = sm.q[a];
        re += qa * (xr * z.x - xi * z.y);
        im += qa * (xr * z.y + xi * z.x);
      }
    __syncthreads();
  }
  return make_double2(re, im);
}

/* sk[k] of n atoms. With `out` (mapped host memory) the S(k) is the
 * adsorbates' and block x leaves {sum kf |S|^2, sum kf Re(S_fw^* S)} of its
 * wave vectors in out[2 x ..]. */
__global__ void __launch_bounds__(SK_THREADS) k_structure_factor(const RgpuSys *sysp, const double *xyz, const double *q,
                                                                int n, double2 *sk, double *out)
{
  extern __shared__ __align__(16) unsigned char smem[];
  SkSmem &sm = *(SkSmem *)smem;
  const RgpuSys &S = *sysp;
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank(), blk = blockIdx.x / csize;
  cl.barrier_arrive();
  const int k = blk * SK_THREADS + threadIdx.x;
  const bool live = k < S.nk;
  const char4 kv = live ? S.kvec[k] : make_char4(0, 0, 0, 0);
  cl.barrier_wait();
  for (int c = rank; c < SK_PARTS; c += csize) {
    const double2 v = sk_sum(S, sm, xyz, q, n, c, kv, live);
    *cl.map_shared_rank(&sm.part[c][threadIdx.x], 0) = v;
  }
  cl.sync();
  if (rank) return;
  double2 t = make_double2(0.0, 0.0);
  for (int c = 0; c < SK_PARTS; c++) {
    t.x += sm.part[c][threadIdx.x].x;
    t.y += sm.part[c][threadIdx.x].y;
  }
  __syncthreads();
  double ea = 0.0, eh = 0.0;
  if (live) {
    sk[k] = t;
    if (out) {
      const double kf = S.kfactor[k];
      const double2 sf = S.sk_fw[k];
      ea = kf * (t.x * t.x + t.y * t.y);
      eh = kf * (sf.x * t.x + sf.y * t.y);
    }
  }
  if (!out) return;
  block_sum2(ea, eh, sm.red);
  if (threadIdx.x == 0) {
    out[2 * blk] = ea;
    out[2 * blk + 1] = eh;
  }
}

/* S_ads(k) of every system of an engine from its positions (the batched
 * upload): block (x, y) = wave vectors x * SK_THREADS.. of system y */
__global__ void __launch_bounds__(SK_THREADS) k_upload_sk(const RgpuSys *systems)
{
  extern __shared__ __align__(16) unsigned char smem[];
  SkSmem &sm = *(SkSmem *)smem;
  const RgpuSys &S = systems[blockIdx.y];
  const int k = blockIdx.x * SK_THREADS + threadIdx.x;
  if (blockIdx.x * SK_THREADS >= S.nk) return;
  const bool live = k < S.nk;
  const char4 kv = live ? S.kvec[k] : make_char4(0, 0, 0, 0);
  double2 t = make_double2(0.0, 0.0);
  for (int c = 0; c < SK_PARTS; c++) {
    const double2 v = sk_sum(S, sm, S.ads_xyz, nullptr, *S.nmol * S.natom, c, kv, live);
    t.x += v.x;
    t.y += v.y;
  }
  if (live) S.sk_ads[k] = t;
}

static cudaError_t sk_launch(const RgpuSys *d_sys, const double *d_xyz, const double *d_q, int n, int nk, double2 *d_sk,
                             double *d_out, cudaStream_t st)
{
  if (nk <= 0) return cudaSuccess;
  if (n <= 0 && !d_out) return cudaMemsetAsync(d_sk, 0, sizeof(double2) * (size_t)nk, st);
  const int blocks = (nk + SK_THREADS - 1) / SK_THREADS;
  /* CTAs that share the atoms of a block of wave vectors: a table's worth of
   * atoms each, as long as all CTAs run at once (148 SMs, 2 CTAs each) */
  int c = SK_PARTS;
  while (c > 1 && (c * blocks > 296 || SK_ATOMS * (c - 1) >= n)) c >>= 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(blocks * c), 1, 1);
  cfg.blockDim = dim3(SK_THREADS, 1, 1);
  cfg.dynamicSmemBytes = sizeof(SkSmem);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_structure_factor, d_sys, d_xyz, d_q, n, d_sk, d_out);
}

cudaError_t rgpu_structure_factor_launch(const RgpuSys *d_sys, const double *d_xyz, const double *d_q, int n,
                                         int nk, double2 *d_sk, cudaStream_t st)
{
  return sk_launch(d_sys, d_xyz, d_q, n, nk, d_sk, nullptr, st);
}

cudaError_t rgpu_ads_fourier_launch(const RgpuSys *d_sys, const double *d_xyz, int n, int nk, double2 *d_sk, double *d_out,
                                    int *blocks, cudaStream_t st)
{
  *blocks = (nk + SK_THREADS - 1) / SK_THREADS;
  if (*blocks > RGPU_FOURIER_BLOCKS) return cudaErrorInvalidValue;
  return sk_launch(d_sys, d_xyz, nullptr, n, nk, d_sk, d_out, st);
}

cudaError_t rgpu_upload_sk_launch(const RgpuSys *d_systems, int n, int max_nk, cudaStream_t st)
{
  if (n <= 0 || max_nk <= 0) return cudaSuccess;
  k_upload_sk<<<dim3((unsigned)((max_nk + SK_THREADS - 1) / SK_THREADS), (unsigned)n), SK_THREADS, sizeof(SkSmem), st>>>(d_systems);
  return cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Ewald Fourier difference of ns signed sites, writing dS(k) of the candidate
 * into d_ds (for a later accept) and {e_ads, e_host} into out (mapped host
 * memory). One cluster of CTAs splits the wave vectors; each CTA builds the
 * (small) phase tables of the FP64 path for itself. Bound by latency: the
 * descriptor, the table, one or two wave vectors a thread, two reductions (11.4
 * us for a displaced CO2 under the profiler, cold; 14 with one CTA). */
#define DELTA_CLUSTER 8

template <int MIXED>
__global__ void __launch_bounds__(256) k_ewald_delta(const RgpuSys *sysp, const __grid_constant__ RgpuSites in, int ns,
                                                     double2 *d_ds, double *out, int kw)
{
  __shared__ RgpuSys S;
  __shared__ EwSite sites[2 * RGPU_MAX_ATOMS];
  /* phase tables of the FP64 path; the mixed path forms its phases directly */
  __shared__ typename PhaseT<MIXED>::T tab[MIXED == 1 ? 1 : 2 * RGPU_MAX_ATOMS * 3 * 41];
  __shared__ double red[72];
  __shared__ double part[DELTA_CLUSTER][2];
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  cl.barrier_arrive();
  load_sys(&S, sysp);
  if (threadIdx.x < ns) {
    const int s = threadIdx.x;
    bead_set(sites[s].b, S, in.xyz[s][0], in.xyz[s][1], in.xyz[s][2], 0, -1);
    sites[s].q = in.q[s];
  }
  __syncthreads();
  ewald_phases<MIXED>(S, sites, ns, tab, kw);
  __syncthreads();
  double ea = 0.0, eh = 0.0;
  for (int k = rank * blockDim.x + threadIdx.x; k < S.nk; k += csize * blockDim.x) {
    double2 d = ewald_dS<MIXED>(tab, kw, sites, ns, S.kvec[k]);
    double2 so = S.sk_ads[k];
    double2 sf = S.sk_fw[k];
    double kf = S.kfactor[k];
    ea += kf * (2.0 * (so.x * d.x + so.y * d.y) + d.x * d.x + d.y * d.y);
    eh += kf * (sf.x * d.x + sf.y * d.y);
    d_ds[k] = d;
  }
  block_sum2(ea, eh, red);
  cl.barrier_wait();
  if (threadIdx.x == 0) {
    double *p = cl.map_shared_rank(&part[rank][0], 0);
    p[0] = ea;
    p[1] = eh;
  }
  cl.sync();
  if (rank == 0 && threadIdx.x < 2) {
    double t = 0.0;
    for (int c = 0; c < csize; c++) t += part[c][threadIdx.x];
    out[threadIdx.x] = t;
  }
}

__global__ void k_ewald_accept(const RgpuSys *sysp, const double2 *d_ds)
{
  const RgpuSys *S = sysp;
  int nk = S->nk;
  double2 *sk = S->sk_ads;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
    double2 a = sk[k], d = d_ds[k];
    sk[k] = make_double2(a.x + d.x, a.y + d.y);
  }
}

cudaError_t rgpu_ewald_delta_launch(int mixed, const RgpuSys *d_sys, const RgpuSites &in, int ns, int nk, double2 *d_ds,
                                    double *d_out, int kw, cudaStream_t st)
{
  if (ns < 1 || ns > 2 * RGPU_MAX_ATOMS || kw > 41) return cudaErrorInvalidValue;
  int c = DELTA_CLUSTER;
  while (c > 1 && 256 * (c - 1) >= nk) c >>= 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, mixed ? k_ewald_delta<1> : k_ewald_delta<0>, d_sys, in, ns, d_ds, d_out, kw);
}

cudaError_t rgpu_ewald_accept_launch(const RgpuSys *d_sys, const double2 *d_ds, int nk, cudaStream_t st)
{
  int blocks = (nk + 255) / 256;
  if (blocks < 1) blocks = 1;
  k_ewald_accept<<<blocks, 256, 0, st>>>(d_sys, d_ds);
  return cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
__device__ __forceinline__ void record_set(const RgpuSys &S, int i, int m, int a, const double *p, int4 *rec32,
                                           AdsRec64 *rec64)
{
  int xi, yi, zi;
  rgpu_fix3(S, p[0], p[1], p[2], xi, yi, zi);
  rec32[i] = make_int4(xi, yi, zi, m * 16 + a);
  AdsRec64 r;
  r.x = p[0]; r.y = p[1]; r.z = p[2]; r.tag = m * 16 + a;
  rec64[i] = r;
}

/* adsorbate records (fixed-point and FP64) from the authoritative positions;
 * nmol >= 0 also becomes the system's molecule count */
__global__ void k_build_records(const RgpuSys *sysp, int nads, int nmol, int4 *rec32, AdsRec64 *rec64)
{
  const RgpuSys *S = sysp;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && nmol >= 0) *S->nmol = nmol;
  if (i >= nads) return;
  const int m = i / S->natom, a = i - m * S->natom;
  record_set(*S, i, m, a, S->ads_xyz + 3 * i, rec32, rec64);
}

cudaError_t rgpu_records_launch(const RgpuSys *d_sys, int nads, int nmol, int4 *d_rec32, void *d_rec64, cudaStream_t st)
{
  if (nads <= 0 && nmol < 0) return cudaSuccess;
  k_build_records<<<nads > 128 ? (nads + 127) / 128 : 1, 128, 0, st>>>(d_sys, nads, nmol, d_rec32, (AdsRec64 *)d_rec64);
  return cudaGetLastError();
}

/* molecule m's positions and records, and the molecule count */
__global__ void k_set_molecule(const RgpuSys *sysp, const __grid_constant__ RgpuSites in, int m, int nmol, int4 *rec32,
                               AdsRec64 *rec64)
{
  const RgpuSys &S = *sysp;
  const int a = threadIdx.x;
  if (a == 0) *S.nmol = nmol;
  if (m < 0 || a >= S.natom) return;
  const int i = m * S.natom + a;
  const double p[3] = {in.xyz[a][0], in.xyz[a][1], in.xyz[a][2]};
  for (int c = 0; c < 3; c++) S.ads_xyz[3 * i + c] = p[c];
  record_set(S, i, m, a, p, rec32, rec64);
}

cudaError_t rgpu_set_molecule_launch(const RgpuSys *d_sys, const RgpuSites &in, int m, int nmol, int4 *d_rec32,
                                     void *d_rec64, cudaStream_t st)
{
  k_set_molecule<<<1, 32, 0, st>>>(d_sys, in, m, nmol, d_rec32, (AdsRec64 *)d_rec64);
  return cudaGetLastError();
}
