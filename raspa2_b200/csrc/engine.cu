/* Kernels of the B200 GCMC energy path.
 *
 *  - rgpu_engine_kernel: the persistent batched MC engine. One thread-block
 *    cluster owns one simulation box for the whole launch. The framework and
 *    the wave vectors are split between the CTAs of the cluster (each stages
 *    its share, with its share of S(k), in shared memory); every CTA keeps a
 *    full copy of the adsorbate records, draws the same counter-based random
 *    numbers and takes the same decisions. The step loop is a sequence of
 *    stages, each one energy evaluation: all threads place its positions, all
 *    warps evaluate (one place in the code, whatever the move), one cluster
 *    barrier makes every CTA's per-position sums readable, all threads add
 *    them up in rank order through distributed shared memory, so all CTAs see
 *    bitwise identical totals, and warp 0 of every CTA does the bookkeeping of
 *    the move and describes the next stage. Each cluster advances its box by `nsteps` MC
 *    moves (translation, rotation, CBMC insertion, CBMC deletion:
 *    src/mc_moves.c:1529, :2636, :6941, :7150) without returning to the host;
 *    FP64 and mixed runs see identical random streams.
 *  - the batched state transfer of an engine's systems.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "rgpu_chain.h"
#include "rgpu_device.cuh"
#include "rgpu_engine.h"
#include "rgpu_grid.cuh"

namespace cg = cooperative_groups;

/* eval_plan makes at most max(warps, positions) <= 64 framework units and no
 * more adsorbate units than that */
#define RGPU_MAX_UNITS 128
#define RGPU_MAX_WARPS 32
#define RGPU_RND 64           /* random slots tabulated per MC step (the trial orientations are drawn on their own) */
#define RGPU_FIXED_BYTES 26624 /* shared-memory slot of the fixed block */

/* ------------------------------------------------------------------------ */
/* shared-memory plan of the engine (offsets in bytes from the dynamic base).
 * fw_items: framework records of this CTA's share (tiles * RGPU_TILE), fwd_items:
 * their FP64 positions (FP64 path only), tiles: tile records of the share, k_items: wave
 * vectors of the share staged with their S(k) (0: read from global memory). The
 * block whose size is fixed (Fixed) comes first. */
struct EngineLayout {
  size_t fw, fwd, tiles, ads, q, tab, kvec, kf, skfw, skads, ang, total;
};

__host__ __device__ inline size_t rgpu_align(size_t x) { return (x + 255) & ~(size_t)255; }

/* bend and dihedral trigonometry of every trial of a chain growth stage
 * (flexible-chain builds only): {cos theta, sin theta, cos phi, sin phi,
 * torsion Rosenbluth factor} for beads 2.. natom-1 and each trial */
#define RGPU_ANG_STRIDE 5
#define RGPU_ANG_TABLE (RGPU_ANG_STRIDE * (RGPU_MAX_ATOMS - 2) * RGPU_MAX_TRIALS)
#define RGPU_ANG_DOUBLES (RGPU_ANG_TABLE + RGPU_MAX_ATOMS)   /* + the bend angle of each bead (chain_scheme 0) */

__host__ __device__ inline EngineLayout engine_layout(int mixed, int fw_items, int fwd_items, int tiles, int max_ads_atoms,
                                                      int kw, int k_items, int nwarps, int flex)
{
  EngineLayout L;
  size_t o = RGPU_FIXED_BYTES;
  L.fw = o; o = rgpu_align(o + (size_t)fw_items * sizeof(int4));
  L.fwd = o; o = rgpu_align(o + (size_t)fwd_items * sizeof(double4));
  L.tiles = o; o = rgpu_align(o + (size_t)tiles * sizeof(TileRec));
  L.ads = o; o = rgpu_align(o + (size_t)max_ads_atoms * (mixed ? sizeof(int4) : sizeof(AdsRec64)));
  /* per-warp pair queues: r2 (FP32, or FP64 for mixed = 2), charge, type; the
   * FP64 path queues atom indices */
  L.q = o; o = rgpu_align(o + (size_t)nwarps * 64 * (mixed == 2 ? 16 : (mixed ? 12 : 4)));
  /* per-site phase tables (none on the mixed path) */
  L.tab = o; o = rgpu_align(o + (mixed == 1 ? 0 : (size_t)2 * RGPU_MAX_ATOMS * 3 * kw * sizeof(double2)));
  L.kvec = o; o = rgpu_align(o + (size_t)k_items * sizeof(char4));
  L.kf = o; o = rgpu_align(o + (size_t)k_items * sizeof(double));
  L.skfw = o; o = rgpu_align(o + (size_t)k_items * sizeof(double2));
  L.skads = o; o = rgpu_align(o + (size_t)k_items * sizeof(double2));
  L.ang = o; o = rgpu_align(o + (flex ? 2 * RGPU_ANG_DOUBLES * sizeof(double) : 0));   /* growth, retrace */
  L.total = o;
  return L;
}

size_t rgpu_engine_smem_bytes(int mixed, int fw_items, int fwd_items, int tiles, int max_ads_atoms, int kw, int k_items,
                              int threads, int flex)
{
  return engine_layout(mixed, fw_items, fwd_items, tiles, max_ads_atoms, kw, k_items, threads / 32, flex).total;
}

/* The bookkeeping between evaluations is straight-line code that one warp runs
 * once per stage: it is bound by instruction fetch (compiled inline at each
 * use, with an evaluation in each move, the kernel had 520 to 800 KB of code,
 * several times an SM's instruction cache, and an addition cost about 30
 * cycles there). So one evaluation is inlined, into the loop; what is used
 * more than once beside it is a function of its own; and the work that can be
 * spread over threads (placing positions, adding up CTAs' sums) is done by all
 * of them between barriers, which cost some 500 cycles. Code now 120 to 270
 * KB. Measured (upload, moves, states read back), before and after: 64 mixed
 * CO2 boxes, 1000 moves each, 27.3 and 21.0 ms; one FP64 CO2 box, 200 moves,
 * 4.25 and 3.36 ms; 32 hexane boxes over grids, 100 moves, 4.45 and 3.87 ms. */
#define RGPU_COLD __noinline__

/* floor(2^32 / n) + 1 (less one for powers of two: 2^32 / n) for 2 <= n <= 64, 0
 * for n <= 1: x / n is the high half of its product with x, for x < 2^26 */
#define M1(n) ((unsigned)((4294967296ULL + (n) - 1) / (n)))
#define M8(n) M1(n), M1(n + 1), M1(n + 2), M1(n + 3), M1(n + 4), M1(n + 5), M1(n + 6), M1(n + 7)
static __constant__ unsigned c_magic[66] = {0, 0, M8(2), M8(10), M8(18), M8(26), M8(34), M8(42), M8(50), M8(58)};
#undef M8
#undef M1

/* One evaluation stage of the step loop, written by warp 0 and read by every
 * thread after the barrier that opens the stage. */
struct __align__(16) Stage {
  int ph;                     /* PH_*: what the stage evaluates, and what warp 0 does with it */
  int P, check;               /* bead positions to evaluate, how many of them test single pairs for overlap */
  int ns;                     /* Ewald sites to sum (0: none) */
  int ap;                     /* the last sites summed are still to be added to S_ads(k) */
  int db;                     /* buffer to draw step dstep's random numbers into (-1: none) */
  unsigned long long dstep;
  int sample;                 /* the step before ended: its state enters the ensemble sums */
  int first;                  /* the first stage of a step: the move is counted */
  /* the move: its type, molecule, whether a deletion or reinsertion has its
   * retrace orientations evaluated with the first-bead trials, the buffer of
   * the step's random numbers, steps done in this launch */
  int mv, m, one, buf;
  long long it;
  int ci, k;                  /* chains: bead of the growth and its trials */
  int r0, r1, rP;             /* chains: retrace beads of the stage, and their positions */
  int alo, ahi;               /* this CTA's adsorbate atoms */
  unsigned mf, ma;            /* chunk bounds: floor(2^32 / cf) + 1 and the same of ca (0 for one chunk) */
  int plan[8];                /* cf | ca << 16: the chunks of a position in each CTA of the cluster */
};
enum {
  PH_END, PH_SKIP,            /* launch done; step without an evaluation */
  PH_DISP,                    /* translation, rotation */
  PH_SWAP1, PH_SWAP2, PH_SWAPEW,     /* rigid insertion, deletion, Widom: first bead, orientations, Ewald sum */
  PH_REINS1, PH_REINSOLD, PH_REINS2, PH_REINSEW,  /* rigid reinsertion: first bead (and the old orientations), those
                                                    * by themselves, new orientations, Ewald sum */
  PH_TABLE, PH_GROW, PH_RETRACE, PH_CHAINEND   /* flexible chains */
};

/* outcome of a set of CBMC trials (cbmc_trials) */
struct Trials {
  double w_sum, w_sel;        /* sum of the weights, the selected trial's weight */
  double e[4];                /* the selected trial's energies */
  int sel, any;               /* the selected trial; whether any is valid */
};

/* broadcast/control block in shared memory */
struct Ctl {
  Stage st[3];                /* the current stage c, and the next: c + 1 as warp 0 describes it, c + 2 as warp 1
                               * does ahead of it (mod 3) */
  int which;                  /* which of them the next stage is */
  int cur;                    /* the current stage, for warp 0 */
  double rnd[3][RGPU_RND];    /* uniforms by slot, of three steps (step index mod 3) */
  double csn[3][2];           /* cos, sin of the step's rotation move */
  int mvn[3];                 /* move type of the step */
  long long it;               /* steps done in this launch */
  double energy[RGPU_NE];     /* running energies (written back by rank 0) */
  long long cnt[RGPU_NCNT];   /* move counters [0, RGPU_CNT_PAIRS) and reinsertion counters (rank 0's written back) */
  Trials tr[2];
  double u[4];                /* energies of the chosen configuration */
  double uo[4];               /* energies of the retraced old configuration (reinsertion) */
  double rosen;
  double rosen_old;
  double first[3];            /* chosen first bead */
  /* flexible chains: chosen bead positions of the configuration being grown
   * or retraced, intramolecular energy */
  double cp[RGPU_MAX_ATOMS][3];
  /* a retrace's beads: trial weight sum, the old bead's host VDW, adsorbate
   * VDW, intramolecular LJ and bonded energy, any valid trial */
  double rb[RGPU_MAX_ATOMS][6];
  double co[RGPU_MAX_ATOMS][3];  /* the old beads of a reinsertion's retrace */
  double uintra;
  __align__(16) double ewt[2][2];   /* this CTA's Ewald sums {e_ads, e_host}, by buffer */
  double ew[2];               /* the cluster's, of the stage */
  int nmol;
  int fail;
  int accept;                 /* the last Ewald sites summed were accepted */
  int sel;
  int nads;                   /* adsorbate atoms = nmol * natom */
  int status;                 /* RGPU_ERR_* bits */
  unsigned long long work[2]; /* work done: (k, site) products, k terms */
  long long cyc[2];           /* clock cycles in evaluations and Ewald sums */
  double sums[RGPU_NSUM];     /* ensemble sums of this launch */
  int next;                   /* unit counter of eval_units */
  int nextk, ewdone;          /* shares of the wave vectors taken, and summed */
  int ov;                     /* an overlap in the stage, in any CTA */
  int ovf[2];                 /* overlap flag of this CTA's evaluation, by buffer */
  int done[RGPU_MAX_POS];     /* units done of each position */
  unsigned long long wcnt[RGPU_MAX_WARPS][3];   /* pairs visited, in cut-off, charged in cut-off, by warp */
};
static_assert(sizeof(Stage) % 16 == 0, "stages are 16-byte aligned");

/* what is kept for a flexible chain's growth, in place of a rigid molecule's
 * orientation trials */
struct Growth {
  double ub[2][RGPU_MAX_TRIALS];  /* bonded energies of a bead's trials, by bead parity */
  double frame[RGPU_MAX_TRIALS][9];   /* the next bead's frame, should this trial be chosen (chain_frame) */
  double lj[RGPU_MAX_TRIALS];  /* intramolecular LJ of the current bead's trials (beads 4..) */
  double sel[3][RGPU_MAX_ATOMS];   /* uniforms that choose among a growth's trials, by bead, of three steps */
  double theta[3][RGPU_MAX_ATOMS];   /* bend angles of a growth's beads, of three steps */
};

/* The part of shared memory whose size does not depend on the systems, at its
 * start: the bookkeeping reaches it with addresses known to the compiler,
 * without pointers (which, in functions of their own, would be generic ones:
 * a dependent load each, and slower loads behind them). */
struct __align__(256) Fixed {
  RgpuSys S;
  Ctl C;
  BeadPos pos[RGPU_MAX_POS];
  double2 u[RGPU_MAX_UNITS];
  double4 part[2][RGPU_MAX_POS];   /* this CTA's sums {host VDW, host real, adsorbate VDW, adsorbate real} of each
                                    * position, by buffer */
  double4 tot[RGPU_MAX_POS];       /* the cluster's, of the stage */
  EwSite sites[2 * RGPU_MAX_ATOMS];
  double red[2 * RGPU_MAX_WARPS];
  union {
    double rot[3][2][RGPU_MAX_TRIALS][4];  /* quaternions of the orientation trials (new, retrace), of three steps */
    Growth gr;
  };
  uint64_t step0;                  /* first MC step of the launch */
  unsigned ads, ang;               /* offsets of the adsorbate records and of the chain trial trigonometry
                                    * ([2][RGPU_ANG_DOUBLES]: of a growth and of a retrace stage) */
  int rank, csize;
};
static_assert(sizeof(Fixed) <= RGPU_FIXED_BYTES, "fixed block exceeds its shared-memory slot");

__device__ __forceinline__ unsigned char *smem_at(unsigned offset)
{
  extern __shared__ __align__(256) unsigned char smem[];
  return smem + offset;
}
__device__ __forceinline__ Fixed &fx() { return *(Fixed *)smem_at(0); }
__device__ __forceinline__ double *fx_ang() { return (double *)smem_at(fx().ang); }

/* selects the build of a function of the bookkeeping */
template <int MIXED, bool FLEX>
struct Build {};

/* what the evaluation keeps in registers */
template <int MIXED, bool FLEX>
struct Eng {
  EvalSlice sl;
  EvalScratch sc;
  typename PhaseT<MIXED>::T *tab;
  int kw;
  int k0, k1;                /* this CTA's wave vectors */
  uint64_t step0;            /* first MC step of the launch */
  int rank, csize;
  int xb;                    /* buffer of the next evaluation (same sequence in every thread and CTA) */
};

/* Position of atom a of molecule m. FP64 records carry the position; on the
 * mixed path the FP64 positions stay in global memory (ads_xyz), which every
 * CTA of the cluster writes with the same values on each accepted move. */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void atom_xyz(Build<MIXED, FLEX> E, int m, int a, double *p)
{
  const int idx = m * fx().S.natom + a;
  if (MIXED) {
    const double *x = fx().S.ads_xyz + 3 * idx;
    p[0] = x[0]; p[1] = x[1]; p[2] = x[2];
  } else {
    const AdsRec64 &r = ((const AdsRec64 *)smem_at(fx().ads))[idx];
    p[0] = r.x; p[1] = r.y; p[2] = r.z;
  }
}

template <int MIXED, bool FLEX>
__device__ RGPU_COLD void atom_store(Build<MIXED, FLEX> E, int m, int a, const double *p)
{
  const RgpuSys &S = fx().S;
  const int idx = m * S.natom + a;
  if (MIXED) {
    double *x = fx().S.ads_xyz + 3 * idx;
    x[0] = p[0]; x[1] = p[1]; x[2] = p[2];
    int xi, yi, zi;
    rgpu_fix3(S, p[0], p[1], p[2], xi, yi, zi);
    ((int4 *)smem_at(fx().ads))[idx] = make_int4(xi, yi, zi, m * 16 + a);
  } else {
    AdsRec64 r;
    r.x = p[0]; r.y = p[1]; r.z = p[2]; r.tag = m * 16 + a;
    ((AdsRec64 *)smem_at(fx().ads))[idx] = r;
  }
}

/* RotationAround{X,Y,Z}Axis, src/utils.c:876-936; cs, sn of the angle */
__device__ __forceinline__ void rotate_axis(double *c, int axis, double cs, double sn)
{
  double x = c[0], y = c[1], z = c[2];
  if (axis == 0) { c[1] = cs * y + sn * z; c[2] = -sn * y + cs * z; }
  else if (axis == 1) { c[0] = cs * x - sn * z; c[2] = sn * x + cs * z; }
  else { c[0] = cs * x + sn * y; c[1] = -sn * x + cs * y; }
}

__device__ RGPU_COLD double2 cold_sincos(double x)
{
  double sn, cs;
  sincos(x, &sn, &cs);
  return make_double2(sn, cs);
}

__device__ RGPU_COLD double2 cold_uniforms(const RgpuSys &S, uint64_t step, uint32_t blk)
{
  double u[2];
  rgpu_uniform_pair(S.seed, S.sys_id, step, blk, u);
  return make_double2(u[0], u[1]);
}

/* RandomArrayRotationMatrix (Shoemake), src/utils.c:835-874, in two parts:
 * the quaternion, which needs the trigonometry, and its matrix */
__device__ __forceinline__ void random_quaternion(double x0, double y1, double y2, double *u)
{
  y1 *= 2.0 * M_PI;
  y2 *= 2.0 * M_PI;
  double r1 = sqrt(1.0 - x0), r2 = sqrt(x0);
  const double2 a = cold_sincos(y1), b = cold_sincos(y2);   /* {sin, cos} */
  u[0] = b.y * r2; u[1] = a.x * r1; u[2] = a.y * r1; u[3] = b.x * r2;
}

__device__ __forceinline__ void rotation_matrix(const double *u, double R[3][3])
{
  const double u0 = u[0], u1 = u[1], u2 = u[2], u3 = u[3];
  double ci = 2.0 * u0 * u0 - 1.0, ce = 2.0 * u0;
  R[0][0] = ci + 2.0 * u1 * u1;
  R[1][1] = ci + 2.0 * u2 * u2;
  R[2][2] = ci + 2.0 * u3 * u3;
  R[1][2] = 2.0 * u2 * u3 - ce * u1;
  R[2][0] = 2.0 * u3 * u1 - ce * u2;
  R[0][1] = 2.0 * u1 * u2 - ce * u3;
  R[2][1] = 2.0 * u3 * u2 + ce * u1;
  R[0][2] = 2.0 * u1 * u3 + ce * u2;
  R[1][0] = 2.0 * u2 * u1 + ce * u3;
}

/* share [lo, hi) of n items for rank r of c (1 <= c <= 8; n far below
 * 2^28, so n * c fits in 32 bits) */
__device__ __forceinline__ void share(int n, int r, int c, int &lo, int &hi)
{
  lo = n * r / c;
  hi = n * (r + 1) / c;
}

__device__ __forceinline__ bool has_ewald(const RgpuSys &S) { return S.ewald && S.mol_charged; }

/* ------------------------------------------------------------------------ */
__device__ double chain_ref_theta(const RgpuSys &S, int i, int stage, uint64_t step, int lane, const double (*old)[3]);

/* Random numbers, move type, rotation of a displacement, quaternions of the
 * orientation trials and bend angles of a growth of MC step `step`, into buffer db, by
 * threads t0, t0 + nt, .... All of it depends on the step alone. The warps
 * that wait for warp 0's bookkeeping draw it two steps ahead (a step's tables
 * have to be visible when warp 0 starts it, in the same section in which it
 * ends the step before), so it costs the step loop no time of its own. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void draw_step(Build<MIXED, FLEX> E, uint64_t step, int db, int t0, int nt)
{
  const RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  /* thread i < nr: block i of the table; nr + j, j < 16: orientation trial j;
   * j < 32: retrace orientation j - 16 of a reinsertion; j = 32: the move */
  const int nr = RGPU_RND / 2;
  const bool chain = FLEX && S.flexible;   /* j = 33..36: the choices among a growth's trials */
#pragma unroll 1
  for (int i = t0; i < nr + (chain ? 37 : 33); i += nt) {
    const int j = i - nr, t = j & 15, old = j >> 4;
    const uint32_t slot = (old ? SLOT_ORIENT_OLD : SLOT_ORIENT) + 4 * t;
    double2 u = cold_uniforms(S, step, j < 0 ? (uint32_t)i : (j > 32 ? (RGPU_SLOT_CHAIN_SEL >> 1) + j - 33 : 0u));
    if (j < 0 || j > 32) {
      double *r = j < 0 ? &C.rnd[db][2 * i] : &fx().gr.sel[db][2 * (j - 33)];
      r[0] = u.x;
      r[1] = u.y;
      continue;
    }
    int mv = 0;
    while (mv < 5 && u.x >= S.cum[mv]) mv++;
    const bool turn = j == 32 && mv == 1;
    if (j == 32) C.mvn[db] = mv;
    else if (mv < 2 || t >= S.ntrial || S.natom == 1 || (old && mv != 4) || (FLEX && S.flexible)) continue;
    u = cold_uniforms(S, step, j == 32 ? SLOT_VNEW >> 1 : slot >> 1);
    if (turn) {
      const double2 sc = cold_sincos((2.0 * u.x - 1.0) * S.max_rotation);
      C.csn[db][0] = sc.y;
      C.csn[db][1] = sc.x;
    }
    if (j == 32) continue;
    const double2 v = cold_uniforms(S, step, (slot >> 1) + 1);
    random_quaternion(u.x, u.y, v.x, fx().rot[db][old][t]);
  }
  if (chain && S.chain_scheme == 0) {
    /* the bend angles of a growth's beads, one warp each */
    __syncwarp();
    const double u0 = cold_uniforms(S, step, 0u).x;
    int mv = 0;
    while (mv < 5 && u0 >= S.cum[mv]) mv++;
    if (mv == 2 || mv >= 4)
      for (int i = 2 + (t0 >> 5); i < S.natom; i += nt >> 5) {
        const double th = chain_ref_theta(S, i, 0, step, threadIdx.x & 31, nullptr);
        if ((threadIdx.x & 31) == 0) fx().gr.theta[db][i] = th;
      }
  }
}

static_assert(SLOT_VNEW % 2 == 0 && SLOT_MOVE == 0 && SLOT_ORIENT % 2 == 0 && SLOT_ORIENT_OLD % 2 == 0 &&
                  RGPU_SLOT_CHAIN_SEL % 2 == 0,
              "draw_step takes the first uniform of a block");

/* ------------------------------------------------------------------------ */
/* Placing a stage's positions and Ewald sites: thread i < P places position i,
 * thread P + j site j (the moves' drivers below say what they are). */

/* bead j of orientation trial t about o, with the trials' quaternions Q;
 * keep >= 0: trial 0 is molecule keep's own orientation */
template <int MIXED, bool FLEX>
__device__ __forceinline__ int orientation_bead(Build<MIXED, FLEX> E, const double *o, const double (*Q)[4], int i,
                                                int keep, double *p)
{
  const RgpuSys &S = fx().S;
  const int nb = S.natom - 1, sb = S.start_bead;
  const int t = small_div(i, nb), j = i - t * nb, a = j < sb ? j : j + 1;
  if (t == 0 && keep >= 0) {
    atom_xyz(E, keep, a, p);
    return a;
  }
  const double c[3] = {S.mol_ref[a][0] - S.mol_ref[sb][0], S.mol_ref[a][1] - S.mol_ref[sb][1],
                       S.mol_ref[a][2] - S.mol_ref[sb][2]};
  double R[3][3];
  rotation_matrix(Q[t], R);
  p[0] = o[0] + c[0] * R[0][0] + c[1] * R[0][1] + c[2] * R[0][2];
  p[1] = o[1] + c[0] * R[1][0] + c[1] * R[1][1] + c[2] * R[1][2];
  p[2] = o[2] + c[0] * R[2][0] + c[1] * R[2][1] + c[2] * R[2][2];
  return a;
}

/* atom a of the configuration chosen among the last evaluation's trials */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void chosen_atom(Build<MIXED, FLEX> E, int a, double *p)
{
  const RgpuSys &S = fx().S;
  const Ctl &C = fx().C;
  const int sb = S.start_bead;
  if (a == sb) {
    p[0] = C.first[0]; p[1] = C.first[1]; p[2] = C.first[2];
  } else {
    const BeadPos &b = fx().pos[C.sel * (S.natom - 1) + (a < sb ? a : a - 1)];
    p[0] = b.x; p[1] = b.y; p[2] = b.z;
  }
}

/* position of trial t of bead i of a chain grown onto beads x[0..i-1], with
 * the stage's table of trial angles */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void chain_position(Build<MIXED, FLEX> E, uint64_t step, int stage, int i, int t,
                                               const double (*x)[3], const double *ang, double *p)
{
  const RgpuSys &S = fx().S;
  if (i == 0) {
    rgpu_box_point(S, rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, 0, t, 0)),
                   rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, 0, t, 1)),
                   rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, 0, t, 2)), p);
  } else if (i == 1) {
    chain_trial(S, x, i, [&](int d) { return rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, t, d)); }, p);
  } else {
    const double *a = ang + RGPU_ANG_STRIDE * ((i - 2) * RGPU_MAX_TRIALS + t);
    chain_place_trig(i >= 3 ? x[i - 3] : nullptr, x[i - 2], x[i - 1], S.bond, a[0], a[1], a[2], a[3], p);
  }
}

template <int MIXED, bool FLEX>
__device__ __forceinline__ void place(Build<MIXED, FLEX> E, const Stage &g, int i)
{
  const RgpuSys &S = fx().S;
  const Ctl &C = fx().C;
  const int na = S.natom, sb = S.start_bead, nf = S.ntrial_first, buf = g.buf, ph = g.ph, m = g.m;
  const double *R = C.rnd[buf];
  const bool site = i >= g.P;
  const int j = site ? i - g.P : i;
  double p[3], q = 0.0;
  int a = 0, excl = m;
  if (ph == PH_DISP) {
    /* the new positions, then the old ones; the sites are the same with
     * charges of opposite sign */
    a = j < na ? j : j - na;
    q = j < na ? S.mol_q[a] : -S.mol_q[a];
    atom_xyz(E, m, a, p);
    if (j < na) {
      const double vnew = 2.0 * R[SLOT_VNEW] - 1.0;
      int axis = (int)(3.0 * R[SLOT_AXIS]);
      if (axis > 2) axis = 2;
      if (g.mv == 0) {
        const double d = vnew * S.max_translation;
        if (axis == 0) p[0] += d;
        else if (axis == 1) p[1] += d;
        else p[2] += d;
      } else {
        double o[3];
        atom_xyz(E, m, sb, o);
        double c[3] = {p[0] - o[0], p[1] - o[1], p[2] - o[2]};
        rotate_axis(c, axis, C.csn[buf][0], C.csn[buf][1]);
        p[0] = c[0] + o[0]; p[1] = c[1] + o[1]; p[2] = c[2] + o[2];
      }
    }
  } else if (FLEX && (ph == PH_GROW || ph == PH_RETRACE)) {
    const uint64_t step = fx().step0 + (uint64_t)g.it;
    if (j < g.k) {
      a = g.ci;
      excl = g.mv == 4 ? m : -1;
      if (a >= 2) {
        /* in the frame that the last bead's choice left */
        const double *t = fx_ang() + RGPU_ANG_STRIDE * ((a - 2) * RGPU_MAX_TRIALS + j);
        chain_place_frame(fx().gr.frame[C.sel], C.cp[a - 1], S.bond, t[0], t[1], t[2], t[3], p);
      } else {
        chain_position(E, step, 0, a, j, C.cp, fx_ang(), p);
      }
    } else {
      /* retrace trials: bead a of the group, trial t in growth order; trial
       * 0 of each bead is the old bead */
      const double (*old)[3] = ph == PH_GROW ? C.co : C.cp;
      const int nt = S.ntrial;
      int t = j - g.k;
      a = g.r0;
      while (t >= (a == 0 ? nf : nt)) {
        t -= a == 0 ? nf : nt;
        a++;
      }
      if (t == 0) {
        p[0] = old[a][0]; p[1] = old[a][1]; p[2] = old[a][2];
      } else {
        chain_position(E, step, 1, a, t, old, fx_ang() + (ph == PH_GROW ? RGPU_ANG_DOUBLES : 0), p);
      }
    }
  } else if (ph == PH_SWAPEW || ph == PH_REINSEW) {
    /* the chosen configuration, then a reinsertion's old one */
    a = j < na ? j : j - na;
    q = j < na && g.mv != 3 ? S.mol_q[a] : -S.mol_q[a];
    if (j < na) chosen_atom(E, a, p);
    else atom_xyz(E, m, a, p);
  } else if (site) {
    /* a one-evaluation deletion's removed molecule */
    a = j;
    q = -S.mol_q[a];
    atom_xyz(E, m, a, p);
  } else {
    const bool insert = ph <= PH_SWAPEW && g.mv != 3, second = ph == PH_SWAP2 || ph == PH_REINS2;
    const bool reinsold = ph == PH_REINS1 || ph == PH_REINSOLD;
    const int n1 = second || ph == PH_REINSOLD ? 0 : (reinsold ? nf + 1 : nf);   /* first-bead positions */
    if (insert) excl = -1;
    if (j < n1) {
      a = sb;
      /* new first-bead trials; the old first bead is a deletion's trial 0
       * and the position after a reinsertion's trials */
      if (ph == PH_REINS1 ? j == nf : (!insert && j == 0)) atom_xyz(E, m, sb, p);
      else rgpu_box_point(S, R[SLOT_FIRST + 3 * j + 2], R[SLOT_FIRST + 3 * j + 1], R[SLOT_FIRST + 3 * j + 0], p);
    } else {
      double o[3];
      if (second) { o[0] = C.first[0]; o[1] = C.first[1]; o[2] = C.first[2]; }
      else atom_xyz(E, m, sb, o);
      a = orientation_bead(E, o, fx().rot[buf][reinsold], j - n1, insert || ph == PH_REINS2 ? -1 : m, p);
    }
  }
  BeadPos b;
  bead_set(b, S, p[0], p[1], p[2], a, excl);
  if (!site) fx().pos[j] = b;
  if (g.ns && (site || ph == PH_DISP)) {
    EwSite &t = fx().sites[j];
    t.b = b;
    t.q = q;
  }
}

/* ------------------------------------------------------------------------ */
/* The evaluation of a stage: pair sums of its positions on this CTA's share,
 * the pending S_ads(k) update and the Ewald sum of its sites on this CTA's
 * wave vectors, one cluster barrier; then the cluster's totals of every
 * position (fx().tot) and of the Ewald sum (C.ew), each CTA's part added in rank
 * order, and a block barrier. All threads call.
 *
 * The Ewald work follows the pair units and fills their tail (with a fixed
 * share per warp a stage waited for the warps that had two pair units before
 * theirs). On the mixed path it needs no phase table; the other paths build one
 * per stage. */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void eval_stage(Eng<MIXED, FLEX> &E, const Stage &g)
{
  Ctl &C = fx().C;
  RgpuSys &S = fx().S;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const long long t0 = clock64();
  const EwSite *sites = fx().sites;
  if (MIXED != 1 && g.ns) {
    ewald_phases<MIXED>(S, sites, g.ns, E.tab, E.kw);
    __syncthreads();
  }
  if (g.ns && threadIdx.x == 0) {
    C.work[0] += (unsigned long long)(E.k1 - E.k0) * g.ns;
    C.work[1] += (unsigned long long)(E.k1 - E.k0);
  }
  double4 *part = fx().part[E.xb];
  if (FLEX && S.use_grid && E.rank == 0) {
    /* host VDW from the bead types' energy grids (one CTA of the cluster):
     * 8 lanes per position, 4 positions per warp, before the pair units */
#pragma unroll 1
    for (int base = w * 4; base < g.P; base += nw * 4) {
      const int p = base + (lane >> 3);
      const bool live = p < g.P;
      const double x[3] = {live ? fx().pos[p].x : 0.0, live ? fx().pos[p].y : 0.0, live ? fx().pos[p].z : 0.0};
      const double v = rgpu_grid_value8(S.grid[live ? fx().pos[p].atom : 0], S.grid_geom, x, lane & 7, live);
      double vq = 0.0;
      if (S.use_coul_grid) {
        /* real-space charge energy: the bead charge times the unit-charge
         * Coulomb grid (InterpolateCoulombGrid, src/grids.c:1200) */
        const double q = live ? S.mol_q[fx().pos[p].atom] : 0.0;
        vq = q * rgpu_grid_value8(S.coul_grid, S.coul_geom, x, lane & 7, live && q != 0.0, false);
      }
      if (live && (lane & 7) == 0) {
        part[p].x = v;
        part[p].y = vq;
        if (p < g.check && v >= S.overlap) C.ovf[E.xb] = 1;
      }
    }
  }
  if (FLEX && g.ph == PH_GROW && g.ci >= 4 && w == nw - 1 && lane < g.k) {
    /* the trials' LJ with the chain, for warp 0's choice */
    const double p[3] = {fx().pos[lane].x, fx().pos[lane].y, fx().pos[lane].z};
    fx().gr.lj[lane] = chain_intra_lj(S, C.cp, g.ci, p);
  }
  if (g.P) {
    E.sc.ovf = &C.ovf[E.xb];
    E.sc.part = part;
    E.sl.ads_lo = g.alo;
    E.sl.ads_hi = g.ahi;
    const int pl = g.plan[E.rank];
    eval_units<MIXED>(S, E.sl, fx().pos, g.P, g.check, E.sc, pl & 0xffff, pl >> 16, g.mf, g.ma);
  }
  if (g.ns || g.ap) {
    /* the shares of the wave vectors, one per warp of the block, taken as the
     * warps run out of pair units; the last to finish adds them up in order */
    for (;;) {
      int u = 0;
      if (lane == 0) u = atomicAdd(&C.nextk, 1);
      u = __shfl_sync(RGPU_FULL, u, 0);
      if (u >= nw) break;
      ewald_share<MIXED>(S, E.tab, E.kw, sites, g.ns, g.ap, E.k0, E.k1, u, fx().red);
      if (!g.ns) continue;
      int d = 0;
      if (lane == 0) {
        __threadfence_block();
        d = atomicAdd(&C.ewdone, 1);
        __threadfence_block();
      }
      if (__shfl_sync(RGPU_FULL, d, 0) == nw - 1) {
        __syncwarp();           /* lane 0's fences before the other lanes' reads of the shares */
        const double ea = warp_sum(lane < nw ? fx().red[2 * lane] : 0.0), eh = warp_sum(lane < nw ? fx().red[2 * lane + 1] : 0.0);
        if (lane == 0) {
          C.ewt[E.xb][0] = ea;
          C.ewt[E.xb][1] = eh;
          C.ewdone = 0;
        }
      }
    }
  }
  cl.sync();
  /* term k of position p: thread 4 p + k */
  const bool grids = FLEX && S.use_grid;
#pragma unroll 1
  for (int e = threadIdx.x; e < 4 * g.P; e += blockDim.x) {
    const double *own = (const double *)part + e;
    const bool host = (e & 2) == 0;
    double t = 0.0;
#pragma unroll 1
    for (int q0 = 0; q0 < E.csize; q0 += 8) {
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int q = q0 + j;
        v[j] = 0.0;
        if (q < E.csize) {
          const int pl = g.plan[q];
          if (host ? (grids ? q == 0 : (pl & 0xffff) != 0) : (pl >> 16) != 0)
            v[j] = E.csize > 1 ? *cl.map_shared_rank(own, q) : *own;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; j++) t += v[j];
    }
    ((double *)fx().tot)[e] = t;
  }
  if (w == nw - 1) {
    /* the last warp: Ewald totals (lane q: CTA q's) and the overlap flag */
    double2 t = make_double2(0.0, 0.0);
    int o = 0;
    if (lane < E.csize) {
      const double2 *ow = (const double2 *)C.ewt[E.xb];
      const int *of = &C.ovf[E.xb];
      if (E.csize > 1) {
        ow = cl.map_shared_rank(ow, lane);
        of = cl.map_shared_rank(of, lane);
      }
      if (g.ns) t = *ow;
      o = *of;
    }
    o = __any_sync(RGPU_FULL, o);
    double ea = 0.0, eh = 0.0;
#pragma unroll 1
    for (int q = 0; g.ns && q < E.csize; q++) {
      ea += __shfl_sync(RGPU_FULL, t.x, q);
      eh += __shfl_sync(RGPU_FULL, t.y, q);
    }
    if (lane == 0) {
      C.ew[0] = ea;
      C.ew[1] = eh;
      C.ov = o;
    }
  }
  if (threadIdx.x == 0) {
    C.next = C.nextk = 0;       /* counters of the next evaluation */
    C.ovf[E.xb ^ 1] = 0;        /* read last before this stage's cluster barrier */
    C.cyc[g.P ? 0 : 1] += clock64() - t0;
  }
  E.xb ^= 1;
  __syncthreads();
}

/* The functions from here to end_stage are run by warp 0 of every CTA, all
 * lanes converged, where they do not say otherwise. E is the handle's copy in
 * shared memory, which warp 0 alone updates. Every CTA of the cluster holds
 * the same totals and takes the same decisions. */

__device__ __forceinline__ int stage_after(int c, int n) { return c + n >= 3 ? c + n - 3 : c + n; }

/* the stage just evaluated */
__device__ __forceinline__ const Stage &cur() { return fx().C.st[fx().C.cur]; }

/* Describes stage n, which follows stage c: what it evaluates, and the chunks
 * of a position in every CTA (lane q: CTA q). */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void fill_stage(Build<MIXED, FLEX> E, Stage &n, const Stage &c, int ph, int P, int check, int ns)
{
  const RgpuSys &S = fx().S;
  const int lane = threadIdx.x & 31, q = lane;
  if (P && q < fx().csize) {
    const unsigned mc = c_magic[fx().csize];
    const int nads = fx().C.nads;
    int t0 = S.ntile * q, t1 = S.ntile * (q + 1), a0 = nads * q, a1 = nads * (q + 1);
    if (fx().csize > 1) {
      t0 = (int)__umulhi((unsigned)t0, mc);
      t1 = (int)__umulhi((unsigned)t1, mc);
      a0 = (int)__umulhi((unsigned)a0, mc);
      a1 = (int)__umulhi((unsigned)a1, mc);
    }
    if (FLEX && S.use_grid) t1 = t0;
    const EvalPlan pl = eval_plan(P, t1 - t0, a1 - a0, blockDim.x >> 5, RGPU_MAX_UNITS, 2);
    n.plan[q] = pl.cf | pl.ca << 16;
    if (q == fx().rank) {
      n.alo = a0;
      n.ahi = a1;
      n.mf = c_magic[pl.cf];
      n.ma = c_magic[pl.ca];
    }
  }
  if (lane == 0) {
    n.ph = ph;
    n.P = P;
    n.check = check;
    n.ns = ns;
    n.db = -1;
    n.first = 0;
    n.k = n.rP = 0;
    n.mv = c.mv;
    n.m = c.m;
    n.one = c.one;
    n.buf = c.buf;
    n.it = c.it;
  }
}

/* the stage that follows in the same move */
__device__ __forceinline__ Stage &next_of() { return fx().C.st[stage_after(fx().C.cur, 1)]; }

template <int MIXED, bool FLEX>
__device__ __forceinline__ void next_stage(Build<MIXED, FLEX> E, int ph, int P, int check, int ns)
{
  fill_stage(E, next_of(), cur(), ph, P, check, ns);
}

/* an accepted move's sites are added to S_ads(k) in the next stage (end_stage
 * passes them on) */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void accept_sites(Build<MIXED, FLEX> E)
{
  if (has_ewald(fx().S) && threadIdx.x == 0) fx().C.accept = 1;
}

__device__ RGPU_COLD double cold_exp(double x) { return exp(x); }

/* exp(x) and exp(y), by two lanes */
__device__ __forceinline__ void exp_pair(double x, double y, double &ex, double &ey)
{
  const double r = cold_exp((threadIdx.x & 1) ? y : x);
  ex = __shfl_sync(RGPU_FULL, r, 0);
  ey = __shfl_sync(RGPU_FULL, r, 1);
}

/* inclusive sum over the lanes up to each one */
__device__ __forceinline__ double warp_scan(double v)
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(RGPU_FULL, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

/* SelectTrialPosition (src/cbmc.c:563-599) among the weights w of lanes < n,
 * cum their sums up to each lane: the first trial whose cumulative weight
 * reaches u times their sum; trial 0 where that is zero or NaN (weights that
 * all underflow, or overflow and cancel), as the reference's loop takes it */
__device__ __forceinline__ int select_trial(double w, double cum, int n, double u)
{
  const int lane = threadIdx.x & 31;
  const double target = u * __shfl_sync(RGPU_FULL, cum, 31);
  if (!(target > 0.0)) return 0;
  const unsigned hit = __ballot_sync(RGPU_FULL, lane < n && w > 0.0 && !(cum < target));
  return hit ? __ffs(hit) - 1 : n - 1;
}

/* Rosenbluth bookkeeping of n trials (lane t = trial t, nb beads each at
 * positions off + t*nb + j) into out. First bead (nb = 1, first = true):
 * overlap when any energy reaches the criterion (src/cbmc.c:699-701);
 * orientations: when a bead's host VDW energy does (src/cbmc.c:1210-1215).
 * LJ biasing (src/cbmc.c:734-735, :1432-1436). select: a trial is chosen with
 * usel, else trial 0 is. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void cbmc_trials(Build<MIXED, FLEX> E, int off, int n, int nb, bool first, bool select, double usel,
                                      Trials *out)
{
  const int lane = threadIdx.x & 31;
  const RgpuSys &S = fx().S;
  double4 e = make_double4(0.0, 0.0, 0.0, 0.0);
  int ov = lane >= n;
  if (lane < n)
#pragma unroll 1
    for (int j = 0; j < nb; j++) {
      const double4 r = fx().tot[off + lane * nb + j];
      ov |= r.x >= S.overlap || (first && (r.y >= S.overlap || r.z >= S.overlap || r.w >= S.overlap));
      e.x += r.x; e.y += r.y; e.z += r.z; e.w += r.w;
    }
  const double bf = -S.beta * (e.x + e.z);
  const double w = ov ? 0.0 : cold_exp(bf);
  const bool any = __any_sync(RGPU_FULL, !ov);
  const double cum = warp_scan(w), w_sum = __shfl_sync(RGPU_FULL, cum, 31);
  int s = 0;
  if (select && any) {
    if (w_sum > 1e-200 && w_sum < 1e200) {
      s = select_trial(w, cum, n, usel);
    } else {
      /* the weights leave FP64's range: relative to the largest, as
       * SelectTrialPosition forms them */
      double largest = ov ? -DBL_MAX : bf;
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) largest = fmax(largest, __shfl_xor_sync(RGPU_FULL, largest, o));
      const double ws = ov ? 0.0 : cold_exp(bf - largest);
      s = select_trial(ws, warp_scan(ws), n, usel);
    }
  }
  if (lane == s) {
    out->w_sum = w_sum;
    out->w_sel = w;
    out->e[0] = e.x; out->e[1] = e.y; out->e[2] = e.z; out->e[3] = e.w;
    out->sel = s;
    out->any = any;
  }
  __syncwarp();
}

/* adds sgn times the energies u and the Fourier terms to the running totals
 * (lane 0) */
__device__ __forceinline__ void add_energies(Ctl &C, double sgn, const double *u, double d_host, double d_ads)
{
  C.energy[RGPU_E_HOST_VDW] += sgn * u[0];
  C.energy[RGPU_E_HOST_REAL] += sgn * u[1];
  C.energy[RGPU_E_ADS_VDW] += sgn * u[2];
  C.energy[RGPU_E_ADS_REAL] += sgn * u[3];
  C.energy[RGPU_E_HOST_FOURIER] += d_host;
  C.energy[RGPU_E_ADS_FOURIER] += d_ads;
}

/* ------------------------------------------------------------------------ */
/* translation (mv=0) and rotation (mv=1):
 * TranslationMoveAdsorbate src/mc_moves.c:1529-1762, RotationMoveAdsorbate :2636.
 * One stage: the na new positions, the na old ones, the Ewald sum. */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void end_displace(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int na = S.natom, lane = threadIdx.x;
  if (C.ov) {
    if (lane == 0) C.cnt[RGPU_CNT_OVERLAP]++;
    return;
  }
  /* lane k < 4: change of energy term k */
  const double *tot = (const double *)fx().tot + (lane & 3);
  double dl = 0.0;
#pragma unroll 1
  for (int j = 0; j < na; j++) dl += tot[4 * j] - tot[4 * (na + j)];
  double d_ads = 0.0, d_host = 0.0;
  if (has_ewald(S)) {
    /* the exclusion energy of a rigid molecule is the same before and
     * after the displacement (the reference's difference of the two is
     * zero up to rounding) */
    ewald_finish(S, C.ew[0], C.ew[1], S.excl_mol, S.excl_mol, 0, 0.0, d_ads, d_host);
  }
  double u[4];
#pragma unroll
  for (int k = 0; k < 4; k++) u[k] = __shfl_sync(RGPU_FULL, dl, k);
  const double du = u[0] + u[1] + u[2] + u[3] + d_ads + d_host;
  const double pacc = cold_exp(-S.beta * du);
  const bool accept = C.rnd[buf][SLOT_ACCEPT] < pacc;
  if (lane == 0) {
    if (!isfinite(du)) C.status |= RGPU_ERR_NONFINITE;
    if (accept) {
      C.cnt[RGPU_CNT_ACCEPT + cur().mv]++;
      add_energies(C, 1.0, u, d_host, d_ads);
    }
  }
  if (accept) {
    if (lane < na) {
      const double p[3] = {fx().pos[lane].x, fx().pos[lane].y, fx().pos[lane].z};
      atom_store(E, cur().m, lane, p);
    }
    accept_sites(E);
  }
}

/* ------------------------------------------------------------------------ */
/* CBMC insertion / deletion of a rigid molecule grown from the starting bead
 * (widom: a test insertion that only samples its Rosenbluth weight,
 * WidomAdsorbateMove src/mc_moves.c:7844-8030):
 * GrowMolecule src/cbmc.c:3056-3181 and RetraceMolecule :2928-3054 with
 * HandleFirstBead :623-795, Rosen/RosenOld :2762-2926, the rigid-group branch
 * of GenerateTrialOrientationsSimpleSphere :1480-1578 and
 * ComputeExternalEnergies :1154-1478, LJ biasing; acceptance of
 * SwapAddAdsorbateMove src/mc_moves.c:7016 and SwapRemoveAdsorbateMove :7228.
 * Stages: first-bead trials, orientation trials, Ewald sum. A deletion retraces
 * the old molecule: its first bead and orientation are trial 0 of each stage,
 * known up front, so both stages' trials and the Ewald sum of the removed
 * molecule go into one evaluation (first-bead trials at positions 0..nf,
 * orientation t's beads at nf + t*nb + j) when they fit. */
/* acceptance of an insertion, deletion or Widom sample whose weight and
 * energies stand in C */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void accept_swap(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int mv = cur().mv, nmol = C.nmol, na = S.natom, m = cur().m;
  const bool insert = mv != 3, widom = mv == 5;
  /* LJ-biasing correction, src/cbmc.c:3171-3178 / :3044-3051 */
  double d_ads = 0.0, d_host = 0.0, lj, f;
  if (has_ewald(S)) {
    const double ex = S.excl_mol;      /* rigid molecule */
    const double net = nmol * S.mol_charge;
    if (insert) ewald_finish(S, C.ew[0], C.ew[1], ex, 0.0, 1, net, d_ads, d_host);
    else ewald_finish(S, C.ew[0], C.ew[1], 0.0, ex, -1, net, d_ads, d_host);
  }
  exp_pair(-S.beta * (C.u[1] + C.u[3]), (insert ? -S.beta : S.beta) * (d_ads + d_host), lj, f);
  const double rosen = C.rosen * lj;
  double pacc;
  if (insert) pacc = rosen * f * S.fugacity_beta_v / (1.0 + nmol);
  else pacc = (double)nmol / (rosen * f * S.fugacity_beta_v);
  const bool accept = !widom && C.rnd[buf][SLOT_ACCEPT] < pacc;
  __syncwarp();
  if (threadIdx.x == 0) {
    if (!(pacc == pacc)) C.status |= RGPU_ERR_NONFINITE;
    if (widom) C.sums[RGPU_SUM_WIDOM_W] += rosen * f;
    if (accept) {
      C.cnt[RGPU_CNT_ACCEPT + mv]++;
      add_energies(C, insert ? 1.0 : -1.0, C.u, d_host, d_ads);
      C.nmol = insert ? nmol + 1 : nmol - 1;
      C.nads = C.nmol * na;
    }
  }
  if (accept) {
    if (threadIdx.x < na) {
      double p[3];
      if (insert) {
        chosen_atom(E, threadIdx.x, p);
        atom_store(E, nmol, threadIdx.x, p);
      } else if (m != nmol - 1) {
        /* RemoveAdsorbateMolecule (src/molecule.c:3193): the last molecule
         * takes the freed slot */
        atom_xyz(E, nmol - 1, threadIdx.x, p);
        atom_store(E, m, threadIdx.x, p);
      }
    }
    accept_sites(E);
  }
}

/* the configuration is chosen: its Ewald sum, or the acceptance. Returns
 * whether the step is done. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD bool grown_swap(Build<MIXED, FLEX> E, int buf)
{
  if (has_ewald(fx().S)) {
    next_stage(E, PH_SWAPEW, 0, 0, fx().S.natom);
    return false;
  }
  accept_swap(E, buf);
  return true;
}

/* after the first-bead trials (and, in a one-evaluation deletion, the
 * retrace orientations); returns whether the step is done */
template <int MIXED, bool FLEX>
__device__ __forceinline__ bool end_swap1(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const bool insert = cur().mv != 3, one = cur().one != 0;
  const int na = S.natom, nf = S.ntrial_first, nt = S.ntrial, nb = na - 1;
  const Trials &a = C.tr[0], &b = C.tr[1];
  cbmc_trials(E, 0, nf, 1, true, insert, C.rnd[buf][SLOT_FIRST_SELECT], &C.tr[0]);
  double rosen = a.w_sum / (double)nf;
  bool fail = !a.any || (insert && rosen < 1e-150);
  const bool both = !fail && one && na > 1;
  if (both) {
    /* the retrace orientations (trial 0 is the old one, not selected) */
    cbmc_trials(E, nf, nt, nb, false, false, 0.0, &C.tr[1]);
    fail = !b.any;
    rosen *= b.w_sum / (double)nt;
  }
  if (threadIdx.x < 4) C.u[threadIdx.x] = both ? a.e[threadIdx.x] + b.e[threadIdx.x] : a.e[threadIdx.x];
  if (threadIdx.x == 0) {
    C.rosen = rosen;
    C.sel = a.sel;
    const BeadPos &p = fx().pos[a.sel];
    C.first[0] = p.x; C.first[1] = p.y; C.first[2] = p.z;
    if (fail) C.cnt[RGPU_CNT_OVERLAP]++;
  }
  __syncwarp();
  if (fail) return true;
  if (one) {
    accept_swap(E, buf);
    return true;
  }
  if (na == 1) return grown_swap(E, buf);
  next_stage(E, PH_SWAP2, nt * nb, 0, 0);
  return false;
}

/* the orientation trials enter C; returns whether the growth failed */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD bool add_orientations(Build<MIXED, FLEX> E, bool grow, int buf)
{
  Ctl &C = fx().C;
  const int nt = fx().S.ntrial;
  const Trials &a = C.tr[0];
  cbmc_trials(E, 0, nt, fx().S.natom - 1, false, grow, C.rnd[buf][SLOT_ORIENT_SELECT], &C.tr[0]);
  const double rosen = C.rosen * (a.w_sum / (double)nt);
  const bool fail = !a.any || (grow && rosen < 1e-150);
  __syncwarp();
  if (threadIdx.x < 4) C.u[threadIdx.x] += a.e[threadIdx.x];
  if (threadIdx.x == 0) {
    C.rosen = rosen;
    C.sel = a.sel;
    if (fail) C.cnt[RGPU_CNT_OVERLAP]++;
  }
  __syncwarp();
  return fail;
}

/* ------------------------------------------------------------------------ */
/* CBMC reinsertion of molecule m, ReinsertionAdsorbateMove src/mc_moves.c:4415-4600:
 * a new configuration is grown with m excluded (GrowMolecule, CBMC_INSERTION)
 * and the old one retraced (RetraceMolecule, CBMC_RETRACE_REINSERTION): the
 * old first bead alone, its weight completed with the new growth's other
 * first-bead trials (src/cbmc.c:750-762), and the old orientation among
 * nt - 1 fresh ones. Accepted with probability
 * exp(-beta dU_Fourier) W(new) / W(old).
 * Stage 1 holds the nf new first-bead trials, the old first bead and the
 * retrace orientations (all known up front), these in a stage of their own
 * where they do not fit (RGPU_MAX_POS positions); stage 2 the new
 * orientations around the chosen first bead; stage 3 the Ewald sum of both. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void accept_reinsert(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int na = S.natom;
  /* LJ-biasing corrections of both Rosenbluth weights, src/cbmc.c:3171-3178, :3044-3051 */
  const double rosen_new = C.rosen * cold_exp(-S.beta * (C.u[1] + C.u[3]));
  const double rosen_old = C.rosen_old * cold_exp(-S.beta * (C.uo[1] + C.uo[3]));
  double d_ads = 0.0, d_host = 0.0;
  if (has_ewald(S)) ewald_finish(S, C.ew[0], C.ew[1], S.excl_mol, S.excl_mol, 0, 0.0, d_ads, d_host);
  const double pacc = cold_exp(-S.beta * (d_ads + d_host)) * rosen_new / rosen_old;
  const bool accept = C.rnd[buf][SLOT_ACCEPT] < pacc;
  if (threadIdx.x == 0) {
    if (!(pacc == pacc)) C.status |= RGPU_ERR_NONFINITE;
    if (accept) {
      C.cnt[RGPU_CNT_REINS_ACCEPT]++;
      double u[4];
      for (int k = 0; k < 4; k++) u[k] = C.u[k] - C.uo[k];
      add_energies(C, 1.0, u, d_host, d_ads);
    }
  }
  if (accept) {
    if (threadIdx.x < na) {
      double p[3];
      chosen_atom(E, threadIdx.x, p);
      atom_store(E, cur().m, threadIdx.x, p);
    }
    accept_sites(E);
  }
}

/* the new configuration is chosen: its Ewald sum, or the acceptance */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD bool grown_reinsert(Build<MIXED, FLEX> E, int buf)
{
  if (has_ewald(fx().S)) {
    next_stage(E, PH_REINSEW, 0, 0, 2 * fx().S.natom);
    return false;
  }
  accept_reinsert(E, buf);
  return true;
}

/* the retrace orientations (trial 0 = the old one) at positions off.. of the
 * last evaluation complete the old configuration's weight and energies;
 * returns whether none is valid */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD bool old_orientations(Build<MIXED, FLEX> E, int off)
{
  Ctl &C = fx().C;
  const int nt = fx().S.ntrial;
  const Trials &b = C.tr[1];
  cbmc_trials(E, off, nt, fx().S.natom - 1, false, false, 0.0, &C.tr[1]);
  if (threadIdx.x < 4) C.uo[threadIdx.x] += b.e[threadIdx.x];
  if (threadIdx.x == 0) {
    C.rosen_old *= b.w_sum / (double)nt;
    if (!b.any) C.cnt[RGPU_CNT_OVERLAP]++;
  }
  __syncwarp();
  return !b.any;
}

template <int MIXED, bool FLEX>
__device__ __forceinline__ bool end_reinsert1(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int na = S.natom, nf = S.ntrial_first, nt = S.ntrial, nb = na - 1;
  const Trials &a = C.tr[0];
  cbmc_trials(E, 0, nf, 1, true, true, C.rnd[buf][SLOT_FIRST_SELECT], &C.tr[0]);
  /* the old first bead */
  const double4 r = fx().tot[nf];
  const bool ovo = r.x >= S.overlap || r.y >= S.overlap || r.z >= S.overlap || r.w >= S.overlap;
  const double w_old1 = ovo ? 0.0 : cold_exp(-S.beta * (r.x + r.z));
  const double rosen = a.w_sum / (double)nf;
  const bool fail = !a.any || rosen < 1e-150 || ovo;
  if (threadIdx.x == 0) {
    const double ro[4] = {r.x, r.y, r.z, r.w};
    C.rosen = rosen;
    C.rosen_old = (w_old1 + (a.w_sum - a.w_sel)) / (double)nf;
    C.sel = a.sel;
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
      C.u[k] = a.e[k];
      C.uo[k] = ro[k];
    }
    const BeadPos &p = fx().pos[a.sel];
    C.first[0] = p.x; C.first[1] = p.y; C.first[2] = p.z;
    if (fail) C.cnt[RGPU_CNT_OVERLAP]++;
  }
  __syncwarp();
  if (fail) return true;
  if (na == 1) return grown_reinsert(E, buf);
  const bool one = cur().one != 0;
  if (one && old_orientations(E, nf + 1)) return true;
  next_stage(E, one ? PH_REINS2 : PH_REINSOLD, nt * nb, 0, 0);
  return false;
}

/* after retrace orientations in a stage of their own; returns whether the
 * step is done */
template <int MIXED, bool FLEX>
__device__ __forceinline__ bool end_reinsert_old(Build<MIXED, FLEX> E)
{
  if (old_orientations(E, 0)) return true;
  next_stage(E, PH_REINS2, fx().S.ntrial * (fx().S.natom - 1), 0, 0);
  return false;
}

/* ------------------------------------------------------------------------ */
/* The bend angle and dihedral of trial t of bead i >= 2, as chain_trial
 * draws them, by a group of 8 lanes (lane8 = lane % 8; every lane of the
 * warp calls): lane8 l forms proposals l, l + 8, ... of the bend angle and
 * of the dihedral, and the lowest accepted proposal of each wins, so the
 * result is chain_trial's (its proposals are tried in order and the first
 * accepted one is taken). The draws need no bead position, so a whole
 * growth stage's angles are drawn at once, before its first bead. A group
 * with live = false only takes part in the warp's votes. */
__device__ __forceinline__ void chain_angles_group(const RgpuSys &S, int i, int stage, int t, bool live,
                                                   uint64_t step, int lane, double &theta, double &phi)
{
  auto U = [&](int d) { return rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, t, d)); };
  const int k = 3 * RGPU_CHAIN_TRIES, l8 = lane & 7;
  const unsigned gmask = 0xffu << (lane & ~7);
  theta = S.bend_theta0;
  phi = M_PI;
  bool th_done = !live, ph_done = !live || i < 3;
  if (live && i == 2) phi = 2.0 * M_PI * U(k) - M_PI;
  for (int base = 0; base < RGPU_CHAIN_TRIES; base += 8) {
    if (!__any_sync(RGPU_FULL, !(th_done && ph_done))) break;
    const int a = base + l8;
    double th = 0.0, f = 0.0;
    bool okt = false, okp = false;
    if (!th_done) {
      const double u1 = U(3 * a), u2 = U(3 * a + 1), u3 = U(3 * a + 2);
      th = S.bend_theta0 + S.bend_sigma * sqrt(-2.0 * log(1.0 - u1)) * cos(2.0 * M_PI * u2);
      okt = th > 0.0 && th < M_PI && u3 < sin(th);
    }
    if (!ph_done) {
      f = 2.0 * M_PI * U(k + 2 * a) - M_PI;
      okp = U(k + 2 * a + 1) < exp(-S.beta * (chain_torsion_energy(S, cos(f)) - S.torsion_min));
    }
    const unsigned bt = __ballot_sync(RGPU_FULL, okt) & gmask, bp = __ballot_sync(RGPU_FULL, okp) & gmask;
    const double ts = __shfl_sync(RGPU_FULL, th, bt ? __ffs(bt) - 1 : lane);
    const double fs = __shfl_sync(RGPU_FULL, f, bp ? __ffs(bp) - 1 : lane);
    if (!th_done && bt) {
      theta = ts;
      th_done = true;
    }
    if (!ph_done && bp) {
      phi = fs;
      ph_done = true;
    }
  }
}

/* The bend angle shared by the trials of bead i >= 2 in the reference's
 * scheme (chain_scheme 0): a growth draws it from sin(theta) exp(-beta
 * U_bend) (proposals in the slots of trial RGPU_REF_THETA_TRIAL from
 * RGPU_REF_THETA_SLOT on, tried in order: the lanes try 32 at once and the
 * lowest accepted wins), the distribution the reference's internal
 * Metropolis chain (src/cbmc.c:1822-2106) samples; a retrace (old !=
 * nullptr) keeps the old bead's angle. Every lane of the warp calls and
 * gets the angle. */
__device__ __noinline__ double chain_ref_theta(const RgpuSys &S, int i, int stage, uint64_t step, int lane,
                                                  const double (*old)[3])
{
  if (old) return chain_angle(old[i - 2], old[i - 1], old[i]);
  for (int base = 0; base < RGPU_CHAIN_TRIES; base += 32) {
    const int k = RGPU_REF_THETA_SLOT + 3 * (base + lane);
    auto U = [&](int d) { return rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, RGPU_REF_THETA_TRIAL, d)); };
    const double u1 = U(k), u2 = U(k + 1), u3 = U(k + 2);
    const double th = S.bend_theta0 + S.bend_sigma * sqrt(-2.0 * log(1.0 - u1)) * cos(2.0 * M_PI * u2);
    const unsigned ok = __ballot_sync(RGPU_FULL, th > 0.0 && th < M_PI && u3 < sin(th));
    if (ok) return __shfl_sync(RGPU_FULL, th, __ffs(ok) - 1);
  }
  return S.bend_theta0;
}

/* The reference's bonded trials (chain_scheme 0; GenerateTrialOrientationsMCScheme,
 * src/cbmc.c:1580-2480, for a linear chain) of trial t of bead i >= 2 with
 * the bead's bend angle theta, by one warp (every lane calls), into
 * a[0..4] (lane 0 writes):
 * - the dihedral: ntors uniform candidates (slot k of the trial), one chosen
 *   by its torsion Boltzmann factor with SelectTrialPosition's rule
 *   (src/cbmc.c:563-599, 2403-2408; one uniform in slot
 *   RGPU_REF_TORS_SEL_SLOT). Candidates 2p and 2p+1 come from one Philox
 *   block and belong to lane p % 32 of row p / 32; the cumulative sum runs
 *   row by row as warp scans. A retrace's trial 0 keeps the old dihedral as
 *   its candidate 0 and chooses it. Without a torsion (bead 2) the dihedral
 *   is uniform (src/cbmc.c:2410);
 * - the torsion Rosenbluth factor: the mean of exp(-beta U_torsion) over
 *   candidates 0 .. ntrial-1, the reference's ComputeNormalizedRosenbluthWeight
 *   (src/cbmc.c:542-552 sums up to the global NumberOfTrialPositions; called
 *   at :2401); 1 for bead 2. */
template <bool F32>
__device__ __noinline__ void chain_ref_trial(const RgpuSys &S, int i, int stage, int t, uint64_t step, int lane,
                                                const double (*old)[3], double theta, double *a)
{
  /* F32 (the mixed engine): the candidates' Boltzmann factors in FP32, the
   * chosen dihedral itself from its FP64 uniform as in FP64 */
  typedef typename std::conditional<F32, float, double>::type T;
  const bool keep_old = old && t == 0;
  double phi = 0.0, wt = 1.0;
  if (i == 2) {
    if (!keep_old) phi = 2.0 * M_PI * rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, t, 0)) - M_PI;
  } else {
    const int n = S.ntors, nt = S.ntrial, rows = (n + 63) >> 6;
    const T beta = (T)S.beta;
    const T p0 = (T)S.torsion[0], p1 = (T)S.torsion[1], p2 = (T)S.torsion[2], p3 = (T)S.torsion[3];
    T bf[RGPU_TORS_ROWS][2];
    T big = (T)-1e30, wsum = 0;
#pragma unroll
    for (int j = 0; j < RGPU_TORS_ROWS; j++) {
      const int k0 = 2 * (lane + 32 * j);
      bf[j][0] = bf[j][1] = (T)-1e30;
      if (j < rows && k0 < n) {
        double u[2];
        float uf[2];
        if (F32) {
          /* the leading 24 bits of the two FP64 uniforms of the block
           * (rgpu_uniform_pair: o[0] and o[2] head their 53 bits) */
          uint32_t o[4];
          rgpu_philox((uint32_t)step, (uint32_t)(step >> 32), chain_slot(stage, i, t, k0) >> 1, S.sys_id,
                      (uint32_t)S.seed, (uint32_t)(S.seed >> 32), o);
          uf[0] = (float)(o[0] >> 8) * 5.9604644775390625e-8f;   /* 2^-24 */
          uf[1] = (float)(o[2] >> 8) * 5.9604644775390625e-8f;
        } else {
          rgpu_uniform_pair(S.seed, S.sys_id, step, chain_slot(stage, i, t, k0) >> 1, u);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int k = k0 + h;
          if (k < n) {
            T c;
            if (keep_old && k == 0) c = (T)chain_cos_dihedral(old[i - 3], old[i - 2], old[i - 1], old[i]);
            else if (F32) c = (T)-cospif(2.0f * uf[h]);
            else c = (T)cos(2.0 * M_PI * u[h] - M_PI);
            if (F32) {
              /* chain_torsion_energy in FP32 */
              const T c2 = (T)2 * c * c - (T)1, c3 = c * ((T)4 * c * c - (T)3);
              bf[j][h] = -beta * (p0 + p1 * ((T)1 + c) + p2 * ((T)1 - c2) + p3 * ((T)1 + c3));
            } else {
              bf[j][h] = -beta * (T)chain_torsion_energy(S, (double)c);
            }
            big = big > bf[j][h] ? big : bf[j][h];
            if (k < nt) wsum += F32 ? (T)__expf((float)bf[j][h]) : (T)exp((double)bf[j][h]);
          }
        }
      }
    }
    for (int o = 16; o; o >>= 1) {
      const T ob = __shfl_xor_sync(RGPU_FULL, big, o);
      big = big > ob ? big : ob;
      wsum += __shfl_xor_sync(RGPU_FULL, wsum, o);
    }
    wt = (double)wsum / (double)nt;
    if (!keep_old) {
      /* the shifted factors, once: summed here, scanned below */
      T tot = 0;
#pragma unroll
      for (int j = 0; j < RGPU_TORS_ROWS; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const bool v = j < rows && 2 * (lane + 32 * j) + h < n;
          bf[j][h] = v ? (F32 ? (T)__expf((float)(bf[j][h] - big)) : (T)exp((double)(bf[j][h] - big))) : (T)0;
          tot += bf[j][h];
        }
      for (int o = 16; o; o >>= 1) tot += __shfl_xor_sync(RGPU_FULL, tot, o);
      const T target =
          (T)rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, t, RGPU_REF_TORS_SEL_SLOT)) * tot;
      /* the first candidate whose cumulative sum reaches the target, row
       * by row; none (rounding only): the last, where the serial search
       * stops */
      int kc = n - 1;
      T before = 0;
      bool done = false;
#pragma unroll
      for (int j = 0; j < RGPU_TORS_ROWS; j++) {
        if (!done && j < rows) {
          const int k0 = 2 * (lane + 32 * j);
          const T e0 = bf[j][0], e1 = bf[j][1];
          const T part = e0 + e1;
          T incl = part;
          for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(RGPU_FULL, incl, o);
            if (lane >= o) incl += y;
          }
          const T c0 = before + (incl - part) + e0;
          const int mine = (k0 < n && c0 >= target) ? k0 : ((k0 + 1 < n && c0 + e1 >= target) ? k0 + 1 : -1);
          const unsigned hit = __ballot_sync(RGPU_FULL, mine >= 0);
          if (hit) {
            kc = __shfl_sync(RGPU_FULL, mine, __ffs(hit) - 1);
            done = true;
          }
          before += __shfl_sync(RGPU_FULL, incl, 31);
        }
      }
      if (lane == 0) {
        const double uk = rgpu_uniform(S.seed, S.sys_id, step, chain_slot(stage, i, t, kc));
        if (F32) {
          /* phi = 2 pi u - pi: cos phi = -cospi(2u), sin phi = -sinpi(2u) */
          double sn, cs;
          sincospi(2.0 * uk, &sn, &cs);
          a[2] = -cs;
          a[3] = -sn;
          a[0] = cos(theta);
          a[1] = sin(theta);
          a[4] = wt;
          return;
        }
        phi = 2.0 * M_PI * uk - M_PI;
      }
    }
  }
  if (lane == 0) {
    a[0] = cos(theta);
    a[1] = sin(theta);
    a[2] = cos(phi);
    a[3] = sin(phi);
    a[4] = wt;
  }
}

/* The bend angles and dihedrals of beads 2.. of every trial of a growth
 * stage into `tab`, with each trial's torsion Rosenbluth factor. The
 * reference's scheme (S.chain_scheme 0): one warp per (bead, trial); a
 * retrace passes the old configuration `old` (published by a barrier
 * before the call). Independent draws (S.chain_scheme 1): 8 lanes per
 * (bead, trial), four per warp, and factor 1. The (bead, trial) tasks are
 * shared out over the warps of all CTAs of the cluster; after a cluster
 * barrier each CTA copies the other CTAs' rows from their shared memory.
 * All threads of the cluster call; the caller's next barrier publishes the
 * table. */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void chain_angles_table(Build<MIXED, FLEX> E, uint64_t step, int stage, double *tab,
                                                   const double (*old)[3], const double *ahead)
{
  const RgpuSys &S = fx().S;
  const int na = S.natom, nt = S.ntrial;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int ntask = na > 2 ? (na - 2) * nt : 0;
  const int gw = fx().rank * nw + (threadIdx.x >> 5), ngw = nw * fx().csize;   /* warp of the cluster */
  const int per = S.chain_scheme == 0 ? 1 : 4;                           /* tasks a warp takes at once */
  if (S.chain_scheme == 0) {
    /* each bead's bend angle once (a retrace's here, one warp per bead, in every
     * CTA; a growth's was drawn ahead), then one warp per (bead, trial); a
     * retrace's angles sit after the table */
    const double *theta = ahead;
    if (old) {
      double *th = tab + RGPU_ANG_TABLE;
      theta = th;
      for (int i = 2 + (threadIdx.x >> 5); i < na; i += nw) {
        const double v = chain_ref_theta(S, i, stage, step, lane, old);
        if (lane == 0) th[i] = v;
      }
      __syncthreads();
    }
    for (int task = gw; task < ntask; task += ngw) {
      const int i = 2 + task / nt, t = task % nt;
      chain_ref_trial<(MIXED != 0)>(S, i, stage, t, step, lane, old, theta[i],
                             tab + RGPU_ANG_STRIDE * ((i - 2) * RGPU_MAX_TRIALS + t));
    }
  } else {
    for (int t0 = gw * 4; t0 < ntask; t0 += ngw * 4) {
      const int task = t0 + (lane >> 3);
      const bool live = task < ntask;
      const int i = live ? 2 + task / nt : 2, t = live ? task % nt : 0;
      double th, ph;
      chain_angles_group(S, i, stage, t, live, step, lane, th, ph);
      if (live && (lane & 7) == 0) {
        double *a = tab + RGPU_ANG_STRIDE * ((i - 2) * RGPU_MAX_TRIALS + t);
        a[0] = cos(th);
        a[1] = sin(th);
        a[2] = cos(ph);
        a[3] = sin(ph);
        a[4] = 1.0;
      }
    }
  }
  if (fx().csize > 1) {
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    for (int task = threadIdx.x; task < ntask; task += blockDim.x) {
      const int owner = ((task / per) % ngw) / nw;
      if (owner == fx().rank) continue;
      const int off = RGPU_ANG_STRIDE * ((task / nt) * RGPU_MAX_TRIALS + task % nt);
      const double *src = cl.map_shared_rank(tab, owner) + off;
      for (int d = 0; d < RGPU_ANG_STRIDE; d++) tab[off + d] = src[d];
    }
    /* no CTA writes this table again before the next cluster barrier (the
     * evaluation that follows ends with one), so the peers' reads are done
     * by then */
  }
}

/* Beads of a retrace taken in one evaluation: from bead i0 on, as many as
 * fit `room` positions (at least one; room >= RGPU_MAX_TRIALS). */
__device__ __forceinline__ int retrace_group_end(int i0, int na, int nf, int nt, int room, int &P)
{
  int i1 = i0;
  P = 0;
  while (i1 < na && P + (i1 == 0 ? nf : nt) <= room) {
    P += i1 == 0 ? nf : nt;
    i1++;
  }
  return i1;
}

/* Bookkeeping of retrace beads [i0, i1) evaluated at positions off.. of
 * the last evaluation: warp w0 + g takes bead i0 + g (warps w0, w0 + 1, ... of the
 * block), sums its weights and leaves in C.rb[i] the sum,
 * the old bead's host and adsorbate VDW, intramolecular LJ and bonded
 * energy, and whether any trial was valid. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void retrace_book(Build<MIXED, FLEX> E, int i0, int i1, int off,
                                             const double (*old)[3], const double *ang, int w0)
{
  const RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int nf = S.ntrial_first, nt = S.ntrial;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (warp < w0) return;
  for (int g = warp - w0; g < i1 - i0; g += nw - w0) {
    const int i = i0 + g, k = i == 0 ? nf : nt;
    const int o0 = off + (i0 == 0 ? (i == 0 ? 0 : nf + (i - 1) * nt) : g * nt);
    double lj = 0.0, bf = 0.0;
    int ov = 0;
    const double4 rt = fx().tot[o0 + (lane < k ? lane : 0)];
    const double r[4] = {rt.x, rt.y, rt.z, rt.w};
    if (lane < k) {
      const BeadPos &q = fx().pos[o0 + lane];
      const double p[3] = {q.x, q.y, q.z};
      lj = chain_intra_lj(S, old, i, p);
      ov = r[0] >= S.overlap || r[1] >= S.overlap || r[2] >= S.overlap || r[3] >= S.overlap || lj >= S.overlap;
      bf = -S.beta * (r[0] + r[2] + lj);
    }
    const bool valid = lane < k && !ov;
    const double w = valid ? cold_exp(bf) : 0.0;
    const bool any = __ballot_sync(RGPU_FULL, valid) != 0u;
    const double wsum = warp_sum(w);
    if (lane == 0) {
      double *rb = C.rb[i];
      /* with the old trial's torsion Rosenbluth factor (1 for independent draws) */
      rb[0] = i >= 2 ? wsum * ang[RGPU_ANG_STRIDE * ((i - 2) * RGPU_MAX_TRIALS) + 4] : wsum;
      rb[1] = r[0];
      rb[2] = r[2];
      rb[3] = lj;
      rb[4] = i >= 2 ? chain_bonded_energy(S, old, i, old[i]) : 0.0;
      rb[5] = any ? 1.0 : 0.0;
    }
  }
}

/* Thread 0: the retrace beads [i0, i1) into the Rosenbluth weight and the
 * energies, in growth order, stopping at the first bead without a valid
 * trial. */
__device__ __forceinline__ void retrace_combine(Ctl &C, int i0, int i1, int nf, int nt)
{
  for (int i = i0; i < i1 && !C.fail; i++) {
    const double *rb = C.rb[i];
    C.rosen *= rb[0] / (double)(i == 0 ? nf : nt);
    C.u[0] += rb[1];
    C.u[2] += rb[2];
    C.uintra += rb[3];
    if (i >= 2) C.uintra += rb[4];
    if (rb[5] == 0.0) {
      C.fail = 1;
      C.cnt[RGPU_CNT_OVERLAP]++;
    }
  }
}

/* ------------------------------------------------------------------------ */
/* CBMC growth and retrace of a flexible chain, bead by bead from atom 0
 * (GrowMolecule / RetraceMolecule, src/cbmc.c:2928-3181, for a linear chain):
 * the first bead from nf trials (random in the box; for a retrace trial 0 is
 * the old bead), every other bead from nt trials of the stage's angle table.
 * The weight of a trial is exp(-beta (host VDW + adsorbate VDW + LJ with the
 * chain's beads four or more bonds back)); a trial overlaps when one of them
 * reaches the criterion. Ctl holds the Rosenbluth weight (product over beads
 * of sum w / trials), the chosen beads (cp), their host and adsorbate VDW
 * (u[0], u[2]) and the intramolecular energy (uintra: bonded + LJ).
 *
 * Growth: one stage per bead. Warp 0 selects a trial; meanwhile other warps
 * form what each trial would need if chosen (beside_grow): the next bead's
 * frame, the bonded energy (the chosen one's is added in the next stage) and
 * the next stage's description.
 *
 * Retrace: the beads it "chooses" are the old ones, known before anything is
 * evaluated, so the trial sets of several beads are placed together and
 * evaluated at once: beads are taken in growth order in groups whose trials
 * fit one evaluation (RGPU_MAX_POS positions; for 6 beads of 16 trials and 8
 * first-bead trials, two evaluations instead of six). Each bead's weights are
 * summed by one warp, and the Rosenbluth weight and the energies are combined
 * bead by bead in growth order, stopping at the first bead without a valid
 * trial, as the bead-by-bead retrace does. The trials draw the same random
 * numbers as that retrace (counter-based, by stage, bead and trial). A
 * reinsertion's retrace rides along with its growth's first evaluations, one
 * group each, in the positions after the growth's trials. */
/* the angle tables of a chain move: its growth's, or its retrace's; a
 * reinsertion's both. All threads call. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void chain_tables(Build<MIXED, FLEX> E, const Stage &g)
{
  Ctl &C = fx().C;
  const int mv = g.mv;
  const uint64_t step = fx().step0 + (uint64_t)g.it;
#pragma unroll 1
  for (int t = 0; t < (mv == 4 ? 2 : 1); t++) {
    const bool old = mv == 3 || t == 1;
    double (*x)[3] = t ? C.co : C.cp;
    if (old) {
      if (threadIdx.x < fx().S.natom) atom_xyz(E, g.m, threadIdx.x, x[threadIdx.x]);
      __syncthreads();          /* the old configuration, read by the table */
    }
    chain_angles_table(E, step, old ? 1 : 0, fx_ang() + t * RGPU_ANG_DOUBLES, old ? x : nullptr, fx().gr.theta[g.buf]);
  }
}

/* Stage for bead i of a growth (k trials), with
 * the retrace beads from r0 on that ride along (r0 = natom: none) */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void grow_stage(Build<MIXED, FLEX> E, Stage &n, const Stage &c, int i, int k, int r0)
{
  const RgpuSys &S = fx().S;
  int r1 = r0, rP = 0;
  if (r0 < S.natom) r1 = retrace_group_end(r0, S.natom, S.ntrial_first, S.ntrial, RGPU_MAX_POS - k, rP);
  fill_stage(E, n, c, PH_GROW, k + rP, 0, 0);
  if ((threadIdx.x & 31) == 0) {
    n.ci = i;
    n.k = k;
    n.r0 = r0;
    n.r1 = r1;
    n.rP = rP;
  }
}

/* stage for the retrace group of a deletion from bead i0 on */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void retrace_stage(Build<MIXED, FLEX> E, int i0)
{
  const RgpuSys &S = fx().S;
  int P;
  const int i1 = retrace_group_end(i0, S.natom, S.ntrial_first, S.ntrial, RGPU_MAX_POS, P);
  next_stage(E, PH_RETRACE, P, 0, 0);
  if (threadIdx.x == 0) {
    Stage &n = next_of();
    n.r0 = i0;
    n.r1 = i1;
    n.rP = P;
  }
}

/* warp 0, after the angle tables */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void end_table(Build<MIXED, FLEX> E)
{
  const RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int mv = cur().mv;
  if (threadIdx.x == 0) {
    C.rosen = 1.0;
    C.u[0] = C.u[1] = C.u[2] = C.u[3] = 0.0;
    C.uintra = 0.0;
    C.fail = 0;
  }
  if (mv == 3) {
    retrace_stage(E, 0);
    return;
  }
  grow_stage(E, next_of(), cur(), 0, S.ntrial_first, mv == 4 ? 0 : S.natom);
}

/* warp 0, after the trials of bead g.ci: returns whether the step is done
 * (the growth failed) */
template <int MIXED, bool FLEX>
__device__ __forceinline__ bool end_grow(Build<MIXED, FLEX> E, const Stage &g)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int i = g.ci, k = g.k, lane = threadIdx.x;
  double lj = 0.0, bf = 0.0;
  int ov = 0;
  const double4 rt = fx().tot[lane < k ? lane : 0];
  const double r[4] = {rt.x, rt.y, rt.z, rt.w};
  const BeadPos &q = fx().pos[lane];
  if (lane < k) {
    if (i >= 4) lj = fx().gr.lj[lane];
    ov = r[0] >= S.overlap || r[1] >= S.overlap || r[2] >= S.overlap || r[3] >= S.overlap || lj >= S.overlap;
    bf = -S.beta * (r[0] + r[2] + lj);
  }
  const bool valid = lane < k && !ov;
  const double w = valid ? cold_exp(bf) : 0.0;
  const bool any = __any_sync(RGPU_FULL, valid);
  const double cum = warp_scan(w), wsum = __shfl_sync(RGPU_FULL, cum, 31);
  int sel = 0;
  /* SelectTrialPosition (src/cbmc.c:563-599) on the weights themselves */
  if (any) sel = select_trial(w, cum, k, fx().gr.sel[g.buf][i]);
  const double hv = __shfl_sync(RGPU_FULL, r[0], sel), av = __shfl_sync(RGPU_FULL, r[2], sel);
  const double ljs = __shfl_sync(RGPU_FULL, lj, sel);
  /* with the chosen trial's torsion Rosenbluth factor (src/cbmc.c:2793; 1
   * for independent draws) */
  const double rosen =
      C.rosen * (wsum / (double)k * (i >= 2 ? fx_ang()[RGPU_ANG_STRIDE * ((i - 2) * RGPU_MAX_TRIALS + sel) + 4] : 1.0));
  const bool fail = !any || rosen < 1e-150;
  __syncwarp();
  if (lane == sel) {
    C.cp[i][0] = q.x;
    C.cp[i][1] = q.y;
    C.cp[i][2] = q.z;
  }
  if (lane == 0) {
    if (i - 1 >= 2) C.uintra += fx().gr.ub[(i - 1) & 1][C.sel];   /* the last bead's bonded energy (beside_grow) */
    C.rosen = rosen;
    C.u[0] += hv;
    C.u[2] += av;
    C.uintra += ljs;
    C.sel = sel;
    if (fail) C.cnt[RGPU_CNT_OVERLAP]++;
  }
  __syncwarp();
  return fail;
}

/* what the other warps do while warp 0 chooses among the trials of bead g.ci:
 * the bookkeeping of a riding retrace group, the frame that each trial would
 * give the next bead, the trials' bonded energies (warp 0 writes only
 * C.cp[ci]), the stage that follows a growth that did not fail */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void beside_grow(Build<MIXED, FLEX> E, Stage &n, const Stage &g)
{
  const RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, i = g.ci;
  if (g.r1 > g.r0) retrace_book(E, g.r0, g.r1, g.k, C.co, fx_ang() + RGPU_ANG_DOUBLES, 1);
  /* a warp each, as far as the block has them (warp 1 describes the next step) */
  if (w == (nw > 2 ? 2 : 1) && i >= 1 && lane < g.k) {
    const double p[3] = {fx().pos[lane].x, fx().pos[lane].y, fx().pos[lane].z};
    chain_frame(i >= 2 ? C.cp[i - 2] : nullptr, C.cp[i - 1], p, fx().gr.frame[lane]);
  }
  if (w == (nw > 3 ? 3 : 1) && i >= 2 && lane < g.k) {
    const double p[3] = {fx().pos[lane].x, fx().pos[lane].y, fx().pos[lane].z};
    fx().gr.ub[i & 1][lane] = chain_bonded_energy(S, C.cp, i, p);
  }
  if (w == (nw > 4 ? 4 : 1)) {
    __syncwarp();
    if (i + 1 < S.natom) grow_stage(E, n, g, i + 1, S.ntrial, g.r1);
    else fill_stage(E, n, g, PH_CHAINEND, 0, 0, 0);
  }
}

/* Acceptance of a chain insertion, deletion or Widom sample
 * (SwapAddAdsorbateMove src/mc_moves.c:7016, SwapRemoveAdsorbateMove :7228,
 * WidomAdsorbateMove :7844; uncharged chains, no Fourier part). */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void accept_swap_chain(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int na = S.natom, nmol = C.nmol, m = cur().m, mv = cur().mv;
  const bool insert = mv != 3, widom = mv == 5;
  double pacc;
  if (insert) pacc = C.rosen * S.fugacity_beta_v / (1.0 + nmol);
  else pacc = (double)nmol / (C.rosen * S.fugacity_beta_v);
  const bool accept = !widom && C.rnd[buf][SLOT_ACCEPT] < pacc;
  __syncwarp();
  if (threadIdx.x == 0) {
    if (!(pacc == pacc)) C.status |= RGPU_ERR_NONFINITE;
    if (widom) C.sums[RGPU_SUM_WIDOM_W] += C.rosen;
    if (accept) {
      C.cnt[RGPU_CNT_ACCEPT + mv]++;
      const double sgn = insert ? 1.0 : -1.0;
      C.energy[RGPU_E_HOST_VDW] += sgn * C.u[0];
      C.energy[RGPU_E_ADS_VDW] += sgn * C.u[2];
      C.energy[RGPU_E_INTRA] += sgn * C.uintra;
      C.nmol = insert ? nmol + 1 : nmol - 1;
      C.nads = C.nmol * na;
    }
  }
  if (accept && threadIdx.x < na) {
    if (insert) {
      atom_store(E, nmol, threadIdx.x, C.cp[threadIdx.x]);
    } else if (m != nmol - 1) {
      double p[3];
      atom_xyz(E, nmol - 1, threadIdx.x, p);
      atom_store(E, m, threadIdx.x, p);
    }
  }
}

/* CBMC reinsertion of a flexible chain (ReinsertionAdsorbateMove,
 * src/mc_moves.c:4415): a new configuration grown with molecule m left out,
 * the old one retraced; accepted with W(new) / W(old). The retrace's beads
 * are combined after a successful growth, as a retrace run after it would. */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void accept_reinsert_chain(Build<MIXED, FLEX> E, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  const int na = S.natom;
  bool accept = false;
  if (threadIdx.x == 0) {
    const double w_new = C.rosen, dl0 = C.u[0], dl2 = C.u[2], intra = C.uintra;
    C.rosen = 1.0;
    C.u[0] = C.u[1] = C.u[2] = C.u[3] = 0.0;
    C.uintra = 0.0;
    retrace_combine(C, 0, na, S.ntrial_first, S.ntrial);
    if (!C.fail) {
      const double pacc = w_new / C.rosen;
      if (!(pacc == pacc)) C.status |= RGPU_ERR_NONFINITE;
      accept = C.rnd[buf][SLOT_ACCEPT] < pacc;
      if (accept) {
        C.cnt[RGPU_CNT_REINS_ACCEPT]++;
        C.energy[RGPU_E_HOST_VDW] += dl0 - C.u[0];
        C.energy[RGPU_E_ADS_VDW] += dl2 - C.u[2];
        C.energy[RGPU_E_INTRA] += intra - C.uintra;
      }
    }
  }
  accept = __shfl_sync(RGPU_FULL, accept, 0);
  if (accept && threadIdx.x < na) atom_store(E, cur().m, threadIdx.x, C.cp[threadIdx.x]);
}

/* warp 0, after a growth's last bead */
template <int MIXED, bool FLEX>
__device__ __forceinline__ void end_chain(Build<MIXED, FLEX> E, int buf)
{
  Ctl &C = fx().C;
  const int last = fx().S.natom - 1;
  if (last >= 2 && threadIdx.x == 0) C.uintra += fx().gr.ub[last & 1][C.sel];
  __syncwarp();
  if (cur().mv == 4) accept_reinsert_chain(E, buf);
  else accept_swap_chain(E, buf);
}

/* warp 0, after a retrace group of a deletion: returns whether the step is
 * done */
template <int MIXED, bool FLEX>
__device__ __forceinline__ bool end_retrace(Build<MIXED, FLEX> E, const Stage &g, int buf)
{
  RgpuSys &S = fx().S;
  Ctl &C = fx().C;
  if (threadIdx.x == 0) retrace_combine(C, g.r0, g.r1, S.ntrial_first, S.ntrial);
  __syncwarp();
  if (C.fail) return true;
  if (g.r1 < S.natom) {
    retrace_stage(E, g.r1);
    return false;
  }
  accept_swap_chain(E, buf);
  return true;
}

/* ------------------------------------------------------------------------ */
/* The state after a step enters the ensemble sums (one thread, in the stage
 * that follows, before warp 0 changes it again) */
__device__ __forceinline__ void sample_step(Ctl &C)
{
  const double n = (double)C.nmol;
  const double u = C.energy[0] + C.energy[1] + C.energy[2] + C.energy[3] + C.energy[4] + C.energy[5] +
                   C.energy[RGPU_E_INTRA];
  C.sums[RGPU_SUM_SAMPLES] += 1.0;
  C.sums[RGPU_SUM_N] += n;
  C.sums[RGPU_SUM_N2] += n * n;
  C.sums[RGPU_SUM_U] += u;
  C.sums[RGPU_SUM_UN] += u * n;
  C.sums[RGPU_SUM_U2] += u * u;
}

/* counts the move that stage g opens (the same thread) */
__device__ __forceinline__ void count_step(Ctl &C, const Stage &g)
{
  const int mv = g.mv;
  const bool skip = g.ph == PH_SKIP;
  /* a displacement or reinsertion without a molecule is not counted (the
   * reference returns before counting); a swap or Widom move always is */
  if (skip && (mv <= 1 || mv == 4)) return;
  C.cnt[RGPU_CNT_MOVES]++;
  if (mv <= 3) C.cnt[RGPU_CNT_ATTEMPT + mv]++;
  if (mv == 4) C.cnt[RGPU_CNT_REINS_ATTEMPT]++;
  if (mv == 2 && skip) C.status |= RGPU_ERR_MAXMOL;
  if (mv == 5) C.sums[RGPU_SUM_WIDOM_N] += 1.0;   /* overlap samples count with weight 0 */
}

/* Describes in n the first stage of step `it` (random numbers in buffer buf),
 * which follows stage c, for the molecules there are now. One warp. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void start_step(Build<MIXED, FLEX> E, Stage &n, const Stage &c, long long it, int buf, long long nsteps,
                                     uint64_t step_end)
{
  const RgpuSys &S = fx().S;
  const Ctl &C = fx().C;
  const int na = S.natom, nf = S.ntrial_first, trials = S.ntrial * (na - 1);
  const int mv = C.mvn[buf], nmol = C.nmol;
  const int first = mv == 4 ? nf + 1 : nf;   /* first-bead positions */
  const bool end = !(it < nsteps && fx().step0 + (uint64_t)it < step_end);
  const bool ew = has_ewald(S), one = (mv == 3 || mv == 4) && first + trials <= RGPU_MAX_POS;
  int ph, P = 0, check = 0, ns = 0, m = nmol;
  if (mv != 2 && mv != 5) {
    m = (int)(C.rnd[buf][SLOT_MOLECULE] * nmol);
    if (m >= nmol) m = nmol - 1;
  }
  if (end) {
    ph = PH_END;
  } else if (mv <= 1 ? (nmol == 0 || (mv == 1 && na == 1)) : (mv == 2 ? nmol >= S.maxmol : mv != 5 && nmol == 0)) {
    ph = PH_SKIP;
  } else if (mv <= 1) {
    ph = PH_DISP;
    P = 2 * na;
    check = na;
    ns = ew ? 2 * na : 0;
  } else if (FLEX && S.flexible) {
    ph = PH_TABLE;       /* the chain moves begin with a stage that draws the angle tables */
  } else {
    ph = mv == 4 ? PH_REINS1 : PH_SWAP1;
    P = one ? first + trials : first;
    ns = mv == 3 && one && ew ? na : 0;
  }
  fill_stage(E, n, c, ph, P, check, ns);
  if ((threadIdx.x & 31) == 0) {
    n.mv = mv;
    n.m = m;
    n.one = one;
    n.buf = buf;
    n.it = it;
    n.first = !end;
    n.db = end ? -1 : (buf == 0 ? 2 : buf - 1);          /* (it + 2) mod 3 */
    n.dstep = fx().step0 + (uint64_t)it + 2;
  }
}

/* Warp 0 after stage c: the bookkeeping of its move, then the next stage, of
 * this step or of the next one. The latter warp 1 describes meanwhile for an
 * unchanged number of molecules (start_step into stage c + 2); that stands
 * unless the number has changed. */
template <int MIXED, bool FLEX>
__device__ RGPU_COLD void end_stage(Build<MIXED, FLEX> E, int c, long long nsteps, uint64_t step_end, uint64_t avg0)
{
  Ctl &C = fx().C;
  const Stage &g = C.st[c];
  const int ph = g.ph, buf = g.buf, nmol = C.nmol;
  if (threadIdx.x == 0) {
    C.cur = c;
    C.accept = 0;
  }
  __syncwarp();
  bool done = true;
  if (ph == PH_DISP) end_displace(E, buf);
  else if (ph == PH_SWAP1) done = end_swap1(E, buf);
  else if (ph == PH_SWAP2) done = add_orientations(E, g.mv != 3, buf) || grown_swap(E, buf);
  else if (ph == PH_SWAPEW) accept_swap(E, buf);
  else if (ph == PH_REINS1) done = end_reinsert1(E, buf);
  else if (ph == PH_REINSOLD) done = end_reinsert_old(E);
  else if (ph == PH_REINS2) done = add_orientations(E, true, buf) || grown_reinsert(E, buf);
  else if (ph == PH_REINSEW) accept_reinsert(E, buf);
  else if (FLEX && ph == PH_TABLE) { end_table(E); done = false; }
  else if (FLEX && ph == PH_GROW) done = end_grow(E, g);
  else if (FLEX && ph == PH_RETRACE) done = end_retrace(E, g, buf);
  else if (FLEX && ph == PH_CHAINEND) end_chain(E, buf);
  __syncwarp();
  int nx = stage_after(c, 1);
  if (done) {
    if (C.nmol == nmol) nx = stage_after(c, 2);
    else start_step(E, C.st[nx], g, g.it + 1, buf == 2 ? 0 : buf + 1, nsteps, step_end);
  }
  if (threadIdx.x == 0) {
    Stage &n = C.st[nx];
    n.ap = C.accept;
    n.sample = done && fx().step0 + (uint64_t)g.it >= avg0;
    if (done) C.it = g.it + 1;
    C.which = nx;
  }
}

/* ------------------------------------------------------------------------ */
/* Loads a descriptor copy into shared memory. */
__device__ __forceinline__ void load_sys(RgpuSys *dst, const RgpuSys *src)
{
  const uint32_t *s = (const uint32_t *)src;
  uint32_t *d = (uint32_t *)dst;
  for (int i = threadIdx.x; i < (int)(sizeof(RgpuSys) / 4); i += blockDim.x) d[i] = s[i];
  __syncthreads();
}

/* WIDE: compiled for CTAs of up to 1024 threads (64 registers per thread);
 * otherwise up to 512 threads with 128 registers. The engine picks WIDE for
 * CTAs above 512 threads and when several CTAs must share an SM. FLEX:
 * compiled with flexible-chain moves and energy grids; batches of rigid
 * molecules without grids run the build without them, whose register
 * allocation the chain and grid code does not touch. */
template <int MIXED, bool WIDE, bool FLEX>
__global__ void __launch_bounds__(WIDE ? 1024 : 512) rgpu_engine_kernel(RgpuSys *systems, int nsys, long long nsteps,
                                                                       int kw, int max_ads_atoms, int fw_items,
                                                                       int fwd_items, int tile_items, int k_items)
{
  extern __shared__ __align__(256) unsigned char smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  const int sysi = blockIdx.x / csize;
  const int nwarps = blockDim.x >> 5;
  const EngineLayout L = engine_layout(MIXED, fw_items, fwd_items, tile_items, max_ads_atoms, kw, k_items, nwarps, FLEX);
  if (sysi < nsys) {
    Eng<MIXED, FLEX> E;
    const Build<MIXED, FLEX> B;
    E.rank = rank;
    E.csize = csize;
    E.xb = 0;
    E.sc.u = fx().u;
    E.sc.qr2 = MIXED ? (float *)(smem + L.q) : nullptr;
    E.sc.qq = MIXED == 2 ? E.sc.qr2 + nwarps * 128 : nullptr;
    E.sc.qt = MIXED == 2 ? (int *)(E.sc.qq + nwarps * 64) : (MIXED ? nullptr : (int *)(smem + L.q));
    E.tab = (typename PhaseT<MIXED>::T *)(smem + L.tab);
    E.kw = kw;
    Ctl &C = fx().C;
    E.sc.cnt = &C.wcnt[0][0];
    E.sc.next = &C.next;
    E.sc.done = C.done;
    RgpuSys &S = fx().S;
    load_sys(&S, &systems[sysi]);
    /* a system at its step limit (a finished job left in its slot) takes
     * no step in this launch: its CTAs leave before staging anything and
     * write nothing back. All CTAs of the cluster read the same limits, so
     * the whole cluster leaves and none waits at the cluster barrier below. */
    if (S.step[0] >= S.step[1]) return;
    double2 *sk_global = S.sk_ads;
    if (threadIdx.x < 3 * RGPU_MAX_WARPS) (&C.wcnt[0][0])[threadIdx.x] = 0ULL;
    if (blockDim.x < 3 * RGPU_MAX_WARPS && threadIdx.x < 32) (&C.wcnt[0][0])[64 + threadIdx.x] = 0ULL;
    if (threadIdx.x < RGPU_MAX_POS) C.done[threadIdx.x] = 0;   /* blocks have at least 64 threads */
    if (threadIdx.x < RGPU_NCNT) C.cnt[threadIdx.x] = 0;
    if (threadIdx.x < RGPU_NE) C.energy[threadIdx.x] = S.energy[threadIdx.x];
    if (threadIdx.x == 0) {
      C.cyc[0] = C.cyc[1] = 0;
      C.work[0] = C.work[1] = 0ULL;
      C.status = 0;
      C.next = 0;
      C.ovf[0] = C.ovf[1] = 0;
      C.nextk = C.ewdone = 0;
      Fixed &F = fx();
      F.step0 = S.step[0];
      F.ads = (unsigned)L.ads;
      F.ang = (unsigned)L.ang;
      F.rank = rank;
      F.csize = csize;
      C.it = 0;
      C.cur = 0;
      C.which = 0;
      C.accept = 0;
      for (int k = 0; k < RGPU_NSUM; k++) C.sums[k] = 0.0;
      C.nmol = *S.nmol;
      C.nads = C.nmol * S.natom;
    }
    /* this CTA's framework share, staged in shared memory when it fits
     * (smem_fw 1: fixed-point atoms and tiles; 2: FP64 positions too) */
    {
      int t0, t1;
      share(S.ntile, rank, csize, t0, t1);
      E.sl.fw_lo = t0;
      E.sl.fw_hi = t1;
      E.sl.fw = S.fw32;
      E.sl.tiles = S.tiles;
      E.sl.fwd = MIXED ? nullptr : S.fw64t;
      if (S.smem_fw) {
        int4 *dfw = (int4 *)(smem + L.fw);
        TileRec *dt = (TileRec *)(smem + L.tiles);
        for (int i = threadIdx.x; i < (t1 - t0) * RGPU_TILE; i += blockDim.x) dfw[i] = S.fw32[t0 * RGPU_TILE + i];
        for (int i = threadIdx.x; i < t1 - t0; i += blockDim.x) dt[i] = S.tiles[t0 + i];
        E.sl.fw = dfw - (size_t)t0 * RGPU_TILE;
        E.sl.tiles = dt - t0;
      }
      if (!MIXED && S.smem_fw > 1) {
        double4 *d = (double4 *)(smem + L.fwd);
        for (int i = threadIdx.x; i < (t1 - t0) * RGPU_TILE; i += blockDim.x) d[i] = S.fw64t[t0 * RGPU_TILE + i];
        E.sl.fwd = d - (size_t)t0 * RGPU_TILE;
      }
    }
    E.sl.ads = smem + L.ads;
    if (FLEX && S.use_grid) E.sl.fw_hi = E.sl.fw_lo;   /* host VDW from the grids: no framework pairs */
    /* this CTA's wave vectors with their prefactors and S(k) */
    if (S.ewald) share(S.nk, rank, csize, E.k0, E.k1);
    else { E.k0 = 0; E.k1 = 0; }
    const bool k_smem = k_items >= E.k1 - E.k0;
    __syncthreads();
    if (k_smem && E.k1 > E.k0) {
      char4 *kv = (char4 *)(smem + L.kvec);
      double *kf = (double *)(smem + L.kf);
      double2 *sf = (double2 *)(smem + L.skfw);
      double2 *sa = (double2 *)(smem + L.skads);
      for (int i = threadIdx.x; i < E.k1 - E.k0; i += blockDim.x) {
        kv[i] = S.kvec[E.k0 + i];
        kf[i] = S.kfactor[E.k0 + i];
        sf[i] = S.sk_fw[E.k0 + i];
        sa[i] = S.sk_ads[E.k0 + i];
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        S.kvec = kv - E.k0;
        S.kfactor = kf - E.k0;
        S.sk_fw = sf - E.k0;
        S.sk_ads = sa - E.k0;
      }
    }
    /* adsorbate records to shared memory (full copy in every CTA) */
    for (int i = threadIdx.x; i < C.nads; i += blockDim.x) {
      const int mm = i / S.natom, a = i - mm * S.natom;
      const double *x = S.ads_xyz + 3 * i;
      if (MIXED) {
        int xi, yi, zi;
        rgpu_fix3(S, x[0], x[1], x[2], xi, yi, zi);
        ((int4 *)(smem + L.ads))[i] = make_int4(xi, yi, zi, mm * 16 + a);
      } else
        atom_store(B, mm, a, x);
    }
    __syncthreads();
    E.step0 = S.step[0];
    const uint64_t step_end = S.step[1], avg0 = S.step[2];
    const long long t_start = clock64();
    draw_step(B, E.step0, 0, threadIdx.x, blockDim.x);
    draw_step(B, E.step0 + 1, 1, threadIdx.x, blockDim.x);
    __syncthreads();
    if (threadIdx.x < 32) start_step(B, C.st[0], C.st[2], 0, 0, nsteps, step_end);
    if (threadIdx.x == 0) {
      C.st[0].ap = 0;
      C.st[0].sample = 0;
    }
    for (;;) {
      __syncthreads();            /* the stage that warp 0 described */
      const int c = C.which;
      const Stage &g = C.st[c];
      if (threadIdx.x == blockDim.x - 1) {
        if (g.sample) sample_step(C);
        if (g.first) count_step(C, g);
      }
      const int np = g.P + (g.ph == PH_DISP ? 0 : g.ns);
      if (np) {
        for (int i = threadIdx.x; i < np; i += blockDim.x) place(B, g, i);
        __syncthreads();
        eval_stage(E, g);
      } else {
        if (g.ap)
          ewald_share<MIXED>(S, E.tab, E.kw, nullptr, 0, true, E.k0, E.k1, threadIdx.x >> 5, nullptr);
        if (g.ph == PH_END) break;
        if (FLEX && g.ph == PH_TABLE) chain_tables(B, g);
        __syncthreads();          /* also: every thread knows the stage before warp 0 names the next */
      }
      if (FLEX && g.ph == PH_RETRACE) {
        retrace_book(B, g.r0, g.r1, 0, C.cp, fx_ang(), 0);
        __syncthreads();
      }
      if (threadIdx.x < 32) {
        end_stage(B, c, nsteps, step_end, avg0);
      } else {
        /* warp 1: the next step's first stage, should this stage end its step */
        if (threadIdx.x < 64 && g.ph != PH_TABLE)
          start_step(B, C.st[stage_after(c, 2)], g, g.it + 1, g.buf == 2 ? 0 : g.buf + 1, nsteps, step_end);
        if (FLEX && g.ph == PH_GROW) beside_grow(B, C.st[stage_after(c, 1)], g);
        if (g.db >= 0) draw_step(B, g.dstep, g.db, blockDim.x - 1 - threadIdx.x, blockDim.x - 32);
      }
    }
    const long long it = C.it;
    __syncthreads();
    /* write back: positions, molecule count, energies, counters (rank 0);
     * this CTA's share of S(k) and its work counters (every CTA) */
    if (k_smem)
      for (int k = E.k0 + threadIdx.x; k < E.k1; k += blockDim.x) sk_global[k] = S.sk_ads[k];
    if (rank == 0) {
      /* FP64 positions (the mixed path keeps them in global memory already) */
      for (int i = threadIdx.x; !MIXED && i < C.nads; i += blockDim.x) {
        const int mm = i / S.natom, a = i - mm * S.natom;
        double p[3];
        atom_xyz(B, mm, a, p);
        S.ads_xyz[3 * i] = p[0];
        S.ads_xyz[3 * i + 1] = p[1];
        S.ads_xyz[3 * i + 2] = p[2];
      }
      if (threadIdx.x < RGPU_NE) S.energy[threadIdx.x] = C.energy[threadIdx.x];
      if (threadIdx.x == 0) {
        *S.nmol = C.nmol;
        S.step[0] = E.step0 + (uint64_t)it;
        for (int k = 0; k < RGPU_NSUM; k++) S.sums[k] += C.sums[k];
        for (int c = 0; c < RGPU_CNT_PAIRS; c++) S.counters[c] += C.cnt[c];
        S.counters[RGPU_CNT_REINS_ATTEMPT] += C.cnt[RGPU_CNT_REINS_ATTEMPT];
        S.counters[RGPU_CNT_REINS_ACCEPT] += C.cnt[RGPU_CNT_REINS_ACCEPT];
        *S.status |= C.status;
        S.counters[RGPU_CNT_CYCLES] += clock64() - t_start;
        S.counters[RGPU_CNT_CYC_EVAL] += C.cyc[0];
        S.counters[RGPU_CNT_CYC_EWALD] += C.cyc[1];
      }
    }
    if (threadIdx.x < 5) {
      unsigned long long v = 0;
      if (threadIdx.x < 3)
        for (int w = 0; w < nwarps; w++) v += C.wcnt[w][threadIdx.x];
      else
        v = C.work[threadIdx.x - 3];
      atomicAdd((unsigned long long *)&S.counters[RGPU_CNT_PAIRS + threadIdx.x], v);
    }
  }
  /* no CTA may leave while a peer can still read its shared memory */
  cl.sync();
}

/* the kernel build for (mixed, wide, flex) */
using EngineKernel = void (*)(RgpuSys *, int, long long, int, int, int, int, int, int);
static EngineKernel engine_kernel(int mixed, bool wide, bool flex)
{
  if (mixed == 2) return wide ? rgpu_engine_kernel<2, true, false> : rgpu_engine_kernel<2, false, false>;
  if (mixed && wide) return flex ? rgpu_engine_kernel<1, true, true> : rgpu_engine_kernel<1, true, false>;
  if (mixed) return flex ? rgpu_engine_kernel<1, false, true> : rgpu_engine_kernel<1, false, false>;
  return flex ? rgpu_engine_kernel<0, false, true> : rgpu_engine_kernel<0, false, false>;
}

cudaError_t rgpu_engine_prepare(int mixed, bool wide, bool flex, size_t smem)
{
  return cudaFuncSetAttribute(engine_kernel(mixed, wide, flex), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

cudaError_t rgpu_engine_launch(int mixed, RgpuSys *d_systems, int nsys, long long nsteps, int kw,
                               int max_ads_atoms, int fw_items, int fwd_items, int tile_items, int k_items, int cluster,
                               int threads, bool wide, bool flex, cudaStream_t st)
{
  size_t smem = rgpu_engine_smem_bytes(mixed, fw_items, fwd_items, tile_items, max_ads_atoms, kw, k_items, threads, flex);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nsys * cluster), 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  /* the dynamic shared-memory limit is raised by rgpu_engine_prepare, outside
   * any stream capture */
  return cudaLaunchKernelEx(&cfg, engine_kernel(mixed, wide, flex), d_systems, nsys, nsteps, kw, max_ads_atoms,
                            fw_items, fwd_items, tile_items, k_items);
}

/* Batched state transfer of an engine's systems through one staging buffer:
 * system i's region starts at off[i] (8-byte aligned) and holds its state
 * block (RgpuState; for an upload only its nmol field is read), then
 * nmol * natom positions (FP64 xyz). One block per system. */
__global__ void k_gather_states(const RgpuSys *systems, const unsigned long long *off, unsigned char *buf)
{
  const RgpuSys &S = systems[blockIdx.x];
  unsigned char *dst = buf + off[blockIdx.x];
  const RgpuState *st = (const RgpuState *)S.energy;   /* energy is the first field of the block */
  const unsigned long long *src8 = (const unsigned long long *)st;
  unsigned long long *dst8 = (unsigned long long *)dst;
  for (int i = threadIdx.x; i < (int)(sizeof(RgpuState) / 8); i += blockDim.x) dst8[i] = src8[i];
  const int n = st->nmol * S.natom * 3;
  double *xd = (double *)(dst + sizeof(RgpuState));
  for (int i = threadIdx.x; i < n; i += blockDim.x) xd[i] = S.ads_xyz[i];
}

/* with the per-call records of the positions */
__global__ void k_scatter_positions(const RgpuSys *systems, const unsigned long long *off, const unsigned char *buf)
{
  const RgpuSys &S = systems[blockIdx.x];
  const unsigned char *src = buf + off[blockIdx.x];
  const int nmol = ((const RgpuState *)src)->nmol;
  const double *xs = (const double *)(src + sizeof(RgpuState));
  for (int i = threadIdx.x; i < nmol * S.natom * 3; i += blockDim.x) S.ads_xyz[i] = xs[i];
  if (threadIdx.x == 0) *S.nmol = nmol;
  const int na = S.natom;
  for (int i = threadIdx.x; i < nmol * na; i += blockDim.x) {
    const int m = i / na, a = i - m * na;
    const double x = xs[3 * i], y = xs[3 * i + 1], z = xs[3 * i + 2];
    int xi, yi, zi;
    rgpu_fix3(S, x, y, z, xi, yi, zi);
    S.rec32[i] = make_int4(xi, yi, zi, m * 16 + a);
    AdsRec64 r;
    r.x = x; r.y = y; r.z = z; r.tag = m * 16 + a;
    ((AdsRec64 *)S.rec64)[i] = r;
  }
}

cudaError_t rgpu_gather_states_launch(const RgpuSys *d_systems, int n, const unsigned long long *d_off,
                                      unsigned char *d_buf, cudaStream_t st)
{
  if (n <= 0) return cudaSuccess;
  k_gather_states<<<n, 256, 0, st>>>(d_systems, d_off, d_buf);
  return cudaGetLastError();
}

cudaError_t rgpu_scatter_positions_launch(const RgpuSys *d_systems, int n, const unsigned long long *d_off,
                                          const unsigned char *d_buf, cudaStream_t st)
{
  if (n <= 0) return cudaSuccess;
  k_scatter_positions<<<n, 256, 0, st>>>(d_systems, d_off, d_buf);
  return cudaGetLastError();
}
