// md_common.cuh -- shared definitions of the GB300 kernels.
//
// Unit system of the device kernels (both precisions): lengths in units of
// the box length L, magnetic moments in units of mu_u = max_i |mu_i|.  Then
// a real-space term like a3 ~ 1/r^7 stays inside FP32 range (it would
// overflow in SI units), and the results convert to SI with
//   B_unit = facEwald * mu_u / L^3        [T]
//   F_unit = facEwald * mu_u^2 / L^4      [N].
// All Ewald formulas are those of the reference (src/interaction.cpp:353-674)
// rewritten in these units; the conversion factors are applied once per
// particle in the integrator.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "md_types.h"

namespace md {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

template <typename T> struct V4;
template <> struct V4<float> { using t = float4; };
template <> struct V4<double> { using t = double4_32a; };
template <typename T> struct V2;
template <> struct V2<float> { using t = float2; };
template <> struct V2<double> { using t = double2; };

// ------------------------------------------------------------ cell list
// Sorted particle data (cell order).  Written by the cell-list build and,
// for the moments, by the integrator between the two Heun stages.
struct SortedView {
  float4* xf;     // box coordinates (float) + rMag/L: candidate test
  int4* xi;       // fixed-point box coordinates (2^32 per L) + particle index
  double4_32a* xd;  // box coordinates (double) + rMag/L (FP64 path)
  void* mu;       // T4: moment / mu_u, .w = rMag / L
  int* cell;      // cell id of the sorted slot
  int* perm;      // sorted slot -> particle index
  int* rank;      // particle index -> sorted slot
  int* cell_start;  // [ncell + 1]
};

// Per-step control words in device memory (written by the step's own kernels,
// so one captured graph serves every step).
struct StepFlags {
  int rebuild;        // this step rebuilds the cell list and neighbour list
  int overflow;       // the neighbour list did not fit: real space scans cells
  int force;          // host request: rebuild on the next step
  unsigned maxdisp;   // float bits of the largest displacement since the build (box units)
  int refill;         // a neighbour list was longer than its share: the lists lie one after another
  int soverflow;      // the strong-pair list did not fit: every pair stays on the FP32 path
};

// Cell-list build of one system (positions in particle order, FP64).
// The mesh's bricks as the cell order sees them (md_mesh.cuh; M = 0: none).
struct MeshGrid {
  int M, ncx, nbrick, nitem;
  float reach;  // distance a particle may be from the cell it is filed in, box units
  int* plan;
};

struct CellParams {
  int n;
  double invL;
  CellGrid grid;
  float half_skin;          // rebuild threshold: half the list skin, box units
  const double* pos;
  const double* mm;
  const double* magMom_u;
  const double* rMag_u;
  int* cellOf;
  int* count;               // [ncell] zero between builds
  int* tmp;
  SortedView s;
  double* xbuild;           // positions at the last build (may be null)
  StepFlags* flags;
  MeshGrid mesh;
};

// A packed launch runs one kernel over the blocks of several independent
// systems: block b of the grid executes block tasks[b].blk of system
// tasks[b].rep, with that system's parameters.  A system's results in a batch do
// not depend on what else is in it; a context's own calls may take another engine
// (small and large systems, md_kspace_engine_used) and agree within rounding.
struct Task {
  int rep, blk;
};

// Work queue of one persistent packed launch: blocks claim tasks in turn
// (atomic ticket), and the last block to finish resets the counters for the
// next launch (the next replay of the step graph).  Which block runs a task
// does not change the task's result.
struct WorkQ {
  unsigned next, done;
};

// Task loop of a persistent packed kernel: body(t) for every task claimed by
// this block; SYNC adds a block barrier after each task (kernels whose tasks
// use shared memory).
template <bool SYNC, typename F>
__device__ __forceinline__ void for_tasks(const Task* __restrict__ tk, int ntask, WorkQ* wq, F&& body) {
  __shared__ int s_task;
  for (;;) {
    if (threadIdx.x == 0) s_task = (int)atomicAdd(&wq->next, 1u);
    __syncthreads();
    const int q = s_task;
    __syncthreads();  // every thread has read the ticket before thread 0 takes the next
    if (q >= ntask) break;
    body(tk[q]);
    if (SYNC) __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&wq->done, 1u) == gridDim.x - 1) {  // all blocks have stopped claiming
      wq->next = 0;
      wq->done = 0;
      __threadfence();
    }
  }
}

// ------------------------------------------------------- real space
// FP32 loop constants of the packed pair terms (mixed path), computed once on
// the host: the pair loop reads them from the kernel parameters, so nothing
// in it is recomputed from the FP64 fields (GB300's FP64 rate is ~1/64 of
// FP32).  Pair vectors arrive in the fixed-point unit (2^-32 box lengths):
// d_fix = 2^32 d, r2f = 2^64 r^2; the unit scale and the exp -> 2^x
// conversion are folded into the factors.
struct PairK {
  float ke;          // -alpha^2 log2(e): exp(-alpha^2 r^2) = 2^(ke r^2)
  float kz;          // 0.42 alpha: the erfcx fit's denominator 1 + kz r
  float c2an;        // -2 alpha / sqrt(pi)
  float a2a, a2t;    // a2 2^-32 = a2a (-a1) / r^2 + a2t (-t), t the Gaussian term
  float a3a, a3t;    // -a3 2^-96 = a3a (a2 2^-32) / r^2 + a3t (-t)
  float a2fa, a2ft;  // a2 2^-64 of the field-only pass
  float eps;         // contact offset
  float rc2f;        // rc^2 2^64: the cutoff test on r2f
};

// erfcx(z) = exp(z^2) erfc(z) on the mixed path: t Q(t) with t = 1 / (1 + 0.42 z)
// and Q of degree 7, a minimax fit (weighted least squares on Chebyshev nodes,
// Lawson's iteration) over 0 <= z <= 5: relative error 3.2e-8 there, 5e-7 at
// z = 8 (where exp(-z^2) is 1e-28).  One polynomial and no second exponential:
// Numerical Recipes' erfcc = t exp(-z^2 + P(t)), used before, is of degree 9
// with an error of 1.0e-7.
constexpr float kErfcxA = 0.42f;
__host__ __device__ constexpr float erfcx_c(int k) {
  return k == 0   ? 0.2367379418f
         : k == 1 ? 0.240826718f
         : k == 2 ? 0.1874095252f
         : k == 3 ? 0.2917243134f
         : k == 4 ? -0.1721644463f
         : k == 5 ? 0.4843077908f
         : k == 6 ? -0.34481585f
                  : 0.07597403895f;
}

inline PairK make_pair_consts(double alpha, double c2a, double cont_eps, double rc2) {
  const double s32 = 2.3283064365386963e-10, s64 = s32 * s32;  // 2^-32, 2^-64
  const double al2 = alpha * alpha;
  PairK k;
  k.ke = (float)(-al2 * 1.4426950408889634);
  k.kz = (float)((double)kErfcxA * alpha);
  k.c2an = (float)-c2a;
  k.a2a = (float)(-3.0 * s32);
  k.a2t = (float)(-2.0 * al2 * s32);
  k.a3a = (float)(-5.0 * s64);
  k.a3t = (float)(4.0 * al2 * al2 * s32 * s64);
  k.a2fa = (float)(-3.0 * s64);
  k.a2ft = (float)(-2.0 * al2 * s64);
  k.eps = (float)cont_eps;
  k.rc2f = (float)(rc2 * 18446744073709551616.0);
  return k;
}

struct RealParams {
  int n;
  const double* gtab;   // FP64 pair-term tables (real_tables64): [kGIntervals][8]
  const double2* etab;  //   and [kEEntries]
  CellGrid grid;
  double alpha, rc;      // box units
  double rc2;
  double c2a;            // 2 alpha / sqrt(pi)
  double al2, al4;       // alpha^2, alpha^4
  double cont_eps;       // 1e-10 m / L (contact offset, interaction.cpp:120)
  PairK pk;              // FP32 constants of the packed pair terms
  // coating potentials (src/interaction.cpp:766-832), box units / F_unit
  int coat;
  double rcut_sr2;       // (rCutSR / L)^2
  double eff_len;        // effLenSurfMol / L
  double ster, elec, kappa, vdw;  // scaled prefactors
  const double* rMag_u;  // rMag / L by particle index (coating potentials)
  SortedView s;
  void* B;      // [3][n] T, sorted order
  void* F;      // [3][n] T, sorted order (FULL only)
  void* ov;     // [3][n] T, overlap displacement, box units (FULL only)
  double* Ppart;  // [n][3] per-particle pressure sums (FULL only)
  int* err;       // device error word
  // Verlet neighbour list (sorted indices) with a skin: rebuilt when a
  // particle has moved more than skin/2 since the last build.
  double rl2;                 // (rc + skin)^2, box units
  int* nbr;                   // [cap] neighbour indices
  int* nbr_cnt;               // [n]
  int* nbr_off;               // [n + 1]
  long long nbr_cap;
  int nbr_share;              // entries per list while every list fits that many (nbr_cap / n)
  StepFlags* flags;           // rebuild / overflow
  // Strong pairs (mixed path): list entries with |mu_i|^2 |mu_j|^2 >
  // strong_w4sq r^8 at the build (box units, moments in mu_max) carry the
  // sign bit in nbr, are left out of the FP32 field, force and pressure sums
  // (the FP32 pass still pushes them apart when they overlap) and are
  // evaluated in FP64 from the list snbr by the same kernel's warps, one
  // term set per entry into svals; the integrator adds each particle's
  // entries (StrongView).
  int strong;                 // 1: classify at builds and honour the flags
  float strong_w4sq;
  int2* snbr;                 // [scap] (i, j) sorted indices, grouped by i
  int* snbr_cnt;              // [n]
  int* snbr_off;              // [n + 1]
  long long scap;
  double* svals;              // [3][scap] B (+ [3][scap] F, [3][scap] P when FULL) per entry
  // moments of the strong entries: FP64 master directions x |mu| / mu_max
  // (particle order, via s.perm) when the evaluated moments are the master
  // state; null: the sorted view's (FP32 stage moments, exact there)
  const double* smm;
  const double* smag;
};

// The FP64 strong-pair terms of one evaluation, as the integrator reads
// them.  The real-space kernel stores, per 32-entry chunk of the strong list
// and owner particle, the owner's field and force sums at its first entry in
// the chunk, and the chunk's pressure sum at the chunk's first entry.  Slot
// r (entries off[r] .. off[r + 1]) thus adds its partials at off[r] and at
// every chunk start inside its range, in that fixed order; the pressure
// partial of a chunk belongs to the owner of the chunk's first entry.
// off == nullptr: the path is off; the flags say whether the list of the
// last build is in use.
struct StrongView {
  const int* off;
  long long cap;
  const double* B;  // [3][cap] (field of the evaluation)
  const double* F;  // [3][cap] (force, full evaluation)
  const double* P;  // [3][cap] (pressure, full evaluation)
  const StepFlags* flags;
  __device__ __forceinline__ bool usable() const { return off && !flags->overflow && !flags->soverflow; }
  // sums of the 3-component arrays a (and b when given) over slot r's
  // partials; pc: the pressure partials of the chunks slot r starts
  __device__ __forceinline__ bool sums(int r, const double* a, double oa[3], const double* b = nullptr,
                                       double* ob = nullptr, const double* pc = nullptr, double* op = nullptr) const {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      oa[q] = 0.0;
      if (ob) ob[q] = 0.0;
      if (op) op[q] = 0.0;
    }
    if (!usable() || !a) return false;
    const int e0 = max(off[r], 0), e1 = (int)min((long long)off[r + 1], cap);
    if (e0 >= e1) return false;
    for (int e = e0; e < e1; e = (e & ~31) + 32) {
#pragma unroll
      for (int q = 0; q < 3; q++) {
        oa[q] += a[q * cap + e];
        if (b) ob[q] += b[q * cap + e];
        if (pc && (e & 31) == 0) op[q] += pc[q * cap + e];
      }
    }
    return true;
  }
  __device__ __forceinline__ bool sum3(const double* a, int r, double out[3]) const { return sums(r, a, out); }
};

// --------------------------------------------------------- k space
struct KParams {
  int n;
  int kc;
  int nseg, nk;          // segments, padded k count
  int chunk;             // particles per chunk of the structure-factor grid
  int nchunk;
  double two_pi;         // 2 * my_pi (FP64 phases follow the reference's pi)
  const KSeg* seg;       // [nseg] sorted by len (desc): structure-factor threads
  const int* koff;       // [nseg] k index of the segment's first k (sorted order)
  const double* ek;      // [nk] 2 exp(-w n^2) / n^2 (0 for padding), sorted order
  const KSeg* rseg;      // [nseg] the same segments in row order (nz, ny ascending)
  const int* rowpos;     // [nk] sorted k index -> row-order k index
  const int2* chunks;    // [nchk + 1] (first row segment, first row-order k)
  int nchk;              // chunks of <= kKChunk row-order k's (scatter staging)
  double2* Spart;        // [nchunk][nk] partial structure factors
  double* musum_part;    // [nchunk][3]
  double* musum;         // [3]
  void* eS;              // [nk] T2: e(k) * (Sc, Ss)
  double2* S;            // [nk] full structure factor (debug / FP64)
  void* tab;             // [n][3][kc + 1] T2 phase tables of the sorted particles
  double cflux, cforce;  // 4 pi, 8 pi^2 (box units)
  SortedView s;
  void* B;   // [3][n] T sorted
  void* F;   // [3][n] T sorted (FULL only)
  // Tensor-core engine (mixed path): k rows r = (ny, nz), each with nx in
  // [-kc, kc] (column q = nx + kc; k's outside the sphere or the half space
  // have kmap -1 and a zero operand).
  int tc_rows;           // R
  int tc_mt;             // structure-factor M tiles of 64 rows (x U, V)
  int tc_ns;             // structure-factor N: 2 (2kc + 1) rounded up to 16
  int tc_kp;             // scatter K: 2 (2kc + 1) rounded up to 8
  int tc_rt;             // k rows per 128-column scatter tile: 20 (field + force) or 32
  int tc_nt;             // scatter tiles: ceil(R / tc_rt)
  int tc_nst;            // scatter pipeline stages (2 or 3)
  int tc_chunk, tc_nchunk;  // structure-factor particle chunks (multiple of 16)
  const int2* tc_row;    // [R] (ny, nz)
  const float4* tc_rowd; // scatter row descriptors (kspace_tc_row_desc)
  const int* tc_kmap;    // [R][2kc + 1] sorted k index, or -1
  float* tc_part;        // [nchunk][mt][ns][128] FP32 chunk partials (column-major tiles)
  float* tc_w;           // scatter operand image [nt][hi, lo][128][kp] (this evaluation's layout)
  float* tc_bimg;        // per step: X operand tiles per 16 particles [n/16][hi, lo][ns][32]
  float2* tc_tblk;       // per step: Y, Z of each 16 particles [n/16][2][kc + 1][17]
  int tc_scat_smem;      // dynamic shared memory of the scatter launch
  int tc_yz;             // the scatter stages the Y, Z phases in shared memory
  int tc_sfa, tc_sfb;    // structure-factor ring slots (generated, copied)
  // k space by rows (md_krows.cu; rw_T = 0: off): tasks of four |nx| of one row
  int rw_T, rw_R;          // tasks, rows
  int rw_nblk, rw_threads; // structure factor: task blocks, threads per block
  int rw_chunk, rw_nchunk; // particles per chunk, chunks
  int rw_np;               // particles per scatter block
  const int4* rw_task;      // [T] row, ny, nz, first |nx|
  const int* rw_kidx;       // [T][4][+, -] sorted k index, or -1
  const double2* rw_row;    // [R] (ny, nz)
  const int2* rw_rowt;      // [R] first task, tasks
  void* rw_ad;              // [T][4] T4 (A, D)
  // k space through a mesh (md_kmesh.cu; gm_M = 0: off)
  int gm_M, gm_nbrick;     // mesh points per axis, bricks of the spread
  int gm_nitem;            // work items that there is room for (>= bricks)
  int gm_ncx;              // cells per axis of the sorted view
  float gm_reach;          // distance a particle may be from the cell it is filed in, box units
  const float* gm_coef;    // [kMeshW][kMeshDeg + 1] window polynomials, lowest order first
  const float2* gm_fac;    // [R][2 kc + 1] e(n) / omega^6(n), 1 / omega^3(n) of the rows' k vectors
  const float2* gm_tw;     // [M] exp(2 pi i j / M)
  float* gm_part;          // [bricks][3][padded brick]
  float2* gm_z;            // [3][kc + 1][M][M] after the z axis
  float4 *gm_y, *gm_t;     // [kc + 1][2 kc + 1][M] rows before and after the x axis
  float4* gm_b;            // [M][M][M] field mesh
  int* gm_plan;            // work items of the spread and the interpolation
  long long tc_wait;     // SM clock cycles after which an mbarrier wait gives up
  int* err;              // device error word (kErrTcWait on a wait that gave up)
};

// ----------------------------------------------------- integrator
struct IntParams {
  int n;
  double dt, L;
  double B_unit, F_unit;     // SI per unit
  double cself, csurf;       // box units
  double anisConst, velMmConst, magDamp;
  int mobil;
  int noise;                 // MD_NOISE_*
  uint64_t seed;
  int field_kind;
  double magFluxDens, tMag, fieldAmp, fieldFreq;
  const double* xi;          // uploaded unit normals [9][n] for this step
  // master state (orig order, FP64 SoA)
  double *pos, *mm, *ea, *truePos, *posRef;
  // particle constants (orig order)
  const double* magMom_u;    // |mu_i| / mu_u
  const double* rMag_u;      // rMag / L
  // per-particle constants in T (k_int_consts), T4 each: thermal torque, field
  // and force scale (DefThermFluct), 1 / zeta_trans; velEa1, velEa2, |mu| /
  // mu_u, rMag / L
  const void *cA, *cB;
  // the scalars above as T = float sees them
  struct F32 {
    float dt, L, iL, B_unit, F_unit, cself, csurf, anisConst, velMmConst, magDamp;
  } f;
  // work arrays (orig order, T)
  void *k1m, *k1e, *m2, *e2, *th;   // th: [9][n] scaled noise (mixed adaptive solvers: unit normals)
  // stage outputs (sorted order, T)
  const void *Br, *Bk, *Fr, *Fk, *ov;
  // FP64 strong-pair terms: sv.B belongs to the evaluation that gave Br,
  // sv.F and sv.P to the full evaluation (Fr, Ppart); sv.off null when off
  StrongView sv;
  // Reported field only (R = double in demag_si): FP64 unit moments of the
  // evaluation (particle order) and the k-space self-interaction matrix
  // kself = cflux sum_k e(k) n n^T (xx, yy, zz, xy, xz, yz; box units); the
  // k-space sum holds -kself mu_i of each particle's own FP32 moment, which
  // is moved to the FP64 moment.  mexact null: no correction.
  const double* mexact;
  double kself[6];
  SortedView s;
  const double* musum;       // [3] sum of mu' of the evaluated stage
  const double* Ppart;       // [n][3] per-particle pressure sums of the full real-space pass
  double* obs_part;          // [gridDim.x][7]: msd x,y,z, mz, Pxy, Pxz, Pyz
  const double* time;        // device t (double) and step
  const long long* stepno;
  int* err;
  const double* xbuild;      // [3][n] positions at the last neighbour-list build
  StepFlags* flags;          // maxdisp is raised here
};

// One stage (or the accept step) of an adaptive Runge-Kutta attempt.
struct RKStage {
  IntParams p;              // p.Br / p.Bk: the field last evaluated; p.dt: the attempt's step
  void* km[7];              // stage slopes of m, [3][n] T, original order
  void* ke[7];              // stage slopes of n
  void* cm;                 // stage coordinates (m), [3][n] T
  void* ce;                 // stage coordinates (n)
  double a[7];              // weights of k_0..k_s: next stage (stage kernel) / solution (accept)
  double e[7];              // error weights (last stage)
  double nf;                // factor on the thermal field and torque (rescaled on rejections)
  const double2* sTB;       // mixed: scales of torque and field, unrounded, of p.th's unit normals
  int s;                    // stage index (0-based); accept: last weight index
  int last;                 // stage: no next stage, form the error; accept: take (cm, ce)
  unsigned long long* errmax;  // max over particles of the error norm (double bits)
};

struct ObsParams {
  int nblk_int;
  const double* obs_part;
  double p_scale;            // L * F_unit / (2 * volBox) (pair double count)
  double inv_n;
  double dt;
  double* time;
  long long* stepno;
  double* records;           // [cap][8]
  long long* nrec;
  long long cap;
  // packed runs: the system's error word and list overflow, copied to status
  const int* err;
  const StepFlags* flags;
  int* status;               // may be null
};

// ------------------------------------------------------ device helpers
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11): the published
// multipliers and Weyl increments; counter {i, block, step_lo, step_hi}.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

// Standard normals of particle i at step s (torque xyz, field xyz, force xyz,
// three spare): Box-Muller on uniforms (x + 0.5) 2^-32 of Philox blocks {i, b,
// step}; pair j of block j / 2 gives normals 2 j and 2 j + 1.
template <typename T>
__device__ __forceinline__ void box_muller(uint32_t a, uint32_t b, T z[2]) {
  if constexpr (std::is_same<T, float>::value) {
    const float u1 = ((float)a + 0.5f) * 2.3283064365386963e-10f;
    const float u2 = ((float)b + 0.5f) * 2.3283064365386963e-10f;
    float rr = sqrtf(-2.0f * logf(u1)), s, c;
    sincospif(2.0f * u2, &s, &c);
    z[0] = rr * c;
    z[1] = rr * s;
  } else {
    const double u1 = ((double)a + 0.5) * 2.3283064365386963e-10;
    const double u2 = ((double)b + 0.5) * 2.3283064365386963e-10;
    double rr = sqrt(-2.0 * log(u1)), s, c;
    sincospi(2.0 * u2, &s, &c);
    z[0] = rr * c;
    z[1] = rr * s;
  }
}
template <typename T>
__device__ __forceinline__ void philox_pair(uint64_t seed, uint64_t step, uint32_t i, int j, T z[2]) {
  const uint4 r = philox4x32_10(make_uint4(i, (uint32_t)j >> 1, (uint32_t)step, (uint32_t)(step >> 32)),
                                (uint32_t)seed, (uint32_t)(seed >> 32));
  (j & 1) ? box_muller<T>(r.z, r.w, z) : box_muller<T>(r.x, r.y, z);
}
template <typename T>
__device__ __forceinline__ void philox_normals9(uint64_t seed, uint64_t step, uint32_t i, T z[9]) {
#pragma unroll
  for (uint32_t b = 0; b < 3; b++) {
    const uint4 r = philox4x32_10(make_uint4(i, b, (uint32_t)step, (uint32_t)(step >> 32)), (uint32_t)seed,
                                  (uint32_t)(seed >> 32));
    T w[4];
    box_muller<T>(r.x, r.y, w);
    box_muller<T>(r.z, r.w, w + 2);
#pragma unroll
    for (int h = 0; h < 4; h++)
      if (4 * b + h < 9) z[4 * b + h] = w[h];
  }
}

// Sums of W values (a power of two) over the warp with W - 1 + log2(32 / W)
// additions per lane instead of 5 W (FP64 additions: 64 cycles each): each
// butterfly step halves the values a lane carries.  Returns the sum of value
// (lane / (32 / W)).
template <int W, typename T>
__device__ __forceinline__ T warp_sums(T (&v)[W], int lane) {
  int o = 16;
#pragma unroll
  for (int h = W / 2; h >= 1; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < h; q++) {
      const T give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
      v[q] = keep + __shfl_xor_sync(kFull, give, o);
    }
  }
  T s = v[0];
  for (; o >= 1; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  return s;
}

// FP64 <-> FP32 in integer operations (the FP64 pipe takes 64 cycles per warp
// instruction): widening is exact, narrowing truncates; zeros, subnormals,
// infinities and NaN (and what FP32 cannot hold) take the conversion
// instructions.
__device__ __forceinline__ double widen(float v) {
  const unsigned b = __float_as_uint(v);
  if (((b >> 23) & 255u) - 1u >= 254u) return (double)v;
  return __hiloint2double((int)((((b & 0x7fffffffu) >> 3) + (896u << 20)) | (b & 0x80000000u)), (int)(b << 29));
}
__device__ __forceinline__ float narrow(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  if (((hi >> 20) & 0x7ffu) - 897u >= 254u) return (float)v;
  return __uint_as_float((hi & 0x80000000u) | ((((hi & 0x7fffffffu) - (896u << 20)) << 3) | (lo >> 29)));
}

// Box coordinate wrapped to [-0.5, 0.5).
__device__ __forceinline__ double wrap_box(double x, double invL) {
  double xb = x * invL;
  return xb - floor(xb + 0.5);
}

// round(x_box 2^32) as a wrapping 32-bit integer (the fold by whole boxes drops
// out mod 2^32): adding 1.5 2^52 leaves the rounded integer in the low word, two
// FP64 instructions for |x| < 2^17 box lengths.
__device__ __forceinline__ int fixed_box(double x, double invL) {
  const double t = x * (invL * 4294967296.0);
  if ((__double2hiint(t) & 0x7fffffff) < 0x43000000)  // |t| < 2^49
    return __double2loint(t + 6755399441055744.0);
  return (int)(unsigned)(long long)llrint(wrap_box(x, invL) * 4294967296.0);
}

template <typename T>
__device__ __forceinline__ void cmul(T ar, T ai, T br, T bi, T& cr, T& ci) {
  cr = ar * br - ai * bi;
  ci = ar * bi + ai * br;
}

// exp(2 pi i n x) evaluated directly, x in 2^-32 box lengths.
__device__ __forceinline__ float2 phase_direct(int nn, unsigned sfix) {
  const int ph = (int)((unsigned)nn * sfix);  // exact reduction mod one box length
  float s, c;
  sincospif(2.0f * ((float)ph * 2.3283064365386963e-10f), &s, &c);
  return make_float2(c, s);
}

// Device error word bits.
enum : int { kErrNonFinite = 1, kErrQueue = 2, kErrTcWait = 4 };

// Sorted views.  Fixed point: x_fix = round(x_box * 2^32) as a wrapping
// 32-bit integer, so x_fix[j] - x_fix[i] (mod 2^32) is the minimum-image
// difference in units of L / 2^32 (about 4e-16 m at L = 1.7 um).  On a
// rebuild the particle positions are recorded as the list's reference.
template <typename T>
__device__ __forceinline__ void fill_one(const CellParams& p, int k) {
  using T4 = typename V4<T>::t;
  const int n = p.n;
  const SortedView& s = p.s;
  const int i = s.perm[k];
  const bool rb = !p.flags || p.flags->rebuild;
  const double px = p.pos[i], py = p.pos[n + i], pz = p.pos[2 * n + i];
  if (rb) {
    s.rank[i] = k;
    s.cell[k] = p.cellOf[i];
    if (p.xbuild) {
      p.xbuild[i] = px;
      p.xbuild[n + i] = py;
      p.xbuild[2 * n + i] = pz;
    }
  }
  const double rm = p.rMag_u[i];
  if constexpr (std::is_same<T, float>::value) {
    const int4 q = make_int4(fixed_box(px, p.invL), fixed_box(py, p.invL), fixed_box(pz, p.invL), i);
    s.xi[k] = q;
    // float copies for the cell scans (list builds, and every evaluation while
    // the list does not fit)
    const float sc = 2.3283064365386963e-10f;
    if (rb || p.flags->overflow) s.xf[k] = make_float4((float)q.x * sc, (float)q.y * sc, (float)q.z * sc, (float)rm);
  } else {
    const double x = wrap_box(px, p.invL), y = wrap_box(py, p.invL), z = wrap_box(pz, p.invL);
    s.xf[k] = make_float4((float)x, (float)y, (float)z, (float)rm);
    s.xd[k] = make_double4_32a(x, y, z, rm);
  }
  const double mu = p.magMom_u[i];
  T4 m;
  m.x = (T)(p.mm[i] * mu);
  m.y = (T)(p.mm[n + i] * mu);
  m.z = (T)(p.mm[2 * n + i] * mu);
  m.w = (T)rm;
  ((T4*)s.mu)[k] = m;
}

}  // namespace md
