// md_krows.cu -- kernel (c) by k rows on the CUDA cores: the reciprocal-space
// Ewald sums of md_kspace.cu (CompDipInteractEwaldF / CompDipFieldEwaldF,
// src/interaction.cpp:429-514, 588-672, with the phases of EvalSinCos,
// src/interaction.cpp:521-548) for the FP64 path (T = double) and for small
// systems on the mixed path (T = float; krows_wanted).
//
// k vectors are taken by rows r = (ny, nz) and pairs +-nx.  With X = c + i s
// the phase of |nx|, P = Y(ny) Z(nz), U = ny mu_y + nz mu_z and V = mu_x, the
// eight sums over particles of {U, V} x {Re P, Im P} x {c, s} give
// S(+nx) and S(-nx): 4 FMA per k and particle, where advancing a phase from k
// to k takes 7.  The way back is the same: with T = conj(e S), A = T(+nx) +
// T(-nx) and D = T(+nx) - T(-nx),
//   Q_0 = sum c A + i s D,  Q_1 = sum nx (c D + i s A),  Q_2 = sum nx^2 (c A + i s D)
// over nx >= 0 (4 FMA per k for the field, 6 with the force), and per row
//   B += (Re P Q_1, ny Re P Q_0, nz Re P Q_0),
//   F += (mu_x Im P Q_2 + U Im P Q_1, (ny, nz) (mu_x Im P Q_1 + U Im P Q_0)).
// A task is four consecutive |nx| of one row; a row has as many as its length
// needs.
//
// Bound, FP64: the FP64 pipe.  GB300 issues a warp's FP64 instruction in 64
// cycles of an SM quarter, so loads and integer work are free beside it, one
// warp per SM quarter keeps it busy, and what counts is the number of FP64
// instructions and their even spread over all SMs.
// Bound, small mixed systems: latency.  The work of N = 512, kc = 7 is < 1 us
// of FP32; the tensor-core kernels (set-up of tensor memory and barriers,
// generated operand stages, one block per 128 particles in the scatter) took
// 10 + 8 + 10 us per evaluation.
//
// Splits: structure factor = blocks of <= 128 tasks x particle chunks, as many
// chunks as fill the SMs (FP32 sums over <= 512 particles; the partial sums
// are added by k_red_rows, on the mixed path as exact FP32 pairs); scatter =
// 8, 16 or 32 particles x 32, 16 or 8 subsets of the rows per block, the
// fewer particles the smaller the system.
#include <algorithm>

#include "md_common.cuh"
#include "md_kernels.h"

namespace md {

constexpr int kRowTile = 16;      // particles staged per structure-factor tile
constexpr int kRowScat = 256;     // threads of a scatter block
constexpr int kRowPhase = 256;

// Phase tables [3][kc + 1][n].  FP64: block = 32 particles x one axis, its
// warps take the directly evaluated phases (n < 4 and the multiples of 4) in
// turn, then the products (the same values as one thread per particle and
// axis gives, 20 us at N = 1000, in 1/8 of the chain).
__global__ void __launch_bounds__(kRowPhase) k_phase64(CellParams cp, KParams p) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  double2* d = (double2*)smem_raw;  // [direct phases][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kRowPhase / 32;
  const int ax = blockIdx.y, k = blockIdx.x * 32 + lane, kk = min(k, p.n - 1);
  if (ax == 3) {  // the sorted views
    if (w == 0 && k < p.n) fill_one<double>(cp, k);
    return;
  }
  const double xb = wrap_box(cp.pos[(size_t)ax * p.n + cp.s.perm[kk]], cp.invL);
  const int nd = p.kc < 4 ? p.kc + 1 : 4 + (p.kc >> 2);  // 0, 1, 2, 3, 4, 8, 12, ..
  for (int t = w; t < nd; t += nw) {
    const int nn = t < 4 ? t : 4 * (t - 3);
    double2 v = make_double2(1.0, 0.0);
    if (nn) sincos(p.two_pi * (double)nn * xb, &v.y, &v.x);
    d[t * 32 + lane] = v;
  }
  __syncthreads();
  if (k >= p.n) return;
  double2* out = (double2*)p.tab + (size_t)ax * (p.kc + 1) * p.n + k;
  for (int nn = w; nn <= p.kc; nn += nw) {
    double2 v;
    if (nn < 4) {
      v = d[nn * 32 + lane];
    } else {
      const double2 a = d[(3 + (nn >> 2)) * 32 + lane];
      v = a;
      if (nn & 3) {
        const double2 b = d[(nn & 3) * 32 + lane];
        cmul<double>(a.x, a.y, b.x, b.y, v.x, v.y);
      }
    }
    out[(size_t)nn * p.n] = v;
  }
}

// FP32: every phase directly, one thread each (the reduction mod one box
// length is exact in the fixed-point coordinates).
__global__ void __launch_bounds__(kRowPhase) k_phase32(CellParams cp, KParams p) {
  const int k = blockIdx.x * kRowPhase + threadIdx.x, e = blockIdx.y, K1 = p.kc + 1;
  if (k >= p.n) return;
  const int ax = e / K1, nn = e - ax * K1;
  if (ax == 3) {  // the sorted views
    fill_one<float>(cp, k);
    return;
  }
  const int ph = (int)((unsigned)nn * (unsigned)fixed_box(cp.pos[(size_t)ax * p.n + cp.s.perm[k]], cp.invL));
  float s, c;
  sincospif(2.0f * ((float)ph * 2.3283064365386963e-10f), &s, &c);
  ((float2*)p.tab)[(size_t)e * p.n + k] = make_float2(c, s);
}

// Structure-factor partials of blockIdx.x's tasks over chunk blockIdx.y; one
// more column of blocks adds the chunks' moments.
template <typename T>
__global__ void __launch_bounds__(128) k_sf_rows(KParams p) {
  using T2 = typename V2<T>::t;
  using T4 = typename V4<T>::t;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int K1 = p.kc + 1, KX = (p.kc & ~3) + 4;  // |nx| padded to whole tasks
  T4* mus = (T4*)smem_raw;                        // [kRowTile]
  T4* op = mus + kRowTile;                        // [kRowTile][rows of the block]: U P, V P
  T2* X = (T2*)(op + kRowTile * blockDim.x);      // [kRowTile][KX]
  T2* YZ = X + kRowTile * KX;                     // [kRowTile][2][K1]
  const int tid = threadIdx.x, nt = blockDim.x;
  const int p0 = blockIdx.y * p.rw_chunk, p1 = min(p.n, p0 + p.rw_chunk);
  if (blockIdx.x == p.rw_nblk) {  // the extra column: sum of moments of the chunk (surface term)
    if (tid >= 32) return;
    double m[3] = {0.0, 0.0, 0.0};
    for (int q = p0 + tid; q < p1; q += 32) {
      const T4 mu = ((const T4*)p.s.mu)[q];
      m[0] += (double)mu.x;
      m[1] += (double)mu.y;
      m[2] += (double)mu.z;
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
      m[q] = warp_sum(m[q]);
      if (tid == q) p.musum_part[3 * blockIdx.y + q] = m[q];
    }
    return;
  }
  const int t0 = blockIdx.x * nt, t = min(t0 + tid, p.rw_T - 1);
  const int4 tk = p.rw_task[t];  // row, ny, nz, first |nx|
  const int r0 = p.rw_task[t0].x, nr = p.rw_task[min(t0 + nt, p.rw_T) - 1].x - r0 + 1;
  const T2* gtab = (const T2*)p.tab;
  const T2* xt = X + tk.w;
  const T4* ot = op + (tk.x - r0);
  T acc[4][8];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int q = 0; q < 8; q++) acc[u][q] = 0;
  for (int b0 = p0; b0 < p1; b0 += kRowTile) {
    const int tn = min(kRowTile, p1 - b0);
    __syncthreads();
    for (int i = tid; i < KX * kRowTile; i += nt) {
      const int e = i / kRowTile, pp = i - e * kRowTile;
      T2 v = {0, 0};
      if (e < K1 && pp < tn) v = gtab[(size_t)e * p.n + b0 + pp];
      X[pp * KX + e] = v;
    }
    for (int i = tid; i < 2 * K1 * kRowTile; i += nt) {
      const int e = i / kRowTile, pp = i - e * kRowTile;
      if (pp < tn) YZ[pp * 2 * K1 + e] = gtab[(size_t)(K1 + e) * p.n + b0 + pp];
    }
    if (tid < tn) mus[tid] = ((const T4*)p.s.mu)[b0 + tid];
    __syncthreads();
    for (int i = tid; i < nr * tn; i += nt) {
      const int pp = i / nr, r = i - pp * nr;
      const double2 row = p.rw_row[r0 + r];  // ny, nz
      const int ny = (int)row.x, nz = (int)row.y;
      T2 Y = YZ[pp * 2 * K1 + (ny < 0 ? -ny : ny)];
      const T2 Z = YZ[pp * 2 * K1 + K1 + nz];
      if (ny < 0) Y.y = -Y.y;
      T pr, pi;
      cmul<T>(Y.x, Y.y, Z.x, Z.y, pr, pi);
      const T4 mu = mus[pp];
      const T U = (T)row.x * mu.y + (T)row.y * mu.z;
      T4 o;
      o.x = U * pr;
      o.y = U * pi;
      o.z = mu.x * pr;
      o.w = mu.x * pi;
      op[pp * nt + r] = o;
    }
    __syncthreads();
    for (int pp = 0; pp < tn; pp++) {
      const T4 o = ot[pp * nt];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const T2 x = xt[pp * KX + u];
        acc[u][0] += o.x * x.x;
        acc[u][1] += o.y * x.y;
        acc[u][2] += o.x * x.y;
        acc[u][3] += o.y * x.x;
        acc[u][4] += o.z * x.x;
        acc[u][5] += o.w * x.y;
        acc[u][6] += o.z * x.y;
        acc[u][7] += o.w * x.x;
      }
    }
  }
  if (t0 + tid < p.rw_T) {
    T* out = (T*)p.Spart + (size_t)blockIdx.y * 16 * p.rw_T + t;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const T nx = (T)(tk.w + u);
      const T* s = acc[u];
      out[(size_t)(4 * u) * p.rw_T] = (s[0] - s[1]) + nx * (s[4] - s[5]);      // S(+nx)
      out[(size_t)(4 * u + 1) * p.rw_T] = (s[3] + s[2]) + nx * (s[7] + s[6]);
      out[(size_t)(4 * u + 2) * p.rw_T] = (s[0] + s[1]) - nx * (s[4] + s[5]);  // S(-nx)
      out[(size_t)(4 * u + 3) * p.rw_T] = (s[3] - s[2]) - nx * (s[7] - s[6]);
    }
  }
}

// s + v with the rounding error added to c (Knuth): an exact running sum.
__device__ __forceinline__ void add_exact(float& s, float& c, float v) {
  const float t = s + v, b = t - s;
  c += (s - (t - b)) + (v - b);
  s = t;
}

// Chunk partials of 32 tasks and one |nx| offset (blockIdx.y) -> S, and the
// scatter's A, D.  Warp = every 8th chunk; then warp q < 4 adds value q of
// every task over the warps.  FP32 partials are added as exact pairs (s, c).
// S and e S are FP64.
template <typename T>
__global__ void __launch_bounds__(256) k_red_rows(KParams p) {
  constexpr bool F32 = std::is_same<T, float>::value;
  __shared__ T red[8][4][32], redc[F32 ? 8 : 1][4][32];
  __shared__ double tot[4][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, u = blockIdx.y;
  const int t = blockIdx.x * 32 + tx;
  // the k indices and weights (a chain of two loads) first
  int kp = -1, km = -1;
  double ep = 0.0, em = 0.0;
  if (ty == 0 && t < p.rw_T) {
    kp = p.rw_kidx[8 * t + 2 * u];
    km = p.rw_kidx[8 * t + 2 * u + 1];
    if (kp >= 0) ep = p.ek[kp];
    if (km >= 0) em = p.ek[km];
  }
  T v[4] = {0, 0, 0, 0}, e[4] = {0, 0, 0, 0};
  if (t < p.rw_T) {
#pragma unroll 4
    for (int c = ty; c < p.rw_nchunk; c += 8) {
      const T* in = (const T*)p.Spart + ((size_t)c * 16 + 4 * u) * p.rw_T + t;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if constexpr (F32)
          add_exact(v[q], e[q], in[(size_t)q * p.rw_T]);
        else
          v[q] += in[(size_t)q * p.rw_T];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    red[ty][q][tx] = v[q];
    if constexpr (F32) redc[ty][q][tx] = e[q];
  }
  __syncthreads();
  if (ty < 4) {
    T s = red[0][ty][tx];
    if constexpr (F32) {
      T c = redc[0][ty][tx];
#pragma unroll
      for (int g = 1; g < 8; g++) {
        add_exact(s, c, red[g][ty][tx]);
        c += redc[g][ty][tx];
      }
      tot[ty][tx] = (double)s + (double)c;
    } else {
#pragma unroll
      for (int g = 1; g < 8; g++) s += red[g][ty][tx];
      tot[ty][tx] = s;
    }
  }
  __syncthreads();
  if (ty == 0 && t < p.rw_T) {
    double2 tp = make_double2(0.0, 0.0), tm = tp;
    if (kp >= 0) {
      const double2 s = make_double2(tot[0][tx], tot[1][tx]);
      p.S[kp] = s;
      tp = make_double2(ep * s.x, -ep * s.y);
    }
    if (km >= 0) {
      const double2 s = make_double2(tot[2][tx], tot[3][tx]);
      p.S[km] = s;
      tm = make_double2(em * s.x, -em * s.y);
    }
    typename V4<T>::t o;
    o.x = (T)(tp.x + tm.x);
    o.y = (T)(tp.y + tm.y);
    o.z = (T)(tp.x - tm.x);
    o.w = (T)(tp.y - tm.y);
    ((typename V4<T>::t*)p.rw_ad)[4 * (size_t)t + u] = o;
  }
  if (blockIdx.x == 0 && u == 0 && ty == 7) {
    double m[3] = {0.0, 0.0, 0.0};
    for (int c = tx; c < p.rw_nchunk; c += 32)
#pragma unroll
      for (int q = 0; q < 3; q++) m[q] += p.musum_part[3 * c + q];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      m[q] = warp_sum(m[q]);
      if (tx == q) p.musum[q] = m[q];
    }
  }
}

// Field (and force) of NP particles per block; thread = (particle, every
// 256 / NP-th row).
template <typename T, int NP, bool FULL>
__global__ void __launch_bounds__(kRowScat) k_scat_rows(KParams p) {
  using T2 = typename V2<T>::t;
  using T4 = typename V4<T>::t;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  constexpr int RS = kRowScat / NP, NV = FULL ? 6 : 3;
  const int K1 = p.kc + 1, KX = (p.kc & ~3) + 4;
  T2* X = (T2*)smem_raw;   // [KX][NP]
  T2* NX = X + KX * NP;         // [KX][NP] nx X
  T2* YZ = NX + KX * NP;        // [2 K1][NP]
  __shared__ T red[RS][NV][NP];
  const int tid = threadIdx.x, lp = tid % NP, rs = tid / NP;
  const int base = blockIdx.x * NP, k = base + lp;
  const T2* gtab = (const T2*)p.tab;
  for (int i = tid; i < KX * NP; i += kRowScat) {
    const int e = i / NP, q = min(base + i - e * NP, p.n - 1);
    const T2 v = e < K1 ? gtab[(size_t)e * p.n + q] : T2{0, 0};
    X[i] = v;
    NX[i] = T2{(T)e * v.x, (T)e * v.y};
  }
  for (int i = tid; i < 2 * K1 * NP; i += kRowScat) {
    const int e = i / NP, q = min(base + i - e * NP, p.n - 1);
    YZ[i] = gtab[(size_t)(K1 + e) * p.n + q];
  }
  const T4 mu = ((const T4*)p.s.mu)[min(k, p.n - 1)];
  __syncthreads();
  T b[3] = {0, 0, 0}, f[3] = {0, 0, 0};
  for (int r = rs; r < p.rw_R; r += RS) {
    const double2 rw = p.rw_row[r];
    const T rowx = (T)rw.x, rowy = (T)rw.y;
    const int2 tr = p.rw_rowt[r];  // first task, tasks
    const T4* ad = (const T4*)p.rw_ad + 4 * (size_t)tr.x;
    T q0r = 0, q0i = 0, q1r = 0, q1i = 0, q2r = 0, q2i = 0;
    for (int nx = 0; nx < 4 * tr.y; nx += 4) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const T4 w = ad[nx + u];  // A, D
        const T2 x = X[(nx + u) * NP + lp], y = NX[(nx + u) * NP + lp];
        if constexpr (FULL) {
          const T zr = fma(-x.y, w.w, x.x * w.x), zi = fma(x.y, w.z, x.x * w.y);
          const T n2 = (T)((nx + u) * (nx + u));
          q0r += zr;
          q0i += zi;
          q2r = fma(n2, zr, q2r);
          q2i = fma(n2, zi, q2i);
        } else {
          q0r = fma(-x.y, w.w, fma(x.x, w.x, q0r));
          q0i = fma(x.y, w.z, fma(x.x, w.y, q0i));
        }
        q1r = fma(-y.y, w.y, fma(y.x, w.z, q1r));
        q1i = fma(y.y, w.x, fma(y.x, w.w, q1i));
      }
    }
    const int ny = (int)rw.x, nz = (int)rw.y;
    T2 Y = YZ[(ny < 0 ? -ny : ny) * NP + lp];
    const T2 Z = YZ[(K1 + nz) * NP + lp];
    if (ny < 0) Y.y = -Y.y;
    T pr, pi;
    cmul<T>(Y.x, Y.y, Z.x, Z.y, pr, pi);
    const T g0 = pr * q0r - pi * q0i;
    b[0] = fma(-pi, q1i, fma(pr, q1r, b[0]));
    b[1] = fma(rowx, g0, b[1]);
    b[2] = fma(rowy, g0, b[2]);
    if constexpr (FULL) {
      const T h0 = pr * q0i + pi * q0r, h1 = pr * q1i + pi * q1r, h2 = pr * q2i + pi * q2r;
      const T U = rowx * mu.y + rowy * mu.z;
      f[0] = fma(mu.x, h2, fma(U, h1, f[0]));
      const T h = mu.x * h1 + U * h0;
      f[1] = fma(rowx, h, f[1]);
      f[2] = fma(rowy, h, f[2]);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    red[rs][a][lp] = b[a];
    if constexpr (FULL) red[rs][3 + a][lp] = f[a];
  }
  // row subsets added pairwise (fixed order)
  for (int h = RS / 2; h >= 1; h >>= 1) {
    __syncthreads();
    for (int i = tid; i < h * NV * NP; i += kRowScat) (&red[0][0][0])[i] += (&red[0][0][0])[h * NV * NP + i];
  }
  __syncthreads();
  for (int i = tid; i < NV * NP; i += kRowScat) {
    const int a = i / NP, q = base + i - a * NP;
    if (q >= p.n) continue;
    const T s = (&red[0][0][0])[i];
    if (a < 3)
      ((T*)p.B)[a * p.n + q] = -(T)p.cflux * s;
    else
      ((T*)p.F)[(a - 3) * p.n + q] = (T)p.cforce * s;
  }
}

// ------------------------------------------------------------ entry points

static size_t sf_rows_smem(int kc, int threads, bool fp64) {
  const int K1 = kc + 1, KX = (kc & ~3) + 4;
  return (fp64 ? 8 : 4) * (size_t)kRowTile * (4 + 4 * (size_t)threads + 2 * (KX + 2 * K1));
}
static size_t scat_rows_smem(int kc, int np, bool fp64) {
  return (fp64 ? 16 : 8) * (size_t)np * (2 * ((kc & ~3) + 4) + 2 * (kc + 1));
}
static const void* sf_rows_fn(bool fp64) {
  return fp64 ? (const void*)k_sf_rows<double> : (const void*)k_sf_rows<float>;
}

// Tasks are dealt to blocks of equal size (<= 128); the chunk count fills the
// SMs once with the blocks that fit (at least 8 particles per chunk: below,
// staging a tile costs more than the sums; at most 512 summed in FP32).
RowShape krows_shape(int kc, int n, int tasks, int nsm, bool fp64) {
  RowShape s{};
  s.nblk = (tasks + 127) / 128;
  s.threads = ((tasks + s.nblk - 1) / s.nblk + 31) / 32 * 32;
  const size_t sm = sf_rows_smem(kc, s.threads, fp64);
  fp64 ? allow_smem<k_sf_rows<double>>() : allow_smem<k_sf_rows<float>>();
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sf_rows_fn(fp64), s.threads, sm) != cudaSuccess || nb < 1)
    nb = 1;
  int nch = std::max(1, std::min((n + 7) / 8, nb * nsm / s.nblk));
  if (!fp64) nch = std::max(nch, (n + 511) / 512);
  s.chunk = ((n + nch - 1) / nch + 3) / 4 * 4;
  s.nchunk = (n + s.chunk - 1) / s.chunk;
  // few particles per scatter block while that leaves SMs without a block (32 only
  // where their phases fit)
  s.np = n <= 16 * nsm ? 8 : (n <= 32 * nsm || kc > 64 ? 16 : 32);
  return s;
}

int launch_fill_phase_rows(cudaStream_t st, const CellParams& c, const KParams& p, bool fp64) {
  if (fp64) {
    const int nd = p.kc < 4 ? p.kc + 1 : 4 + (p.kc >> 2);
    k_phase64<<<dim3((p.n + 31) / 32, 4), kRowPhase, 32 * sizeof(double2) * (size_t)nd, st>>>(c, p);
  } else {
    k_phase32<<<dim3((p.n + kRowPhase - 1) / kRowPhase, 3 * (p.kc + 1) + 1), kRowPhase, 0, st>>>(c, p);
  }
  return 1;
}

template <typename T, int NP>
static void scat_rows(cudaStream_t st, const KParams& p, bool full) {
  const size_t sm = scat_rows_smem(p.kc, NP, std::is_same<T, double>::value);
  const int g = (p.n + NP - 1) / NP;
  if (full) {
    allow_smem<k_scat_rows<T, NP, true>>();
    k_scat_rows<T, NP, true><<<g, kRowScat, sm, st>>>(p);
  } else {
    allow_smem<k_scat_rows<T, NP, false>>();
    k_scat_rows<T, NP, false><<<g, kRowScat, sm, st>>>(p);
  }
}

template <typename T>
static int krows_t(cudaStream_t st, const KParams& p, bool full, cudaEvent_t* ev) {
  constexpr bool fp64 = std::is_same<T, double>::value;
  const size_t sm = sf_rows_smem(p.kc, p.rw_threads, fp64);
  allow_smem<k_sf_rows<T>>();
  k_sf_rows<T><<<dim3(p.rw_nblk + 1, p.rw_nchunk), p.rw_threads, sm, st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[0], st, cudaEventRecordExternal);
  k_red_rows<T><<<dim3((p.rw_T + 31) / 32, 4), 256, 0, st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[1], st, cudaEventRecordExternal);
  if (p.rw_np == 8)
    scat_rows<T, 8>(st, p, full);
  else if (p.rw_np == 16)
    scat_rows<T, 16>(st, p, full);
  else
    scat_rows<T, 32>(st, p, full);
  return 3;
}

int launch_krows(cudaStream_t st, const KParams& p, bool full, bool fp64, cudaEvent_t* ev) {
  return fp64 ? krows_t<double>(st, p, full, ev) : krows_t<float>(st, p, full, ev);
}

}  // namespace md
