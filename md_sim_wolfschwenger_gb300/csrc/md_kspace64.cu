// md_kspace64.cu -- kernel (c) on the FP64 path: the reciprocal-space Ewald
// sums of md_kspace.cu (CompDipInteractEwaldF / CompDipFieldEwaldF,
// src/interaction.cpp:429-514, 588-672, with the phases of EvalSinCos,
// src/interaction.cpp:521-548), all in FP64.
//
// Bound: the FP64 pipe.  GB300 issues a warp's FP64 instruction in 64 cycles
// of an SM quarter, so loads and integer work are free beside it, one warp per
// SM quarter keeps it busy, and what counts is the number of FP64
// instructions and their even spread over all SMs.
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
// Splits: structure factor = blocks of <= 128 tasks x particle chunks, as many
// chunks as fill the SMs (the partial sums are added by k_red64); scatter =
// 8, 16 or 32 particles x 32, 16 or 8 subsets of the rows per block, the
// fewer particles the smaller the system.
#include <algorithm>

#include "md_common.cuh"
#include "md_kernels.h"

namespace md {

constexpr int kTile64 = 16;      // particles staged per structure-factor tile
constexpr int kScat64 = 256;     // threads of a scatter block
constexpr int kPhase64 = 256;

// Phase tables [3][kc + 1][n]: block = 32 particles x one axis, its warps
// take the directly evaluated phases (n < 4 and the multiples of 4) in turn,
// then the products (the same values as one thread per particle and axis
// gives, 20 us at N = 1000, in 1/8 of the chain).
__global__ void __launch_bounds__(kPhase64) k_phase64(KParams p) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  double2* d = (double2*)smem_raw;  // [direct phases][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kPhase64 / 32;
  const int ax = blockIdx.y, k = blockIdx.x * 32 + lane, kk = min(k, p.n - 1);
  const double4_32a q = p.s.xd[kk];
  const double xb = ax == 0 ? q.x : (ax == 1 ? q.y : q.z);
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

// Structure-factor partials of blockIdx.x's tasks over chunk blockIdx.y.
__global__ void __launch_bounds__(128) k_sf64(KParams p) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int K1 = p.kc + 1, KX = (p.kc & ~3) + 4;        // |nx| padded to whole tasks
  double2* X = (double2*)smem_raw;                      // [kTile64][KX]
  double2* YZ = X + kTile64 * KX;                       // [kTile64][2][K1]
  double4_32a* mus = (double4_32a*)(YZ + kTile64 * 2 * K1);
  double2* op = (double2*)(mus + kTile64);              // [rows of the block][kTile64][2]
  const int tid = threadIdx.x, nt = blockDim.x;
  const int t0 = blockIdx.x * nt, t = min(t0 + tid, p.k64_T - 1);
  const int p0 = blockIdx.y * p.k64_chunk, p1 = min(p.n, p0 + p.k64_chunk);
  const int4 tk = p.k64_task[t];  // row, ny, nz, first |nx|
  const int r0 = p.k64_task[t0].x, nr = p.k64_task[min(t0 + nt, p.k64_T) - 1].x - r0 + 1;
  const double2* gtab = (const double2*)p.tab;
  const double2* xt = X + tk.w;
  const double2* ot = op + (size_t)(tk.x - r0) * kTile64 * 2;
  double acc[4][8];
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int q = 0; q < 8; q++) acc[u][q] = 0.0;
  for (int b0 = p0; b0 < p1; b0 += kTile64) {
    const int tn = min(kTile64, p1 - b0);
    __syncthreads();
    for (int i = tid; i < KX * kTile64; i += nt) {
      const int e = i / kTile64, pp = i - e * kTile64;
      X[pp * KX + e] = (e < K1 && pp < tn) ? gtab[(size_t)e * p.n + b0 + pp] : make_double2(0.0, 0.0);
    }
    for (int i = tid; i < 2 * K1 * kTile64; i += nt) {
      const int e = i / kTile64, pp = i - e * kTile64;
      if (pp < tn) YZ[pp * 2 * K1 + e] = gtab[(size_t)(K1 + e) * p.n + b0 + pp];
    }
    if (tid < tn) mus[tid] = ((const double4_32a*)p.s.mu)[b0 + tid];
    __syncthreads();
    for (int i = tid; i < nr * kTile64; i += nt) {
      const int r = i / kTile64, pp = i - r * kTile64;
      if (pp >= tn) continue;
      const double2 row = p.k64_row[r0 + r];  // ny, nz
      const int ny = (int)row.x, nz = (int)row.y;
      double2 Y = YZ[pp * 2 * K1 + (ny < 0 ? -ny : ny)];
      const double2 Z = YZ[pp * 2 * K1 + K1 + nz];
      if (ny < 0) Y.y = -Y.y;
      double pr, pi;
      cmul<double>(Y.x, Y.y, Z.x, Z.y, pr, pi);
      const double4_32a mu = mus[pp];
      const double U = row.x * mu.y + row.y * mu.z;
      op[i * 2] = make_double2(U * pr, U * pi);
      op[i * 2 + 1] = make_double2(mu.x * pr, mu.x * pi);
    }
    __syncthreads();
    for (int pp = 0; pp < tn; pp++) {
      const double2 a = ot[pp * 2], b = ot[pp * 2 + 1];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const double2 x = xt[pp * KX + u];
        acc[u][0] += a.x * x.x;
        acc[u][1] += a.y * x.y;
        acc[u][2] += a.x * x.y;
        acc[u][3] += a.y * x.x;
        acc[u][4] += b.x * x.x;
        acc[u][5] += b.y * x.y;
        acc[u][6] += b.x * x.y;
        acc[u][7] += b.y * x.x;
      }
    }
  }
  if (t0 + tid < p.k64_T) {
    double* out = (double*)p.Spart + (size_t)blockIdx.y * 16 * p.k64_T + t;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const double nx = (double)(tk.w + u);
      const double* s = acc[u];
      out[(size_t)(4 * u) * p.k64_T] = (s[0] - s[1]) + nx * (s[4] - s[5]);      // S(+nx)
      out[(size_t)(4 * u + 1) * p.k64_T] = (s[3] + s[2]) + nx * (s[7] + s[6]);
      out[(size_t)(4 * u + 2) * p.k64_T] = (s[0] + s[1]) - nx * (s[4] + s[5]);  // S(-nx)
      out[(size_t)(4 * u + 3) * p.k64_T] = (s[3] - s[2]) - nx * (s[7] - s[6]);
    }
  }
  if (blockIdx.x == 0) {
    // sum of moments of this chunk (surface term), warp 0
    if (tid < 32) {
      double m[4] = {0.0, 0.0, 0.0, 0.0};
      for (int q = p0 + tid; q < p1; q += 32) {
        const double4_32a mu = ((const double4_32a*)p.s.mu)[q];
        m[0] += mu.x;
        m[1] += mu.y;
        m[2] += mu.z;
      }
#pragma unroll
      for (int q = 0; q < 3; q++) {
        m[q] = warp_sum(m[q]);
        if (tid == q) p.musum_part[3 * blockIdx.y + q] = m[q];
      }
    }
  }
}

// Chunk partials of 32 tasks and one |nx| offset (blockIdx.y) -> S, and the
// scatter's A, D.
__global__ void __launch_bounds__(256) k_red64(KParams p) {
  __shared__ double red[8][4][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, u = blockIdx.y;
  const int t = blockIdx.x * 32 + tx;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (t < p.k64_T)
    for (int c = ty; c < p.k64_nchunk; c += 8) {
      const double* in = (const double*)p.Spart + ((size_t)c * 16 + 4 * u) * p.k64_T + t;
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] += in[(size_t)q * p.k64_T];
    }
#pragma unroll
  for (int q = 0; q < 4; q++) red[ty][q][tx] = v[q];
  __syncthreads();
  if (ty < 4) {  // value ty of every task
    double s = red[0][ty][tx];
#pragma unroll
    for (int g = 1; g < 8; g++) s += red[g][ty][tx];
    red[0][ty][tx] = s;
  }
  __syncthreads();
  if (ty == 0 && t < p.k64_T) {
    const int kp = p.k64_kidx[8 * t + 2 * u], km = p.k64_kidx[8 * t + 2 * u + 1];
    double2 tp = make_double2(0.0, 0.0), tm = tp;
    if (kp >= 0) {
      const double2 s = make_double2(red[0][0][tx], red[0][1][tx]);
      const double e = p.ek[kp];
      p.S[kp] = s;
      tp = make_double2(e * s.x, -e * s.y);
    }
    if (km >= 0) {
      const double2 s = make_double2(red[0][2][tx], red[0][3][tx]);
      const double e = p.ek[km];
      p.S[km] = s;
      tm = make_double2(e * s.x, -e * s.y);
    }
    double2* ad = p.k64_ad + 2 * (4 * (size_t)t + u);
    ad[0] = make_double2(tp.x + tm.x, tp.y + tm.y);
    ad[1] = make_double2(tp.x - tm.x, tp.y - tm.y);
  }
  if (blockIdx.x == 0 && u == 0 && ty == 7) {
    double m[3] = {0.0, 0.0, 0.0};
    for (int c = tx; c < p.k64_nchunk; c += 32)
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
template <int NP, bool FULL>
__global__ void __launch_bounds__(kScat64) k_scat64(KParams p) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  constexpr int RS = kScat64 / NP, NV = FULL ? 6 : 3;
  const int K1 = p.kc + 1, KX = (p.kc & ~3) + 4;
  double2* X = (double2*)smem_raw;   // [KX][NP]
  double2* NX = X + KX * NP;         // [KX][NP] nx X
  double2* YZ = NX + KX * NP;        // [2 K1][NP]
  __shared__ double red[RS][NV][NP];
  const int tid = threadIdx.x, lp = tid % NP, rs = tid / NP;
  const int base = blockIdx.x * NP, k = base + lp;
  const double2* gtab = (const double2*)p.tab;
  for (int i = tid; i < KX * NP; i += kScat64) {
    const int e = i / NP, q = min(base + i - e * NP, p.n - 1);
    const double2 v = e < K1 ? gtab[(size_t)e * p.n + q] : make_double2(0.0, 0.0);
    X[i] = v;
    NX[i] = make_double2((double)e * v.x, (double)e * v.y);
  }
  for (int i = tid; i < 2 * K1 * NP; i += kScat64) {
    const int e = i / NP, q = min(base + i - e * NP, p.n - 1);
    YZ[i] = gtab[(size_t)(K1 + e) * p.n + q];
  }
  const double4_32a mu = ((const double4_32a*)p.s.mu)[min(k, p.n - 1)];
  __syncthreads();
  double b[3] = {0.0, 0.0, 0.0}, f[3] = {0.0, 0.0, 0.0};
  for (int r = rs; r < p.k64_R; r += RS) {
    const double2 row = p.k64_row[r];
    const int2 tr = p.k64_rowt[r];  // first task, tasks
    const double2* ad = p.k64_ad + 8 * (size_t)tr.x;
    double q0r = 0, q0i = 0, q1r = 0, q1i = 0, q2r = 0, q2i = 0;
    for (int nx = 0; nx < 4 * tr.y; nx += 4) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const double2 A = ad[2 * (nx + u)], D = ad[2 * (nx + u) + 1];
        const double2 x = X[(nx + u) * NP + lp], y = NX[(nx + u) * NP + lp];
        if constexpr (FULL) {
          const double zr = fma(-x.y, D.y, x.x * A.x), zi = fma(x.y, D.x, x.x * A.y);
          const double n2 = (double)((nx + u) * (nx + u));
          q0r += zr;
          q0i += zi;
          q2r = fma(n2, zr, q2r);
          q2i = fma(n2, zi, q2i);
        } else {
          q0r = fma(-x.y, D.y, fma(x.x, A.x, q0r));
          q0i = fma(x.y, D.x, fma(x.x, A.y, q0i));
        }
        q1r = fma(-y.y, A.y, fma(y.x, D.x, q1r));
        q1i = fma(y.y, A.x, fma(y.x, D.y, q1i));
      }
    }
    const int ny = (int)row.x, nz = (int)row.y;
    double2 Y = YZ[(ny < 0 ? -ny : ny) * NP + lp];
    const double2 Z = YZ[(K1 + nz) * NP + lp];
    if (ny < 0) Y.y = -Y.y;
    double pr, pi;
    cmul<double>(Y.x, Y.y, Z.x, Z.y, pr, pi);
    const double g0 = pr * q0r - pi * q0i;
    b[0] = fma(-pi, q1i, fma(pr, q1r, b[0]));
    b[1] = fma(row.x, g0, b[1]);
    b[2] = fma(row.y, g0, b[2]);
    if constexpr (FULL) {
      const double h0 = pr * q0i + pi * q0r, h1 = pr * q1i + pi * q1r, h2 = pr * q2i + pi * q2r;
      const double U = row.x * mu.y + row.y * mu.z;
      f[0] = fma(mu.x, h2, fma(U, h1, f[0]));
      const double h = mu.x * h1 + U * h0;
      f[1] = fma(row.x, h, f[1]);
      f[2] = fma(row.y, h, f[2]);
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
    for (int i = tid; i < h * NV * NP; i += kScat64) (&red[0][0][0])[i] += (&red[0][0][0])[h * NV * NP + i];
  }
  __syncthreads();
  for (int i = tid; i < NV * NP; i += kScat64) {
    const int a = i / NP, q = base + i - a * NP;
    if (q >= p.n) continue;
    const double s = (&red[0][0][0])[i];
    if (a < 3)
      ((double*)p.B)[a * p.n + q] = -p.cflux * s;
    else
      ((double*)p.F)[(a - 3) * p.n + q] = p.cforce * s;
  }
}

// ------------------------------------------------------------ entry points

static size_t sf64_smem(int kc, int threads) {
  const int K1 = kc + 1, KX = (kc & ~3) + 4;
  return 16 * (size_t)kTile64 * (KX + 2 * K1) + 32 * (size_t)kTile64 + 32 * (size_t)threads * kTile64;
}
static size_t scat64_smem(int kc, int np) { return 16 * (size_t)np * (2 * ((kc & ~3) + 4) + 2 * (kc + 1)); }

// Tasks are dealt to blocks of equal size (<= 128); the chunk count fills the
// SMs once with the blocks that fit (at least 8 particles per chunk: below,
// staging a tile costs more than the sums).
K64Shape kspace64_shape(int kc, int n, int tasks, int nsm) {
  K64Shape s{};
  s.nblk = (tasks + 127) / 128;
  s.threads = ((tasks + s.nblk - 1) / s.nblk + 31) / 32 * 32;
  const size_t sm = sf64_smem(kc, s.threads);
  cudaFuncSetAttribute(k_sf64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_sf64, s.threads, sm) != cudaSuccess || nb < 1) nb = 1;
  const int nch = std::max(1, std::min((n + 7) / 8, nb * nsm / s.nblk));
  s.chunk = ((n + nch - 1) / nch + 3) / 4 * 4;
  s.nchunk = (n + s.chunk - 1) / s.chunk;
  return s;
}

int launch_phase64(cudaStream_t st, const KParams& p) {
  const int nd = p.kc < 4 ? p.kc + 1 : 4 + (p.kc >> 2);
  k_phase64<<<dim3((p.n + 31) / 32, 3), kPhase64, 32 * sizeof(double2) * (size_t)nd, st>>>(p);
  return 1;
}

template <int NP>
static void scat64(cudaStream_t st, const KParams& p, bool full) {
  const size_t sm = scat64_smem(p.kc, NP);
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kern<<<(p.n + NP - 1) / NP, kScat64, sm, st>>>(p);
  };
  full ? go(k_scat64<NP, true>) : go(k_scat64<NP, false>);
}

int launch_kspace64(cudaStream_t st, const KParams& p, bool full, cudaEvent_t* ev) {
  const size_t sm = sf64_smem(p.kc, p.k64_threads);
  cudaFuncSetAttribute(k_sf64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_sf64<<<dim3(p.k64_nblk, p.k64_nchunk), p.k64_threads, sm, st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[0], st, cudaEventRecordExternal);
  k_red64<<<dim3((p.k64_T + 31) / 32, 4), 256, 0, st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[1], st, cudaEventRecordExternal);
  // few particles per block while that leaves SMs without a block
  if (p.n <= 2432)
    scat64<8>(st, p, full);
  else if (p.n <= 4864 || p.kc > 64)
    scat64<16>(st, p, full);
  else
    scat64<32>(st, p, full);
  return 3;
}

}  // namespace md
