// md_post.cu -- post-processing on the device: the radial distribution
// function of the current frame, as the reference's analysis script computes
// it (mFiles/radial_dist_fun.m:19-66 of MD_Sim_Wolfschwenger): every pair
// i < j at its minimum-image distance (one wrap per axis, as the script),
// distances below contact clamped to 2 r_mag0, pairs closer than the range
// counted in `bins` equal bins, each count scaled by L^3 / (2 pi dr^3 N^2)
// / (k - 1/2)^2.  The script's inner loop stops at particle N - 1, leaving
// out the pairs with the last particle; include_last chooses between that
// and all pairs.
//
// Kernels.  A range of at most a fifth of the box: the particles are put into
// cells no smaller than the range (counting sort; the order within a cell does
// not matter to integer counts) and a thread per particle walks its 27 cells.
// The bin comes from the FP32 distance of the 32-bit fixed-point coordinates,
// and from the FP64 expression on the master positions only where the FP32
// error could reach a bin's edge, the contact distance or the range (~0.1 % of
// the pairs at 500 bins), so the counts are those of the FP64 expression; FP64
// for every pair in range would cost ~40 instructions of 64 cycles each.
// Bound: the candidates' loads from L1, ~95 per particle at N = 32768 and a
// range of 0.047 L: 546 us per call over all pairs -> 71 us (27 of them this walk).
// Longer ranges, and frames whose particles gather in few cells: all pairs from the
// FP64 master positions; a block takes the particles i of tile x against the 256
// particles j of tile y >= x, staged in shared memory, tile pair after tile pair; an
// FP32 pre-test in box units (with a margin) rejects the pairs far outside the
// range, the rest get their FP64 distance; pairs inside the range go to a per-block
// shared-memory histogram (integer atomics) added to the global counts after each
// tile pair (deterministic integer sums).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "md_ctx_internal.h"

namespace md {

constexpr int kRdfThreads = 256;
constexpr int kRdfMaxBins = 8192;

// The bin of the pair distance in FP64, -1 outside the range.
struct RdfBins {
  double L, range2, rcont, inv_bw;
  int bins;
  __device__ __forceinline__ int bin(double dx, double dy, double dz) const {
    const double half = 0.5 * L;
    dx -= L * (double)(dx > half);
    dx += L * (double)(dx < -half);
    dy -= L * (double)(dy > half);
    dy += L * (double)(dy < -half);
    dz -= L * (double)(dz > half);
    dz += L * (double)(dz < -half);
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 >= range2) return -1;
    double r = sqrt(r2);
    if (r < rcont) r = rcont;
    const int b = (int)floor(r * inv_bw);
    return b < bins ? b : -1;
  }
};

// Cell of each particle and its place in it (any order).  Bit 31 of the index
// marks a particle well outside the box, for which the script's one wrap per
// axis is not the periodic distance: its pairs take the FP64 expression.
constexpr unsigned kRdfOutside = 0x80000000u;
__global__ void __launch_bounds__(kRdfThreads) k_rdf_cells(int n, const double* __restrict__ pos, double invL, int ncx,
                                                           int* __restrict__ count, int4* __restrict__ x,
                                                           int2* __restrict__ cs) {
  const int i = blockIdx.x * kRdfThreads + threadIdx.x;
  if (i >= n) return;
  const double px = pos[i], py = pos[n + i], pz = pos[2 * n + i], lim = 0.625 / invL;
  int4 q;
  q.x = fixed_box(px, invL);
  q.y = fixed_box(py, invL);
  q.z = fixed_box(pz, invL);
  q.w = fabs(px) <= lim && fabs(py) <= lim && fabs(pz) <= lim ? i : (int)((unsigned)i | kRdfOutside);
  auto cell = [&](int v) { return (int)__umulhi((unsigned)v + 0x80000000u, (unsigned)ncx); };
  const int c = (cell(q.z) * ncx + cell(q.y)) * ncx + cell(q.x);
  x[i] = q;
  cs[i] = make_int2(c, atomicAdd(&count[c], 1));
}

// Exclusive sums of the cell counts (one block of 1024 threads).  *crowded: the
// particles' cells hold more than `most` particles on average (count squared, summed).
__global__ void __launch_bounds__(1024) k_rdf_scan(int ncell, const int* __restrict__ count, int* __restrict__ start,
                                                   double most, unsigned long long* __restrict__ crowded) {
  __shared__ int wsum[32];
  __shared__ unsigned long long sq[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int per = (ncell + 1023) / 1024, b = min(t * per, ncell), e = min(ncell, b + per);
  int local = 0;
  unsigned long long s2 = 0;
#pragma unroll 8
  for (int c = b; c < e; c++) {
    const int v = count[c];
    local += v;
    s2 += (unsigned long long)v * (unsigned)v;
  }
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[w] = incl;
  s2 = warp_sum(s2);
  if (lane == 0) sq[w] = s2;
  __syncthreads();
  if (w == 0) {
    s2 = warp_sum(sq[lane]);
    if (lane == 0) *crowded = (double)s2 > most;
    const int v = wsum[lane];
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += u;
    }
    wsum[lane] = inc - v;
  }
  __syncthreads();
  int run = wsum[w] + incl - local;
#pragma unroll 8
  for (int c = b; c < e; c++) {
    start[c] = run;
    run += count[c];
  }
  if (t == 1023) start[ncell] = run;
}

__global__ void __launch_bounds__(kRdfThreads) k_rdf_place(int n, const int4* __restrict__ x,
                                                           const int2* __restrict__ cs, const int* __restrict__ start,
                                                           int4* __restrict__ sorted, int* __restrict__ cellof) {
  const int i = blockIdx.x * kRdfThreads + threadIdx.x;
  if (i >= n) return;
  const int2 c = cs[i];
  const int k = start[c.x] + c.y;
  sorted[k] = x[i];
  cellof[k] = c.x;
}

// Thread = sorted particle and one of its three cell layers (blockIdx.y; a
// thread for all 27 cells leaves ~2 warps per SM quarter at N = 32768 and
// their loads' latency exposed): each pair i < j < jmax once.  inv_f:
// bins per 2^-32 box lengths; tol: bound of the FP32 bin coordinate's error.
__global__ void __launch_bounds__(kRdfThreads) k_rdf_near(int n, const int4* __restrict__ sorted,
                                                          const int* __restrict__ cellof,
                                                          const int* __restrict__ start, int ncx,
                                                          const double* __restrict__ pos, RdfBins rb, float inv_f,
                                                          float tol, int bin_cont, int jmax,
                                                          const unsigned long long* __restrict__ crowded,
                                                          unsigned long long* __restrict__ counts) {
  if (*crowded) return;  // left to k_rdf
  extern __shared__ unsigned int hist[];  // [bins]
  for (int b = threadIdx.x; b < rb.bins; b += kRdfThreads) hist[b] = 0;
  __syncthreads();
  const float cont = (float)(rb.rcont * rb.inv_bw), top = (float)rb.bins;
  const int k = blockIdx.x * kRdfThreads + threadIdx.x;
  if (k < n) {
    const int4 me = sorted[k];
    const int c = cellof[k], mi = me.w & 0x7fffffff;
    const int cx = c % ncx, cy = (c / ncx) % ncx, cz = c / (ncx * ncx);
    auto walk = [&](int a, int e) {
      for (int j = a; j < e; j++) {
        const int4 q = sorted[j];
        const int qi = q.w & 0x7fffffff;
        if (qi <= mi || qi >= jmax) continue;
        const float dx = (float)(q.x - me.x), dy = (float)(q.y - me.y), dz = (float)(q.z - me.z);
        float f = sqrtf(dx * dx + dy * dy + dz * dz) * inv_f;  // bin coordinate
        const float t = fmaf(f, 1e-6f, tol);
        const bool exact = (q.w | me.w) < 0;
        if (f > top + t) continue;
        int b = (int)f;
        const float fr = f - (float)b;
        if (!exact && f < cont - t) {
          b = bin_cont;  // below contact: clamped
        } else if (exact || fr < t || fr > 1.0f - t || fabsf(f - cont) <= t) {
          b = rb.bin(pos[mi] - pos[qi], pos[n + mi] - pos[n + qi], pos[2 * n + mi] - pos[2 * n + qi]);
        }
        if (b >= 0 && b < rb.bins) atomicAdd(&hist[b], 1u);
      }
    };
    const int uz = cz + (int)blockIdx.y - 1, wz = uz < 0 ? ncx - 1 : (uz == ncx ? 0 : uz);
    for (int dy = -1; dy <= 1; dy++) {
      const int wy = cy + dy < 0 ? ncx - 1 : (cy + dy == ncx ? 0 : cy + dy);
      const int* row = start + (wz * ncx + wy) * ncx;
      walk(row[max(cx - 1, 0)], row[min(cx + 1, ncx - 1) + 1]);
      if (cx == 0) walk(row[ncx - 1], row[ncx]);
      if (cx == ncx - 1) walk(row[0], row[1]);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < rb.bins; b += kRdfThreads)
    if (hist[b]) atomicAdd(&counts[b], (unsigned long long)hist[b]);
}

// All pairs, tile pair after tile pair: particles i of tile x against the particles j
// of tile y >= x.
__global__ void __launch_bounds__(kRdfThreads) k_rdf(int n, const double* __restrict__ pos, RdfBins rb,
                                                     float range2_test, int jmax, int ntile,
                                                     unsigned long long* __restrict__ counts) {
  extern __shared__ unsigned char smem_raw[];
  double* tile = (double*)smem_raw;                          // [3][kRdfThreads]
  float* tilef = (float*)(tile + 3 * kRdfThreads);           // [3][kRdfThreads] box units
  unsigned int* hist = (unsigned int*)(tilef + 3 * kRdfThreads);  // [bins]
  const float invL = (float)(1.0 / rb.L);
  const unsigned pairs = (unsigned)ntile * (unsigned)(ntile + 1) / 2;
  for (unsigned q = blockIdx.x; q < pairs; q += gridDim.x) {
    // q = y (y + 1) / 2 + x, x <= y
    unsigned y = min((unsigned)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f), (unsigned)ntile - 1u);
    while (y * (y + 1) / 2 > q) y--;
    while ((y + 1) * (y + 2) / 2 <= q) y++;
    const int i0 = (int)(q - y * (y + 1) / 2) * kRdfThreads, j0 = (int)y * kRdfThreads;
    __syncthreads();
    for (int b = threadIdx.x; b < rb.bins; b += kRdfThreads) hist[b] = 0;
    const int i = i0 + threadIdx.x, jl = j0 + threadIdx.x;
    if (jl < jmax) {
      for (int a = 0; a < 3; a++) {
        const double v = pos[a * n + jl];
        tile[a * kRdfThreads + threadIdx.x] = v;
        tilef[a * kRdfThreads + threadIdx.x] = (float)v * invL;
      }
    }
    __syncthreads();
    if (i < n) {
      const double xi = pos[i], yi = pos[n + i], zi = pos[2 * n + i];
      const float xf = (float)xi * invL, yf = (float)yi * invL, zf = (float)zi * invL;
      const int tn = min(kRdfThreads, jmax - j0);
      for (int t = 0; t < tn; t++) {
        if (j0 + t <= i) continue;
        float fx = xf - tilef[t], fy = yf - tilef[kRdfThreads + t], fz = zf - tilef[2 * kRdfThreads + t];
        // minimum image in box units (|f| may exceed 1/2 just past the faces)
        fx -= rintf(fx);
        fy -= rintf(fy);
        fz -= rintf(fz);
        if (fx * fx + fy * fy + fz * fz > range2_test) continue;
        const int b = rb.bin(xi - tile[t], yi - tile[kRdfThreads + t], zi - tile[2 * kRdfThreads + t]);
        if (b >= 0) atomicAdd(&hist[b], 1u);
      }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < rb.bins; b += kRdfThreads)
      if (hist[b]) atomicAdd(&counts[b], (unsigned long long)hist[b]);
  }
}

}  // namespace md

extern "C" int md_rdf(md_ctx* c, int64_t bins, double range, double r_mag0, int include_last, double* g,
                      uint64_t* counts_out) {
  int st = check_ready(c, true);
  if (st) return st;
  if (bins < 1 || bins > md::kRdfMaxBins || !(range > 0) || !(r_mag0 > 0) || !g)
    return set_err(c, MD_ERR_INVALID, "md_rdf: bins must be 1..%d, range and r_mag0 positive", md::kRdfMaxBins);
  const int n = (int)c->n;
  if ((n + md::kRdfThreads - 1) / md::kRdfThreads > 65535)
    return set_err(c, MD_ERR_UNSUPPORTED, "md_rdf: at most %d particles", 65535 * md::kRdfThreads);
  const double L = c->L, bw = range / (double)bins;
  const int jmax = include_last ? n : n - 1;
  const md::RdfBins rb{L, range * range, 2.0 * r_mag0, 1.0 / bw, (int)bins};
  // cells of at least the range (with a margin above the coordinates' rounding
  // and above the distance that the range test can still accept), ~2
  // particles each at most; five per edge: below, 27 cells hold a fifth of the
  // pairs or more and the tiles over all pairs are faster
  const double rbox = range / L * (1.0 + 1e-4) + 1e-6;
  const int ncx = (int)std::min({1.0 / rbox, std::cbrt(0.5 * n), 128.0});
  const bool cells = ncx >= 5;
  const int ncell = cells ? ncx * ncx * ncx : 0;
  // workspace, kept by the context: sorted x | x | cell, place | counts | crowded | cell
  // counts | starts | cell
  const size_t cb = sizeof(unsigned long long) * (size_t)(md::kRdfMaxBins + 1);
  const size_t need = cb + 8 * (size_t)(ncell + 1) + (cells ? 44 * (size_t)n : 0);
  if (need > c->rdf_cap) {
    dfree(c, c->rdf_ws);
    c->rdf_ws = nullptr;
    c->rdf_cap = 0;
    if ((st = dalloc(c, &c->rdf_ws, need))) return st;
    c->rdf_cap = need;
  }
  const size_t nc = cells ? (size_t)n : 0;
  int4 *sorted = (int4*)c->rdf_ws, *x = sorted + nc;
  int2* cs = (int2*)(x + nc);
  unsigned long long *d_counts = (unsigned long long*)(cs + nc), *crowded = d_counts + bins;
  int *count = (int*)(crowded + 1), *start = count + ncell, *cellof = start + ncell + 1;
  const size_t hb = sizeof(unsigned long long) * (size_t)(bins + 1);
  if (cudaMemsetAsync(d_counts, 0, hb + sizeof(int) * (size_t)ncell, c->stream) != cudaSuccess)
    return set_err(c, MD_ERR_CUDA, "md_rdf: memset failed");
  const int nt = (n + md::kRdfThreads - 1) / md::kRdfThreads;
  auto all_pairs = [&] {
    const size_t smem = (sizeof(double) + sizeof(float)) * 3 * md::kRdfThreads + sizeof(unsigned int) * (size_t)bins;
    md::allow_smem<md::k_rdf>();
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
    // 64 blocks per SM, dealt out as they finish (8, all resident: 689 us against 581
    // at N = 32768)
    const int g = (int)std::min<int64_t>((int64_t)nt * (nt + 1) / 2, 64 * nsm);
    md::k_rdf<<<g, md::kRdfThreads, smem, c->stream>>>(n, c->pos, rb, (float)(rbox * rbox), jmax, nt, d_counts);
  };
  std::vector<unsigned long long> h((size_t)bins + 1);
  auto read = [&] {
    return cudaGetLastError() == cudaSuccess &&
           cudaMemcpyAsync(h.data(), d_counts, hb, cudaMemcpyDeviceToHost, c->stream) == cudaSuccess &&
           cudaStreamSynchronize(c->stream) == cudaSuccess;
  };
  if (cells) {
    // A walk takes ~2.3 us for each particle in a cell (its threads walk one after
    // another); all pairs take 150 us at N = 2048, 201 at 8192, 530 at 32768, 1660 at
    // 65536, 6240 at 131072: equal at ~45, 60, 180, 500, 1750 particles in a
    // particle's cell.  Below ~1500 particles the walk is never much longer.
    const double most = n < 1500 ? 1e300 : (double)n * (45.0 + 1.0e-7 * (double)n * (double)n);
    md::k_rdf_cells<<<nt, md::kRdfThreads, 0, c->stream>>>(n, c->pos, 1.0 / L, ncx, count, x, cs);
    md::k_rdf_scan<<<1, 1024, 0, c->stream>>>(ncell, count, start, most, crowded);
    md::k_rdf_place<<<nt, md::kRdfThreads, 0, c->stream>>>(n, x, cs, start, sorted, cellof);
    const double per_fix = L / 4294967296.0 / bw;  // bins per 2^-32 box lengths
    md::k_rdf_near<<<dim3(nt, 3), md::kRdfThreads, sizeof(unsigned int) * (size_t)bins, c->stream>>>(
        n, sorted, cellof, start, ncx, c->pos, rb, (float)per_fix, (float)(4.0 * per_fix + 1e-9),
        (int)std::floor(rb.rcont * rb.inv_bw), jmax, crowded, d_counts);
    if (!read()) return set_err(c, MD_ERR_CUDA, "md_rdf: kernel or copy failed");
  }
  if (!cells || h[(size_t)bins]) {
    all_pairs();
    if (!read()) return set_err(c, MD_ERR_CUDA, "md_rdf: kernel or copy failed");
  }
  // normalisation of the script: L^3 / (2 pi dr^3 N^2) / (k - 1/2)^2
  const double norm = L * L * L / (2.0 * c->cfg.my_pi * bw * bw * bw * (double)n * (double)n);
  for (int64_t k = 0; k < bins; k++) {
    const double kk = (double)k + 0.5;
    g[k] = (double)h[(size_t)k] * norm / (kk * kk);
    if (counts_out) counts_out[k] = h[(size_t)k];
  }
  return MD_OK;
}
