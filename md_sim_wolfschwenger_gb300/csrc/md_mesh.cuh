// md_mesh.cuh -- bricks of the mesh that large mixed systems take their k space
// through (md_kmesh.cu), and the plan of the work on them, made with the cell order
// (md_cells.cu).
#pragma once
#include "md_common.cuh"

namespace md {

constexpr int kMW = kMeshW;                    // window points per axis (odd: nearest mesh point +- 4)
constexpr int kMH = kMW / 2;
constexpr int kMC = kMeshDeg + 1;              // coefficients per interval
constexpr int kBX = 16, kBY = 8, kBZ = 8;      // brick: mesh points whose particles one block spreads
constexpr int kPX = kBX + kMW - 1, kPY = kBY + kMW - 1, kPZ = kBZ + kMW - 1;  // with the window's reach
static_assert(kPZ == 16 && kPY == 16 && kPX == 24, "padded brick");
constexpr int kPad = kPX * kPY * kPZ;          // points of a padded brick
constexpr int kBrThreads = kPY * kPZ;          // brick kernels: a thread per (y, z) of the padded brick
constexpr int kBrWarps = kBrThreads / 32;      // two rows y of 16 z each
static_assert(kPZ == 16 && kBrThreads == 256, "lanes of a warp: two rows of 16");

// The plan: [extra items][first extra item of each brick][extra items of each brick]
// [item: brick, part | parts << 16 (0: none)].  Item b < bricks is part 0 of brick b.
struct MeshPlan {
  int *total, *first, *extra;
  int2* item;
  __host__ __device__ MeshPlan(int* p, int nbrick)
      : total(p), first(p + 1), extra(p + 1 + nbrick), item((int2*)(p + 2 + 2 * nbrick)) {}
};

// Cells along an axis that hold the particles whose window starts at b0 .. b0 + w - 1
// (kMH points below the nearest mesh point): first one and their number.
__device__ __forceinline__ void brick_cells(int M, int ncx, float h, int b0, int w, int& lo, int& cnt) {
  const float im = 1.0f / (float)M, f = (float)ncx;
  lo = (int)floorf((((float)(b0 + kMH) - 0.5f) * im + 0.5f - h) * f);
  cnt = (int)floorf((((float)(b0 + w + kMH) - 0.5f) * im + 0.5f + h) * f) - lo + 1;
  if (cnt >= ncx) {
    lo = 0;
    cnt = ncx;
  }
  lo %= ncx;
  if (lo < 0) lo += ncx;
}

// The plan.  When particles gather, a brick's block would take most of them one after
// another while the other blocks are done, so bricks with many candidates are split
// into items of about equal candidates when the cells are filled anew.  An item holds
// up to eight times the mean, or 1024: at uniform density every brick is one item, and
// the extra items are at most an eighth of the bricks (their idle blocks cost 3 us per
// step at N = 32768 with a quarter, 1 with an eighth).  N = 32768 all in 0.15^3 of the
// box, kc = 20: step 4233 -> 1389 us (tensor cores 1413); uniform 574.7 -> 576.4.  Made in
// the launches of the cell order: a launch of its own before the spread let the
// real-space blocks take the SMs first, 7 us per step at N = 32768.

// Candidates of brick b, by one warp.
__device__ __forceinline__ void mesh_plan_count(const MeshGrid& g, const int* cell_start, int b, int lane) {
  const int M = g.M, ncx = g.ncx, nbx = (M + kBX - 1) / kBX, nby = M / kBY;
  const int x0 = b % nbx * kBX, y0 = b / nbx % nby * kBY, z0 = b / (nbx * nby) * kBZ;
  int cx, nx, cy, ny, cz, nz, c = 0;
  brick_cells(M, ncx, g.reach, x0, min(kBX, M - x0), cx, nx);
  brick_cells(M, ncx, g.reach, y0, kBY, cy, ny);
  brick_cells(M, ncx, g.reach, z0, kBZ, cz, nz);
  const int hi = min(cx + nx, ncx);
  for (int r = lane; r < ny * nz; r += 32) {
    int iy = cy + r % ny, iz = cz + r / ny;
    if (iy >= ncx) iy -= ncx;
    if (iz >= ncx) iz -= ncx;
    const int* row = cell_start + ((size_t)iz * ncx + iy) * ncx;
    c += row[hi] - row[cx];
    if (cx + nx > ncx) c += row[cx + nx - ncx] - row[0];
  }
  c = __reduce_add_sync(kFull, c);
  if (lane == 0) MeshPlan(g.plan, g.nbrick).extra[b] = c;
}

// The items, by one block, after every brick's candidates.
__device__ __forceinline__ void mesh_plan_items(const MeshGrid& g) {
  __shared__ long long wsum[33];
  __shared__ int scan[33];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5, nb = g.nbrick;
  const MeshPlan plan(g.plan, nb);
  long long mine = 0;
  for (int b = tid; b < nb; b += nt) mine += __ldcg(plan.extra + b);
  mine = warp_sum(mine);
  if (lane == 0) wsum[wid] = mine;
  __syncthreads();
  long long total = 0;
  for (int w = 0; w < nw; w++) total += wsum[w];
  const long long size = max(1024ll, (8 * total + nb - 1) / nb);
  int base = 0;
  for (int b0 = 0; b0 < nb; b0 += nt) {
    const int b = b0 + tid;
    int e = 0;
    if (b < nb) e = max(0, (int)((__ldcg(plan.extra + b) + size - 1) / size) - 1);
    int incl = e;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    __syncthreads();
    if (lane == 31) scan[wid] = incl;
    __syncthreads();
    int at = base + incl - e;
    for (int w = 0; w < nw; w++) {
      if (w < wid) at += scan[w];
      base += scan[w];
    }
    if (b < nb) {
      plan.first[b] = at;
      plan.extra[b] = e;
      plan.item[b] = make_int2(b, (e + 1) << 16);
      for (int q = 0; q < e; q++) plan.item[nb + at + q] = make_int2(b, (q + 1) | (e + 1) << 16);
    }
  }
  for (int q = base + tid; q < g.nitem - nb; q += nt) plan.item[nb + q] = make_int2(0, 0);
  if (tid == 0) *plan.total = base;
}

}  // namespace md
