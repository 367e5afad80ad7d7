// md_kmesh.cu -- kernel (c) of large systems on the mixed path: the reciprocal
// Ewald sums of CompDipInteractEwaldF / CompDipFieldEwaldF
// (src/interaction.cpp:429-514, 588-672) as non-uniform Fourier transforms
// through a mesh of M^3 points, M = 8 ceil(kc / 2) >= 4 kc.  The k vectors,
// e(n) and the formulas are those of md_ktc.cu; work is proportional to the
// particles plus the mesh instead of particles x k vectors.
//
// Window.  omega(z) = exp(beta (sqrt(1 - (2 z / w)^2) - 1)), w = 9 mesh units,
// beta = 2.3 w (the "exponential of semicircle" of Barnett, Magland and af
// Klinteberg, SIAM J. Sci. Comput. 41, 2019), as one polynomial of degree 12 per
// unit interval, which is the window from then on: its Fourier transform
// (mesh_tables) divides the sums.  With g = M x:
//   rho_a(m) = sum_j mu_ja omega3(m - g_j)                        (k_mesh_spread)
//   S(n) = sum_a n_a sum_m rho_a(m) exp(2 pi i n.m / M) / omega^3(n)    (k_mesh_z, _y, _x)
//   b_a(m) = sum_n n_a Re(conj(e S)(n) exp(2 pi i n.m / M)) / omega^3(n)  (k_mesh_x, _yz)
//   B_ia = -cflux sum_m b_a(m) omega3(m - g_i)                     (k_mesh_interp)
//   F_ia = cforce M / (2 pi) sum_m b_a(m) (mu_i . grad omega3)(m - g_i)
// Only the window's values enter S and B, and one derivative F.  (One scalar
// mesh, with derivatives of the window for the moments, the field and the force,
// is a third of the work and measured 1.1e-6 / 4.5e-6 for B / F.)
//
// Precision: k-space part against FP64, rms relative, N = 32768, kc = 15: B 1.5e-7,
// F 2.8e-7 (tensor cores 1.2e-6, 1.3e-6).  The window's own error is 4e-9 in B and
// 2.4e-7 in F, the rest FP32 rounding of sums of ~100 terms.  All sums have a
// fixed order: results are deterministic.
//
// Measured at N = 32768 (M = 64) / 131072 (M = 80), us: spread 29 / 79, the four
// transforms 30 / 50, interpolation 36 / 104 with the force, 29 / 80 without;
// the tensor cores' 135 / 850 and 120 / 700 for the same.
#include <vector>

#include "md_common.cuh"
#include "md_kernels.h"
#include "md_mesh.cuh"

namespace md {

static int mesh_nbx(int M) { return (M + kBX - 1) / kBX; }
int mesh_bricks(int M) { return mesh_nbx(M) * (M / kBY) * (M / kBZ); }
int mesh_items(int M) { return mesh_bricks(M) + mesh_bricks(M) / 8; }
size_t mesh_part_floats(int M) { return (size_t)mesh_items(M) * 3 * kPad; }
size_t mesh_plan_ints(int M) { return 2 + 2 * (size_t)mesh_bricks(M) + 2 * (size_t)mesh_items(M); }

// Brick of the block's item, -1 without one.  A brick's own block does not wait for
// the plan to know where it works.
__device__ __forceinline__ int mesh_brick(const KParams& p) {
  if ((int)blockIdx.x < p.gm_nbrick) return blockIdx.x;
  const int2 item = MeshPlan(p.gm_plan, p.gm_nbrick).item[blockIdx.x];
  return item.y ? item.x : -1;
}

// Nearest mesh point of a fixed-point coordinate (2^32 per box) and s = -2 times
// the distance to it, in [-1, 1]: the argument of the window's polynomials.
__device__ __forceinline__ int mesh_point(int x, int M, float& s) {
  const unsigned long long t = (unsigned long long)(unsigned)x * (unsigned)M + 0x80000000ull;
  const int ip = (int)(t >> 32);
  s = (float)(int)((unsigned)t ^ 0x80000000u) * -4.656612873077393e-10f;  // -2^-31
  return ip;  // 0 .. M (M is point 0)
}

// ---------------------------------------------------------------- bricks
//
// The spread and the interpolation work on bricks of 16 x 8 x 8 mesh points, a
// block each, for the particles whose window starts there; with the window's
// reach a brick has 24 x 16 x 16 points.
template <int NT>
struct BrickScan {
  int pre[NT + 1];    // candidates before row t
  int a0[NT], l0[NT], a1[NT];
  int wsum[NT / 32];
  int place[NT];      // [class][warp]: particles, then the first one's place
  int start[33];      // first particle of each class, and their number
  int first, step;    // of the candidates, for the block's item
};

// Finds the particles of the brick at (x0, y0, z0): the cells that reach into it,
// grown by the distance a particle may have moved since they were filled, are
// searched NT candidates at a time, the part of the block's item every parts-th
// time.  put(k, j, start, s) stores a particle found (sorted index, window start x | y << 8 | z << 16, arguments of the window's
// polynomials); k runs over the classes 4 (x / 2) + y / 2 of the start, and in cell
// order within a class.  chunk(hits) is then called by the whole block, between
// barriers.
template <int NT, typename P, typename C>
__device__ __forceinline__ void brick_particles(const KParams& p, BrickScan<NT>& b, int x0, int y0, int z0, P&& put,
                                                C&& chunk) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int M = p.gm_M, wx = min(kBX, M - x0), ncx = p.gm_ncx;
  int cx, nx, cy, ny, cz, nz;
  brick_cells(M, ncx, p.gm_reach, x0, wx, cx, nx);
  brick_cells(M, ncx, p.gm_reach, y0, kBY, cy, ny);
  brick_cells(M, ncx, p.gm_reach, z0, kBZ, cz, nz);
  if (tid == NT - 1) {  // in a warp that has no row of cells to load below
    const int part = MeshPlan(p.gm_plan, p.gm_nbrick).item[blockIdx.x].y;
    b.first = (part & 0xffff) * NT;
    b.step = (part >> 16) * NT;
  }
  for (int r0 = 0; r0 < ny * nz; r0 += NT) {
    __syncthreads();
    {  // one row of cells per thread, split where it wraps
      const int r = r0 + tid;
      int a0 = 0, l0 = 0, a1 = 0, l1 = 0;
      if (r < ny * nz) {
        int iy = cy + r % ny, iz = cz + r / ny;
        if (iy >= ncx) iy -= ncx;
        if (iz >= ncx) iz -= ncx;
        const int* row = p.s.cell_start + ((size_t)iz * ncx + iy) * ncx;
        const int hi = min(cx + nx, ncx);
        a0 = row[cx];
        l0 = row[hi] - a0;
        if (cx + nx > ncx) {
          a1 = row[0];
          l1 = row[cx + nx - ncx] - a1;
        }
      }
      int incl = l0 + l1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += u;
      }
      if (lane == 31) b.wsum[wid] = incl;
      b.a0[tid] = a0;
      b.l0[tid] = l0;
      b.a1[tid] = a1;
      __syncthreads();
      for (int q = 0; q < wid; q++) incl += b.wsum[q];
      b.pre[tid + 1] = incl;
      if (tid == 0) b.pre[0] = 0;
    }
    __syncthreads();
    const int total = b.pre[NT], nrow = min(NT, ny * nz - r0);
    for (int t0 = b.first; t0 < total; t0 += b.step) {
      const int t = t0 + tid;
      bool in = false;
      int at = 0, j = 0;
      float s[3] = {0.f, 0.f, 0.f};
      if (t < total) {
        int a = 0, e = nrow;  // pre[a] <= t < pre[e]
        while (e - a > 1) {
          const int m = (a + e) >> 1;
          if (b.pre[m] <= t) a = m;
          else e = m;
        }
        const int u = t - b.pre[a];
        j = u < b.l0[a] ? b.a0[a] + u : b.a1[a] + u - b.l0[a];
        const int4 q = p.s.xi[j];
        auto local = [&](int v, int b0, float& sv) {
          int i = mesh_point(v, M, sv) - kMH - b0;
          if (i < 0) i += M;
          return i >= M ? i - M : i;
        };
        const int ix = local(q.x, x0, s[0]), iy = local(q.y, y0, s[1]), iz = local(q.z, z0, s[2]);
        in = ix < wx && iy < kBY && iz < kBZ;
        at = ix | iy << 8 | iz << 16;
      }
      // stable counting sort by the class
      b.place[tid] = 0;
      __syncthreads();
      const int cls = in ? (at >> 1 & 7) * 4 + (at >> 9 & 3) : 32;
      const unsigned same = __match_any_sync(kFull, cls);
      if (in && __ffs(same) - 1 == lane) b.place[cls * (NT / 32) + wid] = __popc(same);
      __syncthreads();
      const int c = b.place[tid];
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += u;
      }
      if (lane == 31) b.wsum[wid] = incl;
      __syncthreads();
      for (int q = 0; q < wid; q++) incl += b.wsum[q];
      b.place[tid] = incl - c;
      if (tid % (NT / 32) == 0) b.start[tid / (NT / 32)] = incl - c;
      if (tid == NT - 1) b.start[32] = incl;
      __syncthreads();
      const int k = in ? b.place[cls * (NT / 32) + wid] + __popc(same & lanemask_lt()) : 0, hits = b.start[32];
      if (in) put(k, j, at, s);
      __syncthreads();
      chunk(hits);
    }
  }
}

// ---------------------------------------------------------------- spread
//
// A thread keeps the 24 points of its (y, z) in registers, as pairs along x, and
// takes the particles one after another, in classes by the place of their window:
// it covers five aligned pairs along x, whose register indices are constants within
// a class, and the rows y of five of the eight warps, each of which takes the
// classes that reach its rows.  The padded bricks go to global memory, where
// k_mesh_z adds the (up to eight) that overlap in a mesh point in a fixed order.
//
// Bound: latency of 16 warps per SM (128 registers a thread), and the last wave: 256
// bricks on 152 SMs at M = 64; 29 us at N = 32768 (37 sorted by x only, with a test
// per particle and warp; 52 adding to the brick in shared memory, a lane per
// (x, y) column, bound by the 729 x 3 read-modify-writes per particle).  16 x 8 x 8
// rather than 8 x 8 x 8: the padded bricks are 6 times the mesh instead of 8 (19 MB
// at M = 64).
constexpr int kNX2 = kPX / 2;                  // a thread's mesh points: float2 pairs along x
constexpr int kSub = 128;                      // particles whose window values are in shared memory at a time
// Window values of a particle in shared memory: x in five pairs aligned to even
// x, y and z with zeros on both sides, so that a thread outside the window reads 0.
constexpr int kWX = 0, kWY = 12, kWZ = 36, kWS = 60, kWPad = 7;
struct SpreadSmem {
  float w[kSub * kWS];
  float4 mu[kBrThreads];
  float s[3][kBrThreads];
  int at[kBrThreads];
  float coef[kMW * kMC];
  double red[3][kBrWarps];
  BrickScan<kBrThreads> scan;
};

static_assert(kBX == 16 && kBX / 2 - 1 + 5 == kNX2, "eight classes of five pairs");

__global__ void __launch_bounds__(kBrThreads, 2) k_mesh_spread(KParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  SpreadSmem& sm = *(SpreadSmem*)smem;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int M = p.gm_M, nbx = (M + kBX - 1) / kBX, nby = M / kBY;
  const int brick = mesh_brick(p), bx = brick % nbx, by = brick / nbx % nby, bz = brick / (nbx * nby);
  if (brick < 0) {
    if (tid < 3) p.musum_part[3 * blockIdx.x + tid] = 0.0;
    return;
  }
  for (int e = tid; e < kSub * kWS; e += kBrThreads) sm.w[e] = 0.f;
  for (int e = tid; e < kMW * kMC; e += kBrThreads) sm.coef[e] = p.gm_coef[e];
  const int y = tid >> 4, z = tid & 15;
  float2 acc[3][kNX2] = {};
  double m0 = 0.0, m1 = 0.0, m2 = 0.0;
  brick_particles(
      p, sm.scan, bx * kBX, by * kBY, bz * kBZ,
      [&](int k, int j, int at, const float (&s)[3]) {
        const float4 mu = ((const float4*)p.s.mu)[j];
        m0 += (double)mu.x;
        m1 += (double)mu.y;
        m2 += (double)mu.z;
        sm.mu[k] = mu;
        sm.s[0][k] = s[0];
        sm.s[1][k] = s[1];
        sm.s[2][k] = s[2];
        sm.at[k] = at;
      },
      [&](int hits) {
        for (int h0 = 0; h0 < hits; h0 += kSub) {
          const int cnt = min(kSub, hits - h0);
          if (h0 > 0) __syncthreads();
          for (int e = tid; e < cnt * 3 * kMW; e += kBrThreads) {
            const int h = e / (3 * kMW), v = e - h * 3 * kMW, ax = v / kMW, i = v - ax * kMW;
            const float sv = sm.s[ax][h0 + h], *c = sm.coef + i * kMC;
            float f = c[kMC - 1];
#pragma unroll
            for (int q = kMC - 2; q >= 0; q--) f = fmaf(f, sv, c[q]);
            const int odd = sm.at[h0 + h] & 1;
            float* w = sm.w + h * kWS;
            w[ax == 0 ? kWX + odd + i : (ax == 1 ? kWY : kWZ) + kWPad + i] = f;
            if (v == 0) w[kWX + (odd ? 0 : kMW)] = 0.f;  // the pair's other half at the window's open end
          }
          __syncthreads();
          // the classes whose rows y reach this warp's
          const int f0 = max(wid - 4, 0), f1 = min(wid, 3) + 1;
#pragma unroll
          for (int I = 0; I < 8; I++) {
            const int e = min(sm.scan.start[4 * I + f1] - h0, cnt);
#pragma unroll 2
            for (int h = max(sm.scan.start[4 * I + f0] - h0, 0); h < e; h++) {
              const int at = sm.at[h0 + h];
              const float* w = sm.w + h * kWS;
              const float4 mu = sm.mu[h0 + h];
              const float v = w[kWY + kWPad + y - (at >> 8 & 255)] * w[kWZ + kWPad + z - (at >> 16)];
              const float vx = v * mu.x, vy = v * mu.y, vz = v * mu.z;
              const float4 a = *(const float4*)(w + kWX), b = *(const float4*)(w + kWX + 4);
              const float2 x[5] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y),
                                   make_float2(b.z, b.w), *(const float2*)(w + kWX + 8)};
#pragma unroll
              for (int q = 0; q < 5; q++) {
                acc[0][I + q] = __ffma2_rn(x[q], make_float2(vx, vx), acc[0][I + q]);
                acc[1][I + q] = __ffma2_rn(x[q], make_float2(vy, vy), acc[1][I + q]);
                acc[2][I + q] = __ffma2_rn(x[q], make_float2(vz, vz), acc[2][I + q]);
              }
            }
          }
        }
      });
  float* out = p.gm_part + (size_t)blockIdx.x * 3 * kPad + tid;
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int a = 0; a < kNX2; a++) {
      out[(c * kPX + 2 * a) * kBrThreads] = acc[c][a].x;
      out[(c * kPX + 2 * a + 1) * kBrThreads] = acc[c][a].y;
    }
  m0 = warp_sum(m0);
  m1 = warp_sum(m1);
  m2 = warp_sum(m2);
  if (lane == 0) {
    sm.red[0][wid] = m0;
    sm.red[1][wid] = m1;
    sm.red[2][wid] = m2;
  }
  __syncthreads();
  if (tid < 3) {
    double t = 0.0;
    for (int q = 0; q < kBrWarps; q++) t += sm.red[tid][q];
    p.musum_part[3 * blockIdx.x + tid] = t;
  }
}

// -------------------------------------------------------- forward transform

// Bricks that hold mesh point m of an axis: (brick, local index) of its own brick
// and, within the window's reach of the brick's start, of the brick before.
struct MeshOver {
  int b[2], l[2], n;
};
__device__ __forceinline__ MeshOver mesh_over(int m, int M, int width) {
  MeshOver o;
  const int nb = (M + width - 1) / width, b = m / width, l = m - b * width;
  o.b[0] = b;
  o.l[0] = l;
  o.n = 1;
  if (l < kMW - 1) {
    const int pb = b > 0 ? b - 1 : nb - 1;
    o.b[1] = pb;
    o.l[1] = min(width, M - pb * width) + l;
    o.n = 2;
  }
  return o;
}

// The transforms along an axis are sums over <= M terms with the phases from a
// table (angles are multiples of 2 pi / M); terms z and M - z, or results +n and
// -n, share their products.

// z axis: block (x, eight y): the mesh lines summed over the bricks, then
// Z_a(nz; x, y) = sum_z rho_a exp(2 pi i nz z / M), nz = 0 .. kc.
//
// Bound: the partial meshes' bytes from L2 (six times the mesh).
constexpr int kMZLines = 8;
__global__ void __launch_bounds__(256) k_mesh_z(KParams p) {
  extern __shared__ __align__(16) float smz[];
  const int M = p.gm_M, H = M / 2, kc1 = p.kc + 1, x = blockIdx.x, y0 = blockIdx.y * kMZLines;
  const int LS = M + 1;                      // line stride: eight lines in eight banks
  float2* tw = (float2*)smz;                 // [M]
  float* line = smz + 2 * M;                 // [3][kMZLines][LS]
  for (int e = threadIdx.x; e < M; e += blockDim.x) tw[e] = p.gm_tw[e];
  const int nbx = (M + kBX - 1) / kBX, nby = M / kBY;
  const MeshOver ox = mesh_over(x, M, kBX);
  static_assert(kMZLines == kBY && kBY == kMW - 1, "a block's lines are one brick row and its neighbour's overhang");
  const int b0 = blockIdx.y, b1 = b0 > 0 ? b0 - 1 : nby - 1;
  const int wid = threadIdx.x >> 5;  // a warp takes one line of each component
  const size_t bs = (size_t)3 * kPad * nbx;
  const MeshPlan plan(p.gm_plan, p.gm_nbrick);
  const bool split = *plan.total > 0;
  for (int z = threadIdx.x & 31; z < M; z += 32) {
    const int bz0 = z >> 3, bz1 = bz0 > 0 ? bz0 - 1 : nby - 1, lz = z & 7;
    float v[3][2] = {};
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int i = 0; i < 2; i++)
        if (i < ox.n) {
          const float* a = p.gm_part + ((size_t)ox.b[i] * 3 + c) * kPad + (ox.l[i] * kPY + wid) * kPZ + lz;
          const float u0 = a[(bz0 * nby + b0) * bs], u1 = a[(bz1 * nby + b0) * bs + 8];
          const float u2 = a[(bz0 * nby + b1) * bs + 8 * kPZ], u3 = a[(bz1 * nby + b1) * bs + 8 * kPZ + 8];
          v[c][i] = (u0 + u1) + (u2 + u3);
        }
#pragma unroll
    for (int c = 0; c < 3; c++) line[(c * kMZLines + wid) * LS + z] = v[c][0] + v[c][1];
  }
  if (split) {  // the extra items of split bricks
    for (int z = threadIdx.x & 31; z < M; z += 32) {
      const int bz0 = z >> 3, bz1 = bz0 > 0 ? bz0 - 1 : nby - 1, lz = z & 7;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int i = q >> 2, by = q & 2 ? b1 : b0, bz = q & 1 ? bz1 : bz0;
        if (i >= ox.n) break;
        const int b = (bz * nby + by) * nbx + ox.b[i];
        const float* a = p.gm_part + (size_t)(p.gm_nbrick + plan.first[b]) * 3 * kPad +
                         (ox.l[i] * kPY + wid + (q & 2 ? 8 : 0)) * kPZ + lz + (q & 1 ? 8 : 0);
        for (int e = plan.extra[b]; e > 0; e--, a += 3 * kPad)
          for (int c = 0; c < 3; c++) line[(c * kMZLines + wid) * LS + z] += a[c * kPad];
      }
    }
  }
  __syncthreads();
  // even and odd parts: line[z] + line[M - z], line[z] - line[M - z]
  for (int e = threadIdx.x; e < 3 * kMZLines * (H - 1); e += blockDim.x) {
    const int l = e / (H - 1), z = 1 + e - l * (H - 1);
    const float a = line[l * LS + z], b = line[l * LS + M - z];
    line[l * LS + z] = a + b;
    line[l * LS + M - z] = a - b;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 3 * kMZLines * kc1; e += blockDim.x) {
    const int c = e / (kMZLines * kc1), q = e - c * kMZLines * kc1, yl = q % kMZLines, nz = q / kMZLines;
    const float* v = line + (c * kMZLines + yl) * LS;
    float re = v[0] + ((nz & 1) ? -v[H] : v[H]), im = 0.f;
    int ph = 0;
#pragma unroll 4
    for (int z = 1; z < H; z++) {
      ph += nz;
      if (ph >= M) ph -= M;
      const float2 t = tw[ph];
      re = fmaf(v[z], t.x, re);
      im = fmaf(v[M - z], t.y, im);
    }
    p.gm_z[(((size_t)c * kc1 + nz) * M + x) * M + y0 + yl] = make_float2(re, im);
  }
}

// y axis: block (nz, eight x): G = ny S_y + nz S_z and S_x of every ny; a
// thread pair per (|ny|, x) takes even and odd y, and both signs of ny.
constexpr int kMYLines = 8;
__global__ void __launch_bounds__(512) k_mesh_y(KParams p) {
  extern __shared__ __align__(16) float smy[];
  const int M = p.gm_M, kc = p.kc, kc1 = kc + 1, Q = 2 * kc + 1, nz = blockIdx.x, x0 = blockIdx.y * kMYLines;
  const int LS = M + 2;            // 16 lanes (8 lines, even and odd y) in 16 bank pairs
  float2* tw = (float2*)smy;       // [M]
  float2* in = tw + M;             // [3][kMYLines][LS]
  for (int e = threadIdx.x; e < M; e += blockDim.x) tw[e] = p.gm_tw[e];
  // eight lines are one run of 8 M values; about six values per thread, loaded together
  for (int e0 = threadIdx.x; e0 < 3 * kMYLines * M; e0 += 8 * blockDim.x) {
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int e = e0 + i * blockDim.x, c = e / (kMYLines * M), q = e - c * kMYLines * M;
      if (c < 3) v[i] = p.gm_z[(((size_t)c * kc1 + nz) * M + x0) * M + q];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int e = e0 + i * blockDim.x, l = e / M;
      if (l < 3 * kMYLines) in[l * LS + e - l * M] = v[i];
    }
  }
  __syncthreads();
  const int half = threadIdx.x & 1, xl = threadIdx.x >> 1 & 7, ny = threadIdx.x >> 4;
  float a[3][4] = {};  // sums of x c, y s, x s, y c
  if (ny <= kc) {
    const float2* v = in + xl * LS + half;
    int ph = half * ny, step = 2 * ny;
    if (step >= M) step -= M;
#pragma unroll 4
    for (int y = 0; y < M; y += 2) {
      const float2 t = tw[ph];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float2 u = v[c * kMYLines * LS + y];
        a[c][0] = fmaf(u.x, t.x, a[c][0]);
        a[c][1] = fmaf(u.y, t.y, a[c][1]);
        a[c][2] = fmaf(u.x, t.y, a[c][2]);
        a[c][3] = fmaf(u.y, t.x, a[c][3]);
      }
      ph += step;
      if (ph >= M) ph -= M;
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int q = 0; q < 4; q++) a[c][q] += __shfl_xor_sync(kFull, a[c][q], 1);
  if (nz == kc && x0 == 0 && threadIdx.x < 96) {  // total moment, in the block with the fewest rows: fixed order
    const int c = threadIdx.x >> 5;
    double m = 0.0;
    for (int b0 = threadIdx.x & 31; b0 < p.gm_nitem; b0 += 512) {
      double v[16];  // loaded together: a trip's latency is most of this block's time
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const int b = b0 + 32 * i;
        v[i] = b < p.gm_nitem ? p.musum_part[3 * b + c] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < 16; i++) m += v[i];
    }
    m = warp_sum(m);
    if ((threadIdx.x & 31) == 0) p.musum[c] = m;
  }
  // the even thread writes +ny, the odd one -ny
  if (ny * ny + nz * nz > kc * kc || (half && (ny == 0 || nz == 0))) return;
  const float sg = half ? -1.f : 1.f, fy = sg * (float)ny, fz = (float)nz;
  float re[3], im[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    re[c] = fmaf(-sg, a[c][1], a[c][0]);
    im[c] = fmaf(sg, a[c][2], a[c][3]);
  }
  p.gm_y[((size_t)nz * Q + (half ? kc - ny : kc + ny)) * M + x0 + xl] =
      make_float4(fmaf(fy, re[1], fz * re[2]), fmaf(fy, im[1], fz * im[2]), re[0], im[0]);
}

// x axis, both ways: block per row (ny, nz): S(n) of its nx, the operand
// W(n) = conj(e S) / omega^3(n), and U = sum_nx W exp(2 pi i nx x / M),
// V = sum_nx nx W exp(..) of every x.  Groups of lanes share the sum over x of
// one |nx|.
constexpr int kMXThreads = 128;
__global__ void __launch_bounds__(kMXThreads) k_mesh_x(KParams p) {
  extern __shared__ __align__(16) float smx[];
  const int M = p.gm_M, kc = p.kc, kc1 = kc + 1, Q = 2 * kc + 1, tid = threadIdx.x;
  const int2 row = p.tc_row[blockIdx.x];  // (ny, nz)
  const int rd = row.y * Q + row.x + kc;
  float4* in = (float4*)smx;              // [M]
  float2* tw = (float2*)(in + M);         // [M]
  float4* pd = (float4*)(tw + M);         // [kc + 1] W(+) + W(-), W(+) - W(-)
  float* red = (float*)(pd + kc1);        // [parts][kc + 1][8]
  for (int e = tid; e < M; e += kMXThreads) {
    tw[e] = p.gm_tw[e];
    in[e] = p.gm_y[(size_t)rd * M + e];
  }
  // factors of the |nx| this thread finishes: e / omega^6, 1 / omega^3 of +nx, -nx
  int kp = -1, km = -1;
  float2 fp = make_float2(0.f, 0.f), fm = fp;
  if (tid < kc1) {
    kp = p.tc_kmap[blockIdx.x * Q + kc + tid];
    fp = p.gm_fac[blockIdx.x * Q + kc + tid];
    if (tid > 0) {
      km = p.tc_kmap[blockIdx.x * Q + kc - tid];
      fm = p.gm_fac[blockIdx.x * Q + kc - tid];
    }
  }
  __syncthreads();
  const int parts = kMXThreads / kc1, part = tid / kc1, ax = tid - part * kc1;
  if (part < parts) {
    float a[8] = {};
    int ph = (int)((long long)part * ax % M), step = (int)((long long)parts * ax % M);
    for (int x = part; x < M; x += parts) {
      const float4 v = in[x];
      const float2 t = tw[ph];
      a[0] = fmaf(v.x, t.x, a[0]);
      a[1] = fmaf(v.y, t.y, a[1]);
      a[2] = fmaf(v.x, t.y, a[2]);
      a[3] = fmaf(v.y, t.x, a[3]);
      a[4] = fmaf(v.z, t.x, a[4]);
      a[5] = fmaf(v.w, t.y, a[5]);
      a[6] = fmaf(v.z, t.y, a[6]);
      a[7] = fmaf(v.w, t.x, a[7]);
      ph += step;
      if (ph >= M) ph -= M;
    }
    float4* o = (float4*)(red + (part * kc1 + ax) * 8);
    o[0] = make_float4(a[0], a[1], a[2], a[3]);
    o[1] = make_float4(a[4], a[5], a[6], a[7]);
  }
  __syncthreads();
  if (tid < kc1) {
    float a[8] = {};
    for (int h = 0; h < parts; h++)
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] += red[(h * kc1 + tid) * 8 + q];
    const float f = (float)tid;
    float2 wp = make_float2(0.f, 0.f), wm = wp;
    if (kp >= 0) {
      const float sr = fmaf(f, a[4] - a[5], a[0] - a[1]), si = fmaf(f, a[6] + a[7], a[2] + a[3]);
      p.S[kp] = make_double2((double)(fp.y * sr), (double)(fp.y * si));
      wp = make_float2(fp.x * sr, -(fp.x * si));
    }
    if (km >= 0) {
      const float sr = fmaf(-f, a[4] + a[5], a[0] + a[1]), si = fmaf(-f, a[7] - a[6], a[3] - a[2]);
      p.S[km] = make_double2((double)(fm.y * sr), (double)(fm.y * si));
      wm = make_float2(fm.x * sr, -(fm.x * si));
    }
    pd[tid] = make_float4(wp.x + wm.x, wp.y + wm.y, wp.x - wm.x, wp.y - wm.y);
  }
  __syncthreads();
  for (int x = tid; x < M; x += kMXThreads) {
    // W+ e + W- e* = P cos + i D sin, and nx times D cos + i P sin
    float ur = pd[0].x, ui = pd[0].y, vr = 0.f, vi = 0.f;
    int ph = 0;
#pragma unroll 4
    for (int h = 1; h < kc1; h++) {
      ph += x;
      if (ph >= M) ph -= M;
      const float4 w = pd[h];
      const float2 t = tw[ph];
      const float f = (float)h, fc = f * t.x, fs = f * t.y;
      ur = fmaf(w.x, t.x, fmaf(-w.w, t.y, ur));
      ui = fmaf(w.y, t.x, fmaf(w.z, t.y, ui));
      vr = fmaf(w.z, fc, fmaf(-w.y, fs, vr));
      vi = fmaf(w.w, fc, fmaf(w.x, fs, vi));
    }
    p.gm_t[(size_t)rd * M + x] = make_float4(ur, ui, vr, vi);
  }
}

// y and z axes back to the mesh: block (two x, eight y): of the rows' U, V the
// sums over ny of (V, ny U, nz U) for every nz, then over nz the real field b, two
// points z and M - z per thread.
constexpr int kMIx = 2, kMIy = 8;
__global__ void __launch_bounds__(256) k_mesh_yz(KParams p) {
  extern __shared__ __align__(16) float smi[];
  const int M = p.gm_M, kc = p.kc, kc1 = kc + 1, Q = 2 * kc + 1;
  const int x0 = blockIdx.x * kMIx, y0 = blockIdx.y * kMIy;
  float4* in = (float4*)smi;                            // [kc1 Q][kMIx]
  float2* tw = (float2*)(in + (size_t)kc1 * Q * kMIx);  // [M]
  float2* mid = tw + M;                                 // [kMIx kMIy][kc1][3]
  for (int e = threadIdx.x; e < M; e += blockDim.x) tw[e] = p.gm_tw[e];
#pragma unroll 4
  for (int e = threadIdx.x; e < kc1 * Q * kMIx; e += blockDim.x)
    in[e] = p.gm_t[(size_t)(e / kMIx) * M + x0 + e % kMIx];
  __syncthreads();
  for (int e = threadIdx.x; e < kc1 * kMIx * kMIy; e += blockDim.x) {
    const int xl = e % kMIx, yl = e / kMIx % kMIy, nz = e / (kMIx * kMIy), y = y0 + yl;
    int m = 0;  // rows within the sphere: |ny| <= m
    while ((m + 1) * (m + 1) + nz * nz <= kc * kc) m++;
    const int lo = nz == 0 ? 0 : -m;
    float vr = 0.f, vi = 0.f, wr = 0.f, wi = 0.f, ur = 0.f, ui = 0.f;
    int ph = (int)((long long)(lo + M) * y % M);
    const float4* r = in + ((size_t)nz * Q + lo + kc) * kMIx + xl;
#pragma unroll 4
    for (int ny = lo; ny <= m; ny++, r += kMIx) {
      const float4 s = *r;
      const float2 t = tw[ph];
      const float er = fmaf(s.x, t.x, -s.y * t.y), ei = fmaf(s.x, t.y, s.y * t.x), f = (float)ny;
      ur += er;
      ui += ei;
      wr = fmaf(f, er, wr);
      wi = fmaf(f, ei, wi);
      vr = fmaf(s.z, t.x, fmaf(-s.w, t.y, vr));
      vi = fmaf(s.z, t.y, fmaf(s.w, t.x, vi));
      ph += y;
      if (ph >= M) ph -= M;
    }
    float2* o = mid + ((size_t)(yl * kMIx + xl) * kc1 + nz) * 3;
    const float fz = (float)nz;
    o[0] = make_float2(vr, vi);
    o[1] = make_float2(wr, wi);
    o[2] = make_float2(fz * ur, fz * ui);
  }
  __syncthreads();
  const int H = M / 2 + 1;
  for (int e = threadIdx.x; e < kMIx * kMIy * H; e += blockDim.x) {
    const int l = e / H, z = e - l * H;
    const float2* o = mid + (size_t)l * kc1 * 3;
    float c0 = 0.f, c1 = 0.f, c2 = 0.f, s0 = 0.f, s1 = 0.f, s2 = 0.f;
    int ph = 0;
#pragma unroll 4
    for (int nz = 0; nz < kc1; nz++, o += 3) {
      const float2 t = tw[ph], u0 = o[0], u1 = o[1], u2 = o[2];
      c0 = fmaf(u0.x, t.x, c0);
      s0 = fmaf(u0.y, t.y, s0);
      c1 = fmaf(u1.x, t.x, c1);
      s1 = fmaf(u1.y, t.y, s1);
      c2 = fmaf(u2.x, t.x, c2);
      s2 = fmaf(u2.y, t.y, s2);
      ph += z;
      if (ph >= M) ph -= M;
    }
    float4* out = p.gm_b + ((size_t)(x0 + l % kMIx) * M + y0 + l / kMIx) * M;
    out[z] = make_float4(c0 - s0, c1 - s1, c2 - s2, 0.f);
    if (z > 0 && z < M - z) out[M - z] = make_float4(c0 + s0, c1 + s1, c2 + s2, 0.f);
  }
}

// ----------------------------------------------------------- interpolation
//
// The brick's field in shared memory, a warp per particle.  Lane 9 axis + i
// evaluates the window's point i of an axis, value and derivative; then lane
// 9 r + c (27 of them) walks the rows y = 3 t + r of the window at z = c; the x, y, z
// factors are applied at the end of their loops, so a mesh point costs six
// multiply-adds (three without the force).
//
// Bound: shared-memory wavefronts (three per 27 mesh points, 27 times per particle)
// and issue: 36 / 29 us at N = 32768, M = 64 (41 / 35 with float4 points, four
// wavefronts; 46 / 37 from global memory, L1; 68 / 53 with the brick in the threads'
// registers, as in the spread, for its sums over the lanes).
// (b_x, b_y) rows are rotated by 9 y, so that the points of 16 lanes on three rows of
// nine lie in 16 pairs of banks; b_z rows are 21 apart (0 .. 8, 21 .. 29, 42 .. 50
// are 27 banks): three wavefronts for 27 points, where float4 takes four.
constexpr int kFZ = 21;
static_assert(kMW == 9 && kPZ == 16 && kPY == 16, "rotation and stride of the brick's rows");
constexpr int kInThreads = 384;
struct InterpSmem {
  float2 fxy[kPX * kPY * kPZ];
  float fz[kPX * kPY * kFZ];
  int j[kInThreads];
  BrickScan<kInThreads> scan;
};
template <bool FULL>
__global__ void __launch_bounds__(kInThreads, 2) k_mesh_interp(KParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  InterpSmem& sm = *(InterpSmem*)smem;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int M = p.gm_M, n = p.n, nbx = (M + kBX - 1) / kBX, nby = M / kBY;
  const int brick = mesh_brick(p);
  if (brick < 0) return;
  const int x0 = brick % nbx * kBX, y0 = brick / nbx % nby * kBY, z0 = brick / (nbx * nby) * kBZ;
  auto fold = [&](int i) { return i >= M ? i - M : i; };
#pragma unroll 8
  for (int e = tid; e < kPX * kPY * kPZ; e += kInThreads) {
    const int x = e / (kPY * kPZ), y = e / kPZ % kPY, z = e % kPZ;
    const float4 v = p.gm_b[((size_t)fold(x0 + x) * M + fold(y0 + y)) * M + fold(z0 + z)];
    sm.fxy[(x * kPY + y) * kPZ + ((z + kMW * y) & (kPZ - 1))] = make_float2(v.x, v.y);
    sm.fz[(x * kPY + y) * kFZ + z] = v.z;
  }
  const int rr = min(lane / kMW, 2), pt = lane % kMW;  // also the axis of the window values
  const bool on = lane < 3 * kMW;
  float cf[kMC];
#pragma unroll
  for (int d = 0; d < kMC; d++) cf[d] = p.gm_coef[pt * kMC + d];
  const float fB = (float)-p.cflux, fF = (float)(p.cforce * (double)M / p.two_pi);
  float *B = (float*)p.B, *F = (float*)p.F;
  brick_particles(
      p, sm.scan, x0, y0, z0,
      [&](int k, int j, int, const float (&)[3]) { sm.j[k] = j; },
      [&](int hits) {
        int kn = 0;
        int4 xn = make_int4(0, 0, 0, 0);
        float4 mn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (wid < hits) {
          kn = sm.j[wid];
          xn = p.s.xi[kn];
          if (FULL) mn = ((const float4*)p.s.mu)[kn];
        }
        for (int h = wid; h < hits; h += kInThreads / 32) {
          const int k = kn;
          const int4 xi = xn;
          const float4 mu = mn;
          if (h + kInThreads / 32 < hits) {  // the next particle
            kn = sm.j[h + kInThreads / 32];
            xn = p.s.xi[kn];
            if (FULL) mn = ((const float4*)p.s.mu)[kn];
          }
          float s0, s1, s2;
          auto start = [&](int v, int b0, float& s) {
            const int i = mesh_point(v, M, s) - kMH - b0;
            return i < 0 ? i + M : i;  // within the brick: less than M
          };
          const int ix = start(xi.x, x0, s0), iy = start(xi.y, y0, s1), iz = start(xi.z, z0, s2);
          const float s = rr == 0 ? s0 : (rr == 1 ? s1 : s2);
          float w = cf[kMC - 1], dw = 0.f;  // omega and, below, omega' (d/dz = 2 d/ds) times the moment
#pragma unroll
          for (int d = kMC - 2; d >= 0; d--) {
            if (FULL) dw = fmaf(dw, s, w);
            w = fmaf(w, s, cf[d]);
          }
          if (FULL) dw *= 2.f * (rr == 0 ? mu.x : (rr == 1 ? mu.y : mu.z));
          const float2* fxy[3];
#pragma unroll
          for (int t = 0; t < 3; t++) {
            const int y = iy + 3 * t + rr;
            fxy[t] = sm.fxy + (ix * kPY + y) * kPZ + ((iz + pt + kMW * y) & (kPZ - 1));
          }
          const float* fz = sm.fz + (ix * kPY + iy + rr) * kFZ + iz + pt;
          // packed: (x, y) and (z, z) of a mesh point against the window value and, in
          // the other half or another sum, its derivative
          float2 gxy[3] = {}, gz[3] = {}, hxy[3] = {};
#pragma unroll 3
          for (int a = 0; a < kMW; a++) {
            const float xv = __shfl_sync(kFull, w, a), xd = FULL ? __shfl_sync(kFull, dw, a) : 0.f;
#pragma unroll
            for (int t = 0; t < 3; t++) {
              const float2 v = fxy[t][a * kPY * kPZ];
              const float z = fz[(a * kPY + 3 * t) * kFZ];
              gxy[t] = __ffma2_rn(v, make_float2(xv, xv), gxy[t]);
              if (FULL) {
                hxy[t] = __ffma2_rn(v, make_float2(xd, xd), hxy[t]);
                gz[t] = __ffma2_rn(make_float2(z, z), make_float2(xv, xd), gz[t]);
              } else {
                gz[t].x = fmaf(z, xv, gz[t].x);
              }
            }
          }
          float zv = __shfl_sync(kFull, w, 2 * kMW + pt), zd = FULL ? __shfl_sync(kFull, dw, 2 * kMW + pt) : 0.f;
          if (!on) zv = zd = 0.f;
          float gy[3] = {}, hy[3] = {};
#pragma unroll
          for (int t = 0; t < 3; t++) {
            const float yv = __shfl_sync(kFull, w, kMW + 3 * t + rr);
            const float g[3] = {gxy[t].x, gxy[t].y, gz[t].x}, q[3] = {hxy[t].x, hxy[t].y, gz[t].y};
            const float yd = FULL ? __shfl_sync(kFull, dw, kMW + 3 * t + rr) : 0.f;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              gy[c] = fmaf(yv, g[c], gy[c]);
              if (FULL) hy[c] = fmaf(yv, q[c], fmaf(yd, g[c], hy[c]));
            }
          }
          if constexpr (FULL) {
            float o[8];
#pragma unroll
            for (int c = 0; c < 3; c++) {
              o[c] = zv * gy[c];
              o[4 + c] = fmaf(zv, hy[c], zd * gy[c]);
            }
            o[3] = o[7] = 0.f;
            const float r = warp_sums<8>(o, lane);
            const int c = lane >> 2;
            if ((lane & 3) == 0 && (c & 3) < 3) {
              if (c < 4)
                B[c * n + k] = fB * r;
              else
                F[(c - 4) * n + k] = fF * r;
            }
          } else {
            float o[4] = {zv * gy[0], zv * gy[1], zv * gy[2], 0.f};
            const float r = warp_sums<4>(o, lane);
            if ((lane & 7) == 0 && lane < 24) B[(lane >> 3) * n + k] = fB * r;
          }
        }
      });
}

// ------------------------------------------------------------- launches

// One item per brick, as long as no plan was made.
void mesh_plan_init(int M, std::vector<int>& out) {
  const int nb = mesh_bricks(M);
  out.assign(mesh_plan_ints(M), 0);
  const MeshPlan plan(out.data(), nb);
  for (int b = 0; b < nb; b++) plan.item[b] = make_int2(b, 1 << 16);
}

int launch_kmesh(cudaStream_t st, const KParams& p, bool full, cudaEvent_t* ev) {
  const int M = p.gm_M, kc1 = p.kc + 1, Q = 2 * p.kc + 1;
  allow_smem<k_mesh_spread>();
  const int items = p.gm_nitem;
  k_mesh_spread<<<items, kBrThreads, sizeof(SpreadSmem), st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[0], st, cudaEventRecordExternal);
  k_mesh_z<<<dim3(M, M / kMZLines), 256, sizeof(float) * (2 * M + 3 * kMZLines * (M + 1)), st>>>(p);
  k_mesh_y<<<dim3(kc1, M / kMYLines), (16 * kc1 + 31) / 32 * 32, sizeof(float2) * (M + 3 * kMYLines * (M + 2)), st>>>(p);
  k_mesh_x<<<p.tc_rows, kMXThreads, sizeof(float) * (6 * M + 4 * kc1 + 8 * kMXThreads), st>>>(p);
  const size_t smi = sizeof(float4) * kc1 * Q * kMIx + sizeof(float2) * (M + kMIx * kMIy * kc1 * 3);
  allow_smem<k_mesh_yz>();
  k_mesh_yz<<<dim3(M / kMIx, M / kMIy), 256, smi, st>>>(p);
  if (ev) cudaEventRecordWithFlags(ev[1], st, cudaEventRecordExternal);
  const size_t smf = sizeof(InterpSmem);
  if (full) {
    allow_smem<k_mesh_interp<true>>();
    k_mesh_interp<true><<<items, kInThreads, smf, st>>>(p);
  } else {
    allow_smem<k_mesh_interp<false>>();
    k_mesh_interp<false><<<items, kInThreads, smf, st>>>(p);
  }
  return 6;
}

}  // namespace md
