// md_real.cu -- kernel (b): real-space Ewald sum of the dipolar field, force
// and pressure, the hard-core overlap push and the short-range coating
// potentials.  Restates, per particle instead of per listed pair:
//   CompInteractVecs overlap handling   src/interaction.cpp:104-129
//   CompDipInteractEwaldR + EvalPressTensLR  src/interaction.cpp:383-422,
//                                         src/postprocessing.cpp:195-200
//   CompDipFieldEwaldR                  src/interaction.cpp:555-582
//   CompSterRep/CompElectrostatRep/CompForceVdW + EvalPressTensSR
//                                       src/interaction.cpp:766-832,
//                                       src/simulation.cpp:648-676
//
// Neighbour search.  The reference lists every pair with r < rc each step
// (all N(N-1)/2 pairs, CompInteractVecs).  Here a Verlet list with a skin
// holds, for each cell-sorted particle, the particles within rc + skin at the
// last build; it is rebuilt (on the device, inside the step) when some
// particle has moved more than skin/2 since then, so every pair that is now
// within rc is in the list.  Each evaluation tests the exact distance
// against rc like the reference.  Build: FP64 path one warp per particle
// (nbr_build64), mixed path one warp per two (nbr_build2); a warp walks the rows
// of its cell stencil, culled to the cells that intersect the search sphere,
// and a ballot compacts the hits (a pass into equal shares of the list's memory; a
// second one, after a prefix sum, when a share was too small).  If the
// list does not fit its capacity the evaluation scans the cells directly, with
// in-range pairs compacted into a per-warp shared-memory queue (correct,
// slower); the host then grows the list.
//
// Evaluation: one warp per particle; lanes take list entries 32 at a time (mixed
// path 64), gather the neighbour's coordinates and moment, and run the pair
// maths (erfc, exp, ~90 flops).  Per-lane sums are reduced with warp shuffles.
//
// Geometry (mixed path): 32-bit fixed-point coordinates (2^32 per box
// length); their wrapping difference is the exact minimum image, converted
// to FP32 once (relative error ~6e-8 in r at any distance).  The FP64 path
// uses FP64 box coordinates and the reference's fold (d > L/2 -> d - L,
// d < -L/2 -> d + L), with an FP32 pre-test that has a small margin.
//
// erfc: exp(-x^2), shared with the Gaussian term, times erfcx from a fit
// (erfcx32) on the mixed path and from tables of polynomials on the FP64 path
// (ewald64).
//
// Overlap push: CompInteractVecs moves cores apart in place while it walks
// the pairs, so later pairs see moved positions.  Here every overlap is
// resolved from the same starting positions (Jacobi): particle i collects
// -1/2 (dCont - r) r_hat_ij over its overlapping neighbours, r is clamped to
// dCont for the Ewald terms, and the displacement is applied with the
// translation step.  For configurations without overlaps the two agree.
//
// Roofline: mixed path FP32/SFU issue bound, FP64 path bound by the FP64 pipe
// (see the FP64 pair terms).  Algorithmic FLOPs per unordered in-range
// pair (counted from the reference formula): 113 full, 58 field only.
#include <algorithm>

#include "md_common.cuh"
#include "md_kernels.h"

namespace md {

constexpr int kRealWarps = 8;  // warps per block: list build, field + force with coating
// of the other passes (smaller blocks give finer occupancy steps)
constexpr int kFieldWarps = 4;

template <typename T>
struct Acc {
  T b0 = 0, b1 = 0, b2 = 0, f0 = 0, f1 = 0, f2 = 0, o0 = 0, o1 = 0, o2 = 0, p0 = 0, p1 = 0, p2 = 0;
};

// The erfcx fit in scalar code.
__device__ __forceinline__ float erfcx32(float z) {
  const float t = __fdividef(1.0f, fmaf(kErfcxA, z, 1.0f));
  float q = erfcx_c(7);
#pragma unroll
  for (int k = 6; k >= 0; k--) q = fmaf(q, t, erfcx_c(k));
  return t * q;
}

// Coating potentials of a pair inside rCutSR (CompSterRep,
// CompElectrostatRep, CompForceVdW): the scalar force along the unit vector,
// in FP64.  rd: the pair distance (clamped to contact here, as the
// reference's list length is); oi, oj: particle indices.
__device__ __forceinline__ double coat_force(const RealParams& p, double rd, int oi, int oj) {
  const double ri = p.rMag_u[oi], rj = p.rMag_u[oj];
  const double dc = ri + rj + p.cont_eps;
  if (rd < dc) rd = dc;
  // steric repulsion is asymmetric: dDelta and the prefactor use the
  // pair's lower particle index as "idx1" (interaction.cpp:768-775)
  const double ra = oi < oj ? ri : rj, rb = oi < oj ? rj : ri;
  const double dDelta = 2.0 * (ra + p.eff_len);
  double s = rd <= dDelta ? (2.0 * rb / (ra + rb)) * p.ster * ra * ra * log(dDelta / rd) : 0.0;
  s += (ri * rj / (ri + rj)) * p.elec * exp(-p.kappa * (rd - ri - rj));
  const double g1 = (rd - ri - rj) * (rd + ri + rj), g2 = rd * rd - (ri - rj) * (ri - rj);
  const double c4 = 4.0 * ri * rj;
  s += -p.vdw * rd * (c4 * c4 * c4) / (6.0 * g1 * g1 * g2 * g2);
  return s;
}

// Ewald pair terms for the pair vector (dx, dy, dz) from i to j (r2 < rc2),
// mixed path, in the direct cell scan.
template <bool FULL, bool COAT>
__device__ __forceinline__ void pair_terms(const RealParams& p, float dx, float dy, float dz, float r2, const float4& mi,
                                           const float4& mj, int oi, int oj, Acc<float>& a) {
  const float ir0 = rsqrtf(r2), r0 = r2 * ir0;
  const float ux = dx * ir0, uy = dy * ir0, uz = dz * ir0;
  float r = r0, ire = ir0;
  const float dcont = mi.w + mj.w + (float)p.cont_eps;
  if (r < dcont) {
    if constexpr (FULL) {
      const float h = 0.5f * (dcont - r);
      a.o0 -= h * ux;
      a.o1 -= h * uy;
      a.o2 -= h * uz;
    }
    r = dcont;
    ire = __fdividef(1.0f, r);
  }
  const float ire2 = ire * ire;
  const float re2 = r * r;
  const float e = __expf(-(float)p.al2 * re2), erfcv = e * erfcx32((float)p.alpha * r);
  const float t = (float)p.c2a * e * ire2;
  const float a1 = erfcv * ire2 * ire + t;
  const float a2 = 3.0f * a1 * ire2 + 2.0f * (float)p.al2 * t;
  const float d1 = mi.x * ux + mi.y * uy + mi.z * uz;
  const float d2 = mj.x * ux + mj.y * uy + mj.z * uz;
  const float c1 = a2 * d2 * re2;
  a.b0 += c1 * ux - a1 * mj.x;
  a.b1 += c1 * uy - a1 * mj.y;
  a.b2 += c1 * uz - a1 * mj.z;
  if constexpr (FULL) {
    const float a3 = 5.0f * a2 * ire2 + 4.0f * (float)p.al4 * t;
    const float m12 = mi.x * mj.x + mi.y * mj.y + mi.z * mj.z;
    const float s1 = (a2 * m12 - a3 * d1 * d2 * re2) * r;
    const float s2 = a2 * r;
    const float vx = s1 * ux + s2 * (d2 * mi.x + d1 * mj.x);
    const float vy = s1 * uy + s2 * (d2 * mi.y + d1 * mj.y);
    const float vz = s1 * uz + s2 * (d2 * mi.z + d1 * mj.z);
    a.f0 -= vx;
    a.f1 -= vy;
    a.f2 -= vz;
    a.p0 += r * ux * vy;
    a.p1 += r * ux * vz;
    a.p2 += r * uy * vz;
    if constexpr (COAT) {
      // pairs inside rCutSR (intRangeSR uses the unclamped distance,
      // interaction.cpp:115), in FP64
      if ((double)r2 < p.rcut_sr2) {
        const float sv = (float)coat_force(p, sqrt((double)dx * dx + (double)dy * dy + (double)dz * dz), oi, oj);
        a.f0 -= sv * ux;
        a.f1 -= sv * uy;
        a.f2 -= sv * uz;
        a.p0 += r * ux * sv * uy;
        a.p1 += r * ux * sv * uz;
        a.p2 += r * uy * sv * uz;
      }
    }
  }
}

// ------------------------------------------------------- FP64 pair terms
// GB300 issues an FP64 instruction of a warp in 64 cycles of an SM quarter
// (2 FMA per SM and cycle, 1/64 of FP32), so the FP64 passes are bound by the
// number of FP64 instructions per pair and by nothing else; table loads,
// integer and FP32 work are free beside them.  Hence
//  - the box fold is decided in FP32 on the float copies of the coordinates
//    (FP64 only next to half a box, where they cannot decide);
//  - 1/r comes from an FP32 seed and one third-order step (5 FP64
//    instructions); conversions between the formats are integer operations;
//  - erfc and exp come from tables (RealParams::gtab, etab): with s = alpha r,
//    exp(-s^2) = E_k P(s^2 - k/64) and erfc(s) + (2 s / sqrt(pi)) exp(-s^2) =
//    exp(-s^2) G(s), G = erfcx(s) + 2 s / sqrt(pi) (with the configuration's pi), each interval of width
//    1/128 a polynomial of degree 5; both to ~1e-16 (Taylor coefficients from
//    the differential equation of erfcx, economised with Chebyshev's T6).
// 78 FP64 instructions per pair (field, force and pressure), 50 for the field
// alone, against ~230 / ~170 with the library's erfc, exp and rsqrt.

// Minimum-image difference b - a of box coordinates, with the reference's
// fold (d > 1/2 -> d - 1, d < -1/2 -> d + 1); af, bf: their float copies.
__device__ __forceinline__ double fold64(double a, double b, float af, float bf) {
  const float d = bf - af;
  const float ad = fabsf(d);
  double v = b - a;
  if (fabsf(ad - 0.5f) < 1e-5f) {
    if (v > 0.5)
      v -= 1.0;
    else if (v < -0.5)
      v += 1.0;
  } else if (ad > 0.5f) {
    v -= __hiloint2double(d > 0.f ? 0x3ff00000 : (int)0xbff00000, 0);
  }
  return v;
}

// Ewald factors at distance r (ire = 1/r, s = alpha r, x = alpha^2 r^2 from
// r^2 itself: the exponential magnifies its error): q = exp(-x) / r^2 and
// g = G(s) / r; the pair coefficient a1 = q g, the Gaussian term t = c2a q.
__device__ __forceinline__ void ewald64(const RealParams& p, double ire, double ire2, double s, double x, double& q,
                                        double& g) {
  const float sf = narrow(s), xf = sf * sf;
  const int k = (int)(sf * 128.0f), kx = (int)fmaf(xf, 64.0f, 0.5f);
  double e, G;
  if ((unsigned)k < (unsigned)kGIntervals) {
    const double2* c = (const double2*)(p.gtab + 8 * k);  // c5, c4, .. c0, centre
    const double2 c01 = c[0], c23 = c[1], c45 = c[2];
    const double u = s - c[3].x;
    const double2 ek = p.etab[kx];  // (k/64, exp(-k/64))
    const double v = ek.x - x;      // exp(v), |v| <= 1/128
    G = fma(fma(fma(fma(fma(c01.x, u, c01.y), u, c23.x), u, c23.y), u, c45.x), u, c45.y);
    constexpr double h2 = 1.0 / 16384.0;  // (1/128)^2: economised exp series of degree 5
    double w = fma(1.0 / 120.0, v, 1.0 / 24.0 + h2 * (48.0 / 32.0 / 720.0));
    w = fma(w, v, 1.0 / 6.0);
    w = fma(w, v, 0.5 - h2 * h2 * (18.0 / 32.0 / 720.0));
    w = fma(w, v, 1.0);
    e = fma(w * ek.y, v, ek.y);
  } else {  // alpha r beyond the tables (s >= 6)
    e = exp(-x);
    G = erfcx(s) + p.c2a / p.alpha * s;
  }
  q = e * ire2;
  g = G * ire;
}

// Pair terms on the FP64 path for sorted particle j and self coordinates
// di / fi, moment mi.
template <bool FULL, bool COAT>
__device__ __forceinline__ void pair64(const RealParams& p, const double4_32a& di, const float4& fi,
                                       const double4_32a& mi, int oi, int j, Acc<double>& a) {
  const double4_32a dj = p.s.xd[j];
  const float4 fj = p.s.xf[j];
  const double4_32a mj = ((const double4_32a*)p.s.mu)[j];
  double dx = fold64(di.x, dj.x, fi.x, fj.x), dy = fold64(di.y, dj.y, fi.y, fj.y), dz = fold64(di.z, dj.z, fi.z, fj.z);
  double r2 = dx * dx + dy * dy + dz * dz;
  if (!(r2 < p.rc2)) return;
  bool sr = false;
  if constexpr (FULL && COAT) sr = r2 < p.rcut_sr2;
  double ire;
  if (r2 > 1e-30) {
    const double y0 = widen(rsqrtf(narrow(r2)));
    const double ee = fma(-r2 * y0, y0, 1.0);
    ire = fma(y0 * ee, fma(0.375, ee, 0.5), y0);
  } else {
    ire = rsqrt(r2);  // (nearly) coincident particles
  }
  double r = r2 * ire;
  const double r0 = r;
  const float dcf = (fi.w + fj.w + p.pk.eps) * 1.00001f;
  if (!(narrow(r) > dcf)) {  // near contact or overlapping
    const double dcont = mi.w + mj.w + p.cont_eps;
    if (r < dcont) {
      if constexpr (FULL) {
        const double h = 0.5 * (dcont - r) * ire;
        a.o0 -= h * dx;
        a.o1 -= h * dy;
        a.o2 -= h * dz;
      }
      // the pair vector rescaled to the contact length
      const double c = dcont * ire;
      dx *= c;
      dy *= c;
      dz *= c;
      r = dcont;
      r2 = r * r;
      ire = 1.0 / r;
    }
  }
  const double ire2 = ire * ire;
  double q, g;
  ewald64(p, ire, ire2, p.alpha * r, p.al2 * r2, q, g);
  const double a1 = q * g, t = p.c2a * q;
  const double a2 = fma(3.0 * ire2, a1, 2.0 * p.al2 * t);
  const double D2 = mj.x * dx + mj.y * dy + mj.z * dz;
  const double e2 = a2 * D2;
  a.b0 = fma(e2, dx, fma(-a1, mj.x, a.b0));
  a.b1 = fma(e2, dy, fma(-a1, mj.y, a.b1));
  a.b2 = fma(e2, dz, fma(-a1, mj.z, a.b2));
  if constexpr (FULL) {
    const double a3 = fma(5.0 * ire2, a2, 4.0 * p.al4 * t);
    const double D1 = mi.x * dx + mi.y * dy + mi.z * dz;
    const double m12 = mi.x * mj.x + mi.y * mj.y + mi.z * mj.z;
    double t1 = fma(-a3 * D1, D2, a2 * m12);
    const double e1 = a2 * D1;
    if constexpr (COAT) {
      if (sr) t1 += coat_force(p, r0, oi, p.s.perm[j]) * ire;  // along d / r
    }
    const double vx = fma(t1, dx, fma(e2, mi.x, e1 * mj.x));
    const double vy = fma(t1, dy, fma(e2, mi.y, e1 * mj.y));
    const double vz = fma(t1, dz, fma(e2, mi.z, e1 * mj.z));
    a.f0 -= vx;
    a.f1 -= vy;
    a.f2 -= vz;
    a.p0 = fma(dx, vy, a.p0);
    a.p1 = fma(dx, vz, a.p1);
    a.p2 = fma(dy, vz, a.p2);
  }
}

// ------------------------------------------------- packed pair terms (FP32)
// Two pairs at once in the halves of float2 operations (Blackwell's packed
// FP32 instructions: one issue slot for two FMAs, the FMA rate unchanged): two
// neighbours of the warp's particle.  Special functions stay scalar.
__device__ __forceinline__ float2 pk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 pk1(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Sums of the list loop.  Field only: b.  Field + force: b of the a1 terms, d
// times 2^32 of the a2 terms, e of a2 (mj.d), f of the force with the opposite sign
// without its terms along mi, p of the pressure's radial terms times 2^32
// (the end of the loop puts them together).
struct Acc2 {
  float2 b0 = {0.f, 0.f}, b1 = {0.f, 0.f}, b2 = {0.f, 0.f};
  float f0 = 0.f, f1 = 0.f, f2 = 0.f, p0 = 0.f, p1 = 0.f, p2 = 0.f;
  float d0 = 0.f, d1 = 0.f, d2 = 0.f, e = 0.f;
};

// Single-instruction approximations (PTX ex2/rsqrt/rcp .approx.ftz); their
// arguments here are never subnormal, so flushing changes nothing.
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Neighbours A and B: fixed-point pair vectors (dxf..), r2f = |d_fix|^2,
// moments ma, mb; inA, inB: the pair is within rc; stA, stB: it is a strong pair
// (its terms are added in FP64; it still pushes).  A pair that adds nothing has no
// weight: out of range it gets a distance of ~4e9 box lengths, where exp(-alpha^2
// r^2) is zero and the coefficients are, for any alpha, below 1e-28; a strong pair
// gets 1 / r = 0.  Same formulas as pair_terms; the pair vector stays
// in fixed-point units, their powers of 2^-32 folded into the constants, and
// the coefficients are negated (the fit's sign), which saves the sign of the
// field's second term.  push: the lane's overlap push in shared memory ([3][32]),
// rare.
//
// Field + force: with e1 = a2 (mi.d), e2 = a2 (mj.d), t1 = a2 m12 - a3 (mi.d)(mj.d)
//   F_ij = t1 d + e2 mi + e1 mj,  P_ab = sum over ordered pairs of d_a F_b.
// mi is the same for the whole list, so e2 mi is summed as e2.  In P the terms
// d_a e2 mi_b and d_a e1 mj_b turn into each other when the pair is taken in the
// other order, which the other particle's list holds, so the total takes
// 2 mi_b sum d_a e2, and that sum is the field's (d): per pair the pressure
// costs the five operations of t1 d_a d_b.  (A particle's own share of P is then
// not the sum over its list; only the total is ever used.)
//
// Bound: FP32 issue and the FMA pipe: 35 packed operations per two pairs for
// the field, 28 packed and 64 scalar with the force (43 and 36 + 90 with
// erfcc, pair weights, a scaled pair vector and P from F_ij).
template <bool FULL>
__device__ __forceinline__ void pair_terms2(const PairK& K, float wdc, float2 dxf, float2 dyf, float2 dzf, float2 r2f,
                                            bool inA, bool inB, bool stA, bool stB, const float4& mi,
                                            const float4& ma, const float4& mb, Acc2& s, float* push) {
  const float far2 = 3e38f;  // in fixed units
  float2 r2 = mul2(pk(inA ? r2f.x : far2, inB ? r2f.y : far2), pk1(5.421010862427522e-20f));  // 2^-64
  float2 ire = pk(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));  // 1 / r
  float2 r = mul2(r2, ire);
  const float2 dcont = pk(wdc + ma.w, wdc + mb.w);
  float2 r2e = r2;  // distance of the exponential
  if (r.x < dcont.x || r.y < dcont.y || stA || stB) {  // rare
    auto clamp = [&](float& rr, float& ir, float& re, float dc, float& x, float& y, float& z) {
      // overlapping cores: pushed apart, the pair vector rescaled to the contact length
      if constexpr (FULL) {
        const float h = 0.5f * (dc - rr) * ir * 2.3283064365386963e-10f;
        push[0] -= h * x;
        push[32] -= h * y;
        push[64] -= h * z;
      }
      const float g = dc * ir;
      x *= g;
      y *= g;
      z *= g;
      rr = dc;
      ir = rcp_ftz(dc);
      re = dc * dc;
    };
    if (r.x < dcont.x) clamp(r.x, ire.x, r2e.x, dcont.x, dxf.x, dyf.x, dzf.x);
    if (r.y < dcont.y) clamp(r.y, ire.y, r2e.y, dcont.y, dxf.y, dyf.y, dzf.y);
    // a strong pair adds nothing here: every coefficient has a factor 1 / r^2
    if (stA) ire.x = 0.f;
    if (stB) ire.y = 0.f;
  }
  const float2 ire2 = mul2(ire, ire);
  const float2 ee = mul2(r2e, pk1(K.ke));
  const float2 e = pk(ex2_ftz(ee.x), ex2_ftz(ee.y));  // exp(-alpha^2 r^2)
  const float2 den = fma2(r, pk1(K.kz), pk1(1.0f));
  const float2 t = pk(rcp_ftz(den.x), rcp_ftz(den.y));  // 1 / (1 + 0.42 alpha r)
  float2 q = pk1(-erfcx_c(7));
#pragma unroll
  for (int k = 6; k >= 0; k--) q = fma2(q, t, pk1(-erfcx_c(k)));
  const float2 erfcn = mul2(mul2(t, e), q);              // -erfc(alpha r)
  const float2 tn = mul2(mul2(e, pk1(K.c2an)), ire2);    // minus the Gaussian term
  const float2 a1n = fma2(mul2(erfcn, ire2), ire, tn);   // -a1
  if constexpr (FULL) {
    // packed coefficients, then each pair in scalar code: packed, the sums take
    // twice the registers, and at 6 blocks per SM the pass took 261 us
    // instead of 250 at 7 (N = 32768)
    const float2 a2 = fma2(mul2(a1n, pk1(K.a2a)), ire2, mul2(tn, pk1(K.a2t)));   // a2 2^-32
    const float2 a3n = fma2(mul2(a2, pk1(K.a3a)), ire2, mul2(tn, pk1(K.a3t)));   // -a3 2^-96
    auto assemble = [&](float a1s, float a2s, float a3s, float dx, float dy, float dz, const float4& mj) {
      const float D1 = fmaf(mi.z, dz, fmaf(mi.y, dy, mi.x * dx));
      const float D2 = fmaf(mj.z, dz, fmaf(mj.y, dy, mj.x * dx));
      const float m12 = fmaf(mi.z, mj.z, fmaf(mi.y, mj.y, mi.x * mj.x));
      const float e2 = a2s * D2, e1 = a2s * D1;
      s.b0.x = fmaf(a1s, mj.x, s.b0.x);
      s.b1.x = fmaf(a1s, mj.y, s.b1.x);
      s.b2.x = fmaf(a1s, mj.z, s.b2.x);
      s.d0 = fmaf(e2, dx, s.d0);
      s.d1 = fmaf(e2, dy, s.d1);
      s.d2 = fmaf(e2, dz, s.d2);
      s.e += e2;
      const float t1 = fmaf(a3s * D1, D2, a2s * m12);
      s.f0 = fmaf(t1, dx, fmaf(e1, mj.x, s.f0));
      s.f1 = fmaf(t1, dy, fmaf(e1, mj.y, s.f1));
      s.f2 = fmaf(t1, dz, fmaf(e1, mj.z, s.f2));
      const float tx = t1 * dx, ty = t1 * dy;
      s.p0 = fmaf(tx, dy, s.p0);
      s.p1 = fmaf(tx, dz, s.p1);
      s.p2 = fmaf(ty, dz, s.p2);
    };
    assemble(a1n.x, a2.x, a3n.x, dxf.x, dyf.x, dzf.x, ma);
    assemble(a1n.y, a2.y, a3n.y, dxf.y, dyf.y, dzf.y, mb);
  } else {
    // B += a2 (mj.d) d - a1 mj
    const float2 mjx = pk(ma.x, mb.x), mjy = pk(ma.y, mb.y), mjz = pk(ma.z, mb.z);
    const float2 D2 = fma2(mjz, dzf, fma2(mjy, dyf, mul2(mjx, dxf)));
    const float2 a2 = fma2(mul2(a1n, pk1(K.a2fa)), ire2, mul2(tn, pk1(K.a2ft)));  // a2 2^-64
    const float2 c1 = mul2(a2, D2);
    s.b0 = fma2(c1, dxf, fma2(a1n, mjx, s.b0));
    s.b1 = fma2(c1, dyf, fma2(a1n, mjy, s.b1));
    s.b2 = fma2(c1, dzf, fma2(a1n, mjz, s.b2));
  }
}

// Own coordinates of sorted particle k.
template <typename T>
struct Self {
  int4 si;
  double4_32a di;
  float x, y, z, w;
  int oi;
};

template <typename T, bool COAT>
__device__ __forceinline__ Self<T> load_self(const RealParams& p, int k) {
  Self<T> s;
  s.si = make_int4(0, 0, 0, 0);
  s.di = make_double4_32a(0, 0, 0, 0);
  if constexpr (std::is_same<T, float>::value) {
    s.si = p.s.xi[k];
    const float sc = 2.3283064365386963e-10f;
    s.x = (float)s.si.x * sc;  // of the cells' scan only
    s.y = (float)s.si.y * sc;
    s.z = (float)s.si.z * sc;
    s.w = 0.f;
    s.oi = s.si.w;
  } else {
    s.di = p.s.xd[k];
    const float4 f = p.s.xf[k];
    s.x = f.x;
    s.y = f.y;
    s.z = f.z;
    s.w = f.w;
    s.oi = COAT ? p.s.perm[k] : 0;
  }
  return s;
}

// Walks the cell-stencil rows of particle k and calls visit(in, j, r2) for
// every batch of 32 candidates (warp-synchronous).  `in` marks the candidates
// within the search radius by their float coordinates, with a margin above
// the rounding of those (a superset: list entries beyond rc carry no weight
// and the direct scan tests each pair again); r2 in box units.  FRESH: the
// cells are those of the coordinates (a build), so the image of a row's cells
// is the image of its particles and the shift is applied to the own position
// once per row; otherwise (the direct scan between builds) and on the one-cell
// grid each difference is folded.
template <bool FRESH, typename T, typename V>
__device__ __forceinline__ void scan_rows(const RealParams& p, int k, int lane, const Self<T>& me, double r2box,
                                          V&& visit) {
  const int ncx = p.grid.ncx, m = p.grid.reach, side = 2 * m + 1, R = side * side;
  const int cell = p.s.cell[k];
  const int cx = cell % ncx, cy = (cell / ncx) % ncx, cz = cell / (ncx * ncx);
  const float inv = 1.0f / (float)ncx;
  const float rt = (float)(sqrt(r2box) * (1.0 + 1e-6) + 2e-7);
  const float rct2 = rt * rt;
  const int* cs = p.s.cell_start;
  const float4* xf = p.s.xf;
  auto scan = [&](int s, int e, float mx, float my, float mz) {
    if (s >= e) return;
    // two batches of 32 candidates per turn, the next two loaded ahead
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 n0 = s + lane < e ? xf[s + lane] : z4, n1 = s + 32 + lane < e ? xf[s + 32 + lane] : z4;
    auto test = [&](int j, const float4& q) {
      float dx = q.x - mx, dy = q.y - my, dz = q.z - mz;
      if constexpr (!FRESH) {
        dx -= rintf(dx);
        dy -= rintf(dy);
        dz -= rintf(dz);
      }
      const float r2 = dx * dx + dy * dy + dz * dz;
      visit(j < e && j != k && r2 < rct2, j, r2);
    };
    for (int j = s + lane; j - lane < e; j += 64) {
      const float4 q0 = n0, q1 = n1;
      if (j + 64 < e) n0 = xf[j + 64];
      if (j + 96 < e) n1 = xf[j + 96];
      test(j, q0);
      if (j - lane + 32 < e) test(j + 32, q1);
    }
  };
  for (int rb = 0; rb < R; rb += 32) {
    const int r = rb + lane;
    int a0 = 0, b0 = 0, a1 = 0, b1 = 0;
    int code = 0;  // images (+1) of the first and second x segment, of y and of z, two bits each
    if (r < R) {
      const int dy = r % side - m, dz = r / side - m;
      const int uy = cy + dy, uz = cz + dz;
      int xlo = cx - m, xhi = cx + m;
      bool ok = true;
      if (ncx > 1) {
        const float ylo = uy * inv - 0.5f, yhi = ylo + inv, zlo = uz * inv - 0.5f, zhi = zlo + inv;
        const float ey = fmaxf(0.f, fmaxf(ylo - me.y, me.y - yhi));
        const float ez = fmaxf(0.f, fmaxf(zlo - me.z, me.z - zhi));
        const float d2 = ey * ey + ez * ez;
        ok = d2 < rct2;
        if (ok) {
          const float w = sqrtf(rct2 - d2);
          xlo = max(xlo, (int)floorf((me.x - w + 0.5f) * ncx));
          xhi = min(xhi, (int)floorf((me.x + w + 0.5f) * ncx));
        }
      }
      if (ok && xlo <= xhi) {
        const int wy = (uy + ncx) % ncx, wz = (uz + ncx) % ncx;
        const int base = (wz * ncx + wy) * ncx;
        const int iy = uy < 0 ? 0 : (uy >= ncx ? 2 : 1), iz = uz < 0 ? 0 : (uz >= ncx ? 2 : 1);
        int i0 = 1, i1 = 1;
        if (xlo < 0) {
          a0 = cs[base + xlo + ncx];
          b0 = cs[base + ncx];
          a1 = cs[base];
          b1 = cs[base + xhi + 1];
          i0 = 0;
        } else if (xhi >= ncx) {
          a0 = cs[base + xlo];
          b0 = cs[base + ncx];
          a1 = cs[base];
          b1 = cs[base + xhi - ncx + 1];
          i1 = 2;
        } else {
          a0 = cs[base + xlo];
          b0 = cs[base + xhi + 1];
        }
        code = i0 | i1 << 2 | iy << 4 | iz << 6;
      }
    }
    const int nr = min(32, R - rb);
    for (int q = 0; q < nr; q++) {
      const int s0 = __shfl_sync(kFull, a0, q), e0 = __shfl_sync(kFull, b0, q);
      const int s1 = __shfl_sync(kFull, a1, q), e1 = __shfl_sync(kFull, b1, q);
      const int cd = __shfl_sync(kFull, code, q);
      // a row of image i holds particles whose periodic copies lie i - 1 boxes on
      const float my = FRESH ? me.y + (float)(1 - (cd >> 4 & 3)) : me.y;
      const float mz = FRESH ? me.z + (float)(1 - (cd >> 6 & 3)) : me.z;
      scan(s0, e0, FRESH ? me.x + (float)(1 - (cd & 3)) : me.x, my, mz);
      scan(s1, e1, FRESH ? me.x + (float)(1 - (cd >> 2 & 3)) : me.x, my, mz);
    }
  }
}

// ------------------------------------------------------- neighbour list

// FP64 path: the neighbours of each particle within rc + skin, one warp per
// particle, into its share of the list's memory, or (SECOND) anew when one was
// longer than that (see nbr_build2).
template <bool SECOND>
__device__ __forceinline__ void nbr_build64(const RealParams& p, int bx) {
  if (SECOND && (p.flags->overflow || !p.flags->refill)) return;
  const int lane = threadIdx.x & 31, k = bx * kRealWarps + (threadIdx.x >> 5);
  if (k >= p.n) return;
  const Self<double> me = load_self<double, false>(p, k);
  const int off = SECOND ? p.nbr_off[k] : k * p.nbr_share, room = SECOND ? 0x7fffffff : p.nbr_share;
  int cnt = 0;
  int* out = p.nbr + off;
  auto visit = [&](bool in, int j, float) {
    const unsigned mask = __ballot_sync(kFull, in);
    const int at = cnt + __popc(mask & lanemask_lt());
    if (in && at < room) out[at] = j;
    cnt += __popc(mask);
  };
  if (p.grid.ncx > 1)
    scan_rows<true, double>(p, k, lane, me, p.rl2, visit);
  else
    scan_rows<false, double>(p, k, lane, me, p.rl2, visit);
  if (!SECOND && lane == 0) {
    p.nbr_cnt[k] = cnt;
    p.nbr_off[k] = off;
  }
}

// Mixed path: one warp builds the lists of two consecutive sorted particles
// (2 w, 2 w + 1), which are close (the cells hold ~4 particles; periodic images
// across the ends of a row): the rows are set up and the candidates loaded
// once for both.
//
// Search.  The pair's bounding box, grown by the list radius, gives the rows of
// cells and per row the x range; 32 rows are set up at a time, one per lane,
// and then taken four at a time by eight lanes each (rows hold ~40 particles),
// the shift to a row's periodic image applied to the own positions.  Where the
// box does not fit into the periodic cell (few cells, or two particles far
// apart), and on the one-cell grid, all particles are tested with a fold.
//
// With strong pairs on, each neighbour is also classified per particle
// (|mu_i|^2 |mu_j|^2 > strong_w4sq r^8 at this build): strong entries carry the
// sign bit in the list and are copied, as (i, j), into the strong list.  A pair is
// classified, with its moment and fixed-point distance fetched, only when it is
// near enough for the largest moment to make it strong.
//
// The first pass writes each list into an equal share of the capacity (1.3 times
// the mean and 64 entries, where the system is uniform) and counts; the second
// fills the strong list, from the near pairs alone, and writes the lists again,
// one after another, when one did not fit its share.  Counting first and filling
// after the scan took 119 + 161 us at N = 20011, this 150 + 36.
constexpr unsigned kStrong = 0x80000000u;
constexpr int kNbrIndex = 0x7fffffff;

template <bool SECOND>
__device__ __forceinline__ void nbr_build2(const RealParams& p, int bx) {
  const bool refill = SECOND && p.flags->refill, cls = p.strong, sfill = SECOND && cls && !p.flags->soverflow;
  if (SECOND && (p.flags->overflow || !(refill || sfill))) return;
  const int lane = threadIdx.x & 31, w = bx * kRealWarps + (threadIdx.x >> 5);
  const int n = p.n, k1 = 2 * w, k2 = min(k1 + 1, n - 1);
  if (k1 >= n) return;
  const bool two = k2 > k1;
  if (SECOND && !refill && p.snbr_cnt[k1] + (two ? p.snbr_cnt[k2] : 0) == 0) return;
  const float4* xf = p.s.xf;
  const float4 f1 = xf[k1], f2 = xf[k2];
  float ex = f2.x - f1.x, ey = f2.y - f1.y, ez = f2.z - f1.z;  // the second particle's nearest image
  ex -= rintf(ex);
  ey -= rintf(ey);
  ez -= rintf(ez);
  const float4* gmu = (const float4*)p.s.mu;
  float m1 = 0.f, m2 = 0.f, near1 = -1.f, near2 = -1.f;
  if (cls) {
    const float4 u = gmu[k1], v = gmu[k2];
    m1 = u.x * u.x + u.y * u.y + u.z * u.z;
    m2 = v.x * v.x + v.y * v.y + v.z * v.z;
    near1 = sqrtf(sqrtf(m1 / p.strong_w4sq)) * 1.001f;  // |mu_j| <= mu_max = 1
    near2 = sqrtf(sqrtf(m2 / p.strong_w4sq)) * 1.001f;
  }
  int c1 = 0, c2 = 0, sc1 = 0, sc2 = 0;
  const int o1 = SECOND ? p.nbr_off[k1] : k1 * p.nbr_share, o2 = SECOND ? p.nbr_off[k2] : k2 * p.nbr_share;
  const int room = SECOND ? 0x7fffffff : p.nbr_share;
  int *out1 = p.nbr + o1, *out2 = p.nbr + o2;
  int2 *so1 = nullptr, *so2 = nullptr;
  if (sfill) {
    so1 = p.snbr + p.snbr_off[k1];
    so2 = p.snbr + p.snbr_off[k2];
  }
  const float rl = (float)(sqrt(p.rl2) * (1.0 + 1e-6) + 2e-7), rl2 = rl * rl;
  auto strong = [&](int k, int j, float mk) {
    const float4 mj = gmu[j];
    const int4 si = p.s.xi[k], sj = p.s.xi[j];
    const float sc = 2.3283064365386963e-10f;
    const float dx = (float)(sj.x - si.x) * sc, dy = (float)(sj.y - si.y) * sc, dz = (float)(sj.z - si.z) * sc;
    const float q2 = dx * dx + dy * dy + dz * dz, q4 = q2 * q2;
    return mk * (mj.x * mj.x + mj.y * mj.y + mj.z * mj.z) > p.strong_w4sq * (q4 * q4);
  };
  auto visit = [&](bool lists, bool strongs, bool valid, int j, float ra, float rb) {
    const bool in1 = valid && ra < rl2 && j != k1, in2 = valid && rb < rl2 && j != k2 && two;
    const unsigned ma = __ballot_sync(kFull, in1), mb = __ballot_sync(kFull, in2);
    unsigned j1 = (unsigned)j, j2 = (unsigned)j;
    const bool n1 = in1 && ra < near1, n2 = in2 && rb < near2;
    if (__any_sync(kFull, n1 || n2)) {
      const bool s1 = n1 && strong(k1, j, m1), s2 = n2 && strong(k2, j, m2);
      const unsigned sa = __ballot_sync(kFull, s1), sb = __ballot_sync(kFull, s2);
      if (strongs && s1) so1[sc1 + __popc(sa & lanemask_lt())] = make_int2(k1, j);
      if (strongs && s2) so2[sc2 + __popc(sb & lanemask_lt())] = make_int2(k2, j);
      if (s1) j1 |= kStrong;
      if (s2) j2 |= kStrong;
      sc1 += __popc(sa);
      sc2 += __popc(sb);
    }
    if (lists) {
      const int a = c1 + __popc(ma & lanemask_lt()), b = c2 + __popc(mb & lanemask_lt());
      if (in1 && a < room) out1[a] = (int)j1;
      if (in2 && b < room) out2[b] = (int)j2;
    }
    c1 += __popc(ma);
    c2 += __popc(mb);
  };
  const int ncx = p.grid.ncx;
  const float inv = 1.0f / (float)ncx;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  auto search = [&](float rt, bool lists, bool strongs) {
    const float rt2 = rt * rt;
    if (ncx > 1 && fmaxf(fmaxf(fabsf(ex), fabsf(ey)), fabsf(ez)) + 2.f * rt < 1.f - 2.f * inv) {
      const float xlo = f1.x + fminf(ex, 0.f), xhi = f1.x + fmaxf(ex, 0.f);
      const float ylo = f1.y + fminf(ey, 0.f), yhi = f1.y + fmaxf(ey, 0.f);
      const float zlo = f1.z + fminf(ez, 0.f), zhi = f1.z + fmaxf(ez, 0.f);
      auto cell = [&](float x) { return (int)floorf((x + 0.5f) * (float)ncx); };
      const int cy0 = cell(ylo - rt), ny = cell(yhi + rt) - cy0 + 1, cz0 = cell(zlo - rt), nz = cell(zhi + rt) - cz0 + 1;
      const int* cs = p.s.cell_start;
      for (int rb = 0; rb < ny * nz; rb += 32) {
        // lane: one row; a0, l0 / a1, l1: its x range, split at the box's end
        const int r = rb + lane;
        int a0 = 0, l0 = 0, a1 = 0, l1 = 0;
        int code = 0;  // images (+1): x of the two segments, y, z, two bits each
        if (r < ny * nz) {
          const int uy = cy0 + r % ny, uz = cz0 + r / ny;
          const float yc = uy * inv - 0.5f, zc = uz * inv - 0.5f;
          const float dy = fmaxf(0.f, fmaxf(yc - yhi, ylo - yc - inv)), dz = fmaxf(0.f, fmaxf(zc - zhi, zlo - zc - inv));
          const float d2 = dy * dy + dz * dz;
          if (d2 < rt2) {
            const float h = sqrtf(rt2 - d2);
            const int x0 = cell(xlo - h), x1 = cell(xhi + h);
            const int iy = uy < 0 ? 0 : (uy >= ncx ? 2 : 1), iz = uz < 0 ? 0 : (uz >= ncx ? 2 : 1);
            const int* row = cs + ((uz - (iz - 1) * ncx) * ncx + (uy - (iy - 1) * ncx)) * ncx;
            int i0 = 1, i1 = 1;
            if (x0 < 0) {
              a0 = row[x0 + ncx];
              l0 = row[ncx] - a0;
              a1 = row[0];
              l1 = row[x1 + 1] - a1;
              i0 = 0;
            } else if (x1 >= ncx) {
              a0 = row[x0];
              l0 = row[ncx] - a0;
              a1 = row[0];
              l1 = row[x1 - ncx + 1] - a1;
              i1 = 2;
            } else {
              a0 = row[x0];
              l0 = row[x1 + 1] - a0;
            }
            code = i0 | i1 << 2 | iy << 4 | iz << 6;
          }
        }
        const int nr = min(32, ny * nz - rb);
        for (int q = 0; q < nr; q += 4) {
          const int src = q + (lane >> 3);  // lanes past the last row hold empty ranges
          const int b0 = __shfl_sync(kFull, a0, src), n0 = __shfl_sync(kFull, l0, src);
          const int b1 = __shfl_sync(kFull, a1, src) - n0, len = n0 + __shfl_sync(kFull, l1, src);
          const int cd = __shfl_sync(kFull, code, src);
          const int top = __reduce_max_sync(kFull, len);
          // a row of image i holds particles whose periodic copies lie i - 1 boxes on
          const float xa = f1.x + (float)(1 - (cd & 3)), xb = f1.x + (float)(1 - (cd >> 2 & 3));
          const float y = f1.y + (float)(1 - (cd >> 4 & 3)), z = f1.z + (float)(1 - (cd >> 6 & 3));
          int t = lane & 7;
          float4 nxt = t < len ? xf[(t < n0 ? b0 : b1) + t] : z4;
          for (int t0 = 0; t0 < top; t0 += 8, t += 8) {
            const float4 c = nxt;
            const int j = (t < n0 ? b0 : b1) + t;
            if (t + 8 < len) nxt = xf[(t + 8 < n0 ? b0 : b1) + t + 8];
            const float dx = c.x - (t < n0 ? xa : xb), dy = c.y - y, dz = c.z - z;
            const float gx = dx - ex, gy = dy - ey, gz = dz - ez;
            visit(lists, strongs, t < len, j, dx * dx + dy * dy + dz * dz, gx * gx + gy * gy + gz * gz);
          }
        }
      }
    } else {
      for (int j0 = 0; j0 < n; j0 += 32) {
        const int j = j0 + lane;
        const float4 c = j < n ? xf[j] : z4;
        float dx = c.x - f1.x, dy = c.y - f1.y, dz = c.z - f1.z;
        dx -= rintf(dx);
        dy -= rintf(dy);
        dz -= rintf(dz);
        float gx = c.x - f2.x, gy = c.y - f2.y, gz = c.z - f2.z;
        gx -= rintf(gx);
        gy -= rintf(gy);
        gz -= rintf(gz);
        visit(lists, strongs, j < n, j, dx * dx + dy * dy + dz * dz, gx * gx + gy * gy + gz * gz);
      }
    }
  };
  if (!SECOND || refill) search(rl, true, false);
  if (sfill) {
    // only the near pairs: well inside the list radius (near1 and near2 hold a
    // margin over the classification, so both passes find the same strong pairs), or
    // the whole of it
    const float nr = fmaxf(near1, near2);
    sc1 = sc2 = 0;
    search(nr < 0.98f * rl2 ? sqrtf(nr) * 1.0001f + 2e-7f : rl, false, true);
  }
  if (!SECOND && lane == 0) {
    p.nbr_cnt[k1] = c1;
    p.nbr_off[k1] = o1;
    if (two) {
      p.nbr_cnt[k2] = c2;
      p.nbr_off[k2] = o2;
    }
    if (cls) {
      p.snbr_cnt[k1] = sc1;
      if (two) p.snbr_cnt[k2] = sc2;
    }
  }
}

template <typename T, bool SECOND>
__device__ __forceinline__ void nbr_build(const RealParams& p, int bx) {
  if (!p.flags->rebuild) return;
  if constexpr (std::is_same<T, float>::value)
    nbr_build2<SECOND>(p, bx);
  else
    nbr_build64<SECOND>(p, bx);
}

// Exclusive scan of cnt[0, n) into off[0, n] by one block of 1024 threads;
// returns the total to every thread.  Offsets saturate at INT_MAX (the list is
// then flagged as overflowing).  Each warp takes a contiguous 32nd, 32
// coalesced values at a time (a run of n / 1024 values per thread touched a
// cache line per thread and load: 28 us at n = 20011).
__device__ __forceinline__ long long block_scan_counts(const int* cnt, int* off, int n) {
  __shared__ long long wsum[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = ((n + 31) / 32 + 31) & ~31;
  const int b = min(w * per, n), e = min(b + per, n);
  long long local = 0;
#pragma unroll 4
  for (int i = b + lane; i < e; i += 32) local += cnt[i];
  local = warp_sum(local);
  if (lane == 0) wsum[w] = local;
  __syncthreads();
  if (w == 0) {
    const long long v = wsum[lane];
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    wsum[lane] = incl - v;
    if (lane == 31) wsum[32] = incl;
  }
  __syncthreads();
  long long run = wsum[w];
  int nxt = b + lane < e ? cnt[b + lane] : 0;
  for (int i0 = b; i0 < e; i0 += 32) {
    const int v = nxt;
    if (i0 + 32 + lane < e) nxt = cnt[i0 + 32 + lane];
    int incl = i0 + lane < e ? v : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    if (i0 + lane < e) off[i0 + lane] = (int)min(run + incl - v, (long long)0x7fffffff);
    run += __shfl_sync(kFull, incl, 31);
  }
  const long long total = wsum[32];
  if (threadIdx.x == 0) off[n] = (int)min(total, (long long)0x7fffffff);
  return total;
}

// Offsets of the Verlet list (block half 0) and of the strong list (half 1);
// flags overflow.
__device__ __forceinline__ void nbr_scan(const RealParams& p, int half) {
  StepFlags* flags = p.flags;
  if (!flags->rebuild) return;
  if (half == 0) {
    // the lists lie in their shares unless one is longer
    int top = 0;
    long long tot = 0;
#pragma unroll 4
    for (int i = threadIdx.x; i < p.n; i += 1024) {
      const int c = p.nbr_cnt[i];
      top = max(top, c);
      tot += c;
    }
    __shared__ long long wsum[32];
    __shared__ int wtop[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    tot = warp_sum(tot);
    top = __reduce_max_sync(kFull, top);
    if (lane == 0) {
      wsum[w] = tot;
      wtop[w] = top;
    }
    __syncthreads();
    tot = warp_sum(wsum[lane]);
    top = __reduce_max_sync(kFull, wtop[lane]);
    const bool refill = top > p.nbr_share;
    if (refill)
      block_scan_counts(p.nbr_cnt, p.nbr_off, p.n);
    else if (threadIdx.x == 0)
      p.nbr_off[p.n] = (int)min(tot, (long long)0x7fffffff);
    if (threadIdx.x == 0) {
      flags->refill = refill;
      flags->overflow = refill && tot > p.nbr_cap ? 1 : 0;
    }
  } else {
    // a build that did not classify leaves the strong list unusable until the
    // next build that does (the FP64 kernels then contribute nothing)
    const long long stot = p.strong ? block_scan_counts(p.snbr_cnt, p.snbr_off, p.n) : 0;
    if (threadIdx.x == 0) flags->soverflow = p.strong ? (stot > p.scap ? 1 : 0) : 1;
  }
}

// ------------------------------------------------------------ strong pairs
//
// The FP32 pair maths rounds every pair term to ~1e-7 of its size.  In a
// polydisperse system the reference's error scale is the contact force of
// the smallest particles, and near-contact pairs of large particles carry
// terms of ~10-100 such contact forces, so those few pairs (~0.2 % of the
// list at N = 32768, log-normal sigma 0.2) hold most of the FP32 error.  They
// are classified at each list build by the force weight |mu_i| |mu_j| / r^4
// and evaluated in FP64 with the reference's formula
// (src/interaction.cpp:396-417), one thread per entry of the strong list.
// The FP32 passes do this work themselves: the warps of k_real take the
// strong list in chunks of 32 entries, spread evenly over the grid, before
// their own particle, so the FP64 pipe (a small fraction of the FP32 rate on
// GB300, otherwise idle here) works under the FP32 pair loop of the other
// warps.  Each entry's terms go to svals; the integrator adds a particle's
// entries in list order (deterministic).  The FP32 pass keeps the overlap
// push of these pairs; the distance is clamped to contact here too.
// g1(s) = erfc(s) + (2 s / sqrt(pi)) exp(-s^2), the factor of 1/r^3 in the
// pair coefficient a1 (s = alpha r).  From its power series for s <= 1.5:
// g1 = 1 - (4 / sqrt(pi)) s^3 sum_k (-1)^k s^2k / (k! (2k + 3)), 18 terms
// (relative error < 3e-10 at s = 1.5, at the FP64 rounding level below
// s = 1), one branch-free polynomial instead of erfc's range branches;
// beyond, with erfc.  ex = exp(-s^2).
__device__ __forceinline__ double ewald_g1(double s, double ex) {
  const double x = s * s;
  if (x <= 2.25) {
    double q = -7.598533119852758e-17;
    q = fma(q, x, 1.3655649521106815e-15);
    q = fma(q, x, -2.317322342975702e-14);
    q = fma(q, x, 3.7002405153966856e-13);
    q = fma(q, x, -5.537601323041936e-12);
    q = fma(q, x, 7.732132217728926e-11);
    q = fma(q, x, -1.0020843354176688e-09);
    q = fma(q, x, 1.1981443140863431e-08);
    q = fma(q, x, -1.3122532963802806e-07);
    q = fma(q, x, 1.3053467000835422e-06);
    q = fma(q, x, -1.1671335200746965e-05);
    q = fma(q, x, 9.259259259259259e-05);
    q = fma(q, x, -0.000641025641025641);
    q = fma(q, x, 0.003787878787878788);
    q = fma(q, x, -0.018518518518518517);
    q = fma(q, x, 0.07142857142857142);
    q = fma(q, x, -0.2);
    q = fma(q, x, 0.3333333333333333);
    return fma(-2.256758334191025 * s * x, q, 1.0);  // 4 / sqrt(pi)
  }
  return erfc(s) + 1.1283791670955126 * s * ex;  // 2 / sqrt(pi)
}

// The FP64 terms of strong entry (i, j): v[0..2] field, and for FULL
// v[3..5] force, v[6..8] pressure.
template <bool FULL>
__device__ __forceinline__ void strong_entry(const RealParams& p, int2 ij, double v[9]) {
  const float4* gmu = (const float4*)p.s.mu;
  const int4 xi = p.s.xi[ij.x], xj = p.s.xi[ij.y];
  const float4 fi = gmu[ij.x], fj = gmu[ij.y];
  const double sc = 2.3283064365386963e-10;  // 2^-32
  // wrapping differences of the fixed-point coordinates: the exact minimum image
  const double dx = (double)(int)((unsigned)xj.x - (unsigned)xi.x) * sc;
  const double dy = (double)(int)((unsigned)xj.y - (unsigned)xi.y) * sc;
  const double dz = (double)(int)((unsigned)xj.z - (unsigned)xi.z) * sc;
  const double r2 = dx * dx + dy * dy + dz * dz;
  double ire = rsqrt(r2), r = r2 * ire;
  const double ux = dx * ire, uy = dy * ire, uz = dz * ire;
  const double dcont = (double)fi.w + (double)fj.w + p.cont_eps;
  if (r < dcont) {
    r = dcont;
    ire = 1.0 / r;
  }
  const double ire2 = ire * ire, re2 = r * r;
  const double ex = exp(-p.al2 * re2);
  const double t = p.c2a * ex * ire2;
  const double a1 = ewald_g1(p.alpha * r, ex) * ire2 * ire;  // = erfc(alpha r) / r^3 + t
  const double a2 = 3.0 * a1 * ire2 + 2.0 * p.al2 * t;
  double mix = fi.x, miy = fi.y, miz = fi.z, mjx = fj.x, mjy = fj.y, mjz = fj.z;
  if (p.smm) {  // the master moments in FP64 (the sorted view holds them rounded to FP32)
    const int n = p.n, pi = p.s.perm[ij.x], pj = p.s.perm[ij.y];
    const double gi = p.smag[pi], gj = p.smag[pj];
    mix = p.smm[pi] * gi;
    miy = p.smm[n + pi] * gi;
    miz = p.smm[2 * n + pi] * gi;
    mjx = p.smm[pj] * gj;
    mjy = p.smm[n + pj] * gj;
    mjz = p.smm[2 * n + pj] * gj;
  }
  const double d2 = mjx * ux + mjy * uy + mjz * uz;
  const double c1 = a2 * d2 * re2;
  v[0] = c1 * ux - a1 * mjx;
  v[1] = c1 * uy - a1 * mjy;
  v[2] = c1 * uz - a1 * mjz;
  if constexpr (FULL) {
    const double a3 = 5.0 * a2 * ire2 + 4.0 * p.al4 * t;
    const double d1 = mix * ux + miy * uy + miz * uz;
    const double m12 = mix * mjx + miy * mjy + miz * mjz;
    const double s1 = (a2 * m12 - a3 * d1 * d2 * re2) * r;
    const double s2 = a2 * r;
    const double vx = s1 * ux + s2 * (d2 * mix + d1 * mjx);
    const double vy = s1 * uy + s2 * (d2 * miy + d1 * mjy);
    const double vz = s1 * uz + s2 * (d2 * miz + d1 * mjz);
    v[3] = -vx;
    v[4] = -vy;
    v[5] = -vz;
    v[6] = r * ux * vy;
    v[7] = r * ux * vz;
    v[8] = r * uy * vz;
  }
}

// The chunks of the strong list that warp k (one warp per particle) takes:
// with C chunks of 32 entries and n warps, every stride-th warp, stride =
// n / C, takes one chunk (or each warp several when C > n).  A chunk's
// entries are grouped by owner particle (list order); the field and force
// terms are added per owner within the chunk (segmented warp sum, fixed
// order) and stored at the owner's first entry in the chunk, so a particle
// has one partial per chunk it spans.  The pressure, needed only as a total,
// is added over the whole chunk and stored at the chunk's first entry.
template <bool FULL>
__device__ __forceinline__ void strong_chunks(const RealParams& p, int k, int lane) {
  const StepFlags* fl = p.flags;
  if (fl->overflow || fl->soverflow) return;
  const int total = (int)min((long long)p.snbr_off[p.n], p.scap);
  const int chunks = (total + 31) >> 5;
  if (chunks == 0) return;
  const int n = p.n;
  const int stride = max(1, n / chunks);
  if (k % stride) return;
  const int step = (n + stride - 1) / stride;
  const size_t cap = (size_t)p.scap;
  constexpr int NS = FULL ? 6 : 3;  // components summed per owner
  for (int c = k / stride; c < chunks; c += step) {
    const int e = c * 32 + lane;
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    int owner = -1 - lane;  // lanes past the end: segments of their own
    if (e < total) {
      const int2 ij = p.snbr[e];
      if ((unsigned)ij.x < (unsigned)n && (unsigned)ij.y < (unsigned)n) {  // always, after a build
        owner = ij.x;
        strong_entry<FULL>(p, ij, v);
      }
    }
    // segmented suffix sums: lane l ends with the sum over [l, end of its run]
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ow = __shfl_down_sync(kFull, owner, o);
      const bool same = lane + o < 32 && ow == owner;
#pragma unroll
      for (int q = 0; q < NS; q++) {
        const double t = __shfl_down_sync(kFull, v[q], o);
        if (same) v[q] += t;
      }
    }
    const int prev = __shfl_up_sync(kFull, owner, 1);
    if (e < total && (lane == 0 || prev != owner)) {
#pragma unroll
      for (int q = 0; q < NS; q++) p.svals[q * cap + e] = v[q];
    }
    if constexpr (FULL) {
#pragma unroll
      for (int q = 6; q < 9; q++) {
        const double t = warp_sum(v[q]);
        if (lane == 0) p.svals[q * cap + e] = t;
      }
    }
  }
}

// ------------------------------------------------------------ evaluation

// Direct scan of particle k's cells when the list did not fit: in-range
// candidates are compacted through the warp's queue q, eval(j) for each.
template <typename T, typename E>
__device__ __forceinline__ void direct_scan(const RealParams& p, int k, int lane, const Self<T>& me, int* q, E&& eval) {
  int head = 0, tail = 0;
  auto flush = [&](int cnt) {
    __syncwarp();
    const int j = lane < cnt ? q[(head + lane) & 63] : 0;
    __syncwarp();
    head += cnt;
    if (lane < cnt) eval(j);
  };
  scan_rows<false, T>(p, k, lane, me, p.rc2, [&](bool in, int j, float) {
    const unsigned mask = __ballot_sync(kFull, in);
    if (in) q[(tail + __popc(mask & lanemask_lt())) & 63] = j;
    tail += __popc(mask);
    if (tail - head >= 32) flush(32);
  });
  if (tail - head > 0) flush(tail - head);
}

// FP64 path: one warp per particle, lanes take list entries.
template <bool FULL, bool COAT, int NW>
__device__ __forceinline__ void real_eval64(const RealParams& p, int bx) {
  __shared__ int q[NW][64];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = bx * NW + wib;
  if (k >= p.n) return;  // whole warp; no block-level synchronisation below
  Acc<double> a;
  const double4_32a mi = ((const double4_32a*)p.s.mu)[k];
  const Self<double> me = load_self<double, COAT>(p, k);
  const float4 mf = make_float4(me.x, me.y, me.z, me.w);
  auto eval = [&](int j) { pair64<FULL, COAT>(p, me.di, mf, mi, me.oi, j, a); };
  if (!p.flags->overflow) {
    const int* lst = p.nbr + p.nbr_off[k];
    const int cnt = p.nbr_cnt[k];
    int jn = lane < cnt ? lst[lane] : 0;
    for (int t0 = 0; t0 < cnt; t0 += 32) {
      const int j = jn;
      const bool valid = t0 + lane < cnt;
      if (t0 + 32 + lane < cnt) jn = lst[t0 + 32 + lane];
      if (valid) eval(j);
    }
  } else {
    direct_scan<double>(p, k, lane, me, q[wib], eval);
  }
  double *B = (double*)p.B, *F = (double*)p.F, *O = (double*)p.ov;
  const int n = p.n;
  if constexpr (FULL) {
    double v[16] = {a.b0, a.b1, a.b2, a.f0, a.f1, a.f2, a.p0, a.p1, a.p2, a.o0, a.o1, a.o2, 0, 0, 0, 0};
    const double s = warp_sums<16>(v, lane);
    const int c = lane >> 1;
    if ((lane & 1) == 0 && c < 12) {
      if (c < 3)
        B[c * n + k] = s;
      else if (c < 6)
        F[(c - 3) * n + k] = s;
      else if (c < 9)
        p.Ppart[3 * k + c - 6] = s;
      else
        O[(c - 9) * n + k] = s;
    }
  } else {
    double v[4] = {a.b0, a.b1, a.b2, 0};
    const double s = warp_sums<4>(v, lane);
    if ((lane & 7) == 0 && lane < 24) B[(lane >> 3) * n + k] = s;
  }
}

constexpr int kNearCap = 128;  // coating pairs a warp queues

// Mixed path: one warp per particle, lanes take two list entries at a time in
// the halves of packed FP32 operations.
//
// Bound: FP32 issue and the FMA pipe (see pair_terms2); 250 / 185 us for field +
// force / field at N = 32768 and 7.5e7 ordered pairs (273 / 193 with the arithmetic
// before).  The list comes from DRAM, ~1 us away, longer than an iteration of a
// warp, so its entries are loaded two iterations (128) ahead.
//
// A list per two particles (the union of their neighbours, each neighbour in
// both halves: gathers and list bytes shared, everything packed) took 293 /
// 182 us: the union is 14 % longer than one list, and the field + force pass
// needs 96 registers.
template <bool FULL, bool COAT, int NW>
__device__ __forceinline__ void real_eval32(const RealParams& p, int bx) {
  __shared__ int q[NW][64];
  __shared__ float pushes[FULL ? NW : 1][3][32];
  constexpr bool NEAR = FULL && COAT;
  __shared__ int nearj[NEAR ? NW : 1][kNearCap], nearn[NEAR ? NW : 1];
  __shared__ float nearf[NEAR ? NW : 1][kNearCap];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kq = bx * NW + wib;
  if (!NEAR && kq >= p.n) return;  // whole warp; only the coating pairs synchronise the block
  const bool on = kq < p.n;
  const int k = NEAR ? min(kq, p.n - 1) : kq;
  float* push = FULL ? &pushes[wib][0][lane] : nullptr;
  if constexpr (FULL) push[0] = push[32] = push[64] = 0.f;
  if constexpr (!COAT) {
    if (p.strong && !p.flags->overflow) strong_chunks<FULL>(p, k, lane);
  }
  const int n = p.n;
  const float4* gmu = (const float4*)p.s.mu;
  const float4 mi = gmu[k];
  Acc2 s;
  int nn = 0;  // coating pairs of this warp waiting in nearj
  // Coating force along the unit vector of the pair (k, j) (sorted indices); 0
  // beyond rCutSR, which is tested on the unclamped distance (interaction.cpp:115).
  auto near_force = [&](int ks, int j) {
    const int4 a = p.s.xi[ks], c = p.s.xi[j];
    const float sc = 2.3283064365386963e-10f;  // 2^-32
    const float dx = (float)(c.x - a.x) * sc, dy = (float)(c.y - a.y) * sc, dz = (float)(c.z - a.z) * sc;
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (!((double)r2 < p.rcut_sr2)) return 0.f;
    return (float)coat_force(p, sqrt((double)dx * dx + (double)dy * dy + (double)dz * dz), a.w, c.w);
  };
  auto near_add = [&](int j, float sv) {
    const int4 a = p.s.xi[k], c = p.s.xi[j];
    const float sc = 2.3283064365386963e-10f;
    const float dx = (float)(c.x - a.x) * sc, dy = (float)(c.y - a.y) * sc, dz = (float)(c.z - a.z) * sc;
    const float r2 = dx * dx + dy * dy + dz * dz, ir = rsqrtf(r2), r = fmaxf(r2 * ir, mi.w + gmu[j].w + (float)p.cont_eps);
    const float ux = dx * ir, uy = dy * ir, uz = dz * ir;
    s.f0 += sv * ux;
    s.f1 += sv * uy;
    s.f2 += sv * uz;
    const float q = r * sv * 4294967296.f;
    s.p0 += q * ux * uy;
    s.p1 += q * ux * uz;
    s.p2 += q * uy * uz;
  };
  if (!p.flags->overflow) {
    const int4 si = p.s.xi[k];
    const float rc2_fix = p.pk.rc2f;  // (rc / (L 2^-32))^2
    const float wdc = mi.w + p.pk.eps;  // own core radius + contact offset
    const int* lst = p.nbr + p.nbr_off[k];
    const int cnt = on ? p.nbr_cnt[k] : 0;
    // flags count only when the context evaluates the strong pairs in FP64
    const unsigned fs = !COAT && p.strong && !p.flags->soverflow ? kStrong : 0u;
    // a margin over rCutSR; near_force decides
    const float near2 = NEAR ? (float)(p.rcut_sr2 * 18446744073709551616.0) * 1.00001f : 0.f;
    // the list is streamed once per pass: evict-first loads leave L1 to the gathers
    auto entry = [&](int t) { return t < cnt ? (unsigned)__ldcs(lst + t) : (unsigned)k; };
    auto process = [&](unsigned ea, unsigned eb, int t) {
      const int ja = (int)(ea & kNbrIndex), jb = (int)(eb & kNbrIndex);
      const int4 sa = p.s.xi[ja], sb = p.s.xi[jb];
      const float4 ma = gmu[ja], mb = gmu[jb];
      // wrapping 32-bit differences are the exact minimum image
      const float2 dxf = pk((float)(sa.x - si.x), (float)(sb.x - si.x));
      const float2 dyf = pk((float)(sa.y - si.y), (float)(sb.y - si.y));
      const float2 dzf = pk((float)(sa.z - si.z), (float)(sb.z - si.z));
      const float2 r2f = fma2(dzf, dzf, fma2(dyf, dyf, mul2(dxf, dxf)));
      const bool inA = t < cnt && r2f.x < rc2_fix, inB = t + 32 < cnt && r2f.y < rc2_fix;
      if constexpr (NEAR) {
        const bool na = inA && r2f.x < near2, nb = inB && r2f.y < near2;
        if (__any_sync(kFull, na || nb)) {
          if (nn > kNearCap - 64) {  // rarely: no room for another 64
            __syncwarp();
            for (int e = lane; e < nn; e += 32) near_add(nearj[wib][e], near_force(k, nearj[wib][e]));
            nn = 0;
            __syncwarp();
          }
          const unsigned a = __ballot_sync(kFull, na), c = __ballot_sync(kFull, nb);
          if (na) nearj[wib][nn + __popc(a & lanemask_lt())] = ja;
          nn += __popc(a);
          if (nb) nearj[wib][nn + __popc(c & lanemask_lt())] = jb;
          nn += __popc(c);
        }
      }
      pair_terms2<FULL>(p.pk, wdc, dxf, dyf, dzf, r2f, inA, inB, inA && (ea & fs), inB && (eb & fs), mi, ma, mb, s,
                        push);
    };
    unsigned n0 = entry(lane), n1 = entry(32 + lane), n2 = entry(64 + lane), n3 = entry(96 + lane);
    for (int t = lane; t - lane < cnt; t += 128) {
      const unsigned c0 = n0, c1 = n1, c2 = n2, c3 = n3;
      n0 = entry(t + 128);
      n1 = entry(t + 160);
      n2 = entry(t + 192);
      n3 = entry(t + 224);
      process(c0, c1, t);
      if (t - lane + 64 < cnt) process(c2, c3, t + 64);
    }
    if constexpr (FULL) {
      s.f0 = fmaf(s.e, mi.x, s.f0);
      s.f1 = fmaf(s.e, mi.y, s.f1);
      s.f2 = fmaf(s.e, mi.z, s.f2);
      s.p0 = fmaf(2.f * s.d0, mi.y, s.p0);
      s.p1 = fmaf(2.f * s.d0, mi.z, s.p1);
      s.p2 = fmaf(2.f * s.d1, mi.z, s.p2);
      s.b0.x = fmaf(s.d0, 2.3283064365386963e-10f, s.b0.x);
      s.b1.x = fmaf(s.d1, 2.3283064365386963e-10f, s.b1.x);
      s.b2.x = fmaf(s.d2, 2.3283064365386963e-10f, s.b2.x);
    }
  } else {
    // the direct scan: scalar
    const Self<float> me = load_self<float, COAT>(p, k);
    Acc<float> a;
    auto eval = [&](int j) {
      const int4 sj = p.s.xi[j];
      const float4 mj = gmu[j];
      const float dxf = (float)(sj.x - me.si.x), dyf = (float)(sj.y - me.si.y), dzf = (float)(sj.z - me.si.z);
      if (dxf * dxf + dyf * dyf + dzf * dzf < p.pk.rc2f) {
        const float sc = 2.3283064365386963e-10f;  // 2^-32
        const float dx = dxf * sc, dy = dyf * sc, dz = dzf * sc;
        pair_terms<FULL, COAT>(p, dx, dy, dz, dx * dx + dy * dy + dz * dz, mi, mj, me.oi, COAT ? sj.w : 0, a);
      }
    };
    direct_scan<float>(p, k, lane, me, q[wib], eval);
    s.b0.x = a.b0;
    s.b1.x = a.b1;
    s.b2.x = a.b2;
    if constexpr (FULL) {
      s.f0 = -a.f0;
      s.f1 = -a.f1;
      s.f2 = -a.f2;
      s.p0 = a.p0 * 4294967296.f;
      s.p1 = a.p1 * 4294967296.f;
      s.p2 = a.p2 * 4294967296.f;
      push[0] = a.o0;
      push[32] = a.o1;
      push[64] = a.o2;
    }
  }
  if constexpr (NEAR) {
    // The coating pairs of the block's particles, one per thread: FP64, few per
    // particle (evaluated as they came, a warp paid the whole FP64 sequence
    // for each of its close pairs, and an FP64 compare for every list entry:
    // 31.6 -> 22.3 us at N = 2744).
    if (lane == 0) nearn[wib] = nn;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) total += nearn[w];
    for (int e = threadIdx.x; e < total; e += NW * 32) {
      int w = 0, t = e;
      while (t >= nearn[w]) t -= nearn[w++];
      nearf[w][t] = near_force(bx * NW + w, nearj[w][t]);
    }
    __syncthreads();
    for (int e = lane; e < nn; e += 32) near_add(nearj[wib][e], nearf[wib][e]);
    if (!on) return;
  }
  float *B = (float*)p.B, *F = (float*)p.F, *O = (float*)p.ov;
  if constexpr (FULL) {
    float v[16] = {s.b0.x, s.b1.x, s.b2.x, s.f0, s.f1, s.f2, s.p0, s.p1, s.p2, push[0], push[32], push[64], 0, 0, 0, 0};
    const float t = warp_sums<16>(v, lane);
    const int c = lane >> 1;
    if ((lane & 1) == 0 && c < 12) {
      if (c < 3)
        B[c * n + k] = t;
      else if (c < 6)
        F[(c - 3) * n + k] = -t;
      else if (c < 9)
        p.Ppart[3 * k + c - 6] = (double)(t * 2.3283064365386963e-10f);
      else
        O[(c - 9) * n + k] = t;
    }
  } else {
    float v[4] = {s.b0.x + s.b0.y, s.b1.x + s.b1.y, s.b2.x + s.b2.y, 0.f};
    const float t = warp_sums<4>(v, lane);
    if ((lane & 7) == 0 && lane < 24) B[(lane >> 3) * n + k] = t;
  }
}

static int num_sms() {
  // initialised once (thread-safe: contexts may be created on several threads)
  static const int nsm = [] {
    int dev = 0, k = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&k, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || k <= 0) k = 148;
    return k;
  }();
  return nsm;
}

// ------------------------------------------------------------ entry points

// Grid-stride over the particle blocks: most steps do not rebuild, and a
// grid of a few blocks per SM then costs one flag read per block.
template <typename T, bool SECOND>
__global__ void __launch_bounds__(kRealWarps * 32) k_nbr_build(RealParams p, int nblk) {
  if (!p.flags->rebuild) return;
  for (int bx = blockIdx.x; bx < nblk; bx += gridDim.x) nbr_build<T, SECOND>(p, bx);
}
__global__ void __launch_bounds__(1024) k_nbr_scan(RealParams p) { nbr_scan(p, blockIdx.x); }
// The FP32 passes without coating keep the occupancy of their pair loops
// (field: 8 blocks of 4 warps per SM, 64 registers; field + force: 7 blocks,
// 72 registers): the FP64 strong-pair code in the same kernel must not
// raise the register count.  Measured at N = 32768: field + force 250 us at 7,
// 259 at 6; field 186 at 8, 188 at 9, 246 at 10 (spills).
template <typename T, bool FULL, bool COAT>
__global__ void __launch_bounds__(((FULL && COAT) ? kRealWarps : kFieldWarps) * 32,
                                  std::is_same<T, float>::value ? (COAT ? 2 : (FULL ? 7 : 8)) : 1) k_real(RealParams p) {
  constexpr int NW = (FULL && COAT) ? kRealWarps : kFieldWarps;
  if constexpr (std::is_same<T, float>::value)
    real_eval32<FULL, COAT, NW>(p, blockIdx.x);
  else
    real_eval64<FULL, COAT, NW>(p, blockIdx.x);
}

// In-range ordered pairs of the last evaluation's geometry.
template <typename T>
__global__ void __launch_bounds__(kRealWarps * 32) k_count_pairs(RealParams p, unsigned long long* out) {
  __shared__ int q[kRealWarps][64];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * kRealWarps + wib;
  if (k >= p.n) return;
  int np = 0;
  const Self<T> me = load_self<T, false>(p, k);
  auto eval = [&](int j) {
    if constexpr (std::is_same<T, float>::value) {
      const int4 s = p.s.xi[j];
      const float dx = (float)(s.x - me.si.x), dy = (float)(s.y - me.si.y), dz = (float)(s.z - me.si.z);
      np += fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < p.pk.rc2f;
    } else {
      const double4_32a s = p.s.xd[j];
      const float4 f = p.s.xf[j];
      const double dx = fold64(me.di.x, s.x, me.x, f.x), dy = fold64(me.di.y, s.y, me.y, f.y),
                   dz = fold64(me.di.z, s.z, me.z, f.z);
      np += dx * dx + dy * dy + dz * dz < p.rc2;
    }
  };
  if (!p.flags->overflow) {
    const int b = p.nbr_off[k], e = b + p.nbr_cnt[k];
    for (int t = b + lane; t < e; t += 32) eval(p.nbr[t] & kNbrIndex);
  } else {
    direct_scan<T>(p, k, lane, me, q[wib], eval);
  }
  np = __reduce_add_sync(kFull, np);
  if (lane == 0) atomicAdd(out, (unsigned long long)np);
}

// persistent: blocks stride over the task table (see md_cells.cu); the
// list build and the pair loop are warp-private (no block barrier)
template <bool SECOND>
__global__ void __launch_bounds__(kRealWarps * 32) k_nbr_build_packed(const RealParams* __restrict__ ps,
                                                                      const Task* __restrict__ tk, int ntask, WorkQ* wq,
                                                                      const unsigned* anyrb) {
  if (!__ldcg(anyrb)) return;  // the whole grid: no system rebuilds this step
  for_tasks<false>(tk, ntask, wq, [&](const Task& t) {
      nbr_build<float, SECOND>(ps[t.rep], t.blk);
  });
}
__global__ void __launch_bounds__(1024) k_nbr_scan_packed(const RealParams* __restrict__ ps) {
  const RealParams p = ps[blockIdx.x];
  nbr_scan(p, blockIdx.y);
}
// the block shape of the single-system passes (k_real): 8 warps with
// coating in the field + force pass, otherwise 4; 6 (field + force) or 8
// (field) blocks per SM (32 systems of 500 to 4000 particles: 6.85 ms per five
// steps; 6.92 at 6 / 7, 6.97 at 5 / 7)
template <bool FULL, bool COAT>
__global__ void __launch_bounds__(((FULL && COAT) ? kRealWarps : kFieldWarps) * 32, COAT ? 2 : (FULL ? 6 : 8))
    k_real_packed(const RealParams* __restrict__ ps, const Task* __restrict__ tk, int ntask, WorkQ* wq, int run) {
  for_tasks<false>(tk, ntask, wq, [&](const Task& t) {
    const RealParams& p = ps[t.rep];
    if constexpr (FULL && COAT) {
      real_eval32<FULL, COAT, kRealWarps>(p, t.blk);
    } else {
#pragma unroll 1
      for (int s = 0; s < run; s++) real_eval32<FULL, COAT, kFieldWarps>(p, run * t.blk + s);
    }
  });
}

// Share of an SM's 228 KB that the FP32 passes ask for as shared memory, in
// percent; the rest is the L1 cache, which serves their gathers (85 % of
// its throughput in the field pass).  They need 25 KB.  Left to itself the driver
// widens the shared part for the k-space kernels on the other stream, and the
// two run each other down: per step at N = 32768 (131072) 779 us (5.07 ms),
// slower than one after the other (715 us, 4.33 ms); at 16 % 672 us (4.27 ms), at
// 60 % 769 us (4.96 ms); 32 small systems together 7.35 -> 6.85 ms per five steps.
constexpr int kRealCarveout = 16;
static void keep_l1(const void* kern) {
  cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, kRealCarveout);
}

int real_blocks(int n) { return (n + kRealWarps - 1) / kRealWarps; }
int real_pass_blocks(int n, int run) { return (n + kFieldWarps * run - 1) / (kFieldWarps * run); }
int nbr_blocks(int n, bool fp64) { return real_blocks(fp64 ? n : (n + 1) / 2); }

int launch_nbr(cudaStream_t st, const RealParams& p, bool fp64) {
  const int nsm = num_sms();
  const int nblk = nbr_blocks(p.n, fp64);
  dim3 grid(std::min(nblk, 8 * nsm)), block(kRealWarps * 32);
  if (fp64)
    k_nbr_build<double, false><<<grid, block, 0, st>>>(p, nblk);
  else
    k_nbr_build<float, false><<<grid, block, 0, st>>>(p, nblk);
  k_nbr_scan<<<2, 1024, 0, st>>>(p);
  if (fp64)
    k_nbr_build<double, true><<<grid, block, 0, st>>>(p, nblk);
  else
    k_nbr_build<float, true><<<grid, block, 0, st>>>(p, nblk);
  return 3;
}

void launch_count_pairs(cudaStream_t st, const RealParams& p, unsigned long long* out, bool fp64) {
  if (fp64)
    k_count_pairs<double><<<real_blocks(p.n), kRealWarps * 32, 0, st>>>(p, out);
  else
    k_count_pairs<float><<<real_blocks(p.n), kRealWarps * 32, 0, st>>>(p, out);
}

int launch_real(cudaStream_t st, const RealParams& p, bool full, bool fp64) {
  const int nw = (full && p.coat) ? kRealWarps : kFieldWarps;
  dim3 grid((p.n + nw - 1) / nw), block(nw * 32);
  if (fp64) {
    if (full)
      p.coat ? k_real<double, true, true><<<grid, block, 0, st>>>(p)
             : k_real<double, true, false><<<grid, block, 0, st>>>(p);
    else
      k_real<double, false, false><<<grid, block, 0, st>>>(p);
  } else {
    keep_l1((const void*)k_real<float, true, false>);
    keep_l1((const void*)k_real<float, false, false>);
    if (full)
      p.coat ? k_real<float, true, true><<<grid, block, 0, st>>>(p)
             : k_real<float, true, false><<<grid, block, 0, st>>>(p);
    else
      k_real<float, false, false><<<grid, block, 0, st>>>(p);
  }
  return 1;
}

int launch_nbr_packed(cudaStream_t st, const RealParams* ps, int R, const Packed& real, const unsigned* anyrb) {
  const int th = kRealWarps * 32;
  if (real.n)
    k_nbr_build_packed<false><<<persistent_grid((const void*)k_nbr_build_packed<false>, th, 0, real.n), th, 0, st>>>(
        ps, real.tasks, real.n, real.wq, anyrb);
  k_nbr_scan_packed<<<dim3(R, 2), 1024, 0, st>>>(ps);
  if (real.n)
    k_nbr_build_packed<true><<<persistent_grid((const void*)k_nbr_build_packed<true>, th, 0, real.n), th, 0, st>>>(
        ps, real.tasks, real.n, real.wq, anyrb);
  return 3;
}

int launch_real_packed(cudaStream_t st, const RealParams* ps, const Packed& real, const Packed& pass, int run, bool full,
                       bool coat) {
  keep_l1((const void*)k_real_packed<true, false>);
  keep_l1((const void*)k_real_packed<false, false>);
  auto go = [&](auto kern, const Packed& tb, int th) {
    kern<<<persistent_grid((const void*)kern, th, 0, tb.n), th, 0, st>>>(ps, tb.tasks, tb.n, tb.wq, run);
  };
  if (full && coat) {
    if (!real.n) return 0;
    go(k_real_packed<true, true>, real, kRealWarps * 32);
  } else {
    if (!pass.n) return 0;
    full ? go(k_real_packed<true, false>, pass, kFieldWarps * 32) : go(k_real_packed<false, false>, pass, kFieldWarps * 32);
  }
  return 1;
}

}  // namespace md
