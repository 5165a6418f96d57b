// Device-side ideal-MHD arithmetic for the B200 step kernels.
//
// Same scheme and operation order as the reference's precision-generic device functions
// (lib/MHDKernels/src/glm_physics.jl): cons2prim/prim2cons :11-23, fast_speed :24-27,
// phys_flux_x :28-34, rot_to/rot_flux_from :36-45 (here a compile-time axis permutation),
// MonCen/minmod :47-59, PPM :188-200, recon offsets :212-223, GLM pair :234-238,
// LLF/HLL :239-252, HLLD (Miyoshi & Kusano 2005) :255-307, riemann/riemann_ct :317-348.
// Compiled with fast math, as the reference's `@fastmath` kernels are.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pmf {

enum { RECON_PLM = 0, RECON_PPM = 1, RECON_PLM_MINMOD = 2 };
// RS_HLLD_CENSUS: HLLD that also counts its single-star degeneracy cases (HlldCensus); only the
// census step instantiates it.
enum { RS_HLLD = 0, RS_HLL = 1, RS_LLF = 2, RS_HLLD_CENSUS = 3 };
enum { BC_PERIODIC = 0, BC_OUTFLOW = 1, BC_REFLECT = 2 };

struct F9 {
  float v[9];
  __device__ __forceinline__ float& operator[](int i) { return v[i]; }
  __device__ __forceinline__ const float& operator[](int i) const { return v[i]; }
};

struct Phys {
  float gamma, smallr, pfl, llf_dmin, llf_pmin;
  // HLLD single-star degeneracy test |denK| < max(1e-12, dtol_rel * bn^2); 0 is the reference's
  // absolute test |denK| < 1e-12 (glm_physics.jl:257)
  float dtol_rel;
};

// Per-thread counts of the HLLD degeneracy census (RS_HLLD_CENSUS): solves, single-star sides
// with |denK| < 1e-12 (the reference's degenerate branch) and sides with 1e-12 <= |denK| <
// 1e-5 bn^2 (sent to the degenerate branch by the relative test only).
struct HlldCensus {
  unsigned solves, ref_sides, rel_sides;
};

// ---- packed FP32 pairs (sm_100 FFMA2 / FMUL2 / FADD2): two independent evaluations of the
// same expression in one instruction, each lane rounded exactly as the scalar operation ----
__device__ __forceinline__ float2 p2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 pb(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
struct P9 {
  float2 v[9];
  __device__ __forceinline__ float2& operator[](int i) { return v[i]; }
  __device__ __forceinline__ const float2& operator[](int i) const { return v[i]; }
};

// Products that meet an add are written as explicit fused multiply-adds or explicitly rounded
// products here and in the solvers below: left to the compiler, which of them fuse depends on the
// instantiation, and the step's instantiations are to give the same bits.

// conserved -> primitive with density and pressure floors (glm_physics.jl:11-18)
__device__ __forceinline__ F9 cons2prim(const F9& c, float g, float smallr, float pfl) {
  const float rho = fmaxf(c[0], smallr);
  const float ir = 1.0f / rho;
  const float m2 = fmaf(c[3], c[3], fmaf(c[2], c[2], c[1] * c[1]));
  const float b2 = fmaf(c[7], c[7], fmaf(c[6], c[6], c[5] * c[5]));
  const float ei = fmaf(-0.5f, b2, fmaf(-0.5f * m2, ir, c[4]));
  const float p = fmaxf((g - 1.0f) * ei, pfl);
  return F9{{rho, __fmul_rn(c[1], ir), __fmul_rn(c[2], ir), __fmul_rn(c[3], ir), p, c[5], c[6], c[7], c[8]}};
}

// primitive -> conserved (glm_physics.jl:19-23)
__device__ __forceinline__ F9 prim2cons(const F9& q, float g) {
  const float rho = q[0], vx = q[1], vy = q[2], vz = q[3], bx = q[5], by = q[6], bz = q[7];
  const float v2 = fmaf(vz, vz, fmaf(vy, vy, vx * vx)), b2 = fmaf(bz, bz, fmaf(by, by, bx * bx));
  const float E = fmaf(0.5f, b2, fmaf(0.5f * rho, v2, q[4] * (1.0f / (g - 1.0f))));
  return F9{{rho, __fmul_rn(rho, vx), __fmul_rn(rho, vy), __fmul_rn(rho, vz), E, bx, by, bz, q[8]}};
}

// fast magnetosonic speed along the normal with normal field bn (glm_physics.jl:24-27)
__device__ __forceinline__ float fast_speed(const F9& q, float g, float bn) {
  float rho = q[0];
  float c2 = g * q[4] / rho;
  float b2 = (q[5] * q[5] + q[6] * q[6] + q[7] * q[7]) / rho;
  float d2 = 0.5f * (b2 + c2);
  return sqrtf(d2 + sqrtf(fmaxf(d2 * d2 - c2 * bn * bn / rho, 0.0f)));
}

// Axis permutations: D = 0, 1, 2 for x, y, z. rot_to maps the global (v, B) ordering to the
// frame whose first component is the D-normal; rot_back maps a flux back (glm_physics.jl:36-45).
template <int D> __device__ __forceinline__ F9 rot_to(const F9& q) {
  if (D == 0) return q;
  if (D == 1) return F9{{q[0], q[2], q[3], q[1], q[4], q[6], q[7], q[5], q[8]}};
  return F9{{q[0], q[3], q[1], q[2], q[4], q[7], q[5], q[6], q[8]}};
}
template <int D> __device__ __forceinline__ F9 rot_back(const F9& f) {
  if (D == 0) return f;
  if (D == 1) return F9{{f[0], f[3], f[1], f[2], f[4], f[7], f[5], f[6], f[8]}};
  return F9{{f[0], f[2], f[3], f[1], f[4], f[6], f[7], f[5], f[8]}};
}

// x-normal ideal-MHD flux; F[Bn] = F[psi] = 0 (glm_physics.jl:28-34)
__device__ __forceinline__ F9 phys_flux_x(const F9& q, float g) {
  float rho = q[0], vx = q[1], vy = q[2], vz = q[3], p = q[4], bx = q[5], by = q[6], bz = q[7];
  float b2 = bx * bx + by * by + bz * bz;
  float ptot = p + 0.5f * b2;
  float E = p / (g - 1.0f) + 0.5f * rho * (vx * vx + vy * vy + vz * vz) + 0.5f * b2;
  float vb = vx * bx + vy * by + vz * bz;
  return F9{{rho * vx, rho * vx * vx + ptot - bx * bx, rho * vx * vy - bx * by, rho * vx * vz - bx * bz,
             (E + ptot) * vx - bx * vb, 0.0f, vx * by - vy * bx, vx * bz - vz * bx, 0.0f}};
}
template <int D> __device__ __forceinline__ F9 dir_flux(const F9& q, float g) {
  return rot_back<D>(phys_flux_x(rot_to<D>(q), g));
}

// minmod limiter (glm_physics.jl:54-59); MonCen is half_moncen below
__device__ __forceinline__ float minmod(float dl, float dr) {
  float sgn = dl >= 0.0f ? 1.0f : -1.0f;
  return dl * dr <= 0.0f ? 0.0f : sgn * fminf(fabsf(dl), fabsf(dr));
}
// Per-axis face offsets about the cell mean. For the PLM limiters dL = -dR, so only dR is
// produced and dL is implied (glm_physics.jl:212-219); PPM produces both (:220-223).
template <int RECON> struct Offsets {
  F9 dR;
  __device__ __forceinline__ float l(int i) const { return -dR[i]; }
};
template <> struct Offsets<RECON_PPM> {
  F9 dL, dR;
  __device__ __forceinline__ float l(int i) const { return dL[i]; }
};

// Offsets kept or replaced by exact zeros (keep = false: the piecewise-constant states of a
// first-order fallback). A select, not a product: an Inf or NaN offset of a bad state still
// gives a zero offset, as the reference's assignment of zeros does (integrator_cube.jl:168-171).
template <int RECON> __device__ __forceinline__ void keep_offsets(Offsets<RECON>& o, bool keep) {
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    o.dR[i] = keep ? o.dR[i] : 0.0f;
    if constexpr (RECON == RECON_PPM) o.dL[i] = keep ? o.dL[i] : 0.0f;
  }
}

// min(|a|, |b|) carrying the sign sign(a) XOR sign(b) (PTX min.xorsign.abs, one instruction).
__device__ __forceinline__ float min_xorsign_abs(float a, float b) {
  float r;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// The same, NaN if either is (the form above returns the other operand's magnitude).
__device__ __forceinline__ float min_xorsign_abs_nan(float a, float b) {
  float r;
  asm("min.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// max(a, b), NaN if either is (fmaxf returns the other operand).
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// Half the MonCen slope, 0.5*moncen(dl, dr) of glm_physics.jl:47-53, from dl, dr and
// q = (dl+dr)/4. With the scalings by powers of two folded, the reference's value is
// 0.5*sgn*min(2*min|dl|,|dr|, |(dl+dr)/2|) = sgn(q)*min(min(|dl|,|dr|), |q|) when dl*dr > 0 and
// 0 otherwise. t = min.xorsign.abs(dl, dr) has magnitude min(|dl|,|dr|) and is positive exactly
// when dl and dr have the same sign, so max(t, 0) is zero wherever the reference returns zero,
// and min.xorsign.abs(max(t, 0), q) carries sgn(q): three instructions, the same value (up to
// the sign of a zero result), every step exact.
__device__ __forceinline__ float half_moncen(float dl, float dr, float q) {
  return min_xorsign_abs(fmaxf(min_xorsign_abs(dl, dr), 0.0f), q);
}
// Local CW84 PPM face offsets, monotonised (glm_physics.jl:188-200), from the differences to the
// lower and upper neighbour. Before the limiter the offsets are L = c - s, R = c + s with
// s = (dl + dr)/4, c = (dr - dl)/12. The reference's cases are: L and R on the same side (an
// extremum): both zero; (q - mid)(R - L) > (R - L)^2/6, that is |L| > 2|R|: L = -2R; likewise
// R = -2L; otherwise unchanged. That is |L| and |R| cut at twice the smaller of the two, or at
// zero where their signs agree: z = max(-min.xorsign(L, R), 0) is that smaller magnitude or
// zero. No branch and no division (the reference's form diverges within a warp and divides
// twice a field: the 192^3 PPM/HLLD step took 1.39 ms with it, 0.73 with this form and the
// solver below). A NaN difference gives NaN offsets, as the reference's form does.
__device__ __forceinline__ void ppm_offsets(float dl, float dr, float& oL, float& oR) {
  const float s = 0.25f * (dl + dr), c = dr - dl;
  const float L = fmaf(1.0f / 12.0f, c, -s), R = fmaf(1.0f / 12.0f, c, s);
  const float z2 = 2.0f * max_nan(-min_xorsign_abs_nan(L, R), 0.0f);
  oL = min_xorsign_abs_nan(L, z2);
  oR = min_xorsign_abs_nan(R, z2);
}

template <int RECON>
__device__ __forceinline__ Offsets<RECON> recon(const F9& mm, const F9& m0, const F9& mp) {
  Offsets<RECON> o;
  if constexpr (RECON == RECON_PLM) {
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float dl = m0[i] - mm[i], dr = mp[i] - m0[i];
      o.dR[i] = half_moncen(dl, dr, 0.25f * (dl + dr));
    }
  } else if constexpr (RECON == RECON_PLM_MINMOD) {
#pragma unroll
    for (int i = 0; i < 9; ++i) o.dR[i] = 0.5f * minmod(m0[i] - mm[i], mp[i] - m0[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      ppm_offsets(m0[i] - mm[i], mp[i] - m0[i], o.dL[i], o.dR[i]);
    }
  }
  return o;
}
template <int RECON> __device__ __forceinline__ F9 face_lo(const F9& mh, const Offsets<RECON>& o) {
  F9 r;
#pragma unroll
  for (int i = 0; i < 9; ++i) r[i] = mh[i] + o.l(i);
  return r;
}
template <int RECON> __device__ __forceinline__ F9 face_hi(const F9& mh, const Offsets<RECON>& o) {
  F9 r;
#pragma unroll
  for (int i = 0; i < 9; ++i) r[i] = mh[i] + o.dR[i];
  return r;
}

// One term of the Hancock predictor (glm_physics.jl:225-231): the x-normal fluxes (D-normal after
// the axis permutation) of the two face states m0 + dR (lane x) and m0 + dL (lane y), added to the
// packed sums `acc` (global component order; FIRST: the sums start here). The sums enter the
// multiply-adds that form each flux, so adding a direction costs no instruction beyond its flux. (It
// rounds at the size of the fluxes, not of their differences. Against extended precision the predicted
// state's error is 1.00-1.02 of that of differences taken per direction in turbulence at CFL 0.2-0.4
// and at most 1.05 in a Mach 10 drift, where the rounding of the state itself dominates; a velocity
// component at rest beside such a drift has 1.6 of an error of 5e-10.) A packed
// subtraction is avoided throughout: negating both lanes of an operand costs two instructions
// beside the packed one (measured 4 issue cycles against 2), so the normal field is negated once.
template <int D, int RECON, bool FIRST>
__device__ __forceinline__ void hancock_term(P9& acc, const F9& m0, const Offsets<RECON>& o, float g) {
  // global -> D-normal component order, as rot_to<D>
  constexpr int perm[3][9] = {{0, 1, 2, 3, 4, 5, 6, 7, 8}, {0, 2, 3, 1, 4, 6, 7, 5, 8}, {0, 3, 1, 2, 4, 7, 5, 6, 8}};
  P9 q;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int j = perm[D][i];
    q[i] = make_float2(m0[j] + o.dR[j], m0[j] + o.l(j));
  }
  const float2 rho = q[0], vx = q[1], vy = q[2], vz = q[3], p = q[4], bx = q[5], by = q[6], bz = q[7];
  const float2 half = pb(0.5f);
  const float2 nbx = mul2(bx, pb(-1.0f));
  const float2 b2 = fma2(bz, bz, fma2(by, by, mul2(bx, bx)));
  const float2 v2 = fma2(vz, vz, fma2(vy, vy, mul2(vx, vx)));
  const float2 vb = fma2(vz, bz, fma2(vy, by, mul2(vx, bx)));
  const float2 h = fma2(mul2(half, rho), v2, fma2(p, pb(1.0f + 1.0f / (g - 1.0f)), b2));  // E + ptot
  const float2 m = mul2(rho, vx);
  // a * b added to component c
  auto mad = [&](int c, float2 a, float2 b) { acc[c] = FIRST ? mul2(a, b) : fma2(a, b, acc[c]); };
  constexpr int M = perm[D][1], V = perm[D][2], W = perm[D][3], BV = perm[D][6], BW = perm[D][7];
  const float2 ptm = fma2(m, vx, fma2(half, b2, p));
  if (FIRST) {
    acc[0] = m;
    acc[M] = fma2(nbx, bx, ptm);
  } else {
    acc[0] = add2(acc[0], m);
    acc[M] = add2(acc[M], fma2(nbx, bx, ptm));
  }
  mad(V, m, vy);
  acc[V] = fma2(nbx, by, acc[V]);
  mad(W, m, vz);
  acc[W] = fma2(nbx, bz, acc[W]);
  mad(4, h, vx);
  acc[4] = fma2(nbx, vb, acc[4]);
  if (D == 0) {  // By and Bz start with x, Bx with y
    acc[BV] = mul2(vx, by);
    acc[BW] = mul2(vx, bz);
  } else if (D == 1) {  // normal By: transverse (Bz, Bx)
    acc[BV] = fma2(vx, by, acc[BV]);
    acc[BW] = mul2(vx, bz);
  } else {
    acc[BV] = fma2(vx, by, acc[BV]);
    acc[BW] = fma2(vx, bz, acc[BW]);
  }
  acc[BV] = fma2(nbx, vy, acc[BV]);
  acc[BW] = fma2(nbx, vz, acc[BW]);
}

// ---- Riemann solvers in the face-normal frame (x-normal after rot_to) -----------------
// LLF / Rusanov (glm_physics.jl:239-244)
__device__ __forceinline__ F9 llf_x(const F9& L, const F9& R, float g, float ch, float fbn, float fpsi) {
  F9 fL = phys_flux_x(L, g), fR = phys_flux_x(R, g), uL = prim2cons(L, g), uR = prim2cons(R, g);
  float smax = fmaxf(fmaxf(fabsf(L[1]) + fast_speed(L, g, L[5]), fabsf(R[1]) + fast_speed(R, g, R[5])), ch);
  F9 f;
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i] = 0.5f * (fL[i] + fR[i]) - 0.5f * smax * (uR[i] - uL[i]);
  f[5] = fbn;
  f[8] = fpsi;
  return f;
}
// HLL (glm_physics.jl:245-252)
__device__ __forceinline__ F9 hll_x(const F9& L, const F9& R, float g, float bn, float fbn, float fpsi) {
  float cfL = fast_speed(L, g, bn), cfR = fast_speed(R, g, bn);
  float SL = fminf(fminf(L[1] - cfL, R[1] - cfR), 0.0f);
  float SR = fmaxf(fmaxf(L[1] + cfL, R[1] + cfR), 0.0f);
  F9 fL = phys_flux_x(L, g), fR = phys_flux_x(R, g), uL = prim2cons(L, g), uR = prim2cons(R, g);
  float invd = 1.0f / (SR - SL);
  F9 f;
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i] = (SR * fL[i] - SL * fR[i] + SL * SR * (uR[i] - uL[i])) * invd;
  f[5] = fbn;
  f[8] = fpsi;
  return f;
}
// HLLD, Miyoshi & Kusano 2005 (glm_physics.jl:255-307). The parts that are the same algebra on the
// two states run as packed pairs (lane x = L, lane y = R).
//
// The reference forms the single-star states of both sides, v* = v - bn b x and b* = (1 + d(S-u) x) b
// with x = (S_M - u) / denK, denK = d(S-u)(S-S_M) - bn^2, the double-star state from them, and the
// flux F_K + S_K (U*_K - U_K) (outer region) or F_K + S*_K U** - (S*_K - S_K) U*_K - S_K U_K (inner
// region) of the side K that the contact leans to. Here the same flux is reduced with
//   S_K - S*_K = denK / (|d(S-u)| + sqrt(d*) |bn|),   D = |S - S_M| + |S* - S_M|,
// so that only what the selected region needs is formed and, but for w in the energy, the inner
// region has no 1/denK:
//   b' = b (1 + s r), r = (S_M - u) / D (s = -1 left, +1 right) takes the place of b* in the
//   double-star averages (v is unchanged there), and with m = d* S_M, t = 0 (outer) or S*_K (inner),
//   y = S_K d* x (outer) or s r (inner):
//   F(mass) = m, F(normal) = m S_M + ptot* - bn^2, F(v) = m v + d* t (v** - v) - bn b (1 + y),
//   F(b) = b (u + (S_K - S_M) y) + t (b** - b) - bn v,
//   F(E) = S_M H / (S_K - S_M) + c w - s sqrt(d*) sgn(bn) t w**,
// ptot* = ptot + d(S-u)(S_M - u), H = (S-u) E - ptot u + bn v.B + S_K ptot*, w = v*.B*, w** = v**.B**,
// c = -S_K bn / (S_K - S_M) (outer) or sgn(bn) S_M denK / (sqrt(d*) D (S_K - S_M)) (inner). Near
// R-degenerate faces, where denK is the rounding residue of two terms of size bn^2, the mass,
// momentum and induction fluxes of the inner region keep FP32 accuracy; the energy's w is quadratic
// in x, so that b_t^2 / denK is left in it.
// Where |u| exceeds the fast speed, S_K is 0 and the flux is F_K. d* S_M and S_M / (S_K - S_M) are that
// only up to the rounding of S_M, which mixes both sides, so for |S_K| < |u|/2 the mass flux is
// d u + S_K (d* - d) and the energy's first term S_K H / (S_K - S_M) - H: exactly F_K at S_K = 0.
// Against extended precision the rounding error of every component is then at most that of the
// reference's form in FP32: 0.3-0.9 of it in the subsonic fan, equal on super-fast faces (with d* S_M
// and S_M / (S_K - S_M) there 2.0 of it in the mass and 1.8 in the normal momentum). It is larger only
// where a face holds a head-on collision of more than Mach 10 (normal momentum, 1.1) or an
// expansion of that strength (induction, 1.1-1.7; the other components 0.02-0.6).
// The step is bounded by instruction issue: with this form, the predictor's sums in multiply-adds
// and the vectorised tile edges the 256^3 GLM step executes 59.7 instead of 71.8 warp
// instructions per cell (1.77 -> 1.55 ms, 1 % of it spent on the side's own flux; constrained
// transport 2.29 -> 2.05 ms).
__device__ __forceinline__ F9 hlld_x(const F9& L, const F9& R, float g, float bn, float fbn, float fpsi,
                                     float dtol_rel, HlldCensus* cen = nullptr) {
  const float2 d = p2(L[0], R[0]), u = p2(L[1], R[1]), v = p2(L[2], R[2]), w = p2(L[3], R[3]);
  const float2 p = p2(L[4], R[4]), by = p2(L[6], R[6]), bz = p2(L[7], R[7]);
  const float2 half = pb(0.5f);
  const float bn2 = bn * bn;
  const float2 nbn2 = pb(-bn2);
  const float2 b2 = fma2(bz, bz, fma2(by, by, pb(bn2)));
  const float2 pt = fma2(half, b2, p);
  // fast speeds (glm_physics.jl:24-27) with the normal field bn
  const float2 id = p2(1.0f / L[0], 1.0f / R[0]);
  const float2 c2 = mul2(mul2(pb(g), p), id);
  const float2 d2 = mul2(half, fma2(b2, id, c2));
  const float2 disc = fma2(d2, d2, mul2(mul2(c2, nbn2), id));
  const float2 in = add2(d2, p2(sqrtf(fmaxf(disc.x, 0.0f)), sqrtf(fmaxf(disc.y, 0.0f))));
  const float cf = sqrtf(fmaxf(in.x, in.y));
  const float SL = fminf(fminf(u.x, u.y) - cf, 0.0f);
  const float SR = fmaxf(fmaxf(u.x, u.y) + cf, 0.0f);
  const float2 S = p2(SL, SR);
  const float2 dSu = mul2(p2(SL - u.x, SR - u.y), d);  // d (S - u) per side
  const float iden = 1.0f / (dSu.y - dSu.x);
  const float SM = __fmul_rn(fmaf(dSu.y, u.y, pt.x) - fmaf(dSu.x, u.x, pt.y), iden);
  const float2 SSM = add2(S, pb(-SM));  // S - SM per side
  const float2 iSSM = p2(1.0f / SSM.x, 1.0f / SSM.y);
  const float2 ds = mul2(dSu, iSSM);
  const float dLs = fmaxf(ds.x, 1e-12f), dRs = fmaxf(ds.y, 1e-12f);
  const float irL = rsqrtf(dLs), irR = rsqrtf(dRs);
  const float sqL = __fmul_rn(dLs, irL), sqR = __fmul_rn(dRs, irR);
  const float abn = fabsf(bn);
  const float SLs = fmaf(-abn, irL, SM), SRs = fmaf(abn, irR, SM);
  const float iDL = 1.0f / fmaf(abn, irL, fabsf(SSM.x)), iDR = 1.0f / fmaf(abn, irR, fabsf(SSM.y));
  float2 r = p2((u.x - SM) * iDL, (SM - u.y) * iDR);  // s r per side
  // Degenerate star state (the fast and Alfven speeds coincide). The reference tests
  // |denK| < 1e-12 (dtol_rel = 0), which is below the FP32 rounding of denK = d(S-u)(S-SM) - bn^2
  // (a difference of two terms of size bn^2). The relative mode (dtol_rel = 1e-5) sends faces with
  // |denK| within 1e-5 bn^2 of zero to the degenerate branch, whose transverse state is the
  // unmodified one (v* = v, b* = b: x = r = 0).
  const float2 denK = fma2(dSu, SSM, nbn2);
  const float dtol = fmaxf(1e-12f, dtol_rel * bn2);
  const bool degL = fabsf(denK.x) < dtol, degR = fabsf(denK.y) < dtol;
  if (cen != nullptr) {
    const float t5 = 1e-5f * bn2, aL = fabsf(denK.x), aR = fabsf(denK.y);
    cen->solves += 1;
    cen->ref_sides += (aL < 1e-12f ? 1u : 0u) + (aR < 1e-12f ? 1u : 0u);
    cen->rel_sides += (aL >= 1e-12f && aL < t5 ? 1u : 0u) + (aR >= 1e-12f && aR < t5 ? 1u : 0u);
  }
  if (degL) r.x = 0.0f;
  if (degR) r.y = 0.0f;
  // double-star transverse state, with the density-root weights wa, wb = 1 - wa
  const float2 bye = fma2(by, r, by), bze = fma2(bz, r, bz);
  const float inv = 1.0f / (sqL + sqR);
  const float wb = sqR * inv, wa = sqL * inv;
  const float c = copysignf(inv, bn), e = sqL * sqR * c;
  const float dv = v.y - v.x, dw = w.y - w.x, dby = bye.y - bye.x, dbz = bze.y - bze.x;
  const float vyss = fmaf(c, dby, fmaf(wb, dv, v.x)), vzss = fmaf(c, dbz, fmaf(wb, dw, w.x));
  const float byss = fmaf(e, dv, fmaf(wa, dby, bye.x)), bzss = fmaf(e, dw, fmaf(wa, dbz, bze.x));
  const float SMbn = SM * bn;
  const float wss = fmaf(vzss, bzss, fmaf(vyss, byss, SMbn));
  // the side the contact leans to
  const bool left = SM >= 0.0f;
  const float dK = left ? d.x : d.y, uK = left ? u.x : u.y, vK = left ? v.x : v.y, wK = left ? w.x : w.y;
  const float pK = left ? p.x : p.y, byK = left ? by.x : by.y, bzK = left ? bz.x : bz.y, SK = left ? SL : SR;
  const float iSSMK = left ? iSSM.x : iSSM.y, dKs = left ? dLs : dRs, irK = left ? irL : irR;
  const float iDK = left ? iDL : iDR, rK = left ? r.x : r.y, SKs = left ? SLs : SRs;
  const float denKK = left ? denK.x : denK.y;
  const bool degK = left ? degL : degR;
  const bool outer = left ? (SLs >= 0.0f) : (SRs < 0.0f);
  const float SuK = SK - uK, dSuK = dK * SuK, SSMK = SK - SM;
  const float bt2 = fmaf(bzK, bzK, byK * byK), vbt = fmaf(wK, bzK, vK * byK);
  const float b2K = fmaf(bn, bn, bt2);
  const float EK = fmaf(0.5f * dK, fmaf(wK, wK, fmaf(vK, vK, uK * uK)), fmaf(pK, 1.0f / (g - 1.0f), 0.5f * b2K));
  const float du = SM - uK, dsSK = dKs * SK;
  const float ptK = fmaf(0.5f, b2K, pK), pts = fmaf(dSuK, du, ptK);
  const float H = fmaf(SK, pts, fmaf(bn, fmaf(uK, bn, vbt), fmaf(SuK, EK, -ptK * uK)));  // G + S_K ptot*
  const float x = degK ? 0.0f : du * (1.0f / denKK);
  const float ws = fmaf(fmaf(dSuK, x, 1.0f), fmaf(-bn * x, bt2, vbt), SMbn);
  const float sgn = copysignf(1.0f, bn);
  const float y = outer ? dsSK * x : rK;
  const float cw = outer ? -SK * bn : sgn * SM * (denKK * (irK * iDK));
  const float by1 = fmaf(bn, y, bn), bu = fmaf(SSMK, y, uK);
  // The side's own flux with a correction of the order of S_K, where that is the smaller part.
  const bool own = fabsf(SK) < 0.5f * fabsf(uK);
  F9 f;
  f[0] = own ? fmaf(SK, dKs - dK, __fmul_rn(dK, uK)) : __fmul_rn(dKs, SM);
  f[1] = fmaf(dSuK, du, fmaf(f[0], SM, fmaf(-bn, bn, ptK)));
  f[2] = fmaf(f[0], vK, -by1 * byK);
  f[3] = fmaf(f[0], wK, -by1 * bzK);
  f[4] = fmaf(iSSMK, fmaf(own ? SK : SM, H, cw * ws), own ? -H : 0.0f);
  f[5] = fbn;
  f[6] = fmaf(bu, byK, -bn * vK);
  f[7] = fmaf(bu, bzK, -bn * wK);
  // The double-star terms enter in the inner region only, not as products with a zero: where the fast
  // speed is below the rounding of u, S_M can equal the other side's S, whose single-star density and
  // with it the double-star state is then not finite, while the flux of side K is.
  if (!outer) {
    const float t = SKs, m = dKs * t;
    f[2] = fmaf(m, vyss - vK, f[2]);
    f[3] = fmaf(m, vzss - wK, f[3]);
    f[4] = fmaf(-sgn * (left ? -sqL : sqR) * t, wss, f[4]);
    f[6] = fmaf(t, byss - byK, f[6]);
    f[7] = fmaf(t, bzss - bzK, f[7]);
  }
  f[8] = fpsi;
  return f;
}

// GLM Riemann problem on a D-normal face (glm_physics.jl:317-329): floors, Dedner pair,
// the selected solver (HLLD with the LLF fallback at low density/pressure), rotate back.
// ich = 1/ch, formed once per launch: the cleaned normal field every solve starts from then
// waits on a multiply, not on a division.
// force_llf: LLF on this face whatever the solver (the masked fallback of the cube kernel,
// integrator_cube.jl:68-83); false except in the radiation-coupled step.
template <int D, int RSOL>
__device__ __forceinline__ F9 riemann_glm(const F9& Lq, const F9& Rq, float ch, float ich, const Phys& P,
                                          HlldCensus* cen = nullptr, bool force_llf = false) {
  F9 L = rot_to<D>(Lq), R = rot_to<D>(Rq);
  L[0] = fmaxf(L[0], P.smallr); L[4] = fmaxf(L[4], P.pfl);
  R[0] = fmaxf(R[0], P.smallr); R[4] = fmaxf(R[4], P.pfl);
  float bns = fmaf(-0.5f * (R[8] - L[8]), ich, 0.5f * (L[5] + R[5]));
  float psis = fmaf(-0.5f * ch, R[5] - L[5], 0.5f * (L[8] + R[8]));
  float fbn = psis, fpsi = __fmul_rn(ch * ch, bns);
  L[5] = bns; R[5] = bns;
  F9 f;
  if constexpr (RSOL == RS_LLF) {
    f = llf_x(L, R, P.gamma, ch, fbn, fpsi);
  } else if constexpr (RSOL == RS_HLL) {
    if (force_llf) f = llf_x(L, R, P.gamma, ch, fbn, fpsi);
    else f = hll_x(L, R, P.gamma, bns, fbn, fpsi);
  } else {
    bool uself = force_llf || (P.llf_dmin > 0.0f && fminf(L[0], R[0]) < P.llf_dmin) ||
                 (P.llf_pmin > 0.0f && fminf(L[4], R[4]) < P.llf_pmin);
    if (uself) f = llf_x(L, R, P.gamma, ch, fbn, fpsi);
    else f = hlld_x(L, R, P.gamma, bns, fbn, fpsi, P.dtol_rel, cen);
  }
  return rot_back<D>(f);
}

// Constrained-transport Riemann problem (glm_physics.jl:336-348): the caller has put the
// staggered face value into both states' normal-B slot; no psi, ch = 0 in the LLF speed.
template <int D, int RSOL>
__device__ __forceinline__ F9 riemann_ct(const F9& Lq, const F9& Rq, const Phys& P, HlldCensus* cen = nullptr,
                                         bool force_llf = false) {
  F9 L = rot_to<D>(Lq), R = rot_to<D>(Rq);
  L[0] = fmaxf(L[0], P.smallr); L[4] = fmaxf(L[4], P.pfl); L[8] = 0.0f;
  R[0] = fmaxf(R[0], P.smallr); R[4] = fmaxf(R[4], P.pfl); R[5] = L[5]; R[8] = 0.0f;
  float bns = L[5];
  F9 f;
  if constexpr (RSOL == RS_LLF) {
    f = llf_x(L, R, P.gamma, 0.0f, 0.0f, 0.0f);
  } else if constexpr (RSOL == RS_HLL) {
    if (force_llf) f = llf_x(L, R, P.gamma, 0.0f, 0.0f, 0.0f);
    else f = hll_x(L, R, P.gamma, bns, 0.0f, 0.0f);
  } else {
    bool uself = force_llf || (P.llf_dmin > 0.0f && fminf(L[0], R[0]) < P.llf_dmin) ||
                 (P.llf_pmin > 0.0f && fminf(L[4], R[4]) < P.llf_pmin);
    if (uself) f = llf_x(L, R, P.gamma, 0.0f, 0.0f, 0.0f);
    else f = hlld_x(L, R, P.gamma, bns, 0.0f, 0.0f, P.dtol_rel, cen);
  }
  return rot_back<D>(f);
}

// `cen` is read only by the census instantiation (RS_HLLD_CENSUS); pass it for the faces to be
// counted, nullptr otherwise.
template <int D, int RSOL, bool CT>
__device__ __forceinline__ F9 riemann(const F9& L, const F9& R, float ch, float ich, const Phys& P,
                                      HlldCensus* cen = nullptr, bool force_llf = false) {
  if constexpr (RSOL != RS_HLLD_CENSUS) cen = nullptr;
  if constexpr (CT) return riemann_ct<D, RSOL>(L, R, P, cen, force_llf);
  else return riemann_glm<D, RSOL>(L, R, ch, ich, P, cen, force_llf);
}

// max over axes of |v_d| + c_f(B_d) of a conserved state (timestep.jl:4-14)
__device__ __forceinline__ float cell_wavespeed(const F9& u, const Phys& P) {
  F9 q = cons2prim(u, P.gamma, P.smallr, P.pfl);
  float sx = fabsf(q[1]) + fast_speed(q, P.gamma, q[5]);
  float sy = fabsf(q[2]) + fast_speed(q, P.gamma, q[6]);
  float sz = fabsf(q[3]) + fast_speed(q, P.gamma, q[7]);
  return fmaxf(sx, fmaxf(sy, sz));
}

// Kahan-compensated accumulation with a persistent remainder (glm_physics.jl:349-359).
// The fast-math build must not reassociate it, so the rounding steps are explicit.
__device__ __forceinline__ float comp_add(float x, float dx, float& r) {
  float inc = __fadd_rn(dx, r);
  float upd = __fadd_rn(x, inc);
  r = __fsub_rn(inc, __fsub_rn(upd, x));
  return upd;
}

// ---- linear (Compton) drag toward a target velocity, glm_physics.jl:63-172 ------------------
// Coefficients of one step with impulse q = Gamma*dt (computed on the host in FP32 with the
// reference's formulas): the face prediction uses the half-step pair (exp(-q/2), phi1(q/2)),
// the cell corrector the full-step pair and the integrated-work coefficients A, C, D.
struct DragCoef {
  float v0[3];       // target velocity
  float fdecay, fphi1;
  float decay, phi1, A, C, D;
};

// Drag-propagated Hancock prediction (glm_physics.jl:71-84 with the face offset folded):
// the face velocity v0 + fd*((m0+d) - v0) + fp*((mh+d) - (m0+d)) equals mh' + fd*d with
// mh' = v0 + fd*(m0 - v0) + fp*(mh - m0), so the cell's predicted velocity is replaced by mh'
// and its velocity offsets are scaled by fd. Density, pressure, B and psi keep their
// hyperbolic midpoint values.
template <int RECON>
__device__ __forceinline__ void drag_predict_cell(F9& mh, const F9& m0, Offsets<RECON>& ox, Offsets<RECON>& oy,
                                                  Offsets<RECON>& oz, const DragCoef& k) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float v0 = k.v0[c];
    mh[1 + c] = v0 + k.fdecay * (m0[1 + c] - v0) + k.fphi1 * (mh[1 + c] - m0[1 + c]);
    ox.dR[1 + c] *= k.fdecay;
    oy.dR[1 + c] *= k.fdecay;
    oz.dR[1 + c] *= k.fdecay;
    if constexpr (RECON == RECON_PPM) {
      ox.dL[1 + c] *= k.fdecay;
      oy.dL[1 + c] *= k.fdecay;
      oz.dL[1 + c] *= k.fdecay;
    }
  }
}

// Cell corrector (glm_physics.jl:128-172): exact momentum response to the trial velocity
// increment and the analytically integrated drag work removed from E, with the density
// floored at smallr and E floored at the new kinetic + magnetic energy + 1e-30. With `rE`
// the work is removed through E's Kahan remainder, which is cleared when the floor applies
// (drag_correct_conserved_compensated!, glm_physics.jl:374-400 with
// _compensated_floor_update!, :361-372).
__device__ __forceinline__ void drag_correct_cell(const F9& u0, F9& t, const DragCoef& k, float smallr,
                                                  float* rE = nullptr) {
  const float rn = fmaxf(t[0], smallr), ro = fmaxf(u0[0], smallr);
  float w[3], dv[3], vn[3], iw[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float vo = u0[1 + c] / ro, vt = t[1 + c] / rn;
    dv[c] = vt - vo;
    w[c] = vo - k.v0[c];
    vn[c] = k.v0[c] + k.decay * w[c] + k.phi1 * dv[c];
    iw[c] = (1.0f - k.decay) * w[c] + (1.0f - k.phi1) * dv[c];
  }
  const float w2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
  const float wdv = w[0] * dv[0] + w[1] * dv[1] + w[2] * dv[2];
  const float dv2 = dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2];
  const float qwork =
      rn * (k.A * w2 + k.C * wdv + k.D * dv2 + k.v0[0] * iw[0] + k.v0[1] * iw[1] + k.v0[2] * iw[2]);
  const float nm0 = rn * vn[0], nm1 = rn * vn[1], nm2 = rn * vn[2];
  const float ek = 0.5f * (nm0 * nm0 + nm1 * nm1 + nm2 * nm2) / rn;
  const float eb = 0.5f * (t[5] * t[5] + t[6] * t[6] + t[7] * t[7]);
  t[0] = rn;
  t[1] = nm0;
  t[2] = nm1;
  t[3] = nm2;
  const float emin = ek + eb + 1e-30f;
  if (rE == nullptr) {
    t[4] = fmaxf(t[4] - qwork, emin);
  } else {
    float e = comp_add(t[4], -qwork, *rE);
    if (e < emin) {
      *rE = 0.0f;
      e = emin;
    }
    t[4] = e;
  }
}

// Admissibility of a trial conserved state (integrator_cube.jl:108-124): finite, density
// at least max(smallr, llf_dmin) and internal energy at least pfl/(gamma-1).
__device__ __forceinline__ bool inadmissible_cell(const F9& r, const Phys& P) {
  const float ir = 1.0f / fmaxf(r[0], P.smallr);
  const float ek = 0.5f * (r[1] * r[1] + r[2] * r[2] + r[3] * r[3]) * ir;
  const float eb = 0.5f * (r[5] * r[5] + r[6] * r[6] + r[7] * r[7]);
  const float eint = r[4] - ek - eb;
  bool finite = isfinite(eint);
#pragma unroll
  for (int v = 0; v < 9; ++v) finite = finite && isfinite(r[v]);
  return !finite || r[0] < fmaxf(P.smallr, P.llf_dmin) || eint < P.pfl / (P.gamma - 1.0f);
}


// Periodic image of index i. On boxes at least a tile wide callers are at most a halo outside, and a few
// compares do what an integer remainder (some 30 instructions) would; the lanes of a partial tile
// on a narrower box go round once per box width.
__device__ __forceinline__ int wrap_index(int i, int n) {
  while (i < 0) i += n;
  while (i >= n) i -= n;
  return i;
}

// BC index map for a logical cell index (boundary.jl:161-175, 0-based): returns the source
// index; *flip = -1 where a reflecting wall mirrors the normal vector components.
__device__ __forceinline__ int bc_index(int i, int n, int code, float* flip) {
  *flip = 1.0f;
  if (code == BC_PERIODIC) return wrap_index(i, n);
  if (code == BC_OUTFLOW) return i < 0 ? 0 : (i >= n ? n - 1 : i);
  int r = i;
  if (i < 0) { *flip = -1.0f; r = -1 - i; }
  else if (i >= n) { *flip = -1.0f; r = 2 * n - 1 - i; }
  // an axis shorter than the 2-cell stencil mirrors past its far end: clamp
  return r < 0 ? 0 : (r >= n ? n - 1 : r);
}

// Programmatic dependent launch. A kernel that begins with wait_previous() / overlap_next() may be
// launched with that attribute: its CTAs are placed while the previous kernel of the stream still
// runs and touch memory only after wait_previous(), which returns when that kernel is complete and
// its writes are visible. overlap_next() comes after the wait, so that the kernel after this one is
// not placed before the one before this one is complete. Such a kernel is resident while its inputs
// are written: it reads them by ordinary loads, never through the non-coherent path (no __ldg, no
// const __restrict__ kernel parameters), whose data must not change while the kernel is resident.
// Both do nothing in an ordinary launch.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void overlap_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace pmf
