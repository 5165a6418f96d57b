// Host form of the device fluxes for test_flux_rounding.py: PHYSICS is physics.cuh with its PTX
// lines replaced by calls of the functions below. The reference arithmetic is Miyoshi & Kusano 2005
// written out once for any precision.
#include <cmath>
#include <cstring>

struct float2 {
  float x, y;
};
static float2 make_float2(float a, float b) { return {a, b}; }
static float once(float r) { volatile float v = r; return v; }  // rounded here, never fused
static float2 __fadd2_rn(float2 a, float2 b) { return {once(a.x + b.x), once(a.y + b.y)}; }
static float2 __fmul2_rn(float2 a, float2 b) { return {once(a.x * b.x), once(a.y * b.y)}; }
static float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
static float __fmul_rn(float a, float b) { return once(a * b); }
static float __fadd_rn(float a, float b) { return once(a + b); }
static float __fsub_rn(float a, float b) { return once(a - b); }
static float rsqrtf(float x) { return 1.0f / sqrtf(x); }
static float __shfl_xor_sync(unsigned, float v, int) { return v; }
using std::isfinite;

static float host_min_xorsign(float a, float b) {
  return copysignf(fminf(fabsf(a), fabsf(b)), (std::signbit(a) != std::signbit(b)) ? -1.0f : 1.0f);
}
static float host_min_xorsign_nan(float a, float b) { return a != a || b != b ? NAN : host_min_xorsign(a, b); }
static float host_max_nan(float a, float b) { return a != a || b != b ? NAN : fmaxf(a, b); }

#include PHYSICS

template <class T> static void hlld(const float* l, const float* r, float gf, float bnf, float dtol, T* F) {
  struct Side {
    T d, u, v, w, p, by, bz, pt, E, vb, ds, vs, ws, bys, bzs, Es, vbs;
  } K[2];
  const T g = gf, bn = bnf;
  for (int s = 0; s < 2; ++s) {
    const float* q = s ? r : l;
    Side& k = K[s];
    k.d = q[0]; k.u = q[1]; k.v = q[2]; k.w = q[3]; k.p = q[4]; k.by = q[6]; k.bz = q[7];
    const T b2 = bn * bn + k.by * k.by + k.bz * k.bz;
    k.pt = k.p + b2 / 2;
    k.E = k.p / (g - 1) + k.d / 2 * (k.u * k.u + k.v * k.v + k.w * k.w) + b2 / 2;
    k.vb = k.u * bn + k.v * k.by + k.w * k.bz;
  }
  auto fast = [&](const Side& k) {
    const T c2 = g * k.p / k.d, b2 = (bn * bn + k.by * k.by + k.bz * k.bz) / k.d, d2 = (c2 + b2) / 2;
    return std::sqrt(d2 + std::sqrt(std::fmax(d2 * d2 - c2 * bn * bn / k.d, T(0))));
  };
  const T c = std::fmax(fast(K[0]), fast(K[1]));
  const T S[2] = {std::fmin(std::fmin(K[0].u, K[1].u) - c, T(0)), std::fmax(std::fmax(K[0].u, K[1].u) + c, T(0))};
  const T a0 = K[0].d * (S[0] - K[0].u), a1 = K[1].d * (S[1] - K[1].u), den = a1 - a0;
  const T SM = (a1 * K[1].u - a0 * K[0].u - K[1].pt + K[0].pt) / den;
  const T pts = (a1 * K[0].pt - a0 * K[1].pt + a0 * a1 * (K[1].u - K[0].u)) / den;
  for (int s = 0; s < 2; ++s) {
    Side& k = K[s];
    const T a = k.d * (S[s] - k.u), dk = a * (S[s] - SM) - bn * bn;
    k.ds = std::fmax(a / (S[s] - SM), T(1e-12));
    k.vs = k.v; k.ws = k.w; k.bys = k.by; k.bzs = k.bz;
    if (std::fabs(dk) >= std::fmax(T(1e-12), dtol * bn * bn)) {
      const T f = bn * (SM - k.u) / dk, q = (a * (S[s] - k.u) - bn * bn) / dk;
      k.vs = k.v - k.by * f; k.ws = k.w - k.bz * f; k.bys = k.by * q; k.bzs = k.bz * q;
    }
    k.vbs = SM * bn + k.vs * k.bys + k.ws * k.bzs;
    k.Es = ((S[s] - k.u) * k.E - k.pt * k.u + pts * SM + bn * (k.vb - k.vbs)) / (S[s] - SM);
  }
  const T sl = std::sqrt(K[0].ds), sr = std::sqrt(K[1].ds), sg = bn >= 0 ? 1 : -1, iv = 1 / (sl + sr);
  const int n = SM >= 0 ? 0 : 1;
  const Side& k = K[n];
  const T Ss = n == 0 ? SM - std::fabs(bn) / sl : SM + std::fabs(bn) / sr;
  const T U[8] = {k.d, k.d * k.u, k.d * k.v, k.d * k.w, k.E, bn, k.by, k.bz};
  const T Us[8] = {k.ds, k.ds * SM, k.ds * k.vs, k.ds * k.ws, k.Es, bn, k.bys, k.bzs};
  const T FK[8] = {k.d * k.u, k.d * k.u * k.u + k.pt - bn * bn, k.d * k.u * k.v - bn * k.by, k.d * k.u * k.w - bn * k.bz,
                   (k.E + k.pt) * k.u - bn * k.vb, 0, k.u * k.by - k.v * bn, k.u * k.bz - k.w * bn};
  if (n == 0 ? Ss >= 0 : Ss < 0) {
    for (int i = 0; i < 8; ++i) F[i] = FK[i] + S[n] * (Us[i] - U[i]);
    return;
  }
  const T vy = (sl * K[0].vs + sr * K[1].vs + (K[1].bys - K[0].bys) * sg) * iv;
  const T vz = (sl * K[0].ws + sr * K[1].ws + (K[1].bzs - K[0].bzs) * sg) * iv;
  const T by = (sl * K[1].bys + sr * K[0].bys + sl * sr * (K[1].vs - K[0].vs) * sg) * iv;
  const T bz = (sl * K[1].bzs + sr * K[0].bzs + sl * sr * (K[1].ws - K[0].ws) * sg) * iv;
  const T vbss = SM * bn + vy * by + vz * bz;
  const T Ess = n == 0 ? k.Es - sl * (k.vbs - vbss) * sg : k.Es + sr * (k.vbs - vbss) * sg;
  const T Uss[8] = {k.ds, k.ds * SM, k.ds * vy, k.ds * vz, Ess, bn, by, bz};
  for (int i = 0; i < 8; ++i) F[i] = FK[i] + Ss * Uss[i] - (Ss - S[n]) * Us[i] - S[n] * U[i];
}

// n faces (9 primitive values a side, the normal field in component 5): the device code's flux, the
// reference arithmetic in FP32 and in extended precision, 8 components each
extern "C" void fluxes(int n, const float* L, const float* R, float g, float dtol, float* dev, float* f32, double* ref) {
  for (int i = 0; i < n; ++i) {
    const float *l = L + 9 * i, *r = R + 9 * i;
    pmf::F9 a, b;
    memcpy(a.v, l, sizeof(a.v));
    memcpy(b.v, r, sizeof(b.v));
    const pmf::F9 f = pmf::hlld_x(a, b, g, l[5], 0.0f, 0.0f, dtol);
    memcpy(dev + 8 * i, f.v, 8 * sizeof(float));
    hlld<float>(l, r, g, l[5], dtol, f32 + 8 * i);
    long double x[8];
    hlld<long double>(l, r, g, l[5], dtol, x);
    for (int c = 0; c < 8; ++c) ref[8 * i + c] = (double)x[c];
  }
}

extern "C" void ppm(int n, const float* dl, const float* dr, float* oL, float* oR) {
  for (int i = 0; i < n; ++i) pmf::ppm_offsets(dl[i], dr[i], oL[i], oR[i]);
}
