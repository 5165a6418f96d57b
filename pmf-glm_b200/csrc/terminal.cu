// Terminal-regime induction (lib/MHDKernels/src/terminal_ct.jl): in the overdamped early-PMF
// regime the gas velocity is the terminal velocity v = (F_Maxwell - c_p grad rho) / (rho Gamma)
// and only the induction equation is advanced, by SSPRK2 with a centred curl (GLM states) or
// the edge-averaged face curl (CT states), plus order-2 or order-4 dissipation.
//
//   pmfmhd_terminal_magnetic_force        <- terminal_magnetic_force!       (terminal_ct.jl:99-106)
//   pmfmhd_terminal_magnetic_force_split  <- terminal_magnetic_force_split! (:117-126)
//   pmfmhd_terminal_velocity_max          <- terminal_velocity_max!         (:226-238)
//   pmfmhd_terminal_ct_induction          <- terminal_ct_induction!         (:502-575)
//   pmfmhd_terminal_ct_euler_from_cell_emf <- terminal_ct_euler_from_cell_emf! (:461-486)
//
// Design: the reference recomputes the terminal EMF of each of a cell's six neighbours inside
// its update kernel (the Maxwell force at the neighbour is an array, the velocity and v x B are
// recomputed per use). Here one kernel computes the Maxwell force, the terminal velocity and
// e = v x B once per cell (the values are the same, computed from the same inputs), and the
// stage kernel takes the curl of that EMF field, for CT through the edge means it forms itself:
// two passes per GLM stage, three per CT stage (the third is the face average). Every grid is
// cubic and periodic.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "aux_kernels.cuh"
#include "host_internal.h"

namespace pmf {
namespace {

// Every kernel below gives a thread one (x, y) column of a 32 x 8 tile and marches it through a
// chunk of z-planes. The wrapped x and y offsets of the stencil are formed once per column and
// the values a plane shares with the next stay in registers, so a load costs one add. (With one
// thread per cell and three integer remainders per neighbour the index arithmetic was most of
// the work: a 128^3 CT subcycle took 473 us.) The loops over planes are unrolled by two (the next plane's
// loads overlap this plane's arithmetic), and the order-4 stages hold four blocks an SM although they
// spill some 100 bytes for it. Against plain loops with the compiler's own register counts:
// order-4 induction 64^3 71 -> 57 us (GLM), 128^3 326 -> 283 (CT) and 221 -> 217 (GLM), 256^3 1.91 ->
// 1.68 ms (CT); 128^3 force 22.9 -> 16.8 us. Indices wrap by selects: wrapped by loops, the lanes beyond
// a small cube went round many times (8^3 GLM induction 43 us, 36 with selects, 40 with one thread per
// cell).
constexpr int kX = 32, kY = 8, kT = kX * kY;

struct Cube {
  int N;
  int zc;  // planes per chunk
};
// Launch grid of a cube: as many chunks as give every SM up to three blocks at once (the planes
// of a chunk are serial), of at most 32 planes (larger cubes have blocks enough).
dim3 tiles_of(Cube& G, int sms) {
  const int tx = (G.N + kX - 1) / kX, ty = (G.N + kY - 1) / kY;
  const int chunks = std::max(1, std::min(G.N, 3 * sms / (tx * ty)));
  G.zc = std::min(32, (G.N + chunks - 1) / chunks);
  return dim3(tx, ty, (G.N + G.zc - 1) / G.zc);
}

// The column of a thread: offsets within a plane of its neighbours up to two cells away. An index is
// a 32-bit sum (plane base + offset) that the fields of a kernel share, so a load costs one
// multiply-add for its address.
struct Column {
  int N, nxy;
  unsigned x[5], y[5];  // x[2 + d], y[2 + d]: wrapped x index and row offset at distance d
  int z0, z1;
  bool in;
  // Periodic image of an index at most two outside: one conditional step reaches it unless N is 1. (The
  // lanes beyond the cube take the last column's offsets, which they do not use.)
  __device__ __forceinline__ static int wrap(int i, int n) {
    const int r = i < 0 ? i + n : (i >= n ? i - n : i);
    return n == 1 ? 0 : r;
  }
  __device__ __forceinline__ explicit Column(const Cube& G) : N(G.N), nxy(G.N * G.N) {
    int i = blockIdx.x * kX + (threadIdx.x & (kX - 1)), j = blockIdx.y * kY + threadIdx.x / kX;
    in = i < N && j < N;
    i = min(i, N - 1);
    j = min(j, N - 1);
#pragma unroll
    for (int d = -2; d <= 2; ++d) {
      x[2 + d] = wrap(i + d, N);
      y[2 + d] = wrap(j + d, N) * N;
    }
    z0 = blockIdx.z * G.zc;
    z1 = min(z0 + G.zc, N);
  }
  __device__ __forceinline__ unsigned at(int dx, int dy) const { return y[2 + dy] + x[2 + dx]; }
  __device__ __forceinline__ unsigned plane(int k) const { return (unsigned)(wrap(k, N) * nxy); }
};

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ float dot(const F3& a, const F3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
struct Field3 {
  const float* __restrict__ x;
  const float* __restrict__ y;
  const float* __restrict__ z;
  __device__ __forceinline__ F3 operator[](unsigned c) const { return F3{x[c], y[c], z[c]}; }
};

// Conservative centred Maxwell-stress divergence (terminal_ct.jl:18-51) from the field at the
// upper (p) and lower (m) neighbour along each direction
__device__ __forceinline__ F3 maxwell_force(const F3 (&p)[3], const F3 (&m)[3], float inv2dx) {
  float t[3][3];  // t[component][direction]
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float bp[3] = {p[d].x, p[d].y, p[d].z}, bm[3] = {m[d].x, m[d].y, m[d].z};
    const float b2p = dot(p[d], p[d]), b2m = dot(m[d], m[d]);
#pragma unroll
    for (int c = 0; c < 3; ++c)
      t[c][d] = c == d ? (bp[c] * bp[c] - 0.5f * b2p) - (bm[c] * bm[c] - 0.5f * b2m) : bp[c] * bp[d] - bm[c] * bm[d];
  }
  return F3{(t[0][0] + t[0][1] + t[0][2]) * inv2dx, (t[1][0] + t[1][1] + t[1][2]) * inv2dx,
            (t[2][0] + t[2][1] + t[2][2]) * inv2dx};
}

struct Terminal {
  float inv2dx, gamma_drag, pressure_coeff, smallr, vcap;
};

// Terminal velocity (terminal_ct.jl:125-145), capped at vcap; rp, rm: the density at the upper
// and lower neighbour along each direction
__device__ __forceinline__ F3 terminal_velocity(float rho, const float (&rp)[3], const float (&rm)[3], F3 f,
                                                const Terminal& P) {
  const float r = fmaxf(rho, P.smallr);
  const float gx = P.pressure_coeff * (rp[0] - rm[0]) * P.inv2dx;
  const float gy = P.pressure_coeff * (rp[1] - rm[1]) * P.inv2dx;
  const float gz = P.pressure_coeff * (rp[2] - rm[2]) * P.inv2dx;
  const float invrg = 1.0f / (r * fmaxf(P.gamma_drag, FLT_EPSILON));
  F3 v{(f.x - gx) * invrg, (f.y - gy) * invrg, (f.z - gz) * invrg};
  const float v2 = v.x * v.x + v.y * v.y + v.z * v.z;
  if (v2 > P.vcap * P.vcap) {
    const float q = P.vcap / sqrtf(v2);
    v.x *= q;
    v.y *= q;
    v.z *= q;
  }
  return v;
}

__global__ void __launch_bounds__(kT) force_kernel(Field3 B, float* __restrict__ fx, float* __restrict__ fy,
                                                   float* __restrict__ fz, float* __restrict__ px,
                                                   float* __restrict__ py, float* __restrict__ pz, Cube G,
                                                   float inv2dx) {
  const Column C(G);
  if (!C.in) return;
  const unsigned o = C.at(0, 0);
  F3 zm = B[C.plane(C.z0 - 1) + o], z0 = B[C.plane(C.z0) + o];
#pragma unroll 2
  for (int k = C.z0; k < C.z1; ++k) {
    const unsigned b = C.plane(k);
    const F3 zp = B[C.plane(k + 1) + o];
    const F3 p[3] = {B[b + C.at(1, 0)], B[b + C.at(0, 1)], zp};
    const F3 m[3] = {B[b + C.at(-1, 0)], B[b + C.at(0, -1)], zm};
    zm = z0;
    z0 = zp;
    const F3 f = maxwell_force(p, m, inv2dx);
    if (px == nullptr) {
      fx[b + o] = f.x;
      fy[b + o] = f.y;
      fz[b + o] = f.z;
      continue;
    }
    // split (terminal_ct.jl:53-69): pressure -grad(B^2/2), tension = remainder (into f*)
    const float ppx = -0.5f * (dot(p[0], p[0]) - dot(m[0], m[0])) * inv2dx;
    const float ppy = -0.5f * (dot(p[1], p[1]) - dot(m[1], m[1])) * inv2dx;
    const float ppz = -0.5f * (dot(p[2], p[2]) - dot(m[2], m[2])) * inv2dx;
    px[b + o] = ppx;
    py[b + o] = ppy;
    pz[b + o] = ppz;
    fx[b + o] = f.x - ppx;
    fy[b + o] = f.y - ppy;
    fz[b + o] = f.z - ppz;
  }
}

// Cell EMF e = v x B with the terminal velocity of the field B (ex null: not stored), and the
// running maximum of |v| (bits of a non-negative float; null: not wanted). 20 loads per cell.
__global__ void __launch_bounds__(kT) cell_emf_kernel(const float* __restrict__ rho, Field3 B, float* __restrict__ ex,
                                                      float* __restrict__ ey, float* __restrict__ ez,
                                                      unsigned int* __restrict__ vmax_bits, Cube G, Terminal P) {
  const Column C(G);
  float vm = 0.0f;
  if (C.in) {
    const unsigned o = C.at(0, 0), xp = C.at(1, 0), xm = C.at(-1, 0), yp = C.at(0, 1), ym = C.at(0, -1);
    unsigned n = C.plane(C.z0 - 1);
    F3 bm = B[n + o];
    float rm = rho[n + o];
    n = C.plane(C.z0);
    F3 b0 = B[n + o];
    float r0 = rho[n + o];
#pragma unroll 2
    for (int k = C.z0; k < C.z1; ++k) {
      const unsigned b = C.plane(k);
      n = C.plane(k + 1);
      const F3 bp = B[n + o];
      const float rp = rho[n + o];
      const F3 p[3] = {B[b + xp], B[b + yp], bp}, m[3] = {B[b + xm], B[b + ym], bm};
      const float rhop[3] = {rho[b + xp], rho[b + yp], rp}, rhom[3] = {rho[b + xm], rho[b + ym], rm};
      const F3 v = terminal_velocity(r0, rhop, rhom, maxwell_force(p, m, P.inv2dx), P);
      if (vmax_bits != nullptr) vm = fmaxf(vm, sqrtf(v.x * v.x + v.y * v.y + v.z * v.z));
      if (ex != nullptr) {
        ex[b + o] = v.y * b0.z - v.z * b0.y;
        ey[b + o] = v.z * b0.x - v.x * b0.z;
        ez[b + o] = v.x * b0.y - v.y * b0.x;
      }
      bm = b0;
      b0 = bp;
      rm = r0;
      r0 = rp;
    }
  }
  if (vmax_bits != nullptr) {
    vm = block_reduce_max(vm);
    if (threadIdx.x == 0) atomicMax(vmax_bits, __float_as_uint(vm));
  }
}

// Dissipation term of one field along a column: the Laplacian (order 2) or the 25-point
// bilaplacian (order 4, terminal_ct.jl:166-181). The sums over the four near neighbours of three
// planes and the centre values of five are kept: 5 or 13 loads per cell.
template <int ORDER> struct Dissip {
  const float* __restrict__ A;
  float cm2, cm1, c0, cp1, cp2, sm, s0, sp;
  __device__ __forceinline__ float near4(unsigned b, const Column& C) const {
    return A[b + C.at(1, 0)] + A[b + C.at(-1, 0)] + A[b + C.at(0, 1)] + A[b + C.at(0, -1)];
  }
  __device__ __forceinline__ Dissip(const float* A_, const Column& C) : A(A_) {
    const unsigned o = C.at(0, 0);
    const int k = C.z0;
    cm1 = A[C.plane(k - 1) + o];
    c0 = A[C.plane(k) + o];
    if (ORDER == 4) {
      cm2 = A[C.plane(k - 2) + o];
      cp1 = A[C.plane(k + 1) + o];
      sm = near4(C.plane(k - 1), C);
      s0 = near4(C.plane(k), C);
    }
  }
  // the term at plane k (the planes of the chunk in order)
  __device__ __forceinline__ float operator()(int k, const Column& C, float invdx2, float eta) {
    const unsigned b = C.plane(k);
    const unsigned o = C.at(0, 0);
    float r;
    if (ORDER == 4) {
      cp2 = A[C.plane(k + 2) + o];
      sp = near4(C.plane(k + 1), C);
      const float a1 = s0 + cp1 + cm1;
      const float a2 = A[b + C.at(2, 0)] + A[b + C.at(-2, 0)] + A[b + C.at(0, 2)] + A[b + C.at(0, -2)] + cp2 + cm2;
      const float dg = A[b + C.at(1, 1)] + A[b + C.at(1, -1)] + A[b + C.at(-1, 1)] + A[b + C.at(-1, -1)] + sp + sm;
      r = -eta * (((42.0f * c0 - 12.0f * a1) + a2 + 2.0f * dg) * invdx2 * invdx2);
      cm2 = cm1;
      sm = s0;
      s0 = sp;
      cm1 = c0;
      c0 = cp1;
      cp1 = cp2;
    } else {
      cp1 = A[C.plane(k + 1) + o];
      r = eta * (((near4(b, C) + cp1 + cm1) - 6.0f * c0) * invdx2);
      cm1 = c0;
      c0 = cp1;
    }
    return r;
  }
};

// Resident blocks an SM asked of a stage kernel (order 2 needs no cap)
template <int ORDER> constexpr int kStageBlocks = ORDER == 4 ? 4 : 1;

struct Stage {
  float dt, inv2dx, invdx, invdx2, eta;
};

// GLM SSPRK2 stage (terminal_ct.jl:240-293). STAGE 0: out = B + dt*rhs(e, B).
// STAGE 1: B <- (B + pB + dt*rhs(e, pB))/2 in place, E follows the magnetic energy.
template <int ORDER, int STAGE>
__global__ void __launch_bounds__(kT, kStageBlocks<ORDER>) glm_stage_kernel(Field3 e, float* bx, float* by, float* bz, float* pbx,
                                                       float* pby, float* pbz, float* __restrict__ E, Cube G,
                                                       Stage S) {
  const Column C(G);
  if (!C.in) return;
  const unsigned o = C.at(0, 0), xp = C.at(1, 0), xm = C.at(-1, 0), yp = C.at(0, 1), ym = C.at(0, -1);
  Dissip<ORDER> dx(STAGE == 0 ? bx : pbx, C), dy(STAGE == 0 ? by : pby, C), dz(STAGE == 0 ? bz : pbz, C);
  unsigned n = C.plane(C.z0 - 1);
  float exm = e.x[n + o], eym = e.y[n + o];
  n = C.plane(C.z0);
  float ex0 = e.x[n + o], ey0 = e.y[n + o];
#pragma unroll 2
  for (int k = C.z0; k < C.z1; ++k) {
    const unsigned b = C.plane(k);
    n = C.plane(k + 1);
    const float exp_ = e.x[n + o], eyp = e.y[n + o];
    const float cx = ((e.z[b + yp] - e.z[b + ym]) - (eyp - eym)) * S.inv2dx;
    const float cy = ((exp_ - exm) - (e.z[b + xp] - e.z[b + xm])) * S.inv2dx;
    const float cz = ((e.y[b + xp] - e.y[b + xm]) - (e.x[b + yp] - e.x[b + ym])) * S.inv2dx;
    exm = ex0;
    ex0 = exp_;
    eym = ey0;
    ey0 = eyp;
    const float rx = cx + dx(k, C, S.invdx2, S.eta), ry = cy + dy(k, C, S.invdx2, S.eta),
                rz = cz + dz(k, C, S.invdx2, S.eta);
    const float ox = bx[b + o], oy = by[b + o], oz = bz[b + o];
    if (STAGE == 0) {
      pbx[b + o] = ox + S.dt * rx;
      pby[b + o] = oy + S.dt * ry;
      pbz[b + o] = oz + S.dt * rz;
    } else {
      const float nx = 0.5f * ((ox + pbx[b + o]) + S.dt * rx);
      const float ny = 0.5f * ((oy + pby[b + o]) + S.dt * ry);
      const float nz = 0.5f * ((oz + pbz[b + o]) + S.dt * rz);
      const float eb0 = 0.5f * (ox * ox + oy * oy + oz * oz);
      const float eb1 = 0.5f * (nx * nx + ny * ny + nz * nz);
      bx[b + o] = nx;
      by[b + o] = ny;
      bz[b + o] = nz;
      E[b + o] = fmaxf((E[b + o] + eb1) - eb0, 1e-30f);
    }
  }
}

// Curl of the edge EMFs on the lower faces of a column's cells, the edge EMF being the mean of
// the four cell EMFs around the edge (terminal_ct.jl:325-345): formed here from the cell EMFs,
// whose plane values are shared by consecutive planes (14 loads per cell), instead of by a pass
// that writes three edge arrays and another that reads them.
struct EdgeCurl {
  Field3 e;
  float xjm, x0, xjp;  // ecx at (j-1, j, j+1) of the plane below
  float yim, y0, yip;  // ecy at (i-1, i, i+1) of the plane below
  float qjm, q0, qjp;  // the same of the current plane
  float wim, w0, wip;
  __device__ __forceinline__ EdgeCurl(const Field3& e_, const Column& C) : e(e_) {
    unsigned b = C.plane(C.z0 - 1);
    xjm = e.x[b + C.at(0, -1)]; x0 = e.x[b + C.at(0, 0)]; xjp = e.x[b + C.at(0, 1)];
    yim = e.y[b + C.at(-1, 0)]; y0 = e.y[b + C.at(0, 0)]; yip = e.y[b + C.at(1, 0)];
    b = C.plane(C.z0);
    qjm = e.x[b + C.at(0, -1)]; q0 = e.x[b + C.at(0, 0)]; qjp = e.x[b + C.at(0, 1)];
    wim = e.y[b + C.at(-1, 0)]; w0 = e.y[b + C.at(0, 0)]; wip = e.y[b + C.at(1, 0)];
  }
  __device__ __forceinline__ static float mean(float c, float a, float b, float ab) { return 0.25f * (((c + a) + b) + ab); }
  // un-normalised curl (differences of edge EMFs) at plane k (the planes of the chunk in order)
  __device__ __forceinline__ F3 operator()(int k, const Column& C) {
    const unsigned b = C.plane(k), bp = C.plane(k + 1);
    const float zc = e.z[b + C.at(0, 0)], zim = e.z[b + C.at(-1, 0)], zjm = e.z[b + C.at(0, -1)];
    const float ez = mean(zc, zim, zjm, e.z[b + C.at(-1, -1)]);
    const float ez_jp = mean(e.z[b + C.at(0, 1)], e.z[b + C.at(-1, 1)], zc, zim);
    const float ez_ip = mean(e.z[b + C.at(1, 0)], zc, e.z[b + C.at(1, -1)], zjm);
    const float ujm = e.x[bp + C.at(0, -1)], u0 = e.x[bp + C.at(0, 0)], ujp = e.x[bp + C.at(0, 1)];
    const float vim = e.y[bp + C.at(-1, 0)], v0 = e.y[bp + C.at(0, 0)], vip = e.y[bp + C.at(1, 0)];
    const float ex = mean(q0, qjm, x0, xjm), ex_jp = mean(qjp, q0, xjp, x0), ex_kp = mean(u0, ujm, q0, qjm);
    const float ey = mean(w0, wim, y0, yim), ey_ip = mean(wip, w0, yip, y0), ey_kp = mean(v0, vim, w0, wim);
    xjm = qjm; x0 = q0; xjp = qjp; yim = wim; y0 = w0; yip = wip;
    qjm = ujm; q0 = u0; qjp = ujp; wim = vim; w0 = v0; wip = vip;
    return F3{(ez_jp - ez) - (ey_kp - ey), (ex_kp - ex) - (ez_ip - ez), (ey_ip - ey) - (ex_jp - ex)};
  }
};

// CT SSPRK2 stage on the faces (terminal_ct.jl:347-407). STAGE 0: pf = f + dt*rate(e, f).
// STAGE 1: f <- (f + pf + dt*rate(e, pf))/2 in place, Kahan-compensated when `comp`.
template <int ORDER, int STAGE>
__global__ void __launch_bounds__(kT, kStageBlocks<ORDER>) face_stage_kernel(Field3 ec, float* fx, float* fy, float* fz, float* pfx,
                                                        float* pfy, float* pfz, float* __restrict__ rbx,
                                                        float* __restrict__ rby, float* __restrict__ rbz, Cube G,
                                                        Stage S, int comp) {
  const Column C(G);
  if (!C.in) return;
  const unsigned o = C.at(0, 0);
  Dissip<ORDER> dx(STAGE == 0 ? fx : pfx, C), dy(STAGE == 0 ? fy : pfy, C), dz(STAGE == 0 ? fz : pfz, C);
  EdgeCurl curl(ec, C);
#pragma unroll 2
  for (int k = C.z0; k < C.z1; ++k) {
    const unsigned b = C.plane(k);
    const F3 u = curl(k, C);
    const float x = u.x * S.invdx + dx(k, C, S.invdx2, S.eta), y = u.y * S.invdx + dy(k, C, S.invdx2, S.eta),
                z = u.z * S.invdx + dz(k, C, S.invdx2, S.eta);
    const float ox = fx[b + o], oy = fy[b + o], oz = fz[b + o];
    if (STAGE == 0) {
      pfx[b + o] = ox + S.dt * x;
      pfy[b + o] = oy + S.dt * y;
      pfz[b + o] = oz + S.dt * z;
    } else if (comp) {
      float r1 = rbx[b + o], r2 = rby[b + o], r3 = rbz[b + o];
      fx[b + o] = comp_add(ox, 0.5f * ((pfx[b + o] - ox) + S.dt * x), r1);
      fy[b + o] = comp_add(oy, 0.5f * ((pfy[b + o] - oy) + S.dt * y), r2);
      fz[b + o] = comp_add(oz, 0.5f * ((pfz[b + o] - oz) + S.dt * z), r3);
      rbx[b + o] = r1;
      rby[b + o] = r2;
      rbz[b + o] = r3;
    } else {
      fx[b + o] = 0.5f * ((ox + pfx[b + o]) + S.dt * x);
      fy[b + o] = 0.5f * ((oy + pfy[b + o]) + S.dt * y);
      fz[b + o] = 0.5f * ((oz + pfz[b + o]) + S.dt * z);
    }
  }
}

// Face average into cell B; with E, E follows the magnetic-energy change (floor smallE)
// (terminal_ct.jl:409-427, ct.jl:205-219 `_ct_bcc_k!` without E).
__global__ void __launch_bounds__(kT) face_average_kernel(const float* __restrict__ fx, const float* __restrict__ fy,
                                                          const float* __restrict__ fz, float* __restrict__ bx,
                                                          float* __restrict__ by, float* __restrict__ bz,
                                                          float* __restrict__ E, float* __restrict__ psi, Cube G,
                                                          int energy_mode) {
  const Column C(G);
  if (!C.in) return;
  const unsigned o = C.at(0, 0);
  float z0 = fz[C.plane(C.z0) + o];
#pragma unroll 2
  for (int k = C.z0; k < C.z1; ++k) {
    const unsigned b = C.plane(k);
    const float zp = fz[C.plane(k + 1) + o];
    const float nx = 0.5f * (fx[b + o] + fx[b + C.at(1, 0)]);
    const float ny = 0.5f * (fy[b + o] + fy[b + C.at(0, 1)]);
    const float nz = 0.5f * (z0 + zp);
    z0 = zp;
    if (energy_mode != 0) {
      const float ox = bx[b + o], oy = by[b + o], oz = bz[b + o];
      if (energy_mode == 1) {  // terminal corrector: E += eb1 - eb0, floored
        const float eb0 = 0.5f * (ox * ox + oy * oy + oz * oz);
        const float eb1 = 0.5f * (nx * nx + ny * ny + nz * nz);
        E[b + o] = fmaxf((E[b + o] + eb1) - eb0, 1e-30f);
      } else {  // face install: E += (|B_new|^2 - |B_old|^2)/2, psi = 0
        E[b + o] = E[b + o] + 0.5f * ((nx * nx + ny * ny + nz * nz) - (ox * ox + oy * oy + oz * oz));
        psi[b + o] = 0.0f;
      }
    }
    bx[b + o] = nx;
    by[b + o] = ny;
    bz[b + o] = nz;
  }
}

// Forward-Euler compensated face update from the cell EMFs' edge means (terminal_ct.jl:461-474)
__global__ void __launch_bounds__(kT) face_euler_kernel(Field3 ec, float* fx, float* fy, float* fz, float* rbx,
                                                        float* rby, float* rbz, Cube G, float dt, float invdx) {
  const Column C(G);
  if (!C.in) return;
  const unsigned o = C.at(0, 0);
  EdgeCurl curl(ec, C);
#pragma unroll 2
  for (int k = C.z0; k < C.z1; ++k) {
    const unsigned b = C.plane(k);
    const F3 u = curl(k, C);
    float r1 = rbx[b + o], r2 = rby[b + o], r3 = rbz[b + o];
    fx[b + o] = comp_add(fx[b + o], dt * u.x * invdx, r1);
    fy[b + o] = comp_add(fy[b + o], dt * u.y * invdx, r2);
    fz[b + o] = comp_add(fz[b + o], dt * u.z * invdx, r3);
    rbx[b + o] = r1;
    rby[b + o] = r2;
    rbz[b + o] = r3;
  }
}

int cube_of(const pmfmhd_grid* g, Cube* G) {
  if (g->nx != g->ny || g->nx != g->nz) return PMFMHD_ESHAPE;  // terminal CT requires a cubic grid
  if (!(g->bc[0] == PMFMHD_BC_PERIODIC && g->bc[1] == PMFMHD_BC_PERIODIC && g->bc[2] == PMFMHD_BC_PERIODIC))
    return PMFMHD_EUNSUPPORTED;
  G->N = g->nx;
  return PMFMHD_OK;
}

}  // namespace
}  // namespace pmf

namespace pmf {
namespace {
using namespace host;
// Maximum terminal speed of U (blocking). Nothing of the caller's is written: the call that asks may
// still be refused for its subcycle limit. (Keeping the EMF of this pass for the first stage would
// save a 128^3 CT subcycle one of its six passes.)
int velocity_max(pmfmhd_ctx* c, const pmfmhd_grid* g, const float* const* U, Cube G, const dim3& tiles,
                 const Terminal& P, double* vmax, cudaStream_t s) {
  PMF_CK(cudaMemsetAsync(c->d_u64, 0, sizeof(unsigned int), s));
  unsigned int* bits = reinterpret_cast<unsigned int*>(c->d_u64);
  cell_emf_kernel<<<tiles, kT, 0, s>>>(U[0], Field3{U[5], U[6], U[7]}, nullptr, nullptr, nullptr, bits, G, P);
  PMF_CK(cudaGetLastError());
  PMF_CK(cudaMemcpyAsync(c->h_pin, bits, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
  PMF_CK(cudaStreamSynchronize(s));
  float v;
  std::memcpy(&v, c->h_pin, sizeof(v));
  *vmax = (double)v;
  return PMFMHD_OK;
}
}  // namespace
}  // namespace pmf

using namespace pmf;
using namespace pmf::host;

extern "C" {

int pmfmhd_terminal_magnetic_force(pmfmhd_ctx* c, const pmfmhd_grid* g, const float* const B[3], float* const F[3],
                                   float* const P[3], void* stream) {
  if (c == nullptr || B == nullptr || F == nullptr) return PMFMHD_EINVAL;
  int rc = check_grid(g);
  if (rc) return rc;
  Cube G;
  if ((rc = cube_of(g, &G))) return rc;
  for (int d = 0; d < 3; ++d)
    if (!B[d] || !F[d] || (P && !P[d])) return PMFMHD_EINVAL;
  const dim3 tiles = tiles_of(G, c->sms);
  force_kernel<<<tiles, kT, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      Field3{B[0], B[1], B[2]}, F[0], F[1], F[2], P ? P[0] : nullptr, P ? P[1] : nullptr, P ? P[2] : nullptr, G,
      1.0f / (2.0f * g->dx));
  PMF_CK(cudaGetLastError());
  return PMFMHD_OK;
}

int pmfmhd_terminal_velocity_max(pmfmhd_ctx* c, const pmfmhd_grid* g, const float* const U[9], float gamma_drag,
                                 float pressure_coeff, float vcap, double* vmax, void* stream) {
  if (c == nullptr || U == nullptr || vmax == nullptr || !U[0] || !U[5] || !U[6] || !U[7]) return PMFMHD_EINVAL;
  int rc = check_grid(g);
  if (rc) return rc;
  Cube G;
  if ((rc = cube_of(g, &G))) return rc;
  const dim3 tiles = tiles_of(G, c->sms);
  const Terminal P{1.0f / (2.0f * g->dx), gamma_drag, pressure_coeff, g->smallr, vcap};
  return velocity_max(c, g, U, G, tiles, P, vmax, reinterpret_cast<cudaStream_t>(stream));
}

int pmfmhd_terminal_ct_induction(pmfmhd_ctx* c, const pmfmhd_grid* g, float* const U[9], float* const scratch[9],
                                 float* ct, float dt, float gamma_drag, float pressure_coeff, float cfl,
                                 float dissipation, int dissipation_order, float vcap, int max_subcycles,
                                 int compensate, int* nsub_out, double* vmax_out, double* eta_out, void* stream) {
  if (c == nullptr || U == nullptr || scratch == nullptr) return PMFMHD_EINVAL;
  int rc = check_grid(g);
  if (rc) return rc;
  Cube G;
  if ((rc = cube_of(g, &G))) return rc;
  for (int f = 0; f < 9; ++f)
    if (!U[f] || !scratch[f]) return PMFMHD_EINVAL;
  if (!(cfl > 0.0f && cfl <= 1.0f) || !(dissipation >= 0.0f && dissipation <= 1.0f)) return PMFMHD_EINVAL;
  if (dissipation_order != 2 && dissipation_order != 4) return PMFMHD_EINVAL;
  if (!std::isfinite(dt) || !std::isfinite(gamma_drag) || !std::isfinite(pressure_coeff)) return PMFMHD_EINVAL;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long n = ncells(g);
  const dim3 tiles = tiles_of(G, c->sms);
  const Terminal P{1.0f / (2.0f * g->dx), gamma_drag, pressure_coeff, g->smallr, vcap};
  auto slot = [&](int q) { return ct + (size_t)q * n; };
  double vmax = 0.0;
  if ((rc = velocity_max(c, g, U, G, tiles, P, &vmax, s))) return rc;
  const double dx = (double)g->dx;
  const long long nsub = std::max<long long>(
      1, (long long)std::ceil((double)dt * vmax / std::max((double)cfl * dx, DBL_EPSILON)));
  if (nsub > max_subcycles) return PMFMHD_EINADMISSIBLE;  // the caller's subcycle limit
  Stage S;
  S.dt = (float)((double)dt / (double)nsub);
  S.inv2dx = 1.0f / (2.0f * g->dx);
  S.invdx = 1.0f / g->dx;
  S.invdx2 = 1.0f / (g->dx * g->dx);
  S.eta = dissipation_order == 4 ? (float)(dissipation / 12.0) * (float)vmax * (g->dx * g->dx * g->dx)
                                 : dissipation * (float)vmax * g->dx;
  const bool o4 = dissipation_order == 4;
  const Field3 B{U[5], U[6], U[7]}, Bp{scratch[5], scratch[6], scratch[7]};  // the predictor's cell B
  for (long long it = 0; it < nsub; ++it) {
    if (ct == nullptr) {
      // GLM: cell EMF -> scratch[1..3], predictor -> scratch[5..7]
      const Field3 e{scratch[1], scratch[2], scratch[3]};
      const auto stage0 = o4 ? glm_stage_kernel<4, 0> : glm_stage_kernel<2, 0>;
      const auto stage1 = o4 ? glm_stage_kernel<4, 1> : glm_stage_kernel<2, 1>;
      cell_emf_kernel<<<tiles, kT, 0, s>>>(U[0], B, scratch[1], scratch[2], scratch[3], nullptr, G, P);
      stage0<<<tiles, kT, 0, s>>>(e, U[5], U[6], U[7], scratch[5], scratch[6], scratch[7], U[4], G, S);
      cell_emf_kernel<<<tiles, kT, 0, s>>>(U[0], Bp, scratch[1], scratch[2], scratch[3], nullptr, G, P);
      stage1<<<tiles, kT, 0, s>>>(e, U[5], U[6], U[7], scratch[5], scratch[6], scratch[7], U[4], G, S);
    } else {
      // CT: workspace in the packed buffer (cell EMF ec*, predicted faces mf*), the predictor's
      // cell B in scratch[5..7]
      const Field3 ec{slot(CT_ECX), slot(CT_ECY), slot(CT_ECZ)};
      const auto stage0 = o4 ? face_stage_kernel<4, 0> : face_stage_kernel<2, 0>;
      const auto stage1 = o4 ? face_stage_kernel<4, 1> : face_stage_kernel<2, 1>;
      cell_emf_kernel<<<tiles, kT, 0, s>>>(U[0], B, slot(CT_ECX), slot(CT_ECY), slot(CT_ECZ), nullptr, G, P);
      stage0<<<tiles, kT, 0, s>>>(ec, slot(CT_BXF), slot(CT_BYF), slot(CT_BZF), slot(CT_MFX), slot(CT_MFY),
                                  slot(CT_MFZ), nullptr, nullptr, nullptr, G, S, 0);
      face_average_kernel<<<tiles, kT, 0, s>>>(slot(CT_MFX), slot(CT_MFY), slot(CT_MFZ), scratch[5], scratch[6],
                                               scratch[7], nullptr, nullptr, G, 0);
      cell_emf_kernel<<<tiles, kT, 0, s>>>(U[0], Bp, slot(CT_ECX), slot(CT_ECY), slot(CT_ECZ), nullptr, G, P);
      stage1<<<tiles, kT, 0, s>>>(ec, slot(CT_BXF), slot(CT_BYF), slot(CT_BZF), slot(CT_MFX), slot(CT_MFY),
                                  slot(CT_MFZ), slot(CT_RBX), slot(CT_RBY), slot(CT_RBZ), G, S, compensate);
      face_average_kernel<<<tiles, kT, 0, s>>>(slot(CT_BXF), slot(CT_BYF), slot(CT_BZF), U[5], U[6], U[7], U[4],
                                               nullptr, G, 1);
    }
  }
  PMF_CK(cudaGetLastError());
  if (nsub_out) *nsub_out = (int)nsub;
  if (vmax_out) *vmax_out = vmax;
  if (eta_out) *eta_out = (double)S.eta;
  return PMFMHD_OK;
}

int pmfmhd_terminal_ct_euler_from_cell_emf(pmfmhd_ctx* c, const pmfmhd_grid* g, float* const U[9], float* ct,
                                           float dt, void* stream) {
  if (c == nullptr || U == nullptr || ct == nullptr) return PMFMHD_EINVAL;
  int rc = check_grid(g);
  if (rc) return rc;
  Cube G;
  if ((rc = cube_of(g, &G))) return rc;
  for (int f = 4; f < 9; ++f)
    if (!U[f]) return PMFMHD_EINVAL;
  if (!std::isfinite(dt)) return PMFMHD_EINVAL;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long n = ncells(g);
  const dim3 tiles = tiles_of(G, c->sms);
  auto slot = [&](int q) { return ct + (size_t)q * n; };
  face_euler_kernel<<<tiles, kT, 0, s>>>(Field3{slot(CT_ECX), slot(CT_ECY), slot(CT_ECZ)}, slot(CT_BXF),
                                         slot(CT_BYF), slot(CT_BZF), slot(CT_RBX), slot(CT_RBY), slot(CT_RBZ), G, dt,
                                         1.0f / g->dx);
  face_average_kernel<<<tiles, kT, 0, s>>>(slot(CT_BXF), slot(CT_BYF), slot(CT_BZF), U[5], U[6], U[7], U[4], U[8], G,
                                           2);
  PMF_CK(cudaGetLastError());
  return PMFMHD_OK;
}

}  // extern "C"
