// kbc_d3q39.cu — the D3Q39 entropic KBC level step on B200: the reference's
// stream_collide_entropic_d3q39! (src/collision/kernel_entropic_d3q39.jl:529-3368) on a level
// without sponge, wall model, AMR parent, thermal coupling or lattice shift, with its lambda
// warm-start cache (src/collision/timestep.jl:1447-1450) and the level ping-pong. Domain faces
// take the default boundary options (:983-1278): k_kbc_fill writes each face value into the ghost
// slot its pull reads before the step; the inlet face is pinned to the inlet equilibrium's mass and
// momentum (:1313-1352); solid cells bounce back (:1602-1613).
//
// One thread per cell, 128 threads per CTA (a quarter of an 8^3 block). A thread pulls its 39
// populations through the block's 27-entry neighbour table (|c| <= 3 < 8, so at most one block hop)
// and parks them in shared memory while the 13-moment Newton solve (warm-started from the cached
// multipliers) runs in registers. Then WALE from the 6 face neighbours' previous velocity, the Mach-pocket
// viscosity, positivity clamp and realizability guard, the mirror split, the entropic alpha, the
// KBC update and the post-collision guards. It writes 39 populations, rho, u and the 13
// multipliers. The step is bound by FP32 issue (a Newton sweep is 117 exponentials, an entropy
// evaluation 39 logarithms and divides), not by its 444 bytes of HBM traffic per cell.
//
// Every operation is the reference's, in its order, as single IEEE binary32 operations (the
// library builds with -fmad=false); exp and log are kbc::exp / kbc::log, shared with the CPU
// restatement, so the step is bit-identical to it. Terms whose coefficient is a compile-time
// zero are left out of sums: adding +-0 to a value changes at most the sign of a zero sum, which no
// later operation of the step can observe.
//
// Layout (library-owned): f[b][k][cell] and lambda[b][m][cell] block-major (FP32), rho and vel in
// the reference layout rho(8,8,8,nb), vel(8,8,8,nb,3).
#include <cstdarg>
#include <cstdio>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "../../include/oal.h"
#include "kbc_math.h"
#include "kbc_d3q39.h"

oal_status oal_internal_set_error(oal_status s, const char* msg);

namespace {

constexpr int Q = 39;
constexpr int kThreads = 128;
// Fast path (CUDA's expf / logf): the cached multipliers start the solve whenever their
// equilibrium matches the target moments within sqrt(KBC_FAST_WARM_GATE * TOL_SQ), i.e. to ~3e-2
// relative. The reference's staleness gate (factor 100, ~2.7e-5 relative) rejects them in nearly
// every cell of an unsteady flow, so every solve restarts from the polynomial guess; both starts
// converge to the same multipliers within the solve's tolerance.
#ifndef KBC_FAST_WARM_GATE
#define KBC_FAST_WARM_GATE 1e8f
#endif
#ifndef KBC_FAST_TOL_SCALE
#define KBC_FAST_TOL_SCALE 1.0f
#endif
#ifndef KBC_NEWTON_MAX
#define KBC_NEWTON_MAX 8  // fast path: full Newton steps before the block-Jacobi fallback
#endif
#ifndef KBC_FAST_MIN_BLOCKS
#define KBC_FAST_MIN_BLOCKS 3  // fast path: CTAs per SM (the 13 x 13 Newton system lives in registers)
#endif
#ifndef KBC_FAST_MAX_SWEEPS
#define KBC_FAST_MAX_SWEEPS 200
#endif
#ifndef KBC_MIN_BLOCKS
#define KBC_MIN_BLOCKS 6  // CTAs per SM the register budget is cut for (33 KB of shared memory each)
#endif

// lattice.jl:177-262, 0-based
__host__ __device__ constexpr int kcx(int k) {
  constexpr int t[Q] = {0, -1, 1, 0, 0, 0, 0, -1, -1, -1, -1, 1, 1, 1, 1, -2, 2, 0, 0, 0,
                        0, -2, -2, 2, 2, -2, -2, 2, 2, 0, 0, 0, 0, -3, 3, 0, 0, 0, 0};
  return t[k];
}
__host__ __device__ constexpr int kcy(int k) {
  constexpr int t[Q] = {0, 0, 0, -1, 1, 0, 0, -1, -1, 1, 1, -1, -1, 1, 1, 0, 0, -2, 2, 0,
                        0, -2, 2, -2, 2, 0, 0, 0, 0, -2, -2, 2, 2, 0, 0, -3, 3, 0, 0};
  return t[k];
}
__host__ __device__ constexpr int kcz(int k) {
  constexpr int t[Q] = {0, 0, 0, 0, 0, -1, 1, -1, 1, -1, 1, -1, 1, -1, 1, 0, 0, 0, 0, -2,
                        2, 0, 0, 0, 0, -2, 2, -2, 2, -2, 2, -2, 2, 0, 0, 0, 0, -3, 3};
  return t[k];
}
__host__ __device__ constexpr int kopp(int k) {
  constexpr int t[Q] = {0, 2, 1, 4, 3, 6, 5, 14, 13, 12, 11, 10, 9, 8, 7, 16, 15, 18, 17, 20,
                        19, 24, 23, 22, 21, 28, 27, 26, 25, 32, 31, 30, 29, 34, 33, 36, 35, 38, 37};
  return t[k];
}
__host__ __device__ constexpr int nbr13(int ox, int oy, int oz) { return (ox + 1) + 3 * (oy + 1) + 9 * (oz + 1); }
__host__ __device__ constexpr float kw(int k) {
  return k < 7 ? float(1.0 / 12) : k < 15 ? float(1.0 / 27) : k < 21 ? float(2.0 / 135) : k < 33 ? float(1.0 / 432)
                                                                                             : float(1.0 / 1620);
}

constexpr float CS2 = float(2.0 / 3.0);
constexpr float F_FLOOR = 1e-15f;

// basis of the 13-moment solve without the constant: (cx, cy, cz, cx^2-cs2, cy^2-cs2, cz^2-cs2,
// cxcy, cxcz, cycz, cx efl, cy efl, cz efl), efl = |c|^2 - 5 cs2 (physics_utils.jl:583-595)
__host__ __device__ constexpr float kbasis(int m, int k) {
  const float cx = float(kcx(k)) - 0.0f, cy = float(kcy(k)) - 0.0f, cz = float(kcz(k)) - 0.0f;
  const float efl = (cx * cx + cy * cy + cz * cz) - 5.0f * CS2;
  return m == 0 ? cx : m == 1 ? cy : m == 2 ? cz : m == 3 ? cx * cx - CS2 : m == 4 ? cy * cy - CS2
       : m == 5 ? cz * cz - CS2 : m == 6 ? cx * cy : m == 7 ? cx * cz : m == 8 ? cy * cz
       : m == 9 ? cx * efl : m == 10 ? cy * efl : cz * efl;
}

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }
// Julia's min / max on floats: NaN in, NaN out
__device__ __forceinline__ float jmax(float a, float b) { return (a != a || b != b) ? qnan() : (a < b ? b : a); }
__device__ __forceinline__ float jmin(float a, float b) { return (a != a || b != b) ? qnan() : (a < b ? a : b); }
__device__ __forceinline__ float jclamp(float v, float lo, float hi) { return v > hi ? hi : (v < lo ? lo : v); }
__device__ __forceinline__ float smooth(float t) { return t * t * (3.0f - 2.0f * t); }
// exp and log: FAST = CUDA's expf / logf (what the reference's Float32 exp and log compile to on
// its CUDA backend, within 2 ulp); otherwise the software routines shared with the CPU restatement
// (kbc_math.h), so that the step is bit-identical to it
template <bool FAST> __device__ __forceinline__ float kexp(float x) {
  if constexpr (FAST) return __expf(x);
  else return kbc::exp(x);
}
template <bool FAST> __device__ __forceinline__ float klog(float x) {
  if constexpr (FAST) return __logf(x);
  else return kbc::log(x);
}
// s + a b: one rounding when FAST (fused), the reference's two otherwise
template <bool FAST> __device__ __forceinline__ float kmad(float a, float b, float s) {
  if constexpr (FAST) return __fmaf_rn(a, b, s);
  else return s + a * b;
}
template <bool FAST = false>
__device__ __forceinline__ float safe_log(float x) { return x > 0.0f ? klog<FAST>(x) : -88.0f; }

struct KbcArgs {
  const float* fin;
  float* fout;
  const float* vin;
  float* vout;
  float* rho;
  float* lam;
  const int32_t* nbr;
  int32_t nb;
  int32_t solver;  // 0 bisection, 1 Newton, 2 approximate, 3 Taylor
  int32_t hrr;     // HRR blend active (hrr_hybrid and hrr_sigma < 0.999)
  float tau, c_wale, nu_bg, amr_sgs_scale, u_inlet, sigma0, hrr_sigma, nu_floor, shock_nu_max;
  float feq_inlet[Q];
  // domain faces and solids (null / 0 on periodic boxes without obstacles)
  const int4* binfo;        // 1-based block coordinates: the inlet-face pin applies at global x = 1
  const uint32_t* bflags;   // BF_NEAR_SOLID blocks carry per-cell solid masks
  const int32_t* mslot;
  const uint32_t* cmask;
  int32_t faces;            // the level has ghost blocks
  float trho, tjx, tjy, tjz;  // moments of feq_inlet, the inlet-face pin's targets
  float warm_gate;          // fast path: squared moment residual (in TOL_SQ units) up to which
                            // the cached multipliers start the solve (the reference: 100)
  const float* sponge;      // [nb*512] or null: the sponge blend toward the inlet state
  const float* wdist;       // [nb*512] or null: wall distance, NaN where there is none
  int32_t sponge_blend;     // sponge_blend_distributions
  float svv_x, svv_yz;      // spectral vanishing viscosity strengths (0 = off)
};

// the face fill of one step: every ghost slot a real cell pulls receives its face value
struct KbcFillArgs {
  float* f;                 // populations in (real + ghost blocks)
  const uint2* entries;     // (block, cell | k << 9) of the pulls whose source is a ghost cell
  int64_t n;
  const int32_t* nbr;
  const int4* binfo;
  kbc::FaceParams F;
  float feq_inlet[Q];
};
constexpr uint32_t kNearSolid = 1u << 1;  // BF_NEAR_SOLID of the geometry

// pair index of direction k > 0 (k and opp(k) share it)
__host__ __device__ constexpr int kpair(int k) {
  constexpr int t[Q] = {-1, 0, 0, 1, 1, 2, 2, 3, 4, 5, 6, 6, 5, 4, 3, 7, 7, 8, 8, 9,
                        9, 10, 11, 11, 10, 12, 13, 13, 12, 14, 15, 15, 14, 16, 16, 17, 17, 18, 18};
  return t[k];
}
constexpr bool pairs_ok() {
  for (int k = 1; k < Q; ++k) {
    if (kpair(k) != kpair(kopp(k)) || kopp(k) == k || kpair(k) < 0 || kpair(k) >= 19) return false;
    for (int j = 1; j < Q; ++j)
      if (j != k && j != kopp(k) && kpair(j) == kpair(k)) return false;
  }
  return kopp(0) == 0;
}
static_assert(pairs_ok(), "pair table");

// Julia's max(x, C) for a constant C that is not NaN: a NaN x stays NaN
__device__ __forceinline__ float maxc(float x, float c) { return x < c ? c : x; }

// Per-CTA tables, built at launch with runtime float arithmetic (the operations of the CPU
// restatement): the 12 basis values of the 13-moment solve and the weight per direction, the pair
// slot of h_k and its sign, and the direction itself.
constexpr int NP = 19;     // direction pairs (k, opp k); slot NP holds the rest direction's h = 0
constexpr int NSLOT = NP + 1;
struct Tables {
  float4 b[Q][4];  // [0..11] basis (cx, cy, cz, cx^2-cs2, cy^2-cs2, cz^2-cs2, cxcy, cxcz, cycz,
                   // cx efl, cy efl, cz efl), [12] weight
  int32_t ps[Q];   // h slot | 0x100 when h_k = -h_slot | 0x200 when k is the first of its pair
  int32_t c[Q];    // (cx + 3) | (cy + 3) << 4 | (cz + 3) << 8 | opp(k) << 12
};

__device__ __forceinline__ void build_tables(Tables& T) {
  for (int k = threadIdx.x; k < Q; k += blockDim.x) {
    int cxi = 0, cyi = 0, czi = 0, opp = 0, pair = 0;
    // lattice.jl:177-262 in order, 0-based
#pragma unroll
    for (int i = 0; i < Q; ++i)
      if (i == k) { cxi = kcx(i); cyi = kcy(i); czi = kcz(i); opp = kopp(i); pair = kpair(i); }
    const float cx = float(cxi) - 0.0f, cy = float(cyi) - 0.0f, cz = float(czi) - 0.0f;
    const float efl = (cx * cx + cy * cy + cz * cz) - 5.0f * CS2;
    float* r = reinterpret_cast<float*>(T.b[k]);
    r[0] = cx; r[1] = cy; r[2] = cz;
    r[3] = cx * cx - CS2; r[4] = cy * cy - CS2; r[5] = cz * cz - CS2;
    r[6] = cx * cy; r[7] = cx * cz; r[8] = cy * cz;
    r[9] = cx * efl; r[10] = cy * efl; r[11] = cz * efl;
    r[12] = k < 7 ? float(1.0 / 12) : k < 15 ? float(1.0 / 27) : k < 21 ? float(2.0 / 135) : k < 33 ? float(1.0 / 432)
                                                                                               : float(1.0 / 1620);
    r[13] = 1.0f / r[12];  // inverse weight (the fast path's entropy sums)
    r[14] = r[15] = 0.0f;
    T.ps[k] = k == 0 ? (NP | 0x200) : (pair | (opp < k ? 0x100 : 0x200));
    T.c[k] = (cxi + 3) | ((cyi + 3) << 4) | ((czi + 3) << 8) | (opp << 12);
  }
}

// exp argument la0 + la1 b0 + ... + la12 b11 of one direction (physics_utils.jl:589-593), every
// term written out in the reference's order
template <bool FAST = false>
__device__ __forceinline__ float lda_row(const float (&la)[13], const float4* row) {
  const float4 r0 = row[0], r1 = row[1], r2 = row[2];
  if constexpr (FAST) {
    float l = __fmaf_rn(la[1], r0.x, la[0]);
    l = __fmaf_rn(la[2], r0.y, l); l = __fmaf_rn(la[3], r0.z, l); l = __fmaf_rn(la[4], r0.w, l);
    l = __fmaf_rn(la[5], r1.x, l); l = __fmaf_rn(la[6], r1.y, l); l = __fmaf_rn(la[7], r1.z, l);
    l = __fmaf_rn(la[8], r1.w, l); l = __fmaf_rn(la[9], r2.x, l); l = __fmaf_rn(la[10], r2.y, l);
    l = __fmaf_rn(la[11], r2.z, l);
    return __fmaf_rn(la[12], r2.w, l);
  }
  float l = la[0] + la[1] * r0.x;
  l = l + la[2] * r0.y;
  l = l + la[3] * r0.z;
  l = l + la[4] * r0.w;
  l = l + la[5] * r1.x;
  l = l + la[6] * r1.y;
  l = l + la[7] * r1.z;
  l = l + la[8] * r1.w;
  l = l + la[9] * r2.x;
  l = l + la[10] * r2.y;
  l = l + la[11] * r2.z;
  l = l + la[12] * r2.w;
  return l;
}
// max(rho w_k exp(clamp(lda)), 1e-15) (physics_utils.jl:594, 759-760)
template <bool FAST = false>
__device__ __forceinline__ float fi_row(float rho, const float (&la)[13], const float4* row) {
  return maxc(rho * row[3].x * kexp<FAST>(jclamp(lda_row<FAST>(la, row), -20.0f, 20.0f)), 1e-15f);
}

// ---- the fast path's Newton pass in raw moments of the direction pairs ------------------------
// A full Newton step needs f_k = rho w_k exp(lda_k) of the 39 directions, their 13 moments and the
// Hessian of the dual problem, H = sum_k f_k b_k b_k^T. Run over a basis table (one exponential, 12
// multiply-adds and 104 accumulations per direction) that is ~5,200 instructions. Here the sums use
// what the lattice is: in the unshifted basis (1, c, c_a^2, c_a c_b, |c|^2 c_a) every entry of H is
// a raw moment, a raw moment needs only the even part f_k + f_opp or the odd part f_k - f_opp of a
// pair, all but a few of the 19 pairs contribute with integer factors or not at all, and the 91
// entries are 44 different moments. lda_k = E +- O splits the same way. Everything is unrolled over
// the pairs (compile-time velocities), ~600 instructions per pass, the populations in registers.
// Newton steps do not depend on the basis; multipliers, targets and the residual test stay in the
// shifted basis of the reference (la[0..12]).
// Measured: see k_kbc_step.

// first direction (positive leading component) of each pair, in the order the moments below use
__host__ __device__ constexpr int kpos(int p) {
  constexpr int t[19] = {2, 4, 6, 14, 13, 12, 11, 16, 18, 20, 24, 23, 28, 27, 32, 31, 34, 36, 38};
  return t[p];
}
constexpr bool kpos_ok() {
  for (int p = 0; p < 19; ++p) {
    const int k = kpos(p);
    const int lead = kcx(k) != 0 ? kcx(k) : kcy(k) != 0 ? kcy(k) : kcz(k);
    if (lead <= 0 || kopp(kopp(k)) != k) return false;
    for (int q = 0; q < p; ++q)
      if (kpos(q) == k || kopp(kpos(q)) == k) return false;
  }
  return true;
}
static_assert(kpos_ok(), "pair order");
__host__ __device__ constexpr int kc2(int k) { return kcx(k) * kcx(k) + kcy(k) * kcy(k) + kcz(k) * kcz(k); }
__host__ __device__ constexpr int kfam(int k) {  // the five shells |c|^2 = 1, 3, 4, 8, 9
  return kc2(k) == 1 ? 0 : kc2(k) == 3 ? 1 : kc2(k) == 4 ? 2 : kc2(k) == 8 ? 3 : 4;
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// f_k = rho w_k exp(lda_k) at the multipliers la; false when some |lda_k| may exceed 20, where the
// reference clamps it (the caller then takes the table path, which clamps)
__device__ __forceinline__ bool eq_pops(float rho, const float (&la)[13], float (&f)[Q]) {
  constexpr float L2E = 1.44269504088896341f, TEN3 = 5.0f * CS2;
  // unshifted multipliers, in units of log 2
  const float l0 = L2E * __fmaf_rn(-CS2, (la[4] + la[5]) + la[6], la[0]);
  float g1[3], q[3], m2[3], mx[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    g1[a] = L2E * __fmaf_rn(-TEN3, la[10 + a], la[1 + a]);
    q[a] = L2E * la[10 + a];
    m2[a] = L2E * la[4 + a];
    mx[a] = L2E * la[7 + a];
  }
  // |lda| <= |l0| + 9 |m2| + 4 |mx| + 3 |g1| + 27 |q| over the directions
  const float bound = fabsf(l0) + 9.0f * (fabsf(m2[0]) + fabsf(m2[1]) + fabsf(m2[2])) +
                      4.0f * (fabsf(mx[0]) + fabsf(mx[1]) + fabsf(mx[2])) +
                      3.0f * (fabsf(g1[0]) + fabsf(g1[1]) + fabsf(g1[2])) +
                      27.0f * (fabsf(q[0]) + fabsf(q[1]) + fabsf(q[2]));
  if (!(bound <= 20.0f * L2E)) return false;
  float g[5][3];
  constexpr float c2f[5] = {1.0f, 3.0f, 4.0f, 8.0f, 9.0f};
#pragma unroll
  for (int s = 0; s < 5; ++s)
#pragma unroll
    for (int a = 0; a < 3; ++a) g[s][a] = __fmaf_rn(c2f[s], q[a], g1[a]);
  f[0] = rho * kw(0) * ex2(l0);
#pragma unroll
  for (int p = 0; p < 19; ++p) {
    const int k = kpos(p), kb = kopp(k), s = kfam(k);
    const int c[3] = {kcx(k), kcy(k), kcz(k)};
    float E = l0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (c[a] != 0) E = __fmaf_rn(float(c[a] * c[a]), m2[a], E);
    if (c[0] * c[1] != 0) E = __fmaf_rn(float(c[0] * c[1]), mx[0], E);
    if (c[0] * c[2] != 0) E = __fmaf_rn(float(c[0] * c[2]), mx[1], E);
    if (c[1] * c[2] != 0) E = __fmaf_rn(float(c[1] * c[2]), mx[2], E);
    float O = 0.0f;
    bool first = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (c[a] != 0) {
        O = first ? float(c[a]) * g[s][a] : __fmaf_rn(float(c[a]), g[s][a], O);
        first = false;
      }
    const float rw = rho * kw(k);
    f[k] = rw * ex2(E + O);
    f[kb] = rw * ex2(E - O);
  }
  return true;
}

// the even and odd pair sums by shell: 1 = (1,0,0), T = (1,1,1), 2 = (2,0,0), D = (2,2,0), 3 = (3,0,0)
struct PairSums {
  float n0;
  float e1[3], t[4], e2[3], d[3][2], e3[3];  // f_k + f_opp; d: planes xy, xz, yz, signs (+,+) and (+,-)
  float o1[3], u[4], o2[3], w[3][2], o3[3];  // f_k - f_opp
};
__device__ __forceinline__ void pair_sums(const float (&f)[Q], PairSums& S) {
  S.n0 = f[0];
  auto pr = [&](int p, float& e, float& o) {
    const int k = kpos(p), kb = kopp(k);
    e = f[k] + f[kb];
    o = f[k] - f[kb];
  };
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    pr(a, S.e1[a], S.o1[a]);
    pr(7 + a, S.e2[a], S.o2[a]);
    pr(16 + a, S.e3[a], S.o3[a]);
    pr(10 + 2 * a, S.d[a][0], S.w[a][0]);
    pr(11 + 2 * a, S.d[a][1], S.w[a][1]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) pr(3 + i, S.t[i], S.u[i]);
}

// One Newton pass at populations f: the residual r of the raw moments (targets: rho, u with
// P_ab = rho (u_a u_b + cs2 delta), Q_a = rho u_a (u^2 + 5 cs2)); returns its square norm in the
// reference's shifted basis. hess(): the raw-moment Hessian, packed as newton_solve takes it.
struct NewtonPass {
  PairSums S;
  float T, XY[3], DXY[3], Bx[3], Qt[3], A[3], Axyz, W[3][2];
  float M2[3], Mx[3];
  __device__ __forceinline__ float residual(const float (&f)[Q], float rho, float ux, float uy, float uz, float (&r)[13]) {
    pair_sums(f, S);
    T = (S.t[0] + S.t[1]) + (S.t[2] + S.t[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      XY[i] = S.d[i][0] + S.d[i][1];
      DXY[i] = S.d[i][0] - S.d[i][1];
      W[i][0] = S.w[i][0] + S.w[i][1];  // odd (2,2,0) sums: first axis of the plane,
      W[i][1] = S.w[i][0] - S.w[i][1];  // second axis
    }
    // planes xy, xz, yz: axis a lies in two of them
    Bx[0] = XY[0] + XY[1]; Bx[1] = XY[0] + XY[2]; Bx[2] = XY[1] + XY[2];
    const float t01 = S.t[0] + S.t[1], t23 = S.t[2] + S.t[3], t02 = S.t[0] + S.t[2], t13 = S.t[1] + S.t[3];
    Qt[0] = t01 - t23;                                // xy signs + + - -
    Qt[1] = t02 - t13;                                // xz       + - + -
    Qt[2] = (S.t[0] + S.t[3]) - (S.t[1] + S.t[2]);    // yz       + - - +
    A[0] = (S.u[0] + S.u[1]) + (S.u[2] + S.u[3]);
    A[1] = (S.u[0] + S.u[1]) - (S.u[2] + S.u[3]);
    A[2] = (S.u[0] + S.u[2]) - (S.u[1] + S.u[3]);
    Axyz = (S.u[0] + S.u[3]) - (S.u[1] + S.u[2]);
#pragma unroll
    for (int a = 0; a < 3; ++a) M2[a] = __fmaf_rn(9.0f, S.e3[a], __fmaf_rn(4.0f, S.e2[a] + Bx[a], S.e1[a] + T));
#pragma unroll
    for (int i = 0; i < 3; ++i) Mx[i] = __fmaf_rn(4.0f, DXY[i], Qt[i]);
    const float M0 = ((S.n0 + T) + ((S.e1[0] + S.e1[1]) + S.e1[2])) + (((S.e2[0] + S.e2[1]) + S.e2[2]) +
                     ((XY[0] + XY[1]) + XY[2])) + ((S.e3[0] + S.e3[1]) + S.e3[2]);
    const float V[3] = {W[0][0] + W[1][0], W[0][1] + W[2][0], W[1][1] + W[2][1]};  // odd (2,2,0) sums with c_a
    float j[3], qm[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      j[a] = __fmaf_rn(3.0f, S.o3[a], __fmaf_rn(2.0f, S.o2[a] + V[a], S.o1[a] + A[a]));
      qm[a] = __fmaf_rn(27.0f, S.o3[a], __fmaf_rn(16.0f, V[a], __fmaf_rn(8.0f, S.o2[a], __fmaf_rn(3.0f, A[a], S.o1[a]))));
    }
    const float u[3] = {ux, uy, uz};
    const float usq = ux * ux + uy * uy + uz * uz;
    r[0] = rho - M0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      r[1 + a] = rho * u[a] - j[a];
      r[4 + a] = rho * __fmaf_rn(u[a], u[a], CS2) - M2[a];
      r[10 + a] = rho * u[a] * (usq + 5.0f * CS2) - qm[a];
    }
    r[7] = rho * ux * uy - Mx[0];
    r[8] = rho * ux * uz - Mx[1];
    r[9] = rho * uy * uz - Mx[2];
    m0 = M0; jm[0] = j[0]; jm[1] = j[1]; jm[2] = j[2]; qmom[0] = qm[0]; qmom[1] = qm[1]; qmom[2] = qm[2];
    float res = r[0] * r[0];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float s2 = __fmaf_rn(-CS2, r[0], r[4 + a]), sq = __fmaf_rn(-5.0f * CS2, r[1 + a], r[10 + a]);
      res = __fmaf_rn(r[1 + a], r[1 + a], res);
      res = __fmaf_rn(s2, s2, res);
      res = __fmaf_rn(r[7 + a], r[7 + a], res);
      res = __fmaf_rn(sq, sq, res);
    }
    return res;
  }
  float m0, jm[3], qmom[3];
  // unknowns: 0: 1; 1-3: c; 4-6: c_a^2; 7-9: c_x c_y, c_x c_z, c_y c_z; 10-12: |c|^2 c
  __device__ __forceinline__ void hess(float (&H)[91]) const {
    auto at = [&](int i, int j2) -> float& { return i >= j2 ? H[i * (i + 1) / 2 + j2] : H[j2 * (j2 + 1) / 2 + i]; };
    // plane index of axes (a, b) and the cross moments' positions
    constexpr int pl[3][3] = {{-1, 0, 1}, {0, -1, 2}, {1, 2, -1}};
    at(0, 0) = m0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      at(1 + a, 0) = jm[a];
      at(4 + a, 0) = M2[a];
      at(7 + a, 0) = Mx[a];
      at(10 + a, 0) = qmom[a];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // c_a c_a, c_a^2 c_a^2, |c|^2 c_a c_a, |c|^4 c_a c_a
      at(1 + a, 1 + a) = M2[a];
      at(4 + a, 4 + a) = __fmaf_rn(81.0f, S.e3[a], __fmaf_rn(16.0f, S.e2[a] + Bx[a], S.e1[a] + T));
      at(10 + a, 1 + a) = __fmaf_rn(81.0f, S.e3[a], __fmaf_rn(32.0f, Bx[a], __fmaf_rn(16.0f, S.e2[a], __fmaf_rn(3.0f, T, S.e1[a]))));
      at(10 + a, 10 + a) = __fmaf_rn(729.0f, S.e3[a], __fmaf_rn(256.0f, Bx[a], __fmaf_rn(64.0f, S.e2[a], __fmaf_rn(9.0f, T, S.e1[a]))));
      // odd: c_a^2 c_a and c_a^2 |c|^2 c_a
      const float V = a == 0 ? W[0][0] + W[1][0] : a == 1 ? W[0][1] + W[2][0] : W[1][1] + W[2][1];
      at(4 + a, 1 + a) = __fmaf_rn(27.0f, S.o3[a], __fmaf_rn(8.0f, S.o2[a] + V, S.o1[a] + A[a]));
      at(10 + a, 4 + a) = __fmaf_rn(243.0f, S.o3[a], __fmaf_rn(64.0f, V, __fmaf_rn(32.0f, S.o2[a], __fmaf_rn(3.0f, A[a], S.o1[a]))));
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (a == b) continue;
        const int p = pl[a][b];
        if (b < a) {
          at(1 + a, 1 + b) = Mx[p];
          at(4 + a, 4 + b) = __fmaf_rn(16.0f, XY[p], T);                       // c_a^2 c_b^2
          at(10 + a, 10 + b) = __fmaf_rn(256.0f, DXY[p], 9.0f * Qt[p]);        // |c|^4 c_a c_b
          at(7 + p, 7 + p) = at(4 + a, 4 + b);
        }
        at(10 + a, 1 + b) = __fmaf_rn(32.0f, DXY[p], 3.0f * Qt[p]);            // |c|^2 c_a c_b
        // (2,2,0) odd sum of plane p with c_a: first axis W[p][0], second W[p][1]
        const float wa = a < b ? W[p][0] : W[p][1];
        const float aab = __fmaf_rn(8.0f, wa, A[a]), aabq = __fmaf_rn(64.0f, wa, 3.0f * A[a]);
        at(4 + b, 1 + a) = aab;                                                // c_b^2 c_a
        at(10 + a, 4 + b) = aabq;                                              // c_b^2 |c|^2 c_a
        // c_a c_b times c_b gives c_b^2 c_a
        at(7 + p, 1 + b) = aab;
        at(10 + b, 7 + p) = aabq;
        at(7 + p, 4 + a) = __fmaf_rn(16.0f, DXY[p], Qt[p]);                    // c_a^3 c_b
      }
    // entries with all three axes: only the (1,1,1) shell
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int p = a == 0 ? 2 : a == 1 ? 1 : 0;  // the plane without axis a
      at(7 + p, 1 + a) = Axyz;
      at(10 + a, 7 + p) = 3.0f * Axyz;
      at(7 + p, 4 + a) = Qt[p];                   // c_a^2 c_b c_c
    }
    at(8, 7) = Qt[2];  // c_x^2 c_y c_z
    at(9, 7) = Qt[1];  // c_x c_y^2 c_z
    at(9, 8) = Qt[0];  // c_x c_y c_z^2
  }
};

// Solves H x = r in place (r becomes x) by a Cholesky factorisation of the packed H; false when
// H is not numerically positive definite.
__device__ __forceinline__ bool newton_solve(float (&H)[91], float (&r)[13]) {
  float inv[13];
#pragma unroll
  for (int j = 0; j < 13; ++j) {
    float s = H[j * (j + 1) / 2 + j];
#pragma unroll
    for (int k = 0; k < j; ++k) s = __fmaf_rn(-H[j * (j + 1) / 2 + k], H[j * (j + 1) / 2 + k], s);
    if (!(s > 0.0f)) return false;
    inv[j] = rsqrtf(s);
#pragma unroll
    for (int i = j + 1; i < 13; ++i) {
      float t = H[i * (i + 1) / 2 + j];
#pragma unroll
      for (int k = 0; k < j; ++k) t = __fmaf_rn(-H[i * (i + 1) / 2 + k], H[j * (j + 1) / 2 + k], t);
      H[i * (i + 1) / 2 + j] = t * inv[j];
    }
  }
#pragma unroll
  for (int i = 0; i < 13; ++i) {
    float t = r[i];
#pragma unroll
    for (int k = 0; k < i; ++k) t = __fmaf_rn(-H[i * (i + 1) / 2 + k], r[k], t);
    r[i] = t * inv[i];
  }
#pragma unroll
  for (int i = 12; i >= 0; --i) {
    float t = r[i];
#pragma unroll
    for (int k = i + 1; k < 13; ++k) t = __fmaf_rn(-H[k * (k + 1) / 2 + i], r[k], t);
    r[i] = t * inv[i];
  }
  return true;
}

// physics_utils.jl:493-736: 13 multipliers by block-Jacobi Newton sweeps, warm-started from the
// cached multipliers when they pass the staleness gate. The fast path solves the same moment
// equations to the same residual tolerance by full Newton steps first (one or two from a warm
// start), keeping the sweeps as its fallback.
template <bool FAST = false>
__device__ __forceinline__ void solve_lambdas(const Tables& T, float rho, float ux, float uy, float uz, float (&la)[13],
                                              float (&fe)[FAST ? Q : 1], float warm_gate = 100.0f) {
  const float OMEGA = 1.5f, F_FLOOR_EQ = 1e-15f;
  const float eps = 1.1920928955078125e-7f;
  const float TOL_SQ = 507.0f * eps * eps * rho * rho * (FAST ? KBC_FAST_TOL_SCALE : 1.0f);
  const float eR = CS2;
  const float usq = ux * ux + uy * uy + uz * uz;
  const float dT = 1.0f - 1.0f;
  const float ef = usq + 5.0f * eR * dT;
  float mt[13];
  mt[0] = rho; mt[1] = rho * ux; mt[2] = rho * uy; mt[3] = rho * uz;
  mt[4] = rho * (ux * ux + eR * dT); mt[5] = rho * (uy * uy + eR * dT); mt[6] = rho * (uz * uz + eR * dT);
  mt[7] = rho * ux * uy; mt[8] = rho * ux * uz; mt[9] = rho * uy * uz;
  mt[10] = rho * ux * ef; mt[11] = rho * uy * ef; mt[12] = rho * uz * ef;
  const float inv_cs2 = 1.0f / CS2, inv_cs4 = inv_cs2 * inv_cs2;
  auto poly_start = [&]() {
    la[0] = -0.5f * usq * inv_cs2; la[1] = ux * inv_cs2; la[2] = uy * inv_cs2; la[3] = uz * inv_cs2;
    la[4] = 0.5f * inv_cs4 * ux * ux; la[5] = 0.5f * inv_cs4 * uy * uy; la[6] = 0.5f * inv_cs4 * uz * uz;
    la[7] = inv_cs4 * ux * uy; la[8] = inv_cs4 * ux * uz; la[9] = inv_cs4 * uy * uz;
    la[10] = 0.0f; la[11] = 0.0f; la[12] = 0.0f;
  };
  if constexpr (FAST) {
    bool cold = la[0] != la[0];
    if (cold) poly_start();
    for (int it = 0; it < KBC_NEWTON_MAX; ++it) {
      const bool held = eq_pops(rho, la, fe);
      NewtonPass np;
      float r[13], res = 0.0f;
      if (held) {
        res = np.residual(fe, rho, ux, uy, uz, r);
        if (res < TOL_SQ) return;
      }
      if (!held || (!cold && it == 0 && res > warm_gate * TOL_SQ)) {
        // staleness gate on the warm start (physics_utils.jl:603-634): a stale one, and one with some
        // |lda| that may exceed 20, gives way to the polynomial start; the sweeps, which clamp, take over
        // where that one leaves the range too
        const bool warm = !cold;
        poly_start();
        cold = true;
        if (warm) continue;
        break;
      }
      float H[91];
      np.hess(H);
      if (!newton_solve(H, r)) break;
      // back to the shifted basis of la
      r[0] = __fmaf_rn(CS2, (r[4] + r[5]) + r[6], r[0]);
#pragma unroll
      for (int a = 0; a < 3; ++a) r[1 + a] = __fmaf_rn(5.0f * CS2, r[10 + a], r[1 + a]);
#pragma unroll
      for (int m = 0; m < 13; ++m) la[m] += jclamp(r[m], -2.0f, 2.0f);
    }
  } else if (la[0] != la[0]) {
    poly_start();
  } else {
    // staleness gate (physics_utils.jl:603-634)
    float gd[13];
#pragma unroll
    for (int m = 0; m < 13; ++m) gd[m] = 0.0f;
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const float4* row = T.b[k];
      const float fi = fi_row<FAST>(rho, la, row);
      const float4 r0 = row[0], r1 = row[1], r2 = row[2];
      gd[0] += fi;
      gd[1] += fi * r0.x; gd[2] += fi * r0.y; gd[3] += fi * r0.z; gd[4] += fi * r0.w;
      gd[5] += fi * r1.x; gd[6] += fi * r1.y; gd[7] += fi * r1.z; gd[8] += fi * r1.w;
      gd[9] += fi * r2.x; gd[10] += fi * r2.y; gd[11] += fi * r2.z; gd[12] += fi * r2.w;
    }
    float gres = 0.0f;
#pragma unroll
    for (int m = 0; m < 13; ++m) gres += (mt[m] - gd[m]) * (mt[m] - gd[m]);
    if (gres > (FAST ? warm_gate : 100.0f) * TOL_SQ) poly_start();
  }
  auto upd = [&](int m, float d, float j) {
    la[m] += j > F_FLOOR_EQ ? jclamp(OMEGA * (mt[m] - d) / j, -2.0f, 2.0f) : 0.0f;
  };
  for (int sweep = 0; sweep < (FAST ? KBC_FAST_MAX_SWEEPS : 200); ++sweep) {
    float d[13], j[13];
#pragma unroll
    for (int m = 0; m < 13; ++m) { d[m] = 0.0f; j[m] = 0.0f; }
#pragma unroll 3
    for (int k = 0; k < Q; ++k) {
      const float4* row = T.b[k];
      const float fi = fi_row<FAST>(rho, la, row);
      const float4 r0 = row[0];
      d[0] += fi; j[0] += fi;
      d[1] = kmad<FAST>(fi, r0.x, d[1]); j[1] = kmad<FAST>(fi * r0.x, r0.x, j[1]);
      d[2] = kmad<FAST>(fi, r0.y, d[2]); j[2] = kmad<FAST>(fi * r0.y, r0.y, j[2]);
      d[3] = kmad<FAST>(fi, r0.z, d[3]); j[3] = kmad<FAST>(fi * r0.z, r0.z, j[3]);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) upd(m, d[m], j[m]);
#pragma unroll 3
    for (int k = 0; k < Q; ++k) {
      const float4* row = T.b[k];
      const float fi = fi_row<FAST>(rho, la, row);
      const float4 r0 = row[0], r1 = row[1], r2 = row[2];
      d[4] = kmad<FAST>(fi, r0.w, d[4]); j[4] = kmad<FAST>(fi * r0.w, r0.w, j[4]);
      d[5] = kmad<FAST>(fi, r1.x, d[5]); j[5] = kmad<FAST>(fi * r1.x, r1.x, j[5]);
      d[6] = kmad<FAST>(fi, r1.y, d[6]); j[6] = kmad<FAST>(fi * r1.y, r1.y, j[6]);
      d[7] = kmad<FAST>(fi, r1.z, d[7]); j[7] = kmad<FAST>(fi * r1.z, r1.z, j[7]);
      d[8] = kmad<FAST>(fi, r1.w, d[8]); j[8] = kmad<FAST>(fi * r1.w, r1.w, j[8]);
      d[9] = kmad<FAST>(fi, r2.x, d[9]); j[9] = kmad<FAST>(fi * r2.x, r2.x, j[9]);
    }
#pragma unroll
    for (int m = 4; m < 10; ++m) upd(m, d[m], j[m]);
#pragma unroll 3
    for (int k = 0; k < Q; ++k) {
      const float4* row = T.b[k];
      const float fi = fi_row<FAST>(rho, la, row);
      const float4 r2 = row[2];
      d[10] = kmad<FAST>(fi, r2.y, d[10]); j[10] = kmad<FAST>(fi * r2.y, r2.y, j[10]);
      d[11] = kmad<FAST>(fi, r2.z, d[11]); j[11] = kmad<FAST>(fi * r2.z, r2.z, j[11]);
      d[12] = kmad<FAST>(fi, r2.w, d[12]); j[12] = kmad<FAST>(fi * r2.w, r2.w, j[12]);
    }
#pragma unroll
    for (int m = 10; m < 13; ++m) upd(m, d[m], j[m]);
    float res = 0.0f;
#pragma unroll
    for (int m = 0; m < 13; ++m) res += (mt[m] - d[m]) * (mt[m] - d[m]);
    if (res < TOL_SQ) break;
  }
  if constexpr (FAST) {
#pragma unroll
    for (int k = 0; k < Q; ++k) fe[k] = fi_row<FAST>(rho, la, T.b[k]);
  }
}

// The mass-corrected equilibrium, kept as its multipliers: f_eq_k = corr * fi_k
// (physics_utils.jl:738-795, kernel_entropic_d3q39.jl:2365-2385)
template <bool FAST = false>
struct Eq {
  float la[13];
  float rho, corr;
  __device__ __forceinline__ float operator()(const Tables& T, int k) const { return corr * fi_row<FAST>(rho, la, T.b[k]); }
};

// HRR blend of the stress part (kernel_entropic_d3q39.jl:2991-3034); k and opp(k) give the same s_fd
struct Hrr {
  int on;
  float sigma, oms, pxx, pyy, pzz, pxy, pxz, pyz;
};
__device__ __forceinline__ float hrr_s(const Tables& T, float s, int k, const Hrr& hr) {
  if (!hr.on) return s;
  const float4 r0 = T.b[k][0];
  const float cx = r0.x, cy = r0.y, cz = r0.z;
  const float Qxx = cx * cx - CS2, Qyy = cy * cy - CS2, Qzz = cz * cz - CS2;
  const float Qxy = cx * cy, Qxz = cx * cz, Qyz = cy * cz;
  const float contraction = Qxx * hr.pxx + Qyy * hr.pyy + Qzz * hr.pzz + 2.0f * (Qxy * hr.pxy + Qxz * hr.pxz + Qyz * hr.pyz);
  const float s_fd = T.b[k][3].x * contraction * (0.5f / (CS2 * CS2));
  return hr.sigma * s + hr.oms * s_fd;
}

// After the split the thread's population column holds a_k = f_eq_k + coeff_s s_k and its h column
// one value per pair (h_opp(k) = -h_k, the rest direction's h in the last slot): the post-collision
// population is a_k + coeff_h h_k, the intermediate the reference forms (:113-133, 3163-3176).
__device__ __forceinline__ float h_at(const Tables& T, const float* sh, int k) {
  const int ps = T.ps[k];
  const float h = sh[(ps & 0xff) * kThreads];
  return (ps & 0x100) ? -h : h;
}

// kernel_entropic_d3q39.jl:113-133
template <bool FAST = false>
__device__ __forceinline__ float entropy_ah(const Tables& T, const float* sa, const float* sh, float coeff_h) {
  float H = 0.0f;
#pragma unroll 3
  for (int k = 0; k < Q; ++k) {
    float fk = sa[k * kThreads] + coeff_h * h_at(T, sh, k);
    fk = maxc(fk, F_FLOOR);
    H = kmad<FAST>(fk, safe_log<FAST>(FAST ? fk * T.b[k][3].y : fk / T.b[k][3].x), H);
  }
  return H;
}

// kernel_entropic_d3q39.jl:417-442: the lower and upper brackets, then up to max_iter midpoints,
// through one entropy evaluation site
template <bool FAST = false>
__device__ __forceinline__ float alpha_bisection(const Tables& T, const float* sa, const float* sh, float beta,
                                                 float H_pre, int max_iter) {
  const float inv_2beta = 0.5f / jmax(beta, 0.01f);
  float lo = jmax(inv_2beta - 0.1f, 0.1f), hi = jmax(inv_2beta + 3.0f, 4.0f);
  float H_lo = 0.0f;
  for (int it = -2; it < max_iter; ++it) {
    const float al = it == -2 ? lo : it == -1 ? hi : 0.5f * (lo + hi);
    const float H = entropy_ah<FAST>(T, sa, sh, 1.0f - 2.0f * beta * al);
    if (it == -2) { H_lo = H; continue; }
    if (it == -1) {
      if (!((H_lo - H_pre) * (H - H_pre) < 0.0f)) return inv_2beta;
      continue;
    }
    if ((H - H_pre) * (H_lo - H_pre) > 0.0f) { lo = al; H_lo = H; } else { hi = al; }
    if ((hi - lo) < 0.005f * (inv_2beta + 1e-6f)) break;
  }
  return 0.5f * (lo + hi);
}

// kernel_entropic_d3q39.jl:444-462 with entropy_and_deriv_at_alpha_39_fused (:192-215)
template <bool FAST = false>
__device__ __forceinline__ float alpha_newton(const Tables& T, const float* sa, const float* sh, float beta, float H_pre) {
  float alpha = 2.0f;
  const float inv_2beta = 0.5f / jmax(beta, 0.01f);
  for (int it = 0; it < 8; ++it) {
    const float coeff_h = 1.0f - 2.0f * beta * alpha;
    float H = 0.0f, dH = 0.0f;
#pragma unroll 3
    for (int k = 0; k < Q; ++k) {
      const float hk = h_at(T, sh, k);
      float fk = sa[k * kThreads] + coeff_h * hk;
      fk = maxc(fk, F_FLOOR);
      const float lr = safe_log<FAST>(FAST ? fk * T.b[k][3].y : fk / T.b[k][3].x);
      H += fk * lr;
      dH += (-2.0f * beta * hk) * (1.0f + lr);
    }
    const float residual = H - H_pre;
    if (fabsf(residual) < 1e-5f) break;
    if (fabsf(dH) < 1e-12f) break;
    const float delta = residual / dH;
    alpha -= delta;
    alpha = jclamp(alpha, jmax(inv_2beta - 0.1f, 0.1f), 6.0f);
    if (fabsf(delta) < 1e-5f) break;
  }
  if (!(alpha > 0.0f)) alpha = inv_2beta;
  return alpha;
}

// kernel_entropic_d3q39.jl:481-528 without its bisection fallback (false: the cell's deviation needs
// the bisection); runs on the arriving populations before the split
template <bool FAST = false>
__device__ __forceinline__ bool alpha_taylor(const Tables& T, const float* sf, const Eq<FAST>& eq, float h_scale, const Hrr& hr,
                                             float beta, float& alpha) {
  auto fneq_of = [&](int k, float& fe) {
    const int kb = (T.c[k] >> 12) & 63;
    fe = eq(T, k);
    const float df = sf[k * kThreads] - fe, dfb = sf[kb * kThreads] - eq(T, kb);
    const float s = hrr_s(T, 0.5f * (df + dfb), k, hr);
    const float h = (0.5f * (df - dfb)) * h_scale;
    return s + h;
  };
  float dev = 0.0f;
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    float fe;
    const float fneq = fneq_of(k, fe);
    const float fk = maxc(fe + fneq, F_FLOOR);
    dev = jmax(dev, fabsf(fneq) / fk);
    if (dev > 0.01f) break;
  }
  const float inv_2beta = 0.5f / jmax(beta, 0.01f);
  if (dev < 1e-6f) { alpha = 2.0f; return true; }
  if (!(dev < 0.01f)) return false;
  float a1 = 0.0f, a2 = 0.0f, a3 = 0.0f, a4 = 0.0f;
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    float fe;
    const float t = fneq_of(k, fe);
    const float fk = maxc(fe + t, F_FLOOR);
    const float inv = 1.0f / fk;
    float p = t * t * inv; a1 += p;
    p *= t * inv; a2 += p;
    p *= t * inv; a3 += p;
    p *= t * inv; a4 += p;
  }
  a1 *= 0.5f; a2 *= -1.0f / 6.0f; a3 *= 1.0f / 12.0f; a4 *= -0.05f;
  if (fabsf(a1) > 1e-20f) {
    const float i1 = 1.0f / a1;
    const float al = 2.0f - 4.0f * a2 * i1 + 16.0f * a2 * a2 * i1 * i1 - 8.0f * a3 * i1 +
                     80.0f * a2 * a3 * i1 * i1 - 80.0f * a2 * a2 * a2 * i1 * i1 * i1 - 16.0f * a4 * i1;
    alpha = jclamp(al, inv_2beta, 6.0f);
  } else {
    alpha = 2.0f;
  }
  return true;
}

// ---- alpha of the fast path from a series of the entropy ---------------------------------------
// The bisection needs the sign of H(alpha) - H_pre, H = sum_k f_k ln(f_k / w_k), at 12 values of
// alpha. Near equilibrium that difference is ~1e-8 while the sums carry ~1e-7 of FP32 rounding, and
// each evaluation is 39 logarithms. With f_k = fe_k (1 + y_k) and ln(fe_k / w_k) = ln(rho corr) +
// lda_k, H splits into the multipliers times the moments of f - fe and sum fe g(y), g(y) = (1 + y)
// ln(1 + y) - y = y^2/2 - y^3/6 + y^4/12 - ...; f - fe = coeff_s s + coeff_h h with s even and h odd in
// the pair, so sum fe g(y) is a polynomial in coeff_h whose coefficients are 12 sums over the pairs,
// gathered once. Mass and momentum of s and h are zero (f_eq has the cell's), which leaves the stress
// moments of s and the energy-flux moments of h. The differences then come out of small quantities
// alone, and the 12 evaluations are a quartic each. The first dropped term is fe y^5 / 20 a direction: at
// |y| = kSeriesRoot 4e-8 for the light shells (w <= 1/432), a tenth of the rounding of the sums it
// replaces, and up to 1.3e-6 for the heaviest. The gate does not ask which shell carries the deviation;
// where the heavy ones do, up to the gate, the dropped terms move alpha by at most 2.5e-3 (median 1.3e-5,
// 4,096 cells against the logarithms in 64 bits), less than the bisection's last interval (3.5e-3). So the
// series decides where |y| stays below kSeriesRoot for |coeff_h| <= kRootReach and the root lies there,
// and below kSeriesFar over the whole bracket (|coeff_h| <= 7), whose far end only has to have the right
// sign; elsewhere the sums of logarithms decide.
constexpr float kSeriesRoot = 0.2f, kSeriesFar = 0.7f, kRootReach = 2.5f;
struct AlphaSeries {
  float a20 = 0.0f, a11 = 0.0f, a02 = 0.0f, a30 = 0.0f, a21 = 0.0f, a12 = 0.0f, a03 = 0.0f;
  float a40 = 0.0f, a31 = 0.0f, a22 = 0.0f, a13 = 0.0f, a04 = 0.0f;
  float P[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, qf[3] = {0.0f, 0.0f, 0.0f};
  float h_sq = 0.0f, y_root = 0.0f, y_far = 0.0f;  // the largest |y| bounds
  static __device__ __forceinline__ float rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
  }
  // the |y| bounds of the cell; true where they admit the series
  __device__ __forceinline__ bool admits(const float* sf, const float (&fe)[Q]) {
    y_root = y_far = fabsf(sf[0] - fe[0]) * rcp(fe[0]);
#pragma unroll
    for (int p = 0; p < 19; ++p) {
      const int k = kpos(p), kb = kopp(k);
      const float df = sf[k * kThreads] - fe[k], db = sf[kb * kThreads] - fe[kb];
      const float s = 0.5f * fabsf(df + db), h = 0.5f * fabsf(df - db), r = rcp(fminf(fe[k], fe[kb]));
      y_root = fmaxf(y_root, __fmaf_rn(kRootReach, h, s) * r);
      y_far = fmaxf(y_far, __fmaf_rn(7.0f, h, s) * r);
    }
    return y_root <= kSeriesRoot && y_far <= kSeriesFar;
  }
  __device__ __forceinline__ void gather(const float* sf, const float (&fe)[Q]) {
    {
      const float s = sf[0] - fe[0], y = s * rcp(fe[0]), s2 = s * y;
      a20 = s2;
      a30 = s2 * y;
      a40 = s2 * y * y;
    }
#pragma unroll
    for (int p = 0; p < 19; ++p) {
      const int k = kpos(p), kb = kopp(k);
      const float df = sf[k * kThreads] - fe[k], db = sf[kb * kThreads] - fe[kb];
      const float s = 0.5f * (df + db), h = 0.5f * (df - db);
      const float rp = rcp(fe[k]), rm = rcp(fe[kb]);
      const float s2 = s * s, sh = s * h, h2 = h * h;
      const float R1 = rp + rm, Q1 = rp - rm;
      a20 = __fmaf_rn(s2, R1, a20);
      a11 = __fmaf_rn(sh, Q1, a11);
      a02 = __fmaf_rn(h2, R1, a02);
      const float rp2 = rp * rp, rm2 = rm * rm;
      const float sR2 = s * (rp2 + rm2), hQ2 = h * (rp2 - rm2);
      a30 = __fmaf_rn(s2, sR2, a30);
      a21 = __fmaf_rn(s2, hQ2, a21);
      a12 = __fmaf_rn(h2, sR2, a12);
      a03 = __fmaf_rn(h2, hQ2, a03);
      const float rp3 = rp2 * rp, rm3 = rm2 * rm;
      const float s2R3 = s2 * (rp3 + rm3), h2R3 = h2 * (rp3 + rm3), shQ3 = sh * (rp3 - rm3);
      a40 = __fmaf_rn(s2, s2R3, a40);
      a31 = __fmaf_rn(s2, shQ3, a31);
      a22 = __fmaf_rn(h2, s2R3, a22);
      a13 = __fmaf_rn(h2, shQ3, a13);
      a04 = __fmaf_rn(h2, h2R3, a04);
      const int c[3] = {kcx(k), kcy(k), kcz(k)};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (c[a] != 0) P[a] = __fmaf_rn(2.0f * float(c[a] * c[a]), s, P[a]);
        if (c[a] != 0) qf[a] = __fmaf_rn(2.0f * float(kc2(k) * c[a]), h, qf[a]);
      }
      if (c[0] * c[1] != 0) P[3] = __fmaf_rn(2.0f * float(c[0] * c[1]), s, P[3]);
      if (c[0] * c[2] != 0) P[4] = __fmaf_rn(2.0f * float(c[0] * c[2]), s, P[4]);
      if (c[1] * c[2] != 0) P[5] = __fmaf_rn(2.0f * float(c[1] * c[2]), s, P[5]);
      h_sq = __fmaf_rn(2.0f, h2, h_sq);
    }
  }
  // kernel_entropic_d3q39.jl:417-442 and the clamp of :3144-3150 on the gathered series; false where
  // the root lies beyond its reach
  __device__ __forceinline__ bool solve(const float (&la)[13], float beta, float& alpha) const {
    alpha = 2.0f;
    if (!(h_sq > 1e-20f)) return true;
    const float cs = 1.0f - 2.0f * beta, cs2 = cs * cs, cs3 = cs2 * cs;
    float ls = 0.0f, lq = 0.0f;
#pragma unroll
    for (int i = 0; i < 6; ++i) ls = __fmaf_rn(la[4 + i], P[i], ls);
#pragma unroll
    for (int a = 0; a < 3; ++a) lq = __fmaf_rn(la[10 + a], qf[a], lq);
    // G(c) = H - H_pre at coeff_h = c, the arriving populations being coeff_s = coeff_h = 1
    const float pre = ((0.5f * a20 + a11) + 0.5f * a02) -
                      ((a30 * (1.0f / 6.0f) + 0.5f * a21) + (0.5f * a12 + a03 * (1.0f / 6.0f))) +
                      ((a40 * (1.0f / 12.0f) + a31 * (1.0f / 3.0f)) + (0.5f * a22 + a13 * (1.0f / 3.0f)) + a04 * (1.0f / 12.0f));
    const float c1 = cs * a11 - 0.5f * cs2 * a21 + cs3 * (1.0f / 3.0f) * a31 + lq;
    const float c2 = 0.5f * ((a02 - cs * a12) + cs2 * a22);
    const float c3 = cs * (1.0f / 3.0f) * a13 - (1.0f / 6.0f) * a03;
    const float c4 = (1.0f / 12.0f) * a04;
    const float c0 = (0.5f * cs2 * a20 - cs3 * (1.0f / 6.0f) * a30 + cs2 * cs2 * (1.0f / 12.0f) * a40) - pre +
                     ((cs - 1.0f) * ls - lq);
    auto G = [&](float al) {
      const float c = 1.0f - 2.0f * beta * al;
      return __fmaf_rn(c, __fmaf_rn(c, __fmaf_rn(c, __fmaf_rn(c, c4, c3), c2), c1), c0);
    };
    const float inv_2beta = 0.5f / fmaxf(beta, 0.01f);
    float lo = fmaxf(inv_2beta - 0.1f, 0.1f), hi = fmaxf(inv_2beta + 3.0f, 4.0f);
    const float G_lo = G(lo), G_hi = G(hi);
    alpha = inv_2beta;
    bool decided = y_far <= kSeriesRoot;
    if ((G_lo < 0.0f && G_hi > 0.0f) || (G_lo > 0.0f && G_hi < 0.0f)) {
      const bool neg = G_lo < 0.0f;
#pragma unroll 1
      for (int it = 0; it < 10; ++it) {
        const float al = 0.5f * (lo + hi), g = G(al);
        if (neg ? g < 0.0f : g > 0.0f) lo = al;
        else hi = al;
        if ((hi - lo) < 0.005f * (inv_2beta + 1e-6f)) break;
      }
      alpha = 0.5f * (lo + hi);
      decided = decided || fabsf(1.0f - 2.0f * beta * alpha) <= kRootReach;
    }
    if (!(alpha > 0.0f)) alpha = inv_2beta;
    alpha = jclamp(alpha, inv_2beta, 6.0f);
    return decided;
  }
};

// The bisection by sums of logarithms with the cell's a_k and h_p in registers (the fast path where
// the series does not decide): the evaluations of alpha_bisection unrolled, ~200 instructions each
// instead of ~550 over the shared columns, in units of log 2 (only signs of differences matter).
__device__ __forceinline__ float lg2(float v) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float entropy_term(float f, int k, float H) {
  const float fk = fmaxf(f, F_FLOOR);
  return __fmaf_rn(fk, lg2(fk * (1.0f / kw(k))), H);
}
__device__ __forceinline__ float entropy_regs(const float (&av)[Q], const float (&hv)[19], float c) {
  float H0 = entropy_term(av[0], 0, 0.0f), H1 = 0.0f;
#pragma unroll
  for (int p = 0; p < 19; ++p) {
    const int k = kpos(p), kb = kopp(k);
    H0 = entropy_term(__fmaf_rn(c, hv[p], av[k]), k, H0);
    H1 = entropy_term(__fmaf_rn(-c, hv[p], av[kb]), kb, H1);
  }
  return H0 + H1;
}
__device__ __forceinline__ float alpha_bisection_regs(const float (&av)[Q], const float (&hv)[19], float beta, float H_pre) {
  const float inv_2beta = 0.5f / fmaxf(beta, 0.01f);
  float lo = fmaxf(inv_2beta - 0.1f, 0.1f), hi = fmaxf(inv_2beta + 3.0f, 4.0f);
  float d_lo = 0.0f;
#pragma unroll 1
  for (int it = -2; it < 10; ++it) {
    const float al = it == -2 ? lo : it == -1 ? hi : 0.5f * (lo + hi);
    const float d = entropy_regs(av, hv, 1.0f - 2.0f * beta * al) - H_pre;
    if (it == -2) { d_lo = d; continue; }
    if (it == -1) {
      if (!(d_lo * d < 0.0f)) return inv_2beta;
      continue;
    }
    if (d * d_lo > 0.0f) lo = al;
    else hi = al;
    if ((hi - lo) < 0.005f * (inv_2beta + 1e-6f)) break;
  }
  return 0.5f * (lo + hi);
}

// The face fill (kernel_entropic_d3q39.jl:983-1278 at the default boundary options): one thread per
// pull whose source lies outside the domain; its value goes to the ghost slot the pull reads (the
// slot (source cell, k) has exactly one reader, the source + c_k).
__global__ void __launch_bounds__(256) k_kbc_fill(const KbcFillArgs a) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= a.n) return;
  const uint2 en = a.entries[e];
  const int b = (int)en.x, cell = (int)(en.y & 511u), k = (int)((en.y >> 9) & 63u);
  const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
  const int4 bi = a.binfo[b];
  const int gx = (bi.x - 1) * 8 + x + 1, gy = (bi.y - 1) * 8 + y + 1, gz = (bi.z - 1) * 8 + z + 1;
  const float v = kbc::face_value(a.F, a.f + (int64_t)b * Q * 512 + cell, 512, a.feq_inlet, k, gx, gy, gz);
  const int sx = x - kcx(k), sy = y - kcy(k), sz = z - kcz(k);
  const int ox = sx < 0 ? -1 : (sx > 7 ? 1 : 0), oy = sy < 0 ? -1 : (sy > 7 ? 1 : 0), oz = sz < 0 ? -1 : (sz > 7 ? 1 : 0);
  const int g = a.nbr[(int64_t)b * 27 + (ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)];
  a.f[((int64_t)g * Q + k) * 512 + ((sx & 7) | ((sy & 7) << 3) | ((sz & 7) << 6))] = v;
}

// Spectral vanishing viscosity inside the step (apply_svv_yz_d3q39_inline! and
// apply_svv_x_d3q39_inline!, kernel_svv_yz_d3q39.jl:142-213 and :252-298, frame shift 0): the
// post-collision f_k less eps times the 5-point bi-Laplacian of the step's INPUT populations along
// y and z (YZ) or along x, centred on f_k itself; a tap past a missing or ghost block or in a solid
// cell reads the cell's own input population (get_pop_neighbor_yz / _x, :78-116, 225-250). The
// 4-moment correction f_k -= w_k (drho + c_k . dj / cs2) then restores the cell's mass and momentum.
// the input populations and solid masks the taps read (passed by value: a reference to the
// kernel's argument block would copy the whole block to local memory)
struct SvvView {
  const float* fin;
  const int32_t* mslot;
  const uint32_t* cmask;
  int32_t nb;
};

// the direction-0 element of the input population at (x, y, z) + d (one axis), or `own`
__device__ __forceinline__ int64_t svv_tap_offset(const SvvView& v, const int32_t* s_nbr, int b, int x, int y, int z,
                                                  int dx, int dy, int dz, int64_t own) {
  const int nx = x + dx, ny = y + dy, nz = z + dz;
  const int ox = nx < 0 ? -1 : (nx > 7 ? 1 : 0), oy = ny < 0 ? -1 : (ny > 7 ? 1 : 0), oz = nz < 0 ? -1 : (nz > 7 ? 1 : 0);
  const int bo = (ox | oy | oz) == 0 ? b : s_nbr[(ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)];
  if (bo < 0 || bo >= v.nb) return own;
  const int c = (nx & 7) | ((ny & 7) << 3) | ((nz & 7) << 6);
  if (v.cmask) {
    const int32_t sl = v.mslot[bo];
    if (sl >= 0 && ((v.cmask[(int64_t)sl * 512 + c] >> 13) & 1u)) return own;
  }
  return (int64_t)bo * Q * 512 + c;
}

// the taps are resolved once per cell (neighbour block, solid masks, fall-back to the cell's own
// input population); each direction then reads them at + k 512
template <bool YZ>
__device__ __forceinline__ void svv_axis(const SvvView a, const Tables& T, const int32_t* s_nbr, int b, int cell,
                                         float eps, float* sf) {
  const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
  const int64_t own = (int64_t)b * Q * 512 + cell;
  constexpr int NT = YZ ? 8 : 4;
  int64_t off[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int s = (j & 3) < 2 ? (j & 3) - 2 : (j & 3) - 1;  // -2, -1, +1, +2
    off[j] = YZ ? (j < 4 ? svv_tap_offset(a, s_nbr, b, x, y, z, 0, s, 0, own) : svv_tap_offset(a, s_nbr, b, x, y, z, 0, 0, s, own))
                : svv_tap_offset(a, s_nbr, b, x, y, z, s, 0, 0, own);
  }
  float d_rho = 0.0f, d_jx = 0.0f, d_jy = 0.0f, d_jz = 0.0f;
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    const float* fk = a.fin + (int64_t)k * 512;
    const float fc = sf[k * kThreads];
    float ff;
    if (YZ) {
      const float by = fk[off[0]] - 4.0f * fk[off[1]] + 6.0f * fc - 4.0f * fk[off[2]] + fk[off[3]];
      const float bz = fk[off[4]] - 4.0f * fk[off[5]] + 6.0f * fc - 4.0f * fk[off[6]] + fk[off[7]];
      ff = fc - eps * (by + bz);
    } else {
      const float bx = fk[off[0]] - 4.0f * fk[off[1]] + 6.0f * fc - 4.0f * fk[off[2]] + fk[off[3]];
      ff = fc - eps * bx;
    }
    const float diff = ff - fc;
    d_rho += diff;
    d_jx += diff * (float(kcx(k)) - 0.0f);
    d_jy += diff * (float(kcy(k)) - 0.0f);
    d_jz += diff * (float(kcz(k)) - 0.0f);
    sf[k * kThreads] = ff;
  }
  const float inv_cs2 = 1.0f / CS2;
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    const float cx = float(kcx(k)) - 0.0f, cy = float(kcy(k)) - 0.0f, cz = float(kcz(k)) - 0.0f;
    const float cu = cx * d_jx + cy * d_jy + cz * d_jz;
    sf[k * kThreads] -= T.b[k][3].x * (d_rho + inv_cs2 * cu);
  }
}

// What bounds the fast instances: FP32 issue. They run ~5,500 thread-instructions per cell (two to
// three Newton passes of ~600 and one or two Cholesky solves of ~650, alpha ~1,200, the rest pull,
// WALE and update) at 168 registers, three CTAs per SM, issue 51 % active (no_instruction and wait
// stalls: the body is straight-line code), with spills of 136 bytes stored and 184 loaded a thread in the
// plain instance, 298 and 492 in the EDGES ones. The body is unrolled over the pairs with the 39
// equilibrium values in registers, guards and blends included; HRR, the other alpha solvers and what
// follows a NaN read the shared columns. Measured on a 96^3 periodic box, two steps per call: 2,660 us with the
// Newton pass over the basis table, alpha from sums of logarithms over the columns and a trip to
// memory per pulled direction; 452 us now while alpha comes from the series, 722 us (3,370 before)
// on a developed flow whose deviations are of the order of f_eq, so that every alpha comes from the
// logarithms and many cells take the positivity blends, which read the equilibrium from registers
// and the column (1,040 us while they evaluated it again). Distance from the 64-bit step after two steps: velocity 3.1e-5 against 2.9e-3 before.
// SVV: the spectral vanishing viscosity is compiled in (a.svv_x or a.svv_yz > 0).
template <bool EDGES, bool FAST, bool SVV = false>
__global__ void __launch_bounds__(kThreads, FAST ? KBC_FAST_MIN_BLOCKS : KBC_MIN_BLOCKS) k_kbc_step(const KbcArgs a) {
  __shared__ Tables T;
  __shared__ int32_t s_nbr[27];
  __shared__ float s_f[Q * kThreads];
  __shared__ float s_h[NSLOT * kThreads];
  const int tid = threadIdx.x;
  const int b = blockIdx.x >> 2;
  const int cell = ((blockIdx.x & 3) << 7) | tid;
  build_tables(T);
  if (tid < 27) s_nbr[tid] = a.nbr[(int64_t)b * 27 + tid];
  __syncthreads();
  float* sf = s_f + tid;
  float* sh = s_h + tid;
  const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
  const int64_t N = (int64_t)a.nb * 512;
  const int64_t ci = (int64_t)b * 512 + cell;
  // solid cells: the cell itself (bit 13) and its face neighbours (WALE stencil)
  const uint32_t solid_mask =
      (EDGES && a.cmask && (a.bflags[b] & kNearSolid)) ? a.cmask[(int64_t)a.mslot[b] * 512 + cell] : 0u;

  // the previous velocities of the six face neighbours (the WALE stencil, physics_utils.jl:2217-2233)
  // and the cached multipliers; the fast path issues these loads before the pull, so that one trip to
  // memory covers all three
  float up[3][3], um[3][3];
  auto load_velocities = [&]() {
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int d = s == 0 ? 1 : -1;
        const int px = x + (ax == 0 ? d : 0), py = y + (ax == 1 ? d : 0), pz = z + (ax == 2 ? d : 0);
        const int ox = px < 0 ? -1 : (px > 7 ? 1 : 0), oy = py < 0 ? -1 : (py > 7 ? 1 : 0), oz = pz < 0 ? -1 : (pz > 7 ? 1 : 0);
        const int bo = s_nbr[(ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)];
        // a neighbour outside the domain (ghost block) or in a solid cell contributes the own
        // velocity (physics_utils.jl:1981-2035); mask bit of the D3Q27 direction whose source it is
        const int sbit = ax == 0 ? (s == 0 ? 12 : 14) : ax == 1 ? (s == 0 ? 10 : 16) : (s == 0 ? 4 : 22);
        const bool own = EDGES && (bo >= a.nb || ((solid_mask >> sbit) & 1u));
        const int64_t c = own ? ci : ((px & 7) | ((py & 7) << 3) | ((pz & 7) << 6)) + 512 * (int64_t)bo;
#pragma unroll
        for (int comp = 0; comp < 3; ++comp) (s == 0 ? up : um)[ax][comp] = a.vin[c + N * comp];
      }
    }
  };
  // STEP 3: WALE from the previous velocity (physics_utils.jl:2217-2233, :2588-2700)
  float g11, g22, g33, S12, S13, S23;
  float nu_eddy = 0.0f;
  auto wale = [&]() {
    float g[9];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp)
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) g[3 * comp + ax] = 0.5f * (up[ax][comp] - um[ax][comp]);
    const float g12 = g[1], g13 = g[2], g21 = g[3], g23 = g[5], g31 = g[6], g32 = g[7];
    g11 = g[0]; g22 = g[4]; g33 = g[8];
    S12 = 0.5f * (g12 + g21); S13 = 0.5f * (g13 + g31); S23 = 0.5f * (g23 + g32);
    const float q11 = g11 * g11 + g12 * g21 + g13 * g31, q12 = g11 * g12 + g12 * g22 + g13 * g32, q13 = g11 * g13 + g12 * g23 + g13 * g33;
    const float q21 = g21 * g11 + g22 * g21 + g23 * g31, q22 = g21 * g12 + g22 * g22 + g23 * g32, q23 = g21 * g13 + g22 * g23 + g23 * g33;
    const float q31 = g31 * g11 + g32 * g21 + g33 * g31, q32 = g31 * g12 + g32 * g22 + g33 * g32, q33 = g31 * g13 + g32 * g23 + g33 * g33;
    const float tr = (q11 + q22 + q33) / 3.0f;
    const float Sd11 = q11 - tr, Sd22 = q22 - tr, Sd33 = q33 - tr;
    const float Sd12 = 0.5f * (q12 + q21), Sd13 = 0.5f * (q13 + q31), Sd23 = 0.5f * (q23 + q32);
    const float OP1 = Sd11 * Sd11 + Sd22 * Sd22 + Sd33 * Sd33 + 2.0f * (Sd12 * Sd12 + Sd13 * Sd13 + Sd23 * Sd23);
    const float OP2 = g11 * g11 + g22 * g22 + g33 * g33 + 2.0f * (S12 * S12 + S13 * S13 + S23 * S23);
    if (OP1 > 1e-12f) {
      const float OP1_32 = OP1 * sqrtf(OP1);
      const float OP2_52 = OP2 * OP2 * sqrtf(jmax(OP2, 1e-12f));
      const float denom = OP2_52 + OP1 * sqrtf(sqrtf(jmax(OP1, 1e-12f)));
      if (denom > 1e-12f) nu_eddy = (a.c_wale * a.c_wale) * OP1_32 / denom;
    }
  };
  Eq<FAST> eq;
  float* lam = a.lam + (int64_t)b * 13 * 512 + cell;
  if constexpr (FAST) {
    load_velocities();
#pragma unroll
    for (int m = 0; m < 13; ++m) eq.la[m] = lam[m * 512];
  }

  // STEP 1-2: pull, moments, density floor and NaN reset (:898-1290, 1616-1650)
  float rho, ux, uy, uz, inv_rho;
  float f_low = F_FLOOR;     // fast path: the smallest arriving population (at most the floor) ...
  bool replaced = false;     // ... unless they were replaced after the pull
  bool unbalanced = false;   // populations and macros may differ in mass or momentum
  {
    float jx = 0.0f, jy = 0.0f, jz = 0.0f;
    rho = 0.0f;
    if constexpr (FAST) {
      // unrolled: the offsets of the 39 pulls share the few shifted coordinates of each axis. All loads
      // come before the first store to the column: the compiler cannot tell the two apart, and one
      // trip to memory per direction was most of the kernel's time
      float v[Q];
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        const int sx = x - kcx(k), sy = y - kcy(k), sz = z - kcz(k);
        const int bo = s_nbr[(sx >> 3) + 3 * (sy >> 3) + 9 * (sz >> 3) + 13];
        v[k] = (a.fin + (int64_t)bo * (Q * 512) + ((sx & 7) | ((sy & 7) << 3) | ((sz & 7) << 6)))[k * 512];
      }
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        const float f = v[k];
        sf[k * kThreads] = f;
        f_low = fminf(f_low, f);
        rho += f;
        jx += f * float(kcx(k));
        jy += f * float(kcy(k));
        jz += f * float(kcz(k));
      }
    } else {
#pragma unroll 13
      for (int k = 0; k < Q; ++k) {
        const int c = T.c[k];
        const int cx = (c & 15) - 3, cy = ((c >> 4) & 15) - 3, cz = ((c >> 8) & 15) - 3;
        const int sx = x - cx, sy = y - cy, sz = z - cz;
        const int ox = sx < 0 ? -1 : (sx > 7 ? 1 : 0), oy = sy < 0 ? -1 : (sy > 7 ? 1 : 0), oz = sz < 0 ? -1 : (sz > 7 ? 1 : 0);
        const int bo = s_nbr[(ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)];
        const float f = a.fin[((int64_t)bo * Q + k) * 512 + ((sx & 7) | ((sy & 7) << 3) | ((sz & 7) << 6))];
        sf[k * kThreads] = f;
        rho += f;
        jx += f * float(cx);
        jy += f * float(cy);
        jz += f * float(cz);
      }
    }
    if (EDGES && (solid_mask & (1u << 13))) {
      // simple bounce-back inside the obstacle (:1602-1613); the multiplier cache is left as it is
      a.vout[ci] = 0.0f; a.vout[ci + N] = 0.0f; a.vout[ci + 2 * N] = 0.0f;
      a.rho[ci] = 1.0f;
#pragma unroll 1
      for (int k = 0; k < Q; ++k) a.fout[((int64_t)b * Q + k) * 512 + cell] = sf[kopp(k) * kThreads];
      return;
    }
    if (EDGES && a.faces && x == 0 && s_nbr[nbr13(-1, 0, 0)] >= a.nb && a.binfo[b].x == 1) {
      // a cell on the inlet face (global x = 1): mass and momentum pinned to the inlet
      // equilibrium's (:1313-1352), then the moments again
      kbc::four_moment_pin(sf, kThreads, a.trho, a.tjx, a.tjy, a.tjz);
      replaced = true;
      rho = 0.0f; jx = 0.0f; jy = 0.0f; jz = 0.0f;
#pragma unroll 1
      for (int k = 0; k < Q; ++k) {
        const float f = sf[k * kThreads];
        rho += f;
        jx += f * float(kcx(k));
        jy += f * float(kcy(k));
        jz += f * float(kcz(k));
      }
    }
    const float rho_raw = rho;
    rho = jmax(rho_raw, 0.01f);
    inv_rho = 1.0f / rho;
    ux = jx * inv_rho; uy = jy * inv_rho; uz = jz * inv_rho;
    const bool is_nan = !(rho_raw == rho_raw) || !(ux == ux) || !(uy == uy) || !(uz == uz);
    if (is_nan || rho_raw < 0.01f) {
      rho = 1.0f; ux = a.u_inlet; uy = 0.0f; uz = 0.0f; inv_rho = 1.0f;
      replaced = unbalanced = true;
#pragma unroll 1
      for (int k = 0; k < Q; ++k) sf[k * kThreads] = a.feq_inlet[k];
    }
  }
  if constexpr (FAST) {
    // the strain rates wait in the (still unused) h column for the HRR blend, where it is on
    wale();
    const float g[6] = {g11, g22, g33, S12, S13, S23};
#pragma unroll
    for (int i = 0; i < 6; ++i) sh[i * kThreads] = g[i];
  }
  // sponge (kernel_entropic_d3q39.jl:1662, 1787-1841; athermal, pre-collision form)
  const float sp = a.sponge ? a.sponge[ci] : 0.0f;
  if (sp > 0.0f) {
    replaced = unbalanced = true;
    rho = rho * (1.0f - sp) + 1.0f * sp;
    ux = ux * (1.0f - sp) + a.u_inlet * sp;
    uy = uy * (1.0f - sp);
    uz = uz * (1.0f - sp);
    if (a.sponge_blend) {
      // the populations toward the inlet equilibrium, then the macros again from them
      rho = 0.0f;
      float jx = 0.0f, jy = 0.0f, jz = 0.0f;
#pragma unroll 1
      for (int k = 0; k < Q; ++k) {
        const float f = sf[k * kThreads] * (1.0f - sp) + a.feq_inlet[k] * sp;
        sf[k * kThreads] = f;
        rho += f;
        jx += f * float(kcx(k));
        jy += f * float(kcy(k));
        jz += f * float(kcz(k));
      }
      rho = jmax(rho, 0.01f);
      inv_rho = 1.0f / rho;
      ux = jx * inv_rho; uy = jy * inv_rho; uz = jz * inv_rho;
    }
  }
  // macro realizability (:2112-2229): the far-bulk bounds away from walls and sponges, the
  // near-wall ones (MacroBoundsPack defaults 0.35 / 2.40) elsewhere
  const float wd = a.wdist ? a.wdist[ci] : __int_as_float(0x7fc00000);
  const bool far_bulk = (wd != wd || wd > 16.0f) && sp < 0.03f;
  bool macro_limited = false;
  {
    const float u_trans = sqrtf(uy * uy + uz * uz);
    const float uxr = ux - 0.0f;
    float uyr = uy - 0.0f, uzr = uz - 0.0f;
    float u_rel = sqrtf(uxr * uxr + uyr * uyr + uzr * uzr);
    const float u_ref = jmax(jmax(a.u_inlet, 0.1f), 0.1f);
    float u_cap = jmin(1.00f, jmax(0.80f, 1.35f * u_ref + 0.15f));
    float u_trans_cap = jmin(0.92f, jmax(0.55f, 1.15f * u_ref + 0.12f));
    if (far_bulk) {
      u_cap = jmin(u_cap, jmin(0.78f, jmax(0.48f, 1.12f * u_ref + 0.08f)));
      u_trans_cap = jmin(u_trans_cap, jmin(0.46f, jmax(0.18f, 0.68f * u_ref + 0.04f)));
    }
    const bool speed_path = u_rel > u_cap;
    const bool trans_path = u_trans > u_trans_cap;
    const float rho_floor = far_bulk ? 0.42f : 0.35f, rho_ceil = far_bulk ? 2.10f : 2.40f;
    const bool density_path = rho < 0.30f || rho > 2.80f || (far_bulk && (rho < rho_floor || rho > rho_ceil)) ||
                              ((rho < 0.45f || rho > 2.20f) && (speed_path || trans_path));
    if (density_path) {
      rho = jclamp(rho, rho_floor, rho_ceil);
      inv_rho = 1.0f / jmax(rho, 0.01f);
      macro_limited = true;
    }
    if (trans_path && u_trans > 1e-8f) {
      const float ts = u_trans_cap / jmax(u_trans, 1e-8f);
      uy *= ts;
      uz *= ts;
      uyr = uy - 0.0f; uzr = uz - 0.0f;
      u_rel = sqrtf(uxr * uxr + uyr * uyr + uzr * uzr);
      macro_limited = true;
    }
    if (speed_path && u_rel > 1e-8f) {
      const float ss = u_cap / jmax(u_rel, 1e-8f);
      ux = 0.0f + uxr * ss;
      uy = 0.0f + uyr * ss;
      uz = 0.0f + uzr * ss;
      macro_limited = true;
    }
  }
  // equilibrium velocity and its cap (:2262-2282)
  float ux_rel = (ux + 0.5f * 0.0f * inv_rho) - 0.0f;
  float uy_rel = (uy + 0.5f * 0.0f * inv_rho) - 0.0f;
  float uz_rel = (uz + 0.5f * 0.0f * inv_rho) - 0.0f;
  bool eq_limited = false;
  {
    const float m = sqrtf(ux_rel * ux_rel + uy_rel * uy_rel + uz_rel * uz_rel);
    if (m > 0.82f) {
      const float sc = 0.82f / jmax(m, 1e-6f);
      ux_rel *= sc; uy_rel *= sc; uz_rel *= sc;
      eq_limited = true;
    }
  }
  a.rho[ci] = rho;
  a.vout[ci] = ux;
  a.vout[ci + N] = uy;
  a.vout[ci + 2 * N] = uz;
  // STEP 3a: multipliers (warm start from the cache) and the mass correction (:2330-2385)
  eq.rho = rho;
  [[maybe_unused]] float fe[FAST ? Q : 1];  // fast path: the equilibrium before the mass correction
  {
    if constexpr (!FAST) {
#pragma unroll
      for (int m = 0; m < 13; ++m) eq.la[m] = lam[m * 512];
    }
    solve_lambdas<FAST>(T, rho, ux_rel, uy_rel, uz_rel, eq.la, fe, a.warm_gate);
#pragma unroll
    for (int m = 0; m < 13; ++m) lam[m * 512] = eq.la[m];
    float sum = 0.0f;
    if constexpr (FAST) {
#pragma unroll
      for (int k = 0; k < Q; ++k) sum += fe[k];
    } else {
#pragma unroll 3
      for (int k = 0; k < Q; ++k) sum += fi_row<FAST>(rho, eq.la, T.b[k]);
    }
    eq.corr = sum > 1e-15f ? rho / sum : 1.0f;
  }
  if constexpr (!FAST) {
    load_velocities();
    wale();
  }
  nu_eddy = jmax(nu_eddy, a.nu_bg * a.amr_sgs_scale);
  // Mach-pocket viscosity (:2777-2806), shock sensor off
  float pocket;
  {
    const float cs_local = sqrtf(jmax(CS2 * jmax(1.0f, 0.2f), 1e-6f));
    const float inv_cs = 1.0f / cs_local;
    const float u_mag = sqrtf(ux * ux + uy * uy + uz * uz);
    const float u_perp = sqrtf(uy * uy + uz * uz);
    const float mach_boost = smooth(jclamp((u_mag * inv_cs - 0.50f) / 0.25f, 0.0f, 1.0f));
    const float perp_boost = smooth(jclamp((u_perp * inv_cs - 0.32f) / 0.25f, 0.0f, 1.0f));
    const float rho_lo = smooth(jclamp((0.90f - rho) / 0.26f, 0.0f, 1.0f));
    const float rho_hi = smooth(jclamp((rho - 1.30f) / 0.70f, 0.0f, 1.0f));
    const float rho_split = jmax(rho_lo, rho_hi);
    pocket = jmax(jmax(perp_boost * jmax(rho_split, 0.0f), mach_boost * rho_split),
                  jmax(0.0f * mach_boost, perp_boost * mach_boost));
    if (pocket > 0.0f) nu_eddy = jmax(nu_eddy, pocket * jmax(5.00f * a.shock_nu_max, 0.24f) * a.amr_sgs_scale);
  }
  nu_eddy = jmax(nu_eddy, a.nu_floor);
  const float tau_eff = 0.5f + ((a.tau - 0.5f) * CS2 + nu_eddy) / CS2;
  const float omega = 1.0f / jmax(tau_eff, 0.500001f);
  const float beta = 0.5f * omega;
  float sigma = a.sigma0;
  if (pocket > 0.0f) sigma = jmax(sigma, jmin(0.995f, 0.80f + 0.195f * pocket));
  const float h_scale = sigma > 0.0f ? 1.0f - sigma : 1.0f;
  Hrr hr;
  hr.on = a.hrr;
  hr.sigma = a.hrr_sigma;
  hr.oms = 1.0f - a.hrr_sigma;
  if (FAST && hr.on) {
    g11 = sh[0]; g22 = sh[kThreads]; g33 = sh[2 * kThreads];
    S12 = sh[3 * kThreads]; S13 = sh[4 * kThreads]; S23 = sh[5 * kThreads];
  }
  if (!FAST || hr.on) {
    const float c = -2.0f * rho * CS2 * jmax(tau_eff - 0.5f, 0.0f);
    hr.pxx = c * g11; hr.pyy = c * g22; hr.pzz = c * g33; hr.pxy = c * S12; hr.pxz = c * S13; hr.pyz = c * S23;
  }
  // STEP 4b: positivity of the arriving populations (:2885-2906)
  {
    bool any_negative = FAST && f_low < F_FLOOR;
    if (!FAST || replaced) {
      any_negative = false;
#pragma unroll 13
      for (int k = 0; k < Q; ++k) any_negative = any_negative || sf[k * kThreads] < F_FLOOR;
    }
    if (any_negative) {
      unbalanced = true;
      float worst = 1.0f;
      if constexpr (FAST) {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = fe[k] * eq.corr, fneq = sf[k * kThreads] - fk;
          if (fneq < 0.0f && fk > F_FLOOR) worst = jmin(worst, (fk - F_FLOOR) / (-fneq + F_FLOOR));
        }
        worst = jclamp(worst, 0.0f, 1.0f);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = fe[k] * eq.corr;
          sf[k * kThreads] = maxc(fk + worst * (sf[k * kThreads] - fk), F_FLOOR);
        }
      } else {
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          const float fneq = sf[k * kThreads] - fe;
          if (fneq < 0.0f && fe > F_FLOOR) worst = jmin(worst, (fe - F_FLOOR) / (-fneq + F_FLOOR));
        }
        worst = jclamp(worst, 0.0f, 1.0f);
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          sf[k * kThreads] = maxc(fe + worst * (sf[k * kThreads] - fe), F_FLOOR);
        }
      }
    }
  }
  // realizability guard (:2907-2958)
  float guard;
  {
    const float u_g = sqrtf(ux * ux + uy * uy + uz * uz);
    const float cs_g = sqrtf(jmax(CS2 * jmax(1.0f, 0.2f), 1e-6f));
    const float mach_gb = smooth(jclamp((u_g / cs_g - 0.62f) / 0.22f, 0.0f, 1.0f));
    const float trans_gb = smooth(jclamp((sqrtf(uy * uy + uz * uz) / cs_g - 0.38f) / 0.22f, 0.0f, 1.0f));
    const float rho_low_g = jclamp((0.88f - rho) / 0.28f, 0.0f, 1.0f);
    const float rho_high_g = jclamp((rho - 1.35f) / 0.65f, 0.0f, 1.0f);
    const float u_ref_g = jmax(jmax(a.u_inlet, 0.1f), 0.54f);
    const float u_spike = jmax(jclamp((u_g - u_ref_g) / 0.24f, 0.0f, 1.0f), 0.85f * jmax(mach_gb, trans_gb));
    const float neq_g = jclamp((0.0f - 0.12f) / 0.35f, 0.0f, 1.0f);
    const float pocket_neq = jmax(jmax(0.0f, neq_g), jmax(mach_gb, trans_gb));
    guard = jmax(jmax(0.0f * jmax(neq_g, mach_gb), rho_low_g * pocket_neq), jmax(rho_high_g, u_spike * pocket_neq));
    guard = jmax(guard, pocket);
    if (eq_limited || macro_limited) guard = jmax(guard, 1.0f);
    if (guard > 0.0f) {
      float sdf = 0.0f, sfe = 0.0f;
      if constexpr (FAST) {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = fe[k] * eq.corr;
          sdf += fabsf(sf[k * kThreads] - fk);
          sfe += fk;
        }
      } else {
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          sdf += fabsf(sf[k * kThreads] - fe);
          sfe += fabsf(fe);
        }
      }
      const float reps = sfe > 1e-10f ? sdf / sfe : 0.0f;
      const float cap = jmax(0.025f, 0.18f - 0.155f * guard);
      if (reps > cap) {
        const float th = jclamp(cap / jmax(reps, 1e-12f), 0.0f, 1.0f);
        if constexpr (FAST) {
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            const float fk = fe[k] * eq.corr;
            sf[k * kThreads] = maxc(fk + th * (sf[k * kThreads] - fk), F_FLOOR);
          }
        } else {
#pragma unroll 1
          for (int k = 0; k < Q; ++k) {
            const float fe = eq(T, k);
            sf[k * kThreads] = maxc(fe + th * (sf[k * kThreads] - fe), F_FLOOR);
          }
        }
      }
    }
  }
  bool post_done = false;  // the fast path's column holds the post-collision populations ...
  bool blended = false;    // ... after the positivity blend and the guard
  if constexpr (FAST) {
    if (a.solver == 0 && !hr.on) {
      const float coeff_s = 1.0f - 2.0f * beta;
#pragma unroll
      for (int k = 0; k < Q; ++k) fe[k] *= eq.corr;
      AlphaSeries A;
      bool decided = false;
      float alpha_f = 2.0f;
      // the series needs populations with the cell's mass and momentum and an unscaled h
      if (sigma == 0.0f && !(guard > 0.0f) && !unbalanced && !macro_limited && !eq_limited && A.admits(sf, fe)) {
        A.gather(sf, fe);
        decided = A.solve(eq.la, beta, alpha_f);
      }
      // a_k = f_eq_k + coeff_s s_k, h per pair, and where the series did not decide the entropy of
      // the arriving populations
      float hv[19], h_sq = 0.0f;
      {
        // f_eq takes the column's place, for the post-collision blends
        float H0 = entropy_term(sf[0], 0, 0.0f), H1 = 0.0f;
        const float f0 = sf[0];
        sf[0] = fe[0];
        fe[0] = fe[0] + coeff_s * (f0 - fe[0]);
#pragma unroll
        for (int p = 0; p < 19; ++p) {
          const int k = kpos(p), kb = kopp(k);
          const float fk = sf[k * kThreads], fb = sf[kb * kThreads];
          sf[k * kThreads] = fe[k];
          sf[kb * kThreads] = fe[kb];
          if (!decided) {
            H0 = entropy_term(fk, k, H0);
            H1 = entropy_term(fb, kb, H1);
          }
          const float df = fk - fe[k], db = fb - fe[kb];
          const float s = coeff_s * (0.5f * (df + db));
          hv[p] = (0.5f * (df - db)) * h_scale;
          fe[k] = fe[k] + s;
          fe[kb] = fe[kb] + s;
          h_sq = __fmaf_rn(2.0f * hv[p], hv[p], h_sq);
        }
        if (!decided) {
          if (h_sq > 1e-20f) {
            const float inv_2beta = 0.5f / fmaxf(beta, 0.01f);
            alpha_f = alpha_bisection_regs(fe, hv, beta, H0 + H1);
            if (!(alpha_f > 0.0f)) alpha_f = inv_2beta;
            alpha_f = jclamp(alpha_f, inv_2beta, 6.0f);
          } else {
            alpha_f = 2.0f;
          }
        }
      }
      // KBC update; the smallest population and their sum checked before the store
      const float coeff = 1.0f - 2.0f * beta * alpha_f;
      float low = fe[0], total = fe[0];
#pragma unroll
      for (int p = 0; p < 19; ++p) {
        const int k = kpos(p), kb = kopp(k);
        fe[k] = __fmaf_rn(coeff, hv[p], fe[k]);
        fe[kb] = __fmaf_rn(-coeff, hv[p], fe[kb]);
        low = fminf(low, fminf(fe[k], fe[kb]));
        total += fe[k] + fe[kb];
      }
      const bool sane = total <= 1e3f;  // no population above 1e3 beside the negative ones, no NaN
      if (sane && low < 0.0f) {
        // positivity blend toward f_eq (as in the general tail)
        float blend = 1.0f;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = sf[k * kThreads], fneq = fe[k] - fk;
          if (fneq < 0.0f && fk > F_FLOOR) blend = fminf(blend, fk / (fk - fneq + F_FLOOR));
        }
        blend = fmaxf(blend, 0.0f);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = sf[k * kThreads];
          fe[k] = fk + blend * (fe[k] - fk);
        }
      }
      if (sane && guard > 0.0f) {
        float sdf = 0.0f, sfe = 0.0f;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          const float fk = sf[k * kThreads];
          sdf += fabsf(fe[k] - fk);
          sfe += fk;
        }
        const float ep = sfe > 1e-10f ? sdf / sfe : 0.0f;
        const float cap = fmaxf(0.025f, 0.22f - 0.195f * guard);
        if (ep > cap) {
          const float th = jclamp(cap / fmaxf(ep, 1e-12f), 0.0f, 1.0f);
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            const float fk = sf[k * kThreads];
            fe[k] = maxc(fk + th * (fe[k] - fk), F_FLOOR);
          }
        }
      }
      float top = fe[0];
#pragma unroll
      for (int k = 1; k < Q; ++k) top = fmaxf(top, fe[k]);
      if (!SVV && sane && top <= 1e3f) {
        float* fo = a.fout + (int64_t)b * Q * 512 + cell;
#pragma unroll
        for (int k = 0; k < Q; ++k) fo[k * 512] = fe[k];
        return;
      }
      blended = sane;
#pragma unroll
      for (int k = 0; k < Q; ++k) sf[k * kThreads] = fe[k];
      post_done = true;
    }
  }
  float coeff_h = 0.0f;
  if (!post_done) {
    // entropy of the arriving populations (:55-62), formed whether or not the alpha search runs
    float H_pre = 0.0f;
#pragma unroll 3
    for (int k = 0; k < Q; ++k) {
      const float fk = maxc(sf[k * kThreads], F_FLOOR);
      H_pre = kmad<FAST>(fk, safe_log<FAST>(FAST ? fk * T.b[k][3].y : fk / T.b[k][3].x), H_pre);
    }
    const float inv_2beta = 0.5f / jmax(beta, 0.01f);
    float alpha = 2.0f;
    bool alpha_done = false;
    if (a.solver == 3) alpha_done = alpha_taylor<FAST>(T, sf, eq, h_scale, hr, beta, alpha);
    // STEP 5: split per pair, a_k = f_eq_k + coeff_s s_k over f_k (:2962-3095)
    const float coeff_s = 1.0f - 2.0f * beta;
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const int ps = T.ps[k];
      if (!(ps & 0x200)) continue;
      const int kb = (T.c[k] >> 12) & 63;
      const float fe = eq(T, k), feb = kb == k ? fe : eq(T, kb);
      const float df = sf[k * kThreads] - fe, dfb = sf[kb * kThreads] - feb;
      const float s = hrr_s(T, 0.5f * (df + dfb), k, hr);
      sh[(ps & 0xff) * kThreads] = (0.5f * (df - dfb)) * h_scale;
      sf[k * kThreads] = fe + coeff_s * s;
      if (kb != k) sf[kb * kThreads] = feb + coeff_s * s;
    }
    float h_norm_sq = 0.0f;
#pragma unroll 13
    for (int k = 0; k < Q; ++k) {
      const float hk = h_at(T, sh, k);
      h_norm_sq += hk * hk;
    }
    // STEP 6: alpha (:3109-3150)
    if (h_norm_sq > 1e-20f) {
      if (a.solver == 1) { alpha = alpha_newton<FAST>(T, sf, sh, beta, H_pre); alpha_done = true; }
      else if (a.solver == 2) {
        float fn = 0.0f;
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          fn += fe * fe;
        }
        alpha = jclamp(2.0f - 0.5f * (h_norm_sq / jmax(fn, 1e-15f)), inv_2beta, 4.0f);
        alpha_done = true;
      }
      if (!alpha_done) alpha = alpha_bisection<FAST>(T, sf, sh, beta, H_pre, 10);
      if (!(alpha > 0.0f)) alpha = inv_2beta;
      alpha = jclamp(alpha, inv_2beta, 6.0f);
    } else {
      alpha = 2.0f;
    }
    coeff_h = 1.0f - 2.0f * beta * alpha;
  }
  // STEP 7-8: KBC, post-collision blend and guard, output (:3153-3368). The zero body force adds
  // +-0 to a sum whose f_eq term is positive, which leaves it unchanged.
  float fmin = 1.0f;
  if (post_done) {
#pragma unroll 13
    for (int k = 0; k < Q; ++k) fmin = jmin(fmin, sf[k * kThreads]);
  } else {
#pragma unroll 13
    for (int k = 0; k < Q; ++k) {
      const float v = sf[k * kThreads] + coeff_h * h_at(T, sh, k);
      sf[k * kThreads] = v;
      fmin = jmin(fmin, v);
    }
  }
  if (fmin < 0.0f && !blended) {
    float blend = 1.0f;
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const float fe = eq(T, k);
      const float fneq = sf[k * kThreads] - fe;
      if (fneq < 0.0f && fe > F_FLOOR) blend = jmin(blend, fe / (fe - fneq + F_FLOOR));
    }
    blend = jmax(blend, 0.0f);
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const float fe = eq(T, k);
      sf[k * kThreads] = fe + blend * (sf[k * kThreads] - fe);
    }
  }
  if (guard > 0.0f && !blended) {
    float sdf = 0.0f, sfe = 0.0f;
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const float fe = eq(T, k);
      sdf += fabsf(sf[k * kThreads] - fe);
      sfe += fabsf(fe);
    }
    const float ep = sfe > 1e-10f ? sdf / sfe : 0.0f;
    const float cap = jmax(0.025f, 0.22f - 0.195f * guard);
    if (ep > cap) {
      const float th = jclamp(cap / jmax(ep, 1e-12f), 0.0f, 1.0f);
#pragma unroll 1
      for (int k = 0; k < Q; ++k) {
        const float fe = eq(T, k);
        sf[k * kThreads] = maxc(fe + th * (sf[k * kThreads] - fe), F_FLOOR);
      }
    }
  }
  if constexpr (SVV) {
    // the filter after the post-collision guard, y-z first, then x; then the positivity
    // re-enforcement of an add-on (kernel_entropic_d3q39.jl:3256-3318)
    const SvvView v{a.fin, a.mslot, a.cmask, a.nb};
    if (a.svv_yz > 0.0f) svv_axis<true>(v, T, s_nbr, b, cell, a.svv_yz, sf);
    if (a.svv_x > 0.0f) svv_axis<false>(v, T, s_nbr, b, cell, a.svv_x, sf);
    if (a.svv_yz > 0.0f || a.svv_x > 0.0f) {
      float fmin_post = sf[0];
#pragma unroll 1
      for (int k = 1; k < Q; ++k) fmin_post = jmin(fmin_post, sf[k * kThreads]);
      if (fmin_post < 0.0f) {
        float blend = 1.0f;
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          const float fneq = sf[k * kThreads] - fe;
          if (fneq < 0.0f && fe > F_FLOOR) blend = jmin(blend, fe / (fe - fneq + F_FLOOR));
        }
        blend = jmax(blend, 0.0f);
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const float fe = eq(T, k);
          sf[k * kThreads] = fe + blend * (sf[k * kThreads] - fe);
        }
      }
    }
  }
  float* fo = a.fout + (int64_t)b * Q * 512 + cell;
#pragma unroll 13
  for (int k = 0; k < Q; ++k) {
    float v = sf[k * kThreads];
    if (!(v == v) || v > 1e3f) v = eq(T, k);
    fo[k * 512] = v;
  }
}

// equilibrium start from rho, u (device float, reference layout): f, vel, rho; lambda = NaN
__global__ void __launch_bounds__(kThreads) k_kbc_init(const float* rho_in, const float* vel_in, float* f, float* vel,
                                                       float* rho, float* lam, int32_t nb) {
  __shared__ Tables T;
  build_tables(T);
  __syncthreads();
  const int b = blockIdx.x >> 2;
  const int cell = ((blockIdx.x & 3) << 7) | threadIdx.x;
  const int64_t N = (int64_t)nb * 512, ci = (int64_t)b * 512 + cell;
  const float r = rho_in[ci], ux = vel_in[ci], uy = vel_in[ci + N], uz = vel_in[ci + 2 * N];
  Eq<> eq;
  eq.rho = r;
  eq.la[0] = qnan();
  float fe[1];
  solve_lambdas(T, r, ux, uy, uz, eq.la, fe);
  float sum = 0.0f;
  for (int k = 0; k < Q; ++k) sum += fi_row(r, eq.la, T.b[k]);
  eq.corr = sum > 1e-15f ? r / sum : 1.0f;
  for (int k = 0; k < Q; ++k) f[((int64_t)b * Q + k) * 512 + cell] = eq(T, k);
#pragma unroll
  for (int m = 0; m < 13; ++m) lam[((int64_t)b * 13 + m) * 512 + cell] = qnan();
  rho[ci] = r;
  vel[ci] = ux; vel[ci + N] = uy; vel[ci + 2 * N] = uz;
}

// FP64 mass and momentum: one CTA per block, per-block partials, then a fixed-order final sum
__global__ void __launch_bounds__(kThreads) k_kbc_mm_part(const float* f, int32_t nb, double* part) {
  const int b = blockIdx.x;
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = threadIdx.x; c < 512; c += kThreads) {
    const float* fc = f + (int64_t)b * Q * 512 + c;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const double v = fc[k * 512];
      m[0] += v; m[1] += v * kcx(k); m[2] += v * kcy(k); m[3] += v * kcz(k);
    }
  }
  __shared__ double s[4][kThreads];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i][threadIdx.x] = m[i];
  __syncthreads();
  for (int w = kThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i][threadIdx.x] += s[i][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 4) part[(int64_t)b * 4 + threadIdx.x] = s[threadIdx.x][0];
}

__global__ void k_kbc_mm_final(const double* part, int32_t nb, double* out) {
  if (threadIdx.x < 4) {
    double acc = 0.0;
    for (int32_t b = 0; b < nb; ++b) acc += part[(int64_t)b * 4 + threadIdx.x];
    out[threadIdx.x] = acc;
  }
}

oal_status fail(oal_status s, const char* fmt, ...) {
  char buf[400];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  return oal_internal_set_error(s, buf);
}

#define KBC_TRY(expr)                                                                                 \
  do {                                                                                                \
    cudaError_t _e = (expr);                                                                          \
    if (_e != cudaSuccess) {                                                                          \
      cudaGetLastError();                                                                             \
      return fail(_e == cudaErrorMemoryAllocation ? OAL_E_OUT_OF_MEMORY : OAL_E_CUDA, "%s: %s", #expr, \
                  cudaGetErrorString(_e));                                                            \
    }                                                                                                 \
  } while (0)

// Host restatement of the inlet equilibrium table (physics_utils.jl:280-460 at rho = 1,
// u = (u_inlet, -0, -0), mass_correct_feq39!, floor 1e-10; timestep.jl:1169-1188): the populations
// of a cell reset after a NaN or a density below 0.01.
void inlet_equilibrium(float u_inlet, float* out) {
  const float cs2 = CS2, rho = 1.0f, ux = u_inlet, uy = -0.0f, uz = -0.0f;
  const float F_FLOOR_EQ = 1e-15f, OMEGA = 1.5f;
  const float eps = std::numeric_limits<float>::epsilon();
  const float TOL_SQ = 507.0f * eps * eps * rho * rho;
  const float usq = ux * ux + uy * uy + uz * uz, dT = 1.0f - 1.0f, dplus2_cs2 = 5.0f * cs2;
  const float ef = usq + 5.0f * cs2 * dT;
  const float mt[13] = {rho, rho * ux, rho * uy, rho * uz, rho * (ux * ux + cs2 * dT), rho * (uy * uy + cs2 * dT),
                        rho * (uz * uz + cs2 * dT), rho * ux * uy, rho * ux * uz, rho * uy * uz,
                        rho * ux * ef, rho * uy * ef, rho * uz * ef};
  const float inv_cs2 = 1.0f / cs2, inv_cs4 = inv_cs2 * inv_cs2;
  float la[13] = {-0.5f * usq * inv_cs2, ux * inv_cs2, uy * inv_cs2, uz * inv_cs2, 0.5f * inv_cs4 * ux * ux,
                  0.5f * inv_cs4 * uy * uy, 0.5f * inv_cs4 * uz * uz, inv_cs4 * ux * uy, inv_cs4 * ux * uz,
                  inv_cs4 * uy * uz, 0.0f, 0.0f, 0.0f};
  // f_i with the parenthesised products of this variant of the solve (la8*cx*cy = (la8*cx)*cy)
  auto f_i = [&](int i) {
    const float cx = float(kcx(i)) - 0.0f, cy = float(kcy(i)) - 0.0f, cz = float(kcz(i)) - 0.0f;
    const float efl = (cx * cx + cy * cy + cz * cz) - dplus2_cs2;
    const float lda = la[0] + la[1] * cx + la[2] * cy + la[3] * cz + la[4] * (cx * cx - cs2) +
                      la[5] * (cy * cy - cs2) + la[6] * (cz * cz - cs2) + la[7] * cx * cy + la[8] * cx * cz +
                      la[9] * cy * cz + la[10] * cx * efl + la[11] * cy * efl + la[12] * cz * efl;
    const float v = rho * kw(i) * kbc::exp(std::min(std::max(lda, -20.0f), 20.0f));
    return v < F_FLOOR_EQ ? F_FLOOR_EQ : v;
  };
  const int g0[4] = {0, 4, 10, 13};
  for (int sweep = 0; sweep < 200; ++sweep) {
    float d[13] = {0}, j[13] = {0};
    for (int g = 0; g < 3; ++g) {
      for (int i = 0; i < Q; ++i) {
        const float fi = f_i(i);
        for (int m = g0[g]; m < g0[g + 1]; ++m) {
          if (m == 0) { d[0] += fi; j[0] += fi; continue; }
          const float b = kbasis(m - 1, i);
          d[m] += fi * b;
          j[m] += fi * b * b;
        }
      }
      for (int m = g0[g]; m < g0[g + 1]; ++m)
        la[m] += j[m] > F_FLOOR_EQ ? std::min(std::max(OMEGA * (mt[m] - d[m]) / j[m], -2.0f), 2.0f) : 0.0f;
    }
    float res = 0.0f;
    for (int m = 0; m < 13; ++m) res += (mt[m] - d[m]) * (mt[m] - d[m]);
    if (res < TOL_SQ) break;
  }
  float fe[Q], sum = 0.0f;
  for (int i = 0; i < Q; ++i) fe[i] = f_i(i);
  for (int i = 0; i < Q; ++i) sum += fe[i];
  if (sum > 1e-15f) {
    const float corr = rho / sum;
    for (int i = 0; i < Q; ++i) fe[i] *= corr;
  }
  for (int i = 0; i < Q; ++i) out[i] = fe[i] < 1e-10f ? 1e-10f : fe[i];
}

}  // namespace

struct KbcLevel {
  int device = 0;
  int32_t nb = 0;
  const int32_t* d_nbr = nullptr;
  KbcGeometry G;
  uint2* d_entries = nullptr;  // face-fill entries
  int64_t n_entries = 0;
  float* f[2] = {nullptr, nullptr};
  float* vel[2] = {nullptr, nullptr};
  float* rho = nullptr;
  float* lam = nullptr;
  double* d_mm_part = nullptr;
  double* d_mm = nullptr;
  int parity = 0;
  int64_t bytes = 0;
  cudaStream_t cap = nullptr;
  // the captured steps by starting parity: an odd number of steps ends on the other buffer
  struct Graph {
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph = nullptr;
    int32_t n = 0;
    oal_step_params p{};
  } gr[2];
  bool exact_math = false;  // kbc_set_exact_math
};

namespace {

void release_graph(KbcLevel::Graph& G) {
  if (G.exec) cudaGraphExecDestroy(G.exec);
  if (G.graph) cudaGraphDestroy(G.graph);
  G = KbcLevel::Graph{};
}
void release_graph(KbcLevel* L) {
  release_graph(L->gr[0]);
  release_graph(L->gr[1]);
}

oal_status resolve(const oal_step_params* p, KbcArgs* a) {
  if (!p) return fail(OAL_E_INVALID_ARG, "null step params");
  if (p->abi_version != OAL_ABI_VERSION)
    return fail(OAL_E_ABI_MISMATCH, "oal_step_params.abi_version %u != %d", p->abi_version, OAL_ABI_VERSION);
  if (p->operator_id != OAL_OP_ENTROPIC_D3Q39)
    return fail(OAL_E_INVALID_ARG, "a D3Q39 level steps with operator_id OAL_OP_ENTROPIC_D3Q39, not %d", p->operator_id);
  if (!(p->tau > 0.5f)) return fail(OAL_E_INVALID_ARG, "tau must exceed 1/2 (got %g)", (double)p->tau);
  if (p->adaptive_omega4 < 0 || p->adaptive_omega4 > 3)
    return fail(OAL_E_INVALID_ARG, "alpha solver (adaptive_omega4) %d: 0 bisection, 1 Newton, 2 approximate, 3 Taylor",
                p->adaptive_omega4);
  if (p->store_post_collision) return fail(OAL_E_UNSUPPORTED, "store_post_collision is not built for the D3Q39 level");
  if (p->wall_model_active) return fail(OAL_E_UNSUPPORTED, "the wall model needs a level with walls");
  std::memset(a, 0, sizeof *a);
  a->solver = p->adaptive_omega4;
  a->hrr = (p->hrr_hybrid == 1 && p->hrr_sigma < 0.999f) ? 1 : 0;
  a->tau = p->tau; a->c_wale = p->c_wale; a->nu_bg = p->nu_sgs_background; a->amr_sgs_scale = p->amr_sgs_scale;
  a->u_inlet = p->u_inlet; a->sigma0 = p->lambda_param; a->hrr_sigma = p->hrr_sigma;
  a->sponge_blend = p->sponge_blend_distributions == 1 ? 1 : 0;
  a->nu_floor = p->nu_sgs_lattice_floor; a->shock_nu_max = p->shock_nu_max;
  if (!(p->svv_x_epsilon >= 0.0f) || !std::isfinite(p->svv_x_epsilon) || !(p->svv_yz_epsilon >= 0.0f) ||
      !std::isfinite(p->svv_yz_epsilon))
    return fail(OAL_E_INVALID_ARG, "svv_x_epsilon and svv_yz_epsilon must be finite and >= 0");
  a->svv_x = p->svv_x_epsilon; a->svv_yz = p->svv_yz_epsilon;
  inlet_equilibrium(p->u_inlet, a->feq_inlet);
  for (int k = 0; k < Q; ++k) {
    const float fe = a->feq_inlet[k];
    a->trho += fe;
    a->tjx += fe * float(kcx(k));
    a->tjy += fe * float(kcy(k));
    a->tjz += fe * float(kcz(k));
  }
  return OAL_OK;
}

oal_status enqueue(KbcLevel* L, const KbcArgs& base, const oal_step_params* p_in, int32_t seed, cudaStream_t st) {
  KbcArgs a = base;
  const int p = L->parity;
  a.fin = L->f[p]; a.fout = L->f[p ^ 1];
  a.vin = L->vel[p]; a.vout = L->vel[p ^ 1];
  a.rho = L->rho; a.lam = L->lam; a.nbr = L->d_nbr; a.nb = L->nb;
  a.binfo = static_cast<const int4*>(L->G.d_binfo);
  a.faces = L->n_entries > 0 ? 1 : 0;
  if (L->G.has_solid) { a.bflags = L->G.d_bflags; a.mslot = L->G.d_mslot; a.cmask = L->G.d_cmask; }
  a.sponge = L->G.d_sponge;
  a.wdist = L->G.d_wdist;
  if (L->n_entries > 0) {
    KbcFillArgs fa;
    fa.f = L->f[p]; fa.entries = L->d_entries; fa.n = L->n_entries; fa.nbr = L->d_nbr; fa.binfo = a.binfo;
    fa.F = kbc::FaceParams{L->G.nx, L->G.ny, L->G.nz, p_in->ymin_wall_bc, p_in->transverse_freestream, seed,
                           p_in->transverse_freestream_blend, p_in->inlet_turbulence, p_in->u_inlet};
    for (int k = 0; k < Q; ++k) fa.feq_inlet[k] = a.feq_inlet[k];
    k_kbc_fill<<<(unsigned)((L->n_entries + 255) / 256), 256, 0, st>>>(fa);
    KBC_TRY(cudaGetLastError());
  }
  const unsigned grid = (unsigned)L->nb * 4;
  a.warm_gate = KBC_FAST_WARM_GATE;
  if (a.svv_x > 0.0f || a.svv_yz > 0.0f) {
    // the filter's instances carry the domain-face and solid logic (a no-op on periodic boxes)
    if (L->exact_math) k_kbc_step<true, false, true><<<grid, kThreads, 0, st>>>(a);
    else k_kbc_step<true, true, true><<<grid, kThreads, 0, st>>>(a);
  } else if (L->exact_math) {
    if (a.faces || a.cmask) k_kbc_step<true, false><<<grid, kThreads, 0, st>>>(a);
    else k_kbc_step<false, false><<<grid, kThreads, 0, st>>>(a);
  } else {
    if (a.faces || a.cmask) k_kbc_step<true, true><<<grid, kThreads, 0, st>>>(a);
    else k_kbc_step<false, true><<<grid, kThreads, 0, st>>>(a);
  }
  KBC_TRY(cudaGetLastError());
  L->parity ^= 1;
  return OAL_OK;
}

}  // namespace

oal_status kbc_create(int device, const KbcGeometry& G, KbcLevel** out) {
  const int32_t nb = G.nb;
  if (!out || nb <= 0 || !G.d_nbr || !G.h_nbr || !G.d_binfo || !G.h_bflags)
    return fail(OAL_E_INVALID_ARG, "kbc_create: bad arguments");
  *out = nullptr;
  if ((int64_t)nb * 4 > 0x7fffffffLL) return fail(OAL_E_TOO_LARGE, "too many blocks");
  KBC_TRY(cudaSetDevice(device));
  // face-fill entries: every (cell, k) of a block with a missing neighbour whose source lies in a
  // ghost block
  std::vector<uint2> entries;
  for (int32_t b = 0; b < nb; ++b) {
    if (G.h_bflags[b] & 1u) continue;  // BF_INTERIOR: all 26 neighbours present
    for (int cell = 0; cell < 512; ++cell) {
      const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
      for (int k = 0; k < Q; ++k) {
        const int sx = x - kcx(k), sy = y - kcy(k), sz = z - kcz(k);
        const int ox = sx < 0 ? -1 : (sx > 7 ? 1 : 0), oy = sy < 0 ? -1 : (sy > 7 ? 1 : 0), oz = sz < 0 ? -1 : (sz > 7 ? 1 : 0);
        if ((ox | oy | oz) == 0) continue;
        const int32_t g = G.h_nbr[(size_t)b * 27 + nbr13(ox, oy, oz)];
        if (g >= nb && g < nb + G.n_ghost) entries.push_back(make_uint2((uint32_t)b, (uint32_t)cell | ((uint32_t)k << 9)));
      }
    }
  }
  auto* L = new KbcLevel();
  L->device = device; L->nb = nb; L->d_nbr = G.d_nbr; L->G = G;
  L->G.h_nbr = nullptr; L->G.h_bflags = nullptr;  // host tables are only read here
  L->n_entries = (int64_t)entries.size();
  const size_t ncell = (size_t)nb * 512;
  const size_t fcell = ncell + (entries.empty() ? 0 : (size_t)G.n_ghost * 512);
  auto alloc = [&](void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
    return e;
  };
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
    e = alloc((void**)&L->f[i], fcell * Q * sizeof(float));
    if (e == cudaSuccess) e = alloc((void**)&L->vel[i], ncell * 3 * sizeof(float));
  }
  if (e == cudaSuccess) e = alloc((void**)&L->rho, ncell * sizeof(float));
  if (e == cudaSuccess) e = alloc((void**)&L->lam, ncell * 13 * sizeof(float));
  if (e == cudaSuccess) e = alloc((void**)&L->d_mm_part, (size_t)nb * 4 * sizeof(double));
  if (e == cudaSuccess) e = alloc((void**)&L->d_mm, 4 * sizeof(double));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&L->cap, cudaStreamNonBlocking);
  if (e == cudaSuccess && !entries.empty()) {
    e = cudaMalloc((void**)&L->d_entries, entries.size() * sizeof(uint2));
    if (e == cudaSuccess) e = cudaMemcpy(L->d_entries, entries.data(), entries.size() * sizeof(uint2), cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    kbc_destroy(L);
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? OAL_E_OUT_OF_MEMORY : OAL_E_CUDA, "D3Q39 level allocation: %s",
                cudaGetErrorString(e));
  }
  L->bytes = (int64_t)fcell * 2 * Q * 4 + (int64_t)ncell * (2 * 3 + 1 + 13) * 4 + (int64_t)nb * 32 + 32 +
             (int64_t)entries.size() * 8;
  *out = L;
  return OAL_OK;
}

void kbc_set_exact_math(KbcLevel* L, bool exact) {
  if (!L || L->exact_math == exact) return;
  L->exact_math = exact;
  release_graph(L);  // a captured graph holds the other kernel
}

void kbc_destroy(KbcLevel* L) {
  if (!L) return;
  cudaSetDevice(L->device);
  release_graph(L);
  for (int i = 0; i < 2; ++i) { cudaFree(L->f[i]); cudaFree(L->vel[i]); }
  cudaFree(L->rho); cudaFree(L->lam); cudaFree(L->d_mm_part); cudaFree(L->d_mm); cudaFree(L->d_entries);
  if (L->cap) cudaStreamDestroy(L->cap);
  cudaGetLastError();
  delete L;
}

oal_status kbc_init_equilibrium(KbcLevel* L, const double* rho, const double* vel) {
  if (!L || !rho || !vel) return fail(OAL_E_INVALID_ARG, "null argument");
  KBC_TRY(cudaSetDevice(L->device));
  const size_t ncell = (size_t)L->nb * 512;
  std::vector<float> hr(ncell), hv(3 * ncell);
  for (size_t i = 0; i < ncell; ++i) hr[i] = (float)rho[i];
  for (size_t i = 0; i < 3 * ncell; ++i) hv[i] = (float)vel[i];
  float *d_r = nullptr, *d_v = nullptr;
  cudaError_t e = cudaMalloc(&d_r, ncell * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&d_v, 3 * ncell * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(d_r, hr.data(), ncell * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d_v, hv.data(), 3 * ncell * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_kbc_init<<<(unsigned)L->nb * 4, kThreads>>>(d_r, d_v, L->f[0], L->vel[0], L->rho, L->lam, L->nb);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  cudaFree(d_r); cudaFree(d_v);
  if (e != cudaSuccess) { cudaGetLastError(); return fail(OAL_E_CUDA, "D3Q39 init_equilibrium: %s", cudaGetErrorString(e)); }
  L->parity = 0;
  release_graph(L);
  return OAL_OK;
}

oal_status kbc_set_state(KbcLevel* L, const double* f, const double* rho, const double* vel) {
  if (!L || !f) return fail(OAL_E_INVALID_ARG, "null argument");
  KBC_TRY(cudaSetDevice(L->device));
  KBC_TRY(cudaDeviceSynchronize());
  const int64_t nb = L->nb, ncell = nb * 512;
  std::vector<float> hf((size_t)ncell * Q);
  for (int64_t b = 0; b < nb; ++b)
    for (int k = 0; k < Q; ++k)
      for (int c = 0; c < 512; ++c) hf[(size_t)((b * Q + k) * 512 + c)] = (float)f[c + 512 * b + ncell * k];
  L->parity = 0;
  KBC_TRY(cudaMemcpy(L->f[0], hf.data(), hf.size() * sizeof(float), cudaMemcpyHostToDevice));
  if (rho) {
    std::vector<float> hr((size_t)ncell);
    for (int64_t i = 0; i < ncell; ++i) hr[(size_t)i] = (float)rho[i];
    KBC_TRY(cudaMemcpy(L->rho, hr.data(), hr.size() * sizeof(float), cudaMemcpyHostToDevice));
  }
  if (vel) {
    std::vector<float> hv((size_t)ncell * 3);
    for (int64_t i = 0; i < 3 * ncell; ++i) hv[(size_t)i] = (float)vel[i];
    KBC_TRY(cudaMemcpy(L->vel[0], hv.data(), hv.size() * sizeof(float), cudaMemcpyHostToDevice));
  }
  std::vector<float> nan((size_t)ncell * 13, std::numeric_limits<float>::quiet_NaN());
  KBC_TRY(cudaMemcpy(L->lam, nan.data(), nan.size() * sizeof(float), cudaMemcpyHostToDevice));
  release_graph(L);
  return OAL_OK;
}

oal_status kbc_get_state(KbcLevel* L, double* f, double* rho, double* vel) {
  if (!L) return fail(OAL_E_INVALID_ARG, "null level");
  KBC_TRY(cudaSetDevice(L->device));
  KBC_TRY(cudaDeviceSynchronize());
  const int64_t nb = L->nb, ncell = nb * 512;
  const int p = L->parity;
  if (f) {
    std::vector<float> hf((size_t)ncell * Q);
    KBC_TRY(cudaMemcpy(hf.data(), L->f[p], hf.size() * sizeof(float), cudaMemcpyDeviceToHost));
    for (int64_t b = 0; b < nb; ++b)
      for (int k = 0; k < Q; ++k)
        for (int c = 0; c < 512; ++c) f[c + 512 * b + ncell * k] = hf[(size_t)((b * Q + k) * 512 + c)];
  }
  if (rho) {
    std::vector<float> hr((size_t)ncell);
    KBC_TRY(cudaMemcpy(hr.data(), L->rho, hr.size() * sizeof(float), cudaMemcpyDeviceToHost));
    for (int64_t i = 0; i < ncell; ++i) rho[i] = hr[(size_t)i];
  }
  if (vel) {
    std::vector<float> hv((size_t)ncell * 3);
    KBC_TRY(cudaMemcpy(hv.data(), L->vel[p], hv.size() * sizeof(float), cudaMemcpyDeviceToHost));
    for (int64_t i = 0; i < 3 * ncell; ++i) vel[i] = hv[(size_t)i];
  }
  return OAL_OK;
}

oal_status kbc_lambda(KbcLevel* L, float* get, const float* set) {
  if (!L) return fail(OAL_E_INVALID_ARG, "null level");
  KBC_TRY(cudaSetDevice(L->device));
  KBC_TRY(cudaDeviceSynchronize());
  const int64_t nb = L->nb, ncell = nb * 512;
  std::vector<float> h((size_t)ncell * 13);
  if (get) {
    KBC_TRY(cudaMemcpy(h.data(), L->lam, h.size() * sizeof(float), cudaMemcpyDeviceToHost));
    for (int64_t b = 0; b < nb; ++b)
      for (int m = 0; m < 13; ++m)
        for (int c = 0; c < 512; ++c) get[c + 512 * b + ncell * m] = h[(size_t)((b * 13 + m) * 512 + c)];
  }
  if (set) {
    for (int64_t b = 0; b < nb; ++b)
      for (int m = 0; m < 13; ++m)
        for (int c = 0; c < 512; ++c) h[(size_t)((b * 13 + m) * 512 + c)] = set[c + 512 * b + ncell * m];
    KBC_TRY(cudaMemcpy(L->lam, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
    release_graph(L);
  }
  return OAL_OK;
}

oal_status kbc_step(KbcLevel* L, const oal_step_params* p, void* stream) {
  if (!L) return fail(OAL_E_INVALID_ARG, "null level");
  KbcArgs a;
  oal_status s = resolve(p, &a);
  if (s != OAL_OK) return s;
  KBC_TRY(cudaSetDevice(L->device));
  return enqueue(L, a, p, p->time_step_seed, static_cast<cudaStream_t>(stream));
}

oal_status kbc_advance(KbcLevel* L, const oal_step_params* p, int32_t n, void* stream) {
  if (!L) return fail(OAL_E_INVALID_ARG, "null level");
  if (n <= 0) return fail(OAL_E_INVALID_ARG, "n_steps must be positive");
  KbcArgs a;
  oal_status s = resolve(p, &a);
  if (s != OAL_OK) return s;
  KBC_TRY(cudaSetDevice(L->device));
  oal_step_params key = *p;
  if (!(p->inlet_turbulence > 0.0f && L->n_entries > 0)) key.time_step_seed = 0;  // the seed only feeds inlet noise
  KbcLevel::Graph& G = L->gr[L->parity];
  const bool hit = G.exec && G.n == n && std::memcmp(&G.p, &key, sizeof key) == 0;
  if (!hit) {
    release_graph(G);
    const int start = L->parity;
    KBC_TRY(cudaStreamBeginCapture(L->cap, cudaStreamCaptureModeThreadLocal));
    oal_status es = OAL_OK;
    for (int i = 0; i < n && es == OAL_OK; ++i) es = enqueue(L, a, p, p->time_step_seed + i, L->cap);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(L->cap, &graph);
    L->parity = start;
    if (es != OAL_OK) { if (graph) cudaGraphDestroy(graph); return es; }
    if (e != cudaSuccess) { cudaGetLastError(); return fail(OAL_E_CUDA, "graph capture: %s", cudaGetErrorString(e)); }
    cudaGraphExec_t exec = nullptr;
    e = cudaGraphInstantiate(&exec, graph, 0);
    if (e != cudaSuccess) {
      cudaGraphDestroy(graph);
      cudaGetLastError();
      return fail(OAL_E_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
    }
    G.exec = exec; G.graph = graph; G.n = n; G.p = key;
  }
  KBC_TRY(cudaGraphLaunch(G.exec, static_cast<cudaStream_t>(stream)));
  if (n & 1) L->parity ^= 1;
  return OAL_OK;
}

oal_status kbc_mass_momentum(KbcLevel* L, double out[4]) {
  if (!L || !out) return fail(OAL_E_INVALID_ARG, "null argument");
  KBC_TRY(cudaSetDevice(L->device));
  k_kbc_mm_part<<<(unsigned)L->nb, kThreads>>>(L->f[L->parity], L->nb, L->d_mm_part);
  KBC_TRY(cudaGetLastError());
  k_kbc_mm_final<<<1, 32>>>(L->d_mm_part, L->nb, L->d_mm);
  KBC_TRY(cudaGetLastError());
  KBC_TRY(cudaMemcpy(out, L->d_mm, 4 * sizeof(double), cudaMemcpyDeviceToHost));
  return OAL_OK;
}

oal_status kbc_device_state(KbcLevel* L, void** f, void** rho, void** vel) {
  if (!L) return fail(OAL_E_INVALID_ARG, "null level");
  if (f) *f = L->f[L->parity];
  if (rho) *rho = L->rho;
  if (vel) *vel = L->vel[L->parity];
  return OAL_OK;
}

int64_t kbc_device_bytes(const KbcLevel* L) { return L ? L->bytes : 0; }

oal_status kbc_layout(const KbcLevel* L, int64_t out[6]) {
  if (!L || !out) return fail(OAL_E_INVALID_ARG, "null argument");
  out[0] = 0; out[1] = out[2] = out[3] = 0; out[4] = (int64_t)Q * 512; out[5] = 512;
  return OAL_OK;
}
