// svv_d3q27.cu — spectral vanishing viscosity of the reference's D3Q27 levels
// (apply_svv_d3q19_postcollision!, src/collision/kernel_svv_yz_d3q39.jl:426-458, with
// apply_svv_d3q19_inline!, :301-375, and the tap helpers get_pop_neighbor_x / _yz, :225-250 and
// :78-116), launched after the step kernels (timestep.jl:1576-1611).
//
// For every fluid cell and direction k, the post-collision population f_k is filtered by the
// 5-point bi-Laplacian of the step's input populations along x (eps_x) and along y and z
// (eps_yz), the centre tap being f_k itself:
//   f_k' = f_k - eps_x (t-2 - 4 t-1 + 6 f_k - 4 t+1 + t+2)_x - eps_yz (...)_y - eps_yz (...)_z
// A tap in a solid cell or past a missing neighbour block reads the cell's own input population
// (a zero-flux wall for the operator). The 4-moment correction f_k' -= w_k (drho + c_k.dj / cs2)
// then restores the cell's mass and momentum, and every population is floored at 1e-12.
//
// One thread per cell, 256 per CTA (half a block; 128 in FP64). A population's address is linear in its
// direction in both layouts (block-major: b 27*512 + k 512 + cell; dense: cell + k PX PY PZ), so a
// thread resolves its twelve taps once — the neighbour block, the solid masks and the fall-back
// to its own slot — into twelve direction-0 offsets, and each direction then costs one load per
// tap (the block's rows, mostly L1 hits) and the arithmetic. The filtered populations wait in
// shared memory (the thread's own column) for the correction. HBM traffic per fluid cell: the
// 27 input populations once, the 27 output populations read and written.
#include <type_traits>

#include "svv_d3q27.h"
#include "vmath.cuh"

namespace oal {

namespace {

// one thread per cell: 256 per CTA (two per block), 128 for FP64 (the filtered populations of a
// CTA in shared memory stay within the 48 KB of static shared memory)
template <class R> constexpr int svv_threads() { return sizeof(R) == 8 ? 128 : 256; }

struct SvvArgs {
  PopIndex pi;
  const int32_t* __restrict__ nbr;    // [nb*27] 0-based, -1 = no neighbour
  int32_t n_real;
  const int32_t* __restrict__ mslot;  // per-block mask slot or -1
  const uint32_t* __restrict__ cmask; // bit 13: the cell itself is solid
  float eps_x, eps_yz;
};

__device__ __forceinline__ bool svv_solid(const SvvArgs& a, int64_t b, int cell) {
  if (!a.mslot) return false;
  const int32_t s = a.mslot[b];
  return s >= 0 && ((a.cmask[(int64_t)s * kCells + cell] >> 13) & 1u);
}

// the direction-0 offset of the input population at (x, y, z) + d along one axis, or `own`
template <class IDX>
__device__ __forceinline__ IDX svv_tap_offset(const SvvArgs& a, int b, int x, int y, int z, int dx, int dy, int dz,
                                              IDX own) {
  const int nx = x + dx, ny = y + dy, nz = z + dz;
  const int ox = nx < 0 ? -1 : (nx >= kBS ? 1 : 0), oy = ny < 0 ? -1 : (ny >= kBS ? 1 : 0),
            oz = nz < 0 ? -1 : (nz >= kBS ? 1 : 0);
  int32_t bb = b;
  if (ox | oy | oz) {
    bb = a.nbr[(int64_t)b * kQ27 + nbr_dir(ox, oy, oz)];
    if (bb < 0 || bb >= a.n_real) return own;
  }
  const int c = (nx & 7) | ((ny & 7) << 3) | ((nz & 7) << 6);
  if (svv_solid(a, bb, c)) return own;
  return (IDX)a.pi(bb, c, 0);
}

template <class S, class R, class IDX>
__global__ void __launch_bounds__(svv_threads<R>(), 3) k_svv(const SvvArgs a, const S* __restrict__ fin, S* __restrict__ fout,
                                                             S* __restrict__ fpost2) {
  constexpr int kT = svv_threads<R>(), kPer = kCells / kT;
  const int b = blockIdx.x / kPer;
  const int cell = (blockIdx.x % kPer) * kT + threadIdx.x;
  if (svv_solid(a, b, cell)) return;
  const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
  const IDX own = (IDX)a.pi(b, cell, 0);
  const IDX kst = (IDX)a.pi.kst;
  const bool fx = a.eps_x > 0.0f, fyz = a.eps_yz > 0.0f;
  // taps: x-2, x-1, x+1, x+2, then y, then z
  IDX t[12];
#pragma unroll
  for (int j = 0; j < 12; ++j) {
    const int axis = j >> 2, s = (j & 3) < 2 ? (j & 3) - 2 : (j & 3) - 1;
    const bool used = axis == 0 ? fx : fyz;
    t[j] = used ? svv_tap_offset<IDX>(a, b, x, y, z, axis == 0 ? s : 0, axis == 1 ? s : 0, axis == 2 ? s : 0, own)
                : own;
  }
  const R ex = R(a.eps_x), eyz = R(a.eps_yz);
  __shared__ R s_fl[kQ27][kT];  // the filtered populations until the correction
  R d_rho = R(0), d_jx = R(0), d_jy = R(0), d_jz = R(0);
#pragma unroll 3
  for (int k = 0; k < kQ27; ++k) {
    const R w = R(q27_w(k)), inv_w = R(1.0 / q27_w(k));
    const S* fk = fin + (IDX)k * kst;
    auto tap = [&](int j) { return Codec<S>::dec(fk[t[j]], w, inv_w); };
    const R fc = Codec<S>::dec(fout[own + (IDX)k * kst], w, inv_w);
    R bilap = R(0);
    if (fx) bilap += ex * ((((tap(0) - R(4) * tap(1)) + R(6) * fc) - R(4) * tap(2)) + tap(3));
    if (fyz) {
      bilap += eyz * ((((tap(4) - R(4) * tap(5)) + R(6) * fc) - R(4) * tap(6)) + tap(7));
      bilap += eyz * ((((tap(8) - R(4) * tap(9)) + R(6) * fc) - R(4) * tap(10)) + tap(11));
    }
    const R ff = fc - bilap;
    const R diff = ff - fc;
    d_rho += diff;
    d_jx += diff * R(q27_cx(k));
    d_jy += diff * R(q27_cy(k));
    d_jz += diff * R(q27_cz(k));
    s_fl[k][threadIdx.x] = ff;
  }
  const R inv_cs2 = R(1) / R(1.0 / 3.0);  // CS2_LATTICE
#pragma unroll
  for (int k = 0; k < kQ27; ++k) {
    const R w = R(q27_w(k)), inv_w = R(1.0 / q27_w(k));
    const R cu = R(q27_cx(k)) * d_jx + R(q27_cy(k)) * d_jy + R(q27_cz(k)) * d_jz;
    R v = s_fl[k][threadIdx.x] - w * (d_rho + inv_cs2 * cu);
    v = v < R(1e-12f) ? R(1e-12f) : v;  // NaN passes
    const S word = Codec<S>::enc(v, w, inv_w);
    fout[own + (IDX)k * kst] = word;
    if (fpost2) fpost2[own + (IDX)k * kst] = word;
  }
}

// ---- two x-adjacent cells per thread (block layout, FP32/FP16/BF16 storage) -------------------
// The same filter with one 32- or 64-bit load per tap pair: the y and z taps of cells (x, x+1)
// are adjacent words, and the x taps of the pair come from the pairs (x-2, x-1), (x, x+1) and
// (x+2, x+3). Each lane keeps its own fall-back flags (a solid target or a missing block selects
// the lane's own input population), so every lane computes exactly what the one-cell kernel does.
// W: the pair's stored word, read where the program reads it (a volatile load: the reads ahead of the
// filter below must not sink to their uses); dec: its two populations (f = w + w d for 16-bit deviations).
template <class S> struct PairIO;
template <> struct PairIO<float> {
  using W = uint2;
  static __device__ __forceinline__ W word(const float* p) {
    W v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
  }
  static __device__ __forceinline__ F2 dec(W v, float) { return f2(__uint_as_float(v.x), __uint_as_float(v.y)); }
  static __device__ __forceinline__ void store(float* p, F2 v, float) {
    float a, b;
    f2split(v, a, b);
    *reinterpret_cast<float2*>(p) = make_float2(a, b);
  }
};
template <> struct PairIO<__half> {
  using W = uint32_t;
  static __device__ __forceinline__ W word(const __half* p) {
    W v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  }
  static __device__ __forceinline__ F2 dec(W v, float w) {
    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&v));
    return vfma(splat<F2>(w), f2(h.x, h.y), splat<F2>(w));
  }
  static __device__ __forceinline__ void store(__half* p, F2 v, float inv_w) {
    float a, b;
    f2split(vfma(v, splat<F2>(inv_w), splat<F2>(-1.0f)), a, b);
    *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
  }
};
template <> struct PairIO<__nv_bfloat16> {
  using W = uint32_t;
  static __device__ __forceinline__ W word(const __nv_bfloat16* p) {
    W v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  }
  static __device__ __forceinline__ F2 dec(W v, float w) {
    const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
    return vfma(splat<F2>(w), f2(h.x, h.y), splat<F2>(w));
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, F2 v, float inv_w) {
    float a, b;
    f2split(vfma(v, splat<F2>(inv_w), splat<F2>(-1.0f)), a, b);
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
  }
};
// max(v, 1e-12) per lane that keeps a NaN
__device__ __forceinline__ float floor_pop(float v) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "f"(1e-12f));
  return r;
}
// the rounded product c v of both lanes by scalar multiplies: a packed multiply whose result a packed
// add consumes may be contracted into one packed FMA, a scalar one may not (-fmad=false)
__device__ __forceinline__ F2 scale2(float c, F2 v) {
  float a, b;
  f2split(v, a, b);
  return f2(c * a, c * b);
}

// the direction-0 offset of the pair starting at (x, y, z) + d (x + dx even), whether its block
// exists, and per lane whether the target cell is solid
template <class IDX>
__device__ __forceinline__ IDX svv_pair_offset(const SvvArgs& a, int b, int x, int y, int z, int dx, int dy, int dz,
                                               IDX own, bool& s0, bool& s1) {
  const int nx = x + dx, ny = y + dy, nz = z + dz;
  const int ox = nx < 0 ? -1 : (nx >= kBS ? 1 : 0), oy = ny < 0 ? -1 : (ny >= kBS ? 1 : 0),
            oz = nz < 0 ? -1 : (nz >= kBS ? 1 : 0);
  int32_t bb = b;
  if (ox | oy | oz) {
    bb = a.nbr[(int64_t)b * kQ27 + nbr_dir(ox, oy, oz)];
    if (bb < 0 || bb >= a.n_real) { s0 = s1 = true; return own; }
  }
  const int c = (nx & 7) | ((ny & 7) << 3) | ((nz & 7) << 6);
  s0 = svv_solid(a, bb, c);
  s1 = svv_solid(a, bb, c + 1);
  return s0 && s1 ? own : (IDX)a.pi(bb, c, 0);
}

// The filter of the 27 directions of a pair of cells, unrolled (weights, velocities and, in the
// library's layout (KST = 512), the directions' offsets are immediates), in packed f32x2 arithmetic
// with the oracle's rounding: products with 4 and with +-1 and 0 are exact, so their multiply-adds are
// one rounding either way; the other products are taken apart (scale2). Filtered values go to s_fl,
// the changes of mass and momentum to acc. PICK: some tap of the pair falls back in one lane only (a
// missing block or two solid cells give the pair's own offset instead).
template <class S, class IDX, bool PICK, int KST, bool X>
__device__ __forceinline__ void svv_pairs_filter(const SvvArgs& a, const S* __restrict__ fin, const S* __restrict__ fout,
                                                 IDX own, const IDX (&t)[10], uint32_t fb, bool fx, bool fyz_x,
                                                 F2 (*s_fl)[128], F2 (&acc)[4]) {
  const float ex = a.eps_x, eyz = a.eps_yz;
  const IDX kst = KST ? (IDX)KST : (IDX)a.pi.kst;
  const bool fyz = !X || fyz_x;  // X = false: y and z taps only, no branch in the loop
  using IO = PairIO<S>;
  using W = typename IO::W;
  const F2 m4 = splat<F2>(-4.0f);
#pragma unroll
  for (int m = 0; m < 4; ++m) acc[m] = splat<F2>(0.0f);
  // the words of a direction: own input, own output, the eight y and z taps, the two x pairs; those of
  // the next directions are on their way while one is filtered (one direction at a time the warps
  // spent two thirds of their time waiting for its ten reads)
  // two (FP32: one) ahead already spill a little at 96 (128) registers: 52 bytes stored, 60 loaded in the
  // FP16 y-z instance; three 72 and 80. With a run-time stride none is read ahead (104 and 120 at most,
  // 64-bit offsets 212 and 356)
  constexpr int kAhead = KST == 0 ? 0 : sizeof(S) == 2 ? 2 : 1;
  W q[kAhead + 1][12];
  auto fetch = [&](int k, W (&d)[12]) {
    const S* fk = fin + (IDX)k * kst;
    d[0] = IO::word(fk + own);
    d[1] = IO::word(fout + own + (IDX)k * kst);
    if (fyz)
#pragma unroll
      for (int j = 0; j < 8; ++j) d[2 + j] = IO::word(fk + t[2 + j]);
    if (X && fx) { d[10] = IO::word(fk + t[0]); d[11] = IO::word(fk + t[1]); }
  };
#pragma unroll
  for (int k = 0; k < kAhead; ++k) fetch(k, q[k]);  // none where kAhead is 0
#pragma unroll
  for (int k = 0; k < kQ27; ++k) {
    const float w = float(q27_w(k));
    if (k + kAhead < kQ27) fetch(k + kAhead, q[(k + kAhead) % (kAhead + 1)]);
    const W (&d)[12] = q[k % (kAhead + 1)];
    const F2 o = IO::dec(d[0], w);  // the pair's own input populations
    const F2 fc = IO::dec(d[1], w);
    const F2 six = scale2(6.0f, fc);
    // lane 0 takes bit, lane 1 bit + 1 of fb
    auto pick = [&](int bit, F2 v, F2 mine) {
      if constexpr (PICK)
        return f2(((fb >> bit) & 1u) ? f2lo(mine) : f2lo(v), ((fb >> (bit + 1)) & 1u) ? f2hi(mine) : f2hi(v));
      else return v;
    };
    auto lap = [&](F2 t0, F2 t1, F2 t2, F2 t3) { return vfma(m4, t2, vfma(m4, t1, t0) + six) + t3; };
    F2 bl = splat<F2>(0.0f);
    if (X && fx) {
      // x - 2, x - 1, x + 1, x + 2 of the two lanes from the pairs (x-2, x-1), (x, x+1), (x+2, x+3)
      const F2 m = IO::dec(d[10], w), p = IO::dec(d[11], w);
      bl = scale2(ex, lap(pick(0, m, o), pick(2, f2(f2hi(m), f2lo(o)), o), pick(4, f2(f2hi(o), f2lo(p)), o), pick(6, p, o)));
    }
    if (fyz) {
#pragma unroll
      for (int a2 = 0; a2 < 2; ++a2) {
        const int j0 = 2 + 4 * a2, bit = 8 + 8 * a2;
        bl = bl + scale2(eyz, lap(pick(bit, IO::dec(d[j0], w), o), pick(bit + 2, IO::dec(d[j0 + 1], w), o),
                                  pick(bit + 4, IO::dec(d[j0 + 2], w), o), pick(bit + 6, IO::dec(d[j0 + 3], w), o)));
      }
    }
    const F2 f = fc - bl, e = f - fc;
    acc[0] = acc[0] + e;
    acc[1] = vfma(e, splat<F2>(float(q27_cx(k))), acc[1]);
    acc[2] = vfma(e, splat<F2>(float(q27_cy(k))), acc[2]);
    acc[3] = vfma(e, splat<F2>(float(q27_cz(k))), acc[3]);
    s_fl[k][threadIdx.x] = f;
  }
}

// Bound by the latency of its DRAM reads: a direction's own input and output words come from DRAM, so
// the bandwidth follows from the directions a warp has in flight. On the 256 x 128 x 128 channel in
// FP16, y-z taps: 651 us with the directions in a loop that formed weights, velocities and addresses at
// run time (290 instructions per pair and direction), 515 us unrolled and packed (~80), 365 us with two
// directions read ahead at 20 warps per SM. The domain faces take the path without selects, because a
// missing block's taps already point at the pair itself.
// X: the x filter is on (then both axes' switches are run-time).
template <class S, class IDX, int KST, bool X>
__global__ void __launch_bounds__(128, sizeof(S) == 4 ? 4 : 5) k_svv_pairs(const SvvArgs a, const S* __restrict__ fin, S* __restrict__ fout,
                                                      S* __restrict__ fpost2) {
  const int b = blockIdx.x >> 1;
  const int base = (blockIdx.x & 1) << 8;
  const int l0 = threadIdx.x << 1;  // the pair's first cell within the CTA's half block
  const int c0 = base + l0;
  const int x = c0 & 7, y = (c0 >> 3) & 7, z = c0 >> 6;
  const bool d0 = svv_solid(a, b, c0), d1 = svv_solid(a, b, c0 + 1);
  if (d0 && d1) return;
  const IDX own = (IDX)a.pi(b, c0, 0);
  const IDX kst = KST ? (IDX)KST : (IDX)a.pi.kst;
  const bool fx = X && a.eps_x > 0.0f, fyz = !X || a.eps_yz > 0.0f;
  // pair taps: 0 (x-2, x-1), 1 (x+2, x+3), 2-5 y-2, y-1, y+1, y+2, 6-9 z-2 .. z+2; fb bit 2j + lane:
  // the lane takes its own input population for tap j (x taps: j 0-3 of the lane's x-2 .. x+2)
  IDX t[10];
  uint32_t fb = 0;
  bool m0, m1, p0, p1;
  t[0] = fx ? svv_pair_offset<IDX>(a, b, x, y, z, -2, 0, 0, own, m0, m1) : own;
  t[1] = fx ? svv_pair_offset<IDX>(a, b, x, y, z, 2, 0, 0, own, p0, p1) : own;
  if (fx) {
    // lane 0 (x): x-2, x-1, x+1 (the pair's second cell), x+2; lane 1 (x+1): x-1, x, x+2, x+3
    fb |= (uint32_t)m0 << 0 | (uint32_t)m1 << 2 | (uint32_t)d1 << 4 | (uint32_t)p0 << 6;
    fb |= (uint32_t)m1 << 1 | (uint32_t)d0 << 3 | (uint32_t)p0 << 5 | (uint32_t)p1 << 7;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int s = (j & 3) < 2 ? (j & 3) - 2 : (j & 3) - 1;
    bool q0 = true, q1 = true;
    t[2 + j] = fyz ? svv_pair_offset<IDX>(a, b, x, y, z, 0, j < 4 ? s : 0, j < 4 ? 0 : s, own, q0, q1) : own;
    if (q0 != q1) fb |= (uint32_t)q0 << (8 + 2 * j) | (uint32_t)q1 << (9 + 2 * j);
  }
  __shared__ F2 s_fl[kQ27][128];
  F2 acc[4];
  // the fall-back selects only where one lane of a tap falls back (cells next to a solid; x taps also
  // next to a missing block); elsewhere the loads are used as they are
  if (fb == 0) svv_pairs_filter<S, IDX, false, KST, X>(a, fin, fout, own, t, fb, fx, fyz, s_fl, acc);
  else svv_pairs_filter<S, IDX, true, KST, X>(a, fin, fout, own, t, fb, fx, fyz, s_fl, acc);
  const float inv_cs2 = 1.0f / float(1.0 / 3.0);  // CS2_LATTICE
#pragma unroll
  for (int k = 0; k < kQ27; ++k) {
    const float w = float(q27_w(k)), inv_w = float(1.0 / q27_w(k));
    // (cx jx + cy jy) + cz jz: exact products
    const F2 cu = vfma(splat<F2>(float(q27_cz(k))), acc[3],
                       vfma(splat<F2>(float(q27_cy(k))), acc[2], scale2(float(q27_cx(k)), acc[1])));
    const F2 v = s_fl[k][threadIdx.x] - scale2(w, acc[0] + scale2(inv_cs2, cu));
    const float v0 = floor_pop(f2lo(v)), v1 = floor_pop(f2hi(v));
    // a solid cell of the pair keeps its stored word
    if (d0 || d1) {
      S* q = fout + own + (IDX)k * kst;
      S* q2 = fpost2 ? fpost2 + own + (IDX)k * kst : nullptr;
      if (!d0) { q[0] = Codec<S>::enc(v0, w, inv_w); if (q2) q2[0] = q[0]; }
      if (!d1) { q[1] = Codec<S>::enc(v1, w, inv_w); if (q2) q2[1] = q[1]; }
    } else {
      PairIO<S>::store(fout + own + (IDX)k * kst, f2(v0, v1), inv_w);
      if (fpost2) PairIO<S>::store(fpost2 + own + (IDX)k * kst, f2(v0, v1), inv_w);
    }
  }
}

template <class S, class R>
cudaError_t enqueue_t(const SvvArgs& a, const void* fin, void* fout, void* fpost2, int32_t nb, int64_t n_elements,
                      cudaStream_t st) {
  constexpr int kT = svv_threads<R>();
  const unsigned grid = (unsigned)nb * (unsigned)(kCells / kT);
  const S* in = static_cast<const S*>(fin);
  S* out = static_cast<S*>(fout);
  S* post = static_cast<S*>(fpost2);
  if constexpr (sizeof(R) == 4) {
    // pairs of x-adjacent cells are aligned words where the strides are even and the arrays start
    // on a word (every block layout this library allocates; a caller's arrays are checked)
    auto aligned = [](const void* p) { return p == nullptr || ((uintptr_t)p % (2 * sizeof(S))) == 0; };
    if (!a.pi.dense && a.pi.bst % 2 == 0 && a.pi.kst % 2 == 0 && aligned(fin) && aligned(fout) && aligned(fpost2)) {
      const bool idx32 = n_elements < (int64_t(1) << 32), own_layout = a.pi.kst == kCells;
      const unsigned ctas = (unsigned)nb * 2u;
      auto go = [&](auto x_on) {
        constexpr bool X = decltype(x_on)::value;
        if (own_layout && idx32) k_svv_pairs<S, uint32_t, kCells, X><<<ctas, 128, 0, st>>>(a, in, out, post);
        else if (own_layout) k_svv_pairs<S, int64_t, kCells, X><<<ctas, 128, 0, st>>>(a, in, out, post);
        else if (idx32) k_svv_pairs<S, uint32_t, 0, X><<<ctas, 128, 0, st>>>(a, in, out, post);
        else k_svv_pairs<S, int64_t, 0, X><<<ctas, 128, 0, st>>>(a, in, out, post);
      };
      if (a.eps_x > 0.0f) go(std::true_type{});
      else go(std::false_type{});
      return cudaGetLastError();
    }
  }
  if (n_elements < (int64_t(1) << 32))
    k_svv<S, R, uint32_t><<<grid, kT, 0, st>>>(a, in, out, post);
  else
    k_svv<S, R, int64_t><<<grid, kT, 0, st>>>(a, in, out, post);
  return cudaGetLastError();
}

}  // namespace

cudaError_t svv_enqueue(int32_t storage, const void* f_in, void* f_out, const PopIndex& pi, int32_t nb,
                        int64_t n_elements, const int32_t* nbr, int32_t n_real, const int32_t* mslot,
                        const uint32_t* cmask, float eps_x, float eps_yz, cudaStream_t st, void* f_post2) {
  if ((eps_x == 0.0f && eps_yz == 0.0f) || nb <= 0) return cudaSuccess;
  SvvArgs a;
  a.pi = pi; a.nbr = nbr; a.n_real = n_real; a.mslot = cmask ? mslot : nullptr; a.cmask = cmask;
  a.eps_x = eps_x; a.eps_yz = eps_yz;
  switch (storage) {
    case 0: return enqueue_t<float, float>(a, f_in, f_out, f_post2, nb, n_elements, st);
    case 1: return enqueue_t<__half, float>(a, f_in, f_out, f_post2, nb, n_elements, st);
    case 2: return enqueue_t<__nv_bfloat16, float>(a, f_in, f_out, f_post2, nb, n_elements, st);
    case 3: return enqueue_t<double, double>(a, f_in, f_out, f_post2, nb, n_elements, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace oal
