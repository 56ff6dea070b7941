// Device-side helpers: nonuniform point generation and kernel taps.
#pragma once

#include "cov3d_internal.cuh"

namespace cov3d {

__device__ __forceinline__ int pmod(int a, int n) {
  int r = a % n;
  return r < 0 ? r + n : r;
}

// a mod n for a in [-n, 2n): the window corners of wrapped points.
__device__ __forceinline__ int wrap1(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// torch.remainder(x + pi, 2 pi) - pi in float32 (poses.py:259-261, nufft_plan.py:327).
__device__ __forceinline__ float wrap_pi(float x) {
  const float two_pi = 6.28318530717958647692f;
  float a = __fadd_rn(x, kPiF);
  // floor(a / (2 pi)) without the division for the one turn that central slices make
  float q = a >= 0.0f && a < two_pi ? 0.0f : a >= two_pi && a < 12.0f ? 1.0f : a < 0.0f && a > -6.0f ? -1.0f
                                                                              : floorf(__fdiv_rn(a, two_pi));
  float r = __fsub_rn(a, __fmul_rn(q, two_pi));
  return __fsub_rn(r, kPiF);
}

// Normalised plane coordinate ceil(i - Lp/2) / (Lp/2) in float32 (ASPIRE grid definition used
// by poses.py:197-213), times float32(pi).
__device__ __forceinline__ float plane_coord(int i, const PointGeom &g) {
  float k = ceilf((float)i - 0.5f * (float)g.Lp);
  return __fmul_rn(kPiF, __fdiv_rn(k, g.plane_half));
}

// Frequency (radians) of point `id` along volume axes 0, 1, 2.
// (ids are below 2^30: 32-bit divisions)
__device__ __forceinline__ void point_freq(const PointGeom &g, int id, float w[3]) {
  const int64_t b = (unsigned)id / (unsigned)g.P;
  const int p = id - (int)b * g.P;
  if (g.kind == kPointsExplicit) {
    const float *base = g.pts + b * 3 * (int64_t)g.P + p;
    w[0] = __ldg(base);
    w[1] = __ldg(base + g.P);
    w[2] = __ldg(base + 2 * (int64_t)g.P);
    if (g.wrap) {
      w[0] = wrap_pi(w[0]);
      w[1] = wrap_pi(w[1]);
      w[2] = wrap_pi(w[2]);
    }
  } else {
    const float *R = g.rot + b * 9;
    const int row = (unsigned)p / (unsigned)g.Lp;
    const int col = p - row * g.Lp;
    const float x = plane_coord(col, g);
    const float y = plane_coord(row, g);
    // pts = flip_axis0(R @ [x, y, 0]): axis 0 <- row 2 of R, axis 2 <- row 0 of R
    w[0] = wrap_pi(__fadd_rn(__fmul_rn(__ldg(R + 6), x), __fmul_rn(__ldg(R + 7), y)));
    w[1] = wrap_pi(__fadd_rn(__fmul_rn(__ldg(R + 3), x), __fmul_rn(__ldg(R + 4), y)));
    w[2] = wrap_pi(__fadd_rn(__fmul_rn(__ldg(R + 0), x), __fmul_rn(__ldg(R + 1), y)));
  }
}

// Fractional centered-grid index of a frequency, in float32.
__device__ __forceinline__ float freq_to_index(const PointGeom &g, float w) {
  if (g.mapping == kMapES) {
    return __fadd_rn(__fmul_rn(w, g.s_es), g.half_n);
  }
  // NufftPlanDiscretized.setpts scaling (nufft_plan.py:113-116), then grid_sample's
  // align_corners unnormalisation ((x + 1) / 2) * (n - 1).
  float x = __fadd_rn(__fmul_rn(w, g.gs_scale), g.gs_off);
  return __fmul_rn(__fmul_rn(__fadd_rn(x, 1.0f), 0.5f), (float)(g.n - 1));
}

__device__ __forceinline__ void point_index(const PointGeom &g, int id, float t[3]) {
  float w[3];
  point_freq(g, id, w);
  t[0] = freq_to_index(g, w[0]);
  t[1] = freq_to_index(g, w[1]);
  t[2] = freq_to_index(g, w[2]);
}

// Records of kSortHalf hold their indices as integers in units of 2^-frac cell, with as many
// fraction bits as leave room for the grid (22 at n = 256): mirrored points then have exactly
// mirrored indices, and a float index of a 256^3 grid is only good to 1.5e-5 cells (white volumes
// project to 1e-6 of the 64-bit result with the integers, to 1.1e-5 with the floats).
constexpr int kDeadIndex = -2147483647 - 1;  // NaN or outside the grid
constexpr int kRotShift = 40;  // rotation coefficients: cells per pixel step, in units of 2^-40
constexpr long long kDeadCoef = -9223372036854775807LL - 1;

// Index of point `id` along axes 0..2.  Rotations: R @ [kx, ky, 0] n / Lp from the image's integer
// coefficients, wrapped to [-n/2, n/2).  Explicit points: w n / (2 pi) with the product's rounding
// error carried along, wrapped when the kernel is periodic or the plan says so.
template <int KT>
__device__ __forceinline__ void point_index_fix(const PointGeom &g, int id, int t[3]) {
  const int one = 1 << g.frac;
  const int64_t b = (unsigned)id / (unsigned)g.P;
  const int p = id - (int)b * g.P;
  const int N = g.n << g.frac, c = (g.n / 2) << g.frac;
  if (g.kind == kPointsRotations) {
    const long long *A = g.rotc + b * 6;
    const int row = (unsigned)p / (unsigned)g.Lp;
    const int kx = p - row * g.Lp - g.Lp / 2, ky = row - g.Lp / 2;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const long long ax = __ldg(A + 2 * d), ay = __ldg(A + 2 * d + 1);
      long long u = ax * kx + ay * ky;
      u = (u + (1LL << (kRotShift - g.frac - 1))) >> (kRotShift - g.frac);
      if (u >= N / 2) u -= N;
      if (u < -(N / 2)) u += N;
      if (u >= N / 2 || u < -(N / 2)) {  // not a rotation: several turns
        u = (u + N / 2) % N;
        u = (u < 0 ? u + N : u) - N / 2;
      }
      t[d] = ax == kDeadCoef || ay == kDeadCoef ? kDeadIndex : (int)u + c;
    }
    return;
  }
  const float *base = g.pts + b * 3 * (int64_t)g.P + p;
  const float fn = (float)g.n;
  const bool wrap = KT == COV3D_KERNEL_ES || g.wrap;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float w = __ldg(base + d * (int64_t)g.P);
    float u = w * g.s_es;
    float e = fmaf(w, g.s_es, -u) + w * g.s_es_lo;
    if (wrap) {
      if (fabsf(u) < 8.0f * fn) {
        u = fmaf(-rintf(u / fn), fn, u);
      } else {  // many turns (or NaN, infinite: dead below)
        const double v = fmod((double)w * ((double)g.s_es + (double)g.s_es_lo), (double)g.n);
        u = (float)v;
        e = (float)(v - (double)u);
        if (fabsf(u) > 0.5f * fn) u -= copysignf(fn, u);
      }
    }
    const float ip = rintf(u);
    e += u - ip;
    if (!(fabsf(ip) <= 0.5f * fn + 4.0f) || !(fabsf(e) <= 2.0f)) {
      t[d] = kDeadIndex;
      continue;
    }
    int v = (int)ip * one + __float2int_rn(e * (float)one);
    if (wrap) {
      if (v >= N / 2) v -= N;
      if (v < -(N / 2)) v += N;
    }
    t[d] = v + c;
  }
}

// First cell of a point's window along one axis, from a float index ...
template <int KT, int W>
__device__ __forceinline__ int first_cell(float t) {
  if (KT == COV3D_KERNEL_NEAREST) return (int)rintf(t);
  if (KT == COV3D_KERNEL_LINEAR) return (int)floorf(t);
  return (int)ceilf(t - 0.5f * (float)W);
}
// ... and from an integer one
template <int KT, int W>
__device__ __forceinline__ int first_cell_fix(int t, int frac) {
  if (KT != COV3D_KERNEL_ES) return t >> frac;
  const int one = 1 << frac;
  return W % 2 == 0 ? ((t + (one - 1)) >> frac) - W / 2 : ((t + (one / 2 - 1)) >> frac) - (W - 1) / 2;
}

// ES kernel value exp(beta * (sqrt(1 - (2x/W)^2) - 1)) for |x| < W/2, else 0, with the fast
// hardware exponential and reciprocal square root (relative error ~1e-6, far below the ES
// approximation error of the NUFFT).
template <int W>
__device__ __forceinline__ float es_weight(float x, float beta) {
  const float y = x * (2.0f / (float)W);
  const float u = 1.0f - y * y;
  return u > 0.0f ? __expf(beta * (u * rsqrtf(u) - 1.0f)) : 0.0f;
}

// Sorted point record written by the sort: grid indices along axes 0..2 (floats, or the bits of
// point_index_fix's integers in records of kSortHalf) and the
// point id, with kNyquistBit set when the point lies on the Nyquist row / column of an
// even-sized image (vol_forward zeroes those pixels, projection_funcs.py:355-358).  Records of
// kSortHalf may also stand for the mirror pixel -k of the id's k (kPairBit; the values there are
// the conjugates), or hold the position of -k instead of the id's own (kConjBit, also with
// kPairBit clear); ids are below 2^29 there, and below 2^30 in kSortFull, which sets neither.
struct SortedPoint {
  float t0, t1, t2;
  unsigned idf;
};
constexpr unsigned kNyquistBit = 1u << 31;
constexpr unsigned kPairBit = 1u << 30;
constexpr unsigned kConjBit = 1u << 29;
// kHalf: the records are of kSortHalf
template <bool HALF>
__device__ __forceinline__ int sp_id(unsigned idf) {
  return (int)(idf & (HALF ? kConjBit - 1 : kPairBit - 1));
}
__device__ __forceinline__ bool sp_nyquist(unsigned idf) { return (idf & kNyquistBit) != 0; }
template <bool HALF>
__device__ __forceinline__ bool sp_pair(unsigned idf) {
  return HALF && (idf & kPairBit) != 0;
}
template <bool HALF>
__device__ __forceinline__ bool sp_conj(unsigned idf) {
  return HALF && (idf & kConjBit) != 0;
}

// Pixel holding -k of pixel p's k on the Lp x Lp image lattice, or -1 (Nyquist row or column of an
// even-sized image); p itself at the centre.
__device__ __forceinline__ int mirror_pixel(int p, int Lp) {
  if (Lp % 2 != 0) return Lp * Lp - 1 - p;
  return (p < Lp || (unsigned)p % (unsigned)Lp == 0) ? -1 : Lp * (Lp + 1) - p;
}
// id of the mirror pixel of a pair's id
__device__ __forceinline__ int mirror_id(const PointGeom &g, int id) {
  const int p = (unsigned)id % (unsigned)g.P;
  return id + (g.Lp % 2 != 0 ? g.P - 1 : g.P + g.Lp) - 2 * p;
}

__device__ __forceinline__ bool on_nyquist(const PointGeom &g, int id) {
  if (g.Lp % 2 != 0) return false;
  const int p = (unsigned)id % (unsigned)g.P;
  return p < g.Lp || ((unsigned)p % (unsigned)g.Lp) == 0;
}

// First cell of the window of a record's index t, and the weight of its tap q (0 <= q < W).
template <int KT, int W, bool HALF>
__device__ __forceinline__ int record_cell(float t, int frac) {
  return HALF ? first_cell_fix<KT, W>(__float_as_int(t), frac) : first_cell<KT, W>(t);
}
// Offset of a record's index t from cell c, in cells.
template <bool HALF>
__device__ __forceinline__ float record_offset(float t, int c, int frac) {
  return HALF ? (float)(__float_as_int(t) - (c << frac)) * __int_as_float((127 - frac) << 23) : t - (float)c;
}
template <int KT, int W, bool HALF>
__device__ __forceinline__ float record_weight(float t, int c0, int q, int frac, float beta) {
  if (KT == COV3D_KERNEL_NEAREST) return 1.0f;
  if (HALF) {  // the offset, of at most W / 2 cells, is exact from n = 256 on and rounded to 24 bits on smaller grids
    const float x = record_offset<true>(t, c0, frac);
    if (KT == COV3D_KERNEL_LINEAR) return q == 0 ? 1.0f - x : x;
    return es_weight<W>(x - (float)q, beta);
  }
  if (KT == COV3D_KERNEL_LINEAR) {
    const float f0 = floorf(t);
    return q == 0 ? (f0 + 1.0f) - t : t - f0;
  }
  return es_weight<W>(t - (float)(c0 + q), beta);
}

// Kernel taps along one axis: window cells c0 .. c0+W-1 and their weights.
template <int KT, int W, bool HALF>
__device__ __forceinline__ int taps(float t, int frac, float beta, float *wt) {
  const int c0 = record_cell<KT, W, HALF>(t, frac);
#pragma unroll
  for (int j = 0; j < W; ++j) wt[j] = record_weight<KT, W, HALF>(t, c0, j, frac, beta);
  return c0;
}

// Groups of neighbouring window corners along axis 2: the windows of the GS corners of a group lie in
// the same COLS (8, or all) of the T = 8 + W - 1 columns of a bin's tile.
template <int W, int COLUMNS = 8>
struct TileGroups {
  static constexpr int T = 8 + W - 1;
  static constexpr int COLS = COLUMNS;
  static constexpr int GS = COLS + 1 - W < 8 ? COLS + 1 - W : 8;  // corners per group
  static constexpr int NG = (8 + GS - 1) / GS;
  __device__ static constexpr int base(int g) {  // first tile column of the group's
    return g * GS < T - COLS ? g * GS : T - COLS;
  }
};

// Adds x to a cell of a grid.  (Spelled out: with its result unused, atomicAdd on a float2 took up to
// twice the kernel's time, depending on the code around it.)
__device__ __forceinline__ void add_cell(float2 *cell, float2 x) {
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(__cvta_generic_to_global(cell)), "f"(x.x), "f"(x.y) : "memory");
}

// CTF at pixel offsets (ka, kb) (row, column) from the image centre: sqrt(1 - w^2) sin(gamma) -
// w cos(gamma) with gamma = c0 K + c1 D + c2 X + d K^2 - ps (see CtfCoef).  gamma reaches a few
// hundred radians at high frequency, so its large terms are formed in double-float arithmetic
// (exact products by fmaf, TwoSum), reduced modulo 2 pi by Cody-Waite with a 2 pi split into a
// 12-bit head (n * head exact for |n| < 2^12) and a float tail, and only the reduced angle goes
// to sincosf: the absolute phase error stays near float rounding of the reduced angle.
__device__ __forceinline__ float ctf_eval(const CtfCoef &c, int ka, int kb) {
  const float K = (float)(ka * ka + kb * kb), D = (float)(ka * ka - kb * kb), X = (float)(2 * ka * kb);
  const float p0 = c.c0h * K, e0 = fmaf(c.c0h, K, -p0);
  const float p1 = c.c1h * D, e1 = fmaf(c.c1h, D, -p1);
  const float p2 = c.c2h * X, e2 = fmaf(c.c2h, X, -p2);
  float s = p0 + p1;
  float bb = s - p0;
  float err = (p0 - (s - bb)) + (p1 - bb);
  const float t = s + p2;
  bb = t - s;
  err += (s - (t - bb)) + (p2 - bb);
  const float lo = err + e0 + e1 + e2 + fmaf(c.c0l, K, fmaf(c.c1l, D, c.c2l * X)) + c.d * K * K - c.ps;
  constexpr float kTwoPiHead = 6.283203125f;          // 3217 / 512
  constexpr float kTwoPiTail = -1.7817820413e-05f;    // 2 pi - head
  constexpr float kInvTwoPi = 0.15915494309189535f;
  const float nq = rintf((t + lo) * kInvTwoPi);
  float r = fmaf(-nq, kTwoPiHead, t);
  r = fmaf(-nq, kTwoPiTail, r) + lo;
  float sn, cs;
  sincosf(r, &sn, &cs);
  return c.sw * sn - c.w * cs;
}

// The CTF factor of point id: the per-pixel array, or the per-image coefficients, or 1.
__device__ __forceinline__ float ctf_factor(const float *ctf, const CtfCoef *ctfc, const PointGeom &g, int id) {
  if (ctf) return __ldg(ctf + id);
  if (!ctfc) return 1.0f;
  const int b = (unsigned)id / (unsigned)g.P;
  const int p = id - b * g.P;
  const int row = (unsigned)p / (unsigned)g.Lp, col = p - row * g.Lp;
  return ctf_eval(ctfc[b], row - g.Lp / 2, col - g.Lp / 2);
}

// The mean's two spread values of a pixel: y * exp(-i (gx sx + gy sy)) * c * ctf (the image
// phase-shifted by -offset, mean.py:201-204) and (c * ctf)^2 / L (the kernel, whose extra 1/L is
// mean.py:215); gx, gy = ceil(k - L/2) 2 pi / L (poses.py:70-89).
__device__ __forceinline__ void mean_value(const MeanSource &s, int id, int P, int L, float2 &v0, float &v1) {
  const int b = (unsigned)id / (unsigned)P;
  const int p = id - b * P;
  float f = s.ctf ? __ldg(s.ctf + id) : 1.0f;
  if (s.contrasts) f *= __ldg(s.contrasts + b);
  float2 y = __ldg(s.images + id);
  if (s.offsets) {
    const int row = (unsigned)p / (unsigned)L, col = p - row * L;
    const float half = 0.5f * (float)L;
    const float gx = __fdiv_rn(__fmul_rn(__fmul_rn(ceilf((float)col - half), 2.0f), kPiF), (float)L);
    const float gy = __fdiv_rn(__fmul_rn(__fmul_rn(ceilf((float)row - half), 2.0f), kPiF), (float)L);
    const float sx = -__ldg(s.offsets + 2 * b), sy = -__ldg(s.offsets + 2 * b + 1);
    const float arg = __fadd_rn(__fmul_rn(gx, sx), __fmul_rn(gy, sy));
    float sn, cs;
    sincosf(arg, &sn, &cs);
    y = make_float2(y.x * cs - y.y * sn, y.x * sn + y.y * cs);
  }
  v0 = make_float2(y.x * f, y.y * f);
  v1 = f * f / (float)L;
}

// Sums of products of floats, no less precise than FP64 and of its range: exact products and their exact
// sum's leading 70 bits in three floats (TwoProd, TwoSum), and the products that floats cannot hold
// exactly, outside 2^-96 .. 2^100, in FP64.  (The FP64 pipe takes two operations per clock and SM: an
// iteration of the mean's CG at L = 128 takes 236 us with every term formed there, 210 here; 191 in pairs of
// floats, 46 bits, whose products lose the range as well.)
struct WideSum {
  float h = 0.0f, m = 0.0f, l = 0.0f;
  double w = 0.0;
  __device__ __forceinline__ static float two_sum(float &s, float x) {  // s + x = s' + the result
    const float t = __fadd_rn(s, x), b = __fsub_rn(t, s);
    const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b));
    s = t;
    return e;
  }
  __device__ __forceinline__ void add_product(float a, float b) {
    const float p = __fmul_rn(a, b);
    if (!(fabsf(p) > 1.2621774e-29f && fabsf(p) < 1.2676506e30f) && a != 0.0f && b != 0.0f) {
      w += (double)a * (double)b;
      return;
    }
    const float e = two_sum(m, __fmaf_rn(a, b, -p)), t = two_sum(h, p);
    l = __fadd_rn(l, __fadd_rn(e, two_sum(m, t)));
  }
  __device__ __forceinline__ double warp_sum() {  // every lane
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float xh = __shfl_xor_sync(0xffffffffu, h, o), xm = __shfl_xor_sync(0xffffffffu, m, o);
      const float xl = __shfl_xor_sync(0xffffffffu, l, o);
      const float t = two_sum(h, xh), e = two_sum(m, xm);
      l = __fadd_rn(__fadd_rn(l, xl), __fadd_rn(e, two_sum(m, t)));
    }
    double v = (double)h + ((double)m + (double)l);
    if (__any_sync(0xffffffffu, w != 0.0)) {  // (also NaN)
      double x = w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      v += x;
    }
    return v;
  }
};

// The next iteration of the CG begins: its direction is formed, the sums of its inner products start.
__device__ __forceinline__ void roll_scalars(CgState *st) {
  st->rz = st->rz_new;
  st->rr = st->rr_new;
  st->rz_new = 0.0;
  st->rr_new = 0.0;
  st->pap[0] = 0.0;
  st->pap[1] = 0.0;
  st->running += 1;
}

// Index maps of the fine grid (FFT-native storage: frequency / voxel offset k at k mod n).
// centered index of storage index s on a grid of size m (fftshift)
__device__ __forceinline__ int native_to_centered(int s, int m) {
  const int c = s + m / 2;
  return c >= m ? c - m : c;
}
// voxel index (0 .. L-1) of storage index s on a zero-padded axis, or -1 for padding
__device__ __forceinline__ int pad_voxel(int s, int L, int n) {
  const int h = L / 2;
  return s < L - h ? s + h : (s >= n - h ? s - n + h : -1);
}
// storage index of voxel j
__device__ __forceinline__ int voxel_store(int j, int L, int n) {
  const int k = j - L / 2;
  return k < 0 ? k + n : k;
}

}  // namespace cov3d
