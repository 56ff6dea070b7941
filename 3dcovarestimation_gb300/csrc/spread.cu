// Spreading ("type-1" half of the NUFFT; the exact adjoint of interp.cu over the same records,
// replacing the reference's grid_sample backward with FP32 global atomics, nufft_plan.py:171-242), over
// the bin-sorted point records of points_sort.cu, whose two views differ by up to 6e-5 cells.  See spread_tile_kernel (ES and linear windows) and
// spread_nearest_kernel for the decompositions.

#include "cov3d_device.cuh"

namespace cov3d {

namespace {

constexpr int kBin = 8;

struct SpreadParams {
  PointGeom g;
  KernelSpec k;
  Bins bins;
  const SortedPoint *pts;
  const int *sub_bin;
  const int *sub_first;
  const int *sub_count;
  const int *bin_off;  // first sorted point of each bin
  const int *nsub;
  const float2 *vals;
  int64_t ips, ics;
  int ch0;
  int nch;  // channels of this launch
  const float *ctf;
  const CtfCoef *ctfc;
  int nyquist;
  float scale;
  float2 *grid;
  int64_t cs, chs;
  int shift;
  int max_sub;
  int half;  // records of kSortHalf
};

// Prologue factor of im_backward: CTF multiply, Nyquist zeroing, scale (projection_funcs.py:385-399).
__device__ __forceinline__ float prologue(const PointGeom &g, int id, const float *ctf, const CtfCoef *ctfc,
                                          int nyquist, float scale) {
  float sc = scale;
  if (nyquist && on_nyquist(g, id)) sc = 0.0f;
  return sc * ctf_factor(ctf, ctfc, g, id);
}

// A subproblem: its points [first, first + cnt) of the sorted order and the tile origin.
struct SubTile {
  int first, cnt, ts0, ts1, ts2;
};

__device__ __forceinline__ SubTile sub_tile(const SpreadParams &a, int sub) {
  const int bin = a.sub_bin[sub];
  const int nb12 = a.bins.nb[1] * a.bins.nb[2];
  SubTile t;
  t.first = a.sub_first[sub];
  t.cnt = a.sub_count[sub];
  t.ts0 = (bin / nb12) * kBin;
  t.ts1 = ((bin / a.bins.nb[2]) % a.bins.nb[1]) * kBin;
  t.ts2 = (bin % a.bins.nb[2]) * kBin;
  return t;
}

// TwoSum (Knuth): s + d = s' + e exactly, e added to the error sum err.
__device__ __forceinline__ void two_sum(float &s, float &err, float d) {
  const float t = __fadd_rn(s, d), b = __fsub_rn(t, s);
  err = __fadd_rn(err, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(d, b)));
  s = t;
}

// Values of the mean's backprojection (mean_cg.cu): channel 0 = y * exp(-i (gx sx + gy sy)) * c * ctf
// (the image phase-shifted by -offset, mean.py:201-204), channel 1 = (c * ctf)^2 / L (the kernel,
// real, whose extra 1/L is mean.py:215).
struct MeanValue {
  MeanSource s;
  __device__ __forceinline__ void operator()(const PointGeom &g, int id, int, float2 &v0, float2 &v1) const {
    mean_value(s, id, g.P, g.Lp, v0, v1.x);
    v1.y = 0.0f;
  }
};
// Channels 2 pair and 2 pair + 1 of an array of point values
struct ArrayValue {
  const float2 *vals;
  int64_t ips, ics;
  int nch;
  __device__ __forceinline__ void operator()(const PointGeom &, int id, int pair, float2 &v0, float2 &v1) const {
    const float2 *v = vals + (int64_t)id * ips + 2 * pair * ics;
    v0 = __ldg(v);
    v1 = 2 * pair + 1 < nch ? __ldg(v + ics) : make_float2(0.f, 0.f);
  }
};

// Nearest-cell spreading, NC pairs of channels per block (blockIdx.y).  A bin's cells belong to its points alone, so
// one block takes the bin (up to kNearestSubs subproblems of it), thread t the bin's cell t: the block
// counting-sorts its points by cell, kNearestThreads at a time, puts a channel pair's values in that
// order into shared memory (two buffers in turn), and every thread adds its cell's values in registers
// (with COMP by TwoSum).  What bounds it is the gather of the points' values and the barriers.  The
// mean's batch of 1024 images of 128^2: 1.75 + 0.11 ms (row tasks over staged values, values made by a
// kernel of their own) -> 0.57 ms.  The points are sorted once for up to five channel pairs, against a
// sort and a launch per pair: 4.17 -> 3.2 ms for 10 channels of 1024 images of 128^2, 77 -> 53 us for 5
// of 256 of 32^2, 111 -> 51 for 20 of 64 of 32^2.
constexpr int kNearestThreads = kBin * kBin * kBin;
constexpr int kNearestSubs = 16;
constexpr int kNearestPairs = 5;

template <bool COMP, int NC, typename Value>
__global__ void __launch_bounds__(kNearestThreads, NC == 1 ? 3 : NC <= 3 ? 2 : 1) spread_nearest_kernel(const SpreadParams a,
                                                                                         const Value value) {
  constexpr int NB = NC > 1 ? 2 : 1;
  __shared__ int s_cnt[kNearestThreads], s_off[kNearestThreads + 1], s_warp[kNearestThreads / 32];
  __shared__ float2 s_v[NB][2][kNearestThreads];
  const int sub = blockIdx.x, pair0 = blockIdx.y * NC, nch = min(2 * NC, a.nch - 2 * pair0);
  if (sub >= *a.nsub) return;
  const int bin = a.sub_bin[sub], first = a.sub_first[sub];
  const int begin = a.bin_off[bin], end = a.bin_off[bin + 1];
  if ((first - begin) % (kNearestSubs * a.max_sub) != 0) return;
  const int last = min(end, first + kNearestSubs * a.max_sub);
  const SubTile st = sub_tile(a, sub);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float2 h[NC][2], l[NC][2];
#pragma unroll
  for (int k = 0; k < NC; ++k) h[k][0] = h[k][1] = l[k][0] = l[k][1] = make_float2(0.f, 0.f);
  bool any = false;
  for (int base = first; base < last; base += kNearestThreads) {
    s_cnt[tid] = 0;
    __syncthreads();  // also: the previous chunk's values have been read
    const bool live = base + tid < last;
    int key = 0, rank = 0, id = 0;
    float sc = 0.0f;
    float2 v0, v1;
    auto load = [&](int pair) {
      value(a.g, id, pair0 + pair, v0, v1);
      v0 = make_float2(v0.x * sc, v0.y * sc);
      v1 = make_float2(v1.x * sc, v1.y * sc);
    };
    if (live) {
      const SortedPoint sp = a.pts[base + tid];
      key = (((int)rintf(sp.t0) - st.ts0) * kBin + (int)rintf(sp.t1) - st.ts1) * kBin + (int)rintf(sp.t2) - st.ts2;
      rank = atomicAdd(s_cnt + key, 1);
      id = sp_id<false>(sp.idf);
      sc = (a.nyquist && sp_nyquist(sp.idf)) ? 0.0f : a.scale;
      sc *= ctf_factor(a.ctf, a.ctfc, a.g, id);
      load(0);
    }
    __syncthreads();
    const int c = s_cnt[tid];
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += s_warp[w];
    const int off = before + incl - c;
    s_off[tid] = off;
    __syncthreads();
    const int slot = live ? s_off[key] + rank : 0;
    any = any || c > 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      if (2 * k >= nch) break;
      float2(&s_v0)[kNearestThreads] = s_v[k & (NB - 1)][0], (&s_v1)[kNearestThreads] = s_v[k & (NB - 1)][1];
      if (live) {
        s_v0[slot] = v0;
        s_v1[slot] = v1;
        if (k + 1 < NC && 2 * k + 2 < nch) load(k + 1);
      }
      __syncthreads();  // (the buffer written next was read before the last one)
      for (int i = off; i < off + c; ++i) {
        const float2 x = s_v0[i], y = s_v1[i];
        if (COMP) {
          two_sum(h[k][0].x, l[k][0].x, x.x);
          two_sum(h[k][0].y, l[k][0].y, x.y);
          two_sum(h[k][1].x, l[k][1].x, y.x);
          two_sum(h[k][1].y, l[k][1].y, y.y);
        } else {
          h[k][0] = __fadd2_rn(h[k][0], x);
          h[k][1] = __fadd2_rn(h[k][1], y);
        }
      }
    }
  }
  if (!any) return;
  const int m0 = st.ts0 + tid / (kBin * kBin), m1 = st.ts1 + (tid / kBin) % kBin, m2 = st.ts2 + tid % kBin;
  const int n = a.g.n;  // a cell with points lies in the grid
  const int64_t cell = ((int64_t)wrap1(m0 + a.shift, n) * n + wrap1(m1 + a.shift, n)) * n + wrap1(m2 + a.shift, n);
  float2 *dst = a.grid + cell * a.cs + (int64_t)(2 * pair0) * a.chs;
  // (atomics also where one block has the whole bin: several plans may add to one grid at a time)
#pragma unroll
  for (int ch = 0; ch < 2 * NC; ++ch)
    if (ch < nch) add_cell(dst + ch * a.chs, __fadd2_rn(h[ch / 2][ch % 2], l[ch / 2][ch % 2]));
}

// Spreading for the ES windows (W = 4 .. 8) and the linear one (W = 2), any number of channels.  One
// block per subproblem (a bin of 8^3 cells and at most max_sub of its points); the cells it can reach
// are a tile of T^3, T = 8 + W - 1.  The block sorts its points by (axis-2 group, l1, l0), l the
// bin-local corner of their window and a group the neighbouring l2 whose windows lie in the same COLS
// tile columns (8, or with ONE all T in one group), and stages a record per point: its weights and its
// channel values.
//
// A warp task is one tile plane, all T rows: lane (h, part, c) owns column c modulo COLS, a part of the
// channels (F floats) and every NH-th point, with acc[T][F / 2] in registers.  The points of a group
// whose windows meet the plane are for each l1 the contiguous range l0 in [plane - W + 1, plane] of the
// sorted order, and with l1 a compile-time constant in the unrolled loop their W rows are fixed
// registers: a point costs a lane F values, W + 2 weights and W * F multiply-adds.  The groups follow
// one another; a column goes to the grid after the last group that reaches it, and its lane takes the
// column COLS further on.
//
// Every cell is added to the grid once per subproblem, from folded sums: the NH lanes' sums meet in
// shuffles, and the ES windows' points are added in pairs.  So a cell's error is that of about half as
// many FP32 additions as it has points in a subproblem and of one atomic addition per subproblem,
// whether the plan asks for `compensated` sums or not.  That is no more than the compensated row sums
// of this kernel's predecessor had (one atomic addition per subproblem of as many points, two or three
// FP32 sums folded by TwoSum).  Relative error of 1024 central slices of 64^2 on 128^3 against 64-bit
// sums, all cells and the 9^3 around the origin, where up to 416 points of a subproblem meet in a cell
// and some 500 subproblems follow one another: values of one sign 1.08e-7 and 1.89e-7 then, 1.06e-7
// and 1.8e-7 here (W = 6, ten channels); noise 1.68e-7 and 2.53e-7, here 1.64e-7 and 2.45e-7; linear
// windows 6.0e-8 and 9.6e-8, here 5.6e-8 to 6.1e-8 and 7.7e-8 to 9.6e-8.  A task per plane pair and group,
// each group's columns added to the grid apart, took 8.6 ms where this takes 10.5 (below), but its 1.85 additions
// per cell and subproblem cost 1.36e-7 and 2.58e-7.
//
// What bounds it: latency at sixteen warps per SM (some 38 instructions for a point's visit to a plane,
// of which it has W), then the flush, W + 7 times W + 7 rows in NG steps, for subproblems of few points.
// 10 channels, W = 6, 1024 images of 128^2 (full records): 15.8 ms the predecessor, 10.5 here; W = 7, one
// channel, 512 images: 11.2 and 2.2; W = 7, 10 channels, 100 images: 3.46 and 3.73.  Bilinear, 10 channels of
// 1024 images: 4.24 and 3.06.
template <int W, int F, int NQ, bool ONE>
struct TileShape {
  using G = TileGroups<W, ONE ? 8 + W - 1 : 8>;
  static constexpr int T = G::T, COLS = G::COLS, NG = G::NG;
  static constexpr int NH = 32 / COLS / NQ;     // subsets of the points
  static constexpr int RH = (T + NH - 1) / NH;  // rows that each of them flushes
  // How a lane folds its sums: the points of a range summed apart (wide windows, of which a cell sees the
  // most points, which in pairs are 1.5e-7 off near the origin against 1.24e-7; the registers leave six
  // warps, 11.2 ms against 10.5 at W = 6), or points added in pairs.
  static constexpr bool RANGES = W >= 7 && NH == 1 && F > 2;
  static constexpr bool PAIRS = W > 2 && !RANGES && (NH == 1 || F == 2);
  static constexpr int WARPS = W == 2 ? 9 : F == 2 ? 14 : RANGES ? 6 : 8;
  static_assert(NH >= 1 && NH <= 3 && T <= 16, "lanes; plane weights of a record");

  // A point's record in floats: the W axis-1 weights twice each (operands of packed multiplies), the
  // axis-2 weights of the group's columns, the axis-0 weights of the T planes; a stride that keeps
  // 16-byte stores of consecutive records free of bank conflicts (4 modulo 8 words).
  static constexpr int W2 = 2 * W, W0 = W2 + COLS, REC = (W0 + T + 3) / 8 * 8 + 4;
  static_assert(W0 + T <= REC, "a record's weights");
  // Its staged channel values: NQ parts of F / 2 channels next to each other.
  static constexpr int VALS = F * NQ;
  __device__ __forceinline__ static void load_values(const float *vp, float2 (&v)[F / 2]) {
    if constexpr (F % 4 == 0) {
#pragma unroll
      for (int f = 0; f < F / 2; f += 2) {
        const float4 x = *reinterpret_cast<const float4 *>(vp + 2 * f);
        v[f] = make_float2(x.x, x.y);
        v[f + 1] = make_float2(x.z, x.w);
      }
    } else {
#pragma unroll
      for (int f = 0; f < F / 2; ++f) v[f] = *reinterpret_cast<const float2 *>(vp + 2 * f);
    }
  }
  // bytes of shared memory: a point's (record, values, id, mirror id, two factors), and the rest
  static constexpr size_t POINT = (REC + VALS + 4) * sizeof(float);
  static constexpr size_t FIXED = T * T * sizeof(long long) + (2 * NG * 64 + 1 + T + 1) * sizeof(int) + 8;
};

// The points of corner row l1 = L1 .. 7 of the lane's subset added to its cells
template <int W, int F, int NQ, bool ONE, int L1>
struct TileRows {
  using S = TileShape<W, F, NQ, ONE>;
  // axis-1 weights (twice each) and the product of the other axes' weights
  __device__ __forceinline__ static float2 weights(const float *rec, int col, int plane, float2 (&w)[W]) {
    const float w02 = rec[S::W0 + plane] * rec[S::W2 + col];
#pragma unroll
    for (int j = 0; j + 1 < W; j += 2) {
      const float4 x = *reinterpret_cast<const float4 *>(rec + 2 * j);
      w[j] = make_float2(x.x, x.y);
      w[j + 1] = make_float2(x.z, x.w);
    }
    if constexpr (W & 1) w[W - 1] = *reinterpret_cast<const float2 *>(rec + 2 * (W - 1));
    return make_float2(w02, w02);
  }
  template <typename Range>
  __device__ __forceinline__ static void run(const Range &range, const float *recs, const float *vals, int cp, int h,
                                             int col, int plane, float2 (&acc)[S::T][F / 2]) {
    constexpr int NH = S::NH;
    int i, iend;
    range(L1, i, iend);
    i += h;
    const float *rec = recs + i * S::REC;
    const float *vp = vals + i * S::VALS + F * cp;
    float2 wa[W], va[F / 2];
    if constexpr (S::RANGES) {
      if (i < iend) {
        float2 t[W][F / 2];
        const float2 sa = weights(rec, col, plane, wa);
        S::load_values(vp, va);
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const float2 x = __fmul2_rn(sa, wa[j]);
#pragma unroll
          for (int f = 0; f < F / 2; ++f) t[j][f] = __fmul2_rn(x, va[f]);
        }
#pragma unroll 1
        for (i += NH; i < iend; i += NH) {
          rec += NH * S::REC, vp += NH * S::VALS;
          const float2 sb = weights(rec, col, plane, wa);
          S::load_values(vp, va);
#pragma unroll
          for (int j = 0; j < W; ++j) {
            const float2 x = __fmul2_rn(sb, wa[j]);
#pragma unroll
            for (int f = 0; f < F / 2; ++f) t[j][f] = __ffma2_rn(x, va[f], t[j][f]);
          }
        }
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
          for (int f = 0; f < F / 2; ++f) acc[L1 + j][f] = __fadd2_rn(acc[L1 + j][f], t[j][f]);
      }
    }
    if constexpr (S::PAIRS) {
#pragma unroll 1
      for (; i + NH < iend; i += 2 * NH, rec += 2 * NH * S::REC, vp += 2 * NH * S::VALS) {
        float2 wb[W], vb[F / 2];
        const float2 sa = weights(rec, col, plane, wa);
        S::load_values(vp, va);
        const float2 sb = weights(rec + NH * S::REC, col, plane, wb);
        S::load_values(vp + NH * S::VALS, vb);
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const float2 x = __fmul2_rn(sa, wa[j]), y = __fmul2_rn(sb, wb[j]);
#pragma unroll
          for (int f = 0; f < F / 2; ++f)
            acc[L1 + j][f] = __fadd2_rn(acc[L1 + j][f], __ffma2_rn(y, vb[f], __fmul2_rn(x, va[f])));
        }
      }
    }
#pragma unroll 1
    for (; !S::RANGES && i < iend; i += NH, rec += NH * S::REC, vp += NH * S::VALS) {
      const float2 sa = weights(rec, col, plane, wa);
      S::load_values(vp, va);
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float2 x = __fmul2_rn(sa, wa[j]);
#pragma unroll
        for (int f = 0; f < F / 2; ++f) acc[L1 + j][f] = __ffma2_rn(x, va[f], acc[L1 + j][f]);
      }
      if (S::PAIRS) break;  // at most one is left
    }
    if constexpr (L1 + 1 < kBin) TileRows<W, F, NQ, ONE, L1 + 1>::run(range, recs, vals, cp, h, col, plane, acc);
  }
};

// The sum over the NH lane subsets of channel f of row k + RH h, in subset h; LANES lanes in a subset.
template <int NH, int LANES, int T, int FH>
__device__ __forceinline__ float2 subset_sum(const float2 (&acc)[T][FH], int k, int f, int h, int lane) {
  constexpr int RH = (T + NH - 1) / NH;
  auto row = [&](int r) { return r < T ? acc[r][f] : make_float2(0.f, 0.f); };
  auto pick = [](bool p, float2 a, float2 b) { return make_float2(p ? a.x : b.x, p ? a.y : b.y); };
  auto from = [](float2 x, int l) {
    return make_float2(__shfl_sync(0xffffffffu, x.x, l), __shfl_sync(0xffffffffu, x.y, l));
  };
  if constexpr (NH == 1) {
    return row(k);
  } else if constexpr (NH == 2) {
    const bool up = h != 0;
    return __fadd2_rn(pick(up, row(k + RH), row(k)), from(pick(up, row(k), row(k + RH)), up ? lane - LANES : lane + LANES));
  } else {  // the rows of the next subset go to it, those of the one before to that
    const int next = h < 2 ? lane + LANES : lane - 2 * LANES, prev = h > 0 ? lane - LANES : lane + 2 * LANES;
    auto of = [&](int s) { return pick(s == 0, row(k), pick(s == 1, row(k + RH), row(k + 2 * RH))); };
    const int h1 = h < 2 ? h + 1 : 0, h2 = h > 0 ? h - 1 : 2;
    return __fadd2_rn(of(h), __fadd2_rn(from(of(h1), prev), from(of(h2), next)));
  }
}

template <int KT, int W, int F, int NQ, bool ONE, bool HALF>
__global__ void __launch_bounds__(TileShape<W, F, NQ, ONE>::WARPS * 32, 2) spread_tile_kernel(const SpreadParams a) {
  constexpr bool ES = KT == COV3D_KERNEL_ES;
  using S = TileShape<W, F, NQ, ONE>;
  using G = typename S::G;
  constexpr int T = G::T, NG = G::NG, NK = NG * 64, COLS = G::COLS, NH = S::NH, RH = S::RH;
  constexpr int FH = F / 2, CH = NQ * FH, VS = S::VALS;  // channels of a lane, of a pass; values of a point
  constexpr int THREADS = S::WARPS * 32;
  extern __shared__ float4 smem4[];
  float *recs = reinterpret_cast<float *>(smem4);                // max_sub * record
  float *vals = recs + (size_t)a.max_sub * S::REC;               // max_sub * VS
  int *s_id = reinterpret_cast<int *>(vals + (size_t)a.max_sub * VS);
  int *s_mid = s_id + a.max_sub;      // ids; mirror ids or -1
  float *s_sc = reinterpret_cast<float *>(s_mid + a.max_sub), *s_scm = s_sc + a.max_sub;
  long long *s_row = reinterpret_cast<long long *>((reinterpret_cast<uintptr_t>(s_scm + a.max_sub) + 7) & ~(uintptr_t)7);
  int *s_cnt = reinterpret_cast<int *>(s_row + T * T), *s_off = s_cnt + NK, *s_col = s_off + NK + 1;
  int *s_task = s_col + T;
  const int sub = blockIdx.x;
  if (sub >= *a.nsub) return;
  const SubTile st = sub_tile(a, sub);
  const int n = a.g.n, tid = threadIdx.x, lane = tid & 31;

  for (int e = tid; e < NK; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  // bin-local window corner, 0 .. 7 (linear: a window that starts one cell before the grid counts
  // from cell 0)
  auto corner = [&](float t, int ts) {
    const int c0 = record_cell<KT, W, HALF>(t, a.g.frac);
    return min(max((ES ? wrap1(c0, n) : c0) - ts, 0), kBin - 1);
  };
  // each thread keeps its points until their place in the sorted order is known, and asks for their
  // values (point-major ones) ahead of the gather
  constexpr int PPT = (kTileMaxSub + THREADS - 1) / (THREADS);
  SortedPoint pt[PPT];
  int pkey[PPT];
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    const int k = tid + u * THREADS;
    pkey[u] = -1;
    if (k < st.cnt) pt[u] = a.pts[st.first + k];
  }
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    if (tid + u * THREADS >= st.cnt) continue;
    const int key = (corner(pt[u].t2, st.ts2) / G::GS) * 64 + corner(pt[u].t1, st.ts1) * 8 + corner(pt[u].t0, st.ts0);
    pkey[u] = key | (atomicAdd(s_cnt + key, 1) << 9);
    if (a.ics == 1) {
      const int id = sp_id<HALF>(pt[u].idf);
      const float2 *v = a.vals + a.ch0;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(v + (int64_t)id * a.ips));
      if (sp_pair<HALF>(pt[u].idf)) asm volatile("prefetch.global.L2 [%0];" ::"l"(v + (int64_t)mirror_id(a.g, id) * a.ips));
    }
  }
  __syncthreads();
  if (tid < 32) {  // exclusive scan of the counters by one warp
    int v[NK / 32], sum = 0;
#pragma unroll
    for (int u = 0; u < NK / 32; ++u) {
      v[u] = s_cnt[tid * (NK / 32) + u];
      sum += v[u];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += t;
    }
    int base = incl - sum;
#pragma unroll
    for (int u = 0; u < NK / 32; ++u) {
      s_off[tid * (NK / 32) + u] = base;
      base += v[u];
    }
    if (tid == 31) s_off[NK] = incl;
  }
  // global offsets of the tile's rows (axes 0, 1) and columns (axis 2): periodic, or (linear) -1
  // outside the grid
  for (int e = tid; e < T * T; e += blockDim.x) {
    const int ra = e / T, rb = e - (e / T) * T;
    const int m0 = wrap1(wrap1(st.ts0 + ra, n) + a.shift, n), m1 = wrap1(wrap1(st.ts1 + rb, n) + a.shift, n);
    s_row[e] = ES || (st.ts0 + ra < n && st.ts1 + rb < n) ? ((int64_t)m0 * n + m1) * n * a.cs : -1;
  }
  for (int e = tid; e < T; e += blockDim.x) s_col[e] = ES || st.ts2 + e < n ? wrap1(wrap1(st.ts2 + e, n) + a.shift, n) : -1;
  __syncthreads();
  // records (a weight is zero outside its window), ids and prologue factors in sorted order
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    const SortedPoint sp = pt[u];
    const int kr = pkey[u];
    if (kr < 0) continue;
    const int slot = s_off[kr & 511] + (kr >> 9);
    const int c0 = record_cell<KT, W, HALF>(sp.t0, a.g.frac), c1 = record_cell<KT, W, HALF>(sp.t1, a.g.frac),
              c2 = record_cell<KT, W, HALF>(sp.t2, a.g.frac);
    const int l0 = (ES ? wrap1(c0, n) : c0) - st.ts0, l2 = (ES ? wrap1(c2, n) : c2) - st.ts2;
    const int b2 = G::base((kr & 511) >> 6);
    float4 *rec = reinterpret_cast<float4 *>(recs + slot * S::REC);
    // the axes' weights at offset i from the window's first cell, zero outside the window
    float x0, x1, x2, y0 = 0.f, y1 = 0.f, y2 = 0.f;
    if (ES) {
      x0 = record_offset<HALF>(sp.t0, c0, a.g.frac);
      x1 = record_offset<HALF>(sp.t1, c1, a.g.frac);
      x2 = record_offset<HALF>(sp.t2, c2, a.g.frac);
    } else {
      x0 = record_weight<KT, W, HALF>(sp.t0, c0, 0, a.g.frac, 0.f);
      y0 = record_weight<KT, W, HALF>(sp.t0, c0, 1, a.g.frac, 0.f);
      x1 = record_weight<KT, W, HALF>(sp.t1, c1, 0, a.g.frac, 0.f);
      y1 = record_weight<KT, W, HALF>(sp.t1, c1, 1, a.g.frac, 0.f);
      x2 = record_weight<KT, W, HALF>(sp.t2, c2, 0, a.g.frac, 0.f);
      y2 = record_weight<KT, W, HALF>(sp.t2, c2, 1, a.g.frac, 0.f);
      if (c1 < st.ts1) {  // the window's first row is before the grid
        x1 = y1;
        y1 = 0.f;
      }
    }
    auto weight = [&](float x, float y, int i) {
      return ES ? es_weight<W>(x - (float)i, a.k.beta) : i == 0 ? x : i == 1 ? y : 0.0f;
    };
    float w[S::REC];
#pragma unroll
    for (int j = 0; j < W; ++j) w[2 * j] = w[2 * j + 1] = weight(x1, y1, j);
#pragma unroll
    for (int j = 0; j < COLS; ++j) w[S::W2 + j] = weight(x2, y2, b2 + j - l2);
#pragma unroll
    for (int j = 0; j < T; ++j) w[S::W0 + j] = weight(x0, y0, j - l0);
#pragma unroll
    for (int j = S::W0 + T; j < S::REC; ++j) w[j] = 0.0f;
#pragma unroll
    for (int u = 0; u < S::REC / 4; ++u) rec[u] = make_float4(w[4 * u], w[4 * u + 1], w[4 * u + 2], w[4 * u + 3]);
    const int id = sp_id<HALF>(sp.idf);
    const float sc = ((a.nyquist && sp_nyquist(sp.idf)) ? 0.0f : a.scale) * ctf_factor(a.ctf, a.ctfc, a.g, id);
    const int mid = sp_pair<HALF>(sp.idf) ? mirror_id(a.g, id) : -1;
    s_id[slot] = sp_conj<HALF>(sp.idf) ? ~id : id;  // a negative id: the value's conjugate
    s_mid[slot] = mid;
    s_sc[slot] = sc;
    if (mid >= 0) s_scm[slot] = a.scale * ctf_factor(a.ctf, a.ctfc, a.g, mid);
  }

  // (lanes past the columns repeat the first one's work and keep it)
  constexpr int LANES = COLS * NQ;  // of a subset
  const bool lane_live = lane < LANES * NH;
  const int q = lane_live ? lane / COLS : 0, c = lane_live ? lane - q * COLS : 0;
  const int cp = q % NQ, h = q / NQ;  // channel part, subset of the points
  for (int p0 = 0; p0 < a.nch; p0 += CH) {
    __syncthreads();
    // this pass's channel values in sorted order.  A record of kSortHalf that stands for a pair of
    // mirror pixels takes the sum of the one's value and the conjugate of the other's, which has
    // the same real part after the inverse transform.
    // Four elements' loads in flight per thread: the gathers' latency is most of the staging.
    constexpr int GU = 4;
    const int total = st.cnt * CH;
    for (int e0 = tid; e0 < total; e0 += GU * THREADS) {
      float2 x[GU], m[GU];
      int sl[GU];
#pragma unroll
      for (int u = 0; u < GU; ++u) {
        const int e = e0 + u * THREADS;
        const int slot = e / CH, ch = e - slot * CH;
        sl[u] = e < total ? slot : -1;
        x[u] = m[u] = make_float2(0.f, 0.f);
        if (e < total && p0 + ch < a.nch) {
          const float2 *src = a.vals + (int64_t)(a.ch0 + p0 + ch) * a.ics;
          const int id = s_id[slot];
          x[u] = __ldg(src + (int64_t)(HALF && id < 0 ? ~id : id) * a.ips);
          if (HALF) {
            const int mid = s_mid[slot];
            if (mid >= 0) m[u] = __ldg(src + (int64_t)mid * a.ips);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < GU; ++u) {
        const int slot = sl[u];
        if (slot < 0) continue;
        const int ch = e0 + u * THREADS - slot * CH;
        const float sc = s_sc[slot];
        float2 v = make_float2(x[u].x * sc, HALF && s_id[slot] < 0 ? -(x[u].y * sc) : x[u].y * sc);
        if (HALF && s_mid[slot] >= 0) {
          const float sm = s_scm[slot];
          v.x = fmaf(m[u].x, sm, v.x);
          v.y = fmaf(-m[u].y, sm, v.y);
        }
        *reinterpret_cast<float2 *>(vals + slot * VS + 2 * ch) = v;
      }
    }
    if (tid == 0) *s_task = 0;
    __syncthreads();

    for (;;) {
      int task = 0;
      if (lane == 0) task = atomicAdd(s_task, 1);
      task = __shfl_sync(0xffffffffu, task, 0);
      if (task >= T) break;
      const int plane = T / 2 + (task & 1 ? -((task + 1) / 2) : task / 2);  // the fullest first
      const int lo = max(plane - W + 1, 0), hi = min(plane, kBin - 1);
      float2 acc[T][FH];
#pragma unroll
      for (int r = 0; r < T; ++r)
#pragma unroll
        for (int f = 0; f < FH; ++f) acc[r][f] = make_float2(0.f, 0.f);
      bool any = false;
#pragma unroll 1
      for (int g = 0; g < NG; ++g) {
        // the lane's column in the group and in the tile
        const int col = NG == 1 ? c : (c - G::base(g)) & (COLS - 1), tc = G::base(g) + col;
        if (s_off[g * 64] != s_off[g * 64 + 64]) {
          any = true;
          auto range = [&](int l1, int &i, int &iend) {
            i = s_off[g * 64 + l1 * 8 + lo];
            iend = s_off[g * 64 + l1 * 8 + hi + 1];
          };
          TileRows<W, F, NQ, ONE, 0>::run(range, recs, vals, cp, h, col, plane, acc);
        }
        if (!any) continue;
        // the columns that no later group reaches go to the global grid
        const bool last = g + 1 == NG, done = last || tc < G::base(g + 1);
        const int co = done && lane_live ? s_col[tc] : -1, ch0 = p0 + cp * FH;
        const int nf = co < 0 ? 0 : a.nch - ch0;  // channels to write
        float2 *const dst0 = a.grid + (int64_t)co * a.cs + (int64_t)(a.ch0 + ch0) * a.chs;
#pragma unroll
        for (int k = 0; k < RH; ++k) {
          const int r = k + RH * h;
          const long long ro = r < T ? s_row[plane * T + r] : -1;
          float2 *dst = dst0 + ro;
#pragma unroll
          for (int f = 0; f < FH; ++f) {
            const float2 x = subset_sum<NH, LANES>(acc, k, f, h, lane);
            if (f < nf && (ro >= 0 || (ES && RH * NH == T)) && (x.x != 0.0f || x.y != 0.0f)) add_cell(dst + f * a.chs, x);
          }
        }
        if (last) break;
#pragma unroll
        for (int r = 0; r < T; ++r)
#pragma unroll
          for (int f = 0; f < FH; ++f)
            if (done) acc[r][f] = make_float2(0.f, 0.f);
      }
    }
  }
}

template <typename Kernel>
int launch_spread_kernel(Kernel kernel, const char *name, size_t smem, const SpreadParams &a, int64_t max_blocks,
                         cudaStream_t st, int warps) {
  if (smem > 227 * 1024) {
    set_error("spreading stage of %zu bytes exceeds shared memory", smem);
    return COV3D_EINVAL;
  }
  if (smem > 32 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(spread)");
  }
  kernel<<<(unsigned)max_blocks, warps * 32, smem, st>>>(a);
  return launched(name);
}

template <int NC, typename Value>
int launch_nearest(const SpreadParams &a, const Value &value, bool comp, int64_t max_blocks, cudaStream_t st) {
  const dim3 grid((unsigned)max_blocks, (unsigned)((a.nch + 2 * NC - 1) / (2 * NC)));
  if (comp) spread_nearest_kernel<true, NC, Value><<<grid, kNearestThreads, 0, st>>>(a, value);
  else spread_nearest_kernel<false, NC, Value><<<grid, kNearestThreads, 0, st>>>(a, value);
  return launched("spread_nearest_kernel");
}

template <int KT, int W, int F, int NQ, bool ONE, bool HALF>
int launch_tile(const SpreadParams &a, int64_t max_blocks, cudaStream_t st) {
  using S = TileShape<W, F, NQ, ONE>;
  if (a.max_sub > kTileMaxSub) {
    set_error("subproblems of %d points; the spreading holds %d", a.max_sub, kTileMaxSub);
    return COV3D_EINVAL;
  }
  return launch_spread_kernel(spread_tile_kernel<KT, W, F, NQ, ONE, HALF>, "spread_tile_kernel",
                              a.max_sub * S::POINT + S::FIXED, a, max_blocks, st, S::WARPS);
}

// Channels in passes of twelve in one launch, then the rest in the layout that holds it.  The linear
// windows' FMAs are few, so all their columns fit one group; the ES windows' bound their time, and eight
// columns waste fewer of them, except for one channel, where the flush of the groups costs more.  Microseconds of
// the layouts tried, ES W = 6: 4 channels of 256 images of 64^2: 422 with one channel a part, 443 with two and
// two subsets, 544 with three; 2 of 256 of 128^2: 1565, 1635 with all columns and two channels a lane; 1 of 64
// of 128^2: 699, 853 with eight columns and four subsets; 10 of 1024 of 128^2: 10519, 12121 with two
// parts of five channels and two subsets.  Linear, 8 channels of 512 images of 64^2: 324, 386 with four
// channels a part.
template <int KT, int W, bool HALF>
int launch_channels(SpreadParams a, int nchan, int64_t max_blocks, cudaStream_t st) {
  constexpr bool linear = W == 2;
  const int rest = nchan % 12, whole = rest > 6 ? nchan : nchan - rest;
  a.ch0 = 0;
  a.nch = whole;
  if constexpr (linear) {
    if (whole > 9) COV3D_TRY((launch_tile<KT, W, 8, 3, true, HALF>(a, max_blocks, st)));
    else if (whole > 0) return launch_tile<KT, W, 6, 3, true, HALF>(a, max_blocks, st);
  } else {
    if (whole > 0) COV3D_TRY((launch_tile<KT, W, 6, 4, false, HALF>(a, max_blocks, st)));
  }
  a.ch0 = whole;
  a.nch = nchan - whole;
  if constexpr (linear) {
    if (a.nch > 3) return launch_tile<KT, W, 4, 3, true, HALF>(a, max_blocks, st);
    if (a.nch > 2) return launch_tile<KT, W, 2, 3, true, HALF>(a, max_blocks, st);
    if (a.nch > 1) return launch_tile<KT, W, 4, 1, true, HALF>(a, max_blocks, st);
    if (a.nch > 0) return launch_tile<KT, W, 2, 1, true, HALF>(a, max_blocks, st);
  } else {
    if (a.nch > 4) return launch_tile<KT, W, 6, 2, false, HALF>(a, max_blocks, st);
    if (a.nch > 2) return launch_tile<KT, W, 2, 4, false, HALF>(a, max_blocks, st);
    if (a.nch > 1) return launch_tile<KT, W, 2, 2, false, HALF>(a, max_blocks, st);
    if (a.nch > 0) return launch_tile<KT, W, 2, 1, true, HALF>(a, max_blocks, st);
  }
  return COV3D_OK;
}

template <int KT, int W>
int launch_w(const SpreadParams &a, int nchan, int64_t max_blocks, cudaStream_t st) {
  return a.half ? launch_channels<KT, W, true>(a, nchan, max_blocks, st)
                : launch_channels<KT, W, false>(a, nchan, max_blocks, st);
}

int launch_nearest_channels(SpreadParams a, int nchan, bool comp, int64_t max_blocks, cudaStream_t st) {
  a.nch = nchan;
  const ArrayValue v{a.vals, a.ips, a.ics, nchan};
  switch ((nchan + 1) / 2) {
    case 1: return launch_nearest<1>(a, v, comp, max_blocks, st);
    case 2: return launch_nearest<2>(a, v, comp, max_blocks, st);
    case 3: return launch_nearest<3>(a, v, comp, max_blocks, st);
    default: return launch_nearest<kNearestPairs>(a, v, comp, max_blocks, st);
  }
}

// Per-image adjoint (no sum over images): direct global atomics, one thread per point.
template <int KT, int W>
__global__ void spread_unagg_kernel(PointGeom g, KernelSpec k, int64_t M, const float2 *__restrict__ vals,
                                    int64_t ips, const float *ctf, const CtfCoef *ctfc, int nyquist, float scale,
                                    float2 *grids) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= M) return;
  const int id = (int)gid;
  const float sc = prologue(g, id, ctf, ctfc, nyquist, scale);
  if (sc == 0.0f) return;
  const int n = g.n;
  float t[3];
  point_index(g, id, t);
  float wt[3][W];
  int c0[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) c0[d] = taps<KT, W, false>(t[d], g.frac, k.beta, wt[d]);
  const float2 x = vals[(int64_t)id * ips];
  const float2 v = make_float2(x.x * sc, x.y * sc);
  float2 *out = grids + (id / g.P) * (int64_t)n * n * n;
  for (int i0 = 0; i0 < W; ++i0) {
    int m0 = c0[0] + i0;
    if (KT == COV3D_KERNEL_ES) m0 = pmod(m0, n);
    else if (m0 < 0 || m0 >= n) continue;
    for (int i1 = 0; i1 < W; ++i1) {
      int m1 = c0[1] + i1;
      if (KT == COV3D_KERNEL_ES) m1 = pmod(m1, n);
      else if (m1 < 0 || m1 >= n) continue;
      for (int i2 = 0; i2 < W; ++i2) {
        int m2 = c0[2] + i2;
        if (KT == COV3D_KERNEL_ES) m2 = pmod(m2, n);
        else if (m2 < 0 || m2 >= n) continue;
        const float w = wt[0][i0] * wt[1][i1] * wt[2][i2];
        float2 *dst = out + ((int64_t)m0 * n + m1) * n + m2;
        atomicAdd(&dst->x, w * v.x);
        atomicAdd(&dst->y, w * v.y);
      }
    }
  }
}

}  // namespace

// What every spreading launch of a plan's points shares.
static int spread_params(cov3d_plan *p, const EpilogueArgs &e, void *grid, int64_t cell_stride, int64_t chan_stride,
                         int shift, SortMode mode, SpreadParams &a, int64_t &max_blocks) {
  if (p->point_kind == kPointsNone || p->n_points == 0) {
    set_error("no points set");
    return COV3D_ESTATE;
  }
  if (p->bins.bs[0] != kBin || p->bins.bs[1] != kBin || p->bins.bs[2] != kBin) {
    set_error("spreading requires %d^3-cell bins", kBin);
    return COV3D_EINVAL;
  }
  COV3D_TRY(need_sorted(p, 1u << mode));
  const SortSet &ss = p->sets[mode];
  a = SpreadParams{};
  a.g = make_geom(p);
  a.k = make_kernel(p);
  a.bins = p->bins;
  a.pts = ss.sorted;
  a.sub_bin = ss.sub_bin;
  a.sub_first = ss.sub_first;
  a.sub_count = ss.sub_count;
  a.bin_off = ss.bin_off;
  a.nsub = ss.nsub;
  a.ctf = e.ctf;
  a.ctfc = e.ctfc;
  a.nyquist = e.nyquist;
  a.scale = e.scale;
  a.grid = static_cast<float2 *>(grid);
  a.cs = cell_stride;
  a.chs = chan_stride;
  a.shift = shift;
  a.max_sub = p->max_sub;
  a.half = mode == kSortHalf;
  max_blocks = p->bins.nbins + p->n_points / p->max_sub + 1;
  return COV3D_OK;
}

int launch_spread(cov3d_plan *p, const void *values, int64_t in_ps, int64_t in_cs, int nchan, const EpilogueArgs &e,
                  void *grid, int64_t cell_stride, int64_t chan_stride, int shift, SortMode mode) {
  SpreadParams a;
  int64_t mb;
  COV3D_TRY(spread_params(p, e, grid, cell_stride, chan_stride, shift, mode, a, mb));
  a.vals = static_cast<const float2 *>(values);
  a.ips = in_ps;
  a.ics = in_cs;
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST: return launch_nearest_channels(a, nchan, p->compensated != 0, mb, p->stream);
    case COV3D_KERNEL_LINEAR: return launch_w<COV3D_KERNEL_LINEAR, 2>(a, nchan, mb, p->stream);
    default:
      switch (p->width) {
        case 4: return launch_w<COV3D_KERNEL_ES, 4>(a, nchan, mb, p->stream);
        case 5: return launch_w<COV3D_KERNEL_ES, 5>(a, nchan, mb, p->stream);
        case 6: return launch_w<COV3D_KERNEL_ES, 6>(a, nchan, mb, p->stream);
        case 7: return launch_w<COV3D_KERNEL_ES, 7>(a, nchan, mb, p->stream);
        case 8: return launch_w<COV3D_KERNEL_ES, 8>(a, nchan, mb, p->stream);
        default: set_error("unsupported ES width %d (supported: 4..8)", p->width); return COV3D_EINVAL;
      }
  }
}

int launch_spread_mean_nearest(cov3d_plan *p, const MeanSource &src, const EpilogueArgs &e, void *grids,
                               int64_t chan_stride) {
  SpreadParams a;
  int64_t mb;
  COV3D_TRY(spread_params(p, e, grids, 1, chan_stride, 0, kSortFull, a, mb));
  a.nch = 2;
  return launch_nearest<1>(a, MeanValue{src}, p->compensated != 0, mb, p->stream);
}

int launch_spread_unaggregated(cov3d_plan *p, const void *values, int64_t in_ps, const EpilogueArgs &e,
                               void *grids) {
  if (p->point_kind == kPointsNone || p->n_points == 0) {
    set_error("no points set");
    return COV3D_ESTATE;
  }
  const PointGeom g = make_geom(p);
  const KernelSpec k = make_kernel(p);
  const int blocks = (int)((p->n_points + 255) / 256);
  const float2 *v = static_cast<const float2 *>(values);
  float2 *out = static_cast<float2 *>(grids);
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST:
      spread_unagg_kernel<COV3D_KERNEL_NEAREST, 1>
          <<<blocks, 256, 0, p->stream>>>(g, k, p->n_points, v, in_ps, e.ctf, e.ctfc, e.nyquist, e.scale, out);
      break;
    case COV3D_KERNEL_LINEAR:
      spread_unagg_kernel<COV3D_KERNEL_LINEAR, 2>
          <<<blocks, 256, 0, p->stream>>>(g, k, p->n_points, v, in_ps, e.ctf, e.ctfc, e.nyquist, e.scale, out);
      break;
    default:
      switch (p->width) {
#define COV3D_UW(Wv)                                                                                     \
  case Wv:                                                                                             \
    spread_unagg_kernel<COV3D_KERNEL_ES, Wv>                                                           \
        <<<blocks, 256, 0, p->stream>>>(g, k, p->n_points, v, in_ps, e.ctf, e.ctfc, e.nyquist, e.scale, out); \
    break;
        COV3D_UW(4) COV3D_UW(5) COV3D_UW(6) COV3D_UW(7) COV3D_UW(8)
#undef COV3D_UW
        default: set_error("unsupported ES width %d", p->width); return COV3D_EINVAL;
      }
  }
  return launched("spread_unagg_kernel");
}

}  // namespace cov3d
