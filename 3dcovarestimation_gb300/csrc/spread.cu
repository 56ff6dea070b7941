// Spreading ("type-1" half of the NUFFT; exact adjoint of interp.cu, replacing the
// reference's grid_sample backward with FP32 global atomics, nufft_plan.py:171-242), over the
// bin-sorted point records of points_sort.cu.  See spread_tile_kernel (ES and linear windows) and
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
__global__ void __launch_bounds__(kNearestThreads, NC <= 2 ? 2 : 1) spread_nearest_kernel(const SpreadParams a,
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
    if (ch < nch) atomicAdd(dst + ch * a.chs, __fadd2_rn(h[ch / 2][ch % 2], l[ch / 2][ch % 2]));
}

// Spreading for the ES windows (W = 4 .. 8) and the linear one (W = 2), any number of channels.  One
// block per subproblem (a bin of 8^3 cells and at most max_sub of its points); the cells it can reach
// are a tile of T^3, T = 8 + W - 1.  The block sorts its points by (axis-2 group, l1, l0), l the bin-local corner of
// their window and a group GS = 9 - W neighbouring l2, so that the windows of a group lie in the
// same 8 tile columns, and stages a record per point (weights) and its channel values.
//
// A warp task is NPL tile planes of one group, all T rows: lane (q, c) owns column c of the group,
// part q % NQ of the channels (F floats) and part q / NQ of the planes (PP of them), with
// acc[PP][T][F / 2] in registers.  The points whose windows meet the planes are for each l1 the
// contiguous range l0 in [first plane - W + 1, last plane] of the sorted order, and with l1 a
// compile-time constant in the unrolled loop their W rows are fixed registers: a point costs a lane
// F values, W + PP + 1 weights and PP * W * F multiply-adds.
//
// What bounds it: latency at twelve warps per SM (issue 47 %, FP32 pipe 32 %, shared wavefronts
// 17 % of their peaks on the B = 256 capture).  At the covariance step's 10 channels, W = 6, a visit
// is some 50 instructions and a point has 3.5 of them.  Its predecessor, lanes owning all 13 tile
// columns of three rows of one plane, had 16 visits and 2.2x the multiply-adds.  Measured on the step at
// L = 128, B = 1024, r = 10: 8.6 -> 5.3 ms, of which staging (sort, weights, gathered values) about
// 2.0 and the flush 0.9; 4.7 with the points in registers, their values asked for ahead and four
// gathers in flight.  One channel at W = 7, 512 images of 128^2: 6.2 -> 1.0 ms.
//
// Each cell's sum is plain FP32 over the points of one group of one subproblem (some 30 terms at
// one point per cell, a third of what the predecessor summed before its first TwoSum fold; two or
// three partial sums folded by TwoSum round to the float sum of the partials), and the partial sums
// meet in FP32 global atomics, so `compensated` changes nothing here.
// per block, two blocks per SM (168 registers); 5 or 4 warps measured 5.8 and 6.8 ms against 5.3 (a
// unrolled point loop is slower too: the ranges hold some ten points), 7 spill
constexpr int kTileWarps = 6;

// A point's record in floats: the W axis-1 weights twice each (operands of packed multiplies), the
// axis-2 weights of the group's 8 columns, the axis-0 weights of up to 16 planes; a stride that keeps
// 16-byte stores of consecutive records free of bank conflicts (4 modulo 8 words).
template <int W>
struct TileRec {
  static constexpr int W2 = (2 * W + 3) / 4 * 4;
  static constexpr int W0 = W2 + 8;
  static constexpr int STRIDE = W <= 2 ? 28 : W <= 6 ? 36 : 44;
  static_assert(W0 + 16 <= STRIDE && STRIDE % 8 == 4, "plane weights; conflict-free stores");
};

template <int F>
struct TileVals {  // floats of a channel part's values, padded to 16 bytes where loads are
  static constexpr int STRIDE = F <= 2 ? F : (F + 3) / 4 * 4;
};

template <int W, int F>
__host__ __device__ constexpr size_t tile_point_bytes(int NQ) {
  return (TileRec<W>::STRIDE + NQ * TileVals<F>::STRIDE + 4) * 4;  // ... id, mirror id, two factors
}
__host__ __device__ constexpr size_t tile_fixed_bytes(int T, int NG) {
  return (size_t)T * T * sizeof(long long) + (size_t)(2 * NG * 64 + 1 + T + 2) * sizeof(int);
}

// The points of corner row l1 = L1 .. 7 added to the lane's cells
template <int W, int F, int NQ, int PP, int L1>
struct TileRows {
  template <typename Range>
  __device__ __forceinline__ static void run(const Range &range, const float *recs, const float *vals, int cp, int col,
                                             int plane, float2 (&acc)[PP][TileGroups<W>::T][F / 2]) {
    using Rec = TileRec<W>;
    int i, iend;
    range(L1, i, iend);
    const float *rec = recs + i * Rec::STRIDE;
    const float *vp = vals + (i * NQ + cp) * TileVals<F>::STRIDE;
#pragma unroll 1
    for (; i < iend; ++i, rec += Rec::STRIDE, vp += NQ * TileVals<F>::STRIDE) {
      const float w2 = rec[Rec::W2 + col];
      float w0[PP];
      if constexpr (PP == 2) {
        const float2 x = *reinterpret_cast<const float2 *>(rec + Rec::W0 + plane);
        w0[0] = x.x;
        w0[1] = x.y;
      } else {
        w0[0] = rec[Rec::W0 + plane];
      }
      float2 w1[W];
#pragma unroll
      for (int j = 0; j + 1 < W; j += 2) {
        const float4 x = *reinterpret_cast<const float4 *>(rec + 2 * j);
        w1[j] = make_float2(x.x, x.y);
        w1[j + 1] = make_float2(x.z, x.w);
      }
      if constexpr (W & 1) w1[W - 1] = *reinterpret_cast<const float2 *>(rec + 2 * (W - 1));
      float2 v[F / 2];
#pragma unroll
      for (int f = 0; f + 1 < F / 2; f += 2) {
        const float4 x = *reinterpret_cast<const float4 *>(vp + 2 * f);
        v[f] = make_float2(x.x, x.y);
        v[f + 1] = make_float2(x.z, x.w);
      }
      if constexpr ((F / 2) & 1) v[F / 2 - 1] = *reinterpret_cast<const float2 *>(vp + F - 2);
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        const float w02 = w0[k] * w2;
        const float2 ww = make_float2(w02, w02);
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const float2 w = __fmul2_rn(ww, w1[j]);
#pragma unroll
          for (int f = 0; f < F / 2; ++f) acc[k][L1 + j][f] = __ffma2_rn(w, v[f], acc[k][L1 + j][f]);
        }
      }
    }
    if constexpr (L1 + 1 < kBin) TileRows<W, F, NQ, PP, L1 + 1>::run(range, recs, vals, cp, col, plane, acc);
  }
};

// F / 2 channels per lane in NQ parts.
// Warps per block: two blocks fit an SM either way (the staged records), and one channel's accumulators
// (one plane and up to 15 rows a lane) leave registers for 14 warps in each, with a point per thread
// and smaller tasks (512 images of 128^2, W = 7: 1.26 -> 1.00 ms against 6 warps and two planes a lane).
__host__ __device__ constexpr int tile_warps(int W, int F) { return W > 2 && F == 2 ? 14 : kTileWarps; }

template <int KT, int W, int F, int NQ, int PP, bool HALF>
__global__ void __launch_bounds__(tile_warps(W, F) * 32, W == 2 ? 4 : 2) spread_tile_kernel(const SpreadParams a) {
  constexpr bool ES = KT == COV3D_KERNEL_ES;
  using G = TileGroups<W>;
  using Rec = TileRec<W>;
  constexpr int VS = TileVals<F>::STRIDE;
  constexpr int T = G::T, NG = G::NG, NK = NG * 64;
  constexpr int CH = NQ * F / 2;                 // channels per pass
  constexpr int NPL = PP * (4 / NQ);             // planes per task
  constexpr int PGS = (T + NPL - 1) / NPL;       // plane groups
  static_assert(PGS * NPL <= 16, "plane weights of a record");
  extern __shared__ float4 smem4[];
  float *recs = reinterpret_cast<float *>(smem4);                // max_sub * record stride
  float *vals = recs + (size_t)a.max_sub * Rec::STRIDE;          // max_sub * NQ * VS
  int *s_id = reinterpret_cast<int *>(vals + (size_t)a.max_sub * NQ * VS);
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
  constexpr int PPT = (kTileMaxSub + tile_warps(W, F) * 32 - 1) / (tile_warps(W, F) * 32);
  SortedPoint pt[PPT];
  int pkey[PPT];
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    const int k = tid + u * tile_warps(W, F) * 32;
    pkey[u] = -1;
    if (k < st.cnt) pt[u] = a.pts[st.first + k];
  }
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    if (tid + u * tile_warps(W, F) * 32 >= st.cnt) continue;
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
    s_row[e] = ES || (st.ts0 + ra < n && st.ts1 + rb < n) ? ((int64_t)m0 * n + m1) * n : -1;
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
    float4 *rec = reinterpret_cast<float4 *>(recs + slot * Rec::STRIDE);
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
    float w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = j < W ? weight(x1, y1, j) : 0.0f;
#pragma unroll
    for (int u = 0; u < Rec::W2 / 4; ++u) rec[u] = make_float4(w[2 * u], w[2 * u], w[2 * u + 1], w[2 * u + 1]);
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = weight(x2, y2, b2 + j - l2);
    rec[Rec::W2 / 4] = make_float4(w[0], w[1], w[2], w[3]);
    rec[Rec::W2 / 4 + 1] = make_float4(w[4], w[5], w[6], w[7]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = 4 * u + j < T ? weight(x0, y0, 4 * u + j - l0) : 0.0f;
      rec[Rec::W0 / 4 + u] = make_float4(w[0], w[1], w[2], w[3]);
    }
    const int id = sp_id<HALF>(sp.idf);
    const float sc = ((a.nyquist && sp_nyquist(sp.idf)) ? 0.0f : a.scale) * ctf_factor(a.ctf, a.ctfc, a.g, id);
    const int mid = sp_pair<HALF>(sp.idf) ? mirror_id(a.g, id) : -1;
    s_id[slot] = sp_conj<HALF>(sp.idf) ? ~id : id;  // a negative id: the value's conjugate
    s_mid[slot] = mid;
    s_sc[slot] = sc;
    if (mid >= 0) s_scm[slot] = a.scale * ctf_factor(a.ctf, a.ctfc, a.g, mid);
  }

  const int q = lane >> 3, c = lane & 7;
  const int cp = q % NQ;  // channel part
  for (int p0 = 0; p0 < a.nch; p0 += CH) {
    __syncthreads();
    // this pass's channel values in sorted order.  A record of kSortHalf that stands for a pair of
    // mirror pixels takes the sum of the one's value and the conjugate of the other's, which has
    // the same real part after the inverse transform.
    // Four elements' loads in flight per thread: the gathers' latency is most of the staging.
    constexpr int GU = 4;
    const int total = st.cnt * CH;
    for (int e0 = tid; e0 < total; e0 += GU * tile_warps(W, F) * 32) {
      float2 x[GU], m[GU];
      int sl[GU];
#pragma unroll
      for (int u = 0; u < GU; ++u) {
        const int e = e0 + u * tile_warps(W, F) * 32;
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
        const int ch = e0 + u * tile_warps(W, F) * 32 - slot * CH;
        const float sc = s_sc[slot];
        float2 v = make_float2(x[u].x * sc, HALF && s_id[slot] < 0 ? -(x[u].y * sc) : x[u].y * sc);
        if (HALF && s_mid[slot] >= 0) {
          const float sm = s_scm[slot];
          v.x = fmaf(m[u].x, sm, v.x);
          v.y = fmaf(-m[u].y, sm, v.y);
        }
        const int part = ch / (F / 2);
        *reinterpret_cast<float2 *>(vals + (slot * NQ + part) * VS + 2 * (ch - part * (F / 2))) = v;
      }
    }
    if (tid == 0) *s_task = 0;
    __syncthreads();

    for (;;) {
      int task = 0;
      if (lane == 0) task = atomicAdd(s_task, 1);
      task = __shfl_sync(0xffffffffu, task, 0);
      if (task >= PGS * NG) break;
      const int g = task / PGS, pa0 = (task - g * PGS) * NPL;
      const int plane = pa0 + (q / NQ) * PP;  // this lane's first plane
      const int lo = max(pa0 - W + 1, 0), hi = min(pa0 + NPL - 1, kBin - 1);
      if (lo > hi || s_off[g * 64] == s_off[g * 64 + 64]) continue;
      float2 acc[PP][T][F / 2];
#pragma unroll
      for (int k = 0; k < PP; ++k)
#pragma unroll
        for (int r = 0; r < T; ++r)
#pragma unroll
          for (int f = 0; f < F / 2; ++f) acc[k][r][f] = make_float2(0.f, 0.f);
      auto range = [&](int l1, int &i, int &iend) {
        i = s_off[g * 64 + l1 * 8 + lo];
        iend = s_off[g * 64 + l1 * 8 + hi + 1];
      };
      TileRows<W, F, NQ, PP, 0>::run(range, recs, vals, cp, c, plane, acc);
      // the finished cells go to the global grid
      const int co = s_col[G::base(g) + c];
      if (!ES && co < 0) continue;
      const int ch0 = p0 + cp * (F / 2);  // this lane's first channel
#pragma unroll
      for (int k = 0; k < PP; ++k) {
        if (plane + k >= T) break;
#pragma unroll
        for (int r = 0; r < T; ++r) {
          const long long ro = s_row[(plane + k) * T + r];
          if (!ES && ro < 0) continue;
          float2 *dst = a.grid + (ro + co) * a.cs + (int64_t)(a.ch0 + ch0) * a.chs;
#pragma unroll
          for (int f = 0; f < F / 2; ++f) {
            const float2 x = acc[k][r][f];
            if (ch0 + f < a.nch && (x.x != 0.0f || x.y != 0.0f)) atomicAdd(dst + f * a.chs, x);
          }
        }
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

template <int KT, int W, int F, int NQ, int PP, bool HALF>
int launch_tile(const SpreadParams &a, int64_t max_blocks, cudaStream_t st) {
  if (a.max_sub > kTileMaxSub) {
    set_error("subproblems of %d points; the spreading holds %d", a.max_sub, kTileMaxSub);
    return COV3D_EINVAL;
  }
  const size_t smem = (size_t)a.max_sub * tile_point_bytes<W, F>(NQ) + 8 +
                      tile_fixed_bytes(TileGroups<W>::T, TileGroups<W>::NG);
  return launch_spread_kernel(spread_tile_kernel<KT, W, F, NQ, PP, HALF>, "spread_tile_kernel", smem, a, max_blocks, st,
                              tile_warps(W, F));
}

// Linear windows: few enough FMAs per point that staging and waiting bound the kernel, so the layouts
// hold at most 3 channels x 9 rows in a lane's registers and four blocks fit an SM (with
// subproblems of 208 points; 10 channels, 1024 images of 128^2: 1.96 ms against 2.20 with 5 channels a
// lane and two blocks of 384 points).  Twelve channels in a pass, then the layout that holds the rest
// (5 channels, 256 images of 32^2: 51 us at two blocks, 41 at four).
template <int KT, int W, bool HALF>
int launch_linear_channels(SpreadParams a, int nchan, int64_t max_blocks, cudaStream_t st) {
  const int rest = nchan % 12, whole = rest > 8 ? nchan : nchan - rest;
  if (whole > 0) {
    a.ch0 = 0;
    a.nch = whole;
    COV3D_TRY((launch_tile<KT, W, 6, 4, 1, HALF>(a, max_blocks, st)));
  }
  a.ch0 = whole;
  a.nch = nchan - whole;
  if (a.nch >= 7) return launch_tile<KT, W, 4, 4, 1, HALF>(a, max_blocks, st);
  if (a.nch >= 3) return launch_tile<KT, W, 6, 2, 1, HALF>(a, max_blocks, st);
  if (a.nch == 2) return launch_tile<KT, W, 4, 1, 1, HALF>(a, max_blocks, st);
  if (a.nch == 1) return launch_tile<KT, W, 2, 1, 2, HALF>(a, max_blocks, st);
  return COV3D_OK;
}

// Passes of ten channels in one launch, then the rest in the layout that holds it (3 channels a lane
// and three blocks of 256 points per SM, as for linear windows: 5.58 ms against 4.74, and 1.07 against
// 0.44 for 5 channels: here the FMAs bound).
template <int KT, int W, bool HALF>
int launch_tile_channels(SpreadParams a, int nchan, int64_t max_blocks, cudaStream_t st) {
  const int rest = nchan % 10, whole = rest > 5 ? nchan : nchan - rest;
  if (whole > 0) {
    a.ch0 = 0;
    a.nch = whole;
    COV3D_TRY((launch_tile<KT, W, 10, 2, 1, HALF>(a, max_blocks, st)));
  }
  a.ch0 = whole;
  a.nch = nchan - whole;
  if (a.nch >= 3) return launch_tile<KT, W, 10, 1, 1, HALF>(a, max_blocks, st);
  if (a.nch == 2) return launch_tile<KT, W, 4, 1, 1, HALF>(a, max_blocks, st);
  if (a.nch == 1) return launch_tile<KT, W, 2, 1, 1, HALF>(a, max_blocks, st);
  return COV3D_OK;
}

template <int KT, int W>
int launch_w(const SpreadParams &a, int nchan, int64_t max_blocks, cudaStream_t st) {
  if constexpr (W == 2) {
    return a.half ? launch_linear_channels<KT, W, true>(a, nchan, max_blocks, st)
                  : launch_linear_channels<KT, W, false>(a, nchan, max_blocks, st);
  } else {
    return a.half ? launch_tile_channels<KT, W, true>(a, nchan, max_blocks, st)
                  : launch_tile_channels<KT, W, false>(a, nchan, max_blocks, st);
  }
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
