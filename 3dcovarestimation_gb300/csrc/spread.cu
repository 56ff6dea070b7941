// Spreading ("type-1" half of the NUFFT; exact adjoint of interp.cu, replacing the
// reference's grid_sample backward with FP32 global atomics, nufft_plan.py:171-242), over the
// bin-sorted point records of points_sort.cu.  See spread_kernel for the decomposition.

#include "cov3d_device.cuh"

namespace cov3d {

namespace {

constexpr int kBin = 8;
constexpr int kSpreadWarps = 16;

struct SpreadParams {
  PointGeom g;
  KernelSpec k;
  Bins bins;
  const SortedPoint *pts;
  const int *sub_bin;
  const int *sub_first;
  const int *sub_count;
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

constexpr int kLMin = -8;   // window corners relative to the bin lie in [kLMin, kLMin + 16)
constexpr int kKeys = 256;  // sort key (l1 - kLMin) * 16 + (l0 - kLMin)
constexpr int kFoldRanges = 3;  // window-corner rows l1 summed in FP32 between compensated folds

// Per-point record staged once per block, in elements of float2 (each weight twice, the operand
// of a packed multiply: spread_kernel) or float (each weight once, splatted in a register:
// spread_rows_kernel, where the bytes shared memory returns per visit are the bound): the
// axis-0 weights by tile plane and the axis-2 weights by tile column, zero
// outside the point's window (the column slot T is always zero, for idle lanes), and the W
// axis-1 weights with ROWS - 1 zeros before them and max(ROWS - 1, 1) after.  A lane's weight
// for tile row b of a point with window corner l1 is then
// rec[plane] * rec[W1 + b - l1] * rec[W2 + column], with no corner arithmetic and no select:
// lanes outside the window read zeros.
template <int W, int ROWS>
struct PointRec {
  static constexpr int T = kBin + W - 1;
  static constexpr int W1 = T + ROWS - 1;            // axis-1 weight o1 at W1 + o1
  static constexpr int Z1 = ROWS > 1 ? ROWS - 1 : 1;  // zeros after the axis-1 weights
  static constexpr int W2 = W1 + W + Z1;             // axis-2 weights by column
  static constexpr int F2 = (W2 + T + 2) / 2 * 2;    // float2 per record (even)
};

// Shared memory after the staged channel values: tile row offsets, point records, sort keys,
// point ids, prologue factors, key counters and offsets, column offsets, the task counter.
struct StageSmem {
  long long *rowoff;  // T * T
  void *rec;          // max_sub * F2 record elements (float2, or float for scalar weights)
  int *key;           // max_sub
  unsigned *pid;      // max_sub: the record's id with kPairBit and kConjBit
  float *sc, *scm;    // max_sub each: factors of the id and of its mirror pixel
  int *cnt, *off;     // kKeys, kKeys + 1
  int *coloff;        // T
  int *task;          // 1
};

__host__ __device__ constexpr size_t stage_bytes(int max_sub, int T, int F2, size_t esize) {
  return (size_t)T * T * sizeof(long long) + (size_t)max_sub * (F2 * esize + 4 * sizeof(int)) +
         (size_t)(2 * kKeys + 2 + T) * sizeof(int);
}

__device__ __forceinline__ StageSmem carve(void *base, int max_sub, int T, int F2, int esize) {
  StageSmem s;
  s.rowoff = static_cast<long long *>(base);
  s.rec = s.rowoff + T * T;
  s.key = reinterpret_cast<int *>(static_cast<char *>(s.rec) + (size_t)max_sub * F2 * esize);
  s.pid = reinterpret_cast<unsigned *>(s.key + max_sub);
  s.sc = reinterpret_cast<float *>(s.pid + max_sub);
  s.scm = s.sc + max_sub;
  s.cnt = reinterpret_cast<int *>(s.scm + max_sub);
  s.off = s.cnt + kKeys;
  s.coloff = s.off + kKeys + 1;
  s.task = s.coloff + T;
  return s;
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

// Stage 1 of both spreading kernels: the block counting-sorts its points by the (axis-1,
// axis-0) corner (l1, l0) of their window and stages, in that order, each point's record, id
// and prologue factor (im_backward's Nyquist zeroing, CTF and scale), then the global offsets
// of the tile's rows and columns.  The caller synchronises before reading them.
// a weight as a record element: twice (a packed-multiply operand) or once
__device__ __forceinline__ void put_weight(float2 *e, float x) { *e = make_float2(x, x); }
__device__ __forceinline__ void put_weight(float *e, float x) { *e = x; }

template <int KT, int W, int ROWS, typename E, bool HALF>
__device__ __forceinline__ void stage_subproblem(const SpreadParams &a, const StageSmem &s, const SubTile &st) {
  using Rec = PointRec<W, ROWS>;
  constexpr int T = Rec::T;
  constexpr int F2 = Rec::F2;
  const int n = a.g.n;
  const int tid = threadIdx.x;
  for (int e = tid; e < kKeys; e += blockDim.x) s.cnt[e] = 0;
  __syncthreads();
  // sort keys and ranks
  for (int k = tid; k < st.cnt; k += blockDim.x) {
    const SortedPoint sp = a.pts[st.first + k];
    int c0 = record_cell<KT, W, HALF>(sp.t0, a.g.frac), c1 = record_cell<KT, W, HALF>(sp.t1, a.g.frac);
    if (KT == COV3D_KERNEL_ES) {
      c0 = wrap1(c0, n);
      c1 = wrap1(c1, n);
    }
    const int key = (min(max(c1 - st.ts1 - kLMin, 0), 15) << 4) | min(max(c0 - st.ts0 - kLMin, 0), 15);
    s.key[k] = key | (atomicAdd(s.cnt + key, 1) << 8);
  }
  __syncthreads();
  if (tid < 32) {  // exclusive scan of the 256 counters by one warp, 8 per lane
    int v[kKeys / 32], sum = 0;
#pragma unroll
    for (int u = 0; u < kKeys / 32; ++u) {
      v[u] = s.cnt[tid * (kKeys / 32) + u];
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
    for (int u = 0; u < kKeys / 32; ++u) {
      s.off[tid * (kKeys / 32) + u] = base;
      base += v[u];
    }
    if (tid == 31) s.off[kKeys] = incl;
  }
  __syncthreads();
  // records, point ids and prologue factors in sorted order
  for (int k = tid; k < st.cnt; k += blockDim.x) {
    const SortedPoint sp = a.pts[st.first + k];
    const int kr = s.key[k];
    const int slot = s.off[kr & 255] + (kr >> 8);
    float w0[W], w1[W], w2[W];
    int c0 = taps<KT, W, HALF>(sp.t0, a.g.frac, a.k.beta, w0);
    taps<KT, W, HALF>(sp.t1, a.g.frac, a.k.beta, w1);
    int c2 = taps<KT, W, HALF>(sp.t2, a.g.frac, a.k.beta, w2);
    if (KT == COV3D_KERNEL_ES) {
      c0 = wrap1(c0, n);
      c2 = wrap1(c2, n);
    }
    E *rec = static_cast<E *>(s.rec) + slot * F2;
    const int l0 = c0 - st.ts0, l2 = c2 - st.ts2;  // bin-local corners, >= 1 - W (zero padding below)
    const float z = 0.0f;
#pragma unroll
    for (int e = 0; e < T; ++e) {
      put_weight(rec + e, z);
      put_weight(rec + Rec::W2 + e, z);
    }
    put_weight(rec + Rec::W2 + T, z);
#pragma unroll
    for (int e = T; e < Rec::W1; ++e) put_weight(rec + e, z);
#pragma unroll
    for (int e = Rec::W1 + W; e < Rec::W2; ++e) put_weight(rec + e, z);
#pragma unroll
    for (int r = 0; r < W; ++r) {
      if (l0 + r >= 0 && l0 + r < T) put_weight(rec + l0 + r, w0[r]);
      if (l2 + r >= 0 && l2 + r < T) put_weight(rec + Rec::W2 + l2 + r, w2[r]);
      put_weight(rec + Rec::W1 + r, w1[r]);
    }
    const int id = sp_id<HALF>(sp.idf);
    float sc = (a.nyquist && sp_nyquist(sp.idf)) ? 0.0f : a.scale;
    sc *= ctf_factor(a.ctf, a.ctfc, a.g, id);
    s.pid[slot] = sp.idf & ~kNyquistBit;
    s.sc[slot] = sc;
    if (sp_pair<HALF>(sp.idf)) s.scm[slot] = a.scale * ctf_factor(a.ctf, a.ctfc, a.g, mirror_id(a.g, id));
  }
  // global offsets of the tile's rows (axes 0, 1) and columns (axis 2)
  for (int e = tid; e < T * T; e += blockDim.x) {
    const int ra = e / T, rb = e - (e / T) * T;
    int m0 = st.ts0 + ra, m1 = st.ts1 + rb;
    bool ok = true;
    if (KT == COV3D_KERNEL_ES) {
      m0 = m0 >= n ? m0 - n : m0;
      m1 = m1 >= n ? m1 - n : m1;
    } else {
      ok = m0 < n && m1 < n;
    }
    m0 += a.shift;
    m1 += a.shift;
    m0 = m0 >= n ? m0 - n : m0;
    m1 = m1 >= n ? m1 - n : m1;
    s.rowoff[e] = ok ? ((int64_t)m0 * n + m1) * n : -1;
  }
  for (int e = tid; e < T; e += blockDim.x) {
    int m2 = st.ts2 + e;
    bool ok = true;
    if (KT == COV3D_KERNEL_ES) {
      m2 = m2 >= n ? m2 - n : m2;
    } else {
      ok = m2 < n;
    }
    m2 += a.shift;
    m2 = m2 >= n ? m2 - n : m2;
    s.coloff[e] = ok ? m2 : -1;
  }
}

// The scaled value of one channel of a staged record: src = values + channel * channel stride.  A
// record of kSortHalf that stands for a pair of mirror pixels takes the sum of the one's value
// and the conjugate of the other's, which has the same real part after the inverse transform.
template <bool HALF>
__device__ __forceinline__ float2 record_value(const SpreadParams &a, const StageSmem &s, int slot, const float2 *src) {
  const unsigned pid = s.pid[slot];
  const float sc = s.sc[slot];
  const int id = sp_id<HALF>(pid);
  const float2 x = __ldg(src + (int64_t)id * a.ips);
  float2 v = make_float2(x.x * sc, sp_conj<HALF>(pid) ? -(x.y * sc) : x.y * sc);
  if (sp_pair<HALF>(pid)) {
    const float sm = s.scm[slot];
    const float2 m = __ldg(src + (int64_t)mirror_id(a.g, id) * a.ips);
    v.x = fmaf(m.x, sm, v.x);
    v.y = fmaf(-m.y, sm, v.y);
  }
  return v;
}

// TwoSum (Knuth) on both lanes of a float2: s + d = s' + e exactly, e added to the error sum
// err.  Differences are fused multiply-adds with -1, which round exactly like a subtraction.
__device__ __forceinline__ void two_sum2(float2 &s, float2 &err, const float2 d) {
  const float2 m1 = make_float2(-1.0f, -1.0f);
  const float2 s2 = __fadd2_rn(s, d);
  const float2 bb = __ffma2_rn(s, m1, s2);   // s2 - s
  const float2 sb = __ffma2_rn(bb, m1, s2);  // s2 - bb
  const float2 e1 = __ffma2_rn(sb, m1, s);   // s - (s2 - bb)
  const float2 e2 = __ffma2_rn(bb, m1, d);   // d - bb
  err = __fadd2_rn(err, __fadd2_rn(e1, e2));
  s = s2;
}

// Lane layout of the row tasks: lane = g * T + c owns tile column c (T = 8 + W - 1 columns)
// and the channel pairs g, g + G, ..., G = 32 / T lane groups.
template <int W>
struct SpreadLanes {
  static constexpr int T = kBin + W - 1;
  static constexpr int G = 32 / T;
};

// Row tasks, for few channels.  One block per subproblem (a bin of 8^3 cells and at most
// max_sub of its points); the cells it can reach form a tile of the bin and a (W-1)-cell halo,
// T^3 cells.  After stage_subproblem, a task is one tile row: plane a, row b.  The points whose
// window covers it are the W contiguous ranges {l1 = b - o1, l0 in [a - W + 1, a]},
// o1 = 0 .. W-1, of the sorted order.  Lane (g, c) keeps the sums of cell (a, b, c) for its
// channel pairs in registers: each group of kFoldRanges ranges is summed in FP32 and, with COMP,
// added to the cell's (hi, lo) pair by a TwoSum, so the error of the cell's accumulation is that
// of one short FP32 sum per group.  The finished row goes to the global grid with one complex
// atomic per cell and channel.  Warps take tasks from a shared counter.  The block needs no
// shared-memory tile: its shared memory is the staged points only.
template <int KT, int W, int CPL, bool COMP, bool HALF>
__global__ void __launch_bounds__(kSpreadWarps * 32, W < 8 ? 2 : 1) spread_kernel(const SpreadParams a) {
  constexpr int T = SpreadLanes<W>::T;
  constexpr int G = SpreadLanes<W>::G;  // lane groups over channel pairs
  constexpr int NP = G * CPL;           // channel pairs staged per group
  using Rec = PointRec<W, 1>;
  constexpr int F2 = Rec::F2;
  extern __shared__ float4 smem4[];
  float4 *s_val = smem4;  // max_sub * NP
  const StageSmem s = carve(s_val + a.max_sub * NP, a.max_sub, T, F2, sizeof(float2));
  const float2 *recs = static_cast<const float2 *>(s.rec);
  const int sub = blockIdx.x;
  if (sub >= *a.nsub) return;
  const SubTile st = sub_tile(a, sub);
  stage_subproblem<KT, W, 1, float2, HALF>(a, s, st);

  const int tid = threadIdx.x, lane = tid & 31;
  const int g = lane / T, c = lane - (lane / T) * T;
  const bool lane_live = g < G;
  const int gv = lane_live ? g : 0;  // idle lanes compute pair 0 and drop it
  const int npairs = (a.nch + 1) / 2;
  for (int p0 = 0; p0 < npairs; p0 += NP) {  // channel groups of NP pairs
    __syncthreads();
    // this group's scaled channel pairs, in sorted order
    for (int e = tid; e < st.cnt * NP; e += blockDim.x) {
      const int slot = e / NP, pp = p0 + (e - (e / NP) * NP);
      const float2 *src = a.vals + (int64_t)(a.ch0 + 2 * pp) * a.ics;
      const float2 v0 = 2 * pp < a.nch ? record_value<HALF>(a, s, slot, src) : make_float2(0.f, 0.f);
      const float2 v1 = 2 * pp + 1 < a.nch ? record_value<HALF>(a, s, slot, src + a.ics) : make_float2(0.f, 0.f);
      s_val[e] = make_float4(v0.x, v0.y, v1.x, v1.y);
    }
    if (tid == 0) *s.task = 0;
    __syncthreads();

    for (;;) {
      int task = 0;
      if (lane == 0) task = atomicAdd(s.task, 1);
      task = __shfl_sync(0xffffffffu, task, 0);
      if (task >= T * T) break;
      const int pa = task / T;
      const int rb = task - pa * T;  // the task's row
      const int b0lo = max(pa - W + 1 - kLMin, 0), b0hi = min(pa - kLMin, 15);
      // cell sums of channel pairs (0, 1) and (2, 3) of each pair group, and their TwoSum errors
      float2 hi01[CPL], hi23[CPL], lo01[CPL], lo23[CPL];
#pragma unroll
      for (int u = 0; u < CPL; ++u) {
        hi01[u] = hi23[u] = lo01[u] = lo23[u] = make_float2(0.f, 0.f);
      }
      bool any = false;
      const float2 *w2c = recs + Rec::W2 + c;  // this lane's column weight, record 0
      for (int l1g = rb; l1g > rb - W; l1g -= kFoldRanges) {
        float2 part01[CPL], part23[CPL];  // packed FP32 (FFMA2), same rounding as fmaf
#pragma unroll
        for (int u = 0; u < CPL; ++u) {
          part01[u] = make_float2(0.f, 0.f);
          part23[u] = make_float2(0.f, 0.f);
        }
        bool in = false;
#pragma unroll
        for (int sr = 0; sr < kFoldRanges; ++sr) {
          const int l1 = l1g - sr;
          const int b1 = l1 - kLMin;
          if (l1 <= rb - W || b1 < 0 || b1 > 15 || b0lo > b0hi) continue;
          const int ibeg = s.off[(b1 << 4) | b0lo], iend = s.off[((b1 << 4) | b0hi) + 1];
          in |= lane_live && ibeg < iend;
          const int k1 = Rec::W1 + (lane_live ? rb - l1 : W);  // a zero slot for idle lanes
          // two points per iteration; a lane whose column is outside a point's window
          // multiplies by a zero weight
          int i = ibeg;
          for (; i + 1 < iend; i += 2) {
            const float2 *ra = recs + i * F2, *rb2 = ra + F2;
            const float2 wa = __fmul2_rn(__fmul2_rn(ra[pa], ra[k1]), w2c[i * F2]);
            const float2 wb = __fmul2_rn(__fmul2_rn(rb2[pa], rb2[k1]), w2c[(i + 1) * F2]);
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
              const float4 xa = s_val[i * NP + gv + G * u];
              const float4 xb = s_val[(i + 1) * NP + gv + G * u];
              part01[u] = __ffma2_rn(wa, make_float2(xa.x, xa.y), part01[u]);
              part23[u] = __ffma2_rn(wa, make_float2(xa.z, xa.w), part23[u]);
              part01[u] = __ffma2_rn(wb, make_float2(xb.x, xb.y), part01[u]);
              part23[u] = __ffma2_rn(wb, make_float2(xb.z, xb.w), part23[u]);
            }
          }
          if (i < iend) {
            const float2 *ra = recs + i * F2;
            const float2 wa = __fmul2_rn(__fmul2_rn(ra[pa], ra[k1]), w2c[i * F2]);
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
              const float4 xa = s_val[i * NP + gv + G * u];
              part01[u] = __ffma2_rn(wa, make_float2(xa.x, xa.y), part01[u]);
              part23[u] = __ffma2_rn(wa, make_float2(xa.z, xa.w), part23[u]);
            }
          }
        }
        if (!in) continue;
        if (!any) {  // the first group: its fold, TwoSum(0, sum), is (sum, 0) exactly
#pragma unroll
          for (int u = 0; u < CPL; ++u) {
            hi01[u] = part01[u];
            hi23[u] = part23[u];
          }
        } else {
#pragma unroll
          for (int u = 0; u < CPL; ++u) {
            if (!COMP) {
              hi01[u] = __fadd2_rn(hi01[u], part01[u]);
              hi23[u] = __fadd2_rn(hi23[u], part23[u]);
            } else {
              two_sum2(hi01[u], lo01[u], part01[u]);
              two_sum2(hi23[u], lo23[u], part23[u]);
            }
          }
        }
        any = true;
      }
      // the finished cell goes to the global grid
      if (!any) continue;
      const long long ro = s.rowoff[pa * T + rb];
      const int co = s.coloff[c];
      if (ro < 0 || co < 0) continue;
#pragma unroll
      for (int u = 0; u < CPL; ++u) {
        const int pp = p0 + gv + G * u;
        const float2 x01 = COMP ? __fadd2_rn(hi01[u], lo01[u]) : hi01[u];
        const float2 x23 = COMP ? __fadd2_rn(hi23[u], lo23[u]) : hi23[u];
        float2 *dst = a.grid + (ro + co) * a.cs + (int64_t)(a.ch0 + 2 * pp) * a.chs;
        if (2 * pp < a.nch && (x01.x != 0.0f || x01.y != 0.0f)) atomicAdd(dst, x01);
        if (2 * pp + 1 < a.nch && (x23.x != 0.0f || x23.y != 0.0f)) atomicAdd(dst + a.chs, x23);
      }
    }
  }
}

// Spreading for the ES windows (W = 4 .. 8), any number of channels.  One block per subproblem (a bin
// of 8^3 cells and at most max_sub of its points); the cells it can reach are a tile of T^3,
// T = 8 + W - 1.  The block sorts its points by (axis-2 group, l1, l0), l the bin-local corner of
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
// columns of three rows of one plane, had 16 visits and 2.2x the multiply-adds.  Measured on the step at L = 128, B = 1024, r = 10: 8.6 -> 5.3 ms, of which staging
// (sort, weights, gathered values) about 2.0, the flush 0.9; one channel at W = 7, 512 images of
// 128^2: 6.2 -> 1.2 ms.
//
// Each cell's sum is plain FP32 over the points of one group of one subproblem (some 30 terms at
// one point per cell, a third of what the predecessor summed before its first TwoSum fold; two or
// three partial sums folded by TwoSum round to the float sum of the partials), and the partial sums
// meet in FP32 global atomics, so `compensated` changes nothing here.
// per block, two blocks per SM (168 registers); 5 or 4 warps measured 5.8 and 6.8 ms against 5.3 (a
// unrolled point loop is slower too: the ranges hold some ten points), 7 spill
constexpr int kTileWarps = 6;
constexpr int kTileMaxSub = 448;  // largest subproblem of an ES plan (three points per thread)

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

// F / 2 channels per lane in NQ parts: 2 x 5 channels per pass, or one part of 5, 2 or 1.
template <int KT, int W, int F, int NQ, int PP, bool HALF>
__global__ void __launch_bounds__(kTileWarps * 32, 2) spread_tile_kernel(const SpreadParams a) {
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
  constexpr int PPT = (kTileMaxSub + kTileWarps * 32 - 1) / (kTileWarps * 32);
  SortedPoint pt[PPT];
  int pkey[PPT];
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    const int k = tid + u * kTileWarps * 32;
    pkey[u] = -1;
    if (k < st.cnt) pt[u] = a.pts[st.first + k];
  }
#pragma unroll
  for (int u = 0; u < PPT; ++u) {
    if (tid + u * kTileWarps * 32 >= st.cnt) continue;
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
    for (int e0 = tid; e0 < total; e0 += GU * kTileWarps * 32) {
      float2 x[GU], m[GU];
      int sl[GU];
#pragma unroll
      for (int u = 0; u < GU; ++u) {
        const int e = e0 + u * kTileWarps * 32;
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
        const int ch = e0 + u * kTileWarps * 32 - slot * CH;
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
                         cudaStream_t st, int warps = kSpreadWarps) {
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

// One launch for all channels: the block sorts and stages its points once.  With three or more
// channel pairs a lane group takes two pairs of a row task (bilinear step: 4.6 against 7.4 ms with
// tasks of three rows over two lane halves), otherwise the (at most two, G >= 2) pairs are spread
// over the lane groups.
template <int KT, int W, bool COMP, bool HALF>
int launch_wc(SpreadParams a, int nchan, int64_t max_blocks, cudaStream_t st) {
  constexpr int T = kBin + W - 1;
  constexpr int G = SpreadLanes<W>::G;
  a.ch0 = 0;
  a.nch = nchan;
  const int npairs = (nchan + 1) / 2;
  if (npairs >= 3) {
    constexpr int CPL = 2;
    const size_t smem = (size_t)a.max_sub * G * CPL * sizeof(float4) +
                        stage_bytes(a.max_sub, T, PointRec<W, 1>::F2, sizeof(float2));
    return launch_spread_kernel(spread_kernel<KT, W, CPL, COMP, HALF>, "spread_kernel", smem, a, max_blocks, st);
  }
  static_assert(2 * G >= 2, "at most two channel pairs spread over the lane groups");
  const size_t smem =
      (size_t)a.max_sub * G * sizeof(float4) + stage_bytes(a.max_sub, T, PointRec<W, 1>::F2, sizeof(float2));
  return launch_spread_kernel(spread_kernel<KT, W, 1, COMP, HALF>, "spread_kernel", smem, a, max_blocks, st);
}

template <int KT, int W, int F, int NQ, int PP, bool HALF>
int launch_tile(const SpreadParams &a, int64_t max_blocks, cudaStream_t st) {
  const size_t smem = (size_t)a.max_sub * tile_point_bytes<W, F>(NQ) + 8 +
                      tile_fixed_bytes(TileGroups<W>::T, TileGroups<W>::NG);
  return launch_spread_kernel(spread_tile_kernel<KT, W, F, NQ, PP, HALF>, "spread_tile_kernel", smem, a, max_blocks, st,
                              kTileWarps);
}

// Passes of ten channels in one launch, then the rest in the layout that holds it.
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
  if (a.nch == 1) return launch_tile<KT, W, 2, 1, 2, HALF>(a, max_blocks, st);
  return COV3D_OK;
}

template <int KT, int W>
int launch_w(SpreadParams a, int nchan, bool comp, int64_t max_blocks, cudaStream_t st) {
  if constexpr (KT != COV3D_KERNEL_NEAREST) {
    return a.half ? launch_tile_channels<KT, W, true>(a, nchan, max_blocks, st)
                  : launch_tile_channels<KT, W, false>(a, nchan, max_blocks, st);
  } else {
    return comp ? launch_wc<KT, W, true, false>(a, nchan, max_blocks, st)
                : launch_wc<KT, W, false, false>(a, nchan, max_blocks, st);
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

int launch_spread(cov3d_plan *p, const void *values, int64_t in_ps, int64_t in_cs, int nchan, const EpilogueArgs &e,
                  void *grid, int64_t cell_stride, int64_t chan_stride, int shift, SortMode mode) {
  if (p->point_kind == kPointsNone || p->n_points == 0) {
    set_error("no points set");
    return COV3D_ESTATE;
  }
  COV3D_TRY(need_sorted(p, 1u << mode));
  const SortSet &ss = p->sets[mode];
  SpreadParams a{};
  a.g = make_geom(p);
  a.k = make_kernel(p);
  a.bins = p->bins;
  a.pts = ss.sorted;
  a.sub_bin = ss.sub_bin;
  a.sub_first = ss.sub_first;
  a.sub_count = ss.sub_count;
  a.nsub = ss.nsub;
  a.vals = static_cast<const float2 *>(values);
  a.ips = in_ps;
  a.ics = in_cs;
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
  if (p->bins.bs[0] != kBin || p->bins.bs[1] != kBin || p->bins.bs[2] != kBin) {
    set_error("spreading requires %d^3-cell bins", kBin);
    return COV3D_EINVAL;
  }
  const int64_t max_blocks = p->bins.nbins + p->n_points / p->max_sub + 1;
  const bool comp = p->compensated != 0;
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST: return launch_w<COV3D_KERNEL_NEAREST, 1>(a, nchan, comp, max_blocks, p->stream);
    case COV3D_KERNEL_LINEAR: return launch_w<COV3D_KERNEL_LINEAR, 2>(a, nchan, comp, max_blocks, p->stream);
    default:
      switch (p->width) {
        case 4: return launch_w<COV3D_KERNEL_ES, 4>(a, nchan, comp, max_blocks, p->stream);
        case 5: return launch_w<COV3D_KERNEL_ES, 5>(a, nchan, comp, max_blocks, p->stream);
        case 6: return launch_w<COV3D_KERNEL_ES, 6>(a, nchan, comp, max_blocks, p->stream);
        case 7: return launch_w<COV3D_KERNEL_ES, 7>(a, nchan, comp, max_blocks, p->stream);
        case 8: return launch_w<COV3D_KERNEL_ES, 8>(a, nchan, comp, max_blocks, p->stream);
        default: set_error("unsupported ES width %d (supported: 4..8)", p->width); return COV3D_EINVAL;
      }
  }
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
