// Interpolation ("type-2" half of the NUFFT, and the reference's grid_sample forward) over
// bin-sorted points: each bin's tile of the fine grid is read from HBM once into shared memory
// and reused by all its points; the projection epilogue (Nyquist zeroing, CTF multiply, 1/L)
// is fused.
#include "cov3d_device.cuh"

namespace cov3d {

namespace {

struct InterpParams {
  PointGeom g;
  KernelSpec k;
  Bins bins;
  const SortedPoint *pts;
  const int *sub_bin;
  const int *sub_first;
  const int *bin_off;  // first sorted point of each bin (exclusive scan of the bin counts)
  const int *nsub;
  const float2 *grid;
  int64_t cs, chs;
  int shift;
  int ch0;
  int nch;  // channels in this pass (<= 2 * CP)
  float2 *out;
  int64_t ops, ocs;
  const float *ctf;
  const CtfCoef *ctfc;
  int nyquist;
  float scale;
  int half;  // records of kSortHalf
  float density;  // points per fine-grid cell
};

constexpr int kBin = 8;
constexpr int kInterpWarps = 24;    // warps per block of the small tiles (two blocks per SM)
// Warps per block: 32 next to the wide windows' large tiles, one block per SM (ES, 10 channels:
// 11.9 against 12.0 ms with 24; the narrow tiles measured slower with 32)
template <int W, int CP>
struct InterpWarps {
  static constexpr int value = (W > 2 && CP >= 3) ? 32 : kInterpWarps;
};
constexpr int kInterpChunk = 1024;  // points staged at a time (20 KB; 2048 measured slightly slower)

// Channel pairs per pass: lanes are (window cell, channel pair) pairs, so W * CP <= 32, and the
// tile (bin + halo) of 2*CP complex channels must fit in shared memory.
template <int W>
struct InterpCP {
  static constexpr int value = W <= 2 ? 16 : 32 / W;
};

// One block per bin (see the kernel's first lines).  The block stages the bin's tile (bin +
// (W-1)-cell halo) of 2*CP channels in shared memory as [cell][channel] complex, then each warp
// takes one point at a time (32 / (W*CP) points for the narrow bilinear and nearest windows):
// lane (j, q) reads the two channels 2q, 2q+1 of tile[row][corner2 + j] for the W*W window
// rows -- W*CP contiguous 16-byte values per row, no bank conflicts -- and accumulates
// weight * value; the W partial sums of each pair are combined by a warp-shuffle tree and the
// epilogue (Nyquist zeroing, CTF, scale) is applied.
template <int KT, int W, int CP, bool HALF>
__global__ void __launch_bounds__(InterpWarps<W, CP>::value * 32) interp_kernel(const InterpParams a) {
  constexpr int T = kBin + W - 1;
  constexpr int CH = 2 * CP;
  constexpr int LANES = W * CP;
  // points per warp iteration: several when a point's W*CP lanes (and its 3W weights) fit more
  // than once into the warp, as for the bilinear and nearest kernels
  constexpr int PPW = (LANES >= 3 * W && 32 / LANES > 1) ? 32 / LANES : 1;
  extern __shared__ float4 tile4[];  // T^3 * CP float4 (= 2 complex), then the point records
  float2 *tile = reinterpret_cast<float2 *>(tile4);
  SortedPoint *s_sp = reinterpret_cast<SortedPoint *>(tile4 + T * T * T * CP);  // kInterpChunk
  // epilogue factors: of the id and, for kSortHalf, of its mirror pixel
  float *s_sc = reinterpret_cast<float *>(s_sp + kInterpChunk);
  const int sub = blockIdx.x;
  if (sub >= *a.nsub) return;
  const int bin = a.sub_bin[sub];
  const int first = a.sub_first[sub];
  // one block per bin: the block of the bin's first subproblem takes all of the bin's points,
  // kInterpChunk at a time, so the tile is staged once per bin (512 points per bin on average
  // at the cov-SGD workload, two subproblems; 14.1 -> 12.6 ms when they were of 288 points)
  if (first != a.bin_off[bin]) return;
  const int last = a.bin_off[bin + 1];
  int cnt = min(kInterpChunk, last - first);
  const int nb12 = a.bins.nb[1] * a.bins.nb[2];
  const int ts0 = (bin / nb12) * kBin;
  const int ts1 = ((bin / a.bins.nb[2]) % a.bins.nb[1]) * kBin;
  const int ts2 = (bin % a.bins.nb[2]) * kBin;
  const int n = a.g.n;
  const int tid = threadIdx.x;

  // stage the tile: per-row global offsets and per-cell axis-2 offsets are tabulated first, then
  // (channel, row, cell) elements are copied with cell fastest for coalesced global reads
  __shared__ long long s_rowoff[T * T];
  __shared__ int s_coloff[T];
  for (int e = tid; e < T * T; e += blockDim.x) {
    const int c0 = e / T, c1 = e - (e / T) * T;
    int m0 = ts0 + c0, m1 = ts1 + c1;
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
    s_rowoff[e] = ok ? ((int64_t)m0 * n + m1) * n * a.cs : -1;
  }
  for (int e = tid; e < T; e += blockDim.x) {
    int m2 = ts2 + e;
    bool ok = true;
    if (KT == COV3D_KERNEL_ES) {
      m2 = m2 >= n ? m2 - n : m2;
    } else {
      ok = m2 < n;
    }
    m2 += a.shift;
    m2 = m2 >= n ? m2 - n : m2;
    s_coloff[e] = ok ? m2 : -1;
  }
  __syncthreads();
  // the subproblem's point records and epilogue factors (Nyquist zeroing, CTF, scale)
  auto stage_points = [&](int from) {
    for (int k = tid; k < cnt; k += blockDim.x) {
      const SortedPoint sp = a.pts[from + k];
      s_sp[k] = sp;
      const int id = sp_id<HALF>(sp.idf);
      const float sc = (a.nyquist && sp_nyquist(sp.idf)) ? 0.0f : a.scale;
      s_sc[k] = sc * ctf_factor(a.ctf, a.ctfc, a.g, id);
      if (sp_pair<HALF>(sp.idf)) s_sc[kInterpChunk + k] = a.scale * ctf_factor(a.ctf, a.ctfc, a.g, mirror_id(a.g, id));
    }
  };
  stage_points(first);
  const float2 *gbase = a.grid + (int64_t)a.ch0 * a.chs;
  // asynchronous copies global -> shared (8 bytes each, zero-filled outside the grid / past the
  // pass's channels), all in flight before one wait.  A warp copies RPW tile rows (channel,
  // plane, row) at a time, lane (s, c2) cell c2 of its row s: the column offset is fixed per
  // lane, and only the row index is decomposed per copy
  {
    constexpr int RPW = 32 / T;
    const int lane = tid & 31, s = lane / T, c2 = lane - (lane / T) * T;
    if (s < RPW) {
      const int co = s_coloff[c2];
      const int64_t co_cs = co >= 0 ? (int64_t)co * a.cs : 0;
      const float2 *src0 = gbase + co_cs;
      const unsigned dst0 = (unsigned)__cvta_generic_to_shared(tile + c2 * CH);
      const int step = (int)(blockDim.x >> 5) * RPW;
      for (int row = (tid >> 5) * RPW + s; row < CH * T * T; row += step) {
        const int ch = row / (T * T);
        const int rowi = row - ch * (T * T);
        const long long ro = s_rowoff[rowi];
        const bool ok = ch < a.nch && ro >= 0 && co >= 0;
        const float2 *src = ok ? src0 + ro + (int64_t)ch * a.chs : gbase;
        const unsigned dst = dst0 + (unsigned)((rowi * T * CH + ch) * sizeof(float2));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0) : "memory");
      }
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  const int warp = tid >> 5, lane = tid & 31;
  // lane = (point slot pp, window cell j along axis 2, channel pair q)
  const int pp = lane / LANES, sl = lane - (lane / LANES) * LANES;
  const int j = sl / CP, q = sl - (sl / CP) * CP;
  const int lane0 = (pp < PPW ? pp : 0) * LANES;  // first lane of this lane's point slot
  const int wl = PPW == 1 ? lane : sl;             // this lane's tap among the point's 3W weights
  // the point slots' taps, per warp and double-buffered by iteration (see below)
  __shared__ __align__(16) float s_w[InterpWarps<W, CP>::value * 2 * PPW * 24];
  int wbuf = 0;
  for (int base = first;;) {
    for (int k0 = warp * PPW; k0 < cnt; k0 += InterpWarps<W, CP>::value * PPW) {
      const int k = k0 + pp;
      const bool pt_ok = pp < PPW && k < cnt;
      const SortedPoint sp = s_sp[pt_ok ? k : k0];
      int c0[3];
      c0[0] = record_cell<KT, W, HALF>(sp.t0, a.g.frac);
      c0[1] = record_cell<KT, W, HALF>(sp.t1, a.g.frac);
      c0[2] = record_cell<KT, W, HALF>(sp.t2, a.g.frac);
      // one kernel weight per lane wl < 3W, then shared through the warp
      float myw = 0.0f;
      if (wl < 3 * W) {
        const int d = wl / W, tq = wl - (wl / W) * W;
        const float td = d == 0 ? sp.t0 : d == 1 ? sp.t1 : sp.t2;
        myw = record_weight<KT, W, HALF>(td, d == 0 ? c0[0] : d == 1 ? c0[1] : c0[2], tq, a.g.frac, a.k.beta);
      }
      // through the warp's slot in shared memory (double-buffered by iteration): axis-0 taps at
      // 0, axis-1 at 8, axis-2 at 16, read back as broadcast 16-byte loads -- five loads and a
      // store instead of 13 shuffles in the queue the tile loads use (11.9 -> 11.5 ms)
      float *ws = s_w + ((warp * 2 + wbuf) * PPW + lane0 / LANES) * 24;
      if (wl < 3 * W) ws[(wl / W) * 8 + wl - (wl / W) * W] = myw;
      __syncwarp();
      float w0[8], w1[8];
      {
        const float4 a0 = *reinterpret_cast<const float4 *>(ws), a1 = *reinterpret_cast<const float4 *>(ws + 4);
        const float4 b0 = *reinterpret_cast<const float4 *>(ws + 8), b1 = *reinterpret_cast<const float4 *>(ws + 12);
        w0[0] = a0.x; w0[1] = a0.y; w0[2] = a0.z; w0[3] = a0.w; w0[4] = a1.x; w0[5] = a1.y; w0[6] = a1.z; w0[7] = a1.w;
        w1[0] = b0.x; w1[1] = b0.y; w1[2] = b0.z; w1[3] = b0.w; w1[4] = b1.x; w1[5] = b1.y; w1[6] = b1.z; w1[7] = b1.w;
      }
      const float wj = ws[16 + (j < W ? j : 0)];
      wbuf ^= 1;
      int l0 = c0[0], l1 = c0[1], l2 = c0[2];
      if (KT == COV3D_KERNEL_ES) {
        l0 = wrap1(l0, n);
        l1 = wrap1(l1, n);
        l2 = wrap1(l2, n);
      }
      l0 -= ts0;
      l1 -= ts1;
      l2 -= ts2;
      const int cell2 = l2 + j;
      const bool lane_ok = pt_ok && cell2 >= 0;
      const float4 *base = tile4 + cell2 * CP + q;
      // two packed FP32 accumulators (FFMA2: one instruction per channel pair of values; the
      // same rounding as two fmaf); each window plane is summed over its rows with the axis-1
      // weights first, then added with its axis-0 weight times this lane's axis-2 weight
      float2 a01 = make_float2(0.f, 0.f), a23 = make_float2(0.f, 0.f);
      if (lane_ok) {
        float2 ww1[W];
  #pragma unroll
        for (int i1 = 0; i1 < W; ++i1) ww1[i1] = make_float2(w1[i1], w1[i1]);
  #pragma unroll
        for (int i0 = 0; i0 < W; ++i0) {
          const int r0 = l0 + i0;
          if (KT != COV3D_KERNEL_ES && r0 < 0) continue;
          float2 p01 = make_float2(0.f, 0.f), p23 = make_float2(0.f, 0.f);
  #pragma unroll
          for (int i1 = 0; i1 < W; ++i1) {
            const int r1 = l1 + i1;
            if (KT != COV3D_KERNEL_ES && r1 < 0) continue;
            const float4 v = base[(r0 * T + r1) * T * CP];
            p01 = __ffma2_rn(ww1[i1], make_float2(v.x, v.y), p01);
            p23 = __ffma2_rn(ww1[i1], make_float2(v.z, v.w), p23);
          }
          const float w0j = w0[i0] * wj;
          const float2 ww0 = make_float2(w0j, w0j);
          a01 = __ffma2_rn(ww0, p01, a01);
          a23 = __ffma2_rn(ww0, p23, a23);
        }
      }
      // the W partial sums of each pair by a shuffle tree over the window cells j (lanes j*CP + q
      // of the slot): at each level cell j adds cell j + h, h = ceil(width / 2)
      float4 s = make_float4(a01.x, a01.y, a23.x, a23.y);
  #pragma unroll
      for (int lvl = 0; lvl < 3; ++lvl) {
        const int wc = lvl == 0 ? W : lvl == 1 ? (W + 1) / 2 : ((W + 1) / 2 + 1) / 2;
        if (wc <= 1) break;
        const int h = (wc + 1) / 2;
        float4 t;
        t.x = __shfl_down_sync(0xffffffffu, s.x, h * CP);
        t.y = __shfl_down_sync(0xffffffffu, s.y, h * CP);
        t.z = __shfl_down_sync(0xffffffffu, s.z, h * CP);
        t.w = __shfl_down_sync(0xffffffffu, s.w, h * CP);
        if (j + h < wc) {
          s.x += t.x;
          s.y += t.y;
          s.z += t.z;
          s.w += t.w;
        }
      }
      if (pt_ok && sl < CP) {
        // epilogue: vol_forward's Nyquist zeroing, CTF multiply and 1/L (projection_funcs.py:355-370)
        const int id = sp_id<HALF>(sp.idf);
        auto put = [&](int64_t to, float sc, float si) {
          float2 *o = a.out + to * a.ops + (int64_t)(a.ch0 + 2 * sl) * a.ocs;
          if (2 * sl < a.nch) o[0] = make_float2(s.x * sc, s.y * si);
          if (2 * sl + 1 < a.nch) o[a.ocs] = make_float2(s.z * sc, s.w * si);
        };
        const float sc = s_sc[k];
        put(id, sc, sp_conj<HALF>(sp.idf) ? -sc : sc);
        if (sp_pair<HALF>(sp.idf)) {  // the mirror pixel's values are the conjugates
          const float sm = s_sc[kInterpChunk + k];
          put(mirror_id(a.g, id), sm, -sm);
        }
      }
    }
    base += kInterpChunk;
    if (base >= last) break;
    cnt = min(kInterpChunk, last - base);
    __syncthreads();  // every warp is done with the previous points
    stage_points(base);
    __syncthreads();
  }
}

// ---------------------------------------------------------------- several points per tile load
//
// The ES windows (W = 4 .. 7) where a bin holds enough points.  The block of a bin sorts its points
// (kGroupChunk at a time) by the corner (axis-2 group, l1, l0) of their window: the windows of up to
// P points of one such bucket, a unit, lie in the same W x W rows and 8 columns of the tile, so each
// tile value loaded from shared memory serves P points.  A warp takes 4 / NQ units at a time; lane
// (unit, column c, channel part q) loads the F floats of its column and part from each row and adds
// them with each point's axis-1 weight, then axis-0 times axis-2 weight, in interp_kernel's order;
// the W columns of a point's window are then summed through shared memory by interp_kernel's tree,
// one lane per point and channel, so every value has interp_kernel's bits.
//
// interp_kernel reads 4 shared-memory wavefronts per row and point (W = 6, ten channels) and is bound
// by them; this one reads 5 per row and unit of 2.2 points on average at one point per cell, and is
// bound by the same pipe (70 %) and by latency at the twelve warps that its registers leave.  Twelve
// warps and chunks of 1024 measured best of 12 / 14 / 16 and 512 / 768 / 1024.  Where it is the
// faster one (group_pass): microseconds before and after, at points per fine-grid cell:
//   W = 6, 10 channels: 11463 -> 10283 at 1.0 (L = 128), 4498 -> 5486 at 0.3, 524 -> 659 at 0.25
//   W = 6, 5 channels: 1435 -> 899 at 1.0, 345 -> 365 at 0.12; 2 channels: 250 -> 199 at 0.12
//   W = 7, 4 channels: 1154 -> 1028 at 0.13; 10 channels: 4007 -> 3701 at 0.26, 1404 -> 1746 at 0.04
//   W = 5, 10 channels: 696 -> 698 at 0.5; W = 4, 10 channels: 747 -> 578 at 0.5
constexpr int kGroupWarps = 12;
constexpr int kGroupChunk = 1024;
constexpr int kUnitPts = 3;  // P: units of three fill 30 of 32 lanes in the column sum (10 channels)
constexpr int kSlot = 52;    // floats of a point's weights: three axes of up to 8, twice each; pad

template <int W, int F, int NQ>
struct GroupShape {
  static constexpr int T = TileGroups<W>::T;
  static constexpr int CH = NQ * F / 2;    // channels per pass
  static constexpr int UG = 4 / NQ;        // units per warp
  static constexpr int NK = TileGroups<W>::NG * 64;
  static constexpr int HC = (W + 1) / 2;   // columns of a window left after the first level of the sum
  static constexpr int RED = UG * kUnitPts * HC * NQ;  // a warp's column sums, in parts
  static constexpr int N1 = F == 5 ? (T * T * T * NQ + 3) / 4 * 4 : 0;  // fifth floats (16-byte multiple)
  static constexpr size_t TILE = (size_t)T * T * T * NQ * 16 + N1 * 4;
  static constexpr size_t bytes(bool half) {
    return TILE + kGroupChunk * (sizeof(SortedPoint) + (half ? 8 : 4) + 4) +
           (size_t)kGroupWarps * (UG * kUnitPts * kSlot + (RED * F + 3) / 4 * 4) * 4 + (2 * NK + 2) * 4 + kGroupChunk;
  }
};

// The four-float parts of a cell are rotated by the cell's index, so that the staging's copies of one
// channel to consecutive cells spread over the banks.
template <int NQ>
__host__ __device__ constexpr int part_slot(int cell, int part) {
  return NQ * cell + ((part + cell) & (NQ - 1));
}

// Column sums of NP points (1 .. P) of this lane's unit, whose window corner is tile cell `cell0` of
// this lane's column
template <int W, int F, int NQ, int NP>
__device__ __forceinline__ void unit_sums(const float4 *tile4, const float *t1, int cell0, int q, const float *const (&slot)[kUnitPts],
                                          const int (&o2)[kUnitPts], int c, float *red4, float *red1) {
  constexpr int T = TileGroups<W>::T;
  const float4 *t4[NQ];  // by the row's rotation
#pragma unroll
  for (int r = 0; r < NQ; ++r) t4[r] = tile4 + NQ * cell0 + ((q + cell0 + r) & (NQ - 1));
  t1 += cell0 * NQ + q;
  float2 w1[NP][W], wj[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
#pragma unroll
    for (int i = 0; i < W; i += 2) {
      const float4 x = *reinterpret_cast<const float4 *>(slot[p] + 16 + 2 * i);
      w1[p][i] = make_float2(x.x, x.y);
      if (i + 1 < W) w1[p][i + 1] = make_float2(x.z, x.w);
    }
    const int j = c - o2[p];
    const float w = j >= 0 && j < W ? slot[p][32 + 2 * j] : 0.0f;  // columns outside the window are not read below
    wj[p] = make_float2(w, w);
  }
  float2 a01[NP], a23[NP];
  float a4[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    a01[p] = a23[p] = make_float2(0.f, 0.f);
    a4[p] = 0.0f;
  }
#pragma unroll
  for (int i0 = 0; i0 < W; ++i0) {
    float2 p01[NP], p23[NP];
    float p4[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      p01[p] = p23[p] = make_float2(0.f, 0.f);
      p4[p] = 0.0f;
    }
#pragma unroll
    for (int i1 = 0; i1 < W; ++i1) {
      constexpr int kT = T;
      const int row = (i0 * kT + i1) * kT;
      const float4 v = t4[row & (NQ - 1)][row * NQ];
      float v4 = 0.0f;
      if constexpr (F == 5) v4 = t1[row * NQ];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        p01[p] = __ffma2_rn(w1[p][i1], make_float2(v.x, v.y), p01[p]);
        p23[p] = __ffma2_rn(w1[p][i1], make_float2(v.z, v.w), p23[p]);
        if constexpr (F == 5) p4[p] = fmaf(w1[p][i1].x, v4, p4[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float2 w0 = __fmul2_rn(*reinterpret_cast<const float2 *>(slot[p] + 2 * i0), wj[p]);
      a01[p] = __ffma2_rn(w0, p01[p], a01[p]);
      a23[p] = __ffma2_rn(w0, p23[p], a23[p]);
      if constexpr (F == 5) a4[p] = fmaf(w0.x, p4[p], a4[p]);
    }
  }
  // first level of the sum over the window's columns j: j + ceil(W / 2) onto j
  constexpr int HC = (W + 1) / 2;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float4 t;
    t.x = __shfl_down_sync(0xffffffffu, a01[p].x, HC * NQ);
    t.y = __shfl_down_sync(0xffffffffu, a01[p].y, HC * NQ);
    t.z = __shfl_down_sync(0xffffffffu, a23[p].x, HC * NQ);
    t.w = __shfl_down_sync(0xffffffffu, a23[p].y, HC * NQ);
    float t4 = 0.0f;
    if constexpr (F == 5) t4 = __shfl_down_sync(0xffffffffu, a4[p], HC * NQ);
    const int j = c - o2[p];
    if (j >= 0 && j < HC) {
      const bool two = j + HC < W;
      float4 s = make_float4(a01[p].x, a01[p].y, a23[p].x, a23[p].y);
      if (two) s = make_float4(s.x + t.x, s.y + t.y, s.z + t.z, s.w + t.w);
      *reinterpret_cast<float4 *>(red4 + (p * HC + j) * NQ * 4) = s;
      if constexpr (F == 5) red1[(p * HC + j) * NQ] = two ? a4[p] + t4 : a4[p];
    }
  }
}

template <int W, int F, int NQ, bool HALF>
__global__ void __launch_bounds__(kGroupWarps * 32) interp_group_kernel(const InterpParams a) {
  constexpr int KT = COV3D_KERNEL_ES;
  using S = GroupShape<W, F, NQ>;
  using G = TileGroups<W>;
  constexpr int T = S::T, NK = S::NK, UG = S::UG, P = kUnitPts;
  extern __shared__ float4 tile4[];
  float4 *t4 = tile4;                                            // [cell][part]: four floats
  float *t1 = reinterpret_cast<float *>(t4 + T * T * T * NQ);    // [cell][part]: the fifth
  SortedPoint *s_sp = reinterpret_cast<SortedPoint *>(t1 + S::N1);
  int *s_unit = reinterpret_cast<int *>(s_sp + kGroupChunk);     // first point | count << 10 | cell << 12
  float *s_w = reinterpret_cast<float *>(s_unit + kGroupChunk);  // weights, per warp
  float *s_red = s_w + kGroupWarps * UG * P * kSlot;             // column sums, per warp
  float *s_sc = s_red + kGroupWarps * ((S::RED * F + 3) / 4 * 4);
  float *s_scm = s_sc + kGroupChunk;
  int *s_cnt = reinterpret_cast<int *>(HALF ? s_scm + kGroupChunk : s_scm), *s_off = s_cnt + NK;  // NK + 1
  unsigned char *s_o2 = reinterpret_cast<unsigned char *>(s_off + NK + 2);  // window's first of the group's columns
  __shared__ long long s_rowoff[T * T];
  __shared__ int s_coloff[T];
  __shared__ int s_nunits;
  const int sub = blockIdx.x;
  if (sub >= *a.nsub) return;
  const int bin = a.sub_bin[sub];
  const int first = a.sub_first[sub];
  if (first != a.bin_off[bin]) return;  // one block per bin
  const int last = a.bin_off[bin + 1];
  const int nb12 = a.bins.nb[1] * a.bins.nb[2];
  const int ts0 = (bin / nb12) * kBin;
  const int ts1 = ((bin / a.bins.nb[2]) % a.bins.nb[1]) * kBin;
  const int ts2 = (bin % a.bins.nb[2]) * kBin;
  const int n = a.g.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  for (int e = tid; e < T * T; e += blockDim.x) {
    const int c0 = e / T, c1 = e - (e / T) * T;
    const int m0 = wrap1(wrap1(ts0 + c0, n) + a.shift, n), m1 = wrap1(wrap1(ts1 + c1, n) + a.shift, n);
    s_rowoff[e] = ((int64_t)m0 * n + m1) * n * a.cs;
  }
  for (int e = tid; e < T; e += blockDim.x) s_coloff[e] = wrap1(wrap1(ts2 + e, n) + a.shift, n);
  __syncthreads();
  // the tile, by asynchronous copies (zeros past the pass's channels): a warp copies RPW tile rows
  // (channel, plane, row) at a time
  {
    constexpr int RPW = 32 / T;
    const float2 *gbase = a.grid + (int64_t)a.ch0 * a.chs;
    const int s = lane / T, c2 = lane - (lane / T) * T;
    if (s < RPW) {
      const float2 *src0 = gbase + (int64_t)s_coloff[c2] * a.cs;
      const unsigned d4 = (unsigned)__cvta_generic_to_shared(t4), d1 = (unsigned)__cvta_generic_to_shared(t1);
      for (int row = warp * RPW + s; row < S::CH * T * T; row += kGroupWarps * RPW) {
        const int ch = row / (T * T), rowi = row - ch * (T * T);
        const int cell = rowi * T + c2;
        unsigned dst;
        if constexpr (F == 5) {
          const int h = ch / 5, cc = ch - h * 5;
          dst = cc == 2 ? d1 + (unsigned)((cell * NQ + 2 * h) * 4)
                        : d4 + (unsigned)(part_slot<NQ>(cell, 2 * h + (cc > 2)) * 16 + (cc > 2 ? cc - 3 : cc) * 8);
        } else {
          dst = d4 + (unsigned)(part_slot<NQ>(cell, ch / 2) * 16 + (ch & 1) * 8);
        }
        const bool ok = ch < a.nch;
        const float2 *src = ok ? src0 + s_rowoff[rowi] + (int64_t)ch * a.chs : gbase;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }

  auto corner = [&](float t, int ts) { return wrap1(record_cell<KT, W, HALF>(t, a.g.frac), n) - ts; };
  const int ug = lane / (8 * NQ), c = (lane / NQ) & 7, q = lane % NQ;
  float *const my_w = s_w + warp * UG * P * kSlot;
  float *const my_red4 = s_red + warp * ((S::RED * F + 3) / 4 * 4), *const my_red1 = my_red4 + S::RED * 4;
  // this lane's part in the two steps between units, fixed for the block: the weights it computes
  // (round r: tap wtap of axis d of point wk of unit lane group wsrc) and the column sum it takes
  // (channel of point sk; lanes past them sk = P)
  constexpr int WR = (UG * P * 3 * W + 31) / 32;
  int wk[WR], wsrc[WR], wfrom[WR], wtap[WR], wto[WR];
#pragma unroll
  for (int r = 0; r < WR; ++r) {
    const int e = lane + 32 * r, pt = e / (3 * W), d = (e - pt * 3 * W) / W, tap = e - pt * 3 * W - d * W;
    wk[r] = pt < UG * P ? pt % P : P;
    wsrc[r] = (pt / P) % UG * 8 * NQ;
    wfrom[r] = (pt % P) * 4 + d;
    wtap[r] = tap;
    wto[r] = pt * kSlot + d * 16 + 2 * tap;
  }
  static_assert(UG * P * S::CH <= 32, "one lane per point and channel");
  const int spt = lane / S::CH, sch = lane - spt * S::CH;
  const int sk = spt < UG * P && sch < a.nch ? spt % P : P, ssrc = (spt / P) % UG * 8 * NQ;
  const bool fifth = F == 5 && sch % 5 == 2;
  const int spart = F == 5 ? 2 * (sch / 5) + (sch % 5 > 2) : sch / 2;
  const int spos = F == 5 ? (sch % 5 > 2 ? sch % 5 - 3 : sch % 5) : sch & 1;
  const int sstep = fifth ? NQ : 4 * NQ;
  const float *const sfrom = fifth ? my_red1 + spt * S::HC * NQ + 2 * (sch / 5)
                                   : my_red4 + (spt * S::HC * NQ + spart) * 4 + 2 * spos;
  float2 *const sout = a.out + (int64_t)(a.ch0 + sch) * a.ocs;
  constexpr int PPT = (kGroupChunk + kGroupWarps * 32 - 1) / (kGroupWarps * 32);  // points per thread

  for (int base = first; base < last; base += kGroupChunk) {
    const int cnt = min(kGroupChunk, last - base);
    for (int e = tid; e < NK; e += blockDim.x) s_cnt[e] = 0;
    __syncthreads();  // also: every warp is done with the previous chunk
    SortedPoint sp[PPT];
    int key[PPT];
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
      const int k = tid + u * kGroupWarps * 32;
      key[u] = -1;
      if (k < cnt) {
        sp[u] = a.pts[base + k];
        const int b = (corner(sp[u].t2, ts2) / G::GS) * 64 + corner(sp[u].t1, ts1) * 8 + corner(sp[u].t0, ts0);
        key[u] = b | (atomicAdd(s_cnt + b, 1) << 9);
      }
    }
    __syncthreads();
    if (warp == 0) {  // exclusive scan of the buckets' point counts; units into the table on the way
      int v[NK / 32], sum = 0, units = 0;
#pragma unroll
      for (int u = 0; u < NK / 32; ++u) {
        v[u] = s_cnt[lane * (NK / 32) + u];
        sum += v[u];
        units += (v[u] + P - 1) / P;
      }
      int ip = sum, iu = units;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, ip, o), y = __shfl_up_sync(0xffffffffu, iu, o);
        if (lane >= o) {
          ip += x;
          iu += y;
        }
      }
      int bp = ip - sum, bu = iu - units;
#pragma unroll
      for (int u = 0; u < NK / 32; ++u) {
        s_off[lane * (NK / 32) + u] = bp;
        const int b = lane * (NK / 32) + u;
        const int cell = (((b & 7) * T + ((b >> 3) & 7)) * T + G::base(b >> 6)) << 12;
        for (int k = 0; k < v[u]; k += P) s_unit[bu++] = (bp + k) | (min(P, v[u] - k) << 10) | cell;
        bp += v[u];
      }
      if (lane == 31) s_nunits = iu;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
      if (key[u] < 0) continue;
      const int slot = s_off[key[u] & 511] + (key[u] >> 9);
      s_sp[slot] = sp[u];
      s_o2[slot] = (unsigned char)(corner(sp[u].t2, ts2) - G::base((key[u] & 511) >> 6));
      const int id = sp_id<HALF>(sp[u].idf);
      const float sc = (a.nyquist && sp_nyquist(sp[u].idf)) ? 0.0f : a.scale;
      s_sc[slot] = sc * ctf_factor(a.ctf, a.ctfc, a.g, id);
      if (sp_pair<HALF>(sp[u].idf)) s_scm[slot] = a.scale * ctf_factor(a.ctf, a.ctfc, a.g, mirror_id(a.g, id));
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    const int nunits = s_nunits;
    for (int u0 = warp * UG; u0 < nunits; u0 += kGroupWarps * UG) {
      const bool live = u0 + ug < nunits;
      const int unit = s_unit[live ? u0 + ug : u0];
      const int slot0 = unit & 1023, np = live ? (unit >> 10) & 3 : 0, cell0 = (unit >> 12) + c;
      // the points' weights, one per lane and round
#pragma unroll
      for (int r = 0; r < WR; ++r) {
        const int ur = UG == 1 ? unit : __shfl_sync(0xffffffffu, unit, wsrc[r]);
        const int nr = UG == 1 ? np : __shfl_sync(0xffffffffu, np, wsrc[r]);
        if (wk[r] < nr) {
          const float t = reinterpret_cast<const float *>(s_sp + (ur & 1023))[wfrom[r]];
          const float w = record_weight<KT, W, HALF>(t, record_cell<KT, W, HALF>(t, a.g.frac), wtap[r], a.g.frac, a.k.beta);
          *reinterpret_cast<float2 *>(my_w + wto[r]) = make_float2(w, w);
        }
      }
      const int npmax = UG == 1 ? np : __reduce_max_sync(0xffffffffu, np);
      int o2[P];
      const float *slot[P];
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int k = p < np ? p : 0;  // past the unit's points (and for idle units): computed, not written
        o2[p] = s_o2[slot0 + k];
        slot[p] = my_w + ((np ? ug : 0) * P + k) * kSlot;
      }
      __syncwarp();
      float *r4 = my_red4 + (ug * P * S::HC * NQ + q) * 4, *r1 = my_red1 + ug * P * S::HC * NQ + q;
      if (npmax == 3) unit_sums<W, F, NQ, 3>(t4, t1, cell0, q, slot, o2, c, r4, r1);
      else if (npmax == 2) unit_sums<W, F, NQ, 2>(t4, t1, cell0, q, slot, o2, c, r4, r1);
      else unit_sums<W, F, NQ, 1>(t4, t1, cell0, q, slot, o2, c, r4, r1);
      const int us = UG == 1 ? unit : __shfl_sync(0xffffffffu, unit, ssrc);
      const int ns = UG == 1 ? np : __shfl_sync(0xffffffffu, np, ssrc);
      __syncwarp();
      // the W columns of each point and channel, and the epilogue: Nyquist zeroing, CTF, 1/L
      if (sk < ns) {
        const int sl = (us & 1023) + sk;
        float2 x[S::HC];
#pragma unroll
        for (int j = 0; j < S::HC; ++j) x[j] = *reinterpret_cast<const float2 *>(sfrom + j * sstep);
#pragma unroll
        for (int lvl = 0; lvl < 2; ++lvl) {
          const int wc = lvl == 0 ? S::HC : (S::HC + 1) / 2;
          if (wc <= 1) break;
          const int hh = (wc + 1) / 2;
#pragma unroll
          for (int j = 0; j < S::HC; ++j)
            if (j + hh < wc) x[j] = __fadd2_rn(x[j], x[j + hh]);
        }
        const unsigned idf = s_sp[sl].idf;
        const int id = sp_id<HALF>(idf);
        const float sc = s_sc[sl];
        sout[(int64_t)id * a.ops] = make_float2(x[0].x * sc, x[0].y * (sp_conj<HALF>(idf) ? -sc : sc));
        if (sp_pair<HALF>(idf)) {  // the mirror pixel's values are the conjugates
          const float sm = s_scm[sl];
          sout[(int64_t)mirror_id(a.g, id) * a.ops] = make_float2(x[0].x * sm, x[0].y * -sm);
        }
      }
      __syncwarp();  // the weights and sums are overwritten next
    }
  }
}

// Points whose window lies entirely outside the grid (zero padding) get zero outputs.
__global__ void interp_dead_kernel(const SortedPoint *__restrict__ pts, const int *__restrict__ off, int64_t nbins,
                                   int nchan, float2 *__restrict__ out, int64_t ops, int64_t ocs, bool half) {
  const int lo = off[nbins], hi = off[nbins + 1];
  for (int k = lo + blockIdx.x * blockDim.x + threadIdx.x; k < hi; k += gridDim.x * blockDim.x) {
    const int64_t id = half ? sp_id<true>(pts[k].idf) : sp_id<false>(pts[k].idf);
    for (int c = 0; c < nchan; ++c) out[id * ops + c * ocs] = make_float2(0.f, 0.f);
  }
}

template <int KT, int W, int CP, bool HALF>
int launch_half(const InterpParams &a, int64_t max_blocks, cudaStream_t st) {
  constexpr int T = kBin + W - 1;
  const size_t smem =
      (size_t)T * T * T * CP * sizeof(float4) + (size_t)kInterpChunk * (sizeof(SortedPoint) + (HALF ? 8 : 4));
  if (smem > 32 * 1024) {  // static shared arrays come on top of the dynamic size
    cudaError_t e = cudaFuncSetAttribute(interp_kernel<KT, W, CP, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(interp_kernel)");
  }
  interp_kernel<KT, W, CP, HALF><<<(unsigned)max_blocks, InterpWarps<W, CP>::value * 32, smem, st>>>(a);
  return launched("interp_kernel");
}

template <int KT, int W, int CP>
int launch_cp(const InterpParams &a, int64_t max_blocks, cudaStream_t st) {
  if constexpr (KT != COV3D_KERNEL_NEAREST) {
    if (a.half) return launch_half<KT, W, CP, true>(a, max_blocks, st);
  }
  return launch_half<KT, W, CP, false>(a, max_blocks, st);
}

template <int W, int F, int NQ, bool HALF>
int launch_group(const InterpParams &a, int64_t max_blocks, cudaStream_t st) {
  const size_t smem = GroupShape<W, F, NQ>::bytes(HALF);
  static_assert(GroupShape<W, F, NQ>::bytes(HALF) <= 224 * 1024, "tile and chunk fit in shared memory");
  cudaError_t e = cudaFuncSetAttribute(interp_group_kernel<W, F, NQ, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(interp_group_kernel)");
  interp_group_kernel<W, F, NQ, HALF><<<(unsigned)max_blocks, kGroupWarps * 32, smem, st>>>(a);
  return launched("interp_group_kernel");
}

// One channel pass of interp_group_kernel in the layout that holds the `left` channels (ten, or five at
// W = 7, whose tile of ten does not fit, then four or two), or 0 channels where interp_kernel is the
// faster one: sharing a tile load between points needs points, and the more channels a pass has, the
// better interp_kernel's own lanes are filled (the figures stand at the kernel).
template <int W, bool HALF>
int group_pass(InterpParams a, int left, int64_t max_blocks, cudaStream_t st, int *ch) {
  const float d = a.density;
  *ch = 0;
  if (W <= 6 && left > 5) {
    if (d < (W == 6 ? 0.75f : 0.5f)) return COV3D_OK;
    *ch = a.nch = min(left, 10);
    if constexpr (W <= 6) return launch_group<W, 5, 4, HALF>(a, max_blocks, st);
  }
  if (left > 2) {
    // W = 7: up to eight channels are one pass of interp_kernel and two of this one
    if (d < (left > 5 && left <= 8 ? 1.0f : 0.2f)) return COV3D_OK;
    *ch = a.nch = min(left, 5);
    return left > 4 ? launch_group<W, 5, 2, HALF>(a, max_blocks, st) : launch_group<W, 4, 2, HALF>(a, max_blocks, st);
  }
  if (d < 0.1f) return COV3D_OK;
  *ch = a.nch = left;
  return launch_group<W, 4, 1, HALF>(a, max_blocks, st);
}

// Channel passes of at most 2*InterpCP<W> channels; a short last pass uses a smaller tile.
template <int KT, int W>
int launch_w(InterpParams a, int nchan, int64_t max_blocks, cudaStream_t st) {
  constexpr int CPMAX = InterpCP<W>::value;
  int done = 0;
  while (done < nchan) {
    const int left = nchan - done;
    a.ch0 = done;
    int s = COV3D_OK, ch = 0;
    if constexpr (KT == COV3D_KERNEL_ES && W <= 7) {
      s = a.half ? group_pass<W, true>(a, left, max_blocks, st, &ch) : group_pass<W, false>(a, left, max_blocks, st, &ch);
      if (s != COV3D_OK) return s;
      done += ch;
      if (ch > 0) continue;
    }
    if (left >= 2 * CPMAX) {
      ch = 2 * CPMAX;
      a.nch = ch;
      s = launch_cp<KT, W, CPMAX>(a, max_blocks, st);
    } else {
      ch = left;
      a.nch = ch;
      if constexpr (W <= 2) {
        // narrow windows: the smallest tile that holds the pass, with several points per warp
        const int need = (left + 1) / 2;
        if (need <= 3) s = launch_cp<KT, W, 3>(a, max_blocks, st);
        else if (need <= 4) s = launch_cp<KT, W, 4>(a, max_blocks, st);
        else if (need <= 5) s = launch_cp<KT, W, 5>(a, max_blocks, st);
        else if (need <= 8) s = launch_cp<KT, W, 8>(a, max_blocks, st);
        else s = launch_cp<KT, W, CPMAX>(a, max_blocks, st);
      } else {
        // up to 2*CPMAX - 1 channels in the full-size tile; 3-4 and 1-2 channels in smaller ones
        if (left > 4) s = launch_cp<KT, W, CPMAX>(a, max_blocks, st);
        else if (left > 2) s = launch_cp<KT, W, (CPMAX > 2 ? 2 : CPMAX)>(a, max_blocks, st);
        else s = launch_cp<KT, W, 1>(a, max_blocks, st);
      }
    }
    if (s != COV3D_OK) return s;
    done += ch;
  }
  return COV3D_OK;
}

}  // namespace

int launch_interp(cov3d_plan *p, const GridArgs &ga, int nchan, void *out, int64_t out_ps, int64_t out_cs,
                  const EpilogueArgs &e, SortMode mode) {
  if (p->point_kind == kPointsNone || p->n_points == 0) {
    set_error("no points set");
    return COV3D_ESTATE;
  }
  COV3D_TRY(need_sorted(p, 1u << mode));
  const SortSet &ss = p->sets[mode];
  InterpParams a{};
  a.g = make_geom(p);
  a.k = make_kernel(p);
  a.bins = p->bins;
  a.pts = ss.sorted;
  a.sub_bin = ss.sub_bin;
  a.sub_first = ss.sub_first;
  a.bin_off = ss.bin_off;
  a.nsub = ss.nsub;
  a.grid = static_cast<const float2 *>(ga.grid);
  a.cs = ga.cell_stride;
  a.chs = ga.chan_stride;
  a.shift = ga.shift;
  a.out = static_cast<float2 *>(out);
  a.ops = out_ps;
  a.ocs = out_cs;
  a.ctf = e.ctf;
  a.ctfc = e.ctfc;
  a.nyquist = e.nyquist;
  a.scale = e.scale;
  a.half = mode == kSortHalf;
  a.density = (float)((double)p->n_points / ((double)p->n * p->n * p->n));
  const int64_t mb = p->bins.nbins + p->n_points / p->max_sub + 1;
  if (p->kernel != COV3D_KERNEL_ES) {
    interp_dead_kernel<<<64, 256, 0, p->stream>>>(a.pts, ss.bin_off, p->bins.nbins, nchan, a.out, out_ps,
                                                  out_cs, a.half != 0);
    COV3D_LAUNCHED("interp_dead_kernel");
  }
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST: return launch_w<COV3D_KERNEL_NEAREST, 1>(a, nchan, mb, p->stream);
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

}  // namespace cov3d
