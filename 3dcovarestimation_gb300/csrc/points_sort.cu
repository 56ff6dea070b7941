// Spatial binning of nonuniform points (counting sort by the first cell of each point's
// kernel window) and the subproblem table used by the spreading kernel.
//
// The reference hands unsorted points to cuFINUFFT with gpu_sort=0 (nufft_plan.py:297) or to
// grid_sample; here every point set is sorted once per setpts/setrot so that interpolation
// reads the grid with spatial locality and spreading can accumulate per-bin tiles in shared
// memory.
#include "cov3d_device.cuh"

namespace cov3d {

namespace {

// The views being sorted by one launch sequence (blockIdx.y).
struct SortView {
  int half;
  int *count, *off, *sub_off, *nsub;
  int *pt_bin, *pt_rank;
  SortedPoint *sorted;
  int *sub_bin, *sub_first, *sub_count;
};
struct SortViews {
  SortView v[kSortModes];
};

// Bin holding the window corner c0 (dead: outside the grid or without an index).
template <int KT, int W>
__device__ __forceinline__ int corner_bin(const PointGeom &g, const Bins &bins, int (&c0)[3], bool dead) {
  int b[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (KT == COV3D_KERNEL_ES) {
      c0[d] = pmod(c0[d], g.n);
    } else {
      if (c0[d] + W - 1 < 0 || c0[d] > g.n - 1) dead = true;
      c0[d] = min(max(c0[d], 0), g.n - 1);
    }
    b[d] = c0[d] / bins.bs[d];
  }
  return dead ? (int)bins.nbins : (b[0] * bins.nb[1] + b[1]) * bins.nb[2] + b[2];
}

template <int KT, int W>
__device__ __forceinline__ int bin_of(const PointGeom &g, const Bins &bins, const float *t) {
  int c0[3];
  bool dead = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c0[d] = first_cell<KT, W>(t[d]);
    if (!(t[d] == t[d])) {  // NaN coordinate: no contribution
      dead = true;
      c0[d] = 0;
    }
  }
  return corner_bin<KT, W>(g, bins, c0, dead);
}

template <int KT, int W>
__device__ __forceinline__ int bin_of_fix(const PointGeom &g, const Bins &bins, const int *t) {
  int c0[3];
  bool dead = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    dead = dead || t[d] == kDeadIndex;
    c0[d] = t[d] == kDeadIndex ? 0 : first_cell_fix<KT, W>(t[d], g.frac);
  }
  return corner_bin<KT, W>(g, bins, c0, dead);
}

// Bin of every point (dead points, whose window misses the grid, go to bin nbins) and its
// rank in the bin.  The lanes of a warp that share a bin (neighbouring pixels mostly do) take
// their ranks from one atomic on the bin's counter, in lane order.
template <int KT, int W>
__device__ __forceinline__ void count_full(const PointGeom &g, const Bins &bins, int64_t M, const SortView &v) {
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = id < M;
  int bin = -1;
  if (valid) {
    float t[3];
    point_index(g, (int)id, t);
    bin = bin_of<KT, W>(g, bins, t);
  }
  const unsigned grp = __match_any_sync(0xffffffffu, bin);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(grp) - 1;
  int base = 0;
  if (valid && lane == leader) base = atomicAdd(v.count + bin, __popc(grp));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (!valid) return;
  v.pt_bin[id] = bin;
  v.pt_rank[id] = base + __popc(grp & ((1u << lane) - 1u));
}

// kSortHalf.  Pixels p and p' = mirror_pixel(p) of an image sample k and -k, where the transform
// of a real volume holds conjugate values, so one record serves both when their indices mirror
// each other about the grid's centre: exactly for points made from rotations, to within
// 1.5e-7 n cells for explicit ones (the float rounding of two wrapped angles; any other pair of
// points gets a record each).  The record holds the mean of the one index and the mirrored other,
// in the half space t0 >= n / 2; its id is the pixel there.  Grid-sample kernels need both windows
// inside the grid as well (zero padding does not mirror: cell 0 is stored, cell n is not).
// Periodic kernels also fold single points into the half space (kConjBit).
struct HalfRecord {
  int t[3];
  unsigned flags;  // kPairBit / kConjBit
  bool swap;       // the pair's id is the mirror pixel
};

__device__ __forceinline__ void fold_single(const PointGeom &g, bool periodic, HalfRecord &r) {
  const int c = (g.n / 2) << g.frac;
  r.flags = 0;
  r.swap = false;
  if (periodic && r.t[0] < c && r.t[0] != kDeadIndex && r.t[1] != kDeadIndex && r.t[2] != kDeadIndex) {
    r.flags = kConjBit;
#pragma unroll
    for (int d = 0; d < 3; ++d) r.t[d] = 2 * c - r.t[d];
  }
}

// The record of the pair of pixels with ids `first` < `second`, the first at index ta; false, with the
// second's index in tb, when the two do not mirror each other.
template <int KT>
__device__ __forceinline__ bool pair_record(const PointGeom &g, const int (&ta)[3], int second, int (&tb)[3],
                                            HalfRecord &r) {
  const int c = (g.n / 2) << g.frac, N = g.n << g.frac, tol = 2 + (int)(1.5e-7f * (float)N);
  bool ok = true;
  if (g.kind == kPointsRotations) {  // the second's is the mirrored first, up to a tie's rounding
#pragma unroll
    for (int d = 0; d < 3; ++d) tb[d] = ta[d] == kDeadIndex ? kDeadIndex : 2 * c - ta[d];
  } else {
    point_index_fix<KT>(g, second, tb);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ok = ok && ta[d] != kDeadIndex && tb[d] != kDeadIndex;
    const int a = ta[d] - c;
    long long s = (long long)a + (tb[d] - c);
    if (KT == COV3D_KERNEL_ES) s = s > N / 2 ? s - N : (s < -(N / 2) ? s + N : s);
    ok = ok && s <= tol && s >= -tol;
    r.t[d] = a - (int)(s >> 1);
  }
  if (!ok) return false;
  r.flags = kPairBit;
  r.swap = r.t[0] < 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) r.t[d] = (r.swap ? -r.t[d] : r.t[d]) + c;
  if (KT != COV3D_KERNEL_ES) {
    const int lo = max(0, 2 * (g.n / 2) - g.n + 1), hi = min(g.n - 1, 2 * (g.n / 2));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int f = first_cell_fix<KT, 2>(r.t[d], g.frac);
      ok = ok && f >= lo && f + 1 <= hi;
    }
  }
  return ok;
}

// count_full for kSortHalf: the thread of the first pixel of a mirror pair decides for both
// (pt_bin -1: no record under that id); the threads of second pixels only keep their warp company.
template <int KT, int W>
__device__ __forceinline__ void count_half(const PointGeom &g, const Bins &bins, int64_t M, const SortView &v) {
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int bin = -1;
  int64_t rec = id;
  if (id < M) {
    const int p = (unsigned)id % (unsigned)g.P, m = mirror_pixel(p, g.Lp);
    if (m < 0 || m >= p) {
      HalfRecord a;
      point_index_fix<KT>(g, (int)id, a.t);
      bool pair = false;
      if (m > p) {
        const int64_t other = id + (m - p);
        HalfRecord b, r;
        pair = pair_record<KT>(g, a.t, (int)other, b.t, r);
        if (pair) {
          rec = r.swap ? other : id;
          v.pt_bin[r.swap ? id : other] = -1;
          a = r;
        } else {
          fold_single(g, KT == COV3D_KERNEL_ES, b);
          const int ob = bin_of_fix<KT, W>(g, bins, b.t);
          v.pt_bin[other] = ob;
          v.pt_rank[other] = atomicAdd(v.count + ob, 1);
        }
      }
      if (!pair) fold_single(g, KT == COV3D_KERNEL_ES, a);
      bin = bin_of_fix<KT, W>(g, bins, a.t);
    }
  }
  const unsigned grp = __match_any_sync(0xffffffffu, bin);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(grp) - 1;
  int base = 0;
  if (bin >= 0 && lane == leader) base = atomicAdd(v.count + bin, __popc(grp));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (bin < 0) return;
  v.pt_bin[rec] = bin;
  v.pt_rank[rec] = base + __popc(grp & ((1u << lane) - 1u));
}

template <int KT, int W>
__global__ void bin_count_kernel(PointGeom g, Bins bins, int64_t M, SortViews views) {
  const SortView &v = views.v[blockIdx.y];
  if constexpr (KT != COV3D_KERNEL_NEAREST) {
    if (v.half) return count_half<KT, W>(g, bins, M, v);
  }
  count_full<KT, W>(g, bins, M, v);
}

template <int KT>
__device__ __forceinline__ void scatter_half(const PointGeom &g, int64_t M, const SortView &v) {
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= M) return;
  const int bin = v.pt_bin[id];
  if (bin < 0) return;
  const int pos = v.off[bin] + v.pt_rank[id];
  const int p = (unsigned)id % (unsigned)g.P, m = mirror_pixel(p, g.Lp);
  HalfRecord a;
  const bool second = m >= 0 && m < p;
  point_index_fix<KT>(g, (int)id + (second ? m - p : 0), a.t);
  bool pair = false;
  if (m >= 0 && m != p) {
    HalfRecord b, r;
    pair = pair_record<KT>(g, a.t, (int)id + (second ? 0 : m - p), b.t, r);
    if (pair) a = r;
    else if (second) a = b;
  }
  if (!pair) fold_single(g, KT == COV3D_KERNEL_ES, a);
  SortedPoint sp;
  sp.t0 = __int_as_float(a.t[0]);
  sp.t1 = __int_as_float(a.t[1]);
  sp.t2 = __int_as_float(a.t[2]);
  sp.idf = (unsigned)id | a.flags | (on_nyquist(g, (int)id) ? kNyquistBit : 0u);
  v.sorted[pos] = sp;
}

// Exclusive scans over a view's bin counts, one block per view: point offsets, and subproblem
// offsets (ceil(count / max_sub) subproblems per live bin).  A chain of passes bounds it, so a pass
// takes eight bins per thread, in 16-byte loads and stores, and the next pass's loads are in flight
// meanwhile (32768 bins, 1024 images of 128^2: 53 us with contiguous chunks per thread, loaded 128
// bytes apart, 32 with four bins and scalar stores, now 22).
constexpr int kScanBins = 8;

__global__ void __launch_bounds__(1024) bin_scan_kernel(int64_t nbins, int max_sub, SortViews views) {
  const SortView &v = views.v[blockIdx.x];
  __shared__ int s_pts[32], s_sub[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t total = nbins + 1;  // includes the dead bin
  int carry_p = 0, carry_s = 0;
  int next[kScanBins];
  auto load = [&](int64_t i0) {
    if (i0 + kScanBins <= total) {
#pragma unroll
      for (int u = 0; u < kScanBins; u += 4) {
        const int4 x = *reinterpret_cast<const int4 *>(v.count + i0 + u);
        next[u] = x.x; next[u + 1] = x.y; next[u + 2] = x.z; next[u + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kScanBins; ++k) next[k] = i0 + k < total ? v.count[i0 + k] : 0;
    }
  };
  load((int64_t)kScanBins * tid);
  for (int64_t base = 0; base < total; base += kScanBins * 1024) {
    const int64_t i0 = base + kScanBins * tid;
    int c[kScanBins], sp = 0, ss = 0, sub[kScanBins];
#pragma unroll
    for (int k = 0; k < kScanBins; ++k) c[k] = next[k];
    if (base + kScanBins * 1024 < total) load(i0 + kScanBins * 1024);
#pragma unroll
    for (int k = 0; k < kScanBins; ++k) {
      sub[k] = i0 + k < nbins ? (c[k] + max_sub - 1) / max_sub : 0;
      sp += c[k];
      ss += sub[k];
    }
    int ip = sp, is = ss;  // inclusive within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ip, o), b = __shfl_up_sync(0xffffffffu, is, o);
      if (lane >= o) {
        ip += a;
        is += b;
      }
    }
    __syncthreads();  // the previous pass has read the warp totals
    if (lane == 31) {
      s_pts[warp] = ip;
      s_sub[warp] = is;
    }
    __syncthreads();
    int wp = s_pts[lane], ws = s_sub[lane];  // every warp scans the 32 warp totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, wp, o), b = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) {
        wp += a;
        ws += b;
      }
    }
    const int before_p = __shfl_sync(0xffffffffu, wp, (warp + 31) & 31), before_s = __shfl_sync(0xffffffffu, ws, (warp + 31) & 31);
    int rp = carry_p + (warp ? before_p : 0) + ip - sp, rs = carry_s + (warp ? before_s : 0) + is - ss;
    int off[kScanBins];
#pragma unroll
    for (int k = 0; k < kScanBins; ++k) {
      off[k] = rp;
      rp += c[k];
      c[k] = rs;  // the subproblem offset
      rs += sub[k];
    }
    if (i0 + kScanBins <= nbins) {
#pragma unroll
      for (int u = 0; u < kScanBins; u += 4) {
        *reinterpret_cast<int4 *>(v.off + i0 + u) = make_int4(off[u], off[u + 1], off[u + 2], off[u + 3]);
        *reinterpret_cast<int4 *>(v.sub_off + i0 + u) = make_int4(c[u], c[u + 1], c[u + 2], c[u + 3]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kScanBins; ++k) {
        if (i0 + k < total) v.off[i0 + k] = off[k];
        if (i0 + k < nbins) v.sub_off[i0 + k] = c[k];
      }
    }
    carry_p += __shfl_sync(0xffffffffu, wp, 31);
    carry_s += __shfl_sync(0xffffffffu, ws, 31);
  }
  if (tid == 0) {
    v.off[total] = carry_p;
    *v.nsub = carry_s;
  }
}

__device__ __forceinline__ void scatter_full(const PointGeom &g, int64_t M, const SortView &v) {
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= M) return;
  const int pos = v.off[v.pt_bin[id]] + v.pt_rank[id];
  float t[3];
  point_index(g, (int)id, t);
  SortedPoint sp;
  sp.t0 = t[0];
  sp.t1 = t[1];
  sp.t2 = t[2];
  sp.idf = (unsigned)id | (on_nyquist(g, (int)id) ? kNyquistBit : 0u);
  v.sorted[pos] = sp;
}

__device__ __forceinline__ void write_subproblems(int64_t b, int64_t nbins, int max_sub, const SortView &v) {
  if (b >= nbins) return;
  const int c = v.count[b];
  const int s0 = v.sub_off[b];
  for (int s = 0; s * max_sub < c; ++s) {
    v.sub_bin[s0 + s] = (int)b;
    v.sub_first[s0 + s] = v.off[b] + s * max_sub;
    v.sub_count[s0 + s] = min(max_sub, c - s * max_sub);
  }
}

// The records in bin order, and in the blocks after the points' the subproblem table.
template <int KT>
__global__ void scatter_kernel(PointGeom g, int64_t M, int64_t nbins, int max_sub, SortViews views) {
  const SortView &v = views.v[blockIdx.y];
  const int64_t pb = (M + blockDim.x - 1) / blockDim.x;
  if (blockIdx.x >= pb) return write_subproblems((blockIdx.x - pb) * blockDim.x + threadIdx.x, nbins, max_sub, v);
  if constexpr (KT != COV3D_KERNEL_NEAREST) {
    if (v.half) return scatter_half<KT>(g, M, v);
  }
  scatter_full(g, M, v);
}

// Before the count: the views' counters to zero and, for new rotations, their index coefficients:
// axis d (row 2 - d of R) moves by coefficient / 2^40 cells per pixel column and row, reduced modulo
// the period n (the indices wrap anyway).
__global__ void sort_begin_kernel(int64_t counters, SortViews views, int nviews, const float *__restrict__ rot,
                                  int64_t n_images, int n, int Lp, long long *__restrict__ rotc) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  for (int m = 0; m < nviews; ++m)
    for (int64_t e = tid; e < counters; e += nt) views.v[m].count[e] = 0;
  if (!rotc) return;
  for (int64_t e = tid; e < n_images * 6; e += nt) {
    const int64_t b = e / 6;
    const int q = (int)(e - b * 6);
    double v = (double)rot[b * 9 + (2 - q / 2) * 3 + (q & 1)] * (double)n / (double)Lp;
    v -= (double)n * rint(v / (double)n);
    rotc[e] = isfinite(v) ? __double2ll_rn(v * (double)(1LL << kRotShift)) : kDeadCoef;
  }
}

template <int KT, int W>
void launch_count(cov3d_plan *p, const PointGeom &g, dim3 grid, const SortViews &views) {
  bin_count_kernel<KT, W><<<grid, 256, 0, p->stream>>>(g, p->bins, p->n_points, views);
}

// Sorts the points into the views of `modes` (bits 1 << SortMode) in one launch sequence.
int sort_points(cov3d_plan *p, unsigned modes) {
  const int64_t M = p->n_points, nb = p->bins.nbins;
  SortViews views{};
  int nv = 0;
  bool half = false;
  for (int m = 0; m < kSortModes; ++m) {
    if (!(modes >> m & 1)) continue;
    COV3D_TRY(reserve_sort(p, M, (SortMode)m));
    SortSet &ss = p->sets[m];
    half = half || m == kSortHalf;
    views.v[nv++] = SortView{m == kSortHalf, ss.bin_count, ss.bin_off, ss.sub_off,
                             ss.nsub, ss.pt_bin, ss.pt_rank, ss.sorted,
                             ss.sub_bin, ss.sub_first, ss.sub_count};
  }
  if (nv == 0) return COV3D_OK;
  long long *rotc = nullptr;
  if (half && p->point_kind == kPointsRotations) {
    COV3D_TRY(grow(p->rotc, p->n_images * 6 * 8));
    rotc = p->rotc.as<long long>();
  }
  const PointGeom g = make_geom(p);
  const int64_t work = nb + 1 > p->n_images * 6 ? nb + 1 : p->n_images * 6;
  sort_begin_kernel<<<(unsigned)((work + 255) / 256 < 608 ? (work + 255) / 256 : 608), 256, 0, p->stream>>>(
      nb + 1, views, nv, p->rot.as<float>(), p->n_images, p->n, p->points_L, rotc);
  COV3D_LAUNCHED("sort_begin_kernel");
  const dim3 blocks((unsigned)((M + 255) / 256), (unsigned)nv);
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST: launch_count<COV3D_KERNEL_NEAREST, 1>(p, g, blocks, views); break;
    case COV3D_KERNEL_LINEAR: launch_count<COV3D_KERNEL_LINEAR, 2>(p, g, blocks, views); break;
    default:
      switch (p->width) {
#define COV3D_W(Wv) \
  case Wv: launch_count<COV3D_KERNEL_ES, Wv>(p, g, blocks, views); break;
        COV3D_W(4) COV3D_W(5) COV3D_W(6) COV3D_W(7) COV3D_W(8)
#undef COV3D_W
        default:
          set_error("unsupported ES width %d", p->width);
          return COV3D_EINVAL;
      }
  }
  COV3D_LAUNCHED("bin_count_kernel");
  bin_scan_kernel<<<nv, 1024, 0, p->stream>>>(nb, p->max_sub, views);
  COV3D_LAUNCHED("bin_scan_kernel");
  const dim3 sblocks(blocks.x + (unsigned)((nb + 255) / 256), (unsigned)nv);
  switch (p->kernel) {
    case COV3D_KERNEL_NEAREST:
      scatter_kernel<COV3D_KERNEL_NEAREST><<<sblocks, 256, 0, p->stream>>>(g, M, nb, p->max_sub, views);
      break;
    case COV3D_KERNEL_LINEAR:
      scatter_kernel<COV3D_KERNEL_LINEAR><<<sblocks, 256, 0, p->stream>>>(g, M, nb, p->max_sub, views);
      break;
    default: scatter_kernel<COV3D_KERNEL_ES><<<sblocks, 256, 0, p->stream>>>(g, M, nb, p->max_sub, views);
  }
  COV3D_LAUNCHED("scatter_kernel");
  for (int m = 0; m < kSortModes; ++m)
    if (modes >> m & 1) p->sets[m].valid = true;
  return COV3D_OK;
}

}  // namespace

// Room for a sort of M points in a view (a no-op when there is enough already).
int reserve_sort(cov3d_plan *p, int64_t M, SortMode mode) {
  SortSet &ss = p->sets[mode];
  if (M <= ss.cap) return COV3D_OK;
  const int64_t nb = p->bins.nbins;
  const int64_t max_subs = nb + M / p->max_sub + 1;
  auto align = [](int64_t bytes) { return (bytes + 255) & ~int64_t(255); };
  const int64_t bins = align((nb + 2) * 4), pts = align(M * 4), subs = align(max_subs * 4);
  ss.cap = -1;
  ss.valid = false;
  COV3D_TRY(grow(ss.mem, 3 * bins + 2 * pts + align(M * (int64_t)sizeof(SortedPoint)) + 3 * subs + 256));
  char *m = ss.mem.as<char>();
  auto take = [&](int64_t bytes) {
    char *q = m;
    m += bytes;
    return q;
  };
  ss.bin_count = reinterpret_cast<int *>(take(bins));
  ss.bin_off = reinterpret_cast<int *>(take(bins));
  ss.sub_off = reinterpret_cast<int *>(take(bins));
  ss.pt_bin = reinterpret_cast<int *>(take(pts));
  ss.pt_rank = reinterpret_cast<int *>(take(pts));
  ss.sorted = reinterpret_cast<SortedPoint *>(take(align(M * (int64_t)sizeof(SortedPoint))));
  ss.sub_bin = reinterpret_cast<int *>(take(subs));
  ss.sub_first = reinterpret_cast<int *>(take(subs));
  ss.sub_count = reinterpret_cast<int *>(take(subs));
  ss.nsub = reinterpret_cast<int *>(take(256));
  ss.cap = M;
  return COV3D_OK;
}

// Pair records need a linear or ES window and ids below 2^29.
static bool pairs_apply(const cov3d_plan *p) {
  return p->kernel != COV3D_KERNEL_NEAREST && p->n_points < (int64_t(1) << 29);
}

// Whether the pairs' view of the current points fits the buffers that it has.
static bool pairs_fit(const cov3d_plan *p) {
  return p->sets[kSortHalf].cap >= p->n_points &&
         (p->point_kind != kPointsRotations || p->rotc.cap >= p->n_images * 6 * 8);
}

static int capturing(const cov3d_plan *p, bool *yes) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  COV3D_CUDA(cudaStreamIsCapturing(p->stream, &cap));
  *yes = cap != cudaStreamCaptureStatusNone;
  return COV3D_OK;
}

SortMode hermitian_mode(const cov3d_plan *p) {
  if (!pairs_apply(p) || p->pairs_off) return kSortFull;
  bool cap = false;
  // a capture cannot allocate the view
  if (!p->sets[kSortHalf].valid && !pairs_fit(p) && (capturing(p, &cap) != COV3D_OK || cap)) return kSortFull;
  return kSortHalf;
}

// The plan's points have changed: the views that operators have used so far are sorted now, on the
// stream that sets the points (so an operator ordered after this call, and a captured one that reads
// the view, find the new points in it); the others on their first use (need_sorted).  Points set
// inside a stream capture reach every view by the replay, also those that nothing has used yet; where
// the pairs' view has no room to be sorted there, the replay would change the points unseen by it, so
// no operator of this plan uses pair records from then on (graphs made before still find theirs).
int new_points(cov3d_plan *p) {
  for (SortSet &ss : p->sets) ss.valid = ss.pending = false;
  const int64_t M = p->n_points;
  if (M <= 0) return COV3D_OK;
  if (M >= (int64_t)(1 << 30)) {
    set_error("too many points (%lld); the limit is 2^30-1 per plan", (long long)M);
    return COV3D_EINVAL;
  }
  bool cap = false;
  COV3D_TRY(capturing(p, &cap));
  if (cap) {
    p->sets[kSortFull].used = true;
    if (!p->sets[kSortFull].mem.ptr) {  // a first allocation is possible here, in the relaxed mode
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      COV3D_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      const int rc = reserve_sort(p, M, kSortFull);
      COV3D_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      COV3D_TRY(rc);
    }
    if (pairs_apply(p)) {
      if (pairs_fit(p)) p->sets[kSortHalf].used = true;
      else p->pairs_off = true;
    }
  }
  unsigned modes = 0;
  for (int m = 0; m < kSortModes; ++m) {
    if (m == kSortHalf && !(pairs_apply(p) && (!p->pairs_off || (p->sets[m].used && pairs_fit(p))))) continue;
    if (p->sets[m].used) modes |= 1u << m;
  }
  COV3D_TRY(sort_points(p, modes));
  if (cap) return COV3D_OK;
  if (!p->points_set) COV3D_CUDA(cudaEventCreateWithFlags(&p->points_set, cudaEventDisableTiming));
  return check_cuda(cudaEventRecord(p->points_set, p->stream), "points event");
}

// A first use outside a capture: the views in `todo` sorted on the caller's stream, after the points.
// Operators of other streams wait for the views' events until they have completed.
static int first_use(cov3d_plan *p, unsigned todo) {
  if (p->points_set) COV3D_CUDA(cudaStreamWaitEvent(p->stream, p->points_set, 0));
  {
    PhaseScope ps(p, kPhaseSort);
    COV3D_TRY(sort_points(p, todo));
  }
  for (int m = 0; m < kSortModes; ++m) {
    if (!(todo >> m & 1)) continue;
    SortSet &ss = p->sets[m];
    ss.valid = false;  // until operators can wait for it
    if (!ss.done) COV3D_CUDA(cudaEventCreateWithFlags(&ss.done, cudaEventDisableTiming));
    COV3D_CUDA(cudaEventRecord(ss.done, p->stream));
    ss.valid = ss.pending = true;
  }
  return COV3D_OK;
}

// A first use inside a capture: sorted on a stream of the plan's own and waited for, so that the sort
// has run and is no part of the graph (as if the view had been sorted when the points were set).  It may
// allocate the view's buffers (in the relaxed mode); it never frees any: a view that nothing has used yet
// has none, or those that cov3d_plan_reserve made.
static int first_use_in_capture(cov3d_plan *p, unsigned todo) {
  if (!p->sort_stream) COV3D_CUDA(cudaStreamCreateWithFlags(&p->sort_stream, cudaStreamNonBlocking));
  if (p->points_set) COV3D_CUDA(cudaStreamWaitEvent(p->sort_stream, p->points_set, 0));
  const cudaStream_t caller = p->stream;
  p->stream = p->sort_stream;
  int rc;
  {
    PhaseScope ps(p, kPhaseSort);
    rc = sort_points(p, todo);
  }
  const int done = check_cuda(cudaStreamSynchronize(p->sort_stream), "sort");
  p->stream = caller;
  return rc != COV3D_OK ? rc : done;
}

// The caller's stream comes after a pending first use of the view; a capture, whose graph may be replayed
// at any time, waits for it here.
static int after_first_use(cov3d_plan *p, SortSet &ss, bool cap) {
  const cudaError_t q = cudaEventQuery(ss.done);
  if (q != cudaSuccess && q != cudaErrorNotReady) return check_cuda(q, "sort event");
  if (q == cudaErrorNotReady) {
    (void)cudaGetLastError();
    if (!cap) return check_cuda(cudaStreamWaitEvent(p->stream, ss.done, 0), "sort event");
    COV3D_CUDA(cudaEventSynchronize(ss.done));
  }
  ss.pending = false;
  return COV3D_OK;
}

// The views in `modes` (bits 1 << SortMode) hold the current points for the caller's stream.
int need_sorted(cov3d_plan *p, unsigned modes) {
  unsigned todo = 0;
  bool wait = false;
  for (int m = 0; m < kSortModes; ++m) {
    if (!(modes >> m & 1)) continue;
    SortSet &ss = p->sets[m];
    ss.used = true;
    if (!ss.valid) todo |= 1u << m;
    else wait = wait || ss.pending;
  }
  if (!todo && !wait) return COV3D_OK;
  bool cap = false;
  COV3D_TRY(capturing(p, &cap));
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // this thread may allocate, ask and wait in a capture
  COV3D_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
  int rc = COV3D_OK;
  for (int m = 0; m < kSortModes && rc == COV3D_OK; ++m)
    if ((modes >> m & 1) && p->sets[m].valid && p->sets[m].pending) rc = after_first_use(p, p->sets[m], cap);
  if (rc == COV3D_OK && todo) {
    rc = cap ? first_use_in_capture(p, todo) : first_use(p, todo);
    if (rc != COV3D_OK)
      for (int m = 0; m < kSortModes; ++m)
        if (todo >> m & 1) p->sets[m].valid = false;
  }
  const int back = check_cuda(cudaThreadExchangeStreamCaptureMode(&mode), "capture mode");
  return rc != COV3D_OK ? rc : back;
}

}  // namespace cov3d
