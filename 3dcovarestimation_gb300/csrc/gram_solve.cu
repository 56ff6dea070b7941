// Per-image r x r contractions of the covariance cost and its hand-written adjoint.
//
// For image b with projections Q_b (P x r, the CTF-weighted central-slice samples of the r
// Fourier-domain eigenvolumes, projection_funcs.py:321-370) and Fourier image y_b:
//   gram_ij = sum_p conj(Q_pi) Q_pj,  h_i = sum_p conj(Q_pi) y_p
// ML objective (raw_cost_maximum_liklihood_fourier_domain, covar_sgd.py:1381-1399, through
// compute_latentMAP_batch, wiener_coords.py:168-203):
//   m = gram / s2 + I,  b = h / s2,  z = m^-1 b,  cost_b = (-Re(b^H z) + logdet m) / 2
//   dcost_b / d conj(Q_pi) = sum_j C_ij Q_pj + u_i y_p,
//   C = (conj(m^-1) + conj(z) z^T) / (2 s2),  u = -conj(z) / (2 s2)
// LS objective (raw_cost_fourier_domain, covar_sgd.py:1320-1347), M = conj(gram), t = conj(h):
//   cost_b = -2 |t|^2 + ||M||_F^2 + 2 s2 tr M,  C = 2 M + 2 s2 I,  u = -2 t
// The r x r factorisations run in FP64 (a few threads per image).
#include "cov3d_device.cuh"

namespace cov3d {

namespace {

constexpr int kMaxRank = 32;
constexpr int kGramChunk = 128;

constexpr int kGramTile = 3;       // products are summed in 3 x 3 register tiles
constexpr int kGramStage = 88000;  // bytes of staged pixels per block: two blocks per SM

// Per-image Gram at any rank and layout: v = (q_0 .. q_{r-1}, y) of a pixel, products conj(v_i) v_j, i <= j.
// One block per image; chunks of kGramChunk pixels are staged in shared memory, nc at a time.  A chunk's
// pixels p = grp, grp + groups, ... make one sum per product, Kahan-added to the totals of that grp over
// the chunks in order, and the totals of the groups are added in order.  The chunk sums are independent:
// a work item is a 3 x 3 tile of products of one chunk and group, which reads 6 staged values for 36 FMAs
// (a thread per product read 2 for 4, and shared memory bound it: r = 20, 300 images of 128^2:
// 1.91 -> 0.43 ms, 0.79 GB; r = 8, 512 of 64^2, channel-major: 172 -> 58 us, 0.13 GB).
__global__ void __launch_bounds__(1024) gram_kernel(const float2 *__restrict__ Q, int64_t q_is, int64_t q_ps,
                                                    int64_t q_cs, const float2 *__restrict__ Y, int P, int r,
                                                    int groups, int nc, int rs, float2 *__restrict__ gram,
                                                    float2 *__restrict__ h, float *__restrict__ yy) {
  constexpr int T = kGramTile;
  extern __shared__ float2 sq[];  // nc chunks of kGramChunk rows of rs values, then nc * groups * J sums
  const int b = blockIdx.x, tid = threadIdx.x;
  const int R1 = r + 1, J = R1 * (R1 + 1) / 2;
  const int nt = (R1 + T - 1) / T, ntile = nt * (nt + 1) / 2;
  const int cstride = kGramChunk * rs + 3;  // (chunks apart in the banks)
  float2 *s_part = sq + nc * cstride;
  const float2 *Qb = Q + (int64_t)b * q_is;
  const float2 *Yb = Y + (int64_t)b * P;
  float2 sum = make_float2(0.f, 0.f), comp = make_float2(0.f, 0.f);
  const bool keeps = tid < groups * J;  // thread grp * J + job holds the totals
  for (int p0 = 0; p0 < P; p0 += nc * kGramChunk) {
    const int np = min(nc * kGramChunk, P - p0);
    auto row = [&](int p) { return sq + (p / kGramChunk) * cstride + (p % kGramChunk) * rs; };
    auto copy = [&](float2 *d, const float2 *s) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(s)
                   : "memory");
    };
    __syncthreads();
    if (q_cs == 1) {
      const int di = blockDim.x % r, dp = blockDim.x / r;
      for (int i = tid % r, p = tid / r; p < np;) {
        copy(row(p) + i, Qb + (int64_t)(p0 + p) * q_ps + i);
        i += di;
        p += dp;
        if (i >= r) {
          i -= r;
          ++p;
        }
      }
    } else {
      for (int i = tid >> 5; i < r; i += blockDim.x >> 5)
        for (int p = tid & 31; p < np; p += 32)
          copy(row(p) + i, Qb + (int64_t)(p0 + p) * q_ps + (int64_t)i * q_cs);
    }
    for (int p = tid; p < np; p += blockDim.x) copy(row(p) + r, Yb + p0 + p);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const int chunks = (np + kGramChunk - 1) / kGramChunk;
    for (int item = tid; item < chunks * groups * ntile; item += blockDim.x) {
      const int tile = item % ntile, cg = item / ntile, grp = cg % groups, c = cg / groups;
      int ti = 0, tj = tile;
      while (tj >= nt - ti) {
        tj -= nt - ti;
        ++ti;
      }
      const int i0 = ti * T, j0 = (ti + tj) * T;
      const int pe = min(kGramChunk, np - c * kGramChunk);
      const float2 *rows = sq + c * cstride;
      float2 part[T][T];
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) part[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int p = grp; p < pe; p += groups) {
        float2 x[T], y[T];
#pragma unroll
        for (int i = 0; i < T; ++i) {
          x[i] = rows[p * rs + i0 + i];
          y[i] = rows[p * rs + j0 + i];
        }
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) {
            part[i][j].x = fmaf(x[i].x, y[j].x, fmaf(x[i].y, y[j].y, part[i][j].x));
            part[i][j].y = fmaf(x[i].x, y[j].y, fmaf(-x[i].y, y[j].x, part[i][j].y));
          }
      }
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) {
          const int vi = i0 + i, vj = j0 + j;
          if (vi <= vj && vj < R1) s_part[cg * J + vi * R1 - vi * (vi - 1) / 2 + vj - vi] = part[i][j];
        }
    }
    __syncthreads();
    if (keeps) {
      for (int c = 0; c < chunks; ++c) {  // Kahan updates of the running totals
        const float2 part = s_part[c * groups * J + tid];
        float yx = part.x - comp.x, tx = sum.x + yx;
        comp.x = (tx - sum.x) - yx;
        sum.x = tx;
        float yyv = part.y - comp.y, ty = sum.y + yyv;
        comp.y = (ty - sum.y) - yyv;
        sum.y = ty;
      }
    }
  }
  __syncthreads();
  // reduce over pixel groups
  if (keeps) s_part[tid] = sum;
  __syncthreads();
  if (tid < J) {
    float2 tot = sum;
    for (int g = 1; g < groups; ++g) {
      tot.x += s_part[g * J + tid].x;
      tot.y += s_part[g * J + tid].y;
    }
    int i = 0, k = tid;
    while (k >= R1 - i) {
      k -= R1 - i;
      ++i;
    }
    const int j = i + k;
    if (j < r) {
      gram[((int64_t)b * r + i) * r + j] = tot;
      if (i != j) gram[((int64_t)b * r + j) * r + i] = make_float2(tot.x, -tot.y);
    } else if (i < r) {
      h[(int64_t)b * r + i] = tot;
    } else {
      yy[b] = tot.x;
    }
  }
}

constexpr int kGramLanes = 64;      // threads per tile of products, striding over the pixels
constexpr int kGramChunkPx = 512;   // pixels staged per chunk
constexpr int kGramBufs = 2;        // staging buffers (a third measured no faster)

// One staged chunk of pixels for the products conj(v_i) v_j of tile (TI, TJ), v a pixel's R projections
// and y (a row of R + 1 in shared memory): part[i * T + j] += ... for i <= j < R + 1
template <int R, int TI, int TJ>
__device__ __forceinline__ void gram_chunk(const float2 *rows, int np, int lane,
                                           float2 (&part)[kGramTile * kGramTile]) {
  constexpr int R1 = R + 1, T = kGramTile;
  for (int p = lane; p < np; p += kGramLanes) {
    float2 x[T], y[T];
#pragma unroll
    for (int i = 0; i < T; ++i) {
      if (TI * T + i < R1) x[i] = rows[p * R1 + TI * T + i];
      if (TI != TJ && TJ * T + i < R1) y[i] = rows[p * R1 + TJ * T + i];
    }
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) {
        if (TI * T + i > TJ * T + j || TJ * T + j >= R1) continue;
        const float2 a = x[i], c = TI == TJ ? x[j] : y[j];
        float2 &t = part[i * T + j];
        t.x = fmaf(a.x, c.x, fmaf(a.y, c.y, t.x));
        t.y = fmaf(a.x, c.y, fmaf(-a.y, c.x, t.y));
      }
  }
}

template <int R>
constexpr int kGramSide = (R + kGramTile) / kGramTile;  // tiles of a side
template <int R>
constexpr int kGramTiles = kGramSide<R> * (kGramSide<R> + 1) / 2;

// gram_chunk of tile number `sub` counted from (TI, TJ) along the upper triangle's rows
template <int R, int TI, int TJ>
__device__ __forceinline__ void gram_tile(int sub, const float2 *rows, int np, int lane,
                                          float2 (&part)[kGramTile * kGramTile]) {
  if (sub == 0) gram_chunk<R, TI, TJ>(rows, np, lane, part);
  else if constexpr (TJ + 1 < kGramSide<R>) gram_tile<R, TI, TJ + 1>(sub - 1, rows, np, lane, part);
  else if constexpr (TI + 1 < kGramSide<R>) gram_tile<R, TI + 1, TI + 1>(sub - 1, rows, np, lane, part);
}

// Per-image Gram for the fused step's layout (point-major Q with r contiguous projections per
// pixel): one block per image, two warps for each 3 x 3 tile of products.  Chunks of kGramChunkPx
// pixels are staged in shared memory by coalesced 8-byte asynchronous copies (double-buffered)
// as rows of r projections and y, 88 bytes apart at r = 10 so the tiles' 8-byte reads are
// free of bank conflicts; every tile reads every pixel of the chunk from there, and each
// thread adds its chunk sums to Kahan-compensated totals.  Reads of shared memory bound it: a
// tile reads 6 values (3 on the diagonal) for 9 products, 48 per pixel at r = 10 where eight
// subsets of 9 products that each read the whole row took 88 (0.61 -> 0.46 ms at 1024 images of
// 128^2, 1.5 GB).
template <int R>
__global__ void __launch_bounds__(kGramTiles<R> * kGramLanes, 1) gram_pixel_kernel(
    const float2 *__restrict__ Q, int64_t q_is, const float2 *__restrict__ Y, int P, float2 *__restrict__ gram,
    float2 *__restrict__ h, float *__restrict__ yy) {
  constexpr int R1 = R + 1, T = kGramTile, PER = T * T, NT = kGramTiles<R> * kGramLanes;
  extern __shared__ float2 srows[];  // kGramBufs * kGramChunkPx * R1
  const int b = blockIdx.x;
  const int sub = threadIdx.x / kGramLanes, lane = threadIdx.x % kGramLanes;
  float2 sum[PER], comp[PER];
#pragma unroll
  for (int kk = 0; kk < PER; ++kk) {
    sum[kk] = make_float2(0.f, 0.f);
    comp[kk] = make_float2(0.f, 0.f);
  }
  const float2 *Qb = Q + (int64_t)b * q_is;
  const float2 *Yb = Y + (int64_t)b * P;
  auto stage = [&](int c, float2 *dst) {
    const int p0 = c * kGramChunkPx, np = min(kGramChunkPx, P - p0);
    const float2 *src = Qb + (int64_t)p0 * R;
    for (int e = threadIdx.x; e < np * R; e += NT) {
      const int p = e / R, i = e - p * R;
      const unsigned d = (unsigned)__cvta_generic_to_shared(dst + p * R1 + i);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src + e) : "memory");
    }
    for (int p = threadIdx.x; p < np; p += NT) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(dst + p * R1 + R);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(Yb + p0 + p) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int nchunks = (P + kGramChunkPx - 1) / kGramChunkPx;
  // kGramBufs - 1 chunks in flight ahead of the one being summed; a buffer is refilled after the
  // barrier that ends the iteration which read it
  for (int c = 0; c < kGramBufs - 1; ++c) {
    if (c < nchunks) stage(c, srows + c * kGramChunkPx * R1);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int c = 0; c < nchunks; ++c) {
    const float2 *cur = srows + (c % kGramBufs) * kGramChunkPx * R1;
    const int cn = c + kGramBufs - 1;
    if (cn < nchunks) stage(cn, srows + (cn % kGramBufs) * kGramChunkPx * R1);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kGramBufs - 1) : "memory");
    __syncthreads();
    const int np = min(kGramChunkPx, P - c * kGramChunkPx);
    float2 part[PER];
#pragma unroll
    for (int kk = 0; kk < PER; ++kk) part[kk] = make_float2(0.f, 0.f);
    gram_tile<R, 0, 0>(sub, cur, np, lane, part);
#pragma unroll
    for (int kk = 0; kk < PER; ++kk) {  // Kahan update of the running totals
      float yx = part[kk].x - comp[kk].x, tx = sum[kk].x + yx;
      comp[kk].x = (tx - sum[kk].x) - yx;
      sum[kk].x = tx;
      float yv = part[kk].y - comp[kk].y, ty = sum[kk].y + yv;
      comp[kk].y = (ty - sum[kk].y) - yv;
      sum[kk].y = ty;
    }
    __syncthreads();  // the buffer is refilled next
  }
  // reduce over the 64 lanes of the tile: shuffles within each warp, then the two warps
  __shared__ float2 red[kGramTiles<R>][2][PER];
  const int w = lane >> 5;
#pragma unroll
  for (int kk = 0; kk < PER; ++kk) {
    float x = sum[kk].x, y = sum[kk].y;
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if ((lane & 31) == 0) red[sub][w][kk] = make_float2(x, y);
  }
  __syncthreads();
  if (lane < PER) {
    const int kk = lane;
    int ti = 0, tj = sub;
    while (tj >= kGramSide<R> - ti) {
      tj -= kGramSide<R> - ti;
      ++ti;
    }
    const int i = ti * T + kk / T, j = (ti + tj) * T + kk % T;
    if (i <= j && j < R1) {
      const float2 t = make_float2(red[sub][0][kk].x + red[sub][1][kk].x, red[sub][0][kk].y + red[sub][1][kk].y);
      if (j < R) {
        gram[((int64_t)b * R + i) * R + j] = t;
        if (i != j) gram[((int64_t)b * R + j) * R + i] = make_float2(t.x, -t.y);
      } else if (i < R) {
        h[(int64_t)b * R + i] = t;
      } else {
        yy[b] = t.x;
      }
    }
  }
}

struct cd {
  double x, y;
};
__device__ __forceinline__ cd cmul(cd a, cd b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ cd cconj(cd a) { return {a.x, -a.y}; }
__device__ __forceinline__ cd csub(cd a, cd b) { return {a.x - b.x, a.y - b.y}; }

// Solve (L L^H) x = rhs in place; the diagonal entry (k, k) of Lm holds {L_kk, 1 / L_kk}.
__device__ void chol_solve(const cd *Lm, int r, cd *x) {
  for (int i = 0; i < r; ++i) {
    cd s = x[i];
    for (int j = 0; j < i; ++j) s = csub(s, cmul(Lm[i * r + j], x[j]));
    const double inv = Lm[i * r + i].y;
    x[i] = {s.x * inv, s.y * inv};
  }
  for (int i = r - 1; i >= 0; --i) {
    cd s = x[i];
    for (int j = i + 1; j < r; ++j) s = csub(s, cmul(cconj(Lm[j * r + i]), x[j]));
    const double inv = Lm[i * r + i].y;
    x[i] = {s.x * inv, s.y * inv};
  }
}

struct SolveArgs {
  int B, r, objective;
  const float2 *gram;
  const float2 *h;
  const float *yy;
  double s2;
  const double *linv;  // (r, r) real symmetric added to gram/s2, or null (identity)
  double wscale;       // scale of C and u (1/B for ML, 1/(B L^4) for LS)
  double cscale;       // scale of the per-image cost
  float2 *C;           // (B, r, r)
  float2 *u;           // (B, r)
  double *cost_b;      // (B) or null
  double *cost_sum;    // scalar accumulator
  double *glog;        // (r) accumulators of d cost / d log_sqrt, or null
  float2 *z_out;       // (B, r) latent coordinates or null
  float2 *m_out;       // (B, r, r) m or null
  int *bad;            // set to 1 if a factorisation failed
};

constexpr int kSolveThreads = 128;

// r + 1 threads per image, kSolveThreads / (r + 1) images per block, each image's matrix in shared
// memory.  ML: thread i < r computes row i of the Cholesky factor column by column (left-looking,
// one barrier per column; every thread of the image forms the pivot itself), then solves for column i
// of m^-1 while thread r solves for z; RMAX sizes the threads' right-hand sides.  Latency is the
// bound, so each image is factored once by all its threads (each of r threads used to factor it alone
// in local memory: 204 -> 84 us at r = 10, B = 1024, 879 -> 235 us at r = 20, B = 300, 64 -> 34 us at r = 10, B = 64); the
// operations and their order are those of one thread's factorisation.
// glog receives d cost / d log s_k (the projections' channel k scaled by s_k), 2 Re sum_p conj(W_pk)
// Q_pk, which m z = b and m^-1 gram / s2 = I - m^-1 (identity prior) turn into
// wscale (1 - (m^-1)_kk - |z_k|^2) for ML -- no cancellation -- and
// wscale (4 sum_i |gram_ik|^2 + 4 s2 gram_kk - 4 |h_k|^2) for LS.
template <int RMAX>
__global__ void __launch_bounds__(kSolveThreads) solve_kernel(const SolveArgs a) {
  extern __shared__ double2 solve_smem[];
  __shared__ double s_glog[kSolveThreads], wsum[kSolveThreads / 32];
  const int r = a.r, ipb = kSolveThreads / (r + 1);
  const int im = threadIdx.x / (r + 1), kc = threadIdx.x - im * (r + 1);
  const int b = blockIdx.x * ipb + im;
  const bool live = im < ipb && b < a.B;
  cd *m = reinterpret_cast<cd *>(solve_smem) + (size_t)(im < ipb ? im : 0) * (r * r + 2 * r);  // r * r
  cd *s_z = m + r * r, *s_b = s_z + r;                                                           // r each
  const float2 *G = a.gram + (int64_t)b * r * r;
  const float2 *hb = a.h + (int64_t)b * r;
  double cost = 0.0, glog = 0.0;
  if (a.objective == 0) {
    if (live) {
      for (int e = kc; e < r * r; e += r + 1) {
        const int i = e / r, j = e - i * r;
        const float2 g = G[e];
        const double add = a.linv ? a.linv[e] : (i == j ? 1.0 : 0.0);
        m[e] = {g.x / a.s2 + add, g.y / a.s2};
        if (a.m_out) a.m_out[(int64_t)b * r * r + e] = make_float2((float)m[e].x, (float)m[e].y);
      }
      if (kc < r) s_b[kc] = {hb[kc].x / a.s2, hb[kc].y / a.s2};
    }
    __syncthreads();
    double logdet = 0.0;
    bool ok = true;
    for (int k = 0; k < r; ++k) {
      cd lik = {0.0, 0.0};
      if (live && ok) {
        double d = m[k * r + k].x;
        for (int j = 0; j < k; ++j) d -= m[k * r + j].x * m[k * r + j].x + m[k * r + j].y * m[k * r + j].y;
        if (!(d > 0.0)) {
          ok = false;  // the same for every thread of the image
          if (kc == 0) atomicExch(a.bad, 1);
        } else {
          const double lkk = sqrt(d), inv = 1.0 / lkk;
          if (kc == r) logdet += 2.0 * log(lkk);
          if (kc == k) {
            lik = {lkk, inv};
          } else if (kc > k && kc < r) {
            cd s = m[kc * r + k];
            for (int j = 0; j < k; ++j) s = csub(s, cmul(m[kc * r + j], cconj(m[k * r + j])));
            lik = {s.x * inv, s.y * inv};
          }
        }
      }
      __syncthreads();  // (k, k) has been read as the pivot's own entry
      if (live && ok && kc >= k && kc < r) m[kc * r + k] = lik;
      __syncthreads();
    }
    cd x[RMAX];
    const bool solves = live && ok;
    if (solves && (kc == r || a.C)) {
      for (int i = 0; i < r; ++i) x[i] = kc == r ? s_b[i] : cd{i == kc ? 1.0 : 0.0, 0.0};
      chol_solve(m, r, x);
    }
    if (solves && kc == r) {
      double bz = 0.0;
      for (int i = 0; i < r; ++i) {
        bz += s_b[i].x * x[i].x + s_b[i].y * x[i].y;
        s_z[i] = x[i];
        if (a.z_out) a.z_out[(int64_t)b * r + i] = make_float2((float)x[i].x, (float)x[i].y);
      }
      cost = 0.5 * (-bz + logdet);
    }
    __syncthreads();
    if (solves && a.C) {
      // C_ij = (conj(minv_ij) + conj(z_i) z_j) / (2 s2), column kc
      const double f = a.wscale / (2.0 * a.s2);
      if (kc < r) {
        const cd zk = s_z[kc];
        glog = a.wscale * (1.0 - x[kc].x - (zk.x * zk.x + zk.y * zk.y));
        for (int i = 0; i < r; ++i) {
          const cd zz = cmul(cconj(s_z[i]), zk);
          a.C[((int64_t)b * r + i) * r + kc] = make_float2((float)((x[i].x + zz.x) * f), (float)((-x[i].y + zz.y) * f));
        }
        a.u[(int64_t)b * r + kc] = make_float2((float)(-zk.x * f), (float)(zk.y * f));
      }
    }
  } else if (live && kc < r) {  // least squares: M = conj(gram), t = conj(h)
    double g2 = 0.0;
    for (int i = 0; i < r; ++i) g2 += (double)G[i * r + kc].x * G[i * r + kc].x + (double)G[i * r + kc].y * G[i * r + kc].y;
    const double h2 = (double)hb[kc].x * hb[kc].x + (double)hb[kc].y * hb[kc].y;
    if (a.C) {
      const double f = a.wscale;
      glog = 4.0 * f * (g2 + a.s2 * G[kc * r + kc].x - h2);
      for (int i = 0; i < r; ++i) {
        const float2 g = G[i * r + kc];  // M_ij = conj(gram_ij)
        a.C[((int64_t)b * r + i) * r + kc] =
            make_float2((float)((2.0 * g.x + (i == kc ? 2.0 * a.s2 : 0.0)) * f), (float)(-2.0 * g.y * f));
      }
      a.u[(int64_t)b * r + kc] = make_float2((float)(-2.0 * hb[kc].x * f), (float)(2.0 * hb[kc].y * f));
    }
    if (kc == 0) {
      double t2 = 0.0, fro = 0.0, tr = 0.0;
      for (int i = 0; i < r; ++i) {
        t2 += (double)hb[i].x * hb[i].x + (double)hb[i].y * hb[i].y;
        tr += G[i * r + i].x;
        for (int j = 0; j < r; ++j) fro += (double)G[i * r + j].x * G[i * r + j].x + (double)G[i * r + j].y * G[i * r + j].y;
      }
      cost = -2.0 * t2 + fro + 2.0 * a.s2 * tr;
    }
  }
  // the image's cost is with one thread: z's, or the first in least squares
  const bool teller = live && kc == (a.objective == 0 ? r : 0);
  cost = teller ? cost * a.cscale : 0.0;
  if (teller && a.cost_b) a.cost_b[b] = cost;
  if (!a.cost_sum) return;
  if (a.glog) {  // the block's images summed per channel
    s_glog[threadIdx.x] = glog;
    __syncthreads();
    if ((int)threadIdx.x < r) {
      double t = 0.0;
      for (int i = 0; i < ipb; ++i) t += s_glog[i * (r + 1) + threadIdx.x];
      atomicAdd(a.glog + threadIdx.x, t);
    }
  }
  // the images' costs summed per block (one FP64 atomic per block)
  for (int o = 16; o > 0; o >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cost;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < kSolveThreads / 32; ++i) t += wsum[i];
    atomicAdd(a.cost_sum, t);
  }
}

// W = C Q + u y on chunks of pixels of one image (Q element (p, i) at
// Q[b*q_is + p*q_ps + i*q_cs], W likewise with its own strides; W may alias Q).
__global__ void __launch_bounds__(256) wpass_kernel(const float2 *Q, int64_t q_is, int64_t q_ps, int64_t q_cs,
                                                    const float2 *__restrict__ Y, const float2 *__restrict__ C,
                                                    const float2 *__restrict__ u, int P, int r, float2 *W,
                                                    int64_t w_is, int64_t w_ps, int64_t w_cs) {
  extern __shared__ float2 sw[];
  float2 *sC = sw;                    // r*r
  float2 *su = sC + r * r;            // r
  float2 *sq = su + r;                // kGramChunk * r
  float2 *sy = sq + kGramChunk * r;   // kGramChunk
  const int b = blockIdx.y;
  const int p0 = blockIdx.x * kGramChunk;
  const int np = min(kGramChunk, P - p0);
  const int tid = threadIdx.x;
  for (int e = tid; e < r * r; e += blockDim.x) sC[e] = C[(int64_t)b * r * r + e];
  for (int e = tid; e < r; e += blockDim.x) su[e] = u[(int64_t)b * r + e];
  const float2 *Qb = Q + (int64_t)b * q_is;
  for (int e = tid; e < np * r; e += blockDim.x) {
    const int pp = e / r, i = e - pp * r;
    sq[e] = Qb[(int64_t)(p0 + pp) * q_ps + (int64_t)i * q_cs];
  }
  for (int e = tid; e < np; e += blockDim.x) sy[e] = Y[(int64_t)b * P + p0 + e];
  __syncthreads();
  float2 *Wb = W + (int64_t)b * w_is;
  for (int e = tid; e < np * r; e += blockDim.x) {
    const int p = e / r, i = e - p * r;
    const float2 yv = sy[p];
    const float2 ui = su[i];
    float2 acc = make_float2(ui.x * yv.x - ui.y * yv.y, ui.x * yv.y + ui.y * yv.x);
    const float2 *crow = sC + i * r;
    const float2 *qp = sq + p * r;
    for (int j = 0; j < r; ++j) {
      const float2 c = crow[j], q = qp[j];
      acc.x = fmaf(c.x, q.x, fmaf(-c.y, q.y, acc.x));
      acc.y = fmaf(c.x, q.y, fmaf(c.y, q.x, acc.y));
    }
    Wb[(int64_t)(p0 + p) * w_ps + (int64_t)i * w_cs] = acc;
  }
}

// W = C Q + u y for channel-major Q and W (a channel's pixels adjacent): one thread per pixel with its r
// projections in registers, C and u broadcast from shared memory.  Memory bounds it; staging the chunk
// for the transposed reads of the kernel above cost 205 us where this takes 46 (r = 8, 512 images of
// 64^2, 0.27 GB).  RMAX is the smallest class that holds r.
template <int RMAX>
__global__ void __launch_bounds__(256) wpass_channel_kernel(const float2 *Q, int64_t q_is, int64_t q_cs,
                                                            const float2 *__restrict__ Y, const float2 *__restrict__ C,
                                                            const float2 *__restrict__ u, int P, int r, float2 *W,
                                                            int64_t w_is, int64_t w_cs) {
  __shared__ float2 sC[RMAX * RMAX], su[RMAX];
  const int b = blockIdx.y;
  for (int e = threadIdx.x; e < r * r; e += blockDim.x) sC[e / r * RMAX + e % r] = C[(int64_t)b * r * r + e];
  for (int e = threadIdx.x; e < r; e += blockDim.x) su[e] = u[(int64_t)b * r + e];
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  const float2 *qp = Q + (int64_t)b * q_is + p;
  float2 *wp = W + (int64_t)b * w_is + p;
  const float2 yv = Y[(int64_t)b * P + p];
  float2 q[RMAX];
#pragma unroll
  for (int j = 0; j < RMAX; ++j) q[j] = j < r ? qp[j * q_cs] : make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < RMAX; ++i) {
    if (i >= r) break;
    const float2 ui = su[i];
    float2 acc = make_float2(ui.x * yv.x - ui.y * yv.y, ui.x * yv.y + ui.y * yv.x);
#pragma unroll
    for (int j = 0; j < RMAX; ++j) {
      if (j < r) {
        const float2 c = sC[i * RMAX + j];
        acc.x = fmaf(c.x, q[j].x, fmaf(-c.y, q[j].y, acc.x));
        acc.y = fmaf(c.x, q[j].y, fmaf(c.y, q[j].x, acc.y));
      }
    }
    wp[i * w_cs] = acc;
  }
}

// wpass for the fused step's layout (point-major, channel stride 1, W over Q in place): one
// thread per pixel holds its r projections and y in registers (16-byte loads), C and u are
// broadcast from shared memory, the r outputs are written back over the pixel's Q (16-byte
// stores).
template <int R>
__global__ void __launch_bounds__(256) wpass_pixel_kernel(float2 *QW, int64_t q_is, int64_t q_ps,
                                                          const float2 *__restrict__ Y, const float2 *__restrict__ C,
                                                          const float2 *__restrict__ u, int P) {
  __shared__ float2 sC[R * R], su[R];
  const int b = blockIdx.y;
  for (int e = threadIdx.x; e < R * R; e += blockDim.x) sC[e] = C[(int64_t)b * R * R + e];
  for (int e = threadIdx.x; e < R; e += blockDim.x) su[e] = u[(int64_t)b * R + e];
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  float2 *qp = QW + (int64_t)b * q_is + (int64_t)p * q_ps;
  float2 q[R];
  // the pixel's R complex values as R/2 16-byte loads (R even, rows 16-byte aligned: checked
  // by the launcher; 0.69 -> 0.56 ms against 8-byte loads)
  float4 *qp4 = reinterpret_cast<float4 *>(qp);
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    const float4 v = qp4[j];
    q[2 * j] = make_float2(v.x, v.y);
    q[2 * j + 1] = make_float2(v.z, v.w);
  }
  const float2 yv = Y[(int64_t)b * P + p];
  float2 w[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float2 ui = su[i];
    float2 acc = make_float2(ui.x * yv.x - ui.y * yv.y, ui.x * yv.y + ui.y * yv.x);
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float2 c = sC[i * R + j];
      acc.x = fmaf(c.x, q[j].x, fmaf(-c.y, q[j].y, acc.x));
      acc.y = fmaf(c.x, q[j].y, fmaf(c.y, q[j].x, acc.y));
    }
    w[i] = acc;
  }
#pragma unroll
  for (int i = 0; i < R / 2; ++i) qp4[i] = make_float4(w[2 * i].x, w[2 * i].y, w[2 * i + 1].x, w[2 * i + 1].y);
}

__global__ void finalize_kernel(const double *acc, int r, double inv_count, double *d_cost, float *glog) {
  const int i = threadIdx.x;
  if (i == 0 && d_cost) *d_cost = acc[0] * inv_count + acc[1];
  if (i < r && glog) glog[i] = (float)acc[8 + i];
}

}  // namespace

int launch_gram(cudaStream_t st, int B, int P, int r, const void *q, int64_t is, int64_t ps, int64_t cs,
                const void *images, void *gram, void *h, float *yy) {
  if (r < 1 || r > kMaxRank) {
    set_error("rank %d out of range (1..%d)", r, kMaxRank);
    return COV3D_EINVAL;
  }
  if (cs == 1 && ps == r && r == 10) {
    const size_t smem = kGramBufs * (size_t)kGramChunkPx * (10 + 1) * sizeof(float2);
    cudaError_t e = cudaFuncSetAttribute(gram_pixel_kernel<10>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gram_pixel_kernel)");
    gram_pixel_kernel<10><<<B, kGramTiles<10> * kGramLanes, smem, st>>>(
        static_cast<const float2 *>(q), is, static_cast<const float2 *>(images), P, static_cast<float2 *>(gram),
        static_cast<float2 *>(h), yy);
    return launched("gram_pixel_kernel");
  }
  const int J = (r + 1) * (r + 2) / 2;
  const int threads = J > 256 ? ((J + 31) / 32) * 32 : 256;
  const int groups = threads / J;
  const int rs = (r + kGramTile) / kGramTile * kGramTile;
  const int cbytes = (kGramChunk * rs + 3) * (int)sizeof(float2);
  int nc = kGramStage / cbytes;
  nc = std::max(1, std::min(std::min(nc, 8), (P + kGramChunk - 1) / kGramChunk));
  const size_t smem = (size_t)nc * (cbytes + groups * J * sizeof(float2));
  // one limit for every rank: calls of several threads set the same
  constexpr int kMost = kGramStage + 8 * 255 * (int)sizeof(float2) + (1 << 14);
  if (smem > (size_t)kMost) {
    set_error("Gram stage of %zu bytes", smem);
    return COV3D_EINVAL;
  }
  COV3D_CUDA(cudaFuncSetAttribute(gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  gram_kernel<<<B, threads, smem, st>>>(static_cast<const float2 *>(q), is, ps, cs, static_cast<const float2 *>(images),
                                        P, r, groups, nc, rs, static_cast<float2 *>(gram), static_cast<float2 *>(h),
                                        yy);
  return launched("gram_kernel");
}

int launch_wpass(cudaStream_t st, int B, int P, int r, const void *q, int64_t is, int64_t ps, int64_t cs,
                 const void *images, const void *C, const void *u, void *w, int64_t wis, int64_t wps, int64_t wcs) {
  if (q == w && is == wis && ps == wps && cs == 1 && wcs == 1 && ps == r && (r == 10 || r == 20) &&
      (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (is & 1) == 0) {
    dim3 g((P + 255) / 256, B);
    float2 *qw = static_cast<float2 *>(w);
    const float2 *y = static_cast<const float2 *>(images);
    const float2 *cc = static_cast<const float2 *>(C), *uu = static_cast<const float2 *>(u);
    if (r == 10) {
      wpass_pixel_kernel<10><<<g, 256, 0, st>>>(qw, is, ps, y, cc, uu, P);
    } else {
      wpass_pixel_kernel<20><<<g, 256, 0, st>>>(qw, is, ps, y, cc, uu, P);
    }
    return launched("wpass_pixel_kernel");
  }
  if (ps == 1 && wps == 1) {
    dim3 g((P + 255) / 256, B);
    auto launch = [&](auto kernel) {
      kernel<<<g, 256, 0, st>>>(static_cast<const float2 *>(q), is, cs, static_cast<const float2 *>(images),
                                static_cast<const float2 *>(C), static_cast<const float2 *>(u), P, r,
                                static_cast<float2 *>(w), wis, wcs);
      return launched("wpass_channel_kernel");
    };
    if (r <= 4) return launch(wpass_channel_kernel<4>);
    if (r <= 8) return launch(wpass_channel_kernel<8>);
    if (r <= 12) return launch(wpass_channel_kernel<12>);
    if (r <= 16) return launch(wpass_channel_kernel<16>);
    if (r <= 20) return launch(wpass_channel_kernel<20>);
    return launch(wpass_channel_kernel<kMaxRank>);
  }
  const size_t smem = (size_t)(r * r + r + kGramChunk * (r + 1)) * sizeof(float2);
  dim3 grid((P + kGramChunk - 1) / kGramChunk, B);
  wpass_kernel<<<grid, 256, smem, st>>>(static_cast<const float2 *>(q), is, ps, cs,
                                        static_cast<const float2 *>(images), static_cast<const float2 *>(C),
                                        static_cast<const float2 *>(u), P, r, static_cast<float2 *>(w), wis, wps,
                                        wcs);
  return launched("wpass_kernel");
}

int launch_solve(cudaStream_t st, int B, int r, int objective, const void *gram, const void *h, double s2,
                 const double *linv, double wscale, double cscale, void *C, void *u, double *cost_b, double *cost_sum,
                 void *z, void *m, int *bad, double *glog) {
  if (r < 1 || r > kMaxRank) {
    set_error("rank %d out of range (1..%d)", r, kMaxRank);
    return COV3D_EINVAL;
  }
  SolveArgs sa{};
  sa.B = B;
  sa.r = r;
  sa.objective = objective;
  sa.gram = static_cast<const float2 *>(gram);
  sa.h = static_cast<const float2 *>(h);
  sa.s2 = s2;
  sa.linv = linv;
  sa.wscale = wscale;
  sa.cscale = cscale;
  sa.C = static_cast<float2 *>(C);
  sa.u = static_cast<float2 *>(u);
  sa.cost_b = cost_b;
  sa.cost_sum = cost_sum;
  sa.glog = glog;
  sa.z_out = static_cast<float2 *>(z);
  sa.m_out = static_cast<float2 *>(m);
  sa.bad = bad;
  static_assert(kMaxRank + 1 <= kSolveThreads, "a thread per column of every image and one for z");
  const int ipb = kSolveThreads / (r + 1);
  const unsigned blocks = (unsigned)((B + ipb - 1) / ipb);
  const size_t smem = objective == 0 ? (size_t)ipb * (r * r + 2 * r) * sizeof(cd) : 0;
  auto launch = [&](auto kernel) -> int {
    // (one limit for every rank: calls of several threads set the same)
    if (smem > 40 * 1024)
      COV3D_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    kernel<<<blocks, kSolveThreads, smem, st>>>(sa);
    return COV3D_OK;
  };
  if (r <= 10) COV3D_TRY(launch(solve_kernel<10>));
  else if (r <= 16) COV3D_TRY(launch(solve_kernel<16>));
  else if (r <= 20) COV3D_TRY(launch(solve_kernel<20>));
  else COV3D_TRY(launch(solve_kernel<kMaxRank>));
  return launched("solve_kernel");
}

int covar_cost_grad(cov3d_plan *p, const cov3d_cost_args *a, double *h_cost, double *d_cost, float *d_grad_vectors,
                    float *d_grad_log_sqrt, double *d_per_image_cost) {
  const int r = a->rank;
  if (r < 1 || r > kMaxRank || r > p->n_trans) {
    set_error("rank %d out of range (1..min(32, n_trans=%d))", r, p->n_trans);
    return COV3D_EINVAL;
  }
  if (!a->d_vectors || !a->d_log_sqrt || !a->d_images || !d_grad_vectors || !d_grad_log_sqrt) {
    set_error("null pointer argument");
    return COV3D_EINVAL;
  }
  if (p->point_kind == kPointsNone || p->points_L != p->L) {
    set_error("points for L=%d images must be set before the cost", p->L);
    return COV3D_ESTATE;
  }
  if (!(a->noise_var > 0.0)) {
    set_error("noise_var must be positive");
    return COV3D_EINVAL;
  }
  COV3D_TRY(need_sorted(p, 1u << kSortFull | 1u << hermitian_mode(p)));  // interpolation | spreading
  const int B = (int)p->n_images;
  const int L = p->L;
  const int P = L * L;
  const int64_t n3 = (int64_t)p->n * p->n * p->n;
  const int64_t M = p->n_points;

  COV3D_TRY(grow(p->fine, n3 * r * 8));
  COV3D_TRY(grow(p->fine2, n3 * r * 8));
  COV3D_TRY(grow(p->q, M * r * 8));
  const int64_t small_bytes = (int64_t)B * (r * r * 8 * 2 + r * 8 * 2 + 8 + 8) + 64;
  COV3D_TRY(grow(p->small, small_bytes));
  float2 *gram = p->small.as<float2>();
  float2 *h = gram + (int64_t)B * r * r;
  float2 *C = h + (int64_t)B * r;
  float2 *u = C + (int64_t)B * r * r;
  float *yy = reinterpret_cast<float *>(u + (int64_t)B * r);
  int *bad = reinterpret_cast<int *>(yy + B);
  double *acc = p->acc.as<double>();

  COV3D_CUDA(cudaMemsetAsync(acc, 0, 64 * sizeof(double), p->stream));
  COV3D_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), p->stream));

  // 1. pack the deapodised, scaled eigenvolumes into the fine grid; 2. forward FFT.  Even L:
  // pruned transforms, staged in fine2 (zeroed before the spread anyway): 2D FFTs over each
  // channel's L support planes, then the axis-0 FFT out of place into fine.
  const bool pruned = prunable(p);
  // fine grids of n = 128 .. 512: hand-written line transforms with the pack, the regulariser
  // (value, and the gradient grid's initial coef * fr * G or zero) and the unpack fused in.  The
  // forward one up to n = 256: at 512 its 32 x 16 split idles half the threads in one stage and
  // measured slower than pack + cuFFT + regulariser (19.0 against 15.4 ms at L = 256, r = 10);
  // the inverse is faster at every size (8.8 against 11.1 ms there).
  // n = 64 has the inverse only: its forward transform keeps cuFFT's rounding, on which the 64-bit
  // cost depends.
  const bool lines_inv = grid_lines_apply(p);
  const bool lines_fwd = lines_inv && line_transforms_apply(p) && p->n <= 256;
  const bool with_reg = a->d_fourier_reg && a->reg_scale != 0.0;
  const bool ml_reg = with_reg && a->objective == 0;  // sum fr |G|^2: fused into the transforms
  const bool ls_reg = with_reg && a->objective != 0;  // |X X^H|^2: GEMMs before the spread (ls_reg.cu)
  const int64_t fr_stride = a->fourier_reg_per_channel ? n3 : 0;
  const float *gcp = a->use_grid_correction ? p->gc1d.as<float>() : nullptr;
  cufftHandle fft = 0, fplanes = 0, faxis0 = 0;
  // Small grids: one launch for all planes of all channels instead of two per channel (the same
  // transforms of each plane, to the bit; 5 channels of 64^3: 103 -> 33 us with axis 0, of 160^3:
  // 226 -> 215; of 200^3 the planes outside the support cost more: 441 against 505).
  const bool all_planes = pruned && !lines_fwd && p->n <= kSmallGrid && fft_ready(p, kAllPlanesKey - r);
  if (pruned) {
    if (!lines_fwd) {  // the forward transform on cuFFT
      if (all_planes) COV3D_TRY(get_fft_all_planes(p, r, &fplanes));
      else COV3D_TRY(get_fft_planes(p, &fplanes));
      COV3D_TRY(get_fft_axis0(p, &faxis0));
    }
  } else {
    COV3D_TRY(get_fft(p, r, &fft));
  }
  const int64_t half_off = (int64_t)(p->n - L / 2) * p->n * p->n;
  if (lines_fwd) {
    PhaseScope ps(p, kPhaseFftFwd);
    COV3D_TRY(step_forward_lines(p, a->d_vectors, a->d_log_sqrt, gcp, r, p->fine2.as<float2>(), p->fine.as<float2>(),
                                 ml_reg ? a->d_fourier_reg : nullptr, fr_stride, a->reg_scale / (2.0 * a->noise_var),
                                 acc + 1, acc + 8));
  } else {
    PhaseScope ps(p, kPhasePack);
    COV3D_TRY(launch_pack(p, a->d_vectors, nullptr, a->d_log_sqrt, a->use_grid_correction, r,
                          pruned ? p->fine2.ptr : p->fine.ptr));
  }
  if (!lines_fwd) {
    PhaseScope ps(p, kPhaseFftFwd);
    if (pruned) {
      if (all_planes) COV3D_TRY(fft2(fplanes, p->fine2.as<float2>(), p->fine2.as<float2>(), CUFFT_FORWARD));
      for (int c = 0; c < r; ++c) {
        float2 *src = p->fine2.as<float2>() + c * n3;
        if (!all_planes) {
          COV3D_TRY(fft2(fplanes, src, src, CUFFT_FORWARD));
          COV3D_TRY(fft2(fplanes, src + half_off, src + half_off, CUFFT_FORWARD));
        }
        COV3D_TRY(fft2(faxis0, src, p->fine.as<float2>() + c * n3, CUFFT_FORWARD));
      }
    } else {
      COV3D_TRY(check_cufft(cufftExecC2C(fft, p->fine.as<cufftComplex>(), p->fine.as<cufftComplex>(), CUFFT_FORWARD),
                            "cufftExecC2C(forward)"));
    }
  }
  // 3. interpolate at the central slices with the fused projection epilogue -> Q (B*P, r)
  const int shift = p->n - p->n / 2;
  GridArgs ga{p->fine.ptr, 1, n3, shift};
  EpilogueArgs ep{a->ctf_params ? nullptr : a->d_ctf, 1, 1.0f / (float)L};
  if (a->ctf_params && a->d_ctf) COV3D_TRY(prepare_ctf_coef(p, a->d_ctf, B, L, &ep.ctfc));
  {
    PhaseScope ps(p, kPhaseInterp);
    COV3D_TRY(launch_interp(p, ga, r, p->q.ptr, r, 1, ep, kSortFull));
  }
  // 4. per-image Gram, 5. FP64 solve -> cost, C, u
  {
    PhaseScope ps(p, kPhaseGram);
    if (a->gram_bf16) {
      COV3D_TRY(launch_gram_bf16(p, p->stream, B, P, r, p->q.ptr, (int64_t)P * r, r, 1, a->d_images, gram, h, yy));
    } else {
      COV3D_TRY(launch_gram(p->stream, B, P, r, p->q.ptr, (int64_t)P * r, r, 1, a->d_images, gram, h, yy));
    }
  }
  const double L4 = (double)L * L * L * L;
  {
    PhaseScope ps(p, kPhaseSolve);
    COV3D_TRY(launch_solve(p->stream, B, r, a->objective, gram, h, a->noise_var, nullptr,
                           a->objective == 0 ? 1.0 / B : 1.0 / (B * L4), a->objective == 0 ? 1.0 : 1.0 / L4, C, u,
                           d_per_image_cost, acc, nullptr, nullptr, bad, acc + 8));
  }
  // 6. dcost/dconj(Q) in place, 7. spread through the adjoint (CTF, Nyquist, 1/L prologue): exact for
  // nearest cells; the other windows' pair records sit up to 6e-5 cells from the 32-bit indices that
  // the projections were taken at, and are the finer ones
  {
    PhaseScope ps(p, kPhaseWpass);
    COV3D_TRY(launch_wpass(p->stream, B, P, r, p->q.ptr, (int64_t)P * r, r, 1, a->d_images, C, u, p->q.ptr,
                           (int64_t)P * r, r, 1));
  }
  // 7'. the regulariser (value and gradient coef * fr * G) initialises the gradient grid, so the
  // spread adds onto it and no zeroing pass is needed; without one, the grid is zeroed
  if (ml_reg && !lines_fwd) {
    PhaseScope ps(p, kPhaseReg);
    COV3D_TRY(launch_ml_reg(p, p->fine.ptr, p->fine2.ptr, a->d_fourier_reg, fr_stride, r,
                            a->reg_scale / (2.0 * a->noise_var), acc + 1, acc + 8, 1));
  }
  if (ls_reg) {  // value and derivative, onto the gradient grid (zero after the line transforms)
    PhaseScope ps(p, kPhaseReg);
    if (!lines_fwd) COV3D_TRY(launch_zero(p, p->fine2.ptr, n3 * r * 8));
    COV3D_TRY(launch_ls_reg(p, p->fine.ptr, p->fine2.ptr, a->d_fourier_reg, fr_stride, r, a->reg_scale / L4,
                            acc + 1, acc + 8));
  }
  {
    PhaseScope ps(p, kPhaseSpread);
    if (!with_reg && !lines_fwd) COV3D_TRY(launch_zero(p, p->fine2.ptr, n3 * r * 8));
    // only the real part of the inverse transform is used: mirror pixels are spread together
    COV3D_TRY(launch_spread(p, p->q.ptr, r, 1, r, ep, p->fine2.ptr, 1, n3, shift, hermitian_mode(p)));
  }
  // 9. adjoint FFT, 10. crop + deapodise + chain rule to the Covar parameters
  if (lines_inv) {
    PhaseScope ps(p, kPhaseFftInv);
    COV3D_TRY(inverse_lines(p, p->fine2.as<float2>(), a->d_log_sqrt, gcp, r, d_grad_vectors, nullptr));
  } else {
    PhaseScope ps(p, kPhaseFftInv);
    COV3D_TRY(grid_fft(p, p->fine2.as<float2>(), r, CUFFT_INVERSE));
  }
  if (!lines_inv) {
    PhaseScope ps(p, kPhaseUnpack);
    COV3D_TRY(launch_unpack_grad(p, p->fine2.ptr, a->d_log_sqrt, a->use_grid_correction, r, d_grad_vectors));
  }
  finalize_kernel<<<1, 64, 0, p->stream>>>(acc, r, 1.0 / B, d_cost, d_grad_log_sqrt);
  COV3D_LAUNCHED("finalize_kernel");
  if (h_cost) {
    COV3D_CUDA(cudaMemcpyAsync(p->h_acc, acc, 8 * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
    int h_bad = 0;
    COV3D_CUDA(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
    COV3D_CUDA(cudaStreamSynchronize(p->stream));
    if (h_bad) {
      set_error("a per-image matrix m was not positive definite");
      return COV3D_ENONFINITE;
    }
    *h_cost = p->h_acc[0] / B + p->h_acc[1];
  }
  return COV3D_OK;
}

}  // namespace cov3d
