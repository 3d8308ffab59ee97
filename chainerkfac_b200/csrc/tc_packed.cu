// Products of operands that lie in memory as fp16 terms (chunks of 128 rows x
// 32 k, GemmDesc::ca / cb): the long products of the inverse, C = alpha A B +
// beta C over many problems in one launch, three tcgen05.mma (kind::f16) per
// product, C += hi*hi + hi*lo + lo*hi, the cross terms in accumulators of their
// own.
//
// A k-block of an operand tile is one bulk copy of 16 KB, already in the layout
// the MMAs read: no value is loaded, split and stored again by every tile that
// uses it.  That is what the tile kernel (tc_tile.cu) spends its time on: a
// 128 x 256 x 32 block takes 1600 ns there with TF32 terms, its MMAs 810, its
// loads alone 630.  1332 tiles with K = 4608 run here at 1335 TFLOP/s of bf16-rate
// MMAs (97 % of what a long cuBLAS loop sustains), the tile kernel reached 580 of
// half that rate.  Bound: long products by the MMAs and the feed from L2 (32 KB
// per SM and 384 cycles of MMAs); the K = 512 ones by their passes over C, so two
// CTAs share an SM, one in its epilogue beside the other's MMAs (three stages of
// 32 KB and half of the tensor memory each).  256 x 256 tiles of two CTAs
// (cta_group::2), which halve the feed, took 690 ns per k-block against 4 x 240 /
// 2 here: not kept.
//
// Warp 0 issues the copies, warp 1 the MMAs, eight warps the epilogue.
//
// Every barrier wait is bounded; a wait that runs out raises a status word
// instead of hanging.
#include <algorithm>
#include <mutex>

#include "gemm_simt.cuh"
#include "tc_common.cuh"

namespace kfac {

// Stages: three for two CTAs an SM.  Six in preconditioning launches without a
// second tile for an SM (148 tiles with K = 4608: 66 us with three, 50 with six);
// the inverse's launches run beside each other and keep room for two (108
// factors of ResNet-50 with their preconditioning: 4384 us, 4500 with six stages
// in its small launches).
constexpr int KP_STAGES_MAX = 6;
constexpr int KP_STAGE = 2 * kChunk;
constexpr int KP_EPI_WARPS = 8;
constexpr int KP_THREADS = 32 * (2 + KP_EPI_WARPS);
constexpr int packed_smem(int stages) { return stages * KP_STAGE + 2048; }
// Longest contraction of one accumulator, in k-blocks of 32.  The tensor core
// adds with truncation, so a sum drifts with the number of MMAs behind it; past
// this many the accumulators are added to C (round to nearest) and start anew.
// Errors of inverses of 27 to 4608 rows against fp64 (Wishart, low-rank, badly
// scaled and non-negative factors, damping 1e-6 to 1e-2), relative to those with
// TF32 terms and a pass over C per 512 k: up to 3.8 without a cut, 1.7 with one
// per 1024 k, 0.43 to 1.02 with 512, counted from the product's first k so that
// a long sum's large leading part does not carry the next panel's.
constexpr int KP_SEGMENT = 16;

static __device__ int g_packed_status = 0;

struct PackInline {
  int n;                       // 0: jobs in device memory
  PackRows j[3 * TT_INLINE];   // three operands a layer
};
static_assert(sizeof(PackInline) <= 3800, "kernel argument space");

struct GradInline {
  int n;
  GradSizes j[TT_INLINE];
};

struct PackedControl {
  unsigned long long full[KP_STAGES_MAX];    // the copies have arrived
  unsigned long long empty[KP_STAGES_MAX];   // the MMAs have read the stage
  unsigned long long accum;              // a segment's accumulators are final
  unsigned long long drained;            // and have been read
  unsigned tmem_base;
  volatile int abort_flag;
  GemmDesc desc;
};
static_assert(sizeof(PackedControl) <= 1024, "packed control block");

__device__ __forceinline__ void bulk_load(unsigned dst, const void* src,
                                          unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(kChunk), "r"(smem_u32(bar))
      : "memory");
}

// Elements of a 16 x 32 piece of C in that order, this lane's first at row r,
// column c: f(i, row offset, column offset) for those stored, which are all
// (WHOLE), or the ones in front of `rows` and `cols` and (lower) not above the
// diagonal.
template <bool WHOLE, typename F>
__device__ __forceinline__ void piece_each(int r, int c, int rows, int cols,
                                           bool lower, F f) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int dr = 8 * ((i >> 1) & 1), dc = 8 * (i >> 2) + (i & 1);
    if (WHOLE || (r + dr < rows && c + dc < cols &&
                  (!lower || c + dc <= r + dr)))
      f(i, dr, dc);
  }
}

// First product of the preconditioning: a 16 x 32 piece of U = grad A_inv^T into
// chunks, rows as k (zeros up to the end of the last k-block).  Rows and columns
// are divided by bounds of the norms of what they are products of, so that an
// entry is held relative to the most that its row and column could make it; the
// rows' sizes are in G_inv's columns, the columns' part and `wide` (the most that
// a row's norm exceeds its size) come out of kf.
// `rs`, `cs`: the lane's two rows' and eight columns' factors.
__device__ __forceinline__ void load_u(const GemmDesc& g, int r, float rs[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    rs[h] = r + 8 * h < g.M ? g.rs[r + 8 * h] : 0.f;
}
__device__ __forceinline__ void load_u_columns(const GemmDesc& g, int c,
                                               float cs[8]) {
  // (columns past the last one: any values, nobody stores their results)
#pragma unroll
  for (int j = 0; j < 8; ++j)
    cs[j] = g.cs[min(c + 8 * (j >> 1) + (j & 1), g.N - 1)];
}
__device__ __forceinline__ void store_u(const GemmDesc& g, const float v[16],
                                        int r, int c, const float rs[2],
                                        const float cs[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int gr = r + 8 * h;
    const bool in = gr < g.M;
    unsigned char* const row = g.pack + (long long)(gr >> 5) * kChunk +
                               (long long)(c >> 7) * g.pack_tile +
                               ((c >> 6) & 1) * 8192;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      unsigned hi, lo;
      split_half2(in ? v[4 * j + 2 * h] * rs[h] * cs[2 * j] : 0.f,
                  in ? v[4 * j + 2 * h + 1] * rs[h] * cs[2 * j + 1] : 0.f, hi, lo);
      const int gc = c + 8 * j;              // (in the piece's half of a tile)
      unsigned char* p =
          row + sw128_chunk_off(gr & 31, (gc & 63) >> 3) + 2 * (gc & 7);
      *reinterpret_cast<unsigned*>(p) = hi;
      *reinterpret_cast<unsigned*>(p + 4096) = lo;
    }
  }
}

// Exponent of the largest norm of a gradient row over its size, by a warp, eight
// rows a load (the array begins at a multiple of 256 bytes).
__device__ __forceinline__ int widest_row(const GemmDesc& g, int lane) {
  unsigned pair = 0x80008000u;           // two shorts
  const int n = g.M >> 3;
#pragma unroll 8
  for (int i = lane; i < n; i += 32) {
    const uint4 w = reinterpret_cast<const uint4*>(g.wide)[i];
    pair = __vmaxs2(__vmaxs2(__vmaxs2(pair, w.x), w.y), __vmaxs2(w.z, w.w));
  }
  int m = max((int)(short)pair, (int)(short)(pair >> 16));
  if (8 * n + lane < g.M) m = max(m, (int)g.wide[8 * n + lane]);
  m = __reduce_max_sync(0xffffffffu, m);
  return m <= kNoExp ? 0 : m;            // (a gradient of zeros)
}

// The second product's epilogue takes a 16 x 32 piece of kf through shared memory and
// has a column a lane: rows of weights, velocities and kf are read and written 128
// bytes at a time, wherever they begin, without a branch between the rows, and the
// next piece's loads come before this one's stores where a CTA has the registers.
// (A lane's values straight from the accumulators, with branches past the edges: 62
// tiles of odd sizes 25.5 us, so 16; 144 tiles of 512 x 4608 20 us either way, 47 MB
// of weights, velocities and kf.)  Bound: 32 bytes a cycle that an SM can store.
constexpr int KF_PITCH = 36;                 // floats
struct KfOld {
  float v[16], p[16];                        // velocities, weights
  int er, ec;                                // exponents: row `lane`, the column
};

// Of a lane's column, weight or bias: first row's place, and from a row to the next.
struct KfColumn {
  long long at, step;
  bool weight, live;
};
__device__ __forceinline__ KfColumn kf_column(const GemmDesc& g, int r0, int c) {
  KfColumn k;
  k.weight = c < g.dW;
  k.live = c < g.N;
  k.step = k.weight ? g.dW : 1;
  k.at = (long long)r0 * k.step + (k.weight ? c : 0);
  return k;
}

__device__ __forceinline__ void load_kf(const GemmDesc& g, int r0, int c0,
                                        int lane, KfOld& o) {
  o.er = g.re[min(r0 + (lane & 15), g.M - 1)];
  o.ec = g.ce[min(c0 + lane, g.N - 1)];
  const KfColumn k = kf_column(g, r0, c0 + lane);
  const float* v = k.weight ? g.vW : g.vb;
  const float* p = k.weight ? g.pW : g.pb;
  const bool on = g.pW != nullptr && k.live;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const bool in = on && r0 + i < g.M;
    o.v[i] = in ? v[k.at + i * k.step] : 0.f;
    o.p[i] = in ? p[k.at + i * k.step] : 0.f;
  }
}

// kf to the weight and bias parts, and the momentum update where the layer has it
// fused.  `piece`: 16 x KF_PITCH floats of this warp's own.
__device__ __forceinline__ void store_kf(const GemmDesc& g, const float v[16],
                                         float* piece, int r0, int c0, int lane,
                                         float lr, float momentum,
                                         const KfOld& o) {
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; i += 2)
    *reinterpret_cast<float2*>(&piece[((lane >> 2) + 8 * ((i >> 1) & 1)) * KF_PITCH +
                                      2 * (lane & 3) + 8 * (i >> 2)]) =
        make_float2(v[i], v[i + 1]);
  __syncwarp();
  const KfColumn k = kf_column(g, r0, c0 + lane);
  float* const okf = k.weight ? g.kfW : g.kfb;
  float* const ov = k.weight ? g.vW : g.vb;
  float* const op = k.weight ? g.pW : g.pb;
  const bool fused = g.pW != nullptr;
  // (values, then stores, each under one condition: with branches between them a
  // row took 250 cycles)
  float kf[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    kf[i] = scale_exp(piece[i * KF_PITCH + lane],
                      __shfl_sync(0xffffffffu, o.er, i) + o.ec);
  const int rows = k.live ? g.M - r0 : 0;
  auto put = [&](float* base, const float (&x)[16], int n) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < n) base[k.at + i * k.step] = x[i];
  };
  put(okf, kf, okf != nullptr ? rows : 0);
  if (!fused) return;
  float w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    kf[i] = momentum * o.v[i] - lr * kf[i];
    w[i] = o.p[i] + kf[i];
  }
  put(ov, kf, rows);
  put(op, w, rows);
}

// Sizes of the rows of gradients (see GradSizes), WARPS warps per row: as many as
// leave the launch one wave (54 layers of ResNet-50: 60 us with eight, 24 with one).
template <int WARPS>
__global__ void __launch_bounds__(256)
grad_rows_kernel(const GradSizes* __restrict__ jobs, int njobs, int rows,
                 const __grid_constant__ GradInline inl) {
  __shared__ int part[8];
  let_next_launch_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row_all = (8 / WARPS) * blockIdx.x + warp / WARPS;
  const bool live = row_all < rows;
  const GradSizes* all = inl.n > 0 ? inl.j : jobs;
  int f = 0;
  for (int i = lane; i < njobs; i += 32)
    if (all[i].row_begin <= row_all) f = i;
  f = (int)__reduce_max_sync(0xffffffffu, (unsigned)f);
  const GradSizes& job = all[f];
  const int row = row_all - job.row_begin, cols = live ? job.cols : 0;
  const float* src = job.src + (long long)row * cols;
  const int at = 32 * (warp % WARPS) + lane;
  constexpr int S = 32 * WARPS;
  int top = kNoExp;
  if (live && job.extra != nullptr && at == 0) top = exp_of(job.extra[row]);
  // (eight loads in flight; past the end the last one again)
  if ((cols & 3) == 0 && (reinterpret_cast<uintptr_t>(job.src) & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    const int n = cols >> 2;
    for (int k0 = at; k0 < n; k0 += 8 * S) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = s4[min(k0 + S * u, n - 1)];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        top = max(max(max(top, exp_of(x[u].x)), exp_of(x[u].y)),
                  max(exp_of(x[u].z), exp_of(x[u].w)));
    }
  } else {
    for (int k0 = at; k0 < cols; k0 += 8 * S) {
      float x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = src[min(k0 + S * u, cols - 1)];
#pragma unroll
      for (int u = 0; u < 8; ++u) top = max(top, exp_of(x[u]));
    }
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (WARPS > 1) {
    if (lane == 0) part[warp] = top;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WARPS; ++i)
      top = max(top, part[warp / WARPS * WARPS + i]);
  }
  if (live && at == 0) job.row[row] = (short)top;
}

// Sizes of the columns behind it, W columns per block and 1024 / W rows at a time:
// as few as leave the launch one wave (W = 8 instead of 32 for 1000 x 1000: 5 us less;
// in two waves, for 512 x 4608, 16 us instead of 6.5).
template <int W>
__global__ void __launch_bounds__(1024)
grad_cols_kernel(const GradSizes* __restrict__ jobs, int njobs,
                 const __grid_constant__ GradInline inl) {
  __shared__ int part[32][W + 1];
  let_next_launch_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GradSizes* all = inl.n > 0 ? inl.j : jobs;
  int f = 0;
  for (int i = lane; i < njobs; i += 32)
    if (all[i].col_begin <= (int)blockIdx.x) f = i;
  f = (int)__reduce_max_sync(0xffffffffu, (unsigned)f);
  const GradSizes job = all[f];
  const int c0 = W * (blockIdx.x - job.col_begin), c = c0 + lane % W;
  const bool tail = c >= job.cols;       // the appended column, or none
  const float* src = tail ? job.extra : job.src + c;
  const long long step = tail ? 1 : job.cols;
  const int total = job.cols + (job.extra != nullptr ? 1 : 0);
  int top = kNoExp;
  wait_for_launch_before();
  if (c < total) {
    constexpr int S = 1024 / W;
    for (int r0 = (32 / W) * warp + lane / W; r0 < job.rows; r0 += 8 * S) {
      float x[8];
      int e[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = min(r0 + S * u, job.rows - 1);
        x[u] = src[r * step];
        e[u] = job.row[r];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (x[u] != 0.f) top = max(top, exp_of(x[u]) - e[u]);
    }
  }
#pragma unroll
  for (int o = W; o < 32; o *= 2)
    top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (lane < W) part[warp][lane] = top;
  __syncthreads();
  if (warp >= W) return;
  top = __reduce_max_sync(0xffffffffu, part[lane][warp]);
  // (not below -126, so that the factor is a normal number; a column of zeros
  // gets that as well)
  if (lane == 0 && c0 + warp < total) job.col[c0 + warp] = (short)max(top, -126);
}

// A row by a warp: its largest value, then (the row is in the L1 cache) the
// scaled terms.  Bound by HBM: 4 bytes read and 4 written per element.
// INV (G_inv): exponents of any size (those of the gradient's columns are 126 at
// most), no norm.
template <bool INV>
__device__ __forceinline__ void pack_row(const PackRows& job, int row,
                                         int lane) {
  const int cols = job.cols;
  const int total = cols + (job.extra != nullptr ? 1 : 0);
  const float* src = job.src + (long long)row * cols;
  const bool vec =
      (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(job.src) & 15) == 0;
  auto load = [&](int k) {
    if (vec && k + 3 < cols) return *reinterpret_cast<const float4*>(src + k);
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      x[e] = k + e < cols ? src[k + e]
             : k + e < total ? job.extra[row] : 0.f;
    return make_float4(x[0], x[1], x[2], x[3]);
  };
  const int sign = job.col_sign;
  // (what stands behind the row's end is not read as an exponent)
  auto load_exp = [&](int k) {
    if (k + 3 < total) return *reinterpret_cast<const short4*>(job.col + k);
    return make_short4(k < total ? job.col[k] : 0,
                       k + 1 < total ? job.col[k + 1] : 0,
                       k + 2 < total ? job.col[k + 2] : 0, 0);
  };
  const int nkb = (total + 31) >> 5;
  unsigned char* dst = job.dst + (long long)(row >> 7) * nkb * kChunk;
  auto store = [&](int k, float y0, float y1, float y2, float y3) {
    unsigned h0, h1, l0, l1;
    split_half2(y0, y1, h0, l0);
    split_half2(y2, y3, h1, l1);
    unsigned char* p = dst + (long long)(k >> 5) * kChunk +
                       sw128_chunk_off(row & 127, (k & 31) >> 3) +
                       8 * ((k >> 2) & 1);
    *reinterpret_cast<uint2*>(p) = make_uint2(h0, h1);
    p = reinterpret_cast<unsigned char*>(reinterpret_cast<uintptr_t>(p) ^ 0x40);
    *reinterpret_cast<uint2*>(p) = make_uint2(l0, l1);
  };
  // Factors and the scaled row inside the range of fp32 with 2^60 to spare below
  // (what is left of a value under that is less than its terms hold): one
  // multiplication for the column and one for the row, and not the exponents
  // added up for every element.
  // (a gradient row of zeros: any small factor of G_inv's column does)
  const unsigned unit = (unsigned)sign << 23;
  auto factor = [&](int e) {
    if (INV) e = max(e, -126);
    return __uint_as_float(0x3f800000u + (unsigned)e * unit);
  };
  auto width = [](int e) { return e == kNoExp ? 0u : (unsigned)abs(e); };
  unsigned widest = 0;
  float peak = 0.f;
  // (four loads in flight; zeros behind the end)
#pragma unroll 1
  for (int k0 = 4 * lane; k0 < total; k0 += 512)
#pragma unroll
  for (int k = k0; k < k0 + 512; k += 128) {
    const float4 x = load(k);
    const short4 e = load_exp(k);
    if (INV)
      widest = max(max(max(widest, width(e.x)), width(e.y)),
                   max(width(e.z), width(e.w)));
    peak = fmaxf(fmaxf(peak, fmaxf(fabsf(x.x * factor(e.x)),
                                   fabsf(x.y * factor(e.y)))),
                 fmaxf(fabsf(x.z * factor(e.z)), fabsf(x.w * factor(e.w))));
  }
  if (INV) widest = __reduce_max_sync(0xffffffffu, widest);
  const unsigned bits =
      __reduce_max_sync(0xffffffffu, __float_as_uint(peak));
  int top = (int)(bits >> 23) - 127, s;
  float sum = 0.f;
  if (widest <= 126 && top >= -60 && top <= 100) {
    s = kChunkExp - top;
    const float f = __uint_as_float((unsigned)(127 + s) << 23);
#pragma unroll 1
    for (int k0 = 4 * lane; k0 < 32 * nkb; k0 += 512)
#pragma unroll
    for (int k = k0; k < k0 + 512; k += 128) {
      const float4 x = load(k);
      const short4 e = load_exp(k);
      const float y0 = x.x * factor(e.x) * f, y1 = x.y * factor(e.y) * f;
      const float y2 = x.z * factor(e.z) * f, y3 = x.w * factor(e.w) * f;
      if (!INV) sum += y0 * y0 + y1 * y1 + y2 * y2 + y3 * y3;
      if (k < 32 * nkb) store(k, y0, y1, y2, y3);
    }
  } else {
    top = 2 * kNoExp;
#pragma unroll 1
    for (int k = 4 * lane; k < total; k += 128) {
      const float4 x = load(k);
      const short4 e = load_exp(k);
      // (a zero, in the row or behind its end, counts for nothing)
      if (x.x != 0.f) top = max(top, exp_of(x.x) + sign * e.x);
      if (x.y != 0.f) top = max(top, exp_of(x.y) + sign * e.y);
      if (x.z != 0.f) top = max(top, exp_of(x.z) + sign * e.z);
      if (x.w != 0.f) top = max(top, exp_of(x.w) + sign * e.w);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (top == 2 * kNoExp) top = 0;            // a row of zeros
    s = kChunkExp - top;
#pragma unroll 1
    for (int k = 4 * lane; k < 32 * nkb; k += 128) {
      const float4 x = load(k);
      const short4 e = load_exp(k);
      const float y0 = scale_exp(x.x, s + sign * e.x);
      const float y1 = scale_exp(x.y, s + sign * e.y);
      const float y2 = scale_exp(x.z, s + sign * e.z);
      const float y3 = scale_exp(x.w, s + sign * e.w);
      if (!INV) sum += y0 * y0 + y1 * y1 + y2 * y2 + y3 * y3;
      store(k, y0, y1, y2, y3);
    }
  }
  if (INV) {
    if (lane == 0) job.exp[row] = (short)-s;
    return;
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) {
    // sum < 2^(f + 1), its root at most 2^n (rounding of the sum: far inside
    // the factor of two that fp16 has left above 2^15)
    const int n = sum == 0.f ? 0 : (exp_of(sum) + 2) >> 1;
    const int z = job.role == PACK_GRAD && sum != 0.f ? job.size[row] : 0;
    job.exp[row] = (short)(sum == 0.f ? kNoExp : n - s - z);
    job.fit[row] = job.role == PACK_GRAD ? scale_exp(1.f, -s - z)
                                         : scale_exp(job.gain, -n);
  }
}

__global__ void __launch_bounds__(256)
pack_rows_kernel(const PackRows* __restrict__ jobs, int njobs, int rows,
                 const __grid_constant__ PackInline inl) {
  const int lane = threadIdx.x & 31;
  const int row_all = blockIdx.x * 8 + (threadIdx.x >> 5);
  let_next_launch_begin();
  if (row_all >= rows) return;
  const PackRows* all = inl.n > 0 ? inl.j : jobs;
  int f = 0;
  for (int i = lane; i < njobs; i += 32)
    if (all[i].row_begin <= row_all) f = i;
  f = (int)__reduce_max_sync(0xffffffffu, (unsigned)f);
  const PackRows job = all[f];
  wait_for_launch_before();
  if (job.role != PACK_G)
    pack_row<false>(job, row_all - job.row_begin, lane);
  else
    pack_row<true>(job, row_all - job.row_begin, lane);
}

// MODE 0: the products of the inverse; 1, 2: first and second product of the
// preconditioning, uncut as a sum of TF32 terms was, with half its MMAs.
template <int MODE, int STAGES>
__global__ void __launch_bounds__(KP_THREADS, STAGES == 3 ? 2 : 1)
packed_tile_kernel(const GemmDesc* __restrict__ descs, int ndesc,
                   const __grid_constant__ TileInline inl, float plr,
                   float momentum) {
  constexpr int kSegment = MODE == 0 ? KP_SEGMENT : 1 << 20;
  constexpr int TN = 128;
  extern __shared__ unsigned char kp_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(kp_smem_raw) + 1023) & ~(uintptr_t)1023);
  PackedControl* ctl =
      reinterpret_cast<PackedControl*>(smem + STAGES * KP_STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x;

  if (warp == 0) {
    if (lane == 0) {
#pragma unroll
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&ctl->full[s], 1);
        mbar_init(&ctl->empty[s], 1);
      }
      mbar_init(&ctl->accum, 1);
      mbar_init(&ctl->drained, KP_EPI_WARPS);
      ctl->abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  } else if (warp == 1) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(2 * TN)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
  } else {
    // the problem this tile belongs to (tile_begin is ascending)
    constexpr int kWords = (int)(sizeof(GemmDesc) / sizeof(int));
    const GemmDesc* src;
    int f = 0;
    if (inl.n > 0) {
#pragma unroll
      for (int i = 1; i < TT_INLINE; ++i)
        if (i < inl.n && inl.d[i].tile_begin <= tile) f = i;
      src = &inl.d[f];
    } else {
      for (int i = lane; i < ndesc; i += 32)
        if (descs[i].tile_begin <= tile) f = i;
      f = (int)__reduce_max_sync(0xffffffffu, (unsigned)f);
      src = descs + f;
    }
    int* dst = reinterpret_cast<int*>(&ctl->desc);
    for (int i = tid - 64; i < kWords; i += 32 * KP_EPI_WARPS)
      dst[i] = reinterpret_cast<const int*>(src)[i];
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  let_next_launch_begin();
  wait_for_launch_before();

  const GemmDesc& g = ctl->desc;
  const unsigned tmem = ctl->tmem_base;
  const int flags = g.flags;
  const int lt = tile - g.tile_begin;
  int bi, bj;
  if (flags & G_LOWER) {
    tri_tile(lt, bi, bj);
  } else {
    bi = lt / g.tiles_n;
    bj = lt - bi * g.tiles_n;
  }
  const int m0 = bi * TN, n0 = bj * TN;
  const bool share_ab = (flags & G_SAME_AB) && bi == bj;
  int kbeg = 0;
  if (flags & G_KBEG_M0) kbeg = max(0, m0 - g.kbeg_off);
  if (flags & G_KBEG_N0) kbeg = max(kbeg, n0);
  const int nkb = max(0, (int)((g.K - kbeg + 31) >> 5));
  const int kb0 = kbeg >> 5, seg0 = kb0 / kSegment;

  if (warp == 0) {
    if (elect_one()) {
      const long long k0 = (long long)kb0 * kChunk;
      const unsigned char* a = g.ca + bi * g.ca_tile + k0;
      const unsigned char* b = g.cb + bj * g.cb_tile + k0;
      const unsigned bytes = share_ab ? kChunk : 2 * kChunk;
      for (int kb = 0; kb < nkb; ++kb, a += kChunk, b += kChunk) {
        const int s = kb % STAGES;
        if (kb >= STAGES &&
            !mbar_wait_status(&ctl->empty[s], ((kb / STAGES) - 1) & 1,
                              &ctl->abort_flag, &g_packed_status))
          break;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     ::"r"(smem_u32(&ctl->full[s])), "r"(bytes)
                     : "memory");
        const unsigned st = smem_u32(smem + s * KP_STAGE);
        if (!share_ab) bulk_load(st, a, &ctl->full[s]);
        bulk_load(st + kChunk, b, &ctl->full[s]);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const bool ka = g.A.kfast != 0, kb_ = g.B.kfast != 0;
      const unsigned idesc = tc_half_desc(TN, !ka, !kb_);
      // from the hi to the lo terms, and from 16 k to the next (16-byte units)
      const unsigned long long lo_a = (ka ? 64 : 4096) >> 4;
      const unsigned long long lo_b = (kb_ ? 64 : 4096) >> 4;
      const unsigned long long adv_a = (ka ? 32 : 2048) >> 4;
      const unsigned long long adv_b = (kb_ ? 32 : 2048) >> 4;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % STAGES;
        const int seg = (kb0 + kb) / kSegment - seg0;
        const bool fresh = kb == 0 || (kb0 + kb) % kSegment == 0;
        if (fresh && seg > 0 &&
            !mbar_wait_status(&ctl->drained, (seg - 1) & 1, &ctl->abort_flag,
                              &g_packed_status))
          break;
        if (!mbar_wait_status(&ctl->full[s], (kb / STAGES) & 1,
                              &ctl->abort_flag, &g_packed_status))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned sb = smem_u32(smem + s * KP_STAGE) + kChunk;
        const unsigned sa = share_ab ? sb : sb - kChunk;
        unsigned long long a = ka ? tc_smem_desc(sa) : tc_smem_desc_mn(sa, 8192);
        unsigned long long b = kb_ ? tc_smem_desc(sb) : tc_smem_desc_mn(sb, 8192);
#pragma unroll
        for (int kk = 0; kk < 2; ++kk, a += adv_a, b += adv_b) {
          const unsigned acc = !fresh || kk != 0;
          tc_mma_half(tmem + TN, a + lo_a, b, idesc, acc);
          tc_mma_half(tmem + TN, a, b + lo_b, idesc, 1);
          tc_mma_half(tmem, a, b, idesc, acc);
        }
        tc_commit(&ctl->empty[s]);
        if (kb + 1 == nkb || (kb0 + kb + 1) % kSegment == 0)
          tc_commit(&ctl->accum);
      }
    }
    __syncwarp();
  } else {
    // ===================== epilogue =====================
    // warp: accumulator rows of quarter q, 32-column pieces h and h + 2, 16 rows
    // at a time straight from the registers (8-byte words of eight rows an
    // instruction: whole 32-byte sectors)
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int rows = g.M, cols = g.N;
    const bool lower = (flags & G_LOWER) != 0;
    // (preconditioning, while the MMAs run; a register of its own for it makes the
    // second product spill: 54 layers of ResNet-50 267 us, 375 so)
    const float alpha =
        MODE == 0 ? g.alpha
                  : scale_exp(g.alpha, MODE == 1 ? -widest_row(g, lane)
                                                 : widest_row(g, lane));
    float beta = (g.beta_until > 0 && m0 >= g.beta_until) ? 0.f : g.beta;
    const float* un = g.unscale;
    const long long ldc = g.ldc;
    const bool vec = (ldc & 1) == 0 &&
                     (reinterpret_cast<uintptr_t>(g.C) & 7) == 0;
    const int lr = lane >> 2, lc = 2 * (lane & 3);
    bool ok = true;
    const int nseg = nkb > 0 ? (kb0 + nkb - 1) / kSegment - seg0 + 1 : 1;
    // The second product of a preconditioning, where a CTA has the registers: what a
    // piece reads is loaded while the piece before it (or the MMAs) runs.  The piece
    // itself goes through the stages, which the MMAs have read by then.
    constexpr bool kAhead = MODE == 2 && STAGES > 3;
    KfOld ahead;
    float* const piece =
        reinterpret_cast<float*>(smem) + (warp - 2) * 16 * KF_PITCH;
    auto load_piece = [&](int u, KfOld& o) {
      const int r0 = m0 + 32 * q + 16 * (u & 1);
      const int c0 = n0 + 32 * h + 64 * (u >> 1);
      if (r0 < rows && c0 < cols) load_kf(g, r0, c0, lane, o);
    };
    if constexpr (kAhead) load_piece(0, ahead);
    float u_rows[2][2], u_cols[2][8];
    if constexpr (MODE == 1) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        load_u(g, m0 + 32 * q + 16 * k + lr, u_rows[k]);
        load_u_columns(g, n0 + 32 * h + 64 * k + lc, u_cols[k]);
      }
    }
    // C of an inverse's product, a piece ahead: with the loads of a piece behind the
    // stores of the one before, an SM had 32 KB under way and a tile's epilogue took
    // as long as the MMAs of 512 k.
    float old_ahead[16];
    auto load_old = [&](int it) {
      const int u = it & 3;
      const int r0 = m0 + 32 * q + 16 * (u & 1);
      const int c0 = n0 + 32 * h + 64 * (u >> 1);
      if ((it < 4 ? beta : 1.f) == 0.f || r0 >= rows || c0 >= cols ||
          (lower && c0 > r0 + 15))
        return;
      const int r = r0 + lr, c = c0 + lc;
      if (vec && r0 + 16 <= rows && c0 + 32 <= cols && (!lower || c0 + 31 <= r0)) {
        const float* p = g.C + (long long)r * ldc + c;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float2 x = *reinterpret_cast<const float2*>(
              p + 8 * ((i >> 1) & 1) * ldc + 8 * (i >> 2));
          old_ahead[i] = x.x;
          old_ahead[i + 1] = x.y;
        }
      } else {
        // (past the edges the last row or column: no branch, all in flight)
        piece_each<true>(r, c, rows, cols, lower, [&](int i, int dr, int dc) {
          old_ahead[i] = g.C[(long long)min(r + dr, rows - 1) * ldc +
                             min(c + dc, cols - 1)];
        });
      }
    };
#pragma unroll 1
    for (int it = MODE == 0 ? -1 : 0; it < 4 * nseg; ++it) {
      const int u = it & 3, seg = it >> 2;
      float old[16];
      if constexpr (MODE == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) old[i] = old_ahead[i];
        if (it + 1 < 4 * nseg) load_old(it + 1);
        if (it < 0) continue;
      }
      if (it == 4) beta = 1.f;             // onto the segments before
      const int r0 = m0 + 32 * q + 16 * (u & 1);
      const int c0 = n0 + 32 * h + 64 * (u >> 1);
      // (U has zeros behind its last row up to the end of the k-block)
      const bool live = r0 < (MODE == 1 ? (rows + 31) & ~31 : rows) &&
                        c0 < cols && !(lower && c0 > r0 + 15);
      const bool whole =
          r0 + 16 <= rows && c0 + 32 <= cols && (!lower || c0 + 31 <= r0);
      const int r = r0 + lr, c = c0 + lc;
      float* p = g.C + (long long)r * ldc + c;
      KfOld kf_old;
      if constexpr (kAhead) {
        kf_old = ahead;
        if (u < 3) load_piece(u + 1, ahead);
      }
      if (u == 0 && nkb > 0) {
        ok = mbar_wait_status(&ctl->accum, seg & 1, &ctl->abort_flag,
                              &g_packed_status);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if (!ok) break;
      float v[16];
      if (nkb > 0 && live) {
        float w[16];
        const unsigned at = tmem + ((unsigned)(32 * q + 16 * (u & 1)) << 16) +
                            (unsigned)(c0 - n0);
        tc_ld_16x32(at, v);
        tc_ld_16x32(at + TN, w);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = alpha * (v[i] + w[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
      }
      if (u == 3 && seg + 1 < nseg) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->drained);
      }
      if (!live) continue;
      if constexpr (MODE == 1) {
        float rs[2], cs[8];
#pragma unroll
        for (int k = 0; k < 2; ++k) rs[k] = u & 1 ? u_rows[1][k] : u_rows[0][k];
#pragma unroll
        for (int k = 0; k < 8; ++k) cs[k] = u > 1 ? u_cols[1][k] : u_cols[0][k];
        store_u(g, v, r, c, rs, cs);
        continue;
      }
      if constexpr (MODE == 2) {
        if constexpr (!kAhead) load_piece(u, kf_old);
        store_kf(g, v, piece, r0, c0, lane, plr, momentum, kf_old);
        continue;
      }
      if (un != nullptr) {
        // (rows and columns past the matrix: inside the vector's padding)
        const float s0 = un[r], s1 = un[r + 8];
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float2 sc = *reinterpret_cast<const float2*>(&un[c + 2 * j]);
          v[j] = v[j] * s0 * sc.x;
          v[j + 1] = v[j + 1] * s0 * sc.y;
          v[j + 2] = v[j + 2] * s1 * sc.x;
          v[j + 3] = v[j + 3] * s1 * sc.y;
        }
      }
      if (beta != 0.f) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] += beta * old[i];
      }
      if (whole && vec) {
#pragma unroll
        for (int i = 0; i < 16; i += 2)
          *reinterpret_cast<float2*>(p + 8 * ((i >> 1) & 1) * ldc +
                                     8 * (i >> 2)) =
              make_float2(v[i], v[i + 1]);
      } else {
        piece_each<false>(r, c, rows, cols, lower, [&](int i, int dr, int dc) {
          p[dr * ldc + dc] = v[i];
        });
      }
      if (flags & G_MIRROR) {
        float* t = g.C + (long long)c * ldc + r;
        if (whole)
          piece_each<true>(r, c, rows, cols, lower, [&](int i, int dr, int dc) {
            t[dc * ldc + dr] = v[i];
          });
        else
          piece_each<false>(r, c, rows, cols, lower, [&](int i, int dr, int dc) {
            t[dc * ldc + dr] = v[i];
          });
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) tc_release(tmem, 2 * TN, ctl->abort_flag != 0);
}

// ------------------------------------------------------------------ host side
struct PackedVariant {
  void (*kernel)(const GemmDesc*, int, const TileInline, float, float);
  int stages;
};
// by mode; the preconditioning also with one CTA an SM
static const PackedVariant kPackedVariants[] = {{packed_tile_kernel<0, 3>, 3},
                                                {packed_tile_kernel<1, 3>, 3},
                                                {packed_tile_kernel<2, 3>, 3},
                                                {packed_tile_kernel<1, 6>, 6},
                                                {packed_tile_kernel<2, 6>, 6}};

int packed_prepare() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  KFAC_CUDA(cudaGetDevice(&dev));
  KFAC_REQUIRE(dev >= 0 && dev < 64, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    for (const PackedVariant& v : kPackedVariants)
      KFAC_CUDA(cudaFuncSetAttribute(
          v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
          packed_smem(v.stages)));
    done[dev] = true;
  }
  return KFAC_OK;
}

int packed_number_tiles(GemmDesc* descs, int n) {
  int total = 0;
  for (int i = 0; i < n; ++i) {
    GemmDesc& g = descs[i];
    const int tm = (g.M + TC_BM - 1) / TC_BM, tn = (g.N + TC_BM - 1) / TC_BM;
    g.tile_begin = total;
    g.tiles_m = tm;
    g.tiles_n = tn;
    total += (g.flags & G_LOWER) ? tm * (tm + 1) / 2 : tm * tn;
  }
  return total;
}

static int launch_mode(int mode, const GemmDesc* descs_dev,
                       const GemmDesc* descs_host, int ndesc, int total_tiles,
                       float lr, float momentum, cudaStream_t stream) {
  if (ndesc <= 0 || total_tiles <= 0) return KFAC_OK;
  const int rc = packed_prepare();
  if (rc != KFAC_OK) return rc;
  TileInline inl;
  inl.n = 0;
  if (ndesc <= TT_INLINE) {
    inl.n = ndesc;
    std::copy(descs_host, descs_host + ndesc, inl.d);
  }
  const bool one = mode > 0 && total_tiles <= sm_count();
  const PackedVariant& v = kPackedVariants[one ? mode + 2 : mode];
  return launch_behind("packed_tile_kernel", mode > 0, v.kernel, total_tiles,
                       KP_THREADS, packed_smem(v.stages), stream, descs_dev,
                       ndesc, inl, lr, momentum);
}

int launch_packed(const GemmDesc* descs_dev, const GemmDesc* descs_host,
                  int ndesc, int total_tiles, cudaStream_t stream) {
  return launch_mode(0, descs_dev, descs_host, ndesc, total_tiles, 0.f, 0.f,
                     stream);
}

int launch_packed_precond(const GemmDesc* descs_dev, const GemmDesc* descs_host,
                          int ndesc, int total_tiles, bool last, float lr,
                          float momentum, cudaStream_t stream) {
  return launch_mode(last ? 2 : 1, descs_dev, descs_host, ndesc, total_tiles, lr,
                     momentum, stream);
}

int grad_group_columns(const int* cols, int n) {
  for (int w = 8; w < 32; w *= 2) {
    long long groups = 0;
    for (int i = 0; i < n; ++i) groups += (cols[i] + w - 1) / w;
    if (groups <= 2 * sm_count()) return w;      // (two blocks an SM)
  }
  return 32;
}

int launch_grad_sizes(const GradSizes* jobs_dev, const GradSizes* jobs_host,
                      int njobs, int rows, int groups, int columns,
                      cudaStream_t stream) {
  if (njobs <= 0 || rows <= 0) return KFAC_OK;
  GradInline inl;
  inl.n = 0;
  if (njobs <= TT_INLINE) {
    inl.n = njobs;
    std::copy(jobs_host, jobs_host + njobs, inl.j);
  }
  int warps = 8;                                 // (eight blocks an SM)
  while (warps > 1 && ceil_div((int64_t)rows * warps, 8) > 8 * sm_count())
    warps /= 2;
  auto* by_rows = warps == 8   ? grad_rows_kernel<8>
                  : warps == 4 ? grad_rows_kernel<4>
                  : warps == 2 ? grad_rows_kernel<2>
                               : grad_rows_kernel<1>;
  const int rc = launch_behind("grad_rows_kernel", false, by_rows,
                               ceil_div((int64_t)rows * warps, 8), 256, 0, stream,
                               jobs_dev, njobs, rows, inl);
  if (rc != KFAC_OK) return rc;
  auto* by_cols = columns == 8    ? grad_cols_kernel<8>
                  : columns == 16 ? grad_cols_kernel<16>
                                  : grad_cols_kernel<32>;
  return launch_behind("grad_cols_kernel", true, by_cols, groups, 1024, 0, stream,
                       jobs_dev, njobs, inl);
}

int launch_pack_rows(const PackRows* jobs_dev, const PackRows* jobs_host,
                     int njobs, int rows, cudaStream_t stream) {
  if (njobs <= 0 || rows <= 0) return KFAC_OK;
  PackInline inl;
  inl.n = 0;
  if (njobs <= 3 * TT_INLINE) {
    inl.n = njobs;
    std::copy(jobs_host, jobs_host + njobs, inl.j);
  }
  return launch_behind("pack_rows_kernel", true, pack_rows_kernel,
                       (int)ceil_div(rows, 8), 256, 0, stream, jobs_dev, njobs,
                       rows, inl);
}

int packed_status_read(int* out) {
  KFAC_CUDA(cudaMemcpyFromSymbol(out, g_packed_status, sizeof(int)));
  return KFAC_OK;
}

}  // namespace kfac
