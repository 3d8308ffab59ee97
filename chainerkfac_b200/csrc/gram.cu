// Factor builds out = alpha X^T X + beta out from staged operands.
//
// Every operand X (rows x columns, in whatever layout the caller holds it) is
// first written once as two bf16 planes, hi and lo with x = hi + lo, rows
// contiguous along the columns (stage_cols_kernel, stage_rows_kernel; HBM-bound).
// The products then need no producer warps: TMA copies 32 rows x 64 columns of
// both planes (8 KB) per instruction straight into the 128-byte-swizzled,
// MN-major operand layout of tcgen05.mma, with zeros past the last column.
// The in-kernel gather that this replaces spent four issue slots per clock on
// addresses, loads and splits and held the tensor cores at 39 % of the bf16
// rate (factors of ResNet-50, 32 images, NCHW: 3790 us in its two launches).
//
// Stride-1 3 x 3 convolutions ("same" padding) do not multiply patches at
// all.  The block of taps (ti, tj) of the patch factor is
//   sum over output positions p of x[c, p + ti] x[c', p + tj],
// and but for the image border it depends on the offset s = tj - ti alone:
// R(s) = sum_q x[c, q] x[c', q + s], 13 offsets up to symmetry instead of 45
// tap pairs.  With rows of the plane on a grid with two zero columns and two
// zero rows behind every image, x[., q + s] is the same plane shifted by a
// number of rows, so R(s) is an ordinary product of the plane with itself,
// and any shift is a legal TMA coordinate.  What R(s) has too much are the
// positions p outside the output: p_y = -1 when both taps look one row down
// (ti_y = tj_y = +1; then q_y = 0), p_y = H when both look up (q_y = H - 1),
// the same along x, and the corner pixel counted twice when both apply:
//   block(ti, tj) = R(s) - Row(ti_y = tj_y)(s_x) - Col(ti_x = tj_x)(s_y)
//                   + Corner.
// The border rows, columns and corners are staged as further rows of the plane
// (two zeros behind every line), their products are short contractions.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "gemm_simt.cuh"
#include "tc_common.cuh"

namespace kfac {

// Whether the products of an operand can be formed without staged planes
// (direct_kernel): no appended column, 16-byte pitches and addresses; with the
// rows contiguous one tile wide only, and images of 32 rows at least (a block
// of 32 rows never spans two of them; a factor built on its own, whose
// workspace is asked for without the image size, does not come here).
bool gram_direct_job(const FactorJob& job) {
  const Operand& X = job.X;
  if (X.mode != 0 || X.extra_idx >= 0 || X.ncols != job.d) return false;
  if (reinterpret_cast<uintptr_t>(X.base) & 15) return false;
  if (X.s_col == 1 && X.period == 1) return X.s_outer % 4 == 0;
  if (!job.grouped || job.d > 256 || X.s_col % 4 != 0) return false;
  if (X.period == 1) return X.s_outer == 1;
  return X.s_inner == 1 && X.period >= 32 && X.period % 4 == 0 &&
         X.s_col == X.period && X.s_outer == X.s_col * X.ncols &&
         job.rows % X.period == 0;
}

// Shifted products pay once the channels fill a good part of a granule; a
// narrower convolution has few columns, and its patches are small too.  Images
// of two rows or columns are mostly border: the zeros around them are more rows
// than they have pixels, and a block of the factor is the small difference of
// large sums (exact zeros came out as 2e-5 of the diagonal).  Below 384 pixels in
// all, the nine groups of products cost more than they save.  us for four factors
// alike, shifted and from patches, 64 and 512 channels:
//   128 images 1x1 55 45, 344 234; 2x2 59 60, 394 323; 3x3 60 68, 460 464;
//   32 images 3x3 58 52, 318 273; 4x4 55 59, 332 325; 7x7 58 71, 417 558;
//   8 images 5x5 52 50, 292 259; 7x7 56 56, 307 303; 14x14 56 71, 384 559.
bool gram_grid_job(const FactorJob& job) {
  const Operand& X = job.X;
  return X.mode == 1 && X.ks == 3 && X.st == 1 && X.pd == 1 &&
         X.extra_idx < 0 && X.C >= 32 && job.rows >= 384 &&
         (long long)(X.H + 2) * (X.W + 2) <= 3LL * X.H * X.W;
}

namespace {

constexpr int GR_BK = 32;                          // rows per stage
constexpr int GR_GRAN = 64;                        // columns per TMA box
constexpr int GR_BOX = GR_BK * GR_GRAN * 2;        // one plane of a box
constexpr int GR_GBYTES = 2 * GR_BOX;              // hi and lo
constexpr int GR_SIDE = 4 * GR_GBYTES;             // 256 columns
constexpr int GR_STAGE = 2 * GR_SIDE;              // 64 KB
constexpr int GR_STAGES = 3;
constexpr int GR_THREADS = 256;
constexpr int GR_TILE = 256 * 256;                 // floats of a partial tile
constexpr int GR_SHIFTS = 13;

// Products of one contraction range of one operand: A granules (64 columns)
// against B granules.
struct GramGroup {
  const void* tmap;
  float* partial;      // [split][tile][column / 4][row][4]
  int row0;            // first plane row
  int nkb;             // k-blocks of 32 rows
  int kb_split;        // k-blocks per split
  int tiles;           // 256 x 256 tiles
  int unit_begin;      // first CTA
  int nga, ngb;        // granules; ngb == 0: lower tiles of X^T X
  int cg;              // column granules of the plane: B granule j holds
                       // columns 64 (j % cg) shifted by shift[j / cg] rows
  int d;               // columns of the plane
  int ashift[2];       // A granule i: columns 64 i, or (cg == 1) shifted rows
  int shift[GR_SHIFTS];
};

struct GrControl {
  GramGroup g;
  unsigned long long full[GR_STAGES];
  unsigned long long empty[GR_STAGES];
  unsigned long long accum;
  unsigned tmem_base;
  volatile int abort_flag;
  int found;
};

constexpr int GR_SMEM =
    GR_STAGES * GR_STAGE + ((int)sizeof(GrControl) + 1023) / 1024 * 1024 + 1024;
static_assert(GR_SMEM <= 227 * 1024, "gram kernel shared memory");

__device__ int g_gram_status;

// MN-major, 128-byte swizzle: 64 columns per 128-byte row of one k; groups of
// 8 k are 1024 bytes apart, the next 64 columns one granule further.
__device__ __forceinline__ unsigned long long gr_desc(unsigned addr) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFF) >> 4);
  d |= (unsigned long long)(GR_GBYTES >> 4) << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  d |= (unsigned long long)2 << 61;
  return d;
}

__device__ __forceinline__ unsigned gr_idesc(int n) {
  // D = f32, A = B = bf16, both MN-major, M = 128, N = n
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
         ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}

__device__ __forceinline__ void gr_mma(unsigned tmem_d, unsigned long long da,
                                       unsigned long long db, unsigned idesc,
                                       unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void gr_load(unsigned dst, const void* tmap, int x,
                                        int y, int z, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::"
      "complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

__host__ __device__ __forceinline__ void tri_of(int t, int& i, int& j) {
  i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  j = t - i * (i + 1) / 2;
}

// Accumulator columns c0, c0 + 1, .. of a warp's 32 rows to its partial tile,
// 32 columns at a time (columns up to the next multiple of 16 past `cend` may
// be stored as well: they exist in the tile and nobody reads them).
__device__ __forceinline__ void store_partial(unsigned taddr, float* p, int c0,
                                              int cend, int step) {
  for (; c0 < cend; c0 += step) {
    float v[16], w[16];
    tc_ld16_pair(taddr + c0, taddr + c0 + 16, v, w);
    float* q = p + (long long)(c0 >> 2) * 1024;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *reinterpret_cast<float4*>(q + i * 1024) =
          make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      *reinterpret_cast<float4*>(q + (4 + i) * 1024) =
          make_float4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    }
  }
}

// One tile of up to 256 x 256 (two 128-row accumulators in tensor memory) over
// one split of the contraction.  Bound by the tensor cores: 12 MMAs of 128 x
// 256 x 16 (1536 cycles) per 64 KB stage.  Warp 0 issues the copies, warp 1
// the MMAs; all eight warps store the accumulators, four consecutive columns
// per thread and rows along the lanes (512 contiguous bytes per instruction).
__global__ void __launch_bounds__(GR_THREADS, 1)
gram_kernel(const GramGroup* __restrict__ groups, int ngroups) {
  extern __shared__ unsigned char gr_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(gr_smem_raw) + 1023) & ~(uintptr_t)1023);
  GrControl* ctl = reinterpret_cast<GrControl*>(smem + GR_STAGES * GR_STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int unit = blockIdx.x;
  for (int i = tid; i < ngroups; i += GR_THREADS) {
    const int lo = groups[i].unit_begin;
    const int hi = i + 1 < ngroups ? groups[i + 1].unit_begin : 0x7fffffff;
    if (lo <= unit && unit < hi) ctl->found = i;
  }
  __syncthreads();
  {
    const int* s = reinterpret_cast<const int*>(groups + ctl->found);
    int* d = reinterpret_cast<int*>(&ctl->g);
    for (int i = tid; i < (int)(sizeof(GramGroup) / sizeof(int));
         i += GR_THREADS)
      d[i] = s[i];
  }
  if (tid == 0) {
    for (int s = 0; s < GR_STAGES; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->accum, 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(512)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const GramGroup& g = ctl->g;
  const unsigned tmem = ctl->tmem_base;
  const int local = unit - g.unit_begin;
  const int split = local / g.tiles, tile = local - split * g.tiles;
  int ti, tj;
  if (g.ngb == 0) {
    tri_of(tile, ti, tj);
  } else {
    const int tb = (g.ngb + 3) >> 2;
    ti = tile / tb;
    tj = tile - ti * tb;
  }
  const bool sym = g.ngb == 0;
  const bool share = sym && ti == tj;
  const int na = min(4, g.nga - 4 * ti);
  const int nb = min(4, (sym ? g.nga : g.ngb) - 4 * tj);
  const int kb0 = split * g.kb_split;
  const int nkb = min(g.kb_split, g.nkb - kb0);
  // columns of B that exist (the last granule of a plain operand is cut)
  const int nvalid = sym ? min(64 * nb, ((g.d - 256 * tj) + 15) & ~15) : 64 * nb;

  if (warp == 0) {
    if (elect_one()) {
      // the tensor maps were written by a copy that precedes this launch
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;"
                   ::"l"(g.tmap) : "memory");
      const unsigned bytes = (unsigned)((share ? 0 : na) + nb) * GR_GBYTES;
      const int la = share ? 0 : na;
      int ax[4], ay[4], bx[4], by[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int ga = 4 * ti + i, gb = 4 * tj + i;
        const bool taps = !sym && g.cg == 1;
        ax[i] = taps ? 0 : GR_GRAN * ga;
        ay[i] = taps && i < 2 ? g.ashift[i] : 0;
        bx[i] = sym ? GR_GRAN * gb : GR_GRAN * (gb % g.cg);
        by[i] = sym || i >= nb ? 0 : g.shift[gb / g.cg];
      }
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % GR_STAGES;
        if (kb >= GR_STAGES &&
            !mbar_wait_status(&ctl->empty[s], ((kb / GR_STAGES) - 1) & 1,
                              &ctl->abort_flag, &g_gram_status))
          break;
        const unsigned bar = smem_u32(&ctl->full[s]);
        asm volatile(
            "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
            ::"r"(bar), "r"(bytes) : "memory");
        const unsigned st = smem_u32(smem + s * GR_STAGE);
        const int r = g.row0 + (kb0 + kb) * GR_BK;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < nb)
            gr_load(st + GR_SIDE + i * GR_GBYTES, g.tmap, bx[i], r + by[i], 0,
                    bar);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < la)
            gr_load(st + i * GR_GBYTES, g.tmap, ax[i], r + ay[i], 0, bar);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      // a diagonal tile needs columns 0..127 only for its first 128 rows
      const unsigned id0 = gr_idesc(share ? min(nvalid, 128) : nvalid);
      const unsigned id1 = gr_idesc(nvalid);
      const bool two = na > 2;
      const unsigned a_off = share ? (unsigned)GR_SIDE : 0u;
      const unsigned long long up = 2 * GR_GBYTES >> 4;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % GR_STAGES;
        if (!mbar_wait_status(&ctl->full[s], (kb / GR_STAGES) & 1,
                              &ctl->abort_flag, &g_gram_status))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned sa = smem_u32(smem + s * GR_STAGE);
        const unsigned long long a_hi = gr_desc(sa + a_off);
        const unsigned long long a_lo = gr_desc(sa + a_off + GR_BOX);
        const unsigned long long b_hi = gr_desc(sa + GR_SIDE);
        const unsigned long long b_lo = gr_desc(sa + GR_SIDE + GR_BOX);
#pragma unroll
        for (int kk = 0; kk < GR_BK / 16; ++kk) {
          const unsigned long long adv = (unsigned long long)(kk * 2048 >> 4);
          const unsigned acc = (kb | kk) != 0;
          gr_mma(tmem, a_lo + adv, b_hi + adv, id0, acc);
          gr_mma(tmem, a_hi + adv, b_lo + adv, id0, 1);
          gr_mma(tmem, a_hi + adv, b_hi + adv, id0, 1);
          if (two) {
            gr_mma(tmem + 256, a_lo + up + adv, b_hi + adv, id1, acc);
            gr_mma(tmem + 256, a_hi + up + adv, b_lo + adv, id1, 1);
            gr_mma(tmem + 256, a_hi + up + adv, b_hi + adv, id1, 1);
          }
        }
        tc_commit(&ctl->empty[s]);
      }
      tc_commit(&ctl->accum);
    }
    __syncwarp();
  }
  // epilogue: warp w holds accumulator rows 128 (w / 4) + 32 (w % 4) + lane
  bool ok = mbar_wait_status(&ctl->accum, 0, &ctl->abort_flag, &g_gram_status);
  ok = __all_sync(0xffffffffu, ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  {
    const int h = warp >> 2, q = warp & 3;
    const int row = 128 * h + 32 * q + lane;
    const int rows = sym ? min(64 * na, g.d - 256 * ti) : 64 * na;
    const int cend = share && h == 0 ? min(nvalid, 128) : nvalid;
    if (ok && 128 * h + 32 * q < rows) {
      float* p = g.partial +
                 ((long long)split * g.tiles + tile) * GR_TILE + row * 4;
      store_partial(tmem + ((unsigned)(32 * q) << 16) + (unsigned)(256 * h), p,
                    0, cend, 32);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) tc_release(tmem, 512, ctl->abort_flag != 0);
}

// ---------------------------------------------------- products without planes
// Plain operands whose rows TMA can read as they are (16-byte pitches and
// addresses).  32 KB of fp32 per stage arrive by TMA, sixteen warps split them
// into the two bf16 planes of the MMA operands, so an element is read from
// memory once per tile and never staged.  Up to 256 columns there is one tile
// per split and the kernel is bound by HBM (96 KB in flight per SM); wider
// factors are bound by the tensor cores and the shared-memory traffic of the
// split.  us per factor, eight in a group (the gather kernel with one k-block
// of loads in flight before): 100 352 x 64 36 -> 10, 100 352 x 256 52 -> 28,
// 25 088 x 512 40 -> 30, 6272 x 1024 41 -> 30, 1568 x 2048 57 -> 28.
//
// Columns contiguous (rows x d): a granule is R rows of 64 columns, MN-major.
// Rows contiguous (KM; n x d x hw, up to 256 columns): sub-blocks of `width`
// columns x 32 rows, K-major with 64-byte swizzle.
constexpr int DR_RAW = 32768;          // fp32 bytes of a stage = bytes of planes
// Two sets of split warps take turns; every slot of either ring belongs to one
// set for good, so that a set waits on each use of its barriers (a wait by
// parity that skips a use may take an older phase for the one it wants).
constexpr int DR_RAWS = 4;             // fp32 slots (2 and 4: 8 % slower)
constexpr int DR_PLANES = 2;           // slots of split planes
static_assert(DR_RAWS % 2 == 0 && DR_PLANES % 2 == 0, "two sets of warps");
constexpr int DR_SPLIT = 16;           // split / epilogue warps
constexpr int DR_THREADS = 32 * (DR_SPLIT + 2);   // and one each: TMA, MMA

struct DirectGroup {
  const void* tmap;
  float* partial;
  int nkb;             // k-blocks of 32 rows
  int kb_split;        // per split: whole stages
  int tiles;
  int unit_begin;
  int d;
  int width;           // columns of a tile side: 64, 128, 256
  int box_rows;        // rows of a TMA box
  int per_image;       // KM: k-blocks of 32 rows per image
};

struct DrControl {
  DirectGroup g;
  unsigned long long raw_full[DR_RAWS], raw_empty[DR_RAWS];
  unsigned long long full[DR_PLANES], empty[DR_PLANES];
  unsigned long long accum;
  unsigned tmem_base;
  volatile int abort_flag;
  int found;
};

// (planes first: a 128-row operand of a 64-column tile reads past its planes,
// into rows of the accumulator that nobody uses)
constexpr int DR_SMEM =
    (DR_RAWS + DR_PLANES) * DR_RAW + ((int)sizeof(DrControl) + 1023) / 1024 * 1024 + 1024;
static_assert(DR_SMEM <= 227 * 1024, "direct kernel shared memory");

__device__ __forceinline__ unsigned long long dr_desc(unsigned addr, int lbo,
                                                      int sbo, int swizzle) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFF) >> 4);
  d |= (unsigned long long)(lbo >> 4) << 16;
  d |= (unsigned long long)(sbo >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  d |= (unsigned long long)swizzle << 61;
  return d;
}

template <bool KM>
__global__ void __launch_bounds__(DR_THREADS, 1)
direct_kernel(const DirectGroup* __restrict__ groups, int ngroups) {
  extern __shared__ unsigned char gr_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(gr_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* raw = smem + DR_PLANES * DR_RAW;
  DrControl* ctl =
      reinterpret_cast<DrControl*>(raw + DR_RAWS * DR_RAW);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int unit = blockIdx.x;
  for (int i = tid; i < ngroups; i += DR_THREADS) {
    const int lo = groups[i].unit_begin;
    const int hi = i + 1 < ngroups ? groups[i + 1].unit_begin : 0x7fffffff;
    if (lo <= unit && unit < hi) ctl->found = i;
  }
  __syncthreads();
  {
    const int* s = reinterpret_cast<const int*>(groups + ctl->found);
    int* d = reinterpret_cast<int*>(&ctl->g);
    for (int i = tid; i < (int)(sizeof(DirectGroup) / sizeof(int));
         i += DR_THREADS)
      d[i] = s[i];
  }
  if (tid == 0) {
    for (int s = 0; s < DR_RAWS; ++s) {
      mbar_init(&ctl->raw_full[s], 1);
      mbar_init(&ctl->raw_empty[s], 8);
    }
    for (int s = 0; s < DR_PLANES; ++s) {
      mbar_init(&ctl->full[s], 8);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->accum, 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == DR_SPLIT + 1) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(512)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const DirectGroup& g = ctl->g;
  const unsigned tmem = ctl->tmem_base;
  const int local = unit - g.unit_begin;
  const int split = local / g.tiles, tile = local - split * g.tiles;
  int ti, tj;
  tri_of(tile, ti, tj);
  const bool share = ti == tj;
  const int width = g.width;
  // rows of a stage: 32 KB of one side, or of both
  const int R = share ? 8192 / width : 16;
  const int row0 = split * g.kb_split * 32;
  const int nst =
      (min(g.kb_split, g.nkb - split * g.kb_split) * 32 + R - 1) / R;
  const int nvalid = min(width, (g.d - 256 * tj + 15) & ~15);
  const bool two = g.d - 256 * ti > 128;

  if (warp == DR_SPLIT) {
    if (elect_one()) {
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;"
                   ::"l"(g.tmap) : "memory");
      for (int st = 0; st < nst; ++st) {
        const int s = st % DR_RAWS;
        if (st >= DR_RAWS &&
            !mbar_wait_status(&ctl->raw_empty[s], ((st / DR_RAWS) - 1) & 1,
                              &ctl->abort_flag, &g_gram_status))
          break;
        const unsigned bar = smem_u32(&ctl->raw_full[s]);
        asm volatile(
            "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
            ::"r"(bar), "r"(DR_RAW) : "memory");
        unsigned dst = smem_u32(raw + s * DR_RAW);
        if (KM) {
          // sub-blocks of 32 rows (of one image each; past the end of an
          // image or of the operand: zeros)
          const int sub = 256 / width;
          for (int q = 0; q < sub; ++q, dst += width * 128) {
            const int b = (row0 >> 5) + st * sub + q;
            const int img = b / g.per_image;
            gr_load(dst, g.tmap, 32 * (b - img * g.per_image), 0, img, bar);
          }
        } else if (share) {
          const int r = row0 + st * R;
          for (int c = 0; c < width; c += 64)
            for (int q = 0; q < R; q += g.box_rows, dst += g.box_rows * 256)
              gr_load(dst, g.tmap, 256 * tj + c, r + q, 0, bar);
        } else {
          const int r = row0 + st * 16;
          for (int c = 0; c < 512; c += 64, dst += 16 * 256)
            gr_load(dst, g.tmap, c < 256 ? 256 * ti + c : 256 * (tj - 1) + c,
                     r, 0, bar);
        }
      }
    }
    __syncwarp();
  } else if (warp == DR_SPLIT + 1) {
    if (elect_one()) {
      const unsigned major = KM ? 0u : (1u << 15) | (1u << 16);
      const unsigned base = (1u << 4) | (1u << 7) | (1u << 10) | major |
                            ((unsigned)(128 >> 4) << 24);
      const unsigned id1 = base | ((unsigned)(nvalid >> 3) << 17);
      const unsigned id0 =
          base | ((unsigned)((share ? min(nvalid, 128) : nvalid) >> 3) << 17);
      // bytes of a plane of one granule (or sub-block); the descriptors of a
      // stage differ by their start address (16-byte units) alone
      const int plane = KM ? width * 64 : R * 128;
      const unsigned long long lo = plane >> 4;
      const unsigned long long to_b = share ? 0 : 8 * plane >> 4;
      const unsigned long long up = (KM ? 128 * 64 : 4 * plane) >> 4;
      const unsigned long long first =
          dr_desc(smem_u32(smem), KM ? 16 : (width == 64 ? 0 : 2 * plane),
                  KM ? 512 : 1024, KM ? 4 : 2);
      // k steps of 16 rows: KM: two per sub-block of 2 * plane bytes
      const unsigned long long odd = (KM ? 32 : 2048) >> 4;
      const unsigned long long even = (KM ? 2 * plane - 32 : 2048) >> 4;
      const int steps = KM ? 2 * (256 / width) : R / 16;
      for (int st = 0; st < nst; ++st) {
        const int s = st % DR_PLANES;
        if (!mbar_wait_status(&ctl->full[s], (st / DR_PLANES) & 1,
                              &ctl->abort_flag, &g_gram_status))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        unsigned long long a = first + (s * DR_RAW >> 4);
        unsigned acc = st != 0;
#pragma unroll 1
        for (int kk = 0; kk < steps; ++kk) {
          const unsigned long long bb = a + to_b;
          gr_mma(tmem, a + lo, bb, id0, acc);
          gr_mma(tmem, a, bb + lo, id0, 1);
          gr_mma(tmem, a, bb, id0, 1);
          if (two) {
            gr_mma(tmem + 256, a + up + lo, bb, id1, acc);
            gr_mma(tmem + 256, a + up, bb + lo, id1, 1);
            gr_mma(tmem + 256, a + up, bb, id1, 1);
          }
          acc = 1;
          a += (kk & 1) ? even : odd;
        }
        tc_commit(&ctl->empty[s]);
      }
      tc_commit(&ctl->accum);
    }
    __syncwarp();
  } else {
    // split: eight warps share a stage and two sets of them take turns (one
    // set needs 3000 cycles from the arrival of a stage to its hand-over).  A
    // thread turns 8 consecutive values into 16 bytes of each plane, four
    // times per stage.  The two halves are read in an order that keeps the
    // lanes of a quarter warp on different banks.
    const int tid = threadIdx.x & 255;
    const int rows = KM ? width : R;       // rows of one plane
    const int sub = KM ? 64 : 128;         // bytes of a plane row
    const int chunk = KM ? tid & 3 : tid & 7;
    unsigned src[4], dst[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int F = (KM ? tid >> 2 : tid >> 3) + (KM ? 64 : 32) * i;
      const int blk = F / rows, r = F - blk * rows;
      src[i] = F * (KM ? 128 : 256) + chunk * 32;
      dst[i] = blk * 2 * rows * sub + r * sub +
               ((KM ? chunk ^ ((r >> 1) & 3) : chunk ^ (r & 7)) << 4);
    }
    const int lo = rows * sub;
    const int h = KM ? (tid >> 2) & 1 : chunk >> 2;
    for (int st = warp >> 3; st < nst; st += 2) {
      const int s = st % DR_RAWS, ps = st % DR_PLANES;
      if (!mbar_wait_status(&ctl->raw_full[s], (st / DR_RAWS) & 1,
                            &ctl->abort_flag, &g_gram_status))
        break;
      const unsigned char* p = raw + s * DR_RAW;
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float4*>(p + src[i] + 16 * h);
        b[i] = *reinterpret_cast<const float4*>(p + src[i] + 16 * (1 - h));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->raw_empty[s]);
      if (st >= DR_PLANES &&
          !mbar_wait_status(&ctl->empty[ps], ((st / DR_PLANES) - 1) & 1,
                            &ctl->abort_flag, &g_gram_status))
        break;
      unsigned char* q = smem + ps * DR_RAW;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        unsigned hi[4], l[4];
        split_bf16x2(a[i].x, a[i].y, hi[0], l[0]);
        split_bf16x2(a[i].z, a[i].w, hi[1], l[1]);
        split_bf16x2(b[i].x, b[i].y, hi[2], l[2]);
        split_bf16x2(b[i].z, b[i].w, hi[3], l[3]);
        *reinterpret_cast<uint4*>(q + dst[i]) =
            h ? make_uint4(hi[2], hi[3], hi[0], hi[1])
              : make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(q + dst[i] + lo) =
            h ? make_uint4(l[2], l[3], l[0], l[1])
              : make_uint4(l[0], l[1], l[2], l[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->full[ps]);
    }
    // epilogue, as in gram_kernel
    bool ok =
        mbar_wait_status(&ctl->accum, 0, &ctl->abort_flag, &g_gram_status);
    ok = __all_sync(0xffffffffu, ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int hh = (warp >> 2) & 1, q = warp & 3;
    const int row = 128 * hh + 32 * q + lane;
    const int cend = share && hh == 0 ? min(nvalid, 128) : nvalid;
    if (ok && 128 * hh + 32 * q < g.d - 256 * ti) {
      float* p = g.partial +
                 ((long long)split * g.tiles + tile) * GR_TILE + row * 4;
      store_partial(tmem + ((unsigned)(32 * q) << 16) + (unsigned)(256 * hh), p,
                    32 * (warp >> 3), cend, 64);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == DR_SPLIT + 1) tc_release(tmem, 512, ctl->abort_flag != 0);
}

// ------------------------------------------------------------------- staging
enum { kSrcStrided = 0, kSrcPatches = 1, kSrcGrid = 2 };

struct StageJob {
  const float* base;
  const float* extra;          // values of the appended column (null: ones)
  unsigned short* hi;          // bf16 bit patterns; lo `plane` elements on
  long long plane;
  long long K;                 // rows of the operand (plane rows: prows)
  int prows;
  int cp, d, ncols, extra_idx; // pitch, columns, stored columns, appended one
  int kind, vec;
  long long s_outer, s_inner, s_col;
  int period;
  int n, C, H, W, ks, st, pd, Ho, Wo, nhwc;
  int line[8];                 // grid: first rows of top, bottom, left, right
                               // lines and of the four corners
  int cblocks;
  int item_begin;
};

constexpr int kStageJobs = 512;
constexpr int kStageRowsC = 128;   // rows per item, columns contiguous
constexpr int kStageRowsK = 64;    // rows per item, rows contiguous

__device__ __forceinline__ void gr_store8(const StageJob& j, int row, int col,
                                          const float v[8]) {
  unsigned h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split_bf16x2(v[2 * i], v[2 * i + 1], h[i], l[i]);
  unsigned short* p = j.hi + (long long)row * j.cp + col;
  *reinterpret_cast<uint4*>(p) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(p + j.plane) = make_uint4(l[0], l[1], l[2], l[3]);
}

// Source of one plane row: offset of its first column, and for patches the
// position of the first tap.  off < 0: a row of zeros.
struct RowSrc {
  long long off;
  int iy, ix;
};

__device__ __forceinline__ RowSrc row_source(const StageJob& j, int r) {
  RowSrc s = {-1, 0, 0};
  if (j.kind == kSrcStrided) {
    if (r < j.K) {
      if (j.period == 1) {
        s.off = (long long)r * j.s_outer;
      } else {
        const int q = r / j.period;
        s.off = q * j.s_outer + (long long)(r - q * j.period) * j.s_inner;
      }
    }
    return s;
  }
  if (j.kind == kSrcPatches) {
    if (r < j.K) {
      const int hw = j.Ho * j.Wo;
      const int n = r / hw, rem = r - n * hw;
      const int oy = rem / j.Wo;
      s.iy = oy * j.st - j.pd;
      s.ix = (rem - oy * j.Wo) * j.st - j.pd;
      s.off = (long long)n * j.C * j.H * j.W;
    }
    return s;
  }
  int n, y, x;
  if (r < j.line[0]) {                   // images, behind one row of zeros
    if (r == 0) return s;
    const int per = (j.H + 2) * (j.W + 2);
    n = (r - 1) / per;
    const int rem = r - 1 - n * per;
    y = rem / (j.W + 2);
    x = rem - y * (j.W + 2);
  } else if (r < j.line[2]) {            // top, bottom
    const int f = r - (r < j.line[1] ? j.line[0] + 1 : j.line[1]);
    if (f < 0) return s;                 // (one row of zeros before the top)
    n = f / (j.W + 2);
    x = f - n * (j.W + 2);
    y = r < j.line[1] ? 0 : j.H - 1;
  } else if (r < j.line[4]) {            // left, right
    const int f = r - (r < j.line[3] ? j.line[2] : j.line[3]);
    n = f / (j.H + 2);
    y = f - n * (j.H + 2);
    x = r < j.line[3] ? 0 : j.W - 1;
  } else {                               // corners: (0,0) (0,W) (H,0) (H,W)
    int k = 0;
    while (k < 3 && r >= j.line[5 + k]) ++k;
    n = r - j.line[4 + k];
    y = (k & 2) ? j.H - 1 : 0;
    x = (k & 1) ? j.W - 1 : 0;
  }
  if (n < j.n && y < j.H && x < j.W)
    s.off = j.nhwc ? (((long long)n * j.H + y) * j.W + x) * j.C
                   : ((long long)n * j.C * j.H + y) * j.W + x;
  return s;
}

__device__ __forceinline__ float patch_value(const StageJob& j,
                                             const RowSrc& s, int c, int ky,
                                             int kx) {
  const int iy = s.iy + ky, ix = s.ix + kx;
  if (iy < 0 || iy >= j.H || ix < 0 || ix >= j.W) return 0.f;
  const long long o = j.nhwc ? ((long long)iy * j.W + ix) * j.C + c
                             : ((long long)c * j.H + iy) * j.W + ix;
  return __ldg(j.base + s.off + o);
}

// Items of a block grow, so its job only moves forward.
__device__ __forceinline__ bool stage_job(const StageJob* jobs, int njobs,
                                          int item, int& ji) {
  const int old = ji;
  if (ji < 0) ji = 0;
  while (ji + 1 < njobs && __ldg(&jobs[ji + 1].item_begin) <= item) ++ji;
  return ji != old;
}

__device__ __forceinline__ void stage_fetch(StageJob& j, const StageJob* src) {
  __syncthreads();
  for (int i = threadIdx.x; i < (int)(sizeof(StageJob) / 4); i += 256)
    reinterpret_cast<int*>(&j)[i] = __ldg(reinterpret_cast<const int*>(src) + i);
  __syncthreads();
}

// Sources that are contiguous along the columns (rows x d matrices,
// channels-last tensors), and patches of them: a thread stages 8 columns of
// four rows, 128 bytes in flight.
__global__ void __launch_bounds__(256, 4)
stage_cols_kernel(const StageJob* __restrict__ jobs, int njobs, int items) {
  __shared__ StageJob j;
  __shared__ RowSrc s_row[2][kStageRowsC];
  int ji = -1, flip = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x, flip ^= 1) {
    if (stage_job(jobs, njobs, item, ji)) stage_fetch(j, jobs + ji);
    const int local = item - j.item_begin;
    const int rb = local / j.cblocks;
    const int col = 64 * (local - rb * j.cblocks) + 8 * (threadIdx.x & 7);
    const int r0 = rb * kStageRowsC;
    if (threadIdx.x < kStageRowsC)
      s_row[flip][threadIdx.x] = row_source(j, r0 + threadIdx.x);
    __syncthreads();
    if (col >= j.cp) continue;
    float v[4][8];
    const bool whole = j.vec && col + 8 <= j.ncols;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const RowSrc s = s_row[flip][(threadIdx.x >> 3) + 32 * i];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[i][k] = 0.f;
      if (s.off < 0) continue;
      if (whole) {
        const float4* p = reinterpret_cast<const float4*>(j.base + s.off + col);
        const float4 a = __ldg(p), b = __ldg(p + 1);
        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
        v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
      } else if (j.kind != kSrcPatches) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (col + k < j.ncols) v[i][k] = __ldg(j.base + s.off + col + k);
      } else {
        const int kk = j.ks * j.ks;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int cc = col + k;
          if (cc < j.ncols) {
            const int c = cc / kk, tap = cc - c * kk;
            const int ky = tap / j.ks;
            v[i][k] = patch_value(j, s, c, ky, tap - ky * j.ks);
          }
        }
      }
    }
    if (j.extra_idx >= col && j.extra_idx < col + 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + (threadIdx.x >> 3) + 32 * i;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (col + k == j.extra_idx)
            v[i][k] = r < j.K ? (j.extra ? j.extra[r] : 1.f) : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + (threadIdx.x >> 3) + 32 * i;
      if (r < j.prows) gr_store8(j, r, col, v[i]);
    }
  }
}

// Sources that are contiguous along the rows of X (NCHW tensors, transposed
// matrices): read with the rows along the lanes, turned in shared memory.  Bound
// by HBM and, below that, by how much of it is in flight: 64 rows x 64 columns
// and 16 independent loads a thread (the activations and gradients of ResNet-50,
// 32 images: 552 us with 32 rows and eight loads, 394 now); of patches, the
// taps' positions come from a table, no load waits for a branch.
__global__ void __launch_bounds__(256, 4)
stage_rows_kernel(const StageJob* __restrict__ jobs, int njobs, int items) {
  __shared__ StageJob j;
  __shared__ RowSrc s_row[kStageRowsK];
  __shared__ int2 s_tap[64];       // offset of the column, ky << 16 | kx (or -1)
  __shared__ float tile[64][kStageRowsK + 1];
  int ji = -1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    if (stage_job(jobs, njobs, item, ji)) stage_fetch(j, jobs + ji);
    const int local = item - j.item_begin;
    const int rb = local / j.cblocks;
    const int c0 = 64 * (local - rb * j.cblocks);
    const int r0 = rb * kStageRowsK;
    if (threadIdx.x < kStageRowsK) {
      s_row[threadIdx.x] = row_source(j, r0 + threadIdx.x);
    } else if (j.kind == kSrcPatches && threadIdx.x >= 192) {
      const int t = threadIdx.x - 192, cc = c0 + t, kk = j.ks * j.ks;
      const int c = cc / kk, tap = cc - c * kk, ky = tap / j.ks;
      const int kx = tap - ky * j.ks;
      s_tap[t] = make_int2((c * j.H + ky) * j.W + kx,
                           cc < j.ncols ? ky << 16 | kx : -1);
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kStageRowsK / 32; ++h) {
      const RowSrc s0 = s_row[lane + 32 * h];
      float v[8];
      if (j.kind != kSrcPatches) {
        const float* p = j.base + s0.off + (long long)(c0 + warp) * j.s_col;
#pragma unroll
        for (int i = 0; i < 8; ++i, p += 8 * j.s_col)
          v[i] = c0 + warp + 8 * i < j.ncols && s0.off >= 0 ? __ldg(p) : 0.f;
      } else {
        const float* p = j.base + s0.off + (long long)s0.iy * j.W + s0.ix;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int2 t = s_tap[warp + 8 * i];
          const int iy = s0.iy + (t.y >> 16), ix = s0.ix + (t.y & 0xffff);
          const bool in = t.y >= 0 && s0.off >= 0 &&
                          (unsigned)iy < (unsigned)j.H &&
                          (unsigned)ix < (unsigned)j.W;
          v[i] = in ? __ldg(p + t.x) : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) tile[warp + 8 * i][lane + 32 * h] = v[i];
    }
    if (j.extra_idx >= c0 && j.extra_idx < c0 + 64) {
      __syncthreads();
      if (threadIdx.x < kStageRowsK) {
        const int r = r0 + threadIdx.x;
        tile[j.extra_idx - c0][threadIdx.x] =
            r < j.K ? (j.extra ? j.extra[r] : 1.f) : 0.f;
      }
    }
    __syncthreads();
    const int cg = 8 * (threadIdx.x & 7);
#pragma unroll
    for (int h = 0; h < kStageRowsK / 32; ++h) {
      const int rr = (threadIdx.x >> 3) + 32 * h;
      if (c0 + cg < j.cp && r0 + rr < j.prows) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = tile[cg + k][rr];
        gr_store8(j, r0 + rr, c0 + cg, v);
      }
    }
    __syncthreads();
  }
}

// -------------------------------------------------------------------- output
struct GramOut {
  float* out;
  float* out2;                 // if set: out2 = a2 * (new out) + b2 * out2
  float a2, b2;
  int d;                       // side of the factor
  int C;                       // channels (shifted products), 0: plain
  int strips;                  // plain: 32 x 128 pieces, else 32 x 32
  float alpha, beta;
  int item_begin;
  // plain: one group; shifted: main, top, bottom, left, right, corners
  const float* partial[9];
  int splits[9];
  int tiles[9];
};

// Sum of the splits of four consecutive columns (4 c4 ..) of one row.
__device__ __forceinline__ float4 split_sum(const float* partial, int splits,
                                            long long stride, long long at) {
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* p = partial + at;
#pragma unroll 8
  for (int s = 0; s < splits; ++s, p += stride) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  return a;
}

__device__ __forceinline__ int out_find(const int* begin, int n, int item) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (begin[mid] <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Strips of 32 rows x 128 columns that cover the lower triangle, row block
// after row block: row blocks 4 q .. 4 q + 3 have q + 1 strips each.
__host__ __device__ __forceinline__ int strips_before(int row_block) {
  const int q = row_block >> 2;
  return 2 * q * (q + 1) + (row_block & 3) * (q + 1);
}

// Output of 32 rows x 32 W columns: sum of the splits (in order), scaling, the
// piece and its mirror image.  All loads of a thread are independent.
template <int W, int UNROLL>
__device__ __forceinline__ void reduce_piece(const GramOut& o, int m0, int n0,
                                             float (*t)[132]) {
  const int d = o.d, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ti = m0 >> 8, tj = n0 >> 8;
  const float alpha = o.alpha, beta = o.beta, a2 = o.a2, b2 = o.b2;
  float* out2 = o.out2;
  float old[4][W];
  if (beta != 0.f) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const int r = m0 + warp + 8 * i, c = n0 + lane + 32 * k;
        old[i][k] = r < d && c <= r ? __ldcg(o.out + (long long)r * d + c) : 0.f;
      }
  }
  {
    const float* p = o.partial[0] +
                     (long long)(ti * (ti + 1) / 2 + tj) * GR_TILE +
                     (long long)(((n0 & 255) >> 2) + warp) * 1024 +
                     4 * ((m0 & 255) + lane);
    const long long stride = (long long)o.tiles[0] * GR_TILE;
    const int splits = o.splits[0];
    // (only columns up to the row exist in a tile on the diagonal)
    bool on[W];
    float4 v[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      on[k] = m0 + lane < d && n0 + 32 * k + 4 * warp <= m0 + lane;
      v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll UNROLL
    for (int s = 0; s < splits; ++s, p += stride)
#pragma unroll
      for (int k = 0; k < W; ++k)
        if (on[k]) {
          const float4 x = __ldcg(reinterpret_cast<const float4*>(p + 8192 * k));
          v[k].x += x.x; v[k].y += x.y; v[k].z += x.z; v[k].w += x.w;
        }
#pragma unroll
    for (int k = 0; k < W; ++k)
      *reinterpret_cast<float4*>(&t[lane][32 * k + 4 * warp]) = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int r = m0 + warp + 8 * i, c = n0 + lane + 32 * k;
      if (r < d && c <= r) {
        float v = alpha * t[warp + 8 * i][lane + 32 * k];
        if (beta != 0.f) v += beta * old[i][k];
        o.out[(long long)r * d + c] = v;
        t[warp + 8 * i][lane + 32 * k] = v;
      }
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4 * W; ++i) {
    const int r = m0 + lane, c = n0 + warp + 8 * i;
    if (r < d && c < r) o.out[(long long)c * d + r] = t[lane][warp + 8 * i];
  }
  if (out2 == nullptr) return;
  // the second output, through the same tile
  float next[4][W];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int r = m0 + warp + 8 * i, c = n0 + lane + 32 * k;
      if (r < d && c <= r) {
        float* p = out2 + (long long)r * d + c;
        float v = a2 * t[warp + 8 * i][lane + 32 * k];
        if (b2 != 0.f) v += b2 * *p;
        *p = v;
        next[i][k] = v;
      }
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k)
      t[warp + 8 * i][lane + 32 * k] = next[i][k];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4 * W; ++i) {
    const int r = m0 + lane, c = n0 + warp + 8 * i;
    if (r < d && c < r) out2[(long long)c * d + r] = t[lane][warp + 8 * i];
  }
}

// Plain factors.  Wide strips where there are many of them and few splits;
// 32 x 32 pieces where a narrow factor was cut into many splits, which a few
// blocks would read one latency after the other (148 columns, 98 splits: 350 us
// in strips, 30 us in pieces).
__global__ void __launch_bounds__(256)
gram_reduce_kernel(const GramOut* __restrict__ outs, int nouts) {
  __shared__ int s_begin[kStageJobs];
  __shared__ float t[32][132];
  for (int i = threadIdx.x; i < nouts; i += 256) s_begin[i] = outs[i].item_begin;
  __syncthreads();
  const GramOut& o = outs[out_find(s_begin, nouts, blockIdx.x)];
  const int item = blockIdx.x - o.item_begin;
  if (!o.strips) {
    int bi, bj;
    tri_of(item, bi, bj);
    reduce_piece<1, 8>(o, 32 * bi, 32 * bj, t);
    return;
  }
  int q = (int)((sqrtf(1.f + 2.f * (float)item) - 1.f) * 0.5f);
  while (2 * (q + 1) * (q + 2) <= item) ++q;
  while (2 * q * (q + 1) > item) --q;
  const int in = item - 2 * q * (q + 1);
  reduce_piece<4, 2>(o, 32 * (4 * q + in / (q + 1)), 128 * (in % (q + 1)), t);
}

// Shifted products -> patch factor.  A block per pair of 8-channel groups
// I >= J sums the splits of every product block [I][J] and [J][I] once into
// shared memory (13 offsets, 3 per border line, 4 corners) and writes the
// 72 x 72 piece of the factor and its mirror image.
constexpr int kXc = 8;
constexpr int kXBlocks = 2 * (GR_SHIFTS + 12) + 4;
constexpr int kXBlk = kXc * (kXc + 1);
constexpr int kXSmem = kXBlocks * kXBlk * 4;

// index of offset (dy, dx), dy > 0 or dy == 0 and dx >= 0
__host__ __device__ __forceinline__ int shift_index(int dy, int dx) {
  return dy == 0 ? dx : 3 + (dy - 1) * 5 + dx + 2;
}

// Granules of the main group when one granule holds all channels: A granules
// are shifts (0,0) and (0,1), so that a B granule at (y, x) gives offsets
// (y, x) and (y, x - 1); these eight give all 13.
__host__ __device__ __forceinline__ void tap_granule(int dy, int dx, int& a,
                                                     int& b) {
  // B granules: (0,1) (0,2) | (1,-1) (1,1) (1,2) | (2,-1) (2,1) (2,2)
  if (dy == 0) {
    a = dx == 0 ? 1 : 0;
    b = dx == 2 ? 1 : 0;
    return;
  }
  const int base = dy == 1 ? 2 : 5;
  a = dx == -2 || dx == 0 ? 1 : 0;
  b = base + (dx <= -1 ? 0 : (dx <= 1 ? 1 : 2));
}

__device__ __forceinline__ long long gram_at(int ga, int gb, int tb, int row,
                                             int col) {
  const int tile = (ga >> 2) * tb + (gb >> 2);
  return (long long)tile * GR_TILE +
         (long long)(((gb & 3) * 64 + col) >> 2) * 1024 +
         4 * ((ga & 3) * 64 + row);
}

constexpr int kXThreads = 4 * 9 * kXc;    // 9 kXc columns, 4 sets of row taps

__global__ void __launch_bounds__(kXThreads, 4)
gram_expand_kernel(const GramOut* __restrict__ outs, int nouts) {
  extern __shared__ float xs[];        // [block][kXc][kXc + 1]
  __shared__ int s_begin[kStageJobs];
  __shared__ int s_tap[81];
  for (int i = threadIdx.x; i < nouts; i += kXThreads) s_begin[i] = outs[i].item_begin;
  if (threadIdx.x < 81) {
    // (ti, tj) -> main block, border blocks; bit 31: roles of I and J swapped
    int a = threadIdx.x / 9, b = threadIdx.x % 9;
    int dy = b / 3 - a / 3, dx = b % 3 - a % 3;
    const bool swap = dy < 0 || (dy == 0 && dx < 0);
    if (swap) { dy = -dy; dx = -dx; const int t = a; a = b; b = t; }
    const int ty = a / 3 - 1, tx = a % 3 - 1;
    int e = 0;
    if (dy == 0 && ty != 0) e |= (1 + (ty > 0 ? 0 : 3) + dx) << 8;
    if (dx == 0 && tx != 0) e |= (1 + (tx > 0 ? 0 : 3) + dy) << 16;
    if (dy == 0 && dx == 0 && ty != 0 && tx != 0)
      e |= (1 + (ty > 0 ? 0 : 2) + (tx > 0 ? 0 : 1)) << 24;
    s_tap[threadIdx.x] = shift_index(dy, dx) | e | (swap ? 1 << 31 : 0);
  }
  __syncthreads();
  const GramOut& o = outs[out_find(s_begin, nouts, blockIdx.x)];
  int bi, bj;
  tri_of(blockIdx.x - o.item_begin, bi, bj);
  const int C = o.C, d = o.d, cg = (C + 63) >> 6;
  const int i0 = kXc * bi, j0 = kXc * bj;
  // blocks: [0, 13) offsets [I][J]; [13, 26) offsets [J][I];
  // then 12 border products [I][J], 12 [J][I], 4 corners [I][J]
  for (int w = threadIdx.x; w < kXBlocks * kXc * kXc / 4;
       w += kXThreads) {
    const int blk = w / (kXc * kXc / 4), e = w % (kXc * kXc / 4);
    const int row = e % kXc, c4 = e / kXc;
    bool flip;
    int grp, gk;
    if (blk < 26) {
      flip = blk >= 13; grp = 0; gk = flip ? blk - 13 : blk;
    } else if (blk < 50) {
      flip = blk >= 38;
      const int k = blk - (flip ? 38 : 26);
      grp = 1 + k / 3; gk = k % 3;
    } else {
      flip = false; grp = 5 + blk - 50; gk = 0;
    }
    const int r = (flip ? j0 : i0) + row, c = (flip ? i0 : j0) + 4 * c4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < C && c < C) {
      int ga = r >> 6, gb, nb;
      if (grp == 0 && cg == 1) {
        const int dy = gk < 3 ? 0 : (gk < 8 ? 1 : 2);
        const int dx = dy == 0 ? gk : gk - 3 - 5 * (dy - 1) - 2;
        tap_granule(dy, dx, ga, gb);
        nb = 8;
      } else {
        gb = gk * cg + (c >> 6);
        nb = (grp == 0 ? GR_SHIFTS : (grp < 5 ? 3 : 1)) * cg;
      }
      v = split_sum(o.partial[grp], o.splits[grp],
                    (long long)o.tiles[grp] * GR_TILE,
                    gram_at(ga, gb, (nb + 3) >> 2, r & 63, c & 63));
    }
    float* q = xs + blk * kXBlk + row * (kXc + 1) + 4 * c4;
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
  }
  __syncthreads();
  // A thread owns one column (channel, tap) and walks the row taps: the blocks
  // a pair of taps needs are looked up once for all row channels.
  const float alpha = o.alpha, beta = o.beta, a2 = o.a2, b2 = o.b2;
  const bool two = o.out2 != nullptr;
  const int col = threadIdx.x % (9 * kXc), set = threadIdx.x / (9 * kXc);
  const int cc = col / 9, ct = col - 9 * cc;
  for (int pass = 0; pass < (bi == bj ? 1 : 2); ++pass) {
    // pass 0: rows in I, columns in J; pass 1: the mirror image
    const int ra = pass ? j0 : i0, ca = pass ? i0 : j0;
    if (ca + cc >= C) continue;
    const int nr = min(kXc, C - ra);
    for (int rt = set; rt < 9; rt += 4) {
      const int tap = s_tap[rt * 9 + ct];
      const int m = tap & 0xff, e1 = (tap >> 8) & 0xff, e2 = (tap >> 16) & 0xff,
                e3 = (tap >> 24) & 0x7f;
      // the offset starts from the member of J (offset zero is symmetric:
      // always read as [I][J])
      const bool ji = m != 0 && ((tap < 0) != (pass != 0));
      const int jo = ji ? 13 * kXBlk : 0, je = ji ? 12 * kXBlk : 0;
      const float* pm = xs + m * kXBlk + jo;
      const float* p1 = e1 ? xs + (25 + e1) * kXBlk + je : nullptr;
      const float* p2 = e2 ? xs + (31 + e2) * kXBlk + je : nullptr;
      const float* p3 = e3 ? xs + (49 + e3) * kXBlk : nullptr;
      // element (row channel rc, column channel cc) of the block
      const bool rows_first = ji == (pass != 0);
      const int sr = rows_first ? kXc + 1 : 1;
      const int at0 = rows_first ? cc : cc * (kXc + 1);
      float* p = o.out + (long long)(9 * ra + rt) * d + 9 * ca + col;
      const long long step = 9LL * d;
      float* second = o.out2 + (p - o.out);
      float old[kXc], old2[kXc];
#pragma unroll
      for (int rc = 0; rc < kXc; ++rc)
        old[rc] = beta != 0.f && rc < nr ? __ldcg(p + rc * step) : 0.f;
      if (two) {
#pragma unroll
        for (int rc = 0; rc < kXc; ++rc)
          old2[rc] = b2 != 0.f && rc < nr ? __ldcg(second + rc * step) : 0.f;
      }
#pragma unroll
      for (int rc = 0; rc < kXc; ++rc) {
        int at = at0 + rc * sr;
        if (m == 0 && bi == bj && cc > rc) at = cc * (kXc + 1) + rc;
        float v = pm[at];
        if (e1) v -= p1[at];
        if (e2) v -= p2[at];
        if (e3) v += p3[at];
        v = fmaf(beta, old[rc], alpha * v);
        if (rc >= nr) continue;
        p[rc * step] = v;
        if (two) second[rc * step] = fmaf(b2, old2[rc], a2 * v);
      }
    }
  }
}

// ----------------------------------------------------------------- host side
// cuTensorMapEncodeTiled through the runtime's driver entry point: the
// library must load on machines without a driver (build checks, CPU tests).
typedef CUresult (*EncodeTiledFn)(
    CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
    CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
    CUtensorMapFloatOOBfill);

int encode_tiled_fn(EncodeTiledFn* out) {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    KFAC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p,
                                      cudaEnableDefault, &q));
    KFAC_REQUIRE(q == cudaDriverEntryPointSuccess && p != nullptr,
                 "factor: the driver has no cuTensorMapEncodeTiled");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  *out = fn;
  return KFAC_OK;
}

inline int up32(long long v) { return (int)((v + 31) & ~31LL); }

// Plan of one job: its plane and its groups of products.
struct JobPlan {
  bool grid;               // shifted products of a 3 x 3 convolution
  int direct;              // no planes: 1 columns, 2 rows contiguous
  int width, per_image;    // direct only
  int cols, cp;            // columns of the plane
  int prows;               // its rows
  int line[8];
  size_t plane_bytes;      // one of the two planes
  int ngroups;
  int row0[9], nkb[9], nga[9], ngb[9], tiles[9], splits[9], kb_split[9];
  size_t partial_bytes;
};

void plan_job(const FactorJob& job, JobPlan& p) {
  const Operand& X = job.X;
  p.grid = gram_grid_job(job);
  p.direct = gram_direct_job(job) ? (X.s_col == 1 && X.period == 1 ? 1 : 2)
                                        : 0;
  if (p.direct) {
    p.cols = job.d;
    p.prows = 0;
    p.plane_bytes = 0;
    p.width = job.d <= 64 ? 64 : (job.d <= 128 ? 128 : 256);
    const int t = (job.d + 255) / 256;
    p.ngroups = 1;
    p.tiles[0] = t * (t + 1) / 2;
    p.nga[0] = (job.d + GR_GRAN - 1) / GR_GRAN;
    // k-blocks of 32 rows
    if (p.direct == 2) {
      const int hw = X.period == 1 ? (int)job.rows : X.period;
      p.per_image = (hw + 31) / 32;
      p.nkb[0] = (int)(job.rows / hw) * p.per_image;
    } else {
      p.nkb[0] = (int)((job.rows + 31) / 32);
    }
    return;
  }
  if (!p.grid) {
    p.cols = job.d;
    p.prows = (int)job.rows;
    p.ngroups = 1;
    p.row0[0] = 0;
    p.nkb[0] = (int)((job.rows + GR_BK - 1) / GR_BK);
    p.nga[0] = (job.d + GR_GRAN - 1) / GR_GRAN;
    p.ngb[0] = 0;
    const int t = (job.d + 255) / 256;
    p.tiles[0] = t * (t + 1) / 2;
  } else {
    p.cols = X.C;
    const int cg = (X.C + GR_GRAN - 1) / GR_GRAN;
    // (a zero row before and after the images: with one granule the A
    // operand is shifted by a row as well)
    const int rows[9] = {up32(1 + (long long)job.n * (X.H + 2) * (X.W + 2)),
                         up32(1 + (long long)job.n * (X.W + 2)),
                         up32((long long)job.n * (X.W + 2)),
                         up32((long long)job.n * (X.H + 2)),
                         up32((long long)job.n * (X.H + 2)),
                         up32(job.n), up32(job.n), up32(job.n), up32(job.n)};
    p.ngroups = 9;
    int r = 0;
    for (int k = 0; k < 9; ++k) {
      if (k > 0) p.line[k - 1] = r;
      p.row0[k] = r;
      p.nkb[k] = rows[k] / GR_BK;
      r += rows[k];
      p.nga[k] = k == 0 && cg == 1 ? 2 : cg;
      p.ngb[k] = k == 0 ? (cg == 1 ? 8 : GR_SHIFTS * cg) : (k < 5 ? 3 : 1) * cg;
      p.tiles[k] = ((p.nga[k] + 3) / 4) * ((p.ngb[k] + 3) / 4);
    }
    p.prows = r;
  }
  p.cp = (p.cols + 7) & ~7;
  p.plane_bytes = ((size_t)p.prows * p.cp * 2 + 255) & ~(size_t)255;
}

// Duration of a k-block of one tile in quarters of a 128 x 256 product (about
// 200 cycles): products of staged planes by the tensor cores, without planes
// by the memory traffic of one tile side.
inline int group_cost(const JobPlan& p, int k) {
  if (p.direct) return p.tiles[0] > 1 ? 8 : p.width / 32;
  return p.nga[k] > 2 ? 8 : 4;
}

// A CTA keeps at least 16 k-blocks so that its prologue and epilogue stay
// amortised, and never accumulates more than 128 (KFAC_TC_MAX_KBLOCKS): the
// tensor core adds each product into the fp32 accumulator with truncation, so
// that a long sum drifts (relative error of a 100 352-row factor of non-negative
// values: 2e-4 when one CTA accumulates 1500 k-blocks, 4.7e-5 at 256, 2e-5 at
// 128); the partial tiles are added with rounding to nearest.
void split_job(JobPlan& p, long long target) {
  // (whole stages: a multiple of four)
  const long long most = factor_max_kblocks(128) & ~3LL;
  p.partial_bytes = 0;
  for (int k = 0; k < p.ngroups; ++k) {
    long long chunk = target / group_cost(p, k);
    // (one tile without planes: eight stages)
    const long long least =
        p.direct && p.tiles[0] == 1 ? 2048 / p.width : 16;
    chunk = std::max(least, std::min(most, chunk));
    const long long sp =
        std::max(std::max(1LL, p.nkb[k] / chunk), (p.nkb[k] + most - 1) / most);
    p.kb_split[k] = (int)((p.nkb[k] + sp - 1) / sp);
    if (p.direct) {
      // whole stages: 16 rows of two sides, or 256 / width k-blocks of one
      // (tiles on the diagonal of a wide factor: 32 rows)
      const int per = p.tiles[0] > 1 ? 1 : 256 / p.width;
      p.kb_split[k] = (p.kb_split[k] + per - 1) / per * per;
    }
    p.splits[k] = (p.nkb[k] + p.kb_split[k] - 1) / p.kb_split[k];
    p.partial_bytes +=
        (size_t)p.splits[k] * p.tiles[k] * GR_TILE * sizeof(float);
  }
}

// Work per CTA: at most two waves over the SMs (KFAC_TC_WAVES), so that the 10 us
// a CTA spends before its first and behind its last product stay small.
long long split_target(const std::vector<JobPlan>& plans, size_t b, size_t e) {
  long long work = 0;
  for (size_t i = b; i < e; ++i)
    for (int k = 0; k < plans[i].ngroups; ++k)
      work += (long long)plans[i].tiles[k] * plans[i].nkb[k] *
              group_cost(plans[i], k);
  return work / (factor_waves() * sm_count()) + 1;
}

// Jobs are worked off in batches whose planes and partial tiles stay below this
// many bytes, so that the workspace does not grow with the network.  A batch's
// partial tiles are counted with the fewest splits its jobs can have; cutting
// them further into two waves of CTAs adds at most a tile each (0.1 GB).  (All
// factors of ResNet-50 at 32 images take 1.4 GB and one batch.  Staging a batch
// beside the products of the one before, in two workspaces, gained nothing: both
// halves are bound by the same memory traffic.)
constexpr size_t kBatchBytesMax = (size_t)2 << 30;

size_t least_bytes(const JobPlan& p) {
  const long long most = factor_max_kblocks(128) & ~3LL;
  long long tiles = 0;
  for (int k = 0; k < p.ngroups; ++k)
    tiles += p.tiles[k] * ((p.nkb[k] + most - 1) / most);
  return 2 * p.plane_bytes + (size_t)tiles * GR_TILE * sizeof(float);
}

size_t batch_end(const std::vector<JobPlan>& plans, size_t b) {
  size_t e = b, bytes = 0;
  while (e < plans.size() && e - b < (size_t)kStageJobs) {
    bytes += least_bytes(plans[e]);
    if (e > b && bytes > kBatchBytesMax) break;
    ++e;
  }
  return e;
}

}  // namespace

static size_t plans_bytes(std::vector<JobPlan>& plans) {
  size_t most = 0;
  for (size_t b = 0, e; b < plans.size(); b = e) {
    e = batch_end(plans, b);
    const long long target = split_target(plans, b, e);
    size_t bytes = 0;
    for (size_t i = b; i < e; ++i) {
      split_job(plans[i], target);
      bytes += 2 * plans[i].plane_bytes + plans[i].partial_bytes;
    }
    most = std::max(most, bytes);
  }
  return most;
}

size_t gram_workspace_bytes(int count, const FactorJob* jobs) {
  std::vector<JobPlan> plans(count);
  for (int i = 0; i < count; ++i) plan_job(jobs[i], plans[i]);
  return plans_bytes(plans);
}

static int gram_prepare() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  KFAC_CUDA(cudaGetDevice(&dev));
  KFAC_REQUIRE(dev >= 0 && dev < 64, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    KFAC_CUDA(cudaFuncSetAttribute(
        gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM));
    KFAC_CUDA(cudaFuncSetAttribute(direct_kernel<false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DR_SMEM));
    KFAC_CUDA(cudaFuncSetAttribute(direct_kernel<true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DR_SMEM));
    KFAC_CUDA(cudaFuncSetAttribute(
        gram_expand_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
        kXSmem));
    done[dev] = true;
  }
  return KFAC_OK;
}

static int upload(const void* host, size_t bytes, cudaStream_t stream,
                  void** dev) {
  const int rc = ring_alloc(bytes, dev);
  if (rc != KFAC_OK) return rc;
  KFAC_CUDA(cudaMemcpyAsync(*dev, host, bytes, cudaMemcpyHostToDevice, stream));
  return KFAC_OK;
}

static int gram_batch(const FactorJob* jobs, std::vector<JobPlan>& plans,
                      size_t b, size_t e, char* ws, EncodeTiledFn encode,
                      cudaStream_t stream) {
  struct alignas(64) Map { CUtensorMap m; };
  const size_t n = e - b;
  const long long target = split_target(plans, b, e);
  std::vector<Map> maps(n);
  std::vector<StageJob> stage[2];       // columns contiguous, rows contiguous
  int sitems[2] = {0, 0};
  std::vector<GramGroup> groups;
  std::vector<DirectGroup> direct[2];   // columns contiguous, rows contiguous
  std::vector<GramOut> outs[2];         // plain, shifted
  int oitems[2] = {0, 0};
  int direct_units[2] = {0, 0};
  void* dev_maps = nullptr;
  int rc = ring_alloc(n * sizeof(Map), &dev_maps);
  if (rc != KFAC_OK) return rc;
  for (size_t i = b; i < e; ++i) {
    const FactorJob& job = jobs[i];
    JobPlan& p = plans[i];
    split_job(p, target);
    const Operand& X = job.X;
    if (p.direct) {
      const bool km = p.direct == 2;
      const long long hw = X.period == 1 ? job.rows : X.period;
      DirectGroup g = {};
      g.tmap = static_cast<const Map*>(dev_maps) + (i - b);
      g.partial = reinterpret_cast<float*>(ws);
      ws += p.partial_bytes;
      g.nkb = p.nkb[0];
      g.kb_split = p.kb_split[0];
      g.tiles = p.tiles[0];
      g.d = job.d;
      g.width = p.width;
      g.box_rows = p.tiles[0] > 1 ? 16 : 8192 / p.width;
      g.per_image = p.per_image;
      const cuuint64_t dims[3] = {(cuuint64_t)(km ? hw : job.d),
                                  (cuuint64_t)(km ? job.d : job.rows),
                                  (cuuint64_t)(km ? job.rows / hw : 1)};
      const cuuint64_t pitch = (cuuint64_t)(km ? X.s_col : X.s_outer) * 4;
      const cuuint64_t strides[2] = {pitch, pitch * dims[1]};
      const cuuint32_t box[3] = {(cuuint32_t)(km ? 32 : GR_GRAN),
                                 (cuuint32_t)(km ? p.width : g.box_rows), 1};
      const cuuint32_t es[3] = {1, 1, 1};
      const CUresult r = encode(
          &maps[i - b].m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)X.base,
          dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS)
        return fail(KFAC_ERR_CUDA,
                    "factor: cuTensorMapEncodeTiled failed (%d) for a %lld x "
                    "%d operand", (int)r, job.rows, job.d);
      direct[km ? 1 : 0].push_back(g);
      GramOut o = {};
      o.out = job.out;
      o.out2 = job.out2;
      o.a2 = job.a2;
      o.b2 = job.b2;
      o.d = job.d;
      o.alpha = job.alpha;
      o.beta = job.beta;
      o.partial[0] = g.partial;
      o.splits[0] = p.splits[0];
      o.tiles[0] = p.tiles[0];
      const int rb = (job.d + 31) / 32;
      o.strips = p.splits[0] <= 4;
      o.item_begin = oitems[0];
      oitems[0] += o.strips ? strips_before(rb) : rb * (rb + 1) / 2;
      outs[0].push_back(o);
      continue;
    }
    StageJob s = {};
    s.base = X.base;
    s.extra = X.extra;
    s.hi = reinterpret_cast<unsigned short*>(ws);
    s.plane = (long long)(p.plane_bytes / 2);
    ws += 2 * p.plane_bytes;
    s.K = job.rows;
    s.prows = p.prows;
    s.cp = p.cp;
    s.d = p.cols;
    s.extra_idx = X.extra_idx;
    s.kind = p.grid ? kSrcGrid : (X.mode == 1 ? kSrcPatches : kSrcStrided);
    s.ncols = p.grid ? X.C : (X.mode == 1 ? X.C * X.ks * X.ks : X.ncols);
    s.s_outer = X.s_outer;
    s.s_inner = X.s_inner;
    s.s_col = p.grid ? (job.nhwc ? 1 : (long long)X.H * X.W) : X.s_col;
    s.period = X.period;
    s.n = job.n;
    s.C = X.C; s.H = X.H; s.W = X.W; s.ks = X.ks; s.st = X.st; s.pd = X.pd;
    s.Ho = X.Ho; s.Wo = X.Wo; s.nhwc = job.nhwc;
    for (int k = 0; k < 8; ++k) s.line[k] = p.grid ? p.line[k] : 0;
    s.cblocks = (p.cp + 63) / 64;
    const bool cols = s.kind == kSrcPatches ? job.nhwc != 0 : s.s_col == 1;
    const bool aligned = (reinterpret_cast<uintptr_t>(X.base) & 15) == 0;
    s.vec = cols && aligned &&
            (p.grid ? X.C % 4 == 0
                    : s.kind == kSrcStrided && X.s_outer % 4 == 0 &&
                          (X.period == 1 || X.s_inner % 4 == 0));
    const int m = cols ? 0 : 1;
    const int rows = cols ? kStageRowsC : kStageRowsK;
    s.item_begin = sitems[m];
    sitems[m] += ((p.prows + rows - 1) / rows) * s.cblocks;
    stage[m].push_back(s);

    const cuuint64_t dims[3] = {(cuuint64_t)p.cols, (cuuint64_t)p.prows, 2};
    const cuuint64_t strides[2] = {(cuuint64_t)p.cp * 2,
                                   (cuuint64_t)p.plane_bytes};
    const cuuint32_t box[3] = {GR_GRAN, GR_BK, 2};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = encode(
        &maps[i - b].m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)s.hi, dims,
        strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return fail(KFAC_ERR_CUDA,
                  "factor: cuTensorMapEncodeTiled failed (%d) for a %d x %d "
                  "plane", (int)r, p.prows, p.cols);

    GramOut o = {};
    o.out = job.out;
    o.out2 = job.out2;
    o.a2 = job.a2;
    o.b2 = job.b2;
    o.d = job.d;
    o.C = p.grid ? X.C : 0;
    o.alpha = job.alpha;
    o.beta = job.beta;
    for (int k = 0; k < p.ngroups; ++k) {
      GramGroup g = {};
      g.tmap = static_cast<const Map*>(dev_maps) + (i - b);
      g.partial = reinterpret_cast<float*>(ws);
      ws += (size_t)p.splits[k] * p.tiles[k] * GR_TILE * sizeof(float);
      g.row0 = p.row0[k];
      g.nkb = p.nkb[k];
      g.kb_split = p.kb_split[k];
      g.tiles = p.tiles[k];
      g.nga = p.nga[k];
      g.ngb = p.ngb[k];
      g.d = p.cols;
      g.cg = (p.cols + GR_GRAN - 1) / GR_GRAN;
      if (p.grid) {
        const int wp = X.W + 2;
        if (k == 0 && g.cg == 1) {
          const int sh[8] = {1, 2, wp - 1, wp + 1, wp + 2,
                             2 * wp - 1, 2 * wp + 1, 2 * wp + 2};
          for (int q = 0; q < 8; ++q) g.shift[q] = sh[q];
          g.ashift[1] = 1;
        } else if (k == 0) {
          for (int dy = 0; dy < 3; ++dy)
            for (int dx = dy == 0 ? 0 : -2; dx < 3; ++dx)
              g.shift[shift_index(dy, dx)] = dy * wp + dx;
        } else {
          for (int q = 0; q < 3; ++q) g.shift[q] = q;
        }
      }
      o.partial[k] = g.partial;
      o.splits[k] = p.splits[k];
      o.tiles[k] = p.tiles[k];
      groups.push_back(g);
    }
    const int t = (X.C + kXc - 1) / kXc;
    const int w = p.grid ? 1 : 0;
    o.item_begin = oitems[w];
    const int rb = (job.d + 31) / 32;
    o.strips = !p.grid && p.splits[0] <= 4;
    oitems[w] += p.grid ? t * (t + 1) / 2
                        : (o.strips ? strips_before(rb) : rb * (rb + 1) / 2);
    outs[w].push_back(o);
  }
  for (int m = 0; m < 2; ++m) {
    std::vector<DirectGroup>& v = direct[m];
    if (v.empty()) continue;
    // longest CTAs first
    const auto cost = [](const DirectGroup& g) {
      return g.kb_split * (g.tiles > 1 ? 8 : g.width / 32);
    };
    std::stable_sort(v.begin(), v.end(),
                     [&](const DirectGroup& x, const DirectGroup& y) {
                       return cost(x) > cost(y);
                     });
    int units = 0;
    for (DirectGroup& g : v) {
      g.unit_begin = units;
      units += g.tiles * ((g.nkb + g.kb_split - 1) / g.kb_split);
    }
    direct_units[m] = units;
  }
  // longest CTAs first
  std::stable_sort(groups.begin(), groups.end(),
                   [](const GramGroup& x, const GramGroup& y) {
                     return x.kb_split * (x.nga > 2 ? 2 : 1) >
                            y.kb_split * (y.nga > 2 ? 2 : 1);
                   });
  int units = 0;
  for (GramGroup& g : groups) {
    g.unit_begin = units;
    units += g.tiles * ((g.nkb + g.kb_split - 1) / g.kb_split);
  }
  KFAC_CUDA(cudaMemcpyAsync(dev_maps, maps.data(), n * sizeof(Map),
                            cudaMemcpyHostToDevice, stream));
  for (int m = 0; m < 2; ++m) {
    if (stage[m].empty()) continue;
    void* dev = nullptr;
    rc = upload(stage[m].data(), stage[m].size() * sizeof(StageJob), stream,
                &dev);
    if (rc != KFAC_OK) return rc;
    const int grid = std::min(sitems[m], sm_count() * 4);
    if (m == 0)
      stage_cols_kernel<<<grid, 256, 0, stream>>>(
          static_cast<const StageJob*>(dev), (int)stage[m].size(), sitems[m]);
    else
      stage_rows_kernel<<<grid, 256, 0, stream>>>(
          static_cast<const StageJob*>(dev), (int)stage[m].size(), sitems[m]);
    KFAC_LAUNCH_CHECK(m == 0 ? "stage_cols_kernel" : "stage_rows_kernel");
  }
  void* dev = nullptr;
  if (units > 0) {
    rc = upload(groups.data(), groups.size() * sizeof(GramGroup), stream, &dev);
    if (rc != KFAC_OK) return rc;
    gram_kernel<<<units, GR_THREADS, GR_SMEM, stream>>>(
        static_cast<const GramGroup*>(dev), (int)groups.size());
    KFAC_LAUNCH_CHECK("gram_kernel");
  }
  for (int m = 0; m < 2; ++m) {
    if (direct[m].empty()) continue;
    rc = upload(direct[m].data(), direct[m].size() * sizeof(DirectGroup),
                stream, &dev);
    if (rc != KFAC_OK) return rc;
    const DirectGroup* d_groups = static_cast<const DirectGroup*>(dev);
    const int n_groups = (int)direct[m].size();
    if (m == 0)
      direct_kernel<false><<<direct_units[m], DR_THREADS, DR_SMEM, stream>>>(
          d_groups, n_groups);
    else
      direct_kernel<true><<<direct_units[m], DR_THREADS, DR_SMEM, stream>>>(
          d_groups, n_groups);
    KFAC_LAUNCH_CHECK("direct_kernel");
  }
  for (int w = 0; w < 2; ++w) {
    if (outs[w].empty()) continue;
    rc = upload(outs[w].data(), outs[w].size() * sizeof(GramOut), stream, &dev);
    if (rc != KFAC_OK) return rc;
    const GramOut* d_outs = static_cast<const GramOut*>(dev);
    if (w == 0)
      gram_reduce_kernel<<<oitems[w], 256, 0, stream>>>(d_outs,
                                                        (int)outs[w].size());
    else
      gram_expand_kernel<<<oitems[w], kXThreads, kXSmem, stream>>>(
          d_outs, (int)outs[w].size());
    KFAC_LAUNCH_CHECK(w == 0 ? "gram_reduce_kernel" : "gram_expand_kernel");
  }
  return KFAC_OK;
}

int run_factor_group_gram(int count, const FactorJob* jobs, void* workspace,
                          size_t workspace_bytes, cudaStream_t stream) {
  if (count <= 0) return KFAC_OK;
  int rc = gram_prepare();
  if (rc != KFAC_OK) return rc;
  EncodeTiledFn encode = nullptr;
  rc = encode_tiled_fn(&encode);
  if (rc != KFAC_OK) return rc;
  std::vector<JobPlan> plans(count);
  for (int i = 0; i < count; ++i) plan_job(jobs[i], plans[i]);
  const size_t need = plans_bytes(plans);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(KFAC_ERR_WORKSPACE,
                "factor: workspace of %zu bytes needed, %zu given", need,
                workspace_bytes);
  for (size_t b = 0, e; b < plans.size(); b = e) {
    e = batch_end(plans, b);
    rc = gram_batch(jobs, plans, b, e, static_cast<char*>(workspace), encode,
                    stream);
    if (rc != KFAC_OK) return rc;
  }
  return KFAC_OK;
}

int gram_status_read(int* out) {
  KFAC_CUDA(cudaMemcpyFromSymbol(out, g_gram_status, sizeof(int)));
  return KFAC_OK;
}

}  // namespace kfac
