// Factor builds (C = alpha X^T X + beta C) on the tensor cores for sm_100a:
// tc_pair_kernel, 256 x 256 tiles, operands gathered from global memory
// (strided views or im2col patches of an NCHW tensor) and split into two bf16
// terms (kind::f16 MMAs, fp32 accumulators in tensor memory), the im2col gather
// laid out with lanes along k.  Every barrier wait is bounded; a wait that
// runs out raises a status word instead of hanging.
#include <algorithm>
#include <mutex>
#include <vector>

#include "gemm_simt.cuh"
#include "tc_common.cuh"

namespace kfac {

constexpr int TC_BN = 256;
constexpr int TC_BK = 32;
constexpr int TC_EPI_PITCH = TC_BN + 1;         // floats
constexpr int TC_TMEM_COLS = 2 * TC_BN;          // two 128-row accumulators

static __device__ int g_tc_status = 0;

// Bounded wait on a phase parity; false if the limit ran out or the CTA is
// already aborting (the status word behind kfac_tc_status is then set).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar,
                                          unsigned parity,
                                          volatile int* abort_flag) {
  return mbar_wait_status(bar, parity, abort_flag, &g_tc_status);
}

// Sources of constant columns: rows of the tile that lie beyond the operand
// read zeros, the appended bias column reads ones; both without branches in
// the hot loop (their address multiplier is 0).
static __device__ __align__(256) float g_zero_page[64];
static __device__ __align__(256) float g_ones_page[64] = {
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};

// A producer task of a strided operand: everything that does not change with k
// is computed once; the element address is
//     p + (long long)o_j * m        (one multiply-add per element)
// where o_j is the k-dependent offset shared by all tasks of the thread.
struct PTask {
  const char* p;    // column base (or the zero / ones page), as bytes
  int m;            // byte multiplier of the k-dependent offset (0 for pages)
  unsigned soff;    // swizzled byte offset inside the stage, ~0u: idle task
};

// Position of a thread's chunk (4 consecutive k) in an operand's row space,
// kept incrementally from k-block to k-block so that the hot loop has no
// integer division.
struct KState {
  int k;           // first k of the chunk (contractions are < 2^31 long)
  int a, b, c;     // strided with a period: k = a * period + b
                   // im2col: k = (a * Ho + b) * Wo + c
};

template <bool IM2COL>
__device__ __forceinline__ void kstate_init(const Operand& op, long long k,
                                            KState& s) {
  s.k = (int)k;
  s.a = s.b = s.c = 0;
  if (IM2COL) {
    const int how = op.Ho * op.Wo;
    s.a = (int)(k / how);
    const int rem = (int)(k - (long long)s.a * how);
    s.b = rem / op.Wo;
    s.c = rem - s.b * op.Wo;
  } else if (op.period != 1) {
    s.a = (int)(k / op.period);
    s.b = (int)(k - (long long)s.a * op.period);
  }
}

template <bool IM2COL, int BK = TC_BK>
__device__ __forceinline__ void kstate_advance(const Operand& op, KState& s) {
  s.k += BK;
  if (IM2COL) {
    s.c += BK;
    while (s.c >= op.Wo) {
      s.c -= op.Wo;
      if (++s.b >= op.Ho) { s.b = 0; ++s.a; }
    }
  } else if (op.period != 1) {
    s.b += BK;
    while (s.b >= op.period) { s.b -= op.period; ++s.a; }
  }
}

// Element offsets of a chunk's 4 k (strided: row offsets; im2col: pixel
// offsets of an unpadded convolution -- a padded input is copied into a
// zero-bordered buffer first, so every tap of every pixel is in range).
// With TAILS, offsets of k at or beyond kend are 0 (a legal address; the
// value is zeroed after the load).
template <bool IM2COL, bool TAILS, int J = 4>
__device__ __forceinline__ void tc_koffsets(const Operand& op,
                                            const KState& ks, int kend,
                                            int o[J]) {
  const int k = ks.k;
  if (IM2COL) {
    int n = ks.a, oy = ks.b, ox = ks.c;
    const int chw = op.C * op.H * op.W;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      o[j] = n * chw + oy * op.st * op.W + ox * op.st;
      if (TAILS && k + j >= kend) o[j] = 0;
      if (++ox >= op.Wo) {
        ox = 0;
        if (++oy >= op.Ho) { oy = 0; ++n; }
      }
    }
    return;
  }
  if (op.period == 1) {
#pragma unroll
    for (int j = 0; j < J; ++j) o[j] = k + j;
  } else {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      int q = ks.a, r = ks.b + j;
      while (r >= op.period) { r -= op.period; ++q; }
      o[j] = (int)((long long)q * op.s_outer + (long long)r * op.s_inner);
    }
  }
  if (TAILS) {
#pragma unroll
    for (int j = 0; j < J; ++j) if (k + j >= kend) o[j] = 0;
  }
}

// True when every 16-byte chunk of a k-contiguous strided operand is aligned
// and contiguous for k-blocks that start at kbeg (uniform for the tile).
__device__ __forceinline__ bool tc_operand_vec(const Operand& op,
                                               long long kbeg) {
  if (op.mode != 0 || !op.kfast) return false;
  if ((reinterpret_cast<uintptr_t>(op.base) & 15) != 0) return false;
  if ((op.s_col & 3) != 0 || (kbeg & 3) != 0) return false;
  if (op.extra_idx >= 0 && op.extra != nullptr) return false;
  if (op.period == 1) return op.s_outer == 1;
  return (op.period & 3) == 0 && (op.s_outer & 3) == 0 && op.s_inner == 1;
}

// Lower-triangular enumeration with 128-row x 256-column tiles: tile (bi, bj)
// exists iff 2 * bj <= bi.  Tiles before row bi: a(a+1) for bi = 2a, (a+1)^2
// for bi = 2a + 1.
__device__ __forceinline__ void tc_tri_tile(int t, int& bi, int& bj) {
  int a = (int)sqrtf((float)t);
  while ((a + 1) * (a + 1) <= t) ++a;
  while (a * a > t) --a;
  if (t < a * (a + 1)) {
    bi = 2 * a - 1;
    bj = t - a * a;
  } else {
    bi = 2 * a;
    bj = t - a * (a + 1);
  }
}

// ---- split-bf16 operands (factor builds) ----
// x = hi + lo with hi = bf16(x), lo = bf16(x - hi): 16 significant bits,
// products hi*hi + hi*lo + lo*hi are exact in the fp32 accumulator.  Halves
// the shared-memory bytes per k of the split-TF32 scheme (stores and tensor
// core operand reads), which is what bounds the tile kernels.
__device__ __forceinline__ void tc_mma_bf16(unsigned tmem_d,
                                            unsigned long long da,
                                            unsigned long long db,
                                            unsigned idesc,
                                            unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void store_split_bf16(unsigned hi_addr,
                                                 unsigned lo_addr, float4 a,
                                                 float4 b) {
  unsigned h[4], l[4];
  split_bf16x2(a.x, a.y, h[0], l[0]);
  split_bf16x2(a.z, a.w, h[1], l[1]);
  split_bf16x2(b.x, b.y, h[2], l[2]);
  split_bf16x2(b.z, b.w, h[3], l[3]);
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hi_addr),
               "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
               : "memory");
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lo_addr),
               "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3])
               : "memory");
}

// ============================================================ X^T X, 256 x 256
// Factor builds (C = alpha X^T X + beta C, lower tiles, mirrored) use a CTA
// tile of 256 x 256: two 128-row accumulators that share one staged set of
// 256 B rows, so a k-block needs 512 operand rows for 65536 outputs instead of
// 384 for 32768; on diagonal tiles the A rows are the B rows and only those
// are staged.  Operands are split into two bf16 terms (see above).  A stage
// holds 32 k as 64-byte rows under the 64-byte swizzle ([A hi][B hi][A lo]
// [B lo], 16 KB each), three stages are in flight, and each 128 x 256
// accumulator takes 256 of the 512 tensor-memory columns (cross terms and
// hi*hi go into the same accumulator, cross terms first).  Partial tiles of
// split contractions keep the 128 x 256 numbering of tc_tri_tile, so
// tc_reduce_kernel serves both kernels.
constexpr int PK_BK = 32;
constexpr int PK_ROWS = 256;                         // rows per operand tile
constexpr int PK_TILE_BYTES = PK_ROWS * PK_BK * 2;   // 16 KB of bf16
constexpr int PK_LO_OFF = 2 * PK_TILE_BYTES;
constexpr int PK_STAGE_BYTES = 4 * PK_TILE_BYTES;    // 64 KB
constexpr int PK_STAGES = 3;
constexpr int PK_PRODUCERS = 512;
constexpr int PK_PWARPS = PK_PRODUCERS / 32;
constexpr int PK_THREADS = PK_PRODUCERS + 32;
constexpr int PK_NTASK = 2 * PK_ROWS * (PK_BK / 8) / PK_PRODUCERS;   // 4

struct __align__(16) PkControl {
  unsigned long long full[PK_STAGES];
  unsigned long long empty[PK_STAGES];
  unsigned long long accum;
  unsigned tmem_base;
  volatile int abort_flag;
  int found;
  GemmDesc desc;
};
constexpr int PK_SMEM_BYTES =
    PK_STAGES * PK_STAGE_BYTES + ((int)sizeof(PkControl) + 1023) / 1024 * 1024 +
    1024;
static_assert(PK_SMEM_BYTES <= 227 * 1024, "pair kernel shared memory");
static_assert(TC_BM * TC_EPI_PITCH * 4 <= PK_STAGES * PK_STAGE_BYTES,
              "epilogue staging tile");

__device__ __forceinline__ unsigned long long pk_smem_desc(unsigned addr) {
  // K-major, 64-byte swizzle: 8-row groups 512 bytes apart.
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFF) >> 4);         // start address
  d |= (unsigned long long)1 << 16;                         // LBO (unused)
  d |= (unsigned long long)(512 >> 4) << 32;                // SBO
  d |= (unsigned long long)1 << 46;                         // descriptor version
  d |= (unsigned long long)4 << 61;                         // SWIZZLE_64B
  return d;
}

// Pair (Bi, Bj), Bj <= Bi, of 256-row blocks from its index Bi(Bi+1)/2 + Bj.
__device__ __forceinline__ void pk_pair(int t, int& Bi, int& Bj) {
  int a = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((a + 1) * (a + 2) / 2 <= t) ++a;
  while (a * (a + 1) / 2 > t) --a;
  Bi = a;
  Bj = t - a * (a + 1) / 2;
}

// STAGED: the operand comes from the bf16 planes of the staging pass through
// TMA: one thread issues, per k-block, a 32 k x 256 row box of each plane for
// the B rows (and the A rows off the diagonal) straight into the stage, in
// the 64-byte-swizzled K-major layout; rows past d and k past K arrive as
// zeros.  The other producer warps wait for the epilogue.
__device__ __forceinline__ void tma_load_2d(unsigned dst, const void* tmap,
                                            int x, int y, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::"
      "complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

template <bool IM2COL, bool TAILS, bool STAGED = false>
__global__ void __launch_bounds__(PK_THREADS, 1)
tc_pair_kernel(const GemmDesc* __restrict__ descs, int ndesc,
               const __grid_constant__ GemmDesc inline_desc) {
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  PkControl* ctl =
      reinterpret_cast<PkControl*>(smem + PK_STAGES * PK_STAGE_BYTES);
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x;
  {
    const GemmDesc* src = &inline_desc;
    if (descs != nullptr) {
      for (int i = tid; i < ndesc; i += PK_THREADS) {
        const int lo = descs[i].tile_begin;
        const int hi = (i + 1 < ndesc) ? descs[i + 1].tile_begin : 0x7fffffff;
        if (lo <= tile && tile < hi) ctl->found = i;
      }
      __syncthreads();
      src = descs + ctl->found;
    }
    const int* s = reinterpret_cast<const int*>(src);
    int* d = reinterpret_cast<int*>(&ctl->desc);
    for (int i = tid; i < (int)(sizeof(GemmDesc) / sizeof(int)); i += PK_THREADS)
      d[i] = s[i];
  }
  if (tid == 0) {
    for (int s = 0; s < PK_STAGES; ++s) {
      mbar_init(&ctl->full[s], STAGED ? 1 : PK_PWARPS);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->accum, 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == PK_PWARPS) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(TC_TMEM_COLS)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const GemmDesc& g = ctl->desc;
  const unsigned tmem = ctl->tmem_base;
  const int nblk = (g.M + PK_ROWS - 1) / PK_ROWS;   // 256-row blocks
  const int npairs = nblk * (nblk + 1) / 2;
  int lt = tile - g.tile_begin, split = 0;
  if (g.splits > 1) {
    split = lt / npairs;
    lt -= split * npairs;
  }
  int Bi, Bj;
  pk_pair(lt, Bi, Bj);
  const int m0 = Bi * PK_ROWS, n0 = Bj * PK_ROWS;
  const bool share = Bi == Bj;
  const int n_valid = min(PK_ROWS, g.N - n0);
  const int n_inst = (n_valid + 15) & ~15;
  const int rows_a = min(PK_ROWS, g.M - m0);
  const bool two = rows_a > TC_BM;                  // second accumulator used
  long long kbeg = 0, kend = g.K;
  if (g.splits > 1) {
    kbeg = (long long)split * g.k_per_split;
    kend = min(g.K, kbeg + g.k_per_split);
  }
  const int nkb = kend > kbeg ? (int)((kend - kbeg + PK_BK - 1) / PK_BK) : 0;

  if (STAGED && warp < PK_PWARPS) {
    // ===================== TMA producer =====================
    if (tid == 0) {
      // the tensor maps were written to device memory by a copy that
      // precedes this launch in the stream
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;"
                   ::"l"(g.tmap_hi) : "memory");
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;"
                   ::"l"(g.tmap_lo) : "memory");
      const unsigned bytes = (share ? 2u : 4u) * PK_TILE_BYTES;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % PK_STAGES;
        if (kb >= PK_STAGES) {
          if (!mbar_wait(&ctl->empty[s], ((kb / PK_STAGES) - 1) & 1,
                         &ctl->abort_flag))
            break;
        }
        const unsigned bar = smem_u32(&ctl->full[s]);
        asm volatile(
            "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
            ::"r"(bar), "r"(bytes) : "memory");
        const unsigned st = smem_u32(smem + s * PK_STAGE_BYTES);
        const int k0 = (int)kbeg + kb * PK_BK;
        tma_load_2d(st + PK_TILE_BYTES, g.tmap_hi, k0, n0, bar);
        tma_load_2d(st + PK_LO_OFF + PK_TILE_BYTES, g.tmap_lo, k0, n0, bar);
        if (!share) {
          tma_load_2d(st, g.tmap_hi, k0, m0, bar);
          tma_load_2d(st + PK_LO_OFF, g.tmap_lo, k0, m0, bar);
        }
      }
    }
  } else if (warp < PK_PWARPS) {
    // ===================== producers =====================
    const Operand X = g.A;                          // A and B are the same
    if (IM2COL) {
      // ---- im2col gather: lanes walk k.  Half a warp reads 32 consecutive
      // output pixels (16 lanes x 2) of one patch-matrix column, the other
      // half the same pixels of the next column: a load instruction touches
      // two to four cache lines instead of up to 32 sectors.  Warp w owns
      // rows 2w + 32 j + h (j = 0..15, h = lane / 16; j < 8: A rows) of the
      // 512 staged rows; a thread keeps the 16 row offsets in registers for
      // the whole tile, loads pixels (k, k+1) of each row per k-block and
      // packs them into one bf16x2 word per tile, so a warp's store covers
      // 128 contiguous bytes.  Rows past the operand's edge read column 0:
      // their products are never stored.  The appended ones column is
      // patched in after the loads.
      const int h = lane >> 4, kp = lane & 15;
      int off[16];
      unsigned ones = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int R = 2 * warp + 32 * j + h;
        const bool is_a = j < 8;
        const int c = (is_a ? m0 : n0 - PK_ROWS) + R;
        int o = 0;
        if (c < X.ncols) {
          const int kk = X.ks * X.ks;
          const int ch = c / kk;
          const int r = c - ch * kk;
          const int ky = r / X.ks;
          const int kx = r - ky * X.ks;
          o = ch * X.H * X.W + ky * X.W + kx;
        } else if (c == X.extra_idx) {
          ones |= 1u << j;
        }
        off[j] = o;
      }
      const int kend_i = (int)kend;
      KState ks;
      kstate_init<true>(X, kbeg + 2 * kp, ks);
      const int chw = X.C * X.H * X.W, sw = X.st * X.W;
      const unsigned lane_off = (unsigned)((((kp >> 2) ^ (warp & 3)) << 4) +
                                           4 * (kp & 3) + h * 64 + warp * 128);
      // offset of the 1024-byte-aligned stage area inside the dynamic array
      const unsigned smem_skew = smem_u32(smem) - smem_u32(tc_smem_raw);
      const int j0 = share ? 8 : 0;
      float x[32];
      for (int kb = 0; kb <= nkb; ++kb) {
        if (kb > 0) {
          const int pb = kb - 1;
          const int s = pb % PK_STAGES;
          if (pb >= PK_STAGES) {
            if (!mbar_wait(&ctl->empty[s], ((pb / PK_STAGES) - 1) & 1,
                           &ctl->abort_flag))
              break;
          }
          // plain stores through a pointer into the shared array: the
          // per-row offsets (2048 j) fold into the instruction's immediate
          unsigned* st = reinterpret_cast<unsigned*>(
              tc_smem_raw + smem_skew + s * PK_STAGE_BYTES + lane_off);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j < j0) continue;
            unsigned hi, lo;
            split_bf16x2(x[2 * j], x[2 * j + 1], hi, lo);
            st[512 * j] = hi;
            st[PK_LO_OFF / 4 + 512 * j] = lo;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->full[s]);
        }
        if (kb < nkb) {
          // pixel offsets of k and k + 1 (k + 1 may start the next image row)
          const bool live0 = !TAILS || ks.k < kend_i;
          const bool live1 = !TAILS || ks.k + 1 < kend_i;
          int o0 = ks.a * chw + ks.b * sw + ks.c * X.st;
          int o1 = o0 + X.st;
          if (ks.c + 1 >= X.Wo) {
            o1 = (ks.b + 1 >= X.Ho) ? (ks.a + 1) * chw
                                    : ks.a * chw + (ks.b + 1) * sw;
          }
          if (!live0) o0 = 0;
          if (!live1) o1 = 0;
          const float* p0 = X.base + o0;
          const float* p1 = X.base + o1;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j < j0) continue;
            x[2 * j] = p0[off[j]];
            x[2 * j + 1] = p1[off[j]];
          }
          if (ones) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (ones & (1u << j)) x[2 * j] = x[2 * j + 1] = 1.f;
          }
          if (TAILS && !live1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (!live0) x[2 * j] = 0.f;
              x[2 * j + 1] = 0.f;
            }
          }
          kstate_advance<true, PK_BK>(X, ks);
        }
      }
    } else {
      const bool kf = IM2COL || X.kfast;
      // per task: 128 of the 512 (A then B) rows; a warp covers 8 rows x 4
      // chunks of a k-contiguous operand, or one chunk of 32 rows of a
      // column-contiguous one
      PTask task[PK_NTASK];
  #pragma unroll
      for (int t = 0; t < PK_NTASK; ++t) {
        const bool is_a = t < PK_NTASK / 2;
        const int band_row = kf ? warp * 8 + (lane >> 2) : 32 * (warp >> 2) + lane;
        const int row = 128 * t + band_row - (is_a ? 0 : PK_ROWS);
        const int rows = is_a ? (share ? 0 : rows_a) : n_inst;
        const int chunk = kf ? (lane & 3) : (warp & 3);
        PTask v;
        v.soff = row < rows
                     ? (unsigned)((is_a ? 0 : PK_TILE_BYTES) + row * 64 +
                                  ((chunk ^ ((row >> 1) & 3)) << 4))
                     : ~0u;
        const float* p = g_zero_page;
        int m = 0;
        if (row < rows) {
          const int c = (is_a ? m0 : n0) + row;
          if (c < X.ncols) {
            p = X.base + (long long)c * X.s_col;
            m = X.period == 1 ? (int)X.s_outer : 1;
          } else if (c == X.extra_idx) {
            if (X.extra) { p = X.extra; m = 1; }
            else p = g_ones_page;
          }
        }
        v.p = reinterpret_cast<const char*>(p);
        v.m = m * 4;
        task[t] = v;
      }
      const int kend_i = (int)kend;
      KState ks;
      kstate_init<IM2COL>(X, kbeg + 8 * (kf ? (lane & 3) : (warp & 3)), ks);
      const unsigned smem_base = smem_u32(smem);
      const bool vec = !IM2COL && tc_operand_vec(X, kbeg);
      // a task is 8 consecutive k of one row: 16 bytes of each bf16 tile
      float4 v[PK_NTASK][2];
      for (int kb = 0; kb <= nkb; ++kb) {
        if (kb > 0) {
          const int pb = kb - 1;
          const int s = pb % PK_STAGES;
          if (pb >= PK_STAGES) {
            if (!mbar_wait(&ctl->empty[s], ((pb / PK_STAGES) - 1) & 1,
                           &ctl->abort_flag))
              break;
          }
          const unsigned st = smem_base + s * PK_STAGE_BYTES;
  #pragma unroll
          for (int t = 0; t < PK_NTASK; ++t)
            if (task[t].soff != ~0u)
              store_split_bf16(st + task[t].soff, st + PK_LO_OFF + task[t].soff,
                               v[t][0], v[t][1]);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->full[s]);
        }
        if (kb < nkb) {
          int o[8];
          tc_koffsets<IM2COL, TAILS, 8>(X, ks, kend_i, o);
          const int k = ks.k;
          const bool tail = TAILS && (k + 7 >= kend_i);
          if (vec && !tail) {
  #pragma unroll
            for (int t = 0; t < PK_NTASK; ++t)
              if (task[t].soff != ~0u) {
                v[t][0] = *reinterpret_cast<const float4*>(
                    task[t].p + (long long)o[0] * task[t].m);
                v[t][1] = *reinterpret_cast<const float4*>(
                    task[t].p + (long long)o[4] * task[t].m);
              }
          } else {
  #pragma unroll
            for (int t = 0; t < PK_NTASK; ++t) {
              if (task[t].soff == ~0u) continue;
              v[t][0].x = *reinterpret_cast<const float*>(task[t].p + (long long)o[0] * task[t].m);
              v[t][0].y = *reinterpret_cast<const float*>(task[t].p + (long long)o[1] * task[t].m);
              v[t][0].z = *reinterpret_cast<const float*>(task[t].p + (long long)o[2] * task[t].m);
              v[t][0].w = *reinterpret_cast<const float*>(task[t].p + (long long)o[3] * task[t].m);
              v[t][1].x = *reinterpret_cast<const float*>(task[t].p + (long long)o[4] * task[t].m);
              v[t][1].y = *reinterpret_cast<const float*>(task[t].p + (long long)o[5] * task[t].m);
              v[t][1].z = *reinterpret_cast<const float*>(task[t].p + (long long)o[6] * task[t].m);
              v[t][1].w = *reinterpret_cast<const float*>(task[t].p + (long long)o[7] * task[t].m);
            }
          }
          if (tail) {
  #pragma unroll
            for (int t = 0; t < PK_NTASK; ++t) {
              if (k + 0 >= kend_i) v[t][0].x = 0.f;
              if (k + 1 >= kend_i) v[t][0].y = 0.f;
              if (k + 2 >= kend_i) v[t][0].z = 0.f;
              if (k + 3 >= kend_i) v[t][0].w = 0.f;
              if (k + 4 >= kend_i) v[t][1].x = 0.f;
              if (k + 5 >= kend_i) v[t][1].y = 0.f;
              if (k + 6 >= kend_i) v[t][1].z = 0.f;
              if (k + 7 >= kend_i) v[t][1].w = 0.f;
            }
          }
          kstate_advance<IM2COL, PK_BK>(X, ks);
        }
      }
    }
  } else {
    // ===================== MMA issuer =====================
    if (elect_one()) {
      const unsigned idesc = tc_bf16_desc(n_inst);
      const unsigned a_off = share ? (unsigned)PK_TILE_BYTES : 0u;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % PK_STAGES;
        if (!mbar_wait(&ctl->full[s], (kb / PK_STAGES) & 1, &ctl->abort_flag))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned sa = smem_u32(smem + s * PK_STAGE_BYTES);
        const unsigned long long a_hi = pk_smem_desc(sa + a_off);
        const unsigned long long a_lo = pk_smem_desc(sa + PK_LO_OFF + a_off);
        const unsigned long long b_hi = pk_smem_desc(sa + PK_TILE_BYTES);
        const unsigned long long b_lo =
            pk_smem_desc(sa + PK_LO_OFF + PK_TILE_BYTES);
        // second accumulator: A rows 128..255 start 128 * 64 bytes later
        const unsigned long long up = (unsigned long long)(TC_BM * 64 >> 4);
#pragma unroll
        for (int kk = 0; kk < PK_BK / 16; ++kk) {
          // 16 bf16 = 32 bytes per MMA along k
          const unsigned long long adv = (unsigned long long)(kk * 32 >> 4);
          const unsigned acc = (kb | kk) != 0;
          tc_mma_bf16(tmem, a_lo + adv, b_hi + adv, idesc, acc);
          tc_mma_bf16(tmem, a_hi + adv, b_lo + adv, idesc, 1);
          tc_mma_bf16(tmem, a_hi + adv, b_hi + adv, idesc, 1);
          if (two) {
            tc_mma_bf16(tmem + TC_BN, a_lo + up + adv, b_hi + adv, idesc, acc);
            tc_mma_bf16(tmem + TC_BN, a_hi + up + adv, b_lo + adv, idesc, 1);
            tc_mma_bf16(tmem + TC_BN, a_hi + up + adv, b_hi + adv, idesc, 1);
          }
        }
        tc_commit(&ctl->empty[s]);
      }
      tc_commit(&ctl->accum);
    }
    __syncwarp();
  }

  // ===================== epilogue =====================
  if (warp < PK_PWARPS) {
    float* stage = reinterpret_cast<float*>(smem);
    if (nkb > 0) {
      mbar_wait(&ctl->accum, 0, &ctl->abort_flag);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    asm volatile("bar.sync 1, %0;" ::"r"(PK_PRODUCERS) : "memory");
    const bool dead = ctl->abort_flag != 0;        // uniform after the barrier
    const float alpha = g.alpha, beta = g.beta;
    const int q = warp & 3, h = warp >> 2;
    for (int tt = 0; tt < (two ? 2 : 1) && !dead; ++tt) {
      const int m0t = m0 + TC_BM * tt;
      const int m_valid = min(TC_BM, g.M - m0t);
      const int nv = min(n_valid, m0t + TC_BM - n0);   // lower triangle
      const int row = q * 32 + lane;
      for (int c0 = h * 16; c0 < n_inst; c0 += 16 * (PK_PWARPS / 4)) {
        float v[16];
        if (nkb > 0) {
          tc_ld16(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(TC_BN * tt + c0), v);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) stage[row * TC_EPI_PITCH + c0 + i] = v[i];
      }
      asm volatile("bar.sync 1, %0;" ::"r"(PK_PRODUCERS) : "memory");
      if (g.splits > 1) {
        // 128 x 256 numbering: row block 2 Bi + tt, column block Bj
        const int lt128 = (tt == 0 ? Bi * (Bi + 1) : (Bi + 1) * (Bi + 1)) + Bj;
        float* p = g.partial +
                   ((long long)split * g.ntiles + lt128) * (TC_BM * TC_BN);
        for (int r = warp; r < TC_BM; r += PK_PWARPS)
          for (int c = lane; c < n_inst; c += 32)
            p[r * TC_BN + c] = stage[r * TC_EPI_PITCH + c];
      } else {
        for (int r = warp; r < m_valid; r += PK_PWARPS) {
          const int gr = m0t + r;
          float* crow = g.C + (long long)gr * g.ldc + n0;
          const int cend = min(nv, gr - n0 + 1);
          float old[TC_BN / 32];
          if (beta != 0.f) {
#pragma unroll
            for (int i = 0; i < TC_BN / 32; ++i) {
              const int c = lane + 32 * i;
              old[i] = c < cend ? crow[c] : 0.f;
            }
          }
#pragma unroll
          for (int i = 0; i < TC_BN / 32; ++i) {
            const int c = lane + 32 * i;
            if (c < cend) {
              float v = alpha * stage[r * TC_EPI_PITCH + c];
              if (beta != 0.f) v += beta * old[i];
              crow[c] = v;
              stage[r * TC_EPI_PITCH + c] = v;
            }
          }
        }
        asm volatile("bar.sync 1, %0;" ::"r"(PK_PRODUCERS) : "memory");
        for (int c = warp; c < nv; c += PK_PWARPS) {
          const int gc = n0 + c;
          for (int r = lane; r < m_valid; r += 32) {
            const int gr = m0t + r;
            if (gc < gr)
              g.C[(long long)gc * g.ldc + gr] = stage[r * TC_EPI_PITCH + c];
          }
        }
      }
      // the second accumulator reuses the staging tile
      asm volatile("bar.sync 1, %0;" ::"r"(PK_PRODUCERS) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == PK_PWARPS) tc_release(tmem, TC_TMEM_COLS, ctl->abort_flag != 0);
}


// Copies of NCHW tensors into buffers with a zero border of `pad` pixels.
// The zero-bordered copies of a grouped factor build in one launch: a work
// item is a run of kPadRun output elements of one job, items are numbered job
// after job, and a block finds its job by bisection in a shared-memory copy of
// the first item of every job.  32 images of 3 x 224 x 224: 105 us with a plane
// per item (96 blocks, one load in flight a thread), 17 now.
struct PadJob {
  const float* src;
  float* dst;
  long long planes;
  int h, w, pad;
  int item_begin;   // first work item of this job
  int nhwc;         // source is channels-last: items are 32 x 32 transposes
  int C;            // channels (channels-last source)
};

constexpr int kPadJobsMax = 256;
constexpr int kPadRun = 4096;      // output elements per item (NCHW source)

__global__ void __launch_bounds__(256)
pad_copy_group_kernel(const PadJob* __restrict__ jobs, int njobs,
                      int total_items) {
  __shared__ int s_begin[kPadJobsMax];
  __shared__ float tile[32][33];
  for (int i = threadIdx.x; i < njobs; i += blockDim.x)
    s_begin[i] = jobs[i].item_begin;
  __syncthreads();
  for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_begin[mid] <= item) lo = mid; else hi = mid - 1;
    }
    const PadJob j = jobs[lo];
    const int wp = j.w + 2 * j.pad, per = (j.h + 2 * j.pad) * wp;
    if (j.nhwc) {
      // (n, h, w, c) -> zero-bordered (n, c, h + 2p, w + 2p): a 32-pixel x
      // 32-channel tile is read along c and written along the pixels; the
      // border was cleared before the launch
      const int hw = j.h * j.w;
      const int ct = (j.C + 31) >> 5, qt = (hw + 31) >> 5;
      int t = item - j.item_begin;
      const int n = t / (ct * qt);
      t -= n * ct * qt;
      const int c0 = (t / qt) << 5, q0 = (t % qt) << 5;
      const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = q0 + ty + 8 * i, c = c0 + tx;
        if (q < hw && c < j.C)
          tile[ty + 8 * i][tx] = j.src[((long long)n * hw + q) * j.C + c];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = c0 + ty + 8 * i, q = q0 + tx;
        if (c < j.C && q < hw) {
          const int y = q / j.w, x = q - y * j.w;
          j.dst[((long long)n * j.C + c) * per + (y + j.pad) * wp + x + j.pad] =
              tile[tx][ty + 8 * i];
        }
      }
      __syncthreads();
      continue;
    }
    const long long first = (long long)(item - j.item_begin) * kPadRun;
    const int count = (int)min((long long)kPadRun, j.planes * per - first);
    const long long plane0 = first / per;
    const int at = (int)(first - plane0 * per);
    const float* src = j.src + plane0 * j.h * j.w;
    float* dst = j.dst + first;
    for (int e = threadIdx.x; e < count; e += 4 * 256) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = at + e + 256 * u, plane = i / per, k = i - plane * per;
        const int yy = k / wp, y = yy - j.pad, x = k - yy * wp - j.pad;
        const bool in = e + 256 * u < count && (unsigned)y < (unsigned)j.h &&
                        (unsigned)x < (unsigned)j.w;
        v[u] = in ? src[((long long)plane * j.h + y) * j.w + x] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e + 256 * u < count) dst[e + 256 * u] = v[u];
    }
  }
}

struct ReduceItem {     // one output tile whose split partials are summed
  const float* partial; // first split's copy of this tile
  float* out;
  long long sstride;    // elements between consecutive splits
  int d, tile, splits;
  float alpha, beta;
};

// `items` == nullptr: every block works on `single`, the item of tile 0 of one
// factor, and takes tile blockIdx.x of it (a lone factor needs no table in
// device memory, so the call neither allocates nor copies one).
__global__ void __launch_bounds__(256)
tc_reduce_kernel(const ReduceItem* __restrict__ items,
                 const __grid_constant__ ReduceItem single, int chunk) {
  // Four lanes share one output element: lane q sums the splits
  // q, q+4, q+8, ... (always in that order), then the four sums are added in
  // a fixed tree, so the result does not depend on scheduling.  Bound by the
  // latency of its loads: a block takes `chunk` elements of its tile, 64 while
  // that leaves SMs idle (100 352 x 64, 196 splits: 248 us with 1024).
  ReduceItem it = items != nullptr ? items[blockIdx.x] : single;
  if (items == nullptr) {
    it.tile = (int)blockIdx.x;
    it.partial += (long long)blockIdx.x * (TC_BM * TC_BN);
  }
  int bi, bj;
  tc_tri_tile(it.tile, bi, bj);
  const int d = it.d;
  const int m0 = bi * TC_BM, n0 = bj * TC_BN;
  const int rows = min(TC_BM, d - m0);
  const int cols = min(min(TC_BN, d - n0), m0 + TC_BM - n0);
  const int q = threadIdx.x & 3;
  const int total = rows * cols;
  for (int e = blockIdx.y * chunk + (threadIdx.x >> 2);
       e < min(total, (int)(blockIdx.y + 1) * chunk); e += 64) {
    const int r = e / cols, c = e - r * cols;
    const float* p = it.partial + r * TC_BN + c;
    // (eight loads in flight: a narrow factor has hundreds of splits)
    float v[8] = {};
    for (int sp = q; sp < it.splits; sp += 32)
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (sp + 4 * u < it.splits) v[u] += p[(sp + 4 * u) * it.sstride];
    float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    const int gr = m0 + r, gc = n0 + c;
    if (q != 0 || gc > gr) continue;
    float* o = it.out + (long long)gr * d + gc;
    float x = it.alpha * s;
    if (it.beta != 0.f) x += it.beta * (*o);
    *o = x;
    if (gc < gr) it.out[(long long)gc * d + gr] = x;
  }
}

// ------------------------------------------------------------------ host side
static int g_engine = 1;

int tc_tiles(GemmDesc& g) {
  g.tiles_m = (g.M + TC_BM - 1) / TC_BM;
  g.tiles_n = (g.N + TC_BN - 1) / TC_BN;
  if (g.flags & G_LOWER) {
    int nt = g.tiles_m, a = nt / 2;
    return (nt & 1) ? (a + 1) * (a + 1) : a * (a + 1);
  }
  return g.tiles_m * g.tiles_n;
}

int tc_prepare() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  KFAC_CUDA(cudaGetDevice(&dev));
  KFAC_REQUIRE(dev >= 0 && dev < 64, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    KFAC_CUDA(cudaFuncSetAttribute(tc_pair_kernel<false, false, true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PK_SMEM_BYTES));
    KFAC_CUDA(cudaFuncSetAttribute(tc_pair_kernel<false, false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PK_SMEM_BYTES));
    KFAC_CUDA(cudaFuncSetAttribute(tc_pair_kernel<false, true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PK_SMEM_BYTES));
    KFAC_CUDA(cudaFuncSetAttribute(tc_pair_kernel<true, false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PK_SMEM_BYTES));
    KFAC_CUDA(cudaFuncSetAttribute(tc_pair_kernel<true, true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PK_SMEM_BYTES));
    done[dev] = true;
  }
  return KFAC_OK;
}

// True when some k-block of the problem can be cut by the end of its
// contraction range (ranges start at multiples of 128 or of k_per_split, both
// multiples of the k-block).
bool tc_desc_has_tails(const GemmDesc& g) {
  if (g.K % TC_BK != 0) return true;
  if (g.splits > 1 && g.k_per_split % TC_BK != 0) return true;
  return false;
}

struct TcFactorSplit {
  int tiles, splits;
  long long k_per_split;
};

// CTAs that cover the lower tiles of a d x d output once.
static int tc_factor_ctas(int d) {
  const int nblk = (d + PK_ROWS - 1) / PK_ROWS;
  return nblk * (nblk + 1) / 2;
}

static int tc_lower_tiles(int d) {
  GemmDesc g = {};
  g.M = g.N = d;
  g.flags = G_LOWER;
  return tc_tiles(g);
}

// Relative duration of one k-block of a CTA of a d x d factor, in 1/512: a
// CTA stages up to 512 operand rows per k-block, d of them when d <= 256; a
// k-block with few rows still costs about a memory round trip.
static long long tc_block_cost(int d) {
  const int rows = d < 512 ? d : 512;
  return rows < 256 ? 256 : rows;
}

// Split of one factor's contraction.  `chunk` is the cost (k-blocks x
// tc_block_cost) a CTA should own; a CTA keeps at least 16 k-blocks so that
// prologue and epilogue stay amortised, and a contraction is only cut when
// that brings its CTAs closer to the target than leaving it whole (partial
// tiles cost a write, a read and the reduce kernel).
// The tensor core adds each MMA's products into the fp32 accumulator with
// truncation, so a sum of N MMAs drifts by up to about N * 2^-25 of its
// magnitude, all in one direction when the addends share a sign (activation
// factors: products of non-negative values; three MMAs per 16 rows here).
// Measured relative error of 100 352-row factors: 2e-4 when one CTA
// accumulates 1500 k-blocks, 4.7e-5 at 256, 2e-5 at 128.  A CTA therefore
// never accumulates more than this many k-blocks (of 32 rows); the partial
// tiles of longer contractions are summed in fp32 by the reduce kernel, with
// rounding to nearest.  256 keeps the drift at half the 1e-4 bound and costs
// nothing measurable here; 128 costs 15 % of the factor stage with this kernel,
// nothing with those of gram.cu.
long long factor_max_kblocks(long long fallback) {
  static const long long v = [] {
    const char* e = getenv("KFAC_TC_MAX_KBLOCKS");
    return e ? atoll(e) : 0LL;
  }();
  return v >= 16 ? v : fallback;
}

static long long tc_max_kblocks() { return factor_max_kblocks(256); }

long long factor_waves() {
  static const long long v = [] {
    const char* e = getenv("KFAC_TC_WAVES");
    return e ? atoll(e) : 0LL;
  }();
  return v > 0 ? v : 2;
}

static TcFactorSplit tc_split_for(long long rows, int d, long long chunk) {
  TcFactorSplit s;
  s.tiles = tc_lower_tiles(d);
  chunk /= tc_block_cost(d);
  if (chunk < 16) chunk = 16;
  if (chunk > tc_max_kblocks()) chunk = tc_max_kblocks();
  const long long kblocks = (rows + TC_BK - 1) / TC_BK;
  // (the nearest number of splits, none longer than the limit)
  long long sp = std::max((kblocks + chunk / 2) / chunk,
                          (kblocks + tc_max_kblocks() - 1) / tc_max_kblocks());
  if (sp < 1) sp = 1;
  long long kps = (kblocks + sp - 1) / sp * TC_BK;
  s.splits = (int)((rows + kps - 1) / kps);
  if (s.splits < 1) s.splits = 1;
  s.k_per_split = kps;
  return s;
}

static TcFactorSplit tc_factor_split(long long rows, int d) {
  // a factor built on its own: aim at two waves of CTAs
  const int tiles = tc_factor_ctas(d);
  const long long kblocks = (rows + TC_BK - 1) / TC_BK;
  long long want = (2LL * sm_count() + tiles - 1) / tiles;   // splits wanted
  if (tiles >= sm_count()) want = 1;
  long long chunk = (kblocks + want - 1) / want;
  return tc_split_for(rows, d, chunk * tc_block_cost(d));
}

// Factor builds read their operands from the staged bf16 planes through TMA
// (stage.cu) when this is on (kfac_set_factor_staging, initial value from
// KFAC_TC_STAGED, default off) and the caller gives workspace; otherwise the
// producer warps gather and split the operands themselves.
static int g_staged = -1;
bool tc_staged() {
  if (g_staged < 0) {
    const char* e = getenv("KFAC_TC_STAGED");
    g_staged = (e != nullptr && atoi(e) != 0) ? 1 : 0;
  }
  return g_staged != 0;
}

size_t tc_factor_workspace_bytes(long long rows, int d, bool staged) {
  TcFactorSplit s = tc_factor_split(rows, d);
  size_t bytes = (staged && tc_staged()) ? tc_stage_bytes(rows, d) : 0;
  if (s.splits > 1)
    bytes += (size_t)s.splits * s.tiles * TC_BM * TC_BN * sizeof(float);
  return bytes;
}

size_t tc_pad_bytes(const Operand& X, int n, int nhwc) {
  // a staging copy is made for a zero border and / or to turn a channels-last
  // tensor into the NCHW planes the gather walks
  if (X.mode != 1 || (X.pd == 0 && !nhwc)) return 0;
  size_t e = (size_t)n * X.C * (X.H + 2 * X.pd) * (X.W + 2 * X.pd);
  return (e * sizeof(float) + 255) & ~(size_t)255;
}

// k-blocks per CTA for a group of factors: total work spread over ~2 waves.
static long long tc_group_chunk(int count, const FactorJob* jobs) {
  long long work = 0;
  for (int i = 0; i < count; ++i)
    work += (long long)tc_factor_ctas(jobs[i].d) *
            ((jobs[i].rows + TC_BK - 1) / TC_BK) * tc_block_cost(jobs[i].d);
  return work / (factor_waves() * sm_count());
}

static size_t tc_pair_workspace_bytes(int count, const FactorJob* jobs,
                                      bool staged) {
  const long long chunk = tc_group_chunk(count, jobs);
  staged = staged && tc_staged();
  size_t total = 0;
  for (int i = 0; i < count; ++i) {
    total += staged ? tc_stage_bytes(jobs[i].rows, jobs[i].d)
                    : tc_pad_bytes(jobs[i].X, jobs[i].n, jobs[i].nhwc);
    TcFactorSplit s = count == 1 ? tc_factor_split(jobs[i].rows, jobs[i].d)
                                 : tc_split_for(jobs[i].rows, jobs[i].d, chunk);
    if (s.splits > 1)
      total += (size_t)s.splits * s.tiles * TC_BM * TC_BN * sizeof(float);
  }
  return total;
}

// Factors that are built from staged planes (gram.cu), unless the caller chose
// the staging pass of stage.cu or gives no workspace:
//  * 3 x 3 convolutions as shifted products (gram_grid_job; 32 images, us per
//    factor before and now: 64 channels 56 x 56 228 -> 78, 256 channels 14 x 14
//    171 -> 62; 8 images of 64 channels 14 x 14 68 -> 41);
//  * plain operands that TMA reads in place, from a million elements on (below
//    that the launches count: all factors of a 1000-1000-10 network at 128
//    rows 43 us with the gather, 72 us without);
//  * other wide factors, where the gather feeds every element to many tiles
//    (NCHW, 1568 x 2048: 68 -> 27; even at 1000 columns, slower below);
//  * patches of other convolutions unless they have few channels (1x1 / 2, 512
//    channels 28 x 28 channels-last: 84 -> 27; 3x3 / 2, 256 channels 28 x 28:
//    199 -> 155; 3x3 with bias, 37 channels 15 x 15: 75 -> 52; even at 16
//    channels; the 3-channel 7x7 stem 160 against 486).
static bool tc_uses_gram(const FactorJob& job) {
  if (tc_staged()) return false;
  if (gram_grid_job(job)) return true;
  if ((double)job.rows * job.d >= 1e6 && gram_direct_job(job)) return true;
  if (job.X.mode == 1 && job.X.C >= 20) return true;
  return job.d >= 1024 && (double)job.rows * job.d >= 2e6;
}

static void tc_by_feed(int count, const FactorJob* jobs, bool staged,
                       std::vector<FactorJob>& gram,
                       std::vector<FactorJob>& pair) {
  for (int i = 0; i < count; ++i)
    (staged && tc_uses_gram(jobs[i]) ? gram : pair).push_back(jobs[i]);
}

size_t tc_factor_group_workspace_bytes(int count, const FactorJob* jobs,
                                       bool staged) {
  std::vector<FactorJob> gram, pair;
  tc_by_feed(count, jobs, staged, gram, pair);
  // (a lone factor may have to be gathered, see run_factor_group_tc)
  if (count == 1) pair.assign(jobs, jobs + 1);
  return std::max(
      gram_workspace_bytes((int)gram.size(), gram.data()),
      tc_pair_workspace_bytes((int)pair.size(), pair.data(), staged));
}

// Whether calls on this stream are being recorded into a graph.
static bool stream_captures(cudaStream_t stream) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cs != cudaStreamCaptureStatusNone;
}

// Per-device helper stream: the strided and the im2col launch of a grouped
// factor build do not depend on each other, and each has a tail of CTAs that
// leaves SMs idle, so they run side by side (fork / join with events).
struct SideStream {
  cudaStream_t stream;
  cudaEvent_t fork, join;
};

static int tc_side_stream(SideStream** out) {
  static std::mutex mu;
  static SideStream side[64];
  static bool made[64] = {false};
  int dev = 0;
  KFAC_CUDA(cudaGetDevice(&dev));
  KFAC_REQUIRE(dev >= 0 && dev < 64, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!made[dev]) {
    KFAC_CUDA(cudaStreamCreateWithFlags(&side[dev].stream, cudaStreamNonBlocking));
    KFAC_CUDA(cudaEventCreateWithFlags(&side[dev].fork, cudaEventDisableTiming));
    KFAC_CUDA(cudaEventCreateWithFlags(&side[dev].join, cudaEventDisableTiming));
    made[dev] = true;
  }
  *out = &side[dev];
  return KFAC_OK;
}

struct alignas(64) TmapBlob {     // a CUtensorMap, opaque here
  unsigned char b[128];
};

static int run_factor_group_pair(int count, const FactorJob* jobs,
                                 void* workspace, size_t workspace_bytes,
                                 cudaStream_t main_stream, bool staged) {
  cudaStream_t stream = main_stream;
  int rc = tc_prepare();
  if (rc != KFAC_OK) return rc;
  staged = staged && tc_staged();
  const size_t need = tc_pair_workspace_bytes(count, jobs, staged);
  if (need > 0 && (workspace == nullptr || workspace_bytes < need))
    return fail(KFAC_ERR_WORKSPACE,
                "factor: workspace of %zu bytes needed, %zu given", need,
                workspace_bytes);
  const long long chunk = tc_group_chunk(count, jobs);
  char* ws = static_cast<char*>(workspace);

  std::vector<GemmDesc> descs[2];       // [0] strided, [1] im2col
  std::vector<ReduceItem> reduces;
  std::vector<PadJob> pads;
  int pad_items = 0;
  const TmapBlob* dev_maps = nullptr;
  if (staged) {
    // staging pass: X^T of every job as two bf16 planes, two tensor maps each
    std::vector<TmapBlob> maps(2 * (size_t)count);
    rc = tc_stage_group(count, jobs, ws, maps.data(), stream);
    if (rc != KFAC_OK) return rc;
    for (int i = 0; i < count; ++i)
      ws += tc_stage_bytes(jobs[i].rows, jobs[i].d);
    void* dev = nullptr;
    rc = ring_alloc(maps.size() * sizeof(TmapBlob), &dev);
    if (rc != KFAC_OK) return rc;
    KFAC_CUDA(cudaMemcpyAsync(dev, maps.data(), maps.size() * sizeof(TmapBlob),
                              cudaMemcpyHostToDevice, stream));
    dev_maps = static_cast<const TmapBlob*>(dev);
  }
  for (int i = 0; i < count; ++i) {
    const FactorJob& job = jobs[i];
    Operand X = job.X;
    if (!staged && X.mode == 1 && (X.pd > 0 || job.nhwc)) {
      // zero-bordered NCHW copy first; the gather then needs no bounds checks
      const size_t pad_bytes = tc_pad_bytes(X, job.n, job.nhwc);
      float* padded = reinterpret_cast<float*>(ws);
      ws += pad_bytes;
      const long long planes = (long long)job.n * X.C;
      const long long total = planes * (X.H + 2 * X.pd) * (X.W + 2 * X.pd);
      KFAC_REQUIRE(total < (1LL << 31), "factor: padded input too large");
      const int per = (X.H + 2 * X.pd) * (X.W + 2 * X.pd);
      PadJob pj;
      pj.src = X.base;
      pj.dst = padded;
      pj.planes = planes;
      pj.h = X.H;
      pj.w = X.W;
      pj.pad = X.pd;
      pj.item_begin = pad_items;
      pj.nhwc = job.nhwc;
      pj.C = X.C;
      if (job.nhwc) {
        if (X.pd > 0)
          KFAC_CUDA(cudaMemsetAsync(padded, 0, pad_bytes, stream));
        pad_items += job.n * ((X.C + 31) / 32) * ((X.H * X.W + 31) / 32);
      } else {
        pad_items += (int)((planes * per + kPadRun - 1) / kPadRun);
      }
      pads.push_back(pj);
      X.base = padded;
      X.H += 2 * X.pd;
      X.W += 2 * X.pd;
      X.pd = 0;
    }
    TcFactorSplit s = count == 1 ? tc_factor_split(job.rows, job.d)
                                 : tc_split_for(job.rows, job.d, chunk);
    GemmDesc g = {};
    g.A = X;
    g.B = X;
    g.C = job.out;
    g.ldc = job.d;
    g.K = job.rows;
    g.M = job.d;
    g.N = job.d;
    g.alpha = job.alpha;
    g.beta = job.beta;
    g.flags = G_LOWER | G_MIRROR | G_SAME_AB;
    g.ntiles = tc_tiles(g);
    g.splits = s.splits;
    g.k_per_split = s.k_per_split;
    g.partial = nullptr;
    if (staged) {
      g.tmap_hi = dev_maps + 2 * i;
      g.tmap_lo = dev_maps + 2 * i + 1;
    }
    if (s.splits > 1) {
      g.partial = reinterpret_cast<float*>(ws);
      ws += (size_t)s.splits * s.tiles * TC_BM * TC_BN * sizeof(float);
      for (int t = 0; t < s.tiles; ++t) {
        ReduceItem it;
        it.partial = g.partial + (long long)t * (TC_BM * TC_BN);
        it.out = job.out;
        it.sstride = (long long)s.tiles * (TC_BM * TC_BN);
        it.d = job.d;
        it.tile = t;
        it.splits = s.splits;
        it.alpha = job.alpha;
        it.beta = job.beta;
        reduces.push_back(it);
      }
    }
    descs[(X.mode == 1 && !staged) ? 1 : 0].push_back(g);
  }
  for (size_t b = 0; b < pads.size(); b += kPadJobsMax) {
    // (more than kPadJobsMax padded inputs in one group: several launches)
    const int nj = (int)std::min<size_t>(kPadJobsMax, pads.size() - b);
    std::vector<PadJob> part(pads.begin() + b, pads.begin() + b + nj);
    const int first = part[0].item_begin;
    for (PadJob& pj : part) pj.item_begin -= first;
    const int items =
        (b + nj < pads.size() ? pads[b + nj].item_begin : pad_items) - first;
    void* dev = nullptr;
    rc = ring_alloc(part.size() * sizeof(PadJob), &dev);
    if (rc != KFAC_OK) return rc;
    KFAC_CUDA(cudaMemcpyAsync(dev, part.data(), part.size() * sizeof(PadJob),
                              cudaMemcpyHostToDevice, stream));
    const int grid = std::min(items, sm_count() * 8);
    pad_copy_group_kernel<<<grid, 256, 0, stream>>>(
        static_cast<const PadJob*>(dev), nj, items);
    KFAC_LAUNCH_CHECK("pad_copy_group_kernel");
  }
  SideStream* side = nullptr;
  if (!descs[0].empty() && !descs[1].empty()) {
    rc = tc_side_stream(&side);
    if (rc != KFAC_OK) return rc;
    KFAC_CUDA(cudaEventRecord(side->fork, main_stream));
    KFAC_CUDA(cudaStreamWaitEvent(side->stream, side->fork, 0));
  }
  for (int m = 0; m < 2; ++m) {
    std::vector<GemmDesc>& v = descs[m];
    if (v.empty()) continue;
    // strided problems on the helper stream when there are both kinds
    stream = (m == 0 && side != nullptr) ? side->stream : main_stream;
    // long-running CTAs first
    // (duration of a CTA ~ its k-blocks times the operand rows it stages)
    std::stable_sort(v.begin(), v.end(), [](const GemmDesc& a, const GemmDesc& b) {
      long long ka = (a.splits > 1 ? a.k_per_split : a.K) * tc_block_cost(a.M);
      long long kb = (b.splits > 1 ? b.k_per_split : b.K) * tc_block_cost(b.M);
      return ka > kb;
    });
    int total = 0;
    for (GemmDesc& g : v) {
      g.tile_begin = total;
      total += tc_factor_ctas(g.M) * (g.splits > 1 ? g.splits : 1);
    }
    bool tails = false;
    for (const GemmDesc& g : v) tails = tails || tc_desc_has_tails(g);
    const GemmDesc* dev_descs = nullptr;
    GemmDesc inl = {};
    if (v.size() == 1) {
      inl = v[0];
    } else {
      void* dev = nullptr;
      rc = ring_alloc(v.size() * sizeof(GemmDesc), &dev);
      if (rc != KFAC_OK) return rc;
      KFAC_CUDA(cudaMemcpyAsync(dev, v.data(), v.size() * sizeof(GemmDesc),
                                cudaMemcpyHostToDevice, stream));
      dev_descs = static_cast<const GemmDesc*>(dev);
    }
    const int nd = (int)v.size();
    if (staged)
      tc_pair_kernel<false, false, true>
          <<<total, PK_THREADS, PK_SMEM_BYTES, stream>>>(dev_descs, nd, inl);
    else if (m == 1 && tails)
      tc_pair_kernel<true, true><<<total, PK_THREADS, PK_SMEM_BYTES, stream>>>(
          dev_descs, nd, inl);
    else if (m == 1)
      tc_pair_kernel<true, false><<<total, PK_THREADS, PK_SMEM_BYTES, stream>>>(
          dev_descs, nd, inl);
    else if (tails)
      tc_pair_kernel<false, true><<<total, PK_THREADS, PK_SMEM_BYTES, stream>>>(
          dev_descs, nd, inl);
    else
      tc_pair_kernel<false, false><<<total, PK_THREADS, PK_SMEM_BYTES, stream>>>(
          dev_descs, nd, inl);
    KFAC_LAUNCH_CHECK("tc_pair_kernel");
  }
  stream = main_stream;
  if (side != nullptr) {
    KFAC_CUDA(cudaEventRecord(side->join, side->stream));
    KFAC_CUDA(cudaStreamWaitEvent(main_stream, side->join, 0));
  }
  if (!reduces.empty()) {
    void* dev = nullptr;
    if (count > 1) {
      rc = ring_alloc(reduces.size() * sizeof(ReduceItem), &dev);
      if (rc != KFAC_OK) return rc;
      KFAC_CUDA(cudaMemcpyAsync(dev, reduces.data(),
                                reduces.size() * sizeof(ReduceItem),
                                cudaMemcpyHostToDevice, stream));
    }
    int dmax = 0;
    long long elems = 0;
    for (const ReduceItem& it : reduces) {
      dmax = it.d > dmax ? it.d : dmax;
      elems += (long long)std::min(it.d, TC_BM) * std::min(it.d, TC_BN);
    }
    // eight blocks of 256 threads on every SM, in multiples of 64 elements
    const long long per = elems / (8ll * sm_count());
    const int chunk =
        (int)std::min(1024ll, std::max(64ll, (per + 63) / 64 * 64));
    const int rmax = dmax < TC_BM ? dmax : TC_BM;
    const int cmax = dmax < TC_BN ? dmax : TC_BN;
    dim3 rgrid((unsigned)reduces.size(), (rmax * cmax + chunk - 1) / chunk);
    // a lone factor: its items are consecutive tiles of one output, passed
    // by value (reduces[0] is tile 0)
    tc_reduce_kernel<<<rgrid, 256, 0, stream>>>(
        static_cast<const ReduceItem*>(dev), reduces[0], chunk);
    KFAC_LAUNCH_CHECK("tc_reduce_kernel");
  }
  return KFAC_OK;
}

int run_factor_group_tc(int count, const FactorJob* jobs, void* workspace,
                        size_t workspace_bytes, cudaStream_t stream,
                        bool staged) {
  for (int i = 0; i < count; ++i) {
    KFAC_REQUIRE(jobs[i].out != nullptr && jobs[i].X.base != nullptr,
                 "factor: null pointer");
    KFAC_REQUIRE(jobs[i].rows > 0 && jobs[i].d > 0 &&
                     jobs[i].rows < (1LL << 31),
                 "factor: rows=%lld d=%d out of range", jobs[i].rows,
                 jobs[i].d);
  }
  std::vector<FactorJob> gram, pair;
  // The feeds of gram.cu copy tables from this call's host memory, which a graph
  // would read again when it is replayed; the gather kernel takes a lone factor's
  // descriptors as arguments.
  if (count == 1 && stream_captures(stream))
    pair.assign(jobs, jobs + 1);
  else
    tc_by_feed(count, jobs, staged, gram, pair);
  // (nothing is queued by a call that fails for want of workspace)
  const size_t need =
      tc_pair_workspace_bytes((int)pair.size(), pair.data(), staged);
  if (need > 0 && (workspace == nullptr || workspace_bytes < need))
    return fail(KFAC_ERR_WORKSPACE,
                "factor: workspace of %zu bytes needed, %zu given", need,
                workspace_bytes);
  if (!gram.empty()) {
    const int rc = run_factor_group_gram((int)gram.size(), gram.data(),
                                         workspace, workspace_bytes, stream);
    if (rc != KFAC_OK) return rc;
  }
  if (pair.empty()) return KFAC_OK;
  const int rc = run_factor_group_pair((int)pair.size(), pair.data(), workspace,
                                       workspace_bytes, stream, staged);
  if (rc != KFAC_OK) return rc;
  return run_second_outputs((int)pair.size(), pair.data(), stream);
}

// Second outputs of factors whose kernels do not write them.
int run_second_outputs(int count, const FactorJob* jobs, cudaStream_t stream) {
  std::vector<const float*> x;
  std::vector<float*> out;
  std::vector<int64_t> n;
  float a2 = 0.f, b2 = 0.f;
  for (int i = 0; i < count; ++i) {
    if (jobs[i].out2 == nullptr) continue;
    x.push_back(jobs[i].out);
    out.push_back(jobs[i].out2);
    n.push_back((int64_t)jobs[i].d * jobs[i].d);
    a2 = jobs[i].a2;
    b2 = jobs[i].b2;
  }
  for (size_t k = 0; k < x.size(); k += 1024) {
    const int part = (int)std::min<size_t>(1024, x.size() - k);
    const int rc = kfac_axpby_group(part, &n[k], a2, &x[k], b2, &out[k],
                                    &out[k], (void*)stream);
    if (rc != KFAC_OK) return rc;
  }
  return KFAC_OK;
}

static FactorJob lone_job(const Operand& X, long long rows, int d, float alpha,
                          float beta, float* out) {
  FactorJob job;
  job.X = X;
  job.rows = rows;
  job.d = d;
  job.n = X.mode == 1 ? (int)(rows / ((long long)X.Ho * X.Wo)) : 0;
  job.nhwc = 0;
  job.grouped = 0;
  job.out2 = nullptr;
  job.a2 = job.b2 = 0.f;
  job.alpha = alpha;
  job.beta = beta;
  job.out = out;
  return job;
}

// Workspace of a factor built on its own from any operand of this geometry.
size_t tc_lone_workspace_bytes(const Operand& X, long long rows, int d) {
  FactorJob job = lone_job(X, rows, d, 1.f, 0.f, nullptr);
  const size_t gather =
      tc_factor_workspace_bytes(rows, d) + tc_pad_bytes(X, job.n);
  // the address and the pitch decide between the feeds: the larger of both
  job.X.s_outer = (X.s_outer + 3) & ~3LL;
  const size_t aligned = tc_factor_group_workspace_bytes(1, &job, true);
  job.X.base = reinterpret_cast<const float*>(sizeof(float));
  return std::max(gather,
                  std::max(aligned,
                           tc_factor_group_workspace_bytes(1, &job, true)));
}

int run_factor_tc(const Operand& X, long long rows, int d, float alpha,
                  float beta, float* out, void* workspace,
                  size_t workspace_bytes, cudaStream_t stream, bool staged) {
  const FactorJob job = lone_job(X, rows, d, alpha, beta, out);
  return run_factor_group_tc(1, &job, workspace, workspace_bytes, stream,
                             staged);
}

int engine() { return g_engine; }

}  // namespace kfac

extern "C" int kfac_set_engine(int engine) {
  if (engine != 0 && engine != 1)
    return kfac::fail(KFAC_ERR_INVALID, "set_engine: engine must be 0 or 1");
  kfac::g_engine = engine;
  return KFAC_OK;
}

extern "C" int kfac_get_engine(void) { return kfac::g_engine; }

extern "C" int kfac_set_factor_staging(int on) {
  kfac::g_staged = on ? 1 : 0;
  return KFAC_OK;
}

extern "C" int kfac_get_factor_staging(void) {
  return kfac::tc_staged() ? 1 : 0;
}

namespace kfac {
// Self-test of the bounded barrier wait every tile kernel relies on: one warp
// waits on a barrier that nothing will ever arrive at, with a short limit.
// The wait must give up, raise the status word it was given and let the
// kernel return.
__global__ void wait_expiry_selftest_kernel(int* status, int* returned) {
  __shared__ unsigned long long bar;
  __shared__ volatile int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  const bool ok = mbar_wait_status(&bar, 0, &abort_flag, status, 1u << 10);
  if (threadIdx.x == 0) *returned = ok ? 1 : 2;
}
}  // namespace kfac

extern "C" int kfac_selftest_wait_expiry(int* status_out, int* returned_out) {
  KFAC_REQUIRE(status_out != nullptr && returned_out != nullptr,
               "selftest_wait_expiry: null pointer");
  int* dev = nullptr;
  KFAC_CUDA(cudaMalloc(&dev, 2 * sizeof(int)));
  cudaError_t e = cudaMemset(dev, 0, 2 * sizeof(int));
  if (e == cudaSuccess) {
    kfac::wait_expiry_selftest_kernel<<<1, 32>>>(dev, dev + 1);
    kfac::count_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  int host[2] = {-1, -1};
  if (e == cudaSuccess)
    e = cudaMemcpy(host, dev, sizeof(host), cudaMemcpyDeviceToHost);
  cudaFree(dev);
  if (e != cudaSuccess)
    return kfac::fail(KFAC_ERR_CUDA, "selftest_wait_expiry: %s",
                      cudaGetErrorString(e));
  *status_out = host[0];
  *returned_out = host[1];
  return KFAC_OK;
}

extern "C" int kfac_tc_status(int* status_out) {
  KFAC_REQUIRE(status_out != nullptr, "tc_status: null pointer");
  KFAC_CUDA(cudaDeviceSynchronize());
  int v = 0;
  KFAC_CUDA(cudaMemcpyFromSymbol(&v, kfac::g_tc_status, sizeof(int)));
  int w = 0, t = 0, u = 0, p = 0;
  int rc = kfac::diag_status_read(&w);
  if (rc == KFAC_OK) rc = kfac::tile_status_read(&t);
  if (rc == KFAC_OK) rc = kfac::gram_status_read(&u);
  if (rc == KFAC_OK) rc = kfac::packed_status_read(&p);
  if (rc != KFAC_OK) return rc;
  *status_out = v | w | t | u | p;
  return KFAC_OK;
}
