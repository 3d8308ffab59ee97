// Tensor-core tile engine for sm_100a: C = alpha A B + beta C over many problems
// in one launch (GemmDesc), operands fp32 in memory, split by every tile into two
// terms, x = hi + lo, C += hi*hi + hi*lo + lo*hi in fp32 accumulators in tensor
// memory (a single TF32 pass misses the 1e-4 bound on large factors).
//
// Two kinds of terms: fp16 (tcgen05.mma kind::f16), where the values' range is
// known - the short products of the inverse that make L and X, see inverse.cu -
// and TF32 (kind::tf32) for the preconditioning of short layers and for the
// refinement.  The long products read operands that were split once
// (tc_packed.cu).
//
// One CTA owns a 128 x TN tile.  Producer warps load the operands from global
// memory with 16-byte loads, one to three 32-k blocks ahead in registers, split them
// and write the 128-byte-swizzled shared-memory layout that the MMA descriptors
// expect (K-major; fp16 terms also MN-major, as they lie in memory); one more warp
// issues the MMAs.  The epilogue (tc_epilogue.cuh) moves 32 x 32 pieces of the
// accumulator TMEM -> registers -> shared memory -> global rows, mirrored rows or
// fp16 chunks.
//
// Bound: the short products of the inverse (K <= 512) by latency: descriptor fetch,
// one trip to L2 per register block, the epilogue; the preconditioning by the
// loads and stores of its operands (a 128 x 256 x 32 block takes 1600 ns with TF32
// terms, its MMAs 810), which is why longer layers go through chunks.  Hence the
// descriptors of small launches travel as kernel arguments, and TN = 128 (half
// the work per CTA, twice the CTAs) is used while 128 x 256 tiles would leave
// SMs idle.  The 128-wide tile has 16 producer warps of one unit and three blocks
// in flight: with eight warps of two units and two blocks a k-block took the
// 1.3 us of a 256-wide one, 0.75 now.
//
// Every barrier wait is bounded; a wait that runs out raises a status word
// instead of hanging.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gemm_simt.cuh"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

namespace kfac {

constexpr int TT_BK = 32;
static __device__ int g_tile_status = 0;

template <int TN, bool HALF>
struct TileMap {
  static constexpr int kProducers = TN == 256 ? 384 : 512;
  static constexpr bool kTwo = TN == 256;         // units per producer thread
  static constexpr int kWarps = kProducers / 32;
  static constexpr int kThreads = kProducers + 32;
  static constexpr int kStages = (TN == 256 ? 2 : 3) * (HALF ? 2 : 1);
  // operand rows of 128 bytes: 32 TF32 values, or both fp16 terms of 32
  static constexpr int kABytes = TC_BM * 128;             // 16 KB
  static constexpr int kBBytes = TN * 128;
  static constexpr int kLo = kABytes + kBBytes;   // TF32: lo tiles, hi before
  static constexpr int kStage = HALF ? kLo : 2 * kLo;
  static constexpr int kTmem = 2 * TN;            // hi*hi, then cross terms
  static constexpr int kSmem = kStages * kStage + 1024 + 1024;
};
constexpr int TT_MAX_STAGES = 6;

struct TileControl {
  unsigned long long full[TT_MAX_STAGES];
  unsigned long long empty[TT_MAX_STAGES];
  unsigned long long accum;
  unsigned tmem_base;
  volatile int abort_flag;
  GemmDesc desc;
};
static_assert(sizeof(TileControl) <= 1024, "tile control block");

// One producer unit: four 16-byte chunks (4 consecutive k of one tile row) per
// 32-k block.  Operands contiguous along k: a warp covers 16 rows, one load
// instruction 4 rows x 128 bytes.  Operands contiguous along the tile rows: a
// warp covers 16 k x 32 rows, a thread a 4 x 4 block that it transposes by
// naming its registers; lanes are laid out so that loads cover 128-byte pieces
// of four k and the stores of a quarter warp fall into different banks.
// Operands whose rows are not 16-byte aligned (the caller's matrices of odd
// sides) are read a float per lane along the contiguous index instead: a load
// instruction still covers one 128-byte piece, of one row (k along the lanes,
// 16 rows of a thread's k) or of one k (rows along the lanes, 16 k of a
// thread's row).
//
// Rows past the operand's last one repeat it: their accumulator rows (columns)
// are never stored.  Only the appended column of a gradient and the end of the
// contraction need values of their own.
struct TileUnit {
  const float* p;        // first element of the unit in the current block
  int o[3];              // 16-byte words: offsets of chunks 1 .. 3
  int step;              // else: elements from one row (kfast) or k to the next
  int adv;               // elements from one block to the next
  int k;                 // first k of the unit in the current block
  int row;               // first row (not kfast: of four consecutive ones)
  int last;              // kfast: rows from there to the operand's last one
  unsigned soff;         // store offset of chunk 0 inside a stage
  int flags;
};
enum { U_KFAST = 1, U_LIVE = 2, U_EXTRA = 4 };

// Rows of an operand can be read as 16-byte words.
__host__ __device__ __forceinline__ bool tile_operand_vec(const Operand& op) {
  const long long ld = op.kfast ? op.s_col : op.s_outer;
  return (reinterpret_cast<uintptr_t>(op.base) & 15) == 0 && (ld & 3) == 0;
}

// `wu`: index of the 32-thread unit among those of its side; `rows`: valid rows
// of the side (units past them stay idle: their rows are never stored).
template <bool VEC>
__device__ __forceinline__ void tile_unit_setup(const Operand& op, int r0,
                                                int wu, int lane,
                                                int rows, unsigned side_off,
                                                TileUnit& u) {
  const bool kf = op.kfast != 0;
  const int ld = kf ? (int)op.s_col : (int)op.s_outer;
  u.flags = kf ? U_KFAST : 0;
  // the unit holds the appended column
  const int first = kf ? 16 * wu : 32 * (wu >> 1), span = kf ? 16 : 32;
  if (first < rows) u.flags |= U_LIVE;
  if (op.extra_idx >= r0 + first && op.extra_idx < r0 + first + span)
    u.flags |= U_EXTRA;
  if (!VEC) {
    const int row = kf ? first : first + lane;
    u.k = kf ? lane : 16 * (wu & 1);
    u.row = r0 + row;
    const int r = min(u.row, op.ncols - 1);
    u.last = op.ncols - 1 - r;
    u.p = op.base + (kf ? (long long)r * ld + u.k : (long long)u.k * ld + r);
    u.step = ld;
    u.adv = kf ? TT_BK : TT_BK * ld;
    u.soff = side_off + (kf ? (unsigned)(row * 128 + 4 * (lane & 3))
                            : (unsigned)(row * 128));
    return;
  }
  if (kf) {
    const int chunk = lane & 7, row = first + (lane >> 3);
    u.k = 4 * chunk;
    u.row = r0 + row;
    const int r = min(u.row, op.ncols - 1);
    u.last = op.ncols - 1 - r;
    u.p = op.base + (long long)r * ld + u.k;
#pragma unroll
    for (int i = 1; i < 4; ++i) u.o[i - 1] = min(4 * i, u.last) * ld;
    u.adv = TT_BK;
    u.soff = side_off + sw128_chunk_off(row, chunk);
  } else {
    const int kq = 4 * (wu & 1) + (lane & 3);
    const int row = first + 4 * (lane >> 2);
    u.k = 4 * kq;
    u.row = r0 + row;
    u.last = 0;
    // (whole words: the pitch covers the last one)
    u.p = op.base + (long long)u.k * ld + min(u.row, (op.ncols - 1) & ~3);
#pragma unroll
    for (int i = 1; i < 4; ++i) u.o[i - 1] = i * ld;
    u.adv = TT_BK * ld;
    u.soff = side_off + sw128_chunk_off(row, kq);
  }
}

template <bool VEC>
__device__ __forceinline__ void tile_unit_load(const Operand& op, TileUnit& u,
                                               int kend, float4 v[4]) {
  if (!(u.flags & U_LIVE)) return;
  const bool kf = (u.flags & U_KFAST) != 0;
  const float* p = u.p;
  if (!VEC) {
    float x[16];
    if (kf) {
      const bool in = u.k < kend;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        x[i] = in ? p[(long long)min(i, u.last) * u.step] : 0.f;
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i, p += u.step)
        x[i] = u.k + i < kend ? *p : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
  } else if (u.k + 3 < kend) {
    v[0] = *reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 1; i < 4; ++i)
      v[i] = *reinterpret_cast<const float4*>(p + u.o[i - 1]);
  } else {
    // the end of the contraction: of every row, or whole k
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* q = i == 0 ? p : p + u.o[i - 1];
      const int left = kf ? kend - u.k : (u.k + i < kend ? 4 : 0);
      v[i].x = left > 0 ? q[0] : 0.f;
      v[i].y = left > 1 ? q[1] : 0.f;
      v[i].z = left > 2 ? q[2] : 0.f;
      v[i].w = left > 3 ? q[3] : 0.f;
    }
  }
  if (u.flags & U_EXTRA) {
    // the appended column (row extra_idx of the tile) of a gradient
    float* x = reinterpret_cast<float*>(v);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int a = i >> 2, b = i & 3;
      const int k = VEC ? (kf ? u.k + b : u.k + a) : (kf ? u.k : u.k + i);
      const int c = VEC ? (kf ? u.row + 4 * a : u.row + b)
                        : (kf ? u.row + i : u.row);
      if (c == op.extra_idx)
        x[i] = k >= kend ? 0.f : (op.extra != nullptr ? op.extra[k] : 1.f);
    }
  }
  u.k += TT_BK;
  u.p += u.adv;
}

template <bool VEC>
__device__ __forceinline__ void tile_unit_store(const TileUnit& u, unsigned st,
                                                unsigned lo, const float4 v[4]) {
  if (!(u.flags & U_LIVE)) return;
  const unsigned at = st + u.soff;
  const int lane = threadIdx.x & 31;
  if (!VEC) {
    if (u.flags & U_KFAST) {
      // k = lane of rows 0 .. 15 (a multiple of 16 rows from the tile's start)
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float4 q = v[i >> 2];
        const float x = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y
                        : (i & 3) == 2 ? q.z : q.w;
        const float h = tf32_round(x);
        const unsigned d = at + 128 * i + (((lane >> 2) ^ (i & 7)) << 4);
        sts32(d, h);
        sts32(d + lo, x - h);
      }
    } else {
      // chunks of row `lane`, from the 16 k of this unit on
      const int half = ((threadIdx.x >> 5) & 1) * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned d = at + (((half + i) ^ (lane & 7)) << 4);
        store_split(d, d + lo, v[i]);
      }
    }
  } else if (u.flags & U_KFAST) {
    // chunk i is 4 i rows down: the swizzle flips with every second step
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned d = (at ^ ((i & 1) ? 0x40u : 0u)) + 512 * i;
      store_split(d, d + lo, v[i]);
    }
  } else {
    store_split(at, at + lo, make_float4(v[0].x, v[1].x, v[2].x, v[3].x));
    const unsigned d1 = (at ^ 0x10u) + 128;
    store_split(d1, d1 + lo, make_float4(v[0].y, v[1].y, v[2].y, v[3].y));
    const unsigned d2 = (at ^ 0x20u) + 256;
    store_split(d2, d2 + lo, make_float4(v[0].z, v[1].z, v[2].z, v[3].z));
    const unsigned d3 = (at ^ 0x30u) + 384;
    store_split(d3, d3 + lo, make_float4(v[0].w, v[1].w, v[2].w, v[3].w));
  }
}

// One producer unit of a product in fp16 terms (all operands have rows of
// 16-byte words).  Operands contiguous along k are stored K-major, 16 rows a
// unit: a 128-byte row holds the hi terms of 32 k, then the lo terms.  A thread
// takes four k of rows 4 (lane / 8) .. + 3, so that the two rows of a half warp's
// 8-byte stores differ in the bit that moves the swizzle across the halves of
// a row.  Operands contiguous along the tile rows are stored MN-major, as they
// are: a unit is 64 rows x 8 k, one swizzle atom (1 KB) per term; 64 rows take
// four atoms of hi and four of lo terms.
struct HalfUnit {
  const float* p;
  int o[3];              // offsets of words 1 .. 3
  int adv;
  int k;
  unsigned soff;
  bool kf, live;
};

// (a unit past the operand's last row reads that one again)
__device__ __forceinline__ void half_unit_setup(const Operand& op, int r0,
                                                int wu, int lane,
                                                int rows, unsigned side_off,
                                                HalfUnit& u) {
  u.kf = op.kfast != 0;
  const int ld = u.kf ? (int)op.s_col : (int)op.s_outer;
  if (u.kf) {
    const int row = 16 * wu + 4 * (lane >> 3), chunk = lane & 7;
    u.live = 16 * wu < rows;
    u.k = 4 * chunk;
    const int r = min(r0 + row, op.ncols - 1);
    u.p = op.base + (long long)r * ld + u.k;
#pragma unroll
    for (int i = 1; i < 4; ++i) u.o[i - 1] = min(i, op.ncols - 1 - r) * ld;
    u.adv = TT_BK;
    u.soff = side_off + sw128_chunk_off(row, chunk >> 1) + 8 * (chunk & 1);
  } else {
    const int group = wu >> 2, octet = wu & 3, kk = lane >> 4;
    const int row = 64 * group + 4 * (lane & 15);
    u.live = 64 * group < rows;
    u.k = 8 * octet + kk;
    // (whole words: the pitch covers the last one)
    u.p = op.base + (long long)u.k * ld + min(r0 + row, (op.ncols - 1) & ~3);
#pragma unroll
    for (int i = 1; i < 4; ++i) u.o[i - 1] = 2 * i * ld;
    u.adv = TT_BK * ld;
    u.soff = side_off + 8192 * group + 1024 * octet +
             sw128_chunk_off(kk, (lane & 15) >> 1) + 8 * (lane & 1);
  }
}

// FULL: the block ends before kend.  No branch around a thread's loads then, so
// that those of several blocks stay in flight across the stores of one (a
// 256-wide k-block took 1600 ns with such a branch, 1150 without).
template <bool FULL>
__device__ __forceinline__ void half_unit_load(HalfUnit& u, int kend,
                                               float4 v[4]) {
  const float* p = u.p;
  if (FULL) {
    v[0] = *reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 1; i < 4; ++i)
      v[i] = *reinterpret_cast<const float4*>(p + u.o[i - 1]);
  } else {
    // the end of the contraction: of every row, or whole k
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* q = i == 0 ? p : p + u.o[i - 1];
      const int left = u.kf ? kend - u.k : (u.k + 2 * i < kend ? 4 : 0);
      v[i].x = left > 0 ? q[0] : 0.f;
      v[i].y = left > 1 ? q[1] : 0.f;
      v[i].z = left > 2 ? q[2] : 0.f;
      v[i].w = left > 3 ? q[3] : 0.f;
    }
  }
  u.k += TT_BK;
  u.p += u.adv;
}

__device__ __forceinline__ void half_unit_store(const HalfUnit& u, unsigned st,
                                                const float4 v[4],
                                                float scale) {
  const unsigned at = st + u.soff;
  // a step of one row (two k) down also flips the swizzle by 16 (32) bytes
  const unsigned flip = u.kf ? 0x10u : 0x20u, step = u.kf ? 128u : 256u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned d = (at ^ (flip * i)) + step * i;
    unsigned h0, h1, l0, l1;
    split_half2(scale * v[i].x, scale * v[i].y, h0, l0);
    split_half2(scale * v[i].z, scale * v[i].w, h1, l1);
    sts64(d, h0, h1);
    sts64(u.kf ? d ^ 0x40u : d + 4096, l0, l1);
  }
}

// PRE: the preconditioning epilogue (every problem of the launch has it).  VEC:
// all operands of the launch have rows of 16-byte words (one kernel with both
// ways of loading spills).  HALF: operands in two fp16 terms (VEC only).
template <int TN, bool PRE, bool VEC, bool HALF>
__global__ void __launch_bounds__(TileMap<TN, HALF>::kThreads, 1)
tc_tile_kernel(const GemmDesc* __restrict__ descs, int ndesc, int tile0,
               const __grid_constant__ TileInline inl, float lr,
               float momentum) {
  static_assert(!HALF || VEC, "fp16 terms need rows of 16-byte words");
  using Map = TileMap<TN, HALF>;
  extern __shared__ unsigned char tt_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tt_smem_raw) + 1023) & ~(uintptr_t)1023);
  TileControl* ctl =
      reinterpret_cast<TileControl*>(smem + Map::kStages * Map::kStage);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = tile0 + blockIdx.x;

  if (warp == Map::kWarps) {
    if (lane == 0) {
#pragma unroll
      for (int s = 0; s < Map::kStages; ++s) {
        mbar_init(&ctl->full[s], Map::kWarps);
        mbar_init(&ctl->empty[s], 1);
      }
      mbar_init(&ctl->accum, 1);
      ctl->abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(Map::kTmem)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
  } else {
    // the problem this tile belongs to (tile_begin is ascending): bisection
    // by every warp, then a copy of the descriptor
    constexpr int kWords = (int)(sizeof(GemmDesc) / sizeof(int));
    int* dst = reinterpret_cast<int*>(&ctl->desc);
    if (inl.n > 0) {
      int f = 0;
#pragma unroll
      for (int i = 1; i < TT_INLINE; ++i)
        if (i < inl.n && inl.d[i].tile_begin <= tile) f = i;
      const int* src = reinterpret_cast<const int*>(&inl.d[f]);
      for (int i = tid; i < kWords; i += Map::kProducers) dst[i] = src[i];
    } else {
      // one round of parallel loads instead of a chain of dependent ones
      int f = 0;
      for (int i = lane; i < ndesc; i += 32)
        if (descs[i].tile_begin <= tile) f = i;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        f = max(f, __shfl_xor_sync(0xffffffffu, f, o));
      const int* src = reinterpret_cast<const int*>(descs + f);
      for (int i = tid; i < kWords; i += Map::kProducers) dst[i] = src[i];
    }
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
    tile_lower<TN>(lt, bi, bj);
  } else {
    bi = lt / g.tiles_n;
    bj = lt - bi * g.tiles_n;
  }
  const int m0 = bi * TC_BM, n0 = bj * TN;
  int n_valid = min(TN, g.N - n0);
  if (flags & G_LOWER) n_valid = min(n_valid, m0 + TC_BM - n0);
  const int n_inst = (n_valid + 15) & ~15;
  const int m_valid = min(TC_BM, g.M - m0);
  int kend = (int)g.K;
  if (flags & G_KEND_M0) kend = min(kend, m0 + TC_BM);
  // a gated-off problem runs no k-blocks and stores nothing
  const bool gated_off = g.gate != nullptr && *g.gate == 0;
  const int nkb =
      gated_off ? 0 : (kend + TT_BK - 1) / TT_BK;

  if (warp < Map::kWarps) {
    // ===================== producers =====================
    // units 0 .. 7 of 32 threads: A rows, then the B rows
    const bool a0 = warp < 8;
    const Operand& op0 = a0 ? g.A : g.B;
    const Operand& op1 = g.B;
    using Unit = typename std::conditional<HALF, HalfUnit, TileUnit>::type;
    Unit u0, u1;
    const float scale0 = HALF ? (a0 ? g.sa : g.sb) : 1.f;
    const float scale1 = HALF ? g.sb : 1.f;
    {
      const int r0 = a0 ? m0 : n0, wu = a0 ? warp : warp - 8;
      const int rows = a0 ? m_valid : n_valid;
      const unsigned side = a0 ? 0 : Map::kABytes;
      if constexpr (HALF) {
        half_unit_setup(op0, r0, wu, lane, rows, side, u0);
        if (Map::kTwo)
          half_unit_setup(op1, n0, warp + Map::kWarps - 8, lane, n_valid,
                          Map::kABytes, u1);
      } else {
        tile_unit_setup<VEC>(op0, r0, wu, lane, rows, side, u0);
        if (Map::kTwo)
          tile_unit_setup<VEC>(op1, n0, warp + Map::kWarps - 8, lane,
                               n_valid, Map::kABytes, u1);
      }
    }
    const unsigned base = smem_u32(smem);
    // blocks that end before kend (fp16 terms)
    const int nfull = kend / TT_BK;
    auto load = [&](int kb, float4* v) {
      if constexpr (HALF) {
        if (kb < nfull) {
          half_unit_load<true>(u0, kend, v);
          if (Map::kTwo) half_unit_load<true>(u1, kend, v + 4);
        } else {
          half_unit_load<false>(u0, kend, v);
          if (Map::kTwo) half_unit_load<false>(u1, kend, v + 4);
        }
      } else {
        tile_unit_load<VEC>(op0, u0, kend, v);
        if (Map::kTwo) tile_unit_load<VEC>(op1, u1, kend, v + 4);
      }
    };
    auto store = [&](int kb, const float4* v) {
      const int s = kb % Map::kStages;
      if (kb >= Map::kStages &&
          !mbar_wait_status(&ctl->empty[s], ((kb / Map::kStages) - 1) & 1,
                            &ctl->abort_flag, &g_tile_status))
        return false;
      const unsigned st = base + s * Map::kStage;
      if constexpr (HALF) {
        half_unit_store(u0, st, v, scale0);
        if (Map::kTwo) half_unit_store(u1, st, v + 4, scale1);
      } else {
        tile_unit_store<VEC>(u0, st, Map::kLo, v);
        if (Map::kTwo) tile_unit_store<VEC>(u1, st, Map::kLo, v + 4);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->full[s]);
      return true;
    };
    constexpr int kVals = Map::kTwo ? 8 : 4;
    float4 va[kVals];
    bool idle = false;
    if constexpr (HALF) idle = !u0.live && !(Map::kTwo && u1.live);
    if (idle) {
      // none of this warp's rows is used: it only keeps the barriers going
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % Map::kStages;
        if (kb >= Map::kStages &&
            !mbar_wait_status(&ctl->empty[s], ((kb / Map::kStages) - 1) & 1,
                              &ctl->abort_flag, &g_tile_status))
          break;
        if (lane == 0) mbar_arrive(&ctl->full[s]);
      }
    } else if (TN == 256 && !HALF) {
      // one block ahead: the MMAs of a block take longer than a trip to L2
      if (nkb > 0) load(0, va);
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb) {
        if (!store(kb, va)) break;
        if (kb + 1 < nkb) load(kb + 1, va);
      }
    } else if (!VEC || TN == 256) {
      float4 vb[kVals];
      if (nkb > 0) load(0, va);
      if (nkb > 1) load(1, vb);
#pragma unroll 1
      for (int kb = 0; kb < nkb; kb += 2) {
        if (!store(kb, va)) break;
        if (kb + 2 < nkb) load(kb + 2, va);
        if (kb + 1 < nkb) {
          if (!store(kb + 1, vb)) break;
          if (kb + 3 < nkb) load(kb + 3, vb);
        }
      }
    } else {
      float4 vb[kVals], vc[kVals];
      if (nkb > 0) load(0, va);
      if (nkb > 1) load(1, vb);
      if (nkb > 2) load(2, vc);
#pragma unroll 1
      for (int kb = 0; kb < nkb; kb += 3) {
        if (!store(kb, va)) break;
        if (kb + 3 < nkb) load(kb + 3, va);
        if (kb + 1 < nkb) {
          if (!store(kb + 1, vb)) break;
          if (kb + 4 < nkb) load(kb + 4, vb);
        }
        if (kb + 2 < nkb) {
          if (!store(kb + 2, vc)) break;
          if (kb + 5 < nkb) load(kb + 5, vc);
        }
      }
    }
  } else {
    if (HALF && elect_one()) {
      // ===================== MMA issuer, fp16 terms =====================
      const bool ka = g.A.kfast != 0, kb_ = g.B.kfast != 0;
      const unsigned idesc = tc_half_desc(n_inst, !ka, !kb_);
      // from the hi to the lo terms, and from 16 k to the next (16-byte units)
      const unsigned long long lo_a = (ka ? 64 : 4096) >> 4;
      const unsigned long long lo_b = (kb_ ? 64 : 4096) >> 4;
      const unsigned long long adv_a = (ka ? 32 : 2048) >> 4;
      const unsigned long long adv_b = (kb_ ? 32 : 2048) >> 4;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % Map::kStages;
        if (!mbar_wait_status(&ctl->full[s], (kb / Map::kStages) & 1,
                              &ctl->abort_flag, &g_tile_status))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned sa = smem_u32(smem + s * Map::kStage);
        const unsigned sb = smem_u32(smem + s * Map::kStage) + Map::kABytes;
        unsigned long long a = ka ? tc_smem_desc(sa) : tc_smem_desc_mn(sa, 8192);
        unsigned long long b = kb_ ? tc_smem_desc(sb) : tc_smem_desc_mn(sb, 8192);
#pragma unroll
        for (int kk = 0; kk < TT_BK / 16; ++kk, a += adv_a, b += adv_b) {
          tc_mma_half(tmem + TN, a + lo_a, b, idesc, (kb | kk) != 0);
          tc_mma_half(tmem + TN, a, b + lo_b, idesc, 1);
          tc_mma_half(tmem, a, b, idesc, (kb | kk) != 0);
        }
        tc_commit(&ctl->empty[s]);
      }
      tc_commit(&ctl->accum);
    }
    if (!HALF && elect_one()) {
      // ===================== MMA issuer =====================
      const unsigned idesc = tc_instr_desc(n_inst);
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % Map::kStages;
        if (!mbar_wait_status(&ctl->full[s], (kb / Map::kStages) & 1,
                              &ctl->abort_flag, &g_tile_status))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned sa = smem_u32(smem + s * Map::kStage);
        const unsigned long long a_hi = tc_smem_desc(sa);
        const unsigned long long b_hi = tc_smem_desc(sa + Map::kABytes);
        const unsigned long long a_lo = tc_smem_desc(sa + Map::kLo);
        const unsigned long long b_lo =
            tc_smem_desc(sa + Map::kLo + Map::kABytes);
#pragma unroll
        for (int kk = 0; kk < TT_BK / 8; ++kk) {
          const unsigned long long adv = (unsigned long long)(kk * 32 >> 4);
          tc_mma(tmem + TN, a_lo + adv, b_hi + adv, idesc, (kb | kk) != 0);
          tc_mma(tmem + TN, a_hi + adv, b_lo + adv, idesc, 1);
          tc_mma(tmem, a_hi + adv, b_hi + adv, idesc, (kb | kk) != 0);
        }
        tc_commit(&ctl->empty[s]);
      }
      tc_commit(&ctl->accum);
    }
    // (the block barrier and the release of the tensor memory are warp-wide)
    __syncwarp();
  }

  // ===================== epilogue =====================
  // warp w: accumulator rows of quarter q, 32-column pieces h, h + G, ...; its
  // own piece of the (drained) first stages
  if (warp < Map::kWarps && !gated_off) {
    TileOut o;
    o.m0 = m0; o.n0 = n0; o.m_valid = m_valid; o.n_valid = n_valid;
    o.lr = lr; o.momentum = momentum;
    tile_epilogue<TN, Map::kWarps / 4, PRE>(
        g, o, tmem, nkb == 0, warp & 3, warp >> 2, lane,
        reinterpret_cast<float*>(smem) + warp * 32 * TT_EP, [&] {
          return mbar_wait_status(&ctl->accum, 0, &ctl->abort_flag,
                                  &g_tile_status);
        });
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == Map::kWarps) tc_release(ctl->tmem_base, Map::kTmem, ctl->abort_flag != 0);
}

// ------------------------------------------------------------------ host side
typedef void (*TileKernel)(const GemmDesc*, int, int, const TileInline, float,
                           float);

struct TileVariant {
  TileKernel kernel;
  int threads, smem;
};

template <int TN, bool PRE, bool VEC, bool HALF = false>
static TileVariant tile_variant() {
  return {tc_tile_kernel<TN, PRE, VEC, HALF>, TileMap<TN, HALF>::kThreads,
          TileMap<TN, HALF>::kSmem};
}

// [128 columns][precondition][16-byte rows]
static const TileVariant kTileVariants[2][2][2] = {
    {{tile_variant<256, false, false>(), tile_variant<256, false, true>()},
     {tile_variant<256, true, false>(), tile_variant<256, true, true>()}},
    {{tile_variant<128, false, false>(), tile_variant<128, false, true>()},
     {tile_variant<128, true, false>(), tile_variant<128, true, true>()}}};
// [128 columns]: fp16 terms
static const TileVariant kHalfVariants[2] = {
    tile_variant<256, false, true, true>(),
    tile_variant<128, false, true, true>()};

int tc_prepare_tiles() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  KFAC_CUDA(cudaGetDevice(&dev));
  KFAC_REQUIRE(dev >= 0 && dev < 64, "device index %d unsupported", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    for (int k = 0; k < 10; ++k) {
      const TileVariant& v = k < 8
                                 ? kTileVariants[k >> 2][(k >> 1) & 1][k & 1]
                                 : kHalfVariants[k - 8];
      KFAC_CUDA(cudaFuncSetAttribute(
          v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
    }
    done[dev] = true;
  }
  return KFAC_OK;
}

static int tile_count(const GemmDesc& g, int tn) {
  const int tm = (g.M + TC_BM - 1) / TC_BM, nn = (g.N + tn - 1) / tn;
  if (!(g.flags & G_LOWER)) return tm * nn;
  if (tn == TC_BM) return tm * (tm + 1) / 2;
  const int a = tm / 2;
  return (tm & 1) ? (a + 1) * (a + 1) : a * (a + 1);
}

static bool tile_desc_vec(const GemmDesc& g) {
  return tile_operand_vec(g.A) && tile_operand_vec(g.B);
}

int tc_number_tiles(GemmDesc* descs, int n, int narrow_max, int* tile_cols) {
  std::stable_partition(descs, descs + n, tile_desc_vec);
  // Narrow tiles (half the work per CTA, but the A rows are loaded, split and
  // read by the MMAs twice as often) up to `narrow_max` of them: as many as
  // there are SMs for a launch that runs alone, three quarters where launches of
  // other streams run beside it.  us with the line at 0, 20, 74, 111, 148 and 222
  // tiles on 148 SMs: inverses of 4608 beside 512 rows 1455, 1439, 1429, 1448,
  // 1438, 1439; 2304 beside 256 699, 684, 669, 669, 668, 667; two of 1024 347, 338,
  // 329, 330, 330, 331; 20 of 600 304, 304, 301, 290, 291, 290; 28 of odd sides 315,
  // 312, 303, 303, 304, 304; 108 factors of ResNet-50 3381, 3386, 3370, 3377, 3383,
  // 3366.  Preconditioning of short layers, wide and narrow: 54 narrow tiles 49 36,
  // 72 49 36.5, 128 57 41, 176 109 109.
  long long narrow = 0;
  for (int i = 0; i < n; ++i) narrow += tile_count(descs[i], 128);
  const int tn = narrow <= narrow_max ? 128 : 256;
  int total = 0;
  for (int i = 0; i < n; ++i) {
    descs[i].tile_begin = total;
    descs[i].tiles_m = (descs[i].M + TC_BM - 1) / TC_BM;
    descs[i].tiles_n = (descs[i].N + tn - 1) / tn;
    total += tile_count(descs[i], tn);
  }
  *tile_cols = tn;
  return total;
}

int launch_tc_grouped(const GemmDesc* descs_dev, const GemmDesc* descs_host,
                      int ndesc, int total_tiles, int tile_cols, bool precond,
                      float lr, float momentum, cudaStream_t stream) {
  if (ndesc <= 0 || total_tiles <= 0) return KFAC_OK;
  const int rc = tc_prepare_tiles();
  if (rc != KFAC_OK) return rc;
  // the problems with 16-byte rows come first (tc_number_tiles); where all
  // tiles fit the chip at once, one launch of the general kernel (1.3 us per
  // k-block of a 128-wide tile) may end sooner than two in a row (0.75 us, and
  // 10 us more).  Both products of 256 x 1024 beside 10 x 301: 92 us in two
  // launches each, 83 us in one; 128 x 2048 beside 127 x 1023: 153 and 120.
  int n_vec = 0;
  while (n_vec < ndesc && tile_desc_vec(descs_host[n_vec])) ++n_vec;
  if (n_vec < ndesc && total_tiles <= sm_count()) {
    long long k[2] = {0, 0};
    for (int i = 0; i < ndesc; ++i)
      k[i >= n_vec] = std::max(k[i >= n_vec], descs_host[i].K / TT_BK);
    if (26 * std::max(k[0], k[1]) <= 15 * k[0] + 26 * k[1] + 200) n_vec = 0;
  }
  for (int k = 0; k < 2; ++k) {
    const int first = k == 0 ? 0 : n_vec, n = k == 0 ? n_vec : ndesc - n_vec;
    if (n == 0) continue;
    const int tile0 = descs_host[first].tile_begin;
    const int end =
        first + n < ndesc ? descs_host[first + n].tile_begin : total_tiles;
    TileInline inl;
    inl.n = 0;
    if (n <= TT_INLINE) {
      inl.n = n;
      std::copy(descs_host + first, descs_host + first + n, inl.d);
    }
    bool half = k == 0 && !precond;
    for (int i = 0; half && i < n; ++i)
      half = (descs_host[first + i].flags & G_HALF) != 0;
    const TileVariant& v =
        half ? kHalfVariants[tile_cols == 128]
             : kTileVariants[tile_cols == 128][precond][k == 0];
    // (a preconditioning's second product begins behind its first)
    const int rc = launch_behind("tc_tile_kernel", precond, v.kernel, end - tile0,
                                 v.threads, v.smem, stream, descs_dev + first, n,
                                 tile0, inl, lr, momentum);
    if (rc != KFAC_OK) return rc;
  }
  return KFAC_OK;
}

int tile_status_read(int* out) {
  KFAC_CUDA(cudaMemcpyFromSymbol(out, g_tile_status, sizeof(int)));
  return KFAC_OK;
}

}  // namespace kfac
