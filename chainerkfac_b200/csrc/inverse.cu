// Batched damped inverse of symmetric positive definite factors.
//
//   W = S (F + add * I) S               (copy; the running average F is kept)
//   W = L L^T                           blocked right-looking Cholesky, NB = 128
//   X = L^-1                            diagonal blocks in the diagonal kernel,
//                                       then row panels as their columns finish
//   inv = S X^T X S                     a panel's contribution at a time
//
// S is diagonal, powers of two that bring the diagonal of W into [1, 4).  That is
// exact, and bounds what the products below work on, so that they can take it as
// two fp16 terms (22 significant bits) of one scale per kind:
//   |W|, |L| < 4, scaled by 2^13;
//   |X|, scaled by 2^4: a column of X has norm sqrt((W^-1)_jj), and an entry of
//   4096 means a condition number above 1.6e7, where a Cholesky factorisation
//   in fp32 has no correct digit left (such entries saturate); small entries
//   are held to 2^-29, the diagonal of X is 1/2 or more;
//   T = L X, of at most twice the norm of a column of X, scaled by 2^3.
//
// A plan precomputes, for a fixed set of matrices, the descriptor lists of
// every grouped-GEMM launch; running it replays them, each launch covering all
// matrices that are still active, with the row panels beside the chain of the
// next panel's diagonal blocks.
#include <vector>
#include <algorithm>
#include <mutex>

#include "gemm_simt.cuh"
#include "tc_common.cuh"

namespace kfac {

constexpr int DB = 128;        // diagonal block
constexpr int PW = 512;        // Cholesky panel width (outer blocking)

struct MatInfo {
  const float* F;
  float* inv;
  // working copies, rows `ld` floats apart (d rounded up to whole 128-byte
  // lines, so that every row is read and written as 16-byte words)
  float* W;       // damped factor, then L (and T^T above the diagonal)
  float* X;       // L^-1
  float* V;       // T of the doubling; X R of the refinement
  int d, ld;
  int partner;
  int role;
  float l2;
  float scale;
  float l2b;      // role 2: floor of the second half of the diagonal
  int id;         // index of the matrix in the plan
  float* diag;    // diagonal of F, `ld` floats (zeros past d)
  float* S;       // the scales, likewise
  // L and X in fp16 chunks (see GemmDesc; NULL: not used), L by 128-row tile,
  // X by 128-column tile, `tile` bytes apart
  unsigned char *PL, *PX;
  long long tile;
};
constexpr float kScaleL = 8192.f, kScaleX = 16.f, kScaleT = 8.f;


__host__ __device__ static int matrix_pitch(int d) { return (d + 31) & ~31; }

__host__ __device__ static size_t matrix_bytes(int d) {
  const size_t bytes = (size_t)d * matrix_pitch(d) * sizeof(float);
  return (bytes + 255) & ~(size_t)255;
}

// Per-run arguments, kept in device memory so that a captured CUDA graph of
// the plan's launches can be replayed with new values: a one-thread kernel
// ahead of the graph writes them.
struct RunParams {
  float damping;
  int use_pi;
  int refine_max_dim;
  float refine_threshold;
};

__global__ void set_run_params_kernel(RunParams* prm, float damping,
                                      int use_pi, int refine_max_dim,
                                      float refine_threshold) {
  prm->damping = damping;
  prm->use_pi = use_pi;
  prm->refine_max_dim = refine_max_dim;
  prm->refine_threshold = refine_threshold;
}

// Also keeps the diagonal (the scales are made of it).  Bound by the latency of
// its loads, so as many threads as a block has and four loads of each in flight
// (4608 and 512 rows: 15 us with 256 threads and a load at a time, 6 so).
constexpr int kTraceThreads = 1024;
__global__ void __launch_bounds__(kTraceThreads) trace_kernel(const MatInfo* __restrict__ mats,
                             float* __restrict__ trace, int* __restrict__ info) {
  let_next_launch_begin();
  const MatInfo mi = mats[blockIdx.x];
  float s = 0.f;
  for (int i0 = threadIdx.x; i0 < mi.d; i0 += 4 * kTraceThreads) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k * kTraceThreads;
      v[k] = i < mi.d ? mi.F[(long long)i * (mi.d + 1)] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k * kTraceThreads;
      if (i < mi.d) mi.diag[i] = v[k];
      s += v[k];
    }
  }
  __shared__ float sh[32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.f;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
      trace[blockIdx.x] = s;
      info[blockIdx.x] = 0;
    }
  }
}

// What is added to the diagonal of matrix i (role 2: to its first and second
// half, scale and shift parameters with floors of their own).
__device__ __forceinline__ float2 damping_of(const MatInfo* mats, int i,
                                             const MatInfo& mi,
                                             const float* trace,
                                             const RunParams* prm) {
  const float damping = prm->damping;
  const float g = fmaxf(mi.l2, damping);
  if (mi.role == 2)
    return make_float2(g * mi.scale, fmaxf(mi.l2b, damping) * mi.scale);
  const float r = sqrtf(g);
  float pi = 1.f;
  if (prm->use_pi && mi.partner >= 0) {
    const MatInfo& mp = mats[mi.partner];
    // pi = sqrt(tr(A) dim(G) / (tr(G) dim(A))) with A the forward factor
    float tA = mi.role == 0 ? trace[i] : trace[mi.partner];
    float tG = mi.role == 0 ? trace[mi.partner] : trace[i];
    float dA = (float)(mi.role == 0 ? mi.d : mp.d);
    float dG = (float)(mi.role == 0 ? mp.d : mi.d);
    pi = sqrtf((tA * dG) / (tG * dA));
  }
  const float v = mi.role == 0 ? pi * r : (1.f / pi) * r;
  return make_float2(v, v);
}

// Power of two s with s^2 x in [1, 4).  An x that is no positive normal number
// fails as a pivot and stays as it is.
__device__ __forceinline__ float equil_scale(float x) {
  if (!(x >= 1.17549435e-38f)) return 1.f;
  const int e = (int)(__float_as_uint(x) >> 23) - 127;
  return __uint_as_float((unsigned)(127 - (e >> 1)) << 23);
}

// W = S (F + add * I) S, blockIdx.y = matrix, blockIdx.x strides over groups of four
// rows, which share the columns' scales and are in flight together.  Only the lower
// triangle and the rest of each diagonal 128-block (which the trailing updates
// read-modify-write) is ever used, so only that is copied.  `equil` off: S = I.
// (Row by row: 28 matrices of up to 856 rows 13.7 us, 4608 and 512 rows 23.5; a warp
// a row 16.6 and 28.9; so 11.9 and 17.3.)
constexpr int kDampRows = 4;
__global__ void __launch_bounds__(256, 4)
damp_copy_kernel(const MatInfo* __restrict__ mats,
                 const float* trace, const RunParams* __restrict__ prm,
                 float* add, float* add2, float* add_out, int equil) {
  let_next_launch_begin();
  const MatInfo mi = mats[blockIdx.y];
  const int d = mi.d;
  if (kDampRows * (int)blockIdx.x >= d) return;
  wait_for_launch_before();
  const float2 ad = damping_of(mats, blockIdx.y, mi, trace, prm);
  const float a_first = ad.x, a_second = ad.y;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    add[blockIdx.y] = a_first;
    add2[blockIdx.y] = a_second;
    if (add_out) add_out[blockIdx.y] = a_first;
  }
  auto damp = [&](int r) {
    return (mi.role == 2 && 2 * r >= d) ? a_second : a_first;
  };
  auto scale = [&](int r, float f) {
    return equil ? equil_scale(f + damp(r)) : 1.f;
  };
  const bool vec = (d & 3) == 0 &&
                   ((reinterpret_cast<uintptr_t>(mi.F) |
                     reinterpret_cast<uintptr_t>(mi.W)) & 15) == 0;
  for (int r0 = kDampRows * blockIdx.x; r0 < d; r0 += kDampRows * gridDim.x) {
    float sr[kDampRows], a[kDampRows];
    const float *src[kDampRows];
    float* dst[kDampRows];
#pragma unroll
    for (int i = 0; i < kDampRows; ++i) {
      const int r = min(r0 + i, d - 1);    // (past the end: the last row again)
      a[i] = damp(r);
      sr[i] = scale(r, mi.diag[r]);
      src[i] = mi.F + (long long)r * d;
      dst[i] = mi.W + (long long)r * mi.ld;
      if (threadIdx.x == 0) mi.S[r] = sr[i];
    }
    const int cend = min(d, (r0 | (DB - 1)) + 1);
    if (vec) {
      // cend is a multiple of 128 or equals d, itself a multiple of 4 here
      const float4* g4 = reinterpret_cast<const float4*>(mi.diag);
#pragma unroll 1
      for (int c4 = threadIdx.x; c4 < (cend >> 2); c4 += 256) {
        float4 v[kDampRows];
#pragma unroll
        for (int i = 0; i < kDampRows; ++i)
          v[i] = reinterpret_cast<const float4*>(src[i])[c4];
        const float4 g = g4[c4];
        const float sx = scale(4 * c4, g.x), sy = scale(4 * c4 + 1, g.y);
        const float sz = scale(4 * c4 + 2, g.z), sw = scale(4 * c4 + 3, g.w);
        if ((r0 >> 2) == c4) {             // (the rows' four diagonal entries)
          v[0].x += a[0];
          v[1].y += a[1];
          v[2].z += a[2];
          v[3].w += a[3];
        }
#pragma unroll
        for (int i = 0; i < kDampRows; ++i)
          reinterpret_cast<float4*>(dst[i])[c4] =
              make_float4(v[i].x * sr[i] * sx, v[i].y * sr[i] * sy,
                          v[i].z * sr[i] * sz, v[i].w * sr[i] * sw);
      }
    } else {
#pragma unroll 2
      for (int c = threadIdx.x; c < cend; c += 256) {
        float v[kDampRows];
#pragma unroll
        for (int i = 0; i < kDampRows; ++i) v[i] = src[i][c];
        const float sc = scale(c, mi.diag[c]);
#pragma unroll
        for (int i = 0; i < kDampRows; ++i) {
          if (min(r0 + i, d - 1) == c) v[i] += a[i];
          dst[i][c] = v[i] * sr[i] * sc;
        }
      }
    }
  }
}


// ------------------------------------------------ look-ahead of the Cholesky
constexpr int DLD = DB + 4;   // shared-memory row pitch of a 128 x 128 block
constexpr int SB = 32;        // sub-block of the diagonal kernel
constexpr int SLP = SB + 4;   // row pitch of a 32 x 32 sub-block
constexpr int DT = 512;       // threads of the diagonal kernel
constexpr int kLookTile = DB * 128;    // one fp16 term of 128 rows x 64 k
constexpr int kLookX = 3 * kLookTile;           // X_pp, see look_load_x
constexpr int kLookBytes = 4 * kLookTile + kLookX;
constexpr int kDiagCols = 2 * DB;               // tensor-memory columns

static __device__ int g_diag_status = 0;

struct DiagControl {
  // look-ahead
  unsigned long long x_here;   // X_pp has arrived
  unsigned long long done[2];  // all MMAs of the first, second product
  // elimination, one for each sub-block and step
  unsigned long long step[4][4];  // eight columns of L_pp are in Ls
  unsigned long long crit[4][4];  // eight columns of the next row-block in S
  // a phase per sub-block
  unsigned long long rows;     // all its columns are stored as operands
  unsigned long long next;     // products with the next sub-block column,
  unsigned long long beyond;   // with the columns beyond
  unsigned tmem_base;
  volatile int abort_flag;
  volatile int grace;          // abort_flag of the wait at the very end
};

// Bounded wait on a phase of a barrier of this kernel; false if the limit ran out
// here or elsewhere in the block (the status word is set at the end).  Shorter than
// mbar_wait_status: see chol_diag_kernel on the size of its code.
__device__ __forceinline__ bool diag_wait(unsigned long long* bar,
                                          unsigned parity,
                                          volatile int* abort_flag) {
  const unsigned addr = smem_u32(bar);
#pragma unroll 1
  for (unsigned i = 0; i < TC_SPIN_LIMIT; ++i) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// The same by a whole warp ahead of its use of tensor memory.
__device__ __forceinline__ bool diag_wait_tmem(unsigned long long* bar,
                                               unsigned parity,
                                               volatile int* abort_flag) {
  const bool ok = diag_wait(bar, parity, abort_flag);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return __all_sync(0xffffffffu, ok);
}

// D(128 x 128) = A B^T over 128 k, 16 at a time: operands as tiles of 64 k by term
// (hi, lo), then the next 64 k.  hi*hi goes to columns [0, 128) of the tensor
// memory, the cross terms to [128, 256).  `lower`: B is X_pp as look_load_x leaves
// it.
__device__ __forceinline__ void look_mma(unsigned tmem, unsigned a, unsigned b,
                                         bool lower) {
  constexpr unsigned long long lo = kLookTile >> 4;
  unsigned long long da = tc_smem_desc(a), db = tc_smem_desc(b), lo_b = lo;
#pragma unroll 1
  for (int kk = 0; kk < 8; ++kk) {
    const int n0 = lower ? 32 * (kk >> 1) : 0;
    const unsigned long long bk = db + (unsigned long long)(n0 * 128 >> 4);
    const unsigned idesc = tc_half_desc(DB - n0, false, false);
    const unsigned d = tmem + n0;
    tc_mma_half(d + DB, da + lo, bk, idesc, kk > 0);
    tc_mma_half(d + DB, da, bk + lo_b, idesc, 1u);
    tc_mma_half(d, da, bk, idesc, kk > 0);
    da += (kk == 3 ? 2 * kLookTile - 96 : 32) >> 4;
    if (kk == 3 && lower) lo_b = lo / 2;
    db += (kk != 3 ? 32 : lower ? 3 * kLookTile / 2 - 96 : 2 * kLookTile - 96) >> 4;
  }
}

// X_pp (columns and rows from xo on) from its chunks to tx, by twelve lanes: rows of
// 64 columns, K-major as a B operand: columns 0 .. 63 hi, then lo, and columns 64
// .. hi and lo of rows 64 .. only (those above are zeros, and not read).
__device__ __forceinline__ void look_load_x(const MatInfo& mi, int xo, unsigned tx,
                                            unsigned long long* bar, int lane) {
  if (lane == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 ::"r"(smem_u32(bar)), "r"(kLookX)
                 : "memory");
  __syncwarp();
  if (lane >= kLookX / 4096) return;
  // 32 rows of one term of 64 columns
  const int h = lane >> 3, term = lane & 1, rc = (h ? lane - 4 : lane) >> 1;
  const unsigned char* src = mi.PX + (long long)(xo / DB) * mi.tile +
                             (long long)(xo / 32 + rc) * kChunk + h * 8192 +
                             term * 4096;
  const unsigned dst =
      tx + (h ? (3 + term) * (kLookTile / 2) : term * kLookTile) + rc * 4096;
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1], 4096, [%2];"
      ::"r"(dst), "l"(src), "r"(smem_u32(bar))
      : "memory");
}

// Sixteen scaled values, columns 16 c .. of 64 of a row, as fp16 terms into the
// row of their tiles.
__device__ __forceinline__ void look_store16(unsigned tile, int row, int c,
                                             const float v[16], float scale) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    unsigned hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      split_half2(scale * v[8 * i + 2 * e], scale * v[8 * i + 2 * e + 1], hi[e],
                  lo[e]);
    const unsigned d = tile + sw128_chunk_off(row, 2 * c + i);
    sts128(d, make_float4(__uint_as_float(hi[0]), __uint_as_float(hi[1]),
                          __uint_as_float(hi[2]), __uint_as_float(hi[3])));
    sts128(d + kLookTile,
           make_float4(__uint_as_float(lo[0]), __uint_as_float(lo[1]),
                       __uint_as_float(lo[2]), __uint_as_float(lo[3])));
  }
}

// 16 bytes global -> shared without a register in between; zeros if !there.
__device__ __forceinline__ void cp_async16(unsigned dst, const float* src,
                                           bool there = true) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst),
               "l"(src), "r"(there ? 16 : 0)
               : "memory");
}

// Eight rows of a 128 x 128 block of fp32 values to ta by a warp, asynchronously, into
// the places of their own terms: piece i of 32 columns in tile i.  Zeros for rows
// from `valid` on.
__device__ __forceinline__ void look_load_a(unsigned ta, const float* block,
                                            long long ld, int row0, int valid,
                                            int lane) {
  const float* src = block + 4 * lane;
  const unsigned dst = ta + (lane >> 3) * kLookTile;
#pragma unroll 2
  for (int row = row0; row < row0 + 8; ++row)
    cp_async16(dst + sw128_chunk_off(row, lane & 7),
               row < valid ? src + row * ld : src, row < valid);
}

// Those rows, once they are there, into their terms, 64 columns at a time.
__device__ __forceinline__ void look_split_a(unsigned char* stage, int row0,
                                             int lane) {
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    __syncwarp();
    const int row = row0 + (lane & 7), c = lane >> 3;
    const float4* src = reinterpret_cast<const float4*>(
        stage + (2 * h + (c >> 1)) * kLookTile + row * 128);
    float v[16];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 u = src[(4 * (c & 1) + e) ^ (row & 7)];
      v[4 * e] = u.x; v[4 * e + 1] = u.y; v[4 * e + 2] = u.z; v[4 * e + 3] = u.w;
    }
    __syncwarp();
    look_store16(smem_u32(stage) + 2 * h * kLookTile, row, c, v, kScaleL);
  }
}

// W_kk (bs x bs) into S; beyond bs the identity, so that the sweeps below run
// over whole sub-blocks.  Asynchronous: the caller waits (diag_load_wait) before
// its next barrier.
__device__ __forceinline__ void diag_load(const float* Wd, long long ld, int bs,
                                          float* S) {
  const int rows = (bs + SB - 1) / SB * SB;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < rows * (DB / 4); idx += DT) {
    const int r = idx >> 5, c = (idx & 31) * 4;
    float* dst = &S[r * DLD + c];
    if (c > (r | (SB - 1))) continue;       // above the diagonal: never read
    if (r < bs && c + 3 < bs) {
      cp_async16(smem_u32(dst), &Wd[r * ld + c]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v = (r == c + e) ? 1.f : 0.f;
        if (r < bs && c + e < bs) v = Wd[r * ld + c + e];
        dst[e] = v;
      }
    }
  }
}

__device__ __forceinline__ void diag_load_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Barriers and tensor memory; needs nothing of the matrix but the number of
// sub-blocks.
__device__ __forceinline__ void diag_begin(DiagControl* ctl, int np) {
  if (threadIdx.x >= 32 && threadIdx.x < 48) {
    const int i = threadIdx.x - 32;
    mbar_init(&ctl->step[i >> 2][i & 3], 1);
    mbar_init(&ctl->crit[i >> 2][i & 3], 1);
    if (i < 2) mbar_init(&ctl->done[i], 1);
    if (i == 3) mbar_init(&ctl->x_here, 1);
    // (a warp per row-block, X^T's new rows, and the warp that has taken the next
    // diagonal sub-block's products out)
    if (i == 0) mbar_init(&ctl->rows, np + 2);
    if (i == 1) mbar_init(&ctl->next, 1);
    if (i == 2) mbar_init(&ctl->beyond, 1);
    ctl->abort_flag = 0;
    ctl->grace = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(kDiagCols)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
    let_next_launch_begin();
  }
}

// The diagonal block of step k has received the updates of all steps before
// k - 1; the update of step k - 1,
//   D = W_kk - L' L'^T,  L' = A' X_pp^T,
// is computed here from A' (block (k, k-1), which the panel solve of step k-1
// leaves as it was) and X_pp (inverse of the previous diagonal block's factor),
// so that this kernel does not have to wait for the panel solve and panel
// update of step k - 1.  Both products run on the tensor cores (tcgen05,
// operands in two fp16 terms, accumulators in tensor memory).  X_pp comes as the
// chunks that the diagonal kernel of step k - 1 left.  Result: D in S.
__device__ __forceinline__ void diag_lookahead(const MatInfo& mi, int o, int bs,
                                               float* S,
                                               unsigned char* stage,
                                               DiagControl* ctl) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long ld = mi.ld;
  const unsigned ta = smem_u32(stage), tx = ta + 4 * kLookTile;
  diag_begin(ctl, (bs + SB - 1) / SB);
  look_load_a(ta, mi.W + (long long)o * ld + (o - DB), ld, 8 * warp, bs, lane);
  asm volatile("cp.async.commit_group;" ::: "memory");
  // (the update is subtracted from it at the end)
  diag_load(mi.W + (long long)o * ld + o, ld, bs, S);
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (warp == 1) {
    __syncwarp();
    // all of the above and the terms of A' may run beside the diagonal kernel of
    // step k - 1; X_pp, and whatever this kernel writes, comes after it
    wait_for_launch_before();
    look_load_x(mi, o - DB, tx, &ctl->x_here, lane);
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  look_split_a(stage, 8 * warp, lane);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = ctl->tmem_base;

  // ---- L' = A' X_pp^T
  if (warp == 0) {
    const bool go = diag_wait(&ctl->x_here, 0, &ctl->abort_flag);
    if (__all_sync(0xffffffffu, go) && elect_one()) {
      look_mma(tmem, ta, tx, true);
      tc_commit(&ctl->done[0]);
    }
    __syncwarp();
  }
  bool ok = diag_wait_tmem(&ctl->done[0], 0, &ctl->abort_flag);

  // ---- L' out of tensor memory, split, into the operand tiles of the second
  // product (A and B are the same matrix)
  const int q = warp & 3, h = warp >> 2;
  const int row = 32 * q + lane;
  const unsigned acc = tmem + ((unsigned)(32 * q) << 16) + (unsigned)(32 * h);
  if (ok) {
    // (the scale of A' X_pp^T is kScaleL kScaleX; L' keeps kScaleL of it)
#pragma unroll 1
    for (int cc = 0; cc < 2; ++cc) {
      float v[16], w[16];
      tc_ld16_pair(acc + 16 * cc, acc + 16 * cc + DB, v, w);
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] += w[e];
      look_store16(ta + 2 * (h >> 1) * kLookTile, row, 2 * (h & 1) + cc, v,
                   1.f / kScaleX);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // ---- L' L'^T
  if (warp == 0 && !ctl->abort_flag && elect_one()) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    look_mma(tmem, ta, ta, false);
    tc_commit(&ctl->done[1]);
  }
  diag_load_wait();
  ok = diag_wait_tmem(&ctl->done[1], 0, &ctl->abort_flag);
  __syncthreads();                      // every thread's part of W_kk is there
  if (ok && h <= q) {                   // sub-blocks on and below the diagonal
    constexpr float s = -1.f / (kScaleL * kScaleL);
#pragma unroll 1
    for (int cc = 0; cc < 2; ++cc) {
      float v[16], w[16];
      tc_ld16_pair(acc + 16 * cc, acc + 16 * cc + DB, v, w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4* s4 = reinterpret_cast<float4*>(
            &S[row * DLD + 32 * h + 16 * cc + 4 * i]);
        float4 d = *s4;
        d.x += s * (v[4 * i] + w[4 * i]);
        d.y += s * (v[4 * i + 1] + w[4 * i + 1]);
        d.z += s * (v[4 * i + 2] + w[4 * i + 2]);
        d.w += s * (v[4 * i + 3] + w[4 * i + 3]);
        *s4 = d;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

// ------------------------------------------------ one 128 x 128 diagonal block
// Shared memory of the diagonal kernel, in floats.
constexpr int LSP = SB + 4;    // row pitch of Ls
constexpr int kDiagTile = DB * 128;            // 128 rows x 32 k of two bf16 terms
struct DiagSmem {
  float S[DB * DLD];          // D / L in the sub-blocks on and below the
                              // diagonal, X^T in those above it
  float XD[4][SB * SLP];      // X_pp^T: inverse of sub-block p of the diagonal
  float Ls[2][SB][LSP];       // L_pp by columns (p & 1: followers that the chain
  float rl[2][SB];            // does not wait for may be behind it), 1 / l_cc
  float pv[SB][8];            // the running step's eight columns
};

// What lies behind S: the rest of DiagSmem, then (at a multiple of 1024 bytes from
// the look-ahead's stages on) the operand tiles of the elimination.
constexpr int kDiagStage =
    (int)((sizeof(DiagSmem) - DB * DLD * sizeof(float) + 1023) / 1024 * 1024) +
    2 * kDiagTile;
static_assert(kDiagStage <= kLookBytes, "diagonal kernel shared memory");

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Named barriers of the diagonal kernel.
constexpr int kRestWarps = 4;  // warps of diag_base_rest
constexpr int kBarNext = 0;    // + step (1, 2): the columns after the next are
                               // up to date
constexpr int kBarDiag = 3;    // the next diagonal sub-block is up to date
constexpr int kBarStore = 4;   // + p: rows SB p .. of X are in shared memory
constexpr int kBarPre = 8;     // earlier products are out of the next sub-block

// Two multiply-adds an instruction; a pair is a register pair.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpair(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Four floats of shared memory as two pairs.
__device__ __forceinline__ ulonglong2 load_pairs(const float* p) {
  return *reinterpret_cast<const ulonglong2*>(p);
}
__device__ __forceinline__ void store_pairs(float* p, f32x2 a, f32x2 b) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a, b);
}

// Pivot k of an 8 x 8 block: r = 1 / sqrt(q) by the approximation and one
// Newton step; `next`, if given, becomes p / sqrt(q) without waiting for r.  The
// step's own error is far below fp32, the roundings of q r, of the last sum and
// (for `next`) of p r leave 1.5 and 2.5 units of 2^-24 (kfac_selftest_pivots).
// CHECK: a pivot that is not positive (or below the smallest normal number)
// counts as failed and becomes 1.
template <bool CHECK>
__device__ __forceinline__ float diag_pivot(float q, float* next) {
  if (CHECK && !(q >= 1.17549435e-38f)) return 1.f;
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
  const float e = fmaf(-(q * r), r, 1.f);
  if (next != nullptr) {
    const float g = *next * r;
    *next = fmaf(0.5f * g, e, g);
  }
  return fmaf(0.5f * r, e, r);
}

__global__ void pivots_selftest_kernel(int count, const float* q, const float* p,
                                       float* rsqrt, float* quot,
                                       float* checked) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  float next = p[i];
  rsqrt[i] = diag_pivot<false>(q[i], &next);
  quot[i] = next;
  checked[i] = diag_pivot<true>(q[i], nullptr);
}

// Cholesky factor of the 8 x 8 block p (lower part, in place), r = reciprocal
// square roots of the pivots.  The row x goes through the triangle on the way: its
// multiply-adds fill the wait for the next pivot.
template <bool CHECK>
__device__ __forceinline__ void diag_chol8(float p[8][8], float r[8],
                                           float x[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float l = k < 7 ? p[k + 1][k] : 0.f;
    r[k] = diag_pivot<CHECK>(p[k][k], k < 7 ? &l : nullptr);
    x[k] *= r[k];
    if (k == 7) break;
    p[k + 1][k] = CHECK ? p[k + 1][k] * r[k] : l;
#pragma unroll
    for (int i = k + 2; i < 8; ++i) p[i][k] *= r[k];
#pragma unroll
    for (int j = k + 1; j < 8; ++j)
#pragma unroll
      for (int i = j; i < 8; ++i) p[i][j] = fmaf(-p[i][k], p[j][k], p[i][j]);
#pragma unroll
    for (int i = k + 1; i < 8; ++i) x[i] = fmaf(-x[k], p[i][k], x[i]);
  }
}

// The pivot block of the running step (lower part) into every lane.
__device__ __forceinline__ void diag_load8(const DiagSmem& sm, int j,
                                           float blk[8][8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int k = 0; k <= i; k += 4) {
      const float4 v = *reinterpret_cast<const float4*>(&sm.pv[j + i][k]);
      blk[i][k] = v.x; blk[i][k + 1] = v.y;
      blk[i][k + 2] = v.z; blk[i][k + 3] = v.w;
    }
}

// Cholesky factor of sub-block p of the diagonal by one warp, a row per lane,
// eight columns per step in registers.  Every lane factors the 8 x 8 pivot
// block redundantly (fetched through shared memory: 36 shuffles measured 300
// cycles more), so that the serial chain per column is one reciprocal square
// root and a few multiply-adds, and the trip through shared memory that brings
// the columns to the other rows comes once in eight columns.  Of a step's
// rank-8 update this warp applies only the part on the next eight columns; the
// columns after those are updated by other warps (diag_base_rest) meanwhile.
__device__ __forceinline__ void diag_base(DiagSmem& sm, DiagControl* ctl, int p,
                                          int lane, int id, int col0, int* info) {
  const float* row = &sm.S[(SB * p + lane) * DLD + SB * p];
  float* const rl = sm.rl[p & 1];
  f32x2 y[4];                  // this lane's row, eight columns
  {
    const ulonglong2 u = load_pairs(row), v = load_pairs(row + 4);
    y[0] = u.x; y[1] = u.y; y[2] = v.x; y[3] = v.y;
  }
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    const int j = 8 * s;
    float blk[8][8], r[8], x[8];
    store_pairs(&sm.pv[lane][0], y[0], y[1]);
    store_pairs(&sm.pv[lane][4], y[2], y[3]);
    __syncwarp();
    diag_load8(sm, j, blk);
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const float2 v = unpair(y[k / 2]);
      x[k] = v.x; x[k + 1] = v.y;
    }
    // (rows above the pivot: unused)
    diag_chol8<false>(blk, r, x);
    if (!(r[7] == r[7])) {
      // some pivot is not positive (every later one is NaN then): report the
      // first, carry on with ones in their place
      diag_load8(sm, j, blk);
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        const float2 v = unpair(y[k / 2]);
        x[k] = v.x; x[k + 1] = v.y;
      }
      diag_chol8<true>(blk, r, x);
      int first = 0;
#pragma unroll
      for (int k = 7; k >= 0; --k)
        if (!(blk[k][k] >= 1.17549435e-38f)) first = j + k + 1;
      if (lane == 0 && first != 0) atomicCAS(&info[id], 0, col0 + first);
    }
    float (*L)[LSP] = &sm.Ls[p & 1][j];
#pragma unroll
    for (int k = 0; k < 8; ++k) L[k][lane] = x[k];
    // (every lane stores the same)
    *reinterpret_cast<float4*>(&rl[j]) = make_float4(r[0], r[1], r[2], r[3]);
    *reinterpret_cast<float4*>(&rl[j + 4]) = make_float4(r[4], r[5], r[6], r[7]);
    __syncwarp();
    if (lane == 0) mbar_arrive(&ctl->step[p][s]);
    if (s == 3) break;
    if (s > 0) bar_sync(kBarNext + s, 32 + 32 * kRestWarps);
    {
      const ulonglong2 u = load_pairs(row + j + 8), v = load_pairs(row + j + 12);
      y[0] = u.x; y[1] = u.y; y[2] = v.x; y[3] = v.y;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const ulonglong2 l = load_pairs(&L[k][j + 8]);
      const ulonglong2 m = load_pairs(&L[k][j + 12]);
      const f32x2 nx = pair(-x[k], -x[k]);
      y[0] = fma2(nx, l.x, y[0]); y[1] = fma2(nx, l.y, y[1]);
      y[2] = fma2(nx, m.x, y[2]); y[3] = fma2(nx, m.y, y[3]);
    }
  }
}

// The part of diag_base's updates that its own warp leaves: step s on columns
// 8 s + 16 .. 31 of the sub-block, in shared memory, four columns per warp.  Each has
// the same columns in both steps: nothing orders one warp's first step before
// another's second.
__device__ __forceinline__ void diag_base_rest(DiagSmem& sm, DiagControl* ctl,
                                               int p, int lane, int h) {
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    diag_wait(&ctl->step[p][s], 0, &ctl->abort_flag);
    const int c = 16 + 4 * h;
    if (c >= 8 * s + 16) {
      const float (*L)[LSP] = &sm.Ls[p & 1][8 * s];
      float* row = &sm.S[(SB * p + lane) * DLD + SB * p + c];
      ulonglong2 u = load_pairs(row);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float x = L[k][lane];
        const ulonglong2 l = load_pairs(&L[k][c]);
        const f32x2 nx = pair(-x, -x);
        u.x = fma2(nx, l.x, u.x); u.y = fma2(nx, l.y, u.y);
      }
      store_pairs(row, u.x, u.y);
      __syncwarp();
    }
    bar_arrive(kBarNext + s + 1, 32 + 32 * kRestWarps);
  }
}

// Eight columns (step s) of a row as three bf16 terms, 24 significant bits, into the
// operand tiles: hi and mid in the halves of a row of the first, lo in the second.
// (lo is cut off, not rounded, which keeps a NaN.)
__device__ __forceinline__ void diag_store_terms(unsigned tile, int row, int s,
                                                 const float x[8]) {
  unsigned hi[4], mid[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x0 = x[2 * i], x1 = x[2 * i + 1];
    const unsigned a0 = __float_as_uint(x0) + 0x8000u;
    const unsigned a1 = __float_as_uint(x1) + 0x8000u;
    hi[i] = __byte_perm(a0, a1, 0x7632);
    const float y0 = x0 - __uint_as_float(a0 & 0xffff0000u);
    const float y1 = x1 - __uint_as_float(a1 & 0xffff0000u);
    const unsigned b0 = __float_as_uint(y0) + 0x8000u;
    const unsigned b1 = __float_as_uint(y1) + 0x8000u;
    mid[i] = __byte_perm(b0, b1, 0x7632);
    lo[i] = __byte_perm(__float_as_uint(y0 - __uint_as_float(b0 & 0xffff0000u)),
                        __float_as_uint(y1 - __uint_as_float(b1 & 0xffff0000u)),
                        0x7632);
  }
  auto put = [&](unsigned t, int chunk, const unsigned v[4]) {
    sts128(t + sw128_chunk_off(row, chunk),
           make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]),
                       __uint_as_float(v[2]), __uint_as_float(v[3])));
  };
  put(tile, s, hi);
  put(tile, 4 + s, mid);
  put(tile + kDiagTile, s, lo);
}

// Step s of a row per lane.  `out` gets the finished values (NULL: a row of L that
// nothing reads but as an operand), `tile` its terms (0: none; row `tile_row`);
// `crit`, if given, is told when they are in `out`.
__device__ __forceinline__ void diag_follow_step(const DiagSmem& sm, int p, int s,
                                                 f32x2 a[SB / 2], float* out,
                                                 unsigned tile, int tile_row,
                                                 int lane,
                                                 unsigned long long* crit) {
  const int j = 8 * s;
  const float (*L)[LSP] = &sm.Ls[p & 1][j];
  float r[8], l[8][8], x[8];
#pragma unroll
  for (int k = 0; k < 8; k += 4) {
    const float4 v = *reinterpret_cast<const float4*>(&sm.rl[p & 1][j + k]);
    r[k] = v.x; r[k + 1] = v.y; r[k + 2] = v.z; r[k + 3] = v.w;
  }
#pragma unroll
  for (int k = 0; k < 7; ++k)
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      if (i + 3 <= k) continue;
      const float4 v = *reinterpret_cast<const float4*>(&L[k][j + i]);
      l[i][k] = v.x; l[i + 1][k] = v.y; l[i + 2][k] = v.z; l[i + 3][k] = v.w;
    }
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const float2 v = unpair(a[k / 2]);
    x[k] = v.x; x[k + 1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] *= r[k];
#pragma unroll
    for (int i = k + 1; i < 8; ++i) x[i] = fmaf(-x[k], l[i][k], x[i]);
  }
  if (out != nullptr) {
    float4* row = reinterpret_cast<float4*>(&out[j]);
    row[0] = make_float4(x[0], x[1], x[2], x[3]);
    row[1] = make_float4(x[4], x[5], x[6], x[7]);
  }
  if (crit != nullptr) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&crit[s]);
  }
  if (tile != 0) diag_store_terms(tile, tile_row, s, x);
  // the registers move down by eight columns
  f32x2 nx[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) nx[k] = pair(-x[k], -x[k]);
#pragma unroll
  for (int c = 0; c < 24; c += 8) {
    if (c >= 24 - j) break;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      const int d = (c + h) / 2;
      f32x2 u = a[d + 4], v = a[d + 5];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const ulonglong2 w = load_pairs(&L[k][j + 8 + c + h]);
        u = fma2(nx[k], w.x, u);
        v = fma2(nx[k], w.y, v);
      }
      a[d] = u; a[d + 1] = v;
    }
  }
}

// D(128 x 32 nc) += rows of the operand tiles times rows 32 c .. of them, in six
// terms (all but mid lo, lo mid and lo lo): columns 32 c .. of the accumulators for
// hi hi, those 128 columns on for the others.  The tensor core adds with
// truncation; products of 8-bit terms leave it little to cut off, and what it cuts
// off the others is below their 2^-8.
__device__ __forceinline__ void diag_mma(unsigned tmem, unsigned tile, int c,
                                         int nc, bool first) {
  constexpr unsigned long long mid = 64 >> 4, lo = kDiagTile >> 4;
  const unsigned idesc = tc_bf16_desc(SB * nc);
  const unsigned d = tmem + SB * c;
  unsigned long long a = tc_smem_desc(tile);
  unsigned long long b = tc_smem_desc(tile + c * SB * 128);
#pragma unroll 1
  for (int kk = 0; kk < 2; ++kk) {
    const unsigned acc = !first || kk > 0;
    tc_mma_half(d + DB, a + lo, b, idesc, acc);
    tc_mma_half(d + DB, a, b + lo, idesc, 1u);
    tc_mma_half(d + DB, a + mid, b + mid, idesc, 1u);
    tc_mma_half(d + DB, a + mid, b, idesc, 1u);
    tc_mma_half(d + DB, a, b + mid, idesc, 1u);
    tc_mma_half(d, a, b, idesc, acc);
    a += 32 >> 4;
    b += 32 >> 4;
  }
}

// Zeros into a warp's lanes of 32 columns of tensor memory.
__device__ __forceinline__ void diag_clear(unsigned taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      ::"r"(taddr), "r"(0)
      : "memory");
}

// 32 columns of a warp's lanes of tensor memory: the hi hi and cross accumulators.
__device__ __forceinline__ void diag_fetch(unsigned t, f32x2 v[SB / 2]) {
#pragma unroll
  for (int cc = 0; cc < SB; cc += 16) {
    float m[16], x[16];
    tc_ld16_pair(t + cc, t + DB + cc, m, x);
#pragma unroll
    for (int i = 0; i < 16; i += 2)
      v[(cc + i) / 2] = pair(m[i] + x[i], m[i + 1] + x[i + 1]);
  }
}

// row <- row L_pp^-T for a row per lane, step by step behind diag_base: row `lane`
// of row-block r, columns of sub-block p.  A row of D (r > p) comes from S less the
// products collected in tensor memory, one of X^T (r < p) is minus them; that of
// X^T's new row-block (r == p) starts as the unit vector e_lane and ends as row
// `lane` of X_pp^T.
__device__ __forceinline__ void diag_follow(DiagSmem& sm, DiagControl* ctl,
                                            unsigned tmem, int p, int r, int lane,
                                            unsigned tile) {
  f32x2 a[SB / 2];
  float* src = &sm.S[(SB * r + lane) * DLD + SB * p];
  float* out = r == p ? &sm.XD[p][lane * SLP] : r <= p + 1 ? src : nullptr;
#pragma unroll
  for (int j = 0; j < SB; j += 4) {
    ulonglong2 v = make_ulonglong2(0, 0);
    if (r > p) v = load_pairs(&src[j]);
    if (r == p && (lane & ~3) == j)
      v = make_ulonglong2(pair(j == lane ? 1.f : 0.f, j + 1 == lane ? 1.f : 0.f),
                          pair(j + 2 == lane ? 1.f : 0.f, j + 3 == lane ? 1.f : 0.f));
    a[j / 2] = v.x; a[j / 2 + 1] = v.y;
  }
  if (p > 0) {
    if (r != p) {
      if (diag_wait_tmem(&ctl->next, (p - 1) & 1, &ctl->abort_flag)) {
        f32x2 t[SB / 2];
        diag_fetch(tmem + ((unsigned)(SB * r) << 16) + (unsigned)(SB * p), t);
        const f32x2 minus = pair(-1.f, -1.f);
#pragma unroll
        for (int j = 0; j < SB / 2; ++j) a[j] = fma2(t[j], minus, a[j]);
      }
    }
    // the products of the sub-block before have read the tiles
    diag_wait(&ctl->beyond, (p - 1) & 1, &ctl->abort_flag);
  }
  unsigned long long* crit = r == p + 1 ? ctl->crit[p] : nullptr;
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    diag_wait(&ctl->step[p][s], 0, &ctl->abort_flag);
    diag_follow_step(sm, p, s, a, out, tile, SB * r + lane, lane, crit);
  }
}

// The next diagonal sub-block loses its row-block's product with itself, eight
// columns as soon as they are there: 16 rows from r0 on, 16 columns from c0 on.
// Lane (rg, cg) holds rows rg + 8 i, columns cg + 4 j, sums over even and odd k.
__device__ __forceinline__ void diag_next(DiagSmem& sm, DiagControl* ctl, int p,
                                          int r0, int c0, int lane) {
  constexpr int CJ = 4;
  const int rg = lane >> 2, cg = lane & 3;
  float* C = &sm.S[(SB * (p + 1) + r0 + rg) * DLD + SB * (p + 1) + c0 + cg];
  const float* A = &sm.S[(SB * (p + 1) + r0 + rg) * DLD + SB * p];
  const float* B = &sm.S[(SB * (p + 1) + c0 + cg) * DLD + SB * p];
  float d[2][CJ];
  f32x2 acc[2][CJ];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      d[i][j] = C[8 * i * DLD + 4 * j];
      acc[i][j] = 0;
    }
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    diag_wait(&ctl->crit[p][s], 0, &ctl->abort_flag);
#pragma unroll 1
    for (int k = 8 * s; k < 8 * s + 8; k += 4) {
      ulonglong2 a[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = load_pairs(&A[8 * i * DLD + k]);
#pragma unroll
      for (int j = 0; j < CJ; ++j) {
        const ulonglong2 b = load_pairs(&B[4 * j * DLD + k]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          acc[i][j] = fma2(a[i].x, b.x, acc[i][j]);
          acc[i][j] = fma2(a[i].y, b.y, acc[i][j]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      const float2 v = unpair(acc[i][j]);
      C[8 * i * DLD + 4 * j] = d[i][j] - (v.x + v.y);
    }
}

// Sub-block (p, u) of X, or its upper or lower half, to global memory: a lane
// takes a 4 x 4 block, four words along the rows of X^T, turned by naming
// registers, so that X and its fp16 terms are stored in words of four columns.
// Lanes are laid out so that a quarter warp's loads fall into different banks.
__device__ __forceinline__ void diag_store(const DiagSmem& sm, const MatInfo& mi,
                                           int o, int bs, int p, int u, int half,
                                           int lane) {
  const long long ld = mi.ld;
  float* Xd = mi.X + (long long)o * ld + o;
  unsigned char* const px = mi.PX + (long long)(o / DB) * mi.tile;
  const int c = 4 * (lane >> 2), r = 16 * half + 4 * (lane & 3);
  float x[4][4];              // [column][row]
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float4 v = *reinterpret_cast<const float4*>(
        u == p ? &sm.XD[u][(c + e) * SLP + r]
               : &sm.S[(SB * u + c + e) * DLD + SB * p + r]);
    x[e][0] = v.x; x[e][1] = v.y; x[e][2] = v.z; x[e][3] = v.w;
  }
  const int gc = SB * u + c;
  const int gr0 = SB * p + r;
  float* dst = Xd + gr0 * ld + gc;
  unsigned char* q = px + (long long)((o + gr0) >> 5) * kChunk + (gc >> 6) * 8192 +
                     8 * ((gc >> 2) & 1);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (gr0 + e >= bs) break;
    // (columns past bs are zeros above the diagonal, inside the row pitch)
    *reinterpret_cast<float4*>(dst + e * ld) =
        make_float4(x[0][e], x[1][e], x[2][e], x[3][e]);
    unsigned h0, h1, l0, l1;
    split_half2(kScaleX * x[0][e], kScaleX * x[1][e], h0, l0);
    split_half2(kScaleX * x[2][e], kScaleX * x[3][e], h1, l1);
    unsigned char* w = q + sw128_chunk_off((gr0 + e) & 31, (gc & 63) >> 3);
    *reinterpret_cast<uint2*>(w) = make_uint2(h0, h1);
    *reinterpret_cast<uint2*>(w + 4096) = make_uint2(l0, l1);
  }
}

// Factor one diagonal block (<= 128 x 128) of W and invert the resulting
// triangle: X_kk <- L_kk^-1 (lower part; nothing reads L_kk itself).  One CTA
// of 16 warps per matrix that still has a block at `step`.
//
// Elimination of [D; I] by four sub-blocks of 32 columns: row-blocks in play at
// sub-block p are p .. 3 of D and 0 .. p of X^T (which starts as I).  Bound:
// the serial chain of 128 pivots.  So per sub-block one warp runs the pivot
// chain alone (diag_base), four apply what it leaves of its own updates, a warp per
// row-block carries the others behind it (diag_follow), and three take the next
// row-block's products out of the next diagonal sub-block, where the chain goes on
// (diag_next).
//
// All other products of the finished columns with the later ones run on the tensor
// cores (tcgen05): the followers leave their rows as bf16 terms, and D(r, c) and
// X^T(r, c) lose rows r times rows c, for all r at once, collected in tensor
// memory over the sub-blocks; first the next column, which the followers fetch,
// then those beyond.  Row-block r takes D's products with columns it does not have
// until X^T's row r begins: its warp clears those accumulators before.
//
// What bounds the work beside the chain, measured in cycles of the block at 128
// rows: these products on the CUDA cores, six warps with 2 x 8 values a lane, took
// 12 800 cycles of shared-memory loads, more than the chain itself takes, and
// delayed its own loads; in two TF32 terms they were as fast as now but left
// inverses of 128 rows 1.24 times the error, in three bf16 terms 0.92 times.
// Followers on mma.sync take 1400 cycles a step, with multiply-adds 550 to 1150.
// And the instruction cache of an SM holds about 2000 instructions: code that does
// not fit, or runs once, costs three cycles an instruction and more, so loops that
// are not the chain's are left rolled (8200 instructions with the look-ahead,
// 46 900 cycles; 3400 now, 42 000; 56 000 before all of this).
//
// A row panel of X is stored when its sub-block is through, beside the next.
//
// 128 rows: 16 us with the launch, 22 us with the look-ahead in front (20.5 and 30
// before), 18 of them behind the end of the kernel in front.
template <bool LOOK>
__global__ void __launch_bounds__(DT, 1)
chol_diag_kernel(const MatInfo* __restrict__ mats, int step, int* info) {
  extern __shared__ __align__(16) float dsm[];
  DiagSmem& sm = *reinterpret_cast<DiagSmem*>(dsm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the operand stages of the look-ahead alias everything behind S, which is
  // written only after its last barrier
  unsigned char* stage = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(dsm + DB * DLD) + 1023) & ~(uintptr_t)1023);
  DiagControl* ctl = reinterpret_cast<DiagControl*>(
      stage + (LOOK ? kLookBytes : kDiagStage));
  const MatInfo mi = mats[blockIdx.x];
  const int id = mi.id;
  const int o = step * DB;
  const int bs = min(DB, mi.d - o);
  const int np = (bs + SB - 1) / SB;      // sub-blocks in use
  if (LOOK) {
    diag_lookahead(mi, o, bs, sm.S, stage, ctl);
  } else {
    diag_load(mi.W + (long long)o * mi.ld + o, mi.ld, bs, sm.S);
    diag_begin(ctl, np);
    diag_load_wait();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = ctl->tmem_base;
  const unsigned tile = smem_u32(stage + kDiagStage - 2 * kDiagTile);

  // A row panel of X is stored by two warps beside the next sub-block, the last
  // one by all that have nothing else to do then.
  constexpr int kStore = 2, kStoreLast = 9;
  int slot = -1, first = np - 1;           // of a storing warp, its first panel
  if (warp == 0) {
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
      if (p > 0) bar_sync(kBarDiag, 128);
      diag_base(sm, ctl, p, lane, id, o + SB * p, info);
    }
  } else if (warp == 1 || (warp >= 4 && warp < 4 + np)) {
    // row-block warp - 4 (its lanes of tensor memory), warp 1: X^T's new rows
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
      const int r = warp == 1 ? p : warp - 4;
      const bool last = p == np - 1;
      if (warp == 1 || r != p) {
        diag_follow(sm, ctl, tmem, p, r, lane, last ? 0u : tile);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      } else if (p > 0 && !last) {
        // from here on row-block r collects rows of X^T.  (Nothing of `next` is read
        // here, but its next phase is waited for by parity: this one has to be over.)
        diag_wait(&ctl->next, (p - 1) & 1, &ctl->abort_flag);
        const bool ok = diag_wait_tmem(&ctl->beyond, (p - 1) & 1, &ctl->abort_flag);
#pragma unroll 1
        for (int c = 2 * (p + 1); ok && c < 2 * np; ++c)
          diag_clear(tmem + ((unsigned)(SB * r) << 16) +
                     (unsigned)(SB * (c >> 1) + DB * (c & 1)));
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      bar_arrive(kBarStore + p, 32 * (np + 1 + (last ? kStoreLast : kStore)));
      if (last) break;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->rows);
    }
  } else if (warp == 3) {
#pragma unroll 1
    for (int p = 0; p < np - 1; ++p) {
      const bool go = diag_wait_tmem(&ctl->rows, p & 1, &ctl->abort_flag);
      if (go && elect_one()) {
#pragma unroll 1
        for (int part = 0; part < 2; ++part) {
          const int c = p + 1 + part, nc = part ? np - 2 - p : 1;
          if (nc > 0) diag_mma(tmem, tile, c, nc, p == 0);
          tc_commit(part ? &ctl->beyond : &ctl->next);
        }
      }
      __syncwarp();
    }
  } else if (warp == 9 || warp == 10 || warp == 11 || warp == 13) {
    const int h = warp == 13 ? 3 : warp - 9;
#pragma unroll 1
    for (int p = 0; p < np; ++p) diag_base_rest(sm, ctl, p, lane, h);
    slot = h + 5;
  } else if (warp == 2 || warp >= 14) {
    const int u = warp == 2 ? 0 : warp - 13, r = warp - 12;
#pragma unroll 1
    for (int p = 0; p < np - 1; ++p) {
      if (p == 0) {
        if (u == 0 && lane == 0) mbar_arrive(&ctl->rows);
      } else {
        if (r == p + 1) {
          // what earlier sub-blocks have collected for the next diagonal one
          if (diag_wait_tmem(&ctl->beyond, (p - 1) & 1, &ctl->abort_flag)) {
            f32x2 t[SB / 2];
            diag_fetch(tmem + ((unsigned)(SB * r) << 16) + (unsigned)(SB * r), t);
            float* row = &sm.S[(SB * r + lane) * DLD + SB * r];
            const f32x2 minus = pair(-1.f, -1.f);
#pragma unroll
            for (int j = 0; j < SB; j += 4) {
              const ulonglong2 v = load_pairs(&row[j]);
              store_pairs(&row[j], fma2(t[j / 2], minus, v.x),
                          fma2(t[j / 2 + 1], minus, v.y));
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->rows);
        }
        bar_sync(kBarPre, 96);
      }
      diag_next(sm, ctl, p, u ? 16 : 0, u == 2 ? 16 : 0, lane);
      bar_arrive(kBarDiag, 128);
    }
    slot = u + 2;
  } else if (warp == 8 || warp == 12) {
    slot = warp == 8 ? 0 : 1;
    first = 0;
  }
  if (slot >= 0) {
#pragma unroll 1
    for (int p = first; p < np; ++p) {
      const int warps = p == np - 1 ? kStoreLast : kStore;
      bar_sync(kBarStore + p, 32 * (np + 1 + warps));
      if (ctl->abort_flag != 0) continue;
#pragma unroll 1
      for (int u = slot; u < 2 * (p + 1); u += warps)
        diag_store(sm, mi, o, bs, p, u >> 1, u & 1, lane);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    if (ctl->abort_flag != 0) {
      // (its own copies have to be over before the block is)
      if (LOOK) mbar_wait_status(&ctl->x_here, 0, &ctl->grace, &g_diag_status);
      if (lane == 0) atomicExch(&g_diag_status, 1);
    }
    tc_release(tmem, kDiagCols, ctl->abort_flag != 0);
  }
}

// The same on engine 0: fp32 multiply-adds and nothing of the kernel above, as the
// tests hold that one against this.  A column of [D; I] at a time, all of it in one
// square of registers: row i is D's until column i is through, then X^T's, which
// begins on the diagonal.  A thread has rows warp + 16 a, columns lane + 32 b.
// Bound by the chain of its 128 steps, a root, a quotient and a barrier each: 56 us
// for 128 rows with the launch (16 by the kernel above; 159 with the square in shared
// memory and two barriers a step).
__global__ void __launch_bounds__(DT, 1)
chol_diag_ffma_kernel(const MatInfo* __restrict__ mats, int step, int* info) {
  constexpr int RA = DB / (DT / 32), CB = DB / 32;
  __shared__ float cols[2][DB];           // the step's column (twice: one barrier)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MatInfo mi = mats[blockIdx.x];
  const int o = step * DB;
  const int bs = min(DB, mi.d - o);
  const long long ld = mi.ld, at = (long long)o * ld + o;
  float m[RA][CB];
#pragma unroll
  for (int a = 0; a < RA; ++a)
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int i = warp + DT / 32 * a, c = lane + 32 * b;
      m[a][b] = i < bs && c <= i ? mi.W[at + i * ld + c] : 0.f;
    }
#pragma unroll
  for (int b0 = 0; b0 < CB; ++b0) {
#pragma unroll 1
    for (int j = 32 * b0; j < min(bs, 32 * b0 + 32); ++j) {
      float* const col = cols[j & 1];
      if (lane == j - 32 * b0) {
#pragma unroll
        for (int a = 0; a < RA; ++a) col[warp + DT / 32 * a] = m[a][b0];
      }
      __syncthreads();
      const float q = col[j];
      const bool positive = q >= 1.17549435e-38f;
      const float r = positive ? 1.f / sqrtf(q) : 1.f;
      if (threadIdx.x == 0 && !positive) atomicCAS(&info[mi.id], 0, o + j + 1);
      float x[RA], y[CB];
#pragma unroll
      for (int a = 0; a < RA; ++a) x[a] = col[warp + DT / 32 * a] * r;
#pragma unroll
      for (int b = b0; b < CB; ++b) y[b] = col[lane + 32 * b] * r;
#pragma unroll
      for (int a = 0; a < RA; ++a) {
        // row-block a / 2: of X^T in front of this one, of D behind it, where what
        // is above the diagonal does not count until the row begins again
        const bool begins = a / 2 == b0 && warp + DT / 32 * a == j;
        if (begins) x[a] = r;
#pragma unroll
        for (int b = b0; b < (a / 2 > b0 ? a / 2 + 1 : CB); ++b) {
          if (b > b0 || lane > j - 32 * b0)
            m[a][b] = fmaf(-x[a], y[b], begins ? 0.f : m[a][b]);
          else if (lane == j - 32 * b0)
            m[a][b] = x[a];
        }
      }
    }
  }
  // (above the diagonal X is zeros from the start)
#pragma unroll
  for (int a = 0; a < RA; ++a)
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int i = warp + DT / 32 * a, c = lane + 32 * b;
      if (c >= i && c < bs) mi.X[at + c * ld + i] = m[a][b];
    }
}

// ------------------------------------------------------------ panel solve
// L = A' X_kk^T for the rows below diagonal block `step`: a CTA per 128 rows
// (blockIdx.x) of a matrix (blockIdx.y), the look-ahead's first product.  W stays as
// it is; L goes to its chunks.  Two CTAs an SM.  One product of 128^3 takes a
// microsecond; the rest is 64 KB of A', 48 KB of X_kk and 64 KB of L for each CTA,
// one after the other, of which A' and its terms come before the wait for the
// diagonal kernel.  (By the tile kernel, which reads X_kk as fp32 and splits it in
// every CTA, 7.5 to 9.5 us a launch; solve and update behind a diagonal kernel 18.5
// us then, 11.5 now.)
constexpr int kSolveThreads = 256;
struct SolveControl {
  unsigned long long x_here, done;
  unsigned tmem_base;
  volatile int abort_flag, grace;
};
constexpr int kSolveSmemBytes = kLookBytes + 64;
static_assert(sizeof(SolveControl) <= 64 && 2 * (kSolveSmemBytes + 1024) <= 227 * 1024,
              "panel solve shared memory");

__global__ void __launch_bounds__(kSolveThreads, 2)
panel_solve_kernel(const MatInfo* __restrict__ mats, int step) {
  extern __shared__ __align__(1024) unsigned char stage[];
  SolveControl* ctl = reinterpret_cast<SolveControl*>(stage + kLookBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MatInfo mi = mats[blockIdx.y];
  const int o = step * DB, r0 = o + DB * (1 + (int)blockIdx.x);
  const int rows = mi.d - r0;
  if (rows <= 0) return;
  const unsigned ta = smem_u32(stage), tx = ta + 4 * kLookTile;
  const float* block = mi.W + (long long)r0 * mi.ld + o;
  look_load_a(ta, block, mi.ld, 8 * warp, rows, lane);
  look_load_a(ta, block, mi.ld, 8 * warp + 64, rows, lane);
  if (warp == 0) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
        ::"r"(smem_u32(&ctl->tmem_base)), "r"(kDiagCols)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"
                 ::: "memory");
    let_next_launch_begin();
  } else if (warp == 1) {
    if (lane == 0) {
      mbar_init(&ctl->x_here, 1);
      mbar_init(&ctl->done, 1);
      ctl->abort_flag = 0;
      ctl->grace = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  }
  diag_load_wait();
  look_split_a(stage, 8 * warp, lane);
  look_split_a(stage, 8 * warp + 64, lane);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  wait_for_launch_before();
  if (warp == 1) look_load_x(mi, o, tx, &ctl->x_here, lane);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = ctl->tmem_base;
  if (warp == 0) {
    const bool go = diag_wait(&ctl->x_here, 0, &ctl->abort_flag);
    if (__all_sync(0xffffffffu, go) && elect_one()) {
      look_mma(tmem, ta, tx, true);
      tc_commit(&ctl->done);
    }
    __syncwarp();
  }
  const bool ok = diag_wait_tmem(&ctl->done, 0, &ctl->abort_flag);
  if (ok) {
    // a warp: 32 rows, 64 columns; A' has been read
    const int q = warp & 3, h = warp >> 2, row = 32 * q + lane;
    const unsigned acc = tmem + ((unsigned)(32 * q) << 16) + (unsigned)(64 * h);
#pragma unroll 1
    for (int cc = 0; cc < 4; ++cc) {
      float v[16], w[16];
      tc_ld16_pair(acc + 16 * cc, acc + 16 * cc + DB, v, w);
      const unsigned chunk = ta + (2 * h + (cc >> 1)) * kChunk;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        unsigned hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // (the scale of A' X_kk^T is kScaleL kScaleX; L keeps kScaleL of it)
          constexpr float s = 1.f / kScaleX;
          const int c = 8 * i + 2 * e;
          split_half2(s * (v[c] + w[c]), s * (v[c + 1] + w[c + 1]), hi[e], lo[e]);
        }
        const unsigned d = chunk + sw128_chunk_off(row, 2 * (cc & 1) + i);
        sts128(d, make_float4(__uint_as_float(hi[0]), __uint_as_float(hi[1]),
                              __uint_as_float(hi[2]), __uint_as_float(hi[3])));
        sts128(d ^ 0x40u,
               make_float4(__uint_as_float(lo[0]), __uint_as_float(lo[1]),
                           __uint_as_float(lo[2]), __uint_as_float(lo[3])));
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1 && lane == 0 && ctl->abort_flag == 0) {
    // (rows past the matrix: zeros, as the chunks' rows there are)
    unsigned char* dst =
        mi.PL + (long long)(r0 / DB) * mi.tile + (long long)(o / 32) * kChunk;
    asm volatile(
        "cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
        ::"l"(dst), "r"(ta), "r"(4 * kChunk)
        : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  if (warp == 0) {
    if (ctl->abort_flag != 0) {
      // (its own copies have to be over before the block is)
      mbar_wait_status(&ctl->x_here, 0, &ctl->grace, &g_diag_status);
      if (lane == 0) atomicExch(&g_diag_status, 1);
    }
    tc_release(tmem, kDiagCols, ctl->abort_flag != 0);
  }
}

// ---------------------------------------------------------------- refinement
// One step of iterative refinement for factors whose fp32 inverse is visibly
// off (ill-conditioned factors: the error of any fp32 inverse grows with the
// condition number).  With R = I - (F + add I) X accumulated in fp64 from the
// fp32 data, X <- X + X R has the error of X squared (times the condition
// number), so one step is enough.  Whether a factor needs the step is decided
// on the device from a probe: for a fixed +-1 vector v,
//   t = X v,  r = v - (F + add I) t,  e = X r   (fp64 accumulation)
// e estimates (X - A^-1) v, so |e| / |t| estimates the relative error of X;
// the step runs when that exceeds `threshold` and d <= `max_dim`.
constexpr int kRefineDimCap = 1024;   // larger factors are not refined

struct RefineItem {
  int mat;          // index into the plan's matrices
  int d;
  int tile_begin;   // first 64 x 64 tile of this matrix in the residual grid
  int pad_;
  double* vec;      // 2 d doubles: t, r
};

__device__ __forceinline__ float probe_sign(int i) {
  unsigned h = (unsigned)i * 2654435761u;
  h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
  return (h & 1u) ? 1.f : -1.f;
}

__device__ __forceinline__ float damp_of_row(const MatInfo& mi, float add,
                                             float add2, int row) {
  return (mi.role == 2 && 2 * row >= mi.d) ? add2 : add;
}

// stage 0: t = X v; stage 1: r = v - (F + add I) t; stage 2: e = X r and
// sums[item] += (|e|^2, |t|^2).  One warp per row, blockIdx.y = item.
__global__ void __launch_bounds__(256)
refine_probe_kernel(const MatInfo* __restrict__ mats,
                    const RefineItem* __restrict__ items,
                    const float* add, const float* add2, double* sums,
                    const RunParams* __restrict__ prm, int stage) {
  let_next_launch_begin();
  wait_for_launch_before();
  if (prm->refine_max_dim <= 0) return;
  const RefineItem it = items[blockIdx.y];
  const MatInfo mi = mats[it.mat];
  const int d = it.d;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (stage == 1 && blockIdx.x == 0 && threadIdx.x == 0) {
    sums[2 * blockIdx.y] = 0.0;
    sums[2 * blockIdx.y + 1] = 0.0;
  }
  if (8 * blockIdx.x >= d) return;
  double* t = it.vec;
  double* r = it.vec + d;
  double s = 0.0;
  if (row < d) {
    const float* mrow = (stage == 1 ? mi.F : mi.inv) + (long long)row * d;
    const double* x = stage == 1 ? t : r;
    // eight loads of the row in flight per lane
    for (int c0 = lane; c0 < d; c0 += 256) {
      float m[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        m[i] = c0 + 32 * i < d ? mrow[c0 + 32 * i] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = c0 + 32 * i;
        if (c < d) s += (double)m[i] * (stage == 0 ? (double)probe_sign(c) : x[c]);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double part[2][8];
  if (lane == 0) {
    double e2 = 0.0, t2 = 0.0;
    if (row < d) {
      if (stage == 0) {
        t[row] = s;
      } else if (stage == 1) {
        const float a = damp_of_row(mi, add[it.mat], add2[it.mat], row);
        r[row] = (double)probe_sign(row) - (s + (double)a * t[row]);
      } else {
        e2 = s * s;
        t2 = t[row] * t[row];
      }
    }
    part[0][threadIdx.x >> 5] = e2;
    part[1][threadIdx.x >> 5] = t2;
  }
  if (stage != 2) return;
  // (one addition per block: the rows of a matrix share two words)
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = 0.0;
    for (int w = 0; w < 8; ++w) v += part[threadIdx.x][w];
    atomicAdd(&sums[2 * blockIdx.y + threadIdx.x], v);
  }
}

// Which matrices the step refines, and how many: one block, as the count has to be
// whole when it is stored.
constexpr int kGateThreads = 256;
__global__ void __launch_bounds__(kGateThreads)
refine_gate_kernel(const RefineItem* __restrict__ items, int n, const double* sums,
                   const RunParams* __restrict__ prm, int* gate,
                   int* refined_count) {
  let_next_launch_begin();
  wait_for_launch_before();
  const int max_dim = prm->refine_max_dim;
  const double thr = (double)prm->refine_threshold;
  int refined = 0;
  for (int i0 = 0; i0 < n; i0 += kGateThreads) {
    const int i = i0 + (int)threadIdx.x;
    int on = 0;
    if (i < n) {
      const double e2 = sums[2 * i], t2 = sums[2 * i + 1];
      // a NaN estimate (broken factorisation) is left alone: info reports it
      on = items[i].d <= max_dim && e2 > thr * thr * t2;
      gate[i] = on;
    }
    refined += __syncthreads_count(on);
  }
  if (threadIdx.x == 0) *refined_count = refined;
}

// R = I - (F + add I) X for a 64 x 64 tile, fp64 accumulation, R stored as
// fp32 into the matrix's W scratch.  256 threads, 4 x 4 outputs each.
__global__ void __launch_bounds__(256)
refine_residual_kernel(const MatInfo* __restrict__ mats,
                       const RefineItem* __restrict__ items, int nitems,
                       const float* add, const float* add2, const int* gate) {
  __shared__ double As[16][64 + 2];   // As[k][i] = A[i0 + i][k0 + k]
  __shared__ double Bs[16][64 + 2];   // Bs[k][j] = X[k0 + k][j0 + j]
  __shared__ int s_item;
  const int tid = threadIdx.x;
  if (tid == 0) {
    int lo = 0, hi = nitems - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (items[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    s_item = lo;
  }
  let_next_launch_begin();
  wait_for_launch_before();
  __syncthreads();
  const int item = s_item;
  if (gate[item] == 0) return;
  const RefineItem it = items[item];
  const MatInfo mi = mats[it.mat];
  const int d = it.d;
  const int nt = (d + 63) >> 6;
  const int lt = blockIdx.x - it.tile_begin;
  const int i0 = (lt / nt) * 64, j0 = (lt % nt) * 64;
  const float a1 = add[it.mat], a2 = add2[it.mat];
  const int ty = tid >> 4, tx = tid & 15;
  double acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
  // loaders: A tile 64 rows x 16 k (thread: row tid / 4, k 4 (tid % 4) ..+3);
  // X tile 16 k x 64 cols (thread: k tid / 16, cols 4 (tid % 16) ..+3)
  const int ar = tid >> 2, ak = (tid & 3) * 4;
  const int bk = tid >> 4, bc = (tid & 15) * 4;
  for (int k0 = 0; k0 < d; k0 += 16) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int gi = i0 + ar, gk = k0 + ak + q;
      double v = 0.0;
      if (gi < d && gk < d) {
        v = (double)mi.F[(long long)gi * d + gk];
        if (gi == gk) v += (double)damp_of_row(mi, a1, a2, gi);
      }
      As[ak + q][ar] = v;
      const int gk2 = k0 + bk, gj = j0 + bc + q;
      Bs[bk][bc + q] =
          (gk2 < d && gj < d) ? (double)mi.inv[(long long)gk2 * d + gj] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = i0 + ty * 4 + i;
    if (gi >= d) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gj = j0 + tx * 4 + j;
      if (gj < d)
        mi.W[(long long)gi * mi.ld + gj] =
            (float)((gi == gj ? 1.0 : 0.0) - acc[i][j]);
    }
  }
}

// inv += Y for the refined matrices; blockIdx.y = item.
__global__ void __launch_bounds__(256)
refine_apply_kernel(const MatInfo* __restrict__ mats,
                    const RefineItem* __restrict__ items,
                    const int* gate) {
  wait_for_launch_before();
  if (gate[blockIdx.y] == 0) return;
  const RefineItem it = items[blockIdx.y];
  const MatInfo mi = mats[it.mat];
  for (int r = blockIdx.x; r < it.d; r += gridDim.x)
    for (int c = threadIdx.x; c < it.d; c += blockDim.x)
      mi.inv[(long long)r * it.d + c] += mi.V[(long long)r * mi.ld + c];
}

constexpr int kDiagControl = 512;
constexpr size_t kDiagSmemBytes =
    DB * DLD * sizeof(float) + 1024 + kDiagStage + kDiagControl;
constexpr size_t kDiagLookSmemBytes =
    DB * DLD * sizeof(float) + 1024 + kLookBytes + kDiagControl;
static_assert(kDiagLookSmemBytes >= kDiagSmemBytes &&
                  kDiagLookSmemBytes <= 227 * 1024 && sizeof(DiagControl) <= kDiagControl,
              "diagonal kernel shared memory");

// Streams of one run: the chain of diagonal kernels, panel solves and updates
// behind it, trailing updates nothing waits for soon, rows of L^-1, and the
// product of those rows.
enum PlanStream { S_CHAIN, S_BULK, S_FAR, S_ROWS, S_PROD, S_COUNT };

struct Launch {
  int tile_cols; // grouped gemm: tile width
  int kind;      // 0 diag kernel, 1 grouped gemm, 2 panel solve
  int off;       // grouped gemm: offset into descs
  int n;         // number of matrices / descs
  int tiles;     // grouped gemm: total tiles; panel solve: of the largest matrix
  int step;      // diag kernel, panel solve: index of the diagonal block
  int stream;    // PlanStream
  // events (indices into the plan's events, -1: none) to wait for first and to
  // record afterwards
  int wait_ev[3];
  int rec_ev;
  bool look;     // diag kernel: with the look-ahead prologue
  bool packed;   // grouped gemm: operands in fp16 chunks

  void wait(int ev) {
    if (ev < 0) return;
    for (int& w : wait_ev)
      if (w < 0) { w = ev; return; }
  }
};

// Status word of the diagonal kernel's bounded waits (read by kfac_tc_status).
int diag_status_read(int* out) {
  KFAC_CUDA(cudaMemcpyFromSymbol(out, g_diag_status, sizeof(int)));
  return KFAC_OK;
}

}  // namespace kfac

using namespace kfac;

struct kfac_inverse_plan {
  int count;
  int device;
  MatInfo* mats_dev;
  float* trace_dev;
  float* add_dev;
  float* scale_dev;        // diag and S of every matrix
  int* info_dev;
  MatInfo* sorted_dev;     // mats_dev, largest first (diagonal kernels)
  GemmDesc* descs_dev;
  std::vector<GemmDesc> descs;       // the same on the host
  std::vector<Launch> launches;
  bool use_tc;
  // refinement (see refine_* kernels)
  float* add2_dev;
  int n_refine;
  int refine_dmax;
  int dmax;                // largest side
  int refine_tiles;
  Launch refine_prod;
  RefineItem* refine_items_dev;
  double* refine_sums_dev;
  double* refine_vec_dev;
  int* refine_gate_dev;
  int* refine_count_dev;
  int refine_max_dim;
  float refine_threshold;
  // CUDA graph of one run (captured on first use)
  RunParams* params_dev;
  std::vector<cudaEvent_t> events;   // edges between the streams
  cudaEvent_t fork_ev, join_ev[S_COUNT];
  cudaStream_t side_stream[S_COUNT]; // streams of plain runs (from S_BULK on),
                                     // made by the first of them
  bool look;
  cudaGraphExec_t graph_exec;
  int* graph_info;
  float* graph_diag;
  long long graph_launches;
  int graph_early;                   // of them, those that begin early
  int run_early;                     // of the last run, -1: plain launches
  bool graph_ok;
};

// fp16 chunks of a matrix: tiles of 128 rows, 32 k a chunk.
static size_t chunk_tile_bytes(int d) {
  return (size_t)((d + DB - 1) / DB) * (DB / 32) * kChunk;
}
static size_t chunk_bytes(int d) {
  return (size_t)((d + DB - 1) / DB) * chunk_tile_bytes(d);
}

// (the matrices begin at a multiple of 256 bytes, wherever the workspace does)
extern "C" size_t kfac_inverse_workspace_bytes(int count, const int* dims) {
  if (count <= 0) return 0;
  size_t total = 255;
  for (int i = 0; i < count; ++i) {
    if (dims[i] <= 0) return 0;
    total += 3 * matrix_bytes(dims[i]) +             // W, X, V
             2 * chunk_bytes(dims[i]);               // L and X in chunks
  }
  return total;
}

extern "C" int kfac_inverse_plan_create(
    int count, const int* dims, const float* const* factors,
    float* const* inverses, const int* partner, const int* role,
    const float* l2_coef, const float* scale, void* workspace,
    size_t workspace_bytes, kfac_inverse_plan** out) {
  KFAC_REQUIRE(out != nullptr, "inverse_plan_create: null plan pointer");
  *out = nullptr;
  KFAC_REQUIRE(count > 0 && dims && factors && inverses && role,
               "inverse_plan_create: null argument or count=%d", count);
  for (int i = 0; i < count; ++i) {
    KFAC_REQUIRE(dims[i] > 0 && dims[i] <= 32768,
                 "inverse_plan_create: dims[%d]=%d out of range", i, dims[i]);
    KFAC_REQUIRE(factors[i] && inverses[i],
                 "inverse_plan_create: null matrix pointer at %d", i);
    KFAC_REQUIRE(role[i] >= 0 && role[i] <= 2,
                 "inverse_plan_create: role[%d]=%d", i, role[i]);
    if (role[i] != 2 && partner && partner[i] >= 0)
      KFAC_REQUIRE(partner[i] < count && role[partner[i]] == 1 - role[i],
                   "inverse_plan_create: partner[%d]=%d is not the other "
                   "factor of a pair", i, partner[i]);
  }
  size_t need = kfac_inverse_workspace_bytes(count, dims);
  if (workspace == nullptr || workspace_bytes < need)
    return fail(KFAC_ERR_WORKSPACE,
                "inverse_plan_create: workspace of %zu bytes needed, %zu given",
                need, workspace_bytes);

  // Blocks of X above the diagonal blocks are never written and are read as
  // zeros by the wide tiles of the triangular-inverse products.
  KFAC_CUDA(cudaMemset(workspace, 0, need));
  const bool use_tc = engine() == 1;
  // the tensor-core engine: operands in fp16 terms, in chunks where they are read
  // more than once
  const int half = use_tc ? G_HALF : 0;
  const int packed = use_tc ? G_PACKED : 0;
  std::vector<MatInfo> mats(count);
  char* ws = reinterpret_cast<char*>(
      (reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255);
  int dmax = 0;
  for (int i = 0; i < count; ++i) {
    MatInfo& m = mats[i];
    const size_t bytes = matrix_bytes(dims[i]);
    m.F = factors[i];
    m.inv = inverses[i];
    m.W = reinterpret_cast<float*>(ws); ws += bytes;
    m.V = reinterpret_cast<float*>(ws); ws += bytes;
    m.X = reinterpret_cast<float*>(ws); ws += bytes;
    m.d = dims[i];
    m.ld = matrix_pitch(dims[i]);
    m.partner = partner ? partner[i] : -1;
    m.role = role[i];
    m.l2 = l2_coef ? l2_coef[i] : 0.f;
    m.scale = scale ? scale[i] : 1.f;
    m.l2b = m.l2;
    m.id = i;
    if (half) {
      m.tile = chunk_tile_bytes(dims[i]);
      m.PX = reinterpret_cast<unsigned char*>(ws); ws += chunk_bytes(dims[i]);
      m.PL = reinterpret_cast<unsigned char*>(ws); ws += chunk_bytes(dims[i]);
    } else {
      m.tile = 0;
      m.PL = m.PX = nullptr;
    }
    dmax = std::max(dmax, dims[i]);
  }
  // diagonals and scales
  size_t n_scale = 0;
  for (const MatInfo& m : mats) n_scale += 2 * (size_t)m.ld;
  float* scale_dev = nullptr;
  cudaError_t e = cudaMalloc(&scale_dev, n_scale * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(scale_dev, 0, n_scale * sizeof(float));
  if (e != cudaSuccess) {
    cudaFree(scale_dev);
    return fail(KFAC_ERR_CUDA, "inverse_plan_create: %s", cudaGetErrorString(e));
  }
  {
    float* sc = scale_dev;
    for (MatInfo& m : mats) {
      m.diag = sc; sc += m.ld;
      m.S = sc; sc += m.ld;
    }
  }
  // large matrices first: their tiles are scheduled first
  std::vector<int> order(count);
  for (int i = 0; i < count; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return dims[a] > dims[b]; });

  std::vector<GemmDesc> descs;
  std::vector<Launch> launches;
  // operands in chunks: L from row r and column k on, X from row k and column m
  auto chunk_l = [](const MatInfo& m, long long r, long long k) {
    return m.PL + (r / DB) * m.tile + k / 32 * kChunk;
  };
  auto chunk_x = [](const MatInfo& m, long long k, long long c) {
    return m.PX + (c / DB) * m.tile + k / 32 * kChunk;
  };
  // products of rows ra and rb of L, from column k on
  auto set_l = [&](GemmDesc& g, const MatInfo& m, long long ra, long long rb,
                   long long k) {
    g.sa = g.sb = kScaleL;
    if (!packed) return;
    g.ca = chunk_l(m, ra, k);
    g.cb = chunk_l(m, rb, k);
    g.ca_tile = g.cb_tile = m.tile;
  };

  int n_events = 0;
  const bool look = packed && [] {
    const char* env = getenv("KFAC_INVERSE_LOOKAHEAD");
    return !(env && env[0] == '0');
  }();
  // without the look-ahead everything but the far updates follows the chain
  const int s_bulk = look ? S_BULK : S_CHAIN;
  const int s_rows = look ? S_ROWS : S_CHAIN;
  const int s_prod = look ? S_PROD : S_CHAIN;
  std::vector<int> diag_ev((dmax + DB - 1) / DB + 1, -1);
  std::vector<int> upd_ev((dmax + DB - 1) / DB + 1, -1);
  auto begin_gemm = [&](int stream) {
    Launch l = {};
    l.kind = 1;
    l.off = (int)descs.size();
    l.stream = stream;
    l.wait_ev[0] = l.wait_ev[1] = l.wait_ev[2] = l.rec_ev = -1;
    return l;
  };
  auto push_desc = [&](Launch& l, GemmDesc g) {
    g.tile_begin = l.tiles;
    if (!use_tc) l.tiles += gemm_desc_tiles(g);
    g.kfW = g.kfb = g.pW = g.pb = g.vW = g.vb = nullptr;
    g.dW = 0;
    g.splits = 1;
    g.ntiles = 0;
    g.k_per_split = 0;
    g.partial = nullptr;
    // (the scales of the fp16 terms come out again with alpha)
    if (g.flags & (G_HALF | G_PACKED)) g.alpha /= g.sa * g.sb;
    l.packed = (g.flags & G_PACKED) != 0;
    descs.push_back(g);
    l.n += 1;
  };
  // append a launch (if it has work); its event, or -1
  auto end_gemm = [&](Launch& l, bool record) {
    if (l.n == 0) return -1;
    if (use_tc && l.kind == 1)
      l.tiles = l.packed
                    ? packed_number_tiles(&descs[l.off], l.n)
                    : tc_number_tiles(&descs[l.off], l.n, 3 * sm_count() / 4,
                                      &l.tile_cols);
    if (record) l.rec_ev = n_events++;
    launches.push_back(l);
    return l.rec_ev;
  };

  // Width of the chain's panels.  Between two panels the chain waits for the
  // last solve and the near part of the trailing update, so matrices of up to
  // two panels are one where the longer panel updates of a step still fit the
  // SMs (5 x 1001 rows 274 us in two, 264 in one).  Where they do not (20 x 1024), or
  // the chain waits for its panel updates anyway (4608 rows), nothing is gained.
  long long step_tiles = 0;
  for (int i = 0; i < count; ++i)
    if (dims[i] > PW)
      step_tiles += (long long)((dims[i] - 1) / DB) * ((dims[i] - DB + 255) / 256);
  const int CW =
      look && dmax <= 2 * PW && step_tiles <= sm_count() ? 2 * PW : PW;

  int prev_far_ev = -1;
  // Two-level Cholesky: panels of CW columns are factored by 128-wide inner steps
  // whose updates stay inside the panel (or one block column more, see `ahead`;
  // short contractions, little work).  The other columns get a panel's share in two
  // parts: everything but the panel right before them while that one's chain
  // runs (far stream; a contraction over all panels so far, so that C is passed
  // over once and not once per panel), and that panel's share when its chain
  // ends (near).
  //
  // The chain carries the diagonal kernels; the diagonal kernel of step k applies
  // step k-1's update to its own block itself (diag_lookahead), so it only waits
  // for the panel update of step k-2.  The panel solves, panel updates and near
  // updates run on the bulk stream behind the chain.  A panel solve leaves W as it
  // is (the look-ahead reads it) and stores L as fp16 chunks, which is how every
  // product reads it.
  //
  // The inverse grows with the factor, a row panel at a time: with X = L^-1,
  //   T = L_p X_<p,  X_p = -X_pp T  (X_pp by doubling from the 128-blocks),
  //   inv += X_p^T X_p,
  // next to the chain of the following panels, which leaves most SMs idle.
  // When the chain ends only the last panel's share is left (a 4608-row matrix:
  // 0.15 ms instead of the 0.95 ms that the whole triangular inverse and
  // product took behind the factorisation).  T^T waits in the unused upper
  // triangle of W.
  int bulk_ev = -1;            // the bulk stream's last launch of this panel
  // Row panel po of the inverse, once the chain is through with it.
  auto row_panel = [&](int po) {
    const int pend = std::min(po + PW, dmax);
    bool first = true;
    for (int b = DB; b < pend - po; b *= 2) {
      // X_pp by doubling: T = L21 X11 (parked in V), then
      // X21 = -X22 T
      Launch g1 = begin_gemm(s_rows);
      std::vector<GemmDesc> second;
      for (int i : order) {
        const int d = dims[i], end = std::min(po + PW, d);
        const MatInfo& m = mats[i];
        const long long ld = m.ld;
        for (long long s = po; s + b < end; s += 2 * b) {
          const int r = (int)std::min<long long>(b, end - s - b);
          GemmDesc g = {};
          g.A = strided_operand(m.W + (s + b) * ld + s, 1, ld, r);
          g.B = strided_operand(m.X + s * ld + s, ld, 1, b);
          g.C = m.V + (s + b) * ld + s;
          g.ldc = ld; g.M = r; g.N = b; g.K = b;
          g.alpha = 1.f; g.beta = 0.f; g.flags = G_KBEG_N0 | packed;
          g.sa = kScaleL; g.sb = kScaleX;
          if (packed) {
            g.ca = chunk_l(m, s + b, s);
            g.cb = chunk_x(m, s, s);
            g.ca_tile = g.cb_tile = m.tile;
          }
          push_desc(g1, g);
          GemmDesc h = {};
          h.A = strided_operand(m.X + (s + b) * ld + s + b, 1, ld, r);
          h.B = strided_operand(m.V + (s + b) * ld + s, ld, 1, b);
          h.C = m.X + (s + b) * ld + s;
          h.ldc = ld; h.M = r; h.N = b; h.K = r;
          h.alpha = -1.f; h.beta = 0.f; h.flags = G_KEND_M0 | half;
          h.sa = kScaleX; h.sb = kScaleT;
          if (packed) {
            h.pack = chunk_x(m, s + b, s); h.pack_tile = m.tile;
            h.pack_scale = kScaleX;
          }
          second.push_back(h);
        }
      }
      if (first) {
        g1.wait(bulk_ev);
        g1.wait(diag_ev[(pend - 1) / DB]);
        if (g1.n > 0) first = false;
      }
      end_gemm(g1, false);
      Launch g2 = begin_gemm(s_rows);
      for (auto& h : second) push_desc(g2, h);
      end_gemm(g2, false);
    }
    Launch rows = begin_gemm(s_rows), next_t = begin_gemm(s_rows);
    if (po > 0) {
      for (int i : order) {
        const int d = dims[i], w = std::min(PW, d - po);
        if (w <= 0) continue;
        const MatInfo& m = mats[i];
        const long long ld = m.ld;
        GemmDesc g = {};
        g.A = strided_operand(m.X + po * ld + po, 1, ld, w);
        g.B = strided_operand(m.W + po, 1, ld, po);   // B(k, n) = T^T[n][k]
        g.C = m.X + po * ld;
        g.ldc = ld; g.M = w; g.N = po; g.K = w;
        g.alpha = -1.f; g.beta = 0.f; g.flags = G_KEND_M0 | half;
        g.sa = kScaleX; g.sb = kScaleT;
        if (packed) {              // nothing reads these rows but as chunks
          g.C = nullptr;
          g.pack = chunk_x(m, po, 0); g.pack_tile = m.tile;
          g.pack_scale = kScaleX;
        }
        push_desc(rows, g);
      }
    }
    if (first) {
      rows.wait(bulk_ev);
      rows.wait(diag_ev[(pend - 1) / DB]);
      if (rows.n > 0) first = false;
    }
    int rows_ev = end_gemm(rows, look);
    // the product, behind the rows (or, for a single panel, the doubling)
    Launch prod = begin_gemm(s_prod);
    for (int i : order) {
      const int d = dims[i], end = std::min(po + PW, d);
      if (end <= po) continue;
      // two panels at a time (half as many passes over inv), but for the last
      // one, which the end of the run waits for
      const bool odd = (po / PW) & 1, last = end == d;
      if (!odd && !last && po + 2 * PW < d) continue;
      const int ks = odd && !last ? po - PW : po;
      const MatInfo& m = mats[i];
      GemmDesc g = {};
      g.A = strided_operand(m.X + (long long)ks * m.ld, m.ld, 1, end);
      g.B = g.A;
      g.C = m.inv; g.ldc = d; g.M = end; g.N = end; g.K = end - ks;
      g.alpha = 1.f; g.beta = ks > 0 ? 1.f : 0.f;
      g.beta_until = ks; g.kbeg_off = ks;
      g.flags = G_LOWER | G_KBEG_M0 | G_SAME_AB | (last ? G_MIRROR : 0) | packed;
      g.sa = g.sb = kScaleX;
      if (packed) {
        g.ca = g.cb = chunk_x(m, ks, 0);
        g.ca_tile = g.cb_tile = m.tile;
      }
      g.unscale = m.S;
      push_desc(prod, g);
    }
    if (look && rows_ev < 0 && !first) {
      rows_ev = n_events++;
      launches.back().rec_ev = rows_ev;      // the doubling's last launch
    }
    if (look && first) {
      prod.wait(bulk_ev);
      prod.wait(diag_ev[(pend - 1) / DB]);
    }
    prod.wait(rows_ev);
    // T^T of the next panel
    next_t.off = (int)descs.size();
    for (int i : order) {
      const int d = dims[i], w = std::min(PW, d - pend);
      if (w <= 0) continue;
      const MatInfo& m = mats[i];
      const long long ld = m.ld;
      GemmDesc g = {};
      g.A = strided_operand(m.X, ld, 1, pend);
      g.B = strided_operand(m.W + pend * ld, 1, ld, w);
      g.C = m.W + pend;
      g.ldc = ld; g.M = pend; g.N = w; g.K = pend;
      g.alpha = 1.f; g.beta = 0.f; g.flags = G_KBEG_M0 | packed;
      g.sa = kScaleX; g.sb = kScaleL;
      if (packed) {
        g.ca = chunk_x(m, 0, 0);
        g.cb = chunk_l(m, pend, 0);
        g.ca_tile = g.cb_tile = m.tile;
      }
      push_desc(next_t, g);
    }
    if (look && first) next_t.wait(bulk_ev);
    end_gemm(next_t, false);
    end_gemm(prod, false);
  };
  // Whether a panel's steps also update the next one's first block column.  The
  // chain then goes on there without waiting for the near update, which only
  // the second block needs.  It pays for matrices of two panels, where the one near
  // update between them is a good part of the chain (16 x 1024 rows 378 us without,
  // 368 with); longer ones wait for their panel updates anyway, which the further
  // column makes longer (2 x 4608 rows 1381 without, 1414 with).  Nor in plans of more
  // row tiles than SMs: beside others, which such plans run, the passes over that
  // column only cost.
  long long row_tiles = 0;
  for (int i = 0; i < count; ++i) row_tiles += (dims[i] + DB - 1) / DB;
  const bool ahead = look && dmax <= 2 * PW && row_tiles <= sm_count();
  const int E = ahead ? DB : 0;
  // Update of the window of columns from s on with columns k .. k + K of L.
  auto window = [&](const MatInfo& m, int d, int s, int k, int K,
                    std::vector<GemmDesc>& out) {
    const int M = d - s, N = std::min(CW, M);
    if (M <= 0) return;
    const long long ld = m.ld;
    const float* rows = m.W + s * ld + k;
    GemmDesc g = {};     // square block on the diagonal: lower tiles
    g.A = strided_operand(rows, 1, ld, N);
    g.B = g.A;
    g.C = m.W + s * ld + s;
    g.ldc = ld; g.M = N; g.N = N; g.K = K;
    g.alpha = -1.f; g.beta = 1.f; g.flags = G_LOWER | G_SAME_AB | packed;
    set_l(g, m, s, s, k);
    out.push_back(g);
    if (M == N) return;
    GemmDesc h = {};     // rectangle below it
    h.A = strided_operand(rows + N * ld, 1, ld, M - N);
    h.B = strided_operand(rows, 1, ld, N);
    h.C = m.W + (long long)(s + N) * ld + s;
    h.ldc = ld; h.M = M - N; h.N = N; h.K = K;
    h.alpha = -1.f; h.beta = 1.f; h.flags = packed;
    set_l(h, m, s + N, s, k);
    out.push_back(h);
  };
  // Whether the near update takes the columns of the panel's last block by
  // themselves, so that the others' part runs beside the last diagonal kernel and
  // the chain waits for 128 k instead of 512.  It costs another pass over the window,
  // behind the far update of the panel before: not where plans fill the SMs (the
  // three of ResNet-50 4092 us without, 4141 with), nor where that update takes as
  // long as a panel, which goes by the squares of the sides: between 6000 rows (2209
  // squares of tiles: 1716 us without, 1685 with) and 2 x 4608 (2592: 1364, 1376).
  long long squares = 0;
  for (int i = 0; i < count; ++i) {
    const long long t = (dims[i] + DB - 1) / DB;
    squares += t * t;
  }
  const bool split_near =
      look && row_tiles <= sm_count() && squares <= 16 * sm_count();
  int near_ev = -1;            // near updates of the panel before
  for (int co = 0; co < dmax; co += CW) {
    const int inner = std::min(CW, dmax - co);
    bulk_ev = -1;
    int last_solve_ev = -1;
    for (int o = co; o < co + inner; o += DB) {
      const bool lk = look && (ahead ? o > 0 : o > co);
      // the matrices that still have a block here are the first of `order`
      Launch dl = begin_gemm(S_CHAIN);
      dl.kind = 0;
      dl.step = o / DB;
      dl.look = lk;
      for (int i : order)
        if (dims[i] > o) dl.n += 1;
      if (lk && o >= 2 * DB && (ahead || o - 2 * DB >= co))
        dl.wait(upd_ev[o / DB - 2]);
      // (without look-ahead all of this is one stream)
      if (look && o == (ahead ? co + DB : co)) dl.wait(near_ev);
      diag_ev[o / DB] = end_gemm(dl, look);

      Launch trsm = begin_gemm(s_bulk);
      if (packed) {
        trsm.kind = 2;
        trsm.step = o / DB;
      }
      for (int i : order) {
        const int d = dims[i];
        const int M = d - o - DB;
        if (M <= 0) continue;
        const MatInfo& m = mats[i];
        const long long ld = m.ld;
        if (packed) {              // (the largest matrix comes first)
          if (trsm.n++ == 0) trsm.tiles = (M + DB - 1) / DB;
          continue;
        }
        GemmDesc g = {};
        float* panel = m.W + (o + DB) * ld + o;
        g.A = strided_operand(panel, 1, ld, M);
        g.B = strided_operand(m.X + o * ld + o, 1, ld, DB);
        g.C = panel; g.ldc = ld; g.M = M; g.N = DB; g.K = DB;
        g.alpha = 1.f; g.beta = 0.f; g.flags = 0;
        push_desc(trsm, g);
      }
      trsm.wait(diag_ev[o / DB]);
      const int solve_ev = end_gemm(trsm, look);
      if (solve_ev >= 0) bulk_ev = last_solve_ev = solve_ev;

      // update the rest of this panel's columns, with `ahead` the block column
      // after them too (full rectangle; entries above the diagonal are written
      // but never read).  With look-ahead the next diagonal block is left to the next
      // diagonal kernel.
      const int skip = look && (ahead || o + DB < co + inner) ? DB : 0;
      Launch upd = begin_gemm(s_bulk);
      for (int i : order) {
        const int d = dims[i];
        const int M = d - o - DB - skip;
        const int N = std::min(co + CW + E, d) - (o + DB);
        if (M <= 0 || N <= 0) continue;
        const MatInfo& m = mats[i];
        const long long ld = m.ld;
        GemmDesc g = {};
        float* panel = m.W + (o + DB + skip) * ld + o;
        const long long coff = (o + DB + skip) * ld + (o + DB);
        g.A = strided_operand(panel, 1, ld, M);
        g.B = strided_operand(m.W + (o + DB) * ld + o, 1, ld, N);
        g.C = m.W + coff;
        g.ldc = ld; g.M = M; g.N = N; g.K = DB;
        g.alpha = -1.f; g.beta = 1.f; g.flags = packed;
        set_l(g, m, o + DB + skip, o + DB, o);
        push_desc(upd, g);
      }
      upd_ev[o / DB] = end_gemm(upd, look);
      if (upd_ev[o / DB] >= 0) bulk_ev = upd_ev[o / DB];
      if (split_near && inner > DB && o + 2 * DB == co + inner) {
        std::vector<GemmDesc> pre_descs;
        for (int i : order)
          window(mats[i], dims[i], co + CW + E, co, inner - DB, pre_descs);
        Launch pre = begin_gemm(S_FAR);
        for (auto& g : pre_descs) push_desc(pre, g);
        pre.wait(solve_ev);      // (and, on this stream, the far update before)
        if (pre.n > 0) prev_far_ev = end_gemm(pre, true);
      }
      // (the last rows of a chain panel come behind its trailing update)
      if ((o + DB) % PW == 0 && o + DB < co + inner) row_panel(o + DB - PW);
    }

    // Updates behind the finished panel, for windows of columns that begin with a
    // panel (`ahead`: one block later): the next window with this panel, the window
    // after it with all panels so far, next to the next panel's chain.  What touches
    // the same tiles is ordered by events (near of a panel after far of the one
    // before).
    Launch near = begin_gemm(s_bulk);
    std::vector<GemmDesc> far_descs;
    std::vector<GemmDesc> near_descs;
    for (int i : order) {
      const int done = split_near ? inner - DB : 0;
      window(mats[i], dims[i], co + CW + E, co + done, CW - done, near_descs);
      window(mats[i], dims[i], co + 2 * CW + E, 0, co + CW, far_descs);
    }
    for (auto& g : near_descs) push_desc(near, g);
    int panel_ev = last_solve_ev;
    if (!look && !far_descs.empty()) {
      // the far part needs the finished panel: an event recorded on the
      // chain right before the near part
      panel_ev = n_events++;
      launches.back().rec_ev = panel_ev;   // last launch of the panel's chain
    }
    near.wait(prev_far_ev);                // far part of the previous panel
    if (near.n > 0) prev_far_ev = -1;
    near_ev = end_gemm(near, look);
    Launch far = begin_gemm(S_FAR);
    for (auto& h : far_descs) push_desc(far, h);
    far.wait(panel_ev);
    if (far.n > 0) prev_far_ev = end_gemm(far, true);
    row_panel((std::min(co + inner, dmax) - 1) / PW * PW);
  }

  // refinement of the matrices of up to kRefineDimCap rows: Y = X R on the
  // tile engine (Y is symmetric: lower tiles, mirrored), gated per matrix
  std::vector<RefineItem> ritems;
  int refine_tiles = 0, refine_dmax = 0;
  long long vec_elems = 0;
  for (int i : order) {
    if (dims[i] > kRefineDimCap) continue;
    RefineItem it;
    it.mat = i;
    it.d = dims[i];
    it.tile_begin = refine_tiles;
    it.pad_ = 0;
    it.vec = reinterpret_cast<double*>(vec_elems);   // offset, fixed up below
    const int nt = (dims[i] + 63) / 64;
    refine_tiles += nt * nt;
    refine_dmax = std::max(refine_dmax, dims[i]);
    vec_elems += 2LL * dims[i];
    ritems.push_back(it);
  }
  Launch refine_prod = begin_gemm(S_CHAIN);

  kfac_inverse_plan* p = new kfac_inverse_plan();
  p->count = count;
  p->launches = launches;
  p->use_tc = use_tc;
  p->mats_dev = nullptr; p->trace_dev = nullptr; p->add_dev = nullptr;
  p->info_dev = nullptr; p->sorted_dev = nullptr; p->descs_dev = nullptr;
  p->add2_dev = nullptr; p->refine_items_dev = nullptr;
  p->refine_sums_dev = nullptr; p->refine_vec_dev = nullptr;
  p->refine_gate_dev = nullptr; p->refine_count_dev = nullptr;
  p->n_refine = (int)ritems.size();
  p->refine_dmax = refine_dmax;
  p->dmax = dmax;
  p->refine_tiles = refine_tiles;
  p->refine_max_dim = kRefineDimCap;
  p->refine_threshold = 3e-5f;
  p->params_dev = nullptr;
  p->fork_ev = nullptr;
  for (int k = 1; k < S_COUNT; ++k)
    p->join_ev[k] = nullptr, p->side_stream[k] = nullptr;
  p->look = look;
  p->graph_exec = nullptr;
  p->graph_info = nullptr;
  p->graph_diag = nullptr;
  p->graph_launches = 0;
  p->graph_early = 0;
  p->run_early = -1;
  {
    const char* env = getenv("KFAC_INVERSE_GRAPH");
    p->graph_ok = !(env && env[0] == '0');
  }
  p->scale_dev = scale_dev;
  e = cudaGetDevice(&p->device);
  if (e == cudaSuccess) e = cudaMalloc(&p->params_dev, sizeof(RunParams));
  if (e == cudaSuccess)
    e = cudaEventCreateWithFlags(&p->fork_ev, cudaEventDisableTiming);
  for (int k = 1; k < S_COUNT && e == cudaSuccess; ++k)
    e = cudaEventCreateWithFlags(&p->join_ev[k], cudaEventDisableTiming);
  for (int k = 0; k < n_events + 1 && e == cudaSuccess; ++k) {
    cudaEvent_t ev = nullptr;
    e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) p->events.push_back(ev);
  }
  if (e == cudaSuccess) e = cudaMalloc(&p->add2_dev, sizeof(float) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->refine_count_dev, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(p->refine_count_dev, 0, sizeof(int));
  if (e == cudaSuccess && !ritems.empty()) {
    const size_t nr = ritems.size();
    e = cudaMalloc(&p->refine_items_dev, sizeof(RefineItem) * nr);
    if (e == cudaSuccess) e = cudaMalloc(&p->refine_sums_dev, sizeof(double) * 2 * nr);
    if (e == cudaSuccess) e = cudaMalloc(&p->refine_vec_dev, sizeof(double) * vec_elems);
    if (e == cudaSuccess) e = cudaMalloc(&p->refine_gate_dev, sizeof(int) * nr);
    if (e == cudaSuccess) {
      for (size_t r = 0; r < nr; ++r) {
        RefineItem& it = ritems[r];
        it.vec = p->refine_vec_dev + reinterpret_cast<long long>(it.vec);
        const int d = it.d;
        const MatInfo& m = mats[it.mat];
        GemmDesc g = {};
        g.A = strided_operand(m.inv, 1, d, d);     // A(k, m) = X[m][k]
        g.B = strided_operand(m.W, m.ld, 1, d);    // B(k, n) = R[k][n]
        g.C = m.V; g.ldc = m.ld; g.M = d; g.N = d; g.K = d;
        g.alpha = 1.f; g.beta = 0.f; g.flags = G_LOWER | G_MIRROR;
        g.gate = p->refine_gate_dev + r;
        push_desc(refine_prod, g);
      }
      e = cudaMemcpy(p->refine_items_dev, ritems.data(),
                     sizeof(RefineItem) * nr, cudaMemcpyHostToDevice);
    }
  }
  if (use_tc && refine_prod.n > 0)
    refine_prod.tiles = tc_number_tiles(&descs[refine_prod.off], refine_prod.n,
                                        sm_count(),
                                        &refine_prod.tile_cols);
  p->refine_prod = refine_prod;
  p->descs = descs;
  if (e == cudaSuccess) e = cudaMalloc(&p->mats_dev, sizeof(MatInfo) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->trace_dev, sizeof(float) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->add_dev, sizeof(float) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->info_dev, sizeof(int) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->sorted_dev, sizeof(MatInfo) * count);
  if (e == cudaSuccess) e = cudaMalloc(&p->descs_dev, sizeof(GemmDesc) * std::max<size_t>(descs.size(), 1));
  if (e == cudaSuccess) e = cudaMemcpy(p->mats_dev, mats.data(), sizeof(MatInfo) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    std::vector<MatInfo> sorted(count);
    for (int i = 0; i < count; ++i) sorted[i] = mats[order[i]];
    e = cudaMemcpy(p->sorted_dev, sorted.data(), sizeof(MatInfo) * count,
                   cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess && !descs.empty()) e = cudaMemcpy(p->descs_dev, descs.data(), sizeof(GemmDesc) * descs.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(chol_diag_kernel<false>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kDiagSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(chol_diag_kernel<true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kDiagLookSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(panel_solve_kernel,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSolveSmemBytes);
  if (e != cudaSuccess) {
    kfac_inverse_plan_destroy(p);
    return fail(KFAC_ERR_CUDA, "inverse_plan_create: %s", cudaGetErrorString(e));
  }
  if (use_tc) {
    int rc = tc_prepare_tiles();
    if (rc == KFAC_OK) rc = packed_prepare();
    if (rc != KFAC_OK) {
      kfac_inverse_plan_destroy(p);
      return rc;
    }
  }
  *out = p;
  return KFAC_OK;
}

// The kernel that the next launch on a capturing stream follows, if it follows
// nothing else.
static cudaGraphNode_t captured_kernel(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  cudaGraphNodeType type = cudaGraphNodeTypeEmpty;
  size_t n = 0;
  if (cudaStreamGetCaptureInfo_v3(st, &cs, nullptr, nullptr, &deps, &edges, &n) !=
          cudaSuccess ||
      n != 1 || cudaGraphNodeGetType(deps[0], &type) != cudaSuccess ||
      type != cudaGraphNodeTypeKernel) {
    cudaGetLastError();
    return nullptr;
  }
  return deps[0];
}

// The next launch on a capturing stream may begin before `node` has ended
// (programmatic dependency: it waits for the rest of it itself), but not before
// anything else that it follows.  `count` goes up if it does.
static cudaError_t begin_before_end_of(cudaStream_t st, cudaGraphNode_t node,
                                       int* count) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n = 0;
  cudaError_t e = cudaStreamGetCaptureInfo_v3(st, &cs, nullptr, nullptr, &deps,
                                              &edges, &n);
  if (e != cudaSuccess) return e;
  std::vector<cudaGraphNode_t> nodes(deps, deps + n);
  std::vector<cudaGraphEdgeData> data(n);
  for (size_t i = 0; i < n; ++i) {
    if (edges != nullptr) data[i] = edges[i];
    if (nodes[i] == node) {
      data[i].from_port = cudaGraphKernelNodePortProgrammatic;
      data[i].type = cudaGraphDependencyTypeProgrammatic;
    }
  }
  e = cudaStreamUpdateCaptureDependencies_v2(
      st, nodes.data(), data.data(), n, cudaStreamSetCaptureDependencies);
  if (e == cudaSuccess)
    *count += (int)std::count(nodes.begin(), nodes.end(), node);
  return e;
}

// Issue every launch of one run into `st` (a real stream, or one that is
// being captured into a graph, `graph`: this plan's own).
static int plan_enqueue(kfac_inverse_plan* p, int* info, float* diag_dev,
                        cudaStream_t main_st, cudaStream_t* side_st, bool graph) {
  cudaStream_t st = main_st;
  cudaStream_t sts[S_COUNT] = {main_st};
  // fork: the side streams start after what precedes this run
  KFAC_CUDA(cudaEventRecord(p->fork_ev, main_st));
  for (int k = 1; k < S_COUNT; ++k) {
    sts[k] = side_st[k];
    KFAC_CUDA(cudaStreamWaitEvent(sts[k], p->fork_ev, 0));
  }
  // A launch that follows one kernel only may begin before that has ended.  (The
  // other engine's kernels do not wait for it themselves.)
  graph = graph && p->use_tc;
  auto early = [&](bool when) -> cudaError_t {
    const cudaGraphNode_t before = graph && when ? captured_kernel(st) : nullptr;
    return before != nullptr ? begin_before_end_of(st, before, &p->graph_early)
                             : cudaSuccess;
  };
  trace_kernel<<<p->count, kTraceThreads, 0, st>>>(p->mats_dev, p->trace_dev, info);
  KFAC_LAUNCH_CHECK("trace_kernel");
  KFAC_CUDA(early(true));
  {
    const dim3 grid(std::min(1024, ceil_div(p->dmax, kDampRows)), p->count);
    damp_copy_kernel<<<grid, 256, 0, st>>>(
        p->mats_dev, p->trace_dev, p->params_dev, p->add_dev, p->add2_dev,
        diag_dev, p->use_tc ? 1 : 0);
    KFAC_LAUNCH_CHECK("damp_copy_kernel");
  }
  cudaGraphNode_t last_diag = nullptr;
  for (const Launch& l : p->launches) {
    st = sts[l.stream];
    for (int ev : l.wait_ev)
      if (ev >= 0) KFAC_CUDA(cudaStreamWaitEvent(st, p->events[ev], 0));
    if (l.kind == 0) {
      // What it reads before the wait comes from launches that it follows wholly, or
      // that the diagonal kernel before it has followed wholly: one without the
      // look-ahead does not begin early itself.  (A layer of 334 x 53, three
      // diagonal blocks in a row: 222.6 us, 217.7 so; one of 4608 x 512 1304, 1294.)
      if (l.look && last_diag != nullptr)
        KFAC_CUDA(begin_before_end_of(st, last_diag, &p->graph_early));
      if (!p->use_tc)
        chol_diag_ffma_kernel<<<l.n, DT, 0, st>>>(p->sorted_dev, l.step, info);
      else if (l.look)
        chol_diag_kernel<true><<<l.n, DT, kDiagLookSmemBytes, st>>>(
            p->sorted_dev, l.step, info);
      else
        chol_diag_kernel<false><<<l.n, DT, kDiagSmemBytes, st>>>(
            p->sorted_dev, l.step, info);
      KFAC_LAUNCH_CHECK("chol_diag_kernel");
      if (graph) last_diag = captured_kernel(st);
    } else if (l.kind == 2) {
      if (last_diag != nullptr)
        KFAC_CUDA(begin_before_end_of(st, last_diag, &p->graph_early));
      panel_solve_kernel<<<dim3(l.tiles, l.n), kSolveThreads, kSolveSmemBytes,
                           st>>>(p->sorted_dev, l.step);
      KFAC_LAUNCH_CHECK("panel_solve_kernel");
    } else {
      // (more tiles than SMs: the next launch's waiting CTAs only take room; 54 pairs
      // of ResNet-50 3993 us so, 4083 without a limit)
      KFAC_CUDA(early(l.tiles <= sm_count()));
      int rc = l.packed
                   ? launch_packed(p->descs_dev + l.off, &p->descs[l.off], l.n,
                                   l.tiles, st)
               : p->use_tc
                   ? launch_tc_grouped(p->descs_dev + l.off, &p->descs[l.off],
                                       l.n, l.tiles, l.tile_cols, false, 0.f,
                                       0.f, st)
                   : launch_grouped_gemm(p->descs_dev + l.off, l.n, l.tiles,
                                         0.f, 0.f, st);
      if (rc != KFAC_OK) return rc;
    }
    if (l.rec_ev >= 0) KFAC_CUDA(cudaEventRecord(p->events[l.rec_ev], st));
  }
  st = main_st;
  for (int k = 1; k < S_COUNT; ++k) {
    KFAC_CUDA(cudaEventRecord(p->join_ev[k], sts[k]));
    KFAC_CUDA(cudaStreamWaitEvent(main_st, p->join_ev[k], 0));
  }
  if (p->n_refine > 0) {
    const dim3 pgrid(ceil_div(p->refine_dmax, 8), p->n_refine);
    for (int stage = 0; stage < 3; ++stage) {
      KFAC_CUDA(early(true));
      refine_probe_kernel<<<pgrid, 256, 0, st>>>(
          p->mats_dev, p->refine_items_dev, p->add_dev, p->add2_dev,
          p->refine_sums_dev, p->params_dev, stage);
      KFAC_LAUNCH_CHECK("refine_probe_kernel");
    }
    KFAC_CUDA(early(true));
    refine_gate_kernel<<<1, kGateThreads, 0, st>>>(
        p->refine_items_dev, p->n_refine, p->refine_sums_dev, p->params_dev,
        p->refine_gate_dev, p->refine_count_dev);
    KFAC_LAUNCH_CHECK("refine_gate_kernel");
    KFAC_CUDA(early(true));
    refine_residual_kernel<<<p->refine_tiles, 256, 0, st>>>(
        p->mats_dev, p->refine_items_dev, p->n_refine, p->add_dev,
        p->add2_dev, p->refine_gate_dev);
    KFAC_LAUNCH_CHECK("refine_residual_kernel");
    KFAC_CUDA(early(true));
    const Launch& l = p->refine_prod;
    int rc = p->use_tc
                 ? launch_tc_grouped(p->descs_dev + l.off, &p->descs[l.off],
                                     l.n, l.tiles, l.tile_cols, false, 0.f,
                                       0.f, st)
                 : launch_grouped_gemm(p->descs_dev + l.off, l.n, l.tiles, 0.f,
                                       0.f, st);
    if (rc != KFAC_OK) return rc;
    KFAC_CUDA(early(true));
    const dim3 agrid(64, p->n_refine);
    refine_apply_kernel<<<agrid, 256, 0, st>>>(p->mats_dev, p->refine_items_dev,
                                               p->refine_gate_dev);
    KFAC_LAUNCH_CHECK("refine_apply_kernel");
  }
  return KFAC_OK;
}

static void plan_drop_graph(kfac_inverse_plan* p) {
  if (p->graph_exec != nullptr) cudaGraphExecDestroy(p->graph_exec);
  p->graph_exec = nullptr;
}

// Side streams of a run, behind its chain.
static cudaError_t make_side_streams(cudaStream_t* side) {
  int lo = 0, hi = 0;
  cudaError_t e = cudaDeviceGetStreamPriorityRange(&lo, &hi);
  for (int k = 1; k < S_COUNT && e == cudaSuccess; ++k)
    if (side[k] == nullptr)
      e = cudaStreamCreateWithPriority(&side[k], cudaStreamNonBlocking, lo);
  return e;
}

// Streams that plans are captured on, one set per device: nothing executes
// during a capture, the graph only keeps their priorities.
struct CaptureStreams {
  std::mutex mu;                     // held from the first launch to the last
  cudaStream_t chain = nullptr;
  cudaStream_t side[S_COUNT] = {};
};

// Capture one run into a graph.  On any failure the plan falls back to plain
// launches.
static void plan_capture(kfac_inverse_plan* p, int* info, float* diag_dev) {
  static CaptureStreams sets[64];
  plan_drop_graph(p);
  CaptureStreams& c = sets[p->device & 63];
  std::lock_guard<std::mutex> lock(c.mu);
  // the chain is latency-bound and uses few SMs: it gets the higher
  // priority, the side streams' tiles fill the rest
  int lo = 0, hi = 0;
  cudaError_t made = cudaDeviceGetStreamPriorityRange(&lo, &hi);
  if (made == cudaSuccess && c.chain == nullptr)
    made = cudaStreamCreateWithPriority(&c.chain, cudaStreamNonBlocking, hi);
  if (made == cudaSuccess) made = make_side_streams(c.side);
  const long long before = launch_count_now();
  if (made != cudaSuccess ||
      cudaStreamBeginCapture(c.chain, cudaStreamCaptureModeRelaxed) !=
          cudaSuccess) {
    cudaGetLastError();
    p->graph_ok = false;
    return;
  }
  p->graph_early = 0;
  const int rc = plan_enqueue(p, info, diag_dev, c.chain, c.side, true);
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamEndCapture(c.chain, &graph);
  const long long captured = launch_count_now() - before;
  count_launches(-captured);          // nothing ran yet
  if (rc == KFAC_OK && e == cudaSuccess && graph != nullptr)
    e = cudaGraphInstantiate(&p->graph_exec, graph, 0);
  if (graph != nullptr) cudaGraphDestroy(graph);
  if (rc != KFAC_OK || e != cudaSuccess || p->graph_exec == nullptr) {
    cudaGetLastError();
    plan_drop_graph(p);
    p->graph_ok = false;
    return;
  }
  p->graph_info = info;
  p->graph_diag = diag_dev;
  p->graph_launches = captured;
}

extern "C" int kfac_inverse_plan_run(kfac_inverse_plan* p, float damping,
                                     int use_pi, int* info_dev,
                                     float* diag_dev, void* stream) {
  KFAC_REQUIRE(p != nullptr, "inverse_plan_run: null plan");
  cudaStream_t st = (cudaStream_t)stream;
  int* info = info_dev ? info_dev : p->info_dev;
  set_run_params_kernel<<<1, 1, 0, st>>>(p->params_dev, damping, use_pi,
                                         p->refine_max_dim,
                                         p->refine_threshold);
  KFAC_LAUNCH_CHECK("set_run_params_kernel");
  if (p->graph_ok) {
    // a caller that is itself capturing gets plain launches in its capture
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
      cudaGetLastError();
      cs = cudaStreamCaptureStatusNone;
    }
    if (cs == cudaStreamCaptureStatusNone) {
      if (p->graph_exec == nullptr || p->graph_info != info ||
          p->graph_diag != diag_dev)
        plan_capture(p, info, diag_dev);
      if (p->graph_exec != nullptr) {
        KFAC_CUDA(cudaGraphLaunch(p->graph_exec, st));
        count_launches(p->graph_launches);
        p->run_early = p->graph_early;
        return KFAC_OK;
      }
    }
  }
  p->run_early = -1;
  KFAC_CUDA(make_side_streams(p->side_stream));
  return plan_enqueue(p, info, diag_dev, st, p->side_stream, false);
}

extern "C" int kfac_inverse_plan_set_refine(kfac_inverse_plan* p, int max_dim,
                                            float threshold) {
  KFAC_REQUIRE(p != nullptr, "inverse_plan_set_refine: null plan");
  KFAC_REQUIRE(max_dim >= 0 && threshold >= 0.f,
               "inverse_plan_set_refine: max_dim=%d threshold=%g", max_dim,
               (double)threshold);
  p->refine_max_dim = max_dim < kRefineDimCap ? max_dim : kRefineDimCap;
  p->refine_threshold = threshold;
  return KFAC_OK;
}

extern "C" int kfac_inverse_plan_early_launches(kfac_inverse_plan* p,
                                                int* early_out) {
  KFAC_REQUIRE(p != nullptr && early_out != nullptr,
               "inverse_plan_early_launches: null argument");
  *early_out = p->run_early;
  return KFAC_OK;
}

extern "C" int kfac_inverse_plan_refined(kfac_inverse_plan* p,
                                         int* refined_out) {
  KFAC_REQUIRE(p != nullptr && refined_out != nullptr,
               "inverse_plan_refined: null argument");
  KFAC_CUDA(cudaDeviceSynchronize());
  KFAC_CUDA(cudaMemcpy(refined_out, p->refine_count_dev, sizeof(int),
                       cudaMemcpyDeviceToHost));
  return KFAC_OK;
}

extern "C" int kfac_inverse_plan_error_estimates(kfac_inverse_plan* p,
                                                 float* estimates_out) {
  KFAC_REQUIRE(p != nullptr && estimates_out != nullptr,
               "inverse_plan_error_estimates: null argument");
  for (int i = 0; i < p->count; ++i) estimates_out[i] = -1.f;
  if (p->n_refine == 0) return KFAC_OK;
  std::vector<RefineItem> items(p->n_refine);
  std::vector<double> sums(2 * (size_t)p->n_refine);
  KFAC_CUDA(cudaDeviceSynchronize());
  KFAC_CUDA(cudaMemcpy(items.data(), p->refine_items_dev,
                       sizeof(RefineItem) * p->n_refine,
                       cudaMemcpyDeviceToHost));
  KFAC_CUDA(cudaMemcpy(sums.data(), p->refine_sums_dev,
                       sizeof(double) * 2 * p->n_refine,
                       cudaMemcpyDeviceToHost));
  for (int r = 0; r < p->n_refine; ++r)
    estimates_out[items[r].mat] =
        sums[2 * r + 1] > 0.0 ? (float)sqrt(sums[2 * r] / sums[2 * r + 1])
                              : -1.f;
  return KFAC_OK;
}

extern "C" int kfac_inverse_plan_set_second_floor(kfac_inverse_plan* p,
                                                  const float* l2_coef_second) {
  KFAC_REQUIRE(p != nullptr && l2_coef_second != nullptr,
               "inverse_plan_set_second_floor: null argument");
  std::vector<MatInfo> mats(p->count);
  KFAC_CUDA(cudaDeviceSynchronize());
  KFAC_CUDA(cudaMemcpy(mats.data(), p->mats_dev, sizeof(MatInfo) * p->count,
                       cudaMemcpyDeviceToHost));
  for (int i = 0; i < p->count; ++i) mats[i].l2b = l2_coef_second[i];
  KFAC_CUDA(cudaMemcpy(p->mats_dev, mats.data(), sizeof(MatInfo) * p->count,
                       cudaMemcpyHostToDevice));
  return KFAC_OK;
}

extern "C" int kfac_selftest_pivots(int count, const float* q, const float* p,
                                    float* rsqrt, float* quot, float* checked,
                                    void* stream) {
  KFAC_REQUIRE(count > 0 && q && p && rsqrt && quot && checked,
               "selftest_pivots: null pointer or count=%d", count);
  pivots_selftest_kernel<<<ceil_div(count, 256), 256, 0,
                           (cudaStream_t)stream>>>(count, q, p, rsqrt, quot,
                                                   checked);
  KFAC_LAUNCH_CHECK("pivots_selftest_kernel");
  return KFAC_OK;
}

extern "C" int kfac_inverse_plan_destroy(kfac_inverse_plan* p) {
  if (p == nullptr) return KFAC_OK;
  plan_drop_graph(p);
  for (int k = 1; k < S_COUNT; ++k) {
    if (p->side_stream[k] != nullptr) cudaStreamDestroy(p->side_stream[k]);
    if (p->join_ev[k] != nullptr) cudaEventDestroy(p->join_ev[k]);
  }
  if (p->fork_ev != nullptr) cudaEventDestroy(p->fork_ev);
  for (cudaEvent_t ev : p->events) cudaEventDestroy(ev);
  cudaFree(p->params_dev);
  cudaFree(p->scale_dev);
  cudaFree(p->add2_dev);
  cudaFree(p->refine_items_dev);
  cudaFree(p->refine_sums_dev);
  cudaFree(p->refine_vec_dev);
  cudaFree(p->refine_gate_dev);
  cudaFree(p->refine_count_dev);
  cudaFree(p->mats_dev);
  cudaFree(p->trace_dev);
  cudaFree(p->add_dev);
  cudaFree(p->info_dev);
  cudaFree(p->sorted_dev);
  cudaFree(p->descs_dev);
  delete p;
  return KFAC_OK;
}
