// tcgen05 / mbarrier building blocks of the kernels on tensor cores: shared-memory
// and instruction descriptors for 128-byte-swizzled operand tiles (TF32 K-major,
// 16-bit values K- or MN-major), MMA issue / commit, accumulator loads from tensor
// memory, bounded barrier waits, and the splits of fp32 values into two TF32, fp16
// or bf16 terms.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace kfac {

constexpr int TC_BM = 128;
constexpr unsigned TC_SPIN_LIMIT = 1u << 22;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// Launches that may begin while the one before still runs (programmatic dependent
// launch): they read nothing that it writes, and write nothing, before
// wait_for_launch_before, which returns when it is complete.  A kernel lets the next
// one begin once it has its tensor memory: the next one's CTAs keep theirs while
// they wait.
// So what any launch of such a row writes is changed while the kernel runs, and a
// parameter that points there is not `__restrict__` (nor read by __ldg): the compiler
// may move reads through one ahead of the wait.  That is for tables written before
// the first of the row.
__device__ __forceinline__ void let_next_launch_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_launch_before() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// True in one lane of a converged warp.  MMAs are issued behind this, not behind
// a comparison of the lane number: the compiler then knows that one thread
// issues them (measured per 128 x 64 x 16 bf16 MMA: 110 cycles against 237).
__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count));
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// Bounded wait on a phase parity; false if the limit ran out or the CTA is
// already aborting.
__device__ __forceinline__ bool mbar_wait_status(unsigned long long* bar,
                                                 unsigned parity,
                                                 volatile int* abort_flag,
                                                 int* status_word,
                                                 unsigned limit = TC_SPIN_LIMIT) {
  const unsigned addr = smem_u32(bar);
  {
    // fast path: the phase is usually complete already; test_wait answers
    // without the suspend machinery of try_wait
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  for (unsigned i = 0; i < limit; ++i) {
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
  atomicExch(status_word, 1);
  return false;
}

__device__ __forceinline__ unsigned long long tc_smem_desc(unsigned addr) {
  // K-major, 128-byte swizzle: 8-row groups 1024 bytes apart.
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFF) >> 4);         // start address
  d |= (unsigned long long)1 << 16;                         // LBO (unused)
  d |= (unsigned long long)(1024 >> 4) << 32;               // SBO
  d |= (unsigned long long)1 << 46;                         // descriptor version
  d |= (unsigned long long)2 << 61;                         // SWIZZLE_128B
  return d;
}

__device__ __forceinline__ unsigned tc_instr_desc(int n) {
  // D = f32, A = B = tf32, both K-major, M = 128, N = n
  return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) |
         ((unsigned)(TC_BM >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(unsigned tmem_d, unsigned long long da,
                                       unsigned long long db, unsigned idesc,
                                       unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

// K-major tiles of 16-bit values have the descriptor above.  MN-major: 64 columns
// per 128-byte row of one k, groups of 8 k 1024 bytes apart, the next 64 columns
// `step` bytes further.
__device__ __forceinline__ unsigned long long tc_smem_desc_mn(unsigned addr,
                                                              unsigned step) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr & 0x3FFFF) >> 4);
  d |= (unsigned long long)(step >> 4) << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  d |= (unsigned long long)2 << 61;
  return d;
}

// D = f32, A = B = f16, M = 128, N = n
__device__ __forceinline__ unsigned tc_half_desc(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | ((unsigned)a_mn << 15) | ((unsigned)b_mn << 16) |
         ((unsigned)(n >> 3) << 17) | ((unsigned)(TC_BM >> 4) << 24);
}

// D = f32, A = B = bf16, both K-major, M = 128, N = n
__device__ __forceinline__ unsigned tc_bf16_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) |
         ((unsigned)(TC_BM >> 4) << 24);
}

__device__ __forceinline__ void tc_mma_half(unsigned tmem_d,
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

__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
      ::"r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tc_ld16(unsigned taddr, float v[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
        "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Two pieces of 16 columns with one wait.
__device__ __forceinline__ void tc_ld16_pair(unsigned ta, unsigned tb,
                                             float v[16], float w[16]) {
  unsigned r[16], s[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
        "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(ta)
      : "memory");
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]),
        "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]),
        "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
      : "r"(tb)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = __uint_as_float(r[i]);
    w[i] = __uint_as_float(s[i]);
  }
}

// 32 columns of 16 accumulator rows of a warp's quarter: v[4 j + 2 h + e] is row
// lane / 4 + 8 h, column 8 j + 2 (lane % 4) + e.  The caller waits
// (tcgen05.wait::ld).
__device__ __forceinline__ void tc_ld_16x32(unsigned taddr, float v[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
        "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Hands a block's tensor memory back, by the warp that took it, behind the block's
// last barrier.  `aborted`: a wait of the block ran out, and the copies and MMAs
// already issued get time to end before the tensor memory, and with the block its
// shared memory, are another's (bounded: 64 us).  Not ahead of that barrier: a warp
// that is done before the others wait would find no flag.
__device__ __forceinline__ void tc_release(unsigned tmem, unsigned columns,
                                           bool aborted) {
  if (aborted) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncwarp();
  }
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
               ::"r"(tmem), "r"(columns)
               : "memory");
}

// Byte offset of element (row, k) inside a K-major SW128 tile (k < 32).
__device__ __forceinline__ int sw128_chunk_off(int row, int chunk) {
  return row * 128 + ((chunk ^ (row & 7)) << 4);
}

__device__ __forceinline__ void sts128(unsigned addr, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
               "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

__device__ __forceinline__ void sts32(unsigned addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// hi = x rounded to TF32 (nearest, ties away from zero), lo = x - hi (exact in
// fp32; the tensor core reads its top 11 bits).  The rounding is two integer
// instructions (add half an ulp of TF32, clear the low 13 bits): cvt.rna
// would be one, but conversions issue on the quarter-rate XU pipe, which the
// producers saturate.
__device__ __forceinline__ float tf32_round(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

__device__ __forceinline__ void store_split(unsigned hi_addr, unsigned lo_addr,
                                            float4 x) {
  float4 h, l;
  h.x = tf32_round(x.x); h.y = tf32_round(x.y);
  h.z = tf32_round(x.z); h.w = tf32_round(x.w);
  l.x = x.x - h.x; l.y = x.y - h.y; l.z = x.z - h.z; l.w = x.w - h.w;
  sts128(hi_addr, h);
  sts128(lo_addr, l);
}

__device__ __forceinline__ void sts64(unsigned addr, unsigned a, unsigned b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b)
               : "memory");
}

// Two values, already scaled into the range of fp16, as fp16 terms y = hi + lo:
// both rounded to nearest, so hi + lo carries 22 significant bits down to 2^-3
// and an absolute error of at most 2^-25 below (fp16 denormals; the tensor core
// takes them as they are).  Finite values beyond the range saturate; what is not
// finite leaves a NaN in lo (y * 0).
__device__ __forceinline__ unsigned half2_sat(float y0, float y1) {
  unsigned r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y1), "f"(y0));
  return r;
}

__device__ __forceinline__ void split_half2(float y0, float y1, unsigned& hi,
                                            unsigned& lo) {
  hi = half2_sat(y0, y1);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = half2_sat(fmaf(y0, 0.f, y0 - f.x), fmaf(y1, 0.f, y1 - f.y));
}

// Floor of the binary logarithm of |x|; kNoExp for zero, 128 for what is not
// finite.  Below the normal numbers -127, which is an upper bound.
constexpr int kNoExp = -4096;
__device__ __forceinline__ int exp_of(float x) {
  const unsigned u = __float_as_uint(x) & 0x7fffffffu;
  return u != 0 ? (int)(u >> 23) - 127 : kNoExp;
}

// x 2^n in two exact steps; n beyond +-252 counts as that, which takes every
// finite x out of the range of fp32 or leaves a zero.
__device__ __forceinline__ float scale_exp(float x, int n) {
  n = max(min(n, 252), -252);
  const int h = n >> 1;
  return x * __uint_as_float((unsigned)(127 + h) << 23) *
         __uint_as_float((unsigned)(127 + n - h) << 23);
}

// Two values as bf16 terms x = hi + lo: one word of each (the first value in the
// low half).  Rounding to bf16 is an integer add of half an ulp (ties away from
// zero); the byte permute then takes the upper halves.  No cvt: conversions issue
// on the quarter-rate XU pipe (measured at 130 % of its sustained peak with
// cvt.rn.bf16x2 in the gather kernel).
__device__ __forceinline__ void split_bf16x2(float x0, float x1, unsigned& hi,
                                             unsigned& lo) {
  const unsigned r0 = __float_as_uint(x0) + 0x8000u;
  const unsigned r1 = __float_as_uint(x1) + 0x8000u;
  hi = __byte_perm(r0, r1, 0x7632);
  const float l0 = x0 - __uint_as_float(r0 & 0xffff0000u);
  const float l1 = x1 - __uint_as_float(r1 & 0xffff0000u);
  lo = __byte_perm(__float_as_uint(l0) + 0x8000u,
                   __float_as_uint(l1) + 0x8000u, 0x7632);
}

// `early`: the launch may begin before the one in front of it has ended.
template <typename... P, typename... A>
static int launch_behind(const char* name, bool early, void (*kernel)(P...),
                         int blocks, int threads, int smem, cudaStream_t stream,
                         A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  KFAC_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  KFAC_LAUNCH_CHECK(name);
  return KFAC_OK;
}

}  // namespace kfac
