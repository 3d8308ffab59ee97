// Epilogue of the tile kernel (tc_tile.cu): 32 x 32 pieces of the accumulators
// TMEM -> registers -> shared memory -> global rows (C = alpha A B), with mirrored
// rows, fp16 chunks of the result and the preconditioning update.
#pragma once

#include "gemm_simt.cuh"
#include "tc_common.cuh"

namespace kfac {

constexpr int TT_EP = 36;         // row pitch of an epilogue piece (floats)
// 32 accumulator columns of this warp's 32 rows (both accumulators added, times
// alpha) into its shared-memory piece, a row per lane.
template <int TN>
__device__ __forceinline__ void tile_acc_piece(unsigned tmem, int q, int c0,
                                               float alpha, bool zero,
                                               float* piece, int lane) {
  const unsigned row = (unsigned)(q * 32) << 16;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[16], w[16];
    if (!zero) {
      tc_ld16_pair(tmem + row + (unsigned)(c0 + 16 * h),
                   tmem + row + (unsigned)(TN + c0 + 16 * h), v, w);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = w[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 16; i += 4)
      *reinterpret_cast<float4*>(&piece[lane * TT_EP + 16 * h + i]) =
          make_float4(alpha * (v[i] + w[i]), alpha * (v[i + 1] + w[i + 1]),
                      alpha * (v[i + 2] + w[i + 2]),
                      alpha * (v[i + 3] + w[i + 3]));
  }
}

// Tile (bi, bj) of lower-triangular problem tile t; 128 x 256 tiles exist iff
// 2 bj <= bi, 128 x 128 tiles iff bj <= bi.
template <int TN>
__device__ __forceinline__ void tile_lower(int t, int& bi, int& bj) {
  if (TN == 128) {
    tri_tile(t, bi, bj);
    return;
  }
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

// Preconditioning epilogue of one 32 x 32 piece: kf to the weight and bias
// parts, and the momentum update where the layer has it fused.
__device__ __forceinline__ void tile_precond(const GemmDesc& g,
                                             const float* piece, int gr0,
                                             int rows, int gc0, int cols,
                                             int lane, float lr,
                                             float momentum) {
  const int dW = g.dW;
  const bool fused = g.pW != nullptr;
  if ((dW & 3) == 0 && gc0 + 31 < dW && cols >= 32 &&
      ((reinterpret_cast<uintptr_t>(g.kfW) | reinterpret_cast<uintptr_t>(g.pW) |
        reinterpret_cast<uintptr_t>(g.vW)) & 15) == 0) {
    const int sub = lane >> 3, wc = 4 * (lane & 7);
    const float* pp = piece + sub * TT_EP + wc;
    long long idx = (long long)(gr0 + sub) * dW + gc0 + wc;
#pragma unroll 1
    for (int i0 = 0; i0 < 8; i0 += 4, idx += 16LL * dW, pp += 16 * TT_EP) {
      float4 ov[4], op[4];
      long long at = idx;
#pragma unroll
      for (int i = 0; i < 4; ++i, at += 4LL * dW) {
        if (!fused || 4 * (i0 + i) + sub >= rows) continue;
        ov[i] = *reinterpret_cast<const float4*>(g.vW + at);
        op[i] = *reinterpret_cast<const float4*>(g.pW + at);
      }
      at = idx;
#pragma unroll
      for (int i = 0; i < 4; ++i, at += 4LL * dW) {
        if (4 * (i0 + i) + sub >= rows) continue;
        const float4 kf = *reinterpret_cast<const float4*>(&pp[4 * i * TT_EP]);
        if (g.kfW) *reinterpret_cast<float4*>(g.kfW + at) = kf;
        if (!fused) continue;
        float4 nv;
        nv.x = momentum * ov[i].x - lr * kf.x;
        nv.y = momentum * ov[i].y - lr * kf.y;
        nv.z = momentum * ov[i].z - lr * kf.z;
        nv.w = momentum * ov[i].w - lr * kf.w;
        *reinterpret_cast<float4*>(g.vW + at) = nv;
        *reinterpret_cast<float4*>(g.pW + at) =
            make_float4(op[i].x + nv.x, op[i].y + nv.y, op[i].z + nv.z,
                        op[i].w + nv.w);
      }
    }
    return;
  }
  // a column per lane, eight rows at a time
  if (lane >= cols) return;
  const bool w = gc0 + lane < dW;
  float* okf = w ? g.kfW : g.kfb;
  float* opar = w ? g.pW : g.pb;
  float* ovel = w ? g.vW : g.vb;
  const long long step = w ? dW : 1;
  long long idx = gr0 * step + (w ? gc0 + lane : 0);
  // (values, then stores, each under one condition: with branches between them a
  // row takes 250 cycles)
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += 8, idx += 8 * step) {
    const int n = rows - r0;
    float ov[8], op[8], kf[8];
    if (opar != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n) {
          ov[i] = ovel[idx + i * step];
          op[i] = opar[idx + i * step];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) kf[i] = piece[(r0 + i) * TT_EP + lane];
    if (okf != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < n) okf[idx + i * step] = kf[i];
    }
    if (opar == nullptr) continue;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      kf[i] = momentum * ov[i] - lr * kf[i];
      op[i] += kf[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) ovel[idx + i * step] = kf[i];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) opar[idx + i * step] = op[i];
  }
}


// Four columns of row `gr` of a result as fp16 terms into its chunks.
__device__ __forceinline__ void pack_store4(const GemmDesc& g, int gr, int gc,
                                            float4 x) {
  const float s = g.pack_scale;
  unsigned h0, h1, l0, l1;
  split_half2(s * x.x, s * x.y, h0, l0);
  split_half2(s * x.z, s * x.w, h1, l1);
  unsigned char* p = g.pack + 8 * ((gc >> 2) & 1);
  p += (long long)(gc >> 7) * g.pack_tile + (long long)(gr >> 5) * kChunk +
       ((gc >> 6) & 1) * 8192 + sw128_chunk_off(gr & 31, (gc & 63) >> 3);
  *reinterpret_cast<uint2*>(p) = make_uint2(h0, h1);
  *reinterpret_cast<uint2*>(p + 4096) = make_uint2(l0, l1);
}

struct TileOut {
  int m0, n0, m_valid, n_valid;
  float lr, momentum;
};

// One warp's share of a tile: accumulator rows of quarter q, 32-column pieces h,
// h + G, ...; `wait` returns once the accumulators are final (false: never).
// `piece`: 32 x TT_EP floats of shared memory of this warp's own.
template <int TN, int G, bool PRE, typename Wait>
__device__ __forceinline__ void tile_epilogue(const GemmDesc& g,
                                              const TileOut& o, unsigned tmem,
                                              bool zero, int q, int h, int lane,
                                              float* piece, Wait wait) {
  const int m0 = o.m0, n0 = o.n0, m_valid = o.m_valid, n_valid = o.n_valid;
  const int flags = g.flags;
  const int row0 = q * 32, rows = min(32, m_valid - row0);
  const bool lower = (flags & G_LOWER) != 0;
  const float alpha = g.alpha;
  float* C = g.C;
  const bool pack = g.pack != nullptr;
  const long long ldc = g.ldc;
  // rows of a piece as 16-byte words: lane -> row 4 i + lane / 8, word lane % 8
  const bool vec = (ldc & 3) == 0 &&
                   (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  const int sub = lane >> 3, wc = 4 * (lane & 7);
  // Pieces whose 32 rows and columns are all stored, in whole words, take a path
  // without a test per row.
  auto whole = [&](int c0) {
    return vec && rows == 32 && c0 + 32 <= n_valid &&
           (!lower || n0 + c0 + 31 <= m0 + row0);
  };
  bool ok = true;
  if (!zero) {
    ok = wait();
    ok = __all_sync(0xffffffffu, ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  for (int c0 = 32 * h; c0 < n_valid && ok; c0 += 32 * G) {
    tile_acc_piece<TN>(tmem, q, c0, alpha, zero, piece, lane);
    __syncwarp();
    if (PRE) {
      if (rows > 0)
        tile_precond(g, piece, m0 + row0, rows, n0 + c0, n_valid - c0, lane,
                     o.lr, o.momentum);
    } else if (whole(c0)) {
      const int gc = n0 + c0 + wc;
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        const int gr = m0 + row0 + sub + 4 * i0;
        const float* pp = &piece[(4 * i0 + sub) * TT_EP + wc];
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          x[i] = *reinterpret_cast<const float4*>(&pp[4 * i * TT_EP]);
        if (pack) {
#pragma unroll
          for (int i = 0; i < 4; ++i) pack_store4(g, gr + 4 * i, gc, x[i]);
        }
        const long long idx = (long long)gr * ldc + gc;
        if (C != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<float4*>(C + idx + 4 * i * ldc) = x[i];
        }
      }
      if (flags & G_MIRROR) {
        // a row per lane, so that a column of the piece is a contiguous store
        float* dst = C + (long long)(n0 + c0) * ldc + m0 + row0 + lane;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 y =
              *reinterpret_cast<const float4*>(&piece[lane * TT_EP + i]);
          dst[i * ldc] = y.x;
          dst[(i + 1) * ldc] = y.y;
          dst[(i + 2) * ldc] = y.z;
          dst[(i + 3) * ldc] = y.w;
        }
      }
    } else if (rows > 0) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        const int r = row0 + 4 * i + sub, c = c0 + wc;
        const int gr = m0 + r;
        const int cend = lower ? min(n_valid, gr - n0 + 1) : n_valid;
        const float4 x =
            *reinterpret_cast<const float4*>(&piece[(4 * i + sub) * TT_EP + wc]);
        const long long idx = (long long)gr * ldc + n0 + c;
        if (r >= m_valid || c >= cend) continue;
        // (packed results have whole words only)
        if (pack) pack_store4(g, gr, n0 + c, x);
        if (C == nullptr) continue;
        if (vec && c + 3 < cend) {
          *reinterpret_cast<float4*>(C + idx) = x;
        } else {
          const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c + e < cend) C[idx + e] = xs[e];
        }
      }
      if (flags & G_MIRROR) {
        // a row per lane, so that a column of the piece is a contiguous store
        const int gr = m0 + row0 + lane;
        if (lane < rows) {
          float* dst = C + (long long)(n0 + c0) * ldc + gr;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 x =
                *reinterpret_cast<const float4*>(&piece[lane * TT_EP + i]);
            const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e, dst += ldc)
              if (c0 + i + e < n_valid && n0 + c0 + i + e < gr) *dst = xs[e];
          }
        }
      }
    }
    __syncwarp();
  }
}

}  // namespace kfac
