// Preconditioning kf = G_inv * [grad_W, grad_b] * A_inv for all layers in two
// grouped launches; the second launch's epilogue splits the result into the
// weight and bias parts and can apply the momentum update in place.  Larger
// calls go through fp16 chunks (tc_packed.cu): sizes of the gradients' rows and
// columns, operands' rows as chunks, U = grad * A_inv^T, kf = G_inv * U.
#include <algorithm>
#include <vector>

#include "gemm_simt.cuh"

using namespace kfac;

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// One layer's operands in chunks and their rows' scales, offsets in bytes.
struct ChunkLayout {
  size_t G, A, g, U;             // G_inv, A_inv, gradient, grad * A_inv^T
  size_t exp_G, exp_A, exp_g;    // exponents of rows
  size_t row, col;               // sizes of the gradient's rows and columns
  size_t fit_A, fit_g;           // factors of U's columns and rows
  size_t total;
};

static ChunkLayout chunk_layout(int dG, int dA) {
  auto chunks = [](int rows, int k) {
    return (size_t)((rows + 127) / 128) * ((k + 31) / 32) * kChunk;
  };
  ChunkLayout c;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += align256(bytes);
    return here;
  };
  c.G = take(chunks(dG, dG));
  c.A = take(chunks(dA, dA));
  c.g = take(chunks(dG, dA));
  c.U = take(chunks(dA, dG));
  // (read in fours up to the end of a k-block)
  c.exp_G = take((dG + 31) * sizeof(short));
  c.exp_A = take((dA + 31) * sizeof(short));
  c.exp_g = take((dG + 31) * sizeof(short));
  c.row = take(dG * sizeof(short));
  c.col = take((dA + 31) * sizeof(short));
  c.fit_A = take(dA * sizeof(float));
  c.fit_g = take(dG * sizeof(float));
  c.total = at;
  return c;
}

// Tables in front of the layers' chunks: two products a layer, then these.
struct ChunkTables {
  size_t jobs, sizes, total;
};

static ChunkTables chunk_tables(int count) {
  ChunkTables t;
  t.jobs = align256(2 * (size_t)count * sizeof(GemmDesc));
  t.sizes = t.jobs + align256(3 * (size_t)count * sizeof(PackRows));
  t.total = t.sizes + align256((size_t)count * sizeof(GradSizes));
  return t;
}

// Whether a call goes through chunks, by its longest layer: three launches more than
// in tiles, but a k-block costs 0.4 us instead of 0.6 - 0.9, or of up to 1.5 where
// the tile kernel cannot load 16-byte words of A_inv and has to append a bias
// column.  k-blocks of the sum over rows count twice: the tile kernel has more
// tiles there, and chunks of a long A_inv cost more to make.  us in tiles and in
// chunks, by 2 kb(dG) + kb(dA):
//   words: 256 x 256 (24) 26 31, 256 x 768 (40) 38 39, 448 x 448 (42) 36 38, 128 x
//     1152 (44) 43 45, 512 x 512 (48) 40 38, 256 x 1024 (48) 45 43, 64 x 2304 (76)
//     62 62, 512 x 4608 (176) 163 138;
//   odd: 189 x 189 (18) 33 40, 253 x 253 (24) 39 41, 317 x 317 (30) 43 43, 64 x 801
//     (30) 47 46, 95 x 855 (33) 54 47, 509 x 509 (48) 59 47;
//   with a bias: 64 x 147 (9) 21 36, 53 x 333 (15) 31 37, 64 x 400 (17) 30 30, 200 x
//     100 (18) 33 31, 10 x 500 (18) 31 30, 200 x 200 (21) 34 31, 400 x 64 (29) 36 30.
static bool chunks_pay(int count, const int* dG, const int* dW,
                       const std::vector<int>& hb) {
  for (int i = 0; i < count; ++i) {
    const int dA = dW[i] + hb[i];
    const int line = hb[i] ? 18 : (dA & 3) != 0 ? 30 : 45;
    if (2 * ((dG[i] + 31) / 32) + (dA + 31) / 32 >= line) return true;
  }
  return false;
}

constexpr float kGainU = 32768.f;

// kfac_precondition through chunks.
static int precondition_chunks(
    int count, const int* dG, const int* dW, const std::vector<int>& hb,
    const float* const* G_inv, const float* const* A_inv,
    const float* const* grad_W, const float* const* grad_b, float* const* kf_W,
    float* const* kf_b, float* const* param_W, float* const* param_b,
    float* const* mom_W, float* const* mom_b, float lr, float momentum, char* ws,
    cudaStream_t st) {
  const ChunkTables at_table = chunk_tables(count);
  const size_t jobs_at = at_table.jobs, sizes_at = at_table.sizes;
  const size_t tables = at_table.total;
  std::vector<char> host(tables, 0);
  GemmDesc* descs = reinterpret_cast<GemmDesc*>(host.data());
  PackRows* jobs = reinterpret_cast<PackRows*>(host.data() + jobs_at);
  GradSizes* sizes = reinterpret_cast<GradSizes*>(host.data() + sizes_at);
  char* const base = ws;
  const GemmDesc* descs_dev = reinterpret_cast<GemmDesc*>(base);
  ws += tables;
  int rows = 0, grad_rows = 0, groups = 0;
  std::vector<int> dA(count);
  for (int i = 0; i < count; ++i) dA[i] = dW[i] + hb[i];
  const int columns = grad_group_columns(dA.data(), count);
  auto at = [](char* base, size_t off) {
    return reinterpret_cast<unsigned char*>(base + off);
  };
  auto vec = [](char* base, size_t off) {
    return reinterpret_cast<float*>(base + off);
  };
  auto exps = [](char* base, size_t off) {
    return reinterpret_cast<short*>(base + off);
  };
  for (int i = 0; i < count; ++i) {
    const int dg = dG[i], dw = dW[i], da = dw + hb[i];
    const ChunkLayout c = chunk_layout(dg, da);
    const long long nkA = (da + 31) / 32, nkG = (dg + 31) / 32;
    // Sums run over the gradient's columns, then over its rows.  The columns are
    // divided by their size and those of A_inv multiplied by it, so that features
    // of any scale are held alike; likewise U's rows and G_inv's columns by the
    // size of the gradient's rows.  (By their norms, which are known when the
    // gradient is packed, G_inv takes a launch of its own: three layers of the
    // MLP 70 us instead of 65.)
    // Errors without: see the tests of rows and features of any scale.
    const float* const bias = hb[i] ? grad_b[i] : nullptr;
    GradSizes& z = sizes[i];
    z = GradSizes();
    z.src = grad_W[i]; z.extra = bias;
    z.row = exps(ws, c.row); z.col = exps(ws, c.col);
    z.rows = dg; z.cols = dw;
    z.row_begin = grad_rows; z.col_begin = groups;
    grad_rows += dg;
    groups += (da + columns - 1) / columns;
    auto job = [&](PackRole role, const float* src, const float* extra,
                   size_t dst, const short* col, int cols, int nrows,
                   size_t exp) -> PackRows& {
      PackRows& j = jobs[3 * i + role];
      j = PackRows();
      j.role = role;
      j.src = src; j.extra = extra; j.dst = at(ws, dst);
      j.col = col; j.col_sign = role == PACK_GRAD ? -1 : 1;
      j.exp = exps(ws, exp);
      j.cols = cols;
      j.row_begin = rows;
      rows += nrows;
      return j;
    };
    PackRows& ja = job(PACK_A, A_inv[i], nullptr, c.A, z.col, da, da, c.exp_A);
    ja.fit = vec(ws, c.fit_A); ja.gain = kGainU;
    PackRows& jG = job(PACK_G, G_inv[i], nullptr, c.G, z.row, dg, dg, c.exp_G);
    PackRows& jg = job(PACK_GRAD, grad_W[i], bias, c.g, z.col, dw, dg, c.exp_g);
    jg.fit = vec(ws, c.fit_g); jg.size = z.row;
    // U = grad * A_inv^T
    GemmDesc& u = descs[i];
    u = GemmDesc();
    u.A.kfast = u.B.kfast = 1;
    u.M = dg; u.N = da; u.K = da;
    u.alpha = 1.f;
    u.ca = at(ws, c.g); u.ca_tile = nkA * kChunk;
    u.cb = at(ws, c.A); u.cb_tile = nkA * kChunk;
    u.pack = at(ws, c.U); u.pack_tile = nkG * kChunk;
    u.rs = jg.fit; u.cs = ja.fit;
    u.wide = jg.exp;
    // kf = G_inv * U, split and (optionally) applied
    GemmDesc& h = descs[count + i];
    h = GemmDesc();
    h.A.kfast = 1;
    h.M = dg; h.N = da; h.K = dg;
    h.ca = at(ws, c.G); h.ca_tile = nkG * kChunk;
    h.cb = u.pack; h.cb_tile = u.pack_tile;
    h.alpha = 1.f / kGainU;
    h.re = jG.exp; h.ce = ja.exp; h.wide = jg.exp;
    const bool fused = param_W && param_W[i];
    h.kfW = kf_W ? kf_W[i] : nullptr;
    h.kfb = (hb[i] && kf_b) ? kf_b[i] : nullptr;
    h.pW = fused ? param_W[i] : nullptr;
    h.vW = fused ? mom_W[i] : nullptr;
    h.pb = (fused && hb[i]) ? param_b[i] : nullptr;
    h.vb = (fused && hb[i]) ? mom_b[i] : nullptr;
    h.dW = dw;
    ws += c.total;
  }
  const int tiles = packed_number_tiles(descs, count);
  packed_number_tiles(descs + count, count);             // the same tiles
  // (the tables of a few layers travel as kernel arguments)
  if (count > kTileInline)
    KFAC_CUDA(cudaMemcpyAsync(base, host.data(), tables,
                              cudaMemcpyHostToDevice, st));
  const PackRows* jobs_dev = reinterpret_cast<PackRows*>(base + jobs_at);
  int rc = launch_grad_sizes(reinterpret_cast<GradSizes*>(base + sizes_at),
                             sizes, count, grad_rows, groups, columns, st);
  if (rc == KFAC_OK)
    rc = launch_pack_rows(reinterpret_cast<PackRows*>(base + jobs_at), jobs,
                          3 * count, rows, st);
  if (rc == KFAC_OK)
    rc = launch_packed_precond(descs_dev, descs, count, tiles, false, lr,
                               momentum, st);
  if (rc == KFAC_OK)
    rc = launch_packed_precond(descs_dev + count, descs + count, count, tiles,
                               true, lr, momentum, st);
  return rc;
}

static size_t tile_workspace(int count, const int* dG, const int* dW,
                             const std::vector<int>& hb) {
  size_t total = align256(2 * (size_t)count * sizeof(GemmDesc));
  for (int i = 0; i < count; ++i)
    total += align256((size_t)dG[i] * (dW[i] + hb[i]) * sizeof(float));
  return total;
}

// The chunks, or T of the tile kernel where the call goes that way (and for a
// workspace at an odd address and the FFMA engine, which take nothing else).
extern "C" size_t kfac_precond_workspace_bytes(int count, const int* dG,
                                               const int* dW,
                                               const int* has_bias) {
  if (count <= 0 || !dG || !dW) return 0;
  std::vector<int> hb(count, 0);
  for (int i = 0; i < count; ++i) hb[i] = has_bias && has_bias[i] ? 1 : 0;
  const size_t tiles = tile_workspace(count, dG, dW, hb);
  if (!chunks_pay(count, dG, dW, hb)) return tiles;
  size_t chunks = chunk_tables(count).total;
  for (int i = 0; i < count; ++i)
    chunks += chunk_layout(dG[i], dW[i] + hb[i]).total;
  return std::max(chunks, tiles);
}

extern "C" int kfac_precondition(
    int count, const int* dG, const int* dW, const float* const* G_inv,
    const float* const* A_inv, const float* const* grad_W,
    const float* const* grad_b, float* const* kf_W, float* const* kf_b,
    float* const* param_W, float* const* param_b, float* const* mom_W,
    float* const* mom_b, float lr, float momentum, void* workspace,
    size_t workspace_bytes, void* stream) {
  KFAC_REQUIRE(count > 0 && dG && dW && G_inv && A_inv && grad_W,
               "precondition: null argument or count=%d", count);
  std::vector<int> hb(count);
  for (int i = 0; i < count; ++i) {
    KFAC_REQUIRE(dG[i] > 0 && dW[i] > 0, "precondition: bad dims at %d", i);
    KFAC_REQUIRE(G_inv[i] && A_inv[i] && grad_W[i],
                 "precondition: null matrix pointer at %d", i);
    hb[i] = (grad_b && grad_b[i]) ? 1 : 0;
    bool fused = param_W && param_W[i];
    KFAC_REQUIRE(fused || (kf_W && kf_W[i]),
                 "precondition: layer %d has neither kf_W nor param_W", i);
    if (fused)
      KFAC_REQUIRE(mom_W && mom_W[i], "precondition: mom_W missing at %d", i);
    if (hb[i]) {
      KFAC_REQUIRE(fused || (kf_b && kf_b[i]),
                   "precondition: layer %d has a bias gradient but no kf_b", i);
      if (fused)
        KFAC_REQUIRE(param_b && param_b[i] && mom_b && mom_b[i],
                     "precondition: param_b/mom_b missing at %d", i);
    }
  }
  size_t need = kfac_precond_workspace_bytes(count, dG, dW, hb.data());
  if (workspace == nullptr || workspace_bytes < need)
    return fail(KFAC_ERR_WORKSPACE,
                "precondition: workspace of %zu bytes needed, %zu given", need,
                workspace_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = static_cast<char*>(workspace);
  if (engine() == 1 && (reinterpret_cast<uintptr_t>(ws) & 15) == 0 &&
      chunks_pay(count, dG, dW, hb))
    return precondition_chunks(count, dG, dW, hb, G_inv, A_inv, grad_W, grad_b,
                               kf_W, kf_b, param_W, param_b, mom_W, mom_b, lr,
                               momentum, ws, st);
  GemmDesc* descs_dev = reinterpret_cast<GemmDesc*>(ws);
  ws += align256(2 * (size_t)count * sizeof(GemmDesc));

  std::vector<GemmDesc> descs(2 * count);
  int tiles1 = 0, tiles2 = 0;
  const bool use_tc = engine() == 1;
  for (int i = 0; i < count; ++i) {
    const int dg = dG[i], dw = dW[i], da = dw + hb[i];
    float* T = reinterpret_cast<float*>(ws);
    ws += align256((size_t)dg * da * sizeof(float));
    // T = G_inv * [grad_W, grad_b]
    GemmDesc& g = descs[i];
    g = GemmDesc();
    g.A = strided_operand(G_inv[i], 1, dg, dg);    // A(k, m) = G_inv[m][k]
    g.B = strided_operand(grad_W[i], dw, 1, dw);   // B(k, n) = grad[k][n]
    if (hb[i]) { g.B.extra_idx = dw; g.B.extra = grad_b[i]; }
    g.C = T; g.ldc = da; g.M = dg; g.N = da; g.K = dg;
    g.alpha = 1.f; g.beta = 0.f; g.flags = 0;
    g.tile_begin = tiles1;
    g.splits = 1;
    if (!use_tc) tiles1 += gemm_desc_tiles(g);
    // kf = T * A_inv, split and (optionally) applied
    GemmDesc& h = descs[count + i];
    h = GemmDesc();
    h.A = strided_operand(T, 1, da, dg);           // A(k, m) = T[m][k]
    h.B = strided_operand(A_inv[i], 1, da, da);    // B(k, n) = A_inv[n][k]
    h.C = nullptr; h.ldc = 0; h.M = dg; h.N = da; h.K = da;
    h.alpha = 1.f; h.beta = 0.f; h.flags = G_PRECOND;
    h.kfW = kf_W ? kf_W[i] : nullptr;
    h.kfb = (hb[i] && kf_b) ? kf_b[i] : nullptr;
    const bool fused = param_W && param_W[i];
    h.pW = fused ? param_W[i] : nullptr;
    h.vW = fused ? mom_W[i] : nullptr;
    h.pb = (fused && hb[i]) ? param_b[i] : nullptr;
    h.vb = (fused && hb[i]) ? mom_b[i] : nullptr;
    h.dW = dw;
    h.tile_begin = tiles2;
    h.splits = 1;
    if (!use_tc) tiles2 += gemm_desc_tiles(h);
  }
  int cols1 = 0, cols2 = 0;
  if (use_tc) {
    tiles1 = tc_number_tiles(descs.data(), count, sm_count(), &cols1);
    tiles2 = tc_number_tiles(descs.data() + count, count, sm_count(), &cols2);
  }
  // (the tile kernel takes the descriptors of a few layers as an argument)
  if (!use_tc || count > kTileInline)
    KFAC_CUDA(cudaMemcpyAsync(descs_dev, descs.data(),
                              descs.size() * sizeof(GemmDesc),
                              cudaMemcpyHostToDevice, st));
  if (use_tc) {
    int rc = launch_tc_grouped(descs_dev, descs.data(), count, tiles1, cols1,
                               false, 0.f, 0.f, st);
    if (rc != KFAC_OK) return rc;
    return launch_tc_grouped(descs_dev + count, descs.data() + count, count,
                             tiles2, cols2, true, lr, momentum, st);
  }
  int rc = launch_grouped_gemm(descs_dev, count, tiles1, 0.f, 0.f, st);
  if (rc != KFAC_OK) return rc;
  return launch_grouped_gemm(descs_dev + count, count, tiles2, lr, momentum, st);
}

// y = M x, one warp per row.
__global__ void symv_split_kernel(const float* __restrict__ m, int d, int d0,
                                  const float* __restrict__ x0,
                                  const float* __restrict__ x1, float* y0,
                                  float* y1, int* nan_flag) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= d) return;
  const float* mr = m + (long long)row * d;
  float s = 0.f;
  for (int c = lane; c < d; c += 32) {
    float xv = c < d0 ? x0[c] : x1[c - d0];
    s += mr[c] * xv;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) {
    if (row < d0) y0[row] = s; else y1[row - d0] = s;
    if (nan_flag && isnan(s)) atomicExch(nan_flag, 1);
  }
}

// The reference's fallback for a block whose preconditioned gradient contains
// NaN (batch_normalization.py:159-173 with _check_nan): use the raw gradient.
// flag[0] is this call's NaN marker (cleared here), flag[1] counts fallbacks.
__global__ void __launch_bounds__(256)
symv_nan_fallback_kernel(int* __restrict__ flag, int d, int d0,
                         const float* __restrict__ x0,
                         const float* __restrict__ x1, float* y0, float* y1) {
  __shared__ int f;
  if (threadIdx.x == 0) f = flag[0];
  __syncthreads();
  if (f == 0) return;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    if (i < d0) y0[i] = x0[i]; else y1[i - d0] = x1[i - d0];
  }
  if (threadIdx.x == 0) {
    flag[0] = 0;
    flag[1] += 1;
  }
}

extern "C" int kfac_symv_split(const float* m, int d, int d0, const float* x0,
                               const float* x1, float* y0, float* y1,
                               int* nan_flag_dev, void* stream) {
  KFAC_REQUIRE(m && x0 && y0 && d > 0 && d0 > 0 && d0 <= d,
               "symv_split: bad argument");
  KFAC_REQUIRE(d0 == d || (x1 && y1), "symv_split: second piece missing");
  int blocks = ceil_div((long long)d * 32, 256);
  symv_split_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(
      m, d, d0, x0, x1, y0, y1, nan_flag_dev);
  KFAC_LAUNCH_CHECK("symv_split_kernel");
  if (nan_flag_dev != nullptr) {
    symv_nan_fallback_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(
        nan_flag_dev, d, d0, x0, x1, y0, y1);
    KFAC_LAUNCH_CHECK("symv_nan_fallback_kernel");
  }
  return KFAC_OK;
}
