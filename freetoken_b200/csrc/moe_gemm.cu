// Grouped expert matrix products: the true 32-bit path (on CUDA cores for few rows an expert and for rows without 16-byte loads,
// else on the tensor cores in three pieces, moe_gemm_split.cuh), and the path for bfloat16 sizes that the tensor-core kernels refuse.
//
// Rows are sorted by expert (expert e owns rows [offsets[e], offsets[e+1])); the row counts are
// only known on the device, so the grid is an upper bound on the row tiles (ceil(R / BM) + experts with rows) and a
// block first finds the expert and rows of its tile from the offsets.
//   gemm1: out[r, n] = act(x[r] . W1[e][n], x[r] . W1[e][I + n])   (gate and up halves together,
//          activation fused; the two products are rounded to the storage dtype first, where the
//          reference stores them, python/freetoken/moe/fused_nvfp4.py:317-344)
//   gemm2: out[r, n] = (a[r] . W2[e][n]) * weight[route of r]      (weight on the 32-bit
//          accumulator, python/freetoken/kernel/triton/fused_moe.py:292-296)
// How many rows an expert got does not change the order of a sum; the mean number of rows a step brings does (it picks the
// kernel: steps of a few rows an expert spread a sum over a warp's lanes).
#include "common.cuh"

namespace ftk {

// What a block's tile is: the expert, its first row and the end of the expert's rows; expert -1 past the last tile.  The
// first warp finds it, 32 experts at a time.
struct ExpertTile { int e, row0, row_end; };
__device__ __forceinline__ ExpertTile find_tile(const int32_t* offsets, int n_experts, int tile, int rows) {
  __shared__ ExpertTile found;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) found.e = -1;
    __syncwarp();
    int before = 0;  // tiles of the experts before these
    for (int i0 = 0; i0 < n_experts; i0 += 32) {
      const int i = i0 + lane;
      const int a = i < n_experts ? offsets[i] : 0, b = i < n_experts ? offsets[i + 1] : 0;
      const int n = (b - a + rows - 1) / rows;
      int upto = n;  // of these 32 up to this lane's
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const int t = tile - before - (upto - n);
      if (t >= 0 && t < n) found = {i, a + t * rows, b};
      before += __shfl_sync(0xffffffffu, upto, 31);
      if (before > tile) break;
    }
  }
  __syncthreads();
  return found;
}

// four elements of a row from column k on; columns and rows that do not exist are zeros
template <bool WIDE, typename T>
__device__ __forceinline__ void load4(const T* row, int k, int K, bool ok, float (&v)[4]) {
  if (WIDE) {  // (rows of a multiple of four elements, on addresses of as many)
    if (ok && k < K) {
      Vec4<T>::load(row + k, v);
      return;
    }
    v[0] = v[1] = v[2] = v[3] = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = ok && k + i < K ? to_float(row[k + i]) : 0.f;
  }
}

template <typename T, bool GATED>
__device__ __forceinline__ T finish(float x, float up, float weight, int act, float alpha, float limit) {
  if (!GATED) return from_float<T>(x * weight);
  return from_float<T>(gated_act(to_float(from_float<T>(x)), to_float(from_float<T>(up)), act, alpha, limit));
}

}  // namespace ftk

#include "moe_gemm_split.cuh"

namespace ftk {

// Tiles of BM rows x 64 gate and 64 up columns (or 128 columns): 128 threads with BM / 8 rows x 8 columns of sums each, k in
// steps of 16 through two shared-memory buffers, the next step's 16-byte loads in flight under this step's products.  What
// bounds it is the FMA pipe: per k a thread reads 16 numbers (four 16-byte loads) for 64 products.  Every sum runs over k in
// order.  (27 TFLOP/s in 32 bits, before moe_gemm_split.cuh took those with 16-byte loads.)
constexpr int kBK = 16, kTiledThreads = 128, kTiledCols = 128;
template <typename T, bool GATED, int BM, bool WIDE>
__global__ void __launch_bounds__(kTiledThreads) moe_gemm_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                       const int32_t* __restrict__ offsets, int n_experts,
                                                       int K, int N, int w_rows,
                                                       const int32_t* __restrict__ sorted_routes,
                                                       const float* __restrict__ route_weights, int n_routes,
                                                       int act, float alpha, float limit, T* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  constexpr int TM = BM / 8, LA = BM + 4, LB = kTiledCols + 4, NA = BM * 4 / kTiledThreads, NB = kTiledCols * 4 / kTiledThreads;
  __shared__ __align__(16) float As[2][kBK][LA];
  __shared__ __align__(16) float Bs[2][kBK][LB];
  const ExpertTile tile = find_tile(offsets, n_experts, blockIdx.y, BM);
  if (tile.e < 0) return;
  const int n0 = blockIdx.x * (GATED ? kTiledCols / 2 : kTiledCols);
  const T* we = w + (size_t)tile.e * w_rows * K;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float ra[NA][4], rb[NB][4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const int i = threadIdx.x + u * kTiledThreads, row = tile.row0 + (i >> 2);
      load4<WIDE>(x + (size_t)row * K, k0 + 4 * (i & 3), K, row < tile.row_end, ra[u]);
    }
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      const int i = threadIdx.x + u * kTiledThreads, c = i >> 2;
      const int n = n0 + (GATED ? c & 63 : c);
      load4<WIDE>(we + (size_t)(GATED && c >= 64 ? N + n : n) * K, k0 + 4 * (i & 3), K, n < N, rb[u]);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const int i = threadIdx.x + u * kTiledThreads;
#pragma unroll
      for (int j = 0; j < 4; ++j) As[buf][4 * (i & 3) + j][i >> 2] = ra[u][j];
    }
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      const int i = threadIdx.x + u * kTiledThreads;
#pragma unroll
      for (int j = 0; j < 4; ++j) Bs[buf][4 * (i & 3) + j][i >> 2] = rb[u][j];
    }
  };
  float acc[TM][8] = {};
  fetch(0);
  put(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < K; k0 += kBK, buf ^= 1) {
    const bool more = k0 + kBK < K;
    if (more) fetch(k0 + kBK);
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
      float a[TM], b[8];
#pragma unroll
      for (int i = 0; i < TM; i += 4) Vec4<float>::load(&As[buf][k][ty * TM + i], reinterpret_cast<float(&)[4]>(a[i]));
      Vec4<float>::load(&Bs[buf][k][tx * 4], reinterpret_cast<float(&)[4]>(b[0]));
      Vec4<float>::load(&Bs[buf][k][64 + tx * 4], reinterpret_cast<float(&)[4]>(b[4]));
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (more) {
      put(buf ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = tile.row0 + ty * TM + i;
    if (row >= tile.row_end) continue;
    float weight = 1.f;
    if (!GATED) {
      const int route = sorted_routes[row];
      weight = (route >= 0 && route < n_routes) ? route_weights[route] : 0.f;
    }
    T* o = out + (size_t)row * N;
#pragma unroll
    for (int h = 0; h < (GATED ? 1 : 2); ++h)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + 64 * h + tx * 4 + j;
        if (n < N) o[n] = finish<T, GATED>(acc[i][4 * h + j], acc[i][4 + j], weight, act, alpha, limit);
      }
  }
}

// Few rows an expert (decode steps): bound by reading the weights once.  A warp takes a gate and an up row of the weights (or
// two rows) at a time, its lanes 16 bytes of each side by side, eight such loads in flight, against up to eight of the expert's
// rows (from L1, shared by the block's warps); the lanes' sums meet in shuffles.  Eight routes over 16 such experts: 19 us for
// each of the two products (46 MB of gate and up rows: 2.4 TB/s at so small a launch); the tiled kernel took 110.
constexpr int kFewWarps = 8, kFewPairs = 2, kFewRows = 8;
template <typename T, bool GATED, int R>
__device__ __forceinline__ void few_rows(const T* x, const T* wa, const T* wb, int K, float (&acc)[2][kFewRows], int nr) {
  const int lane = threadIdx.x & 31;
  constexpr int U = 4;  // steps of 128 elements in flight
  for (int k0 = 4 * lane; k0 < K; k0 += 128 * U) {
    float a[U][4], b[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      load4<true>(wa, k0 + 128 * u, K, true, a[u]);
      load4<true>(wb, k0 + 128 * u, K, true, b[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float v[4];
        load4<true>(x + (size_t)r * K, k0 + 128 * u, K, r < nr, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[0][r] = fmaf(v[j], a[u][j], acc[0][r]);
          acc[1][r] = fmaf(v[j], b[u][j], acc[1][r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    acc[0][r] = warp_sum(acc[0][r]);
    acc[1][r] = warp_sum(acc[1][r]);
  }
}
template <typename T, bool GATED>
__global__ void __launch_bounds__(32 * kFewWarps) moe_gemm_few_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                       const int32_t* __restrict__ offsets, int n_experts,
                                                       int K, int N, int w_rows,
                                                       const int32_t* __restrict__ sorted_routes,
                                                       const float* __restrict__ route_weights, int n_routes,
                                                       int act, float alpha, float limit, T* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const ExpertTile tile = find_tile(offsets, n_experts, blockIdx.y, kFewRows);
  if (tile.e < 0) return;
  const T* we = w + (size_t)tile.e * w_rows * K;
  const T* xr = x + (size_t)tile.row0 * K;
  const int nr = min(kFewRows, tile.row_end - tile.row0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int p = 0; p < kFewPairs; ++p) {
    const int pair = (blockIdx.x * kFewPairs + p) * kFewWarps + warp;
    const int na = GATED ? pair : 2 * pair, nb = GATED ? N + pair : min(2 * pair + 1, N - 1);
    if (na >= N) return;
    const T *wa = we + (size_t)na * K, *wb = we + (size_t)nb * K;
    float acc[2][kFewRows] = {};
    if (nr == 1) few_rows<T, GATED, 1>(xr, wa, wb, K, acc, nr);
    else if (nr == 2) few_rows<T, GATED, 2>(xr, wa, wb, K, acc, nr);
    else if (nr <= 4) few_rows<T, GATED, 4>(xr, wa, wb, K, acc, nr);
    else few_rows<T, GATED, 8>(xr, wa, wb, K, acc, nr);
#pragma unroll
    for (int r = 0; r < kFewRows; ++r) {  // lane r finishes row r
      if (lane != r || r >= nr) continue;
      float weight = 1.f;
      if (!GATED) {
        const int route = sorted_routes[tile.row0 + r];
        weight = (route >= 0 && route < n_routes) ? route_weights[route] : 0.f;
      }
      T* o = out + (size_t)(tile.row0 + r) * N;
      o[na] = finish<T, GATED>(acc[0][r], acc[1][r], weight, act, alpha, limit);
      if (!GATED && 2 * pair + 1 < N) o[nb] = finish<T, GATED>(acc[1][r], 0.f, weight, act, alpha, limit);
    }
  }
}

// Which of them: by the mean number of rows an expert has (the counts are on the device), and 16-byte (bfloat16: 8-byte)
// loads where rows and bases allow them.  Up to 4 rows the kernel for few rows: 16 experts of 1,024 x 1,408 in 32 bits with 1, 2
// and 4 rows each 49 + 31, 50 + 35 and 68 + 46 us for the two products, against 90 + 43 of the tensor cores' 128-row tiles at 5 to
// 64 rows.  In bfloat16 up to 32 rows tiles of 32 rows, one an expert; at 33 an expert has two of them, and tiles of 64 are faster.
// The mean can mislead: 256 rows of 64 experts' four each on one of them are 33 tiles of eight rows, 146 + 133 us
// (the kernels of 32-row tiles before these: 180 + 201).
template <typename T, bool GATED>
static int launch_moe_gemm(const void* x, const void* w, const int32_t* offsets, int n_experts, int K, int N, int w_rows,
                           const int32_t* routes, const float* weights, int n_routes, int act, float alpha, float limit, void* out,
                           cudaStream_t s) {
  const bool wide = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & (4 * sizeof(T) - 1)) == 0;
  auto grid_of = [&](int rows, int cols) { return dim3((N + cols - 1) / cols, (n_routes + rows - 1) / rows + (n_experts < n_routes ? n_experts : n_routes)); };
#define FTK_MOE_GEMM(kern, rows, cols, threads) \
  do { \
    const dim3 grid = grid_of(rows, cols); \
    if (grid.y > 65535u) return -1; \
    FTK_LAUNCH((kern), grid, threads, 0, s, (const T*)x, (const T*)w, offsets, n_experts, K, N, w_rows, routes, weights, n_routes, act, \
               alpha, limit, (T*)out); \
    return 0; \
  } while (0)
  constexpr int cols = GATED ? kTiledCols / 2 : kTiledCols;
  constexpr bool f32 = sizeof(T) == 4;
  auto note = [](const char* gate_up, const char* down) { note_variant(GATED ? gate_up : down); };
  // (tiles of a few rows are the most: with so many experts that a grid cannot hold them, larger ones)
  if (wide && n_routes <= 4 * n_experts && grid_of(kFewRows, 1).y <= 65535u) {
    if (f32) note("expert gate/up product: float32, few rows an expert", "expert down product: float32, few rows an expert");
    else note("expert gate/up product: bfloat16, few rows an expert", "expert down product: bfloat16, few rows an expert");
    FTK_MOE_GEMM((moe_gemm_few_kernel<T, GATED>), kFewRows, (GATED ? 1 : 2) * kFewPairs * kFewWarps, 32 * kFewWarps);
  }
  if constexpr (f32) {
    if (wide) {
      note("expert gate/up product: float32 on the tensor cores", "expert down product: float32 on the tensor cores");
      return launch_moe_gemm_split<GATED>((const float*)x, (const float*)w, offsets, n_experts, K, N, w_rows, routes, weights, n_routes, act, alpha, limit, (float*)out, s);
    }
    note("expert gate/up product: float32 on CUDA cores", "expert down product: float32 on CUDA cores");
  } else {
    note("expert gate/up product: bfloat16 on CUDA cores", "expert down product: bfloat16 on CUDA cores");
    if (wide && n_routes <= 32 * n_experts) FTK_MOE_GEMM((moe_gemm_kernel<T, GATED, 32, true>), 32, cols, kTiledThreads);
    if (wide) FTK_MOE_GEMM((moe_gemm_kernel<T, GATED, 64, true>), 64, cols, kTiledThreads);
  }
  FTK_MOE_GEMM((moe_gemm_kernel<T, GATED, 32, false>), 32, cols, kTiledThreads);
#undef FTK_MOE_GEMM
}

}  // namespace ftk

using namespace ftk;

// Defined in moe_gemm_tc.cu: the tcgen05 kernels for bfloat16; return -1 when the sizes are not
// theirs (the caller then uses the kernels above).
int ftk_moe_gemm1_act_tc(const void* x, const void* w1, const int32_t* expert_offsets, int n_experts,
                         int n_routes, int hidden, int inter, int act, float alpha, float limit, void* out,
                         const int32_t* sorted_routes, int top_k, int n_tokens, cudaStream_t stream);
int ftk_moe_gemm2_tc(const void* a, const void* w2, const int32_t* expert_offsets, const int32_t* sorted_routes,
                     const float* topk_weights, int n_experts, int n_routes, int hidden, int inter, void* out,
                     cudaStream_t stream);

extern "C" int ftk_moe_gemm1_act(const void* x_sorted, const void* w1, int dtype, const int32_t* expert_offsets,
                                 int n_experts, int n_routes, int hidden, int inter, int act, float alpha,
                                 float limit, void* out, void* stream) {
  FTK_REQUIRE(dtype_ok(dtype), "moe_gemm1_act: bad dtype %d", dtype);
  FTK_REQUIRE(act == FTK_ACT_SILU || act == FTK_ACT_SWIGLUOAI, "moe_gemm1_act: unknown activation %d", act);
  FTK_REQUIRE(n_experts >= 1 && n_routes >= 0 && hidden >= 1 && inter >= 1, "moe_gemm1_act: bad sizes");
  if (n_routes == 0) return 0;
  FTK_REQUIRE(x_sorted && w1 && expert_offsets && out, "moe_gemm1_act: null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FTK_BF16) {
    const int rc = ftk_moe_gemm1_act_tc(x_sorted, w1, expert_offsets, n_experts, n_routes, hidden, inter, act, alpha,
                                        limit, out, nullptr, 0, 0, s);
    if (rc >= 0) return rc;
  }
  const int rc = dtype == FTK_F32
      ? launch_moe_gemm<float, true>(x_sorted, w1, expert_offsets, n_experts, hidden, inter, 2 * inter, nullptr, nullptr, n_routes, act,
                                     alpha, limit, out, s)
      : launch_moe_gemm<__nv_bfloat16, true>(x_sorted, w1, expert_offsets, n_experts, hidden, inter, 2 * inter, nullptr, nullptr,
                                             n_routes, act, alpha, limit, out, s);
  FTK_REQUIRE(rc == 0, "moe_gemm1_act: too many row tiles (%d routes, %d experts)", n_routes, n_experts);
  FTK_LAUNCH_CHECK("moe_gemm1_act");
  return 0;
}

// The same from the tokens' rows in their own order: the kernel gathers the rows of each expert itself
// (bfloat16 on the tensor cores only; ftk_moe_gemm1_gather_fits says whether the sizes are taken).
extern "C" int ftk_moe_gemm1_act_gather(const void* x, const void* w1, const int32_t* expert_offsets,
                                        const int32_t* sorted_routes, int top_k, int n_tokens, int n_experts,
                                        int n_routes, int hidden, int inter, int act, float alpha, float limit,
                                        void* out, void* stream) {
  FTK_REQUIRE(act == FTK_ACT_SILU || act == FTK_ACT_SWIGLUOAI, "moe_gemm1_act_gather: unknown activation %d", act);
  FTK_REQUIRE(n_experts >= 1 && n_routes >= 0 && hidden >= 1 && inter >= 1 && top_k >= 1 && n_tokens >= 1,
              "moe_gemm1_act_gather: bad sizes");
  if (n_routes == 0) return 0;
  FTK_REQUIRE(x && w1 && expert_offsets && sorted_routes && out, "moe_gemm1_act_gather: null pointer");
  const int rc = ftk_moe_gemm1_act_tc(x, w1, expert_offsets, n_experts, n_routes, hidden, inter, act, alpha, limit, out,
                                      sorted_routes, top_k, n_tokens, (cudaStream_t)stream);
  FTK_REQUIRE(rc >= 0, "moe_gemm1_act_gather: width %d, expert width %d, %d experts are not taken by the tensor-core "
              "kernel (ask ftk_moe_gemm1_gather_fits first; copy the rows with moe_gather otherwise)", hidden, inter, n_experts);
  return rc;
}

extern "C" int ftk_moe_gemm2(const void* a, const void* w2, int dtype, const int32_t* expert_offsets,
                             const int32_t* sorted_routes, const float* topk_weights, int n_experts, int n_routes,
                             int hidden, int inter, void* out, void* stream) {
  FTK_REQUIRE(dtype_ok(dtype), "moe_gemm2: bad dtype %d", dtype);
  FTK_REQUIRE(n_experts >= 1 && n_routes >= 0 && hidden >= 1 && inter >= 1, "moe_gemm2: bad sizes");
  if (n_routes == 0) return 0;
  FTK_REQUIRE(a && w2 && expert_offsets && sorted_routes && topk_weights && out, "moe_gemm2: null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FTK_BF16) {
    const int rc = ftk_moe_gemm2_tc(a, w2, expert_offsets, sorted_routes, topk_weights, n_experts, n_routes, hidden,
                                    inter, out, s);
    if (rc >= 0) return rc;
  }
  const int rc = dtype == FTK_F32
      ? launch_moe_gemm<float, false>(a, w2, expert_offsets, n_experts, inter, hidden, hidden, sorted_routes, topk_weights, n_routes, 0,
                                      0.f, 0.f, out, s)
      : launch_moe_gemm<__nv_bfloat16, false>(a, w2, expert_offsets, n_experts, inter, hidden, hidden, sorted_routes, topk_weights,
                                              n_routes, 0, 0.f, 0.f, out, s);
  FTK_REQUIRE(rc == 0, "moe_gemm2: too many row tiles (%d routes, %d experts)", n_routes, n_experts);
  FTK_LAUNCH_CHECK("moe_gemm2");
  return 0;
}

// out = x w^T in 32 bits, x [n_rows, k], w [n, k], rows side by side (moe_gemm_split.cuh).
extern "C" int ftk_linear_split(const float* x, const float* w, float* out, int n_rows, int n, int k, void* stream) {
  FTK_REQUIRE(n_rows >= 0 && n >= 1 && k >= 4 && k % 4 == 0, "linear_split: %d rows of %d x %d", n_rows, n, k);
  if (n_rows == 0) return 0;
  FTK_REQUIRE(x && w && out && (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) == 0, "linear_split: operands on 16-byte boundaries");
  note_variant("linear: float32 on the tensor cores");
  const int rc = launch_moe_gemm_split<false>(x, w, nullptr, 1, k, n, n, nullptr, nullptr, n_rows, 0, 0.f, 0.f, out, (cudaStream_t)stream);
  FTK_REQUIRE(rc == 0, "linear_split: too many rows (%d)", n_rows);
  FTK_LAUNCH_CHECK("linear_split");
  return 0;
}
