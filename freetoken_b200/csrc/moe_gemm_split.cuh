// Grouped expert products in 32 bits on the tensor cores.  Included by moe_gemm.cu after find_tile and finish.
//
// A tile is 128 of an expert's rows x 128 weight rows (64 gate and 64 up rows), k in steps of 64.  Every operand is taken apart into
// three bfloat16 numbers whose sum it is (split3; from 2^-110 up exactly), and the six products that reach 2^-24 are taken:
//   a1 b1                    the leading product: a chain of four steps of 16 in one of two places in tensor memory, read and added up in
//                            registers while the next step fills the other (the tensor core's accumulator cuts off instead of rounding)
//   a1 b2 + a2 b1            second order, 2^-9 smaller, and
//   a1 b3 + a2 b2 + a3 b1    third order: in places of their own over all of k
// 512 threads fetch the next step's rows, take them apart into the other buffer and add up; one of them issues.  An infinity or NaN (or
// a number that bfloat16 cannot reach) makes its row or column of the tile NaN: such a result is summed once more as 32-bit fmas.
//
// What bounds it: a step's chain, rows fetched and taken apart into shared memory (busy 63 % of the time), a barrier, 24 products of
// 128 x 128 x 16 (0.8 us; the tensor pipe is busy 46 %).  16
// experts of 1,024 x 1,408, gate/up and down (32-bit fmas on the CUDA cores, now): 8 rows each 111 + 86 and 90 + 43 us, 108 rows 287 + 176
// and 101 + 51, 300 rows 651 + 397 and 238 + 127 (180 TFLOP/s of 32-bit products).  Off from 64 bits by 8.7e-7 and 6.7e-7 with fmas
// in order, by 1.8e-7 and 1.3e-7 here.
#pragma once
#include "tc_common.cuh"

namespace ftk {

constexpr int kSplitRows = 128, kSplitThreads = 512;
constexpr int kSplitImage = 128 * 128;          // bytes of 128 rows of 64 elements
constexpr int kSplitBuffer = 6 * kSplitImage;   // three pieces of the rows, three of the weights
constexpr int kSplitSmem = 2 * kSplitBuffer + 1024;
__device__ int g_split_status[4];  // [0] first error code of a wait that ran out, [1] block; 0 = fine

template <bool GATED>
__global__ void __launch_bounds__(kSplitThreads) moe_gemm_split_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                       const int32_t* __restrict__ offsets, int n_experts,
                                                       int K, int N, int w_rows,
                                                       const int32_t* __restrict__ sorted_routes,
                                                       const float* __restrict__ route_weights, int n_routes,
                                                       int act, float alpha, float limit, float* __restrict__ out, bool fours) {
  extern __shared__ unsigned char split_smem[];
  __shared__ uint64_t done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, share = warp >> 2;
  const uint32_t base = (smem_addr(split_smem) + 1023u) & ~1023u;
  unsigned char* tiles = split_smem + (base - smem_addr(split_smem));
  if (tid == 0) {
    mbar_init(&done[0], 1);
    mbar_init(&done[1], 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  // (no offsets: one matrix for all n_routes rows, without weights of routes)
  const ExpertTile tile = offsets ? find_tile(offsets, n_experts, blockIdx.y, kSplitRows) : ExpertTile{0, (int)blockIdx.y * kSplitRows, n_routes};
  if (tile.e >= 0) {
    const int n0 = blockIdx.x * (GATED ? 64 : 128), rows = min(kSplitRows, tile.row_end - tile.row0);
    const float* we = w + (size_t)tile.e * w_rows * K;
    auto weight_row = [&](int c) { return (size_t)(GATED && c >= 64 ? N + n0 + c - 64 : n0 + c); };  // of the tile's c-th column
    // a thread's eights: row i / 8, columns 8 (i % 8), of both operands
    const int c8 = tid & 7;
    const float* src[4];
    bool live[4];
    unsigned char* dst[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = (tid >> 3) + 64 * (u & 1);
      const bool b = u >= 2;
      live[u] = b ? n0 + (GATED ? r & 63 : r) < N : r < rows;
      src[u] = (b ? we + (live[u] ? weight_row(r) : 0) * K : x + (size_t)(tile.row0 + (live[u] ? r : 0)) * K) + 8 * c8;
      dst[u] = tiles + (b ? 3 * kSplitImage : 0) + r * 128 + ((c8 ^ (r & 7)) << 4);
      if (!live[u]) {
#pragma unroll
        for (int m = 0; m < 6; ++m) *reinterpret_cast<uint4*>(dst[u] + (m / 3) * kSplitBuffer + (m % 3) * kSplitImage) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    float v[4][8];
    auto fetch = [&](int s) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 8; i += 4)
          load4<true>(src[u] + 64 * s, i, K - 64 * s - 8 * c8, live[u], reinterpret_cast<float (&)[4]>(v[u][i]));
    };
    auto put = [&](int buf) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!live[u]) continue;
        uint4 p[3];
        split3(v[u], p);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(dst[u] + buf * kSplitBuffer + m * kSplitImage) = p[m];
      }
    };
    bool bad = false;
    auto wait = [&](int s) {
      // (asking again and again: with waits that sleep the down product takes 66 us instead of 43, with one warp asking and a barrier 50)
      if (!bad && !mbar_wait_spin(&done[s & 1], (uint32_t)(s >> 1) & 1u, &abort_flag)) {
        if (atomicCAS(&g_split_status[0], 0, 701) == 0) g_split_status[1] = blockIdx.x;
        abort_flag = 1;
        bad = true;
      }
      __syncwarp();
      tc_fence_after();
    };
    // this thread's row, and 32 of its columns (16 gate and their up columns)
    const uint32_t mine = tmem + ((uint32_t)(quad * 32) << 16);
    auto column = [&](int j) { return GATED ? (j >> 4) * 64 + share * 16 + (j & 15) : share * 32 + j; };
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.f;
    auto add = [&](int from) {
#pragma unroll
      for (int j = 0; j < 32; j += 16) {
        float r[2][8];
        tmem_ld8_start(mine + from + column(j), r[0]);
        tmem_ld8_start(mine + from + column(j + 8), r[1]);
        tmem_ld8_finish(r);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[j + i] += r[i >> 3][i & 7];
      }
    };
    const int steps = (K + 63) / 64;
    fetch(0);
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
      const int buf = s & 1;
      if (s >= 2) {
        wait(s - 2);
        add(buf * 128);
      }
      put(buf);
      if (s + 1 < steps) fetch(s + 1);
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          constexpr uint32_t id = instr_desc(128);
          const uint32_t at = base + buf * kSplitBuffer;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint64_t a[3], b[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
              a[m] = smem_desc(at + m * kSplitImage) + 2 * k;
              b[m] = smem_desc(at + (3 + m) * kSplitImage) + 2 * k;
            }
            tc_mma(tmem + buf * 128, a[0], b[0], id, k != 0);
            tc_mma(tmem + 256, a[0], b[1], id, s | k);
            tc_mma(tmem + 256, a[1], b[0], id, 1);
            tc_mma(tmem + 384, a[0], b[2], id, s | k);
            tc_mma(tmem + 384, a[1], b[1], id, 1);
            tc_mma(tmem + 384, a[2], b[0], id, 1);
          }
          tc_commit(&done[buf]);
        }
        __syncwarp();
      }
    }
    for (int s = max(0, steps - 2); s < steps; ++s) {
      wait(s);
      add((s & 1) * 128);
    }
    float low[32];
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      float r[2][8];
      tmem_ld8_start(mine + 256 + column(j), r[0]);
      tmem_ld8_start(mine + 384 + column(j), r[1]);
      tmem_ld8_finish(r);
#pragma unroll
      for (int i = 0; i < 8; ++i) low[j + i] = r[0][i] + r[1][i];
    }
    const int r = quad * 32 + lane;
    if (r < rows) {
      const size_t row = (size_t)tile.row0 + r;
      float weight = 1.f;
      if (!GATED && sorted_routes) {
        const int route = sorted_routes[row];
        weight = (route >= 0 && route < n_routes) ? route_weights[route] : 0.f;
      }
      bool odd = false;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        acc[j] += low[j];
        odd |= !(fabsf(acc[j]) < INFINITY);
      }
      if (odd) {
#pragma unroll 1
        for (int j = 0; j < 32; ++j) {
          float y = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) y = i == j ? acc[i] : y;
          if (fabsf(y) < INFINITY || n0 + (GATED ? column(j) & 63 : column(j)) >= N) continue;
          const float *xr = x + row * K, *wr = we + weight_row(column(j)) * K;
          y = 0.f;
          for (int k = 0; k < K; ++k) y = fmaf(xr[k], wr[k], y);
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = i == j ? y : acc[i];
        }
      }
      float* o = out + row * N + n0 + column(0);
      constexpr int kOut = GATED ? 16 : 32;
#pragma unroll
      for (int j = 0; j < kOut; j += 4) {
        float y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = finish<float, GATED>(acc[j + i], acc[(j + i + 16) & 31], weight, act, alpha, limit);
        const int n = n0 + column(0) + j;
        if (fours && n < N) {
          Vec4<float>::store(o + j, y);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n + i < N) o[j + i] = y[i];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

template <bool GATED>
static int launch_moe_gemm_split(const float* x, const float* w, const int32_t* offsets, int n_experts, int K, int N, int w_rows,
                                 const int32_t* routes, const float* weights, int n_routes, int act, float alpha, float limit, float* out,
                                 cudaStream_t s) {
  auto kern = moe_gemm_split_kernel<GATED>;
  const dim3 grid((N + (GATED ? 63 : 127)) / (GATED ? 64 : 128), (n_routes + kSplitRows - 1) / kSplitRows + (!offsets ? 0 : n_experts < n_routes ? n_experts : n_routes));
  if (grid.y > 65535u) return -1;
  FTK_REQUIRE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem) == cudaSuccess,
              "moe_gemm (32 bits): cannot set up the kernel");
  const bool fours = N % 4 == 0 && ((uintptr_t)out & 15) == 0;  // (outputs may start anywhere: rows and weights alone decide on this kernel)
  FTK_LAUNCH(kern, grid, kSplitThreads, kSplitSmem, s, x, w, offsets, n_experts, K, N, w_rows, routes, weights, n_routes, act, alpha, limit, out, fours);
  return 0;
}

int moe_gemm_split_status(int* out) { return take_status(g_split_status, out); }  // (merged into ftk_read_status)
int moe_gemm_split_set_status(int code) { return set_status(g_split_status, code); }

}  // namespace ftk
