// What a state-space layer (and any layer that convolves its projections) needs around the recurrence.
//
// conv_act: out[t, c] = act(bias[c] + sum_j w[c, j] * in(t - taps + 1 + j, c)) over each request's own inputs, on
// rows of the engine's type that may be a view of a projection's columns.  As in short_conv, tiles are aligned to
// requests: tile 0 of a request reads the request's last taps - 1 inputs from its state slot (zeros before the
// sequence starts), and the same threads write the new ones afterwards.  Sums and the activation are 32-bit.
//
// ssm_gates: step sizes dt = softplus(dt_raw + dt_bias) and decays exp(-exp(A_log) dt) per (token, head), 32-bit.
//
// ssm_output, a block per (token, norm group): y = (o + D_h x) silu(z), divided by the root mean square of its
// group, times a weight.
#include "common.cuh"

namespace ftk {

constexpr int kCaTile = 16;      // tokens per tile (at least taps - 1)
constexpr int kCaMaxTaps = 16;
constexpr int kCaThreads = 128;  // four channels a thread
constexpr int kCaAhead = 8;      // rows of a thread on their way or in use

__device__ __forceinline__ float softplus_f(float z) { return z > 0.f ? z + log1pf(expf(-z)) : log1pf(expf(z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }

// What bounds it: instructions, half of them the activation's exponential and division (2.8 of 4 an SM cycle), behind the latency
// of the rows.  2,048 tokens of 8,192 channels, 4 taps, with silu: 43 us with the rows' loads between the divisions, 30 now (67 MB to and
// from memory: 10); 1,024 tokens of 1,536 channels 13.6 and 9.1.  Rows that are not aligned, one number off: 41 and 34, 14.4 and 13.3.
template <typename T, int TAPS>
__global__ void __launch_bounds__(kCaThreads)
conv_act_kernel(const T* __restrict__ x, long long x_stride, const float* __restrict__ w, const float* __restrict__ bias,
                int taps, int act, float* __restrict__ state, const int32_t* __restrict__ state_slots,
                const int32_t* __restrict__ seg_info, int n_segs, int n_slots, T* __restrict__ out, int n_tokens, int C,
                int vec_ok) {
  pdl_wait();
  pdl_trigger();
  const int c0 = (blockIdx.y * kCaThreads + threadIdx.x) * 4;
  if (c0 >= C) return;
  const int nc = min(4, C - c0);
  const bool vec = vec_ok && nc == 4;
  if (TAPS > 0) taps = TAPS;
  // the thread's taps and bias first: they wait for nothing, and the search for the block's request runs beside them
  constexpr int kMost = TAPS > 0 ? TAPS : kCaMaxTaps;
  float wt[kMost][4], bs[4];
  if (TAPS == 4 && nc == 4 && ((uintptr_t)w & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float of[4];
      Vec4<float>::load(w + (size_t)(c0 + i) * 4, of);
#pragma unroll
      for (int j = 0; j < 4; ++j) wt[j][i] = of[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < (TAPS > 0 ? TAPS : taps); ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) wt[j][i] = i < nc ? w[(size_t)(c0 + i) * taps + j] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) bs[i] = (bias && i < nc) ? bias[c0 + i] : 0.f;
  int tile = blockIdx.x, seg = 0, q_start = 0, q_len = 0, kv_len = 0;
  for (; seg < n_segs; ++seg) {
    q_start = seg_info[seg * 4]; q_len = seg_info[seg * 4 + 1]; kv_len = seg_info[seg * 4 + 2];
    const int n = q_len > 0 ? (q_len + kCaTile - 1) / kCaTile : 0;
    if (tile < n) break;
    tile -= n;
  }
  if (seg >= n_segs || q_start < 0 || q_start + q_len > n_tokens || kv_len < q_len) return;
  const int keep = taps - 1;
  const int slot = state_slots[seg];
  const bool has_slot = state && slot >= 0 && slot < n_slots;
  const int before = kv_len - q_len;
  float* st = has_slot ? state + ((size_t)slot * keep) * C + c0 : nullptr;  // row r: the input `keep - r` places back
  const bool first = tile == 0;
  const int t0 = tile * kCaTile, t1 = min(q_len, t0 + kCaTile);
  // input `s` places into the request's tokens of this step (negative: before them)
  auto input = [&](int s, float (&v)[4]) {
    if (s >= 0) {
      const T* r = x + (size_t)(q_start + s) * x_stride + c0;
      if (vec) Vec4<T>::load(r, v);
      else for (int i = 0; i < 4; ++i) v[i] = i < nc ? to_float(r[i]) : 0.f;
    } else {
      const int r = keep + s;  // the slot's row
      for (int i = 0; i < 4; ++i) v[i] = (st && before > 0 && r >= 0 && -s <= before && i < nc) ? st[(size_t)r * C + i] : 0.f;
    }
  };
  // TAPS > 1: the sums that the next tokens have so far, the next one's first.  (An input is added to all of them and they move up by
  // that; a window of inputs would be moved by itself.)
  constexpr int K = TAPS > 1 ? TAPS - 1 : 1;
  float sums[K][4];
  auto add = [&](const float (&in)[4], float (&acc)[4]) {  // acc: the sums of the token whose input it is, all in
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = fmaf(wt[K][i], in[i], sums[0][i]);
#pragma unroll
    for (int r = 0; r + 1 < K; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[r][i] = fmaf(wt[K - 1 - r][i], in[i], sums[r + 1][i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) sums[K - 1][i] = fmaf(wt[0][i], in[i], bs[i]);
  };
  // Aligned rows are seven ahead of their use, every thread's own piece of them in shared memory: in registers they cost blocks on
  // an SM (four rows ahead 93 registers a thread, 67 this way), and behind the branches of the activation's divisions the compiler
  // asks for nothing early.
  using Raw = typename Vec4<T>::Raw;
  __shared__ Raw ring[kCaAhead][kCaThreads];
  const int n = t1 - t0;
  const T* src = x + (size_t)(q_start + t0) * x_stride + c0;
  T* dst = out + (size_t)(q_start + t0) * C + c0;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&ring[0][threadIdx.x]);
  auto ask = [&](int u) {
    if (u < n)
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(mine + (u % kCaAhead) * (uint32_t)sizeof(ring[0])),
                   "l"(src + (size_t)u * x_stride), "n"((int)sizeof(Raw)) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (TAPS > 1) {
    if (vec) {
#pragma unroll
      for (int u = 0; u < kCaAhead - 1; ++u) ask(u);
    }
    float in[4], none[4];
#pragma unroll
    for (int r = 0; r < K; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[r][i] = bs[i];
#pragma unroll
    for (int r = 0; r < K; ++r) {
      input(t0 - K + r, in);
      add(in, none);
    }
  }
  if (TAPS > 1 && vec) {
#pragma unroll 1
    for (int u = 0; u < n; ++u) {
      ask(u + kCaAhead - 1);  // (into the place of the row read last)
      asm volatile("cp.async.wait_group %0;" ::"n"(kCaAhead - 1) : "memory");
      float cur[4], acc[4];
      Vec4<T>::unpack(ring[u % kCaAhead][threadIdx.x], cur);
      add(cur, acc);
      if (act == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = silu_f(acc[i]);
      }
      Vec4<T>::store(dst + (size_t)u * C, acc);
    }
  } else
  for (int t = t0; t < t1; ++t) {
    float cur[4], acc[4];
    input(t, cur);
    if (TAPS > 1) {
      add(cur, acc);
    } else {
      for (int i = 0; i < 4; ++i) acc[i] = bs[i];
      for (int j = 0; j < taps; ++j) {
        float in[4];
        if (j == keep) { for (int i = 0; i < 4; ++i) in[i] = cur[i]; }
        else input(t - keep + j, in);
        for (int i = 0; i < 4; ++i) acc[i] = fmaf(wt[j][i], in[i], acc[i]);
      }
    }
    if (act == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = silu_f(acc[i]);
    }
    T* o = out + (size_t)(q_start + t) * C + c0;
    if (vec) Vec4<T>::store(o, acc);
    else for (int i = 0; i < nc; ++i) o[i] = from_float<T>(acc[i]);
  }
  if (first && st) {  // the new state: the request's last `keep` inputs, oldest first (row r comes from row r + q_len or from the step)
    for (int r = 0; r < keep; ++r) {
      float v[4];
      input(q_len - keep + r, v);
      for (int i = 0; i < nc; ++i) st[(size_t)r * C + i] = v[i];
    }
  }
}

template <typename T>
__global__ void ssm_gates_kernel(const T* __restrict__ dt, long long dt_stride, const float* __restrict__ dt_bias,
                                 const float* __restrict__ a_log, float* __restrict__ dt_out, float* __restrict__ decay_out,
                                 int n_tokens, int H) {
  pdl_wait();
  pdl_trigger();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)n_tokens * H) return;
  const int t = (int)(i / H), h = (int)(i % H);
  const float step = softplus_f(to_float(dt[(size_t)t * dt_stride + h]) + dt_bias[h]);
  dt_out[i] = step;
  decay_out[i] = expf(-expf(a_log[h]) * step);
}

template <typename T>
__global__ void __launch_bounds__(256)
ssm_output_kernel(const float* __restrict__ o32, const T* __restrict__ x, long long x_stride, const float* __restrict__ d_skip,
                  const T* __restrict__ z, long long z_stride, const float* __restrict__ norm_w, int norm_groups, float eps,
                  T* __restrict__ out, int H, int P) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) float sm[];  // [L] the gated values of this group, then 33 floats of scratch
  const size_t t = blockIdx.x;
  const int g = blockIdx.y;
  const int I = H * P, L = I / norm_groups, base = g * L;
  float* scratch = sm + ((L + 3) & ~3);
  float ss = 0.f;
  for (int j = threadIdx.x; j < L; j += blockDim.x) {
    const int c = base + j;
    const float xv = to_float(x[t * x_stride + c]), zv = to_float(z[t * z_stride + c]);
    const float y = fmaf(d_skip[c / P], xv, o32[t * I + c]) * silu_f(zv);
    sm[j] = y;
    ss = fmaf(y, y, ss);
  }
  ss = block_sum(ss, scratch);
  const float r = rsqrtf(ss / (float)L + eps);
  for (int j = threadIdx.x; j < L; j += blockDim.x)
    out[t * I + base + j] = from_float<T>(sm[j] * r * norm_w[base + j]);
}

}  // namespace ftk

using namespace ftk;

extern "C" int ftk_conv_act(const void* x, long long x_stride, int dtype, const float* w, const float* bias, int taps,
                            int act, float* state, int n_slots, const int32_t* state_slots, const int32_t* seg_info,
                            int n_segs, void* out, int n_tokens, int channels, void* stream) {
  FTK_REQUIRE(dtype_ok(dtype), "conv_act: bad dtype %d", dtype);
  FTK_REQUIRE(taps >= 1 && taps <= kCaMaxTaps && taps - 1 <= kCaTile, "conv_act: %d taps (1 to %d taken)", taps, kCaMaxTaps);
  FTK_REQUIRE(n_tokens >= 0 && channels >= 1 && n_segs >= 1 && x_stride >= channels && (act == 0 || act == 1),
              "conv_act: bad sizes");
  if (n_tokens == 0) return 0;
  FTK_REQUIRE(x && w && out && seg_info && state_slots && (taps == 1 || state), "conv_act: null pointer");
  const int quad = 4 * dtype_size(dtype);
  const int vec_ok = channels % 4 == 0 && x_stride % 4 == 0 && (uintptr_t)x % quad == 0 && (uintptr_t)out % quad == 0;
  dim3 grid((n_tokens + kCaTile - 1) / kCaTile + n_segs, (channels + kCaThreads * 4 - 1) / (kCaThreads * 4));
  cudaStream_t s = (cudaStream_t)stream;
#define FTK_CA(TY, N)                                                                                                  \
  FTK_LAUNCH((conv_act_kernel<TY, N>), grid, kCaThreads, 0, s, (const TY*)x, x_stride, w, bias, taps, act, state,    \
             state_slots, seg_info, n_segs, n_slots, (TY*)out, n_tokens, channels, vec_ok)
#define FTK_CA_TAPS(TY)                \
  do {                                 \
    if (taps == 2) FTK_CA(TY, 2);      \
    else if (taps == 3) FTK_CA(TY, 3); \
    else if (taps == 4) FTK_CA(TY, 4); \
    else FTK_CA(TY, 0);                \
  } while (0)
  if (dtype == FTK_F32) FTK_CA_TAPS(float);
  else FTK_CA_TAPS(__nv_bfloat16);
#undef FTK_CA_TAPS
#undef FTK_CA
  FTK_LAUNCH_CHECK("conv_act");
  return 0;
}

extern "C" int ftk_ssm_gates(const void* dt, long long dt_stride, int dtype, const float* dt_bias, const float* a_log,
                             float* dt_out, float* decay_out, int n_tokens, int n_heads, void* stream) {
  FTK_REQUIRE(dtype_ok(dtype), "ssm_gates: bad dtype %d", dtype);
  FTK_REQUIRE(n_tokens >= 0 && n_heads >= 1 && dt_stride >= n_heads, "ssm_gates: bad sizes");
  if (n_tokens == 0) return 0;
  FTK_REQUIRE(dt && dt_bias && a_log && dt_out && decay_out, "ssm_gates: null pointer");
  const long long n = (long long)n_tokens * n_heads;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FTK_F32) FTK_LAUNCH(ssm_gates_kernel<float>, blocks, 256, 0, s, (const float*)dt, dt_stride, dt_bias, a_log, dt_out, decay_out, n_tokens, n_heads);
  else FTK_LAUNCH(ssm_gates_kernel<__nv_bfloat16>, blocks, 256, 0, s, (const __nv_bfloat16*)dt, dt_stride, dt_bias, a_log, dt_out, decay_out, n_tokens, n_heads);
  FTK_LAUNCH_CHECK("ssm_gates");
  return 0;
}

extern "C" int ftk_ssm_output(const float* o32, const void* x, long long x_stride, const float* d_skip, const void* z,
                              long long z_stride, int dtype, const float* norm_w, int norm_groups, float eps, void* out,
                              int n_tokens, int n_heads, int vdim, void* stream) {
  FTK_REQUIRE(dtype_ok(dtype), "ssm_output: bad dtype %d", dtype);
  const long long inner = (long long)n_heads * vdim;
  FTK_REQUIRE(n_tokens >= 0 && n_heads >= 1 && vdim >= 1 && norm_groups >= 1 && norm_groups <= 65535 &&
              inner % norm_groups == 0 && x_stride >= inner && z_stride >= inner, "ssm_output: bad sizes");
  if (n_tokens == 0) return 0;
  FTK_REQUIRE(o32 && x && d_skip && z && norm_w && out, "ssm_output: null pointer");
  const int L = (int)(inner / norm_groups);
  const size_t smem = ((size_t)((L + 3) & ~3) + 33) * sizeof(float);
  FTK_REQUIRE(smem <= 200 * 1024, "ssm_output: norm groups of %d channels do not fit shared memory", L);
  dim3 grid(n_tokens, norm_groups);
  cudaStream_t s = (cudaStream_t)stream;
#define FTK_SSM_OUT(TY)                                                                                         \
  do {                                                                                                          \
    auto kern = ssm_output_kernel<TY>;                                                                          \
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
    FTK_LAUNCH(kern, grid, 256, smem, s, o32, (const TY*)x, x_stride, d_skip, (const TY*)z, z_stride, norm_w,  \
               norm_groups, eps, (TY*)out, n_heads, vdim);                                                      \
  } while (0)
  if (dtype == FTK_F32) FTK_SSM_OUT(float);
  else FTK_SSM_OUT(__nv_bfloat16);
#undef FTK_SSM_OUT
  FTK_LAUNCH_CHECK("ssm_output");
  return 0;
}
