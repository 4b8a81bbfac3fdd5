// The gated delta rule in chunks of 32 tokens, for portions of bfloat16 prompts with one decay a head (delta.cu runs
// everything else token by token).
//
// With S the state as the chunk finds it, c_t = g_1 ... g_t and c_t / c_s the decays behind token s,
//   u_t = beta_t (v_t - c_t S^T k_t - sum_(s < t) (c_t / c_s) (k_s . k_t) u_s)
//   o_t = c_t S^T q_t + sum_(s <= t) (c_t / c_s) (k_s . q_t) u_s            S <- c_C S + sum_s (c_C / c_s) k_s u_s^T,
// so U = T X with X = beta (V - c K S), T = (I + L)^-1, L_ts = beta_t (c_t / c_s) (k_s . k_t), and O = c Q S + A T X.  T, A T and
// the factors of a token depend on the chunk alone: delta_prep_kernel makes them for all chunks side by side (the decays in 64
// bits: where a state lives for hundreds of tokens, their rounding is most of what a result is off).  What is left to do in order (delta_chunk_kernel) is three products a chunk, [K; Q] S, [T; A T] X and
// K^T U, which are 32-bit fmas on the CUDA cores over register tiles.  Decays are running products, never differences of
// logarithms.  The state is rounded once a chunk instead of once a token pair.
//
// What bounds it: shared memory (77 % busy) and the fma pipe (50 %) between four barriers a chunk, with one block an SM, where the
// token-by-token kernel is bound by the chain of sums, shuffles and updates that a token
// pair cannot start before the one before has ended.  q and k stay bfloat16 in shared memory, eight to a 16-byte load, and are
// widened in registers, and fmas go two at a time (fma.rn.f32x2): with 4 x 4 tiles over 32-bit copies the kernel was bound by
// shared memory (87 % busy, 503 us at 48 heads).  The same products on mma.sync, the state in three bfloat16 pieces, took 384 us
// there: that pipe takes a 16 x 8 x 16 product in some 24 cycles, and three pieces make that no faster than the fma pipe.
// 2,048 tokens of one request, both kernels together (token by token -> chunks): 48 heads of 128 x 128 860 -> 405 us, 16 heads
// 538 -> 282.  Distance from 64 bits there: 2.0e-7 -> 1.6e-7, with decays near one 2.5e-6 -> 2.3e-7.
#include "common.cuh"

namespace ftk {

// (delta.cu: the requests of fewer tokens than shorter_than, token by token)
int delta_scan_tokens(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride, const void* b,
                      long long b_stride, const void* a, long long a_stride, float* z, int dtype, const float* a_log, const float* dt_bias,
                      float q_scale, float unit_eps, float* state, int n_slots, const int32_t* state_slots, const int32_t* seg_info,
                      int n_segs, float* out, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim, int shorter_than, void* stream);

constexpr int kDcTokens = 32;                 // tokens a chunk
// scratch of one (chunk, head): rows s of T^T and (A T)^T, columns t in the order of dc_place, then per token beta, beta c rk, c rq, (c_C / c) rk, then c_C
constexpr int kDcMats = kDcTokens * 2 * kDcTokens;
constexpr int kDcBytes = kDcMats * 4 + 4 * kDcTokens * 4 + 16;

struct DeltaChunkArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; const __nv_bfloat16* b; const __nv_bfloat16* a;
  long long q_stride, k_stride, v_stride, b_stride, a_stride;
  const float* a_log; const float* dt_bias;
  float q_scale, unit_eps;
  float* state; int n_slots;
  const int32_t* state_slots; const int32_t* seg_info; int n_segs;
  float* out; int n_tokens, H, G, D, Dv;
  unsigned char* scratch;
  int long_from, n_long, n_chunks;  // requests of long_from tokens and more go in chunks: n_long of them; the chunks that scratch holds
};

__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same added to d by 32-bit additions (products of bfloat16 rows are exact; the tensor core's own additions do not round
// to nearest).
__device__ __forceinline__ void dc_mma_add(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float x[4] = {0.f, 0.f, 0.f, 0.f};
  dc_mma(x, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] += x[i];
}
__device__ __forceinline__ void dc_cp16(void* dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;  // fewer source bytes than 16: the rest is written as zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n));
}
__device__ __forceinline__ uint32_t dc_lds(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// Where row t of T, and right behind it row t of A T, lies among 64: a thread takes tokens that are eight apart.
__host__ __device__ constexpr int dc_place(int t) { return t % 8 * 8 + t / 8 * 2; }

// chunks of a segment; 0 for one that the kernels leave alone
__device__ __forceinline__ int dc_chunks(const DeltaChunkArgs& a, int seg) {
  const int q_start = a.seg_info[seg * 4], q_len = a.seg_info[seg * 4 + 1], kv_len = a.seg_info[seg * 4 + 2];
  if (q_len < a.long_from || q_start < 0 || q_start + q_len > a.n_tokens || kv_len < q_len) return 0;
  return (q_len + kDcTokens - 1) / kDcTokens;
}

// One block per (chunk, key head): the dots of the chunk's rows once for all heads that share them, then a warp a head.
// (W warps, four at least: as many as heads share the rows, up to eight)
template <int D, int W>
__global__ void __launch_bounds__(32 * W) delta_prep_kernel(DeltaChunkArgs a) {
  pdl_wait();
  pdl_trigger();
  constexpr int RL = D + 8;
  __shared__ __align__(16) __nv_bfloat16 sk[kDcTokens * RL], sq[kDcTokens * RL];
  __shared__ float kk[kDcTokens][kDcTokens + 1], qk[kDcTokens][kDcTokens + 1], s2q[kDcTokens];
  extern __shared__ __align__(16) unsigned char prep_smem[];
  float (*sl)[kDcTokens][kDcTokens + 4] = reinterpret_cast<float (*)[kDcTokens][kDcTokens + 4]>(prep_smem);
  __shared__ int found[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {  // which segment's chunk this is
    if (lane == 0) found[0] = -1;
    __syncwarp();
    int before = 0;
    for (int i0 = 0; i0 < a.n_segs; i0 += 32) {
      const int n = i0 + lane < a.n_segs ? dc_chunks(a, i0 + lane) : 0;
      int upto = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const int t = (int)blockIdx.x - before - (upto - n);
      if (t >= 0 && t < n) { found[0] = i0 + lane; found[1] = t; }
      before += __shfl_sync(0xffffffffu, upto, 31);
      if (before > (int)blockIdx.x) break;
    }
  }
  __syncthreads();
  const int seg = found[0];
  if (seg < 0) return;
  const int q_start = a.seg_info[seg * 4] + found[1] * kDcTokens, nb = min(kDcTokens, a.seg_info[seg * 4 + 1] - found[1] * kDcTokens);
  const int g = blockIdx.y, per = a.H / a.G;
  for (int i = threadIdx.x; i < kDcTokens * (D / 8); i += 32 * W) {
    const int t = i / (D / 8), d = i % (D / 8) * 8;
    const size_t tok = (size_t)(q_start + min(t, nb - 1));
    uint4 kv = *reinterpret_cast<const uint4*>(a.k + tok * a.k_stride + (size_t)g * D + d);
    uint4 qv = *reinterpret_cast<const uint4*>(a.q + tok * a.q_stride + (size_t)g * D + d);
    if (t >= nb) kv = qv = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(sk + t * RL + d) = kv;
    *reinterpret_cast<uint4*>(sq + t * RL + d) = qv;
  }
  __syncthreads();
  if (warp < 4) {
    // k_t . k_s and q_t . k_s: warp w takes tokens s = 8 w .. 8 w + 7 of both, for all t
    const int gr = lane >> 2, gc = 2 * (lane & 3);
    float acc[4][4] = {};
#pragma unroll
    for (int kc = 0; kc < D; kc += 16) {
      const uint32_t b0 = dc_lds(sk + (8 * warp + gr) * RL + kc + gc), b1 = dc_lds(sk + (8 * warp + gr) * RL + kc + gc + 8);
#pragma unroll
      for (int m = 0; m < 4; ++m) {  // rows 0-15 and 16-31 of k, then of q
        const __nv_bfloat16* r = (m < 2 ? sk : sq) + (16 * (m & 1) + gr) * RL + kc + gc;
        const uint32_t af[4] = {dc_lds(r), dc_lds(r + 8 * RL), dc_lds(r + 8), dc_lds(r + 8 * RL + 8)};
        dc_mma_add(acc[m], af, b0, b1);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float (*dst)[kDcTokens + 1] = m < 2 ? kk : qk;
      const int r = 16 * (m & 1) + gr, c = 8 * warp + gc;
      dst[r][c] = acc[m][0]; dst[r][c + 1] = acc[m][1];
      dst[r + 8][c] = acc[m][2]; dst[r + 8][c + 1] = acc[m][3];
    }
    // |q|^2, four lanes a token
    const int t = 8 * warp + gr;
    float s = 0.f;
    for (int d = 4 * (lane & 3); d < D; d += 16) {
      float v[4];
      Vec4<__nv_bfloat16>::load(sq + t * RL + d, v);
      s = fmaf(v[0], v[0], fmaf(v[1], v[1], fmaf(v[2], v[2], fmaf(v[3], v[3], s))));
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((lane & 3) == 0) s2q[t] = s;
  }
  __syncthreads();
  const int t = lane;
  // (rows that do not exist are zeros: with unit_eps = 0 they would have no unit vector)
  const float rk = t < nb ? rsqrtf(kk[t][t] + a.unit_eps) : 0.f, rq = t < nb ? rsqrtf(s2q[t] + a.unit_eps) * a.q_scale : 0.f;
  const size_t tok = (size_t)(q_start + min(t, nb - 1));
  for (int hh = warp; hh < per; hh += W) {
    const int h = g * per + hh;
    float beta = 0.f;
    double gt = 1.0;  // (tokens that do not exist add nothing and decay nothing)
    if (t < nb) {
      const double z = (double)__bfloat162float(a.a[tok * a.a_stride + h]) + (double)a.dt_bias[h];
      beta = 1.f / (1.f + expf(-__bfloat162float(a.b[tok * a.b_stride + h])));
      gt = exp(-exp((double)a.a_log[h]) * (z > 0.0 ? z + log1p(exp(-z)) : log1p(exp(z))));
    }
    double c = gt, rest = gt;  // g_1 ... g_t; g_t ... g_C
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, c, o), y = __shfl_down_sync(0xffffffffu, rest, o);
      if (lane >= o) c *= x;
      if (lane + o < 32) rest *= y;
    }
    double behind = __shfl_down_sync(0xffffffffu, rest, 1);  // g_(t + 1) ... g_C
    if (lane == 31) behind = 1.0;
    const double whole = __shfl_sync(0xffffffffu, c, 31);
    // row t of L (or, later, A), from s = t down
    auto rows = [&](bool of_a) {
      double dec = 1.0;
      __syncwarp();
#pragma unroll 4
      for (int s = kDcTokens - 1; s >= 0; --s) {
        const float rks = __shfl_sync(0xffffffffu, rk, s);
        const double gs1 = __shfl_sync(0xffffffffu, gt, min(s + 1, 31));
        if (s < t) dec *= gs1;
        sl[warp][t][s] = of_a ? (s <= t ? (float)(dec * qk[t][s] * rq * rks) : 0.f)
                              : (s < t ? (float)(beta * dec * kk[t][s] * rk * rks) : 0.f);
      }
      __syncwarp();
    };
    rows(false);
    // column `lane` of T: T_tj = -sum_(j <= s < t) L_ts T_sj; then of A T
    float col[kDcTokens];
    auto times_row = [&](int r, int n) {  // row r of what sl holds, its first n elements, times the column
      float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < n; s += 4) {
        const float4 l = *reinterpret_cast<const float4*>(&sl[warp][r][s]);
        x[0] = fmaf(l.x, col[s], x[0]);
        if (s + 1 < n) x[1] = fmaf(l.y, col[s + 1], x[1]);
        if (s + 2 < n) x[2] = fmaf(l.z, col[s + 2], x[2]);
        if (s + 3 < n) x[3] = fmaf(l.w, col[s + 3], x[3]);
      }
      return (x[0] + x[1]) + (x[2] + x[3]);
    };
#pragma unroll
    for (int r = 0; r < kDcTokens; ++r) {
      const float x = times_row(r, r);
      col[r] = r == lane ? 1.f : r < lane ? 0.f : -x;
    }
    float* mats = reinterpret_cast<float*>(a.scratch + ((size_t)blockIdx.x * a.H + h) * kDcBytes);
    float* row = mats + lane * 2 * kDcTokens;
    rows(true);
#pragma unroll
    for (int r = 0; r < kDcTokens; ++r) *reinterpret_cast<float2*>(row + dc_place(r)) = make_float2(col[r], times_row(r, r + 1));
    float* vec = mats + kDcMats;
    vec[t] = beta;
    vec[kDcTokens + t] = (float)(beta * c * rk);
    vec[2 * kDcTokens + t] = (float)(c * rq);
    vec[3 * kDcTokens + t] = (float)(behind * rk);
    if (t == 0) vec[4 * kDcTokens] = (float)whole;
    __syncwarp();
  }
}

// A block owns NV value columns of one (request, head): 2 NV KS threads.  In [K; Q] S a thread has 4 columns of 4 tokens' K and Q
// rows (tokens eight apart: eight lanes read eight rows, in different banks) over a KS-th of the key channels; the partial sums
// meet in shared memory, and each of the KS threads goes on with 4 / KS of the tokens.  In the update it keeps D / (8 KS) channels x
// 4 columns of the state in registers.
template <int D, int NV>
struct DcStage {
  __nv_bfloat16 k[kDcTokens * (D + 8)], q[kDcTokens * (D + 8)], v[kDcTokens * NV];
  float m[kDcMats];
  float vec[4 * kDcTokens + 4];
};
template <int D, int NV, int KS>
struct DcShared {
  DcStage<D, NV> stage[2];
  float s[D][NV];                // the state as the chunk finds it
  float part[KS][64][NV];        // partial sums
  float x[kDcTokens][NV], u[kDcTokens][NV];
};
__device__ __forceinline__ void dc_load4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <int N>
__device__ __forceinline__ void dc_words(const __nv_bfloat16* p, uint32_t (&w)[N]) {  // N = 1, 2 or 4 words, as aligned as that
  if constexpr (N == 1) {
    w[0] = *reinterpret_cast<const uint32_t*>(p);
  } else if constexpr (N == 2) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    w[0] = t.x; w[1] = t.y;
  } else {
    const uint4 t = *reinterpret_cast<const uint4*>(p);
    w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
  }
}

template <int D, int NV, int KS>
__global__ void __launch_bounds__(2 * NV * KS) delta_chunk_kernel(DeltaChunkArgs a) {
  pdl_wait();
  pdl_trigger();
  constexpr int kThreads = 2 * NV * KS, CG = NV / 4, NT = 4 / KS, DT = D / (8 * KS), LD = D + 8;
  extern __shared__ __align__(16) unsigned char dc_smem[];
  DcShared<D, NV, KS>& sh = *reinterpret_cast<DcShared<D, NV, KS>*>(dc_smem);
  const int h = blockIdx.y, col0 = blockIdx.z * NV;
  const int tid = threadIdx.x, lane = tid & 31;
  // the block's request: the blockIdx.x-th of those that go in chunks (every warp looks for it)
  int seg = -1, n_chunks = 0, before = 0, left = blockIdx.x;  // before: chunks of the requests in front of it
  for (int i0 = 0; i0 < a.n_segs && seg < 0; i0 += 32) {
    const int n = i0 + lane < a.n_segs ? dc_chunks(a, i0 + lane) : 0;
    const unsigned some = __ballot_sync(0xffffffffu, n > 0);
    const int at = left < __popc(some) ? (int)__fns(some, 0, left + 1) : 32;  // its lane
    left -= __popc(some);
    int sum = lane < at ? n : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    before += sum;
    if (at < 32) {
      seg = i0 + at;
      n_chunks = __shfl_sync(0xffffffffu, n, at);
    }
  }
  // (a table whose requests overlap, or more of them long than the caller said: chunks that no scratch was laid out for)
  if (seg < 0 || before + n_chunks > a.n_chunks) return;
  const int q_start = a.seg_info[seg * 4], q_len = a.seg_info[seg * 4 + 1], kv_len = a.seg_info[seg * 4 + 2];
  const int slot = a.state_slots[seg];
  if (slot < 0 || slot >= a.n_slots) return;
  const int hqk = h / (a.H / a.G);
  auto fetch = [&](int ch) {
    DcStage<D, NV>& st = sh.stage[ch & 1];
    const int t0 = ch * kDcTokens, nb = min(kDcTokens, q_len - t0);
    constexpr int per = D / 8;
    for (int i = tid; i < kDcTokens * per; i += kThreads) {
      const int t = i / per, d = i % per * 8;
      const bool in = t < nb;
      const size_t tok = (size_t)(q_start + t0 + (in ? t : 0));
      dc_cp16(st.k + t * LD + d, a.k + tok * a.k_stride + (size_t)hqk * D + d, in);
      dc_cp16(st.q + t * LD + d, a.q + tok * a.q_stride + (size_t)hqk * D + d, in);
    }
    for (int i = tid; i < kDcTokens * (NV / 8); i += kThreads) {
      const int t = i / (NV / 8), d = i % (NV / 8) * 8;
      const bool in = t < nb && col0 + d < a.Dv;
      const size_t tok = (size_t)(q_start + t0 + (in ? t : 0));
      dc_cp16(st.v + t * NV + d, a.v + tok * a.v_stride + (size_t)h * a.Dv + (in ? col0 + d : 0), in);
    }
    const unsigned char* src = a.scratch + ((size_t)(before + ch) * a.H + h) * kDcBytes;
    for (int i = tid; i < kDcMats / 4; i += kThreads) dc_cp16(st.m + 4 * i, src + (size_t)i * 16, true);
    for (int i = tid; i < kDcTokens + 1; i += kThreads) dc_cp16(st.vec + 4 * i, src + kDcMats * 4 + (size_t)i * 16, true);
    asm volatile("cp.async.commit_group;\n" ::);
  };
  fetch(0);
  const int c0 = tid % CG * 4, tg = tid / CG % 8, kr = tid / (8 * CG);
  const int dg = tid / CG * DT;  // the thread's channels of the state
  const bool live = col0 + c0 < a.Dv;  // (value channels come in multiples of 16)
  float* sta = a.state + (((size_t)slot * a.H + h) * a.Dv + (live ? col0 + c0 : 0)) * D + dg;
  const bool fresh = kv_len == q_len;
  float s[DT][4];
#pragma unroll
  for (int i = 0; i < DT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = !fresh && live ? sta[(size_t)j * D + i] : 0.f;
#pragma unroll 1
  for (int ch = 0; ch < n_chunks; ++ch) {
#pragma unroll
    for (int i = 0; i < DT; ++i) *reinterpret_cast<float4*>(&sh.s[dg + i][c0]) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // the chunk's rows have landed, the state lies in shared memory, the chunk before is through
    if (ch + 1 < n_chunks) fetch(ch + 1);
    const DcStage<D, NV>& st = sh.stage[ch & 1];
    {
      // [K; Q] S, a token's two rows as a pair
      uint64_t acc[4][4] = {};
      const __nv_bfloat16* kp = st.k + tg * LD + kr * (D / KS);
      const __nv_bfloat16* qp = st.q + tg * LD + kr * (D / KS);
      const float* sp = &sh.s[kr * (D / KS)][c0];
#pragma unroll 2
      for (int d0 = 0; d0 < D / KS; d0 += 8) {
        uint32_t kw[4][4], qw[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dc_words(kp + 8 * i * LD + d0, kw[i]);
          dc_words(qp + 8 * i * LD + d0, qw[i]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float y[4];
          dc_load4(sp + (d0 + e) * NV, y);
          uint64_t y2[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) y2[j] = f2_pair(y[j], y[j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t x = e & 1 ? f2_pair(bf2_high(kw[i][e >> 1]), bf2_high(qw[i][e >> 1])) : f2_pair(bf2_low(kw[i][e >> 1]), bf2_low(qw[i][e >> 1]));
#pragma unroll
            for (int j = 0; j < 4; ++j) f2_fma(acc[i][j], x, y2[j]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float k4[4], q4[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) f2_unpair(acc[i][j], k4[j], q4[j]);
        float* dst = &sh.part[kr][8 * tg + 2 * i][c0];
        *reinterpret_cast<float4*>(dst) = make_float4(k4[0], k4[1], k4[2], k4[3]);
        *reinterpret_cast<float4*>(dst + NV) = make_float4(q4[0], q4[1], q4[2], q4[3]);
      }
    }
    __syncthreads();
    // this thread's tokens from here on: tg + 8 (kr NT + i)
    uint64_t r[NT][4];
    const int place = 8 * tg + 2 * NT * kr;
    bool odd = false;  // an infinite or NaN X
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      float k4[4], q4[4];
      dc_load4(&sh.part[0][place + 2 * i][c0], k4);
      dc_load4(&sh.part[0][place + 2 * i + 1][c0], q4);
#pragma unroll
      for (int e = 1; e < KS; ++e) {
        float y[4], z[4];
        dc_load4(&sh.part[e][place + 2 * i][c0], y);
        dc_load4(&sh.part[e][place + 2 * i + 1][c0], z);
#pragma unroll
        for (int j = 0; j < 4; ++j) { k4[j] += y[j]; q4[j] += z[j]; }
      }
      const int t = tg + 8 * (kr * NT + i);
      const float be = st.vec[t], bs = st.vec[kDcTokens + t], os = st.vec[2 * kDcTokens + t];
      float v[4];
      Vec4<__nv_bfloat16>::load(st.v + t * NV + c0, v);
      const float4 xt = make_float4(fmaf(be, v[0], -bs * k4[0]), fmaf(be, v[1], -bs * k4[1]), fmaf(be, v[2], -bs * k4[2]), fmaf(be, v[3], -bs * k4[3]));
      *reinterpret_cast<float4*>(&sh.x[t][c0]) = xt;
      odd |= !(fabsf(xt.x) < INFINITY && fabsf(xt.y) < INFINITY && fabsf(xt.z) < INFINITY && fabsf(xt.w) < INFINITY);
#pragma unroll
      for (int j = 0; j < 4; ++j) r[i][j] = f2_pair(0.f, os * q4[j]);
    }
    odd = __syncthreads_or(odd);
    // [T; A T] X, again a token's two rows as a pair.  This thread's tokens all lie in front of 8 NT (kr + 1), and what a row has behind
    // its token is zero.  But zero times an infinity or NaN is NaN: with such an X in the chunk a row stops at its own token.
    auto term = [&](int e, bool to_own) {
      float y[4];
      dc_load4(&sh.x[e][c0], y);
      uint64_t x[NT];
#pragma unroll
      for (int i = 0; i < NT; i += 2) {
        if constexpr (NT == 1) {
          x[0] = *reinterpret_cast<const uint64_t*>(st.m + e * 2 * kDcTokens + place);
        } else {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(st.m + e * 2 * kDcTokens + place + 2 * i);
          x[i] = w.x; x[i + 1] = w.y;
        }
      }
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        if (to_own && e > tg + 8 * (kr * NT + i)) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) f2_fma(r[i][j], x[i], f2_pair(y[j], y[j]));
      }
    };
    const int upto = 8 * NT * (kr + 1);
    if (!odd) {
#pragma unroll 8
      for (int e = 0; e < upto; ++e) term(e, false);
    } else {
#pragma unroll 1
      for (int e = 0; e < upto; ++e) term(e, true);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = tg + 8 * (kr * NT + i), tok = ch * kDcTokens + t;
      float u[4], o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) f2_unpair(r[i][j], u[j], o[j]);
      const float ks = st.vec[3 * kDcTokens + t];
      *reinterpret_cast<float4*>(&sh.u[t][c0]) = make_float4(ks * u[0], ks * u[1], ks * u[2], ks * u[3]);
      if (live && tok < q_len)
        *reinterpret_cast<float4*>(a.out + ((size_t)(q_start + tok) * a.H + h) * a.Dv + col0 + c0) = make_float4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
    // S <- c_C S + K^T ((c_C / c) rk U), channels in pairs
    const float whole = st.vec[4 * kDcTokens];
    uint64_t add[DT / 2][4] = {};
#pragma unroll 8
    for (int e = 0; e < kDcTokens; ++e) {
      uint32_t w[DT / 2];
      float y[4];
      dc_words(st.k + e * LD + dg, w);
      dc_load4(&sh.u[e][c0], y);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t y2 = f2_pair(y[j], y[j]);
#pragma unroll
        for (int i = 0; i < DT / 2; ++i) f2_fma(add[i][j], f2_pair(bf2_low(w[i]), bf2_high(w[i])), y2);
      }
    }
#pragma unroll
    for (int i = 0; i < DT; i += 2)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x, y;
        f2_unpair(add[i / 2][j], x, y);
        s[i][j] = fmaf(whole, s[i][j], x);
        s[i + 1][j] = fmaf(whole, s[i + 1][j], y);
      }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < DT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sta[(size_t)j * D + i] = s[i][j];
  }
}

template <int D, int NV, int KS>
static int launch_delta_chunks_as(const DeltaChunkArgs& a, cudaStream_t s) {
  const dim3 grid(a.n_long, a.H, (a.Dv + NV - 1) / NV);
  const size_t smem = sizeof(DcShared<D, NV, KS>);
  static_assert(sizeof(DcShared<D, NV, KS>) <= 227 * 1024, "shared memory");
  auto kern = delta_chunk_kernel<D, NV, KS>;
  FTK_REQUIRE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess,
              "delta_scan (chunks): cannot set up the kernel");
  constexpr size_t sl = kDcTokens * (kDcTokens + 4) * sizeof(float);  // a warp's share of the triangles' shared memory
  if (a.H / a.G > 4) {
    auto prep = delta_prep_kernel<D, 8>;
    FTK_REQUIRE(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(8 * sl)) == cudaSuccess,
                "delta_scan (chunks): cannot set up the kernel");
    FTK_LAUNCH(prep, dim3(a.n_chunks, a.G), 256, 8 * sl, s, a);
  } else {
    FTK_LAUNCH((delta_prep_kernel<D, 4>), dim3(a.n_chunks, a.G), 128, 4 * sl, s, a);
  }
  FTK_LAUNCH_CHECK("delta_scan (chunks, triangles)");
  FTK_LAUNCH(kern, grid, 2 * NV * KS, smem, s, a);
  FTK_LAUNCH_CHECK("delta_scan (chunks)");
  return 0;
}

// Columns a block.  16, twelve warps' worth of 48 shared out over three blocks, while that leaves SMs without a third block; else
// 48 with twelve warps, three a scheduler.  Chunk kernel alone, 2,048 tokens of 128 key channels, 16 heads of 128 (128 blocks of
// 16 columns): 282 us, blocks of 48 columns 385; 48 heads (384 and 144 blocks): 435 and 387 us.  Blocks of 32 and 64 columns and
// other splits of the channels: 440 to 470 us at 48 heads.  (Token by token: 860 us at 48 heads, 538 at 16.)  48 divides neither 64
// nor 128: of 64 value columns a third of the second block's work is for nothing, and 48 heads with four requests of 256 tokens take
// 175 us against 162 token by token; such steps do not come here (parts/delta.py: chunks_pay).
template <int D>
static int launch_delta_chunks(const DeltaChunkArgs& a, cudaStream_t s) {
  const long long blocks = (long long)a.n_long * a.H * ((a.Dv + 15) / 16);
  return blocks > 2 * 148 ? launch_delta_chunks_as<D, 48, 4>(a, s) : launch_delta_chunks_as<D, 16, 4>(a, s);
}

}  // namespace ftk

using namespace ftk;

// Bytes of scratch for steps of n_tokens tokens of which n_segs requests go in chunks, or 0 where the sizes are not taken.
extern "C" long long ftk_delta_chunk_scratch(int dtype, int n_tokens, int n_segs, int n_heads, int n_kv_heads, int dim, int vdim) {
  if (dtype != FTK_BF16 || (dim != 64 && dim != 128) || vdim < 16 || vdim % 16 || vdim > 65535 * 16 || n_heads < 1 || n_heads > 65535 ||
      n_kv_heads < 1 || n_heads % n_kv_heads || n_tokens < 1 || n_segs < 1)
    return 0;
  return ((long long)n_tokens / kDcTokens + n_segs) * n_heads * kDcBytes;
}

extern "C" int ftk_delta_scan_chunks(const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                                     long long v_stride, const void* b, long long b_stride, const void* a, long long a_stride,
                                     int dtype, const float* a_log, const float* dt_bias, float q_scale, float unit_eps, float* state,
                                     int n_slots, const int32_t* state_slots, const int32_t* seg_info, int n_segs, float* out,
                                     int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim, int long_from, int n_long, void* scratch,
                                     long long scratch_bytes, void* stream) {
  FTK_REQUIRE(long_from >= 1 && n_long >= 1 && n_long <= n_segs, "delta_scan (chunks): %d of %d requests of %d tokens and more", n_long,
              n_segs, long_from);
  const long long need = ftk_delta_chunk_scratch(dtype, n_tokens, n_long, n_heads, n_kv_heads, dim, vdim);
  FTK_REQUIRE(need > 0, "delta_scan (chunks): type %d, heads of %d x %d, %d tokens are not taken", dtype, dim, vdim, n_tokens);
  FTK_REQUIRE(q && k && v && b && a && a_log && dt_bias && state && state_slots && seg_info && out && scratch,
              "delta_scan (chunks): null pointer");
  FTK_REQUIRE(scratch_bytes >= need, "delta_scan (chunks): %lld bytes of scratch, %lld needed", scratch_bytes, need);
  FTK_REQUIRE((q_stride | k_stride | v_stride) % 8 == 0 &&
                  (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch | (uintptr_t)out) & 15) == 0,
              "delta_scan (chunks): rows, outputs and scratch on 16-byte boundaries");
  DeltaChunkArgs d;
  d.q = (const __nv_bfloat16*)q; d.k = (const __nv_bfloat16*)k; d.v = (const __nv_bfloat16*)v;
  d.b = (const __nv_bfloat16*)b; d.a = (const __nv_bfloat16*)a;
  d.q_stride = q_stride; d.k_stride = k_stride; d.v_stride = v_stride; d.b_stride = b_stride; d.a_stride = a_stride;
  d.a_log = a_log; d.dt_bias = dt_bias; d.q_scale = q_scale; d.unit_eps = unit_eps;
  d.state = state; d.n_slots = n_slots; d.state_slots = state_slots; d.seg_info = seg_info; d.n_segs = n_segs;
  d.out = out; d.n_tokens = n_tokens; d.H = n_heads; d.G = n_kv_heads; d.D = dim; d.Dv = vdim;
  d.scratch = (unsigned char*)scratch;
  d.long_from = long_from; d.n_long = n_long; d.n_chunks = n_tokens / kDcTokens + n_long;
  if (n_long < n_segs) {
    const int rc = delta_scan_tokens(q, q_stride, k, k_stride, v, v_stride, b, b_stride, a, a_stride, nullptr, dtype, a_log, dt_bias, q_scale,
                                     unit_eps, state, n_slots, state_slots, seg_info, n_segs, out, n_tokens, n_heads, n_kv_heads, dim, vdim,
                                     long_from, stream);
    if (rc) return rc;
  }
  note_variant("delta rule: chunks of 32 tokens");
  return dim == 64 ? launch_delta_chunks<64>(d, (cudaStream_t)stream) : launch_delta_chunks<128>(d, (cudaStream_t)stream);
}
