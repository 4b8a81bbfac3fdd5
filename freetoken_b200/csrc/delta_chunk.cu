// The gated delta rule in chunks of 64 tokens, for portions of bfloat16 prompts with one decay a head (delta.cu runs everything else token
// by token).
//
// With S the state as 64 tokens find it, c_t = g_1 ... g_t and c_t / c_s the decays behind token s,
//   u_t = beta_t (v_t - c_t S^T k_t - sum_(s < t) (c_t / c_s) (k_s . k_t) u_s)
//   o_t = c_t S^T q_t + sum_(s <= t) (c_t / c_s) (k_s . q_t) u_s            S <- c_C S + sum_s (c_C / c_s) k_s u_s^T,
// so U = T X with X = beta (V - c K S), T = (I + L)^-1, L_ts = beta_t (c_t / c_s) (k_s . k_t), and O = c Q S + A T X.  T, A T and
// the factors of a token depend on the chunks alone: delta_prep_kernel makes them for all chunks side by side (the decays in 64
// bits: where a state lives for hundreds of tokens, their rounding is most of what a result is off), T from the inverses of
// its diagonal blocks of 16.  What is left to do in order (delta_chunk_kernel) is three products: [K; Q] S, [T; A T] X and K^T U.
// Decays are running products, never differences of logarithms.  The state is rounded once in 64 tokens.
//
// The three products run on tcgen05, in 32 bits: K and Q are bfloat16 as they lie, and S, T, X and U are taken apart into three
// bfloat16 numbers each, every piece rounded to the nearest, whose sum is the 32-bit one (exactly from 2^-110 up).  Of T X the six products
// that reach 2^-24 are taken.  The tensor core's accumulator cuts off instead of rounding, so the products of the leading pieces are
// chains of two steps, added up in registers; the other pieces' are 2^-8 smaller.  What is most of a sum where decays are strong goes
// through registers by itself: the diagonals of T and A T, and the newest token's share of the state.
//
// What bounds it: the chain of a chunk, product, registers, shared memory, product, which no other block can hide: an SM's
// tensor pipe is at work about a third of the time.  With 64 columns a block, 48 heads of 128 x 128: 5.2 us a chunk (product 0.8, registers 1.1,
// product 0.8, registers 0.7, product 0.5, registers 1.0, and what has gone through registers since); 16 columns a block, 16 heads: 2.9.
// 2,048 tokens of one request, prep and chunks together (token by token, 32-bit fmas on the CUDA cores in chunks of 32, now): 48 heads of
// 128 x 128 857, 431 and 234 us, 16 heads 529, 282 and 122; 16 heads of 64 x 64 493, 292 and 109.  Distance of outputs and states from 64
// bits (512 tokens, heads of 128; token by token, as fmas, now): 1.5e-7 and 1.3e-7, 1.3 and 0.95, 1.2 and 0.85; with decays near one 16
// and 21, 2.2 and 1.7, 1.6 and 1.3; of e^-12 1.1 and 0.91, 1.1 and 0.86, 1.0 and 0.80.
#include "tc_common.cuh"

namespace ftk {

// (delta.cu: the requests of fewer tokens than shorter_than, token by token)
int delta_scan_tokens(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride, const void* b,
                      long long b_stride, const void* a, long long a_stride, float* z, int dtype, const float* a_log, const float* dt_bias,
                      float q_scale, float unit_eps, float* state, int n_slots, const int32_t* state_slots, const int32_t* seg_info,
                      int n_segs, float* out, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim, int shorter_than, void* stream);

__device__ int g_delta_status[4];  // [0] first error code of a wait that ran out, [1] block; 0 = fine

constexpr int kDcTokens = 64;  // tokens of a chunk
constexpr float kDcMost = 3.38e38f;  // what bfloat16 reaches: larger numbers' first piece would be an infinity
// Scratch of 64 tokens: a key head's [K; Q] as the tensor core reads it (per 64 channels 128 rows of 128 bytes, swizzled), then a
// head's [T; A T] without their diagonals the same way (three pieces of 128 rows of 64 tokens), per token beta, beta c rk, c rq,
// (c_C / c) rk and A's diagonal, and c_C.
constexpr int kDcImage = 128 * 128;  // bytes of 128 rows
constexpr int kDcHeadBytes = 3 * kDcImage + 5 * kDcTokens * 4 + 16;
__host__ __device__ constexpr long long dc_row_bytes(int H, int G, int D) { return (long long)G * (D / 64) * kDcImage + (long long)H * kDcHeadBytes; }

struct DeltaChunkArgs {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; const __nv_bfloat16* b; const __nv_bfloat16* a;
  long long q_stride, k_stride, v_stride, b_stride, a_stride;
  const float* a_log; const float* dt_bias;
  float q_scale, unit_eps;
  float* state; int n_slots;
  const int32_t* state_slots; const int32_t* seg_info; int n_segs;
  float* out; int n_tokens, H, G, D, Dv;
  unsigned char* scratch; long long row_bytes;
  int long_from, n_chunks;  // requests of long_from tokens and more go in chunks; the rows (of 64 tokens) that scratch holds
  int first_req, n_req, row0, row1;  // of those requests this pass's, and which rows of each
};

// rows of 64 tokens of a segment; 0 for one that no pass takes
__device__ __forceinline__ int dc_chunks(const DeltaChunkArgs& a, int seg) {
  const int q_start = a.seg_info[seg * 4], q_len = a.seg_info[seg * 4 + 1], kv_len = a.seg_info[seg * 4 + 2];
  if (q_len < a.long_from || q_start < 0 || q_start + q_len > a.n_tokens || kv_len < q_len) return 0;
  return (q_len + kDcTokens - 1) / kDcTokens;
}

// Of those the pass's: `rows` of the `index`-th request that goes in chunks.
__device__ __forceinline__ int dc_pass_rows(const DeltaChunkArgs& a, int rows, int index) {
  return rows > 0 && index >= a.first_req && index < a.first_req + a.n_req ? max(0, min(rows, a.row1) - a.row0) : 0;
}

// Four warps a head, two heads a block: shared memory of one
constexpr int kDcBlock = 16, kDcBlocks = kDcTokens / kDcBlock, kDcLine = kDcTokens + 4;
struct DcTeam {
  float l[kDcTokens][kDcLine];  // L, then A, then A T (rows of tokens; blocks of 16 above the diagonal are not used)
  float t[kDcTokens][kDcLine];  // T
  double g[kDcTokens];          // a token's decay;
  double upto[kDcTokens], behind[kDcTokens];  // the decays of its 16 tokens up to and with it, and behind it (times 1 / |k|);
  double total[kDcBlocks];      // of all of each 16
  float beta[kDcTokens];
};
// (the image lies there until the dots are done; from a border of 1,024 bytes on)
template <int D>
constexpr size_t dc_prep_smem() { return 1024 + (D / 64 * kDcImage > 2 * (int)sizeof(DcTeam) ? D / 64 * kDcImage : 2 * sizeof(DcTeam)); }
__device__ __forceinline__ void dc_bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dc_stores_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }  // what they copy has been read

// One block per (64 tokens, key head): the dots of the rows once for all heads that share them, then four warps a head.  T and A T in
// blocks of 16 x 16, a warp a block, a lane a column and half of the rows: one piece of code of 130 fmas for all of their products.
// (A lane a column of 64 and everything
// unrolled: 117 us at 48 heads and 2,048 tokens, the instructions' fetches in the way; now 63.)
template <int D>
__global__ void __launch_bounds__(256, 2) delta_prep_kernel(DeltaChunkArgs a) {
  constexpr int kThreads = 256, kParts = D / 32;
  extern __shared__ unsigned char dyn_smem[];
  __shared__ float kk[kDcTokens][kDcTokens + 1], qk[kDcTokens][kDcTokens + 1], srk[kDcTokens], srq[kDcTokens];
  __shared__ int found[2], abort_flag;
  __shared__ uint64_t dots_done;
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_addr(dyn_smem) + 1023u) & ~1023u;
  unsigned char* prep_smem = dyn_smem + (base - smem_addr(dyn_smem));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&dots_done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_slot, kParts * kDcTokens);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();  // (once the block has its columns: delta_chunk_kernel's may take what is left and hold it until this kernel has ended)
  if (warp == 0) {  // which segment's this is
    if (lane == 0) found[0] = -1;
    __syncwarp();
    int before = 0, requests = 0;
    for (int i0 = 0; i0 < a.n_segs; i0 += 32) {
      const int all = i0 + lane < a.n_segs ? dc_chunks(a, i0 + lane) : 0;
      const unsigned some = __ballot_sync(0xffffffffu, all > 0);
      const int n = dc_pass_rows(a, all, requests + __popc(some & ((1u << lane) - 1u)));
      requests += __popc(some);
      int upto = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const int t = (int)blockIdx.x - before - (upto - n);
      if (t >= 0 && t < n) { found[0] = i0 + lane; found[1] = a.row0 + t; }
      before += __shfl_sync(0xffffffffu, upto, 31);
      if (before > (int)blockIdx.x) break;
    }
  }
  __syncthreads();
  const uint32_t tmem = tmem_slot;
  const int seg = found[0];
  if (seg < 0) {
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kParts * kDcTokens);
    return;
  }
  const int q_start = a.seg_info[seg * 4] + found[1] * kDcTokens, nb = min(kDcTokens, a.seg_info[seg * 4 + 1] - found[1] * kDcTokens);
  const int g = blockIdx.y, per = a.H / a.G;
  unsigned char* row = a.scratch + (size_t)blockIdx.x * a.row_bytes;
  for (int i = threadIdx.x; i < kDcTokens * (D / 8); i += kThreads) {
    const int t = i / (D / 8), d = i % (D / 8) * 8;
    const size_t tok = (size_t)(q_start + min(t, nb - 1));
    uint4 kv = *reinterpret_cast<const uint4*>(a.k + tok * a.k_stride + (size_t)g * D + d);
    uint4 qv = *reinterpret_cast<const uint4*>(a.q + tok * a.q_stride + (size_t)g * D + d);
    if (t >= nb) kv = qv = make_uint4(0u, 0u, 0u, 0u);
    unsigned char* im = prep_smem + d / 64 * kDcImage + t * 128 + ((((d >> 3) & 7) ^ (t & 7)) << 4);
    *reinterpret_cast<uint4*>(im) = kv;
    *reinterpret_cast<uint4*>(im + kDcTokens * 128) = qv;
  }
  fence_async_smem();
  __syncthreads();
  // k_t . k_s and q_t . k_s: [K; Q] K^T, chains of two steps in columns of their own
  if (warp == 0) {
    if (elect_one()) {
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const uint64_t rows = smem_desc(base + (k >> 2) * kDcImage) + 2 * (k & 3);
        tc_mma(tmem + (k >> 1) * kDcTokens, rows, rows, instr_desc(kDcTokens), k & 1);
      }
      tc_commit(&dots_done);
      if (blockIdx.z == 0)
        for (int d = 0; d < D / 64; ++d) dc_bulk_store(row + (size_t)(g * (D / 64) + d) * kDcImage, base + d * kDcImage, kDcImage);
    }
    __syncwarp();
  }
  for (int t0 = 8 * warp; t0 < kDcTokens; t0 += 64) {  // |q|^2, four lanes a token
    const int t = t0 + (lane >> 2);
    float s = 0.f;
    for (int d = 4 * (lane & 3); d < D; d += 16) {
      float v[4];
      Vec4<__nv_bfloat16>::load(
          reinterpret_cast<const __nv_bfloat16*>(prep_smem + d / 64 * kDcImage + (kDcTokens + t) * 128 + ((((d >> 3) & 7) ^ (t & 7)) << 4) + (d & 4) * 2), v);
      s += fmaf(v[0], v[0], v[1] * v[1]) + fmaf(v[2], v[2], v[3] * v[3]);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    // (rows that do not exist are zeros: with unit_eps = 0 they would have no unit vector)
    if ((lane & 3) == 0) srq[t] = t < nb ? rsqrtf(s + a.unit_eps) * a.q_scale : 0.f;
  }
  if (!mbar_wait(&dots_done, 0, &abort_flag)) {
    atomicCAS(&g_delta_status[0], 0, 506);
    abort_flag = 1;
  }
  __syncwarp();
  tc_fence_after();
  {
    const int t = (warp & 1) * 32 + lane;
    float (*dst)[kDcTokens + 1] = warp & 2 ? qk : kk;
#pragma unroll
    for (int c = 0; c < kDcTokens / 2; c += 8) {
      const int s0 = (warp >> 2) * (kDcTokens / 2) + c;
      float r[kParts][8];
#pragma unroll
      for (int m = 0; m < kParts; ++m) tmem_ld8_start(tmem + ((uint32_t)((warp & 3) * 32) << 16) + m * kDcTokens + s0, r[m]);
      tmem_ld8_finish(r);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float y = r[0][i] + r[1][i];
        if constexpr (kParts == 4) y += r[2][i] + r[3][i];
        dst[t][s0 + i] = y;
      }
    }
  }
  if (warp == 0) dc_stores_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kParts * kDcTokens);
  for (int t = threadIdx.x; t < kDcTokens; t += kThreads) srk[t] = t < nb ? rsqrtf(kk[t][t] + a.unit_eps) : 0.f;
  __syncthreads();
  // (the warps' blocks of the two teams lie the other way round: the longest chains on different schedulers)
  const int team = warp >> 2, j = team ? 3 - (warp & 3) : warp & 3, tt = threadIdx.x & 127, col = lane & 15, upper = lane >> 4;
  DcTeam& sh = reinterpret_cast<DcTeam*>(prep_smem)[team];
  auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory"); };
  const int hh = blockIdx.z * 2 + team;
  if (hh < per) {
    const int h = g * per + hh;
    unsigned char* image = row + (size_t)a.G * (D / 64) * kDcImage + (size_t)h * kDcHeadBytes;
    double upto = 1.0, rest = 1.0;
    if (tt < kDcTokens) {
      const size_t tok = (size_t)(q_start + min(tt, nb - 1));
      float beta = 0.f;
      double gt = 1.0;  // (tokens that do not exist add nothing and decay nothing)
      if (tt < nb) {
        const double z = (double)__bfloat162float(a.a[tok * a.a_stride + h]) + (double)a.dt_bias[h];
        beta = 1.f / (1.f + expf(-__bfloat162float(a.b[tok * a.b_stride + h])));
        gt = exp(-exp((double)a.a_log[h]) * (z > 0.0 ? z + log1p(exp(-z)) : log1p(exp(z))));
      }
      upto = rest = gt;
#pragma unroll
      for (int o = 1; o < kDcBlock; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, upto, o, kDcBlock), y = __shfl_down_sync(0xffffffffu, rest, o, kDcBlock);
        if (col >= o) upto *= x;
        if (col + o < kDcBlock) rest *= y;
      }
      rest = __shfl_down_sync(0xffffffffu, rest, 1, kDcBlock);
      if (col == kDcBlock - 1) { rest = 1.0; sh.total[tt / kDcBlock] = upto; }
      sh.g[tt] = gt;
      sh.upto[tt] = upto;
      sh.behind[tt] = rest * srk[tt];
      sh.beta[tt] = beta;
    }
    meet();
    if (tt < kDcTokens) {
      for (int m = 0; m < tt / kDcBlock; ++m) upto *= sh.total[m];
      for (int m = kDcBlocks - 1; m > tt / kDcBlock; --m) rest *= sh.total[m];
      float* vec = reinterpret_cast<float*>(image + 3 * kDcImage);
      vec[tt] = sh.beta[tt];
      vec[kDcTokens + tt] = (float)(sh.beta[tt] * upto * srk[tt]);
      vec[2 * kDcTokens + tt] = (float)(upto * srq[tt]);
      vec[3 * kDcTokens + tt] = (float)(rest * srk[tt]);
      if (tt == 0) vec[5 * kDcTokens] = (float)((sh.total[0] * sh.total[1]) * (sh.total[2] * sh.total[3]));
    }
    // L or A, 16 entries of a row a thread and turn
    auto fill = [&](bool of_a) {
      const int t = tt & (kDcTokens - 1), own = t / kDcBlock;
      const float (*dots)[kDcTokens + 1] = of_a ? qk : kk;
      const double left = of_a ? (double)srq[t] : (double)sh.beta[t] * srk[t];
#pragma unroll 1
      for (int m = tt / kDcTokens; m <= own; m += 2) {
        const bool here = m == own;
        double f = left;  // the row's factor; in its own 16 tokens times the decays so far, from the token on backwards
        if (!here) {
          f *= sh.upto[t];
          for (int x = m + 1; x < own; ++x) f *= sh.total[x];
        }
#pragma unroll
        for (int e = kDcBlock - 4; e >= 0; e -= 4) {
          float y[4];
#pragma unroll
          for (int i = 3; i >= 0; --i) {
            const int s = kDcBlock * m + e + i;
            if (here && s < t) f *= sh.g[s + 1];
            const double x = f * (here ? (double)srk[s] : sh.behind[s]) * (double)dots[t][s];
            y[i] = s < t || (of_a && s == t) ? (float)x : 0.f;
          }
          *reinterpret_cast<float4*>(&sh.l[t][kDcBlock * m + e]) = make_float4(y[0], y[1], y[2], y[3]);
        }
      }
    };
    fill(false);
    meet();
    // this lane's half of a block's rows (every other one: the two that a warp reads at a time lie in different banks) times a column;
    // `own`: only up to a row's own column
    auto block_times = [&](const float* rows0, const float (&x)[kDcBlock], bool own, float (&y)[kDcBlock / 2]) {
#pragma unroll
      for (int r = 0; r < kDcBlock / 2; ++r) {
        const float* l = rows0 + (2 * r + upper) * kDcLine;
        float z[2] = {0.f, 0.f};
#pragma unroll
        for (int s = 0; s < kDcBlock; s += 4) {
          const float4 w = *reinterpret_cast<const float4*>(l + s);
          const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (!own || s + i <= 2 * r + upper) z[i & 1] = fmaf(v[i], x[s + i], z[i & 1]);
        }
        y[r] += z[0] + z[1];
      }
    };
    auto column = [&](int k, int c, float (&x)[kDcBlock]) {  // of block (k, c) of T
#pragma unroll
      for (int s = 0; s < kDcBlock; ++s) x[s] = sh.t[kDcBlock * k + s][kDcBlock * c + col];
    };
    {
      // the block's inverse, column by column: T_tj = -sum_(j <= s < t) L_ts T_sj
      float x[kDcBlock];
#pragma unroll
      for (int r = 0; r < kDcBlock; ++r) {
        float z[2] = {0.f, 0.f};
#pragma unroll
        for (int s = 0; s < r; ++s) z[s & 1] = fmaf(sh.l[kDcBlock * j + r][kDcBlock * j + s], x[s], z[s & 1]);
        x[r] = r == col ? 1.f : r < col ? 0.f : -(z[0] + z[1]);
      }
#pragma unroll
      for (int r = 0; r < kDcBlock; ++r)
        if (r / (kDcBlock / 2) == upper) sh.t[kDcBlock * j + r][kDcBlock * j + col] = x[r];
    }
    meet();
    // the blocks below it: T_ij = -T_ii sum_(j <= k < i) L_ik T_kj
#pragma unroll 1
    for (int i = j + 1; i < kDcBlocks; ++i) {
      float x[kDcBlock], y[kDcBlock / 2] = {}, z[kDcBlock / 2] = {};
#pragma unroll 1
      for (int k = j; k < i; ++k) {
        column(k, j, x);
        block_times(&sh.l[kDcBlock * i][kDcBlock * k], x, false, y);
      }
#pragma unroll
      for (int r = 0; r < kDcBlock / 2; ++r) {
        const float other = __shfl_xor_sync(0xffffffffu, y[r], 16);
        x[2 * r] = upper ? other : y[r];
        x[2 * r + 1] = upper ? y[r] : other;
      }
      block_times(&sh.t[kDcBlock * i][kDcBlock * i], x, true, z);
#pragma unroll
      for (int r = 0; r < kDcBlock / 2; ++r) sh.t[kDcBlock * i + 2 * r + upper][kDcBlock * j + col] = -z[r];
      __syncwarp();
    }
    meet();
    fill(true);
    meet();
    // A T: the blocks (i, c) of this warp, their products (i - c + 1) shared out evenly
    float y[4][kDcBlock / 2] = {};
    const int mine[4] = {j == 0 ? 30 : j == 1 ? 20 : j == 2 ? 31 : 32, j == 0 ? 0 : j == 1 ? 10 : j == 2 ? 21 : 11, j == 3 ? 22 : -1, j == 3 ? 33 : -1};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (mine[m] < 0) continue;
      const int i = mine[m] / 10, c = mine[m] % 10;
      float x[kDcBlock];
#pragma unroll 1
      for (int k = c; k < i; ++k) {
        column(k, c, x);
        block_times(&sh.l[kDcBlock * i][kDcBlock * k], x, false, y[m]);
      }
      column(i, c, x);
      block_times(&sh.l[kDcBlock * i][kDcBlock * i], x, true, y[m]);
    }
    meet();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (mine[m] < 0) continue;
#pragma unroll
      for (int r = 0; r < kDcBlock / 2; ++r) sh.l[kDcBlock * (mine[m] / 10) + 2 * r + upper][kDcBlock * (mine[m] % 10) + col] = y[m][r];
    }
    meet();
    // [T; A T] as the tensor core reads it, eight columns of a row a thread and turn
#pragma unroll 2
    for (int e = tt; e < 2 * kDcTokens * 8; e += 128) {
      const int r = e >> 3, t = r & (kDcTokens - 1), c = (e & 7) * 8;
      const float* src = r < kDcTokens ? &sh.t[t][c] : &sh.l[t][c];
      uint4 w[3] = {};
      if (c / kDcBlock <= t / kDcBlock) {
        float v[8];
        Vec4<float>::load(src, reinterpret_cast<float (&)[4]>(v[0]));
        Vec4<float>::load(src + 4, reinterpret_cast<float (&)[4]>(v[4]));
        if (c == (t & ~7)) {  // the diagonals (T's are ones) go through registers
          float own = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (c + i != t) continue;
            own = v[i];
            v[i] = 0.f;
          }
          if (r != t) reinterpret_cast<float*>(image + 3 * kDcImage)[4 * kDcTokens + t] = own;
        }
        split3(v, w);
      }
#pragma unroll
      for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(image + m * kDcImage + r * 128 + (((e & 7) ^ (r & 7)) << 4)) = w[m];
    }
    if (blockIdx.z == 0 && warp == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
}

// shared memory of the chunk kernel, from a border of 1,024 bytes on
template <int NV>
struct DcPlace {
  static constexpr int kq = 0, t = kq + 4 * kDcImage;                // [K; Q] of two rows of chunks; the pieces of [T; A T]
  static constexpr int s = t + 3 * kDcImage;                         // the state's pieces: rows of key channels
  static constexpr int s_piece = NV == 64 ? kDcImage : 2 * NV;       // (64 columns fill the 128 bytes of a row, 16 columns' three pieces lie in one)
  static constexpr int x = s + (NV == 64 ? 3 : 1) * kDcImage;        // X's, then U's: rows of tokens
  static constexpr int x_piece = NV == 64 ? kDcImage / 2 : 2 * NV;
  static constexpr int o = x + (NV == 64 ? 3 : 1) * kDcImage / 2;    // X from K's rows to Q's, then outputs on their way: rows of tokens, in different banks
  static constexpr int o_row = NV * 4 + 16;
  static constexpr int bytes = o + kDcTokens * o_row;
};
__device__ __forceinline__ void dc_bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  mbar_expect_tx(bar, bytes);
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(smem_addr(bar)) : "memory");
}
// Whether one of them may be no number, or one that bfloat16 cannot reach (kDcMost, or a little less).
template <int N>
__device__ __forceinline__ bool dc_none(const float (&y)[N]) {
  uint64_t z = 0;
#pragma unroll
  for (int j = 0; j < N; j += 2) f2_fma(z, f2_mul(f2_pair(y[j], y[j + 1]), f2_pair(1.0079f, 1.0079f)), 0);  // (an infinity times zero is a NaN)
  float a, b;
  f2_unpair(z, a, b);
  return !(a + b == 0.f);
}

// Columns with an infinite or NaN number in the 64 tokens from token `first` on, once more, as delta.cu runs them (in pairs of tokens): an
// infinity taken apart into pieces is a NaN, and so is what has infinities of both signs, which depends on where they meet.  A warp takes a
// column: `state` [NV][D] holds them as the chunk finds them, and is left as it leaves them; outputs go out from a column's
// first such token on.
template <int D, int NV>
__device__ __noinline__ void dc_by_token(const DeltaChunkArgs& a, float* state, const int* first_odd, int first, int nb, int h, int col0) {
  constexpr int N = D / 32;
  const int lane = threadIdx.x & 31, hqk = h / (a.H / a.G);
  const float neg_rate = -expf(a.a_log[h]), bias = a.dt_bias[h];
  for (int c = threadIdx.x >> 5; c < NV; c += blockDim.x >> 5) {
    const int from = first_odd[c];
    if (from >= kDcTokens || col0 + c >= a.Dv) continue;
    float s[N];
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = state[c * D + lane + 32 * i];
    for (int t = 0; t < nb; t += 2) {
      const bool two = t + 1 < nb;  // (an odd last token's partner: zeros that decay nothing)
      float k[2][N], q[2][N], g[2], beta[2], v[2], kq[2], dot[6] = {};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const bool in = e == 0 || two;
        const size_t tok = (size_t)(first + t + (in ? e : 0));
#pragma unroll
        for (int i = 0; i < N; ++i) {
          k[e][i] = in ? __bfloat162float(a.k[tok * a.k_stride + (size_t)hqk * D + lane + 32 * i]) : 0.f;
          q[e][i] = in ? __bfloat162float(a.q[tok * a.q_stride + (size_t)hqk * D + lane + 32 * i]) : 0.f;
        }
        const float z = __bfloat162float(a.a[tok * a.a_stride + h]) + bias;
        g[e] = in ? expf(neg_rate * (z > 0.f ? z + log1pf(expf(-z)) : log1pf(expf(z)))) : 1.f;
        beta[e] = in ? 1.f / (1.f + expf(-__bfloat162float(a.b[tok * a.b_stride + h]))) : 0.f;
        v[e] = in ? __bfloat162float(a.v[tok * a.v_stride + (size_t)h * a.Dv + col0 + c]) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          dot[e] = fmaf(k[e][i], k[e][i], dot[e]);
          dot[2 + e] = fmaf(q[e][i], q[e][i], dot[2 + e]);
          kq[e] = i ? fmaf(q[e][i], k[e][i], kq[e]) : q[e][i] * k[e][i];
        }
        dot[4] = fmaf(k[0][i], k[1][i], dot[4]);
        dot[5] = fmaf(k[0][i], q[1][i], dot[5]);
      }
      float rk[2], rq[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        rk[e] = e == 0 || two ? rsqrtf(warp_sum(dot[e]) + a.unit_eps) : 0.f;
        rq[e] = e == 0 || two ? rsqrtf(warp_sum(dot[2 + e]) + a.unit_eps) * a.q_scale : 0.f;
        kq[e] = warp_sum(kq[e]) * rq[e] * rk[e];
      }
      const float kk = warp_sum(dot[4]) * rk[0] * rk[1], kqab = warp_sum(dot[5]) * rk[0] * rq[1];
      float r[2] = {0.f, 0.f}, p[2] = {0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          k[e][i] *= rk[e];
          r[e] = fmaf(s[i], k[e][i], r[e]);
          p[e] = fmaf(s[i], q[e][i] * rq[e], p[e]);
        }
        r[e] = warp_sum(r[e]);
        p[e] = warp_sum(p[e]);
      }
      const float ua = beta[0] * (v[0] - g[0] * r[0]);
      const float ub = two ? beta[1] * (v[1] - g[1] * fmaf(g[0], r[1], kk * ua)) : 0.f;
      const float gab = g[0] * g[1], wa = g[1] * ua;
#pragma unroll
      for (int i = 0; i < N; ++i) s[i] = fmaf(gab, s[i], two ? fmaf(wa, k[0][i], ub * k[1][i]) : wa * k[0][i]);
      if (lane < 2 && t + lane >= from && (lane == 0 || two)) {
        const float o = lane == 0 ? fmaf(g[0], p[0], kq[0] * ua) : fmaf(g[1], fmaf(g[0], p[1], kqab * ua), kq[1] * ub);
        a.out[((size_t)(first + t + lane) * a.H + h) * a.Dv + col0 + c] = o;
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) state[c * D + lane + 32 * i] = s[i];
  }
}

// A block owns NV value columns of one (request, head).  A thread has a row (a token of K, of Q; a key channel) and 8 or 16 of the
// columns.  Products, by one thread (columns of NV in tensor memory; each is read before the next is issued, so all use the same):
//   [K; Q] S      two 16-channel steps of the leading piece each in columns of their own (up to 4), the second and third piece (4, 5)
//   [T; A T] X    (without the diagonals) 32 tokens each of the leading pieces' product (0, 1), second order (2), third (3)
//   K^T U         the same
template <int NV>
constexpr int dc_threads() { return NV == 64 ? 512 : 256; }
template <int D, int NV>
__global__ void __launch_bounds__(dc_threads<NV>()) delta_chunk_kernel(const __grid_constant__ DeltaChunkArgs a) {
  constexpr int NH = NV * 128 / dc_threads<NV>(), NG = NH / 8;  // columns a thread, eights of them
  using At = DcPlace<NV>;
  extern __shared__ unsigned char dc_smem[];
  __shared__ uint64_t kq_full[2], t_full, mma_done;
  __shared__ uint32_t tmem_slot;
  __shared__ float newest[NV];
  __shared__ int abort_flag, odd_flag[2], first_odd[NV];  // the first token that has no number, per column
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, share = warp >> 2;
  const uint32_t base = (smem_addr(dc_smem) + 1023u) & ~1023u;
  unsigned char* tiles = dc_smem + (base - smem_addr(dc_smem));
  if (tid == 0) {
    mbar_init(&kq_full[0], 1);
    mbar_init(&kq_full[1], 1);
    mbar_init(&t_full, 1);
    mbar_init(&mma_done, 1);
    abort_flag = odd_flag[0] = odd_flag[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < NV) first_odd[tid] = kDcTokens;
  if (warp == 0) tmem_alloc(&tmem_slot, NV == 64 ? 512 : 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot, my_tmem = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(share * NH);
  const int h = blockIdx.y, col0 = blockIdx.z * NV + share * NH;
  // the block's request: the blockIdx.x-th of the pass's (every warp looks for it)
  int seg = -1, n_chunks = 0, before = 0, left = a.first_req + blockIdx.x, requests = 0;  // before: rows of the requests in front of it
  for (int i0 = 0; i0 < a.n_segs && seg < 0; i0 += 32) {
    const int all = i0 + lane < a.n_segs ? dc_chunks(a, i0 + lane) : 0;
    const unsigned some = __ballot_sync(0xffffffffu, all > 0);
    const int n = dc_pass_rows(a, all, requests + __popc(some & ((1u << lane) - 1u)));
    const int at = left < __popc(some) ? (int)__fns(some, 0, left + 1) : 32;  // its lane
    left -= __popc(some);
    requests += __popc(some);
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
  if (seg < 0 || before + n_chunks > a.n_chunks) n_chunks = 0;
  const int slot = n_chunks ? a.state_slots[seg] : -1;
  if (slot < 0 || slot >= a.n_slots) n_chunks = 0;
  if (n_chunks) {
    // (of the request's tokens those that no pass before has taken; what they left in the slot goes on)
    const int q_start = a.seg_info[seg * 4] + a.row0 * kDcTokens, q_len = a.seg_info[seg * 4 + 1] - a.row0 * kDcTokens;
    const bool fresh = a.row0 == 0 && a.seg_info[seg * 4 + 2] == a.seg_info[seg * 4 + 1];
    const unsigned char* rows = a.scratch + (size_t)before * a.row_bytes;
    const unsigned char* kq_src = rows + (size_t)(h / (a.H / a.G)) * (D / 64) * kDcImage;
    const unsigned char* head_src = rows + (size_t)a.G * (D / 64) * kDcImage + (size_t)h * kDcHeadBytes;
    auto load_kq = [&](int ch) {
      dc_bulk_load(base + At::kq + (ch & 1) * 2 * kDcImage, kq_src + (size_t)ch * a.row_bytes, D / 64 * kDcImage, &kq_full[ch & 1]);
    };
    auto load_t = [&](int ch) { dc_bulk_load(base + At::t, head_src + (size_t)ch * a.row_bytes, 3 * kDcImage, &t_full); };
    int kq_issued = 0, t_issued = 0, kq_seen = 0, t_seen = 0;  // (thread 0)
    if (tid == 0) {
      load_kq(0);
      load_t(0);
      kq_issued = t_issued = 1;
      if (n_chunks > 1) { load_kq(1); kq_issued = 2; }
    }
    const int row = quad * 32 + lane, t = row & (kDcTokens - 1);  // (rows 0 to 63: K's tokens, then Q's)
    const bool of_k = quad < 2, channel = row < D;
    // what a token's row needs beside the products, a chunk ahead: its values, beta and factors
    uint4 v_next[NG];
    float f_next[3], whole_next;
    auto fetch = [&](int ch) {
      const float* vec = reinterpret_cast<const float*>(head_src + (size_t)ch * a.row_bytes + 3 * kDcImage);
      whole_next = vec[5 * kDcTokens];
      if (of_k) {
        const bool in = ch * kDcTokens + t < q_len;
        const __nv_bfloat16* src = a.v + (size_t)(q_start + (in ? ch * kDcTokens + t : 0)) * a.v_stride + (size_t)h * a.Dv;
#pragma unroll
        for (int i = 0; i < NG; ++i)
          v_next[i] = in && col0 + 8 * i < a.Dv ? *reinterpret_cast<const uint4*>(src + col0 + 8 * i) : make_uint4(0u, 0u, 0u, 0u);
        f_next[0] = vec[t];
        f_next[1] = vec[kDcTokens + t];
        f_next[2] = vec[3 * kDcTokens + t];
      } else {
        f_next[0] = vec[2 * kDcTokens + t];
        f_next[1] = vec[4 * kDcTokens + t];
      }
    };
    fetch(0);
    float* sta = a.state + (((size_t)slot * a.H + h) * a.Dv + col0) * D + row;
    float s[NH];
#pragma unroll
    for (int j = 0; j < NH; ++j) s[j] = channel && !fresh && col0 + j < a.Dv ? sta[(size_t)j * D] : 0.f;
    // eight columns as three pieces into row `r` of an operand
    auto put = [&](int at, int piece, int r, int i, const float (&x)[8]) {
      uint4 w[3];
      split3(x, w);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const int g8 = share * NG + i;
        const int off = NV == 64 ? m * piece + ((g8 ^ (r & 7)) << 4) : (((m * NV / 8 + g8) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(tiles + at + r * 128 + off) = w[m];
      }
    };
    uint32_t phase = 0;
    bool bad = false;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      if (bad) return;
      if (!mbar_wait(bar, parity, &abort_flag)) {
        atomicCAS(&g_delta_status[0], 0, code);
        abort_flag = 1;
        bad = true;
      }
    };
    constexpr uint32_t id1 = instr_desc(NV) | kMnMajorB, id2 = instr_desc(2 * NV) | kMnMajorB;
#pragma unroll 1
    for (int ch = 0; ch < n_chunks; ++ch) {
      const uint32_t kq = base + At::kq + (ch & 1) * 2 * kDcImage;
      if (channel) {
#pragma unroll
        for (int i = 0; i < NG; ++i) put(At::s, At::s_piece, row, i, reinterpret_cast<const float (&)[8]>(s[8 * i]));
      }
      fence_async_smem();
      tc_fence_before();
      if (__syncthreads_or(bad)) break;
      if (warp == 0) {
        wait(&kq_full[ch & 1], (uint32_t)(ch >> 1) & 1u, 501);
        ++kq_seen;
        tc_fence_after();
        __syncwarp();
        if (elect_one()) {
          odd_flag[(ch + 1) & 1] = 0;
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint64_t ad = smem_desc(kq + (k >> 2) * kDcImage) + 2 * (k & 3);
            const uint32_t bs = base + At::s + k * 2048;
            tc_mma(tmem + (k >> 1) * NV, ad, smem_desc_mn(bs, kDcImage), id1, k & 1);
            tc_mma(tmem + 4 * NV, ad, smem_desc_mn(bs + At::s_piece, kDcImage), id2, k != 0);
          }
          tc_commit(&mma_done);
        }
        __syncwarp();
      }
      uint4 v[NG];
      const float f0 = f_next[0], f1 = f_next[1], f2 = f_next[2], whole = whole_next;
#pragma unroll
      for (int i = 0; i < NG; ++i) v[i] = v_next[i];
      if (ch + 1 < n_chunks) fetch(ch + 1);
      wait(&mma_done, phase, 502);
      phase ^= 1;
      __syncwarp();
      tc_fence_after();
      float o[NH];  // K's rows: X, which T's ones on the diagonal pass on; Q's: what the state gives, and X times A's diagonal
      // What a row of T and A T has behind its token is zero, but zero times an infinity or NaN is NaN: such an X (or one that bfloat16
      // cannot reach) goes into the product as zero, and its column token by token from there on.
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        constexpr int kParts = D / 32;
        float r[kParts + 2][8], y[8];
#pragma unroll
        for (int m = 0; m < kParts; ++m) tmem_ld8_start(my_tmem + m * NV + 8 * i, r[m]);
        tmem_ld8_start(my_tmem + 4 * NV + 8 * i, r[kParts]);
        tmem_ld8_start(my_tmem + 5 * NV + 8 * i, r[kParts + 1]);
        tmem_ld8_finish(r);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          y[j] = r[0][j] + r[1][j];
          if constexpr (kParts == 4) y[j] += r[2][j] + r[3][j];
          y[j] += r[kParts][j] + r[kParts + 1][j];
        }
        if (of_k) {
          const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
          for (int j = 0; j < 8; ++j) y[j] = fmaf(f0, j & 1 ? bf2_high(w[j >> 1]) : bf2_low(w[j >> 1]), -f1 * y[j]);
          if (dc_none<8>(y)) {
            odd_flag[ch & 1] = 1;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (fabsf(y[j]) < kDcMost) continue;
              atomicMin(&first_odd[share * NH + 8 * i + j], t);
              y[j] = 0.f;
            }
          }
          put(At::x, At::x_piece, row, i, y);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[8 * i + j] = y[j];
#pragma unroll
          for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(tiles + At::o + t * At::o_row + (share * NH + 8 * i + j) * 4) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) o[8 * i + j] = f0 * y[j];
        }
      }
      fence_async_smem();
      tc_fence_before();
      if (__syncthreads_or(bad)) break;
      if (warp == 0) {
        wait(&t_full, (uint32_t)ch & 1u, 503);
        ++t_seen;
        tc_fence_after();
        __syncwarp();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t t1 = smem_desc(base + At::t) + 2 * k, t2 = smem_desc(base + At::t + kDcImage) + 2 * k,
                           t3 = smem_desc(base + At::t + 2 * kDcImage) + 2 * k;
            const uint64_t x1 = smem_desc_mn(base + At::x + k * 2048, kDcImage / 2), x2 = smem_desc_mn(base + At::x + k * 2048 + At::x_piece, kDcImage / 2);
            tc_mma(tmem + (k >> 1) * NV, t1, x1, id1, k & 1);
            tc_mma(tmem + 2 * NV, t1, x2, id2, k != 0);
            tc_mma(tmem + 2 * NV, t2, x1, id2, 1);
            tc_mma(tmem + 3 * NV, t3, x1, id1, 1);
          }
          tc_commit(&mma_done);
        }
        __syncwarp();
      }
      if (!of_k) {
#pragma unroll
        for (int j = 0; j < NH; j += 4) {
          const float4 x = *reinterpret_cast<const float4*>(tiles + At::o + t * At::o_row + (share * NH + j) * 4);
          o[j] = fmaf(f1, x.x, o[j]); o[j + 1] = fmaf(f1, x.y, o[j + 1]); o[j + 2] = fmaf(f1, x.z, o[j + 2]); o[j + 3] = fmaf(f1, x.w, o[j + 3]);
        }
      }
      float u[NH];
      wait(&mma_done, phase, 504);
      phase ^= 1;
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        float r[4][8];
#pragma unroll
        for (int m = 0; m < 4; ++m) tmem_ld8_start(my_tmem + m * NV + 8 * i, r[m]);
        tmem_ld8_finish(r);
#pragma unroll
        for (int j = 0; j < 8; ++j) u[8 * i + j] = (r[0][j] + r[1][j]) + (r[2][j] + r[3][j]);
      }
#pragma unroll
      for (int j = 0; j < NH; ++j) u[j] += o[j];
      if (dc_none<NH>(u)) {
        odd_flag[ch & 1] = 1;
#pragma unroll
        for (int j = 0; j < NH; ++j)
          if (!(fabsf(u[j]) < kDcMost)) atomicMin(&first_odd[share * NH + j], t);
      }
      if (tid == 0 && ch + 1 < n_chunks && !bad) {
        load_t(ch + 1);
        ++t_issued;
      }
      const int last = min(kDcTokens, q_len - ch * kDcTokens) - 1;  // the newest token: the largest share of the state where decays are strong
      const float k_last = channel ? __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(
          tiles + At::kq + (ch & 1) * 2 * kDcImage + (row >> 6) * kDcImage + last * 128 + ((((row >> 3) & 7) ^ (last & 7)) << 4) + (row & 7) * 2)) : 0.f;
      if (of_k) {
#pragma unroll
        for (int j = 0; j < NH; ++j) {
          u[j] *= f2;
          if (t == last) {
            newest[share * NH + j] = u[j];
            u[j] = 0.f;
          }
        }
#pragma unroll
        for (int i = 0; i < NG; ++i) put(At::x, At::x_piece, row, i, reinterpret_cast<const float (&)[8]>(u[8 * i]));
      }
      fence_async_smem();
      tc_fence_before();
      if (__syncthreads_or(bad)) break;
      const bool some_odd = odd_flag[ch & 1] != 0;
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t kt = smem_desc_mn(kq + k * 2048, kDcImage);
            tc_mma(tmem + (k >> 1) * NV, kt, smem_desc_mn(base + At::x + k * 2048, kDcImage / 2), id1 | kMnMajorA, k & 1);
            tc_mma(tmem + 2 * NV, kt, smem_desc_mn(base + At::x + k * 2048 + At::x_piece, kDcImage / 2), id2 | kMnMajorA, k != 0);
          }
          tc_commit(&mma_done);
        }
        __syncwarp();
      }
      if (!of_k) {
        const int tok0 = ch * kDcTokens;
        float* dst = a.out + ((size_t)(q_start + tok0) * a.H + h) * a.Dv + (int)blockIdx.z * NV;
        const size_t stride = (size_t)a.H * a.Dv;
        if constexpr (NV == 64) {  // through shared memory: whole rows of 64 columns, 16 threads a row
          const int me = share * 64 + t, c = me % 16 * 4;
#pragma unroll
          for (int j = 0; j < NH; j += 4)
            *reinterpret_cast<float4*>(tiles + At::o + t * At::o_row + (share * NH + j) * 4) = make_float4(u[j], u[j + 1], u[j + 2], u[j + 3]);
          asm volatile("bar.sync 1, %0;" ::"n"(dc_threads<NV>() / 2) : "memory");
          if ((int)blockIdx.z * NV + c < a.Dv) {
#pragma unroll
            for (int r = me / 16; r < kDcTokens; r += dc_threads<NV>() / 32)
              if (tok0 + r < q_len) *reinterpret_cast<float4*>(dst + r * stride + c) = *reinterpret_cast<const float4*>(tiles + At::o + r * At::o_row + c * 4);
          }
        } else if (tok0 + t < q_len) {
#pragma unroll
          for (int j = 0; j < NH; j += 4)
            if (col0 + j < a.Dv)
              *reinterpret_cast<float4*>(dst + t * stride + share * NH + j) = make_float4(u[j], u[j + 1], u[j + 2], u[j + 3]);
        }
      }
      wait(&mma_done, phase, 505);
      phase ^= 1;
      __syncwarp();
      tc_fence_after();
      if (tid == 0 && ch + 2 < n_chunks && !bad) {
        load_kq(ch + 2);
        ++kq_issued;
      }
      if (some_odd) {  // (the state as the chunk found it, where its pieces were)
        float* found = reinterpret_cast<float*>(tiles + At::s);
        if (channel) {
#pragma unroll
          for (int j = 0; j < NH; ++j) found[(share * NH + j) * D + row] = s[j];
        }
        __syncthreads();
        dc_by_token<D, NV>(a, found, first_odd, q_start + ch * kDcTokens, min(kDcTokens, q_len - ch * kDcTokens), h, (int)blockIdx.z * NV);
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        float r[4][8];
#pragma unroll
        for (int m = 0; m < 4; ++m) tmem_ld8_start(my_tmem + m * NV + 8 * i, r[m]);
        tmem_ld8_finish(r);
        if (channel) {
#pragma unroll
          for (int j = 0; j < 8; ++j) s[8 * i + j] = fmaf(k_last, newest[share * NH + 8 * i + j], fmaf(whole, s[8 * i + j], (r[0][j] + r[1][j]) + (r[2][j] + r[3][j])));
        }
      }
      if (some_odd) {
        const float* found = reinterpret_cast<const float*>(tiles + At::s);
        if (channel) {
#pragma unroll
          for (int j = 0; j < NH; ++j)
            if (first_odd[share * NH + j] < kDcTokens) s[j] = found[(share * NH + j) * D + row];
        }
        __syncthreads();
        if (tid < NV) first_odd[tid] = kDcTokens;
      }
    }
    if (tid == 0 && abort_flag) {  // copies still in flight
      g_delta_status[1] = blockIdx.x;
      abort_flag = 0;
      for (; kq_seen < kq_issued; ++kq_seen) mbar_wait(&kq_full[kq_seen & 1], (uint32_t)(kq_seen >> 1) & 1u, &abort_flag);
      for (; t_seen < t_issued; ++t_seen) mbar_wait(&t_full, (uint32_t)t_seen & 1u, &abort_flag);
    }
    if (channel && !bad) {
#pragma unroll
      for (int j = 0; j < NH; ++j)
        if (col0 + j < a.Dv) sta[(size_t)j * D] = s[j];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, NV == 64 ? 512 : 128);
}

template <int D, int NV>
static int launch_delta_chunks_as(const DeltaChunkArgs& a, cudaStream_t s) {
  auto prep = delta_prep_kernel<D>;
  auto kern = delta_chunk_kernel<D, NV>;
  constexpr int prep_smem = (int)dc_prep_smem<D>(), smem = DcPlace<NV>::bytes + 1024;
  static_assert(smem <= 227 * 1024 && NV * D * 4 <= (NV == 64 ? 3 : 1) * kDcImage, "shared memory, and room for the state where its pieces lie");
  FTK_REQUIRE(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem) == cudaSuccess &&
                  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess,
              "delta_scan (chunks): cannot set up the kernels");
  FTK_LAUNCH(prep, dim3(a.n_chunks, a.G, (a.H / a.G + 1) / 2), 256, prep_smem, s, a);
  FTK_LAUNCH_CHECK("delta_scan (chunks, triangles)");
  FTK_LAUNCH(kern, dim3(a.n_req, a.H, (a.Dv + NV - 1) / NV), dc_threads<NV>(), smem, s, a);
  FTK_LAUNCH_CHECK("delta_scan (chunks)");
  return 0;
}

// Columns a block: by the rounds of blocks over the SMs and what a chunk takes, 3.0 us with 16 columns, 5.0 with 64 (and 3 more
// a block).  16 heads of 128 columns, 2,048 tokens: 123 us with 16 (128 blocks); 48 heads 228 with 64 (96 blocks), three rounds with 16.
template <int D>
static int launch_delta_chunks(const DeltaChunkArgs& a, int tokens, cudaStream_t s) {  // tokens: of the pass, about
  const long long pairs = max(1, tokens / kDcTokens / a.n_req);  // (of a request, about)
  auto rounds = [&](int cols) { return ((long long)a.n_req * a.H * ((a.Dv + cols - 1) / cols) + 147) / 148; };
  return rounds(64) * (3 + 5 * pairs) < rounds(16) * 3 * pairs ? launch_delta_chunks_as<D, 64>(a, s) : launch_delta_chunks_as<D, 16>(a, s);
}

int delta_chunk_status(int* out) { return take_status(g_delta_status, out); }  // (merged into ftk_read_status)
int delta_chunk_set_status(int code) { return set_status(g_delta_status, code); }

}  // namespace ftk

using namespace ftk;

// Bytes of scratch for steps of n_tokens tokens of which n_segs requests go in chunks, or 0 where the sizes are not taken.
extern "C" long long ftk_delta_chunk_scratch(int dtype, int n_tokens, int n_segs, int n_heads, int n_kv_heads, int dim, int vdim) {
  if (dtype != FTK_BF16 || (dim != 64 && dim != 128) || vdim < 16 || vdim % 16 || vdim > 65535 * 16 || n_heads < 1 || n_heads > 65535 ||
      n_kv_heads < 1 || n_heads % n_kv_heads || n_tokens < 1 || n_segs < 1)
    return 0;
  return ((long long)n_tokens / kDcTokens + n_segs) * dc_row_bytes(n_heads, n_kv_heads, dim);
}

extern "C" int ftk_delta_scan_chunks(const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                                     long long v_stride, const void* b, long long b_stride, const void* a, long long a_stride,
                                     int dtype, const float* a_log, const float* dt_bias, float q_scale, float unit_eps, float* state,
                                     int n_slots, const int32_t* state_slots, const int32_t* seg_info, int n_segs, float* out,
                                     int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim, int long_from, int n_long,
                                     const int32_t* passes, int n_passes, void* scratch, long long scratch_bytes, void* stream) {
  FTK_REQUIRE(long_from >= 1 && n_long >= 1 && n_long <= n_segs, "delta_scan (chunks): %d of %d requests of %d tokens and more", n_long,
              n_segs, long_from);
  const long long need = ftk_delta_chunk_scratch(dtype, n_tokens, n_long, n_heads, n_kv_heads, dim, vdim);
  FTK_REQUIRE(need > 0, "delta_scan (chunks): type %d, heads of %d x %d, %d tokens are not taken", dtype, dim, vdim, n_tokens);
  FTK_REQUIRE(q && k && v && b && a && a_log && dt_bias && state && state_slots && seg_info && out && scratch,
              "delta_scan (chunks): null pointer");
  const long long row_bytes = dc_row_bytes(n_heads, n_kv_heads, dim);
  if (!passes) {  // one, of all rows
    n_passes = 1;
    FTK_REQUIRE(scratch_bytes >= need, "delta_scan (chunks): %lld bytes of scratch, %lld needed", scratch_bytes, need);
  }
  FTK_REQUIRE(n_passes >= 1, "delta_scan (chunks): no pass");
  for (int i = 0; passes && i < n_passes; ++i) {
    const int32_t* p = passes + 5 * i;
    FTK_REQUIRE(p[0] >= 0 && p[1] >= 1 && p[1] <= n_long - p[0] && p[2] >= 0 && p[3] > p[2] && p[4] >= 1 && p[4] * row_bytes <= scratch_bytes,
                "delta_scan (chunks): a pass of %d rows (%d to %d of %d requests from the %d-th on)", p[4], p[2], p[3], p[1], p[0]);
  }
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
  d.scratch = (unsigned char*)scratch; d.row_bytes = row_bytes;
  d.long_from = long_from;
  if (n_long < n_segs) {
    const int rc = delta_scan_tokens(q, q_stride, k, k_stride, v, v_stride, b, b_stride, a, a_stride, nullptr, dtype, a_log, dt_bias, q_scale,
                                     unit_eps, state, n_slots, state_slots, seg_info, n_segs, out, n_tokens, n_heads, n_kv_heads, dim, vdim,
                                     long_from, stream);
    if (rc) return rc;
  }
  note_variant("delta rule: chunks of 64 tokens, tcgen05");
  for (int i = 0; i < n_passes; ++i) {
    const int32_t whole[5] = {0, n_long, 0, 0x7fffffff, n_tokens / kDcTokens + n_long};
    const int32_t* p = passes ? passes + 5 * i : whole;
    const int tokens = passes ? p[4] * kDcTokens : n_tokens;
    d.first_req = p[0]; d.n_req = p[1]; d.row0 = p[2]; d.row1 = p[3]; d.n_chunks = p[4];
    const int rc = dim == 64 ? launch_delta_chunks<64>(d, tokens, (cudaStream_t)stream) : launch_delta_chunks<128>(d, tokens, (cudaStream_t)stream);
    if (rc) return rc;
  }
  return 0;
}
