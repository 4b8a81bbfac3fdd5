// Gated linear attention over portions of several chunks, chunks of at most 64 tokens as products (bfloat16 rows, 64 or 128 key
// channels, 64 to 128 value channels).  Included by recurrent.cu after GlaArgs and its helpers; everything else runs the
// recurrence token by token there.
//
// With a_r the decays (per key channel) and S the state a chunk starts from:
//   o_t = (q_t prod_(r <= t) a_r) S + sum_(s <= t) P_ts v_s,      P_ts = sum_d q_t[d] k_s[d] prod_(s < r <= t) a_r[d]
//   S <- (prod a_r) S + sum_s (k_s prod_(r > s) a_r) v_s^T
// so a chunk's contribution to the state and its outputs are matrix products of 64 rows.  P is where decays per channel bite: a
// factor 1 / prod a_r could leave the 32-bit range.  So the decays between s and t are split at borders of 4 and of 16 tokens
// into factors that are all products of decays (at most 1): keys decayed to the end of their group, queries from the start of
// theirs, and the groups between them.
//   gla_local_kernel   a block a (chunk, head): decays, P, the chunk's contribution L and its decay product; P goes to where the
//                      outputs will lie (a row's first 64 columns), the decayed queries to where the decay logits lay
//   gla_walk_kernel    a thread a state element: S_(c+1) = P_c S_c + L_c over a request's chunks, the start states to where the
//                      contributions lay, the final state to the slot
//   gla_out_kernel     a block a (chunk, head): [decayed q | P] [S; V]
// P's sums are 32-bit fmas on the CUDA cores (two at a time, fma.rn.f32x2); the contributions and the outputs run on tcgen05 with
// 32-bit operands taken apart into three bfloat16 numbers each (split3).  What is most of a sum where decays are strong goes through
// registers: the two newest tokens of a contribution, an output's own token.  The decays are products of at most 9 factors instead of a
// running product.
//
// 48 heads of 128 x 128, 2,048 tokens, a decay per channel, cold caches: contributions 212 us, carry 48 and outputs 130 with all products
// as 32-bit fmas, 174, 48 and 90 now, 318 in a row (one decay a head 284; 16 heads 118 and 94; token by token 226, 99 and 359 with their
// waits).  The layer 973 -> 690 -> 634 us.  Outputs and states against 64 bits (1,024 tokens; as fmas, now): 1.4e-7 and 0.98e-7, 1.2 and
// 0.85; where the decays are close to 1 2.8 and 2.0, 1.8 and 1.5; with decays of e^-6 a token, where a result is one token's product,
// 0.89 and 0.25, 0.86 and 0.25; with one decay of 0.88 for all channels 1.05 and 0.60, 1.04 and 0.62.
#pragma once
#include "tc_common.cuh"

namespace ftk {

__device__ int g_gla_status[4];  // [0] first error code of a wait that ran out, [1] block; 0 = fine
constexpr int kGcTokens = 64, kGcBlock = 16, kGcBlocks = kGcTokens / kGcBlock;

// hi + lo <- (hi + lo) (x + xlo): products of given decays are kept in two words until they are used.  (The same decay at every
// token would otherwise leave the same error at every step, 64 times a chunk.  Decays from logits are summed up as logarithms.)
__device__ __forceinline__ void gc_times(float& hi, float& lo, float x, float xlo) {
  const float p = hi * x;
  lo = fmaf(lo, x, fmaf(hi, xlo, fmaf(hi, x, -p)));
  hi = p;
}
__device__ __forceinline__ void gc_settle(float& hi, float& lo) {
  const float s = hi + lo;
  lo = lo - (s - hi);
  hi = s;
}

// What a block of the two chunk kernels works on; false for a chunk that is not theirs.
struct GcChunk { int seg, tok0, n, place, n_seg_chunks, slot; size_t row0; int pos0; };
__device__ __forceinline__ bool gc_chunk(const GlaArgs& a, int c, GcChunk& x) {
  const int32_t* ch = a.chunks + (size_t)c * 4;
  x.seg = ch[0]; x.tok0 = ch[1]; x.n = ch[2]; x.place = ch[3];
  if (x.seg < 0 || x.seg >= a.n_segs || x.n <= 0 || x.n > kGcTokens) return false;
  const int q_start = a.seg_info[x.seg * 4], q_len = a.seg_info[x.seg * 4 + 1], kv_len = a.seg_info[x.seg * 4 + 2];
  x.n_seg_chunks = a.seg_chunks[x.seg * 2 + 1];
  if (x.n_seg_chunks <= 1 || x.tok0 < 0 || x.tok0 + x.n > q_len || q_start < 0 || q_start + q_len > a.n_tokens) return false;
  x.slot = a.state_slots[x.seg];
  x.row0 = (size_t)(q_start + x.tok0);
  x.pos0 = kv_len - q_len + x.tok0;
  return x.slot >= 0 && x.slot < a.n_slots;
}
__device__ __forceinline__ void gc_widen(const uint4& w, float (&y)[8]) {
  y[0] = bf2_low(w.x); y[1] = bf2_high(w.x); y[2] = bf2_low(w.y); y[3] = bf2_high(w.y);
  y[4] = bf2_low(w.z); y[5] = bf2_high(w.z); y[6] = bf2_low(w.w); y[7] = bf2_high(w.w);
}
// Eight adjacent elements of a row, rotated (every load issued before the first is used, where the pairs allow it).
__device__ __forceinline__ void gc_rotated8(const GlaArgs& a, const __nv_bfloat16* row, int pos, int d, float (&y)[8]) {
  const int n_rot = a.n_rot, half = n_rot >> 1;
  const float* cs = a.rope + (size_t)min(pos, a.max_pos - 1) * n_rot;
  const bool turned = d < n_rot, low = d < half;
  float c[8], sn[8], o[8];
  if (!a.rope_neighbours && half % 8 == 0) {  // all eight in one half
    const int at = turned ? low ? d : d - half : 0;
    const uint4 x = *reinterpret_cast<const uint4*>(row + d), other = *reinterpret_cast<const uint4*>(row + (turned ? low ? d + half : d - half : d));
    Vec4<float>::load(cs + at, reinterpret_cast<float (&)[4]>(c[0]));
    Vec4<float>::load(cs + at + 4, reinterpret_cast<float (&)[4]>(c[4]));
    Vec4<float>::load(cs + half + at, reinterpret_cast<float (&)[4]>(sn[0]));
    Vec4<float>::load(cs + half + at + 4, reinterpret_cast<float (&)[4]>(sn[4]));
    gc_widen(x, y);
    gc_widen(other, o);
    if (turned) {
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = low ? y[j] * c[j] - o[j] * sn[j] : y[j] * c[j] + o[j] * sn[j];
    }
  } else if (a.rope_neighbours && n_rot % 8 == 0) {  // four pairs
    const int at = turned ? d >> 1 : 0;
    const uint4 x = *reinterpret_cast<const uint4*>(row + d);
    Vec4<float>::load(cs + at, reinterpret_cast<float (&)[4]>(c[0]));
    Vec4<float>::load(cs + half + at, reinterpret_cast<float (&)[4]>(sn[0]));
    gc_widen(x, o);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = !turned ? o[j] : j & 1 ? o[j] * c[j >> 1] + o[j - 1] * sn[j >> 1] : o[j] * c[j >> 1] - o[j + 1] * sn[j >> 1];
  } else {
    rotated4(row, cs, d, n_rot, a.rope_neighbours, reinterpret_cast<float (&)[4]>(y[0]));
    rotated4(row, cs, d + 4, n_rot, a.rope_neighbours, reinterpret_cast<float (&)[4]>(y[4]));
  }
}

// Sums over eight neighbouring lanes of 16 values each; a lane is left with those at 2 * (its place of eight), and one more.
__device__ __forceinline__ void gc_scatter_sums(float (&v)[16], int place) {
#pragma unroll
  for (int w = 8; w >= 2; w >>= 1) {
    const bool upper = place & (w >> 1);
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float give = upper ? v[j] : v[j + w], keep = upper ? v[j + w] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, w >> 1);
    }
  }
}

// From a border of 1,024 bytes on.  Once the pairs are done, the keys' three pieces lie over the queries and what follows them.
template <int D, int VT>  // VT: rows of 64 value columns (with one, the other half of the tile's rows is anything: its results are left alone)
struct GcLocal {
  static constexpr int LD = D + 4;
  unsigned char v[VT * kGcTokens * 128];            // the values (bfloat16) as the tensor core reads them: rows of 64 columns
  float q[kGcTokens][LD];
  float lam4[kGcTokens / 4][D], lam[kGcBlocks][D];  // the decays of 4 and of 16 tokens,
  float low4[kGcTokens / 4][D], low[kGcBlocks][D];  // and what rounding took from them, or their logarithms
  float k[kGcTokens][LD];
  static constexpr int piece = D / 64 * kGcTokens * 128;
  static_assert(3 * piece <= (kGcTokens * LD + 2 * (kGcTokens / 4 + kGcBlocks) * D) * 4, "room for the keys' pieces");
};

// The dots of 4 queries and 4 keys whose groups (of 4 or 16 tokens) have `between` others between them, with those decays `mid`
// (rows of D); eight lanes a tile, a lane every eighth 16 bytes of a row.  A lane stores two of the sums.
template <int D, int LD>
__device__ __forceinline__ void gc_pairs(const float* k, const float* q, const float* mid, int between, int place, bool on, float* pout, size_t prow, int rows) {
  uint64_t acc[16] = {};
  if (on) {
#pragma unroll
    for (int e = 0; e < D / 32; ++e) {
      const int d = 4 * (place + 8 * e);
      ulonglong2 kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) kv[i] = *reinterpret_cast<const ulonglong2*>(k + i * LD + d);
      if (between > 0) {
        ulonglong2 m = *reinterpret_cast<const ulonglong2*>(mid + d);
        if (between > 1) {
          const ulonglong2 m1 = *reinterpret_cast<const ulonglong2*>(mid + D + d);
          m.x = f2_mul(m.x, m1.x);
          m.y = f2_mul(m.y, m1.y);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          kv[i].x = f2_mul(kv[i].x, m.x);
          kv[i].y = f2_mul(kv[i].y, m.y);
        }
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(q + t * LD + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          f2_fma(acc[4 * t + i], qv.x, kv[i].x);
          f2_fma(acc[4 * t + i], qv.y, kv[i].y);
        }
      }
    }
  }
  float sums[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float x, y;
    f2_unpair(acc[i], x, y);
    sums[i] = x + y;
  }
  gc_scatter_sums(sums, place);
  const int t = place >> 1;
  if (on && t < rows) *reinterpret_cast<float2*>(pout + t * prow + 2 * (place & 1)) = make_float2(sums[0], sums[1]);
}

// Whether one of eight is no number.
__device__ __forceinline__ bool gc_none(const float (&y)[8]) {
  uint64_t z = 0;
#pragma unroll
  for (int j = 0; j < 8; j += 2) f2_fma(z, f2_pair(y[j], y[j + 1]), 0);  // (an infinity times zero is a NaN)
  float a, b;
  f2_unpair(z, a, b);
  return !(a + b == 0.f);
}

// An element of a chunk's contribution that is no number as the tensor core has it, as 32-bit fmas: an infinity taken apart into pieces
// is a NaN, and its product with another number's pieces of both signs is one.  (Such keys and values as they stand at the end of their 16
// tokens: later decays change no infinity.  From `newest` on keys have no pieces.)
template <int D, int VT>
__device__ __noinline__ float gc_contribution(const GcLocal<D, VT>& sh, int d, int j, int newest) {
  const unsigned char* pieces = reinterpret_cast<const unsigned char*>(sh.q) + (d >> 6) * (kGcTokens * 128) + (d & 7) * 2;
  const unsigned char* values = sh.v + (j >> 6) * (kGcTokens * 128) + (j & 7) * 2;
  float y = 0.f;
  for (int t = 0; t < kGcTokens; ++t) {
    const int at = t * 128 + ((((d >> 3) & 7) ^ (t & 7)) << 4);
    float k = 0.f;
    for (int m = 2; m >= 0 && t < newest; --m) k += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(pieces + m * GcLocal<D, VT>::piece + at));
    const float v = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(values + t * 128 + ((((j >> 3) & 7) ^ (t & 7)) << 4)));
    y = fmaf(fabsf(k) < INFINITY && fabsf(v) < INFINITY && t < newest ? k : sh.k[t][d], v, y);
  }
  return y;
}

// What bounds it: loads, decays and the pairs' sums on the fma pipe, one after the other between barriers, with two blocks an SM.  The
// logits come through shared memory so that the decays are a loop of four instead of 32 copies of the code (a block's first pass
// 38,000 -> 28,000 cycles).  The contribution, as L^T = V^T K, is on tcgen05, keys in three pieces (split3):
// 212 -> 174 us against fmas (cold caches).
template <int D, int VT>
__global__ void __launch_bounds__(2 * D, 256 / D) gla_local_kernel(GlaArgs a) {
  constexpr int kThreads = 2 * D, LD = D + 4, kLanes = D / 8;  // lanes a token
  extern __shared__ unsigned char gc_smem[];
  __shared__ uint64_t mma_done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t base = (smem_addr(gc_smem) + 1023u) & ~1023u;
  GcLocal<D, VT>& sh = *reinterpret_cast<GcLocal<D, VT>*>(gc_smem + (base - smem_addr(gc_smem)));
  const int c = blockIdx.x / a.H, h = blockIdx.x % a.H, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;  // (heads side by side: whole rows)
  if (tid == 0) {
    mbar_init(&mma_done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 2 * D);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  GcChunk x;
  if (!gc_chunk(a, c, x)) {
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 2 * D);
    return;
  }
  const int n = x.n;
  const __nv_bfloat16* vb = (const __nv_bfloat16*)a.v + (size_t)h * a.Dv;
  for (int i = tid; i < kGcTokens * 8 * VT; i += kThreads) {
    const int t = i / (8 * VT), j = i % (8 * VT);
    const bool in = t < n && 8 * j < a.Dv;
    gla_cp16(sh.v + (j >> 3) * (kGcTokens * 128) + t * 128 + (((j & 7) ^ (t & 7)) << 4), in ? vb + (x.row0 + t) * a.v_stride + 8 * j : vb, in);
  }
  gla_cp_commit();
  float* pout = a.out + (x.row0 * a.H + h) * a.Dv;  // P's rows, where the outputs will lie
  const size_t prow = (size_t)a.H * a.Dv;
  // a thread takes 4 tokens x 8 channels from memory: their pairs, then keys decayed to the end of the four, queries from its
  // start.  Tokens that do not exist add nothing and decay nothing.
  {
    const int d = tid % kLanes * 8, t0 = tid / kLanes * 4;
    const __nv_bfloat16* qb = (const __nv_bfloat16*)a.q + (size_t)(h / a.qk_div) * D;
    const __nv_bfloat16* kb = (const __nv_bfloat16*)a.k + (size_t)(h / a.qk_div) * D;
    float k[4][8], q[4][8], w[4][8], logs[8];
    if (!a.a_head) {  // (through shared memory: a place that only this thread uses before the queries come)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float* z = a.z + ((x.row0 + min(t0 + i, n - 1)) * a.H + h) * D + d;
        gla_cp16(&sh.q[t0 + i][d], z, true);
        gla_cp16(&sh.q[t0 + i][d + 4], z + 4, true);
      }
      gla_cp_commit();
    }
    if (!a.rope) {
      uint4 kw[4], qw[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const size_t tok = x.row0 + min(t0 + i, n - 1);
        kw[i] = *reinterpret_cast<const uint4*>(kb + tok * a.k_stride + d);
        qw[i] = *reinterpret_cast<const uint4*>(qb + tok * a.q_stride + d);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) { gc_widen(kw[i], k[i]); gc_widen(qw[i], q[i]); }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = min(t0 + i, n - 1);
        gc_rotated8(a, kb + (x.row0 + t) * a.k_stride, x.pos0 + t, d, k[i]);
        gc_rotated8(a, qb + (x.row0 + t) * a.q_stride, x.pos0 + t, d, q[i]);
      }
    }
    if (!a.a_head) {
      float bias[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        bias[j] = a.z_bias ? a.z_bias[(size_t)h * D + d + j] : 0.f;
        logs[j] = 0.f;
      }
      gla_cp_wait_all();
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        float y[8];
        Vec4<float>::load(&sh.q[t0 + i][d], reinterpret_cast<float (&)[4]>(y[0]));
        Vec4<float>::load(&sh.q[t0 + i][d + 4], reinterpret_cast<float (&)[4]>(y[4]));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float l = t0 + i < n ? log_decay_of(y[j] + bias[j], a.inv_tau) : 0.f;
          logs[j] += l;
          y[j] = expf(l);
        }
        Vec4<float>::store(&sh.q[t0 + i][d], reinterpret_cast<float (&)[4]>(y[0]));
        Vec4<float>::store(&sh.q[t0 + i][d + 4], reinterpret_cast<float (&)[4]>(y[4]));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        Vec4<float>::load(&sh.q[t0 + i][d], reinterpret_cast<float (&)[4]>(w[i][0]));
        Vec4<float>::load(&sh.q[t0 + i][d + 4], reinterpret_cast<float (&)[4]>(w[i][4]));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float y = t0 + i < n ? a.a_head[(x.row0 + t0 + i) * a.a_head_stride + h] : 1.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) w[i][j] = y;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool in = t0 + i < n;
      const float kf = in ? a.k_fac ? a.k_fac[(x.row0 + t0 + i) * a.H + h] : 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        k[i][j] = in ? k[i][j] * kf : 0.f;
        q[i][j] = in ? q[i][j] * a.q_scale : 0.f;
      }
    }
    float p[10];
    int at = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int t = s; t < 4; ++t) {
        if (t > s) {
#pragma unroll
          for (int j = 0; j < 8; ++j) k[s][j] *= w[t][j];
        }
        p[at] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) p[at] = fmaf(k[s][j], q[t][j], p[at]);
        ++at;
      }
    {
      float hi[8], lo[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (a.a_head) {
          hi[j] = w[0][j];
          lo[j] = 0.f;
#pragma unroll
          for (int i = 1; i < 4; ++i) gc_times(hi[j], lo[j], w[i][j], 0.f);
          gc_settle(hi[j], lo[j]);
        } else {
          hi[j] = expf(logs[j]);
          lo[j] = logs[j];
        }
      }
      Vec4<float>::store(&sh.lam4[t0 / 4][d], reinterpret_cast<float (&)[4]>(hi[0]));
      Vec4<float>::store(&sh.lam4[t0 / 4][d + 4], reinterpret_cast<float (&)[4]>(hi[4]));
      Vec4<float>::store(&sh.low4[t0 / 4][d], reinterpret_cast<float (&)[4]>(lo[0]));
      Vec4<float>::store(&sh.low4[t0 / 4][d + 4], reinterpret_cast<float (&)[4]>(lo[4]));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (i > 0) w[i][j] *= w[i - 1][j];
        q[i][j] *= w[i][j];
      }
      Vec4<float>::store(&sh.k[t0 + i][d], reinterpret_cast<float (&)[4]>(k[i][0]));
      Vec4<float>::store(&sh.k[t0 + i][d + 4], reinterpret_cast<float (&)[4]>(k[i][4]));
      Vec4<float>::store(&sh.q[t0 + i][d], reinterpret_cast<float (&)[4]>(q[i][0]));
      Vec4<float>::store(&sh.q[t0 + i][d + 4], reinterpret_cast<float (&)[4]>(q[i][4]));
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < 10; ++i) p[i] += __shfl_xor_sync(0xffffffffu, p[i], o);
    at = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int t = s; t < 4; ++t) {
        if (tid % kLanes == at % kLanes && t0 + t < n) pout[(t0 + t) * prow + t0 + s] = p[at];
        ++at;
      }
  }
  __syncthreads();
  // pairs of fours J < I in a block of 16
  for (int i = tid; i < kGcBlocks * 6 * 8; i += kThreads) {  // (whole warps of it are on or off)
    const int pr = (i >> 3) % 6, b = (i >> 3) / 6, I = pr < 1 ? 1 : pr < 3 ? 2 : 3, J = pr - (I * (I - 1)) / 2;
    const int t0 = b * kGcBlock + 4 * I, s0 = b * kGcBlock + 4 * J;
    gc_pairs<D, LD>(sh.k[s0], sh.q[t0], sh.lam4[4 * b + J + 1], I - J - 1, i & 7, t0 < n, pout + t0 * prow + s0, prow, n - t0);
  }
  __syncthreads();
  // keys decayed to the end of their 16, queries from the start of theirs
  {
    const int d = tid % (D / 4) * 4;
    for (int t = tid / (D / 4); t < kGcTokens; t += kThreads / (D / 4)) {
      const int b = t / kGcBlock, u = t / 4 % 4;
      ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(&sh.k[t][d]), qv = *reinterpret_cast<const ulonglong2*>(&sh.q[t][d]);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        if (m == u) continue;
        const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(&sh.lam4[4 * b + m][d]);
        ulonglong2& y = m > u ? kv : qv;
        y.x = f2_mul(y.x, l.x);
        y.y = f2_mul(y.y, l.y);
      }
      *reinterpret_cast<ulonglong2*>(&sh.k[t][d]) = kv;
      *reinterpret_cast<ulonglong2*>(&sh.q[t][d]) = qv;
    }
    for (int i = tid; i < kGcBlocks * D; i += kThreads) {
      const int b = i / D, e = i % D;
      float hi = sh.lam4[4 * b][e], lo = sh.low4[4 * b][e];
      if (a.a_head) {
#pragma unroll
        for (int m = 1; m < 4; ++m) gc_times(hi, lo, sh.lam4[4 * b + m][e], sh.low4[4 * b + m][e]);
        gc_settle(hi, lo);
      } else {
        lo = (lo + sh.low4[4 * b + 1][e]) + (sh.low4[4 * b + 2][e] + sh.low4[4 * b + 3][e]);
        hi = expf(lo);
      }
      sh.lam[b][e] = hi;
      sh.low[b][e] = lo;
    }
  }
  gla_cp_wait_all();
  __syncthreads();
  // pairs of blocks J < I
  for (int i = tid; i < 6 * 16 * 8; i += kThreads) {
    const int pr = i >> 7, I = pr < 1 ? 1 : pr < 3 ? 2 : 3, J = pr - (I * (I - 1)) / 2, tile = (i >> 3) & 15;
    const int t0 = I * kGcBlock + 4 * (tile >> 2), s0 = J * kGcBlock + 4 * (tile & 3);
    gc_pairs<D, LD>(sh.k[s0], sh.q[t0], sh.lam[min(J + 1, kGcBlocks - 1)], I - J - 1, i & 7, t0 < n, pout + t0 * prow + s0, prow, n - t0);
  }
  if (!a.a_head) {  // the queries, decayed from the chunk's start (one decay for all channels: gla_out_kernel's)
    const int d = tid % (D / 4) * 4;
    for (int t = tid / (D / 4); t < n; t += kThreads / (D / 4)) {
      ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&sh.q[t][d]);
      for (int m = 0; m < t / kGcBlock; ++m) {
        const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(&sh.lam[m][d]);
        qv.x = f2_mul(qv.x, l.x);
        qv.y = f2_mul(qv.y, l.y);
      }
      *reinterpret_cast<ulonglong2*>(a.z + ((x.row0 + t) * a.H + h) * D + d) = qv;
    }
  }
  if (tid < D) {
    float hi = sh.lam[0][tid], lo = sh.low[0][tid];
    if (a.a_head) {
#pragma unroll
      for (int m = 1; m < kGcBlocks; ++m) gc_times(hi, lo, sh.lam[m][tid], sh.low[m][tid]);
      hi += lo;
    } else {
      hi = expf((lo + sh.low[1][tid]) + (sh.low[2][tid] + sh.low[3][tid]));
    }
    a.decay_prod[((size_t)c * a.H + h) * D + tid] = hi;
  }
  // the chunk's contribution: keys decayed to its end, in three pieces; a thread has eight channels of a token of every 16
  {
    constexpr int kPass = kThreads / kLanes;  // tokens at a time
    static_assert(kPass == kGcBlock, "the tokens of a pass lie in one block of 16");
    const int d = tid % kLanes * 8, t0 = tid / kLanes;
    uint64_t lam[kGcBlocks - 1][4];
#pragma unroll
    for (int b = 1; b < kGcBlocks; ++b)
#pragma unroll
      for (int j = 0; j < 4; ++j) lam[b - 1][j] = *reinterpret_cast<const uint64_t*>(&sh.lam[b][d + 2 * j]);
    __syncthreads();  // the queries and the decays have been read
    unsigned char* pieces = reinterpret_cast<unsigned char*>(sh.q);
#pragma unroll
    for (int b = 0; b < kGcBlocks; ++b) {
      const int t = b * kGcBlock + t0;
      float y[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint64_t kv = *reinterpret_cast<const uint64_t*>(&sh.k[t][d + 2 * j]);
#pragma unroll
        for (int m = b + 1; m < kGcBlocks; ++m) kv = f2_mul(kv, lam[m - 1][j]);
        f2_unpair(kv, y[2 * j], y[2 * j + 1]);
      }
      if (t >= n - 2 && t < n) {  // (the newest tokens' are added in registers, from here)
        Vec4<float>::store(&sh.k[t][d], reinterpret_cast<float (&)[4]>(y[0]));
        Vec4<float>::store(&sh.k[t][d + 4], reinterpret_cast<float (&)[4]>(y[4]));
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = 0.f;
      }
      uint4 w[3];
      split3(y, w);
      unsigned char* dst = pieces + (d >> 6) * (kGcTokens * 128) + t * 128 + ((((d >> 3) & 7) ^ (t & 7)) << 4);
#pragma unroll
      for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(dst + m * sh.piece) = w[m];
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    if (elect_one()) {
      constexpr uint32_t id = instr_desc(D) | kMnMajorA | kMnMajorB;
      const uint32_t v0 = smem_addr(sh.v), k0 = smem_addr(sh.q);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint64_t v = smem_desc_mn(v0 + k * 2048, kGcTokens * 128);
        tc_mma(tmem, v, smem_desc_mn(k0 + k * 2048, kGcTokens * 128), id, k != 0);
        tc_mma(tmem + D, v, smem_desc_mn(k0 + GcLocal<D, VT>::piece + k * 2048, kGcTokens * 128), id, k != 0);
        tc_mma(tmem + D, v, smem_desc_mn(k0 + 2 * GcLocal<D, VT>::piece + k * 2048, kGcTokens * 128), id, 1);
      }
      tc_commit(&mma_done);
    }
    __syncwarp();
  }
  if (!mbar_wait(&mma_done, 0, &abort_flag)) {
    if (atomicCAS(&g_gla_status[0], 0, 602) == 0) g_gla_status[1] = blockIdx.x;
    abort_flag = 1;
  }
  __syncwarp();
  tc_fence_after();
  {
    // The two newest tokens' share, the largest where decays are strong, is added last and by itself: the accumulator cuts off instead of
    // rounding.  (Two sums of 32 tokens, read one after the other, bring states 0 to 2 % closer to 64 bits; with them, with the sum of an
    // infinity's element written out eight times and with outputs of four sums of 16 a retention layer of 16 heads of 128, 572 tokens took
    // 91 us instead of 77.)
    const int j = (warp & 3) * 32 + lane;  // a value column; 64 channels of it
    const uint32_t my_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 64);
    auto value = [&](int t) {
      return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(sh.v + (j >> 6) * (kGcTokens * 128) + t * 128 + ((((j >> 3) & 7) ^ (t & 7)) << 4) + (j & 7) * 2));
    };
    const bool two = n >= 2, mine = j < 64 * VT;
    const float v_last = mine ? value(n - 1) : 0.f, v_before = mine && two ? value(n - 2) : 0.f;
    const float *k_last = &sh.k[n - 1][(warp >> 2) * 64], *k_before = two ? k_last - LD : k_last;
    float* dst = a.carry + (((size_t)c * a.H + h) * D + (warp >> 2) * 64) * a.Dv + j;
#pragma unroll 1
    for (int i = 0; i < 64; i += 8) {
      float r[2][8], k[2][8], y[8];
      tmem_ld8_start(my_tmem + i, r[0]);
      tmem_ld8_start(my_tmem + D + i, r[1]);
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        Vec4<float>::load(k_last + i + e, reinterpret_cast<float (&)[4]>(k[0][e]));
        Vec4<float>::load(k_before + i + e, reinterpret_cast<float (&)[4]>(k[1][e]));
      }
      tmem_ld8_finish(r);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = fmaf(k[0][e], v_last, fmaf(k[1][e], v_before, r[0][e] + r[1][e]));
      if (j < a.Dv) {
        if (gc_none(y)) {
#pragma unroll 1
          for (int e = 0; e < 8; ++e) {
            float z = 0.f;
#pragma unroll
            for (int f = 0; f < 8; ++f) z = e == f ? y[f] : z;
            if (fabsf(z) < INFINITY) continue;
            z = gc_contribution<D, VT>(sh, (warp >> 2) * 64 + i + e, j, n - 2);
#pragma unroll
            for (int f = 0; f < 8; ++f) y[f] = e == f ? z : y[f];
          }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[(size_t)(i + e) * a.Dv] = y[e];
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 2 * D);
}

// A thread per two state elements of a (segment, head) walks the segment's chunks, the next eight contributions in flight while
// eight are added up.
__global__ void __launch_bounds__(256) gla_walk_kernel(GlaArgs a) {
  pdl_wait();
  pdl_trigger();
  const int seg = blockIdx.y, h = blockIdx.z;
  const int first = a.seg_chunks[seg * 2], n = a.seg_chunks[seg * 2 + 1];
  if (n <= 1 || first < 0 || first + n > a.n_chunks) return;
  const int slot = a.state_slots[seg];
  if (slot < 0 || slot >= a.n_slots) return;
  const size_t DV = (size_t)a.D * a.Dv;
  const size_t e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 2;
  if (e >= DV) return;
  const int d = (int)(e / a.Dv);
  const bool fresh = a.seg_info[seg * 4 + 2] - a.seg_info[seg * 4 + 1] == 0;
  float* st = a.state + ((size_t)slot * a.H + h) * DV + e;
  float* l = a.carry + ((size_t)first * a.H + h) * DV + e;
  const float* w = a.decay_prod + ((size_t)first * a.H + h) * a.D + d;
  const size_t ls = (size_t)a.H * DV, ws = (size_t)a.H * a.D;
  constexpr int kAhead = 8;
  float2 s = make_float2(0.f, 0.f), x[2][kAhead];
  float p[2][kAhead];
  if (!fresh) s = *reinterpret_cast<const float2*>(st);
  auto load = [&](int b, int c0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (c0 + u < n) {
        x[b][u] = *reinterpret_cast<const float2*>(l + (c0 + u) * ls);
        p[b][u] = w[(c0 + u) * ws];
      }
  };
  auto walk = [&](int b, int c0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (c0 + u < n) {
        *reinterpret_cast<float2*>(l + (c0 + u) * ls) = s;
        s.x = fmaf(p[b][u], s.x, x[b][u].x);
        s.y = fmaf(p[b][u], s.y, x[b][u].y);
      }
  };
  load(0, 0);
  for (int c0 = 0; c0 < n; c0 += 2 * kAhead) {
    load(1, c0 + kAhead);
    walk(0, c0);
    load(0, c0 + 2 * kAhead);
    walk(1, c0 + kAhead);
  }
  *reinterpret_cast<float2*>(st) = s;
}

// What gla_out_kernel has in shared memory, from a border of 1,024 bytes on: 64 channels of the start state (three pieces of two rows of
// 64 value columns) and of the queries (three pieces), later P, and the values; all as the tensor core reads them.
struct GoPlace {
  static constexpr int tile = 64 * 128;  // 64 rows of 128 bytes
  static constexpr int s = 0, q = s + 6 * tile, v = q + 3 * tile, bytes = v + 2 * tile;
};

// Outputs of a chunk: o^T = S^T q^T + V^T P^T, 128 value columns (rows of the tensor core's tile) x 64 tokens.  Two threads a value column.  S,
// q and P are taken apart into three bfloat16 numbers each (split3) and the six products that reach 2^-24 are taken (with V, which is
// bfloat16, three); the leading pieces' products are chains of two steps of 16, added up in registers.  Two blocks an SM; what bounds them is
// memory's latency (2.4 TB/s: loads, taking apart, products and stores of a block follow one another; the tensor pipe is 13 % busy).
// 130 -> 94 us against fmas (cold caches).
template <int D>
__global__ void __launch_bounds__(256, 2) gla_out_kernel(GlaArgs a) {
  constexpr int kStages = D / 64;
  extern __shared__ unsigned char go_smem[];
  __shared__ uint64_t mma_done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, first_odd[128];  // the first token whose value is no number, per column
  __shared__ float dec[kGcTokens], own[kGcTokens];  // own: P's diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, half = warp >> 2;
  const uint32_t base = (smem_addr(go_smem) + 1023u) & ~1023u;
  unsigned char* tiles = go_smem + (base - smem_addr(go_smem));
  if (tid == 0) {
    mbar_init(&mma_done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 128) first_odd[tid] = kGcTokens;
  if (warp == 0) tmem_alloc(&tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  const int c = blockIdx.x / a.H, h = blockIdx.x % a.H, Dv = a.Dv;
  GcChunk x;
  if (gc_chunk(a, c, x)) {
    const int n = x.n;
    const float* start = a.carry + ((size_t)c * a.H + h) * D * Dv;
    const float* pin = a.out + (x.row0 * a.H + h) * Dv;
    const size_t row = (size_t)a.H * Dv;
    // eight elements of a row of 128 bytes and more, as they lie in memory, and where they go: rows of `per` eights
    float sv[4][8], qv[2][8];
    auto load8 = [](const float* p, bool in, float (&y)[8]) {
      if (in) {
        Vec4<float>::load(p, reinterpret_cast<float (&)[4]>(y[0]));
        Vec4<float>::load(p + 4, reinterpret_cast<float (&)[4]>(y[4]));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = 0.f;
      }
    };
    auto put8 = [&](int at, int piece, int r, int c8, const float (&y)[8]) {
      uint4 w[3];
      split3(y, w);
      unsigned char* dst = tiles + at + (c8 >> 3) * GoPlace::tile + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
#pragma unroll
      for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(dst + m * piece) = w[m];
    };
    auto load_s = [&](int st) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + 256 * u, d = i >> 4, c8 = i & 15;
        load8(start + (size_t)(64 * st + d) * Dv + 8 * c8, 8 * c8 < Dv, sv[u]);
      }
    };
    const __nv_bfloat16* qb = (const __nv_bfloat16*)a.q + (size_t)(h / a.qk_div) * D;
    auto load_q8 = [&](int t, int d, float (&y)[8]) {
      if (!a.a_head) {
        load8(a.z + ((x.row0 + t) * a.H + h) * D + d, t < n, y);
      } else if (t < n) {  // one decay for all channels: the queries once more from their rows
        if (a.rope) gc_rotated8(a, qb + (x.row0 + t) * a.q_stride, x.pos0 + t, d, y);
        else gc_widen(*reinterpret_cast<const uint4*>(qb + (x.row0 + t) * a.q_stride + d), y);
      } else {
        load8(nullptr, false, y);
      }
    };
    auto load_q = [&](int st) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = tid + 256 * u;
        load_q8(i >> 3, 64 * st + (i & 7) * 8, qv[u]);
      }
    };
    load_s(0);
    load_q(0);
    {
      // The values.  A row of P holds zeros behind its own token, but zero times an infinity or NaN is NaN: such a value goes in as
      // zero, and its column is summed up once more from its token on.
      const __nv_bfloat16* vb = (const __nv_bfloat16*)a.v + (size_t)h * Dv;
      uint4 w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + 256 * u, t = i >> 4, c8 = i & 15;
        w[u] = t < n && 8 * c8 < Dv ? *reinterpret_cast<const uint4*>(vb + (x.row0 + t) * a.v_stride + 8 * c8) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + 256 * u, t = i >> 4, c8 = i & 15;
        uint32_t* y = reinterpret_cast<uint32_t*>(&w[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool lo = (y[j] & 0x7f80u) == 0x7f80u, hi = (y[j] & 0x7f800000u) == 0x7f800000u;
          if (lo) atomicMin(&first_odd[8 * c8 + 2 * j], t);
          if (hi) atomicMin(&first_odd[8 * c8 + 2 * j + 1], t);
          y[j] &= (lo ? 0u : 0xffffu) | (hi ? 0u : 0xffff0000u);
        }
        *reinterpret_cast<uint4*>(tiles + GoPlace::v + (c8 >> 3) * GoPlace::tile + t * 128 + (((c8 & 7) ^ (t & 7)) << 4)) = w[u];
      }
    }
    if (a.a_head) {
      if (tid < 32) {
        const double w0 = 2 * tid < n ? a.a_head[(x.row0 + 2 * tid) * a.a_head_stride + h] : 1.f;
        const double w1 = w0 * (2 * tid + 1 < n ? a.a_head[(x.row0 + 2 * tid + 1) * a.a_head_stride + h] : 1.f);
        double up = w1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xffffffffu, up, o);
          if (tid >= o) up *= y;
        }
        double before = __shfl_up_sync(0xffffffffu, up, 1);
        if (tid == 0) before = 1.;
        dec[2 * tid] = (float)(before * w0);
        dec[2 * tid + 1] = (float)(before * w1);
      }
      __syncthreads();
    }
    auto put_stage = [&]() {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + 256 * u;
        put8(GoPlace::s, 2 * GoPlace::tile, i >> 4, i & 15, sv[u]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = tid + 256 * u;
        if (a.a_head) {
          const float f = a.q_scale * dec[i >> 3];
#pragma unroll
          for (int j = 0; j < 8; ++j) qv[u][j] *= f;
        }
        put8(GoPlace::q, GoPlace::tile, i >> 3, i & 7, qv[u]);
      }
    };
    bool bad = false;
    uint32_t phase = 0;
    auto wait = [&]() {
      if (!bad && !mbar_wait(&mma_done, phase, &abort_flag)) {
        if (atomicCAS(&g_gla_status[0], 0, 601) == 0) g_gla_status[1] = blockIdx.x;
        abort_flag = 1;
        bad = true;
      }
      phase ^= 1;
      __syncwarp();
      tc_fence_after();
    };
    // columns of 64 in tensor memory: two chains of the leading pieces, the second order, the third
    const uint32_t my_tmem = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 32);
    constexpr uint32_t id1 = instr_desc(64) | kMnMajorA, id2 = instr_desc(128) | kMnMajorA;
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.f;
    auto add_chains = [&]() {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        float r[2][8];
        tmem_ld8_start(my_tmem + i, r[0]);
        tmem_ld8_start(my_tmem + 64 + i, r[1]);
        tmem_ld8_finish(r);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i + j] = (acc[i + j] + r[0][j]) + r[1][j];
      }
    };
#pragma unroll 1
    for (int st = 0; st < kStages; ++st) {
      put_stage();
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t s1 = smem_desc_mn(base + GoPlace::s + k * 2048, GoPlace::tile), s2 = smem_desc_mn(base + GoPlace::s + 2 * GoPlace::tile + k * 2048, GoPlace::tile),
                           s3 = smem_desc_mn(base + GoPlace::s + 4 * GoPlace::tile + k * 2048, GoPlace::tile);
            const uint64_t q1 = smem_desc(base + GoPlace::q) + 2 * k, q2 = smem_desc(base + GoPlace::q + GoPlace::tile) + 2 * k;
            tc_mma(tmem + (k >> 1) * 64, s1, q1, id1, k & 1);
            tc_mma(tmem + 128, s1, q2, id2, st | k);
            tc_mma(tmem + 128, s2, q1, id2, 1);
            tc_mma(tmem + 192, s3, q1, id1, 1);
          }
          tc_commit(&mma_done);
        }
        __syncwarp();
      }
      if (st + 1 < kStages) {
        load_s(st + 1);
        load_q(st + 1);
      } else {  // P (what lies behind the diagonal was not written)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = tid + 256 * u, t = i >> 3, s0 = (i & 7) * 8;
          const float* p = pin + (size_t)min(t, n - 1) * row + s0;
          load8(p, t < n && s0 + 7 <= t, qv[u]);
          if (t < n && s0 <= t && s0 + 7 > t) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (s0 + j <= t) qv[u][j] = p[j];
          }
        }
      }
      wait();
      add_chains();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = tid + 256 * u, t = i >> 3, s0 = (i & 7) * 8;
      if (s0 == (t & ~7)) {  // (a token's own value, the largest share where decays are strong: added in registers)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (s0 + j == t) {
            own[t] = qv[u][j];
            qv[u][j] = 0.f;
          }
      }
      put8(GoPlace::q, GoPlace::tile, i >> 3, i & 7, qv[u]);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t v = smem_desc_mn(base + GoPlace::v + k * 2048, GoPlace::tile);
          tc_mma(tmem + (k >> 1) * 64, v, smem_desc(base + GoPlace::q) + 2 * k, id1, k & 1);
          tc_mma(tmem + 128, v, smem_desc(base + GoPlace::q + GoPlace::tile) + 2 * k, id2, 1);
        }
        tc_commit(&mma_done);
      }
      __syncwarp();
    }
    wait();
    const int j = quad * 32 + lane, odd_from = j < Dv ? first_odd[j] : kGcTokens;
    float* o = a.out + (x.row0 * a.H + h) * Dv + j;
    bool odd = j < Dv && odd_from < n;
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
      float r[4][8];
#pragma unroll
      for (int m = 0; m < 4; ++m) tmem_ld8_start(my_tmem + 64 * m + i, r[m]);
      tmem_ld8_finish(r);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int t = half * 32 + i + e;
        const float v = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(
            tiles + GoPlace::v + (j >> 6) * GoPlace::tile + t * 128 + ((((j >> 3) & 7) ^ (t & 7)) << 4) + (j & 7) * 2));
        acc[i + e] = fmaf(t < n ? own[t] : 0.f, v, ((acc[i + e] + (r[2][e] + r[3][e])) + r[0][e]) + r[1][e]);
      }
      if (j < Dv) odd |= gc_none(reinterpret_cast<const float (&)[8]>(acc[i]));
    }
    // Such an output as 32-bit fmas, and up to its own token: an infinity taken apart into pieces is a NaN.  (All of them before one is
    // stored: P lies where they go.)
    if (__syncthreads_or(odd)) {
      const __nv_bfloat16* vb = (const __nv_bfloat16*)a.v + (size_t)h * Dv + j;
#pragma unroll 1
      for (int i = 0; i < (odd ? 32 : 0); ++i) {
        const int t = half * 32 + i;
        float y = 0.f;
#pragma unroll
        for (int e = 0; e < 32; ++e) y = e == i ? acc[e] : y;
        if (t >= n || (t < odd_from && fabsf(y) < INFINITY)) continue;
        y = 0.f;
        for (int d = 0; d < D; d += 8) {
          float q[8];
          load_q8(t, d, q);
#pragma unroll
          for (int e = 0; e < 8; ++e) y = fmaf(a.a_head ? q[e] * (a.q_scale * dec[t]) : q[e], start[(size_t)(d + e) * Dv + j], y);
        }
        for (int s = 0; s <= t; ++s) y = fmaf(pin[(size_t)t * row + s], __bfloat162float(vb[(x.row0 + s) * a.v_stride]), y);
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[e] = e == i ? y : acc[e];
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int t = half * 32 + i;
      if (t < n && j < Dv) o[(size_t)t * row] = acc[i];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// Whether a step's long portions go as products (the chunks are the host's: none may be longer than 64; where they do not pay the
// host names no length, parts/gla.py: longest_chunk).  Shorter chunks than 32 would leave more than half of a product's rows empty.  A
// layer, token by token against products, one request of 65, 128 and 256 tokens: 48 heads of 128 159 and 130, 167 and 138, 177 and
// 155 us; 16 heads of 64 87 and 65, 87 and 69, 95 and 69; one decay a head, 16 heads of 64 61 and 57, 61 and 61, 62 and 62.
inline bool gla_chunks_fit(const GlaArgs& a, int longest_chunk) {
  const uintptr_t at = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out | (uintptr_t)a.carry | (uintptr_t)a.state | (a.a_head ? 0 : (uintptr_t)a.z);
  return (a.D == 64 || a.D == 128) && a.Dv >= 64 && a.Dv <= 128 && a.Dv % 8 == 0 && !a.ones_col && longest_chunk >= 32 &&
         longest_chunk <= kGcTokens && (long long)a.n_chunks * a.H <= 0x7fffffff && (a.q_stride | a.k_stride | a.v_stride) % 8 == 0 && (at & 15) == 0;
}

template <int D, int VT>
static int launch_gla_chunks_as(const GlaArgs& a, cudaStream_t s) {
  auto local = gla_local_kernel<D, VT>;
  auto outs = gla_out_kernel<D>;
  constexpr int sl = (int)sizeof(GcLocal<D, VT>) + 1024, so = GoPlace::bytes + 1024;
  FTK_REQUIRE(cudaFuncSetAttribute(local, cudaFuncAttributeMaxDynamicSharedMemorySize, sl) == cudaSuccess &&
                  cudaFuncSetAttribute(outs, cudaFuncAttributeMaxDynamicSharedMemorySize, so) == cudaSuccess,
              "gla_scan: cannot set up the chunk kernels");
  FTK_LAUNCH(local, (unsigned)a.n_chunks * a.H, 2 * D, sl, s, a);
  FTK_LAUNCH_CHECK("gla_scan (chunk products)");
  const size_t DV = (size_t)a.D * a.Dv;
  FTK_LAUNCH(gla_walk_kernel, dim3((unsigned)((DV / 2 + 255) / 256), a.n_segs, a.H), 256, 0, s, a);
  FTK_LAUNCH_CHECK("gla_scan (states)");
  FTK_LAUNCH(outs, (unsigned)a.n_chunks * a.H, 256, so, s, a);
  FTK_LAUNCH_CHECK("gla_scan (outputs)");
  return 0;
}

int gla_chunks_status(int* out) { return take_status(g_gla_status, out); }  // (merged into ftk_read_status)
int gla_chunks_set_status(int code) { return set_status(g_gla_status, code); }

inline int launch_gla_chunks(const GlaArgs& a, cudaStream_t s) {
  return a.D == 128 ? launch_gla_chunks_as<128, 2>(a, s) : a.Dv <= 64 ? launch_gla_chunks_as<64, 1>(a, s) : launch_gla_chunks_as<64, 2>(a, s);
}

}  // namespace ftk
