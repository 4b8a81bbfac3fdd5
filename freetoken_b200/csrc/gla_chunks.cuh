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
// All 32-bit fmas on the CUDA cores (two at a time, fma.rn.f32x2), 8 x 8 sums a thread.  Three fmas an element of the state and
// token become two, over register tiles, and the decays are products of at most 9 factors instead of a running product.
//
// 48 heads of 128 x 128, 2,048 tokens, a decay per channel, each kernel with its wait for the one before: decays 53 us,
// contributions 226, carry 99 and outputs 359 token by token; 207, 84 and 137 for these three.  The layer 973 -> 690 us, with
// one decay a head 949 -> 653; 16 heads 371 -> 231, 16 heads of 64 181 -> 134, 300 tokens 212 -> 159.  Against 64 bits the
// outputs are off by 1.0e-7 either way, and by 3.0e-7 instead of 3.6e-6 where the decays are close to 1.  The fmas alone would
// take 100 us at 1.9 GHz.
#pragma once

namespace ftk {

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

// TC value columns a thread in the contribution: Dv <= 16 TC
template <int D, int TC>
struct GcLocal {
  static constexpr int LD = D + 4;
  float k[kGcTokens][LD], q[kGcTokens][LD];
  float lam4[kGcTokens / 4][D], lam[kGcBlocks][D];  // the decays of 4 and of 16 tokens,
  float low4[kGcTokens / 4][D], low[kGcBlocks][D];  // and what rounding took from them, or their logarithms
  uint16_t v[kGcTokens][16 * TC];                   // (bfloat16)
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

// What bounds it: the fmas and shared memory about equally, with 2 blocks an SM and a barrier between the passes (fma pipe 45 %
// busy, shared memory 47 %).  A third of a block's time goes by before its first products, on loads and decays; the logits come through shared
// memory so that the decays are a loop of four instead of 32 copies of the code (a block's first pass 38,000 -> 28,000 cycles).
template <int D, int TC>
__global__ void __launch_bounds__(2 * D, 256 / D) gla_local_kernel(GlaArgs a) {
  pdl_wait();
  pdl_trigger();
  constexpr int kThreads = 2 * D, LD = D + 4, kLanes = D / 8;  // lanes a token
  extern __shared__ __align__(16) unsigned char gc_smem[];
  GcLocal<D, TC>& sh = *reinterpret_cast<GcLocal<D, TC>*>(gc_smem);
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  GcChunk x;
  if (!gc_chunk(a, c, x)) return;
  const int n = x.n;
  const __nv_bfloat16* vb = (const __nv_bfloat16*)a.v + (size_t)h * a.Dv;
  for (int i = tid; i < kGcTokens * 2 * TC; i += kThreads) {
    const int t = i / (2 * TC), j = i % (2 * TC) * 8;
    const bool in = t < n && j < a.Dv;
    gla_cp16(&sh.v[t][j], in ? vb + (x.row0 + t) * a.v_stride + j : vb, in);
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
  // the chunk's contribution: 8 channels (in pairs) x TC columns (fours, 64 apart) a thread, decayed from block to block
  {
    const int cg = tid % 16 * 4, dg = tid / 16 * 8;
    uint64_t acc[4][TC] = {};
#pragma unroll 1
    for (int b = 0; b < kGcBlocks; ++b) {
      if (b > 0) {
        const ulonglong2 l0 = *reinterpret_cast<const ulonglong2*>(&sh.lam[b][dg]), l1 = *reinterpret_cast<const ulonglong2*>(&sh.lam[b][dg + 4]);
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          acc[0][j] = f2_mul(acc[0][j], l0.x);
          acc[1][j] = f2_mul(acc[1][j], l0.y);
          acc[2][j] = f2_mul(acc[2][j], l1.x);
          acc[3][j] = f2_mul(acc[3][j], l1.y);
        }
      }
#pragma unroll 4
      for (int s = b * kGcBlock; s < (b + 1) * kGcBlock; ++s) {
        const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(&sh.k[s][dg]), k1 = *reinterpret_cast<const ulonglong2*>(&sh.k[s][dg + 4]);
        uint32_t w[TC / 2];
#pragma unroll
        for (int g = 0; g < TC / 4; ++g) {
          const uint2 t = *reinterpret_cast<const uint2*>(&sh.v[s][cg + 64 * g]);
          w[2 * g] = t.x;
          w[2 * g + 1] = t.y;
        }
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          const float v = j & 1 ? bf2_high(w[j >> 1]) : bf2_low(w[j >> 1]);
          const uint64_t v2 = f2_pair(v, v);
          f2_fma(acc[0][j], k0.x, v2);
          f2_fma(acc[1][j], k0.y, v2);
          f2_fma(acc[2][j], k1.x, v2);
          f2_fma(acc[3][j], k1.y, v2);
        }
      }
    }
    float* dst = a.carry + (((size_t)c * a.H + h) * D + dg) * a.Dv + cg;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float lo[TC], hi[TC];
#pragma unroll
      for (int j = 0; j < TC; ++j) f2_unpair(acc[i][j], lo[j], hi[j]);
#pragma unroll
      for (int j = 0; j < TC; j += 4) {
        if (cg + 16 * j >= a.Dv) continue;
        *reinterpret_cast<float4*>(dst + (size_t)(2 * i) * a.Dv + 16 * j) = make_float4(lo[j], lo[j + 1], lo[j + 2], lo[j + 3]);
        *reinterpret_cast<float4*>(dst + (size_t)(2 * i + 1) * a.Dv + 16 * j) = make_float4(hi[j], hi[j + 1], hi[j + 2], hi[j + 3]);
      }
    }
  }
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

// Stages of the start state: 16 channels, half of them from each half.
template <int D, int TC>
struct GcOut {
  static constexpr int LD = D + 4, LP = kGcTokens + 4, kStage = 16 * 16 * TC, kBuffers = 4;
  float q[kGcTokens][LD];
  float s[kBuffers][kStage];
  float p[kGcTokens][LP];
  uint16_t v[kGcTokens][16 * TC];  // (bfloat16)
  float dec[kGcTokens];
  float next[16 * TC];             // a row of the state behind the chunk
  int odd;                         // whether a value of the chunk is infinite or NaN
};
// 8 tokens (eight apart: their rows lie in different banks) x TC columns (fours, 64 apart) a thread, and two threads for them: each takes half of
// the channels and half of the tokens (sums of 96 terms instead of 192, and 16 warps an SM).  Bound by the fmas.  The start state
// before P and V: small terms first (1.0e-7 off instead of 1.5e-7).  Fours of columns 64 apart: eight together cost two
// wavefronts a load (167 -> 132 us).
template <int D, int TC>
__global__ void __launch_bounds__(256, 2) gla_out_kernel(GlaArgs a) {
  pdl_wait();
  pdl_trigger();
  using Shared = GcOut<D, TC>;
  constexpr int kThreads = 256, LD = D + 4, LP = kGcTokens + 4, kStages = D / 16, kBuffers = Shared::kBuffers, kPer = kGcTokens * D / 8 / kThreads;
  extern __shared__ __align__(16) unsigned char gc_smem[];
  Shared& sh = *reinterpret_cast<Shared*>(gc_smem);
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  GcChunk x;
  if (!gc_chunk(a, c, x)) return;
  const int n = x.n, Dv = a.Dv;
  const float* start = a.carry + ((size_t)c * a.H + h) * D * Dv;
  auto fetch = [&](int st) {  // (a group of copies for every stage, an empty one behind the last)
    if (st < kStages) {
      float* to = sh.s[st % kBuffers];
      for (int i = tid; i < 16 * 4 * TC; i += kThreads) {
        const int d = i / (4 * TC), j = i % (4 * TC) * 4;
        const bool in = j < Dv;
        gla_cp16(to + d * 16 * TC + j, in ? start + (size_t)(8 * st + d + (d >> 3) * (D / 2 - 8)) * Dv + j : start, in);
      }
    }
    gla_cp_commit();
  };
  const __nv_bfloat16* vb = (const __nv_bfloat16*)a.v + (size_t)h * Dv;
  if (!a.a_head) {
    for (int i = tid; i < kGcTokens * (D / 4); i += kThreads) {
      const int t = i / (D / 4), d = i % (D / 4) * 4;
      gla_cp16(&sh.q[t][d], t < n ? a.z + ((x.row0 + t) * a.H + h) * D + d : a.z, t < n);
    }
  }
  fetch(0);  // (and the queries)
  for (int i = tid; i < kGcTokens * 2 * TC; i += kThreads) {
    const int t = i / (2 * TC), j = i % (2 * TC) * 8;
    const bool in = t < n && j < Dv;
    gla_cp16(&sh.v[t][j], in ? vb + (x.row0 + t) * a.v_stride + j : vb, in);
  }
  const float* pin = a.out + (x.row0 * a.H + h) * Dv;
  for (int i = tid; i < kGcTokens * (kGcTokens / 4); i += kThreads) {  // (what lies behind the diagonal was not written)
    const int t = i / (kGcTokens / 4), s = i % (kGcTokens / 4) * 4;
    gla_cp16(&sh.p[t][s], t < n ? pin + (size_t)t * a.H * Dv + s : pin, t < n && s <= t);
  }
  if (4 * tid < Dv) {
    const float* next = x.place + 1 < x.n_seg_chunks && c + 1 < a.n_chunks ? start + (size_t)a.H * D * Dv : a.state + ((size_t)x.slot * a.H + h) * D * Dv;
    gla_cp16(&sh.next[4 * tid], next + 4 * tid, true);
  }
  fetch(1);  // (and P and V)
  fetch(2);
  if (a.a_head) {  // one decay for all channels: the queries once more from their rows
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
      sh.dec[2 * tid] = (float)(before * w0);
      sh.dec[2 * tid + 1] = (float)(before * w1);
    }
    const __nv_bfloat16* qb = (const __nv_bfloat16*)a.q + (size_t)(h / a.qk_div) * D;
    const int d = tid % (D / 8) * 8, t0 = tid / (D / 8), step = kThreads / (D / 8);
    uint4 w[kPer];
    if (!a.rope) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) w[i] = *reinterpret_cast<const uint4*>(qb + (x.row0 + min(t0 + step * i, n - 1)) * a.q_stride + d);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int t = t0 + step * i;
      float y[8];
      if (a.rope) gc_rotated8(a, qb + (x.row0 + min(t, n - 1)) * a.q_stride, x.pos0 + min(t, n - 1), d, y);
      else gc_widen(w[i], y);
      const float f = a.q_scale * sh.dec[t];
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = t < n ? y[j] * f : 0.f;
      Vec4<float>::store(&sh.q[t][d], reinterpret_cast<float (&)[4]>(y[0]));
      Vec4<float>::store(&sh.q[t][d + 4], reinterpret_cast<float (&)[4]>(y[4]));
    }
  }
  const int cg = tid % 16 * 4, tg = tid / 16 % 8, half = tid / 128;
  uint64_t acc[8][TC / 2] = {};
  // four more of a row's terms: times four rows of columns in pairs
  auto step4 = [&](uint64_t (&row)[TC / 2], const float* at, const uint64_t (&y)[4][TC / 2]) {
    float f[4];
    Vec4<float>::load(at, f);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint64_t f2 = f2_pair(f[e], f[e]);
#pragma unroll
      for (int j = 0; j < TC / 2; ++j) f2_fma(row[j], f2, y[e][j]);
    }
  };
#pragma unroll 1
  for (int st = 0; st < kStages; ++st) {
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    static_assert(kBuffers == 4, "two stages in flight behind the one that is waited for");
    __syncthreads();
    fetch(st + kBuffers - 1);
    const float* from = sh.s[st % kBuffers] + half * 8 * 16 * TC + cg;
#pragma unroll
    for (int d = 0; d < 8; d += 4) {
      uint64_t y[4][TC / 2];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < TC / 2; j += 2) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(from + (d + e) * 16 * TC + 32 * j);
          y[e][j] = t.x; y[e][j + 1] = t.y;
        }
#pragma unroll
      for (int i = 0; i < 8; ++i) step4(acc[i], &sh.q[tg + 8 * i][half * (D / 2) + 8 * st + d], y);
    }
    if (st == 1 && tid < kGcTokens) {  // P has come: the rest of the 16-byte words on the diagonal
      for (int s = tid + 1; s <= (tid | 3); ++s) sh.p[tid][s] = 0.f;
    } else if (st == 1 && tid < kGcTokens + 32) {
      // Whether one of the chunk's values is infinite or NaN: what the chunk adds to its column of the state is then not finite,
      // nor is the state behind the chunk, of which one row tells.  (A row of P must then stop at its own token: what it has
      // behind is zero, and zero times such a value is NaN.)
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      if (4 * (tid - kGcTokens) < Dv) Vec4<float>::load(&sh.next[4 * (tid - kGcTokens)], y);
      const bool odd = __any_sync(0xffffffffu, !(fabsf(y[0]) < INFINITY && fabsf(y[1]) < INFINITY && fabsf(y[2]) < INFINITY && fabsf(y[3]) < INFINITY));
      if (tid == kGcTokens) sh.odd = odd;
    }
  }
  static_assert(kStages >= 4, "a barrier between P's last words, the flag and their readers");
  if (sh.odd) {  // token by token, each row up to its own
#pragma unroll 1
    for (int s = 4 * half; s < n; s += (s & 3) == 3 ? 5 : 1) {
      uint64_t y[TC / 2];
#pragma unroll
      for (int j = 0; j < TC / 2; j += 2) {
        const uint2 w = *reinterpret_cast<const uint2*>(&sh.v[s][cg + 32 * j]);
        y[j] = f2_pair(bf2_low(w.x), bf2_high(w.x));
        y[j + 1] = f2_pair(bf2_low(w.y), bf2_high(w.y));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (tg + 8 * i < s) continue;
        const float f = sh.p[tg + 8 * i][s];
        const uint64_t f2 = f2_pair(f, f);
#pragma unroll
        for (int j = 0; j < TC / 2; ++j) f2_fma(acc[i][j], f2, y[j]);
      }
    }
  } else {
#pragma unroll 1
    for (int s = 4 * half; s < n; s += 8) {
      uint64_t y[4][TC / 2];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int j = 0; j < TC / 2; j += 2) {
          const uint2 w = *reinterpret_cast<const uint2*>(&sh.v[s + e][cg + 32 * j]);
          y[e][j] = f2_pair(bf2_low(w.x), bf2_high(w.x));
          y[e][j + 1] = f2_pair(bf2_low(w.y), bf2_high(w.y));
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * i + 7 >= s) step4(acc[i], &sh.p[tg + 8 * i][s], y);  // (rows before s: zeros)
    }
  }
  // the upper threads' sums go through shared memory, where the stages lay
  __syncthreads();
  uint64_t* other = reinterpret_cast<uint64_t*>(sh.s) + (tid & 127);
  static_assert(sizeof(sh.s) >= 128 * 4 * TC * 8, "room for half of the sums");
  if (half) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TC / 2; ++j) other[(i * (TC / 2) + j) * 128] = acc[i][j];
  }
  __syncthreads();
  if (half) return;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TC / 2; ++j) acc[i][j] = f2_add(acc[i][j], other[(i * (TC / 2) + j) * 128]);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = tg + 8 * i;
    if (t >= n) continue;
    float* o = a.out + ((x.row0 + t) * a.H + h) * Dv + cg;
#pragma unroll
    for (int j = 0; j < TC / 2; j += 2) {
      if (cg + 32 * j >= Dv) continue;
      float4 f;
      f2_unpair(acc[i][j], f.x, f.y);
      f2_unpair(acc[i][j + 1], f.z, f.w);
      *reinterpret_cast<float4*>(o + 32 * j) = f;
    }
  }
}

// Whether a step's long portions go as products (the chunks are the host's: none may be longer than 64; where they do not pay the
// host names no length, parts/gla.py: longest_chunk).  Shorter chunks than 32 would leave more than half of a product's rows empty.  A
// layer, token by token against products, one request of 65, 128 and 256 tokens: 48 heads of 128 159 and 130, 167 and 138, 177 and
// 155 us; 16 heads of 64 87 and 65, 87 and 69, 95 and 69; one decay a head, 16 heads of 64 61 and 57, 61 and 61, 62 and 62.
inline bool gla_chunks_fit(const GlaArgs& a, int longest_chunk) {
  const uintptr_t at = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out | (uintptr_t)a.carry | (uintptr_t)a.state | (a.a_head ? 0 : (uintptr_t)a.z);
  return (a.D == 64 || a.D == 128) && a.Dv >= 64 && a.Dv <= 128 && a.Dv % 8 == 0 && !a.ones_col && longest_chunk >= 32 &&
         longest_chunk <= kGcTokens && (a.q_stride | a.k_stride | a.v_stride) % 8 == 0 && (at & 15) == 0;
}

template <int D, int TC>
static int launch_gla_chunks_as(const GlaArgs& a, cudaStream_t s) {
  auto local = gla_local_kernel<D, TC>;
  auto outs = gla_out_kernel<D, TC>;
  constexpr int sl = (int)sizeof(GcLocal<D, TC>), so = (int)sizeof(GcOut<D, TC>);
  FTK_REQUIRE(cudaFuncSetAttribute(local, cudaFuncAttributeMaxDynamicSharedMemorySize, sl) == cudaSuccess &&
                  cudaFuncSetAttribute(outs, cudaFuncAttributeMaxDynamicSharedMemorySize, so) == cudaSuccess,
              "gla_scan: cannot set up the chunk kernels");
  FTK_LAUNCH(local, dim3(a.n_chunks, a.H), 2 * D, sl, s, a);
  FTK_LAUNCH_CHECK("gla_scan (chunk products)");
  const size_t DV = (size_t)a.D * a.Dv;
  FTK_LAUNCH(gla_walk_kernel, dim3((unsigned)((DV / 2 + 255) / 256), a.n_segs, a.H), 256, 0, s, a);
  FTK_LAUNCH_CHECK("gla_scan (states)");
  FTK_LAUNCH(outs, dim3(a.n_chunks, a.H), 256, so, s, a);
  FTK_LAUNCH_CHECK("gla_scan (outputs)");
  return 0;
}

inline int launch_gla_chunks(const GlaArgs& a, cudaStream_t s) {
  if (a.D == 64) return a.Dv <= 64 ? launch_gla_chunks_as<64, 4>(a, s) : launch_gla_chunks_as<64, 8>(a, s);
  return a.Dv <= 64 ? launch_gla_chunks_as<128, 4>(a, s) : launch_gla_chunks_as<128, 8>(a, s);
}

}  // namespace ftk
