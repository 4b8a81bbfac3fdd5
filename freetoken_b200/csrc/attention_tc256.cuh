// The tcgen05 attention kernel for heads of 256 (and cached latent rows that wide).  Included by attention.cu after
// attention_tc.cuh, whose helpers and status words it uses.
//
// As in the one-tile kernel a tile is 128 query rows of one KV head and keys come in tiles of 128, but an output row takes
// 256 TMEM columns and a key tile 64 KB, so two things are laid out differently:
//   TMEM   S x2 (128 columns each) and O (256) fill all 512 columns; a tile's probabilities go as bfloat16 over the first 64
//          columns of its own scores.  S(j + 1) may overwrite P(j - 1) because the pipe executes a thread's products in the
//          order of issue: S(0) | S(1) P(0)V | S(2) P(1)V | ...
//   shared memory   Q (64 KB) and rings of key rows in steps of 64 (32 KB each).  One slab for keys and values (latent
//          attention): a ring of five, each given back as soon as the product over its 64 keys is done, so that most of the
//          next tile arrives under this tile's products; two whole tiles would leave a tile's load (about 1 us) in every
//          round.  Separate slabs: one key tile and one value tile.
// What bounds it: per key tile 16 products of 128 x 128 x 16 and 8 of 128 x 256 x 16, about 1.4 us of the tensor pipe at
// the rate this pipe takes them from one thread; the softmax (4 warps, a row a thread) runs under them.  48 heads on one
// cached row of 256, 2,048 tokens: 1,502 us on mma.sync (64-row tiles), 166 us here (620 TFLOP/s, the tensor pipe 36 % busy).
// It takes a window, kept first tokens and a sink; no bias by distance, no soft cap.  A KV head may be taken as `kv_split`
// heads of the same keys: 48 heads on one row fill 96 of a tile's 128 rows, three times 16 heads fill all of them.
#pragma once
#include "attention_tc.cuh"

namespace ftk {

constexpr int kTcWideD = 256;
constexpr int kTcWideSub = 64;                          // key rows per step of a ring
constexpr int kTcWideRingTied = 5, kTcWideRing = 2;      // steps per ring: one slab; keys and values apart
constexpr int kTcWideQHalf = 128 * 128;                  // bytes of 64 columns of the query tile
constexpr int kTcWideSmem = 4 * kTcWideQHalf + 4 * kTcWideRingTied * kTcWideSub * 128 + 1024;

__global__ void __launch_bounds__(kTcThreads)
attention_tc_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, AttnParams p) {
  extern __shared__ unsigned char dyn_smem[];
  __shared__ uint64_t q_full, q_empty, o_free, k_full[kTcWideRingTied], k_empty[kTcWideRingTied], v_full[kTcWideRing],
      v_empty[kTcWideRing], s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_work = p.n_items * p.Hkv;
  const int n_rounds = (n_work + (int)gridDim.x - 1) / (int)gridDim.x;
  auto piece = [&](int i) {  // rounds run to and fro over the CTAs: the list is sorted by length
    return i * (int)gridDim.x + ((i & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };
  const bool tied = p.k == p.v;
  const int ring_k = tied ? kTcWideRingTied : kTcWideRing;  // steps of the key ring
  const uint32_t k_half = (uint32_t)(ring_k * kTcWideSub * 128), v_half = (uint32_t)(kTcWideRing * kTcWideSub * 128);
  const uint32_t base = (smem_addr(dyn_smem) + 1023u) & ~1023u;
  unsigned char* tiles = dyn_smem + (base - smem_addr(dyn_smem));
  const uint32_t k_off = 4 * kTcWideQHalf, v_off = tied ? k_off : k_off + 4 * k_half;
  const uint32_t val_half = tied ? k_half : v_half;  // of the ring that holds the values

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    mbar_init(&q_empty, 1);
    mbar_init(&o_free, 4);
    for (int s = 0; s < kTcWideRingTied; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < kTcWideRing; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4); mbar_init(&pv_done[s], 1); }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();  // set up while the kernel before this one still runs; what it wrote is read from here on
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  volatile int* abortp = &abort_flag;
  const int G = p.G;
  auto tiles_of = [](const Item& it) { return it.ok ? (it.ke - it.kb + kTcKeys - 1) / kTcKeys : 0; };
  auto fail = [&](int code) {
    atomicCAS(&g_attn_status[0], 0, code);
    abort_flag = 1;
  };

  if (warp == 0 || warp == 6) {
    // ------------------------------------------------------------ TMA producers: warp 0 keys (and queries), warp 6 values
    // One lane per box of 16 keys x 64 columns: lane = 4 * (box of the step) + (column quarter).
    if (lane < 16 && !(warp == 6 && tied)) {
      const int kv = warp == 6, box = lane >> 2, h = lane & 3;
      const CUtensorMap* map = kv ? &map_v : &map_k;
      uint64_t* full = kv ? v_full : k_full;
      uint64_t* empty = kv ? v_empty : k_empty;
      const int ring = kv ? kTcWideRing : ring_k;
      unsigned char* dst0 = tiles + (kv ? v_off + h * v_half : k_off + h * k_half) + box * 2048;
      bool ok = true;
      int gs = 0;  // steps of all pieces so far
      int qi = 0;  // pieces with tiles so far
      for (int i_round = 0; i_round < n_rounds && ok; ++i_round) {
        const int w = piece(i_round);
        if (w >= n_work) continue;
        const Item it = load_item(p, p.n_items - 1 - w / p.Hkv);
        const int kvh = w % p.Hkv;
        const int n_tiles = tiles_of(it);
        if (n_tiles == 0) continue;
        if (!kv) {  // the queries, once the products of the piece before have read theirs
          if (!__all_sync(0x0000ffffu, mbar_wait(&q_empty, (uint32_t)(qi & 1) ^ 1u, abortp))) {
            if (lane == 0) fail(410);
            ok = false;
            break;
          }
          if (lane == 0) {
            mbar_expect_tx(&q_full, (uint32_t)(4 * 128 * G * (kTcRows / G)));
            for (int hh = 0; hh < 4; ++hh)  // (d, head, token): rows land as token-major, head-minor
              tma_load_3d(tiles + hh * kTcWideQHalf, &map_q, &q_full, hh * 64, kvh * G, it.q_start + it.tok0);
          }
        }
        ++qi;
        const int32_t* bt = p.block_table + (size_t)it.bt_row * p.bt_stride;
        const int slab_head = kvh / p.kv_split;
        auto page_of = [&](int u) {  // this lane's page of step u: looked up a step ahead
          const int key = it.kb + u * kTcWideSub + 16 * box;
          int page = 0;
          if (key < it.ke) {
            const int slot = (key + it.shift(p, key)) / p.P;
            page = slot < p.bt_stride ? bt[slot] : 0;
            if (page < 0 || page >= p.num_pages) page = 0;
          }
          return page;
        };
        int page_next = page_of(0);
        for (int u = 0; u < 2 * n_tiles && ok; ++u, ++gs) {
          const int st = gs % ring;
          const int key0 = it.kb + u * kTcWideSub;
          const int n_box = max(0, min(4, (it.ke - key0 + 15) >> 4));  // boxes that hold keys of the request
          const int key = key0 + 16 * box;
          const int page = page_next;
          page_next = page_of(u + 1);
          const int row = (page * p.slab_heads + slab_head) * p.P + (key + it.shift(p, key)) % p.P;
          if (!__all_sync(0x0000ffffu, mbar_wait(&empty[st], (uint32_t)((gs / ring) & 1) ^ 1u, abortp))) {
            if (lane == 0) fail(401 + kv);
            ok = false;
            break;
          }
          if (lane == 0) mbar_expect_tx(&full[st], (uint32_t)n_box * 4 * 2048);  // (no boxes: an arrival)
          __syncwarp(0x0000ffffu);
          if (box < n_box) tma_load_2d(dst0 + st * kTcWideSub * 128, map, &full[st], h * 64, row);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (lane 0); the warp zeroes dead value rows
    constexpr uint32_t idesc_qk = instr_desc(kTcKeys), idesc_qk_half = instr_desc(kTcWideSub);
    constexpr uint32_t idesc_pv = instr_desc(kTcWideD) | (1u << 16);  // B (values) MN-major
    const uint32_t q_s = base, k_s = base + k_off, v_s = base + v_off;
    uint64_t* val_full = tied ? k_full : v_full;
    uint64_t* val_empty = tied ? k_empty : v_empty;
    const int ring_v = tied ? ring_k : kTcWideRing;
    bool ok = true;
    int g0 = 0;  // tiles of the pieces before this one
    int qi = 0;  // pieces with tiles before this one
    for (int i_round = 0; i_round < n_rounds && ok; ++i_round) {
      const int w = piece(i_round);
      if (w >= n_work) continue;
      const Item it = load_item(p, p.n_items - 1 - w / p.Hkv);
      const int n_tiles = tiles_of(it);
      if (n_tiles == 0) continue;
      if (!all_of_warp(mbar_wait(&q_full, (uint32_t)(qi & 1), abortp))) {
        if (lane == 0) fail(403);
        ok = false;
        break;
      }
      bool fine = true;  // this lane's waits; the warp votes on them once a key tile
      for (int j = 0; j <= n_tiles && ok; ++j) {
        if (j < n_tiles) {
          const int g = g0 + j, s0 = (2 * g) % ring_k, s1 = (2 * g + 1) % ring_k;
          if (!mbar_wait2(&k_full[s0], (uint32_t)((2 * g) / ring_k) & 1u, &k_full[s1], (uint32_t)((2 * g + 1) / ring_k) & 1u, abortp)) { fail(404); fine = false; }
          tc_fence_after();
          if (elect_one()) if (fine) {
            const uint32_t d = tmem + (uint32_t)((g & 1) * kTcKeys);
            if (s1 > s0) {  // the tile's two steps lie one behind the other
#pragma unroll
              for (int kk = 0; kk < 16; ++kk) {  // 16 elements of the head dimension per MMA
                const uint64_t a = smem_desc(q_s + (kk >> 2) * kTcWideQHalf) + 2 * (kk & 3);
                const uint64_t b = smem_desc(k_s + (kk >> 2) * k_half + s0 * (kTcWideSub * 128)) + 2 * (kk & 3);
                tc_mma(d, a, b, idesc_qk, kk != 0);
              }
            } else {  // the ring's end lies between them
#pragma unroll 1
              for (int x = 0; x < 2; ++x) {
                const uint32_t rows = k_s + (x ? s1 : s0) * (kTcWideSub * 128);
#pragma unroll
                for (int kk = 0; kk < 16; ++kk) {
                  const uint64_t a = smem_desc(q_s + (kk >> 2) * kTcWideQHalf) + 2 * (kk & 3);
                  const uint64_t b = smem_desc(rows + (kk >> 2) * k_half) + 2 * (kk & 3);
                  tc_mma(d + x * kTcWideSub, a, b, idesc_qk_half, kk != 0);
                }
              }
            }
            if (!tied) { tc_commit(&k_empty[s0]); tc_commit(&k_empty[s1]); }
            tc_commit(&s_full[g & 1]);
            if (j == n_tiles - 1) tc_commit(&q_empty);  // the next piece's queries may come
          }
          __syncwarp();
        }
        if (j >= 1) {
          const int i = j - 1, g = g0 + i, s0 = (2 * g) % ring_v, s1 = (2 * g + 1) % ring_v;
          bool here = mbar_wait(&p_full[g & 1], (uint32_t)(g >> 1) & 1u, abortp);
          // (one slab: the steps have been waited for before the first product)
          if (here && !tied)
            here = mbar_wait2(&val_full[s0], (uint32_t)((2 * g) / ring_v) & 1u, &val_full[s1], (uint32_t)((2 * g + 1) / ring_v) & 1u, abortp);
          if (here && i == 0) here = mbar_wait(&o_free, (uint32_t)(qi & 1) ^ 1u, abortp);  // the piece before has read its output
          if (!here) { fail(405); fine = false; }
          // value rows that no row of the tile reads are zeroed, whatever lies there: in front of a window's first key
          // (but for the kept first tokens), and past the request's end
          const int key0 = it.kb + i * kTcKeys;
          auto clear = [&](int from, int to) {
            for (int x = lane; x < (to - from) * 32; x += 32) {
              const int r = from + (x >> 5), h = (x >> 3) & 3, c = x & 7;
              const int ring_row = (r < kTcWideSub ? s0 : s1) * kTcWideSub + (r & (kTcWideSub - 1));
              *reinterpret_cast<uint4*>(tiles + v_off + h * val_half + ring_row * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_async_smem();
          };
          if (p.window > 0) {
            const int first = key0 + it.shift(p, key0);
            const int from = max(0, p.keep_first - first), dead = min(kTcKeys, it.lo - first);
            if (dead > from) clear(from, dead);
          }
          if (it.ke - key0 < kTcKeys) clear(it.ke - key0, kTcKeys);
          __syncwarp();
          tc_fence_after();
          if (elect_one()) if (fine) {
            const uint32_t d = tmem + 2 * kTcKeys;
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {  // 16 keys per MMA
              const uint32_t a = tmem + (uint32_t)((g & 1) * kTcKeys + kk * 8);
              const uint64_t b = smem_desc_mn(v_s + (kk < 4 ? s0 : s1) * (kTcWideSub * 128) + (kk & 3) * 2048, val_half);
              tc_mma_ts(d, a, b, idesc_pv, (i | kk) != 0);
              if (kk == 3) tc_commit(&val_empty[s0]);
            }
            tc_commit(&val_empty[s1]);
            tc_commit(&pv_done[g & 1]);
          }
          __syncwarp();
        }
        ok = all_of_warp(fine);
      }
      g0 += n_tiles;
      ++qi;
    }
  } else {
    // ------------------------------------------------------------ softmax and epilogue (warps 2..5), one row per thread
    const int quad = warp & 3;
    const int r = quad * 32 + lane;  // row of the tile = TMEM lane
    const float sl2 = p.scale * 1.4426950408889634f;
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
    const uint32_t o_addr = lane_addr + 2 * kTcKeys;
    bool ok = true;
    int g0 = 0;  // tiles of the pieces before this one
    for (int i_round = 0; i_round < n_rounds && ok; ++i_round) {
      const int w = piece(i_round);
      if (w >= n_work) continue;
      const Item it = load_item(p, p.n_items - 1 - w / p.Hkv);
      const int kvh = w % p.Hkv;
      const int n_tiles = tiles_of(it);
      const int R = it.ok ? it.ntok * G : 0;
      const int pos_base = it.kv_len - it.q_len + it.tok0;
      const int qpos = r < R ? pos_base + r / G : -1;
      // what the row may read: as in the one-tile kernel
      const int hi = r < R ? (p.keep_span ? qpos : min(it.ke - 1, qpos)) : 0x7fffffff;
      const int lo = (p.window > 0 && r < R) ? max(0, qpos - p.window + 1) : 0;
      const int keep = p.keep_first;
      const unsigned int hidden = (unsigned int)max(0, lo - keep);
      float m_used = -INFINITY, l = 0.f;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int g = g0 + j;
        if (!__all_sync(0xffffffffu, mbar_wait(&s_full[g & 1], (uint32_t)((g >> 1) & 1), abortp))) {
          if (lane == 0) fail(406);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t s_addr = lane_addr + (uint32_t)((g & 1) * kTcKeys);
        const int key0 = it.kb + j * kTcKeys + it.shift(p, it.kb + j * kTcKeys);
        const bool interior = __all_sync(0xffffffffu, key0 + kTcKeys - 1 <= hi && (key0 >= lo || key0 + kTcKeys <= keep));
        float v[128];
        tmem_ld32_start(s_addr, v);
        tmem_ld32_start(s_addr + 32, v + 32);
        tmem_ld32_start(s_addr + 64, v + 64);
        tmem_ld32_start(s_addr + 96, v + 96);
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32_finish(reinterpret_cast<float(&)[32]>(v[32 * c]));
        if (!interior) {
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (key0 + i > hi || (unsigned int)(key0 + i - keep) < hidden) v[i] = -INFINITY;
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], v[i]);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;  // the scale is positive
        // move the running maximum only when it grew by more than 8 (or is not set yet)
        float alpha = 1.f;
        if (mx > m_used + 8.f || (m_used == -INFINITY && mx > -INFINITY)) {
          alpha = m_used == -INFINITY ? 0.f : tc_exp2(m_used - mx);
          m_used = mx;
        }
        l *= alpha;
        if (__any_sync(0xffffffffu, alpha != 1.f) && j > 0) {  // O must hold every product so far before it is scaled
          if (!__all_sync(0xffffffffu, mbar_wait(&pv_done[(g - 1) & 1], (uint32_t)(((g - 1) >> 1) & 1), abortp))) {
            if (lane == 0) fail(409);
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < kTcWideD / 32; ++c) {
            float o[32];
            tmem_ld32(o_addr + c * 32, o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= alpha;
            tmem_st32(o_addr + c * 32, o);
          }
        }
        const float mb = m_used == -INFINITY ? 0.f : m_used;
        float sum[2] = {0.f, 0.f};
        // probabilities as bfloat16 over the first 64 columns of the scores (which are all in registers by now)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = tc_exp2(fmaf(v[c * 32 + i], sl2, -mb));  // exp2(-inf) = 0 for masked keys
            const float p1 = tc_exp2(fmaf(v[c * 32 + i + 1], sl2, -mb));
            sum[0] += p0;
            sum[1] += p1;
            pk[i >> 1] = tc_pack(p0, p1);
          }
          tmem_st16u(s_addr + (uint32_t)(c * 16), pk);
        }
        l += sum[0] + sum[1];
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g & 1]);
      }
      // ---- epilogue
      if (ok && n_tiles > 0) {
        // (two barriers: the last tile's product may still have the one before it in flight, whose phase has the same parity)
        const int gl = g0 + n_tiles - 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&pv_done[gl & 1], (uint32_t)((gl >> 1) & 1), abortp))) {
          if (lane == 0) fail(408);
          ok = false;
        }
        tc_fence_after();
      }
      if (ok && it.ok) {
        const bool live = n_tiles > 0;
        const int tok = it.q_start + it.tok0 + r / G;
        if (it.nsplit == 1) {
          // (a sink in the denominator: e^sink relative to the running maximum, which is in the exp2 domain)
          const float lt = l + (p.has_sink ? exp2f((p.sink_heads ? __ldg(p.sink_heads + kvh * G + r % G) : p.sink) * 1.4426950408889634f - m_used) : 0.f);
          const float inv = lt > 0.f ? 1.f / lt : 0.f;
          __nv_bfloat16* dst = (__nv_bfloat16*)p.out + ((size_t)tok * p.Hq + kvh * G + r % G) * kTcWideD;
#pragma unroll 1
          for (int c = 0; c < kTcWideD / 32; ++c) {
            float o[32];
            if (live) tmem_ld32(o_addr + c * 32, o);
            if (r < R) {
#pragma unroll
              for (int q4 = 0; q4 < 4; ++q4) {
                uint4 pk;
                pk.x = tc_pack(live ? o[8 * q4] * inv : 0.f, live ? o[8 * q4 + 1] * inv : 0.f);
                pk.y = tc_pack(live ? o[8 * q4 + 2] * inv : 0.f, live ? o[8 * q4 + 3] * inv : 0.f);
                pk.z = tc_pack(live ? o[8 * q4 + 4] * inv : 0.f, live ? o[8 * q4 + 5] * inv : 0.f);
                pk.w = tc_pack(live ? o[8 * q4 + 6] * inv : 0.f, live ? o[8 * q4 + 7] * inv : 0.f);
                *reinterpret_cast<uint4*>(dst + c * 32 + q4 * 8) = pk;
              }
            }
          }
        } else {
          const size_t slot = ((size_t)(it.base + it.split) * p.Hkv + kvh) * p.tile_rows + r;
#pragma unroll 1
          for (int c = 0; c < kTcWideD / 32; ++c) {
            float o[32];
            if (live) tmem_ld32(o_addr + c * 32, o);
            if (r < R) {
#pragma unroll
              for (int q4 = 0; q4 < 8; ++q4)
                *reinterpret_cast<float4*>(p.part_o + slot * kTcWideD + c * 32 + q4 * 4) =
                    live ? make_float4(o[4 * q4], o[4 * q4 + 1], o[4 * q4 + 2], o[4 * q4 + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
          if (r < R) {
            p.part_ml[slot * 2] = m_used == -INFINITY ? -INFINITY : m_used * 0.6931471805599453f;
            p.part_ml[slot * 2 + 1] = l;
          }
        }
      }
      if (n_tiles > 0) {  // the output accumulator has been read: the next piece's first product may overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_free);
      }
      g0 += n_tiles;
    }
  }
  // ---------------------------------------------------------------- teardown
  if (abort_flag) {
    if (threadIdx.x == 0) g_attn_status[1] = blockIdx.x;
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // let copies in flight land before the CTA leaves
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

inline int launch_attention_tc_wide(const AttnParams& p, int n_tokens, cudaStream_t s) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attention_tc_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcWideSmem) != cudaSuccess) return 2;
    configured = true;
  }
  CUtensorMap mq, mk, mv;
  {
    // queries [T, Hq, D] seen as (d, head, token); a box is (64, group, tokens per tile)
    const uint64_t dims[3] = {(uint64_t)kTcWideD, (uint64_t)p.Hq, (uint64_t)n_tokens};
    const uint64_t strides[2] = {(uint64_t)kTcWideD * 2, (uint64_t)p.Hq * kTcWideD * 2};
    const uint32_t box[3] = {64, (uint32_t)p.G, (uint32_t)(kTcRows / p.G)};
    if (!make_map(&mq, p.q, 3, dims, strides, box)) return 4;
  }
  {
    // a slab [pages, heads, P, D] seen as rows of D; a box is 16 rows of one page x 64 elements
    const uint64_t dims[2] = {(uint64_t)kTcWideD, (uint64_t)p.num_pages * p.slab_heads * p.P};
    const uint64_t strides[1] = {(uint64_t)kTcWideD * 2};
    const uint32_t box[2] = {64, 16};
    if (!make_map(&mk, p.k, 2, dims, strides, box) || !make_map(&mv, p.v, 2, dims, strides, box)) return 4;
  }
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 1;
  }
  const long long n_work = (long long)p.n_items * p.Hkv;  // one CTA per SM, each takes every sms-th piece of work
  const int grid = (int)(n_work < sms ? n_work : sms);
  FTK_LAUNCH(attention_tc_wide_kernel, grid, kTcThreads, kTcWideSmem, s, mq, mk, mv, p);
  return 0;
}

}  // namespace ftk
