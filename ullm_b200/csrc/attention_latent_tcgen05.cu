// Paged attention of prompt portions over latent keys in bfloat16 on the 5th-generation tensor cores: ONE kv head whose rows
// are dk elements wide and whose values are the first dv elements of the same rows, shared by all query heads (absorbed latent
// attention: dk = 448, dv = 384 for a latent of 384 and a rotated part of 64).
//
// Bound by the tensor cores: a (query, key) pair costs 2 (dk + dv) operations per head, 56 GFLOP for 2,048 tokens of 16 heads,
// 35 us at the card's rate.  The mma.sync kernel of attention_window.cu took 361 us there: its three column groups form the
// weights three times over and exchange partial scores through shared memory.
//
// A block owns 128 rows, (token, head) pairs of one request, so that every key row that is loaded serves all heads of 128 /
// heads tokens.  It walks the keys 64 at a time; a tile of key rows is loaded ONCE and is both operands: K (K-major) of the
// scores and V (MN-major, its first dv columns) of the output.
//
//   S[128 x 64]   = Q K^T     dk / 16 steps, A and B from shared memory; two accumulators of 64 columns in turn
//   P             = 2^(S * scale - m)   one thread per row; written as packed bfloat16 over the first half of S's columns
//   O[128 x dv]  += P V       A from tensor memory; two products of at most 192 columns (O takes 384 columns of tensor memory,
//                             S the other 128)
//
// The MMA thread issues S of the next tile before P V of this one whenever that tile has landed, so that the softmax of a tile
// runs behind the products of its neighbours.  Shared memory: Q (112 KB at dk = 448) and two key tiles (56 KB each): 128-key
// tiles would leave room for one only.  The reference point of a row's exponents moves only when its maximum grows by more than
// 2^8, as in attention_prefill_pair.cu; O is rescaled in tensor memory then.
//
// Every wait on an mbarrier is bounded (ULLM_STATUS_TIMEOUT in the status word; the block then waits, bounded, for the copies that
// it has in flight, and leaves).
#include <cuda.h>

#include "common.cuh"
#include "tcgen05_attention.cuh"
#include "tma_host.cuh"

#define LA_ROWS 128
#define LA_KEYS 64
#define LA_THREADS 192  // warps 0-3: softmax; 4: loads; 5: MMA
#define LA_MAX_DK 448
#define LA_MAX_DV 384
#define LA_CHUNK_Q (LA_ROWS * 128)  // 64 columns of the rows
#define LA_CHUNK_K (LA_KEYS * 128)
#define LA_BARRIER_BYTES 256

struct LaParams {
  const int* block_table;
  const int* req_slots;
  const int* cu_q;
  const int* kv_len;
  __nv_bfloat16* out;
  long long out_stride;
  int* status;
  int max_pages, num_requests, heads, nk, nv, page_size, window;  // nk, nv: key and value columns / 64
  float scale_log2;
  long long num_pages;
};

__global__ void __launch_bounds__(LA_THREADS, 1)
latent_attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const LaParams p) {
  // (no static shared memory, so that the dynamic region starts on a 1024-byte boundary; if it did not, the block would leave)
  extern __shared__ __align__(16) unsigned char la_raw[];
  if ((tp_smem(la_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 60, (int)(tp_smem(la_raw) & 1023u));
    return;
  }
  unsigned char* q_s = la_raw;
  unsigned char* k_s = q_s + p.nk * LA_CHUNK_Q;
  const int k_bytes = p.nk * LA_CHUNK_K;
  uint64_t* bars = reinterpret_cast<uint64_t*>(k_s + 2 * k_bytes);
  uint64_t& q_full = bars[0];
  uint64_t* k_full = bars + 1;   // [2] the key tile has landed
  uint64_t* k_empty = bars + 3;  // [2] P V of the tile is done: nothing reads it any more, and O holds it
  uint64_t* s_full = bars + 5;   // [2] the scores are in tensor memory
  uint64_t* p_ready = bars + 7;  // [2] the weights are (one arrival per warp)
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 9);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.heads, tpt = LA_ROWS / G;  // tokens of a block
  pdl_wait();

  // ---- which request and which of its token tiles (numbered from the back: those with the most keys first) ----------
  const int tile_id = (int)gridDim.x - 1 - (int)blockIdx.x;
  int r = -1, first = 0, q_len = 0, q_begin = 0;
  {
    int running = 0;
    for (int i = 0; i < p.num_requests; ++i) {
      const int b = p.cu_q[i], n = p.cu_q[i + 1] - b, nt = (n + tpt - 1) / tpt;
      if (tile_id < running + nt) {
        r = i;
        first = (tile_id - running) * tpt;
        q_len = n;
        q_begin = b;
        break;
      }
      running += nt;
    }
  }
  if (r < 0) return;
  const int kvl = p.kv_len[r], ntok = min(tpt, q_len - first), rows_valid = ntok * G;
  const int p0 = kvl - q_len + first;  // position of the block's first token
  const int dv = p.nv * 64;
  if (kvl <= 0 || p0 < 0) {
    for (int i = tid; i < rows_valid * dv; i += LA_THREADS) {
      const int row = i / dv, d = i - row * dv;
      p.out[(long long)(q_begin + first + row / G) * p.out_stride + (long long)(row % G) * dv + d] = __float2bfloat16_rn(0.f);
    }
    return;
  }
  const int first_key = first_seen(p0, p.window), last_key = p0 + ntok - 1;  // what some row of the block sees
  const int k_start = first_key / LA_KEYS * LA_KEYS;
  const int tiles = (last_key - k_start) / LA_KEYS + 1;
  const int* bt = p.block_table + (long long)p.req_slots[r] * p.max_pages;

  if (tid == 0) {
    tp_mbar_init(&q_full, 1);
    for (int s = 0; s < 2; ++s) {
      tp_mbar_init(&k_full[s], 1);
      tp_mbar_init(&k_empty[s], 1);
      tp_mbar_init(&s_full[s], 1);
      tp_mbar_init(&p_ready[s], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tp_smem(&tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    // (Only now: a kernel behind this one must not hold tensor memory that this one waits for; and only behind pdl_wait(): decode attention
    // beside this kernel takes its own start for the end of everything in front of this one.)
    pdl_launch_dependents();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot, tmem_s0 = tmem + LA_MAX_DV;  // O in columns 0 .. dv - 1, S in 384 + 64 (tile & 1)

  if (warp == 4) {
    // ---- loads: lane pg knows page pg of the tile, the tile's boxes (a page x 64 columns) are dealt over the lanes ----
    if (lane == 0) tp_mbar_expect_tx(&q_full, p.nk * LA_CHUNK_Q);
    __syncwarp();
    if (lane < p.nk) tp_tma_3d(q_s + lane * LA_CHUNK_Q, &map_q, &q_full, lane * 64, 0, q_begin + first);
    const int ppt = LA_KEYS / p.page_size, boxes = p.nk * ppt;
    auto page_of = [&](int t) -> int {
      const int key = k_start + t * LA_KEYS + lane * p.page_size;
      int page = -1;
      if (lane < ppt && key < kvl) {
        // A page that some row sees has to be there.  (A tile may begin before the first key any row sees; pages there may have
        // been given back: zero-filled and masked.)
        page = bt[key / p.page_size];
        if (page < 0 || page >= p.num_pages) {
          if (key + p.page_size > first_key && key <= last_key) ullm_report(p.status, ULLM_STATUS_PAGE, r, page);
          page = -1;
        }
      }
      return page >= 0 ? page : (int)p.num_pages;  // (out of the map's range: the box is filled with zeros)
    };
    int pages = page_of(0), issued = 0;
    bool ok = true;
    for (int t = 0; t < tiles && ok; ++t) {
      const int next = t + 1 < tiles ? page_of(t + 1) : 0;
      const int s = t & 1;
      if (lane == 0 && !tp_mbar_wait(&k_empty[s], ((t >> 1) & 1) ^ 1)) {
        ullm_report(p.status, ULLM_STATUS_TIMEOUT, 61, t);
        ok = false;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      if (lane == 0) tp_mbar_expect_tx(&k_full[s], k_bytes);
      __syncwarp();
      for (int b0 = 0; b0 < boxes; b0 += 32) {
        const int b = b0 + lane, pg = b % ppt, page = __shfl_sync(0xffffffffu, pages, pg);
        if (b < boxes)
          tp_tma_4d(k_s + s * k_bytes + (b / ppt) * LA_CHUNK_K + pg * p.page_size * 128, &map_k, &k_full[s], (b / ppt) * 64, 0, 0,
                    page);
      }
      pages = next;
      issued = t + 1;
    }
    if (lane == 0) {  // (a block in which a role gave up does not leave copies behind that are still on their way)
      tp_mbar_wait(&q_full, 0);
      for (int t = max(0, issued - 2); t < issued; ++t) tp_mbar_wait(&k_full[t & 1], (t >> 1) & 1);
    }
    __syncwarp();
  } else if (warp == 5) {
    if (lane == 0) {
      // ---- MMA --------------------------------------------------------------------------------------------------
      const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LA_KEYS >> 3) << 17) |
                               ((uint32_t)(LA_ROWS >> 4) << 24);
      // O in one product, or (more than 256 columns) in two: N0 and N1 chunks of 64 columns; B is MN-major
      const int n0 = p.nv <= 4 ? p.nv : (p.nv + 1) / 2, n1 = p.nv - n0;
      const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(LA_ROWS >> 4) << 24);
      const uint32_t idesc_o0 = idesc_o | ((uint32_t)(n0 * 8) << 17), idesc_o1 = idesc_o | ((uint32_t)(n1 * 8) << 17);
      const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
      const uint32_t q_lo = ((tp_smem(q_s) & 0x3FFFF) >> 4) | (1u << 16);
      const uint32_t k_addr = (tp_smem(k_s) & 0x3FFFF) >> 4;
      auto mma_ss = [&](uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t acc) {
        asm volatile(
            "{\n .reg .b64 da, db;\n .reg .pred p;\n mov.b64 da, {%1, %3};\n mov.b64 db, {%2, %3};\n"
            " setp.ne.b32 p, %5, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n}\n"
            ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc_s), "r"(acc)
            : "memory");
      };
      auto mma_ts = [&](uint32_t d, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
        asm volatile(
            "{\n .reg .b64 db;\n .reg .pred p;\n mov.b64 db, {%2, %3};\n"
            " setp.ne.b32 p, %5, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}\n"
            ::"r"(d), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(acc)
            : "memory");
      };
      auto scores = [&](int t) {
        const uint32_t k_lo = (k_addr + (t & 1) * (k_bytes >> 4)) | (1u << 16), d = tmem_s0 + (t & 1) * LA_KEYS;
        for (int c = 0; c < p.nk; ++c) {
          const uint32_t a = q_lo + c * (LA_CHUNK_Q >> 4), b = k_lo + c * (LA_CHUNK_K >> 4);
          mma_ss(d, a, b, c > 0 ? 1u : 0u);
          mma_ss(d, a + 2, b + 2, 1u);
          mma_ss(d, a + 4, b + 4, 1u);
          mma_ss(d, a + 6, b + 6, 1u);
        }
        tp_commit(&s_full[t & 1]);
      };
      bool ok = tp_mbar_wait(&q_full, 0);
      if (!ok) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 62, 0);
      if (ok && !tp_mbar_wait(&k_full[0], 0)) {
        ullm_report(p.status, ULLM_STATUS_TIMEOUT, 63, 0);
        ok = false;
      }
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        scores(0);
      }
      for (int t = 0; t < tiles && ok; ++t) {
        // the next tile's scores first if the tile is there; else behind this tile's output product
        const bool more = t + 1 < tiles;
        bool scored = false;
        if (more && tp_mbar_test(&k_full[(t + 1) & 1], ((t + 1) >> 1) & 1)) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          scores(t + 1);
          scored = true;
        }
        if (!tp_mbar_spin(&p_ready[t & 1], (t >> 1) & 1)) {
          ullm_report(p.status, ULLM_STATUS_TIMEOUT, 64, t);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // (MN-major: the leading-dimension field is the distance of neighbouring chunks of 64 columns)
        const uint32_t v_lo = (k_addr + (t & 1) * (k_bytes >> 4)) | ((uint32_t)(LA_CHUNK_K >> 4) << 16);
        const uint32_t w = tmem_s0 + (t & 1) * LA_KEYS;
#pragma unroll
        for (int ks = 0; ks < LA_KEYS / 16; ++ks) {  // 16 keys: 8 columns of P, two 8-key groups of the tile
          const uint32_t acc = (t > 0 || ks > 0) ? 1u : 0u;
          mma_ts(tmem, w + ks * 8, v_lo + ks * (2048 >> 4), idesc_o0, acc);
          if (n1 > 0) mma_ts(tmem + n0 * 64, w + ks * 8, v_lo + n0 * (LA_CHUNK_K >> 4) + ks * (2048 >> 4), idesc_o1, acc);
        }
        tp_commit(&k_empty[t & 1]);
        if (more && !scored) {
          if (!tp_mbar_wait(&k_full[(t + 1) & 1], ((t + 1) >> 1) & 1)) {
            ullm_report(p.status, ULLM_STATUS_TIMEOUT, 63, t + 1);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          scores(t + 1);
        }
      }
    }
  } else {
    // ---- softmax: a thread owns row `tid` (tensor-memory lane `tid`) ------------------------------------------------
    const int row = tid;
    const bool row_ok = row < rows_valid;
    const int pos = row_ok ? p0 + row / G : -1, lo = first_seen(pos, p.window);
    const int lo_last = first_seen(p0 + ntok - 1, p.window);  // what the block's last token sees first
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int t = 0; t < tiles && ok; ++t) {
      const int key0 = k_start + t * LA_KEYS;
      if (!tp_mbar_wait(&s_full[t & 1], (t >> 1) & 1)) {
        if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 65, t);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_s = tmem_s0 + (t & 1) * LA_KEYS + lane_base;
      uint32_t sr[LA_KEYS];
      tp_tmem_ld32_nowait(tmem_s, sr);
      tp_tmem_ld32_nowait(tmem_s + 32, sr + 32);
      tp_tmem_ld_wait();
      if (rows_valid < LA_ROWS || key0 + LA_KEYS - 1 > p0 || key0 < lo_last) {
#pragma unroll
        for (int k = 0; k < LA_KEYS; ++k)
          if (!(key0 + k <= pos && key0 + k >= lo)) sr[k] = 0xff800000u;  // -inf
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int k = 0; k < LA_KEYS / 2; ++k)
        mx[k & 3] = tp_max3(mx[k & 3], __uint_as_float(sr[2 * k]), __uint_as_float(sr[2 * k + 1]));
      const float m_cand = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
      const float m_new = (m == -INFINITY || m_cand - m > 8.f) ? m_cand : m;
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = m == -INFINITY ? 1.f : tp_ex2(m - m_use);  // (no key seen yet: O and l are still zero)
      m = m_new;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const float a = tp_ex2(fmaf(__uint_as_float(sr[2 * k]), p.scale_log2, -m_use));
        const float b = tp_ex2(fmaf(__uint_as_float(sr[2 * k + 1]), p.scale_log2, -m_use));
        sum[(2 * k) & 3] += a;
        sum[(2 * k + 1) & 3] += b;
        pk[k] = tp_pack_bf16(a, b);
      }
      tp_tmem_st32_nowait(tmem_s, pk);
      l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      // Slots past the request's length may hold anything, which must not reach O.  The scores that read the tile are done
      // (awaited above), its output product is not issued yet: the columns that serve as values are cleared.
      if (key0 + LA_KEYS > kvl) {
        unsigned char* v_t = k_s + (t & 1) * k_bytes;
        const int first_bad = max(0, kvl - key0), pieces = p.nv * 8;
        for (int x = row; x < (LA_KEYS - first_bad) * pieces; x += 128) {
          const int key = first_bad + x / pieces, ch = x % pieces;
          *reinterpret_cast<uint4*>(v_t + (ch >> 3) * LA_CHUNK_K + key * 128 + (ch & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      if (t > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // O shares the reference point: once the product of the tile before is in it, this warp's rows are rescaled
        if (!tp_mbar_wait(&k_empty[(t - 1) & 1], ((t - 1) >> 1) & 1)) {
          if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 66, t);
          ok = false;
        } else {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c = 0; c < dv; c += 8) {
            uint32_t v[8];
            tp_tmem_ld8_nowait(tmem + lane_base + c, v);
            tp_tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * alpha);
            tp_tmem_st8_nowait(tmem + lane_base + c, v);
          }
        }
      }
      tp_tmem_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tp_mbar_arrive(&p_ready[t & 1]);  // (also after a failed wait: the MMA thread is not left waiting)
    }
    if (ok && !tp_mbar_wait(&k_empty[(tiles - 1) & 1], ((tiles - 1) >> 1) & 1)) {
      if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 67, tiles);
      ok = false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const float inv = l > 0.f ? 1.f / l : 0.f;
    __nv_bfloat16* op = p.out + (long long)(q_begin + first + row / G) * p.out_stride + (long long)(row % G) * dv;
#pragma unroll 1
    for (int c = 0; c < dv; c += 32) {
      uint32_t v[32];
      tp_tmem_ld32_nowait(tmem + lane_base + c, v);  // (all lanes of the warp take part)
      tp_tmem_ld_wait();
      if (row_ok && ok) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 x;
          x.x = tp_pack_bf16(__uint_as_float(v[q * 8 + 0]) * inv, __uint_as_float(v[q * 8 + 1]) * inv);
          x.y = tp_pack_bf16(__uint_as_float(v[q * 8 + 2]) * inv, __uint_as_float(v[q * 8 + 3]) * inv);
          x.z = tp_pack_bf16(__uint_as_float(v[q * 8 + 4]) * inv, __uint_as_float(v[q * 8 + 5]) * inv);
          x.w = tp_pack_bf16(__uint_as_float(v[q * 8 + 6]) * inv, __uint_as_float(v[q * 8 + 7]) * inv);
          *reinterpret_cast<uint4*>(op + c + q * 8) = x;
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// One kv head of dk = a multiple of 64 up to 448 with values in its first dv = a multiple of 64 up to 384 elements, a power-of-two
// number (up to 128) of query heads, pages of 8 to 64 tokens.
extern "C" int ullm_latent_attention_supported(int dk, int dv, int num_q, int num_kv, int page_size) {
  if (num_kv != 1 || num_q <= 0 || num_q > LA_ROWS || (num_q & (num_q - 1))) return 0;
  if (dk <= 0 || dk % 64 || dk > LA_MAX_DK || dv <= 0 || dv % 64 || dv > LA_MAX_DV || dv > dk) return 0;
  return page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64;
}

// Arguments as `ullm_window_attention` with values inside the key rows and none of its options.  UNSUPPORTED where rows do not
// start on 16-byte borders.
extern "C" int ullm_latent_attention(const void* q, long long q_row_stride, void* out, long long out_stride,
                                     const void* k_cache, const int* block_table, int max_pages, const int* req_slots,
                                     const int* cu_q, const int* kv_len, int tokens, int num_requests, int num_q, int num_kv,
                                     int dk, int dv, int page_size, int window, float scale, long long num_pages, int* status,
                                     void* stream) {
  if (tokens < 0 || num_requests <= 0 || max_pages <= 0) return ULLM_ERR_BAD_SIZE;
  if (!ullm_latent_attention_supported(dk, dv, num_q, num_kv, page_size)) return ULLM_ERR_UNSUPPORTED;
  if (q_row_stride % 8 || out_stride % 8 || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)out) & 15)) return ULLM_ERR_UNSUPPORTED;
  if (q_row_stride < (long long)num_q * dk || out_stride < (long long)num_q * dv || num_pages >= 0x7fffffffLL) return ULLM_ERR_BAD_SIZE;
  if (tokens == 0) return ULLM_OK;
  UllmTmaEncodeFn enc = ullm_tma_encode();
  if (enc == nullptr) return ULLM_ERR_LAUNCH;
  // Q: [tokens][heads][dk]; a box gathers 64 columns of the heads of a block's tokens
  const int tpt = LA_ROWS / num_q;
  CUtensorMap mq, mk;
  cuuint64_t dims[3] = {(cuuint64_t)dk, (cuuint64_t)num_q, (cuuint64_t)tokens};
  cuuint64_t strides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)q_row_stride * 2};
  cuuint32_t box[3] = {64, (cuuint32_t)num_q, (cuuint32_t)tpt};
  cuuint32_t estr[3] = {1, 1, 1};
  if (enc(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      !ullm_tma_map_kv(k_cache, num_pages, page_size, 1, dk, page_size, &mk))
    return ULLM_ERR_LAUNCH;
  const size_t smem = (size_t)(dk / 64) * (LA_CHUNK_Q + 2 * LA_CHUNK_K) + LA_BARRIER_BYTES;
  static size_t have = 0;
  if (smem > have) {
    if (cudaFuncSetAttribute(latent_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have = smem;
  }
  LaParams p = {};
  p.block_table = block_table;
  p.req_slots = req_slots;
  p.cu_q = cu_q;
  p.kv_len = kv_len;
  p.out = (__nv_bfloat16*)out;
  p.out_stride = out_stride;
  p.status = status;
  p.max_pages = max_pages;
  p.num_requests = num_requests;
  p.heads = num_q;
  p.nk = dk / 64;
  p.nv = dv / 64;
  p.page_size = page_size;
  p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.num_pages = num_pages;
  return ullm_launch_kernel(latent_attention_kernel, dim3((tokens + tpt - 1) / tpt + num_requests), dim3(LA_THREADS), smem,
                            (cudaStream_t)stream, mq, mk, p);
}
