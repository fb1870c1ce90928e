// Paged causal attention in 32-bit arithmetic for head sizes 64 and 128: what the 32-bit engine and float16 run instead of
// the general kernel (attention_generic.cu) where no option beyond a window or a stretch of positions is asked for.  Rows of
// the batch, positions, windows and the block tables as there; every product, sum, maximum and exponential is 32-bit.
//
// The general kernel gives a warp one (token, head): each lane walks a key of its own (rows 512 bytes apart), a key is read
// once per query row, and a dot product is one serial chain of head_dim multiply-adds.  At Qwen3-0.6B sizes that took 749 us
// per layer for prompts of 170 + 341 tokens and 589 us for 8 decoded tokens with 300 to 700 keys; these two take 51 and 29 us:
//
//   * rows of prompt portions (requests that bring more than one token): a block owns PT_ROWS (token, query head) rows of ONE
//     kv head.  Two groups of 128 threads walk the keys, 32 at a time and in turn, each with K and V of its tile in shared memory
//     and with maxima, sums and outputs of its own, which meet at the end: one loads while the other multiplies, and the longest
//     row tile, which sets the time at the prompt lengths of a step (hundreds of tokens), is walked in half the turns.  A thread
//     forms 4 rows x 2 keys of the scores and 4 rows x 8 columns of the output from 16-byte reads.  One group with tiles of 64 keys:
//     prompts of 170 + 341 tokens 81 us, 100 tokens 30, 500 108, 2,048 861; two of 32: 69, 24, 91, 749 (16 query heads of 128); with
//     K and V of the next tile on their way (cp.async; K behind the scores, V behind the outputs) 67, 24, 87, 710; with two multiply-
//     adds an instruction (fma.rn.f32x2: even and odd channels of a score sum up apart) 63, 22, 81, 650; with the kv heads of a row
//     tile as neighbours in the grid, the row tiles of most keys first, so that an SM gets a long one and a short one 51, 22, 71, 552.
//     32 rows and not 64: half a tile's rows are half its time.
//   * decoded tokens (requests that bring one): a block of 8 warps owns (request, kv head); eight lanes share a key, so a
//     warp reads whole 128-byte lines of four keys at a time, and the 32 groups of eight lanes keep running maxima and sums
//     of their own, which meet in shared memory at the end.  Bound by the latency of its loads: a step has only requests x
//     kv heads such blocks.
#include "common.cuh"

#define PT_ROWS 32
#define PT_KEYS 32                         // keys of a tile
#define PT_GROUPS 2                        // groups of threads with tiles of their own
#define PT_GROUP_THREADS 128
#define PT_THREADS (PT_GROUPS * PT_GROUP_THREADS)
#define PT_PAD 4  // floats between rows of K, V and Q beyond head_dim: neighbouring rows start 4 banks apart
#define PT_PS (PT_KEYS + 4)

// four neighbouring elements as 32-bit values, from an address that is a multiple of their size
__device__ __forceinline__ float4 pl_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 pl_load4(const __half* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void pl_store4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void pl_store4(__half* p, const float4& v) {
  uint2 raw;
  *reinterpret_cast<__half2*>(&raw.x) = __floats2half2_rn(v.x, v.y);
  *reinterpret_cast<__half2*>(&raw.y) = __floats2half2_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = raw;
}
__device__ __forceinline__ float pl_dot(const float4& a, const float4& b, float s) {
  s = fmaf(a.x, b.x, s);
  s = fmaf(a.y, b.y, s);
  s = fmaf(a.z, b.z, s);
  return fmaf(a.w, b.w, s);
}
__device__ __forceinline__ void pl_axpy(float p, const float4& v, float4& o) {
  o.x = fmaf(p, v.x, o.x);
  o.y = fmaf(p, v.y, o.y);
  o.z = fmaf(p, v.z, o.z);
  o.w = fmaf(p, v.w, o.w);
}

// pairs of neighbouring 32-bit values, multiplied and added two at a time
struct __align__(16) pl_four { unsigned long long lo, hi; };
__device__ __forceinline__ void pl_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pl_twice(float x) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
  return v;
}
__device__ __forceinline__ void pl_axpy2(unsigned long long p, const pl_four& v, float4& o) {
  unsigned long long lo, hi;
  asm("mov.b64 %0, {%1, %2};" : "=l"(lo) : "f"(o.x), "f"(o.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(hi) : "f"(o.z), "f"(o.w));
  pl_fma2(lo, p, v.lo);
  pl_fma2(hi, p, v.hi);
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(lo));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.z), "=f"(o.w) : "l"(hi));
}
// four neighbouring elements into shared memory, as 32-bit values: 32-bit ones arrive behind the thread's back (pl_wait), others at once.
// None of them read: zeros.
__device__ __forceinline__ void pl_bring(float* dst, const float* src, bool there) {
  const unsigned at = (unsigned)__cvta_generic_to_shared(dst), bytes = there ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pl_bring(float* dst, const __half* src, bool there) {
  *reinterpret_cast<float4*>(dst) = there ? pl_load4(src) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void pl_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void pl_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// whether one of them is infinite or NaN
__device__ __forceinline__ bool pl_odd(const float4& v) {
  return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, v.w * 0.f))) != 0.f;  // (a zero times either is NaN)
}

template <typename T, int D>
__global__ void __launch_bounds__(PT_THREADS, 2)
plain_attention_prompt_kernel(const T* q, long long q_row_stride, T* __restrict__ out,
                              const T* k_cache, const T* v_cache,
                              const int* block_table, int max_pages, const int* req_slots,
                              const int* cu_q, const int* kv_len, const int* token_req,
                              int requests, int num_q, int num_kv, int page_size, int window, float scale,
                              long long num_pages, int* status) {
  constexpr int ST = D + PT_PAD;
  constexpr int CV = D / 64;  // groups of four output columns a thread owns
  extern __shared__ __align__(16) float pl_smem[];
  const int tid = threadIdx.x, group = tid / PT_GROUP_THREADS, gt = tid % PT_GROUP_THREADS, tx = gt & 15, ty = gt >> 4;
  float* qs = pl_smem;                                                             // [PT_ROWS][ST]
  float* ks = qs + PT_ROWS * ST + group * (2 * PT_KEYS * ST + PT_ROWS * PT_PS);    // [PT_KEYS][ST], a group's own
  float* vs = ks + PT_KEYS * ST;                                                   // [PT_KEYS][ST]
  float* ps = vs + PT_KEYS * ST;                                                   // [PT_ROWS][PT_PS]
  __shared__ long long slot_all[PT_GROUPS][2][PT_KEYS];                            // of a tile and of the one behind it
  __shared__ float m_s[PT_ROWS], l_s[PT_ROWS];                                     // of the second group, at the end
  pdl_launch_dependents();
  pdl_wait();
  const int gq = num_q / num_kv, per = PT_ROWS / gq;  // query heads per kv head; tokens of a row tile
  // which request and which of its row tiles (requests of one token are the other kernel's, requests of none have no rows)
  int r = 0, tile = blockIdx.x / num_kv, t0 = 0, n = 0;
  for (; r < requests; ++r) {
    t0 = cu_q[r];
    n = cu_q[r + 1] - t0;
    if (n <= 1) continue;
    const int tiles = (n + per - 1) / per;
    if (tile < tiles) {
      tile = tiles - 1 - tile;  // (the tiles with the most keys first)
      break;
    }
    tile -= tiles;
  }
  if (r >= requests) return;
  const int kh = blockIdx.x % num_kv;
  const int row0 = tile * per, rows = min(per, n - row0) * gq;  // row i: token row0 + i / gq, query head i % gq
  const int kvl = kv_len[r];
  const int pos0 = kvl - n + row0;
  if (!__syncthreads_or(tid * gq < rows && token_req[t0 + row0 + tid] >= 0 && kvl > 0)) {
    for (int i = tid; i < rows * D; i += PT_THREADS) {
      const int row = i / D, e = i - row * D;
      out[(long long)(t0 + row0 + row / gq) * num_q * D + (long long)(kh * gq + row % gq) * D + e] = from_f32<T>(0.f);
    }
    return;
  }
  for (int i = tid; i < PT_ROWS * (D / 4); i += PT_THREADS) {
    const int row = i / (D / 4), e = (i - row * (D / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows)
      v = pl_load4(q + (long long)(t0 + row0 + row / gq) * q_row_stride + (long long)(kh * gq + row % gq) * D + e);
    *reinterpret_cast<float4*>(qs + row * ST + e) = v;
  }
  int pos[4], first[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pos[i] = pos0 + (ty * 4 + i) / gq;
    first[i] = first_seen(pos[i], window);
  }
  float m[4], l[4];
  float4 o[4][CV];
  const int* bt = block_table + (long long)req_slots[r] * max_pages;
  const long long kv_row = (long long)num_kv * D;
  const int last = pos0 + (rows - 1) / gq;
  auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(PT_GROUP_THREADS) : "memory"); };
  auto look_up = [&](int base, int buf) {  // where the keys of a tile lie; -1: none
    if (gt >= PT_KEYS) return;
    const int key = base + gt;
    long long slot = -1;
    if (key <= last) {
      const int page = bt[key / page_size];
      if (page < 0 || page >= num_pages) ullm_report(status, ULLM_STATUS_PAGE, t0 + row0, page);
      else slot = (long long)page * page_size + key % page_size;
    }
    slot_all[group][buf][gt] = slot;
  };
  auto bring = [&](float* dst, const T* cache, int buf) {
#pragma unroll 4
    for (int i = gt; i < PT_KEYS * (D / 4); i += PT_GROUP_THREADS) {
      const int key = i / (D / 4), e = (i - key * (D / 4)) * 4;
      const long long slot = slot_all[group][buf][key];
      pl_bring(dst + key * ST + e, cache + (slot >= 0 ? slot : 0) * kv_row + (long long)kh * D + e, slot >= 0);
    }
  };
  // A weight of zero must not meet a value that a row does not see and that is infinite or NaN: where an output is not finite, the
  // tile's rows run once more, and each adds up only what it sees.
  bool odd = false;
#pragma unroll 1
  for (;;) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
#pragma unroll
      for (int c = 0; c < CV; ++c) o[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();  // Q is in place; what the groups left to one another has been read
    int turn = 0;
    const int start = max(0, first_seen(pos0, window)) + group * PT_KEYS;
    look_up(start, 0);
    group_sync();
    bring(ks, k_cache, 0);
    pl_commit();
    bring(vs, v_cache, 0);
    pl_commit();
    look_up(start + PT_GROUPS * PT_KEYS, 1);
#pragma unroll 1
    for (int base = start; base <= last; base += PT_GROUPS * PT_KEYS, turn ^= 1) {
      const long long* slot_s = slot_all[group][turn];
      pl_wait<1>();
      group_sync();  // K is there, and the places of the keys behind
      // scores of rows 4 ty .. + 3 against keys tx, tx + 16
      float s[4][2];
      {
        unsigned long long w[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i][0] = w[i][1] = 0ull;
#pragma unroll 4
        for (int e = 0; e < D; e += 4) {
          pl_four a[4], b[2];
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const pl_four*>(qs + (ty * 4 + i) * ST + e);
#pragma unroll
          for (int j = 0; j < 2; ++j) b[j] = *reinterpret_cast<const pl_four*>(ks + (tx + 16 * j) * ST + e);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              pl_fma2(w[i][j], a[i].lo, b[j].lo);
              pl_fma2(w[i][j], a[i].hi, b[j].hi);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float x, y;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(w[i][j]));
            s[i][j] = x + y;
          }
      }
      bool there[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) there[j] = slot_s[tx + 16 * j] >= 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int key = base + tx + 16 * j;
          s[i][j] = (there[j] && key >= first[i] && key <= pos[i]) ? s[i][j] * scale : -INFINITY;
        }
        float top = fmaxf(s[i][0], s[i][1]);
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
        const float m2 = fmaxf(m[i], top);
        const float keep = m2 == -INFINITY ? 1.f : expf(m[i] - m2);  // (no key seen yet: nothing to rescale)
        l[i] *= keep;  // (the sum of this lane's own keys)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float p = s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - m2);
          ps[(ty * 4 + i) * PT_PS + tx + 16 * j] = p;
          l[i] += p;
        }
        m[i] = m2;
#pragma unroll
        for (int c = 0; c < CV; ++c) o[i][c].x *= keep, o[i][c].y *= keep, o[i][c].z *= keep, o[i][c].w *= keep;
      }
      pl_wait<0>();
      group_sync();  // V is there, K has been read  (a row's weights are written and read by the 16 lanes that own the row)
      bring(ks, k_cache, turn ^ 1);
      pl_commit();
      if (odd) {  // each row adds up the keys that it sees
#pragma unroll 1
        for (int key = 0; key < PT_KEYS; ++key) {
          if (slot_s[key] < 0) continue;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (base + key < first[i] || base + key > pos[i]) continue;
            const float p = ps[(ty * 4 + i) * PT_PS + key];
#pragma unroll
            for (int c = 0; c < CV; ++c) pl_axpy(p, *reinterpret_cast<const float4*>(vs + key * ST + c * 64 + tx * 4), o[i][c]);
          }
        }
      } else {
#pragma unroll 2
        for (int key = 0; key < PT_KEYS; key += 4) {
          float4 p[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(ps + (ty * 4 + i) * PT_PS + key);
#pragma unroll
          for (int c = 0; c < CV; ++c) {
            const float* vp = vs + key * ST + c * 64 + tx * 4;
            const pl_four v0 = *reinterpret_cast<const pl_four*>(vp), v1 = *reinterpret_cast<const pl_four*>(vp + ST),
                          v2 = *reinterpret_cast<const pl_four*>(vp + 2 * ST), v3 = *reinterpret_cast<const pl_four*>(vp + 3 * ST);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              pl_axpy2(pl_twice(p[i].x), v0, o[i][c]);
              pl_axpy2(pl_twice(p[i].y), v1, o[i][c]);
              pl_axpy2(pl_twice(p[i].z), v2, o[i][c]);
              pl_axpy2(pl_twice(p[i].w), v3, o[i][c]);
            }
          }
        }
      }
      group_sync();  // V has been read
      bring(vs, v_cache, turn ^ 1);
      pl_commit();
      look_up(base + 2 * PT_GROUPS * PT_KEYS, turn);
    }
    pl_wait<0>();  // (the tile behind the last one: zeros)
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
#pragma unroll
      for (int c = 0; c < CV; ++c) bad |= pl_odd(o[i][c]);
    }
    if (odd || !__syncthreads_or(bad)) break;
    odd = true;
  }
  // the groups meet: the second one's rows lie in its tile of keys
  if (group == 1) {
    group_sync();  // (its last tile has been read)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (tx == 0) m_s[ty * 4 + i] = m[i], l_s[ty * 4 + i] = l[i];
#pragma unroll
      for (int c = 0; c < CV; ++c) *reinterpret_cast<float4*>(ks + (ty * 4 + i) * ST + c * 64 + tx * 4) = o[i][c];
    }
  }
  __syncthreads();
  if (group == 1) return;
  const float* rest = ks + 2 * PT_KEYS * ST + PT_ROWS * PT_PS;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = ty * 4 + i;
    if (row >= rows) continue;
    // (a group that saw no key of the row has a maximum of -infinity, and adds nothing)
    const float m2 = fmaxf(m[i], m_s[row]);
    const float f0 = m[i] == -INFINITY ? 0.f : expf(m[i] - m2), f1 = m_s[row] == -INFINITY ? 0.f : expf(m_s[row] - m2);
    const float sum = l[i] * f0 + l_s[row] * f1;
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    const bool padding = token_req[t0 + row0 + row / gq] < 0;
    T* dst = out + (long long)(t0 + row0 + row / gq) * num_q * D + (long long)(kh * gq + row % gq) * D + tx * 4;
#pragma unroll
    for (int c = 0; c < CV; ++c) {
      const float4 b = *reinterpret_cast<const float4*>(rest + row * ST + c * 64 + tx * 4);
      const float4 v = make_float4((o[i][c].x * f0 + b.x * f1) * inv, (o[i][c].y * f0 + b.y * f1) * inv,
                                   (o[i][c].z * f0 + b.z * f1) * inv, (o[i][c].w * f0 + b.w * f1) * inv);
      pl_store4(dst + c * 64, padding ? make_float4(0.f, 0.f, 0.f, 0.f) : v);
    }
  }
}

#define PD_WARPS 8
#define PD_GROUPS (PD_WARPS * 4)

// GQ query heads of a kv head at a time (grid z counts them)
template <typename T, int D, int GQ>
__global__ void __launch_bounds__(PD_WARPS * 32)
plain_attention_decode_kernel(const T* q, long long q_row_stride, T* __restrict__ out,
                              const T* k_cache, const T* v_cache,
                              const int* block_table, int max_pages, const int* req_slots,
                              const int* cu_q, const int* kv_len, const int* token_req,
                              int tokens, int requests, int num_q, int num_kv, int page_size, int window, float scale,
                              long long num_pages, int* status) {
  constexpr int P = D / 32;           // pieces of four channels a lane holds: 4 (lane % 8) + 32 i
  constexpr int U = GQ * P > 8 ? 1 : 2;  // keys of a group in flight, as far as the registers reach
  __shared__ float m_s[GQ][PD_GROUPS], l_s[GQ][PD_GROUPS];
  __shared__ __align__(16) float o_s[PD_WARPS][D];
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x, kh = blockIdx.y, t = cu_q[r];
  for (int x = cu_q[requests] + r; x < tokens; x += requests)  // (rows behind the last request's are padding, and zeros)
    for (int e = threadIdx.x; e < GQ * D; e += PD_WARPS * 32)
      out[((long long)x * num_q + kh * (num_q / num_kv) + blockIdx.z * GQ) * D + e] = from_f32<T>(0.f);
  if (cu_q[r + 1] - t != 1) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane & 7, group = tid >> 3;
  const int h0 = kh * (num_q / num_kv) + blockIdx.z * GQ;
  T* dst = out + ((long long)t * num_q + h0) * D;
  const int kvl = kv_len[r];
  if (token_req[t] < 0 || kvl <= 0) {  // padding row
    for (int i = tid; i < GQ * D; i += PD_WARPS * 32) dst[i] = from_f32<T>(0.f);
    return;
  }
  const int pos = kvl - 1, lo = first_seen(pos, window);
  float4 qv[GQ][P], o[GQ][P];
  float m[GQ], l[GQ];
#pragma unroll
  for (int g = 0; g < GQ; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      qv[g][i] = pl_load4(q + (long long)t * q_row_stride + (long long)(h0 + g) * D + i * 32 + sub * 4);
      o[g][i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  const int* bt = block_table + (long long)req_slots[r] * max_pages;
  const long long kv_row = (long long)num_kv * D;
  // (all lanes of a warp make the same number of turns: the shuffles below need every one of them)
  for (int base = lo + warp * 4; base <= pos; base += U * PD_GROUPS) {
    long long at[U];
    float4 kv[U][P], vv[U][P];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int key = base + u * PD_GROUPS + (lane >> 3);
      at[u] = -1;
      if (key <= pos) {
        const int page = bt[key / page_size];
        if (page < 0 || page >= num_pages) {
          if (sub == 0) ullm_report(status, ULLM_STATUS_PAGE, t, page);
        } else {
          at[u] = ((long long)page * page_size + key % page_size) * kv_row + (long long)kh * D + sub * 4;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < P; ++i) {
        kv[u][i] = vv[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at[u] >= 0) {
          kv[u][i] = pl_load4(k_cache + at[u] + i * 32);
          vv[u][i] = pl_load4(v_cache + at[u] + i * 32);
        }
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float s[GQ];
#pragma unroll
      for (int g = 0; g < GQ; ++g) {
        s[g] = 0.f;
#pragma unroll
        for (int i = 0; i < P; ++i) s[g] = pl_dot(qv[g][i], kv[u][i], s[g]);
      }
#pragma unroll
      for (int x = 4; x > 0; x >>= 1)
#pragma unroll
        for (int g = 0; g < GQ; ++g) s[g] += __shfl_xor_sync(0xffffffffu, s[g], x);
#pragma unroll
      for (int g = 0; g < GQ; ++g) {
        const float sc = at[u] >= 0 ? s[g] * scale : -INFINITY, m2 = fmaxf(m[g], sc);
        const float keep = m2 == -INFINITY ? 1.f : expf(m[g] - m2), p = sc == -INFINITY ? 0.f : expf(sc - m2);
        l[g] = l[g] * keep + p;
        m[g] = m2;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          o[g][i].x *= keep, o[g][i].y *= keep, o[g][i].z *= keep, o[g][i].w *= keep;
          pl_axpy(p, vv[u][i], o[g][i]);
        }
      }
    }
  }
  if (sub == 0) {
#pragma unroll
    for (int g = 0; g < GQ; ++g) m_s[g][group] = m[g], l_s[g][group] = l[g];
  }
  __syncthreads();
#pragma unroll
  for (int g = 0; g < GQ; ++g) {
    float top = -INFINITY, sum = 0.f;
    for (int i = 0; i < PD_GROUPS; ++i) top = fmaxf(top, m_s[g][i]);
    for (int i = 0; i < PD_GROUPS; ++i) sum += m_s[g][i] == -INFINITY ? 0.f : l_s[g][i] * expf(m_s[g][i] - top);
    const float f = (m[g] == -INFINITY ? 0.f : expf(m[g] - top)) * (sum > 0.f ? 1.f / sum : 0.f);
#pragma unroll
    for (int i = 0; i < P; ++i) {
      float4 v = make_float4(o[g][i].x * f, o[g][i].y * f, o[g][i].z * f, o[g][i].w * f);
#pragma unroll
      for (int x = 8; x < 32; x <<= 1) {  // the four keys of the warp
        v.x += __shfl_xor_sync(0xffffffffu, v.x, x);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, x);
        v.z += __shfl_xor_sync(0xffffffffu, v.z, x);
        v.w += __shfl_xor_sync(0xffffffffu, v.w, x);
      }
      if (lane < 8) *reinterpret_cast<float4*>(&o_s[warp][i * 32 + sub * 4]) = v;
    }
    __syncthreads();
    for (int e = tid; e < D; e += PD_WARPS * 32) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < PD_WARPS; ++w) v += o_s[w][e];
      dst[g * D + e] = from_f32<T>(v);
    }
    __syncthreads();
  }
}

template <typename T, int D>
static int plain_launch(const void* q, long long q_row_stride, void* out, const void* k_cache, const void* v_cache,
                        const int* block_table, int max_pages, const int* req_slots, const int* cu_q, const int* kv_len,
                        const int* token_req, int tokens, int requests, int longest, int num_q, int num_kv, int page_size,
                        int window, float scale, long long num_pages, int* status, cudaStream_t st) {
  const int gq = num_q / num_kv;
  if (longest != 1 || tokens != requests) {  // (as many rows as requests alone says nothing: a request may bring none)
    constexpr int ST = D + PT_PAD;
    constexpr size_t smem = ((size_t)(PT_ROWS + PT_GROUPS * 2 * PT_KEYS) * ST + (size_t)PT_GROUPS * PT_ROWS * PT_PS) * sizeof(float);
    static bool allowed = false;
    if (!allowed) {
      if (cudaFuncSetAttribute(plain_attention_prompt_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess) {
        cudaGetLastError();
        return ULLM_ERR_LAUNCH;
      }
      allowed = true;
    }
    const int per = PT_ROWS / gq;
    const long long tiles = tokens / per + requests;
    if (tiles * num_kv > 0x7fffffffLL) return ULLM_ERR_BAD_SIZE;
    const int rc = ullm_launch_kernel(plain_attention_prompt_kernel<T, D>, dim3((int)(tiles * num_kv)), dim3(PT_THREADS), smem, st,
                                      (const T*)q, q_row_stride, (T*)out, (const T*)k_cache, (const T*)v_cache, block_table,
                                      max_pages, req_slots, cu_q, kv_len, token_req, requests, num_q, num_kv, page_size, window,
                                      scale, num_pages, status);
    if (rc != ULLM_OK || (requests == 1 && longest > 1 && longest == tokens)) return rc;
  }
#define PD_GO(GQ)                                                                                                        \
  return ullm_launch_kernel(plain_attention_decode_kernel<T, D, GQ>, dim3(requests, num_kv, gq / GQ), dim3(PD_WARPS * 32), \
                            0, st, (const T*)q, q_row_stride, (T*)out, (const T*)k_cache, (const T*)v_cache, block_table, \
                            max_pages, req_slots, cu_q, kv_len, token_req, tokens, requests, num_q, num_kv, page_size,     \
                            window, scale, num_pages, status)
  if (gq % 4 == 0) PD_GO(4);
  if (gq % 2 == 0) PD_GO(2);
  PD_GO(1);
#undef PD_GO
}

// Sizes and types these kernels take: head sizes 64 and 128, float32 or float16, at most 32 query heads per kv head; the
// caller keeps the general kernel for everything else.
extern "C" int ullm_attention_plain_supported(int dtype, int head_dim, int num_q, int num_kv) {
  return (dtype == ULLM_DTYPE_F32 || dtype == ULLM_DTYPE_F16) && (head_dim == 64 || head_dim == 128) && num_kv > 0 &&
         num_q % num_kv == 0 && num_q / num_kv >= 1 && num_q / num_kv <= PT_ROWS && num_kv <= 65535;
}

// Arguments as `ullm_paged_attention_generic`, the number of requests (cu_q holds one more entry) and how many tokens the longest
// of them brings (0: not known; a step of which all requests are known to bring one token saves a launch).  UNSUPPORTED where
// the rows do not allow 16-byte (float16: 8-byte) reads.
extern "C" int ullm_attention_plain(int dtype, const void* q, long long q_row_stride, void* out, const void* k_cache,
                                    const void* v_cache, const int* block_table, int max_pages, const int* req_slots,
                                    const int* cu_q, const int* kv_len, const int* token_req, int tokens, int requests,
                                    int longest, int num_q, int num_kv, int head_dim, int page_size, int window, float scale,
                                    long long num_pages, int* status, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (tokens < 0 || requests < 0 || longest < 0 || page_size <= 0 || max_pages <= 0) return ULLM_ERR_BAD_SIZE;
  if (!ullm_attention_plain_supported(dtype, head_dim, num_q, num_kv) || q_row_stride % 4) return ULLM_ERR_UNSUPPORTED;
  const uintptr_t align = dtype == ULLM_DTYPE_F32 ? 15 : 7;
  if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) & align) return ULLM_ERR_UNSUPPORTED;
  if (tokens == 0) return ULLM_OK;
  if (requests == 0)  // (all rows are padding)
    return cudaMemsetAsync(out, 0, (size_t)tokens * num_q * head_dim * (dtype == ULLM_DTYPE_F32 ? 4 : 2), st) == cudaSuccess ? ULLM_OK
                                                                                                                             : ULLM_ERR_LAUNCH;
#define PL_GO(T, D)                                                                                                       \
  return plain_launch<T, D>(q, q_row_stride, out, k_cache, v_cache, block_table, max_pages, req_slots, cu_q, kv_len,       \
                            token_req, tokens, requests, longest, num_q, num_kv, page_size, window, scale, num_pages, status, st)
  if (dtype == ULLM_DTYPE_F32) {
    if (head_dim == 64) PL_GO(float, 64);
    PL_GO(float, 128);
  }
  if (head_dim == 64) PL_GO(__half, 64);
  PL_GO(__half, 128);
#undef PL_GO
}
