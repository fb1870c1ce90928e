// The recurrence of csrc/mlstm.cu for prompt portions in bfloat16, MCH_Q tokens at a time on the tensor cores, all chunks side
// by side.
//
// With b_t the sum of the log forget gates of the chunk's tokens up to t, i_s the log input gates, (S, n, m) the state in front
// of the chunk and B = b of its last token, m' the maximum behind it:
//
//   m_t = b_t + max(m, max_{s <= t} (i_s - b_s))                   the running maximum
//   P_ts = exp(b_t - m_t + i_s - b_s) q_t . k_s   (s <= t)          the scores, weighted
//   o_t = (exp(b_t + m - m_t) S^T q_t + sum_s P_ts v_s) / (max(|exp(b_t + m - m_t) n . q_t + sum_s P_ts|, exp(-m_t)) + 1e-6)
//   S'  = exp(B + m - m') S + sum_s exp(B - b_s + i_s - m') k_s v_s^T          (n' alike)
//
// Four kernels: `gates` forms the sums, maxima and weights of every token (a walk over the chunks with one number each, the rest
// side by side), `fold` every chunk's own contribution to S and n, `scan` walks the chunks of a request element by element and
// leaves in front of every chunk the state it starts from, `out` forms the outputs.
//
// What bounds it: the state that is written and read once per chunk (32 chunks x 8 heads x 128 x 256 at 2,048 tokens: 34 MB a
// time, mostly L2) and the latency of a block's phases; the tensor pipe has 3 GFLOP to do.  The token-by-token kernel is a chain
// of 2,048 dependent steps: 766 us per layer at these sizes.
//
// Precision: 32-bit throughout.  q, k and v are exact bfloat16 operands; every 32-bit operand (weighted keys, weighted scores,
// the state) enters as THREE bfloat16 terms (value, rest, rest of the rest: 24 bits); the tensor core sums 16 products of each and
// ordinary 32-bit additions do the rest; the sums b are 64-bit, so that a difference of two of them keeps what products of the
// gates would.  Median error of an output row against 64 bits at 8 heads of 128 x 256, 2,048 tokens, gates that keep long: 3.5e-7
// (one chain of tensor-core sums: 6.1e-7; the token-by-token kernel: 6.6e-7); 256 x 512: 3.0e-7 (7.7e-7, 5.8e-7).
//
// mma.sync m16n8k16: a tcgen05 tile would want 128 rows where a chunk has 64, and the operands are formed in registers.
#include "common.cuh"

#define MCH_Q 64
#define MCH_THREADS 256
#define MCH_WARPS 8
#define MCH_PS 72  // elements between rows of the weighted scores in shared memory

__device__ __forceinline__ void mch_ldsm4(unsigned (&r)[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void mch_ldsm4t(unsigned (&r)[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void mch_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += a b as a sum of its own: the tensor core cuts its sums instead of rounding them, which over a row of channels would show.
// Three terms of one operand (a[i] or b0[i], b1[i]) meet in it, smallest first.
__device__ __forceinline__ void mch_add(float (&c)[4], const float (&t)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += t[e];
}
__device__ __forceinline__ void mch_mma_apart(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mch_mma(t, a, b0, b1);
  mch_add(c, t);
}
__device__ __forceinline__ void mch_mma_a3(float (&c)[4], const unsigned (&a)[3][4], unsigned b0, unsigned b1) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 2; i >= 0; --i) mch_mma(t, a[i], b0, b1);
  mch_add(c, t);
}
__device__ __forceinline__ void mch_mma_b3(float (&c)[4], const unsigned (&a)[4], const unsigned (&b0)[3], const unsigned (&b1)[3]) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 2; i >= 0; --i) mch_mma(t, a, b0[i], b1[i]);
  mch_add(c, t);
}
// (v0, v1) as three pairs of bfloat16: rounded values, rounded rests, rounded rests of those
__device__ __forceinline__ void mch_split(float v0, float v1, unsigned& hi, unsigned& mid, unsigned& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
  v0 -= __bfloat162float(h.x);
  v1 -= __bfloat162float(h.y);
  const __nv_bfloat162 m = __floats2bfloat162_rn(v0, v1);
  const __nv_bfloat162 l = __floats2bfloat162_rn(v0 - __bfloat162float(m.x), v1 - __bfloat162float(m.y));
  hi = *reinterpret_cast<const unsigned*>(&h);
  mid = *reinterpret_cast<const unsigned*>(&m);
  lo = *reinterpret_cast<const unsigned*>(&l);
}

// What the kernels share of a step.  Per token and head (arrays [heads][tokens]): row = b_t - m_t and col = i_s - b_s (64-bit),
// from_state = exp(b_t + m - m_t), to_state = exp(B - b_s + i_s - m'), floor = exp(-m_t); per chunk and head: keep =
// exp(B + m - m').  fold [(chunk * heads + head)][vdim + 1][dim]: S^T and behind it n.
struct MchScratch {
  double* row;
  double* col;
  float* from_state;
  float* to_state;
  float* floor;
  float* keep;
  float* fold;
};

// Chunk `tile` of the step: its first token and its tokens (0: there is no such chunk).  Chunks are counted over the requests
// that bring more than `least` tokens.
__device__ __forceinline__ int mch_find(int tile, const int* cu_q, int requests, int least, int& t0) {
  for (int i = 0; i < requests; ++i) {
    const int b = cu_q[i], n = cu_q[i + 1] - b;
    if (n <= least) continue;
    const int nt = (n + MCH_Q - 1) / MCH_Q;
    if (tile < nt) {
      t0 = b + tile * MCH_Q;
      return min(MCH_Q, n - tile * MCH_Q);
    }
    tile -= nt;
  }
  return 0;
}
__device__ __forceinline__ int mch_first_tile(int req, const int* cu_q, int least) {
  int tile = 0;
  for (int i = 0; i < req; ++i) {
    const int m = cu_q[i + 1] - cu_q[i];
    if (m > least) tile += (m + MCH_Q - 1) / MCH_Q;
  }
  return tile;
}

__device__ __forceinline__ float mch_log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// One block per (head, request); a warp takes a chunk at a time, a lane two neighbouring tokens.
__global__ void __launch_bounds__(MCH_THREADS)
mlstm_chunk_gates_kernel(const float* gates, const float* __restrict__ bias_i, const float* __restrict__ bias_f,
                         float cap, float* state, long long state_stride, long long m_off,
                         const int* cu_q, const int* req_slots, const int* token_req,
                         int tokens, int least, int heads, int num_slots, MchScratch sc, int* status) {
  extern __shared__ __align__(16) unsigned char mch_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.x, req = blockIdx.y;
  const int t0 = cu_q[req], n = cu_q[req + 1] - t0;
  if (n <= least || token_req[t0] < 0) return;
  const int slot = req_slots[req];
  if (slot < 0 || slot >= num_slots) {
    if (threadIdx.x == 0) ullm_report(status, ULLM_STATUS_SLOT, req, slot);
    return;
  }
  const int chunks = (n + MCH_Q - 1) / MCH_Q, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* sum_s = reinterpret_cast<double*>(mch_smem);  // [chunks]: B
  double* top_s = sum_s + chunks;                       // [chunks]: max (i_s - b_s)
  float* m_s = reinterpret_cast<float*>(top_s + chunks);  // [chunks + 1]: m in front of every chunk
  const float bi = bias_i != nullptr ? bias_i[head] : 0.f, bf = bias_f != nullptr ? bias_f[head] : 0.f;
  // sums and differences of the lane's two tokens (past the chunk's end: a gate that neither forgets nor takes)
  auto two = [&](int c, double (&b)[2], double (&d)[2]) {
    float gi[2], gf[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int t = c * MCH_Q + 2 * lane + j;
      gi[j] = -INFINITY;
      gf[j] = 0.f;
      if (t < n) {
        const float* g = gates + (long long)(t0 + t) * 2 * heads;
        gi[j] = cap * tanhf((g[head] + bi) / cap);
        gf[j] = mch_log_sigmoid(cap * tanhf((g[heads + head] + bf) / cap));
      }
    }
    double sum = (double)gf[0] + (double)gf[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const double in_front = __shfl_up_sync(0xffffffffu, sum, 1);
    b[0] = (lane > 0 ? in_front : 0.0) + (double)gf[0];  // (not from the sum behind: a gate that is NaN reaches no token in front of it)
    b[1] = sum;
    d[0] = (double)gi[0] - b[0];
    d[1] = (double)gi[1] - b[1];
  };
  for (int c = warp; c < chunks; c += MCH_WARPS) {
    double b[2], d[2];
    two(c, b, d);
    double top = fmax(d[0], d[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 31) sum_s[c] = b[1];
    if (lane == 0) top_s[c] = top;
  }
  __syncthreads();
  float* st_m = state + (long long)slot * state_stride + m_off + head;
  if (threadIdx.x == 0) {
    float m = *st_m;
    for (int c = 0; c < chunks; ++c) {
      m_s[c] = m;
      m = (float)(sum_s[c] + fmax((double)m, top_s[c]));
    }
    m_s[chunks] = m;
    *st_m = m;
  }
  __syncthreads();
  const int tile0 = mch_first_tile(req, cu_q, least);
  for (int c = warp; c < chunks; c += MCH_WARPS) {
    double b[2], d[2];
    two(c, b, d);
    const double m0 = (double)m_s[c], m1 = (double)m_s[c + 1], all = sum_s[c];
    double top = fmax(d[0], d[1]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, top, o);
      if (lane >= o) top = fmax(top, v);
    }
    double before = __shfl_up_sync(0xffffffffu, top, 1);
    if (lane == 0) before = -INFINITY;
    const double upto[2] = {fmax(before, d[0]), top};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int t = c * MCH_Q + 2 * lane + j;
      if (t >= n) continue;
      const long long at = (long long)head * tokens + t0 + t;
      const float m = (float)(b[j] + fmax(m0, upto[j]));
      sc.row[at] = b[j] - (double)m;
      sc.col[at] = d[j];
      sc.from_state[at] = expf((float)(b[j] + m0 - (double)m));
      sc.to_state[at] = expf((float)(all + d[j] - m1));
      sc.floor[at] = expf(-m);
    }
    if (lane == 0) sc.keep[(long long)(tile0 + c) * heads + head] = expf((float)(all + m0 - m1));
  }
}

// rows of `cols` bfloat16 of the chunk into shared memory, cols + 8 apart, rows past the chunk's end zero
__device__ __forceinline__ void mch_load(__nv_bfloat16* dst, const __nv_bfloat16* src, long long row_stride, int cols, int cn) {
  const int pieces = cols >> 3;
  for (int i = threadIdx.x; i < MCH_Q * pieces; i += MCH_THREADS) {
    const int row = i / pieces, ch = (i - row * pieces) << 3;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (row < cn) x = *reinterpret_cast<const uint4*>(src + (long long)row * row_stride + ch);
    *reinterpret_cast<uint4*>(dst + row * (cols + 8) + ch) = x;
  }
}

// fold[tile, head] = sum_s v_s (to_state_s k_s)^T, and behind it sum_s to_state_s k_s
__global__ void __launch_bounds__(MCH_THREADS)
mlstm_chunk_fold_kernel(const __nv_bfloat16* qkv, long long row_stride, int k_off, int v_off,
                        const int* cu_q, const int* token_req, int requests, int tokens, int least,
                        int heads, int dim, int vdim, MchScratch sc) {
  extern __shared__ __align__(16) unsigned char mch_smem[];
  __shared__ float to_s[MCH_Q];
  pdl_launch_dependents();
  pdl_wait();
  int t0 = 0;
  const int tile = blockIdx.x, head = blockIdx.y;
  const int cn = mch_find(tile, cu_q, requests, least, t0);
  if (cn == 0 || token_req[t0] < 0) return;
  const int kb = dim + 8, vb = vdim + 8;
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(mch_smem);  // [MCH_Q][kb]
  __nv_bfloat16* v_s = k_s + MCH_Q * kb;                            // [MCH_Q][vb]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MCH_Q) to_s[tid] = tid < cn ? sc.to_state[(long long)head * tokens + t0 + tid] : 0.f;
  mch_load(k_s, qkv + (long long)t0 * row_stride + k_off + head * dim, row_stride, dim, cn);
  mch_load(v_s, qkv + (long long)t0 * row_stride + v_off + head * vdim, row_stride, vdim, cn);
  __syncthreads();
  float* out = sc.fold + ((long long)tile * heads + head) * (vdim + 1) * dim;
  for (int ch = tid; ch < dim; ch += MCH_THREADS) {
    float s = 0.f;
    for (int r = 0; r < MCH_Q; ++r) s = fmaf(to_s[r], __bfloat162float(k_s[r * kb + ch]), s);
    out[(long long)vdim * dim + ch] = s;
  }
  const int mat = lane >> 3;
  for (int n0 = warp * 8; n0 < dim; n0 += MCH_WARPS * 8) {  // eight key channels of the state
    const int ch = n0 + (lane >> 2);
    unsigned b[4][2][3];
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = s * 16 + h * 8 + (lane & 3) * 2;
        mch_split(to_s[r] * __bfloat162float(k_s[r * kb + ch]), to_s[r + 1] * __bfloat162float(k_s[(r + 1) * kb + ch]),
                  b[s][h][0], b[s][h][1], b[s][h][2]);
      }
    for (int m0 = 0; m0 < vdim; m0 += 16) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        unsigned a[4];
        mch_ldsm4t(a, v_s + (s * 16 + (mat >> 1) * 8 + (lane & 7)) * vb + m0 + (mat & 1) * 8);
        mch_mma_b3(acc, a, b[s][0], b[s][1]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(out + (long long)(m0 + (lane >> 2) + 8 * h) * dim + n0 + (lane & 3) * 2) =
            make_float2(acc[2 * h], acc[2 * h + 1]);
    }
  }
}

// fold <- the state in front of every chunk; state <- the state behind the last.  Two neighbouring key channels per thread.
__global__ void mlstm_chunk_scan_kernel(float* state, long long state_stride, const int* cu_q,
                                        const int* req_slots, const int* token_req, int least,
                                        int heads, int dim, int vdim, int num_slots, MchScratch sc) {
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, head = blockIdx.y;
  const int t0 = cu_q[req], n = cu_q[req + 1] - t0;
  if (n <= least || token_req[t0] < 0) return;
  const int slot = req_slots[req];
  if (slot < 0 || slot >= num_slots) return;  // (reported by the gates' kernel)
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) * 2, size = dim * vdim;
  if (e >= size + dim) return;
  const int tile0 = mch_first_tile(req, cu_q, least), chunks = (n + MCH_Q - 1) / MCH_Q;
  const long long step = (long long)heads * (size + dim);
  float* f = sc.fold + ((long long)tile0 * heads + head) * (size + dim) + e;
  const float* keep = sc.keep + (long long)tile0 * heads + head;
  float2* st = reinterpret_cast<float2*>(state + (long long)slot * state_stride +
                                         (e < size ? (long long)head * size + e
                                                   : (long long)heads * size + (long long)head * dim + e - size));
  float2 s = *st;
  constexpr int U = 8;
  for (int c0 = 0; c0 < chunks; c0 += U) {
    float2 d[U];
    float a[U];
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (c0 + j < chunks) {
        d[j] = *reinterpret_cast<const float2*>(f + (c0 + j) * step);
        a[j] = keep[(long long)(c0 + j) * heads];
      }
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (c0 + j < chunks) {
        *reinterpret_cast<float2*>(f + (c0 + j) * step) = s;
        s.x = fmaf(a[j], s.x, d[j].x);
        s.y = fmaf(a[j], s.y, d[j].y);
      }
  }
  *st = s;
}

// A block: (chunk, head).  Scores: warp w has rows 16 (w & 3) .. + 15 against the keys of its half (w >> 2).  Outputs: a warp has
// 16 value columns at a time, transposed (rows value columns, columns tokens), so that each part of the state is split into its
// terms by one warp only.
__global__ void __launch_bounds__(MCH_THREADS, 2)
mlstm_chunk_out_kernel(const __nv_bfloat16* qkv, long long row_stride, int q_off, int k_off, int v_off,
                       float q_scale, const int* cu_q, const int* token_req, int requests, int tokens,
                       int least, int heads, int dim, int vdim, MchScratch sc, float* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char mch_smem[];
  __shared__ double row_s[MCH_Q], col_s[MCH_Q];
  __shared__ float from_s[MCH_Q], floor_s[MCH_Q], den_s[MCH_Q], sum_s[2][MCH_Q], nq_s[MCH_Q];
  pdl_launch_dependents();
  pdl_wait();
  int t0 = 0;
  const int tile = blockIdx.x, head = blockIdx.y;
  const int cn = mch_find(tile, cu_q, requests, least, t0);
  if (cn == 0 || token_req[t0] < 0) return;
  const int kb = dim + 8, vb = vdim + 8;
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(mch_smem);  // [MCH_Q][kb]
  __nv_bfloat16* k_s = q_s + MCH_Q * kb;                            // [MCH_Q][kb]
  __nv_bfloat16* v_s = k_s + MCH_Q * kb;                            // [MCH_Q][vb]
  __nv_bfloat16* p_s = v_s + MCH_Q * vb;                            // [3][MCH_Q][MCH_PS]: the weighted scores' terms
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mat = lane >> 3, g = lane >> 2, cp = (lane & 3) * 2;
  if (tid < MCH_Q) {
    const long long at = (long long)head * tokens + t0 + (tid < cn ? tid : 0);
    row_s[tid] = sc.row[at];
    col_s[tid] = sc.col[at];
    from_s[tid] = sc.from_state[at] * q_scale;
    floor_s[tid] = sc.floor[at];
  }
  const __nv_bfloat16* src = qkv + (long long)t0 * row_stride;
  mch_load(q_s, src + q_off + head * dim, row_stride, dim, cn);
  mch_load(k_s, src + k_off + head * dim, row_stride, dim, cn);
  mch_load(v_s, src + v_off + head * vdim, row_stride, vdim, cn);
  const float* st = sc.fold + ((long long)tile * heads + head) * (vdim + 1) * dim;
  __syncthreads();
  {
    const int r0 = (warp & 3) * 16, j0 = (warp >> 2) * 4;  // rows, and the first of four tiles of eight keys
    float sum[2] = {0.f, 0.f};
    if (j0 * 8 < r0 + 16) {
      float acc[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
      for (int kk = 0; kk < dim; kk += 16) {
        unsigned a[4];
        mch_ldsm4(a, q_s + (r0 + (mat & 1) * 8 + (lane & 7)) * kb + kk + (mat >> 1) * 8);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          unsigned b[4];
          mch_ldsm4(b, k_s + ((j0 + j) * 8 + (mat >> 1) * 8 + (lane & 7)) * kb + kk + (mat & 1) * 8);
          mch_mma_apart(acc[j], a, b[0], b[1]);
          mch_mma_apart(acc[j + 1], a, b[2], b[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = r0 + g + 8 * h, s = (j0 + j) * 8 + cp;
          float w[2];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            w[x] = (s + x <= t && t < cn) ? acc[j][2 * h + x] * q_scale * expf((float)(row_s[t] + col_s[s + x])) : 0.f;
            sum[h] += w[x];
          }
          unsigned p[3];
          mch_split(w[0], w[1], p[0], p[1], p[2]);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned*>(p_s + ((i * MCH_Q) + t) * MCH_PS + s) = p[i];
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
      if ((lane & 3) == 0) sum_s[warp >> 2][r0 + g + 8 * h] = sum[h];
    }
    // n . q of eight rows per warp
    const float* n0 = st + (long long)vdim * dim;
    float dot[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) dot[i] = 0.f;
    for (int e = lane; e < dim; e += 32) {
      const float nv = n0[e];
#pragma unroll
      for (int i = 0; i < 8; ++i) dot[i] = fmaf(nv, __bfloat162float(q_s[(warp * 8 + i) * kb + e]), dot[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      dot[i] = warp_sum(dot[i]);
      if (lane == 0) nq_s[warp * 8 + i] = dot[i];
    }
  }
  __syncthreads();
  if (tid < MCH_Q) den_s[tid] = fmaxf(fabsf(sum_s[0][tid] + sum_s[1][tid] + from_s[tid] * nq_s[tid]), floor_s[tid]) + 1e-6f;
  __syncthreads();
  for (int m0 = warp * 16; m0 < vdim; m0 += MCH_WARPS * 16) {
    float acc[8][4];
    // A weight of zero must not meet an infinite or NaN value of a later token: where one shows, the columns again, the tokens'
    // values without the tensor core, each by those that see it.
    bool odd = false;
#pragma unroll 1
    for (;;) {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
      const float* sp = st + (long long)(m0 + g) * dim + cp;
      const long long down = (long long)8 * dim;
      float2 x[4], y[4];
      x[0] = *reinterpret_cast<const float2*>(sp);
      x[1] = *reinterpret_cast<const float2*>(sp + down);
      x[2] = *reinterpret_cast<const float2*>(sp + 8);
      x[3] = *reinterpret_cast<const float2*>(sp + down + 8);
      for (int kk = 0; kk < dim; kk += 16) {
        const int nx = kk + 16 < dim ? kk + 16 : kk;
        y[0] = *reinterpret_cast<const float2*>(sp + nx);
        y[1] = *reinterpret_cast<const float2*>(sp + down + nx);
        y[2] = *reinterpret_cast<const float2*>(sp + nx + 8);
        y[3] = *reinterpret_cast<const float2*>(sp + down + nx + 8);
        unsigned a[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mch_split(x[i].x, x[i].y, a[0][i], a[1][i], a[2][i]);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          unsigned b[4];
          mch_ldsm4(b, q_s + (j * 8 + (mat >> 1) * 8 + (lane & 7)) * kb + kk + (mat & 1) * 8);
          mch_mma_a3(acc[j], a, b[0], b[1]);
          mch_mma_a3(acc[j + 1], a, b[2], b[3]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = y[i];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float f0 = from_s[j * 8 + cp], f1 = from_s[j * 8 + cp + 1];
        acc[j][0] *= f0, acc[j][1] *= f1, acc[j][2] *= f0, acc[j][3] *= f1;
      }
      if (odd) {
#pragma unroll 1
        for (int s = 0; s < cn; ++s) {
          const __nv_bfloat16* vp = v_s + s * vb + m0 + g;
          const float lo = __bfloat162float(vp[0]), hi = __bfloat162float(vp[8]);
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int x2 = 0; x2 < 2; ++x2) {
              const int t = j * 8 + cp + x2;
              if (s > t) continue;
              const __nv_bfloat16* p = p_s + t * MCH_PS + s;
              const float w = (__bfloat162float(p[2 * MCH_Q * MCH_PS]) + __bfloat162float(p[MCH_Q * MCH_PS])) + __bfloat162float(p[0]);
              acc[j][x2] = fmaf(w, lo, acc[j][x2]);
              acc[j][2 + x2] = fmaf(w, hi, acc[j][2 + x2]);
            }
        }
        break;
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        unsigned a[4];
        mch_ldsm4t(a, v_s + (s * 16 + (mat >> 1) * 8 + (lane & 7)) * vb + m0 + (mat & 1) * 8);
#pragma unroll
        for (int j = 2 * s; j < 8; j += 2) {  // (earlier tokens do not see these keys)
          unsigned b[4][3];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            unsigned r[4];
            mch_ldsm4(r, p_s + (i * MCH_Q + j * 8 + (mat >> 1) * 8 + (lane & 7)) * MCH_PS + s * 16 + (mat & 1) * 8);
            b[0][i] = r[0], b[1][i] = r[1], b[2][i] = r[2], b[3][i] = r[3];
          }
          mch_mma_b3(acc[j], a, b[0], b[1]);
          mch_mma_b3(acc[j + 1], a, b[2], b[3]);
        }
      }
      if (!__any_sync(0xffffffffu, any_odd(acc))) break;
      odd = true;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int x2 = 0; x2 < 2; ++x2) {
        const int t = j * 8 + cp + x2;
        if (t >= cn) continue;
        float* dst = out + ((long long)(t0 + t) * heads + head) * vdim + m0 + g;
        dst[0] = acc[j][x2] / den_s[t];
        dst[8] = acc[j][2 + x2] / den_s[t];
      }
  }
}

static size_t mch_fold_smem(int dim, int vdim) { return (size_t)MCH_Q * (dim + 8 + vdim + 8) * 2; }
static size_t mch_out_smem(int dim, int vdim) { return (size_t)MCH_Q * (2 * (dim + 8) + vdim + 8 + 3 * MCH_PS) * 2; }

// Sizes the chunked form takes (bfloat16): key and value sizes that are multiples of 16, as far as the shared memory reaches.
extern "C" int ullm_mlstm_chunk_supported(int heads, int dim, int vdim) {
  return heads > 0 && heads <= 65535 && dim > 0 && vdim > 0 && dim % 16 == 0 && vdim % 16 == 0 &&
         mch_out_smem(dim, vdim) <= 220 * 1024;
}
// Chunks a step has at most: every request that brings more than `least` tokens leaves one of them unfilled.
static int mch_tiles(int tokens, int requests, int least) {
  const int chunked = tokens / (least + 1);
  return tokens / MCH_Q + (requests < chunked ? requests : chunked);
}
// Floats of scratch for a step of `tokens` tokens and `requests` requests.
extern "C" long long ullm_mlstm_chunk_floats(int tokens, int requests, int heads, int dim, int vdim, int least) {
  const long long per_token = (long long)heads * tokens * (2 + 2 + 3);
  return per_token + (long long)mch_tiles(tokens, requests, least) * heads * ((long long)dim * (vdim + 1) + 1) + 16;
}

// Arguments as `ullm_mlstm_recurrence`; `scratch`: ullm_mlstm_chunk_floats floats on a 16-byte border.  Runs the requests that
// bring MORE than `least` tokens and leaves the others alone.
extern "C" int ullm_mlstm_chunk(const void* qkv, long long row_stride, int q_off, int k_off, int v_off, const float* gates,
                                const float* bias_i, const float* bias_f, float* scratch, float* state, long long state_stride,
                                const int* cu_q, const int* req_slots, const int* token_req, float* out, int tokens,
                                int requests, int heads, int dim, int vdim, float q_scale, float cap, int num_slots, int least,
                                int* status, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (tokens < 0 || requests < 0 || num_slots <= 0 || scratch == nullptr || least < 0) return ULLM_ERR_BAD_SIZE;
  if (!ullm_mlstm_chunk_supported(heads, dim, vdim) || requests > 65535 || tokens > MCH_Q * 4096) return ULLM_ERR_UNSUPPORTED;
  if (state_stride < (long long)heads * dim * (vdim + 1) + heads) return ULLM_ERR_BAD_SIZE;
  if (row_stride % 8 || q_off % 8 || k_off % 8 || v_off % 8 || state_stride % 2 || (((uintptr_t)qkv | (uintptr_t)scratch) & 15) ||
      ((uintptr_t)state & 7))
    return ULLM_ERR_UNSUPPORTED;
  if (tokens == 0 || requests == 0) return ULLM_OK;
  const int tiles = mch_tiles(tokens, requests, least);
  if (tiles == 0) return ULLM_OK;
  const long long ht = (long long)heads * tokens;
  MchScratch sc;
  sc.fold = scratch;  // (dim is a multiple of 16: what follows starts on a 16-byte border)
  sc.row = reinterpret_cast<double*>(scratch + (long long)tiles * heads * dim * (vdim + 1));
  sc.col = sc.row + ht;
  sc.from_state = reinterpret_cast<float*>(sc.col + ht);
  sc.to_state = sc.from_state + ht;
  sc.floor = sc.to_state + ht;
  sc.keep = sc.floor + ht;
  const size_t gs = (size_t)(tokens / MCH_Q + 2) * 20, fs = mch_fold_smem(dim, vdim), os = mch_out_smem(dim, vdim);
  static size_t have[3] = {48 * 1024, 48 * 1024, 48 * 1024};
  if (gs > have[0]) {
    if (cudaFuncSetAttribute(mlstm_chunk_gates_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gs) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have[0] = gs;
  }
  if (fs > have[1]) {
    if (cudaFuncSetAttribute(mlstm_chunk_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fs) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have[1] = fs;
  }
  if (os > have[2]) {
    if (cudaFuncSetAttribute(mlstm_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)os) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have[2] = os;
  }
  const __nv_bfloat16* x = (const __nv_bfloat16*)qkv;
  int rc = ullm_launch_kernel(mlstm_chunk_gates_kernel, dim3(heads, requests), dim3(MCH_THREADS), gs, st, gates, bias_i, bias_f,
                              cap, state, state_stride, (long long)heads * dim * (vdim + 1), cu_q, req_slots, token_req, tokens,
                              least, heads, num_slots, sc, status);
  if (rc != ULLM_OK) return rc;
  rc = ullm_launch_kernel(mlstm_chunk_fold_kernel, dim3(tiles, heads), dim3(MCH_THREADS), fs, st, x, row_stride, k_off, v_off,
                          cu_q, token_req, requests, tokens, least, heads, dim, vdim, sc);
  if (rc != ULLM_OK) return rc;
  rc = ullm_launch_kernel(mlstm_chunk_scan_kernel, dim3((dim * (vdim + 1) / 2 + 127) / 128, heads, requests), dim3(128), 0, st,
                          state, state_stride, cu_q, req_slots, token_req, least, heads, dim, vdim, num_slots, sc);
  if (rc != ULLM_OK) return rc;
  return ullm_launch_kernel(mlstm_chunk_out_kernel, dim3(tiles, heads), dim3(MCH_THREADS), os, st, x, row_stride, q_off, k_off,
                            v_off, q_scale, cu_q, token_req, requests, tokens, least, heads, dim, vdim, sc, out);
}
