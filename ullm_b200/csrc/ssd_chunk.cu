// The recurrence of csrc/ssd.cu for prompt portions in bfloat16, SSC_Q tokens at a time on the tensor cores.
//
// With a_t the logarithm of the decay, c_t = a_1 + .. + a_t inside a chunk, and S the state in front of the chunk:
//
//   y_t = e^(c_t) C_t^T S + sum_{s <= t} e^(c_t - c_s) dt_s (C_t . B_s) x_s + D x_t
//   S'  = e^(c_Q) S + sum_s B_s (e^(c_Q - c_s) dt_s x_s)^T
//
// Three kernels.  `scores` forms what depends on one chunk alone: C_t . B_s, the same for all heads of a group, and every
// head's sums and weights.  `walk` takes a request's chunks in order: a block owns (request, head, 16 columns of S), keeps its
// part of S in 32-bit accumulators, leaves it in front of every chunk in scratch, and does nothing else on the way, so that
// what follows one another is a load that was asked for three chunks ahead, 16 tensor instructions and one multiply-add.
// `out` forms the outputs of all chunks side by side.
//
// What bounds it: the walk's chain (32 chunks at 2,048 tokens) and the states on their way through the scratch (a chunk's
// heads x columns x rows x 4 bytes: 34 MB each way at 32 heads, 64 columns, 128 rows); the tensor pipe has 2 GFLOP to do.
// Measured there, per layer: walk 27 us, out 25 us; one kernel that formed the outputs as it walked took 83 us (its blocks of
// eight warps, one per SM, spent 2.6 us on a chunk).
//
// Precision: everything is accumulated in 32-bit.  B, C and x are exact bfloat16 operands; the 32-bit operands (the
// weighted scores, the weighted x, the state in the read-out) enter as TWO bfloat16 terms, the rounded value and the rounded
// rest, so that a product keeps 16 bits of them or more, and no chunk ever sees a state rounded to 16 bits.
//
// mma.sync m16n8k16; accumulator and operand fragments as in csrc/attention_window.cu.
#include "ssd_chunk_core.cuh"

#define SSC_PT 16        // columns of S of a block of the walk, and of a warp of the read-out
#define SSC_OUT_WARPS 8

// What the kernels share of a step, chunks counted over the requests that bring more than `least` tokens.
struct SscScratch {
  float* front;   // [chunk][head][pdim][n_state]: S^T in front of the chunk
  float2* steps;  // [head][tokens]: c_t and dt_t
  float* weight;  // [head][tokens]: e^(c_Q - c_t) dt_t
  float* total;   // [chunk][head]: e^(c_Q)
};

// Chunk `tile` of the step: its request, first token and tokens (0: there is no such chunk).
__device__ __forceinline__ int ssc_find(int tile, const int* cu_q, int requests, int least, int& req, int& t0) {
  for (int i = 0; i < requests; ++i) {
    const int b = cu_q[i], n = cu_q[i + 1] - b;
    if (n <= least) continue;
    const int nt = (n + SSC_Q - 1) / SSC_Q;
    if (tile < nt) {
      req = i;
      t0 = b + tile * SSC_Q;
      return min(SSC_Q, n - tile * SSC_Q);
    }
    tile -= nt;
  }
  return 0;
}

// scores[(group * tokens + t) * SSC_Q + s] = C_t . B_s for the tokens s <= t of t's chunk (others: undefined).  The blocks
// behind the groups' (blockIdx.y == groups) form the heads' running sums and weights, a warp per head at a time.
__global__ void __launch_bounds__(SSC_THREADS)
ssd_scores_kernel(const __nv_bfloat16* xbc, long long row_stride, int b_off, int c_off, int n_state, int groups,
                  const float* dt, const float* log_decay, long long dt_stride, int heads,
                  const int* cu_q, const int* token_req, int requests, int tokens, int least,
                  float* __restrict__ scores, SscScratch sc) {
  extern __shared__ __align__(16) unsigned char sc_smem[];
  pdl_launch_dependents();
  pdl_wait();
  int t0 = 0, req = 0;
  const int cn = ssc_find(blockIdx.x, cu_q, requests, least, req, t0);
  if (cn == 0 || token_req[t0] < 0) return;
  if (blockIdx.y >= groups) {
    const int lane = threadIdx.x & 31;
    for (int head = threadIdx.x >> 5; head < heads; head += SSC_THREADS / 32) {
      float a[2], d[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = 2 * lane + i;
        const long long at = (long long)(t0 + t) * dt_stride + head;
        a[i] = t < cn ? log_decay[at] : 0.f;
        d[i] = t < cn ? dt[at] : 0.f;
      }
      float run = a[0] + a[1];  // the inclusive sum over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      const float total = __shfl_sync(0xffffffffu, run, 31);
      const float cu[2] = {run - a[1], run};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const long long at = (long long)head * tokens + t0 + 2 * lane + i;
        if (2 * lane + i < cn) {
          sc.steps[at] = make_float2(cu[i], d[i]);
          sc.weight[at] = expf(total - cu[i]) * d[i];
        }
      }
      if (lane == 0) sc.total[(long long)blockIdx.x * heads + head] = expf(total);
    }
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = blockIdx.y;
  const int rs = n_state * 2 + 16;  // bytes between rows
  unsigned char* c_s = sc_smem;
  unsigned char* b_s = sc_smem + SSC_Q * rs;
  const int pieces = n_state / 8;
  for (int i = tid; i < SSC_Q * pieces; i += SSC_THREADS) {
    const int row = i / pieces, ch = i - row * pieces;
    const bool ok = row < cn;
    const __nv_bfloat16* src = xbc + (long long)(t0 + (ok ? row : 0)) * row_stride + group * n_state + ch * 8;
    ssc_cp_async_16(c_s + row * rs + ch * 16, src + c_off, ok);
    ssc_cp_async_16(b_s + row * rs + ch * 16, src + b_off, ok);
  }
  ssc_commit();
  ssc_wait<0>();
  __syncthreads();
  if (warp * 16 >= cn) return;
  float acc[SSC_Q / 8][4];
#pragma unroll
  for (int j = 0; j < SSC_Q / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  const int mat = lane >> 3;
  const unsigned char* ap = c_s + (warp * 16 + (mat & 1) * 8 + (lane & 7)) * rs + (mat >> 1) * 16;
  const unsigned char* bp = b_s + ((mat >> 1) * 8 + (lane & 7)) * rs + (mat & 1) * 16;
  for (int k = 0; k < n_state / 16; ++k) {
    unsigned a[4];
    ssc_ldsm4(a, ap + k * 32);
#pragma unroll
    for (int j = 0; j < SSC_Q / 8; j += 2) {
      if (j / 2 > warp) continue;  // (above the diagonal)
      unsigned b[4];
      ssc_ldsm4(b, bp + j * 8 * rs + k * 32);
      ssc_mma(acc[j], a, b[0], b[1]);
      ssc_mma(acc[j + 1], a, b[2], b[3]);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = warp * 16 + (lane >> 2) + h * 8;
    if (row >= cn) continue;
    float* dst = scores + ((long long)group * tokens + t0 + row) * SSC_Q + (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < SSC_Q / 8; ++j)
      if (j / 2 <= warp) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
  }
}

// n_state = 32 * NT, four warps (warp w the columns w N / 4 .. of S^T [16][N]); DEPTH: buffers of a chunk's rows, which arrive by
// cp.async.  What a chunk adds is summed apart from S: its tensor instructions do not wait for the chunk before it.
template <int NT, int DEPTH>
__global__ void __launch_bounds__(SSC_THREADS)
ssd_walk_kernel(const __nv_bfloat16* xbc, long long row_stride, int b_off, float* state,
                long long state_stride, const int* cu_q, const int* req_slots,
                const int* token_req, int heads, int pdim, int per_group, int tokens, int num_slots, int least,
                SscScratch sc, int* status) {
  constexpr int N = 32 * NT, NW = N / 4;  // NW: a warp's columns of S^T
  constexpr int RS = N * 2 + 16, XS = SSC_PT * 2 + 16;  // bytes between rows of B and of x
  constexpr int BB = SSC_Q * RS, XB = SSC_Q * XS, STAGE = BB + XB + (SSC_Q + 4) * 4;
  extern __shared__ __align__(16) unsigned char sc_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int req = blockIdx.z, head = blockIdx.y, p0 = blockIdx.x * SSC_PT;
  const int t0 = cu_q[req], n = cu_q[req + 1] - t0;
  if (n <= least || token_req[t0] < 0) return;
  const int slot = req_slots[req];
  if (slot < 0 || slot >= num_slots) {
    if (threadIdx.x == 0) ullm_report(status, ULLM_STATUS_SLOT, req, slot);
    return;
  }
  int tile0 = 0;
  for (int i = 0; i < req; ++i) {
    const int m = cu_q[i + 1] - cu_q[i];
    if (m > least) tile0 += (m + SSC_Q - 1) / SSC_Q;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mat = lane >> 3;
  const int chunks = (n + SSC_Q - 1) / SSC_Q;
  const __nv_bfloat16* b_src = xbc + (long long)t0 * row_stride + b_off + (head / per_group) * N;
  const __nv_bfloat16* x_src = xbc + (long long)t0 * row_stride + head * pdim + p0;
  auto issue = [&](int c) {  // one group of copies, an empty one past the last chunk
    if (c < chunks) {
      unsigned char* st = sc_smem + (c % DEPTH) * STAGE;
      const int cn = min(SSC_Q, n - c * SSC_Q);
      constexpr int PIECES = N / 8;
      for (int i = tid; i < SSC_Q * PIECES; i += SSC_THREADS) {
        const int row = i / PIECES, ch = i - row * PIECES;
        const bool ok = row < cn;
        ssc_cp_async_16(st + row * RS + ch * 16, b_src + (long long)(c * SSC_Q + (ok ? row : 0)) * row_stride + ch * 8, ok);
      }
      {
        static_assert(SSC_Q * SSC_PT / 8 == SSC_THREADS, "a piece of x per thread");
        const int row = tid >> 1, ch = tid & 1;
        const bool ok = row < cn;
        ssc_cp_async_16(st + BB + row * XS + ch * 16, x_src + (long long)(c * SSC_Q + (ok ? row : 0)) * row_stride + ch * 8, ok);
      }
      if (tid < SSC_Q)
        ssc_cp_async_4(st + BB + XB + tid * 4, sc.weight + (long long)head * tokens + t0 + c * SSC_Q + (tid < cn ? tid : 0), tid < cn);
      else if (tid == SSC_Q)
        ssc_cp_async_4(st + BB + XB + SSC_Q * 4, sc.total + (long long)(tile0 + c) * heads + head, true);
    }
    ssc_commit();
  };
#pragma unroll
  for (int c = 0; c < DEPTH - 1; ++c) issue(c);
  // S^T fragments: rows p = lane / 4 (+ 8), columns n = warp * NW + 8 j + 2 (lane % 4) (+ 1)
  const long long mine = (long long)(lane >> 2) * N + warp * NW + (lane & 3) * 2;
  float* st_head = state + (long long)slot * state_stride + ((long long)head * pdim + p0) * N + mine;
  float* front = sc.front + (((long long)tile0 * heads + head) * pdim + p0) * N + mine;
  const long long front_step = (long long)heads * pdim * N;
  float S[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 v = *reinterpret_cast<const float2*>(st_head + 8 * h * N + 8 * j);
      S[j][2 * h] = v.x;
      S[j][2 * h + 1] = v.y;
    }
  for (int c = 0; c < chunks; ++c) {
    ssc_wait<DEPTH - 2>();
    __syncthreads();  // chunk c is there, and everyone is done with the buffer that is filled next
    issue(c + DEPTH - 1);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(front + c * front_step + 8 * h * N + 8 * j) = make_float2(S[j][2 * h], S[j][2 * h + 1]);
    const unsigned char* st = sc_smem + (c % DEPTH) * STAGE;
    const float* w_s = reinterpret_cast<const float*>(st + BB + XB);
    float d[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) d[j][0] = d[j][1] = d[j][2] = d[j][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < SSC_Q / 16; ++ks) {
      // x^T, weighted, as two terms: columns (tokens) ks 16 + 8 (q >> 1) + 2 (lane % 4) (+ 1)
      unsigned x[4], ah[4], al[4];
      ssc_ldsm4t(x, st + BB + (ks * 16 + (mat >> 1) * 8 + (lane & 7)) * XS + (mat & 1) * 16);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 w = *reinterpret_cast<const float2*>(w_s + ks * 16 + (q >> 1) * 8 + (lane & 3) * 2);
        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&x[q]);
        ssc_split(__bfloat162float(v.x) * w.x, __bfloat162float(v.y) * w.y, ah[q], al[q]);
      }
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        // (with one tile per warp the second half of the load is the next warp's, or the row's padding: unused)
        unsigned b[4];
        ssc_ldsm4t(b, st + (ks * 16 + (mat & 1) * 8 + (lane & 7)) * RS + (warp * NW + j * 8 + (mat >> 1) * 8) * 2);
        ssc_mma(d[j], ah, b[0], b[1]);
        if (NT > 1) ssc_mma(d[NT > 1 ? j + 1 : j], ah, b[2], b[3]);
        ssc_mma(d[j], al, b[0], b[1]);
        if (NT > 1) ssc_mma(d[NT > 1 ? j + 1 : j], al, b[2], b[3]);
      }
    }
    const float total = w_s[SSC_Q];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(total, S[j][e], d[j][e]);
  }
  ssc_wait<0>();
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float2*>(st_head + 8 * h * N + 8 * j) = make_float2(S[j][2 * h], S[j][2 * h + 1]);
}

// A block: (chunk, group, 128 columns of the group's heads), a warp 16 of them (they lie in one head).  The outputs are formed
// transposed (rows columns of S, columns tokens): every part of the state is split into its terms by one warp only, and is
// used for all the chunk's tokens from registers.
__global__ void __launch_bounds__(SSC_OUT_WARPS * 32, 2)
ssd_out_kernel(const __nv_bfloat16* xbc, long long row_stride, int c_off, const float* __restrict__ d_skip,
               const float* scores, const int* cu_q, const int* req_slots,
               const int* token_req, float* __restrict__ out, int requests, int heads, int n_state, int pdim,
               int per_group, int tokens, int num_slots, int least, SscScratch sc) {
  constexpr int THREADS = SSC_OUT_WARPS * 32, COLS = SSC_OUT_WARPS * SSC_PT;
  constexpr int XS = COLS * 2 + 16;  // bytes between rows of x
  extern __shared__ __align__(16) unsigned char sc_smem[];
  pdl_launch_dependents();
  pdl_wait();
  int t0 = 0, req = 0;
  const int tile = blockIdx.x, group = blockIdx.y;
  const int cn = ssc_find(tile, cu_q, requests, least, req, t0);
  if (cn == 0 || token_req[t0] < 0) return;
  const int slot = req_slots[req];
  if (slot < 0 || slot >= num_slots) return;  // (reported by the walk)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mat = lane >> 3, g = lane >> 2, cp = (lane & 3) * 2;
  const int col0 = blockIdx.z * COLS, cols = min(COLS, per_group * pdim - col0);  // of the group's columns
  const int RS = n_state * 2 + 16;
  float* g_s = reinterpret_cast<float*>(sc_smem);                                  // [SSC_Q][SSC_G_STRIDE]
  float2* step_s = reinterpret_cast<float2*>(g_s + SSC_Q * SSC_G_STRIDE) + warp * SSC_Q;  // the warp's head: c_t, dt_t
  unsigned char* x_s = sc_smem + SSC_Q * SSC_G_STRIDE * 4 + SSC_OUT_WARPS * SSC_Q * 8;    // [SSC_Q][XS]
  unsigned char* c_s = x_s + SSC_Q * XS;                                                  // [SSC_Q][RS]
  const __nv_bfloat16* rows = xbc + (long long)t0 * row_stride;
  const int pieces = n_state >> 3, xp = cols >> 3;
  for (int i = tid; i < SSC_Q * pieces; i += THREADS) {
    const int row = i / pieces, ch = i - row * pieces;
    const bool ok = row < cn;
    ssc_cp_async_16(c_s + row * RS + ch * 16, rows + (ok ? row : 0) * row_stride + c_off + group * n_state + ch * 8, ok);
  }
  for (int i = tid; i < SSC_Q * xp; i += THREADS) {
    const int row = i / xp, ch = i - row * xp;
    const bool ok = row < cn;
    ssc_cp_async_16(x_s + row * XS + ch * 16, rows + (ok ? row : 0) * row_stride + group * per_group * pdim + col0 + ch * 8, ok);
  }
  for (int i = tid; i < SSC_Q * SSC_Q / 4; i += THREADS) {
    const int row = i / (SSC_Q / 4), ch = i - row * (SSC_Q / 4);
    // (only what lies on or below the diagonal's 16 x 16 blocks was written)
    const bool ok = row < cn && (ch >> 2) <= (row >> 4);
    ssc_cp_async_16(g_s + row * SSC_G_STRIDE + ch * 4, scores + ((long long)group * tokens + t0 + (ok ? row : 0)) * SSC_Q + ch * 4, ok);
  }
  ssc_commit();
  const bool works = warp * SSC_PT < cols;  // (a warp without columns only helps with the loads)
  const int in_group = col0 + (works ? warp * SSC_PT : 0);
  const int head = group * per_group + in_group / pdim, p0 = in_group % pdim;
#pragma unroll
  for (int i = 0; i < SSC_Q / 32; ++i) {
    const int t = lane + 32 * i;
    step_s[t] = sc.steps[(long long)head * tokens + t0 + (t < cn ? t : 0)];
  }
  const float* sp = sc.front + (((long long)tile * heads + head) * pdim + p0 + g) * n_state + cp;
  const int down = 8 * n_state;
  float2 x[4], y[4];
  x[0] = *reinterpret_cast<const float2*>(sp);
  x[1] = *reinterpret_cast<const float2*>(sp + down);
  x[2] = *reinterpret_cast<const float2*>(sp + 8);
  x[3] = *reinterpret_cast<const float2*>(sp + down + 8);
  const float skip = d_skip[head];
  ssc_wait<0>();
  __syncthreads();
  if (!works) return;
  float acc[SSC_Q / 8][4];
#pragma unroll
  for (int j = 0; j < SSC_Q / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  for (int kk = 0; kk < n_state; kk += 16) {  // what the state in front of the chunk gives
    const int nx = kk + 16 < n_state ? kk + 16 : kk;
    y[0] = *reinterpret_cast<const float2*>(sp + nx);
    y[1] = *reinterpret_cast<const float2*>(sp + down + nx);
    y[2] = *reinterpret_cast<const float2*>(sp + nx + 8);
    y[3] = *reinterpret_cast<const float2*>(sp + down + nx + 8);
    unsigned ah[4], al[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ssc_split(x[i].x, x[i].y, ah[i], al[i]);
#pragma unroll
    for (int j = 0; j < SSC_Q / 8; j += 2) {
      unsigned b[4];
      ssc_ldsm4(b, c_s + (j * 8 + (mat >> 1) * 8 + (lane & 7)) * RS + (kk + (mat & 1) * 8) * 2);
      ssc_mma(acc[j], ah, b[0], b[1]);
      ssc_mma(acc[j + 1], ah, b[2], b[3]);
      ssc_mma(acc[j], al, b[0], b[1]);
      ssc_mma(acc[j + 1], al, b[2], b[3]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = y[i];
  }
#pragma unroll
  for (int j = 0; j < SSC_Q / 8; ++j) {
    const float f0 = expf(step_s[j * 8 + cp].x), f1 = expf(step_s[j * 8 + cp + 1].x);
    acc[j][0] *= f0, acc[j][1] *= f1, acc[j][2] *= f0, acc[j][3] *= f1;
  }
  // what the tokens of this chunk leave to one another: the weighted scores as two terms, token j * 8 + g against the tokens s
#pragma unroll
  for (int ks = 0; ks < SSC_Q / 16; ++ks) {
    unsigned a[4];
    ssc_ldsm4t(a, x_s + (ks * 16 + (mat >> 1) * 8 + (lane & 7)) * XS + (warp * SSC_PT + (mat & 1) * 8) * 2);
    const int s0 = ks * 16 + cp;
    const float2 e0 = step_s[s0], e1 = step_s[s0 + 1], e2 = step_s[s0 + 8], e3 = step_s[s0 + 9];
#pragma unroll
    for (int j = 2 * ks; j < SSC_Q / 8; ++j) {  // (earlier tokens do not see these)
      const int t = j * 8 + g;
      const float ct = step_s[t].x;
      const float2 ga = *reinterpret_cast<const float2*>(g_s + t * SSC_G_STRIDE + s0);
      const float2 gb = *reinterpret_cast<const float2*>(g_s + t * SSC_G_STRIDE + s0 + 8);
      const float v0 = s0 <= t ? ga.x * (__expf(ct - e0.x) * e0.y) : 0.f, v1 = s0 + 1 <= t ? ga.y * (__expf(ct - e1.x) * e1.y) : 0.f;
      const float v2 = s0 + 8 <= t ? gb.x * (__expf(ct - e2.x) * e2.y) : 0.f, v3 = s0 + 9 <= t ? gb.y * (__expf(ct - e3.x) * e3.y) : 0.f;
      unsigned bh[2], bl[2];
      ssc_split(v0, v1, bh[0], bl[0]);
      ssc_split(v2, v3, bh[1], bl[1]);
      ssc_mma(acc[j], a, bh[0], bh[1]);
      ssc_mma(acc[j], a, bl[0], bl[1]);
    }
  }
#pragma unroll
  for (int j = 0; j < SSC_Q / 8; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = j * 8 + cp + i;
      if (t >= cn) continue;
      const __nv_bfloat16* xr = reinterpret_cast<const __nv_bfloat16*>(x_s + t * XS) + warp * SSC_PT + g;
      float* dst = out + ((long long)(t0 + t) * heads + head) * pdim + p0 + g;
      dst[0] = acc[j][i] + skip * __bfloat162float(xr[0]);
      dst[8] = acc[j][2 + i] + skip * __bfloat162float(xr[8]);
    }
}

// Sizes the chunked form takes (bfloat16): states of 32, 64, 128 or 256 rows, columns a multiple of 16.
extern "C" int ullm_ssd_chunk_supported(int heads, int n_state, int pdim, int groups) {
  return heads > 0 && groups > 0 && heads % groups == 0 && heads <= 65535 && pdim > 0 && pdim % 16 == 0 &&
         (n_state == 32 || n_state == 64 || n_state == 128 || n_state == 256);
}
extern "C" int ullm_ssd_chunk_tokens(void) { return SSC_Q; }

// Chunks a step has at most: every request that brings more than `least` tokens leaves one of them unfilled.
static int ssc_tiles(int tokens, int requests, int least) {
  const int chunked = tokens / (least + 1);
  return tokens / SSC_Q + (requests < chunked ? requests : chunked);
}
// Floats of `scratch` for a step of `tokens` tokens and `requests` requests.
extern "C" long long ullm_ssd_chunk_scratch(int tokens, int requests, int heads, int n_state, int pdim, int least) {
  return (long long)ssc_tiles(tokens, requests, least) * heads * ((long long)pdim * n_state + 1) + 3LL * heads * tokens;
}

template <int NT, int DEPTH>
static int walk_go(const __nv_bfloat16* xbc, long long row_stride, int b_off, float* state, long long state_stride,
                   const int* cu_q, const int* req_slots, const int* token_req, int tokens, int requests, int heads, int pdim,
                   int groups, int num_slots, int least, const SscScratch& sc, int* status, cudaStream_t st) {
  constexpr size_t smem = (size_t)DEPTH * (SSC_Q * (32 * NT * 2 + 16) + SSC_Q * (SSC_PT * 2 + 16) + (SSC_Q + 4) * 4);
  static_assert(smem <= 227 * 1024, "a walk's buffers fit the shared memory");
  static int attr_set = 0;
  if (!attr_set) {
    if (cudaFuncSetAttribute(ssd_walk_kernel<NT, DEPTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    attr_set = 1;
  }
  return ullm_launch_kernel(ssd_walk_kernel<NT, DEPTH>, dim3(pdim / SSC_PT, heads, requests), dim3(SSC_THREADS), smem, st, xbc,
                            row_stride, b_off, state, state_stride, cu_q, req_slots, token_req, heads, pdim, heads / groups,
                            tokens, num_slots, least, sc, status);
}

// Arguments as `ullm_ssd_recurrence`; `scores`: scratch of groups * tokens * SSC_Q floats, `scratch`: ullm_ssd_chunk_scratch
// floats, both on 16-byte borders.  Runs the requests that bring MORE than `least` tokens and leaves the others alone.
extern "C" int ullm_ssd_chunk(const void* xbc, long long row_stride, int b_off, int c_off, const float* dt,
                              const float* log_decay, const float* d_skip, float* scores, float* scratch, float* state,
                              long long state_stride, const int* cu_q, const int* req_slots, const int* token_req, float* out,
                              int tokens, int requests, int heads, int n_state, int pdim, int groups, int num_slots,
                              int least, int* status, void* stream, long long dt_stride) {
  cudaStream_t st = (cudaStream_t)stream;
  if (tokens < 0 || requests < 0 || num_slots <= 0 || scores == nullptr || scratch == nullptr || least < 0) return ULLM_ERR_BAD_SIZE;
  if (!ullm_ssd_chunk_supported(heads, n_state, pdim, groups) || requests > 65535) return ULLM_ERR_UNSUPPORTED;
  const int per_group = heads / groups, col_blocks = (per_group * pdim + SSC_OUT_WARPS * SSC_PT - 1) / (SSC_OUT_WARPS * SSC_PT);
  if (groups > 65534 || col_blocks > 65535) return ULLM_ERR_UNSUPPORTED;
  if (state_stride < (long long)heads * pdim * n_state || state_stride % 2) return ULLM_ERR_BAD_SIZE;
  if (row_stride % 8 || b_off % 8 || c_off % 8 || (((uintptr_t)xbc | (uintptr_t)scores | (uintptr_t)scratch) & 15) ||
      (((uintptr_t)state | (uintptr_t)out) & 7))
    return ULLM_ERR_BAD_SIZE;
  if (tokens == 0 || requests == 0) return ULLM_OK;
  const int tiles = ssc_tiles(tokens, requests, least);  // an upper bound on the chunks, however the tokens are spread
  if (tiles == 0) return ULLM_OK;
  SscScratch sc;
  sc.front = scratch;  // (n_state is a multiple of 32: what follows starts on a 16-byte border)
  sc.steps = reinterpret_cast<float2*>(scratch + (long long)tiles * heads * pdim * n_state);
  sc.weight = reinterpret_cast<float*>(sc.steps + (long long)heads * tokens);
  sc.total = sc.weight + (long long)heads * tokens;
  const size_t sc_smem = (size_t)2 * SSC_Q * (n_state * 2 + 16);
  const size_t out_smem = (size_t)SSC_Q * (SSC_G_STRIDE * 4 + SSC_OUT_WARPS * 8 + (SSC_OUT_WARPS * SSC_PT * 2 + 16) + n_state * 2 + 16);
  static size_t have[2] = {48 * 1024, 48 * 1024};
  if (sc_smem > have[0]) {
    if (cudaFuncSetAttribute(ssd_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sc_smem) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have[0] = sc_smem;
  }
  if (out_smem > have[1]) {
    if (cudaFuncSetAttribute(ssd_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    have[1] = out_smem;
  }
  const __nv_bfloat16* x = (const __nv_bfloat16*)xbc;
  int rc = ullm_launch_kernel(ssd_scores_kernel, dim3(tiles, groups + 1), dim3(SSC_THREADS), sc_smem, st, x, row_stride, b_off,
                              c_off, n_state, groups, dt, log_decay, dt_stride, heads, cu_q, token_req, requests, tokens, least,
                              scores, sc);
  if (rc != ULLM_OK) return rc;
#define SSC_WALK(NT, DEPTH)                                                                                                  \
  rc = walk_go<NT, DEPTH>(x, row_stride, b_off, state, state_stride, cu_q, req_slots, token_req, tokens, requests, heads, pdim, \
                          groups, num_slots, least, sc, status, st)
  switch (n_state) {
    case 32: SSC_WALK(1, 4); break;
    case 64: SSC_WALK(2, 4); break;
    case 128: SSC_WALK(4, 4); break;
    default: SSC_WALK(8, 3);
  }
#undef SSC_WALK
  if (rc != ULLM_OK) return rc;
  return ullm_launch_kernel(ssd_out_kernel, dim3(tiles, groups, col_blocks), dim3(SSC_OUT_WARPS * 32), out_smem, st, x,
                            row_stride, c_off, d_skip, (const float*)scores, cu_q, req_slots, token_req, out, requests, heads,
                            n_state, pdim, per_group, tokens, num_slots, least, sc);
}
