// The grouped product of routed experts (csrc/moe.cu, `moe_grouped_linear`) for steps of at most 16 tokens, bfloat16: the chosen
// experts' matrices streamed once.
//
// Bound by memory: 8 tokens with 2 of 16 experts (gated, 1,024 x 2,048) reach about 10 experts, 84 MB of gate and up rows, 13 us
// at the copy rate.  The mma.sync kernel of moe.cu took 41 us there: a block of four warps keeps 64 x 64 tiles of both operands
// in flight by cp.async, a sixth of what the SM needs, and pads an expert's one or two rows to 64.  Measured, first and second
// product, with cold caches, against that kernel: 1 token 12.5 + 10.4 us for 34 + 17; 8 tokens 27 + 18 for 41 + 23; 16 tokens
// 36 + 23 for 43 + 32; 32 experts of 2,048 x 4,096: 1 token 25 + 15 for 58 + 32, 16 tokens 133 + 78 for 198 + 117.
//
// The streaming scheme of linear_stream.cu (its shared pieces in linear_stream_core.cuh): units of 32 weight rows (gated: 16 gate
// rows and the same 16 of up) dealt round robin to two blocks per SM; one thread fills a ring of stages (32 rows x 256 k by one or
// two TMA boxes, and the tokens' rows), eight mma.sync warps (weights as the 16-row operand, tokens as its 8 columns) share a
// stage by row half and k quarter and meet in shared memory at the end of a unit.  What is different:
//   * which experts have rows only the device knows: behind `griddepcontrol.wait` a block lists them from `offsets`, and unit u
//     belongs to the (u / units per expert)-th of them.  (So the ring cannot be filled in front of the wait.)
//   * in the first product every expert meets ALL tokens of the step (the tensor instruction has room for 8 or 16 anyway), and
//     only the results of the tokens that chose it are stored, at their places: no gathered copy of the rows.  In the second an
//     expert's rows are neighbours: its box begins at its first place.
//
// A token may name an expert more than once (a router's choices never do; the product itself is defined for any).  In the first
// product a result then goes to several places, found place by place; in the second an expert can have more rows than the tensor
// instruction has columns, and its matrix is streamed once per 8 NT of them.
//
// Every wait on an mbarrier is bounded (ULLM_STATUS_TIMEOUT in the status word; a block that gives up waits, bounded, for the
// copies it has in flight, and returns).
#include "linear_stream_core.cuh"
#include "moe_act.cuh"

#define MS_MAX_TOKENS 16
#define MS_MAX_EXPERTS 1024
#define MS_MAX_PASSES 64  // of 8 NT places of one expert (16 tokens of 64 choices all at one expert)
#define MS_SMEM_KB 100  // ring and partial sums of a block: two blocks per SM beside the static arrays

struct MsParams {
  const int* offsets;        // [experts + 1]
  const int* sorted;         // the pair at every place
  const float* pair_weight;  // [pairs] or null
  __nv_bfloat16* out;        // [pairs, n_out]
  int experts, top, from_tokens, n_out, rows, k_blocks, units_per_expert, stages;
  int gated, act;
  float limit, alpha;
  int* status;
};

__device__ __forceinline__ void ms_store(const MsParams& p, int at, int col, float r, float up, float sc) {
  const float y = p.gated ? moe_gate_act(p.act, r * sc, up * sc, p.limit, p.alpha) : moe_plain_act(p.act, r * sc);
  p.out[(size_t)at * p.n_out + col] = __float2bfloat16_rn(y);
}

// A result that goes to several places.  (Not inlined: sixteen copies of it in the tail of every unit made the kernel's code eight
// times as long.)
__device__ __noinline__ void ms_store_many(const MsParams& p, int lo, int n_e, int token, int col, float r, float up) {
#pragma unroll 1
  for (int q = 0; q < n_e; ++q) {
    const int pair = p.sorted[lo + q];
    if (pair / p.top == token) ms_store(p, lo + q, col, r, up, p.pair_weight != nullptr ? p.pair_weight[pair] : 1.f);
  }
}

template <int NT>
__global__ void __launch_bounds__(LS_THREADS, 2)
moe_stream_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ MsParams p) {
  constexpr int X_BOX_BYTES = 8 * NT * 128;  // 8 NT rows x 64 k
  constexpr int STAGE_BYTES = LS_W_STAGE_BYTES + 4 * X_BOX_BYTES;
  extern __shared__ unsigned char ms_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[LS_MAX_STAGES], empty_bar[LS_MAX_STAGES];
  __shared__ unsigned short live_s[MS_MAX_EXPERTS + MS_MAX_PASSES];  // the experts that have rows (the low 10 bits), and the pass over their places
  __shared__ int count_s, abort_flag, many_s;
  __shared__ int place_s[MS_MAX_TOKENS];    // where the unit's result of every token goes (-1: nowhere)
  __shared__ float scale_s[MS_MAX_TOKENS];
  pdl_launch_dependents();
  unsigned char* ring = (unsigned char*)(((uintptr_t)ms_smem_raw + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(ring + p.stages * STAGE_BYTES);  // [8 warps][32 lanes][NT][4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], LS_CONSUMER_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  pdl_wait();
  if (warp == 0) {
    int n = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int rows = e < p.experts ? p.offsets[e + 1] - p.offsets[e] : 0;
      const int passes = p.from_tokens ? (rows > 0 ? 1 : 0) : (rows + 8 * NT - 1) / (8 * NT);
      const unsigned mask = __ballot_sync(0xffffffffu, passes > 0);
      int at = n + __popc(mask & ((1u << lane) - 1u)), all = __popc(mask);
      if (__any_sync(0xffffffffu, passes > 1)) {
        int sum = passes;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += v;
        }
        at = n + sum - passes;
        all = __shfl_sync(0xffffffffu, sum, 31);
      }
      for (int i = 0; i < passes; ++i) live_s[at + i] = (unsigned short)(e | i << 10);
      n += all;
    }
    if (lane == 0) count_s = n;
  }
  __syncthreads();
  const int num_units = count_s * p.units_per_expert, grid = (int)gridDim.x;
  const int my_units = num_units > (int)blockIdx.x ? (num_units - 1 - (int)blockIdx.x) / grid + 1 : 0;
  const int total_it = my_units * p.k_blocks;

  if (warp == LS_CONSUMER_WARPS) {
    if (lane == 0) {
      // ---- loads -----------------------------------------------------------------------------------------------
      int slot = 0, round = 0;
      bool ok = true;
      for (int ui = 0; ui < my_units && ok; ++ui) {
        const int u = (int)blockIdx.x + ui * grid, a = u / p.units_per_expert, v = u - a * p.units_per_expert;
        const int e = live_s[a] & 1023, x_row = p.from_tokens ? 0 : p.offsets[e] + (live_s[a] >> 10) * 8 * NT;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (round > 0 && !mbar_wait(&empty_bar[slot], (round - 1) & 1)) {
            ullm_report(p.status, ULLM_STATUS_TIMEOUT, 56, ui);
            abort_flag = 1;
            ok = false;
            break;
          }
          unsigned char* st = ring + slot * STAGE_BYTES;
          mbar_expect_tx(&full_bar[slot], STAGE_BYTES);
          if (p.gated) {
            tma_load_3d(st, &w_map, &full_bar[slot], 0, e * p.rows + v * 16, kb * 4);
            tma_load_3d(st + 8192, &w_map, &full_bar[slot], 0, e * p.rows + p.n_out + v * 16, kb * 4);
          } else {
            tma_load_3d(st, &w_map, &full_bar[slot], 0, e * p.rows + v * 32, kb * 4);
          }
          tma_load_3d(st + LS_W_STAGE_BYTES, &x_map, &full_bar[slot], 0, x_row, kb * 4);
          if (++slot == p.stages) slot = 0, ++round;
        }
      }
    }
  } else {
    // ---- products ----------------------------------------------------------------------------------------------
    const int mt = warp & 1, kq = warp >> 1, g = lane >> 2, t = lane & 3;
    const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_chunk = lane >> 4;
    const int b_row = (lane & 7) + (lane >> 4) * 8, b_chunk = (lane >> 3) & 1;
    bool failed = false;
    int s = 0;
    uint32_t parity = 0;
    for (int ui = 0; ui < my_units; ++ui) {
      const int u = (int)blockIdx.x + ui * grid, ea = u / p.units_per_expert, v = u - ea * p.units_per_expert;
      const int e = live_s[ea] & 1023, lo = p.offsets[e] + (live_s[ea] >> 10) * 8 * NT;
      const int n_e = p.from_tokens ? p.offsets[e + 1] - lo : min(p.offsets[e + 1] - lo, 8 * NT);
      if (warp == 0) {  // (read by the finishing warps behind the unit's barrier)
        if (lane < MS_MAX_TOKENS) place_s[lane] = -1, scale_s[lane] = 1.f;
        __syncwarp();
        int col = 32 + lane;  // (no token's)
        if (lane < n_e) {
          const int pair = p.sorted[lo + lane];
          col = p.from_tokens ? pair / p.top : lane;
          if (col < MS_MAX_TOKENS) {
            place_s[col] = lo + lane;
            if (p.pair_weight != nullptr) scale_s[col] = p.pair_weight[pair];
          }
        }
        bool many = n_e > 32;
        if (p.from_tokens) {  // (as many tokens as places, unless one comes twice)
          const unsigned seen = __reduce_or_sync(0xffffffffu, col < MS_MAX_TOKENS ? 1u << col : 0u);
          many |= __popc(seen) != __popc(__ballot_sync(0xffffffffu, col < MS_MAX_TOKENS));
        }
        if (lane == 0) many_s = many ? 1 : 0;  // (some token's result goes to several places)
      }
      float acc[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!failed && !__all_sync(0xffffffffu, mbar_wait(&full_bar[s], parity))) {
          ullm_report(p.status, ULLM_STATUS_TIMEOUT, 57, ui);  // (the whole warp gives up together)
          abort_flag = 1;
          failed = true;
        }
        uint32_t a[4][4], b[4][2 * NT];
        if (!failed) {
          // (gated: two boxes [4 chunks][16 rows][128 B]; else one [4 chunks][32 rows][128 B])
          const uint32_t wbox = lin_smem(ring + s * STAGE_BYTES + (p.gated ? (mt * 4 + kq) * 2048 : kq * 4096 + mt * 2048));
          const uint32_t xbox = lin_smem(ring + s * STAGE_BYTES + LS_W_STAGE_BYTES + kq * X_BOX_BYTES);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            ls_ldmatrix4(a[j], wbox + a_row * 128 + (((j * 2 + a_chunk) ^ (a_row & 7)) << 4));
            if constexpr (NT == 1) {
              const int r = lane & 7, c = (lane >> 3) & 1;
              ls_ldmatrix2(b[j][0], b[j][1], xbox + r * 128 + (((j * 2 + c) ^ r) << 4));
            } else {
              uint32_t t4[4];
              ls_ldmatrix4(t4, xbox + b_row * 128 + (((j * 2 + b_chunk) ^ (b_row & 7)) << 4));
              b[j][0] = t4[0], b[j][1] = t4[1], b[j][2] = t4[2], b[j][3] = t4[3];
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);
        if (!failed) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int n = 0; n < NT; ++n) ls_mma(acc[n], a[j], b[j][2 * n], b[j][2 * n + 1]);
        }
        if (++s == p.stages) s = 0, parity ^= 1;
      }
      // ---- the k quarters meet; quarter 0's warps (gated: the one of the gate rows) finish the unit ----------------
#pragma unroll
      for (int n = 0; n < NT; ++n)
        *reinterpret_cast<float4*>(red + ((size_t)(warp * 32 + lane) * NT + n) * 4) =
            make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
      ls_bar_sync_consumers();
      if (kq == 0 && (!p.gated || mt == 0) && !failed) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          float r[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // in quarter order: the same sum whatever the timing
            const float4 x = *reinterpret_cast<const float4*>(red + ((size_t)((q * 2 + mt) * 32 + lane) * NT + n) * 4);
            r[0] += x.x, r[1] += x.y, r[2] += x.z, r[3] += x.w;
            if (p.gated) {
              const float4 y = *reinterpret_cast<const float4*>(red + ((size_t)((q * 2 + 1) * 32 + lane) * NT + n) * 4);
              up[0] += y.x, up[1] += y.y, up[2] += y.z, up[3] += y.w;
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // accumulator element i: weight row g + 8 (i >> 1), token 8 n + 2 t + (i & 1)
            const int m = n * 8 + 2 * t + (i & 1);
            const int col = p.gated ? v * 16 + g + 8 * (i >> 1) : v * 32 + mt * 16 + g + 8 * (i >> 1);
            if (col >= p.n_out) continue;
            if (many_s == 0) {
              if (place_s[m] >= 0) ms_store(p, place_s[m], col, r[i], up[i], scale_s[m]);
            } else {
              ms_store_many(p, lo, n_e, m, col, r[i], up[i]);
            }
          }
        }
      }
      ls_bar_sync_consumers();  // (sums and places are read: the next unit may overwrite them)
    }
  }
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      int last = -1;
      for (int it = s; it < total_it; it += p.stages) last = it;
      if (last >= 0) mbar_wait(&full_bar[s], (last / p.stages) & 1);
    }
  }
}

template <int NT>
static int ms_launch(const CUtensorMap& w, const CUtensorMap& x, MsParams p, int sms, cudaStream_t st) {
  constexpr int STAGE_BYTES = LS_W_STAGE_BYTES + 4 * 8 * NT * 128;
  const int red = LS_CONSUMER_WARPS * 32 * NT * 4 * (int)sizeof(float);
  p.stages = (MS_SMEM_KB * 1024 - 1024 - red) / STAGE_BYTES;
  const size_t smem = (size_t)p.stages * STAGE_BYTES + red + 1024;
  static bool allowed = false;
  if (!allowed) {
    if (cudaFuncSetAttribute(moe_stream_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM_KB * 1024) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    cudaFuncSetAttribute(moe_stream_kernel<NT>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    allowed = true;
  }
  return ullm_launch_kernel(moe_stream_kernel<NT>, dim3(2 * sms), dim3(LS_THREADS), smem, st, w, x, p);
}

// Arguments as `ullm_moe_grouped_linear` in bfloat16 with the weights one after the other, and the status word; x contiguous,
// pairs / top tokens (at most 16).  UNSUPPORTED for sizes and alignments that the boxes cannot take.
extern "C" int ullm_moe_stream(const void* x, const void* weights, const int* offsets, const int* sorted,
                               const float* pair_weight, void* out, int pairs, int experts, int top, int rows_from_pairs,
                               int n_out, int k_dim, int gated, int act, float limit, float alpha, int* status, void* stream) {
  if (pairs < 0 || experts <= 0 || top <= 0 || n_out <= 0 || k_dim <= 0) return ULLM_ERR_BAD_SIZE;
  if (gated && (act < 0 || act > 2)) return ULLM_ERR_UNSUPPORTED;
  if (gated && act == 2 && !(limit > 0.f)) return ULLM_ERR_BAD_SIZE;
  const int tokens = pairs / top, NT = tokens <= 8 ? 1 : 2;
  if (pairs % top || tokens > MS_MAX_TOKENS || pairs > MS_MAX_PASSES * 8 * NT || experts > MS_MAX_EXPERTS || k_dim % 64 || n_out % (gated ? 16 : 32) ||
      (((uintptr_t)x | (uintptr_t)weights) & 15))
    return ULLM_ERR_UNSUPPORTED;
  if (pairs == 0) return ULLM_OK;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
      sms = 0;
      return ULLM_ERR_LAUNCH;
    }
  }
  MsParams p = {};
  p.offsets = offsets;
  p.sorted = sorted;
  p.pair_weight = pair_weight;
  p.out = (__nv_bfloat16*)out;
  p.experts = experts;
  p.top = top;
  p.from_tokens = rows_from_pairs ? 1 : 0;
  p.n_out = n_out;
  p.rows = (gated ? 2 : 1) * n_out;
  p.k_blocks = (k_dim + LS_BK - 1) / LS_BK;
  p.units_per_expert = n_out / (gated ? 16 : 32);
  p.gated = gated ? 1 : 0;
  p.act = act;
  p.limit = limit;
  p.alpha = alpha;
  p.status = status;
  CUtensorMap wm, xm;
  if (!ls_chunked_map(weights, (long long)experts * p.rows, k_dim, gated ? 16 : 32, &wm) ||
      !ls_chunked_map(x, rows_from_pairs ? tokens : pairs, k_dim, 8 * NT, &xm))
    return ULLM_ERR_LAUNCH;
  return NT == 1 ? ms_launch<1>(wm, xm, p, sms, (cudaStream_t)stream) : ms_launch<2>(wm, xm, p, sms, (cudaStream_t)stream);
}
