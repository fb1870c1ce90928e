// The grouped product of routed experts (csrc/moe.cu, `moe_grouped_linear`) for steps of many rows, bfloat16, on the 5th-
// generation tensor cores:  out[p] = f(W_e . (s_p * x[row(p)])) for every place p of every expert e.
//
// Bound by the tensor cores: at 2,048 tokens with 2 of 16 experts of 1,024 x 2,048 each (gated) the two products are 52 GFLOP,
// 31 us at the card's rate; measured with cold caches 58 + 33 us (69 + 37 with the MMAs issued by a lane in a branch of its own, whose
// descriptors take 58 clocks an instruction to uniform registers; 512 tokens then 46 + 25, bound by the 201 MB of matrices).  The mma.sync kernel of moe.cu takes 140 + 88 us there: tiles of 64 x 64 read both operands from
// shared memory once per 64 columns, and its warps spend their issue slots on ldmatrix.
//
// A persistent kernel, one block per SM, built as linear_tcgen05_large.cu: warp 0 loads, warp 1 issues the MMAs (M = 128,
// N = 256, K = 16; the whole warp, one lane elected), warps 2..5 drain the accumulators; four stages of 48 KB; two accumulators in tensor memory, so
// that a tile's activation and stores run behind the next tile's products.  What is different:
//
//   * a tile is 128 places of ONE expert x 256 rows of its matrix (gated: 128 gate rows and the same 128 rows of up, a
//     box each).  How many tiles there are only the device knows: every block forms the running count of row
//     tiles from `offsets` and takes the tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the row tiles of one expert and column
//     tile are neighbours, so that blocks that run together share the matrix rows in L2.
//   * x lies in place order already: the first product's rows are gathered by `moe_gather_rows` in a launch of its own (17 MB
//     written, 6 us at 2,048 tokens).  Loading them by tile::gather4, four rows a load, was slower than the mma.sync kernel: a
//     stage of 32 such loads took 1.4 us, three times as long as its products.
//   * a box of x is only as many rows high as the step has pairs (16, 32, 64 or 128): what the other rows of a stage hold is
//     multiplied too, into rows of the accumulator that are never stored.
//
// Every wait on an mbarrier is bounded (ULLM_STATUS_TIMEOUT in the status word, then the block waits, bounded, for the copies that
// it has in flight, and leaves).
#include "moe_act.cuh"
#include "tcgen05_util.cuh"

#define MT_BM 128
#define MT_BN 256
#define MT_BK 64
#define MT_STAGES 4
#define MT_THREADS 192
#define MT_A_BYTES (MT_BM * 128)
#define MT_B_BYTES (MT_BN * 128)
#define MT_STAGE_BYTES (MT_A_BYTES + MT_B_BYTES)
#define MT_MAX_EXPERTS 1024

struct MtParams {
  const int* offsets;         // [experts + 1]
  const int* sorted;          // the pair at every place (for its weight)
  const float* pair_weight;   // [pairs] or null
  __nv_bfloat16* out;         // [pairs, n_out]
  int experts, n_out, n_tiles, k_blocks;
  int box_rows, gated, act;
  float limit, alpha;
  int* status;
};

// Tile `tile` of the step: its expert (searched from the caller's `e` on; tiles only grow), its first place, its places, its
// column tile.
__device__ __forceinline__ void mt_find(const int* first, const int* offsets, int n_tiles, int tile, int& e, int& p0, int& rows,
                                        int& nt) {
  while ((long long)first[e + 1] * n_tiles <= tile) ++e;
  const int here = first[e + 1] - first[e], rem = tile - first[e] * n_tiles;
  nt = rem / here;
  const int lo = offsets[e], hi = offsets[e + 1];
  p0 = lo + (rem - nt * here) * MT_BM;
  rows = min(MT_BM, hi - p0);
}

// A thread's row of the tile out of tensor memory, activated, stored.  The gate without branches: with the division of
// `moe_gate_act`, whose slow path keeps a thread's 128 elements in series, the last tile's end took 20 us more (63 for 44 us at 32
// to 512 tokens, 87 for 69 at 2,048).
template <int ACT, bool GATED>
__device__ __forceinline__ void mt_store(const MtParams& p, uint32_t taddr, float sc, __nv_bfloat16* dst, int col0, bool on) {
  constexpr int COLS = GATED ? MT_BN / 2 : MT_BN;
#pragma unroll 1
  for (int c = 0; c < COLS; c += 16) {
    float v[16];
    tmem_ld16(taddr + c, v);
    if (GATED) {
      float u[16];
      tmem_ld16(taddr + MT_BN / 2 + c, u);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = moe_gate_act_flat<ACT>(v[i] * sc, u[i] * sc, p.limit, p.alpha);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = moe_plain_act(ACT, v[i] * sc);
    }
    if (on) {  // (n_out is a multiple of 8)
      const int col = col0 + c;
      uint4 w[2];
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      if (col < p.n_out) *reinterpret_cast<uint4*>(dst + col) = w[0];
      if (col + 8 < p.n_out) *reinterpret_cast<uint4*>(dst + col + 8) = w[1];
    }
  }
}

__global__ void __launch_bounds__(MT_THREADS, 1)
moe_grouped_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                           const MtParams p) {
  extern __shared__ unsigned char mt_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MT_STAGES], empty_bar[MT_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int wait_flag[2];
  __shared__ int first_s[MT_MAX_EXPERTS + 1];  // row tiles in front of every expert
  unsigned char* tiles = (unsigned char*)(((uintptr_t)mt_smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < MT_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full[0], 1);
    mbar_init(&acc_full[1], 1);
    mbar_init(&acc_empty[0], 4);
    mbar_init(&acc_empty[1], 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(lin_smem(&tmem_base_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    pdl_launch_dependents();  // (only now: a kernel behind this one must not hold tensor memory that this one waits for)
  }
  pdl_wait();
  if (warp == 0) {  // running count of row tiles, 32 experts at a time
    int before = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int n = e < p.experts ? (p.offsets[e + 1] - p.offsets[e] + MT_BM - 1) / MT_BM : 0;
      int sum = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (e < p.experts) first_s[e] = before + sum - n;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first_s[p.experts] = before;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = tmem_base_slot;
  const int num_tiles = first_s[p.experts] * p.n_tiles;

  if (warp == 0) {
    if (lane == 0) {
      // ---- loads -----------------------------------------------------------------------------------------------
      const uint32_t bytes = MT_B_BYTES + (uint32_t)p.box_rows * 128;
      int s = 0, e = 0, issued = 0;
      uint32_t parity = 1;  // a fresh barrier passes a wait on parity 1
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int p0, rows, nt;
        mt_find(first_s, p.offsets, p.n_tiles, tile, e, p0, rows, nt);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait(&empty_bar[s], parity)) {
            ullm_report(p.status, ULLM_STATUS_TIMEOUT, 51, kb);
            ok = false;
            break;
          }
          mbar_expect_tx(&full_bar[s], bytes);
          unsigned char* a = tiles + s * MT_STAGE_BYTES;
          if (p.gated) {
            tma_load_3d(a + MT_A_BYTES, &map_w, &full_bar[s], kb * MT_BK, nt * (MT_BN / 2), 2 * e);
            tma_load_3d(a + MT_A_BYTES + MT_B_BYTES / 2, &map_w, &full_bar[s], kb * MT_BK, nt * (MT_BN / 2), 2 * e + 1);
          } else {
            tma_load_3d(a + MT_A_BYTES, &map_w, &full_bar[s], kb * MT_BK, nt * MT_BN, e);
            tma_load_3d(a + MT_A_BYTES + MT_B_BYTES / 2, &map_w, &full_bar[s], kb * MT_BK, nt * MT_BN + MT_BN / 2, e);
          }
          tma_load_2d(a, &map_x, &full_bar[s], kb * MT_BK, p0);
          if (++s == MT_STAGES) s = 0, parity ^= 1;
          ++issued;
        }
      }
      // (a block in which a role gave up does not leave copies behind that are still on their way)
      for (int i = issued > MT_STAGES ? issued - MT_STAGES : 0; i < issued; ++i) mbar_wait(&full_bar[i % MT_STAGES], (i / MT_STAGES) & 1);
    }
  } else if (warp == 1) {
    // ---- MMAs (the whole warp, see `umma_bf16_warp`) -----------------------------------------------------------------------
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MT_BN >> 3) << 17) | ((uint32_t)(MT_BM >> 4) << 24);
    const uint64_t a0 = umma_desc(tiles);
    const uint32_t full0 = lin_smem(&full_bar[0]), empty0 = lin_smem(&empty_bar[0]), lead = elect_one();
    int s = 0, it = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++it) {
      const int buf = it & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1))) {
        if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 54, it);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem_d + (uint32_t)(buf * MT_BN);
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait_addr(full0 + 8 * s, phase))) {
          if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 52, kb);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t a = a0 + (uint64_t)(s * (MT_STAGE_BYTES >> 4)), b = a + (MT_A_BYTES >> 4);
        umma_bf16_warp(lead, d, a, b, idesc, kb > 0 ? 1u : 0u);
        umma_bf16_warp(lead, d, a + 2, b + 2, idesc, 1u);
        umma_bf16_warp(lead, d, a + 4, b + 4, idesc, 1u);
        umma_bf16_warp(lead, d, a + 6, b + 6, idesc, 1u);
        umma_commit_warp(lead, empty0 + 8 * s);
        if (++s == MT_STAGES) s = 0, phase ^= 1;
      }
      if (ok) umma_commit_warp(lead, lin_smem(&acc_full[buf]));
    }
  } else {
    // ---- results: a thread owns one place of the tile -----------------------------------------------------------------
    const int quarter = warp & 3, et = threadIdx.x - 64;
    int it = 0, e = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++it) {
      int p0, rows, nt;
      mt_find(first_s, p.offsets, p.n_tiles, tile, e, p0, rows, nt);
      const int buf = it & 1, row = quarter * 32 + lane;
      const bool on = row < rows;
      float sc = 1.f;
      if (on && p.pair_weight != nullptr) sc = p.pair_weight[p.sorted[p0 + row]];
      // (one thread waits, bounded, and tells the others, so that all 128 take the same way out)
      if (et == 0) {
        const bool got = mbar_wait(&acc_full[buf], (it >> 1) & 1);
        if (!got) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 53, it);
        wait_flag[it & 1] = got ? 1 : 0;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (wait_flag[it & 1] == 0) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_d + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * MT_BN);
      __nv_bfloat16* dst = p.out + (long long)(p0 + row) * p.n_out;
      const int cols = p.gated ? MT_BN / 2 : MT_BN;
      if (quarter * 32 < rows) {  // (a warp without places has nothing to read)
        if (!p.gated) {
          if (p.act == 3) mt_store<3, false>(p, taddr, sc, dst, nt * cols, on);
          else mt_store<-1, false>(p, taddr, sc, dst, nt * cols, on);
        } else if (p.act == 0) {
          mt_store<0, true>(p, taddr, sc, dst, nt * cols, on);
        } else if (p.act == 2) {
          mt_store<2, true>(p, taddr, sc, dst, nt * cols, on);
        } else {
          mt_store<1, true>(p, taddr, sc, dst, nt * cols, on);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(512) : "memory");
  }
}

// a bfloat16 tensor of two or three dimensions, boxes of 64 columns x box_rows (x box_deep), 128-byte swizzle
static bool mt_map(CUtensorMap* m, const void* ptr, long long cols, long long rows, long long deep, long long row_bytes,
                   int box_rows, int box_deep) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)deep};
  cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)row_bytes * (cuuint64_t)rows};
  cuuint32_t box[3] = {MT_BK, (cuuint32_t)box_rows, (cuuint32_t)box_deep};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, deep > 0 ? 3 : 2, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// out[p] = x[sorted[p] / top] for every place p that belongs to an expert, 16 bytes at a time
__global__ void moe_gather_rows_kernel(const uint4* x, long long x_stride, const int* sorted,
                                       const int* offsets, int experts, int top, uint4* __restrict__ out,
                                       int pieces) {
  pdl_launch_dependents();
  pdl_wait();
  const int p = blockIdx.x;
  if (p >= offsets[experts]) return;  // (what `sorted` holds behind them was never written)
  const uint4* src = x + (long long)(sorted[p] / top) * x_stride;
  for (int i = threadIdx.x; i < pieces; i += blockDim.x) out[(long long)p * pieces + i] = src[i];
}

// Arguments as `ullm_moe_grouped_linear` in bfloat16, with the weights one after the other, and the status word; `gathered`
// [pairs, k_dim]: where rows_from_pairs has its rows gathered (unused otherwise).  UNSUPPORTED for sizes and alignments that the
// loads or the 16-byte stores cannot take.
extern "C" int ullm_moe_grouped_tcgen05(const void* x, long long x_stride, void* gathered, const void* weights,
                                        const int* offsets, const int* sorted, const float* pair_weight, void* out, int pairs,
                                        int experts, int top, int rows_from_pairs, int n_out, int k_dim, int gated, int act,
                                        float limit, float alpha, int* status, void* stream) {
  if (pairs < 0 || experts <= 0 || top <= 0 || n_out <= 0 || k_dim <= 0) return ULLM_ERR_BAD_SIZE;
  if (gated && (act < 0 || act > 2)) return ULLM_ERR_UNSUPPORTED;
  if (gated && act == 2 && !(limit > 0.f)) return ULLM_ERR_BAD_SIZE;
  if (rows_from_pairs && gathered == nullptr) return ULLM_ERR_UNSUPPORTED;
  if (experts > MT_MAX_EXPERTS || k_dim % 8 || x_stride % 8 || n_out % 8 ||
      (((uintptr_t)x | (uintptr_t)weights | (uintptr_t)out | (uintptr_t)gathered) & 15))
    return ULLM_ERR_UNSUPPORTED;
  if (pairs == 0) return ULLM_OK;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(moe_grouped_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             MT_STAGES * MT_STAGE_BYTES + 1024) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    sms = n;
  }
  cudaStream_t st = (cudaStream_t)stream;
  MtParams p;
  p.offsets = offsets;
  p.sorted = sorted;
  p.pair_weight = pair_weight;
  p.out = (__nv_bfloat16*)out;
  p.experts = experts;
  p.n_out = n_out;
  p.n_tiles = (n_out + (gated ? MT_BN / 2 : MT_BN) - 1) / (gated ? MT_BN / 2 : MT_BN);
  p.k_blocks = (k_dim + MT_BK - 1) / MT_BK;
  p.box_rows = MT_BM;
  while (p.box_rows > 16 && p.box_rows / 2 >= pairs) p.box_rows /= 2;  // (no expert has more places than the step has pairs)
  p.gated = gated ? 1 : 0;
  p.act = act;
  p.limit = limit;
  p.alpha = alpha;
  p.status = status;
  const long long most = ((long long)(pairs + MT_BM - 1) / MT_BM + experts) * p.n_tiles;  // tiles, whatever the routing
  if (most > 0x7fffffffLL) return ULLM_ERR_BAD_SIZE;
  const void* rows = rows_from_pairs ? gathered : x;
  CUtensorMap map_x, map_w;
  if (!mt_map(&map_x, rows, k_dim, pairs, 0, (rows_from_pairs ? (long long)k_dim : x_stride) * 2, p.box_rows, 1) ||
      !mt_map(&map_w, weights, k_dim, n_out, (long long)experts * (gated ? 2 : 1), (long long)k_dim * 2,
              MT_BN / 2, 1))
    return ULLM_ERR_LAUNCH;
  if (rows_from_pairs) {
    const int pieces = k_dim / 8;
    int threads = 64;
    while (threads < 256 && threads < pieces) threads <<= 1;
    const int rc = ullm_launch_kernel(moe_gather_rows_kernel, dim3(pairs), dim3(threads), 0, st, (const uint4*)x, x_stride / 8,
                                      sorted, offsets, experts, top, (uint4*)gathered, pieces);
    if (rc != ULLM_OK) return rc;
  }
  return ullm_launch_kernel(moe_grouped_tcgen05_kernel, dim3((int)(most < sms ? most : sms)), dim3(MT_THREADS),
                            (size_t)MT_STAGES * MT_STAGE_BYTES + 1024, st, map_x, map_w, p);
}
