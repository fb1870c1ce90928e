// out[M, N] = x[M, K] . w[N, K]^T (+ bias) in float32 for many rows, on the 5th-generation tensor cores.
//
// Every float32 operand, times 2^24, is the sum of three bfloat16 numbers, the rounded value, the rounded rest and the rest of that.
// The 24 bits of a number from 2^-126 on then lie at 2^-125 and above, so that none of them is lost under bfloat16's smallest
// exponent (2^-133 without the factor: a number below 2^-110 would lose its last bits); the results are scaled back.  Of the nine products of terms the six down to 2^-16 of the first are
// formed, h h + h m + m h + m m + h l + l h; what is left out is 2^-24 of a product, half a unit in its last place.  The sums of a
// k block of 64 run in tensor memory, smallest products first, and are then added to float32 registers by ordinary rounded
// additions: the tensor core's own additions do not round to nearest, and over a whole row of K that would show.
//
// What bounds it: the products themselves, 12 or 24 per k block, and the splitting of w (22 instructions for four values) and shared
// memory close behind (288 KB per k block of 128 x 128 results: 2,250 cycles, for 1,536 of the tensor pipe).  So x is split once, by a
// kernel of its own, into three planes that TMA brings; w, which is read by few blocks each, is split on the way in.  The library's
// float32 product is bound by its multiply-add instructions.  Measured with cold caches, against the library: 511 rows, 4,096 columns of
// k 1,024 34 us for 92; 6,144 of 1,024 54 for 150; 1,024 of 3,072 42 for 90; 100 rows, 6,144 of 1,024 24.  Errors against 64 bits there:
// 1.0e-7 to 1.5e-7, the library's 5.7e-7 to 2.0e-6.
//
// Warps 0..7 load rows of w (one or two k blocks ahead, in registers; four more are asked for into L2: 31.7 and 29.7 us for 511 x 1,024 x
// 2,048 when that was brought in, 31.7 with it since the issuing warps wait for their stage), split them and store the terms in K-major 128-byte-swizzled tiles; a thread of warp 0 asks for the planes of x; warps 16 and 17
// issue the products, a k block each in turn (one thread for all of them paced everything, 1,500 clocks a k block of 32 columns: 52 us for
// 511 x 1,024 x 3,072); warps 8..15 add the block sums up, a quarter of the rows and half of the columns each.  Two or three stages, two
// or four block sums in tensor memory.  BN from 32 to 128, so that the tiles fill the SMs.
//
// Infinities, NaN, operands from 2^104 on and sums from 2^80 on (which the factor takes to infinity) turn a sum into an infinity or
// NaN that float32 may not show: such a result is formed again with multiply-adds from the rows themselves.
//
// Every wait on an mbarrier is bounded (ULLM_STATUS_TIMEOUT in the status word, then the role leaves, and the others after it).
#include "ring_turns.h"
#include "tcgen05_util.cuh"

#define FS_BM 128
#define FS_BK 64
#define FS_ISSUERS 2
#define FS_FETCH 4  // k blocks of w that are asked for into L2 beyond those in registers
#define FS_THREADS ((16 + FS_ISSUERS) * 32)
#define FS_A_BYTES (FS_BM * 128)  // one term of x

// two neighbouring floats in one 64-bit register, the low one first, for the instructions that work on both
__device__ __forceinline__ unsigned long long fs_pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
// v as two bfloat16, and v without them
__device__ __forceinline__ unsigned fs_term(unsigned long long& v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  const unsigned t = *reinterpret_cast<const unsigned*>(&h);
  const unsigned long long taken = fs_pair(__uint_as_float(t << 16), __uint_as_float(t & 0xffff0000u)), minus = fs_pair(-1.f, -1.f);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(taken), "l"(minus));
  return t;
}
#define FS_UP 0x1p24f
#define FS_DOWN 0x1p-48f
// four neighbouring values as three groups of four bfloat16
__device__ __forceinline__ void fs_split(const float4& v, uint2& h, uint2& m, uint2& l) {
  unsigned long long a = fs_pair(v.x, v.y), b = fs_pair(v.z, v.w);
  const unsigned long long up = fs_pair(FS_UP, FS_UP);
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(up));
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(b) : "l"(up));
  h.x = fs_term(a), h.y = fs_term(b);
  m.x = fs_term(a), m.y = fs_term(b);
  l.x = fs_term(a), l.y = fs_term(b);
}

// x [M][K] as three planes of bfloat16 terms [3][M][stride]; four values per thread
__global__ void f32_terms_kernel(const float* x, __nv_bfloat16* __restrict__ terms, int M, int K, int stride) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_row = K / 4;
  const long long n = (long long)M * per_row, plane = (long long)M * stride;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / per_row;
    const int c = (int)(i - row * per_row) * 4;
    uint2 h, m, l;
    fs_split(*reinterpret_cast<const float4*>(x + row * K + c), h, m, l);
    __nv_bfloat16* d = terms + row * stride + c;
    *reinterpret_cast<uint2*>(d) = h;
    *reinterpret_cast<uint2*>(d + plane) = m;
    *reinterpret_cast<uint2*>(d + 2 * plane) = l;
  }
}

struct FsParams {
  const float* x;
  const float* w;
  const float* bias;
  float* out;
  int M, N, K;
  int* status;
};

template <int BN>
__global__ void __launch_bounds__(FS_THREADS, 1) linear_f32_split_kernel(const __grid_constant__ CUtensorMap x_map, const FsParams p) {
  constexpr int FS_STAGES = BN <= 64 ? 3 : 2, AHEAD = BN <= 64 ? 2 : 1;  // AHEAD: k blocks of w on their way
  // Up to 64 columns the terms of w stand side by side as up to 3 BN columns of ONE instruction per term of x, whose sums of a kind
  // meet in the same columns: 12 instructions per k block instead of 24 (an instruction's time hardly falls below 64 columns).
  constexpr bool JOINED = BN <= 64;
  constexpr int FS_SUMS = BN == 64 ? 2 : 4, SUM_COLS = JOINED ? 3 * BN : BN;  // block sums in tensor memory, columns of one
  constexpr int B_BYTES = BN * 128, STAGE = 3 * (FS_A_BYTES + B_BYTES);
  constexpr int TMEM_COLS = 512;  // FS_SUMS * SUM_COLS are 384 or 512
  constexpr int HALF = BN / 2;  // columns of an adding warp
  extern __shared__ unsigned char fs_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[FS_STAGES], empty_bar[FS_STAGES], acc_full[FS_SUMS], acc_empty[FS_SUMS];
  __shared__ uint32_t tmem_slot;
  unsigned char* tiles = (unsigned char*)(((uintptr_t)fs_smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (p.M + FS_BM - 1) / FS_BM;
  const int m0 = (int)(blockIdx.x % m_tiles) * FS_BM, n0 = (int)(blockIdx.x / m_tiles) * BN;  // (neighbours share rows of w)
  const int k_blocks = (p.K + FS_BK - 1) / FS_BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < FS_STAGES; ++s) {
      mbar_init(&full_bar[s], 9);  // eight splitting warps, and the planes of x
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < FS_SUMS; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(lin_smem(&tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    pdl_launch_dependents();  // (only now: a kernel behind this one must not hold tensor memory that this one waits for)
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = tmem_slot;
  // w into L2 some k blocks before a thread loads it: its registers hold one or two blocks, too few for the way from memory
  auto fetch = [&](int kb) {
    if (kb >= k_blocks) return;
    for (int i = threadIdx.x; i < BN * 2; i += 256) {
      const long long row = n0 + (i >> 1), col = (long long)kb * FS_BK + (i & 1) * 32;
      if (row < p.N && col < p.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + row * p.K + col));
    }
  };
  if (warp < 8)
    for (int kb = 0; kb < AHEAD + FS_FETCH; ++kb) fetch(kb);
  pdl_wait();

  if (warp < 8) {
    // ---- terms: 16 threads take the 64 values of a row of the k block, the block's 256 threads 16 rows at a time --------------
    const int row0 = threadIdx.x >> 4, c4 = threadIdx.x & 15;
    float4 rb[AHEAD][BN / 16];
    const float* ws = p.w + (long long)(n0 + row0) * p.K + c4 * 4;
    const long long down = 16LL * p.K;
    const bool whole = n0 + BN <= p.N && p.K % FS_BK == 0;  // (nothing to check row by row)
    auto load = [&](float4 (&r)[BN / 16], int kb) {
      const float* src = ws + kb * FS_BK;
      if (whole) {
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) r[i] = __ldg(reinterpret_cast<const float4*>(src + i * down));
      } else {
#pragma unroll
        for (int i = 0; i < BN / 16; ++i)
          r[i] = (n0 + row0 + 16 * i < p.N && kb * FS_BK + c4 * 4 < p.K) ? __ldg(reinterpret_cast<const float4*>(src + i * down))
                                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
#pragma unroll
    for (int q = 0; q < AHEAD; ++q)
      if (q < k_blocks) load(rb[q], q);
    // (rows 16 apart: the swizzle's row & 7 is the thread's own)
    const int at = 3 * FS_A_BYTES + row0 * 128 + (((c4 >> 1) ^ (row0 & 7)) << 4) + (c4 & 1) * 8;
    int s = 0, issued = 0;
    uint32_t parity = 1;
    bool ok = true;
    for (int kb0 = 0; kb0 < k_blocks && ok; kb0 += AHEAD) {
#pragma unroll
      for (int q = 0; q < AHEAD; ++q) {
        const int kb = kb0 + q;
        if (kb >= k_blocks || !ok) break;
        if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], parity))) {
          if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 61, kb);
          ok = false;
          break;
        }
        unsigned char* st = tiles + s * STAGE;
        if (threadIdx.x == 0) {
          mbar_expect_tx(&full_bar[s], 3 * FS_A_BYTES);
#pragma unroll
          for (int t = 0; t < 3; ++t) tma_load_3d(st + t * FS_A_BYTES, &x_map, &full_bar[s], kb * FS_BK, m0, t);
        }
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {
          uint2 h, m, l;
          fs_split(rb[q][i], h, m, l);
          unsigned char* d = st + at + i * 2048;
          *reinterpret_cast<uint2*>(d) = h;
          *reinterpret_cast<uint2*>(d + B_BYTES) = m;
          *reinterpret_cast<uint2*>(d + 2 * B_BYTES) = l;
        }
        if (kb + AHEAD < k_blocks) load(rb[q], kb + AHEAD);
        fetch(kb + AHEAD + FS_FETCH);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
        if (++s == FS_STAGES) s = 0, parity ^= 1;
        issued = kb + 1;
      }
    }
    if (threadIdx.x == 0)  // (a block that gives up does not leave copies behind that are still on their way)
      for (int kb = issued > FS_STAGES ? issued - FS_STAGES : 0; kb < issued; ++kb)
        mbar_wait(&full_bar[kb % FS_STAGES], (kb / FS_STAGES) & 1);
  } else if (warp >= 16) {
    // ---- products: two warps take the k blocks in turn, each block with a stage and a block sum of its own, so that one's waits and
    // commits pass while the other's products run (a warp stands still while the tensor core's queue is full) --------------------------
    // (How neither takes an old use of a stage or a sum for the present one: ring_turns.h.)
    static_assert(FS_ISSUERS <= FS_STAGES && FS_ISSUERS <= FS_SUMS, "what ring_issue_turn asks for");
    auto idesc = [](int columns) {
      return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns >> 3) << 17) | ((uint32_t)(FS_BM >> 4) << 24);
    };
    const uint64_t desc0 = umma_desc(tiles);
    const uint32_t lead = elect_one();
    for (int kb = warp - 16; kb < k_blocks; kb += FS_ISSUERS) {
      const int s = kb % FS_STAGES, buf = kb % FS_SUMS;
      const bool turn = ring_issue_turn(kb, FS_STAGES, FS_SUMS, [&](RingBarrier which, int i, unsigned parity) {
        return mbar_wait(which == RING_STAGE_EMPTY ? &empty_bar[i] : which == RING_STAGE_FULL ? &full_bar[i] : &acc_empty[i], parity);
      });
      if (!__all_sync(0xffffffffu, turn)) {
        if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 62, kb);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem_d + (uint32_t)(buf * SUM_COLS);
      const uint64_t a = desc0 + (uint64_t)((s * STAGE) >> 4), b = a + (3 * FS_A_BYTES >> 4);
      constexpr uint32_t A1 = FS_A_BYTES >> 4, B1 = B_BYTES >> 4;
      if (JOINED) {  // columns 0: h h; BN: h m + m h; 2 BN: h l + m m + l h
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_warp(lead, d, a + 2 * k, b + 2 * k, idesc(3 * BN), k > 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_warp(lead, d + BN, a + A1 + 2 * k, b + 2 * k, idesc(2 * BN), 1u);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_warp(lead, d + 2 * BN, a + 2 * A1 + 2 * k, b + 2 * k, idesc(BN), 1u);
      } else {
        const uint32_t ta[6] = {2 * A1, 0, A1, A1, 0, 0}, tb[6] = {0, 2 * B1, B1, 0, B1, 0};  // l h, h l, m m, m h, h m, h h
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_warp(lead, d, a + ta[t] + 2 * k, b + tb[t] + 2 * k, idesc(BN), t > 0 || k > 0 ? 1u : 0u);
      }
      umma_commit_warp(lead, lin_smem(&empty_bar[s]));
      umma_commit_warp(lead, lin_smem(&acc_full[buf]));
    }
  } else {
    // ---- sums ------------------------------------------------------------------------------------------------------------
    const int quarter = warp & 3, c0 = ((warp - 8) >> 2) * HALF;
    float acc[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
    bool ok = true;
    int buf = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < k_blocks; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], phase))) {
        if (lane == 0) ullm_report(p.status, ULLM_STATUS_TIMEOUT, 63, kb);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t = tmem_d + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * SUM_COLS + c0);
#pragma unroll
      for (int c = 0; c < HALF; c += 16) {
        float v[16];
        if (JOINED) {  // the smaller products first
          float u[16];
          tmem_ld16(t + 2 * BN + c, v);
          tmem_ld16(t + BN + c, u);
#pragma unroll
          for (int i = 0; i < 16; ++i) u[i] += v[i];
          tmem_ld16(t + c, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] += u[i];
        } else {
          tmem_ld16(t + c, v);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += v[i];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      if (++buf == FS_SUMS) buf = 0, phase ^= 1;
    }
    const int row = m0 + quarter * 32 + lane;
    if (ok && row < p.M) {
      float* dst = p.out + (long long)row * p.N + n0 + c0;
      unsigned long long odd = 0;  // the columns whose sum is infinite or NaN
#pragma unroll
      for (int c = 0; c < HALF; c += 4) {
        const int col = n0 + c0 + c;
        if (col < p.N) {  // (N is a multiple of 4)
          float v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[i] = acc[c + i] * FS_DOWN;
            if (!(fabsf(acc[c + i]) <= 3.4028234e38f)) odd |= 1ull << (c + i);
            if (p.bias != nullptr) v[i] += __ldg(p.bias + col + i);
          }
          *reinterpret_cast<float4*>(dst + c) = make_float4(v[0], v[1], v[2], v[3]);
        }
      }
      // (In a loop of its own: beside every result, unrolled, it was 20 us of code to fetch on the way past, at 128 columns.)
#pragma unroll 1
      while (odd != 0) {
        const int c = __ffsll(odd) - 1, col = n0 + c0 + c;
        odd &= odd - 1;
        const float *xr = p.x + (long long)row * p.K, *wr = p.w + (long long)col * p.K;
        float sum = 0.f;
#pragma unroll 1
        for (int k = 0; k < p.K; ++k) sum = fmaf(xr[k], wr[k], sum);
        if (p.bias != nullptr) sum += __ldg(p.bias + col);
        dst[c] = sum;
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 16) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(TMEM_COLS));
  }
}

template <int BN>
static int fs_go(const CUtensorMap& x_map, const FsParams& p, long long tiles, cudaStream_t st) {
  constexpr int smem = (BN <= 64 ? 3 : 2) * 3 * (FS_A_BYTES + BN * 128) + 1024;
  static_assert(smem <= 227 * 1024 - 256, "the stages fit the shared memory");
  static int attr_set = 0;
  if (!attr_set) {
    if (cudaFuncSetAttribute(linear_f32_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return ULLM_ERR_LAUNCH;
    }
    attr_set = 1;
  }
  return ullm_launch_kernel(linear_f32_split_kernel<BN>, dim3((unsigned)tiles), dim3(FS_THREADS), (size_t)smem, st, x_map, p);
}

// Columns per tile by (waves of tiles) x (ns of a k block, measured: 511 rows, 1,024 columns of k 1,024 to 4,096 in tiles of 32, 64,
// 96 and 128: 21.5 to 52, 23.5 to 61, 27.7 to 81, 31.7 to 85 us in one wave each, the last three before the issuing warps waited for their
// stage, which added 2 us to the first and nothing to its slope); the wider tile where both agree.  0: the device's SM count cannot be
// read.
extern "C" int ullm_linear_f32_split_columns(int M, int N) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      return 0;
    sms = n;
  }
  const double ns[4] = {640., 770., 950., 1070.};
  int best = 0;
  double least = 0.;
  for (int bn = 128; bn >= 32; bn -= 32) {
    const long long tiles = (long long)((M + FS_BM - 1) / FS_BM) * ((N + bn - 1) / bn);
    const double cost = (double)((tiles + sms - 1) / sms) * ns[bn / 32 - 1];
    if (best == 0 || cost < least) best = bn, least = cost;
  }
  return best;
}
// bfloat16 numbers of the planes of x
extern "C" long long ullm_linear_f32_split_terms(int M, int K) { return 3LL * M * ((K + 7) / 8 * 8); }

// All contiguous, 16-byte aligned, K and N multiples of 4; `bias` [N] or null; `terms`: scratch of ullm_linear_f32_split_terms
// bfloat16 numbers.  UNSUPPORTED for anything else (nothing has run).
extern "C" int ullm_linear_f32_split(const float* x, const float* w, const float* bias, float* out, void* terms, int M, int N, int K,
                                     int* status, void* stream) {
  if (M < 0 || N <= 0 || K <= 0 || terms == nullptr) return ULLM_ERR_BAD_SIZE;
  if (N % 4 || K % 4 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out | (uintptr_t)terms) & 15)) return ULLM_ERR_UNSUPPORTED;
  if (M == 0) return ULLM_OK;
  const FsParams p = {x, w, bias, out, M, N, K, status};
  const int best = ullm_linear_f32_split_columns(M, N);
  if (best == 0) return ULLM_ERR_LAUNCH;
  const long long tiles = (long long)((M + FS_BM - 1) / FS_BM) * ((N + best - 1) / best);
  if (tiles > 0x7fffffffLL) return ULLM_ERR_UNSUPPORTED;
  const int stride = (K + 7) / 8 * 8;
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return ULLM_ERR_LAUNCH;
  CUtensorMap x_map;
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
  cuuint64_t strides[2] = {(cuuint64_t)stride * 2, (cuuint64_t)stride * 2 * M};
  cuuint32_t box[3] = {FS_BK, FS_BM, 1}, estr[3] = {1, 1, 1};
  if (enc(&x_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, terms, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return ULLM_ERR_LAUNCH;
  cudaStream_t st = (cudaStream_t)stream;
  const long long pieces = ((long long)M * (K / 4) + 255) / 256;
  const int rc = ullm_launch_kernel(f32_terms_kernel, dim3((unsigned)(pieces < 2368 ? pieces : 2368)), dim3(256), 0, st, x,
                                    (__nv_bfloat16*)terms, M, K, stride);
  if (rc != ULLM_OK) return rc;
  if (best == 128) return fs_go<128>(x_map, p, tiles, st);
  if (best == 96) return fs_go<96>(x_map, p, tiles, st);
  if (best == 64) return fs_go<64>(x_map, p, tiles, st);
  return fs_go<32>(x_map, p, tiles, st);
}
