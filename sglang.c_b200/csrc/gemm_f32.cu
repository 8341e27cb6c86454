// C[M,N] = A[M,K] · W[N,K]^T (+ bias[N]) with an optional activation, or added into a 32-bit residual stream in
// place: the products of the 32-bit path on the 5th-generation tensor cores.
//
// Every 32-bit number is cut, exactly, into three bfloat16 pieces (8 bits of its mantissa each: x = x1 + x2 + x3),
// and of the nine products of pieces the six that matter are summed in 32 bits:
//   a·w = a1 w3 + a2 w2 + a3 w1 + a1 w2 + a2 w1 + a1 w1        (what is left out is below 2^-22 |a w|, and of either sign)
// A product of pieces is exact; the sums over a chunk of FK = 64 k are made in tensor memory, the small terms first, and
// the chunks' sums are added in 32-bit registers (rounded to nearest), one after another.  That order depends on nothing:
// an output has the same bits whatever the number of rows, the tile, or the number of blocks that share a tile's K.  The
// error against float64 is below that of one accumulator taking k = 0..K-1 (normal numbers, K = 768: 9.0e-8 of the
// result's norm against 4.0e-7; K = 3,072: 1.5e-7 against 9.3e-7), because a chain of K roundings becomes one of K / 64 and
// short ones inside the chunks.  (Tensor memory cuts where registers round: with two chunks to a sum in tensor memory the
// error was five times as large.)
// An output that is no finite number (an infinity or NaN among its operands, whose pieces are no numbers, or an
// overflow) is computed again as a plain chain of multiply-adds, so that infinities come out as they do there.  Numbers
// below 2^-110 end where bfloat16 does: their last piece is a multiple of 2^-133.
//
// W's rows are the MMA's 128-row side and the tokens its N, for every number of tokens.  A block's warps each have one
// task, so that none waits for another's latencies: one brings W's chunks by TMA and WW cut them into tensor memory
// (both ahead of the dependency wait: weights do not change; the MMA then reads only the tokens' pieces from shared
// memory, with both there its reads would take longer than the multiplications), AW load the tokens' numbers and cut
// them into shared memory in the 128-byte swizzle, one issues the MMAs, DW add up the chunks' sums and finish the tile.
//
// What bounds it: for many tokens shared memory (128 x 128 outputs and 64 k take 272 KB of it: 2,176 clocks of about 2,600
// measured, where the six multiplications take 1,536): 768 x 768 x 1,872 tokens 19.3 us (multiply-adds: 69.3), 3,072 x 768 57
// (205), 768 x 3,072 61 (249).  For few, a chain of latencies: the launch, a chunk's cut, its sums' way (K = 768, 8 tokens:
// 5 to 7 us; over K 3,072 8.0, where an output's chain of multiply-adds took 12.6).
#include <atomic>

#include "common.cuh"
#include "tc_common.cuh"

SGLC_DEFINE_ERROR_STRING()

namespace {
using namespace tc;

constexpr int FM = 128;          // features of a tile: MMA M, TMEM lanes
constexpr int FK = 64;           // k of a chunk: 128 bytes of bfloat16, one swizzle row
constexpr int W_BYTES = FM * FK * 4;
constexpr int MOST_RANKS = 16;
constexpr int SMS = 148;
constexpr int A_COLS = 3 * FK / 2;      // tensor-memory columns of a chunk of W: three planes of 32

struct F32Args {
  const float* A; const float* W; const float* bias;
  float* out; float* residual;
  int M, N, K, lda, ldo, act;
  int chunks, ranks, per_rank;          // chunks of K; blocks that share a tile, and the chunks each takes
  int tiles_n, tiles;
  int* err;
  // Not null: the columns from q_cols on are keys and values of the step's tokens ([keys of `heads` heads of `dim`][values
  // likewise]) and go into the paged cache [page][2][heads][page][dim] at slots[token] (negative: nowhere), not into out.
  float* cache;
  const int* slots;
  int q_cols, heads, dim, page, n_pages;
};
// where a token's slot lies in the cache, and where a column lies in a page
__device__ __forceinline__ long long slot_at(const F32Args& p, int m) {
  const int slot = m < p.M ? p.slots[m] : -1, page = slot / p.page;
  if (slot < 0 || page >= p.n_pages) return -1;
  return ((long long)page * 2 * p.heads * p.page + slot % p.page) * p.dim;
}
__device__ __forceinline__ long long column_at(const F32Args& p, int f) {
  const int c = f - p.q_cols;
  return (long long)(c / p.dim) * p.page * p.dim + c % p.dim;
}

// The pieces of two numbers, packed (the first one in the low half): the upper half of x; what that leaves, rounded to eight
// bits (c = 65537 r, c - (c - r): Veltkamp's splitting); and the rest, which is exact (24 bits of mantissa).  Two numbers an
// instruction where there is one, the work shared between the multiply-add units and the bit operations of half their
// rate.  (Conversions to bfloat16 go through the special-function unit at an eighth of the rate.)
__device__ __forceinline__ float2 fma2(float2 x, float2 y, float2 z) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(reinterpret_cast<unsigned long long&>(x)), "l"(reinterpret_cast<unsigned long long&>(y)),
        "l"(reinterpret_cast<unsigned long long&>(z)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 mul2(float2 x, float2 y) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(x)), "l"(reinterpret_cast<unsigned long long&>(y)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  const float2 minus = make_float2(-1.0f, -1.0f);
  p1 = __byte_perm(u0, u1, 0x7632);
  const float2 h = make_float2(__uint_as_float(u0 & 0xffff0000u), __uint_as_float(u1 & 0xffff0000u));
  const float2 r = fma2(h, minus, make_float2(x0, x1));
  const float2 c = mul2(r, make_float2(65537.0f, 65537.0f));
  const float2 g = fma2(fma2(r, minus, c), minus, c);
  p2 = __byte_perm(__float_as_uint(g.x), __float_as_uint(g.y), 0x7632);
  const float2 s = fma2(g, minus, r);
  p3 = __byte_perm(__float_as_uint(s.x), __float_as_uint(s.y), 0x7632);
}

// D (+)= A·B with A in tensor memory.
__device__ __forceinline__ void mma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 16 lanes x 8 columns: thread t gives registers 0, 1 to lane (base + t/4), columns 2(t%4), +1, and 2, 3 to lane base + t/4 + 8.
__device__ __forceinline__ void tmem_st_16x256b_x1(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ bool finite(float s) { return fabsf(s) <= 3.402823466e38f; }
// An output as a plain chain of multiply-adds, k = 0..K-1.  (Few loads at once: a function that takes more registers
// costs the kernels that call it 2 % where none is called.)
__device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
  float s = 0.0f;
#pragma unroll 2
  for (int k = 0; k < K / 4; k++) {
    const float4 x = reinterpret_cast<const float4*>(a)[k], y = reinterpret_cast<const float4*>(w)[k];
    s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
  }
  return s;
}
// Whether there is a NaN among the 16-byte pieces first, first + step, ... of a row.
__device__ __forceinline__ bool any_nan(const float* row, int K, int first, int step) {
  bool nan = false;
#pragma unroll 4
  for (int k = first; k < K / 4; k += step) {
    const float4 x = reinterpret_cast<const float4*>(row)[k];
    nan = nan || x.x != x.x || x.y != x.y || x.z != x.z || x.w != x.w;
  }
  return nan;
}
// A token's outputs of a warp's features (a row of w each) that are no finite numbers, made again (v where `bad` is false).  A NaN among
// the token's numbers, which the warp looks for together, or among a feature's makes the output NaN without a chain: in a step
// whose values have become NaN a chain for every output took hundreds of times the tile (1,872 tokens, 768 over 768 5.4 ms,
// now 0.09, with a NaN in each row of w 0.12, and 0.02 where all is finite; 768 over 3,072 22.4 ms, now 0.25).  w_nan: what
// was found out about the lane's row of w; -1: nothing yet.
struct Again { float v; int w_nan; };
__device__ __noinline__ Again plain_again(const float* a, const float* w, int K, bool bad, float v, int w_nan) {
  const bool a_nan = __any_sync(0xffffffffu, any_nan(a, K, threadIdx.x & 31, 32));
  if (bad) {
    if (!a_nan && w_nan < 0) w_nan = any_nan(w, K, 0, 1);
    v = a_nan || w_nan > 0 ? __int_as_float(0x7fffffff) : plain_dot(a, w, K);
  }
  __syncwarp();
  return {v, w_nan};
}
// The same where blocks share a tile, whose outputs are few: given up where it has become NaN (8 tokens, 768 over 3,072, all NaN
// 236 -> 17 us).
__device__ __noinline__ float plain_until_nan(const float* a, const float* w, int K) {
  float s = 0.0f;
  for (int k0 = 0; k0 < K && s == s; k0 += FK) {
    const int n = min(FK, K - k0) / 4;
#pragma unroll 4
    for (int k = 0; k < n; k++) {
      const float4 x = reinterpret_cast<const float4*>(a + k0)[k], y = reinterpret_cast<const float4*>(w + k0)[k];
      s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
    }
  }
  return s;
}

// Blocks walk tiles (features fastest), all of K each; or, CLUSTER, the blocks of a cluster share one tile: rank r takes the
// chunks r * per_rank .. and gives each chunk's sums to the block that owns the feature.
template <int NT, int WW, int AW, int DW, bool CLUSTER>
__global__ void __launch_bounds__((WW + AW + DW + (NT >= 64 ? 3 : 2)) * 32, NT == 16 ? 2 : 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ F32Args p) {
  constexpr bool A_TMA = NT >= 64;                      // the tokens' numbers come through shared memory, too
  constexpr int W_STAGES = CLUSTER || NT == 128 || NT == 16 ? 2 : 3;
  constexpr int PF = NT <= 32 ? 2 : 1;                  // chunks of A whose loads are in flight
  constexpr int GROUPS_K = 16 / WW;                     // groups of 16 k of a chunk that a warp cuts of W
  constexpr int AT = AW * 32;
  constexpr int BI = NT * 8 / AT;                       // 16-byte pieces a thread writes of a chunk of A's plane
  constexpr int CW = NT * 4 / DW;                       // columns of the accumulator a warp reads
  constexpr int PLANE = NT * 128, STAGE = 3 * PLANE;
  constexpr int COLS = 2 * NT + 2 * A_COLS <= 256 ? 256 : 512;
  constexpr int NTP = NT + 4;                           // padded row of a chunk's sums
  static_assert((A_TMA ? NT / 4 % AW == 0 : NT * 8 % AT == 0) && CW % 16 == 0 && (WW == 4 || WW == 8), "whole pieces");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* w_ring = smem + 2 * STAGE;                   // W_STAGES chunks of W: two boxes of 128 rows x 32 floats
  constexpr int A_BYTES = A_TMA ? NT * FK * 4 : 0;
  uint8_t* a_ring = w_ring + W_STAGES * W_BYTES;        // two chunks of A likewise
  float* red = reinterpret_cast<float*>(a_ring + 2 * A_BYTES);             // the sums of all chunks for this block's features
  __shared__ uint64_t ready[2], done[2], read[2],       // a chunk is cut, its MMAs have ended, its sums have been taken
       w_full[W_STAGES], w_empty[W_STAGES], a_full[2], a_empty[2],
       taken;                                           // (CLUSTER) all chunks' sums have been taken
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3;
  const int rank = CLUSTER ? blockIdx.z : 0;
  const int c0 = rank * p.per_rank, n = min(p.chunks - c0, p.per_rank);       // (every rank has at least one chunk)
  const int first = CLUSTER ? blockIdx.y * gridDim.x + blockIdx.x : blockIdx.x, step = CLUSTER ? p.tiles : gridDim.x;
  const int total = (p.tiles - first + step - 1) / step * n;              // chunks of this block, tile after tile

  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(&done[i], 1);
      mbar_init(&ready[i], WW + AW);
      mbar_init(&read[i], DW);
      mbar_init(&a_full[i], 1);
      mbar_init(&a_empty[i], AW);
    }
    for (int i = 0; i < W_STAGES; i++) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], WW);
    }
    mbar_init(&taken, DW);
    abort_s = 0;
    mbar_fence_init();
  }
  __syncwarp();
  // A block of a cluster never waits for another one while it holds tensor memory, except for its start, and that is ahead of
  // the allocation: the columns are given back before the blocks wait for one another's sums.  Otherwise two clusters of
  // launches in two streams, this kernel's and one of bfloat16 products, could each hold on one SM what the other one's
  // block waits for there, for good.
  if (CLUSTER) cluster_arrive_relaxed();                // (waited for ahead of the first store into a peer's memory)
  if (warp == 0) {
    tmem_alloc(&tmem_s, COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // Behind the allocation: blocks of the launch behind, which hold tensor memory while they wait for this one, come
  // only when every block of this one has its own.
  pdl_launch_dependents();
  const uint32_t tmem = tmem_s;
  const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
  bool held = true;                                     // (warp 0: the columns)

  if (warp < WW) {
    // ---- cut W ----
    // Lane l of tensor memory has the feature row in which the lowest three bits of l are turned round by one: the rows r
    // and r + 4 that a quarter of a warp's 16-byte reads touches lie on different banks in the swizzle, the rows r and r + 1
    // would not.
    const int q = lane & 3, g8 = lane >> 2, w_row = quarter * 32 + (g8 & 1) * 4 + (g8 >> 1), g0 = warp / 4 * GROUPS_K;
    for (int it = 0; it < total; it++) {
      const int st = it & 1, s = it % W_STAGES;
      mbar_wait(&w_full[s], (it / W_STAGES) & 1, abort_flag);
      if (it >= 2) {
        mbar_wait(&done[st], ((it >> 1) - 1) & 1, abort_flag);
        tc_fence_after_sync();
      }
#pragma unroll
      for (int e = 0; e < GROUPS_K; e += 2) {
        float4 r[2][2][2];
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
              const int row = w_row + h * 16 + c * 8, g = g0 + e + x;
              r[x][h][c] = *reinterpret_cast<const float4*>(w_ring + s * W_BYTES + (g >> 1) * (W_BYTES / 2) + row * 128 +
                                                            (((4 * (g & 1) + q) ^ (row & 7)) << 4));
            }
        if (e + 2 >= GROUPS_K) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&w_empty[s]);
        }
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t v[3][4];
#pragma unroll
            for (int c = 0; c < 2; c++) {
              split_pair(r[x][h][c].x, r[x][h][c].y, v[0][2 * c], v[1][2 * c], v[2][2 * c]);
              split_pair(r[x][h][c].z, r[x][h][c].w, v[0][2 * c + 1], v[1][2 * c + 1], v[2][2 * c + 1]);
            }
#pragma unroll
            for (int pl = 0; pl < 3; pl++)
              tmem_st_16x256b_x1(lanes + ((uint32_t)(h * 16) << 16) + 2 * NT + st * A_COLS + pl * (FK / 2) + 8 * (g0 + e + x),
                                 v[pl][0], v[pl][1], v[pl][2], v[pl][3]);
          }
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[st]);
    }
  } else if (warp >= WW + DW && warp < WW + DW + AW) {
    // ---- load and cut the tokens' numbers ----
    if constexpr (A_TMA) {
      // Eight rows and four 16-byte pieces a warp: the rows that a quarter of its reads and writes touches, r and r with its
      // bits 0 and 2 turned over, lie on different banks in both swizzles.
      const int j4 = lane & 3, low = (lane >> 2 & 1) | (lane >> 4) << 1 | ((lane >> 2 ^ lane >> 3) & 1) << 2, aw = warp - WW - DW;
      for (int it = 0; it < total; it++) {
        const int st = it & 1;
        mbar_wait(&a_full[st], (it >> 1) & 1, abort_flag);
        if (it >= 2) mbar_wait(&done[st], ((it >> 1) - 1) & 1, abort_flag);
#pragma unroll
        for (int x = 0; x < NT / 4 / AW; x++) {
          const int i = aw + x * AW, half = i & 1, row = (i >> 1) * 8 + low, j = 4 * half + j4;
          float4 r[2];
#pragma unroll
          for (int s = 0; s < 2; s++)
            r[s] = *reinterpret_cast<const float4*>(a_ring + st * A_BYTES + half * (NT * 128) + row * 128 + (((2 * j4 + s) ^ (row & 7)) << 4));
          uint32_t v[3][4];
#pragma unroll
          for (int s = 0; s < 2; s++) {
            split_pair(r[s].x, r[s].y, v[0][2 * s], v[1][2 * s], v[2][2 * s]);
            split_pair(r[s].z, r[s].w, v[0][2 * s + 1], v[1][2 * s + 1], v[2][2 * s + 1]);
          }
          uint8_t* dst = smem + st * STAGE + row * 128 + ((j ^ (row & 7)) << 4);
#pragma unroll
          for (int pl = 0; pl < 3; pl++)
            *reinterpret_cast<uint4*>(dst + pl * PLANE) = make_uint4(v[pl][0], v[pl][1], v[pl][2], v[pl][3]);
        }
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&a_empty[st]);
          mbar_arrive(&ready[st]);
        }
      }
    } else {
      const int t = tid - (WW + DW) * 32;
      float4 rb[PF][BI][2];
      int l_tile = first, l_chunk = 0;                    // what is loaded next
      auto load = [&](float4 (&r)[BI][2]) {
        const int m0 = l_tile / p.tiles_n * NT, kc = (c0 + l_chunk) * FK;
#pragma unroll
        for (int b = 0; b < BI; b++) {
          const int x = t + b * AT, j = x & 7, m = m0 + (x >> 3);
#pragma unroll
          for (int s = 0; s < 2; s++) {
            const int k = kc + 8 * j + 4 * s;
            r[b][s] = m < p.M && k < p.K ? *reinterpret_cast<const float4*>(p.A + (size_t)m * p.lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        if (++l_chunk == n) {
          l_chunk = 0;
          l_tile += step;
        }
      };
      pdl_wait();
#pragma unroll
      for (int u = 0; u < PF; u++)
        if (u < total) load(rb[u]);
      for (int i0 = 0; i0 < total; i0 += PF) {
#pragma unroll
        for (int u = 0; u < PF; u++) {
          const int it = i0 + u, st = it & 1;
          if (it >= total) break;
          if (it >= 2) mbar_wait(&done[st], ((it >> 1) - 1) & 1, abort_flag);
#pragma unroll
          for (int b = 0; b < BI; b++) {
            const int x = t + b * AT, j = x & 7, row = x >> 3;
            uint32_t v[3][4];
#pragma unroll
            for (int s = 0; s < 2; s++) {
              split_pair(rb[u][b][s].x, rb[u][b][s].y, v[0][2 * s], v[1][2 * s], v[2][2 * s]);
              split_pair(rb[u][b][s].z, rb[u][b][s].w, v[0][2 * s + 1], v[1][2 * s + 1], v[2][2 * s + 1]);
            }
            uint8_t* dst = smem + st * STAGE + row * 128 + ((j ^ (row & 7)) << 4);
#pragma unroll
            for (int pl = 0; pl < 3; pl++)
              *reinterpret_cast<uint4*>(dst + pl * PLANE) = make_uint4(v[pl][0], v[pl][1], v[pl][2], v[pl][3]);
          }
          fence_async_proxy();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ready[st]);
          if (it + PF < total) load(rb[u]);
        }
      }
    }
  } else if (warp == WW + DW + AW) {
    // ---- W by TMA ----
    if (elect_one()) {
      int issued = 0, tile = first, chunk = 0;
      for (int it = 0; it < total; it++) {
        const int s = it % W_STAGES;
        if (it >= W_STAGES && !mbar_wait(&w_empty[s], (it / W_STAGES - 1) & 1, abort_flag)) break;
        mbar_expect_tx(&w_full[s], W_BYTES);
        for (int h = 0; h < 2; h++)
          tma_load_2d(w_ring + s * W_BYTES + h * (W_BYTES / 2), &map_w, &w_full[s], (c0 + chunk) * FK + 32 * h,
                      tile % p.tiles_n * FM);
        issued = it + 1;
        if (++chunk == n) {
          chunk = 0;
          tile += step;
        }
      }
      if (*abort_flag)                                  // (no block may end with copies under way)
        for (int i = max(0, issued - W_STAGES); i < issued; i++) mbar_wait(&w_full[i % W_STAGES], (i / W_STAGES) & 1, abort_flag);
    }
    __syncwarp();
  } else if (A_TMA && warp == WW + DW + AW + 2) {
    // ---- A by TMA ----
    if (elect_one()) {
      pdl_wait();
      int issued = 0, tile = first, chunk = 0;
      for (int it = 0; it < total; it++) {
        const int s = it & 1;
        if (it >= 2 && !mbar_wait(&a_empty[s], ((it >> 1) - 1) & 1, abort_flag)) break;
        mbar_expect_tx(&a_full[s], A_BYTES);
        for (int h = 0; h < 2; h++)
          tma_load_2d(a_ring + s * A_BYTES + h * (A_BYTES / 2), &map_a, &a_full[s], (c0 + chunk) * FK + 32 * h, tile / p.tiles_n * NT);
        issued = it + 1;
        if (++chunk == n) {
          chunk = 0;
          tile += step;
        }
      }
      if (*abort_flag)
        for (int i = max(0, issued - 2); i < issued; i++) mbar_wait(&a_full[i & 1], (i >> 1) & 1, abort_flag);
    }
    __syncwarp();
  } else if (warp == WW + DW + AW + 1) {
    // ---- MMAs ----
    if (elect_one()) {
      constexpr uint32_t idesc = idesc_bf16_f32(FM, NT);
      constexpr int WP[6] = {2, 1, 0, 1, 0, 0}, AP[6] = {0, 1, 2, 0, 1, 0};
      for (int it = 0; it < total; it++) {
        const int st = it & 1;
        if (!mbar_wait(&ready[st], (it >> 1) & 1, abort_flag)) break;
        if (it >= 2 && !mbar_wait(&read[st], ((it >> 1) - 1) & 1, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t d = tmem + st * NT, w0 = tmem + 2 * NT + st * A_COLS;
        const uint64_t a0 = smem_desc_k_sw128(smem_u32(smem + st * STAGE));
#pragma unroll
        for (int t = 0; t < 6; t++)
#pragma unroll
          for (int g = 0; g < FK / 16; g++)
            mma_bf16_ta(d, w0 + WP[t] * (FK / 2) + 8 * g, a0 + (uint64_t)(AP[t] * PLANE / 16 + 2 * g), idesc, t + g > 0 ? 1u : 0u);
        mma_commit(&done[st]);
      }
    }
    __syncwarp();
  } else {
    // ---- add up, and finish ----
    const int part = (warp - WW) / 4, my_row = quarter * 32 + (lane & 24) + (lane & 1) * 4 + ((lane & 7) >> 1);
    const int rows_per = CLUSTER ? (FM + p.ranks - 1) / p.ranks : FM;
    float sum[CW];
    bool ok = true, peers = false;
    pdl_wait();
    for (int i0 = 0, tile = first; tile < p.tiles; i0 += n, tile += step) {
      const int n0 = tile % p.tiles_n * FM, m0 = tile / p.tiles_n * NT;
      __syncwarp();
      for (int i = 0; i < n; i++) {
        const int st = (i0 + i) & 1;
        ok = mbar_wait(&done[st], ((i0 + i) >> 1) & 1, abort_flag) && ok;
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < CW; c += 16) {
          uint32_t r[16];
          tmem_ld_32x16(lanes + st * NT + part * CW + c, r);
          tmem_ld_wait();
          if (CLUSTER || i == 0) {
#pragma unroll
            for (int j = 0; j < 16; j++) sum[c + j] = __uint_as_float(r[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j++) sum[c + j] += __uint_as_float(r[j]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&read[st]);
        if constexpr (CLUSTER) {
          if (i == n - 1 && lane == 0) mbar_arrive(&taken);
          if (!peers) {
            cluster_wait();
            peers = true;
          }
          const uint32_t remote = map_to_peer(red + ((size_t)(c0 + i) * rows_per + my_row % rows_per) * NTP + part * CW, my_row / rows_per);
#pragma unroll
          for (int j = 0; j < CW; j += 4)
            st_peer_v4(remote + 4u * j, __float_as_uint(sum[j]), __float_as_uint(sum[j + 1]), __float_as_uint(sum[j + 2]),
                       __float_as_uint(sum[j + 3]));
        }
      }
      if constexpr (!CLUSTER) {
        const int f = n0 + my_row, mt = m0 + part * CW;
        if (__any_sync(0xffffffffu, !ok || *abort_flag)) continue;
        const float b = p.bias && f < p.N ? p.bias[f] : 0.0f;
        bool all = true;
#pragma unroll
        for (int j = 0; j < CW; j++) all = all && finite(sum[j]);
        if (__any_sync(0xffffffffu, !all)) {
          int w_nan = -1;
          float kept[CW];                               // (in memory: a loop that is not unrolled is the least code beside the usual path)
#pragma unroll
          for (int j = 0; j < CW; j++) kept[j] = sum[j];
#pragma unroll 1
          for (int j = 0; j < CW; j++) {
            const float v = kept[j];
            const bool bad = f < p.N && mt + j < p.M && !finite(v);
            if (!__any_sync(0xffffffffu, bad)) continue;
            const Again again = plain_again(p.A + (size_t)(mt + j) * p.lda, p.W + (size_t)f * p.K, p.K, bad, v, w_nan);
            kept[j] = again.v;
            w_nan = again.w_nan;
          }
#pragma unroll
          for (int j = 0; j < CW; j++) sum[j] = kept[j];
        }
        if (p.act != SGLC_ACT_NONE) {
#pragma unroll
          for (int j = 0; j < CW; j++) sum[j] = apply_act(sum[j] + b, p.act);
        } else {
#pragma unroll
          for (int j = 0; j < CW; j++) sum[j] += b;
        }
        if (p.cache && n0 + FM > p.q_cols) {            // (some of the tile's columns; whole warps: a lane finds a token's place)
          float* col = f >= p.q_cols ? p.cache + column_at(p, f) : nullptr;
#pragma unroll
          for (int c = 0; c < CW; c += 32) {
            const long long mine = lane < CW - c ? slot_at(p, mt + c + lane) : -1;
#pragma unroll
            for (int j = 0; j < (CW < 32 ? CW : 32); j++) {
              if (c + j >= CW) break;
              const long long at = __shfl_sync(0xffffffffu, mine, j);
              if (col && f < p.N && at >= 0) col[at] = sum[c + j];
            }
          }
          if (col) continue;
        }
        if (f >= p.N) continue;
        float* o = (p.residual ? p.residual : p.out) + (size_t)mt * p.ldo + f;
        if (p.residual) {
#pragma unroll
          for (int c = 0; c < CW; c += 16) {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = mt + c + j < p.M ? o[(size_t)(c + j) * p.ldo] : 0.0f;
#pragma unroll
            for (int j = 0; j < 16; j++) sum[c + j] = v[j] + sum[c + j];
          }
        }
#pragma unroll
        for (int j = 0; j < CW; j++)
          if (mt + j < p.M) o[(size_t)j * p.ldo] = sum[j];
      }
    }
  }
  if constexpr (CLUSTER) {
    // a thread finishes four tokens of a feature at a time, neighbouring threads neighbouring features; what the first
    // round reads besides the sums is on its way while the blocks wait for one another
    constexpr int FIN = DW * 32;
    const bool fin = warp >= WW && warp < WW + DW;
    const int rows_per = (FM + p.ranks - 1) / p.ranks, t = fin ? tid - WW * 32 : FM * NT;      // (FM * NT: beyond all items)
    const int n0 = blockIdx.x * FM, m0 = blockIdx.y * NT;
    const int row0 = rank * rows_per, rows = min(rows_per, FM - row0), items = fin ? max(rows, 0) * (NT / 4) : 0;
    float bias = 0.0f, res[4] = {};
    auto fetch = [&](int x) {
      const int f = n0 + row0 + x % rows, m = m0 + x / rows * 4;
      if (f >= p.N) return;
      bias = p.bias ? p.bias[f] : 0.0f;
#pragma unroll
      for (int j = 0; j < 4; j++) res[j] = p.residual && m + j < p.M ? p.residual[(size_t)(m + j) * p.ldo + f] : 0.0f;
    };
    if (t < items) fetch(t);
    __syncwarp();
    if (!fin) cluster_wait();                           // (the adding warps have waited for the peers' start)
    cluster_arrive();
    if (warp == 0) {
      const bool all = mbar_wait(&taken, 0, abort_flag);
      if (__all_sync(0xffffffffu, all && !*abort_flag)) {
        held = false;
        tc_fence_after_sync();
        tmem_dealloc(tmem, COLS);
      }
    }
    cluster_wait();
    if (!*abort_flag)
      for (int x = t; x < items; x += FIN) {
        const int lr = x % rows, col = x / rows * 4, f = n0 + row0 + lr;
        if (x != t) fetch(x);
        if (f >= p.N) continue;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 6
        for (int g = 0; g < p.chunks; g++) {
          const float4 v = *reinterpret_cast<const float4*>(red + ((size_t)g * rows_per + lr) * NTP + col);
          if (g == 0) s = v;
          else {
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
          }
        }
        float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int m = m0 + col + j;
          if (m >= p.M) break;
          if (!finite(v[j])) v[j] = plain_until_nan(p.A + (size_t)m * p.lda, p.W + (size_t)f * p.K, p.K);
          const float y = apply_act(v[j] + bias, p.act);
          if (p.cache && f >= p.q_cols) {
            const long long at = slot_at(p, m);
            if (at >= 0) p.cache[at + column_at(p, f)] = y;
          } else if (p.residual) p.residual[(size_t)m * p.ldo + f] = res[j] + y;
          else p.out[(size_t)m * p.ldo + f] = y;
        }
      }
  }
  __syncthreads();
  if (tid == 0 && *abort_flag) atomicOr(p.err, SGLC_FLAG_WAIT);
  if (warp == 0 && held) tmem_dealloc(tmem, COLS);
}

constexpr size_t MOST_SMEM = 226 * 1024, TWO_SMEM = 112 * 1024;      // a block's at most; and where two share an SM
constexpr size_t smem_bytes(int NT, bool cluster, int chunks, int ranks) {
  const size_t rows_per = (FM + ranks - 1) / ranks;
  // No more blocks on an SM than its tensor memory serves (two of 256 columns, one of 512): one more would only wait for
  // columns, and keep its cluster's other blocks waiting.
  const size_t least = NT <= 32 ? 76 * 1024 : 114 * 1024;
  const size_t sums = cluster ? chunks * rows_per * (NT + 4) * 4 : 0;
  const size_t need = 1024 + 2 * 3 * NT * 128 + (NT >= 64 ? 2 * NT * FK * 4 : 0) + (cluster || NT == 128 || NT == 16 ? 2 : 3) * W_BYTES + sums;
  return need < least ? least : need;
}

template <int NT, int WW, int AW, int DW, bool CLUSTER>
struct Form {
  static constexpr int THREADS = (WW + AW + DW + (NT >= 64 ? 3 : 2)) * 32;
  static int prepare() {
    static const int rc = [] {
      auto* kernel = gemm_f32_kernel<NT, WW, AW, DW, CLUSTER>;
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST_SMEM);
      if (e == cudaSuccess && CLUSTER) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      return (int)e;
    }();
    return rc;
  }
  // How many clusters of so many blocks the device runs at once (by its groups of SMs: 18 of 6 blocks, say, where 148 SMs
  // would hold 24), with the most shared memory a form has at two blocks an SM, or at one.
  static int at_once(int ranks, size_t smem) {
    static std::atomic<int> known[MOST_RANKS + 1][2];
    const bool one = smem > TWO_SMEM;
    int n = known[ranks][one].load();
    if (n == 0) {
      cudaLaunchAttribute at;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = at.val.clusterDim.y = 1;
      at.val.clusterDim.z = ranks;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1, 1, ranks);
      cfg.blockDim = dim3(THREADS);
      cfg.dynamicSmemBytes = one ? MOST_SMEM : TWO_SMEM;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      if (prepare() != 0 || cudaOccupancyMaxActiveClusters(&n, gemm_f32_kernel<NT, WW, AW, DW, CLUSTER>, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = -1;
      }
      known[ranks][one].store(n);
    }
    return n;
  }
  static int launch(const F32Args& p, cudaStream_t stream) {
    const size_t smem = smem_bytes(NT, CLUSTER, p.chunks, p.ranks);
    if (smem > MOST_SMEM) return SGLC_ERR_UNSUPPORTED;
    if (const int rc = prepare()) return rc;
    CUtensorMap map_w, map_a = {};
    if (!make_map_f32_2d(&map_w, p.W, p.N, p.K, p.K, FM)) return SGLC_ERR_UNSUPPORTED;
    if (NT >= 64 && !make_map_f32_2d(&map_a, p.A, p.M, p.K, p.lda, NT)) return SGLC_ERR_UNSUPPORTED;
    constexpr int most = SMS * (NT == 16 ? 2 : 1);
    const dim3 grid = CLUSTER ? dim3(p.tiles_n, p.tiles / p.tiles_n, p.ranks) : dim3(p.tiles < most ? p.tiles : most);
    return sglc_launch(gemm_f32_kernel<NT, WW, AW, DW, CLUSTER>, grid, dim3(THREADS), smem, stream, CLUSTER ? p.ranks : 1, true, map_w,
                       map_a, p);
  }
};
template <bool CLUSTER> using Form16 = Form<16, 4, 2, 4, CLUSTER>;
template <bool CLUSTER> using Form32 = Form<32, 8, 2, 4, CLUSTER>;
template <bool CLUSTER> using Form64 = Form<64, 4, 4, 8, CLUSTER>;
using Form96 = Form<96, 4, 4, 8, false>;
using Form128 = Form<128, 4, 4, 8, false>;

void cut(F32Args& p, int nt, int ranks) {
  if (ranks > p.chunks) ranks = p.chunks;
  p.per_rank = (p.chunks + ranks - 1) / ranks;
  p.ranks = (p.chunks + p.per_rank - 1) / p.per_rank;
  p.tiles = p.tiles_n * ((p.M + nt - 1) / nt);
}
int run(const F32Args& p, int nt, cudaStream_t stream) {
  const bool cl = p.ranks > 1;
  switch (nt) {
    case 16: return cl ? Form16<true>::launch(p, stream) : Form16<false>::launch(p, stream);
    case 32: return cl ? Form32<true>::launch(p, stream) : Form32<false>::launch(p, stream);
    case 64: return cl ? Form64<true>::launch(p, stream) : Form64<false>::launch(p, stream);
    case 96: return cl ? SGLC_ERR_UNSUPPORTED : Form96::launch(p, stream);
    default: return cl ? SGLC_ERR_UNSUPPORTED : Form128::launch(p, stream);
  }
}

int g_f32_nt = 0, g_f32_ranks = 0;          // tuning hook: 0 lets the launcher choose

// The form by time, in us as measured: a chunk's of each tile, and a launch's besides; with a tile's K shared by blocks
// also the sums' way to their owners.
int choose(F32Args& p) {
  if (g_f32_nt) {
    cut(p, g_f32_nt, g_f32_ranks > 0 ? g_f32_ranks : 1);
    return g_f32_nt;
  }
  static const struct { int nt; double chunk, alone, shared; } FORMS[] = {
      {16, 0.89, 1.5, 3.3}, {32, 1.10, 2.3, 4.4}, {64, 1.05, 3.2, 6.4}, {96, 1.19, 5.0, 0.0}, {128, 1.45, 5.7, 0.0}};
  static const int RANKS[] = {1, 2, 3, 4, 6, 8, 12, 16};
  double best = 1e30;
  int nt = 128, ranks = 1;
  for (const auto& f : FORMS) {
    if (f.nt <= 64 && (p.M + f.nt - 1) / f.nt > 65535) continue;
    for (const int r : RANKS) {
      if (r > 1 && (f.shared == 0.0 || r > p.chunks)) break;
      F32Args t = p;
      cut(t, f.nt, r);
      double us;
      if (t.ranks == 1) {
        us = (double)((t.tiles + SMS - 1) / SMS) * t.chunks * f.chunk + f.alone;
      } else {
        const size_t smem = smem_bytes(f.nt, true, t.chunks, t.ranks);
        if (smem > MOST_SMEM) continue;
        // (at the least: all clusters at once, or there is no gain over the blocks alone)
        us = t.per_rank * f.chunk + f.shared + 0.00125 * t.chunks * f.nt;
        if (us >= best) continue;
        const int n = f.nt == 16 ? Form16<true>::at_once(t.ranks, smem) : f.nt == 32 ? Form32<true>::at_once(t.ranks, smem)
                                                                                    : Form64<true>::at_once(t.ranks, smem);
        if (n <= 0 || t.tiles > n) continue;
      }
      if (us < best) {
        best = us;
        nt = f.nt;
        ranks = t.ranks;
      }
    }
  }
  cut(p, nt, ranks);
  return nt;
}
}  // namespace

SGLC_API void sglc_gemm_f32_set_form(int nt, int ranks) { g_f32_nt = nt; g_f32_ranks = ranks; }

static int start(F32Args& p, cudaStream_t stream) {
  if (p.K % 4 != 0 || p.lda % 4 != 0 || (((uintptr_t)p.A | (uintptr_t)p.W) & 15) != 0) return SGLC_ERR_UNSUPPORTED;
  if ((long long)p.tiles_n * ((p.M + 15) / 16) > 1 << 30) return SGLC_ERR_UNSUPPORTED;
  const int nt = choose(p);
  return run(p, nt, stream);
}

// Whether the 32-bit path takes this kernel for a product (else gemm_simt.cu).  Nothing here follows the number of rows, so
// that a token's results do not either.  From K = 640 on it is the faster one at most sizes, and a few rows over K 640 to
// 768 are what it loses at; below, a step of few rows would lose more than it is worth (us, the kernels of gemm_simt.cu and
// this one, at 8, 64 and 1,872 rows: 1,024 columns over K 512 3.8 / 4.9, 9.6 / 6.1, 62.5 / 17.3; 768 over 768 4.5 / 5.1, 12.7
// / 6.6, 69.3 / 19.3; 2,304 over 768 6.3 / 6.1, 16.2 / 11.5, 154 / 40; 768 over 3,072 12.6 / 8.0, 40.6 / 13.3, 249 / 61;
// 1,600 over 1,600 10.7 / 7.6, 25.2 / 13.1, 259 / 64; 50,257 over 768 41.8 / 35.0, 195 / 45).  Narrow products, behind a layer norm
// of 1.9: 12 columns over K 640 5.9 / 6.7, 6.6 / 6.9, 23.6 / 14.1; over 768 6.2 / 6.1, 7.2 / 6.5, 26.9 / 15.0; over 3,072 13.8 /
// 8.1, 19.1 / 8.5, 70.7 / 63.6; and 768 over 640 5.7 / 7.2, 12.5 / 8.2, 60 / 18.
SGLC_API int sglc_gemm_f32_supports(int N, int K, int lda) { return K % 4 == 0 && lda % 4 == 0 && K >= 640; }

// A: [M,K] with row stride lda (elements); W: [N,K] contiguous; bias: float[N] or null; all 32-bit.  If `residual` is
// given (float [M,N], row stride ldo) the result is added into it and `out` is not written.  Needs whole 16-byte pieces:
// K and lda multiples of 4, A and W aligned.
SGLC_API int sglc_gemm_f32(const float* A, const float* W, const float* bias, float* out, float* residual, int M, int N, int K,
                           int lda, int ldo, int act, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return SGLC_OK;
  if (K <= 0) return SGLC_ERR_ARGUMENT;
  F32Args p = {A, W, bias, out, residual, M, N, K, lda, ldo, act, (K + FK - 1) / FK, 1, 0, (N + FM - 1) / FM, 0, err,
               nullptr, nullptr, 0, 0, 0, 0, 0};
  return start(p, stream);
}

// The query/key/value projection of a layer that owns its cache (32-bit, float [n_pages][2][heads][page][dim]): the queries
// into the first q_cols columns of out, keys and values straight into the cache at slots[token], with the bits that
// sglc_gemm_f32 gives (a launch and a pass over the keys and values less).
SGLC_API int sglc_gemm_f32_kv(const float* A, const float* W, const float* bias, float* out, int M, int N, int K, int lda, int ldo,
                              float* cache, const int* slots, int q_cols, int heads, int dim, int page, int n_pages, int* err,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return SGLC_OK;
  if (K <= 0 || q_cols < 0 || heads <= 0 || dim <= 0 || page <= 0 || N != q_cols + 2 * heads * dim) return SGLC_ERR_ARGUMENT;
  F32Args p = {A, W, bias, out, nullptr, M, N, K, lda, ldo, SGLC_ACT_NONE, (K + FK - 1) / FK, 1, 0, (N + FM - 1) / FM, 0, err,
               cache, slots, q_cols, heads, dim, page, n_pages};
  return start(p, stream);
}
