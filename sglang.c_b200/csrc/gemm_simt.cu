// C[M,N] = A[M,K] · W[N,K]^T (+ bias[N]) with an optional activation, or added
// into a 32-bit residual stream in place.  Plain FFMA on the CUDA cores: the
// 32-bit path of the model (no tensor-core mode, no reduced-precision products),
// and the fallback of the bfloat16 path for shapes the tensor-core kernel refuses.
// Every output element is one accumulator that takes k = 0..K-1 in ascending
// order, so a row's result does not depend on M or on its place in the batch.
// The reference's counterpart: sgl_matmul (src/ops.c:160-197) on the CPU and
// cublasSgemm / k_gemm_nt (src/cuda_backend.cu:2843-2867, 333-349) on the GPU.
// Weights are stored [N,K] (the reference transposes Conv1D weights the same
// way at upload, src/cuda_backend.cu:5232-5241).
#include "common.cuh"

SGLC_DEFINE_ERROR_STRING()

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TA, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
                 TO* __restrict__ out, float* __restrict__ residual, int M, int N, int K,
                 int lda, int ldo, int act) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.0f;

  // each thread stages 4 consecutive k of one row of A and of W
  int lrow = threadIdx.x / 4, lk = (threadIdx.x % 4) * 4;
  for (int k0 = 0; k0 < K; k0 += BK) {
    {
      int m = m0 + lrow;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        int k = k0 + lk + j;
        As[lk + j][lrow] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.0f;
      }
      int n = n0 + lrow;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        int k = k0 + lk + j;
        Ws[lk + j][lrow] = (n < N && k < K) ? to_f32(W[(size_t)n * K + k]) : 0.0f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; k++) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; i++) a[i] = As[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; j++) w[j] = Ws[k][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; i++) {
    int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      int n = n0 + tx * TN + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      v = apply_act(v, act);
      if (residual) {
        size_t o = (size_t)m * ldo + n;
        residual[o] = residual[o] + v;
      } else {
        out[(size_t)m * ldo + n] = from_f32<TO>(v);
      }
    }
  }
}
__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = on ? 16 : 0;                         // 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float part(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Many rows (a prompt portion of the 32-bit path), blocks of 64 x 64.  A warp has the 64 rows of 16 features, a lane
// 8 x 4 outputs; rows of A and W lie in shared memory as they lie in memory (36 floats apart: eight rows' 16-byte
// reads fall on all 32 banks), brought by asynchronous copies four k-tiles ahead, and leave it four k ahead of
// their use.  A 16-byte read costs one pass for the eight rows all quarters of a warp share and four for the four
// features, so the rows are on the side that costs one.  One accumulator per output, k ascending: the same
// bits from every kernel of this file.
// 672 x 768 x 768: 63.6 -> 32.6 us, over K 3,072 245 -> 111 us, 1,872 x 768 over K 3,072 347 -> 254 us (35 TFLOP/s).  Bound
// by how many registers a multiply-add's operands can be read a cycle (ncu: 0.58 of the multiply-add pipe, issue
// slots 0.70, warps ready): the pair kernel below is what gets around that where there are rows enough.
constexpr int LK = 32, LPITCH = LK + 4;

constexpr int TILE_M = 64, TILE_N = 64, TILE_ST = 4;

__global__ void __launch_bounds__(128, 3)
gemm_simt_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                      float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int lda,
                      int ldo, int act) {
  constexpr int BMT = TILE_M, BNT = TILE_N, TN = 4, ST = TILE_ST, STAGE = (BMT + BNT) * LPITCH;
  constexpr int STEP = 16;                           // rows a pass of the block's 16-byte copies covers
  extern __shared__ __align__(16) float ring[];      // [ST][BMT rows of A, then BNT of W][LPITCH]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BMT, n0 = blockIdx.x * BNT;
  const int n_tiles = (K + LK - 1) / LK;
  const int crow = tid / 8, ck = (tid % 8) * 4;
  // (weight rows beyond the last are copies of it, their outputs are not stored; token rows beyond the last are zeros, for
  // every block would ask for the same lines again: 65 tokens of 12,288 columns over K 768 122.8 -> 68.8 us)
  auto ask_w = [&](int tile, int st) {
    float* to = ring + st * STAGE + BMT * LPITCH + crow * LPITCH + ck;
    const int k = tile * LK + ck;
    const bool on = k < K;                           // (K is a multiple of 4: a piece lies inside or outside)
    const float* from = W + (on ? k : 0);
#pragma unroll
    for (int r = 0; r < BNT / STEP; r++)
      cp_async16_zfill(to + r * STEP * LPITCH, from + (size_t)min(n0 + crow + r * STEP, N - 1) * K, on);
  };
  auto ask_a = [&](int tile, int st) {
    float* to = ring + st * STAGE + crow * LPITCH + ck;
    const int k = tile * LK + ck;
    const bool on = k < K;
    const float* from = A + (on ? k : 0);
#pragma unroll
    for (int r = 0; r < BMT / STEP; r++)
      cp_async16_zfill(to + r * STEP * LPITCH, from + (size_t)min(m0 + crow + r * STEP, M - 1) * lda, on && m0 + crow + r * STEP < M);
  };
  for (int t = 0; t < ST; t++) {
    if (t < n_tiles) { ask_a(t, t); ask_w(t, t); }
    cp_async_commit();
  }
  const int row = lane & 7, feat = warp * 4 * TN + (lane >> 3);     // + 8 i, + 4 j
  float acc[8][TN];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.0f;
  float4 a[2][8], w[2][TN];
  auto take = [&](int to, int st, int k) {           // four k of this lane's rows and features into registers
    const float* as = ring + st * STAGE + row * LPITCH + k;
    const float* ws = ring + st * STAGE + (BMT + feat) * LPITCH + k;
#pragma unroll
    for (int j = 0; j < TN; j++) w[to][j] = *reinterpret_cast<const float4*>(ws + 4 * j * LPITCH);
#pragma unroll
    for (int i = 0; i < 8; i++) a[to][i] = *reinterpret_cast<const float4*>(as + 8 * i * LPITCH);
  };
  cp_async_wait<ST - 1>();
  __syncthreads();
  take(0, 0, 0);
  int st = 0;
  for (int tile = 0; tile < n_tiles; tile++) {
#pragma unroll
    for (int g = 0; g < LK / 4; g++) {
      // the next group's values leave shared memory while this group's are multiplied
      if (g + 1 < LK / 4) {
        take((g + 1) & 1, st, (g + 1) * 4);
      } else {
        cp_async_wait<ST - 2>();
        __syncthreads();                             // tile + 1 has landed; this tile's stage is free
        if (tile + ST < n_tiles) { ask_a(tile + ST, st); ask_w(tile + ST, st); }
        cp_async_commit();
        if (++st == ST) st = 0;
        take(0, st, 0);                              // (behind the last tile: a stage that is not used)
      }
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) acc[i][j] = fmaf(part(a[g & 1][i], e), part(w[g & 1][j], e), acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int m = m0 + row + 8 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int n = n0 + feat + 4 * j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      v = apply_act(v, act);
      const size_t o = (size_t)m * ldo + n;
      if (residual) residual[o] = residual[o] + v;
      else out[o] = v;
    }
  }
}

// Few rows (a decode step of the 32-bit path): the weights are read once, and an output is a chain of K
// dependent multiply-adds (four clocks each), which is what bounds the narrow products.  A block is one
// warp with 4 MR rows of 8 NF features, a lane MR x NF outputs, with no barrier between warps, and few
// instructions beside the chain.  Tiles of 64 k come through a ring of ST stages by asynchronous
// 16-byte copies.  A 16-byte read costs one pass for the eight features all quarters of the warp share and
// four for the four rows (rows lie 68 floats apart: no bank conflicts).  k ascending, one accumulator: the
// same bits as the kernels above.
// 8 rows: 768 columns 7.4 -> 4.8 us, over K 3,072 23.6 -> 12.6 us (its chain alone 6.4), 50,257 columns 84 -> 44 us (154 MB:
// 24 us at the copy rate).
constexpr int SK = 64, PITCH = SK + 4;

template <int MR, int NF, int ST>
__global__ void __launch_bounds__(32)
gemm_simt_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                      float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int lda,
                      int ldo, int act) {
  constexpr int RA = 4 * MR, RW = 8 * NF, STAGE = (RA + RW) * PITCH;
  extern __shared__ __align__(16) float ring[];      // [ST][RA rows, then RW weight rows][PITCH]
  const int lane = threadIdx.x;
  const int m0 = blockIdx.y * RA, n0 = blockIdx.x * RW;
  const int n_tiles = (K + SK - 1) / SK;
  const int crow = lane >> 4, ck = (lane & 15) * 4;  // a pass of the warp's copies: two rows
  // Where this lane's pieces come from (one warp has to issue everything: what a tile costs beside its chain is
  // kept to the copies themselves).  Weight rows beyond the last are copies of it, their outputs are not stored;
  // token rows beyond the last are zeros (copies would have every block ask for the same lines again).
  const float* pw[RW / 2];
  const float* pa[RA / 2];
  bool on_a[RA / 2];
#pragma unroll
  for (int r = 0; r < RW / 2; r++) pw[r] = W + (size_t)min(n0 + crow + 2 * r, N - 1) * K + ck;
#pragma unroll
  for (int r = 0; r < RA / 2; r++) {
    const int m = m0 + crow + 2 * r;
    on_a[r] = m < M;
    pa[r] = A + (on_a[r] ? (size_t)m * lda : 0) + ck;
  }
  const unsigned to0 = (unsigned)__cvta_generic_to_shared(ring) + (crow * PITCH + ck) * 4;
  auto copy = [](unsigned to, const float* from, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(on ? 16 : 0));
  };
  auto ask_w = [&](int tile, int st) {
    const bool on = tile * SK + ck < K;              // (K is a multiple of 4: a piece lies inside or outside)
    const int at = on ? tile * SK : 0;
#pragma unroll
    for (int r = 0; r < RW / 2; r++) copy(to0 + (st * STAGE + (RA + 2 * r) * PITCH) * 4, pw[r] + (on ? at : -ck), on);
  };
  auto ask_a = [&](int tile, int st) {
    const bool on = tile * SK + ck < K;
    const int at = on ? tile * SK : 0;
#pragma unroll
    for (int r = 0; r < RA / 2; r++) copy(to0 + (st * STAGE + 2 * r * PITCH) * 4, pa[r] + (on ? at : -ck), on && on_a[r]);
  };
  for (int t = 0; t < ST - 1; t++) {
    if (t < n_tiles) { ask_w(t, t); ask_a(t, t); }
    cp_async_commit();
  }
  float acc[MR][NF];
#pragma unroll
  for (int i = 0; i < MR; i++)
#pragma unroll
    for (int j = 0; j < NF; j++) acc[i][j] = 0.0f;
  const int row = lane >> 3, feat = lane & 7;        // + 4 i, + 8 j
  int st = 0, st_in = ST - 1;
  for (int tile = 0; tile < n_tiles; tile++) {
    cp_async_wait<ST - 2>();
    __syncwarp();                                    // tile `tile` has landed; the stage of tile-1 is free
    if (tile + ST - 1 < n_tiles) { ask_w(tile + ST - 1, st_in); ask_a(tile + ST - 1, st_in); }
    cp_async_commit();
    const float* as = ring + st * STAGE + row * PITCH;
    const float* ws = ring + st * STAGE + (RA + feat) * PITCH;
    if (++st == ST) st = 0;
    if (++st_in == ST) st_in = 0;
#pragma unroll(NF * MR > 8 ? 4 : 16)
    for (int k = 0; k < SK; k += 4) {
      float4 a[MR], w[NF];
#pragma unroll
      for (int i = 0; i < MR; i++) a[i] = *reinterpret_cast<const float4*>(as + 4 * i * PITCH + k);
#pragma unroll
      for (int j = 0; j < NF; j++) w[j] = *reinterpret_cast<const float4*>(ws + 8 * j * PITCH + k);
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int i = 0; i < MR; i++)
#pragma unroll
          for (int j = 0; j < NF; j++) acc[i][j] = fmaf(part(a[i], e), part(w[j], e), acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < MR; i++) {
    const int m = m0 + row + 4 * i;
#pragma unroll
    for (int j = 0; j < NF; j++) {
      const int n = n0 + feat + 8 * j;
      if (m >= M || n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      v = apply_act(v, act);
      const size_t o = (size_t)m * ldo + n;
      if (residual) residual[o] = residual[o] + v;
      else out[o] = v;
    }
  }
}

// 9 to 16 rows of some thousand features: with few features a block and 128 threads to it enough weights are on their way
// without any of a lane's chains being longer.  A block takes 16 rows of 16 features; tiles of 32 k come through a ring of
// eight shared-memory stages by asynchronous 16-byte copies, seven tiles ahead of the arithmetic; a thread owns two
// rows of one feature, k ascending: the same bits again.  16 rows, this kernel and the best of one-warp blocks: 2,304 columns
// over K 768 8.3 and 9.0 us, 3,072 10.6 and 11.3, 4,096 over 1,024 13.9 and 15.8.
constexpr int FEW_M = 16, FEW_N = 16, FEW_K = 32, FEW_ST = 8, FEW_PITCH = FEW_K + 4;

__global__ void __launch_bounds__(128)
gemm_simt_few_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int lda,
                     int ldo, int act) {
  __shared__ __align__(16) float As[FEW_ST][FEW_M][FEW_PITCH];
  __shared__ __align__(16) float Ws[FEW_ST][FEW_N][FEW_PITCH];
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * FEW_M, n0 = blockIdx.x * FEW_N;
  const int lrow = tid / 8, lk = (tid % 8) * 4;      // this thread's 16-byte piece of a tile row
  const int n_tiles = (K + FEW_K - 1) / FEW_K;
  auto issue = [&](int tile) {
    if (tile < n_tiles) {
      const int st = tile % FEW_ST, k = tile * FEW_K + lk;
      const bool kin = k < K;                        // (K is a multiple of 4: a piece lies inside or outside)
      const int m = m0 + lrow;
      cp_async16_zfill(&As[st][lrow][lk], A + (size_t)(m < M ? m : 0) * lda + (kin ? k : 0), kin && m < M);
      const int n = n0 + lrow;
      cp_async16_zfill(&Ws[st][lrow][lk], W + (size_t)(n < N ? n : 0) * K + (kin ? k : 0), kin && n < N);
    }
    cp_async_commit();
  };
  for (int t = 0; t < FEW_ST - 1; t++) issue(t);
  float acc[2] = {0.0f, 0.0f};
  for (int tile = 0; tile < n_tiles; tile++) {
    cp_async_wait<FEW_ST - 2>();
    __syncthreads();                                 // tile `tile` has landed; the stage of tile-1 is free
    issue(tile + FEW_ST - 1);
    const int st = tile % FEW_ST;
#pragma unroll
    for (int k = 0; k < FEW_K; k += 4) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[st][2 * ty][k]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[st][2 * ty + 1][k]);
      const float4 w0 = *reinterpret_cast<const float4*>(&Ws[st][tx][k]);
      acc[0] = fmaf(a0.x, w0.x, acc[0]); acc[1] = fmaf(a1.x, w0.x, acc[1]);
      acc[0] = fmaf(a0.y, w0.y, acc[0]); acc[1] = fmaf(a1.y, w0.y, acc[1]);
      acc[0] = fmaf(a0.z, w0.z, acc[0]); acc[1] = fmaf(a1.z, w0.z, acc[1]);
      acc[0] = fmaf(a0.w, w0.w, acc[0]); acc[1] = fmaf(a1.w, w0.w, acc[1]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int m = m0 + 2 * ty + i;
    const int n = n0 + tx;
    if (m >= M || n >= N) continue;
    float v = acc[i];
    if (bias) v += bias[n];
    v = apply_act(v, act);
    const size_t o = (size_t)m * ldo + n;
    if (residual) residual[o] = residual[o] + v;
    else out[o] = v;
  }
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// A load that stays where it is written: ahead of the arithmetic that covers its way from memory.
__device__ __forceinline__ float4 load_early(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
constexpr int PK = 16;

// Many rows and features: blocks of 128 x 64 or 128 x 128, a thread 8 x 8 outputs (runs of 4, so that a warp's reads are
// broadcasts and contiguous), the tiles turned to k-major on their way through registers.  Two features of a row
// are one packed multiply-add, each half rounded as a single one, which reads its operands as pairs.  1,872 rows:
// 2,304 columns 170 -> 155 us (43 TFLOP/s of the 73.6 that packed multiply-adds alone reach here), 3,072 columns
// 264 -> 204 us.
template <int BMT, int BNT, int BLOCKS>
__global__ void __launch_bounds__(BMT / 8 * (BNT / 8), BLOCKS)
gemm_simt_pair_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                      float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int lda,
                      int ldo, int act) {
  constexpr int TX = BNT / 8, THREADS = BMT / 8 * TX, C4 = 2;              // C4: runs of 4 features a thread has
  constexpr int NA = BMT * PK / 4 / THREADS, NB = BNT * PK / 4 / THREADS;  // 16-byte pieces a thread stages
  constexpr int WX = TX < 8 ? TX : 8;                                      // a warp: WX x 32 / WX threads
  static_assert(NA * THREADS * 4 == BMT * PK && NB * THREADS * 4 == BNT * PK, "");
  __shared__ __align__(16) float As[2][PK][BMT + 4];
  __shared__ __align__(16) float Ws[2][PK][BNT + 4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = warp % (TX / WX) * WX + lane % WX, ty = warp / (TX / WX) * (32 / WX) + lane / WX;
  const int m0 = blockIdx.y * BMT, n0 = blockIdx.x * BNT;
  const int lrow = tid / 4, lk = (tid % 4) * 4;      // rows lrow, lrow + THREADS / 4, ...; four k from lk
  // (rows beyond the last are copies of it: their outputs are not stored)
  const float* pa[NA];
  const float* pw[NB];
#pragma unroll
  for (int r = 0; r < NA; r++) pa[r] = A + (size_t)min(m0 + lrow + THREADS / 4 * r, M - 1) * lda;
#pragma unroll
  for (int r = 0; r < NB; r++) pw[r] = W + (size_t)min(n0 + lrow + THREADS / 4 * r, N - 1) * K;
  float4 ra[NA], rw[NB];
  auto load_a = [&](int k) {
    const bool on = k < K;                           // (K is a multiple of 4: a piece lies inside or outside)
#pragma unroll
    for (int r = 0; r < NA; r++) ra[r] = on ? load_early(pa[r] + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  auto load_w = [&](int k) {
    const bool on = k < K;
#pragma unroll
    for (int r = 0; r < NB; r++) rw[r] = on ? load_early(pw[r] + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int r = 0; r < NA; r++) {
      const int c = lrow + THREADS / 4 * r;
      As[buf][lk + 0][c] = ra[r].x; As[buf][lk + 1][c] = ra[r].y;
      As[buf][lk + 2][c] = ra[r].z; As[buf][lk + 3][c] = ra[r].w;
    }
#pragma unroll
    for (int r = 0; r < NB; r++) {
      const int c = lrow + THREADS / 4 * r;
      Ws[buf][lk + 0][c] = rw[r].x; Ws[buf][lk + 1][c] = rw[r].y;
      Ws[buf][lk + 2][c] = rw[r].z; Ws[buf][lk + 3][c] = rw[r].w;
    }
  };
  unsigned long long acc[8][2 * C4];                 // [row][pair of features]
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 2 * C4; j++) acc[i][j] = 0ull;
  load_w(lk);
  load_a(lk);
  sstore(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < K; k0 += PK, buf ^= 1) {
    const bool more = k0 + PK < K;
    if (more) { load_a(k0 + PK + lk); load_w(k0 + PK + lk); }
    float4 a0[2], a1[2];
    ulonglong2 w4[2][C4];
    auto take = [&](int to, int k) {
      a0[to] = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
      a1[to] = *reinterpret_cast<const float4*>(&As[buf][k][BMT / 2 + ty * 4]);
#pragma unroll
      for (int r = 0; r < C4; r++) w4[to][r] = *reinterpret_cast<const ulonglong2*>(&Ws[buf][k][BNT / C4 * r + tx * 4]);
    };
    take(0, 0);
#pragma unroll
    for (int k = 0; k < PK; k++) {
      if (k + 1 < PK) take((k + 1) & 1, k + 1);
      const float4 x = a0[k & 1], y = a1[k & 1];
      const unsigned long long a[8] = {pack2(x.x, x.x), pack2(x.y, x.y), pack2(x.z, x.z), pack2(x.w, x.w),
                                       pack2(y.x, y.x), pack2(y.y, y.y), pack2(y.z, y.z), pack2(y.w, y.w)};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int r = 0; r < C4; r++) {
          fma2(acc[i][2 * r], a[i], w4[k & 1][r].x);
          fma2(acc[i][2 * r + 1], a[i], w4[k & 1][r].y);
        }
    }
    if (more) sstore(buf ^ 1);                       // (its readers passed the barrier of the tile before)
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int m = m0 + (i < 4 ? ty * 4 + i : BMT / 2 + ty * 4 + i - 4);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 2 * C4; j++) {
      const float2 both = *reinterpret_cast<const float2*>(&acc[i][j]);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int n = n0 + BNT / C4 * (j / 2) + tx * 4 + (j % 2) * 2 + e;
        if (n >= N) continue;
        float v = e ? both.y : both.x;
        if (bias) v += bias[n];
        v = apply_act(v, act);
        const size_t o = (size_t)m * ldo + n;
        if (residual) residual[o] = residual[o] + v;
        else out[o] = v;
      }
    }
  }
}

// Blocks of 128 x 64, a thread 8 x 4 outputs (two corners of 4 x 4, so that a warp's shared-memory reads are broadcasts and
// contiguous runs), single multiply-adds; the next k-tile is on its way from global memory into registers while this one
// is multiplied.  Where each SM has two of such blocks it is ahead of the packed kernel: 800 x 2,304 x 768 93.9 us, packed
// 99.3; 1,280 x 1,536 x 768 93.3 and 98.8; with three of the packed kernel's blocks or one of either the others win.
constexpr int BLK_M = 128, BLK_N = 64, BLK_K = 16;

__global__ void __launch_bounds__(256, 2)          // two blocks an SM: at most 128 registers a thread
gemm_simt_block_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                       float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int lda,
                       int ldo, int act) {
  __shared__ __align__(16) float As[2][BLK_K][BLK_M + 4];
  __shared__ __align__(16) float Ws[2][BLK_K][BLK_N + 4];
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BLK_M, n0 = blockIdx.x * BLK_N;
  const int lrow = tid / 4, lk = (tid % 4) * 4;      // rows lrow and lrow + 64, four k from lk
  float4 ra[2], rw;
  auto gload = [&](int k0) {
    const int k = k0 + lk;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int m = m0 + lrow + 64 * r;
      ra[r] = (m < M && k < K) ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k)
                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    const int n = n0 + lrow;
    rw = (n < N && k < K) ? *reinterpret_cast<const float4*>(W + (size_t)n * K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int c = lrow + 64 * r;
      As[buf][lk + 0][c] = ra[r].x; As[buf][lk + 1][c] = ra[r].y;
      As[buf][lk + 2][c] = ra[r].z; As[buf][lk + 3][c] = ra[r].w;
    }
    Ws[buf][lk + 0][lrow] = rw.x; Ws[buf][lk + 1][lrow] = rw.y;
    Ws[buf][lk + 2][lrow] = rw.z; Ws[buf][lk + 3][lrow] = rw.w;
  };
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
  gload(0);
  sstore(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < K; k0 += BLK_K, buf ^= 1) {
    const bool more = k0 + BLK_K < K;
    if (more) gload(k0 + BLK_K);
#pragma unroll
    for (int k = 0; k < BLK_K; k++) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][k][64 + ty * 4]);
      const float4 w4 = *reinterpret_cast<const float4*>(&Ws[buf][k][tx * 4]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    if (more) sstore(buf ^ 1);                       // (its readers passed the barrier of the tile before)
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      v = apply_act(v, act);
      const size_t o = (size_t)m * ldo + n;
      if (residual) residual[o] = residual[o] + v;
      else out[o] = v;
    }
  }
}

struct SimtArgs {
  const float *A, *W, *bias;
  float *out, *residual;
  int M, N, K, lda, ldo, act;
};

// None of these kernels starts early behind the kernel ahead (programmatic dependent launch): blocks that wait
// beside the running ones take up room unevenly, and a launch of about one block an SM then lasts twice as long (63
// against 33 us for 672 x 768 x 768; 24 tokens for eight requests 25.6 against 23.1 ms).
template <int MR, int NF, int ST>
int launch_rows(const SimtArgs& p, cudaStream_t stream) {
  constexpr int smem = ST * (4 * MR + 8 * NF) * PITCH * 4;
  auto* kernel = gemm_simt_rows_kernel<MR, NF, ST>;
  static bool configured = false;
  if (smem > 48 * 1024 && !configured) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return sglc_launch(kernel, dim3((p.N + 8 * NF - 1) / (8 * NF), (p.M + 4 * MR - 1) / (4 * MR)), dim3(32), smem, stream, 1,
                     false, p.A, p.W, p.bias, p.out, p.residual, p.M, p.N, p.K, p.lda, p.ldo, p.act);
}

int launch_tile(const SimtArgs& p, cudaStream_t stream) {
  constexpr int smem = TILE_ST * (TILE_M + TILE_N) * LPITCH * 4;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_simt_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return sglc_launch(gemm_simt_tile_kernel, dim3((p.N + TILE_N - 1) / TILE_N, (p.M + TILE_M - 1) / TILE_M), dim3(128), smem,
                     stream, 1, false, p.A, p.W, p.bias, p.out, p.residual, p.M, p.N, p.K, p.lda, p.ldo, p.act);
}

int launch_few(const SimtArgs& p, cudaStream_t stream) {
  return sglc_launch(gemm_simt_few_kernel, dim3((p.N + FEW_N - 1) / FEW_N, (p.M + FEW_M - 1) / FEW_M), dim3(128), 0, stream, 1,
                     false, p.A, p.W, p.bias, p.out, p.residual, p.M, p.N, p.K, p.lda, p.ldo, p.act);
}

int launch_block(const SimtArgs& p, cudaStream_t stream) {
  return sglc_launch(gemm_simt_block_kernel, dim3((p.N + BLK_N - 1) / BLK_N, (p.M + BLK_M - 1) / BLK_M), dim3(256), 0, stream, 1,
                     false, p.A, p.W, p.bias, p.out, p.residual, p.M, p.N, p.K, p.lda, p.ldo, p.act);
}

template <int BMT, int BNT, int BLOCKS>
int launch_pair(const SimtArgs& p, cudaStream_t stream) {
  return sglc_launch(gemm_simt_pair_kernel<BMT, BNT, BLOCKS>, dim3((p.N + BNT - 1) / BNT, (p.M + BMT - 1) / BMT),
                     dim3(BMT / 8 * (BNT / 8)), 0, stream, 1, false, p.A, p.W, p.bias, p.out, p.residual, p.M, p.N, p.K,
                     p.lda, p.ldo, p.act);
}

// Tuning hook: 0 (default) lets the launcher choose the kernel.
int g_simt_form = 0;
enum { FORM_ROWS = 1, FORM_ROWS_WIDE, FORM_TILE, FORM_PAIR, FORM_PAIR_WIDE, FORM_FEW, FORM_BLOCK };

int choose_form(int M, int N) {
  if (M <= 64) return FORM_ROWS;
  // Else by time, in us at K = 768 (every form's grows with K alike), measured at 200 to 2,048 rows: so many
  // full waves of resident blocks, and a rest that takes less the fewer blocks an SM has.
  auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  auto waves = [](long long blocks, int resident, const double* us) {       // us[i]: i + 1 blocks an SM
    const long long wave = 148LL * resident, rest = blocks % wave;
    return (double)(blocks / wave) * us[resident - 1] + (rest ? us[(rest + 147) / 148 - 1] : 0.0);
  };
  static const double tile_us[] = {33.0, 54.0, 72.0}, pair_us[] = {64.0, 99.0, 131.0}, wide_us[] = {98.0, 159.0}, block_us[] = {62.0, 94.0};
  const double rows = 6.6 * (double)tiles(16, 32) / 148.0;
  const struct { int form; double us; } t[] = {{FORM_ROWS_WIDE, rows < 17.0 ? 17.0 : rows},
                                               {FORM_TILE, waves(tiles(64, 64), 3, tile_us)},
                                               {FORM_PAIR, waves(tiles(128, 64), 3, pair_us)},
                                               {FORM_PAIR_WIDE, waves(tiles(128, 128), 2, wide_us)},
                                               {FORM_BLOCK, waves(tiles(128, 64), 2, block_us)}};
  int best = 0;
  for (int i = 1; i < 5; i++)
    if (t[i].us < t[best].us) best = i;
  return t[best].form;
}

int simt_f32(const SimtArgs& p, cudaStream_t stream) {
  switch (g_simt_form ? g_simt_form : choose_form(p.M, p.N)) {
    case FORM_ROWS_WIDE: return launch_rows<4, 4, 4>(p, stream);
    case FORM_TILE: return launch_tile(p, stream);
    case FORM_PAIR: return launch_pair<128, 64, 3>(p, stream);
    case FORM_PAIR_WIDE: return launch_pair<128, 128, 2>(p, stream);
    case FORM_FEW: return launch_few(p, stream);
    case FORM_BLOCK: return launch_block(p, stream);
  }
  // Few rows, by the narrowest: the chain of K multiply-adds bounds a product, so a lane has one output; wider
  // ones, where shared-memory reads do, more; the vocabulary's head, where enough weights have to be on their way,
  // most, with a short ring so that more warps fit.  (us at 8 rows, one / two / four features a lane: 768 columns
  // 4.8 (a row a lane) / 9.1 / 11.4, over K 3,072 12.6 / 29.9 / 37.9, 2,304 columns 7.5 / 9.5 / 11.9, 50,257
  // columns 67.9 / 52.7 / 43.8.)
  if (p.M <= 4) return p.N <= 8192 ? launch_rows<1, 1, 10>(p, stream) : launch_rows<1, 2, 4>(p, stream);
  if (p.M <= 8) {
    if (p.N > 8192) return launch_rows<2, 4, 3>(p, stream);
  } else if (p.M <= 16) {
    // (us at 16 rows, 8 rows of 8 features a block, of 16, of 32 and 16 rows of 32: 4,800 columns over K 1,600 30.6 / 23.9 /
    // 26.2 / 42.1, 6,400 over 1,600 41.0 / 27.3 / 26.4 / 31.5, 8,200 over 768 21.8 / 19.3 / 17.6 / 21.8, 12,288 - / 28.0 / 23.8 / 22.3.)
    if (p.N > 10240) return launch_rows<4, 4, 3>(p, stream);
    if (p.N > 4608) return launch_rows<2, 4, 3>(p, stream);
    if (p.N > 1792) return launch_few(p, stream);
  } else if (p.N > 8192) {
    return launch_rows<4, 4, 3>(p, stream);
  }
  if (p.M <= 16) {
    if (p.N <= 1024) return launch_rows<1, 1, 10>(p, stream);
    return p.N <= 2304 ? launch_rows<2, 1, 10>(p, stream) : launch_rows<2, 2, 8>(p, stream);
  }
  return p.N <= 1024 ? launch_rows<2, 1, 10>(p, stream) : launch_rows<2, 4, 5>(p, stream);
}
}  // namespace

// A: [M,K] with row stride lda (elements); W: [N,K] contiguous; bias: float[N] or null.
// If `residual` is given (float [M,N], row stride ldo) the result is added into it and
// `out` is not written; else `out` ([M,N], row stride ldo, out_dtype) takes it.
SGLC_API void sglc_gemm_simt_set_form(int form) { g_simt_form = form; }

SGLC_API int sglc_gemm_simt(const void* A, const void* W, const float* bias, void* out,
                            float* residual, int M, int N, int K, int lda, int ldo, int in_dtype,
                            int out_dtype, int act, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return SGLC_OK;
  if (K <= 0) return SGLC_ERR_ARGUMENT;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return SGLC_ERR_UNSUPPORTED;
  const bool f32 = in_dtype == SGLC_F32 && (out_dtype == SGLC_F32 || residual);
  const bool wide_loads = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  if (f32 && wide_loads) {
    return simt_f32(SimtArgs{(const float*)A, (const float*)W, bias, (float*)out, residual, M, N, K, lda, ldo, act}, stream);
  } else if (in_dtype == SGLC_F32 && (out_dtype == SGLC_F32 || residual)) {
    gemm_simt_kernel<float, float, float><<<grid, 256, 0, stream>>>(
        (const float*)A, (const float*)W, bias, (float*)out, residual, M, N, K, lda, ldo, act);
  } else if (in_dtype == SGLC_BF16 && (out_dtype == SGLC_F32 || residual)) {
    gemm_simt_kernel<__nv_bfloat16, __nv_bfloat16, float><<<grid, 256, 0, stream>>>(
        (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, bias, (float*)out, residual, M, N, K, lda,
        ldo, act);
  } else if (in_dtype == SGLC_BF16 && out_dtype == SGLC_BF16) {
    gemm_simt_kernel<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, stream>>>(
        (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, bias, (__nv_bfloat16*)out, residual, M, N,
        K, lda, ldo, act);
  } else {
    return SGLC_ERR_ARGUMENT;
  }
  return sglc_launch_status();
}
