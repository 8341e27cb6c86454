// The gated matrix-state recurrence with a skip (matrix_state.cu),
//   S <- g_t S + b_t k_t v_t^T,    o_t = S^T q_t + skip v_t,      g_t = exp(-rate b_t), rate = exp(A_log),
// over portions of many tokens, in chunks of SC_Q tokens that do not wait for one another (the state-space
// duality of Mamba-2).  With c_i = sum_{t <= i} log g_t counted from a chunk's start and S_in the state ahead
// of the chunk,
//   o_i = exp(c_i) S_in^T q_i + sum_{j <= i} exp(c_i - c_j) b_j (q_i . k_j) v_j + skip v_i
//   S_out = exp(c_last) S_in + sum_j exp(c_last - c_j) b_j k_j v_j^T
// in three launches: every chunk's own contribution to S_out and its products q_i . k_j (per group, shared by the
// group's heads); a pass over the chunks of each request that turns contributions into states ahead of
// each chunk; the read-outs.  All of it is 32-bit multiply-adds on tiles in shared memory; the sums c_i are kept as
// a pair of floats, so that their differences are as exact as a 32-bit number allows however far c_i has run.
// A token by token walk takes T dependent steps; this takes about as many multiply-adds and no chain.
//
// And the same recurrence for steps in which every request brings one token (state_step_kernel): a state is read
// and written once, four columns a thread, all of a thread's rows asked for before the first is worked on.
#include "common.cuh"

SGLC_DEFINE_ERROR_STRING()

constexpr int SC_Q = 64;          // tokens of a chunk
constexpr int SC_V = 64;          // value columns of a tile
constexpr int SC_N = 128;         // state rows of a tile of the contributions
constexpr int SC_PAD = 4;         // floats behind a row of a tile: 16-byte rows, the rows of a warp on different banks
constexpr int SC_LQ = SC_Q + SC_PAD;
constexpr int SC_MAX_DIM = 256;
constexpr int SC_THREADS = 256;

struct ScArgs {
  const float* q; long long q_stride;       // [T][..], group g at columns g*N
  const float* k; long long k_stride;
  const float* v; long long v_stride;       // head h at columns h*V
  const float* b; long long b_stride;       // [T][..], head h at column h: the input weights
  const float* A_log; const float* skip;    // [H]; skip may be null
  float* out; long long out_stride;         // [T][H*V]
  float* state;                             // [n_slots][H][N][V]
  float* S;                                 // [n_chunks][H][N][V]: contributions, then states ahead of the chunks
  float* qk;                                // [n_chunks][G][SC_Q][SC_Q], (i, j)
  float* total;                             // [n_chunks][H]: exp(c_last)
  const int* q_start; const int* state_slots;
  int R, H, G, N, V, n_slots, n_chunks;
  int vec;                                  // rows of q, k, v and out go four entries at a time
  int* err;
};

struct Chunk { int r, t0, len; };

// The step's chunks in order: request after request, each cut from its own first token.  Called by whole warps.
__device__ __forceinline__ Chunk find_chunk(const ScArgs& p, int c) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int r0 = 0; r0 < p.R; r0 += 32) {
    const int r = r0 + lane;
    int a = 0, n = 0;
    if (r < p.R) {
      a = p.q_start[r];
      n = p.q_start[r + 1] - a;
    }
    const int mine = (n + SC_Q - 1) / SC_Q;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    const int lo = before + incl - mine;
    const unsigned hit = __ballot_sync(0xffffffffu, c >= lo && c < lo + mine);
    if (hit) {
      const int src = __ffs(hit) - 1;
      const int ra = __shfl_sync(0xffffffffu, a, src), rn = __shfl_sync(0xffffffffu, n, src), rl = __shfl_sync(0xffffffffu, lo, src);
      const int off = (c - rl) * SC_Q;
      return {r0 + src, ra + off, min(SC_Q, rn - off)};
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return {-1, 0, 0};
}

// c_i of a chunk and the input weights, by one whole warp (two neighbouring tokens a lane); tokens behind the
// end: weight zero, no decay.
__device__ __forceinline__ void chunk_sums(const ScArgs& p, int h, const Chunk& ck, float* hi, float* lo, float* bs) {
  const int lane = threadIdx.x & 31;
  const float rate = expf(p.A_log[h]);
  float w[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int i = 2 * lane + e;
    w[e] = i < ck.len ? p.b[(size_t)(ck.t0 + i) * p.b_stride + h] : 0.0f;
    bs[i] = w[e];
  }
  const double a0 = -(double)(rate * w[0]), a1 = -(double)(rate * w[1]);
  double s = a0 + a1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += x;
  }
  const double c1 = s, c0 = s - a1;
  hi[2 * lane] = (float)c0; lo[2 * lane] = (float)(c0 - (double)(float)c0);
  hi[2 * lane + 1] = (float)c1; lo[2 * lane + 1] = (float)(c1 - (double)(float)c1);
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void copy16(float* dst, const float* src, bool on) {      // (off: zeros)
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_end_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// rows 0 .. n_rows - 1 of src, columns c0 .. c0 + width - 1 of rows that end at column n, into dst[row][ld]; rows
// from `len` on and columns from n on are zeros.  width is a multiple of 4.
__device__ __forceinline__ void stage(const float* src, long long stride, int n_rows, int len, int c0, int width, int n, bool vec,
                                      float* dst, int ld) {
  if (vec) {
    const int w4 = width / 4;
    for (int x = threadIdx.x; x < n_rows * w4; x += SC_THREADS) {
      const int i = x / w4, c = (x - i * w4) * 4;
      const bool on = i < len && c0 + c < n;
      copy16(dst + i * ld + c, on ? src + (size_t)i * stride + c0 + c : src, on);
    }
  } else {
#pragma unroll 4
    for (int x = threadIdx.x; x < n_rows * width; x += SC_THREADS) {
      const int i = x / width, c = x - i * width;
      dst[i * ld + c] = (i < len && c0 + c < n) ? src[(size_t)i * stride + c0 + c] : 0.0f;
    }
  }
}
// acc[i][j] += a.(row i, entry e) * b[e].(column j), four entries
__device__ __forceinline__ void fma64(float (&acc)[4][4], const float4 (&a)[4], const float4 (&b)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      acc[i][0] = fmaf(av[e], b[e].x, acc[i][0]); acc[i][1] = fmaf(av[e], b[e].y, acc[i][1]);
      acc[i][2] = fmaf(av[e], b[e].z, acc[i][2]); acc[i][3] = fmaf(av[e], b[e].w, acc[i][3]);
    }
  }
}
__device__ __forceinline__ void fma16(float (&acc)[4][4], const float4& a, const float4& b) {
  const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    acc[i][0] = fmaf(av[i], b.x, acc[i][0]); acc[i][1] = fmaf(av[i], b.y, acc[i][1]);
    acc[i][2] = fmaf(av[i], b.z, acc[i][2]); acc[i][3] = fmaf(av[i], b.w, acc[i][3]);
  }
}
// acc += A rows ty*4 .. +3 (row stride lda) times B (row stride SC_V), over n entries (a multiple of 4)
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float* A, int lda, const float* B, int n, int ty, int tx) {
  const float* ar = A + ty * 4 * lda;
  const float* br = B + tx * 4;
#pragma unroll 2
  for (int e = 0; e < n; e += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = ld4(ar + i * lda + e);
#pragma unroll
    for (int i = 0; i < 4; i++) b[i] = ld4(br + (e + i) * SC_V);
    fma64(acc, a, b);
  }
}

// Grid (chunks, H * row tiles + G, column tiles).  Blocks y < H * row tiles: a tile [SC_N x SC_V] of a head's
// contribution; the others (z = 0): a group's products q_i . k_j.
__global__ void __launch_bounds__(SC_THREADS)
chunk_terms_kernel(const ScArgs p) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float hi[SC_Q], lo[SC_Q], bs[SC_Q];
  pdl_launch_dependents();
  const int c = blockIdx.x, tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int row_tiles = (p.N + SC_N - 1) / SC_N;
  const bool products = (int)blockIdx.y >= p.H * row_tiles;
  const int h = products ? 0 : blockIdx.y / row_tiles, n0 = products ? 0 : blockIdx.y % row_tiles * SC_N, v0 = blockIdx.z * SC_V;
  pdl_wait();
  const Chunk ck = find_chunk(p, c);
  if (ck.r < 0 || (products && blockIdx.z != 0)) return;
  if (products) {
    const int g = blockIdx.y - p.H * row_tiles, np = (p.N + 3) / 4 * 4, ld = np + SC_PAD;
    float* qs = sm;
    float* ks = sm + SC_Q * ld;
    stage(p.q + (size_t)ck.t0 * p.q_stride + (size_t)g * p.N, p.q_stride, SC_Q, ck.len, 0, np, p.N, p.vec, qs, ld);
    stage(p.k + (size_t)ck.t0 * p.k_stride + (size_t)g * p.N, p.k_stride, SC_Q, ck.len, 0, np, p.N, p.vec, ks, ld);
    copies_end_group();
    copies_wait<0>();
    __syncthreads();
    float acc[4][4] = {};
#pragma unroll 2
    for (int e = 0; e < np; e += 4) {                 // (columns j = tx + 16 i: the lanes' rows on different banks)
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = ld4(qs + (ty * 4 + i) * ld + e);
#pragma unroll
      for (int i = 0; i < 4; i++) b[i] = ld4(ks + (tx + 16 * i) * ld + e);
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    float* o = p.qk + ((size_t)c * p.G + g) * SC_Q * SC_Q;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) o[(ty * 4 + i) * SC_Q + tx + 16 * j] = acc[i][j];
    return;
  }
  // k_j v_j^T times exp(c_last - c_j) b_j (taken by v)
  float* ks = sm;
  float* vs = sm + SC_Q * SC_N;
  const int g = h / (p.H / p.G), rows = min(SC_N, (p.N - n0 + 3) / 4 * 4);
  stage(p.v + (size_t)ck.t0 * p.v_stride + (size_t)h * p.V, p.v_stride, SC_Q, ck.len, v0, SC_V, p.V, p.vec, vs, SC_V);
  stage(p.k + (size_t)ck.t0 * p.k_stride + (size_t)g * p.N, p.k_stride, SC_Q, ck.len, n0, rows, p.N, p.vec, ks, SC_N);
  copies_end_group();
  if (tid < 32) chunk_sums(p, h, ck, hi, lo, bs);
  copies_wait<0>();
  __syncthreads();
  if (tid == 0 && n0 == 0 && v0 == 0) p.total[(size_t)c * p.H + h] = expf(hi[ck.len - 1] + lo[ck.len - 1]);
  for (int x = tid; x < SC_Q * SC_V / 4; x += SC_THREADS) {
    const int j = x / (SC_V / 4);
    const float f = bs[j] * expf((hi[ck.len - 1] - hi[j]) + (lo[ck.len - 1] - lo[j]));
    float4 v = ld4(vs + x * 4);
    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
    *reinterpret_cast<float4*>(vs + x * 4) = v;
  }
  __syncthreads();
  const bool two = rows > SC_N / 2;           // rows in the tile's second half
  const bool a_on = ty * 4 < rows, b_on = two && SC_N / 2 + ty * 4 < rows;    // (no row of this thread: nothing to do)
  float a0[4][4] = {}, a1[4][4] = {};
  if (b_on) {
#pragma unroll 4
    for (int j = 0; j < ck.len; j++) {
      const float4 b = ld4(vs + j * SC_V + tx * 4);
      fma16(a0, ld4(ks + j * SC_N + ty * 4), b);
      fma16(a1, ld4(ks + j * SC_N + SC_N / 2 + ty * 4), b);
    }
  } else if (a_on) {
#pragma unroll 4
    for (int j = 0; j < ck.len; j++) fma16(a0, ld4(ks + j * SC_N + ty * 4), ld4(vs + j * SC_V + tx * 4));
  }
  float* o = p.S + ((size_t)c * p.H + h) * p.N * p.V;
  auto write = [&](const float (&a)[4][4], int first) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int n = first + i, v = v0 + tx * 4;
      if (n >= p.N) continue;
      if (p.vec) {
        if (v < p.V) *reinterpret_cast<float4*>(o + (size_t)n * p.V + v) = make_float4(a[i][0], a[i][1], a[i][2], a[i][3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (v + e < p.V) o[(size_t)n * p.V + v + e] = a[i][e];
      }
    }
  };
  if (a_on) write(a0, n0 + ty * 4);
  if (b_on) write(a1, n0 + SC_N / 2 + ty * 4);
}

// Grid (requests, H, pieces of the state): contributions -> states ahead of the chunks, the last state kept.
constexpr int SC_AHEAD = 8;      // chunks whose contributions are asked for together
template <typename TV>
__global__ void __launch_bounds__(SC_THREADS)
chunk_pass_kernel(const ScArgs p) {
  __shared__ int first_s;
  pdl_launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31;
  pdl_wait();
  if (threadIdx.x < 32) {
    int n = 0;
    for (int x = lane; x < r; x += 32) n += (p.q_start[x + 1] - p.q_start[x] + SC_Q - 1) / SC_Q;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) first_s = n;
  }
  __syncthreads();
  const int first = first_s, count = (p.q_start[r + 1] - p.q_start[r] + SC_Q - 1) / SC_Q;
  const int slot = p.state_slots[r];
  if (count <= 0 || !sglc_index_ok(slot, p.n_slots, p.err)) return;
  constexpr int W = sizeof(TV) / 4;
  const long long size = (long long)p.N * p.V / W, i = (long long)blockIdx.z * SC_THREADS + threadIdx.x;
  if (i >= size) return;
  TV* st = reinterpret_cast<TV*>(p.state) + ((size_t)slot * p.H + h) * size + i;
  TV* ch = reinterpret_cast<TV*>(p.S) + ((size_t)first * p.H + h) * size + i;
  const float* d = p.total + (size_t)first * p.H + h;
  const size_t step = (size_t)p.H * size;
  TV s = *st;
  for (int c0 = 0; c0 < count; c0 += SC_AHEAD) {
    TV own[SC_AHEAD];
    float dec[SC_AHEAD];
#pragma unroll
    for (int e = 0; e < SC_AHEAD; e++)
      if (c0 + e < count) {
        own[e] = ch[(c0 + e) * step];
        dec[e] = d[(size_t)(c0 + e) * p.H];
      }
#pragma unroll
    for (int e = 0; e < SC_AHEAD; e++)
      if (c0 + e < count) {
        ch[(c0 + e) * step] = s;
        if constexpr (W == 4) {
          s.x = fmaf(dec[e], s.x, own[e].x); s.y = fmaf(dec[e], s.y, own[e].y);
          s.z = fmaf(dec[e], s.z, own[e].z); s.w = fmaf(dec[e], s.w, own[e].w);
        } else {
          s = fmaf(dec[e], s, own[e]);
        }
      }
  }
  *st = s;
}

// Grid (chunks, H, column tiles): a head's read-outs of a chunk.
__global__ void __launch_bounds__(SC_THREADS)
chunk_read_kernel(const ScArgs p) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float hi[SC_Q], lo[SC_Q], bs[SC_Q];
  pdl_launch_dependents();
  const int c = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * SC_V, tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  pdl_wait();
  const Chunk ck = find_chunk(p, c);
  if (ck.r < 0) return;
  const int g = h / (p.H / p.G), np = (p.N + 3) / 4 * 4, ld = np + SC_PAD;
  float* qs = sm;                               // [SC_Q][ld]
  float* ss = qs + SC_Q * ld;                   // [np][SC_V]
  float* ms = ss + np * SC_V;                   // [SC_Q i][SC_LQ j]
  float* vs = ms + SC_Q * SC_LQ;                // [SC_Q][SC_V]
  stage(p.q + (size_t)ck.t0 * p.q_stride + (size_t)g * p.N, p.q_stride, SC_Q, ck.len, 0, np, p.N, p.vec, qs, ld);
  stage(p.S + ((size_t)c * p.H + h) * p.N * p.V, p.V, np, p.N, v0, SC_V, p.V, p.vec, ss, SC_V);
  copies_end_group();
  stage(p.qk + ((size_t)c * p.G + g) * SC_Q * SC_Q, SC_Q, SC_Q, SC_Q, 0, SC_Q, SC_Q, true, ms, SC_LQ);
  stage(p.v + (size_t)ck.t0 * p.v_stride + (size_t)h * p.V, p.v_stride, SC_Q, ck.len, v0, SC_V, p.V, p.vec, vs, SC_V);
  copies_end_group();
  if (tid < 32) chunk_sums(p, h, ck, hi, lo, bs);
  copies_wait<1>();
  __syncthreads();
  float acc[4][4] = {};
  tile_product(acc, qs, ld, ss, np, ty, tx);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float f = expf(hi[ty * 4 + i] + lo[ty * 4 + i]);
#pragma unroll
    for (int e = 0; e < 4; e++) acc[i][e] *= f;
  }
  copies_wait<0>();
  __syncthreads();
  const float skip = p.skip ? p.skip[h] : 0.0f;
  for (int x = tid; x < SC_Q * SC_Q; x += SC_THREADS) {
    const int i = x / SC_Q, j = x % SC_Q;
    float m = 0.0f;
    if (j <= i && i < ck.len) m = expf((hi[i] - hi[j]) + (lo[i] - lo[j])) * bs[j] * ms[i * SC_LQ + j];
    if (j == i) m += skip;
    ms[i * SC_LQ + j] = m;
  }
  __syncthreads();
  tile_product(acc, ms, SC_LQ, vs, (tid / 32 + 1) * 8, ty, tx);        // (no row of this warp sees a later token)
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int t = ty * 4 + i, v = v0 + tx * 4;
    if (t >= ck.len) continue;
    float* o = p.out + (size_t)(ck.t0 + t) * p.out_stride + (size_t)h * p.V + v;
    if (p.vec) {
      if (v < p.V) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (v + e < p.V) o[e] = acc[i][e];
    }
  }
}

SGLC_API int sglc_state_chunk() { return SC_Q; }

// ws: float, n_chunks * (H * N * V + G * SC_Q * SC_Q + H) entries, n_chunks being at least the chunks of the
// step (sum over requests of ceil(tokens / SC_Q)).
SGLC_API int sglc_state_chunks(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                               long long v_stride, const float* b, long long b_stride, const float* A_log,
                               const float* skip, float* out, long long out_stride, float* state, int n_slots,
                               const int* q_start, const int* state_slots, int R, int H, int G, int N, int V,
                               float* ws, int n_chunks, int* err, cudaStream_t stream) {
  if (R <= 0 || n_chunks <= 0) return SGLC_OK;
  if (H <= 0 || G <= 0 || H % G != 0 || N <= 0 || V <= 0 || !A_log || !ws) return SGLC_ERR_ARGUMENT;
  const int row_tiles = (N + SC_N - 1) / SC_N, col_tiles = (V + SC_V - 1) / SC_V;
  if (N > SC_MAX_DIM || (long long)H * row_tiles + G > 65535 || col_tiles > 65535) return SGLC_ERR_UNSUPPORTED;
  ScArgs p = {};
  p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = v; p.v_stride = v_stride; p.b = b; p.b_stride = b_stride;
  p.A_log = A_log; p.skip = skip; p.out = out; p.out_stride = out_stride; p.state = state; p.n_slots = n_slots;
  p.q_start = q_start; p.state_slots = state_slots; p.R = R; p.H = H; p.G = G; p.N = N; p.V = V; p.n_chunks = n_chunks; p.err = err;
  p.qk = ws;                                                     // (first: whole 16-byte pieces whatever the sizes)
  p.S = p.qk + (size_t)n_chunks * G * SC_Q * SC_Q;
  p.total = p.S + (size_t)n_chunks * H * N * V;
  auto al = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
  if (!al(ws)) return SGLC_ERR_ARGUMENT;
  p.vec = N % 4 == 0 && V % 4 == 0 && (q_stride | k_stride | v_stride | out_stride) % 4 == 0 && al(q) && al(k) && al(v) && al(out);
  const int np = (N + 3) / 4 * 4;
  size_t smem1 = (size_t)SC_Q * (SC_N + SC_V) * 4;
  if ((size_t)2 * SC_Q * (np + SC_PAD) * 4 > smem1) smem1 = (size_t)2 * SC_Q * (np + SC_PAD) * 4;
  const size_t smem3 = ((size_t)SC_Q * (np + SC_PAD) + (size_t)np * SC_V + SC_Q * (SC_LQ + SC_V)) * 4;
  cudaFuncSetAttribute(chunk_terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
  cudaFuncSetAttribute(chunk_read_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3);
  int rc = sglc_launch(chunk_terms_kernel, dim3(n_chunks, H * row_tiles + G, col_tiles), dim3(SC_THREADS), smem1, stream, 1, true, p);
  if (rc != SGLC_OK) return rc;
  const bool four = ((long long)N * V) % 4 == 0 && al(state);
  const long long pieces = ((long long)N * V / (four ? 4 : 1) + SC_THREADS - 1) / SC_THREADS;
  rc = four ? sglc_launch(chunk_pass_kernel<float4>, dim3(R, H, (unsigned)pieces), dim3(SC_THREADS), 0, stream, 1, true, p)
            : sglc_launch(chunk_pass_kernel<float>, dim3(R, H, (unsigned)pieces), dim3(SC_THREADS), 0, stream, 1, true, p);
  if (rc != SGLC_OK) return rc;
  return sglc_launch(chunk_read_kernel, dim3(n_chunks, H, col_tiles), dim3(SC_THREADS), smem3, stream, 1, true, p);
}

// ---- the gated delta rule, and the recurrence of fixed decay, in chunks -------------------------------------------
// With r_ij = g_(j+1) .. g_i (products taken token by token: a decay of zero stays one), c_i = g_1 .. g_i, S_in the
// state ahead of a chunk and C its last token:
//   delta rule   u_i = b_i (v_i - (g_i S_(i-1))^T k_i), that is  (I + L) U = diag(b) V - diag(b c) K S_in,
//                L_ij = b_i r_ij (k_i . k_j) for j < i;  so  U = U0 - W S_in  with  (I + L) [W | U0] = diag(b) [diag(c) K | V]
//   decay form   u_i = v_i
//   o_i   = c_i S_in^T q_i + sum_{j <= i} r_ij (q_i . k_j) u_j
//   S_out = c_C S_in + sum_j r_Cj k_j u_j^T = A S_in + B,  A = c_C I - sum_j r_Cj k_j w_j^T,  B = sum_j r_Cj k_j u0_j^T
// in three launches: a chunk's products, its triangular system (forward substitution, a column a thread, in
// registers), A and B; a pass over the chunks of each request, S <- A S + B, eight columns a block; the read-outs.
// All 32-bit multiply-adds, in the order of the tokens where one depends on another.  The walk token by token
// (matrix_state.cu) is a chain of T dependent steps of 215 ns with most of the GPU idle; this does about twice
// the multiply-adds with every SM at work.  2 x 1,024 tokens: delta rule, 12 heads of 64, 232 -> 80 us (38, 24 and 21:
// the first bound by shared memory reads and the chain of the triangular system, the second a chain of 16 chunks, 1.4
// us each); fixed decay with silu of its inputs, 3 heads, 174 -> 35 (20, 5 and 10).  Key sizes up to 64 (three blocks'
// tiles then fit into an SM's shared memory); value columns in tiles of 64.
constexpr int DC_LD = 64 + SC_PAD, DC_TILE = 64 * DC_LD;
constexpr int DC_PASS_COLS = 8, DC_PASS_RING = 4;
constexpr int DC_TERM_THREADS = 128;      // (three blocks an SM: 34 chunks of 12 heads then take one round)

struct DcArgs {
  const float* q; long long q_stride;       // [T][..], group g at columns g*D
  const float* k; long long k_stride;
  const float* v; long long v_stride;       // head h at columns h*V
  const float* gates; long long gates_stride;   // delta rule: [T][2H]: b, then the decays
  const float* head_decay;                  // decay form: [H]
  float* out; long long out_stride;         // [T][H*V]
  float* state;                             // [n_slots][H][D][V]
  float* qk;                                // [n_chunks][H][64][64]: r_ij (q_i . k_j), zero above the diagonal
  float* W;                                 // [n_chunks][H][64][64]
  float* A;                                 // [n_chunks][H][64][64]
  float* U;                                 // [n_chunks][H][tiles][64][64]: U0
  float* S;                                 // [n_chunks][H][tiles][64][64]: B, then the states ahead of the chunks
  float* total;                             // [n_chunks][H]: c_C
  const int* q_start; const int* state_slots;
  int R, H, G, D, V, tiles, n_slots, n_chunks;
  int vec, silu_in;
  int* err;
};

__device__ __forceinline__ float dc_silu(float v) { return v / (1.0f + expf(-v)); }

// 64 rows of src, columns c0 .. c0 + 63 of rows that end at column n, into dst; zeros outside.
template <int NT>      // NT: the block's threads
__device__ __forceinline__ void dc_stage(const float* src, long long stride, int len, int c0, int n, bool vec, float* dst) {
  if (vec) {
    for (int x = threadIdx.x; x < 64 * 16; x += NT) {
      const int i = x >> 4, c = (x & 15) * 4;
      const bool on = i < len && c0 + c < n;
      copy16(dst + i * DC_LD + c, on ? src + (size_t)i * stride + c0 + c : src, on);
    }
  } else {
    for (int x = threadIdx.x; x < 64 * 64; x += NT) {
      const int i = x >> 6, c = x & 63;
      dst[i * DC_LD + c] = (i < len && c0 + c < n) ? src[(size_t)i * stride + c0 + c] : 0.0f;
    }
  }
}
__device__ __forceinline__ void dc_stage64(const float* src, float* dst) {        // a whole tile of the workspace
  for (int x = threadIdx.x; x < 64 * 16; x += blockDim.x) copy16(dst + (x >> 4) * DC_LD + (x & 15) * 4, src + x * 4, true);
}
// (rows and columns beyond a tile's are zeros and stay so: a division of zero is a slow one)
// FAST: whole tiles a few entries at a time; without it the least code, for the delta rule, which no layer asks for a silu:
// its kernels run straight through code that has to be fetched (the terms of 2 x 1,024 tokens in a layer's chain of
// launches 38.2 us, 44.8 with both loops unrolled).
template <int NT, bool FAST>
__device__ __forceinline__ void dc_silu_tile(float* t, int rows, int cols) {
  if (FAST && rows >= 64 && cols >= 64) {
#pragma unroll 4
    for (int x = threadIdx.x; x < 64 * 64; x += NT) t[(x >> 6) * DC_LD + (x & 63)] = dc_silu(t[(x >> 6) * DC_LD + (x & 63)]);
    return;
  }
#pragma unroll 1
  for (int x = threadIdx.x; x < 64 * 64; x += NT) {
    float* e = t + (x >> 6) * DC_LD + (x & 63);
    if ((x >> 6) < rows && (x & 63) < cols) *e = dc_silu(*e);
  }
}
// A sum of short sums rounds less than one long one, as the walk's partial sums do: 64 entries go eight at a time, in
// pairs; and what a sum is added to, it is added to once.  (Against 64 bits, six draws of gates, keys and
// values as a layer makes them, 256 to 2,048 tokens: 1.60e-7, the walk 1.62e-7; sums of sixteen that start from their
// addend 1.85e-7.)
// acc[half][i][j] += a row (32 half + ty*4 + i) . b row (tx + 16 j), by 128 threads
__device__ __forceinline__ void dc_rows_product(float (&acc)[2][4][4], const float* a, const float* b, int ty, int tx) {
#pragma unroll 1
  for (int e0 = 0; e0 < 64; e0 += 16) {
    float sum[2][2][4][4] = {};
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
      for (int e = e0 + 8 * n; e < e0 + 8 * n + 8; e += 4) {
        float4 y[4];
#pragma unroll
        for (int j = 0; j < 4; j++) y[j] = ld4(b + (tx + 16 * j) * DC_LD + e);
#pragma unroll
        for (int f = 0; f < 2; f++)
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float4 x = ld4(a + (32 * f + ty * 4 + i) * DC_LD + e);
#pragma unroll
            for (int j = 0; j < 4; j++) {
              float& s = sum[n][f][i][j];
              s = fmaf(x.x, y[j].x, s); s = fmaf(x.y, y[j].y, s); s = fmaf(x.z, y[j].z, s); s = fmaf(x.w, y[j].w, s);
            }
          }
      }
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[f][i][j] += sum[0][f][i][j] + sum[1][f][i][j];
  }
}
// acc[half][i][j] += sum over rows e of a(e, 32 half + ty*4 + i) b(e, tx*4 + j), by 128 threads
__device__ __forceinline__ void dc_columns_product(float (&acc)[2][4][4], const float* a, const float* b, int ty, int tx) {
#pragma unroll 1
  for (int e0 = 0; e0 < 64; e0 += 16) {
    float sum[2][4][4] = {};
#pragma unroll 8
    for (int e = e0; e < e0 + 16; e++) {
      const float4 y = ld4(b + e * DC_LD + tx * 4);
      fma16(sum[0], ld4(a + e * DC_LD + ty * 4), y);
      fma16(sum[1], ld4(a + e * DC_LD + 32 + ty * 4), y);
    }
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[f][i][j] += sum[f][i][j];
  }
}
// acc += a rows ty*4 .. +3 (n entries of each, a multiple of 8) times b's rows, columns tx*4 .. +3, by 256 threads
__device__ __forceinline__ void dc_product(float (&acc)[4][4], const float* a, const float* b, int n, int ty, int tx) {
#pragma unroll 1
  for (int e0 = 0; e0 < n; e0 += 8) {
    float sum[4][4] = {};
#pragma unroll
    for (int e = e0; e < e0 + 8; e += 4) {
      float4 x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; i++) x[i] = ld4(a + (ty * 4 + i) * DC_LD + e);
#pragma unroll
      for (int i = 0; i < 4; i++) y[i] = ld4(b + (e + i) * DC_LD + tx * 4);
      fma64(sum, x, y);
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] += sum[i][j];
  }
}
// The eight terms at the diagonal of a lower triangular a (e0: their first; a warp has the rows e0 .. e0 + 7), each row's
// up to its own: a zero times a later token's infinity or NaN is not zero, and would reach the tokens before it.
__device__ __forceinline__ void dc_product_diagonal(float (&acc)[4][4], const float* a, const float* b, int e0, int ty, int tx) {
  float sum[4][4] = {};
#pragma unroll
  for (int e = e0; e < e0 + 8; e++) {
    const float4 y = ld4(b + e * DC_LD + tx * 4);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (e > ty * 4 + i) continue;
      const float x = a[(ty * 4 + i) * DC_LD + e];
      sum[i][0] = fmaf(x, y.x, sum[i][0]); sum[i][1] = fmaf(x, y.y, sum[i][1]);
      sum[i][2] = fmaf(x, y.z, sum[i][2]); sum[i][3] = fmaf(x, y.w, sum[i][3]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] += sum[i][j];
}
__device__ __forceinline__ void dc_write64(float* o, const float (&a)[2][4][4], int ty, int tx) {
#pragma unroll
  for (int f = 0; f < 2; f++)
#pragma unroll
    for (int i = 0; i < 4; i++)
      *reinterpret_cast<float4*>(o + (32 * f + ty * 4 + i) * 64 + tx * 4) = make_float4(a[f][i][0], a[f][i][1], a[f][i][2], a[f][i][3]);
}

// Grid (chunks, H, column tiles).
template <bool DELTA>
__global__ void __launch_bounds__(DC_TERM_THREADS, 3)
delta_terms_kernel(const DcArgs p) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float bs[64], gs[64], cs[64], rl[64];      // b, g, c_i, r_Cj
  float* ks = sm;                               // K
  float* qs = sm + DC_TILE;                     // Q, then W
  float* vs = sm + 2 * DC_TILE;                 // V, then U0
  float* ls = sm + 3 * DC_TILE;                 // r, then L / b
  const int c = blockIdx.x, h = blockIdx.y, z = blockIdx.z, tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  pdl_wait();
  ScArgs f = {};
  f.q_start = p.q_start;
  f.R = p.R;
  const Chunk ck = find_chunk(f, c);
  if (ck.r < 0) return;
  const int g = h / (p.H / p.G);
  dc_stage<DC_TERM_THREADS>(p.k + (size_t)ck.t0 * p.k_stride + (size_t)g * p.D, p.k_stride, ck.len, 0, p.D, p.vec, ks);
  if (z == 0) dc_stage<DC_TERM_THREADS>(p.q + (size_t)ck.t0 * p.q_stride + (size_t)g * p.D, p.q_stride, ck.len, 0, p.D, p.vec, qs);
  dc_stage<DC_TERM_THREADS>(p.v + (size_t)ck.t0 * p.v_stride + (size_t)h * p.V, p.v_stride, ck.len, z * 64, p.V, p.vec, vs);
  copies_end_group();
  if (tid < 64) {                               // (behind the end: weight zero, no decay)
    const bool on = tid < ck.len;
    bs[tid] = !on ? 0.0f : DELTA ? p.gates[(size_t)(ck.t0 + tid) * p.gates_stride + h] : 1.0f;
    gs[tid] = !on ? 1.0f : DELTA ? p.gates[(size_t)(ck.t0 + tid) * p.gates_stride + p.H + h] : p.head_decay[h];
  }
  __syncthreads();
  if (tid < 64) {                               // r_ij of column j, downwards
    float r = 1.0f;
    for (int i = 0; i < 64; i++) {
      r = i <= tid ? 1.0f : r * gs[i];
      ls[i * DC_LD + tid] = i < tid ? 0.0f : r;
    }
    rl[tid] = r;
  } else if (tid == 64) {
    float r = 1.0f;
    for (int i = 0; i < 64; i++) { r *= gs[i]; cs[i] = r; }
    if (z == 0) p.total[(size_t)c * p.H + h] = r;
  }
  copies_wait<0>();
  __syncthreads();
  if (p.silu_in) {
    dc_silu_tile<DC_TERM_THREADS, !DELTA>(ks, ck.len, p.D);
    if (z == 0) dc_silu_tile<DC_TERM_THREADS, !DELTA>(qs, ck.len, p.D);
    dc_silu_tile<DC_TERM_THREADS, !DELTA>(vs, ck.len, p.V - z * 64);
    __syncthreads();
  }
  const size_t at = ((size_t)c * p.H + h) * 4096, atz = (((size_t)c * p.H + h) * p.tiles + z) * 4096;
  if (z == 0) {
    float acc[2][4][4] = {};
    dc_rows_product(acc, qs, ks, ty, tx);
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int row = 32 * f + ty * 4 + i, col = tx + 16 * j;
          p.qk[at + row * 64 + col] = col <= row ? acc[f][i][j] * ls[row * DC_LD + col] : 0.0f;
        }
  }
  if (DELTA) {
    float acc[2][4][4] = {};
    dc_rows_product(acc, ks, ks, ty, tx);
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {           // (each entry of r is read and replaced by one thread)
          const int row = 32 * f + ty * 4 + i;
          float* e = ls + row * DC_LD + tx + 16 * j;
          *e *= acc[f][i][j];
        }
    __syncthreads();                            // (and Q has been read)
    {
      // forward substitution: thread c < 64 the column c of W, the others a column of U0
      const bool w = tid < 64;
      const int col = tid & 63;
      if (!w || z == 0) {
        float x[64];
#pragma unroll
        for (int i = 0; i < 64; i++) {
          // (four sums side by side: a row's chain is a quarter as long)
          float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
          for (int j4 = 0; j4 < i; j4 += 4) {
            const float4 l = ld4(ls + i * DC_LD + j4);
            s1 = fmaf(-l.x, x[j4], s1);
            if (j4 + 1 < i) s2 = fmaf(-l.y, x[j4 + 1], s2);
            if (j4 + 2 < i) s3 = fmaf(-l.z, x[j4 + 2], s3);
            if (j4 + 3 < i) s0 = fmaf(-l.w, x[j4 + 3], s0);
          }
          const float s = (s0 + s1) + (s2 + s3);
          x[i] = bs[i] * (w ? fmaf(cs[i], ks[i * DC_LD + col], s) : vs[i * DC_LD + col] + s);
        }
        float* to = w ? qs : vs;
#pragma unroll
        for (int i = 0; i < 64; i++) to[i * DC_LD + col] = x[i];
      }
    }
  }
  __syncthreads();
  for (int x = tid; x < 64 * 16; x += DC_TERM_THREADS) {      // (all that is read of K from here on carries r_Cj)
    float4* e = reinterpret_cast<float4*>(ks + (x >> 4) * DC_LD + (x & 15) * 4);
    const float r = rl[x >> 4];
    *e = make_float4(e->x * r, e->y * r, e->z * r, e->w * r);
    if (DELTA) {
      if (z == 0) *reinterpret_cast<float4*>(p.W + at + x * 4) = ld4(qs + (x >> 4) * DC_LD + (x & 15) * 4);
      *reinterpret_cast<float4*>(p.U + atz + x * 4) = ld4(vs + (x >> 4) * DC_LD + (x & 15) * 4);
    }
  }
  __syncthreads();
  float b[2][4][4] = {};
  dc_columns_product(b, ks, vs, ty, tx);
  dc_write64(p.S + atz, b, ty, tx);
  if (DELTA && z == 0) {
    float a[2][4][4] = {};
    dc_columns_product(a, ks, qs, ty, tx);
#pragma unroll
    for (int f = 0; f < 2; f++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) a[f][i][j] = (32 * f + ty * 4 + i == tx * 4 + j ? cs[63] : 0.0f) - a[f][i][j];
    dc_write64(p.A + at, a, ty, tx);
  }
}

// Grid (requests, H, pieces of 8 columns): S <- A S + B from chunk to chunk.  A thread keeps two entries of the state; in
// the product it has two rows and an eighth of their terms (the eighths are added behind a barrier).  All that a chunk
// brings comes through a ring of asynchronous copies.  Bound by what shared memory hands to registers.
template <bool DELTA>
__global__ void __launch_bounds__(SC_THREADS)
delta_pass_kernel(const DcArgs p) {
  constexpr int C = DC_PASS_COLS, RING = DC_PASS_RING;
  extern __shared__ __align__(16) float sm[];        // delta rule: RING tiles of A
  constexpr int PARTS = 8;
  __shared__ __align__(16) float bring[RING][64 * C], ss[DELTA ? 64 * C : 4], part[DELTA ? PARTS : 1][DELTA ? 64 * C : 4];
  __shared__ float tring[RING];
  __shared__ int first_s;
  const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, d = tid / 4, c2 = tid % 4 * 2, v0 = blockIdx.z * C;
  const int slot = p.state_slots[r];
  if (tid < 32) {
    int n = 0;
    for (int x = tid; x < r; x += 32) n += (p.q_start[x + 1] - p.q_start[x] + SC_Q - 1) / SC_Q;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (tid == 0) first_s = n;
  }
  __syncthreads();
  const int first = first_s, count = (p.q_start[r + 1] - p.q_start[r] + SC_Q - 1) / SC_Q;
  if (count <= 0 || !sglc_index_ok(slot, p.n_slots, p.err)) return;
  float* st = p.state + (((size_t)slot * p.H + h) * p.D + d) * p.V + v0 + c2;
  const bool on0 = d < p.D && v0 + c2 < p.V, on1 = d < p.D && v0 + c2 + 1 < p.V;
  float s0 = on0 ? st[0] : 0.0f, s1 = on1 ? st[1] : 0.0f;
  float* tile = p.S + (((size_t)first * p.H + h) * p.tiles + v0 / 64) * 4096 + v0 % 64;
  const size_t step = (size_t)p.H * p.tiles * 4096;
  auto ask = [&](int c) {
    if (c < count) {
      if (DELTA) dc_stage64(p.A + ((size_t)(first + c) * p.H + h) * 4096, sm + c % RING * DC_TILE);
      if (tid < 128) copy16(bring[c % RING] + tid * 4, tile + c * step + (tid >> 1) * 64 + (tid & 1) * 4, true);
      else if (!DELTA && tid == 128) {
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(&tring[c % RING]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(p.total + (size_t)(first + c) * p.H + h) : "memory");
      }
    }
    copies_end_group();
  };
  for (int c = 0; c < RING - 1; c++) ask(c);
  for (int c = 0; c < count; c++) {
    ask(c + RING - 1);
    if (DELTA) *reinterpret_cast<float2*>(ss + d * C + c2) = make_float2(s0, s1);
    copies_wait<RING - 1>();
    __syncthreads();                                 // chunk c is there (its contribution has left its place) and S is
    *reinterpret_cast<float2*>(tile + c * step + d * 64 + c2) = make_float2(s0, s1);
    const float2 own = *reinterpret_cast<const float2*>(bring[c % RING] + d * C + c2);
    if (DELTA) {
      const int row = tid & 31, q = tid >> 5;          // (rows `row` and `row` + 32, an eighth of their terms)
      const float* a = sm + c % RING * DC_TILE + row * DC_LD + q * 8;
      float acc[2][C] = {};
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        const float4 a0 = ld4(a + e), a1 = ld4(a + 32 * DC_LD + e);
        const float av[2][4] = {{a0.x, a0.y, a0.z, a0.w}, {a1.x, a1.y, a1.z, a1.w}};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 x = ld4(ss + (q * 8 + e + i) * C), y = ld4(ss + (q * 8 + e + i) * C + 4);
#pragma unroll
          for (int w = 0; w < 2; w++) {
            acc[w][0] = fmaf(av[w][i], x.x, acc[w][0]); acc[w][1] = fmaf(av[w][i], x.y, acc[w][1]);
            acc[w][2] = fmaf(av[w][i], x.z, acc[w][2]); acc[w][3] = fmaf(av[w][i], x.w, acc[w][3]);
            acc[w][4] = fmaf(av[w][i], y.x, acc[w][4]); acc[w][5] = fmaf(av[w][i], y.y, acc[w][5]);
            acc[w][6] = fmaf(av[w][i], y.z, acc[w][6]); acc[w][7] = fmaf(av[w][i], y.w, acc[w][7]);
          }
        }
      }
#pragma unroll
      for (int w = 0; w < 2; w++) {
        float* to = &part[q][(row + 32 * w) * C];
        *reinterpret_cast<float4*>(to) = make_float4(acc[w][0], acc[w][1], acc[w][2], acc[w][3]);
        *reinterpret_cast<float4*>(to + 4) = make_float4(acc[w][4], acc[w][5], acc[w][6], acc[w][7]);
      }
      __syncthreads();
      float2 sum[PARTS];
#pragma unroll
      for (int x = 0; x < PARTS; x++) sum[x] = *reinterpret_cast<const float2*>(&part[x][d * C + c2]);
      s0 = own.x + (((sum[0].x + sum[1].x) + (sum[2].x + sum[3].x)) + ((sum[4].x + sum[5].x) + (sum[6].x + sum[7].x)));
      s1 = own.y + (((sum[0].y + sum[1].y) + (sum[2].y + sum[3].y)) + ((sum[4].y + sum[5].y) + (sum[6].y + sum[7].y)));
    } else {
      const float t = tring[c % RING];
      s0 = fmaf(t, s0, own.x);
      s1 = fmaf(t, s1, own.y);
      __syncthreads();                               // (the slot may be filled again)
    }
  }
  if (on0) st[0] = s0;
  if (on1) st[1] = s1;
}

// Grid (chunks, H, column tiles): the read-outs.
template <bool DELTA>
__global__ void __launch_bounds__(SC_THREADS, 3)
delta_read_kernel(const DcArgs p) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float gs[64], cs[64];
  float* ss = sm;                               // S_in
  float* qs = sm + DC_TILE;
  float* us = sm + 2 * DC_TILE;                 // delta rule: W, then U; decay form: V
  float* ms = sm + 3 * DC_TILE;
  const int c = blockIdx.x, h = blockIdx.y, z = blockIdx.z, tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  ScArgs f = {};
  f.q_start = p.q_start;
  f.R = p.R;
  const Chunk ck = find_chunk(f, c);
  if (ck.r < 0) return;
  const int g = h / (p.H / p.G);
  const size_t at = ((size_t)c * p.H + h) * 4096, atz = (((size_t)c * p.H + h) * p.tiles + z) * 4096;
  dc_stage64(p.S + atz, ss);
  dc_stage<SC_THREADS>(p.q + (size_t)ck.t0 * p.q_stride + (size_t)g * p.D, p.q_stride, ck.len, 0, p.D, p.vec, qs);
  if (DELTA) dc_stage64(p.W + at, us);
  else dc_stage<SC_THREADS>(p.v + (size_t)ck.t0 * p.v_stride + (size_t)h * p.V, p.v_stride, ck.len, z * 64, p.V, p.vec, us);
  copies_end_group();
  dc_stage64(p.qk + at, ms);
  copies_end_group();
  if (tid < 64) gs[tid] = tid >= ck.len ? 1.0f : DELTA ? p.gates[(size_t)(ck.t0 + tid) * p.gates_stride + p.H + h] : p.head_decay[h];
  float4 u0[4];
  if (DELTA) {
#pragma unroll
    for (int i = 0; i < 4; i++) u0[i] = ld4(p.U + atz + (ty * 4 + i) * 64 + tx * 4);
  }
  copies_wait<1>();
  __syncthreads();
  if (tid == 0) {
    float r = 1.0f;
    for (int i = 0; i < 64; i++) { r *= gs[i]; cs[i] = r; }
  }
  if (p.silu_in) {
    dc_silu_tile<SC_THREADS, !DELTA>(qs, ck.len, p.D);
    if (!DELTA) dc_silu_tile<SC_THREADS, !DELTA>(us, ck.len, p.V - z * 64);
    __syncthreads();
  }
  if (DELTA) {                                           // U0 - W S
    float w[4][4] = {};
    dc_product(w, us, ss, 64, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; i++) u0[i] = make_float4(u0[i].x - w[i][0], u0[i].y - w[i][1], u0[i].z - w[i][2], u0[i].w - w[i][3]);
  }
  float acc[4][4] = {};
  dc_product(acc, qs, ss, 64, ty, tx);
  copies_wait<0>();
  __syncthreads();                                       // (W has been read, c_i are there)
  if (DELTA) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      *reinterpret_cast<float4*>(us + (ty * 4 + i) * DC_LD + tx * 4) = u0[i];
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[i][e] *= cs[ty * 4 + i];
  __syncthreads();
  dc_product(acc, ms, us, tid / 32 * 8, ty, tx);         // (no row of this warp sees a later token)
  dc_product_diagonal(acc, ms, us, tid / 32 * 8, ty, tx);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int t = ty * 4 + i, v = z * 64 + tx * 4;
    if (t >= ck.len) continue;
    float* o = p.out + (size_t)(ck.t0 + t) * p.out_stride + (size_t)h * p.V + v;
    if (p.vec) {
      if (v < p.V) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (v + e < p.V) o[e] = acc[i][e];
    }
  }
}

// (no early start of the later two behind one another: blocks that wait take up the room of running ones unevenly)
template <bool DELTA>
static int launch_delta_chunks(const DcArgs& p, dim3 grid, dim3 pass, cudaStream_t stream) {
  constexpr int smem = 4 * DC_TILE * 4, pass_smem = DELTA ? DC_PASS_RING * DC_TILE * 4 : 0;
  static bool configured = false;
  if (!configured) {
    auto allow = [](auto* kernel, int bytes) {
      return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : cudaSuccess;
    };
    cudaError_t e = allow(delta_terms_kernel<DELTA>, smem);
    if (e == cudaSuccess) e = allow(delta_read_kernel<DELTA>, smem);
    if (e == cudaSuccess) e = allow(delta_pass_kernel<DELTA>, pass_smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  int rc = sglc_launch(delta_terms_kernel<DELTA>, grid, dim3(DC_TERM_THREADS), smem, stream, 1, true, p);
  if (rc == SGLC_OK) rc = sglc_launch(delta_pass_kernel<DELTA>, pass, dim3(SC_THREADS), pass_smem, stream, 1, false, p);
  if (rc == SGLC_OK) rc = sglc_launch(delta_read_kernel<DELTA>, grid, dim3(SC_THREADS), smem, stream, 1, false, p);
  return rc;
}

// gates: the delta rule's [T][2H] (b, then the decays), or null with head_decay [H]: the decay form.  silu_in:
// silu of q, k and v first.  ws: float, n_chunks * H * (1 + 4096 * (delta rule: 3 + 2 tiles; decay form: 1 + tiles))
// entries, tiles = ceil(V / 64), n_chunks being at least the chunks of the step.
SGLC_API int sglc_delta_chunks(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                               long long v_stride, const float* gates, long long gates_stride, const float* head_decay,
                               float* out, long long out_stride, float* state, int n_slots, const int* q_start,
                               const int* state_slots, int R, int H, int G, int D, int V, int silu_in, float* ws,
                               int n_chunks, int* err, cudaStream_t stream) {
  if (R <= 0 || n_chunks <= 0) return SGLC_OK;
  if (H <= 0 || G <= 0 || H % G != 0 || D <= 0 || V <= 0 || !ws || (!gates) == (!head_decay)) return SGLC_ERR_ARGUMENT;
  const int tiles = (V + 63) / 64, pieces = (V + DC_PASS_COLS - 1) / DC_PASS_COLS;
  if (D > 64 || H > 65535 || pieces > 65535) return SGLC_ERR_UNSUPPORTED;
  DcArgs p = {};
  p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = v; p.v_stride = v_stride;
  p.gates = gates; p.gates_stride = gates_stride; p.head_decay = head_decay; p.out = out; p.out_stride = out_stride;
  p.state = state; p.n_slots = n_slots; p.q_start = q_start; p.state_slots = state_slots;
  p.R = R; p.H = H; p.G = G; p.D = D; p.V = V; p.tiles = tiles; p.n_chunks = n_chunks; p.silu_in = silu_in; p.err = err;
  const size_t unit = (size_t)n_chunks * H * 4096;
  p.qk = ws;
  p.S = p.qk + unit;
  float* end = p.S + unit * tiles;
  if (gates) {
    p.W = end;
    p.A = p.W + unit;
    p.U = p.A + unit;
    end = p.U + unit * tiles;
  }
  p.total = end;
  auto al = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; };
  if (!al(ws)) return SGLC_ERR_ARGUMENT;
  p.vec = D % 4 == 0 && V % 4 == 0 && (q_stride | k_stride | v_stride | out_stride) % 4 == 0 && al(q) && al(k) && al(v) && al(out);
  const dim3 grid(n_chunks, H, tiles), pass(R, H, pieces);
  return gates ? launch_delta_chunks<true>(p, grid, pass, stream) : launch_delta_chunks<false>(p, grid, pass, stream);
}

// Every request brings one token (token r is request r's).  Grid (requests, H, column tiles of SS_COLS); a
// thread keeps W columns of every SS_ROWS-th row.
constexpr int SS_COLS = 64, SS_DEEP = 8;
template <int W>      // 4: rows 16 bytes at a time; 1: any sizes
__global__ void __launch_bounds__(SC_THREADS)
state_step_kernel(const ScArgs p, const float* __restrict__ decay, long long decay_stride) {
  constexpr int CT = SS_COLS / W, ROWS = SC_THREADS / CT;        // threads over the columns, rows side by side
  __shared__ float part[ROWS][SS_COLS];
  __shared__ float ks[SC_MAX_DIM], qs[SC_MAX_DIM];
  pdl_launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x;
  const int cx = tid % CT, rx = tid / CT, col = blockIdx.z * SS_COLS + cx * W;
  const bool on = col < p.V;
  const int slot = p.state_slots[r];                             // (nothing a kernel of the step writes)
  if (!sglc_index_ok(slot, p.n_slots, p.err)) return;
  float* st = p.state + ((size_t)slot * p.H + h) * p.N * p.V + col;
  pdl_wait();
  for (int n = tid; n < p.N; n += SC_THREADS) {
    ks[n] = p.k[(size_t)r * p.k_stride + (size_t)g * p.N + n];
    qs[n] = p.q[(size_t)r * p.q_stride + (size_t)g * p.N + n];
  }
  const float b = p.b[(size_t)r * p.b_stride + h], gd = decay[(size_t)r * decay_stride + h];
  float v[W], bv[W], acc[W];
#pragma unroll
  for (int e = 0; e < W; e++) {
    v[e] = on ? p.v[(size_t)r * p.v_stride + (size_t)h * p.V + col + e] : 0.0f;
    bv[e] = b * v[e];
    acc[e] = 0.0f;
  }
  __syncthreads();
  for (int n0 = rx; n0 < p.N; n0 += ROWS * SS_DEEP) {
    float S[SS_DEEP][W];
#pragma unroll
    for (int d = 0; d < SS_DEEP; d++) {
      const int n = n0 + d * ROWS;
      if (on && n < p.N) {
        if constexpr (W == 4) {
          const float4 s = ld4(st + (size_t)n * p.V);
          S[d][0] = s.x; S[d][1] = s.y; S[d][2] = s.z; S[d][3] = s.w;
        } else {
          S[d][0] = st[(size_t)n * p.V];
        }
      }
    }
#pragma unroll
    for (int d = 0; d < SS_DEEP; d++) {
      const int n = n0 + d * ROWS;
      if (on && n < p.N) {
        const float k = ks[n], q = qs[n];
#pragma unroll
        for (int e = 0; e < W; e++) {
          S[d][e] = fmaf(k, bv[e], gd * S[d][e]);
          acc[e] = fmaf(q, S[d][e], acc[e]);
        }
        if constexpr (W == 4) *reinterpret_cast<float4*>(st + (size_t)n * p.V) = make_float4(S[d][0], S[d][1], S[d][2], S[d][3]);
        else st[(size_t)n * p.V] = S[d][0];
      }
    }
  }
#pragma unroll
  for (int e = 0; e < W; e++) part[rx][cx * W + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.z * SS_COLS + tid;
  if (tid < SS_COLS && c < p.V) {
    float o = 0.0f;
#pragma unroll
    for (int x = 0; x < ROWS; x++) o += part[x][tid];
    if (p.skip) o = fmaf(p.skip[h], p.v[(size_t)r * p.v_stride + (size_t)h * p.V + c], o);
    p.out[(size_t)r * p.out_stride + (size_t)h * p.V + c] = o;
  }
}

// S <- decay S + b k v^T, o = S^T q + skip v for R requests of one token each; b and decay: float rows, head h in column h.
SGLC_API int sglc_state_step(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                             long long v_stride, const float* b, const float* decay, long long gates_stride,
                             const float* skip, float* out, long long out_stride, float* state, int n_slots,
                             const int* state_slots, int R, int H, int G, int N, int V, int* err, cudaStream_t stream) {
  if (R <= 0) return SGLC_OK;
  if (H <= 0 || G <= 0 || H % G != 0 || N <= 0 || V <= 0 || !b || !decay) return SGLC_ERR_ARGUMENT;
  const int tiles = (V + SS_COLS - 1) / SS_COLS;
  if (N > SC_MAX_DIM || H > 65535 || tiles > 65535) return SGLC_ERR_UNSUPPORTED;
  ScArgs p = {};
  p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = v; p.v_stride = v_stride; p.b = b; p.b_stride = gates_stride;
  p.skip = skip; p.out = out; p.out_stride = out_stride; p.state = state; p.n_slots = n_slots; p.state_slots = state_slots;
  p.R = R; p.H = H; p.G = G; p.N = N; p.V = V; p.err = err;
  const dim3 grid(R, H, tiles);
  if (V % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0)
    return sglc_launch(state_step_kernel<4>, grid, dim3(SC_THREADS), 0, stream, 1, true, p, decay, gates_stride);
  return sglc_launch(state_step_kernel<1>, grid, dim3(SC_THREADS), 0, stream, 1, true, p, decay, gates_stride);
}

// The delta rule and the fixed decay where every request brings one token: a block has 64 value columns of a
// (request, head), a thread four columns of every 16th row in registers; all that a block reads is asked for at once.
// The walk's arithmetic: S <- g S;  u = b (v - S^T k)  or  v;  S <- S + k u^T;  o = S^T q.  Bound by latency.
// Launch behind launch, heads of 64: 8 requests, delta rule, 12 heads 5.8 -> 2.6 us, decay, 3 heads 3.8 -> 2.3; 64 requests
// 13.9 -> 4.7 and 5.9 -> 3.3 (the walk of matrix_state.cu waits for a token's inputs and for its state in turn).
template <bool DELTA, int DR>      // DR: rows a thread keeps (key sizes up to 16 DR)
__global__ void __launch_bounds__(SC_THREADS)
delta_step_kernel(const DcArgs p) {
  __shared__ __align__(16) float us[64], part[8][64];
  __shared__ float ks[16 * DR], qs[16 * DR];
  pdl_launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x, lane = tid & 31;
  const int cx = tid % 16, rx = tid / 16, v0 = blockIdx.z * 64, col = v0 + cx * 4;
  const int slot = p.state_slots[r];                 // (nothing a kernel of the step writes)
  if (!sglc_index_ok(slot, p.n_slots, p.err)) return;
  float* st = p.state + ((size_t)slot * p.H + h) * p.D * p.V + col;
  pdl_wait();
  float4 S[DR];
#pragma unroll
  for (int i = 0; i < DR; i++) {
    const int n = rx + 16 * i;
    S[i] = (n < p.D && col < p.V) ? ld4(st + (size_t)n * p.V) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  float b = 1.0f, gd = 0.0f, v = 0.0f;
  if (DELTA) {
    b = p.gates[(size_t)r * p.gates_stride + h];
    gd = p.gates[(size_t)r * p.gates_stride + p.H + h];
  } else {
    gd = p.head_decay[h];
  }
  if (tid < 64 && v0 + tid < p.V) {
    v = p.v[(size_t)r * p.v_stride + (size_t)h * p.V + v0 + tid];
    if (p.silu_in) v = dc_silu(v);
  }
  if (!DELTA && tid < 64) us[tid] = v;
  for (int n = tid; n < 16 * DR; n += SC_THREADS) {
    float k = 0.0f, q = 0.0f;
    if (n < p.D) {
      k = p.k[(size_t)r * p.k_stride + (size_t)g * p.D + n];
      q = p.q[(size_t)r * p.q_stride + (size_t)g * p.D + n];
      if (p.silu_in) { k = dc_silu(k); q = dc_silu(q); }
    }
    ks[n] = k;
    qs[n] = q;
  }
  __syncthreads();
  // the sum of a column's products with a vector, over the rows: left to thread `column`
  auto columns = [&](const float* with) {
    float a[4] = {};
#pragma unroll
    for (int i = 0; i < DR; i++) {
      const float w = with[rx + 16 * i];
      a[0] = fmaf(S[i].x, w, a[0]); a[1] = fmaf(S[i].y, w, a[1]); a[2] = fmaf(S[i].z, w, a[2]); a[3] = fmaf(S[i].w, w, a[3]);
    }
#pragma unroll
    for (int e = 0; e < 4; e++) a[e] += __shfl_xor_sync(0xffffffffu, a[e], 16);
    if (lane < 16) *reinterpret_cast<float4*>(&part[tid >> 5][cx * 4]) = make_float4(a[0], a[1], a[2], a[3]);
    __syncthreads();
    if (tid >= 64) return 0.0f;
    const float (*w)[64] = part;
    return ((w[0][tid] + w[1][tid]) + (w[2][tid] + w[3][tid])) + ((w[4][tid] + w[5][tid]) + (w[6][tid] + w[7][tid]));
  };
#pragma unroll
  for (int i = 0; i < DR; i++) { S[i].x *= gd; S[i].y *= gd; S[i].z *= gd; S[i].w *= gd; }
  if (DELTA) {
    const float x = columns(ks);
    if (tid < 64) us[tid] = b * (v - x);
    __syncthreads();
  }
  const float4 u = ld4(us + cx * 4);
#pragma unroll
  for (int i = 0; i < DR; i++) {
    const int n = rx + 16 * i;
    if (n >= p.D) continue;
    const float k = ks[n];
    S[i].x = fmaf(k, u.x, S[i].x); S[i].y = fmaf(k, u.y, S[i].y); S[i].z = fmaf(k, u.z, S[i].z); S[i].w = fmaf(k, u.w, S[i].w);
    if (col < p.V) *reinterpret_cast<float4*>(st + (size_t)n * p.V) = S[i];
  }
  const float o = columns(qs);
  if (tid < 64 && v0 + tid < p.V) p.out[(size_t)r * p.out_stride + (size_t)h * p.V + v0 + tid] = o;
}

// Arguments as sglc_delta_chunks, for R requests of one token each (row r is request r's); value sizes that are
// multiples of 4.
SGLC_API int sglc_delta_step(const float* q, long long q_stride, const float* k, long long k_stride, const float* v,
                             long long v_stride, const float* gates, long long gates_stride, const float* head_decay,
                             float* out, long long out_stride, float* state, int n_slots, const int* state_slots, int R,
                             int H, int G, int D, int V, int silu_in, int* err, cudaStream_t stream) {
  if (R <= 0) return SGLC_OK;
  if (H <= 0 || G <= 0 || H % G != 0 || D <= 0 || V <= 0 || (!gates) == (!head_decay)) return SGLC_ERR_ARGUMENT;
  const int tiles = (V + 63) / 64;
  if (D > SC_MAX_DIM || V % 4 != 0 || H > 65535 || tiles > 65535 || (reinterpret_cast<uintptr_t>(state) & 15)) return SGLC_ERR_UNSUPPORTED;
  DcArgs p = {};
  p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = v; p.v_stride = v_stride;
  p.gates = gates; p.gates_stride = gates_stride; p.head_decay = head_decay; p.out = out; p.out_stride = out_stride;
  p.state = state; p.n_slots = n_slots; p.state_slots = state_slots;
  p.R = R; p.H = H; p.G = G; p.D = D; p.V = V; p.silu_in = silu_in; p.err = err;
  const dim3 grid(R, H, tiles), block(SC_THREADS);
  if (gates) {
    if (D <= 64) return sglc_launch(delta_step_kernel<true, 4>, grid, block, 0, stream, 1, true, p);
    if (D <= 128) return sglc_launch(delta_step_kernel<true, 8>, grid, block, 0, stream, 1, true, p);
    return sglc_launch(delta_step_kernel<true, 16>, grid, block, 0, stream, 1, true, p);
  }
  if (D <= 64) return sglc_launch(delta_step_kernel<false, 4>, grid, block, 0, stream, 1, true, p);
  if (D <= 128) return sglc_launch(delta_step_kernel<false, 8>, grid, block, 0, stream, 1, true, p);
  return sglc_launch(delta_step_kernel<false, 16>, grid, block, 0, stream, 1, true, p);
}
