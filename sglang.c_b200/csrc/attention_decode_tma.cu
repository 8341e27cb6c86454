// Attention for single decoded tokens, keys and values staged through shared memory by TMA.
// The same arithmetic and the same merge as attention_decode.cu (one block per (token, head,
// key range); ranges merged in range order inside a thread-block cluster), but the range's
// pages are brought in as one 5-D TMA box per page and K/V instead of per-thread loads held in
// registers.  A block then needs few registers and about 40 KB of shared memory, so five or
// more blocks fit on an SM: at large batches, where the register version is bound by how many
// blocks an SM holds, this one keeps several times more bytes in flight.
// Head sizes 64 and 128, bfloat16, up to 8 key ranges (other cases: attention_decode.cu).
// The reference's counterparts are named in attention_decode.cu.
#include <string.h>

#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "tc_common.cuh"

SGLC_DEFINE_ERROR_STRING()

namespace {
using namespace tc;
constexpr int THREADS = 128;
constexpr int WARPS = THREADS / 32;

__device__ __forceinline__ void bf16x8_to_f32(const uint4& u, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void st_peer_f32(uint32_t raddr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(raddr), "f"(v) : "memory");
}

struct Args {
  const __nv_bfloat16* q;
  int q_stride;
  __nv_bfloat16* cache;
  const int* block_table;
  int bt_stride;
  const int* token_req;      // null: token t is the step's t-th request
  const int* positions;
  const int* token_list;     // null: the launch serves tokens 0..T-1
  __nv_bfloat16* out;
  int o_stride;
  int H, Hkv, page_size;
  float scale;
  int window;
  int n_splits, chunk_cap, rows_cap, nb_max;
  const __nv_bfloat16* k_new;   // optional: the step's own keys / values and their cache slots
  const __nv_bfloat16* v_new;
  int new_stride;
  const int* slots;
  int* err;
};

template <int D>
__global__ void __launch_bounds__(THREADS)
attention_decode_tma_kernel(const __grid_constant__ CUtensorMap map_kv, const Args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  // [K rows_cap x D][V rows_cap x D][part WARPS*D floats][pages nb_max][records 8*(D+2)]
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem);
  __nv_bfloat16* sV = sK + (size_t)a.rows_cap * D;
  float* part = reinterpret_cast<float*>(sV + (size_t)a.rows_cap * D);
  int* spage = reinterpret_cast<int*>(part + WARPS * D);
  float* recs = reinterpret_cast<float*>(spage + a.nb_max);
  __shared__ float red[2 * WARPS];                    // the warps' maxima, then their sums
  __shared__ int s_meta[2];
  __shared__ int s_abort;
  __shared__ __align__(8) uint64_t load_bar;
  __shared__ __align__(8) uint64_t merge_bar;

  const int t = a.token_list ? a.token_list[blockIdx.x] : blockIdx.x;
  const int h = blockIdx.y, sp = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_splits = a.n_splits, ps = a.page_size;
  pdl_launch_dependents();
  if (tid == 0) {
    mbar_init(&load_bar, 1);
    if (n_splits > 1 && sp == 0) mbar_init(&merge_bar, (uint32_t)(n_splits - 1));
    s_abort = 0;
    mbar_fence_init();
  }
  if (n_splits > 1) {
    // block 0's merge barrier exists before any block may signal it: arrive now, wait later
    __syncwarp();
    cluster_arrive();
  }
  // Before waiting for the kernel ahead: the step's metadata and the pages of EARLIER
  // positions, which that kernel cannot have written.
  if (a.token_req == nullptr) {
    const int* bt = a.block_table + (size_t)t * a.bt_stride;
    for (int i = tid; i < a.nb_max; i += THREADS) spage[i] = bt[i];
    if (tid == 0) { s_meta[0] = t; s_meta[1] = a.positions[t]; }
  } else {
    if (tid == 0) { s_meta[0] = a.token_req[t]; s_meta[1] = a.positions[t]; }
  }
  __syncthreads();
  const int r = s_meta[0];
  const int pos = s_meta[1];
  if (a.token_req != nullptr) {
    const int* bt = a.block_table + (size_t)r * a.bt_stride;
    int need = pos / ps + 1;
    if (need > a.nb_max) need = a.nb_max;
    for (int i = tid; i < need; i += THREADS) spage[i] = bt[i];
    __syncthreads();
  }
  const int lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  const int n = pos - lo + 1;
  int chunk = (n + n_splits - 1) / n_splits;
  if (chunk > a.chunk_cap) chunk = a.chunk_cap;      // cannot happen when the host sized chunk_cap
  const int k0 = lo + sp * chunk;
  int k1 = k0 + chunk;
  if (k1 > pos + 1) k1 = pos + 1;
  const int nk = k1 > k0 ? k1 - k0 : 0;
  const int G = a.H / a.Hkv;
  const int hk = h / G;
  const int pg0 = k0 / ps;
  const int pg1 = nk > 0 ? (k1 - 1) / ps : pg0 - 1;   // inclusive
  const int row0 = k0 - pg0 * ps;                     // the range's first key within the staged pages
  if (tid == 0 && nk > 0) {
    const int npg = pg1 - pg0 + 1;
    mbar_expect_tx(&load_bar, (uint32_t)npg * 2u * (uint32_t)ps * (uint32_t)D * 2u);
    for (int pi = pg0; pi <= pg1; pi++) {
      const int page = spage[pi];
      tma_load_5d(sK + (size_t)(pi - pg0) * ps * D, &map_kv, &load_bar, 0, 0, hk, 0, page);
      tma_load_5d(sV + (size_t)(pi - pg0) * ps * D, &map_kv, &load_bar, 0, 0, hk, 1, page);
    }
  }
  pdl_wait();
  // now the kernel ahead is complete: the query, and the token's own key and value (asked for side by side,
  // ahead of the wait for the staged pages)
  // LPR lanes share one key's row (16 bytes each): a warp reads KG whole rows at a time
  constexpr int LPR = D / 8;
  constexpr int KG = 32 / LPR;
  const int kg = lane / LPR, dl = lane % LPR;
  const uint4 q_raw = reinterpret_cast<const uint4*>(a.q + (size_t)t * a.q_stride + (size_t)h * D)[dl];
  const bool fused = a.k_new != nullptr;
  const bool own = nk > 0 && pos >= k0 && pos < k1;
  uint4 k_own = make_uint4(0u, 0u, 0u, 0u), v_own = k_own;
  __nv_bfloat16* kdst = nullptr;
  const size_t page_elems = (size_t)2 * a.Hkv * ps * D;
  const size_t head_off = (size_t)hk * ps * D, v_off = (size_t)a.Hkv * ps * D;
  if (own && tid < LPR) {
    // the token's own row: from the step's rows (and into the cache), or re-read from the cache,
    // where the kernel ahead put it after the page was requested
    const __nv_bfloat16* ksrc;
    const __nv_bfloat16* vsrc;
    if (fused) {
      ksrc = a.k_new + (size_t)t * a.new_stride + (size_t)hk * D;
      vsrc = a.v_new + (size_t)t * a.new_stride + (size_t)hk * D;
    } else {
      ksrc = a.cache + (size_t)spage[pos / ps] * page_elems + head_off + (size_t)(pos % ps) * D;
      vsrc = ksrc + v_off;
    }
    k_own = reinterpret_cast<const uint4*>(ksrc)[tid];
    v_own = reinterpret_cast<const uint4*>(vsrc)[tid];
    if (fused && h % G == 0) {
      const int slot = a.slots[t];
      if (slot >= 0) kdst = a.cache + (size_t)(slot / ps) * page_elems + head_off + (size_t)(slot % ps) * D;
    }
  }
  bool ok = true;
  if (nk > 0) {
    volatile int* af = &s_abort;
    ok = mbar_wait(&load_bar, 0, af);
  }
  if (own) {
    if (ok && tid < LPR) {
      const int row = pos - pg0 * ps;
      reinterpret_cast<uint4*>(sK + (size_t)row * D)[tid] = k_own;
      reinterpret_cast<uint4*>(sV + (size_t)row * D)[tid] = v_own;
      if (kdst) {
        reinterpret_cast<uint4*>(kdst)[tid] = k_own;
        reinterpret_cast<uint4*>(kdst + v_off)[tid] = v_own;
      }
    }
    __syncthreads();
  }

  // Every warp walks its own keys with a maximum and a sum of its own, four groups of rows at a time so that
  // their reads, their sums over the lanes and their exponentials do not wait for one another; the warps meet once.
  // (With the block's maximum and sum taken first, between barriers, and one group at a time a launch took 7.9 us in
  // the chain of a step of eight requests at context 512, now 5.9, and 5.8 for one request, now 4.8.  What is left is a
  // chain: the dependency's return, the query's way from L2, two passes, the cluster's exchange.)
  // A pass takes as many groups as are left, up to four: one of four for the last few keys costs their instructions all the
  // same (eight requests of 320 keys, 80 a block: 6.3 us instead of 5.8; of 272, 5.8 instead of 5.5).
  const int stride = WARPS * KG;
  float qreg[8];
  bf16x8_to_f32(q_raw, qreg);
#pragma unroll
  for (int y = 0; y < 8; y++) qreg[y] *= a.scale;
  float m_run = -INFINITY, l_run = 0.0f, acc[8];      // l_run, acc: this lane group's keys
#pragma unroll
  for (int y = 0; y < 8; y++) acc[y] = 0.0f;
  auto pass = [&](int wb, auto groups) {               // the keys wb + u stride + kg (the same for the whole warp)
    constexpr int UNROLL = decltype(groups)::value;
    float s[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const int i = wb + u * stride + kg;
      uint4 row = make_uint4(0u, 0u, 0u, 0u);
      if (i < nk) row = *reinterpret_cast<const uint4*>(sK + (size_t)(row0 + i) * D + dl * 8);
      float f[8];
      bf16x8_to_f32(row, f);
      float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
      for (int y = 0; y < 8; y += 2) {
        s0 = fmaf(qreg[y], f[y], s0);
        s1 = fmaf(qreg[y + 1], f[y + 1], s1);
      }
      s[u] = s0 + s1;
    }
#pragma unroll
    for (int o = 1; o < LPR; o <<= 1)
#pragma unroll
      for (int u = 0; u < UNROLL; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
    float m_new = m_run;
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      if (wb + u * stride + kg >= nk) s[u] = -INFINITY;
      m_new = fmaxf(m_new, s[u]);
    }
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
    const float m_use = m_new == -INFINITY ? 0.0f : m_new;
    const float corr = expf(m_run - m_use);            // (the first keys: exp(-inf) = 0)
    m_run = m_new;
    l_run *= corr;
#pragma unroll
    for (int y = 0; y < 8; y++) acc[y] *= corr;
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const int i = wb + u * stride + kg;
      if (i < nk) {
        const float w = expf(s[u] - m_use);
        l_run += w;
        const uint4 row = *reinterpret_cast<const uint4*>(sV + (size_t)(row0 + i) * D + dl * 8);
        float f[8];
        bf16x8_to_f32(row, f);
#pragma unroll
        for (int y = 0; y < 8; y++) acc[y] = fmaf(w, f[y], acc[y]);
      }
    }
  };
  if (ok) {
    int wb = warp * KG;
    for (; wb + 2 * stride < nk; wb += 4 * stride) pass(wb, std::integral_constant<int, 4>{});
    if (wb + stride < nk) pass(wb, std::integral_constant<int, 2>{});
    else if (wb < nk) pass(wb, std::integral_constant<int, 1>{});
  }
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    l_run += __shfl_xor_sync(0xffffffffu, l_run, o);
#pragma unroll
    for (int y = 0; y < 8; y++) acc[y] += __shfl_xor_sync(0xffffffffu, acc[y], o);
  }
  if (kg == 0) {
#pragma unroll
    for (int y = 0; y < 8; y += 4)
      *reinterpret_cast<float4*>(part + warp * D + dl * 8 + y) = make_float4(acc[y], acc[y + 1], acc[y + 2], acc[y + 3]);
  }
  if (lane == 0) {
    red[warp] = m_run;
    red[WARPS + warp] = l_run;
  }
  __syncthreads();
  float m = red[0];
#pragma unroll
  for (int w = 1; w < WARPS; w++) m = fmaxf(m, red[w]);
  float l = 0.0f, f_w[WARPS];
#pragma unroll
  for (int w = 0; w < WARPS; w++) {
    f_w[w] = red[w] == -INFINITY ? 0.0f : expf(red[w] - m);
    l += red[WARPS + w] * f_w[w];
  }
  auto block_out = [&](int d) {                        // the block's unnormalised result
    float o = 0.0f;
#pragma unroll
    for (int w = 0; w < WARPS; w++) o = fmaf(part[w * D + d], f_w[w], o);
    return o;
  };

  __nv_bfloat16* op = a.out + (size_t)t * a.o_stride + (size_t)h * D;
  if (n_splits == 1) {
    if (!ok) {
      if (tid == 0 && a.err) atomicExch(a.err, 1);
      return;
    }
    const float inv = 1.0f / l;
    for (int d = tid; d < D; d += THREADS) op[d] = __float2bfloat16_rn(block_out(d) * inv);
    return;
  }
  // Blocks 1.. send their (m, l, o) to block 0's shared memory and signal its barrier; block 0
  // waits for all of them (with a limit) and merges in range order.  Nothing remote is touched by
  // a block after its signal, and block 0 outlives every store into it (when its wait runs out,
  // through the cluster's hardware barrier: see there).
  constexpr int rec = D + 2;
  __syncwarp();
  cluster_wait();                    // pairs with the arrive at the top: block 0's barrier exists
  float* mine = recs + (size_t)sp * rec;
  if (sp != 0) {
    const uint32_t dst = map_to_peer(mine, 0);
    for (int d = tid; d < D; d += THREADS) st_peer_f32(dst + (uint32_t)(2 + d) * 4u, block_out(d));
    if (tid == 0) {
      st_peer_f32(dst, ok ? m : -INFINITY);
      st_peer_f32(dst + 4u, ok ? l : 0.0f);
      if (!ok && a.err) atomicExch(a.err, 1);
    }
    __syncthreads();
    if (tid == 0) mbar_arrive_peer(map_to_peer(&merge_bar, 0));
    return;
  }
  for (int d = tid; d < D; d += THREADS) mine[2 + d] = block_out(d);
  if (tid == 0) {
    mine[0] = m;
    mine[1] = l;
  }
  __syncthreads();
  {
    volatile int* af = &s_abort;
    if (!mbar_wait_cluster(&merge_bar, 0, af) || !ok) {
      if (tid == 0 && a.err) atomicExch(a.err, 1);
      // a peer that has not signalled may still be storing into this block's shared memory: the
      // cluster's hardware barrier completes when every block of it has arrived or exited, and
      // the peers exit right after their stores, so this block leaves after the last of them
      cluster_arrive();
      cluster_wait();
      return;
    }
  }
  // lane s holds range s's maximum and sum (an empty range: sum 0)
  const float m_s = lane < n_splits ? recs[lane * rec] : -INFINITY, l_s = lane < n_splits ? recs[lane * rec + 1] : 0.0f;
  const float M = warp_max(l_s > 0.0f ? m_s : -INFINITY);
  const float f_s = l_s > 0.0f ? expf(m_s - M) : 0.0f;
  const float inv = 1.0f / warp_sum(l_s * f_s);
  for (int d0 = 0; d0 < D; d0 += THREADS) {
    const int d = d0 + tid;
    if (d0 + warp * 32 >= D) break;
    float o = 0.0f;
    for (int s = 0; s < n_splits; s++) {
      const float f = __shfl_sync(0xffffffffu, f_s, s);
      if (f > 0.0f) o = fmaf(recs[s * rec + 2 + d], f, o);
    }
    op[d] = __float2bfloat16_rn(o * inv);
  }
}

// ---- host: the cache as a 5-D tensor, one box = one page's rows of one head (no swizzle) ----
struct KeyKV { const void* p; int D, ps, Hkv, n_pages, swizzled; };
std::mutex g_mutex;
std::vector<std::pair<KeyKV, CUtensorMap>> g_kvmaps;

// swizzled: boxes 64 elements (128 bytes) wide in the 128-byte swizzle (the streaming kernel's
// ldmatrix reads), else whole rows as they lie
bool get_kv_map(CUtensorMap* out, const void* cache, int D, int ps, int Hkv, int n_pages, bool swizzled = false) {
  std::lock_guard<std::mutex> lock(g_mutex);
  for (auto& e : g_kvmaps)
    if (e.first.p == cache && e.first.D == D && e.first.ps == ps && e.first.Hkv == Hkv &&
        e.first.n_pages == n_pages && e.first.swizzled == (int)swizzled) {
      *out = e.second;
      return true;
    }
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn || ((uintptr_t)cache & 15) || ps > 256 || D > 256) return false;
  cuuint64_t dims[5] = {(cuuint64_t)D, (cuuint64_t)ps, (cuuint64_t)Hkv, 2, (cuuint64_t)n_pages};
  cuuint64_t strides[4] = {(cuuint64_t)D * 2, (cuuint64_t)ps * D * 2, (cuuint64_t)Hkv * ps * D * 2,
                           (cuuint64_t)2 * Hkv * ps * D * 2};
  cuuint32_t box[5] = {(cuuint32_t)(swizzled ? 64 : D), (cuuint32_t)ps, 1, 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUtensorMap m;
  CUresult rc = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(cache), dims, strides, box,
                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return false;
  if (g_kvmaps.size() > 1024) g_kvmaps.clear();
  g_kvmaps.push_back({KeyKV{cache, D, ps, Hkv, n_pages, (int)swizzled}, m});
  *out = m;
  return true;
}

// ---- streaming variant for large batches -------------------------------------------------
// A fixed number of blocks per SM, each walking a list of (token, head) items.  One warp feeds
// a ring of shared-memory stages (64 keys and their values each) with the item's pages by TMA,
// in the 128-byte swizzle, and runs ahead of the four warps that consume them, across item
// boundaries, so a block never waits for a round trip between items: at large batches the
// one-shot kernels are bound by block lifetime times the number of blocks an SM holds, this
// one by bytes.  The four warps share every stage through the warp-level tensor-core
// instruction, the query being row 0 of a 16-row operand: each warp takes the scores of 16 of
// the stage's keys, the scores meet in shared memory (one block barrier a stage), every warp
// then does the same softmax step on all 64 and takes a quarter of the head's output columns.
// (The same sums on the CUDA cores cost eight times the instructions, and the kernel was bound
// by instruction issue.)  No merge at the end of an item: each warp holds the item's maximum
// and sum and its own columns.  The token's own key and value come from the step's rows (or
// the cache) by plain loads after the dependency wait, and are written into the cache here.
// 2^x by the special-function unit (arguments here are <= 0 up to rounding; -inf gives 0)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
// D[16x8] += A[16x16] B[16x8], bfloat16 operands, float accumulators; rows 8..15 of A are zero here
__device__ __forceinline__ void mma_row0(float* d, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

struct StreamArgs {
  Args b;
  int n_items;        // tokens served x heads
  int n_stages;
};
constexpr int S_SPLIT = 2;                 // blocks of a cluster that shares items (it then has one item)
constexpr int S_WARPS = 4;                  // consumer warps; warp S_WARPS produces
constexpr int S_THREADS = (S_WARPS + 1) * 32;
constexpr int S_MAX_STAGES = 8;
constexpr int S_PMAX = 8;                   // page ids held per producer lane: 256 pages per item
constexpr int S_TILE = 64;                  // keys per stage
constexpr int S_WHOLE_TILES = 4;            // tiles of an item that a cluster does not share

struct ItemGeom {
  int lo, first_page, k_base, n_rows, n_tiles, n_pages;
};
__device__ __forceinline__ ItemGeom item_geom(int pos, int window, int ps) {
  ItemGeom g;
  g.lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  g.first_page = g.lo / ps;
  g.k_base = g.first_page * ps;
  g.n_rows = pos - g.k_base;                       // cached rows ahead of the token's own
  g.n_tiles = (g.n_rows + S_TILE - 1) / S_TILE;
  g.n_pages = (g.n_rows + ps - 1) / ps;
  return g;
}

// SPLIT: clusters share items; the plain form is compiled without it.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(S_THREADS)
attention_decode_stream_kernel(const __grid_constant__ CUtensorMap map_kv, const StreamArgs sa) {
  const Args& a = sa.b;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // the 128-byte swizzle is a function of the address: stages start on 1024-byte boundaries
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int DH = D / 64;                // 128-byte column blocks of a row
  constexpr int NT = D / 8;                 // 8-wide output tiles of the head
  constexpr int NT_W = NT / S_WARPS;        // ... of one warp
  constexpr int KS = D / 16;                // 16-deep steps over the head dimension
  constexpr int LPR = D / 8;                // lanes that share the token's own row
  constexpr int HALF_BYTES = S_TILE * 128;               // one column block of a K or V tile
  constexpr int KV_BYTES = DH * HALF_BYTES;              // K (or V) of a stage
  constexpr int STAGE_BYTES = 2 * KV_BYTES;
  const int ps = a.page_size;
  const int tile_pages = S_TILE / ps;
  const int NS = sa.n_stages;
  __shared__ __align__(8) uint64_t full[S_MAX_STAGES];
  __shared__ __align__(8) uint64_t empty[S_MAX_STAGES];
  __shared__ float s_scores[2][S_TILE];     // a stage's scores, written by quarters, read by all
  __shared__ int s_abort;
  __shared__ __align__(8) uint64_t merge_bar;          // block 0 of a cluster: the others' shares are there
  __shared__ float recs[SPLIT ? (S_SPLIT - 1) * (D + 2) : 1];  // ... and lie here: (max, sum, D unnormalised results)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H, G = a.H / a.Hkv, rank = blockIdx.z;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], S_WARPS);
    }
    if (SPLIT) mbar_init(&merge_bar, (S_SPLIT - 1) * S_WARPS);
    s_abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  if (SPLIT) cluster_arrive();                         // (its other half stands ahead of the first remote store)
  volatile int* af = &s_abort;
  // this block's tiles of an item: all of them, or its rank's run of them
  // (an item of few tiles: the first rank's alone)
  auto shared_item = [&](const ItemGeom& g) { return SPLIT && g.n_tiles > S_WHOLE_TILES; };
  auto first_tile = [&](const ItemGeom& g) {
    if (!shared_item(g)) return SPLIT && rank != 0 ? g.n_tiles : 0;
    return min(g.n_tiles, rank * ((g.n_tiles + S_SPLIT - 1) / S_SPLIT));
  };
  auto last_tile = [&](const ItemGeom& g) {
    if (!shared_item(g)) return g.n_tiles;
    return min(g.n_tiles, (rank + 1) * ((g.n_tiles + S_SPLIT - 1) / S_SPLIT));
  };
  auto token_of = [&](int item) { int ti = item / H; return a.token_list ? a.token_list[ti] : ti; };
  // A block's items: one of every run of gridDim.x, counted from the front in even runs and from
  // the back in odd ones.  A caller that lists long tokens first thus gives every block long and
  // short items alike.
  auto after = [&](int item) {
    const int k = item / (int)gridDim.x + 1;
    return k * (int)gridDim.x + ((k & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  };

  if (warp == S_WARPS) {
    // ---- producer: metadata and pages of EARLIER positions only, which the kernel ahead
    // cannot have written, so nothing here waits for it ----
    auto pos_of = [&](int item) { return item < sa.n_items ? a.positions[token_of(item)] : 0; };
    auto load_ids = [&](int item, int pos, int* pid) {
      const int t = token_of(item);
      const int r = a.token_req ? a.token_req[t] : t;
      const ItemGeom g = item_geom(pos, a.window, ps);
      const int* bt = a.block_table + (size_t)r * a.bt_stride + g.first_page;
#pragma unroll
      for (int k = 0; k < S_PMAX; k++) {
        int i = k * 32 + lane;
        pid[k] = i < g.n_pages ? bt[i] : 0;
      }
    };
    int it = 0;
    int item = blockIdx.x;
    int pos_cur = pos_of(item), pos_nxt = pos_of(after(item));
    int pid_cur[S_PMAX], pid_nxt[S_PMAX];
    if (item < sa.n_items) load_ids(item, pos_cur, pid_cur);
    bool ok = true;
    while (item < sa.n_items && ok) {
      const int item_n = after(item);
      if (item_n < sa.n_items) load_ids(item_n, pos_nxt, pid_nxt);
      const int pos_n2 = pos_of(after(item_n));
      const ItemGeom g = item_geom(pos_cur, a.window, ps);
      const int hk = (item % H) / G;
      const int j_end = last_tile(g);
      for (int j = first_tile(g); j < j_end && ok; j++, it++) {
        const int s = it % NS;
        if (it >= NS) {
          int w = 1;
          if (lane == 0) w = mbar_wait(&empty[s], ((it / NS) - 1) & 1, af) ? 1 : 0;
          ok = __shfl_sync(0xffffffffu, w, 0) != 0;
          if (!ok) break;
        }
        const int pg0 = j * tile_pages;
        const int npg = min(tile_pages, g.n_pages - pg0);
        uint8_t* sk = smem + (size_t)s * STAGE_BYTES;
        uint8_t* sv = sk + KV_BYTES;
        if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)npg * 2u * (uint32_t)ps * (uint32_t)D * 2u);
        __syncwarp();
        // the lane that holds a page's id issues its copies: the pages of a stage go out side by side
        const int p = (lane - pg0) & 31;                 // this lane's page within the stage, if < npg
        if (p < npg) {
          const int idx = pg0 + p;
          int page = 0;
#pragma unroll
          for (int k = 0; k < S_PMAX; k++)
            if (k == (idx >> 5)) page = pid_cur[k];
#pragma unroll
          for (int hb = 0; hb < DH; hb++) {
            tma_load_5d(sk + hb * HALF_BYTES + p * ps * 128, &map_kv, &full[s], hb * 64, 0, hk, 0, page);
            tma_load_5d(sv + hb * HALF_BYTES + p * ps * 128, &map_kv, &full[s], hb * 64, 0, hk, 1, page);
          }
        }
      }
      item = item_n;
      pos_cur = pos_nxt;
      pos_nxt = pos_n2;
#pragma unroll
      for (int k = 0; k < S_PMAX; k++) pid_cur[k] = pid_nxt[k];
    }
    if (!ok && lane == 0) {
      // wait, with a limit, for the copies still in flight before the block may exit
      for (int i = max(0, it - NS); i < it; i++) mbar_wait(&full[i % NS], (i / NS) & 1, af);
    }
    if (SPLIT) {
      __syncwarp();
      cluster_wait();
    }
    return;
  }

  // ---- consumers ----
  const int gq = lane >> 2, tq = lane & 3;          // row group and column pair of the MMA fragments
  const int dl = lane % LPR;
  const float cexp = a.scale * 1.4426950408889634f; // scores in base-2 exponent units
  const size_t page_elems = (size_t)2 * a.Hkv * ps * D;
  const size_t v_off = (size_t)a.Hkv * ps * D;
  const bool fused = a.k_new != nullptr;
  // what an item needs from global memory is requested one item ahead: the position (step
  // metadata, readable at once), and the query as row 0 of the MMA's 16 x 16 operand (lanes
  // 0..3 hold it, the others zeros), which the kernel ahead writes
  int item = blockIdx.x;
  int t_nxt = item < sa.n_items ? token_of(item) : 0;
  int pos_nxt = item < sa.n_items ? a.positions[t_nxt] : 0;
  uint32_t qa_nxt[KS][2];
#pragma unroll
  for (int ks = 0; ks < KS; ks++) qa_nxt[ks][0] = qa_nxt[ks][1] = 0u;
  auto fetch_q = [&](int item_) {
    if (gq == 0) {
      const uint32_t* qp = reinterpret_cast<const uint32_t*>(a.q + (size_t)t_nxt * a.q_stride + (size_t)(item_ % H) * D);
#pragma unroll
      for (int ks = 0; ks < KS; ks++) {
        qa_nxt[ks][0] = qp[8 * ks + tq];
        qa_nxt[ks][1] = qp[8 * ks + 4 + tq];
      }
    }
  };
  pdl_wait();       // queries and the step's own keys and values come from the kernel ahead
  if (item < sa.n_items) fetch_q(item);
  int it = 0;
  for (; item < sa.n_items; item = after(item)) {
    const int t = t_nxt, pos = pos_nxt, h = item % H, hk = h / G;
    uint32_t qa[KS][2];
#pragma unroll
    for (int ks = 0; ks < KS; ks++) {
      qa[ks][0] = qa_nxt[ks][0];
      qa[ks][1] = qa_nxt[ks][1];
    }
    // the token's own key and value: every warp scores the key (lanes 0..LPR-1 hold 8 elements
    // of the query and of the key each) and takes the value's elements of its own columns
    const __nv_bfloat16* ksrc;
    const __nv_bfloat16* vsrc;
    int slot = -1;
    if (fused) {
      ksrc = a.k_new + (size_t)t * a.new_stride + (size_t)hk * D;
      vsrc = a.v_new + (size_t)t * a.new_stride + (size_t)hk * D;
      if (warp == 0) slot = a.slots[t];
    } else {
      const int r = a.token_req ? a.token_req[t] : t;
      const int page = a.block_table[(size_t)r * a.bt_stride + pos / ps];
      ksrc = a.cache + (size_t)page * page_elems + (size_t)hk * ps * D + (size_t)(pos % ps) * D;
      vsrc = ksrc + v_off;
    }
    uint4 kn = make_uint4(0u, 0u, 0u, 0u), qrow = kn, vn = kn;
    if (lane < LPR) {
      kn = reinterpret_cast<const uint4*>(ksrc)[dl];
      qrow = reinterpret_cast<const uint4*>(a.q + (size_t)t * a.q_stride + (size_t)h * D)[dl];
      if (warp == 0) vn = reinterpret_cast<const uint4*>(vsrc)[dl];
    }
    uint32_t v_own[NT_W];      // the value's elements 8 (NT_W warp + u) + 2 tq, +1 (lanes 0..3 use them)
#pragma unroll
    for (int u = 0; u < NT_W; u++)
      v_own[u] = reinterpret_cast<const uint32_t*>(vsrc)[4 * (NT_W * warp + u) + tq];
    if (after(item) < sa.n_items) {
      t_nxt = token_of(after(item));
      pos_nxt = a.positions[t_nxt];
      fetch_q(after(item));
    }
    const ItemGeom g = item_geom(pos, a.window, ps);
    float m_run = -INFINITY, l_run = 0.0f;      // l_run: this lane's share of the sum
    float o[NT_W][4];
#pragma unroll
    for (int u = 0; u < NT_W; u++) o[u][0] = o[u][1] = o[u][2] = o[u][3] = 0.0f;
    const int j_end = last_tile(g);
    for (int j = first_tile(g); j < j_end; j++, it++) {
      const int s = it % NS;
      bool ok = !*af && mbar_wait(&full[s], (it / NS) & 1, af);
      ok = __all_sync(0xffffffffu, ok);
      const uint32_t sk = smem_u32(smem + (size_t)s * STAGE_BYTES);
      const uint32_t sv = sk + KV_BYTES;
      const int key0 = g.k_base + j * S_TILE;
      const bool whole = key0 >= g.lo && key0 + S_TILE <= pos;
      float* sc_buf = s_scores[it & 1];
      if (ok) {
        if (!whole && lane < 16) {
          // rows that hold no key of this item may hold anything: their values are zeroed (a
          // zero weight times a non-number would still spoil the sum), their scores masked below
          const int row = 16 * warp + lane, key = key0 + row;
          if (key < g.lo || key >= pos) {
#pragma unroll
            for (int hb = 0; hb < DH; hb++)
#pragma unroll
              for (int c = 0; c < 8; c++)
                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(sv + hb * HALF_BYTES + row * 128 + c * 16), "r"(0u) : "memory");
          }
        }
        // scores of this warp's 16 keys (two tiles of 8) against row 0
        float sc[2][4];
#pragma unroll
        for (int u = 0; u < 2; u++) sc[u][0] = sc[u][1] = sc[u][2] = sc[u][3] = 0.0f;
        {
          const int mi = lane >> 3, row = lane & 7;
#pragma unroll
          for (int kp = 0; kp < KS; kp += 2) {
            const int c = 2 * kp + mi;                   // 16-byte column of the row
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const int key = 16 * warp + 8 * u + row;
              uint32_t b0, b1, b2, b3;
              ldmatrix_x4(sk + (c >> 3) * HALF_BYTES + key * 128 + (((c & 7) ^ (key & 7)) << 4), b0, b1, b2, b3);
              mma_row0(sc[u], qa[kp][0], qa[kp][1], b0, b1);
              mma_row0(sc[u], qa[kp + 1][0], qa[kp + 1][1], b2, b3);
            }
          }
        }
        if (gq == 0) {
#pragma unroll
          for (int u = 0; u < 2; u++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const int i = 16 * warp + 8 * u + 2 * tq + e;
              const int key = key0 + i;
              sc_buf[i] = (whole || (key >= g.lo && key < pos)) ? sc[u][e] * cexp : -INFINITY;
            }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(S_WARPS * 32) : "memory");     // scores and zeroed rows are there for all
      if (ok) {
        const float s0 = sc_buf[lane], s1 = sc_buf[lane + 32];
        const float m_new = fmaxf(m_run, warp_max(fmaxf(s0, s1)));
        if (m_new > -INFINITY) {
          const float corr = ex2(m_run - m_new);           // 0 at the first keys (m_run = -inf)
          const float p0 = ex2(s0 - m_new), p1 = ex2(s1 - m_new);
          m_run = m_new;
          l_run = l_run * corr + (p0 + p1);
#pragma unroll
          for (int u = 0; u < NT_W; u++) {
            o[u][0] *= corr;
            o[u][1] *= corr;
          }
          // the weights as row 0 of the MMA's 16 x 16 operand, 16 keys a step: this lane needs
          // keys 16 kk + 2 tq + {0, 1, 8, 9}; key i sits in lane i % 32 (p0 for i < 32, else p1)
          uint32_t pa[4][2];
#pragma unroll
          for (int kk = 0; kk < 4; kk++) {
            const float pv = kk < 2 ? p0 : p1;
            const int l0 = (16 * kk) % 32 + 2 * tq;
            const float w0 = __shfl_sync(0xffffffffu, pv, l0), w1 = __shfl_sync(0xffffffffu, pv, l0 + 1);
            const float w2 = __shfl_sync(0xffffffffu, pv, l0 + 8), w3 = __shfl_sync(0xffffffffu, pv, l0 + 9);
            pa[kk][0] = pack_bf16x2(w0, w1);
            pa[kk][1] = pack_bf16x2(w2, w3);
          }
          const int mi = lane >> 3, row = lane & 7;
#pragma unroll
          for (int kk = 0; kk < 4; kk++) {
            const int key = 16 * kk + (mi & 1) * 8 + row;
#pragma unroll
            for (int u = 0; u < NT_W; u += 2) {
              const int c = NT_W * warp + u + (mi >> 1);
              uint32_t b0, b1, b2, b3;
              ldmatrix_x4_trans(sv + (c >> 3) * HALF_BYTES + key * 128 + (((c & 7) ^ (key & 7)) << 4), b0, b1, b2, b3);
              mma_row0(o[u], pa[kk][0], pa[kk][1], b0, b1);
              mma_row0(o[u + 1], pa[kk][0], pa[kk][1], b2, b3);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);       // the stage may be refilled
    }
    if (!shared_item(g)) {
      if (SPLIT && rank != 0) break;
    } else {
      // the shares of the cluster's other blocks: pushed to block 0, which merges them in the order of the keys.
      // Nothing remote is touched by a block after its signal, and block 0 outlives every store into it.
      __syncwarp();
      cluster_wait();                                    // block 0's barrier exists
      if (rank != 0) {
        const uint32_t dst = map_to_peer(recs + (rank - 1) * (D + 2), 0);
        const float l_all = warp_sum(l_run);
        if (warp == 0 && lane == 0) {
          st_peer_f32(dst, *af ? -INFINITY : m_run);
          st_peer_f32(dst + 4u, *af ? 0.0f : l_all);
        }
        if (gq == 0) {
#pragma unroll
          for (int u = 0; u < NT_W; u++) {
            const uint32_t at = dst + (uint32_t)(2 + 8 * (NT_W * warp + u) + 2 * tq) * 4u;
            st_peer_f32(at, o[u][0]);
            st_peer_f32(at + 4u, o[u][1]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_peer(map_to_peer(&merge_bar, 0));
        break;
      }
      bool there = mbar_wait_cluster(&merge_bar, 0, af);
      there = __all_sync(0xffffffffu, there);
      if (!there) {
        // a block that has not signalled may still be storing here: the cluster's hardware barrier completes
        // when every block of it has arrived or exited, and the others exit right after their stores
        cluster_arrive();
        cluster_wait();
        break;
      }
      l_run = warp_sum(l_run);
      for (int x = 0; x < S_SPLIT - 1; x++) {
        const float* rec = recs + x * (D + 2);
        if (rec[1] == 0.0f) continue;                    // (an empty run of keys; a sum that is no number goes into the result)
        const float m_new = fmaxf(m_run, rec[0]), c0 = ex2(m_run - m_new), c1 = ex2(rec[0] - m_new);
        m_run = m_new;
        l_run = l_run * c0 + rec[1] * c1;
#pragma unroll
        for (int u = 0; u < NT_W; u++) {
          const int col = 2 + 8 * (NT_W * warp + u) + 2 * tq;
          o[u][0] = o[u][0] * c0 + rec[col] * c1;
          o[u][1] = o[u][1] * c0 + rec[col + 1] * c1;
        }
      }
      l_run = lane == 0 ? l_run : 0.0f;                  // (the lanes' shares are summed below)
    }
    // the token's own key and value, and the result
    {
      float fq[8], fk[8];
      bf16x8_to_f32(qrow, fq);
      bf16x8_to_f32(kn, fk);
      float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
      for (int y = 0; y < 8; y += 2) {
        s0 = fmaf(fq[y], fk[y], s0);
        s1 = fmaf(fq[y + 1], fk[y + 1], s1);
      }
      const float s_own = warp_sum(s0 + s1) * cexp;          // lanes beyond the row hold zeros
      const float m_fin = fmaxf(m_run, s_own);
      const float corr = ex2(m_run - m_fin), pw = ex2(s_own - m_fin);
      const float l_fin = warp_sum(l_run) * corr + pw;
      if (gq == 0 && !*af) {
        const float inv = 1.0f / l_fin;
        __nv_bfloat16* op = a.out + (size_t)t * a.o_stride + (size_t)h * D;
#pragma unroll
        for (int u = 0; u < NT_W; u++) {
          const __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(&v_own[u]);
          const float2 vf = __bfloat1622float2(vv);
          const float y0 = (o[u][0] * corr + pw * vf.x) * inv, y1 = (o[u][1] * corr + pw * vf.y) * inv;
          *reinterpret_cast<uint32_t*>(op + 8 * (NT_W * warp + u) + 2 * tq) = pack_bf16x2(y0, y1);
        }
      }
      if (warp == 0 && lane < LPR && fused && slot >= 0 && h % G == 0) {
        __nv_bfloat16* kdst = a.cache + (size_t)(slot / ps) * page_elems + (size_t)hk * ps * D + (size_t)(slot % ps) * D;
        reinterpret_cast<uint4*>(kdst)[dl] = kn;
        reinterpret_cast<uint4*>(kdst + v_off)[dl] = vn;
      }
    }
  }
  if (tid == 0 && *af && a.err) atomicExch(a.err, 1);
}

template <int D>
int launch(const CUtensorMap& mkv, const Args& a, int T, cudaStream_t stream) {
  size_t smem = (size_t)2 * a.rows_cap * D * 2 +
                ((size_t)WARPS * D + (size_t)a.nb_max + (size_t)8 * (D + 2)) * 4;
  if (smem > 200 * 1024) return SGLC_ERR_UNSUPPORTED;
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(attention_decode_tma_kernel<D>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaFuncSetAttribute(attention_decode_tma_kernel<D>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    configured = smem;
  }
  dim3 grid(T, a.H, a.n_splits);
  return sglc_launch(attention_decode_tma_kernel<D>, grid, dim3(THREADS), smem, stream, a.n_splits, true, mkv, a);
}
}  // namespace

// Whether this kernel takes the case (else: the register-staged kernel of attention_decode.cu).
SGLC_API int sglc_attention_decode_tma_supports(int D, int page_size, int n_splits) {
  return (D == 64 || D == 128) && page_size >= 1 && page_size <= 256 && n_splits >= 1 && n_splits <= 8;
}

// Arguments as sglc_attention_decode (without the global-memory scratch); n_pages: pages of
// the cache tensor; token_list: optional list of the T tokens to serve.
SGLC_API int sglc_attention_decode_tma(const void* q, int q_stride, void* cache, const int* block_table,
                                       int bt_stride, const int* token_req, const int* positions,
                                       void* out, int o_stride, int T, int H, int Hkv, int D,
                                       int page_size, float scale, int window, int max_keys,
                                       int n_splits, const void* k_new, const void* v_new,
                                       int new_stride, const int* slots, int* err,
                                       const int* token_list, int n_pages, cudaStream_t stream) {
  if (T <= 0) return SGLC_OK;
  if (H <= 0 || Hkv <= 0 || H % Hkv != 0 || page_size <= 0 || max_keys <= 0 || n_pages <= 0)
    return SGLC_ERR_ARGUMENT;
  if (!sglc_attention_decode_tma_supports(D, page_size, n_splits) || H > 65535) return SGLC_ERR_UNSUPPORTED;
  if (q_stride % 8 != 0 || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15)) return SGLC_ERR_UNSUPPORTED;
  if (k_new && (!v_new || !slots || new_stride % 8 != 0 || ((uintptr_t)k_new & 15) || ((uintptr_t)v_new & 15)))
    return SGLC_ERR_UNSUPPORTED;
  if ((page_size * D * 2) % 128 != 0) return SGLC_ERR_UNSUPPORTED;   // page blocks stay 128-byte aligned in shared memory
  CUtensorMap mkv;
  if (!get_kv_map(&mkv, cache, D, page_size, Hkv, n_pages)) return SGLC_ERR_UNSUPPORTED;
  Args a;
  a.q = (const __nv_bfloat16*)q; a.q_stride = q_stride;
  a.cache = (__nv_bfloat16*)cache;
  a.block_table = block_table; a.bt_stride = bt_stride;
  a.token_req = token_req; a.positions = positions; a.token_list = token_list;
  a.out = (__nv_bfloat16*)out; a.o_stride = o_stride;
  a.H = H; a.Hkv = Hkv; a.page_size = page_size;
  a.scale = scale; a.window = window;
  a.n_splits = n_splits;
  int eff = window > 0 && window < max_keys ? window : max_keys;
  a.chunk_cap = (eff + n_splits - 1) / n_splits;
  // whole pages are staged: the range may start and end inside a page
  a.rows_cap = ((a.chunk_cap + page_size - 1) / page_size + 1) * page_size;
  a.nb_max = (max_keys + page_size - 1) / page_size;
  if (a.nb_max > bt_stride) a.nb_max = bt_stride;
  a.k_new = (const __nv_bfloat16*)k_new; a.v_new = (const __nv_bfloat16*)v_new;
  a.new_stride = new_stride; a.slots = slots;
  a.err = err;
  if (D == 64) return launch<64>(mkv, a, T, stream);
  return launch<128>(mkv, a, T, stream);
}

// Whether the streaming kernel takes the case: head sizes 64 and 128, pages of 8, 16, 32 or 64
// positions (a stage holds 64 keys in whole pages, each page box on a 1024-byte boundary), and
// at most 256 pages per item.
SGLC_API int sglc_attention_decode_stream_supports(int D, int page_size, int max_keys, int window) {
  if (!(D == 64 || D == 128)) return 0;
  if (!(page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64)) return 0;
  int eff = window > 0 && window < max_keys ? window : max_keys;
  if ((eff + page_size - 1) / page_size + 1 > 32 * S_PMAX) return 0;
  return 1;
}

// Which of this file's kernels takes heads of 64: the split-key kernel with so many blocks an item (1 to 8), or (0) the
// streaming one; -1 where the rules by items and blocks stand.  By an estimate of the time in us, of what was measured behind
// a layer norm (17 numbers of items from 12 to 768, contexts of 60 to 960, alike and ragged, pages of 16): a block's walk over
// its keys, the merge in a cluster, what all blocks together do, and rounds of blocks where shared memory, sized by
// max_keys, does not hold all of them at once (clusters leave up to an eighth of the places empty).  Before, an item had a
// block for every 64 to 128 keys whatever was resident, and from 160 items on all went to the streaming kernel.  Before and
// now, us with the norm's 1.9: 96 items of 700 keys (of at most 1,024) 11.4, 7.5 and of 960 12.8, 8.5; 12 of 60 5.2, 4.3; 192
// of 200 9.2, 6.7, of 350 9.1, 7.7; 208 of 512 10.2, 9.2; 336 of 200 9.4, 7.0; 480 of 100 10.9, 6.4, of 200 15.7, 11.7; 144 of
// 700 13.0, 11.3.
// Of one to seven items the older rule dealt up to 32 shares, merged through memory, where eight in a cluster are the faster: one
// item of 1,024 / 2,048 / 4,096 keys 9.9, 6.3 / 11.1, 7.5 / 11.1, 10.0; seven 10.1, 6.5 / 12.1, 7.8 / 12.4, 10.3.  Contexts
// of 1,100 to 4,000 keys (12 to 500 items, alike and ragged): a second round of clusters costs what a first one does there; with
// the factor of the shorter ones 48 items of 3,200 went to the streaming kernel in 28.1 (eight shares 19.7), 96 ragged ones
// of up to 2,048 in 19.7 (16.9).  As it is, it is 1 % on average from the best of each of 160 such launches.
SGLC_API int sglc_attention_decode_form(int T, int H, int D, int page_size, int max_keys, int window) {
  if (D != 64 || page_size < 1 || page_size > 64 || (page_size * D * 2) % 128 != 0 || T <= 0 || H <= 0 || max_keys <= 0) return -1;
  const long long n = (long long)T * H;
  const int eff = window > 0 && window < max_keys ? window : max_keys;
  const double keys = 0.8 * eff;
  int best = -1;
  double best_us = 1e30;
  if (sglc_attention_decode_stream_supports(D, page_size, max_keys, window) && n >= 24) {
    const long long rounds = (n + 443) / 444;
    best_us = n * 2 <= 444 && eff > 256 ? 5.3 + 0.01 * keys : 1.0 + (double)rounds * (4.6 + 0.0155 * keys);
    best = 0;
  }
  // (the share that attention_decode.cu's rule deals stays where the two are about even)
  int dealt = (int)((2 * 148 + n - 1) / n);
  if (dealt < (max_keys + 127) / 128) dealt = (max_keys + 127) / 128;
  if (dealt > (max_keys + 63) / 64) dealt = (max_keys + 63) / 64;
  if (dealt > 8) dealt = 8;
  const int nb = (max_keys + page_size - 1) / page_size;
  for (int s = 1; s <= 8 && n * s <= 1536; s++) {
    const int chunk = (eff + s - 1) / s, rows = ((chunk + page_size - 1) / page_size + 1) * page_size;
    const int smem = 2 * rows * D * 2 + (WARPS * D + nb + 8 * (D + 2)) * 4;
    if (smem > 200 * 1024) continue;
    int here = 227 * 1024 / (smem + 2048);
    if (here > 10) here = 10;
    const int at_once = (int)(148 * here * (s == 1 ? 1.0 : s == 2 ? 0.97 : s == 3 ? 0.92 : 0.88));
    const long long blocks = n * s, rounds = (blocks + at_once - 1) / at_once;
    double us = (double)rounds * ((s == 1 ? 3.5 : 4.75) + 0.0135 * keys / s) + 0.0027 * (double)(blocks < at_once ? blocks : at_once);
    if (rounds > 1 && s > 1 && eff <= 1024) us *= 1.7;      // (clusters of a second round wait for whole groups of places)
    if (s == dealt) us -= 0.3;
    if (us < best_us) {
      best_us = us;
      best = s;
    }
  }
  return best;
}

// Same arguments and result as sglc_attention_decode_tma (n_splits has no meaning here: a block
// walks whole (token, head) items).  Meant for many items; any number is served.
SGLC_API int sglc_attention_decode_stream(const void* q, int q_stride, void* cache, const int* block_table,
                                          int bt_stride, const int* token_req, const int* positions,
                                          void* out, int o_stride, int T, int H, int Hkv, int D,
                                          int page_size, float scale, int window, int max_keys,
                                          const void* k_new, const void* v_new, int new_stride,
                                          const int* slots, int* err, const int* token_list,
                                          int n_pages, cudaStream_t stream) {
  if (T <= 0) return SGLC_OK;
  if (H <= 0 || Hkv <= 0 || H % Hkv != 0 || page_size <= 0 || max_keys <= 0 || n_pages <= 0)
    return SGLC_ERR_ARGUMENT;
  if (!sglc_attention_decode_stream_supports(D, page_size, max_keys, window)) return SGLC_ERR_UNSUPPORTED;
  if (q_stride % 8 != 0 || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15)) return SGLC_ERR_UNSUPPORTED;
  if (k_new && (!v_new || !slots || new_stride % 8 != 0 || ((uintptr_t)k_new & 15) || ((uintptr_t)v_new & 15)))
    return SGLC_ERR_UNSUPPORTED;
  if ((page_size * D * 2) % 128 != 0) return SGLC_ERR_UNSUPPORTED;
  if ((long long)T * H > 0x7fffffffLL) return SGLC_ERR_UNSUPPORTED;
  CUtensorMap mkv;
  if (!get_kv_map(&mkv, cache, D, page_size, Hkv, n_pages, true)) return SGLC_ERR_UNSUPPORTED;
  StreamArgs sa;
  memset(&sa, 0, sizeof(sa));
  Args& a = sa.b;
  a.q = (const __nv_bfloat16*)q; a.q_stride = q_stride;
  a.cache = (__nv_bfloat16*)cache;
  a.block_table = block_table; a.bt_stride = bt_stride;
  a.token_req = token_req; a.positions = positions; a.token_list = token_list;
  a.out = (__nv_bfloat16*)out; a.o_stride = o_stride;
  a.H = H; a.Hkv = Hkv; a.page_size = page_size;
  a.scale = scale; a.window = window;
  a.n_splits = 1;
  a.k_new = (const __nv_bfloat16*)k_new; a.v_new = (const __nv_bfloat16*)v_new;
  a.new_stride = new_stride; a.slots = slots;
  a.err = err;
  sa.n_items = T * H;
  const size_t stage_bytes = (size_t)2 * S_TILE * D * 2;   // 64 keys and 64 values
  // three blocks per SM (two at head size 128), and as many stages as then fit, three at least
  int n_stages = (int)(((size_t)72 * 1024 - 1024) / stage_bytes);
  if (n_stages > S_MAX_STAGES) n_stages = S_MAX_STAGES;
  if (n_stages < 3) n_stages = 3;
  sa.n_stages = n_stages;
  const size_t smem = (size_t)n_stages * stage_bytes + 1024;
  if (smem > 200 * 1024) return SGLC_ERR_UNSUPPORTED;
  static int n_sm = 0;
  if (n_sm == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n_sm <= 0) n_sm = 148;
  }
  int per_sm = (int)((220 * 1024) / (smem + 2048));
  if (per_sm > 3) per_sm = 3;
  if (per_sm < 1) per_sm = 1;
  int grid = n_sm * per_sm;
  // Items of 64 entries that leave half of the resident blocks without work are shared by clusters of two blocks (of 128 they
  // would be fewer than come here): 208 items of 350 to 700
  // keys 14.3 -> 9.7 us a launch (28 MB of keys and values, 4.3 us at the copy rate).  An item of up to S_WHOLE_TILES tiles
  // stays with its cluster's first block, and where no item can have more the launch is the plain one (its items
  // have the same bits; a cluster costs it 0.2 to 1.2 us: 192 items of 32 / 100 / 200 keys 4.3 / 5.1 / 7.3 us plain, 5.0 /
  // 6.1 / 7.7 in pairs; from 272 on the pairs win, 8.4 -> 7.6).  So a token's bits follow its own keys and the number of
  // items, and not max_keys.
  const int most_rows = (window > 0 && window < max_keys ? window + page_size - 1 : max_keys) - 1;
  const bool split = D == 64 && sa.n_items * 2 <= grid && most_rows > S_WHOLE_TILES * S_TILE;
  if (split || grid > sa.n_items) grid = sa.n_items;
  auto kern = split ? attention_decode_stream_kernel<64, true>
              : D == 64 ? attention_decode_stream_kernel<64, false>
                        : attention_decode_stream_kernel<128, false>;
  static size_t configured[3] = {0, 0, 0};
  size_t& conf = configured[split ? 2 : D == 64 ? 0 : 1];
  if (smem > 48 * 1024 && smem > conf) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    conf = smem;
  }
  return sglc_launch(kern, dim3(grid, 1, split ? S_SPLIT : 1), dim3(S_THREADS), smem, stream, split ? S_SPLIT : 1, true, mkv, sa);
}
