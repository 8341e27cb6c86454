// Causal attention over the paged cache for any mix of prompt portions and single decoded
// tokens.  All arithmetic is 32-bit:
//   s[p] = (q·K_p)*scale for the keys p the query may see (p <= its position,
//   and p > position - window if a window is set); m = max s; e = exp(s-m);
//   o = sum_p e[p]*V_p / sum_p e[p]
// (reference src/gpt2.c:238-270; GPU twin k_attn, src/cuda_backend.cu:1600-1651).
// A (token, head) is one warp.  It takes its keys in tiles of 32 by absolute position (tile k
// holds positions 32k..32k+31: a lane a key for the scores, the softmax statistics kept online
// from tile to tile, then a lane per output dimension over the tile's values), so its order of
// additions depends only on its own first and last visible key, never on the rest of the batch:
// the result is the same, bit for bit, however the tokens were cut into steps.  The tokens of a
// block that belong to one request share each tile of that request's keys and values in shared
// memory (a block of eight consecutive tokens of a prompt portion reads them once instead of
// eight times: the reference's kernel, one block per token, reads them per token).  This is the
// kernel of the 32-bit path and the general fallback of the bfloat16 path.
#include <limits.h>

#include <type_traits>

#include "common.cuh"

SGLC_DEFINE_ERROR_STRING()

// Four consecutive cache elements as 32-bit floats, by one load (p is aligned to four elements).
__device__ __forceinline__ void load4(const float* p, float* v) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float* v) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
  v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
}

// W: tokens of a block (a warp each).  Threads beyond the tokens' warps only help to stage tiles.
// EXT: the form with a value size DV of its own (a page then holds Hkv x page_size x D keys
// followed by Hkv x page_size x DV values), a chunk mask (a query sees only keys of its own chunk of
// `chunk` positions, counted from position 0) and a sink per head (a learned score that joins the
// softmax's denominator once, with no key and no value), and an output gate (a head's result times
// the sigmoid of a number per head, or of one per entry).  Without EXT these arguments are unused.
// NA: columns of the output a lane holds (a head's value size is at most 32 * NA).
struct OutGate {
  const float* z;                 // pre-activations, rows `stride` apart (null: no gate)
  long long stride;
  int per_head;                   // 1: z[t][h]; 0: z[t][h * DV + d]
};
__device__ __forceinline__ float out_gate(const OutGate& g, long long t, int h, int DV, int d) {
  const float z = g.z[t * g.stride + (g.per_head ? h : h * DV + d)];
  return 1.0f / (1.0f + expf(-z));
}

template <typename TQ, typename TC, typename TO, int W, int THREADS, bool EXT, int NA>
__global__ void __launch_bounds__(THREADS, NA > 8 ? 1 : THREADS == 256 ? 3 : 4)     // (registers capped so that three blocks of 256 share an SM)
attention_simt_kernel(const TQ* __restrict__ q, int q_stride, const TC* __restrict__ cache,
                      const int* __restrict__ block_table, int bt_stride,
                      const int* __restrict__ token_req, const int* __restrict__ positions,
                      TO* __restrict__ out, int o_stride, int T, int H, int Hkv, int D, int page_size,
                      float scale, int window, int n_pages, int* err, int kv_shared,
                      int DV_arg, int chunk, const float* __restrict__ sinks, int n_splits,
                      float* __restrict__ part_ws, int head_rows, const OutGate gate) {
  const int DV = EXT ? DV_arg : D;
  // head_rows (EXT, a step of single tokens): the block's warps are the query heads that share one
  // key/value head, all of ONE token (blockIdx.x), instead of consecutive tokens of one head: the
  // tile of keys and values is staged once for all of them
  const bool hrows = EXT && head_rows;
  const int grp = H / Hkv;
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_req[W], s_lo[W], s_pos[W];
  // padded key rows: a lane a key without bank conflicts (by 4 where rows are read 16 bytes at a time)
  const bool wide = D % 4 == 0;
  const int DP = wide ? D + 4 : D + 1;
  float* Ks = smem;                           // [32][DP]
  float* Vs = Ks + 32 * DP;                   // [32][D]
  float* pw = Vs + 32 * DV;                   // [W][32]: a tile's weights (16-byte aligned whatever D is)
  float* qs = pw + W * 32;                    // [W][D]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hk = hrows ? (int)blockIdx.y : (int)blockIdx.y / grp;
  const int h = hrows ? hk * grp + min(warp, grp - 1) : (int)blockIdx.y;      // this warp's query head
  const int t0 = hrows ? (int)blockIdx.x : (int)blockIdx.x * W;
  const int my_t = hrows ? t0 : t0 + warp;                                     // this warp's token
  if (tid < W) {
    const int t = hrows ? t0 : t0 + tid;
    const bool on = hrows ? tid < grp : t < T;
    const int pos = on ? positions[t] : -1;
    s_req[tid] = on ? token_req[t] : -1;
    s_pos[tid] = pos;
    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (EXT && chunk > 0 && pos >= 0) lo = max(lo, pos / chunk * chunk);
    s_lo[tid] = lo;
  }
  const bool mine = warp < W && (hrows ? warp < grp : t0 + warp < T);
  if (mine) {
    const TQ* qp = q + (size_t)my_t * q_stride + (size_t)h * D;
    for (int d = lane; d < D; d += 32) qs[warp * D + d] = to_f32(qp[d]);
  }
  __syncthreads();
  const int my_req = mine ? s_req[warp] : -2, my_lo = mine ? s_lo[warp] : 0, my_pos = mine ? s_pos[warp] : -1;
  float m = -INFINITY, l = 0.0f;
  float acc[NA];                              // dims lane, lane + 32, ... of the output
#pragma unroll
  for (int i = 0; i < NA; i++) acc[i] = 0.0f;
  // kv_shared: a page holds one block of rows that are keys and values at once (a latent)
  const size_t page_elems = EXT && !kv_shared ? (size_t)Hkv * page_size * (D + DV) : (size_t)(kv_shared ? 1 : 2) * Hkv * page_size * D;
  const size_t head_off = (size_t)hk * page_size * D, v_off = kv_shared ? 0 : (size_t)Hkv * page_size * D;

  // The tokens of a block that belong to one request (a run: a request's tokens lie together)
  // share the tiles of that request's keys and values; the runs of a block take turns.
  for (int lead = 0; lead < W; lead++) {
    const int rl = s_req[lead];
    if (rl < 0 || (lead > 0 && s_req[lead - 1] == rl)) continue;         // not the start of a run
    int lo_min = s_lo[lead], pos_max = s_pos[lead];
    for (int w = lead + 1; w < W && s_req[w] == rl; w++) {
      lo_min = min(lo_min, s_lo[w]);
      pos_max = max(pos_max, s_pos[w]);
    }
    const int* bt = block_table + (size_t)rl * bt_stride;
    int kt_first = lo_min / 32, kt_end = pos_max / 32 + 1;
    if (EXT && part_ws) {
      // the keys in sight dealt to the blocks of grid.z in runs of whole tiles (a step of single
      // tokens: a block has one token, so the run follows from its own first and last key)
      const int per = (kt_end - kt_first + n_splits - 1) / n_splits;
      kt_first += (int)blockIdx.z * per;
      kt_end = min(kt_end, kt_first + per);
    }
    for (int kt = kt_first; kt < kt_end; kt++) {
      const int key0 = kt * 32;
      __syncthreads();                        // the tile before has been used by everybody
      {
        // THREADS/32 threads bring one key and its value: the page is looked up once a key, and a
        // thread's loads do not depend on one another
        constexpr int TPK = THREADS / 32;
        const int j = tid / TPK, part = tid % TPK, p = key0 + j;
        const TC* kp = nullptr;
        if (p >= lo_min && p <= pos_max) {
          const int page = bt[p / page_size];
          if (sglc_index_ok(page, n_pages, err))
            kp = cache + (size_t)page * page_elems + head_off + (size_t)(p % page_size) * D;
        }
        if (EXT) {
          const TC* vp = kp && kv_shared ? kp : kp ? cache + (size_t)(bt[p / page_size]) * page_elems + (size_t)Hkv * page_size * D +
                                  ((size_t)hk * page_size + p % page_size) * DV
                            : nullptr;
          if (D % 4 == 0 && DV % 4 == 0) {      // (rows, pages and both blocks of a page start at multiples of four)
            for (int d = part * 4; d < D; d += 4 * TPK) {
              float k4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
              if (kp) load4(kp + d, k4);
              *reinterpret_cast<float4*>(&Ks[j * DP + d]) = make_float4(k4[0], k4[1], k4[2], k4[3]);
            }
            for (int d = part * 4; d < DV; d += 4 * TPK) {
              float v4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
              if (vp) load4(vp + d, v4);
              *reinterpret_cast<float4*>(&Vs[j * DV + d]) = make_float4(v4[0], v4[1], v4[2], v4[3]);
            }
          } else {
            for (int d = part; d < D; d += TPK) Ks[j * DP + d] = kp ? to_f32(kp[d]) : 0.0f;
            for (int d = part; d < DV; d += TPK) Vs[j * DV + d] = vp ? to_f32(vp[d]) : 0.0f;
          }
        } else if (D % 4 == 0) {
          for (int d = part * 4; d < D; d += 4 * TPK) {
            float k4[4] = {0.0f, 0.0f, 0.0f, 0.0f}, v4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (kp) {
              load4(kp + d, k4);
              load4(kp + v_off + d, v4);
            }
            *reinterpret_cast<float4*>(&Ks[j * DP + d]) = make_float4(k4[0], k4[1], k4[2], k4[3]);
            *reinterpret_cast<float4*>(&Vs[j * D + d]) = make_float4(v4[0], v4[1], v4[2], v4[3]);
          }
        } else {
          for (int d = part; d < D; d += TPK) {
            Ks[j * DP + d] = kp ? to_f32(kp[d]) : 0.0f;
            Vs[j * D + d] = kp ? to_f32(kp[v_off + d]) : 0.0f;
          }
        }
      }
      __syncthreads();
      // a token takes the tile if it belongs to the run and the tile holds keys it may see
      if (my_req == rl && key0 <= my_pos && key0 + 31 >= my_lo) {
        const int key = key0 + lane;
        const bool valid = key >= my_lo && key <= my_pos;
        const float* qv = qs + warp * D;
        const float* kr = Ks + lane * DP;
        float sc = 0.0f;
        if (wide) {                           // (the same additions in the same order, four a load)
          for (int d = 0; d < D; d += 4) {
            const float4 q4 = *reinterpret_cast<const float4*>(qv + d);
            const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
            sc = fmaf(q4.x, k4.x, sc);
            sc = fmaf(q4.y, k4.y, sc);
            sc = fmaf(q4.z, k4.z, sc);
            sc = fmaf(q4.w, k4.w, sc);
          }
        } else {
          for (int d = 0; d < D; d++) sc = fmaf(qv[d], kr[d], sc);
        }
        sc = valid ? sc * scale : -INFINITY;
        const float m_new = fmaxf(m, warp_max(sc));
        const float corr = expf(m - m_new);                             // (first tile: exp(-inf) = 0)
        const float p = valid ? expf(sc - m_new) : 0.0f;
        l = l * corr + warp_sum(p);
        m = m_new;
        pw[warp * 32 + lane] = p;
        __syncwarp();
        float pj[32];                         // the tile's weights, read once for all output columns
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 p4 = *reinterpret_cast<const float4*>(&pw[warp * 32 + j]);
          pj[j] = p4.x; pj[j + 1] = p4.y; pj[j + 2] = p4.z; pj[j + 3] = p4.w;
        }
#pragma unroll
        for (int i = 0; i < NA; i++) {
          const int d = lane + 32 * i;
          if (d < DV) {
            float a = acc[i] * corr;
#pragma unroll
            for (int j = 0; j < 32; j++) a = fmaf(pj[j], Vs[j * DV + d], a);
            acc[i] = a;
          }
        }
        __syncwarp();
      }
    }
  }
  if (EXT && part_ws) {
    // this block's share of the keys: maximum, sum and unnormalised result, for the merge
    if (mine) {
      float* rec = part_ws + (((size_t)my_t * H + h) * n_splits + blockIdx.z) * (DV + 2);
      if (lane == 0) { rec[0] = m; rec[1] = l; }
#pragma unroll
      for (int i = 0; i < NA; i++) {
        const int d = lane + 32 * i;
        if (d < DV) rec[2 + d] = acc[i];
      }
    }
    return;
  }
  if (mine) {
    TO* op = out + (size_t)my_t * o_stride + (size_t)h * DV;
    float inv = 1.0f / l;
    if (EXT && sinks) {                        // the sink joins the denominator: exp(sink - max) once
      const float sk = sinks[h], m_all = fmaxf(m, sk);
      inv = expf(m - m_all) / (l * expf(m - m_all) + expf(sk - m_all));
    }
    const bool gated = EXT && gate.z;
#pragma unroll
    for (int i = 0; i < NA; i++) {
      const int d = lane + 32 * i;
      if (d < DV) op[d] = from_f32<TO>(gated ? acc[i] * inv * out_gate(gate, my_t, h, DV, d) : acc[i] * inv);
    }
  }
}

// ---- the 32-bit path's own two forms (head sizes that are multiples of 4, up to 128; no extensions) -----------
// The same arithmetic in the same order as the kernel above, so the same bits; what differs is who does it and
// how the tiles come.  The kernel above spends its time on shared-memory reads (of 128 multiply-adds a lane and
// tile, 104 reads) and on waits for tiles that nothing covers.
__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct F32Args {
  const float* q; int q_stride;
  const float* cache;
  const int* block_table; int bt_stride;
  const int* token_req; const int* positions;
  float* out; int o_stride;
  int T, H, Hkv, D, page_size;
  float scale;
  int window, n_pages, kv_shared;
  int* err;
};
// key p of request row bt: its key row (the value row lies v_off behind it); null where the page id is bad
__device__ __forceinline__ const float* f32_row(const F32Args& a, const int* bt, int p, size_t page_elems, size_t head_off) {
  const int page = bt[p / a.page_size];
  if (!sglc_index_ok(page, a.n_pages, a.err)) return nullptr;
  return a.cache + (size_t)page * page_elems + head_off + (size_t)(p % a.page_size) * a.D;
}

// Prompt portions: a warp has FP_Q consecutive tokens, so a key or a value leaves shared memory once for all of
// them; eight warps a block share the tiles, which come by asynchronous copies one tile ahead.
// 1,872 tokens of three prompts (up to 780 keys), 12 heads of 64: 280 -> 170 us.  Bound by shared-memory reads (224 passes
// a warp and tile beside 128 cycles of multiply-adds); eight tokens a warp would halve them but leave one block
// an SM: 194 us.  The last tokens of a prompt, which see the most keys, go first.
constexpr int FP_Q = 4, FP_W = 8 * FP_Q;
template <int NA>      // head sizes up to 32 NA
__global__ void __launch_bounds__(256, 2)
attention_f32_portion_kernel(const F32Args a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_req[FP_W], s_lo[FP_W], s_pos[FP_W];
  pdl_launch_dependents();
  const int D = a.D, DP = D + 4, tile_floats = 32 * (DP + D);
  float* qs = smem + 2 * tile_floats;                // [FP_W][D]
  float* pw = qs + FP_W * D;                         // [FP_W][32]: a tile's weights
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x, hk = h / (a.H / a.Hkv);
  const int t0 = (gridDim.y - 1 - blockIdx.y) * FP_W;                    // (a prompt's last tokens see the most keys: first)
  const size_t page_elems = (size_t)(a.kv_shared ? 1 : 2) * a.Hkv * a.page_size * D;
  const size_t head_off = (size_t)hk * a.page_size * D, v_off = a.kv_shared ? 0 : (size_t)a.Hkv * a.page_size * D;
  pdl_wait();
  if (tid < FP_W) {
    const int t = t0 + tid;
    const bool on = t < a.T;
    const int pos = on ? a.positions[t] : -1;
    s_req[tid] = on ? a.token_req[t] : -1;
    s_pos[tid] = pos;
    s_lo[tid] = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  }
  for (int x = tid; x < FP_W * D; x += 256) {
    const int w = x / D, d = x - w * D;
    qs[x] = t0 + w < a.T ? a.q[(size_t)(t0 + w) * a.q_stride + (size_t)h * D + d] : 0.0f;
  }
  __syncthreads();
  int my_req[FP_Q], my_lo[FP_Q], my_pos[FP_Q];
  float m[FP_Q], l[FP_Q], acc[FP_Q][NA];
#pragma unroll
  for (int i = 0; i < FP_Q; i++) {
    my_req[i] = s_req[warp * FP_Q + i]; my_lo[i] = s_lo[warp * FP_Q + i]; my_pos[i] = s_pos[warp * FP_Q + i];
    m[i] = -INFINITY; l[i] = 0.0f;
#pragma unroll
    for (int n = 0; n < NA; n++) acc[i][n] = 0.0f;
  }
  const float* qv = qs + warp * FP_Q * D;
  float* pv = pw + warp * FP_Q * 32;
  for (int lead = 0; lead < FP_W; lead++) {
    const int rl = s_req[lead];
    if (rl < 0 || (lead > 0 && s_req[lead - 1] == rl)) continue;         // not the start of a run
    int lo_min = s_lo[lead], pos_max = s_pos[lead];
    for (int w = lead + 1; w < FP_W && s_req[w] == rl; w++) {
      lo_min = min(lo_min, s_lo[w]);
      pos_max = max(pos_max, s_pos[w]);
    }
    const int* bt = a.block_table + (size_t)rl * a.bt_stride;
    const int kt_first = lo_min / 32, kt_end = pos_max / 32 + 1;
    auto ask = [&](int kt) {                          // eight threads bring one key and its value
      if (kt < kt_end) {
        float* ks = smem + (kt & 1) * tile_floats;
        float* vs = ks + 32 * DP;
        const int j = tid >> 3, part = tid & 7, p = kt * 32 + j;
        const float* kp = (p >= lo_min && p <= pos_max) ? f32_row(a, bt, p, page_elems, head_off) : nullptr;
        for (int d = part * 4; d < D; d += 32) {
          copy16_or_zero(ks + j * DP + d, kp ? kp + d : a.cache, kp != nullptr);
          copy16_or_zero(vs + j * D + d, kp ? kp + v_off + d : a.cache, kp != nullptr);
        }
      }
      copies_commit();
    };
    __syncthreads();                                  // (the run before is done with the tiles)
    ask(kt_first);
    for (int kt = kt_first; kt < kt_end; kt++) {
      ask(kt + 1);
      copies_wait<1>();
      __syncthreads();                                // tile kt has landed
      const int key0 = kt * 32;
      bool on[FP_Q];
      bool any = false;
#pragma unroll
      for (int i = 0; i < FP_Q; i++) {
        on[i] = my_req[i] == rl && key0 <= my_pos[i] && key0 + 31 >= my_lo[i];
        any = any || on[i];
      }
      if (any) {
        const float* ks = smem + (kt & 1) * tile_floats;
        const float* vs = ks + 32 * DP;
        const float* kr = ks + lane * DP;
        float sc[FP_Q], corr[FP_Q];
#pragma unroll
        for (int i = 0; i < FP_Q; i++) sc[i] = 0.0f;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
          for (int i = 0; i < FP_Q; i++) {
            const float4 q4 = *reinterpret_cast<const float4*>(qv + i * D + d);
            sc[i] = fmaf(q4.x, k4.x, sc[i]);
            sc[i] = fmaf(q4.y, k4.y, sc[i]);
            sc[i] = fmaf(q4.z, k4.z, sc[i]);
            sc[i] = fmaf(q4.w, k4.w, sc[i]);
          }
        }
        const int key = key0 + lane;
#pragma unroll
        for (int i = 0; i < FP_Q; i++) {
          corr[i] = 1.0f;
          if (!on[i]) continue;
          const bool valid = key >= my_lo[i] && key <= my_pos[i];
          const float s = valid ? sc[i] * a.scale : -INFINITY;
          const float m_new = fmaxf(m[i], warp_max(s));
          corr[i] = expf(m[i] - m_new);                                 // (first tile: exp(-inf) = 0)
          const float p = valid ? expf(s - m_new) : 0.0f;
          l[i] = l[i] * corr[i] + warp_sum(p);
          m[i] = m_new;
          pv[i * 32 + lane] = p;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < FP_Q; i++)
#pragma unroll
          for (int n = 0; n < NA; n++)
            if (on[i]) acc[i][n] *= corr[i];
        // Four keys' values at a time.  In a tile that some of the warp's tokens see in part, their sums leave the other keys
        // out (the weight zero times an infinite value is not zero), and keys that none of them sees are passed over.
        auto add_four = [&](int j, auto whole) {
          float4 p4[FP_Q];
#pragma unroll
          for (int i = 0; i < FP_Q; i++) p4[i] = *reinterpret_cast<const float4*>(pv + i * 32 + j);
#pragma unroll
          for (int n = 0; n < NA; n++) {
            const int d = min(lane + 32 * n, D - 1);                    // (lanes beyond the head size: not stored)
            const float v0 = vs[j * D + d], v1 = vs[(j + 1) * D + d], v2 = vs[(j + 2) * D + d], v3 = vs[(j + 3) * D + d];
#pragma unroll
            for (int i = 0; i < FP_Q; i++)
              if (on[i]) {
                const int key4 = key0 + j;
                auto sees = [&](int e) { return decltype(whole)::value || (key4 + e >= my_lo[i] && key4 + e <= my_pos[i]); };
                float x = acc[i][n];
                if (sees(0)) x = fmaf(p4[i].x, v0, x);
                if (sees(1)) x = fmaf(p4[i].y, v1, x);
                if (sees(2)) x = fmaf(p4[i].z, v2, x);
                if (sees(3)) x = fmaf(p4[i].w, v3, x);
                acc[i][n] = x;
              }
          }
        };
        int any_lo = INT_MAX, any_pos = -1, all_lo = 0, all_pos = INT_MAX;       // keys that some, that all of the tokens see
#pragma unroll
        for (int i = 0; i < FP_Q; i++)
          if (on[i]) {
            any_lo = min(any_lo, my_lo[i]); any_pos = max(any_pos, my_pos[i]);
            all_lo = max(all_lo, my_lo[i]); all_pos = min(all_pos, my_pos[i]);
          }
        if (key0 >= all_lo && key0 + 31 <= all_pos) {
#pragma unroll 2
          for (int j = 0; j < 32; j += 4) add_four(j, std::true_type{});
        } else {
#pragma unroll 1
          for (int j = 0; j < 32; j += 4) {
            const int key4 = key0 + j;
            if (key4 + 3 < any_lo || key4 > any_pos) continue;
            if (key4 >= all_lo && key4 + 3 <= all_pos) add_four(j, std::true_type{});
            else add_four(j, std::false_type{});
          }
        }
        __syncwarp();
      }
      __syncthreads();                                // everybody is done with tile kt: the next but one may come
    }
  }
#pragma unroll
  for (int i = 0; i < FP_Q; i++) {
    const int t = t0 + warp * FP_Q + i;
    if (t >= a.T) continue;
    const float inv = 1.0f / l[i];
    float* op = a.out + (size_t)t * a.o_stride + (size_t)h * D;
#pragma unroll
    for (int n = 0; n < NA; n++)
      if (lane + 32 * n < D) op[lane + 32 * n] = acc[i][n] * inv;
  }
}

// Single tokens: a block has one (token, head).  Rounds of two tiles come through three stages of asynchronous copies;
// while warps 0 and 1 walk the softmax and the sums over the values of one round (a half of the head's columns
// each, the chain from tile to tile), warps 2 and 3 make the next round's scores, a tile each.
// Eight requests of 60 to 140 keys, 12 heads: 12.3 -> 6.2 us in a decode step's chain.
template <int NA>      // head sizes up to 64 NA
__global__ void __launch_bounds__(128)
attention_f32_single_kernel(const F32Args a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float scores[2][64], pw[2][32];
  pdl_launch_dependents();
  const int D = a.D, DP = D + 4, stage_floats = 64 * (DP + D);
  float* qs = smem + 3 * stage_floats;               // [D]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = blockIdx.x, h = blockIdx.y, hk = h / (a.H / a.Hkv);
  const size_t page_elems = (size_t)(a.kv_shared ? 1 : 2) * a.Hkv * a.page_size * D;
  const size_t head_off = (size_t)hk * a.page_size * D, v_off = a.kv_shared ? 0 : (size_t)a.Hkv * a.page_size * D;
  pdl_wait();
  const int pos = a.positions[t];
  const int lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  const int* bt = a.block_table + (size_t)a.token_req[t] * a.bt_stride;
  const int kt_first = lo / 32, n_rounds = (pos / 32 + 1 - kt_first + 1) / 2;
  auto ask = [&](int r) {                             // two threads bring one key and its value
    if (r < n_rounds) {
      float* ks = smem + (r % 3) * stage_floats;
      float* vs = ks + 64 * DP;
      const int j = tid >> 1, p = (kt_first + 2 * r) * 32 + j;
      const float* kp = (p >= lo && p <= pos) ? f32_row(a, bt, p, page_elems, head_off) : nullptr;
      for (int d = (tid & 1) * 4; d < D; d += 8) {
        copy16_or_zero(ks + j * DP + d, kp ? kp + d : a.cache, kp != nullptr);
        copy16_or_zero(vs + j * D + d, kp ? kp + v_off + d : a.cache, kp != nullptr);
      }
    }
    copies_commit();
  };
  auto score = [&](int r) {                           // by warps 2 and 3
    const int j = (warp - 2) * 32 + lane, key = (kt_first + 2 * r) * 32 + j;
    const float* kr = smem + (r % 3) * stage_floats + j * DP;
    float sc = 0.0f;
#pragma unroll 8
    for (int d = 0; d < D; d += 4) {
      const float4 q4 = *reinterpret_cast<const float4*>(qs + d);
      const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
      sc = fmaf(q4.x, k4.x, sc);
      sc = fmaf(q4.y, k4.y, sc);
      sc = fmaf(q4.z, k4.z, sc);
      sc = fmaf(q4.w, k4.w, sc);
    }
    scores[r & 1][j] = (key >= lo && key <= pos) ? sc * a.scale : -INFINITY;
  };
  ask(0);
  ask(1);
  for (int d = tid; d < D; d += 128) qs[d] = a.q[(size_t)t * a.q_stride + (size_t)h * D + d];
  copies_wait<1>();
  __syncthreads();
  if (warp >= 2) score(0);
  float m = -INFINITY, l = 0.0f, acc[NA];
#pragma unroll
  for (int n = 0; n < NA; n++) acc[n] = 0.0f;
  for (int r = 0; r < n_rounds; r++) {
    copies_wait<0>();
    __syncthreads();                                  // round r + 1 has landed, round r's scores are there, stage r - 1 is free
    ask(r + 2);
    if (warp >= 2) {
      if (r + 1 < n_rounds) score(r + 1);
    } else {
      const float* vs = smem + (r % 3) * stage_floats + 64 * DP;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if ((kt_first + 2 * r + u) * 32 > pos) break;
        const float s = scores[r & 1][u * 32 + lane];
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);                             // (first tile: exp(-inf) = 0)
        const float p = s != -INFINITY ? expf(s - m_new) : 0.0f;
        l = l * corr + warp_sum(p);
        m = m_new;
        pw[warp][lane] = p;
        __syncwarp();
        float pj[32];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 p4 = *reinterpret_cast<const float4*>(&pw[warp][j]);
          pj[j] = p4.x; pj[j + 1] = p4.y; pj[j + 2] = p4.z; pj[j + 3] = p4.w;
        }
#pragma unroll
        for (int n = 0; n < NA; n++) {
          const int d = min((warp + 2 * n) * 32 + lane, D - 1);
          float x = acc[n] * corr;
#pragma unroll
          for (int j = 0; j < 32; j++) x = fmaf(pj[j], vs[(u * 32 + j) * D + d], x);
          acc[n] = x;
        }
        __syncwarp();
      }
    }
  }
  if (warp < 2) {
    const float inv = 1.0f / l;
    float* op = a.out + (size_t)t * a.o_stride + (size_t)h * D;
#pragma unroll
    for (int n = 0; n < NA; n++) {
      const int d = (warp + 2 * n) * 32 + lane;
      if (d < D) op[d] = acc[n] * inv;
    }
  }
}

// Which kernel takes a 32-bit launch without extensions: the general one, or one of the two above (the same bits from each).
//   Portions: the kernel of four tokens a warp needs a quarter of the blocks for four times the tokens, so it pays where the
//   general kernel's blocks (eight tokens of a head) would take more than one round of the 444 that run at once, and
//   where a block's tokens belong to few requests, for runs of different requests take turns in a block.  Measured, head
//   sizes 64 and 128, general kernel and this one: one prompt of 128 tokens, 12 heads (192 general blocks) 13.7 and 20.6 us,
//   384 (576) 51.9 and 59.3, 512 (768) 79.8 and 73.3, 1,000 (1,500) 246 and 142; 16 portions of 16 tokens behind 640 keys 77
//   and 131, of 32 149 and 98; two tokens each of 16 requests of 640 keys 133 and 680; 31 single tokens of 640 keys beside a
//   portion of 481 364 and 1,236.  At head size 32 tiles are small: 8 x 120 (1,440) 33 and 36, 2 x 320 (960) 48 and 43.
//   Single tokens: a block of the pipelined kernel is two to three times as fast as a general one, but an SM holds fewer of
//   them (two at head size 64, one beyond, the general kernel's four): it pays as long as its rounds are no more than the
//   general kernel's.  Blocks, head size, keys: 192 / 64 / 140 11.5 and 8.3 us, 384 / 64 / 140 12.8 and 14.8, 768 / 64 / 140
//   26.5 and 21.8, 3,072 / 64 / 140 72.9 and 77.2; 128 / 128 / 140 14.4 and 8.7, 384 / 128 / 140 18.3 and 24.5, 2,048 / 128 /
//   140 77.5 and 128; 3,072 / 32 / 140 57.7 and 39.6.
// n_portions: how many requests the tokens belong to where each brings several (0: not known, or single tokens among
// them).
enum { F32_GENERAL = 0, F32_PORTIONS = 1, F32_SINGLES = 2 };
static size_t f32_single_smem(int D) { return ((size_t)3 * 64 * (2 * D + 4) + D) * sizeof(float); }
static int f32_form(int T, int H, int D, int max_q_len, int n_portions) {
  if (D % 4 != 0 || D > 128) return F32_GENERAL;
  if (max_q_len <= 1) {
    const long long blocks = (long long)T * H;
    const int here = (int)(228 * 1024 / (f32_single_smem(D) + 1024));            // blocks an SM holds
    const long long rounds = (blocks + 148 * here - 1) / (148 * here), general = (blocks + 591) / 592;
    return here >= 4 || rounds == 1 || (here >= 2 && rounds <= 3 && rounds * here < general * 4) ? F32_SINGLES : F32_GENERAL;
  }
  const long long blocks = (long long)((T + 7) / 8) * H;
  if (n_portions <= 0 || (T + FP_W - 1) / FP_W > 65535) return F32_GENERAL;
  return (D >= 64 ? blocks >= 640 && T >= 32 * n_portions : blocks >= 960 && T >= 160 * n_portions) ? F32_PORTIONS : F32_GENERAL;
}
SGLC_API int sglc_attention_f32_form(int T, int H, int D, int max_q_len, int n_portions) {
  return f32_form(T, H, D, max_q_len, n_portions);
}

template <void (*KERNEL)(const F32Args)>
static int launch_f32(dim3 grid, int threads, size_t smem, const F32Args& a, cudaStream_t stream) {
  static size_t configured = 48 * 1024;
  if (smem > configured) {
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = smem;
  }
  return sglc_launch(KERNEL, grid, dim3(threads), smem, stream, 1, true, a);
}

// q: first query element of token 0 (rows q_stride apart, heads side by side); cache: one
// layer's pages; block_table: [n_requests][bt_stride] page ids; token_req[t]: row of the
// block table for token t; positions[t]: absolute position of token t (its own key is the
// last one it sees); out: [T][o_stride].  max_keys: the most keys any token of this launch
// sees.  q/out dtype = act_dtype, cache dtype = cache_dtype.  n_pages and err serve the
// bounds-check build (page ids are compared with n_pages; err gets the flag).  max_q_len: the
// longest portion of the step (1: every request brings one token, and a block takes one token); n_portions:
// see f32_form.
static int attention_simt_run(const void* q, int q_stride, const void* cache,
                              const int* block_table, int bt_stride, const int* token_req,
                              const int* positions, void* out, int o_stride, int T, int H,
                              int Hkv, int D, int page_size, float scale, int window,
                              int max_keys, int act_dtype, int cache_dtype, int n_pages, int* err,
                              int max_q_len, int n_portions, int kv_shared, cudaStream_t stream, bool ext = false, int DV = 0,
                              int chunk = 0, const float* sinks = nullptr, int n_splits = 1, float* part_ws = nullptr,
                              OutGate gate = OutGate{nullptr, 0, 0}) {
  if (T <= 0) return SGLC_OK;
  if (!ext) DV = D;
  if (DV <= 0 || chunk < 0 || (kv_shared && DV > D)) return SGLC_ERR_ARGUMENT;
  if (DV > (ext ? 768 : 256)) return SGLC_ERR_UNSUPPORTED;
  if (H <= 0 || Hkv <= 0 || H % Hkv != 0 || D <= 0 || page_size <= 0 || max_keys <= 0)
    return SGLC_ERR_ARGUMENT;
  if (H > 65535 || D > (ext ? 768 : 256)) return SGLC_ERR_UNSUPPORTED;
  // single tokens of many requests share nothing: a token a block; portions: eight tokens a block
  const bool single = max_q_len <= 1;
  const int form = !ext && act_dtype == SGLC_F32 && cache_dtype == SGLC_F32 && ((uintptr_t)cache & 15) == 0
                       ? f32_form(T, H, D, max_q_len, n_portions) : F32_GENERAL;
  if (form != F32_GENERAL) {
    F32Args a = {};
    a.q = (const float*)q; a.q_stride = q_stride; a.cache = (const float*)cache; a.block_table = block_table;
    a.bt_stride = bt_stride; a.token_req = token_req; a.positions = positions; a.out = (float*)out; a.o_stride = o_stride;
    a.T = T; a.H = H; a.Hkv = Hkv; a.D = D; a.page_size = page_size; a.scale = scale; a.window = window;
    a.n_pages = n_pages; a.kv_shared = kv_shared; a.err = err;
    if (form == F32_SINGLES)
      return D <= 64 ? launch_f32<attention_f32_single_kernel<1>>(dim3(T, H), 128, f32_single_smem(D), a, stream)
                     : launch_f32<attention_f32_single_kernel<2>>(dim3(T, H), 128, f32_single_smem(D), a, stream);
    const size_t smem = ((size_t)2 * 32 * (2 * D + 4) + (size_t)FP_W * (D + 32)) * sizeof(float);
    const dim3 grid(H, (T + FP_W - 1) / FP_W);
    return D <= 64 ? launch_f32<attention_f32_portion_kernel<2>>(grid, 256, smem, a, stream)
                   : launch_f32<attention_f32_portion_kernel<4>>(grid, 256, smem, a, stream);
  }
  const int W = single ? 1 : 8;
  const size_t smem = ((size_t)32 * (D % 4 == 0 ? D + 4 : D + 1) + (size_t)32 * DV + (size_t)W * D + (size_t)W * 32) * sizeof(float);
  if (smem > 224 * 1024) return SGLC_ERR_UNSUPPORTED;
  if (part_ws && (!ext || !single || n_splits < 1 || n_splits > 32)) return SGLC_ERR_ARGUMENT;
  dim3 grid((T + W - 1) / W, H, part_ws ? n_splits : 1);
  // single tokens whose shares are merged afterwards: where 2 to 8 query heads share a key/value
  // head, a block takes them all (the eight-warp form, its warps being heads of one token)
  int head_rows = (part_ws && H / Hkv >= 2 && H / Hkv <= 8) ? 1 : 0;
  const size_t smem_rows = ((size_t)32 * (D % 4 == 0 ? D + 4 : D + 1) + (size_t)32 * DV + (size_t)8 * D + (size_t)8 * 32) * sizeof(float);
  if (smem_rows > 224 * 1024) head_rows = 0;
  const bool wide_v = DV > 256;
  if (head_rows) {
    const dim3 grid_rows(T, Hkv, n_splits);
#define LAUNCH_RN(TQ, TC, TO, NA)                                                                      \
  do {                                                                                                 \
    if (smem_rows > 48 * 1024)                                                                         \
      cudaFuncSetAttribute(attention_simt_kernel<TQ, TC, TO, 8, 256, true, NA>,                        \
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_rows);               \
    attention_simt_kernel<TQ, TC, TO, 8, 256, true, NA><<<grid_rows, 256, smem_rows, stream>>>(        \
        (const TQ*)q, q_stride, (const TC*)cache, block_table, bt_stride, token_req, positions,        \
        (TO*)out, o_stride, T, H, Hkv, D, page_size, scale, window, n_pages, err, kv_shared, DV,       \
        chunk, sinks, n_splits, part_ws, 1, gate);                                                     \
  } while (0)
#define LAUNCH_R(TQ, TC, TO)                                                                           \
  do {                                                                                                 \
    if (wide_v) LAUNCH_RN(TQ, TC, TO, 24);                                                             \
    else LAUNCH_RN(TQ, TC, TO, 8);                                                                     \
  } while (0)
    if (act_dtype == SGLC_F32 && cache_dtype == SGLC_F32) LAUNCH_R(float, float, float);
    else if (act_dtype == SGLC_BF16 && cache_dtype == SGLC_BF16) LAUNCH_R(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else return SGLC_ERR_ARGUMENT;
#undef LAUNCH_R
#undef LAUNCH_RN
    return sglc_launch_status();
  }
#define LAUNCH_E(TQ, TC, TO, WW, TH, EX, NA)                                                           \
  do {                                                                                                 \
    if (smem > 48 * 1024)                                                                              \
      cudaFuncSetAttribute(attention_simt_kernel<TQ, TC, TO, WW, TH, EX, NA>,                          \
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                    \
    attention_simt_kernel<TQ, TC, TO, WW, TH, EX, NA><<<grid, TH, smem, stream>>>(                      \
        (const TQ*)q, q_stride, (const TC*)cache, block_table, bt_stride, token_req, positions,        \
        (TO*)out, o_stride, T, H, Hkv, D, page_size, scale, window, n_pages, err, kv_shared, DV,       \
        chunk, sinks, n_splits, part_ws, 0, gate);                                                     \
  } while (0)
#define LAUNCH(TQ, TC, TO, WW, TH)                                                                     \
  do {                                                                                                 \
    if (ext && wide_v) LAUNCH_E(TQ, TC, TO, WW, TH, true, 24);                                         \
    else if (ext) LAUNCH_E(TQ, TC, TO, WW, TH, true, 8);                                               \
    else LAUNCH_E(TQ, TC, TO, WW, TH, false, 8);                                                       \
  } while (0)
  if (act_dtype == SGLC_F32 && cache_dtype == SGLC_F32) {
    if (single) LAUNCH(float, float, float, 1, 128);
    else LAUNCH(float, float, float, 8, 256);
  } else if (act_dtype == SGLC_BF16 && cache_dtype == SGLC_BF16) {
    if (single) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16, 1, 128);
    else LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16, 8, 256);
  } else {
    return SGLC_ERR_ARGUMENT;
  }
#undef LAUNCH
#undef LAUNCH_E
  return sglc_launch_status();
}

SGLC_API int sglc_attention_simt(const void* q, int q_stride, const void* cache,
                                 const int* block_table, int bt_stride, const int* token_req,
                                 const int* positions, void* out, int o_stride, int T, int H,
                                 int Hkv, int D, int page_size, float scale, int window,
                                 int max_keys, int act_dtype, int cache_dtype, int n_pages, int* err,
                                 int max_q_len, int n_portions, cudaStream_t stream) {
  return attention_simt_run(q, q_stride, cache, block_table, bt_stride, token_req, positions, out, o_stride,
                            T, H, Hkv, D, page_size, scale, window, max_keys, act_dtype, cache_dtype,
                            n_pages, err, max_q_len, n_portions, 0, stream);
}

// The same over a cache whose pages hold one block of rows [Hkv][page_size][D] that serve as keys
// and as values (attention over a latent that both are read from): cache [n_pages][1][Hkv][page_size][D].
SGLC_API int sglc_attention_simt_shared(const void* q, int q_stride, const void* cache,
                                        const int* block_table, int bt_stride, const int* token_req,
                                        const int* positions, void* out, int o_stride, int T, int H,
                                        int Hkv, int D, int page_size, float scale, int window,
                                        int max_keys, int act_dtype, int cache_dtype, int n_pages, int* err,
                                        int max_q_len, int n_portions, cudaStream_t stream) {
  return attention_simt_run(q, q_stride, cache, block_table, bt_stride, token_req, positions, out, o_stride,
                            T, H, Hkv, D, page_size, scale, window, max_keys, act_dtype, cache_dtype,
                            n_pages, err, max_q_len, n_portions, 1, stream);
}

// The extended form: values of size DV beside keys of size D (cache [n_pages][Hkv x page_size x D keys |
// Hkv x page_size x DV values]; out rows hold H heads of DV), `chunk` > 0: a query sees the keys of its
// own chunk of so many positions only; `sinks` (float [H] or null): a score per head that joins the
// softmax's denominator.
// kv_shared: the cache's pages hold one block of rows [Hkv][page_size][D] that are keys, and whose first
// DV entries are values.  gate (float, rows gate_stride apart, or null): the heads' results are
// multiplied by its sigmoid, one number per head (gate_per_head) or one per entry.
SGLC_API int sglc_attention_simt_ext(const void* q, int q_stride, const void* cache,
                                     const int* block_table, int bt_stride, const int* token_req,
                                     const int* positions, void* out, int o_stride, int T, int H,
                                     int Hkv, int D, int DV, int page_size, float scale, int window, int chunk,
                                     const float* sinks, int max_keys, int act_dtype, int cache_dtype, int n_pages,
                                     int* err, int max_q_len, int kv_shared, const float* gate, long long gate_stride,
                                     int gate_per_head, cudaStream_t stream) {
  return attention_simt_run(q, q_stride, cache, block_table, bt_stride, token_req, positions, out, o_stride,
                            T, H, Hkv, D, page_size, scale, window, max_keys, act_dtype, cache_dtype,
                            n_pages, err, max_q_len, 0, kv_shared, stream, true, DV, chunk, sinks, 1, nullptr,
                            OutGate{gate, gate_stride, gate_per_head});
}

// The merge behind a launch that dealt a token's keys to several blocks (a step of single tokens):
// the shares' maxima, sums and unnormalised results [T][H][n_splits][DV + 2] become the head's
// result, the sink (if any) joining the denominator once.  A warp 32 entries of a (token, head), the first
// eight shares' on their way beside the maxima and sums: one round trip instead of one a 32 entries (8 tokens, 12
// heads of 64, 5 shares in a decode step 4.1 -> 2.6 us).
constexpr int MERGE_SHARES = 8;
template <typename TO>
__global__ void __launch_bounds__(128)
attention_merge_kernel(const float* part_ws, int n_splits, const float* __restrict__ sinks, TO* __restrict__ out, int o_stride,
                       int T, int H, int DV, const OutGate gate) {
  pdl_launch_dependents();
  const int chunks = (DV + 31) / 32;
  const long long at = (long long)blockIdx.x * 4 + (threadIdx.x >> 5), item = at / chunks;
  const int lane = threadIdx.x & 31, d = (int)(at % chunks) * 32 + lane;
  pdl_wait();
  if (item >= (long long)T * H) return;
  const int t = (int)(item / H), h = (int)(item % H);
  const bool by_entry = gate.z && !gate.per_head;
  const float* rec = part_ws + (size_t)item * n_splits * (DV + 2);
  float v[MERGE_SHARES];
#pragma unroll
  for (int j = 0; j < MERGE_SHARES; j++) v[j] = j < n_splits && d < DV ? rec[(size_t)j * (DV + 2) + 2 + d] : 0.0f;
  // lane s holds share s's maximum and sum (an empty share: -inf and 0, its results zero)
  const float ms = lane < n_splits ? rec[(size_t)lane * (DV + 2)] : -INFINITY;
  const float ls = lane < n_splits ? rec[(size_t)lane * (DV + 2) + 1] : 0.0f;
  const float sk = sinks ? sinks[h] : -INFINITY;
  const float z_head = gate.z && gate.per_head ? gate.z[t * gate.stride + h] : 0.0f;
  const float z = by_entry && d < DV ? gate.z[t * gate.stride + (long long)h * DV + d] : 0.0f;
  const float M = fmaxf(warp_max(ls > 0.0f ? ms : -INFINITY), sk);
  const float f = ls > 0.0f ? expf(ms - M) : 0.0f;
  const float L = warp_sum(ls * f) + (sinks ? expf(sk - M) : 0.0f);
  float inv = 1.0f / L;
  if (gate.z && gate.per_head) inv *= 1.0f / (1.0f + expf(-z_head));
  float o = 0.0f;
  for (int s0 = 0; s0 < n_splits; s0 += MERGE_SHARES) {
    if (s0 > 0) {
#pragma unroll
      for (int j = 0; j < MERGE_SHARES; j++)
        v[j] = s0 + j < n_splits && d < DV ? rec[(size_t)(s0 + j) * (DV + 2) + 2 + d] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < MERGE_SHARES; j++)
      if (s0 + j < n_splits) o = fmaf(v[j], __shfl_sync(0xffffffffu, f, s0 + j), o);
  }
  o *= inv;
  if (by_entry) o *= 1.0f / (1.0f + expf(-z));
  if (d < DV) out[(size_t)t * o_stride + (size_t)h * DV + d] = from_f32<TO>(o);
}

// The extended form for a step of single tokens with each token's keys dealt to n_splits blocks:
// part_ws holds T x H x n_splits x (DV + 2) floats; two launches (the shares, then the merge).
SGLC_API int sglc_attention_simt_ext_split(const void* q, int q_stride, const void* cache,
                                           const int* block_table, int bt_stride, const int* token_req,
                                           const int* positions, void* out, int o_stride, int T, int H,
                                           int Hkv, int D, int DV, int page_size, float scale, int window, int chunk,
                                           const float* sinks, int max_keys, int act_dtype, int cache_dtype,
                                           int n_pages, int* err, int kv_shared, const float* gate,
                                           long long gate_stride, int gate_per_head, int n_splits, float* part_ws,
                                           cudaStream_t stream) {
  if (T <= 0) return SGLC_OK;
  if (!part_ws || n_splits < 1) return SGLC_ERR_ARGUMENT;
  const int code = attention_simt_run(q, q_stride, cache, block_table, bt_stride, token_req, positions, out, o_stride,
                                      T, H, Hkv, D, page_size, scale, window, max_keys, act_dtype, cache_dtype,
                                      n_pages, err, 1, 0, kv_shared, stream, true, DV, chunk, nullptr, n_splits, part_ws);
  if (code != SGLC_OK) return code;
  const dim3 grid((unsigned)(((long long)T * H * ((DV + 31) / 32) + 3) / 4));
  const OutGate g{gate, gate_stride, gate_per_head};
  if (act_dtype == SGLC_F32)
    return sglc_launch(attention_merge_kernel<float>, grid, dim3(128), 0, stream, 1, true, (const float*)part_ws,
                       n_splits, sinks, (float*)out, o_stride, T, H, DV, g);
  return sglc_launch(attention_merge_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, 1, true,
                     (const float*)part_ws, n_splits, sinks, (__nv_bfloat16*)out, o_stride, T, H, DV, g);
}
