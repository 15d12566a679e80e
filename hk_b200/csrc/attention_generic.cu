// Generic attention over the paged cache, for every head size, group size and window, in
// float (the true 32-bit path) or bf16 storage with fp32 arithmetic.
//
// One block per (token, query head).  The token at position p of request slot s reads keys
// j in [max(0, p - window + 1), p] (window <= 0: all of [0, p]) through the slot's block table;
// its own key was written by the cache-write kernel earlier in the same step.  Four warps take
// the keys round-robin, each keeping an online softmax state (max, sum, weighted values); the
// four states are merged in a fixed order.  Nothing depends on which other tokens are in the
// batch, so the result at a position is the same under every way of cutting the work.  In float, heads and values of up
// to 128 take `attention_f32_kernel` further down (a block per run of a request's rows and key head), with the same promise.
// Values may have another width than keys (`vd`: pages [page][G][page_tokens][vd], out [n, H * vd]).  With
// `sink` = 1 the softmax has one more term in its denominator, a key whose score is 0 and that has no value:
// p_j = exp(s_j) / (1 + sum exp(s_j)); with `sinks` (one float per query head) that key's score is sinks[h] instead of 0.
// Further options, each off at 0 or null:
//   softcap c   a score becomes c * tanh(score / c) before the softmax;
//   chunk s     a token also sees no key before the start of its own block of s positions, (p / s) * s, counted from
//               position 0 of the request;
//   v_stride    elements between the values of consecutive tokens of a page; when it is not vd the values lie inside
//               wider rows: a cache that keeps ONE tensor per token whose first vd dims are the value (v_pages = k_pages,
//               v_stride = hd);
//   dist        float [H, dist_n]: the score of a key n positions back is raised by dist[h, min(n, dist_n - 1)] (behind the
//               scale and the cap; a bias learned per distance, the last entry standing for all further ones);
//   gate        fp32 logits [n, gate_ld >= H * vd]: the output is multiplied by gate_scale * sigmoid(gate[t, h * vd + d]).
//
// Reference counterpart: `attention`, src/cuda_device.zig:1494-1594 (block per (token, head),
// warp per position, online softmax); scale on q first: src/engine/attention_kernel.zig:109.
#include <math_constants.h>

#include "common.cuh"

#define AG_WARPS 4

struct AgOptions {
  float softcap;
  int chunk;
  int v_stride;
  const float* sinks;
  const float* gate;
  long long gate_ld;
  float gate_scale;
  const float* dist;
  int dist_n;
};

// AG_MAX_PER_LANE: dims per lane, 8 for widths up to 256, 20 up to 640
template <typename T, int AG_MAX_PER_LANE>
__global__ void __launch_bounds__(AG_WARPS * 32)
attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pages,
                         const T* __restrict__ v_pages, const int* __restrict__ block_table,
                         int table_stride, const int* __restrict__ positions,
                         const int* __restrict__ slot_of_token, T* __restrict__ out, int H, int G, int hd,
                         int page_tokens, int window, float scale, int vd, int sink, AgOptions opt) {
  extern __shared__ float smem[];  // [AG_WARPS][vd] values, then [AG_WARPS] max, [AG_WARPS] sum
  float* acc_s = smem;
  float* m_s = smem + AG_WARPS * vd;
  float* l_s = m_s + AG_WARPS;

  int t = blockIdx.x / H, h = blockIdx.x % H;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int g = h / (H / G);
  int pos = positions[t];
  const int* bt = block_table + (size_t)slot_of_token[t] * table_stride;
  int lo = window > 0 ? max(0, pos - window + 1) : 0;
  if (opt.chunk > 0) lo = max(lo, (pos / opt.chunk) * opt.chunk);
  const float cap = opt.softcap, inv_cap = opt.softcap > 0.f ? 1.0f / opt.softcap : 0.f;

  float qr[AG_MAX_PER_LANE], acc[AG_MAX_PER_LANE];
  const T* qp = q + ((size_t)t * H + h) * hd;
#pragma unroll
  for (int i = 0; i < AG_MAX_PER_LANE; ++i) {
    int d = lane + 32 * i;
    qr[i] = d < hd ? to_f32<T>(qp[d]) * scale : 0.f;
    acc[i] = 0.f;
  }
  float m = -CUDART_INF_F, l = 0.f;
  for (int j = lo + wid; j <= pos; j += AG_WARPS) {
    int page = bt[j / page_tokens];
    if (page < 0) continue;  // never scheduled by the host; keeps the reads in bounds
    const size_t at = ((size_t)page * G + g) * page_tokens + (j % page_tokens);
    const T* kp = k_pages + at * hd;
    const T* vp = v_pages + at * opt.v_stride;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < AG_MAX_PER_LANE; ++i) {
      int d = lane + 32 * i;
      if (d < hd) s = fmaf(qr[i], to_f32<T>(kp[d]), s);
    }
    s = warp_sum(s);
    if (cap > 0.f) s = cap * tanhf(s * inv_cap);
    if (opt.dist) s += opt.dist[(size_t)h * opt.dist_n + min(pos - j, opt.dist_n - 1)];
    float mn = fmaxf(m, s);
    float corr = expf(m - mn);
    float p = expf(s - mn);
    l = l * corr + p;
#pragma unroll
    for (int i = 0; i < AG_MAX_PER_LANE; ++i) {
      int d = lane + 32 * i;
      if (d < vd) acc[i] = acc[i] * corr + p * to_f32<T>(vp[d]);
    }
    m = mn;
  }
#pragma unroll
  for (int i = 0; i < AG_MAX_PER_LANE; ++i) {
    int d = lane + 32 * i;
    if (d < vd) acc_s[wid * vd + d] = acc[i];
  }
  if (lane == 0) {
    m_s[wid] = m;
    l_s[wid] = l;
  }
  __syncthreads();
  const float sink_score = sink && opt.sinks ? opt.sinks[h] : 0.f;
  float mm = sink ? sink_score : m_s[0];   // the sink's score takes part in the maximum
#pragma unroll
  for (int w = sink ? 0 : 1; w < AG_WARPS; ++w) mm = fmaxf(mm, m_s[w]);
  float f[AG_WARPS], lt = 0.f;
#pragma unroll
  for (int w = 0; w < AG_WARPS; ++w) {
    f[w] = m_s[w] == -CUDART_INF_F ? 0.f : expf(m_s[w] - mm);
    lt += l_s[w] * f[w];
  }
  if (sink) lt += expf(sink_score - mm);
  T* op = out + ((size_t)t * H + h) * vd;
  for (int d = threadIdx.x; d < vd; d += blockDim.x) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < AG_WARPS; ++w) a += acc_s[w * vd + d] * f[w];
    a /= lt;
    if (opt.gate) a = a * opt.gate_scale / (1.0f + expf(-opt.gate[(size_t)t * opt.gate_ld + (size_t)h * vd + d]));
    op[d] = from_f32<T>(a);
  }
}

template <typename T, int PER>
static int ag_launch(const void* q, const void* k_pages, const void* v_pages, const int* block_table, int table_stride,
                     const int* positions, const int* slot_of_token, void* out, int n, int H, int G, int hd, int page_tokens,
                     int window, float scale, int vd, int sink, AgOptions opt, cudaStream_t s) {
  size_t smem = (size_t)(AG_WARPS * vd + 2 * AG_WARPS) * sizeof(float);
  unsigned blocks = (unsigned)((long long)n * H);
  attention_generic_kernel<T, PER><<<blocks, AG_WARPS * 32, smem, s>>>(
      (const T*)q, (const T*)k_pages, (const T*)v_pages, block_table, table_stride, positions, slot_of_token, (T*)out, H, G, hd,
      page_tokens, window, scale, vd, sink, opt);
  return hk_launch_status();
}

HK_API int hk_attention_generic(const void* q, const void* k_pages, const void* v_pages, int dtype,
                                const int* block_table, int table_stride, const int* positions,
                                const int* slot_of_token, void* out, int n, int H, int G, int hd,
                                int page_tokens, int window, float scale, int vd, int sink, const float* sinks, float softcap,
                                int chunk, int v_stride, const float* gate, long long gate_ld, float gate_scale, const float* dist,
                                int dist_n, void* stream) {
  if (n <= 0) return 0;
  const int widest = hd > vd ? hd : vd;
  if (widest > 640 || hd < 1 || G < 1 || H % G != 0 || vd < 1 || v_stride < vd || softcap < 0.f || chunk < 0 ||
      (dist && dist_n < 1))
    return HK_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  AgOptions opt = {softcap, chunk, v_stride, sinks, gate, gate_ld, gate_scale, dist, dist_n};
  if (dtype != HK_F32 && dtype != HK_BF16) return HK_ERR_UNSUPPORTED;
#define AG_GO(T, PER) ag_launch<T, PER>(q, k_pages, v_pages, block_table, table_stride, positions, slot_of_token, out, n, H, G, hd, \
                                        page_tokens, window, scale, vd, sink, opt, s)
  if (widest <= 256) return dtype == HK_F32 ? AG_GO(float, 8) : AG_GO(bf16, 8);
  return dtype == HK_F32 ? AG_GO(float, 20) : AG_GO(bf16, 20);
#undef AG_GO
}

// ------------------------------------------------------------------ float32, in runs of tokens
// The same attention in float: a block takes an item {first query row, query tokens, slot,
// position of the first} for one key/value head, 32 rows = (token, head of the group) pairs, so 64 keys at a time are read once
// for all of them.  Scores and sums are register tiles of multiply-adds over 16-byte loads of shared memory (4 x 4 scores a thread
// along the head's dims, 4 x 8 sums); the next tile's keys arrive while this one's probabilities are made, the next values while
// the next scores are.  Every option of the kernel above.  A row's result is the same to the bit whatever run it stands in, also
// beside rows that are not finite: a tile with keys that some row does not see looks for NaN and Inf among its values (a
// probability of zero would not keep them out) and, if there are any, adds for every row the keys that it sees alone.  Up
// to 8 rows (single tokens) do a quarter of the arithmetic.  Bound by what shared memory delivers (two thirds of the fp32 rate).
// 16 heads of 128 over 8, us, the kernel above and this: 509 tokens 484 and 139; single tokens behind 2,000: one 415 and 360, 64 (32
// heads) 1,697 and 869; 2,048 tokens of 32 heads 13,658 and 2,040 (2,018 without the look at the values).
namespace {
constexpr int AF_ROWS = 32, AF_KEYS = 64, AF_HD = 128, AF_LD = AF_HD + 4, AF_LDP = AF_KEYS + 4, AF_TH = 128;
struct AfItem {
  int q_row0, n_tokens, slot, pos0;
};
struct AfSmem {
  float q[AF_ROWS * AF_LD], k[AF_KEYS * AF_LD], v[AF_KEYS * AF_LD], p[AF_ROWS * AF_LDP];
  float corr[AF_ROWS], inv[AF_ROWS];
  int page_ok[AF_KEYS];
};
__device__ __forceinline__ void af_copy16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
}  // namespace

// RI: rows a thread (8 RI rows of the tile are worked on).
template <int RI>
__device__ __forceinline__ void attention_f32_item(AfSmem& sm, const AfItem it, const int g, const float* __restrict__ q,
                                                   const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                                                   const int* __restrict__ block_table, int table_stride, float* __restrict__ out, int H, int G,
                                                   int hd, int page_tokens, int window, float scale, int vd, int sink, const AgOptions& opt) {
  const int group = H / G, rows = it.n_tokens * group;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int* bt = block_table + (size_t)it.slot * table_stride;
  auto first_key = [&](int pos) {
    int lo = window > 0 ? max(0, pos - window + 1) : 0;
    return opt.chunk > 0 ? max(lo, (pos / opt.chunk) * opt.chunk) : lo;
  };
  // tiles lie at multiples of 64 keys, so that a row's sums are cut in the same places whatever run it is in
  const int kv_lo = first_key(it.pos0) / AF_KEYS * AF_KEYS, kv_hi = it.pos0 + it.n_tokens;
  const int tiles = (kv_hi - kv_lo + AF_KEYS - 1) / AF_KEYS;
  // a tile's keys or values: a key's row in 32 pieces of 16 bytes, what does not exist as zeros
  auto fetch = [&](const float* pages, float* dst, int tile, int width, size_t stride) {
    for (int e = tid; e < AF_KEYS * (AF_HD / 4); e += AF_TH) {
      const int r = e / (AF_HD / 4), d = (e % (AF_HD / 4)) * 4, j = kv_lo + tile * AF_KEYS + r;
      const int page = j < kv_hi ? bt[j / page_tokens] : -1;
      const bool in = page >= 0 && d < width;
      const float* src = in ? pages + (((size_t)page * G + g) * page_tokens + (j % page_tokens)) * stride + d : pages;
      af_copy16(dst + r * AF_LD + d, src, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(k_pages, sm.k, 0, hd, hd);
  fetch(v_pages, sm.v, 0, vd, opt.v_stride);
  for (int e = tid; e < 8 * RI * (AF_HD / 4); e += AF_TH) {
    const int r = e / (AF_HD / 4), d = (e % (AF_HD / 4)) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows && d < hd) {
      x = *reinterpret_cast<const float4*>(q + ((size_t)(it.q_row0 + r / group) * H + g * group + r % group) * hd + d);
      x = make_float4(x.x * scale, x.y * scale, x.z * scale, x.w * scale);
    }
    *reinterpret_cast<float4*>(sm.q + r * AF_LD + d) = x;
  }
  const float cap = opt.softcap, inv_cap = cap > 0.f ? 1.0f / cap : 0.f;
  // the softmax's state of row tid / 4, alike in its four threads
  const int sr = tid >> 2, sc = (tid & 3) * 16;
  float m = -CUDART_INF_F, l = 0.f;
  float4 acc[RI][2];
#pragma unroll
  for (int i = 0; i < RI; ++i) acc[i][0] = acc[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int t = 0; t < tiles; ++t) {
    const int j0 = kv_lo + t * AF_KEYS;
    if (tid < AF_KEYS) sm.page_ok[tid] = j0 + tid < kv_hi && bt[(j0 + tid) / page_tokens] >= 0;
    asm volatile("cp.async.wait_group 1;" ::: "memory");          // the keys
    __syncthreads();
    float s[RI][4];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
    for (int d = 0; d < hd; d += 4) {
      float4 a[RI], b[4];
#pragma unroll
      for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(sm.q + (ty + 8 * i) * AF_LD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(sm.k + (tx + 16 * j) * AF_LD + d);
#pragma unroll
      for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int r = ty + 8 * i, pos = it.pos0 + r / group, lo = first_key(pos), h = g * group + r % group;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = j0 + tx + 16 * j;
        float x = s[i][j];
        if (cap > 0.f) x = cap * tanhf(x * inv_cap);
        const bool see = r < rows && key >= lo && key <= pos && sm.page_ok[tx + 16 * j];
        if (opt.dist && see) x += opt.dist[(size_t)h * opt.dist_n + min(pos - key, opt.dist_n - 1)];
        sm.p[r * AF_LDP + tx + 16 * j] = see ? x : -CUDART_INF_F;
      }
    }
    __syncthreads();
    if (t + 1 < tiles) fetch(k_pages, sm.k, t + 1, hd, hd);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    if (sr < 8 * RI) {           // a whole warp or none
      float* row = sm.p + sr * AF_LDP + sc;
      float4 x[4];
      float top = -CUDART_INF_F;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = *reinterpret_cast<const float4*>(row + 4 * e);
        top = fmaxf(top, fmaxf(fmaxf(x[e].x, x[e].y), fmaxf(x[e].z, x[e].w)));
      }
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float mn = fmaxf(m, top), safe = mn == -CUDART_INF_F ? 0.f : mn;
      const float corr = expf(m - safe);                          // m = -inf: 0
      float sum = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = make_float4(expf(x[e].x - safe), expf(x[e].y - safe), expf(x[e].z - safe), expf(x[e].w - safe));
        sum += (x[e].x + x[e].y) + (x[e].z + x[e].w);
        *reinterpret_cast<float4*>(row + 4 * e) = x[e];
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      l = fmaf(l, corr, sum);
      m = mn;
      if ((tid & 3) == 0) sm.corr[sr] = corr;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");          // the values
    bool apart = false;                                           // NaN or Inf among values that some row does not see
    if (j0 < first_key(it.pos0 + it.n_tokens - 1) || j0 + AF_KEYS - 1 > it.pos0) {
      float odd = 0.f;                                            // NaN if one of the pieces that this thread fetched holds any
#pragma unroll 4
      for (int e = tid; e < AF_KEYS * (AF_HD / 4); e += AF_TH) {
        const float4 x = *reinterpret_cast<const float4*>(sm.v + (e / (AF_HD / 4)) * AF_LD + (e % (AF_HD / 4)) * 4);
        odd = fmaf(x.x, 0.f, fmaf(x.y, 0.f, fmaf(x.z, 0.f, fmaf(x.w, 0.f, odd))));
      }
      apart = __syncthreads_or(odd != 0.f);
    } else {
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const float c = sm.corr[ty + 8 * i];
#pragma unroll
      for (int b = 0; b < 2; ++b) acc[i][b] = make_float4(acc[i][b].x * c, acc[i][b].y * c, acc[i][b].z * c, acc[i][b].w * c);
    }
    if (!apart) {
#pragma unroll 2
      for (int c = 0; c < AF_KEYS; c += 4) {
        float4 p[RI];
#pragma unroll
        for (int i = 0; i < RI; ++i) p[i] = *reinterpret_cast<const float4*>(sm.p + (ty + 8 * i) * AF_LDP + c);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 v0 = *reinterpret_cast<const float4*>(sm.v + (c + e) * AF_LD + 4 * tx);
          const float4 v1 = *reinterpret_cast<const float4*>(sm.v + (c + e) * AF_LD + 64 + 4 * tx);
#pragma unroll
          for (int i = 0; i < RI; ++i) {
            const float w = e == 0 ? p[i].x : e == 1 ? p[i].y : e == 2 ? p[i].z : p[i].w;
            acc[i][0] = make_float4(fmaf(w, v0.x, acc[i][0].x), fmaf(w, v0.y, acc[i][0].y), fmaf(w, v0.z, acc[i][0].z), fmaf(w, v0.w, acc[i][0].w));
            acc[i][1] = make_float4(fmaf(w, v1.x, acc[i][1].x), fmaf(w, v1.y, acc[i][1].y), fmaf(w, v1.z, acc[i][1].z), fmaf(w, v1.w, acc[i][1].w));
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        const int r = ty + 8 * i, pos = it.pos0 + r / group;
#pragma unroll 1
        for (int c = max(0, first_key(pos) - j0); c < min(AF_KEYS, pos + 1 - j0); ++c) {
          const float w = sm.p[r * AF_LDP + c];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const float4 x = *reinterpret_cast<const float4*>(sm.v + c * AF_LD + 64 * b + 4 * tx);
            acc[i][b] = make_float4(fmaf(w, x.x, acc[i][b].x), fmaf(w, x.y, acc[i][b].y), fmaf(w, x.z, acc[i][b].z), fmaf(w, x.w, acc[i][b].w));
          }
        }
      }
    }
    __syncthreads();
    if (t + 1 < tiles) fetch(v_pages, sm.v, t + 1, vd, opt.v_stride);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if ((tid & 3) == 0 && sr < 8 * RI) {
    float scale_by = 1.f;
    if (sink && sr < rows) {                                      // one more term of the denominator, a key without a value
      const float score = opt.sinks ? opt.sinks[g * group + sr % group] : 0.f, mm = fmaxf(m, score);
      scale_by = expf(m - mm);
      l = fmaf(l, scale_by, expf(score - mm));
    }
    sm.inv[sr] = l > 0.f ? scale_by / l : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = ty + 8 * i;
    if (r >= rows) continue;
    const size_t row = (size_t)it.q_row0 + r / group;
    const int h = g * group + r % group;
    const float inv = sm.inv[r];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int d = 64 * b + 4 * tx;
      if (d >= vd) continue;
      float y[4] = {acc[i][b].x * inv, acc[i][b].y * inv, acc[i][b].z * inv, acc[i][b].w * inv};
      if (opt.gate)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = y[e] * opt.gate_scale / (1.0f + expf(-opt.gate[row * opt.gate_ld + (size_t)h * vd + d + e]));
      *reinterpret_cast<float4*>(out + (row * H + h) * vd + d) = make_float4(y[0], y[1], y[2], y[3]);
    }
  }
}

__global__ void __launch_bounds__(AF_TH, 2)
attention_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                     const int* __restrict__ block_table, int table_stride, const AfItem* __restrict__ items, float* __restrict__ out, int H,
                     int G, int hd, int page_tokens, int window, float scale, int vd, int sink, AgOptions opt) {
  extern __shared__ __align__(16) uint8_t af_raw[];
  AfSmem& sm = *reinterpret_cast<AfSmem*>(af_raw);
  const AfItem it = items[blockIdx.x / G];
  if (it.n_tokens * (H / G) <= 8)
    attention_f32_item<1>(sm, it, blockIdx.x % G, q, k_pages, v_pages, block_table, table_stride, out, H, G, hd, page_tokens, window, scale, vd,
                          sink, opt);
  else
    attention_f32_item<4>(sm, it, blockIdx.x % G, q, k_pages, v_pages, block_table, table_stride, out, H, G, hd, page_tokens, window, scale, vd,
                          sink, opt);
}

// Query tokens an item may hold for groups of `group` heads (0: the kernel does not take the group).
HK_API int hk_attention_f32_tokens(int group) { return group >= 1 && group <= AF_ROWS ? AF_ROWS / group : 0; }

// The arguments of hk_attention_generic in float, with items int32 [n_items, 4] as above (each row of the step in one of them).
// Refuses (HK_ERR_UNSUPPORTED) heads above 128, sizes that are no multiple of 4, groups above 32 and misaligned pointers.
HK_API int hk_attention_f32(const float* q, const float* k_pages, const float* v_pages, const int* block_table, int table_stride,
                            const int* items, int n_items, float* out, int H, int G, int hd, int page_tokens, int window, float scale,
                            int vd, int sink, const float* sinks, float softcap, int chunk, int v_stride, const float* gate,
                            long long gate_ld, float gate_scale, const float* dist, int dist_n, void* stream) {
  if (n_items <= 0) return 0;
  if (G < 1 || H % G != 0 || !hk_attention_f32_tokens(H / G) || hd < 4 || hd > AF_HD || (hd & 3) || vd < 4 || vd > AF_HD || (vd & 3) ||
      v_stride < vd || (v_stride & 3) || page_tokens < 1 || softcap < 0.f || chunk < 0 || (dist && dist_n < 1))
    return HK_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15) return HK_ERR_UNSUPPORTED;
  const AgOptions opt = {softcap, chunk, v_stride, sinks, gate, gate_ld, gate_scale, dist, dist_n};
  if (int e = hk_allow_smem<attention_f32_kernel>(sizeof(AfSmem))) return e;
  return hk_launch(attention_f32_kernel, dim3((unsigned)n_items * (unsigned)G), dim3(AF_TH), sizeof(AfSmem), (cudaStream_t)stream, q, k_pages,
                   v_pages, block_table, table_stride, (const AfItem*)items, out, H, G, hd, page_tokens, window, scale, vd, sink, opt);
}
