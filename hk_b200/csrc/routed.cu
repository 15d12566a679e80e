// A feed-forward of experts with a router: every token goes to `top` of `E` small feed-forwards.
//
// Everything that depends on the router's choice stays on the device, so the launches of a step depend
// on its number of rows alone (a decode step through it can be captured in a graph):
//   1. route:   one block per token takes the E router logits (float32 products of the token's vector with
//               the router's rows, summed in a fixed order), picks the `top` largest (the lower index wins a
//               tie) and gives them the softmax over the chosen logits as weights (`bias`: a float per expert that is
//               added to its logit first).  A second mode scores every
//               expert by itself: s = sigmoid(logit); the choice is made on s + correction (a float per expert),
//               optionally among the experts of the best `keep` of `groups` equal groups of neighbours (a
//               group's score: the sum of its two largest choice scores), and the weights are the chosen
//               experts' s over their sum (+ norm_eps), times a factor.  A third mode takes s = softmax over all the
//               logits, chooses on s + correction and gives the chosen s themselves (times a factor) as weights.
//               The router's matrix may carry further
//               rows behind the experts' (`extra`): their logits' sigmoids are handed out per token (a gate
//               of a sublayer that every token uses).
//               The last outputs of the router may stand for no feed-forward at all (identities: such a choice gives
//               back the token's vector); the sort leaves their pairs out and the combine adds the vector itself.
//   2. sort:    one CTA counts the (token, choice) pairs per expert, lays the experts' rows out one after
//               the other (`perm`: sorted place -> pair, `inv`: pair -> sorted place) and cuts every
//               expert's rows into tiles of so many rows (`tiles`: expert and first row, -1 for unused).
//   3. experts: a grouped product over those tiles: tile rows are gathered through `perm` (in bfloat16 by a kernel
//               of its own, before the tensor-core product of gemm_pair.cu), the weights are
//               the tile's expert's; first gate and up with silu(gate) * up (or the clamped
//               activation) in the epilogue, then down.
//               A row's result does not depend on its place in a tile: every output element is one chain of
//               k = 0..K-1 (the FMA kernel) or one of steps of 16 k (the tensor cores).
//   4. combine: y[t] = sum over the token's choices, in the order of the choices, of weight * expert output.
#include <math_constants.h>

#include "common.cuh"

#define RT_BM 64
#define RT_BN 64
#define RT_BK 16

// ------------------------------------------------------------------------------------ 1. route
#define RK_WARPS 8
struct RouteOpts {
  int mode;                  // 0: softmax over the chosen logits; 1: sigmoid scores; 2: softmax over all logits, not renormalised
  const float* correction;   // modes 1 and 2: added to the scores for the choice alone (null: nothing)
  int groups, keep;          // mode 1: the choice is made inside the best `keep` of `groups` groups (groups 0: everywhere)
  float scale, norm_eps;     // mode 1: weights = s / (sum s + norm_eps) * scale; mode 2: weights = s * scale
  int extra;                 // rows of w behind the E experts' rows
  float* extra_out;          // [n, extra]: the sigmoids of those rows' logits
  const float* bias;         // [E + extra]: added to the logits (null: nothing)
};

template <typename T>
__global__ void __launch_bounds__(RK_WARPS * 32)
route_topk_kernel(const T* __restrict__ x, const float* __restrict__ w, int* __restrict__ ids, float* __restrict__ weights, int n,
                  int d, int n_experts, int top, RouteOpts opt) {
  extern __shared__ float sm[];               // [RK_WARPS][E] partial logits, then [E] logits, [n_experts] scores, [groups] x 2
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t = blockIdx.x;                   // a block per token: its warps share the token's vector
  int E = n_experts + opt.extra;              // rows of the router's matrix
  float* part = sm;
  float* z = sm + (size_t)RK_WARPS * E;
  float* score = z + E;
  float* gscore = score + n_experts;
  float* gkept = gscore + opt.groups;
  const T* xr = x + (size_t)t * d;
  for (int e0 = 0; e0 < E; e0 += 8) {          // eight experts per pass over the token's vector
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    if ((d & 3) == 0 && (((uintptr_t)w | (uintptr_t)xr) & 15) == 0) {
      // four consecutive elements a thread: 16-byte reads of the router's rows, all eight experts' in flight together
      for (int i = threadIdx.x * 4; i < d; i += RK_WARPS * 32 * 4) {
        const float x0 = to_f32<T>(xr[i]), x1 = to_f32<T>(xr[i + 1]), x2 = to_f32<T>(xr[i + 2]), x3 = to_f32<T>(xr[i + 3]);
        float4 wv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          wv[j] = e0 + j < E ? *reinterpret_cast<const float4*>(w + (size_t)(e0 + j) * d + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = fmaf(x3, wv[j].w, fmaf(x2, wv[j].z, fmaf(x1, wv[j].y, fmaf(x0, wv[j].x, acc[j]))));
      }
    } else {
      for (int i = threadIdx.x; i < d; i += RK_WARPS * 32) {
        const float xv = to_f32<T>(xr[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (e0 + j < E) acc[j] = fmaf(xv, w[(size_t)(e0 + j) * d + i], acc[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sum = warp_sum(acc[j]);
      if (lane == 0 && e0 + j < E) part[(size_t)wid * E + e0 + j] = sum;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += RK_WARPS * 32) {       // the warps' shares in warp order
    float sum = 0.f;
#pragma unroll
    for (int wv = 0; wv < RK_WARPS; ++wv) sum += part[(size_t)wv * E + e];
    z[e] = opt.bias != nullptr ? sum + opt.bias[e] : sum;
  }
  __syncthreads();
  if (wid != 0) return;
  E = n_experts;
  if (opt.mode == 2) {
    float top_z = -CUDART_INF_F, sum = 0.f;
    for (int e = lane; e < E; e += 32) top_z = fmaxf(top_z, z[e]);
    top_z = warp_max(top_z);
    for (int e = lane; e < E; e += 32) {
      score[e] = expf(z[e] - top_z);
      sum += score[e];
    }
    sum = warp_sum(sum);
    for (int e = lane; e < E; e += 32) {
      const float sc = score[e] / sum;
      score[e] = sc;
      z[e] = opt.correction != nullptr ? sc + opt.correction[e] : sc;
    }
    __syncwarp();
  }
  if (opt.mode == 1) {
    for (int e = lane; e < E; e += 32) {
      const float sc = 1.0f / (1.0f + expf(-z[e]));
      score[e] = sc;
      z[e] = opt.correction != nullptr ? sc + opt.correction[e] : sc;
    }
    for (int e = lane; e < opt.extra; e += 32) opt.extra_out[(size_t)t * opt.extra + e] = 1.0f / (1.0f + expf(-z[E + e]));
    __syncwarp();
    if (opt.groups > 0 && opt.keep < opt.groups) {
      const int size = E / opt.groups;
      for (int g = lane; g < opt.groups; g += 32) {          // a group's score: its two largest choice scores
        float a = -CUDART_INF_F, b = -CUDART_INF_F;
        for (int e = g * size; e < (g + 1) * size; ++e) {
          const float v = z[e];
          if (v > a) {
            b = a;
            a = v;
          } else if (v > b) {
            b = v;
          }
        }
        gscore[g] = size > 1 ? a + b : a;
        gkept[g] = 0.f;
      }
      __syncwarp();
      for (int k = 0; k < opt.keep; ++k) {                   // the best groups, the lower index winning a tie
        float best = -CUDART_INF_F;
        int bi = 0x7fffffff;
        for (int g = lane; g < opt.groups; g += 32) {
          const float v = gscore[g];
          if (gkept[g] == 0.f && (v > best || bi == 0x7fffffff)) {
            best = v;
            bi = g;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) {
            best = ov;
            bi = oi;
          }
        }
        if (lane == 0 && bi < opt.groups) gkept[bi] = 1.f;
        __syncwarp();
      }
      for (int e = lane; e < E; e += 32)
        if (gkept[e / size] == 0.f) z[e] = -CUDART_INF_F;
      __syncwarp();
    }
  }
  float first = 0.f, mine = 0.f, total = 0.f;
  int mine_id = 0;
  for (int k = 0; k < top; ++k) {
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = z[e];
      if (v > best) {                          // ascending e: the first maximum of this lane
        best = v;
        bi = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (k == 0) first = best;
    // mode 0: the first chosen logit is the largest; modes 1 and 2: the expert's own score, without the correction
    const float p = opt.mode != 0 ? (bi < E ? score[bi] : 0.f) : expf(best - first);
    total += p;
    if (lane == (k & 31)) {                    // lane k keeps choice k (top <= 32)
      mine = p;
      mine_id = bi;
    }
    if (lane == 0 && bi < E) z[bi] = -CUDART_INF_F;
    __syncwarp();
  }
  if (lane < top) {
    ids[(size_t)t * top + lane] = mine_id < E ? mine_id : 0;
    weights[(size_t)t * top + lane] = opt.mode == 1 ? mine / (total + opt.norm_eps) * opt.scale : opt.mode == 2 ? mine * opt.scale : mine / total;
  }
}

HK_API int hk_route_topk(const void* x, int dtype, const float* w, int* ids, float* weights, int n, int d, int E, int top, int mode,
                         const float* correction, int groups, int keep, float scale, float norm_eps, int extra, float* extra_out,
                         const float* bias, void* stream) {
  if (n <= 0) return 0;
  if (E < 1 || top < 1 || top > E || top > 32 || E > 2048 || mode < 0 || mode > 2 || extra < 0 || extra > 64) return HK_ERR_UNSUPPORTED;
  if (mode == 0 && (correction != nullptr || groups != 0 || extra != 0)) return HK_ERR_UNSUPPORTED;
  if (mode == 2 && (groups != 0 || extra != 0)) return HK_ERR_UNSUPPORTED;
  if (groups < 0 || (groups > 0 && (E % groups || keep < 1 || keep > groups)) || (extra > 0 && extra_out == nullptr)) return HK_ERR_UNSUPPORTED;
  const RouteOpts opt = {mode, correction, groups, keep, scale, norm_eps, extra, extra_out, bias};
  const size_t smem = ((size_t)(RK_WARPS + 1) * (E + extra) + E + 2 * groups) * sizeof(float);
  dim3 grid((unsigned)n);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HK_F32) {
    if (int e = hk_allow_smem<route_topk_kernel<float>>(smem)) return e;
    return hk_launch(route_topk_kernel<float>, grid, dim3(RK_WARPS * 32), smem, s, (const float*)x, w, ids, weights, n, d, E, top, opt);
  }
  if (dtype == HK_BF16) {
    if (int e = hk_allow_smem<route_topk_kernel<bf16>>(smem)) return e;
    return hk_launch(route_topk_kernel<bf16>, grid, dim3(RK_WARPS * 32), smem, s, (const bf16*)x, w, ids, weights, n, d, E, top, opt);
  }
  return HK_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------------------------ 2. sort
// offsets[E + 1], perm[pairs], inv[pairs], tiles[max_tiles][2].  A pair whose id is E or more (an identity) has no sorted
// place: its inv is -1.
__global__ void __launch_bounds__(1024)
route_sort_kernel(const int* __restrict__ ids, int pairs, int E, int bm, int* __restrict__ offsets, int* __restrict__ perm,
                  int* __restrict__ inv, int* __restrict__ tiles, int max_tiles) {
  extern __shared__ int smi[];                // counts[E], cursor[E]
  int* counts = smi;
  int* cursor = smi + E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x)
    if (ids[p] < E) atomicAdd(&counts[ids[p]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, tile = 0;
    for (int e = 0; e < E; ++e) {
      offsets[e] = at;
      cursor[e] = at;
      for (int r = 0; r < counts[e] && tile < max_tiles; r += bm) {
        tiles[2 * tile] = e;
        tiles[2 * tile + 1] = at + r;
        ++tile;
      }
      at += counts[e];
    }
    offsets[E] = at;
    for (; tile < max_tiles; ++tile) {
      tiles[2 * tile] = -1;
      tiles[2 * tile + 1] = 0;
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    if (ids[p] >= E) {
      inv[p] = -1;
      continue;
    }
    const int at = atomicAdd(&cursor[ids[p]], 1);
    perm[at] = p;
    inv[p] = at;
  }
}

HK_API int hk_route_sort(const int* ids, int pairs, int E, int tile_rows, int* offsets, int* perm, int* inv, int* tiles, int max_tiles,
                         void* stream) {
  if (pairs <= 0) return 0;
  if (E > 4096 || tile_rows < 1) return HK_ERR_UNSUPPORTED;
  return hk_launch(route_sort_kernel, dim3(1), dim3(1024), (size_t)2 * E * sizeof(int), (cudaStream_t)stream, ids, pairs, E,
                   tile_rows, offsets, perm, inv, tiles, max_tiles);
}

HK_API int hk_route_tile_rows() { return RT_BM; }

// xs[p, :] = x[perm[p] / top, :] for the sorted places p < *placed: the tokens' vectors in the experts' order (bf16, d % 8 == 0).
__global__ void route_gather_kernel(const bf16* __restrict__ x, const int* __restrict__ perm, const int* __restrict__ placed, int top,
                                    bf16* __restrict__ xs, int d) {
  const int p = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (p >= *placed) return;             // (identities have no place)
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)p * d);
  const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)(perm[p] / top) * d);
  for (int i = threadIdx.x; i < d / 8; i += blockDim.x) dst[i] = from[i];
}

HK_API int hk_route_gather(const void* x, const int* perm, const int* placed, int top, void* xs, int pairs, int d, void* stream) {
  if (pairs <= 0) return 0;
  if ((d & 7) || (((uintptr_t)x | (uintptr_t)xs) & 15)) return HK_ERR_UNSUPPORTED;
  return hk_launch_pdl(route_gather_kernel, dim3((unsigned)pairs), dim3(d >= 2048 ? 256 : 128), 0, (cudaStream_t)stream, (const bf16*)x, perm,
                       placed, top, (bf16*)xs, d);
}

// Sort and gather at once for steps of few pairs: a block per pair finds its place by counting the pairs before it (lower expert, or
// the same and earlier) and brings the token's vector there; one more block lays out `offsets` and `tiles`.  Bound by its launch: the
// counting is pairs / 256 loads a thread.
__global__ void __launch_bounds__(256)
route_place_kernel(const bf16* __restrict__ x, const int* __restrict__ ids, int pairs, int E, int top, int bm, int* __restrict__ offsets,
                   int* __restrict__ inv, int* __restrict__ tiles, int max_tiles, bf16* __restrict__ xs, int d) {
  extern __shared__ int smi[];                // the last block: counts[E]
  __shared__ int before;
  const int p = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (p == pairs) {
    for (int e = threadIdx.x; e < E; e += 256) smi[e] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < pairs; i += 256)
      if (ids[i] < E) atomicAdd(&smi[ids[i]], 1);
    __syncthreads();
    if (threadIdx.x != 0) return;
    int at = 0, tile = 0;
    for (int e = 0; e < E; ++e) {
      offsets[e] = at;
      for (int r = 0; r < smi[e] && tile < max_tiles; r += bm, ++tile) {
        tiles[2 * tile] = e;
        tiles[2 * tile + 1] = at + r;
      }
      at += smi[e];
    }
    offsets[E] = at;
    for (; tile < max_tiles; ++tile) {
      tiles[2 * tile] = -1;
      tiles[2 * tile + 1] = 0;
    }
    return;
  }
  const int e = ids[p];
  if (e >= E) {                               // an identity: it has no place
    if (threadIdx.x == 0) inv[p] = -1;
    return;
  }
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  int mine = 0;
  for (int i = threadIdx.x; i < pairs; i += 256) mine += ids[i] < e || (ids[i] == e && i < p);
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&before, mine);
  __syncthreads();
  const int place = before;
  if (threadIdx.x == 0) inv[p] = place;
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)place * d);
  const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)(p / top) * d);
  for (int i = threadIdx.x; i < d / 8; i += 256) dst[i] = from[i];
}

// ------------------------------------------------------------------------------------ 3. experts
struct GluAct {
  int clamped;               // 0: silu(gate) * up; 1: g sigmoid(slope g) (u + 1), g = min(gate, limit), u = clamp(up, -limit, limit)
  float limit, slope;
};
__device__ __forceinline__ float glu_value(float g, float u, GluAct act) {
  if (act.clamped) {
    g = fminf(g, act.limit);
    u = fminf(fmaxf(u, -act.limit), act.limit);
    return g / (1.0f + expf(-act.slope * g)) * (u + 1.0f);
  }
  return g / (1.0f + expf(-g)) * u;
}

// out rows are sorted places.  GATED: w is [E][2N][K] = N gate rows then N up rows per expert, out[p, n] (type TO) =
// the gated activation `act` of the two.  Otherwise w is [E][N][K] and out[p, n] (float) = a[p] . w[e][n].  `gather`: row p of `a` is row
// perm[p] / top of the tensor (the token's vector); else row p.
template <typename T, typename TO, bool GATED>
__global__ void __launch_bounds__(256)
grouped_gemm_kernel(const T* __restrict__ a, const T* __restrict__ w, TO* __restrict__ out, const int* __restrict__ tiles,
                    const int* __restrict__ offsets, const int* __restrict__ perm, int top, int gather, int N, int K, GluAct act) {
  __shared__ float As[RT_BK][RT_BM + 4];
  __shared__ float Ws[GATED ? 2 : 1][RT_BK][RT_BN + 4];
  __shared__ int rows[RT_BM];
  const int e = tiles[2 * blockIdx.y];
  if (e < 0) return;
  const int p0 = tiles[2 * blockIdx.y + 1];
  const int p_end = min(p0 + RT_BM, offsets[e + 1]);
  const int tid = threadIdx.x;
  if (tid < RT_BM) {
    const int p = p0 + tid;
    rows[tid] = p < p_end ? (gather ? perm[p] / top : p) : -1;
  }
  __syncthreads();
  const int n0 = blockIdx.x * RT_BN;
  const int tx = tid & 15, ty = tid >> 4;
  const T* we = w + (size_t)e * (GATED ? 2 : 1) * N * K;
  float acc[GATED ? 2 : 1][4][4];
#pragma unroll
  for (int s = 0; s < (GATED ? 2 : 1); ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[s][i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += RT_BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = tid + j * 256;
      const int r = i >> 4, c = i & 15;
      const int gk = k0 + c, gn = n0 + r;
      const int src = rows[r];
      As[c][r] = (src >= 0 && gk < K) ? to_f32<T>(a[(size_t)src * K + gk]) : 0.f;
      Ws[0][c][r] = (gn < N && gk < K) ? to_f32<T>(we[(size_t)gn * K + gk]) : 0.f;
      if (GATED) Ws[GATED ? 1 : 0][c][r] = (gn < N && gk < K) ? to_f32<T>(we[(size_t)(N + gn) * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < RT_BK; ++kk) {
      float av[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int s = 0; s < (GATED ? 2 : 1); ++s) {
        float wv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[j] = Ws[s][kk][tx * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[s][i][j] = fmaf(av[i], wv[j], acc[s][i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = p0 + ty * 4 + i;
    if (p >= p_end) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float val = acc[0][i][j];
      if (GATED) {
        val = glu_value(val, acc[GATED ? 1 : 0][i][j], act);
      }
      out[(size_t)p * N + gn] = from_f32<TO>(val);
    }
  }
}

HK_API int hk_grouped_gemm(const void* a, const void* w, int dtype, void* out, const int* tiles, int max_tiles, const int* offsets,
                           const int* perm, int top, int gather, int N, int K, int gated, int clamped, float limit, float slope,
                           void* stream) {
  if (max_tiles <= 0 || N <= 0) return 0;
  if (max_tiles > 65535) return HK_ERR_UNSUPPORTED;
  const GluAct act = {clamped, limit, slope};
  dim3 grid((unsigned)((N + RT_BN - 1) / RT_BN), (unsigned)max_tiles);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HK_F32) {
    if (gated)
      return hk_launch(grouped_gemm_kernel<float, float, true>, grid, dim3(256), 0, s, (const float*)a, (const float*)w, (float*)out,
                       tiles, offsets, perm, top, gather, N, K, act);
    return hk_launch(grouped_gemm_kernel<float, float, false>, grid, dim3(256), 0, s, (const float*)a, (const float*)w, (float*)out,
                     tiles, offsets, perm, top, gather, N, K, act);
  }
  if (dtype == HK_BF16) {
    if (gated)
      return hk_launch(grouped_gemm_kernel<bf16, bf16, true>, grid, dim3(256), 0, s, (const bf16*)a, (const bf16*)w, (bf16*)out, tiles,
                       offsets, perm, top, gather, N, K, act);
    return hk_launch(grouped_gemm_kernel<bf16, float, false>, grid, dim3(256), 0, s, (const bf16*)a, (const bf16*)w, (float*)out, tiles,
                     offsets, perm, top, gather, N, K, act);
  }
  return HK_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------------------------ 4. combine
// y[t, :] (= or +=) factor * (sum_k weights[t, k] * ys[inv[t * top + k], :] (+ shared_gate[t] * shared[t, :], the result of
// a sublayer that every token uses, when `shared` is given; a null gate counts as 1)).  A choice whose inv is negative is
// an identity: it adds weights[t, k] * x[t, :], the token's own vector.
template <typename T>
__global__ void route_combine_kernel(const float* __restrict__ ys, const int* __restrict__ inv, const float* __restrict__ weights,
                                     float* __restrict__ y, int d, int top, int accumulate, const float* __restrict__ shared,
                                     const float* __restrict__ shared_gate, const T* __restrict__ x, float factor) {
  const int t = blockIdx.x;
  pdl_wait();
  const float sg = shared != nullptr ? (shared_gate != nullptr ? shared_gate[t] : 1.0f) : 0.f;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < d; i += gridDim.y * blockDim.x) {
    float acc = 0.f;
    for (int k = 0; k < top; ++k) {
      const int at = inv[(size_t)t * top + k];
      const float v = at >= 0 ? ys[(size_t)at * d + i] : x != nullptr ? to_f32<T>(x[(size_t)t * d + i]) : 0.f;
      acc = fmaf(weights[(size_t)t * top + k], v, acc);
    }
    if (shared != nullptr) acc = fmaf(sg, shared[(size_t)t * d + i], acc);
    float* o = y + (size_t)t * d + i;
    *o = accumulate ? fmaf(factor, acc, *o) : factor * acc;
  }
}

HK_API int hk_route_combine(const float* ys, const int* inv, const float* weights, float* y, int n, int d, int top, int accumulate,
                            const float* shared, const float* shared_gate, const void* x, int x_dtype, float factor, void* stream) {
  if (n <= 0) return 0;
  // a block per token; where the tokens alone do not fill the SMs (decode steps) a token's columns are spread over blocks
  const int threads = d >= 1024 ? 256 : 128;
  int split = 1;
  while (split < 16 && (long long)n * split < 2 * 148 && split * threads < d) split <<= 1;
  const dim3 grid((unsigned)n, (unsigned)split);
  cudaStream_t s = (cudaStream_t)stream;
  if (x_dtype == HK_F32)
    return hk_launch_pdl(route_combine_kernel<float>, grid, dim3(threads), 0, s, ys, inv, weights, y, d, top, accumulate, shared, shared_gate,
                     (const float*)x, factor);
  if (x_dtype == HK_BF16)
    return hk_launch_pdl(route_combine_kernel<bf16>, grid, dim3(threads), 0, s, ys, inv, weights, y, d, top, accumulate, shared, shared_gate,
                     (const bf16*)x, factor);
  return HK_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------------------------ 2 to 4 at once
// Everything behind the choice for a step of few (token, choice) pairs in bf16: sort and gather, the two grouped products
// (`grouped`: hk_gemm_pair_grouped of the library beside this one), combine.  One call, because such a step waits for the host: 64
// tokens of 4,096 by eight experts of 2,048 take the GPU 90 us, and a wrapper around each launch made the pass 171.
// w_gate_up [E][2 F][d], w_down [E][d][F]; scratch: hk_routed_experts_scratch bytes, 16-byte aligned; the rest as hk_route_combine.
typedef int (*GroupedProduct)(const void* a, const void* w, void* out, int M, int N, int K, long long ldo, int epilogue, int n_groups,
                              const int* tiles, int max_tiles, const int* offsets, int tile_rows, int pairs, int* status, float limit,
                              float slope, void* stream);
namespace {
struct ExpertsScratch {
  size_t offsets, inv, tiles, xs, h, ys, bytes;
  int max_tiles;
  ExpertsScratch(int pairs, int E, int d, int F, int tile_rows) {
    size_t at = 0;
    auto take = [&](size_t n) { const size_t r = at; at += (n + 255) & ~(size_t)255; return r; };
    max_tiles = pairs / tile_rows + (E < pairs ? E : pairs);
    offsets = take((size_t)(E + 1) * 4);
    inv = take((size_t)pairs * 4);
    tiles = take((size_t)max_tiles * 8);
    xs = take((size_t)pairs * d * 2);
    h = take((size_t)pairs * F * 2);
    ys = take((size_t)pairs * d * 4);
    bytes = at;
  }
};
}  // namespace

HK_API long long hk_routed_experts_scratch(int pairs, int E, int d, int F, int tile_rows) {
  return (long long)ExpertsScratch(pairs, E, d, F, tile_rows).bytes;
}

HK_API int hk_routed_experts(const void* grouped, const void* x, const int* ids, const float* weights, const void* w_gate_up,
                             const void* w_down, float* y, void* scratch, int n, int d, int F, int E, int top, int tile_rows, int epilogue,
                             float limit, float slope, int accumulate, const float* shared, const float* shared_gate, int identities,
                             float factor, int sm_pairs, int* status, void* stream) {
  if (n <= 0) return 0;
  if (grouped == nullptr || E < 1 || E > 4096 || top < 1 || (d & 7) || (F & 7) || tile_rows < 32 || (((uintptr_t)x | (uintptr_t)scratch) & 15))
    return HK_ERR_UNSUPPORTED;
  const int pairs = n * top;
  const ExpertsScratch sc(pairs, E, d, F, tile_rows);
  char* base = reinterpret_cast<char*>(scratch);
  int *offsets = (int*)(base + sc.offsets), *inv = (int*)(base + sc.inv), *tiles = (int*)(base + sc.tiles);
  const GroupedProduct product = (GroupedProduct)grouped;
  if (int e = hk_launch_pdl(route_place_kernel, dim3((unsigned)pairs + 1), dim3(256), (size_t)E * sizeof(int), (cudaStream_t)stream, (const bf16*)x,
                            ids, pairs, E, top, tile_rows, offsets, inv, tiles, sc.max_tiles, (bf16*)(base + sc.xs), d))
    return e;
  if (int e = product(base + sc.xs, w_gate_up, base + sc.h, pairs, 2 * F, d, F, epilogue, E, tiles, sc.max_tiles, offsets, tile_rows, sm_pairs,
                      status, limit, slope, stream))
    return e;
  if (int e = product(base + sc.h, w_down, base + sc.ys, pairs, d, F, d, 0, E, tiles, sc.max_tiles, offsets, tile_rows, sm_pairs, status, limit,
                      slope, stream))
    return e;
  return hk_route_combine((const float*)(base + sc.ys), inv, weights, y, n, d, top, accumulate, shared, shared_gate, identities ? x : nullptr,
                          HK_BF16, factor, stream);
}
