// The short causal convolution per channel that some mixers put behind their projections, with the request's last inputs
// kept in its state slot between steps (float32).
//
// A step's batch is described by a segment table int32 [n_seg, 3] = (state slot, first row, rows), as for the recurrent
// mixers' scans; an output depends on the inputs before it alone, never on the cut of the prompt, the batch or the slot.
#include "common.cuh"

// ------------------------------------------------------------------ short causal convolution per channel
// y[t, c] = act(bias[c] + sum_j w[c, j] * x[t - (taps - 1) + j, c]) over the rows of every segment, with act = silu (1) or
// the identity (0) and a bias or none: the last column of w is the current token's.  The sum and the activation are
// float32; y is float32 or the storage type.  The inputs before a segment's first row come from the request's tail
// (state [slots, taps - 1, C], the last taps - 1 inputs of the request, zero at its start), which the same call
// moves on.  x (float32) and y are column slices [n, C] of wider matrices.  A thread owns one channel of one chunk
// of a segment's tokens; the threads of the first chunk read the old tail before they write the new one, and
// nobody else touches it.
#define SC_TOKENS 32
#define SC_GROUP 8
#define SC_MAX_TAPS 16

__device__ __forceinline__ float conv_act(float z, int act) { return act ? z / (1.0f + expf(-z)) : z; }

// The thread walks its tokens in groups of SC_GROUP: the group's inputs are loaded at once (each input is read once; the
// taps - 1 before them stay in registers from the group before), then the group's outputs are summed, oldest tap first.
// A segment of one row (a decoded token) takes a path of its own with the same sum.  TAPS: the most taps an instance holds.
template <typename T, int TAPS>
__global__ void __launch_bounds__(128)
short_conv_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ w, const float* __restrict__ bias,
                  const int* __restrict__ segs, float* __restrict__ tail, T* __restrict__ y, long long ldy, int C, int taps, int act) {
  const int seg = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int slot = segs[seg * 3], row0 = segs[seg * 3 + 1], count = segs[seg * 3 + 2];
  const int t0 = blockIdx.z * SC_TOKENS;
  if (c >= C || t0 >= count) return;
  const int back = taps - 1;
  float* tl = tail + (size_t)slot * back * C + c;
  auto input = [&](int r) -> float {            // the request's input r rows from the segment's first (r may be negative)
    return r >= 0 ? x[(size_t)(row0 + r) * ldx + c] : tl[(size_t)(back + r) * C];
  };
  float wr[TAPS];                               // wr[s]: the weight of the input s tokens back
  float hist[TAPS];                             // hist[s], s >= 1: the input s tokens before the group's first
  if (TAPS == 4 && taps == 4 && ((uintptr_t)w & 15) == 0) {
    const float4 q = *reinterpret_cast<const float4*>(w + (size_t)c * 4);
    wr[0] = q.w; wr[TAPS > 1 ? 1 : 0] = q.z; wr[TAPS > 2 ? 2 : 0] = q.y; wr[TAPS > 3 ? 3 : 0] = q.x;
  } else {
#pragma unroll
    for (int s = 0; s < TAPS; ++s) wr[s] = s <= back ? w[(size_t)c * taps + back - s] : 0.f;
  }
#pragma unroll
  for (int s = 0; s < TAPS; ++s) hist[s] = (s >= 1 && s <= back) ? input(t0 - s) : 0.f;
  const float first = bias != nullptr ? bias[c] : 0.f;
  if (count == 1) {
    const float now = x[(size_t)row0 * ldx + c];
    float acc = first;
#pragma unroll
    for (int s = TAPS - 1; s >= 1; --s)
      if (s <= back) acc = fmaf(wr[s], hist[s], acc);
    acc = fmaf(wr[0], now, acc);
    y[(size_t)row0 * ldy + c] = from_f32<T>(conv_act(acc, act));
#pragma unroll
    for (int s = TAPS - 1; s >= 2; --s)
      if (s <= back) tl[(size_t)(back - s) * C] = hist[s - 1];
    if (back > 0) tl[(size_t)(back - 1) * C] = now;
    return;
  }
  const int t1 = min(count, t0 + SC_TOKENS);
  for (int tg = t0; tg < t1; tg += SC_GROUP) {
    float nw[SC_GROUP];
#pragma unroll
    for (int u = 0; u < SC_GROUP; ++u) nw[u] = tg + u < t1 ? x[(size_t)(row0 + tg + u) * ldx + c] : 0.f;
    float acc[SC_GROUP];
#pragma unroll
    for (int u = 0; u < SC_GROUP; ++u) acc[u] = first;
#pragma unroll
    for (int s = TAPS - 1; s >= 0; --s) {
      if (s <= back) {
#pragma unroll
        for (int u = 0; u < SC_GROUP; ++u) acc[u] = fmaf(wr[s], u >= s ? nw[u >= s ? u - s : 0] : hist[u >= s ? 0 : s - u], acc[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < SC_GROUP; ++u)
      if (tg + u < t1) y[(size_t)(row0 + tg + u) * ldy + c] = from_f32<T>(conv_act(acc[u], act));
    float next[TAPS];
#pragma unroll
    for (int s = 1; s < TAPS; ++s) next[s] = s <= SC_GROUP ? nw[s <= SC_GROUP ? SC_GROUP - s : 0] : hist[s <= SC_GROUP ? 0 : s - SC_GROUP];
#pragma unroll
    for (int s = 1; s < TAPS; ++s) hist[s] = next[s];
  }
  if (blockIdx.z == 0 && back > 0) {
    float keep[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
      if (j < back) keep[j] = input(count - back + j);
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
      if (j < back) tl[(size_t)j * C] = keep[j];
  }
}

// The same for up to four taps and channels in whole 16-byte pieces: a thread makes four channels of eight tokens, everything it reads
// asked for at once, with the sums in the same order.  A block's tokens are found by counting through the segments, so that no block is
// launched for tokens that do not exist.  Bound by its bytes and the activations (which steps take it, and both times: see short_conv).
#define SCV_TOKENS 8
template <typename T>
__global__ void __launch_bounds__(128)
short_conv_vec_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ w, const float* __restrict__ bias,
                      const int* __restrict__ segs, int n_seg, float* __restrict__ tail, T* __restrict__ y, long long ldy, int C, int taps,
                      int act) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, back = taps - 1;
  int left = blockIdx.x, seg = -1, count = 0;
  for (int base = 0; base < n_seg; base += 32) {
    const int mine = base + lane < n_seg ? segs[(base + lane) * 3 + 2] : 0, chunks = (mine + SCV_TOKENS - 1) / SCV_TOKENS;
    int upto = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, upto > left);
    if (past) {
      const int l = __ffs(past) - 1;
      seg = base + l;
      count = __shfl_sync(0xffffffffu, mine, l);
      left -= __shfl_sync(0xffffffffu, upto - chunks, l);
      break;
    }
    left -= __shfl_sync(0xffffffffu, upto, 31);
  }
  const int c = (blockIdx.y * 128 + threadIdx.x) * 4;
  if (seg < 0 || c >= C) return;
  const int slot = segs[seg * 3], row0 = segs[seg * 3 + 1], t0 = left * SCV_TOKENS;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float* tl = tail + (size_t)slot * back * C + c;
  const float* xp = x + (size_t)row0 * ldx + c;
  float in[SCV_TOKENS + 3][4], wr[4][4], b[4];
#pragma unroll
  for (int i = 0; i < SCV_TOKENS + 3; ++i) {
    const int r = t0 - 3 + i;
    float4 v = zero;
    if (r >= 0) {
      if (r < count && (i >= 3 || 3 - i <= back)) v = *reinterpret_cast<const float4*>(xp + (size_t)r * ldx);
    } else if (-r <= back) {
      v = *reinterpret_cast<const float4*>(tl + (size_t)(back + r) * C);
    }
    in[i][0] = v.x; in[i][1] = v.y; in[i][2] = v.z; in[i][3] = v.w;
  }
  const float4 bv = bias != nullptr ? *reinterpret_cast<const float4*>(bias + c) : zero;
  b[0] = bv.x; b[1] = bv.y; b[2] = bv.z; b[3] = bv.w;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (taps == 4) {
      const float4 v = *reinterpret_cast<const float4*>(w + (size_t)(c + e) * 4);
      wr[0][e] = v.w; wr[1][e] = v.z; wr[2][e] = v.y; wr[3][e] = v.x;
    } else {
#pragma unroll
      for (int s = 0; s < 4; ++s) wr[s][e] = s <= back ? w[(size_t)(c + e) * taps + back - s] : 0.f;
    }
  }
#pragma unroll
  for (int u = 0; u < SCV_TOKENS; ++u) {
    if (t0 + u >= count) break;
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[e] = b[e];
#pragma unroll
      for (int s = 3; s >= 0; --s)
        if (s <= back) acc[e] = fmaf(wr[s][e], in[3 + u - s][e], acc[e]);
      acc[e] = conv_act(acc[e], act);
    }
    T* dst = y + (size_t)(row0 + t0 + u) * ldy + c;
    if (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(dst)) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[0], acc[1]), hi = __floats2bfloat162_rn(acc[2], acc[3]);
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
  if (t0 == 0) {                // the first block of tokens has read the old tail: the last `back` inputs take its place
    float4 keep[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int r = count - back + j;
      auto held = [&](int e) { return r == -1 ? in[2][e] : r == -2 ? in[1][e] : in[0][e]; };       // (selects: an address would cost local memory)
      if (j < back) keep[j] = r >= 0 ? *reinterpret_cast<const float4*>(xp + (size_t)r * ldx) : make_float4(held(0), held(1), held(2), held(3));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < back) *reinterpret_cast<float4*>(tl + (size_t)j * C) = keep[j];
  }
}

template <typename T, int TAPS>
static int short_conv(const float* x, long long ldx, const float* w, const float* bias, const int* segs, int n_seg, int n_rows, float* tail,
                      T* y, long long ldy, int C, int taps, int act, cudaStream_t s) {
  // a step of single rows needs no second block of tokens; else as many as the longest segment may have
  const int longest = n_rows - n_seg + 1, portions = (longest + SC_TOKENS - 1) / SC_TOKENS;
  // Four channels a thread: the walk's threads go through up to 32 tokens one group of eight after the other and its blocks are counted for
  // segments that are all as long as one may be, but finding a block's segment takes a look at all of them.  us, walk / four channels:
  // one segment of 64, 512 and 2,048 tokens of 4,096 channels 6.7 / 5.3, 8.4 / 7.3, 20.0 / 17.3, four of 512 tokens of 6,144 29.0 / 25.5,
  // 300 of 7 460 / 45, 16 single rows beside 512 tokens 16.0 / 10.6; 1,024 single rows beside 512 tokens 462 / 127, 4,096 beside 64 407 /
  // 1,245 (so: at most 256 segments for each portion of tokens).  Portions of 8 tokens and less are one group to the walk as well: 64
  // single rows beside 8 tokens of 2,048 channels 4.1 / 6.1.  Single rows alone, of 6,144 channels: 16 of them 2.9 / 3.4, 32 4.1 / 3.8,
  // 128 9.2 / 8.5, 256 15.8 / 16.8; of 2,048 64 3.1 / 3.6, 96 4.3 / 4.1, 256 6.9 / 8.2.
  const bool wide = longest == 1 ? n_seg <= 128 && (long long)n_seg * ((C + 127) / 128) >= 1536 : longest > 16 && n_seg <= 256LL * portions;
  if (wide && taps <= 4 && !(C & 3) && !(ldx & 3) && !(ldy & 3) &&
      !(((uintptr_t)x | (uintptr_t)w | (uintptr_t)bias | (uintptr_t)tail | (uintptr_t)y) & 15))
    return hk_launch_pdl(short_conv_vec_kernel<T>, dim3((unsigned)(n_rows / SCV_TOKENS + n_seg), (unsigned)((C + 511) / 512)), dim3(128), 0, s, x, ldx, w,
                     bias, segs, n_seg, tail, y, ldy, C, taps, act);
  dim3 grid((unsigned)n_seg, (unsigned)((C + 127) / 128), (unsigned)portions);
  return hk_launch(short_conv_kernel<T, TAPS>, grid, dim3(128), 0, s, x, ldx, w, bias, segs, tail, y, ldy, C, taps, act);
}

HK_API int hk_short_conv(const float* x, long long ldx, const float* w, const float* bias, const int* segs, int n_seg, int n_rows,
                         float* tail, void* y, int y_dtype, long long ldy, int C, int taps, int act, void* stream) {
  if (n_seg <= 0 || n_rows <= 0 || C <= 0) return 0;
  if (taps < 1 || taps > SC_MAX_TAPS || act < 0 || act > 1 || n_rows < n_seg) return HK_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
#define SHORT_CONV(T)                                                                                                     \
  (taps <= 4 ? short_conv<T, 4>(x, ldx, w, bias, segs, n_seg, n_rows, tail, (T*)y, ldy, C, taps, act, s)                  \
             : short_conv<T, SC_MAX_TAPS>(x, ldx, w, bias, segs, n_seg, n_rows, tail, (T*)y, ldy, C, taps, act, s))
  if (y_dtype == HK_F32) return SHORT_CONV(float);
  if (y_dtype == HK_BF16) return SHORT_CONV(bf16);
  return HK_ERR_UNSUPPORTED;
#undef SHORT_CONV
}
