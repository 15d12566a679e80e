// Recurrences with a matrix state per head, prompt portions: what recurrent.cu walks token by token, here in chunks of 32 tokens.
// Per head, S [dk, dv] and per token a record (d, a*u, u, k, r, v):
//     S_t = diag(d_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T,   o_t = S_t^T r_t
// With P_t the product of a chunk's decays up to token t, S_0 its start state and w_t = u_t^T S_(t-1), in exact arithmetic
//     (I + Auu) W = U~ S_0 + Auk V,     O = R~ S_0 + Ark V - Aru W,     S = P_last S_0 + K'^T V - AU'^T W
// where Axy[t, s] = sum_i x_t[i] y_s[i] (decays between s and t, up to t - 1 for x = u: s < t, up to t for x = r: s <= t),
// U~ and R~ are the rows of u and r decayed from the chunk's start and K', AU' those of k and a*u decayed to its end.  W is
// linear in S_0, so a chunk is two matrices and two offsets that do not depend on it:
//   1. local:  a block per (chunk, head) solves the unit triangular system for [U~ | Auk V] and writes
//              P [dk], M [dk, dk], B [dk, dv] with S = P S_0 + (M S_0 + B), Rq [32, dk] and Ov [32, dv] (to `out`) with
//              O = Rq S_0 + Ov;
//   2. walk:   a block per (request, head, 16 or 32 value columns) goes through the request's chunks, S in registers.
// Without a removal term (retention, matrix memory) there is no M and no system to solve, and P is one number: see below.
// P S_0 is added last: what is summed before it is small where decays are weak, and rounds less.
//
// Products run on mma.sync with float32 factors in three bf16 pieces each, sums, decays and everything else are float32 (one number per
// token: 64 bits), decays are products of the tokens' decays (never differences of logarithms): an
// entry of the four matrices carries the rounding of the decays between its two tokens, as the walk token by token does.
// Where the decay is one number per token the products between every two tokens are made one by one; where it is one per
// channel (generalised delta rule) rows are scaled by P_t and 1 / P_s, which holds while a chunk's decay stays above 2^-64
// (the launcher's condition on decay_scale).
//
// A value, key, gate or decay that is NaN or Inf reaches its own token and later ones, as in the walk: a product with zeros above the
// diagonal would not keep it out, so a chunk with such a factor of a triangular matrix takes multiply-adds that leave them out.  (An Inf
// may come out as NaN: its pieces do not add up.)
//
// One request of 2,048 tokens at 64 heads of 64 x 64, walk token by token (L2 cold) / chunks on float32 multiply-adds -> here (launches back to
// back): generalised rule 988 / 421 -> 338 us, gated rule 978 / 388 -> 294, matrix memory 1,074 / 265 -> 227, retention 605 / 180 -> 168; of 512
// tokens 257 / 118 -> 98, 257 / 111 -> 82, 288 / 69 -> 60, 161 / 51 -> 47.
// Relative error against 64 bits, outputs and states, multiply-adds -> here, means of three seeds at 2,048 tokens: generalised rule 6.7e-7 and
// 7.2e-7 -> 6.2e-7 and 7.1e-7, gated rule 4.0e-7 and 3.5e-7 -> 3.4e-7 and 3.2e-7, matrix memory 1.67e-7 and 1.05e-7 -> 1.50e-7 and 0.72e-7,
// retention 1.92e-7 and 1.32e-7 -> 1.38e-7 and 0.97e-7; smaller alike, by 3 to 30 %, at 1,000 tokens of 32 heads and at 512 of 64.
#include <math_constants.h>

#include "common.cuh"

namespace {

constexpr int CQ = 32;          // tokens of a chunk
constexpr int NT = 64;          // state rows (keys are filled up with zeros)
constexpr int LD = NT + 4;      // floats between rows in shared memory: eight rows' 16-byte pieces lie in different banks
constexpr int NTH = 128;
constexpr int MFLOATS = NT * NT + NT;      // M of a chunk and head, and behind it P

struct Chunk {
  int row0, count;              // its rows of the step
};
struct Request {
  int slot, chunk0, chunks;
};

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 mul4(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}
__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void fma4(float4& c, float a, float4 b) {
  c.x = fmaf(a, b.x, c.x);
  c.y = fmaf(a, b.y, c.y);
  c.z = fmaf(a, b.z, c.z);
  c.w = fmaf(a, b.w, c.w);
}

// The products of a chunk's decays, one number g per token, in 64 bits: the same decay in every token (retention) would round the
// same way in every product, chunk after chunk.  A lane per token: `win` [5][CQ], the products of 1, 2, 4, 8 and 16 tokens up to its
// own; `from` [CQ] = g[0] .. g[t], and what `from` of the last token is short of the product.  (Each product as a chain of its own, 32
// long, took a warp 5,600 clocks that the block waited for.)
__device__ __forceinline__ void decay_windows(float g, double* win, float* from, float* rest, int lane) {
  double x = g;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    win[j * CQ + lane] = x;
    const double y = __shfl_up_sync(0xffffffffu, x, 1 << j);
    if (lane >= 1 << j) x *= y;
  }
  from[lane] = (float)x;
  if (lane == CQ - 1) *rest = (float)(x - (double)(float)x);
}
// g[s + 1] .. g[t] for s <= t, 0 above: the windows that make up t - s
__device__ __forceinline__ float decay_between(const double* win, int t, int s) {
  if (s > t) return 0.f;
  double x = 1.;
  int at = t;
#pragma unroll
  for (int j = 0; j < 5; ++j)
    if ((t - s) >> j & 1) {
      x *= win[j * CQ + at];
      at -= 1 << j;
    }
  return (float)x;
}

// What a rule reads: columns slices of one matrix of row stride ld, and the rule's own.
struct DeltaIn {
  const float *q, *k, *v;       // generalised: r, k, v
  long long ld;
  const float *x, *y;           // generalised: al (stride ld), wl (stride ldx); gated: beta and decay logits (stride ldx)
  long long ldx;
  const float *xb, *yb;         // generalised: a_bias, w_bias; gated: A_log, dt_bias
  float s0, s1;                 // generalised: decay_scale, key_eps; gated: q_scale, unit_eps
  int H, G, dk, dv;
};

struct DeltaSmem {
  float ur[2 * CQ * LD];        // rows u, then r; the first half becomes X
  float ka[2 * CQ * LD];        // rows k, then a*u
  float vs[CQ * LD];
  float a[2 * CQ * LD];         // rows u, r; columns k, a*u (before that: the decays; behind it, on the k columns: Ark V)
  float w[CQ * LD];             // the decays' products, then Auk V, then W
  float pc[NT];                 // the chunk's decay per channel
  float g[CQ], gb[CQ], from[CQ], rest[4];
  double win[5 * CQ];
};

}  // namespace

// ------------------------------------------------------------------ products on the tensor cores
// mma.sync (16 x 8 x 16, bf16, float32 sums): a float32 factor is cut into three bf16 numbers whose sum it is, and of the nine products
// of two such factors the six of the largest pieces are taken, the first in a sum of its own.
namespace {
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// The largest pieces, of finite numbers always finite: what would round up to an infinity, the last 0.2 % of float32's range, gives the
// largest bf16 number, and zeros in the other factor still make zeros of it.
__device__ __forceinline__ uint32_t pack_first(float lo, float hi) {
  uint32_t v;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}
// two float32 numbers as three pairs of bf16 whose sums they are, `step` words apart
__device__ __forceinline__ void split3(float2 x, uint32_t* out, int step) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    out[p * step] = p == 0 ? pack_first(x.x, x.y) : pack_bf16(x.x, x.y);
    x.x -= __uint_as_float(out[p * step] << 16);
    x.y -= __uint_as_float(out[p * step] & 0xffff0000u);
  }
}
// big += the product of the largest pieces, small += the five next
__device__ __forceinline__ void mma_split(float* big, float* small, const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
  mma_bf16(small, a[2], b[0]);
  mma_bf16(small, a[1], b[1]);
  mma_bf16(small, a[0], b[2]);
  mma_bf16(small, a[1], b[0]);
  mma_bf16(small, a[0], b[1]);
  mma_bf16(big, a[0], b[0]);
}

// Fragments of a float32 matrix in shared memory, cut into pieces; g = lane / 4, q = lane % 4.
// A operand, 16 rows by 16 k, rows side by side: `a` at (row g, k 2 q); the rows times f0 (g) and f1 (g + 8)
__device__ __forceinline__ void frag_rows(const float* a, int ld, float f0, float f1, uint32_t (&out)[3][4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float2 x = *reinterpret_cast<const float2*>(a + 8 * (e & 1) * ld + 8 * (e >> 1));
    x.x *= e & 1 ? f1 : f0;
    x.y *= e & 1 ? f1 : f0;
    split3(x, &out[0][e], 4);
  }
}
// A operand from a matrix that lies the other way round, k by k: `a` at (k 2 q, row g); all times f, or the k times their own (f at 2 q)
__device__ __forceinline__ void frag_turned(const float* a, int ld, float f, uint32_t (&out)[3][4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float* p = a + 8 * (e >> 1) * ld + 8 * (e & 1);
    split3(make_float2(p[0] * f, p[ld] * f), &out[0][e], 4);
  }
}
__device__ __forceinline__ void frag_turned(const float* a, int ld, const float* f, uint32_t (&out)[3][4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int k = 8 * (e >> 1);
    const float* p = a + k * ld + 8 * (e & 1);
    split3(make_float2(p[0] * f[k], p[ld] * f[k + 1]), &out[0][e], 4);
  }
}
__device__ __forceinline__ bool finite4(float4 v) {
  return fabsf(v.x) < CUDART_INF_F && fabsf(v.y) < CUDART_INF_F && fabsf(v.z) < CUDART_INF_F && fabsf(v.w) < CUDART_INF_F;
}
// B operand, 16 k by 8 columns: `b` at (column g, k 2 q) of a matrix column by column ...
__device__ __forceinline__ void frag_columns(const float* b, uint32_t (&out)[3][2]) {
#pragma unroll
  for (int e = 0; e < 2; ++e) split3(*reinterpret_cast<const float2*>(b + 8 * e), &out[0][e], 2);
}
// ... or at (k 2 q, column g) of one k by k
__device__ __forceinline__ void frag_k(const float* b, int ld, uint32_t (&out)[3][2]) {
#pragma unroll
  for (int e = 0; e < 2; ++e) split3(make_float2(b[8 * e * ld], b[(8 * e + 1) * ld]), &out[0][e], 2);
}

}  // namespace

// ------------------------------------------------------------------ 1. local part with a removal term
// Bound by the instructions that bring and cut the products' operands (IPC 2.1 of 4, tensor pipe 26 %, shared memory 60 %): 0.9 M
// multiply-adds a block, the records' two sigmoids and two exponentials an entry, the triangular system.  70 KB of shared memory and 128
// threads: three blocks share an SM; with 256 threads 396 us instead of 364 (2,048 tokens, 64 heads, with the walk).  A warp has 32 rows
// by 32 columns of most products, so that what it cuts serves two of them: 16 rows by 64 took 364 us, this 348 (gated: 325 and 316).
template <bool GATED>
__global__ void __launch_bounds__(NTH, 3)
delta_local_kernel(const DeltaIn in, const Chunk* __restrict__ chunks, float* __restrict__ mm, float* __restrict__ rq,
                   float* __restrict__ bb, float* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  DeltaSmem& sm = *reinterpret_cast<DeltaSmem*>(smem_raw);
  const int H = in.H, dk = in.dk, dv = in.dv;
  const int c = blockIdx.x / H, h = blockIdx.x % H;
  const Chunk ch = chunks[c];
  const int tid = threadIdx.x;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);

  // ---- the tokens' records; a token's row in four threads
  {
    const int t = tid >> 2, i0 = (tid & 3) * 16;
    const bool row_in = t < ch.count;
    const size_t row = (size_t)(ch.row0 + (row_in ? t : 0));
    const int hk = GATED ? h / (H / in.G) : h;
    const float* kp = in.k + row * in.ld + (size_t)hk * dk;
    const float* qp = in.q + row * in.ld + (size_t)hk * dk;
    float4 kr[4], qr[4];
    float sk = 0.f, sq = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = row_in && i0 + 4 * j < dk;
      kr[j] = ok ? ld4(kp + i0 + 4 * j) : zero;
      qr[j] = ok ? ld4(qp + i0 + 4 * j) : zero;
      sk = dot4(kr[j], kr[j], sk);
      sq = dot4(qr[j], qr[j], sq);
    }
    sk += __shfl_xor_sync(0xffffffffu, sk, 1);
    sk += __shfl_xor_sync(0xffffffffu, sk, 2);
    const float kinv = row_in ? 1.0f / sqrtf(sk + in.s1) : 0.f;      // (a row that is not there has no length)
    float beta = 0.f;
    if (GATED) {
      sq += __shfl_xor_sync(0xffffffffu, sq, 1);
      sq += __shfl_xor_sync(0xffffffffu, sq, 2);
      const float qinv = row_in ? in.s0 / sqrtf(sq + in.s1) : 0.f;
      float g = 1.f;
      if (row_in) {
        beta = sigmoid_f(in.x[row * in.ldx + h]);
        g = expf(-expf(in.xb[h]) * softplus_f(in.y[row * in.ldx + h] + in.yb[h]));
      }
      if ((tid & 3) == 0) {
        sm.g[t] = g;
        sm.gb[t] = g * beta;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 u = mul4(kr[j], kinv);
        st4(sm.ur + t * LD + i0 + 4 * j, u);
        st4(sm.ka + t * LD + i0 + 4 * j, u);
        st4(sm.ur + (CQ + t) * LD + i0 + 4 * j, mul4(qr[j], qinv));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + 4 * j;
        float4 u = zero, au = zero, d = make_float4(1.f, 1.f, 1.f, 1.f);
        if (row_in && i < dk) {
          const float4 al = ld4(in.x + row * in.ld + (size_t)h * dk + i), wl = ld4(in.y + row * in.ldx + (size_t)h * dk + i);
          const float4 ab = ld4(in.xb + (size_t)h * dk + i), wb = ld4(in.yb + (size_t)h * dk + i);
          u = mul4(kr[j], kinv);
          au = make_float4(sigmoid_f(al.x + ab.x) * u.x, sigmoid_f(al.y + ab.y) * u.y, sigmoid_f(al.z + ab.z) * u.z, sigmoid_f(al.w + ab.w) * u.w);
          d = make_float4(expf(-in.s0 * sigmoid_f(wl.x + wb.x)), expf(-in.s0 * sigmoid_f(wl.y + wb.y)),
                          expf(-in.s0 * sigmoid_f(wl.z + wb.z)), expf(-in.s0 * sigmoid_f(wl.w + wb.w)));
        }
        st4(sm.ur + t * LD + i, u);
        st4(sm.ka + t * LD + i, kr[j]);
        st4(sm.ka + (CQ + t) * LD + i, au);
        st4(sm.ur + (CQ + t) * LD + i, qr[j]);
        st4(sm.a + t * LD + i, d);
      }
    }
    const float vf = GATED ? beta : 1.f;
    const float* vp = in.v + row * in.ld + (size_t)h * dv + blockIdx.y * NT;
    const int ncols = min(NT, dv - (int)blockIdx.y * NT);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + 4 * j;
      st4(sm.vs + t * LD + i, row_in && i < ncols ? mul4(ld4(vp + i), vf) : zero);
    }
  }
  __syncthreads();
  if (GATED) {
    if (tid < CQ) decay_windows(sm.g[tid], sm.win, sm.from, sm.rest, tid);
    __syncthreads();
    for (int e = tid; e < CQ * CQ; e += NTH) sm.w[(e / CQ) * LD + e % CQ] = decay_between(sm.win, e / CQ, e % CQ);
  } else {
    // a channel's decays in two threads: rows of u and r are decayed from the start, those of k and a*u back to it
    const int i = tid & 63;
    float p = 1.f;
    if (tid < 64) {
#pragma unroll 8
      for (int t = 0; t < ch.count; ++t) {
        const float d = sm.a[t * LD + i];
        sm.ur[t * LD + i] *= p;
        p *= d;
        sm.ur[(CQ + t) * LD + i] *= p;
      }
      sm.pc[i] = p;
    } else {
#pragma unroll 8
      for (int t = 0; t < ch.count; ++t) {
        p *= sm.a[t * LD + i];
        const float b = 1.0f / p;
        sm.ka[t * LD + i] *= b;
        sm.ka[(CQ + t) * LD + i] *= b;
      }
    }
  }
  __syncthreads();

  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  // ---- the four matrices: rows u, r against columns k, a*u (gated: a*u is a number times k).  A warp has the 32 tokens of u or of r
  // against those of k or of a*u, so that a piece that was cut serves two products (gated: 16 tokens against all of k); columns of
  // tokens above its own it leaves out
  {
    constexpr int MT = GATED ? 1 : 2;           // row tiles of 16
    const bool read = warp >= 2;
    const int r0 = read ? CQ : 0, t0 = GATED ? (warp & 1) * 16 : 0, c0 = GATED ? 0 : (warp & 1) * CQ;
    float big[MT][4][4] = {}, small[MT][4][4] = {};
#pragma unroll
    for (int k = 0; k < NT / 16; ++k) {
      uint32_t a[MT][3][4];
#pragma unroll
      for (int m = 0; m < MT; ++m) frag_rows(sm.ur + (r0 + t0 + 16 * m + g) * LD + k * 16 + 2 * q, LD, 1.f, 1.f, a[m]);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (8 * n <= t0 + 16 * MT - 1) {
          uint32_t b[3][2];
          frag_columns(sm.ka + (c0 + 8 * n + g) * LD + k * 16 + 2 * q, b);
#pragma unroll
          for (int m = 0; m < MT; ++m)
            if (8 * n <= t0 + 16 * m + 15) mma_split(big[m][n], small[m][n], a[m], b);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = t0 + 16 * m + g + 8 * (e >> 1), s = 8 * n + 2 * q + (e & 1);
          const bool in_tri = (read ? s <= t : s < t) && t < ch.count;
          float x = in_tri ? big[m][n][e] + small[m][n][e] : 0.f;
          float* dst = sm.a + (r0 + t) * LD + c0 + s;
          if (GATED) {
            x *= in_tri ? sm.w[(read ? t : t - 1) * LD + s] : 0.f;
            dst[CQ] = in_tri ? x * sm.gb[s] : 0.f;
          }
          *dst = x;
        }
  }
  // (what is not finite would spread through products with zeros: such a chunk takes FMAs that leave out what is above the diagonal)
  bool ordinary = true;
#pragma unroll
  for (int j = 0; j < CQ * NT / 4 / NTH; ++j) {
    const int e = tid + j * NTH;
    ordinary = ordinary && finite4(ld4(sm.vs + (e / (NT / 4)) * LD + (e % (NT / 4)) * 4));
  }
  ordinary = __syncthreads_and(ordinary);
  if (GATED) {
    // rows decayed from the chunk's start and to its end (the products' last row), which the matrices did not want
    for (int e = tid; e < CQ * (NT / 4); e += NTH) {
      const int t = e / (NT / 4), i = (e % (NT / 4)) * 4;
      const float f = sm.from[t], fb = t ? sm.from[t - 1] : 1.f, to = sm.w[(CQ - 1) * LD + t];
      st4(sm.ur + t * LD + i, mul4(ld4(sm.ur + t * LD + i), fb));
      st4(sm.ur + (CQ + t) * LD + i, mul4(ld4(sm.ur + (CQ + t) * LD + i), f));
      const float4 k = mul4(ld4(sm.ka + t * LD + i), to);
      st4(sm.ka + t * LD + i, k);
      st4(sm.ka + (CQ + t) * LD + i, mul4(k, sm.gb[t]));
    }
    __syncthreads();
  }

  // ---- [Auk ; Ark] V: into w, and over the k columns of the matrices (Ark V's columns 32 and up where Ark was).  A warp has the 32
  // rows of one of the two by half of the columns
  const bool lower = warp >= 2;
  const int d0 = (warp & 1) * (NT / 2);
  {
    float big[2][4][4] = {}, small[2][4][4] = {};
    const float* rows = sm.a + (lower ? CQ : 0) * LD;
    if (ordinary) {
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        uint32_t a[2][3][4];
#pragma unroll
        for (int m = k; m < 2; ++m) frag_rows(rows + (16 * m + g) * LD + k * 16 + 2 * q, LD, 1.f, 1.f, a[m]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          uint32_t b[3][2];
          frag_k(sm.vs + (k * 16 + 2 * q) * LD + d0 + 8 * n + g, LD, b);
#pragma unroll
          for (int m = k; m < 2; ++m) mma_split(big[m][n], small[m][n], a[m], b);
        }
      }
    } else {
      for (int s = 0; s < CQ; ++s)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = 16 * m + g + 8 * (e >> 1);
            if (lower ? s > t : s >= t) continue;
            const float x = rows[t * LD + s];
#pragma unroll
            for (int n = 0; n < 4; ++n) big[m][n][e] = fmaf(x, sm.vs[s * LD + d0 + 8 * n + 2 * q + (e & 1)], big[m][n][e]);
          }
    }
    __syncthreads();            // everyone has read the k columns of the matrices
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = 16 * m + g + 8 * i, d = d0 + 8 * n + 2 * q;
          float* dst = lower ? sm.a + (t + (d >= CQ ? CQ : 0)) * LD + (d & (CQ - 1)) : sm.w + t * LD + d;
          *reinterpret_cast<float2*>(dst) =
              make_float2(big[m][n][2 * i] + small[m][n][2 * i], big[m][n][2 * i + 1] + small[m][n][2 * i + 1]);
        }
  }
  __syncthreads();

  // ---- (I + Auu) [X | W] = [U~ | Auk V]: a column a thread, in place
  {
    float* col = tid < NT ? sm.ur + tid : sm.w + (tid - NT);
    const float* tri = sm.a + CQ;
    float x[CQ];
#pragma unroll
    for (int t = 0; t < CQ; ++t) x[t] = col[t * LD];
#pragma unroll
    for (int t = 1; t < CQ; ++t) {
      float s0 = x[t], s1 = 0.f;
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 a = ld4(tri + t * LD + s);        // 0 from s = t on
        s0 = fmaf(-a.x, x[s], s0);
        if (s + 1 < t) s1 = fmaf(-a.y, x[s + 1], s1);
        if (s + 2 < t) s0 = fmaf(-a.z, x[s + 2], s0);
        if (s + 3 < t) s1 = fmaf(-a.w, x[s + 3], s1);
      }
      x[t] = s0 + s1;
    }
#pragma unroll
    for (int t = 1; t < CQ; ++t) col[t * LD] = x[t];
#pragma unroll
    for (int t = 0; t < CQ; ++t) ordinary = ordinary && fabsf(x[t]) < CUDART_INF_F;
  }
  ordinary = __syncthreads_and(ordinary);

  const size_t item = (size_t)c * H + h;
  const int col0 = blockIdx.y * NT, ncols = min(NT, dv - col0);
  // ---- Rq = R~ - Aru X,  Ov = Ark V - Aru W: a warp has the 32 tokens of one of the two by half of the columns
  {
    const float* xw = lower ? sm.w : sm.ur;
    const float* rows = sm.a + CQ * LD + CQ;
    float big[2][4][4] = {}, small[2][4][4] = {};
    if (ordinary) {
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        uint32_t a[2][3][4];
#pragma unroll
        for (int m = k; m < 2; ++m) frag_rows(rows + (16 * m + g) * LD + k * 16 + 2 * q, LD, -1.f, -1.f, a[m]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          uint32_t b[3][2];
          frag_k(xw + (k * 16 + 2 * q) * LD + d0 + 8 * n + g, LD, b);
#pragma unroll
          for (int m = k; m < 2; ++m) mma_split(big[m][n], small[m][n], a[m], b);
        }
      }
    } else {
      for (int s = 0; s < CQ; ++s)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = 16 * m + g + 8 * (e >> 1);
            if (s > t) continue;
            const float x = -rows[t * LD + s];
#pragma unroll
            for (int n = 0; n < 4; ++n) big[m][n][e] = fmaf(x, xw[s * LD + d0 + 8 * n + 2 * q + (e & 1)], big[m][n][e]);
          }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = 16 * m + g + 8 * i, d = d0 + 8 * n + 2 * q;
          const float2 onto = *reinterpret_cast<const float2*>(lower ? sm.a + (t + (d >= CQ ? CQ : 0)) * LD + (d & (CQ - 1)) : sm.ur + (CQ + t) * LD + d);
          const float2 y = make_float2(onto.x + (big[m][n][2 * i] + small[m][n][2 * i]), onto.y + (big[m][n][2 * i + 1] + small[m][n][2 * i + 1]));
          if (!lower) {
            if (blockIdx.y == 0) *reinterpret_cast<float2*>(rq + (item * CQ + t) * NT + d) = y;
          } else if (t < ch.count && d < ncols) {
            *reinterpret_cast<float2*>(out + ((size_t)(ch.row0 + t) * H + h) * dv + col0 + d) = y;
          }
        }
  }
  // ---- M = -AU'^T X and P,  B = K'^T V - AU'^T W: a warp has 32 rows by half of the columns
  {
    const int row0 = (warp >> 1) * 32 + g;
    uint32_t kk[2][CQ / 16][3][4], au[2][CQ / 16][3][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        frag_turned(sm.ka + (k * 16 + 2 * q) * LD + row0 + 16 * m, LD, 1.f, kk[m][k]);
        frag_turned(sm.ka + (CQ + k * 16 + 2 * q) * LD + row0 + 16 * m, LD, -1.f, au[m][k]);
      }
#pragma unroll 1
    for (int n = 0; n < 4; ++n) {
      float mb[2][4] = {}, ms[2][4] = {}, vb[2][4] = {}, vsm[2][4] = {};
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        const int at = (k * 16 + 2 * q) * LD + d0 + 8 * n + g;
        uint32_t b[3][2];
        frag_k(sm.ur + at, LD, b);
#pragma unroll
        for (int m = 0; m < 2; ++m) mma_split(mb[m], ms[m], au[m][k], b);
        frag_k(sm.vs + at, LD, b);
#pragma unroll
        for (int m = 0; m < 2; ++m) mma_split(vb[m], vsm[m], kk[m][k], b);
        frag_k(sm.w + at, LD, b);
#pragma unroll
        for (int m = 0; m < 2; ++m) mma_split(vb[m], vsm[m], au[m][k], b);
      }
      const int d = d0 + 8 * n + 2 * q;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int row = row0 + 16 * m + 8 * i;
          const float f = GATED ? 1.f : sm.pc[row];
          if (blockIdx.y == 0)
            *reinterpret_cast<float2*>(mm + item * MFLOATS + row * NT + d) =
                make_float2((mb[m][2 * i] + ms[m][2 * i]) * f, (mb[m][2 * i + 1] + ms[m][2 * i + 1]) * f);
          if (row < dk && d < ncols)
            *reinterpret_cast<float2*>(bb + (item * dk + row) * dv + col0 + d) =
                make_float2((vb[m][2 * i] + vsm[m][2 * i]) * f, (vb[m][2 * i + 1] + vsm[m][2 * i + 1]) * f);
        }
    }
    if (blockIdx.y == 0 && tid < NT) mm[item * MFLOATS + NT * NT + tid] = GATED ? sm.from[CQ - 1] : sm.pc[tid];
  }
}

// ------------------------------------------------------------------ rules without a removal term
// Retention (q, k turned by position, k times a factor, one decay per head) and the matrix memory (q times a factor, k times
// the token's input gate, the forget gate as decay; columns dv and up of the padded value: 1, then zeros).  Nothing here is a
// chain but the states' sum over chunks, so:
//   1. states:  a block per (chunk, head) makes B = K'^T V and the chunk's decay;
//   2. carry:   a thread per four state entries goes through a request's chunks and leaves every chunk's start state in B's place;
//   3. outputs: a block per (chunk, head) makes A V + R~ S_0.
// (As two kernels, the second walking the chunks with the outputs' products, one request of 2,048 tokens at 64 heads of 64 took
// 103 + 141 us, the walk bound by the latency of a chain that these three do not have.)  A block of the outputs waits for memory and for
// its decays (17,000 of its 24,600 clocks before the windows of `decay_windows`, the products 6,700).
struct DecayIn {
  const float *q, *k, *v;
  long long ld;
  const float *cos_t, *sin_t;   // retention
  const int* positions;
  int rot;
  const float* decay;           // retention: [H]
  const float* gates;           // matrix memory: [n, H, 3]
  float scale;                  // retention: k's factor; matrix memory: q's
  int H, dk, dv, dvp;           // dvp: the state's columns (retention: dv)
};

namespace {
constexpr int LA = CQ + 4;
struct StatesSmem {
  float k[CQ * LD], vs[CQ * LD];
  float from[CQ], rest[4];
  double win[5 * CQ];
};
struct OutSmem {
  float q[CQ * LD], k[CQ * LD], vs[CQ * LD], a[CQ * LA], st[NT * LD];     // (behind a row's NT numbers four more columns fit)
  float from[CQ], rest[4];
  double win[5 * CQ];
};
// The columns of a pass from col0 on: the last ones go along if they fit into the rows of shared memory.
__device__ __forceinline__ int pass_columns(int left) { return left <= LD ? left : NT; }

// A chunk's q (or none), k and first value columns, and the windows of its decays.  Ends behind a barrier.
template <bool MEMORY, bool WITH_Q, typename S>
__device__ __forceinline__ void decay_rows(const DecayIn& in, const Chunk& ch, int h, S& sm, float* sq) {
  const int H = in.H, dk = in.dk, dv = in.dv, tid = threadIdx.x;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int t = tid >> 2, i0 = (tid & 3) * 16;
  const bool row_in = t < ch.count;
  const size_t row = (size_t)(ch.row0 + (row_in ? t : 0));
  const float* kp = in.k + row * in.ld + (size_t)h * dk;
  const float* qp = in.q + row * in.ld + (size_t)h * dk;
  const float* vp = in.v + row * in.ld + (size_t)h * dv;
  const float kf = MEMORY ? (row_in ? in.gates[(row * H + h) * 3 + 1] : 1.f) : in.scale;
  float4 kr[4], qr[4], vr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = i0 + 4 * j;
    kr[j] = row_in && i < dk ? ld4(kp + i) : zero;
    if (WITH_Q) qr[j] = row_in && i < dk ? ld4(qp + i) : zero;
    vr[j] = row_in && i < min(NT, dv) ? ld4(vp + i) : zero;
  }
  // turned below, a pair of dims (i, i + rot / 2) a thread: the angles are asked for here
  constexpr int PAIRS = CQ * (NT / 2) / NTH;
  const int half = MEMORY ? 0 : in.rot >> 1;
  float cs[PAIRS], sn[PAIRS];
  if (!MEMORY)
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
      const int e = tid + j * NTH, r = half ? e / half : CQ;
      const bool turned = r < ch.count;
      const size_t at = turned ? (size_t)in.positions[ch.row0 + r] * half + (e - r * half) : 0;
      cs[j] = turned ? in.cos_t[at] : 1.f;
      sn[j] = turned ? in.sin_t[at] : 0.f;
    }
  if (tid < CQ) {
    const bool has = tid < ch.count;
    decay_windows(!has ? 1.f : MEMORY ? in.gates[((size_t)(ch.row0 + tid) * H + h) * 3] : in.decay[h], sm.win, sm.from, sm.rest, tid);
  } else if (tid < 2 * CQ) {    // columns NT and up, where they go along with the first pass (the matrix memory's first one past dv: 1)
    const int r = tid - CQ;
    float4 x = zero;
    if (r < ch.count) {
      if (dv > NT) x = ld4(in.v + (size_t)(ch.row0 + r) * in.ld + (size_t)h * dv + NT);
      else if (MEMORY && dv == NT) x.x = 1.f;
    }
    st4(sm.vs + r * LD + NT, x);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = i0 + 4 * j;
    st4(sm.k + t * LD + i, MEMORY ? mul4(kr[j], kf) : kr[j]);
    if (WITH_Q) st4(sq + t * LD + i, MEMORY ? mul4(qr[j], in.scale) : qr[j]);
    st4(sm.vs + t * LD + i, vr[j]);
  }
  __syncthreads();
  if (MEMORY && dv < NT)
    for (int r = tid; r < ch.count; r += NTH) sm.vs[r * LD + dv] = 1.f;
  if (!MEMORY) {
    // in place, k times its factor
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
      const int e = tid + j * NTH, r = half ? e / half : CQ;
      if (r >= ch.count) break;
      float* k = sm.k + r * LD + e - r * half;
      const float k0 = k[0], k1 = k[half];
      k[0] = (k0 * cs[j] - k1 * sn[j]) * kf;
      k[half] = (k1 * cs[j] + k0 * sn[j]) * kf;
      if (WITH_Q) {
        float* q = sq + r * LD + e - r * half;
        const float q0 = q[0], q1 = q[half];
        q[0] = q0 * cs[j] - q1 * sn[j];
        q[half] = q1 * cs[j] + q0 * sn[j];
      }
    }
    const int plain = dk - in.rot;
    for (int e = tid; e < CQ * plain; e += NTH) sm.k[(e / plain) * LD + in.rot + e % plain] *= kf;
  }
  __syncthreads();
}

// The value columns from col0 on (and the matrix memory's column of ones); zeros up to LD.
template <bool MEMORY>
__device__ __forceinline__ void next_columns(const DecayIn& in, const Chunk& ch, int h, int col0, float* vs) {
  for (int e = threadIdx.x; e < CQ * LD; e += NTH) {
    const int t = e / LD, d = col0 + e % LD;
    float x = 0.f;
    if (t < ch.count) x = d < in.dv ? in.v[(size_t)(ch.row0 + t) * in.ld + (size_t)h * in.dv + d] : MEMORY && d == in.dv ? 1.f : 0.f;
    vs[e] = x;
  }
}
}  // namespace

template <bool MEMORY>
__global__ void __launch_bounds__(NTH)
decay_states_kernel(const DecayIn in, const Chunk* __restrict__ chunks, float2* __restrict__ pp, float* __restrict__ bb) {
  __shared__ __align__(16) StatesSmem sm;
  const int H = in.H, dk = in.dk, dvp = in.dvp;
  const int c = blockIdx.x / H, h = blockIdx.x % H;
  const Chunk ch = chunks[c];
  const int tid = threadIdx.x;
  const size_t item = (size_t)c * H + h;
  decay_rows<MEMORY, false>(in, ch, h, sm, nullptr);
  if (tid == 0) pp[item] = make_float2(sm.from[CQ - 1], sm.rest[0]);
  // a warp has 16 rows of the state, all columns
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  uint32_t a[CQ / 16][3][4];
#pragma unroll
  for (int k = 0; k < CQ / 16; ++k) {
    float to[10];               // the decays from the lane's tokens to the chunk's end
#pragma unroll
    for (int e = 0; e < 4; ++e) to[8 * (e >> 1) + (e & 1)] = decay_between(sm.win, CQ - 1, k * 16 + 2 * q + 8 * (e >> 1) + (e & 1));
    frag_turned(sm.k + (k * 16 + 2 * q) * LD + warp * 16 + g, LD, to, a[k]);
  }
  for (int col0 = 0, ncols; col0 < dvp; col0 += ncols) {
    ncols = pass_columns(dvp - col0);
    if (col0) {
      __syncthreads();
      next_columns<MEMORY>(in, ch, h, col0, sm.vs);
      __syncthreads();
    }
#pragma unroll 2
    for (int n = 0; n < (ncols + 7) / 8; ++n) {
      float big[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        uint32_t v[3][2];
        frag_k(sm.vs + (k * 16 + 2 * q) * LD + 8 * n + g, LD, v);
        mma_split(big, small, a[k], v);
      }
      const int d = 8 * n + 2 * q;
      if (d < ncols)            // (dvp is a multiple of 4)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int row = warp * 16 + g + 8 * i;
          if (row < dk)
            *reinterpret_cast<float2*>(bb + (item * dk + row) * dvp + col0 + d) = make_float2(big[2 * i] + small[2 * i], big[2 * i + 1] + small[2 * i + 1]);
        }
    }
  }
}

// A thread owns four state entries of a request and head.  Eight chunks' B and decays are asked for at once.
__global__ void __launch_bounds__(NTH)
decay_carry_kernel(const Request* __restrict__ requests, const float2* __restrict__ pp, float* __restrict__ bb, float* __restrict__ state,
                   int H, int entries) {
  const Request rq = requests[blockIdx.x / H];
  const int h = blockIdx.x % H, e = (blockIdx.y * NTH + threadIdx.x) * 4;
  if (e >= entries) return;
  float* sp = state + ((size_t)rq.slot * H + h) * entries + e;
  float* bp = bb + ((size_t)rq.chunk0 * H + h) * entries + e;
  const float2* p = pp + (size_t)rq.chunk0 * H + h;
  float4 s = ld4(sp);
  constexpr int AT_ONCE = 8;
  for (int c0 = 0; c0 < rq.chunks; c0 += AT_ONCE) {
    float4 x[AT_ONCE];
    float2 d[AT_ONCE];
#pragma unroll
    for (int j = 0; j < AT_ONCE; ++j)
      if (c0 + j < rq.chunks) {
        x[j] = ld4(bp + (size_t)(c0 + j) * H * entries);
        d[j] = p[(size_t)(c0 + j) * H];
      }
#pragma unroll
    for (int j = 0; j < AT_ONCE; ++j)
      if (c0 + j < rq.chunks) {
        st4(bp + (size_t)(c0 + j) * H * entries, s);
        fma4(x[j], d[j].y, s);
        fma4(x[j], d[j].x, s);
        s = x[j];
      }
  }
  st4(sp, s);
}

template <bool MEMORY>
__global__ void __launch_bounds__(NTH)
decay_out_kernel(const DecayIn in, const Chunk* __restrict__ chunks, const float* __restrict__ start, float* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  OutSmem& sm = *reinterpret_cast<OutSmem*>(smem_raw);
  const int H = in.H, dk = in.dk, dvp = in.dvp;
  const int c = blockIdx.x / H, h = blockIdx.x % H;
  const Chunk ch = chunks[c];
  const int tid = threadIdx.x;
  const float* sp = start + ((size_t)c * H + h) * dk * dvp;
  auto fetch_state = [&](int col0) {            // its columns from col0 on; what does not exist as zeros
    for (int e = tid; e < NT * (LD / 4); e += NTH) {
      const int i = e / (LD / 4), d = (e % (LD / 4)) * 4;
      const bool ok = i < dk && col0 + d < dvp;
      cp_async16_or_zero(sm.st + i * LD + d, ok ? sp + (size_t)i * dvp + col0 + d : sp, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch_state(0);
  decay_rows<MEMORY, true>(in, ch, h, sm, sm.q);
  // a warp has 16 tokens, and half of the keys (columns)
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, t0 = (warp & 1) * 16, side = warp >> 1;
  const float f0 = sm.from[t0 + g], f1 = sm.from[t0 + g + 8];
  // ---- A = (q k^T) times the decays between the tokens (keys 16 and up concern no token below them)
  if (side == 0 || t0) {
    float big[2][4] = {}, small[2][4] = {};
#pragma unroll
    for (int k = 0; k < NT / 16; ++k) {
      uint32_t a[3][4];
      frag_rows(sm.q + (t0 + g) * LD + k * 16 + 2 * q, LD, 1.f, 1.f, a);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        uint32_t b[3][2];
        frag_columns(sm.k + (side * 16 + 8 * n + g) * LD + k * 16 + 2 * q, b);
        mma_split(big[n], small[n], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = t0 + g + 8 * (e >> 1), s = side * 16 + 8 * n + 2 * q + (e & 1);
        sm.a[t * LA + s] = s <= t ? (big[n][e] + small[n][e]) * decay_between(sm.win, t, s) : 0.f;
      }
  } else {
    for (int e = lane; e < 16 * 16; e += 32) sm.a[(e >> 4) * LA + 16 + (e & 15)] = 0.f;
  }
  for (int col0 = 0, ncols; col0 < dvp; col0 += ncols) {
    ncols = pass_columns(dvp - col0);
    if (col0) {
      __syncthreads();
      fetch_state(col0);
      next_columns<MEMORY>(in, ch, h, col0, sm.vs);
      __syncthreads();
    }
    // a product with zeros above the diagonal would bring a value that is not finite to earlier tokens: such a chunk takes FMAs
    bool ordinary = true;
    for (int e = tid; e < CQ * LD / 4; e += NTH) ordinary = ordinary && finite4(ld4(sm.vs + 4 * e));
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const bool all = __syncthreads_and(ordinary);          // and the state and A are there
    if (all) {
      const int tiles = (ncols + 7) / 8;
      constexpr int NJ = (LD / 8 + 2) / 2;                  // column tiles side, side + 2, ..
      float big[NJ][4] = {}, small[NJ][4] = {};
#pragma unroll
      for (int k = 0; k < CQ / 16; ++k) {
        if (16 * k > t0) break;
        uint32_t a[3][4];
        frag_rows(sm.a + (t0 + g) * LA + k * 16 + 2 * q, LA, 1.f, 1.f, a);
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (side + 2 * j < tiles) {
            uint32_t b[3][2];
            frag_k(sm.vs + (k * 16 + 2 * q) * LD + (side + 2 * j) * 8 + g, LD, b);
            mma_split(big[j], small[j], a, b);
          }
      }
#pragma unroll
      for (int k = 0; k < NT / 16; ++k) {
        uint32_t a[3][4];
        frag_rows(sm.q + (t0 + g) * LD + k * 16 + 2 * q, LD, f0, f1, a);
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (side + 2 * j < tiles) {
            uint32_t b[3][2];
            frag_k(sm.st + (k * 16 + 2 * q) * LD + (side + 2 * j) * 8 + g, LD, b);
            mma_split(big[j], small[j], a, b);
          }
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int d = (side + 2 * j) * 8 + 2 * q;
        if (d < ncols)          // (dvp is a multiple of 4)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int t = t0 + g + 8 * i;
            if (t < ch.count)
              *reinterpret_cast<float2*>(out + ((size_t)(ch.row0 + t) * H + h) * dvp + col0 + d) =
                  make_float2(big[j][2 * i] + small[j][2 * i], big[j][2 * i + 1] + small[j][2 * i + 1]);
          }
      }
      continue;
    }
    for (int e = tid; e < CQ * ncols; e += NTH) {
      const int t = e / ncols, d = e % ncols;
      float x = 0.f, y = 0.f;
      for (int s = 0; s <= t; ++s) x = fmaf(sm.a[t * LA + s], sm.vs[s * LD + d], x);
#pragma unroll 8
      for (int i = 0; i < NT; ++i) y = fmaf(sm.q[t * LD + i] * sm.from[t], sm.st[i * LD + d], y);
      if (t < ch.count) out[((size_t)(ch.row0 + t) * H + h) * dvp + col0 + d] = x + y;
    }
  }
}

// ------------------------------------------------------------------ 2. walk
// S <- P S + (M S + B) and O = Rq S + Ov over a request's chunks.  A block owns DVS value columns of a head and has a warp per 16 rows
// of [M ; Rq].  The four warps of M keep S in float32 registers (the tensor core's result layout) and leave its pieces in shared memory, two copies in
// turn, for all six; what a chunk brings comes through a ring, a chunk ahead.
// One request of 2,048 tokens at 64 heads of 64 x 64: 173 us with multiply-adds (7 wide loads of shared memory for 24 pairs of them were
// the bound), 117 with the pieces, 107 here, where a chunk's copies take one address a round of rows (issue slots 53 % before that,
// tensor pipe 32 %: the pieces again).
namespace {
template <int DVS>
struct WalkShape {
  static constexpr int ROWS = NT + CQ;                                 // rows of [M ; Rq]
  static constexpr int LM = NT + 8, LO = DVS + 8, LS = NT + 8;         // numbers between rows: neighbouring rows in other banks
  static constexpr int OFF = ROWS * LM, P = OFF + ROWS * LO;           // [B ; Ov] and P behind them
  static constexpr int STAGE = P + NT;
  static constexpr int STAGES = 2, THREADS = ROWS / 16 * 32;           // (two blocks an SM; three stages would leave one)
  static constexpr int PLANE = DVS * LS;                               // bf16 of one piece of S, column by column
  static constexpr size_t SMEM = (size_t)STAGES * STAGE * sizeof(float) + (size_t)2 * 3 * PLANE * sizeof(bf16);
};
}  // namespace

template <int DVS>
__global__ void __launch_bounds__(WalkShape<DVS>::THREADS, 2)
chunk_walk_kernel(const Request* __restrict__ requests, const Chunk* __restrict__ chunks, const float* __restrict__ mm,
                  const float* __restrict__ rq, const float* __restrict__ bb, float* __restrict__ state, float* __restrict__ out,
                  int H, int dk, int dv) {
  using K = WalkShape<DVS>;
  constexpr int NN = DVS / 8;                   // column tiles
  extern __shared__ __align__(16) float ws[];
  bf16* planes = reinterpret_cast<bf16*>(ws + K::STAGES * K::STAGE);
  const Request r = requests[blockIdx.x / H];
  const int h = blockIdx.x % H, col0 = blockIdx.y * DVS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  float* sp = state + ((size_t)r.slot * H + h) * dk * dv;
  const int row0 = chunks[r.chunk0].row0, rows = CQ * (r.chunks - 1) + chunks[r.chunk0 + r.chunks - 1].count;
  // a chunk's copies, chunk after chunk: a thread has the same columns of rows that lie a fixed number apart
  constexpr int RM = K::THREADS / (NT / 4), RB = K::THREADS / (DVS / 4);
  static_assert(K::ROWS % RM == 0 && K::ROWS % RB == 0, "whole rounds of rows");
  const int mr = tid / (NT / 4), br = tid / (DVS / 4), bd = (tid % (DVS / 4)) * 4;
  const float* mp = mm + ((size_t)r.chunk0 * H + h) * MFLOATS + tid * 4;
  const float* qp = rq + ((size_t)r.chunk0 * H + h) * CQ * NT + tid * 4;
  const float* bp = bb + (((size_t)r.chunk0 * H + h) * dk + br) * dv + col0 + bd;
  const float* op = out + ((size_t)row0 * H + h) * dv + col0 + bd;
  const bool bcol = col0 + bd < dv;
  auto fetch = [&](int c) {
    float* st = ws + (c % K::STAGES) * K::STAGE;
#pragma unroll
    for (int j = 0; j < K::ROWS / RM; ++j)
      cp_async16(st + (mr + j * RM) * K::LM + (tid % (NT / 4)) * 4, mr + j * RM < NT ? mp + j * K::THREADS * 4 : qp + j * K::THREADS * 4 - NT * NT);
    if (tid < NT / 4) cp_async16(st + K::P + 4 * tid, mp + NT * NT);
#pragma unroll
    for (int j = 0; j < K::ROWS / RB; ++j) {
      const int row = br + j * RB, t = c * CQ + row - NT;
      const bool in = bcol && (row < NT ? row < dk : t < rows);
      const float* src = row < NT ? bp + (size_t)(j * RB) * dv : op + (ptrdiff_t)t * H * dv;
      cp_async16_or_zero(st + K::OFF + row * K::LO + bd, in ? src : bb, in);
    }
    mp += (size_t)H * MFLOATS;
    qp += (size_t)H * CQ * NT;
    bp += (size_t)H * dk * dv;
  };
#pragma unroll
  for (int c = 0; c < K::STAGES - 1; ++c) {
    if (c < r.chunks) fetch(c);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // a lane's entries of S: rows mrow and mrow + 8, columns 8 n + 2 q and the next
  const bool moves = warp < NT / 16;
  const int mrow = warp * 16 + g;
  float S[NN][4];
  auto publish = [&](int copy) {
    bf16* p = planes + (size_t)copy * 3 * K::PLANE;
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float x = S[n][e];
        bf16* at = p + (8 * n + 2 * q + (e & 1)) * K::LS + mrow + 8 * (e >> 1);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const bf16 piece = k == 0 ? __ushort_as_bfloat16((unsigned short)pack_first(x, 0.f)) : __float2bfloat16_rn(x);
          at[k * K::PLANE] = piece;
          x -= __bfloat162float(piece);
        }
      }
  };
  if (moves) {
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = mrow + 8 * (e >> 1), d = col0 + 8 * n + 2 * q + (e & 1);
        S[n][e] = i < dk && d < dv ? sp[(size_t)i * dv + d] : 0.f;
      }
    publish(0);
  }
  for (int c = 0; c < r.chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(K::STAGES - 2) : "memory");
    __syncthreads();            // chunk c is there, S's pieces are written, and the stage of chunk c - 1 may be filled again
    if (c + K::STAGES - 1 < r.chunks) fetch(c + K::STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* st = ws + (c % K::STAGES) * K::STAGE;
    const bf16* sb = planes + (size_t)(c & 1) * 3 * K::PLANE + g * K::LS + 2 * q;
    float big[NN][4], small[NN][4];
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) big[n][e] = small[n][e] = 0.f;
    const float* ap = st + mrow * K::LM + 2 * q;
#pragma unroll
    for (int k = 0; k < NT / 16; ++k) {
      uint32_t a[3][4];
      frag_rows(ap + k * 16, K::LM, 1.f, 1.f, a);
#pragma unroll
      for (int n = 0; n < NN; ++n) {
        uint32_t b[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            b[p][e] = *reinterpret_cast<const uint32_t*>(sb + p * K::PLANE + n * 8 * K::LS + k * 16 + 8 * e);
        mma_split(big[n], small[n], a, b);
      }
    }
    const float* off = st + K::OFF + mrow * K::LO + 2 * q;
    if (moves) {
      const float p0 = st[K::P + mrow], p1 = st[K::P + mrow + 8];
#pragma unroll
      for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 o = *reinterpret_cast<const float2*>(off + 8 * i * K::LO + 8 * n);
          S[n][2 * i] = fmaf(i ? p1 : p0, S[n][2 * i], big[n][2 * i] + small[n][2 * i] + o.x);
          S[n][2 * i + 1] = fmaf(i ? p1 : p0, S[n][2 * i + 1], big[n][2 * i + 1] + small[n][2 * i + 1] + o.y);
        }
      publish((c + 1) & 1);
    } else {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = c * CQ + mrow + 8 * i - NT;
        if (t >= rows) continue;
        float* o = out + ((size_t)(row0 + t) * H + h) * dv + col0 + 2 * q;
#pragma unroll
        for (int n = 0; n < NN; ++n) {
          const float2 v = *reinterpret_cast<const float2*>(off + 8 * i * K::LO + 8 * n);
          if (col0 + 8 * n + 2 * q < dv)        // (dv is a multiple of 4)
            *reinterpret_cast<float2*>(o + 8 * n) = make_float2(big[n][2 * i] + small[n][2 * i] + v.x, big[n][2 * i + 1] + small[n][2 * i + 1] + v.y);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (moves)
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = mrow + 8 * (e >> 1), d = col0 + 8 * n + 2 * q + (e & 1);
        if (i < dk && d < dv) sp[(size_t)i * dv + d] = S[n][e];
      }
}

namespace {

template <int DVS>
int run_walk(const int* requests, int n_requests, const int* chunks, const float* mm, const float* rq, const float* bb, float* state,
             float* out, int H, int dk, int dv, cudaStream_t s) {
  using K = WalkShape<DVS>;
  if (int e = hk_allow_smem<chunk_walk_kernel<DVS>>(K::SMEM)) return e;
  return hk_launch(chunk_walk_kernel<DVS>, dim3((unsigned)(n_requests * H), (unsigned)((dv + DVS - 1) / DVS)), dim3(K::THREADS), K::SMEM,
                   s, (const Request*)requests, (const Chunk*)chunks, mm, rq, bb, state, out, H, dk, dv);
}

bool sizes_fit(int H, int dk, int dv, int dvp) { return H >= 1 && dk >= 4 && dk <= NT && !(dk & 3) && dv >= 4 && !(dv & 3) && !(dvp & 3); }

template <bool GATED>
int run_delta(const DeltaIn& in, const int* chunks, int n_chunks, const int* requests, int n_requests, float* scratch, float* state,
              float* out, cudaStream_t s) {
  float* rq = scratch;
  float* mm = rq + (size_t)n_chunks * in.H * CQ * NT;
  float* bb = mm + (size_t)n_chunks * in.H * MFLOATS;
  if (int e = hk_allow_smem<delta_local_kernel<GATED>>(sizeof(DeltaSmem))) return e;
  if (int e = hk_launch(delta_local_kernel<GATED>, dim3((unsigned)(n_chunks * in.H), (unsigned)((in.dv + NT - 1) / NT)), dim3(NTH), sizeof(DeltaSmem),
                        s, in, (const Chunk*)chunks, mm, rq, bb, out))
    return e;
  // 32 columns a block read M and Rq half as often as 16; 16 where 32 would leave SMs idle
  if ((long long)n_requests * in.H * ((in.dv + 31) / 32) >= 148)
    return run_walk<32>(requests, n_requests, chunks, mm, rq, bb, state, out, in.H, in.dk, in.dv, s);
  return run_walk<16>(requests, n_requests, chunks, mm, rq, bb, state, out, in.H, in.dk, in.dv, s);
}

template <bool MEMORY>
int run_decay(const DecayIn& in, const int* chunks, int n_chunks, const int* requests, int n_requests, float* scratch, float* state,
              float* out, cudaStream_t s) {
  float2* pp = reinterpret_cast<float2*>(scratch);
  float* bb = scratch + (((size_t)n_chunks * in.H * 2 + 3) & ~(size_t)3);
  const dim3 grid((unsigned)(n_chunks * in.H));
  const int entries = in.dk * in.dvp;
  if (int e = hk_launch(decay_states_kernel<MEMORY>, grid, dim3(NTH), 0, s, in, (const Chunk*)chunks, pp, bb)) return e;
  if (int e = hk_launch(decay_carry_kernel, dim3((unsigned)(n_requests * in.H), (unsigned)((entries / 4 + NTH - 1) / NTH)), dim3(NTH), 0, s,
                        (const Request*)requests, (const float2*)pp, bb, state, in.H, entries))
    return e;
  if (int e = hk_allow_smem<decay_out_kernel<MEMORY>>(sizeof(OutSmem))) return e;
  return hk_launch(decay_out_kernel<MEMORY>, grid, dim3(NTH), sizeof(OutSmem), s, in, (const Chunk*)chunks, (const float*)bb, out);
}

}  // namespace

// Floats of scratch for `n_chunks` chunks (16-byte aligned); `removal`: a rule with a removal term.
HK_API long long hk_delta_chunks_scratch(int n_chunks, int H, int dk, int dvp, int removal) {
  const long long items = (long long)n_chunks * H;
  return items * dk * dvp + (removal ? items * (CQ * NT + MFLOATS) : ((items * 2 + 3) & ~3ll));
}

// The arguments of hk_delta_rule_scan, with chunks int32 [n_chunks, 2] = (first row, rows <= 32), a request's chunks one after
// the other and all but its last of 32 rows; requests int32 [n_requests, 3] = (state slot, first chunk, chunks).  Refuses
// (HK_ERR_UNSUPPORTED) keys above 64, sizes that are no multiple of 4, rows or pointers off a 16-byte boundary, and decays
// that could bring a chunk's product below 2^-64 (decay_scale above 1.38).
HK_API int hk_delta_rule_chunks(const float* r, const float* k, const float* v, const float* al, long long ld, const float* wl, long long ldw,
                                const float* a_bias, const float* w_bias, const int* chunks, int n_chunks, const int* requests,
                                int n_requests, float* scratch, float* state, float* out, int H, int dk, int dv, float decay_scale,
                                float key_eps, void* stream) {
  if (n_chunks <= 0 || n_requests <= 0) return 0;
  if (!sizes_fit(H, dk, dv, dv) || (ld & 3) || (ldw & 3) || !(decay_scale >= 0.f && decay_scale <= 1.38f)) return HK_ERR_UNSUPPORTED;
  if (((uintptr_t)r | (uintptr_t)k | (uintptr_t)v | (uintptr_t)al | (uintptr_t)wl | (uintptr_t)a_bias | (uintptr_t)w_bias | (uintptr_t)scratch |
       (uintptr_t)state | (uintptr_t)out) & 15)
    return HK_ERR_UNSUPPORTED;
  const DeltaIn in = {r, k, v, ld, al, wl, ldw, a_bias, w_bias, decay_scale, key_eps, H, H, dk, dv};
  return run_delta<false>(in, chunks, n_chunks, requests, n_requests, scratch, state, out, (cudaStream_t)stream);
}

// The arguments of hk_gated_delta_scan, chunks and requests as above.
HK_API int hk_gated_delta_chunks(const float* q, const float* k, const float* v, long long ld, const float* bl, const float* al, long long ldg,
                                 const float* a_log, const float* dt_bias, const int* chunks, int n_chunks, const int* requests,
                                 int n_requests, float* scratch, float* state, float* out, int H, int G, int dk, int dv, float q_scale,
                                 float unit_eps, void* stream) {
  if (n_chunks <= 0 || n_requests <= 0) return 0;
  if (!sizes_fit(H, dk, dv, dv) || G < 1 || H % G || (ld & 3)) return HK_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch | (uintptr_t)state | (uintptr_t)out) & 15) return HK_ERR_UNSUPPORTED;
  const DeltaIn in = {q, k, v, ld, bl, al, ldg, a_log, dt_bias, q_scale, unit_eps, H, G, dk, dv};
  return run_delta<true>(in, chunks, n_chunks, requests, n_requests, scratch, state, out, (cudaStream_t)stream);
}

// The arguments of hk_retention_scan, chunks and requests as above.
HK_API int hk_retention_chunks(const float* q, const float* k, const float* v, long long ld, const float* cos_t, const float* sin_t, int rot,
                               const int* positions, const float* decay, const int* chunks, int n_chunks, const int* requests,
                               int n_requests, float* scratch, float* state, float* out, int H, int dk, int dv, float k_scale,
                               void* stream) {
  if (n_chunks <= 0 || n_requests <= 0) return 0;
  if (!sizes_fit(H, dk, dv, dv) || (ld & 3) || rot < 0 || rot > dk || (rot & 1)) return HK_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch | (uintptr_t)state | (uintptr_t)out) & 15) return HK_ERR_UNSUPPORTED;
  const DecayIn in = {q, k, v, ld, cos_t, sin_t, positions, rot, decay, nullptr, k_scale, H, dk, dv, dv};
  return run_decay<false>(in, chunks, n_chunks, requests, n_requests, scratch, state, out, (cudaStream_t)stream);
}

// The matrix memory behind its gates (`gates` [n, H, 3] as hk_mlstm_gates leaves them); state [slots, H, dk, dvp], out [n, H dvp].
HK_API int hk_mlstm_chunks(const float* q, const float* k, const float* v, long long ld, const float* gates, const int* chunks, int n_chunks,
                           const int* requests, int n_requests, float* scratch, float* state, float* out, int H, int dk, int dv,
                           float q_scale, void* stream) {
  if (n_chunks <= 0 || n_requests <= 0) return 0;
  const int dvp = (dv + 1 + 3) & ~3;
  if (!sizes_fit(H, dk, dv, dvp) || (ld & 3)) return HK_ERR_UNSUPPORTED;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch | (uintptr_t)state | (uintptr_t)out) & 15) return HK_ERR_UNSUPPORTED;
  const DecayIn in = {q, k, v, ld, nullptr, nullptr, nullptr, 0, nullptr, gates, q_scale, H, dk, dv, dvp};
  return run_decay<true>(in, chunks, n_chunks, requests, n_requests, scratch, state, out, (cudaStream_t)stream);
}
