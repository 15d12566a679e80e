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
//   2. walk:   a block per (request, head, 16 or 32 value columns) goes through the request's chunks, S in shared memory.
// Without a removal term (retention, matrix memory) there is no M and no system to solve, and P is one number: see below.
// P S_0 is added last: what is summed before it is small where decays are weak, and rounds less.
//
// All arithmetic is float32 multiply-adds, decays are products of the tokens' decays (never differences of logarithms): an
// entry of the four matrices carries the rounding of the decays between its two tokens, as the walk token by token does.
// Where the decay is one number per token the products between every two tokens are made one by one; where it is one per
// channel (generalised delta rule) rows are scaled by P_t and 1 / P_s, which holds while a chunk's decay stays above 2^-64
// (the launcher's condition on decay_scale).
//
// A value, key, gate or decay that is NaN or Inf reaches its own token and later ones, as in the walk: the products with triangular
// matrices leave out what stands above the diagonal (`triangle_rows`), which a zero there would not keep out.
//
// One request of 2,048 tokens at 64 heads of 64 x 64 (walk token by token -> here, L2 cold): generalised rule 988 -> 433 us, gated
// rule 978 -> 402, matrix memory 1,074 -> 284, retention 605 -> 206; of 1,000 at 32 heads 390 -> 140, 390 -> 138, 417 -> 103,
// 241 -> 64; at 64 heads of 64 tokens level (42 -> 38, 46 -> 40, 54 -> 40, 32 -> 30), of 128 75 -> 48, 79 -> 48, 89 -> 46, 50 -> 36.
// (With the triangular products whole: 429, 400, 284, 212 at 2,048 tokens.)
// Relative error against 64 bits at 2,048 tokens: 5.3e-7 -> 5.1e-7, 5.5e-7 -> 5.3e-7, 7.1e-7 -> 7.0e-7, 5.2e-7 -> 1.9e-7.
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
__device__ __forceinline__ float at4(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}
// two multiply-adds at once, each rounded as fmaf rounds
__device__ __forceinline__ ulonglong2 ld_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ void fma_pairs(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(unsigned long long c) {
  return __uint_as_float((uint32_t)c) + __uint_as_float((uint32_t)(c >> 32));
}
// the same as dot4 in two sums
__device__ __forceinline__ void dot4_by_two(float4 a, float4 b, float* c) {
  c[0] = fmaf(a.z, b.z, fmaf(a.x, b.x, c[0]));
  c[1] = fmaf(a.w, b.w, fmaf(a.y, b.y, c[1]));
}
__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void fma4(float4& c, float a, float4 b) {
  c.x = fmaf(a, b.x, c.x);
  c.y = fmaf(a, b.y, c.y);
  c.z = fmaf(a, b.z, c.z);
  c.w = fmaf(a, b.w, c.w);
}

// acc[i] (N rows, row i's token ty + 8 (i & 3)) += sign * a[row i, s] * b[s, :] over the tokens s below limit(i), a row's own at most:
// `a` row ty + 8 i with ROWS floats between rows, `b` four columns with LD between tokens.  The two values of ty in a warp lie
// in one group of four tokens, so a warp skips the groups above the diagonal as one, half of all.
template <int N, int ROWS, int SIGN, int NB, typename Limit>
__device__ __forceinline__ void triangle_rows(float4 (&acc)[NB][N], const float* a, const float* (&b)[NB], int ty, Limit limit) {
#pragma unroll 2
  for (int s = 0; s < CQ; s += 4) {
    float4 x[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) x[n][j] = ld4(b[n] + (s + j) * LD);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int end = limit(i);
      if (s >= (end + 3 & ~3)) continue;
      const float4 w = ld4(a + (ty + 8 * i) * ROWS + s);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (s + j < end)
#pragma unroll
          for (int n = 0; n < NB; ++n) fma4(acc[n][i], SIGN * at4(w, j), x[n][j]);
    }
  }
}

// The products of a chunk's decays, one number g[t] per token: gam[t][s] = g[s + 1] .. g[t] for s <= t (0 above), `from` [CQ]
// = g[0] .. g[t], and what `from` of the last token is short of the product.  One warp, a lane per s, in 64 bits: the same
// decay in every token (retention) would round the same way in every product, chunk after chunk.
__device__ __forceinline__ void decay_products(const float* g, float* gam, int ldg, float* from, float* rest, int lane) {
  double run = 0., all = 1.;
#pragma unroll
  for (int t = 0; t < CQ; ++t) {
    const double x = g[t];
    run = t == lane ? 1. : run * x;
    all *= x;
    gam[t * ldg + lane] = (float)run;
    if (lane == 0) from[t] = (float)all;
  }
  if (lane == 0) *rest = (float)(all - (double)(float)all);
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
};

}  // namespace

// ------------------------------------------------------------------ 1. local part with a removal term
// Bound by its multiply-adds (0.9 M a block, of which a third of the rate goes to operands that no register keeps: 8 x 4
// outputs a thread from 16-byte loads of shared memory).  70 KB of shared memory and 128 threads: three blocks share an SM.
template <bool GATED>
__global__ void __launch_bounds__(NTH, 3)
delta_local_kernel(const DeltaIn in, const Chunk* __restrict__ chunks, float* __restrict__ mm, float* __restrict__ rq,
                   float* __restrict__ bb, float* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  DeltaSmem& sm = *reinterpret_cast<DeltaSmem*>(smem_raw);
  const int H = in.H, dk = in.dk, dv = in.dv;
  const int c = blockIdx.x / H, h = blockIdx.x % H;
  const Chunk ch = chunks[c];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
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
    if (tid < 32) decay_products(sm.g, sm.w, LD, sm.from, sm.rest, tid);
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

  // ---- the four matrices: rows u, r against columns k, a*u (gated: a*u is a number times k)
  {
    constexpr int NC = GATED ? 2 : 4;
    unsigned long long acc[8][NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[i][j] = 0ull;
#pragma unroll 2
    for (int e = 0; e < NT; e += 4) {
      ulonglong2 b[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) b[j] = ld_pairs(sm.ka + (tx + 16 * j) * LD + e);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const ulonglong2 a = ld_pairs(sm.ur + (ty + 8 * i) * LD + e);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          fma_pairs(acc[i][j], a.x, b[j].x);
          fma_pairs(acc[i][j], a.y, b[j].y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = ty + 8 * (i & 3);
      const bool read = i >= 4;
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int s = tx + 16 * (j & 1);
        const bool in_tri = (read ? s <= t : s < t) && t < ch.count;
        float x = in_tri ? pair_sum(acc[i][j]) : 0.f;
        float* dst = sm.a + (ty + 8 * i) * LD + tx + 16 * j;
        if (GATED) {
          x *= in_tri ? sm.w[(read ? t : t - 1) * LD + s] : 0.f;
          dst[CQ] = in_tri ? x * sm.gb[s] : 0.f;
        }
        *dst = x;
      }
    }
  }
  __syncthreads();
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

  // ---- [Auk ; Ark] V
  {
    float4 acc[1][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[0][i] = zero;
    const float* v[1] = {sm.vs + 4 * tx};
    triangle_rows<8, LD, 1>(acc, sm.a, v, ty, [&](int i) { return ty + 8 * (i & 3) + (i >= 4 ? 1 : 0); });
    __syncthreads();            // everyone has read the k columns of the matrices
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty + 8 * i;
      st4(sm.w + t * LD + 4 * tx, acc[0][i]);
      st4(sm.a + (t + (tx >= 8 ? CQ : 0)) * LD + 4 * (tx & 7), acc[0][4 + i]);
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
  }
  __syncthreads();

  const size_t item = (size_t)c * H + h;
  const int col0 = blockIdx.y * NT, ncols = min(NT, dv - col0);
  // ---- Rq = R~ - Aru X,  Ov = Ark V - Aru W
  {
    float4 ro[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty + 8 * i;
      ro[0][i] = ld4(sm.ur + (CQ + t) * LD + 4 * tx);
      ro[1][i] = ld4(sm.a + (t + (tx >= 8 ? CQ : 0)) * LD + 4 * (tx & 7));
    }
    const float* xw[2] = {sm.ur + 4 * tx, sm.w + 4 * tx};
    triangle_rows<4, LD, -1>(ro, sm.a + CQ * LD + CQ, xw, ty, [&](int i) { return ty + 8 * i + 1; });
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty + 8 * i;
      if (blockIdx.y == 0) st4(rq + (item * CQ + t) * NT + 4 * tx, ro[0][i]);
      if (t < ch.count && 4 * tx < ncols) st4(out + ((size_t)(ch.row0 + t) * H + h) * dv + col0 + 4 * tx, ro[1][i]);
    }
  }
  // ---- M = -AU'^T X and P,  B = K'^T V - AU'^T W
  {
    float4 m[8], b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = b[i] = zero;
#pragma unroll 2
    for (int s = 0; s < CQ; ++s) {
      const float4 x = ld4(sm.ur + s * LD + 4 * tx), w = ld4(sm.w + s * LD + 4 * tx), v = ld4(sm.vs + s * LD + 4 * tx);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float4 k = ld4(sm.ka + s * LD + 8 * ty + 4 * half), au = ld4(sm.ka + (CQ + s) * LD + 8 * ty + 4 * half);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma4(m[4 * half + j], -at4(au, j), x);
          fma4(b[4 * half + j], at4(k, j), v);
          fma4(b[4 * half + j], -at4(au, j), w);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 8 * ty + i;
      const float p = GATED ? sm.from[CQ - 1] : sm.pc[row];
      float4 x = m[i];
      float4 y = b[i];
      if (!GATED) {
        x = mul4(x, p);
        y = mul4(y, p);
      }
      if (blockIdx.y == 0) {
        st4(mm + item * MFLOATS + row * NT + 4 * tx, x);
        if (tx == 0) mm[item * MFLOATS + NT * NT + row] = p;
      }
      if (row < dk && 4 * tx < ncols) st4(bb + (item * dk + row) * dv + col0 + 4 * tx, y);
    }
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
// 103 + 141 us, the walk bound by the latency of a chain that these three do not have.)
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
  float gam[CQ * LA], g[CQ], from[CQ], rest[4];
};
struct OutSmem {
  float q[CQ * LD], k[CQ * LD], vs[CQ * LD], a[CQ * LA], st[NT * LD];
  float gam[CQ * LA], g[CQ], from[CQ], rest[4];
};

// A chunk's q (or none), k and first 64 value columns, and the products of its decays.  Ends behind a barrier.
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
  if ((tid & 3) == 0) sm.g[t] = !row_in ? 1.f : MEMORY ? in.gates[(row * H + h) * 3] : in.decay[h];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = i0 + 4 * j;
    st4(sm.k + t * LD + i, MEMORY ? mul4(kr[j], kf) : kr[j]);
    if (WITH_Q) st4(sq + t * LD + i, MEMORY ? mul4(qr[j], in.scale) : qr[j]);
    st4(sm.vs + t * LD + i, vr[j]);
  }
  __syncthreads();
  if (tid < 32) decay_products(sm.g, sm.gam, LA, sm.from, sm.rest, tid);
  if (MEMORY && dv < NT)
    for (int r = tid; r < ch.count; r += NTH) sm.vs[r * LD + dv] = 1.f;
  if (!MEMORY) {
    // turned in place, a pair of dims (i, i + rot / 2) a thread, then k times its factor
    const int half = in.rot >> 1;
    for (int e = tid; e < CQ * half; e += NTH) {
      const int r = e / half, i = e % half;
      if (r >= ch.count) continue;
      const size_t at = (size_t)in.positions[ch.row0 + r] * half + i;
      const float cs = in.cos_t[at], sn = in.sin_t[at];
      float* k = sm.k + r * LD + i;
      const float k0 = k[0], k1 = k[half];
      k[0] = (k0 * cs - k1 * sn) * kf;
      k[half] = (k1 * cs + k0 * sn) * kf;
      if (WITH_Q) {
        float* q = sq + r * LD + i;
        const float q0 = q[0], q1 = q[half];
        q[0] = q0 * cs - q1 * sn;
        q[half] = q1 * cs + q0 * sn;
      }
    }
    const int plain = dk - in.rot;
    for (int e = tid; e < CQ * plain; e += NTH) sm.k[(e / plain) * LD + in.rot + e % plain] *= kf;
  }
  __syncthreads();
}

// The next 64 value columns from col0 on (and the matrix memory's column of ones).
template <bool MEMORY>
__device__ __forceinline__ void next_columns(const DecayIn& in, const Chunk& ch, int h, int col0, float* vs) {
  for (int e = threadIdx.x; e < CQ * NT; e += NTH) {
    const int t = e / NT, d = col0 + e % NT;
    float x = 0.f;
    if (t < ch.count) x = d < in.dv ? in.v[(size_t)(ch.row0 + t) * in.ld + (size_t)h * in.dv + d] : MEMORY && d == in.dv ? 1.f : 0.f;
    vs[t * LD + e % NT] = x;
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
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const size_t item = (size_t)c * H + h;
  decay_rows<MEMORY, false>(in, ch, h, sm, nullptr);
  for (int e = tid; e < CQ * (NT / 4); e += NTH) {
    const int t = e / (NT / 4), i = (e % (NT / 4)) * 4;
    st4(sm.k + t * LD + i, mul4(ld4(sm.k + t * LD + i), sm.gam[(CQ - 1) * LA + t]));
  }
  if (tid == 0) pp[item] = make_float2(sm.from[CQ - 1], sm.rest[0]);
  for (int col0 = 0; col0 < dvp; col0 += NT) {
    const int ncols = min(NT, dvp - col0);
    if (col0) {
      __syncthreads();
      next_columns<MEMORY>(in, ch, h, col0, sm.vs);
    }
    __syncthreads();
    if (ncols <= 8) {           // a few columns
      for (int e = tid; e < dk * ncols; e += NTH) {
        const int i = e / ncols, d = e % ncols;
        float x = 0.f;
#pragma unroll 8
        for (int s = 0; s < CQ; ++s) x = fmaf(sm.k[s * LD + i], sm.vs[s * LD + d], x);
        bb[(item * dk + i) * dvp + col0 + d] = x;
      }
      continue;
    }
    float4 b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < CQ; ++s) {
      const float4 v = ld4(sm.vs + s * LD + 4 * tx);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float4 k = ld4(sm.k + s * LD + 8 * ty + 4 * half);
#pragma unroll
        for (int i = 0; i < 4; ++i) fma4(b[4 * half + i], at4(k, i), v);
      }
    }
    if (4 * tx < ncols)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * ty + i < dk) st4(bb + (item * dk + 8 * ty + i) * dvp + col0 + 4 * tx, b[i]);
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
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const float* sp = start + ((size_t)c * H + h) * dk * dvp;
  auto fetch_state = [&](int col0) {            // its 64 columns from col0 on; what does not exist as zeros
    for (int e = tid; e < NT * (NT / 4); e += NTH) {
      const int i = e / (NT / 4), d = (e % (NT / 4)) * 4;
      const bool ok = i < dk && col0 + d < dvp;
      cp_async16_or_zero(sm.st + i * LD + d, ok ? sp + (size_t)i * dvp + col0 + d : sp, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch_state(0);
  decay_rows<MEMORY, true>(in, ch, h, sm, sm.q);
  // ---- A = (q k^T) times the decays between the tokens
  {
    float acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0][0] = acc[i][0][1] = acc[i][1][0] = acc[i][1][1] = 0.f;
#pragma unroll 4
    for (int e = 0; e < NT; e += 4) {
      const float4 b0 = ld4(sm.k + tx * LD + e), b1 = ld4(sm.k + (tx + 16) * LD + e);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = ld4(sm.q + (ty + 8 * i) * LD + e);
        dot4_by_two(a, b0, acc[i][0]);
        dot4_by_two(a, b1, acc[i][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = ty + 8 * i, s = tx + 16 * j;
        sm.a[t * LA + s] = s <= t ? (acc[i][j][0] + acc[i][j][1]) * sm.gam[t * LA + s] : 0.f;
      }
  }
  __syncthreads();
  for (int e = tid; e < CQ * (NT / 4); e += NTH) {
    float* q = sm.q + (e / (NT / 4)) * LD + (e % (NT / 4)) * 4;
    st4(q, mul4(ld4(q), sm.from[e / (NT / 4)]));
  }
  for (int col0 = 0; col0 < dvp; col0 += NT) {
    const int ncols = min(NT, dvp - col0);
    if (col0) {
      __syncthreads();
      fetch_state(col0);
      next_columns<MEMORY>(in, ch, h, col0, sm.vs);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (ncols <= 8) {           // a few columns
      for (int e = tid; e < CQ * ncols; e += NTH) {
        const int t = e / ncols, d = e % ncols;
        float x = 0.f, y = 0.f;
        for (int s = 0; s <= t; ++s) x = fmaf(sm.a[t * LA + s], sm.vs[s * LD + d], x);
#pragma unroll 8
        for (int i = 0; i < NT; ++i) y = fmaf(sm.q[t * LD + i], sm.st[i * LD + d], y);
        if (t < ch.count) out[((size_t)(ch.row0 + t) * H + h) * dvp + col0 + d] = x + y;
      }
      continue;
    }
    float4 o[1][4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[0][i] = y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* values[1] = {sm.vs + 4 * tx};
    triangle_rows<4, LA, 1>(o, sm.a, values, ty, [&](int i) { return ty + 8 * i + 1; });
#pragma unroll 2
    for (int s = 0; s < NT; s += 4) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = ld4(sm.st + (s + j) * LD + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = ld4(sm.q + (ty + 8 * i) * LD + s);
#pragma unroll
        for (int j = 0; j < 4; ++j) fma4(y[i], at4(x, j), v[j]);
      }
    }
    if (4 * tx < ncols)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = ty + 8 * i;
        if (t < ch.count)
          st4(out + ((size_t)(ch.row0 + t) * H + h) * dvp + col0 + 4 * tx,
              make_float4(o[0][i].x + y[i].x, o[0][i].y + y[i].y, o[0][i].z + y[i].z, o[0][i].w + y[i].w));
      }
  }
}

// ------------------------------------------------------------------ 2. walk
// S <- P S + (M S + B) and O = Rq S + Ov over a request's chunks.  A block owns DVS value columns of a head: S lies in shared
// memory (column by column, two copies in turn), and what a chunk brings comes through a ring of three stages, two chunks
// ahead.  A thread makes four columns of three rows (two of M, one of Rq) from 16-byte loads along the inner dimension, in
// sums over even and odd places.  Bound by the bytes that its loads bring from shared memory (128 a clock and SM, also where
// lanes read the same place): 7 loads for 12 outputs.
// A chunk takes 2.7 us (64 heads, 256 blocks of 128 threads), with 3 x 2 outputs a thread as long, with 6 x 4 and two warps a
// block 3.1.
namespace {
template <int DVS>
struct WalkShape {
  static constexpr int ROWS = NT + CQ;                                 // rows of [M ; Rq]
  static constexpr int OFF = ROWS * LD, P = OFF + ROWS * DVS;          // [B ; Ov] and P behind them
  static constexpr int STAGE = P + NT;
  static constexpr int STAGES = 3, THREADS = DVS * 8;
  static constexpr size_t SMEM = (size_t)(STAGES * STAGE + 2 * DVS * LD) * sizeof(float);
};
}  // namespace

template <int DVS>
__global__ void __launch_bounds__(DVS * 8)
chunk_walk_kernel(const Request* __restrict__ requests, const Chunk* __restrict__ chunks, const float* __restrict__ mm,
                  const float* __restrict__ rq, const float* __restrict__ bb, float* __restrict__ state, float* __restrict__ out,
                  int H, int dk, int dv) {
  using K = WalkShape<DVS>;
  extern __shared__ __align__(16) float ws[];
  float* sbuf = ws + K::STAGES * K::STAGE;
  const Request r = requests[blockIdx.x / H];
  const int h = blockIdx.x % H, col0 = blockIdx.y * DVS;
  const int tid = threadIdx.x, tx = tid % (DVS / 4), ty = tid / (DVS / 4);      // ty in 0 .. 31
  float* sp = state + ((size_t)r.slot * H + h) * dk * dv;
  const int row0 = chunks[r.chunk0].row0, rows = CQ * (r.chunks - 1) + chunks[r.chunk0 + r.chunks - 1].count;
  // a thread's pieces of a chunk: the same places every time, a chunk further on
  constexpr int NP = K::ROWS * (NT / 4) / K::THREADS, NO = K::ROWS * (DVS / 4) / K::THREADS;
  static_assert(K::ROWS * (NT / 4) % K::THREADS == 0 && K::ROWS * (DVS / 4) % K::THREADS == 0, "whole pieces a thread");
  auto fetch = [&](int c) {
    float* st = ws + (c % K::STAGES) * K::STAGE;
    const size_t item = (size_t)(r.chunk0 + c) * H + h;
    const float *m = mm + item * MFLOATS, *q = rq + item * CQ * NT;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int e = tid + j * K::THREADS, row = e / (NT / 4), i = (e % (NT / 4)) * 4;
      cp_async16_or_zero(st + row * LD + i, row < NT ? m + e * 4 : q + e * 4 - NT * NT, true);
    }
    if (tid < NT / 4) cp_async16_or_zero(st + K::P + 4 * tid, m + NT * NT + 4 * tid, true);
#pragma unroll
    for (int j = 0; j < NO; ++j) {
      const int e = tid + j * K::THREADS, row = e / (DVS / 4), d = (e % (DVS / 4)) * 4, t = c * CQ + row - NT;
      const bool in = col0 + d < dv && (row < NT ? row < dk : t < rows);
      const float* src = row < NT ? bb + (item * dk + row) * dv : out + ((size_t)(row0 + t) * H + h) * dv;
      cp_async16_or_zero(st + K::OFF + row * DVS + d, in ? src + col0 + d : bb, in);
    }
  };
#pragma unroll
  for (int c = 0; c < K::STAGES - 1; ++c) {
    if (c < r.chunks) fetch(c);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int e = tid; e < NT * DVS; e += K::THREADS) {
    const int i = e / DVS, d = e % DVS;
    sbuf[d * LD + i] = i < dk && col0 + d < dv ? sp[(size_t)i * dv + col0 + d] : 0.f;
  }
  for (int c = 0; c < r.chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(K::STAGES - 2) : "memory");
    __syncthreads();            // chunk c is there, S is written, and the stage of chunk c - 1 may be filled again
    if (c + K::STAGES - 1 < r.chunks) fetch(c + K::STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* st = ws + (c % K::STAGES) * K::STAGE;
    const float* off = st + K::OFF;
    const float* s = sbuf + (c & 1) * DVS * LD;
    float* sn = sbuf + ((c + 1) & 1) * DVS * LD;
    constexpr int DQ = DVS / 4;
    unsigned long long acc[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
    for (int e = 0; e < NT; e += 4) {
      ulonglong2 x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = ld_pairs(s + (tx + DQ * j) * LD + e);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const ulonglong2 a = ld_pairs(st + (ty + 32 * i) * LD + e);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma_pairs(acc[i][j], a.x, x[j].x);
          fma_pairs(acc[i][j], a.y, x[j].y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = ty + 32 * i;
      const float p = st[K::P + row];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int d = tx + DQ * j;
        sn[d * LD + row] = fmaf(p, s[d * LD + row], pair_sum(acc[i][j]) + off[row * DVS + d]);
      }
    }
#pragma unroll
    for (int i = 2; i < 3; ++i) {
      const int row = ty + 32 * i, t = c * CQ + row - NT;
      float* o = out + ((size_t)(row0 + t) * H + h) * dv + col0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int d = tx + DQ * j;
        if (t < rows && col0 + d < dv) o[d] = pair_sum(acc[i][j]) + off[row * DVS + d];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const float* s = sbuf + (r.chunks & 1) * DVS * LD;
  for (int e = tid; e < NT * DVS; e += K::THREADS) {
    const int i = e / DVS, d = e % DVS;
    if (i < dk && col0 + d < dv) sp[(size_t)i * dv + col0 + d] = s[d * LD + i];
  }
}

namespace {

template <int DVS>
int run_walk(const int* requests, int n_requests, const int* chunks, const float* mm, const float* rq, const float* bb, float* state,
             float* out, int H, int dk, int dv, cudaStream_t s) {
  using K = WalkShape<DVS>;
  static HkSmemCache cache;
  if (int e = hk_allow_smem(chunk_walk_kernel<DVS>, K::SMEM, cache)) return e;
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
  static HkSmemCache cache;
  if (int e = hk_allow_smem(delta_local_kernel<GATED>, sizeof(DeltaSmem), cache)) return e;
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
  static HkSmemCache cache;
  if (int e = hk_allow_smem(decay_out_kernel<MEMORY>, sizeof(OutSmem), cache)) return e;
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
