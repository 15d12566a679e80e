// Generic matrix product for every shape: out[M, N] (fp32) = a[M, K] * w[N, K]^T, optionally
// added onto what `out` holds (the residual sum).  Operands are float (the true 32-bit path:
// plain FMA, no reduced-precision matrix mode) or bf16 (the fallback of the serving path for
// shapes the tensor-core kernels refuse).  Float operands whose rows are whole 16-byte pieces take `gemm_f32_kernel`,
// which sums even and odd k apart, both in order; `gemm_generic_kernel` takes the rest and accumulates k = 0..K-1 in
// order in one fp32 register.  Which of the two depends on K and the operands alone, so a row's result does not depend on M
// or on the tile it is in.
//
// Reference counterpart: `gemm_<fmt>` tiled kernel, src/cuda_device.zig:237-285.
#include "common.cuh"

#define GG_BM 64
#define GG_BN 64
#define GG_BK 16

// ----------------------------------------------------------------------------- float operands in whole 16-byte pieces
// Bound by the fp32 FMA pipe (prompt rows) or by the latency of the weights' slices (a few rows).  A block makes a BM x BN tile of one
// product (of one head: blockIdx.z) from a ring of STAGES slices of BK columns that cp.async fills; both operands stay as
// they lie in memory, a row's BK columns side by side, so nothing is transposed and a thread reads four k of a row with
// one 16-byte load: TM + TN loads for 4 TM TN FMAs, which run in pairs (even k, odd k): an output is the sum over even k plus
// the sum over odd k, each in order, whatever the tile is.  A row of a slice is BK + 4 floats: eight rows' 16-byte pieces fall into
// different banks.  A thread's rows and columns lie BM / TM and BN / TN apart (neighbouring lanes read neighbouring rows).
struct F32Product {
  const float *a, *w;
  float* out;
  int M, N, K;
  long long lda, a_head, ldw, w_head, ldo, o_head;
  int accumulate;
  const float* gate;        // per-head products only: the result times gate_scale * sigmoid(gate)
  long long gate_ld;
  int gate_heads;
  float gate_scale;
};

__device__ __forceinline__ void gg_cp_async16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}

// two single-precision fused multiply-adds, each rounded as fmaf rounds
__device__ __forceinline__ void gg_fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
struct F32Tile {
  static constexpr int LD = BK + 4, TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  static constexpr size_t SMEM = (size_t)STAGES * (BM + BN) * LD * sizeof(float);
};

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
__global__ void __launch_bounds__(BM / TM * (BN / TN))
gemm_f32_kernel(const F32Product p) {
  using T = F32Tile<BM, BN, TM, TN, BK, STAGES>;
  constexpr int LD = T::LD, TX = T::TX, TY = T::TY, PIECES = BK / 4;
  extern __shared__ __align__(16) float gg_sm[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX, h = blockIdx.z;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const float* a = p.a + (size_t)h * p.a_head;
  const float* w = p.w + (size_t)h * p.w_head;
  const int slices = (p.K + BK - 1) / BK;
  auto fetch = [&](int s) {
    float* dst = gg_sm + (size_t)(s % STAGES) * (BM + BN) * LD;
    const int k0 = s * BK;
#pragma unroll
    for (int e = tid; e < (BM + BN) * PIECES; e += T::THREADS) {
      const int r = e / PIECES, c = (e % PIECES) * 4;
      const int row = r < BM ? m0 + r : n0 + r - BM;
      const bool in = row < (r < BM ? p.M : p.N) && k0 + c < p.K;
      const float* src = r < BM ? a : w;
      gg_cp_async16(dst + r * LD + c, in ? src + (size_t)row * (r < BM ? p.lda : p.ldw) + k0 + c : src, in);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < slices) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  unsigned long long acc[TM][TN];               // the sums over even k and over odd k
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  for (int s = 0; s < slices; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                            // slice s is there, and slice s - 1's stage may be filled again
    if (s + STAGES - 1 < slices) fetch(s + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* As = gg_sm + (size_t)(s % STAGES) * (BM + BN) * LD + ty * LD;
    const float* Ws = gg_sm + (size_t)(s % STAGES) * (BM + BN) * LD + (BM + tx) * LD;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 av[TM], wv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(As + i * TY * LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(Ws + j * TX * LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) gg_fma2(acc[i][j], av[i].x, wv[j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) gg_fma2(acc[i][j], av[i].y, wv[j].y);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  float* out = p.out + (size_t)h * p.o_head;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * TY;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * TX;
      if (n >= p.N) continue;
      float v = __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
      if (p.gate) v = p.gate_scale * v / (1.0f + expf(-p.gate[(size_t)m * p.gate_ld + (p.gate_heads ? h : h * p.N + n)]));
      float* o = out + (size_t)m * p.ldo + n;
      *o = p.accumulate ? *o + v : v;
    }
  }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
static int gemm_f32_launch(const F32Product& p, int heads, cudaStream_t s) {
  using T = F32Tile<BM, BN, TM, TN, BK, STAGES>;
  const long long rows = ((long long)p.M + BM - 1) / BM;
  if (rows > 65535 || heads > 65535) return HK_ERR_UNSUPPORTED;
  if (int e = hk_allow_smem<gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>>(T::SMEM)) return e;
  return hk_launch(gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>, dim3((unsigned)((p.N + BN - 1) / BN), (unsigned)rows, (unsigned)heads),
                   dim3(T::THREADS), T::SMEM, s, p);
}

static bool gg_aligned(const F32Product& p) {
  return !(p.K & 3) && !(p.lda & 3) && !(p.ldw & 3) && !(p.a_head & 3) && !(p.w_head & 3) && !(((uintptr_t)p.a | (uintptr_t)p.w) & 15);
}

// The tile: by rows, then by what the busiest of 148 SMs has to make.  Measured (us, L2 cold, K = 1,024 to 3,072; the 64 x 64
// tiles without a ring before: 255 a product on average over a layer of 1,024 wide at 509 rows):
//   509 x 6144 x 1024: 64 x 64 172, 64 x 32 172, 128 x 128 246;   2048 x 12288 x 2048: 2,214 (47 TFLOP/s), 2,446, 2,604
//   509 x 1024 x 3072: 64 x 64 109, 64 x 32 105, 128 x 64 215;    100 x 1024 x 3072: 64 x 64 107, 64 x 32 70, 32 x 32 45
//   up to 8 rows: 4096 x 4096: 8 x 16 tiles 39, 8 x 32 47;        24576 x 4096: 160, 116
//   up to 16 rows: 13 x 6144 x 1024: 16 x 16 tiles 21, 16 x 32 25
// A multiply-add with three registers of its own runs at two thirds of the pipe's rate (measured 23.6 T/s against 36 with
// one operand kept), two packed ones at 28 T/s: that and not the loads bounds the large tiles.
static int gemm_f32(const F32Product& p, int heads, cudaStream_t s) {
  const long long wide = 148 * 64;              // columns from which 32-wide tiles of a few rows give every SM two
  if (p.M <= 8) {
    if ((long long)p.N * heads < wide) return gemm_f32_launch<8, 16, 1, 1, 128, 3>(p, heads, s);
    return gemm_f32_launch<8, 32, 2, 2, 128, 3>(p, heads, s);
  }
  if (p.M <= 16) {
    if ((long long)p.N * heads < wide) return gemm_f32_launch<16, 16, 2, 2, 128, 4>(p, heads, s);
    return gemm_f32_launch<16, 32, 2, 2, 128, 3>(p, heads, s);
  }
  auto tiles = [&](int bm, int bn) { return (((long long)p.M + bm - 1) / bm) * (((long long)p.N + bn - 1) / bn) * heads; };
  auto busiest = [&](int bm, int bn) { return (double)((tiles(bm, bn) + 147) / 148) * bm * bn; };
  if (1.3 * busiest(32, 32) < busiest(64, 32)) return gemm_f32_launch<32, 32, 4, 2, 64, 3>(p, heads, s);
  if (tiles(64, 64) <= 4 * 148) return gemm_f32_launch<64, 32, 4, 4, 32, 3>(p, heads, s);
  return gemm_f32_launch<64, 64, 8, 4, 32, 3>(p, heads, s);
}

template <typename T>
__global__ void __launch_bounds__(256)
gemm_generic_kernel(const T* __restrict__ a, const T* __restrict__ w, float* __restrict__ out, int M,
                    int N, int K, long long lda, long long ldw, long long ldo, int accumulate) {
  __shared__ float As[GG_BK][GG_BM + 4];
  __shared__ float Ws[GG_BK][GG_BN + 4];
  int tid = threadIdx.x;
  int m0 = blockIdx.y * GG_BM, n0 = blockIdx.x * GG_BN;
  int tx = tid & 15, ty = tid >> 4;  // thread computes rows ty*4.., cols tx*4..
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += GG_BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int i = tid + j * 256;
      int r = i >> 4, c = i & 15;
      int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32<T>(a[(size_t)gm * lda + gk]) : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? to_f32<T>(w[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GG_BK; ++kk) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float* o = out + (size_t)gm * ldo + gn;
      *o = accumulate ? *o + acc[i][j] : acc[i][j];
    }
  }
}

HK_API int hk_gemm_generic(const void* a, const void* w, int dtype, float* out, int M, int N, int K,
                           long long lda, long long ldw, long long ldo, int accumulate, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HK_F32) {
    const F32Product p = {(const float*)a, (const float*)w, out, M, N, K, lda, 0, ldw, 0, ldo, 0, accumulate, nullptr, 0, 0, 0.f};
    if (gg_aligned(p)) {
      const int e = gemm_f32(p, 1, s);
      if (e != HK_ERR_UNSUPPORTED) return e;
    }
  }
  dim3 grid((N + GG_BN - 1) / GG_BN, (M + GG_BM - 1) / GG_BM);
  if (grid.y > 65535) return HK_ERR_UNSUPPORTED;
  if (dtype == HK_F32)
    gemm_generic_kernel<float><<<grid, 256, 0, s>>>((const float*)a, (const float*)w, out, M, N, K, lda,
                                                   ldw, ldo, accumulate);
  else if (dtype == HK_BF16)
    gemm_generic_kernel<bf16><<<grid, 256, 0, s>>>((const bf16*)a, (const bf16*)w, out, M, N, K, lda, ldw,
                                                  ldo, accumulate);
  else
    return HK_ERR_UNSUPPORTED;
  return hk_launch_status();
}

// ----------------------------------------------------------------------------- one small product per head
// out[t, h, :N] = a[t, h, :K] * w[h]^T for every head h: w is [heads][N][K]; a's and out's rows of one token lie
// `lda` / `ldo` elements apart and their heads `a_head` / `o_head` elements apart (so the output may be a column
// slice of wider rows).  The output takes the storage type or fp32.  Same tiles and summation order as above, the
// head in blockIdx.z.  With `gate` (fp32 logits, row stride gate_ld, head h at column h * N, or one number per head at
// column h with gate_heads = 1) the result is multiplied by gate_scale * sigmoid(gate).
template <typename T, typename TO>
__global__ void __launch_bounds__(256)
gemm_heads_kernel(const T* __restrict__ a, const T* __restrict__ w, TO* __restrict__ out, int M, int N, int K,
                  long long lda, long long a_head, long long ldo, long long o_head, const float* __restrict__ gate,
                  long long gate_ld, int gate_heads, float gate_scale) {
  __shared__ float As[GG_BK][GG_BM + 4];
  __shared__ float Ws[GG_BK][GG_BN + 4];
  const int tid = threadIdx.x, h = blockIdx.z;
  const int m0 = blockIdx.y * GG_BM, n0 = blockIdx.x * GG_BN;
  const int tx = tid & 15, ty = tid >> 4;
  a += (size_t)h * a_head;
  w += (size_t)h * N * K;
  out += (size_t)h * o_head;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += GG_BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int i = tid + j * 256;
      int r = i >> 4, c = i & 15;
      int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32<T>(a[(size_t)gm * lda + gk]) : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? to_f32<T>(w[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GG_BK; ++kk) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (gate) v = gate_scale * v / (1.0f + expf(-gate[(size_t)gm * gate_ld + (gate_heads ? h : h * N + gn)]));
      out[(size_t)gm * ldo + gn] = from_f32<TO>(v);
    }
  }
}

HK_API int hk_gemm_heads(const void* a, const void* w, int dtype, void* out, int out_dtype, int M, int N, int K, int heads,
                         long long lda, long long a_head, long long ldo, long long o_head, const float* gate, long long gate_ld,
                         int gate_heads, float gate_scale, void* stream) {
  if (M <= 0 || N <= 0 || heads <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == HK_F32 && out_dtype == HK_F32) {
    const F32Product p = {(const float*)a, (const float*)w, (float*)out, M, N, K, lda, a_head, K, (long long)N * K, ldo, o_head, 0, gate, gate_ld,
                          gate_heads, gate_scale};
    if (gg_aligned(p)) {
      const int e = gemm_f32(p, heads, s);
      if (e != HK_ERR_UNSUPPORTED) return e;
    }
  }
  dim3 grid((N + GG_BN - 1) / GG_BN, (M + GG_BM - 1) / GG_BM, heads);
  if (grid.y > 65535 || grid.z > 65535) return HK_ERR_UNSUPPORTED;
  if (dtype == HK_F32 && out_dtype == HK_F32)
    gemm_heads_kernel<float, float><<<grid, 256, 0, s>>>((const float*)a, (const float*)w, (float*)out, M, N, K, lda, a_head, ldo, o_head, gate, gate_ld, gate_heads, gate_scale);
  else if (dtype == HK_BF16 && out_dtype == HK_BF16)
    gemm_heads_kernel<bf16, bf16><<<grid, 256, 0, s>>>((const bf16*)a, (const bf16*)w, (bf16*)out, M, N, K, lda, a_head, ldo, o_head, gate, gate_ld, gate_heads, gate_scale);
  else if (dtype == HK_BF16 && out_dtype == HK_F32)
    gemm_heads_kernel<bf16, float><<<grid, 256, 0, s>>>((const bf16*)a, (const bf16*)w, (float*)out, M, N, K, lda, a_head, ldo, o_head, gate, gate_ld, gate_heads, gate_scale);
  else
    return HK_ERR_UNSUPPORTED;
  return hk_launch_status();
}
