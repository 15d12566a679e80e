// bf16 matrix product on pairs of SMs: out[M, N] = a[M, K] * w[N, K]^T with fp32 accumulation in tensor memory, for more rows
// than a batch that decodes.  The weights are the tensor core's M side: a pair of CTAs (a cluster of two) makes tiles of 256
// weight rows by up to 256 rows of a (`tcgen05.mma.cta_group::2`, 256 x w x 16), each CTA holding 128 of the weight rows and half
// of the rows of a in its shared memory and 128 of the result's rows in its tensor memory.
//
//   warp 0      (both CTAs) TMA producer into a ring of stages of 64 k; its copies complete on the first CTA's barrier
//   warp 1      (first CTA) one lane issues the products and commits stage releases and accumulators to both CTAs
//   warps 2..9  (both CTAs) epilogue, two warps to 32 weight rows: a lane holds one weight row's results for 32 rows of a at a
//               time, so that a warp's store covers 32 neighbouring numbers of one row of `out`
//
// Why pairs, and why this way round: a tile of 128 x 256 on one SM reads 48 KB of operands for its 64 k, half of a 256 x 256 tile
// 32 KB, which the L2 and the shared memory both feel; and with the rows of a on the N side their number is filled up to a
// multiple of 32 instead of 128 (the tiles of a product share them evenly: widths differ by 32 at most).
// Two accumulators of 256 columns let a tile's epilogue run under the next tile's products; with four epilogue warps a CTA
// instead of eight a short K (2,048) waited for it (12,288 x 2,048 gated by 527 rows 35 us instead of 26).
//
// Against the kernel of gemm_tc.cu at the width and slices that it would get (us, one B200, weights from the HBM, launches back to
// back):
//     K = 4,096   rows     300    527  1,000  2,048        K = 12,288 by N = 4,096  rows     300    527  1,000  2,048
//     N =  6,144  before  20.4   30.0   45.7   86.4                                 before  39.4   52.8   82.4  158.6
//                 now     17.5   23.6   40.3   75.5                                 now     33.1   47.1   74.4  143.5
//     N = 16,384  before  48.4   72.6  109.5  206.1        K = 2,048 by N = 8,256   before  16.7   23.3   32.9   64.3
//                 now     39.2   58.7  101.4  177.9                                 now     13.9   19.2   29.5   56.9
// 2,048 rows by 16,384 x 4,096 run at 1,536 TFLOP/s: the products alone take 128 of the 179 us, the loads alone 103, and the
// 134 MB of float32 results cost the rest in part.  A single wave of short tiles is bound by what surrounds them: of the 16 us
// of 256 rows by 4,096 x 4,096, 8 pass without a product (launch, barriers, the first copy, the last store).
//
// K may be cut into slices (few tiles, long K): an item of work is then a tile's slice, whose sums go to `partial`, and
// `gemm_pair_add_kernel` adds a tile's slices in the order of k.  (Shares of K cut evenly over all pairs, each ending one tile and
// starting another, were slower than whole tiles or equal slices at nearly every shape: a partial tile is 256 KB to write and read.)
// Every mbarrier wait is bounded, as in gemm_tc.cu; no copy is multicast.
#include "gemm_tc.cuh"

namespace {

constexpr int FT = 256;                 // weight rows of a tile
constexpr int PAIR_THREADS = 320;
constexpr int MAX_W = 256;              // the widest tile; also the distance of the two accumulators in tensor memory
constexpr int PAIR_STAGES = 12;
constexpr int W_BYTES = 128 * BK * 2;   // a stage's weight rows in one CTA
constexpr int PAIR_CONTROL = 1024;
constexpr int PAIR_RING = 227 * 1024 - 2 * 1024;

struct PairShape {
  int M, N, K;
  int tiles_m, units;       // tiles along the rows of a, which share `units` = ceil(M / 32) blocks of 32 rows evenly
  int kb, slices;           // K blocks of 64; slices that a tile's are cut into
  int tiles;                // tiles in all; items of work = tiles * slices
};

__host__ __device__ inline int widest(const PairShape& s) { return 32 * ((s.units + s.tiles_m - 1) / s.tiles_m); }

// The grouped form (a feed-forward of experts): a's rows are sorted by group, tile g = tiles[2 g] (its group; -1 from the first
// unused one on) has up to `rows` of them from tiles[2 g + 1] on, none past offsets[group + 1], and group e's weights are the N rows
// from e N on.
struct PairGroups {
  const int *tiles, *offsets;
  int max_tiles, rows;
};

// One item: weight rows from w_row on (the tile's column `tf` of N), `width` rows of a from t0 on of which those below `end` count,
// K blocks [k0, k1).
struct PairItem {
  int tile, tf, w_row, t0, width, end, k0, k1;
  template <bool GLU>
  static __device__ __forceinline__ PairItem plain(const PairShape& s, int item) {
    PairItem it;
    const int slice = item / s.tiles;
    it.tile = item - slice * s.tiles;
    it.tf = it.tile / s.tiles_m;
    const int tm = it.tile - it.tf * s.tiles_m, lo = tm * s.units / s.tiles_m, hi = (tm + 1) * s.units / s.tiles_m;
    it.t0 = 32 * lo;
    it.width = 32 * (hi - lo);
    it.end = min(s.M, 32 * hi);
    it.w_row = it.tf * (GLU ? FT / 2 : FT);
    it.k0 = (int)((long long)s.kb * slice / s.slices);
    it.k1 = (int)((long long)s.kb * (slice + 1) / s.slices);
    return it;
  }
  template <bool GLU>
  static __device__ __forceinline__ PairItem grouped(const PairShape& s, const PairGroups& g, int used, int item) {
    PairItem it;
    it.tf = item / used;
    it.tile = item - it.tf * used;
    const int e = g.tiles[2 * it.tile];
    it.t0 = g.tiles[2 * it.tile + 1];
    it.end = min(it.t0 + g.rows, g.offsets[e + 1]);
    it.width = (it.end - it.t0 + 31) & ~31;
    it.w_row = e * s.N + it.tf * (GLU ? FT / 2 : FT);
    it.k0 = 0;
    it.k1 = s.kb;
    return it;
  }
};
// Floats of one item's sums in `partial`: [CTA][quarter of its rows][row of a][lane]
__host__ __device__ inline size_t item_floats(int width) { return (size_t)FT * width; }

struct PairControl {
  uint64_t full[PAIR_STAGES], empty[PAIR_STAGES];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int filled_by_other;          // in the first CTA: how many stages the second one has filled in all (-1: it has not said)
};
static_assert(sizeof(PairControl) <= PAIR_CONTROL, "control block too large");

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {      // the same place in the pair's CTA `rank`
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void put_in_cta(const volatile int* at, uint32_t rank, int value) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_cta(smem_u32((const void*)at), rank)), "r"(value) : "memory");
}
// A wait that gives up tells the other CTA too.
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t other) {
  if (mbar_wait(bar, parity, abort_flag)) return true;
  put_in_cta(abort_flag, other, 1);
  return false;
}
// Giving up, in the first CTA, where all copies are counted: lets those that are still on their way land, in both CTAs.  The two may
// have stopped at different stages: what the other one brought alone is still to be expected, what it did not bring counts as there.
__device__ __forceinline__ void let_copies_land(PairControl& sm, int mine, int stages, uint32_t bytes) {
  const volatile int* said = &sm.filled_by_other;
  for (uint32_t spin = 0; spin < WAIT_LIMIT && *said < 0; ++spin) {}
  const int others = max(*said, 0), most = max(mine, others);
  for (int i = max(most - stages, 0); i < most; ++i) {
    uint64_t* full = &sm.full[i % stages];
    if (i >= mine) mbar_expect_tx(full, bytes);
    if (i >= others) asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(full)), "r"(bytes) : "memory");
    for (uint32_t spin = 0; spin < WAIT_LIMIT; ++spin)
      if (mbar_try_wait(full, (uint32_t)(i / stages) & 1u)) break;
  }
}
// Copies into this CTA that complete on a barrier of either CTA of the pair.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t* bar) {        // to the barrier at this place in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// The rows of `out` that a chunk is added onto, for the lane's weight row f.
__device__ __forceinline__ void load_onto(const float* out, long long ldo, int f, int t0, int M, int N, float (&y)[32]) {
  const float* o = out + (size_t)t0 * ldo + f;
  const int count = f < N ? M - t0 : 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) y[j] = j < count ? o[j * ldo] : 0.f;
}

// 32 rows of `out` from t0 on, of the lane's weight row `f`.
__device__ __forceinline__ void store_rows(const float (&v)[32], float* out, long long ldo, int f, int t0, int M, int N) {
  float* o = out + (size_t)t0 * ldo + f;
  const int count = f < N ? M - t0 : 0;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j < count) o[j * ldo] = v[j];
}
// The same narrowed to bf16.
template <int EPI>
__device__ __forceinline__ void narrow_rows(const float (&v)[32], void* out, long long ldo, int f, int t0, int M, int N, GluParams gp) {
  // two rows of `out` in a word; then lanes 2 i and 2 i + 1 swap halves, so that a word is two columns of one row
  uint32_t p[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    __nv_bfloat162 x;
    const float a = v[2 * k], b = v[2 * k + 1];
    x.x = EPI == EPI_NARROW ? __float2bfloat16_rn(a) : squared_relu(a, gp);
    x.y = EPI == EPI_NARROW ? __float2bfloat16_rn(b) : squared_relu(b, gp);
    p[k] = *reinterpret_cast<uint32_t*>(&x);
  }
  const bool odd = f & 1;
  const int f0 = f & ~1, t1 = t0 + (odd ? 16 : 0);
  bf16* o = reinterpret_cast<bf16*>(out) + (size_t)t1 * ldo + f0;
  const bool wide = f0 + 1 < N && !(ldo & 1) && !((uintptr_t)out & 3);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? p[k] : p[8 + k], 1);
    const uint32_t lo = odd ? got : p[k], hi = odd ? p[8 + k] : got;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (t1 + 2 * k + e >= M) continue;
      const uint32_t word = __byte_perm(lo, hi, e ? 0x7632 : 0x5410);
      bf16* at = o + (2 * k + e) * ldo;
      if (wide) *reinterpret_cast<uint32_t*>(at) = word;
      else {
        if (f0 < N) at[0] = __ushort_as_bfloat16((unsigned short)word);
        if (f0 + 1 < N) at[1] = __ushort_as_bfloat16((unsigned short)(word >> 16));
      }
    }
  }
}

// Gated: even lanes hold gates, odd lanes their ups (`f`: the lane pair's column of `out`, F of them).
template <int EPI>
__device__ __forceinline__ void emit_gated(const float (&v)[32], void* out, long long ldo, int f, int t0, int M, int F, GluParams gp) {
  const int lane = threadIdx.x & 31;
  const bool up = lane & 1, second = lane & 2;
  uint32_t p[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {         // a lane's 16 rows: the gate lane takes the first half
    __nv_bfloat162 x;
    float r[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int j = 2 * k + e;
      const float got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[16 + j], 1);
      const float g = up ? got : v[j], u = up ? v[16 + j] : got;
      r[e] = glu_pair<EPI>(g, u, gp);
    }
    x = __floats2bfloat162_rn(r[0], r[1]);
    p[k] = *reinterpret_cast<uint32_t*>(&x);
  }
  const int f0 = f & ~1, t1 = t0 + (up ? 16 : 0) + (second ? 8 : 0);
  bf16* o = reinterpret_cast<bf16*>(out) + (size_t)t1 * ldo + f0;
  const bool wide = f0 + 1 < F && !(ldo & 1) && !((uintptr_t)out & 3);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, second ? p[k] : p[4 + k], 2);
    const uint32_t lo = second ? got : p[k], hi = second ? p[4 + k] : got;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (t1 + 2 * k + e >= M) continue;
      const uint32_t word = __byte_perm(lo, hi, e ? 0x7632 : 0x5410);
      bf16* at = o + (2 * k + e) * ldo;
      if (wide) *reinterpret_cast<uint32_t*>(at) = word;
      else {
        if (f0 < F) at[0] = __ushort_as_bfloat16((unsigned short)word);
        if (f0 + 1 < F) at[1] = __ushort_as_bfloat16((unsigned short)(word >> 16));
      }
    }
  }
}

// The lane's weight row (gated: its pair's column of `out`) in tile column `tf`.
template <int EPI>
__device__ __forceinline__ int lane_row(int tf, int rank, int quarter, int lane) {
  return IS_GLU(EPI) ? tf * (FT / 2) + rank * 64 + quarter * 16 + (lane >> 1) : tf * FT + rank * 128 + quarter * 32 + lane;
}
template <int EPI>
__device__ __forceinline__ void emit(const float (&v)[32], void* out, long long ldo, int f, int t0, int M, int N, GluParams gp) {
  if constexpr (IS_GLU(EPI)) emit_gated<EPI>(v, out, ldo, f, t0, M, N >> 1, gp);
  else if constexpr (EPI == EPI_STORE || EPI == EPI_ADD) store_rows(v, reinterpret_cast<float*>(out), ldo, f, t0, M, N);
  else narrow_rows<EPI>(v, out, ldo, f, t0, M, N, gp);
}

// map_a: boxes of half the widest tile's rows; map_w: 128 weight rows, gated 64 of [K, 2, F] so that gate and up rows alternate.
template <int EPI, bool GROUPED>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, void* __restrict__ out,
                 const PairShape s, const PairGroups g, long long ldo, int stages, float* __restrict__ partial, int* __restrict__ status,
                 GluParams gp) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  PairControl& sm = *reinterpret_cast<PairControl*>(base);
  uint8_t* ring = base + PAIR_CONTROL;
  volatile int* abort_flag = &sm.abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1, other = rank ^ 1;
  const int max_w = GROUPED ? g.rows : widest(s);
  const uint32_t stage_bytes = W_BYTES + (uint32_t)max_w * BK;           // (max_w / 2 rows of 128 bytes)

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.tmem_full[b], 1);
      mbar_init(&sm.tmem_empty[b], 16);
    }
    sm.abort_flag = 0;
    sm.filled_by_other = -1;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(2u * MAX_W) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();                  // the other CTA's barriers are there
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  pdl_wait();

  int used = 0;                 // tiles that have rows
  if (GROUPED) {
    for (int t = lane; t < g.max_tiles; t += 32) used += g.tiles[2 * t] >= 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) used += __shfl_xor_sync(0xffffffffu, used, o);
  }
  const int first_item = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int items = GROUPED ? used * s.tiles : s.tiles * s.slices;
  auto item_of = [&](int i) {
    if constexpr (GROUPED) return PairItem::grouped<IS_GLU(EPI)>(s, g, used, i);
    else return PairItem::plain<IS_GLU(EPI)>(s, i);
  };
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = first_item; i < items && ok; i += pairs) {
        const PairItem it = item_of(i);
        const int row = it.t0 + (int)rank * (it.width >> 1);
        for (int kb = it.k0; kb < it.k1; ++kb) {
          if (!pair_wait(&sm.empty[stage], phase ^ 1u, abort_flag, other)) { ok = false; break; }
          const uint32_t st = smem_u32(ring) + (uint32_t)stage * stage_bytes;
          if (rank == 0) mbar_expect_tx(&sm.full[stage], 2 * stage_bytes);
          const uint32_t bar = in_cta(smem_u32(&sm.full[stage]), 0);
          if (IS_GLU(EPI)) pair_load_3d(st, &map_w, bar, kb * BK, 0, it.w_row + (int)rank * 64);
          else pair_load_2d(st, &map_w, bar, kb * BK, it.w_row + (int)rank * 128);
          pair_load_2d(st + W_BYTES, &map_a, bar, kb * BK, row);
          ++issued;
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      pdl_launch_dependents();
      if (rank == 1) put_in_cta(&sm.filled_by_other, 0, issued);
      // A stage's release is a signal of the tensor core to both CTAs that no thread orders: a CTA may not leave, nor its shared memory
      // go to another block, before the last ones have come.
      for (int i = issued > stages ? issued - stages : 0; i < issued && ok; ++i)
        ok = pair_wait(&sm.empty[i % stages], (uint32_t)(i / stages) & 1u, abort_flag, other);
      if (*abort_flag && rank == 0) let_copies_land(sm, issued, stages, stage_bytes);
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int stage = 0, local = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = first_item; i < items && ok; i += pairs) {
        const PairItem it = item_of(i);
        // fp32 accumulate, bf16 x bf16, both K-major, N = width, M = 256
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(it.width >> 3) << 17) | ((uint32_t)(FT >> 4) << 24);
        const int buf = local & 1;
        if (!pair_wait(&sm.tmem_empty[buf], ((uint32_t)(local >> 1) & 1u) ^ 1u, abort_flag, other)) break;
        ++local;
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(buf * MAX_W);
        for (int kb = it.k0; kb < it.k1; ++kb) {
          if (!pair_wait(&sm.full[stage], phase, abort_flag, other)) { ok = false; break; }
          tc_fence_after();
          const uint32_t st = smem_u32(ring) + (uint32_t)stage * stage_bytes;
          const uint64_t dw = make_smem_desc(st), da = make_smem_desc(st + W_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            pair_mma(d, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, (kb > it.k0 || k > 0) ? 1u : 0u);
          pair_commit(&sm.empty[stage]);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (ok) pair_commit(&sm.tmem_full[buf]);
      }
    }
  } else {
    const int quarter = warp & 3;           // the tensor-memory lanes this warp may read: 32 * quarter ..
    const int first = (warp - 2) >> 2 ? 32 : 0;       // its chunks of 32 rows of a: every other one
    int local = 0;
    for (int i = first_item; i < items; i += pairs) {
      const PairItem it = item_of(i);
      const int buf = local & 1;
      const uint32_t use = (uint32_t)(local >> 1) & 1u;
      ++local;
      const int f = lane_row<EPI>(it.tf, (int)rank, quarter, lane);
      const bool whole = s.slices == 1;
      // what a whole tile is added onto does not depend on the product: asked for a chunk ahead
      float y[32];
      const float* onto = reinterpret_cast<const float*>(out);
      if (EPI == EPI_ADD && whole) load_onto(onto, ldo, f, it.t0 + first, it.end, s.N, y);
      if (!__all_sync(0xffffffffu, pair_wait(&sm.tmem_full[buf], use, abort_flag, other))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * MAX_W);
      float* part = whole ? nullptr
                          : partial + i * item_floats(max_w) + ((size_t)(rank * 4 + quarter) * max_w) * 32 + lane;
#pragma unroll 1
      for (int c = first; c < it.width; c += 64) {
        uint32_t v[32];
        tmem_ld32(taddr + (uint32_t)c, v);
        tmem_ld_wait();
        if (!whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) part[(c + j) * 32] = __uint_as_float(v[j]);
        } else if (EPI == EPI_ADD) {
          float sum[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] = y[j] + __uint_as_float(v[j]);
          if (c + 64 < it.width) load_onto(onto, ldo, f, it.t0 + c + 64, it.end, s.N, y);
          store_rows(sum, reinterpret_cast<float*>(out), ldo, f, it.t0 + c, it.end, s.N);
        } else {
          float sum[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] = __uint_as_float(v[j]);
          emit<EPI>(sum, out, ldo, f, it.t0 + c, it.end, s.N, gp);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta(smem_u32(&sm.tmem_empty[buf]), 0)) : "memory");
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && sm.abort_flag) atomicExch(status, 1);
  pair_sync();                  // nobody leaves while the other still signals it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * MAX_W) : "memory");
  }
}

// Adds a tile's slices in the order of k and finishes it.  A block per (tile, CTA's half, 32 rows of a), a warp per quarter of the
// half's weight rows.
template <int EPI>
__global__ void __launch_bounds__(128)
gemm_pair_add_kernel(const float* __restrict__ partial, void* __restrict__ out, const PairShape s, long long ldo, GluParams gp) {
  const PairItem it = PairItem::plain<IS_GLU(EPI)>(s, (int)blockIdx.x >> 1);
  const int rank = blockIdx.x & 1, c = blockIdx.y * 32, quarter = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int max_w = widest(s), f = lane_row<EPI>(it.tf, rank, quarter, lane);
  const float* p = partial + it.tile * item_floats(max_w) + ((size_t)(rank * 4 + quarter) * max_w + c) * 32 + lane;
  pdl_launch_dependents();
  pdl_wait();                   // (every block: the kernel after this one relies on it for the product before)
  if (c >= it.width || it.t0 + c >= s.M) return;
  float sum[32], y[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) sum[j] = __ldcs(p + j * 32);
  if (EPI == EPI_ADD) load_onto(reinterpret_cast<const float*>(out), ldo, f, it.t0 + c, s.M, s.N, y);
  for (int r = 1; r < s.slices; ++r) {
    p += s.tiles * item_floats(max_w);
#pragma unroll
    for (int j = 0; j < 32; ++j) sum[j] += __ldcs(p + j * 32);
  }
  if (EPI == EPI_ADD)
#pragma unroll
    for (int j = 0; j < 32; ++j) sum[j] = y[j] + sum[j];
  emit<EPI>(sum, out, ldo, f, it.t0 + c, s.M, s.N, gp);
}

// [groups][2][F][K], row f of a group's gates beside row f of its ups: 64 such pairs from row 2 F group + f on
bool make_gated_map(CUtensorMap* map, const void* ptr, int F, int cols, int groups) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, 2, (cuuint64_t)F * (2 * groups - 1)};
  cuuint64_t strides[2] = {(cuuint64_t)F * cols * 2, (cuuint64_t)cols * 2};
  cuuint32_t box[3] = {(cuuint32_t)BK, 2, 64};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int EPI, bool GROUPED>
int launch_pair(const CUtensorMap& ma, const CUtensorMap& mw, void* out, const PairShape& s, const PairGroups& g, long long ldo, int pairs,
                float* partial, int* status, GluParams gp, cudaStream_t stream) {
  const int stage_bytes = W_BYTES + (GROUPED ? g.rows : widest(s)) * BK;
  const int stages = min(PAIR_STAGES, PAIR_RING / stage_bytes);
  const size_t smem = (size_t)stages * stage_bytes + PAIR_CONTROL + 1024;
  if (int e = hk_allow_smem<gemm_pair_kernel<EPI, GROUPED>>(smem)) return e;
  const long long items = (long long)s.tiles * (GROUPED ? g.max_tiles : s.slices);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (items < pairs ? (int)items : pairs)));
  cfg.blockDim = dim3(PAIR_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (int e = (int)cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI, GROUPED>, ma, mw, out, s, g, ldo, stages, partial, status, gp)) return e;
  if (GROUPED || s.slices == 1) return 0;
  return hk_launch_pdl(gemm_pair_add_kernel<EPI>, dim3((unsigned)(2 * s.tiles), (unsigned)(widest(s) / 32)), dim3(128), 0, stream,
                       (const float*)partial, out, s, ldo, gp);
}

}  // namespace

// Floats of scratch for the partial sums of `slices` slices (the tiles as for hk_gemm_pair).
HK_API long long hk_gemm_pair_partial_floats(int M, int N, int tiles_m, int slices) {
  const int units = (M + 31) / 32, width = 32 * ((units + tiles_m - 1) / tiles_m);
  return (long long)item_floats(width) * ((N + FT - 1) / FT) * tiles_m * slices;
}

// out = a w^T with the epilogues of hk_gemm_tc (0 store, 1 add, 2 to 4 gated, 5 squared relu, 6 narrowed; `limit` and `slope` as
// there).  tiles_m: tiles along the rows of a, of at most 256 rows each; slices: how many slices K is cut into (above 1, `partial`
// holds hk_gemm_pair_partial_floats of scratch); pairs: pairs of SMs at work.  `status`: a device int that a timed-out wait sets.
// Refuses (HK_ERR_UNSUPPORTED) K that is no multiple of 8, a or w off a 16-byte boundary, gated products of odd N, and more rows than
// 32-bit products of tiles and blocks of 32 rows hold (from about four million on).
HK_API int hk_gemm_pair(const void* a, const void* w, void* out, int M, int N, int K, long long ldo, int epilogue, int tiles_m, int slices,
                        int pairs, float* partial, int* status, float limit, float slope, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 7) || ((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return HK_ERR_UNSUPPORTED;
  if (epilogue < EPI_STORE || epilogue > EPI_NARROW || (IS_GLU(epilogue) && (N & 1))) return HK_ERR_UNSUPPORTED;
  PairShape s;
  s.M = M, s.N = N, s.K = K;
  s.units = (M + 31) / 32;
  s.kb = (K + BK - 1) / BK;
  s.tiles_m = tiles_m;
  s.slices = slices;
  if (tiles_m < 1 || tiles_m > s.units || widest(s) > MAX_W || slices < 1 || slices > s.kb || pairs < 1) return HK_ERR_UNSUPPORTED;
  if ((long long)tiles_m * s.units > 0x7fffffffLL) return HK_ERR_UNSUPPORTED;      // (a tile's rows are found with 32-bit products)
  const long long tiles = (long long)((N + FT - 1) / FT) * tiles_m;
  if (tiles * slices > 0x3fffffffLL || (slices > 1 && partial == nullptr)) return HK_ERR_UNSUPPORTED;
  s.tiles = (int)tiles;
  CUtensorMap ma, mw;
  if (!make_map(&ma, a, M, K, widest(s) / 2)) return HK_ERR_UNSUPPORTED;
  if (!(IS_GLU(epilogue) ? make_gated_map(&mw, w, N / 2, K, 1) : make_map(&mw, w, N, K, 128))) return HK_ERR_UNSUPPORTED;
  const GluParams gp = {limit, slope};
  const PairGroups none = {};
  cudaStream_t st = (cudaStream_t)stream;
  switch (epilogue) {
    case EPI_STORE: return launch_pair<EPI_STORE, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    case EPI_ADD: return launch_pair<EPI_ADD, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    case EPI_SWIGLU: return launch_pair<EPI_SWIGLU, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    case EPI_GEGLU: return launch_pair<EPI_GEGLU, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    case EPI_CLAMPGLU: return launch_pair<EPI_CLAMPGLU, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    case EPI_SQRELU: return launch_pair<EPI_SQRELU, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
    default: return launch_pair<EPI_NARROW, false>(ma, mw, out, s, none, ldo, pairs, partial, status, gp, st);
  }
}

// The grouped form: a has M rows sorted by group, w is [n_groups][N][K], out has a's rows: out[p] = a[p] w[group of p]^T for the rows that
// tiles int32 [max_tiles, 2] = (group, first row; group -1 from the first unused tile on) name, at most tile_rows (a multiple of 32 up
// to 256) of each and none past offsets[group + 1].  Epilogue 0 (fp32 store), 2 or 4 (gated, w[group] = [N/2 gate rows | N/2 up rows]).
HK_API int hk_gemm_pair_grouped(const void* a, const void* w, void* out, int M, int N, int K, long long ldo, int epilogue, int n_groups,
                                const int* tiles, int max_tiles, const int* offsets, int tile_rows, int pairs, int* status, float limit,
                                float slope, void* stream) {
  if (M <= 0 || N <= 0 || n_groups <= 0 || max_tiles <= 0) return 0;
  if (K <= 0 || (K & 7) || ((uintptr_t)a & 15) || ((uintptr_t)w & 15) || pairs < 1) return HK_ERR_UNSUPPORTED;
  if ((epilogue != EPI_STORE && epilogue != EPI_SWIGLU && epilogue != EPI_CLAMPGLU) || (IS_GLU(epilogue) && (N & 1))) return HK_ERR_UNSUPPORTED;
  if (tile_rows < 32 || tile_rows > MAX_W || (tile_rows & 31)) return HK_ERR_UNSUPPORTED;
  if ((long long)n_groups * N > 0x7fffffffLL) return HK_ERR_UNSUPPORTED;
  PairShape s = {};
  s.M = M, s.N = N, s.K = K;
  s.kb = (K + BK - 1) / BK;
  s.slices = 1;
  s.tiles = (N + FT - 1) / FT;          // (of one tile of rows)
  if ((long long)s.tiles * max_tiles > 0x3fffffffLL) return HK_ERR_UNSUPPORTED;
  const PairGroups g = {tiles, offsets, max_tiles, tile_rows};
  CUtensorMap ma, mw;
  if (!make_map(&ma, a, M, K, tile_rows / 2)) return HK_ERR_UNSUPPORTED;
  if (!(IS_GLU(epilogue) ? make_gated_map(&mw, w, N / 2, K, n_groups) : make_map(&mw, w, n_groups * N, K, 128))) return HK_ERR_UNSUPPORTED;
  const GluParams gp = {limit, slope};
  cudaStream_t st = (cudaStream_t)stream;
  if (epilogue == EPI_STORE) return launch_pair<EPI_STORE, true>(ma, mw, out, s, g, ldo, pairs, nullptr, status, gp, st);
  if (epilogue == EPI_SWIGLU) return launch_pair<EPI_SWIGLU, true>(ma, mw, out, s, g, ldo, pairs, nullptr, status, gp, st);
  return launch_pair<EPI_CLAMPGLU, true>(ma, mw, out, s, g, ldo, pairs, nullptr, status, gp, st);
}
