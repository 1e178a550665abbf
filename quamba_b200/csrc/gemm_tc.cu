// int8 x int8 -> int32 GEMM on the Blackwell tensor cores (tcgen05.mma kind::i8, TMEM accumulator),
// operands streamed by TMA into 128-byte-swizzled shared memory.
//
//   C[m, n] = sum_k A[m, k] * W[n, k]      A (M, K) and W (N, K) both K-contiguous int8.
//
// One persistent kernel in two forms, both walking tiles of TR rows x bn columns (bn a runtime value: a multiple of 16 for the
// one-CTA instruction, of 32 for the pair's, the shapes kind::i8 is defined for):
//   * pair: two CTAs of a cluster share a 256 x bn tile (cta_group::2).  Each holds its 128 rows of A and HALF of the bn rows
//     of W, so a K step brings (128 + bn / 2) * 32 bytes through a CTA's shared memory where one CTA on its own would bring
//     (128 + bn) * 32.  Each CTA's producer loads its own halves and counts them on the LEADER's barrier; the leader issues
//     every MMA, and its commits release the stages and announce the accumulators in both CTAs.  No load is multicast.
//   * single: one CTA, up to 128 rows: batched decode, where the weights are streamed once and M fills no second CTA.  Where
//     the columns alone do not put a CTA on every SM, K is cut over the CTAs of a cluster: each accumulates its share, leaves
//     the int32 partial tile in its shared memory, and after a cluster barrier finishes a slice of the columns from all of
//     them (integers: the sum is the same in any order).
// Warp 0 produces (one elected lane), warp 1 owns the TMEM allocation and issues the MMAs (one elected lane), warps 2..9 run
// the epilogue: two accumulators in tensor memory, so that the epilogue of a tile overlaps the main loop of the next one.
//
// What bounds it, as measured at 16384 x 10240 x 2560 (1.92 POP/s before, 3.36 after):
//   * the epilogue: with one global load per element for its column scale and 16-byte stores scattered over 32 rows, draining
//     a 128 x 256 tile took 16000 cycles against 10240 of MMAs; see store_piece64;
//   * the single issuing and producing threads: some 400 cycles of dependent instructions per stage, hence two slabs of K
//     (eight MMAs) per stage and one 3-D load per operand and stage;
//   * L2: the tile order keeps a band of A in L2 while W passes by (16384 x 4096 x 8192: 440 -> 329 us);
//   * then the power cap: at 1.4 GHz under a sustained load the tensor pipe is busy 85 % of the time.
// Out-of-range rows / columns / K tails are zero-filled by TMA and masked or dropped in the epilogue, so M, N and K need no
// padding (K and the row pitches only have to be multiples of 16 bytes, the TMA rule).  Every wait is bounded; on expiry the
// kernel records QB_ERR_TIMEOUT in the device status word, frees its TMEM and returns.
#include <algorithm>
#include "tc_common.cuh"
#include "linear_epilogue.cuh"

namespace qb {

namespace {

constexpr int BM = 128, BK = 128;   // rows of A per CTA; bytes of K per slab = one swizzle atom row
constexpr int kMaxBN = 256;         // columns of a tile, and of a TMEM accumulator
constexpr int kSlabs = 2;           // slabs per stage
constexpr int kMaxStages = 8;
constexpr int kThreads = 64 + 256;
constexpr int kEpiWarps = 8;

using namespace tc;

// 32 consecutive accumulator columns of one output row -> scaled, converted, stored (16-byte stores when the layout allows).
__device__ __forceinline__ void store_chunk(const uint32_t (&r)[32], int m, int nb, int M, int N, const Epilogue& ep) {
  if (nb >= N) return;  // whole warp agrees
  if (ep.transpose) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (m < M && nb + j < N) ep.store((int)r[j], m, nb + j);
  } else if (m < M) {
    const bool full = nb + 32 <= N;
    if (ep.out_kind == kOutF16 && full && (ep.out_stride % 8 == 0) &&
        ((reinterpret_cast<uintptr_t>(ep.out) & 15) == 0) && (nb % 8 == 0)) {
      __half* dst = static_cast<__half*>(ep.out) + (int64_t)m * ep.out_stride + nb;
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        __align__(16) __half2 h[4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
          h[t] = __floats2half2_rn(ep.scaled((int)r[j + 2 * t], m, nb + j + 2 * t),
                                   ep.scaled((int)r[j + 2 * t + 1], m, nb + j + 2 * t + 1));
        *reinterpret_cast<uint4*>(dst + j) = *reinterpret_cast<const uint4*>(h);
      }
    } else if ((ep.out_kind == kOutS8Rne || ep.out_kind == kOutS8Away) && full && (ep.out_stride % 16 == 0) &&
               ((reinterpret_cast<uintptr_t>(ep.out) & 15) == 0) && (nb % 16 == 0)) {
      int8_t* dst = static_cast<int8_t*>(ep.out) + (int64_t)m * ep.out_stride + nb;
#pragma unroll
      for (int j = 0; j < 32; j += 16) {
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int b = j + 4 * t;
          w[t] = pack4_s8(ep.to_s8(ep.scaled((int)r[b], m, nb + b)), ep.to_s8(ep.scaled((int)r[b + 1], m, nb + b + 1)),
                          ep.to_s8(ep.scaled((int)r[b + 2], m, nb + b + 2)),
                          ep.to_s8(ep.scaled((int)r[b + 3], m, nb + b + 3)));
        }
        *reinterpret_cast<uint4*>(dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (nb + j < N) ep.store((int)r[j], m, nb + j);
    }
  }
}

// The epilogue of aligned row-major outputs, 64 columns of a warp's 32 rows at a time: scales from shared memory (one read per
// four columns for the whole warp instead of one cached global load per element), conversion, and the converted piece leaves
// through a swizzled shared-memory buffer and one TMA store, so that global memory sees whole 64- or 128-byte row pieces; rows
// and columns outside the matrix are dropped by the store.  The fp32 steps and their order are those of Epilogue::scaled.
// int8: clamp, then round half to even by adding 1.5 * 2^23, whose low mantissa byte is the two's complement result (the
// conversion pipe, 16 results a clock, is left to the int32 -> fp32 conversions).  The clamp would make -128 of a NaN where every
// other form of the product stores 0, so a piece with a scale that could give one (|acc| <= 2^31: a column scale from 2^96 on can
// overflow, which times a row scale of 0 is NaN) tests its values; knowing costs one vote per piece of 64 columns.
constexpr int kOutBuf = 32 * 128;        // bytes of a warp's buffer: 32 rows of 64 fp16 or int8
__device__ __forceinline__ uint32_t round_s8_bits(float v) { return __float_as_uint(fminf(fmaxf(v, -128.0f), 127.0f) + 12582912.0f); }

__device__ __forceinline__ void store_piece64(const uint32_t (&r0)[32], const uint32_t (&r1)[32], const float* scale, float row_scale, bool f16,
                                              uint8_t* buf, int lane, const CUtensorMap* map, int n0, int m0) {
  if (lane == 0) bulk_wait_read<0>();    // the piece before has left the buffer
  __syncwarp();
  const bool tame = __all_sync(0xffffffffu, fabsf(scale[lane]) < 0x1p96f && fabsf(scale[lane + 32]) < 0x1p96f && fabsf(row_scale) < INFINITY);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
      float v[16];
#pragma unroll
      for (int t = 0; t < 16; t += 4) {
        const float4 cs = *reinterpret_cast<const float4*>(scale + h * 32 + j + t);
        const float c[4] = {cs.x, cs.y, cs.z, cs.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) v[t + e] = ((float)(int)(h == 0 ? r0[j + t + e] : r1[j + t + e]) * c[e]) * row_scale;
      }
      if (f16) {                         // 128-byte rows: 16-byte piece p of row r sits at p ^ (r & 7)
        uint4 w[2];
        __half2* hp = reinterpret_cast<__half2*>(w);
#pragma unroll
        for (int t = 0; t < 8; ++t) hp[t] = __floats2half2_rn(v[2 * t], v[2 * t + 1]);
        const int p = (h * 32 + j) / 8;
        *reinterpret_cast<uint4*>(buf + lane * 128 + ((p ^ (lane & 7)) << 4)) = w[0];
        *reinterpret_cast<uint4*>(buf + lane * 128 + (((p + 1) ^ (lane & 7)) << 4)) = w[1];
      } else {                           // 64-byte rows: piece p of row r sits at p ^ ((r >> 1) & 3)
        if (!tame) {
#pragma unroll
          for (int t = 0; t < 16; ++t) v[t] = v[t] == v[t] ? v[t] : 0.0f;
        }
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t lo = __byte_perm(round_s8_bits(v[4 * t]), round_s8_bits(v[4 * t + 1]), 0x0040);
          const uint32_t hi = __byte_perm(round_s8_bits(v[4 * t + 2]), round_s8_bits(v[4 * t + 3]), 0x0040);
          w[t] = __byte_perm(lo, hi, 0x5410);
        }
        const int p = (h * 32 + j) / 16;
        *reinterpret_cast<uint4*>(buf + lane * 64 + ((p ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_2d(map, buf, f16 ? n0 * 2 : n0, m0);
    bulk_commit();
  }
}

constexpr int kFixedSmem = kEpiWarps * kOutBuf + 2 * kMaxBN * (int)sizeof(float) + 256;   // output buffers, scales, barriers
constexpr int kSmemLimit = 232448;                                                       // 227 KB

struct TileShape {
  int bn;            // tile columns
  int a_rows;        // rows of A a CTA loads (128, or fewer where M is: the MMA's 128-row read then runs on into whatever
                     // follows, which only reaches output rows that are dropped)
  int stages, stage_bytes, ring_bytes;
  int band;          // tile rows per band of the tile order
  int splits;        // single form: CTAs of a cluster that share one tile's K
  int slab_maps;     // 3-D maps (K a multiple of 128), else one 2-D load per slab
  int tma_out;       // outputs leave by TMA
};

__device__ __forceinline__ int4 ld_cluster_int4(uint32_t addr) {
  int4 v;
  asm volatile("ld.shared::cluster.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

template <bool kPair>
__global__ void __launch_bounds__(kThreads, 1)
gemm_s8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_o,
               int M, int N, int K, const TileShape ts, Epilogue ep, int* status, int early) {
  if (early) grid_dependency_launch();
  // aligned for the swizzle patterns, and at the same offset in both CTAs: the leader's descriptors and barrier addresses
  // are used for its peer's shared memory
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* out_buf = smem + ts.ring_bytes;
  float* scales = reinterpret_cast<float*>(out_buf + kEpiWarps * kOutBuf);   // [2][kMaxBN]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(scales + 2 * kMaxBN);     // (pair: the leader's are used)
  uint64_t* empty_bar = full_bar + kMaxStages;                               // one set per CTA
  uint64_t* acc_full = empty_bar + kMaxStages;                               // [2], one set per CTA
  uint64_t* acc_empty = acc_full + 2;                                        // [2] (pair: the leader's are used)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  constexpr int kCtas = kPair ? 2 : 1, kRows = kCtas * BM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = kPair ? cluster_rank() : 0u;
  const int group = kPair ? 2 : ts.splits;                                   // CTAs of a cluster
  const int unit = blockIdx.x / group, units = gridDim.x / group;
  const int split = !kPair && ts.splits > 1 ? (int)cluster_rank() : 0;
  const int bn = ts.bn, w_rows = bn / kCtas;
  const int tiles_m = (M + kRows - 1) / kRows, tiles_n = (N + bn - 1) / bn;
  const int tiles = tiles_m * tiles_n;
  const int all_kb = (K + kSlabs * BK - 1) / (kSlabs * BK);                  // stages per tile
  const int kb_begin = split * all_kb / ts.splits, num_kb = (split + 1) * all_kb / ts.splits - kb_begin;
  const int my_tiles = unit < tiles ? (tiles - unit + units - 1) / units : 0;
  // Tile order: bands of tile rows, M-fastest inside a band.  Units that run at the same time read the same W tile, and a
  // band's rows of A stay in L2 while all of W passes by.
  auto tile_at = [&](int i, int& m0, int& n0) {
    const int t = unit + i * units, per_band = ts.band * tiles_n, g = t / per_band, r = t - g * per_band;
    const int rows = min(ts.band, tiles_m - g * ts.band), tn = r / rows;
    m0 = (g * ts.band + (r - tn * rows)) * kRows + (int)rank * BM;
    n0 = tn * bn;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < ts.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], kCtas); }
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_w);
    if (ts.tma_out) prefetch_tensormap(&tmap_o);
  }
  if (warp == 1) {
    if (kPair) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (kPair) cluster_sync();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // launched as a programmatic dependent: barriers, tensor memory and descriptors above were set up while the kernel
  // before this one may still have been running; A (and per-row scales) are read from here on, by TMA or past L1
  grid_dependency_wait();

  if (warp == 0) {
    if (lane == 0) {
      const int a_slab = ts.a_rows * BK, w_slab = w_rows * BK;
      const uint32_t bytes = (uint32_t)(kCtas * kSlabs * (a_slab + w_slab));
      const uint32_t bar0 = kPair ? map_to_rank(full_bar, 0) : smem_u32(full_bar);
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        int m0, n0;
        tile_at(i, m0, n0);
        n0 += (int)rank * w_rows;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_spin(&empty_bar[s], ph, status, QB_ERR_TIMEOUT);
          if (!ok) break;
          uint8_t* sa = smem + s * ts.stage_bytes;
          uint8_t* sw = sa + kSlabs * a_slab;
          const uint32_t bar = bar0 + 8u * (uint32_t)s;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
          const int k0 = (kb_begin + kb) * kSlabs;
          if (ts.slab_maps) {
            tma_load_3d<kPair>(sa, &tmap_a, bar, 0, m0, k0);
            tma_load_3d<kPair>(sw, &tmap_w, bar, 0, n0, k0);
          } else {
#pragma unroll
            for (int j = 0; j < kSlabs; ++j) {
              tma_load_2d<kPair>(sa + j * a_slab, &tmap_a, bar, (k0 + j) * BK, m0);
              tma_load_2d<kPair>(sw + j * w_slab, &tmap_w, bar, (k0 + j) * BK, n0);
            }
          }
          if (++s == ts.stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = make_idesc(/*c=s32*/ 2, /*a=s8*/ 1, /*b=s8*/ 1, 0, 0, kRows, (uint32_t)bn);
      const SmemDesc da0 = make_smem_desc2(smem_u32(smem), 16, 1024, kSwizzle128B);
      const uint32_t a_slab = (uint32_t)(ts.a_rows * BK), w_slab = (uint32_t)(w_rows * BK);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const int b = i & 1;
        ok = mbar_wait_spin(&acc_empty[b], (uint32_t)(((i >> 1) & 1) ^ 1), status, QB_ERR_TIMEOUT);  // the epilogue has drained it
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + (uint32_t)(b * kMaxBN);
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_spin(&full_bar[s], ph, status, QB_ERR_TIMEOUT);
          if (!ok) break;
          tc_fence_after_sync();
          const SmemDesc da = desc_advance(da0, (uint32_t)(s * ts.stage_bytes));
          const SmemDesc dw = desc_advance(da, kSlabs * a_slab);
#pragma unroll
          for (int j = 0; j < kSlabs; ++j) {
            const SmemDesc daj = desc_advance(da, j * a_slab), dwj = desc_advance(dw, j * w_slab);
#pragma unroll
            for (int k = 0; k < BK / 32; ++k) {
              if (kPair) umma_i8_pair(acc, desc_advance(daj, k * 32), desc_advance(dwj, k * 32), idesc, (kb | j | k) != 0 ? 1u : 0u);
              else umma_i8(acc, desc_advance(daj, k * 32), desc_advance(dwj, k * 32), idesc, (kb | j | k) != 0 ? 1u : 0u);
            }
          }
          if (kPair) umma_commit_pair(&empty_bar[s]); else umma_commit(&empty_bar[s]);   // frees the stage once read
          if (++s == ts.stages) { s = 0; ph ^= 1; }
        }
        if (kPair) umma_commit_pair(&acc_full[b]); else umma_commit(&acc_full[b]);      // (arrives even after an aborted loop)
      }
    }
  } else {
    // Epilogue warp w may touch TMEM lanes [32 * (w % 4), 32 * (w % 4) + 32); the two warps of a quarter share its columns.
    const int q = warp & 3, ew = warp - 2;
    const int half = ew >> 2;
    const bool lead = warp == 2 && lane == 0;
    // 64-column pieces; where bn is no multiple of 64 the last one starts at bn - 64 and repeats columns of the one before
    const int pieces = (bn + 63) / 64;
    const int p_begin = half == 0 ? 0 : (pieces + 1) / 2, p_end = half == 0 ? (pieces + 1) / 2 : pieces;
    const int part_pitch = bn * 4 + 16;       // conflict-free 16-byte accesses by 32 rows
    const uint32_t leader_empty = kPair ? map_to_rank(acc_empty, 0) : 0u;
    for (int i = 0; i < my_tiles; ++i) {
      const int b = i & 1;
      int m0, n0;
      tile_at(i, m0, n0);
      const int n_end = min(N, n0 + bn);      // columns past the tile belong to the next one (or to nobody)
      const int m = m0 + q * 32 + lane;
      // the tile's column scales and this lane's row scale, while the accumulator is still being computed
      float* sc = scales + b * kMaxBN;
      float row_scale = 0.0f;
      if (ts.tma_out || (ts.splits > 1 && !ep.use_alpha)) {   // (with the scalar by value there are no scale pointers)
        const int c = threadIdx.x - 64;
        if (c < bn) sc[c] = n0 + c < N ? ep.col_scale[ep.col_per ? n0 + c : 0] : 0.0f;
        row_scale = ep.row_scale[ep.row_per ? min(m, M - 1) : 0];
      }
      // one thread polls, the eight warps meet at a named barrier that also carries the outcome (and publishes the scales)
      uint32_t ok = 1;
      if (lead) ok = mbar_wait(&acc_full[b], (uint32_t)((i >> 1) & 1), status, QB_ERR_TIMEOUT) ? 1u : 0u;
      uint32_t all_ok;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                   : "=r"(all_ok) : "r"(ok) : "memory");
      if (!all_ok) break;
      tc_fence_after_sync();
      const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * kMaxBN);
      auto release = [&]() {
        tc_fence_before_sync();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (lead) { if (kPair) mbar_arrive_remote(leader_empty + 8u * (uint32_t)b); else mbar_arrive(&acc_empty[b]); }
      };
#pragma unroll 1
      for (int p = p_begin; p < p_end; ++p) {
        const int c = max(min(p * 64, bn - 64), 0);
        uint32_t r0[32], r1[32];
        tmem_ld_32x32(acc + (uint32_t)c, r0);
        tmem_ld_32x32(acc + (uint32_t)c + 32, r1);
        tmem_ld_wait();
        if (p + 1 == p_end) release();        // the last columns are in registers: hand the accumulator back before storing them
        if (n0 + c >= N || m0 + q * 32 >= M) continue;
        if (!kPair && ts.splits > 1) {        // the partial tile, in the stages (every MMA that read them has completed)
          int4* dst = reinterpret_cast<int4*>(smem + (q * 32 + lane) * part_pitch + c * 4);
          if (m < M) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              dst[j] = make_int4(r0[4 * j], r0[4 * j + 1], r0[4 * j + 2], r0[4 * j + 3]);
              dst[8 + j] = make_int4(r1[4 * j], r1[4 * j + 1], r1[4 * j + 2], r1[4 * j + 3]);
            }
          }
        } else if (ts.tma_out) {
          store_piece64(r0, r1, sc + c, row_scale, ep.out_kind == kOutF16, out_buf + ew * kOutBuf, lane, &tmap_o, n0 + c, m0 + q * 32);
        } else {
          store_chunk(r0, m, n0 + c, M, n_end, ep);
          store_chunk(r1, m, n0 + c + 32, M, n_end, ep);
        }
      }
      if (p_begin == p_end) release();        // a half without pieces still takes part in the hand-over
    }
    if (ts.tma_out && lane == 0) bulk_wait_all<0>();
  }
  if (!kPair && ts.splits > 1) {
    __syncwarp();                             // the producing and the issuing lane come back to their warps: the barrier is .aligned
    cluster_sync();                           // all partial tiles are in shared memory
    int m0, n0;
    tile_at(0, m0, n0);
    const int quads = bn / 4, q_begin = split * quads / ts.splits, q_count = (split + 1) * quads / ts.splits - q_begin;
    const uint32_t base = smem_u32(smem), pitch = (uint32_t)(bn * 4 + 16);
    const bool vec = !ep.transpose && ep.out_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(ep.out) & 7) == 0 && N % 4 == 0 &&
                     (ep.out_kind == kOutF16 || ep.out_kind == kOutS8Rne) && !ep.use_alpha;
    for (int i = threadIdx.x; i < M * q_count; i += kThreads) {
      const int m = i / q_count, c = (q_begin + i % q_count) * 4;
      const uint32_t addr = base + (uint32_t)m * pitch + (uint32_t)c * 4;
      int4 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {           // all shares of a quad are in flight together
        if (r < ts.splits) {
          uint32_t ra;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(r));
          v[r] = ld_cluster_int4(ra);
        }
      }
      int a4[4] = {0, 0, 0, 0};
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < ts.splits) { a4[0] += v[r].x; a4[1] += v[r].y; a4[2] += v[r].z; a4[3] += v[r].w; }
      if (vec && n0 + c < N) {
        const float rs = ep.row_scale[ep.row_per ? m : 0];
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = ((float)a4[e] * scales[c + e]) * rs;
        const int64_t at = (int64_t)m * ep.out_stride + n0 + c;
        if (ep.out_kind == kOutF16) {
          __half2 h[2] = {__floats2half2_rn(f[0], f[1]), __floats2half2_rn(f[2], f[3])};
          *reinterpret_cast<uint2*>(static_cast<__half*>(ep.out) + at) = *reinterpret_cast<const uint2*>(h);
        } else {
          *reinterpret_cast<uint32_t*>(static_cast<int8_t*>(ep.out) + at) = pack4_s8(rint_s8(f[0]), rint_s8(f[1]), rint_s8(f[2]), rint_s8(f[3]));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n0 + c + e < N) ep.store(a4[e], m, n0 + c + e);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (kPair || ts.splits > 1) cluster_sync();    // no CTA leaves while its peer's loads, commits or MMAs may still touch its shared memory
  if (warp == 1) {
    tc_fence_after_sync();
    if (kPair) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
  }
}

// ---- issue-rate measurement of tcgen05.mma kind::i8 -------------------------------------------------------------------
// One CTA per SM; operands (pseudo-random int8, the 128-byte-swizzled tile shapes of the GEMM above) sit in shared memory
// and are never reloaded; one thread issues `groups` x four M128 N256 K32 MMAs into two alternating accumulators and
// commits each group of four to a ring of mbarriers it waits on two groups behind, the way the GEMM's stage ring paces it.
// What comes out is the tensor pipe's dense int8 rate with shared-memory operands and no epilogue: the denominator of the
// GEMM rooflines.
constexpr int kPeakRing = 4;
constexpr int kPeakBytes = BM * BK + kMaxBN * BK;
__global__ void __launch_bounds__(128, 1) i8_mma_peak_kernel(int groups, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPeakBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kPeakRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kPeakBytes / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(smem)[i] = (uint32_t)(i * 2654435761u) ^ (blockIdx.x * 40503u);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPeakRing; ++s) mbar_init(&bars[s], 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes of the operands -> async proxy (MMA)
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc = make_idesc(2, 1, 1, 0, 0, BM, kMaxBN);
    const SmemDesc da = make_smem_desc2(smem_u32(smem), 16, 1024, kSwizzle128B);
    const SmemDesc dw = desc_advance(da, BM * BK);
    bool ok = true;
    for (int g = 0; g < groups && ok; ++g) {
      if (g >= kPeakRing) ok = mbar_wait_spin(&bars[g % kPeakRing], (uint32_t)(((g / kPeakRing) - 1) & 1), status, QB_ERR_TIMEOUT);
      if (!ok) break;
      const uint32_t acc = tmem_base + (uint32_t)((g & 1) * kMaxBN);
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_i8(acc, desc_advance(da, k * 32), desc_advance(dw, k * 32), idesc, g >= 2 ? 1u : (k ? 1u : 0u));
      umma_commit(&bars[g % kPeakRing]);
    }
    // drain: the last kPeakRing groups
    for (int g = max(0, groups - kPeakRing); g < groups && ok; ++g)
      ok = mbar_wait_spin(&bars[g % kPeakRing], (uint32_t)((g / kPeakRing) & 1), status, QB_ERR_TIMEOUT);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encoder() {
  static EncodeTiledFn fn = nullptr;
  if (fn != nullptr) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(p);
  return fn;
}

}  // namespace

int encode_tmap_2d_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes,
                      uint32_t box_rows, uint32_t box_cols, bool swizzle64) {
  EncodeTiledFn enc = get_encoder();
  QB_REQUIRE(enc != nullptr, QB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t gdim[2] = {cols, rows};
  const cuuint64_t gstride[1] = {pitch_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QB_REQUIRE(r == CUDA_SUCCESS, QB_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return QB_OK;
}

int encode_tmap_slabs_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows, uint32_t slabs) {
  EncodeTiledFn enc = get_encoder();
  QB_REQUIRE(enc != nullptr, QB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t gdim[3] = {128, rows, cols / 128};
  const cuuint64_t gstride[2] = {pitch_bytes, 128};
  const cuuint32_t box[3] = {128, box_rows, slabs};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), gdim, gstride, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QB_REQUIRE(r == CUDA_SUCCESS, QB_ERR_CUDA, "cuTensorMapEncodeTiled (slabs) failed with code %d", (int)r);
  return QB_OK;
}

int encode_tmap_4d(CUtensorMap* out, bool f16, bool swizzle128, const void* base, const uint64_t dims[4],
                   const uint64_t strides_bytes[3], const uint32_t box[4]) {
  EncodeTiledFn enc = get_encoder();
  QB_REQUIRE(enc != nullptr, QB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t gdim[4] = {dims[0], dims[1], dims[2], dims[3]};
  const cuuint64_t gstride[3] = {strides_bytes[0], strides_bytes[1], strides_bytes[2]};
  const cuuint32_t bx[4] = {box[0], box[1], box[2], box[3]};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(out, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base),
                         gdim, gstride, bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QB_REQUIRE(r == CUDA_SUCCESS, QB_ERR_CUDA, "cuTensorMapEncodeTiled (4-D) failed with code %d", (int)r);
  return QB_OK;
}

int encode_tmap_f16_4d(CUtensorMap* out, const void* base, const uint64_t dims[4], const uint64_t strides_bytes[3],
                       const uint32_t box[4]) {
  return encode_tmap_4d(out, true, true, base, dims, strides_bytes, box);
}

// Tile columns of the pair form: the multiple of 32 whose rounds of the grid cost least.  Measured time per stage (two slabs, all
// SMs busy, 8192 rows): 745 ns at 256 columns, 654 at 192, 618 at 160, 574 at 128, 493 at 64 -- about 430 + 1.2 bn, the issuing
// threads' share and the operand traffic -- so a wide tile is nearly free and what counts is the number of rounds.
int pick_pair_bn(int64_t M, int64_t N, int64_t units) {
  static const int widths[] = {256, 224, 192, 160, 128, 96, 64};
  int best = 256;
  int64_t best_cost = INT64_MAX;
  for (int w : widths) {
    const int64_t rounds = ceil_div(ceil_div(M, 2 * BM) * ceil_div(N, w), units), cost = rounds * (430 * 5 + 6 * w);
    if (cost < best_cost) { best_cost = cost; best = w; }
  }
  return best;
}
// The single form (at most 128 rows).  Without a split: the narrowest multiple of 16 (and at least 64) columns that needs one
// round of CTAs, so that all of them stream weights at once.  Where that leaves SMs idle, K is split over clusters of two, four
// or eight: what a CTA takes is its stages times what a stage brings, plus about two stages' worth for the exchange.
// (16 rows, 5120 -> 2560: 40 CTAs of 20 stages, 11.7 us; 128 CTAs of 2 to 3 stages, 6 us.)
struct SingleShape { int bn, splits; };
int cluster_capacity(int splits);            // CTAs of clusters of `splits` that are resident at once
SingleShape pick_single(int64_t N, int64_t K, int a_rows) {
  const int64_t stages = ceil_div(K, kSlabs * BK);
  SingleShape best{(int)std::min<int64_t>(kMaxBN, std::max<int64_t>(64, ceil_div(ceil_div(N, sm_count()), 16) * 16)), 1};
  int64_t best_cost = stages * (best.bn + a_rows + 64);
  if (ceil_div(N, 64) * 2 > sm_count()) return best;      // the columns alone occupy half the SMs: the exchange costs more than it gives
  for (int splits = 2; splits <= 8 && splits <= stages; splits *= 2)
    for (int bn = 64; bn <= kMaxBN; bn += 16) {
      if (ceil_div(N, bn) * splits > cluster_capacity(splits)) continue;
      const int64_t cost = (ceil_div(stages, splits) + 2) * (bn + a_rows + 64);
      if (cost < best_cost) { best_cost = cost; best = SingleShape{bn, splits}; }
    }
  return best;
}

template <bool kPair>
int launch_gemm(const int8_t* A, int64_t lda, const int8_t* W, int64_t ldw, int M, int N, int K, int bn, int splits, const Epilogue& ep, int* status,
                cudaStream_t st) {
  constexpr int kCtas = kPair ? 2 : 1;
  QB_REQUIRE(bn % (16 * kCtas) == 0 && bn <= kMaxBN, QB_ERR_UNSUPPORTED, "int8 GEMM: no MMA of %d columns", bn);
  TileShape ts{};
  ts.bn = bn;
  ts.splits = splits;
  ts.a_rows = M >= BM ? BM : (int)ceil_div(M, 8) * 8;
  ts.stage_bytes = kSlabs * BK * (ts.a_rows + bn / kCtas);
  ts.stages = std::min(kMaxStages, (kSmemLimit - kFixedSmem) / ts.stage_bytes);
  ts.slab_maps = K % BK == 0;
  const int64_t tiles_m = ceil_div(M, kCtas * BM), tiles = tiles_m * ceil_div(N, bn);
  // a band of at most 32 MB of A (L2 holds 126 MB, W tiles and outputs pass through it too)
  ts.band = (int)std::min<int64_t>(tiles_m, std::max<int64_t>(1, (32 << 20) / ((int64_t)kCtas * BM * K)));
  const int esize = ep.out_kind == kOutF16 ? 2 : 1;
  ts.tma_out = splits == 1 && !ep.transpose && !ep.use_alpha && (ep.out_kind == kOutF16 || ep.out_kind == kOutS8Rne) && aligned(ep.out, 16) &&
               ep.out_stride * esize % 16 == 0;
  CUtensorMap ta, tw, to{};
  int rc;
  if (ts.slab_maps) {
    rc = encode_tmap_slabs_u8(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, ts.a_rows, kSlabs);
    if (rc == QB_OK) rc = encode_tmap_slabs_u8(&tw, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, (uint32_t)(bn / kCtas), kSlabs);
  } else {
    rc = encode_tmap_2d_u8(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, ts.a_rows, BK);
    if (rc == QB_OK) rc = encode_tmap_2d_u8(&tw, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, (uint32_t)(bn / kCtas), BK);
  }
  if (rc == QB_OK && ts.tma_out)
    rc = encode_tmap_2d_u8(&to, ep.out, (uint64_t)M, (uint64_t)N * esize, (uint64_t)ep.out_stride * esize, 32, 64 * esize, esize == 1);
  if (rc != QB_OK) return rc;
  // the stages also hold the partial tile of a split
  const size_t ring = std::max<size_t>((size_t)ts.stages * ts.stage_bytes, splits > 1 ? (size_t)ts.a_rows * (bn * 4 + 16) : 0);
  ts.ring_bytes = (int)ceil_div((int64_t)ring, 1024) * 1024;
  static PerDeviceOnce attr;
  rc = attr.run([]() -> int {
    QB_CUDA_OK(cudaFuncSetAttribute(gemm_s8_kernel<kPair>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    return QB_OK;
  });
  if (rc != QB_OK) return rc;
  const size_t smem = (size_t)ts.ring_bytes + kFixedSmem;
  const int group = kPair ? 2 : splits;
  const unsigned grid = (unsigned)(std::min<int64_t>(tiles, sm_count() / group) * group);
  const int early = early_overlap() ? 1 : 0;
  if (group > 1)
    launch_dependent_cluster(gemm_s8_kernel<kPair>, (unsigned)group, dim3(grid), dim3(kThreads), smem, st, ta, tw, to, M, N, K, ts, ep, status, early);
  else
    launch_dependent(gemm_s8_kernel<kPair>, dim3(grid), dim3(kThreads), smem, st, ta, tw, to, M, N, K, ts, ep, status, early);
  QB_LAUNCH_OK("gemm_s8_kernel");
  return QB_OK;
}

int cluster_capacity(int splits) {
  static std::atomic<int> cached[64][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
  int c = cached[dev][splits].load(std::memory_order_relaxed);
  if (c == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)splits * 64);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemLimit;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(gemm_s8_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_s8_kernel<false>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      n = 0;
    }
    c = n > 0 ? n * splits : -1;
    cached[dev][splits].store(c, std::memory_order_relaxed);
  }
  return std::min(c, sm_count());
}

int launch_tensor_core_gemm(const int8_t* A, int64_t lda, const int8_t* W, int64_t ldw, int M, int N, int K,
                            const Epilogue& ep, cudaStream_t st) {
  // TMA rules: 16-byte aligned bases and pitches; the inner extent must cover whole 16-byte units.
  if (K % 16 != 0 || lda % 16 != 0 || ldw % 16 != 0 || !aligned(A, 16) || !aligned(W, 16)) return QB_ERR_UNSUPPORTED;
  if (M < 9) return QB_ERR_UNSUPPORTED;   // a few rows are weight-streaming work for the dp4a kernel
  int* status = device_status_ptr();
  QB_REQUIRE(status != nullptr, QB_ERR_CUDA, "device status word unavailable");
  if (path_override(QB_PATH_GEMM_SMALL_TILES)) return launch_gemm<false>(A, lda, W, ldw, M, N, K, 128, 1, ep, status, st);
  if (M <= BM) {
    const SingleShape s = pick_single(N, K, (int)ceil_div(M, 8) * 8);
    return launch_gemm<false>(A, lda, W, ldw, M, N, K, s.bn, s.splits, ep, status, st);
  }
  if (sm_count() < 2) return launch_gemm<false>(A, lda, W, ldw, M, N, K, kMaxBN, 1, ep, status, st);
  return launch_gemm<true>(A, lda, W, ldw, M, N, K, pick_pair_bn(M, N, sm_count() / 2), 1, ep, status, st);
}

}  // namespace qb

extern "C" int qb_gemm_tile(int32_t m, int32_t n, int32_t k, int32_t* rows, int32_t* cols, int32_t* splits) {
  using namespace qb;
  QB_REQUIRE(m > 8 && n > 0 && k > 0 && rows && cols && splits, QB_ERR_INVALID_ARG, "gemm_tile: bad arguments");
  QB_REQUIRE(sm_count() > 1, QB_ERR_CUDA, "gemm_tile: no device");
  const SingleShape s = m <= BM ? pick_single(n, k, (int)ceil_div(m, 8) * 8) : SingleShape{pick_pair_bn(m, n, sm_count() / 2), 1};
  *rows = m <= BM ? BM : 2 * BM;
  *cols = s.bn;
  *splits = s.splits;
  return QB_OK;
}

// Measures the dense int8 tensor rate of the current device (see i8_mma_peak_kernel): runs `repeats` launches of `groups`
// MMA groups per SM on `stream`, times them with CUDA events and returns TOP/s in *tops.  Blocks the host.
extern "C" int qb_i8_mma_peak(int groups, int repeats, void* stream, double* tops, double* ms) {
  using namespace qb;
  QB_REQUIRE(groups > 0 && repeats > 0 && tops != nullptr, QB_ERR_INVALID_ARG, "i8_mma_peak: bad arguments");
  int* status = device_status_ptr();
  QB_REQUIRE(status != nullptr, QB_ERR_CUDA, "device status word unavailable");
  static PerDeviceOnce attr;
  constexpr int smem = kPeakBytes + 1024 + 256;
  const int rc = attr.run([]() -> int {
    QB_CUDA_OK(cudaFuncSetAttribute(i8_mma_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return QB_OK;
  });
  if (rc != QB_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  QB_CUDA_OK(cudaEventCreate(&e0));
  QB_CUDA_OK(cudaEventCreate(&e1));
  const int sms = sm_count();
  i8_mma_peak_kernel<<<sms, 128, smem, st>>>(groups, status);   // warm-up
  QB_CUDA_OK(cudaEventRecord(e0, st));
  for (int r = 0; r < repeats; ++r) i8_mma_peak_kernel<<<sms, 128, smem, st>>>(groups, status);
  QB_CUDA_OK(cudaEventRecord(e1, st));
  QB_CUDA_OK(cudaEventSynchronize(e1));
  QB_LAUNCH_OK("i8_mma_peak_kernel");
  float t = 0.f;
  QB_CUDA_OK(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const double ops = 2.0 * BM * kMaxBN * 32 * 4.0 * groups * (double)sms * repeats;
  *tops = ops / (t * 1e-3) / 1e12;
  if (ms != nullptr) *ms = t;
  return QB_OK;
}
