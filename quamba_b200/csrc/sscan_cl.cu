// Mamba1 int8 selective scan on channel-last tensors (sm_100a): u / delta / z rows of channels and B / C rows of states per
// token, exactly as in_proj, conv1d, x_proj and dt_proj write them.  (The sequence-last kernel in sscan.cu serves callers of
// the extension-level interface; a layer that goes through it has to transpose five tensors first.)
//
// Bound: every (token, channel) needs 16 exponentials and two more for the softplus.  At 16 MUFU results per clock and SM
// that is 1.125 clocks per (token, channel), 0.33 ms for 16 x 1024 tokens of 5120 channels, while its bytes take 0.06 ms.
// What stands in the way of that figure is everything else a (token, channel) issues, so:
//   * the states are walked in pairs with packed fp32 (fma.rn.f32x2), which halves the issue slots of four multiply-adds;
//   * silu(z) is a 256-entry table (z is one byte);
//   * tokens are read straight from global memory, a few ahead; only B and C (shared by all channels) pass through shared
//     memory, widened once per warp, and where there are enough rows two channels per lane share their reads.
// Measured at that size: 0.48 ms (1.6 clocks); the sequence-last kernel takes 0.68 ms after 0.34 ms of transposes.  (Taking a
// part of the exponentials on the fma pipe, by range reduction and a degree-5 polynomial, was slower at every share: the
// kernel is then bound by issue slots.)
//
// Few rows (one short prompt): lanes share a channel, and the sequence is cut into segments, one warp each, in one CTA.
// Every warp first runs its segment from a zero state without outputs (state and summed delta), the prefixes are folded
// through shared memory, and the segment is run again from its true initial state.  512 tokens of 1536 channels: 23 us,
// against 155 us for one serial walk per channel.
#include <algorithm>
#include "tc_common.cuh"
#include "sscan_fwd.cuh"

namespace qb {
namespace {

constexpr int kN = 16;            // states per channel
constexpr int kG = 8;             // tokens fetched ahead and staged together
constexpr int kChunk = 2048;      // the reference keeps the state after every 2048 steps
constexpr int kMaxSegs = 16;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ f2 exp2_mufu2(f2 x) {
  float a, b;
  unpack2(x, a, b);
  return pack2(fast_exp2(a), fast_exp2(b));
}
// bytes -> floats without a conversion instruction: a sign-extended byte added to the bits of 1.5 * 2^23, or byte k of a word
// of biased bytes (v + 128) under the exponent of 2^23
__device__ __forceinline__ float s8f(int v) { return __int_as_float(0x4B400000 + v) - 12582912.0f; }
__device__ __forceinline__ float s8f(uint32_t biased, int k) { return __uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7650 + k)) - 8388736.0f; }

struct Scales { float u, dt, bias, Dv; int softplus; };

// kPairs state pairs of each of kC channels: one token; y[c] is this lane's part of channel c's output without the D term.
// What the channels of a lane share is the read of B and C: a broadcast LDS.128 still returns 512 bytes to the register file,
// and at one channel per lane those returns (4 KB per token and warp) keep the shared-memory pipe busy for 32 clocks of the
// 36 that the MUFU needs.
template <int kPairs, int kC>
struct Lane {
  f2 A[kC][kPairs], h[kC][kPairs];
  template <bool kOut>
  __device__ __forceinline__ void step(const float (&delta)[kC], const float (&du)[kC], const ulonglong2* __restrict__ sB,
                                       const ulonglong2* __restrict__ sC, float (&out)[kC]) {
    f2 y[kC][2];
#pragma unroll
    for (int c = 0; c < kC; ++c) y[c][0] = y[c][1] = 0ull;
#pragma unroll
    for (int i = 0; i < kPairs; i += 2) {
      const ulonglong2 bv = sB[i / 2];
      const f2 b2[2] = {bv.x, bv.y};
      f2 c2[2] = {0ull, 0ull};
      if (kOut) { const ulonglong2 cv = sC[i / 2]; c2[0] = cv.x; c2[1] = cv.y; }
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        const f2 dd = pack2(delta[c], delta[c]), dud = pack2(du[c], du[c]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const f2 x = mul2(dd, A[c][i + j]);
          const f2 e = exp2_mufu2(x);
          h[c][i + j] = fma2(e, h[c][i + j], mul2(b2[j], dud));
          if (kOut) y[c][j] = fma2(h[c][i + j], c2[j], y[c][j]);
        }
      }
    }
    if constexpr (kOut) {
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        float a, b;
        unpack2(add2(y[c][0], y[c][1]), a, b);
        out[c] = a + b;
      }
    }
  }
};

// Sums token j's partial results over the kLanes lanes of a channel and leaves token `sub`'s total in lane `sub`.
template <int kLanes>
__device__ __forceinline__ float own_total(const float (&y)[kLanes], int sub) {
  if (kLanes == 1) return y[0];
  if (kLanes == 2) {
    const float got = __shfl_xor_sync(0xffffffffu, sub ? y[0] : y[kLanes - 1], 1);
    return (sub ? y[kLanes - 1] : y[0]) + got;
  }
  const bool hi = sub & 2;
  const float a = (hi ? y[kLanes - 2] : y[0]) + __shfl_xor_sync(0xffffffffu, hi ? y[0] : y[kLanes - 2], 2);
  const float b = (hi ? y[kLanes - 1] : y[1 % kLanes]) + __shfl_xor_sync(0xffffffffu, hi ? y[1 % kLanes] : y[kLanes - 1], 2);
  return ((sub & 1) ? b : a) + __shfl_xor_sync(0xffffffffu, (sub & 1) ? a : b, 1);
}

// kLanes lanes share a channel, 16 / kLanes states each, and take turns with what a token costs besides its states: of
// kLanes consecutive tokens lane `sub` loads, widens, applies the softplus and finishes the output of one, and passes delta
// and delta * u round by shuffles.  kSeg: the CTA's warps are the segments of one group of channels, else they are groups
// of channels of their own.
template <int kLanes, bool kSeg>
__global__ void __launch_bounds__(kSeg ? 32 * kMaxSegs : 64, kSeg ? 1 : (kLanes == 1 ? 6 : kLanes == 2 ? 10 : 20))
sscan_cl_kernel(qb_sscan_fwd_args a, int seg_len, int early) {
  constexpr int kPairs = kN / 2 / kLanes, kCh = 32 / kLanes, kOwn = kG / kLanes;
  extern __shared__ __align__(16) float dyn[];              // per warp 2 x kG x 32 floats of B | C; then the segments' summaries
  __shared__ float s_silu[256];
  if (early) grid_dependency_launch();
  grid_dependency_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int b = blockIdx.y;                                  // uniform, so that the loads below are uniform base + 32-bit offset
  const int grp = kSeg ? (int)blockIdx.x : (int)blockIdx.x * warps + warp;
  const int sub = lane % kLanes;
  const int d = grp * kCh + lane / kLanes;
  const bool ok = d < a.dim;
  const int dd = min(d, a.dim - 1);
  const int has_z = a.z != nullptr;

  Lane<kPairs, 1> st;
  Scales s;
  s.u = *a.u_scale; s.dt = *a.delta_scale; s.softplus = a.delta_softplus;
  s.Dv = a.D != nullptr ? (*a.D_scale) * (float)a.D[dd] : 0.0f;
  s.bias = a.delta_bias != nullptr ? (*a.delta_bias_scale) * (float)a.delta_bias[dd] : 0.0f;
  const float sA = *a.A_scale;
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const int8_t* q = a.A_log + (int64_t)dd * kN + (sub * kPairs + i) * 2;
    st.A[0][i] = pack2(-__expf(sA * (float)q[0]) * kLog2e, -__expf(sA * (float)q[1]) * kLog2e);
    st.h[0][i] = 0ull;
  }
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s_silu[i] = has_z ? silu_mufu(*a.z_scale * (float)(i - 128)) : 1.0f;
  __syncthreads();

  const int8_t* up = a.u + (int64_t)b * a.u_sb;
  const int8_t* dp = a.delta + (int64_t)b * a.delta_sb;
  const int8_t* zp = has_z ? a.z + (int64_t)b * a.z_sb : up;
  // B and C: lane (4 rows of 8) reads word lane % 8 of tokens lane / 8 and 4 + lane / 8: words 0..3 are B, 4..7 are C
  const bool isC = lane & 4;
  const int8_t* bc = isC ? a.Cm + (int64_t)b * a.C_sb : a.Bm + (int64_t)b * a.B_sb;
  const int u_sl = (int)a.u_sl, d_sl = (int)a.delta_sl, bc_sl = (int)(isC ? a.C_sl : a.B_sl), z_sl = (int)(has_z ? a.z_sl : a.u_sl);
  const float bc_scale = isC ? *a.C_scale : *a.B_scale;
  float* stage = dyn + warp * (2 * kG * 32);
  __half* out = static_cast<__half*>(a.out) + (int64_t)b * a.seqlen * a.dim;

  const int l_begin = kSeg ? warp * seg_len : 0;
  const int l_end = kSeg ? min(a.seqlen, l_begin + seg_len) : a.seqlen;

  auto store_state = [&](int8_t* dst) {
    const float s_st = *a.ssm_state_scale;
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      float x, y;
      unpack2(st.h[0][i], x, y);
      dst[(sub * kPairs + i) * 2] = (int8_t)round_away_s8(x / s_st);
      dst[(sub * kPairs + i) * 2 + 1] = (int8_t)round_away_s8(y / s_st);
    }
  };

  // walks [l_begin, l_end); kOut: writes y and the states, else returns the sum of delta over this lane's tokens
  auto walk = [&](auto out_tag) -> float {
    constexpr bool kOut = decltype(out_tag)::value;
    int ru[kOwn], rd[kOwn], rz[kOwn];
    uint32_t rb[2];
    float sum = 0.0f;
    const int last = l_end - 1;                              // slots past the end read the last token again and are switched off
    auto fetch = [&](int l0) {
#pragma unroll
      for (int t = 0; t < kOwn; ++t) {
        const int l = min(l0 + t * kLanes + sub, last);
        ru[t] = ld_act(up + (uint32_t)(l * u_sl + dd));
        rd[t] = ld_act(dp + (uint32_t)(l * d_sl + dd));
        if (kOut) rz[t] = ld_act(zp + (uint32_t)(l * z_sl + dd));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        rb[i] = ld_act(reinterpret_cast<const uint32_t*>(bc + (uint32_t)(min(l0 + 4 * i + (lane >> 3), last) * bc_sl)) + (lane & 3));
    };
    if (l_begin < l_end) fetch(l_begin);
    int buf = 0;
    for (int l0 = l_begin; l0 < l_end; l0 += kG, buf ^= 1) {
      float* sbc = stage + buf * (kG * 32);
      float delta[kOwn], du[kOwn], skip[kOwn], gate[kOwn];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t w = rb[i] ^ 0x80808080u;
        *reinterpret_cast<float4*>(sbc + (4 * i + (lane >> 3)) * 32 + (lane & 7) * 4) =
            make_float4(bc_scale * s8f(w, 0), bc_scale * s8f(w, 1), bc_scale * s8f(w, 2), bc_scale * s8f(w, 3));
      }
#pragma unroll
      for (int t = 0; t < kOwn; ++t) {
        const float u = s.u * s8f(ru[t]);
        float dl = fmaf(s.dt, s8f(rd[t]), s.bias);
        if (s.softplus) dl = softplus_fast(dl);
        if (l0 + t * kLanes + sub >= l_end) dl = 0.0f;        // a spare slot: decay 1, input 0
        delta[t] = dl;
        du[t] = dl * u;
        if (kOut) {
          skip[t] = s.Dv * u;
          gate[t] = s_silu[rz[t] + 128];
        }
        sum += dl;
      }
      __syncwarp();
      if (l0 + kG < l_end) fetch(l0 + kG);                  // in flight during this group's arithmetic
#pragma unroll
      for (int t = 0; t < kOwn; ++t) {
        float y[kLanes];
#pragma unroll
        for (int j = 0; j < kLanes; ++j) {
          const float dj[1] = {kLanes == 1 ? delta[t] : __shfl_sync(0xffffffffu, delta[t], j, kLanes)};
          const float duj[1] = {kLanes == 1 ? du[t] : __shfl_sync(0xffffffffu, du[t], j, kLanes)};
          const ulonglong2* r = reinterpret_cast<const ulonglong2*>(sbc + (t * kLanes + j) * 32);
          float part[1];
          st.template step<kOut>(dj, duj, r + sub * (kPairs / 2), r + kN / 4 + sub * (kPairs / 2), part);
          y[j] = part[0];
        }
        if (kOut) {
          const int l = l0 + t * kLanes + sub;
          const float v = (own_total<kLanes>(y, sub) + skip[t]) * gate[t];
          if (ok && l < l_end) out[(uint32_t)(l * a.dim + dd)] = __float2half_rn(v);
        }
      }
      if (kOut && ok) {
        const int l = min(l0 + kG, l_end);                  // kChunk is a multiple of kG, and so are the segments' starts
        const int nchunks = (a.seqlen + kChunk - 1) / kChunk;
        if (a.x_states != nullptr && (l % kChunk == 0 || l == a.seqlen))
          store_state(a.x_states + (((int64_t)b * a.dim + d) * nchunks + (l - 1) / kChunk) * kN);
        if (a.final_state != nullptr && l == a.seqlen) store_state(a.final_state + ((int64_t)b * a.dim + d) * kN);
      }
    }
    return sum;
  };

  if (kSeg) {
    // summary of a segment and lane: kN / kLanes states and the summed delta, [segment][value][lane]
    constexpr int kVals = 2 * kPairs + 1;
    float* sums = dyn + warps * (2 * kG * 32);
    float sum = walk(std::false_type{});
#pragma unroll
    for (int o = 1; o < kLanes; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float* mine = sums + (warp * kVals) * 32 + lane;
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      float x, y;
      unpack2(st.h[0][i], x, y);
      mine[(2 * i) * 32] = x;
      mine[(2 * i + 1) * 32] = y;
    }
    mine[(2 * kPairs) * 32] = sum;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPairs; ++i) st.h[0][i] = 0ull;
    for (int w = 0; w < warp; ++w) {
      const float* o = sums + (w * kVals) * 32 + lane;
      const f2 dsum = pack2(o[(2 * kPairs) * 32], o[(2 * kPairs) * 32]);
#pragma unroll
      for (int i = 0; i < kPairs; ++i)
        st.h[0][i] = fma2(exp2_mufu2(mul2(dsum, st.A[0][i])), st.h[0][i], pack2(o[(2 * i) * 32], o[(2 * i + 1) * 32]));
    }
    __syncwarp();
  }
  walk(std::true_type{});
}

// Two adjacent channels per lane, 64 per warp, one warp per CTA: the form for enough rows (64 channels of one sequence) to
// put two warps on every scheduler.  The rows of a launch are rarely a whole number of waves of resident warps (16 sequences
// of 5120 channels are 1280 rows on 1184 slots), and a second wave of a few rows takes as long as the first, so the
// (row, token) space is cut into equal contiguous ranges, one per resident warp: a range is the tail of one row, whole rows,
// and the head of another.  A warp runs its head first and publishes the state after it, and runs its tail last, when the
// warp before it has long published the state the tail starts from.  A head never waits, so neither does the grid.
constexpr int kWideG = 4;          // tokens fetched ahead
constexpr int kWideState = kN * 2 * 32;   // floats handed over per row
constexpr int kStatusScanHandOver = 302;

__global__ void __launch_bounds__(32, 8)
sscan_cl_wide_kernel(qb_sscan_fwd_args a, int groups, int len_pad, int per, float* states, unsigned* flags, int* status, int early) {
  __shared__ __align__(16) float stage[2 * kWideG * 32];
  __shared__ float s_silu[256];
  if (early) grid_dependency_launch();
  grid_dependency_wait();
  const int lane = threadIdx.x;
  const int has_z = a.z != nullptr;
  const float su = *a.u_scale, sdt = *a.delta_scale, sA = *a.A_scale;
  for (int i = lane; i < 256; i += 32) s_silu[i] = has_z ? silu_mufu(*a.z_scale * (float)(i - 128)) : 1.0f;
  __syncwarp();
  // B and C: lane (four rows of eight) reads word lane % 8 of token lane / 8: words 0..3 are B, 4..7 are C
  const bool isC = lane & 4;
  const float bc_scale = isC ? *a.C_scale : *a.B_scale;
  const int u_sl = (int)a.u_sl, d_sl = (int)a.delta_sl, z_sl = (int)(has_z ? a.z_sl : a.u_sl), bc_sl = (int)(isC ? a.C_sl : a.B_sl);

  const int64_t total = (int64_t)a.batch * groups * len_pad;
  const int64_t start = (int64_t)blockIdx.x * per, end = min(total, start + per);
  const int r_first = (int)(start / len_pad), r_last = (int)(end / len_pad);
  const int tail_from = (int)(start % len_pad), head_to = (int)(end % len_pad);
  const int whole_from = r_first + (tail_from != 0);
  // pieces in the order head, whole rows, tail
  for (int r = head_to != 0 ? r_last : whole_from, kind = head_to != 0 ? 0 : 1;;) {
    if (kind == 1 && r >= r_last) {
      if (tail_from == 0) break;
      kind = 2;
      r = r_first;
    }
    const int l_begin = kind == 2 ? tail_from : 0;
    const int l_end = min(a.seqlen, kind == 0 ? head_to : len_pad);
    const int b = r / groups;
    const int d = (r % groups) * 64 + 2 * lane;
    const bool ok = d < a.dim;                               // dim is even
    const int dd = min(d, a.dim - 2);
    Lane<kN / 2, 2> st;
    float Dv[2], bias[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      Dv[c] = a.D != nullptr ? (*a.D_scale) * (float)a.D[dd + c] : 0.0f;
      bias[c] = a.delta_bias != nullptr ? (*a.delta_bias_scale) * (float)a.delta_bias[dd + c] : 0.0f;
#pragma unroll
      for (int i = 0; i < kN / 2; ++i) {
        const int8_t* q = a.A_log + (int64_t)(dd + c) * kN + i * 2;
        st.A[c][i] = pack2(-__expf(sA * (float)q[0]) * kLog2e, -__expf(sA * (float)q[1]) * kLog2e);
        st.h[c][i] = 0ull;
      }
    }
    if (kind == 2) {
      unsigned seen = 0;
      const long long t0 = clock64();
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flags + blockIdx.x - 1) : "memory");
        if (seen != 0) break;
        if (clock64() - t0 > tc::kWaitBudgetCycles) {
          atomicCAS(status, 0, kStatusScanHandOver);
          return;
        }
        __nanosleep(64);
      }
      const float4* in = reinterpret_cast<const float4*>(states + (int64_t)(blockIdx.x - 1) * kWideState) + lane;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < kN / 2; i += 2) {
          const float4 v = __ldcg(in + (c * (kN / 4) + i / 2) * 32);
          st.h[c][i] = pack2(v.x, v.y);
          st.h[c][i + 1] = pack2(v.z, v.w);
        }
    }
    const int8_t* up = a.u + (int64_t)b * a.u_sb;
    const int8_t* dp = a.delta + (int64_t)b * a.delta_sb;
    const int8_t* zp = has_z ? a.z + (int64_t)b * a.z_sb : up;
    const int8_t* bc = isC ? a.Cm + (int64_t)b * a.C_sb : a.Bm + (int64_t)b * a.B_sb;
    __half* out = static_cast<__half*>(a.out) + (int64_t)b * a.seqlen * a.dim;

    uint16_t ru[kWideG], rd[kWideG], rz[kWideG];
    uint32_t rb;
    const int last = l_end - 1;                              // slots past the end read the last token again and are switched off
    auto fetch = [&](int l0) {
#pragma unroll
      for (int t = 0; t < kWideG; ++t) {
        const int l = min(l0 + t, last);
        ru[t] = ld_act(reinterpret_cast<const uint16_t*>(up + (uint32_t)(l * u_sl + dd)));
        rd[t] = ld_act(reinterpret_cast<const uint16_t*>(dp + (uint32_t)(l * d_sl + dd)));
        rz[t] = ld_act(reinterpret_cast<const uint16_t*>(zp + (uint32_t)(l * z_sl + dd)));
      }
      rb = ld_act(reinterpret_cast<const uint32_t*>(bc + (uint32_t)(min(l0 + (lane >> 3), last) * bc_sl)) + (lane & 3));
    };
    fetch(l_begin);
    int buf = 0;
    for (int l0 = l_begin; l0 < l_end; l0 += kWideG, buf ^= 1) {
      float* sbc = stage + buf * (kWideG * 32);
      {
        const uint32_t w = rb ^ 0x80808080u;
        *reinterpret_cast<float4*>(sbc + (lane >> 3) * 32 + (lane & 7) * 4) =
            make_float4(bc_scale * s8f(w, 0), bc_scale * s8f(w, 1), bc_scale * s8f(w, 2), bc_scale * s8f(w, 3));
      }
      float delta[kWideG][2], du[kWideG][2], skip[kWideG][2], gate[kWideG][2];
#pragma unroll
      for (int t = 0; t < kWideG; ++t) {
        const uint32_t wu = ru[t] ^ 0x8080u, wd = rd[t] ^ 0x8080u, wz = rz[t] ^ 0x8080u;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float u = su * s8f(wu, c);
          float dl = fmaf(sdt, s8f(wd, c), bias[c]);
          if (a.delta_softplus) dl = softplus_fast(dl);
          if (l0 + t >= l_end) dl = 0.0f;                    // a spare slot: decay 1, input 0
          delta[t][c] = dl;
          du[t][c] = dl * u;
          skip[t][c] = Dv[c] * u;
          gate[t][c] = s_silu[__byte_perm(wz, 0u, 0x4440 + c)];
        }
      }
      __syncwarp();
      if (l0 + kWideG < l_end) fetch(l0 + kWideG);          // in flight during this group's arithmetic
#pragma unroll
      for (int t = 0; t < kWideG; ++t) {
        const ulonglong2* row = reinterpret_cast<const ulonglong2*>(sbc + t * 32);
        float y[2];
        st.template step<true>(delta[t], du[t], row, row + kN / 4, y);
        const int l = l0 + t;
        if (ok && l < l_end)
          *reinterpret_cast<__half2*>(out + (uint32_t)(l * a.dim + dd)) =
              __floats2half2_rn((y[0] + skip[t][0]) * gate[t][0], (y[1] + skip[t][1]) * gate[t][1]);
      }
      const int l = min(l0 + kWideG, l_end);                // kChunk is a multiple of kWideG, and so are the cuts
      const bool at_chunk = a.x_states != nullptr && (l % kChunk == 0 || l == a.seqlen), at_end = a.final_state != nullptr && l == a.seqlen;
      if (ok && (at_chunk || at_end)) {
        const float s_st = *a.ssm_state_scale;
        const int nchunks = (a.seqlen + kChunk - 1) / kChunk;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t q[4];
#pragma unroll
          for (int i = 0; i < kN / 2; i += 2) {
            float x[4];
            unpack2(st.h[c][i], x[0], x[1]);
            unpack2(st.h[c][i + 1], x[2], x[3]);
            q[i / 2] = pack4_s8(round_away_s8(x[0] / s_st), round_away_s8(x[1] / s_st), round_away_s8(x[2] / s_st), round_away_s8(x[3] / s_st));
          }
          const int64_t ch = (int64_t)b * a.dim + d + c;
          const uint4 v = make_uint4(q[0], q[1], q[2], q[3]);
          if (at_chunk) *reinterpret_cast<uint4*>(a.x_states + (ch * nchunks + (l - 1) / kChunk) * kN) = v;
          if (at_end) *reinterpret_cast<uint4*>(a.final_state + ch * kN) = v;
        }
      }
    }
    if (kind == 0) {
      float4* o = reinterpret_cast<float4*>(states + (int64_t)blockIdx.x * kWideState) + lane;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < kN / 2; i += 2) {
          float4 v;
          unpack2(st.h[c][i], v.x, v.y);
          unpack2(st.h[c][i + 1], v.z, v.w);
          o[(c * (kN / 4) + i / 2) * 32] = v;
        }
      __threadfence();
      __syncwarp();
      if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flags + blockIdx.x), "r"(1u) : "memory");
      kind = 1;
      r = whole_from;
    } else if (kind == 1) {
      ++r;
    } else {
      break;
    }
    __syncwarp();
  }
}

template <int kLanes, bool kSeg>
int launch(const qb_sscan_fwd_args& a, int warps, int seg_len, cudaStream_t st) {
  const int groups = (int)ceil_div(a.dim, 32 / kLanes);
  const dim3 grid((unsigned)(kSeg ? groups : ceil_div(groups, warps)), (unsigned)a.batch);
  const size_t smem = (size_t)warps * (2 * kG * 32 + (kSeg ? (kN / kLanes + 1) * 32 : 0)) * sizeof(float);
  static PerDeviceOnce attr;
  const int rc = attr.run([]() -> int {
    QB_CUDA_OK(cudaFuncSetAttribute(sscan_cl_kernel<kLanes, kSeg>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    return QB_OK;
  });
  if (rc != QB_OK) return rc;
  launch_dependent(sscan_cl_kernel<kLanes, kSeg>, grid, dim3((unsigned)warps * 32), smem, st, a, seg_len, early_overlap() ? 1 : 0);
  QB_LAUNCH_OK("sscan_cl_kernel");
  return QB_OK;
}

}  // namespace

// resident warps of the wide kernel: one warp per CTA
int wide_slots() { return sm_count() * 8; }

int64_t sscan_workspace_bytes(int batch, int dim) {
  const int64_t rows = (int64_t)batch * ceil_div(dim, 64);
  return rows > wide_slots() ? (int64_t)wide_slots() * (kWideState * sizeof(float) + sizeof(unsigned)) : 0;
}

int run_sscan_channel_last(const qb_sscan_fwd_args& a, cudaStream_t st) {
  QB_REQUIRE(a.dstate == kN && a.n_groups == 1, QB_ERR_UNSUPPORTED, "sscan_fwd: the channel-last form takes dstate 16 and one B / C group");
  const int64_t top = std::max({a.u_sl, a.delta_sl, a.z_sl, a.B_sl, a.C_sl, (int64_t)a.dim});
  QB_REQUIRE(aligned(a.Bm, 4) && aligned(a.Cm, 4) && a.B_sl % 4 == 0 && a.B_sb % 4 == 0 && a.C_sl % 4 == 0 && a.C_sb % 4 == 0, QB_ERR_INVALID_ARG,
             "sscan_fwd: rows of B and C of the channel-last form must be 4-byte aligned");
  QB_REQUIRE(top >= 0 && top * a.seqlen < (1ll << 31) && a.batch < 65536, QB_ERR_TOO_LARGE, "sscan_fwd: a sequence of the channel-last form spans 2^31 elements");
  const int64_t rows = (int64_t)a.batch * ceil_div(a.dim, 64);
  const int64_t slots = wide_slots();
  const bool pairs = a.dim % 2 == 0 && aligned(a.u, 2) && aligned(a.delta, 2) && aligned(a.z, 2) && (a.u_sl | a.u_sb | a.delta_sl | a.delta_sb | a.z_sl | a.z_sb) % 2 == 0 &&
                     aligned(a.x_states, 16) && aligned(a.final_state, 16);
  // two channels per lane from 0.8 of the slots on: below that the one-channel form's second warp per scheduler wins
  const int64_t need = sscan_workspace_bytes(a.batch, a.dim);
  if (pairs && rows * 5 >= slots * 4 && (need == 0 || (a.workspace != nullptr && a.workspace_bytes >= need))) {
    const int len_pad = (int)ceil_div(a.seqlen, kWideG) * kWideG;
    const int64_t warps = std::min(rows, slots);
    const int per = (int)(ceil_div(ceil_div(rows * len_pad, warps), kWideG) * kWideG);
    float* states = static_cast<float*>(a.workspace);
    unsigned* flags = need > 0 ? reinterpret_cast<unsigned*>(states + slots * kWideState) : nullptr;
    if (need > 0) QB_CUDA_OK(cudaMemsetAsync(flags, 0, slots * sizeof(unsigned), st));
    int* status = device_status_ptr();
    QB_REQUIRE(status != nullptr, QB_ERR_CUDA, "device status word unavailable");
    launch_dependent(sscan_cl_wide_kernel, dim3((unsigned)ceil_div(rows * len_pad, per)), dim3(32), 0, st, a, (int)ceil_div(a.dim, 64), len_pad, per, states, flags, status,
                     early_overlap() ? 1 : 0);
    QB_LAUNCH_OK("sscan_cl_wide_kernel");
    return QB_OK;
  }
  // Fewer rows: lanes share channels until there are about eight warps per SM (each sharing step costs shuffles and more
  // instructions per state, so only as many lanes as that takes), then the sequence is cut as well, at least 16 tokens per
  // segment.  4 x 1024 tokens of 5120 channels (640 warps at one lane per channel): 197 us with two lanes, 267 us segmented.
  const int64_t base = (int64_t)a.batch * ceil_div(a.dim, 32), want = (int64_t)sm_count() * 8;
  if (base >= want || a.seqlen < 32) return launch<1, false>(a, 2, a.seqlen, st);
  if (base * 2 >= want) return launch<2, false>(a, 2, a.seqlen, st);
  if (base * 4 >= want) return launch<4, false>(a, 2, a.seqlen, st);
  const int64_t segs = std::max<int64_t>(2, std::min(std::min<int64_t>(kMaxSegs, a.seqlen / 16), ceil_div(want * 2, base * 4)));
  const int seg_len = (int)ceil_div(ceil_div(a.seqlen, segs), kG) * kG;
  return launch<4, true>(a, (int)ceil_div(a.seqlen, seg_len), seg_len, st);
}

}  // namespace qb
