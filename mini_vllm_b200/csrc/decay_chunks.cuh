// Recurrences with one decay per head and token over chunks of 128 tokens on the tcgen05 tensor cores (ragged steps, bf16).
//
// Both users carry S [N, vdim] through S <- keep_t S + take_t k_t v_t^T, o_t = S^T q_t, with the gates' logarithms (base 2) in R and E:
//
//   o_t = f 2^{R_t + m} (q_t S0) + sum_{s <= t} M_ts v_s         M_ts = (q_t . k_s) 2^{R_t + E_s} D_s
//   S   <- 2^{R_end + m} S0 + sum_s k_s (2^{R_end + E_s} W_s v_s)^T
//
//   state space   R_t = F_t, E_s = -F_s, m = 0, D_s = W_s = dt_s, f = 1 (and + skip on the diagonal of M);  F_t = sum_{s <= t} a dt_s
//   matrix memory R_t = -max(m, max_{s <= t} E_s), E_s = i_s - F_s, m the running maximum in front of the chunk, D_s = f = q_scale, W_s = 1;
//                 F_t = sum_{s <= t} f_s; the maximum behind the chunk is F_end - R_end.  The normaliser is one more column of S, whose
//                 values are 1: a tile of its own.
//
// Every exponent that is used is <= 0.  Inside a block b of 32 tokens 2^{R_t + E_s} is one exponential; across blocks it is the product of
// 2^{R_t - R_b} and 2^{E_s + R_b}, R_b that of the last token of the keys' block: three exponentials a row and one a key.
// F itself, a sum over up to 128 tokens, would round differences that count away.  It is never formed: every token's E and R are measured
// from the middle of its own block, E + B_b and R - B_b with B_b = F after 16 of the block's tokens, beside the steps from one B to the
// next, all of them sums over 16 or 32 tokens.
//
// A CTA walks one sequence (or segment) for one head and 64 columns of v: products of 128 x 128 and 128 x 64 with fp32 accumulators in
// tensor memory.  q, k and v are bf16 and enter exactly; M, S and the scaled values enter as bf16 high + low part, so every factor has 16
// significant bits; S itself stays in fp32 registers.  The matrix memory's scaled values have a third part: its chunks of 16 tokens carried
// every sixteenth weight, the largest, exactly, and with two parts a state was 1.18 times as far from 64 bits as with those (2.05e-6).
//   warps 0..7    M, which goes to tensor memory as an operand, and the scaled values of the next chunk; rows of 32 by warp mod 4, two
//                 warps a row
//   warps 8..15   S and the outputs, shared out alike
//   warp 16       TMA: q, k and v of the next chunk while this one is worked on (two stages; one of q where the third part takes its place)
//   warps 17, 19  tcgen05.mma
//   warp 18       gates of the next chunk
// What bounds it: the issue of the warps that make M and the scaled values; by operations the products need 2,048 tensor-core cycles per 128
// tokens, head and 64 columns.  mma.sync, which this replaces for prompts that fill its chunks, took its own issue for most of the time.
// Measured: 6 prompts of 500 to 2,500 tokens (10,148 in all), state space with 64 heads of 64 x 128: 158 us (280 before); matrix memory with 16
// heads of 128 x 128 and its norm: 242 us (387 before).
#pragma once
#include "chunk_common.cuh"
#include "host_util.cuh"

namespace mvb {

constexpr int kDecayChunk = 128;

struct DecayChunkParams {
  const __nv_bfloat16 *a, *i; int64_t a_stride, i_stride;      // raw gates [tokens, heads]: step, or forget and input
  const float *a_bias, *i_bias, *a_log2e, *skip;               // [heads]
  float cap, q_scale;
  __nv_bfloat16* y; int64_t y_stride;                          // state space: the output
  float *o, *nq, *mt; const float* m0;                         // matrix memory: outputs [tokens, heads, vdim], n . q, m; m in front of the step
  float *state, *n_state, *m_state; const int32_t* slots; int64_t num_slots;
  const int32_t* cu; const int64_t* positions;
  int num_seqs, heads, per_group, n, vdim, vp;
  int seg; float *seg_state, *seg_keep;                        // as in state_space.cu
  int* dev_status;
};

// a descriptor that starts `units` of 16 bytes further on (its address is in the low word, and stays there)
__device__ __forceinline__ uint64_t desc_plus(uint64_t d, uint32_t units) { return (d & 0xffffffff00000000ull) | (static_cast<uint32_t>(d) + units); }

template <int KB, bool EXP>                                    // 64 KB state channels
struct DecayCfg {
  static constexpr int TILE = kDecayChunk * 128;               // 128 rows of 64 bf16
  static constexpr int K = EXP ? 0 : KB * TILE, V = K + KB * TILE, STAGE = V + TILE, PARTS = EXP ? 3 : 2;
  static constexpr int Q_STAGES = EXP ? 1 : 2, Q = EXP ? 2 * STAGE : 0, Q_TILE = EXP ? 0 : STAGE;
  static constexpr int XS = 2 * STAGE + (EXP ? KB * TILE : 0), ST = XS + PARTS * TILE, S_PART = KB * 64 * 128, TABLES = ST + 2 * S_PART;
  // in floats; CS: 2^{E + R_b} (times D); X3: D or R; STEP: m + B_0, B_1 - B_0, B_2 - B_1, B_3 - B_2
  static constexpr int E = 0, CS = 128, X3 = 224, STEP = 352, TABLE = 356;
  static constexpr int BARS = TABLES + 2 * TABLE * 4;
  // pairs: by chunk parity, where whoever waits could otherwise be two phases behind
  enum { K_FULL = 0, K_EMPTY = 2, Q_FULL = 4, Q_EMPTY = 6, V_FULL = 8, V_EMPTY = 10, TAB = 12, TAB_EMPTY = 14, G_FULL = 16, M_READY = 18,
         XS_READY = 20, DS_FULL, S_READY, INTER, Y_FULL, Y_FREE, NUM_BARS };
  static constexpr int SMEM = BARS + NUM_BARS * 8 + 8;
  static constexpr int THREADS = 20 * 32;
  static constexpr int T_M = 0, T_YI = 256, T_DS = 320, T_YA = 448;                      // tensor memory columns; two buffers of M
  static_assert(SMEM <= 232448, "");
  static __device__ __forceinline__ int q_stage(int c) { return c & (Q_STAGES - 1); }      // of chunk c, and the parity of its barriers
  static __device__ __forceinline__ uint32_t q_parity(int c) { return (c / Q_STAGES) & 1; }
};

// The sequence that is k-th in length, the longest first (n <= 32): CTAs start in about this order, so that no long one starts last.
// With more sequences there are waves enough; ranking 64 took longer than it gave (single chunks: 0.73 instead of 0.92 times the speed).
__device__ __forceinline__ int by_length(const int32_t* cu, int n, int k) {
  const int lane = threadIdx.x & 31, mine = lane < n ? cu[lane + 1] - cu[lane] : -1;
  int rank = 0;
  for (int j = 0; j < n; ++j) {
    const int other = __shfl_sync(0xffffffffu, mine, j);
    rank += other > mine || (other == mine && j < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < n && rank == k)) - 1;
}

// The normaliser alone decides the size of an output, and its terms may cancel, so none of it is cut to 16 bits: its part of M is added up
// in fp32 by the warps that make M, and its weights and its state enter the products with a third bf16 part, in columns that are free there.
__device__ __forceinline__ uint4 three_parts(float x) {
  const float h = bf16_round(x), m = bf16_round(x - h);
  return make_uint4(pack_bf16(h, m), pack_bf16(x - h - m, 0.f), 0u, 0u);
}

// a pair of values times w as bf16 high and low parts, and what those two leave
template <bool THREE>
__device__ __forceinline__ void split_value(uint32_t v, float w, uint32_t& hi, uint32_t& lo, uint32_t& third) {
  const float x = bf16_lo(v) * w, y = bf16_hi(v) * w;
  if constexpr (THREE) {
    const float2 minus = make_float2(-1.f, -1.f);
    hi = pack_bf16(x, y);
    const float2 rest = fma_f32x2(make_float2(bf16_lo(hi), bf16_hi(hi)), minus, make_float2(x, y));      // (exact)
    lo = pack_bf16(rest.x, rest.y);
    const float2 last = fma_f32x2(make_float2(bf16_lo(lo), bf16_hi(lo)), minus, rest);
    third = pack_bf16(last.x, last.y);
  } else {
    split_pair(x, y, hi, lo);
  }
}

// EXP: matrix memory.  STATES: only what a segment adds to the state, and what it leaves of the one before, is wanted.
template <int KB, bool EXP, bool STATES>
__global__ void __launch_bounds__(DecayCfg<KB, EXP>::THREADS, 1)
decay_chunk_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                   const DecayChunkParams p) {
  using C = DecayCfg<KB, EXP>;
  constexpr int L = kDecayChunk;
  constexpr float kToLog2 = 1.4426950408889634f, kFromLog2 = 0.6931471805599453f;
  extern __shared__ __align__(1024) uint8_t decay_smem[];      // (128-byte swizzle: 1024-byte boundaries)
  uint8_t* smem = decay_smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BARS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NUM_BARS);
  volatile uint32_t* failed = tmem_slot + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y;
  int s = blockIdx.z, begin, end;
  if (p.seg == 0) {
    if (p.num_seqs <= 32) s = by_length(p.cu, p.num_seqs, s);
    begin = p.cu[s]; end = p.cu[s + 1];
  } else {                                        // the sequence and the rows of a segment slot
    int lo = 0, hi = p.num_seqs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (p.cu[mid] / p.seg + mid <= s) lo = mid; else hi = mid;
    }
    begin = p.cu[lo] + (s - (p.cu[lo] / p.seg + lo)) * p.seg;
    end = min(begin + p.seg, p.cu[lo + 1]);
    s = lo;
  }
  const int n_tok = end - begin;
  const bool last = end == p.cu[s + 1];
  if (n_tok <= 0 || (STATES && last)) return;     // (the whole CTA, before anything is allocated)
  const int n_chunks = (n_tok + L - 1) / L, col0 = blockIdx.x * 64;
  const bool ones = EXP && col0 == p.vdim;        // the normaliser's tile
  int64_t slot = -1;
  if (p.state != nullptr) {
    slot = p.slots[s];
    if (slot >= p.num_slots) { if (tid == 0) report(p.dev_status, kDevBadSlot, s); slot = -1; }
  }

  if (tid == 0) {
    for (int b = 0; b < C::NUM_BARS; ++b) {
      const int kind = b < C::XS_READY ? b & ~1 : b;
      const bool by_eight = kind == C::M_READY || kind == C::TAB_EMPTY || (kind == C::Q_EMPTY && !EXP) || b == C::XS_READY || b == C::S_READY || b == C::Y_FREE;
      mbar_init(&bars[b], by_eight ? 8 : (kind == C::K_EMPTY && !STATES) || kind == C::Q_EMPTY ? 2 : 1);
    }
    *failed = 0;
    fence_mbar_init();
  }
  if (warp == 17) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, lanes = tmem + (static_cast<uint32_t>(warp & 3) << 21);
  auto wait = [&](int bar, uint32_t parity, int where) -> bool {
    if (mbar_try_wait(&bars[bar], parity)) return true;
    return mbar_wait_or_fail(&bars[bar], parity, failed, p.dev_status, where);
  };
  // every lane that wrote before has its writes seen by whom the barrier lets go on
  auto arrive = [&](int bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bar]);
  };
  auto table = [&](int c) { return reinterpret_cast<float*>(smem + C::TABLES) + (c & 1) * C::TABLE; };

  if (warp == 16) {
    // ============================ producer ==========================================================
    if (lane == 0) {
      const int group = h / p.per_group;
      int ks = 0, vs = 0, qs = 0;                 // chunks requested
      for (int c = 0; c < n_chunks; ++c) {
        const int st = c & 1, row = begin + c * L;
        const uint32_t before = ((c >> 1) - 1) & 1;
        uint8_t* base = smem + st * C::STAGE;
        if (c >= 2 && !wait(C::K_EMPTY + st, before, 10)) break;
        mbar_arrive_expect_tx(&bars[C::K_FULL + st], KB * C::TILE);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) tma_load_3d(base + C::K + kb * C::TILE, &k_map, &bars[C::K_FULL + st], kb * 64, group, row);
        ks = c + 1;
        if (c >= 2 && !wait(C::V_EMPTY + st, before, 11)) break;
        if (ones) mbar_arrive(&bars[C::V_FULL + st]);
        else {
          mbar_arrive_expect_tx(&bars[C::V_FULL + st], C::TILE);
          tma_load_3d(base + C::V, &v_map, &bars[C::V_FULL + st], col0, h, row);
        }
        vs = c + 1;
        if (STATES) continue;
        const int qst = C::q_stage(c);
        if (c >= C::Q_STAGES && !wait(C::Q_EMPTY + qst, C::q_parity(c - C::Q_STAGES), 12)) break;
        mbar_arrive_expect_tx(&bars[C::Q_FULL + qst], KB * C::TILE);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) tma_load_3d(smem + C::Q + qst * C::Q_TILE + kb * C::TILE, &q_map, &bars[C::Q_FULL + qst], kb * 64, group, row);
        qs = c + 1;
      }
      // no copy may be in flight when the CTA ends
      for (int c = max(ks - 2, 0); c < ks; ++c) mbar_wait(&bars[C::K_FULL + (c & 1)], (c >> 1) & 1);
      for (int c = max(vs - 2, 0); c < vs; ++c) mbar_wait(&bars[C::V_FULL + (c & 1)], (c >> 1) & 1);
      for (int c = max(qs - C::Q_STAGES, 0); c < qs; ++c) mbar_wait(&bars[C::Q_FULL + C::q_stage(c)], C::q_parity(c));
    }
    __syncwarp();
  } else if (warp == 17) {
    // ============================ tcgen05.mma: q k^T, M v ============================================
    if (lane == 0 && !STATES) {
      constexpr uint32_t ID_G = umma_idesc_bf16(128, 128, false, false), ID_Y = umma_idesc_bf16(128, 64, false, true);
      const uint32_t base = smem_u32(smem);
      auto scores = [&](int c) {                  // over an older M, whose product has been issued
        const uint32_t stage = base + (c & 1) * C::STAGE;
        const uint64_t q = umma_desc_sw128(base + C::Q + C::q_stage(c) * C::Q_TILE, 16, 1024), k = umma_desc_sw128(stage + C::K, 16, 1024);
        if (!wait(C::K_FULL + (c & 1), (c >> 1) & 1, 20) || !wait(C::Q_FULL + C::q_stage(c), C::q_parity(c), 21)) return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4 * KB; ++ks) {
          const uint32_t o = (ks / 4 * C::TILE + ks % 4 * 32) >> 4;
          umma_bf16_ss(tmem + C::T_M + (c & 1) * 128, desc_plus(q, o), desc_plus(k, o), ID_G, ks > 0);
        }
        umma_commit(&bars[C::K_EMPTY + (c & 1)]);
        if (EXP) umma_commit(&bars[C::Q_EMPTY]);
        umma_commit(&bars[C::G_FULL + (c & 1)]);
        return true;
      };
      bool ok = scores(0);
      for (int c = 0; c < n_chunks && ok; ++c) {
        if (c + 1 < n_chunks && !(ok = scores(c + 1))) break;
        ok = wait(C::M_READY + (c & 1), (c >> 1) & 1, 22) && wait(C::V_FULL + (c & 1), (c >> 1) & 1, 23) && (c == 0 || wait(C::Y_FREE, (c - 1) & 1, 24));
        if (!ok) break;
        tc_fence_after();
        if (ones) {                               // M has been added up; plain arrivals, which hand those sums on
          mbar_arrive(&bars[C::V_EMPTY + (c & 1)]);
          mbar_arrive(&bars[C::Y_FULL]);
          continue;
        }
        const uint64_t v = umma_desc_sw128(base + (c & 1) * C::STAGE + C::V, 16, 1024);
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16_ts(tmem + C::T_YA, tmem + C::T_M + (c & 1) * 128 + ks * 16 + part * 8, desc_plus(v, ks * 2048 >> 4), ID_Y, part > 0 || ks > 0);
        umma_commit(&bars[C::V_EMPTY + (c & 1)]);
        umma_commit(&bars[C::Y_FULL]);
      }
    }
    __syncwarp();
  } else if (warp == 19) {
    // ============================ tcgen05.mma: what the chunk adds to S, q S0 ==========================
    // (a second thread: one alone would be busy issuing for longer than the products take)
    if (lane == 0) {
      constexpr uint32_t ID_DS = umma_idesc_bf16(128, 128, true, true), ID_DT = umma_idesc_bf16(128, 64, true, true), ID_Y = umma_idesc_bf16(128, 64, false, true);
      const uint32_t base = smem_u32(smem);
      // the scaled values' high and low parts side by side: one product of 128 columns for both; a third part on top of the low ones
      const uint64_t xs = umma_desc_sw128(base + C::XS, C::TILE, 1024), sd = umma_desc_sw128(base + C::ST, 16, 1024);
      const uint64_t xt = umma_desc_sw128(base + C::XS + 2 * C::TILE, 16, 1024);
      for (int c = 0; c < n_chunks; ++c) {
        const uint32_t stage = base + (c & 1) * C::STAGE;
        // k; scaled values; S, and what the last chunk added has been read
        if (!wait(C::K_FULL + (c & 1), (c >> 1) & 1, 30) || !wait(C::XS_READY, c & 1, 31) || !wait(C::S_READY, c & 1, 32)) break;
        tc_fence_after();
        // k as it lies is the first operand, its channels the rows (with 64 of them, twice)
        const uint64_t kt = umma_desc_sw128(stage + C::K, KB == 2 ? C::TILE : 0, 1024);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma_bf16_ss(tmem + C::T_DS, desc_plus(kt, ks * 2048 >> 4), desc_plus(xs, ks * 2048 >> 4), ID_DS, ks > 0);
        if (EXP && !ones) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma_bf16_ss(tmem + C::T_DS + 64, desc_plus(kt, ks * 2048 >> 4), desc_plus(xt, ks * 2048 >> 4), ID_DT, true);
        }
        umma_commit(&bars[C::DS_FULL]);
        umma_commit(&bars[C::K_EMPTY + (c & 1)]);
        if (STATES) {
          umma_commit(&bars[C::V_EMPTY + (c & 1)]);
          continue;
        }
        if (!wait(C::Q_FULL + C::q_stage(c), C::q_parity(c), 33) || (c > 0 && !wait(C::Y_FREE, (c - 1) & 1, 34))) break;
        tc_fence_after();
        const uint64_t q = umma_desc_sw128(base + C::Q + C::q_stage(c) * C::Q_TILE, 16, 1024);
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
          for (int ks = 0; ks < 4 * KB; ++ks)
            umma_bf16_ss(tmem + C::T_YI, desc_plus(q, (ks / 4 * C::TILE + ks % 4 * 32) >> 4), desc_plus(sd, (part * C::S_PART + ks * 2048) >> 4), ID_Y,
                         part > 0 || ks > 0);
        if (EXP) umma_commit(&bars[C::Q_EMPTY]);
        umma_commit(&bars[C::INTER]);
      }
    }
    __syncwarp();
  } else if (warp == 18) {
    // ============================ gates ==============================================================
    // lane: tokens 4 lane .. 4 lane + 3
    const float a_log2e = EXP ? 0.f : p.a_log2e[h], a_bias = p.a_bias[h], i_bias = EXP ? p.i_bias[h] : 0.f;
    float m = EXP ? p.m0[s * p.heads + h] * kToLog2 : 0.f, kept = 0.f;
    float raw[4], raw_i[4];
    auto request = [&](int c) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = c * L + lane * 4 + j;
        raw[j] = t < n_tok ? __bfloat162float(p.a[(begin + t) * p.a_stride + h]) : 0.f;
        if (EXP) raw_i[j] = t < n_tok ? __bfloat162float(p.i[(begin + t) * p.i_stride + h]) : 0.f;
      }
    };
    request(0);
    for (int c = 0; c < n_chunks; ++c) {
      float F[4], D[4], E[4], R[4], cs[4], run = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {               // a token past the end changes nothing
        const bool in = c * L + lane * 4 + j < n_tok;
        if constexpr (EXP) {
          run += in ? -softplus_f(-(p.cap * tanhf((raw[j] + a_bias) / p.cap))) * kToLog2 : 0.f;
          D[j] = in ? p.cap * tanhf((raw_i[j] + i_bias) / p.cap) * kToLog2 : -INFINITY;      // (log input gate)
        } else {
          D[j] = in ? softplus_fast(raw[j] + a_bias) : 0.f;
          run += a_log2e * D[j];
        }
        F[j] = run;
      }
      if (c + 1 < n_chunks) request(c + 1);
      // F - B: sums inside half a block (four lanes), from the middle on or up to it
      float before = run;
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, before, off, 4);
        if ((lane & 3) >= off) before += up;
      }
      const float first = __shfl_sync(0xffffffffu, before, (lane & 24) | 3);
      const float ref = fabsf(first) < INFINITY ? first : 0.f;      // (a gate that is not finite must not reach the tokens in front of it)
      before = __shfl_up_sync(0xffffffffu, before, 1);
      before = ((lane & 3) == 0 ? 0.f : before) + (lane & 4 ? first - ref : -ref);
#pragma unroll
      for (int j = 0; j < 4; ++j) F[j] += before;
      const float f_end = __shfl_sync(0xffffffffu, F[3], lane | 7), f_last = __shfl_up_sync(0xffffffffu, f_end, 8);      // of the block, of the last
      float step = lane < 8 ? ref + m : ref + f_last;               // from the last block's B to the own one
      if constexpr (EXP) {
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) { E[j] = D[j] - F[j]; top = fmaxf(top, E[j]); R[j] = top; }
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
          const float up = __shfl_up_sync(0xffffffffu, top, off, 8);
          if ((lane & 7) >= off) top = fmaxf(top, up);
        }
        // the maximum in front of the block, by way of the blocks before it
        float ahead = __shfl_sync(0xffffffffu, step, 0);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const float next = fmaxf(ahead, __shfl_sync(0xffffffffu, top, b * 8 + 7)) + __shfl_sync(0xffffffffu, step, b * 8 + 8);
          if (lane >= b * 8 + 8) ahead = next;
        }
        const float up = __shfl_up_sync(0xffffffffu, top, 1);
        if ((lane & 7) != 0) ahead = fmaxf(ahead, up);
#pragma unroll
        for (int j = 0; j < 4; ++j) R[j] = -fmaxf(R[j], ahead);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) { E[j] = -F[j]; R[j] = F[j]; }
      }
      const float r_block = __shfl_sync(0xffffffffu, R[3], lane | 7);
#pragma unroll
      for (int j = 0; j < 4; ++j) cs[j] = fast_exp2(E[j] + r_block) * (EXP ? 1.f : D[j]);
      const bool ok = c < 2 || (wait(C::V_EMPTY + (c & 1), ((c >> 1) - 1) & 1, 35) && wait(C::TAB_EMPTY + (c & 1), ((c >> 1) - 1) & 1, 36));
      if (!__all_sync(0xffffffffu, ok)) break;
      float* tab = table(c);
      *reinterpret_cast<float4*>(tab + C::E + lane * 4) = make_float4(E[0], E[1], E[2], E[3]);
      *reinterpret_cast<float4*>(tab + C::X3 + lane * 4) = EXP ? make_float4(R[0], R[1], R[2], R[3]) : make_float4(D[0], D[1], D[2], D[3]);
      if (lane < 24) *reinterpret_cast<float4*>(tab + C::CS + lane * 4) = make_float4(cs[0], cs[1], cs[2], cs[3]);
      if ((lane & 7) == 0) tab[C::STEP + (lane >> 3)] = step;
      arrive(C::TAB + (c & 1));
      if constexpr (EXP) {
        if (ones) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int t = c * L + lane * 4 + j;
            if (t < n_tok) p.mt[static_cast<int64_t>(begin + t) * p.heads + h] = (F[j] - R[j]) * kFromLog2;
          }
        }
        m = __shfl_sync(0xffffffffu, F[3] - R[3], 31);
      }
      if constexpr (STATES) {
        float sum = f_end;
#pragma unroll
        for (int b = 0; b < 4; ++b) sum += __shfl_sync(0xffffffffu, step, b * 8);
        kept += __shfl_sync(0xffffffffu, sum, 31);
      }
    }
    if (EXP && ones && lane == 0 && slot >= 0 && !*failed) p.m_state[slot * p.heads + h] = m * kFromLog2;
    if (STATES && blockIdx.x == 0 && lane == 0) p.seg_keep[static_cast<int64_t>(blockIdx.z) * p.heads + h] = fast_exp2(kept);
  } else if (warp < 8) {
    // ============================ M, scaled values ======================================================
    // Loops instead of straight code wherever registers allow it: with everything unrolled the state space's case took 236 us instead of 153.
    const int quad = warp & 3, row = quad * 32 + lane, half = warp >> 2, sw = (row & 7) << 4;
    auto r_of = [&](const float* tab, int t) { return EXP ? tab[C::X3 + t] : -tab[C::E + t]; };
    auto scale_values = [&](int c) {
      const int n = c >> 1 & 1;
      if (!__all_sync(0xffffffffu, wait(C::TAB + (c & 1), n, 50))) return false;
      const float* tab = table(c);
      const bool in = c * L + row < n_tok;
      // 2^{R_end + E} D, for all but the last block as 2^{R_end - R_b} 2^{E + R_b} D
      const float4 step = *reinterpret_cast<const float4*>(tab + C::STEP);
      float w = r_of(tab, L - 1) + (quad == 3 ? tab[C::E + row] : -r_of(tab, quad * 32 + 31));
      w += quad < 1 ? (step.w + step.z) + step.y : quad < 2 ? step.w + step.z : quad < 3 ? step.w : 0.f;
      w = fast_exp2(w) * (quad < 3 ? tab[C::CS + row] : EXP ? 1.f : tab[C::X3 + row]);
      const bool ok = wait(C::V_FULL + (c & 1), n, 51) && wait(C::K_FULL + (c & 1), n, 57) && (c == 0 || wait(C::DS_FULL, (c - 1) & 1, 58));
      if (!__all_sync(0xffffffffu, ok)) return false;
      uint8_t* stage = smem + (c & 1) * C::STAGE;
      if (!in) {                                  // rows behind the last token may hold anything: zeros
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
        for (int j = half * 4; j < half * 4 + 4; ++j) {
          const int at = row * 128 + j * 16;
          if (!ones) *reinterpret_cast<uint4*>(stage + C::V + at) = zero;
#pragma unroll
          for (int kb = 0; kb < KB; ++kb) *reinterpret_cast<uint4*>(stage + C::K + kb * C::TILE + at) = zero;
#pragma unroll
          for (int part = 0; part < C::PARTS; ++part) *reinterpret_cast<uint4*>(smem + C::XS + part * C::TILE + at) = zero;
        }
      } else if (ones) {
#pragma unroll 1
        for (int j = half * 4; j < half * 4 + 4; ++j) {
          uint8_t* at = smem + C::XS + row * 128 + ((j * 16) ^ sw);
          *reinterpret_cast<uint4*>(at) = j == 0 ? three_parts(w) : make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(at + C::TILE) = make_uint4(0u, 0u, 0u, 0u);
        }
      } else {
#pragma unroll 1
        for (int j = half * 4; j < half * 4 + 4; j += 2) {
          uint4 x[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const uint4*>(stage + C::V + row * 128 + (((j + i) * 16) ^ sw));
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint4 hi, lo, third = make_uint4(0u, 0u, 0u, 0u);
            split_value<EXP>(x[i].x, w, hi.x, lo.x, third.x); split_value<EXP>(x[i].y, w, hi.y, lo.y, third.y);
            split_value<EXP>(x[i].z, w, hi.z, lo.z, third.z); split_value<EXP>(x[i].w, w, hi.w, lo.w, third.w);
            uint8_t* at = smem + C::XS + row * 128 + (((j + i) * 16) ^ sw);
            if (EXP) *reinterpret_cast<uint4*>(at + 2 * C::TILE) = third;
            *reinterpret_cast<uint4*>(at) = hi;
            *reinterpret_cast<uint4*>(at + C::TILE) = lo;
          }
        }
      }
      fence_proxy_async();
      arrive(C::XS_READY);
      return true;
    };
    bool going = scale_values(0);
    if constexpr (STATES) {
      for (int c = 1; c < n_chunks && going; ++c) going = scale_values(c);
    } else if (going) {
      const float skip = EXP ? 0.f : p.skip[h];
      for (int c = 0; c < n_chunks; ++c) {
        const float* tab = table(c);              // (waited for with the scaled values)
        const float r = r_of(tab, row);
        float rb = r;                             // the row's R, measured from the middle of the keys' block
        if (!__all_sync(0xffffffffu, wait(C::G_FULL + (c & 1), (c >> 1) & 1, 41))) break;
        tc_fence_after();
        const uint32_t m_at = lanes + C::T_M + (c & 1) * 128;
        float sum = 0.f;                          // of the row's part of M (the normaliser's tile)
        // 16 keys at a time, in place: eight columns of high parts, eight of low ones; zeros behind the last key a row can see
#pragma unroll 1
        for (int b = 6 + half; b >= 0; b -= 2) {
          uint32_t g[16];
          if (b <= 2 * quad + 1) {
            tmem_ld_32x16(m_at + b * 16, g);
            float f = 0.f;
            if ((b >> 1) != quad) {
              rb += tab[C::STEP + (b >> 1) + 1];
              f = fast_exp2(rb - r_of(tab, (b | 1) * 16 + 15)) * (EXP ? p.q_scale : 1.f);
            }
            tmem_wait_ld();
            if ((b >> 1) == quad) {
              const int own = row - b * 16;       // the key on the diagonal
#pragma unroll
              for (int j = 0; j < 16; j += 4) {
                const float4 e = *reinterpret_cast<const float4*>(tab + C::E + b * 16 + j);
                float4 d = make_float4(p.q_scale, p.q_scale, p.q_scale, p.q_scale);
                if constexpr (!EXP) d = *reinterpret_cast<const float4*>(tab + C::X3 + b * 16 + j);
                const float ev[4] = {e.x, e.y, e.z, e.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  float x = j + i <= own ? __uint_as_float(g[j + i]) * fast_exp2(r + ev[i]) * dv[i] : 0.f;
                  if (!EXP && j + i == own) x += skip;
                  g[j + i] = __float_as_uint(x);
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; j += 4) {
                const float4 w = *reinterpret_cast<const float4*>(tab + C::CS + b * 16 + j);
                g[j] = __float_as_uint(__uint_as_float(g[j]) * f * w.x);
                g[j + 1] = __float_as_uint(__uint_as_float(g[j + 1]) * f * w.y);
                g[j + 2] = __float_as_uint(__uint_as_float(g[j + 2]) * f * w.z);
                g[j + 3] = __float_as_uint(__uint_as_float(g[j + 3]) * f * w.w);
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) g[j] = 0u;
          }
          if (ones) {
#pragma unroll
            for (int j = 8; j > 0; j >>= 1)
#pragma unroll
              for (int i = 0; i < j; ++i) g[i] = __float_as_uint(__uint_as_float(g[i]) + __uint_as_float(g[i + j]));
            sum += __uint_as_float(g[0]);
            continue;
          }
          uint32_t m[16];
#pragma unroll
          for (int j = 0; j < 8; ++j) split_pair(__uint_as_float(g[2 * j]), __uint_as_float(g[2 * j + 1]), m[j], m[8 + j]);
          tmem_st_32x16(m_at + b * 16, m);
        }
        tmem_wait_st();
        if (ones) reinterpret_cast<float*>(smem + (c & 1) * C::STAGE + C::V)[half * L + row] = sum;      // (where its values would be)
        tc_fence_before();
        arrive(C::M_READY + (c & 1));
        if (c + 1 < n_chunks && !scale_values(c + 1)) break;
      }
    }
  } else {
    // ============================ state, outputs ========================================================
    const int row = (tid - 256) & 127, sw = (row & 7) << 4, half = (warp >> 2) & 1;      // of S: channel `row`; of the chunk: token `row`
    const int64_t states = static_cast<int64_t>(p.n) * p.vp;
    const bool holds = row < 64 * KB;
    const float* from = nullptr;                  // the state in front, and where the one behind goes (nullptr: nowhere)
    float* to = nullptr;
    float* home = slot < 0 ? nullptr : ones ? p.n_state + (slot * p.heads + h) * p.n : p.state + (slot * p.heads + h) * states;
    if (p.seg != 0) {
      float* here = p.seg_state + (static_cast<int64_t>(blockIdx.z) * p.heads + h) * states;
      if (STATES) to = here; else from = here;
      if (!STATES && last) to = home;
    } else {
      if (home != nullptr && p.positions[begin] != 0) from = home;
      to = home;
    }
    // 16 columns of a row of S as operand
    auto store_operand = [&](int k, const float (&x)[16]) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint4 hi, lo;
        split_pair(x[8 * j], x[8 * j + 1], hi.x, lo.x); split_pair(x[8 * j + 2], x[8 * j + 3], hi.y, lo.y);
        split_pair(x[8 * j + 4], x[8 * j + 5], hi.z, lo.z); split_pair(x[8 * j + 6], x[8 * j + 7], hi.w, lo.w);
        if (ones && k == 0 && j == 0) hi = three_parts(x[0]), lo = make_uint4(0u, 0u, 0u, 0u);
        uint8_t* at = smem + C::ST + row * 128 + (((k * 2 + j) * 16) ^ sw);
        *reinterpret_cast<uint4*>(at) = hi;
        *reinterpret_cast<uint4*>(at + C::S_PART) = lo;
      }
    };
    float S[2][16];                               // columns 32 half .. + 31 of the row
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = half * 2 + i;
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!STATES && from != nullptr && holds) {
          if (!ones) w = *reinterpret_cast<const float4*>(from + static_cast<int64_t>(row) * p.vp + col0 + k * 16 + j);
          else if (k == 0 && j == 0) w.x = from[row];
        }
        S[i][j] = w.x; S[i][j + 1] = w.y; S[i][j + 2] = w.z; S[i][j + 3] = w.w;
      }
      if (!STATES && holds) store_operand(k, S[i]);
    }
    fence_proxy_async();
    arrive(C::S_READY);
    bool ok = true;
    for (int c = 0; c < n_chunks && ok; ++c) {
      const bool more = c + 1 < n_chunks;
      ok = __all_sync(0xffffffffu, wait(C::TAB + (c & 1), (c >> 1) & 1, 54));
      if (!ok) break;
      const float* tab = table(c);
      const float4 step = *reinterpret_cast<const float4*>(tab + C::STEP);      // m + B of the row's block, and of the last
      const int q = warp & 3;
      const float own = step.x + (q > 0 ? step.y : 0.f) + (q > 1 ? step.z : 0.f) + (q > 2 ? step.w : 0.f), base = step.x + step.y + step.z + step.w;
      const float keep = fast_exp2(base + (EXP ? tab[C::X3 + L - 1] : -tab[C::E + L - 1]));
      const float r = own + (EXP ? tab[C::X3 + row] : -tab[C::E + row]);
      ok = wait(C::DS_FULL, c & 1, 52);
      if (!STATES) ok = ok && wait(C::INTER, c & 1, 53);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = half * 2 + i;
        uint32_t hi[16], lo[16];
        tmem_ld_32x16(lanes + C::T_DS + k * 16, hi);
        tmem_ld_32x16(lanes + C::T_DS + 64 + k * 16, lo);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float add = __uint_as_float(hi[j]) + __uint_as_float(lo[j]);
          if (ones) add = j == 0 ? __uint_as_float(hi[0]) + (__uint_as_float(hi[1]) + __uint_as_float(hi[2])) : 0.f;
          S[i][j] = fmaf(S[i][j], keep, add);
        }
        if (!STATES && more && holds) store_operand(k, S[i]);
      }
      if (more) {
        fence_proxy_async();
        tc_fence_before();                        // (what the chunk added has been read)
        arrive(C::S_READY);
      }
      arrive(C::TAB_EMPTY + (c & 1));
      if constexpr (!STATES) {
        ok = __all_sync(0xffffffffu, wait(C::Y_FULL, c & 1, 56));
        if (!ok) break;
        tc_fence_after();
        const float f = fast_exp2(r) * (EXP ? p.q_scale : 1.f);
        const bool in = c * L + row < n_tok;
        const int64_t t = begin + c * L + row;
        uint8_t* out_s = smem + C::Q + C::q_stage(c) * C::Q_TILE;
#pragma unroll 1
        for (int k = half * 2; k < half * 2 + 2; ++k) {
          uint32_t yi[16], ya[16];
          tmem_ld_32x16(lanes + C::T_YI + k * 16, yi);
          tmem_ld_32x16(lanes + C::T_YA + k * 16, ya);
          tmem_wait_ld();
          float y[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] = fmaf(__uint_as_float(yi[j]), f, __uint_as_float(ya[j]));
          if constexpr (EXP) {
            if (ones) {
              const float n0 = __uint_as_float(yi[0]) + (__uint_as_float(yi[1]) + __uint_as_float(yi[2]));
              const float* sums = reinterpret_cast<const float*>(smem + (c & 1) * C::STAGE + C::V);
              if (k == 0 && in) p.nq[t * p.heads + h] = fmaf(n0, f, sums[row] + sums[L + row]);
            } else if (in) {
              float4* o = reinterpret_cast<float4*>(p.o + (t * p.heads + h) * p.vdim + col0 + k * 16);
#pragma unroll
              for (int j = 0; j < 4; ++j) o[j] = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
            }
          } else {                                // through the chunk's queries, which nobody needs any more
#pragma unroll
            for (int j = 0; j < 2; ++j)
              *reinterpret_cast<uint4*>(out_s + row * 128 + (((k * 2 + j) * 16) ^ sw)) =
                  make_uint4(pack_bf16(y[8 * j], y[8 * j + 1]), pack_bf16(y[8 * j + 2], y[8 * j + 3]), pack_bf16(y[8 * j + 4], y[8 * j + 5]),
                             pack_bf16(y[8 * j + 6], y[8 * j + 7]));
          }
        }
        tc_fence_before();
        arrive(C::Y_FREE);
        if constexpr (!EXP) {
          const int unit = half * 4 + (lane & 3), first = (warp & 3) * 32 + (lane >> 2);
          __nv_bfloat16* yg = p.y + static_cast<int64_t>(h) * p.vdim + col0 + unit * 8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {           // a warp's own part of 32 rows, four lanes a row
            const int tl = first + i * 8;
            if (c * L + tl < n_tok)
              *reinterpret_cast<uint4*>(yg + (begin + c * L + tl) * p.y_stride) =
                  *reinterpret_cast<const uint4*>(out_s + tl * 128 + ((unit ^ (tl & 7)) << 4));
          }
          fence_proxy_async();
        }
        if (!EXP) arrive(C::Q_EMPTY + (c & 1));
      }
    }
    ok = __all_sync(0xffffffffu, ok && *failed == 0);
    if (to != nullptr && ok && holds) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = half * 2 + i;
        if (ones) {
          if (k == 0) to[row] = S[i][0];
        } else {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(to + static_cast<int64_t>(row) * p.vp + col0 + k * 16 + j) = make_float4(S[i][j], S[i][j + 1], S[i][j + 2], S[i][j + 3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 17) tmem_dealloc(tmem, 512);
}

// The maps of q, k and v; rows of the last two dimensions are read in boxes of 64 channels x 128 tokens
static int decay_maps(CUtensorMap (&maps)[3], const void* q, const void* k, const void* v, int64_t stride, int tokens, int groups, int n, int heads,
                      int vdim) {
  int rc = make_kv_tensor_map(&maps[0], q, tokens, groups, n, stride, kDecayChunk);
  if (rc == kOk) rc = make_kv_tensor_map(&maps[1], k, tokens, groups, n, stride, kDecayChunk);
  if (rc == kOk) rc = make_kv_tensor_map(&maps[2], v, tokens, heads, vdim, stride, kDecayChunk);
  return rc;
}
// what the kernel takes: 64 or 128 state channels, whole 64-column tiles, rows that TMA can read
static inline bool decay_chunks_take(int n, int vdim) { return (n == 64 || n == 128) && vdim % 64 == 0; }
static inline bool decay_chunks_read(const void* q, const void* k, const void* v, int64_t stride) {
  return stride > 0 && stride % 8 == 0 && is_aligned(q, 16) && is_aligned(k, 16) && is_aligned(v, 16);
}
// - and prompts that fill its chunks, by the average: the kernels for shorter chunks win with less, and a step that mixes a long prompt with
// single tokens has a short average.  Time of those over time here, tiles (CTAs a sequence) T, on 148 SMs, prompts of one length:
//     tokens          32    64    96   128   192   256   384   512   768
//     state space, 128 states   16 x T 64   0.51  0.68  0.94  1.09  1.03  1.38  1.52  1.61  1.68      32 x T 64   0.43  0.58  0.83  0.99  0.96  1.28  1.43
//     state space,  64 states   16 x T 64   0.39  0.49  0.64  0.79  0.72  0.94  1.03  1.09  1.14       8 x T 32   0.52  0.64  0.82  0.95  0.86  1.07  1.18
//     matrix memory, 128        16 x T 48   0.53  0.73  0.93  1.12  1.06  1.34  1.43  1.48  1.57       4 x T 48   0.66  0.82  0.94  1.12  0.96  1.17  1.27
//     matrix memory,  64         6 x T 32   0.68  0.73  0.84  0.95  0.84  0.96  1.00  1.00  1.02      32 x T  8   0.60  0.71  0.83  0.89  0.84  0.96  1.03
//   every tile with an SM to itself: state space 0.86 / 1.07 / 1.43 at 32 / 64 / 96 tokens; matrix memory 0.83 / 0.91 / 1.00 and 0.93 to 1.39 at 160
// One long prompt beside n - 1 single tokens, average 96: 0.64 to 0.74 (state space, which cuts the long one into segments), 1.5 to 2.0 (matrix
// memory, whose old kernel does not); average 192 and up: faster here, or cut into segments (state_space.cu).
static inline bool decay_chunks_filled(bool exp_gates, int n, int tokens, int num_seqs, int64_t tiles) {
  const bool alone = num_seqs * tiles <= sm_count();
  return tokens >= (alone && !exp_gates ? 64ll : alone || n == 128 ? 200ll : 512ll) * num_seqs;
}

template <int KB, bool EXP, bool STATES>
static int launch_decay_pass(const CUtensorMap (&maps)[3], const DecayChunkParams& p, unsigned z, cudaStream_t st) {
  struct Tag {};
  auto kernel = &decay_chunk_kernel<KB, EXP, STATES>;
  const int rc = opt_in_dynamic_smem<Tag>(reinterpret_cast<const void*>(kernel), DecayCfg<KB, EXP>::SMEM);
  if (rc != kOk) return rc;
  kernel<<<dim3(p.vdim / 64 + (EXP ? 1 : 0), p.heads, z), DecayCfg<KB, EXP>::THREADS, DecayCfg<KB, EXP>::SMEM, st>>>(maps[0], maps[1], maps[2], p);
  return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

}  // namespace mvb
