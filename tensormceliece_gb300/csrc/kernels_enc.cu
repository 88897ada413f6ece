// Encapsulation kernels: fixed-weight sampling (lane per request) and the
// finalize step (ciphertext assembly + session-key hash).
//
// Reference behaviour: gen_e / syndrome / operation_enc of libmceliece
// (mceliece-gpu-params/ref/348864.cuh:3434-3565, 8192128.cuh:5967-6006;
// mc:crypto_kem/348864/vec/encrypt.c:41-132, kem_enc.c:18).
#include <stdlib.h>

#include "host_keys.h"
#include "kernels.h"
#include "device_common.cuh"

namespace gmc {

// ---------------------------------------------------------------- sampling
// Randomness is the per-request seed chain: attempt j draws
// SHAKE256({64} || state, cand_bytes) and the next state is the first 32
// bytes of that draw. Candidates are little-endian 16-bit words masked to m
// bits; for n < 2^m the first t values below n are kept, else all t. A
// repeated position rejects the attempt (only the set of positions matters,
// as in the library's sort-and-compare).
// Forms: sample_pipe_kernel and, for small batches, sample_few_kernel (below, the
// defaults), and this lane-per-request sample_kernel (GMC_SAMPLE_PIPELINE=0).
// Work split: each lane owns one request and runs its Keccak chain; lanes
// take requests from a launch-wide counter whenever their previous request
// is done, so a request that needs many attempts does not hold the warp's
// other lanes idle. Small batches leave lanes idle instead (only the first
// `lanes` of each warp take requests): more warps share the batch, so the
// Keccak latency is hidden across warps and the warp-serial repeat check and
// syndrome gather below run over fewer requests per warp. After every
// attempt the warp checks, one lane's
// candidates at a time, for repeats with a single n-bit bitmap per warp
// (atomicOr returns the previous word); on success that bitmap is the error
// vector e, written out by the whole warp (coalesced) together with e[mt:n]
// shifted to bit 0 (the syndrome GEMM operand). Only the touched bitmap
// words are cleared.
// S row = T e[mt:n]: XOR of the columns of TT (row j = column j of T, row k
// zero) at the request's t positions; positions < mt read the zero row.
// Each half-warp reads whole rows, lane c of a half the 16-byte chunk c, so a
// load instruction covers two rows contiguously (positions 2i and 2i + 1);
// the halves are added by one shuffle and lane c stores words 4c .. 4c + 3.
// The loop is unrolled 32 times: a warp gathers one request's columns at a
// time, so the loads in flight per lane set how many L2 round trips a
// request costs (2 for t = 128; unrolled 8 times it took 8, and 0.45 against
// 0.42-0.43 ms for 65536 requests).
template <int SET, typename PosFn>
__device__ __forceinline__ void sparse_syndrome_row(PosFn pos_of, const uint32_t *__restrict__ TT, int ldtt,
                                                    uint32_t *__restrict__ srow, int lane) {
  using p = P<SET>;
  constexpr int MW4 = (p::mw + 3) / 4;
  static_assert(MW4 <= 16, "a syndrome row fits half a warp of 16-byte chunks");
  const int c = lane & 15;
  uint4 acc = make_uint4(0, 0, 0, 0);
  if (c < MW4) {
#pragma unroll 32
    for (int i = lane >> 4; i < p::t; i += 2) {
      const int pos = pos_of(i);
      const uint4 v =
          reinterpret_cast<const uint4 *>(TT + (size_t)(pos >= p::mt ? pos - p::mt : p::k) * ldtt)[c];
      acc.x ^= v.x;
      acc.y ^= v.y;
      acc.z ^= v.z;
      acc.w ^= v.w;
    }
  }
  acc.x ^= __shfl_xor_sync(0xffffffffu, acc.x, 16);
  acc.y ^= __shfl_xor_sync(0xffffffffu, acc.y, 16);
  acc.z ^= __shfl_xor_sync(0xffffffffu, acc.z, 16);
  acc.w ^= __shfl_xor_sync(0xffffffffu, acc.w, 16);
  if (lane < MW4) {
    const uint32_t q4[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int e2 = 0; e2 < 4; e2++)
      if (4 * lane + e2 < p::mw) srow[4 * lane + e2] = q4[e2];
  }
}

template <int SET>
struct SampleLayout {
  using p = P<SET>;
  static constexpr int bm_words = (p::ew + 1) & ~1;
  static constexpr int cand_u16 = 32 * p::t;  // candidate c of lane l at c*32 + (l ^ 2(c%16))
  static constexpr int warp_bytes = bm_words * 4 + cand_u16 * 2;
};

__device__ __forceinline__ int cand_slot(int c, int l) { return c * 32 + (l ^ ((c & 15) << 1)); }

template <int SET, bool SPARSE>
__global__ void __launch_bounds__(kSampleThreadsMax) sample_kernel(const uint8_t *__restrict__ seeds, const Segs segs,
                                                                uint32_t *__restrict__ E, int lde,
                                                                uint32_t *__restrict__ Ens, int ldx,
                                                                const GemmKeys keys, uint32_t *__restrict__ S,
                                                                int lds, unsigned int *__restrict__ counter,
                                                                int lanes) {
  using p = P<SET>;
  using LY = SampleLayout<SET>;
  constexpr int NCW = (p::t + 31) / 32;
  extern __shared__ __align__(16) uint32_t sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *bm = sm + warp * (LY::warp_bytes / 4);
  uint16_t *cand = reinterpret_cast<uint16_t *>(bm + LY::bm_words);
  chain_trigger();
  for (int w = lane; w < LY::bm_words; w += 32) bm[w] = 0;
  __syncwarp();
  const long long N = seg_rows(segs);
  bool has = false, exhausted = lane >= lanes;  // idle lanes never take a request
  long long op = 0;
  int myseg = 0;
  uint64_t st[4] = {0, 0, 0, 0};
  constexpr int ncand = p::cand_bytes / 2;  // 16-bit candidates per attempt
  constexpr int nlanes = (ncand + 3) / 4;   // output lanes holding them
  constexpr uint32_t mask = p::q - 1;
  constexpr int sh = p::mt % 32, w0 = p::mt / 32;
#pragma unroll 1
  while (true) {
    // lanes without a request take the next ones (rows that are segment gaps are skipped)
    const uint32_t need = __ballot_sync(0xffffffffu, !has && !exhausted);
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned int base = 0;
      if (lane == leader) base = atomicAdd(counter, (unsigned int)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if ((need >> lane) & 1) {
        const long long idx = (long long)base + __popc(need & ((1u << lane) - 1));
        if (idx >= N) {
          exhausted = true;
        } else {
          op = idx;
          has = seg_live(segs, idx, &myseg);
          if (has) {
            const uint8_t *sd = seeds + 32 * idx;
#pragma unroll
            for (int i = 0; i < 4; i++) {
              uint64_t v = 0;
#pragma unroll
              for (int b = 0; b < 8; b++) v |= (uint64_t)sd[8 * i + b] << (8 * b);
              st[i] = v;
            }
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, has)) {
      if (__all_sync(0xffffffffu, exhausted)) break;
      continue;
    }
    // one attempt per lane that holds a request
    int count = 0;
    uint64_t nst[4] = {0, 0, 0, 0};
    if (has) {
      uint64_t s[25];
#pragma unroll
      for (int i = 0; i < 25; i++) s[i] = 0;
      s[0] = 64ull | (st[0] << 8);
      s[1] = (st[0] >> 56) | (st[1] << 8);
      s[2] = (st[1] >> 56) | (st[2] << 8);
      s[3] = (st[2] >> 56) | (st[3] << 8);
      s[4] = (st[3] >> 56) | (0x1Full << 8);
      s[16] = 0x8000000000000000ull;
      keccak_f1600(s);
      nst[0] = s[0];
      nst[1] = s[1];
      nst[2] = s[2];
      nst[3] = s[3];
#pragma unroll 1
      for (int base = 0; base < nlanes && count < p::t; base += 17) {
        if (base) keccak_f1600(s);
#pragma unroll
        for (int i = 0; i < 17; i++) {
          if (base + i < nlanes) {
            const uint64_t l = s[i];
#pragma unroll
            for (int h = 0; h < 4; h++) {
              const uint32_t v = (uint32_t)(l >> (16 * h)) & mask;
              const bool take = (4 * (base + i) + h < ncand) && (count < p::t) && (p::full || v < (uint32_t)p::n);
              if (take) {
                cand[cand_slot(count, lane)] = (uint16_t)v;
                count++;
              }
            }
          }
        }
      }
    }
    __syncwarp();
    // repeats, one lane's candidate set at a time
    uint32_t pend = __ballot_sync(0xffffffffu, has && count == p::t);
    uint32_t okmask = 0;
#pragma unroll 1
    while (pend) {
      const int r = __ffs(pend) - 1;
      pend &= pend - 1;
      uint32_t vv[NCW];
      bool dup = false;
#pragma unroll
      for (int i = 0; i < NCW; i++) {
        const int c = lane + 32 * i;
        vv[i] = 0xFFFFFFFFu;
        if (c < p::t) {
          const uint32_t v = cand[cand_slot(c, r)];
          vv[i] = v;
          const uint32_t bit = 1u << (v & 31);
          dup |= (atomicOr(&bm[v >> 5], bit) & bit) != 0;
        }
      }
      const bool anydup = __any_sync(0xffffffffu, dup);
      const long long opr = __shfl_sync(0xffffffffu, op, r);
      if (!anydup) {
        okmask |= 1u << r;
        uint32_t *erow = E + opr * lde;
        for (int w = lane; w < p::ew; w += 32) erow[w] = bm[w];
        if (SPARSE) {
          sparse_syndrome_row<SET>([&](int c) { return (int)cand[cand_slot(c, r)]; },
                                   keys.TT[__shfl_sync(0xffffffffu, myseg, r)], keys.ldtt, S + opr * lds, lane);
        } else {
          uint32_t *xrow = Ens + opr * ldx;
          for (int w = lane; w < p::kw; w += 32) {
            const uint32_t lo = bm[w0 + w];
            const uint32_t hi = (w0 + w + 1 < p::ew) ? bm[w0 + w + 1] : 0u;
            xrow[w] = sh ? ((lo >> sh) | (hi << (32 - sh))) : lo;
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < NCW; i++)
        if (vv[i] != 0xFFFFFFFFu) bm[vv[i] >> 5] = 0;
      __syncwarp();
    }
    if (has) {
      if ((okmask >> lane) & 1) {
        has = false;
      } else {
        st[0] = nst[0];
        st[1] = nst[1];
        st[2] = nst[2];
        st[3] = nst[3];
      }
    }
  }
}

// ---------------------------------------------------------------- pipelined sampling
// A Keccak state is held by two lanes (keccak_f1600_pair), a warp holds 16, and
// all permute in lockstep: a step is one permutation. The warp then checks
// every attempt whose last block landed (candidate filter, first t kept,
// repeats) and finishes the successful ones, one at a time. An attempt needs P
// blocks (P = 2 for 348864 and 8192128, 3 for 460896, 4 for 6688128 and
// 6960119). Two ways to fill the 16 pairs:
//  - pair per request, while the launch has more requests than pairs: a pair
//    runs its request's blocks in turn, P steps an attempt, and takes the next
//    request from the launch-wide counter after a success. No permutation is
//    wasted;
//  - group of P pairs per request, for the few requests left to a warp once the
//    counter has run out, and for batches that do not fill the pairs: the seed
//    chain's next state is the first 32 bytes of an attempt's first block, so
//    pair 0 of the group starts the next attempt (absorb 64 || state, permute) at
//    every step while pair r permutes the state that pair r - 1 left in shared
//    memory a step earlier (block r of an older attempt). An attempt completes
//    every step, P times as fast for the chain, at P - 1 speculative attempts
//    per request; the slowest of 65536 requests needs about 24 attempts.
// 65536 requests, sampler with the sparse syndrome, against one lane per state in
// speculative groups of 2 or 4 lanes throughout: 348864 212 / 273 us, 460896
// 416 / 586, 6688128 677 / 817, 6960119 559 / 698, 8192128 377 / 428; 3001
// requests: 72 / 104, 105 / 184, 175 / 243, 128 / 173, 124 / 173 us.
// Bound: the Keccak instructions and the per-attempt checks while the counter
// lasts, then the longest chains (a step of one warp is about 7100 cycles of
// Keccak and 3500 around it).
template <int SET>
struct PipeLayout {
  using p = P<SET>;
  static constexpr int perms = (p::cand_bytes + 135) / 136;  // Keccak-f blocks per attempt
  static constexpr int NP = 16;                              // pairs per warp
  static constexpr int NG = NP / perms;                      // groups per warp
  static constexpr int raw_words = (p::cand_bytes + 7) / 8;  // u64 words of one attempt's draw
  static constexpr int slot_words = raw_words | 1;           // odd u64 stride: slots on distinct banks
  static constexpr int bm_words = (p::ew + 1) & ~1;
  static constexpr int cand_off = bm_words * 4;
  static constexpr int state_off = cand_off + (p::t * 2 + 7) / 8 * 8;  // [25][32] u32 block states
  static constexpr int ring_off = state_off + 25 * 32 * 4;
  static constexpr int warp_bytes = ring_off + NP * slot_words * 8;
  static_assert(raw_words <= 17 * perms && raw_words > 17 * (perms - 1) && raw_words > 4, "pipeline geometry");
};

// A complete attempt's candidates in raw (a warp, uniform arguments): filter, first t kept, repeats; a success writes e
// (and e[mt:n] or the syndrome). bm is all zero before and after.
template <int SET, bool SPARSE>
__device__ __forceinline__ bool check_attempt(const uint16_t *raw, uint32_t *bm, uint16_t *cand, int lane,
                                              uint32_t *__restrict__ E, int lde, uint32_t *__restrict__ Ens, int ldx,
                                              const GemmKeys &keys, uint32_t *__restrict__ S, int lds, long long opr,
                                              int seg) {
  using p = P<SET>;
  constexpr int NCW = (p::t + 31) / 32, ncand = p::cand_bytes / 2;
  constexpr uint32_t mask = p::q - 1;
  constexpr int sh = p::mt % 32, w0 = p::mt / 32;
  if constexpr (!p::full) {
    int total = 0;
#pragma unroll
    for (int base = 0; base < ncand; base += 32) {
      const int i = base + lane;
      uint32_t v = 0;
      bool keep = false;
      if (i < ncand) {
        v = raw[i] & mask;
        keep = v < (uint32_t)p::n;
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, keep);
      const int idx = total + __popc(bal & ((1u << lane) - 1));
      if (keep && idx < p::t) cand[idx] = (uint16_t)v;
      total += __popc(bal);
    }
    __syncwarp();
    if (total < p::t) return false;  // too few candidates below n (warp-uniform)
  }
  auto pos_of = [&](int c) -> int { return p::full ? (int)(raw[c] & mask) : (int)cand[c]; };
  uint32_t vv[NCW];
  bool dup = false;
#pragma unroll
  for (int i = 0; i < NCW; i++) {
    const int c = lane + 32 * i;
    vv[i] = 0xFFFFFFFFu;
    if (c < p::t) {
      const uint32_t v = (uint32_t)pos_of(c);
      vv[i] = v;
      const uint32_t bit = 1u << (v & 31);
      dup |= (atomicOr(&bm[v >> 5], bit) & bit) != 0;
    }
  }
  const bool good = !__any_sync(0xffffffffu, dup);
  if (good) {
    uint32_t *erow = E + opr * lde;
    for (int w = lane; w < p::ew; w += 32) erow[w] = bm[w];
    if (SPARSE) {
      sparse_syndrome_row<SET>(pos_of, keys.TT[seg], keys.ldtt, S + opr * lds, lane);
    } else {
      uint32_t *xrow = Ens + opr * ldx;
      for (int w = lane; w < p::kw; w += 32) {
        const uint32_t lo = bm[w0 + w];
        const uint32_t hi = (w0 + w + 1 < p::ew) ? bm[w0 + w + 1] : 0u;
        xrow[w] = sh ? ((lo >> sh) | (hi << (32 - sh))) : lo;
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < NCW; i++)
    if (vv[i] != 0xFFFFFFFFu) bm[vv[i] >> 5] = 0;
  __syncwarp();
  return good;
}

// A block per request, for batches that leave most of the GPU idle: a warp per
// block of an attempt, each on a whole Keccak state (KeccakWarp), and one that
// checks. At step s warp r permutes block r of attempt s - r, warp 0 the seed chain
// and each other warp the state that warp r - 1 left a step earlier; the last warp
// checks attempt s - P, complete since the step before. A step is one permutation
// of 24 x 207 cycles and a barrier, against about 9000 cycles in the kernels above,
// at six times their instructions. 256 requests: 348864 34 us against 43, 6960119
// 83 / 112, 8192128 74 / 108; the line to those forms: sample_few_per_sm.
template <int SET, bool SPARSE>
__global__ void __launch_bounds__((PipeLayout<SET>::perms + 1) * 32)
    sample_few_kernel(const uint8_t *__restrict__ seeds, const Segs segs, uint32_t *__restrict__ E, int lde,
                      uint32_t *__restrict__ Ens, int ldx, const GemmKeys keys, uint32_t *__restrict__ S, int lds) {
  using p = P<SET>;
  using LY = PipeLayout<SET>;
  constexpr int PP = LY::perms, RW = LY::raw_words, SLOTS = PP + 1;
  __shared__ __align__(16) uint64_t raw[SLOTS][LY::slot_words], state[PP][2][25];
  __shared__ uint32_t bm[LY::bm_words];
  __shared__ uint16_t cand[p::t];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  chain_trigger();
  const long long op = blockIdx.x;
  int seg;
  if (!seg_live(segs, op, &seg)) return;
  for (int w = threadIdx.x; w < LY::bm_words; w += SLOTS * 32) bm[w] = 0;
  uint64_t st = 0;  // warp 0: word `lane` of the current attempt's state (lanes 0 .. 3)
  if (warp == 0 && lane < 4) {
    const uint8_t *sd = seeds + 32 * op + 8 * lane;
#pragma unroll
    for (int b = 0; b < 8; b++) st |= (uint64_t)sd[b] << (8 * b);
  }
  const KeccakWarp kw(lane);
  __syncthreads();
#pragma unroll 1
  for (int s = 0;; s++) {
    const int j = s - warp;  // the attempt this warp works on
    int good = 0;
    if (j >= 0) {
      if (warp < PP) {
        uint64_t a;
        if (warp == 0) {  // absorb {64} || state
          const uint64_t below = __shfl_up_sync(0xffffffffu, st, 1);
          a = lane < 4 ? st << 8 : lane == 4 ? 0x1F00ull : lane == 16 ? 0x8000000000000000ull : 0ull;
          if (lane <= 4) a |= lane ? below >> 56 : 64ull;
        } else {
          a = state[warp - 1][(s - 1) & 1][lane < 25 ? lane : 0];
        }
        kw.permute(a);
        if (warp == 0) st = a;
        const int w = 17 * warp + lane;
        if (lane < 17 && w < RW) raw[j % SLOTS][w] = a;
        if (warp + 1 < PP && lane < 25) state[warp][s & 1][lane] = a;
      } else {
        good = check_attempt<SET, SPARSE>(reinterpret_cast<const uint16_t *>(raw[j % SLOTS]), bm, cand, lane, E, lde,
                                          Ens, ldx, keys, S, lds, op, seg);
      }
    }
    // every warp leaves after the same step: a flag in shared memory could be set by the checking warp's next step
    // before a late warp has read it
    if (__syncthreads_or(good)) break;
  }
}

// groups = 0: pair per request first, then the warp's last requests as groups; else only groups, at most `groups`
// per warp
template <int SET, bool SPARSE>
__global__ void __launch_bounds__(kSampleThreadsMax)
    sample_pipe_kernel(const uint8_t *__restrict__ seeds, const Segs segs, uint32_t *__restrict__ E, int lde,
                       uint32_t *__restrict__ Ens, int ldx, const GemmKeys keys, uint32_t *__restrict__ S, int lds,
                       unsigned int *__restrict__ counter, int groups) {
  using p = P<SET>;
  using LY = PipeLayout<SET>;
  constexpr int PP = LY::perms, NG = LY::NG, RW = LY::raw_words;
  extern __shared__ __align__(16) uint32_t sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = lane & 1, pair = lane >> 1;
  uint8_t *wb = reinterpret_cast<uint8_t *>(sm) + (size_t)warp * LY::warp_bytes;
  uint32_t *bm = reinterpret_cast<uint32_t *>(wb);
  uint16_t *cand = reinterpret_cast<uint16_t *>(wb + LY::cand_off);
  uint32_t *sts = reinterpret_cast<uint32_t *>(wb + LY::state_off);
  uint32_t *ring = reinterpret_cast<uint32_t *>(wb + LY::ring_off);
  chain_trigger();
  for (int w = lane; w < LY::bm_words; w += 32) bm[w] = 0;
  __syncwarp();
  const long long N = seg_rows(segs);
  const bool seed_words = (reinterpret_cast<uintptr_t>(seeds) & 3) == 0;
  // the request of this pair (its group's, in lanes of pair 0): words 2i + half of the current attempt's state
  bool has = false;
  long long op = 0;
  int myseg = 0;
  uint32_t st[4] = {0, 0, 0, 0};

  // pairs that want a request take the next ones (segment gaps are skipped); false when the counter has run out
  auto fetch = [&](bool want) -> bool {
    const uint32_t need = __ballot_sync(0xffffffffu, want && half == 0);
    bool more = true;
    if (need) {
      const int leader = __ffs(need) - 1;
      unsigned int base = 0;
      if (lane == leader) base = atomicAdd(counter, (unsigned int)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (want) {
        const long long idx = (long long)base + __popc(need & ((1u << (lane & ~1)) - 1));
        if (idx >= N) {
          more = false;
        } else {
          op = idx;
          has = seg_live(segs, idx, &myseg);
          if (has) {
            const uint8_t *sd = seeds + 32 * idx + 4 * half;
#pragma unroll
            for (int i = 0; i < 4; i++) {
              uint32_t v = 0;
              if (seed_words) {
                v = *reinterpret_cast<const uint32_t *>(sd + 8 * i);
              } else {
#pragma unroll
                for (int b = 0; b < 4; b++) v |= (uint32_t)sd[8 * i + b] << (8 * b);
              }
              st[i] = v;
            }
          }
        }
      }
    }
    return more;
  };
  // SHAKE256 absorb of {64} || state
  auto absorb = [&](uint32_t (&A)[25]) {
    uint32_t prev = 64u << 24;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, st[i], 1);
      A[i] = __funnelshift_l(half ? o : prev, st[i], 8);
      prev = o;
    }
    A[4] = half ? 0u : __funnelshift_l(prev, 0x1Fu, 8);
#pragma unroll
    for (int i = 5; i < 25; i++) A[i] = 0;
    if (half) A[16] = 0x80000000u;
  };
  // block r's output words go to an attempt's slot
  auto squeeze = [&](const uint32_t (&A)[25], int slot, int r) {
    uint32_t *dst = ring + (size_t)slot * LY::slot_words * 2 + half;
#pragma unroll
    for (int i = 0; i < 17; i++) {
      const int w = 17 * r + i;
      if (w < RW) dst[2 * w] = A[i];
    }
  };
  auto check = [&](int slot, long long opr, int seg) -> bool {
    return check_attempt<SET, SPARSE>(reinterpret_cast<const uint16_t *>(ring + (size_t)slot * LY::slot_words * 2), bm,
                                      cand, lane, E, lde, Ens, ldx, keys, S, lds, opr, seg);
  };

  bool exhausted = false;
  if (groups == 0) {
    // pair per request
    int blk = 0;  // the block of the current attempt this step permutes
    uint32_t nst[4] = {0, 0, 0, 0};
#pragma unroll 1
    while (true) {
      if (!fetch(!has && !exhausted)) exhausted = true;
      const uint32_t live = __ballot_sync(0xffffffffu, has && half == 0);
      if (__all_sync(0xffffffffu, exhausted || has) && __any_sync(0xffffffffu, exhausted) && __popc(live) <= NG) break;
      if (!live) continue;
      uint32_t A[25];
      absorb(A);
      if (blk) {
#pragma unroll
        for (int i = 0; i < 25; i++) A[i] = sts[i * 32 + lane];
      }
      keccak_f1600_pair(A, half);
      squeeze(A, pair, blk);
      if (blk == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) nst[i] = A[i];
      }
      blk++;
      if (blk < PP) {
#pragma unroll
        for (int i = 0; i < 25; i++) sts[i * 32 + lane] = A[i];
      }
      __syncwarp();
      uint32_t pend = __ballot_sync(0xffffffffu, has && blk == PP && half == 0);
      uint32_t succ = 0;  // bit per pair's even lane
#pragma unroll 1
      while (pend) {
        const int o = __ffs(pend) - 1;
        pend &= pend - 1;
        if (check(o >> 1, __shfl_sync(0xffffffffu, op, o), __shfl_sync(0xffffffffu, myseg, o))) succ |= 1u << o;
      }
      if (blk == PP || !has) {  // (an idle pair's next request starts at block 0)
        blk = 0;
        if ((succ >> (lane & ~1)) & 1) has = false;
#pragma unroll
        for (int i = 0; i < 4; i++) st[i] = nst[i];
      }
    }
    // the warp's last requests as groups, each from the start of its current attempt
    {
      const uint32_t live = __ballot_sync(0xffffffffu, has && half == 0);
      const int g = pair / PP, cnt = __popc(live);
      int src = lane;
      uint32_t l = live;
      for (int i = 0; i < cnt; i++) {  // g-th live pair
        if (i == g) src = (__ffs(l) - 1) | half;
        l &= l - 1;
      }
      op = __shfl_sync(0xffffffffu, op, src);
      myseg = __shfl_sync(0xffffffffu, myseg, src);
#pragma unroll
      for (int i = 0; i < 4; i++) st[i] = __shfl_sync(0xffffffffu, st[i], src);
      has = pair == g * PP && g < cnt;
      exhausted = true;
    }
    __syncwarp();
  }

  // group of PP pairs per request
  const int g = pair / PP, r = pair - g * PP;
  const bool chain = r == 0 && g < (groups ? groups : NG) && g < NG;  // the pair that owns the request and its chain
  if (!chain) {
    has = false;
    exhausted = true;
  }
  int attempt = 0, att = 0;
  bool valid = false;  // this pair holds block r of attempt att of the group's request
#pragma unroll 1
  while (true) {
    const bool idle = !has;
    if (!fetch(!has && !exhausted)) exhausted = true;
    if (idle && has) attempt = 0;
    if (!__any_sync(0xffffffffu, has || valid)) {
      if (__all_sync(0xffffffffu, exhausted)) break;
      continue;
    }
    // pair 0 of a group starts its request's next attempt; pair r > 0 continues the state pair r - 1 left a step
    // earlier
    uint32_t A[25];
    absorb(A);
    if (r == 0) {
      valid = has;
      att = attempt;
    } else {
#pragma unroll
      for (int i = 0; i < 25; i++) A[i] = sts[i * 32 + lane - 2];
    }
    __syncwarp();  // every predecessor state read before this step's states overwrite them
    keccak_f1600_pair(A, half);
#pragma unroll
    for (int i = 0; i < 25; i++) sts[i * 32 + lane] = A[i];
    if (valid) {
      squeeze(A, g * PP + att % PP, r);
      if (r == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) st[i] = A[i];
        attempt++;
      }
    }
    __syncwarp();
    uint32_t pend = __ballot_sync(0xffffffffu, valid && r == PP - 1 && half == 0);
    uint32_t succ = 0;  // bit per group
#pragma unroll 1
    while (pend) {
      const int o = __ffs(pend) - 1;
      pend &= pend - 1;
      const int gg = (o >> 1) / PP, owner = gg * PP * 2;
      const int a = __shfl_sync(0xffffffffu, att, o);
      if (check(gg * PP + a % PP, __shfl_sync(0xffffffffu, op, owner), __shfl_sync(0xffffffffu, myseg, owner)))
        succ |= 1u << gg;
    }
    // a success ends the request: its younger attempts in flight are dropped
    if ((succ >> g) & 1) {
      valid = false;
      if (r == 0) has = false;
    }
    // block r of an attempt moves one pair along the group (its state is in shared memory)
    const bool vin = __shfl_up_sync(0xffffffffu, valid ? 1 : 0, 2) != 0;
    const int ain = __shfl_up_sync(0xffffffffu, att, 2);
    if (r > 0) {
      valid = vin && g < NG;
      att = ain;
    }
  }
}

// ---------------------------------------------------------------- finalize
// c = e[0:mt] xor (T e[mt:n]); K = SHAKE256(1 || e || c). When the public
// key's padding bits are set (6960119 only), c and K are zeroed
// (mc:crypto_kem/6960119/vec/kem_enc.c:21-66).
// Bound by the integer ALU (10 Keccak-f per request for 8192128). WARP: a warp
// per request, for launches that leave most of the GPU idle (hash_warp_form);
// else two lanes per request, 16 requests per warp: 8192128, 65536 requests
// 206 us against 271 us with one lane per request, where a scheduler held 4 or
// 3 warps of whole permutations (7 or 6 of half ones now) and the ciphertext
// was stored a byte at a time by the lane that hashed it (whole rows by the
// warp now).
// the ciphertext words of one request, C0 || C1 (C1: plaintext confirmation)
template <int SET, bool PC>
struct EncHashSrc {
  using p = P<SET>;
  const uint32_t *er, *sr;  // e and T e[mt:n]
  const uint32_t *c1;       // 8 words of C1 (registers)
  __device__ uint32_t e(int w) const { return er[w]; }
  __device__ uint32_t c0(int w) const {
    if (w >= p::mw) return 0u;
    uint32_t v = er[w] ^ sr[w];
    if (w == p::mt / 32 && (p::mt % 32)) v &= (1u << (p::mt % 32)) - 1u;
    return v;
  }
  __device__ uint32_t c1w(int w) const {
    uint32_t v = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) v = w == i ? c1[i] : v;
    return v;
  }
  __device__ uint32_t c(int w) const {
    constexpr int W0 = p::synd_bytes / 4;
    if (!PC) return c0(w);
    if (w < W0) return c0(w);
    if (p::synd_bytes % 4 == 0) return c1w(w - W0);
    if (w == W0) return c0(w) | (c1[0] << 16);
    return (c1w(w - W0 - 1) >> 16) | (c1w(w - W0) << 16);
  }
};

template <int SET, bool PC, bool WARP>
__global__ void __launch_bounds__(kTailThreads, WARP ? 1 : PC ? kTailBlocksPerSM - 2 : kTailBlocksPerSM)
    finalize_kernel(const uint32_t *__restrict__ E, int lde, const uint32_t *__restrict__ S, int lds,
                    uint8_t *__restrict__ C, uint8_t *__restrict__ K, const Segs segs, uint32_t pk_bad_mask) {
  using p = P<SET>;
  constexpr int SB = p::synd_bytes, CB = SB + (PC ? 32 : 0);  // C0 bytes, ciphertext bytes
  constexpr int RPW = WARP ? 1 : 16;                          // requests per warp
  const int lane = threadIdx.x & 31, half = lane & 1;
  const long long op0 = ((long long)blockIdx.x * (kTailThreads / 32) + (threadIdx.x >> 5)) * RPW;
  const int r = WARP ? 0 : lane >> 1;
  int seg;
  const bool live = seg_live(segs, op0 + r, &seg);
  const uint32_t livemask = __ballot_sync(0xffffffffu, live);
  if (!livemask) return;
  chain_wait();
  const uint32_t badmask = __ballot_sync(0xffffffffu, (pk_bad_mask >> seg) & 1u);
  // lanes of rows that are not live hash the warp's first live row and store nothing
  const long long op = live ? op0 + r : op0 + (WARP ? 0 : (__ffs(livemask) - 1) >> 1);
  uint32_t c1[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const EncHashSrc<SET, PC> src{E + op * lde, S + op * lds, c1};
  uint32_t own[4];
  // plaintext confirmation: C1 = SHAKE256(2 || e, 32) (mc:crypto_kem/348864pc/vec/kem_enc.c:32)
  if constexpr (PC) {
    const EncOnlySrc esrc{src.er};
    if constexpr (WARP) {
      const uint64_t h = kem_hash_warp<p::e_bytes, 1 + p::e_bytes>(2u, esrc, lane);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint64_t v = __shfl_sync(0xffffffffu, h, i);
        c1[2 * i] = (uint32_t)v;
        c1[2 * i + 1] = (uint32_t)(v >> 32);
      }
    } else {
      kem_hash_pair<p::e_bytes, 1 + p::e_bytes>(own, 2u, esrc, half);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, own[i], 1);
        c1[2 * i] = half ? o : own[i];
        c1[2 * i + 1] = half ? own[i] : o;
      }
    }
  }
  if constexpr (WARP) {
    const uint64_t h = kem_hash_warp<p::e_bytes, p::pre_bytes + (PC ? 32 : 0)>(1u, src, lane);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint64_t v = __shfl_sync(0xffffffffu, h, i);
      own[i] = half ? (uint32_t)(v >> 32) : (uint32_t)v;
    }
  } else {
    kem_hash_pair<p::e_bytes, p::pre_bytes + (PC ? 32 : 0)>(own, 1u, src, half);
  }
  const bool bad = (badmask >> lane) & 1u;
  if (live && (!WARP || lane < 2)) {
    if (bad) {
#pragma unroll
      for (int i = 0; i < 4; i++) own[i] = 0;
    }
    store_hash_words(K + op * 32, own, half);
    if constexpr (PC) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; i++) v[i] = bad ? 0u : half ? c1[2 * i + 1] : c1[2 * i];
      store_hash_words(C + op * CB + SB, v, half);
    }
  }
  // C0 of the warp's rows, in the widest units that divide a row at this buffer's alignment
  const uint32_t *Eb = E + op0 * lde, *Sb = S + op0 * lds;
  uint8_t *cb = C + op0 * CB;
  auto c0_of = [&](int row, int w) -> uint32_t {
    uint32_t v = Eb[(long long)row * lde + w] ^ Sb[(long long)row * lds + w];
    if (w == p::mt / 32 && (p::mt % 32)) v &= (1u << (p::mt % 32)) - 1u;
    return ((badmask >> (WARP ? 0 : 2 * row)) & 1u) ? 0u : v;
  };
  auto row_live = [&](int row) { return ((livemask >> (WARP ? 0 : 2 * row)) & 1u) != 0; };
  const uintptr_t align = reinterpret_cast<uintptr_t>(C);
  if (SB % 4 == 0 && CB % 4 == 0 && (align & 3) == 0) {
    constexpr int U = SB / 4;
    for (int x = lane; x < RPW * U; x += 32) {
      const int row = x / U, w = x - row * U;
      if (row_live(row)) *reinterpret_cast<uint32_t *>(cb + row * CB + 4 * w) = c0_of(row, w);
    }
  } else if (SB % 2 == 0 && CB % 2 == 0 && (align & 1) == 0) {
    constexpr int U = SB / 2;
    for (int x = lane; x < RPW * U; x += 32) {
      const int row = x / U, w = x - row * U;
      if (row_live(row))
        *reinterpret_cast<uint16_t *>(cb + row * CB + 2 * w) = (uint16_t)(c0_of(row, w >> 1) >> (16 * (w & 1)));
    }
  } else {
    for (int x = lane; x < RPW * SB; x += 32) {
      const int row = x / SB, w = x - row * SB;
      if (row_live(row)) cb[row * CB + w] = (uint8_t)(c0_of(row, w >> 2) >> (8 * (w & 3)));
    }
  }
}

// ---------------------------------------------------------------- column image of T
// One warp per (32 rows, 32 columns) block: lane b holds row 32w + b's word of
// the block, ballot j gives column 32jw + j's bits of those rows.
__global__ void transpose_pk_kernel(const uint32_t *__restrict__ T, int lda, int mt, int k, uint32_t *__restrict__ TT,
                                    int ldtt) {
  const int lane = threadIdx.x & 31;
  const long long task = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int mw = (mt + 31) / 32, kw = (k + 31) / 32;
  if (task >= (long long)mw * kw) return;  // warp-uniform
  const int w = (int)(task % mw), jw = (int)(task / mw);
  const int row = 32 * w + lane;
  const uint32_t x = row < mt ? T[(size_t)row * lda + jw] : 0u;
  uint32_t mine = 0;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const uint32_t v = __ballot_sync(0xffffffffu, (x >> j) & 1u);
    mine = (lane == j) ? v : mine;
  }
  const int col = 32 * jw + lane;
  if (col < k) TT[(size_t)col * ldtt + w] = mine;
}

cudaError_t launch_transpose_pk(const uint32_t *T, int lda, int mt, int k, uint32_t *TT, int ldtt, cudaStream_t st) {
  const long long warps = (long long)((mt + 31) / 32) * ((k + 31) / 32);
  transpose_pk_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(T, lda, mt, k, TT, ldtt);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- launchers
// A warp per request while every SM scheduler has at most one such warp (see
// KeccakWarp): beyond that its six-fold instruction count outweighs its
// latency. Rows that are not live exit at once and do not count.
constexpr int kHashWarpsPerSM = 4;
bool hash_warp_form(const Segs &segs) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return seg_live_rows(segs) <= (long long)kHashWarpsPerSM * sms;
}

// GMC_SAMPLE_PIPELINE=0 in the environment (read once per process) puts
// every batch on the lane-per-request sampler instead of the pipelined one.
static bool sample_pipelined() {
  static const bool on = [] {
    const char *v = getenv("GMC_SAMPLE_PIPELINE");
    return !(v && v[0] == '0');
  }();
  return on;
}
// whether a batch takes the block-per-request sampler (which has no tuned parameters)
bool sample_few_form(int set, const Segs &segs) {
  const gmc_setinfo &S = set_info(set);
  const bool full = S.n == S.q;
  const int perms = ((full ? 2 : 4) * S.t + 135) / 136;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sample_pipelined() && seg_live_rows(segs) <= (long long)sample_few_per_sm(perms, full) * sms;
}
template <int SET, bool SPARSE>
static cudaError_t launch_sample_mode(const uint8_t *seeds, const Segs &segs, uint32_t *E, int lde, uint32_t *Ens,
                                     int ldx, const GemmKeys &keys, uint32_t *S, int lds, int threads,
                                     unsigned int *counter, cudaStream_t st, int sample_sm_warps,
                                     void (*mark)(const char *, cudaStream_t)) {
  const long long N = seg_rows(segs);
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t err;
  constexpr int PP = PipeLayout<SET>::perms;
  if (sample_few_form(SET, segs)) {
    sample_few_kernel<SET, SPARSE>
        <<<(unsigned)N, (PP + 1) * 32, 0, st>>>(seeds, segs, E, lde, Ens, ldx, keys, S, lds);
    err = cudaGetLastError();
    if (mark) mark(SPARSE ? "enc_sample_syndrome" : "enc_sample", st);
    return err;
  }
  const int smem = (threads / 32) * SampleLayout<SET>::warp_bytes;
  err = cudaFuncSetAttribute(sample_kernel<SET, SPARSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (kSampleThreadsMax / 32) * SampleLayout<SET>::warp_bytes);
  if (err != cudaSuccess) return err;
  if ((err = cudaMemsetAsync(counter, 0, sizeof(unsigned int), st)) != cudaSuccess) return err;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sample_kernel<SET, SPARSE>, threads, smem);
  if (per_sm < 1) per_sm = 1;
  // fewer lanes than requests: a lane that finishes early takes further
  // requests, so the last slow chains hold few warps (kSampleWarpsPerSM)
  const int warps = threads / 32;
  int per_sm_target = (kSampleWarpsPerSM + warps - 1) / warps;
  // pipelined form: 16 resident warps per SM while the batch fills them (8 / 12 / 16 / 20 / 24 warps, 8192128,
  // 65536 requests: 490 / 404 / 377 / 384 / 398 us); as groups only, two warps per scheduler before a warp gets a
  // further group (8192128, 3001 requests, one / two warps: 142 / 124 us)
  if (sample_pipelined()) {
    using PL = PipeLayout<SET>;
    auto kern = sample_pipe_kernel<SET, SPARSE>;
    const int psmem = warps * PL::warp_bytes;
    err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (kSampleThreadsMax / 32) * PL::warp_bytes);
    if (err != cudaSuccess) return err;
    int pper = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pper, kern, threads, psmem);
    if (pper < 1) pper = 1;
    const int want_warps = sample_sm_warps > 0 ? sample_sm_warps : kSamplePipeWarps;
    const int ptarget = (want_warps + warps - 1) / warps < pper ? (want_warps + warps - 1) / warps : pper;
    const long long resident = (long long)sms * ptarget;  // blocks
    // groups per warp where groups hold the whole batch: as many as keep one warp on every scheduler
    int groups = 1;
    while (groups < PL::NG && (long long)groups * 4 * sms * kSampleGroupWarps < N) groups++;
    if ((long long)groups * resident * warps < N) groups = 0;  // pair per request
    const long long per_block = (long long)warps * (groups ? groups : PL::NP);
    const long long need = (N + per_block - 1) / per_block;
    const long long blocks = need < resident ? need : resident;
    kern<<<(unsigned)blocks, threads, psmem, st>>>(seeds, segs, E, lde, Ens, ldx, keys, S, lds, counter, groups);
    err = cudaGetLastError();
    if (mark) mark(SPARSE ? "enc_sample_syndrome" : "enc_sample", st);
    return err;
  }
  if (per_sm_target > per_sm) per_sm_target = per_sm;
  // active lanes per warp: the smallest power of two (<= 32) with which the
  // resident warps hold the whole batch at once
  const long long warp_slots = (long long)sms * per_sm_target * warps;
  int lanes = 1;
  while (lanes < 32 && (long long)lanes * warp_slots < N) lanes <<= 1;
  const long long per_block = (long long)warps * lanes;
  const long long need = (N + per_block - 1) / per_block;
  const long long resident = (long long)sms * per_sm_target;
  const long long blocks = need < resident ? need : resident;
  sample_kernel<SET, SPARSE><<<(unsigned)blocks, threads, smem, st>>>(seeds, segs, E, lde, Ens, ldx, keys, S, lds,
                                                                      counter, lanes);
  err = cudaGetLastError();
  if (mark) mark(SPARSE ? "enc_sample_syndrome" : "enc_sample", st);
  return err;
}

template <int SET>
cudaError_t launch_sample(const uint8_t *seeds, const Segs &segs, uint32_t *E, int lde, uint32_t *Ens, int ldx,
                          const GemmKeys *sparse, uint32_t *S, int lds, int threads, unsigned int *counter,
                          cudaStream_t st, int sm_warps, void (*mark)(const char *, cudaStream_t)) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  if ((threads != 32 && threads != 64 && threads != 128) || !counter || sm_warps < 0) return cudaErrorInvalidValue;
  if (sparse) {
    if (!S || lds < P<SET>::mw || sparse->ldtt < 64) return cudaErrorInvalidValue;
    for (int i = 0; i < segs.nseg; i++)
      if (!sparse->TT[i]) return cudaErrorInvalidValue;
    return launch_sample_mode<SET, true>(seeds, segs, E, lde, Ens, ldx, *sparse, S, lds, threads, counter, st,
                                         sm_warps, mark);
  }
  return launch_sample_mode<SET, false>(seeds, segs, E, lde, Ens, ldx, GemmKeys{}, S, lds, threads, counter, st,
                                        sm_warps, mark);
}

template <int SET>
cudaError_t launch_finalize(const uint32_t *E, int lde, const uint32_t *S, int lds, uint8_t *C, uint8_t *K,
                            const Segs &segs, uint32_t pk_bad_mask, bool pc, cudaStream_t st) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  auto launch = [&](auto kern, int rows_per_block) {
    return launch_chained(segs, kern, (unsigned)((N + rows_per_block - 1) / rows_per_block), kTailThreads, 0, st, E, lde, S,
                          lds, C, K, segs, pk_bad_mask);
  };
  if (hash_warp_form(segs))
    return pc ? launch(finalize_kernel<SET, true, true>, kTailThreads / 32)
              : launch(finalize_kernel<SET, false, true>, kTailThreads / 32);
  return pc ? launch(finalize_kernel<SET, true, false>, kTailThreads / 2)
            : launch(finalize_kernel<SET, false, false>, kTailThreads / 2);
}

#define GMC_INST_ENC(SET)                                                                                        \
  template cudaError_t launch_sample<SET>(const uint8_t *, const Segs &, uint32_t *, int, uint32_t *, int,       \
                                          const GemmKeys *, uint32_t *, int, int, unsigned int *, cudaStream_t,  \
                                          int, void (*)(const char *, cudaStream_t));                            \
  template cudaError_t launch_finalize<SET>(const uint32_t *, int, const uint32_t *, int, uint8_t *, uint8_t *, \
                                            const Segs &, uint32_t, bool, cudaStream_t);
GMC_INST_ENC(0)
GMC_INST_ENC(1)
GMC_INST_ENC(2)
GMC_INST_ENC(3)
GMC_INST_ENC(4)

}  // namespace gmc
