// Decapsulation kernels.
//
//  pack_ct     ciphertext bytes -> 32-bit words (the front-end GEMM operand)
//  decode      2t syndromes (from the front-end GEMM, or straight from the
//              ciphertext bytes in small batches) -> Berlekamp-Massey ->
//              additive FFT over all 2^m field elements -> error positions
//              at the key's support, weight; a warp per request, or 32
//              requests per word, by batch size
//  dec_tail    K = SHAKE256(b || (e or s) || c), implicit rejection, and the
//              6960119 ciphertext-padding rule
//
// Reference behaviour: decrypt / operation_dec of libmceliece
// (mceliece-gpu-params/ref/348864.cuh:3251-3406, 3615-3650;
// mc:crypto_kem/348864/vec/decrypt.c:135, kem_dec.c:19;
// mc:crypto_kem/6960119/vec/kem_dec.c:21-78). Only the outcome is defined
// there: a weight-t error with the received syndrome is unique, so any exact
// decoder yields the same session key. The BM update rule follows the
// library's (mc:crypto_kem/348864/vec/bm.c:156) on its fixed arrays of t + 1
// coefficients, so locators agree with the oracle's stage output as well.
#include <algorithm>
#include <type_traits>

#include "host_keys.h"
#include "kernels.h"
#include "device_common.cuh"

namespace gmc {

// Copies a field table of n 16-bit entries to shared memory by the whole block,
// 16 bytes a thread (both sides 16-byte aligned; n is rounded up to whole
// units). A block of few warps spends most of a small launch here if it copies
// entry by entry: one 8192128 request, Berlekamp-Massey 125 -> 92 us, roots
// 29 -> 25 us.
__device__ __forceinline__ void copy_table(void *dst, const void *src, int n) {
  const int units = (2 * n + 15) / 16;
#pragma unroll 8
  for (int i = threadIdx.x; i < units; i += blockDim.x)
    reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
}

// ---------------------------------------------------------------- pack_ct
template <int SET, bool PC>
__global__ void pack_ct_kernel(const uint8_t *__restrict__ C, const Segs segs, uint32_t *__restrict__ X, int ldx) {
  using p = P<SET>;
  constexpr int CB = p::synd_bytes + (PC ? 32 : 0);  // ciphertext row bytes
  chain_trigger();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long op = idx / ldx;
  const int w = (int)(idx % ldx);
  if (op >= seg_rows(segs)) return;
  int seg;
  uint32_t v = 0;  // rows past a segment's live requests stay zero
  if (seg_live(segs, op, &seg)) {
    const uint8_t *c = C + op * CB;
#pragma unroll
    for (int b = 0; b < 4; b++) {
      int x = 4 * w + b;
      if (x < p::synd_bytes) v |= (uint32_t)c[x] << (8 * b);
    }
  }
  X[op * ldx + w] = v;
}

// ---------------------------------------------------------------- front end of small batches
// The syndromes S2 = F C0 of a few live requests (kFrontFewBytes) straight from
// the ciphertext bytes: a warp holds 32 rows of F (lane = row, the whole row
// in registers) and goes through 16 requests whose words a block shares; a word
// costs one LOP3 (acc ^= a & x) and the 32 parities of a request are one ballot.
// Packing the ciphertexts and the tensor-core product take two launches, and
// the product's tiles of 128 requests a fixed time: 8192128 20.6 us for up to
// 1000 requests, against 6.1 for one request here, 8.1 for 64 and 11 for 256 (348864
// 16.5, against 6.0, 6.4 and 7.5). Bound by the load of the rows and the launch.
template <int SET, bool PC>
__global__ void __launch_bounds__(kFrontFewWarps * 32) dec_front_few_kernel(const uint8_t *__restrict__ C, const Segs segs,
                                                                           const GemmKeys keys, int ldf,
                                                                           uint32_t *__restrict__ S2, int lds2) {
  using p = P<SET>;
  constexpr int CB = p::synd_bytes + (PC ? 32 : 0);  // ciphertext row bytes
  constexpr int U = (p::synd_bytes + 15) / 16;       // 16-byte units of a row
  constexpr int NW = p::s2w, RG = (NW + kFrontFewWarps - 1) / kFrontFewWarps, OPS = 16;
  __shared__ __align__(16) uint32_t xs[OPS][4 * U];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  chain_trigger();
  const long long op0 = (long long)(blockIdx.x / RG) * OPS;  // 16 rows never straddle segments
  const int seg = seg_find(segs, op0);
  const long long nlive = segs.row0[seg] + segs.nreq[seg] - op0;
  if (nlive <= 0) return;
  const int live = nlive < OPS ? (int)nlive : OPS;
  const int w = blockIdx.x % RG * kFrontFewWarps + warp;  // word of the syndromes: rows 32 w .. 32 w + 31
  uint4 a[U];
  if (w < NW) {
    const uint4 *row = reinterpret_cast<const uint4 *>(keys.A[seg] + (size_t)(32 * w + lane) * ldf);
#pragma unroll
    for (int u = 0; u < U; u++) a[u] = row[u];
  }
  // ciphertext rows on 4-byte boundaries (they may lie in host memory: few loads)
  const bool words = p::synd_bytes % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 3) == 0;
  for (int i = threadIdx.x; i < live * 4 * U; i += kFrontFewWarps * 32) {
    const int r = i / (4 * U), x = i % (4 * U);
    const uint8_t *c = C + (op0 + r) * CB;
    uint32_t v = 0;
    if (words) {
      if (4 * x < p::synd_bytes) v = reinterpret_cast<const uint32_t *>(c)[x];
    } else {
#pragma unroll
      for (int b = 0; b < 4; b++)
        if (4 * x + b < p::synd_bytes) v |= (uint32_t)c[4 * x + b] << (8 * b);
    }
    xs[r][x] = v;
  }
  __syncthreads();
  if (w >= NW) return;
  uint32_t mine = 0;
#pragma unroll 2
  for (int r = 0; r < live; r++) {
    uint32_t acc[4] = {0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint4 x = reinterpret_cast<const uint4 *>(xs[r])[u];
      acc[0] ^= a[u].x & x.x;
      acc[1] ^= a[u].y & x.y;
      acc[2] ^= a[u].z & x.z;
      acc[3] ^= a[u].w & x.w;
    }
    const uint32_t par = __ballot_sync(0xffffffffu, __popc(acc[0] ^ acc[1] ^ acc[2] ^ acc[3]) & 1);
    if (lane == r) mine = par;
  }
  if (lane < live) S2[(op0 + lane) * lds2 + w] = mine;
}

// ---------------------------------------------------------------- BM
// One warp per group of 32 requests, bit-sliced: bit q of every word belongs
// to request 32g + q, and a GF(2^m) value of all 32 requests is m words
// (planes). Coefficient i >= 1 of C (connection polynomial, C_0 = 1) lives in
// lane (i-1)%32, slot (i-1)/32, as m plane registers; B and the syndromes sit in
// per-warp shared memory as planes. Per iteration n:
//   d = s_n + sum_i C_i s_{n-i}: carry-less plane products accumulated
//       unreduced, one reduction, then one XOR reduction instruction per plane;
//   f = d/b per request: lane q extracts its request's d, divides with the
//       log tables (L and log b are per-request scalars in lane q) and the
//       32 quotients are sliced back by ballot;
//   C_i += f B_i (bit-sliced product onto C_i, one reduction), and
//       B <- x (upd ? C_old : B) with the per-request update mask from a ballot.
// This is the library's update rule (mc:crypto_kem/348864/vec/bm.c:156) on
// fixed arrays of t+1 coefficients, per request; the slot loops stop at the
// largest degree bound of the group: before iteration n, deg C <= L and
// deg B <= n+1-L, so the discrepancy needs i <= min(L, t) and the update
// i <= min(max(L, n+1-L), t). Rows that are not live run with zero
// syndromes (d = 0) and write nothing.
// Both arrays are rings that turn with n: s_{n-i} and B_i have fixed entries for
// the iterations that use them. Multiplying B by x moves nothing, so iterations
// in which no request of the group takes the new B (every second one as long as
// no discrepancy is 0) write nothing; entry i of B is read and replaced by the
// lane that holds C_i, without barriers. The syndrome ring is filled 32 planes at
// a time by a transpose of one word of every request's packed syndromes.
// Shared memory per warp is what fourteen warps per SM can hold (one round
// for 2048 groups on 152 SMs): iteration n reads s_{n-t} .. s_n only, and a fill
// reaches at most three syndromes ahead; B keeps coefficients 0..t; the exponent
// table keeps the q-1 entries the division indexes. Lanes above deg C in an
// active discrepancy slot read ring entries of other iterations: C_i = 0 there
// (coefficients above t are never updated), so they add nothing.
// A warp's instructions all go through one of the SM's four schedulers, so 13 or
// 14 groups in a block take the time of 16. One or two groups more than a multiple
// of four therefore change warps, to the two schedulers with fewer, after 11/16 of
// their iterations (half of their work, and a little more because the second half
// ends alone); C and the scalars pass through the group's rows of Sig. Not with
// fewer than eight groups below them, where the second half alone is longer than
// what the schedulers gain.
// 8192128: 65536 requests 1072 us, 40000 822, 32768 680; without split groups
// 1201 (91% of the XOR pipe's rate), 922 and 680; before, with B moved by one entry
// and the coefficient C_0 computed with the others, 1335, 1024 and 782. Cut after
// 10 / 12 / 13 sixteenths: 65536 1084 / 1094 / 1119.
template <int SET>
struct BMLayout {
  using p = P<SET>;
  static constexpr int Q = p::q, T = p::t, M = p::m;
  static constexpr int NS = (T + 31) / 32;
  static constexpr int R = T + 4;                              // syndrome ring entries
  static constexpr int RB = T + 1;                             // B ring entries
  static constexpr int exp_off = 0, log_off = Q;               // u16 tables (exp: indexes 0..q-2)
  static constexpr int shared_u32 = Q;
  static constexpr int s_words = R * M;                        // syndrome planes [j mod R][b]
  static constexpr int b_words = RB * M;                       // B_i of iteration n: [(i - n) mod RB][b]
  static constexpr int warp_u32 = s_words + b_words;
  static constexpr int bytes(int warps) { return shared_u32 * 4 + warps * warp_u32 * 4; }
  static_assert(32 * NS * M <= warp_u32, "C planes are staged in the warp's area");
  static_assert(32 + M - 1 <= 4 * M, "the planes of a fill at iteration n belong to s_n .. s_(n+3)");
};

// bit j of lane l -> bit l of lane j
__device__ __forceinline__ uint32_t transpose32(uint32_t v, int lane) {
  uint32_t m = 0x0000FFFFu;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t o = __shfl_xor_sync(0xffffffffu, v, s);
    v = (lane & s) ? ((o >> s) & m) | (v & ~m) : (v & m) | ((o & m) << s);
    m ^= m << (s >> 1);
  }
  return v;
}

// acc (2M-1 planes, unreduced) -> r (M planes) mod the field polynomial, in
// three-input XORs: with h_j the plane of x^(M+j), x^13 = x^4 + x^3 + x + 1
// (x^12 = x^3 + 1); h_0 .. h_2 first take what falls back above x^(M-1)
template <int M>
__device__ __forceinline__ void bs_reduce(uint32_t (&r)[M], const uint32_t (&acc)[2 * M - 1]) {
  uint32_t h[M];
#pragma unroll
  for (int j = 0; j < M - 1; j++) h[j] = acc[M + j];
  h[M - 1] = 0;
  if constexpr (M == 13) {
    h[0] ^= acc[22] ^ acc[23];
    h[1] ^= acc[23] ^ acc[24];
    h[2] ^= acc[24];
    uint32_t pr[M];  // h_k + h_(k-1)
#pragma unroll
    for (int k = 0; k < M; k++) pr[k] = k ? h[k] ^ h[k - 1] : h[0];
#pragma unroll
    for (int k = 0; k < M; k++) r[k] = k >= 3 ? acc[k] ^ pr[k] ^ pr[k - 3] : acc[k] ^ pr[k];
  } else {
    h[0] ^= acc[21];
    h[1] ^= acc[22];
#pragma unroll
    for (int k = 0; k < M; k++) r[k] = k >= 3 ? acc[k] ^ h[k] ^ h[k - 3] : acc[k] ^ h[k];
  }
}

template <int SET>
__global__ void __launch_bounds__(kBMBlockWarps * 32, 1) dec_bm_kernel(const uint32_t *__restrict__ S2, int lds2,
                                                                  FieldDev fd, const Segs segs,
                                                                  uint16_t *__restrict__ Sig, int nwb) {
  using p = P<SET>;
  using LY = BMLayout<SET>;
  constexpr int M = p::m, Q = p::q, T = p::t, D = p::fft_d;
  constexpr int NS = LY::NS, R = LY::R, RB = LY::RB;
  constexpr int SIG = 1 << D;
  static_assert(M == 12 || M == 13, "field polynomial");
  extern __shared__ __align__(16) uint32_t bsm[];
  uint16_t *gexp = reinterpret_cast<uint16_t *>(bsm) + LY::exp_off;
  uint16_t *glog = reinterpret_cast<uint16_t *>(bsm) + LY::log_off;
  chain_trigger();
  copy_table(gexp, fd.gexp, Q);
  copy_table(glog, fd.glog, Q);
  __syncthreads();
  chain_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long N = seg_rows(segs);
  const long long ngroups = (N + 31) / 32;
  // each block (one per SM) takes an equal contiguous share of the groups and
  // its warps stride over it: with a grid-wide stride, 2048 groups over 152 x 8
  // warps left 48 SMs with half the work of the others
  const long long g_lo = ngroups * blockIdx.x / gridDim.x, g_hi = ngroups * (blockIdx.x + 1) / gridDim.x;
  // one or two groups more than a multiple of four: their second half goes to the other two schedulers
  const int mine = (int)(g_hi - g_lo), base = mine & ~3, extra = mine - base;
  const bool halves = mine <= nwb && base >= 8 && (extra == 1 || extra == 2) &&
                      32 * (base + 2 + extra) <= (int)blockDim.x;  // the block has the warps for it
  const bool second = halves && warp >= base + 2;
  const int area = second ? warp - 2 : warp;  // the group's index in the block and its shared memory
  if (area >= nwb || (halves && area >= mine)) return;
  uint32_t *SP = bsm + LY::shared_u32 + area * LY::warp_u32;
  uint32_t *BP = SP + LY::s_words;
  for (long long g = g_lo + area; g < g_hi; g += nwb) {
    const bool split = halves && area >= base && 32 * (g + 1) <= N;
    if (second && !split) return;
    const long long op = g * 32 + lane;
    int seg;
    const bool live = op < N && seg_live(segs, op, &seg);
    constexpr int SW = (2 * T * M + 31) / 32;  // words of packed syndromes
    const uint32_t *srow = S2 + op * lds2;
    // C = 1, B = x
    uint32_t C[NS][M];
#pragma unroll
    for (int k = 0; k < NS; k++)
#pragma unroll
      for (int b = 0; b < M; b++) C[k][b] = 0u;
    if (!second)
      for (int w = lane; w < LY::b_words; w += 32) BP[w] = (w == M) ? 0xFFFFFFFFu : 0u;
    int L = 0, lb = 0;  // this lane's request: LFSR length, log b
    // this lane's request's packed syndromes: `have` bits of the current ones in sbits, word wn next (its value in
    // word_n), of which the planes go to ring word 32 wn mod R M + lane
    uint64_t sbits = 0;
    int have = 0, wn = 0, fill = lane;
    uint32_t word_n = live ? srow[0] : 0u;
    int es = (R - 1 - lane) % R;  // ring entry of s_{n-1-lane}
    int eb = 1 + lane;            // ring entry of B_{1+lane}
    int e0 = 0;                   // ring entry of B_0
    int n = 0;
    // a split group's registers between its halves, in its rows of Sig: C, L, log b, the syndrome bits
    uint32_t *save = reinterpret_cast<uint32_t *>(Sig + g * 32 * SIG) + lane;
    static_assert((NS * M + 5) * 32 * 4 <= 32 * SIG * 2, "the registers fit the rows of 32 locators");
    constexpr int CUT = 2 * T * kBMCutNum / 16;
    if (second) {
      asm volatile("bar.sync %0, 64;" ::"r"(1 + area - base) : "memory");
#pragma unroll
      for (int k = 0; k < NS; k++)
#pragma unroll
        for (int b = 0; b < M; b++) C[k][b] = save[(k * M + b) * 32];
      L = (int)save[(NS * M) * 32];
      lb = (int)save[(NS * M + 1) * 32];
      sbits = save[(NS * M + 2) * 32] | (uint64_t)save[(NS * M + 3) * 32] << 32;
      word_n = save[(NS * M + 4) * 32];
      // the rest follows from n: every syndrome bit below M n is used, in whole words
      n = CUT;
      wn = (CUT * M + 31) / 32;
      have = 32 * wn - CUT * M;
      fill = (32 * wn + lane) % (R * M);
      es = (CUT + R - 1 - lane) % R;
      e0 = (RB - CUT % RB) % RB;
      eb = (e0 + 1 + lane) % RB;
    }
    const int n_end = split && !second ? CUT : 2 * T;
#pragma unroll 1
    for (; n < n_end; n++) {
      if (have < M) {  // uniform
        SP[fill] = transpose32(word_n, lane);
        fill += 32;
        if (fill >= R * M) fill -= R * M;
        sbits |= (uint64_t)word_n << have;
        have += 32;
        wn++;
        word_n = live && wn < SW ? srow[wn] : 0u;  // consumed two or three iterations later
        __syncwarp();
      }
      uint32_t dq = (uint32_t)sbits & ((1u << M) - 1);  // s_n of this lane's request (C_0 = 1)
      sbits >>= M;
      have -= M;
      const int Lc = L < T ? L : T;
      int Lu = (L > n + 1 - L) ? L : n + 1 - L;
      Lu = Lu < T ? Lu : T;
      const int bd = (int)__reduce_max_sync(0xffffffffu, live ? (unsigned)Lc : 0u);
      const int bu = (int)__reduce_max_sync(0xffffffffu, live ? (unsigned)Lu : 0u);
      // discrepancy planes of the other coefficients
      if (bd > 0) {
        uint32_t acc[2 * M - 1], d[M];
#pragma unroll
        for (int k = 0; k < 2 * M - 1; k++) acc[k] = 0;
#pragma unroll
        for (int k = 0; k < NS; k++) {
          if (32 * k < bd) {
            int e = es - 32 * k;
            if (e < 0) e += R;
            const uint32_t *sp = SP + e * M;
#pragma unroll
            for (int b2 = 0; b2 < M; b2++) {
              const uint32_t sv = sp[b2];
#pragma unroll
              for (int b1 = 0; b1 < M; b1++) acc[b1 + b2] ^= C[k][b1] & sv;
            }
          }
        }
        bs_reduce<M>(d, acc);
#pragma unroll
        for (int b = 0; b < M; b++) d[b] = __reduce_xor_sync(0xffffffffu, d[b]);
#pragma unroll
        for (int b = 0; b < M; b++) dq ^= ((d[b] >> lane) & 1u) << b;
      }
      // this lane's request: f = d / b, the update decision
      const bool upd = dq != 0 && 2 * L <= n;
      uint32_t fq = 0;
      int ld = 0;
      if (dq) {
        ld = glog[dq];
        int lf = ld - lb;
        if (lf < 0) lf += Q - 1;
        fq = gexp[lf];
      }
      uint32_t f[M];
#pragma unroll
      for (int b = 0; b < M; b++) f[b] = __ballot_sync(0xffffffffu, (fq >> b) & 1u);
      const uint32_t U = __ballot_sync(0xffffffffu, upd);
      const bool anyf = __any_sync(0xffffffffu, dq != 0);
      if (upd) {
        L = n + 1 - L;
        lb = ld;
      }
      // C_i += f B_i; B_{i+1} <- (U ? C_i(old) : B_i) in B_i's entry
      if (anyf) {
#pragma unroll
        for (int k = 0; k < NS; k++) {
          if (32 * k < bu && 32 * k + lane < T) {  // coefficients above t stay zero
            int e = eb + 32 * k;
            if (e >= RB) e -= RB;
            uint32_t *bp = BP + e * M;
            uint32_t bi[M], acc[2 * M - 1];
#pragma unroll
            for (int b = 0; b < M; b++) bi[b] = bp[b];
            if (U) {
#pragma unroll
              for (int b = 0; b < M; b++) bp[b] = (U & C[k][b]) | (~U & bi[b]);
            }
#pragma unroll
            for (int x = 0; x < 2 * M - 1; x++) acc[x] = x < M ? C[k][x] : 0u;
#pragma unroll
            for (int j = 0; j < M; j++)
#pragma unroll
              for (int b = 0; b < M; b++) acc[j + b] ^= bi[b] & f[j];
            bs_reduce<M>(C[k], acc);
          }
        }
      }
      // B_1 <- U ? C_0 : B_0 = 0 in B_0's entry; the next B_0 is 0, in the entry of B_t
      const int et = e0 ? e0 - 1 : RB - 1;
      __syncwarp();
      if (lane < M) {
        if (lane == 0) BP[e0 * M] = U;
        BP[et * M + lane] = 0;
      }
      e0 = et;
      eb = eb ? eb - 1 : RB - 1;
      es = es + 1 < R ? es + 1 : 0;
      __syncwarp();
    }
    if (n_end < 2 * T) {  // the other warp goes on with this group
#pragma unroll
      for (int k = 0; k < NS; k++)
#pragma unroll
        for (int b = 0; b < M; b++) save[(k * M + b) * 32] = C[k][b];
      save[(NS * M) * 32] = (uint32_t)L;
      save[(NS * M + 1) * 32] = (uint32_t)lb;
      save[(NS * M + 2) * 32] = (uint32_t)sbits;
      save[(NS * M + 3) * 32] = (uint32_t)(sbits >> 32);
      save[(NS * M + 4) * 32] = word_n;
      __threadfence_block();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + area - base) : "memory");
      return;
    }
    // sigma(x) = sum_deg C[t-deg] x^deg -> FFT coefficient slots (deg < 2^d);
    // coefficients are < 2^m <= 2^13, so bit 15 of the constant coefficient
    // is free for the flag of a final length L != t
#pragma unroll
    for (int k = 0; k < NS; k++)
#pragma unroll
      for (int b = 0; b < M; b++) SP[(lane + 32 * k) * M + b] = C[k][b];
    const uint32_t flags = __ballot_sync(0xffffffffu, L != T);
    __syncwarp();
    const int b = lane & 15;
#pragma unroll 1
    for (int u = 0; u < SIG / 8; u++) {
      uint32_t wd[4];
#pragma unroll
      for (int x = 0; x < 4; x++) {  // two coefficients: planes b of degree deg in the half-warps
        const int deg = 8 * u + 2 * x + (lane >> 4), i = T - deg;
        uint32_t v = 0;
        if (b < M && i >= 1) v = SP[(i - 1) * M + b];
        if (b == 0 && i == 0) v = 0xFFFFFFFFu;
        if (b == 15 && deg == 0) v = flags;
        wd[x] = transpose32(v, lane);
      }
      if (live) reinterpret_cast<uint4 *>(Sig + op * SIG)[u] = make_uint4(wd[0], wd[1], wd[2], wd[3]);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- BM, constant-time form
// Bit-sliced products with both operands in registers (the multiplier a is
// warp-uniform in the callers below): Horner over the planes of a, as bs_mul.
template <int M>
__device__ __forceinline__ void bs_mul_reg(uint32_t (&r)[M], const uint32_t (&a)[M], const uint32_t (&b)[M]) {
#pragma unroll
  for (int i = 0; i < M; i++) r[i] = b[i] & a[M - 1];
#pragma unroll
  for (int j = M - 2; j >= 0; j--) {
    const uint32_t top = r[M - 1];
#pragma unroll
    for (int i = M - 1; i > 0; i--) r[i] = r[i - 1];
    r[0] = top;
    if (M == 13) {
      r[1] ^= top;
      r[3] ^= top;
      r[4] ^= top;
    } else {
      r[3] ^= top;
    }
#pragma unroll
    for (int i = 0; i < M; i++) r[i] ^= b[i] & a[j];
  }
}

// r = a^2: the planes spread to the even positions, then the reduction
template <int M>
__device__ __forceinline__ void bs_sqr(uint32_t (&r)[M], const uint32_t (&a)[M]) {
  uint32_t acc[2 * M - 1];
#pragma unroll
  for (int k = 0; k < 2 * M - 1; k++) acc[k] = (k & 1) ? 0u : a[k >> 1];
  bs_reduce<M>(r, acc);
}

template <int M>
__device__ __forceinline__ void bs_sqr_n(uint32_t (&r)[M], const uint32_t (&a)[M], int n) {
#pragma unroll
  for (int i = 0; i < M; i++) r[i] = a[i];
#pragma unroll 1
  for (int k = 0; k < n; k++) {
    uint32_t t[M];
    bs_sqr<M>(t, r);
#pragma unroll
    for (int i = 0; i < M; i++) r[i] = t[i];
  }
}

// r = a^(2^M - 2) = a^-1 (0 for a = 0), by the chain of a^(2^k - 1):
// M = 13: k = 1, 2, 3, 6, 12, then one squaring; M = 12: k = 1, 2, 3, 5, 6, 11.
template <int M>
__device__ __forceinline__ void bs_inv(uint32_t (&r)[M], const uint32_t (&a)[M]) {
  uint32_t t[M], a2[M], a3[M];
  bs_sqr<M>(t, a);
  bs_mul_reg<M>(a2, t, a);  // a^(2^2 - 1)
  bs_sqr<M>(t, a2);
  bs_mul_reg<M>(a3, t, a);  // a^(2^3 - 1)
  if (M == 13) {
    uint32_t a6[M], a12[M];
    bs_sqr_n<M>(t, a3, 3);
    bs_mul_reg<M>(a6, t, a3);  // a^(2^6 - 1)
    bs_sqr_n<M>(t, a6, 6);
    bs_mul_reg<M>(a12, t, a6);  // a^(2^12 - 1)
    bs_sqr<M>(r, a12);
  } else {
    uint32_t a5[M], a6[M], a11[M];
    bs_sqr_n<M>(t, a3, 2);
    bs_mul_reg<M>(a5, t, a2);  // a^(2^5 - 1)
    bs_sqr_n<M>(t, a3, 3);
    bs_mul_reg<M>(a6, t, a3);  // a^(2^6 - 1)
    bs_sqr_n<M>(t, a6, 5);
    bs_mul_reg<M>(a11, t, a5);  // a^(2^11 - 1)
    bs_sqr<M>(r, a11);
  }
}

// The bit-sliced arithmetic of dec_bm_kernel with nothing that depends on the
// syndromes in an address, a branch or a trip count:
//  - inversion-free update, no division d / b and no log tables: with b the
//    discrepancy of the last length change, C <- b C + d B (B carrying its x
//    shift). By induction C = lambda C_lib for a nonzero scalar lambda per
//    request (a product of b's), with the same length L and the same update
//    decisions as the library's rule (d != 0 exactly when the library's d is),
//    also under the truncation to t + 1 coefficients;
//  - slot bounds from n alone: deg C <= L <= n and deg B <= n + 1;
//  - at the end every coefficient is multiplied by lambda^-1 (C_0 = lambda;
//    one bit-sliced inversion per group), which gives the library's locator
//    (C_0 = 1) exactly.
// The update decisions stay per-request masks (ballots), L is selected, never
// branched on.
// A block holds one group of 32 requests, a warp per slot of 32 coefficients
// (lane l of warp k holds C_i, i = 1 + 32 k + l): the two products of an
// iteration take one slot's time, and a slot's planes (C, B, b, d) fit in
// registers. Every warp adds up its slot's part of the discrepancy; the parts
// meet in shared memory behind the iteration's one barrier, and every warp sums
// them and keeps b and L itself. C_0 = lambda is held by one more warp as planes
// in shared memory: its two products an iteration (lambda s_n and the next
// lambda, b lambda) have one coefficient, so they are spread over the lanes by
// output plane instead (a 33rd coefficient would cost a slot of its own).
// B_i of iteration n sits at ring entry (i - n) mod (t + 2), so the new
// B_{i+1} = (U ? C_i : B_i) replaces B_i in place.
// Bound by the integer ALU: three plane products per coefficient and iteration.
// 8192128, 8192 / 65536 requests: 425 / 2540 us, against 1095 / 3260 us with a
// warp per group holding all its slots (250 registers, 8 warps per SM, and at
// 8192 requests one or two warps on each SM).
template <int SET>
struct BMCtLayout {
  using p = P<SET>;
  static constexpr int T = p::t, M = p::m;
  static constexpr int NS = (T + 31) / 32;             // coefficient warps per block; warp NS holds lambda
  static constexpr int R = T + 2;                      // ring entries of B
  static constexpr int zero_len = 16;                  // u32: zero planes (s_j, j < 0)
  static constexpr int part_off = zero_len;            // discrepancy parts, 16 words per warp, two buffers
  static constexpr int part_len = 2 * (NS + 1) * 16;
  static constexpr int lam_off = part_off + part_len;  // lambda's planes at 16 .. 16 + M - 1, zeros around them
  static constexpr int lam_len = 64;
  static constexpr int prod_off = lam_off + lam_len;     // the unreduced planes of the lambda warp's two products
  static constexpr int prod_len = 96;
  static constexpr int s_off = prod_off + prod_len;    // syndrome planes [j][b], then C planes
  static constexpr int s_len = (2 * T * M + 31) / 32 * 32;
  static constexpr int b_off = s_off + s_len;          // B planes [ring entry][b]
  static constexpr int b_len = R * M;
  static constexpr int bytes = (b_off + b_len) * 4;
  static_assert((32 * NS + 1) * M <= s_len, "C planes are staged in the syndrome area");
};

// the first M (at most 16) words of shared memory to d, four at a time
template <int M>
__device__ __forceinline__ void load_planes(uint32_t (&d)[M], const uint32_t *src) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const uint4 v = reinterpret_cast<const uint4 *>(src)[q];
    d[4 * q] = v.x;
    d[4 * q + 1] = v.y;
    d[4 * q + 2] = v.z;
    d[4 * q + 3] = v.w;
  }
  if constexpr (M == 13) d[12] = src[12];
}
template <int M>
__device__ __forceinline__ void store_planes(uint32_t *dst, const uint32_t (&d)[M]) {
#pragma unroll
  for (int q = 0; q < 3; q++)
    reinterpret_cast<uint4 *>(dst)[q] = make_uint4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
  if constexpr (M == 13) dst[12] = d[12];
}

template <int SET>
__global__ void __launch_bounds__((BMCtLayout<SET>::NS + 1) * 32, kBMCtBlocksPerSM)
    dec_bm_ct_kernel(const uint32_t *__restrict__ S2, int lds2, const Segs segs, uint16_t *__restrict__ Sig) {
  using p = P<SET>;
  using LY = BMCtLayout<SET>;
  constexpr int M = p::m, T = p::t, D = p::fft_d;
  constexpr int NS = LY::NS, R = LY::R, THREADS = 32 * (NS + 1);
  constexpr int SIG = 1 << D;
  static_assert(M == 12 || M == 13, "field polynomial");
  extern __shared__ __align__(16) uint32_t csm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t *ZP = csm;
  uint32_t *SP = csm + LY::s_off, *BP = csm + LY::b_off, *LAM = csm + LY::lam_off + 16,
           *PROD = csm + LY::prod_off;
  const long long op = (long long)blockIdx.x * 32 + lane;
  int seg;
  const bool live = seg_live(segs, op, &seg);
  chain_trigger();
  if (!__any_sync(0xffffffffu, live)) return;  // the same for every warp
  chain_wait();
  const uint32_t *srow = S2 + op * lds2;
  for (int x = threadIdx.x; x < LY::s_off; x += THREADS) csm[x] = 0u;
  for (int w = warp; w < LY::s_len / 32; w += NS + 1) SP[32 * w + lane] = transpose32(live ? srow[w] : 0u, lane);
  for (int x = threadIdx.x; x < LY::b_len; x += THREADS) BP[x] = x == M ? 0xFFFFFFFFu : 0u;  // B = x
  __syncthreads();
  if (threadIdx.x == 0) LAM[0] = 0xFFFFFFFFu;  // C = 1
  uint32_t C[M], bq[M];  // C_i of this lane; b of every request (warp-uniform planes)
#pragma unroll
  for (int b = 0; b < M; b++) {
    C[b] = 0u;
    bq[b] = b == 0 ? 0xFFFFFFFFu : 0u;
  }
  const int i = 1 + threadIdx.x;  // this lane's coefficient (warps below NS)
  const bool in = i <= T;
  int idx = i, idx0 = 0;  // ring entries of B_i and of B_0 (never read: B_0 = 0; replaced by the new B_1)
  int L = 0;              // this lane's request
  // the lambda warp: bit j of rmask = coefficient of x^lane in x^(M + j) mod the field polynomial
  uint32_t rmask = 0;
  {
    uint32_t v = M == 13 ? 0x1Bu : 0x9u;
    for (int j = 0; j < M - 1; j++) {
      rmask |= ((v >> lane) & 1u) << j;
      v = (v << 1) ^ ((v >> (M - 1)) & 1u ? (1u << M) | (M == 13 ? 0x1Bu : 0x9u) : 0u);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int n = 0; n < 2 * T; n++) {
    const int bu = n + 1 < T ? n + 1 : T;  // deg C <= L <= n, deg B <= n + 1
    uint32_t *part = csm + LY::part_off + (n & 1) * ((NS + 1) * 16);
    uint32_t lam = 0;         // lambda warp: plane `lane` of lambda
    uint32_t acc[2 * M - 1];  // b C_i, then b C_i + d B_i, unreduced
    if (warp == NS) {
      // output plane k = lane of lambda s_n and of b lambda
      uint32_t c = 0, e = 0;
#pragma unroll
      for (int j = 0; j < M; j++) {
        const uint32_t lv = LAM[lane - j];  // zero outside lambda's planes (16 below, 19 above)
        c ^= lv & SP[n * M + j];
        e ^= lv & bq[j];
      }
      lam = LAM[lane];
      // plane M lands on a 16-byte boundary
      PROD[16 - M + lane] = c;
      PROD[48 + 16 - M + lane] = e;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const uint4 hc = reinterpret_cast<const uint4 *>(PROD + 16)[q], he = reinterpret_cast<const uint4 *>(PROD + 64)[q];
        const uint32_t vc[4] = {hc.x, hc.y, hc.z, hc.w}, ve[4] = {he.x, he.y, he.z, he.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t m = 0u - ((rmask >> (4 * q + k)) & 1u);
          c ^= vc[k] & m;
          e ^= ve[k] & m;
        }
      }
      if (lane < M) {
        part[16 * NS + lane] = c;
        LAM[lane] = e;
      }
    } else if (32 * warp < bu) {
      uint32_t d[M];
#pragma unroll
      for (int k = 0; k < 2 * M - 1; k++) acc[k] = 0;
      const int j = n - i;  // s_j, j < 0 reads the zero planes
      const uint32_t *sp = j >= 0 ? SP + j * M : ZP;
#pragma unroll
      for (int b2 = 0; b2 < M; b2++) {
        const uint32_t sv = sp[b2];
#pragma unroll
        for (int b1 = 0; b1 < M; b1++) acc[b1 + b2] ^= C[b1] & sv;
      }
      bs_reduce<M>(d, acc);
#pragma unroll
      for (int b = 0; b < M; b++) d[b] = __reduce_xor_sync(0xffffffffu, d[b]);
      // b C_i under the latency of the reductions
#pragma unroll
      for (int k = 0; k < 2 * M - 1; k++) acc[k] = 0;
#pragma unroll
      for (int b2 = 0; b2 < M; b2++)
#pragma unroll
        for (int b1 = 0; b1 < M; b1++) acc[b1 + b2] ^= bq[b1] & C[b2];
      if (lane == 0) store_planes<M>(part + 16 * warp, d);
    }
    __syncthreads();
    // the parts of warps that hold no coefficient yet are zero
    uint32_t d[M];
    load_planes<M>(d, part + 16 * NS);
#pragma unroll
    for (int k = 0; k < NS; k++) {
      uint32_t v[M];
      load_planes<M>(v, part + 16 * k);
#pragma unroll
      for (int b = 0; b < M; b++) d[b] ^= v[b];
    }
    uint32_t nz = 0;
#pragma unroll
    for (int b = 0; b < M; b++) nz |= d[b];
    const uint32_t U = nz & __ballot_sync(0xffffffffu, 2 * L <= n);
    L = ((U >> lane) & 1u) ? n + 1 - L : L;
    if (warp == NS) {
      if (lane < M) BP[idx0 * M + lane] = U & lam;  // B_1 <- (U ? C_0(old) : B_0 = 0)
    } else if (32 * warp < bu) {
      // C_i <- b C_i + d B_i; B_{i+1} <- (U ? C_i(old) : B_i)
      uint32_t *bp = BP + idx * M;
#pragma unroll
      for (int b2 = 0; b2 < M; b2++) {
        const uint32_t bi = in ? bp[b2] : 0u;
#pragma unroll
        for (int b1 = 0; b1 < M; b1++) acc[b1 + b2] ^= d[b1] & bi;
        if (i < T) bp[b2] = (U & C[b2]) | (~U & bi);
      }
      bs_reduce<M>(C, acc);  // stays zero above t
    }
    idx = idx == 0 ? R - 1 : idx - 1;
    idx0 = idx0 == 0 ? R - 1 : idx0 - 1;
#pragma unroll
    for (int b = 0; b < M; b++) bq[b] = (U & d[b]) | (~U & bq[b]);
  }
  __syncthreads();  // the syndromes are read no more
  // C <- C / C_0 (C_0 = lambda != 0)
  if (warp < NS) {
    uint32_t c0[M], inv[M], r[M];
    load_planes<M>(c0, LAM);
    bs_inv<M>(inv, c0);
    bs_mul_reg<M>(r, inv, C);
#pragma unroll
    for (int b = 0; b < M; b++) SP[i * M + b] = r[b];
  } else if (lane < M) {
    SP[lane] = lane == 0 ? 0xFFFFFFFFu : 0u;
  }
  __syncthreads();
  // the locator by degree, 8 coefficients (16 bytes of the request's row) at a time
  if (live) {
    uint4 *sig = reinterpret_cast<uint4 *>(Sig + op * SIG);
#pragma unroll 1
    for (int u = warp; u < SIG / 8; u += NS + 1) {
      uint32_t wd[4] = {0, 0, 0, 0};
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int deg = 8 * u + e, ci = T - deg;
        uint32_t v = 0;
        if (ci >= 0) {
#pragma unroll
          for (int b = 0; b < M; b++) v |= ((SP[ci * M + b] >> lane) & 1u) << b;
        }
        v |= (deg == 0 && L != T) ? 0x8000u : 0u;
        wd[e >> 1] |= v << (16 * (e & 1));
      }
      sig[u] = make_uint4(wd[0], wd[1], wd[2], wd[3]);
    }
  }
}

// ---------------------------------------------------------------- BM, latency form
// Used for small batches (fewer requests than the bit-sliced forms need to
// fill the GPU): one warp per request (persistent grid), coefficient i =
// 1 + 32 k + lane of C (connection polynomial) in slot k of a lane as its log
// only; C_0 = 1 is implicit. The update C_i += f B_i is done in the log domain
// with Zech logarithms, log(a + b) = log a + zech(log b - log a), one table
// lookup instead of an antilog and a log. Any log at or above the zero
// sentinel 2q-2 means 0. B = x^s B' is kept unshifted: B' (the connection
// polynomial before the last length change, as logs) sits in a per-warp shared
// array behind a guard of 2t zero logs, so B_i is the entry at i - s and the
// per-iteration shift is s += 1. The syndrome logs sit behind a 32-entry zero
// guard, so the discrepancy reads s_{n-i} for every lane of an active slot
// without a per-lane test (C_i = 0 above deg C). Coefficients above t are never
// updated, as in the library's fixed-size arrays.
// Degree bounds used to skip empty slots (exact, also for undecodable input):
// before iteration n, deg C <= L and deg B <= n+1-L, so both loops need
// coefficients i <= min(max(L, n+1-L), t), a bound that never falls. The
// iterations therefore run in ceil(t / 32) loops, one per number of active
// slots, each with straight-line slot code: the slots' table lookups overlap.
// With a test per slot their latencies added up: 8192128, 1 / 2048 / 8192 /
// 20000 (6688128) requests 92 / 114 / 258 / 625 us, against 58 / 74 / 199 /
// 459 us with the straight loops. Four warps per request with a barrier an iteration were slower
// (66 us for one request, 338 against 105 us for 4096).
// AHEAD, for blocks of at most kBMLatCopyWarps requests: the chain of one
// iteration is the bound there, and in it the discrepancy waits for the update
// of C. d_{n+1} = e + f q with e = sum_i C_i s_{n+1-i} of the C before the update
// and q = sum_i B_i s_{n+1-i}; when B becomes x C, q becomes that e, and else B is
// multiplied by x while n grows by one, so q stays, but for the term of a B_t that
// the multiplication moves out of the fixed arrays (deg B <= n+1-L; it counts only
// in sequences whose length ends above t: the next update makes L = n+1-L). So the
// dot product and the update of C run at the same time, without branches on d. One request 58 -> 45
// us, 2048 requests 74 -> 72; with full blocks the longer code loses (20000
// requests 461 -> 508), where the bound is the bank conflicts of the table
// lookups (about 9 shared-memory wavefronts a slot).
template <int SET>
struct BMLatLayout {
  using p = P<SET>;
  static constexpr int Q = p::q, T = p::t;
  static constexpr int NS = (T + 31) / 32;
  static constexpr int exp_off = 0, log_off = 2 * Q, zech_off = 3 * Q;
  static constexpr int shared_u16 = 4 * Q;
  static constexpr int sguard = 32, bguard = 2 * T;
  static constexpr int s_off = 0, s_len = sguard + 2 * T;          // per warp, u16
  static constexpr int raw_off = s_len, raw_len = 2 * T;
  static constexpr int b_off = raw_off + raw_len, b_len = bguard + 1 + 32 * NS;
  static constexpr int warp_u16 = (b_off + b_len + 1) & ~1;
  static constexpr int bytes(int warps) { return shared_u16 * 2 + warps * warp_u16 * 2; }
};

template <int SET, bool AHEAD>
__global__ void __launch_bounds__((AHEAD ? kBMLatCopyWarps : kBMLatWarps) * 32, 2) dec_bm_lat_kernel(const uint32_t *__restrict__ S2, int lds2,
                                                                  FieldDev fd, const Segs segs,
                                                                  uint16_t *__restrict__ Sig, int nwb) {
  using p = P<SET>;
  using LY = BMLatLayout<SET>;
  constexpr int M = p::m, Q = p::q, T = p::t, D = p::fft_d;
  constexpr int ZL = GFLog<M>::zero_log;
  constexpr int NS = LY::NS;
  constexpr int NSY = (2 * T + 31) / 32;
  constexpr int SIG = 1 << D;
  extern __shared__ __align__(16) uint16_t lsm[];
  uint16_t *gexp = lsm + LY::exp_off;
  uint16_t *glog = lsm + LY::log_off;
  uint16_t *zech = lsm + LY::zech_off;
  chain_trigger();
  copy_table(gexp, fd.gexp, 2 * Q);
  copy_table(glog, fd.glog, Q);
  copy_table(zech, fd.zech, Q);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint16_t *wsm = lsm + LY::shared_u16 + warp * LY::warp_u16;
  uint16_t *slog = wsm + LY::s_off + LY::sguard;  // slog[-32 .. -1] = zero logs
  uint16_t *sraw = wsm + LY::raw_off;
  uint16_t *blog = wsm + LY::b_off + LY::bguard;  // blog[-2t .. -1] = zero logs
  if (warp < nwb) {
    for (int i = lane; i < LY::sguard; i += 32) wsm[LY::s_off + i] = (uint16_t)ZL;
    for (int i = lane; i < LY::bguard; i += 32) wsm[LY::b_off + i] = (uint16_t)ZL;
  }
  __syncthreads();
  if (warp >= nwb) return;  // warps that only help to copy the tables
  chain_wait();
  const long long N = seg_rows(segs);
  const long long nwarps = (long long)gridDim.x * nwb;
  for (long long op = (long long)blockIdx.x * nwb + warp; op < N; op += nwarps) {
    int seg;
    if (!seg_live(segs, op, &seg)) continue;  // warp-uniform
    const uint32_t *srow = S2 + op * lds2;
#pragma unroll
    for (int k = 0; k < NSY; k++) {
      const int j = lane + 32 * k;
      if (j < 2 * T) {
        const int b = j * M, w = b >> 5, sh = b & 31;
        uint32_t v = srow[w] >> sh;
        if (sh + M > 32) v |= srow[w + 1] << (32 - sh);
        v &= Q - 1;
        sraw[j] = (uint16_t)v;
        slog[j] = glog[v];
      }
    }
    // B' = 1, s = 1 (B = x)
    for (int j = lane; j <= 32 * NS; j += 32) blog[j] = j == 0 ? 0 : (uint16_t)ZL;
    __syncwarp();
    uint32_t lC[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) lC[k] = ZL;
    int L = 0, sft = 1, n = 0;
    uint32_t lb = 0;        // log b, b = 1
    uint32_t d = sraw[0];   // AHEAD: the discrepancy of iteration n
    uint32_t lq = slog[0];  // AHEAD: log q, q = sum_i B_i s_{n+1-i}
    // the iterations that need K slots
    auto iterate = [&](auto slots) {
      constexpr int K = decltype(slots)::value;
#pragma unroll 1
      for (; n < 2 * T; n++) {
        if (K < NS && (L > 32 * K || n + 1 - L > 32 * K)) return;
        if constexpr (AHEAD) {
          if (K == NS && n - L >= T) {  // x moved B_t out of the array: its term leaves q
            const uint32_t q = gexp[min(lq, (uint32_t)ZL)] ^ gf_mul_log<M>(gexp, blog[T + 1 - sft], slog[n - T]);
            lq = glog[q];
          }
          const uint16_t *sn = slog + n - lane, *bs = blog + 1 + lane - sft;
          const uint32_t ld = glog[d];
          const bool upd = d != 0 && n >= 2 * L;
          uint32_t dp = 0, lbi[K], lco[K];
#pragma unroll
          for (int k = 0; k < K; k++) dp ^= gf_mul_log<M>(gexp, lC[k], sn[-32 * k]);
#pragma unroll
          for (int k = 0; k < K; k++) lbi[k] = bs[32 * k];
          // e = sum_i C_i s_{n+1-i} (of no use after the last iteration, where sraw[2t] is another array's)
          uint32_t e = __reduce_xor_sync(0xffffffffu, dp);
          // f = d / b; no f for d = 0
          int lf = (int)ld - (int)lb;
          lf += lf < 0 ? Q - 1 : 0;
          const uint32_t fq = gf_mul_log<M>(gexp, d ? lf : (int)ZL, (int)lq);
#pragma unroll
          for (int k = 0; k < K; k++) {
            // log(C_i + f B_i): pl = log(f B_i); zero f B_i keeps C_i, zero C_i takes pl
            constexpr uint32_t Q1 = Q - 1;
            const uint32_t lc = lC[k];
            lco[k] = lc;
            uint32_t pl = (uint32_t)lf + lbi[k];
            pl = min(pl, pl - Q1);                      // < q-1 when B_i != 0
            uint32_t kk = pl - lc;                      // log(f B_i / C_i) mod q-1
            kk = min(kk + Q1, kk);
            const uint32_t z = zech[min(kk, Q1 - 1)];   // index clamped for the zero cases
            uint32_t nl = lc + z;
            nl = min(nl, nl - Q1);                      // >= 2q-2 when the sum is 0
            nl = (lc >= (uint32_t)ZL) ? pl : nl;
            nl = (d == 0 || lbi[k] >= (uint32_t)ZL) ? lc : nl;
            if (32 * (k + 1) <= T || 1 + lane + 32 * k <= T) lC[k] = nl;  // coefficients above t stay zero
          }
          __syncwarp();  // every lane has read B' before it is replaced
#pragma unroll
          for (int k = 0; k < K; k++)
            if (upd) blog[1 + lane + 32 * k] = (uint16_t)lco[k];
          __syncwarp();
          e ^= sraw[n + 1];
          const uint32_t dnext = e ^ fq;
          const uint32_t le = glog[e & (Q - 1)];
          if (upd) {
            L = n + 1 - L;
            lb = ld;
            lq = le;  // B is x C_n from here on
            sft = 0;
          }
          d = dnext;
          sft++;
        } else {
          const uint16_t *sn = slog + n - 1 - lane, *bs = blog + 1 + lane - sft;
          uint32_t dp = 0, lbi[K];
#pragma unroll
          for (int k = 0; k < K; k++) dp ^= gf_mul_log<M>(gexp, lC[k], sn[-32 * k]);
#pragma unroll
          for (int k = 0; k < K; k++) lbi[k] = bs[32 * k];
          const uint32_t d = __reduce_xor_sync(0xffffffffu, dp) ^ sraw[n];
          if (d) {
            const bool upd = (n >= 2 * L);
            const int ld = glog[d];
            int lf = ld - (int)lb;
            if (lf < 0) lf += Q - 1;
            uint32_t lco[K];
#pragma unroll
            for (int k = 0; k < K; k++) {
              // log(C_i + f B_i): pl = log(f B_i); zero B_i keeps C_i, zero C_i takes pl
              constexpr uint32_t Q1 = Q - 1;
              const uint32_t lc = lC[k];
              lco[k] = lc;
              uint32_t pl = (uint32_t)lf + lbi[k];
              pl = min(pl, pl - Q1);                      // < q-1 when B_i != 0
              uint32_t kk = pl - lc;                      // log(f B_i / C_i) mod q-1
              kk = min(kk + Q1, kk);
              const uint32_t z = zech[min(kk, Q1 - 1)];   // index clamped for the zero cases
              uint32_t nl = lc + z;
              nl = min(nl, nl - Q1);                      // >= 2q-2 when the sum is 0
              nl = (lc >= (uint32_t)ZL) ? pl : nl;
              nl = (lbi[k] >= (uint32_t)ZL) ? lc : nl;
              if (32 * (k + 1) <= T || 1 + lane + 32 * k <= T) lC[k] = nl;  // coefficients above t stay zero
            }
            if (upd) {
              __syncwarp();  // every lane has read B' before it is replaced
#pragma unroll
              for (int k = 0; k < K; k++) blog[1 + lane + 32 * k] = (uint16_t)lco[k];
              __syncwarp();
              L = n + 1 - L;
              lb = ld;
              sft = 0;
            }
          }
          sft++;
        }
      }
    };
    iterate(std::integral_constant<int, 1>{});
    iterate(std::integral_constant<int, 2>{});
    if constexpr (NS > 2) iterate(std::integral_constant<int, 3>{});
    if constexpr (NS > 3) iterate(std::integral_constant<int, 4>{});
    static_assert(NS >= 2 && NS <= 4, "one loop per number of active slots");
    // sigma(x) = sum_deg C[t-deg] x^deg -> FFT coefficient slots (deg < 2^d);
    // coefficients are < 2^m <= 2^13, so bit 15 of the constant coefficient
    // is free for the flag of a final length L != t
    uint16_t *sig = Sig + op * SIG;
    for (int x = T + lane; x < SIG; x += 32) sig[x] = x == T ? 1 : 0;
#pragma unroll
    for (int k = 0; k < NS; k++) {
      const int i = 1 + lane + 32 * k;
      const uint32_t c = gexp[min(lC[k], (uint32_t)ZL)];
      if (i <= T) sig[T - i] = (uint16_t)(c | ((i == T && L != T) ? 0x8000u : 0u));
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- root finding
// One warp per request: additive FFT of sigma over all 2^m field elements
// (Gao-Mateer, basis beta_i = 2^i so point c is the element c), the error
// positions and the weight.
// The top-down part (twist + radix conversion) turns the 2^d coefficients
// into 2^d leaf constants. Every bottom-up butterfly level has stride < 2^d,
// so the 2^m evaluations split into 2^(m-d) independent chunks of 2^d
// consecutive elements that all start from the same leaves.
// The bottom-up pass is bit-sliced over the chunks: a 32-bit word carries one
// bit plane of the same element slot of 32 chunks, so a butterfly of 32
// chunks is one bit-sliced GF(2^m) product (m^2 AND-XOR steps and the
// reduction) instead of 64 table lookups. Lane and register slot together
// address the 2^d slots; a level whose pair bit is a lane bit first swaps
// that lane bit with the register bit of the oldest finished level (one
// shuffle per plane of half the slots), so every butterfly is in-register.
// A root (sigma(a) = 0, with a^(2^d) added for the separate leading term via
// Frobenius tables, since (hi + lo)^(2^d) = hi^(2^d) + lo^(2^d)) is mapped to
// its code position through the key's inverse support table; only roots touch
// that table.
template <int SET, bool CT>
struct RootLayout {
  using p = P<SET>;
  static constexpr int Q = p::q, D = p::fft_d, SIG = 1 << D, NC = Q >> D, NH = NC / 32, M = p::m;
  // u16 region: the table form's log/antilog tables and twist logs, or (constant-time form) the
  // multiplication columns c x^i of every twist constant c; then the Frobenius table
  static constexpr int exp_off = 0, exp_len = CT ? 0 : 2 * Q;
  static constexpr int log_off = exp_off + exp_len, log_len = CT ? 0 : Q;
  static constexpr int twist_off = log_off + log_len, twist_len = CT ? (2 << D) * M : 2 << D;
  static constexpr int frlo_off = twist_off + twist_len, frlo_len = SIG;
  static constexpr int shared_u16 = frlo_off + frlo_len;
  static_assert(log_off % 8 == 0 && twist_off % 8 == 0 && frlo_off % 8 == 0 && shared_u16 % 8 == 0,
                "tables are copied in 16-byte units");
  // u32 region: bit-sliced butterfly constants (one row of NH * M planes per level and block), bit-sliced frob_hi
  static constexpr int abs_stride = alpha_bs_stride(NH * M);
  static constexpr int abs_off = shared_u16 / 2, abs_len = ((SIG - 1) * abs_stride + 3) & ~3;
  static constexpr int fhbs_off = abs_off + abs_len, fhbs_len = (NH * M + 3) & ~3;
  static constexpr int shared_u32 = fhbs_off + fhbs_len;
  static constexpr int ewp = (p::ew + 1) & ~1;
  // per warp (u32): e words | roots [t] (element, then pos << 16 | element)
  static constexpr int roots_off = ewp;
  static constexpr int warp_u32 = (roots_off + p::t + 1) & ~1;
  static constexpr int bytes(int warps) { return shared_u32 * 4 + warps * warp_u32 * 4; }
};

// Chunk-slot index held by (lane, register slot j = j0 + 2 j1) while level l
// of the bottom-up pass is processed (l = -1: after the last level).
// Register bit 0 pairs at every level but one: a level whose pair bit is a
// lane bit first swaps that lane bit with register bit 0, whose slot bit
// (the level before) is finished. D = 7 (4 slots per lane) starts with
// slot bits 6, 5 in register bits 0, 1 and lane bits 0..4 = slot bits 0..4;
// level 5 pairs on register bit 1. D = 6 (2 slots) starts with slot bit 5 in
// register bit 0.
template <int D>
__device__ __forceinline__ int chunk_slot(int l, int lane, int j) {
  const int j0 = j & 1, j1 = j >> 1;
  if (D == 7) {
    if (l >= 5) return lane | (j1 << 5) | (j0 << 6);
    if (l < 0) return j0 | ((lane & 15) << 1) | (j1 << 5) | ((lane >> 4) << 6);
    return (lane & ((1 << l) - 1)) | (j0 << l) | (((lane >> l) & ((1 << (4 - l)) - 1)) << (l + 1)) | (j1 << 5) |
           ((lane >> 4) << 6);
  } else {
    if (l >= 5) return lane | (j0 << 5);
    if (l < 0) return j0 | (lane << 1);
    return (lane & ((1 << l) - 1)) | (j0 << l) | ((lane >> l) << (l + 1));
  }
}

// r = a * b in GF(2^M), bit-sliced (plane i = bit i of 32 elements), Horner
// over the planes of a (read from shared memory one plane per step):
// r <- r x + a_j b, where r x reduces by x^M = x^4 + x^3 + x + 1 (M = 13) or
// x^3 + 1 (M = 12), the field polynomials of the log/antilog tables.
// M^2 AND-XOR steps plus 3 (1) XORs per step; only r and b stay live.
template <int M>
__device__ __forceinline__ void bs_mul(uint32_t (&r)[M], const uint32_t *__restrict__ a, const uint32_t (&b)[M]) {
  {
    const uint32_t aj = a[M - 1];
#pragma unroll
    for (int i = 0; i < M; i++) r[i] = b[i] & aj;
  }
#pragma unroll
  for (int j = M - 2; j >= 0; j--) {
    const uint32_t top = r[M - 1];
#pragma unroll
    for (int i = M - 1; i > 0; i--) r[i] = r[i - 1];
    r[0] = top;
    if (M == 13) {
      r[1] ^= top;
      r[3] ^= top;
      r[4] ^= top;
    } else {
      r[3] ^= top;
    }
    const uint32_t aj = a[j];
#pragma unroll
    for (int i = 0; i < M; i++) r[i] ^= b[i] & aj;
  }
}

// One radix-conversion step of the top-down pass on the coefficient slots
// x = lane + 32 j held in registers: with tau = 2^pb (a bit of x), pass 1
// adds slot x + tau into every slot x whose bits (pb+1, pb) are (1, 0), then
// pass 2 adds slot x + tau into every slot whose bits are (0, 1) (whose
// partner is a pass-1 target). Bits 0..4 of x are lane bits, bits 5.. the
// register index: a pair inside a lane is an XOR, a pair across lanes one
// shuffle per register.
template <int VPL>
__device__ __forceinline__ void radix_step(uint32_t (&v)[VPL], int pb, int lane) {
  if (pb >= 5) {  // bits 6, 5 = register bits 1, 0 (VPL == 4)
    if constexpr (VPL == 4) {
      v[2] ^= v[3];
      v[1] ^= v[2];
    }
  } else if (pb == 4) {  // bit 5 = register bit 0, bit 4 = lane bit 4
    const bool hi = (lane & 16) != 0;
#pragma unroll
    for (int j = 1; j < VPL; j += 2) {  // (1, 0) <- (1, 1): register bit 0 set, partner lane ^ 16
      const uint32_t got = __shfl_xor_sync(0xffffffffu, v[j], 16);
      if (!hi) v[j] ^= got;
    }
#pragma unroll
    for (int j = 0; j < VPL; j += 2) {  // (0, 1) <- (1, 0): register j + 1 of lane ^ 16
      const uint32_t got = __shfl_xor_sync(0xffffffffu, v[j + 1], 16);
      if (hi) v[j] ^= got;
    }
  } else {  // both lane bits
    const int b = (lane >> pb) & 3;
#pragma unroll
    for (int j = 0; j < VPL; j++) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, v[j], 1 << pb);
      if (b == 2) v[j] ^= got;
    }
#pragma unroll
    for (int j = 0; j < VPL; j++) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, v[j], 3 << pb);
      if (b == 1) v[j] ^= got;
    }
  }
}

// the even bits of x, compacted into the low 16 bits
__device__ __forceinline__ uint32_t comp_even16(uint32_t x) {
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  x = (x | (x >> 8)) & 0x0000FFFFu;
  return x;
}
// exchanges the bits at p and p + d for every p in mask
__device__ __forceinline__ uint32_t delta_swap(uint32_t x, int d, uint32_t mask) {
  const uint32_t t = ((x >> d) ^ x) & mask;
  return x ^ t ^ (t << d);
}
// bit i -> bit bitrev_5(i): index bits 0 <-> 4 and 1 <-> 3 exchanged
__device__ __forceinline__ uint32_t rev5_bits(uint32_t x) {
  x = delta_swap(x, 15, 0x0000AAAAu);
  return delta_swap(x, 6, 0x00CC00CCu);
}

// v * c for a public constant c given by its columns c x^i (i < M): no
// address or branch depends on v
template <int M>
__device__ __forceinline__ uint32_t gf_mul_cols(uint32_t v, const uint16_t *cols) {
  uint32_t r = 0;
#pragma unroll
  for (int i = 0; i < M; i++) r ^= (uint32_t)cols[i] & (0u - ((v >> i) & 1u));
  return r;
}

// CT: the constant-time form (the twist multiplies by table-free columns; the
// tables indexed by coefficient values are not loaded)
template <int SET, bool CT>
__global__ void __launch_bounds__(kRootWarps * 32, 2) dec_root_kernel(const uint16_t *__restrict__ Sig,
                                                                   const DecKeys keys, FieldDev fd, const Segs segs,
                                                                   uint32_t *__restrict__ E, int lde,
                                                                   int *__restrict__ okout) {
  using p = P<SET>;
  using LY = RootLayout<SET, CT>;
  constexpr int M = p::m, Q = p::q, T = p::t, D = p::fft_d, SIG = LY::SIG, NH = LY::NH;
  constexpr int NW = (p::n + 31) / 32;
  constexpr int VPL = SIG / 32;  // chunk slots per lane
  constexpr int LOGV = (VPL == 4) ? 2 : 1;
  static_assert(VPL == (1 << LOGV) && NH == 2, "chunk geometry: 64 chunks, two halves of 32");
  static_assert(M == 12 || M == 13, "field polynomial");
  extern __shared__ __align__(16) uint32_t rsm[];
  uint16_t *sh16 = reinterpret_cast<uint16_t *>(rsm);
  uint16_t *gexp = sh16 + LY::exp_off;
  uint16_t *glog = sh16 + LY::log_off;
  uint16_t *tlog = sh16 + LY::twist_off;
  uint16_t *frlo = sh16 + LY::frlo_off;
  uint32_t *abs_ = rsm + LY::abs_off;
  uint32_t *fhbs = rsm + LY::fhbs_off;
  chain_trigger();
  if constexpr (CT) {
    copy_table(tlog, fd.fft_twist_cols, LY::twist_len);
  } else {
    copy_table(gexp, fd.gexp, 2 * Q);
    copy_table(glog, fd.glog, Q);
    copy_table(tlog, fd.fft_twist_log, 2 << D);
  }
  copy_table(frlo, fd.frob_lo, SIG);
  copy_table(abs_, fd.fft_alpha_bs, 2 * (SIG - 1) * LY::abs_stride);
  copy_table(fhbs, fd.frob_hi_bs, 2 * NH * M);
  __syncthreads();
  chain_wait();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *wbase = rsm + LY::shared_u32 + warp * LY::warp_u32;
  uint32_t *esm = wbase;
  uint32_t *roots = wbase + LY::roots_off;

  const long long N = seg_rows(segs);
  const int nwb = blockDim.x >> 5;  // warps per block (a launch parameter up to kRootWarps)
  const long long nwarps = (long long)gridDim.x * nwb;
  for (long long op = (long long)blockIdx.x * nwb + warp; op < N; op += nwarps) {
    int seg;
    if (!seg_live(segs, op, &seg)) continue;  // warp-uniform
    const DecKeyDev &key = keys.k[seg];
    const uint16_t *sig = Sig + op * SIG;
    for (int w = lane; w < NW; w += 32) esm[w] = 0;
    // top-down, in registers: lane holds the coefficient slots x = lane + 32 j
    // (j < VPL): twist by the level's first basis element, then radix-convert
    // g(x) = g0(x^2+x) + x g1(x^2+x) on the 2^l interleaved sub-polynomials
    uint32_t vv[VPL];
#pragma unroll
    for (int j = 0; j < VPL; j++) vv[j] = sig[lane + 32 * j];
    const bool bad_length = (__shfl_sync(0xffffffffu, vv[0], 0) >> 15) != 0;  // BM ended with L != t
    vv[0] &= 0x7FFFu;
#pragma unroll 1
    for (int l = 0; l < D; l++) {
      if (l) {
        const int tw0 = (2 << D) - (2 << (D - l));
        if constexpr (CT) {
#pragma unroll
          for (int j = 0; j < VPL; j++) vv[j] = gf_mul_cols<M>(vv[j], tlog + (tw0 + ((lane + 32 * j) >> l)) * M);
        } else {
#pragma unroll
          for (int j = 0; j < VPL; j++) vv[j] = gf_mul_log<M>(gexp, glog[vv[j]], tlog[tw0 + ((lane + 32 * j) >> l)]);
        }
      }
#pragma unroll 1
      for (int pb = D - 2; pb >= l; pb--) radix_step<VPL>(vv, pb, lane);
    }
    __syncwarp();  // esm cleared before the root stores below
    // leaves in the bottom-up pass's slot order (chunk_slot at level D - 1)
    uint32_t leaf[VPL];
    if constexpr (VPL == 4) {  // slot = lane | j1 << 5 | j0 << 6
      leaf[0] = vv[0];
      leaf[1] = vv[2];
      leaf[2] = vv[1];
      leaf[3] = vv[3];
    } else {  // slot = lane | j << 5
#pragma unroll
      for (int j = 0; j < VPL; j++) leaf[j] = vv[j];
    }

    uint32_t zm0[VPL], zm1[VPL];  // constant-time form: the zero masks of both chunk halves
    // table form: the roots, listed per half as found. sigma is monic of
    // degree t, so it has at most t zeros; each lane writes its own at an
    // offset from a warp prefix sum of the counts (shared memory only)
    int nfound = 0;
#pragma unroll 1
    for (int h = 0; h < NH; h++) {
      uint32_t v[VPL][M];
#pragma unroll
      for (int j = 0; j < VPL; j++)
#pragma unroll
        for (int b = 0; b < M; b++) v[j][b] = 0u - ((leaf[j] >> b) & 1u);
      // one loop body for every level (a runtime loop keeps the unrolled
      // bit-sliced products small enough for the instruction cache)
#pragma unroll 1
      for (int l = D - 1; l >= 0; l--) {
        if (VPL == 4 && l == D - 2) {
          // pairs on register bit 1 (slot bit 5)
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const int xh = chunk_slot<D>(l, lane, j) >> (l + 1);
            const uint32_t *ap = abs_ + ((SIG - (SIG >> l)) + xh) * LY::abs_stride + h * M;
            uint32_t pr[M];
            bs_mul<M>(pr, ap, v[j + 2]);
#pragma unroll
            for (int b = 0; b < M; b++) {
              v[j][b] ^= pr[b];
              v[j + 2][b] ^= v[j][b];
            }
          }
          continue;
        }
        if (l < D - LOGV) {
          // lane bit l <-> register bit 0: the lane with lane bit 0 keeps its
          // slots with register bit 0 and trades the others with its partner
          const bool lo = ((lane >> l) & 1) == 0;
#pragma unroll
          for (int j = 0; j < VPL; j += 2) {
#pragma unroll
            for (int b = 0; b < M; b++) {
              const uint32_t send = lo ? v[j + 1][b] : v[j][b];
              const uint32_t got = __shfl_xor_sync(0xffffffffu, send, 1 << l);
              if (lo) v[j + 1][b] = got;
              else v[j][b] = got;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < VPL; j += 2) {
          const int xh = chunk_slot<D>(l, lane, j) >> (l + 1);
          const uint32_t *ap = abs_ + ((SIG - (SIG >> l)) + xh) * LY::abs_stride + h * M;
          uint32_t pr[M];
          bs_mul<M>(pr, ap, v[j + 1]);
#pragma unroll
          for (int b = 0; b < M; b++) {
            v[j][b] ^= pr[b];
            v[j + 1][b] ^= v[j][b];
          }
        }
      }
      // zero planes -> roots; slot VPL * lane + j of chunk 32 h + k
      uint32_t zero[VPL];
#pragma unroll
      for (int j = 0; j < VPL; j++) {
        // read here, not hoisted out of the chunk loop (the root stores below
        // may alias), so the per-plane masks are not held across it
        const uint32_t frl = p::lead ? frlo[chunk_slot<D>(-1, lane, j)] : 0u;
        uint32_t nz = 0;
#pragma unroll
        for (int b = 0; b < M; b++) {
          uint32_t w = v[j][b];
          if (p::lead) w ^= fhbs[h * M + b] ^ (0u - ((frl >> b) & 1u));
          nz |= w;
        }
        zero[j] = ~nz;
      }
      if constexpr (CT) {
#pragma unroll
        for (int j = 0; j < VPL; j++) {
          if (h == 0) zm0[j] = zero[j];
          else zm1[j] = zero[j];
        }
        continue;
      }
      int mine = 0;
#pragma unroll
      for (int j = 0; j < VPL; j++) mine += __popc(zero[j]);
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      int off = nfound + incl - mine;
      nfound += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
      for (int j = 0; j < VPL; j++) {
        uint32_t z = zero[j];
        while (z) {
          const int k = __ffs(z) - 1;
          z &= z - 1;
          if (off < T) roots[off] = (uint32_t)(((32 * h + k) << D) | chunk_slot<D>(-1, lane, j));
          off++;
        }
      }
    }
    if constexpr (CT) {
      // the error vector in field-element order with bit-reversed index, the input order of the key's Benes
      // network: word w holds y[32 w + i] = zero(alpha) for alpha = bitrev_m(32 w + i), i.e. the slot
      // bitrev_d(w >> 1) of the chunks 2 bitrev_5(i) + (w & 1). Lane and register j hold that slot's zero
      // masks over all 64 chunks: every other bit, compacted, with its 5-bit index reversed.
      static_assert(M - D == 6, "64 chunks of 2^d slots");
      uint32_t *erow = E + op * lde;
#pragma unroll
      for (int j = 0; j < VPL; j++) {
        const int sl = chunk_slot<D>(-1, lane, j);
        const int wb = (int)(__brev((unsigned)sl) >> (32 - D)) << 1;
#pragma unroll
        for (int b0 = 0; b0 < 2; b0++) {
          const uint32_t e32 = comp_even16(zm0[j] >> b0) | (comp_even16(zm1[j] >> b0) << 16);
          erow[wb | b0] = rev5_bits(e32);
        }
      }
      if (lane == 0) okout[op] = bad_length ? 0 : 1;  // the weight is checked after the Benes network
      __syncwarp();
      continue;
    }
    // code positions of the listed roots: independent loads, lane r taking
    // entries r, r + 32, ...
    constexpr int NSC = (T + 31) / 32;
    const int nroots = nfound < T ? nfound : T;
    __syncwarp();
    int weight = 0;
    {
      uint32_t pos[NSC];
#pragma unroll
      for (int k = 0; k < NSC; k++) {
        const int r = lane + 32 * k;
        pos[k] = r < nroots ? key.invL[roots[r]] : 0xFFFFu;
      }
#pragma unroll
      for (int k = 0; k < NSC; k++) {
        const int r = lane + 32 * k;
        if (r < nroots && pos[k] < (uint32_t)p::n) {
          weight++;
          atomicOr(&esm[pos[k] >> 5], 1u << (pos[k] & 31));
        }
      }
    }
    weight = __reduce_add_sync(0xffffffffu, weight);
    __syncwarp();

    // Accept when BM's length L is t and sigma's roots are t support elements.
    // The library compares the 2t syndromes of the found error with the received
    // ones as well; that comparison cannot fail then (and for L != t no error of
    // weight t has these syndromes, whose complexity would be t):
    // - The received word is binary: its syndromes are those of f' / f mod g^2, f
    //   the product of x - L_i over its ones. With f = f0^2 + x f1^2 and s = a^2 +
    //   x b^2, (s f)' = (a f1 + b f0)^2 in characteristic 2, so (s f)' = 0 mod g^2 iff
    //   a f1 + b f0 = 0 mod g: t linear equations for the t + 1 coefficients of an s
    //   of degree <= t. Some s != 0 solves them, and s f' / f = s' mod g^2.
    // - L = t and distinct roots L_1 .. L_t of sigma: the syndromes are
    //   sum_i c_i w2_i L_i^j with no c_i = 0 (else L < t), i.e. f' / f = w / sigma mod
    //   g^2 with w coprime to sigma, deg w < t. So s w = s' sigma mod g^2, and exactly,
    //   as both have degree < 2t: sigma divides s, s = k sigma, w = sigma' and every
    //   c_i is 1, which is the found error's sequence.
    // Reading the key's syndromes at the t positions for the comparison took 82 of
    // 1062 us (8192128, 65536 requests; 27 KB per request from L2).
    const bool ok = (weight == T) && !bad_length;
    uint32_t *erow = E + op * lde;
    for (int it = lane; it < NW; it += 32) erow[it] = esm[it];
    if (lane == 0) okout[op] = ok ? 1 : 0;
    __syncwarp();
  }
}

// ---------------------------------------------------------------- root finding, request-sliced form
// For large batches. dec_root_kernel slices over the 32 chunks of one request,
// so every butterfly constant is a different element in every bit of a word
// and lane and a product costs m^2 AND-XOR steps and the reduction (about 200
// instructions). Here a word holds one plane of 32 requests and the lanes hold
// 16 such groups (and two slots with the same constant), so a butterfly's
// constant is one scalar for the whole warp and its product is a sum of shifted
// planes: kSlicedWindow bits of the constant at a time select one of 8 sums by
// branch, 62 XORs on average, 27 more for the reduction.
// Three kernels: dec_leaf (top-down pass, eight groups per block), dec_fft (the
// bottom-up butterflies of one chunk of 512 requests at a time in shared memory;
// zero masks out) and dec_pos (zero masks to error vectors in code order, weight).
// The x^t term of the sets with t = 2^d is folded into the leaves and one
// constant per chunk (build_fft_tables).
// 8192128, 65536 requests: 793 us against 980 us for dec_root_kernel; of 32768,
// dec_fft takes 360 us (221 M warp instructions, 54% of them XORs, the rest
// branches, moves and shared memory; 2.1 issued per cycle and SM, where its 16
// warps wait for branch targets), dec_leaf 45 and dec_pos 31. Windows of 2 bits:
// dec_fft 369 us. Selected sums instead of branches (what the compiler makes of
// if chains): 481. The product's code once per butterfly, 14 times: 383, waiting
// for instructions a third of the time.
constexpr int kSlicedWindow = 3;

template <int SET>
struct SlicedLayout {
  using p = P<SET>;
  static constexpr int D = p::fft_d, M = p::m, POS = 1 << D, CHUNKS = p::q >> D;
  static constexpr int GPS = 16;                    // groups of 32 requests per tile
  static constexpr int tile_words = POS * M * GPS;  // [slot][plane][group]
  static constexpr int LGPS = 8;                    // groups per block of dec_leaf
  static constexpr int leaf_bytes = POS * M * LGPS * 4;
  static constexpr int leaf_threads = 1024;
  static constexpr int off(int l) { return p::q - (p::q >> l); }  // butterfly constants of level l
  static_assert(D >= 6 && D <= 7 && CHUNKS == 64 && GPS % LGPS == 0 && LGPS % 4 == 0, "pass geometry");
};

// acc[w ..] += b V, V the value of a window of W bits of a constant
template <int M, int W, int NB, int V>
__device__ __forceinline__ void sliced_add(uint32_t (&acc)[NB][2 * M - 1], uint32_t (*const (&b)[NB])[M], int w) {
#pragma unroll
  for (int i = 0; i < NB; i++)
#pragma unroll
    for (int k = 0; k < M + W - 1; k++) {
      uint32_t x = 0;
#pragma unroll
      for (int j = 0; j < W; j++)
        if ((V >> j & 1) && k - j >= 0 && k - j < M) x ^= (*b[i])[k - j];
      if (w + k < 2 * M - 1) {
        acc[i][w + k] ^= x;
        asm volatile("" : "+r"(acc[i][w + k]));  // stays in its branch (sunk below it: a move per branch)
      }
    }
}

// the same for a window f that is the same in the whole warp
template <int M, int W, int NB>
__device__ __forceinline__ void sliced_window(uint32_t (&acc)[NB][2 * M - 1], uint32_t (*const (&b)[NB])[M],
                                              int w, uint32_t f) {
  switch (f & ((1u << W) - 1)) {
    case 0: asm volatile(""); break;
    case 1: sliced_add<M, W, NB, 1>(acc, b, w); break;
    case 2: sliced_add<M, W, NB, 2>(acc, b, w); break;
    case 3: sliced_add<M, W, NB, 3>(acc, b, w); break;
    case 4: sliced_add<M, W, NB, 4>(acc, b, w); break;
    case 5: sliced_add<M, W, NB, 5>(acc, b, w); break;
    case 6: sliced_add<M, W, NB, 6>(acc, b, w); break;
    case 7: sliced_add<M, W, NB, 7>(acc, b, w); break;
    default: break;
  }
}

// acc += b c for NB elements and one constant
template <int M, int NB>
__device__ __forceinline__ void sliced_mul(uint32_t (&acc)[NB][2 * M - 1], uint32_t (*const (&b)[NB])[M], uint32_t c) {
  constexpr int W = kSlicedWindow;
#pragma unroll
  for (int w = 0; w + W <= M; w += W) sliced_window<M, W, NB>(acc, b, w, (c >> w) & ((1u << W) - 1));
  if (M % W) sliced_window<M, M % W ? M % W : 1, NB>(acc, b, M - M % W, c >> (M - M % W));
}

// NB butterflies with one constant: lo <- lo + c hi, hi <- lo + hi
template <int M, int NB>
__device__ __forceinline__ void sliced_butterflies(uint32_t (*const (&lo)[NB])[M], uint32_t (*const (&hi)[NB])[M],
                                                   uint32_t c) {
  uint32_t acc[NB][2 * M - 1];
#pragma unroll
  for (int i = 0; i < NB; i++)
#pragma unroll
    for (int k = 0; k < 2 * M - 1; k++) acc[i][k] = k < M ? (*lo[i])[k] : 0u;
  sliced_mul<M, NB>(acc, hi, c);
#pragma unroll
  for (int i = 0; i < NB; i++) {
    bs_reduce<M>(*lo[i], acc[i]);
#pragma unroll
    for (int k = 0; k < M; k++) (*hi[i])[k] ^= (*lo[i])[k];
  }
}

// Block per LGPS groups of a tile: the coefficients transposed into planes in
// shared memory, then level by level (twist, radix conversions) in place.
template <int SET>
__global__ void __launch_bounds__(SlicedLayout<SET>::leaf_threads, 1024 / SlicedLayout<SET>::leaf_threads) dec_leaf_kernel(const uint16_t *__restrict__ Sig, FieldDev fd, const Segs segs,
                                                          uint32_t *__restrict__ Lf, int *__restrict__ okout) {
  using p = P<SET>;
  using LY = SlicedLayout<SET>;
  constexpr int M = p::m, D = LY::D, POS = LY::POS, G = LY::LGPS, THREADS = LY::leaf_threads, WARPS = THREADS / 32;
  extern __shared__ __align__(16) uint32_t tile[];  // [slot][plane][group]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long grp0 = (long long)blockIdx.x * G;
  // units of four coefficients
  for (int hu = warp; hu < POS / 4; hu += WARPS) {
    const int u = hu >> 1, half = hu & 1;
    {  // lane b of half e: plane b of coefficient 8 u + 4 half + 2 k + e
      uint32_t x[2][G];
#pragma unroll
      for (int g = 0; g < G; g++) {
        const long long op = 32 * (grp0 + g) + lane;
        int seg;
        const bool live = op < seg_rows(segs) && seg_live(segs, op, &seg);
        const uint2 c = live ? reinterpret_cast<const uint2 *>(Sig + op * POS)[2 * u + half] : make_uint2(0, 0);
        if (u == 0 && half == 0 && live) okout[op] = (c.x & 0x8000u) ? 0 : 1;  // BM ended with L != t
        x[0][g] = transpose32(c.x, lane);
        x[1][g] = transpose32(c.y, lane);
      }
      const int b = lane & 15;
      if (b < M) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
          uint4 *dst = reinterpret_cast<uint4 *>(tile + ((8 * u + 4 * half + 2 * k + (lane >> 4)) * M + b) * G);
#pragma unroll
          for (int g = 0; g < G; g += 4) dst[g / 4] = make_uint4(x[k][g], x[k][g + 1], x[k][g + 2], x[k][g + 3]);
        }
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < D; l++) {
    if (l) {
      // slot i times twist[i >> l]: the slots of a warp share the constant (two at l = 1, then 32 / G)
      const uint16_t *tw = fd.fft_twist_log + (2 << D) - (2 << (D - l));
      const int per = l == 1 ? 2 : 32 / G, e = lane / G;
#pragma unroll 1
      for (int i = warp * per; i < POS; i += WARPS * per) {
        const uint32_t c = __reduce_or_sync(0xffffffffu, fd.gexp[tw[i >> l]]);
        if (e < per) {
          uint32_t *w = tile + (i + e) * (M * G) + lane % G;
          uint32_t v[M], acc[1][2 * M - 1];
#pragma unroll
          for (int k = 0; k < 2 * M - 1; k++) acc[0][k] = 0;
#pragma unroll
          for (int k = 0; k < M; k++) v[k] = w[k * G];
          sliced_mul<M, 1>(acc, {&v}, c);
          bs_reduce<M>(v, acc[0]);
#pragma unroll
          for (int k = 0; k < M; k++) w[k * G] = v[k];
        }
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int pb = D - 2; pb >= l; pb--) {
      // quarters of every block of 4 2^pb slots: a2 += a3, a1 += a2
      const int s = 1 << pb;
      for (int t = threadIdx.x; t < POS / 4 * (M * G); t += THREADS) {
        const int q = t / (M * G), i = ((q >> pb) << (pb + 2)) | (q & (s - 1));
        uint32_t *w = tile + i * (M * G) + t % (M * G);
        const uint32_t a2 = w[2 * s * (M * G)] ^ w[3 * s * (M * G)];
        w[2 * s * (M * G)] = a2;
        w[s * (M * G)] ^= a2;
      }
      __syncthreads();
    }
  }
  uint32_t *out = Lf + (grp0 / LY::GPS) * LY::tile_words + grp0 % LY::GPS;
  for (int t = threadIdx.x; t < POS * M * (G / 4); t += THREADS) {
    const int row = t / (G / 4), c4 = t % (G / 4) * 4;
    uint4 v = *reinterpret_cast<const uint4 *>(tile + row * G + c4);
    if (p::lead) {
      const uint32_t x = 0u - ((fd.lead_leaf[row / M] >> (row % M)) & 1u);
      v.x ^= x;
      v.y ^= x;
      v.z ^= x;
      v.w ^= x;
    }
    *reinterpret_cast<uint4 *>(out + row * LY::GPS + c4) = v;
  }
}

// An item is one chunk of one tile; its levels run in three passes of tasks of
// four slots in registers, through the tile in shared memory in between:
//   pass 0  levels D-1, D-2: slots p0 + e 2^(D-2), from the leaves
//   pass 1  levels D-3, D-4: block = the two top slot bits, slots p0 + e 2^(D-4)
//   pass 2  the rest: block of 8 slots, slots p0 + 2 e, and level 0 across the
//           half-warps; zero masks out
// All levels share one loop body with two copies of the product's code (14 KB).
template <int SET>
__global__ void __launch_bounds__(256, 2) dec_fft_kernel(const uint32_t *__restrict__ Lf, FieldDev fd, long long items,
                                                         long long ngroups, uint32_t *__restrict__ Z) {
  using p = P<SET>;
  using LY = SlicedLayout<SET>;
  constexpr int M = p::m, D = LY::D, POS = LY::POS, GPS = LY::GPS, TASKS = POS / 8;
  extern __shared__ __align__(16) uint32_t tile[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane & 15, h = lane >> 4;  // group of the tile; bit 0 of the slot
  const uint32_t hm = h ? 0xFFFFFFFFu : 0u;
  const uint16_t *__restrict__ alpha = fd.fft_alpha;
  auto swap12 = [](uint32_t (&v)[4][M]) {
#pragma unroll
    for (int b = 0; b < M; b++) {
      const uint32_t x = v[1][b];
      v[1][b] = v[2][b];
      v[2][b] = x;
    }
  };
  const long long lo = items * blockIdx.x / gridDim.x, hi = items * (blockIdx.x + 1) / gridDim.x;
  for (long long it = lo; it < hi; it++) {
    const long long sg = it / LY::CHUNKS;
    const int chunk = (int)(it % LY::CHUNKS);
#pragma unroll 1
    for (int pass = 0; pass < 3; pass++) {
      if (pass) __syncthreads();
#pragma unroll 1
      for (int t = warp; t < TASKS; t += 8) {
        constexpr int LOW = TASKS / 4;  // pass 1: tasks per block
        const int blk = pass == 0 ? 0 : pass == 1 ? t / LOW : t;
        const int p0 = pass == 0 ? 2 * t + h : pass == 1 ? blk * (POS / 4) + 2 * (t % LOW) + h : 8 * t + h;
        const int s = pass == 0 ? POS / 4 : pass == 1 ? POS / 16 : 2;
        const uint32_t *src = (pass == 0 ? Lf + sg * LY::tile_words : tile) + p0 * (M * GPS) + g;
        uint32_t v[4][M];
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
          for (int b = 0; b < M; b++) v[e][b] = src[(e * s * M + b) * GPS];
        if (p::lead && pass == 0 && t == 0) {
          const uint32_t kc = fd.lead_chunk[chunk];
#pragma unroll
          for (int b = 0; b < M; b++) v[0][b] ^= (0u - ((kc >> b) & 1u)) & ~hm;
        }
        // level of the first step and the index of its block's constant; the next level's are 2 i and 2 i + 1
        const int l0 = D - 1 - 2 * pass;
        const int i0 = pass == 0 ? chunk : pass == 1 ? 4 * chunk + blk : (chunk << (D - 3)) + blk;
        const bool skip = D == 6 && pass == 2;  // (its second level is level 1)
        if (skip) swap12(v);
        const int steps = pass == 2 ? 3 : 2;
#pragma unroll 1
        for (int step = skip ? 1 : 0; step < steps; step++) {
          uint32_t ca, cb;
          if (step == 0) {
            ca = cb = alpha[(p::q - (p::q >> l0)) + i0];
          } else if (step == 1) {
            const int l = pass == 2 ? 1 : l0 - 1;
            ca = alpha[(p::q - (p::q >> l)) + 2 * i0];
            cb = alpha[(p::q - (p::q >> l)) + 2 * i0 + 1];
          } else {
            // level 0 pairs the half-warps: half 0 takes the slot pairs e = 0, 1, half 1 the pairs 2, 3, whose
            // constants are x^2 more (the level's constants are 2 i for the index i); v holds e = 0, 2, 1, 3
            ca = alpha[(chunk << (D - 1)) + 4 * blk];
            cb = alpha[(chunk << (D - 1)) + 4 * blk + 1];
#pragma unroll
            for (int b = 0; b < M; b++) {
              const uint32_t g0 = __shfl_xor_sync(0xffffffffu, h ? v[0][b] : v[1][b], 16);
              const uint32_t g1 = __shfl_xor_sync(0xffffffffu, h ? v[2][b] : v[3][b], 16);
              const uint32_t lo0 = h ? g0 : v[0][b], hi0 = h ? v[1][b] : g0;
              const uint32_t lo1 = h ? g1 : v[2][b], hi1 = h ? v[3][b] : g1;
              v[0][b] = lo0;
              v[2][b] = hi0;
              v[1][b] = lo1;
              v[3][b] = hi1;
            }
          }
          ca = __reduce_or_sync(0xffffffffu, ca);  // uniform: branches, no masks
          cb = __reduce_or_sync(0xffffffffu, cb);
          sliced_butterflies<M, 1>({&v[0]}, {&v[2]}, ca);
          sliced_butterflies<M, 1>({&v[1]}, {&v[3]}, cb);
          if (step == 0) swap12(v);  // -> e = 0, 2, 1, 3: the pairs of the next level
        }
        if (pass < 2) {
          uint32_t *dst = tile + p0 * (M * GPS) + g;
#pragma unroll
          for (int b = 0; b < M; b++) {
            dst[b * GPS] = v[0][b];
            dst[(s * M + b) * GPS] = v[2][b];
            dst[(2 * s * M + b) * GPS] = v[1][b];
            dst[(3 * s * M + b) * GPS] = v[3][b];
          }
        } else {
          uint32_t z[4];
#pragma unroll
          for (int j = 0; j < 2; j++) {
            // half 1: x^2 hi more on both outputs, hi = their sum
            const int j0 = j, j1 = j + 2;
            uint32_t f1[M], acc[2 * M - 1], fix[M], nu = 0, nv = 0;
#pragma unroll
            for (int k = 0; k < 2 * M - 1; k++) acc[k] = 0;
#pragma unroll
            for (int b = 0; b < M; b++) {
              f1[b] = (v[j0][b] ^ v[j1][b]) & hm;
              acc[b + 2] = f1[b];
            }
            bs_reduce<M>(fix, acc);
#pragma unroll
            for (int b = 0; b < M; b++) {
              nu |= v[j0][b] ^ fix[b];
              nv |= v[j1][b] ^ fix[b];
            }
            z[2 * j] = ~nu;
            z[2 * j + 1] = ~nv;
          }
          const long long grp = sg * GPS + g;
          if (grp < ngroups)
            *reinterpret_cast<uint4 *>(Z + grp * p::q + chunk * POS + 8 * t + 4 * h) = make_uint4(z[0], z[1], z[2], z[3]);
        }
      }
    }
    __syncthreads();  // the tile is read no more
  }
}

// Block per group: word w of 32 requests' error vectors is the transpose of the
// zero masks at the support elements of positions 32 w .. 32 w + 31.
template <int SET>
__global__ void __launch_bounds__(256) dec_pos_kernel(const uint32_t *__restrict__ Z, const DecKeys keys,
                                                      const Segs segs, uint32_t *__restrict__ E, int lde,
                                                      int *__restrict__ okio) {
  using p = P<SET>;
  constexpr int Q = p::q, N = p::n, NW = (N + 31) / 32;
  extern __shared__ __align__(16) uint32_t zs[];
  __shared__ int wsum[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long op = 32LL * blockIdx.x + lane;
  int seg;
  const bool live = seg_live(segs, op, &seg);
  if (!__any_sync(0xffffffffu, live)) return;  // the same for every warp
  seg = seg_find(segs, 32LL * blockIdx.x);
  for (int i = threadIdx.x; i < Q / 4; i += 256)
    reinterpret_cast<uint4 *>(zs)[i] = reinterpret_cast<const uint4 *>(Z + (long long)blockIdx.x * Q)[i];
  __syncthreads();
  const uint16_t *__restrict__ L = keys.k[seg].L;
  int weight = 0;
  for (int w0 = 4 * warp; w0 < NW; w0 += 32) {
    uint32_t x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int pos = 32 * (w0 + k) + lane;
      x[k] = transpose32(pos < N ? zs[L[pos]] : 0u, lane);
      weight += __popc(x[k]);
    }
    if (live) {
      uint32_t *row = E + op * lde + w0;
      if (w0 + 4 <= NW) {
        *reinterpret_cast<uint4 *>(row) = make_uint4(x[0], x[1], x[2], x[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (w0 + k < NW) row[k] = x[k];
      }
    }
  }
  wsum[warp][lane] = weight;
  __syncthreads();
  if (warp == 0 && live) {
    weight = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) weight += wsum[k][lane];
    if (weight != p::t) okio[op] = 0;
  }
}

// ---------------------------------------------------------------- tail
// K = SHAKE256(b || (e or s) || c), s the key's n/8 bytes (stored zero-padded
// to whole 16-byte units). The choice is a mask, not an address
// (mc:crypto_kem/348864/vec/kem_dec.c:51-55): every word is (e & mask) |
// (s & ~mask), with both read by the same loads whatever the outcome.
// Two lanes per request or a warp per request, as finalize_kernel. 8192128,
// 65536 requests: 198 us against 241 us with one lane per request; one
// request 31 us against 86 us.
template <int SET, bool PC>
struct DecHashSrc {
  using p = P<SET>;
  static constexpr int CB = p::synd_bytes + (PC ? 32 : 0);
  const uint32_t *er, *sr;
  const uint8_t *ct;
  uint32_t mask;
  bool words;  // ciphertext rows on 4-byte boundaries
  __device__ uint32_t pick(uint32_t e, uint32_t s) const { return (e & mask) | (s & ~mask); }
  __device__ uint32_t e(int w) const { return pick(er[w], sr[w]); }
  __device__ uint32_t c(int w) const {
    if (4 * w >= CB) return 0u;
    if (words) return reinterpret_cast<const uint32_t *>(ct)[w];
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (4 * w + k < CB) v |= (uint32_t)ct[4 * w + k] << (8 * k);
    return v;
  }
};

template <int SET, bool PC, bool WARP>
__global__ void __launch_bounds__(kTailThreads, WARP ? 1 : PC ? kTailBlocksPerSM - 2 : kTailBlocksPerSM)
    dec_tail_kernel(const uint32_t *__restrict__ E, int lde, const int *__restrict__ okin,
                    const uint8_t *__restrict__ Cin, const DecKeys keys, uint8_t *__restrict__ K,
                    int *__restrict__ rc, const Segs segs) {
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
  // lanes of rows that are not live hash the warp's first live row and store nothing
  const int src_lane = live ? lane : __ffs(livemask) - 1;
  const long long op = op0 + (WARP ? 0 : src_lane >> 1);
  seg = __shfl_sync(0xffffffffu, seg, src_lane);
  bool ok = okin[op] != 0;
  const uint8_t *c = Cin + op * CB;
  const uint32_t *erow = E + op * lde;
  if constexpr (PC) {
    // plaintext confirmation (mc:crypto_kem/348864pc/vec/kem_dec.c:43-48): SHAKE256(2 || e, 32) of the
    // decoded e must equal C1 (its value when decoding failed does not change the outcome)
    const EncOnlySrc esrc{erow};
    uint32_t diff = 0;
    auto c1word = [&](int j) -> uint32_t {
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) v |= (uint32_t)c[SB + 4 * j + k] << (8 * k);
      return v;
    };
    if constexpr (WARP) {
      const uint64_t h = kem_hash_warp<p::e_bytes, 1 + p::e_bytes>(2u, esrc, lane);
      if (lane < 4) diff = ((uint32_t)h ^ c1word(2 * lane)) | ((uint32_t)(h >> 32) ^ c1word(2 * lane + 1));
      diff = __reduce_or_sync(0xffffffffu, diff);
    } else {
      uint32_t cf[4];
      kem_hash_pair<p::e_bytes, 1 + p::e_bytes>(cf, 2u, esrc, half);
#pragma unroll
      for (int i = 0; i < 4; i++) diff |= cf[i] ^ c1word(2 * i + half);
      diff |= __shfl_xor_sync(0xffffffffu, diff, 1);
    }
    ok = ok && diff == 0;
  }
  const DecHashSrc<SET, PC> src{erow, reinterpret_cast<const uint32_t *>(keys.k[seg].s), c, ok ? 0xFFFFFFFFu : 0u,
                                (CB % 4 == 0) && ((reinterpret_cast<uintptr_t>(Cin) & 3) == 0)};
  uint32_t h[4];
  if constexpr (WARP) {
    const uint64_t hw = kem_hash_warp<p::e_bytes, p::pre_bytes + (PC ? 32 : 0)>(ok ? 1u : 0u, src, lane);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint64_t v = __shfl_sync(0xffffffffu, hw, i);
      h[i] = half ? (uint32_t)(v >> 32) : (uint32_t)v;
    }
  } else {
    kem_hash_pair<p::e_bytes, p::pre_bytes + (PC ? 32 : 0)>(h, ok ? 1u : 0u, src, half);
  }
  if (!live || (WARP && lane >= 2)) return;
  bool pad_bad = false;
  if (p::mt % 8) pad_bad = (c[SB - 1] >> (p::mt % 8)) != 0;
  if (pad_bad) {
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = 0xFFFFFFFFu;
  }
  store_hash_words(K + op * 32, h, half);
  if (rc && half == 0) rc[op] = pad_bad ? -1 : 0;
}

// ---------------------------------------------------------------- launchers
template <int SET>
cudaError_t launch_pack_ct(const uint8_t *C, const Segs &segs, uint32_t *X, int ldx, bool pc, cudaStream_t st) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  const long long total = N * ldx;
  if (pc)
    pack_ct_kernel<SET, true><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(C, segs, X, ldx);
  else
    pack_ct_kernel<SET, false><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(C, segs, X, ldx);
  return cudaGetLastError();
}

template <int SET>
cudaError_t launch_dec_front_few(const uint8_t *C, const Segs &segs, const GemmKeys &keys, int ldf, uint32_t *S2,
                                 int lds2, bool pc, cudaStream_t st) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  constexpr int RG = (P<SET>::s2w + kFrontFewWarps - 1) / kFrontFewWarps;
  const unsigned blocks = (unsigned)((N + 15) / 16 * RG);
  if (pc)
    dec_front_few_kernel<SET, true><<<blocks, kFrontFewWarps * 32, 0, st>>>(C, segs, keys, ldf, S2, lds2);
  else
    dec_front_few_kernel<SET, false><<<blocks, kFrontFewWarps * 32, 0, st>>>(C, segs, keys, ldf, S2, lds2);
  return cudaGetLastError();
}

template <typename K>
static int persistent_blocks(K kernel, int threads, int smem, long long work_items, int items_per_block) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm < 1) per_sm = 1;
  long long need = (work_items + items_per_block - 1) / items_per_block;
  long long blocks = (long long)sms * per_sm;
  return (int)(blocks < need ? blocks : need);
}

// Warps per block of the bit-sliced forms: at most `warps`, and no more than
// the groups of 32 requests need to spread over every SM (1024 groups take 7
// warps on 147 SMs, not 14 on 74).
static int bm_block_warps(long long N, int warps) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1) return warps;
  const long long per_sm = ((N + 31) / 32 + sms - 1) / sms;
  return per_sm < warps ? (int)(per_sm > 0 ? per_sm : 1) : warps;
}

template <int SET>
cudaError_t launch_dec_bm(const uint32_t *S2, int lds2, FieldDev fd, const Segs &segs, uint16_t *Sig,
                          cudaStream_t st, int warps, bool ct) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  if (warps < 0 || warps > kBMWarps) return cudaErrorInvalidValue;
  if (warps == 0) warps = kBMWarps;
  if (ct) {  // constant-time form, every batch size
    using LY = BMCtLayout<SET>;
    cudaError_t err =
        cudaFuncSetAttribute(dec_bm_ct_kernel<SET>, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::bytes);
    if (err != cudaSuccess) return err;
    return launch_chained(segs, dec_bm_ct_kernel<SET>, (unsigned)((N + 31) / 32), (LY::NS + 1) * 32, LY::bytes, st, S2, lds2,
                          segs, Sig);
  }
  if (!dec_bm_bitsliced_form(SET, N, ct)) {  // small batch: warp per request (lower latency per request)
    // warps per block: as few rounds over two blocks per SM as kBMLatWarps
    // allows, all of them full
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long blocks = 2LL * (sms > 0 ? sms : 1);
    const long long rounds = (N + blocks * kBMLatWarps - 1) / (blocks * kBMLatWarps);
    const int lw = (int)((N + blocks * rounds - 1) / (blocks * rounds));
    const int smem_l = BMLatLayout<SET>::bytes(lw);
    const int threads = 32 * (lw < kBMLatCopyWarps ? kBMLatCopyWarps : lw);
    auto launch = [&](auto kern) {
      cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             BMLatLayout<SET>::bytes(kBMLatWarps));
      if (err != cudaSuccess) return err;
      const int gl = persistent_blocks(kern, threads, smem_l, N, lw);
      return launch_chained(segs, kern, gl, threads, smem_l, st, S2, lds2, fd, segs, Sig, lw);
    };
    return lw <= kBMLatCopyWarps ? launch(dec_bm_lat_kernel<SET, true>) : launch(dec_bm_lat_kernel<SET, false>);
  }
  warps = bm_block_warps(N, warps);
  const int smem_bm = BMLayout<SET>::bytes(warps), threads = 32 * std::min((warps + 3) & ~3, kBMBlockWarps);
  cudaError_t err = cudaFuncSetAttribute(dec_bm_kernel<SET>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         BMLayout<SET>::bytes(kBMWarps));
  if (err != cudaSuccess) return err;
  const int gb = persistent_blocks(dec_bm_kernel<SET>, threads, smem_bm, (N + 31) / 32, warps);
  return launch_chained(segs, dec_bm_kernel<SET>, gb, threads, smem_bm, st, S2, lds2, fd, segs, Sig, warps);
}

template <int SET, bool CT>
static cudaError_t launch_dec_root_form(const uint16_t *Sig, const DecKeys &keys,
                                        FieldDev fd, const Segs &segs, uint32_t *E, int lde, int *ok,
                                        cudaStream_t st, int warps) {
  const long long N = seg_rows(segs);
  const int smem_rt = RootLayout<SET, CT>::bytes(warps);
  cudaError_t err = cudaFuncSetAttribute(dec_root_kernel<SET, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         RootLayout<SET, CT>::bytes(kRootWarps));
  if (err != cudaSuccess) return err;
  const int gr = persistent_blocks(dec_root_kernel<SET, CT>, warps * 32, smem_rt, N, warps);
  return launch_chained(segs, dec_root_kernel<SET, CT>, gr, warps * 32, smem_rt, st, Sig, keys, fd, segs, E, lde, ok);
}

template <int SET>
static cudaError_t launch_dec_root_sliced(const uint16_t *Sig, const DecKeys &keys, FieldDev fd, const Segs &segs,
                                          uint32_t *E, int lde, int *ok,
                                          cudaStream_t st, uint8_t *work) {
  using p = P<SET>;
  using LY = SlicedLayout<SET>;
  const long long N = seg_rows(segs), ngroups = N / 32, nsg = (ngroups + LY::GPS - 1) / LY::GPS;
  uint32_t *Lf = reinterpret_cast<uint32_t *>(work), *Z = Lf + nsg * LY::tile_words;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaFuncSetAttribute(dec_leaf_kernel<SET>, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::leaf_bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dec_fft_kernel<SET>, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::tile_words * 4);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(dec_pos_kernel<SET>, cudaFuncAttributeMaxDynamicSharedMemorySize, p::q * 4);
  if (e != cudaSuccess) return e;
  dec_leaf_kernel<SET><<<(unsigned)((ngroups + LY::LGPS - 1) / LY::LGPS), LY::leaf_threads, LY::leaf_bytes, st>>>(Sig, fd, segs, Lf, ok);
  const long long items = nsg * LY::CHUNKS;
  dec_fft_kernel<SET><<<(unsigned)std::min<long long>(items, 2LL * sms), 256, LY::tile_words * 4, st>>>(Lf, fd, items, ngroups,
                                                                                                  Z);
  dec_pos_kernel<SET><<<(unsigned)ngroups, 256, p::q * 4, st>>>(Z, keys, segs, E, lde, ok);
  return cudaGetLastError();
}

template <int SET>
cudaError_t launch_dec_root(const uint16_t *Sig, const DecKeys &keys, FieldDev fd, const Segs &segs, uint32_t *E,
                            int lde, int *ok, cudaStream_t st, int warps, bool ct,
                            uint8_t *work) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  if (warps < 0 || warps > kRootWarps) return cudaErrorInvalidValue;
  if (warps == 0) warps = kRootWarps;
  // (rows of E are written in 16-byte units)
  if (work && dec_root_work_bytes(SET, N, ct) && lde % 4 == 0 && (reinterpret_cast<uintptr_t>(E) & 15) == 0) {
    if (!fd.fft_alpha) return cudaErrorInvalidValue;
    return launch_dec_root_sliced<SET>(Sig, keys, fd, segs, E, lde, ok, st, work);
  }
  if (ct) {
    if (!fd.fft_twist_cols) return cudaErrorInvalidValue;
    return launch_dec_root_form<SET, true>(Sig, keys, fd, segs, E, lde, ok, st, warps);
  }
  return launch_dec_root_form<SET, false>(Sig, keys, fd, segs, E, lde, ok, st, warps);
}

// ---------------------------------------------------------------- constant-time positions
// The key's Benes network (its sk control bits, 2m - 1 layers of conditional
// swaps with strides 2^0 .. 2^(m-1) .. 2^0) applied to the field-order error
// vector y (y[v] = e at field element bitrev_m(v)) gives x[i] = y[pi(i)] with
// L_i = bitrev_m(pi(i)), i.e. the error at code position i: the same network
// and bit order that define the support (support_gen in the library). Warp per
// request, the q-bit vector in registers (word w = lane + 32 r); every layer
// touches every word with the control words as masks, so nothing depends on the
// error's positions. Then: bits >= n cleared, weight == t folded into ok.
// (The dense product that compared the found error's syndromes, which cannot
// differ, took 107 of the 150 us of this stage: 8192128, 8192 requests.)
// a layer whose pairs are registers r and r + DR of one lane (stride 2^s, s >= 10)
template <int WPL, int DR>
__device__ __forceinline__ void benes_reg_layer(uint32_t (&x)[WPL], const uint32_t *cw, int lane, int s) {
#pragma unroll
  for (int r = 0; r < WPL; r++) {
    if ((r & DR) || r + DR >= WPL) continue;
    const int wlo = lane + 32 * r;
    const uint32_t c = __ldg(cw + (((wlo >> (s - 4)) << (s - 5)) | (wlo & (32 * DR - 1))));
    const uint32_t t = (x[r] ^ x[r + DR]) & c;
    x[r] ^= t;
    x[r + DR] ^= t;
  }
}

template <int SET>
__global__ void __launch_bounds__(256) benes_ct_kernel(uint32_t *__restrict__ E, int lde, int *__restrict__ okio,
                                                       const DecKeys keys, const Segs segs) {
  using p = P<SET>;
  constexpr int M = p::m, Q = p::q, T = p::t, N = p::n;
  constexpr int WPL = Q / 32 / 32;  // words per lane
  constexpr int LW = Q / 64;         // control words per layer
  chain_trigger();
  chain_wait();
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long NR = seg_rows(segs);
  for (long long op = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); op < NR; op += nwarps) {
    int seg;
    if (!seg_live(segs, op, &seg)) continue;  // warp-uniform
    const uint32_t *cond = keys.k[seg].cond;
    uint32_t *row = E + op * lde;
    uint32_t x[WPL];
#pragma unroll
    for (int r = 0; r < WPL; r++) x[r] = row[lane + 32 * r];
#pragma unroll 1
    for (int li = 0; li < 2 * M - 1; li++) {
      const int s = li < M ? li : 2 * M - 2 - li;
      const uint32_t *cw = cond + li * LW;
      if (s < 5) {
        const int d = 1 << s;
#pragma unroll
        for (int r = 0; r < WPL; r++) {
          const int w = lane + 32 * r;
          uint32_t c = (__ldg(cw + (w >> 1)) >> (16 * (w & 1))) & 0xFFFFu;
          // deposit the 16 control bits at the pairs' lower positions (bit s of the position clear)
#pragma unroll
          for (int pb = 3; pb >= 0; pb--) {
            if (pb >= s) {
              const uint32_t mp = pb == 3 ? 0xFF00FF00u : pb == 2 ? 0xF0F0F0F0u : pb == 1 ? 0xCCCCCCCCu : 0xAAAAAAAAu;
              c = (c & ~mp) | ((c & mp) << (1 << pb));
            }
          }
          const uint32_t t = ((x[r] >> d) ^ x[r]) & c;
          x[r] ^= t ^ (t << d);
        }
      } else if (s < 10) {  // partner word in lane ^ 2^(s-5)
        const int dl = 1 << (s - 5);
#pragma unroll
        for (int r = 0; r < WPL; r++) {
          const int wlo = (lane & ~dl) + 32 * r;
          const uint32_t c = __ldg(cw + (((wlo >> (s - 4)) << (s - 5)) | (wlo & (dl - 1))));
          const uint32_t xp = __shfl_xor_sync(0xffffffffu, x[r], dl);
          x[r] ^= (x[r] ^ xp) & c;
        }
      } else if (s == 10) {  // partner word in register r ^ 2^(s-10)
        benes_reg_layer<WPL, 1>(x, cw, lane, 10);
      } else if (s == 11) {
        benes_reg_layer<WPL, 2>(x, cw, lane, 11);
      } else {
        benes_reg_layer<WPL, 4>(x, cw, lane, 12);
      }
    }
    int weight = 0;
#pragma unroll
    for (int r = 0; r < WPL; r++) {
      const int w = lane + 32 * r;
      const uint32_t keep = 32 * w + 32 <= N ? 0xFFFFFFFFu : 32 * w >= N ? 0u : (1u << (N % 32)) - 1u;
      x[r] &= keep;
      weight += __popc(x[r]);
      if (w < lde) row[w] = x[r];
    }
    weight = __reduce_add_sync(0xffffffffu, weight);
    if (lane == 0) okio[op] = okio[op] & (weight == T ? 1 : 0);
  }
}

template <int SET>
cudaError_t launch_dec_ct_finish(const DecKeys &keys, const Segs &segs, uint32_t *E, int lde, int *ok,
                                 cudaStream_t st) {
  using p = P<SET>;
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  if (lde < p::q / 32) return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long want = (N + 7) / 8;
  const int blocks = (int)(want < 8LL * sms ? want : 8LL * sms);
  return launch_chained(segs, benes_ct_kernel<SET>, blocks, 256, 0, st, E, lde, ok, keys, segs);
}

template <int SET>
cudaError_t launch_dec_tail(const uint32_t *E, int lde, const int *ok, const uint8_t *C, const DecKeys &keys,
                            uint8_t *K, int *rc, const Segs &segs, bool pc, cudaStream_t st) {
  const long long N = seg_rows(segs);
  if (N <= 0) return cudaSuccess;
  auto launch = [&](auto kern, int rows_per_block) {
    return launch_chained(segs, kern, (unsigned)((N + rows_per_block - 1) / rows_per_block), kTailThreads, 0, st, E, lde, ok, C,
                          keys, K, rc, segs);
  };
  if (hash_warp_form(segs))
    return pc ? launch(dec_tail_kernel<SET, true, true>, kTailThreads / 32)
              : launch(dec_tail_kernel<SET, false, true>, kTailThreads / 32);
  return pc ? launch(dec_tail_kernel<SET, true, false>, kTailThreads / 2)
            : launch(dec_tail_kernel<SET, false, false>, kTailThreads / 2);
}

bool dec_front_few_form(int set, const Segs &segs) {
  const gmc_setinfo &S = set_info(set);
  return seg_live_rows(segs) * S.synd_bytes * ((2 * S.t * S.m + 31) / 32) <= kFrontFewBytes;
}

bool dec_bm_bitsliced_form(int set, long long rows, bool ct) {
  return !ct && rows >= bm_bitsliced_min_rows(set_info(set).t);
}

// scratch of the request-sliced root finder, 0 where the batch takes the chunk-sliced one
size_t dec_root_work_bytes(int set, long long rows, bool ct) {
  if (ct || rows < kRootSlicedMinRows) return 0;
  auto bytes = [&](long long tile_words, long long q) {
    return (size_t)((rows + 511) / 512 * tile_words * 4 + rows / 32 * q * 4);
  };
  switch (set) {
    case 0: return bytes(SlicedLayout<0>::tile_words, P<0>::q);
    case 1: return bytes(SlicedLayout<1>::tile_words, P<1>::q);
    case 2: return bytes(SlicedLayout<2>::tile_words, P<2>::q);
    case 3: return bytes(SlicedLayout<3>::tile_words, P<3>::q);
    default: return bytes(SlicedLayout<4>::tile_words, P<4>::q);
  }
}

#define GMC_INST_DEC(SET)                                                                                       \
  template cudaError_t launch_pack_ct<SET>(const uint8_t *, const Segs &, uint32_t *, int, bool, cudaStream_t);       \
  template cudaError_t launch_dec_front_few<SET>(const uint8_t *, const Segs &, const GemmKeys &, int, uint32_t *, int, \
                                                 bool, cudaStream_t);                                            \
  template cudaError_t launch_dec_bm<SET>(const uint32_t *, int, FieldDev, const Segs &, uint16_t *,             \
                                         cudaStream_t, int, bool);                                               \
  template cudaError_t launch_dec_root<SET>(const uint16_t *, const DecKeys &, FieldDev, const Segs &,          \
                                            uint32_t *, int, int *, cudaStream_t, int, bool, uint8_t *);         \
  template cudaError_t launch_dec_tail<SET>(const uint32_t *, int, const int *, const uint8_t *, const DecKeys &, \
                                            uint8_t *, int *, const Segs &, bool, cudaStream_t);                 \
  template cudaError_t launch_dec_ct_finish<SET>(const DecKeys &, const Segs &, uint32_t *, int, int *,            \
                                                 cudaStream_t);
GMC_INST_DEC(0)
GMC_INST_DEC(1)
GMC_INST_DEC(2)
GMC_INST_DEC(3)
GMC_INST_DEC(4)

}  // namespace gmc
