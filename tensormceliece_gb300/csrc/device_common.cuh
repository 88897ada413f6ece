// Device primitives shared by the encapsulation and decapsulation kernels:
// Keccak-f[1600] on one lane, two lanes or a warp, the KEM hash, GF(2^m) log/antilog helpers.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>
#include "params.h"

namespace gmc {

// ---------------------------------------------------------------- Keccak
// FIPS 202 round constants, produced at compile time by the degree-8 LFSR
// x^8 + x^6 + x^5 + x^4 + 1 (FIPS 202, algorithm 5).
struct KeccakRC {
  uint64_t v[24];
  constexpr KeccakRC() : v() {
    unsigned r = 1;
    for (int ir = 0; ir < 24; ir++) {
      uint64_t c = 0;
      for (int j = 0; j < 7; j++) {
        if (r & 1) c |= 1ull << ((1 << j) - 1);
        r = ((r << 1) ^ ((r & 0x80) ? 0x71 : 0)) & 0xFF;
      }
      v[ir] = c;
    }
  }
};
static constexpr KeccakRC kKeccakRC{};
static __constant__ uint64_t c_keccak_rc[24] = {
    kKeccakRC.v[0],  kKeccakRC.v[1],  kKeccakRC.v[2],  kKeccakRC.v[3],  kKeccakRC.v[4],  kKeccakRC.v[5],
    kKeccakRC.v[6],  kKeccakRC.v[7],  kKeccakRC.v[8],  kKeccakRC.v[9],  kKeccakRC.v[10], kKeccakRC.v[11],
    kKeccakRC.v[12], kKeccakRC.v[13], kKeccakRC.v[14], kKeccakRC.v[15], kKeccakRC.v[16], kKeccakRC.v[17],
    kKeccakRC.v[18], kKeccakRC.v[19], kKeccakRC.v[20], kKeccakRC.v[21], kKeccakRC.v[22], kKeccakRC.v[23]};

__device__ __forceinline__ uint64_t rotl64(uint64_t x, int n) {
  return (x << n) | (x >> (64 - n));
}

// One Keccak-f[1600] permutation on 25 lanes held in registers. The
// rotation offsets follow rho's (x,y) walk; pi maps lane (x,y) to (y,2x+3y).
__device__ __forceinline__ void keccak_f1600(uint64_t A[25]) {
#pragma unroll 1
  for (int round = 0; round < 24; ++round) {
    uint64_t C0 = A[0] ^ A[5] ^ A[10] ^ A[15] ^ A[20];
    uint64_t C1 = A[1] ^ A[6] ^ A[11] ^ A[16] ^ A[21];
    uint64_t C2 = A[2] ^ A[7] ^ A[12] ^ A[17] ^ A[22];
    uint64_t C3 = A[3] ^ A[8] ^ A[13] ^ A[18] ^ A[23];
    uint64_t C4 = A[4] ^ A[9] ^ A[14] ^ A[19] ^ A[24];
    uint64_t D0 = C4 ^ rotl64(C1, 1);
    uint64_t D1 = C0 ^ rotl64(C2, 1);
    uint64_t D2 = C1 ^ rotl64(C3, 1);
    uint64_t D3 = C2 ^ rotl64(C4, 1);
    uint64_t D4 = C3 ^ rotl64(C0, 1);
    // theta + rho + pi: B[y + 5*((2x+3y)%5)] = rot(A[x+5y] ^ D[x], r(x,y))
    uint64_t B0 = A[0] ^ D0;
    uint64_t B10 = rotl64(A[1] ^ D1, 1);
    uint64_t B20 = rotl64(A[2] ^ D2, 62);
    uint64_t B5 = rotl64(A[3] ^ D3, 28);
    uint64_t B15 = rotl64(A[4] ^ D4, 27);
    uint64_t B16 = rotl64(A[5] ^ D0, 36);
    uint64_t B1 = rotl64(A[6] ^ D1, 44);
    uint64_t B11 = rotl64(A[7] ^ D2, 6);
    uint64_t B21 = rotl64(A[8] ^ D3, 55);
    uint64_t B6 = rotl64(A[9] ^ D4, 20);
    uint64_t B7 = rotl64(A[10] ^ D0, 3);
    uint64_t B17 = rotl64(A[11] ^ D1, 10);
    uint64_t B2 = rotl64(A[12] ^ D2, 43);
    uint64_t B12 = rotl64(A[13] ^ D3, 25);
    uint64_t B22 = rotl64(A[14] ^ D4, 39);
    uint64_t B23 = rotl64(A[15] ^ D0, 41);
    uint64_t B8 = rotl64(A[16] ^ D1, 45);
    uint64_t B18 = rotl64(A[17] ^ D2, 15);
    uint64_t B3 = rotl64(A[18] ^ D3, 21);
    uint64_t B13 = rotl64(A[19] ^ D4, 8);
    uint64_t B14 = rotl64(A[20] ^ D0, 18);
    uint64_t B24 = rotl64(A[21] ^ D1, 2);
    uint64_t B9 = rotl64(A[22] ^ D2, 61);
    uint64_t B19 = rotl64(A[23] ^ D3, 56);
    uint64_t B4 = rotl64(A[24] ^ D4, 14);
    // chi + iota
    A[0] = B0 ^ (~B1 & B2);  A[1] = B1 ^ (~B2 & B3);  A[2] = B2 ^ (~B3 & B4);
    A[3] = B3 ^ (~B4 & B0);  A[4] = B4 ^ (~B0 & B1);
    A[5] = B5 ^ (~B6 & B7);  A[6] = B6 ^ (~B7 & B8);  A[7] = B7 ^ (~B8 & B9);
    A[8] = B8 ^ (~B9 & B5);  A[9] = B9 ^ (~B5 & B6);
    A[10] = B10 ^ (~B11 & B12); A[11] = B11 ^ (~B12 & B13); A[12] = B12 ^ (~B13 & B14);
    A[13] = B13 ^ (~B14 & B10); A[14] = B14 ^ (~B10 & B11);
    A[15] = B15 ^ (~B16 & B17); A[16] = B16 ^ (~B17 & B18); A[17] = B17 ^ (~B18 & B19);
    A[18] = B18 ^ (~B19 & B15); A[19] = B19 ^ (~B15 & B16);
    A[20] = B20 ^ (~B21 & B22); A[21] = B21 ^ (~B22 & B23); A[22] = B22 ^ (~B23 & B24);
    A[23] = B23 ^ (~B24 & B20); A[24] = B24 ^ (~B20 & B21);
    A[0] ^= c_keccak_rc[round];
  }
}

// Keccak-f[1600] on two neighbouring lanes: lane 2s + h of a warp holds the
// low (h = 0) or high (h = 1) 32 bits of all 25 words of state s, so a rotation
// takes the other half from the neighbour (one shuffle) and every other step is
// lane-local. All 32 lanes must call. A lone permutation is bound by its own
// instruction stream (180 ALU instructions a round at one per two cycles): the
// pair form issues half of them per lane. 10 permutations measured on one GPU:
// 38 us against 54 us for the one-lane form up to 4096 states, 172 against
// 196 us for 65536 (a finer grain over the four schedulers of each SM). The
// 29 shuffles a round run in their own pipe. Rotations by IMAD (multiply by a
// power of two) instead of funnel shifts were slower in either form.
__device__ __forceinline__ void keccak_f1600_pair(uint32_t (&A)[25], int half) {
  constexpr int off[25] = {0,  1,  62, 28, 27, 36, 44, 6,  55, 20, 3,  10, 43,
                           25, 39, 41, 45, 15, 21, 8,  18, 2,  61, 56, 14};
#pragma unroll 1
  for (int round = 0; round < 24; ++round) {
    uint32_t C[5], R[5], B[25];
#pragma unroll
    for (int x = 0; x < 5; x++) C[x] = A[x] ^ A[x + 5] ^ A[x + 10] ^ A[x + 15] ^ A[x + 20];
#pragma unroll
    for (int x = 0; x < 5; x++) R[x] = __funnelshift_l(__shfl_xor_sync(0xffffffffu, C[x], 1), C[x], 1);
#pragma unroll
    for (int y = 0; y < 5; y++)
#pragma unroll
      for (int x = 0; x < 5; x++) {
        const uint32_t v = A[x + 5 * y] ^ C[(x + 4) % 5] ^ R[(x + 1) % 5];
        const int r = off[x + 5 * y];
        uint32_t w = v;
        if (r) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 1);
          w = r < 32 ? __funnelshift_l(o, v, r) : __funnelshift_l(v, o, r - 32);
        }
        B[y + 5 * ((2 * x + 3 * y) % 5)] = w;
      }
#pragma unroll
    for (int y = 0; y < 5; y++)
#pragma unroll
      for (int x = 0; x < 5; x++)
        A[x + 5 * y] = B[x + 5 * y] ^ (~B[(x + 1) % 5 + 5 * y] & B[(x + 2) % 5 + 5 * y]);
    const uint64_t rc = c_keccak_rc[round];
    A[0] ^= half ? (uint32_t)(rc >> 32) : (uint32_t)rc;
  }
}

// Keccak-f[1600] on a whole warp: lane x + 5y holds word (x, y) (lanes 25..31
// repeat lane 0). The lowest latency per permutation (10 in 30 us against 38 us
// for the pair form and 54 us for the one-lane form), at 6 times their
// instructions per state: for launches that leave most of the GPU idle.
struct KeccakWarp {
  int s1, s2, s3, s4;  // the other words of this word's column
  int xm, xp;          // a word of columns x - 1 and x + 1
  int g0, g1, g2;      // before pi: the words that become (x, y), (x + 1, y), (x + 2, y)
  int rot;             // rho offset
  bool first;          // word (0, 0)
  __device__ explicit KeccakWarp(int lane) {
    const int l = lane < 25 ? lane : 0, x = l % 5, y = l / 5;
    s1 = x + 5 * ((y + 1) % 5);
    s2 = x + 5 * ((y + 2) % 5);
    s3 = x + 5 * ((y + 3) % 5);
    s4 = x + 5 * ((y + 4) % 5);
    xm = (x + 4) % 5 + 5 * y;
    xp = (x + 1) % 5 + 5 * y;
    g0 = source(x, y);
    g1 = source((x + 1) % 5, y);
    g2 = source((x + 2) % 5, y);
    // rho's walk: (1, 0), then (x, y) -> (y, 2x + 3y), offsets (t + 1)(t + 2) / 2
    rot = 0;
    int wx = 1, wy = 0;
    for (int t = 0; t < 24; t++) {
      if (wx == x && wy == y) rot = ((t + 1) * (t + 2) / 2) & 63;
      const int nx = wy, ny = (2 * wx + 3 * wy) % 5;
      wx = nx;
      wy = ny;
    }
    first = l == 0;
  }
  // the word that pi moves to (X, Y): (x, y) -> (y, 2x + 3y), so y = X and x = (Y - 3X) / 2 mod 5
  static __device__ int source(int X, int Y) { return ((Y - 3 * X + 15) * 3) % 5 + 5 * X; }
  __device__ __forceinline__ void permute(uint64_t &a) const {
    const int r = rot & 31;
    const bool swap = rot >= 32;
#pragma unroll 1
    for (int round = 0; round < 24; ++round) {
      const uint64_t C = a ^ sh(a, s1) ^ sh(a, s2) ^ sh(a, s3) ^ sh(a, s4);
      const uint64_t cm = sh(C, xm), cp = sh(C, xp);
      const uint64_t v = a ^ cm ^ rotl64(cp, 1);
      const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32), p = swap ? hi : lo, q = swap ? lo : hi;
      const uint64_t b = (uint64_t)__funnelshift_l(q, p, r) | ((uint64_t)__funnelshift_l(p, q, r) << 32);
      a = sh(b, g0) ^ (~sh(b, g1) & sh(b, g2));
      if (first) a ^= c_keccak_rc[round];
    }
  }
  static __device__ __forceinline__ uint64_t sh(uint64_t v, int src) { return __shfl_sync(0xffffffffu, v, src); }
};

// ---------------------------------------------------------------- KEM hash
// The hash preimage is b || e || c: 32-bit word j of it is the funnel of words
// j - 1 and j of the stream e || c (word -1: b in its top byte). A source Src
// gives the stream of one request:
//   e(w)  word w of e (bits past EB bytes are zero)
//   c(w)  word w of c (zero past c)
// Words are loaded a block of 34 ahead of the permutation that absorbs them.
template <int EB, typename Src>
__device__ __forceinline__ uint32_t kem_stream_word(const Src &src, int w) {
  constexpr int EW = EB / 4;
  static_assert(EB % 4 == 0 || EB % 4 == 2, "e ends on a half word");
  if (w < EW) return src.e(w);
  if (EB % 4 == 0) return src.c(w - EW);
  if (w == EW) return src.e(w) | (src.c(0) << 16);
  return (src.c(w - EW - 1) >> 16) | (src.c(w - EW) << 16);
}

template <int EB, typename Src>
__device__ __forceinline__ uint2 kem_stream_pair(const Src &src, int w) {
  return make_uint2(kem_stream_word<EB>(src, w), kem_stream_word<EB>(src, w + 1));
}

// e alone (the plaintext-confirmation hash)
struct EncOnlySrc {
  const uint32_t *er;
  __device__ uint32_t e(int w) const { return er[w]; }
  __device__ uint32_t c(int) const { return 0u; }
};

// SHAKE256 (first 32 output bytes) of b || e || c, PRE bytes, two lanes per
// request (keccak_f1600_pair; every lane of the warp must call): lane half h
// returns the output's 32-bit words 2i + h in out[i].
template <int EB, int PRE, typename Src>
__device__ __forceinline__ void kem_hash_pair(uint32_t (&out)[4], uint32_t b, const Src &src, int half) {
  constexpr int NB = PRE / 136 + 1, rem = PRE % 136;
  uint32_t A[25];
#pragma unroll
  for (int i = 0; i < 25; i++) A[i] = 0;
  uint32_t cur[17];  // this lane's words 2i + half of the block
  auto load = [&](int blk) {
    if (34 * (blk + 1) <= EB / 4) {
#pragma unroll
      for (int i = 0; i < 17; i++) cur[i] = src.e(34 * blk + 2 * i + half);
    } else {
#pragma unroll
      for (int i = 0; i < 17; i++) cur[i] = kem_stream_word<EB>(src, 34 * blk + 2 * i + half);
    }
  };
  load(0);
  uint32_t prev = b << 24;  // the neighbour's last word (of use to half 0: its word 2i - 1)
#pragma unroll 1
  for (int blk = 0; blk < NB; blk++) {
#pragma unroll
    for (int i = 0; i < 17; i++) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, cur[i], 1);
      A[i] ^= __funnelshift_l(half ? o : prev, cur[i], 8);
      prev = o;
    }
    if (blk + 1 < NB) {
      load(blk + 1);
    } else {
      if (half == (rem % 8) / 4) A[rem / 8] ^= 0x1Fu << (8 * (rem % 4));
      if (half) A[16] ^= 0x80000000u;
    }
    keccak_f1600_pair(A, half);
  }
#pragma unroll
  for (int i = 0; i < 4; i++) out[i] = A[i];
}

// The same with a warp per request (KeccakWarp): lane i < 4 returns the output's 64-bit word i.
template <int EB, int PRE, typename Src>
__device__ __forceinline__ uint64_t kem_hash_warp(uint32_t b, const Src &src, int lane) {
  constexpr int NB = PRE / 136 + 1, rem = PRE % 136;
  const KeccakWarp kw(lane);
  uint64_t a = 0;
  uint2 cur = lane < 17 ? kem_stream_pair<EB>(src, 2 * lane) : make_uint2(0u, 0u);
  uint32_t carry = b << 24;
#pragma unroll 1
  for (int blk = 0; blk < NB; blk++) {
    uint32_t prev = __shfl_up_sync(0xffffffffu, cur.y, 1);
    if (lane == 0) prev = carry;
    carry = __shfl_sync(0xffffffffu, cur.y, 16);
    if (lane < 17) {
      a ^= (uint64_t)__funnelshift_l(prev, cur.x, 8) | ((uint64_t)__funnelshift_l(cur.x, cur.y, 8) << 32);
      if (blk + 1 < NB) {
        cur = kem_stream_pair<EB>(src, 34 * (blk + 1) + 2 * lane);
      } else {
        if (lane == rem / 8) a ^= 0x1Full << (8 * (rem % 8));
        if (lane == 16) a ^= 0x8000000000000000ull;
      }
    }
    kw.permute(a);
  }
  return a;
}

// Stores the 4 words 2i + h of a 32-byte output (v[i], lane half h) at any byte alignment.
__device__ __forceinline__ void store_hash_words(uint8_t *dst, const uint32_t (&v)[4], int half) {
  if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
    uint32_t *d = reinterpret_cast<uint32_t *>(dst);
#pragma unroll
    for (int i = 0; i < 4; i++) d[2 * i + half] = v[i];
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) dst[4 * (2 * i + half) + k] = (uint8_t)(v[i] >> (8 * k));
  }
}

// ---------------------------------------------------------------- GF(2^m)
// Log/antilog representation: log[0] = 2q-2 (sentinel), exp has 2q-1 entries
// with exp[2q-2] = 0, so a*b = exp[min(log a + log b, 2q-2)] without branches.
template <int M>
struct GFLog {
  static constexpr int q = 1 << M;
  static constexpr int zero_log = 2 * q - 2;
  static constexpr int exp_size = 2 * q - 1;
};

template <int M>
__device__ __forceinline__ uint16_t gf_mul_log(const uint16_t *__restrict__ ex, int la, int lb) {
  int s = la + lb;
  s = s < GFLog<M>::zero_log ? s : GFLog<M>::zero_log;
  return ex[s];
}

}  // namespace gmc
