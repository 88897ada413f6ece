// Kernel launchers of the engine (host-callable, templated per parameter set).
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>
#include "params.h"

namespace gmc {

constexpr int kSampleWarpsPerSM = 8;     // sampler: resident warps per SM (lanes fetch requests)
// Sampler: requests per SM up to which a request gets a block (P Keccak blocks per attempt; full: n = 2^m, where an
// attempt fails twice as often and the chains are longer). us, block per request / pairs and groups: 348864 (P = 2) 608
// requests 36 / 44, 2000 55 / 61, 3001 73 / 71; 460896 (P = 3) 608 63 / 80, 2000 100 / 101; 6960119 (P = 4) 608
// 87 / 113, 1200 108 / 119, 3001 165 / 130; 8192128 (P = 2, full) 608 75 / 109, 3001 98 / 122, 4500 116 / 131.
constexpr int sample_few_per_sm(int perms, bool full) { return full ? 30 : 36 / perms; }
constexpr int kSamplePipeWarps = 16;     // pipelined sampler: resident warps per SM unless tuned
constexpr int kSampleGroupWarps = 2;     // its groups: warps per scheduler before a warp gets a further group
constexpr int kSampleThreadsMax = 128;  // sampler block size is a launch parameter (32, 64 or 128)
// hash kernels: 64-thread blocks, 32 requests each (two lanes per request), 14
// of them resident per SM, so that 65536 requests run in one wave of 13-14
// blocks per SM
constexpr int kTailThreads = 64;
constexpr int kTailBlocksPerSM = 14;
constexpr int kFrontFewWarps = 4;  // front end of small batches: warps per block
// It is taken while live requests x ciphertext bytes x syndrome words, four times what its blocks read of the
// ciphertexts, stay below this (145 requests of 8192128, 682 of 348864). On device buffers it would win up to about
// 600 and 1000 requests, but the ciphertexts may lie in host memory: host calls of 8192128 with 128 / 256 / 600
// requests 121 / 131 / 162 us, against 124 / 126 / 154 with the product, 348864 with 600 requests 89 / 91 us.
constexpr long long kFrontFewBytes = 3 << 20;
constexpr int kBMWarps = 14;    // Berlekamp-Massey kernel: default and largest warps per block (32 requests per warp)
constexpr int kBMBlockWarps = 16;  // its block: the warps that finish split groups are in addition
constexpr int kBMCutNum = 11;      // a split group changes warps after this many sixteenths of its iterations
constexpr int kBMCtBlocksPerSM = 3;  // its constant-time form: blocks (groups of 32 requests) resident per SM
constexpr int kBMLatWarps = 24;  // Berlekamp-Massey latency form: largest warps per block (one request per warp)
constexpr int kBMLatCopyWarps = 8;  // its smallest block: warps without a request help to copy the tables
// Berlekamp-Massey: smaller batches take the latency form, a warp per request. The bit-sliced form, a warp per 32
// requests, takes the same time until every SM has seven warps. us, bit-sliced / latency form: 348864 20000 rows
// 197 / 174, 24576 198 / 217; 460896 28672 rows 428 / 404, 30720 430 / 464; 6960119 625 / 561, 622 / 641; 8192128
// 682 / 625, 680 / 705, 36864 rows 679 / 845.
constexpr long long bm_bitsliced_min_rows(int t) { return t <= 64 ? 22528 : 29696; }
// Root finding: smaller batches take the warp-per-request form. us, request-sliced / warp per request: 12288 rows
// 205 / 205 (8192128), 201 / 201 (6960119), 95 / 90 (348864); 14336 rows 205 / 226, 202 / 222, 96 / 98; 65536 rows
// 793 / 980, 778 / 970, 343 / 407.
constexpr long long kRootSlicedMinRows = 14000;
constexpr int kRootWarps = 8;  // root-finding kernel: default and largest warps per block

// ---------------------------------------------------------------- segments
// A launch covers up to kMaxSegs segments (one key each) laid out back to back
// in "padded row" space: segment s owns rows [row0[s], row0[s+1]), its live
// requests are the first nreq[s] of them, row0[] are multiples of kGemmOpPad
// (so no GEMM tile straddles two keys). Rows past a segment's live count are
// never read from or written to caller buffers. A single-key batch of n
// requests is the one-segment case {row0 = {0, round_up(n, kGemmOpPad)}}.
constexpr int kMaxSegs = 16;
struct Segs {
  int nseg;
  long long row0[kMaxSegs + 1];
  long long nreq[kMaxSegs];
};
inline long long seg_live_rows(const Segs &S) {
  long long live = 0;
  for (int i = 0; i < S.nseg; i++) live += S.nreq[i];
  return live;
}
#ifdef __CUDACC__
__host__ __device__ inline long long seg_rows(const Segs &S) { return S.row0[S.nseg]; }
__device__ inline int seg_find(const Segs &S, long long row) {
  int s = 0;
#pragma unroll 1
  for (int i = 1; i < S.nseg; i++)
    if (row >= S.row0[i]) s = i;
  return s;
}
// segment of a row and whether it is a live request
__device__ inline bool seg_live(const Segs &S, long long row, int *seg) {
  const int s = seg_find(S, row);
  *seg = s;
  return row < S.row0[S.nseg] && row - S.row0[s] < S.nreq[s];
}
#endif

// ---------------------------------------------------------------- chained launches
// The kernels of a batch form a chain, each reading what the one before wrote.
// In small batches all but the first are launched with programmatic stream
// serialization: a kernel may start as soon as every block of its predecessor
// has started (chain_trigger, first thing in each kernel) and runs its prologue
// (table copies, barrier set-up) under the predecessor's tail; chain_wait, before
// the first access to anything an earlier kernel wrote, waits for the
// predecessor's completion, and through its own wait for the whole chain.
// Decapsulation of 1 / 280 requests of 8192128 takes 111 / 126 us against 126 /
// 134 us with plain launches, of 280 of 348864 63 against 74 us. The line is at
// two requests per SM (of 152): beyond it a kernel that starts early finds some
// SMs still held by its predecessor and is placed unevenly (608 requests of
// 8192128: 153 against 139 us, constant-time decapsulation of 8192: 1110
// against 807 us).
#ifdef __CUDACC__
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif
constexpr int kChainMaxRequests = 304;
template <typename... P, typename... A>
cudaError_t launch_chained(const Segs &batch, void (*kern)(P...), unsigned blocks, unsigned threads, size_t smem,
                           cudaStream_t st, A &&...args) {
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.gridDim = dim3(blocks);
  lc.blockDim = dim3(threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  lc.attrs = at;
  lc.numAttrs = seg_live_rows(batch) <= kChainMaxRequests ? 1 : 0;
  return cudaLaunchKernelEx(&lc, kern, static_cast<P>(args)...);
}

// GF(2) GEMM engines for Out[op] = parity(A[row] & X[op]) over KW words.
// GEMM_SPARSE is the encapsulation-only alternative: e has weight t, so
// T e[mt:n] is the XOR of the <= t columns of T at e's positions, gathered by
// the sampler from a column-major image of T (no GEMM launch).
enum GemmEngine { GEMM_POPC = 0, GEMM_B1MMA = 1, GEMM_TC = 2, GEMM_SPARSE = 3 };

// Tiling of every engine: A padded to a multiple of kGemmRowTile rows and X
// to a multiple of kGemmOpTile requests, K to a multiple of kGemmKTile words.
constexpr int kGemmRowTile = 128;
constexpr int kGemmOpTile = 64;
constexpr int kGemmKTile = 8;

// Request-operand buffers (X) are padded to a multiple of kGemmOpPad rows.
constexpr int kGemmOpPad = 256;

// tcgen05 engine tiling: the key's FP8 image is kept in slices of kTcM rows;
// a CTA tile is 128 requests x 2 kTcM key rows, kTcKB bits of K per pipeline
// stage (4 MMAs of K = 32), up to kTcStages stage buffers. kTcN is the N of
// the FP8 peak measurement (128 x 256 x 32, the engine's MMA shape).
constexpr int kTcM = 128;
constexpr int kTcN = 256;
constexpr int kTcKB = 128;
constexpr int kTcStages = 4;

// Key matrices of the segments of a GEMM launch (same shape for all: one set).
// A8: the key matrix pre-expanded to FP8 stage images (GEMM_TC only).
// TT: public keys only, the columns of T as rows of ldtt words (column k is
// zero, the target of positions below mt), for GEMM_SPARSE.
struct GemmKeys {
  const uint32_t *A[kMaxSegs];
  const uint8_t *A8[kMaxSegs];
  const uint32_t *TT[kMaxSegs];
  int ldtt;
  int tc_stages;  // tcgen05 engine pipeline depth (2, 3 or 4; 0 = default 4)
};
// Out rows follow X rows (padded row space). err: device word set to 1 when a
// tensor-core CTA gave up on a bounded wait.
cudaError_t launch_gf2_gemm_seg(int engine, const GemmKeys &keys, const Segs &segs, int lda, int rows_pad,
                                const uint32_t *X, int ldx, int kw_pad, uint32_t *Out, int ldo, int out_words,
                                int *err, cudaStream_t st);
// single-key form: X has n_pad rows (multiple of kGemmOpPad), N live requests
cudaError_t launch_gf2_gemm(int engine, const uint32_t *A, const uint8_t *A8, int lda, int rows_pad,
                            const uint32_t *X, int ldx, long long n_pad, int kw_pad, uint32_t *Out, int ldo,
                            int out_words, long long N, int *err, cudaStream_t st);
size_t tc_a8_bytes(int rows_pad, int kw_pad);
// measured MMA rate of the engine's tcgen05 instruction (FP8 E4M3, M = 128, N = 256, K = 32), MACs per second;
// err_dev: a device word set to 1 if a bounded wait expired
cudaError_t time_tc_f8_peak(double *mac_per_s, int *err_dev, cudaStream_t st);
// measured rate of the legacy mma.sync m8n8k128 .b1 AND.POPC (register operands), bit-MACs per second
cudaError_t time_b1_peak(double *mac_per_s, int *out_dev, cudaStream_t st);
cudaError_t launch_expand_a(const uint32_t *A, int lda, int rows_pad, int kw_pad, uint8_t *A8, cudaStream_t st);
cudaError_t launch_gf2_gemm_tc(const GemmKeys &keys, const Segs &segs, int rows_pad, const uint32_t *X, int ldx,
                               int kw_pad, uint32_t *Out, int ldo, int out_words, int *err, cudaStream_t st);
cudaError_t launch_gf2_gemm_b1(const GemmKeys &keys, const Segs &segs, int lda, int rows_pad, const uint32_t *X,
                               int ldx, int kw_pad, uint32_t *Out, int ldo, int out_words, cudaStream_t st);
Segs one_segment(long long n);
// hash kernels: whether a launch takes a warp per request (kernels_enc.cu)
bool hash_warp_form(const Segs &segs);
// the forms that a batch takes, shared by the launchers and the autotuner (which times only parameters that its
// batch's forms read): the block-per-request sampler (kernels_enc.cu), the front end of a few decapsulations
// (kernels_dec.cu; not with an engine set by the caller) and the bit-sliced Berlekamp-Massey
bool sample_few_form(int set, const Segs &segs);
bool dec_front_few_form(int set, const Segs &segs);
bool dec_bm_bitsliced_form(int set, long long rows, bool ct);

// Encapsulation: seeds / C / K rows in padded row space; E, Ens, S have
// seg_rows(segs) rows. pk_bad_mask bit s: segment s's public key has
// nonzero padding bits (6960119), its c and K are zeroed.
// TT (k + 1 rows of ldtt words, zeroed by the caller): row j = column j of T
// (mt bits); row k stays zero.
cudaError_t launch_transpose_pk(const uint32_t *T, int lda, int mt, int k, uint32_t *TT, int ldtt, cudaStream_t st);

// Dense mode (sparse == nullptr): writes E and Ens (e[mt:n] at bit 0, the
// GEMM operand). Sparse mode: writes E and S = T e[mt:n] (lds words per row)
// from sparse->TT, and not Ens.
// counter: 4 bytes of device scratch (zeroed here, on st) that nothing else
// touches until the sampler ends; the pipelines lend the first word of the
// buffer the sampler does not write (S in dense mode, Ens in sparse mode).
// sm_warps: resident warps per SM of the pipelined sampler (0 = the default, kSamplePipeWarps).
// mark (optional): called after each kernel with its stage name (profiling).
template <int SET>
cudaError_t launch_sample(const uint8_t *seeds, const Segs &segs, uint32_t *E, int lde, uint32_t *Ens, int ldx,
                          const GemmKeys *sparse, uint32_t *S, int lds, int threads, unsigned int *counter,
                          cudaStream_t st, int sm_warps = 0, void (*mark)(const char *, cudaStream_t) = nullptr);
// C rows: synd_bytes, or synd_bytes + 32 with plaintext confirmation (pc):
// C0 || SHAKE256(2 || e, 32), K = SHAKE256(1 || e || C0 || C1).
template <int SET>
cudaError_t launch_finalize(const uint32_t *E, int lde, const uint32_t *S, int lds, uint8_t *C, uint8_t *K,
                            const Segs &segs, uint32_t pk_bad_mask, bool pc, cudaStream_t st);

// Per-key decapsulation state on the device (built once per secret key).
struct DecKeyDev {
  const uint16_t *L;     // support element of each code position [n]
  const uint16_t *invL;  // code position of each field element, 0xFFFF off the support [2^m]
  const uint8_t *s;      // implicit-rejection string [n/8]
  const uint32_t *cond;  // the sk's Benes control bits ((2m - 1) 2^(m-1) bits, as 32-bit words)
};

// Per-field / per-set device tables (shared by all keys of a set). Every table
// starts on a 16-byte boundary and is followed by readable memory up to the
// next one (the kernels copy whole 16-byte units).
constexpr int kFieldAlign = 8;  // u16 entries
struct FieldDev {
  const uint16_t *gexp;   // [2q-1]
  const uint16_t *glog;   // [q]
  const uint16_t *fft_twist_log;  // concatenated per level l = 0..d-1: [2^(d-l)]
  const uint16_t *frob_lo;        // x^(2^d) for x < 2^d
  // bit-sliced over 32 chunks per word (bit k: chunk 32 h + k), plane b = bit b
  const uint32_t *fft_alpha_bs;   // [2^d - 2^(d-l) + xh][alpha_bs_stride(H m)], entry h m + b: alpha_{l, (c << (d-1-l)) + xh}
  const uint32_t *frob_hi_bs;     // [h][m]: (c 2^d)^(2^d)
  const uint16_t *zech;           // [q]: log(1 + g^k), zech[0] = 3q (zero)
  // request-sliced root finding (null where not built): butterfly constants [q], level l from q - (q >> l); the x^t
  // term's leaves [2^d] and per-chunk constants
  const uint16_t *fft_alpha = nullptr, *lead_leaf = nullptr, *lead_chunk = nullptr;
  // [2^(d+1)][m]: for the twist constant c of each fft_twist_log entry, c x^i (i < m), so a product
  // with c needs no table indexed by the other factor (constant-time form); null where not built
  const uint16_t *fft_twist_cols = nullptr;
};

// Per-key decapsulation tables of the segments of a launch.
struct DecKeys {
  DecKeyDev k[kMaxSegs];
};

// Decapsulation: C / K / rc rows in padded row space; X, S2, Sig, E, ok have
// seg_rows(segs) rows.
// C rows of synd_bytes (+ 32 with pc); only C0 is packed.
template <int SET>
cudaError_t launch_pack_ct(const uint8_t *C, const Segs &segs, uint32_t *X, int ldx, bool pc, cudaStream_t st);
// The 2t packed syndromes of a small batch from the ciphertext bytes (keys.A: the secret keys' F, rows of ldf words).
template <int SET>
cudaError_t launch_dec_front_few(const uint8_t *C, const Segs &segs, const GemmKeys &keys, int ldf, uint32_t *S2,
                                 int lds2, bool pc, cudaStream_t st);
// Berlekamp-Massey: S2 (2t packed syndromes) -> Sig [N][2^fft_d] u16, the
// error locator's coefficients by degree (the leading x^t term is implicit
// when t = 2^fft_d).
// warps: warps per block of the bit-sliced form (1..kBMWarps; 0 = kBMWarps).
// ct: the constant-time form (inversion-free, no tables, slot bounds from the
// iteration alone; the same locators).
template <int SET>
cudaError_t launch_dec_bm(const uint32_t *S2, int lds2, FieldDev fd, const Segs &segs, uint16_t *Sig,
                          cudaStream_t st, int warps = 0, bool ct = false);
// Root finding and acceptance (BM's length flag, weight): Sig -> E (error vectors), ok.
// warps: warps per block (1..kRootWarps; 0 = kRootWarps), one request per warp.
// ct: the twist multiplies by table-free columns (needs fd.fft_twist_cols).
template <int SET>
cudaError_t launch_dec_root(const uint16_t *Sig, const DecKeys &keys, FieldDev fd, const Segs &segs, uint32_t *E,
                            int lde, int *ok, cudaStream_t st, int warps = 0, bool ct = false,
                            uint8_t *work = nullptr);
// work (16-byte aligned): scratch of the request-sliced form for batches of `rows` padded rows; 0 bytes (or a null
// pointer): the warp-per-request form
size_t dec_root_work_bytes(int set, long long rows, bool ct);
// Constant-time decapsulation, after launch_dec_root(ct = true) left the field-order error vectors in E and the
// BM-length flag in ok: the key's Benes network to code order (E in place), weight == t into ok. E rows: lde >= q/32.
template <int SET>
cudaError_t launch_dec_ct_finish(const DecKeys &keys, const Segs &segs, uint32_t *E, int lde, int *ok,
                                 cudaStream_t st);
// With pc the decoded e must also give SHAKE256(2 || e, 32) = C1 (else implicit
// rejection), and the session-key preimage covers C0 || C1.
template <int SET>
cudaError_t launch_dec_tail(const uint32_t *E, int lde, const int *ok, const uint8_t *C, const DecKeys &keys,
                            uint8_t *K, int *rc, const Segs &segs, bool pc, cudaStream_t st);

}  // namespace gmc
