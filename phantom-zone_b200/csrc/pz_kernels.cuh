// pz_kernels.cuh -- parameter blocks shared by the kernels and the host runtime.
#pragma once
#include "pz_device.cuh"

namespace pz {

constexpr int MAX_KS_D = 16;   // key-switch decomposition count bound
// Revision of the blind-rotation kernels: bumped with every change to their
// code, so that a profile taken on one revision is not reported for another.
constexpr const char *BR_KERNEL_REVISION = "br-v18";
constexpr int MAX_AUTO_SLOTS = 16;

// Everything the blind rotation needs for one parameter set + server key.
struct BrParams {
  RingConsts rc;
  Decomp da, db, dauto;
  u32 d_a, d_b, d_auto;
  u32 rgsw_rows, auto_rows;
  u32 n, br_q, w, g, emb;
  u32 ks_mask;                     // q_ks - 1: key-switched words are read modulo q_ks
  double q_ks_f, br_q_f;           // mod_switch_odd operands (pbs.rs:416-420)
  u32 auto_k[MAX_AUTO_SLOTS];      // automorphism element mod 2N per key slot
  const unsigned short *dlog;      // [br_q]
  const u64 *tv;                   // [6][br_q/2] test vectors
  const u64 *rgsw;                 // [n][rgsw_rows][N] device layout, scaled by the key form
  const u64 *autos;                // [w+1][auto_rows][N]
  const u32 *out_idx;              // optional scatter: output of gate ct -> LWE out_idx[ct]
  u32 *err;                        // the context's device error word (DEVERR_* bits)
  long long wait_limit;            // of a wait for a copy or another CTA, in clock cycles; 0: gives up at once
  // FFT form of the same keys (N = 2048 one-digit sets; null: not built) and its twiddle tables
  const void *fft_rgsw, *fft_autos, *fft_tw;
};

// Gate prelude + mod-down + LWE key switch.
struct KsParams {
  u64 Q, qby4;
  u32 mask;                 // q_ks - 1
  double q_ks_f, Q_f;       // pbs.rs:128-132 operands
  Decomp dks;
  u32 d, n, N;
  u32 ksk_stride;           // u32 words per KSK row (>= n+1)
  u32 out_stride;           // u32 words per output LWE (>= n+1)
  u32 raw;                  // inputs are combined LWEs: skip the gate prelude
  const u32 *ksk;           // [d N][ksk_stride]
  // The same KSK as byte planes for the tensor-core key switch (null: not
  // built): plane p holds bits 8p..8p+7 of every entry, in blocks of 32 rows
  // ([planes][d N / 32][ksk8_cols][32], rows permuted inside a block so that
  // one 8-byte load gives a thread its mma fragment; ksk8_cols = n + 1
  // rounded up to KSM_COLS, zero-padded).
  const unsigned char *ksk8;
  u32 planes, ksk8_cols;
  // Optional gather (circuit wires): input i of gate ct is LWE
  // c{i}[in{i}[ct] & WIRE_MASK], negated (q - x) when bit 31 is set.
  const u32 *in0, *in1;
};

// One CTA of the ragged key switch: `count` (<= 16) consecutive items of
// one session descriptor, starting at item `first`.
struct KsTile {
  u32 desc, first, count;
};
constexpr int KS_TILE_CT = 16;

constexpr u32 WIRE_NEG = 0x80000000u;
constexpr u32 WIRE_MASK = 0x7fffffffu;

// Gate codes 0..5 (and, nand, or, nor, xor, xnor).  GATE_RAW marks an input
// that is already the combined LWE (no prelude); the low bits then select
// the test vector.
constexpr unsigned char GATE_RAW = 0x80;

cudaError_t launch_key_convert(int logn, const u64 *in, u64 *out, size_t npolys, const RingConsts &rc,
                               u64 c, u64 cs, cudaStream_t s);
// err: the context's device error word (DEVERR_* bits)
cudaError_t launch_ntt_fwd(int logn, u64 *polys, size_t count, const RingConsts &rc, u32 *err, cudaStream_t s);
cudaError_t launch_ntt_inv(int logn, u64 *polys, size_t count, const RingConsts &rc, u32 *err, cudaStream_t s);
cudaError_t launch_ext_product(int logn, bool d1, const BrParams &P, u64 *rlwe, const u32 *idx,
                               size_t count, int trivial, cudaStream_t s);
cudaError_t launch_auto(int logn, bool d1, const BrParams &P, u64 *rlwe, const u32 *slot, size_t count,
                        int trivial, cudaStream_t s);
// reduce_output: leave every output word reduced mod q_ks (otherwise the
// words may carry multiples of q_ks, and consumers mask with q_ks - 1)
// ct: ciphertexts per CTA (8, 16 or 32)
// Tensor-core key switch: KSM_ROWS ciphertexts x KSM_COLS output columns
// per CTA; launch_ks takes ct = KS_CT_MMA for it.
constexpr int KSM_ROWS = 64, KSM_COLS = 224, KS_CT_MMA = 64;
inline u32 ksk8_cols(u32 n) { return (n + 1 + KSM_COLS - 1) / KSM_COLS * KSM_COLS; }
inline u32 ksk8_planes(u32 mask) {  // bytes of q_ks - 1
  u32 bits = 0;
  while (bits < 32 && (mask >> bits)) bits++;
  return (bits + 7) / 8;
}
// KSK rows (u32, stride ksk_stride, d N rows, n + 1 used columns) -> byte planes
cudaError_t launch_ksk_planes(const u32 *ksk, u32 rows, u32 stride, u32 n, u32 planes, unsigned char *out,
                              cudaStream_t s);
cudaError_t launch_ks(const KsParams &P, const unsigned char *gates, const u64 *c0, const u64 *c1,
                      size_t count, u32 *out, cudaStream_t s, bool reduce_output, int ct = KS_TILE_CT);
cudaError_t launch_pbs(int logn, bool d1, const BrParams &P, const u32 *ks, u32 ks_stride,
                       const unsigned char *gates, u64 *out, size_t count, u64 *rlwe_dbg,
                       int grid_limit, cudaStream_t s, int variant);
// Launch shapes of the N = 2048 one-digit sets.  0, 1, 2 and 4: one CTA per
// ciphertext, or by batch size on part of an SM, on one or on two (names of one
// shape, kept for callers that set them).  3: every ciphertext on a cluster of two
// CTAs (lower latency, for small batches).
constexpr int PBS_SPLIT = 3, PBS_MAX_VARIANT = 4;
// Ragged batches (several sessions / parameter sets in one launch): per-item
// descriptors in device memory; max_* bound the sizes over the descriptors.
cudaError_t launch_ks_ragged(const KsParams *d_descs, const KsTile *d_tiles, size_t ntiles, size_t count,
                             u32 max_n, u32 max_N, u32 max_d, const unsigned char *gates, const u64 *wires,
                             const u32 *in0, const u32 *in1, u32 *out, u32 out_stride, cudaStream_t s);
// The ragged key switch on the tensor cores: tiles of up to KSM_ROWS items,
// every session's key with its byte planes (KsParams::ksk8), d <= 16.
cudaError_t launch_ks_mma_ragged(const KsParams *d_descs, const KsTile *d_tiles, size_t ntiles, size_t count,
                                 u32 max_n, u32 max_N, u32 max_d, const unsigned char *gates, const u64 *wires,
                                 const u32 *in0, const u32 *in1, u32 *out, u32 out_stride, cudaStream_t s);
cudaError_t launch_pbs_ragged(int logn, bool d1, const BrParams *d_descs, const u32 *item_desc, u32 max_br_q,
                              u32 max_n, const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out,
                              const u32 *out_idx, size_t count, int grid_limit, cudaStream_t s, int variant,
                              bool fft);  // fft: every descriptor in use has its key's FFT form
// dynamic shared memory of a kernel, opted into once per device and size
cudaError_t opt_in_smem(const void *kernel, size_t bytes);
// FFT form (pz_fft.cu): the twiddle tables of a device, the bytes and the
// conversion of `keys` keys of rows_per_key device rows, and the one-digit
// N = 2048 blind rotation over it.
cudaError_t fft_tables(void **out);
size_t fft_key_bytes(size_t keys);
cudaError_t launch_fft_key(const u64 *rows, u32 rows_per_key, size_t keys, const RingConsts &rc, const void *tables,
                           void *out, cudaStream_t s);
cudaError_t launch_pbs_fft(const BrParams &P, const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out,
                           size_t count, u64 *rlwe_dbg, int grid, cudaStream_t s, bool split);
// How many ciphertexts a blind rotation of `count` is best filled up to where more
// are waiting, with the FFT form or without.
size_t pbs_fill(size_t count, size_t sms, bool fft);
cudaError_t pbs_fft_per_sm(u32 br_q, u32 n, int *ctas);  // resident CTAs per SM (as four ciphertexts)
cudaError_t pbs_fft_clusters(u32 br_q, u32 n, size_t *clusters);  // resident clusters of the two-SM form
cudaError_t launch_pbs_fft_ragged(const BrParams *d_descs, const u32 *item_desc, u32 max_br_q, u32 max_n, const u32 *ks,
                                  u32 ks_stride, const unsigned char *gates, u64 *out, const u32 *out_idx,
                                  size_t count, int grid, cudaStream_t s, bool split);
cudaError_t launch_fft_product(const BrParams &P, u64 *rlwe, const u32 *idx, size_t count, int trivial,
                               cudaStream_t s);
cudaError_t launch_fft_auto(const BrParams &P, u64 *rlwe, const u32 *slot, size_t count, cudaStream_t s);
// Non-interactive key switch over FFT products (pz_fft_ni.cu; one-bit digits,
// d = NI_FFT_D).  Bytes of a user's key form, of `rows` values' transformed
// digits (and what may be read beyond them) and of one (value, user)'s sums;
// `keys`: device array of the users' key forms.
constexpr u32 NI_FFT_D = 50;
size_t ni_fft_key_bytes(u32 d);
size_t ni_fft_digit_bytes(u32 d, size_t rows);
size_t ni_fft_sum_bytes();
cudaError_t launch_ni_fft_key(const u64 *rows, u32 d, const void *tables, void *out,
                              cudaStream_t s);  // rows: [2 d][N] coefficients
// out = rlwe_key_switch(in), [rows][2][N]
cudaError_t launch_ni_fft_switch(const u64 *in, u64 *out, size_t rows, u32 d, const Decomp &dp,
                                 const void *const *keys, const void *tables, void *digits, void *sums, u32 *err,
                                 cudaStream_t s);
// Key aggregation: row v = row % (ra + rb) of LWE index idx0 + row / (ra + rb),
// switched for every user, the user's NI RGSW row added and stored into the
// leader's RGSW (rlwe x rgsw shape: rows A(-sm), B(-sm), A(m), B(m); only its
// last zero-encryption and last -a value) or, for every other user t in
// increasing id, into others[t][index]: rows v / ra + v for zero-encryption
// values, 2 ra + r / 2 ra + rb + r for -a values.
struct NiRowUser {
  const u64 *self_leader, *not_leader;
  u32 seg_b, seg_e;
};
struct NiRows {
  u32 ra, rb, max_d, max_l, per_user, idx0, cnt;
  const NiRowUser *users;
  u64 *leader, *others;
};
cudaError_t launch_ni_fft_rows(const u64 *vals, size_t rows, u32 users, u32 d, const Decomp &dp, const NiRows &R,
                               const void *const *keys, const void *tables, void *digits, void *sums, u32 *err,
                               cudaStream_t s);
cudaError_t launch_not(const u64 *in, u64 *out, size_t words, u64 q, cudaStream_t s);
cudaError_t launch_imad_probe(int blocks, int threads, u32 iters, u32 *sink, cudaStream_t s);
cudaError_t launch_pipe_probe(int kind, int blocks, int threads, u32 iters, u32 *sink, cudaStream_t s);
// per launch: blocks * threads * iters * 16 * 8 multiply-adds
size_t pbs_smem_bytes(int logn, u32 br_q, u32 n);
// blind-rotation items resident at once for a launch shape (whole-wave size)
cudaError_t pbs_slots(int logn, bool d1, u32 br_q, u32 n, int variant, size_t *slots);

}  // namespace pz
