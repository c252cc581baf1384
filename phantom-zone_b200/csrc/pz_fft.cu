// pz_fft.cu -- the blind rotation, external product and automorphism of the
// N = 2048 one-digit parameter sets over exact FP64 FFT products (pz_fft.cuh).
#include <algorithm>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "pz_blind.cuh"
#include "pz_fft.cuh"
#include "pz_internal.h"

namespace pz {
namespace fft {

constexpr int N = 2048;
constexpr unsigned short OP_END = 0xffffu;  // after the schedule's last operation

// Key form of the blind rotation.  One CTA per (key block, row).  rows_per_key
// device rows per key: 4 for RGSW (A(-sm), B(-sm), A(m), B(m)), 2 for
// automorphism keys (A, B), whose second digit half uses 2^AUTO_CUT times the row.
__global__ void __launch_bounds__(256)
    fft_key_kernel(const u64 *rows, cplx *out, u32 rows_per_key, RingConsts rc, const double4 *tw) {
  __shared__ u64 coef[N];
  extern __shared__ double dyn[];
  const u32 key = blockIdx.x >> 2, in = (blockIdx.x >> 1) & 1, o = blockIdx.x & 1;
  const u32 row = rows_per_key == 4 ? 2 * in + o : o;
  key_coefficients(rows + ((size_t)key * rows_per_key + row) * N, coef, rc, rows_per_key == 2 && in ? AUTO_CUT : 0);
  for (int limb = 0; limb < LIMBS; limb++) {
    key_limb<LIMBS, LIMB_BITS>(coef, limb, dyn, tw);
    cplx *dst = out + (size_t)key * KEY_BLOCK + (size_t)(o * LIMBS + limb) * 2 * M;
    for (int e = threadIdx.x; e < M; e += 256) dst[(2 * eval_register(e) + in) * T + eval_thread(e)] = key_value(dyn, e);
  }
}

// ---------------------------------------------------------------------------
// The operations of a blind rotation.  A group of T threads transforms one
// polynomial at a time.
//   QUAD   a CTA of one group, four CTAs per SM: both forward transforms, then
//          for a and for b the three limbs of the key one after the other.
//   TRIO   a CTA of three groups, one for each limb, one CTA per SM: groups 0
//          and 1 transform the two digit polynomials, every group multiplies
//          both with its limb and transforms back (a, then b), and the groups'
//          parts are added up.  For batches that leave QUAD's places empty.
//   SPLIT  TRIO on a cluster of two CTAs, rank 0 for a and rank 1 for b: both
//          transform both digit polynomials, and the new digits go to both.
//          For batches that leave SMs idle.
// Shared memory: exchange buffers (M complex words; two per group, one in SPLIT) | what passes from an operation to the next: b or its digits
// (N words), a's digits (N ints) | SPLIT: the groups' next blocks of the
// key | twiddles | the schedule.  In TRIO and SPLIT the second part is
// there twice: an operation reads one and writes the other, while other threads
// may still be reading.  QUAD has no room for it: b (or its digits) sits in the
// exchange buffer that the last transform did not use, and is read before the
// operation's first barrier.
// Bounds: QUAD the FP64 pipe (49 % busy), issue (54 %) and four warps per
// scheduler, the register file being full; TRIO and SPLIT the barriers and fixed
// latencies between FP64 phases and integer ones.  With integer transforms 3552
// ciphertexts took 228 ms (QUAD 170), 148 took 13.3 (TRIO 8.6), one 10.1 (SPLIT
// 5.6).
// The key: QUAD loads it into registers, four CTAs covering for each other;
// TRIO early into more of them (each block while the digits or the output before
// are transformed); SPLIT has each block copied (cp.async.bulk) into shared
// memory as soon as the one before has been used, an operation ahead.
// ---------------------------------------------------------------------------
enum Form { QUAD, TRIO, SPLIT };
template <Form F>
struct Shape {
  static constexpr int GROUPS = F == QUAD ? 1 : LIMBS, THREADS = GROUPS * T, CTAS = F == QUAD ? 4 : 1;
  static constexpr size_t X_WORDS = (F == SPLIT ? 1 : 2) * GROUPS * 2 * M;
  static constexpr size_t PASS_WORDS = F == QUAD ? N / 2 : 2 * (N + N / 2);
  static constexpr size_t KEY_WORDS = F == SPLIT ? GROUPS * 4 * M : 0;
  static constexpr size_t WORDS = X_WORDS + PASS_WORDS + KEY_WORDS + 2 * TW_WORDS;
  // tensor memory: the transformed digit polynomials (64 columns), the turns
  // (32 per group), then QUAD: the permuted b of an automorphism until it is
  // added, TRIO and SPLIT: each group's part of each output (32 columns each)
  static constexpr u32 SPEC = 0, TURN = 64, PART = TURN + 32 * GROUPS, COLS = F == QUAD ? 128 : 512;
  static size_t smem_bytes(u32 br_q, u32 n) {
    return WORDS * 8 + (((size_t)4 + (n + br_q / 2 + 1) * 2 + 15) & ~(size_t)15);
  }
};
template <Form F>
struct Smem {
  typedef Shape<F> H;
  u64 *x;  // the groups' buffers
  __device__ __forceinline__ explicit Smem(u64 *s) : x(s) {}
  __device__ __forceinline__ cplx *buffer(int g, u32 q) const {
    return (cplx *)(x + (F == SPLIT ? (u32)g : 2 * g + q) * (2 * M));
  }
  __device__ __forceinline__ cplx *key(int g) const { return (cplx *)(x + H::X_WORDS + H::PASS_WORDS + g * 4 * M); }
  // what passes to operation i, before whose first transform the group's next buffer is q: an
  // automorphism's permuted b, or the digits of b; the digits of a
  __device__ __forceinline__ long long *ub(u32 i, u32 q) const {
    return F == QUAD ? (long long *)buffer(0, q ^ 1) : (long long *)(x + H::X_WORDS + (i & 1) * (N + N / 2));
  }
  __device__ __forceinline__ int *db(u32 i, u32 q) const { return (int *)ub(i, q); }
  __device__ __forceinline__ int *da(u32 i) const {
    return F == QUAD ? (int *)(x + H::X_WORDS) : (int *)(x + H::X_WORDS + (i & 1) * (N + N / 2) + N);
  }
  __device__ __forceinline__ cplx *tw() const { return (cplx *)(x + H::X_WORDS + H::PASS_WORDS + H::KEY_WORDS); }
  __device__ __forceinline__ u32 *nops() const { return (u32 *)(x + H::WORDS); }
  __device__ __forceinline__ unsigned short *ops() const { return (unsigned short *)(nops() + 1); }
};

namespace cg = cooperative_groups;
template <int V>
struct Int {
  static constexpr int value = V;
};
// Barrier of the CTA that also orders tensor memory between warps.
__device__ __forceinline__ void op_sync() {
  tmem_wait_store();
  tmem_before_barrier();
  __syncthreads();
  tmem_after_barrier();
}

// SPLIT's digits wait in their own order, those of coefficients t + T m and t +
// T (m + 1) for even m side by side, and an automorphism reads them permuted:
// what goes to the other CTA goes by 8-byte stores to neighbouring places (one
// gate 6.67 -> 6.01 ms against 4-byte stores to permuted ones; as bulk copies 6.16).
__device__ __forceinline__ int pair_place(int e) {
  const int m = e / T;
  return m / 2 * 2 * T + 2 * (e % T) + (m & 1);
}

// The digits of one polynomial (half 0: a's, or their low halves under an
// automorphism; half 1: b's, or the high halves of a's).
template <Form F>
__device__ __forceinline__ void load_digits(int (&v)[16], int half, u32 i, u32 q, bool is_auto, u32 k, const Smem<F> &S,
                                            const Place &p) {
  const int *d = half == 0 || is_auto ? S.da(i) : S.db(i, q);
  if (F != SPLIT) {
#pragma unroll
    for (int m = 0; m < 16; m++) v[m] = d[p.t + T * m];
  } else if (is_auto) {
    u32 inv = k * (2 - k * k);  // of k mod 2^6, then 2^12 = 2 N
    inv *= 2 - k * inv;
    u32 e = (u32)p.t * inv;
#pragma unroll
    for (int m = 0; m < 16; m++, e += T * inv) v[m] = d[pair_place(e & (N - 1))];
  } else {
#pragma unroll
    for (int m = 0; m < 16; m += 2) {
      const int2 x = ((const int2 *)d)[m / 2 * T + p.t];
      v[m] = x.x;
      v[m + 1] = x.y;
    }
  }
  if (is_auto) {
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int hi = (v[m] + (1 << (AUTO_CUT - 1))) >> AUTO_CUT;
      v[m] = half ? hi : v[m] - (hi << AUTO_CUT);
    }
  }
}
__device__ __forceinline__ void to_complex(cplx (&z)[8], const int (&v)[16]) {
#pragma unroll
  for (int m = 0; m < 16; m++) (m < 8 ? z[m & 7].r : z[m & 7].i) = i2d(v[m]);
}

// points r and r + 1: the transformed digits (tensor memory) times the keys
__device__ __forceinline__ void products(cplx (&z)[8], int r, u32 spec, const cplx &a0, const cplx &b0, const cplx &a1,
                                         const cplx &b1) {
  cplx u0, u1, v0, v1;
  tmem_load4(spec + 8 * r, u0, u1, v0, v1);
  z[r].r = fma(u0.r, a0.r, fma(-u0.i, a0.i, fma(v0.r, b0.r, -(v0.i * b0.i))));
  z[r].i = fma(u0.r, a0.i, fma(u0.i, a0.r, fma(v0.r, b0.i, v0.i * b0.r)));
  z[r + 1].r = fma(u1.r, a1.r, fma(-u1.i, a1.i, fma(v1.r, b1.r, -(v1.i * b1.i))));
  z[r + 1].i = fma(u1.r, a1.i, fma(u1.i, a1.r, fma(v1.r, b1.i, v1.i * b1.r)));
}

// What becomes of output o of an operation: `nx` (the next one, i + 1) reads
// digits, an automorphism X -> X^k those of a and b itself, permuted; after
// the last operation (OP_END) emit(o, c, v) gets coefficient c in [0, Q).
struct Next {
  bool end, is_auto;
  u32 k;
  __device__ __forceinline__ Next(u32 nx, const BrParams &P)
      : end(nx == OP_END), is_auto(!end && (nx & OP_AUTO)), k(is_auto ? P.auto_k[nx & OP_SLOT] : 1u) {}
};
// C values of output o: coefficients t + T (m0 + m), as sums of the limbs.  q:
// the group's next buffer after the operation.  far_bar: the other CTA's barrier
// for the digits sent there.
template <int C, Form F, class Emit>
__device__ __forceinline__ void pass_on(const u64 (&acc)[C], int m0, int o, u32 i, u32 q, const Next &nx,
                                        const Smem<F> &S, u32 far_bar, int rank, const Place &p, const Emit &emit) {
  long long c[C];
  u32 worst = 0, at = (u32)(p.t + T * m0) * nx.k;
#pragma unroll
  for (int m = 0; m < C; m++, at += T * nx.k) {
    c[m] = settle(acc[m]);
    if (at & N) c[m] = -c[m];  // X^N = -1
    worst = max(worst, edge(c[m]));
  }
  at = (u32)(p.t + T * m0) * nx.k;
  if (nx.end) {
#pragma unroll
    for (int m = 0; m < C; m++) {
      const long long v = centre(c[m]);
      emit(o, p.t + T * (m0 + m), (u64)(v < 0 ? v + (long long)Q_N2048 : v));
    }
  } else if (o == 1 && nx.is_auto) {
    long long *dst = S.ub(i + 1, q);
#pragma unroll
    for (int m = 0; m < C; m++, at += T * nx.k) dst[at & (N - 1)] = c[m];
  } else {
    if (worst > EDGE) {
#pragma unroll
      for (int m = 0; m < C; m++) c[m] = centre(c[m]);
    }
    // (c + half) >> 37 or 30, see digit()
    const long long half = nx.is_auto ? 1ll << (AUTO_IGN - 1) : 1ll << (RLRG_IGN - 1);
    const int more = nx.is_auto ? 0 : RLRG_IGN - AUTO_IGN;
    int *dst = o ? S.db(i + 1, q) : S.da(i + 1);
    auto digit_of = [&](long long v) { return (int)((v + half) >> AUTO_IGN) >> more; };
    if constexpr (F == SPLIT) {
      dst += 2 * (m0 / 2 * T + p.t);
      const u32 far = cluster_addr(dst, rank ^ 1);
#pragma unroll
      for (int m = 0; m < C; m += 2) {
        const int2 d = make_int2(digit_of(c[m]), digit_of(c[m + 1]));
        remote_store2(far + 4 * m * T, d.x, d.y, far_bar);
        *(int2 *)(dst + m * T) = d;
      }
    } else {
#pragma unroll
      for (int m = 0; m < C; m++, at += T * nx.k) dst[at & (N - 1)] = digit_of(c[m]);
    }
  }
}

// Operation i, `op`, on what S holds for it, leaving there what the next one
// reads.  q: the exchange buffer the group's next transform writes.  tm: this
// warp's tensor memory.  The bodies are kept small (one copy of each
// transform): with larger ones, two polynomials at a time, a third of the issue
// slots waited for instructions.
template <class Emit>
__device__ __forceinline__ void op_quad(u32 i, u32 op, u32 nx_op, const cplx *key, const cplx *next_key,
                                        const BrParams &P, const Smem<QUAD> &S, u32 &q, u32 tm, const Place &p,
                                        const Emit &emit) {
  typedef Shape<QUAD> H;
  const int t = p.t;
  const bool is_auto = (op & OP_AUTO) != 0;
  cplx z[8];
  {
    int y[16];
    load_digits(y, 0, i, q, is_auto, 1u, S, p);
    to_complex(z, y);
    load_digits(y, 1, i, q, is_auto, 1u, S, p);
    if (is_auto) {  // b, before its buffer is written
#pragma unroll
      for (int h = 0; h < 2; h++) {
        u64 b[8];
#pragma unroll
        for (int m = 0; m < 8; m++) b[m] = (u64)S.ub(i, q)[t + T * (8 * h + m)];
        tmem_store8(tm + H::PART + 16 * h, b);
      }
    }
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
      forward<H::GROUPS>(z, S.buffer(0, q), S.tw(), p);
      q ^= 1;
#pragma unroll
      for (int c = 0; c < 4; c++) tmem_store2(tm + H::SPEC + 16 * c + 8 * half, z[2 * c], z[2 * c + 1]);
      to_complex(z, y);
    }
    tmem_wait_store();
  }
  const Next nx(nx_op, P);
  const cplx *kp = key + t;
#pragma unroll 1
  for (int o = 0; o < 2; o++) {
    u64 acc[16];
#pragma unroll
    for (int m = 0; m < 16; m++) acc[m] = 0;
    if (o == 1 && is_auto) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        u64 b[8];
        tmem_load8(tm + H::PART + 16 * h, b);
#pragma unroll
        for (int m = 0; m < 8; m++) acc[8 * h + m] = b[m];
      }
    }
#pragma unroll 1
    for (int l = 0; l < LIMBS; l++) {
      // the next block of the key, into L2 while this one is worked on
      if (t == 0) {
        const cplx *nb = (o == 1 && l == LIMBS - 1) ? next_key : kp + 2 * M;
        if (nb) prefetch_l2(nb, 2 * M * (u32)sizeof(cplx));
      }
      cplx kx[2][2], ky[2][2];
      auto fetch = [&](int c) {  // the key at points 2 c and 2 c + 1
#pragma unroll
        for (int e = 0; e < 2; e++) {
          kx[c & 1][e] = ld_key(kp + (2 * (2 * c + e)) * T);
          ky[c & 1][e] = ld_key(kp + (2 * (2 * c + e) + 1) * T);
        }
      };
      fetch(0);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (c < 3) fetch(c + 1);
        products(z, 2 * c, tm + H::SPEC, kx[c & 1][0], ky[c & 1][0], kx[c & 1][1], ky[c & 1][1]);
      }
      kp += 2 * M;
      inverse<H::GROUPS>(z, S.buffer(0, q), S.tw(), p);
      q ^= 1;
      if (l == 0) {
#pragma unroll
        for (int m = 0; m < 16; m++) add_limb0(acc[m], m < 8 ? z[m & 7].r : z[m & 7].i);
      } else if (l == 1) {
#pragma unroll
        for (int m = 0; m < 16; m++) add_limb1(acc[m], m < 8 ? z[m & 7].r : z[m & 7].i);
      } else {
#pragma unroll
        for (int m = 0; m < 16; m++) add_limb2(acc[m], m < 8 ? z[m & 7].r : z[m & 7].i);
      }
    }
    // the operation's eight transforms leave q as it was; the next operation
    // starts with the other buffer
    pass_on(acc, 0, o, i, q ^ 1, nx, S, 0u, 0, p, emit);
  }
  q ^= 1;
}

// The waits of SPLIT, each bounded (BrParams::wait_limit, about a second).  One
// that runs out in operation i sets DEVERR_MBAR_TIMEOUT and makes operation i + 1
// the schedule's last: the whole CTA reads that at the top of i + 1, sends no more
// digits and leaves the ciphertexts after this one undone, whereupon the other
// CTA's waits run out too.  The results are not valid, but every barrier is met and
// what is in flight ends before the CTA does: a whole operation lies between the
// last digits that it sends and its end, and a group asks for no copy before it has
// waited for the last, which drain() does where a wait gave up.  (With `lost` read
// at each wait, copy and message, or once per operation, one gate took 3 to 6 %
// more.)
constexpr u32 GAVE_UP = 0x80000000u;
struct Waits {
  u64 *key;   // one per group: its block of the key has arrived
  u64 *msg;   // SPLIT, by parity of the operation: the other CTA's digits for it
  int *lost;  // shared: a wait ran out
  u32 *err;
  const long long *limit;    // shared
  u32 key_phase, msg_phase;  // completed phases (key: GAVE_UP and the first that is not; msg: bit per barrier)
  bool fresh;                // the item's first operation: no message
  int rank;
  __device__ __forceinline__ bool over() const { return *(volatile int *)lost != 0; }
  __device__ __forceinline__ void ran_out(u32 i, const Smem<SPLIT> &S) const {
    *(volatile int *)lost = 1;
    if (i + 2 < *S.nops()) S.ops()[i + 2] = OP_END;
    atomicOr(err, DEVERR_MBAR_TIMEOUT);
  }
  // the group's block of the key for operation i
  __device__ __forceinline__ void wait_key(u32 i, const Smem<SPLIT> &S, const Place &p) {
    if (!mbar_wait(key + p.g, key_phase & 1, *limit)) {
      ran_out(i, S);
      key_phase = (key_phase | GAVE_UP) - 1;
    }
    key_phase++;
  }
  // for the item's first operation
  __device__ __forceinline__ void first_key(const cplx *k, const Smem<SPLIT> &S, const Place &p) const {
    if (p.t == 0) {
      fence_proxy_async_smem();
      bulk_load(S.key(p.g), k + (size_t)(rank * LIMBS + p.g) * 2 * M, 2 * M * (u32)sizeof(cplx), key + p.g);
    }
  }
  __device__ __forceinline__ void drain(const Place &p) const {
    if (p.t == 0 && (key_phase & GAVE_UP)) mbar_wait(key + p.g, key_phase & 1);
  }
  // SPLIT, before operation i = the one whose parity `at` is: the other CTA's
  // digits.  Rank 0 sends a's digits for every operation, rank 1 b's for an
  // external product and one word for an automorphism, so that neither gets two
  // operations ahead.
  __device__ __forceinline__ void message(u32 i, u32 op, const Smem<SPLIT> &S) {
    const u32 b = i & 1;
    if (!fresh) {
      if (threadIdx.x == 0) mbar_expect(msg + b, rank == 1 || !(op & OP_AUTO) ? N * 4u : 4u);
      if (!mbar_wait_cluster(msg + b, (msg_phase >> b) & 1, *limit)) ran_out(i, S);
      msg_phase ^= 1u << b;
    }
    fresh = false;
  }
};

template <Form F, class Emit>
__device__ __forceinline__ void op_trio(u32 i, u32 op, u32 nx_op, Next &now, const cplx *key, const cplx *next_key,
                                        const BrParams &P, const Smem<F> &S, Waits &W, int rank, u32 &q, u32 tm,
                                        const Place &p, const Emit &emit) {
  typedef Shape<F> H;
  const int t = p.t, g = p.g;
  const bool is_auto = (op & OP_AUTO) != 0;
  Next nx = now;
  if (F == SPLIT) nx = Next(nx_op, P);
  // the next operation's key, into L2 while this one is worked on
  if (threadIdx.x == 0 && next_key) {
    if (F == SPLIT) prefetch_l2(next_key + (size_t)rank * LIMBS * 2 * M, LIMBS * 2 * M * (u32)sizeof(cplx));
    else prefetch_l2(next_key, (u32)(KEY_BLOCK * sizeof(cplx)));
  }
  cplx z[8];
  if (g < 2) {
    int v[16];
    load_digits(v, g, i, q, is_auto, now.k, S, p);
    to_complex(z, v);
  }
  // this group's limb of the key for the first output
  const cplx *kp = key + (size_t)g * 2 * M + t;
  cplx kx[8], ky[8];
  auto fetch = [&]() {
#pragma unroll
    for (int r = 0; r < 8; r++) {
      kx[r] = ld_key(kp + (2 * r) * T);
      ky[r] = ld_key(kp + (2 * r + 1) * T);
    }
  };
  // SPLIT: some of the block's points into registers while the digits are
  // transformed (the products would wait for all of it otherwise, 96 KB in 770
  // cycles: one gate 5.96 -> 5.78 ms together with the sums dealt out 6, 6 and 4;
  // of 2 to 5 points 3 are the fastest, 5.60 ms against 5.66 to 5.79)
  constexpr int EARLY = 3;
  const cplx *const sk = F == SPLIT ? S.key(g) + t : nullptr;
  auto take = [&]() {
    if constexpr (F == SPLIT) {
      W.wait_key(i, S, p);
#pragma unroll
      for (int r = 0; r < EARLY; r++) {
        kx[r] = sk[2 * r * T];
        ky[r] = sk[(2 * r + 1) * T];
      }
    }
  };
  if (F == TRIO) fetch();
  if (g < 2) {
    forward<H::GROUPS>(z, S.buffer(g, q), S.tw(), p, take);
    if (F == TRIO) q ^= 1;
#pragma unroll
    for (int c = 0; c < 4; c++) tmem_store2(tm + H::SPEC + 16 * c + 8 * g, z[2 * c], z[2 * c + 1]);
  } else {
    take();
  }
  op_sync();
#pragma unroll 1
  for (int o = F == SPLIT ? rank : 0; o < (F == SPLIT ? rank + 1 : 2); o++) {
    if constexpr (F == SPLIT) {
#pragma unroll
      for (int r = EARLY; r < 8; r++) {
        kx[r] = sk[2 * r * T];
        ky[r] = sk[(2 * r + 1) * T];
      }
#pragma unroll
      for (int r = 0; r < 8; r += 2) products(z, r, tm + H::SPEC, kx[r], ky[r], kx[r + 1], ky[r + 1]);
    } else {
#pragma unroll
      for (int r = 0; r < 8; r += 2) products(z, r, tm + H::SPEC, kx[r], ky[r], kx[r + 1], ky[r + 1]);
      if (o == 0) {
        kp += (size_t)LIMBS * 2 * M;
        fetch();
      }
    }
    if constexpr (F == SPLIT) {
      group_sync<H::GROUPS>(p);  // the exchange buffer and the block of the key have been used
      if (t == 0 && next_key && !(W.key_phase & GAVE_UP)) {  // (as a method of Waits: 5.60 -> 5.71 ms)
        fence_proxy_async_smem();
        bulk_load(S.key(g), next_key + (size_t)(rank * LIMBS + g) * 2 * M, 2 * M * (u32)sizeof(cplx), W.key + g);
      }
    }
    inverse<H::GROUPS>(z, S.buffer(g, q), S.tw(), p);
    if (F == TRIO) q ^= 1;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      u64 v[8];
#pragma unroll
      for (int m = 0; m < 8; m++) v[m] = 0;
      if (g == 0) {
#pragma unroll
        for (int m = 0; m < 8; m++) add_limb0(v[m], h ? z[m].i : z[m].r);
      } else if (g == 1) {
#pragma unroll
        for (int m = 0; m < 8; m++) add_limb1(v[m], h ? z[m].i : z[m].r);
      } else {
#pragma unroll
        for (int m = 0; m < 8; m++) add_limb2(v[m], h ? z[m].i : z[m].r);
      }
      tmem_store8(tm + H::PART + 32 * (3 * o + g) + 16 * h, v);
    }
  }
  op_sync();
  if (F == TRIO) nx = Next(nx_op, P);
  // the sums, dealt out to the groups: SPLIT values 0-5, 6-11, 12-15 of the
  // output (limb 2 takes its group longest), TRIO the 16 of a and then those of b, 12, 12 and 8
  const u32 far_bar = F == SPLIT ? cluster_addr(W.msg + ((i + 1) & 1), rank ^ 1) : 0;
  auto finish = [&](auto count, int o, int m0) {
    constexpr int C = decltype(count)::value;
    u64 acc[C];
    tmem_sum3<C>(tm + H::PART + 32 * 3 * o + 2 * m0, acc);
    if (o == 1 && is_auto) {
#pragma unroll
      for (int m = 0; m < C; m++) acc[m] += (u64)S.ub(i, q)[t + T * (m0 + m)];
    }
    pass_on(acc, m0, o, i, q, nx, S, far_bar, rank, p, emit);
  };
  if (F == SPLIT) {
    if (g < 2) finish(Int<6>(), rank, 6 * g);
    else finish(Int<4>(), rank, 12);
    if (rank == 1 && nx.is_auto && threadIdx.x == 0) remote_store(cluster_addr(S.db(i + 1, q), 0), 0, far_bar);
  } else {
#pragma unroll 1
    for (int u = 3 * g; u < min(3 * g + 3, 8); u++) finish(Int<4>(), u >> 2, 4 * (u & 3));
  }
  now = nx;
}

__device__ __forceinline__ const cplx *op_key(const BrParams &P, u32 op) {
  return (op & OP_AUTO) ? (const cplx *)P.fft_autos + (size_t)(op & OP_SLOT) * KEY_BLOCK
                        : (const cplx *)P.fft_rgsw + (size_t)(op & OP_INDEX) * KEY_BLOCK;
}

// One gate bootstrap.
template <Form F>
__device__ __forceinline__ void fft_item(const BrParams &P, int ct, const u32 *kso, u32 gcode, u64 *out, u64 *rlwe_dbg,
                                         u64 *smem, Waits &W, int rank, u32 tm) {
  typedef Shape<F> H;
  const Smem<F> S(smem);
  const Place p(threadIdx.x % T, threadIdx.x / T, tm + H::TURN + 32 * (threadIdx.x / T));
  // the bucket arrays are only needed while the schedule is built: they, like
  // its scratch (the first 2 N words), share the exchange buffers; of the first
  // N words the counters and keys take less than 10 KB, and QUAD has the
  // buckets' starts and members behind them
  SchedSmem sched;
  sched.start = (unsigned short *)(F == QUAD ? smem + 1280 : smem + 2 * N);
  sched.list = sched.start + (P.br_q >> 1) + 1;
  sched.ops = S.ops();
  sched.nops = S.nops();
  build_schedule<11, H::THREADS>(P, kso, smem, sched);
  __syncthreads();
  const unsigned short *ops = S.ops();
  const u32 nops = *S.nops();
  u32 i = 0, q = 0;
  {
    // b: the rotated test polynomial, and the automorphisms of the trivial
    // RLWE (runtime.rs:625-642), which only permute it; a = 0
    long long *from = (long long *)smem, *to = from + N;
    const TestRotation tr(P, kso, gcode);
#pragma unroll 1
    for (int c = threadIdx.x; c < N; c += H::THREADS) from[c] = (long long)tr.at((u32)c);
#pragma unroll 1
    for (; ops[i] & OP_AUTO; i++) {
      const u32 k = P.auto_k[ops[i] & OP_SLOT];
      __syncthreads();
#pragma unroll 1
      for (int c = threadIdx.x; c < N; c += H::THREADS) {
        const u32 at = (u32)c * k;
        to[at & (N - 1)] = (at & N) ? -from[c] : from[c];
      }
      long long *const x = from;
      from = to;
      to = x;
    }
    __syncthreads();
    constexpr int PER = (N + H::THREADS - 1) / H::THREADS;
    int d[PER];
#pragma unroll
    for (int m = 0; m < PER; m++) {
      const int c = threadIdx.x + H::THREADS * m;
      if (c < N) d[m] = digit<RLRG_IGN>(centre(from[c]));
    }
    if (F == QUAD) __syncthreads();  // b's digits go where b was, or beside it
#pragma unroll
    for (int m = 0; m < PER; m++) {
      const int c = threadIdx.x + H::THREADS * m;
      if (c < N) {
        S.db(i, q)[F == SPLIT ? pair_place(c) : c] = d[m];
        S.da(i)[c] = 0;
      }
    }
  }
  u64 *dst = out + (size_t)(P.out_idx ? P.out_idx[ct] : (u32)ct) * (N + 1);
  auto emit = [&](int o, int c, u64 v) {
    // sample extract at index 0 (pbs.rs:423-449)
    if (o == 0) dst[c == 0 ? 1 : 1 + N - c] = c == 0 ? v : Q_N2048 - v;
    else if (c == 0) dst[0] = v;
    if (rlwe_dbg) rlwe_dbg[((size_t)ct * 2 + o) * N + c] = v;
  };
  if constexpr (F == SPLIT) {
    const bool over = W.over();  // uniform: the last item's waits are behind a barrier
    __syncthreads();  // the barriers are there; the last item's blocks have been used
    if (!over) W.first_key(op_key(P, ops[i]), S, p);
    cg::this_cluster().sync();  // the other CTA is ready for what it is sent, too
    if (over) return;
  }
  W.fresh = true;
  u32 op = ops[i];
  Next now(op, P);
#pragma unroll 1
  for (; F == SPLIT ? op != OP_END : i < nops; i++) {  // (TRIO by the first: 8.55 -> 8.60 ms)
    const u32 nx_op = i + 1 < nops ? ops[i + 1] : OP_END;
    const cplx *key = op_key(P, op), *next_key = nx_op != OP_END ? op_key(P, nx_op) : nullptr;
    if constexpr (F == SPLIT) W.message(i, op, S);
    op_sync();
    if constexpr (F == QUAD) op_quad(i, op, nx_op, key, next_key, P, S, q, tm, p, emit);
    else op_trio(i, op, nx_op, now, key, next_key, P, S, W, rank, q, tm, p, emit);
    op = nx_op;
  }
}

// Tensor memory of the CTA: this warp's address of its lanes.
template <Form F>
__device__ __forceinline__ u32 tmem_begin(u32 *slot) {
  if (threadIdx.x < 32) tmem_alloc<Shape<F>::COLS>(slot);
  __syncthreads();
  return *slot + (((threadIdx.x >> 5) & 3) << 21);  // lane 32 (w mod 4) in bits 16 and up
}
template <Form F>
__device__ __forceinline__ void tmem_end(u32 *slot) {
  __syncthreads();
  if (threadIdx.x < 32) tmem_free<Shape<F>::COLS>(*slot);
}

// Ciphertexts [begin, end) of a batch (gates of one key; descs and item_desc
// null), or of a ragged one: ciphertext ct uses the parameter set and server key of descriptor
// item_desc[ct] and its output goes to out_idx[ct].  SPLIT: launched in
// clusters of two, both on the same items.
template <Form F>
__global__ void __launch_bounds__(Shape<F>::THREADS, Shape<F>::CTAS)
    pbs_fft_kernel(const __grid_constant__ BrParams P, const BrParams *descs, const u32 *item_desc, const u32 *out_idx,
                   const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out, int begin, int end,
                   u64 *rlwe_dbg) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ BrParams sp;
  __shared__ u32 tmem_slot;
  const u32 tm = tmem_begin<F>(&tmem_slot);
  const int rank = F == SPLIT ? (int)cg::this_cluster().block_rank() : 0;
  __shared__ u64 bars[5];
  __shared__ int lost;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 5; b++) mbar_init(bars + b, 1);
    lost = 0;
    mbar_init_fence();
  }
  Waits W{bars, bars + 3, &lost, nullptr, &sp.wait_limit, 0, 0, false, rank};
  const int step = F == SPLIT ? gridDim.x / 2 : gridDim.x;
  const int first = begin + (int)(F == SPLIT ? blockIdx.x / 2 : blockIdx.x);
  for (int ct = first; ct < end; ct += step) {
    __syncthreads();  // the previous item is done with sp
    if (threadIdx.x == 0) {
      sp = descs ? descs[item_desc[ct]] : P;
      if (descs) sp.out_idx = out_idx;
    }
    __syncthreads();
    if (ct == first) {
      cplx *tw = Smem<F>(smem).tw();
      for (int i = threadIdx.x; i < TW_WORDS; i += Shape<F>::THREADS) tw[i] = ldc((const cplx *)sp.fft_tw + i);
    }
    W.err = sp.err;
    fft_item<F>(sp, ct, ks + (size_t)ct * ks_stride, gates[ct], out, rlwe_dbg, smem, W, rank, tm);
  }
  if constexpr (F == SPLIT) {
    W.drain(Place(threadIdx.x % T, threadIdx.x / T, 0));
    cg::this_cluster().sync();  // nobody leaves while the other may still send
  }
  tmem_end<F>(&tmem_slot);
}

// External products (AUTO: automorphisms) by themselves: one operation per
// ciphertext, QUAD's, CTAs taking ciphertexts in turn (bound like it; 4096
// products of I_2P 283 us with integer transforms -> 228).  An index out of range
// leaves its ciphertext unchanged.  Inputs need not be canonical: the digits
// are the decomposer's for any word.
template <bool AUTO>
__global__ void __launch_bounds__(T, 4)
    op_fft_kernel(const __grid_constant__ BrParams P, u64 *rlwe, const u32 *idx, size_t count, int trivial) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u32 tmem_slot;
  const u32 tm = tmem_begin<QUAD>(&tmem_slot);
  const Smem<QUAD> S(smem);
  const int t = threadIdx.x;
  const Place p(t, 0, tm + Shape<QUAD>::TURN);
  for (int i = t; i < TW_WORDS; i += T) S.tw()[i] = ldc((const cplx *)P.fft_tw + i);
  u32 q = 0;
  for (size_t c = blockIdx.x; c < count; c += gridDim.x) {
    const u32 i = idx[c];
    if (AUTO ? i > P.w : i >= P.n) continue;  // uniform
    const u32 op = AUTO ? OP_AUTO | i : i;
    const cplx *key = op_key(P, op);
    if (t == 0) prefetch_l2(key, 2 * M * (u32)sizeof(cplx));
    u64 *x = rlwe + c * 2 * N;
    __syncthreads();  // the last ciphertext's use of S
    int *da = S.da(0), *db = S.db(0, q);
    long long *ub = S.ub(0, q);
    if (AUTO) {
      u32 at = (u32)t * P.auto_k[i];
#pragma unroll
      for (int m = 0; m < 16; m++, at += T * P.auto_k[i]) {
        const u64 a = x[t + T * m];
        const long long b = (long long)reduce_n2048(x[N + t + T * m]);
        da[at & (N - 1)] = digit_any<AUTO_LOGB, AUTO_IGN>((at & N) ? Q_N2048 - a : a);
        ub[at & (N - 1)] = (at & N) ? -b : b;
      }
    } else {
#pragma unroll
      for (int m = 0; m < 16; m++) {
        da[t + T * m] = trivial ? 0 : digit_any<RLRG_LOGB, RLRG_IGN>(x[t + T * m]);  // a = 0 (runtime.rs:790)
        db[t + T * m] = digit_any<RLRG_LOGB, RLRG_IGN>(x[N + t + T * m]);
      }
    }
    op_sync();
    op_quad(0, op, OP_END, key, nullptr, P, S, q, tm, p, [&](int o, int e, u64 v) { x[o * N + e] = v; });
  }
  tmem_end<QUAD>(&tmem_slot);
}

}  // namespace fft

using fft::cplx;

cudaError_t fft_tables(void **out) {
  std::vector<double> h((size_t)fft::TW_WORDS * 2 + 4 * 1024, 0.0);
  std::vector<long double> phi(1024);
  phi[1] = 0.125L;
  for (int i = 1; i < 512; i++) {
    phi[2 * i] = phi[i] / 2;
    phi[2 * i + 1] = phi[i] / 2 + 0.25L;
  }
  const long double two_pi = 6.283185307179586476925286766559005768L;
  double *full = h.data() + (size_t)fft::TW_WORDS * 2;  // y(s, k) at (1 << s) + k, hi and lo parts
  for (int i = 1; i < 1024; i++) {
    const long double c = cosl(two_pi * phi[i]), s = sinl(two_pi * phi[i]);
    full[4 * i] = (double)c;
    full[4 * i + 1] = (double)(c - (long double)(double)c);
    full[4 * i + 2] = (double)s;
    full[4 * i + 3] = (double)(s - (long double)(double)s);
  }
  auto put = [&](int at, int level, int k) {
    h[2 * at] = full[4 * ((1 << level) + k)];
    h[2 * at + 1] = full[4 * ((1 << level) + k) + 2];
  };
  for (int b = 0; b < 8; b++) {
    put(fft::TW_R1 + b, 3, b);
    put(fft::TW_R1 + 8 + b, 4, 2 * b);
    put(fft::TW_R1 + 16 + b, 5, 4 * b);
    put(fft::TW_R1 + 24 + b, 5, 4 * b + 2);
  }
  for (int b = 0; b < 32; b++) {
    put(fft::TW_R2 + b, 6, 2 * b);
    put(fft::TW_R2 + 32 + b, 7, 4 * b);
    put(fft::TW_R2 + 64 + b, 7, 4 * b + 2);
  }
  for (int t = 0; t < 128; t++) {
    for (int p4 = 0; p4 < 2; p4++) {
      const int node = ((t >> 5) << 6) | (((t >> 2) & 7) << 3) | (p4 << 2) | (t & 3);
      put(fft::TW_R3 + 256 * p4 + t, 8, node);
      put(fft::TW_R3 + 256 * p4 + 128 + t, 9, 2 * node);
    }
  }
  void *d = nullptr;
  cudaError_t e = dev_malloc(&d, h.size() * 8);
  if (e == cudaSuccess) e = cudaMemcpy(d, h.data(), h.size() * 8, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    d = nullptr;
  }
  *out = d;
  return e;
}

size_t fft_key_bytes(size_t keys) { return keys * fft::KEY_BLOCK * sizeof(cplx); }

cudaError_t launch_fft_key(const u64 *rows, u32 rows_per_key, size_t keys, const RingConsts &rc, const void *tables,
                           void *out, cudaStream_t s) {
  if (keys == 0) return cudaSuccess;
  const double4 *tw = (const double4 *)((const cplx *)tables + fft::TW_WORDS);
  fft::fft_key_kernel<<<(unsigned)(4 * keys), 256, fft::KEY_SMEM, s>>>(rows, (cplx *)out, rows_per_key, rc, tw);
  return cudaGetLastError();
}

// From the resources: the occupancy calculator answers one CTA per SM for every
// kernel that allocates tensor memory, and four run (592 ciphertexts take 30.3 ms,
// 148 take 15.1).
cudaError_t pbs_fft_per_sm(u32 br_q, u32 n, int *ctas) {
  typedef fft::Shape<fft::QUAD> H;
  const size_t smem = H::smem_bytes(br_q, n);
  cudaFuncAttributes a;
  int dev = 0, shared = 0, reserved = 0, regs = 0;
  cudaError_t e = cudaFuncGetAttributes(&a, fft::pbs_fft_kernel<fft::QUAD>);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&shared, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&regs, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  if (e != cudaSuccess) return e;
  const size_t by_shared = (size_t)shared / (smem + a.sharedSizeBytes + reserved);
  const size_t by_regs = (size_t)regs / ((size_t)std::max(a.numRegs, 1) * H::THREADS);
  *ctas = (int)std::min({by_shared, by_regs, (size_t)(512 / H::COLS)});
  return cudaSuccess;
}

struct Batch {  // the arguments of pbs_fft_kernel
  const BrParams &P;
  const BrParams *descs;
  const u32 *item_desc, *out_idx, *ks;
  u32 ks_stride;
  const unsigned char *gates;
  u64 *out, *rlwe_dbg;
  u32 br_q, n;  // the largest of the batch
};
// The launch of `grid` CTAs (SPLIT: clusters) of form F, its attribute in attr.
template <fft::Form F>
static cudaError_t form_config(u32 br_q, u32 n, int grid, cudaStream_t s, cudaLaunchConfig_t *cfg,
                               cudaLaunchAttribute *attr) {
  typedef fft::Shape<F> H;
  const size_t smem = H::smem_bytes(br_q, n);
  *cfg = {};
  cfg->gridDim = dim3((unsigned)(F == fft::SPLIT ? 2 * grid : grid));
  cfg->blockDim = dim3(H::THREADS);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim = {2, 1, 1};
  cfg->attrs = attr;
  cfg->numAttrs = F == fft::SPLIT ? 1 : 0;
  return opt_in_smem((const void *)fft::pbs_fft_kernel<F>, smem);
}
template <fft::Form F>
static cudaError_t launch_form(const Batch &b, size_t begin, size_t end, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  cudaError_t e = form_config<F>(b.br_q, b.n, grid, s, &cfg, attr);
  if (e != cudaSuccess) return e;
  e = cudaLaunchKernelEx(&cfg, fft::pbs_fft_kernel<F>, b.P, b.descs, b.item_desc, b.out_idx, b.ks, b.ks_stride, b.gates,
                         b.out, (int)begin, (int)end, b.rlwe_dbg);
  return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t pbs_fft_clusters(u32 br_q, u32 n, size_t *clusters) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int m = 0;
  cudaError_t e = form_config<fft::SPLIT>(br_q, n, 1, nullptr, &cfg, attr);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&m, fft::pbs_fft_kernel<fft::SPLIT>, &cfg);
  *clusters = (size_t)std::max(m, 1);
  return e;
}
static cudaError_t launch_form(fft::Form form, const Batch &b, size_t begin, size_t end, int grid, cudaStream_t s) {
  switch (form) {
    case fft::SPLIT: return launch_form<fft::SPLIT>(b, begin, end, grid, s);
    case fft::TRIO: return launch_form<fft::TRIO>(b, begin, end, grid, s);
    default: return launch_form<fft::QUAD>(b, begin, end, grid, s);
  }
}

// The forms by batch size.  NI_8P on 148 SMs, ms: SPLIT 5.6 for up to 74
// ciphertexts; TRIO 8.6 for up to 148 and again for each 148 more; QUAD 15.1,
// 18.9, 24.2 and 30.3 for up to 148, 296, 444 and 592, and from there 28.3 per
// 592, but 39.6 for 600 (the last few take as long as on an idle GPU).  So,
// with as many CTAs as ciphertexts:
//   up to 148     SPLIT (if asked for) or TRIO
//   up to 222     148 in TRIO, the rest in SPLIT (180: 18.8 -> 14.1)
//   up to 296     TRIO (18.9 -> 16.9)
//   up to 370     296 in TRIO, the rest in SPLIT (300: 23.9 -> 22.5)
//   more          QUAD; of more than 592, up to 74 or 148 above a multiple of 592
//                 go by themselves, in SPLIT or TRIO (600: 39.6 -> 36.0)
// With fewer CTAs (a limited grid) the form by their number.
static cudaError_t launch_fft(const Batch &b, size_t count, int grid, bool split, cudaStream_t s) {
  int dev = 0, sm = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
  const size_t sms = (size_t)sm, half = sms / 2;
  if (split) return launch_form(fft::SPLIT, b, 0, count, grid, s);
  if ((size_t)grid < count || count <= sms || b.rlwe_dbg)
    return launch_form((size_t)grid <= sms ? fft::TRIO : fft::QUAD, b, 0, count, grid, s);
  const fft::Form form = count <= 2 * sms + half ? fft::TRIO : fft::QUAD;
  const size_t wave = form == fft::TRIO ? sms : 4 * sms, over = count % wave;
  const bool peel = count > wave && over > 0 && over <= (form == fft::TRIO ? half : sms);
  const size_t whole = peel ? count - over : count;
  const cudaError_t e = launch_form(form, b, 0, whole, (int)whole, s);
  if (e != cudaSuccess || !peel) return e;
  return launch_form(over <= half ? fft::SPLIT : fft::TRIO, b, whole, count, (int)over, s);
}

// By the table above, full rounds of QUAD take 0.048 ms per ciphertext.  What fills
// up places for less is worth adding: to 148 (from 74 on two SMs 0.041), from
// there to 296 (0.056, but 148 to 222 0.074), from 296 to 592 (0.045), and above
// whole rounds to 148 (0.058; 74 on two SMs 0.076).  The integer kernels: rounds of
// three per SM, and whole SMs below.
size_t pbs_fill(size_t count, size_t sms, bool fft) {
  auto up = [](size_t x, size_t step) { return std::max<size_t>(1, (x + step - 1) / step) * step; };
  const size_t round = (fft ? 4 : 3) * sms;
  if (count <= (fft ? 2 * sms : round)) return up(count, sms);
  const size_t over = count % round;
  return fft && count > round && over > 0 && over <= sms ? count - over + sms : up(count, round);
}

cudaError_t launch_pbs_fft(const BrParams &P, const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out,
                           size_t count, u64 *rlwe_dbg, int grid, cudaStream_t s, bool split) {
  const Batch b{P, nullptr, nullptr, nullptr, ks, ks_stride, gates, out, rlwe_dbg, P.br_q, P.n};
  return launch_fft(b, count, grid, split, s);
}

cudaError_t launch_pbs_fft_ragged(const BrParams *d_descs, const u32 *item_desc, u32 max_br_q, u32 max_n, const u32 *ks,
                                  u32 ks_stride, const unsigned char *gates, u64 *out, const u32 *out_idx,
                                  size_t count, int grid, cudaStream_t s, bool split) {
  const BrParams none{};
  const Batch b{none, d_descs, item_desc, out_idx, ks, ks_stride, gates, out, nullptr, max_br_q, max_n};
  return launch_fft(b, count, grid, split, s);
}

template <bool AUTO>
static cudaError_t launch_op(const BrParams &P, u64 *rlwe, const u32 *idx, size_t count, int trivial, cudaStream_t s) {
  constexpr size_t smem = fft::Shape<fft::QUAD>::WORDS * 8;
  const cudaError_t e = opt_in_smem((const void *)fft::op_fft_kernel<AUTO>, smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned grid = (unsigned)std::min<size_t>(count, (size_t)4 * sms);
  fft::op_fft_kernel<AUTO><<<grid, fft::T, smem, s>>>(P, rlwe, idx, count, trivial);
  return cudaGetLastError();
}
cudaError_t launch_fft_product(const BrParams &P, u64 *rlwe, const u32 *idx, size_t count, int trivial,
                               cudaStream_t s) {
  return launch_op<false>(P, rlwe, idx, count, trivial, s);
}
cudaError_t launch_fft_auto(const BrParams &P, u64 *rlwe, const u32 *slot, size_t count, cudaStream_t s) {
  return launch_op<true>(P, rlwe, slot, count, 0, s);
}

}  // namespace pz
