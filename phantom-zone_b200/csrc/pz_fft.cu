// pz_fft.cu -- the blind rotation, external product and automorphism of the
// N = 2048 one-digit parameter sets over exact FP64 FFT products (pz_fft.cuh).
#include <algorithm>
#include <cmath>
#include <vector>

#include "pz_blind.cuh"
#include "pz_fft.cuh"
#include "pz_internal.h"

namespace pz {
namespace fft {

constexpr int N = 2048;
constexpr u32 OP_END = 0xffffffffu;

// ---------------------------------------------------------------------------
// Key form: the device rows (evaluation domain, K N^{-1}) back to
// coefficients, cut into limbs, and each limb transformed in double-double
// arithmetic, scaled by 1 / M (exact) and rounded once.
// ---------------------------------------------------------------------------
struct dd {
  double h, l;
};
__device__ __forceinline__ dd dd_norm(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
  const double s = a.h + b.h, bb = s - a.h;
  const double e = (a.h - (s - bb)) + (b.h - bb);
  return dd_norm(s, e + (a.l + b.l));
}
__device__ __forceinline__ dd dd_neg(dd a) { return {-a.h, -a.l}; }
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
  const double p = a.h * b.h;
  const double e = fma(a.h, b.h, -p);
  return dd_norm(p, e + (a.h * b.l + a.l * b.h));
}

// One CTA per (key block, row).  rows_per_key device rows per key: 4 for RGSW
// (A(-sm), B(-sm), A(m), B(m)), 2 for automorphism keys (A, B), whose second
// digit half uses 2^AUTO_CUT times the row.
__global__ void __launch_bounds__(256)
    fft_key_kernel(const u64 *rows, cplx *out, u32 rows_per_key, RingConsts rc, const double4 *tw) {
  __shared__ u64 coef[N];
  extern __shared__ double dyn[];
  double *re_h = dyn, *re_l = dyn + M, *im_h = dyn + 2 * M, *im_l = dyn + 3 * M;
  const int j = threadIdx.x;
  const u32 key = blockIdx.x >> 2, in = (blockIdx.x >> 1) & 1, o = blockIdx.x & 1;
  const u32 row = rows_per_key == 4 ? 2 * in + o : o;
  const u64 *src = rows + ((size_t)key * rows_per_key + row) * N;
  u64 x[8];
#pragma unroll
  for (int r = 0; r < 8; r++) x[r] = src[dev_index<11>(j, r)];
  ntt_inv<11>(x, coef, rc);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; r++) {
    u64 v = reduce2(x[r], Q_N2048);
    if (rows_per_key == 2 && in)  // 2^12 v mod Q
      v = reduce2(reduce_n2048(((v & ((1ull << (54 - AUTO_CUT)) - 1)) << AUTO_CUT) + 77823ull * (v >> (54 - AUTO_CUT))),
                  Q_N2048);
    coef[pos_coef<11>(j, r)] = v;
  }
  for (int limb = 0; limb < LIMBS; limb++) {
    __syncthreads();
    auto cut = [&](u64 u) -> double {
      long long v = u > (Q_N2048 >> 1) ? (long long)(u - Q_N2048) : (long long)u;
      long long k = 0;
      for (int l = 0; l <= limb; l++) {
        k = l + 1 < LIMBS ? ((v + (1 << (LIMB_BITS - 1))) & ((1 << LIMB_BITS) - 1)) - (1 << (LIMB_BITS - 1)) : v;
        v = (v - k) >> LIMB_BITS;
      }
      return (double)k;
    };
    for (int e = j; e < M; e += 256) {
      re_h[e] = cut(coef[e]);
      im_h[e] = cut(coef[e + M]);
      re_l[e] = im_l[e] = 0;
    }
    for (int s = 0; s < 10; s++) {
      const int half = M >> (s + 1);
      __syncthreads();
      for (int e = j; e < M / 2; e += 256) {
        const int k = e / half, a = k * 2 * half + e % half, b = a + half;
        const double4 w = tw[(1 << s) + k];  // y(s, k): re hi, re lo, im hi, im lo
        const dd wr{w.x, w.y}, wi{w.z, w.w};
        const dd ar{re_h[a], re_l[a]}, ai{im_h[a], im_l[a]}, br{re_h[b], re_l[b]}, bi{im_h[b], im_l[b]};
        const dd tr = dd_add(dd_mul(wr, br), dd_neg(dd_mul(wi, bi)));
        const dd ti = dd_add(dd_mul(wr, bi), dd_mul(wi, br));
        const dd pr = dd_add(ar, tr), pi = dd_add(ai, ti), mr = dd_add(ar, dd_neg(tr)), mi = dd_add(ai, dd_neg(ti));
        re_h[a] = pr.h; re_l[a] = pr.l; im_h[a] = pi.h; im_l[a] = pi.l;
        re_h[b] = mr.h; re_l[b] = mr.l; im_h[b] = mi.h; im_l[b] = mi.l;
      }
    }
    __syncthreads();
    cplx *dst = out + (size_t)key * KEY_BLOCK + (size_t)(o * LIMBS + limb) * 2 * M;
    for (int e = j; e < M; e += 256) {  // evaluation position e, layout E
      const int t = ((e >> 8) << 5) | (((e >> 5) & 7) << 2) | ((e >> 2) & 3), r = (((e >> 4) & 1) << 2) | (e & 3);
      dst[(2 * r + in) * T + t] = cplx{re_h[e] * (1.0 / M), im_h[e] * (1.0 / M)};
    }
  }
}

// ---------------------------------------------------------------------------
// The operations of a blind rotation, on a CTA of T threads.
// Shared memory: two exchange buffers (M complex words each) | a's digits (N
// ints) | twiddles | the schedule.  Between an operation and the next, b's
// digits (N ints) or the permuted b of an automorphism (N words) sit in the
// exchange buffer that the last transform did not use.
// ---------------------------------------------------------------------------
constexpr size_t X_WORDS = 4 * M, DA_WORDS = N / 2, TWS_WORDS = 2 * TW_WORDS;
constexpr size_t FFT_WORDS = X_WORDS + DA_WORDS + TWS_WORDS;
struct Smem {
  u64 *x;  // the buffers
  int *da;
  cplx *tw;
  unsigned short *ops;
  u32 *nops;
  __device__ __forceinline__ explicit Smem(u64 *s)
      : x(s), da((int *)(s + X_WORDS)), tw((cplx *)(s + X_WORDS + DA_WORDS)),
        ops((unsigned short *)(s + FFT_WORDS) + 2), nops((u32 *)(s + FFT_WORDS)) {}
  __device__ __forceinline__ u64 *buffer(u32 q) const { return x + q * (2 * M); }
};
static size_t fft_smem_bytes(u32 br_q, u32 n) {
  return FFT_WORDS * 8 + (((size_t)4 + (n + br_q / 2 + 1) * 2 + 15) & ~(size_t)15);
}
__device__ __forceinline__ void load_twiddles(const BrParams &P, const Smem &S) {
  for (int i = threadIdx.x; i < TW_WORDS; i += T) S.tw[i] = ldc((const cplx *)P.fft_tw + i);
}

// One operation `op` on what S holds for it, leaving there what the next one,
// `nx`, reads: the digits of both polynomials for an external product; a's
// digits and b, both under X -> X^k, for an automorphism; after the last
// operation (OP_END) emit(o, i, v) gets coefficient i of output o (0: a, 1: b)
// in [0, Q).  q: the buffer the next transform writes (b is in the other one).
// tm: this warp's tensor memory.
// The body is kept small (one copy of each transform): larger forms, with two
// polynomials at a time, spent a third of their issue slots waiting for
// instructions.
template <class Emit>
__device__ __forceinline__ void fft_op(u32 op, u32 nx, const cplx *key, const cplx *next_key, const BrParams &P,
                                       const Smem &S, u32 &q, u32 tm, const Place &p,
                                       const Emit &emit) {
  const int t = p.t;
  const bool is_auto = (op & OP_AUTO) != 0;
  cplx z[8];
  {
    int y[16];
    if (is_auto) {
      const u64 *ub = S.buffer(q ^ 1);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        u64 b[8];
#pragma unroll
        for (int m = 0; m < 8; m++) b[m] = ub[t + T * (8 * h + m)];
        tmem_store8(tm + SPEC_COLS + 16 * h, b);
      }
#pragma unroll
      for (int m = 0; m < 16; m++) {
        const int d = S.da[t + T * m];
        y[m] = (d + (1 << (AUTO_CUT - 1))) >> AUTO_CUT;
        (m < 8 ? z[m & 7].r : z[m & 7].i) = i2d(d - (y[m] << AUTO_CUT));
      }
    } else {
      const int *db = (const int *)S.buffer(q ^ 1);
#pragma unroll
      for (int m = 0; m < 16; m++) {
        (m < 8 ? z[m & 7].r : z[m & 7].i) = i2d(S.da[t + T * m]);
        y[m] = db[t + T * m];
      }
    }
#pragma unroll 1
    for (int i = 0; i < 2; i++) {
      forward(z, (cplx *)S.buffer(q), S.tw, p);
      q ^= 1;
#pragma unroll
      for (int c = 0; c < 4; c++) tmem_store2(tm + 16 * c + 8 * i, z[2 * c], z[2 * c + 1]);
#pragma unroll
      for (int m = 0; m < 16; m++) (m < 8 ? z[m & 7].r : z[m & 7].i) = i2d(y[m]);
    }
    tmem_wait_store();
  }
  const bool end = nx == OP_END, nx_auto = !end && (nx & OP_AUTO);
  const u32 k = nx_auto ? P.auto_k[nx & OP_SLOT] : 1u;
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
        tmem_load8(tm + SPEC_COLS + 16 * h, b);
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
        cplx px[2], py[2];
        tmem_load4(tm + 16 * c, px[0], px[1], py[0], py[1]);
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const cplx &u = px[e], &v = py[e], &a = kx[c & 1][e], &b = ky[c & 1][e];
          z[2 * c + e].r = fma(u.r, a.r, fma(-u.i, a.i, fma(v.r, b.r, -(v.i * b.i))));
          z[2 * c + e].i = fma(u.r, a.i, fma(u.i, a.r, fma(v.r, b.i, v.i * b.r)));
        }
      }
      kp += 2 * M;
      inverse(z, (cplx *)S.buffer(q), S.tw, p);
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
    long long c[16];
    u32 worst = 0, at = (u32)t * k;
#pragma unroll
    for (int m = 0; m < 16; m++, at += T * k) {
      c[m] = settle(acc[m]);
      if (at & N) c[m] = -c[m];  // X^N = -1
      worst = max(worst, edge(c[m]));
    }
    at = (u32)t * k;
    if (end) {
#pragma unroll
      for (int m = 0; m < 16; m++) {
        const long long v = centre(c[m]);
        emit(o, t + T * m, (u64)(v < 0 ? v + (long long)Q_N2048 : v));
      }
    } else if (o == 1 && nx_auto) {
      long long *dst = (long long *)S.buffer(q);
#pragma unroll
      for (int m = 0; m < 16; m++, at += T * k) dst[at & (N - 1)] = c[m];
    } else {
      if (worst > EDGE) {
#pragma unroll
        for (int m = 0; m < 16; m++) c[m] = centre(c[m]);
      }
      // (c + half) >> 37 or 30, see digit()
      const long long half = nx_auto ? 1ll << (AUTO_IGN - 1) : 1ll << (RLRG_IGN - 1);
      const int more = nx_auto ? 0 : RLRG_IGN - AUTO_IGN;
      int *dst = o ? (int *)S.buffer(q) : S.da;
#pragma unroll
      for (int m = 0; m < 16; m++, at += T * k) dst[at & (N - 1)] = (int)((c[m] + half) >> AUTO_IGN) >> more;
    }
  }
  q ^= 1;
}

__device__ __forceinline__ const cplx *op_key(const BrParams &P, u32 op) {
  return (op & OP_AUTO) ? (const cplx *)P.fft_autos + (size_t)(op & OP_SLOT) * KEY_BLOCK
                        : (const cplx *)P.fft_rgsw + (size_t)(op & OP_INDEX) * KEY_BLOCK;
}

// One gate bootstrap.
__device__ __forceinline__ void fft_item(const BrParams &P, int ct, const u32 *kso, u32 gcode, u64 *out, u64 *rlwe_dbg,
                                         u64 *smem, u32 tm) {
  const int t = threadIdx.x;
  const Smem S(smem);
  const Place p(t, tm + SPEC_COLS + B_COLS);
  // the bucket arrays are only needed while the schedule is built: they, like
  // its scratch (the first 2 N words), share the exchange buffers; the counters
  // and keys take less than 10 KB of the first N words, the buckets' starts and
  // members fit behind them
  SchedSmem sched;
  sched.start = (unsigned short *)((char *)S.x + 10240);
  sched.list = sched.start + (P.br_q >> 1) + 1;
  sched.ops = S.ops;
  sched.nops = S.nops;
  build_schedule<11, T>(P, kso, smem, sched);
  __syncthreads();
  const u32 nops = *S.nops;
  u32 i = 0, q = 0;
  {
    // b: the rotated test polynomial, and the automorphisms of the trivial
    // RLWE (runtime.rs:625-642), which only permute it; a = 0
    long long *from = (long long *)S.buffer(0), *to = (long long *)S.buffer(1);
    const TestRotation tr(P, kso, gcode);
#pragma unroll 1
    for (int c = t; c < N; c += T) from[c] = (long long)tr.at((u32)c);
#pragma unroll 1
    for (; S.ops[i] & OP_AUTO; i++) {
      const u32 k = P.auto_k[S.ops[i] & OP_SLOT];
      __syncthreads();
#pragma unroll 1
      for (int c = t; c < N; c += T) {
        const u32 at = (u32)c * k;
        to[at & (N - 1)] = (at & N) ? -from[c] : from[c];
      }
      long long *const x = from;
      from = to;
      to = x;
    }
    __syncthreads();
    int d[N / T];
#pragma unroll
    for (int m = 0; m < N / T; m++) d[m] = digit<RLRG_IGN>(centre(from[t + T * m]));
    __syncthreads();  // the digits go where b was, or beside it
    int *db = (int *)S.buffer(q ^ 1);
#pragma unroll
    for (int m = 0; m < N / T; m++) {
      db[t + T * m] = d[m];
      S.da[t + T * m] = 0;
    }
  }
  u64 *dst = out + (size_t)(P.out_idx ? P.out_idx[ct] : (u32)ct) * (N + 1);
#pragma unroll 1
  for (; i < nops; i++) {
    const u32 op = S.ops[i], nx = i + 1 < nops ? (u32)S.ops[i + 1] : OP_END;
    __syncthreads();
    fft_op(op, nx, op_key(P, op), nx != OP_END ? op_key(P, nx) : nullptr, P, S, q, tm, p, [&](int o, int c, u64 v) {
      // sample extract at index 0 (pbs.rs:423-449)
      if (o == 0) dst[c == 0 ? 1 : 1 + N - c] = c == 0 ? v : Q_N2048 - v;
      else if (c == 0) dst[0] = v;
      if (rlwe_dbg) rlwe_dbg[((size_t)ct * 2 + o) * N + c] = v;
    });
  }
}

// Tensor memory of the CTA: this warp's address of its lanes.
__device__ __forceinline__ u32 tmem_begin(u32 *slot) {
  if (threadIdx.x < 32) tmem_alloc(slot);
  __syncthreads();
  return *slot + ((threadIdx.x >> 5) << 21);  // lane 32 w in bits 16 and up
}
__device__ __forceinline__ void tmem_end(u32 *slot) {
  __syncthreads();
  if (threadIdx.x < 32) tmem_free(*slot);
}

__global__ void __launch_bounds__(T, 4)
    pbs_fft_kernel(BrParams P, const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out, int count,
                   u64 *rlwe_dbg) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u32 tmem_slot;
  load_twiddles(P, Smem(smem));
  const u32 tm = tmem_begin(&tmem_slot);
  for (int ct = blockIdx.x; ct < count; ct += gridDim.x)
    fft_item(P, ct, ks + (size_t)ct * ks_stride, gates[ct], out, rlwe_dbg, smem, tm);
  tmem_end(&tmem_slot);
}

// Ragged batch: ciphertext ct uses the parameter set and server key of
// descriptor item_desc[ct]; outputs scatter to out_idx[ct].
__global__ void __launch_bounds__(T, 4)
    pbs_fft_ragged_kernel(const BrParams *descs, const u32 *item_desc, const u32 *ks, u32 ks_stride,
                          const unsigned char *gates, u64 *out, const u32 *out_idx, int count) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ BrParams sp;
  __shared__ u32 tmem_slot;
  const u32 tm = tmem_begin(&tmem_slot);
  for (int ct = blockIdx.x; ct < count; ct += gridDim.x) {
    __syncthreads();  // the previous item is done with sp
    if (threadIdx.x == 0) {
      sp = descs[item_desc[ct]];
      sp.out_idx = out_idx;
    }
    __syncthreads();
    if (ct == (int)blockIdx.x) load_twiddles(sp, Smem(smem));
    fft_item(sp, ct, ks + (size_t)ct * ks_stride, gates[ct], out, nullptr, smem, tm);
  }
  tmem_end(&tmem_slot);
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
  cudaError_t e = cudaMalloc(&d, h.size() * 8);
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
  fft::fft_key_kernel<<<(unsigned)(4 * keys), 256, 4 * fft::M * 8, s>>>(rows, (cplx *)out, rows_per_key, rc, tw);
  return cudaGetLastError();
}

cudaError_t pbs_fft_per_sm(u32 br_q, u32 n, int *ctas) {
  const size_t smem = fft::fft_smem_bytes(br_q, n);
  const cudaError_t e = opt_in_smem((const void *)fft::pbs_fft_kernel, smem);
  return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fft::pbs_fft_kernel, fft::T, smem);
}

cudaError_t launch_pbs_fft(const BrParams &P, const u32 *ks, u32 ks_stride, const unsigned char *gates, u64 *out,
                           size_t count, u64 *rlwe_dbg, int grid, cudaStream_t s) {
  const size_t smem = fft::fft_smem_bytes(P.br_q, P.n);
  const cudaError_t e = opt_in_smem((const void *)fft::pbs_fft_kernel, smem);
  if (e != cudaSuccess) return e;
  fft::pbs_fft_kernel<<<grid, fft::T, smem, s>>>(P, ks, ks_stride, gates, out, (int)count, rlwe_dbg);
  return cudaGetLastError();
}

cudaError_t launch_pbs_fft_ragged(const BrParams *d_descs, const u32 *item_desc, u32 max_br_q, u32 max_n, const u32 *ks,
                                  u32 ks_stride, const unsigned char *gates, u64 *out, const u32 *out_idx,
                                  size_t count, int grid, cudaStream_t s) {
  const size_t smem = fft::fft_smem_bytes(max_br_q, max_n);
  const cudaError_t e = opt_in_smem((const void *)fft::pbs_fft_ragged_kernel, smem);
  if (e != cudaSuccess) return e;
  fft::pbs_fft_ragged_kernel<<<grid, fft::T, smem, s>>>(d_descs, item_desc, ks, ks_stride, gates, out, out_idx,
                                                        (int)count);
  return cudaGetLastError();
}

}  // namespace pz
