// pz_fft_ni.cu -- the non-interactive key switch over exact FP64 FFT products
// (pz_fft.cuh): rlwe_key_switch of a batch of values (rgsw/runtime.rs:1001-1063)
// for one user's ui_to_s key or, in key aggregation, for every user's.
//
//   out = sum_j digit_j(v) K_j      for both rows (A, B) of K, j < d
//
// The digits are the d = 50 one-bit signed digits of a value, in {-1, 0, 1}, so
// two limbs of 27 bits do: sum_j ||digit_j|| ||k_j|| <= 50 * 2^5.5 * 2^(26 + 5.5)
// < 2^42.7, the transforms' and keys' error is 81 u of that (pz_fft.cuh) and that of
// the sum of 50 products, 100 roundings in a chain, 100 sqrt2 u: 223 u, less than
// 2^-2.4 < 1/2 in every coefficient.
//
// A batch of 24 values takes 65 us (the integer transforms took 95 with their
// digits split over CTAs); three users' 620-index key 13 ms (37).
//
// Three kernels: the digits of every value transformed once; per point the
// product of the matrix [values x digits] with the user's [digits x (rows,
// limbs)]; and the transforms back.
#include <algorithm>

#include "pz_blind.cuh"
#include "pz_fft.cuh"
#include "pz_internal.h"

namespace pz {
namespace fft {

constexpr int N = 2048;
constexpr int NI_LIMBS = 2, NI_BITS = 27, NI_OUTS = 2 * NI_LIMBS;
constexpr int NI_LANES = 32, NI_BLOCKS = M / NI_LANES;  // points of a product CTA
// Spectra: point r T + t of thread t's register r in layout E.  Keys:
// [block of 32 points][digit][row A, B][limb][point], so that a product CTA's
// part is contiguous.

// One CTA per key row (A rows, then B rows; coefficients).
__global__ void __launch_bounds__(256)
    ni_fft_key_kernel(const u64 *rows, cplx *out, u32 d, const double4 *tw) {
  __shared__ u64 coef[N];
  extern __shared__ double dyn[];
  const u32 o = blockIdx.x / d, digit = blockIdx.x % d;
  for (int e = threadIdx.x; e < N; e += 256)
    coef[e] = reduce2(reduce_n2048(rows[(size_t)blockIdx.x * N + e]), Q_N2048);
  for (int limb = 0; limb < NI_LIMBS; limb++) {
    key_limb<NI_LIMBS, NI_BITS>(coef, limb, dyn, tw);
    for (int e = threadIdx.x; e < M; e += 256) {
      const int p = eval_register(e) * T + eval_thread(e);
      out[(((size_t)(p / NI_LANES) * d + digit) * NI_OUTS + o * NI_LIMBS + limb) * NI_LANES + p % NI_LANES] =
          key_value(dyn, e);
    }
  }
}

// `per` digits of a value at a time per CTA, [row][digit][point].  NEG: the value
// is -A of RLWE `row` (elwise_neg_mut, 0 -> q).  With one-bit digits the
// decomposer (a 1 followed by a 1 becomes -1 and a carry) is the non-adjacent
// form, whose digit j is bit j + 1 of 3 v minus bit j + 1 of v.
template <bool NEG>
__global__ void __launch_bounds__(T, 4)
    ni_fft_digits_kernel(const u64 *vals, cplx *out, size_t rows, u32 per, Decomp dp, const cplx *twiddles) {
  constexpr u32 d = NI_FFT_D;
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u32 tmem_slot;
  cplx *X = (cplx *)smem, *tw = X + 2 * M;
  const int t = threadIdx.x;
  if (t < 32) tmem_alloc<32>(&tmem_slot);
  for (int i = t; i < TW_WORDS; i += T) tw[i] = ldc(twiddles + i);
  __syncthreads();
  const Place p(t, 0, tmem_slot + ((u32)(t >> 5) << 21));
  const u32 parts = (d + per - 1) / per;
  u32 q = 0;
  for (size_t task = blockIdx.x; task < rows * parts; task += gridDim.x) {
    const size_t row = task / parts;
    const u32 j0 = (u32)(task % parts) * per, j1 = min(d, j0 + per);
    u64 v[16], v3[16];
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const u64 x = vals[row * (NEG ? 2 * N : N) + t + T * m];
      v[m] = decomp_init(NEG ? dp.q - x : x, dp);
      v3[m] = 3 * v[m];
    }
#pragma unroll 1
    for (u32 j = j0; j < j1; j++) {
      cplx z[8];
#pragma unroll
      for (int m = 0; m < 16; m++) {
        const int digit = (int)((u32)(v3[m] >> (j + 1)) & 1u) - (int)((u32)(v[m] >> (j + 1)) & 1u);
        (m < 8 ? z[m & 7].r : z[m & 7].i) = i2d(digit);
      }
      forward<1>(z, X + q * M, tw, p);
      q ^= 1;
      cplx *o = out + (row * d + j) * M + t;
#pragma unroll
      for (int r = 0; r < 8; r++) o[r * T] = z[r];
    }
  }
  __syncthreads();
  if (t < 32) tmem_free<32>(tmem_slot);
}

// Which (row, user) pairs are wanted.  In aggregation rows come R = ra + rb per
// LWE index, and the leader of an index only needs its rows ra - 1 and R - 1.
struct NiWanted {
  u32 R, ra, per_user, idx0;  // R = 0: every row
  __device__ __forceinline__ bool operator()(size_t row, u32 user) const {
    if (R == 0) return true;
    const u32 v = (u32)(row % R), idx = idx0 + (u32)(row / R);
    return user != idx / per_user || v == ra - 1 || v == R - 1;
  }
};

// out[row][user][output, limb][point] = sum_j digits[row][j][point] key[user][j][output, limb][point].
// A CTA holds one user's keys of 32 points (100 KB, one bulk copy) and a warp
// works on ROWS = 4 rows at a time, a lane on a point: 16 complex sums in
// registers, 64 multiply-adds for four 16-byte loads from shared memory and
// four from the digits, whose next AHEAD steps are on their way.  Rows past the
// last are read from the scratch behind it and not stored.  Bound by the digits
// (0.8 MB per row, larger than L2 together): 15,500 rows for three users take
// 4.4 ms, of which their multiply-adds alone are 2.1.  Where four rows per
// warp would leave warps idle it is ROWS = 1 and deeper loads: 24 rows take 23
// instead of 36 us.
template <int ROWS, int AHEAD>
__global__ void __launch_bounds__(256, 2)
    ni_fft_product_kernel(const cplx *digits, const cplx *const *keys, cplx *out, size_t rows, NiWanted wanted,
                          u32 *err) {
  constexpr int d = NI_FFT_D;
  static_assert(d % AHEAD == 0, "whole turns");
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u64 bar;
  const cplx *ks = (const cplx *)smem;
  const u32 block = blockIdx.x, user = blockIdx.y, users = gridDim.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
    bulk_load(smem, keys[user] + (size_t)block * d * NI_OUTS * NI_LANES, d * NI_OUTS * NI_LANES * sizeof(cplx), &bar);
  }
  __syncthreads();
  if (!__syncthreads_and(mbar_wait(&bar, 0))) {
    if (threadIdx.x == 0) {
      atomicOr(err, DEVERR_MBAR_TIMEOUT);
      mbar_wait(&bar, 0);  // bounded: the copy this CTA still has in flight
    }
    return;
  }
  const size_t groups = (rows + ROWS - 1) / ROWS;
  for (size_t g = blockIdx.z * 8 + warp; g < groups; g += 8 * gridDim.z) {
    bool any = false;
#pragma unroll
    for (int v = 0; v < ROWS; v++) any |= g * ROWS + v < rows && wanted(g * ROWS + v, user);
    if (!any) continue;
    const cplx *dp = digits + g * ROWS * d * M + block * NI_LANES + lane;
    cplx acc[ROWS][NI_OUTS], x[AHEAD][ROWS];
#pragma unroll
    for (int v = 0; v < ROWS; v++)
#pragma unroll
      for (int o = 0; o < NI_OUTS; o++) acc[v][o] = cplx{0.0, 0.0};
#pragma unroll
    for (int a = 0; a < AHEAD; a++)
#pragma unroll
      for (int v = 0; v < ROWS; v++) x[a][v] = ldc(dp + (v * d + a) * M);
    const cplx *kp = ks + lane;
#pragma unroll 1
    for (int j = 0; j < d; j += AHEAD) {
      dp += AHEAD * M;
#pragma unroll
      for (int a = 0; a < AHEAD; a++) {
#pragma unroll
        for (int o = 0; o < NI_OUTS; o++) {
          const cplx k = *kp;
          kp += NI_LANES;
#pragma unroll
          for (int v = 0; v < ROWS; v++) {
            cplx &s = acc[v][o];
            s.r = fma(x[a][v].r, k.r, fma(-x[a][v].i, k.i, s.r));
            s.i = fma(x[a][v].r, k.i, fma(x[a][v].i, k.r, s.i));
          }
        }
        if (j + AHEAD < d) {
#pragma unroll
          for (int v = 0; v < ROWS; v++) x[a][v] = ldc(dp + (v * d + a) * M);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < ROWS; v++) {
      const size_t row = g * ROWS + v;
      if (row >= rows) break;
      cplx *o = out + (row * users + user) * NI_OUTS * M + block * NI_LANES + lane;
#pragma unroll
      for (int i = 0; i < NI_OUTS; i++) o[i * M] = acc[v][i];
    }
  }
}

// The transforms back: output o (A, B) of (row, user), canonical; put(row,
// user, o, i, v) stores coefficient i.
template <class Put>
__device__ __forceinline__ void ni_fft_outputs(const cplx *sums, size_t rows, u32 users, const NiWanted &wanted,
                                               const cplx *twiddles, u64 *smem, u32 *tmem_slot, const Put &put) {
  cplx *X = (cplx *)smem, *tw = X + 2 * M;
  const int t = threadIdx.x;
  if (t < 32) tmem_alloc<32>(tmem_slot);
  for (int i = t; i < TW_WORDS; i += T) tw[i] = ldc(twiddles + i);
  __syncthreads();
  const Place p(t, 0, *tmem_slot + ((u32)(t >> 5) << 21));
  u32 q = 0;
  for (size_t task = blockIdx.x; task < rows * users * 2; task += gridDim.x) {
    const int o = (int)(task & 1);
    const u32 user = (u32)((task >> 1) % users);
    const size_t row = (task >> 1) / users;
    if (!wanted(row, user)) continue;
    long long acc[16];
#pragma unroll 1
    for (int l = 0; l < NI_LIMBS; l++) {
      const cplx *s = sums + ((row * users + user) * NI_OUTS + o * NI_LIMBS + l) * M + t;
      cplx z[8];
#pragma unroll
      for (int r = 0; r < 8; r++) z[r] = ldc(s + r * T);
      inverse<1>(z, X + q * M, tw, p);
      q ^= 1;
#pragma unroll
      for (int m = 0; m < 16; m++) {
        const long long v =
            __double_as_longlong((m < 8 ? z[m & 7].r : z[m & 7].i) + ROUND) - (long long)ROUND_BITS;
        // 2^27 v = 2^27 (v mod 2^27) + 77823 floor(v / 2^27) (mod Q)
        if (l == 0) acc[m] = v;
        else acc[m] += ((v & ((1ll << NI_BITS) - 1)) << NI_BITS) + (long long)(int)(v >> NI_BITS) * 77823ll;
      }
    }
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const long long c = centre(settle_sum((u64)acc[m]));
      put(row, user, o, t + T * m, (u64)(c < 0 ? c + (long long)Q_N2048 : c));
    }
  }
  __syncthreads();
  if (t < 32) tmem_free<32>(*tmem_slot);
}

// rlwe_key_switch: (A', B') = sums, B' += B of the input
__global__ void __launch_bounds__(T, 4)
    ni_fft_switch_kernel(const cplx *sums, size_t rows, const cplx *twiddles, const u64 *in, u64 *out) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u32 tmem_slot;
  ni_fft_outputs(sums, rows, 1, NiWanted{0, 0, 1, 0}, twiddles, smem, &tmem_slot,
                 [&](size_t row, u32, int o, int i, u64 v) {
                   const size_t at = (row * 2 + o) * N + i;
                   out[at] = o ? add_mod(v, in[at], Q_N2048) : v;
                 });
}

// Key aggregation: the rows of the RGSWs (see NiRows)
__global__ void __launch_bounds__(T, 4)
    ni_fft_rows_kernel(const cplx *sums, size_t rows, u32 users, NiRows R, const cplx *twiddles) {
  extern __shared__ __align__(128) u64 smem[];
  __shared__ u32 tmem_slot;
  const u32 RR = R.ra + R.rb, rows1 = 2 * RR;
  ni_fft_outputs(sums, rows, users, NiWanted{RR, R.ra, R.per_user, R.idx0}, twiddles, smem, &tmem_slot,
                 [&](size_t row, u32 u, int o, int i, u64 x) {
                   const u32 v = (u32)(row % RR), c = (u32)(row / RR), idx = R.idx0 + c, L = idx / R.per_user;
                   const bool to_a = v < R.ra;  // -sm rows add the NI row to A, m rows to B
                   const NiRowUser &U = R.users[u];
                   const u64 *ct;
                   u64 *dst;
                   if (u == L) {
                     ct = U.self_leader + ((size_t)(idx - U.seg_b) * R.max_l + (R.max_l - 1)) * N;
                     dst = R.leader + ((size_t)c * 4 + (to_a ? 0 : 2) + o) * N;
                   } else {
                     const u32 pos = idx < U.seg_b ? idx : idx - (U.seg_e - U.seg_b);
                     const u32 row_ct = to_a ? R.max_d - R.ra + v : R.max_d - R.rb + (v - R.ra);
                     ct = U.not_leader + ((size_t)pos * R.max_d + row_ct) * N;
                     const u32 row_out = to_a ? v + o * R.ra : 2 * R.ra + (v - R.ra) + o * R.rb;
                     dst = R.others + (((size_t)(u < L ? u : u - 1) * R.cnt + c) * rows1 + row_out) * N;
                   }
                   dst[i] = to_a == (o == 0) ? add_mod(x, ct[i], Q_N2048) : x;
                 });
}

constexpr size_t TRANSFORM_SMEM = (size_t)(2 * M + TW_WORDS) * sizeof(cplx);

}  // namespace fft

using fft::cplx;

static int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

size_t ni_fft_key_bytes(u32 d) { return (size_t)d * fft::NI_OUTS * fft::M * sizeof(cplx); }
size_t ni_fft_digit_bytes(u32 d, size_t rows) { return (rows + 3) * d * fft::M * sizeof(cplx); }
size_t ni_fft_sum_bytes() { return (size_t)fft::NI_OUTS * fft::M * sizeof(cplx); }

cudaError_t launch_ni_fft_key(const u64 *rows, u32 d, const void *tables, void *out, cudaStream_t s) {
  const double4 *tw = (const double4 *)((const cplx *)tables + fft::TW_WORDS);
  fft::ni_fft_key_kernel<<<2 * d, 256, fft::KEY_SMEM, s>>>(rows, (cplx *)out, d, tw);
  return cudaGetLastError();
}

static cudaError_t digits_and_products(const u64 *vals, bool neg, size_t rows, u32 users, u32 d, const Decomp &dp,
                                       const void *const *keys, const void *tables, void *digits, void *sums,
                                       const fft::NiWanted &wanted, u32 *err, cudaStream_t s) {
  const int sms = sm_count();
  auto *dk = neg ? fft::ni_fft_digits_kernel<true> : fft::ni_fft_digits_kernel<false>;
  cudaError_t e = opt_in_smem((const void *)dk, fft::TRANSFORM_SMEM);
  if (e != cudaSuccess) return e;
  // ten digits per task, fewer where that would leave places empty
  const u32 per = (u32)std::max<size_t>(1, std::min<size_t>(10, rows * d / (4 * (size_t)sms)));
  const size_t tasks = rows * ((d + per - 1) / per);
  dk<<<(unsigned)std::min<size_t>(tasks, (size_t)4 * sms), fft::T, fft::TRANSFORM_SMEM, s>>>(
      vals, (cplx *)digits, rows, per, dp, (const cplx *)tables);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // two CTAs per SM, over blocks of points, users and ranges of rows; four rows
  // per warp where every warp of them gets some
  const size_t smem = (size_t)d * fft::NI_OUTS * fft::NI_LANES * sizeof(cplx);
  const size_t places = std::max<size_t>(1, (size_t)2 * sms / ((size_t)fft::NI_BLOCKS * users));
  const bool wide = rows >= 4 * 8 * places;
  auto *pk = wide ? fft::ni_fft_product_kernel<4, 2> : fft::ni_fft_product_kernel<1, 10>;
  if ((e = opt_in_smem((const void *)pk, smem)) != cudaSuccess) return e;
  const size_t groups = wide ? (rows + 3) / 4 : rows;
  const unsigned z = (unsigned)std::min<size_t>((groups + 7) / 8, places);
  pk<<<dim3(fft::NI_BLOCKS, users, z), 256, smem, s>>>((const cplx *)digits, (const cplx *const *)keys, (cplx *)sums,
                                                       rows, wanted, err);
  return cudaGetLastError();
}

cudaError_t launch_ni_fft_switch(const u64 *in, u64 *out, size_t rows, u32 d, const Decomp &dp,
                                 const void *const *keys, const void *tables, void *digits, void *sums, u32 *err,
                                 cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  cudaError_t e = digits_and_products(in, true, rows, 1, d, dp, keys, tables, digits, sums, fft::NiWanted{0, 0, 1, 0},
                                      err, s);
  if (e == cudaSuccess) e = opt_in_smem((const void *)fft::ni_fft_switch_kernel, fft::TRANSFORM_SMEM);
  if (e != cudaSuccess) return e;
  fft::ni_fft_switch_kernel<<<(unsigned)std::min<size_t>(2 * rows, (size_t)4 * sm_count()), fft::T,
                              fft::TRANSFORM_SMEM, s>>>((const cplx *)sums, rows, (const cplx *)tables, in, out);
  return cudaGetLastError();
}

cudaError_t launch_ni_fft_rows(const u64 *vals, size_t rows, u32 users, u32 d, const Decomp &dp, const NiRows &R,
                               const void *const *keys, const void *tables, void *digits, void *sums, u32 *err,
                               cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  cudaError_t e = digits_and_products(vals, false, rows, users, d, dp, keys, tables, digits, sums,
                                      fft::NiWanted{R.ra + R.rb, R.ra, R.per_user, R.idx0}, err, s);
  if (e == cudaSuccess) e = opt_in_smem((const void *)fft::ni_fft_rows_kernel, fft::TRANSFORM_SMEM);
  if (e != cudaSuccess) return e;
  fft::ni_fft_rows_kernel<<<(unsigned)std::min<size_t>(2 * rows * users, (size_t)4 * sm_count()), fft::T,
                            fft::TRANSFORM_SMEM, s>>>((const cplx *)sums, rows, users, R, (const cplx *)tables);
  return cudaGetLastError();
}

}  // namespace pz
