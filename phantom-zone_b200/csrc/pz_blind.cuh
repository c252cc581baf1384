// pz_blind.cuh -- the blind rotation's schedule and test polynomial, shared by
// the integer (pz_kernels.cu) and FFT (pz_fft.cu) kernels.
#pragma once
#include "pz_kernels.cuh"

namespace pz {

// Operation codes of the blind-rotation schedule: an external product with
// RGSW key `i` is `i`; an automorphism with key slot v (0 = -g) is
// OP_AUTO | v, plus OP_TRIVIAL while the accumulator is still trivial.
// OP_KEEPB marks an operation whose successor is a non-trivial automorphism:
// it leaves b in the evaluation domain (scaled by N^{-1}, values < 2q), where
// the automorphism permutes it and adds it before its own inverse transform,
// so b skips one inverse and one forward-domain round trip.
constexpr u32 OP_AUTO = 0x8000u, OP_TRIVIAL = 0x4000u, OP_KEEPB = 0x2000u, OP_SLOT = 0x00ffu,
              OP_INDEX = 0x1fffu;

// pbs.rs:416-420
__device__ __forceinline__ u32 mod_switch_odd(u32 v, double from_q, double to_q) {
  u64 odd = (u64)floor(__ddiv_rn(__dmul_rn((double)v, to_q), from_q));
  return (u32)(odd + ((odd & 1ull) ^ 1ull));
}

// Shared-memory arrays of the blind-rotation schedule, after `regions` x N words.
struct SchedSmem {
  unsigned short *start, *list, *ops;
  u32 *nops;
};
template <int LOGN>
__device__ __forceinline__ SchedSmem sched_smem(u64 *smem, int regions, u32 R, u32 n) {
  constexpr int N = 1 << LOGN;
  SchedSmem m;
  m.start = (unsigned short *)(smem + regions * N);  // R + 1
  m.list = m.start + (R + 1);                         // n
  m.ops = m.list + n;                                 // n + R + 1
  m.nops = (u32 *)(((size_t)(m.ops + n + R + 1) + 3) & ~(size_t)3);
  return m;
}

// Odd mod-switch, dlog buckets (pbs.rs:147-161, stable in LWE index) and the
// blind-rotation schedule (pbs.rs:240-414) of one key-switched LWE, built in
// shared memory by the whole CTA (regions 0 and 1 of smem are scratch).
template <int LOGN, int TH = NttShape<LOGN>::T>
__device__ __forceinline__ void build_schedule(const BrParams &P, const u32 *kso, u64 *smem, const SchedSmem &S) {
  constexpr int N = 1 << LOGN, T = TH;  // TH: the CTA's threads
  const u32 R = P.br_q >> 1, q4 = P.br_q >> 2, n = P.n;
  const int j = threadIdx.x, lane = j & 31, warp = j >> 5;
  u64 *sm = smem;
  unsigned short *s_start = S.start, *s_list = S.list, *s_ops = S.ops;
  u32 *s_nops = S.nops;
  {
    // ---- odd mod-switch + dlog buckets (pbs.rs:147-161), stable in LWE index
    u32 *cnt = (u32 *)sm;                                 // R counters (region 0)
    unsigned short *keys = (unsigned short *)(cnt + R);   // n keys (region 0)
    u32 *fill = (u32 *)(sm + N);                          // R fill counters (region 1)
    u32 *scan = fill + R;                                 // T partial sums (region 1)
    __syncthreads();
    for (u32 b = j; b < R; b += T) { cnt[b] = 0; fill[b] = 0; }
    __syncthreads();
    for (u32 i = j; i < n; i += T) {
      const u32 odd = mod_switch_odd(kso[1 + i] & P.ks_mask, P.q_ks_f, P.br_q_f);
      const u32 k = P.dlog[odd];
      keys[i] = (unsigned short)k;
      atomicAdd(&cnt[k], 1u);
    }
    __syncthreads();
    {  // exclusive scan of cnt[0..R) into s_start, s_start[R] = n
      const u32 per = (R + T - 1) / T;
      const u32 b0 = j * per;
      u32 local = 0;
      for (u32 b = b0; b < b0 + per && b < R; b++) local += cnt[b];
      u32 incl = local;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        u32 y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) scan[warp] = incl;
      __syncthreads();
      u32 woff = 0;
      for (int w2 = 0; w2 < warp; w2++) woff += scan[w2];
      u32 run = woff + incl - local;
      for (u32 b = b0; b < b0 + per && b < R; b++) {
        s_start[b] = (unsigned short)run;
        run += cnt[b];
      }
      if (j == 0) s_start[R] = (unsigned short)n;
    }
    __syncthreads();
    if (warp == 0) {  // stable placement: within a bucket, increasing LWE index
      for (u32 i0 = 0; i0 < n; i0 += 32) {
        const u32 i = i0 + lane;
        const bool valid = i < n;
        const u32 k = valid ? keys[i] : 0xFFFFu;
        const u32 peers = __match_any_sync(0xffffffffu, k);
        const u32 rank = __popc(peers & ((1u << lane) - 1u));
        if (valid) s_list[s_start[k] + fill[k] + rank] = (unsigned short)i;
        __syncwarp();
        if (valid && rank == 0) fill[k] += __popc(peers);
        __syncwarp();
      }
    }
    __syncthreads();
    // ---- the blind-rotation schedule (pbs.rs:240-414): buckets of -g^k for
    // k = q/4-1..1, -g^0, +g^k, +g^0 (R - 1 down to 0), each followed by an
    // automorphism when the next bucket is non-empty, the window w is reached or
    // k == 1; the automorphisms before the first external product act on a
    // trivial RLWE.  Thread j takes buckets R - 1 - p, p0 <= p < p1: where the
    // window starts and how many automorphisms come before are scans over the
    // threads (one thread walking over all took 0.25 ms, 4 % of one gate).
    int *part = (int *)scan;  // per warp: maxima, then (from 32) sums
    const u32 per = (R + T - 1) / T;
    const int p0 = (int)min(per * j, R), p1 = (int)min(per * (j + 1), R);
    // an automorphism follows whatever the window (b == q4: -g^0, with slot 0)
    auto forced = [&](u32 b) {
      return b != 0 && (b == q4 || b == 1 || b == q4 + 1 || s_start[b - 1] != s_start[b]);
    };
    int last = -1;
    for (int p = p0; p < p1; p++)
      if (forced(R - 1 - p)) last = p;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, last, o);
      if (lane >= o) last = max(last, y);
    }
    if (lane == 31) part[warp] = last;
    last = __shfl_up_sync(0xffffffffu, last, 1);
    if (lane == 0) last = -1;
    __syncthreads();
    for (int w2 = 0; w2 < warp; w2++) last = max(last, part[w2]);
    const u32 v0 = (u32)(p0 - last - 1) % P.w;
    // every bucket of this thread: put(bucket, an automorphism follows, its slot)
    auto walk = [&](auto put) {
      u32 v = v0;
      for (int p = p0; p < p1; p++) {
        const u32 b = R - 1 - (u32)p;
        v++;
        const bool f = forced(b), follows = f || (b != 0 && v == P.w);
        put(b, follows, b == q4 ? 0u : v);
        if (follows) v = 0;
      }
    };
    int mine = 0;
    walk([&](u32, bool follows, u32) { mine += follows; });
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) part[32 + warp] = incl;
    __syncthreads();
    u32 before = (u32)(incl - mine);
    for (int w2 = 0; w2 < warp; w2++) before += (u32)part[32 + w2];
    walk([&](u32 b, bool follows, u32 slot) {
      u32 no = n - s_start[b + 1] + before;
      for (u32 t = s_start[b]; t < s_start[b + 1]; t++) s_ops[no++] = s_list[t];
      if (follows) {
        s_ops[no] = (unsigned short)(OP_AUTO | (s_start[b] == n ? OP_TRIVIAL : 0u) | slot);
        before++;
      }
    });
    if (p0 < p1 && p1 == (int)R) *s_nops = n + before;
    __syncthreads();
    // b stays in the evaluation domain before a non-trivial automorphism
    const u32 nops = *s_nops;
    for (u32 o = j; o + 1 < nops; o += T)
      if ((s_ops[o + 1] & (OP_AUTO | OP_TRIVIAL)) == OP_AUTO) s_ops[o] |= (unsigned short)OP_KEEPB;
  }
}

// Trivial test RLWE's b: X^{g * odd(b)} * tv, embedded (pbs.rs:163-211), in
// the coefficient layout of this thread (test_rlwe_b).
struct TestRotation {
  const u64 *tv;
  u64 q;
  u32 R, emb, mexp;
  bool msign;
  __device__ __forceinline__ TestRotation(const BrParams &P, const u32 *kso, u32 gcode)
      : q(P.rc.q), R(P.br_q >> 1), emb(P.emb) {
    const u32 odd_b = mod_switch_odd(kso[0] & P.ks_mask, P.q_ks_f, P.br_q_f);
    mexp = (u32)(((u64)P.g * odd_b) % P.br_q);
    msign = true;
    if (mexp > R) { mexp -= R; msign = false; }
    u32 gi = gcode & 7u;
    if (gi > 5) gi = 5;  // codes are validated on the host; never index past the 6 test vectors
    tv = P.tv + (size_t)gi * R;
  }
  // coefficient p of the rotated, embedded test polynomial
  __device__ __forceinline__ u64 at(u32 p) const {
    if (p % emb) return 0;
    const u32 o = p / emb;
    u32 s;
    bool sg;
    if (o >= mexp) { s = o - mexp; sg = msign; } else { s = o + R - mexp; sg = !msign; }
    const u64 t = tv[s];
    return sg ? t : q - t;
  }
};
template <int LOGN>
__device__ __forceinline__ void test_rlwe_b(const BrParams &P, const u32 *kso, u32 gcode, u64 (&b)[8]) {
  const TestRotation tr(P, kso, gcode);
#pragma unroll
  for (int r = 0; r < 8; r++) b[r] = tr.at((u32)pos_coef<LOGN>(threadIdx.x, r));
}

// L2 prefetch of a blind-rotation operation's key rows (none for a trivial
// automorphism).
template <int LOGN>
__device__ __forceinline__ void prefetch_next_key(const BrParams &P, u32 op) {
  constexpr size_t N = (size_t)1 << LOGN;
  if (op & OP_AUTO) {
    if (!(op & OP_TRIVIAL))
      prefetch_l2(P.autos + (size_t)(op & OP_SLOT) * P.auto_rows * N, P.auto_rows * (u32)N * 8);
  } else {
    prefetch_l2(P.rgsw + (size_t)(op & OP_INDEX) * P.rgsw_rows * N, P.rgsw_rows * (u32)N * 8);
  }
}

}  // namespace pz
