// pz_fft.cuh -- exact negacyclic products modulo Q = 2^54 - 77823 (N = 2048)
// through double-precision FFTs.
//
// A product of a digit polynomial d (small signed integers) with a key
// polynomial K mod Q is a negacyclic convolution over the integers, reduced
// mod Q at the end.  K, centred in (-Q/2, Q/2], is cut into three signed
// limbs of 18 bits, K = k0 + 2^18 k1 + 2^36 k2 with |k_l| <= 2^17, and each
// d k_l is computed by a complex FFT of length M = 1024 (coefficient j as the
// real part and j + 1024 as the imaginary part of c_j, in
// C[t]/(t^1024 - i)), rounded to the nearest integer and recombined mod Q.
//
// The rounding is exact for every input.  With u = 2^-53 and to first order, write
// S = sum ||d|| ||k_l|| over an operation's two products, |d| <= 2^16: S <=
// 2 * 2^(16 + 5.5) * 2^(17 + 5.5) = 2^45.  Each of these is at most c u S in every
// output coefficient, and the c add up to 87: 87 u 2^45 < 0.35 < 1/2.  (Measured:
// below 2^-8.)
//   forward, 40: a butterfly's t = a + w b has two roundings per component, of
//   a + Re(w) b and of t, and w one; 2a - t repeats them and adds its own.  In the
//   2-norm of the pair, with |a|^2 + |b|^2 = 1, that is u (sqrt2 |a + Re(w) b| +
//   sqrt2 |t| + |2a - t| + sqrt2 |b|) <= u (sqrt2 sqrt5 + sqrt3 sqrt2) < 5.7 u
//   against the pair's norm of sqrt2: 4 u per level, ten levels; the spectra's
//   errors reach a coefficient as a sum over the points, at most (Cauchy-Schwarz)
//   the product of the 2-norms of the error and of the key's spectrum.
//   products, 6: four roundings in a chain per component, 4 sqrt2 u.
//   keys, 1: transformed in double-double and rounded once.
//   inverse, 40: of a + b one rounding, of conj(w) (a - b) three and w's own: 4 u
//   (|a| + |b|) per butterfly.  Summed over the values that a coefficient is made
//   of, whose 1-norm no level increases and which is at most S (Cauchy-Schwarz), 4
//   u S per level, ten levels.
//
// Why FFTs: on B200 an FP64 multiply-add costs what a 32-bit integer one
// does, and a complex radix-2 butterfly over 2048 real coefficients takes 6
// (forward) or 8 (inverse) of them for two coefficient pairs, where an
// integer butterfly mod Q takes about 20 instructions for one.
#pragma once
#include "pz_kernels.cuh"

namespace pz {
namespace fft {

constexpr int M = 1024;          // complex length
constexpr int T = 128;           // threads per polynomial (a group), 8 complex values each
constexpr int LIMBS = 3, LIMB_BITS = 18;
constexpr int POLY_W = M;        // complex words (16 bytes) of one transformed limb
// One key block = the operand of one operation: [output a, b][limb][point 0..7]
// [digit polynomial x, y][thread], complex.
constexpr size_t KEY_BLOCK = (size_t)2 * LIMBS * 2 * M;  // complex words (192 KB)
// automorphism digits (24 bits) are cut in two so that the same bound holds
constexpr int AUTO_CUT = 12;

struct cplx {
  double r, i;
};

// Twiddle tables (complex words).  Node k of level s of the tree holds
// t^(M / 2^s) - z; its twiddle y has y^2 = z.  y = exp(2 pi i phi) with
// phi(0, 0) = 1/8, phi(s + 1, 2k) = phi/2, phi(s + 1, 2k + 1) = phi/2 + 1/4, so a
// right sibling's twiddle is i times the left one's and only left ones are kept.
//   levels 0-2: constants; levels 3-5: [4][8 nodes of level 3]; levels 6, 7:
//   [3][32 nodes of level 5]; levels 8, 9: [4][128 threads] (the twiddles of
//   levels 8 and 9 for p4 = 0, then for p4 = 1; see the layouts below).
constexpr int TW_R1 = 0, TW_R2 = TW_R1 + 32, TW_R3 = TW_R2 + 96, TW_WORDS = TW_R3 + 512;
// levels 0-2: exp(i pi/4), exp(i pi/8), exp(i pi/16), exp(5 i pi/16)
#define PZ_FFT_C0                                                                                   \
  cplx{0.70710678118654752440, 0.70710678118654752440}, cplx{0.92387953251128675613, 0.38268343236508977173}, \
      cplx{0.98078528040323044913, 0.19509032201612826785}, cplx{0.55557023301960222474, 0.83146961230254523708}

__device__ __forceinline__ cplx ldc(const cplx *p) {
  cplx v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.r), "=d"(v.i) : "l"(p));
  return v;
}
__device__ __forceinline__ cplx ld_key(const cplx *p) {
  cplx v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.r), "=d"(v.i) : "l"(p));
  return v;
}

// forward butterfly (a, b) -> (a + w b, a - w b): six multiply-adds
__device__ __forceinline__ void fbf(cplx &a, cplx &b, double wr, double wi) {
  double tr = fma(wr, b.r, a.r), ti = fma(wr, b.i, a.i);
  tr = fma(-wi, b.i, tr);
  ti = fma(wi, b.r, ti);
  b.r = fma(2.0, a.r, -tr);
  b.i = fma(2.0, a.i, -ti);
  a.r = tr;
  a.i = ti;
}
// inverse butterfly (a, b) -> (a + b, conj(w) (a - b))
__device__ __forceinline__ void ibf(cplx &a, cplx &b, double wr, double wi) {
  const double dr = a.r - b.r, di = a.i - b.i;
  a.r += b.r;
  a.i += b.i;
  b.r = fma(wr, dr, wi * di);
  b.i = fma(wr, di, -(wi * dr));
}

// three levels on 8 values; c1, c2 and (c3, c4) are the left twiddles of the
// round's levels
__device__ __forceinline__ void fwd8(cplx (&x)[8], const cplx &c1, const cplx &c2, const cplx &c3, const cplx &c4) {
#pragma unroll
  for (int r = 0; r < 4; r++) fbf(x[r], x[r + 4], c1.r, c1.i);
  fbf(x[0], x[2], c2.r, c2.i);
  fbf(x[1], x[3], c2.r, c2.i);
  fbf(x[4], x[6], -c2.i, c2.r);
  fbf(x[5], x[7], -c2.i, c2.r);
  fbf(x[0], x[1], c3.r, c3.i);
  fbf(x[2], x[3], -c3.i, c3.r);
  fbf(x[4], x[5], c4.r, c4.i);
  fbf(x[6], x[7], -c4.i, c4.r);
}
__device__ __forceinline__ void inv8(cplx (&x)[8], const cplx &c1, const cplx &c2, const cplx &c3, const cplx &c4) {
  ibf(x[0], x[1], c3.r, c3.i);
  ibf(x[2], x[3], -c3.i, c3.r);
  ibf(x[4], x[5], c4.r, c4.i);
  ibf(x[6], x[7], -c4.i, c4.r);
  ibf(x[0], x[2], c2.r, c2.i);
  ibf(x[1], x[3], c2.r, c2.i);
  ibf(x[4], x[6], -c2.i, c2.r);
  ibf(x[5], x[7], -c2.i, c2.r);
#pragma unroll
  for (int r = 0; r < 4; r++) ibf(x[r], x[r + 4], c1.r, c1.i);
}

__device__ __forceinline__ void fwd4(cplx &a, cplx &b, cplx &c, cplx &d, double w1r, double w1i, const cplx &w2) {
  fbf(a, c, w1r, w1i);
  fbf(b, d, w1r, w1i);
  fbf(a, b, w2.r, w2.i);
  fbf(c, d, -w2.i, w2.r);
}
__device__ __forceinline__ void inv4(cplx &a, cplx &b, cplx &c, cplx &d, double w1r, double w1i, const cplx &w2) {
  ibf(a, b, w2.r, w2.i);
  ibf(c, d, -w2.i, w2.r);
  ibf(a, c, w1r, w1i);
  ibf(b, d, w1r, w1i);
}

// Tensor memory.  Warps of equal number in the groups of a CTA share 32 lanes
// of it, and their threads of equal number hold the same positions of their
// polynomials, so it is where the groups meet without the shared-memory pipe,
// besides saving registers.
template <u32 COLS>
__device__ __forceinline__ void tmem_alloc(u32 *slot) {  // one warp; slot in shared memory
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(COLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <u32 COLS>
__device__ __forceinline__ void tmem_free(u32 base) {  // the same warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(COLS));
}
// One 32-bit word into the other CTA's shared memory, counted there on *bar.
__device__ __forceinline__ void remote_store(u32 addr, int v, u32 bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
               : "memory");
}
// ... two of them (8-byte aligned)
__device__ __forceinline__ void remote_store2(u32 addr, int a, int b, u32 bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr), "r"(a),
               "r"(b), "r"(bar)
               : "memory");
}
// this CTA's shared address in CTA `rank` of the cluster
__device__ __forceinline__ u32 cluster_addr(const void *p, u32 rank) {
  u32 a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  return a;
}
// mbar_wait for writes of the cluster
__device__ __forceinline__ bool mbar_wait_cluster(u64 *bar, u32 parity, long long limit = MBAR_WAIT_LIMIT) {
  const u32 a = smem_addr(bar);
  const long long t0 = clock64();
  while (limit > 0) {
    u32 done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit) break;
  }
  return false;
}
__device__ __forceinline__ void mbar_expect(u64 *bar, u32 bytes) {  // one arrival
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// around a barrier between one warp's accesses and another's
__device__ __forceinline__ void tmem_before_barrier() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_after_barrier() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// two complex values -> 8 columns
__device__ __forceinline__ void tmem_store2(u32 addr, const cplx &a, const cplx &b) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<8>;\n\t"
      "mov.b64 {r0, r1}, %1;\n\tmov.b64 {r2, r3}, %2;\n\tmov.b64 {r4, r5}, %3;\n\tmov.b64 {r6, r7}, %4;\n\t"
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7};\n\t"
      "}" ::"r"(addr),
      "d"(a.r), "d"(a.i), "d"(b.r), "d"(b.i)
      : "memory");
}
// 16 columns -> four complex values
__device__ __forceinline__ void tmem_load4(u32 addr, cplx &a, cplx &b, cplx &c, cplx &d) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<16>;\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, "
      "r15}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n\t"
      "mov.b64 %0, {r0, r1};\n\tmov.b64 %1, {r2, r3};\n\tmov.b64 %2, {r4, r5};\n\tmov.b64 %3, {r6, r7};\n\t"
      "mov.b64 %4, {r8, r9};\n\tmov.b64 %5, {r10, r11};\n\tmov.b64 %6, {r12, r13};\n\tmov.b64 %7, {r14, r15};\n\t"
      "}"
      : "=d"(a.r), "=d"(a.i), "=d"(b.r), "=d"(b.i), "=d"(c.r), "=d"(c.i), "=d"(d.r), "=d"(d.i)
      : "r"(addr)
      : "memory");
}
// eight 64-bit words <-> 16 columns
__device__ __forceinline__ void tmem_store8(u32 addr, const u64 (&v)[8]) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<16>;\n\t"
      "mov.b64 {r0, r1}, %1;\n\tmov.b64 {r2, r3}, %2;\n\tmov.b64 {r4, r5}, %3;\n\tmov.b64 {r6, r7}, %4;\n\t"
      "mov.b64 {r8, r9}, %5;\n\tmov.b64 {r10, r11}, %6;\n\tmov.b64 {r12, r13}, %7;\n\tmov.b64 {r14, r15}, %8;\n\t"
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, "
      "r14, r15};\n\t"
      "}" ::"r"(addr),
      "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3]), "l"(v[4]), "l"(v[5]), "l"(v[6]), "l"(v[7])
      : "memory");
}
__device__ __forceinline__ void tmem_load8(u32 addr, u64 (&v)[8]) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<16>;\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, "
      "r15}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n\t"
      "mov.b64 %0, {r0, r1};\n\tmov.b64 %1, {r2, r3};\n\tmov.b64 %2, {r4, r5};\n\tmov.b64 %3, {r6, r7};\n\t"
      "mov.b64 %4, {r8, r9};\n\tmov.b64 %5, {r10, r11};\n\tmov.b64 %6, {r12, r13};\n\tmov.b64 %7, {r14, r15};\n\t"
      "}"
      : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(v[4]), "=l"(v[5]), "=l"(v[6]), "=l"(v[7])
      : "r"(addr)
      : "memory");
}

// three groups of 2 C columns, 32 apart -> the sums of C 64-bit words
template <int C>
__device__ __forceinline__ void tmem_sum3(u32 addr, u64 (&v)[C]) {
  static_assert(C == 2 || C == 4 || C == 6, "");
  if constexpr (C == 2)
    asm volatile(
        "{\n\t"
        ".reg .b32 r<12>;\n\t.reg .u64 a, b, c;\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r0, r1, r2, r3}, [%2];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r4, r5, r6, r7}, [%3];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r8, r9, r10, r11}, [%4];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n\t"
        "mov.b64 a, {r0, r1};\n\tmov.b64 b, {r4, r5};\n\tmov.b64 c, {r8, r9};\n\tadd.u64 a, a, b;\n\tadd.u64 %0, a, c;\n\t"
        "mov.b64 a, {r2, r3};\n\tmov.b64 b, {r6, r7};\n\tmov.b64 c, {r10, r11};\n\tadd.u64 a, a, b;\n\tadd.u64 %1, a, c;\n\t"
        "}"
        : "=l"(v[0]), "=l"(v[1])
        : "r"(addr), "r"(addr + 32), "r"(addr + 64)
        : "memory");
  else if constexpr (C == 4)
    asm volatile(
        "{\n\t"
        ".reg .b32 r<24>;\n\t.reg .u64 a, b, c;\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {r0, r1, r2, r3, r4, r5, r6, r7}, [%4];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {r8, r9, r10, r11, r12, r13, r14, r15}, [%5];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {r16, r17, r18, r19, r20, r21, r22, r23}, [%6];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n\t"
        "mov.b64 a, {r0, r1};\n\tmov.b64 b, {r8, r9};\n\tmov.b64 c, {r16, r17};\n\tadd.u64 a, a, b;\n\tadd.u64 %0, a, c;\n\t"
        "mov.b64 a, {r2, r3};\n\tmov.b64 b, {r10, r11};\n\tmov.b64 c, {r18, r19};\n\tadd.u64 a, a, b;\n\tadd.u64 %1, a, c;\n\t"
        "mov.b64 a, {r4, r5};\n\tmov.b64 b, {r12, r13};\n\tmov.b64 c, {r20, r21};\n\tadd.u64 a, a, b;\n\tadd.u64 %2, a, c;\n\t"
        "mov.b64 a, {r6, r7};\n\tmov.b64 b, {r14, r15};\n\tmov.b64 c, {r22, r23};\n\tadd.u64 a, a, b;\n\tadd.u64 %3, a, c;\n\t"
        "}"
        : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
        : "r"(addr), "r"(addr + 32), "r"(addr + 64)
        : "memory");
  else {
    u64 w[4], x[2];
    tmem_sum3<4>(addr, w);
    tmem_sum3<2>(addr + 8, x);
#pragma unroll
    for (int m = 0; m < 4; m++) v[m] = w[m];
    v[4] = x[0];
    v[5] = x[1];
  }
}

// Two lane bits and two register bits change places through tensor memory,
// without the load/store unit: 32x32b accesses have a lane's registers in
// consecutive columns of its row; 16x256b accesses spread eight columns of a
// row, a double each two, over four neighbouring lanes.  Stored the first way
// and loaded the second, the double that lane (l4 l3 l2 l1 l0) held in columns
// 8 c + 2 (q1 q0) arrives in lane (l2 l1 l0 q1 q0), register (c, l4, l3).  COLS
// picks which two register bits of the eight complex values are q: 1: bits 2
// and 1 (the other is bit 0), 2: bits 1 and 0 (the other is bit 2).  On arrival
// the register index is (other, l4, l3).
template <int COLS>
__device__ __forceinline__ void turn_put(u32 addr, const cplx (&x)[8]) {
  if constexpr (COLS == 1)
    asm volatile(
        "{\n\t"
        ".reg .b32 r<32>;\n\t"
        "mov.b64 {r0, r1}, %1;\n\t"
        "mov.b64 {r8, r9}, %2;\n\t"
        "mov.b64 {r16, r17}, %3;\n\t"
        "mov.b64 {r24, r25}, %4;\n\t"
        "mov.b64 {r2, r3}, %5;\n\t"
        "mov.b64 {r10, r11}, %6;\n\t"
        "mov.b64 {r18, r19}, %7;\n\t"
        "mov.b64 {r26, r27}, %8;\n\t"
        "mov.b64 {r4, r5}, %9;\n\t"
        "mov.b64 {r12, r13}, %10;\n\t"
        "mov.b64 {r20, r21}, %11;\n\t"
        "mov.b64 {r28, r29}, %12;\n\t"
        "mov.b64 {r6, r7}, %13;\n\t"
        "mov.b64 {r14, r15}, %14;\n\t"
        "mov.b64 {r22, r23}, %15;\n\t"
        "mov.b64 {r30, r31}, %16;\n\t"
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15, r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31};\n\t"
        "}"
        : 
        : "r"(addr), "d"(x[0].r), "d"(x[0].i), "d"(x[1].r), "d"(x[1].i), "d"(x[2].r), "d"(x[2].i), "d"(x[3].r), "d"(x[3].i), "d"(x[4].r), "d"(x[4].i), "d"(x[5].r), "d"(x[5].i), "d"(x[6].r), "d"(x[6].i), "d"(x[7].r), "d"(x[7].i)
        : "memory");
  else
    asm volatile(
        "{\n\t"
        ".reg .b32 r<32>;\n\t"
        "mov.b64 {r0, r1}, %1;\n\t"
        "mov.b64 {r8, r9}, %2;\n\t"
        "mov.b64 {r2, r3}, %3;\n\t"
        "mov.b64 {r10, r11}, %4;\n\t"
        "mov.b64 {r4, r5}, %5;\n\t"
        "mov.b64 {r12, r13}, %6;\n\t"
        "mov.b64 {r6, r7}, %7;\n\t"
        "mov.b64 {r14, r15}, %8;\n\t"
        "mov.b64 {r16, r17}, %9;\n\t"
        "mov.b64 {r24, r25}, %10;\n\t"
        "mov.b64 {r18, r19}, %11;\n\t"
        "mov.b64 {r26, r27}, %12;\n\t"
        "mov.b64 {r20, r21}, %13;\n\t"
        "mov.b64 {r28, r29}, %14;\n\t"
        "mov.b64 {r22, r23}, %15;\n\t"
        "mov.b64 {r30, r31}, %16;\n\t"
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15, r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31};\n\t"
        "}"
        : 
        : "r"(addr), "d"(x[0].r), "d"(x[0].i), "d"(x[1].r), "d"(x[1].i), "d"(x[2].r), "d"(x[2].i), "d"(x[3].r), "d"(x[3].i), "d"(x[4].r), "d"(x[4].i), "d"(x[5].r), "d"(x[5].i), "d"(x[6].r), "d"(x[6].i), "d"(x[7].r), "d"(x[7].i)
        : "memory");
}
__device__ __forceinline__ void turn_take(u32 addr, cplx (&x)[8]) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<32>;\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n\t"
      "mov.b64 %0, {r0, r1};\n\t"
      "mov.b64 %1, {r4, r5};\n\t"
      "mov.b64 %2, {r2, r3};\n\t"
      "mov.b64 %3, {r6, r7};\n\t"
      "mov.b64 %4, {r16, r17};\n\t"
      "mov.b64 %5, {r20, r21};\n\t"
      "mov.b64 %6, {r18, r19};\n\t"
      "mov.b64 %7, {r22, r23};\n\t"
      "mov.b64 %8, {r8, r9};\n\t"
      "mov.b64 %9, {r12, r13};\n\t"
      "mov.b64 %10, {r10, r11};\n\t"
      "mov.b64 %11, {r14, r15};\n\t"
      "mov.b64 %12, {r24, r25};\n\t"
      "mov.b64 %13, {r28, r29};\n\t"
      "mov.b64 %14, {r26, r27};\n\t"
      "mov.b64 %15, {r30, r31};\n\t"
      "}"
      : "=d"(x[0].r), "=d"(x[0].i), "=d"(x[1].r), "=d"(x[1].i), "=d"(x[2].r), "=d"(x[2].i), "=d"(x[3].r), "=d"(x[3].i), "=d"(x[4].r), "=d"(x[4].i), "=d"(x[5].r), "=d"(x[5].i), "=d"(x[6].r), "=d"(x[6].i), "=d"(x[7].r), "=d"(x[7].i)
      : "r"(addr), "r"(addr + (16u << 16))
      : "memory");
}
// ... and back.
__device__ __forceinline__ void turn_put_back(u32 addr, const cplx (&x)[8]) {
  asm volatile(
      "{\n\t"
      ".reg .b32 r<32>;\n\t"
      "mov.b64 {r0, r1}, %2;\n\t"
      "mov.b64 {r4, r5}, %3;\n\t"
      "mov.b64 {r2, r3}, %4;\n\t"
      "mov.b64 {r6, r7}, %5;\n\t"
      "mov.b64 {r16, r17}, %6;\n\t"
      "mov.b64 {r20, r21}, %7;\n\t"
      "mov.b64 {r18, r19}, %8;\n\t"
      "mov.b64 {r22, r23}, %9;\n\t"
      "mov.b64 {r8, r9}, %10;\n\t"
      "mov.b64 {r12, r13}, %11;\n\t"
      "mov.b64 {r10, r11}, %12;\n\t"
      "mov.b64 {r14, r15}, %13;\n\t"
      "mov.b64 {r24, r25}, %14;\n\t"
      "mov.b64 {r28, r29}, %15;\n\t"
      "mov.b64 {r26, r27}, %16;\n\t"
      "mov.b64 {r30, r31}, %17;\n\t"
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15};\n\t"
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%1], {r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31};\n\t"
      "}"
      : 
      : "r"(addr), "r"(addr + (16u << 16)), "d"(x[0].r), "d"(x[0].i), "d"(x[1].r), "d"(x[1].i), "d"(x[2].r), "d"(x[2].i), "d"(x[3].r), "d"(x[3].i), "d"(x[4].r), "d"(x[4].i), "d"(x[5].r), "d"(x[5].i), "d"(x[6].r), "d"(x[6].i), "d"(x[7].r), "d"(x[7].i)
      : "memory");
}
template <int COLS>
__device__ __forceinline__ void turn_take_back(u32 addr, cplx (&x)[8]) {
  if constexpr (COLS == 1)
    asm volatile(
        "{\n\t"
        ".reg .b32 r<32>;\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15, r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r8, r9};\n\t"
        "mov.b64 %2, {r16, r17};\n\t"
        "mov.b64 %3, {r24, r25};\n\t"
        "mov.b64 %4, {r2, r3};\n\t"
        "mov.b64 %5, {r10, r11};\n\t"
        "mov.b64 %6, {r18, r19};\n\t"
        "mov.b64 %7, {r26, r27};\n\t"
        "mov.b64 %8, {r4, r5};\n\t"
        "mov.b64 %9, {r12, r13};\n\t"
        "mov.b64 %10, {r20, r21};\n\t"
        "mov.b64 %11, {r28, r29};\n\t"
        "mov.b64 %12, {r6, r7};\n\t"
        "mov.b64 %13, {r14, r15};\n\t"
        "mov.b64 %14, {r22, r23};\n\t"
        "mov.b64 %15, {r30, r31};\n\t"
        "}"
        : "=d"(x[0].r), "=d"(x[0].i), "=d"(x[1].r), "=d"(x[1].i), "=d"(x[2].r), "=d"(x[2].i), "=d"(x[3].r), "=d"(x[3].i), "=d"(x[4].r), "=d"(x[4].i), "=d"(x[5].r), "=d"(x[5].i), "=d"(x[6].r), "=d"(x[6].i), "=d"(x[7].r), "=d"(x[7].i)
        : "r"(addr)
        : "memory");
  else
    asm volatile(
        "{\n\t"
        ".reg .b32 r<32>;\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {r0, r1, r2, r3, r4, r5, r6, r7, r8, r9, r10, r11, r12, r13, r14, r15, r16, r17, r18, r19, r20, r21, r22, r23, r24, r25, r26, r27, r28, r29, r30, r31}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "mov.b64 %1, {r8, r9};\n\t"
        "mov.b64 %2, {r2, r3};\n\t"
        "mov.b64 %3, {r10, r11};\n\t"
        "mov.b64 %4, {r4, r5};\n\t"
        "mov.b64 %5, {r12, r13};\n\t"
        "mov.b64 %6, {r6, r7};\n\t"
        "mov.b64 %7, {r14, r15};\n\t"
        "mov.b64 %8, {r16, r17};\n\t"
        "mov.b64 %9, {r24, r25};\n\t"
        "mov.b64 %10, {r18, r19};\n\t"
        "mov.b64 %11, {r26, r27};\n\t"
        "mov.b64 %12, {r20, r21};\n\t"
        "mov.b64 %13, {r28, r29};\n\t"
        "mov.b64 %14, {r22, r23};\n\t"
        "mov.b64 %15, {r30, r31};\n\t"
        "}"
        : "=d"(x[0].r), "=d"(x[0].i), "=d"(x[1].r), "=d"(x[1].i), "=d"(x[2].r), "=d"(x[2].i), "=d"(x[3].r), "=d"(x[3].i), "=d"(x[4].r), "=d"(x[4].i), "=d"(x[5].r), "=d"(x[5].i), "=d"(x[6].r), "=d"(x[6].i), "=d"(x[7].r), "=d"(x[7].i)
        : "r"(addr)
        : "memory");
}

// Layouts of the 1024 positions p = (p9 .. p0); level s works on bit 9 - s.
//          warp        lane               registers
//   C      p6 p5       p4 .. p0           p9 p8 p7    coefficients, levels 0-2
//   1      p9 p8       p3 p2 p1 p0 p7     p6 p5 p4    levels 3-5
//   2      p9 p8       p1 p0 p7 p6 p5     p4 p3 p2    levels 6, 7
//   E      p9 p8       p7 p6 p5 p3 p2     p4 p1 p0    levels 8, 9, evaluation order
// C <-> 1 goes through shared memory (M words of 16 bytes); p7 is XORed into
// address bit 2, so that neither side has bank conflicts.  A group's two
// buffers take turns: a transform writes the one that the whole group finished
// reading before the barrier of the transform in between, so one barrier per
// transform is enough.  (SPLIT has another barrier between any two transforms of a
// group, and one buffer.)  1 <-> 2 <-> E stay inside a warp and go through tensor memory:
// the shared-memory pipe, which also delivers the keys, was the busiest unit
// with them.
struct Place {
  int t, g, c, b;  // thread of group g; buffer index of its register 0 in layouts C and 1
  u32 turn;        // this warp's tensor memory for the turns
  __device__ __forceinline__ Place(int t_, int g_, u32 turn_) : t(t_), g(g_), turn(turn_) {
    const int w = t >> 5, l = t & 31;
    c = t;
    b = ((w << 8) | ((l & 1) << 7) | (l >> 1)) ^ ((l & 1) << 2);
  }
};
// The barrier of one of GROUPS groups (0 is the block's).
template <int GROUPS>
__device__ __forceinline__ void group_sync(const Place &p) {
  if (GROUPS == 1) __syncthreads();
  else if (p.g == 0) asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
  else if (p.g == 1) asm volatile("bar.sync 2, %0;" ::"n"(T) : "memory");
  else asm volatile("bar.sync 3, %0;" ::"n"(T) : "memory");
}
// register r of layout C is at p.c + 128 r, with the XOR for odd r
__device__ __forceinline__ int at_c(const Place &p, int r) { return (p.c ^ ((r & 1) << 2)) + 128 * r; }
__device__ __forceinline__ int at_1(const Place &p, int r) { return p.b + 16 * r; }

struct Nothing {
  __device__ __forceinline__ void operator()() const {}
};
// Forward transform, layout C -> E, through buffer X.  meanwhile(): loads from
// shared memory that are to run under the levels after the exchange.
template <int GROUPS, class Meanwhile = Nothing>
__device__ __forceinline__ void forward(cplx (&x)[8], cplx *X, const cplx *tw, const Place &p,
                                        const Meanwhile &meanwhile = Nothing()) {
  fwd8(x, PZ_FFT_C0);
#pragma unroll
  for (int r = 0; r < 8; r++) X[at_c(p, r)] = x[r];
  group_sync<GROUPS>(p);
#pragma unroll
  for (int r = 0; r < 8; r++) x[r] = X[at_1(p, r)];
  meanwhile();
  const int w = p.t >> 5, l = p.t & 31;
  {
    const cplx *c = tw + TW_R1 + 2 * w + (l & 1);
    fwd8(x, c[0], c[8], c[16], c[24]);
  }
  turn_put<1>(p.turn, x);
  tmem_wait_store();
  turn_take(p.turn, x);
  {
    const cplx *c = tw + TW_R2 + 8 * w + (l & 7);
    const cplx c1 = c[0], c2 = c[32], c3 = c[64];
    fwd4(x[0], x[1], x[2], x[3], c1.r, c1.i, c2);
    fwd4(x[4], x[5], x[6], x[7], -c1.i, c1.r, c3);
  }
  turn_put<2>(p.turn, x);
  tmem_wait_store();
  turn_take(p.turn, x);
  {
    const cplx *c = tw + TW_R3 + p.t;
    const cplx c1 = c[0], c2 = c[128], c3 = c[256], c4 = c[384];
    fwd4(x[0], x[1], x[2], x[3], c1.r, c1.i, c2);
    fwd4(x[4], x[5], x[6], x[7], c3.r, c3.i, c4);
  }
}

// Inverse transform (without the factor 1 / M, which the keys carry), E -> C.
template <int GROUPS>
__device__ __forceinline__ void inverse(cplx (&x)[8], cplx *X, const cplx *tw, const Place &p) {
  const int w = p.t >> 5, l = p.t & 31;
  {
    const cplx *c = tw + TW_R3 + p.t;
    const cplx c1 = c[0], c2 = c[128], c3 = c[256], c4 = c[384];
    inv4(x[0], x[1], x[2], x[3], c1.r, c1.i, c2);
    inv4(x[4], x[5], x[6], x[7], c3.r, c3.i, c4);
  }
  turn_put_back(p.turn, x);
  tmem_wait_store();
  turn_take_back<2>(p.turn, x);
  {
    const cplx *c = tw + TW_R2 + 8 * w + (l & 7);
    const cplx c1 = c[0], c2 = c[32], c3 = c[64];
    inv4(x[0], x[1], x[2], x[3], c1.r, c1.i, c2);
    inv4(x[4], x[5], x[6], x[7], -c1.i, c1.r, c3);
  }
  turn_put_back(p.turn, x);
  tmem_wait_store();
  turn_take_back<1>(p.turn, x);
  {
    const cplx *c = tw + TW_R1 + 2 * w + (l & 1);
    inv8(x, c[0], c[8], c[16], c[24]);
  }
#pragma unroll
  for (int r = 0; r < 8; r++) X[at_1(p, r)] = x[r];
  group_sync<GROUPS>(p);
#pragma unroll
  for (int r = 0; r < 8; r++) x[r] = X[at_c(p, r)];
  inv8(x, PZ_FFT_C0);
}

// small signed integer -> double without the conversion unit
__device__ __forceinline__ double i2d(int v) {
  return __hiloint2double(0x43300000, v ^ (int)0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
}

// Recombination.  z + 1.5 2^52 rounds z (|z| < 2^46) to the nearest integer
// and leaves it, in two's complement, in the low bits of the double's word.
// With h = floor(z / 2^(54 - s)) and 2^54 = 77823 (mod Q),
//   2^s z = 2^s (z mod 2^(54 - s)) + 77823 h   (mod Q)   for s = 18, 36.
constexpr double ROUND = 6755399441055744.0;      // 1.5 * 2^52
constexpr u64 ROUND_BITS = 0x4338000000000000ull;  // its word
// what the words of ROUND add to the sum of the three limbs, below
constexpr u64 ROUND_SUM = ROUND_BITS + 77823ull * (ROUND_BITS >> 36);

__device__ __forceinline__ void add_limb0(u64 &acc, double z) { acc += (u64)__double_as_longlong(z + ROUND); }
__device__ __forceinline__ void add_limb1(u64 &acc, double z) {
  const u64 w = (u64)__double_as_longlong(z + ROUND);
  acc += ((w << 18) & ((1ull << 54) - 1)) + (u64)(u32)(w >> 36) * 77823u;
}
__device__ __forceinline__ void add_limb2(u64 &acc, double z) {
  const u64 w = (u64)__double_as_longlong(z + ROUND);
  acc += ((u64)(((u32)w & 0x3ffffu) << 4) << 32) + (u64)((long long)(int)(u32)(w >> 18) * 77823ll);
}
// The sum of the limbs (once ROUND_SUM is taken off in (-2^47, 2^55 + 2^47), with
// an automorphism's b, of at most 2 Q, in (-2^56, 2^57)) -> a representative mod Q
// in [-2^53 - 2^20, 2^53 + 2^20].
__device__ __forceinline__ long long settle_sum(u64 acc) {
  const int h = ((int)(acc >> 32) + (1 << 21)) >> 22;
  return (long long)(acc - ((u64)((u32)h << 22) << 32)) + (long long)h * 77823ll;
}
__device__ __forceinline__ long long settle(u64 acc) { return settle_sum(acc - ROUND_SUM); }
// The decomposer's centred form, [-(Q + 1)/2, (Q - 3)/2] (decomposer.rs:217-234:
// v >= Q >> 1 -> v - Q), of a representative in (-1.5 Q, 1.5 Q).
__device__ __forceinline__ long long centre(long long c) {
  if (c >= (long long)(Q_N2048 >> 1)) c -= (long long)Q_N2048;
  else if (c < -(long long)((Q_N2048 + 1) >> 1)) c += (long long)Q_N2048;
  return c;
}
// how near |c| is to 2^53: at most EDGE means that centre() has nothing to do
constexpr u32 EDGE = 0x3ffffdu;
__device__ __forceinline__ u32 edge(long long c) { return (u32)((int)(c >> 32) + 0x1fffff); }
// The signed digit of a centred value: one digit above IGN dropped bits is
// the rounded quotient itself (decomposer.rs:217-300: the digit k of the
// rounded value r, less 2^LOGB when k is above half the base, or equal to it
// with the next bit set, is r again, since r lies in [-2^(LOGB - 1), 2^(LOGB - 1)]).
template <int IGN>
__device__ __forceinline__ int digit(long long c) {
  return (int)((c + (1ll << (IGN - 1))) >> IGN);
}
// The decomposer's signed digit of any 64-bit word (one outside [0, Q) may
// round above half the base).
template <int LOGB, int IGN>
__device__ __forceinline__ int digit_any(u64 v) {
  if (v >= (Q_N2048 >> 1)) v = v - Q_N2048;
  const u32 r = (u32)(v >> IGN) + (u32)((v >> (IGN - 1)) & 1ull);
  const u32 k = r & ((1u << LOGB) - 1u), half = 1u << (LOGB - 1);
  const bool c = k > half || (k == half && ((r >> LOGB) & 1u));
  return (int)k - (c ? (1 << LOGB) : 0);
}
static_assert(RLRG_LOGB + RLRG_IGN == 54 && AUTO_LOGB + AUTO_IGN == 54, "one digit covers Q");

// ---------------------------------------------------------------------------
// Key form: device rows (evaluation domain, K N^{-1}) back to coefficients, cut
// into limbs, and each limb transformed in double-double arithmetic, scaled by
// 1 / M (exact) and rounded once.  CTAs of 256 threads.
// ---------------------------------------------------------------------------
// Double-double arithmetic (Dekker 1971; the two-sum Knuth's, the product's low
// part by a fused multiply-add).
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

constexpr size_t KEY_SMEM = 4 * M * sizeof(double);  // re, im: high and low parts
// position e in layout E
__device__ __forceinline__ int eval_thread(int e) { return ((e >> 8) << 5) | (((e >> 5) & 7) << 2) | ((e >> 2) & 3); }
__device__ __forceinline__ int eval_register(int e) { return (((e >> 4) & 1) << 2) | (e & 3); }

// coef (shared, N words) = the row's coefficients times 2^up mod Q
__device__ __forceinline__ void key_coefficients(const u64 *row, u64 *coef, const RingConsts &rc, int up) {
  const int j = threadIdx.x;
  u64 x[8];
#pragma unroll
  for (int r = 0; r < 8; r++) x[r] = row[dev_index<11>(j, r)];
  ntt_inv<11>(x, coef, rc);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; r++) {
    u64 v = reduce2(x[r], Q_N2048);
    if (up) v = reduce2(reduce_n2048(((v & ((1ull << (54 - up)) - 1)) << up) + 77823ull * (v >> (54 - up))), Q_N2048);
    coef[pos_coef<11>(j, r)] = v;
  }
}
// work (shared) = the transform of limb `limb` of LIMBS_ limbs of BITS bits
template <int LIMBS_, int BITS>
__device__ __forceinline__ void key_limb(const u64 *coef, int limb, double *work, const double4 *tw) {
  double *re_h = work, *re_l = work + M, *im_h = work + 2 * M, *im_l = work + 3 * M;
  const int j = threadIdx.x;
  auto cut = [&](u64 u) -> double {
    long long v = u > (Q_N2048 >> 1) ? (long long)(u - Q_N2048) : (long long)u, k = 0;
    for (int l = 0; l <= limb; l++) {
      k = l + 1 < LIMBS_ ? ((v + (1 << (BITS - 1))) & ((1 << BITS) - 1)) - (1 << (BITS - 1)) : v;
      v = (v - k) >> BITS;
    }
    return (double)k;
  };
  __syncthreads();
  for (int e = j; e < M; e += 256) {
    re_h[e] = cut(coef[e]);
    im_h[e] = cut(coef[e + M]);
    re_l[e] = im_l[e] = 0;
  }
  for (int s = 0; s < 10; s++) {
    const int half = M >> (s + 1);
    __syncthreads();
    for (int e = j; e < M / 2; e += 256) {
      const int k = e >> (9 - s), a = k * 2 * half + (e & (half - 1)), b = a + half;
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
}
__device__ __forceinline__ cplx key_value(const double *work, int e) {
  return cplx{work[e] * (1.0 / M), work[2 * M + e] * (1.0 / M)};
}

}  // namespace fft
}  // namespace pz
