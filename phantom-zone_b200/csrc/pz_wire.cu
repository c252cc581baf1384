// pz_wire.cu -- wire formats (the reference has none): device-form server
// keys and circuits as flat byte strings, for checkpoint / restore and for
// handing work between processes of a serving deployment.
//
// Key blob: a 64-byte header followed by the device-form arrays exactly as
// they sit in device memory (RGSW and auto keys in the evaluation domain,
// scaled by the context's key-form constant -- N^{-1}, or N^{-1} 2^64 for
// Montgomery products -- in the per-thread layout; the LWE KSK as u32 rows
// of ks_stride words).  The evaluation domain depends on the NTT root and
// the scale on the build's multiply-accumulate reduction, so the header
// (version 2) records both and an import into a context with another root,
// key form or parameter set is refused.  Import is a plain copy, and the
// key's derived forms (KSK byte planes, FFT form) made from it on the device.
//
// (The circuit blob lives with the circuit in pz_circuit.cu.)
#include <cstring>
#include <vector>

#include "pz_internal.h"

using pz::u32;
using pz::u64;

namespace {

constexpr u64 KEY_MAGIC = 0x31305945594b5a50ull;  // "PZKEY01"

struct KeyHeader {
  u64 magic;
  u32 version, param_id;
  u64 root;
  u64 rgsw_bytes, autos_bytes, ksk_bytes;
  u64 key_form;  // the scale of the RGSW and auto key rows (br_conv_c)
  u64 reserved;
};
static_assert(sizeof(KeyHeader) == 64, "key header is 64 bytes");

void key_sizes(const pz_ctx *c, size_t *rgsw, size_t *autos, size_t *ksk) {
  const pz_params &P = c->P;
  *rgsw = (size_t)P.lwe_n * P.rgsw_rows * P.rlwe_n * 8;
  *autos = (size_t)P.n_auto_keys * P.auto_rows * P.rlwe_n * 8;
  *ksk = (size_t)P.lwe_d * P.rlwe_n * pz::ks_stride(P) * 4;
}

// Whether a blob is a key of this context's.
pz_status check_blob(pz_ctx *c, const void *buf, size_t size) {
  KeyHeader h;
  if (size < sizeof h) return pz::fail(c, PZ_ERR_INVALID_ARGUMENT, "pz_key_import: truncated blob");
  memcpy(&h, buf, sizeof h);
  size_t rg, au, ks;
  key_sizes(c, &rg, &au, &ks);
  if (h.magic != KEY_MAGIC || h.version < 1 || h.version > 2)
    return pz::fail(c, PZ_ERR_INVALID_ARGUMENT, "pz_key_import: not a key blob");
  // version 1 blobs carried Montgomery-form rows without recording it
  const u64 form = h.version == 1 ? c->conv_c : h.key_form;
  if (form != c->br_conv_c)
    return pz::fail(c, PZ_ERR_KEY_MISMATCH, "pz_key_import: key rows in another device form (other build)");
  if (h.param_id != (u32)c->param_id) return pz::fail(c, PZ_ERR_KEY_MISMATCH, "pz_key_import: other parameter set");
  if (h.root != c->root) return pz::fail(c, PZ_ERR_KEY_MISMATCH, "pz_key_import: exported under another NTT root");
  if (h.rgsw_bytes != rg || h.autos_bytes != au || h.ksk_bytes != ks || size != sizeof h + rg + au + ks)
    return pz::fail(c, PZ_ERR_INVALID_ARGUMENT, "pz_key_import: sizes do not match the parameter set");
  return PZ_OK;
}

cudaError_t copy_in(u64 **dst, const unsigned char *src, size_t bytes) {
  cudaError_t e = pz::dev_malloc(dst, bytes);
  return e == cudaSuccess ? cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice) : e;
}
template <typename T>
void drop(pz_key *k, T **p, size_t bytes) {
  if (*p) k->bytes -= bytes;
  cudaFree(*p);
  *p = nullptr;
}

}  // namespace

namespace pz {
ManagedBytes managed_key_bytes(const pz_ctx *c) {
  size_t rg, au, ks;
  key_sizes(c, &rg, &au, &ks);
  const size_t planes = ksk8_bytes(c), ksk = planes ? planes : ks;
  const bool fft = c->d_fft && c->key_fft;
  return {rg + au + ksk, fft ? fft_key_bytes(c->P.lwe_n) + fft_key_bytes(c->P.n_auto_keys) + ksk : rg + au + ksk};
}

// The integer rows of k, from the blob.
static cudaError_t load_rows(pz_key *k, const void *blob) {
  size_t rg, au, ks;
  key_sizes(k->ctx, &rg, &au, &ks);
  const unsigned char *p = (const unsigned char *)blob + sizeof(KeyHeader);
  cudaError_t e = copy_in(&k->d_rgsw, p, rg);
  if (e == cudaSuccess) e = copy_in(&k->d_autos, p + rg, au);
  if (e == cudaSuccess) k->bytes += rg + au;
  return e;
}
// The FFT form in the place of the integer rows, if there is memory for it.
static cudaError_t rows_to_fft(pz_key *k) {
  size_t rg, au, ks;
  key_sizes(k->ctx, &rg, &au, &ks);
  const cudaError_t e = build_fft_key(k->ctx, k, k->ctx->stream);
  if (k->d_fft_rgsw) {
    drop(k, &k->d_rgsw, rg);
    drop(k, &k->d_autos, au);
  }
  return e;
}

pz_status managed_import(pz_ctx *c, const void *blob, size_t size, bool fft, pz_key **out) {
  *out = nullptr;
  const pz_status s = check_blob(c, blob, size);
  if (s != PZ_OK) return s;
  std::lock_guard<std::mutex> lock(c->mu);
  PZ_CK(c, cudaSetDevice(c->device));
  size_t rg, au, ks;
  key_sizes(c, &rg, &au, &ks);
  pz_key *k = new pz_key();
  k->ctx = c;
  // each form in the place of what it was made from, so that little more than the
  // key's bytes is held at a time
  cudaError_t e = dev_malloc(&k->d_ksk, ks);
  if (e == cudaSuccess)
    e = cudaMemcpy(k->d_ksk, (const unsigned char *)blob + sizeof(KeyHeader) + rg + au, ks, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) k->bytes = ks;
  if (e == cudaSuccess) e = build_ksk8(c, k, c->stream);
  if (k->d_ksk8) drop(k, &k->d_ksk, ks);
  if (e == cudaSuccess) e = load_rows(k, blob);
  if (e == cudaSuccess && fft) e = rows_to_fft(k);
  if (e != cudaSuccess) {
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    free_key_arrays(k);
    delete k;
    return cuda_fail(c, "managed key import", e);
  }
  *out = k;
  return PZ_OK;
}

pz_status managed_to_integer(pz_key *k, const void *blob) {
  pz_ctx *c = k->ctx;
  std::lock_guard<std::mutex> lock(c->mu);
  PZ_CK(c, cudaSetDevice(c->device));
  const size_t au = fft_key_bytes(c->P.n_auto_keys);
  drop(k, &k->d_fft_rgsw, fft_key_bytes(c->P.lwe_n));
  drop(k, &k->d_fft_autos, au);
  PZ_CK(c, load_rows(k, blob));
  return PZ_OK;
}

pz_status managed_to_fft(pz_key *k) {
  std::lock_guard<std::mutex> lock(k->ctx->mu);
  PZ_CK(k->ctx, cudaSetDevice(k->ctx->device));
  PZ_CK(k->ctx, rows_to_fft(k));
  return PZ_OK;
}
}  // namespace pz

extern "C" {

pz_status pz_key_export(const pz_key *k, void *buf, size_t capacity, size_t *size) {
  if (!k || !size) return PZ_ERR_INVALID_ARGUMENT;
  pz_ctx *c = k->ctx;
  size_t rg, au, ks;
  key_sizes(c, &rg, &au, &ks);
  const size_t total = sizeof(KeyHeader) + rg + au + ks;
  *size = total;
  if (!buf) return PZ_OK;  // size query
  if (capacity < total) return pz::fail(c, PZ_ERR_INVALID_ARGUMENT, "pz_key_export: buffer too small");
  PZ_CK(c, cudaSetDevice(c->device));
  KeyHeader h{};
  h.magic = KEY_MAGIC;
  h.version = 2;
  h.key_form = c->br_conv_c;
  h.param_id = (u32)c->param_id;
  h.root = c->root;
  h.rgsw_bytes = rg;
  h.autos_bytes = au;
  h.ksk_bytes = ks;
  unsigned char *p = (unsigned char *)buf;
  memcpy(p, &h, sizeof h);
  p += sizeof h;
  PZ_CK(c, cudaMemcpy(p, k->d_rgsw, rg, cudaMemcpyDeviceToHost));
  PZ_CK(c, cudaMemcpy(p + rg, k->d_autos, au, cudaMemcpyDeviceToHost));
  PZ_CK(c, cudaMemcpy(p + rg + au, k->d_ksk, ks, cudaMemcpyDeviceToHost));
  return PZ_OK;
}

pz_status pz_key_import(pz_ctx *c, const void *buf, size_t size, pz_key **out) {
  if (!c || !buf || !out) return PZ_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  const pz_status s = check_blob(c, buf, size);
  if (s != PZ_OK) return s;
  size_t rg, au, ks;
  key_sizes(c, &rg, &au, &ks);
  std::lock_guard<std::mutex> lock(c->mu);
  PZ_CK(c, cudaSetDevice(c->device));
  pz_key *k = new pz_key();
  k->ctx = c;
  k->bytes = rg + au + ks;
  const unsigned char *p = (const unsigned char *)buf + sizeof(KeyHeader);
  cudaError_t e = pz::dev_malloc(&k->d_rgsw, rg);
  if (e == cudaSuccess) e = pz::dev_malloc(&k->d_autos, au);
  if (e == cudaSuccess) e = pz::dev_malloc(&k->d_ksk, ks);
  if (e == cudaSuccess) e = cudaMemcpy(k->d_rgsw, p, rg, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(k->d_autos, p + rg, au, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(k->d_ksk, p + rg + au, ks, cudaMemcpyHostToDevice);
  // derived on the device; the blob carries only the u32 rows and the integer form
  if (e == cudaSuccess) e = pz::build_key_forms(c, k, c->stream);
  if (e != cudaSuccess) {
    pz::free_key_arrays(k);
    delete k;
    return pz::cuda_fail(c, "pz_key_import", e);
  }
  *out = k;
  return PZ_OK;
}

}  // extern "C"
