// hb_boot_tc.cu -- constant tables and launches of the tensor-core bootstrapping kernel
// (hb_boot_tc.cuh).

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "../../include/hb_gpu.h"
#include "hb_boot_tc.cuh"
#include "hb_launch.cuh"
#include "hb_runtime.h"

using hb::GateJob;
using F = hb::Goldilocks;
using Geo = hb::TcGeo;

namespace hbrt {
namespace {

uint32_t brv(uint32_t x, uint32_t bits) {
  uint32_t r = 0;
  for (uint32_t b = 0; b < bits; ++b) r |= ((x >> b) & 1u) << (bits - 1 - b);
  return r;
}

// The byte matrices of both passes in the operand layout of hb_tc.cuh and the twist between them, for
// the primitive 2N-th root psi of the field's NTT tables.
std::vector<unsigned char> build_tc(uint64_t psi) {
  constexpr uint32_t N = Geo::N;
  std::vector<uint64_t> pw(2 * N);
  pw[0] = 1;
  for (uint32_t i = 1; i < 2 * N; ++i) pw[i] = hb::host_mulmod<F>(pw[i - 1], psi);
  std::vector<unsigned char> t(Geo::TAB_BYTES, 0);
  unsigned char *b1 = t.data(), *b2 = b1 + Geo::B1_BYTES;
  uint64_t *tw = reinterpret_cast<uint64_t *>(b2 + Geo::B2_BYTES);
  for (uint32_t a = 0; a < 64; ++a) {
    const uint32_t k1 = brv(a, 6);
    for (uint32_t j1 = 0; j1 < 64; ++j1) {
      const uint64_t w = pw[16 * j1 * (2 * k1 + 1) % (2 * N)];
      for (uint32_t c = 0; c < 8; ++c) b1[(j1 / 16) * Geo::B1_LBO + (a * 8 + c) * 16 + j1 % 16] = (unsigned char)(w >> (8 * c));
    }
    for (uint32_t j0 = 0; j0 < 16; ++j0) tw[a * 16 + j0] = pw[j0 * (2 * k1 + 1) % (2 * N)];
  }
  for (uint32_t q = 0; q < 16; ++q) {  // column group q: slot b = (q >> 1) + 8 (q & 1)
    const uint32_t k0 = brv((q >> 1) + 8 * (q & 1), 4);
    for (uint32_t j0 = 0; j0 < 16; ++j0) {
      uint64_t w = pw[128 * k0 * j0 % (2 * N)];
      for (uint32_t i = 0; i < 8; ++i) {  // byte i of the pass-2 input: the entry times 2^(8 i)
        const uint32_t k = j0 * 8 + i;
        for (uint32_t c = 0; c < 8; ++c) b2[(k / 16) * Geo::B2_LBO + (q * 8 + c) * 16 + k % 16] = (unsigned char)(w >> (8 * c));
        w = hb::host_mulmod<F>(w, (uint64_t)256);
      }
    }
  }
  return t;
}

template <bool KSC, bool EXT = false>
int launch(hb_ctx *ctx, const hb::BootParams<uint64_t> &prm, const unsigned char *tab, cudaStream_t stream,
           const hb::TcExt &ext = {}) {
  auto kern = hb::bootstrap_tc_kernel<KSC, EXT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Geo::SMEM);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "bootstrap smem attribute");
  const unsigned grid = std::max(1u, std::min<unsigned>(prm.total_batches, (unsigned)ctx->sms));
  kern<<<grid, Geo::THREADS + Geo::AUX, Geo::SMEM, stream>>>(prm, tab, ext);
  e = cudaGetLastError();
  return e == cudaSuccess ? HB_OK : cuda_fail(ctx, e, "bootstrap launch");
}

}  // namespace

void tc_tables(hb_ctx *ctx, int field_id, uint32_t ring_dim) {
  if (ctx->tc_tables || field_id != HB_FIELD_GOLDILOCKS || ring_dim != Geo::N) return;
  DevTables *tb;
  if (tables(ctx, field_id, Geo::LOGN, &tb, 3)) return;
  const std::vector<unsigned char> t = build_tc(tb->psi);
  void *d = nullptr;
  // without room for them the butterfly form runs; the error is not the caller's
  cudaError_t e = dev_constant(ctx, t.size(), &d);
  if (e == cudaSuccess && (e = upload(ctx, d, t.data(), t.size())) != cudaSuccess) dev_free(ctx, d);
  if (e == cudaSuccess)
    ctx->tc_tables = d;
  else
    cudaGetLastError();
}

bool tc_applies(const hb_ctx *ctx, const hb_params &p, int T, int G) {
  return ctx->tc_tables && p.field_id == HB_FIELD_GOLDILOCKS && T == 128 && G == Geo::G && !p.lwe_ternary && p.ring_dim == Geo::N &&
         p.br_bits <= 8 && p.ks_bits <= 8;
}

int launch_tc(hb_ctx *ctx, const hb_keys *keys, const GateJob *djobs, int njobs, uint32_t batches, int *status,
              cudaStream_t stream) {
  const DevTables *tb = &ctx->tables[HB_FIELD_GOLDILOCKS][Geo::LOGN][3];  // built with the keys, as the tensor tables
  const unsigned char *tab = (const unsigned char *)ctx->tc_tables;
  hb::BootParams<uint64_t> prm{};
  boot_params(prm, ctx, keys, tb);
  prm.jobs = djobs;
  prm.njobs = njobs;
  prm.total_batches = batches;
  if (status) prm.status = status;
  return ks_dim(keys->p) < keys->p.ring_dim ? launch<true>(ctx, prm, tab, stream) : launch<false>(ctx, prm, tab, stream);
}

int launch_tc_ext(hb_ctx *ctx, const void *rgsw, uint32_t bits, uint32_t len, const void *in, void *out, size_t count) {
  const DevTables *tb = &ctx->tables[HB_FIELD_GOLDILOCKS][Geo::LOGN][3];
  const unsigned char *tab = (const unsigned char *)ctx->tc_tables;
  hb::BootParams<uint64_t> prm{};
  prm.bsk = (const uint64_t *)rgsw;
  prm.tw = (const uint64_t *)tb->tw;
  prm.itw = (const uint64_t *)tb->itw;
  prm.len = len;
  prm.bits = bits;
  prm.status = ctx->d_status;
  prm.budget = wait_budget(ctx);
  prm.withhold = ctx->withhold_keys;
  // at most 2^32 - 1 batches a launch
  for (size_t at = 0; at < count;) {
    const size_t part = std::min(count - at, (size_t)0xFFFFFF00u * Geo::G);
    prm.total_batches = (uint32_t)((part + Geo::G - 1) / Geo::G);
    const int rc = launch<false, true>(ctx, prm, tab, ctx->stream,
                                       {(const uint64_t *)in + at * 2 * Geo::N, (uint64_t *)out + at * 2 * Geo::N, part});
    if (rc) return rc;
    at += part;
  }
  return HB_OK;
}

}  // namespace hbrt
