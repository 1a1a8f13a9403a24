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

template <bool KSC>
int launch(hb_ctx *ctx, const hb::BootParams<uint64_t> &prm, const unsigned char *tab, cudaStream_t stream) {
  auto kern = hb::bootstrap_tc_kernel<KSC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Geo::SMEM);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "bootstrap smem attribute");
  const unsigned grid = std::max(1u, std::min<unsigned>(prm.total_batches, (unsigned)ctx->sms));
  kern<<<grid, Geo::THREADS + Geo::AUX, Geo::SMEM, stream>>>(prm, tab);
  e = cudaGetLastError();
  return e == cudaSuccess ? HB_OK : cuda_fail(ctx, e, "bootstrap launch");
}

}  // namespace

int tc_tables(hb_ctx *ctx, const hb_params &p) {
  if (ctx->tc_tables || p.field_id != HB_FIELD_GOLDILOCKS || p.ring_dim != Geo::N) return HB_OK;
  DevTables *tb;
  int rc = tables(ctx, p.field_id, Geo::LOGN, &tb, 3);
  if (rc) return rc;
  const std::vector<unsigned char> t = build_tc(tb->psi);
  void *d = nullptr;
  rc = dev_alloc(ctx, t.size(), &d);
  if (rc) return rc;
  const cudaError_t e = cudaMemcpy(d, t.data(), t.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    dev_free(ctx, d);
    return cuda_fail(ctx, e, "tensor table upload");
  }
  ctx->tc_tables = d;
  return HB_OK;
}

bool tc_applies(const hb_params &p, int T, int G) {
  return p.field_id == HB_FIELD_GOLDILOCKS && T == 128 && G == Geo::G && !p.lwe_ternary && p.ring_dim == Geo::N &&
         p.br_bits <= 8 && p.ks_bits <= 8;
}

int launch_tc(hb_ctx *ctx, const hb_keys *keys, const GateJob *djobs, int njobs, uint32_t batches, int *status,
              cudaStream_t stream) {
  const DevTables *tb = &ctx->tables[HB_FIELD_GOLDILOCKS][Geo::LOGN][3];  // built with the keys, as the tensor tables
  const unsigned char *tab = (const unsigned char *)ctx->tc_tables;
  if (!tb->tw || !tab) return fail(ctx, HB_ERR_INVALID, "keys were not prepared on this context");
  hb::BootParams<uint64_t> prm{};
  boot_params(prm, ctx, keys, tb);
  prm.jobs = djobs;
  prm.njobs = njobs;
  prm.total_batches = batches;
  if (status) prm.status = status;
  return ks_dim(keys->p) < keys->p.ring_dim ? launch<true>(ctx, prm, tab, stream) : launch<false>(ctx, prm, tab, stream);
}

}  // namespace hbrt
