// hb_runtime.h -- host-side context and key handles shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <string>
#include <utility>
#include <vector>

#include "../../include/hb_gpu.h"
#include "hb_shape.h"

namespace hb {
struct GateJob;
}

namespace hbrt {

struct DevTables {
  void *tw = nullptr;   // N entries of F::Tw: psi^brv(k) (the 32-bit fields: with its Shoup quotient)
  void *itw = nullptr;  // psi^-brv(k), the same way
  unsigned long long n_inv = 0;      // multiplier giving x * N^-1
  unsigned long long key_scale = 0;  // multiplier applied to key words at upload
  unsigned long long psi = 0;        // the primitive 2N-th root of the tables
};

struct Scratch {
  void *ptr = nullptr;
  size_t cap = 0;
};

}  // namespace hbrt

struct hb_ctx {
  int device = 0;
  int sms = 148;
  cudaStream_t stream = nullptr;
  cudaStream_t uploads = nullptr;  // copies of tables (hbrt::upload)
  int *d_status = nullptr;
  size_t budget = 0;
  size_t in_use = 0;
  std::vector<std::pair<void *, size_t>> sizes;
  std::string err;
  hbrt::DevTables tables[3][13][6];  // [field][log2 N][log2 words per thread]
  void *tc_tables = nullptr;                    // byte matrices of bootstrap_tc_kernel
  hbrt::Scratch jobs, io, mux_tmp;
  std::atomic<unsigned long long> launches{0};  // bootstrap kernel launches issued by this context
  long long wait_limit = 0;                     // SM clock cycles per bounded wait; 0 = default
  int withhold_keys = 0;                        // test hook: bootstrap launches issue no key copies
  // latency-form clusters the GPU holds with one cluster CTA per SM ([Goldilocks, 32-bit fields] x
  // [T = 64, 128]); -1 unknown. Atomic: the serving loop's worker thread launches on the context too.
  std::atomic<int> dp_clusters[4] = {-1, -1, -1, -1};
  // device address of the allocation-free MUX's in-library array, looked up by the first such call
  // on this context (a context made after a device reset looks it up again)
  void *noalloc_addr = nullptr;
};

struct hb_keys {
  hb_params p{};
  void *bsk = nullptr;
  void *ksk = nullptr;
  size_t bytes = 0;
  int threads_per_gate = 64;  // T: key slot layout and kernel group size
  int gates_per_cta = 4;      // persistent-kernel variant (autotuned)
  double gates_per_s = 0;   // measured by hb_autotune (0: not calibrated)
};

namespace hbrt {
int fail(hb_ctx *ctx, int code, const char *fmt, ...);
int cuda_fail(hb_ctx *ctx, cudaError_t e, const char *what);
int dev_alloc(hb_ctx *ctx, size_t bytes, void **out);
cudaError_t dev_constant(hb_ctx *ctx, size_t bytes, void **out);
// Host words to the device, there for every stream when this returns and not waiting for the context's work. (A
// copy on the legacy stream from pageable memory may return once the words are staged, and the library's streams
// are not ordered behind that stream.)
inline cudaError_t upload(const hb_ctx *ctx, void *dst, const void *src, size_t bytes) {
  const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->uploads);
  return e == cudaSuccess ? cudaStreamSynchronize(ctx->uploads) : e;
}
void dev_free(hb_ctx *ctx, void *p);
int scratch(hb_ctx *ctx, Scratch &s, size_t bytes);
int tables(hb_ctx *ctx, int field_id, uint32_t logn, DevTables **out, uint32_t logv = 4);
int check_status(hb_ctx *ctx);
long long wait_budget(const hb_ctx *ctx);
// The key switch's dimension n' = next_pow2(n) (fhe_core/src/key_switch/rlwe.rs:40-43).
uint32_t ks_dim(const hb_params &p);
// A launch of a key set's jobs: its shape (hb_shape.h; shared: among other launches), the jobs laid out in its batches (their number), and one
// persistent bootstrapping launch over the job table on the device.
hb::LaunchShape launch_shape(const hb_ctx *ctx, const hb_keys *keys, const std::vector<hb::GateJob> &jobs, bool shared);
uint32_t lay_out(std::vector<hb::GateJob> &jobs, int gates_per_cta);
int launch_set(hb_ctx *ctx, hb_keys *keys, hb::LaunchShape shape, const hb::GateJob *djobs, int njobs,
               uint32_t batches, cudaStream_t stream);
// The tensor-core form of the persistent kernel (hb_boot_tc.cu): its tables, built with the keys (where they
// cannot be, or on a context that did not prepare the keys, the butterfly form serves); whether it covers a
// parameter set under a (T, G) variant; one launch over a device job table in place
// (status: another status word than the context's, or null).
void tc_tables(hb_ctx *ctx, int field_id, uint32_t ring_dim);
bool tc_applies(const hb_ctx *ctx, const hb_params &p, int T, int G);
int launch_tc(hb_ctx *ctx, const hb_keys *keys, const hb::GateJob *djobs, int njobs, uint32_t batches, int *status,
              cudaStream_t stream);
// External products over Goldilocks, N = 1024, bases up to 2^8, on a context with the tables.
int launch_tc_ext(hb_ctx *ctx, const void *rgsw, uint32_t bits, uint32_t len, const void *in, void *out, size_t count);
// The job record of `count` single-bootstrap gates (NAND..MAJORITY) of parameter set p.
int gate_job(const hb_params &p, int gate, const void *c0, const void *c1, const void *c2, void *out,
             uint32_t count, hb::GateJob *job);
}  // namespace hbrt
