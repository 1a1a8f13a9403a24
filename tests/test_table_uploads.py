"""Tables are on the device when the call that makes them returns. hb_boot_tc.cu, compiled for the host side of a fake
CUDA runtime in which a copy lands only when its stream is waited for (as the runtime may do with pageable
memory, the legacy stream included): after tc_tables no copy may be outstanding, whatever stream a launch then
takes, and the context's own stream was not waited for. Where the copy fails the buffer is given back and the
context has no tables. The other copies of the library name their stream too."""

import glob
import os
import re
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hasteboots_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>
#include "hb_runtime.h"

static int failing, live;
static std::vector<cudaStream_t> waited;
struct Copy { void *dst; std::vector<char> words; cudaStream_t stream; };
static std::vector<Copy> queue;
static cudaError_t copy(void *dst, const void *src, size_t n, cudaStream_t st) {
  if (failing) return cudaErrorUnknown;
  queue.push_back({dst, std::vector<char>((const char *)src, (const char *)src + n), st});
  return cudaSuccess;
}
extern "C" {
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return copy(d, s, n, nullptr); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) { return copy(d, s, n, st); }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  waited.push_back(st);
  std::vector<Copy> left;
  for (auto &c : queue)
    if (c.stream == st) memcpy(c.dst, c.words.data(), c.words.size()); else left.push_back(c);
  queue = left;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t *, const void *) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { static void *p; return &p; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
char __cudaInitModule(void **) { return 1; }
}
namespace hbrt {
int cuda_fail(hb_ctx *, cudaError_t, const char *) { return HB_ERR_CUDA; }
long long wait_budget(const hb_ctx *) { return 0; }
uint32_t ks_dim(const hb_params &) { return 1024; }
cudaError_t dev_constant(hb_ctx *ctx, size_t bytes, void **out) {
  *out = calloc(1, bytes);
  ++live;
  ctx->sizes.push_back({*out, 0});
  return cudaSuccess;
}
void dev_free(hb_ctx *ctx, void *p) {
  if (!p) return;
  --live;
  ctx->sizes.clear();
  free(p);
}
int tables(hb_ctx *ctx, int f, uint32_t logn, DevTables **out, uint32_t logv) {
  DevTables &t = ctx->tables[f][logn][logv];
  t.psi = 7;  // any odd word: the values do not matter here
  *out = &t;
  return HB_OK;
}
}
int main(int, char **argv) {
  hb_ctx ctx;
  ctx.stream = (cudaStream_t)0x1000;
  ctx.uploads = (cudaStream_t)0x2000;

  failing = argv[1][0] == 'f';
  hbrt::tc_tables(&ctx, HB_FIELD_GOLDILOCKS, 1024);
  int waits_for_work = 0, words = 0;
  for (auto st : waited) waits_for_work += st == ctx.stream;
  if (ctx.tc_tables) words = ((unsigned char *)ctx.tc_tables)[0];
  printf("%d %d %d %d %d\n", (int)queue.size(), waits_for_work, ctx.tc_tables != nullptr, live, words);
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver():
    nvcc = os.environ.get("NVCC", "nvcc")
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    d = tempfile.mkdtemp()
    src, obj, exe = (os.path.join(d, f) for f in ("driver.cpp", "tc.o", "driver"))
    open(src, "w").write(DRIVER)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-c",
                    os.path.join(CSRC, "hb_boot_tc.cu"), "-o", obj], check=True)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", src, obj, "-o", exe], check=True)
    return exe


def _run(driver, what):
    return [int(x) for x in subprocess.run([driver, what], capture_output=True, text=True, check=True).stdout.split()]


def test_tensor_tables_are_there_when_the_call_returns(driver):
    outstanding, waits_for_work, there, live, first_byte = _run(driver, "copy")
    assert outstanding == 0 and there == 1 and live == 1
    assert waits_for_work == 0
    assert first_byte == 1  # the entry psi^0


def test_a_failed_copy_gives_the_buffer_back(driver):
    outstanding, _, there, live, _ = _run(driver, "fail")
    assert (outstanding, there, live) == (0, 0, 0)


def test_no_copy_on_the_legacy_stream():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert not re.search(r"\bcudaMem(cpy|set)\(", open(path).read()), path
