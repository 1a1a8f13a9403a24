// hb_shape.h -- the shapes of launches. Of one over a list of jobs (a batch, a serving wave, a layer of the
// allocation-free MUX): gates per CTA, and the butterfly or the tensor-core form; batches of a launch do not span
// jobs, so jobs of a few gates leave every batch short. Of a batch of external products: which form takes which.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace hb {

struct LaunchShape {
  int gates_per_cta;
  bool tensor;
};

// How long a batch holds its CTA by the gates in it, in halves of what one more gate adds. Measured on B200, ms of a
// batch of 1, 2, 3, 4 gates in the butterfly form with 128 threads a gate: GOLDILOCKS 28.7, 38.3, 50.0, 63.7, ZAMA 43.2,
// 58.5, 76.5, 97.5; the tensor-core form lasts its four gates whether they are there or not: 45.8 and 69.5. With 64
// threads (two warps) a gate, two gates last as long as one: 2, 4, 6, 8 of DEFAULT_TERNARY 26.4, 32.2, 43.9, 57.0, BABYBEAR
// 12.1, 15.4, 19.9, 23.7, CUSTOM_TERNARY 7.4, 9.0, 12.5, 15.4.
constexpr uint32_t kTensorBatch = 8;
inline uint32_t batch_lasts(uint32_t gates, int threads_per_gate, bool tensor) {
  if (tensor) return kTensorBatch;
  return threads_per_gate >= 128 ? 2 * gates + 3 : (gates + 1) / 2 * 4 + 4;
}

// How long a launch of its own lasts, its longest CTA (CTA i of sms takes batches i, i + sms, ...), and how long it holds
// SMs in all.
struct LaunchLasts {
  uint64_t longest, total;
};
inline LaunchLasts launch_lasts(const std::vector<uint32_t> &counts, uint64_t sms, int gates_per_cta, int threads_per_gate,
                                bool tensor) {
  std::vector<uint64_t> cta(sms, 0);
  uint64_t at = 0, total = 0;
  for (uint32_t c : counts)
    while (c) {
      const uint32_t b = std::min<uint32_t>(c, (uint32_t)gates_per_cta), lasts = batch_lasts(b, threads_per_gate, tensor);
      cta[at] += lasts;
      total += lasts;
      at = at + 1 == sms ? 0 : at + 1;
      c -= b;
    }
  return {*std::max_element(cta.begin(), cta.end()), total};
}

// tuned: the keys' variant; variants: the batched ones compiled for them and their group size; tensor: whether the
// tensor-core form covers the keys under `tuned`; latency: whether the one-gate form may be taken; shared: whether
// other launches (of other key sets, of the wave before) take the SMs that this one leaves.
//
// One gate per CTA while every gate gets an SM of its own. Else a launch of its own takes the tensor-core form or the
// variant, up to the tuned one, that is over first, the smallest of those that last the same (absent groups of a larger
// CTA poll for keys). What one shape for all job lists cost: 300 GOLDILOCKS jobs of one gate 87 ms in the butterfly
// form, 137 in the tensor-core form, of three gates 150 and 137; 40 DEFAULT_TERNARY jobs of 30 gates 87 ms six per CTA,
// 113 eight. Among other launches it takes the form that holds SMs for less, and the smallest variant whose CTAs, were
// they full, got an SM each (24 jobs of BABYBEAR, GOLDILOCKS and ZAMA in one graph: 277 ms, 282 with the BABYBEAR
// launch of 1179 gates cut in sixes, its shortest alone).
inline LaunchShape launch_shape(const std::vector<uint32_t> &counts, uint64_t sms, int tuned, std::vector<int> variants,
                                int threads_per_gate, bool tensor, bool latency, bool shared) {
  uint64_t gates = 0;
  for (uint32_t c : counts) gates += c;
  if (tuned <= 1 || (latency && gates <= sms)) return {1, false};
  std::sort(variants.begin(), variants.end());
  LaunchLasts tc{~0ull, ~0ull};
  if (tensor) tc = launch_lasts(counts, sms, tuned, threads_per_gate, true);
  if (shared) {
    if (tensor && tc.total <= launch_lasts(counts, sms, tuned, threads_per_gate, false).total) return {tuned, true};
    for (int g : variants)
      if (g <= tuned && (gates + (uint64_t)g - 1) / (uint64_t)g <= sms) return {g, false};
    return {tuned, false};
  }
  LaunchShape best{tuned, tensor};
  uint64_t shortest = tc.longest;
  for (int g : variants) {
    if (g > tuned) break;
    const uint64_t lasts = launch_lasts(counts, sms, g, threads_per_gate, false).longest;
    if (lasts < shortest) {
      shortest = lasts;
      best = {g, false};
    }
  }
  return best;
}

// External products over Goldilocks, N = 1024, digits of a byte: how many of the last RLWEs the butterfly form takes,
// the tensor-core form the whole rounds of four per SM before them. The latter lasts four RLWEs per SM whether they
// are there or not, so a rest of more than two per SM goes to it and a smaller one is shorter in the butterfly form.
// l = 13, B = 2^5 on B200, butterfly / tensor form: 148 RLWEs 66 / 98 us, 296 93 / 99, 444 122 / 99, 592 153 / 100, 4096
// 994 / 677. With few digits it saves little or nothing a round (592 RLWEs, l = 1, 2, 3: 25.1 / 29.6, 35.3 / 33.2, 45.5 /
// 41.4), and the rest's launch of its own costs more than a CTA's last one or two RLWEs in the butterfly form alone
// (593: 33.3 / 46.8, 47.5 / 53.7, 60.4 / 65.9; l = 4: 74.2 / 74.1), for two digits after five rounds also more than
// any batch of its (2964: 184.5 / 190.9).
inline size_t external_products_by_butterflies(size_t count, uint32_t len, size_t sms) {
  const size_t round = 4 * sms;
  size_t rest = count % round;
  if (rest > 2 * sms) rest = 0;
  const bool tail_pays = len > 3 || rest == 0 || (rest > 2 && (len == 3 || count < 5 * round));
  return len > 1 && tail_pays ? rest : count;
}

}  // namespace hb
