// hb_boot_tc.cuh -- persistent batched bootstrapping over Goldilocks with the gadget digits' transforms on
// the tensor cores (tcgen05, exact u8 x u8 -> s32 products).
//
// A digit polynomial (coefficients below 2^8) is transformed as 1024 = 64 x 16, j = 16 j1 + j0 and
// k = k1 + 64 k0:
//   Y[k1][j0] = psi^(j0 (2 k1 + 1)) sum_j1 d[16 j1 + j0] psi^(16 j1 (2 k1 + 1)),
//   X[k1 + 64 k0] = sum_j0 Y[k1][j0] omega_16^(k0 j0).
// Both sums are matrix products with constant matrices whose entries are split into bytes: pass 1
// multiplies the digits (one byte each) by the bytes of its entries, pass 2 the bytes of Y by the
// bytes of (entry * 2^(8 i) mod Q), i the byte of Y, so that the field reduction of pass 2 is folded
// into its matrix. Every sum of products is at most 128 255^2 < 2^23, exact in the s32 accumulators, and a
// word is recombined from its eight byte columns with about 20 integer instructions.
//
// What bounds it: the integer pipes. Per transformed word a thread issues about 20 instructions for each
// recombination, 19 for the twist between the passes and 31 for the products with both key polynomials;
// the butterfly network of bootstrap_kernel issues about 160 and 34. ncu, 592 gates: ALU 56 %,
// multiply pipe 54 %, tensor core 10 % of the time. Measured on B200, one wave of 592 gates: GOLDILOCKS 63.7 ->
// 45.7 ms, ZAMA 97.5 -> 69.3 ms. For the 32-bit
// fields, whose butterflies are 8 to 11 instructions, the same form measured no faster than bootstrap_kernel
// (BABYBEAR 12.8 against 12.4 ms), so it is built for Goldilocks only.
#pragma once

#include "hb_handover.h"
#include "hb_kernels.cuh"
#include "hb_tc.cuh"

namespace hb {

struct TcGeo {
  using W = uint64_t;
  static constexpr int LOGN = 10, N = 1 << LOGN, G = 4;  // gates per CTA; T = 128 key layout
  // Four warpgroups compute; a fifth holds the warp that issues the MMAs and the one that copies keys. The
  // block launches with 96 registers a thread; the fifth group hands its share over (32 stay, the others
  // take 112: 512 x 112 + 128 x 32 = 640 x 96).
  static constexpr int THREADS = 512, AUX = 128, COMPUTE_REGS = 112, AUX_REGS = 32;
  static_assert(THREADS * COMPUTE_REGS + AUX * AUX_REGS <= (THREADS + AUX) * 96, "register split above the launch's total");
  // A unit of work is two digits of all four gates for half the k1: 256 accumulator columns after each pass
  // (pass 1: 32 k1 x 8 bytes; pass 2: two digits x 16 k0 x 8 bytes), the 512 of tensor memory together.
  static constexpr uint32_t B1_LBO = 512 * 16, B1_BYTES = 4 * B1_LBO;  // 64 k1 x 8 bytes by K = 64 j1
  static constexpr uint32_t B2_LBO = 128 * 16, B2_BYTES = 8 * B2_LBO;  // 16 k0 x 8 bytes by K = 16 j0 x 8 bytes
  static constexpr uint32_t TWIST_BYTES = N * 8;
  static constexpr uint32_t TAB_BYTES = B1_BYTES + B2_BYTES + TWIST_BYTES;
  static constexpr uint32_t A1_LBO = 128 * 16, A1_BYTES = 4 * A1_LBO;
  // 16 bytes of padding per K chunk: a warp's stores of 16 j0 x 2 gates hit distinct banks
  static constexpr uint32_t A2_LBO = 128 * 16 + 16, A2_TILE = 8 * A2_LBO, A2_BYTES = 2 * A2_TILE;
  // The transformed digits of a unit wait in shared memory between the stage that takes them and the one that
  // multiplies them: registers hold the sums. The inverse twiddles are read through L1.
  static constexpr uint32_t X_BYTES = 8 * THREADS * sizeof(W);
  static constexpr int STAGES = 2;                            // key stages of one unit each
  static constexpr uint32_t DIGIT_WORDS = N, STAGE_WORDS = 2 * DIGIT_WORDS;
  static constexpr int MS_STEPS = 256;                        // rotations kept per gate
  static constexpr int XPAD = 8;                              // words between the gates' inverse-transform buffers
  static_assert(G * (N + XPAD) * sizeof(W) <= A2_BYTES + A1_BYTES, "inverse buffers alias the pass-2 operands");
  static constexpr size_t SMEM = (size_t)TAB_BYTES + X_BYTES + A2_BYTES + A1_BYTES + (size_t)G * 2 * N * sizeof(W) +
                                 (size_t)STAGES * STAGE_WORDS * sizeof(W) + sizeof(uint16_t) * G * MS_STEPS +
                                 sizeof(uint64_t) * (STAGES + 1) + 16;
  static_assert(SMEM <= 232448, "shared memory of a CTA");
};

// Word from its byte columns c_0 .. c_7 (each at most 128 255^2, so that c_i + 2^8 c_(i+1) fits 32
// bits): lo + hi 2^32 + top 2^64 with a small top, worth top (2^32 - 1) mod Q; a carry of that sum is
// worth 2^32 - 1 once more. ALU shifts and carry chains: wide multiplies by 2^16 and 2^32 - 1 in their place
// hold the multiply pipe (26 against 18 of its cycles a word, 28.1 against 23.4 cycles in all).
__device__ __forceinline__ uint64_t tc_word(const uint32_t *c) {
  const uint32_t w0 = c[0] + (c[1] << 8), w1 = c[2] + (c[3] << 8);
  const uint32_t w2 = c[4] + (c[5] << 8), w3 = c[6] + (c[7] << 8);
  uint32_t r0, r1;
  asm("{\n\t.reg .u32 t, f, c0;\n\t"
      "shf.l.clamp.b32 f, %3, %5, 16;\n\t"
      "shl.b32 t, %3, 16;\n\t"
      "add.cc.u32 %0, %2, t;\n\t"
      "addc.cc.u32 %1, %4, f;\n\t"
      "shr.u32 t, %5, 16;\n\t"
      "addc.u32 t, t, 0;\n\t"  // top < 2^17
      "sub.cc.u32 %0, %0, t;\n\t"
      "subc.u32 f, t, 0;\n\t"  // with top = 0 there is no borrow
      "add.cc.u32 %1, %1, f;\n\t"
      "addc.u32 c0, 0, 0;\n\t"
      "neg.s32 c0, c0;\n\t"
      "add.cc.u32 %0, %0, c0;\n\t"
      "addc.u32 %1, %1, 0;\n\t}"
      : "=&r"(r0), "=&r"(r1)
      : "r"(w0), "r"(w1), "r"(w2), "r"(w3));
  return glx::join(r0, r1);
}
// x w + 2^32 - 1 mod Q: the 128-bit product by wide multiply-adds on aligned word pairs (x0 w0 | x1 w1 and
// x0 w1 + x1 w0), then the reduction without its last subtraction (tc_unshift takes the constant out): 24
// cycles of the multiply pipe a warp where the compiler's 64-bit lowering takes 34.
__device__ __forceinline__ uint64_t tc_twist(uint64_t x, uint64_t w) {
  uint32_t x0, x1, w0, w1, e0, e1, e2, e3, m0, m1, m2;
  glx::split(x, x0, x1);
  glx::split(w, w0, w1);
  glx::split((uint64_t)x0 * w0, e0, e1);
  glx::split((uint64_t)x1 * w1, e2, e3);
  glx::split((uint64_t)x0 * w1, m0, m1);
  asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32 %2, 0, 0;"
      : "+r"(m0), "+r"(m1), "=r"(m2)
      : "r"(x1), "r"(w0));
  asm("add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %2, %2, %5;"
      : "+r"(e1), "+r"(e2), "+r"(e3)
      : "r"(m0), "r"(m1), "r"(m2));
  // e0 .. e3 = lo + e2 2^64 + e3 2^96 = lo + A - (2^32 - 1) with A = fold_hi(e2, e3); a carry of lo + A
  // is worth 2^32 - 1 (and lo + A < A <= 2^64 - 2^32 then)
  uint32_t a0, a1, r0, r1;
  glx::split(glx::fold_hi(e2, e3), a0, a1);
  asm("{\n\t.reg .u32 c;\n\t"
      "add.cc.u32 %0, %2, %4;\n\t"
      "addc.cc.u32 %1, %3, %5;\n\t"
      "addc.u32 c, 0, 0;\n\t" HB_GL_ADD_EPS_C "}"
      : "=&r"(r0), "=&r"(r1)
      : "r"(e0), "r"(e1), "r"(a0), "r"(a1));
  return glx::join(r0, r1);
}
// What the constant offset of tc_twist's results (2^32 - 1 at every j0) adds up to: 16 (2^32 - 1) at k0 = 0,
// nothing elsewhere (the sixteenth roots of unity sum to zero).
__device__ __forceinline__ uint64_t tc_unshift(uint64_t x) { return glx::sub_c(x, 16ull * 0xFFFFFFFFu); }

// Sum of products x k over the digits of a step: 160 bits that take the products unreduced -- a digit pair's
// x0 k0 and x1 k1 by wide multiply-adds straight onto the words, its cross terms summed first and added at
// word 1 -- and are reduced once per step (glx::mac_lazy, a 96-bit sum of folded products, measured 31
// cycles a product in a warp where this takes 22). Word pairs are held as 64-bit values so that the wide
// multiply-adds find them in aligned registers (47.9 -> 46.4 ms per 592 GOLDILOCKS gates).
struct TcAcc {
  uint64_t e01, e23;
  uint32_t e4;
  __device__ __forceinline__ void clear() {
    e01 = e23 = 0;
    e4 = 0;
  }
  __device__ __forceinline__ void direct(uint32_t x0, uint32_t x1, uint32_t k0, uint32_t k1) {
    asm("{\n\t.reg .u32 a, b, c, d;\n\t"
        "mov.b64 {a, b}, %0;\n\t"
        "mov.b64 {c, d}, %1;\n\t"
        "mad.lo.cc.u32 a, %3, %5, a;\n\t"
        "madc.hi.cc.u32 b, %3, %5, b;\n\t"
        "madc.lo.cc.u32 c, %4, %6, c;\n\t"
        "madc.hi.cc.u32 d, %4, %6, d;\n\t"
        "addc.u32 %2, %2, 0;\n\t"
        "mov.b64 %0, {a, b};\n\t"
        "mov.b64 %1, {c, d};\n\t}"
        : "+l"(e01), "+l"(e23), "+r"(e4)
        : "r"(x0), "r"(x1), "r"(k0), "r"(k1));
  }
  __device__ __forceinline__ static void cross(uint64_t &m01, uint32_t &m2, uint32_t a, uint32_t b) {
    asm("{\n\t.reg .u32 a, b;\n\t"
        "mov.b64 {a, b}, %0;\n\t"
        "mad.lo.cc.u32 a, %2, %3, a;\n\t"
        "madc.hi.cc.u32 b, %2, %3, b;\n\t"
        "addc.u32 %1, %1, 0;\n\t"
        "mov.b64 %0, {a, b};\n\t}"
        : "+l"(m01), "+r"(m2)
        : "r"(a), "r"(b));
  }
  __device__ __forceinline__ void merge(uint64_t m01, uint32_t m2) {
    asm("{\n\t.reg .u32 a, b, c, d, m0, m1;\n\t"
        "mov.b64 {a, b}, %0;\n\t"
        "mov.b64 {c, d}, %1;\n\t"
        "mov.b64 {m0, m1}, %3;\n\t"
        "add.cc.u32 b, b, m0;\n\t"
        "addc.cc.u32 c, c, m1;\n\t"
        "addc.cc.u32 d, d, %4;\n\t"
        "addc.u32 %2, %2, 0;\n\t"
        "mov.b64 %0, {a, b};\n\t"
        "mov.b64 %1, {c, d};\n\t}"
        : "+l"(e01), "+l"(e23), "+r"(e4)
        : "l"(m01), "r"(m2));
  }
  __device__ __forceinline__ void mac(uint64_t x, uint64_t k) {
    uint32_t x0, x1, k0, k1, m2 = 0;
    glx::split(x, x0, x1);
    glx::split(k, k0, k1);
    direct(x0, x1, k0, k1);
    uint64_t m01 = (uint64_t)x0 * k1;
    cross(m01, m2, x1, k0);
    merge(m01, m2);
  }
  __device__ __forceinline__ void mac2(uint64_t x, uint64_t kx, uint64_t y, uint64_t ky) {
    uint32_t x0, x1, k0, k1, y0, y1, l0, l1, m2 = 0;
    glx::split(x, x0, x1);
    glx::split(kx, k0, k1);
    glx::split(y, y0, y1);
    glx::split(ky, l0, l1);
    direct(x0, x1, k0, k1);
    direct(y0, y1, l0, l1);
    uint64_t m01 = (uint64_t)x0 * k1;
    cross(m01, m2, x1, k0);
    cross(m01, m2, y0, l1);
    cross(m01, m2, y1, l0);
    merge(m01, m2);
  }
  // e0 .. e3 reduced, minus e4 2^32 (2^128 = -2^32 mod Q). e4 counts carries, at most one per direct and per
  // merge: below 2^32 - 1 for any number of digits, as e4 2^32 < Q needs.
  __device__ __forceinline__ uint64_t value() const {
    return glx::sub_c(glx::reduce_canon((uint32_t)e01, (uint32_t)(e01 >> 32), (uint32_t)e23, (uint32_t)(e23 >> 32)),
                      (uint64_t)e4 << 32);
  }
};

// Four bytes (x[i] >> sh) & mask of words x[0..3], mask replicated in every byte of mask4.
__device__ __forceinline__ uint32_t tc_digits4(const uint64_t *x, uint32_t sh, uint32_t mask4) {
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    v[i] = sh < 32 ? __funnelshift_r((uint32_t)x[i], (uint32_t)(x[i] >> 32), sh) : (uint32_t)(x[i] >> 32) >> (sh - 32);
  const uint32_t p01 = __byte_perm(v[0], v[1], 0x0040), p23 = __byte_perm(v[2], v[3], 0x0040);
  return __byte_perm(p01, p23, 0x5410) & mask4;
}

// Same bootstrap, jobs and keys (T = 128 layout) as bootstrap_kernel with G = 4 over Goldilocks and a binary
// LWE key; gadget and key-switch bases up to 2^8. tab: the tensor tables (TcGeo::TAB_BYTES). KSC as there.
//
// EXT: external products instead (ext_product_kernel): ext's RLWEs, four to a batch, times the RGSW at p.bsk --
// one step without a rotation or an accumulator, its E read from global memory.
struct TcExt {
  const uint64_t *in;
  uint64_t *out;
  unsigned long long count;
};
template <bool KSC, bool EXT = false>
__global__ void __launch_bounds__(TcGeo::THREADS + TcGeo::AUX, 1)
    bootstrap_tc_kernel(const BootParams<uint64_t> p, const unsigned char *__restrict__ tab, const TcExt ext) {
  using F = Goldilocks;
  using W = uint64_t;
  using Geo = TcGeo;
  using NT = GroupNtt<F, Geo::LOGN, 128, false>;
  constexpr int N = Geo::N, G = Geo::G, S = Geo::STAGES, V = NT::V;
  constexpr int kMmaWarp = Geo::THREADS / 32, kKeyWarp = kMmaWarp + 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *s_b1 = smem_raw, *s_b2 = s_b1 + Geo::B1_BYTES;
  const W *s_twist = reinterpret_cast<const W *>(s_b2 + Geo::B2_BYTES);
  W *s_x = reinterpret_cast<W *>(smem_raw + Geo::TAB_BYTES);
  unsigned char *s_a2 = reinterpret_cast<unsigned char *>(s_x) + Geo::X_BYTES, *s_a1 = s_a2 + Geo::A2_BYTES;
  W *s_acc = reinterpret_cast<W *>(s_a1 + Geo::A1_BYTES);
  W *s_k = s_acc + G * 2 * N;
  uint16_t *s_ms = reinterpret_cast<uint16_t *>(s_k + S * Geo::STAGE_WORDS);
  uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_ms + G * Geo::MS_STEPS);  // key stages, then the MMAs
  uint64_t *s_mma = s_bar + S;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_mma + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = tid >> 7, t = tid & 127;       // gate of the coefficient-domain work, thread in its group
  const int part_w = warp & 3, cg = warp >> 2;  // TMEM lane quarter and column quarter
  constexpr int ALL = Geo::THREADS + Geo::AUX;
  for (uint32_t i = tid; i < Geo::TAB_BYTES / 16; i += ALL)
    reinterpret_cast<uint4 *>(smem_raw)[i] = reinterpret_cast<const uint4 *>(tab)[i];
  for (uint32_t i = tid; i < Geo::A1_BYTES / 16; i += ALL)
    reinterpret_cast<uint4 *>(s_a1)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int s = 0; s < S; ++s) mbar_init(&s_bar[s], 32);
    mbar_init(s_mma, 1);
    mbar_fence_init();
    *s_abort = 0;
  }
  if (warp == kMmaWarp) tc::alloc(s_tmem, 512);
  tc::fence_async_smem();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t d1 = tmem, d2 = tmem + 256, lane_off = (uint32_t)(part_w * 32) << 16;

  GroupSync<128> sync{1 + g};
  W *acc_a = s_acc + g * 2 * N, *acc_b = acc_a + N;
  W *xbuf = reinterpret_cast<W *>(s_a2) + g * (N + Geo::XPAD);
  uint16_t *ms = s_ms + g * Geo::MS_STEPS;
  const uint32_t n = EXT ? 0 : p.n;  // EXT: step 0 alone
  const uint32_t ks_chunks = KSC ? p.ks_chunks : 1;
  // pairs of digits per part (a blind-rotation step has parts E.a and E.b, the key switch one per chunk)
  const uint32_t br_pairs = (p.len + 1) / 2, ks_pairs = (p.ks_len + 1) / 2;
  const uint32_t br_units = 2 * br_pairs * 2, ks_units = ks_chunks * ks_pairs * 2;
  const uint32_t my_batches =
      blockIdx.x < p.total_batches ? (p.total_batches - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  // A unit's end: every compute thread has written its operands of the next MMAs and read the last
  // accumulators. Compute threads only arrive; the MMA and key warps wait, issue the MMAs, whose completion
  // (s_mma) is what the compute threads wait for, and refill the key stage that was multiplied. (From the
  // compute warps themselves the issue, which lasts as long as the MMAs run, held all others up: 5800
  // cycles a unit.) Handovers take two named barriers in turn (hb_handover.h).
  constexpr int kStop = 6, kHandoverThreads = Geo::THREADS + 64;
  static_assert(kTcHandoverEven > G && kTcHandoverOdd > kStop && kTcHandoverEven < kStop, "named barriers overlap");

  if (warp >= kMmaWarp) {
    setmaxnreg_dec<Geo::AUX_REGS>();
    auto handed_over = [&](auto k) -> bool {  // handover k of the step, known up to its parity
      bar_sync<tc_handover_barrier(decltype(k)::value), kHandoverThreads>();
      tc::fence_after();
      return *s_abort == 0;
    };
    constexpr std::integral_constant<uint32_t, 0> even{};
    constexpr std::integral_constant<uint32_t, 1> odd{};
    if (warp == kMmaWarp) {
      const uint64_t a1 = tc::smem_desc(smem_u32(s_a1), Geo::A1_LBO, 128), b1 = tc::smem_desc(smem_u32(s_b1), Geo::B1_LBO, 128);
      const uint64_t a2 = tc::smem_desc(smem_u32(s_a2), Geo::A2_LBO, 128), b2 = tc::smem_desc(smem_u32(s_b2), Geo::B2_LBO, 128);
      // pass 1 of a unit's half (half < 2) and pass 2 of ne digits
      auto issue = [&](uint32_t half, uint32_t ne) {
        if (tc::elect_one()) {
          if (half < 2) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
              tc::mma_u8(d1, a1 + s * (2 * Geo::A1_LBO / 16), b1 + half * 256 + s * (2 * Geo::B1_LBO / 16),
                         tc::idesc_u8(128, 256), s > 0);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (i < (int)ne)
#pragma unroll
              for (int s = 0; s < 4; ++s)
                tc::mma_u8(d2 + i * 128, a2 + (i * Geo::A2_TILE + s * 2 * Geo::A2_LBO) / 16,
                           b2 + s * (2 * Geo::B2_LBO / 16), tc::idesc_u8(128, 128), s > 0);
          tc::commit(s_mma);
        }
        __syncwarp();
      };
      uint32_t groups = 0;
      for (uint32_t b = 0; b < my_batches; ++b)
        for (uint32_t step = 0; step <= n; ++step) {
          const bool ks = !EXT && step == n;
          const uint32_t L = ks ? p.ks_len : p.len, pairs = (L + 1) / 2;
          const uint32_t units = ks ? ks_units : br_units;
          if (!handed_over(even)) goto aux_done;  // the first pair's digits
          issue(0, 0);
          ++groups;
          // The two forms differ in what ptxas leaves of the compute warps' registers: 592 GOLDILOCKS gates 46.1 ms
          // two stages a turn, 45.7 one; 4096 external products 677 and 686 us.
          uint32_t pair = 0;
          if constexpr (EXT) {
            for (uint32_t u = 0;; u += 2) {  // units is even
              if (!handed_over(odd)) goto aux_done;  // unit u twisted, unit u - 1 taken, unit u - 2 multiplied
              if (u == units) break;
              const uint32_t ne = 2 * pair + 1 < L ? 2 : 1;
              issue(1, ne);
              ++groups;
              if (!handed_over(even)) goto aux_done;
              issue(u + 2 < units ? 0 : 2, ne);
              ++groups;
              if (++pair == pairs) pair = 0;
            }
          } else {
            uint32_t half = 0;
            for (uint32_t u = 0; u <= units; ++u) {
              bar_sync<kHandoverThreads>(tc_handover_barrier(u + 1));
              tc::fence_after();
              if (*s_abort) goto aux_done;
              if (u < units) {
                issue(u + 1 < units ? half ^ 1 : 2, 2 * pair + 1 < L ? 2 : 1);
                ++groups;
              }
              if (half == 1 && ++pair == pairs) pair = 0;
              half ^= 1;
            }
          }
        }
    aux_done:
      // MMAs in flight (after an abort) complete before the CTA ends
      if (groups) mbar_wait_bounded(s_mma, (groups - 1) & 1, kDrainBudget);
      __syncwarp();
    } else if (warp == kKeyWarp) {
      // Key stream: rows in consumption order (a blind-rotation step's digits of E.a and E.b; after the last
      // step the key switch's), a unit at a time into the next stage.
      const W *row = p.withhold ? nullptr : p.bsk;
      const uint32_t br_rows = (EXT ? 1 : n) * 2 * p.len;
      uint32_t kd = 0, khalf = 0, kks = 0, kleft = br_rows, kbatches = my_batches, kst = 0;
      auto copy_keys = [&]() {
        if (!row || !kbatches) return;
        const uint32_t L = kks ? p.ks_len : p.len, ne = kd + 1 < L ? 2 : 1;
        W *dst = s_k + kst * Geo::STAGE_WORDS;
        // word (v, a, i) of a polynomial sits at v 128 + 2 a + i: 64 consecutive words per v and half
        const W *src = row + khalf * 64 + lane * 2;
        dst += lane * 2;
#pragma unroll 8
        for (uint32_t i = 0; i < ne * 16; ++i) cp_async16(dst + i * 64, src + i * 128);
        cp_async_arrive(&s_bar[kst]);
        kst = kst + 1 == S ? 0 : kst + 1;
        khalf ^= 1;
        if (khalf) return;
        row += ne * 2 * N;
        kleft -= ne;
        kd = kd + ne == L ? 0 : kd + ne;
        if (kleft == 0) {  // the next section: the key switch, or the next batch's rotation
          if (!EXT) kks ^= 1;
          row = kks ? p.ksk : p.bsk;
          kleft = kks ? ks_chunks * p.ks_len : br_rows;
          kbatches -= kks ^ 1;
        }
      };
      for (int s = 0; s < S; ++s) copy_keys();
      for (uint32_t b = 0; b < my_batches; ++b)
        for (uint32_t step = 0; step <= n; ++step) {
          const uint32_t units = !EXT && step == n ? ks_units : br_units;
          if (!handed_over(even)) goto key_done;
          if (b != 0 || step != 0) copy_keys();  // the stage of the last unit multiplied
          for (uint32_t u = 0;; u += 2) {  // units is even
            if (!handed_over(odd)) goto key_done;
            if (u >= 2) copy_keys();
            if (u == units) break;
            if (!handed_over(even)) goto key_done;
            if (u >= 2) copy_keys();
          }
        }
    key_done:
      cp_async_wait_all();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == kMmaWarp) tc::dealloc(tmem, 512);
    return;
  }

  // ---- compute threads ----
  setmaxnreg_inc<Geo::COMPUTE_REGS>();
  uint32_t key_st = 0, key_par = 0;  // stage and phase of the key unit the next multiply takes
  uint32_t mma_par = 1;              // phase of the last MMA group handed over
  bool bad = false;                  // a wait of this thread ran out
  bool stopped = false;              // the auxiliary warps still expect handovers
  // Handover k of a step, k known up to its parity.
  auto handover = [&](auto k) {
    tc::fence_async_smem();
    tc::fence_before();
    bar_arrive<tc_handover_barrier(decltype(k)::value), kHandoverThreads>();
  };
  // Barrier of the compute threads; true when a wait of some thread ran out. A thread whose wait ran out
  // goes on (later waits return at once) until the next of these.
  auto barrier_stop = [&]() -> bool { return bar_or<kStop, Geo::THREADS>(bad); };

  for (uint32_t batch = blockIdx.x; batch < p.total_batches; batch += gridDim.x) {
    int jx = 0;
    if constexpr (!EXT)
      while (jx + 1 < p.njobs && p.jobs[jx + 1].first_batch <= batch) ++jx;
    const GateJob &job = p.jobs[jx];
    const unsigned long long item = (unsigned long long)batch * G + g;  // EXT
    const uint32_t gate = EXT ? 0 : (batch - job.first_batch) * G + g;
    const bool active = EXT ? item < ext.count : gate < job.count;
    const size_t lwe_words = (size_t)n + 1;

    // ---- input combine + modulus switch (as bootstrap_kernel) of coefficient k; absent gates rotate zeros
    // by zero ----
    auto rotation = [&](uint32_t k) -> uint16_t {
      if (!active) return 0;
      W c = small_mul<F>((reinterpret_cast<const W *>(job.in0) + gate * lwe_words)[k], job.s0);
      if (job.in1) c = F::canon(F::add(c, small_mul<F>((reinterpret_cast<const W *>(job.in1) + gate * lwe_words)[k], job.s1)));
      if (job.in2) c = F::canon(F::add(c, small_mul<F>((reinterpret_cast<const W *>(job.in2) + gate * lwe_words)[k], job.s2)));
      if (k == n) c = F::canon(F::add(c, (W)job.add_b));
      return (uint16_t)modswitch<F>(c, 2 * N);
    };
    // ---- ACC = (0, LUT * X^{-b}) (fhe_core/src/blind_rotation/rlwe/binary.rs:40-64) ----
    if constexpr (!EXT) {
      const uint32_t bt = rotation(n);  // every thread of the group the same
      const int e = bt ? (int)(2 * N - bt) : 0;
      const W *lut = reinterpret_cast<const W *>(job.lut);
      for (int k = t; k < N; k += 128) {
        int s = k - e;
        bool neg = false;
        if (s < 0) {
          s += N;
          neg = true;
          if (s < 0) {
            s += N;
            neg = false;
          }
        }
        W f = 0;
        if (active) f = lut ? F::canon(lut[s]) : (W)((uint32_t)s < job.lut_mid ? job.lut_lo : job.lut_hi);
        acc_a[k] = 0;
        acc_b[k] = neg ? F::neg_ref(f) : f;
      }
    }
    sync();

    // ---- steps 0 .. n-1: blind rotation; step n: key switch ----
    for (uint32_t step = 0; step <= n; ++step) {
      const bool ks = !EXT && step == n, last = step == n && batch + gridDim.x >= p.total_batches;
      const uint32_t L = ks ? p.ks_len : p.len, bits = ks ? p.ks_bits : p.bits;
      const uint32_t pairs = ks ? ks_pairs : br_pairs, units = ks ? ks_units : br_units;
      if constexpr (!EXT)
        if (step < n && step % Geo::MS_STEPS == 0) {  // the group's threads are past the rotations before
          for (uint32_t k = t; k < Geo::MS_STEPS && step + k < n; k += 128) ms[k] = rotation(step + k);
          sync();
        }
      const uint32_t mask4 = ((1u << bits) - 1) * 0x01010101u;
      const int j0 = t & 15, jb = t >> 4;  // the thread's coefficients: 16 (8 jb + i) + j0
      // E of the part, 8 words a thread, kept in local memory (read back once per digit pair): registers
      // hold the sums instead.
      W e_mem[8];
      asm volatile("" ::"l"(e_mem) : "memory");
      auto load_part = [&](uint32_t prt) {
        if constexpr (EXT) {
          const W *y = ext.in + (item * 2 + prt) * N;
#pragma unroll
          for (int i = 0; i < 8; ++i) e_mem[i] = active ? F::value(y[16 * (8 * jb + i) + j0]) : 0;
        } else if (!ks) {
          // E = ACC * (X^r - 1) (lattice/src/rlwe.rs:437-487) in the reference's representation, then
          // canonical for the unsigned decomposition
          const int r = (int)ms[step % Geo::MS_STEPS];
          const W *y = prt == 0 ? acc_a : acc_b;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int k = 16 * (8 * jb + i) + j0;
            const int s = k - r;
            W rot;
            if (s >= 0) {
              rot = y[s];
            } else if (s >= -N) {
              rot = F::neg_ref(y[s + N]);
            } else {
              rot = y[s + 2 * N];
            }
            e_mem[i] = F::value(F::sub(rot, y[k]));
          }
        } else if (!KSC) {
          // p = -acc.a (lattice/src/rlwe.rs:1147-1166)
#pragma unroll
          for (int i = 0; i < 8; ++i) e_mem[i] = F::value(F::neg_ref(acc_a[16 * (8 * jb + i) + j0]));
        } else {
          // chunk prt of the key switch in dimension n' < N (as bootstrap_kernel's KSC)
          const uint32_t c = prt, kn = p.ks_n, stride = N / kn;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t k = 16 * (8 * jb + i) + j0;
            W d = 0;
            if (k % stride == 0) {
              const uint32_t u = k / stride;
              const W w = u != 0 ? acc_a[N - (c + 1) * kn + u]
                                 : (c == 0 ? F::neg_ref(F::neg_ref(acc_a[0])) : F::neg_ref(acc_a[N - c * kn]));
              d = F::value(F::neg_ref(w));
            }
            e_mem[i] = d;
          }
        }
      };
      // The next two digits of the gate's part to rows d 64 + g 16 + j0 of the pass-1 operand.
      uint32_t bp = 0, bpart = 0;  // pair and part to build
      auto build_pair = [&]() {
        const uint32_t pi = bp;
        if (pi == 0) load_part(bpart);
        if (++bp == pairs) {
          bp = 0;
          ++bpart;
        }
        asm volatile("" ::: "memory");
        W e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = e_mem[i];
        unsigned char *dst = s_a1 + (g * 16 + j0) * 16 + (jb >> 1) * Geo::A1_LBO + (jb & 1) * 8;
#pragma unroll
        for (int d = 0; d < 2; ++d)
          if (2 * pi + d < L) {
            const uint32_t sh = (2 * pi + d) * bits;
            uint2 w;
            w.x = tc_digits4(e, sh, mask4);
            w.y = tc_digits4(e + 4, sh, mask4);
            *reinterpret_cast<uint2 *>(dst + d * 64 * 16) = w;
          }
      };
      // Pass 1 of a unit out of TMEM (lane: digit, gate, j0; the warp's 8 values of k1), twisted, to the pass-2
      // operand (row: k1, gate; K: j0 and byte).
      auto twist_unit = [&](uint32_t half, uint32_t ne) {
        const uint32_t row = part_w * 32 + lane;
        const uint32_t d = row >> 6, gg = (row >> 4) & 3, jj = row & 15;
        if (d >= ne) return;  // warp-uniform: a warp holds rows of one digit
        unsigned char *dst = s_a2 + d * Geo::A2_TILE + (jj / 2) * Geo::A2_LBO + (jj & 1) * 8 + gg * 16;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[16];
          tc::ld16(r, d1 + lane_off + cg * 64 + c * 16);
          tc::ld_wait(r);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t al = cg * 8 + c * 2 + i;  // k1 (bit-reversed) in the half
            *reinterpret_cast<W *>(dst + al * 64) =
                tc_twist(tc_word(r + i * 8), s_twist[(half * 32 + al) * 16 + jj]);
          }
        }
      };
      // Pass 2 of a unit: the thread's transformed digits at slots (a, b), a = 32 half + 8 part_w + lane / 4
      // of gate lane % 4, b = 2 cg + (q >> 1) + 8 (q & 1).
      auto x_at = [&](int d, int q) -> W & { return s_x[(d * 4 + q) * Geo::THREADS + tid]; };
      auto take_unit = [&](uint32_t ne) {
#pragma unroll
        for (int d = 0; d < 2; ++d)
          if (d < (int)ne)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t r[16];
              tc::ld16(r, d2 + lane_off + d * 128 + cg * 32 + c * 16);
              tc::ld_wait(r);
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                W v = tc_word(r + i * 8);
                if (c == 0 && i == 0 && cg == 0) v = tc_unshift(v);  // k0 = 0
                x_at(d, c * 2 + i) = v;
              }
            }
      };
      TcAcc acc_x[2][4], acc_y[2][4];  // [32 values of k1][q]
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc_x[m][q].clear();
          acc_y[m][q].clear();
        }
      auto mac_unit = [&](auto half_c, uint32_t ne) {
        constexpr int half = decltype(half_c)::value;
        if (!mbar_wait_bounded(&s_bar[key_st], key_par, bad ? 0 : p.budget) && !bad) {
          bad = true;
          atomicOr(p.status, STATUS_TIMEOUT);
        }
        const W *k = s_k + key_st * Geo::STAGE_WORDS;
        if (++key_st == S) {
          key_st = 0;
          key_par ^= 1;
        }
#pragma unroll
        for (int vv = 0; vv < 2; ++vv) {
          struct alignas(16) Two { W w[2]; };
          const W *kv = k + (2 * cg + vv) * 64 + 2 * (8 * part_w + (lane >> 2));
          const Two kx0 = *reinterpret_cast<const Two *>(kv), ky0 = *reinterpret_cast<const Two *>(kv + 512);
          if (ne == 2) {
            const Two kx1 = *reinterpret_cast<const Two *>(kv + 1024), ky1 = *reinterpret_cast<const Two *>(kv + 1536);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const W x0 = x_at(0, 2 * vv + i), x1 = x_at(1, 2 * vv + i);
              acc_x[half][2 * vv + i].mac2(x0, kx0.w[i], x1, kx1.w[i]);
              acc_y[half][2 * vv + i].mac2(x0, ky0.w[i], x1, ky1.w[i]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const W x0 = x_at(0, 2 * vv + i);
              acc_x[half][2 * vv + i].mac(x0, kx0.w[i]);
              acc_y[half][2 * vv + i].mac(x0, ky0.w[i]);
            }
          }
        }
      };

      // Units in a software pipeline: while the tensor core runs pass 1 of unit u and pass 2 of unit
      // u - 1, the threads multiply unit u - 2 with its keys; then they twist unit u and take unit u - 1.
      build_pair();
      handover(std::integral_constant<uint32_t, 0>{});
      mma_par ^= 1;
      uint32_t pair = 0;  // unit u's pair in its part
      uint32_t ne0 = L > 1 ? 2 : 1, ne1 = 0, ne2 = 0;  // digits of units u, u - 1, u - 2
      auto stage = [&](uint32_t u, auto half_c) {
        constexpr int half = decltype(half_c)::value;  // of units u and u - 2
        if (u >= 2) mac_unit(half_c, ne2);
        // Always waited for, whatever the launch's limit and after a key wait ran out too: a thread that ran
        // ahead of the auxiliary warps would arrive twice at one handover (hb_handover.h). Nothing but the
        // tensor core's own completion is waited for here, about 2 s a unit if it never came.
        if (!mbar_wait_bounded(s_mma, mma_par, kDrainBudget) && !bad) {
          bad = true;
          atomicOr(p.status, STATUS_TIMEOUT);
        }
        tc::fence_after();
        if (u < units) twist_unit(half, ne0);
        if (u >= 1) take_unit(ne1);
        if (u + 1 < units && half == 1) build_pair();
        handover(std::integral_constant<uint32_t, half + 1>{});
        if (u < units) mma_par ^= 1;
        ne2 = ne1;
        ne1 = ne0;
        if (half == 1) {
          if (++pair == pairs) pair = 0;
          ne0 = 2 * pair + 1 < L ? 2 : 1;
        }
      };
      for (uint32_t u = 0; u <= units; ++u) {
        if (u % 2 == 0)
          stage(u, std::integral_constant<int, 0>{});
        else
          stage(u, std::integral_constant<int, 1>{});
      }
      mac_unit(std::integral_constant<int, 1>{}, ne2);

      // ---- inverse transforms and accumulator update (or extraction) ----
      W b0 = 0;
      W *out = EXT ? ext.out + item * 2 * N : reinterpret_cast<W *>(job.out) + gate * lwe_words;
      if (ks) b0 = F::canon(F::add(acc_b[0], (W)(F::P >> 3)));  // evaluate.rs:52
      W sum[2][4], sum_b[2][4];  // of the a polynomial (h = 0), then the b polynomial
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          sum[m][q] = acc_x[m][q].value();
          sum_b[m][q] = acc_y[m][q].value();
        }
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        W *tb = reinterpret_cast<W *>(s_a2) + (lane & 3) * (N + Geo::XPAD);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int slot = (32 * m + 8 * part_w + (lane >> 2)) * 16 + 2 * cg + (q >> 1) + 8 * (q & 1);
            tb[NT::phys(slot)] = sum[m][q];
            sum[m][q] = sum_b[m][q];
          }
        if (barrier_stop()) {
          stopped = !last;
          goto aborted;
        }
        W f[V];
#pragma unroll
        for (int v = 0; v < V; ++v) f[v] = xbuf[NT::phys(NT::slot_pos(t, v))];
        sync();
        int ping = 0;
        NT::inverse(f, xbuf, ping, p.itw, t, sync);
        if constexpr (EXT) {
          if (active)
#pragma unroll
            for (int v = 0; v < V; ++v) out[h * N + NT::natural_pos(t, v)] = F::canon(f[v]);
        } else if (!ks) {
          W *y = h == 0 ? acc_a : acc_b;
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int k = NT::natural_pos(t, v);
            y[k] = F::add(y[k], F::canon(f[v]));  // RLWE::add_assign_element_wise
          }
        } else if (active) {
          // extract_partial_lwe_locally (lattice/src/rlwe.rs:393-402), as bootstrap_kernel
          const int kn = KSC ? (int)p.ks_n : N, ks_stride = N / kn;
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int k = NT::natural_pos(t, v);
            const W val = F::canon(f[v]);
            if (h == 0) {
              if (!KSC || k % ks_stride == 0) {
                const int u = KSC ? k / ks_stride : k;
                if (u == 0)
                  out[0] = val;
                else if (u >= kn - (int)n + 1)
                  out[kn - u] = F::neg_ref(val);
              }
            } else if (k == 0) {
              out[n] = F::canon(F::add(val, b0));
            }
          }
        }
        if (h == 0 && barrier_stop()) {  // the buffers take the b polynomial next
          stopped = !last;
          goto aborted;
        }
      }
      sync();
    }
  }

aborted:
  if (stopped) {  // the auxiliary warps stop at this handover, the first of a step that is not begun
    *s_abort = 1;
    handover(std::integral_constant<uint32_t, 0>{});
  }
  tc::fence_before();
  __syncthreads();
}

}  // namespace hb
