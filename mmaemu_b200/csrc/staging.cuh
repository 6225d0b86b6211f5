// Device code shared by the kernels that work on 128 x 128 output tiles and 32-wide k-tiles (kernel_fast.cu, kernel_umma.cu):
// tile numbering, the codes a thread decodes, mbarriers and bulk copies, and the power base of the exponent pass.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "fast_math.cuh"

namespace mmb {
namespace {

constexpr int BM = 128, BN = 128, KT = 32, THREADS = 256;
constexpr size_t UMMA_TILE_BYTES = 16384;      // operand image of 128 rows and 32 k for the tcgen05 kernels

// The power base of a format pair's tensor-core exponent pass (2^8, 2^5 or 2^4 per unit of exponent): see
// block_strip_mma and fast_math.cuh.
__host__ __device__ constexpr int tc_pow_mul(int fa, int fb) {
  return (fa == MMB200_FMT_E4M3 && fb == MMB200_FMT_E4M3) ? 8 : ((fa == MMB200_FMT_E5M2 && fb == MMB200_FMT_E5M2) ? 4 : 5);
}

// Output tile of a CTA. Tiles are numbered in bands of BAND tile columns, row by row inside a band, so that the CTAs that
// run at the same time share a band of B tiles that stays in L2 (a band of 16 decoded tile columns of K = 4096 is about
// 70 MB) while the A tiles stream through once per band.
constexpr int BAND = 16;
__device__ __forceinline__ void tile_of_cta(int tiles_m, int tiles_n, int band, int idx, int& tile_m, int& tile_n) {
  const int per_band = band * tiles_m, b = idx / per_band, rem = idx - b * per_band;
  const int w = min(band, tiles_n - b * band);
  tile_m = rem / w;
  tile_n = b * band + rem % w;
}
__device__ __forceinline__ void tile_of_cta(const Params& p, int idx, int& tile_m, int& tile_n) {
  tile_of_cta(p.tiles_m, p.tiles_n, BAND, idx, tile_m, tile_n);
}

// ---------------------------------------------------------------------------------------------------------------
// Quantise prologue (the scalar conversion is fm::quantise_e4m3 in fast_math.cuh).
// The 16 codes of row `row` starting at element k of one operand: the caller's FP8 codes, or -- operand A with the
// quantise prologue -- the codes of 16 activations, which are also written to the codes array.
template <bool IS_A>
__device__ __forceinline__ uint4 load_codes16(const Params& p, int row, int rows, int k) {
  if (row >= rows || k >= p.K) return make_uint4(0, 0, 0, 0);
  if (!IS_A || !p.a_hp) {
    const uint8_t* src = (IS_A ? p.A : p.B) + (long long)row * (IS_A ? p.lda : p.ldb) + k;
    if (!p.byte_loads) return __ldg(reinterpret_cast<const uint4*>(src));
    // K or a leading dimension that is no multiple of 16, or an operand that is not 16-byte aligned: byte by byte
    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (k + q < p.K) w[q / 4] |= (uint32_t)__ldg(src + q) << (8 * (q % 4));
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  const float scale = __ldg(p.a_quant_scale);
  float x[16];
  if (p.a_hp_dtype == MMB200_HP_F32) {
    const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.a_hp) + (long long)row * p.ld_hp + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 f = __ldg(src + q);
      x[4 * q] = __fmul_rn(f.x, scale); x[4 * q + 1] = __fmul_rn(f.y, scale);
      x[4 * q + 2] = __fmul_rn(f.z, scale); x[4 * q + 3] = __fmul_rn(f.w, scale);
    }
  } else {                        // bf16: torch multiplies in bf16 -- the scale and the product are rounded to bf16
    const float scale_b = __uint_as_float((uint32_t)f32_to_bf16_bits(scale) << 16);
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.a_hp) + (long long)row * p.ld_hp + k);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint4 w = __ldg(src + q);
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float lo = __fmul_rn(__uint_as_float(ws[h] << 16), scale_b);
        const float hi = __fmul_rn(__uint_as_float(ws[h] & 0xFFFF0000u), scale_b);
        x[8 * q + 2 * h] = __uint_as_float((uint32_t)f32_to_bf16_bits(lo) << 16);
        x[8 * q + 2 * h + 1] = __uint_as_float((uint32_t)f32_to_bf16_bits(hi) << 16);
      }
    }
  }
  uint32_t w4[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    w4[q] = fm::quantise_e4m3(x[4 * q]) | (fm::quantise_e4m3(x[4 * q + 1]) << 8) | (fm::quantise_e4m3(x[4 * q + 2]) << 16) |
            (fm::quantise_e4m3(x[4 * q + 3]) << 24);
  const uint4 codes = make_uint4(w4[0], w4[1], w4[2], w4[3]);
  *reinterpret_cast<uint4*>(p.a_codes + (long long)row * p.lda + k) = codes;
  return codes;
}

// Decodes 4 codes (non-finite ones become +0 in `w`, their classes are ORed into `seen`) for the tensor-core kernels: fp16
// pairs h01, h23 (exact) and the bf16 powers of the exponent pass p01, p23: exponent field bias + mul * ec (ec = clamped
// exponent - smallest exponent of the format; 0 for zero codes; fast_math.cuh). The fp16 value has the code's exponent in
// bits 10..14 once subnormals are raised to the smallest normal, so two 16-bit lanes take a maximum, a mask and, unless
// mul = 8, a shift and a multiply: the byte-parallel decode of the CUDA-core kernels took 15 instructions per code here and
// was most of the 16-row kernels' time.
template <int FA, int FB, bool IS_A>
__device__ __forceinline__ void decode4(uint32_t& w, uint32_t& h01, uint32_t& h23, uint32_t& p01, uint32_t& p23, uint32_t& seen) {
  constexpr int FMT = IS_A ? FA : FB, MUL = tc_pow_mul(FA, FB);
  constexpr bool E4 = FMT == MMB200_FMT_E4M3;
  const uint32_t nf = ((w & 0x7F7F7F7Fu) + (E4 ? 0x01010101u : 0x04040404u)) & 0x80808080u;
  if (nf) {                                                      // rare: 0x7F of E4M3 (NaN), >= 0x7C of E5M2 (Inf, NaN)
    if (E4) {
      seen |= 1u;
    } else {
      const uint32_t frac = ((w & 0x03030303u) + 0x7F7F7F7Fu) & 0x80808080u;
      seen |= ((nf & frac) ? 1u : 0u) | ((nf & ~frac) ? 2u : 0u);
    }
    w &= ~((nf >> 7) * 0xFFu);
  }
  if (E4) {
    asm("{.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\tcvt.rn.f16x2.e4m3x2 %1, hi;}"
        : "=r"(h01), "=r"(h23) : "r"(w));
  } else {                                                       // an E5M2 code is the high byte of an fp16
    h01 = __byte_perm(w, 0u, 0x1404);
    h23 = __byte_perm(w, 0u, 0x3424);
  }
  auto power = [](uint32_t h) -> uint32_t {
    constexpr uint32_t SMALLEST = E4 ? 0x24002400u : 0x04000400u;          // 2^-6, 2^-14
    constexpr int OFF = E4 ? 9 : 1;                                        // fp16 exponent field of ec = 0
    const __half2 v = *reinterpret_cast<const __half2*>(&h), least = *reinterpret_cast<const __half2*>(&SMALLEST);
    const __half2 m = __hmax2(__habs2(v), least);
    const uint32_t nonzero = __hne2_mask(v, __float2half2_rn(0.0f));
    const uint32_t x = *reinterpret_cast<const uint32_t*>(&m) & 0x7C007C00u;
    uint32_t lane;                                                         // field << 7 in both halves
    static_assert(MUL != 8 || (int)fm::POW8_BIAS == 8 * OFF, "E4M3: 8 times the fp16 field is the power's field");
    if (MUL == 8) lane = x;                                                // OFF and the bias cancel
    else if (MUL == 5) lane = (x >> 3) * 5u + (uint32_t)((int)fm::POW5_BIAS - 5 * OFF) * 0x00800080u;
    else lane = (x >> 1) + (uint32_t)((int)(IS_A ? fm::POW4_BIAS_A : fm::POW4_BIAS_B) - 4 * OFF) * 0x00800080u;
    return lane & nonzero;
  };
  p01 = power(h01);
  p23 = power(h23);
}

__device__ __forceinline__ uint32_t smem_addr(const void* ptr) { return (uint32_t)__cvta_generic_to_shared(ptr); }

constexpr int WAIT_POLLS = 1 << 22;        // default bound of every mbarrier wait (each poll suspends for up to ~1 us)

__device__ __forceinline__ void mbar_init(unsigned long long* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Bounded wait for the phase with the given parity: at most `polls` polls. Returns false if the bound ran out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, int polls) {
  const uint32_t addr = smem_addr(bar);
  for (int i = 0; i < polls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
// Bulk copy global -> shared (both 16-byte aligned, size a multiple of 16), completion counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}

}  // namespace
}  // namespace mmb
