// Products and exponent pass of a block as tcgen05.mma with accumulators in TMEM. Serves E4M3 x E4M3 and the mixed pairs on
// unsplit plans, and any plan cut into K slices (kernel_fast.cu, launch_staged, holds the rule); the scalar steps around the
// products are those of block_strip_mma (fast_math.cuh).
//
// Products. tcgen05.mma kind::f8f6f4 adds the accumulator and 32 products in one step: every summand is aligned to the
// largest exponent among them and cut, toward zero, below 25 fraction bits of that exponent; the sum is then cut to fp32.
// An accumulator of +-1.5 * 2^(E+12) (plus four times the model's accumulator) therefore makes the instruction truncate
// every product at 2^(E-13), the model's unit. fp32 holds the sum in units of four of these, so every product is fed four
// times: an instruction takes 8 k. The operand image holds each code twice in 16 bytes (8 k), and the descriptors' stride
// between the two 16-byte halves of K is zero, so both halves read the same bytes.
// Exponent pass: kind::f16 on bf16 powers of the operands' exponents (fast_math.cuh, mma_exponent).
// tests/test_mma_products_gpu.py checks the instruction's rounding against the integer kernel.
//
// Tiles: 128 rows, two halves of NW columns each, so that the tensor cores run one half's products while the warps of the
// other half compute. An MMA of 64 columns takes as long as one of 128 (95 and 97 cycles; 161 with 256), so NW = 128 is
// the better shape where the output has enough 256-column tiles and TMEM holds R and the exponent sums: one sum per block.
// NW = 64 otherwise, and for K slices.
//
// TMEM (512 columns x 128 lanes of 32 bits): offset accumulators R in columns 0 .. 2 NW - 1, exponent sums behind them (two
// sets with NW = 64). The running sums of slow accumulation take the last 128 columns with NW = 64; with NW = 128 TMEM is full
// and they live in shared memory (128 KB), which leaves two stages of operand images instead of four. Nothing is kept in
// registers between blocks.
//
// Roles: 16 warps run the scalar steps (warp w: lanes 32 (w % 4) .., a quarter w / 4 of the columns); one thread issues the
// MMAs, one thread the bulk copies of the operand images. Every wait is bounded.
//
// What bounds it. Per output and block the warps issue 4 instructions for the half-rate INT pipe and 2 FMAs beside TMEM loads
// and stores (one column per cycle each): 8 cycles per scheduler and 32 outputs at best. Measured: 13 with fast accumulation
// (8192 x 24576 x 8192, 18.1 ms), 18 with slow (4096-cube, 1.21 ms; INT pipe 61 % busy). The rest is the latency from a half's
// stores of R over its MMAs to its next loads, which the other half covers only in part, and with slow accumulation the chain
// end, a pass over TMEM of its own every 128 k (0.92 ms without it on the same tiles).
#include <atomic>

#include "staging.cuh"

namespace mmb {
namespace {

constexpr int EPI_WARPS = 16, EPI_THREADS = EPI_WARPS * 32, UMMA_THREADS = EPI_THREADS + 64;
constexpr uint32_t R_ZERO = 0x3FC00000u;       // 1.5: an offset accumulator that stands for +0 (fm::mma_end)

// One decoded k-tile of 128 rows: eight 16-byte chunks per row, chunk-major, so that each chunk array is a K-major operand
// without swizzle (8-row core matrices of 128 contiguous bytes, row groups 128 bytes apart).
//   chunk c < 4:  codes of k = 8 c .. 8 c + 7, each twice (non-finite codes as +0)
//   chunk 4 + c:  bf16 powers 2^(mul * exponent + const) of k = 8 c .. 8 c + 7 (0 for zero codes)
struct UmmaTile {
  uint4 c[8][128];
};
static_assert(sizeof(UmmaTile) == UMMA_TILE_BYTES, "tile layout");
template <int NW>
struct UmmaStage { UmmaTile a, b[NW / 64]; };
template <int NW, bool PARTS>
struct SmemUmma {                              // NW columns per half: 64 (5 stages of 32 KB) or 128 (4 stages of 48 KB; 2 with sums)
  static constexpr int RING = NW == 64 ? 5 : (PARTS ? 2 : 4);
  UmmaStage<NW> stage[RING];                   // later: the image of the output tile (of one half of it)
  float part[PARTS ? 2 * NW : 1][128];         // running sums of slow accumulation, [column][row], where TMEM is full
  unsigned long long full[RING];               // the stage's copies have landed
  unsigned long long empty[RING];              // the MMAs that read the stage are done
  unsigned long long ready[2];                 // half h: every warp has stored R of the block (and read its exponent sums)
  unsigned long long done[2];                  // half h: products of the block and exponent sums of the next one are done
  unsigned long long drain;
  uint32_t tmem;
};

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Shared-memory descriptor of a K-major operand without swizzle: `k_stride` bytes between the 16-byte halves of K, 128 bytes
// between groups of 8 rows.
__device__ __forceinline__ uint64_t umma_desc(const void* ptr, uint32_t k_stride) {
  return ((uint64_t)(smem_addr(ptr) >> 4) & 0x3FFF) | ((uint64_t)(k_stride >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
         (1ull << 46);
}
__device__ __forceinline__ void umma_f8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(1) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[8], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[16], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
               "[%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
               "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// The registers of a load may be read from here on (after tmem_wait_ld).
template <int N>
__device__ __forceinline__ void tmem_use(uint32_t (&r)[N]) {
#pragma unroll
  for (int q = 0; q < N; ++q) asm volatile("" : "+r"(r[q])::"memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float chain_result4(float acc) { return __fmul_rn(fm::chain_cut(acc), 0.25f); }

// One CTA per (k-tile, 128-row block) of one operand: writes the operand image and ORs the non-finite classes of the rows.
template <int FA, int FB, bool IS_A>
__global__ void __launch_bounds__(THREADS) predecode_umma_kernel(const __grid_constant__ Params p) {
  const int tid = threadIdx.x, kt = blockIdx.x, rb = blockIdx.y, rows = IS_A ? p.M : p.N;
  UmmaTile& tile = reinterpret_cast<UmmaTile*>(IS_A ? p.ws_a : p.ws_b)[(long long)rb * p.k_tiles + kt];
  int* flags = IS_A ? p.ws_flag_a : p.ws_flag_b;
  const int lrow = tid % 128, lhalf = tid / 128, row = rb * 128 + lrow;
  const uint4 raw = load_codes16<IS_A>(p, row, rows, kt * KT + 16 * lhalf);
  uint32_t w4[4] = {raw.x, raw.y, raw.z, raw.w}, seen = 0, v[4][2], e[4][2];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    uint32_t h01, h23;
    decode4<FA, FB, IS_A>(w4[w], h01, h23, e[w][0], e[w][1], seen);
    v[w][0] = __byte_perm(w4[w], 0u, 0x1100);
    v[w][1] = __byte_perm(w4[w], 0u, 0x3322);
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    tile.c[2 * lhalf + c][lrow] = make_uint4(v[2 * c][0], v[2 * c][1], v[2 * c + 1][0], v[2 * c + 1][1]);
    tile.c[4 + 2 * lhalf + c][lrow] = make_uint4(e[2 * c][0], e[2 * c][1], e[2 * c + 1][0], e[2 * c + 1][1]);
  }
  if (seen) atomicOr(&flags[row], (int)seen);
}

template <int NFMA, int FA, int FB, bool SLOW, int NW, bool SLICED>
__global__ void __launch_bounds__(UMMA_THREADS, 1) umma_kernel(const __grid_constant__ Params p) {
  constexpr bool PARTS = SLOW && !SLICED && NW == 128; // running sums in shared memory
  using Smem = SmemUmma<NW, PARTS>;
  constexpr bool POW256 = tc_pow_mul(FA, FB) == 8;
  constexpr int RING = Smem::RING, WC = NW / 2;        // columns of a warp
  constexpr int BPT = KT / NFMA;                       // blocks per k-tile
  constexpr bool TWO_SUMS = !POW256 && NFMA == 32;     // a block takes the larger of two 16-term sums
  constexpr bool AHEAD = NW == 64 && !TWO_SUMS;        // two sets of sums: those of a block are computed one block ahead
  constexpr int CHAIN = 128 / NFMA;                    // blocks per chain (unsplit slow accumulation)
  constexpr int COL_S = 2 * NW;
  constexpr int COL_PART = 384;                        // running sums of chain results (slow accumulation, NW = 64)
  constexpr int CHUNK = TWO_SUMS ? 8 : 16;             // columns a warp handles at a time; the next ones are being loaded
  static_assert(NW == 64 || !TWO_SUMS, "TMEM holds one set of sums for 256 columns");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  int tile_m, tile_n;                                  // tile_n in units of 2 NW columns
  tile_of_cta(p.tiles_m, (p.N + 2 * NW - 1) / (2 * NW), BAND * 64 / NW, (int)blockIdx.x, tile_m, tile_n);
  const int m0 = tile_m * BM, n0 = tile_n * 2 * NW;
  // k-tiles in order, or this K slice's part of the plan's sequence
  const int t0 = SLICED ? p.slice_start[blockIdx.y] : 0;
  const int T = SLICED ? p.slice_start[blockIdx.y + 1] - t0 : p.k_tiles, NB = T * BPT;
  const int H = n0 + NW >= p.N ? 1 : 2;                // halves with columns of the problem
  if (tid == 0) {
    for (int q = 0; q < RING; ++q) { mbar_init(&sm.full[q], 1); mbar_init(&sm.empty[q], 1); }
    for (int h = 0; h < 2; ++h) { mbar_init(&sm.ready[h], EPI_WARPS / 2); mbar_init(&sm.done[h], 1); }
    mbar_init(&sm.drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == EPI_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&sm.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = sm.tmem;
  bool ok = true;
  const int h = (warp % EPI_WARPS) / 8;                                               // the warp's half (scalar steps)
  const uint32_t my = tmem + ((uint32_t)(32 * (warp % 4)) << 16) + WC * (warp / 4);   // its lanes and first column
  if (warp == EPI_WARPS + 1) {
    // ---- bulk copies of the operand images
    if (lane == 0) {
      const UmmaTile* ga = reinterpret_cast<const UmmaTile*>(p.ws_a) + (long long)tile_m * p.k_tiles;
      const int nb = (NW == 128 && n0 + 128 < p.N) ? 2 : 1;                           // 128-column images of B
      const UmmaTile* gb = reinterpret_cast<const UmmaTile*>(p.ws_b) + (long long)tile_n * (NW / 64) * p.k_tiles;
      int issued = 0;
      for (int t = 0; t < T; ++t) {
        const int s = t % RING, kt = SLICED ? (int)(__ldg(p.ws_seq + t0 + t) & SEQ_TILE_MASK) : t;
        if (t >= RING && !mbar_wait(&sm.empty[s], ((t / RING) - 1) & 1, p.wait_polls)) { ok = false; break; }
        mbar_expect_tx(&sm.full[s], (uint32_t)sizeof(UmmaTile) * (1 + nb) + (uint32_t)p.test_announce_extra);
        bulk_load(&sm.stage[s].a, ga + kt, sizeof(UmmaTile), &sm.full[s]);
        for (int q = 0; q < nb; ++q)
          bulk_load(&sm.stage[s].b[q], gb + (long long)q * p.k_tiles + kt, sizeof(UmmaTile), &sm.full[s]);
        issued = t + 1;
      }
      // the CTA must not end while a copy may be in flight: wait for the last copy into every stage (bounded)
      for (int t = issued > RING ? issued - RING : 0; t < issued; ++t)
        if (!mbar_wait(&sm.full[t % RING], (t / RING) & 1, p.wait_polls)) ok = false;
    }
    __syncwarp();
  } else if (warp == EPI_WARPS) {
    // ---- MMA issue
    if (lane == 0) {
      constexpr uint32_t SHAPE = (1u << 4) | ((uint32_t)(NW >> 3) << 17) | ((128u >> 4) << 24);   // fp32 out, N = NW, M = 128
      constexpr uint32_t ID_F8 = SHAPE | ((FA == MMB200_FMT_E5M2 ? 1u : 0u) << 7) | ((FB == MMB200_FMT_E5M2 ? 1u : 0u) << 10);
      constexpr uint32_t ID_BF16 = SHAPE | (1u << 7) | (1u << 10);
      int landed = 0;                                  // k-tiles seen complete
      bool issued = false;
      auto need = [&](int t) {
        while (ok && landed <= t) {
          ok = mbar_wait(&sm.full[landed % RING], (landed / RING) & 1, p.wait_polls);
          ++landed;
        }
      };
      // first row (column of the output) of half q of a chunk of B
      auto b_rows = [&](const UmmaStage<NW>& st, int chunk, int q) { return NW == 64 ? &st.b[0].c[chunk][64 * q] : &st.b[q % (NW / 64)].c[chunk][0]; };
      auto exponents = [&](int b, int q) {             // sums of powers of block b, columns of half q
        need(b / BPT);
        if (!ok) return;
        const UmmaStage<NW>& st = sm.stage[(b / BPT) % RING];
        issued = true;
#pragma unroll
        for (int i = 0; i < NFMA / 16; ++i) {
          const int step = NFMA == 32 ? i : b % BPT, set = TWO_SUMS ? i : (AHEAD ? (b & 1) : 0);
          umma_bf16(tmem + COL_S + 2 * NW * set + NW * q, umma_desc(&st.a.c[4 + 2 * step][0], 2048),
                    umma_desc(b_rows(st, 4 + 2 * step, q), 2048), ID_BF16, POW256 && i > 0 ? 1u : 0u);
        }
      };
      for (int q = 0; q < H && ok; ++q) {
        exponents(0, q);
        if (ok) umma_commit(&sm.done[q]);
      }
      if (AHEAD && NB > 1)
        for (int q = 0; q < H && ok; ++q) exponents(1, q);
      for (int b = 0; b < NB && ok; ++b) {
        const int t = b / BPT;
        const UmmaStage<NW>& st = sm.stage[t % RING];
        for (int q = 0; q < H && ok; ++q) {
          if (!mbar_wait(&sm.ready[q], b & 1, p.wait_polls)) { ok = false; break; }
          fence_after();
#pragma unroll
          for (int i = 0; i < NFMA / 8; ++i) {
            const int c = NFMA == 32 ? i : 2 * (b % BPT) + i;
            umma_f8(tmem + NW * q, umma_desc(&st.a.c[c][0], 0), umma_desc(b_rows(st, c, q), 0), ID_F8);
          }
          issued = true;
          if (!AHEAD && b + 1 < NB) exponents(b + 1, q);
          if (!ok) break;
          umma_commit(&sm.done[q]);
          if (q == H - 1 && b % BPT == BPT - 1 && t + RING < T) umma_commit(&sm.empty[t % RING]);
          if (AHEAD && b + 2 < NB) exponents(b + 2, q);
        }
      }
      if (issued) {                                    // nothing in flight when the TMEM is given back
        umma_commit(&sm.drain);
        mbar_wait(&sm.drain, 0, WAIT_POLLS);
      }
    }
    __syncwarp();
  } else if (h < H) {
    // ---- the scalar steps: block start of block b, from R of block b - 1
    const bool rows = m0 + 32 * (warp % 4) < p.M;      // a warp without rows of the problem only keeps the barriers
    uint32_t zero[CHUNK];
#pragma unroll
    for (int q = 0; q < CHUNK; ++q) zero[q] = R_ZERO;
    for (int c = 0; c < WC; c += CHUNK) tmem_st(my + c, zero);
    float* sums = &sm.part[PARTS ? WC * (warp / 4) : 0][32 * (warp % 4) + lane];
    if (PARTS) {
      for (int c = 0; c < WC; ++c) sums[c * 128] = 0.0f;
    } else if (SLOW && !SLICED) {
      const uint32_t none[CHUNK] = {};
      for (int c = 0; c < WC; c += CHUNK) tmem_st(my + c + COL_PART, none);
    }
    tmem_wait_st();
    // K slices: where the chain results of this thread's first column go, [chain][column][row] of the tile
    float* dst = nullptr;
    if (SLICED)
      dst = p.ws_chains + ((size_t)blockIdx.x * p.n_chains + p.chain_base[blockIdx.y]) * (BM * BN) +
            (size_t)(WC * (warp / 4)) * BM + 32 * (warp % 4) + lane;
    for (int b = 0; b <= NB; ++b) {
      ok = __all_sync(0xFFFFFFFFu, mbar_wait(&sm.done[h], b & 1, p.wait_polls));
      if (!ok) break;
      fence_after();
      bool chain_end = b == NB && !SLICED;
      if (SLICED) chain_end = b > 0 && b % BPT == 0 && seq_emits(__ldg(p.ws_seq + t0 + b / BPT - 1), SLOW ? 1 : 0);
      else if (SLOW) chain_end = b > 0 && (b == NB || b % CHAIN == 0);
      if ((SLOW || SLICED) && chain_end && rows) {     // the chain's result joins the running sum, or goes to scratch memory
#pragma unroll 1
        for (int c = 0; c < WC; c += CHUNK) {
          uint32_t r[CHUNK], part[CHUNK];
          tmem_ld(r, my + c);
          if constexpr (!SLICED && !PARTS) tmem_ld(part, my + c + COL_PART);
          tmem_wait_ld();
          tmem_use(r);
          if constexpr (!SLICED && !PARTS) tmem_use(part);
#pragma unroll
          for (int q = 0; q < CHUNK; ++q) {
            const float v = chain_result4(fm::mma_end(__uint_as_float(r[q])));
            if constexpr (SLICED) dst[(size_t)(c + q) * BM] = v;
            else if constexpr (PARTS) sums[(c + q) * 128] = __fadd_rn(sums[(c + q) * 128], v);
            else part[q] = __float_as_uint(__fadd_rn(__uint_as_float(part[q]), v));
          }
          if constexpr (!SLICED && !PARTS) tmem_st(my + c + COL_PART, part);
          tmem_st(my + c, zero);
        }
        tmem_wait_st();
        if (SLICED) dst += BM * BN;
      }
      if (b == NB) break;
      if (rows) {
        uint32_t r[2][CHUNK], s0[2][CHUNK], s1[2][CHUNK];
        auto load = [&](int c, int w) {
          tmem_ld(s0[w], my + c + COL_S + (AHEAD ? 2 * NW * (b & 1) : 0));
          if constexpr (TWO_SUMS) tmem_ld(s1[w], my + c + COL_S + 2 * NW);
          tmem_ld(r[w], my + c);
        };
        load(0, 0);
#pragma unroll
        for (int c = 0; c < WC; c += CHUNK) {
          const int w = (c / CHUNK) & 1;
          tmem_wait_ld();
          tmem_use(s0[w]);
          if constexpr (TWO_SUMS) tmem_use(s1[w]);
          tmem_use(r[w]);
          if (c + CHUNK < WC) load(c + CHUNK, w ^ 1);
#pragma unroll
          for (int q = 0; q < CHUNK; ++q) {
            float S = __uint_as_float(s0[w][q]);
            if constexpr (TWO_SUMS) S = fmaxf(S, __uint_as_float(s1[w][q]));
            const float a = fm::mma_end(__uint_as_float(r[w][q]));
            r[w][q] = __float_as_uint(fm::mma_start(a, fm::mma_unit(a, fm::mma_exponent<FA, FB>(S))));
          }
          tmem_st(my + c, r[w]);
        }
        tmem_wait_st();
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.ready[h]);
    }
  }
  // One decision for the whole CTA; after it no MMA and no copy touches the stages.
  if (!ok && p.status) atomicExch(p.status, 1);
  const bool bad = __syncthreads_or(ok ? 0 : 1) != 0;
  if (!SLICED && !bad && warp < EPI_WARPS) {           // a K slice has stored its chains; the combine kernel writes the output
    Epilogue epi;
    epi.init(p);
    const int lr = 32 * (warp % 4) + lane, gm = m0 + lr;
    const int row_flag = p.patch_nonfinite && gm < p.M ? p.ws_flag_a[gm] : 0;
    // an image of 128 x 128 outputs for both halves (NW = 64) or for one after the other; rows of it are written out by all
    // the warps. Elements beyond M or N are parked too and not written out.
#pragma unroll 1
    for (int half = 0; half < NW / 64; ++half) {
      const int nc = n0 + 128 * half;
      if (nc >= p.N) break;
      if (h < H && (NW == 64 || h == half)) {
#pragma unroll 1
        for (int c = 0; c < WC; c += CHUNK) {
          uint32_t r[CHUNK];
          float v[CHUNK];
          const int lc = (WC * (warp / 4) + c) % 128, gn = nc + lc;
          if constexpr (PARTS) {
#pragma unroll
            for (int q = 0; q < CHUNK; ++q) v[q] = sm.part[WC * (warp / 4) + c + q][lr];
          } else {
            tmem_ld(r, my + c + (SLOW ? COL_PART : 0));
            tmem_wait_ld();
            tmem_use(r);
#pragma unroll
            for (int q = 0; q < CHUNK; ++q) v[q] = SLOW ? __uint_as_float(r[q]) : chain_result4(fm::mma_end(__uint_as_float(r[q])));
          }
          // non-finite classes: one look for the warp's rows and these columns, then element by element where one is set
          const int col = gn + lane % CHUNK, col_flag = p.patch_nonfinite && col < p.N ? p.ws_flag_b[col] : 0;
          if (__any_sync(0xFFFFFFFFu, row_flag | col_flag)) {
#pragma unroll
            for (int q = 0; q < CHUNK; ++q) {
              const int flag = row_flag | __shfl_sync(0xFFFFFFFFu, col_flag, q);
              uint32_t bits;
              if (flag && gm < p.M && gn + q < p.N &&
                  nonfinite_patch(flag, p.A + (long long)gm * p.lda, p.B + (long long)(gn + q) * p.ldb, p.K, p.fmt_a, p.fmt_b, bits))
                v[q] = __uint_as_float(bits);
            }
          }
          epi.park_row(smem_raw, lr, lc, v);
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
      epi.flush(p, smem_raw, m0, nc, tid, EPI_THREADS);
      if (NW == 128) asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
    }
  }
  fence_before();
  __syncthreads();
  if (warp == EPI_WARPS) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

template <int FA, int FB, bool IS_A>
cudaError_t launch_predecode(const Params& p, cudaStream_t stream, int* launches) {
  predecode_umma_kernel<FA, FB, IS_A><<<dim3((unsigned)p.k_tiles, (unsigned)(IS_A ? p.tiles_m : p.tiles_n)), THREADS, 0, stream>>>(p);
  const cudaError_t err = cudaGetLastError();
  if (err == cudaSuccess) *launches += 1;
  return err;
}

template <int NFMA, int FA, int FB, bool SLOW, int NW, bool SLICED>
cudaError_t launch_kernel(const Params& p, cudaStream_t stream, int* launches) {
  auto kern = umma_kernel<NFMA, FA, FB, SLOW, NW, SLICED>;
  constexpr size_t SMEM = sizeof(SmemUmma<NW, SLOW && !SLICED && NW == 128>);
  static_assert(SMEM <= 232448, "shared memory of a CTA");
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
  if (err != cudaSuccess) return err;
  const long long tiles = (long long)p.tiles_m * ((p.N + 2 * NW - 1) / (2 * NW));
  kern<<<dim3((unsigned)tiles, SLICED ? (unsigned)p.slices : 1u), UMMA_THREADS, SMEM, stream>>>(p);
  err = cudaGetLastError();
  if (err == cudaSuccess) *launches += 1;
  return err;
}

template <int NFMA, int FA, int FB>
cudaError_t launch_main(const Params& p, cudaStream_t stream, int* launches) {
  if (p.slices > 1)
    return p.plan_group ? launch_kernel<NFMA, FA, FB, true, 64, true>(p, stream, launches)
                        : launch_kernel<NFMA, FA, FB, false, 64, true>(p, stream, launches);
  if constexpr (tc_pow_mul(FA, FB) == 8 || NFMA == 16) {
    if (p.wide_tiles)
      return p.fast ? launch_kernel<NFMA, FA, FB, false, 128, false>(p, stream, launches)
                    : launch_kernel<NFMA, FA, FB, true, 128, false>(p, stream, launches);
  }
  return p.fast ? launch_kernel<NFMA, FA, FB, false, 64, false>(p, stream, launches)
                : launch_kernel<NFMA, FA, FB, true, 64, false>(p, stream, launches);
}

template <int FA, int FB>
cudaError_t launch(const Params& p, int nfma, cudaStream_t stream, int* launches) {
  cudaError_t err;
  if (!p.only_b && (err = launch_predecode<FA, FB, true>(p, stream, launches)) != cudaSuccess) return err;
  if (p.only_b || !p.shared_b) {
    if ((err = launch_predecode<FA, FB, false>(p, stream, launches)) != cudaSuccess) return err;
  }
  if (p.only_b) return cudaSuccess;
  return nfma == 16 ? launch_main<16, FA, FB>(p, stream, launches) : launch_main<32, FA, FB>(p, stream, launches);
}

}  // namespace

cudaError_t launch_umma(const Params& p, int nfma, cudaStream_t stream, int* launches) {
  switch (p.fmt_a * 2 + p.fmt_b) {
    case 0: return launch<MMB200_FMT_E4M3, MMB200_FMT_E4M3>(p, nfma, stream, launches);
    case 1: return launch<MMB200_FMT_E4M3, MMB200_FMT_E5M2>(p, nfma, stream, launches);
    case 2: return launch<MMB200_FMT_E5M2, MMB200_FMT_E4M3>(p, nfma, stream, launches);
    default: return cudaErrorInvalidValue;             // E5M2 x E5M2: umma_supports says no
  }
}

}  // namespace mmb
