// FP64-accurate complex GEMM on the 5th-generation tensor cores (tcgen05): the plain
// form of the dense contraction's GEMM (_contract_dense, src/tensor/contract.cpp:133-162
// of the reference sums complex<double> products over the closed indices).
//
// C (M x N) = A (M x K) B (K x N), complex128; here A is given as A'' (M x K row-major)
// and B as B'' (N x K row-major, the contracted index innermost in both).
//
// Real form: C^ (2M x N) = A^ (2M x 2K) B^^T with, for complex row m and column k,
//     A^[2m][2k] = Re a, A^[2m][2k+1] = -Im a, A^[2m+1][2k] = Im a, A^[2m+1][2k+1] = Re a,
//     B^[n][2k] = Re b, B^[n][2k+1] = Im b,
// so rows 2m / 2m+1 of C^ are Re / Im of C[m].
//
// Digits (the Ozaki scheme, ozaki.cuh): every real of complex row m of A is cut into six
// balanced base-256 digits at the row's largest exponent ea[m] (x ~= sum_i d_i 2^(-8i)
// 2^(ea - 1030), 48 significant bits relative to the row's largest element), every real
// of column n of B at eb[n]. Each digit is an integer of at most 8 significant bits:
// exact in bf16, and the product of two digits is exact in FP32. Then
//     C^[r][n] = 2^(ea + eb - 2060) sum_l 2^(-8l) S_l,  S_l = sum_{i+j=l} sum_k dA_i dB_j,
// levels l = 0..5 (the 21 digit pairs i + j <= 5; the dropped levels lie below 2^-48).
// Exactness: over a chunk of 128 reals of K (8 K-steps of 16) every level sum stays
// within 2^24 in magnitude (level 5: 128 * (2 * 256 * 128 + 4 * 128 * 128) = 2^24), so
// the tensor core's FP32 accumulators hold each chunk's level sums exactly. After each
// chunk the epilogue drains them from tensor memory and accumulates
//     T += S_0 2^24 + S_1 2^16 + S_2 2^8 + S_3   (exact, 64-bit integer),
//     F += S_4 + 2^-8 S_5                           (FP32; it lies below 2^-32 of T's scale),
// and at the end C^ = 2^(ea + eb - 2084) (T + 2^-8 F), rounded once to a double.
// The result is therefore accurate to ~2^-48 of the largest product magnitudes of its
// row and column, independent of K: FP64-level for the 1e-12 relative-L2 bar.
//
// Tile: 128 rows of C^ (64 complex rows) x 64 columns. Per K-step the stage holds the six A
// digits (128 rows x 16 bf16 each, 24 KB) and the six B digits stacked along N (64 rows
// each, 12 KB), all in the UMMA K-major core-matrix layout (8 rows x 16 bytes; LBO 128 B,
// SBO 256 B). A digit i meets B digits 0 .. 5 - i, 64 (6 - i) rows, in one tcgen05.mma
// (kind::f16, bf16 in, FP32 out; two of half the rows where they exceed 256) into the
// level columns 64 i ..: 8 MMAs per K-step. (Two halves of 32 columns, 12 MMAs, read the A
// digits twice and took 920 cycles a K-step, which shared memory bounds at 704; this reads
// 74 KB, 592 cycles against the tensor pipe's 672.) Tensor memory: 6 levels x 64 columns.
// CTA (persistent, one per SM): warp 0 streams each K-step's 36 KB stage with bulk copies
// into a 5-stage ring, warp 1's elected thread issues the MMAs and commits, warps 2-17 (four
// per TMEM lane quarter, 16 columns each) drain the level sums after each chunk and write
// the result (or, with split K, the exact partials T and F that a reduction kernel sums).
// The drain goes from level 5 to level 0 and frees each level by itself, and the next
// chunk's first two K-steps go A digit 5 first, which touches level 5 only, so the MMAs
// follow the drain down the levels instead of waiting for all of it. Measured at M 4096,
// N 2048, K 1024: the whole contraction 1580 us -> 1210 (the GEMM alone 1394 -> ~1020 us,
// 1.4 PFLOP/s of digit products) against two half tiles, eight drain warps and chunks
// drained whole. In cycles of a chunk: 9840, of which MMAs 5930, waits for the drain 2180 (it
// takes 2660) and for stages 1730 (36 KB a K-step from L2). One such K-step instead of two
// makes the contraction 3.6 % slower (it hides less), three 2.7 % (more MMAs); bringing A to L2
// ahead of the ring and a sixth stage change nothing.
// Every wait is bounded by a clock limit; on expiry the CTA records an error flag
// (qtnh_take_device_errors, bits 16-18), stops and frees its tensor memory.
//
// Rows or columns holding an infinity or NaN (largest exponent 0x7FF) are recomputed in
// FP64 by a fix-up kernel after the GEMM; results outside the double range are scaled
// with scalbn (overflow to infinity, gradual underflow), as FP64 arithmetic would give.

#include <algorithm>

#include "cuda_common.cuh"
#include "ozaki.cuh"

namespace qtnh_impl {

// bit 0: producer wait expired, bit 1: MMA wait expired, bit 2: epilogue wait expired
__device__ unsigned int g_ozg_error;

namespace {

constexpr int OG_M = 128;                  // rows of C^ per tile (64 complex rows)
constexpr int OG_N = 64;                   // columns of C per tile
constexpr int OG_EN = 16;                  // columns an epilogue thread drains
constexpr int OG_D = oz::NS;               // digits per real
constexpr int OG_L = oz::NL;               // levels kept
constexpr int OG_KSTEP = 16;               // bf16 K per MMA
constexpr uint32_t OG_CHUNK = 8;           // K-steps whose level sums are exact in FP32
constexpr uint32_t OG_HEAD = 2;            // first K-steps of a chunk issued digit by digit, behind the drain
constexpr int OG_A_DIGIT = OG_M * OG_KSTEP * 2;   // 4096 bytes
constexpr int OG_A_BLOCK = OG_D * OG_A_DIGIT;     // 24576 bytes: six A digits of one K-step
constexpr int OG_B_DIGIT = OG_N * OG_KSTEP * 2;   // 2048 bytes
constexpr int OG_B_BLOCK = OG_D * OG_B_DIGIT;     // 12288 bytes: six B digits of one K-step
constexpr int OG_STAGE = OG_A_BLOCK + OG_B_BLOCK;  // 36864 bytes
constexpr int OG_STAGES = 5;
constexpr int OG_THREADS = 576;  // warp 0 producer, warp 1 MMA, warps 2-17 epilogue
constexpr uint32_t OG_EPI_WARPS = 16;
constexpr uint32_t OG_TMEM_COLS = 512;
constexpr long long OG_WAIT_CYCLES = 1ll << 32;  // ~2 s at 2 GHz
constexpr uint32_t OG_SPECIAL = 0x7FFu;          // largest exponent of a row with an inf/NaN
static_assert(OG_L * OG_N <= OG_TMEM_COLS, "level sums exceed tensor memory");
static_assert(OG_N * OG_L <= 2 * 256, "an MMA's N is at most 256");

struct OzParams {
  const uint8_t* a_planes;  // MT x KS blocks of OG_A_BLOCK bytes
  const uint8_t* b_planes;  // NT x KS blocks of OG_B_BLOCK bytes
  const uint32_t* ea;       // largest biased exponent of each complex row of A (0: all zero)
  const uint32_t* eb;       // largest biased exponent of each column of B
  double2* C;               // M x N row-major (one slice)
  long long* tpart;         // S x (MT * OG_M) x (NT * OG_N) exact partials T (several slices)
  float* fpart;             // the same shape: partials F
  uint64_t M, N;
  uint32_t MT, NT, KS;      // row tiles of C^, column tiles, K-steps
  uint32_t S, SK;           // K-slices, K-steps per slice (a multiple of OG_CHUNK)
};

struct OgSmem {
  uint8_t stage[OG_STAGES][OG_STAGE];
  uint64_t full[OG_STAGES];
  uint64_t empty[OG_STAGES];
  uint64_t tfull;   // a chunk's level sums are complete
  uint64_t tempty[OG_L];  // the epilogue has drained a level
  uint64_t last;          // all MMAs issued are complete (after an expired wait)
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_thread(uint64_t* bar, uint32_t parity, volatile int* abort) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort != 0 || clock64() - t0 > OG_WAIT_CYCLES) return false;
  }
  return true;
}
// After an expired wait: gives the copies of the stages in flight time to land (~0.5 ms at most).
__device__ __forceinline__ void mbar_drain(uint64_t* full, uint32_t it) {
  const long long t0 = clock64();
  for (uint32_t x = it > (uint32_t)OG_STAGES ? it - OG_STAGES : 0; x < it; ++x)
    while (!mbar_try_wait(&full[x % OG_STAGES], (x / OG_STAGES) & 1u) && clock64() - t0 < (1 << 20)) {
    }
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort) {
  const long long t0 = clock64();
  while (true) {
    const bool ok = mbar_try_wait(bar, parity);
    if (__all_sync(0xffffffffu, ok)) return true;
    if (__any_sync(0xffffffffu, *abort != 0 || clock64() - t0 > OG_WAIT_CYCLES)) return false;
  }
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major, no swizzle, LBO 128 B, SBO 256 B, descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(256u >> 4) << 32) |
         (1ull << 46);
}

// kind::f16, D F32 (bits 4-5), A and B BF16 (bits 7-9, 10-12), K-major, N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t og_idesc(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((uint32_t)(OG_M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// A digit i of a stage (sd: the descriptor of its first byte) x its B digits j0 .. j1 - 1
// (stacked) -> levels i + j0 .. i + j1 - 1. One thread issues all: the descriptors are sums
// of constants and the stage's.
__device__ __forceinline__ void issue_digit(uint32_t tmem, uint64_t sd, int i, int j0, int j1, uint32_t acc) {
  const int rows = OG_N * (j1 - j0), parts = rows > 256 ? 2 : 1, n = rows / parts;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (q * n < rows && n > 0) {
      const int r0 = j0 * OG_N + q * n;  // first stacked B row
      umma_bf16(tmem + (uint32_t)(i * OG_N + r0), sd + (uint64_t)(i * (OG_A_DIGIT >> 4)),
                sd + (uint64_t)((OG_A_BLOCK + r0 * OG_KSTEP * 2) >> 4), og_idesc((uint32_t)n), acc);
    }
  }
}

// 16 consecutive 32-bit TMEM columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[OG_EN]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__global__ void __launch_bounds__(OG_THREADS, 1) gemm_oz6_umma_kernel(const __grid_constant__ OzParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  OgSmem& sm = *reinterpret_cast<OgSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint64_t ntiles = (uint64_t)p.MT * p.NT * p.S;
  // tile -> (column tile fastest, row tile, K-slice): neighbouring CTAs share the A rows
  auto tile_coords = [&](uint64_t tile, uint64_t& mt, uint64_t& nt, uint32_t& k0, uint32_t& k1) {
    nt = tile % p.NT;
    const uint64_t rest = tile / p.NT;
    mt = rest % p.MT;
    const uint32_t sl = (uint32_t)(rest / p.MT);
    k0 = sl * p.SK;
    k1 = min(p.KS, k0 + p.SK);
  };

  if (tid == 0) {
    sm.abort = 0;
    for (int s = 0; s < OG_STAGES; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.tfull, 1);
    for (int l = 0; l < OG_L; ++l) mbar_init(&sm.tempty[l], OG_EPI_WARPS);
    mbar_init(&sm.last, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(OG_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ---- producer: one elected thread streams each K-step's digits ----
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (uint64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
        uint64_t mt, nt;
        uint32_t k0, k1;
        tile_coords(tile, mt, nt, k0, k1);
        for (uint32_t ks = k0; ks < k1; ++ks, ++it) {
          const uint32_t s = it % OG_STAGES, ph = (it / OG_STAGES) & 1u;
          if (!mbar_wait_thread(&sm.empty[s], ph ^ 1u, &sm.abort)) {
            atomicOr(&g_ozg_error, 1u);
            sm.abort = 1;
            ok = false;
            mbar_drain(sm.full, it);
            break;
          }
          mbar_arrive_expect_tx(&sm.full[s], (uint32_t)OG_STAGE);
          bulk_g2s(&sm.stage[s][0], p.a_planes + (mt * p.KS + ks) * (uint64_t)OG_A_BLOCK, OG_A_BLOCK, &sm.full[s]);
          bulk_g2s(&sm.stage[s][OG_A_BLOCK], p.b_planes + (nt * p.KS + ks) * (uint64_t)OG_B_BLOCK, OG_B_BLOCK,
                   &sm.full[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA: one elected thread; a chunk of up to OG_CHUNK K-steps per accumulation ----
    if (lane == 0) {
      uint32_t st = 0, ph = 0, ch = 0;
      bool ok = true;
      const uint64_t sdesc = smem_desc(smem_u32(&sm.stage[0][0]));
      for (uint64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
        uint64_t mt, nt;
        uint32_t k0, k1;
        tile_coords(tile, mt, nt, k0, k1);
        for (uint32_t c0 = k0; ok && c0 < k1; c0 += OG_CHUNK, ++ch) {
          const uint32_t c1 = min(k1, c0 + OG_CHUNK);
          // the first K-steps: A digit 5 of all of them, then digit 4, ..: digit i needs levels
          // i .. 5 of the last chunk drained; on the first K-step it is the first to write level i
          const uint32_t g = min(c1 - c0, OG_HEAD);
          uint64_t sd[OG_HEAD];
          uint64_t* eb[OG_HEAD];
#pragma unroll
          for (uint32_t x = 0; x < OG_HEAD; ++x) {
            sd[x] = sdesc + (uint64_t)(st * (OG_STAGE >> 4));
            eb[x] = &sm.empty[st];
            if (x < g) {
              ok = ok && mbar_wait_thread(&sm.full[st], ph, &sm.abort);
              if (++st == OG_STAGES) st = 0, ph ^= 1u;
            }
          }
#pragma unroll
          for (int i = OG_D - 1; i >= 0; --i) {
            ok = ok && mbar_wait_thread(&sm.tempty[i], (ch & 1u) ^ 1u, &sm.abort);
            if (!ok) break;
            tc_fence_after();
            issue_digit(tmem, sd[0], i, 0, 1, 0u);
            issue_digit(tmem, sd[0], i, 1, OG_L - i, 1u);
            if (i == 0) umma_commit(eb[0]);  // the stage is free once its MMAs have read it
#pragma unroll
            for (uint32_t x = 1; x < OG_HEAD; ++x) {
              if (x >= g) break;
              issue_digit(tmem, sd[x], i, 0, OG_L - i, 1u);
              if (i == 0) umma_commit(eb[x]);
            }
          }
          for (uint32_t ks = c0 + g; ok && ks < c1; ++ks) {
            ok = mbar_wait_thread(&sm.full[st], ph, &sm.abort);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d = sdesc + (uint64_t)(st * (OG_STAGE >> 4));
#pragma unroll
            for (int i = 0; i < OG_D; ++i) issue_digit(tmem, d, i, 0, OG_L - i, 1u);
            umma_commit(&sm.empty[st]);
            if (++st == OG_STAGES) st = 0, ph ^= 1u;
          }
          if (!ok) {
            atomicOr(&g_ozg_error, 2u);
            sm.abort = 1;
            break;
          }
          umma_commit(&sm.tfull);
        }
      }
      // stopped early: the MMAs issued finish before tensor memory is freed (limited as well)
      if (!ok) {
        umma_commit(&sm.last);
        const long long t0 = clock64();
        while (!mbar_try_wait(&sm.last, 0) && clock64() - t0 < (1 << 20)) {
        }
      }
    }
  } else {
    // ---- epilogue: warp w drains TMEM lanes 32 (w % 4) .. +31, columns 16 ((w - 2) / 4) .. +15 ----
    const int q = warp & 3, h = (warp - 2) >> 2, r = q * 32 + lane;
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * OG_EN);
    uint32_t ch = 0;
    bool ok = true;
    for (uint64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
      uint64_t mt, nt;
      uint32_t k0, k1;
      tile_coords(tile, mt, nt, k0, k1);
      long long T[OG_EN];
      float F[OG_EN];
#pragma unroll
      for (int c = 0; c < OG_EN; ++c) T[c] = 0, F[c] = 0.0f;
      for (uint32_t c0 = k0; c0 < k1; c0 += OG_CHUNK, ++ch) {
        if (!mbar_wait_warp(&sm.tfull, ch & 1u, &sm.abort)) {
          atomicOr(&g_ozg_error, 4u);
          sm.abort = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        // level 5 first: the next chunk's MMAs on a level start when all warps have read it
        uint32_t va[OG_EN], vb[OG_EN];
        auto freed = [&](int l) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.tempty[l]);
        };
        auto add = [&](const uint32_t(&v)[OG_EN], int shift) {
#pragma unroll
          for (int c = 0; c < OG_EN; ++c) oz::gemm_add_high(__uint_as_float(v[c]), shift, T[c]);
        };
        tmem_ld16(tbase + 5 * OG_N, va);
        tmem_wait_ld();
        freed(5);
        tmem_ld16(tbase + 4 * OG_N, vb);
        tmem_wait_ld();
        freed(4);
#pragma unroll
        for (int c = 0; c < OG_EN; ++c) oz::gemm_add_low(__uint_as_float(vb[c]), __uint_as_float(va[c]), F[c]);
        tmem_ld16(tbase + 3 * OG_N, va);
        tmem_wait_ld();
        freed(3);
        tmem_ld16(tbase + 2 * OG_N, vb);
        add(va, 0);
        tmem_wait_ld();
        freed(2);
        tmem_ld16(tbase + 1 * OG_N, va);
        add(vb, 8);
        tmem_wait_ld();
        freed(1);
        tmem_ld16(tbase, vb);
        add(va, 16);
        tmem_wait_ld();
        freed(0);
        add(vb, 24);
      }
      if (!ok) break;
      const uint64_t R = mt * OG_M + (uint64_t)r;  // row of C^: complex row R / 2, part R % 2
      const uint64_t n0 = nt * OG_N + (uint64_t)(h * OG_EN);
      if (p.S > 1) {
        const uint64_t ld = (uint64_t)p.NT * OG_N;
        const uint64_t base = ((uint64_t)(k0 / p.SK) * p.MT * OG_M + R) * ld + n0;
#pragma unroll
        for (int c = 0; c < OG_EN; c += 2) {
          *reinterpret_cast<longlong2*>(p.tpart + base + c) = make_longlong2(T[c], T[c + 1]);
        }
#pragma unroll
        for (int c = 0; c < OG_EN; c += 4) {
          *reinterpret_cast<float4*>(p.fpart + base + c) = make_float4(F[c], F[c + 1], F[c + 2], F[c + 3]);
        }
        continue;
      }
      // one slice: the even lane (Re row) writes the thread's first 8 columns, the odd lane (Im
      // row) the other 8; each receives the other part from its partner
      const uint64_t m = R >> 1;
      const bool odd = (lane & 1) != 0;
      const uint32_t ea = m < p.M ? p.ea[m] : 0u;
#pragma unroll
      for (int x = 0; x < OG_EN / 2; ++x) {
        // columns x (kept by the even lane) and 8 + x (kept by the odd lane)
        const uint64_t nlo = n0 + (uint64_t)x, nhi = nlo + OG_EN / 2;
        const uint32_t eblo = nlo < p.N ? p.eb[nlo] : 0u, ebhi = nhi < p.N ? p.eb[nhi] : 0u;
        const double vlo = oz::gemm_finish(T[x], F[x], oz::gemm_scale(ea, eblo));
        const double vhi = oz::gemm_finish(T[OG_EN / 2 + x], F[OG_EN / 2 + x], oz::gemm_scale(ea, ebhi));
        const double keep = odd ? vhi : vlo;
        const double recv = __shfl_xor_sync(0xffffffffu, odd ? vlo : vhi, 1);
        const uint64_t nk = odd ? nhi : nlo;
        if (m < p.M && nk < p.N) p.C[m * p.N + nk] = odd ? make_double2(recv, keep) : make_double2(keep, recv);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OG_TMEM_COLS) : "memory");
  }
}

// Largest biased exponent of each of `rows` rows of X (rows x K complex128, row-major):
// one warp per row; 0 for an all-zero row, 0x7FF when the row holds an infinity or NaN.
__global__ void row_exponent_kernel(const double2* __restrict__ X, uint64_t rows, uint64_t K,
                                    uint32_t* __restrict__ e) {
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  for (uint64_t row = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    const double2* x = X + row * K;
    uint32_t key = 0;
    for (uint64_t k = lane; k < K; k += 32) {
      const double2 v = x[k];
      key = max(key, max(oz::group_key(df::words(v.x)), oz::group_key(df::words(v.y))));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
    if (lane == 0) e[row] = oz::key_exponent(key);
  }
}

// Byte offset of the 16-byte core row (row rr of the tile, K-core kc) in digit `i` of
// the A block of (row tile, K-step).
__device__ __forceinline__ uint64_t og_a_offset(uint64_t row, uint64_t kc, int i, uint32_t KS) {
  const uint64_t mt = row >> 7, rr = row & 127;
  return ((mt * KS + (kc >> 1)) * OG_D + (uint64_t)i) * OG_A_DIGIT + ((rr >> 3) << 8) + ((kc & 1) << 7) + ((rr & 7) << 4);
}
// The same for B: column n (tile n / 64, row n % 64).
__device__ __forceinline__ uint64_t og_b_offset(uint64_t n, uint64_t kc, int j, uint32_t KS) {
  const uint64_t nt = n >> 6, rr = n & 63;
  return ((nt * KS + (kc >> 1)) * OG_D + (uint64_t)j) * OG_B_DIGIT + ((rr >> 3) << 8) + ((kc & 1) << 7) + ((rr & 7) << 4);
}

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) { return oz::pack(lo, hi); }

// A^ digits: thread per (complex row m, K-core kc = complex columns 4 kc .. 4 kc + 3),
// consecutive threads on consecutive rows (their 16-byte core rows are contiguous).
// Rows 2m (Re a, -Im a) and 2m + 1 (Im a, Re a). Padding rows and columns are zero.
__global__ void oz_digits_a_kernel(const double2* __restrict__ A, const uint32_t* __restrict__ ea, uint64_t M,
                                   uint64_t K, uint64_t Mc, uint32_t KS, uint8_t* __restrict__ planes) {
  const uint64_t kcs = (uint64_t)KS * 2;
  const uint64_t total = Mc * kcs;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t m = t % Mc, kc = t / Mc;
    const uint32_t e = m < M ? ea[m] : 0u;
    const uint32_t es = oz::digit_scale(e);
    float re[4][OG_D], im[4][OG_D];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const uint64_t k = kc * 4 + x;
      const double2 a = (m < M && k < K && e != OG_SPECIAL) ? A[m * K + k] : make_double2(0.0, 0.0);
      oz::digits(df::words(a.x), es, re[x]);
      oz::digits(df::words(a.y), es, im[x]);
    }
#pragma unroll
    for (int i = 0; i < OG_D; ++i) {
      // row 2m: (Re, -Im) per complex column; row 2m + 1: (Im, Re)
      const uint4 r0 = make_uint4(bf16_pair(re[0][i], -im[0][i]), bf16_pair(re[1][i], -im[1][i]),
                                  bf16_pair(re[2][i], -im[2][i]), bf16_pair(re[3][i], -im[3][i]));
      const uint4 r1 = make_uint4(bf16_pair(im[0][i], re[0][i]), bf16_pair(im[1][i], re[1][i]),
                                  bf16_pair(im[2][i], re[2][i]), bf16_pair(im[3][i], re[3][i]));
      *reinterpret_cast<uint4*>(planes + og_a_offset(2 * m, kc, i, KS)) = r0;
      *reinterpret_cast<uint4*>(planes + og_a_offset(2 * m + 1, kc, i, KS)) = r1;
    }
  }
}

// B^ digits: thread per (column n, K-core kc = complex rows 4 kc .. 4 kc + 3) of B''
// (N x K row-major): B^[n][2k] = Re b, B^[n][2k+1] = Im b.
__global__ void oz_digits_b_kernel(const double2* __restrict__ Bt, const uint32_t* __restrict__ eb, uint64_t N,
                                   uint64_t K, uint64_t Nc, uint32_t KS, uint8_t* __restrict__ planes) {
  const uint64_t kcs = (uint64_t)KS * 2;
  const uint64_t total = Nc * kcs;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t n = t % Nc, kc = t / Nc;
    const uint32_t e = n < N ? eb[n] : 0u;
    const uint32_t es = oz::digit_scale(e);
    float re[4][OG_D], im[4][OG_D];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const uint64_t k = kc * 4 + x;
      const double2 b = (n < N && k < K && e != OG_SPECIAL) ? Bt[n * K + k] : make_double2(0.0, 0.0);
      oz::digits(df::words(b.x), es, re[x]);
      oz::digits(df::words(b.y), es, im[x]);
    }
#pragma unroll
    for (int j = 0; j < OG_D; ++j) {
      const uint4 v = make_uint4(bf16_pair(re[0][j], im[0][j]), bf16_pair(re[1][j], im[1][j]),
                                 bf16_pair(re[2][j], im[2][j]), bf16_pair(re[3][j], im[3][j]));
      *reinterpret_cast<uint4*>(planes + og_b_offset(n, kc, j, KS)) = v;
    }
  }
}

// C[m][n] from the S slices' exact partials of rows 2m (Re) and 2m + 1 (Im) of C^.
__global__ void oz_reduce_kernel(const long long* __restrict__ Tp, const float* __restrict__ Fp, uint32_t S,
                                 uint64_t rows, uint64_t ld, const uint32_t* __restrict__ ea,
                                 const uint32_t* __restrict__ eb, double2* __restrict__ C, uint64_t M, uint64_t N) {
  const uint64_t total = M * N;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t m = i / N, n = i % N;
    long long tr = 0, ti = 0;
    float fr = 0.0f, fi = 0.0f;
    for (uint32_t s = 0; s < S; ++s) {
      const uint64_t b = (uint64_t)s * rows * ld + (2 * m) * ld + n;
      tr += Tp[b];
      fr += Fp[b];
      ti += Tp[b + ld];
      fi += Fp[b + ld];
    }
    const int e = oz::gemm_scale(ea[m], eb[n]);
    C[i] = make_double2(oz::gemm_finish(tr, fr, e), oz::gemm_finish(ti, fi, e));
  }
}

// Outputs of rows of A or columns of B that hold an infinity or NaN, in FP64 (the
// digits cannot carry them); the kernel returns at once unless `flag` is set.
__global__ void oz_special_kernel(const double2* __restrict__ A, const double2* __restrict__ Bt,
                                  const uint32_t* __restrict__ ea, const uint32_t* __restrict__ eb,
                                  const uint32_t* __restrict__ flag, double2* __restrict__ C, uint64_t M, uint64_t N,
                                  uint64_t K) {
  if (*flag == 0u) return;
  const uint64_t total = M * N;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t m = i / N, n = i % N;
    if (ea[m] != OG_SPECIAL && eb[n] != OG_SPECIAL) continue;
    double2 acc = make_double2(0.0, 0.0);
    for (uint64_t k = 0; k < K; ++k) acc = cfma(A[m * K + k], Bt[n * K + k], acc);
    C[i] = acc;
  }
}

// Flags whether any row exponent is 0x7FF.
__global__ void oz_any_special_kernel(const uint32_t* __restrict__ e, uint64_t n, uint32_t* __restrict__ flag) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    if (e[i] == OG_SPECIAL) atomicOr(flag, 1u);
}

}  // namespace

// C (M x N) = A'' (M x K) B''^T, with A'' and B'' (N x K) complex128 row-major, on the
// tensor cores through exact digit products (see the file header).
void gemm_oz6(const void* Av, const void* Btv, void* Cv, uint64_t M, uint64_t N, uint64_t K, void* stream) {
  if (M == 0 || N == 0) return;
  const c128* A = static_cast<const c128*>(Av);
  const c128* Bt = static_cast<const c128*>(Btv);
  c128* C = static_cast<c128*>(Cv);
  cudaStream_t s = (cudaStream_t)stream;
  if (K == 0) {
    check_cuda(cudaMemsetAsync(C, 0, M * N * sizeof(c128), s), "zero C");
    return;
  }
  const uint64_t Kp = (K + 7) / 8 * 8;  // complex K padded: 2 Kp reals = KS K-steps
  const uint32_t KS = (uint32_t)(2 * Kp / OG_KSTEP);
  OzParams p{};
  p.MT = (uint32_t)((2 * M + OG_M - 1) / OG_M);
  p.NT = (uint32_t)((N + OG_N - 1) / OG_N);
  p.KS = KS;
  p.M = M;
  p.N = N;
  p.C = C;
  const uint64_t a_bytes = (uint64_t)p.MT * KS * OG_A_BLOCK;
  const uint64_t b_bytes = (uint64_t)p.NT * KS * OG_B_BLOCK;
  // split K over chunk-aligned slices when the tiles alone would leave SMs idle
  const uint64_t tiles = (uint64_t)p.MT * p.NT;
  const uint32_t chunks = (KS + OG_CHUNK - 1) / OG_CHUNK;
  uint32_t S = 1;
  if (tiles < (uint64_t)sm_count()) S = (uint32_t)std::min<uint64_t>(chunks, ((uint64_t)sm_count() + tiles - 1) / tiles);
  p.SK = ((chunks + S - 1) / S) * OG_CHUNK;
  p.S = (KS + p.SK - 1) / p.SK;
  const uint64_t rows = (uint64_t)p.MT * OG_M, ld = (uint64_t)p.NT * OG_N;
  const uint64_t part = p.S > 1 ? (uint64_t)p.S * rows * ld : 0;
  const uint64_t e_bytes = ((M + N + 64) * sizeof(uint32_t) + 255) / 256 * 256;
  const uint64_t bytes = a_bytes + b_bytes + e_bytes + part * (sizeof(long long) + sizeof(float));
  uint8_t* ws = static_cast<uint8_t*>(workspace_alloc(bytes, stream));
  try {
    uint8_t* apl = ws;
    uint8_t* bpl = ws + a_bytes;
    uint32_t* ea = reinterpret_cast<uint32_t*>(ws + a_bytes + b_bytes);
    uint32_t* eb = ea + M;
    uint32_t* flag = eb + N;
    p.a_planes = apl;
    p.b_planes = bpl;
    p.ea = ea;
    p.eb = eb;
    p.tpart = p.S > 1 ? reinterpret_cast<long long*>(ws + a_bytes + b_bytes + e_bytes) : nullptr;
    p.fpart = p.S > 1 ? reinterpret_cast<float*>(ws + a_bytes + b_bytes + e_bytes + part * sizeof(long long)) : nullptr;
    row_exponent_kernel<<<grid_for((M + 7) / 8, 8), 256, 0, s>>>(A, M, K, ea);
    row_exponent_kernel<<<grid_for((N + 7) / 8, 8), 256, 0, s>>>(Bt, N, K, eb);
    count_launch(2);
    const uint64_t Mc = (uint64_t)p.MT * (OG_M / 2), Nc = (uint64_t)p.NT * OG_N;
    oz_digits_a_kernel<<<grid_for((Mc * 2 * KS + 255) / 256, 8), 256, 0, s>>>(A, ea, M, K, Mc, KS, apl);
    oz_digits_b_kernel<<<grid_for((Nc * 2 * KS + 255) / 256, 8), 256, 0, s>>>(Bt, eb, N, K, Nc, KS, bpl);
    count_launch(2);
    const size_t smem = sizeof(OgSmem);
    check_cuda(cudaFuncSetAttribute(gemm_oz6_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "gemm_oz6_umma_kernel shared memory");
    const int grid = (int)std::min<uint64_t>((uint64_t)p.MT * p.NT * p.S, (uint64_t)sm_count());
    gemm_oz6_umma_kernel<<<grid, OG_THREADS, smem, s>>>(p);
    count_launch();
    if (p.S > 1) {
      oz_reduce_kernel<<<grid_for((M * N + 255) / 256, 8), 256, 0, s>>>(p.tpart, p.fpart, p.S, rows, ld, ea, eb, C, M,
                                                                          N);
      count_launch();
    }
    // rows / columns with an infinity or NaN: recomputed in FP64 on the device (in the
    // common case the second kernel reads the cleared flag and returns)
    check_cuda(cudaMemsetAsync(flag, 0, sizeof(uint32_t), s), "clear flag");
    oz_any_special_kernel<<<grid_for((M + N + 255) / 256, 2), 256, 0, s>>>(ea, M + N, flag);
    oz_special_kernel<<<grid_for((M * N + 255) / 256, 4), 256, 0, s>>>(A, Bt, ea, eb, flag, C, M, N, K);
    count_launch(2);
    check_cuda(cudaGetLastError(), "digit GEMM launch");
  } catch (...) {
    workspace_free(ws, stream);
    throw;
  }
  workspace_free(ws, stream);
}

uint32_t take_ozg_error() {
  uint32_t v = 0;
  check_cuda(cudaMemcpyFromSymbol(&v, g_ozg_error, sizeof(v)), "read device error flags");
  const uint32_t zero = 0;
  check_cuda(cudaMemcpyToSymbol(g_ozg_error, &zero, sizeof(zero)), "clear device error flags");
  return v;
}

}  // namespace qtnh_impl
