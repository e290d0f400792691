// FP64-accurate products on the integer tensor cores (see ozaki.hpp).
//
// ozk_gemm_kernel<S, T>: one CTA of 128 threads (256 for the narrow tiles) per
// output tile of 128 rows x CN columns.  Thread 0 of warp 0 streams 64-byte K slices of the S digit
// planes of both operands into a ring of shared-memory stages by TMA
// (cp.async.bulk.tensor, 64-byte swizzle, completion on an mbarrier per
// stage); thread 0 of warp 1 issues, per stage and per 32-byte K step, the
// S(S+1)/2 digit products (tcgen05.mma.cta_group::1.kind::i8, both operands
// K-major in shared memory, signed 8-bit, 32-bit integer accumulators) into
// S accumulators of 128 x CN in tensor memory, one per digit-weight group
// (the products of one X plane with a stack of W planes as one MMA of N up
// to 256, see ozk_issue_kstep), and frees each stage with tcgen05.commit on
// its "empty" mbarrier.  After
// the last stage all warps read their 32 rows of the accumulators
// (tcgen05.ld 32x32b), combine the groups with their powers of two, apply
// the row and column exponents (loaded by warps 2 and 3 while the products
// run) and store their row segments.
//
// Two digit formats: signed 8-bit digits multiplied by tcgen05.mma
// kind::i8 into 32-bit integer accumulators, or the same digits held in
// bf16 (every integer of magnitude <= 256 is exact there) multiplied by
// kind::f16 into FP32 accumulators, exact while every partial sum stays
// below 2^24 in magnitude (S * 64 * 64 * Kp < 2^24, checked on the host).
// The products are bit-identical; which is faster depends on the tensor
// pipe's integer and bf16 rates, so callers time both.
//
// Four shapes: one CTA per SM per tile (all 512 tensor-memory columns, CN
// = 144 / 112 / 96 / 64 columns for S = 3 / 4 / 5 / 6-7, up to four
// stages); for S <= 5, two CTAs per SM (256 columns each, CN = 64 / 64 / 48,
// two stages), where one CTA's epilogue overlaps the other's products; for S
// <= 5 the persistent ozk_gemm_pers_kernel (one CTA per SM, its weights' tile
// of width 64 / 64 / 48 resident, two accumulator sets); and, for 8-bit
// digits, tiles of 16 columns for operands of few rows, where the wide tiles
// leave most SMs without one.
//
// Every mbarrier wait is bounded (2^20 polls).  A wait that runs out marks
// the tile's rows in the caller's status words; the producer then waits
// (bounded) for the copies it issued that nobody consumed, the epilogue
// waits (bounded) for the issued products, and tensor memory is freed
// before the CTA exits.  TMA loads read this GPU's own memory only and use
// no cluster multicast.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ozaki.hpp"
#include "tma.cuh"

namespace scy {
namespace {

constexpr int OZK_BM = 128;  // rows per tile (tensor-memory lanes)
constexpr int OZK_BK = 64;   // bytes of K per stage (one 64-byte swizzle row)
constexpr int OZK_POLLS = 1 << 20;
constexpr int OZK_SMEM_BUDGET = 220 * 1024;

// PAIR = 0: one CTA per SM; PAIR = 1: two (S <= 5); PAIR = 2: narrow tiles
// for few rows
constexpr int OZK_NARROW = 16;
__host__ __device__ constexpr int ozk_cn(int S, int pair = 0) {
  return pair == 2 ? OZK_NARROW : pair ? (S <= 4 ? 64 : 48) : (S <= 3 ? 144 : S == 4 ? 112 : S == 5 ? 96 : 64);
}
__host__ __device__ constexpr int ozk_tmem_cols(int pair) { return pair == 2 ? 128 : pair ? 256 : 512; }
__host__ __device__ constexpr int ozk_stage_bytes(int S, int pair = 0) {
  return S * OZK_BM * OZK_BK + S * ozk_cn(S, pair) * OZK_BK;
}
__host__ __device__ constexpr int ozk_stages(int S, int pair = 0) {
  return pair == 1 ? 2 : OZK_SMEM_BUDGET / ozk_stage_bytes(S, pair) > 4 ? 4 : OZK_SMEM_BUDGET / ozk_stage_bytes(S, pair);
}
// the stage ring starts on a 1024-byte (one CTA per SM) or 512-byte (two)
// boundary: the 64-byte swizzle repeats every 512 bytes
__host__ __device__ constexpr int ozk_align(int pair) { return pair == 1 ? 512 : 1024; }
__host__ __device__ constexpr int ozk_smem_bytes(int S, int pair = 0) {
  return ozk_stages(S, pair) * ozk_stage_bytes(S, pair) + ozk_align(pair);
}
// the persistent shape (S <= 5): the two-CTAs-per-SM tile width (S * CN <=
// 256, so two accumulator sets fit the 512 tensor-memory columns), all nkb
// K slices of the weights' tile resident, and as many stages of X as fit
// beside them (0: does not fit)
__host__ __device__ constexpr int ozk_pers_x_bytes(int S) { return S * OZK_BM * OZK_BK; }
__host__ __device__ constexpr int ozk_pers_w_bytes(int S) { return S * ozk_cn(S, 1) * OZK_BK; }
constexpr int OZK_PERS_MAX_STAGES = 4;
constexpr int OZK_PERS_MAX_SLICES = 16;
inline int ozk_pers_stages(int S, int nkb) {
  const int left = 227 * 1024 - 1024 - 1024 - nkb * ozk_pers_w_bytes(S);  // static, alignment, weights
  const int st = left > 0 ? left / ozk_pers_x_bytes(S) : 0;
  return nkb > OZK_PERS_MAX_SLICES || st < 2 ? 0 : st > OZK_PERS_MAX_STAGES ? OZK_PERS_MAX_STAGES : st;
}
// per CTA beside the stages: the reserved kilobyte, the barriers and the
// epilogue's exponent factors (CN + 128 doubles)
static_assert(2 * (ozk_smem_bytes(5, 1) + 1024 + 256 + 8 * (ozk_cn(5, 1) + 128)) <= 228 * 1024,
              "two CTAs per SM do not fit");
static_assert(2 * (ozk_smem_bytes(4, 1) + 1024 + 256 + 8 * (ozk_cn(4, 1) + 128)) <= 228 * 1024,
              "two CTAs per SM do not fit");
static_assert(2 * (ozk_smem_bytes(3, 1) + 1024 + 256 + 8 * (ozk_cn(3, 1) + 128)) <= 228 * 1024,
              "two CTAs per SM do not fit");

// shared-memory matrix descriptor (tcgen05 format): K-major operand whose
// rows are 64 bytes with 64-byte swizzling, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);  // start address, 16-byte units
  d |= (uint64_t)1u << 16;                  // leading byte offset (unused by swizzled K-major layouts)
  d |= (uint64_t)(512u >> 4) << 32;         // stride byte offset: next 8-row group
  d |= (uint64_t)1u << 46;                  // descriptor version of sm_100
  d |= (uint64_t)4u << 61;                  // layout: 64-byte swizzle
  return d;
}

// 2^e as a double (exact), by its bit pattern in the normal range
__device__ __forceinline__ double pow2i(int e) {
  return (e >= -1022 && e <= 1023) ? __longlong_as_double((long long)(e + 1023) << 52) : ldexp(1.0, e);
}

// instruction descriptor: signed 8-bit A and B, K-major, 32-bit integer
// accumulator, M = 128, N = n
__host__ __device__ constexpr uint32_t umma_idesc_s8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZK_BM >> 4) << 24);
}

// instruction descriptor: bf16 A and B, K-major, FP32 accumulator, M = 128,
// N = n
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZK_BM >> 4) << 24);
}

__device__ __forceinline__ void umma_s8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[16]) { tmem_ld16(taddr, v); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[8]) { tmem_ld8(taddr, v); }

// The digit products of one 32-byte K step: X plane p times the stack of W
// planes 1 .. S+1-p.  Their products belong to the consecutive groups
// p-1 .. S-1, whose accumulators are consecutive in tensor memory, and the
// W planes are consecutive CN-row blocks of the stage, so one MMA of N =
// planes x CN (at most 256) covers as many of them as fit: the A tile is read
// once per MMA instead of once per product.  Integer (and the exact FP32)
// sums are the same in any order.  first: the tile's first K step (the
// products of X plane 1 start every group).
template <int S, int CN, int BF>
__device__ __forceinline__ void ozk_issue_kstep(uint32_t tacc, uint32_t xa, uint32_t wa, int ks, bool first) {
  constexpr int PER = 256 / CN;  // W planes per MMA
#pragma unroll
  for (int p = 1; p <= S; ++p) {
#pragma unroll
    for (int j0 = 1; j0 <= S + 1 - p; j0 += PER) {
      const int np = (S + 2 - p - j0) < PER ? (S + 2 - p - j0) : PER;
      const uint64_t ad = umma_desc_sw64(xa + (p - 1) * OZK_BM * OZK_BK + ks * 32);
      const uint64_t bd = umma_desc_sw64(wa + (j0 - 1) * CN * OZK_BK + ks * 32);
      const uint32_t idesc = BF ? umma_idesc_bf16(np * CN) : umma_idesc_s8(np * CN);
      const uint32_t acc = (first && p == 1) ? 0u : 1u;
      if (BF)
        umma_bf16(tacc + (p + j0 - 2) * CN, ad, bd, idesc, acc);
      else
        umma_s8(tacc + (p + j0 - 2) * CN, ad, bd, idesc, acc);
    }
  }
}

// Threads of a tile: four warps, or eight for the narrow tiles, where the
// epilogue (S FP64 conversions and sums an output) is a third of the kernel.
__host__ __device__ constexpr int ozk_threads(int pair) { return pair == 2 ? 256 : 128; }

template <int S, typename T, int PAIR, int BF>
__global__ void __launch_bounds__(ozk_threads(PAIR), PAIR == 1 ? 2 : 1)
    ozk_gemm_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw,
                    const int* __restrict__ ex, const int* __restrict__ ew, T* __restrict__ D, long ldd, int rows,
                    int cout, int nks, unsigned* __restrict__ status, int rows_per_status, unsigned bit) {
  constexpr int CN = ozk_cn(S, PAIR);
  constexpr int XB = S * OZK_BM * OZK_BK;
  constexpr int WB = S * CN * OZK_BK;
  constexpr int ST = ozk_stages(S, PAIR);
  constexpr int NT = ozk_threads(PAIR), EC = PAIR == 2 ? 8 : 16;  // columns a warp combines at a time
  constexpr int TC = ozk_tmem_cols(PAIR);
  constexpr unsigned AL = ozk_align(PAIR);
  static_assert(S * CN <= TC, "accumulators exceed tensor memory");
  static_assert(PAIR != 1 || S <= 5, "two CTAs per SM only for S <= 5");
  static_assert(CN % 16 == 0 && CN >= 16 && CN <= 256, "invalid MMA N");
  extern __shared__ __align__(1024) unsigned char ozk_smem_raw[];
  __shared__ __align__(8) uint64_t full[ST], empty[ST], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int consumed, failed;
  __shared__ double s_sw[CN], s_xs[OZK_BM];  // 2^ew of the tile's columns, 2^ex of its rows
  // tiles on a 1024- or 512-byte boundary (the swizzle pattern repeats every 512 B)
  unsigned char* smem = ozk_smem_raw + ((AL - (smem_u32(ozk_smem_raw) & (AL - 1))) & (AL - 1));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // column tiles vary fastest (the CTAs that run together share a row tile
  // of X and spread over the tiles of W), and each CTA starts its K loop at
  // its own stage (integer partial sums are exact in any order), so the
  // CTAs reading one W tile at a time read different parts of it
  const int c0 = blockIdx.x * CN, m0 = blockIdx.y * OZK_BM;

  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&done, 1);
    fence_mbar_init();
    consumed = 0;
    failed = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "n"(TC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  // K in 32-byte MMA steps (nks), two per 64-byte stage; the last stage may
  // hold one.  N of the products: the tile's columns rounded up to 16 (the
  // last column tile is narrower than CN)
  const int nkb = (nks + 1) / 2;
  const int rot = (int)((blockIdx.x * 7u + blockIdx.y) % (unsigned)nkb);
  const int nmma = min(CN, (cout - c0 + 15) / 16 * 16);
  int issued = 0;
  if (warp == 0 && lane == 0) {
    // the weights (laid out at set-up) of the first stages ahead of the wait
    // for the kernel that makes X: with this and the sweeps' tables loaded
    // likewise, four chained steps take 1208 us at 401 x 401 and 813 at 101 x
    // 101 (1262 and 848 with the wait first)
    for (int q = 0; q < min(ST, nkb); ++q) {
      mbar_expect_tx(&full[q], XB + WB);
      tma_load_3d(smem + q * (XB + WB) + XB, &mw, &full[q], (q + rot) % nkb * (OZK_BK / (BF ? 2 : 1)), c0, 0);
    }
  }
  __syncwarp();
  chain_enter();
  if (warp >= 2) {
    // the epilogue's exponent factors, loaded while the products run
    for (int i = threadIdx.x - 64; i < CN + OZK_BM; i += NT - 64) {
      if (i < CN)
        s_sw[i] = c0 + i < cout ? pow2i(ew[c0 + i]) : 0.0;
      else
        s_xs[i - CN] = m0 + (i - CN) < rows ? pow2i(ex[m0 + (i - CN)]) : 0.0;
    }
  }
  if (warp == 0 && lane == 0) {
    // producer
    for (int q = 0; q < nkb; ++q) {
      const int st = q % ST, kb = (q + rot) % nkb;
      if (q >= ST && !mbar_wait(&empty[st], ((q / ST) - 1) & 1, OZK_POLLS)) {
        failed = 1;
        break;
      }
      unsigned char* sx = smem + st * (XB + WB);
      if (q >= ST) mbar_expect_tx(&full[st], XB + WB);
      // x coordinate in digits: 64 bytes of K per stage
      tma_load_3d(sx, &mx, &full[st], kb * (OZK_BK / (BF ? 2 : 1)), m0, 0);
      if (q >= ST) tma_load_3d(sx + XB, &mw, &full[st], kb * (OZK_BK / (BF ? 2 : 1)), c0, 0);
      ++issued;
    }
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    int q = 0;
    for (; q < nkb; ++q) {
      const int st = q % ST, kb = (q + rot) % nkb;
      if (!mbar_wait(&full[st], (q / ST) & 1, OZK_POLLS)) {
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t xa = smem_u32(smem + st * (XB + WB));
      const uint32_t wa = xa + XB;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        if (2 * kb + ks >= nks) break;
        ozk_issue_kstep<S, CN, BF>(tmem, xa, wa, ks, q == 0 && ks == 0);
      }
      umma_commit(&empty[st]);
    }
    consumed = q;
    umma_commit(&done);  // arrives once every product issued above has completed
  }
  __syncthreads();
  if (warp == 0 && lane == 0) {
    // copies issued but never consumed (only after a wait ran out)
    for (int q = consumed; q < issued; ++q) mbar_wait(&full[q % ST], (q / ST) & 1, OZK_POLLS);
  }
  // one decision for the whole block: the warp-collective tensor-memory
  // loads below run in every warp or in none
  const bool ok = __syncthreads_and(mbar_wait(&done, 0, OZK_POLLS) ? 1 : 0) && !failed;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok) {
    if (threadIdx.x == 0 && status) {
      const int r1 = min(m0 + OZK_BM, rows) - 1;
      for (int q = m0 / rows_per_status; q <= r1 / rows_per_status; ++q) atomicOr(status + q, bit);
    }
  } else {
    // epilogue: warp w owns tensor-memory lanes 32 (w % 4) .. + 31 (rows);
    // a thread combines its row's groups, EC columns at a time (of eight
    // warps, every second EC columns), applies the exponent factors (exact
    // powers of two, loaded during the products) and stores the values of
    // its row segment
    const int rl = (warp & 3) * 32 + lane, row = m0 + rl;
    const double xs = s_xs[rl];
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int cc = (warp >> 2) * EC; cc < nmma; cc += NT / 128 * EC) {
      uint32_t v[S][EC];
#pragma unroll
      for (int g = 0; g < S; ++g) tmem_ld(tl + g * CN + cc, v[g]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      double acc[EC];
      if constexpr (S <= 5) {
        // sum_g P_g 2^(-7 (g+2)) as one 64-bit integer (|P_g| < 2^24, so
        // the Horner sum stays below 2^52) times 2^(-7 (S+1)): exact, the
        // same value as the FP64 sum below, with one conversion per output
#pragma unroll
        for (int q = 0; q < EC; ++q) {
          long long h = 0;
#pragma unroll
          for (int g = 0; g < S; ++g) h = (h << 7) + (long long)(BF ? (int)__uint_as_float(v[g][q]) : (int)v[g][q]);
          acc[q] = (double)h * pow2i(-7 * (S + 1));
        }
      } else {
        // smallest weights first; the five smallest as one 64-bit integer
        // (below 2^53 while |P_g| < 2^24, as their FP64 sum, so the same
        // value: one conversion instead of five)
#pragma unroll
        for (int q = 0; q < EC; ++q) {
          long long h = 0;
#pragma unroll
          for (int g = S - 5; g < S; ++g)
            h = (h << 7) + (long long)(BF ? (int)__uint_as_float(v[g][q]) : (int)v[g][q]);
          acc[q] = (double)h * pow2i(-7 * (S + 1));
        }
#pragma unroll
        for (int g = S - 6; g >= 0; --g) {
          const double wgt = pow2i(-7 * (g + 2));
#pragma unroll
          for (int q = 0; q < EC; ++q)
            acc[q] += (BF ? (double)__uint_as_float(v[g][q]) : (double)(int)v[g][q]) * wgt;
        }
      }
      if (row < rows) {
        T* drow = D + (long)row * ldd + c0 + cc;
#pragma unroll
        for (int q = 0; q < EC; ++q)
          if (c0 + cc + q < cout) drow[q] = (T)((acc[q] * xs) * s_sw[cc + q]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TC) : "memory");
}

// four consecutive FP64 values to a 32-byte boundary in one store
__device__ __forceinline__ void st_v4(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// ozk_gemm_pers_kernel<S, T, BF> (S <= 5): the same product as a persistent
// kernel for many rows.  A CTA (one per SM) keeps one column tile of CN
// columns (CN of the two-CTAs-per-SM shape, S * CN <= 256): all K slices of
// its W digits stay in shared memory, so only X streams, through a ring of
// nst stages, and it walks the row tiles b / ntc, + G_ct, .. of its column
// (b = blockIdx.x, column tile b % ntc, G_ct the CTAs of that column).  The
// S W planes of a K slice lie one behind the other, so the products of an X
// plane with all its W planes are one MMA of N = (S + 1 - p) CN <= 240: five
// MMAs a 32-byte K step at S = 5.  The accumulators are double-buffered in
// tensor memory (columns 0..255 and 256..511), so the epilogue of one row
// tile runs while the products of the next are issued.  Thread 0 of warp 0
// loads, thread 0 of warp 1 issues the products and marks a buffer complete
// (accf, by tcgen05.commit); warps 4..11 (tensor-memory lanes 32 (w % 4) ..,
// the column chunks split between the two warps of a quadrant) read, combine
// and store it and mark it free (acce, one arrival per warp).  A thread
// stores its row's columns as whole 32-byte sectors where the row is aligned.
// Same digit formats and the same results as ozk_gemm_kernel.  Every wait is
// bounded; a role whose wait runs out stops, the others stop at their next
// bounded wait or at the shared flag, issued copies and products are awaited
// (bounded) before the tensor memory is freed, and the rows of every tile
// of the CTA are marked in the caller's status words.
template <int S, typename T, int BF>
__global__ void __launch_bounds__(384, 1)
    ozk_gemm_pers_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw,
                         const int* __restrict__ ex, const int* __restrict__ ew, T* __restrict__ D, long ldd,
                         int rows, int cout, int nks, int nst, unsigned* __restrict__ status, int rows_per_status,
                         unsigned bit) {
  chain_enter();
  constexpr int CN = ozk_cn(S, 1);
  constexpr int XB = ozk_pers_x_bytes(S);
  constexpr int WB = ozk_pers_w_bytes(S);
  constexpr int EW = 8;  // epilogue warps
  static_assert(S <= 5 && S * CN <= 256, "two accumulator sets must fit the tensor memory");
  static_assert(CN % 16 == 0 && CN >= 32, "invalid MMA N");
  extern __shared__ __align__(1024) unsigned char ozk_smem_raw[];
  __shared__ __align__(8) uint64_t full[OZK_PERS_MAX_STAGES], empty[OZK_PERS_MAX_STAGES], wbar[OZK_PERS_MAX_SLICES],
      accf[2], acce[2], done;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int failed;
  __shared__ int issued_q, consumed_q, issued_w;
  __shared__ double s_sw[CN];  // 2^ew of the column tile
  unsigned char* smem = ozk_smem_raw + ((1024u - (smem_u32(ozk_smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntc = (cout + CN - 1) / CN, ntr = (rows + OZK_BM - 1) / OZK_BM;
  const int ct = blockIdx.x % ntc, rt0 = blockIdx.x / ntc, rstep = ((int)gridDim.x - ct + ntc - 1) / ntc;
  const int c0 = ct * CN;
  const int nkb = (nks + 1) / 2;
  unsigned char* sw = smem;             // [nkb][S][CN][64 bytes]
  unsigned char* sx = smem + nkb * WB;  // [nst][S][128][64 bytes]

  if (threadIdx.x == 0) {
    for (int i = 0; i < nst; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < nkb; ++i) mbar_init(&wbar[i], 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], EW);
    }
    mbar_init(&done, 1);
    fence_mbar_init();
    failed = 0;
    issued_q = 0;
    consumed_q = 0;
    issued_w = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 2)
    for (int i = lane; i < CN; i += 32) s_sw[i] = c0 + i < cout ? pow2i(ew[c0 + i]) : 0.0;
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == 0 && lane == 0) {
    // producer
    int q = 0;
    bool ok = true;
    for (int rt = rt0; rt < ntr && ok && !failed; rt += rstep) {
      for (int k = 0; k < nkb; ++k) {
        if (rt == rt0) {
          mbar_expect_tx(&wbar[k], WB);
          tma_load_3d(sw + k * WB, &mw, &wbar[k], k * (OZK_BK / (BF ? 2 : 1)), c0, 0);
          issued_w = k + 1;
        }
        const int st = q % nst;
        if (q >= nst && !mbar_wait(&empty[st], ((q / nst) - 1) & 1, OZK_POLLS)) {
          failed = 1;
          ok = false;
          break;
        }
        mbar_expect_tx(&full[st], XB);
        tma_load_3d(sx + st * XB, &mx, &full[st], k * (OZK_BK / (BF ? 2 : 1)), rt * OZK_BM, 0);
        ++q;
      }
    }
    issued_q = q;
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    int q = 0, i = 0;
    bool ok = true;
    for (int rt = rt0; rt < ntr && ok && !failed; rt += rstep, ++i) {
      const int b = i & 1;
      if (i >= 2 && !mbar_wait(&acce[b], ((i >> 1) - 1) & 1, OZK_POLLS)) {
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tb = tmem + (uint32_t)(b * 256);
      for (int k = 0; k < nkb; ++k) {
        const int st = q % nst;
        if (!mbar_wait(&wbar[k], 0, OZK_POLLS) || !mbar_wait(&full[st], (q / nst) & 1, OZK_POLLS)) {
          failed = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t xa = smem_u32(sx + st * XB);
        const uint32_t wa = smem_u32(sw + k * WB);
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          if (2 * k + ks >= nks) break;
          ozk_issue_kstep<S, CN, BF>(tb, xa, wa, ks, k == 0 && ks == 0);
        }
        umma_commit(&empty[st]);
        ++q;
      }
      if (!ok) break;
      umma_commit(&accf[b]);  // arrives once the tile's products have completed
    }
    consumed_q = q;
    umma_commit(&done);
  } else if (warp >= 4) {
    // epilogue
    const int wq = warp & 3, half = (warp - 4) >> 2;
    const int nc = min(CN, cout - c0);  // columns of the tile
    const bool vec = sizeof(T) == 8 && (ldd & 3) == 0 && (reinterpret_cast<uintptr_t>(D) & 31) == 0;
    int i = 0;
    for (int rt = rt0; rt < ntr; rt += rstep, ++i) {
      const int b = i & 1;
      const int row = rt * OZK_BM + wq * 32 + lane;
      const double xs = row < rows ? pow2i(ex[row]) : 0.0;
      const bool got = mbar_wait(&accf[b], (i >> 1) & 1, OZK_POLLS);
      if (!__all_sync(0xffffffffu, got ? 1 : 0) || failed) {
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tl = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(b * 256);
#pragma unroll 1
      for (int cc = half * 16; cc < nc; cc += 32) {
        uint32_t v[S][16];
#pragma unroll
        for (int g = 0; g < S; ++g) tmem_ld16(tl + g * CN + cc, v[g]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        double o[16];
#pragma unroll
        for (int q2 = 0; q2 < 16; ++q2) {
          // the digit groups as one 64-bit integer (see ozk_gemm_kernel)
          long long h = 0;
#pragma unroll
          for (int g = 0; g < S; ++g) h = (h << 7) + (long long)(BF ? (int)__uint_as_float(v[g][q2]) : (int)v[g][q2]);
          o[q2] = (((double)h * pow2i(-7 * (S + 1))) * xs) * s_sw[cc + q2];
        }
        if (row < rows) {
          T* drow = D + (long)row * ldd + c0 + cc;
          if constexpr (sizeof(T) == 8) {
            if (vec) {
#pragma unroll
              for (int q4 = 0; q4 < 16; q4 += 4)
                if (cc + q4 + 3 < nc) {
                  st_v4(drow + q4, o[q4], o[q4 + 1], o[q4 + 2], o[q4 + 3]);
                } else {
#pragma unroll
                  for (int q2 = q4; q2 < q4 + 4; ++q2)
                    if (cc + q2 < nc) drow[q2] = o[q2];
                }
              continue;
            }
          }
#pragma unroll
          for (int q2 = 0; q2 < 16; ++q2)
            if (cc + q2 < nc) drow[q2] = (T)o[q2];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_expect_tx(&acce[b], 0);  // this warp's arrival: the buffer's lanes are read
    }
  }
  __syncthreads();
  if (warp == 0 && lane == 0) {
    // copies issued but never consumed (only after a wait ran out)
    for (int q = consumed_q; q < issued_q; ++q) mbar_wait(&full[q % nst], (q / nst) & 1, OZK_POLLS);
    for (int k = 0; k < issued_w; ++k) mbar_wait(&wbar[k], 0, OZK_POLLS);
  }
  const bool okd = __syncthreads_and(mbar_wait(&done, 0, OZK_POLLS) ? 1 : 0) && !failed;
  if (!okd && threadIdx.x == 0 && status) {
    for (int rt = rt0; rt < ntr; rt += rstep) {
      const int m0 = rt * OZK_BM, r1 = min(m0 + OZK_BM, rows) - 1;
      for (int qq = m0 / rows_per_status; qq <= r1 / rows_per_status; ++qq) atomicOr(status + qq, bit);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// digits of one row per warp, the row held in registers (Kp <= 32 NT): lane l
// takes positions 32 c + l, so the loads are coalesced whatever the row's
// alignment and the digits of a plane leave as whole 32-byte sectors (64-byte
// in bf16).  The row's exponent is the largest exponent field in it (an
// integer maximum); a row with no normal value, or with an infinity or NaN,
// takes it from the largest magnitude.  A digit is rint(t) by adding and
// taking off 1.5 2^52 (round to nearest even; the integer stands in the sum's
// low word), so no conversion instruction is needed.
template <typename Tin, int BF, int NT>
__global__ void __launch_bounds__(256) ozk_split_kernel(const Tin* __restrict__ X, long ldx, int rows, int K, int Kp,
                                                        int S, unsigned char* __restrict__ dig, long plane,
                                                        int* __restrict__ expo) {
  chain_enter();
  const int row = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const Tin* x = X + (long)row * ldx + lane;
  double t[NT];
  int em = 0;
#pragma unroll
  for (int c = 0; c < NT; ++c) {
    t[c] = 32 * c + lane < K ? (double)x[32 * c] : 0.0;
    em = max(em, __double2hiint(t[c]) & 0x7ff00000);
  }
  em = __reduce_max_sync(0xffffffffu, em) >> 20;
  int e = em - 1023 + 2;
  if (em == 0 || em == 0x7ff) {
    double m = 0.0;
#pragma unroll
    for (int c = 0; c < NT; ++c) m = fmax(m, fabs(t[c]));
    m = warp_max(m);
    e = m > 0.0 ? ilogb(m) + 2 : 0;
  }
  if (lane == 0) expo[row] = e;
  const bool fits = 7 - e >= -1022 && 7 - e <= 1023;  // 2^(7 - e) is a normal number
  const double sc = fits ? __longlong_as_double((long long)(7 - e + 1023) << 52) : 1.0;
  constexpr double kRint = 6755399441055744.0;  // 1.5 2^52
  const long at = (long)row * Kp + lane;
#pragma unroll
  for (int c = 0; c < NT; ++c) {
    if (32 * c + lane >= Kp) break;
    double v = fits ? t[c] * sc : ldexp(t[c], 7 - e);
    for (int i = 0; i < S; ++i) {
      const double s = __dadd_rn(v, kRint);
      const int d = __double2loint(s);
      v = __dmul_rn(__dsub_rn(v, __dsub_rn(s, kRint)), 128.0);
      if (BF)
        reinterpret_cast<uint16_t*>(dig)[(long)i * plane + at + 32 * c] =
            (uint16_t)(__float_as_uint((float)d) >> 16);  // exact for |d| <= 256
      else
        dig[(long)i * plane + at + 32 * c] = (unsigned char)d;
    }
  }
}

template <int S, typename T, int PAIR, int BF>
int prepare_one() {
  // the shared-memory limit is a per-device function attribute
  static unsigned long long attr_set = 0;
  int dev = 0;
  SCY_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !(attr_set >> dev & 1ull)) {
    SCY_CUDA_TRY(cudaFuncSetAttribute(ozk_gemm_kernel<S, T, PAIR, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      ozk_smem_bytes(S, PAIR)));
    if (dev >= 0 && dev < 64) attr_set |= 1ull << dev;
  }
  return SCY_OK;
}

template <int S, typename T, int BF>
int prepare_pers() {
  static unsigned long long attr_set = 0;
  int dev = 0;
  SCY_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !(attr_set >> dev & 1ull)) {
    SCY_CUDA_TRY(cudaFuncSetAttribute(ozk_gemm_pers_kernel<S, T, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      227 * 1024 - 1024));
    if (dev >= 0 && dev < 64) attr_set |= 1ull << dev;
  }
  return SCY_OK;
}

template <int S, int BF>
int prepare_sb() {
  int rc = prepare_one<S, double, 0, BF>();
  if (rc == SCY_OK) rc = prepare_one<S, float, 0, BF>();
  if constexpr (S <= 5) {
    if (rc == SCY_OK) rc = prepare_one<S, double, 1, BF>();
    if (rc == SCY_OK) rc = prepare_one<S, float, 1, BF>();
    if (rc == SCY_OK) rc = prepare_pers<S, double, BF>();
    if (rc == SCY_OK) rc = prepare_pers<S, float, BF>();
  }
  if constexpr (BF == 0) {
    if (rc == SCY_OK) rc = prepare_one<S, double, 2, 0>();
    if (rc == SCY_OK) rc = prepare_one<S, float, 2, 0>();
  }
  return rc;
}

// multiprocessors of the current device (cached per device)
int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kNumSMs;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = kNumSMs;
    cached[dev] = n;
  }
  return cached[dev];
}

template <int S>
int prepare_s() {
  const int rc = prepare_sb<S, 0>();
  return rc != SCY_OK ? rc : prepare_sb<S, 1>();
}

template <int S, typename T, int PAIR, int BF>
int launch_gemm(const OzkOperand& x, const CUtensorMap& wmap, const OzkOperand& w, T* D, long ldd, int cout,
                cudaStream_t s, unsigned* status, int rows_per_status, unsigned bit) {
  constexpr int CN = ozk_cn(S, PAIR);
  {
    const int rc = prepare_one<S, T, PAIR, BF>();
    if (rc != SCY_OK) return rc;
  }
  const dim3 grid((cout + CN - 1) / CN, (x.rows + OZK_BM - 1) / OZK_BM);
  launch(x.chain, ozk_gemm_kernel<S, T, PAIR, BF>, grid, ozk_threads(PAIR), ozk_smem_bytes(S, PAIR), s, x.map, wmap,
         x.expo.as<int>(), w.expo.as<int>(), D, ldd, x.rows, cout, x.Kp * x.esz / 32, status, rows_per_status, bit);
  SCY_LAUNCH_CHECK();
  return SCY_OK;
}

// the persistent shape: one CTA per SM (at most one per tile); *used = 0
// where the weights' tile does not fit beside two stages
template <int S, typename T, int BF>
int launch_pers(const OzkOperand& x, const OzkOperand& w, T* D, long ldd, int cout, cudaStream_t s,
                unsigned* status, int rows_per_status, unsigned bit, int* used) {
  constexpr int CN = ozk_cn(S, 1);
  const int nks = x.Kp * x.esz / 32, nkb = (nks + 1) / 2, nst = ozk_pers_stages(S, nkb);
  *used = nst > 0;
  if (!nst) return SCY_OK;
  SCY_TRY((prepare_pers<S, T, BF>()));
  const long ntiles = (long)((cout + CN - 1) / CN) * ((x.rows + OZK_BM - 1) / OZK_BM);
  const int grid = (int)std::min<long>(ntiles, sm_count());
  const int smem = nkb * ozk_pers_w_bytes(S) + nst * ozk_pers_x_bytes(S) + 1024;
  launch(x.chain, ozk_gemm_pers_kernel<S, T, BF>, grid, 384, smem, s, x.map, w.map_pair, x.expo.as<int>(),
         w.expo.as<int>(), D, ldd, x.rows, cout, nks, nst, status, rows_per_status, bit);
  SCY_LAUNCH_CHECK();
  return SCY_OK;
}

template <int S, typename T, int BF>
int launch_variant_b(const OzkOperand& x, const OzkOperand& w, T* D, long ldd, int cout, cudaStream_t s,
                     unsigned* status, int rps, unsigned bit, int pair) {
  if constexpr (S <= 5) {
    if (pair == 2) {
      int used = 0;
      SCY_TRY((launch_pers<S, T, BF>(x, w, D, ldd, cout, s, status, rps, bit, &used)));
      if (used) return SCY_OK;
    }
    if (pair == 1 || pair == 2) return launch_gemm<S, T, 1, BF>(x, w.map_pair, w, D, ldd, cout, s, status, rps, bit);
  }
  if constexpr (BF == 0) {
    if (pair == 3) return launch_gemm<S, T, 2, 0>(x, w.map_narrow, w, D, ldd, cout, s, status, rps, bit);
  }
  return launch_gemm<S, T, 0, BF>(x, w.map, w, D, ldd, cout, s, status, rps, bit);
}

template <int S, typename T>
int launch_variant(const OzkOperand& x, const OzkOperand& w, T* D, long ldd, int cout, cudaStream_t s,
                   unsigned* status, int rps, unsigned bit, int pair) {
  if (x.esz == 2) return launch_variant_b<S, T, 1>(x, w, D, ldd, cout, s, status, rps, bit, pair);
  return launch_variant_b<S, T, 0>(x, w, D, ldd, cout, s, status, rps, bit, pair);
}

template <typename T>
int gemm_any(const OzkOperand& x, const OzkOperand& w, T* D, long ldd, int cout, cudaStream_t s, unsigned* status,
             int rps, unsigned bit, int pair) {
  if (x.S != w.S || x.Kp != w.Kp || x.K != w.K || x.esz != w.esz || cout > w.rows || cout < 1 || x.rows < 1 ||
      w.box_rows != ozk_cn(w.S) || x.box_rows != OZK_BM || rps < 1 || pair < 0 || pair > 3 ||
      ((pair == 1 || pair == 2) && (w.S > 5 || w.box_rows_pair != ozk_cn(w.S, 1))) ||
      (pair == 3 && (w.box_rows_narrow != OZK_NARROW || w.esz != 1))) {
    set_error("ozk_gemm: operands do not match (S %d/%d, K %d/%d, cout %d, W rows %d, shape %d)", x.S,
              w.S, x.K, w.K, cout, w.rows, pair);
    return SCY_ERR_ARG;
  }
  switch (x.S) {
    case 3: return launch_variant<3, T>(x, w, D, ldd, cout, s, status, rps, bit, pair);
    case 4: return launch_variant<4, T>(x, w, D, ldd, cout, s, status, rps, bit, pair);
    case 5: return launch_variant<5, T>(x, w, D, ldd, cout, s, status, rps, bit, pair);
    case 6: return launch_variant<6, T>(x, w, D, ldd, cout, s, status, rps, bit, pair);
    case 7: return launch_variant<7, T>(x, w, D, ldd, cout, s, status, rps, bit, pair);
    default: break;
  }
  set_error("ozk_gemm: %d digit planes (3 to 7 are built)", x.S);
  return SCY_ERR_ARG;
}

}  // namespace

int ozk_cols_per_tile(int S) { return ozk_cn(S); }
int ozk_cols_per_tile_pair(int S) { return S <= 5 ? ozk_cn(S, 1) : 0; }

int ozk_prepare(int S) {
  switch (S) {
    case 3: return prepare_s<3>();
    case 4: return prepare_s<4>();
    case 5: return prepare_s<5>();
    case 6: return prepare_s<6>();
    case 7: return prepare_s<7>();
    default: break;
  }
  set_error("ozk_prepare: %d digit planes (3 to 7 are built)", S);
  return SCY_ERR_ARG;
}

int OzkOperand::alloc_weights(int S_, int rows_, int K_, int esz_) {
  SCY_TRY(alloc(S_, rows_, K_, ozk_cols_per_tile(S_), esz_));
  box_rows_pair = ozk_cols_per_tile_pair(S_);
  if (box_rows_pair > 0 &&
      tma_map_3d_sw64(&map_pair, dig.p, esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8,
                      Kp, rows, S, Kp * esz, plane * esz, OZK_BK / esz, box_rows_pair, S) != SCY_OK)
    return SCY_ERR_CUDA;
  if (esz == 1) {
    box_rows_narrow = OZK_NARROW;
    if (tma_map_3d_sw64(&map_narrow, dig.p, CU_TENSOR_MAP_DATA_TYPE_UINT8, Kp, rows, S, Kp, plane, OZK_BK,
                        box_rows_narrow, S) != SCY_OK)
      return SCY_ERR_CUDA;
  }
  return SCY_OK;
}

bool ozk_narrow_better(int S, int rows, int cols) {
  const long wide = (long)((cols + ozk_cn(S) - 1) / ozk_cn(S)) * ((rows + OZK_BM - 1) / OZK_BM);
  return 2 * wide <= kNumSMs;
}

bool ozk_bf16_exact(int S, int K) {
  const long Kp = (K + 15) / 16 * 16;
  return (long)S * 64 * 64 * Kp < (1L << 24);
}

int OzkOperand::alloc(int S_, int rows_, int K_, int box_rows_, int esz_) {
  if (S_ < 3 || S_ > 7 || rows_ < 1 || K_ < 1 || K_ > 1024 || box_rows_ < 8 || box_rows_ > 256 ||
      (esz_ != 1 && esz_ != 2) || (esz_ == 2 && !ozk_bf16_exact(S_, K_))) {
    set_error("OzkOperand: invalid shape (S %d, rows %d, K %d, box rows %d, digit bytes %d)", S_, rows_, K_,
              box_rows_, esz_);
    return SCY_ERR_ARG;
  }
  S = S_;
  rows = rows_;
  K = K_;
  esz = esz_;
  const int kq = OZK_BK / esz;  // digits per 64-byte stage row (the TMA box; zero-filled past Kp)
  const int ke = 32 / esz;      // digits per MMA K step
  Kp = (K + ke - 1) / ke * ke;
  box_rows = box_rows_;
  plane = (long)rows * Kp;
  SCY_TRY(dig.alloc((size_t)S * plane * esz));
  SCY_TRY(expo.alloc((size_t)rows * sizeof(int)));
  // zero once: the K padding of every row stays zero
  SCY_CUDA_TRY(cudaMemset(dig.p, 0, (size_t)S * plane * esz));
  SCY_CUDA_TRY(cudaMemset(expo.p, 0, (size_t)rows * sizeof(int)));
  if (tma_map_3d_sw64(&map, dig.p, esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, Kp,
                      rows, S, Kp * esz, plane * esz, kq, box_rows, S) != SCY_OK)
    return SCY_ERR_CUDA;
  return SCY_OK;
}

template <typename Tin, int BF>
static void launch_split(OzkOperand& o, const Tin* X, long ldx, cudaStream_t s) {
  const int blocks = (int)(((long)o.rows * 32 + 255) / 256);
  unsigned char* d = o.dig.as<unsigned char>();
  int* ex = o.expo.as<int>();
  if (o.Kp <= 128)
    launch(o.chain, ozk_split_kernel<Tin, BF, 4>, blocks, 256, 0, s, X, ldx, o.rows, o.K, o.Kp, o.S, d, o.plane, ex);
  else if (o.Kp <= 256)
    launch(o.chain, ozk_split_kernel<Tin, BF, 8>, blocks, 256, 0, s, X, ldx, o.rows, o.K, o.Kp, o.S, d, o.plane, ex);
  else if (o.Kp <= 512)
    launch(o.chain, ozk_split_kernel<Tin, BF, 16>, blocks, 256, 0, s, X, ldx, o.rows, o.K, o.Kp, o.S, d, o.plane, ex);
  else
    launch(o.chain, ozk_split_kernel<Tin, BF, 32>, blocks, 256, 0, s, X, ldx, o.rows, o.K, o.Kp, o.S, d, o.plane, ex);
}

template <typename Tin>
static int split_any(OzkOperand& o, const Tin* X, long ldx, cudaStream_t s) {
  // K <= 1024 (OzkOperand::alloc)
  if (o.esz == 2)
    launch_split<Tin, 1>(o, X, ldx, s);
  else
    launch_split<Tin, 0>(o, X, ldx, s);
  SCY_LAUNCH_CHECK();
  return SCY_OK;
}

int ozk_split(OzkOperand& o, const double* X, long ldx, cudaStream_t s) { return split_any(o, X, ldx, s); }
int ozk_split(OzkOperand& o, const float* X, long ldx, cudaStream_t s) { return split_any(o, X, ldx, s); }

int ozk_set_host(OzkOperand& o, const double* W, long ldw, cudaStream_t s) {
  std::vector<int8_t> dig((size_t)o.S * o.plane, 0);
  std::vector<uint16_t> dig2(o.esz == 2 ? (size_t)o.S * o.plane : 0, 0);
  std::vector<int> ex(o.rows, 0);
  for (int r = 0; r < o.rows; ++r) {
    const double* x = W + (long)r * ldw;
    double m = 0.0;
    for (int k = 0; k < o.K; ++k) m = std::fmax(m, std::fabs(x[k]));
    const int e = m > 0.0 ? std::ilogb(m) + 2 : 0;
    ex[r] = e;
    for (int k = 0; k < o.K; ++k) {
      double t = std::ldexp(x[k], 7 - e);
      for (int i = 0; i < o.S; ++i) {
        const double d = std::nearbyint(t);
        t = (t - d) * 128.0;
        const size_t at = (size_t)i * o.plane + (size_t)r * o.Kp + k;
        if (o.esz == 2) {
          // bf16 pattern of the integer digit: the upper half of its FP32 pattern
          const float f = (float)d;
          uint32_t u;
          std::memcpy(&u, &f, 4);
          dig2[at] = (uint16_t)(u >> 16);
        } else {
          dig[at] = (int8_t)(int)d;
        }
      }
    }
  }
  if (o.esz == 2)
    SCY_CUDA_TRY(cudaMemcpyAsync(o.dig.p, dig2.data(), dig2.size() * 2, cudaMemcpyHostToDevice, s));
  else
    SCY_CUDA_TRY(cudaMemcpyAsync(o.dig.p, dig.data(), dig.size(), cudaMemcpyHostToDevice, s));
  SCY_CUDA_TRY(cudaMemcpyAsync(o.expo.p, ex.data(), ex.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  SCY_CUDA_TRY(cudaStreamSynchronize(s));
  return SCY_OK;
}

int ozk_gemm(const OzkOperand& x, const OzkOperand& w, double* D, long ldd, int cout, cudaStream_t s,
             unsigned* status, int rows_per_status, unsigned bit, int pair) {
  return gemm_any<double>(x, w, D, ldd, cout, s, status, rows_per_status, bit, pair);
}

int ozk_gemm(const OzkOperand& x, const OzkOperand& w, float* D, long ldd, int cout, cudaStream_t s,
             unsigned* status, int rows_per_status, unsigned bit, int pair) {
  return gemm_any<float>(x, w, D, ldd, cout, s, status, rows_per_status, bit, pair);
}

}  // namespace scy

// ---------------------------------------------------------------------------
// C ABI: the product on its own (set-up and digit planes allocated per call)
extern "C" scy_status scy_ozaki_matmul(const double* X, long ldx, int rows, int K, const double* W, long ldw,
                                       int cols, int S, double* D, long ldd, int ctas_per_sm, int bf16_digits) {
  using namespace scy;
  if (!X || !W || !D || rows < 1 || cols < 1 || K < 1 || ldx < K || ldw < K || ldd < cols ||
      (ctas_per_sm < 0 || ctas_per_sm > 2) || (ctas_per_sm != 1 && S > 5) ||
      (bf16_digits && !ozk_bf16_exact(S, K))) {
    set_error("scy_ozaki_matmul: invalid arguments");
    return SCY_ERR_ARG;
  }
  const int esz = bf16_digits ? 2 : 1;
  OzkOperand x, w;
  SCY_TRY(x.alloc(S, rows, K, 128, esz));
  SCY_TRY(w.alloc_weights(S, cols, K, esz));
  cudaStream_t s = 0;
  SCY_TRY(ozk_set_host(w, W, ldw, s));
  SCY_TRY(ozk_split(x, X, ldx, s));
  DevBuf status;
  SCY_TRY(status.alloc(sizeof(unsigned)));
  SCY_CUDA_TRY(cudaMemsetAsync(status.p, 0, sizeof(unsigned), s));
  SCY_TRY(ozk_gemm(x, w, D, ldd, cols, s, status.as<unsigned>(), 1 << 30, 1u,
                   ctas_per_sm == 2 ? 1 : ctas_per_sm == 0 ? 2 : 0));
  unsigned st = 0;
  SCY_CUDA_TRY(cudaMemcpyAsync(&st, status.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  SCY_CUDA_TRY(cudaStreamSynchronize(s));
  if (st) {
    set_error("scy_ozaki_matmul: a pipeline wait in the product kernel ran out");
    return SCY_ERR_CUDA;
  }
  return SCY_OK;
}
