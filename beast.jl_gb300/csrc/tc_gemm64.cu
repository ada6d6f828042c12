// tc_gemm64.cu -- the trailing updates of the complex FP64 LU on the FP16 tensor cores.
//
//   C -= A B   with C (M x N), A (M x K), B (K x N) complex128, column-major
//
// GB300 runs FP64 at 1/1500 of its FP16 tensor rate (measured: the shared-memory tiled FP64 kernel
// this replaces ran at 0.69 TFLOP/s, 90% of an FP64 solve of order 6007).  Each operand row /
// column is therefore written in 7-bit digits of a fixed-point number (slice64.h; Ozaki et
// al., Numer. Algorithms 59 (2012), with the tensor-core form of Mukunoki et al., ISC 2020) and
// the product summed digit by digit, eight of the nine digits unless a block asks for the last:
//   C' = sum_l 2^(-12 - 7 l) D_l,   D_l = sum_{i + j = l} A'_i B'_j,   l = 0 .. 7
// on the real 2x2 form of the complex product (the layout of tc_gemm.cu: A' has rows 2m, 2m+1
// = [[re, -im], [im, re]], B' columns hold (re, im) per k).  D_l is a sum of at most (l + 1) 2K
// products of magnitude at most 2^12: with K <= 256 an integer of at most 2^24, exact in the FP32
// accumulators.  What is dropped (digits beyond 2^-56 of the row's and the column's largest
// magnitude, pairs i + j > 7) is small against those two magnitudes, not against every entry's own sum.
// Two things keep it below an FP64 sum's own rounding (slice64.h):
//   - the columns of A are levelled by powers of two and the rows of B by their inverses before the
//     digits are taken (k_balance): rows of a matrix in different units lose nothing.  Without it an
//     order-300 system with half its rows scaled by 1e-8 came out with an error of 1e-9 (1e-15 with);
//   - the product S of the entries' magnitudes is taken first.  Where a sum and its entry of C are both below 2^-10
//     of the row's and the column's scale, the block of 64 columns takes the ninth digit (nine more pairs), and below
//     2^-17 it goes to the FP64 units, 64 x 64 at a time (gemm64_tiles).  Hardly any block does in EFIE and Helmholtz
//     matrices of real wavenumbers, a few hundredths take the ninth digit in second-kind ones of flat surfaces, a tenth
//     under a kernel that decays by e^6 over the surface; under one that decays by e^40 half the work is the FP64
//     units' and a solve takes as long as on those alone at worst.
// measured against LAPACK's solutions in tests/test_gpu_lu_paths.py.
//
// k_tc_gemm64: persistent CTAs over 128 x TNT tiles of C'; after S the levels run from the smallest
// contribution (l = 7) to the largest (and l = 8 where it is asked for), each as one K loop over its l + 1 digit pairs through the
// 4-stage TMA ring into one of two TMEM accumulators, while four epilogue warps add the previous
// level to C (one FP64 addition per value: -D 2^sh is built from the bits of D).  A tile's C
// values belong to one CTA and are added to in a fixed order: the result is deterministic.
//   measured (one GB300): M = N = 5000, K = 1024 in 9.13 ms (8.80 without the magnitudes and the ninth digit), 22.4
//   TFLOP/s of FP64 products (808 TFLOP/s of FP16 ones) where the FP64 units gave 0.69; against sums in 128 bits the
//   update's error is 2.0e-16 .. 3.5e-16 on random operands (FP64 sums: 3.8e-16 .. 1.1e-15).  The order-6007 solve's
//   updates: 827 -> 50 ms.
//   bound: the tensor pipe at large M, N (36 digit pairs: 72 K MACs per real value of C against
//   8 FP64 additions, which take 0.85 of the time of the MMAs at K = 256); the FP64 additions at
//   K = 64.
//   TNT = 256 when its tiles fill the SMs; 64 below (the last blocks of a factorisation and small
//   matrices): four times the CTAs share the additions and the digit loops.
#include <algorithm>

#include "internal.h"
#include "slice64.h"
#include "tc_ptx.h"

// the listed 64 x 64 blocks of the update on the FP64 units (linalg.cu)
cudaError_t gemm64_tiles(const int2* list, const int* count, double2* C, int64_t ldc, const double2* A, int64_t lda,
                         const double2* B, int64_t ldb, int64_t m, int64_t n, int k, int grid, cudaStream_t st);

namespace {

using slice64::SLICES;
constexpr int PLANES = SLICES + 1;  // digits held of each operand

constexpr int TM = 128, TK = 64, STAGES = 4;
constexpr int KMAX = 256;  // complex columns of A per launch: (l + 1) 2K 2^12 <= 2^24 for l = 7
constexpr int A_BYTES = TM * TK * 2;
// the accumulations of a tile, in order: the magnitudes, levels 7 .. 0, and level 8 in two (nine pairs would not be
// exact in one) where a block asks for it
constexpr int STEPS = SLICES + 1, NINE_A = 5;
struct Step {
  int level, i0, i1;  // pairs (i, level - i) for i0 <= i < i1
};
__device__ __forceinline__ Step step_at(int st) {
  const int l = SLICES - st;  // 0: the magnitudes
  if (st == 0) return Step{0, 0, 1};
  if (st < STEPS) return Step{l, 0, l + 1};
  return st == STEPS ? Step{SLICES, 0, NINE_A} : Step{SLICES, NINE_A, PLANES};
}
constexpr int GROUP = 8;  // row tiles taken together, column by column

template <int TNT>
struct Tile {
  static constexpr int B_BYTES = TNT * TK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;
};

// tile index -> first real row and first column: groups of GROUP row tiles, column by column
__device__ __forceinline__ void tile_at(int tile, int ntm, int ntn, int& mt, int& nt) {
  const int per = GROUP * ntn, g = tile / per, l = tile - g * per;
  const int rows = min(GROUP, ntm - g * GROUP);
  mt = g * GROUP + l % rows;
  nt = l / rows;
}

// M2 = 2M real rows of C' at Cr (ldr doubles per column), N columns; A' slice i at rows i M2, B'
// slice j at rows j N of their tensor maps; nk stages of TK halves per digit pair.  tmP, tmQ: the magnitudes of A (a
// row per complex row) and B, nkS stages.  Blocks left to the FP64
// units: their (row, column) indices in units of 64 in list, their number in count
template <int TNT>
__global__ void __launch_bounds__(192, 1)
    k_tc_gemm64(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmQ, double* Cr, int64_t ldr,
                int M2, int N, const int* __restrict__ ea, const int* __restrict__ eb, int nk, int nkS, int2* list,
                int* count, int* status) {
  constexpr int STAGE_BYTES = Tile<TNT>::STAGE_BYTES;
  extern __shared__ unsigned char smraw[];
  const uint32_t base = (smem_u32(smraw) + 1023u) & ~1023u;
  unsigned char* gbase = smraw + (base - smem_u32(smraw));
  // full[STAGES], empty[STAGES], tfull[2], tempty[2], done, spread
  uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + STAGES * STAGE_BYTES);
  const int B_FULL = 0, B_EMPTY = STAGES, B_TFULL = 2 * STAGES, B_TEMPTY = 2 * STAGES + 2, B_DONE = 2 * STAGES + 4,
            B_SPREAD = 2 * STAGES + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 7);
  __shared__ int s_abort_mem, s_wide_mem[2][4];
  // by parity of a CTA's tiles, per epilogue warp: groups of 64 columns left to the FP64 units (bits 0 .. 3) and with the
  // ninth digit (bits 4 .. 7)
  volatile int(*s_wide)[4] = s_wide_mem;
  volatile int* s_abort = &s_abort_mem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntm = (M2 + TM - 1) / TM, ntn = (N + TNT - 1) / TNT, ntiles = ntm * ntn;

  if (threadIdx.x == 0) {
    *s_abort = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(bars + B_FULL + s), 1);
      mbar_init(smem_u32(bars + B_EMPTY + s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(bars + B_TFULL + a), 1);
      mbar_init(smem_u32(bars + B_TEMPTY + a), 4);  // one arrival per epilogue warp
    }
    mbar_init(smem_u32(bars + B_DONE), 1);
    mbar_init(smem_u32(bars + B_SPREAD), 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * TNT)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // true when tile number ord of this CTA asks for the ninth digit (known once its magnitudes are read); false at once
  // when a wait has given up
  auto nine = [&](int ord) {
    if (!mbar_wait(smem_u32(bars + B_SPREAD), ord & 1, status, s_abort)) return false;
    volatile int* w = s_wide[ord & 1];
    return ((w[0] | w[1] | w[2] | w[3]) >> 4) != 0;
  };

  if (warp == 0 && lane == 0) {
    // ---- TMA producer
    uint32_t it = 0;
    int ord = 0;
    for (int tile = blockIdx.x; tile < ntiles && !*s_abort; tile += gridDim.x, ++ord) {
      int mt, nt;
      tile_at(tile, ntm, ntn, mt, nt);
      for (int st = 0; st < STEPS + 2 && !*s_abort; ++st) {
        if (st == STEPS && !nine(ord)) break;
        const Step p = step_at(st);
        for (int i = p.i0; i < p.i1 && !*s_abort; ++i)
          for (int kb = 0; kb < (st == 0 ? nkS : nk); ++kb, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(smem_u32(bars + B_EMPTY + s), ((it / STAGES) & 1) ^ 1, status, s_abort)) break;
            const uint32_t sa = base + s * STAGE_BYTES, full = smem_u32(bars + B_FULL + s);
            mbar_expect_tx(full, STAGE_BYTES);
            if (st == 0) {
              tma_load_2d(sa, &tmP, kb * TK, mt * (TM / 2), full);
              tma_load_2d(sa + A_BYTES, &tmQ, kb * TK, nt * TNT, full);
            } else {
              tma_load_2d(sa, &tmA, kb * TK, i * M2 + mt * TM, full);
              tma_load_2d(sa + A_BYTES, &tmB, kb * TK, (p.level - i) * N + nt * TNT, full);
            }
          }
      }
    }
    // no copy may still be landing in shared memory when the CTA exits (bounded, whatever the
    // abort state)
    int no_abort = 0;
    for (uint32_t j = it > (uint32_t)STAGES ? it - STAGES : 0; j < it; ++j)
      mbar_wait(smem_u32(bars + B_FULL + j % STAGES), (j / STAGES) & 1, status, &no_abort);
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer: D f32, A / B f16, both K-major, M = 128, N = TNT
    const uint32_t idesc = (1u << 4) | ((uint32_t)(TNT >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    uint32_t it = 0;
    int t = 0, ord = 0;  // accumulations of all tiles, in order
    for (int tile = blockIdx.x; tile < ntiles && !*s_abort; tile += gridDim.x, ++ord)
      for (int st = 0; st < STEPS + 2 && !*s_abort; ++st, ++t) {
        if (st == STEPS && !nine(ord)) break;
        const Step p = step_at(st);
        const int a = t & 1;
        if (!mbar_wait(smem_u32(bars + B_TEMPTY + a), ((t >> 1) & 1) ^ 1, status, s_abort)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + (uint32_t)(a * TNT);
        const int steps = st == 0 ? nkS : (p.i1 - p.i0) * nk;
        for (int kb = 0; kb < steps; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(smem_u32(bars + B_FULL + s), (it / STAGES) & 1, status, s_abort)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
#pragma unroll
          for (int kk = 0; kk < TK / 16; ++kk)
            mma_f16(acc, smem_desc(sa + kk * 32), smem_desc(sb + kk * 32), idesc, (kb | kk) ? 1u : 0u);
          mma_commit(smem_u32(bars + B_EMPTY + s));
        }
        if (*s_abort) break;
        mma_commit(smem_u32(bars + B_TFULL + a));
      }
    // every MMA issued above has completed once this phase does (waited for even after an abort)
    mma_commit(smem_u32(bars + B_DONE));
    int no_abort = 0;
    mbar_wait(smem_u32(bars + B_DONE), 0, status, &no_abort);
  } else if (warp >= 2) {
    // ---- epilogue: warp w owns TMEM lanes 32 (w % 4) .. +31, a thread one real row of the tile
    const int q = warp & 3;
    int t = 0, ord = 0;
    bool live = true;
    for (int tile = blockIdx.x; tile < ntiles && live; tile += gridDim.x, ++ord) {
      int mt, nt;
      tile_at(tile, ntm, ntn, mt, nt);
      const int row = mt * TM + q * 32 + lane, n0 = nt * TNT;
      const bool in = row < M2;
      const int er = in ? ea[row >> 1] : 0;
      double* c0 = Cr + row + (int64_t)n0 * ldr;
      const int ncol = min(TNT, N - n0);
      int wide = 0;  // as s_wide, of all four warps
      for (int st = 0; st < (wide >> 4 ? STEPS + 2 : STEPS); ++st, ++t) {
        const int a = t & 1;
        if (!mbar_wait(smem_u32(bars + B_TFULL + a), (t >> 1) & 1, status, s_abort)) {
          live = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * TNT);
        auto release = [&]() {  // accumulator read: hand it back to the MMA warp
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bars + B_TEMPTY + a)) : "memory");
        };
        if (st == 0) {
          // small sums whose entry of C is small too, a thread a complex row (the first two warps; the accumulator's
          // other rows are the next tile's)
          const int cr = mt * (TM / 2) + q * 32 + lane;
          const bool inc = q < 2 && 2 * cr < M2;
          const int ec = inc ? ea[cr] : 0;
          const double* cz = Cr + 2 * (int64_t)cr + (int64_t)n0 * ldr;
          int found = 0;
          for (int c = 0; c < ncol && q < 2; c += 16) {
            float v[16];
            tmem_ld16(tb + (uint32_t)c, v);
            uint32_t low = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              low |= (uint32_t)(v[j] > 0.f && v[j] < 1.f / (1 << slice64::SPREAD_BITS)) << j;
            const int g = c >> 6;
            if (!inc) low = 0;
            for (; low && !((found >> g) & 1); low &= low - 1) {
              const int jj = __ffs(low) - 1, j = c + jj;
              if (j >= ncol) break;
              const double x = cz[j * ldr], y = cz[j * ldr + 1];
              const int e = ec + eb[n0 + j];
              float s = 0.f;
#pragma unroll
              for (int u = 0; u < 16; ++u) s = u == jj ? v[u] : s;
              if (!slice64::spread_small(x, y, e, slice64::SPREAD_BITS)) continue;
              found |= 16 << g;
              if (s < 1.f / (1 << slice64::SPREAD_BITS_FP64) && slice64::spread_small(x, y, e, slice64::SPREAD_BITS_FP64))
                found |= 1 << g;
            }
            __syncwarp();  // (the accumulator is read by the whole warp)
          }
          release();
          // the four warps agree
          found = (int)__reduce_or_sync(0xffffffffu, (unsigned)found);
          if (lane == 0) {
            s_wide[ord & 1][q] = found & ~((found & 15) << 4);
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bars + B_SPREAD)) : "memory");
          }
          if (!mbar_wait(smem_u32(bars + B_SPREAD), ord & 1, status, s_abort)) {
            live = false;
            break;
          }
          wide = s_wide[ord & 1][0] | s_wide[ord & 1][1] | s_wide[ord & 1][2] | s_wide[ord & 1][3];
          if (q == 0 && lane == 0)
            for (int g = 0; g < TNT / 64; ++g)
              if ((wide >> g) & 1) list[atomicAdd(count, 1)] = make_int2(mt, nt * (TNT / 64) + g);
          continue;
        }
        // columns of this accumulation: level 8 those with the ninth digit, none of the FP64 units' any
        const int skip = (wide & 15) | (st >= STEPS ? ~(wide >> 4) & 15 : 0);
        const int l = step_at(st).level;
        const int sh0 = er - 12 - 7 * l;
        for (int c = 0; c < ncol; c += 16) {
          if ((skip >> (c >> 6)) & 1) continue;
          float v[16];
          double z[16];
          tmem_ld16(tb + (uint32_t)c, v);
          // exponents of the 16 columns, one per lane
          const int ec = c + (lane & 15) < ncol ? eb[n0 + c + (lane & 15)] : 0;
          double* cc = c0 + (int64_t)c * ldr;
          if (ncol - c >= 16) {
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = in ? cc[j * ldr] : 0.0;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              z[j] += slice64::neg_scaled(v[j], sh0 + __shfl_sync(0xffffffffu, ec, j));
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (in) cc[j * ldr] = z[j];
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const double p = slice64::neg_scaled(v[j], sh0 + __shfl_sync(0xffffffffu, ec, j));
              if (in && j < ncol - c) cc[j * ldr] += p;
            }
          }
        }
        release();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TNT) : "memory");
  }
}

// the digit pair (lo half, hi half) as two FP16 numbers: 1536 + d is exact in the half's last ten
// bits
__device__ __forceinline__ __half2 digits_h2(int lo, int hi) {
  const uint32_t u = (uint32_t)((0x6600 + lo) & 0xFFFF) | ((uint32_t)(0x6600 + hi) << 16);
  __half2 h;
  memcpy(&h, &u, 4);
  return __hsub2(h, __half2half2(__ushort_as_half((unsigned short)0x6600)));
}

// s_k of the columns of A: the power of two above a column's largest magnitude, a column per CTA
__global__ void __launch_bounds__(512) k_balance(const double2* A, int64_t lda, int64_t M, int* sk, int* count) {
  __shared__ uint32_t red[16];
  const double2* col = A + (int64_t)blockIdx.x * lda;
  uint32_t mx = 0;
#pragma unroll 4
  for (int64_t m = threadIdx.x; m < M; m += 512) {
    const double2 a = col[m];
    mx = max(mx, max(slice64::abs_hi(a.x), slice64::abs_hi(a.y)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int j = 1; j < 16; ++j) mx = max(mx, red[j]);
    sk[blockIdx.x] = slice64::balance_exponent(mx);
    if (blockIdx.x == 0) *count = 0;
  }
}

// the nine digits of (x, y): put(slice, digit of x, digit of y); returns the pair's magnitude
template <typename Put>
__device__ __forceinline__ __half slice_value(double2 a, int e, Put put) {
  int dr[PLANES], di[PLANES];
  const int64_t X = slice64::fixed62(a.x, e), Y = slice64::fixed62(a.y, e);
  slice64::digits9(X, dr);
  slice64::digits9(Y, di);
#pragma unroll
  for (int s = 0; s < PLANES; ++s) put(s, dr[s], di[s]);
  const bool zero = ((slice64::bits_of(a.x) | slice64::bits_of(a.y)) << 1) == 0;
  return __float2half_rn(slice64::spread_magnitude(X, Y, zero));
}

// A' slices of 32 rows of A per CTA: row maxima, then 32 x 64 tiles transposed through shared
// memory so that every warp writes whole row segments of each slice
__device__ __forceinline__ void slice_a(int bid, const double2* A, int64_t lda, int M, int K, const int* sk, __half2* Ap,
                                        __half* P, int* ea) {
  __shared__ int red[8][33];
  __shared__ double2 tile[32][65];
  __shared__ int s_e[32], s_k[KMAX];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m0 = bid * 32, m = m0 + lane;
  if (threadIdx.x < K) s_k[threadIdx.x] = sk[threadIdx.x];
  __syncthreads();
  int key = slice64::KEY_ZERO;
  if (m < M)
    for (int k = w; k < K; k += 8) {
      const double2 a = A[m + (int64_t)k * lda];
      key = max(key, max(slice64::scaled_key(a.x, -s_k[k]), slice64::scaled_key(a.y, -s_k[k])));
    }
  red[w][lane] = key;
  __syncthreads();
  if (w == 0) {
    for (int j = 1; j < 8; ++j) key = max(key, red[j][lane]);
    s_e[lane] = slice64::key_exponent(key);
    if (m < M) ea[m] = s_e[lane];
  }
  __syncthreads();
  for (int k0 = 0; k0 < K; k0 += 64) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + w + 8 * j;
      tile[lane][w + 8 * j] = (m < M && k < K) ? A[m + (int64_t)k * lda] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      const int r = w + 8 * i, mr = m0 + r;
      if (mr < M) {
        const int e = s_e[r];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = lane + 32 * h, k = k0 + kk;
          if (k < K) {
            __half2* row0 = Ap + (int64_t)(2 * mr) * K + k;  // 2K halves = K half2 per row
            P[(int64_t)mr * K + k] = slice_value(tile[r][kk], e + s_k[k], [&](int s, int dr, int di) {
              __half2* row = row0 + (int64_t)s * 2 * M * K;
              row[0] = digits_h2(dr, -di);
              row[K] = digits_h2(di, dr);
            });
          }
        }
      }
    }
    __syncthreads();
  }
}

// B' slices, one warp per column
__device__ __forceinline__ void slice_b(int bid, const double2* B, int64_t ldb, int K, int N, const int* sk, __half2* Bp,
                                        __half* Q, int* eb) {
  const int lane = threadIdx.x & 31;
  const int j = bid * 8 + (threadIdx.x >> 5);
  if (j >= N) return;
  const double2* col = B + (int64_t)j * ldb;
  int key = slice64::KEY_ZERO;
  for (int k = lane; k < K; k += 32) key = max(key, max(slice64::scaled_key(col[k].x, sk[k]), slice64::scaled_key(col[k].y, sk[k])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
  const int e = slice64::key_exponent(key);
  if (lane == 0) eb[j] = e;
  for (int k = lane; k < K; k += 32)
    Q[(int64_t)j * K + k] = slice_value(
        col[k], e - sk[k], [&](int s, int dr, int di) { Bp[((int64_t)s * N + j) * K + k] = digits_h2(dr, di); });
}

// both operands in one launch: CTAs [0, nA) 32 rows of A each, the rest 8 columns of B each
__global__ void __launch_bounds__(256) k_slice(const double2* A, int64_t lda, const double2* B, int64_t ldb, int M,
                                               int N, int K, const int* sk, __half2* Ap, __half* P, int* ea,
                                               __half2* Bp, __half* Q, int* eb, int nA) {
  if ((int)blockIdx.x < nA)
    slice_a(blockIdx.x, A, lda, M, K, sk, Ap, P, ea);
  else
    slice_b(blockIdx.x - nA, B, ldb, K, N, sk, Bp, Q, eb);
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

template <int TNT>
int run(beast_ctx* ctx, const CUtensorMap& tmA, const CUtensorMap& tmP, const __half2* Bp, const __half* Q, double* Cr,
        int64_t ldr, int M2, int N, int K, const int* ea, const int* eb, int2* list, int* count) {
  CUtensorMap tmB, tmQ;
  if (!make_map(&tmB, Bp, (uint64_t)2 * K, (uint64_t)PLANES * N, (uint64_t)2 * K * 2, TK, TNT, true,
                CU_TENSOR_MAP_DATA_TYPE_FLOAT16) ||
      !make_map(&tmQ, Q, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, TK, TNT, true, CU_TENSOR_MAP_DATA_TYPE_FLOAT16))
    return beast_fail(ctx, BEAST_ERR_CUDA, "tensor map encode (B' slices) failed");
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_tc_gemm64<TNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<TNT>::SMEM));
  const int tiles = ((M2 + TM - 1) / TM) * ((N + TNT - 1) / TNT);
  k_tc_gemm64<TNT><<<std::min(tiles, std::max(1, ctx->num_sms)), 192, Tile<TNT>::SMEM, ctx->stream>>>(
      tmA, tmB, tmP, tmQ, Cr, ldr, M2, N, ea, eb, 2 * K / TK, (K + TK - 1) / TK, list, count, ctx->d_flag);
  BEAST_CUDA_TRY(ctx, cudaGetLastError());
  return BEAST_OK;
}

}  // namespace

// 64 x 64 blocks of an M x N update, and the workspace it takes
static int64_t max_blocks(int64_t M, int64_t N) { return ((2 * M + TM - 1) / TM) * ((N + 63) / 64); }
size_t tc_gemm64_work_bytes(int64_t M, int64_t N, int K) {
  const int64_t k = std::min(K, KMAX);
  return al256((size_t)PLANES * M * k * 8) + al256((size_t)PLANES * N * k * 4) + al256((size_t)M * k * 2) +
         al256((size_t)N * k * 2) + al256((size_t)M * 4) + al256((size_t)N * 4) +
         al256(KMAX * 4) + al256((size_t)max_blocks(M, N) * 8 + 8);
}

// C -= A B (complex128): C at (M x N, ldc), A (M x K, lda), B (K x N, ldb), K a multiple of 32,
// taken KMAX columns at a time.  A wait that runs out sets bit 4 of the context's status word.
int tc_gemm64_sub(beast_ctx* ctx, double2* C, int64_t ldc, const double2* A, int64_t lda, const double2* B, int64_t ldb,
                  int64_t M, int64_t N, int K, void* work, size_t work_bytes) {
  if (K % 32 != 0 || 2 * M * PLANES > INT32_MAX || N * PLANES > INT32_MAX || tc_gemm64_work_bytes(M, N, K) > work_bytes)
    return beast_fail(ctx, BEAST_ERR_ARG, "sliced FP64 update: unsupported block");
  for (int k0 = 0; k0 < K; k0 += KMAX) {
    const int k = std::min(KMAX, K - k0);
    char* w = static_cast<char*>(work);
    auto take = [&](size_t bytes) {
      char* p = w;
      w += al256(bytes);
      return p;
    };
    __half2* Ap = reinterpret_cast<__half2*>(take((size_t)PLANES * M * k * 8));
    __half2* Bp = reinterpret_cast<__half2*>(take((size_t)PLANES * N * k * 4));
    __half* P = reinterpret_cast<__half*>(take((size_t)M * k * 2));
    __half* Q = reinterpret_cast<__half*>(take((size_t)N * k * 2));
    int* ea = reinterpret_cast<int*>(take((size_t)M * 4));
    int* eb = reinterpret_cast<int*>(take((size_t)N * 4));
    int* sk = reinterpret_cast<int*>(take(KMAX * 4));
    int* count = reinterpret_cast<int*>(w);
    int2* list = reinterpret_cast<int2*>(w) + 1;
    const double2 *Ak = A + (int64_t)k0 * lda, *Bk = B + k0;
    {
      // A read twice and B once, nine digits of 2 (A') and 1 (B') FP16 pairs and a magnitude written per element
      ProfScope ps(ctx, PK_CONVERT, (double)M * k * (32 + 74) + (double)N * k * (16 + 38), 2);
      const int nA = (int)((M + 31) / 32), nB = (int)((N + 7) / 8);
      k_balance<<<(unsigned)k, 512, 0, ctx->stream>>>(Ak, lda, M, sk, count);
      k_slice<<<(unsigned)(nA + nB), 256, 0, ctx->stream>>>(Ak, lda, Bk, ldb, (int)M, (int)N, k, sk, Ap, P, ea, Bp, Q,
                                                            eb, nA);
      BEAST_CUDA_TRY(ctx, cudaGetLastError());
    }
    CUtensorMap tmA, tmP;
    if (!make_map(&tmA, Ap, (uint64_t)2 * k, (uint64_t)PLANES * 2 * M, (uint64_t)2 * k * 2, TK, TM, true,
                  CU_TENSOR_MAP_DATA_TYPE_FLOAT16) ||
        !make_map(&tmP, P, (uint64_t)k, (uint64_t)M, (uint64_t)k * 2, TK, TM, true, CU_TENSOR_MAP_DATA_TYPE_FLOAT16))
      return beast_fail(ctx, BEAST_ERR_CUDA, "tensor map encode (A' slices) failed");
    const bool wide = ((2 * M + TM - 1) / TM) * ((N + 255) / 256) >= ctx->num_sms;
    {
      ProfScope ps(ctx, PK_TCGEMM, 8.0 * k * (double)M * N);
      double* Cr = reinterpret_cast<double*>(C);
      const int rc = wide ? run<256>(ctx, tmA, tmP, Bp, Q, Cr, 2 * ldc, (int)(2 * M), (int)N, k, ea, eb, list, count)
                          : run<64>(ctx, tmA, tmP, Bp, Q, Cr, 2 * ldc, (int)(2 * M), (int)N, k, ea, eb, list, count);
      if (rc) return rc;
    }
    ProfScope ps(ctx, PK_GEMM, 0.0);
    BEAST_CUDA_TRY(ctx, gemm64_tiles(list, count, C, ldc, Ak, lda, Bk, ldb, M, N, k, std::max(1, 2 * ctx->num_sms),
                                     ctx->stream));
  }
  return BEAST_OK;
}

bool tc_gemm64_supported() { return encode_fn() != nullptr; }
