// linalg.cu -- dense complex LU with partial pivoting, triangular solves, FP64 matvec.
//
// Replaces LAPACK zgetrf/zgetrs behind `\` (src/solvers/lusolver.jl:30, src/solvers/lu.jl:40-47)
// for a device-resident matrix.  Right-looking blocked LU:
//   k_panel    cooperative kernel over the column panel: per column a pivot search over all
//              CTAs (max |re|+|im|, first index on ties -- the izamax rule) by one exchange
//              through slots that are their own ready flags, the row swap and the rank-1
//              update (a bounded wait that gives up sets a status word and the kernel
//              returns; nothing hangs)
//   k_laswp    the panel's row interchanges applied to the other columns
//   k_trsm_tile   U12 = L11^{-1} A12 and (unpivoted path, after k_getrf64 on the diagonal
//                 block) L21 = A21 U11^{-1}
//   k_lu_inv64(_pair) + k_panel_apply   the unpivoted c64 panel: diagonal block LU with the
//                 inverses of its triangles, then both triangular solves as products
//   A22 -= L21 U12: on the tensor cores (tc_gemm.cu for c64, tc_gemm64.cu for c128), else
//                 k_gemm (complex, tiled through shared memory)
// The element type is complex FP64 (c128) or complex FP32 (c64).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "fsplit.h"
#include "internal.h"

// the pivot allocation of a factorisation: ipiv[n], perm[n], then (256-byte aligned) the
// inverses of the 64 x 64 diagonal blocks of L and U
size_t lu_aux_bytes(int64_t n, int dtype) {
  size_t head = ((size_t)2 * n * sizeof(int) + 255) & ~(size_t)255;
  size_t el = dtype == BEAST_C64 ? 8 : 16;
  return head + (size_t)((n + 63) / 64) * 2 * 4096 * el;
}
void* lu_dinv(const int* ipiv, int64_t n) {
  size_t head = ((size_t)2 * n * sizeof(int) + 255) & ~(size_t)255;
  return (void*)(reinterpret_cast<const char*>(ipiv) + head);
}

bool tc_gemm_supported(const void* A, int64_t lda, int K);
size_t tc_gemm_work_bytes(int64_t M, int64_t N, int K);
int tc_gemm_sub(beast_ctx* ctx, float2* Mat, int64_t lda, int64_t rowA, int64_t colA, int64_t colB,
                int64_t M0, int64_t N0, int64_t M1, int64_t N1, int K, void* work, size_t work_bytes,
                bool prepped);
int tc_gemm_sym(beast_ctx* ctx, float2* Mat, int64_t lda, int64_t rowA, int64_t colA, int64_t rowB, int64_t M0,
                int64_t N0, int K, bool lower, void* work, size_t work_bytes, bool prepped, int64_t a_skip = 0);
size_t tc_gemm64_work_bytes(int64_t M, int64_t N, int K);
int tc_gemm64_sub(beast_ctx* ctx, double2* C, int64_t ldc, const double2* A, int64_t lda, const double2* B, int64_t ldb,
                  int64_t M, int64_t N, int K, void* work, size_t work_bytes);
bool tc_gemm64_supported();

namespace {

template <typename R>
struct CT;
template <>
struct CT<double> {
  typedef double2 T;
};
template <>
struct CT<float> {
  typedef float2 T;
};

template <typename T>
__device__ __forceinline__ T cmk(double re, double im);
template <>
__device__ __forceinline__ double2 cmk<double2>(double re, double im) {
  return make_double2(re, im);
}
template <>
__device__ __forceinline__ float2 cmk<float2>(double re, double im) {
  return make_float2((float)re, (float)im);
}

template <typename T>
__device__ __forceinline__ void cfms(T& acc, T a, T b) {  // acc -= a b, four fused multiply-adds
  acc.x = fma(-a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(-a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}

// ---- panel factorisation ---------------------------------------------------------------
// Cooperative launch (all CTAs co-resident); a CTA keeps its slice of the panel's rows in shared
// memory for the whole panel.  What bounds it is the chain per column -- the pivot is chosen over all
// CTAs, and an FP64 instruction holds its quarter of an SM for 64 cycles -- so a column has one
// one-sided exchange, no grid barrier, and few FP64 instructions one after the other:
//   - every CTA publishes its candidate (|re| + |im| as an integer key, row index), the candidate's row
//     (the owner of row j that row too) and the candidate's reciprocal into slots of this column that
//     start as sentinels (all ones; the host fills them before the launch): a value that is not the
//     sentinel is its own ready flag, so there is no fence, counter or second round trip.  The
//     candidate goes to a slot of its own for every reader: a line that many SMs poll while it is
//     written reaches some of them 2 us late (5.2 us per column at 30 CTAs, against 2.9);
//   - warp 0 of every CTA reads all candidates, takes the same pivot (largest, first index on ties:
//     the izamax rule) and reads the winner's row and reciprocal;
//   - meanwhile the other warps do the previous column's rank-1 update: only the next column, the
//     candidate's row and row j have to be up to date before the exchange;
//   - a thread per row forms the multiplier, updates the next column and that entry's key.
// Measured: order 480 (8 panels) 4.0 -> 1.36 ms, order 6007 (94 panels) 56 -> 20.3 ms against a
// grid barrier per column with the whole update between two of them.
// A wait that runs out sets *status (the host reports BEAST_ERR_TIMEOUT) and every CTA returns.
constexpr unsigned long long PANEL_SENT = ~0ull;
constexpr int PANEL_POLLS = 1 << 21;  // of one slot: about a second
constexpr int PANEL_ROWS = 16;        // least rows per CTA
constexpr int PANEL_CAND = 5;         // candidates a lane reads at a time

__device__ __forceinline__ unsigned long long panel_word(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return u == PANEL_SENT ? 0x7FF8000000000000ull : u;  // another NaN
}
__device__ __forceinline__ void panel_put2(unsigned long long* slot, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void panel_put(unsigned long long* slot, double2 v) {
  panel_put2(slot, panel_word(v.x), panel_word(v.y));
}
__device__ __forceinline__ void panel_put(unsigned long long* slot, float2 v) {
  const unsigned long long u = ((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x);
  *reinterpret_cast<volatile unsigned long long*>(slot) = u == PANEL_SENT ? 0x7FC000007FC00000ull : u;
}
__device__ __forceinline__ void panel_value(const unsigned long long* u, double2& v) {
  v = make_double2(__longlong_as_double((long long)u[0]), __longlong_as_double((long long)u[1]));
}
__device__ __forceinline__ void panel_value(const unsigned long long* u, float2& v) {
  v = make_float2(__uint_as_float((unsigned)(u[0] & 0xffffffffull)), __uint_as_float((unsigned)(u[0] >> 32)));
}
__device__ __forceinline__ void panel_load(const unsigned long long* p, unsigned long long (&u)[1]) {
  u[0] = *reinterpret_cast<const volatile unsigned long long*>(p);
}
__device__ __forceinline__ void panel_load(const unsigned long long* p, unsigned long long (&u)[2]) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u[0]), "=l"(u[1]) : "l"(p) : "memory");
}
// waits (bounded) until the N slots of W words at p[0 .. N) (null: none) are written, all of them
// requested together: a read of another CTA's slot takes most of a microsecond; false: gave up.
// (A slot of two words is read by one instruction and may still arrive half by half: each word is
// its own flag.)
template <int N, int W>
__device__ __forceinline__ bool panel_wait(const unsigned long long* const* p, unsigned long long (*u)[W]) {
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int c = 0; c < W; ++c) u[k][c] = p[k] ? PANEL_SENT : 0ull;
  for (int it = 0; it < PANEL_POLLS; ++it) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (u[k][0] == PANEL_SENT || u[k][W - 1] == PANEL_SENT) panel_load(p[k], u[k]);
#pragma unroll
    for (int k = 0; k < N; ++k) ok &= u[k][0] != PANEL_SENT && u[k][W - 1] != PANEL_SENT;
    if (ok) return true;
  }
  return false;
}
// 8-byte words of the exchange slots of one column, panel of nb columns on G CTAs: for each CTA the G
// candidates (key, index), then G reciprocals, G rows and row j
template <typename T>
__host__ __device__ inline size_t panel_column_words(int nb, int G) {
  const size_t W = sizeof(T) / 8;
  return (2 * (size_t)G * G + (size_t)G * W + ((size_t)G + 1) * nb * W + 1) & ~(size_t)1;  // 16-byte columns
}

// pivot key of a value: ordered like |re| + |im|, 1 for zero, 0 for a NaN (never a pivot)
template <typename T>
__device__ __forceinline__ unsigned long long panel_key(T a) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(fabs((double)a.x) + fabs((double)a.y));
  return u > 0x7FF0000000000000ull ? 0ull : u + 1ull;
}
// the warp's largest key, the smallest index among equals
__device__ __forceinline__ void panel_best(unsigned long long& key, int& idx, int& who) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, idx, o), w2 = __shfl_xor_sync(0xffffffffu, who, o);
    if (k2 > key || (k2 == key && i2 < idx)) {
      key = k2;
      idx = i2;
      who = w2;
    }
  }
}
// |z|^2 in a range where it and its reciprocal are normal numbers
__device__ __forceinline__ bool square_in_range(double den) { return den >= 0x1p-1000 && den <= 0x1p1000; }
// 1 / z for any z by a power of two taken out of it (infinite below 2^-1024); zero for zero, NaN for what is
// not finite
__device__ __noinline__ double2 recip_scaled(double2 z) {
  const double m = fmax(fabs(z.x), fabs(z.y));
  if (m == 0.0) return make_double2(0.0, 0.0);
  if (!(m <= 1.7976931348623157e308) || isnan(z.x) || isnan(z.y)) return make_double2(nan(""), nan(""));
  const int e = ilogb(m);
  const double x = scalbn(z.x, -e), y = scalbn(z.y, -e), den = x * x + y * y;
  return make_double2(scalbn(x / den, -e), scalbn(-y / den, -e));
}
// (1 / piv) in the factorisation's arithmetic, by one division (an FP64 division is 30 instructions
// on the column's chain); zero for a zero pivot
__device__ __forceinline__ double2 panel_recip(double2 piv) {
  const double den = piv.x * piv.x + piv.y * piv.y;
  if (!square_in_range(den)) return recip_scaled(piv);
  const double id = 1.0 / den;
  return make_double2(piv.x * id, -piv.y * id);
}
__device__ __forceinline__ float2 panel_recip(float2 piv) {
  const double den = (double)piv.x * piv.x + (double)piv.y * piv.y, id = den != 0.0 ? 1.0 / den : 0.0;
  return make_float2((float)(piv.x * id), (float)(-piv.y * id));
}

template <typename T>
__global__ void __launch_bounds__(256) k_panel(T* A, int64_t lda, int64_t n, int64_t j0, int nb, int rows_per, int* ipiv,
                                               int* info, unsigned long long* slots, int* status) {
  constexpr int W = sizeof(T) / 8, NONE = 0x7fffffff;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = nb + 1;  // padded row stride (bank spread)
  T* S = reinterpret_cast<T*>(smraw);   // rows_per x ld
  T* Ub = S + (size_t)rows_per * ld;    // pivot rows of this column and the last one (2 x nb)
  T* Rj = Ub + 2 * nb;                  // row j, for the owner of the pivot's row
  __shared__ unsigned long long s_key[8];
  __shared__ int s_row[8], s_bad, s_go[2];  // s_go: the column (by parity) has a usable pivot
  __shared__ int s_p;
  __shared__ T s_inv;
  const int G = (int)gridDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t r0 = j0 + (int64_t)blockIdx.x * rows_per;
  const int nloc = (int)(n - r0 < (int64_t)rows_per ? (n - r0 > 0 ? n - r0 : 0) : (int64_t)rows_per);
  for (int e = tid; e < nloc * nb; e += blockDim.x) {
    const int i = e % nloc, k = e / nloc;
    S[i * ld + k] = A[(r0 + i) + (j0 + k) * lda];
  }
  if (tid == 0) s_bad = 0;
  __syncthreads();
  // keys of column 0, per warp
  {
    unsigned long long key = 0;
    int row = NONE, who = 0;
    for (int i = tid; i < nloc; i += 256) {
      const unsigned long long k2 = panel_key(S[i * ld]);
      if (k2 > key) {
        key = k2;
        row = i;
      }
    }
    panel_best(key, row, who);
    if (lane == 0) {
      s_key[warp] = key;
      s_row[warp] = row;
    }
  }
  __syncthreads();
  for (int jj = 0; jj < nb; ++jj) {
    const int64_t j = j0 + jj;
    unsigned long long* cand = slots + jj * panel_column_words<T>(nb, G);
    unsigned long long* invs = cand + 2 * (size_t)G * G;
    unsigned long long* rows = invs + (size_t)G * W;
    unsigned long long* rowj = rows + (size_t)G * nb * W;
    T* U = Ub + (jj & 1) * nb;              // this column's pivot row
    const T* Up = Ub + ((jj + 1) & 1) * nb;  // the last one's
    const int lj = (j >= r0 && j < r0 + nloc) ? (int)(j - r0) : -1;
    const bool pend = jj > 0 && s_go[(jj + 1) & 1];
    // 1. the CTA's candidate from the warps' keys; its row and row j brought up to date and published
    int li = -1;
    unsigned long long lkey = 0;
    {
      int row = NONE;
#pragma unroll
      for (int w = 0; w < 8; ++w)
        if (s_key[w] > lkey || (s_key[w] == lkey && lkey > 0 && s_row[w] < row)) {
          lkey = s_key[w];
          row = s_row[w];
        }
      if (lkey > 0) li = row;
    }
    for (int b = tid; b < G; b += 256)
      panel_put2(cand + 2 * ((size_t)b * G + blockIdx.x), lkey,
                 (unsigned long long)(li >= 0 ? (unsigned)(r0 + li) : (unsigned)NONE));
    if (warp < 4) {
      const int rw = warp < 2 ? li : (lj != li ? lj : -1), k = (warp & 1) * 32 + lane;
      if (rw >= 0 && k < nb) {
        T c = S[rw * ld + k];
        if (pend && k > jj) {
          cfms(c, S[rw * ld + jj - 1], Up[k]);
          S[rw * ld + k] = c;
        }
        if (warp < 2) panel_put(rows + ((size_t)blockIdx.x * nb + k) * W, c);
        if (rw == lj) panel_put(rowj + (size_t)k * W, c);
      }
    } else if (warp == 4 && lane == 0 && li >= 0) {
      panel_put(invs + (size_t)blockIdx.x * W, panel_recip(S[li * ld + jj]));
    }
    if (warp > 0) {
      // 2a. the last column's update of the other rows (columns beyond jj)
      const int ncol = nb - jj - 1;
      if (pend && ncol > 0) {
        const int ibeg = j > r0 ? (int)(j - r0 < nloc ? j - r0 : nloc) : 0;
        const float inv = 1.0f / (float)ncol;
        const int tot = (nloc - ibeg) * ncol;
        for (int e = tid - 32; e < tot; e += 224) {
          // e / ncol: a CTA's rows x columns take at most 220 KB, so e < 2^15 and the product is within 2^-7 / ncol of
          // (e + 1/2) / ncol
          const int q = (int)(((float)e + 0.5f) * inv);
          const int i = ibeg + q, k = jj + 1 + (e - q * ncol);
          if (i == li || i == lj) continue;
          T c = S[i * ld + k];
          cfms(c, S[i * ld + jj - 1], Up[k]);
          S[i * ld + k] = c;
        }
      }
    } else {
      // 2b. the pivot over all candidates, its row and its reciprocal
      unsigned long long key = 0;
      int p = NONE, w = 0;
      bool ok = true;
      for (int b0 = 0; b0 < G; b0 += 32 * PANEL_CAND) {
        const unsigned long long* q[PANEL_CAND];
        unsigned long long u[PANEL_CAND][2];
#pragma unroll
        for (int c = 0; c < PANEL_CAND; ++c) {
          const int b = b0 + 32 * c + lane;
          q[c] = b < G ? cand + 2 * ((size_t)blockIdx.x * G + b) : nullptr;
        }
        ok = ok && panel_wait<PANEL_CAND, 2>(q, u);
#pragma unroll
        for (int c = 0; c < PANEL_CAND; ++c)
          if (u[c][0] > key || (u[c][0] == key && key > 0 && (int)u[c][1] < p)) {
            key = u[c][0];
            p = (int)u[c][1];
            w = b0 + 32 * c + lane;
          }
      }
      ok = __all_sync(0xffffffffu, ok);
      panel_best(key, p, w);
      const bool sing = key <= 1ull;  // exactly singular column: recorded, no interchange
      if (sing) p = (int)j;
      const unsigned long long* src = sing ? rowj : rows + (size_t)w * nb * W;
      const int lp = (p != (int)j && p >= r0 && p < r0 + nloc) ? (int)(p - r0) : -1;
      T inv;
      inv.x = inv.y = 0;
      {
        // entries lane and lane + 32 of the pivot's row and (for the owner of the pivot's row) of
        // row j, and the reciprocal
        const unsigned long long* q[5];
        unsigned long long u[5][W];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = lane + 32 * h;
          q[h] = k < nb ? src + (size_t)k * W : nullptr;
          q[2 + h] = k < nb && lp >= 0 ? rowj + (size_t)k * W : nullptr;
        }
        q[4] = lane == 0 && !sing ? invs + (size_t)w * W : nullptr;
        ok = ok && panel_wait<5, W>(q, u);
        ok = __all_sync(0xffffffffu, ok);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = lane + 32 * h;
          T v;
          if (k < nb) {
            panel_value(u[h], v);
            U[k] = v;
            panel_value(u[2 + h], v);
            if (lp >= 0) Rj[k] = v;
          }
        }
        if (!sing) panel_value(u[4], inv);
      }
      if (lane == 0) {
        s_p = p;
        s_inv = inv;
        const bool over = isinf(inv.x) || isinf(inv.y);  // a pivot too small for its reciprocal: as a zero one
        s_go[jj & 1] = !over && (inv.x != 0 || inv.y != 0);
        if (!ok) {
          s_bad = 1;
          atomicOr(status, 1);
        }
        if (blockIdx.x == 0) {
          ipiv[j] = p;
          if ((sing || over) && *info == 0) *info = (int)j + 1;
        }
      }
    }
    __syncthreads();
    if (s_bad) return;
    // 3. the interchange; the multipliers and the next column of own rows below j, and its keys (the
    // pivot's old row takes columns jj and jj + 1 from row j directly)
    unsigned long long key = 0;
    int row = NONE, who = 0;
    const int p = s_p;
    const int lp = (p != (int)j && p >= r0 && p < r0 + nloc) ? (int)(p - r0) : -1;
    if (tid >= 192) {
      const int k = tid - 192;
      if (k < nb) {
        if (lp >= 0 && k != jj && k != jj + 1) S[lp * ld + k] = Rj[k];
        if (p != (int)j && lj >= 0) S[lj * ld + k] = U[k];
      }
    }
    {
      const bool go = s_go[jj & 1];
      const T inv = s_inv;
      const int ibeg = (j + 1 - r0) > 0 ? (int)((j + 1 - r0) < nloc ? (j + 1 - r0) : nloc) : 0;
      for (int i = ibeg + tid; i < nloc; i += 256) {
        T l = i == lp ? Rj[jj] : S[i * ld + jj];
        if (i == lp) S[i * ld + jj] = l;
        if (go) {
          const T a = l;
          l.x = a.x * inv.x - a.y * inv.y;
          l.y = a.x * inv.y + a.y * inv.x;
          S[i * ld + jj] = l;
        }
        if (jj + 1 < nb) {
          T c = i == lp ? Rj[jj + 1] : S[i * ld + jj + 1];
          if (go) cfms(c, l, U[jj + 1]);
          if (go || i == lp) S[i * ld + jj + 1] = c;
          const unsigned long long k2 = panel_key(c);
          if (k2 > key) {
            key = k2;
            row = i;
          }
        }
      }
    }
    panel_best(key, row, who);
    if (lane == 0) {
      s_key[warp] = key;
      s_row[warp] = row;
    }
    __syncthreads();
  }
  for (int e = tid; e < nloc * nb; e += blockDim.x) {
    const int i = e % nloc, k = e / nloc;
    A[(r0 + i) + (j0 + k) * lda] = S[i * ld + k];
  }
}

// ---- row interchanges ipiv[p0, p1) applied (in order) to columns [c0, c1) ----------------
template <typename T>
__global__ void k_laswp(T* A, int64_t lda, int64_t c0, int64_t c1, int64_t p0, int64_t p1,
                        const int* ipiv) {
  int64_t col = c0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (col >= c1) return;
  for (int64_t r = p0; r < p1; ++r) {
    int64_t p = ipiv[r];
    if (p != r) {
      T a = A[r + col * lda];
      A[r + col * lda] = A[p + col * lda];
      A[p + col * lda] = a;
    }
  }
}

// ---- LU of a diagonal block without pivoting (mixed path) --------------------------------
// A[j0:j0+kb, j0:j0+kb] = L11 U11 in place, kb <= 64, one CTA of 256 threads in shared
// memory, blocked by 16 columns (three barriers per 16 pivots):
//   1. warp 0 factors the 64 x 16 column slab in registers (lane l holds rows l and l + 32;
//      the pivot row is broadcast with shuffles, so the 16 pivot steps need no block barrier);
//   2. U12 of the slab's rows, one column per thread (unit lower 16 x 16 substitution);
//   3. rank-16 update of the trailing block by all threads.
// A zero pivot sets *info (1-based column) and the kernel stops.
constexpr int TRI = 64;

template <typename T>
__device__ __forceinline__ void cfma(T& acc, T a, T b) {  // acc += a b
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}
template <typename T>
__device__ __forceinline__ T cmulx(T a, T b) {
  T r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
// r = 1 / p; false for p = 0.  FP32: the hardware reciprocal (rcp.approx, within 1 ulp) --
// this is on the serial pivot chain of the unpivoted mixed-precision LU, whose result is
// refined in FP64 anyway; FP64: IEEE division
__device__ __forceinline__ float rcp_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ bool crecip(float2 p, float2& r) {
  const float den = p.x * p.x + p.y * p.y;
  if (den == 0.f) return false;
  const float id = rcp_f(den);
  r.x = p.x * id;
  r.y = -p.y * id;
  return true;
}
__device__ __forceinline__ bool crecip(double2 p, double2& r) {
  const double den = p.x * p.x + p.y * p.y;
  if (den == 0.0) return false;
  const double id = 1.0 / den;
  r.x = p.x * id;
  r.y = -p.y * id;
  return true;
}

template <typename T>
__device__ __forceinline__ T shfl_c(T v, int src) {
  T r;
  r.x = __shfl_sync(0xffffffffu, v.x, src);
  r.y = __shfl_sync(0xffffffffu, v.y, src);
  return r;
}

template <typename T>
__global__ void __launch_bounds__(256) k_getrf64(T* A, int64_t lda, int64_t j0, int kb, int* info) {
  constexpr int LD = TRI + 1, PB = 16;
  extern __shared__ unsigned char smraw[];
  T* D = reinterpret_cast<T*>(smraw);  // row-major, ld LD, zero outside kb x kb
  __shared__ int s_zero;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the block, 16 loads per thread issued before their stores so that they overlap
  {
    T v[TRI * TRI / 256];
#pragma unroll
    for (int j = 0; j < TRI * TRI / 256; ++j) {
      const int e = tid + 256 * j, r = e % TRI, k = e / TRI;
      v[j] = (r < kb && k < kb) ? A[(j0 + r) + (j0 + k) * lda] : T{0, 0};
    }
#pragma unroll
    for (int j = 0; j < TRI * TRI / 256; ++j) {
      const int e = tid + 256 * j;
      D[(e % TRI) * LD + e / TRI] = v[j];
    }
  }
  if (tid == 0) s_zero = 0;
  __syncthreads();
  for (int k0 = 0; k0 < kb; k0 += PB) {
    const int nbk = min(PB, kb - k0);
    // 1. the column slab k0 .. k0+15 by warp 0
    if (warp == 0) {
      T a[2][PB];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < PB; ++c) a[h][c] = D[(lane + 32 * h) * LD + k0 + c];
      int zero_at = 0;
#pragma unroll
      for (int k = 0; k < PB; ++k) {
        if (k < nbk && zero_at == 0) {  // uniform over the warp
          const int pr = k0 + k, ow = pr & 31, oh = pr >> 5;
          T u[PB];
#pragma unroll
          for (int c = k; c < PB; ++c) u[c] = shfl_c(oh ? a[1][c] : a[0][c], ow);
          T ip;
          if (!crecip(u[k], ip)) {
            zero_at = pr + 1;
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int i = lane + 32 * h;
              if (i > pr && i < kb) {
                const T l = cmulx(a[h][k], ip);
                a[h][k] = l;
#pragma unroll
                for (int c = k + 1; c < PB; ++c) cfms(a[h][c], l, u[c]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < PB; ++c) D[(lane + 32 * h) * LD + k0 + c] = a[h][c];
      if (lane == 0 && zero_at) s_zero = zero_at;
    }
    __syncthreads();
    if (s_zero) {  // uniform
      if (tid == 0) atomicCAS(info, 0, (int)(j0 + s_zero));
      return;
    }
    const int c1 = k0 + PB;  // first column right of the slab (the slab is complete here)
    if (c1 >= kb) break;
    // 2. U12 = L11^{-1} A12 for the slab's 16 rows, one column per thread
    if (tid < kb - c1) {
      const int c = c1 + tid;
      T x[PB];
#pragma unroll
      for (int i = 0; i < PB; ++i) x[i] = D[(k0 + i) * LD + c];
#pragma unroll
      for (int i = 1; i < PB; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) cfms(x[i], D[(k0 + i) * LD + k0 + j], x[j]);
#pragma unroll
      for (int i = 1; i < PB; ++i) D[(k0 + i) * LD + c] = x[i];
    }
    __syncthreads();
    // 3. rank-16 update of the trailing block
    const int w = kb - c1;
    for (int e = tid; e < w * w; e += 256) {
      const int r = c1 + e / w, c = c1 + e % w;
      T acc = D[r * LD + c];
#pragma unroll
      for (int j = 0; j < PB; ++j) cfms(acc, D[r * LD + k0 + j], D[(k0 + j) * LD + c]);
      D[r * LD + c] = acc;
    }
    __syncthreads();
  }
  for (int e = tid; e < kb * kb; e += 256) {
    const int r = e % kb, k = e / kb;
    A[(j0 + r) + (j0 + k) * lda] = D[r * LD + k];
  }
}

// ---- diagonal block LU together with the inverses of its triangles ---------------------
// For the unpivoted c64 path: the 64 x 64 block at (j0, j0) (kb x kb, the rest padded with
// the identity) is factored by forward elimination on [A | I] -- eliminating below the pivot
// turns the identity part of the rows into L^{-1} (it lives in the strictly lower positions
// the elimination has just emptied), while the upper part becomes U -- and in the same pass
// X = (U^T)^{-1} = (U^{-1})^T is built by forward elimination on U^T, whose multipliers
// U[k][r] are the pivot row itself.  Step k (rows r > k), with d = 1 / U[k][k]:
//   S1[r][c] -= (A[r][k] d) P1[c]   (P1 = row k of S1 with 0 at column k)
//   S1[r][k]  = -A[r][k] d          (L^{-1}[r][k] after this step; L[r][k] = A[r][k] d)
//   S2[r][c] -= (U[k][r] d) P2[c]   (P2 = row k of S2, before its own scaling)
//   S2[k][c] *= d
// Each thread holds a 4 x 4 tile of S1 and of S2 in registers (rows 4 rb.., columns 4 cb..;
// a warp = 2 row blocks x 16 column blocks).  After each step the owners of row k+1, of
// column k+1 and of the pivot publish P1, P2, the column and 1 / pivot in shared memory
// (double-buffered by step parity): one block barrier per step.  The step loop is unrolled
// by 4, so the tile slot of row / column k is known at compile time and the code is short
// (this kernel runs alone on one SM between wide launches: it is latency-bound and starts
// with cold instruction caches).  Output: the factors in A, Linv and Uinv (column-major
// 64 x 64, identity beyond kb) in inv.  A zero pivot sets *info (1-based column) and the
// kernel stops.
template <typename T>
__device__ __forceinline__ int pidx(int c) {  // conflict-free index of the published rows
  return c + (c >> 2);
}

// SYM: only the lower triangle of the block is current (symmetric updates); the upper one
// is taken from it by symmetry, the elimination on U^T is skipped and, U = D L^T,
// U^{-1} = (L^{-1})^T D^{-1} is formed from L^{-1} and the pivots at the end.
// TR x TC: the tile a thread owns (rows x columns): 4 x 4 (256 threads) or 2 x 4 (512); 2 x 2 tiles:
// k_lu_inv64_pair.  The arithmetic per element is the same for every tile.
template <typename T, bool SYM, int TR = 4, int TC = TR>
__global__ void __launch_bounds__(TRI * TRI / (TR * TC)) k_lu_inv64(T* A, int64_t lda, int64_t j0, int kb, int* info,
                                                                   T* inv) {
  constexpr bool sym = SYM;
  constexpr int NT = TRI * TRI / (TR * TC);  // threads
  constexpr int NCB = TRI / TC;              // column blocks: 32 (a warp) or 16 (half a warp)
  static_assert(TC % TR == 0 && (NCB == 32 || NCB == 16), "tile: TR divides TC, TC = 2 or 4");
  constexpr int LD = TRI + 1, PL = TRI + TRI / 4;
  extern __shared__ unsigned char smraw[];
  T* Ls = reinterpret_cast<T*>(smraw);  // 64 x LD: staging, then the L factor, then Linv
  __shared__ T p1[2][PL], p2[2][PL], lc[2][TRI];
  __shared__ T dv[2];
  __shared__ int s_zero[2];  // 1-based column of a zero pivot, by step parity
  // the panel products launched after this kernel may start their loads now (they wait for
  // its results before reading them)
  asm volatile("griddepcontrol.launch_dependents;");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cb = NCB == 16 ? (lane & 15) : lane, rb = NCB == 16 ? 2 * warp + (lane >> 4) : warp;
  const int r0 = TR * rb, c0 = TC * cb;
  const T zero = cmk<T>(0.0, 0.0), one = cmk<T>(1.0, 0.0);
  // coalesced load through shared memory (identity padding beyond kb)
  for (int e = tid; e < TRI * TRI; e += NT) {
    const int r = e & (TRI - 1), c = e >> 6;
    const int rr = (sym && c > r) ? c : r, cc = (sym && c > r) ? r : c;
    Ls[r * LD + c] = (r < kb && c < kb) ? A[(j0 + rr) + (j0 + cc) * lda] : (r == c ? one : zero);
  }
  if (tid < 2) s_zero[tid] = 0;
  __syncthreads();
  T s1[TR][TC], s2[TR][TC];
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      s1[i][j] = Ls[(r0 + i) * LD + c0 + j];
      s2[i][j] = (r0 + i == c0 + j) ? one : zero;
    }
  // publish row 0, column 0 and the first pivot's reciprocal
  if (rb == 0)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      p1[0][pidx<T>(c0 + j)] = (c0 + j == 0) ? zero : s1[0][j];
      if (!SYM) p2[0][pidx<T>(c0 + j)] = s2[0][j];
    }
  if (cb == 0)
#pragma unroll
    for (int i = 0; i < TR; ++i) lc[0][r0 + i] = s1[i][0];
  if (rb == 0 && cb == 0) {
    T d;
    if (!crecip(s1[0][0], d)) s_zero[0] = 1;
    dv[0] = d;
  }
  __syncthreads();  // the staging buffer is free from here on (L factor)
  // steps unrolled by TC: column k is slot kk of column block kq, row k slot kk % TR of row
  // block k / TR (TR divides TC), so every register index below is known at compile time
  for (int kq = 0; kq < TRI / TC; ++kq) {
#pragma unroll
    for (int kk = 0; kk < TC; ++kk) {
      const int k = TC * kq + kk, b = kk & 1;
      if (s_zero[b]) {  // uniform
        if (tid == 0) atomicCAS(info, 0, (int)(j0 + s_zero[b]));
        return;
      }
      const T d = dv[b];
      if (r0 + TR - 1 > k) {  // some row of the tile is below the pivot
        T l1[TR], l2[TR], q1[TC], q2[TC];
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          l1[i] = cmulx(lc[b][r0 + i], d);
          l2[i] = cmulx(p1[b][pidx<T>(r0 + i)], d);
        }
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          q1[j] = p1[b][pidx<T>(c0 + j)];
          q2[j] = p2[b][pidx<T>(c0 + j)];
        }
#pragma unroll
        for (int i = 0; i < TR; ++i)
          if (r0 + i > k) {
#pragma unroll
            for (int j = 0; j < TC; ++j) {
              cfms(s1[i][j], l1[i], q1[j]);
              if (!SYM) cfms(s2[i][j], l2[i], q2[j]);
            }
            if (cb == kq) {  // column k: L^{-1}[r][k] = -l, and the L factor
              s1[i][kk].x = -l1[i].x;
              s1[i][kk].y = -l1[i].y;
              Ls[(r0 + i) * LD + k] = l1[i];
            }
          }
      }
      if (!SYM && rb == k / TR)  // row k of X is final
#pragma unroll
        for (int j = 0; j < TC; ++j) s2[kk % TR][j] = cmulx(s2[kk % TR][j], d);
      // publish step k + 1
      if (k + 1 < TRI) {
        const int kn = k + 1, bn = b ^ 1;
        const int qr = kn / TR, ir = (kk + 1) % TR, qc = kn / TC, ic = (kk + 1) % TC;
        if (rb == qr)
#pragma unroll
          for (int j = 0; j < TC; ++j) {
            p1[bn][pidx<T>(c0 + j)] = (c0 + j == kn) ? zero : s1[ir][j];
            if (!SYM) p2[bn][pidx<T>(c0 + j)] = s2[ir][j];
          }
        if (cb == qc)
#pragma unroll
          for (int i = 0; i < TR; ++i) lc[bn][r0 + i] = s1[i][ic];
        if (rb == qr && cb == qc) {
          T dn;
          if (!crecip(s1[ir][ic], dn)) s_zero[bn] = kn + 1;
          dv[bn] = dn;
        }
      }
      __syncthreads();
    }
  }
  // U (upper part of S1) joins the L factor in Ls; the factored block goes back to A
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j)
      if (c0 + j >= r0 + i) Ls[(r0 + i) * LD + c0 + j] = s1[i][j];
  __syncthreads();
  for (int e = tid; e < kb * kb; e += NT) {
    const int r = e % kb, c = e / kb;
    A[(j0 + r) + (j0 + c) * lda] = Ls[r * LD + c];
  }
  __syncthreads();
  // Linv (column-major, inv[c * 64 + r] = Linv[r][c]) through Ls; Uinv = X^T, so row r of X
  // is column r of Uinv (inv[4096 + r * 64 + c] = X[r][c]), written by the tile owners;
  // symmetric: X[r][c] = Linv[r][c] / d_r
  if (SYM) {
    __shared__ T s_dinv[TRI];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j)
        if (c0 + j == r0 + i) {  // the tile holding the pivot of row r0 + i
          T di;
          crecip(s1[i][j], di);  // nonzero: the elimination checked every pivot
          s_dinv[r0 + i] = di;
        }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      const T di = s_dinv[r0 + i];
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        const int r = r0 + i, c = c0 + j;
        s2[i][j] = c < r ? cmulx(s1[i][j], di) : (c == r ? di : zero);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      const int r = r0 + i, c = c0 + j;
      Ls[r * LD + c] = c < r ? s1[i][j] : (c == r ? one : zero);
      inv[TRI * TRI + r * TRI + c] = s2[i][j];
    }
  __syncthreads();
  for (int e = tid; e < TRI * TRI; e += NT) {
    const int r = e & (TRI - 1), c = e >> 6;
    inv[e] = Ls[r * LD + c];
  }
}

// two neighbouring complex values of shared memory (the first at an even place) in one load
__device__ __forceinline__ void ld_two(const float2* p, float2& a, float2& b) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
__device__ __forceinline__ void ld_two(const double2* p, double2& a, double2& b) {
  a = p[0];
  b = p[1];
}

// k_lu_inv64 on 2 x 2 tiles (1024 threads), two steps per barrier.  A step of that kernel is 57 instructions
// a warp on eight warps per scheduler and then a chain through shared memory and the barrier (28 us a
// block, 55% of it issuing).  Here the tile that holds the 2 x 2 pivot block eliminates in it before it
// publishes, and every thread forms the second pivot row's and column's entries that it needs itself:
// the same operations on every element, in the same order, as one step at a time.  25.9 us a block; the
// chain pivot - publish - barrier is now what the warps wait for (per panel, job of 30,720: 48.6 -> 46.1).
template <typename T, bool SYM>
__global__ void __launch_bounds__(TRI * TRI / 4) k_lu_inv64_pair(T* A, int64_t lda, int64_t j0, int kb, int* info, T* inv) {
  constexpr bool sym = SYM;
  constexpr int TR = 2, TC = 2, NT = TRI * TRI / 4, LD = TRI + 1;
  extern __shared__ unsigned char smraw[];
  T* Ls = reinterpret_cast<T*>(smraw);  // 64 x LD: staging, then the L factor, then Linv
  __shared__ __align__(16) T p1[2][2][TRI], p2[2][2][SYM ? 2 : TRI], lc[2][TRI][2], dv[2][4];  // dv: d0, d1, l10, u01
  __shared__ int s_zero[2];  // 1-based column of a zero pivot, by parity of the pair of steps
  asm volatile("griddepcontrol.launch_dependents;");
  const int tid = threadIdx.x, rb = tid >> 5, cb = tid & 31;
  const int r0 = TR * rb, c0 = TC * cb;
  const T zero = cmk<T>(0.0, 0.0), one = cmk<T>(1.0, 0.0);
  for (int e = tid; e < TRI * TRI; e += NT) {
    const int r = e & (TRI - 1), c = e >> 6;
    const int rr = (sym && c > r) ? c : r, cc = (sym && c > r) ? r : c;
    Ls[r * LD + c] = (r < kb && c < kb) ? A[(j0 + rr) + (j0 + cc) * lda] : (r == c ? one : zero);
  }
  if (tid < 2) s_zero[tid] = 0;
  __syncthreads();
  T s1[TR][TC], s2[TR][TC];
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      s1[i][j] = Ls[(r0 + i) * LD + c0 + j];
      s2[i][j] = (r0 + i == c0 + j) ? one : zero;
    }
  // rows and columns 2 kq, 2 kq + 1 of S1 (the column of the first pivot as the second row has it after the
  // first step), the pivots' reciprocals and the block's multiplier
  auto publish = [&](int b, int kq) {
    if (rb == kq) {
      if (cb == kq) {
        T d0 = zero, d1 = zero;
        const bool ok = crecip(s1[0][0], d0);
        const T l = cmulx(s1[1][0], d0);
        T piv = s1[1][1];
        cfms(piv, l, s1[0][1]);
        if (!ok)
          s_zero[b] = 2 * kq + 1;
        else if (!crecip(piv, d1))
          s_zero[b] = 2 * kq + 2;
        dv[b][0] = d0;
        dv[b][1] = d1;
        dv[b][2] = l;
        dv[b][3] = s1[0][1];
        T nl;
        nl.x = -l.x;
        nl.y = -l.y;
        p1[b][0][c0] = zero;
        p1[b][1][c0] = nl;
      } else {
        p1[b][0][c0] = s1[0][0];
        p1[b][1][c0] = s1[1][0];
      }
      p1[b][0][c0 + 1] = s1[0][1];
      p1[b][1][c0 + 1] = s1[1][1];
      if constexpr (!SYM)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) p2[b][i][c0 + j] = s2[i][j];
    } else if (cb == kq) {
#pragma unroll
      for (int i = 0; i < TR; ++i) {
        lc[b][r0 + i][0] = s1[i][0];
        lc[b][r0 + i][1] = s1[i][1];
      }
    }
  };
  publish(0, 0);
  __syncthreads();  // the staging buffer is free from here on (L factor)
#pragma unroll 1
  for (int kq = 0; kq < TRI / 2; ++kq) {
    const int b = kq & 1, k = 2 * kq;
    if (s_zero[b]) {  // uniform
      if (tid == 0) atomicCAS(info, 0, (int)(j0 + s_zero[b]));
      return;
    }
    if (rb >= kq) {
      T d0, d1, l10, u01, q0[TC], q1[TC], x0[TC], x1[TC];
      ld_two(&dv[b][0], d0, d1);
      ld_two(&dv[b][2], l10, u01);
      ld_two(&p1[b][0][c0], q0[0], q0[1]);
      ld_two(&p1[b][1][c0], q1[0], q1[1]);
      if constexpr (!SYM) {
        ld_two(&p2[b][0][c0], x0[0], x0[1]);
        ld_two(&p2[b][1][c0], x1[0], x1[1]);
      }
      const T m01 = cmulx(u01, d0);  // the multiplier of X's row k + 1
      if (rb == kq) {  // row k + 1: the first step
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          cfms(s1[1][j], l10, q0[j]);
          if constexpr (!SYM) {
            cfms(s2[1][j], m01, x0[j]);
            s2[0][j] = cmulx(s2[0][j], d0);
            s2[1][j] = cmulx(s2[1][j], d1);
          }
        }
        if (cb == kq) {
          s1[1][0].x = -l10.x;
          s1[1][0].y = -l10.y;
          Ls[(k + 1) * LD + k] = l10;
        }
      } else {
        // the second pivot row after the first step (its entry at column k is there already, at k + 1 none)
#pragma unroll
        for (int j = 0; j < TC; ++j) {
          cfms(q1[j], l10, q0[j]);
          if constexpr (!SYM) cfms(x1[j], m01, x0[j]);
        }
        if (cb == kq) q1[1] = zero;
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          T a0, a1;
          ld_two(&lc[b][r0 + i][0], a0, a1);
          const T l0 = cmulx(a0, d0);
          cfms(a1, l0, u01);
          const T l1 = cmulx(a1, d1);
#pragma unroll
          for (int j = 0; j < TC; ++j) cfms(s1[i][j], l0, q0[j]);
          if (cb == kq) {
            s1[i][0].x = -l0.x;
            s1[i][0].y = -l0.y;
          }
#pragma unroll
          for (int j = 0; j < TC; ++j) cfms(s1[i][j], l1, q1[j]);
          if (cb == kq) {
            s1[i][1].x = -l1.x;
            s1[i][1].y = -l1.y;
            Ls[(r0 + i) * LD + k] = l0;
            Ls[(r0 + i) * LD + k + 1] = l1;
          }
          if constexpr (!SYM) {
            const T u0 = p1[b][0][r0 + i];
            T u1 = p1[b][1][r0 + i];
            cfms(u1, l10, u0);
            const T m0 = cmulx(u0, d0), m1 = cmulx(u1, d1);
#pragma unroll
            for (int j = 0; j < TC; ++j) {
              cfms(s2[i][j], m0, x0[j]);
              cfms(s2[i][j], m1, x1[j]);
            }
          }
        }
      }
      if (kq + 1 < TRI / 2) publish(b ^ 1, kq + 1);
    }
    __syncthreads();
  }
  // U (upper part of S1) joins the L factor in Ls; the factored block goes back to A
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j)
      if (c0 + j >= r0 + i) Ls[(r0 + i) * LD + c0 + j] = s1[i][j];
  __syncthreads();
  for (int e = tid; e < kb * kb; e += NT) {
    const int r = e % kb, c = e / kb;
    A[(j0 + r) + (j0 + c) * lda] = Ls[r * LD + c];
  }
  __syncthreads();
  // Linv (column-major, inv[c * 64 + r] = Linv[r][c]) through Ls; Uinv = X^T, so row r of X
  // is column r of Uinv (inv[4096 + r * 64 + c] = X[r][c]), written by the tile owners;
  // symmetric: X[r][c] = Linv[r][c] / d_r
  if (SYM) {
    __shared__ T s_dinv[TRI];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j)
        if (c0 + j == r0 + i) {  // the tile holding the pivot of row r0 + i
          T di;
          crecip(s1[i][j], di);  // nonzero: the elimination checked every pivot
          s_dinv[r0 + i] = di;
        }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      const T di = s_dinv[r0 + i];
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        const int r = r0 + i, c = c0 + j;
        s2[i][j] = c < r ? cmulx(s1[i][j], di) : (c == r ? di : zero);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) {
      const int r = r0 + i, c = c0 + j;
      Ls[r * LD + c] = c < r ? s1[i][j] : (c == r ? one : zero);
      inv[TRI * TRI + r * TRI + c] = s2[i][j];
    }
  __syncthreads();
  for (int e = tid; e < TRI * TRI; e += NT) {
    const int r = e & (TRI - 1), c = e >> 6;
    inv[e] = Ls[r * LD + c];
  }
}

// ---- blocked triangular solves on 64-wide triangles ---------------------------------------
// Both TRSMs of the LU are batches of independent triangular systems of order kb <= 64 that
// share one triangle of the factored diagonal block at (j0, j0):
//   left  (U12 = L11^{-1} A12): one system per column of A12, unit lower L11;
//   right (unpivoted path, L21 = A21 U11^{-1}): one system per row of A21, upper U11.
// A CTA stages NS systems (coalesced global loads) as X[k][s] in shared memory and the
// triangle as M[k][c] = coefficient of x_k in equation c (k < c).  LPS neighbouring lanes
// share a system and substitute in blocks of 16 unknowns, lane j owning UPL = 16 / LPS unknowns
// of each block from UPL j on:
//   x_c = (a_c - sum_{k<c} M[k][c] x_k) * d_c     (d_c = 1 or 1/U_cc);
// the terms of earlier blocks are split over the lanes, and inside a block each solved
// unknown is passed to the other lanes by a shuffle.
// Complex FP64: 16 systems per CTA and eight lanes per system.  A warp's 2500 FP64 instructions on eight
// systems of four lanes, one every 64 cycles, set the kernel's 160 us whatever the number of systems;
// half of that on four times the warps takes 41 us for a few hundred systems.
template <typename T>
struct TrsmTile {
  static constexpr int LPS = sizeof(T) == 8 ? 4 : 8;     // lanes per system
  static constexpr int UPL = 16 / LPS;                   // unknowns of a block of 16 per lane
  static constexpr int NS = sizeof(T) == 8 ? 64 : 16;    // systems per CTA
  static constexpr int NT = LPS * NS;                    // threads per CTA
  static constexpr int MLD = sizeof(T) == 8 ? 66 : 65;   // row stride of M
};

template <typename T>
size_t trsm_tile_smem() {
  return ((size_t)TRI * TrsmTile<T>::MLD + TRI + (size_t)TRI * (TrsmTile<T>::NS + 1)) * sizeof(T);
}

template <typename T, typename RT, bool RIGHT>
__global__ void __launch_bounds__(TrsmTile<T>::NT) k_trsm_tile(T* A, int64_t lda, int64_t j0, int kb,
                                                               int64_t s0, int64_t s1) {
  constexpr int NS = TrsmTile<T>::NS, NT = TrsmTile<T>::NT, MLD = TrsmTile<T>::MLD, LDX = NS + 1;
  constexpr int LPS = TrsmTile<T>::LPS, UPL = TrsmTile<T>::UPL;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* M = reinterpret_cast<T*>(smraw);  // TRI x MLD
  T* dinv = M + TRI * MLD;             // TRI
  T* X = dinv + TRI;                   // TRI x LDX
  const int tid = threadIdx.x;
  const int64_t sb = s0 + (int64_t)blockIdx.x * NS;  // first system of this CTA
  const T zero = {0, 0};

  // the triangle (zero outside kb x kb and on/below the diagonal of M) and the systems X[k][s]; each
  // thread issues up to 16 loads before their stores
  constexpr int LB = 16, NX = TRI * NS / NT;
  static_assert(TRI * TRI % (LB * NT) == 0 && NX * NT == TRI * NS, "staging");
#pragma unroll 1
  for (int e0 = 0; e0 < TRI * TRI; e0 += LB * NT) {
    T v[LB];
#pragma unroll
    for (int j = 0; j < LB; ++j) {
      const int e = e0 + tid + NT * j;
      const int r = e % TRI, k = e / TRI;  // global element (j0 + r, j0 + k), coalesced along r
      v[j] = (r < kb && k < kb) ? A[(j0 + r) + (j0 + k) * lda] : zero;
    }
#pragma unroll
    for (int j = 0; j < LB; ++j) {
      const int e = e0 + tid + NT * j;
      const int r = e % TRI, k = e / TRI;
      if (RIGHT) {
        M[r * MLD + k] = r < k ? v[j] : zero;  // U[r][k]: coefficient of x_r in equation k
        if (r == k) {
          T d = zero;
          if (r < kb) {
            const RT den = v[j].x * v[j].x + v[j].y * v[j].y;
            d.x = v[j].x / den;
            d.y = -v[j].y / den;
          }
          dinv[r] = d;
        }
      } else {
        M[k * MLD + r] = r > k ? v[j] : zero;  // L[r][k]: coefficient of x_k in equation r
      }
    }
  }
  {
    T v[NX];
#pragma unroll
    for (int j = 0; j < NX; ++j) {
      const int e = tid + NT * j;
      if (RIGHT) {
        const int s = e % NS, k = e / NS;  // row sb + s, column j0 + k: coalesced along s
        v[j] = (k < kb && sb + s < s1) ? A[(sb + s) + (j0 + k) * lda] : zero;
      } else {
        const int k = e % TRI, s = e / TRI;  // row j0 + k, column sb + s: coalesced along k
        v[j] = (k < kb && sb + s < s1) ? A[(j0 + k) + (sb + s) * lda] : zero;
      }
    }
#pragma unroll
    for (int j = 0; j < NX; ++j) {
      const int e = tid + NT * j;
      if (RIGHT)
        X[(e / NS) * LDX + e % NS] = v[j];
      else
        X[(e % TRI) * LDX + e / TRI] = v[j];
    }
  }
  __syncthreads();

  // substitution: lanes LPS s .. LPS s + LPS - 1 own system s, lane j of them unknowns
  // UPL j .. UPL j + UPL - 1 of each block of 16
  const int s = tid / LPS, j = tid % LPS, qbase = (tid & 31) & ~(LPS - 1);
  T* x = X + s;
  const int nblk = (kb + 15) / 16;
  for (int B = 0; B < nblk; ++B) {
    const int c0 = 16 * B, cj = c0 + UPL * j;
    T acc[UPL];
#pragma unroll
    for (int i = 0; i < UPL; ++i) acc[i] = x[(cj + i) * LDX];
    // c0 is a multiple of 16: four earlier unknowns per pass, their loads issued together
    for (int k = 0; k < c0; k += 4) {
      T xk[4], mk[4][UPL];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        xk[u] = x[(k + u) * LDX];
#pragma unroll
        for (int i = 0; i < UPL; ++i) mk[u][i] = M[(k + u) * MLD + cj + i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < UPL; ++i) cfms(acc[i], mk[u][i], xk[u]);
    }
#pragma unroll
    for (int cc = 0; cc < 16; ++cc) {
      const int jo = cc / UPL, io = cc % UPL;
      if (RIGHT && j == jo) {
        const T d = dinv[c0 + cc];
        acc[io] = cmulx(acc[io], d);
      }
      const T xc = shfl_c(acc[io], qbase + jo);  // the solved unknown c0 + cc
      if (j == jo) x[(c0 + cc) * LDX] = xc;
#pragma unroll
      for (int i = 0; i < UPL; ++i)
        if (UPL * j + i > cc) cfms(acc[i], M[(c0 + cc) * MLD + cj + i], xc);
    }
  }
  __syncthreads();

  // write the solved systems back
  for (int m0 = 0; m0 < TRI * NS / NT; ++m0) {
    const int e = tid + NT * m0;
    if (RIGHT) {
      const int s2 = e % NS, k = e / NS;
      if (k < kb && sb + s2 < s1) A[(sb + s2) + (j0 + k) * lda] = X[k * LDX + s2];
    } else {
      const int k = e % TRI, s2 = e / TRI;
      if (k < kb && sb + s2 < s1) A[(j0 + k) + (sb + s2) * lda] = X[k * LDX + s2];
    }
  }
}

// ---- unpivoted c64 panel: both triangular solves as products with the inverses ----------
// After k_lu_inv64 (kb = 64, inverses in inv: Linv then Uinv, column-major 64 x 64), with
// s0 = j0 + 64:
//   CTA b <  nR:  L21 rows s0 + 64 b .. +63:          X = A21 Uinv  (a system per row)
//   CTA b >= nR:  U12 columns s0 + 64 (b - nR) .. +63: X = Linv A12  (a system per column)
// Both are C[x][y] = sum_k W[k][s] N[k][v] over 64 x 64 x 64: s runs over the 64 systems
// (W: A21 / A12), v over the inverse's free index (N: Uinv / Linv), and N[k][v] = 0 for
// k > v (the triangle).  A complex multiply-add is two packed FP32 FMAs,
//   acc += (a.x, a.x) (b.x, b.y) + (-a.y, a.y) (b.y, b.x),
// so W is staged as float4 (a.x, a.x, -a.y, a.y) and N as float4 (b.x, b.y, b.y, b.x): one
// 16-byte load per operand and no register shuffling.  K is staged in two halves of 32.
// A thread owns 4 systems (lanes 0..15 of a half-warp at stride 16) times 4 free indices,
// dealt out so that every warp does the same work: warp w takes 4w .. 4w+3 and
// 60-4w .. 63-4w (half-warp h the pairs at +2h), all four up to k = 4w+4, the upper two up
// to 64-4w -- 544 complex multiply-adds per thread in every warp.  The result is staged
// system-major in shared memory, stored coalesced and, when the tensor-core update follows
// (Ap / Bp not null), written once more as its FP16 operands with 16-byte stores: L21 rows
// expanded and row-scaled as A', U12 columns scaled as B' (layout and scale rule of the
// update's own operand preparation).
constexpr int PA_KH = 32;   // k per staged half
constexpr int PA_LD4 = 65;  // staged operand rows: 64 float4 + 1
constexpr int PA_CLD = 65;  // staged result columns
size_t panel_apply_smem() { return (size_t)2 * PA_KH * PA_LD4 * sizeof(float4) + 4 * 64 * sizeof(float); }

__device__ __forceinline__ void cmac2(float2& acc, float4 a, float4 b) {
  acc = __ffma2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y), acc);
  acc = __ffma2_rn(make_float2(a.z, a.w), make_float2(b.z, b.w), acc);
}

// Symmetric factorisation (nB >= 0; launched with nR CTAs, right side only): U12 = D L21^T
// is not stored; its FP16 B' columns for the first nB systems (the rest of the mid block)
// are written from L21 and the pivots D = diag(U11) instead.
// rb0: index of the first CTA's block (the grid covers blocks rb0 .. of the 2 nR, or nR)
template <int NS>
__global__ void __launch_bounds__(256, NS == 64 ? 2 : 3) k_panel_apply(float2* A, int64_t lda, int64_t j0, int64_t n,
                                                        const float2* inv, int nR, __half2* Ap,
                                                        float* inv_sa, __half2* Bp, float* inv_sb, int nB,
                                                        int rb0) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float4* Ws = reinterpret_cast<float4*>(smraw);  // W[k][s], k of the current half
  float4* Ns = Ws + PA_KH * PA_LD4;               // N[k][v]
  float* red = reinterpret_cast<float*>(Ns + PA_KH * PA_LD4);  // 4 x 64 partial maxima
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bi = (int)blockIdx.x + rb0;
  const bool right = bi < nR;
  const int64_t s0 = j0 + TRI;
  const int64_t b0 = s0 + (int64_t)(right ? bi : bi - nR) * NS;  // first system
  constexpr int NU = NS / 16;         // systems per thread
  constexpr int QN = 256 / NS;        // threads per system in the maxima passes
  constexpr int QV = TRI / QN;        // free indices per such thread
  const float2 zero = make_float2(0.f, 0.f);
  const int sl = lane & 15, h = lane >> 4;
  const int vlo = 4 * warp + 2 * h, vhi = 60 - 4 * warp + 2 * h;  // free indices vlo, vlo+1, vhi, vhi+1
  const int k1 = 4 * warp + 4, k2 = 64 - 4 * warp;
  float2 acc[NU][4];  // [system u][free index: vlo, vlo+1, vhi, vhi+1]
#pragma unroll
  for (int u = 0; u < NU; ++u)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[u][j] = zero;

  for (int kh = 0; kh < 2; ++kh) {
    const int kb0 = kh * PA_KH;
    if (kh) __syncthreads();  // the first half is consumed
    {
      // 8 + 8 elements per thread, e = tid + 256 t; coalesced along the contiguous index:
      //   right W: s = e & 63, k = e >> 6 (A21 column k)   N: k = e & 31, v = e >> 5 (Uinv column v)
      //   left  W: k = e & 31, s = e >> 5 (A12 column s)   N: v = e & 63, k = e >> 6 (Linv column k)
      constexpr int TW = NS * PA_KH / 256;  // W elements per thread (N: 8)
      float2 w[TW], v[8];
#pragma unroll
      for (int t = 0; t < TW; ++t) {
        const int e = tid + 256 * t;
        if (right) {
          const int s = e % NS, k = e / NS;
          w[t] = b0 + s < n ? A[(b0 + s) + (j0 + kb0 + k) * lda] : zero;
        } else {
          const int k = e & 31, s = e >> 5;
          w[t] = b0 + s < n ? A[(j0 + kb0 + k) + (b0 + s) * lda] : zero;
        }
      }
      // launched as a programmatic dependent of the diagonal block's elimination: the rows of
      // A21 / A12 above are final already, the inverses (and the pivots below) only after this
      // wait (a no-op for an ordinary launch); `inv` is not declared __restrict__ and is read
      // through L2, so that no load of it is scheduled or served from before the wait
      if (kh == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int e = tid + 256 * t;
        v[t] = __ldcg(right ? inv + 4096 + (e >> 5) * 64 + kb0 + (e & 31) : inv + (kb0 + (e >> 6)) * 64 + (e & 63));
      }
#pragma unroll
      for (int t = 0; t < TW; ++t) {
        const int e = tid + 256 * t;
        const float4 wv = make_float4(w[t].x, w[t].x, -w[t].y, w[t].y);
        if (right)
          Ws[(e / NS) * PA_LD4 + (e % NS)] = wv;
        else
          Ws[(e & 31) * PA_LD4 + (e >> 5)] = wv;
      }
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int e = tid + 256 * t;
        const float4 nv = make_float4(v[t].x, v[t].y, v[t].y, v[t].x);
        if (right)
          Ns[(e & 31) * PA_LD4 + (e >> 5)] = nv;
        else
          Ns[(e >> 6) * PA_LD4 + (e & 63)] = nv;
      }
    }
    __syncthreads();
    // all four free indices for k < k1 (inside the first half), the upper two for k < k2
    const int e1 = kh == 0 ? k1 : kb0, e2 = min(k2, kb0 + PA_KH);
#pragma unroll 2
    for (int k = kb0; k < e1; ++k) {
      const float4* wr = Ws + (k - kb0) * PA_LD4 + sl;
      const float4* nr = Ns + (k - kb0) * PA_LD4;
      const float4 n0 = nr[vlo], n1 = nr[vlo + 1], n2 = nr[vhi], n3 = nr[vhi + 1];
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const float4 a = wr[16 * u];
        cmac2(acc[u][0], a, n0);
        cmac2(acc[u][1], a, n1);
        cmac2(acc[u][2], a, n2);
        cmac2(acc[u][3], a, n3);
      }
    }
#pragma unroll 2
    for (int k = e1; k < e2; ++k) {
      const float4* wr = Ws + (k - kb0) * PA_LD4 + sl;
      const float4* nr = Ns + (k - kb0) * PA_LD4;
      const float4 n2 = nr[vhi], n3 = nr[vhi + 1];
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const float4 a = wr[16 * u];
        cmac2(acc[u][2], a, n2);
        cmac2(acc[u][3], a, n3);
      }
    }
  }
  __syncthreads();  // every warp is done with Ws / Ns
  // stage C system-major, Cs[s][v] (s: system, v: free index)
  float2* Cs = reinterpret_cast<float2*>(smraw);
  __shared__ float s_scale[64];
  const int vv[4] = {vlo, vlo + 1, vhi, vhi + 1};
#pragma unroll
  for (int u = 0; u < NU; ++u)
#pragma unroll
    for (int j = 0; j < 4; ++j) Cs[(sl + 16 * u) * PA_CLD + vv[j]] = acc[u][j];
  __syncthreads();
  // the solved systems, coalesced: right -- A[b0 + s, j0 + v] (along s); left -- A[j0 + v,
  // b0 + s] (along v)
#pragma unroll 4
  for (int t = 0; t < NS / 4; ++t) {
    const int e = tid + 256 * t;
    if (right) {
      const int sy = e % NS, v = e / NS;
      if (b0 + sy < n) A[(b0 + sy) + (j0 + v) * lda] = Cs[sy * PA_CLD + v];
    } else {
      const int v = e & 63, sy = e >> 6;
      if (b0 + sy < n) A[(j0 + v) + (b0 + sy) * lda] = Cs[sy * PA_CLD + v];
    }
  }
  // FP16 operands of the update: right -- the A' row pair of each system (2 x 64 half2);
  // left -- the B' column of each system (64 half2).  Scale: 2^sh from the system's largest
  // |re|, |im| (partial maxima over quarters of v, then one per system).
  __half2* const dst = right ? Ap : Bp;
  if (dst == nullptr) return;  // uniform over the CTA
  {
    const int sy = tid % NS, q = tid / NS;
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < QV; ++i) {
      const float2 a = Cs[sy * PA_CLD + QV * q + i];
      mx = fmaxf(mx, fmaxf(fabsf(a.x), fabsf(a.y)));
    }
    red[q * NS + sy] = mx;
    __syncthreads();
    if (q == 0) {
      for (int qq = 1; qq < QN; ++qq) mx = fmaxf(mx, red[qq * NS + sy]);
      const int sh = tc_scale_shift(mx);
      s_scale[sy] = ldexpf(1.f, sh);
      if (b0 + sy < n) (right ? inv_sa : inv_sb)[b0 + sy - s0] = ldexpf(1.f, -sh);
    }
    __syncthreads();
  }
  if (right && nB > (int)(b0 - s0)) {
    // symmetric: B' column of system s (< nB) = D (row s of L21), its own scale
    __shared__ float2 s_d[64];
    __shared__ float s_tsc[64];
    // the pivots are the elimination's output: through L2 (the rows of A21 read before the
    // wait may have brought a line of the diagonal block into L1 before it was written)
    if (tid < 64) s_d[tid] = __ldcg(A + (j0 + tid) + (j0 + tid) * lda);
    __syncthreads();
    const int sy = tid % NS, q = tid / NS;
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < QV; ++i) {
      const float2 a = cmulx(Cs[sy * PA_CLD + QV * q + i], s_d[QV * q + i]);
      mx = fmaxf(mx, fmaxf(fabsf(a.x), fabsf(a.y)));
    }
    red[q * NS + sy] = mx;
    __syncthreads();
    if (q == 0) {
      for (int qq = 1; qq < QN; ++qq) mx = fmaxf(mx, red[qq * NS + sy]);
      const int sh = tc_scale_shift(mx);
      s_tsc[sy] = ldexpf(1.f, sh);
      if (b0 + sy - s0 < nB) inv_sb[b0 + sy - s0] = ldexpf(1.f, -sh);
    }
    __syncthreads();
    const int v0 = 4 * (lane & 15);
    for (int sp = 2 * warp; sp < NS; sp += 16) {
      const int s2 = sp + (lane >> 4);
      if (b0 + s2 - s0 < nB) {
        const float sc = s_tsc[s2];
        const float2* cr = Cs + s2 * PA_CLD + v0;
        __half2 hv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = cmulx(cr[i], s_d[v0 + i]);
          hv[i] = __floats2half2_rn(a.x * sc, a.y * sc);
        }
        *reinterpret_cast<uint4*>(Bp + (b0 + s2 - s0) * TRI + v0) = *reinterpret_cast<const uint4*>(hv);
      }
    }
  }
  // 16-byte stores: a lane converts 4 consecutive v of one system; right -- one system per
  // warp pass (lanes 0..15 row 2m, 16..31 row 2m+1: 512 contiguous bytes), left -- two
  // systems per pass (256 bytes each)
  const int v0 = 4 * (lane & 15);
  if (right) {
    for (int sy = warp; sy < NS; sy += 8) {
      if (b0 + sy >= n) break;
      const float sc = s_scale[sy];
      const float2* cr = Cs + sy * PA_CLD + v0;
      __half2 hv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = cr[i];
        hv[i] = (lane < 16) ? __floats2half2_rn(a.x * sc, -a.y * sc) : __floats2half2_rn(a.y * sc, a.x * sc);
      }
      const int64_t m = b0 + sy - s0;
      *reinterpret_cast<uint4*>(Ap + (2 * m + (lane >> 4)) * TRI + v0) = *reinterpret_cast<const uint4*>(hv);
    }
  } else {
    for (int sp = 2 * warp; sp < NS; sp += 16) {
      const int sy = sp + (lane >> 4);
      if (b0 + sy < n) {
        const float sc = s_scale[sy];
        const float2* cr = Cs + sy * PA_CLD + v0;
        __half2 hv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = cr[i];
          hv[i] = __floats2half2_rn(a.x * sc, a.y * sc);
        }
        const int64_t m = b0 + sy - s0;
        *reinterpret_cast<uint4*>(Bp + m * TRI + v0) = *reinterpret_cast<const uint4*>(hv);
      }
    }
  }
}

// ---- symmetric factorisation helpers ---------------------------------------------------
// B (K x N, ld K) = D L^T with L = rows of the matrix (N x K at L, ld lda) and D the pivots on
// the diagonal at dg (stride lda + 1): the explicit operand of the CUDA-core fallback update
template <typename T>
__global__ void k_dlt(const T* L, const T* dg, int64_t lda, int K, int N, T* B) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= (int64_t)K * N) return;
  const int k = (int)(e % K), c = (int)(e / K);
  B[e] = cmulx(dg[(int64_t)k * (lda + 1)], L[c + (int64_t)k * lda]);
}

// U = D L^T above the 64 x 64 diagonal blocks: block (I, J), I < J, from the transposed block
// (J, I) of L and the pivots of rows 64 I..: U[i][j] = d_i L[j][i] (the diagonal blocks
// already hold U11 from k_lu_inv64)
// One CTA per block pair I < J (linear index J (J - 1) / 2 + I: no CTA on or below the diagonal).
template <typename T>
__global__ void __launch_bounds__(256) k_sym_upper(T* A, int64_t lda, int64_t n) {
  const int64_t L = blockIdx.x;
  int J = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)L)) * 0.5f);
  while ((int64_t)J * (J - 1) / 2 > L) --J;
  while ((int64_t)(J + 1) * J / 2 <= L) ++J;
  const int I = (int)(L - (int64_t)J * (J - 1) / 2);
  __shared__ T t[64][65];
  __shared__ T d[64];
  const int64_t r0 = 64 * (int64_t)I, c0 = 64 * (int64_t)J;
  const int tid = threadIdx.x;
  if (tid < 64) d[tid] = r0 + tid < n ? A[(r0 + tid) * (lda + 1)] : T{0, 0};
  for (int e = tid; e < 64 * 64; e += 256) {
    const int j = e & 63, i = e >> 6;  // L[c0 + j][r0 + i], coalesced along j
    t[i][j] = (c0 + j < n && r0 + i < n) ? A[(c0 + j) + (r0 + i) * lda] : T{0, 0};
  }
  __syncthreads();
  for (int e = tid; e < 64 * 64; e += 256) {
    const int i = e & 63, j = e >> 6;  // U[r0 + i][c0 + j], coalesced along i
    if (r0 + i < n && c0 + j < n) A[(r0 + i) + (c0 + j) * lda] = cmulx(d[i], t[i][j]);
  }
}

// Lookahead of the symmetric factorisation: the diagonal block at p0 takes the previous
// panel's contribution just before its elimination, block -= L D L^T with L = A[p0.., p0-64..]
// (kb x 64, the block row the previous panel has just solved) and D that panel's pivots
// A[p0-64+k, p0-64+k].  Only the lower triangle with the diagonal (what the symmetric
// elimination reads), FP32 sums.  A thread owns a 4 x 4 tile; tiles above the diagonal idle.
constexpr int SDU_LD = 65;
size_t sym_diag_update_smem() { return (size_t)2 * 64 * SDU_LD * sizeof(float2); }
__global__ void __launch_bounds__(256) k_sym_diag_update(float2* A, int64_t lda, int64_t p0, int kb) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* Ls = reinterpret_cast<float2*>(smraw);  // Ls[k LD + r] = L[r][k]
  float2* Ds = Ls + 64 * SDU_LD;                  // Ds[k LD + c] = d_k L[c][k]
  const int tid = threadIdx.x;
  const int64_t q0 = p0 - 64;
  for (int e = tid; e < 64 * 64; e += 256) {
    const int r = e & 63, k = e >> 6;  // column k of L, coalesced along r
    const float2 l = r < kb ? A[(p0 + r) + (q0 + k) * lda] : make_float2(0.f, 0.f);
    Ls[k * SDU_LD + r] = l;
    Ds[k * SDU_LD + r] = cmulx(A[(q0 + k) * (lda + 1)], l);
  }
  __syncthreads();
  const int tr = tid >> 4, tc = tid & 15;
  if (tc > tr) return;
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < 64; ++k) {
    float2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = Ls[k * SDU_LD + 4 * tr + i];
      b[i] = Ds[k * SDU_LD + 4 * tc + i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) cfma(acc[i][j], a[i], b[j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = 4 * tr + i, c = 4 * tc + j;
      if (r >= c && r < kb) {
        float2& x = A[(p0 + r) + (p0 + c) * lda];
        x = make_float2(x.x - acc[i][j].x, x.y - acc[i][j].y);
      }
    }
}

// sampled asymmetry: sums of |a_ij - a_ji|^2 and |a_ij|^2 + |a_ji|^2 over rows i = s p, columns
// j = s q < i (FP64 sums, atomically added)
template <typename T>
__global__ void k_asym_sample(const T* A, int64_t lda, int64_t n, int64_t s, double* out) {
  const int64_t np = (n + s - 1) / s;
  double dsum = 0, nsum = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < np * np; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = (e % np) * s, j = (e / np) * s;
    if (j >= i) continue;
    const T a = A[i + j * lda], b = A[j + i * lda];
    const double dr = (double)a.x - (double)b.x, di = (double)a.y - (double)b.y;
    dsum += dr * dr + di * di;
    nsum += (double)a.x * a.x + (double)a.y * a.y + (double)b.x * b.x + (double)b.y * b.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
    nsum += __shfl_xor_sync(0xffffffffu, nsum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, dsum);
    atomicAdd(out + 1, nsum);
  }
}

// copy of the block-lower part of a c64 matrix: column j from row 64 floor(j / 64) down (what
// the symmetric factorisation reads; the rest of the copy is written at its end).  Two rows
// per thread (16-byte accesses when lda and ldf are even and the bases 16-byte aligned).
__global__ void __launch_bounds__(256) k_copy_lower_c64(int64_t n, const float2* A, int64_t lda, float2* F,
                                                       int64_t ldf, int vec) {
  // a CTA per column, two elements per thread and step (one 16-byte access when aligned)
  for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
    const float2* a = A + j * lda;
    float2* f = F + j * ldf;
    for (int64_t i = (j / 64) * 64 + 2 * threadIdx.x; i < n; i += 2 * 256) {
      if (vec && i + 1 < n) {
        *reinterpret_cast<float4*>(f + i) = __ldcs(reinterpret_cast<const float4*>(a + i));
      } else {
        f[i] = a[i];
        if (i + 1 < n) f[i + 1] = a[i + 1];
      }
    }
  }
}

// the same block-lower part from a c128 matrix, rounded to c64 by integer operations: a CTA
// per column (its rows from the first row of the column's diagonal block on), four streaming
// loads in flight per thread -- no CTA of the grid falls wholly above the diagonal
__global__ void __launch_bounds__(256) k_convert_lower_c128(int64_t n, const double2* A, int64_t lda, float2* F,
                                                           int64_t ldf) {
  auto cvt = [](double2 a) { return make_float2(fsplit::to_float_rn(a.x), fsplit::to_float_rn(a.y)); };
  for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
    const double2* a = A + j * lda;
    float2* f = F + j * ldf;
    int64_t i = (j / 64) * 64 + threadIdx.x;
    for (; i + 3 * 256 < n; i += 4 * 256) {
      double2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldcs(a + i + u * 256);
#pragma unroll
      for (int u = 0; u < 4; ++u) f[i + u * 256] = cvt(v[u]);
    }
    for (; i < n; i += 256) f[i] = cvt(__ldcs(a + i));
  }
}

// ---- C -= A B  (complex; C m x n, A m x k, B k x n; all column-major with ld) -------------
constexpr int GT = 64, GK = 8;
// the GT x GT tile at (bm, bn), by a CTA of 256 threads
template <typename T, typename R>
__device__ __forceinline__ void gemm_tile(T* C, int64_t ldc, const T* Am, int64_t lda, const T* Bm, int64_t ldb, int64_t m,
                                          int64_t n, int k, int64_t bm, int64_t bn) {
  __shared__ R As[2][GK][GT + 1];
  __shared__ R Bs[2][GK][GT + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  R cr[4][4], ci[4][4];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) cr[i][j] = ci[i][j] = 0;
  for (int k0 = 0; k0 < k; k0 += GK) {
    // load A tile GT x GK and B tile GK x GT (256 threads, 2 elements each)
    for (int e = threadIdx.x; e < GT * GK; e += 256) {
      int r = e % GT, c = e / GT;
      int64_t gr = bm + r;
      int gc = k0 + c;
      T a = (gr < m && gc < k) ? Am[gr + gc * lda] : cmk<T>(0, 0);
      As[0][c][r] = a.x;
      As[1][c][r] = a.y;
      int rb = e % GK, cb = e / GK;
      int64_t gcol = bn + cb;
      int grow = k0 + rb;
      T b = (gcol < n && grow < k) ? Bm[grow + gcol * ldb] : cmk<T>(0, 0);
      Bs[0][rb][cb] = b.x;
      Bs[1][rb][cb] = b.y;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      R ar[4], ai[4], br[4], bi[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ar[i] = As[0][kk][tx + 16 * i];
        ai[i] = As[1][kk][tx + 16 * i];
        br[i] = Bs[0][kk][ty + 16 * i];
        bi[i] = Bs[1][kk][ty + 16 * i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          cr[i][j] += ar[i] * br[j] - ai[i] * bi[j];
          ci[i][j] += ar[i] * bi[j] + ai[i] * br[j];
        }
    }
    __syncthreads();
  }
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      int64_t r = bm + tx + 16 * i, c = bn + ty + 16 * j;
      if (r < m && c < n) {
        T v = C[r + c * ldc];
        C[r + c * ldc] = cmk<T>(v.x - cr[i][j], v.y - ci[i][j]);
      }
    }
}
template <typename T, typename R>
__global__ void __launch_bounds__(256) k_gemm_sub(T* C, int64_t ldc, const T* Am, int64_t lda, const T* Bm, int64_t ldb,
                                                  int64_t m, int64_t n, int k) {
  gemm_tile<T, R>(C, ldc, Am, lda, Bm, ldb, m, n, k, blockIdx.x * (int64_t)GT, blockIdx.y * (int64_t)GT);
}
// the GT x GT tiles that tc_gemm64.cu leaves to the FP64 units, by (row, column) index
__global__ void __launch_bounds__(256) k_gemm_tiles(const int2* list, const int* count, double2* C, int64_t ldc,
                                                    const double2* Am, int64_t lda, const double2* Bm, int64_t ldb,
                                                    int64_t m, int64_t n, int k) {
  const int items = *count;
  for (int i = blockIdx.x; i < items; i += gridDim.x)
    gemm_tile<double2, double>(C, ldc, Am, lda, Bm, ldb, m, n, k, list[i].x * (int64_t)GT, list[i].y * (int64_t)GT);
}

// ---- triangular solves on one right-hand side ------------------------------------------
// diagonal block solve by one CTA (rows [k0, k0+kb)); lower=1: unit lower, forward;
// lower=0: upper, backward
template <typename T>
__global__ void k_trsv_block(const T* A, int64_t lda, T* b, int64_t k0, int kb, int lower) {
  extern __shared__ unsigned char smraw[];
  T* D = reinterpret_cast<T*>(smraw);  // kb x kb diagonal block, column-major
  __shared__ double xr[128], xi[128];
  for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
    int r = e % kb, c = e / kb;
    D[e] = A[(k0 + r) + (k0 + c) * lda];
  }
  for (int i = threadIdx.x; i < kb; i += blockDim.x) {
    xr[i] = b[k0 + i].x;
    xi[i] = b[k0 + i].y;
  }
  __syncthreads();
  if (lower) {
    for (int k = 0; k < kb; ++k) {
      double vr = xr[k], vi = xi[k];
      for (int i = k + 1 + threadIdx.x; i < kb; i += blockDim.x) {
        T l = D[i + k * kb];
        xr[i] -= l.x * vr - l.y * vi;
        xi[i] -= l.x * vi + l.y * vr;
      }
      __syncthreads();
    }
  } else {
    for (int k = kb - 1; k >= 0; --k) {
      if (threadIdx.x == 0) {
        T d = D[k + k * kb];
        double den = (double)d.x * d.x + (double)d.y * d.y;
        double r = (xr[k] * d.x + xi[k] * d.y) / den, im = (xi[k] * d.x - xr[k] * d.y) / den;
        xr[k] = r;
        xi[k] = im;
      }
      __syncthreads();
      double vr = xr[k], vi = xi[k];
      for (int i = threadIdx.x; i < k; i += blockDim.x) {
        T u = D[i + k * kb];
        xr[i] -= u.x * vr - u.y * vi;
        xi[i] -= u.x * vi + u.y * vr;
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < kb; i += blockDim.x) b[k0 + i] = cmk<T>(xr[i], xi[i]);
}

// b[rows] -= A[rows, k0:k0+kb] x[k0:k0+kb]  for rows in [r0, r1)
template <typename T>
__global__ void k_trsv_update(const T* A, int64_t lda, T* b, int64_t k0, int kb, int64_t r0,
                              int64_t r1) {
  int64_t i = r0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= r1) return;
  double sr = 0, si = 0;
  for (int k = 0; k < kb; ++k) {
    T a = A[i + (k0 + k) * lda];
    T x = b[k0 + k];
    sr += (double)a.x * x.x - (double)a.y * x.y;
    si += (double)a.x * x.y + (double)a.y * x.x;
  }
  T v = b[i];
  b[i] = cmk<T>(v.x - sr, v.y - si);
}

// ---- inverses of the 64 x 64 diagonal blocks of L (unit lower) and U (upper) ----------
// dinv + b * 2 * 4096: Linv_b then Uinv_b, column-major 64 x 64 (identity beyond rb)
template <typename T, typename RT>
__global__ void k_invert_diag(const T* A, int64_t lda, int64_t n, T* dinv) {
  extern __shared__ unsigned char smraw[];
  T* D = reinterpret_cast<T*>(smraw);   // 64 x 65 row-major
  T* X = D + 64 * 65;                   // 64 columns x 65 (column j of the inverse)
  const int b = blockIdx.x;
  const int64_t r0 = (int64_t)b * 64;
  const int rb = (int)(n - r0 < 64 ? n - r0 : 64);
  for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) {
    int i = e % 64, c = e / 64;
    T v;
    v.x = (RT)(i == c ? 1 : 0);
    v.y = 0;
    if (i < rb && c < rb) v = A[(r0 + i) + (r0 + c) * lda];
    D[i * 65 + c] = v;
  }
  __syncthreads();
  const int j = threadIdx.x;  // one column of each inverse per thread
  T* x = X + j * 65;
  T* Lout = dinv + (int64_t)b * 2 * 4096;
  T* Uout = Lout + 4096;
  // L x = e_j (unit lower)
  for (int i = 0; i < 64; ++i) {
    T v;
    v.x = (RT)(i == j ? 1 : 0);
    v.y = 0;
    if (i > j)
      for (int m = j; m < i; ++m) {
        T l = D[i * 65 + m], xm = x[m];
        v.x -= l.x * xm.x - l.y * xm.y;
        v.y -= l.x * xm.y + l.y * xm.x;
      }
    x[i] = v;
  }
  for (int i = 0; i < 64; ++i) Lout[j * 64 + i] = x[i];
  // U x = e_j (upper)
  for (int i = 63; i >= 0; --i) {
    T v;
    v.x = (RT)(i == j ? 1 : 0);
    v.y = 0;
    if (i < j)
      for (int m = i + 1; m <= j; ++m) {
        T u = D[i * 65 + m], xm = x[m];
        v.x -= u.x * xm.x - u.y * xm.y;
        v.y -= u.x * xm.y + u.y * xm.x;
      }
    if (i > j) {
      v.x = 0;
      v.y = 0;
    } else {
      T d = D[i * 65 + i];
      RT den = d.x * d.x + d.y * d.y;
      T q;
      q.x = (v.x * d.x + v.y * d.y) / den;
      q.y = (v.y * d.x - v.x * d.y) / den;
      if constexpr (sizeof(T) == 16)
        if (!square_in_range(den) && (d.x != 0 || d.y != 0)) q = cmulx(v, recip_scaled(d));
      v = q;
    }
    x[i] = v;
  }
  for (int i = 0; i < 64; ++i) Uout[j * 64 + i] = x[i];
}

// ---- triangular solve on one right-hand side as a wavefront ------------------------------
// Block rows of 64 are owned round-robin by co-resident CTAs (cooperative launch).  The
// solution is written to `out`, which starts filled with a sentinel (a NaN bit pattern that
// arithmetic does not produce), so a solved value is its own "ready" flag: a thread that
// needs block k spins (bounded) on exactly the 16 values it multiplies, with no counter, no
// fence and no block barrier inside the dependency walk.  The factor block of the next
// dependency and the thread's slice of the diagonal block's inverse are loaded ahead.  After
// the walk the CTA solves its diagonal block (inverse matvec) and stores its 64 values.
// lower = 1: unit lower, forward; lower = 0: upper, backward.  rhs: the right-hand side
// (read only).  Arithmetic in RT.  A wait that runs out sets status bit 8 and uses zeros.
// Several right-hand sides run side by side, per_rhs CTAs each (their chains of blocks do not
// depend on one another, and one chain leaves most of every SM idle): three at order 6007 in complex
// FP64 take as long as one.  A block row's sum has the same order whatever the number of CTAs.
constexpr unsigned long long SENT32 = 0x7FC0DEAD7FC0DEADull;  // two FP32 NaNs, payload 0xDEAD
constexpr unsigned long long SENT64 = 0x7FF8DEADBEEF0001ull;  // one FP64 NaN with a payload
constexpr long long TRSV_SPIN_MAX = 1LL << 22;

// a solved value as it is in memory (read from L2, never from a stale L1 line), and whether
// it is still the sentinel (for c128 each 8-byte half is checked: a 16-byte store may land
// in two parts)
__device__ __forceinline__ float2 ld_raw(const float2* p) {
  const unsigned long long u = *reinterpret_cast<const volatile unsigned long long*>(p);
  float2 v;
  v.x = __uint_as_float((unsigned)(u & 0xffffffffull));
  v.y = __uint_as_float((unsigned)(u >> 32));
  return v;
}
__device__ __forceinline__ double2 ld_raw(const double2* p) {
  const volatile unsigned long long* q = reinterpret_cast<const volatile unsigned long long*>(p);
  double2 v;
  v.x = __longlong_as_double((long long)q[0]);
  v.y = __longlong_as_double((long long)q[1]);
  return v;
}
__device__ __forceinline__ bool is_sent(float2 v) {
  return (((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x)) == SENT32;
}
__device__ __forceinline__ bool is_sent(double2 v) {
  return (unsigned long long)__double_as_longlong(v.x) == SENT64 ||
         (unsigned long long)__double_as_longlong(v.y) == SENT64;
}

// (grid.y: right-hand sides, ld apart)
template <typename T>
__global__ void k_fill_sentinel(T* v, int64_t n, int64_t ld) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long* u = reinterpret_cast<unsigned long long*>(v + blockIdx.y * ld + i);
  if (sizeof(T) == 8) {
    u[0] = SENT32;
  } else {
    u[0] = SENT64;
    u[1] = SENT64;
  }
}

// ring of factor blocks for the wavefront solve: stages of 16 x 256 elements
template <typename T>
struct TrsvRing {
  static constexpr int STG = sizeof(T) == 8 ? 3 : 2;
  static constexpr size_t BYTES = (size_t)STG * 16 * 256 * sizeof(T);
};
// one element global -> shared, asynchronously (zero-filled when !in: nothing is read)
__device__ __forceinline__ void cp_async_el(float2* dst, const float2* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_el(double2* dst, const double2* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <typename T, typename RT>
__global__ void __launch_bounds__(256) k_trsv_wave(const T* A, int64_t lda, int64_t n, const T* rhs, int64_t ldr, T* out,
                                                   int64_t ldo, int per_rhs, int lower, int* status, const T* dinv,
                                                   long long spin_max) {
  rhs += (blockIdx.x / per_rhs) * ldr;
  out += (blockIdx.x / per_rhs) * ldo;
  constexpr int STG = TrsvRing<T>::STG;
  extern __shared__ __align__(16) unsigned char trsv_smraw[];
  T* ring = reinterpret_cast<T*>(trsv_smraw);  // STG x 16 x 256 elements
  __shared__ RT sr[64], si[64];
  __shared__ RT pr[4][64], pim[4][64];
  const int nblk = (int)((n + 63) / 64);
  const int tid = threadIdx.x, r = tid & 63, q = tid >> 6;
  const T zero = {0, 0};
  bool timed_out = false;
  for (int t = blockIdx.x % per_rhs; t < nblk; t += per_rhs) {
    const int b = lower ? t : nblk - 1 - t;
    const int64_t r0 = (int64_t)b * 64;
    const int rb = (int)(n - r0 < 64 ? n - r0 : 64);
    // this thread's 16 entries of the diagonal block's inverse (row r, columns q*16..)
    const T* Di = dinv + (int64_t)b * 2 * 4096 + (lower ? 0 : 4096);
    T dv[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) dv[c] = Di[(q * 16 + c) * 64 + r];
    // the block's right-hand side, needed right after the last dependency
    const T bv = (tid < rb) ? rhs[r0 + tid] : zero;
    // this thread's 16 entries of the factor block of dependency s (row r0 + r) go into ring
    // stage s % TRSV_STG by cp.async: each thread reads back only what it copied itself, so
    // the walk needs no barrier
    auto issue_blk = [&](int s) {
      if (s < t) {
        const int k = lower ? s : nblk - 1 - s;
        const int64_t c0 = (int64_t)k * 64;
        const int cb = (int)(n - c0 < 64 ? n - c0 : 64);
        const T* Ar = A + (r0 + r) + c0 * lda;
        T* st = ring + (size_t)(s % STG) * 16 * 256;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int col = q * 16 + c;
          const bool in = r < rb && col < cb;
          cp_async_el(st + c * 256 + tid, in ? Ar + (int64_t)col * lda : A, in);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the solved values of dependency s: lane l of a warp (all its lanes share q) reads value
    // q*16 + (l & 15) as it is in memory (maybe still the sentinel): the warp's 16 values
    // are one 128-byte line, so one request per warp per poll, and they are passed to every
    // lane with shuffles once all are written
    const int lane = tid & 31;
    auto load_x = [&](int s) -> T {
      const int k = lower ? s : nblk - 1 - s;
      const int c = q * 16 + (lane & 15);
      return c < (int)(n - (int64_t)k * 64) ? ld_raw(out + (int64_t)k * 64 + c) : zero;
    };
    RT ar = 0, ai = 0;
    T x1 = zero, x2 = zero;
#pragma unroll
    for (int j = 0; j < STG - 1; ++j) issue_blk(j);
    if (t > 0) x1 = load_x(0);
    if (t > 1) x2 = load_x(1);
    for (int s = 0; s < t; ++s) {
      issue_blk(s + STG - 1);
      // solved values two dependencies ahead are requested before this one is used
      T v = x1;
      x1 = x2;
      if (s + 2 < t) x2 = load_x(s + 2);
      cp_async_wait<STG - 1>();  // this thread's copies of dependency s have landed
      const T* st = ring + (size_t)(s % STG) * 16 * 256;
      T cur[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) cur[c] = st[c * 256 + tid];
      long long it = 0;
      while (!__all_sync(0xffffffffu, !is_sent(v))) {  // warp-uniform
        if (++it > spin_max) {
          if (!timed_out) atomicOr(status, 8);
          timed_out = true;
          if (is_sent(v)) v = zero;
          break;
        }
        if (is_sent(v)) v = load_x(s);
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const T xc = shfl_c(v, c);
        ar += (RT)cur[c].x * (RT)xc.x - (RT)cur[c].y * (RT)xc.y;
        ai += (RT)cur[c].x * (RT)xc.y + (RT)cur[c].y * (RT)xc.x;
      }
    }
    cp_async_wait<0>();
    pr[q][r] = ar;
    pim[q][r] = ai;
    __syncthreads();
    if (tid < 64) {
      RT vr = 0, vi = 0;
      if (tid < rb) {
        vr = (RT)bv.x - (pr[0][tid] + pr[1][tid] + pr[2][tid] + pr[3][tid]);
        vi = (RT)bv.y - (pim[0][tid] + pim[1][tid] + pim[2][tid] + pim[3][tid]);
      }
      sr[tid] = vr;
      si[tid] = vi;
    }
    __syncthreads();
    // x_b = inv(D_b) * rhs_b  (64 x 64 matvec, 4 quarter sums per row)
    {
      RT accr = 0, acci = 0;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const T m = dv[c];
        accr += (RT)m.x * sr[q * 16 + c] - (RT)m.y * si[q * 16 + c];
        acci += (RT)m.x * si[q * 16 + c] + (RT)m.y * sr[q * 16 + c];
      }
      pr[q][r] = accr;
      pim[q][r] = acci;
    }
    __syncthreads();
    if (tid < rb) {
      T o;
      o.x = pr[0][tid] + pr[1][tid] + pr[2][tid] + pr[3][tid];
      o.y = pim[0][tid] + pim[1][tid] + pim[2][tid] + pim[3][tid];
      __stcg(out + r0 + tid, o);
    }
    __syncthreads();  // pr / pim are rewritten by the next block row
  }
}

// out[i] = in[perm[i]]: the row interchanges of the factorisation applied as one gather
template <typename T>
__global__ void k_permute(const T* in, int64_t ldi, T* out, int64_t ldo, const int* perm, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[blockIdx.y * ldo + i] = in[blockIdx.y * ldi + perm[i]];
}

// ---- FP64 matvec y = alpha A x + beta y  (A c128 or c64) --------------------------------
// Column slabs of the partial sums (grid.y): as many row blocks x slabs as fill whole waves of the
// CTAs the chip holds (mv_slabs), up to
constexpr int MV_MAX_SLABS = 64;
// x (complex FP64) split into float hi + lo parts: (re_hi, im_hi, re_lo, im_lo)
__global__ void k_split_x(int64_t n, const double* x, float4* xs) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xr = x[2 * i], xi = x[2 * i + 1];
  float rh = (float)xr, ih = (float)xi;
  xs[i] = make_float4(rh, ih, (float)(xr - (double)rh), (float)(xi - (double)ih));
}

// s_hi + s_lo += p with the rounding error of the addition kept (TwoSum)
__device__ __forceinline__ void two_sum_acc(float& sh, float& sl, float p) {
  float s = __fadd_rn(sh, p);
  float bb = __fsub_rn(s, sh);
  float t = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  sh = s;
  sl = __fadd_rn(sl, t);
}

// partial sums of A x for a c64 matrix with FP64-level accuracy from FP32 arithmetic:
// each product a * x_hi is split exactly into p + e (e = fma(a, x_hi, -p)), p is added with
// TwoSum, e and a * x_lo go to the low part (compensated dot product of Ogita, Rump and
// Oishi, SIAM J. Sci. Comput. 26 (2005)).
__global__ void k_gemv_partial_c64_df(int64_t n, const float2* A, int64_t lda, const float4* xs,
                                      double* part) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int s = blockIdx.y;
  int64_t c0 = n * s / gridDim.y, c1 = n * (s + 1) / gridDim.y;
  if (i >= n) return;
  float shr = 0.f, slr = 0.f, shi = 0.f, sli = 0.f;
  for (int64_t j = c0; j < c1; ++j) {
    float2 a = A[i + j * lda];
    float4 xv = xs[j];
    float p, e;
    p = __fmul_rn(a.x, xv.x);
    e = fmaf(a.x, xv.x, -p);
    two_sum_acc(shr, slr, p);
    slr = __fadd_rn(slr, e);
    p = __fmul_rn(-a.y, xv.y);
    e = fmaf(-a.y, xv.y, -p);
    two_sum_acc(shr, slr, p);
    slr = __fadd_rn(slr, e);
    slr = __fadd_rn(slr, __fsub_rn(__fmul_rn(a.x, xv.z), __fmul_rn(a.y, xv.w)));
    p = __fmul_rn(a.x, xv.y);
    e = fmaf(a.x, xv.y, -p);
    two_sum_acc(shi, sli, p);
    sli = __fadd_rn(sli, e);
    p = __fmul_rn(a.y, xv.x);
    e = fmaf(a.y, xv.x, -p);
    two_sum_acc(shi, sli, p);
    sli = __fadd_rn(sli, e);
    sli = __fadd_rn(sli, __fadd_rn(__fmul_rn(a.x, xv.w), __fmul_rn(a.y, xv.z)));
  }
  part[2 * (s * n + i)] = (double)shr + (double)slr;
  part[2 * (s * n + i) + 1] = (double)shi + (double)sli;
}

// the same with two rows per thread: one 16-byte load brings a[i, j] and a[i+1, j] (even i,
// even lda), and the two rows are independent accumulation chains.  The real and imaginary
// parts of a row travel as the two lanes of packed FP32 operations (sm_100 FFMA2 / FADD2 /
// FMUL2, each lane rounded as its scalar counterpart):
//   (re, im) += (a_r, a_r) (x_r, x_i) + (a_i, a_i) (-x_i, x_r),
// every product kept exactly (TwoProduct: p and fma(a, x, -p)) and added to the high part with
// its rounding error (TwoSum); the low-part terms (x's low half) in plain FP32.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {  // a - b, one rounding
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
// sh + sl += A X with the product's and the sum's rounding errors kept; nX = -X gives the negated
// product without a negation (the packed operations have no sign modifiers)
__device__ __forceinline__ void cdf_prod2(float2 A, float2 X, float2 nX, float2& sh, float2& sl) {
  const float2 np = __fmul2_rn(A, nX);        // -p
  const float2 e = __ffma2_rn(A, X, np);      // A X - p
  const float2 t = sub2(sh, np);
  const float2 bb = sub2(t, sh);
  const float2 v = sub2(sh, sub2(t, bb));     // TwoSum(sh, p): v - (np + bb)
  sl = __fadd2_rn(sl, __fadd2_rn(v, sub2(e, __fadd2_rn(np, bb))));
  sh = t;
}
// one column of the vector as the packed operands of both parts: (x_r, x_i) with A_r, (-x_i, x_r)
// with A_i, their negatives and the low halves
struct MvX {
  float2 X1, X2, n1, n2, L1, L2;
};
__device__ __forceinline__ MvX mv_x(float4 v) {
  MvX x;
  x.X1 = make_float2(v.x, v.y);
  x.n1 = make_float2(-v.x, -v.y);
  x.X2 = make_float2(x.n1.y, v.x);
  x.n2 = make_float2(v.y, x.n1.x);
  x.L1 = make_float2(v.z, v.w);
  x.L2 = make_float2(-v.w, v.z);
  return x;
}
__device__ __forceinline__ void cdf_acc2(float ar, float ai, const MvX& x, float2& sh, float2& sl) {
  const float2 A = make_float2(ar, ar), B = make_float2(ai, ai);
  cdf_prod2(A, x.X1, x.n1, sh, sl);
  cdf_prod2(B, x.X2, x.n2, sh, sl);
  sl = __ffma2_rn(A, x.L1, sl);
  sl = __ffma2_rn(B, x.L2, sl);
}
__global__ void k_gemv_partial_c64_df2(int64_t n, const float2* A, int64_t lda, const float4* xs,
                                       double* part) {
  const int64_t i = 2 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
  const int s = blockIdx.y;
  const int64_t c0 = n * s / gridDim.y, c1 = n * (s + 1) / gridDim.y;
  if (i >= n) return;
  const bool two = i + 1 < n;
  float2 h0 = make_float2(0.f, 0.f), l0 = h0, h1 = h0, l1 = h0;
#pragma unroll 4
  for (int64_t j = c0; j < c1; ++j) {
    const MvX x = mv_x(xs[j]);
    float4 a;
    if (two) {
      a = *reinterpret_cast<const float4*>(A + i + j * lda);
    } else {
      const float2 a0 = A[i + j * lda];
      a = make_float4(a0.x, a0.y, 0.f, 0.f);
    }
    cdf_acc2(a.x, a.y, x, h0, l0);
    cdf_acc2(a.z, a.w, x, h1, l1);
  }
  part[2 * (s * n + i)] = (double)h0.x + (double)l0.x;
  part[2 * (s * n + i) + 1] = (double)h0.y + (double)l0.y;
  if (two) {
    part[2 * (s * n + i + 1)] = (double)h1.x + (double)l1.x;
    part[2 * (s * n + i + 1) + 1] = (double)h1.y + (double)l1.y;
  }
}

// partial sums of A x for a c128 matrix on the FP32 pipes: each entry split into hi + lo
// floats (fsplit.h), hi * x_hi kept exactly (TwoProduct) and added with TwoSum, the terms of
// the low parts (hi * x_lo, lo * x_hi) accumulated in FP32 -- the compensated dot product of
// k_gemv_partial_c64_df2 with the matrix's own low part added.  About 2^-47 relative per
// product, against a few FP64 multiply-adds per entry at GB300's FP64 rate.
// Two rows (128 apart) per thread share the vector's loads and operand pairs; the eight matrix
// loads of four columns are in flight before their arithmetic: 2.72 ms at n = 30720 (5.6 TB/s; one row
// per thread and 32 slabs: 3.08 ms), 0.200 ms at n = 7213 (0.217).
constexpr int MV_ROWS = 256;  // rows per CTA of 128 threads
__global__ void __launch_bounds__(128) k_gemv_partial_c128_df(int64_t n, const double2* A, int64_t lda, const float4* xs,
                                                              double* part) {
  const int64_t i0 = blockIdx.x * (int64_t)MV_ROWS + threadIdx.x, i1 = i0 + 128;
  const int s = blockIdx.y;
  const int64_t c0 = n * s / gridDim.y, c1 = n * (s + 1) / gridDim.y;
  const bool in0 = i0 < n, in1 = i1 < n;
  float2 h0 = make_float2(0.f, 0.f), l0 = h0, h1 = h0, l1 = h0;
  auto term = [&](float2 ar, float2 ai, const MvX& x, float2& h, float2& l) {
    cdf_acc2(ar.x, ai.x, x, h, l);
    l = __ffma2_rn(make_float2(ar.y, ar.y), x.X1, l);
    l = __ffma2_rn(make_float2(ai.y, ai.y), x.X2, l);
  };
  const double2 zero = make_double2(0.0, 0.0);
  const double2 *A0 = A + (in0 ? i0 : 0), *A1 = A + (in1 ? i1 : 0);
  auto column = [&](const double2 a, const double2 b, const float4 xv) {
    const MvX x = mv_x(xv);
    float2 r, i;
    fsplit::split_f64_fast(a.x, &r.x, &r.y);
    fsplit::split_f64_fast(a.y, &i.x, &i.y);
    term(r, i, x, h0, l0);
    fsplit::split_f64_fast(b.x, &r.x, &r.y);
    fsplit::split_f64_fast(b.y, &i.x, &i.y);
    term(r, i, x, h1, l1);
  };
  int64_t j = c0;
  for (; j + 4 <= c1; j += 4) {
    double2 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a[u] = in0 ? __ldcs(A0 + (j + u) * lda) : zero;
      b[u] = in1 ? __ldcs(A1 + (j + u) * lda) : zero;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) column(a[u], b[u], xs[j + u]);
  }
  for (; j < c1; ++j) column(in0 ? __ldcs(A0 + j * lda) : zero, in1 ? __ldcs(A1 + j * lda) : zero, xs[j]);
  if (in0) {
    part[2 * (s * n + i0)] = (double)h0.x + (double)l0.x;
    part[2 * (s * n + i0) + 1] = (double)h0.y + (double)l0.y;
  }
  if (in1) {
    part[2 * (s * n + i1)] = (double)h1.x + (double)l1.x;
    part[2 * (s * n + i1) + 1] = (double)h1.y + (double)l1.y;
  }
}

// y = alpha (sum of the slabs) + beta y: 64 rows per CTA, the slabs of a row dealt over four threads
__global__ void __launch_bounds__(256) k_gemv_reduce(int64_t n, int slabs, const double* part, double* y, double alpha,
                                                     double beta) {
  __shared__ double2 sp[4][64];
  const int r = threadIdx.x & 63, q = threadIdx.x >> 6;
  const int64_t i = blockIdx.x * (int64_t)64 + r;
  double2 a = make_double2(0.0, 0.0);
  if (i < n)
#pragma unroll 4
    for (int s = q; s < slabs; s += 4) {
      const double2 v = reinterpret_cast<const double2*>(part)[s * n + i];
      a.x += v.x;
      a.y += v.y;
    }
  sp[q][r] = a;
  __syncthreads();
  if (q > 0 || i >= n) return;
  const double sr = (sp[0][r].x + sp[1][r].x) + (sp[2][r].x + sp[3][r].x);
  const double si = (sp[0][r].y + sp[1][r].y) + (sp[2][r].y + sp[3][r].y);
  double yr = beta == 0.0 ? 0.0 : beta * y[2 * i], yi = beta == 0.0 ? 0.0 : beta * y[2 * i + 1];
  y[2 * i] = alpha * sr + yr;
  y[2 * i + 1] = alpha * si + yi;
}

__global__ void k_c128_to_c64(int64_t rows, int64_t cols, const double* s, int64_t lds, float* d,
                              int64_t ldd) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t c = blockIdx.y;
  for (; c < cols; c += gridDim.y)
    if (i < rows) {
      // rounded by integer operations: a conversion instruction runs on GB300's FP64 pipe
      d[2 * (i + c * ldd)] = fsplit::to_float_rn(s[2 * (i + c * lds)]);
      d[2 * (i + c * ldd) + 1] = fsplit::to_float_rn(s[2 * (i + c * lds) + 1]);
    }
}
__global__ void k_c64_to_c128(int64_t rows, int64_t cols, const float* s, int64_t lds, double* d,
                              int64_t ldd) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t c = blockIdx.y;
  for (; c < cols; c += gridDim.y)
    if (i < rows) {
      d[2 * (i + c * ldd)] = fsplit::f2d(s[2 * (i + c * lds)]);
      d[2 * (i + c * ldd) + 1] = fsplit::f2d(s[2 * (i + c * lds) + 1]);
    }
}

__global__ void k_axpy(int64_t n, double ar, double ai, const double* x, double* y) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xr = x[2 * i], xi = x[2 * i + 1];
  y[2 * i] += ar * xr - ai * xi;
  y[2 * i + 1] += ar * xi + ai * xr;
}

// deterministic sum of |x|^2: fixed grid, per-block partials, single-block final pass
__global__ void k_norm2_part(int64_t n, const double* x, double* part) {
  __shared__ double s[256];
  double acc = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    acc += x[2 * i] * x[2 * i] + x[2 * i + 1] * x[2 * i + 1];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}
__global__ void k_sum_part(int np, const double* part, double* out) {
  __shared__ double s[256];
  double acc = 0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) acc += part[i];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0];
}

// w -= sum_k h_k V_k
__global__ void k_gemv_sub(int64_t n, int m, const double* V, int64_t ldv, const double* h, double* w) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double sr = 0, si = 0;
  for (int k = 0; k < m; ++k) {
    double vr = V[2 * (i + k * ldv)], vi = V[2 * (i + k * ldv) + 1];
    double hr = h[2 * k], hi = h[2 * k + 1];
    sr += hr * vr - hi * vi;
    si += hr * vi + hi * vr;
  }
  w[2 * i] -= sr;
  w[2 * i + 1] -= si;
}

// ---- the Arnoldi step of GMRES ----------------------------------------------------------
// One kernel per pass over the basis: a CTA owns GM_ROWS rows of w and
//   0: forms them from the matvec's slabs,      then dots with V_0 .. V_k
//   1: subtracts V h of the first pass,          then dots again (the reorthogonalisation)
//   2: subtracts V h of the second pass,         then the norm
// with its rows in shared memory between the two halves, and the last CTA to finish adds the
// CTAs' partial sums in order (deterministic; no second launch, no host round trip).  The whole
// iteration is then five launches, its coefficients and norm read back once.
// Dots: a warp takes four basis vectors at a time, its eight partial sums reduced over the lanes
// by halving (nine additions instead of forty).
constexpr int GM_ROWS = 64, GM_THREADS = 256;

// out[8 values of a warp]: lane 4 j writes value j's total (j = 0 .. 7, re / im of four vectors)
__device__ __forceinline__ double gm_reduce8(double* v, int lane) {
#pragma unroll
  for (int half = 4, o = 16; half >= 1; half >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double keep = up ? v[i + half] : v[i], give = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// mode as above; k1 = k + 1 basis vectors; h_in: their coefficients (modes 1, 2); out: k1 complex
// sums (modes 0, 1) or the squared norm (mode 2); part: [gridDim.x][2 k1]; count: zero at entry and exit
__global__ void __launch_bounds__(GM_THREADS) k_gm_step(int mode, int64_t n, int k1, int slabs, const double* slab,
                                                        const double* V, double* w, const double* h_in, double* part,
                                                        unsigned int* count, double* out) {
  __shared__ double2 sw[GM_ROWS];
  __shared__ double2 sp[GM_THREADS / GM_ROWS][GM_ROWS];
  __shared__ bool s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid % GM_ROWS, q = tid / GM_ROWS;
  const int64_t r0 = blockIdx.x * (int64_t)GM_ROWS, row = r0 + r;
  const bool in = row < n;
  // ---- this CTA's rows of w
  {
    double2 a = make_double2(0.0, 0.0);
    if (in) {
      if (mode == 0) {
        for (int s = q; s < slabs; s += GM_THREADS / GM_ROWS) {
          const double2 v = reinterpret_cast<const double2*>(slab)[s * n + row];
          a.x += v.x;
          a.y += v.y;
        }
      } else {
        const double2* h = reinterpret_cast<const double2*>(h_in);
#pragma unroll 4
        for (int k = q; k < k1; k += GM_THREADS / GM_ROWS) {
          const double2 v = reinterpret_cast<const double2*>(V)[k * n + row], c = h[k];
          a.x = fma(c.x, v.x, fma(-c.y, v.y, a.x));
          a.y = fma(c.x, v.y, fma(c.y, v.x, a.y));
        }
      }
    }
    sp[q][r] = a;
    __syncthreads();
    if (q == 0) {
      double2 t = make_double2((sp[0][r].x + sp[1][r].x) + (sp[2][r].x + sp[3][r].x),
                               (sp[0][r].y + sp[1][r].y) + (sp[2][r].y + sp[3][r].y));
      if (in) {
        double2* wr = reinterpret_cast<double2*>(w) + row;
        if (mode > 0) {
          const double2 o = *wr;
          t = make_double2(o.x - t.x, o.y - t.y);
        }
        *wr = t;
      }
      sw[r] = t;  // (rows beyond n: zero)
    }
    __syncthreads();
  }
  // ---- partial sums over them
  const int nv = mode == 2 ? 1 : 2 * k1;
  double* mine = part + (size_t)blockIdx.x * nv;
  if (mode == 2) {
    if (warp == 0) {
      const double2 a = sw[lane], b = sw[lane + 32];
      double v = (a.x * a.x + a.y * a.y) + (b.x * b.x + b.y * b.y);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) mine[0] = v;
    }
  } else {
    const double2 w0 = sw[lane], w1 = sw[lane + 32];
    const bool in0 = r0 + lane < n, in1 = r0 + lane + 32 < n;
    const double2 zero = make_double2(0.0, 0.0);
    for (int k0 = 4 * warp; k0 < k1; k0 += 4 * (GM_THREADS / 32)) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double2* vk = reinterpret_cast<const double2*>(V) + (int64_t)(k0 + u) * n + r0 + lane;
        const bool ok = k0 + u < k1;
        const double2 a = ok && in0 ? vk[0] : zero, b = ok && in1 ? vk[32] : zero;
        v[2 * u] = fma(a.x, w0.x, fma(a.y, w0.y, fma(b.x, w1.x, b.y * w1.y)));
        v[2 * u + 1] = fma(a.x, w0.y, fma(-a.y, w0.x, fma(b.x, w1.y, -(b.y * w1.x))));
      }
      const double t = gm_reduce8(v, lane);
      const int j = 2 * k0 + (lane >> 2);
      if ((lane & 3) == 0 && j < nv) mine[j] = t;
    }
  }
  // ---- the last CTA adds the partial sums, in the CTAs' order
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int j = tid; j < nv; j += GM_THREADS) {
    double a[4] = {0, 0, 0, 0};
    const int nb = (int)gridDim.x;
    for (int b = 0; b < nb; b += 16) {  // 16 loads in flight
      double v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = b + u < nb ? __ldcg(part + (size_t)(b + u) * nv + j) : 0.0;
#pragma unroll
      for (int u = 0; u < 16; ++u) a[u & 3] += v[u];
    }
    out[j] = (a[0] + a[1]) + (a[2] + a[3]);
  }
  if (tid == 0) *count = 0;
}

// v = w / |w| with |w|^2 on the device (0 for w = 0), and v as float pairs for the next matvec
__global__ void k_gm_next(int64_t n, const double* w, const double* norm2, double* v, float4* xs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double nrm = sqrt(*norm2), inv = nrm > 0.0 ? 1.0 / nrm : 0.0;
  const double2 a = reinterpret_cast<const double2*>(w)[i], b = make_double2(inv * a.x, inv * a.y);
  reinterpret_cast<double2*>(v)[i] = b;
  const float rh = (float)b.x, ih = (float)b.y;
  xs[i] = make_float4(rh, ih, (float)(b.x - (double)rh), (float)(b.y - (double)ih));
}

template <typename T, typename R>
struct LUSteps {
  beast_ctx* ctx;
  T* A;
  int64_t lda, n;
  int* ipiv;
  cudaStream_t st;
  size_t tcwork_bytes;
  int laswp(int64_t c0, int64_t c1, int64_t p0, int64_t p1) {
    if (c1 <= c0 || p1 <= p0) return BEAST_OK;
    ProfScope ps(ctx, PK_LASWP, (double)(c1 - c0) * (p1 - p0) * 2 * sizeof(T));
    k_laswp<T><<<(unsigned)((c1 - c0 + 255) / 256), 256, 0, st>>>(A, lda, c0, c1, p0, p1, ipiv);
    BEAST_CUDA_TRY(ctx, cudaGetLastError());
    return BEAST_OK;
  }
  // U12 = L11^{-1} A12 for columns [c0, c1), L11 = the diagonal block at j0
  int trsm(int64_t j0, int kb, int64_t c0, int64_t c1) {
    if (c1 <= c0) return BEAST_OK;
    ProfScope ps(ctx, PK_TRSM, 4.0 * (double)(c1 - c0) * kb * kb);
    constexpr int NS = TrsmTile<T>::NS;
    k_trsm_tile<T, R, false><<<(unsigned)((c1 - c0 + NS - 1) / NS), TrsmTile<T>::NT, trsm_tile_smem<T>(), st>>>(
        A, lda, j0, kb, c0, c1);
    BEAST_CUDA_TRY(ctx, cudaGetLastError());
    return BEAST_OK;
  }
  // A[r0:r0+m, c0:c0+nc] -= A[r0:r0+m, k0:k0+k] A[k0:k0+k, c0:c0+nc]
  int gemm(int64_t r0, int64_t m, int64_t c0, int64_t nc, int64_t k0, int k, void* tcwork) {
    return gemm2(r0, m, c0, nc, 0, 0, k0, k, tcwork);
  }
  // the same on an L-shaped region: rows [r0, r0+m0) of columns [c0, c0+n0), then rows
  // [r0, r0+m1) (m1 <= m0) of the next n1 columns -- one tensor-core launch for both
  // whether gemm2 with these sizes runs (and on the tensor cores)
  static bool gemm2_runs(int64_t m0, int64_t n0, int64_t m1, int64_t n1, int k) {
    return m0 > 0 && k > 0 && (n0 > 0 || (m1 > 0 && n1 > 0));
  }
  bool gemm2_tc(int64_t m0, int64_t n0, int64_t n1, int k, const void* tcwork) const {
    return sizeof(T) == 8 && tcwork && m0 >= 64 && n0 + n1 >= 64 && k % 32 == 0;
  }
  // complex FP64: digit-sliced tensor-core products (tc_gemm64.cu) for every update (a 32 x 32
  // block with K = 64 takes 50 us there and 440 us on the FP64 units of one SM); the FP64 units
  // only without the workspace
  bool gemm64_tc(int k, const void* tcwork) const { return sizeof(T) == 16 && tcwork && k % 32 == 0; }
  // prepped: the FP16 operands are already in tcwork (k_panel_apply wrote them)
  int gemm2(int64_t r0, int64_t m0, int64_t c0, int64_t n0, int64_t m1, int64_t n1, int64_t k0, int k,
            void* tcwork, bool prepped = false) {
    if (!gemm2_runs(m0, n0, m1, n1, k)) return BEAST_OK;
    const bool tc = gemm2_tc(m0, n0, n1, k, tcwork);
    if (tc)  // brackets its operand preparation and its tensor-core launch separately
      return tc_gemm_sub(ctx, reinterpret_cast<float2*>(A), lda, r0, k0, c0, m0, n0, m1, n1, k, tcwork,
                         tcwork_bytes, prepped);
    const int64_t ms[2] = {m0, m1}, cs[2] = {c0, c0 + n0}, ns[2] = {n0, n1};
    for (int r = 0; r < 2; ++r) {
      if (ms[r] <= 0 || ns[r] <= 0) continue;
      if (gemm64_tc(k, tcwork)) {
        double2* Ad = reinterpret_cast<double2*>(A);
        int rc = tc_gemm64_sub(ctx, Ad + r0 + cs[r] * lda, lda, Ad + r0 + k0 * lda, lda, Ad + k0 + cs[r] * lda, lda, ms[r],
                               ns[r], k, tcwork, tcwork_bytes);
        if (rc) return rc;
        continue;
      }
      ProfScope ps(ctx, PK_GEMM, 8.0 * (double)k * (double)ms[r] * ns[r]);
      dim3 g((unsigned)((ms[r] + GT - 1) / GT), (unsigned)((ns[r] + GT - 1) / GT));
      k_gemm_sub<T, R><<<g, 256, 0, st>>>(A + r0 + cs[r] * lda, lda, A + r0 + k0 * lda, lda, A + k0 + cs[r] * lda,
                                          lda, ms[r], ns[r], k);
      BEAST_CUDA_TRY(ctx, cudaGetLastError());
    }
    return BEAST_OK;
  }
  // symmetric update: A[rowA.., rowB..] (m x nc) -= L1 D L2^T, L1 = A[rowA.., colA..],
  // L2 = A[rowB.., colA..], D the pivots on the diagonal at colA..; lower: only the tiles on or
  // below the diagonal (tensor cores; the CUDA-core fallback updates the whole rectangle)
  bool symgemm_tc(int64_t m, int64_t nc, int k, const void* tcwork) const {
    return sizeof(T) == 8 && tcwork && m >= 64 && nc >= 64 && k % 32 == 0;
  }
  // a_skip: the prepped operands were written for a_skip more rows above rowA
  int symgemm(int64_t rowA, int64_t m, int64_t rowB, int64_t nc, int64_t colA, int k, bool lower, void* tcwork,
              bool prepped = false, int64_t a_skip = 0) {
    if (m <= 0 || nc <= 0 || k <= 0) return BEAST_OK;
    const bool tc = symgemm_tc(m, nc, k, tcwork);
    if (tc)  // brackets its operand preparation and its tensor-core launch separately
      return tc_gemm_sym(ctx, reinterpret_cast<float2*>(A), lda, rowA, colA, rowB, m, nc, k, lower, tcwork,
                         tcwork_bytes, prepped, prepped ? a_skip : 0);
    ProfScope ps(ctx, PK_GEMM, 8.0 * (double)k * (double)m * nc);
    T* B = nullptr;
    BEAST_CUDA_TRY(ctx, cudaMallocAsync(&B, (size_t)k * nc * sizeof(T), st));
    const int64_t tot = (int64_t)k * nc;
    k_dlt<T><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(A + rowB + colA * lda, A + colA + colA * lda, lda, k,
                                                            (int)nc, B);
    dim3 g((unsigned)((m + GT - 1) / GT), (unsigned)((nc + GT - 1) / GT));
    k_gemm_sub<T, R><<<g, 256, 0, st>>>(A + rowA + rowB * lda, lda, A + rowA + colA * lda, lda, B, k, m, nc, k);
    BEAST_CUDA_TRY(ctx, cudaGetLastError());
    BEAST_CUDA_TRY(ctx, cudaFreeAsync(B, st));
    return BEAST_OK;
  }
};

// Two-level right-looking LU: column blocks of NB are factored with nb-wide panels (panel,
// interchanges, TRSM and GEMM restricted to the block); then the block's interchanges are
// applied to the other columns and the trailing matrix gets one rank-NB update
// (TRSM for U12, GEMM with K = NB -- on the tensor cores for complex FP32).
//
// sym (unpivoted c64 with 64-wide panels; A near complex-symmetric, the factors serving as the
// preconditioner of a refined solve): an LDL^T-type factorisation that keeps only the lower
// triangle current -- the diagonal blocks are factored from their lower triangle mirrored,
// U12 = D L21^T is never formed in FP32 (the updates take it from L21 and the pivots), the
// in-block and mid-block updates cover only the rows below, the trailing update only the
// tiles on or below the diagonal: about half the work.  At the end U = D L^T is written above
// the diagonal blocks, so the factors have the layout of the LU.
template <typename T, typename R>
int lu_factor_t(beast_ctx* ctx, int64_t n, T* A, int64_t lda, int* ipiv, int* info, bool pivot, bool sym) {
  cudaStream_t st = ctx->stream;
  const int G0 = std::max(1, ctx->num_sms);
  const size_t smem_cap = 220 * 1024;
  // panel width: 64; with pivoting the cooperative panel kernel holds its share of the panel's
  // rows in shared memory, which narrows the panel for very tall matrices
  int nb = 64;
  const int64_t rows0 = (n + G0 - 1) / G0;
  if (pivot) {
    while (nb > 8 && (size_t)(rows0 * (nb + 1) + 3 * nb) * sizeof(T) > smem_cap) nb /= 2;
    if ((size_t)(rows0 * (nb + 1) + 3 * nb) * sizeof(T) > smem_cap)
      return beast_fail(ctx, BEAST_ERR_ARG, "matrix too large for the shared-memory panel");
  }
  // outer / mid block widths in columns: 16 and 4 panels (with pivoting a single level);
  // unpivoted, BEAST_LU_NB / BEAST_LU_NB2 override them (multiples of the panel width, the
  // mid width dividing the outer one, the outer one at most TC_SYM_KMAX)
  int NB = 16 * nb;
  int64_t NB2 = pivot ? NB : 4 * nb;
  if (!pivot) {
    const char* e1 = getenv("BEAST_LU_NB");
    const char* e2 = getenv("BEAST_LU_NB2");
    const int b1 = e1 ? atoi(e1) : NB, b2 = e2 ? atoi(e2) : (int)NB2;
    if (b2 >= nb && b2 % nb == 0 && b1 >= b2 && b1 % b2 == 0 && b1 <= TC_SYM_KMAX) {
      NB = b1;
      NB2 = b2;
    }
  }
  const size_t panel_smem = (size_t)(std::max<int64_t>(rows0, PANEL_ROWS) * (nb + 1) + 3 * nb) * sizeof(T);
  if (pivot)
    BEAST_CUDA_TRY(ctx, allow_shared((const void*)k_panel<T>));
  // unpivoted c64 with 64-wide panels: k_lu_inv64 also inverts the block's triangles and
  // k_panel_apply does both triangular solves (and the FP16 operands of the in-block update)
  const bool apply_path = !pivot && sizeof(T) == 8 && nb == TRI;
  sym = sym && apply_path;
  const size_t getrf_sm = (size_t)TRI * (TRI + 1) * sizeof(T);
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_getrf64<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64_pair<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64_pair<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64<T, false, 2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu_inv64<T, true, 2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)getrf_sm));
  // the diagonal-block elimination with 2 x 2 tiles on 1024 threads (default), 2 x 4 tiles on 512
  // (BEAST_LU_DIAG_TILE=24) or 4 x 4 tiles on 256 (BEAST_LU_DIAG_TILE=4): the same arithmetic
  // per element, different thread counts
  const char* dt_env = getenv("BEAST_LU_DIAG_TILE");
  const int dtile = dt_env && dt_env[0] == '4' ? 44 : (dt_env && dt_env[0] == '2' && dt_env[1] == '4' ? 24 : 22);
  if (apply_path)
    BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_panel_apply<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)panel_apply_smem()));
    BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_panel_apply<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)panel_apply_smem()));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_trsm_tile<T, R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)trsm_tile_smem<T>()));
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_trsm_tile<T, R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)trsm_tile_smem<T>()));
  if (pivot) {
    int occ = 0;
    BEAST_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_panel<T>, 256, panel_smem));
    if (occ < 1) return beast_fail(ctx, BEAST_ERR_CUDA, "panel kernel does not fit on an SM");
  }
  const size_t slot_bytes = pivot ? panel_column_words<T>(nb, G0) * nb * 8 : 0;
  size_t need = slot_bytes + 256;
  char* scr = nullptr;
  BEAST_CUDA_TRY(ctx, cudaMallocAsync(&scr, need, st));
  unsigned long long* slots = reinterpret_cast<unsigned long long*>(scr + 256);
  int* dinfo = reinterpret_cast<int*>(scr);       // first zero pivot (1-based)
  int* dstatus = dinfo + 1;                        // a panel wait that ran out
  auto diag = [&](bool sy, int64_t jd, int kd, T* out_inv, cudaStream_t s_) {
    if (dtile == 22 && sy)
      k_lu_inv64_pair<T, true><<<1, TRI * TRI / 4, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
    else if (dtile == 22)
      k_lu_inv64_pair<T, false><<<1, TRI * TRI / 4, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
    else if (dtile == 24 && sy)
      k_lu_inv64<T, true, 2, 4><<<1, TRI * TRI / 8, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
    else if (dtile == 24)
      k_lu_inv64<T, false, 2, 4><<<1, TRI * TRI / 8, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
    else if (sy)
      k_lu_inv64<T, true><<<1, 256, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
    else
      k_lu_inv64<T, false><<<1, 256, getrf_sm, s_>>>(A, lda, jd, kd, dinfo, out_inv);
  };
  BEAST_CUDA_TRY(ctx, cudaMemsetAsync(scr, 0, 256, st));
  BEAST_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), st));
  // tensor-core workspace: the FP16 operands of the largest update (M, N <= n, K <= NB)
  void* tcwork = nullptr;
  size_t tcwork_bytes = 0;
  if (sizeof(T) == 8 && tc_gemm_supported(A, lda, NB) && n > NB) {
    tcwork_bytes = tc_gemm_work_bytes(n, n, NB);
    BEAST_CUDA_TRY(ctx, cudaMallocAsync(&tcwork, tcwork_bytes, st));
  }
  // complex FP64: the digit slices of the largest update; without the memory for them the updates
  // stay on the FP64 units
  if (sizeof(T) == 16 && pivot && n > nb && tc_gemm64_supported()) {
    tcwork_bytes = tc_gemm64_work_bytes(n, n, NB);
    if (cudaMallocAsync(&tcwork, tcwork_bytes, st) != cudaSuccess) {
      cudaGetLastError();
      tcwork = nullptr;
    }
  }
  LUSteps<T, R> S{ctx, A, lda, n, ipiv, st, tcwork_bytes};
  // lookahead (symmetric path with tensor-core updates; BEAST_LU_LOOKAHEAD=1): while a panel's
  // other rows and its update run on the context's stream, the second stream solves the next
  // panel's block row, updates and eliminates the next diagonal block.  ahead: this panel's
  // elimination has run there (event la_ev[lu_par]).
  const char* la_env = getenv("BEAST_LU_LOOKAHEAD");
  const bool la = sym && tcwork && la_env && la_env[0] == '1' && ctx_lookahead_streams(ctx);
  if (la)
    BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_sym_diag_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sym_diag_update_smem()));
  bool ahead = false;
  int lu_par = 0;

  int rc = BEAST_OK;
  // unpivoted, the outer block is factored in mid blocks of NB2 columns: the panels update
  // only their mid block (and its rows beyond it), the mid block updates the rest of the
  // outer block with K = NB2, and the outer block the trailing matrix with K = NB -- fewer
  // passes of narrow (K = nb) updates over the same columns
  for (int64_t J0 = 0; J0 < n && rc == BEAST_OK; J0 += NB) {
    const int64_t J1 = std::min<int64_t>(n, J0 + NB);
    for (int64_t M0 = J0; M0 < J1 && rc == BEAST_OK; M0 += NB2) {
    const int64_t M1 = std::min<int64_t>(J1, M0 + NB2);
    for (int64_t j0 = M0; j0 < M1 && rc == BEAST_OK; j0 += nb) {
      int kb = (int)std::min<int64_t>(nb, M1 - j0);
      int64_t M = n - j0;
      // rows per CTA: the panel over all SMs, at least PANEL_ROWS (an exchange among fewer CTAs is
      // shorter, and the update of so few rows hides under it)
      int rows_per = (int)std::max<int64_t>(PANEL_ROWS, (M + G0 - 1) / G0);
      int G = (int)((M + rows_per - 1) / rows_per);
      size_t sm = (size_t)(rows_per * (kb + 1) + 3 * kb) * sizeof(T);
      if (pivot) {
        void* args[] = {&A, &lda, &n, &j0, &kb, &rows_per, &ipiv, &dinfo, &slots, &dstatus};
        {
          ProfScope ps(ctx, PK_PANEL, 8.0 * (double)M * kb * kb / 2);
          BEAST_CUDA_TRY(ctx, cudaMemsetAsync(slots, 0xFF, panel_column_words<T>(kb, G) * kb * 8, st));
          BEAST_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((void*)k_panel<T>, G, 256, args, sm, st));
        }
        // interchanges inside the column block
        if ((rc = S.laswp(J0, j0, j0, j0 + kb))) break;
        if ((rc = S.laswp(j0 + kb, J1, j0, j0 + kb))) break;
      }
      // the in-block update (all rows below, mid-block columns) and, unpivoted, the mid
      // block's rows of the columns beyond it, as one L-shaped update
      const int64_t u_m0 = n - j0 - kb, u_n0 = M1 - j0 - kb, u_m1 = pivot ? 0 : M1 - j0 - kb,
                    u_n1 = pivot ? 0 : n - M1;
      bool applied = false, prepped = false;
      // lookahead for this panel: a full next panel inside the mid block with rows below it
      const bool next = la && kb == TRI && j0 + 2 * TRI <= M1 && n - j0 - kb > TRI;
      const int64_t skip = next ? TRI : 0;  // rows of the in-block update left to the second stream
      if (!pivot) {
        // no pivoting: diagonal block LU, then L21 = A21 U11^{-1} for every row below
        ProfScope ps(ctx, PK_PANEL, 8.0 * (double)M * kb * kb / 2, 0);
        constexpr int NS = TrsmTile<T>::NS;
        const int64_t rb = n - j0 - kb;
        T* dblk = apply_path ? reinterpret_cast<T*>(lu_dinv(ipiv, n)) + (j0 / TRI) * 2 * TRI * TRI : nullptr;
        ctx->launches += ahead ? 0 : 1;
        if (ahead)
          BEAST_CUDA_TRY(ctx, cudaStreamWaitEvent(st, ctx->la_ev[lu_par], 0));
        else if (apply_path)
          diag(sym, j0, kb, dblk, st);
        else
          k_getrf64<T><<<1, 256, getrf_sm, st>>>(A, lda, j0, kb, dinfo);
        if (apply_path && kb == TRI && rb > 0) {
          // L21 and U12 (every column to the right: no later interchange touches these rows)
          // in one launch, with the FP16 operands of the update below when it runs on the
          // tensor cores
          // (symmetric: L21 only, and the update is rows below x the rest of the mid block)
          const int64_t nBs = sym ? u_n0 : 0;
          prepped = sym ? (nBs > 0 && S.symgemm_tc(u_m0 - skip, nBs, kb, tcwork))
                        : (S.gemm2_runs(u_m0, u_n0, u_m1, u_n1, kb) && S.gemm2_tc(u_m0, u_n0, u_n1, kb, tcwork));
          void *Apv = nullptr, *Bpv = nullptr;
          float *isa = nullptr, *isb = nullptr;
          if (prepped) tc_gemm_operands(tcwork, u_m0, sym ? nBs : u_n0 + u_n1, kb, &Apv, &isa, &Bpv, &isb);
          const int nR = (int)((rb + 63) / 64);
          float2* Af = reinterpret_cast<float2*>(A);
          const float2* inv = reinterpret_cast<const float2*>(dblk);
          const int nBp = prepped ? (int)nBs : 0;
          if (next) {
            // second stream: block row j0 + 64 (its L rows and operands), then the next diagonal
            // block's update and elimination; it has to see this panel's elimination and the
            // previous in-block update (both on it, or both here)
            cudaStream_t ax = ctx->aux;
            if (ahead) {
              BEAST_CUDA_TRY(ctx, cudaStreamWaitEvent(ax, ctx->la_ev[3], 0));
            } else {
              BEAST_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[4], st));
              BEAST_CUDA_TRY(ctx, cudaStreamWaitEvent(ax, ctx->la_ev[4], 0));
            }
            k_panel_apply<64><<<1, 256, panel_apply_smem(), ax>>>(Af, lda, j0, n, inv, nR, static_cast<__half2*>(Apv),
                                                              isa, static_cast<__half2*>(Bpv), isb, nBp, 0);
            BEAST_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[2], ax));
            k_sym_diag_update<<<1, 256, sym_diag_update_smem(), ax>>>(Af, lda, j0 + TRI, TRI);
            diag(true, j0 + TRI, TRI, dblk + 2 * TRI * TRI, ax);
            lu_par ^= 1;
            BEAST_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[lu_par], ax));
            ctx->launches += 3;
            // here: the other block rows, then (after the second stream's operands) the update
            if (nR > 1) {
              k_panel_apply<64><<<(unsigned)(nR - 1), 256, panel_apply_smem(), st>>>(
                  Af, lda, j0, n, inv, nR, static_cast<__half2*>(Apv), isa, static_cast<__half2*>(Bpv), isb, nBp, 1);
              ctx->launches += 1;
            }
            BEAST_CUDA_TRY(ctx, cudaStreamWaitEvent(st, ctx->la_ev[2], 0));
          } else {
            // 32 systems per CTA: twice the CTAs of half the work, so that more warps hide the
            // shared-memory latency of the triangular products
            const int nR32 = (int)((rb + 31) / 32);
            // a programmatic dependent launch: its CTAs take the SMs the one-CTA elimination
            // leaves idle and load their rows while it runs
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(sym ? nR32 : 2 * nR32));
            cfg.blockDim = dim3(256);
            cfg.dynamicSmemBytes = panel_apply_smem();
            cfg.stream = st;
            cudaLaunchAttribute pdl[1];
            pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            pdl[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = pdl;
            cfg.numAttrs = 1;
            BEAST_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, k_panel_apply<32>, Af, lda, j0, n, inv, nR32,
                                                   static_cast<__half2*>(Apv), isa, static_cast<__half2*>(Bpv), isb,
                                                   nBp, 0));
            ctx->launches += 1;
          }
          applied = true;
        } else if (rb > 0) {
          k_trsm_tile<T, R, true><<<(unsigned)((rb + NS - 1) / NS), TrsmTile<T>::NT, trsm_tile_smem<T>(), st>>>(
              A, lda, j0, kb, j0 + kb, n);
          ctx->launches += 1;
        }
        BEAST_CUDA_TRY(ctx, cudaGetLastError());
      }
      // TRSM + GEMM for the rest of the block.  Unpivoted, no later interchange touches
      // these rows, so U12 of this panel is solved for every column to its right at once and
      // the block's rows of the columns beyond the block are updated here too (what the
      // pivoted path does per panel after the block).
      if (sym) {
        // with the next panel's elimination running on the second stream, the update's
        // persistent grid leaves two SMs to it (a CTA of the update needs a whole SM: one held
        // by the elimination would hold back the update's tiles until it ends)
        ctx->tc_sm_reserve = next ? 2 : 0;
        rc = S.symgemm(j0 + kb + skip, u_m0 - skip, j0 + kb, u_n0, j0, kb, false, tcwork, prepped, skip);
        ctx->tc_sm_reserve = 0;
        if (rc) break;
        if (next) BEAST_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[3], st));
        ahead = next;
        continue;
      }
      if (!applied && (rc = S.trsm(j0, kb, j0 + kb, pivot ? J1 : n))) break;
      if ((rc = S.gemm2(j0 + kb, u_m0, j0 + kb, u_n0, u_m1, u_n1, j0, kb, tcwork, prepped))) break;
    }
    if (rc) break;
    // mid-block update: rows below x the rest of the outer block, and the rest of the outer
    // block's rows x the columns beyond it (K = NB2; nothing when pivoting: NB2 = NB)
    if (M1 < J1) {
      rc = sym ? S.symgemm(M1, n - M1, M1, J1 - M1, M0, (int)(M1 - M0), false, tcwork)
               : S.gemm2(M1, n - M1, M1, J1 - M1, J1 - M1, n - J1, M0, (int)(M1 - M0), tcwork);
      if (rc) break;
    }
    }
    if (rc) break;
    // the block's interchanges on the columns left and right of it
    if (pivot) {
      if ((rc = S.laswp(0, J0, J0, J1))) break;
      if ((rc = S.laswp(J1, n, J0, J1))) break;
    }
    if (J1 < n && sym) {
      rc = S.symgemm(J1, n - J1, J1, n - J1, J0, (int)(J1 - J0), true, tcwork);
    } else if (J1 < n) {
      // U12 = L11^{-1} A12 (blocked: nb-row TRSM, then GEMM on the rows below inside the
      // block); done per panel above when unpivoted
      for (int64_t j0 = J0; pivot && j0 < J1 && rc == BEAST_OK; j0 += nb) {
        int kb = (int)std::min<int64_t>(nb, J1 - j0);
        if ((rc = S.trsm(j0, kb, J1, n))) break;
        if ((rc = S.gemm(j0 + kb, J1 - j0 - kb, J1, n - J1, j0, kb, tcwork))) break;
      }
      if (rc) break;
      // trailing update with K = NB
      rc = S.gemm(J1, n - J1, J1, n - J1, J0, (int)(J1 - J0), tcwork);
    }
  }
  if (la) {  // nothing of the second stream outlives the factorisation
    BEAST_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[4], ctx->aux));
    BEAST_CUDA_TRY(ctx, cudaStreamWaitEvent(st, ctx->la_ev[4], 0));
  }
  if (tcwork) cudaFreeAsync(tcwork, st);
  int hinfo[3] = {0, 0, 0};
  BEAST_CUDA_TRY(ctx, cudaMemcpyAsync(&hinfo[0], dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
  BEAST_CUDA_TRY(ctx, cudaMemcpyAsync(&hinfo[1], dstatus, sizeof(int), cudaMemcpyDeviceToHost, st));
  BEAST_CUDA_TRY(ctx, cudaMemcpyAsync(&hinfo[2], ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  BEAST_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  BEAST_CUDA_TRY(ctx, cudaFreeAsync(scr, st));
  if (rc) return rc;
  if (hinfo[1]) return beast_fail(ctx, BEAST_ERR_TIMEOUT, "LU panel: exchange timed out");
  if (hinfo[2] & 4) return beast_fail(ctx, BEAST_ERR_TIMEOUT, "LU tensor-core update: wait timed out");
  *info = hinfo[0];
  // the sequential interchanges ipiv[0..n) as one permutation: perm[i] = source row of row i
  std::vector<int> hp(n), perm(n);
  for (int64_t i = 0; i < n; ++i) perm[i] = (int)i;
  if (pivot) {
    BEAST_CUDA_TRY(ctx, cudaMemcpy(hp.data(), ipiv, n * sizeof(int), cudaMemcpyDeviceToHost));
    for (int64_t k = 0; k < n; ++k) std::swap(perm[k], perm[hp[k]]);
  } else {
    BEAST_CUDA_TRY(ctx, cudaMemcpy(ipiv, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice));
  }
  BEAST_CUDA_TRY(ctx, cudaMemcpy(ipiv + n, perm.data(), n * sizeof(int), cudaMemcpyHostToDevice));
  if (sym) {  // U = D L^T above the diagonal blocks
    const int64_t nbk = (n + 63) / 64;
    ProfScope ps(ctx, PK_CONVERT, (double)n * n * sizeof(T));
    if (nbk > 1) k_sym_upper<T><<<(unsigned)(nbk * (nbk - 1) / 2), 256, 0, st>>>(A, lda, n);
    BEAST_CUDA_TRY(ctx, cudaGetLastError());
  }
  // inverses of the diagonal blocks for the triangular solves (already written by k_lu_inv64
  // on the apply path)
  if (apply_path) return BEAST_OK;
  const size_t ism = (size_t)2 * 64 * 65 * sizeof(T);
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_invert_diag<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ism));
  k_invert_diag<T, R><<<(unsigned)((n + 63) / 64), 64, ism, st>>>(A, lda, n, reinterpret_cast<T*>(lu_dinv(ipiv, n)));
  BEAST_CUDA_TRY(ctx, cudaGetLastError());
  return BEAST_OK;
}

// P b -> forward sweep -> backward sweep for up to `batch` right-hand sides at a time: tmp (n values
// each) is the permuted right-hand side, then the backward sweep's output, copied back into b
template <typename T, typename RT>
int trsv_pair(beast_ctx* ctx, int64_t n, const T* A, int64_t lda, const int* perm, T* B, int64_t ldb,
              int64_t nrhs, T* tmp, int batch, const T* dinv) {
  cudaStream_t st = ctx->stream;
  const int nblk = (int)((n + 63) / 64);
  const size_t ring = TrsvRing<T>::BYTES;
  BEAST_CUDA_TRY(ctx, cudaFuncSetAttribute(k_trsv_wave<T, RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring));
  int occ = 0;
  BEAST_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_trsv_wave<T, RT>, 256, ring));
  const int cap = ctx->num_sms * std::max(occ, 1);
  int* status = ctx->d_flag;
  long long spin_max = ctx->trsv_spin_max > 0 ? ctx->trsv_spin_max : TRSV_SPIN_MAX;
  const unsigned ge = (unsigned)((n + 255) / 256);
  // a stale status from an earlier call must not be reported for this one
  BEAST_CUDA_TRY(ctx, cudaMemsetAsync(status, 0, sizeof(int), st));
  for (int64_t rr = 0; rr < nrhs; rr += batch) {
    const int nr = (int)std::min<int64_t>(std::min(batch, cap), nrhs - rr);
    batch = std::min(batch, cap);
    int per = std::max(1, std::min(nblk, cap / nr));
    T* b = B + rr * ldb;
    // the two triangular solves read the factors once: n^2 elements
    ProfScope ps(ctx, PK_TRSV, (double)n * n * sizeof(T), 5);
    const dim3 g2(ge, (unsigned)nr);
    int64_t ldt = n, ldbb = ldb;
    k_permute<T><<<g2, 256, 0, st>>>(b, ldb, tmp, n, perm, n);
    k_fill_sentinel<T><<<g2, 256, 0, st>>>(b, n, ldb);
    int lower = 1;
    const T* in = tmp;
    T* outp = b;
    {
      void* args[] = {&A, &lda, &n, &in, &ldt, &outp, &ldbb, &per, &lower, &status, &dinv, &spin_max};
      BEAST_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((void*)k_trsv_wave<T, RT>, per * nr, 256, args, ring, st));
    }
    k_fill_sentinel<T><<<g2, 256, 0, st>>>(tmp, n, n);
    lower = 0;
    in = b;
    outp = tmp;
    {
      void* args[] = {&A, &lda, &n, &in, &ldbb, &outp, &ldt, &per, &lower, &status, &dinv, &spin_max};
      BEAST_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((void*)k_trsv_wave<T, RT>, per * nr, 256, args, ring, st));
    }
    BEAST_CUDA_TRY(ctx, cudaMemcpy2DAsync(b, (size_t)ldb * sizeof(T), tmp, (size_t)n * sizeof(T), (size_t)n * sizeof(T), nr,
                                          cudaMemcpyDeviceToDevice, st));
  }
  BEAST_CUDA_TRY(ctx, cudaGetLastError());
  return BEAST_OK;
}

// right-hand sides solved side by side (each keeps at least 19 CTAs of one per SM)
constexpr int TRSV_BATCH = 8;
template <typename T, typename RT>
int lu_solve_t(beast_ctx* ctx, int64_t n, const T* A, int64_t lda, const int* perm, T* B,
               int64_t ldb, int64_t nrhs, const T* dinv) {
  cudaStream_t st = ctx->stream;
  if (nrhs <= 0) return BEAST_OK;
  T* tmp = nullptr;
  const int batch = (int)std::min<int64_t>(nrhs, TRSV_BATCH);
  BEAST_CUDA_TRY(ctx, cudaMallocAsync(&tmp, (size_t)n * batch * sizeof(T), st));
  int rc = trsv_pair<T, RT>(ctx, n, A, lda, perm, B, ldb, nrhs, tmp, batch, dinv);
  BEAST_CUDA_TRY(ctx, cudaFreeAsync(tmp, st));
  return rc;
}

// ---- allocation-free triangular solve ----------------------------------------------------
// Scratch of beast_lu_solve_noalloc: one right-hand side of up to NOALLOC_MAX_N complex128
// values (the permuted right-hand side, then the backward sweep's output).
// Held by every GPU that loads the library, for the life of the process; calls take turns on it.
constexpr int64_t NOALLOC_MAX_N = 65536;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_MAX_N * 16];

template <typename T, typename RT>
int lu_solve_fixed_scratch(beast_ctx* ctx, int64_t n, const T* A, int64_t lda, const int* perm, T* B,
                           int64_t ldb, int64_t nrhs, unsigned char* scratch, const T* dinv) {
  // the scratch keeps the previous call's values; every value it is read for is written
  // first in this call (the permutation, then the sentinel fill)
  return trsv_pair<T, RT>(ctx, n, A, lda, perm, B, ldb, nrhs, reinterpret_cast<T*>(scratch), 1, dinv);
}

}  // namespace

cudaError_t gemm64_tiles(const int2* list, const int* count, double2* C, int64_t ldc, const double2* A, int64_t lda,
                         const double2* B, int64_t ldb, int64_t m, int64_t n, int k, int grid, cudaStream_t st) {
  static_assert(GT == 64, "tc_gemm64.cu lists blocks of 64");
  k_gemm_tiles<<<(unsigned)grid, 256, 0, st>>>(list, count, C, ldc, A, lda, B, ldb, m, n, k);
  return cudaGetLastError();
}

int lu_factor_dev(beast_ctx* ctx, int64_t n, void* A, int64_t lda, int dtype, int* ipiv, int* info,
                  bool pivot, bool sym) {
  if (dtype == BEAST_C64) return lu_factor_t<float2, float>(ctx, n, (float2*)A, lda, ipiv, info, pivot, sym);
  return lu_factor_t<double2, double>(ctx, n, (double2*)A, lda, ipiv, info, pivot, false);
}

double asym_sample(beast_ctx* ctx, int64_t n, const void* A, int64_t lda, int dtype) {
  if (n < 2) return 0.0;
  const int64_t s = std::max<int64_t>(1, n / 1400);  // about 10^6 pairs
  double* d = nullptr;
  if (cudaMallocAsync(&d, 2 * sizeof(double), ctx->stream) != cudaSuccess) return 1.0;
  cudaMemsetAsync(d, 0, 2 * sizeof(double), ctx->stream);
  if (dtype == BEAST_C64)
    k_asym_sample<float2><<<1024, 256, 0, ctx->stream>>>((const float2*)A, lda, n, s, d);
  else
    k_asym_sample<double2><<<1024, 256, 0, ctx->stream>>>((const double2*)A, lda, n, s, d);
  double h[2] = {0, 0};
  cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream);
  cudaFreeAsync(d, ctx->stream);
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return 1.0;
  return h[1] > 0 ? std::sqrt(2.0 * h[0] / h[1]) : 0.0;
}

// ipiv holds 2n ints: the pivots, then the permutation built by lu_factor_dev
int lu_solve_dev(beast_ctx* ctx, int64_t n, const void* A, int64_t lda, int dtype, const int* ipiv,
                 void* B, int64_t ldb, int64_t nrhs) {
  if (dtype == BEAST_C64)
    return lu_solve_t<float2, float>(ctx, n, (const float2*)A, lda, ipiv + n, (float2*)B, ldb, nrhs,
                                     (const float2*)lu_dinv(ipiv, n));
  return lu_solve_t<double2, double>(ctx, n, (const double2*)A, lda, ipiv + n, (double2*)B, ldb, nrhs,
                                     (const double2*)lu_dinv(ipiv, n));
}

// waits for the context stream and reports a triangular-solve flag wait that ran out (status
// bit 8, cleared at the start of every solve by trsv_pair)
int trsv_check(beast_ctx* ctx) {
  BEAST_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  int status = 0;
  BEAST_CUDA_TRY(ctx, cudaMemcpy(&status, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost));
  if (status & 8) return beast_fail(ctx, BEAST_ERR_TIMEOUT, "triangular solve: flag wait timed out");
  return BEAST_OK;
}

// slabs of an n x n matvec: the most slabs (32 below order 2048, where the sum over the slabs
// counts) whose CTAs fill their waves to 97%, else the count that fills them best.  Many short CTAs
// even out the ends of the load streams: order 7213 takes 227 us in one full wave of 31 slabs and
// 205 us in two.
static int mv_slabs(int64_t n, int64_t row_blocks, const void* kernel) {
  int dev = 0, sms = 1, occ = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 128, 0) != cudaSuccess || occ < 1) occ = 1;
  const double cap = (double)sms * occ;
  int best = 1;
  double fill = -1.0;
  for (int s = n < 2048 ? 32 : MV_MAX_SLABS; s >= 8; --s) {
    if (s > n) continue;
    const double w = (double)row_blocks * s / cap, f = w / std::ceil(w);
    if (f >= 0.97) return s;
    if (f > fill) {
      fill = f;
      best = s;
    }
  }
  return best;
}

// the partial sums of A x over column slabs into part [slabs][n][2]; returns the slab count
static int gemv_partial(int64_t n, const void* A, int64_t lda, int a_c64, const float4* xs, double* part,
                        cudaStream_t st) {
  const bool pair = a_c64 && lda % 2 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  const int rows = a_c64 && !pair ? 128 : 256;
  const int64_t rb = (n + rows - 1) / rows;
  const void* kern = !a_c64 ? (const void*)k_gemv_partial_c128_df
                            : (pair ? (const void*)k_gemv_partial_c64_df2 : (const void*)k_gemv_partial_c64_df);
  const int slabs = mv_slabs(n, rb, kern);
  dim3 g((unsigned)rb, (unsigned)slabs);
  if (!a_c64)
    k_gemv_partial_c128_df<<<g, 128, 0, st>>>(n, (const double2*)A, lda, xs, part);
  else if (pair)
    k_gemv_partial_c64_df2<<<g, 128, 0, st>>>(n, (const float2*)A, lda, xs, part);
  else
    k_gemv_partial_c64_df<<<g, 128, 0, st>>>(n, (const float2*)A, lda, xs, part);
  return slabs;
}

// scratch per call from the device's stream-ordered pool (cheap once the pool holds memory;
// nothing shared between contexts, streams or devices)
cudaError_t gemv_dev(int64_t n, const void* A, int64_t lda, int a_c64, const double* x, double* y,
                     double alpha, double beta, cudaStream_t st) {
  const size_t need = (size_t)MV_MAX_SLABS * n * 2 * sizeof(double) + (size_t)n * sizeof(float4) + 256;
  double* part = nullptr;
  cudaError_t e = cudaMallocAsync(&part, need, st);
  if (e != cudaSuccess) return e;
  float4* xs = reinterpret_cast<float4*>(part + (size_t)MV_MAX_SLABS * n * 2);
  k_split_x<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, xs);
  const int slabs = gemv_partial(n, A, lda, a_c64, xs, part, st);
  k_gemv_reduce<<<(unsigned)((n + 63) / 64), 256, 0, st>>>(n, slabs, part, y, alpha, beta);
  e = cudaGetLastError();
  cudaFreeAsync(part, st);
  return e;
}

// ---- GMRES on the device: the workspace of one solve and one Arnoldi step
size_t gmres_work_bytes(int64_t n, int m) {
  const size_t nb = (size_t)((n + GM_ROWS - 1) / GM_ROWS);
  return (size_t)MV_MAX_SLABS * n * 16 + (size_t)n * 16 + nb * 2 * (m + 1) * 8 + 4096;
}
// v_k = w / |w| (|w|^2 at norm2) and its matvec's slabs
cudaError_t gmres_matvec(int64_t n, const void* A, int64_t lda, int a_c64, const double* w, const double* norm2,
                         double* vk, void* work, int* slabs, cudaStream_t st) {
  double* slab = static_cast<double*>(work);
  float4* xs = reinterpret_cast<float4*>(slab + (size_t)MV_MAX_SLABS * n * 2);
  k_gm_next<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, w, norm2, vk, xs);
  *slabs = gemv_partial(n, A, lda, a_c64, xs, slab, st);
  return cudaGetLastError();
}
// w = A v_k from the slabs, orthogonalised twice against v_0 .. v_k: out = h1 (k + 1 complex), h2, |w|^2
cudaError_t gmres_orthogonalise(int64_t n, int k, int slabs, const double* V, double* w, void* work,
                                unsigned int* count, double* out, cudaStream_t st) {
  double* slab = static_cast<double*>(work);
  double* part = slab + (size_t)MV_MAX_SLABS * n * 2 + (size_t)n * 2;
  const unsigned nb = (unsigned)((n + GM_ROWS - 1) / GM_ROWS);
  double* h2 = out + 2 * (k + 1);
  k_gm_step<<<nb, GM_THREADS, 0, st>>>(0, n, k + 1, slabs, slab, V, w, nullptr, part, count, out);
  k_gm_step<<<nb, GM_THREADS, 0, st>>>(1, n, k + 1, slabs, slab, V, w, out, part, count, h2);
  k_gm_step<<<nb, GM_THREADS, 0, st>>>(2, n, k + 1, slabs, slab, V, w, h2, part, count, h2 + 2 * (k + 1));
  return cudaGetLastError();
}

cudaError_t copy_lower_c64(int64_t n, const void* A, int64_t lda, void* F, int64_t ldf, cudaStream_t st) {
  const int vec = (lda % 2 == 0 && ldf % 2 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(F) & 15) == 0)
                      ? 1
                      : 0;
  if (n <= 0) return cudaSuccess;
  k_copy_lower_c64<<<(unsigned)std::min<int64_t>(n, 65535), 256, 0, st>>>(n, (const float2*)A, lda, (float2*)F, ldf,
                                                                          vec);
  return cudaGetLastError();
}

cudaError_t convert_lower_c128_to_c64(int64_t n, const void* A, int64_t lda, void* F, int64_t ldf, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_convert_lower_c128<<<(unsigned)std::min<int64_t>(n, 65535), 256, 0, st>>>(n, (const double2*)A, lda, (float2*)F,
                                                                              ldf);
  return cudaGetLastError();
}
cudaError_t convert_c128_to_c64(int64_t rows, int64_t cols, const double* src, int64_t lds, float* dst,
                                int64_t ldd, cudaStream_t st) {
  dim3 g((unsigned)((rows + 255) / 256), (unsigned)std::min<int64_t>(cols, 65535));
  k_c128_to_c64<<<g, 256, 0, st>>>(rows, cols, src, lds, dst, ldd);
  return cudaGetLastError();
}
cudaError_t convert_c64_to_c128(int64_t rows, int64_t cols, const float* src, int64_t lds, double* dst,
                                int64_t ldd, cudaStream_t st) {
  dim3 g((unsigned)((rows + 255) / 256), (unsigned)std::min<int64_t>(cols, 65535));
  k_c64_to_c128<<<g, 256, 0, st>>>(rows, cols, src, lds, dst, ldd);
  return cudaGetLastError();
}
cudaError_t vec_axpy(int64_t n, double ar, double ai, const double* x, double* y, cudaStream_t st) {
  k_axpy<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, ar, ai, x, y);
  return cudaGetLastError();
}
cudaError_t vec_copy(int64_t n, const double* x, double* y, cudaStream_t st) {
  return cudaMemcpyAsync(y, x, (size_t)n * 2 * sizeof(double), cudaMemcpyDeviceToDevice, st);
}
cudaError_t vec_norm2(int64_t n, const double* x, double* out, cudaStream_t st) {
  double* npart = nullptr;
  cudaError_t e = cudaMallocAsync(&npart, 256 * sizeof(double), st);
  if (e != cudaSuccess) return e;
  k_norm2_part<<<256, 256, 0, st>>>(n, x, npart);
  k_sum_part<<<1, 256, 0, st>>>(256, npart, out);
  e = cudaGetLastError();
  cudaFreeAsync(npart, st);
  return e;
}
cudaError_t vec_gemv_sub(int64_t n, int m, const double* V, int64_t ldv, const double* h, double* w,
                         cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  k_gemv_sub<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, m, V, ldv, h, w);
  return cudaGetLastError();
}

// Device address of the fixed scratch, looked up once per device with that device current.
// (In host code the array's name is only a host-side stand-in, never a device address.)
static unsigned char* noalloc_scratch(beast_ctx* ctx) {
  static std::mutex mtx;
  static unsigned char* addr[64] = {nullptr};
  std::lock_guard<std::mutex> lk(mtx);
  if (ctx->device < 0 || ctx->device >= 64) return nullptr;
  if (!addr[ctx->device]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return nullptr;
    addr[ctx->device] = static_cast<unsigned char*>(p);
  }
  return addr[ctx->device];
}

extern "C" int beast_lu_solve_noalloc(beast_ctx* ctx, const beast_lu* lu, int64_t nrhs, void* B,
                                      int64_t ldb) {
  if (!ctx) return BEAST_ERR_ARG;
  if (!lu || !B || nrhs < 0 || ldb < lu->n)
    return beast_fail(ctx, BEAST_ERR_ARG, "invalid solve arguments");
  if (lu->n > NOALLOC_MAX_N)
    return beast_fail(ctx, BEAST_ERR_ARG,
                      "beast_lu_solve_noalloc: n = " + std::to_string(lu->n) +
                          " exceeds the fixed scratch limit of " + std::to_string(NOALLOC_MAX_N) +
                          " unknowns; use beast_lu_solve");
  BEAST_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  unsigned char* scratch = noalloc_scratch(ctx);
  if (!scratch) return beast_fail(ctx, BEAST_ERR_CUDA, "cudaGetSymbolAddress of the fixed scratch failed");
  // one call at a time per GPU (contexts and host threads share the scratch); every way out has waited for the stream
  static std::mutex turn[64];
  std::lock_guard<std::mutex> lk(turn[ctx->device]);
  int rc;
  if (lu->dtype == BEAST_C64)
    rc = lu_solve_fixed_scratch<float2, float>(ctx, lu->n, (const float2*)lu->A, lu->lda, lu->ipiv + lu->n,
                                               (float2*)B, ldb, nrhs, scratch,
                                               (const float2*)lu_dinv(lu->ipiv, lu->n));
  else
    rc = lu_solve_fixed_scratch<double2, double>(ctx, lu->n, (const double2*)lu->A, lu->lda,
                                                 lu->ipiv + lu->n, (double2*)B, ldb, nrhs, scratch,
                                                 (const double2*)lu_dinv(lu->ipiv, lu->n));
  if (rc) {
    cudaStreamSynchronize(ctx->stream);
    return rc;
  }
  return trsv_check(ctx);
}
