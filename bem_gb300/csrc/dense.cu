// Dense complex linear algebra, complex128 (plain path) and complex64 (mixed path):
//   LU with partial pivoting (the zgetrf of inverse(), src/util/DenseMatrix.cpp:65-77),
//   the corresponding solve, and a complex GEMM (src/util/MatrixOperations.cpp:70-74).
//
// All matrices are column-major with interleaved (re, im) values, as the
// reference's ComplexDenseMatrix stores them (src/util/DenseMatrix.h:195-198).
//
// LU: right-looking, panel width 64 (complex128) or 128 (complex64, in pairs).  A
// panel is factored by one thread-block cluster with its rows in registers
// (panel_cluster_kernel; a cooperative grid beyond 16384 rows), then the row
// interchanges are applied outside the panel, the U12 block is solved with the
// unit-lower L11 (tri_block_kernel) and the trailing matrix is updated by the
// complex GEMM.
// Pivot choice is LAPACK's: the first row of largest |re|+|im| (izamax).
#include "bemgpu_internal.h"
#include "panel_slots.h"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace {

constexpr int NB = 64;  // panel width of the FP64 LU and of the blocked solves
constexpr int NB_MAX = 128;  // widest LU panel (complex64: LuCfg<float>)
// LU panel width per type: complex64 uses 128-wide panels so that the trailing
// updates are K = 128 tensor-core products (half the passes over the trailing
// matrix of 64-wide panels); complex128 keeps 64 (its diagonal block must fit
// the triangular-solve kernel's shared memory).
template <typename T>
struct LuCfg {
  static constexpr int NBL = 64;
};
template <>
struct LuCfg<float> {
  static constexpr int NBL = 128;
};

template <typename T>
struct V2;
template <>
struct V2<double> {
  typedef double2 type;
  __device__ __forceinline__ static double2 make(double a, double b) { return make_double2(a, b); }
};
template <>
struct V2<float> {
  typedef float2 type;
  __device__ __forceinline__ static float2 make(float a, float b) { return make_float2(a, b); }
};

template <typename T>
struct cx {
  T r, i;
};
template <typename T>
__device__ __forceinline__ cx<T> cmul(cx<T> a, cx<T> b) {
  return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r};
}
template <typename T>
__device__ __forceinline__ cx<T> cld(const T *A, int64_t idx) {
  typename V2<T>::type v = reinterpret_cast<const typename V2<T>::type *>(A)[idx];
  return {v.x, v.y};
}
template <typename T>
__device__ __forceinline__ void cst(T *A, int64_t idx, cx<T> v) {
  reinterpret_cast<typename V2<T>::type *>(A)[idx] = V2<T>::make(v.r, v.i);
}
template <typename T>
__device__ __forceinline__ cx<T> crecip(cx<T> a) {
  T d = a.r * a.r + a.i * a.i;
  return {a.r / d, -a.i / d};
}

// ---------------- panel factorization ----------------
struct PivCand {
  double val;
  int idx;
  int pad;
};

constexpr int PANEL_THREADS = 256;

// Step jj of the panel [k0, k0+w): applies the pending scale + rank-1 update
// of column jj-1 to rows >= k0+jj, then selects and swaps the pivot of column jj.
// With jj == w it only applies the final scale of column w-1.
template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) panel_step_kernel(T *A, int64_t lda, int n, int k0, int w, int jj,
                                                                   int *ipiv, int *info, PivCand *cand,
                                                                   unsigned int *counter) {
  const int r0 = k0 + jj;  // first active row
  const int nrows = n - r0;
  double bestv = -1.0;
  int besti = 0x7fffffff;
  if (jj > 0) {
    const int pr = k0 + jj - 1;  // pivot row/column of the previous step
    const cx<T> piv = cld(A, pr + lda * (int64_t)pr);
    const bool zero = (piv.r == T(0) && piv.i == T(0));
    const cx<T> rp = zero ? cx<T>{0, 0} : crecip(piv);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nrows; t += gridDim.x * blockDim.x) {
      const int r = r0 + t;
      cx<T> l = cld(A, r + lda * (int64_t)pr);
      if (!zero) {
        l = cmul(l, rp);
        cst(A, r + lda * (int64_t)pr, l);
      }
      for (int c = jj; c < w; c++) {
        const int64_t col = (int64_t)(k0 + c) * lda;
        const cx<T> u = cld(A, pr + col);
        cx<T> a = cld(A, r + col);
        a.r -= l.r * u.r - l.i * u.i;
        a.i -= l.r * u.i + l.i * u.r;
        cst(A, r + col, a);
        if (c == jj) {
          const double v = fabs((double)a.r) + fabs((double)a.i);
          if (v > bestv || (v == bestv && r < besti)) { bestv = v; besti = r; }
        }
      }
    }
  } else {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nrows; t += gridDim.x * blockDim.x) {
      const int r = r0 + t;
      const cx<T> a = cld(A, r + lda * (int64_t)(k0));
      const double v = fabs((double)a.r) + fabs((double)a.i);
      if (v > bestv || (v == bestv && r < besti)) { bestv = v; besti = r; }
    }
  }
  if (jj == w) return;  // final scale only
  // block argmax
  __shared__ double sv[PANEL_THREADS];
  __shared__ int si[PANEL_THREADS];
  __shared__ bool last;
  sv[threadIdx.x] = bestv;
  si[threadIdx.x] = besti;
  __syncthreads();
  for (int s = PANEL_THREADS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      const double v2 = sv[threadIdx.x + s];
      const int i2 = si[threadIdx.x + s];
      if (v2 > sv[threadIdx.x] || (v2 == sv[threadIdx.x] && i2 < si[threadIdx.x])) {
        sv[threadIdx.x] = v2;
        si[threadIdx.x] = i2;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    cand[blockIdx.x] = {sv[0], si[0], 0};
    __threadfence();
    const unsigned int prev = atomicAdd(counter, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // last CTA: global argmax, record the pivot, swap rows inside the panel
  __shared__ int piv_row;
  if (threadIdx.x == 0) {
    double bv = -1.0;
    int bi = r0;
    for (int b = 0; b < gridDim.x; b++) {
      const volatile PivCand *vc = (const volatile PivCand *)cand + b;
      const double cv = vc->val;
      const int ci = vc->idx;
      if (ci == 0x7fffffff) continue;
      if (cv > bv || (cv == bv && ci < bi)) { bv = cv; bi = ci; }
    }
    if (bv == 0.0) {
      bi = r0;
      if (*info == 0) *info = r0 + 1;
    }
    ipiv[r0] = bi;
    piv_row = bi;
    *counter = 0u;
  }
  __syncthreads();
  const int p = piv_row;
  if (p != r0) {
    for (int c = threadIdx.x; c < w; c += blockDim.x) {
      const int64_t col = (int64_t)(k0 + c) * lda;
      const cx<T> a = cld(A, r0 + col), b = cld(A, p + col);
      cst(A, r0 + col, b);
      cst(A, p + col, a);
    }
  }
}

// Where the content of position d comes from once the interchanges ipiv[k1..k2)
// (in order, as laswp applies them) are done: d led back through them.  piv holds
// ipiv[k1..k2) in shared memory.
__device__ __forceinline__ int interchange_source(const int *piv, int k1, int k2, int d) {
  int x = d;
#pragma unroll 8
  for (int k = k2 - 1; k >= k1; k--) {
    const int p = piv[k - k1];
    x = x == k ? p : x == p ? k : x;
  }
  return x;
}

// The row interchanges ipiv[0..n) as one permutation: perm[i] = the row whose
// content ends in row i, and its inverse.  Every row leads itself back (n steps
// of shared-memory broadcasts: ~20 us at n = 7680, where one thread's replay of
// the swaps took 295).
constexpr int PERM_MAX_N = 49152;  // 192 KB of shared memory; beyond, the pivots are read from global memory

__global__ void __launch_bounds__(128) perm_from_ipiv_kernel(const int *__restrict__ ipiv, int n, int *__restrict__ perm,
                                                             int *__restrict__ inverse, int staged) {
  extern __shared__ int perm_smem[];
  if (staged)
    for (int i = threadIdx.x; i < n; i += blockDim.x) perm_smem[i] = ipiv[i];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = staged ? interchange_source(perm_smem, 0, n, i) : interchange_source(ipiv, 0, n, i);
  perm[i] = s;
  inverse[s] = i;
}

// out[i, c] = B[perm[i], c] for complex64 column-major B (n x ncols).
__global__ void gather_rows_c64_kernel(const float *__restrict__ B, int64_t ldb, const int *__restrict__ perm, int n,
                                       float *__restrict__ out, int64_t ldo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t c = blockIdx.y;
  if (i >= n) return;
  reinterpret_cast<float2 *>(out)[i + ldo * c] = reinterpret_cast<const float2 *>(B)[perm[i] + ldb * c];
}

// The interchanges of a panel of at most LASWP_MAXW rows on columns [c0, c1):
// thread t of a CTA has one of the at most 2 w touched rows (the panel's own and
// the pivot rows below it), knows its source (interchange_source), and moves that
// entry of LASWP_COLS columns at a time, all loads before the stores.  Each entry
// moves once.  (One warp's replay of the swaps took most of the 22 us of a launch
// at n = 7680; this takes ~6.)
constexpr int LASWP_MAXW = 128;
constexpr int LASWP_COLS = 8;

template <typename T>
__global__ void __launch_bounds__(2 * LASWP_MAXW)
    laswp_perm_kernel(T *A, int64_t lda, int c0, int c1, int k1, int k2, const int *ipiv) {
  __shared__ int piv[LASWP_MAXW];
  const int t = threadIdx.x, m = k2 - k1;
  for (int k = t; k < m; k += blockDim.x) piv[k] = ipiv[k1 + k];
  __syncthreads();
  const int d = t < m ? k1 + t : t < 2 * m ? piv[t - m] : -1;
  const bool mine = t < m || (t < 2 * m && d >= k2);
  const int src = mine ? interchange_source(piv, k1, k2, d) : d;
  const bool on = mine && src != d;
  for (int c = c0 + blockIdx.x * LASWP_COLS; c < c1; c += gridDim.x * LASWP_COLS) {
    cx<T> v[LASWP_COLS];
#pragma unroll
    for (int e = 0; e < LASWP_COLS; e++)
      if (on && c + e < c1) v[e] = cld(A, src + (int64_t)(c + e) * lda);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < LASWP_COLS; e++)
      if (on && c + e < c1) cst(A, d + (int64_t)(c + e) * lda, v[e]);
  }
}

// ---------------- cooperative panel factorization ----------------
// The whole panel [k0, k0 + w) in one cooperative launch: CTA g keeps rows
// [k0 + g chunk, k0 + (g+1) chunk) of the panel in shared memory (row-major),
// and per column j: (1) each CTA publishes its local pivot candidate (value,
// row, the row's w entries) and, if it owns the diagonal row, that row;
// (2) one grid barrier; (3) every CTA reduces the G candidates to the same
// pivot, the owners of the diagonal and pivot rows exchange them, and each
// CTA scales column j and applies the rank-1 update to its own rows.  One
// barrier per column (candidate slots double-buffered by column parity); the
// barrier's spin is bounded and sets *err when it runs out.  Same pivots and
// arithmetic as the one-launch-per-column kernel above.
constexpr int COOP_THREADS = 256;
constexpr unsigned COOP_SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ void arrive_release_u32(unsigned *p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename T>
__global__ void __launch_bounds__(COOP_THREADS)
    panel_coop_kernel(T *A, int64_t lda, int n, int k0, int w, int chunk, int *ipiv, int *info, T *cval,
                      int *crow, T *cdata_raw, T *drow_raw, unsigned *counter, int *err,
                      unsigned long long *best, int64_t strideA) {
  typedef typename V2<T>::type T2;
  extern __shared__ __align__(16) unsigned char coop_smem[];
  {
    // a batch of equal-size matrices (blockIdx.y): its own matrix, pivots,
    // candidate slots and barrier; the CTAs of different matrices never wait
    // on one another
    const int64_t bb = blockIdx.y;
    A += bb * strideA;
    ipiv += bb * n;
    info += bb;
    cval += bb * 2 * gridDim.x;
    crow += bb * 2 * gridDim.x;
    cdata_raw += bb * 2 * 2 * (int64_t)gridDim.x * w;
    drow_raw += bb * 2 * 2 * (int64_t)w;
    counter += bb;
    best += 4 * bb;
  }
  T2 *P = reinterpret_cast<T2 *>(coop_smem);  // chunk x w, P[i * w + c]
  T2 *prow = P + (int64_t)chunk * w;           // the pivot (U) row of the current column
  T2 *A2 = reinterpret_cast<T2 *>(A);
  T2 *cdata = reinterpret_cast<T2 *>(cdata_raw);
  T2 *drow = reinterpret_cast<T2 *>(drow_raw);
  __shared__ T red_v[COOP_THREADS / 32];
  __shared__ int red_i[COOP_THREADS / 32], red_w[COOP_THREADS / 32];
  __shared__ int s_row, s_win;
  __shared__ bool s_abort, s_zero;
  const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rbeg = k0 + g * chunk, rend = min(n, rbeg + chunk);
  const int nloc = max(0, rend - rbeg);
  for (int idx = tid; idx < nloc * w; idx += COOP_THREADS) {
    const int i = idx % nloc, c = idx / nloc;
    P[i * w + c] = A2[(rbeg + i) + lda * (int64_t)(k0 + c)];
  }
  if (tid == 0) s_abort = false;
  __syncthreads();
  for (int j = 0; j < w; j++) {
    const int dr = k0 + j, par = j & 1;
    // (1) local candidate: first row of largest |re| + |im| in column j, rows >= dr
    T bv = T(-1);
    int bi = 0x7fffffff;
    for (int i = tid; i < nloc; i += COOP_THREADS) {
      const int r = rbeg + i;
      if (r < dr) continue;
      const T2 a = P[i * w + j];
      const T v = fabs(a.x) + fabs(a.y);
      if (v > bv || (v == bv && r < bi)) {
        bv = v;
        bi = r;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const T v2 = __shfl_xor_sync(0xffffffffu, bv, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
      if (v2 > bv || (v2 == bv && i2 < bi)) {
        bv = v2;
        bi = i2;
      }
    }
    if (lane == 0) {
      red_v[wid] = bv;
      red_i[wid] = bi;
    }
    __syncthreads();
    // warp 0 publishes the CTA's candidate (value, row, row data) and the
    // diagonal row, then its lane 0 takes the grid barrier; the other warps
    // wait at the CTA barrier that follows
    if (wid == 0) {
      if (lane == 0) {
        for (int q = 1; q < COOP_THREADS / 32; q++)
          if (red_v[q] > bv || (red_v[q] == bv && red_i[q] < bi)) {
            bv = red_v[q];
            bi = red_i[q];
          }
        if constexpr (sizeof(T) == 4) {
          // complex64: the candidate goes into one packed key per column (slot
          // j % 3), magnitude bits over the complemented row, so the largest
          // key is the largest |re| + |im| and, among equal ones, the first row
          if (bi != 0x7fffffff)
            atomicMax(best + j % 3, ((unsigned long long)__float_as_uint((float)bv) << 32) |
                                        (unsigned long long)(0xffffffffu - (unsigned)bi));
        } else {
          cval[par * G + g] = bv;
          crow[par * G + g] = bi;
        }
      }
      bi = __shfl_sync(0xffffffffu, bi, 0);
      if (bi != 0x7fffffff)
        for (int c = lane; c < w; c += 32) cdata[(int64_t)(par * G + g) * w + c] = P[(bi - rbeg) * w + c];
      if (dr >= rbeg && dr < rend)
        for (int c = lane; c < w; c += 32) drow[par * w + c] = P[(dr - rbeg) * w + c];
      __syncwarp();
      // (2) grid barrier
      if (lane == 0) {
        // the warp's publishing writes (ordered before by the warp barrier and
        // the fence) are released with the arrival; the acquire load orders
        // the reads after the CTA barrier below
        __threadfence();
        arrive_release_u32(counter);
        const unsigned target = (unsigned)G * (unsigned)(j + 1);
        unsigned it = 0;
        while (ld_acquire_u32(counter) < target) {
          if (++it > COOP_SPIN_LIMIT) {
            atomicExch(err, 1);
            s_abort = true;
            break;
          }
        }
      }
    }
    __syncthreads();
    if (s_abort) return;
    // (3) the pivot, the pivot (U) row into shared memory, and the interchange
    if constexpr (sizeof(T) == 4) {
      if (wid == 0) {
        int row = 0, win = -1, zi = 0;
        if (lane == 0) {
          const unsigned long long key = __ldcg(best + j % 3);
          // slot (j - 1) % 3 was read by every CTA before it arrived here; it
          // is next used at column j + 2, after the barrier this CTA passes later
          if (g == 0 && j >= 1) atomicExch(best + (j - 1) % 3, 0ull);
          zi = (key >> 32) == 0ull;
          row = zi ? dr : (int)(0xffffffffu - (unsigned)(key & 0xffffffffull));
          win = zi ? -1 : (row - k0) / chunk;
          if (g == 0) {
            ipiv[dr] = row;
            if (zi && *info == 0) *info = dr + 1;
          }
          s_zero = zi != 0;
          s_row = row;
        }
        row = __shfl_sync(0xffffffffu, row, 0);
        win = __shfl_sync(0xffffffffu, win, 0);
        for (int c = lane; c < w; c += 32)
          prow[c] = (row == dr || win < 0) ? __ldcg(drow + par * w + c)
                                           : __ldcg(cdata + (int64_t)(par * G + win) * w + c);
        __syncwarp();
        if (row != dr) {
          if (dr >= rbeg && dr < rend)
            for (int c = lane; c < w; c += 32) P[(dr - rbeg) * w + c] = prow[c];
          if (row >= rbeg && row < rend)
            for (int c = lane; c < w; c += 32) P[(row - rbeg) * w + c] = __ldcg(drow + par * w + c);
        }
      }
      __syncthreads();
    } else {
    bv = T(-1);
    bi = 0x7fffffff;
    int bw = 0;
    if constexpr (sizeof(T) == 8) {
    for (int q = tid; q < G; q += COOP_THREADS) {
      const T v = __ldcg(cval + par * G + q);
      const int r = __ldcg(crow + par * G + q);
      if (r == 0x7fffffff) continue;
      if (v > bv || (v == bv && r < bi)) {
        bv = v;
        bi = r;
        bw = q;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const T v2 = __shfl_xor_sync(0xffffffffu, bv, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
      const int w2 = __shfl_xor_sync(0xffffffffu, bw, o);
      if (v2 > bv || (v2 == bv && i2 < bi)) {
        bv = v2;
        bi = i2;
        bw = w2;
      }
    }
    if (lane == 0) {
      red_v[wid] = bv;
      red_i[wid] = bi;
      red_w[wid] = bw;
    }
    __syncthreads();
    if (tid == 0) {
      int win = bw;
      for (int q = 1; q < COOP_THREADS / 32; q++)
        if (red_v[q] > bv || (red_v[q] == bv && red_i[q] < bi)) {
          bv = red_v[q];
          bi = red_i[q];
          win = red_w[q];
        }
      if (bi == 0x7fffffff) win = -1;
      const bool zero = !(bv > T(0));
      if (zero) bi = dr;
      s_zero = zero;
      s_row = bi;
      s_win = win;
      if (g == 0) {
        ipiv[dr] = bi;
        if (zero && *info == 0) *info = dr + 1;
      }
    }
    __syncthreads();
    }
      const int p = s_row;
      for (int c = tid; c < w; c += COOP_THREADS) {
        T2 v;
        if (p == dr || s_win < 0) {
          const T2 *src = drow + par * w + c;
          v = __ldcg(src);
        } else {
          v = __ldcg(cdata + (int64_t)(par * G + s_win) * w + c);
        }
        prow[c] = v;
      }
      __syncthreads();
      if (p != dr) {
        if (dr >= rbeg && dr < rend)
          for (int c = tid; c < w; c += COOP_THREADS) P[(dr - rbeg) * w + c] = prow[c];
        if (p >= rbeg && p < rend)
          for (int c = tid; c < w; c += COOP_THREADS) P[(p - rbeg) * w + c] = __ldcg(drow + par * w + c);
      }
      __syncthreads();
    }
    // scale column j below the diagonal and the rank-1 update of columns > j,
    // one warp per row (the row's multiplier is read before it is overwritten)
    const bool zero = s_zero;
    const T2 pv = prow[j];
    const cx<T> rp = zero ? cx<T>{0, 0} : crecip(cx<T>{pv.x, pv.y});
    for (int i = wid; i < nloc; i += COOP_THREADS / 32) {
      if (rbeg + i <= dr) continue;
      const T2 a0 = P[i * w + j];
      T2 l = a0;
      if (!zero) {
        const cx<T> ls = cmul(cx<T>{a0.x, a0.y}, rp);
        l = V2<T>::make(ls.r, ls.i);
      }
      __syncwarp();
      if (lane == 0) P[i * w + j] = l;
      for (int c = j + 1 + lane; c < w; c += 32) {
        const T2 u = prow[c];
        T2 a = P[i * w + c];
        a.x -= l.x * u.x - l.y * u.y;
        a.y -= l.x * u.y + l.y * u.x;
        P[i * w + c] = a;
      }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < nloc * w; idx += COOP_THREADS) {
    const int i = idx % nloc, c = idx / nloc;
    A2[(rbeg + i) + lda * (int64_t)(k0 + c)] = P[i * w + c];
  }
}

// ---------------- panel factorization by one thread-block cluster ----------------
//
// A sub-panel of SW columns, rows [k0, n), by a cluster of up to 16 CTAs: each
// thread holds RPT rows in registers, so a column costs no pass over shared
// memory, and the pivot exchange is one hop through distributed shared memory
// instead of a barrier over the whole grid.  Per column j:
//   1. every CTA finds its candidate (largest |re| + |im|, the first position
//      among equals, as izamax): a reduction per warp, one CTA barrier;
//   2. the candidate's warp writes the row into the CTA's rows in shared memory
//      and sends it (header: key, position, 1/pivot) to every CTA of the
//      cluster with asynchronous stores that count into the receiver's mbarrier;
//   3. every warp waits for the G messages, picks the same winner, and updates
//      its rows.
// Rows never move: a row knows its position (LAPACK's interchanges applied to
// the position only), and goes to its place when the sub-panel is written back.
// The registers rotate: column j is always a[0], the update writes column c to
// a[c - 1], so that the loop over j needs no register indexing; it runs in four
// phases of SW/4 columns whose width shrinks with the columns left.
// Messages are double-buffered by column parity: a CTA sends for column j + 1
// only after every CTA's message for column j, which each sends after all its
// warps are done with column j - 1.
// Afterwards the cluster applies the interchanges to the rest of the panel
// [p0, p1) and solves the columns right of the sub-panel with its unit-lower
// triangle; what is left of the panel's update is one product
// (panel_update_kernel).
//
// Bound by latency: a complex64 column is ~2060 cycles at up to 128 rows a CTA
// (candidate 300, row out 150, reciprocal 190, sends 370, their flight 210,
// choice 330, update 420) and ~2600 at 480, against ~8700 for a column of the
// kernel above, whose exchange is a barrier over 152 CTAs.  The panels of a
// factorization with what belongs to them (interchanges, updates inside the
// panel): N = 7680 32.7 -> 18.1 ms, N = 1152 4.3 -> 2.3 ms; complex128 N = 1152
// 10.8 -> 6.2 ms.
constexpr int CP_MAX_THREADS = 512;
constexpr int CP_MAX_CLUSTER = 16;
constexpr unsigned CP_SPIN_LIMIT = 1u << 20;

template <typename T>
struct CpHeader;
template <>
struct CpHeader<float> {
  unsigned key, pos;
  float rr, ri;  // reciprocal of the pivot
};
template <>
struct __align__(16) CpHeader<double> {
  unsigned lo, pos;
  unsigned key, pad;
  double rr, ri;
};

__device__ __forceinline__ uint32_t cp_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cp_map(uint32_t addr, int cta) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
// 16 bytes to a CTA of the cluster, counted into its mbarrier.
__device__ __forceinline__ void cp_send16(uint32_t dst, uint32_t bar, uint4 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
// The messages come from other CTAs: acquired at the cluster's scope, as the stores' completion releases them.
__device__ __forceinline__ bool cp_try_wait(uint32_t bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void cp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Pivot keys: magnitude bits (complex128: high word, then low word); 0 for
// zero and NaN, which are no pivots.
__device__ __forceinline__ void cp_key(float re, float im, unsigned &hi, unsigned &lo) {
  const float v = fabsf(re) + fabsf(im);
  hi = v > 0.f ? __float_as_uint(v) : 0u;
  lo = 0u;
}
__device__ __forceinline__ void cp_key(double re, double im, unsigned &hi, unsigned &lo) {
  const double v = fabs(re) + fabs(im);
  const unsigned long long b = v > 0.0 ? (unsigned long long)__double_as_longlong(v) : 0ull;
  hi = (unsigned)(b >> 32);
  lo = (unsigned)b;
}
// The warp's largest (hi, lo), the smallest position among equals.
template <typename T>
__device__ __forceinline__ void cp_reduce(unsigned &hi, unsigned &lo, unsigned &pos) {
  const unsigned m = __reduce_max_sync(0xffffffffu, hi);
  bool in = hi == m;
  hi = m;
  if (sizeof(T) == 8) {
    const unsigned ml = __reduce_max_sync(0xffffffffu, in ? lo : 0u);
    in = in && lo == ml;
    lo = ml;
  }
  pos = __reduce_min_sync(0xffffffffu, in ? pos : 0xffffffffu);
}

// crecip(a) by a whole warp: one division for both parts, the even lanes' and the odd
// lanes'.
template <typename T>
__device__ __forceinline__ cx<T> cp_recip(cx<T> a, int lane) {
  const T d = a.r * a.r + a.i * a.i;
  const T q = (lane & 1 ? -a.i : a.r) / d;
  return {__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1)};
}

template <typename T, int SW, int RPT>
struct CpSmem {
  static constexpr int ROW = SW + 16 / (int)(2 * sizeof(T));  // complex entries of a padded row: 16-byte aligned
  static constexpr int MSG = SW * 2 * (int)sizeof(T) + (int)sizeof(CpHeader<T>);
  static constexpr size_t bytes(int chunk) {
    return (size_t)(2 * CP_MAX_CLUSTER + 1) * MSG + (size_t)SW * ROW * 2 * sizeof(T) + (size_t)chunk * ROW * 2 * sizeof(T);
  }
};

template <typename T, int SW, int RPT>
__global__ void __launch_bounds__(CP_MAX_THREADS, 1)
    panel_cluster_kernel(T *A, int64_t lda, int n, int k0, int w, int p0, int p1, int chunk, int *ipiv, int *info,
                         int *err, int64_t strideA) {
  typedef typename V2<T>::type T2;
  typedef CpSmem<T, SW, RPT> S;
  constexpr int ROW = S::ROW, MSG = S::MSG, HP = (int)sizeof(CpHeader<T>) / 16;
  extern __shared__ __align__(16) unsigned char cp_smem_raw[];
  unsigned char *msg = cp_smem_raw;                                        // [2][CP_MAX_CLUSTER][MSG]
  T2 *out = reinterpret_cast<T2 *>(msg + 2 * CP_MAX_CLUSTER * MSG);        // the candidate's row, as sent
  T2 *LU = reinterpret_cast<T2 *>(msg + (2 * CP_MAX_CLUSTER + 1) * MSG);   // [SW][ROW] the factored diagonal block
  T2 *P = LU + SW * ROW;                                                   // [chunk][ROW] the CTA's rows, final values
  __shared__ __align__(8) unsigned long long bars[2];
  constexpr int WARPS = CP_MAX_THREADS / 32;  // the warps' candidates, by panel_slot_set()
  __shared__ unsigned s_hi[PANEL_SLOT_SETS][WARPS], s_lo[PANEL_SLOT_SETS][WARPS], s_pos[PANEL_SLOT_SETS][WARPS];
  __shared__ int s_piv[SW];
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x, nwarps = nt >> 5;
  const int G = gridDim.x, g = blockIdx.x;
  {
    const int64_t bb = blockIdx.y;  // a batch of equal-size matrices: one cluster each
    A += bb * strideA;
    ipiv += bb * n;
    info += bb;
  }
  T2 *A2 = reinterpret_cast<T2 *>(A);
  const T2 zero2 = V2<T>::make(0, 0);
  if (tid == 0) {
    s_abort = 0;
    for (int k = 0; k < 2; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cp_smem(&bars[k])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // rows into registers
  T2 a[RPT][SW];
  unsigned pos[RPT];
  bool act[RPT];
#pragma unroll
  for (int r = 0; r < RPT; r++) {
    const int i = tid + r * nt, row = k0 + g * chunk + i;
    act[r] = i < chunk && row < n;
    pos[r] = (unsigned)row;
#pragma unroll
    for (int c = 0; c < SW; c++) a[r][c] = act[r] && c < w ? A2[row + lda * (int64_t)(k0 + c)] : zero2;
  }
  cp_cluster_sync();

  int j = 0;
  auto step = [&](auto width) {
    constexpr int W = decltype(width)::value;  // registers in use: columns j .. j + W - 1
    const int par = j & 1;
    const unsigned dr = (unsigned)(k0 + j);
    const uint32_t bar = cp_smem(&bars[par]);
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(G * (W * 2 * (int)sizeof(T) + (int)sizeof(CpHeader<T>))) : "memory");
    // 1. the CTA's candidate
    unsigned hi = 0, lo = 0, cp = 0xffffffffu;
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      unsigned h, l;
      cp_key(a[r][0].x, a[r][0].y, h, l);
      if (!act[r]) h = l = 0;
      const unsigned q = act[r] ? pos[r] : 0xffffffffu;
      const bool better = r == 0 || h > hi || (h == hi && (l > lo || (l == lo && q < cp)));
      hi = better ? h : hi;
      lo = better ? l : lo;
      cp = better ? q : cp;
    }
    cp_reduce<T>(hi, lo, cp);
    const int set = panel_slot_set(j);
    if (lane == 0) {
      s_hi[set][wid] = hi;
      s_lo[set][wid] = lo;
      s_pos[set][wid] = cp;
    }
    __syncthreads();
    hi = lane < nwarps ? s_hi[set][lane] : 0u;
    lo = lane < nwarps ? s_lo[set][lane] : 0u;
    cp = lane < nwarps ? s_pos[set][lane] : 0xffffffffu;
    cp_reduce<T>(hi, lo, cp);
    // 2. its warp sends the row (warp 0 an empty message when there is none)
    int own = -1;
#pragma unroll
    for (int r = 0; r < RPT; r++)
      if (act[r] && pos[r] == cp) own = tid + r * nt;
    const unsigned who = __ballot_sync(0xffffffffu, own >= 0);
    if (who || (cp == 0xffffffffu && wid == 0)) {
      const int from = who ? __ffs(who) - 1 : 0;
      T2 pv = a[0][0];
#pragma unroll
      for (int r = 0; r < RPT; r++)
        if (own == tid + r * nt) {
          pv = a[r][0];
#pragma unroll
          for (int c = 0; c < W; c++) out[c] = a[r][c];
        }
      pv.x = __shfl_sync(0xffffffffu, pv.x, from);
      pv.y = __shfl_sync(0xffffffffu, pv.y, from);
      CpHeader<T> h;
      if (sizeof(T) == 8) reinterpret_cast<unsigned *>(&h)[0] = lo;
      h.key = who ? hi : 0u;
      h.pos = cp;
      const cx<T> rp = who && (hi | lo) ? cp_recip(cx<T>{pv.x, pv.y}, lane) : cx<T>{0, 0};  // (warp-uniform)
      h.rr = rp.r;
      h.ri = rp.i;
      __syncwarp();
      const uint32_t to = cp_smem(msg + (par * CP_MAX_CLUSTER + g) * MSG);
      constexpr int PIECES = W * 2 * (int)sizeof(T) / 16, PER = 32 / PIECES;  // 16-byte pieces, CTAs per round
      if (lane < PER * PIECES) {
        const int q = lane % PIECES;
        const uint4 v = reinterpret_cast<const uint4 *>(out)[q];
        const uint32_t at = to + (int)sizeof(CpHeader<T>) + 16 * q;
        for (int cta = lane / PIECES; cta < G; cta += PER) cp_send16(cp_map(at, cta), cp_map(bar, cta), v);
      }
      for (int cta = lane / HP; cta < G; cta += 32 / HP) {
        const int q = lane % HP;
        const uint4 v = reinterpret_cast<const uint4 *>(&h)[HP == 1 || q == 0 ? 0 : HP - 1];
        cp_send16(cp_map(to + 16 * q, cta), cp_map(bar, cta), v);
      }
    }
    // 3. the G messages
    {
      const unsigned ph = (unsigned)(j >> 1) & 1u;
      unsigned it = 0;
      while (!s_abort && !cp_try_wait(bar, ph))
        if (++it > CP_SPIN_LIMIT) {
          atomicExch(err, 1);
          s_abort = 1;
        }
    }
    const unsigned char *in = msg + par * CP_MAX_CLUSTER * MSG;
    unsigned wh = 0, wl = 0;
    if (lane < G) {
      const CpHeader<T> *hd = reinterpret_cast<const CpHeader<T> *>(in + lane * MSG);
      wh = hd->key;
      if (sizeof(T) == 8) wl = reinterpret_cast<const unsigned *>(hd)[0];
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, wh);
    bool best = lane < G && wh == top;
    unsigned topl = 0;
    if (sizeof(T) == 8) {
      topl = __reduce_max_sync(0xffffffffu, best ? wl : 0u);
      best = best && wl == topl;
    }
    unsigned win = __ballot_sync(0xffffffffu, best);
    if (__popc(win) > 1) {  // equal magnitudes: the first position
      const unsigned q = best ? reinterpret_cast<const CpHeader<T> *>(in + lane * MSG)->pos : 0xffffffffu;
      const unsigned first = __reduce_min_sync(0xffffffffu, q);
      win = __ballot_sync(0xffffffffu, best && q == first);
    }
    const bool none = top == 0u && topl == 0u;  // no pivot in this column: the row at its place stays
    const int wc = win ? __ffs(win) - 1 : 0;
    const CpHeader<T> *hd = reinterpret_cast<const CpHeader<T> *>(in + wc * MSG);
    const T2 *u = reinterpret_cast<const T2 *>(in + wc * MSG + sizeof(CpHeader<T>));  // columns j, j + 1, ...
    // (clamped: after a wait that ran out the message may be of any content, and a
    // position addresses rows)
    const unsigned pv = none ? dr : min(hd->pos, (unsigned)n - 1u);
    if (tid == 0) {
      s_piv[j] = s_abort ? (int)dr : (int)pv;
      if (g == 0) {
        ipiv[dr] = s_abort ? (int)dr : (int)pv;
        if (none && *info == 0) *info = (int)dr + 1;
      }
    }
    const cx<T> rp = {hd->rr, hd->ri};
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      const int i = tid + r * nt;
      if (act[r]) {
        if (pos[r] == pv) {  // the pivot row: its U part is final
          act[r] = false;
          pos[r] = dr;
#pragma unroll
          for (int c = 0; c < W; c++)
            if (j + c < SW) P[i * ROW + j + c] = a[r][c];
        } else {
          if (pos[r] == dr) pos[r] = pv;
          // without a pivot the column stays and nothing is updated
          const cx<T> m = cmul(cx<T>{a[r][0].x, a[r][0].y}, rp);
          const cx<T> l = none ? cx<T>{a[r][0].x, a[r][0].y} : m;
          P[i * ROW + j] = V2<T>::make(l.r, l.i);
          const T fr = none ? T(0) : m.r, fi = none ? T(0) : m.i;
#pragma unroll
          for (int c = 1; c < W; c++) {
            const T2 uc = u[c];
            a[r][c - 1].x = fma(fi, uc.y, fma(-fr, uc.x, a[r][c].x));
            a[r][c - 1].y = fma(-fi, uc.x, fma(-fr, uc.y, a[r][c].y));
          }
        }
      }
    }
    j++;
  };
  constexpr int Q = SW / 4;
#pragma unroll 1
  while (j < min(w, Q)) step(std::integral_constant<int, SW>{});
#pragma unroll 1
  while (j < min(w, 2 * Q)) step(std::integral_constant<int, SW - Q>{});
#pragma unroll 1
  while (j < min(w, 3 * Q)) step(std::integral_constant<int, SW - 2 * Q>{});
#pragma unroll 1
  while (j < w) step(std::integral_constant<int, SW - 3 * Q>{});
  __syncthreads();
  // the rows to their places
#pragma unroll
  for (int r = 0; r < RPT; r++) {
    const int i = tid + r * nt;
    if (i < chunk && k0 + g * chunk + i < n && !s_abort)
      for (int c = 0; c < w; c++) A2[pos[r] + lda * (int64_t)(k0 + c)] = P[i * ROW + c];
  }
  cp_cluster_sync();  // release and acquire: the rows are in L2 for the whole cluster
  // the rest of the panel: interchanges, and U12 = L11^-1 A12 on the right.
  // Entry d of a column comes from where d leads back through the interchanges.
  const int nc = (k0 - p0) + (p1 - k0 - w);
  if (nc > 0) {
#pragma unroll 8
    for (int c = wid; c < w; c += nwarps)
      if (lane < w) LU[lane * ROW + c] = __ldcg(A2 + k0 + lane + lda * (int64_t)(k0 + c));
    __syncthreads();
    const int d1 = k0 + lane, d2 = lane < w ? s_piv[lane] : 0;
    const bool on1 = lane < w, on2 = lane < w && d2 >= k0 + w;
    int s1 = d1, s2 = d2;
    for (int q = w - 1; q >= 0; q--) {
      const int p = s_piv[q], t = k0 + q;
      s1 = s1 == t ? p : s1 == p ? t : s1;
      s2 = s2 == t ? p : s2 == p ? t : s2;
    }
    constexpr int NC = 4;  // columns in flight per warp
    for (int q0 = (g * nwarps + wid) * NC; q0 < nc; q0 += G * nwarps * NC) {
      T2 x1[NC], x2[NC];
      T2 *b[NC];
#pragma unroll
      for (int e = 0; e < NC; e++) {
        const int q = min(q0 + e, nc - 1);  // the last column again where there are fewer
        b[e] = A2 + lda * (int64_t)(q < k0 - p0 ? p0 + q : k0 + w + (q - (k0 - p0)));
        x1[e] = on1 ? b[e][s1] : zero2;
        x2[e] = on2 ? b[e][s2] : zero2;
      }
      __syncwarp();
      if (q0 + NC > k0 - p0)
        for (int i = 0; i + 1 < w; i++) {
          const T2 l = lane > i && on1 ? LU[lane * ROW + i] : zero2;
#pragma unroll
          for (int e = 0; e < NC; e++) {
            const T xr = __shfl_sync(0xffffffffu, x1[e].x, i), xi = __shfl_sync(0xffffffffu, x1[e].y, i);
            if (q0 + e >= k0 - p0) {
              x1[e].x -= l.x * xr - l.y * xi;
              x1[e].y -= l.x * xi + l.y * xr;
            }
          }
        }
#pragma unroll
      for (int e = 0; e < NC; e++)
        if (q0 + e < nc) {
          if (on1) b[e][d1] = x1[e];
          if (on2) b[e][d2] = x2[e];
        }
    }
  }
  cp_cluster_sync();  // no CTA leaves while another's message to it may be under way
}

// C (m x n) -= A (m x K) B (K x n), K = 8..32: what a sub-panel leaves to the rest
// of its panel.  One CTA per TM x TN tile with the whole K in shared memory: a
// single load round and barrier, and small tiles so that the few columns still
// spread over the GPU (a 128 x 64 tile took 30 us where this takes ~5).
template <typename T, int K>
struct PuCfg;
template <>
struct PuCfg<float, 32> { static constexpr int TM = 64, TN = 32, PR = 4, PC = 2; };
template <>
struct PuCfg<float, 16> { static constexpr int TM = 64, TN = 32, PR = 4, PC = 2; };
template <>
struct PuCfg<double, 8> { static constexpr int TM = 32, TN = 8, PR = 1, PC = 1; };
template <>
struct PuCfg<double, 4> { static constexpr int TM = 32, TN = 8, PR = 1, PC = 1; };
template <typename T, int K>
__global__ void __launch_bounds__(256) panel_update_kernel(int m, int n, int k, const T *__restrict__ A, const T *__restrict__ B,
                                                           T *__restrict__ C, int64_t ld, int64_t strideA) {
  typedef typename V2<T>::type T2;
  typedef PuCfg<T, K> Cfg;
  constexpr int TM = Cfg::TM, TN = Cfg::TN, PR = Cfg::PR, PC = Cfg::PC, TX = TM / PR;
  static_assert(TX * (TN / PC) == 256, "256 threads");
  __shared__ T2 As[K][TM], Bs[K][TN];
  const int64_t off = strideA * blockIdx.z;
  const T2 *A2 = reinterpret_cast<const T2 *>(A + off), *B2 = reinterpret_cast<const T2 *>(B + off);
  T2 *C2 = reinterpret_cast<T2 *>(C + off);
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN, tid = threadIdx.x;
  const T2 zero = V2<T>::make(0, 0);
#pragma unroll
  for (int q = tid; q < TM * K; q += 256) {
    const int r = q % TM, c = q / TM;
    As[c][r] = m0 + r < m && c < k ? A2[m0 + r + ld * (int64_t)c] : zero;
  }
#pragma unroll
  for (int q = tid; q < TN * K; q += 256) {
    const int r = q % K, c = q / K;
    Bs[r][c] = n0 + c < n && r < k ? B2[r + ld * (int64_t)(n0 + c)] : zero;
  }
  const int tx = tid % TX, ty = tid / TX;
  T2 acc[PR][PC];
#pragma unroll
  for (int r = 0; r < PR; r++)
#pragma unroll
    for (int c = 0; c < PC; c++) {
      const int row = m0 + tx + TX * r, col = n0 + ty * PC + c;
      acc[r][c] = row < m && col < n ? C2[row + ld * (int64_t)col] : zero;
    }
  __syncthreads();
#pragma unroll
  for (int kk = 0; kk < K; kk++) {
    T2 a[PR], b[PC];
#pragma unroll
    for (int r = 0; r < PR; r++) a[r] = As[kk][tx + TX * r];
#pragma unroll
    for (int c = 0; c < PC; c++) b[c] = Bs[kk][ty * PC + c];
#pragma unroll
    for (int r = 0; r < PR; r++)
#pragma unroll
      for (int c = 0; c < PC; c++) {
        acc[r][c].x = fma(-a[r].x, b[c].x, fma(a[r].y, b[c].y, acc[r][c].x));
        acc[r][c].y = fma(-a[r].x, b[c].y, fma(-a[r].y, b[c].x, acc[r][c].y));
      }
  }
#pragma unroll
  for (int r = 0; r < PR; r++)
#pragma unroll
    for (int c = 0; c < PC; c++) {
      const int row = m0 + tx + TX * r, col = n0 + ty * PC + c;
      if (row < m && col < n) C2[row + ld * (int64_t)col] = acc[r][c];
    }
}

// B[0:w, :] <- T^{-1} B for the w x w (w <= W) unit-lower or upper triangle T: NC
// right-hand sides per CTA in shared memory, in blocks of 32 rows: the block's
// own triangle by substitution (a warp has NC / warps columns, lane = row), then
// its product with the rows that remain.
//
// The block column's triangle and the rows under (over) it come by cp.async, all
// of a thread's copies in flight at once; complex64 keeps two buffers, so the next
// block's copies run under this one's work (complex128 would leave one CTA per SM
// with two).  Loaded one after the other, with the row and column of each element
// from a division, a launch took 57 us where it now takes 23 (complex64, w = 128), 34
// and 45 where it takes 28 and 35 (complex128, w = 64, lower and upper): the 32
// dependent steps of each block are what is left.
//
// Complex64 (NC = 32): the update is most of the work and runs from shared
// memory at one load per 3.7 FMA.  Complex128 (NC = 4, a warp per scheduler):
// bound by the FP64 pipe, so the columns spread over as many SMs as there are.
template <typename T>
struct TriCfg;
template <>
struct TriCfg<float> { static constexpr int NC = 32, THREADS = 256, BUFS = 2; };
template <>
struct TriCfg<double> { static constexpr int NC = 4, THREADS = 128, BUFS = 1; };

// One complex element to shared memory, or zero.
template <typename T2>
__device__ __forceinline__ void cp_async_elem(T2 *dst, const T2 *src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(sizeof(T2)), "r"(valid ? (int)sizeof(T2) : 0)
               : "memory");
}

template <typename T, int W, bool UPPER>
__global__ void __launch_bounds__(TriCfg<T>::THREADS) tri_block_kernel(const T *Ad, int64_t lda, int w, T *B, int64_t ldb,
                                                                       int ncols) {
  typedef typename V2<T>::type T2;
  constexpr int NC = TriCfg<T>::NC, THREADS = TriCfg<T>::THREADS, WARPS = THREADS / 32, CPW = NC / WARPS;
  constexpr int RPP = THREADS / NC, PER = (W - 32) / RPP;  // rows per pass of the update, passes
  constexpr int BUFS = TriCfg<T>::BUFS, XS = NC + 1;  // an odd row stride: a warp's lanes along the rows meet other banks
  static_assert(THREADS % W == 0 && THREADS % 32 == 0, "a thread's copies keep one row");
  extern __shared__ __align__(16) unsigned char tri_raw[];
  T2 *X = reinterpret_cast<T2 *>(tri_raw);  // [W][XS]
  T2 *Tb = X + W * XS;                      // [BUFS][W][33] the triangle's columns of one block
  T2 *rd = Tb + BUFS * W * 33;              // [W] reciprocals of the diagonal (upper)
  const T2 *A2 = reinterpret_cast<const T2 *>(Ad);
  T2 *B2 = reinterpret_cast<T2 *>(B);
  const T2 zero = V2<T>::make(0, 0);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n0 = blockIdx.x * NC;
  const int nblk = (w + 31) / 32;
  const int row = tid % W;  // of this thread's copies
  auto load_block = [&](int q) {
    const int b = UPPER ? nblk - 1 - q : q, o = b * 32;
    if (row >= (UPPER ? 0 : o) && row < (UPPER ? min(w, o + 32) : w)) {
      const T2 *src = A2 + row + lda * (int64_t)o;
      T2 *dst = Tb + (q % BUFS) * (W * 33) + row * 33;
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += THREADS / W) {
        const int c = c0 + tid / W;
        const bool in = o + c < w;
        cp_async_elem(dst + c, in ? src + lda * (int64_t)c : src, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c0 = 0; c0 < NC; c0 += THREADS / W) {
    const int c = c0 + tid / W;
    const bool in = row < w && n0 + c < ncols;
    cp_async_elem(X + row * XS + c, in ? B2 + row + ldb * (int64_t)(n0 + c) : B2, in);
  }
  load_block(0);
  if (UPPER)
    for (int r = tid; r < W; r += THREADS) {
      cx<T> d = {1, 0};
      if (r < w) d = crecip(cld(Ad, r + lda * (int64_t)r));
      rd[r] = V2<T>::make(d.r, d.i);
    }
#pragma unroll 1
  for (int q = 0; q < nblk; q++) {
    const int b = UPPER ? nblk - 1 - q : q, o = b * 32;
    const T2 *Ts = Tb + (q % BUFS) * (W * 33);
    if (q > 0) {
      __syncthreads();  // the previous block's readers are done
      if (BUFS == 1) load_block(q);
    }
    if (BUFS == 2 && q + 1 < nblk) {
      load_block(q + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    {
      const int row = o + lane;
      T2 x[CPW];
#pragma unroll
      for (int e = 0; e < CPW; e++) x[e] = row < W ? X[row * XS + wid * CPW + e] : zero;
      const int m = min(32, w - o);
      for (int i0 = 0; i0 < m; i0++) {
        const int i = UPPER ? m - 1 - i0 : i0;
        const T2 t = row < w && (UPPER ? lane < i : lane > i) ? Ts[row * 33 + i] : zero;
        const T2 rdi = UPPER ? rd[o + i] : zero;
#pragma unroll
        for (int e = 0; e < CPW; e++) {
          if (UPPER && lane == i) {
            const cx<T> y = cmul(cx<T>{x[e].x, x[e].y}, cx<T>{rdi.x, rdi.y});
            x[e] = V2<T>::make(y.r, y.i);
          }
          const T xr = __shfl_sync(0xffffffffu, x[e].x, i), xi = __shfl_sync(0xffffffffu, x[e].y, i);
          x[e].x -= t.x * xr - t.y * xi;
          x[e].y -= t.x * xi + t.y * xr;
        }
      }
#pragma unroll
      for (int e = 0; e < CPW; e++)
        if (row < W) X[row * XS + wid * CPW + e] = x[e];
    }
    __syncthreads();
    // the remaining rows: [o + 32, w) below, or [0, o) above
    const int u0 = UPPER ? 0 : o + 32, u1 = UPPER ? o : w;
    if (u1 > u0) {
      const int c = tid % NC, ry = tid / NC;
      T2 acc[PER];
#pragma unroll
      for (int e = 0; e < PER; e++) {
        const int r = u0 + ry + RPP * e;
        acc[e] = r < u1 ? X[r * XS + c] : zero;
      }
#pragma unroll 4
      for (int k = 0; k < 32; k++) {
        const T2 x = o + k < W ? X[(o + k) * XS + c] : zero;
#pragma unroll
        for (int e = 0; e < PER; e++) {
          const int r = u0 + ry + RPP * e;
          if (r < u1) {
            const T2 t = Ts[r * 33 + k];
            acc[e].x = fma(t.y, x.y, fma(-t.x, x.x, acc[e].x));
            acc[e].y = fma(-t.y, x.x, fma(-t.x, x.y, acc[e].y));
          }
        }
      }
#pragma unroll
      for (int e = 0; e < PER; e++) {
        const int r = u0 + ry + RPP * e;
        if (r < u1) X[r * XS + c] = acc[e];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int c0 = 0; c0 < NC; c0 += THREADS / W) {
    const int c = c0 + tid / W;
    if (row < w && n0 + c < ncols) B2[row + ldb * (int64_t)(n0 + c)] = X[row * XS + c];
  }
}

// ---------------- complex GEMM (FMA pipes) ----------------
// C = alpha op(A) B + beta C, BM x BN complex tile per CTA, TM x TN per thread, MINB
// CTAs per SM (0: as many registers as it takes).  AHEAD: the next BK-deep K step is loaded into registers while one is
// multiplied from shared memory (two buffers, one barrier a step).  Not in 128 x 64
// FP32 tiles, whose 64 sums a thread leave no registers for it: with 139 of them one CTA was
// resident where two hide each other's loads better (2500^3 3.66 ms against 2.98; the
// accumulating 4096 x 4096 x 512 1.94 against 1.51).
// COMP: the FP32 sums of each BK-deep K tile are added into a two-float
// (hi + lo) running sum (TwoSum), so accumulation error does not grow with K;
// TC is the output type (double to accumulate FP32 products into an FP64 C).
template <typename T, int BM, int BN, int TM, int TN, int BK, bool CONJ_A, int MINB, bool AHEAD, typename TC = T,
          bool COMP = false>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB)
    cgemm_fma_kernel(int m, int n, int k, cx<T> alpha, const T *__restrict__ A, int64_t lda, const T *__restrict__ B,
                     int64_t ldb, cx<TC> beta, TC *__restrict__ C, int64_t ldc, int64_t sA, int64_t sB, int64_t sC) {
  typedef typename V2<T>::type T2;
  // strided batch: problem blockIdx.z (strides in elements of T / TC)
  A += sA * blockIdx.z;
  B += sB * blockIdx.z;
  C += sC * blockIdx.z;
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  constexpr int PA = BM * BK / THREADS, PB = BN * BK / THREADS;  // elements a thread loads per K step
  static_assert(PA * THREADS == BM * BK && PB * THREADS == BN * BK, "whole loads");
  constexpr int BUFS = AHEAD ? 2 : 1;
  __shared__ T2 As[BUFS][BK][BM];
  __shared__ T2 Bs[BUFS][BK][BN];
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const T2 *A2 = reinterpret_cast<const T2 *>(A);
  const T2 *B2 = reinterpret_cast<const T2 *>(B);
  T2 va[PA], vb[PB];  // the next K step, on its way
  auto load = [&](int kk0) {
#pragma unroll
    for (int e = 0; e < PA; e++) {
      const int idx = threadIdx.x + THREADS * e;
      const int r = CONJ_A ? idx / BK : idx % BM, kk = CONJ_A ? idx % BK : idx / BM;
      const int gr = m0 + r, gk = kk0 + kk;
      T2 v = V2<T>::make(0, 0);
      if (gr < m && gk < k) v = CONJ_A ? A2[gk + lda * (int64_t)gr] : A2[gr + lda * (int64_t)gk];
      if (CONJ_A) v.y = -v.y;
      va[e] = v;
    }
#pragma unroll
    for (int e = 0; e < PB; e++) {
      const int idx = threadIdx.x + THREADS * e;
      const int kk = idx % BK, c = idx / BK;
      const int gk = kk0 + kk, gc = n0 + c;
      vb[e] = gk < k && gc < n ? B2[gk + ldb * (int64_t)gc] : V2<T>::make(0, 0);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int e = 0; e < PA; e++) {
      const int idx = threadIdx.x + THREADS * e;
      As[buf][CONJ_A ? idx % BK : idx / BM][CONJ_A ? idx / BK : idx % BM] = va[e];
    }
#pragma unroll
    for (int e = 0; e < PB; e++) {
      const int idx = threadIdx.x + THREADS * e;
      Bs[buf][idx % BK][idx / BK] = vb[e];
    }
  };
  cx<T> acc[TM][TN];
  cx<T> lo[COMP ? TM : 1][COMP ? TN : 1];
  cx<T> part[COMP ? TM : 1][COMP ? TN : 1];
#pragma unroll
  for (int a = 0; a < TM; a++)
#pragma unroll
    for (int b = 0; b < TN; b++) acc[a][b] = {0, 0};
  if (COMP) {
#pragma unroll
    for (int a = 0; a < (COMP ? TM : 1); a++)
#pragma unroll
      for (int b = 0; b < (COMP ? TN : 1); b++) { lo[a][b] = {0, 0}; part[a][b] = {0, 0}; }
  }
  if (AHEAD) load(0);
  int buf = 0;
  for (int kk0 = 0; kk0 < k; kk0 += BK, buf ^= AHEAD) {
    if (!AHEAD) {
      if (kk0 > 0) __syncthreads();
      load(kk0);
    }
    store(buf);
    __syncthreads();  // and, with two buffers, everyone is done with the other one
    if (AHEAD && kk0 + BK < k) load(kk0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      T2 a[TM], b[TN];
#pragma unroll
      for (int q = 0; q < TM; q++) a[q] = As[buf][kk][ty + TY * q];
#pragma unroll
      for (int q = 0; q < TN; q++) b[q] = Bs[buf][kk][tx + TX * q];
#pragma unroll
      for (int p = 0; p < TM; p++)
#pragma unroll
        for (int q = 0; q < TN; q++) {
          cx<T> &d = COMP ? part[COMP ? p : 0][COMP ? q : 0] : acc[p][q];
          d.r = fma(a[p].x, b[q].x, d.r);
          d.r = fma(-a[p].y, b[q].y, d.r);
          d.i = fma(a[p].x, b[q].y, d.i);
          d.i = fma(a[p].y, b[q].x, d.i);
        }
    }
    if (COMP) {
#pragma unroll
      for (int p = 0; p < TM; p++)
#pragma unroll
        for (int q = 0; q < TN; q++) {
          cx<T> &h = acc[p][q];
          cx<T> &l = lo[COMP ? p : 0][COMP ? q : 0];
          cx<T> &x = part[COMP ? p : 0][COMP ? q : 0];
          // TwoSum (Knuth): h + x = s + e exactly
          T s_ = h.r + x.r, bp = s_ - h.r;
          l.r += (h.r - (s_ - bp)) + (x.r - bp);
          h.r = s_;
          s_ = h.i + x.i; bp = s_ - h.i;
          l.i += (h.i - (s_ - bp)) + (x.i - bp);
          h.i = s_;
          x = {0, 0};
        }
    }
  }
  typedef typename V2<TC>::type C2t;
  C2t *C2 = reinterpret_cast<C2t *>(C);
  const bool beta0 = (beta.r == TC(0) && beta.i == TC(0));
#pragma unroll
  for (int p = 0; p < TM; p++)
#pragma unroll
    for (int q = 0; q < TN; q++) {
      const int r = m0 + ty + TY * p, c = n0 + tx + TX * q;
      if (r < m && c < n) {
        cx<TC> av = {(TC)acc[p][q].r, (TC)acc[p][q].i};
        if (COMP) {
          av.r += (TC)lo[COMP ? p : 0][COMP ? q : 0].r;
          av.i += (TC)lo[COMP ? p : 0][COMP ? q : 0].i;
        }
        cx<TC> v = cmul(cx<TC>{(TC)alpha.r, (TC)alpha.i}, av);
        if (!beta0) {
          const C2t o = C2[r + ldc * (int64_t)c];
          const cx<TC> ob = cmul(beta, cx<TC>{o.x, o.y});
          v.r += ob.r;
          v.i += ob.i;
        }
        C2[r + ldc * (int64_t)c] = V2<TC>::make(v.r, v.i);
      }
    }
}

// One launch (nb > 1: a strided batch).
//
// FP64 runs at 2 FMA a cycle and SM, so any tile keeps its pipe busy (four warps are
// enough, and 16 x 16 reads no more than the L2 gives) and what counts is how evenly
// the tiles fill the SMs: the 53 products of a complex128 solve of n = 1152 took 20.7 ms in
// 64 x 64 tiles, 13.8 in 32 x 32, 12.3 in 32 x 16 and 11.5 in 16 x 16.
//
// FP32: the tile whose waves take least.  64 x 64 runs at 0.86 of 128 x 64's rate (2500^3 3.20 and
// 2.98 ms) and 32 x 32, bound by its reads of shared memory, at half; but 5000 x 300 x 300 takes 119 us in
// 64 x 64 tiles, three to an SM, against 132, and the joins of a triangle's inverse
// are a few small products, which left most SMs idle in 128 x 64 tiles
// (the 12 of an n = 1152 solve 551 -> 205 us).
template <typename T, bool CONJ_A>
void launch_gemm_fma(bemgpu_ctx_s *ctx, int m, int n, int k, cx<T> alpha, const T *A, int64_t lda, const T *B, int64_t ldb,
                     cx<T> beta, T *C, int64_t ldc, cudaStream_t st, int nb = 1, int64_t sA = 0, int64_t sB = 0,
                     int64_t sC = 0) {
  constexpr int MAX_COLS = 65535 * 16;  // what a grid of the narrowest tiles covers
  for (; n > MAX_COLS; n -= MAX_COLS, B += 2 * ldb * (int64_t)MAX_COLS, C += 2 * ldc * (int64_t)MAX_COLS)
    launch_gemm_fma<T, CONJ_A>(ctx, m, MAX_COLS, k, alpha, A, lda, B, ldb, beta, C, ldc, st, nb, sA, sB, sC);
  auto grid = [&](int bm, int bn) { return dim3((m + bm - 1) / bm, (n + bn - 1) / bn, nb); };
  if constexpr (sizeof(T) == 8) {
    cgemm_fma_kernel<double, 16, 16, 1, 2, 16, CONJ_A, 0, true>
        <<<grid(16, 16), 128, 0, st>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC);
  } else {
    auto cost = [&](int bm, int bn, double rate) {
      const dim3 g = grid(bm, bn);
      const int64_t tiles = (int64_t)g.x * g.y * g.z;
      return (double)((tiles + ctx->num_sms - 1) / ctx->num_sms) * bm * bn / rate;
    };
    const double c0 = cost(128, 64, 1.0), c1 = cost(64, 64, 0.86), c2 = cost(32, 32, 0.55);
    if (c2 < c1 && c2 < c0)
      cgemm_fma_kernel<float, 32, 32, 2, 2, 16, CONJ_A, 0, true>
          <<<grid(32, 32), 256, 0, st>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC);
    else if (c1 < c0)
      cgemm_fma_kernel<float, 64, 64, 4, 4, 8, CONJ_A, 3, true>
          <<<grid(64, 64), 256, 0, st>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC);
    else
      cgemm_fma_kernel<float, 128, 64, 8, 4, 8, CONJ_A, 2, false>
          <<<grid(128, 64), 256, 0, st>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC);
  }
  ctx->launches++;
}

template <typename T, int W>
constexpr int tri_smem_bytes() { return (W * (TriCfg<T>::NC + 1) + TriCfg<T>::BUFS * W * 33 + W) * (int)sizeof(typename V2<T>::type); }

template <typename T>
int set_tri_attrs(bemgpu_ctx_s *ctx) {
  static bool done[BEM_MAX_DEVICES] = {false};
  if (done[ctx->device]) return BEMGPU_OK;
  constexpr int NBL = LuCfg<T>::NBL;
  BEM_CUDA_TRY(ctx, cudaFuncSetAttribute(tri_block_kernel<T, NB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         tri_smem_bytes<T, NB>()));
  BEM_CUDA_TRY(ctx, cudaFuncSetAttribute(tri_block_kernel<T, NB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         tri_smem_bytes<T, NB>()));
  BEM_CUDA_TRY(ctx, cudaFuncSetAttribute(tri_block_kernel<T, NBL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         tri_smem_bytes<T, NBL>()));
  done[ctx->device] = true;
  return BEMGPU_OK;
}

template <typename T, int W, bool UPPER>
void launch_tri_block(bemgpu_ctx_s *ctx, const T *Ad, int64_t lda, int w, T *B, int64_t ldb, int ncols, cudaStream_t st) {
  ProfScope ps(ctx, BEMGPU_K_TRSM, st, 4.0 * w * w * ncols, 4.0 * sizeof(T) * w * ncols);
  constexpr int NC = TriCfg<T>::NC;
  tri_block_kernel<T, W, UPPER>
      <<<(ncols + NC - 1) / NC, TriCfg<T>::THREADS, tri_smem_bytes<T, W>(), st>>>(Ad, lda, w, B, ldb, ncols);
  ctx->launches++;
}

// The interchanges ipiv[k1..k2) on columns [c0, c1), at most 128 rows a launch.
template <typename T>
void launch_laswp(bemgpu_ctx_s *ctx, T *A, int64_t lda, int c0, int c1, int k1, int k2, const int *ipiv,
                  cudaStream_t st) {
  if (c1 <= c0) return;
  ProfScope ps(ctx, BEMGPU_K_LU_PANEL, st, 0.0, 8.0 * sizeof(T) * (k2 - k1) * (double)(c1 - c0));
  const int g = std::min((c1 - c0 + LASWP_COLS - 1) / LASWP_COLS, 8 * ctx->num_sms);
  for (int k = k1; k < k2; k += LASWP_MAXW) {
    laswp_perm_kernel<T><<<g, 2 * LASWP_MAXW, 0, st>>>(A, lda, c0, c1, k, std::min(k2, k + LASWP_MAXW), ipiv);
    ctx->launches++;
  }
}

template <typename T>
int gemm_fma(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const T alpha[2], const T *A, int64_t lda,
             const T *B, int64_t ldb, const T beta[2], T *C, int64_t ldc, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return BEMGPU_OK;
  cx<T> al = {alpha[0], alpha[1]}, be = {beta[0], beta[1]};
  ProfScope ps(ctx, kind, stream, 8.0 * m * n * k,
               2.0 * sizeof(T) * ((double)m * k + (double)k * n + 2.0 * m * n));
  if (opA == 'C')
    launch_gemm_fma<T, true>(ctx, m, n, k, al, A, lda, B, ldb, be, C, ldc, stream);
  else
    launch_gemm_fma<T, false>(ctx, m, n, k, al, A, lda, B, ldb, be, C, ldc, stream);
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

}  // namespace

// Trailing / off-diagonal updates of the complex64 path go through bem_cgemm,
// which uses the tensor-core kernel where one is available (gemm_tc.cu).
int bem_zgemm(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const double alpha[2], const double *A,
              int64_t lda, const double *B, int64_t ldb, const double beta[2], double *C, int64_t ldc,
              cudaStream_t stream) {
  return gemm_fma<double>(ctx, kind, opA, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}

// C (complex128) = alpha A B + beta C with complex64 A, B: FP32 products,
// compensated accumulation (per 8-deep K tile in FP32, across tiles as a
// two-float sum), FP64 output.
int bem_cgemm_comp64_fma(bemgpu_ctx_s *ctx, int kind, int m, int n, int k, const float alpha[2], const float *A,
                         int64_t lda, const float *B, int64_t ldb, const double beta[2], double *C, int64_t ldc,
                         cudaStream_t stream) {
  if (m <= 0 || n <= 0) return BEMGPU_OK;
  dim3 grd((m + 63) / 64, (n + 63) / 64);
  cx<float> al = {alpha[0], alpha[1]};
  cx<double> be = {beta[0], beta[1]};
  ProfScope ps(ctx, kind, stream, 8.0 * m * n * k, 8.0 * ((double)m * k + (double)k * n) + 32.0 * m * n);
  cgemm_fma_kernel<float, 64, 64, 4, 4, 8, false, 1, true, double, true>
      <<<grd, 256, 0, stream>>>(m, n, k, al, A, lda, B, ldb, be, C, ldc, 0, 0, 0);
  ctx->launches++;
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

int bem_cgemm_fma(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const float alpha[2], const float *A,
                  int64_t lda, const float *B, int64_t ldb, const float beta[2], float *C, int64_t ldc,
                  cudaStream_t stream) {
  return gemm_fma<float>(ctx, kind, opA, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}

namespace {

template <typename T>
int gemm_any(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const T alpha[2], const T *A, int64_t lda,
             const T *B, int64_t ldb, const T beta[2], T *C, int64_t ldc, cudaStream_t stream);
template <>
int gemm_any<double>(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const double alpha[2],
                     const double *A, int64_t lda, const double *B, int64_t ldb, const double beta[2], double *C,
                     int64_t ldc, cudaStream_t stream) {
  return bem_zgemm(ctx, kind, opA, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}
template <>
int gemm_any<float>(bemgpu_ctx_s *ctx, int kind, char opA, int m, int n, int k, const float alpha[2],
                    const float *A, int64_t lda, const float *B, int64_t ldb, const float beta[2], float *C,
                    int64_t ldc, cudaStream_t stream) {
  return bem_cgemm(ctx, kind, opA, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}

constexpr int COOP_MAX_SMEM = 226 * 1024;  // below the 227 KB per-CTA limit, with room for the static part

// Factors the panel [k0, k0 + w) with one cooperative launch; returns false
// (nothing launched) when the panel does not fit the cooperative kernel.
template <typename T>
bool panel_coop(bemgpu_ctx_s *ctx, T *A, int64_t lda, int n, int k0, int w, int *d_ipiv, int *d_info,
                cudaStream_t stream, int &rc, int nb = 1, int64_t strideA = 0) {
  typedef typename V2<T>::type T2;
  rc = BEMGPU_OK;
  const int rows = n - k0;
  int G = std::max(1, std::min(ctx->num_sms, (rows + 15) / 16));
  {
    // fewer, fuller CTAs leave SMs to the other lanes' products while this
    // latency-bound panel runs (BEMGPU_TUNE_PANEL_CTAS), as far as shared
    // memory holds their rows
    const int cap = ctx->tune.panel_ctas;
    const int max_chunk = (int)(COOP_MAX_SMEM / (sizeof(T2) * (size_t)w)) - 1;
    if (cap > 0) G = std::max(std::min(G, cap), (rows + max_chunk - 1) / max_chunk);
  }
  if (nb > 1) {
    // a batch shares about the CTAs one panel would take (more rows per CTA,
    // up to what shared memory holds), so that its cooperative launch does
    // not need more of the GPU than a single panel's
    const int max_chunk = (int)(COOP_MAX_SMEM / (sizeof(T2) * (size_t)w)) - 1;
    G = std::max((rows + max_chunk - 1) / max_chunk, (G + nb - 1) / nb);
  }
  const int chunk = (rows + G - 1) / G;
  const size_t smem = sizeof(T2) * (size_t)(chunk + 1) * w;
  if (smem > (size_t)COOP_MAX_SMEM) return false;
  static bool attr[64][2] = {};
  const int ti = sizeof(T) == 8 ? 1 : 0;
  if (!attr[ctx->device][ti]) {
    if (cudaFuncSetAttribute(panel_coop_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, COOP_MAX_SMEM) !=
        cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    attr[ctx->device][ti] = true;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, panel_coop_kernel<T>, COOP_THREADS, smem) !=
          cudaSuccess ||
      per_sm * ctx->num_sms < G * nb) {
    cudaGetLastError();
    return false;
  }
  // candidate slots and barriers per matrix of the batch (the kernel offsets
  // them by blockIdx.y: 2 G values, rows and rows of w entries, 2 w for the
  // diagonal row, one counter, four pivot keys)
  T *cval = (T *)bem_workspace(ctx, "coop_cval", sizeof(T) * 2 * (size_t)G * nb);
  int *crow = (int *)bem_workspace(ctx, "coop_crow", sizeof(int) * 2 * (size_t)G * nb);
  T *cdata = (T *)bem_workspace(ctx, "coop_cdata", sizeof(T2) * 2 * (size_t)G * w * nb);
  T *drow = (T *)bem_workspace(ctx, "coop_drow", sizeof(T2) * 2 * (size_t)w * nb);
  unsigned *counter = (unsigned *)bem_workspace(ctx, "coop_counter", sizeof(unsigned) * (size_t)nb);
  unsigned long long *best =
      (unsigned long long *)bem_workspace(ctx, "coop_best", 4 * sizeof(unsigned long long) * (size_t)nb);
  int *err = (int *)bem_workspace(ctx, "tc_err", sizeof(int));
  if (!cval || !crow || !cdata || !drow || !counter || !best || !err || G > 1024 || w > NB_MAX) {
    rc = bem_fail(ctx, BEMGPU_ERR_OOM, "getrf: panel workspace");
    return true;
  }
  if (!ctx->tc_err_ready) {
    cudaMemsetAsync(err, 0, sizeof(int), stream);
    ctx->tc_err_ready = true;
  }
  cudaMemsetAsync(counter, 0, sizeof(unsigned) * (size_t)nb, stream);
  cudaMemsetAsync(best, 0, 4 * sizeof(unsigned long long) * (size_t)nb, stream);
  int n_ = n, k0_ = k0, w_ = w, chunk_ = chunk;
  void *args[] = {&A,    &lda,  &n_,    &k0_,  &w_,      &chunk_, &d_ipiv, &d_info,
                  &cval, &crow, &cdata, &drow, &counter, &err,    &best,   &strideA};
  const double cb = 2.0 * sizeof(T);
  ProfScope ps(ctx, BEMGPU_K_LU_PANEL, stream, 4.0 * (double)rows * w * w * nb, cb * 2.0 * rows * w * nb);
  const cudaError_t e = cudaLaunchCooperativeKernel((const void *)panel_coop_kernel<T>, dim3(G, nb),
                                                    dim3(COOP_THREADS), args, smem, stream);
  ctx->launches++;
  if (e != cudaSuccess) {
    cudaGetLastError();
    rc = bem_fail(ctx, BEMGPU_ERR_CUDA, "getrf: cooperative panel launch: %s", cudaGetErrorString(e));
  }
  return true;
}

// The panel [k0, k0 + w) in sub-panels, each by one cluster (panel_cluster_kernel)
// and one product for what is left of the panel.  False (nothing launched) when
// the rows do not fit a cluster's registers or the device cannot place one.
//
// Sub-panel width: 32 columns of one row per thread are 64 registers; from 8192
// rows on half as many columns of two rows.  Complex128: 8 columns, since a
// warp's FP64 instruction holds its scheduler's pipe for 64 cycles and the
// update of a wider sub-panel would be most of a column's time (the product that
// follows has the whole GPU).  CTAs: 32 rows each, at most 16: a hop to another
// CTA costs no more than one to the own (~200 cycles).
template <typename T, int SW, int RPT>
bool cluster_ready(bemgpu_ctx_s *ctx) {
  static signed char state[BEM_MAX_DEVICES] = {};  // 0 unknown, 1 usable, -1 not: a property of the device
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  signed char &st = state[ctx->device];
  if (st == 0) {
    auto kern = panel_cluster_kernel<T, SW, RPT>;
    const size_t smem = CpSmem<T, SW, RPT>::bytes(CP_MAX_THREADS * RPT);
    bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
              cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ok) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(CP_MAX_CLUSTER);
      cfg.blockDim = dim3(CP_MAX_THREADS);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute at = {};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = CP_MAX_CLUSTER;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      int clusters = 0;
      ok = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0;
    }
    if (!ok) cudaGetLastError();
    st = ok ? 1 : -1;
  }
  return st > 0;
}

template <typename T, int SW, int RPT>
int panel_cluster_run(bemgpu_ctx_s *ctx, T *A, int64_t lda, int n, int k0, int w, int *d_ipiv, int *d_info, int *err,
                      cudaStream_t stream, int nb, int64_t strideA) {
  constexpr int PER = 32;
  for (int p = k0; p < k0 + w; p += SW) {
    const int sw = std::min(SW, k0 + w - p), rows = n - p;
    int G = 1;
    while (G < CP_MAX_CLUSTER && rows > G * PER) G *= 2;
    // BEMGPU_TUNE_PANEL_CTAS: fewer CTAs as far as their threads hold the rows
    while (ctx->tune.panel_ctas > 0 && G > ctx->tune.panel_ctas && rows <= G / 2 * CP_MAX_THREADS * RPT) G /= 2;
    const int chunk = (rows + G - 1) / G;
    // four warps at least: they share the panel's other columns
    const int nt = std::max(128, std::min(CP_MAX_THREADS, ((chunk + RPT - 1) / RPT + 31) / 32 * 32));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G, nb);
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = CpSmem<T, SW, RPT>::bytes(chunk);
    cfg.stream = stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = G;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    {
      const double cb = 2.0 * sizeof(T);
      ProfScope ps(ctx, BEMGPU_K_LU_PANEL, stream, 4.0 * (double)rows * sw * sw * nb, cb * 2.0 * rows * sw * nb);
      const cudaError_t e = cudaLaunchKernelEx(&cfg, panel_cluster_kernel<T, SW, RPT>, A, lda, n, p, sw, k0, k0 + w,
                                               chunk, d_ipiv, d_info, err, strideA);
      ctx->launches++;
      if (e != cudaSuccess) {
        cudaGetLastError();
        return bem_fail(ctx, BEMGPU_ERR_CUDA, "getrf: cluster panel launch: %s", cudaGetErrorString(e));
      }
    }
    const int nr = n - p - sw, nc = k0 + w - p - sw;
    if (nr > 0 && nc > 0) {
      typedef PuCfg<T, SW> Cfg;
      ProfScope ps(ctx, BEMGPU_K_LU_PANEL, stream, 8.0 * nr * nc * sw * nb,
                   2.0 * sizeof(T) * ((double)nr * sw + (double)sw * nc + 2.0 * nr * nc) * nb);
      panel_update_kernel<T, SW><<<dim3((nr + Cfg::TM - 1) / Cfg::TM, (nc + Cfg::TN - 1) / Cfg::TN, nb), 256, 0, stream>>>(
          nr, nc, sw, A + 2 * (p + sw + lda * (int64_t)p), A + 2 * (p + lda * (int64_t)(p + sw)),
          A + 2 * (p + sw + lda * (int64_t)(p + sw)), lda, strideA);
      ctx->launches++;
      BEM_CUDA_TRY(ctx, cudaGetLastError());
    }
  }
  return BEMGPU_OK;
}

template <typename T>
bool panel_cluster(bemgpu_ctx_s *ctx, T *A, int64_t lda, int n, int k0, int w, int *d_ipiv, int *d_info,
                   cudaStream_t stream, int &rc, int nb = 1, int64_t strideA = 0) {
  constexpr int SW = sizeof(T) == 8 ? 8 : 32;
  const int rows = n - k0, cap = CP_MAX_CLUSTER * CP_MAX_THREADS;
  rc = BEMGPU_OK;
  if (rows > 2 * cap || !(rows <= cap ? cluster_ready<T, SW, 1>(ctx) : cluster_ready<T, SW / 2, 2>(ctx))) return false;
  int *err = (int *)bem_workspace(ctx, "tc_err", sizeof(int));
  if (!err) {
    rc = bem_fail(ctx, BEMGPU_ERR_OOM, "getrf: panel workspace");
    return true;
  }
  if (!ctx->tc_err_ready) {
    cudaMemsetAsync(err, 0, sizeof(int), stream);
    ctx->tc_err_ready = true;
  }
  rc = rows <= cap ? panel_cluster_run<T, SW, 1>(ctx, A, lda, n, k0, w, d_ipiv, d_info, err, stream, nb, strideA)
                   : panel_cluster_run<T, SW / 2, 2>(ctx, A, lda, n, k0, w, d_ipiv, d_info, err, stream, nb, strideA);
  return true;
}

// LU with partial pivoting of nb equal-size matrices A + i strideA (pivots
// d_ipiv + i n, info d_info + i): every panel of the batch in the same launches (a
// cluster, or its own CTAs and barrier in a cooperative grid, for each matrix), the
// interchanges, triangular blocks and trailing updates per matrix.  Each matrix gets the
// arithmetic of a batch of one.
template <typename T>
int getrf_impl(bemgpu_ctx_s *ctx, T *A0, int64_t lda, int n, int *d_ipiv0, int *d_info0, cudaStream_t stream,
               int nb = 1, int64_t strideA = 0) {
  if (int rc0 = set_tri_attrs<T>(ctx)) return rc0;
  PivCand *cand = (PivCand *)bem_workspace(ctx, "lu_cand", sizeof(PivCand) * 1024);
  unsigned int *counter = (unsigned int *)bem_workspace(ctx, "lu_counter", sizeof(unsigned int));
  if (!cand || !counter) return bem_fail(ctx, BEMGPU_ERR_OOM, "getrf: workspace");
  BEM_CUDA_TRY(ctx, cudaMemsetAsync(counter, 0, sizeof(unsigned int), stream));
  BEM_CUDA_TRY(ctx, cudaMemsetAsync(d_info0, 0, sizeof(int) * (size_t)nb, stream));
  const T mone[2] = {T(-1), T(0)}, one[2] = {T(1), T(0)};
  const double cb = 2.0 * sizeof(T);  // bytes per complex element
  constexpr int NBL = LuCfg<T>::NBL;
  // complex64 super-blocks (BEMGPU_TUNE_LU_SUPER): panels in pairs A, B.
  // After A only B's columns take A's update; after B the rows of B and then
  // the trailing matrix beyond the pair take both at once, the latter as one
  // K = 2 NBL product (half the passes over the trailing matrix).  The same
  // updates as one panel at a time, associated differently.
  const bool super = sizeof(T) == 4 && ctx->tune.lu_super != 0;
  for (int k0 = 0; k0 < n; k0 += NBL) {
    const int w = std::min(NBL, n - k0);
    const int rows = n - k0;
    const bool first_half = super && (k0 / NBL) % 2 == 0;   // panel A (its B follows when k0 + w < n)
    const bool second_half = super && (k0 / NBL) % 2 == 1;  // panel B
    const int K0 = second_half ? k0 - NBL : k0;              // the pair's first column
    const int blocks = std::max(1, std::min(ctx->num_sms * 2, (rows + PANEL_THREADS - 1) / PANEL_THREADS));
    int prc = BEMGPU_OK;
    bool coop = ctx->coop_panel &&
                (panel_cluster<T>(ctx, A0, lda, n, k0, w, d_ipiv0, d_info0, stream, prc, nb, strideA) ||
                 panel_coop<T>(ctx, A0, lda, n, k0, w, d_ipiv0, d_info0, stream, prc, nb, strideA));
    if (prc) return prc;
    if (!coop && nb > 1 && ctx->coop_panel) {
      // the batch's panels do not fit at once: one cooperative panel per matrix
      coop = true;
      for (int i = 0; i < nb && coop; i++) {
        coop = panel_coop<T>(ctx, A0 + i * strideA, lda, n, k0, w, d_ipiv0 + (int64_t)i * n, d_info0 + i, stream,
                             prc);
        if (prc) return prc;
      }
      if (!coop && nb > 1) return bem_fail(ctx, BEMGPU_ERR_ARG, "getrf: batched panel does not fit");
    }
    for (int i = 0; i < nb; i++) {
      T *A = A0 + i * strideA;
      int *d_ipiv = d_ipiv0 + (int64_t)i * n;
      int *d_info = d_info0 + i;
      for (int jj = 0; !coop && jj <= w; jj++) {
        ProfScope ps(ctx, BEMGPU_K_LU_PANEL, stream, 8.0 * (rows - jj) * (w - jj), cb * 2 * (rows - jj) * (w - jj));
        panel_step_kernel<T><<<blocks, PANEL_THREADS, 0, stream>>>(A, lda, n, k0, w, jj, d_ipiv, d_info, cand,
                                                                   counter);
        ctx->launches++;
      }
      BEM_CUDA_TRY(ctx, cudaGetLastError());
      // interchanges to the left and right of the panel
      static_assert(NBL <= LASWP_MAXW, "panel wider than the interchange kernel's permutation");
      launch_laswp<T>(ctx, A, lda, 0, k0, k0, k0 + w, d_ipiv, stream);
      if (k0 + w < n) {
        const int nr = n - k0 - w;
        T *A11 = A + 2 * (k0 + lda * (int64_t)k0);
        T *A12 = A + 2 * (k0 + lda * (int64_t)(k0 + w));
        launch_laswp<T>(ctx, A, lda, k0 + w, n, k0, k0 + w, d_ipiv, stream);
        if (second_half) {
          // panel A's update of B's rows beyond the pair:
          // A[k0:k0+w, k0+w:n] -= L[k0:k0+w, K0:k0] U[K0:k0, k0+w:n]
          int rc = gemm_any<T>(ctx, BEMGPU_K_LU_GEMM, 'N', w, nr, k0 - K0, mone, A + 2 * (k0 + lda * (int64_t)K0),
                               lda, A + 2 * (K0 + lda * (int64_t)(k0 + w)), lda, one, A12, lda, stream);
          if (rc) return rc;
        }
        launch_tri_block<T, NBL, false>(ctx, A11, lda, w, A12, lda, nr, stream);
        T *A22 = A + 2 * (k0 + w + lda * (int64_t)(k0 + w));
        int rc;
        if (first_half) {
          // panel B's columns only; the rest waits for B
          T *A21 = A + 2 * (k0 + w + lda * (int64_t)k0);
          rc = gemm_any<T>(ctx, BEMGPU_K_LU_GEMM, 'N', nr, std::min(NBL, nr), w, mone, A21, lda, A12, lda, one, A22,
                           lda, stream);
        } else {
          // the trailing matrix from the pair's panels at once (K = k0 + w - K0)
          T *L21 = A + 2 * (k0 + w + lda * (int64_t)K0);
          T *U12 = A + 2 * (K0 + lda * (int64_t)(k0 + w));
          rc = gemm_any<T>(ctx, BEMGPU_K_LU_GEMM, 'N', nr, nr, k0 + w - K0, mone, L21, lda, U12, lda, one, A22, lda,
                           stream);
        }
        if (rc) return rc;
      }
      BEM_CUDA_TRY(ctx, cudaGetLastError());
    }
  }
  return BEMGPU_OK;
}

template <typename T>
int getrs_impl(bemgpu_ctx_s *ctx, const T *A, int64_t lda, int n, const int *d_ipiv, T *B, int64_t ldb, int nrhs,
               cudaStream_t stream) {
  if (int rc0 = set_tri_attrs<T>(ctx)) return rc0;
  const T mone[2] = {T(-1), T(0)}, one[2] = {T(1), T(0)};
  const double cb = 2.0 * sizeof(T);
  launch_laswp<T>(ctx, B, ldb, 0, nrhs, 0, n, d_ipiv, stream);
  // forward: L Y = P B
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int w = std::min(NB, n - k0);
    const T *L11 = A + 2 * (k0 + lda * (int64_t)k0);
    T *Bk = B + 2 * (int64_t)k0;
    launch_tri_block<T, NB, false>(ctx, L11, lda, w, Bk, ldb, nrhs, stream);
    if (k0 + w < n) {
      const T *L21 = A + 2 * (k0 + w + lda * (int64_t)k0);
      int rc = gemm_any<T>(ctx, BEMGPU_K_SOLVE_GEMM, 'N', n - k0 - w, nrhs, w, mone, L21, lda, Bk, ldb, one,
                           B + 2 * (int64_t)(k0 + w), ldb, stream);
      if (rc) return rc;
    }
  }
  // backward: U X = Y
  const int nblk = (n + NB - 1) / NB;
  for (int bi = nblk - 1; bi >= 0; bi--) {
    const int k0 = bi * NB;
    const int w = std::min(NB, n - k0);
    const T *U11 = A + 2 * (k0 + lda * (int64_t)k0);
    T *Bk = B + 2 * (int64_t)k0;
    launch_tri_block<T, NB, true>(ctx, U11, lda, w, Bk, ldb, nrhs, stream);
    if (k0 > 0) {
      const T *U01 = A + 2 * (lda * (int64_t)k0);
      int rc = gemm_any<T>(ctx, BEMGPU_K_SOLVE_GEMM, 'N', k0, nrhs, w, mone, U01, lda, Bk, ldb, one, B, ldb, stream);
      if (rc) return rc;
    }
  }
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

}  // namespace

int bem_zgetrf(bemgpu_ctx_s *ctx, double *A, int64_t lda, int n, int *d_ipiv, int *d_info, cudaStream_t stream) {
  return getrf_impl<double>(ctx, A, lda, n, d_ipiv, d_info, stream);
}
int bem_zgetrs(bemgpu_ctx_s *ctx, const double *A, int64_t lda, int n, const int *d_ipiv, double *B, int64_t ldb,
               int nrhs, cudaStream_t stream) {
  return getrs_impl<double>(ctx, A, lda, n, d_ipiv, B, ldb, nrhs, stream);
}
namespace {

constexpr int NBO = 512;  // super-block of the FP64-class LU and solve

__global__ void identity_block_kernel(double *X, int64_t ld, int w) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (r >= w) return;
  reinterpret_cast<double2 *>(X)[r + ld * (int64_t)c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
}

// X (w x ncols, ld ldx) <- T^{-1} X for the w x w triangle T at (A, lda):
// unit lower (UPPER false) or upper; 64-row diagonal blocks in FP64
// (tri_block_kernel), off-diagonal updates as 5-slice exact products.
int tri_solve_exact(bemgpu_ctx_s *ctx, const double *A, int64_t lda, int w, bool upper, double *X, int64_t ldx,
                    int ncols, cudaStream_t st) {
  const int nblk = (w + NB - 1) / NB;
  int rc = BEMGPU_OK;
  for (int q = 0; q < nblk && !rc; q++) {
    const int bi = upper ? nblk - 1 - q : q;
    const int j0 = bi * NB, jw = std::min(NB, w - j0);
    double *Xj = X + 2 * (int64_t)j0;
    if (upper)
      launch_tri_block<double, NB, true>(ctx, A + 2 * (j0 + lda * (int64_t)j0), lda, jw, Xj, ldx, ncols, st);
    else
      launch_tri_block<double, NB, false>(ctx, A + 2 * (j0 + lda * (int64_t)j0), lda, jw, Xj, ldx, ncols, st);
    const int m = upper ? j0 : w - j0 - jw;  // rows still to update
    if (m > 0) {
      ExactOperand oa, ob;
      const double *Ablk = upper ? A + 2 * (lda * (int64_t)j0) : A + 2 * (j0 + jw + lda * (int64_t)j0);
      rc = bem_exact_prep(ctx, "ts_A", true, Ablk, lda, m, jw, -1.0, 5, oa, st);
      if (!rc) rc = bem_exact_prep(ctx, "ts_B", false, Xj, ldx, ncols, jw, 1.0, 5, ob, st);
      if (!rc) rc = bem_exact_gemm(ctx, BEMGPU_K_TRSM, oa, ob, upper ? X : Xj + 2 * (int64_t)jw, ldx, 1, st);
    }
  }
  return rc;
}

// Dst (m x ncols) (+)= sign * Ablk (m x k) * Bblk (k x ncols) as a 5-slice exact
// product; Bblk may be Dst itself when accumulate is 0 (it is sliced first).
int exact_mul(bemgpu_ctx_s *ctx, int kind, const double *Ablk, int64_t lda, int m, int k, double sign,
              const double *Bblk, int64_t ldb, int ncols, double *Dst, int64_t ldd, int accumulate, cudaStream_t st) {
  ExactOperand oa, ob;
  int rc = bem_exact_prep(ctx, "xm_A", true, Ablk, lda, m, k, sign, 5, oa, st);
  if (!rc) rc = bem_exact_prep(ctx, "xm_B", false, Bblk, ldb, ncols, k, 1.0, 5, ob, st);
  if (!rc) rc = bem_exact_gemm(ctx, kind, oa, ob, Dst, ldd, accumulate, st);
  return rc;
}

}  // namespace

// FP64-class LU on the tensor cores, blocked twice: 512-column super-panels
// are factored by 64-column panels whose updates stay inside the
// super-panel; then the super-panel's pivots are applied to the other
// columns, U12 = L11^{-1} A12 with the inverse of the 512 x 512 unit-lower
// diagonal block, and A22 -= A21 U12 as one K = 512 exact product.  The
// inverses of the diagonal super-blocks (L and U) are kept for
// bem_zgetrs_exact ("lu_Lb", "lu_Ub": n x 512, block K at rows [K0, K0+512)).
int bem_zgetrf_exact(bemgpu_ctx_s *ctx, double *A, int64_t lda, int n, int *d_ipiv, int *d_info, cudaStream_t stream) {
  if (int rc0 = set_tri_attrs<double>(ctx)) return rc0;
  double *Lb = (double *)bem_workspace(ctx, "lu_Lb", 16 * (size_t)n * NBO);
  double *Ub = (double *)bem_workspace(ctx, "lu_Ub", 16 * (size_t)n * NBO);
  if (!Lb || !Ub) return bem_fail(ctx, BEMGPU_ERR_OOM, "getrf_exact: workspace");
  BEM_CUDA_TRY(ctx, cudaMemsetAsync(d_info, 0, sizeof(int), stream));
  int rc = BEMGPU_OK;
  for (int K0 = 0; K0 < n && !rc; K0 += NBO) {
    const int WO = std::min(NBO, n - K0);
    for (int k0 = K0; k0 < K0 + WO && !rc; k0 += NB) {
      const int w = std::min(NB, K0 + WO - k0);
      int prc = BEMGPU_OK;
      const bool coop = ctx->coop_panel && (panel_cluster<double>(ctx, A, lda, n, k0, w, d_ipiv, d_info, stream, prc) ||
                                            panel_coop<double>(ctx, A, lda, n, k0, w, d_ipiv, d_info, stream, prc));
      if (prc) return prc;
      if (!coop) {  // one launch per column when the panel does not fit the cooperative kernel
        PivCand *cand = (PivCand *)bem_workspace(ctx, "lu_cand", sizeof(PivCand) * 1024);
        unsigned int *counter = (unsigned int *)bem_workspace(ctx, "lu_counter", sizeof(unsigned int));
        if (!cand || !counter) return bem_fail(ctx, BEMGPU_ERR_OOM, "getrf_exact: workspace");
        BEM_CUDA_TRY(ctx, cudaMemsetAsync(counter, 0, sizeof(unsigned int), stream));
        const int rows = n - k0;
        const int blocks = std::max(1, std::min(ctx->num_sms * 2, (rows + PANEL_THREADS - 1) / PANEL_THREADS));
        for (int jj = 0; jj <= w; jj++) {
          ProfScope ps(ctx, BEMGPU_K_LU_PANEL, stream, 8.0 * (rows - jj) * (w - jj), 32.0 * (rows - jj) * (w - jj));
          panel_step_kernel<double><<<blocks, PANEL_THREADS, 0, stream>>>(A, lda, n, k0, w, jj, d_ipiv, d_info, cand,
                                                                           counter);
          ctx->launches++;
        }
      }
      launch_laswp<double>(ctx, A, lda, K0, k0, k0, k0 + w, d_ipiv, stream);
      launch_laswp<double>(ctx, A, lda, k0 + w, K0 + WO, k0, k0 + w, d_ipiv, stream);
      const int nc = K0 + WO - k0 - w;  // super-panel columns right of this panel
      if (nc > 0) {
        launch_tri_block<double, NB, false>(ctx, A + 2 * (k0 + lda * (int64_t)k0), lda, w,
                                            A + 2 * (k0 + lda * (int64_t)(k0 + w)), lda, nc, stream);
        if (k0 + w < n)
          rc = exact_mul(ctx, BEMGPU_K_LU_GEMM, A + 2 * (k0 + w + lda * (int64_t)k0), lda, n - k0 - w, w, -1.0,
                         A + 2 * (k0 + lda * (int64_t)(k0 + w)), lda, nc, A + 2 * (k0 + w + lda * (int64_t)(k0 + w)),
                         lda, 1, stream);
      }
    }
    if (rc) break;
    launch_laswp<double>(ctx, A, lda, 0, K0, K0, K0 + WO, d_ipiv, stream);
    launch_laswp<double>(ctx, A, lda, K0 + WO, n, K0, K0 + WO, d_ipiv, stream);
    // inverses of the diagonal super-block's triangles
    const double *AKK = A + 2 * (K0 + lda * (int64_t)K0);
    double *LbK = Lb + 2 * (int64_t)K0, *UbK = Ub + 2 * (int64_t)K0;
    identity_block_kernel<<<dim3((WO + 255) / 256, WO), 256, 0, stream>>>(LbK, n, WO);
    identity_block_kernel<<<dim3((WO + 255) / 256, WO), 256, 0, stream>>>(UbK, n, WO);
    ctx->launches += 2;
    rc = tri_solve_exact(ctx, AKK, lda, WO, false, LbK, n, WO, stream);
    if (!rc) rc = tri_solve_exact(ctx, AKK, lda, WO, true, UbK, n, WO, stream);
    if (rc || K0 + WO >= n) continue;
    const int nr = n - K0 - WO;
    double *A12 = A + 2 * (K0 + lda * (int64_t)(K0 + WO));
    rc = exact_mul(ctx, BEMGPU_K_TRSM, LbK, n, WO, WO, 1.0, A12, lda, nr, A12, lda, 0, stream);
    if (!rc)
      rc = exact_mul(ctx, BEMGPU_K_LU_GEMM, A + 2 * (K0 + WO + lda * (int64_t)K0), lda, nr, WO, -1.0, A12, lda, nr,
                     A + 2 * (K0 + WO + lda * (int64_t)(K0 + WO)), lda, 1, stream);
  }
  if (!rc) BEM_CUDA_TRY(ctx, cudaGetLastError());
  return rc;
}

// B <- A^{-1} B with the factors and diagonal-block inverses of
// bem_zgetrf_exact: row interchanges, then per 512-row super-block one exact
// product with the block's inverse and one K = 512 exact update of the rest.
int bem_zgetrs_exact(bemgpu_ctx_s *ctx, const double *A, int64_t lda, int n, const int *d_ipiv, double *B, int64_t ldb,
                     int nrhs, cudaStream_t stream) {
  const double *Lb = (const double *)bem_workspace(ctx, "lu_Lb", 16 * (size_t)n * NBO);
  const double *Ub = (const double *)bem_workspace(ctx, "lu_Ub", 16 * (size_t)n * NBO);
  if (!Lb || !Ub) return bem_fail(ctx, BEMGPU_ERR_OOM, "getrs_exact: workspace");
  launch_laswp<double>(ctx, B, ldb, 0, nrhs, 0, n, d_ipiv, stream);
  int rc = BEMGPU_OK;
  for (int K0 = 0; K0 < n && !rc; K0 += NBO) {  // forward: L Y = P B
    const int WO = std::min(NBO, n - K0);
    double *BK = B + 2 * (int64_t)K0;
    rc = exact_mul(ctx, BEMGPU_K_SOLVE_GEMM, Lb + 2 * (int64_t)K0, n, WO, WO, 1.0, BK, ldb, nrhs, BK, ldb, 0, stream);
    if (!rc && K0 + WO < n)
      rc = exact_mul(ctx, BEMGPU_K_SOLVE_GEMM, A + 2 * (K0 + WO + lda * (int64_t)K0), lda, n - K0 - WO, WO, -1.0, BK,
                     ldb, nrhs, B + 2 * (int64_t)(K0 + WO), ldb, 1, stream);
  }
  const int nblk = (n + NBO - 1) / NBO;
  for (int bi = nblk - 1; bi >= 0 && !rc; bi--) {  // backward: U X = Y
    const int K0 = bi * NBO, WO = std::min(NBO, n - K0);
    double *BK = B + 2 * (int64_t)K0;
    rc = exact_mul(ctx, BEMGPU_K_SOLVE_GEMM, Ub + 2 * (int64_t)K0, n, WO, WO, 1.0, BK, ldb, nrhs, BK, ldb, 0, stream);
    if (!rc && K0 > 0)
      rc = exact_mul(ctx, BEMGPU_K_SOLVE_GEMM, A + 2 * (lda * (int64_t)K0), lda, K0, WO, -1.0, BK, ldb, nrhs, B, ldb, 1,
                     stream);
  }
  if (!rc) BEM_CUDA_TRY(ctx, cudaGetLastError());
  return rc;
}

int bem_cgetrf_batch(bemgpu_ctx_s *ctx, float *A, int64_t strideA, int nb, int64_t lda, int n, int *d_ipiv,
                     int *d_info, cudaStream_t stream) {
  if (nb < 1) return BEMGPU_OK;
  return getrf_impl<float>(ctx, A, lda, n, d_ipiv, d_info, stream, nb, strideA);
}

int bem_cgetrf(bemgpu_ctx_s *ctx, float *A, int64_t lda, int n, int *d_ipiv, int *d_info, cudaStream_t stream) {
  return getrf_impl<float>(ctx, A, lda, n, d_ipiv, d_info, stream);
}
int bem_cgetrs(bemgpu_ctx_s *ctx, const float *A, int64_t lda, int n, const int *d_ipiv, float *B, int64_t ldb,
               int nrhs, cudaStream_t stream) {
  return getrs_impl<float>(ctx, A, lda, n, d_ipiv, B, ldb, nrhs, stream);
}

// ---------------- explicit triangular inverses (complex64 mixed path) ----------------
// The correction solves of the refinement apply W32^{-1} = U^{-1} L^{-1} P to
// n_t right-hand sides several times per frequency.  Forming L^{-1} and U^{-1}
// once (recursive blocked inversion, ztrtri-style, whose work is large GEMMs)
// turns every solve into two large tensor-core GEMMs instead of 2 n / 64
// dependent rank-64 steps.
namespace {

// In-place inverses of the 64 x 64 diagonal blocks of X (n x n, ld ldx; the
// last block may be smaller): unit lower (UPPER = false) or upper.  CTA b
// inverts block b; four threads of a warp hold a column, rows i % 4 each, and take it
// column by column of the triangle (the row updates of a column do not depend on one
// another; a dot product per entry by one thread a column took 58 us a launch for the
// lower and 65 us for the upper triangle where this takes 32 for both).
constexpr int TRI_INV_RS = 68;  // row stride of R: four columns of a half warp meet different banks
constexpr int TRI_INV_SMEM = (64 * 65 + 64 * TRI_INV_RS + 64) * 8;

template <bool UPPER>
__device__ __forceinline__ void tri_inv_block(float *X0, int64_t ldx, int n, float2 *tri_smem) {
  float2(*T)[65] = reinterpret_cast<float2(*)[65]>(tri_smem);                            // T[col][row]
  float2(*R)[TRI_INV_RS] = reinterpret_cast<float2(*)[TRI_INV_RS]>(tri_smem + 64 * 65);  // R[col][row]
  float2 *rd = tri_smem + 64 * 65 + 64 * TRI_INV_RS;                                     // reciprocal diagonal (upper)
  const int o = blockIdx.x * 64, w = min(64, n - o), tid = threadIdx.x;
  float2 *X = reinterpret_cast<float2 *>(X0) + o + ldx * o;
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int r = tid & 63, c = (tid >> 6) + 4 * e;
    if (r < w && c < w) T[c][r] = X[r + ldx * (int64_t)c];
    R[c][r] = make_float2(r == c ? 1.f : 0.f, 0.f);
  }
  __syncthreads();
  if (UPPER) {
    if (tid < w) {
      const float2 d = T[tid][tid];
      const float dd = d.x * d.x + d.y * d.y;
      rd[tid] = make_float2(d.x / dd, -d.y / dd);
    }
    __syncthreads();
  }
  const int j = tid >> 2, p = tid & 3, j0 = (tid & ~31) >> 2;  // column, share of its rows, the warp's first column
  float2 *x = R[j];
  if (!UPPER) {
    for (int k = j0; k < w; k++) {
      const float2 xk = x[k];
      if (k >= j && j < w)
#pragma unroll 4
        for (int i = k + 1 + ((p - k - 1) & 3); i < w; i += 4) {
          const float2 l = T[k][i];
          float2 v = x[i];
          v.x -= l.x * xk.x - l.y * xk.y;
          v.y -= l.x * xk.y + l.y * xk.x;
          x[i] = v;
        }
      __syncwarp();
    }
  } else {
    for (int k = min(w - 1, j0 + 7); k >= 0; k--) {
      const float2 s = x[k], d = rd[k];
      const float2 xk = make_float2(s.x * d.x - s.y * d.y, s.x * d.y + s.y * d.x);
      __syncwarp();
      if (k <= j && j < w) {
        if (p == (k & 3)) x[k] = xk;
#pragma unroll 4
        for (int i = p; i < k; i += 4) {
          const float2 u = T[k][i];
          float2 v = x[i];
          v.x -= u.x * xk.x - u.y * xk.y;
          v.y -= u.x * xk.y + u.y * xk.x;
          x[i] = v;
        }
      }
      __syncwarp();
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int r = tid & 63, c = (tid >> 6) + 4 * e;
    if (r < w && c < w) X[r + ldx * (int64_t)c] = R[c][r];
  }
}

// Both triangles: blockIdx.y 0 lower, 1 upper.
__global__ void __launch_bounds__(256) tri_inv_block_kernel(float *L, float *U, int64_t ldx, int n) {
  extern __shared__ float2 tri_smem[];
  if (blockIdx.y == 0)
    tri_inv_block<false>(L, ldx, n, tri_smem);
  else
    tri_inv_block<true>(U, ldx, n, tri_smem);
}

// The unit-lower factor (ones on the diagonal, zeros above) and the upper factor
// (zeros below) of the packed LU.
__global__ void tri_extract_kernel(const float *__restrict__ LU, int64_t ld, int n, float *__restrict__ L,
                                   float *__restrict__ U) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (r >= n) return;
  const float2 v = reinterpret_cast<const float2 *>(LU)[r + ld * (int64_t)c], zero = make_float2(0.f, 0.f);
  const int64_t i = r + (int64_t)n * c;
  reinterpret_cast<float2 *>(L)[i] = r > c ? v : r == c ? make_float2(1.f, 0.f) : zero;
  reinterpret_cast<float2 *>(U)[i] = r > c ? zero : v;
}

// In-place inversion of a triangle X (n x n, ld n) whose 64 x 64 diagonal
// blocks are already inverted (tri_inv_block_kernel), bottom up: at block size
// b the pairs of adjacent inverted b-blocks at offsets o = 0, 2b, 4b, ... are
// joined, lower: X21 = -X22 (L21 X11), upper: X12 = -X11 (U12 X22).  Below
// 512 all full pairs of a level are two strided-batch launches on the FMA
// pipes (hundreds of tiny products become six launches); from 512 up each
// pair is two tensor-core products.
int tri_inv_bottom_up(bemgpu_ctx_s *ctx, bool upper, float *X, int n, float *tmp, cudaStream_t st) {
  const float one[2] = {1.f, 0.f}, mone[2] = {-1.f, 0.f}, zero[2] = {0.f, 0.f};
  int rc = BEMGPU_OK;
  for (int b = NB; b < n && !rc; b *= 2) {
    const int full = n / (2 * b);  // pairs with both blocks b wide
    const int o_last = full * 2 * b;
    const int b2_last = std::min(b, n - o_last - b);  // ragged pair at o_last, if any
    auto at = [&](int r, int c) { return X + 2 * ((int64_t)r + (int64_t)n * c); };
    if (b < 512 && full > 0) {
      const int64_t sx = 2 * ((int64_t)2 * b + (int64_t)n * 2 * b), st_ = 2 * (int64_t)b * b;
      const cx<float> c1 = {1.f, 0.f}, cm1 = {-1.f, 0.f}, c0 = {0.f, 0.f};
      ProfScope ps(ctx, BEMGPU_K_TRSM, st, 16.0 * full * (double)b * b * b, 48.0 * full * (double)b * b);
      if (!upper) {
        launch_gemm_fma<float, false>(ctx, b, b, b, c1, at(b, 0), n, at(0, 0), n, c0, tmp, b, st, full,
                                      sx, sx, st_);
        launch_gemm_fma<float, false>(ctx, b, b, b, cm1, at(b, b), n, tmp, b, c0, at(b, 0), n, st, full,
                                      sx, st_, sx);
      } else {
        launch_gemm_fma<float, false>(ctx, b, b, b, c1, at(0, b), n, at(b, b), n, c0, tmp, b, st, full,
                                      sx, sx, st_);
        launch_gemm_fma<float, false>(ctx, b, b, b, cm1, at(0, 0), n, tmp, b, c0, at(0, b), n, st, full,
                                      sx, st_, sx);
      }
      BEM_CUDA_TRY(ctx, cudaGetLastError());
    }
    for (int pi = (b < 512 ? full : 0); pi <= full && !rc; pi++) {
      const int o = pi * 2 * b, bb = pi < full ? b : b2_last;
      if (bb <= 0) continue;
      if (!upper) {
        rc = bem_cgemm(ctx, BEMGPU_K_TRSM, 'N', bb, b, b, one, at(o + b, o), n, at(o, o), n, zero, tmp, bb, st);
        if (!rc)
          rc = bem_cgemm(ctx, BEMGPU_K_TRSM, 'N', bb, b, bb, mone, at(o + b, o + b), n, tmp, bb, zero, at(o + b, o), n,
                         st);
      } else {
        rc = bem_cgemm(ctx, BEMGPU_K_TRSM, 'N', b, bb, bb, one, at(o, o + b), n, at(o + b, o + b), n, zero, tmp, b, st);
        if (!rc)
          rc = bem_cgemm(ctx, BEMGPU_K_TRSM, 'N', b, bb, b, mone, at(o, o), n, tmp, b, zero, at(o, o + b), n, st);
      }
    }
  }
  return rc;
}

}  // namespace

int bem_ctri_inverses(bemgpu_ctx_s *ctx, const float *LU, int64_t ld, int n, float *Linv, float *Uinv,
                      cudaStream_t st) {
  float *tmp = (float *)bem_workspace(ctx, "tri_tmp", 8 * (size_t)(n / 2 + NB) * (size_t)(n / 2 + NB));
  if (!tmp) return bem_fail(ctx, BEMGPU_ERR_OOM, "tri_inverses: workspace");
  {
    ProfScope ps(ctx, BEMGPU_K_TRSM, st, 0.0, 24.0 * (double)n * n);
    const dim3 g((n + 255) / 256, n);
    tri_extract_kernel<<<g, 256, 0, st>>>(LU, ld, n, Linv, Uinv);
    ctx->launches++;
  }
  {
    static bool attr[64] = {false};
    if (!attr[ctx->device]) {
      BEM_CUDA_TRY(ctx, cudaFuncSetAttribute(tri_inv_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             TRI_INV_SMEM));
      attr[ctx->device] = true;
    }
    const int nb = (n + NB - 1) / NB;
    ProfScope ps(ctx, BEMGPU_K_TRSM, st, 2.0 * nb * 4.0 * NB * NB * NB / 3.0, 2.0 * 16.0 * NB * (double)n);
    tri_inv_block_kernel<<<dim3(nb, 2), 256, TRI_INV_SMEM, st>>>(Linv, Uinv, n, n);
    ctx->launches++;
  }
  int rc = tri_inv_bottom_up(ctx, false, Linv, n, tmp, st);
  if (!rc) rc = tri_inv_bottom_up(ctx, true, Uinv, n, tmp, st);
  if (rc) return rc;
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

namespace {

// T(:, c) = Linv(:, inverse[row0 + c]): L^-1 applied to the interchanged identity
// column row0 + c, whose 1 the interchanges have taken to row inverse[row0 + c].
__global__ void gather_linv_cols_kernel(const float *__restrict__ Linv, int n, const int *__restrict__ inverse, int row0,
                                        float *__restrict__ T) {
  const int c = blockIdx.x;
  const float2 *src = reinterpret_cast<const float2 *>(Linv) + (int64_t)n * inverse[row0 + c];
  float2 *dst = reinterpret_cast<float2 *>(T) + (int64_t)n * c;
  for (int r = threadIdx.x; r < n; r += blockDim.x) dst[r] = src[r];
}

}  // namespace

int *bem_row_permutation(bemgpu_ctx_s *ctx, const int *d_ipiv, int n, cudaStream_t st) {
  int *perm = (int *)bem_workspace(ctx, "lu_perm", 2 * sizeof(int) * (size_t)n);
  if (!perm) return nullptr;
  if (!ctx->perm_ready) {
    if (cudaFuncSetAttribute(perm_from_ipiv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(int) * PERM_MAX_N)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    ctx->perm_ready = true;
  }
  const bool staged = n <= PERM_MAX_N;
  ProfScope ps(ctx, BEMGPU_K_LU_PANEL, st, 0.0, 12.0 * n);
  perm_from_ipiv_kernel<<<(n + 127) / 128, 128, staged ? sizeof(int) * (size_t)n : 0, st>>>(d_ipiv, n, perm, perm + n,
                                                                                            staged);
  ctx->launches++;
  return perm;
}

namespace {

// D = T S for a triangle T (tri as bem_cgemm_tc's) of n rows.
int tri_product(bemgpu_ctx_s *ctx, const float *T, int n, const float *S, int64_t lds, float *D, int64_t ldd, int nrhs,
                int tri, cudaStream_t st) {
  if (ctx->gemm_engine != 2 && n >= 64 && nrhs >= 64)  // tensor cores, the zero triangle skipped
    return bem_cgemm_tc(ctx, BEMGPU_K_SOLVE_GEMM, n, nrhs, n, 1.f, T, n, S, lds, D, ldd, TC_OUT_F32, 0, st, tri);
  const float one[2] = {1.f, 0.f}, zero[2] = {0.f, 0.f};
  return bem_cgemm(ctx, BEMGPU_K_SOLVE_GEMM, 'N', n, nrhs, n, one, T, n, S, lds, zero, D, ldd, st);
}

}  // namespace

// B = W32^-1 E_t for the identity columns row0 .. row0 + nrhs: the interchanges
// and L^-1 reduce to gathering columns of L^-1, then one product with U^-1.
int bem_capply_inverse_identity(bemgpu_ctx_s *ctx, const float *Linv, const float *Uinv, int n, const int *perm,
                                int row0, float *B, int64_t ldb, int nrhs, float *tmp, cudaStream_t st) {
  {
    ProfScope ps(ctx, BEMGPU_K_SOLVE_GEMM, st, 0.0, 16.0 * (double)n * nrhs);
    gather_linv_cols_kernel<<<nrhs, 256, 0, st>>>(Linv, n, perm + n, row0, tmp);
    ctx->launches++;
  }
  return tri_product(ctx, Uinv, n, tmp, n, B, ldb, nrhs, 2, st);
}

// out = U^-1 L^-1 P B: the interchanged rows are gathered into out, the two
// products go to B and back.
int bem_capply_inverse(bemgpu_ctx_s *ctx, const float *Linv, const float *Uinv, int n, const int *perm, float *B,
                       int64_t ldb, int nrhs, float *out, cudaStream_t st) {
  {
    ProfScope ps(ctx, BEMGPU_K_LU_PANEL, st, 0.0, 16.0 * (double)n * nrhs);
    gather_rows_c64_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)nrhs), 256, 0, st>>>(B, ldb, perm, n, out, n);
    ctx->launches++;
  }
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  const int rc = tri_product(ctx, Linv, n, out, n, B, ldb, nrhs, 1, st);
  return rc ? rc : tri_product(ctx, Uinv, n, B, ldb, out, n, nrhs, 2, st);
}
