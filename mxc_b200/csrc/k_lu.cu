// LU of the redundant diagonal block A_rr with partial pivoting and the solve
// A_rr V_r = U_r^T (h2matrix.cpp:375-379, 399-400: PartialPivLU, then solve).
#include "common.cuh"
#include "kernels.h"

#include <cfloat>

namespace h2b {

// Factorization, one CTA per box: pivot = first row of largest magnitude in
// column k among rows k..n-1, the column below it divided by it, rank-1 update
// of the trailing block.  Blocked by panels of NB columns.  In FP64, and in
// FP32 in shared memory, every element takes its updates one multiply-add at a
// time in the order of k, so the factor is bit for bit that of the unblocked
// elimination -- which matters for the ill-conditioned reference
// configuration, whose substitution moves by tens of percent with the rounding
// order.  FP32 in global scratch (SUMS) subtracts a panel's NB products from an
// element of the trailing block as one sum, which keeps the rounding error of a
// diagonally dominant block at 2.5e-7 of it from 256 to 900 rows (one at a time:
// 1.9e-6 to 6.5e-6, so a substitution's root block moved by 2e-6 and the result
// of its BF16 copy by 1e-4).
//
// Bound: the chain of pivots.  A panel's rows live in registers (RPT rows of
// NB columns per thread) and a pivot costs two barriers: the warps' candidates
// (integer maxima of the magnitudes' bit patterns), then the pivot row, which
// its owner publishes.  Rows are exchanged in the other columns once per
// panel, and the trailing block is read and written once per panel instead of
// once per pivot.  The block stays in shared memory up to about 168 KB, else
// in the task's global scratch (L2).  Solve included, 64 boxes of n = 212 FP64
// went from 7.4 to 0.87 ms, one of n = 200 from 4.6 to 0.71, 1 to 256 boxes of
// n = 128 FP32 from 0.51-0.62 to 0.20-0.37; a pivot is about 2,500 clocks
// (candidates 900, division and update 700).
// The factor (column-major, ld n) goes to the task's work, prow receives the
// row of the right-hand sides that lands in row i of P B.
constexpr int LU_TT = 64;  // trailing tile

// Key of a magnitude: larger value, larger key; NaN 0 (never a pivot).
__device__ __forceinline__ unsigned long long lu_key(double v) {
  return v == v ? (unsigned long long)__double_as_longlong(fabs(v)) + 1ULL : 0ULL;
}
__device__ __forceinline__ unsigned long long lu_key(float v) {
  return v == v ? (unsigned long long)__float_as_uint(fabsf(v)) + 1ULL : 0ULL;
}
// Warp-wide largest key, and the smallest row that has it.
template <typename T>
__device__ __forceinline__ void lu_warp_best(unsigned long long& key, int& row) {
  unsigned m;
  if constexpr (sizeof(T) == 8) {
    const unsigned hi = (unsigned)(key >> 32);
    m = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == m ? (unsigned)key : 0u);
    const unsigned long long best = ((unsigned long long)m << 32) | lo;
    row = (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)row : 0x7fffffffu);
    key = best;
  } else {
    m = __reduce_max_sync(0xffffffffu, (unsigned)key);
    row = (int)__reduce_min_sync(0xffffffffu, (unsigned)key == m ? (unsigned)row : 0x7fffffffu);
    key = m;
  }
}

template <typename T, int NT, int NB, int RPT, bool SMEM>
__global__ void __launch_bounds__(NT) k_lu_factor(const LuSolveTask<T>* __restrict__ tasks) {
  constexpr int NW = NT / 32;
  constexpr bool SUMS = !SMEM && sizeof(T) == 4;
  const LuSolveTask<T> t = tasks[blockIdx.x];
  const int n = t.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (n <= 0) {
    if (tid == 0) *t.info = 0;
    return;
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) T s_prow[2][NB];
  __shared__ unsigned long long s_key[2][NW];
  __shared__ int s_row[2][NW];
  __shared__ T s_l11[NB][NB + 1];
  __shared__ T Ls[NB][LU_TT + 1], Us[NB][LU_TT + 1];
  const int ld = SMEM ? (n | 1) : n;
  int* piv = reinterpret_cast<int*>(smem_raw);  // n
  int* pm = piv + n;                            // n: the panel's net exchange, identity outside it
  int* prow = pm + n;                           // n
  T* a = SMEM ? reinterpret_cast<T*>(smem_raw + (3 * sizeof(int) * (size_t)n + 15) / 16 * 16) : t.work;
  for (int c = warp; c < n; c += NW)
    for (int r = lane; r < n; r += 32) a[r + (size_t)c * ld] = t.A[r + (i64)c * t.lda];
  for (int i = tid; i < n; i += NT) pm[i] = prow[i] = i;
  double det = 1.;
  int swaps = 0;
  __syncthreads();
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int kb = min(NB, n - k0), j0 = k0 + kb;
    // Panel: rows k0 + tid + NT i in registers.  A row stays with its thread:
    // an exchange swaps the rows' positions (pos) only, and each row is
    // written back at the position it ends in.
    T x[RPT][NB];
    int pos[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int r = k0 + tid + NT * i;
      pos[i] = r < n ? r : -1;
#pragma unroll
      for (int j = 0; j < NB; j++) x[i][j] = (r < n && j < kb) ? a[r + (size_t)(k0 + j) * ld] : T(0);
    }
    // Four pivots per turn of the loop, then the registers rotate by four, so
    // that the pivot columns are always x[.][0..3] (all NB pivots unrolled, the
    // code ran at the pace of its instruction fetches); after NB / 4 turns
    // every column is back in its place.  Columns already done sit at the end
    // and take no update.
#pragma unroll 1
    for (int jq = 0; jq < NB; jq += 4) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int jj = jq + q, k = k0 + jj, b = q & 1;
        if (jj < kb) {
          unsigned long long key = 0;
          int row = 0x7fffffff;
#pragma unroll
          for (int i = 0; i < RPT; i++) {
            const unsigned long long ki = pos[i] >= k ? lu_key(x[i][q]) : 0ULL;
            if (ki > key || (ki == key && ki != 0ULL && pos[i] < row)) { key = ki; row = pos[i]; }
          }
          lu_warp_best<T>(key, row);
          if (lane == 0) {
            s_key[b][warp] = key;
            s_row[b][warp] = row;
          }
          __syncthreads();
          key = lane < NW ? s_key[b][lane] : 0ULL;
          row = lane < NW ? s_row[b][lane] : 0x7fffffff;
          lu_warp_best<T>(key, row);
          const int p = key == 0 ? k : row;  // a column of NaNs: no exchange
#pragma unroll
          for (int i = 0; i < RPT; i++) {
            if (pos[i] == p) {
#pragma unroll
              for (int j = 0; j < NB; j++) s_prow[b][j] = x[i][j];
              pos[i] = k;
            } else if (pos[i] == k) {
              pos[i] = p;
            }
          }
          if (tid == 0) piv[k] = p;
          __syncthreads();
          const T pv = s_prow[b][q];
          det *= (double)pv;
          swaps += p != k;
#pragma unroll
          for (int i = 0; i < RPT; i++) {
            if (pos[i] > k && pv != T(0)) x[i][q] = x[i][q] / pv;
            const T l = pos[i] > k ? x[i][q] : T(0);
#pragma unroll
            for (int g = 0; g < NB; g += 16)
              if (g < NB - jq) {
                const int ge = NB - jq - g;  // live columns from g on
#pragma unroll
                for (int j = g; j < g + 16 && j < NB; j++)
                  if (j > q) x[i][j] -= l * (j - g < ge ? s_prow[b][j] : T(0));
              }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        T f[4];
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = x[i][j];
#pragma unroll
        for (int j = 0; j + 4 < NB; j++) x[i][j] = x[i][j + 4];
#pragma unroll
        for (int j = 0; j < 4; j++) x[i][NB - 4 + j] = f[j];
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; i++)
      if (pos[i] >= 0) {
#pragma unroll
        for (int j = 0; j < NB; j++)
          if (j < kb) {
            a[pos[i] + (size_t)(k0 + j) * ld] = x[i][j];
            if (pos[i] < j0) s_l11[pos[i] - k0][j] = x[i][j];
          }
      }
    if (tid == 0)
      for (int k = k0; k < j0; k++) {
        const int q = piv[k];
        int s = pm[k];
        pm[k] = pm[q];
        pm[q] = s;
        s = prow[k];
        prow[k] = prow[q];
        prow[q] = s;
      }
    __syncthreads();
    // The panel's row exchanges in every other column: at most 2 kb rows move,
    // read into registers before any is written, four columns in flight.
    {
      constexpr int EX = 2 * NB > 32 ? 2 * NB / 32 : 1;
      int d[EX], src[EX];
#pragma unroll
      for (int u = 0; u < EX; u++) {
        const int e = lane + 32 * u;
        d[u] = e < kb ? k0 + e : e < 2 * kb ? piv[k0 + e - kb] : -1;
        src[u] = d[u] >= 0 ? pm[d[u]] : -1;
        if (src[u] == d[u]) d[u] = -1;  // the row stays
      }
      for (int c = warp; c < n; c += 4 * NW) {
        T v[4][EX];
#pragma unroll
        for (int w = 0; w < 4; w++) {
          const int cc = c + w * NW;
          const bool on = cc < n && (cc < k0 || cc >= j0);
#pragma unroll
          for (int u = 0; u < EX; u++) v[w][u] = (on && d[u] >= 0) ? a[src[u] + (size_t)cc * ld] : T(0);
        }
        __syncwarp();
#pragma unroll
        for (int w = 0; w < 4; w++) {
          const int cc = c + w * NW;
          const bool on = cc < n && (cc < k0 || cc >= j0);
#pragma unroll
          for (int u = 0; u < EX; u++)
            if (on && d[u] >= 0) a[d[u] + (size_t)cc * ld] = v[w][u];
        }
      }
    }
    __syncthreads();
    for (int e = tid; e < 2 * kb; e += NT) {
      const int r = e < kb ? k0 + e : piv[k0 + e - kb];
      pm[r] = r;
    }
    if (j0 >= n) break;
    // U12: unit-lower solve of the panel's rows, a column per thread.
    for (int c = j0 + tid; c < n; c += NT) {
      T* ac = a + (size_t)c * ld + k0;
      T u[NB];
#pragma unroll
      for (int i = 0; i < NB; i++) u[i] = i < kb ? ac[i] : T(0);
#pragma unroll
      for (int i = 0; i < NB; i++)
#pragma unroll
        for (int r = i + 1; r < NB; r++)
          if (r < kb) u[r] -= s_l11[r][i] * u[i];
#pragma unroll
      for (int i = 0; i < NB; i++)
        if (i < kb) ac[i] = u[i];
    }
    __syncthreads();
    // Trailing block, LU_TT x LU_TT tiles, updates in the order of k.  acc: the
    // element itself, or (SUMS) minus the panel's products.
    constexpr int GX = 16, GY = NT / GX, TY = LU_TT / GY, TX = LU_TT / GX;
    const int tx = tid % GX, ty = tid / GX;
    for (int tc = j0; tc < n; tc += LU_TT)
      for (int tr = j0; tr < n; tr += LU_TT) {
        T acc[TX][TY];  // rows tx + GX u, columns ty + GY v
#pragma unroll
        for (int v = 0; v < TY; v++)
#pragma unroll
          for (int u = 0; u < TX; u++) {
            const int r = tr + tx + GX * u, c = tc + ty + GY * v;
            acc[u][v] = (!SUMS && r < n && c < n) ? a[r + (size_t)c * ld] : T(0);
          }
        for (int e = tid; e < LU_TT * NB; e += NT) {
          const int rr = e % LU_TT, i = e / LU_TT;
          Ls[i][rr] = (tr + rr < n && i < kb) ? a[(tr + rr) + (size_t)(k0 + i) * ld] : T(0);
        }
        if (tr == j0)
          for (int e = tid; e < LU_TT * NB; e += NT) {
            const int i = e % NB, cc = e / NB;
            Us[i][cc] = (tc + cc < n && i < kb) ? a[(k0 + i) + (size_t)(tc + cc) * ld] : T(0);
          }
        __syncthreads();
#pragma unroll 4
        for (int i = 0; i < kb; i++) {
          T lv[TX], uv[TY];
#pragma unroll
          for (int u = 0; u < TX; u++) lv[u] = Ls[i][tx + GX * u];
#pragma unroll
          for (int v = 0; v < TY; v++) uv[v] = Us[i][ty + GY * v];
#pragma unroll
          for (int u = 0; u < TX; u++)
#pragma unroll
            for (int v = 0; v < TY; v++) acc[u][v] -= lv[u] * uv[v];
        }
        if (SUMS)
#pragma unroll
          for (int v = 0; v < TY; v++)
#pragma unroll
            for (int u = 0; u < TX; u++) {
              const int r = tr + tx + GX * u, c = tc + ty + GY * v;
              if (r < n && c < n) acc[u][v] += a[r + (size_t)c * ld];
            }
#pragma unroll
        for (int v = 0; v < TY; v++)
#pragma unroll
          for (int u = 0; u < TX; u++) {
            const int r = tr + tx + GX * u, c = tc + ty + GY * v;
            if (r < n && c < n) a[r + (size_t)c * ld] = acc[u][v];
          }
        __syncthreads();
      }
  }
  __syncthreads();
  if (SMEM)
    for (int c = warp; c < n; c += NW)
      for (int r = lane; r < n; r += 32) t.work[r + (i64)c * n] = a[r + (size_t)c * ld];
  for (int k = tid; k < n; k += NT) {
    t.ipiv[k] = piv[k];
    t.prow[k] = prow[k];
  }
  if (tid == 0) {
    // Eigen's determinant: product of U's diagonal times the permutation sign.
    *t.info = fabs((swaps & 1) ? -det : det) <= DBL_MIN ? 1 : 0;
  }
}

// X = A^{-1} B from the factor: row interchanges, unit-lower forward and upper
// backward substitution, LU_CT right-hand-side columns per CTA (a column per
// thread), 32 rows at a time in registers, left-looking across row blocks
// with the factor's columns staged in shared memory so that a block's
// multipliers come as 16-byte broadcasts.  Bound by FMA issue; the columns of
// a box spread over several CTAs, so a level of few boxes is not one SM's work.
// Right-hand sides and solution have row r contiguous over the columns
// (B[c + r ldb]), as U_r^T and V_r are laid out in the ULV.
constexpr int LU_CT = 128, LU_JT = 32;

template <typename T>
__global__ void __launch_bounds__(LU_CT) k_lu_trsm(const LuSolveTask<T>* __restrict__ tasks) {
  constexpr int PS = 32 + 16 / sizeof(T);
  const LuSolveTask<T> t = tasks[blockIdx.x];
  const int n = t.n, tid = threadIdx.x, c = blockIdx.y * LU_CT + tid;
  if (n <= 0 || (int)blockIdx.y * LU_CT >= t.m) return;
  const bool cv = c < t.m;
  __shared__ __align__(16) T P[LU_JT * PS];  // P[j][i] = factor(b0 + i, jb + j)
  const T* __restrict__ a = t.work;
  T* X = t.X + c;
  T r[32];
  // r -= factor(block rows, columns [j0, j1)) X[j0..j1), eight columns at a
  // time with the next eight X rows already on their way, and the next panel
  // tile in registers while one is used.
  auto update = [&](int b0, int bs, int j0, int j1) {
    if (j0 >= j1) return;
    constexpr int PT = 32 * LU_JT / LU_CT;
    T pre[PT], x[8];
    auto fetch = [&](int jb) {
#pragma unroll
      for (int e = 0; e < PT; e++) {
        const int i = tid & 31, j = jb + (tid >> 5) + e * (LU_CT / 32);
        pre[e] = (i < bs && j < j1) ? a[(b0 + i) + (i64)j * n] : T(0);
      }
    };
    auto fetch_x = [&](int j) {
#pragma unroll
      for (int u = 0; u < 8; u++) x[u] = (cv && j + u < j1) ? X[(i64)(j + u) * t.ldx] : T(0);
    };
    fetch(j0);
    fetch_x(j0);
    for (int jb = j0; jb < j1; jb += LU_JT) {
      const int je = min(jb + LU_JT, j1);
      __syncthreads();
#pragma unroll
      for (int e = 0; e < PT; e++) P[((tid >> 5) + e * (LU_CT / 32)) * PS + (tid & 31)] = pre[e];
      __syncthreads();
      if (je < j1) fetch(je);
      for (int j = jb; j < je; j += 8) {
        T y[8];
#pragma unroll
        for (int u = 0; u < 8; u++) y[u] = x[u];
        if (j + 8 < j1) fetch_x(j + 8);
#pragma unroll
        for (int u = 0; u < 8; u++) {
          if (j + u >= je) break;
          const T* p = P + (j + u - jb) * PS;
#pragma unroll
          for (int i = 0; i < 32; i++) r[i] -= p[i] * y[u];
        }
      }
    }
  };
  auto load_diag = [&](int b0, int bs) {
    __syncthreads();
    for (int e = tid; e < 32 * 32; e += LU_CT) {
      const int i = e & 31, j = e >> 5;
      P[j * PS + i] = (i < bs && j < bs) ? a[(b0 + i) + (i64)(b0 + j) * n] : T(0);
    }
    __syncthreads();
  };
  auto store = [&](int b0, int bs) {
    if (cv)
#pragma unroll
      for (int i = 0; i < 32; i++)
        if (i < bs) X[(i64)(b0 + i) * t.ldx] = r[i];
  };
  for (int b0 = 0; b0 < n; b0 += 32) {  // L y = P b
    const int bs = min(32, n - b0);
#pragma unroll
    for (int i = 0; i < 32; i++) r[i] = (cv && i < bs) ? t.B[c + (i64)t.prow[b0 + i] * t.ldb] : T(0);
    update(b0, bs, 0, b0);
    load_diag(b0, bs);
#pragma unroll
    for (int jj = 0; jj < 32; jj++)
      if (jj < bs) {
#pragma unroll
        for (int i = jj + 1; i < 32; i++) r[i] -= P[jj * PS + i] * r[jj];
      }
    store(b0, bs);
  }
  for (int b0 = (n - 1) / 32 * 32; b0 >= 0; b0 -= 32) {  // U x = y
    const int bs = min(32, n - b0);
#pragma unroll
    for (int i = 0; i < 32; i++) r[i] = (cv && i < bs) ? X[(i64)(b0 + i) * t.ldx] : T(0);
    update(b0, bs, b0 + 32, n);
    load_diag(b0, bs);
#pragma unroll
    for (int jj = 31; jj >= 0; jj--)
      if (jj < bs) {
        r[jj] = r[jj] / P[jj * PS + jj];
#pragma unroll
        for (int i = 0; i < jj; i++) r[i] -= P[jj * PS + i] * r[jj];
      }
    store(b0, bs);
  }
}

template <typename T>
cudaError_t launch_lu_solve(const LuSolveTask<T>* d_tasks, int ntasks, int maxn, int maxm, cudaStream_t st) {
  if (ntasks == 0) return cudaSuccess;
  if (maxn > 2048) return cudaErrorInvalidValue;  // rows of a panel held in registers
  const size_t ints = (3 * sizeof(int) * (size_t)maxn + 15) / 16 * 16;
  const size_t mat = sizeof(T) * (size_t)maxn * (maxn | 1);
  // The static tiles take up to 42 KB (FP64, NB 32) of the 227 KB.
  const bool in_smem = maxn <= 256 && ints + mat <= 168 * 1024;
  const size_t smem = ints + (in_smem ? mat : 0) + 16;
  auto go = [&](auto kern, int nt) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    note_launch();
    kern<<<ntasks, nt, smem, st>>>(d_tasks);
    return cudaGetLastError();
  };
  cudaError_t e;
  if (in_smem) e = go(k_lu_factor<T, 256, 32, 1, true>, 256);
  else if (maxn <= 512) e = go(k_lu_factor<T, 512, 32, 1, false>, 512);
  // Beyond, as many columns as the registers hold (64 a thread of 512).
  else if (maxn <= 1024) e = go(k_lu_factor<T, 512, sizeof(T) == 4 ? 32 : 16, 2, false>, 512);
  else e = go(k_lu_factor<T, 512, sizeof(T) == 4 ? 16 : 8, 4, false>, 512);
  if (e != cudaSuccess || maxm <= 0) return e;
  note_launch();
  k_lu_trsm<T><<<dim3(ntasks, (maxm + LU_CT - 1) / LU_CT), LU_CT, 0, st>>>(d_tasks);
  return cudaGetLastError();
}
template cudaError_t launch_lu_solve<double>(const LuSolveTask<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_lu_solve<float>(const LuSolveTask<float>*, int, int, int, cudaStream_t);

}  // namespace h2b
