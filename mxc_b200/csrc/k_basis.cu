// Shared-basis compression kernels (compute_basis, h2matrix.cpp:13-63).
//
// One CTA per box of a tree level.  Step 1 (k_sample_tsqr) forms the R
// factor of the far-field sample block XF = K(far samples, box bodies)
// without materialising XF: sample rows are generated 32 at a time into
// shared memory and folded into R with Householder reflectors on
// (row j of R, tile column j).  Step 2 (k_cpqr) runs the column-pivoted
// Householder QR of R with Eigen 3.4's ColPivHouseholderQR pivot, norm
// downdate and rank rules (in a cluster's shared memory where it fits,
// k_cpqr.cu).  Step 3 (k_interp, k_basis_build) forms the interpolative
// decomposition [I, R11^-1 R12], permutes the box bodies skeleton-first and
// builds either the ID basis (operator mode) or, for the caller's orthogonal
// completion, U_ID (preconditioner mode).
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <cfloat>

namespace h2b {

template <typename T> struct Tiny;
template <> struct Tiny<double> { static __device__ double v() { return DBL_MIN; } };
template <> struct Tiny<float> { static __device__ float v() { return FLT_MIN; } };

constexpr int TS_THREADS = 256;
constexpr int TS_MAXCOL = 8;  // columns owned per thread: M <= 2048

// R (row-major M x M per box, zero on entry) of the sample block.  TR
// sample rows per tile (32, or 16 / 8 for wide boxes so the tile fits in
// shared memory); lane r of the reflector warp holds tile row r.
template <typename T, int TR>
__global__ void __launch_bounds__(TS_THREADS) k_sample_tsqr(
    KernelParams kp, const double* __restrict__ bodies, const double* __restrict__ pts,
    const i64* __restrict__ xoff, const i64* __restrict__ dims, const int* __restrict__ sidx,
    const i64* __restrict__ soff, T* __restrict__ Rws, const i64* __restrict__ qoff) {
  const int box = blockIdx.x;
  const int M = (int)dims[box];
  const i64 S = soff[box + 1] - soff[box];
  if (M == 0 || S == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);            // 32 x M, row-major
  T* vbuf = tile + TR * M;                             // 32
  double* sp = reinterpret_cast<double*>(vbuf + 32);   // 32 x 3
  __shared__ T s_tau;

  T* R = Rws + qoff[box];
  const int* my_sidx = sidx + soff[box];
  const double* bp = pts + 3 * xoff[box];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  double px[TS_MAXCOL], py[TS_MAXCOL], pz[TS_MAXCOL];
#pragma unroll
  for (int k = 0; k < TS_MAXCOL; k++) {
    int c = tid + k * TS_THREADS;
    px[k] = c < M ? bp[3 * c] : 0.;
    py[k] = c < M ? bp[3 * c + 1] : 0.;
    pz[k] = c < M ? bp[3 * c + 2] : 0.;
  }

  int rows = 0;  // rows of R that can be nonzero so far
  for (i64 t0 = 0; t0 < S; t0 += TR) {
    const int nrows = (int)((S - t0) < TR ? (S - t0) : TR);
    if (tid < nrows) {
      const double* q = bodies + 3 * (i64)my_sidx[t0 + tid];
      sp[3 * tid] = q[0];
      sp[3 * tid + 1] = q[1];
      sp[3 * tid + 2] = q[2];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TS_MAXCOL; k++) {
      int c = tid + k * TS_THREADS;
      if (c < M)
        for (int r = 0; r < TR; r++)
          tile[r * M + c] = r < nrows ? (T)kernel_fast_pair(kp, sp[3 * r], sp[3 * r + 1], sp[3 * r + 2], px[k], py[k], pz[k]) : T(0);
    }
    __syncthreads();
    const int jend = (rows + nrows) < M ? (rows + nrows) : M;
    for (int j = 0; j < jend; j++) {
      const int owner = j % TS_THREADS;
      if (warp == (owner >> 5)) {
        // Reflector on (R[j][j], tile[:, j]), computed by the owner's warp:
        // lane r holds tile row r.
        T x = lane < nrows ? tile[lane * M + j] : T(0);
        T sig = x * x;
        for (int o = 16; o > 0; o >>= 1) sig += __shfl_xor_sync(0xffffffffu, sig, o);
        T alpha = R[(i64)j * M + j];
        T tau = 0, scale = 0, beta = alpha;
        if (sig > Tiny<T>::v()) {
          T nrm = sqrt(alpha * alpha + sig);
          beta = alpha >= T(0) ? -nrm : nrm;
          tau = (beta - alpha) / beta;
          scale = T(1) / (alpha - beta);
        }
        vbuf[lane] = x * scale;
        if (lane == 0) {
          s_tau = tau;
          R[(i64)j * M + j] = beta;
        }
      }
      __syncthreads();
      const T tau = s_tau;
      if (tau != T(0)) {
#pragma unroll
        for (int k = 0; k < TS_MAXCOL; k++) {
          int c = tid + k * TS_THREADS;
          if (c > j && c < M) {
            T w = R[(i64)j * M + c];
            for (int r = 0; r < nrows; r++) w += vbuf[r] * tile[r * M + c];
            w *= tau;
            R[(i64)j * M + c] -= w;
            for (int r = 0; r < nrows; r++) tile[r * M + c] -= w * vbuf[r];
          }
        }
      }
      __syncthreads();
    }
    rows = jend;
  }
}

// Column-pivoted Householder QR (Eigen 3.4 ColPivHouseholderQR::computeInPlace
// restated) of the K x M row-major matrix in Rws.  ``steps`` bounds the
// number of pivots taken (min(K, M) in threshold mode, the fixed rank in
// fixed-rank mode; the first ``steps`` rows of R do not depend on later
// steps).  Writes perm (position k holds the original column), maxpivot and
// the nonzero-pivot count.
template <typename T>
__global__ void __launch_bounds__(256) k_cpqr(const i64* __restrict__ dims, const i64* __restrict__ krows,
                                              T* __restrict__ Rws, const i64* __restrict__ qoff,
                                              int* __restrict__ perm_out, const i64* __restrict__ xoff,
                                              double* __restrict__ maxpiv_out, int* __restrict__ nonzero_out,
                                              i64 step_cap) {
  const int box = blockIdx.x;
  const int M = (int)dims[box];
  const int K = (int)krows[box];
  if (M == 0 || K == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* nu = reinterpret_cast<double*>(smem_raw);  // updated norms
  double* nd = nu + M;                               // direct norms
  T* ess = reinterpret_cast<T*>(nd + M);             // K
  int* perm = reinterpret_cast<int*>(ess + K);       // M
  __shared__ double red_v[32];
  __shared__ int red_i[32];
  __shared__ T red_t[32];
  __shared__ int s_nonzero;
  __shared__ double s_maxpiv;

  T* W = Rws + qoff[box];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int size = K < M ? K : M;
  int steps = size;
  if (step_cap >= 0 && step_cap < steps) steps = (int)step_cap;

  for (int c = tid; c < M; c += nt) {
    double s = 0.;
    for (int r = 0; r < K; r++) {
      double v = (double)W[(i64)r * M + c];
      s += v * v;
    }
    nu[c] = sqrt(s);
    nd[c] = nu[c];
    perm[c] = c;
  }
  __syncthreads();
  double mx = 0.;
  int mi = 0;
  for (int c = tid; c < M; c += nt)
    if (nu[c] > mx) { mx = nu[c]; mi = c; }
  argmax_first(mx, mi, red_v, red_i);
  const double eps = (sizeof(T) == 8) ? DBL_EPSILON : (double)FLT_EPSILON;
  const double thr_helper = (mx * eps) * (mx * eps) / (double)K;
  const double downdate_thr = sqrt(eps);
  if (tid == 0) {
    s_nonzero = size;
    s_maxpiv = 0.;
  }
  __syncthreads();

  for (int k = 0; k < steps; k++) {
    double bv = -1.;
    int bi = 0x7fffffff;
    for (int c = k + tid; c < M; c += nt)
      if (nu[c] > bv) { bv = nu[c]; bi = c; }
    argmax_first(bv, bi, red_v, red_i);
    // No candidate compares greater when every norm is NaN: keep column k
    // rather than index outside the matrix.
    if (bi < k || bi >= M) bi = k;
    if (tid == 0) {
      if (s_nonzero == size && bv * bv < thr_helper * (double)(K - k)) s_nonzero = k;
      if (bi != k) {
        double t = nu[k]; nu[k] = nu[bi]; nu[bi] = t;
        t = nd[k]; nd[k] = nd[bi]; nd[bi] = t;
        int ti = perm[k]; perm[k] = perm[bi]; perm[bi] = ti;
      }
    }
    if (bi != k)
      for (int r = tid; r < K; r += nt) {
        T t = W[(i64)r * M + k];
        W[(i64)r * M + k] = W[(i64)r * M + bi];
        W[(i64)r * M + bi] = t;
      }
    __syncthreads();
    // Householder on column k, rows k..K-1.
    T part = 0;
    for (int r = k + 1 + tid; r < K; r += nt) {
      T v = W[(i64)r * M + k];
      part += v * v;
    }
    T tsq = BlockReduce<T>::sum(part, red_t);
    T c0 = W[(i64)k * M + k];
    T tau = 0, beta = c0, scale = 0;
    if (tsq > Tiny<T>::v()) {
      beta = sqrt(c0 * c0 + tsq);
      if (c0 >= T(0)) beta = -beta;
      scale = T(1) / (c0 - beta);
      tau = (beta - c0) / beta;
    }
    for (int r = k + 1 + tid; r < K; r += nt) {
      T e = W[(i64)r * M + k] * scale;
      ess[r] = e;
      W[(i64)r * M + k] = e;
    }
    if (tid == 0) {
      W[(i64)k * M + k] = beta;
      double ab = fabs((double)beta);
      if (ab > s_maxpiv) s_maxpiv = ab;
    }
    __syncthreads();
    for (int j = k + 1 + tid; j < M; j += nt) {
      if (tau != T(0)) {
        T w = W[(i64)k * M + j];
        for (int r = k + 1; r < K; r++) w += ess[r] * W[(i64)r * M + j];
        w *= tau;
        W[(i64)k * M + j] -= w;
        for (int r = k + 1; r < K; r++) W[(i64)r * M + j] -= w * ess[r];
      }
      if (nu[j] != 0.) {
        double t = fabs((double)W[(i64)k * M + j]) / nu[j];
        t = (1. + t) * (1. - t);
        if (t < 0.) t = 0.;
        double t2 = t * (nu[j] / nd[j]) * (nu[j] / nd[j]);
        if (t2 <= downdate_thr) {
          double s = 0.;
          for (int r = k + 1; r < K; r++) {
            double v = (double)W[(i64)r * M + j];
            s += v * v;
          }
          nd[j] = sqrt(s);
          nu[j] = nd[j];
        } else {
          nu[j] *= sqrt(t);
        }
      }
    }
    __syncthreads();
  }
  for (int c = tid; c < M; c += nt) perm_out[xoff[box] + c] = perm[c];
  if (tid == 0) {
    maxpiv_out[box] = s_maxpiv;
    nonzero_out[box] = s_nonzero;
  }
}

// Rank rule and interpolation coefficients: T = R11^{-1} R12 in place (rows
// 0..rank-1, columns rank..M-1 of the packed row-major factor in W).  One CTA
// per box and 128 columns, a column per thread: back substitution by 32-row
// blocks held in registers, R11 (scaled by the reciprocal pivots) staged in
// shared memory so that a row block's multipliers come as 16-byte broadcasts.
// Each element takes its updates from the last row upwards, unscaled, and is
// divided by its pivot at the end, so the order of the operations does not
// depend on the blocks.  Bound by FP64 FMA issue; with one barrier per row
// and one CTA per box this was bound by the barriers (0.49 ms a level at 256
// x 256 boxes of rank 128, whatever the number of boxes).
constexpr int INTERP_NT = 128, INTERP_JT = 64;

template <typename T>
__global__ void __launch_bounds__(INTERP_NT) k_interp(const i64* __restrict__ dims, const i64* __restrict__ krows,
                                                      T* __restrict__ Rws, const i64* __restrict__ qoff,
                                                      const double* __restrict__ maxpiv,
                                                      const int* __restrict__ nonzero, i64* __restrict__ ranks_out,
                                                      double epi) {
  constexpr int PS = 32 + 16 / sizeof(T);  // panel stride: 16-byte aligned columns, spread over the banks
  const int box = blockIdx.x, tid = threadIdx.x;
  const int M = (int)dims[box], K = (int)krows[box];
  __shared__ __align__(16) T P[INTERP_JT * PS];  // P[j][i] = R11[b0 + i][j0 + j]
  T* W = Rws + qoff[box];
  int rank = 0;
  if (M > 0 && K > 0) {
    if (epi < 1.) {
      const double thr = fabs(maxpiv[box]) * epi;
      const int nz = nonzero[box];
      for (int i0 = 0; i0 < nz; i0 += INTERP_NT) {
        const int i = i0 + tid;
        rank += __syncthreads_count(i < nz && fabs((double)W[(i64)i * M + i]) > thr);
      }
    } else {
      rank = min(min(K, M), (int)floor(fmin(epi, 2147483647.)));
    }
  }
  if (blockIdx.y == 0 && tid == 0) ranks_out[box] = rank;
  if (!(0 < rank && rank < M)) return;
  const int cb = rank + blockIdx.y * INTERP_NT;
  if (cb >= M) return;
  const int c = cb + tid;
  const bool cv = c < M;
  for (int b0 = (rank - 1) / 32 * 32; b0 >= 0; b0 -= 32) {
    const int bs = min(32, rank - b0);
    T r[32];
#pragma unroll
    for (int i = 0; i < 32; i++) r[i] = (cv && i < bs) ? W[(i64)(b0 + i) * M + c] : T(0);
    // Columns from the last one down to the block's own triangle.
    for (int je = rank; je > b0;) {
      const bool diag = je <= b0 + 32;
      const int jb = diag ? b0 : max(b0 + 32, je - INTERP_JT);
      __syncthreads();
      for (int e = tid; e < 32 * INTERP_JT; e += INTERP_NT) {
        const int j = e % INTERP_JT, i = e / INTERP_JT;
        T v = T(0);
        if (i < bs && jb + j < je) v = W[(i64)(b0 + i) * M + jb + j] * (T(1) / W[(i64)(jb + j) * (M + 1)]);
        P[j * PS + i] = v;
      }
      __syncthreads();
      if (diag) break;
      for (int j = je - 1; j >= jb; j -= 8) {
        T x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = (cv && j - u >= jb) ? W[(i64)(j - u) * M + c] : T(0);
#pragma unroll
        for (int u = 0; u < 8; u++) {
          if (j - u < jb) break;
          const T* p = P + (j - u - jb) * PS;
#pragma unroll
          for (int i = 0; i < 32; i++) r[i] -= p[i] * x[u];
        }
      }
      je = jb;
    }
#pragma unroll
    for (int jj = 31; jj >= 0; jj--) {
      if (jj >= bs) continue;
      const T* p = P + jj * PS;
#pragma unroll
      for (int i = 0; i < jj; i++) r[i] -= p[i] * r[jj];
    }
    if (cv)
#pragma unroll
      for (int i = 0; i < 32; i++)
        if (i < bs) W[(i64)(b0 + i) * M + c] = r[i];
  }
  if (cv)
#pragma unroll 8
    for (int i = 0; i < rank; i++) W[(i64)i * M + c] = W[(i64)i * M + c] / W[(i64)i * (M + 1)];
}

// The box basis from the interpolation coefficients, BASIS_COLS columns of a
// box per CTA.  Q (col-major, in/out) holds the incoming Q (identity at a
// leaf, the children's R blocks above); R (col-major, out, zero on entry).
// Operator mode: Q = P [I; T^T], zero columns after, R = I.  Orthogonal mode:
// U_ID = P [I; T^T] goes to R's slot and Q keeps the incoming Q (the caller
// forms triu(Q) U_ID, its QR and Q).  The first CTA of a box also puts its
// bodies in skeleton-first order.
constexpr int BASIS_COLS = 32;

template <typename T>
__global__ void __launch_bounds__(256) k_basis_build(const i64* __restrict__ dims, const i64* __restrict__ krows,
                                                     const T* __restrict__ Rws, T* __restrict__ Q, T* __restrict__ Rm,
                                                     const i64* __restrict__ qoff, const int* __restrict__ perm_in,
                                                     const i64* __restrict__ xoff, double* __restrict__ pts,
                                                     const i64* __restrict__ ranks, int orth) {
  const int box = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int M = (int)dims[box], i0 = blockIdx.y * BASIS_COLS;
  if (M == 0 || krows[box] == 0 || i0 >= M) return;
  const int rank = (int)ranks[box], w = min(BASIS_COLS, M - i0);
  const T* W = Rws + qoff[box];
  T* Qb = Q + qoff[box];
  T* Rb = Rm + qoff[box];
  if (!(0 < rank && rank < M)) {
    // R = upper triangle of the incoming Q, Q = identity (h2matrix.cpp:57-60).
    for_each_rc(M, w, [&](int r, int c, int) {
      const i64 e = r + (i64)(i0 + c) * M;
      Rb[e] = r <= i0 + c ? Qb[e] : T(0);
      Qb[e] = r == i0 + c ? T(1) : T(0);
    });
    return;
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int* perm = reinterpret_cast<int*>(smem_raw);                                 // M
  double* sp = reinterpret_cast<double*>(smem_raw + ((4 * M + 15) / 16) * 16);  // 3 M
  double* bp = pts + 3 * xoff[box];
  for (int c = tid; c < M; c += nt) perm[c] = perm_in[xoff[box] + c];
  if (i0 == 0)
    for (int e = tid; e < 3 * M; e += nt) sp[e] = bp[e];
  __syncthreads();
  if (i0 == 0)
    for (int e = tid; e < 3 * M; e += nt) bp[e] = sp[3 * perm[e / 3] + e % 3];
  T* out = orth ? Rb : Qb;
  for_each_rc(M, orth ? min(w, rank - i0) : w, [&](int k, int c, int) {
    const int i = i0 + c;
    T v = T(0);
    if (i < rank) v = k < rank ? (k == i ? T(1) : T(0)) : W[(i64)i * M + k];
    out[(i64)perm[k] + (i64)i * M] = v;
  });
  if (!orth)
    for (int i = i0 + tid; i < min(i0 + w, rank); i += nt) Rb[(i64)i * M + i] = T(1);
}

// ---------------------------------------------------------------- launchers

template <typename T>
cudaError_t launch_sample_tsqr(const KernelParams& kp, const double* bodies, const double* pts, const i64* xoff,
                               const i64* dims, const int* sidx, const i64* soff, T* Rws, const i64* qoff,
                               int nboxes, int maxM, cudaStream_t st) {
  if (nboxes == 0) return cudaSuccess;
  if (maxM > TS_THREADS * TS_MAXCOL) return cudaErrorInvalidValue;
  int tr = 32;
  while (tr > 8 && sizeof(T) * (tr * (size_t)maxM + 32) + sizeof(double) * 96 > 200 * 1024) tr /= 2;
  size_t smem = sizeof(T) * (tr * (size_t)maxM + 32) + sizeof(double) * 96;
  if (smem > 220 * 1024) return cudaErrorInvalidValue;  // box too large for one tile in shared memory
  auto fn = tr == 32 ? k_sample_tsqr<T, 32> : tr == 16 ? k_sample_tsqr<T, 16> : k_sample_tsqr<T, 8>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  note_launch();
  fn<<<nboxes, TS_THREADS, smem, st>>>(kp, bodies, pts, xoff, dims, sidx, soff, Rws, qoff);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_cpqr(const i64* dims, const i64* krows, T* Rws, const i64* qoff, int* perm, const i64* xoff,
                        double* maxpiv, int* nonzero, i64 step_cap, double epi, int nboxes, int maxM, cudaStream_t st) {
  if (nboxes == 0) return cudaSuccess;
  // Threshold (operator) bases whose matrix fits the shared memory of a
  // cluster.  Fixed-rank ones keep k_cpqr and its order of the sums: they are
  // formed here only in the mode that follows the reference's own sequence,
  // whose factorization amplifies the rounding of the bases to percents on the
  // ill-conditioned reference configuration.
  if (step_cap < 0) {
    bool done = false;
    const cudaError_t e = launch_cpqr_cluster<T>(dims, krows, Rws, qoff, perm, xoff, maxpiv, nonzero, 0.5 * epi,
                                                 nboxes, maxM, st, &done);
    if (e != cudaSuccess || done) return e;
  }
  size_t smem = 2 * sizeof(double) * maxM + sizeof(T) * maxM + sizeof(int) * maxM + 64;
  auto fn = k_cpqr<T>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  note_launch();
  fn<<<nboxes, 256, smem, st>>>(dims, krows, Rws, qoff, perm, xoff, maxpiv, nonzero, step_cap);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_basis_finish(const i64* dims, const i64* krows, T* Rws, T* Q, T* R, const i64* qoff,
                                const int* perm, const i64* xoff, const double* maxpiv, const int* nonzero,
                                double* pts, i64* ranks, double epi, int orth, int nboxes, int maxM,
                                cudaStream_t st) {
  if (nboxes == 0) return cudaSuccess;
  note_launch();
  k_interp<T><<<dim3(nboxes, (maxM + INTERP_NT - 1) / INTERP_NT), INTERP_NT, 0, st>>>(dims, krows, Rws, qoff, maxpiv,
                                                                                      nonzero, ranks, epi);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const size_t smem = ((4 * (size_t)maxM + 15) / 16) * 16 + sizeof(double) * 3 * maxM;
  e = cudaFuncSetAttribute(k_basis_build<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  note_launch();
  k_basis_build<T><<<dim3(nboxes, (maxM + BASIS_COLS - 1) / BASIS_COLS), 256, smem, st>>>(
      dims, krows, Rws, Q, R, qoff, perm, xoff, pts, ranks, orth);
  return cudaGetLastError();
}

#define INST(T)                                                                                                     \
  template cudaError_t launch_sample_tsqr<T>(const KernelParams&, const double*, const double*, const i64*,       \
                                             const i64*, const int*, const i64*, T*, const i64*, int, int,       \
                                             cudaStream_t);                                                       \
  template cudaError_t launch_cpqr<T>(const i64*, const i64*, T*, const i64*, int*, const i64*, double*, int*,    \
                                      i64, double, int, int, cudaStream_t);                                       \
  template cudaError_t launch_basis_finish<T>(const i64*, const i64*, T*, T*, T*, const i64*, const int*,         \
                                              const i64*, const double*, const int*, double*, i64*, double, int,  \
                                              int, int, cudaStream_t);
INST(double)
INST(float)
#undef INST

}  // namespace h2b

namespace h2b {

// Gathers each box's far-sample bodies into one contiguous array.
__global__ void k_gather_points(const double* __restrict__ bodies, const int* __restrict__ idx, i64 n,
                                double* __restrict__ out) {
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const double* p = bodies + 3 * (i64)idx[i];
    out[3 * i] = p[0];
    out[3 * i + 1] = p[1];
    out[3 * i + 2] = p[2];
  }
}

cudaError_t launch_gather_points(const double* bodies, const int* idx, i64 n, double* out, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  int grid = (int)((n + 255) / 256);
  grid = grid > 4096 ? 4096 : grid;
  note_launch();
  k_gather_points<<<grid, 256, 0, st>>>(bodies, idx, n, out);
  return cudaGetLastError();
}

}  // namespace h2b

namespace h2b {

// Blocked pivoted Cholesky of the Gram matrix G = XF^T XF (M x M per box,
// symmetric), stopped after ``steps`` pivots: the largest remaining Schur
// diagonal (the squared column norm a column-pivoted QR of XF would pick) is
// the pivot, so pivots and rows of R equal those of ColPivHouseholderQR in
// exact arithmetic (h2matrix.cpp:27).  Once the Schur diagonal falls to
// rounding noise of the FP64 Gram matrix (16 eps max diag), the pivots still to
// be taken get the row [floor, 0, ..., 0] with floor = sqrt(eps max diag):
// their interpolation coefficients come out exactly zero.
//
// k_pivchol_panel takes up to PC_NB pivots left-looking: row k of R is G's row
// of the pivot minus the panel's earlier rows, and the Schur diagonal loses
// R[k][j]^2.  Columns never move: thread j keeps its columns' position in the
// pivoted order (exchanged as swaps would) and their Schur diagonal in
// registers, the panel's rows of R are in shared memory (SM; in R itself for
// boxes too wide), and a pivot costs one barrier, the read of G's row from L2
// and the chain of the panel's rows.  k_pivchol_update subtracts
// R_panel^T R_panel from all of G, on the FP64 tensor cores (finished columns
// too: nothing reads those).  The panel that takes the last pivot puts R's rows
// in pivoted order, where k_cpqr leaves them, and writes perm.
//
// Bound: the latency of that chain, about 1.5 us a pivot.  With the rows and
// columns of G and R exchanged in memory and four barriers a pivot it was 5 us
// (0.6 ms a level of 128 pivots for 1 to 128 boxes), and the updates, planned on
// the host as GEMMs of the shrinking trailing blocks, left gaps of 0.5 ms a
// level: 65,536 bodies, nine levels, 5.8 -> 2.4 ms of kernels.
constexpr int PC_NB = 32, PC_NT = 256, PC_T = 64;

__device__ __forceinline__ unsigned long long pc_key(double v) {
  // Larger value, larger key; values not above -1 and NaN have key 0.
  if (!(v > -1.)) return 0ULL;
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ULL);
}
__device__ __forceinline__ double pc_value(unsigned long long key) {
  return __longlong_as_double((long long)((key >> 63) ? (key & 0x7fffffffffffffffULL) : ~key));
}
// Warp-wide largest key, and the smallest tag that has it.
__device__ __forceinline__ void pc_warp_best(unsigned long long& key, unsigned& tag) {
  const unsigned hi = (unsigned)(key >> 32), m = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = __reduce_max_sync(0xffffffffu, hi == m ? (unsigned)key : 0u);
  const unsigned long long best = ((unsigned long long)m << 32) | lo;
  tag = __reduce_min_sync(0xffffffffu, key == best ? tag : 0xffffffffu);
  key = best;
}

template <int CPT, bool SM>
__global__ void __launch_bounds__(PC_NT) k_pivchol_panel(const i64* __restrict__ dims,
                                                         const i64* __restrict__ steps_box, const double* __restrict__ G,
                                                         double* __restrict__ Rws, const i64* __restrict__ qoff,
                                                         int* __restrict__ perm_g, const i64* __restrict__ xoff,
                                                         double* __restrict__ state, int k0) {
  constexpr int NW = PC_NT / 32;
  const int box = blockIdx.x;
  const int M = (int)dims[box];
  const int steps = (int)steps_box[box];
  if (M == 0 || k0 >= steps) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long s_key[2][NW];
  __shared__ unsigned s_tag[2][NW];
  const double* g = G + qoff[box];
  double* R = Rws + qoff[box];
  double* Rp = SM ? reinterpret_cast<double*>(smem_raw) : R + (i64)k0 * M;  // the panel's rows, ld M
  int* perm = perm_g + xoff[box];  // positions of the columns until the last panel
  double* st = state + 3 * (i64)box;  // [rfloor, noise threshold, noise flag]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Best own column not yet taken, over the whole box; b: buffer.
  auto best = [&](unsigned long long& key, unsigned& tag, int b) {
    pc_warp_best(key, tag);
    if (lane == 0) {
      s_key[b][warp] = key;
      s_tag[b][warp] = tag;
    }
    __syncthreads();
    key = lane < NW ? s_key[b][lane] : 0ULL;
    tag = lane < NW ? s_tag[b][lane] : 0xffffffffu;
    pc_warp_best(key, tag);
  };
  int pos[CPT];
  double dsch[CPT];
#pragma unroll
  for (int u = 0; u < CPT; u++) {
    const int j = tid + u * PC_NT;
    pos[u] = j >= M ? -1 : k0 == 0 ? j : perm[j];
    dsch[u] = pos[u] >= k0 ? g[(i64)j * M + j] : 0.;
  }
  double rfloor, noise;
  bool noise_mode = false;
  if (k0 == 0) {
    unsigned long long key = 0;
    unsigned tag = 0;
#pragma unroll
    for (int u = 0; u < CPT; u++)
      if (pos[u] >= 0 && dsch[u] > 0. && pc_key(dsch[u]) > key) key = pc_key(dsch[u]);
    best(key, tag, 1);
    const double dmax = key ? pc_value(key) : 0.;
    const double rf = sqrt(DBL_EPSILON * dmax);
    rfloor = rf > 0. ? rf : DBL_MIN;
    noise = 16. * DBL_EPSILON * dmax;
    if (tid == 0) {
      st[0] = rfloor;
      st[1] = noise;
    }
  } else {
    rfloor = st[0];
    noise = st[1];
    noise_mode = st[2] != 0.;
  }
  const int kend = (k0 + PC_NB < steps) ? k0 + PC_NB : steps;
  for (int k = k0; k < kend; k++) {
    unsigned long long key = 0;
    unsigned tag = 0xffffffffu;  // position << 16 | column
#pragma unroll
    for (int u = 0; u < CPT; u++)
      if (pos[u] >= k) {
        const unsigned long long ku = pc_key(dsch[u]);
        const unsigned tu = ((unsigned)pos[u] << 16) | (unsigned)(tid + u * PC_NT);
        if (ku > key || (ku == key && tu < tag)) { key = ku; tag = tu; }
      }
    best(key, tag, (k - k0) & 1);
    const int p = (int)(tag >> 16), pc = (int)(tag & 0xffffu);
    double d = key ? pc_value(key) : __longlong_as_double(0x7ff8000000000000LL);
    if (!(d > noise)) noise_mode = true;
    double v[CPT];
    if (!noise_mode) {
#pragma unroll
      for (int u = 0; u < CPT; u++) {
        const int j = tid + u * PC_NT;
        v[u] = j < M ? g[(i64)pc * M + j] : 0.;
      }
    }
    const double rkk = sqrt(d);
    const double inv = 1. / rkk;
#pragma unroll
    for (int u = 0; u < CPT; u++) {
      const int j = tid + u * PC_NT;
      if (j == pc)
        pos[u] = k;
      else if (pos[u] == k)
        pos[u] = p;
    }
    if (noise_mode) {
#pragma unroll
      for (int u = 0; u < CPT; u++)
        if (pos[u] >= k) v[u] = pos[u] == k ? rfloor : 0.;
    } else {
#pragma unroll 8
      for (int i = 0; i < k - k0; i++) {
        const double m = Rp[(size_t)i * M + pc];
#pragma unroll
        for (int u = 0; u < CPT; u++) {
          const int j = tid + u * PC_NT;
          if (j < M) v[u] -= m * Rp[(size_t)i * M + j];
        }
      }
#pragma unroll
      for (int u = 0; u < CPT; u++) {
        if (pos[u] == k) {
          v[u] = rkk;
        } else {
          v[u] *= inv;
          dsch[u] -= v[u] * v[u];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < CPT; u++) {
      const int j = tid + u * PC_NT;
      if (j >= M) continue;
      const double x = pos[u] >= k ? v[u] : 0.;
      if (SM) Rp[(size_t)(k - k0) * M + j] = x;
      R[(i64)k * M + j] = x;
    }
    if (!SM) __threadfence_block();
  }
  if (tid == 0) st[2] = noise_mode ? 1. : 0.;
  if (kend < steps) {
#pragma unroll
    for (int u = 0; u < CPT; u++)
      if (pos[u] >= 0) perm[tid + u * PC_NT] = pos[u];
    return;
  }
  // Last panel: the rows in pivoted order, eight at a time.
  __syncthreads();
  for (int k = 0; k < steps; k += 8) {
    double v[8][CPT];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int u = 0; u < CPT; u++)
        v[i][u] = (k + i < steps && pos[u] >= 0) ? R[(i64)(k + i) * M + tid + u * PC_NT] : 0.;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int u = 0; u < CPT; u++)
        if (k + i < steps && pos[u] >= 0) R[(i64)(k + i) * M + pos[u]] = v[i][u];
  }
#pragma unroll
  for (int u = 0; u < CPT; u++)
    if (pos[u] >= 0) perm[pos[u]] = tid + u * PC_NT;
}

// G -= R_panel^T R_panel for one 64 x 64 tile of one box: mma.sync m8n8k4,
// four warps of 32 x 32.
__global__ void __launch_bounds__(128) k_pivchol_update(const i64* __restrict__ dims,
                                                        const i64* __restrict__ steps_box, double* __restrict__ G,
                                                        const double* __restrict__ Rws, const i64* __restrict__ qoff,
                                                        int k0) {
  constexpr int LD = PC_T + 4;
  const int box = blockIdx.x, M = (int)dims[box], steps = (int)steps_box[box];
  if (M == 0 || k0 + PC_NB >= steps) return;  // no pivot left to take
  const int nt = (M + PC_T - 1) / PC_T, r0 = (int)blockIdx.y / nt * PC_T, c0 = (int)blockIdx.y % nt * PC_T;
  if (r0 >= M) return;
  __shared__ double As[PC_NB][LD], Bs[PC_NB][LD];
  const double* R = Rws + qoff[box] + (i64)k0 * M;
  double* g = G + qoff[box];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp >> 1, wn = warp & 1;
  const int fr = lane >> 2, fk = lane & 3;
  for (int e = tid; e < PC_NB * PC_T; e += 128) {
    const int i = e / PC_T, j = e % PC_T;
    As[i][j] = r0 + j < M ? -R[(i64)i * M + r0 + j] : 0.;
    Bs[i][j] = c0 + j < M ? R[(i64)i * M + c0 + j] : 0.;
  }
  __syncthreads();
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.;
#pragma unroll
  for (int ks = 0; ks < PC_NB; ks += 4) {
    double a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = As[ks + fk][wm * 32 + i * 8 + fr];
#pragma unroll
    for (int j = 0; j < 4; j++) b[j] = Bs[ks + fk][wn * 32 + j * 8 + fr];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                     : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                     : "d"(a[i]), "d"(b[j]));
  }
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = r0 + wm * 32 + i * 8 + fr, c = c0 + wn * 32 + j * 8 + 2 * fk + h;
        if (r < M && c < M) acc[i][j][h] = g[r + (i64)c * M] + acc[i][j][h];
      }
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = r0 + wm * 32 + i * 8 + fr, c = c0 + wn * 32 + j * 8 + 2 * fk + h;
        if (r < M && c < M) g[r + (i64)c * M] = acc[i][j][h];
      }
}

cudaError_t launch_pivchol(const i64* dims, const i64* steps_box, double* G, double* Rws, const i64* qoff, int* perm,
                           const i64* xoff, double* state, int maxsteps, int nboxes, int maxM, cudaStream_t st) {
  if (nboxes == 0) return cudaSuccess;
  if (maxM > 8 * PC_NT) return cudaErrorInvalidValue;
  const size_t smem = sizeof(double) * (size_t)PC_NB * maxM;
  const bool sm = smem <= 200 * 1024;
  auto go = [&](auto kern, int k0) {
    if (sm) {
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    note_launch();
    kern<<<nboxes, PC_NT, sm ? smem : 0, st>>>(dims, steps_box, G, Rws, qoff, perm, xoff, state, k0);
    return cudaGetLastError();
  };
  const int nt = (maxM + PC_T - 1) / PC_T;
  for (int k0 = 0; k0 < maxsteps; k0 += PC_NB) {
    const cudaError_t e = maxM <= PC_NT       ? go(k_pivchol_panel<1, true>, k0)
                          : maxM <= 2 * PC_NT ? go(k_pivchol_panel<2, true>, k0)
                          : sm                ? go(k_pivchol_panel<4, true>, k0)
                                              : go(k_pivchol_panel<8, false>, k0);
    if (e != cudaSuccess) return e;
    if (k0 + PC_NB >= maxsteps) break;
    note_launch();
    k_pivchol_update<<<dim3(nboxes, nt * nt), 128, 0, st>>>(dims, steps_box, G, Rws, qoff, k0);
    const cudaError_t e2 = cudaGetLastError();
    if (e2 != cudaSuccess) return e2;
  }
  return cudaSuccess;
}

}  // namespace h2b

namespace h2b {

// T of the compact-WY form Q = H_0 ... H_{r-1} = I - V T V^T (forward,
// column by column: T[i][i] = tau_i, T[0:i, i] = -tau_i T[0:i,0:i] S[0:i, i]
// with S = V^T V), one CTA per box, r x r column-major at Tb + toff[box].
// Blocked: the 32 x 32 diagonal blocks are independent and are formed one
// per warp with the recurrence (lane j keeps row j of its block in
// registers, the column -tau_i S[0:i, i] is shared by shuffles; no barrier);
// the blocks above the diagonal follow from the product rule of compact-WY
// factors, T[A, B] = -T[A, A] S[A, B] T[B, B], for the leading columns A of
// each column block B in turn (two barriers per block instead of two per
// column).
constexpr int WY_B = 32;

template <typename T>
__device__ __forceinline__ void wy_diag_block(const WyTask<T>& t, int off, int bs, int lane) {
  const int r = t.r;
  T row[WY_B];
#pragma unroll
  for (int l = 0; l < WY_B; l++) row[l] = T(0);
#pragma unroll
  for (int i = 0; i < WY_B; i++) {
    if (i < bs) {
      const T tau = t.taus[off + i];
      const T c = lane < i ? -tau * t.S[(off + lane) + (i64)(off + i) * r] : T(0);
      T v = T(0);
#pragma unroll
      for (int l = 0; l < WY_B; l++) {
        const T cl = __shfl_sync(0xffffffffu, c, l);
        if (l < i) v += row[l] * cl;
      }
      if (lane < i) row[i] = v;
      if (lane == i) row[i] = tau;
    }
  }
  if (lane < bs) {
#pragma unroll
    for (int l = 0; l < WY_B; l++)
      if (l < bs) t.Tm[(off + lane) + (i64)(off + l) * r] = row[l];
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_wy_t(const WyTask<T>* __restrict__ tasks) {
  const WyTask<T> t = tasks[blockIdx.x];
  const int r = t.r;
  if (r <= 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* X = reinterpret_cast<T*>(smem_raw);  // (r - 32) x 32, column-major, ld r
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int nb = (r + WY_B - 1) / WY_B;
  // Zero the strictly lower triangle (the blocks below write only the upper part).
  for (i64 e = threadIdx.x; e < (i64)r * r; e += blockDim.x) {
    const int row = (int)(e % r), colm = (int)(e / r);
    if (row > colm) t.Tm[e] = T(0);
  }
  for (int b = warp; b < nb; b += nw) wy_diag_block(t, b * WY_B, min(WY_B, r - b * WY_B), lane);
  __syncthreads();
  for (int b = 1; b < nb; b++) {
    const int off = b * WY_B, bs = min(WY_B, r - off), p = off;
    // X = S[0:p, B] T[B, B]  (T[B, B] upper triangular)
    for (int e = threadIdx.x; e < p * bs; e += blockDim.x) {
      const int j = e % p, c = e / p;
      T v = T(0);
      for (int k = 0; k <= c; k++) v += t.S[j + (i64)(off + k) * r] * t.Tm[(off + k) + (i64)(off + c) * r];
      X[j + c * p] = v;
    }
    __syncthreads();
    // T[0:p, B] = -T[0:p, 0:p] X  (T[0:p, 0:p] upper triangular)
    for (int e = threadIdx.x; e < p * bs; e += blockDim.x) {
      const int j = e % p, c = e / p;
      T v = T(0);
      for (int k = j; k < p; k++) v += t.Tm[j + (i64)k * r] * X[k + c * p];
      t.Tm[j + (i64)(off + c) * r] = -v;
    }
    __syncthreads();
  }
}

template <typename T>
cudaError_t launch_wy_t(const WyTask<T>* d_tasks, int ntasks, int maxr, cudaStream_t st) {
  if (ntasks == 0) return cudaSuccess;
  const size_t smem = sizeof(T) * (size_t)std::max(1, maxr - WY_B) * WY_B;
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k_wy_t<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  note_launch();
  k_wy_t<T><<<ntasks, 256, smem, st>>>(d_tasks);
  return cudaGetLastError();
}
template cudaError_t launch_wy_t<double>(const WyTask<double>*, int, int, cudaStream_t);
template cudaError_t launch_wy_t<float>(const WyTask<float>*, int, int, cudaStream_t);

}  // namespace h2b

namespace h2b {

// One Householder panel of the M x rank matrix W (column-major, ld M) of a
// box: columns k0..k0+nb-1, rows k0..M-1, factored with the reference's
// reflector convention (beta = -sign(c0) * norm).  Writes back R (upper) and
// the reflector tails (lower), the explicit unit lower-trapezoidal V of the
// panel to Vp ((M-k0) x nb), the panel's compact-WY T (nb x nb, I - V T V^T =
// H_k0 ... H_k0+nb-1) to Tp and its taus.  k_qr_update applies the panel to the
// trailing columns.
//
// Bound: the chain of columns.  k_qr_panel keeps the panel in registers (rows
// over the lanes, RPL per lane; warp w the columns w, w + 8, ...) and needs two
// barriers per column -- the column published to shared memory, its norm's
// partial sums -- so a column costs the latency of one norm, one square root,
// a division and one dot product; with the panel in shared memory and a block
// reduction per column it was 5 us a column whatever the number of boxes
// (65,536 bodies, rank 128: panels and updates 6.7 -> 3.5 ms over eight levels).
// The sums keep their order (row k + 1 + i in lane i mod 32 of the norm and the
// dot products), hence the rotations.  Taller panels run k_qr_panel_smem.
template <typename T>
__device__ __forceinline__ void qr_panel_finish(const QrPanelTask<T>& t, const T* P, T* Tl, T* sc, const T* tau, int m,
                                                int nb, int k0) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  T* Wp = t.W + (i64)k0 + (i64)k0 * t.M;
  // S[l][i] = V(:,l)^T V(:,i) for l < i (V unit lower: V[i][i] = 1, zero above),
  // four l of one i at a time.
  for (int e = warp; e < nb * ((nb + 3) / 4); e += nw) {
    const int i = e % nb, l0 = e / nb * 4;
    if (l0 >= i) continue;
    T s[4] = {0, 0, 0, 0};
    for (int r = i + 1 + lane; r < m; r += 32) {
      const T x = P[r + (size_t)i * m];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (l0 + u < i) s[u] += P[r + (size_t)(l0 + u) * m] * x;
    }
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < 4; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
    if (lane == 0)
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (l0 + u < i) Tl[l0 + u + i * nb] = s[u] + P[i + (size_t)(l0 + u) * m];  // row i of V(:,l) times V[i][i] = 1
  }
  __syncthreads();
  // T recurrence, one warp: column i of S is staged in sc, then
  // T[:i, i] = -tau_i T[:i,:i] S[:i, i] and T[i][i] = tau_i.
  if (warp == 0) {
    for (int i = 0; i < nb; i++) {
      for (int j = lane; j < i; j += 32) sc[j] = Tl[j + i * nb];
      __syncwarp();
      for (int j = lane; j < i; j += 32) {
        T v = 0;
        for (int l = j; l < i; l++) v += Tl[j + l * nb] * sc[l];
        Tl[j + i * nb] = -tau[i] * v;
      }
      if (lane == 0) Tl[i + i * nb] = tau[i];
      __syncwarp();
    }
  } else {
    for (int e = tid - 32, n = nt - 32; e < m * nb; e += n) {
      const int r = e % m, j = e / m;
      Wp[r + (i64)j * t.M] = P[e];
      t.Vp[e] = r < j ? T(0) : (r == j ? T(1) : P[e]);
    }
  }
  __syncthreads();
  for (int e = tid; e < nb * nb; e += nt) {
    int r = e % nb, c = e / nb;
    t.Tp[e] = r <= c ? Tl[e] : T(0);
  }
  for (int j = tid; j < nb; j += nt) t.taus[k0 + j] = tau[j];
}

constexpr int QP_NT = 256, QP_NB = 32;

template <typename T, int RPL>
__global__ void __launch_bounds__(QP_NT) k_qr_panel(const QrPanelTask<T>* __restrict__ tasks, int k0) {
  constexpr int NW = QP_NT / 32, CPW = QP_NB / NW;
  const QrPanelTask<T> t = tasks[blockIdx.x];
  if (k0 >= t.rank) return;
  const int m = t.M - k0, nb = min(QP_NB, t.rank - k0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* P = reinterpret_cast<T*>(smem_raw);  // m x nb, ld m
  T* Tl = P + (size_t)m * nb;             // nb x nb
  __shared__ T col[2][RPL * 32];          // published column
  __shared__ T tau[QP_NB], sc[QP_NB], red[2][NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* Wp = t.W + (i64)k0 + (i64)k0 * t.M;
  T x[CPW][RPL];
#pragma unroll
  for (int u = 0; u < CPW; u++)
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i, c = warp + NW * u;
      x[u][i] = (r < m && c < nb) ? Wp[r + (i64)c * t.M] : T(0);
    }
  for (int j = 0; j < nb; j++) {
    const int ow = j % NW, os = j / NW, b = j & 1;
    if (warp == ow) {
#pragma unroll
      for (int u = 0; u < CPW; u++)
        if (u == os)
#pragma unroll
          for (int i = 0; i < RPL; i++) col[b][lane + 32 * i] = x[u][i];
    }
    __syncthreads();
    // Norm below the diagonal, in the order of a block reduction over rows.
    T part = 0;
    for (int r = j + 1 + tid; r < m; r += QP_NT) part += col[b][r] * col[b][r];
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) red[b][warp] = part;
    T v[RPL];
#pragma unroll
    for (int i = 0; i < RPL; i++) v[i] = col[b][lane + 32 * i];
    const T c0 = col[b][j];
    __syncthreads();
    const T* rb = red[b];
    const T tsq = ((rb[0] + rb[4]) + (rb[2] + rb[6])) + ((rb[1] + rb[5]) + (rb[3] + rb[7]));
    T tj = 0, beta = c0, scale = 0;
    if (tsq > Tiny<T>::v()) {
      beta = sqrt(c0 * c0 + tsq);
      if (c0 >= T(0)) beta = -beta;
      scale = T(1) / (c0 - beta);
      tj = (beta - c0) / beta;
    }
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i;
      v[i] = (r > j && r < m) ? v[i] * scale : T(0);
    }
    if (warp == ow) {
#pragma unroll
      for (int u = 0; u < CPW; u++)
        if (u == os)
#pragma unroll
          for (int i = 0; i < RPL; i++) {
            const int r = lane + 32 * i;
            if (r > j) x[u][i] = v[i];
            if (r == j) x[u][i] = beta;
          }
      if (lane == 0) tau[j] = tj;
    }
    if (tj != T(0) && warp + NW * (CPW - 1) > j) {  // else none of this warp's columns is left
      T w[CPW], cj[CPW];
#pragma unroll
      for (int u = 0; u < CPW; u++) {
        T s = 0;
#pragma unroll
        for (int i = 0; i < RPL; i++) s += v[i] * x[u][i];
        cj[u] = __shfl_sync(0xffffffffu, x[u][0], j);  // row j (j < 32)
        w[u] = __shfl_sync(0xffffffffu, s, (lane + j + 1) & 31);
      }
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < CPW; u++) w[u] += __shfl_xor_sync(0xffffffffu, w[u], o);
#pragma unroll
      for (int u = 0; u < CPW; u++) {
        if (warp + NW * u <= j) continue;
        const T wu = (w[u] + cj[u]) * tj;
#pragma unroll
        for (int i = 0; i < RPL; i++) {
          const int r = lane + 32 * i;
          if (r > j)
            x[u][i] -= wu * v[i];
          else if (r == j)
            x[u][i] -= wu;
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < CPW; u++)
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i, c = warp + NW * u;
      if (r < m && c < nb) P[r + (size_t)c * m] = x[u][i];
    }
  __syncthreads();
  qr_panel_finish(t, P, Tl, sc, tau, m, nb, k0);
}

template <typename T>
__global__ void __launch_bounds__(256) k_qr_panel_smem(const QrPanelTask<T>* __restrict__ tasks, int k0, int nbmax) {
  const QrPanelTask<T> t = tasks[blockIdx.x];
  if (k0 >= t.rank) return;
  const int m = t.M - k0, nb = min(nbmax, t.rank - k0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* P = reinterpret_cast<T*>(smem_raw);  // m x nb, ld m
  T* tau = P + (size_t)m * nb;            // nb
  T* Tl = tau + nb;                       // nb x nb
  T* sc = Tl + (size_t)nb * nb;           // nb
  __shared__ T red[32];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const T* Wp = t.W + (i64)k0 + (i64)k0 * t.M;
  for_each_rc(m, nb, [&](int r, int j, int e) {
    P[e] = Wp[r + (i64)j * t.M];
  });
  __syncthreads();
  for (int j = 0; j < nb; j++) {
    T* cj = P + (size_t)j * m;
    T part = 0;
    for (int r = j + 1 + tid; r < m; r += nt) part += cj[r] * cj[r];
    T tsq = BlockReduce<T>::sum(part, red);
    T c0 = cj[j];
    T tj = 0, beta = c0, scale = 0;
    if (tsq > Tiny<T>::v()) {
      beta = sqrt(c0 * c0 + tsq);
      if (c0 >= T(0)) beta = -beta;
      scale = T(1) / (c0 - beta);
      tj = (beta - c0) / beta;
    }
    __syncthreads();
    for (int r = j + 1 + tid; r < m; r += nt) cj[r] *= scale;
    if (tid == 0) {
      cj[j] = beta;
      tau[j] = tj;
    }
    __syncthreads();
    if (tj != T(0))
      for (int jj = j + 1 + warp; jj < nb; jj += nw) {
        T* c2 = P + (size_t)jj * m;
        T w = 0;
        for (int r = j + 1 + lane; r < m; r += 32) w += cj[r] * c2[r];
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        w = (w + c2[j]) * tj;
        if (lane == 0) c2[j] -= w;
        for (int r = j + 1 + lane; r < m; r += 32) c2[r] -= w * cj[r];
      }
    __syncthreads();
  }
  qr_panel_finish(t, P, Tl, sc, tau, m, nb, k0);
}

// The panel applied to the trailing columns, A -= V (T^T (V^T A)): one CTA per
// box and QU_C columns of A (rows k0..M-1).  The three products run in one
// launch (three GEMM launches and their host-built task lists a panel before):
// FP64 on the tensor cores (mma.sync m8n8k4, V and A read where they lie, their
// four consecutive k of a fragment being one 32-byte sector), FP32 on the FMA
// pipe (bases of the Householder mode only).
constexpr int QU_C = 32;

template <typename T>
__global__ void __launch_bounds__(256) k_qr_update(const QrPanelTask<T>* __restrict__ tasks, int k0, int nbmax) {
  constexpr int LD = 36;
  const QrPanelTask<T> t = tasks[blockIdx.x];
  const int nb = min(nbmax, t.rank - k0), m = t.M - k0;
  const int c0 = k0 + nb + blockIdx.y * QU_C;
  if (nb <= 0 || c0 >= t.rank) return;
  const int nc = min(QU_C, t.rank - c0);
  __shared__ T Y[QU_C][LD], Y2[QU_C][LD], Ts[QU_C][LD];  // [column][row]
  const T* V = t.Vp;  // m x nb, ld m
  T* A = t.W + k0 + (i64)c0 * t.M;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < 32 * 32; e += 256) {
    const int r = e & 31, c = e >> 5;
    Ts[c][r] = (r < nb && c < nb) ? t.Tp[r + c * nb] : T(0);
  }
  if constexpr (sizeof(T) == 8) {
    const int fr = lane >> 2, fk = lane & 3;
    auto mma = [](double (&d)[2], double a, double b) {
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                   : "+d"(d[0]), "+d"(d[1])
                   : "d"(a), "d"(b));
    };
    // Y = V^T A: warp w has rows 8 (w % 4).. and the two column groups w / 4, + 2.
    const int yr = 8 * (warp & 3) + fr, yc = 8 * (warp >> 2) + fr;
    double y[2][2] = {{0., 0.}, {0., 0.}};
    const bool av = yr < nb, bv0 = yc < nc, bv1 = yc + 16 < nc;
    const double *va = V + (i64)yr * m + fk, *a0 = A + (i64)yc * t.M + fk, *a1 = a0 + 16 * (i64)t.M;
    for (int k = 0; k < m; k += 32) {
      double fa[8], f0[8], f1[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const bool kv = k + 4 * i + fk < m;
        fa[i] = (av && kv) ? va[k + 4 * i] : 0.;
        f0[i] = (bv0 && kv) ? a0[k + 4 * i] : 0.;
        f1[i] = (bv1 && kv) ? a1[k + 4 * i] : 0.;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        mma(y[0], fa[i], f0[i]);
        mma(y[1], fa[i], f1[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) Y[8 * (warp >> 2) + 16 * i + 2 * fk + h][yr] = y[i][h];
    __syncthreads();
    // Y2 = T^T Y (T[k][row] at Ts[row][k]).
    y[0][0] = y[0][1] = y[1][0] = y[1][1] = 0.;
#pragma unroll
    for (int k = 0; k < 32; k += 4)
#pragma unroll
      for (int i = 0; i < 2; i++) mma(y[i], Ts[yr][k + fk], Y[yc + 16 * i][k + fk]);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) Y2[8 * (warp >> 2) + 16 * i + 2 * fk + h][yr] = y[i][h];
    __syncthreads();
    // A -= V Y2, 16 rows x 32 columns a warp at a time.
    for (int r0 = 16 * warp; r0 < m; r0 += 128) {
      double acc[2][4][2];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.;
      double fa[2][8];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int r = r0 + 8 * i + fr, kk = 4 * k + fk;
          fa[i][k] = (r < m && kk < nb) ? -V[r + (i64)kk * m] : 0.;
        }
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const double f = Y2[8 * j + fr][4 * k + fk];
          mma(acc[0][j], fa[0][k], f);
          mma(acc[1][j], fa[1][k], f);
        }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int r = r0 + 8 * i + fr, c = 8 * j + 2 * fk + h;
            if (r < m && c < nc) acc[i][j][h] = A[r + (i64)c * t.M] + acc[i][j][h];
          }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int r = r0 + 8 * i + fr, c = 8 * j + 2 * fk + h;
            if (r < m && c < nc) A[r + (i64)c * t.M] = acc[i][j][h];
          }
    }
  } else {
    for (int e = tid; e < 32 * 32; e += 256) {
      const int r = e & 31, c = e >> 5;
      T s = T(0);
      if (r < nb && c < nc)
        for (int k = 0; k < m; k++) s += V[k + (i64)r * m] * A[k + (i64)c * t.M];
      Y[c][r] = s;
    }
    __syncthreads();
    for (int e = tid; e < 32 * 32; e += 256) {
      const int r = e & 31, c = e >> 5;
      T s = T(0);
      for (int k = 0; k <= r; k++) s += Ts[r][k] * Y[c][k];
      Y2[c][r] = s;
    }
    __syncthreads();
    for_each_rc(m, nc, [&](int r, int c, int) {
      T s = T(0);
      for (int k = 0; k < nb; k++) s += V[r + (i64)k * m] * Y2[c][k];
      A[r + (i64)c * t.M] -= s;
    });
  }
}

int qr_panel_width(int maxM, size_t elem) {
  if (maxM <= 512) return QP_NB;
  int nb = QP_NB;
  while (nb > 1 && elem * ((size_t)maxM * nb + 2 * nb + (size_t)nb * nb) > 190 * 1024) nb--;
  return nb;
}

template <typename T>
cudaError_t launch_blocked_qr(const QrPanelTask<T>* d_tasks, int ntasks, int maxM, int maxr, cudaStream_t st) {
  if (ntasks == 0) return cudaSuccess;
  const int nb = qr_panel_width(maxM, sizeof(T));
  for (int k0 = 0; k0 < maxr; k0 += nb) {
    const int m = maxM - k0;
    auto go = [&](auto kern, auto... more) {
      const size_t smem = sizeof(T) * ((size_t)m * nb + 2 * nb + (size_t)nb * nb) + 16;
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      note_launch();
      kern<<<ntasks, 256, smem, st>>>(d_tasks, k0, more...);
      return cudaGetLastError();
    };
    // 256 rows: 8 a lane; up to 512: 16.
    cudaError_t e = maxM > 512 ? go(k_qr_panel_smem<T>, nb) : m <= 256 ? go(k_qr_panel<T, 8>) : go(k_qr_panel<T, 16>);
    if (e != cudaSuccess) return e;
    if (k0 + nb >= maxr) break;
    note_launch();
    k_qr_update<T><<<dim3(ntasks, (maxr - k0 - nb + QU_C - 1) / QU_C), 256, 0, st>>>(d_tasks, k0, nb);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template cudaError_t launch_blocked_qr<double>(const QrPanelTask<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_blocked_qr<float>(const QrPanelTask<float>*, int, int, int, cudaStream_t);

}  // namespace h2b

namespace h2b {

// After the blocked QR of W (M x rank): R's slot gets triu(W[:rank, :rank]),
// W becomes the explicit unit lower-trapezoidal V, Q the identity (for the
// compact-WY formation that follows).
// gridDim.y CTAs per box, each its own columns.
template <typename T>
__global__ void __launch_bounds__(256) k_qr_extract(const QrExtractTask<T>* __restrict__ tasks) {
  const QrExtractTask<T> t = tasks[blockIdx.x];
  const int M = t.M, r = t.rank, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = blockIdx.y * 8 + warp; c < M; c += gridDim.y * 8) {
    const i64 o = (i64)c * M;
#pragma unroll 4
    for (int i = lane; i < M; i += 32) {
      const T w = c < r ? t.W[o + i] : T(0);
      t.R[o + i] = (c < r && i <= c) ? w : T(0);
      t.Q[o + i] = i == c ? T(1) : T(0);
      if (c < r && i <= c) t.W[o + i] = i == c ? T(1) : T(0);
    }
  }
}

template <typename T>
cudaError_t launch_qr_extract(const QrExtractTask<T>* d_tasks, int ntasks, cudaStream_t st) {
  if (ntasks == 0) return cudaSuccess;
  note_launch();
  k_qr_extract<T><<<dim3(ntasks, 8), 256, 0, st>>>(d_tasks);
  return cudaGetLastError();
}
template cudaError_t launch_qr_extract<double>(const QrExtractTask<double>*, int, cudaStream_t);
template cudaError_t launch_qr_extract<float>(const QrExtractTask<float>*, int, cudaStream_t);

}  // namespace h2b
