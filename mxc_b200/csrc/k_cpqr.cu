// Column-pivoted Householder QR of every box of a level, the matrix of one
// box spread over the shared memory of a thread-block cluster.
#include "common.cuh"
#include "kernels.h"

#include <cfloat>
#include <cooperative_groups.h>

namespace h2b {

namespace cg = cooperative_groups;

// Column-pivoted Householder QR (Eigen 3.4 ColPivHouseholderQR::computeInPlace
// restated: h2matrix.cpp:27) of the K x M row-major matrix in Rws, K <= M, K
// pivots or
// until the largest remaining norm is below stop_rel times the largest pivot
// (a remaining column's later pivots are no larger than its norm now, so with
// stop_rel under the caller's rank threshold none of them counts and no row
// of R they would give is read; the columns left over keep their order).
// Writes the rows of R in pivoted column order (entries below
// the diagonal are left as they were), perm (position k holds the original
// column), maxpivot and the nonzero-pivot count.
//
// Bound: the serial chain of pivots -- pick a column, form its reflector,
// apply it to every other column -- one box at a time per CTA group.  The
// matrix (312 x 312 FP64 = 779 KB at the 20,000-body run's leaves) does not
// fit one SM, and every pass over it through L2 cost about 90 us per pivot.
// So a cluster of CL CTAs holds it: CTA q keeps the columns [q nc, (q + 1)
// nc) in shared memory, column-major with an odd leading dimension, for the
// whole factorization; a pivot costs one cluster barrier (each CTA sends its
// best column norm to all others through distributed shared memory) and one
// read of the pivot column from its owner, from which every CTA forms the
// reflector itself.  Columns never move: each keeps its position in the
// pivoted order, exchanged as the reference's swaps would.  A warp applies
// the reflector to a few columns at a time, their rows over the lanes, the
// reflector in registers (RPL rows per lane) for the whole step; the norm
// downdates run one thread per column afterwards.  The 20,000-body operator's
// five levels (64 to 1 boxes of up to 312 columns, eps 1e-8) went from 102 to
// 6.3 ms, half of that by stopping at the threshold; a pivot of a 312-column
// box over 4 CTAs takes about 11,000 clocks: 6,600 for the columns (FP64
// latency and the shuffles of the dot products), the rest for the barriers,
// the reflector's square root and divisions and the downdates.
template <typename T>
struct CpqrTiny;
template <>
struct CpqrTiny<double> { static __device__ double v() { return DBL_MIN; } };
template <>
struct CpqrTiny<float> { static __device__ float v() { return FLT_MIN; } };

constexpr int CPQR_NT = 512;
constexpr int CPQR_MAXCL = 16;

__host__ __device__ constexpr int cpqr_ld(int K) { return K | 1; }

template <typename T>
size_t cpqr_smem(int M, int cl) {
  const size_t nc = (size_t)((M + cl - 1) / cl);
  return 2 * sizeof(double) * nc + sizeof(T) * (nc * cpqr_ld(M) + M + nc) + sizeof(int) * nc + 32;
}

// Warp-wide largest key, and the smallest tag that has it.
__device__ __forceinline__ void cpqr_warp_best(unsigned long long& key, unsigned& tag) {
  const unsigned hi = (unsigned)(key >> 32), m = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = __reduce_max_sync(0xffffffffu, hi == m ? (unsigned)key : 0u);
  const unsigned long long best = ((unsigned long long)m << 32) | lo;
  tag = __reduce_min_sync(0xffffffffu, key == best ? tag : 0xffffffffu);
  key = best;
}

template <typename T, int RPL>
__global__ void __launch_bounds__(CPQR_NT) k_cpqr_cluster(const i64* __restrict__ dims, const i64* __restrict__ krows,
                                                          T* __restrict__ Rws, const i64* __restrict__ qoff,
                                                          int* __restrict__ perm_out, const i64* __restrict__ xoff,
                                                          double* __restrict__ maxpiv_out,
                                                          int* __restrict__ nonzero_out, double stop_rel) {
  constexpr int NW = CPQR_NT / 32, CG = RPL <= 8 ? 3 : RPL <= 12 ? 2 : 1, RG = 4;
  cg::cluster_group cl = cg::this_cluster();
  const int CL = (int)cl.num_blocks(), q = (int)cl.block_rank();
  const int box = blockIdx.x / CL;
  const int M = (int)dims[box], K = (int)krows[box];
  if (M == 0 || K == 0) return;
  const int ldk = cpqr_ld(K), nc = (M + CL - 1) / CL, c0 = q * nc, ncl = max(0, min(nc, M - c0));
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* nu = reinterpret_cast<double*>(smem_raw);  // updated norms of the own columns
  double* nd = nu + nc;                              // direct norms
  T* cols = reinterpret_cast<T*>(nd + nc);           // nc columns of K rows
  T* vbuf = cols + (size_t)nc * ldk;                 // pivot column, rows 0..K-1
  T* betas = vbuf + K;                               // diagonal of R of retired columns
  int* pos = reinterpret_cast<int*>(betas + nc);     // position in the pivoted order
  __shared__ unsigned long long cand_k[2][CPQR_MAXCL], red_k[NW];
  __shared__ unsigned cand_c[2][CPQR_MAXCL], red_c[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T* W = Rws + qoff[box];
  for (int r = warp; r < K; r += NW)
    for (int l = lane; l < ncl; l += 32) cols[(size_t)l * ldk + r] = W[(i64)r * M + c0 + l];
  __syncthreads();
  for (int l = warp; l < ncl; l += NW) {
    double s = 0.;
    for (int r = lane; r < K; r += 32) {
      const double v = (double)cols[(size_t)l * ldk + r];
      s += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      nu[l] = nd[l] = sqrt(s);
      pos[l] = c0 + l;
    }
  }
  // Of the whole cluster: the first candidates go to the other CTAs' shared
  // memory, which may be written only once those CTAs are known to run.
  cl.sync();
  int steps = K < M ? K : M;
  const double eps = (sizeof(T) == 8) ? DBL_EPSILON : (double)FLT_EPSILON;
  const double downdate_thr = sqrt(eps);
  double thr_helper = 0., maxpiv = 0.;
  int nonzero = steps;

  for (int k = 0; k < steps; k++) {
    // 1. Best own column: largest norm, smallest position on ties (integer
    //    maxima of the norms' bit patterns; a NaN norm has key 0, so with NaNs
    //    only the column at position k is taken).
    unsigned long long key = 0;
    unsigned tag = 0xffffffffu;  // position << 16 | column
    for (int l = tid; l < ncl; l += CPQR_NT) {
      const int p = pos[l];
      const double v = nu[l];
      const unsigned long long kv = v >= 0. ? (unsigned long long)__double_as_longlong(v) + 1ULL : 0ULL;
      const unsigned tv = ((unsigned)p << 16) | (unsigned)(c0 + l);
      if (p >= k && (kv > key || (kv == key && tv < tag))) { key = kv; tag = tv; }
    }
    cpqr_warp_best(key, tag);
    if (lane == 0) { red_k[warp] = key; red_c[warp] = tag; }
    __syncthreads();
    if (warp == 0) {
      key = lane < NW ? red_k[lane] : 0ULL;
      tag = lane < NW ? red_c[lane] : 0xffffffffu;
      cpqr_warp_best(key, tag);
      if (lane < CL) {
        *cl.map_shared_rank(&cand_k[k & 1][q], lane) = key;
        *cl.map_shared_rank(&cand_c[k & 1][q], lane) = tag;
      }
    }
    cl.sync();
    key = lane < CL ? cand_k[k & 1][lane] : 0ULL;
    tag = lane < CL ? cand_c[k & 1][lane] : 0xffffffffu;
    cpqr_warp_best(key, tag);
    const int bp = (int)(tag >> 16), bc = (int)(tag & 0xffffu);
    const double bv = key ? __longlong_as_double((long long)(key - 1ULL)) : -1.;
    if (bv >= 0. && bv < stop_rel * maxpiv) {  // uniform over the cluster
      steps = k;
      break;
    }
    if (k == 0) thr_helper = bv > 0. ? (bv * eps) * (bv * eps) / (double)K : 0.;
    if (nonzero == steps && bv * bv < thr_helper * (double)(K - k)) nonzero = k;
    // 2. Reflector of the pivot column, read from its owner; the column is
    //    not written again, so no barrier protects the read.
    const int owner = bc / nc;
    const T* pc = cl.map_shared_rank(cols, owner) + (size_t)(bc - owner * nc) * ldk;
    for (int r = k + tid; r < K; r += CPQR_NT) vbuf[r] = pc[r];
    for (int l = tid; l < ncl; l += CPQR_NT) {  // the exchange of positions k and bp
      if (c0 + l == bc)
        pos[l] = k;
      else if (pos[l] == k)
        pos[l] = bp;
    }
    __syncthreads();
    const T c0v = vbuf[k];
    T v[RPL];
    T part[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i;
      v[i] = (r > k && r < K) ? vbuf[r] : T(0);
      part[i & 3] += v[i] * v[i];
    }
    T tsq = (part[0] + part[1]) + (part[2] + part[3]);
    for (int o = 16; o > 0; o >>= 1) tsq += __shfl_xor_sync(0xffffffffu, tsq, o);
    T tau = 0, beta = c0v, scale = 0;
    if (tsq > CpqrTiny<T>::v()) {
      beta = sqrt(c0v * c0v + tsq);
      if (c0v >= T(0)) beta = -beta;
      scale = T(1) / (c0v - beta);
      tau = (beta - c0v) / beta;
    }
    maxpiv = fmax(maxpiv, fabs((double)beta));
    if (tid == 0 && owner == q) betas[bc - c0] = beta;
    // 3. Columns c -= tau (v^T c) v with v = (1, scale pc[k+1..]).
    if (tau != T(0)) {
#pragma unroll
      for (int i = 0; i < RPL; i++) v[i] *= scale;
      // CG columns at a time, so that their loads and shuffles overlap.
      for (int l0 = warp; l0 < ncl; l0 += NW * CG) {
        T x[CG][RPL], w[CG], ck[CG];
        T* c[CG];
        bool on[CG];
#pragma unroll
        for (int u = 0; u < CG; u++) {
          const int l = l0 + NW * u;
          on[u] = l < ncl && pos[l] > k;
          c[u] = cols + (size_t)(on[u] ? l : l0) * ldk + lane;
          ck[u] = c[u][k - lane];
          w[u] = 0;
        }
        // Groups of RG row blocks, skipped whole above row k and past row K:
        // within a group every load is in flight before the first use.
#pragma unroll
        for (int g = 0; g < RPL; g += RG)
          if (32 * (g + RG) > k && 32 * g < K) {
#pragma unroll
            for (int i = g; i < g + RG; i++)
#pragma unroll
              for (int u = 0; u < CG; u++) x[u][i] = lane + 32 * i < K ? c[u][32 * i] : T(0);
            T s[CG];
#pragma unroll
            for (int u = 0; u < CG; u++) s[u] = 0;
#pragma unroll
            for (int i = g; i < g + RG; i++)
#pragma unroll
              for (int u = 0; u < CG; u++) s[u] += v[i] * x[u][i];
#pragma unroll
            for (int u = 0; u < CG; u++) w[u] += s[u];
          }
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < CG; u++) w[u] += __shfl_xor_sync(0xffffffffu, w[u], o);
#pragma unroll
        for (int u = 0; u < CG; u++) w[u] = (w[u] + ck[u]) * tau;
#pragma unroll
        for (int g = 0; g < RPL; g += RG)
          if (32 * (g + RG) > k && 32 * g < K) {
#pragma unroll
            for (int i = g; i < g + RG; i++)
#pragma unroll
              for (int u = 0; u < CG; u++) {
                const int r = lane + 32 * i;
                if (on[u] && r >= k && r < K) c[u][32 * i] = r == k ? ck[u] - w[u] : x[u][i] - w[u] * v[i];
              }
          }
        __syncwarp();
      }
    }
    __syncthreads();
    // 4. Norm downdates, a column per thread; a warp sums the columns whose
    //    downdated norm is no longer trusted together (nearly every pivot has
    //    one: summed by its own thread it took longer than all the rest).
    for (int l0 = warp * 32; l0 < ncl; l0 += CPQR_NT) {
      const int l = l0 + lane;
      bool fresh = false;
      if (l < ncl && pos[l] > k && nu[l] != 0.) {
        double t = fabs((double)cols[(size_t)l * ldk + k]) / nu[l];
        t = (1. + t) * (1. - t);
        if (t < 0.) t = 0.;
        const double t2 = t * (nu[l] / nd[l]) * (nu[l] / nd[l]);
        fresh = t2 <= downdate_thr;
        if (!fresh) nu[l] *= sqrt(t);
      }
      for (unsigned m = __ballot_sync(0xffffffffu, fresh); m; m &= m - 1) {
        const int u = __ffs(m) - 1;
        const T* c = cols + (size_t)(l0 + u) * ldk;
        double s = 0.;
        for (int r = k + 1 + lane; r < K; r += 32) {
          const double x = (double)c[r];
          s += x * x;
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == u) nu[l] = nd[l] = sqrt(s);
      }
    }
  }
  // Every CTA is done reading the others' columns (and W, long ago).
  cl.sync();
  for (int r = warp; r < steps; r += NW)
    for (int l = lane; l < ncl; l += 32) {
      const int p = pos[l];
      if (p >= r) W[(i64)r * M + p] = p == r ? betas[l] : cols[(size_t)l * ldk + r];
    }
  for (int l = tid; l < ncl; l += CPQR_NT) perm_out[xoff[box] + pos[l]] = c0 + l;
  if (q == 0 && tid == 0) {
    maxpiv_out[box] = maxpiv;
    nonzero_out[box] = min(nonzero, steps);
  }
}

template <typename T, int RPL>
static cudaError_t cpqr_cluster_go(const i64* dims, const i64* krows, T* Rws, const i64* qoff, int* perm,
                                   const i64* xoff, double* maxpiv, int* nonzero, double stop_rel, int nboxes, int cl,
                                   size_t smem, cudaStream_t st, bool* launched) {
  auto fn = k_cpqr_cluster<T, RPL>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && cl > 8) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nboxes * cl));
  cfg.blockDim = dim3(CPQR_NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cl > 8) {  // a size the device may have no room for
    int nclus = 0;
    e = cudaOccupancyMaxActiveClusters(&nclus, fn, &cfg);
    if (e != cudaSuccess || nclus < 1) {
      cudaGetLastError();
      return cudaSuccess;
    }
  }
  note_launch();
  e = cudaLaunchKernelEx(&cfg, fn, dims, krows, Rws, qoff, perm, xoff, maxpiv, nonzero, stop_rel);
  *launched = e == cudaSuccess;
  return e;
}

template <typename T>
cudaError_t launch_cpqr_cluster(const i64* dims, const i64* krows, T* Rws, const i64* qoff, int* perm,
                                const i64* xoff, double* maxpiv, int* nonzero, double stop_rel, int nboxes, int maxM,
                                cudaStream_t st, bool* launched) {
  *launched = false;
  constexpr size_t kMax = 200 * 1024;
  int cl = 1;
  while (cl <= CPQR_MAXCL && cpqr_smem<T>(maxM, cl) > kMax) cl *= 2;
  if (cl > CPQR_MAXCL || maxM > 768) return cudaSuccess;
  // A level with few boxes leaves SMs idle: more CTAs per box shorten a pivot.
  while (cl < 8 && nboxes * cl * 2 <= 148 && maxM / (cl * 2) >= 32) cl *= 2;
  const size_t smem = cpqr_smem<T>(maxM, cl);
  auto go = maxM <= 256   ? cpqr_cluster_go<T, 8>
            : maxM <= 384 ? cpqr_cluster_go<T, 12>
            : maxM <= 512 ? cpqr_cluster_go<T, 16>
                          : cpqr_cluster_go<T, 24>;
  return go(dims, krows, Rws, qoff, perm, xoff, maxpiv, nonzero, stop_rel, nboxes, cl, smem, st, launched);
}
template cudaError_t launch_cpqr_cluster<double>(const i64*, const i64*, double*, const i64*, int*, const i64*,
                                                 double*, int*, double, int, int, cudaStream_t, bool*);
template cudaError_t launch_cpqr_cluster<float>(const i64*, const i64*, float*, const i64*, int*, const i64*,
                                                double*, int*, double, int, int, cudaStream_t, bool*);

}  // namespace h2b
