// Multi-right-hand-side block apply by rows: C_task (m x n, n <= 16) =
// beta C + sum_e alpha_e A_e B_e with A_e and B_e as stored (column-major).
#include "common.cuh"
#include "kernels.h"

#include <cstdint>
#include <type_traits>

namespace h2b {

// One CTA per 32 RL rows of a task, the whole sum over k inside it: the
// entries' columns are cut into chunks of AP_KC, dealt to the CTA's warps in
// turn, and the warps' sums are added in order through shared memory (no
// partial results in HBM, no second launch).  A lane owns RL adjacent rows and
// all NR columns; a chunk of A goes straight from HBM to registers (a warp
// reads 32 RL consecutive rows of a column), the chunk of B through the warp's
// own shared memory as 16-byte broadcasts, and the next chunk's loads are in
// flight while one is multiplied.  No barrier runs inside the loop.
//
// FP32 multiplies are plain FP32 (packed pairs, fma.rn.f32x2); BF16 blocks are
// widened and multiplied in FP32.
//
// Bound: the latency of one CTA -- task and entry reads, one chunk's loads per
// AP_KC NW columns, the sum over the warps -- about 8 us a launch at K 256,
// where the shared-memory ring took 15 with the launch that adds its partial
// sums.  With at most 4 columns also the faster kernel where HBM bounds it (4.5
// TB/s against 3.7; the exception is a substitution of 262,144 bodies in FP32
// with one or two columns, 1,608 against 1,583 us); with 16 the ring is (a warp
// reads 256 or 512 bytes of a column here, the ring 512 to 2,048).
constexpr int AP_KC = 16, AP_EMAX = 64;

template <typename AT, typename T>
struct ApEntry {
  const AT* A;
  const T* B;
  i64 lda, ldb;
  int k, vec;
  T alpha;
};

template <typename T>
__device__ __forceinline__ void ap_load(const GemmEntry<T>& e, ApEntry<T, T>& o) {
  o.A = e.A; o.B = e.B; o.lda = e.lda; o.ldb = e.ldb; o.k = e.k; o.alpha = e.alpha;
}
__device__ __forceinline__ void ap_load(const BfEntry& e, ApEntry<__nv_bfloat16, float>& o) {
  o.A = e.A; o.B = e.B; o.lda = e.lda; o.ldb = e.ldb; o.k = e.k; o.alpha = e.alpha * *e.scale;
}

// RL adjacent elements of a column.
template <typename AT, int RL>
struct ApVec;
template <> struct ApVec<float, 1> { using V = float; };
template <> struct ApVec<float, 2> { using V = float2; };
template <> struct ApVec<double, 1> { using V = double; };
template <> struct ApVec<double, 2> { using V = double2; };
template <> struct ApVec<__nv_bfloat16, 2> { using V = __nv_bfloat162; };

__device__ __forceinline__ float ap_up(float v) { return v; }
__device__ __forceinline__ double ap_up(double v) { return v; }
__device__ __forceinline__ float ap_up(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename V>
__device__ __forceinline__ V ap_zero() { return V{}; }
template <>
__device__ __forceinline__ __nv_bfloat16 ap_zero() { return __float2bfloat16(0.f); }
template <>
__device__ __forceinline__ __nv_bfloat162 ap_zero() { return __floats2bfloat162_rn(0.f, 0.f); }

template <typename AT, typename T, typename ENT, int NR, int RL, int NW>
__global__ void __launch_bounds__(NW * 32, sizeof(T) * RL * NR <= 128 ? 2 : 1) k_apply(const GemmTask<T>* __restrict__ tasks,
                                                   const ENT* __restrict__ ents, const int2* __restrict__ tiles) {
  using V = typename ApVec<AT, RL>::V;
  constexpr int ROWS = 32 * RL, HALF = NR > 1 ? NR / 2 : 1;
  constexpr bool PACK = sizeof(T) == 4 && NR > 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);  // B chunks [NW][AP_KC][NR], then partial sums [NW][NR][ROWS]
  __shared__ ApEntry<AT, T> s_ent[AP_EMAX];
  __shared__ int s_c0[AP_EMAX + 1];
  const int2 tl = tiles[blockIdx.x];
  const GemmTask<T> task = tasks[tl.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = tl.y * ROWS, row = m0 + lane * RL;
  T* bs = sm + (size_t)warp * AP_KC * NR;
  const int bk = lane & (AP_KC - 1), bj = (lane / AP_KC) * HALF;  // B element(s) this lane stages

  T acc[RL][NR];
#pragma unroll
  for (int i = 0; i < RL; i++)
#pragma unroll
    for (int j = 0; j < NR; j++) acc[i][j] = T(0);

  for (int eb = task.e0; eb < task.e1; eb += AP_EMAX) {
    const int ne = min(AP_EMAX, task.e1 - eb);
    __syncthreads();
    if (warp == 0) {
      int n[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = 2 * lane + u;
        n[u] = 0;
        if (e < ne) {
          ApEntry<AT, T> o;
          ap_load(ents[eb + e], o);
          o.vec = (reinterpret_cast<uintptr_t>(o.A) & (RL * sizeof(AT) - 1)) == 0 && (o.lda & (RL - 1)) == 0;
          s_ent[e] = o;
          n[u] = (max(o.k, 0) + AP_KC - 1) / AP_KC;
        }
      }
      int s = n[0] + n[1];
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += x;
      }
      s_c0[2 * lane + 1] = s - n[1];
      s_c0[2 * lane + 2] = s;
      if (lane == 0) s_c0[0] = 0;
    }
    __syncthreads();
    const int total = s_c0[ne];
    int e = 0;
    V a[AP_KC];
    T b[HALF];
    auto fetch = [&](int c) {
      while (c >= s_c0[e + 1]) e++;
      const ApEntry<AT, T>& en = s_ent[e];
      const int k0 = (c - s_c0[e]) * AP_KC, kn = en.k - k0;
      const AT* p = en.A + row + (i64)k0 * en.lda;
      const i64 lda = en.lda;
      if (en.vec && row + RL <= task.m) {
#pragma unroll
        for (int u = 0; u < AP_KC; u++) a[u] = u < kn ? *reinterpret_cast<const V*>(p + u * lda) : ap_zero<V>();
      } else {
#pragma unroll
        for (int u = 0; u < AP_KC; u++) {
          AT x[RL];
#pragma unroll
          for (int i = 0; i < RL; i++) x[i] = (u < kn && row + i < task.m) ? p[u * lda + i] : ap_zero<AT>();
          if constexpr (RL == 1) a[u] = x[0];
          else { a[u].x = x[0]; a[u].y = x[1]; }
        }
      }
      const T* q = en.B + k0 + bk;
#pragma unroll
      for (int j = 0; j < HALF; j++) {
        const int col = bj + j;
        b[j] = (bk < kn && col < task.n) ? en.alpha * q[(i64)col * en.ldb] : T(0);
      }
    };
    if (warp < total) fetch(warp);
    for (int c = warp; c < total; c += NW) {
      V x[AP_KC];
#pragma unroll
      for (int u = 0; u < AP_KC; u++) x[u] = a[u];
      __syncwarp();
      if (NR > 1 || lane < AP_KC)
#pragma unroll
        for (int j = 0; j < HALF; j++) bs[bk * NR + bj + j] = b[j];
      __syncwarp();
      if (c + NW < total) fetch(c + NW);
#pragma unroll
      for (int u = 0; u < AP_KC; u++) {
        T r[RL];
        if constexpr (RL == 1) r[0] = ap_up(x[u]);
        else { r[0] = ap_up(x[u].x); r[1] = ap_up(x[u].y); }
        if constexpr (PACK) {
#pragma unroll
          for (int i = 0; i < RL; i++) {
            unsigned long long aa;
            asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(r[i]));
#pragma unroll
            for (int j = 0; j < NR; j += 2) {
              const unsigned long long bb = *reinterpret_cast<const unsigned long long*>(bs + u * NR + j);
              unsigned long long cc;
              asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(acc[i][j]), "f"(acc[i][j + 1]));
              asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
              asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][j]), "=f"(acc[i][j + 1]) : "l"(cc));
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < NR; j++) {
            const T bv = bs[u * NR + j];
#pragma unroll
            for (int i = 0; i < RL; i++) acc[i][j] += r[i] * bv;
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NR; j++)
#pragma unroll
    for (int i = 0; i < RL; i++) sm[(size_t)(warp * NR + j) * ROWS + lane * RL + i] = acc[i][j];
  __syncthreads();
  for (int o = tid; o < NR * ROWS; o += NW * 32) {
    const int j = o / ROWS, r = m0 + o % ROWS;
    if (r >= task.m || j >= task.n) continue;
    T s = sm[o];
#pragma unroll
    for (int w = 1; w < NW; w++) s += sm[(size_t)w * NR * ROWS + o];
    T* p = task.C + r + (i64)j * task.ldc;
    *p = task.beta == T(0) ? s : task.beta * *p + s;
  }
}

template <typename AT, typename T, typename ENT, int NR, int RL, int NW>
static cudaError_t apply_go(const GemmTask<T>* tasks, const ENT* ents, const int2* tiles, int ntiles,
                            cudaStream_t st) {
  constexpr size_t smem = sizeof(T) * (size_t)NW * NR * (32 * RL > AP_KC ? 32 * RL : AP_KC);
  auto kern = k_apply<AT, T, ENT, NR, RL, NW>;
  if (smem > 40 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  note_launch();
  kern<<<ntiles, NW * 32, smem, st>>>(tasks, ents, tiles);
  return cudaGetLastError();
}

int apply_rows_per_cta(int rl) { return 32 * rl; }
// Rows per lane up to which k_apply is built.  FP64 with at most 8 columns has
// one: two rows of a chunk in use and two on their way fill the 128 registers of
// a thread at two CTAs per SM and spilled (substitution of 65,536 bodies, FP64: 4
// columns 1,302 us with two rows, 981 with one; 8 columns of 32,768: 845, 740).
// With 16 two rows are the faster form (32,768: 856, 899), as in FP32 (65,536, 1
// column: 650, 785).
int apply_max_rl(size_t elem, int nr) { return elem == 8 && nr <= 8 ? 1 : 2; }

template <typename AT, typename T, typename ENT>
static cudaError_t apply_any(int nr, int rl, const GemmTask<T>* tasks, const ENT* ents, const int2* tiles, int ntiles,
                             cudaStream_t st) {
  if (ntiles == 0) return cudaSuccess;
#define H2B_APPLY(N)                                                                             \
  if (nr <= N) {                                                                                 \
    if constexpr (sizeof(T) == 4 || N > 8) {                                                     \
      if (rl == 2) return apply_go<AT, T, ENT, N, 2, 8>(tasks, ents, tiles, ntiles, st);         \
    }                                                                                            \
    if constexpr (sizeof(AT) >= 4) {                                                             \
      if (rl == 1) return apply_go<AT, T, ENT, N, 1, 8>(tasks, ents, tiles, ntiles, st);         \
    }                                                                                            \
  }
  H2B_APPLY(1)
  H2B_APPLY(2)
  H2B_APPLY(4)
  H2B_APPLY(8)
  H2B_APPLY(16)
#undef H2B_APPLY
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_apply(int nr, int rl, const GemmTask<T>* tasks, const GemmEntry<T>* ents, const int2* tiles,
                         int ntiles, cudaStream_t st) {
  return apply_any<T, T, GemmEntry<T>>(nr, rl, tasks, ents, tiles, ntiles, st);
}
template cudaError_t launch_apply<double>(int, int, const GemmTask<double>*, const GemmEntry<double>*, const int2*,
                                          int, cudaStream_t);
template cudaError_t launch_apply<float>(int, int, const GemmTask<float>*, const GemmEntry<float>*, const int2*, int,
                                         cudaStream_t);
cudaError_t launch_apply_bf16(int nr, const GemmTask<float>* tasks, const BfEntry* ents, const int2* tiles, int ntiles,
                              cudaStream_t st) {
  return apply_any<__nv_bfloat16, float, BfEntry>(nr, 2, tasks, ents, tiles, ntiles, st);
}

}  // namespace h2b
