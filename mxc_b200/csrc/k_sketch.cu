// Full-far-field random-sign sketch for the interpolative bases
// (compute_basis, h2matrix.cpp:13-63; build extension, sampling mode 2).
//
// The reference factors the whole far block XF = K(far bodies, box bodies)
// (S x M, S up to the number of bodies) with a Householder QR and runs the
// column-pivoted QR on its R.  Capping S by strided samples keeps the cost
// down but loses accuracy on the unsampled far bodies: the nearest far boxes
// carry most of the numerical rank and a stride of 1 in 16 misses it (at
// 262,144 points, 16,000 samples leave 2e-9 relative ID error where the
// whole far field gives 3e-12).  Here every far body is used, through the
// M x M product Y = Omega XF with a random-sign Omega: Y has the column
// geometry of XF up to the sketch's distortion, so the pivoted QR of Y picks
// skeletons and interpolation coefficients of nearly whole-far-field
// accuracy (randomized ID, Halko, Martinsson and Tropp 2011), and the cost is
// one GEMM of 2 M^2 S flops per box on the FP64 tensor cores with XF never
// stored: each 16-body slab of XF is generated into shared memory next to
// the 16 x 128 slab of signs it meets.
//
// Omega(a, f) = -1 when bit (a mod 64) of mix64(body_f * MUL_F + (a div 64) *
// MUL_W + ADD) is set, else +1 (splitmix64 finaliser); body_f is the body's
// index in the tree-sorted array, so the matrix does not depend on the order
// in which a box's far list is walked.  Boxes whose far list has at most M
// bodies take XF itself (compute_basis's K == N branch).
#include "common.cuh"
#include "kernels.h"

#include <cmath>
#include <cstdint>
#include <type_traits>

namespace h2b {

namespace {

constexpr int SK_TN = 64, SK_KS = 16, SK_CS = SK_KS + 4, SK_MAXW = 10, SK_WORDS = SK_MAXW / 2 + 1;

__device__ __forceinline__ unsigned long long sk_mix64(unsigned long long z) {
  z ^= z >> 30;
  z *= 0xBF58476D1CE4E5B9ull;
  z ^= z >> 27;
  z *= 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ unsigned long long sk_word(i64 body, int w) {
  return sk_mix64((unsigned long long)body * 0x9E3779B97F4A7C15ull + (unsigned long long)w * 0xD1B54A32D192ED03ull +
                  0x2545F4914F6CDD1Dull);
}

__device__ __forceinline__ void sk_dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Barrier of the whole block that its warps reach at different places, each
// warp as one (__syncthreads() would have to be the same one for all threads).
__device__ __forceinline__ void sk_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }

// Body index of entry f (0 <= f < S) of a box's far list: ranges r0..r1-1
// hold [rstart[r], rstart[r] + count) with rend[r] the running count; the
// walk starts at a range known to begin at or before f.
__device__ __forceinline__ i64 sk_body(i64 f, i64 from, i64 r0, const i64* __restrict__ rstart,
                                       const i64* __restrict__ rend) {
  i64 r = from;
  while (f >= rend[r]) r++;
  return rstart[r] + (f - (r == r0 ? 0 : rend[r - 1]));
}

}  // namespace

// One CTA per {box, row tile, 64-column tile, part of the far list} of Y: 32 WM
// rows, 2 WM warps of 32 x 32 (4 x 4 m8n8k4 fragments each; 64 x 32, with half
// the warps, was 8% slower) and one that
// prepares the slabs.  Per 16-body slab the warps evaluate the 16 x 64 entries
// of XF into a [column][20] shared tile laid out like the fragment loads and
// multiply; one barrier per slab.  The last warp runs ahead -- the body indices
// three slabs, the coordinates' loads two, coordinates and sign words in shared
// memory one -- so no warp that multiplies waits for a load.
//
// Bound: the FP64 tensor pipe, 2 M^2 S flops per box, plus one evaluation (about
// 25 FP64 instructions) per 32 WM multiply-adds.  Hence one row tile up to 320
// rows, evenly cut beyond (tiles of 128 computed 384 rows for 312 and evaluated
// XF three times), and the far list cut into parts where the tiles fill the
// chip's last wave badly (k_sketch_sum adds them).  20,000 bodies, five levels: 20.5 -> 14.4 ms (19.5 TFLOP/s of
// the 36.8 of the pipe; leaves of 312 bodies 12.9 -> 9.2) against 128-row tiles
// in one piece, the slab's far bodies fetched by a multiplying warp.
// CTAs per SM.  They leave a thread 80 registers with 3 or 10 row groups, 96 with
// 4, 8 or 9 and up to 128 otherwise; with the 64 of the accumulators that is
// tight: Laplace spills 220 bytes at 80, 16 to 60 at 96 and none beyond (every
// kind: 336, up to 76, none).
__host__ __device__ constexpr int sketch_ctas(int wm) { return wm <= 3 ? 3 : wm <= 4 ? 2 : 1; }

// KIND: the kernel kind where it is known at compile time (Laplace: without the
// other kinds' sincos and exp a third less is spilled), -1 to read kp_in.
template <int WM, int KIND>
__global__ void __launch_bounds__(64 * WM + 32, sketch_ctas(WM))
    k_sketch(KernelParams kp_in, const double* __restrict__ bodies, const double* __restrict__ pts,
             const i64* __restrict__ xoff, const i64* __restrict__ dims, const i64* __restrict__ qoff,
             const i64* __restrict__ roff, const i64* __restrict__ rstart, const i64* __restrict__ rend,
             const int4* __restrict__ tiles, int parts, i64 pstride, double* __restrict__ Y, float* __restrict__ F) {
  constexpr int TM = 32 * WM, NMMA = 64 * WM;  // threads that multiply
  __shared__ __align__(16) double xf[2][SK_TN * SK_CS];
  __shared__ double fc[2][SK_KS * 3];
  __shared__ int fv[2][SK_KS];
  __shared__ unsigned long long sw[3][SK_KS][SK_WORDS];
  __shared__ double xs[SK_TN * 3];

  KernelParams kp = kp_in;
  if (KIND >= 0) kp.kind = KIND;
  const int4 tl = tiles[blockIdx.x];
  const int box = tl.x;
  const int M = (int)dims[box];
  const int a0 = tl.y * TM, c0 = tl.z * SK_TN;
  const i64 r0 = roff[box], r1 = roff[box + 1];
  const i64 S = r1 > r0 ? rend[r1 - 1] : 0;
  double* W = Y + (i64)tl.w * pstride + qoff[box];  // F (FP32 bases in one piece): stored there instead
  const double* X = pts + 3 * xoff[box];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (M == 0 || S == 0) return;

  if (S <= (i64)M) {
    // Whole far block: rows a < S of W are K(F_a, X_c).
    if (tl.w) return;
    for (int e = tid; e < TM * SK_TN; e += blockDim.x) {
      const int a = a0 + e / SK_TN, c = c0 + e % SK_TN;
      if ((i64)a >= S || c >= M) continue;
      const i64 body = sk_body(a, r0, r0, rstart, rend);
      const double v = kernel_fast_pair(kp, bodies[3 * body], bodies[3 * body + 1], bodies[3 * body + 2], X[3 * c],
                                        X[3 * c + 1], X[3 * c + 2]);
      if (F)
        F[qoff[box] + (i64)a * M + c] = (float)v;
      else
        W[(i64)a * M + c] = v;
    }
    return;
  }

  const int nslab_all = (int)((S + SK_KS - 1) / SK_KS);
  const int s0 = (int)((i64)nslab_all * tl.w / parts), s1 = (int)((i64)nslab_all * (tl.w + 1) / parts);
  for (int e = tid; e < SK_TN * 3; e += blockDim.x) xs[e] = c0 + e / 3 < M ? X[3 * c0 + e] : 0.;

  if (warp == 2 * WM) {
    // The preparing warp: lane f (and f + 16) follows body f of a slab.
    const int f = lane & (SK_KS - 1);
    i64 cur = r0, body1 = -1, body2 = -1;  // bodies of slabs +1 (coordinates loaded) and +2
    double q0 = 0., q1 = 0., q2 = 0.;
    auto body_of = [&](int sl) -> i64 {
      const i64 i = (i64)sl * SK_KS + f;
      if (sl >= s1 || i >= S) return -1;
      while (i >= rend[cur]) cur++;
      return rstart[cur] + (i - (cur == r0 ? 0 : rend[cur - 1]));
    };
    auto load = [&](i64 b) {
      q0 = b >= 0 ? bodies[3 * b] : 0.;
      q1 = b >= 0 ? bodies[3 * b + 1] : 0.;
      q2 = b >= 0 ? bodies[3 * b + 2] : 0.;
    };
    auto publish = [&](int sl, i64 b) {
      if (lane < SK_KS) {
        fv[sl & 1][f] = b >= 0;
        fc[sl & 1][3 * f] = q0;
        fc[sl & 1][3 * f + 1] = q1;
        fc[sl & 1][3 * f + 2] = q2;
      }
      for (int w = lane / SK_KS; w < SK_WORDS; w += 2) sw[sl % 3][f][w] = b >= 0 ? sk_word(b, (a0 >> 6) + w) : 0ull;
    };
    if (s0 < s1) {  // the range that holds the part's first body
      i64 lo = r0, hi = r1 - 1;
      const i64 i0 = (i64)s0 * SK_KS;
      while (lo < hi) {
        const i64 mid = (lo + hi) / 2;
        if (rend[mid] <= i0) lo = mid + 1;
        else hi = mid;
      }
      cur = lo;
    }
    body1 = body_of(s0);
    load(body1);
    publish(s0, body1);
    body1 = body_of(s0 + 1);
    load(body1);
    body2 = body_of(s0 + 2);
    sk_barrier();
    for (int sl = s0; sl < s1; sl++) {
      publish(sl + 1, body1);
      body1 = body2;
      load(body1);
      body2 = body_of(sl + 3);
      sk_barrier();
    }
    return;
  }

  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.;

  sk_barrier();
  const int wm = warp >> 1, wn = warp & 1;
  const int row32 = a0 + 32 * wm;                      // the warp's first row
  const int wsel = (row32 >> 6) - (a0 >> 6);           // its sign word
  const int bit0 = (row32 & 32) + (lane >> 2);         // fragment row's bit in that word
  for (int sl = s0; sl < s1; sl++) {
    const int b = sl & 1;
    for (int e = tid; e < SK_KS * SK_TN; e += NMMA) {
      const int fl = e & (SK_KS - 1), cl = e / SK_KS;
      double v = 0.;
      if (c0 + cl < M && fv[b][fl])
        v = kernel_fast_pair(kp, fc[b][3 * fl], fc[b][3 * fl + 1], fc[b][3 * fl + 2], xs[3 * cl], xs[3 * cl + 1],
                             xs[3 * cl + 2]);
      xf[b][cl * SK_CS + fl] = v;
    }
    sk_barrier();
    const double* bs = xf[b] + (wn * 32 + (lane >> 2)) * SK_CS + (lane & 3);
#pragma unroll
    for (int ks = 0; ks < SK_KS; ks += 4) {
      const unsigned long long word = sw[sl % 3][ks + (lane & 3)][wsel];
      double av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) av[i] = ((word >> (bit0 + 8 * i)) & 1ull) ? -1. : 1.;
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = bs[j * 8 * SK_CS + ks];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) sk_dmma(acc[i][j], av[i], bv[j]);
    }
  }

  // D fragment of m8n8k4: lane holds row lane >> 2, columns 2 (lane & 3) + {0, 1}.
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int a = row32 + i * 8 + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int col = c0 + wn * 32 + j * 8 + 2 * (lane & 3) + h;
        if (a >= M || col >= M) continue;
        if (F)
          F[qoff[box] + (i64)a * M + col] = (float)acc[i][j][h];
        else
          W[(i64)a * M + col] = acc[i][j][h];
      }
  }
}

// Rws = the parts' sum, in order (the first part alone where the box takes its
// far block itself).
template <typename T>
__global__ void __launch_bounds__(256) k_sketch_sum(const i64* __restrict__ dims, const i64* __restrict__ qoff,
                                                    const i64* __restrict__ roff, const i64* __restrict__ rend,
                                                    const double* __restrict__ Y, int parts, i64 pstride,
                                                    T* __restrict__ Rws) {
  const int box = blockIdx.x;
  const i64 M = dims[box], n = M * M, q = qoff[box];
  const i64 S = roff[box + 1] > roff[box] ? rend[roff[box + 1] - 1] : 0;
  if (S == 0) return;
  const int np = S <= M ? 1 : parts;
  for (i64 e = (i64)blockIdx.y * blockDim.x + threadIdx.x; e < n; e += (i64)gridDim.y * blockDim.x) {
    if (S <= M && e >= S * M) return;
    double s = Y[q + e];
    for (int p = 1; p < np; p++) s += Y[p * pstride + q + e];
    Rws[q + e] = (T)s;
  }
}

// Tile rows for boxes of up to M: as few tiles as SK_MAXW row groups allow, evenly.
int sketch_tile_rows(int M) {
  const int t = (M + 32 * SK_MAXW - 1) / (32 * SK_MAXW);
  return ((M + t - 1) / t + 31) / 32 * 32;
}
int sketch_tile_cols() { return SK_TN; }
// Parts of the far list for `tiles` tiles: the fewest that fill the last wave to
// nine tenths (at most 8, of at least 16 slabs; one from 8 waves on).
int sketch_parts(i64 tiles, int tile_rows, i64 bodies) {
  const double slots = 148. * sketch_ctas(tile_rows / 32);
  int best = 1;
  double bw = 0.;
  for (int p = 1; p <= 8 && (p == 1 || bodies / SK_KS / p >= 16); p++) {
    const double u = tiles * p / slots, use = u / std::ceil(u);
    if (use > bw + 0.02) { bw = use; best = p; }
    if (use >= 0.9 || tiles >= 8 * slots) break;
  }
  return best;
}

template <typename T>
cudaError_t launch_sketch(const KernelParams& kp, const double* bodies, const double* pts, const i64* xoff,
                          const i64* dims, const i64* qoff, const i64* roff, const i64* rstart, const i64* rend,
                          const int4* d_tiles, int ntiles, int tile_rows, int parts, i64 pstride, double* Y, T* Rws,
                          int nboxes, cudaStream_t st) {
  if (ntiles == 0) return cudaSuccess;
  float* f32 = nullptr;
  if constexpr (std::is_same<T, float>::value) f32 = parts == 1 ? Rws : nullptr;
  auto go = [&](auto kern, int wm) {
    note_launch();
    kern<<<ntiles, 64 * wm + 32, 0, st>>>(kp, bodies, pts, xoff, dims, qoff, roff, rstart, rend, d_tiles, parts,
                                          pstride, Y, f32);
    return cudaGetLastError();
  };
  cudaError_t e = cudaErrorInvalidValue;
  switch (tile_rows / 32) {
#define H2B_SK(W) \
  case W: e = kp.kind == KERNEL_LAPLACE ? go(k_sketch<W, KERNEL_LAPLACE>, W) : go(k_sketch<W, -1>, W); break;
    H2B_SK(1) H2B_SK(2) H2B_SK(3) H2B_SK(4) H2B_SK(5) H2B_SK(6) H2B_SK(7) H2B_SK(8) H2B_SK(9) H2B_SK(10)
#undef H2B_SK
  }
  if (e != cudaSuccess || parts == 1) return e;
  note_launch();
  k_sketch_sum<T><<<dim3(nboxes, 16), 256, 0, st>>>(dims, qoff, roff, rend, Y, parts, pstride, Rws);
  return cudaGetLastError();
}

template cudaError_t launch_sketch<double>(const KernelParams&, const double*, const double*, const i64*, const i64*,
                                           const i64*, const i64*, const i64*, const i64*, const int4*, int, int, int,
                                           i64, double*, double*, int, cudaStream_t);
template cudaError_t launch_sketch<float>(const KernelParams&, const double*, const double*, const i64*, const i64*,
                                          const i64*, const i64*, const i64*, const i64*, const int4*, int, int, int,
                                          i64, double*, float*, int, cudaStream_t);

}  // namespace h2b
