// Batched complex128 matrix inverse: blocked Gauss-Jordan with partial
// pivoting, a CTA or a small cluster per matrix.
//
// Replaces the batched inverse of qttools kernels/linalg/inv.py:6-40
// (numpy.linalg.inv on CPU; cupy.linalg.solve(a, I) -> cuBLAS batched
// getrf/getrs on NVIDIA GPUs). Every diagonal Schur-complement block of the
// RGF forward sweep and every Sancho-Rubio step inverts through here, or through
// the kernels of zinv_cluster.cu (n <= 256, few matrices) and zinv_wide.cu
// (n > 512, few matrices), to which zinv_ex dispatches.
//
// Three kernels by block size, one scheme (in place in X, panels K of NB columns):
//   1. factor X[:, K] column by column: pivot = argmax_{r >= k} |Re|+|Im| (the
//      izamax measure of LAPACK), eliminate every other row. Afterwards the
//      panel holds T, the Gauss-Jordan transform of this panel:
//      T = [A_KK^-1 ; -A_RK A_KK^-1] in block form;
//   2. with the panel's row interchanges, update all other columns J:
//        X[:, J] = [0 ; X[R, J]] + T X[K, J]
//      a complex GEMM on the FP64 tensor pipe (DMMA).
// Finally the columns are permuted back. n^3 complex multiply-adds = 8 n^3 flops.
//   n <= 512:  zinv3_kernel, panel in registers, interchanges folded into the
//              update, columns split over up to 8 CTAs, or (n <= 103) the matrix
//              resident in shared memory;
//   n <= 720:  zinv2_kernel, panel and pivot rows in shared memory;
//   n <= 1024: zinv_kernel, one 32-column tile of the pivot rows at a time.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "gj_panel.cuh"

namespace cg = cooperative_groups;

namespace qtx {
namespace {

// 720 < n <= 1024, one CTA per matrix: the row interchanges of a panel are staged
// with each 32-column tile of the update.
constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;
constexpr int JW = 32;  // column-tile width of the trailing update

__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// 1 / (a + ib) by Smith's algorithm (avoids overflow of a^2 + b^2).
__device__ __forceinline__ z64 zrecip(z64 z) {
  if (fabs(z.x) >= fabs(z.y)) {
    if (z.x == 0.0 && z.y == 0.0) return make_double2(0.0, 0.0);
    const double r = z.y / z.x;
    const double den = z.x + z.y * r;
    return make_double2(1.0 / den, -r / den);
  }
  const double r = z.x / z.y;
  const double den = z.x * r + z.y;
  return make_double2(r / den, -1.0 / den);
}

__device__ __forceinline__ double cabs1(z64 z) { return fabs(z.x) + fabs(z.y); }

template <int NB>
struct Smem {
  static constexpr int PS = NB + 4;  // panel row stride (= 4 mod 8 in 16 B units)
  static constexpr int YS = JW + 2;  // Y row stride (= 2 mod 8)
  static constexpr int NA = 2 * NB;  // rows a panel's pivoting can touch
  static size_t bytes(int n) {
    size_t s = (size_t)n * PS * sizeof(z64);  // panel
    s += (size_t)NB * YS * sizeof(z64);       // Y tile
    s += (size_t)NA * JW * sizeof(z64);       // staged old values of the affected rows
    s += (size_t)2 * NB * sizeof(z64);        // scaled pivot row, old row k
    s += (size_t)WARPS * (sizeof(double) + sizeof(int));
    s += (size_t)3 * NA * sizeof(int);  // affected rows, their sources, source slots
    s += (size_t)3 * n * sizeof(int);   // pivot rows, column sources, row -> slot map
    return s + 64;
  }
};

template <int NB>
__global__ void __launch_bounds__(THREADS, 1) zinv_kernel(int n, int64_t batch, MatRef A, MatRef X,
                                                        int* info, const int* active) {
  using S = Smem<NB>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  z64* P = reinterpret_cast<z64*>(smem_raw);
  z64* Y = P + (size_t)n * S::PS;
  z64* stage = Y + NB * S::YS;
  z64* prow = stage + S::NA * JW;
  z64* rowk = prow + NB;
  double* red_v = reinterpret_cast<double*>(rowk + NB);
  int* red_i = reinterpret_cast<int*>(red_v + WARPS);
  int* aff_row = red_i + WARPS;      // affected row indices
  int* aff_src = aff_row + S::NA;    // row whose old value each affected row receives
  int* aff_sslot = aff_src + S::NA;  // slot of that source row in the stage
  int* pivrow = aff_sslot + S::NA;
  int* colsrc = pivrow + n;
  int* slot_of = colsrc + n;  // row -> stage slot, -1 if the row is not affected

  for (int r = threadIdx.x; r < n; r += THREADS) slot_of[r] = -1;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int g = lane >> 2;
  const int tq = lane & 3;

  for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
    if (active != nullptr && active[b] == 0) continue;
    const z64* a = at<const z64>(A, b);
    z64* x = at<z64>(X, b);
    const int64_t lda = A.ld, ldx = X.ld;
    if (a != x) {
      for (int64_t idx = tid; idx < (int64_t)n * n; idx += THREADS) {
        const int r = (int)(idx / n), c = (int)(idx % n);
        x[(int64_t)r * ldx + c] = a[(int64_t)r * lda + c];
      }
    }
    int singular_at = 0;
    __syncthreads();

    for (int k0 = 0; k0 < n; k0 += NB) {
      const int nbp = min(NB, n - k0);
      // 1. Stage the panel (zero-padded to NB columns).
      for (int idx = tid; idx < n * NB; idx += THREADS) {
        const int r = idx / NB, c = idx % NB;
        P[r * S::PS + c] = (c < nbp) ? x[(int64_t)r * ldx + k0 + c] : make_double2(0.0, 0.0);
      }
      __syncthreads();

      // 2. Factor the panel.
      for (int kk = 0; kk < nbp; ++kk) {
        const int k = k0 + kk;
        double best = -1.0;
        int besti = k;
        for (int r = k + tid; r < n; r += THREADS) {
          const double v = cabs1(P[r * S::PS + kk]);
          if (v > best) {
            best = v;
            besti = r;
          }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const double ov = __shfl_xor_sync(0xffffffffu, best, off);
          const int oi = __shfl_xor_sync(0xffffffffu, besti, off);
          if (ov > best || (ov == best && oi < besti)) {
            best = ov;
            besti = oi;
          }
        }
        if (lane == 0) {
          red_v[warp] = best;
          red_i[warp] = besti;
        }
        __syncthreads();
        best = red_v[0];
        besti = red_i[0];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) {
          const double ov = red_v[w];
          const int oi = red_i[w];
          if (ov > best || (ov == best && oi < besti)) {
            best = ov;
            besti = oi;
          }
        }
        const int p = besti;
        if (best == 0.0 && singular_at == 0) singular_at = k + 1;
        // Nobody writes P in this phase, so every thread can read the pivot.
        const z64 dpiv = zrecip(P[p * S::PS + kk]);
        if (tid < NB) {
          const int c = tid;
          rowk[c] = P[k * S::PS + c];
          prow[c] = (c == kk) ? dpiv : zmul(P[p * S::PS + c], dpiv);
        }
        if (tid == 0) pivrow[k] = p;
        __syncthreads();
        // Eliminate; rows k and p are swapped on the fly (row p receives the
        // old row k, row k becomes the scaled pivot row).
        for (int r = tid; r < n; r += THREADS) {
          if (r == k) {
            for (int c = 0; c < NB; ++c) P[r * S::PS + c] = prow[c];
            continue;
          }
          const z64* src = (r == p) ? rowk : P + r * S::PS;
          const z64 f = src[kk];
          for (int c = 0; c < NB; ++c) {
            if (c == kk) continue;
            const z64 v = src[c];
            P[r * S::PS + c] = make_double2(v.x - (f.x * prow[c].x - f.y * prow[c].y),
                                            v.y - (f.x * prow[c].y + f.y * prow[c].x));
          }
          const z64 m = zmul(f, dpiv);
          P[r * S::PS + kk] = make_double2(-m.x, -m.y);
        }
        __syncthreads();
      }

      // 3. The panel's row interchanges as a permutation of the (at most
      //    2 NB) rows they touch: affected row aff_row[a] receives the old
      //    content of row aff_src[a], staged in slot aff_sslot[a].
      __shared__ int s_na;
      if (tid == 0) {
        int na = 0;
        for (int kk = 0; kk < nbp; ++kk) {
          const int k = k0 + kk, p = pivrow[k];
          int ik = slot_of[k], ip = slot_of[p];
          if (ik < 0) {
            ik = na++;
            aff_row[ik] = k;
            aff_src[ik] = k;
            slot_of[k] = ik;
          }
          if (ip < 0) {
            ip = na++;
            aff_row[ip] = p;
            aff_src[ip] = p;
            slot_of[p] = ip;
          }
          const int t = aff_src[ik];
          aff_src[ik] = aff_src[ip];
          aff_src[ip] = t;
        }
        for (int a = 0; a < na; ++a) aff_sslot[a] = slot_of[aff_src[a]];
        s_na = na;
      }
      __syncthreads();
      const int na = s_na;

      // 4. Trailing update of every other column tile:
      //      X[:, J] <- [0 ; X[R, J]] + T[:, K] X[K, J]   (rows permuted).
      for (int j0 = 0; j0 < n; j0 += JW) {
        // Columns of the panel itself are computed but never stored.
        if (j0 >= k0 && j0 + JW <= k0 + nbp) continue;
        for (int idx = tid; idx < na * JW; idx += THREADS) {
          const int a = idx / JW, c = idx % JW;
          const int gc = j0 + c;
          stage[a * JW + c] = (gc < n && (gc < k0 || gc >= k0 + nbp))
                                  ? x[(int64_t)aff_row[a] * ldx + gc]
                                  : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int idx = tid; idx < NB * JW; idx += THREADS) {
          const int kk = idx / JW, c = idx % JW;
          Y[kk * S::YS + c] =
              (kk < nbp) ? stage[aff_sslot[slot_of[k0 + kk]] * JW + c] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        const int mtiles = (n + 15) / 16;
        for (int base = warp; base < mtiles; base += 2 * WARPS) {
          double cre[2][JW / 8][4], cim[2][JW / 8][4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r0 = (base + h * WARPS) * 16;
#pragma unroll
            for (int j = 0; j < JW / 8; ++j)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int r = r0 + g + ((q >> 1) << 3);
                const int cl = j * 8 + 2 * tq + (q & 1);
                const int c = j0 + cl;
                z64 v = make_double2(0.0, 0.0);
                if (r < n && c < n && !(r >= k0 && r < k0 + nbp) && (c < k0 || c >= k0 + nbp)) {
                  const int sl = slot_of[r];
                  v = (sl >= 0) ? stage[aff_sslot[sl] * JW + cl] : x[(int64_t)r * ldx + c];
                }
                cre[h][j][q] = v.x;
                cim[h][j][q] = v.y;
              }
          }
#pragma unroll
          for (int k4 = 0; k4 < NB; k4 += 4) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int ra = (base + h * WARPS) * 16 + g;
              const z64 v0 = (ra < n) ? P[ra * S::PS + k4 + tq] : make_double2(0, 0);
              const z64 v1 = (ra + 8 < n) ? P[(ra + 8) * S::PS + k4 + tq] : make_double2(0, 0);
              const double nai0 = -v0.y, nai1 = -v1.y;
#pragma unroll
              for (int j = 0; j < JW / 8; ++j) {
                const z64 bv = Y[(k4 + tq) * S::YS + j * 8 + g];
                mma_f64(cre[h][j], v0.x, v1.x, bv.x);
                mma_f64(cim[h][j], v0.x, v1.x, bv.y);
              }
#pragma unroll
              for (int j = 0; j < JW / 8; ++j) {
                const z64 bv = Y[(k4 + tq) * S::YS + j * 8 + g];
                mma_f64(cre[h][j], nai0, nai1, bv.y);
                mma_f64(cim[h][j], v0.y, v1.y, bv.x);
              }
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r0 = (base + h * WARPS) * 16;
#pragma unroll
            for (int j = 0; j < JW / 8; ++j)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int r = r0 + g + ((q >> 1) << 3);
                const int c = j0 + j * 8 + 2 * tq + (q & 1);
                if (r < n && c < n && (c < k0 || c >= k0 + nbp))
                  x[(int64_t)r * ldx + c] = make_double2(cre[h][j][q], cim[h][j][q]);
              }
          }
        }
        __syncthreads();
      }
      if (tid == 0)
        for (int a = 0; a < na; ++a) slot_of[aff_row[a]] = -1;

      // 5. Write the panel back.
      for (int idx = tid; idx < n * nbp; idx += THREADS) {
        const int r = idx / nbp, c = idx % nbp;
        x[(int64_t)r * ldx + k0 + c] = P[r * S::PS + c];
      }
      __syncthreads();
    }

    // Undo the column permutation: swaps applied from the last pivot back.
    if (tid == 0) {
      for (int c = 0; c < n; ++c) colsrc[c] = c;
      for (int k = n - 1; k >= 0; --k) {
        const int p = pivrow[k];
        if (p != k) {
          const int t = colsrc[k];
          colsrc[k] = colsrc[p];
          colsrc[p] = t;
        }
      }
    }
    __syncthreads();
    // Row-wise gather through the (now free) panel buffer, one warp per row.
    z64* rowbuf = P + (size_t)warp * n;
    for (int r = warp; r < n; r += WARPS) {
      for (int c = lane; c < n; c += 32) rowbuf[c] = x[(int64_t)r * ldx + colsrc[c]];
      __syncwarp();
      for (int c = lane; c < n; c += 32) x[(int64_t)r * ldx + c] = rowbuf[c];
      __syncwarp();
    }
    // Report the first singular block seen for this stack entry (callers
    // zero `info` once per entry point).
    if (tid == 0 && info != nullptr && singular_at != 0 && info[b] == 0) info[b] = singular_at;
    __syncthreads();
  }
}

template <int NB>
int launch(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  const size_t smem = Smem<NB>::bytes(n);
  if (smem > kMaxDynamicSmem) {
    set_error("zinv: block size too large for the shared-memory panel");
    return QTX_ERR_UNSUPPORTED;
  }
  QTX_TRY(allow_dynamic_smem(zinv_kernel<NB>));
  const unsigned grid = (unsigned)(batch < 1048576 ? batch : 1048576);
  ProfScope prof(QTX_KERNEL_ZINV, 8.0 * (double)n * n * n * (double)batch, s);
  zinv_kernel<NB><<<grid, THREADS, smem, s>>>(n, batch, A, X, info, active);
  QTX_CHECK_LAUNCH();
  return QTX_OK;
}

// ---------------------------------------------------------------------------
// One CTA per matrix for 512 < n <= 720: the same Gauss-Jordan with the same
// pivot rule, reorganised so that the trailing update runs without barriers.
// Per panel of NB columns:
//   1. stage the n x NB panel (odd row stride: row-per-thread access is
//      conflict-free) and factor it (one barrier pair per column, the next
//      column's pivot candidate found during the elimination);
//   2. apply the panel's row interchanges to the other columns in global
//      memory: the <= 2 NB affected rows are read into registers, then
//      written to their new places;
//   3. stage the pivot rows Y = X[K, :] (other columns) once;
//   4. every warp updates its 16-row slices over all column tiles:
//      X[r, J] = (r in K ? 0 : X[r, J]) + T[r, :] Y[:, J]  (DMMA), with no
//      barrier, so 16 warps overlap their loads and MMAs;
//   5. write the panel transform T back into X[:, K].
constexpr int T2 = 512;
constexpr int W2 = T2 / 32;
constexpr int JN = 2;    // n8 tiles per column tile of the trailing update
constexpr int PV = 8;  // elements per thread of one row-interchange block

template <int NB>
struct Smem2 {
  static constexpr int PS = NB + 1;
  // Y row stride: covers whole 16-column tiles, 2 mod 8 in 16-byte units.
  __host__ __device__ static int ys(int n) { return ((n + 15) / 16) * 16 + 2; }
  static size_t bytes(int n) {
    size_t s = (size_t)n * PS * sizeof(z64);          // panel
    s += (size_t)NB * ys(n) * sizeof(z64);            // pivot rows Y
    s += (size_t)2 * NB * sizeof(z64);                // scaled pivot row, old row k
    s += (size_t)2 * W2 * (sizeof(double) + sizeof(int));
    s += (size_t)2 * (2 * NB) * sizeof(int);          // affected rows and their sources
    s += (size_t)2 * n * sizeof(int) + 16;            // pivot rows, column sources
    return s + 64;
  }
};

template <int NB>
__global__ void __launch_bounds__(T2, 1) zinv2_kernel(int n, int64_t batch, MatRef A, MatRef X, int* info,
                                                      const int* active) {
  using S = Smem2<NB>;
  // Column block of the row-interchange pass: all 2 NB affected rows of CW
  // columns fit T2 x PV registers.
  constexpr int CW = (T2 * PV) / (2 * NB);
  static_assert(NB % 4 == 0 && 2 * NB * CW <= T2 * PV, "panel width and interchange block");
  constexpr int PS = S::PS;
  const int YS = S::ys(n);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  z64* P = reinterpret_cast<z64*>(smem_raw);
  z64* Y = P + (size_t)n * PS;
  z64* prow = Y + (size_t)NB * YS;
  z64* rowk = prow + NB;
  double* red_v = reinterpret_cast<double*>(rowk + NB);  // 2 x W2
  int* red_i = reinterpret_cast<int*>(red_v + 2 * W2);   // 2 x W2
  int* aff_row = red_i + 2 * W2;                         // 2 NB
  int* aff_src = aff_row + 2 * NB;                       // 2 NB
  int* pivrow = aff_src + 2 * NB;                        // n
  int* colsrc = pivrow + n;                              // n
  __shared__ int s_na, s_sing;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tq = lane & 3;
  for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
    if (active != nullptr && active[b] == 0) continue;
    const z64* a = at<const z64>(A, b);
    z64* x = at<z64>(X, b);
    const int64_t ldx = X.ld;
    if (a != x) {
      for (int64_t idx = tid; idx < (int64_t)n * n; idx += T2) {
        const int r = (int)(idx / n), c = (int)(idx % n);
        x[(int64_t)r * ldx + c] = a[(int64_t)r * A.ld + c];
      }
    }
    if (tid == 0) s_sing = 0;
    __syncthreads();

    for (int k0 = 0; k0 < n; k0 += NB) {
      const int nbp = min(NB, n - k0);
      // 1. Stage the panel and factor it.
      for (int idx = tid; idx < n * NB; idx += T2) {
        const int r = idx / NB, c = idx % NB;
        P[r * PS + c] = (c < nbp) ? x[(int64_t)r * ldx + k0 + c] : make_double2(0.0, 0.0);
      }
      __syncthreads();
      double best = -1.0;
      int besti = k0;
      for (int r = k0 + tid; r < n; r += T2) {
        const double v = cabs1(P[r * PS]);
        if (v > best || (v == best && r < besti)) {
          best = v;
          besti = r;
        }
      }
      for (int kk = 0; kk < nbp; ++kk) {
        const int k = k0 + kk;
        const int buf = kk & 1;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const double ov = __shfl_xor_sync(0xffffffffu, best, off);
          const int oi = __shfl_xor_sync(0xffffffffu, besti, off);
          if (ov > best || (ov == best && oi < besti)) {
            best = ov;
            besti = oi;
          }
        }
        if (lane == 0) {
          red_v[buf * W2 + warp] = best;
          red_i[buf * W2 + warp] = besti;
        }
        __syncthreads();
        best = red_v[buf * W2];
        besti = red_i[buf * W2];
#pragma unroll
        for (int w = 1; w < W2; ++w) {
          const double ov = red_v[buf * W2 + w];
          const int oi = red_i[buf * W2 + w];
          if (ov > best || (ov == best && oi < besti)) {
            best = ov;
            besti = oi;
          }
        }
        const int p = besti;
        if (best <= 0.0 && tid == 0 && s_sing == 0) s_sing = k + 1;
        const z64 dpiv = zrecip(P[p * PS + kk]);
        if (tid < NB) {
          rowk[tid] = P[k * PS + tid];
          prow[tid] = (tid == kk) ? dpiv : zmul(P[p * PS + tid], dpiv);
        }
        if (tid == 0) pivrow[k] = p;
        __syncthreads();
        best = -1.0;
        besti = k + 1;
        for (int r = tid; r < n; r += T2) {
          if (r == k) {
#pragma unroll
            for (int c = 0; c < NB; ++c) P[r * PS + c] = prow[c];
            continue;
          }
          const z64* src = (r == p) ? rowk : P + r * PS;
          const z64 f = src[kk];
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            if (c == kk) continue;
            const z64 v = src[c];
            const z64 q = prow[c];
            P[r * PS + c] = make_double2(v.x - (f.x * q.x - f.y * q.y), v.y - (f.x * q.y + f.y * q.x));
          }
          const z64 m = zmul(f, dpiv);
          P[r * PS + kk] = make_double2(-m.x, -m.y);
          if (kk + 1 < nbp && r > k) {
            const double v = cabs1(P[r * PS + kk + 1]);
            if (v > best || (v == best && r < besti)) {
              best = v;
              besti = r;
            }
          }
        }
      }
      // 2. The panel's interchanges as a permutation of the affected rows:
      //    row aff_row[a] receives the old content of row aff_src[a].
      if (tid == 0) {
        int na = 0;
        for (int kk = 0; kk < nbp; ++kk) {
          const int k = k0 + kk, p = pivrow[k];
          int ik = -1, ip = -1;
          for (int u = 0; u < na; ++u) {
            if (aff_row[u] == k) ik = u;
            if (aff_row[u] == p) ip = u;
          }
          if (ik < 0) {
            ik = na++;
            aff_row[ik] = k;
            aff_src[ik] = k;
          }
          if (ip < 0) {
            ip = na++;
            aff_row[ip] = p;
            aff_src[ip] = p;
          }
          const int t = aff_src[ik];
          aff_src[ik] = aff_src[ip];
          aff_src[ip] = t;
        }
        s_na = na;
      }
      __syncthreads();
      const int na = s_na;
      const int oc = n - nbp;  // columns outside the panel
      // In column blocks of CW: all affected rows of a column move within
      // one block (read all, barrier, write all).
      for (int cb = 0; cb < oc; cb += CW) {
        z64 v[PV];
#pragma unroll
        for (int u = 0; u < PV; ++u) {
          const int li = tid + u * T2;
          const int aa = li / CW, cc = cb + li % CW;
          if (aa < na && cc < oc) {
            const int c = cc + (cc >= k0 ? nbp : 0);
            v[u] = x[(int64_t)aff_src[aa] * ldx + c];
          }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PV; ++u) {
          const int li = tid + u * T2;
          const int aa = li / CW, cc = cb + li % CW;
          if (aa < na && cc < oc) {
            const int c = cc + (cc >= k0 ? nbp : 0);
            x[(int64_t)aff_row[aa] * ldx + c] = v[u];
          }
        }
        __syncthreads();
      }
      // 3. Pivot rows (other columns) into Y.
      const int ny = YS - 2;  // columns of whole tiles; those >= n stay zero
      for (int idx = tid; idx < NB * ny; idx += T2) {
        const int kk = idx / ny, c = idx % ny;
        Y[kk * YS + c] = (kk < nbp && c < n && (c < k0 || c >= k0 + nbp))
                             ? x[(int64_t)(k0 + kk) * ldx + c]
                             : make_double2(0.0, 0.0);
      }
      __syncthreads();
      // 4. Trailing update, one 16-row slice per warp at a time, no barriers.
      const int mtiles = (n + 15) / 16;
      for (int mt = warp; mt < mtiles; mt += W2) {
        const int r0 = mt * 16;
        // A fragments of this slice for all k (the panel transform rows).
        for (int j0 = 0; j0 < n; j0 += 8 * JN) {
          if (j0 >= k0 && j0 + 8 * JN <= k0 + nbp) continue;  // inside the panel
          double cre[JN][4], cim[JN][4];
#pragma unroll
          for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int r = r0 + g + ((q >> 1) << 3);
              const int c = j0 + j * 8 + 2 * tq + (q & 1);
              z64 v = make_double2(0.0, 0.0);
              if (r < n && c < n && !(r >= k0 && r < k0 + nbp) && (c < k0 || c >= k0 + nbp))
                v = x[(int64_t)r * ldx + c];
              cre[j][q] = v.x;
              cim[j][q] = v.y;
            }
#pragma unroll
          for (int k4 = 0; k4 < NB; k4 += 4) {
            const int ra = r0 + g;
            const z64 v0 = (ra < n) ? P[ra * PS + k4 + tq] : make_double2(0.0, 0.0);
            const z64 v1 = (ra + 8 < n) ? P[(ra + 8) * PS + k4 + tq] : make_double2(0.0, 0.0);
            const double nai0 = -v0.y, nai1 = -v1.y;
            double br[JN], bi[JN];
#pragma unroll
            for (int j = 0; j < JN; ++j) {
              const z64 bv = Y[(k4 + tq) * YS + j0 + j * 8 + g];
              br[j] = bv.x;
              bi[j] = bv.y;
            }
#pragma unroll
            for (int j = 0; j < JN; ++j) {
              mma_f64(cre[j], v0.x, v1.x, br[j]);
              mma_f64(cim[j], v0.x, v1.x, bi[j]);
            }
#pragma unroll
            for (int j = 0; j < JN; ++j) {
              mma_f64(cre[j], nai0, nai1, bi[j]);
              mma_f64(cim[j], v0.y, v1.y, br[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int r = r0 + g + ((q >> 1) << 3);
              const int c = j0 + j * 8 + 2 * tq + (q & 1);
              if (r < n && c < n && (c < k0 || c >= k0 + nbp))
                x[(int64_t)r * ldx + c] = make_double2(cre[j][q], cim[j][q]);
            }
        }
      }
      __syncthreads();
      // 5. The panel transform back into X[:, K].
      for (int idx = tid; idx < n * nbp; idx += T2) {
        const int r = idx / nbp, c = idx % nbp;
        x[(int64_t)r * ldx + k0 + c] = P[r * PS + c];
      }
      __syncthreads();
    }

    // Undo the column permutation: swaps applied from the last pivot back.
    if (tid == 0) {
      for (int c = 0; c < n; ++c) colsrc[c] = c;
      for (int k = n - 1; k >= 0; --k) {
        const int p = pivrow[k];
        if (p != k) {
          const int t = colsrc[k];
          colsrc[k] = colsrc[p];
          colsrc[p] = t;
        }
      }
    }
    __syncthreads();
    // Row-wise gather through the (now free) panel buffer: PS rows fit.
    const int nbufs = PS < W2 ? PS : W2;
    if (warp < nbufs) {
      z64* rowbuf = P + (size_t)warp * n;
      for (int r = warp; r < n; r += nbufs) {
        for (int c = lane; c < n; c += 32) rowbuf[c] = x[(int64_t)r * ldx + colsrc[c]];
        __syncwarp();
        for (int c = lane; c < n; c += 32) x[(int64_t)r * ldx + c] = rowbuf[c];
        __syncwarp();
      }
    }
    if (tid == 0 && info != nullptr && s_sing != 0 && info[b] == 0) info[b] = s_sing;
    __syncthreads();
  }
}

template <int NB>
int launch2(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  const size_t smem = Smem2<NB>::bytes(n);
  if (smem > kMaxDynamicSmem) {
    set_error("zinv: block size too large for the shared-memory panel");
    return QTX_ERR_UNSUPPORTED;
  }
  QTX_TRY(allow_dynamic_smem(zinv2_kernel<NB>));
  const unsigned grid = (unsigned)(batch < 131072 ? batch : 131072);
  ProfScope prof(QTX_KERNEL_ZINV, 8.0 * (double)n * n * n * (double)batch, s);
  zinv2_kernel<NB><<<grid, T2, smem, s>>>(n, batch, A, X, info, active);
  QTX_CHECK_LAUNCH();
  return QTX_OK;
}

// ---------------------------------------------------------------------------
// n <= 512: one thread-block cluster of C CTAs per matrix (C = 1 at full
// batches), the CTAs splitting the columns; panels of 16 columns.
// Per panel:
//   1. every CTA factors the panel itself (gj_panel.cuh; the same arithmetic on
//      the same data, so the same transform and pivots) -- no broadcast;
//      rows are not interchanged, the factorization only says where they go;
//   2. the pivot rows Y of this CTA's columns are staged, and, once every CTA of
//      the cluster has loaded the panel (a split cluster barrier), the owner of
//      its columns writes the transform T there;
//   3. all row slices but the pivots' own are updated, X[r, J] <- X[src(r), J]
//      + T[r, :] Y[:, J] (DMMA): src(r) is r, or the row of K that LAPACK's
//      interchanges would have moved to r, so the interchange costs no pass of
//      its own. The tiles of 16 x 16 are dealt to the warps evenly;
//   4. after a barrier (slices read rows of K) the pivots' slice becomes T Y.
// A cluster barrier ends the panel when C > 1 (other CTAs read the next panel
// through L2). Finally the columns are gathered in the order of the pivoting.
//
// RES: the matrix stays in shared memory from load to store (n <= 103, one
// CTA); otherwise each panel is a pass over the matrix in L2 / HBM, which at
// 256 x 256 x 148 moves 5 GB a launch, about half of its time.
struct Smem3 {
  static constexpr int NB = 16;
  __host__ __device__ static int rows(int n) { return (n + 15) & ~15; }
  // Columns of the widest CTA of a C-way split (whole panels).
  __host__ __device__ static int bound(int n, int C, int q) {
    const int v = (int)(((int64_t)n * q / C + NB - 1) / NB) * NB;
    return v < n ? v : n;
  }
  __host__ __device__ static int ys(int n, int C) {  // Y row stride: 2 mod 8 in 16-byte units
    int w = 0;
    for (int q = 0; q < C; ++q) {
      const int c = bound(n, C, q + 1) - bound(n, C, q);
      w = c > w ? c : w;
    }
    return rows(w) + 2;
  }
  __host__ __device__ static int xs(int n) { return n | 1; }  // resident row stride (odd)
  static size_t bytes(int n, int C, bool res) {
    size_t s = (size_t)rows(n) * NB * sizeof(z64) + (size_t)NB * ys(n, C) * sizeof(z64);
    if (res) s += (size_t)n * xs(n) * sizeof(z64);
    return s + (size_t)4 * rows(n) * sizeof(int);
  }
};

// Element (r, c) of the panel transform in shared memory: conflict-free both
// for a thread per row and for the DMMA fragments.
__device__ __forceinline__ int tix(int r, int c) { return r * 16 + (c ^ (((r & 1) << 2) | ((r >> 1) & 3))); }

template <int TH, int RPL, bool RES>
__global__ void __launch_bounds__(TH, 512 / TH) zinv3_kernel(int n, int64_t batch, MatRef A, MatRef X, int* info,
                                                            const int* active, int csplit) {
  using S = Smem3;
  constexpr int NB = S::NB, WARPS3 = TH / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_begin();
  const int np = S::rows(n), YS = S::ys(n, csplit), XS = S::xs(n);
  z64* T = reinterpret_cast<z64*>(smem_raw);
  z64* Y = T + (size_t)np * NB;
  z64* Xs = Y + (size_t)NB * YS;
  int* srcrow = reinterpret_cast<int*>(RES ? Xs + (size_t)n * XS : Xs);
  int* orig = srcrow + np;      // 2 x np: original row of each position
  int* colsrc = orig + 2 * np;  // np
  __shared__ int s_sing;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tq = lane & 3;
  const int rank = (int)(blockIdx.x % csplit);
  const int c_lo = S::bound(n, csplit, rank), c_hi = S::bound(n, csplit, rank + 1), cw = c_hi - c_lo;
  const int mtiles = np / 16, ntiles = (cw + 15) / 16;
  auto cluster_sync = [&]() {
    if (csplit > 1) cg::this_cluster().sync();
  };

  for (int64_t b = blockIdx.x / csplit; b < batch; b += gridDim.x / csplit) {
    if (active != nullptr && active[b] == 0) continue;
    const z64* a = at<const z64>(A, b);
    z64* xg = at<z64>(X, b);
    z64* x = RES ? Xs : xg;
    const int64_t ldx = RES ? XS : X.ld;
    if (RES || a != xg || A.ld != X.ld) {
      for (int idx = tid; idx < n * cw; idx += TH) {
        const int r = idx / cw, c = c_lo + idx % cw;
        x[r * ldx + c] = a[(int64_t)r * A.ld + c];
      }
    }
    for (int r = tid; r < n; r += TH) orig[r] = r;
    if (tid == 0) s_sing = 0;
    __syncthreads();
    cluster_sync();

    int cur = 0;
    for (int k0 = 0; k0 < n; k0 += NB) {
      const int nbp = min(NB, n - k0), kt = k0 / NB;
      // 1. Factor the panel.
      gj_factor_panel<NB, RPL <= 4 ? 2 : 1>(
          n, k0, nbp,
          [=](int r, int c) { return RES ? x[r * ldx + k0 + c] : __ldcg(&x[r * ldx + k0 + c]); },
          [=](int r, int c, z64 v) { T[tix(r, c)] = v; },
          [=](int r, int pos) {
            srcrow[pos] = r;
            orig[(cur ^ 1) * np + pos] = orig[cur * np + r];
          },
          &s_sing);
      cur ^= 1;
      // This CTA's loads of the panel are done. The owner may store the
      // transform over X[:, K] only when that holds for every CTA of the
      // cluster, so all arrive here and wait ahead of that store; the pivot rows
      // are staged meanwhile. (All CTAs factor in step, so the wait
      // is short: 256 x 18 530 -> 536 us, 384 x 37 1.68 -> 1.70 ms, 512 x 21 2.24 -> 2.25.)
      if (!RES && csplit > 1) cg::this_cluster().barrier_arrive();
      __syncthreads();
      // 2. Pivot rows of this CTA's other columns; the transform into X[:, K].
      const bool pin = k0 >= c_lo && k0 < c_hi;
      for (int kk = warp; kk < NB; kk += WARPS3) {
        const z64* xr = kk < nbp ? x + srcrow[k0 + kk] * ldx + c_lo : nullptr;
        const int p0 = k0 - c_lo, p1 = p0 + nbp;  // the panel's columns: not used
#pragma unroll 4
        for (int j = lane; j < YS - 2; j += 32)
          Y[kk * YS + j] = (xr != nullptr && j < cw && (j < p0 || j >= p1)) ? xr[j] : make_double2(0.0, 0.0);
      }
      if (!RES && csplit > 1) cg::this_cluster().barrier_wait();
      {
        const int c = tid % NB;
        if (c >= nbp) {  // columns of T that the factorization left unwritten
          for (int r = tid / NB; r < n; r += TH / NB) T[tix(r, c)] = make_double2(0.0, 0.0);
        } else if (pin) {
#pragma unroll 4
          for (int r = tid / NB; r < n; r += TH / NB) x[r * ldx + k0 + c] = T[tix(r, c)];
        }
      }
      __syncthreads();
      // 3./4. Tiles of 16 x 16 outside the panel's columns, dealt evenly in
      // row-slice order. A tile's elements are loaded (the accumulators) while
      // the one before is multiplied.
      const int pt = pin ? (k0 - c_lo) / 16 : ntiles, nt = ntiles - (pin ? 1 : 0);
      auto load_c = [&](int mt, int j0, double(&re)[2][4], double(&im)[2][4]) {
        const int ra = mt * 16 + g, cl = j0 + 2 * tq;
        const z64* s0 = ra < n ? x + srcrow[ra] * ldx + c_lo + cl : nullptr;
        const z64* s1 = ra + 8 < n ? x + srcrow[ra + 8] * ldx + c_lo + cl : nullptr;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const z64* sr = (q >> 1) ? s1 : s0;
            const int o = j * 8 + (q & 1);
            const z64 v = (sr != nullptr && cl + o < cw) ? sr[o] : make_double2(0.0, 0.0);
            re[j][q] = v.x;
            im[j][q] = v.y;
          }
      };
      auto update = [&](int mt, int j0, double(&re)[2][4], double(&im)[2][4]) {
#pragma unroll
        for (int k4 = 0; k4 < NB; k4 += 4) {
          const z64 v0 = T[tix(mt * 16 + g, k4 + tq)], v1 = T[tix(mt * 16 + g + 8, k4 + tq)];
          z64 y[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) y[j] = Y[(k4 + tq) * YS + j0 + j * 8 + g];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            mma_f64(re[j], v0.x, v1.x, y[j].x);
            mma_f64(im[j], v0.x, v1.x, y[j].y);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            mma_f64(re[j], -v0.y, -v1.y, y[j].y);
            mma_f64(im[j], v0.y, v1.y, y[j].x);
          }
        }
        const int cl = j0 + 2 * tq;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = mt * 16 + g + ((q >> 1) << 3), cc = cl + j * 8 + (q & 1);
            if (r < n && cc < cw) x[r * ldx + c_lo + cc] = make_double2(re[j][q], im[j][q]);
          }
      };
      const int total = (mtiles - 1) * nt;
      const int u0 = (int)((int64_t)total * warp / WARPS3), u1 = (int)((int64_t)total * (warp + 1) / WARPS3);
      if (u0 < u1) {
        int m = u0 / nt, j = u0 % nt;
        double re[2][4], im[2][4], nre[2][4], nim[2][4];
        auto slice = [&](int v) { return v >= kt ? v + 1 : v; };
        auto column = [&](int v) { return (v >= pt ? v + 1 : v) * 16; };
        load_c(slice(m), column(j), re, im);
#pragma unroll 1
        for (int u = u0; u < u1; ++u) {
          const int mt = slice(m), j0 = column(j);
          if (++j == nt) {
            j = 0;
            ++m;
          }
          if (u + 1 < u1) load_c(slice(m), column(j), nre, nim);
          update(mt, j0, re, im);
#pragma unroll
          for (int jj = 0; jj < 2; ++jj)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              re[jj][q] = nre[jj][q];
              im[jj][q] = nim[jj][q];
            }
        }
      }
      __syncthreads();
      for (int u = warp; u < nt; u += WARPS3) {
        double re[2][4] = {}, im[2][4] = {};
        update(kt, (u >= pt ? u + 1 : u) * 16, re, im);
      }
      __syncthreads();
      cluster_sync();
    }

    // Position s holds original row orig[s], so column s of the result is
    // column orig[s] of the inverse. Rows rank, rank + C, ... are gathered
    // (through L2: the other CTAs wrote their columns).
    for (int s = tid; s < n; s += TH) colsrc[orig[cur * np + s]] = s;
    __syncthreads();
    if (RES) {
      for (int idx = tid; idx < n * n; idx += TH) {
        const int r = idx / n, c = idx % n;
        xg[(int64_t)r * X.ld + c] = x[r * ldx + colsrc[c]];
      }
    } else {
      // Each warp holds a whole row in registers between reading and writing.
      for (int r = rank + warp * csplit; r < n; r += WARPS3 * csplit) {
        z64 v[RPL];  // n <= 32 RPL
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
          const int c = lane + 32 * i;
          if (c < n) v[i] = __ldcg(&x[r * ldx + colsrc[c]]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
          const int c = lane + 32 * i;
          if (c < n) x[r * ldx + c] = v[i];
        }
      }
    }
    if (tid == 0 && rank == 0 && info != nullptr && s_sing != 0 && info[b] == 0) info[b] = s_sing;
    __syncthreads();
    // the next matrix's copy must not overwrite rows still being gathered
    cluster_sync();
  }
}

template <int TH, int RPL, bool RES>
int configure3(int n, int64_t batch, int c, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, cudaStream_t s) {
  const size_t smem = Smem3::bytes(n, c, RES);
  QTX_TRY((allow_dynamic_smem(zinv3_kernel<TH, RPL, RES>)));
  const int64_t mats = batch < 131072 ? batch : 131072;
  *cfg = {};
  cfg->gridDim = dim3((unsigned)(mats * c), 1, 1);
  cfg->blockDim = dim3(TH, 1, 1);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)c;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return QTX_OK;
}

template <int TH, int RPL, bool RES>
int launch3(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s, int c) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  QTX_TRY((configure3<TH, RPL, RES>(n, batch, c, &cfg, &attr, s)));
  ProfScope prof(QTX_KERNEL_ZINV, 8.0 * (double)n * n * n * (double)batch, s);
  return launch_chained(zinv3_kernel<TH, RPL, RES>, cfg.gridDim, cfg.blockDim, cfg.dynamicSmemBytes, s, c, n, batch, A,
                        X, info, active, c);
}

// Clusters of c CTAs of the column-split kernel that the GPU runs at once.
int active_clusters(int n, int c) {
  static thread_local std::vector<std::pair<int64_t, int>> cache;  // ((device, n, c), clusters)
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const int64_t key = ((int64_t)dev << 32) + (int64_t)n * 16 + c;
  for (auto& e : cache)
    if (e.first == key) return e.second;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  int nc = 0;
  cudaError_t e = cudaErrorUnknown;
  if (n <= 128) {
    if (configure3<512, 4, false>(n, 148, c, &cfg, &attr, nullptr) == QTX_OK)
      e = cudaOccupancyMaxActiveClusters(&nc, zinv3_kernel<512, 4, false>, &cfg);
  } else if (n <= 256) {
    if (configure3<512, 8, false>(n, 148, c, &cfg, &attr, nullptr) == QTX_OK)
      e = cudaOccupancyMaxActiveClusters(&nc, zinv3_kernel<512, 8, false>, &cfg);
  } else {
    if (configure3<512, 16, false>(n, 148, c, &cfg, &attr, nullptr) == QTX_OK)
      e = cudaOccupancyMaxActiveClusters(&nc, zinv3_kernel<512, 16, false>, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    nc = 0;
  }
  cache.emplace_back(key, nc);
  return nc;
}

static_assert(sizeof(GjPanelSmem<16>) + 64 <= 1024, "static shared memory beside kMaxDynamicSmem");
bool fits_resident(int n) { return n <= 128 && Smem3::bytes(n, 1, true) <= kMaxDynamicSmem; }

// Column split of the n <= 512 kernel: the largest C <= 8 with batch x C within
// the SM count, at least 32 columns per CTA, and all batch clusters
// co-resident; at least two where one CTA's pivot rows and transform do not fit
// (n > 432).
// (Powers of two alone left 64 of 148 SMs idle at n = 512, batch 42: 5.0 ms
// against 3.6 with C = 3.) Inverse path 4 forces the largest power of two
// that the block size allows.
int column_split(int n, int64_t batch) {
  const int path = inverse_path();
  int least = 1;
  while (Smem3::bytes(n, least, false) > kMaxDynamicSmem) ++least;
  if (path != 0 && path != 4) return least;
  if (path == 4) {
    int c = 1;
    while (c < 8 && n / (2 * c) >= 32) c *= 2;
    return c > least ? c : least;
  }
  int c = (int)std::min<int64_t>(std::min(8, n / 32), num_sms() / std::max<int64_t>(batch, 1));
  while (c > least && active_clusters(n, c) < batch) --c;
  return c > least ? c : least;
}

int launch_split(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  // A resident block is not split: n = 100, batch 74 161 us against 165 us in
  // two CTAs through L2.
  if (inverse_path() != 4 && fits_resident(n)) {
    if (n <= 64) return launch3<256, 2, true>(n, batch, A, X, info, active, s, 1);
    return launch3<512, 4, true>(n, batch, A, X, info, active, s, 1);
  }
  const int c = column_split(n, batch);
  if (n <= 128) return launch3<512, 4, false>(n, batch, A, X, info, active, s, c);
  if (n <= 256) return launch3<512, 8, false>(n, batch, A, X, info, active, s, c);
  return launch3<512, 16, false>(n, batch, A, X, info, active, s, c);
}

}  // namespace

int zinv(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  if (n <= 0 || batch <= 0) return QTX_OK;
  if (A.null() || X.null()) {
    set_error("zinv: null matrix");
    return QTX_ERR_ARG;
  }
  if (zinv_prefers_cluster(n, batch)) return zinv_cluster(n, batch, A, X, info, active, s);
  if (n <= 512) return launch_split(n, batch, A, X, info, active, s);
  if (n <= 720) return launch2<8>(n, batch, A, X, info, active, s);
  if (n <= 1024) return launch<8>(n, batch, A, X, info, active, s);
  set_error("zinv: block sizes above 1024 are not supported");
  return QTX_ERR_UNSUPPORTED;
}

}  // namespace qtx
