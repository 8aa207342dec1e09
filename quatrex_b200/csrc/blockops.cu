// Memory-bound block kernels of the NEGF path: elementwise combinations
// with conjugate transposes, the anti-Hermitian projection of X^<, X^> with
// the density epilogue, traces of products (Meir-Wingreen current), the
// per-energy norms of the Sancho-Rubio convergence test and OBC residuals,
// and complex128 <-> complex64 conversion.
//
// The elementwise kernels and traces are templates over the stored element
// type (complex128 = double2 for the FP64 path, complex64 = float2 for the
// mixed path); arithmetic is done in double either way. Transposed operands
// are staged through a 32x32 shared-memory tile (one padding column) so
// global loads and stores stay coalesced. Reductions cut an entry into fixed
// bands of rows that the CTAs of a thread-block cluster sum (warp shuffles, one
// shared-memory combine per band) and add in order: deterministic.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace qtx {
namespace {

constexpr int TILE = 32;
constexpr int ROWS = 8;  // threads per tile column: block = 32 x 8

__device__ __forceinline__ z64 ld2(const double2& v) { return v; }
__device__ __forceinline__ z64 ld2(const float2& v) { return make_double2(v.x, v.y); }
template <typename T>
__device__ __forceinline__ T st2(z64 v);
template <>
__device__ __forceinline__ double2 st2<double2>(z64 v) {
  return v;
}
template <>
__device__ __forceinline__ float2 st2<float2>(z64 v) {
  return make_float2((float)v.x, (float)v.y);
}

struct CombineArgs {
  MatRef out;
  Addend t[kMaxAddends];
  int nterms;
  int m, n;
  int64_t batch;
  const int* active;
};

// out = sum_t coef_t op_t(X_t) on 32x32 tiles; grid (tiles_n, tiles_m, batch).
template <typename T>
__global__ void __launch_bounds__(TILE* ROWS) combine_kernel(const CombineArgs a) {
  __shared__ z64 tile[TILE][TILE + 1];
  const int c0 = blockIdx.x * TILE, r0 = blockIdx.y * TILE;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int64_t b = blockIdx.z; b < a.batch; b += gridDim.z) {
    if (a.active != nullptr && a.active[b] == 0) continue;
    z64 acc[TILE / ROWS];
#pragma unroll
    for (int i = 0; i < TILE / ROWS; ++i) acc[i] = make_double2(0.0, 0.0);
    for (int t = 0; t < a.nterms; ++t) {
      const Addend& ad = a.t[t];
      const T* p = at<const T>(ad.m, b);
      if (!ad.conj_trans) {
#pragma unroll
        for (int i = 0; i < TILE / ROWS; ++i) {
          const int r = r0 + ty + i * ROWS, c = c0 + tx;
          if (r < a.m && c < a.n) acc[i] = zfma(ad.coef, ld2(p[(int64_t)r * ad.m.ld + c]), acc[i]);
        }
      } else {
        // op(X)[r][c] = conj(X[c][r]): load the (c0, r0) tile of X coalesced.
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TILE / ROWS; ++i) {
          const int xr = c0 + ty + i * ROWS, xc = r0 + tx;  // X row = out col
          tile[ty + i * ROWS][tx] =
              (xr < a.n && xc < a.m) ? ld2(p[(int64_t)xr * ad.m.ld + xc]) : make_double2(0.0, 0.0);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TILE / ROWS; ++i) {
          const int r = r0 + ty + i * ROWS, c = c0 + tx;
          if (r < a.m && c < a.n) acc[i] = zfma(ad.coef, zconj(tile[tx][ty + i * ROWS]), acc[i]);
        }
      }
    }
    T* o = at<T>(a.out, b);
#pragma unroll
    for (int i = 0; i < TILE / ROWS; ++i) {
      const int r = r0 + ty + i * ROWS, c = c0 + tx;
      if (r < a.m && c < a.n) o[(int64_t)r * a.out.ld + c] = st2<T>(acc[i]);
    }
  }
}

// out_k = 0.5 (X_k - X_k^H) for `count` (1 or 2) stacks in one launch;
// density[b * ds + off + r] = Im X_0[r][r].
struct AntihermArgs {
  MatRef X[2], out[2];
};
template <typename T>
__global__ void __launch_bounds__(TILE* ROWS)
    antiherm_kernel(int n, int64_t batch, int count, const AntihermArgs args, double* density, int64_t ds,
                    int64_t doff) {
  __shared__ z64 tile[TILE][TILE + 1];
  chain_begin();
  const int c0 = blockIdx.x * TILE, r0 = blockIdx.y * TILE;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int64_t z = blockIdx.z; z < batch * count; z += gridDim.z) {
    const int k = z >= batch ? 1 : 0;
    const int64_t b = z - k * batch;
    const MatRef& X = args.X[k];
    const MatRef& out = args.out[k];
    double* dens = k == 0 ? density : nullptr;
    const T* x = at<const T>(X, b);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TILE / ROWS; ++i) {
      const int xr = c0 + ty + i * ROWS, xc = r0 + tx;
      tile[ty + i * ROWS][tx] = (xr < n && xc < n) ? ld2(x[(int64_t)xr * X.ld + xc]) : make_double2(0, 0);
    }
    __syncthreads();
    T* o = out.null() ? nullptr : at<T>(out, b);
#pragma unroll
    for (int i = 0; i < TILE / ROWS; ++i) {
      const int r = r0 + ty + i * ROWS, c = c0 + tx;
      if (r < n && c < n) {
        const z64 v = ld2(x[(int64_t)r * X.ld + c]);
        const z64 w = tile[tx][ty + i * ROWS];  // X[c][r]
        const z64 h = make_double2(0.5 * (v.x - w.x), 0.5 * (v.y + w.y));
        if (o != nullptr) o[(int64_t)r * out.ld + c] = st2<T>(h);
        if (dens != nullptr && r == c) dens[b * ds + doff + r] = h.y;
      }
    }
  }
}

template <typename V>
__device__ __forceinline__ V block_sum(V v, V* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  V s = 0;
  const int nw = blockDim.x >> 5;
  for (int w = 0; w < nw; ++w) s += red[w];
  return s;
}

// Reductions of one stack entry. An entry is cut into kChunks bands of rows,
// each band is summed by one CTA (the S CTAs of the entry's thread-block
// cluster take the bands rank, rank + S, ...), and rank 0 adds the bands in
// order through distributed shared memory: the result depends neither on
// timing nor on S. One CTA per entry leaves most SMs idle below 148 entries
// and each thread with few loads in flight: the Sancho-Rubio measure of 128
// entries of 256 x 256 took 205 us, against 41 us at the HBM rate.
constexpr int kChunks = 8;
constexpr int RT = 256;  // threads

// Sum of the kChunks band partials (V values each) of this cluster's entry,
// valid in rank 0's thread 0.
template <int V>
__device__ __forceinline__ void cluster_total(cg::cluster_group& cluster, double (&part)[kChunks][V], double (&tot)[V]) {
  cluster.sync();
  if (cluster.block_rank() == 0 && threadIdx.x == 0) {
    const int S = (int)cluster.num_blocks();
#pragma unroll
    for (int v = 0; v < V; ++v) tot[v] = 0.0;
    for (int q = 0; q < kChunks; ++q) {
      const double* pq = cluster.map_shared_rank(&part[q][0], q % S);
#pragma unroll
      for (int v = 0; v < V; ++v) tot[v] += pq[v];
    }
  }
  cluster.sync();  // the partials stay readable until rank 0 has summed them
}

struct TraceArgs {
  int count;  // 1 or 2 products
  MatRef X[2], Y[2];
  z64 coef[2];
};

// res[b] = sum_k coef_k Tr(X_k Y_k), Tr(X Y) = sum_{r,c} X[r][c] Y[c][r] on
// 32 x 32 tiles (the Y tile staged transposed).
template <typename T>
__global__ void __launch_bounds__(RT) trace_kernel(int n, int64_t batch, const TraceArgs args, z64* res, int64_t rs,
                                                   int64_t roff) {
  __shared__ z64 tile[TILE][TILE + 1];
  __shared__ double red[RT / 32];
  __shared__ double part[kChunks][4];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  chain_begin();
  cg::cluster_group cluster = cg::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int64_t b = blockIdx.x / S;  // uniform within a cluster
  const int tiles = (n + TILE - 1) / TILE;
  for (int q = rank; q < kChunks; q += S) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    const int t0 = tiles * q / kChunks, t1 = tiles * (q + 1) / kChunks;
    for (int k = 0; k < args.count && b < batch; ++k) {
      const T* x = at<const T>(args.X[k], b);
      const T* y = at<const T>(args.Y[k], b);
      const int64_t ldx = args.X[k].ld, ldy = args.Y[k].ld;
      double sre = 0.0, sim = 0.0;
      for (int r0 = t0 * TILE; r0 < t1 * TILE; r0 += TILE)
        for (int c0 = 0; c0 < n; c0 += TILE) {
          z64 xv[TILE / ROWS], yv[TILE / ROWS];
#pragma unroll
          for (int i = 0; i < TILE / ROWS; ++i) {
            const int yr = c0 + ty + i * ROWS, yc = r0 + tx;
            yv[i] = (yr < n && yc < n) ? ld2(y[(int64_t)yr * ldy + yc]) : make_double2(0, 0);
            const int r = r0 + ty + i * ROWS, c = c0 + tx;
            xv[i] = (r < n && c < n) ? ld2(x[(int64_t)r * ldx + c]) : make_double2(0, 0);
          }
          __syncthreads();
#pragma unroll
          for (int i = 0; i < TILE / ROWS; ++i) tile[ty + i * ROWS][tx] = yv[i];
          __syncthreads();
#pragma unroll
          for (int i = 0; i < TILE / ROWS; ++i) {
            if (r0 + ty + i * ROWS < n && c0 + tx < n) {
              const z64 w = tile[tx][ty + i * ROWS];  // Y[c][r]
              sre += xv[i].x * w.x - xv[i].y * w.y;
              sim += xv[i].x * w.y + xv[i].y * w.x;
            }
          }
        }
      s[2 * k] = sre;
      s[2 * k + 1] = sim;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double p = block_sum(s[v], red);
      if (threadIdx.x == 0) part[q][v] = p;
    }
  }
  double tot[4];
  cluster_total<4>(cluster, part, tot);
  if (b < batch && rank == 0 && threadIdx.x == 0) {
    z64 v = zmul(args.coef[0], make_double2(tot[0], tot[1]));
    if (args.count > 1) v = zadd(v, zmul(args.coef[1], make_double2(tot[2], tot[3])));
    res[b * rs + roff] = v;
  }
}

// sum over the m x n elements of f(x, y) (V values), then done(b, totals).
template <typename T, int V, class F, class Done>
__global__ void __launch_bounds__(RT) reduce_kernel(int m, int n, int64_t batch, MatRef X, MatRef Y, F f, Done done,
                                                    const int* active) {
  __shared__ double red[RT / 32];
  __shared__ double part[kChunks][V];
  chain_begin();
  cg::cluster_group cluster = cg::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int64_t b = blockIdx.x / S;
  if (b >= batch || (active != nullptr && active[b] == 0)) return;  // whole clusters
  const T* x = at<const T>(X, b);
  const T* y = at<const T>(Y, b);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = rank; q < kChunks; q += S) {
    double s[V];
#pragma unroll
    for (int v = 0; v < V; ++v) s[v] = 0.0;
    const int r1 = (int)((int64_t)m * (q + 1) / kChunks);
    for (int r = (int)((int64_t)m * q / kChunks) + warp; r < r1; r += RT / 32) {
      const T* xr = x + (int64_t)r * X.ld;
      const T* yr = y + (int64_t)r * Y.ld;
#pragma unroll 4
      for (int c = lane; c < n; c += 32) f(ld2(xr[c]), ld2(yr[c]), s);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const double p = block_sum(s[v], red);
      if (threadIdx.x == 0) part[q][v] = p;
    }
  }
  double tot[V];
  cluster_total<V>(cluster, part, tot);
  if (rank == 0 && threadIdx.x == 0) done(b, tot);
}

// |z|. x^2 + y^2 over- and underflows only where the square of |z| that is summed
// does too; an infinite part counts as infinite beside a NaN, as in hypot: an
// energy that overflows has not converged, and the batch-wide maximum skips NaN.
__device__ __forceinline__ double modulus(z64 z) {
  return isinf(z.x) || isinf(z.y) ? INFINITY : sqrt(z.x * z.x + z.y * z.y);
}
// (|x| + |y|)^2; delta[b] = sqrt(sum) / 2.
struct DeltaTerm {
  __device__ __forceinline__ void operator()(z64 a, z64 w, double (&s)[1]) const {
    const double v = modulus(a) + modulus(w);
    s[0] += v * v;
  }
};
struct DeltaDone {
  double* delta;
  __device__ void operator()(int64_t b, const double (&t)[1]) const { delta[b] = 0.5 * sqrt(t[0]); }
};
// |x - y|^2 and |x|^2.
struct DiffTerm {
  __device__ __forceinline__ void operator()(z64 a, z64 w, double (&s)[2]) const {
    const double dr = a.x - w.x, di = a.y - w.y;
    s[0] += dr * dr + di * di;
    s[1] += a.x * a.x + a.y * a.y;
  }
};
struct DiffDone {
  double *nd, *nx, *rel;
  __device__ void operator()(int64_t b, const double (&t)[2]) const {
    if (nd != nullptr) nd[b] = sqrt(t[0]);
    if (nx != nullptr) nx[b] = sqrt(t[1]);
    if (rel != nullptr) rel[b] = sqrt(t[0]) / sqrt(t[1]);
  }
};
// Re conj(y) x.
struct InnerTerm {
  __device__ __forceinline__ void operator()(z64 a, z64 w, double (&s)[1]) const { s[0] += a.x * w.x + a.y * w.y; }
};
struct InnerDone {
  double* out;
  __device__ void operator()(int64_t b, const double (&t)[1]) const { out[b] = t[0]; }
};

template <typename TI, typename TO>
__global__ void convert_kernel(int m, int n, int64_t batch, MatRef in, MatRef out) {
  const int64_t per = (int64_t)m * n, total = per * batch;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = i / per, e = i % per;
    const int r = (int)(e / n), c = (int)(e % n);
    at<TO>(out, b)[(int64_t)r * out.ld + c] = st2<TO>(ld2(at<const TI>(in, b)[(int64_t)r * in.ld + c]));
  }
}

unsigned grid_z(int64_t batch) { return (unsigned)(batch < 65535 ? batch : 65535); }

// CTAs (a cluster) per entry of a reduction: a power of two up to kChunks while
// all CTAs of the batch are resident at once (8 per SM).
int reduce_split(int64_t batch) {
  int S = 1;
  while (S < kChunks && batch * S * 2 <= 8 * (int64_t)num_sms()) S *= 2;
  return S;
}

template <typename T, int V, class F, class Done>
int reduce_t(int m, int n, int64_t batch, MatRef X, MatRef Y, F f, Done done, const int* active, cudaStream_t s) {
  if (m <= 0 || n <= 0 || batch <= 0) return QTX_OK;
  ProfScope prof(QTX_KERNEL_REDUCE, 2.0 * sizeof(T) * m * n * (double)batch, s);
  const int S = reduce_split(batch);
  return launch_chained(reduce_kernel<T, V, F, Done>, dim3((unsigned)(batch * S)), dim3(RT), 0, s, S, m, n, batch, X, Y,
                        f, done, active);
}

template <typename T>
int combine_t(int m, int n, int64_t batch, MatRef out, const Addend* terms, int nterms,
              const int* active, cudaStream_t s) {
  if (m <= 0 || n <= 0 || batch <= 0) return QTX_OK;
  CombineArgs a{};
  a.out = out;
  a.m = m;
  a.n = n;
  a.batch = batch;
  a.active = active;
  a.nterms = 0;
  for (int t = 0; t < nterms; ++t) {
    if (terms[t].m.null()) continue;
    if (a.nterms >= kMaxAddends) {
      set_error("combine: too many terms");
      return QTX_ERR_ARG;
    }
    a.t[a.nterms++] = terms[t];
  }
  dim3 grid((n + TILE - 1) / TILE, (m + TILE - 1) / TILE, grid_z(batch));
  ProfScope prof(QTX_KERNEL_BLOCKOPS, (double)sizeof(T) * m * n * (double)batch * (a.nterms + 1), s);
  combine_kernel<T><<<grid, dim3(TILE, ROWS), 0, s>>>(a);
  QTX_CHECK_LAUNCH();
  return QTX_OK;
}

template <typename T>
int antiherm_t(int n, int64_t batch, int count, const MatRef* X, const MatRef* out, double* density,
               int64_t dens_stride, int64_t dens_off, cudaStream_t s) {
  if (n <= 0 || batch <= 0) return QTX_OK;
  AntihermArgs args{};
  for (int k = 0; k < count; ++k) {
    args.X[k] = X[k];
    args.out[k] = out[k];
  }
  dim3 grid((n + TILE - 1) / TILE, (n + TILE - 1) / TILE, grid_z(batch * count));
  ProfScope prof(QTX_KERNEL_BLOCKOPS, 2.0 * sizeof(T) * n * n * (double)batch * count, s);
  return launch_chained(antiherm_kernel<T>, grid, dim3(TILE, ROWS), 0, s, 1, n, batch, count, args, density,
                        dens_stride, dens_off);
}

template <typename T>
int trace_t(int n, int64_t batch, int count, const MatRef* X, const MatRef* Y, const z64* coef, z64* result,
            int64_t rstride, int64_t roff, cudaStream_t s) {
  if (n <= 0 || batch <= 0 || count <= 0) return QTX_OK;
  TraceArgs args{};
  args.count = count;
  for (int k = 0; k < count; ++k) {
    args.X[k] = X[k];
    args.Y[k] = Y[k];
    args.coef[k] = coef[k];
  }
  ProfScope prof(QTX_KERNEL_REDUCE, 2.0 * sizeof(T) * n * n * (double)batch * count, s);
  const int S = reduce_split(batch);
  return launch_chained(trace_kernel<T>, dim3((unsigned)(batch * S)), dim3(RT), 0, s, S, n, batch, args, result,
                        rstride, roff);
}

template <typename TI, typename TO>
int convert_t(int m, int n, int64_t batch, MatRef in, MatRef out, cudaStream_t s) {
  if (m <= 0 || n <= 0 || batch <= 0) return QTX_OK;
  const int64_t total = (int64_t)m * n * batch;
  const int64_t want = (total + 255) / 256;
  const unsigned blocks = (unsigned)(want < 148 * 64 ? want : 148 * 64);
  ProfScope prof(QTX_KERNEL_FORMAT, (double)(sizeof(TI) + sizeof(TO)) * (double)total, s);
  convert_kernel<TI, TO><<<blocks, 256, 0, s>>>(m, n, batch, in, out);
  QTX_CHECK_LAUNCH();
  return QTX_OK;
}

}  // namespace

int zcombine(int m, int n, int64_t batch, MatRef out, const Addend* terms, int nterms,
             const int* active, cudaStream_t s) {
  return combine_t<double2>(m, n, batch, out, terms, nterms, active, s);
}
int ccombine(int m, int n, int64_t batch, MatRef out, const Addend* terms, int nterms,
             const int* active, cudaStream_t s) {
  return combine_t<float2>(m, n, batch, out, terms, nterms, active, s);
}

int zantiherm(int n, int64_t batch, int count, const MatRef* X, const MatRef* out, double* density,
              int64_t dens_stride, int64_t dens_off, cudaStream_t s) {
  return antiherm_t<double2>(n, batch, count, X, out, density, dens_stride, dens_off, s);
}
int cantiherm(int n, int64_t batch, int count, const MatRef* X, const MatRef* out, double* density,
              int64_t dens_stride, int64_t dens_off, cudaStream_t s) {
  return antiherm_t<float2>(n, batch, count, X, out, density, dens_stride, dens_off, s);
}

int ztrace_prod(int n, int64_t batch, int count, const MatRef* X, const MatRef* Y, const z64* coef, z64* result,
                int64_t rstride, int64_t roff, cudaStream_t s) {
  return trace_t<double2>(n, batch, count, X, Y, coef, result, rstride, roff, s);
}
int ctrace_prod(int n, int64_t batch, int count, const MatRef* X, const MatRef* Y, const z64* coef, z64* result,
                int64_t rstride, int64_t roff, cudaStream_t s) {
  return trace_t<float2>(n, batch, count, X, Y, coef, result, rstride, roff, s);
}

int sr_delta(int n, int64_t batch, MatRef X, MatRef Y, double* delta, const int* active, cudaStream_t s) {
  return reduce_t<double2, 1>(n, n, batch, X, Y, DeltaTerm{}, DeltaDone{delta}, active, s);
}

int znorm_diff(int n, int64_t batch, MatRef X, MatRef Y, double* nrm_diff, double* nrm,
               double* rel, cudaStream_t s) {
  return reduce_t<double2, 2>(n, n, batch, X, Y, DiffTerm{}, DiffDone{nrm_diff, nrm, rel}, nullptr, s);
}

int zre_inner(int m, int n, int64_t batch, MatRef P, MatRef G, double* out, cudaStream_t s) {
  return reduce_t<double2, 1>(m, n, batch, P, G, InnerTerm{}, InnerDone{out}, nullptr, s);
}

int convert_c64_to_c128(int m, int n, int64_t batch, MatRef in, MatRef out, cudaStream_t s) {
  return convert_t<float2, double2>(m, n, batch, in, out, s);
}
int convert_c128_to_c64(int m, int n, int64_t batch, MatRef in, MatRef out, cudaStream_t s) {
  return convert_t<double2, float2>(m, n, batch, in, out, s);
}

}  // namespace qtx
