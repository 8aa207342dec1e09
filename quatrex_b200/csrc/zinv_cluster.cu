// Batched complex128 inverse with the whole matrix on chip: one thread-block
// cluster per matrix, Gauss-Jordan with partial pivoting in distributed
// shared memory.
//
// Replaces the same batched inverse of qttools kernels/linalg/inv.py:6-40 as
// zinv.cu (numpy.linalg.inv / cupy.linalg.solve(a, I)), with the same pivot
// rule (largest |Re| + |Im| at or below the diagonal, lowest row on ties) and
// the same info convention (1-based column of the first zero pivot).
//
// Why: the column-split kernel streams the n x n matrix through L2 or HBM once
// per 16-column panel (16 passes at n = 256); the multi-CTA path pays three
// launches per panel. While all clusters of a batch are resident, a cluster of
// C = ceil(n / 32) CTAs (8 at n = 256) holds the matrix entirely in shared
// memory -- 32 columns per CTA -- and runs every panel on chip:
//
//   load:   each CTA fetches its 32 columns with TMA (cp.async.bulk.tensor,
//           3-D tensor map over (re/im doubles, rows, batch), 128-byte
//           swizzle, no multicast) into four [rows][8 complex] chunks;
//   panel:  the CTA owning the 16 columns of panel K factors them in place
//           (gj_panel.cuh), then arrives on the cluster barrier;
//   update: every CTA receives the panel transform T = X[:, K] and the row
//           moves from the owner (bulk copies) and updates its own columns,
//             X[r, J] = (r in K ? 0 : X[src(r), J]) + T[r, :] Y[:, J],
//           Y = X[src(K), J], with FP64 tensor-core MMAs (mma.sync m16n8k4, 4M
//           complex split); src carries the row interchanges;
//   store:  columns are gathered back through DSMEM in the inverse column
//           order of the pivoting and written with coalesced stores.
//
// HBM traffic is the algorithmic minimum (read and write the matrix once).
// One cluster barrier per panel; the owner of the next panel factors it as
// soon as its own update is done while the other CTAs finish theirs.
// Every wait on the TMA mbarrier is bounded: on a time-out the CTA records
// the error (qtx_zinv_cluster_status), keeps taking part in every cluster
// barrier so that no CTA of the cluster waits forever, and its results are
// not to be used.
#include <cooperative_groups.h>
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "gj_panel.cuh"

namespace cg = cooperative_groups;

namespace qtx {

__device__ int g_zinv_cluster_error = 0;

namespace {

constexpr int CW = 32;          // columns per CTA
constexpr int CNB = 16;         // panel width
constexpr int CT = 512;         // threads per CTA
constexpr int CWARPS = CT / 32;
constexpr int YS = CW + 2;      // Y row stride (complex)
constexpr long long kWait = 1ll << 26;

__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Element (r, j) of a CTA's 32 columns: four chunks of [npad rows][8
// complex], 16-byte unit swizzled with the row (the TMA SWIZZLE_128B layout).
__device__ __forceinline__ int xoff(int npad, int r, int j) {
  return (j >> 3) * (npad * 8) + r * 8 + ((j & 7) ^ (r & 7));
}

struct ClusterSmem {
  // byte offsets inside the dynamic shared memory (base aligned to 1024)
  int npad;
  size_t x, t, y, src, orig, colsrc, bar, total;
  __host__ __device__ explicit ClusterSmem(int n) {
    npad = (n + 15) & ~15;
    x = 0;                                                  // 4 chunks [npad][8]
    t = x + (size_t)4 * npad * 8 * sizeof(z64);             // 2 chunks [npad][8]
    y = t + (size_t)2 * npad * 8 * sizeof(z64);             // [CNB][YS]
    src = y + (size_t)CNB * YS * sizeof(z64);               // 2 x npad ints
    orig = src + (size_t)2 * npad * sizeof(int);            // 2 x npad ints
    colsrc = orig + (size_t)2 * npad * sizeof(int);         // npad ints
    bar = (colsrc + (size_t)npad * sizeof(int) + 15) & ~(size_t)15;  // 2 mbarriers
    total = bar + 16 + 1024;  // + alignment slack of the base
  }
};

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
  for (long long it = 0; it < kWait; ++it) {
    uint32_t done = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(saddr(bar)), "r"(parity));
    if (done) return true;
  }
  return false;
}

template <int C>
__global__ void __launch_bounds__(CT, 1)
    zinv_cluster_kernel(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active,
                        const __grid_constant__ CUtensorMap tmap, int use_tma) {
  chain_begin();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int64_t b = blockIdx.x / C;
  if (b >= batch) return;  // whole clusters only: blockIdx.x / C is uniform in a cluster
  if (active != nullptr && active[b] == 0) return;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const ClusterSmem L(n);
  const int npad = L.npad;
  z64* Xs = reinterpret_cast<z64*>(base + L.x);
  z64* Ts = reinterpret_cast<z64*>(base + L.t);
  z64* Ys = reinterpret_cast<z64*>(base + L.y);
  // row of X that each position receives, by panel parity: the owner may factor
  // the next panel while this one's copies to the others are in flight
  int* const srcbuf = reinterpret_cast<int*>(base + L.src);
  int* orig = reinterpret_cast<int*>(base + L.orig);   // original row of each position (2 buffers)
  int* colsrc = reinterpret_cast<int*>(base + L.colsrc);
  uint64_t* lbar = reinterpret_cast<uint64_t*>(base + L.bar);  // the load of A
  uint64_t* tbar = lbar + 1;                                    // the panel transforms
  __shared__ int s_sing, s_first;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tq = lane & 3;
  const int col0 = rank * CW;  // first global column of this CTA
  const size_t chunk = (size_t)npad * 8;  // complex elements per 8-column chunk

  // ---- load this CTA's 32 columns --------------------------------------
  for (int r = tid; r < npad; r += CT) srcbuf[r] = srcbuf[npad + r] = orig[r] = r;
  if (tid == 0) {
    s_sing = 0;
    s_first = 0x7fffffff;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(lbar)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(tbar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();
  if (use_tma) {
    if (tid == 0) {
      const uint32_t bytes = 4u * (uint32_t)n * 128u;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(lbar)), "r"(bytes)
                   : "memory");
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int x = 2 * (col0 + 8 * i);  // in doubles: 16-byte aligned
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(saddr(Xs + i * chunk)),
            "l"(&tmap), "r"(x), "r"(0), "r"((int)b), "r"(saddr(lbar))
            : "memory");
      }
    }
    if (warp == 0 && !mbar_wait_bounded(lbar, 0) && lane == 0) atomicExch(&g_zinv_cluster_error, 1);
  } else {
    const z64* a = at<const z64>(A, b);
    for (int idx = tid; idx < n * CW; idx += CT) {
      const int r = idx / CW, j = idx % CW, c = col0 + j;
      Xs[xoff(npad, r, j)] = c < n ? a[(int64_t)r * A.ld + c] : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  cluster.sync();  // every CTA resident and loaded before any DSMEM access

  // ---- panels -----------------------------------------------------------
  uint32_t tphase = 0;
  int cur = 0;
  for (int k0 = 0; k0 < n; k0 += CNB) {
    const int owner = k0 / CW, kl = k0 - owner * CW;
    const int nbp = min(CNB, n - k0);
    const bool own = rank == owner;
    int* const srcrow = srcbuf + ((k0 / CNB) & 1) * npad;
    const uint32_t tbytes = (uint32_t)(2 * chunk * sizeof(z64)) + (uint32_t)npad * sizeof(int);

    if (own) {
      gj_factor_panel<CNB, C <= 4 ? 2 : 1>(
          n, k0, nbp, [=](int r, int c) { return Xs[xoff(npad, r, kl + c)]; },
          [=](int r, int c, z64 v) { Xs[xoff(npad, r, kl + c)] = v; },
          [=](int r, int pos) { srcrow[pos] = r; }, &s_sing);
      // the panel's stores must be visible to the bulk copies below
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    } else if (tid == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(tbar)), "r"(tbytes)
                   : "memory");
    }
    // Every CTA has finished reading the previous transform and the owner
    // has factored this panel.
    cluster_arrive();
    cluster_wait();
    if (own && tid == 0) {
      // The transform (columns kl..kl+15: two whole chunks) and the row moves
      // to every other CTA of the cluster (bulk copies, no multicast).
      const uint32_t src_t = saddr(Xs + (size_t)(kl >> 3) * chunk);
      const uint32_t src_p = saddr(srcrow);
      for (int r = 0; r < C; ++r) {
        if (r == rank) continue;
        const uint32_t mb = cluster_addr(saddr(tbar), r);
        asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                cluster_addr(saddr(Ts), r)),
            "r"(src_t), "r"((uint32_t)(2 * chunk * sizeof(z64))), "r"(mb)
            : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                cluster_addr(saddr(srcrow), r)),
            "r"(src_p), "r"((uint32_t)(npad * sizeof(int))), "r"(mb)
            : "memory");
      }
    }
    if (!own) {
      if (warp == 0 && !mbar_wait_bounded(tbar, tphase) && lane == 0) atomicExch(&g_zinv_cluster_error, 1);
      tphase ^= 1u;
      __syncthreads();
    }
    const z64* T = own ? Xs + (size_t)(kl >> 3) * chunk : Ts;

    // Pivot rows of this CTA's other columns, one element per thread.
    {
      const int kk = tid / CW, j = tid % CW;
      const bool use = kk < nbp && !(own && j >= kl && j < kl + CNB);
      Ys[kk * YS + j] = use ? Xs[xoff(npad, srcrow[k0 + kk], j)] : make_double2(0.0, 0.0);
    }
    for (int r = tid; r < n; r += CT) orig[(cur ^ 1) * npad + r] = orig[cur * npad + srcrow[r]];
    cur ^= 1;
    __syncthreads();

    // Update in tiles of 16 rows x 8 columns dealt to the warps, the owner
    // without the panel's two: first the slices other than the pivots', from
    // the rows that LAPACK's interchanges would have brought there, then (those
    // read rows of K) the pivots'. One warp applying the interchanges ahead of
    // an update of whole 16-row slices took 18 of 37 kcycles per panel at
    // n = 128.
    const int mtiles = npad >> 4, kt = k0 / CNB, nt = own ? 2 : 4;
    for (int phase = 0; phase < 2; ++phase) {
      const int units = phase == 0 ? (mtiles - 1) * nt : nt;
      for (int u = warp; u < units; u += CWARPS) {
        int mt = u / nt, jt = u % nt;
        if (phase == 1)
          mt = kt;
        else if (mt >= kt)
          ++mt;
        if (own && jt * 8 >= kl) jt += 2;
        const int ra = mt * 16 + g;
        const int q0 = srcrow[ra], q1 = srcrow[ra + 8];
        double cre[4], cim[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          z64 v = make_double2(0.0, 0.0);
          if (phase == 0) v = Xs[xoff(npad, (q >> 1) ? q1 : q0, jt * 8 + 2 * tq + (q & 1))];
          cre[q] = v.x;
          cim[q] = v.y;
        }
#pragma unroll
        for (int k4 = 0; k4 < CNB; k4 += 4) {
          const int ka = k4 + tq;
          const z64 v0 = T[(ka >> 3) * chunk + ra * 8 + ((ka & 7) ^ (ra & 7))];
          const z64 v1 = T[(ka >> 3) * chunk + (ra + 8) * 8 + ((ka & 7) ^ ((ra + 8) & 7))];
          const z64 bv = Ys[ka * YS + jt * 8 + g];
          mma_f64(cre, v0.x, v1.x, bv.x);
          mma_f64(cim, v0.x, v1.x, bv.y);
          mma_f64(cre, -v0.y, -v1.y, bv.y);
          mma_f64(cim, v0.y, v1.y, bv.x);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = ra + ((q >> 1) << 3);
          if (r < n) Xs[xoff(npad, r, jt * 8 + 2 * tq + (q & 1))] = make_double2(cre[q], cim[q]);
        }
      }
      __syncthreads();
    }
  }

  // ---- column permutation and store --------------------------------------
  // Position s holds original row orig[s]: column s of the Gauss-Jordan result
  // is column orig[s] of the inverse.
  for (int s = tid; s < n; s += CT) colsrc[orig[cur * npad + s]] = s;
  if (tid == 0) {
    if (s_sing != 0) atomicMin(cluster.map_shared_rank(&s_first, 0), s_sing);
  }
  __syncthreads();
  cluster.sync();  // every update and every first-singular report done
  {
    z64* x = at<z64>(X, b);
    const int ncols = min(CW, n - col0);
    // a warp stores 32 consecutive output columns of one row (512 bytes)
    const int jj = tid % CW;
    const int src = jj < ncols ? colsrc[col0 + jj] : 0;
    const z64* rX = cluster.map_shared_rank(Xs, src / CW);
    const int sj = src % CW;
    for (int r0 = tid / CW; r0 < n; r0 += 4 * (CT / CW)) {
      z64 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + u * (CT / CW);
        if (r < n && jj < ncols) v[u] = rX[xoff(npad, r, sj)];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + u * (CT / CW);
        if (r < n && jj < ncols) x[(int64_t)r * X.ld + col0 + jj] = v[u];
      }
    }
  }
  if (rank == 0 && tid == 0 && info != nullptr && s_first != 0x7fffffff && info[b] == 0) info[b] = s_first;
  cluster.sync();  // no CTA leaves while another still reads its shared memory
}

// ---- host side -----------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static std::once_flag once;
  static EncodeTiled fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  });
  return fn;
}

// 3-D tensor map (re/im doubles, rows, batch) of A with a 16 x n box, or
// false when the layout does not allow one (then plain loads are used).
bool make_map(CUtensorMap* map, int n, int64_t batch, const MatRef& A) {
  EncodeTiled enc = encode_fn();
  if (enc == nullptr) return false;
  const uintptr_t p = reinterpret_cast<uintptr_t>(A.p);
  if ((p & 15) != 0 || A.stride <= 0 || A.ld < n || batch > 0x7fffffff) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)2 * n, (cuuint64_t)n, (cuuint64_t)batch};
  const cuuint64_t strides[2] = {(cuuint64_t)A.ld * sizeof(z64), (cuuint64_t)A.stride * sizeof(z64)};
  if (strides[0] >= (1ull << 40) || strides[1] >= (1ull << 40)) return false;
  const cuuint32_t box[3] = {16, (cuuint32_t)n, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, A.p, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <int C>
int launch_cluster(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  const ClusterSmem L(n);
  const size_t smem = L.total;
  QTX_TRY(allow_dynamic_smem(zinv_cluster_kernel<C>));
  CUtensorMap map;
  const int use_tma = make_map(&map, n, batch, A) ? 1 : 0;
  if (!use_tma) memset(&map, 0, sizeof(map));
  ProfScope prof(QTX_KERNEL_ZINV, 8.0 * (double)n * n * n * (double)batch, s);
  return launch_chained(zinv_cluster_kernel<C>, dim3((unsigned)(batch * C)), dim3(CT), smem, s, C, n, batch, A, X, info,
                        active, map, use_tma);
}

}  // namespace

size_t zinv_cluster_smem(int n) { return ClusterSmem(n).total; }

int zinv_cluster(int n, int64_t batch, MatRef A, MatRef X, int* info, const int* active, cudaStream_t s) {
  if (n <= 0 || batch <= 0) return QTX_OK;
  if (n > 8 * CW || batch * ((n + CW - 1) / CW) > 0x7fffffffll) {
    set_error("zinv_cluster: block size above 256 or batch too large");
    return QTX_ERR_UNSUPPORTED;
  }
  switch ((n + CW - 1) / CW) {
    case 1: return launch_cluster<1>(n, batch, A, X, info, active, s);
    case 2: return launch_cluster<2>(n, batch, A, X, info, active, s);
    case 3: return launch_cluster<3>(n, batch, A, X, info, active, s);
    case 4: return launch_cluster<4>(n, batch, A, X, info, active, s);
    case 5: return launch_cluster<5>(n, batch, A, X, info, active, s);
    case 6: return launch_cluster<6>(n, batch, A, X, info, active, s);
    case 7: return launch_cluster<7>(n, batch, A, X, info, active, s);
    default: return launch_cluster<8>(n, batch, A, X, info, active, s);
  }
}

int zinv_cluster_status_take(int* flag) {
  int h = 0;
  QTX_CHECK_CUDA(cudaMemcpyFromSymbol(&h, g_zinv_cluster_error, sizeof(int)));
  if (h) {
    const int zero = 0;
    QTX_CHECK_CUDA(cudaMemcpyToSymbol(g_zinv_cluster_error, &zero, sizeof(int)));
  }
  *flag = h;
  return QTX_OK;
}

}  // namespace qtx
