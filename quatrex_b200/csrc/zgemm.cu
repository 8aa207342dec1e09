// Batched complex128 GEMM on the sm_100a FP64 tensor pipe.
//
// Every block product of the RGF recursions (qttools
// greens_function_solver/rgf.py:71-110,234-428) and of the Sancho-Rubio
// decimation (boundary_conditions/obc/sancho_rubio.py:64-71) goes through
// this kernel. tcgen05 has no FP64 kind, so FP64 products are issued as
// warp-level DMMA (mma.sync m16n8k4 .f64) -- on B200 the FP64 tensor and
// vector rates are equal, and DMMA needs 8x fewer issue slots than DFMA.
//
// Complex arithmetic uses the 3M (Gauss) form on interleaved operands: the
// three real MMAs  Ar Br,  Ai Bi  and  (Ar + Ai)(Br + Bi)  give
// Re = p1 - p2  and  Im = p3 - p1 - p2  in the epilogue. A conjugated operand
// flips the sign of its imaginary part in the sums and of p2 (compile time).
// Conjugate-transposed operands are staged k-major so every fragment load
// stays conflict-free (strides = 4 mod 8 or 2 mod 8 in 16-byte units).
//
// The DMMA pipe is the bound (36.4-37.0 TFLOP/s from registers alone), so the
// design keeps it fed:
//  * CTA tile 32 x 32, four warps of 16 x 16, four CTAs per SM. The 64 x 64
//    tile of an earlier version (two CTAs, 254 registers) shared more operands
//    per load, but eight warps per SM left the pipe idle 17 % of the time, and
//    its few large tiles filled the last wave badly: 256^3 x 148 487 -> 468 us,
//    256^3 x 64 244 -> 208 us, 288^3 x 24 178 -> 119 us, 128^3 x 16 24 -> 12.5
//    us, 160^3 x 100 141 -> 84 us; with an addend 519 -> 478 us at 256^3 x 148.
//    64 x 32 and 32 x 64 tiles at three CTAs per SM and k-slices of 16 measured
//    the same or slower at every size. 84 % DMMA + 4 % for the sums in ncu.
//  * Per k-step of 4 the three passes p1, p2, p3 are issued back to back; the
//    real parts of the next step are loaded (8-byte loads) right after p1,
//    which frees their registers, the imaginary parts after p2, so a load has
//    a pass of MMAs to land. The stage barrier (cp.async, STAGES buffers of BK)
//    sits after p1 of a stage's last step: by then the stage has been read, so
//    its buffer is refilled at once.
//  * The epilogue works on the accumulator fragments: one store covers 128
//    contiguous bytes of a row (lanes tq), its transposed counterpart 128 bytes
//    of a column (lanes g), so the addends, the second output and the
//    conjugate-transposed second store are coalesced in either orientation
//    without a shared-memory tile.
//  * Warps whose 16 x 16 (or 16 x 8) part lies outside the matrix issue no
//    MMAs: a block of 200 costs 13 x 12.5 of them instead of 16 x 16.
#include "common.cuh"

namespace qtx {
namespace {

constexpr int THREADS = 128;    // 2 x 2 warps
constexpr int NT = 2;           // 16 x 8 fragments per warp, side by side
constexpr int WM = 16;          // rows and
constexpr int WN = 8 * NT;      // columns of a warp tile
constexpr int BM = 2 * WM;
constexpr int BN = 2 * WN;
constexpr int BK = 8;
constexpr int STAGES = 4;
constexpr int CTAS_PER_SM = 4;

// Shared-memory strides (complex elements).
constexpr int S_RK = BK + 4;  // [row][k] layouts: stride = 4 mod 8
template <int R>
constexpr int s_kr() {  // [k][row] layouts: stride = 2 mod 8
  return R + 2;
}
template <int R, bool RK>
constexpr int stage_elems() {
  return RK ? R * S_RK : BK * s_kr<R>();
}

__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem, bool pred) {
  const int bytes = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
// The barrier of the CTA, reached from main loops of different active size
// (each warp runs one of them).
__device__ __forceinline__ void cta_barrier() { asm volatile("bar.sync 0, %0;\n" ::"n"(THREADS) : "memory"); }

__device__ __forceinline__ double lds64(uint32_t addr) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(addr));
  return v;
}

// Copies BK-wide slices of one operand tile of R rows (M for op(A), N for
// op(B)) into the stages. RK: the global rows are the M / N index, k is
// contiguous ([row][k] in shared memory); otherwise the rows are the k index
// ([k][row]). Out-of-range elements are zero-filled.
template <int R, bool RK>
struct Loader {
  const z64* base;  // in range: the address of a zero-filled element
  const z64* p;     // this thread's element of the next slice
  int64_t ld;
  int rows, k;  // rows left from this thread's row; its k within a slice
  uint32_t off;

  __device__ __forceinline__ Loader(const z64* g, int64_t ld_, int total, int r0, int tid) {
    base = g;
    ld = ld_;
    if (RK) {
      const int r = tid / BK;
      k = tid % BK;
      rows = total - (r0 + r);
      p = g + (int64_t)(r0 + r) * ld + k;
      off = (uint32_t)(r * S_RK + k) * 16u;
    } else {
      const int r = tid % R;
      k = tid / R;
      rows = total - (r0 + r);
      p = g + (int64_t)k * ld + (r0 + r);
      off = (uint32_t)(k * s_kr<R>() + r) * 16u;
    }
  }
  // krem: k values left from the start of this slice.
  __device__ __forceinline__ void load(uint32_t sm, int krem) {
    constexpr int ITERS = R * BK / THREADS;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      if (RK) {
        constexpr int RS = THREADS / BK;
        const bool ok = it * RS < rows && k < krem;
        cp_async16(sm + off + it * RS * S_RK * 16, ok ? p + (int64_t)(it * RS) * ld : base, ok);
      } else {
        constexpr int KS = THREADS / R;
        const bool ok = 0 < rows && k + it * KS < krem;
        cp_async16(sm + off + it * KS * s_kr<R>() * 16, ok ? p + (int64_t)(it * KS) * ld : base, ok);
      }
    }
    p += RK ? BK : BK * ld;
  }
};

constexpr int kMaxGroup = 4;
struct KernelArgs {
  int count;
  GemmDesc d[kMaxGroup];
};

struct Acc {
  double p1[NT][4], p2[NT][4], p3[NT][4];
};

// All k-steps of a warp with NTA active fragments (0: it only copies and
// synchronises).
template <int OPA, int OPB, int NTA>
__device__ __forceinline__ void main_loop(Acc& acc, uint32_t as, uint32_t bs, uint32_t a_off, uint32_t b_off,
                                          Loader<BM, OPA == 0>& la, Loader<BN, OPB == 1>& lb, int K, int KT) {
  constexpr int A_BYTES = stage_elems<BM, OPA == 0>() * 16;
  constexpr int B_BYTES = stage_elems<BN, OPB == 1>() * 16;
  constexpr int NA = NTA > 0 ? NTA : 1;
  constexpr bool ON = NTA > 0;
  // byte offsets of a row of A / column of B and of a k
  constexpr int A_ROW = (OPA == 0 ? S_RK : 1) * 16, A_K = (OPA == 0 ? 1 : s_kr<BM>()) * 16;
  constexpr int B_ROW = (OPB == 1 ? S_RK : 1) * 16, B_K = (OPB == 1 ? 1 : s_kr<BN>()) * 16;
  double ar[2], ai[2], br[NA], bi[NA];
  auto load_re = [&](uint32_t a, uint32_t b, int kk) {
    ar[0] = lds64(a + (uint32_t)(kk * A_K));
    ar[1] = lds64(a + (uint32_t)(8 * A_ROW + kk * A_K));
#pragma unroll
    for (int j = 0; j < NTA; ++j) br[j] = lds64(b + (uint32_t)(j * 8 * B_ROW + kk * B_K));
  };
  auto load_im = [&](uint32_t a, uint32_t b, int kk) {
    ai[0] = lds64(a + (uint32_t)(kk * A_K + 8));
    ai[1] = lds64(a + (uint32_t)(8 * A_ROW + kk * A_K + 8));
#pragma unroll
    for (int j = 0; j < NTA; ++j) bi[j] = lds64(b + (uint32_t)(j * 8 * B_ROW + kk * B_K + 8));
  };
  cp_async_wait<STAGES - 1>();
  cta_barrier();
  uint32_t a_cur = as + a_off, b_cur = bs + b_off;
  if (ON) {
    load_re(a_cur, b_cur, 0);
    load_im(a_cur, b_cur, 0);
  }
  int st = 0, krem = K - STAGES * BK;
  for (int kt = 0; kt < KT; ++kt) {
#pragma unroll
    for (int h = 0; h < BK / 4; ++h) {
      const bool last = h == BK / 4 - 1;
      double sa[2], sb[NA];
      if (ON) {
#pragma unroll
        for (int q = 0; q < 2; ++q) sa[q] = OPA ? ar[q] - ai[q] : ar[q] + ai[q];
#pragma unroll
        for (int j = 0; j < NTA; ++j) sb[j] = OPB ? br[j] - bi[j] : br[j] + bi[j];
#pragma unroll
        for (int j = 0; j < NTA; ++j) mma_f64(acc.p1[j], ar[0], ar[1], br[j]);
      }
      uint32_t an = a_cur, bn = b_cur;
      if (last) {
        // This stage has been read by every warp once they all arrive; the
        // next one has landed.
        cp_async_wait<STAGES - 2>();
        cta_barrier();
        if (krem > 0) {
          la.load(as + st * A_BYTES, krem);
          lb.load(bs + st * B_BYTES, krem);
        }
        cp_async_commit();
        krem -= BK;
        st = st + 1 == STAGES ? 0 : st + 1;
        an = as + a_off + st * A_BYTES;
        bn = bs + b_off + st * B_BYTES;
      }
      const int kn = last ? 0 : 4 * (h + 1);
      if (ON) {
        load_re(an, bn, kn);
#pragma unroll
        for (int j = 0; j < NTA; ++j) mma_f64(acc.p2[j], ai[0], ai[1], bi[j]);
        load_im(an, bn, kn);
#pragma unroll
        for (int j = 0; j < NTA; ++j) mma_f64(acc.p3[j], sa[0], sa[1], sb[j]);
      }
      a_cur = an;
      b_cur = bn;
    }
  }
}

// Element (r, c) of op(X) of an addend, zero outside the matrix.
__device__ __forceinline__ z64 addend_at(const z64* p, int64_t rs, int64_t cs, double sg, bool ok, int r, int c) {
  const z64 x = ok ? p[r * rs + c * cs] : make_double2(0.0, 0.0);
  return make_double2(x.x, sg * x.y);
}

template <int OPA, int OPB>
__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) zgemm_kernel(const __grid_constant__ KernelArgs args) {
  constexpr int A_BYTES = stage_elems<BM, OPA == 0>() * 16;
  constexpr int B_BYTES = stage_elems<BN, OPB == 1>() * 16;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_begin();
  const uint32_t as = smem_u32(smem_raw);
  const uint32_t bs = as + STAGES * A_BYTES;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int g = lane >> 2;
  const int tq = lane & 3;
  const int m0 = blockIdx.y * BM;
  const int n0 = blockIdx.x * BN;
  const int M = args.d[0].M, N = args.d[0].N, K = args.d[0].K;
  const int KT = (K + BK - 1) / BK;
  const int64_t batch = args.d[0].batch;

  for (int64_t z = blockIdx.z; z < batch * args.count; z += gridDim.z) {
    const int set = args.count == 1 ? 0 : (int)(z / batch);
    const int64_t b = args.count == 1 ? z : z - set * batch;
    const GemmDesc& d = args.d[set];
    if (d.active != nullptr && d.active[b] == 0) continue;
    // Edge tiles leave their last warps idle: alternate which schedulers
    // host those.
    const int warp = (tid >> 5) ^ ((z & 1) ? 3 : 0);
    const int wm0 = (warp >> 1) * WM;
    const int wn0 = (warp & 1) * WN;
    const z64* Ag = d.a_ptrs ? d.a_ptrs[b] : at<const z64>(d.A, b);
    const z64* Bg = d.b_ptrs ? d.b_ptrs[b] : at<const z64>(d.B, b);

    Acc acc;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc.p1[j][q] = acc.p2[j][q] = acc.p3[j][q] = 0.0;
    if (KT > 0) {
      Loader<BM, OPA == 0> la(Ag, d.A.ld, M, m0, tid);
      Loader<BN, OPB == 1> lb(Bg, d.B.ld, N, n0, tid);
#pragma unroll
      for (int s = 0; s < STAGES; ++s) {
        if (s < KT) {
          la.load(as + s * A_BYTES, K - s * BK);
          lb.load(bs + s * B_BYTES, K - s * BK);
        }
        cp_async_commit();
      }
      const uint32_t a_off =
          OPA == 0 ? (uint32_t)((wm0 + g) * S_RK + tq) * 16u : (uint32_t)(tq * s_kr<BM>() + wm0 + g) * 16u;
      const uint32_t b_off =
          OPB == 1 ? (uint32_t)((wn0 + g) * S_RK + tq) * 16u : (uint32_t)(tq * s_kr<BN>() + wn0 + g) * 16u;
      const int cols = M > m0 + wm0 ? N - n0 - wn0 : 0;  // columns this warp has to compute
      if (cols > 8)
        main_loop<OPA, OPB, 2>(acc, as, bs, a_off, b_off, la, lb, K, KT);
      else if (cols > 0)
        main_loop<OPA, OPB, 1>(acc, as, bs, a_off, b_off, la, lb, K, KT);
      else
        main_loop<OPA, OPB, 0>(acc, as, bs, a_off, b_off, la, lb, K, KT);
      cp_async_wait<0>();
      if (gridDim.z < batch * args.count) cta_barrier();  // the stages serve the next entry
    }

    // Epilogue on the fragments: element (j, q) is row r0 + 8 (q / 2), column
    // c0 + 8 j + q % 2.
    const int r0 = m0 + wm0 + g, c0 = n0 + wn0 + 2 * tq;
    auto row = [&](int q) { return r0 + ((q >> 1) << 3); };
    auto col = [&](int j, int q) { return c0 + j * 8 + (q & 1); };
    auto inside = [&](int j, int q) { return row(q) < M && col(j, q) < N; };
    z64 v[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double x1 = acc.p1[j][q], x2 = acc.p2[j][q], x3 = acc.p3[j][q];
        v[j][q] = zmul(d.alpha, (OPA ^ OPB) ? make_double2(x1 + x2, x3 - (x1 - x2))
                                            : make_double2(x1 - x2, x3 - (x1 + x2)));
      }
    // Adds coef op(D) of addend t to w, all loads first.
    auto add = [&](int t, z64(&w)[NT][4]) {
      const Addend& ad = d.add[t];
      const z64* p = (t == 0 && d.d_ptrs) ? d.d_ptrs[b] : at<const z64>(ad.m, b);
      const int64_t rs = ad.conj_trans ? 1 : ad.m.ld, cs = ad.conj_trans ? ad.m.ld : 1;
      const double sg = ad.conj_trans ? -1.0 : 1.0;
      z64 x[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) x[j][q] = addend_at(p, rs, cs, sg, inside(j, q), row(q), col(j, q));
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[j][q] = zfma(ad.coef, x[j][q], w[j][q]);
    };
    for (int t = 0; t < d.nadd; ++t) add(t, v);
    if (!d.C3.null()) {
      z64 w[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[j][q] = zmul(d.scale3, v[j][q]);
      for (int t = d.nadd; t < d.nadd + d.nadd3; ++t) add(t, w);
      z64* out = at<z64>(d.C3, b);
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (inside(j, q)) out[(int64_t)row(q) * d.C3.ld + col(j, q)] = w[j][q];
    }
    if (!d.C.null()) {
      z64* out = d.c_ptrs ? d.c_ptrs[b] : at<z64>(d.C, b);
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (inside(j, q)) out[(int64_t)row(q) * d.C.ld + col(j, q)] = v[j][q];
    }
    if (!d.C2.null()) {
      z64* out = at<z64>(d.C2, b);
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (inside(j, q)) out[(int64_t)col(j, q) * d.C2.ld + row(q)] = zmul(d.coef2, zconj(v[j][q]));
    }
  }
}

template <int OPA, int OPB>
int launch(const KernelArgs& args, cudaStream_t s) {
  const GemmDesc& d = args.d[0];
  constexpr size_t smem =
      (size_t)STAGES * (stage_elems<BM, OPA == 0>() + stage_elems<BN, OPB == 1>()) * sizeof(z64);
  static_assert(smem <= 48 * 1024, "no opt-in of dynamic shared memory needed");
  const int64_t z = d.batch * args.count;
  dim3 grid((d.N + BN - 1) / BN, (d.M + BM - 1) / BM, (unsigned)(z < 65535 ? z : 65535));
  ProfScope prof(QTX_KERNEL_ZGEMM, 8.0 * d.M * d.N * (double)d.K * (double)z, s);
  return launch_chained(zgemm_kernel<OPA, OPB>, grid, dim3(THREADS), smem, s, 1, args);
}

bool aligned16(const MatRef& m) { return (reinterpret_cast<uintptr_t>(m.p) & 15u) == 0; }

}  // namespace

namespace {

// Checks one product and brings it into the form the kernel takes (zero
// operands and addends dropped). *skip: nothing to do.
int normalize(const GemmDesc& d, GemmDesc* out, bool* skip) {
  *skip = false;
  if (d.M <= 0 || d.N <= 0 || d.batch <= 0) {
    *skip = true;
    return QTX_OK;
  }
  if (d.K < 0 || d.nadd < 0 || d.nadd3 < 0 || d.nadd + d.nadd3 > kMaxAddends) {
    set_error("zgemm: invalid sizes or addend count");
    return QTX_ERR_ARG;
  }
  const bool grouped = d.a_ptrs || d.b_ptrs || d.c_ptrs || d.d_ptrs;
  if (grouped && (d.K <= 0 || !d.a_ptrs || !d.b_ptrs || !d.c_ptrs || d.nadd > 1 || d.nadd3 > 0 ||
                  (d.nadd == 1 && !d.d_ptrs) || !d.C2.null() || !d.C3.null())) {
    set_error("zgemm: the grouped form needs A, B and C tables, K > 0, at most one addend (with its table) "
              "and no second outputs");
    return QTX_ERR_ARG;
  }
  GemmDesc dd = d;
  if (!grouped && dd.K > 0 && (dd.A.null() || dd.B.null())) {
    // A zero operand: the product vanishes; only the addends remain.
    dd.K = 0;
    dd.A = dd.C.null() ? dd.C3 : dd.C;
    dd.B = dd.A;
  }
  if ((dd.K > 0 && (!aligned16(dd.A) || !aligned16(dd.B))) || !aligned16(dd.C) || !aligned16(dd.C2) ||
      !aligned16(dd.C3)) {
    set_error("zgemm: complex128 operands must be 16-byte aligned");
    return QTX_ERR_ARG;
  }
  for (int t = 0; !grouped && t < dd.nadd + dd.nadd3; ++t) {
    if (dd.add[t].m.null()) {  // drop zero addends
      for (int u = t; u + 1 < dd.nadd + dd.nadd3; ++u) dd.add[u] = dd.add[u + 1];
      if (t < dd.nadd)
        --dd.nadd;
      else
        --dd.nadd3;
      --t;
      if (dd.nadd + dd.nadd3 <= 0) break;
    }
  }
  if (dd.K == 0) {
    // Pure epilogue: the tile loop runs zero iterations.
    if (dd.A.null()) dd.A = dd.C.null() ? dd.C3 : dd.C;
    if (dd.B.null()) dd.B = dd.A;
  }
  *out = dd;
  return QTX_OK;
}

bool emulated(const GemmDesc& d, void** scr, size_t* bytes) {
  if (d.a_ptrs || d.K <= 0 || gemm_slices() <= 0 || !oz_supported(d.K, gemm_slices())) return false;
  *scr = oz_bound(bytes);
  return *scr != nullptr;
}

int dispatch(const KernelArgs& args, cudaStream_t s) {
  switch (args.d[0].opA * 2 + args.d[0].opB) {
    case 0: return launch<0, 0>(args, s);
    case 1: return launch<0, 1>(args, s);
    case 2: return launch<1, 0>(args, s);
    default: return launch<1, 1>(args, s);
  }
}

}  // namespace

int zgemm(const GemmDesc& d, cudaStream_t s) { return zgemm_many(&d, 1, s); }

// Consecutive products of the same sizes and operations share a launch: the
// lesser and greater products of a sweep and the independent products of a
// step fill the GPU together (a 64-block batch of 32 has 128 tiles a product)
// and pay one launch and one last wave instead of one each.
int zgemm_many(const GemmDesc* d, int count, cudaStream_t s) {
  KernelArgs args;
  args.count = 0;
  auto flush = [&]() {
    const int st = args.count > 0 ? dispatch(args, s) : (int)QTX_OK;
    args.count = 0;
    return st;
  };
  for (int k = 0; k < count; ++k) {
    GemmDesc dd;
    bool skip = false;
    QTX_TRY(normalize(d[k], &dd, &skip));
    if (skip) continue;
    void* scr = nullptr;
    size_t bytes = 0;
    if (emulated(dd, &scr, &bytes)) {
      QTX_TRY(flush());
      QTX_TRY(zgemm_oz(dd, gemm_slices(), scr, bytes, s));
      continue;
    }
    const GemmDesc& f = args.d[0];
    if (args.count == kMaxGroup ||
        (args.count > 0 && (dd.M != f.M || dd.N != f.N || dd.K != f.K || dd.batch != f.batch || dd.opA != f.opA ||
                            dd.opB != f.opB)))
      QTX_TRY(flush());
    args.d[args.count++] = dd;
  }
  return flush();
}

}  // namespace qtx
