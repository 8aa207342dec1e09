// Batched complex64 GEMM on the 5th-generation tensor cores (tcgen05, sm_100a)
// with split-TF32 products accumulated in FP32 (the mixed-precision path).
//
//   out = alpha op(A) op(B) + sum_t coef_t op_t(D_t)     (complex64 in / out)
//
// Each FP32 operand x is split into x_hi = tf32(x) and x_lo = tf32(x - x_hi);
// a real product is a_hi b_hi + a_hi b_lo + a_lo b_hi (the lo*lo term is
// below FP32 rounding). A complex product is the 4M combination of real
// products. op(B) is staged as the stack [-Bi; Br; Bi], so that with the
// accumulators [Re | Im] side by side Ar [Br | Bi] and Ai [-Bi | Br] are MMAs
// of N = 128: six tcgen05.mma.kind::tf32 per K step of 8, which read 48 KB of
// shared memory where twelve of N = 64 read 72 KB (576 of its cycles against
// 391 of the tensor pipe).
//
// CTA tile 128 x 64 (one UMMA M=128, N=128 real), K block 32 FP32 (128-byte
// rows, SWIZZLE_128B K-major), eight warps, one buffer of split planes (112 KB)
// so that two CTAs share an SM and one's prologue/epilogue overlaps the other's
// MMAs. While the tensor cores run the MMAs of block kb (issued by one
// thread), all warps load block kb+1 from global memory into registers, wait
// for the MMAs (tcgen05.commit -> mbarrier), then split and store the planes.
// Accumulators live in TMEM (Re in columns 0-63, Im in 64-127) and are read
// back with tcgen05.ld. The epilogue goes through a padded shared-memory tile
// so that global reads and writes are coalesced in either orientation:
// row-per-lane for conjugate-transposed addends and the transposed store,
// column-per-lane for everything else. Every mbarrier wait is bounded; on a
// time-out the CTA raises the error flag, skips its epilogue, frees its TMEM
// and returns.
#include "common.cuh"

namespace qtx {
namespace {

constexpr int TM = 128;       // UMMA M
constexpr int TN = 64;        // UMMA N
constexpr int TK = 32;        // fp32 elements per K block (128 B rows)
constexpr int THREADS = 256;  // eight warps
constexpr int PLANE_A = TM * TK * 4;  // bytes of one A plane (16 KB)
constexpr int PLANE_B = TN * TK * 4;  // bytes of one B plane (8 KB)
// op(A): re/im x hi/lo; op(B): the stack -im, re, im for hi and for lo.
constexpr int PLANES_BYTES = 4 * PLANE_A + 6 * PLANE_B;
constexpr int CTAS_PER_SM = 2;                               // one plane buffer each
constexpr int S_LD = TN + 1;                                 // padded epilogue tile row (float2)
constexpr int A_TASKS = TM * (TK / 4) / THREADS;             // 4 row-chunks of op(A) per thread
constexpr int B_TASKS = TN * (TK / 4) / THREADS;             // 2 row-chunks of op(B) per thread
constexpr int TMEM_COLS = 128;
constexpr long long kWaitLimit = 1ll << 26;  // bounded mbarrier polls

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ float tf32_trunc(float x) {
  return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
}

// Byte offset of the 16-byte chunk holding (row, k4-chunk) in a SWIZZLE_128B
// K-major tile: 8-row groups of 1024 B, chunk index XOR (row % 8).
__device__ __forceinline__ uint32_t sw128_offset(int row, int chunk) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

// UMMA shared-memory descriptor, K-major SWIZZLE_128B, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)(1) << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;     // stride byte offset: next 8-row group
  d |= (uint64_t)1 << 46;               // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;               // SWIZZLE_128B
  return d;
}

// Instruction descriptor: D f32, A/B tf32, K-major both, N = 128, M = 128.
__host__ __device__ constexpr uint32_t make_idesc() {
  return (1u << 4)                  // D format f32
         | (2u << 7)                // A tf32
         | (2u << 10)               // B tf32
         | ((uint32_t)((2 * TN) >> 3) << 17)
         | ((uint32_t)(TM >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity));
  return ok != 0;
}

// Bounded wait; returns false on time-out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (long long i = 0; i < kWaitLimit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
      smem_addr(bar)));
}

__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::);
}

struct Args {
  int M, N, K;
  int64_t batch;
  MatRef A, B;
  int opA, opB;
  float2 alpha;
  struct Add {
    MatRef m;
    float2 coef;
    int ct;
  } add[kMaxAddends];
  int nadd, nadd3;
  MatRef C, C2, C3;
  float2 coef2, scale3;
  int* err;
};

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

struct Regs {
  float2 a[A_TASKS][4];
  float2 b[B_TASKS][4];
};

// Task t of op(A): (row, chunk of 4 k). Lanes walk the memory-contiguous index.
template <int OPA>
__device__ __forceinline__ void a_task(int t, int& row, int& chunk) {
  if (OPA == 0) {
    row = t >> 3;
    chunk = t & 7;
  } else {
    row = t & (TM - 1);
    chunk = t >> 7;
  }
}
template <int OPB>
__device__ __forceinline__ void b_task(int t, int& row, int& chunk) {
  if (OPB == 1) {
    row = t >> 3;
    chunk = t & 7;
  } else {
    row = t & (TN - 1);
    chunk = t >> 6;
  }
}

// A K-contiguous operand with VEC (16-byte aligned, even leading dimension) is
// read two complex numbers per load, pair t of (row, pair of k): 16 lanes read a
// row's 256 bytes of the K block. Four k per thread in two such loads, a gap of
// 16 bytes between lanes, took 16 wavefronts a load instead of 4, and the L1 /
// shared data pipe is what bounds this kernel (loads and stores 154 k wavefronts
// and the MMAs' operand reads 98 k in 253 k cycles; tensor pipe 39 %): 148
// products of 256^3 NN 148 -> 134 us, NT 157 -> 144 us. With op(A) in TMEM,
// which spares the pipe those stores and reads, the chain of fetch, split and
// MMA bounds it instead: 140 and 149 us (143 and 169 us with two K blocks of 16
// in flight).
__device__ __forceinline__ void pair_task(int t, int& row, int& pair) {
  row = t >> 4;
  pair = t & 15;
}

// Pair `pair` of k of row gr (rows of X are K-contiguous); zeros outside.
__device__ __forceinline__ float4 load_pair(const c32* X, int64_t ld, int gr, int rows, int gk, int K) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (gr < rows && gk + 1 < K) {
    v = *reinterpret_cast<const float4*>(X + (int64_t)gr * ld + gk);
  } else if (gr < rows && gk < K) {
    const float2 w = X[(int64_t)gr * ld + gk];
    v = make_float4(w.x, w.y, 0.f, 0.f);
  }
  return v;
}

// Global -> registers for one K block (all loads issued back to back).
template <int OPA, int OPB, bool VEC>
__device__ __forceinline__ void load_regs(const Args& a, const c32* Ag, const c32* Bg, Regs& R, int m0,
                                          int n0, int k0, int tid) {
  if (OPA == 0 && VEC) {
#pragma unroll
    for (int i = 0; i < 2 * A_TASKS; ++i) {
      int row, pair;
      pair_task(tid + i * THREADS, row, pair);
      const float4 v = load_pair(Ag, a.A.ld, m0 + row, a.M, k0 + 2 * pair, a.K);
      R.a[i >> 1][(i & 1) * 2] = make_float2(v.x, v.y);
      R.a[i >> 1][(i & 1) * 2 + 1] = make_float2(v.z, v.w);
    }
  } else {
#pragma unroll
    for (int i = 0; i < A_TASKS; ++i) {
      int row, chunk;
      a_task<OPA>(tid + i * THREADS, row, chunk);
      const int gr = m0 + row;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gk = k0 + chunk * 4 + e;
        float2 v = make_float2(0.f, 0.f);
        if (gr < a.M && gk < a.K) {
          if (OPA == 0) {
            v = Ag[(int64_t)gr * a.A.ld + gk];
          } else {
            v = Ag[(int64_t)gk * a.A.ld + gr];
            v.y = -v.y;
          }
        }
        R.a[i][e] = v;
      }
    }
  }
  if (OPB == 1 && VEC) {
#pragma unroll
    for (int i = 0; i < 2 * B_TASKS; ++i) {
      int row, pair;
      pair_task(tid + i * THREADS, row, pair);
      const float4 v = load_pair(Bg, a.B.ld, n0 + row, a.N, k0 + 2 * pair, a.K);
      R.b[i >> 1][(i & 1) * 2] = make_float2(v.x, -v.y);
      R.b[i >> 1][(i & 1) * 2 + 1] = make_float2(v.z, -v.w);
    }
  } else {
#pragma unroll
    for (int i = 0; i < B_TASKS; ++i) {
      int row, chunk;
      b_task<OPB>(tid + i * THREADS, row, chunk);
      const int gn = n0 + row;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gk = k0 + chunk * 4 + e;
        float2 v = make_float2(0.f, 0.f);
        if (gn < a.N && gk < a.K) {
          if (OPB == 0) {
            v = Bg[(int64_t)gk * a.B.ld + gn];
          } else {
            v = Bg[(int64_t)gn * a.B.ld + gk];
            v.y = -v.y;
          }
        }
        R.b[i][e] = v;
      }
    }
  }
}

__device__ __forceinline__ void split4(const float2 (&v)[4], float4& hr, float4& lr, float4& hi, float4& li) {
  float* phr = &hr.x;
  float* plr = &lr.x;
  float* phi = &hi.x;
  float* pli = &li.x;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float rh = tf32_trunc(v[e].x), ih = tf32_trunc(v[e].y);
    phr[e] = rh;
    plr[e] = tf32_trunc(v[e].x - rh);
    phi[e] = ih;
    pli[e] = tf32_trunc(v[e].y - ih);
  }
}

__device__ __forceinline__ float4 neg4(float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); }

// hi and lo of two values.
__device__ __forceinline__ void split2(float x, float y, float2& h, float2& l) {
  h = make_float2(tf32_trunc(x), tf32_trunc(y));
  l = make_float2(tf32_trunc(x - h.x), tf32_trunc(y - h.y));
}

__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }

// Registers -> the split planes (SWIZZLE_128B K-major).
template <int OPA, int OPB, bool VEC>
__device__ __forceinline__ void store_planes(const Regs& R, uint8_t* planes, int tid) {
  uint8_t* pb = planes + 4 * PLANE_A;
  if (OPA == 0 && VEC) {
#pragma unroll
    for (int i = 0; i < 2 * A_TASKS; ++i) {
      int row, pair;
      pair_task(tid + i * THREADS, row, pair);
      const float2 u = R.a[i >> 1][(i & 1) * 2], v = R.a[i >> 1][(i & 1) * 2 + 1];
      float2 hr, lr, hi, li;
      split2(u.x, v.x, hr, lr);
      split2(u.y, v.y, hi, li);
      const uint32_t off = sw128_offset(row, pair >> 1) + 8 * (pair & 1);
      *reinterpret_cast<float2*>(planes + off) = hr;
      *reinterpret_cast<float2*>(planes + PLANE_A + off) = lr;
      *reinterpret_cast<float2*>(planes + 2 * PLANE_A + off) = hi;
      *reinterpret_cast<float2*>(planes + 3 * PLANE_A + off) = li;
    }
  } else {
#pragma unroll
    for (int i = 0; i < A_TASKS; ++i) {
      int row, chunk;
      a_task<OPA>(tid + i * THREADS, row, chunk);
      float4 hr, lr, hi, li;
      split4(R.a[i], hr, lr, hi, li);
      const uint32_t off = sw128_offset(row, chunk);
      *reinterpret_cast<float4*>(planes + off) = hr;
      *reinterpret_cast<float4*>(planes + PLANE_A + off) = lr;
      *reinterpret_cast<float4*>(planes + 2 * PLANE_A + off) = hi;
      *reinterpret_cast<float4*>(planes + 3 * PLANE_A + off) = li;
    }
  }
  if (OPB == 1 && VEC) {
#pragma unroll
    for (int i = 0; i < 2 * B_TASKS; ++i) {
      int row, pair;
      pair_task(tid + i * THREADS, row, pair);
      const float2 u = R.b[i >> 1][(i & 1) * 2], v = R.b[i >> 1][(i & 1) * 2 + 1];
      float2 hr, lr, hi, li;
      split2(u.x, v.x, hr, lr);
      split2(u.y, v.y, hi, li);
      const uint32_t off = sw128_offset(row, pair >> 1) + 8 * (pair & 1);
      *reinterpret_cast<float2*>(pb + off) = neg2(hi);
      *reinterpret_cast<float2*>(pb + PLANE_B + off) = hr;
      *reinterpret_cast<float2*>(pb + 2 * PLANE_B + off) = hi;
      *reinterpret_cast<float2*>(pb + 3 * PLANE_B + off) = neg2(li);
      *reinterpret_cast<float2*>(pb + 4 * PLANE_B + off) = lr;
      *reinterpret_cast<float2*>(pb + 5 * PLANE_B + off) = li;
    }
  } else {
#pragma unroll
    for (int i = 0; i < B_TASKS; ++i) {
      int row, chunk;
      b_task<OPB>(tid + i * THREADS, row, chunk);
      float4 hr, lr, hi, li;
      split4(R.b[i], hr, lr, hi, li);
      const uint32_t off = sw128_offset(row, chunk);
      *reinterpret_cast<float4*>(pb + off) = neg4(hi);
      *reinterpret_cast<float4*>(pb + PLANE_B + off) = hr;
      *reinterpret_cast<float4*>(pb + 2 * PLANE_B + off) = hi;
      *reinterpret_cast<float4*>(pb + 3 * PLANE_B + off) = neg4(li);
      *reinterpret_cast<float4*>(pb + 4 * PLANE_B + off) = lr;
      *reinterpret_cast<float4*>(pb + 5 * PLANE_B + off) = li;
    }
  }
}

// The six MMAs of one K step (8 fp32), each over the 128 accumulator columns
// [Re | Im]: += Ar [Br | Bi] and += Ai [-Bi | Br], small terms first.
__device__ __forceinline__ void issue_kstep(uint32_t tmem, uint32_t sa, uint32_t sb, int kk,
                                            bool first) {
  const uint32_t koff = (uint32_t)kk * 32;  // bytes along the 128-byte row
  const uint64_t arh = make_desc(sa + 0 * PLANE_A + koff), arl = make_desc(sa + 1 * PLANE_A + koff);
  const uint64_t aih = make_desc(sa + 2 * PLANE_A + koff), ail = make_desc(sa + 3 * PLANE_A + koff);
  const uint64_t bih = make_desc(sb + 0 * PLANE_B + koff), brh = make_desc(sb + 1 * PLANE_B + koff);
  const uint64_t bil = make_desc(sb + 3 * PLANE_B + koff), brl = make_desc(sb + 4 * PLANE_B + koff);
  constexpr uint32_t ID = make_idesc();
  mma_tf32(tmem, arl, brh, ID, first ? 0u : 1u);
  mma_tf32(tmem, arh, brl, ID, 1u);
  mma_tf32(tmem, arh, brh, ID, 1u);
  mma_tf32(tmem, ail, bih, ID, 1u);
  mma_tf32(tmem, aih, bil, ID, 1u);
  mma_tf32(tmem, aih, bih, ID, 1u);
}

constexpr int PA = 8;  // accumulator columns per epilogue step

// Eight accumulator columns of this lane's row.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&v)[PA]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}

constexpr int kMaxGroup = 4;
struct GroupArgs {
  int count;
  Args a[kMaxGroup];
};

template <int OPA, int OPB, bool VEC>
__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) cgemm_tc_kernel(const __grid_constant__ GroupArgs ga) {
  // 1024-byte alignment for the SWIZZLE_128B atoms.
  extern __shared__ __align__(1024) uint8_t smem[];
  chain_begin();
  uint8_t* planes = smem;
  float2* tile = reinterpret_cast<float2*>(smem);  // epilogue tile [TM][S_LD], reuses the planes
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + PLANES_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int m0 = blockIdx.y * TM;
  const int n0 = blockIdx.x * TN;
  const int64_t batch = ga.a[0].batch;
  const int KB = (ga.a[0].K + TK - 1) / TK;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  bool ok = true;
  Regs R;

  for (int64_t z = blockIdx.z; z < batch * ga.count && ok; z += gridDim.z) {
    const int set = (int)(z / batch);
    const int64_t b = z - set * batch;
    const Args& a = ga.a[set];
    const c32* Ag = at<const c32>(a.A, b);
    const c32* Bg = at<const c32>(a.B, b);
    if (KB > 0) {
      load_regs<OPA, OPB, VEC>(a, Ag, Bg, R, m0, n0, 0, tid);
      store_planes<OPA, OPB, VEC>(R, planes, tid);
      fence_async_smem();
      __syncthreads();
    }
    for (int kb = 0; kb < KB; ++kb) {
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        const uint32_t sa = smem_addr(planes);
        const uint32_t sb = sa + 4 * PLANE_A;
#pragma unroll
        for (int kk = 0; kk < TK / 8; ++kk) issue_kstep(tmem, sa, sb, kk, kb == 0 && kk == 0);
        mma_commit(bar);
      }
      const bool more = kb + 1 < KB;
      if (more) load_regs<OPA, OPB, VEC>(a, Ag, Bg, R, m0, n0, (kb + 1) * TK, tid);
      // One thread polls the MMA-completion barrier; the others wait at the
      // block barrier instead of spinning on shared memory.
      if (tid == 0 && !mbar_wait(bar, phase)) ok = false;
      phase ^= 1u;
      ok = __syncthreads_and(ok);
      if (more && ok) {
        store_planes<OPA, OPB, VEC>(R, planes, tid);
        fence_async_smem();
      }
      if (!__syncthreads_and(ok)) {
        ok = false;
        break;
      }
    }
    if (!ok) break;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);

    // Phase A (warps 0-3 and 4-7 split the columns; lane = tile row, the
    // TMEM lane quarter of warp w is w % 4): alpha * acc + ct addends -> tile.
    {
      const int wl = warp & 3;
      const int rl = wl * 32 + lane;
      const int r = m0 + rl;
      const uint32_t lane_base = tmem + ((uint32_t)(wl * 32) << 16);
      const int cbeg = (warp >> 2) * (TN / 2);
#pragma unroll 1
      for (int c0 = cbeg; c0 < cbeg + TN / 2; c0 += PA) {
        uint32_t vr[PA], vi[PA];
        if (KB > 0) {
          tmem_ld8(lane_base + (uint32_t)c0, vr);
          tmem_ld8(lane_base + (uint32_t)(TN + c0), vi);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
        } else {
#pragma unroll
          for (int j = 0; j < PA; ++j) vr[j] = vi[j] = 0u;
        }
        float2 v[PA];
#pragma unroll
        for (int j = 0; j < PA; ++j)
          v[j] = cmulf(a.alpha, make_float2(__uint_as_float(vr[j]), __uint_as_float(vi[j])));
        for (int t = 0; t < a.nadd; ++t) {
          const auto& ad = a.add[t];
          if (!ad.ct) continue;
          const c32* p = at<const c32>(ad.m, b) + (int64_t)(n0 + c0) * ad.m.ld + r;
          float2 x[PA];  // all loads first
#pragma unroll
          for (int j = 0; j < PA; ++j)
            x[j] = (r < a.M && n0 + c0 + j < a.N) ? p[(int64_t)j * ad.m.ld] : make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < PA; ++j) {
            const float2 y = cmulf(ad.coef, make_float2(x[j].x, -x[j].y));
            v[j].x += y.x;
            v[j].y += y.y;
          }
        }
#pragma unroll
        for (int j = 0; j < PA; ++j) tile[rl * S_LD + c0 + j] = v[j];
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();

    // Phase B (a warp takes four rows at a time, lane = tile column and
    // column + 32): the addends read row-wise, C3 and C. All loads of an
    // addend are issued before their use: one element at a time (as before)
    // exposed a memory latency per element and addend, 180 us for an NT product
    // of 64 x 256^3 with addends against 104 us without.
    constexpr int PB = 4;
#pragma unroll 1
    for (int rb = warp * PB; rb < TM; rb += (THREADS / 32) * PB) {
      if (m0 + rb >= a.M) break;
      float2 v[PB][2];
      auto inside = [&](int k, int h) { return m0 + rb + k < a.M && n0 + lane + 32 * h < a.N; };
      auto add_rows = [&](int t, float2(&w)[PB][2]) {
        const auto& ad = a.add[t];
        const int64_t rs = ad.ct ? 1 : ad.m.ld, cs = ad.ct ? ad.m.ld : 1;
        const c32* p = at<const c32>(ad.m, b) + (m0 + rb) * rs + (n0 + lane) * cs;
        float2 x[PB][2];
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            x[k][h] = inside(k, h) ? p[k * rs + 32 * h * cs] : make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 y = cmulf(ad.coef, make_float2(x[k][h].x, ad.ct ? -x[k][h].y : x[k][h].y));
            w[k][h].x += y.x;
            w[k][h].y += y.y;
          }
      };
#pragma unroll
      for (int k = 0; k < PB; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) v[k][h] = tile[(rb + k) * S_LD + lane + 32 * h];
      for (int t = 0; t < a.nadd; ++t)
        if (!a.add[t].ct) add_rows(t, v);
      if (!a.C3.null()) {
        float2 w[PB][2];
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h) w[k][h] = cmulf(a.scale3, v[k][h]);
        for (int t = a.nadd; t < a.nadd + a.nadd3; ++t) add_rows(t, w);
        c32* out = at<c32>(a.C3, b) + (int64_t)(m0 + rb) * a.C3.ld + n0 + lane;
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (inside(k, h)) out[(int64_t)k * a.C3.ld + 32 * h] = w[k][h];
      }
      if (!a.C.null()) {
        c32* out = at<c32>(a.C, b) + (int64_t)(m0 + rb) * a.C.ld + n0 + lane;
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (inside(k, h)) out[(int64_t)k * a.C.ld + 32 * h] = v[k][h];
      }
      if (!a.C2.null()) {
#pragma unroll
        for (int k = 0; k < PB; ++k)
#pragma unroll
          for (int h = 0; h < 2; ++h) tile[(rb + k) * S_LD + lane + 32 * h] = v[k][h];
      }
    }

    // Phase C (lane = tile row): the conjugate-transposed store C2.
    if (!a.C2.null()) {
      __syncthreads();
      c32* out = at<c32>(a.C2, b);
#pragma unroll 8
      for (int e = tid; e < TM * TN; e += THREADS) {
        const int rl = e % TM, cl = e / TM;
        const int r = m0 + rl, c = n0 + cl;
        if (r >= a.M || c >= a.N) continue;
        const float2 v = tile[rl * S_LD + cl];
        out[(int64_t)c * a.C2.ld + r] = cmulf(a.coef2, make_float2(v.x, -v.y));
      }
    }
    __syncthreads();
  }
  if (!ok && tid == 0 && ga.a[0].err != nullptr) atomicExch(ga.a[0].err, 1);
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
}

template <int OPA, int OPB, bool VEC>
int launch_v(const GroupArgs& ga, cudaStream_t s) {
  static_assert(TM * S_LD * (int)sizeof(float2) <= PLANES_BYTES, "epilogue tile must fit the planes");
  const Args& a = ga.a[0];
  const size_t smem = (size_t)PLANES_BYTES + 64;
  QTX_CHECK_CUDA(cudaFuncSetAttribute(cgemm_tc_kernel<OPA, OPB, VEC>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t z = a.batch * ga.count;
  dim3 grid((a.N + TN - 1) / TN, (a.M + TM - 1) / TM, (unsigned)(z < 65535 ? z : 65535));
  ProfScope prof(QTX_KERNEL_CGEMM, 8.0 * a.M * a.N * (double)a.K * (double)z, s);
  return launch_chained(cgemm_tc_kernel<OPA, OPB, VEC>, grid, dim3(THREADS), smem, s, 1, ga);
}

bool vec_ok(const MatRef& m) {
  return (reinterpret_cast<uintptr_t>(m.p) & 15u) == 0 && (m.ld % 2) == 0 && (m.stride % 2) == 0;
}

template <int OPA, int OPB>
int launch(const GroupArgs& ga, cudaStream_t s) {
  // The 16-byte path reads the K-contiguous operands; all must allow it.
  bool vec = true;
  for (int k = 0; k < ga.count; ++k)
    vec = vec && (OPA != 0 || vec_ok(ga.a[k].A)) && (OPB != 1 || vec_ok(ga.a[k].B));
  if (vec) return launch_v<OPA, OPB, true>(ga, s);
  return launch_v<OPA, OPB, false>(ga, s);
}

int dispatch(const GroupArgs& ga, int op, cudaStream_t s) {
  switch (op) {
    case 0: return launch<0, 0>(ga, s);
    case 1: return launch<0, 1>(ga, s);
    case 2: return launch<1, 0>(ga, s);
    default: return launch<1, 1>(ga, s);
  }
}

}  // namespace

int cgemm_tc(const CGemmDesc& d, cudaStream_t s) { return cgemm_tc_many(&d, 1, s); }

// As zgemm_many: consecutive products of one shape share a launch.
int cgemm_tc_many(const CGemmDesc* list, int count, cudaStream_t s) {
  GroupArgs ga;
  ga.count = 0;
  int op = 0;
  auto flush = [&]() {
    const int st = ga.count > 0 ? dispatch(ga, op, s) : (int)QTX_OK;
    ga.count = 0;
    return st;
  };
  for (int i = 0; i < count; ++i) {
    const CGemmDesc& d = list[i];
    if (d.M <= 0 || d.N <= 0 || d.batch <= 0) continue;
    if (d.nadd < 0 || d.nadd3 < 0 || d.nadd + d.nadd3 > kMaxAddends ||
        (d.K > 0 && (d.A.null() || d.B.null())) || (d.C.null() && d.C3.null())) {
      set_error("cgemm_tc: invalid arguments (null operand or output, or too many addends)");
      return QTX_ERR_ARG;
    }
    const Args& f = ga.a[0];
    if (ga.count == kMaxGroup ||
        (ga.count > 0 && (d.M != f.M || d.N != f.N || d.K != f.K || d.batch != f.batch || d.err != f.err ||
                          d.opA * 2 + d.opB != op)))
      QTX_TRY(flush());
    op = d.opA * 2 + d.opB;
    Args a{};
    a.M = d.M;
    a.N = d.N;
    a.K = d.K;
    a.batch = d.batch;
    a.A = d.A;
    a.B = d.B;
    a.opA = d.opA;
    a.opB = d.opB;
    a.alpha = d.alpha;
    for (int t = 0; t < d.nadd + d.nadd3; ++t) {
      if (d.add[t].m.null()) continue;
      const int k = a.nadd + a.nadd3;
      a.add[k].m = d.add[t].m;
      a.add[k].coef = d.add[t].coef;
      a.add[k].ct = d.add[t].conj_trans;
      if (t < d.nadd)
        ++a.nadd;
      else
        ++a.nadd3;
    }
    a.C = d.C;
    a.C2 = d.C2;
    a.C3 = d.C3;
    a.coef2 = d.coef2;
    a.scale3 = d.scale3;
    a.err = d.err;
    ga.a[ga.count++] = a;
  }
  return flush();
}

}  // namespace qtx
