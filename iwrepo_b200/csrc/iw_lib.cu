// B200 time step of the stratified Boussinesq solver (Fourier x,y /
// Legendre multidomain penalty z) and its C ABI (include/iw_b200.h).
//
// One step (main.f:653-1066) on device-resident fields:
//   K_A  k_stageA_t    maxcalc/convec round-trip projection, w mean = 0, z-derivatives of
//                      u, v, w on the FP64 tensor cores (k_stageA_r, k_stageA: FMA pipes)  (z columns)
//   K_B  k_yfft        y-inverse of u,v,w,rho, dz(u,v,w), and i ky (u,v,w)      (planes)
//   K_C  k_xrow_reg    x-inverse of 13 rows -> skew-symmetric products, buoyancy, upwind
//                      interface penalty, paddle -> x-forward with i kx folded in
//                      (k_xrow_nl: lengths it does not cover)                   (rows)
//   K_D  k_yfft        y-forward with i ky folded in                            (planes)
//        k_wviscrot    rotational viscous pressure BC, beside K_B..K_D          (walls)
//   K_E  k_stageE_t    S = B + dz(Z), SS extrapolation, BDF u*, history, Fourier x Legendre
//                      filter on the FP64 tensor cores (k_stageE_r, k_stageE_f32, k_stageE:
//                      FMA pipes)                                               (z columns)
//   K_F  k_press_tc    pressure Poisson (divergence, solve, filter, projection), with the
//                      refined columns in k_solve_cta beside it
//        k_solve_tc    u,v / w / rho Helmholtz solves, filters, mean mode, one launch
//                      (other variants: k_solve_sys, k_solve_sys2, k_solve_cta; k_press_g /
//                      k_visc with the band LU when the handle asks for the reference's LU)
//   K_H  interface averaging: planes next to interfaces go to physical space,
//        the averaging change comes back; every plane gets the spectral effect
//        of the round trip.
// Around the step (iw_restart.inl, iw_output.inl, iw_postp.inl): the adaptive
// time step's CFL numbers (k_xrow_stats), restart files, field and animation
// dumps, Legendre spectra (k_speclegen) and the TKE budget (k_row_dot,
// k_sub_rowmean), written by a host thread from pinned buffers.
// The penalty systems (penalty.f + band_lu.f) are assembled on the device
// (k_build_systems, k_assemble_band) when epsilon changes (steps 1-3 and a dt change), one per distinct
// kx^2+ky^2 and system type, then factored (band LU) or turned into block
// inverses of their distinct subdomain blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "../../include/iw_b200.h"
#include "iw_fft.cuh"
#include "iw_layout.h"
#include "iw_kernels.cuh"

using namespace iw;

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
static thread_local std::string g_err;
static thread_local int g_status = 0;
static int set_err(int code, const std::string& msg) {
  g_err = msg;
  g_status = code;
  return code;
}
#define CK(x)                                                                            \
  do {                                                                                   \
    cudaError_t e_ = (x);                                                                \
    if (e_ != cudaSuccess) {                                                             \
      cudaGetLastError(); /* reported here: no later check finds it again */             \
      return set_err(IW_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));      \
    }                                                                                    \
  } while (0)

// Launch errors.  A successful cudaFuncSetAttribute resets the runtime's record of a launch that failed
// before it, so both go through set_smem, which keeps the first error of the thread until it is asked for.
namespace iw {
inline thread_local cudaError_t g_launch_error = cudaSuccess;
}
static inline void keep_launch_error(cudaError_t e) {  // (an event that is not ready yet is no error)
  if (e != cudaSuccess && e != cudaErrorNotReady && g_launch_error == cudaSuccess) g_launch_error = e;
}
// Dynamic shared memory that launches of the kernel may ask for.  The limit is the kernel's, not the caller's: it only
// grows, so that no thread lowers it between another thread's call and its launch.
struct SmemLimits {
  std::mutex mu;
  std::unordered_map<const void*, size_t> set;
};
inline SmemLimits& smem_limits() {
  static SmemLimits l;
  return l;
}
template <typename K>
static inline void set_smem(K* kernel, size_t bytes) {
  keep_launch_error(cudaGetLastError());
  SmemLimits& l = smem_limits();
  std::lock_guard<std::mutex> lk(l.mu);
  size_t& have = l.set[(const void*)kernel];
  const size_t want = std::max(have, bytes);
  const cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
  if (e == cudaSuccess)
    have = want;
  else
    cudaGetLastError();
  keep_launch_error(e);
}
static inline cudaError_t launch_error() {
  keep_launch_error(cudaGetLastError());
  const cudaError_t e = g_launch_error;
  g_launch_error = cudaSuccess;
  return e;
}

// ---------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }

// (re, im) pair of one complex value stored as two T
template <typename T>
struct Pair;
template <>
struct Pair<float> {
  typedef float2 t;
};
template <>
struct Pair<double> {
  typedef double2 t;
};

// ===========================================================================
// K_A: round-trip projection + w(1,1,:)=0 + z derivatives.
// Thread per (real x index i, y index j, subdomain ks, field q).
// Inputs F (spectral state n); outputs F1 = P(F) (w mean zeroed) and dz(F1).
// P is the exact effect of horfft(+1) followed by horfft(-1) (maxcalc,
// various.f:726-729,848-851): the kx=0 column becomes Hermitian in ky, the
// x-Nyquist column keeps its real part divided by ny, all else is unchanged.
// ===========================================================================
template <typename T>
__device__ __forceinline__ T proj_val(const Geo& g, const T* __restrict__ f, int i, int j, int k) {
  if (i < 2) {
    int jp = (g.ny - j) % g.ny;
    T a = f[fidx<T>(g, i, j, k)];
    T b = f[fidx<T>(g, i, jp, k)];
    return i == 0 ? (T)0.5 * (a + b) : (T)0.5 * (a - b);
  }
  if (i >= g.nx) {
    return i == g.nx ? f[fidx<T>(g, i, j, k)] * (T)g.scaley : (T)0;
  }
  return f[fidx<T>(g, i, j, k)];
}

// Roundings written out (no contraction left to the compiler): the tiled and
// register-column stage A give the same bits whatever their loop structure.
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_t(double a, double b) { return __dmul_rn(a, b); }

// Asynchronous bulk copies into shared memory, completed on an mbarrier;
// every wait is bounded by the global timer.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// global -> shared bulk copy (16-byte aligned addresses, size a multiple of 16)
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// wait for phase `ph` of an mbarrier, for at most `limit_ns`; false if it gave up
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t ph, uint64_t limit_ns) {
  const uint64_t t0 = global_ns();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(ph)
        : "memory");
    if (ok) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
}

// Tiled z-column kernels: a block owns 32 consecutive real x indices of one
// (y index, subdomain) and keeps the N x 32 tile in shared memory; the N x N
// operators (D, filter) are applied with compact loops over the tile.
constexpr int kTX = 32;   // x points per tile (one warp wide)
constexpr int kTW = 8;    // warps per block

template <typename T>
__global__ void __launch_bounds__(kTX* kTW) k_stageA(Geo g, const T* __restrict__ F0, const T* __restrict__ F1_,
                                                     const T* __restrict__ F2_, const T* __restrict__ F3_,
                                                     T* __restrict__ O0, T* __restrict__ O1, T* __restrict__ O2,
                                                     T* __restrict__ O3, T* __restrict__ Z0, T* __restrict__ Z1,
                                                     T* __restrict__ Z2, T* __restrict__ Z3, int proj,
                                                     int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = g.N;
  T* sD = (T*)smraw;             // N*N
  T* tile = sD + N * N;          // N*kTX
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) sD[t] = (T)g.D[t];
  const int q = blockIdx.z;
  const T* F = q == 0 ? F0 : q == 1 ? F1_ : q == 2 ? F2_ : F3_;
  T* O = q == 0 ? O0 : q == 1 ? O1 : q == 2 ? O2 : O3;
  T* Z = q == 0 ? Z0 : q == 1 ? Z1 : q == 2 ? Z2 : Z3;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * kTX + lane;
  const int j = blockIdx.y % g.ny, ks = blockIdx.y / g.ny;
  const bool act = i < g.nxpp;
  for (int k = w; k < N; k += kTW) {
    const int kk = ks * N + k;
    T x = 0;
    if (act) {
      x = proj ? proj_val<T>(g, F, i, j, kk) : F[fidx<T>(g, i, j, kk)];
      if (!isfinite(x)) err[0] = 1;  // the state of the last step holds a NaN or Inf
      if (q == 2 && j == 0 && i < 2) x = (T)0;  // wc(1,1,:) = 0, solver.f:66-69
      O[fidx<T>(g, i, j, kk)] = x;
    }
    tile[k * kTX + lane] = x;
  }
  __syncthreads();
  if (!act || Z == nullptr) return;
  const T fac = (T)g.hfac[ks];
  for (int k1 = w; k1 < N; k1 += kTW) {
    const T* dr = sD + k1 * N;
    T s = 0;
#pragma unroll 4
    for (int k2 = 0; k2 < N; ++k2) s = fma_t(dr[k2], tile[k2 * kTX + lane], s);
    Z[fidx<T>(g, i, j, ks * N + k1)] = mul_t(s, fac);
  }
}

// ===========================================================================
// y transforms (CFFT99 semantics, horfft.f:21-30,51-57): LOT = nx/2 columns,
// the x-Nyquist column is never transformed; forward is scaled by 1/ny (the
// Nyquist column too).  One CTA per (plane, tile of TX kx columns, job).
// Job modes:
//   0 inverse:  dst = Yinv(src)
//   1 inverse:  dst = Yinv(i ky src)
//   2 forward:  dst = Yfwd(src)/ny
//   3 forward:  dst = Yfwd(src)/ny + i ky Yfwd(src2)/ny
// ===========================================================================
template <typename T>
struct YJob {
  const T* src;
  const T* src2;
  T* dst;
  int mode;
};
template <typename T>
struct YJobs {
  YJob<T> j[16];
};

// ny = 1: every transform is the identity (ky = 0, scale 1)
template <typename T>
__global__ void __launch_bounds__(256) k_y1(YJobs<T> jobs, size_t nc) {
  typedef typename cplx_t<T>::type C;
  const YJob<T> jb = jobs.j[blockIdx.y];
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nc && (jb.mode == 1 || jb.src != jb.dst)) ((C*)jb.dst)[e] = jb.mode == 1 ? cmk<C>(0, 0) : ((const C*)jb.src)[e];
}

// slots per padded y column: >= fpadlen(ny) and = 2 (mod 16), so that the
// TX columns of a tile sit in different banks
__host__ __device__ __forceinline__ int ystride(int ny) {
  int s = fpadlen(ny);
  return s + ((2 - s) % 16 + 16) % 16;
}

// Layout of a tile of TX columns: 16 FP32 values or 8 FP64 values meet per access, so 8 columns of
// FP32 meet with two rows each (layout 1, stride 2 mod 16), every other wide tile with one (odd
// stride).  With layout 0 and stride 2 throughout the y
// transforms of 256^2 x 200 FP64 took 605 + 626 us, they take 561 + 579.
template <typename T, int TX>
struct YLay {
  static constexpr int L = TX < 8 || sizeof(T) == 8 ? 0 : TX == 8 ? 1 : 2;
  static constexpr int JP = L == 0 ? 1 : 2;  // pad slots per 16 rows
  __host__ __device__ static int stride(int ny) {
    if (TX < 8) return ystride(ny);
    const int s = flay<L == 0 ? 0 : 2>((ny - 1) | 1) + 1, want = sizeof(T) == 4 && TX == 8 ? 2 : 1;
    return s + ((want - s) % 16 + 16) % 16;
  }
};

// CTAs per SM: a single transform of a long column of the compile-time plans gains from a third CTA
// (80 registers: 512^2 x 396 FP32 inverse 2.43 -> 2.13 ms, 256^2 x 200 FP64 561 -> 499 us); two
// transforms (mode 3) lose by it (2.69 -> 2.94 ms, 580 -> 643 us with the other four).  Narrow tiles (a column per
// warp) hold no twiddles over rows: four CTAs in FP64 for short columns (two: 72 -> 97 us, 64^2 x 68, 2 columns).
template <typename T, int TX, int DPT, bool POW2, int MC, bool TWO>
struct YOcc {
  static constexpr int v =
      TX < 8 ? (sizeof(T) == 4 ? (DPT <= 8 ? 4 : DPT <= 16 ? 2 : 1) : (DPT <= 4 ? 4 : DPT <= 8 ? 2 : 1))
             : !TWO && MC > 0 && MC * (int)sizeof(T) >= 2048 && MC <= 512 && FftOcc<T, DPT, POW2>::v == 2
                   ? 3
                   : FftOcc<T, DPT, POW2>::v;
};
template <typename T, int TX, int DPT, bool POW2, bool TWO, int MC = 0>
__global__ void __launch_bounds__(256, (YOcc<T, TX, DPT, POW2, MC, TWO>::v)) k_yfft(Geo g, YJobs<T> jobs, FftPlan pl,
                                              const typename cplx_t<T>::type* __restrict__ Wy) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ny = MC > 0 ? MC : g.ny;  // a constant with a compile-time plan
  typedef YLay<T, TX> Y;
  constexpr int YL = Y::L;
  const int RSY = Y::stride(ny);
  C* A = (C*)smraw;
  C* A2 = A + (size_t)TX * RSY;
  const YJob<T> jb = jobs.j[blockIdx.z];
  const int k = blockIdx.y;
  const int ii0 = blockIdx.x * TX;
  const bool fwd = jb.mode >= 2;
  constexpr bool two = TWO;  // mode 3
  // load: column ii0+b, row j -> A[b*RSY + flay<YL>(j)] (all copies in flight at once).
  // With 256 threads and TX | 256 a thread keeps its column b and steps j by
  // JS = 256/TX, so both addresses advance by fixed strides.
  constexpr int JS = 256 / TX;
  static_assert(JS % 16 == 0, "the padded smem stride of a j step must be a constant");
  const int tb = threadIdx.x % TX, tj = threadIdx.x / TX;
  const int iit = ii0 + tb;
  const bool colok = iit < g.nxhp;
  const size_t gstep = (size_t)JS * g.nxpp;
  // mode 1 with a compile-time length: the i ky factor is applied as the
  // values arrive (plain loads, all in flight), not in a second pass over the
  // shared tile
  constexpr bool kyload = MC > 0 && MC % JS == 0;
  const bool mulky = kyload && jb.mode == 1;
  // With a compile-time plan whose first pass has nb0 = MC / R0 butterflies, a
  // multiple of JS, a thread's loaded values (rows tj + JS it) hold every input
  // of its first-pass butterflies (rows j + nb0 r, j = tj + JS m).  The first
  // Stockham pass (Ns = 1, no twiddles) then runs in registers as the values
  // arrive, and the warps start at the second pass: one shared-memory write and
  // one read less per value.  The x-Nyquist column keeps its raw values.
  constexpr int R0 = MC > 0 ? 1 << CtPlan<(MC > 0 ? MC : 2)>::bits(0) : 1;
  constexpr int NB0 = MC > 0 ? MC / R0 : 1;
  constexpr bool fuse1 = MC > 0 && R0 <= 8 && NB0 % JS == 0 && CtPlan<(MC > 0 ? MC : 2)>::np > 1;
  // Likewise the last pass (Ns = MC / RL, as many butterflies): butterfly j
  // writes rows j + Ns r, all of them rows of the thread with tj = j mod JS
  // when Ns is a multiple of JS, so it runs as the values are stored.
  constexpr int NPS = CtPlan<(MC > 0 ? MC : 2)>::np;
  constexpr int RL = MC > 0 ? 1 << CtPlan<(MC > 0 ? MC : 2)>::bits(NPS - 1) : 1;
  constexpr int NSL = MC > 0 ? MC / RL : 1;
  constexpr bool fuseL = fuse1 && NPS >= 2 && RL <= 8 && NSL % JS == 0;
  if constexpr (fuse1) {
    constexpr int NIT = MC / JS, NBT = NB0 / JS;
    const bool tr = iit < g.nxh;
    const size_t g0 = fidx<T>(g, 2 * iit, tj, k);
#pragma unroll 1
    for (int hh = 0; hh < (two ? 2 : 1); ++hh) {
      const C* s1 = (const C*)((hh ? jb.src2 : jb.src) + g0);
      C* row = (hh ? A2 : A) + tb * RSY;
      C v[NIT];
#pragma unroll
      for (int it = 0; it < NIT; ++it) v[it] = colok ? s1[(size_t)it * (gstep / 2)] : cmk<C>(0, 0);
      if (jb.mode == 1) {
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
          const T ky = (T)g.yw[tj + it * JS];
          v[it] = cmk<C>(-(ky * v[it].y), ky * v[it].x);
        }
      }
      if (tr) {
#pragma unroll
        for (int mb = 0; mb < NBT; ++mb) {
          C w[R0];
#pragma unroll
          for (int r = 0; r < R0; ++r) w[r] = v[mb + r * NBT];  // row tj + JS mb + NB0 r
          dft_reg<C, R0>(w, !fwd);
          const int b0 = (tj + JS * mb) * R0;
#pragma unroll
          for (int r = 0; r < R0; ++r) row[flay<YL>(b0 + r)] = w[r];
        }
      } else {
#pragma unroll
        for (int it = 0; it < NIT; ++it) row[flay<YL>(tj) + it * (JS + Y::JP * (JS / 16))] = v[it];
      }
    }
  } else if (mulky) {
    const size_t g0 = fidx<T>(g, 2 * iit, tj, k);
    C* d = A + tb * RSY + flay<YL>(tj);
    const C* s1 = (const C*)(jb.src + g0);
    C v[kyload ? MC / JS : 1];
#pragma unroll
    for (int it = 0; it < (kyload ? MC / JS : 1); ++it)
      v[it] = colok ? s1[(size_t)it * (gstep / 2)] : cmk<C>(0, 0);
#pragma unroll
    for (int it = 0; it < (kyload ? MC / JS : 1); ++it) {
      const T ky = (T)g.yw[tj + it * JS];
      d[it * (JS + Y::JP * (JS / 16))] = cmk<C>(-(ky * v[it].y), ky * v[it].x);
    }
  } else {
    const size_t g0 = fidx<T>(g, 2 * iit, tj, k);
    C* d = A + tb * RSY + flay<YL>(tj);
    const C* s1 = (const C*)(jb.src + g0);
    const C* s2 = two ? (const C*)(jb.src2 + g0) : s1;
    for (int j = tj; j < ny; j += JS) {
      if (colok) {
        cp_async_c<C>(d, s1);
        if (two) cp_async_c<C>(d + TX * RSY, s2);
      } else {
        *d = cmk<C>(0, 0);
        if (two) d[TX * RSY] = cmk<C>(0, 0);
      }
      d += JS + Y::JP * (JS / 16);
      s1 = (const C*)((const T*)s1 + gstep);
      s2 = (const C*)((const T*)s2 + gstep);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  if (jb.mode == 1 && !mulky) {
    for (int t = threadIdx.x; t < TX * ny; t += blockDim.x) {
      const int b = t % TX, j = t / TX;
      const T ky = (T)g.yw[j];
      C* d = A + b * RSY + flay<YL>(j);
      const C v = *d;
      *d = cmk<C>(-(ky * v.y), ky * v.x);
    }
    __syncthreads();
  }
  // the x-Nyquist column (ii = nxh) is not transformed
  const int nb = ny > 1 ? max(0, min(TX, g.nxh - ii0)) : 0;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int gmax = MC > 0 ? CtRows<(MC > 0 ? MC : 2)>::G : nw * TX;  // columns a warp takes at a time
  const int gb = gmax > 1 ? max(1, min(gmax, ((two ? 2 : 1) * nb + nw - 1) / nw)) : 1;
  const int ng = gb > 1 ? (nb + gb - 1) / gb : nb;  // groups of gb columns
  {
    for (int q = threadIdx.x >> 5; q < (two ? 2 : 1) * ng; q += nw) {
      const int r = (q < ng ? q : q - ng) * gb;
      C* row = (q < ng ? A : A2) + r * RSY;
      const int G = min(gb, nb - r);
      if constexpr (fuseL)  // the first pass ran at load, the last runs at the store
        fft_passes_ct<C, (MC > 0 ? MC : 2), 1, NPS - 1, R0, YL>(row, RSY, G, Wy, !fwd, lane);
      else if constexpr (fuse1)
        fft_passes_ct<C, (MC > 0 ? MC : 2), 1, NPS, R0, YL>(row, RSY, G, Wy, !fwd, lane);  // the first pass ran at load
      else if constexpr (MC > 0)
        fft_warp_ct<C, MC, YL>(row, RSY, G, Wy, !fwd, lane);
      else
        fft_warp<C, DPT, POW2, YL, (TX < 8)>(row, RSY, G, pl, Wy, !fwd, lane);  // 8 warps: one column each
    }
  }
  __syncthreads();
  const T sc = fwd ? (T)g.scaley : (T)1;
  if constexpr (fuseL) {
    if (!colok) return;
    const bool tr = iit < g.nxh;  // the x-Nyquist column holds raw values
    const C* ra = A + tb * RSY;
    const C* rb = A2 + tb * RSY;
    C* o0 = (C*)(jb.dst + fidx<T>(g, 2 * iit, 0, k));
    const size_t ys = (size_t)g.nxpp / 2;  // one y row, in complex values
#pragma unroll 1
    for (int mb = 0; mb < NSL / JS; ++mb) {
      const int j = tj + JS * mb;  // butterfly of the last pass (Ns = NSL, step 1)
      C va[RL], vb[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        va[r] = ra[flay<YL>(j + r * NSL)];
        if (two) vb[r] = rb[flay<YL>(j + r * NSL)];
      }
      if (tr) {
#pragma unroll
        for (int r = 1; r < RL; ++r) {
          C tw = Wy[r * j];
          if (!fwd) tw.y = -tw.y;
          va[r] = cmul(va[r], tw);
          if (two) vb[r] = cmul(vb[r], tw);
        }
        dft_reg<C, RL>(va, !fwd);
        if (two) dft_reg<C, RL>(vb, !fwd);
      }
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int y = j + r * NSL;
        C o = cmk<C>(va[r].x * sc, va[r].y * sc);
        if (two) {
          const C w2 = cmk<C>(vb[r].x * sc, vb[r].y * sc);
          const T ky = (T)g.yw[y];
          o = cmk<C>(o.x - ky * w2.y, o.y + ky * w2.x);
        }
        o0[(size_t)y * ys] = o;
      }
    }
    return;
  }
  if (colok) {
    const C* d = A + tb * RSY + flay<YL>(tj);
    C* o1 = (C*)(jb.dst + fidx<T>(g, 2 * iit, tj, k));
    for (int j = tj; j < ny; j += JS) {
      const C v = *d;
      C o = cmk<C>(v.x * sc, v.y * sc);
      if (two) {
        const C v2 = d[TX * RSY];
        const C w2 = cmk<C>(v2.x * sc, v2.y * sc);
        const T ky = (T)g.yw[j];
        o = cmk<C>(o.x - ky * w2.y, o.y + ky * w2.x);
      }
      *o1 = o;
      d += JS + Y::JP * (JS / 16);
      o1 = (C*)((T*)o1 + gstep);
    }
  }
}

// ===========================================================================
// x transforms of rows.  Real length nx = 2M through complex length M.
// ===========================================================================
template <typename C, typename T>
__device__ __forceinline__ void xinv_prep(const T* __restrict__ row, C* Z, int M, const C* __restrict__ Wn, int mulkx,
                                          T kxstep, int t0, int nthr) {
  // row: nxhp complex (interleaved); optional multiply by i*kx (kx = m*kxstep)
  for (int k = t0; k < M; k += nthr) {
    C Xk = cmk<C>(row[2 * k], row[2 * k + 1]);
    C Xm = cmk<C>(row[2 * (M - k)], row[2 * (M - k) + 1]);
    if (mulkx) {
      T a = kxstep * (T)k, b = kxstep * (T)(M - k);
      Xk = cmk<C>(-(a * Xk.y), a * Xk.x);
      Xm = cmk<C>(-(b * Xm.y), b * Xm.x);
    }
    if (k == 0) {
      Xk.y = 0;
      Xm.y = 0;
    }
    C s = cadd(Xk, cconj(Xm));
    C d = csub(Xk, cconj(Xm));
    C w = Wn[k];  // exp(-2 pi i k/N); need i*conj(w)*d
    C wc = cconj(w);
    C t = cmul(wc, d);
    Z[k] = cmk<C>(s.x - t.y, s.y + t.x);
  }
}

// forward post: Z = FFT_M(z) -> X_k k=0..M (scaled by 1/N)
template <typename C>
__device__ __forceinline__ C xfwd_post(const C* Z, int k, int M, const C* __restrict__ Wn, decltype(C().x) invN) {
  typedef decltype(C().x) T;
  if (k == 0) return cmk<C>((Z[0].x + Z[0].y) * invN, (T)0);
  if (k == M) return cmk<C>((Z[0].x - Z[0].y) * invN, (T)0);
  C a = Z[k], b = cconj(Z[M - k]);
  C e = cmk<C>((T)0.5 * (a.x + b.x), (T)0.5 * (a.y + b.y));
  C dd = csub(a, b);
  C o = cmk<C>((T)0.5 * dd.y, (T)-0.5 * dd.x);  // (a-b)/(2i)
  C w = Wn[k];
  C wo = cmul(w, o);
  return cmk<C>((e.x + wo.x) * invN, (e.y + wo.y) * invN);
}

// Parameters of the fused NL row kernel.
template <typename T>
struct NLArgs {
  const T* in[10];  // (kx,y): u v w t | dy u v w | dz u v w
  T* out[11];       // (kx,y): Au Av Aw At | uv vv vw vt | uw ww wt
  double coef_buoy; // N^2 / rhograd
  double rg;        // rhograd
  double tau_pen[IW_MAX_SUBD];  // 0.5/omega*(2/zh)
  int forcing;
  double f_xk, f_xm, f_om, f_t, f_amp_u, f_amp_w, f_amp_r;  // paddle
  double dx;
};

// In-place pre-pass of the inverse real transform for the pair (kk, M-kk) of a
// padded row holding X_0..X_M: Z_k = (X_k + conj X_{M-k}) + i conj(W_k) (X_k - conj X_{M-k}),
// after the optional multiplication by i kx.  0 <= kk <= M/2.
template <typename C, typename T>
__device__ __forceinline__ void xprep_pair(C* row, int kk, int M, const C* __restrict__ Wn, bool mulkx, T kxstep) {
  const int km = M - kk;
  const C X0 = row[fpad(kk)], X1 = row[fpad(km)];
  auto zk = [&](C Xk, C Xm, int k) {
    if (mulkx) {
      const T a = kxstep * (T)k, b = kxstep * (T)(M - k);
      Xk = cmk<C>(-(a * Xk.y), a * Xk.x);
      Xm = cmk<C>(-(b * Xm.y), b * Xm.x);
    }
    if (k == 0) {
      Xk.y = 0;
      Xm.y = 0;
    }
    const C s = cadd(Xk, cconj(Xm));
    const C d = csub(Xk, cconj(Xm));
    const C t = cmul(cconj(Wn[k]), d);
    return cmk<C>(s.x - t.y, s.y + t.x);
  };
  const C z0 = zk(X0, X1, kk);
  if (kk > 0 && kk < km) row[fpad(km)] = zk(X1, X0, km);
  row[fpad(kk)] = z0;
}

// forward post on a padded row: Z = FFT_M(z) -> X_k, k = 0..M (scaled by 1/N)
template <typename C>
__device__ __forceinline__ C xfwd_post_p(const C* row, int k, int M, const C* __restrict__ Wn,
                                         decltype(C().x) invN) {
  typedef decltype(C().x) T;
  if (k == 0 || k == M) {
    const C z = row[0];
    return k == 0 ? cmk<C>((z.x + z.y) * invN, (T)0) : cmk<C>((z.x - z.y) * invN, (T)0);
  }
  const C a = row[fpad(k)], b = cconj(row[fpad(M - k)]);
  const C e = cmk<C>((T)0.5 * (a.x + b.x), (T)0.5 * (a.y + b.y));
  const C dd = csub(a, b);
  const C o = cmk<C>((T)0.5 * dd.y, (T)-0.5 * dd.x);  // (a-b)/(2i)
  const C wo = cmul(Wn[k], o);
  return cmk<C>((e.x + wo.x) * invN, (e.y + wo.y) * invN);
}

// slots per padded x row (M+1 half-complex values)
__host__ __device__ __forceinline__ int xstride(int M) { return fpadlen(M + 1); }

// K_C: CTA per (j,k) row; 17 padded rows of M+1 values in shared memory; each
// warp transforms whole rows in place.
template <typename T, int DPT, bool POW2, int MC = 0>
__global__ void __launch_bounds__(256, (FftOcc<T, DPT, POW2>::v)) k_xrow_nl(Geo g, NLArgs<T> a, FftPlan pl,
                                                 const typename cplx_t<T>::type* __restrict__ Wm,
                                                 const typename cplx_t<T>::type* __restrict__ Wn) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int M = MC > 0 ? MC : g.nx / 2;  // a constant with a compile-time plan
  const int RS = xstride(M);
  C* buf = (C*)smraw;
  const int j = blockIdx.x, k = blockIdx.y;
  const int N = g.N;
  const int kl = k % N, ks = k / N;
  const bool nb_lo = (kl == 0 && k > 0);
  const bool nb_hi = (kl == N - 1 && k < g.nz - 1);
  const int knb = nb_lo ? k - 1 : k + 1;
  const int nrow = 13 + ((nb_lo || nb_hi) ? 4 : 0);
  const T kxs = (T)g.xw[1];
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nthr >> 5;
  // rows 0..3 u v w t, 4..6 dx of u v w, 7..9 dy, 10..12 dz, 13..16 neighbour u v w t:
  // half-complex rows (M+1 values), all copies in flight at once
  // Element offsets of this (j, k) row and of the neighbour's, once per CTA.
  // A thread keeps its kk and walks the rows (fixed strides, no index
  // arithmetic per copy); kk = M, the last value of a row, goes to thread r.
  const size_t roff = fidx<T>(g, 0, j, k), roffn = fidx<T>(g, 0, j, knb);
  auto rsrc = [&](int r) -> const C* {
    return (const C*)((r < 4 ? a.in[r] : r < 7 ? a.in[r - 4] : r < 13 ? a.in[r - 3] : a.in[r - 13]) + (r < 13 ? roff : roffn));
  };
  for (int kk = tid; kk < M; kk += nthr) {
    C* d = buf + fpad(kk);
#pragma unroll
    for (int r = 0; r < 17; ++r)
      if (r < nrow) cp_async_c<C>(d + r * RS, rsrc(r) + kk);
  }
  if (tid < nrow) cp_async_c<C>(buf + tid * RS + fpad(M), rsrc(tid) + M);
  cp_async_wait_all();
  __syncthreads();
  const int nh = M / 2 + 1;
  const int H2 = M / 2;
  if (MC > 0 && nthr % H2 == 0) {
    // a thread keeps its pair kk < M/2 and steps over rows by nthr/(M/2);
    // the middle pair kk = M/2 goes to thread r
    const int kk = tid % H2, rs = nthr / H2;
    for (int r = tid / H2; r < nrow; r += rs) xprep_pair<C, T>(buf + r * RS, kk, M, Wn, r >= 4 && r < 7, kxs);
    if (tid < nrow) xprep_pair<C, T>(buf + tid * RS, H2, M, Wn, tid >= 4 && tid < 7, kxs);
  } else {
    for (int q = tid; q < nrow * nh; q += nthr) {
      const int r = q / nh, kk = q - r * nh;
      xprep_pair<C, T>(buf + r * RS, kk, M, Wn, r >= 4 && r < 7, kxs);
    }
  }
  __syncthreads();
  const int gmax = MC > 0 ? CtRows<(MC > 0 ? MC : 2)>::G : 17;  // rows a warp takes at a time
  {
    const int gb = min(gmax, (nrow + nw - 1) / nw);
    for (int r = wid * gb; r < nrow; r += nw * gb) {
      if constexpr (MC > 0)
        fft_warp_ct<C, MC>(buf + r * RS, RS, min(gb, nrow - r), Wm, true, lane);
      else
        fft_warp<C, DPT, POW2>(buf + r * RS, RS, min(gb, nrow - r), pl, Wm, true, lane);
    }
  }
  __syncthreads();
  // physical value i of row r
  auto P = [&](int r, int i) -> T& { return ((T*)(buf + r * RS))[2 * fpad(i >> 1) + (i & 1)]; };
  const int nx = 2 * M;
  // upwind interface penalty (solver.f:700-839); products overwrite rows 0..12
  for (int i = tid; i < nx; i += nthr) {
    const T u = P(0, i), v = P(1, i), w = P(2, i), t = P(3, i);
    const T ux = P(4, i), vx = P(5, i), wx = P(6, i);
    const T uy = P(7, i), vy = P(8, i), wy = P(9, i);
    const T uz = P(10, i), vz = P(11, i), wz = P(12, i);
    T qu = (T)-0.5 * (u * ux + v * uy + w * uz);
    T qv = (T)-0.5 * (u * vx + v * vy + w * vz);
    T qw = (T)-0.5 * (u * wx + v * wy + w * wz) + (T)a.coef_buoy * t;
    T qt = -(w * (T)a.rg);
    if (nb_lo && w > (T)0) {  // bottom point of subdomain ks: inflow from below
      const T tau = (T)a.tau_pen[ks], al = w;
      qu -= tau * (al * u - al * P(13, i));
      qv -= tau * (al * v - al * P(14, i));
      qw -= tau * (al * w - al * P(15, i));
      qt -= tau * (al * t - al * P(16, i));
    }
    if (nb_hi && w < (T)0) {
      const T tau = (T)a.tau_pen[ks], ga = -w;
      qu -= tau * (ga * u - ga * P(13, i));
      qv -= tau * (ga * v - ga * P(14, i));
      qw -= tau * (ga * w - ga * P(15, i));
      qt -= tau * (ga * t - ga * P(16, i));
    }
    if (a.forcing == IW_PADDLE_ALL_LEVELS || (a.forcing == IW_PADDLE_ABOVE_BOTTOM && k > 0)) {
      double xx = (double)i * a.dx, zz = g.zg[k];
      double arg = a.f_xk * xx - a.f_om * a.f_t;
      double sf, cf;
      sincos(arg, &sf, &cf);
      double czm = cos(a.f_xm * zz), szm = sin(a.f_xm * zz);
      qu += (T)(a.f_amp_u * czm * sf);
      qw += (T)(a.f_amp_w * szm * cf);
      qt += (T)(a.f_amp_r * szm * sf);
    }
    // 13 rows to transform: Qu Qv Qw Qt | uu uv uw ut | vv vw vt | ww wt
    P(0, i) = qu;
    P(1, i) = qv;
    P(2, i) = qw;
    P(3, i) = qt;
    P(4, i) = (T)-0.5 * u * u;
    P(5, i) = (T)-0.5 * u * v;
    P(6, i) = (T)-0.5 * u * w;
    P(7, i) = -(u * t);
    P(8, i) = (T)-0.5 * v * v;
    P(9, i) = (T)-0.5 * v * w;
    P(10, i) = -(v * t);
    P(11, i) = (T)-0.5 * w * w;
    P(12, i) = -(w * t);
  }
  __syncthreads();
  {
    const int gb = min(gmax, (13 + nw - 1) / nw);
    for (int r = wid * gb; r < 13; r += nw * gb) {
      if constexpr (MC > 0)
        fft_warp_ct<C, MC>(buf + r * RS, RS, min(gb, 13 - r), Wm, false, lane);
      else
        fft_warp<C, DPT, POW2>(buf + r * RS, RS, min(gb, 13 - r), pl, Wm, false, lane);
    }
  }
  __syncthreads();
  const T invN = (T)1 / (T)nx;
  // outputs: A_q = X(Q_q) + i kx X(P_uq) for q = u v w t ; then uv vv vw vt uw ww wt
  // a thread keeps its kk and writes it in all 11 output rows; kk = M goes
  // to thread o
  auto outv = [&](int o, int kk) -> C {
    if (o < 4) {
      const C x1 = xfwd_post_p<C>(buf + o * RS, kk, M, Wn, invN);
      const C x2 = xfwd_post_p<C>(buf + (4 + o) * RS, kk, M, Wn, invN);
      const T kx = kxs * (T)kk;
      return cmk<C>(x1.x - kx * x2.y, x1.y + kx * x2.x);
    }
    // map: 4->uv(5) 5->vv(8) 6->vw(9) 7->vt(10) 8->uw(6) 9->ww(11) 10->wt(12)
    const int sr = o == 4 ? 5 : o == 5 ? 8 : o == 6 ? 9 : o == 7 ? 10 : o == 8 ? 6 : o == 9 ? 11 : 12;
    return xfwd_post_p<C>(buf + sr * RS, kk, M, Wn, invN);
  };
  for (int kk = tid; kk < M; kk += nthr) {
#pragma unroll 1
    for (int o = 0; o < 11; ++o) *((C*)(a.out[o] + roff) + kk) = outv(o, kk);
  }
  if (tid < 11) *((C*)(a.out[tid] + roff) + M) = outv(tid, M);
}

// K_C for complex lengths M = R0 NB with R0 in {2, 4, 6, 8, 10} and NB in {8, 16, 32}, i.e.
// the plan R0 * (NB / 2) * 2: each value passes through shared memory four times per
// transform pair of passes less than in k_xrow_nl, which is bound by that traffic.
//   1. A lane loads the spectrum of butterflies it and NB - it of a row's first pass
//      (their R0 values each are each other's mirror images k, M - k), so the pre-pass of the
//      real transform and the radix-R0 pass run in registers; a warp holds 64 / NB rows.
//   2. The middle pass (radix NB / 2) in place, still within the warp.
//   3. The last inverse pass (radix 2), the products and the first forward pass in
//      registers: a thread owns values p and p + M/2 of all 13 rows.
//   4. The forward middle pass, then the last pass (radix R0) of butterflies it and NB - it
//      with the post-pass of the real transform, the i kx fold of the advective form and the
//      stores, in registers.  The fold needs rows Q_q and u q at once: they sit in the two
//      halves of a warp.
// Lane it = 0 has the two butterflies 0 and NB / 2, which are their own mirror images: its
// pairs are regrouped with selects, the middle value k = M/2 is one extra value E.
// Measured against k_xrow_nl (which then also carried the three rows of d rho): 512^2 x 396 FP32
// 5.56 -> 3.39 ms, 256^2 x 200 FP64 1.96 -> 0.96 ms, 192 x 120 x 110 FP32 401 -> 123 us, 64^2 x 68 FP64
// 83 -> 29 us.  At 512^2 it moves its 21 fields at 2.6 TB/s, bound by instruction issue (2.6 per cycle)
// and in FP64 by the L1 data path (twiddles and rows, 72 %).
// Threads per SM: 512 in FP32 (128 registers; with 640 a thread of R0 = 8 spills: 3.39 -> 3.94 ms),
// 384 in FP64 (168 registers: 1.02 against 1.05 ms with 256), but 256 for R0 < 6, whose rows are so
// short that loads in flight count (64^2: 29 against 38 us).  From R0 = 6 on the indexes and twiddles
// of a lane are made anew in every round; kept over the rounds they cost spills (3.70 -> 4.65 ms).
// Place of value i of a row: padded (FP32), or exchanged within groups of 8 (FP64, whose 16-byte
// values meet in 8 banks: strides 2, 8 and 16 then fall in different ones, and no space is lost).
template <typename C>
__device__ __forceinline__ int xpos(int i) {
  return sizeof(C) == 16 ? i ^ ((i >> 3) & 7) : fpad(i);
}
template <typename T, int R0, int NB>
struct XReg {
  static constexpr int M = R0 * NB, RM = NB / 2, I = NB / 2, G = 32 / I, YR = G / 2;
  static constexpr int threads = 16 * R0;  // = YR M / 2
  static constexpr int RS = sizeof(T) == 8 ? M : M + (M - 1) / 16;
  static constexpr size_t smem = (size_t)17 * YR * RS * 2 * sizeof(T);
  static constexpr int ctas = (sizeof(T) == 4 ? 512 : R0 < 6 ? 256 : 384) / threads;
};

// Radix-R pass (output stride NS before it) over the first lim of the G rows at base, all
// lanes of a warp.
template <typename C, int M, int R, int NS, int G, bool INV>
__device__ __forceinline__ void xreg_pass(C* base, int RS, int lim, const C* __restrict__ W, int lane) {
  constexpr int nb = M / R, RPI = 32 / nb, NIT = G / RPI;  // rows at a time, rounds
  constexpr int CV = sizeof(C) == 8 ? 16 : 8, CH = CV / R < 1 ? 1 : CV / R < NIT ? CV / R : NIT;
  constexpr int step = M / (NS * R);
  static_assert(nb <= 32 && G % RPI == 0 && NIT % CH == 0, "rows do not divide");
  const int g = lane / nb, j = lane % nb, jq = j / NS, jm = j % NS;
  if (RPI * nb < 32 && g >= RPI) lim = 0;  // idle lanes
  C* row = base + g * RS;
#pragma unroll 1
  for (int c = 0; c < NIT; c += CH, row += CH * RPI * RS) {
    C v[CH][R];
#pragma unroll
    for (int q = 0; q < CH; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r) v[q][r] = cmk<C>(0, 0);  // (not carried from round to round)
    if (g + c * RPI < lim) {
#pragma unroll
      for (int q = 0; q < CH; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (q == 0 || g + (c + q) * RPI < lim) v[q][r] = row[q * RPI * RS + xpos<C>(j + r * nb)];
#pragma unroll
      for (int r = 1; r < R; ++r) {
        C tw = W[r * jm * step];
        if (INV) tw.y = -tw.y;
#pragma unroll
        for (int q = 0; q < CH; ++q) v[q][r] = cmul(v[q][r], tw);
      }
#pragma unroll
      for (int q = 0; q < CH; ++q) dft_reg<C, R>(v[q], INV);
    }
    __syncwarp();
    if (g + c * RPI < lim) {
#pragma unroll
      for (int q = 0; q < CH; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (q == 0 || g + (c + q) * RPI < lim) row[q * RPI * RS + xpos<C>(jq * NS * R + jm + r * NS)] = v[q][r];
    }
  }
  __syncwarp();
}

template <typename T, int R0, int NB>
__global__ void __launch_bounds__(XReg<T, R0, NB>::threads, (XReg<T, R0, NB>::ctas))
    k_xrow_reg(Geo g, const __grid_constant__ NLArgs<T> a, const typename cplx_t<T>::type* __restrict__ Wm,
               const typename cplx_t<T>::type* __restrict__ Wn) {
  typedef typename cplx_t<T>::type C;
  typedef XReg<T, R0, NB> X;
  constexpr int M = X::M, I = X::I, G = X::G, YR = X::YR, RS = X::RS, RM = X::RM, H = R0 / 2, M2 = M / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* buf = (C*)smraw;
  const int j0 = blockIdx.x * YR, k = blockIdx.y;
  const int kl = k % g.N, ks = k / g.N;
  const bool nb_lo = (kl == 0 && k > 0);
  const bool nb_hi = (kl == g.N - 1 && k < g.nz - 1);
  const int knb = nb_lo ? k - 1 : k + 1;
  const T kxs = (T)g.xw[1];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int nw = X::threads / 32;
  const int gr = lane / I;
  // rows (r, y): 0..3 u v w t, 4..6 dx of u v w, 7..9 dy, 10..12 dz, 13..16 neighbour u v w t
  const int nrow = (13 + ((nb_lo || nb_hi) ? 4 : 0)) * YR;
#pragma unroll 1
  for (int g0 = wid * G; g0 < nrow; g0 += nw * G) {
    int it = lane % I;
    if (R0 >= 6) asm volatile("" : "+r"(it));  // (not kept over the rounds)
    const bool self = it == 0;
    const int jb = self ? NB / 2 : NB - it;
    // pair q of a lane: k = kq(q) and M - k
    const int khi = self ? NB / 2 - NB * H : it;
    auto kq = [&](int q) { return (q < H ? it : khi) + NB * q; };
    const T fit = (T)it, fkhi = (T)khi;
    auto fkq = [&](int q) { return (q < H ? fit : fkhi) + (T)(NB * q); };
    const int row = g0 + gr, r = row / YR, jy = j0 + row % YR;
    const bool act = row < nrow && jy < g.ny;
    const bool dx = r >= 4 && r < 7;
    C P[R0], Q[R0], E = cmk<C>(0, 0);
    if (act) {
      const T* f = a.in[r < 4 ? r : r < 7 ? r - 4 : r < 13 ? r - 3 : r - 13];
      const C* src = (const C*)(f + fidx<T>(g, 0, jy, r < 13 ? k : knb));
#pragma unroll
      for (int q = 0; q < R0; ++q) {
        P[q] = src[kq(q)];
        Q[q] = src[M - kq(q)];
      }
      if (self) E = src[M2];
    } else {
#pragma unroll
      for (int q = 0; q < R0; ++q) P[q] = Q[q] = cmk<C>(0, 0);
    }
#pragma unroll
    for (int q = 0; q < R0; ++q) {
      if (dx) {
        const T ka = kxs * fkq(q), kb = kxs * ((T)M - fkq(q));
        P[q] = cmk<C>(-(ka * P[q].y), ka * P[q].x);
        Q[q] = cmk<C>(-(kb * Q[q].y), kb * Q[q].x);
      }
      if (q == 0 && self) P[0].y = Q[0].y = 0;
      // Z_k = s + i t, Z_{M-k} = conj(s) + i conj(t); s = X_k + conj X_{M-k}, t = conj(W_k) (X_k - conj X_{M-k})
      const C s = cadd(P[q], cconj(Q[q])), d = csub(P[q], cconj(Q[q]));
      const C t = cmul(cconj(Wn[kq(q)]), d);
      P[q] = cmk<C>(s.x - t.y, s.y + t.x);
      Q[q] = cmk<C>(s.x + t.y, t.x - s.y);
    }
    if (dx) {
      const T ke = kxs * (T)M2;
      E = cmk<C>(-(ke * E.y), ke * E.x);
    }
    E = cmk<C>((T)2 * E.x, (T)-2 * E.y);  // k = M/2: 2 conj(X)
    C va[R0], vb[R0];
#pragma unroll
    for (int q = 0; q < R0; ++q) {
      va[q] = q < H ? P[q] : self ? (q == H ? E : Q[R0 - q]) : P[q];
      vb[q] = self ? (q < H ? P[q + H] : Q[R0 - 1 - q + H]) : Q[R0 - 1 - q];
    }
    dft_reg<C, R0>(va, true);
    dft_reg<C, R0>(vb, true);
    C* rw = buf + (row < nrow ? row : 0) * RS;
    if (row < nrow) {
#pragma unroll
      for (int q = 0; q < R0; ++q) {
        rw[xpos<C>(it * R0 + q)] = va[q];
        rw[xpos<C>(jb * R0 + q)] = vb[q];
      }
    }
    __syncwarp();
    xreg_pass<C, M, RM, R0, G, true>(buf + g0 * RS, RS, nrow - g0, Wm, lane);
  }
  __syncthreads();
  const int p = tid % M2, yr = tid / M2;
  // values 2p, 2p+1 (c = 0, 1 of element 0) and 2p+M, 2p+M+1 (element 1) of row r
  const C *c0 = buf + yr * RS + xpos<C>(p), *c1 = buf + yr * RS + xpos<C>(p + M2);
  C tw = Wm[p];
  tw.y = -tw.y;
  struct V {
    C e[2];
  };
  auto get = [&](int r) {
    V o;
    o.e[0] = c0[r * YR * RS];
    o.e[1] = cmul(c1[r * YR * RS], tw);
    dft_reg<C, 2>(o.e, true);
    return o;
  };
  auto put = [&](int r, V o) {
    dft_reg<C, 2>(o.e, false);
    C* d = buf + (r * YR + yr) * RS;
    d[xpos<C>(2 * p)] = o.e[0];
    d[xpos<C>(2 * p + 1)] = o.e[1];
  };
#define IW_V(o, expr)                                            \
  _Pragma("unroll") for (int e = 0; e < 2; ++e) {                \
    { T& o_ = o.e[e].x; const int c = 0; (void)c; o_ = (expr); } \
    { T& o_ = o.e[e].y; const int c = 1; (void)c; o_ = (expr); } \
  }
#define IW_C(v) (c == 0 ? v.e[e].x : v.e[e].y)
  V u = get(0), v = get(1), w = get(2), t = get(3);
  V qu, qv, qw, qt;
  {
    const V ux = get(4), vx = get(5), wx = get(6);
    IW_V(qu, IW_C(u) * IW_C(ux))
    IW_V(qv, IW_C(u) * IW_C(vx))
    IW_V(qw, IW_C(u) * IW_C(wx))
    const V uy = get(7), vy = get(8), wy = get(9);
    IW_V(qu, IW_C(qu) + IW_C(v) * IW_C(uy))
    IW_V(qv, IW_C(qv) + IW_C(v) * IW_C(vy))
    IW_V(qw, IW_C(qw) + IW_C(v) * IW_C(wy))
    const V uz = get(10), vz = get(11), wz = get(12);
    IW_V(qu, (T)-0.5 * (IW_C(qu) + IW_C(w) * IW_C(uz)))
    IW_V(qv, (T)-0.5 * (IW_C(qv) + IW_C(w) * IW_C(vz)))
    IW_V(qw, (T)-0.5 * (IW_C(qw) + IW_C(w) * IW_C(wz)) + (T)a.coef_buoy * IW_C(t))
    IW_V(qt, -(IW_C(w) * (T)a.rg))
  }
  // upwind interface penalty (solver.f:700-839): inflow from below at the bottom point of
  // subdomain ks, from above at its top point
  if (nb_lo || nb_hi) {
    const T tau = (T)a.tau_pen[ks];
    V al;
    IW_V(al, nb_lo ? (IW_C(w) > (T)0 ? IW_C(w) : (T)0) : (IW_C(w) < (T)0 ? -IW_C(w) : (T)0))
    auto pen = [&](V& q, const V& f, int r) {
      const V n = get(r);
      IW_V(q, IW_C(al) != (T)0 ? IW_C(q) - tau * (IW_C(al) * IW_C(f) - IW_C(al) * IW_C(n)) : IW_C(q))
    };
    pen(qu, u, 13);
    pen(qv, v, 14);
    pen(qw, w, 15);
    pen(qt, t, 16);
  }
  if (a.forcing == IW_PADDLE_ALL_LEVELS || (a.forcing == IW_PADDLE_ABOVE_BOTTOM && k > 0)) {
    const double zz = g.zg[k], czm = cos(a.f_xm * zz), szm = sin(a.f_xm * zz);
    double sf[2][2], cf[2][2];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        sincos(a.f_xk * ((double)(2 * p + M * e + c) * a.dx) - a.f_om * a.f_t, &sf[e][c], &cf[e][c]);
    IW_V(qu, IW_C(qu) + (T)(a.f_amp_u * czm * sf[e][c]))
    IW_V(qw, IW_C(qw) + (T)(a.f_amp_w * szm * cf[e][c]))
    IW_V(qt, IW_C(qt) + (T)(a.f_amp_r * szm * sf[e][c]))
  }
  __syncthreads();
  // rows to transform: Qu uu Qv uv Qw uw Qt ut vv vw vt ww wt
  {
    V o;
    put(0, qu);
    put(2, qv);
    put(4, qw);
    put(6, qt);
    IW_V(o, (T)-0.5 * IW_C(u) * IW_C(u)) put(1, o);
    IW_V(o, (T)-0.5 * IW_C(u) * IW_C(v)) put(3, o);
    IW_V(o, (T)-0.5 * IW_C(u) * IW_C(w)) put(5, o);
    IW_V(o, -(IW_C(u) * IW_C(t))) put(7, o);
    IW_V(o, (T)-0.5 * IW_C(v) * IW_C(v)) put(8, o);
    IW_V(o, (T)-0.5 * IW_C(v) * IW_C(w)) put(9, o);
    IW_V(o, -(IW_C(v) * IW_C(t))) put(10, o);
    IW_V(o, (T)-0.5 * IW_C(w) * IW_C(w)) put(11, o);
    IW_V(o, -(IW_C(w) * IW_C(t))) put(12, o);
  }
#undef IW_V
#undef IW_C
  __syncthreads();
  const T hN = (T)0.5 / (T)(2 * M);
#pragma unroll 1
  for (int g0 = wid * G; g0 < 13 * YR; g0 += nw * G) {
    int it = lane % I;
    if (R0 >= 6) asm volatile("" : "+r"(it));  // (not kept over the rounds)
    const bool self = it == 0;
    const int jb = self ? NB / 2 : NB - it;
    // pair q of a lane: k = kq(q) and M - k
    const int khi = self ? NB / 2 - NB * H : it;
    auto kq = [&](int q) { return (q < H ? it : khi) + NB * q; };
    const T fit = (T)it, fkhi = (T)khi;
    auto fkq = [&](int q) { return (q < H ? fit : fkhi) + (T)(NB * q); };
    xreg_pass<C, M, RM, 2, G, false>(buf + g0 * RS, RS, G, Wm, lane);  // (a last row pair may hold one unused row)
    const int row = g0 + gr, r = row / YR, jy = j0 + row % YR;
    const C* rw = buf + row * RS;
    C va[R0], vb[R0];
#pragma unroll
    for (int q = 0; q < R0; ++q) {
      va[q] = rw[xpos<C>(it + NB * q)];
      vb[q] = rw[xpos<C>(jb + NB * q)];
    }
#pragma unroll
    for (int q = 1; q < R0; ++q) {
      // the twiddles of butterfly jb = NB - it are conj(W^(q it)) times the R0-th roots w^q, which
      // shift its outputs by one place; butterfly 0 has none
      const C tw = Wm[q * (self ? NB / 2 : it)];
      va[q] = cmul(va[q], self ? cmk<C>(1, 0) : tw);
      vb[q] = cmul(vb[q], cconj(tw));
    }
    dft_reg<C, R0>(va, false);
    dft_reg<C, R0>(vb, false);
    {
      const C v0 = vb[0];
#pragma unroll
      for (int q = 0; q + 1 < R0; ++q) vb[q] = vb[q + 1];
      vb[R0 - 1] = v0;
    }
    // X_k = e + W_k o, X_{M-k} = conj(e - W_k o); e = (Z_k + conj Z_{M-k}) / 2N,
    // o = (Z_k - conj Z_{M-k}) / 2iN (k = 0: Z_M = Z_0; k = M/2: conj Z)
    const bool fold = g0 < 8 * YR;  // r = 0..7: A_q = X(Q_q) + i kx X(u q)
    const bool odd = lane >= 16;    // the row u q of a pair
    const int dst = fold ? (odd ? (r == 3 ? 4 : r == 5 ? 8 : -1) : r >> 1)
                         : r == 8 ? 5 : r == 9 ? 6 : r == 10 ? 7 : r == 11 ? 9 : r == 12 ? 10 : -1;
    const bool act = dst >= 0 && jy < g.ny;
    C* out = act ? (C*)(a.out[dst] + fidx<T>(g, 0, jy, k)) : nullptr;
    auto emit = [&](C x, int kk, T fk, bool on) {
      if (fold) {
        C y;
        y.x = __shfl_down_sync(0xffffffffu, x.x, 16);
        y.y = __shfl_down_sync(0xffffffffu, x.y, 16);
        const T kx = kxs * fk;
        if (!odd) x = cmk<C>(x.x - kx * y.y, x.y + kx * y.x);
      }
      if (on && act) out[kk] = x;
    };
#pragma unroll
    for (int q = 0; q < R0; ++q) {
      const C A = q < H ? va[q] : self ? vb[q - H] : va[q];
      const C B = cconj(self ? (q == 0 ? va[0] : q < H ? va[R0 - q] : vb[R0 - 1 - q + H]) : vb[R0 - 1 - q]);
      const C e = cmk<C>(hN * (A.x + B.x), hN * (A.y + B.y));
      const C o = cmul(Wn[kq(q)], cmk<C>(hN * (A.y - B.y), -(hN * (A.x - B.x))));
      emit(cadd(e, o), kq(q), fkq(q), true);
      emit(cconj(csub(e, o)), M - kq(q), (T)M - fkq(q), true);
    }
    emit(cmk<C>((T)2 * hN * va[H].x, (T)-2 * hN * va[H].y), M2, (T)M2, self);
    __syncwarp();
  }
}

// ===========================================================================
// K_E: per (field q, real x index i, y index j, subdomain ks):
//   S    = B + (2/h) D Z                     (NL term at level n, spectral)
//   wnl  = fac1 S + fac2 Sn + fac3 Snm at the walls (w only, solver.f:267-284)
//   F2   = P(F1)                             (end-of-rhsfm round trip)
//   F*   = dt (fac1 S + fac2 Sn + fac3 Snm) + bdf1 F2 + bdf2 Fn + bdf3 Fnm
//   Snm <- S (becomes Sn), Fnm <- F2 (becomes Fn)      (solver.f:447-478)
//   F   <- cf(ii,j) * L F* per subdomain    (filter_3dlegenfourier)
// ===========================================================================
struct Coefs {
  double fac1, fac2, fac3, bdf1, bdf2, bdf3, bdfv, dt;
};

// u* = dt (extrapolated NL) + bdf1 F2 + bdf2 Fn + bdf3 Fnm, combined in FP64
// whatever the storage type: in FP32 the rounded coefficients (1/3) would
// make bdf1 + bdf2 + bdf3 differ from bdfv and bias every step the same way.
template <typename T>
__device__ __forceinline__ T bdf_combine(const Coefs& c, T se, T F2, T fn, T fnm) {
  return (T)(c.dt * (double)se + c.bdf1 * (double)F2 + c.bdf2 * (double)fn + c.bdf3 * (double)fnm);
}
// the same with every rounding written out
template <typename T>
__device__ __forceinline__ T bdf_combine_rn(const Coefs& c, T se, T F2, T fn, T fnm) {
  return (T)__fma_rn(c.bdf3, (double)fnm,
                     __fma_rn(c.bdf2, (double)fn, __fma_rn(c.bdf1, (double)F2, __dmul_rn(c.dt, (double)se))));
}


// one point of K_E: S = B + fac (D Z), u* from the BDF combination of the
// extrapolated S
template <typename T>
__device__ __forceinline__ void stageE_point(const Coefs& c, T fac, T f1, T f2, T f3, T b, T dz, T sn, T snm, T F2,
                                             T fn, T fnm, T& S, T& fsv) {
  S = fma_t(dz, fac, b);
  const T se = fma_t(f3, snm, fma_t(f2, sn, mul_t(f1, S)));
  fsv = bdf_combine_rn<T>(c, se, F2, fn, fnm);
}
// the extrapolated S in FP64 at the walls (the wall data of w)
template <typename T>
__device__ __forceinline__ double stageE_wall(T f1, T f2, T f3, T S, T sn, T snm) {
  return __fma_rn((double)f3, (double)snm, __fma_rn((double)f2, (double)sn, __dmul_rn((double)f1, (double)S)));
}
// the filtered value: cf (L f) = g + (cf - 1) g with g = f + (L - I) f
__device__ __forceinline__ double stageE_filtered(double f, double lf, double cfm1) {
  const double gv = __dadd_rn(f, lf);
  return __fma_rn(cfm1, gv, gv);
}

template <typename T>
struct EArgs {
  const T* B[4];
  const T* Z[4];
  const T* F1[4];
  const T* Fn[4];
  const T* Snold[4];
  T* Snm_w[4];  // in: S_{n-2}; out: S (new level n-1 after rotation)
  T* Fnm_w[4];  // in: F_{n-2}; out: F2 (new level n-1)
  T* F[4];      // out: filtered u*
  double* wnl;  // (nxpp,ny,2)
  int filter;
};

template <typename T>
__device__ __forceinline__ void stageE_tile(const Geo& g, const EArgs<T>& a, const Coefs& c) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = g.N;
  double* sL = (double*)smraw;  // N*N, L - I in FP64 (see below)
  T* sD = (T*)(sL + N * N);     // N*N
  T* tz = sD + N * N;           // N*kTX: Z tile
  T* tf = tz + N * kTX;         // N*kTX: F* tile
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    sD[t] = (T)g.D[t];
    sL[t] = g.Lfil[t] - (t / N == t % N ? 1.0 : 0.0);
  }
  const int q = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * kTX + lane;
  const int j = blockIdx.y % g.ny, ks = blockIdx.y / g.ny;
  const bool act = i < g.nxpp;
  for (int k = w; k < N; k += kTW) tz[k * kTX + lane] = act ? a.Z[q][fidx<T>(g, i, j, ks * N + k)] : (T)0;
  __syncthreads();
  const T fac = (T)g.hfac[ks];
  const T f1 = (T)c.fac1, f2 = (T)c.fac2, f3 = (T)c.fac3;
  for (int k1 = w; k1 < N; k1 += kTW) {
    T fsv = 0;
    if (act) {
      const int kk = ks * N + k1;
      const size_t p = fidx<T>(g, i, j, kk);
      const T* dr = sD + k1 * N;
      T s = 0;
#pragma unroll 4
      for (int k2 = 0; k2 < N; ++k2) s += dr[k2] * tz[k2 * kTX + lane];
      const T S = a.B[q][p] + s * fac;
      const T sn = a.Snold[q][p];
      const T snm = a.Snm_w[q][p];
      if (q == 2 && ((kk == 0) || (kk == g.nz - 1))) {
        const int side = kk == 0 ? 0 : 1;
        a.wnl[(size_t)i + (size_t)g.nxpp * ((size_t)j + (size_t)g.ny * side)] =
            (double)f1 * (double)S + (double)f2 * (double)sn + (double)f3 * (double)snm;
      }
      const T se = f1 * S + f2 * sn + f3 * snm;
      const T F2 = proj_val<T>(g, a.F1[q], i, j, kk);
      const T fn = a.Fn[q][p];
      const T fnm = a.Fnm_w[q][p];
      fsv = bdf_combine<T>(c, se, F2, fn, fnm);
      a.Snm_w[q][p] = S;
      a.Fnm_w[q][p] = F2;
    }
    tf[k1 * kTX + lane] = fsv;
  }
  __syncthreads();
  if (!act) return;
  // The Legendre filter acts on the state itself every step: L - I has O(1)
  // entries (a projector onto the damped modes), so FP32 entries would add
  // the same rounding error to the state each step.  It runs in FP64 with
  // one rounding of the result; cf - 1 is small for the energetic modes.
  const double cfm1 = a.filter ? g.cfour[(size_t)j * g.nxhp + (i >> 1)] - 1.0 : 0.0;
  for (int k1 = w; k1 < N; k1 += kTW) {
    T o;
    if (a.filter) {
      const double* lr = sL + k1 * N;
      double s = 0;
#pragma unroll 4
      for (int k2 = 0; k2 < N; ++k2) s += lr[k2] * (double)tf[k2 * kTX + lane];
      const double gv = (double)tf[k1 * kTX + lane] + s;  // L f = f + (L - I) f
      o = (T)(gv + cfm1 * gv);                            // cf g = g + (cf - 1) g
    } else {
      o = tf[k1 * kTX + lane];
    }
    a.F[q][fidx<T>(g, i, j, ks * N + k1)] = o;
  }
}

// z operators of the register-column kernels: kernel parameters, i.e. served
// from the constant bank
template <typename T, int NM>
struct ZOp {
  T D[NM * NM];       // D[k1*NM + k2], zero outside N x N
  double L[NM * NM];  // precombined Legendre filter minus the identity, same layout (FP64, see k_stageE)
};
// The tiled K_E kernels.  FP32 fields: at most 32 registers so that 8 CTAs
// fit on an SM (the kernel waits on global loads, more resident warps pay);
// FP64 fields: the compiler's own allocation.
template <typename T>
__global__ void __launch_bounds__(kTX* kTW) k_stageE(Geo g, EArgs<T> a, Coefs c) {
  stageE_tile<T>(g, a, c);
}
static __global__ void __launch_bounds__(kTX* kTW, 8) k_stageE_f32(Geo g, EArgs<float> a, Coefs c) {
  stageE_tile<float>(g, a, c);
}

// ---------------------------------------------------------------------------
// Register-column variants of K_A and K_E for N <= 33.  A thread owns one
// (x, y) point of one subdomain and keeps its N values of the column in
// registers; thread t addresses element t of every z-plane, so each warp
// reads and writes 128-byte contiguous runs.  The N x N operators (D and the
// precombined filter minus the identity, zero-padded to NM x NM; a filter
// close to the identity is applied as f + (L - I) f so that rounding its
// entries does not bias every step) are kernel parameters, i.e. they
// sit in the constant bank, and the fully unrolled products take them as
// immediate operands: about one instruction per multiply-add.
// ---------------------------------------------------------------------------

template <typename T, int NM>
__global__ void __launch_bounds__(128) k_stageA_r(Geo g, const __grid_constant__ ZOp<T, NM> op,
                                                   const T* __restrict__ F0, const T* __restrict__ F1_,
                                                   const T* __restrict__ F2_, const T* __restrict__ F3_,
                                                   T* __restrict__ O0, T* __restrict__ O1, T* __restrict__ O2,
                                                   T* __restrict__ O3, T* __restrict__ Z0, T* __restrict__ Z1,
                                                   T* __restrict__ Z2, T* __restrict__ Z3, int proj,
                                                   int* __restrict__ err) {
  const int q = blockIdx.z, ks = blockIdx.y, N = g.N;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.plane) return;
  const int i = (int)(t % g.nxpp), j = (int)(t / g.nxpp);
  const T* F = q == 0 ? F0 : q == 1 ? F1_ : q == 2 ? F2_ : F3_;
  T* O = q == 0 ? O0 : q == 1 ? O1 : q == 2 ? O2 : O3;
  T* Z = q == 0 ? Z0 : q == 1 ? Z1 : q == 2 ? Z2 : Z3;
  const bool wzero = q == 2 && j == 0 && i < 2;  // wc(1,1,:) = 0, solver.f:66-69
  // the projection changes only the kx = 0 and Nyquist columns: every other
  // point is a plain copy, read and written with fixed plane strides
  const bool special = proj && (i < 2 || i >= g.nx);
  const size_t pl = g.plane, o0 = (size_t)(ks * N) * pl + t;
  T col[NM];
  bool bad = false;
  if (!special) {
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      T x = 0;
      if (k < N) {
        x = F[o0 + (size_t)k * pl];
        bad |= !isfinite(x);
        if (wzero) x = (T)0;
        O[o0 + (size_t)k * pl] = x;
      }
      col[k] = x;
    }
  } else {
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      T x = 0;
      if (k < N) {
        x = proj_val<T>(g, F, i, j, ks * N + k);
        bad |= !isfinite(x);
        if (wzero) x = (T)0;
        O[o0 + (size_t)k * pl] = x;
      }
      col[k] = x;
    }
  }
  if (bad) err[0] = 1;  // the state of the last step holds a NaN or Inf
  if (Z == nullptr) return;
  const T fac = (T)g.hfac[ks];
#pragma unroll
  for (int k1 = 0; k1 < NM; ++k1) {
    if (k1 < N) {
      T s = 0;
#pragma unroll
      for (int k2 = 0; k2 < NM; ++k2) s = fma_t(op.D[k1 * NM + k2], col[k2], s);
      Z[o0 + (size_t)k1 * pl] = mul_t(s, fac);
    }
  }
}

template <typename T, int NM>
__global__ void __launch_bounds__(128) k_stageE_r(Geo g, EArgs<T> a, Coefs c, const __grid_constant__ ZOp<T, NM> op) {
  const int q = blockIdx.z, ks = blockIdx.y, N = g.N;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.plane) return;
  const int i = (int)(t % g.nxpp), j = (int)(t / g.nxpp);
  T zc[NM];
#pragma unroll
  for (int k = 0; k < NM; ++k) zc[k] = k < N ? a.Z[q][(size_t)(ks * N + k) * g.plane + t] : (T)0;
  const T fac = (T)g.hfac[ks];
  const T f1 = (T)c.fac1, f2 = (T)c.fac2, f3 = (T)c.fac3;
  const T* Bq = a.B[q];
  const T* Snq = a.Snold[q];
  const T* F1q = a.F1[q];
  const T* Fnq = a.Fn[q];
  T* Snmq = a.Snm_w[q];
  T* Fnmq = a.Fnm_w[q];
  // Rolling window: the inputs of row k1+PF are loaded before the stores of
  // row k1, so the loads of several rows are in flight at once (the pointers
  // are not known to be distinct, so the compiler would not hoist them).
  constexpr int PF = 4;
  T wb[PF], wsn[PF], wsnm[PF], wf2[PF], wfn[PF], wfnm[PF];
#pragma unroll
  for (int k1 = 0; k1 < PF; ++k1) {
    if (k1 < N) {
      const int kk = ks * N + k1;
      const size_t p = (size_t)kk * g.plane + t;
      wb[k1] = Bq[p];
      wsn[k1] = Snq[p];
      wsnm[k1] = Snmq[p];
      wf2[k1] = proj_val<T>(g, F1q, i, j, kk);
      wfn[k1] = Fnq[p];
      wfnm[k1] = Fnmq[p];
    }
  }
  T fs[NM];
#pragma unroll
  for (int k1 = 0; k1 < NM; ++k1) {
    T fsv = 0;
    if (k1 < N) {
      const int sl = k1 % PF;
      const T b = wb[sl], sn = wsn[sl], snm = wsnm[sl], F2 = wf2[sl], fn = wfn[sl], fnm = wfnm[sl];
      if (k1 + PF < NM && k1 + PF < N) {
        const int kn = ks * N + k1 + PF;
        const size_t pn = (size_t)kn * g.plane + t;
        wb[sl] = Bq[pn];
        wsn[sl] = Snq[pn];
        wsnm[sl] = Snmq[pn];
        wf2[sl] = proj_val<T>(g, F1q, i, j, kn);
        wfn[sl] = Fnq[pn];
        wfnm[sl] = Fnmq[pn];
      }
      const int kk = ks * N + k1;
      const size_t p = (size_t)kk * g.plane + t;
      T s = 0;
#pragma unroll
      for (int k2 = 0; k2 < NM; ++k2) s += op.D[k1 * NM + k2] * zc[k2];
      const T S = b + s * fac;
      if (q == 2 && ((kk == 0) || (kk == g.nz - 1)))
        a.wnl[t + (kk == 0 ? 0 : g.plane)] = (double)f1 * (double)S + (double)f2 * (double)sn + (double)f3 * (double)snm;
      const T se = f1 * S + f2 * sn + f3 * snm;
      fsv = bdf_combine<T>(c, se, F2, fn, fnm);
      Snmq[p] = S;
      Fnmq[p] = F2;
    }
    fs[k1] = fsv;
  }
  const double cfm1 = a.filter ? g.cfour[(size_t)j * g.nxhp + (i >> 1)] - 1.0 : 0.0;
#pragma unroll
  for (int k1 = 0; k1 < NM; ++k1) {
    if (k1 < N) {
      T o;
      if (a.filter) {
        double s = 0;
#pragma unroll
        for (int k2 = 0; k2 < NM; ++k2) s += op.L[k1 * NM + k2] * (double)fs[k2];  // (L - I) f in FP64
        const double gv = (double)fs[k1] + s;
        o = (T)(gv + cfm1 * gv);
      } else {
        o = fs[k1];
      }
      a.F[q][(size_t)(ks * N + k1) * g.plane + t] = o;
    }
  }
}

// rotational viscous term at the walls (solver.f:318-394, rotvisc 1210-1253):
// wviscrot = -nu * (fac1 rot(n) + fac2 rot(n-1) + fac3 rot(n-2)),
// rot = (kx^2+ky^2) w + i kx du/dz + i ky dv/dz at k0.  A CTA takes 32 columns of
// one y index and wall; its six warps form du/dz and dv/dz of the three levels,
// each the chain of N multiply-adds, and the first warp puts them together.
template <typename T>
__global__ void __launch_bounds__(192) k_wviscrot(Geo g, const T* __restrict__ u1, const T* __restrict__ v1,
                                                  const T* __restrict__ w1, const T* __restrict__ un,
                                                  const T* __restrict__ vn, const T* __restrict__ wn,
                                                  const T* __restrict__ unm, const T* __restrict__ vnm,
                                                  const T* __restrict__ wnm, Coefs c, double xnu,
                                                  double* __restrict__ wvr) {
  __shared__ double sd[6][2][32];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5, l = wq >> 1;
  const int ii = blockIdx.x * 32 + lane, j = blockIdx.y, side = blockIdx.z;
  const bool act = ii < g.nxhp;
  const int N = g.N, ks = side == 0 ? 0 : g.ns - 1, k0 = side == 0 ? 0 : N - 1;
  const double fac = g.hfac[ks];
  // level n goes through the projection; only the kx = 0 and Nyquist columns change
  const bool special = l == 0 && (ii == 0 || ii == g.nxh);
  const T* F = (wq & 1) ? (l == 0 ? v1 : l == 1 ? vn : vnm) : (l == 0 ? u1 : l == 1 ? un : unm);
  double dr = 0, di = 0;
  if (act) {
    const double* D = g.D + (size_t)k0 * N;
    if (special) {
      for (int k2 = 0; k2 < N; ++k2) {
        dr += D[k2] * (double)proj_val<T>(g, F, 2 * ii, j, ks * N + k2);
        di += D[k2] * (double)proj_val<T>(g, F, 2 * ii + 1, j, ks * N + k2);
      }
    } else {
      typedef typename Pair<T>::t P2;
      const T* p = F + fidx<T>(g, 2 * ii, j, ks * N);
#pragma unroll 8
      for (int k2 = 0; k2 < N; ++k2) {
        const P2 v = *(const P2*)(p + (size_t)k2 * g.plane);
        dr += D[k2] * (double)v.x;
        di += D[k2] * (double)v.y;
      }
    }
  }
  sd[wq][0][lane] = dr * fac;
  sd[wq][1][lane] = di * fac;
  __syncthreads();
  if (wq != 0 || !act) return;
  const double xw = g.xw[ii], yw = g.yw[j];
  const int kk0 = ks * N + k0;
  double rr = 0, ri = 0;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const T* W = m == 0 ? w1 : m == 1 ? wn : wnm;
    const double wr = m == 0 ? (double)proj_val<T>(g, W, 2 * ii, j, kk0) : (double)W[fidx<T>(g, 2 * ii, j, kk0)];
    const double wi = m == 0 ? (double)proj_val<T>(g, W, 2 * ii + 1, j, kk0) : (double)W[fidx<T>(g, 2 * ii + 1, j, kk0)];
    const double dur = sd[2 * m][0][lane], dui = sd[2 * m][1][lane], dvr = sd[2 * m + 1][0][lane],
                 dvi = sd[2 * m + 1][1][lane];
    const double re = xw * xw * wr + yw * yw * wr - xw * dui - yw * dvi;
    const double im = xw * xw * wi + yw * yw * wi + xw * dur + yw * dvr;
    const double f = m == 0 ? c.fac1 : m == 1 ? c.fac2 : c.fac3;
    rr += f * re;
    ri += f * im;
  }
  const size_t base = (size_t)g.nxpp * ((size_t)j + (size_t)g.ny * side) + 2 * ii;
  wvr[base] = -(xnu * rr);
  wvr[base + 1] = -(xnu * ri);
}

// ===========================================================================
// Band factorisation (penalty.f:403-634 assembly, band_lu.f:19-34 packing,
// bandludcmp.f:238-440 SGBTF2).  The arithmetic follows the reference order with
// no fused multiply-add, so the factors equal the CPU ones bit for bit.  Assembly: one
// CTA per system, a warp per subdomain.
// ===========================================================================
struct SysDesc {
  double eps;
  double tau1_bot, tau2_top;  // for the RHS boundary rows
  int ifbcbot, ifbctop;
  int pad[2];
};

struct FactorArgs {
  const SysDesc* sys = nullptr;
  const double* pen = nullptr;  // per system: 6*ns (alpha,beta,gamma,delta,tau1,tau2)
  double* ab = nullptr;         // per system: ldab*nz
  int nsys = 0;
  const double* D = nullptr;
  const double* D2 = nullptr;
  const double* zh = nullptr;  // ns
};

__device__ __forceinline__ double& ABr(double* ab, int ldab, int r, int c) {
  return ab[(size_t)(r - 1) + (size_t)ldab * (size_t)(c - 1)];
}

static __global__ void k_assemble_band(Geo g, FactorArgs fa) {
  const int s = blockIdx.x, lane = threadIdx.x & 31;
  const int n = g.nz, N = g.N, ns = g.ns, kl = N, ku = N, ldab = 2 * kl + ku + 1;
  double* ab = fa.ab + (size_t)s * ldab * n;
  const double eps = fa.sys[s].eps;
  const double* pen = fa.pen + (size_t)s * 6 * ns;
  const double *pa = pen, *pb = pen + ns, *pg = pen + 2 * ns, *pd = pen + 3 * ns, *pt1 = pen + 4 * ns,
               *pt2 = pen + 5 * ns;
  const double* d = fa.D;
  const double* d2 = fa.D2;
  // zero the band
  for (size_t t = threadIdx.x; t < (size_t)ldab * n; t += blockDim.x) ab[t] = 0.0;
  __syncthreads();
  // A(r,c) 0-based -> band row kl+ku+1+r-c (1-based), column c+1
#define AEL(r, c) ABr(ab, ldab, kl + ku + 1 + (r) - (c), (c) + 1)
  for (int ks = threadIdx.x >> 5; ks < ns; ks += blockDim.x >> 5) {  // a warp per subdomain: its own rows
    const double ybar = fa.zh[ks];
    const double ybarl = ks > 0 ? fa.zh[ks - 1] : 0.0;
    const double ybarr = ks < ns - 1 ? fa.zh[ks + 1] : 0.0;
    const int km = ks * N;
    const double h2 = rmul(2.0 / ybar, 2.0 / ybar);
    const double eh = rmul(eps, h2);
    for (int t = lane; t < N * N; t += 32) {
      int k1 = t / N, k2 = t % N;
      AEL(km + k1, km + k2) = -rmul(eh, d2[k1 * N + k2]);
    }
    __syncwarp();
    for (int k1 = lane; k1 < N; k1 += 32) AEL(km + k1, km + k1) = radd(AEL(km + k1, km + k1), 1.0);
    __syncwarp();
    if (lane == 0) AEL(km, km) = radd(AEL(km, km), rmul(pt1[ks], pa[ks]));
    __syncwarp();
    {
      double cf = -__ddiv_rn(rmul(rmul(rmul(pt1[ks], pb[ks]), eps), 2.0), ybar);
      for (int k = lane; k < N; k += 32) AEL(km, km + k) = radd(AEL(km, km + k), rmul(cf, d[0 * N + k]));
    }
    __syncwarp();
    if (lane == 0) AEL(km + N - 1, km + N - 1) = radd(AEL(km + N - 1, km + N - 1), rmul(pt2[ks], pg[ks]));
    __syncwarp();
    {
      double cf = __ddiv_rn(rmul(rmul(rmul(pt2[ks], pd[ks]), eps), 2.0), ybar);
      for (int k = lane; k < N; k += 32)
        AEL(km + N - 1, km + k) = radd(AEL(km + N - 1, km + k), rmul(cf, d[(N - 1) * N + k]));
    }
    __syncwarp();
    if (ns > 1 && ks != 0) {
      if (lane == 0) AEL(km, km) = rsub(AEL(km, km), rmul(rmul(0.5, pt1[ks]), pa[ks]));
      __syncwarp();
      double cf = __ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt1[ks]), pb[ks]), eps), 2.0), ybar);
      for (int k = lane; k < N; k += 32) AEL(km, km + k) = radd(AEL(km, km + k), rmul(cf, d[0 * N + k]));
      __syncwarp();
      for (int k = lane; k < N; k += 32) AEL(km, km - N + k) = 0.0;
      __syncwarp();
      if (lane == 0) AEL(km, km - 1) = -rmul(rmul(0.5, pt1[ks]), pa[ks]);
      __syncwarp();
      cf = __ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt1[ks]), pb[ks]), eps), 2.0), ybarl);
      for (int k = lane; k < N; k += 32)
        AEL(km, km - N + k) = radd(AEL(km, km - N + k), rmul(cf, d[(N - 1) * N + k]));
      __syncwarp();
    }
    if (ns > 1 && ks != ns - 1) {
      if (lane == 0) AEL(km + N - 1, km + N - 1) = rsub(AEL(km + N - 1, km + N - 1), rmul(rmul(0.5, pt2[ks]), pg[ks]));
      __syncwarp();
      double cf = -__ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt2[ks]), pd[ks]), eps), 2.0), ybar);
      for (int k = lane; k < N; k += 32)
        AEL(km + N - 1, km + k) = radd(AEL(km + N - 1, km + k), rmul(cf, d[(N - 1) * N + k]));
      __syncwarp();
      // a(km+1, km+nzloc+k) = 0: outside the band for nzloc >= 2 except the
      // row's own band part, which is zero here already
      if (lane == 0) AEL(km + N - 1, km + N) = rsub(AEL(km + N - 1, km + N), rmul(rmul(0.5, pt2[ks]), pg[ks]));
      __syncwarp();
      cf = -__ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt2[ks]), pd[ks]), eps), 2.0), ybarr);
      for (int k = lane; k < N; k += 32)
        AEL(km + N - 1, km + N + k) = radd(AEL(km + N - 1, km + N + k), rmul(cf, d[0 * N + k]));
      __syncwarp();
    }
  }
#undef AEL
}

// SGBTF2 (bandludcmp.f:238-440), one CTA per system.  The columns a step touches (j .. j + kl
// + ku) live in a ring in shared memory; the next ones arrive by cp.async eight steps
// ahead, and a finished column goes back to global memory.  In a step, lanes take the rows and
// warps the columns of the update; warp 0 updates column j + 1 first, finds its pivot and
// forms the next multipliers while the other warps finish, so a step is one barrier and
// no dependent access to global memory.  Bound by warp 0's chain (update, maximum over lanes,
// reciprocal).  The arithmetic of every element and its order are the reference's.
constexpr int kLuThreads = 256, kLuAhead = 8;
__host__ __device__ inline int lu_ring(int N) { return 2 * N + 2 + kLuAhead; }
__host__ __device__ inline size_t lu_smem(int N) {
  return ((size_t)lu_ring(N) * (3 * N + 1) + 2 * (N + 2)) * sizeof(double);
}
// Pivot and multipliers of column j (cj, updated by the steps before) by one warp: the
// first row of the largest |a|, rows kv .. kv + km; the multipliers go to lb[1 .. km]
// and the column.  Returns the pivot's row, or -1 - row for a zero pivot.
static __device__ __forceinline__ int lu_pivot(double* cj, double* lb, int kv, int km, int lane) {
  double best = -1.0;
  int bi = 1 << 30;
  for (int i = lane; i <= km; i += 32) {
    const double v = fabs(cj[kv + i]);
    if (v > best) {
      best = v;
      bi = i;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob > best || (ob == best && oi < bi)) {
      best = ob;
      bi = oi;
    }
  }
  if (bi > km) bi = 0;  // only NaNs
  const double piv = cj[kv + bi], top = cj[kv];
  __syncwarp();
  if (piv == 0.0) return -1 - bi;
  const double rcp = km > 0 ? __ddiv_rn(1.0, piv) : 0.0;
  for (int i = 1 + lane; i <= km; i += 32) {
    const double l = rmul(rcp, i == bi ? top : cj[kv + i]);
    lb[i] = l;
    cj[kv + i] = l;
  }
  if (lane == 0) cj[kv] = piv;
  __syncwarp();
  return bi;
}
static __global__ void __launch_bounds__(kLuThreads) k_band_lu(int n, int N, double* __restrict__ abs_, int* __restrict__ ipivs,
                                                               int* __restrict__ infos) {
  extern __shared__ __align__(16) double sml[];
  __shared__ int sjp[2];
  const int kl = N, ku = N, kv = kl + ku, ldab = 2 * kl + ku + 1, W = lu_ring(N);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nth = blockDim.x, nw = nth >> 5;
  double* ab = abs_ + (size_t)blockIdx.x * ldab * n;
  int* ipiv = ipivs + (size_t)blockIdx.x * n;
  double* ring = sml;                    // column j at ring + (j % W) ldab
  double* lbs = ring + (size_t)W * ldab;  // multipliers of steps of either parity
  // column c (0-based): the kl fill rows start as 0
  auto fetch = [&](int c, int slot) {
    if (c < n) {
      double* d = ring + (size_t)slot * ldab;
      const double* s = ab + (size_t)c * ldab;
      for (int r = tid; r < ldab; r += nth) {
        if (r < kl)
          d[r] = 0.0;
        else
          cp_async_c<float2>((float2*)(d + r), (const float2*)(s + r));
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int c = 0; c < kv + 1 + kLuAhead; ++c) fetch(c, c);
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kLuAhead) : "memory");  // columns <= kv
  __syncthreads();
  if (wid == 0) {
    const int p = lu_pivot(ring, lbs, kv, min(kl, n - 1), lane);
    if (lane == 0) {
      sjp[0] = p;
      ipiv[0] = (p >= 0 ? p : -1 - p) + 1;
    }
  }
  int ju = 0, info = 0, sj = 0;  // last column touched so far (0-based), slot of column j
  int sf = kv + 1 + kLuAhead;    // slot of column j + kv + 1 + kLuAhead: held column j - 1
  if (sf >= W) sf -= W;
  for (int j = 0; j < n; ++j) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kLuAhead - 1) : "memory");  // columns <= j + kv + 1
    __syncthreads();  // step j - 1 and the pivot of column j are done
    fetch(j + kv + 1 + kLuAhead, sf);
    const int km = min(kl, n - 1 - j), jp = sjp[j & 1];
    const double* lb = lbs + (j & 1) * (N + 2);
    const double* cj = ring + (size_t)sj * ldab;
    if (jp >= 0) {
      ju = max(ju, min(j + ku + jp, n - 1));
      // rows i = 1 + lane (and 33 + lane) of columns j + 1 .. ju; warp 0 takes column j + 1 alone
      const int i0 = 1 + lane, i1 = 33 + lane;
      const double l0 = i0 <= km ? lb[i0] : 0.0, l1 = i1 <= km ? lb[i1] : 0.0;
      for (int cc = wid == 0 ? 1 : 1 + wid; cc <= ju - j; cc += wid == 0 ? 1 << 20 : nw - 1) {
        int sl = sj + cc;
        if (sl >= W) sl -= W;
        double* col = ring + (size_t)sl * ldab + kv - cc;  // row i of the step at col[i]
        const double y = col[jp], t0 = col[0];
        const double x0 = i0 <= km ? (i0 == jp ? t0 : col[i0]) : 0.0, x1 = i1 <= km ? (i1 == jp ? t0 : col[i1]) : 0.0;
        __syncwarp();
        const double temp = -y;
        if (i0 <= km) col[i0] = y != 0.0 ? radd(x0, rmul(l0, temp)) : x0;
        if (i1 <= km) col[i1] = y != 0.0 ? radd(x1, rmul(l1, temp)) : x1;
        if (lane == 0) col[0] = y;
        __syncwarp();
      }
    } else if (info == 0) {
      info = j + 1;
    }
    if (wid == 0 && j + 1 < n) {
      int sn = sj + 1;
      if (sn >= W) sn -= W;
      const int p = lu_pivot(ring + (size_t)sn * ldab, lbs + ((j + 1) & 1) * (N + 2), kv, min(kl, n - 2 - j), lane);
      if (lane == 0) {
        sjp[(j + 1) & 1] = p;
        ipiv[j + 1] = j + 1 + (p >= 0 ? p : -1 - p) + 1;
      }
    }
    for (int r = tid; r < ldab; r += nth) ab[(size_t)j * ldab + r] = cj[r];
    if (++sj >= W) sj -= W;
    if (++sf >= W) sf -= W;
  }
  if (tid == 0) infos[blockIdx.x] = info;
}

// ===========================================================================
// Warp-cooperative banded solve (SGBTRS 'N' + STBSV, bandludcmp.f:883-1069)
// for nr right-hand sides b[r*n + row] in shared memory; same arithmetic as
// the reference (no FMA) so results equal the CPU ones bit for bit.
// ===========================================================================
static __device__ void band_solve_warp(const double* __restrict__ ab, const int* __restrict__ ipiv, double* b, int nr,
                                int n, int kl, int ku, int lane) {
  // The factor entries a step needs do not depend on the data, so they are
  // fetched PF steps ahead into a register ring (indices are compile-time
  // constants after unrolling), hiding the global-memory latency that would
  // otherwise stall every step of the sequential sweep.
  constexpr int PF = 8;
  const int ldab = 2 * kl + ku + 1;
  const int kd = ku + kl + 1;
  const int i0 = lane + 1, i1 = lane + 33;
  int rl[PF];
  double rm0[PF], rm1[PF];
#pragma unroll
  for (int d = 0; d < PF; ++d) {
    const int j = 1 + d;
    rl[d] = 0;
    rm0[d] = rm1[d] = 0.0;
    if (j <= n - 1) {
      const int lm = min(kl, n - j);
      const double* col = ab + (size_t)ldab * (j - 1);
      rl[d] = __ldg(ipiv + j - 1);
      if (i0 <= lm) rm0[d] = __ldg(col + kd + i0 - 1);
      if (i1 <= lm) rm1[d] = __ldg(col + kd + i1 - 1);
    }
  }
  for (int jb = 1; jb <= n - 1; jb += PF) {
#pragma unroll
    for (int d = 0; d < PF; ++d) {
      const int j = jb + d;
      if (j <= n - 1) {
        const int lm = min(kl, n - j);
        const int l = rl[d];
        const double m0 = rm0[d], m1 = rm1[d];
        const int jn = j + PF;
        if (jn <= n - 1) {
          const int lmn = min(kl, n - jn);
          const double* coln = ab + (size_t)ldab * (jn - 1);
          rl[d] = __ldg(ipiv + jn - 1);
          rm0[d] = (i0 <= lmn) ? __ldg(coln + kd + i0 - 1) : 0.0;
          rm1[d] = (i1 <= lmn) ? __ldg(coln + kd + i1 - 1) : 0.0;
        }
        for (int r = 0; r < nr; ++r) {
          double* br = b + (size_t)r * n;
          const double bj = br[j - 1];
          const double bl = br[l - 1];
          const double y = (l != j) ? bl : bj;
          double nv0 = 0, nv1 = 0;
          if (i0 <= lm) {
            int row = j + i0;
            double old = (row == l) ? bj : br[row - 1];
            nv0 = (y != 0.0) ? radd(old, rmul(m0, -y)) : old;
          }
          if (i1 <= lm) {
            int row = j + i1;
            double old = (row == l) ? bj : br[row - 1];
            nv1 = (y != 0.0) ? radd(old, rmul(m1, -y)) : old;
          }
          __syncwarp();
          if (i0 <= lm) br[j + i0 - 1] = nv0;
          if (i1 <= lm) br[j + i1 - 1] = nv1;
          if (lane == 0) br[j - 1] = y;
          __syncwarp();
        }
      }
    }
  }
  // back substitution with the upper band (STBSV)
  const int k = kl + ku, kplus1 = k + 1;
  double rdg[PF], rv0[PF], rv1[PF], rv2[PF];
  // lane's rows below j are i = j-1-lane-32m; AB(kplus1-j+i, j) = col[k-1-lane-32m]
  const int o0 = k - 1 - lane, o1 = k - 1 - lane - 32, o2 = k - 1 - lane - 64;
#pragma unroll
  for (int d = 0; d < PF; ++d) {
    const int j = n - d;
    rdg[d] = rv0[d] = rv1[d] = rv2[d] = 0.0;
    if (j >= 1) {
      const double* col = ab + (size_t)ldab * (j - 1);
      rdg[d] = __ldg(col + kplus1 - 1);
      if (o0 >= 0) rv0[d] = __ldg(col + o0);
      if (o1 >= 0) rv1[d] = __ldg(col + o1);
      if (o2 >= 0) rv2[d] = __ldg(col + o2);
    }
  }
  for (int jb = n; jb >= 1; jb -= PF) {
#pragma unroll
    for (int d = 0; d < PF; ++d) {
      const int j = jb - d;
      if (j >= 1) {
        const double dg = rdg[d];
        const double v0 = rv0[d], v1 = rv1[d], v2 = rv2[d];
        const int jn = j - PF;
        if (jn >= 1) {
          const double* coln = ab + (size_t)ldab * (jn - 1);
          rdg[d] = __ldg(coln + kplus1 - 1);
          rv0[d] = (o0 >= 0) ? __ldg(coln + o0) : 0.0;
          rv1[d] = (o1 >= 0) ? __ldg(coln + o1) : 0.0;
          rv2[d] = (o2 >= 0) ? __ldg(coln + o2) : 0.0;
        }
        const int lo = max(1, j - k);
        const int ia = j - 1 - lane, ib = ia - 32, ic = ia - 64;
        for (int r = 0; r < nr; ++r) {
          double* br = b + (size_t)r * n;
          double xj = br[j - 1];
          if (xj != 0.0) {
            xj = __ddiv_rn(xj, dg);
            double n0 = 0, n1 = 0, n2 = 0;
            if (ia >= lo) n0 = rsub(br[ia - 1], rmul(xj, v0));
            if (ib >= lo) n1 = rsub(br[ib - 1], rmul(xj, v1));
            if (ic >= lo) n2 = rsub(br[ic - 1], rmul(xj, v2));
            __syncwarp();
            if (ia >= lo) br[ia - 1] = n0;
            if (ib >= lo) br[ib - 1] = n1;
            if (ic >= lo) br[ic - 1] = n2;
            if (lane == 0) br[j - 1] = xj;
            __syncwarp();
          }
        }
      }
    }
  }
}

// Legendre filter of solution columns (filtering.f:729-808, filter_legenpen),
// same order of operations as the reference.  One lane per subdomain column.
static __device__ void legen_filter_cols(double* b, int nr, int n, int N, int ns, const double* __restrict__ wg,
                                  const double* __restrict__ alpol, const double* __restrict__ sigma, int lane) {
  const int nzm = N - 1;
  for (int t = lane; t < nr * ns; t += 32) {
    double* f = b + (size_t)(t / ns) * n + (size_t)(t % ns) * N;
    double af[kMaxN];
    for (int kk = 0; kk <= nzm; ++kk) {
      double sum = 0.0;
      for (int k1 = 0; k1 < N; ++k1) sum = radd(sum, rmul(rmul(wg[k1], f[k1]), alpol[kk * N + k1]));
      double a = (kk == nzm) ? rmul(rmul(0.5, (double)nzm), sum) : rmul((double)kk + 0.5, sum);
      af[kk] = rmul(a, sigma[kk]);
    }
    for (int k1 = 0; k1 < N; ++k1) {
      double sum = 0.0;
      for (int kk = 0; kk <= nzm; ++kk) sum = radd(sum, rmul(af[kk], alpol[kk * N + k1]));
      f[k1] = sum;
    }
  }
}

struct SolveTabs {
  const double* ab;      // ldab*nz per system
  const int* ipiv;       // nz per system
  const SysDesc* sys;
  const int* col_sys;    // per column (j*nxhp+ii): system index (-1: none)
  const double* wg;
  const double* alpol;   // N*N: alpol[k*N + k1] = P_k(z_k1)
  const double* sigma;   // N
  const double* meang;   // nz: 1 - fzgaus(z) (mean-u damping) or null
  const int* col_order;  // columns sorted by kx^2+ky^2, so neighbouring warps share a factor
};

// K_G: viscous/diffusive solves.  role 0: u and v (4 RHS, one factor),
// role 1: w, role 2: rho.  Warp per column.
template <typename T>
__global__ void k_visc(Geo g, SolveTabs tb, T* __restrict__ F0, T* __restrict__ F1, double rdiv, int role, int cpen,
                       int meanu) {
  extern __shared__ __align__(16) double sm[];
  const int warps = blockDim.x / 32;
  const int wid = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int cw = blockIdx.x * warps + wid;
  const int ncol = g.nxhp * g.ny;
  if (cw >= ncol) return;
  const int c = tb.col_order[cw];
  const int n = g.nz, N = g.N;
  const int nr = role == 0 ? 4 : 2;
  double* b = sm + (size_t)wid * 4 * n;
  const int j = c / g.nxhp, ii = c % g.nxhp;
  const bool lzero = (ii == 0 && j == 0);
  const int s = tb.col_sys[c];
  T* Fs[2] = {F0, F1};
  if (s < 0) {  // w of the (0,0) mode is zero (calcuvwt.f:488-496)
    for (int k = lane; k < n; k += 32) {
      F0[fidx<T>(g, 2 * ii, j, k)] = 0;
      F0[fidx<T>(g, 2 * ii + 1, j, k)] = 0;
    }
    return;
  }
  const SysDesc sd = tb.sys[s];
  const double eps = sd.eps;
  for (int r = 0; r < nr; ++r) {
    T* F = Fs[r / 2];
    int part = r & 1;
    for (int k = lane; k < n; k += 32) {
      double x = (double)F[fidx<T>(g, 2 * ii + part, j, k)];
      double rh = -__ddiv_rn(x, rdiv);
      b[(size_t)r * n + k] = -rmul(rh, eps);
    }
  }
  __syncwarp();
  if (lane == 0) {
    // homogeneous boundary values: Dirichlet adds tau*0, Neumann tau*0*eps
    for (int r = 0; r < nr; ++r) {
      double* br = b + (size_t)r * n;
      br[0] = sd.ifbcbot == 0 ? radd(br[0], rmul(sd.tau1_bot, 0.0)) : rsub(br[0], rmul(rmul(sd.tau1_bot, 0.0), eps));
      br[n - 1] = sd.ifbctop == 0 ? radd(br[n - 1], rmul(sd.tau2_top, 0.0))
                                  : radd(br[n - 1], rmul(rmul(sd.tau2_top, 0.0), eps));
    }
  }
  __syncwarp();
  const int ldab = 3 * N + 1;
  band_solve_warp(tb.ab + (size_t)s * ldab * n, tb.ipiv + (size_t)s * n, b, nr, n, N, N, lane);
  if (cpen) {
    legen_filter_cols(b, nr, n, N, g.ns, tb.wg, tb.alpol, tb.sigma, lane);
    __syncwarp();
  }
  for (int r = 0; r < nr; ++r) {
    T* F = Fs[r / 2];
    int part = r & 1;
    for (int k = lane; k < n; k += 32) {
      double x = b[(size_t)r * n + k];
      if (role == 0 && r < 2 && lzero && meanu) x = rmul(tb.meang[k], x);
      F[fidx<T>(g, 2 * ii + part, j, k)] = (T)x;
    }
  }
}

// ===========================================================================
// Block-inverse solve of the viscous / diffusive penalty systems.
// The penalty matrix A is block diagonal in N x N subdomain blocks A_ks, plus
// coupling in the first row of block ks to all of block ks-1 (vector c_ks)
// and in its last row to all of block ks+1 (vector d_ks).  With
// y = A_ks^-1 b_ks, p_ks = A_ks^-1 e_0, q_ks = A_ks^-1 e_{N-1}:
//     x_ks = y_ks - p_ks sigma_ks - q_ks tau_ks,
//     sigma_ks = c_ks . x_{ks-1},  tau_ks = d_ks . x_{ks+1},
// and the 2(ns-1) interface scalars solve a small dense system M z = r.
// A_ks^-1 is formed once per system (FP64 Gauss-Jordan, partial pivoting),
// stored column major per block in TI (float for the mixed path).
// ===========================================================================
struct BlockInv {
  // per system: nb distinct blocks of N*N, [block][col][row].  Subdomain ks
  // uses block bmap[ks]: a block is fixed by epsilon, the subdomain height and
  // whether it has neighbours below and above, so with equal heights the
  // interior subdomains share one inverse.
  const void* ainv;
  int nb;
  int bmap[IW_MAX_SUBD];
  const double* minv;   // per system: m*m, m = 2(ns-1), row major
  const double* pen;    // per system: 6*ns penalty parameters
  const SysDesc* sys;
  const int* col_sys;
  const int* col_order;
  const double* lvec;   // per system: m*N left vectors (see k_solve_cta)
};

// ===========================================================================
// Tables of the block-inverse solves, one CTA per system, straight from epsilon:
// penalty parameters (penalty.f:57-157), the distinct subdomain blocks and the
// coupling vectors (penalty.f:403-634, the operations of k_assemble_band in its
// order), Gauss-Jordan inverses with partial pivoting, left vectors, interface
// matrix and its inverse, the Legendre filter folded into the inverses.  Everything
// stays in shared memory until the tables are written; no band, no workspace, nothing on
// the host.  Bound by the serial pivot steps (two barriers each); a system's blocks
// are few, so several CTAs per SM hide them.
// ===========================================================================
struct BuildArgs {
  int N, ns, nb, nsys, nraw;  // nraw: systems that also keep their unfiltered inverses
  int bot, top;               // boundary conditions (0 Dirichlet, 1 Neumann)
  double c0;                  // epsilon = 1 / (ak + c0)
  double facdir, facneumn, facrobin;
  int bmap[IW_MAX_SUBD], brep[IW_MAX_SUBD];
  const double *ak, *D, *D2, *zh, *L;  // L: filter to fold in, or null
  SysDesc* sys;
  double *pen, *ainv, *ainv_raw, *lvec, *minv;
};
// penalty.f:57-157 (h_param_set, with every rounding written out)
static __device__ void d_param_set(const BuildArgs& b, int ifbc, double eps, double ybar, double& a0, double& b0,
                                   double& t0) {
  const double omega = __ddiv_rn(2., (double)((b.N + 1) * (b.N + 2)));
  if (ifbc == 0) {
    const double h = __ddiv_rn(2., ybar), fac = rmul(b.facdir, rmul(h, h));
    a0 = 1.;
    b0 = 0.;
    t0 = __ddiv_rn(rmul(fac, eps), rmul(omega, omega));
  } else if (ifbc == 1) {
    a0 = 0.;
    b0 = 1.;
    t0 = __ddiv_rn(__ddiv_rn(rmul(b.facneumn, 2.), ybar), omega);
  } else {
    a0 = 1.;
    b0 = 1.;
    const double dn = __ddiv_rn(1., rmul(omega, eps));
    const double t1 = __dsqrt_rn(radd(rmul(omega, omega), rmul(eps, omega)));
    const double t2 = rsub(rmul(2., omega), rmul(2., t1));
    const double facm = __ddiv_rn(1., eps) >= 1.e5 ? b.facrobin : 1.;
    t0 = __ddiv_rn(rmul(rmul(rmul(facm, dn), radd(eps, t2)), 2.), ybar);
  }
}
// Gauss-Jordan on the n x 2 n matrix A (right half: the identity) by nthr threads that
// meet at barrier bar; columns left of the pivot hold zeros in the pivot row and are skipped
static __device__ void gauss_jordan(double* A, int n, int* piv, double* pinv, int tid, int nthr, int bar) {
  const int lane = tid & 31, w = tid >> 5, nw = nthr >> 5, n2 = 2 * n;
  auto sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nthr) : "memory"); };
  for (int col = 0; col < n; ++col) {
    if (w == 0) {  // the first row of the largest |A(r, col)|, r >= col
      double best = -1.0;
      int bi = col;
      for (int r = col + lane; r < n; r += 32) {
        const double v = fabs(A[r * n2 + col]);
        if (v > best) {
          best = v;
          bi = r;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
        }
      }
      if (lane == 0) {
        *piv = bi;
        *pinv = __ddiv_rn(1.0, A[bi * n2 + col]);
      }
    }
    sync();
    const int bi = *piv;
    const double iv = *pinv;
    for (int c = col + tid; c < n2; c += nthr) {
      const double p = A[bi * n2 + c];
      if (bi != col) A[bi * n2 + c] = A[col * n2 + c];
      A[col * n2 + c] = rmul(p, iv);
    }
    sync();
    for (int r = w; r < n; r += nw) {
      if (r == col) continue;
      const double f = A[r * n2 + col];
      __syncwarp();
      if (f != 0.0)
        for (int c = col + lane; c < n2; c += 32) A[r * n2 + c] = __fma_rn(-f, A[col * n2 + c], A[r * n2 + c]);
    }
    sync();
  }
}
constexpr int kBuildGroups = 3;  // blocks inverted at the same time, two warps each
__host__ __device__ inline size_t build_smem(int N, int ns) {
  const size_t m = 2 * (size_t)(ns - 1);
  return ((size_t)kBuildGroups * N * 2 * N + 2 * (size_t)ns * N + 2 * m + m * 2 * m + 6 * (size_t)ns + 4) * sizeof(double);
}
static __global__ void __launch_bounds__(64 * kBuildGroups) k_build_systems(const __grid_constant__ BuildArgs b) {
  extern __shared__ __align__(16) double smb[];
  __shared__ int piv[kBuildGroups];
  __shared__ double pinv[kBuildGroups];
  const int N = b.N, ns = b.ns, m = 2 * (ns - 1), s = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
  const int gr = tid >> 6, gt = tid & 63;  // group of two warps and the thread in it
  double* M = smb + gr * N * 2 * N;        // N x 2 N
  double* cv = smb + kBuildGroups * N * 2 * N;  // c_ks (row 0 of block ks against block ks - 1)
  double* dv = cv + ns * N;       // d_ks (row N - 1 of block ks against block ks + 1)
  double* ends = dv + ns * N;     // first and last entry of every left vector
  double* A = ends + 2 * m;       // interface matrix, m x 2 m
  double* pen = A + m * 2 * m;
  double *pa = pen, *pb = pen + ns, *pg = pen + 2 * ns, *pd = pen + 3 * ns, *pt1 = pen + 4 * ns, *pt2 = pen + 5 * ns;
  const double eps = __ddiv_rn(1., radd(b.ak[s], b.c0));
  for (int ks = tid; ks < ns; ks += nthr) {
    d_param_set(b, ks == 0 ? b.bot : 2, eps, b.zh[ks], pa[ks], pb[ks], pt1[ks]);
    d_param_set(b, ks == ns - 1 ? b.top : 2, eps, b.zh[ks], pg[ks], pd[ks], pt2[ks]);
  }
  __syncthreads();
  for (int q = tid; q < 6 * ns; q += nthr) b.pen[(size_t)s * 6 * ns + q] = pen[q];
  if (tid == 0) {
    SysDesc sd;
    sd.eps = eps;
    sd.tau1_bot = pt1[0];
    sd.tau2_top = pt2[ns - 1];
    sd.ifbcbot = b.bot;
    sd.ifbctop = b.top;
    sd.pad[0] = sd.pad[1] = 0;
    b.sys[s] = sd;
  }
  for (int q = tid; q < ns * N; q += nthr) {
    const int ks = q / N, k = q - ks * N;
    double c = 0.0, d = 0.0;
    if (ks > 0) {
      if (k == N - 1) c = -rmul(rmul(0.5, pt1[ks]), pa[ks]);
      c = radd(c, rmul(__ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt1[ks]), pb[ks]), eps), 2.0), b.zh[ks - 1]), b.D[(N - 1) * N + k]));
    }
    if (ks < ns - 1) {
      if (k == 0) d = rsub(0.0, rmul(rmul(0.5, pt2[ks]), pg[ks]));
      d = radd(d, rmul(-__ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt2[ks]), pd[ks]), eps), 2.0), b.zh[ks + 1]), b.D[k]));
    }
    cv[q] = c;
    dv[q] = d;
  }
  __syncthreads();
  for (int blk = gr; blk < b.nb; blk += kBuildGroups) {
    const int ks = b.brep[blk];
    const double ybar = b.zh[ks], h = __ddiv_rn(2.0, ybar), eh = rmul(eps, rmul(h, h));
    const bool lo = ns > 1 && ks != 0, hi = ns > 1 && ks != ns - 1;
    const double t1b = rmul(rmul(rmul(pt1[ks], pb[ks]), eps), 2.0), t2d = rmul(rmul(rmul(pt2[ks], pd[ks]), eps), 2.0);
    const double cf1 = -__ddiv_rn(t1b, ybar), cf2 = __ddiv_rn(t2d, ybar);
    const double cl = __ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt1[ks]), pb[ks]), eps), 2.0), ybar);
    const double ch = -__ddiv_rn(rmul(rmul(rmul(rmul(0.5, pt2[ks]), pd[ks]), eps), 2.0), ybar);
    for (int q = gt; q < N * 2 * N; q += 64) {
      const int r = q / (2 * N), c = q - r * 2 * N;
      double v = 0.0;
      if (c >= N) {
        v = c - N == r ? 1.0 : 0.0;
      } else {
        v = -rmul(eh, b.D2[r * N + c]);
        if (r == c) v = radd(v, 1.0);
        if (r == 0) {
          if (c == 0) v = radd(v, rmul(pt1[ks], pa[ks]));
          v = radd(v, rmul(cf1, b.D[c]));
          if (lo) {
            if (c == 0) v = rsub(v, rmul(rmul(0.5, pt1[ks]), pa[ks]));
            v = radd(v, rmul(cl, b.D[c]));
          }
        }
        if (r == N - 1) {
          if (c == N - 1) v = radd(v, rmul(pt2[ks], pg[ks]));
          v = radd(v, rmul(cf2, b.D[(N - 1) * N + c]));
          if (hi) {
            if (c == N - 1) v = rsub(v, rmul(rmul(0.5, pt2[ks]), pg[ks]));
            v = radd(v, rmul(ch, b.D[(N - 1) * N + c]));
          }
        }
      }
      M[q] = v;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + gr) : "memory");
    gauss_jordan(M, N, piv + gr, pinv + gr, gt, 64, 1 + gr);
    // the inverse is M(r, N + c): tables column major
    double* out = b.ainv + ((size_t)s * b.nb + blk) * N * N;
    double* raw = s < b.nraw ? b.ainv_raw + ((size_t)s * b.nb + blk) * N * N : nullptr;
    for (int q = gt; q < N * N; q += 64) {
      const int c = q / N, r = q - c * N;
      const double v = M[r * 2 * N + N + c];
      if (raw) raw[q] = v;
      if (b.L) {
        const double* lr = b.L + (size_t)r * N;
        double a = 0.0;
        for (int j = 0; j < N; ++j) a = __fma_rn(lr[j], M[j * 2 * N + N + c], a);
        out[q] = a;
      } else {
        out[q] = v;
      }
    }
    // left vectors of the subdomains with this block: c_{ks+1} (e = ks) and d_{ks-1} (e = ns - 2 + ks)
    for (int q = gt; q < m * N; q += 64) {
      const int e = q / N, c = q - e * N;
      const int kb = e < ns - 1 ? e : e - (ns - 1) + 1;
      if (b.bmap[kb] != blk) continue;
      const double* v = e < ns - 1 ? cv + (e + 1) * N : dv + (kb - 1) * N;
      double a = 0.0;
      for (int k = 0; k < N; ++k) a = __fma_rn(M[k * 2 * N + N + c], v[k], a);
      b.lvec[((size_t)s * m + e) * N + c] = a;
      if (c == 0) ends[2 * e] = a;
      if (c == N - 1) ends[2 * e + 1] = a;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + gr) : "memory");
  }
  __syncthreads();
  if (m == 0) return;
  // unknowns: sigma_ks (ks = 1 .. ns-1) -> ks - 1, tau_ks (ks = 0 .. ns-2) -> ns - 1 + ks
  for (int q = tid; q < m * 2 * m; q += nthr) A[q] = (q % (2 * m)) - m == q / (2 * m) ? 1.0 : 0.0;
  __syncthreads();
  for (int row = tid; row < m; row += nthr) {
    const int ks = row < ns - 1 ? row : row - (ns - 1) + 1;  // the block the row's coupling vector acts on
    A[row * 2 * m + row] += 1.0;
    if (ks >= 1) A[row * 2 * m + (ks - 1)] += ends[2 * row];
    if (ks <= ns - 2) A[row * 2 * m + (ns - 1 + ks)] += ends[2 * row + 1];
  }
  __syncthreads();
  gauss_jordan(A, m, piv, pinv, tid, nthr, 0);
  for (int q = tid; q < m * m; q += nthr) b.minv[(size_t)s * m * m + q] = A[(q / m) * 2 * m + m + q % m];
}

// ===========================================================================
// Grouped solves: one warp per task = up to G columns that share one system
// (same kx^2+ky^2, adjacent in the sorted column order).  All right-hand
// sides of the task advance together through each elimination step, so the
// factor column is fetched once per step for all of them.
// ===========================================================================
struct Task {
  int sys;    // system index (-1: no system, e.g. pressure of the (0,0) mode)
  int first;  // index into the sorted column order
  int count;  // columns in the task (<= G)
};

// SGBTRS + STBSV arithmetic for R <= RM right-hand sides b[r*n + row]
template <int RM>
__device__ void band_solve_multi(const double* __restrict__ ab, const int* __restrict__ ipiv, double* b, int R, int n,
                                 int kl, int ku, int lane) {
  constexpr int PF = 4;
  const int ldab = 2 * kl + ku + 1, kd = ku + kl + 1;
  const int i0 = lane + 1, i1 = lane + 33;
  int rl[PF];
  double rm0[PF], rm1[PF];
#pragma unroll
  for (int d = 0; d < PF; ++d) {
    const int j = 1 + d;
    rl[d] = 0;
    rm0[d] = rm1[d] = 0.0;
    if (j <= n - 1) {
      const int lm = min(kl, n - j);
      const double* col = ab + (size_t)ldab * (j - 1);
      rl[d] = __ldg(ipiv + j - 1);
      if (i0 <= lm) rm0[d] = __ldg(col + kd + i0 - 1);
      if (i1 <= lm) rm1[d] = __ldg(col + kd + i1 - 1);
    }
  }
  for (int jb = 1; jb <= n - 1; jb += PF) {
#pragma unroll
    for (int d = 0; d < PF; ++d) {
      const int j = jb + d;
      if (j <= n - 1) {
        const int lm = min(kl, n - j);
        const int l = rl[d];
        const double m0 = rm0[d], m1 = rm1[d];
        const int jn = j + PF;
        if (jn <= n - 1) {
          const int lmn = min(kl, n - jn);
          const double* coln = ab + (size_t)ldab * (jn - 1);
          rl[d] = __ldg(ipiv + jn - 1);
          rm0[d] = (i0 <= lmn) ? __ldg(coln + kd + i0 - 1) : 0.0;
          rm1[d] = (i1 <= lmn) ? __ldg(coln + kd + i1 - 1) : 0.0;
        }
        double y[RM], nv0[RM], nv1[RM];
        const int row0 = j + i0, row1 = j + i1;
#pragma unroll
        for (int r = 0; r < RM; ++r)
          if (r < R) {
            const double* br = b + (size_t)r * n;
            const double bj = br[j - 1], bl = br[l - 1];
            y[r] = (l != j) ? bl : bj;
            if (i0 <= lm) {
              const double old = (row0 == l) ? bj : br[row0 - 1];
              nv0[r] = (y[r] != 0.0) ? radd(old, rmul(m0, -y[r])) : old;
            }
            if (i1 <= lm) {
              const double old = (row1 == l) ? bj : br[row1 - 1];
              nv1[r] = (y[r] != 0.0) ? radd(old, rmul(m1, -y[r])) : old;
            }
          }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RM; ++r)
          if (r < R) {
            double* br = b + (size_t)r * n;
            if (i0 <= lm) br[row0 - 1] = nv0[r];
            if (i1 <= lm) br[row1 - 1] = nv1[r];
            if (lane == 0) br[j - 1] = y[r];
          }
        __syncwarp();
      }
    }
  }
  const int k = kl + ku, kplus1 = k + 1;
  double rdg[PF], rv0[PF], rv1[PF], rv2[PF];
  const int o0 = k - 1 - lane, o1 = k - 1 - lane - 32, o2 = k - 1 - lane - 64;
#pragma unroll
  for (int d = 0; d < PF; ++d) {
    const int j = n - d;
    rdg[d] = rv0[d] = rv1[d] = rv2[d] = 0.0;
    if (j >= 1) {
      const double* col = ab + (size_t)ldab * (j - 1);
      rdg[d] = __ldg(col + kplus1 - 1);
      if (o0 >= 0) rv0[d] = __ldg(col + o0);
      if (o1 >= 0) rv1[d] = __ldg(col + o1);
      if (o2 >= 0) rv2[d] = __ldg(col + o2);
    }
  }
  for (int jb = n; jb >= 1; jb -= PF) {
#pragma unroll
    for (int d = 0; d < PF; ++d) {
      const int j = jb - d;
      if (j >= 1) {
        const double dg = rdg[d];
        const double v0 = rv0[d], v1 = rv1[d], v2 = rv2[d];
        const int jn = j - PF;
        if (jn >= 1) {
          const double* coln = ab + (size_t)ldab * (jn - 1);
          rdg[d] = __ldg(coln + kplus1 - 1);
          rv0[d] = (o0 >= 0) ? __ldg(coln + o0) : 0.0;
          rv1[d] = (o1 >= 0) ? __ldg(coln + o1) : 0.0;
          rv2[d] = (o2 >= 0) ? __ldg(coln + o2) : 0.0;
        }
        const int lo = max(1, j - k);
        const int ia = j - 1 - lane, ib = ia - 32, ic = ia - 64;
        double xj[RM], n0[RM], n1[RM], n2[RM];
#pragma unroll
        for (int r = 0; r < RM; ++r)
          if (r < R) {
            const double* br = b + (size_t)r * n;
            xj[r] = br[j - 1];
            if (xj[r] != 0.0) {
              xj[r] = __ddiv_rn(xj[r], dg);
              if (ia >= lo) n0[r] = rsub(br[ia - 1], rmul(xj[r], v0));
              if (ib >= lo) n1[r] = rsub(br[ib - 1], rmul(xj[r], v1));
              if (ic >= lo) n2[r] = rsub(br[ic - 1], rmul(xj[r], v2));
            }
          }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RM; ++r)
          if (r < R && xj[r] != 0.0) {
            double* br = b + (size_t)r * n;
            if (ia >= lo) br[ia - 1] = n0[r];
            if (ib >= lo) br[ib - 1] = n1[r];
            if (ic >= lo) br[ic - 1] = n2[r];
            if (lane == 0) br[j - 1] = xj[r];
          }
        __syncwarp();
      }
    }
  }
}

// K_F grouped: pressure for the columns of one task (calcuvwt.f:87-229)
template <typename T, int G>
__global__ void k_press_g(Geo g, SolveTabs tb, const Task* __restrict__ tasks, int ntask, T* __restrict__ U,
                          T* __restrict__ V, T* __restrict__ W, const double* __restrict__ wnl,
                          const double* __restrict__ wvr, int cpen, int kstart) {
  extern __shared__ __align__(16) double sm[];
  const int warps = blockDim.x / 32, wid = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int t = blockIdx.x * warps + wid;
  if (t >= ntask) return;
  const Task tk = tasks[t];
  const int n = g.nz, N = g.N;
  double* B = sm + (size_t)wid * 2 * G * n;
  const int R = 2 * tk.count;
  const double dt = g.dt;
  const int s = tk.sys;
  if (s >= 0) {
    const SysDesc sd = tb.sys[s];
    const double eps = sd.eps;
    for (int ci = 0; ci < tk.count; ++ci) {
      const int c = tb.col_order[tk.first + ci];
      const int j = c / g.nxhp, ii = c % g.nxhp;
      const double xw = g.xw[ii], yw = g.yw[j];
      double* rr = B + (size_t)(2 * ci) * n;
      double* ri = rr + n;
      for (int k = lane; k < n; k += 32) {
        const int ks = k / N, k1 = k % N;
        double sr = 0.0, si = 0.0;
        for (int k2 = 0; k2 < N; ++k2) {
          const double dd = g.D[k1 * N + k2];
          sr = radd(sr, rmul(dd, (double)W[fidx<T>(g, 2 * ii, j, ks * N + k2)]));
          si = radd(si, rmul(dd, (double)W[fidx<T>(g, 2 * ii + 1, j, ks * N + k2)]));
        }
        const double fac = g.hfac[ks];
        const double dwr = rmul(sr, fac), dwi = rmul(si, fac);
        const double ur = (double)U[fidx<T>(g, 2 * ii, j, k)], ui = (double)U[fidx<T>(g, 2 * ii + 1, j, k)];
        const double vr = (double)V[fidx<T>(g, 2 * ii, j, k)], vi = (double)V[fidx<T>(g, 2 * ii + 1, j, k)];
        double dr = radd(radd(0.0, -rmul(xw, ui)), -rmul(yw, vi));
        double di = radd(radd(0.0, rmul(xw, ur)), rmul(yw, vr));
        dr = radd(dr, dwr);
        di = radd(di, dwi);
        rr[k] = -rmul(__ddiv_rn(dr, dt), eps);
        ri[k] = -rmul(__ddiv_rn(di, dt), eps);
      }
      __syncwarp();
      if (lane == 0) {
        const size_t p1 = (size_t)g.nxpp * j + 2 * ii, p2 = (size_t)g.nxpp * (j + g.ny) + 2 * ii;
        const double bcrbot = radd(wnl[p1], wvr[p1]), bcibot = radd(wnl[p1 + 1], wvr[p1 + 1]);
        const double bcrtop = radd(wnl[p2], wvr[p2]), bcitop = radd(wnl[p2 + 1], wvr[p2 + 1]);
        rr[0] = rsub(rr[0], rmul(rmul(sd.tau1_bot, bcrbot), eps));
        ri[0] = rsub(ri[0], rmul(rmul(sd.tau1_bot, bcibot), eps));
        rr[n - 1] = radd(rr[n - 1], rmul(rmul(sd.tau2_top, bcrtop), eps));
        ri[n - 1] = radd(ri[n - 1], rmul(rmul(sd.tau2_top, bcitop), eps));
      }
      __syncwarp();
    }
    const int ldab = 3 * N + 1;
    band_solve_multi<2 * G>(tb.ab + (size_t)s * ldab * n, tb.ipiv + (size_t)s * n, B, R, n, N, N, lane);
    if (cpen) {
      legen_filter_cols(B, R, n, N, g.ns, tb.wg, tb.alpol, tb.sigma, lane);
      __syncwarp();
    }
  } else {
    for (int q = lane; q < R * n; q += 32) B[q] = 0.0;
    __syncwarp();
  }
  for (int ci = 0; ci < tk.count; ++ci) {
    const int c = tb.col_order[tk.first + ci];
    const int j = c / g.nxhp, ii = c % g.nxhp;
    const bool lzero = (ii == 0 && j == 0);
    const double dtx = rmul(dt, g.xw[ii]), dty = rmul(dt, g.yw[j]);
    const double* rr = B + (size_t)(2 * ci) * n;
    const double* ri = rr + n;
    for (int k = lane; k < n; k += 32) {
      const size_t pr = fidx<T>(g, 2 * ii, j, k), pi = pr + 1;
      if (k < kstart) {
        U[pr] = 0;
        U[pi] = 0;
        V[pr] = 0;
        V[pi] = 0;
        W[pr] = 0;
        W[pi] = 0;
        continue;
      }
      const double phr = rr[k], phi = ri[k];
      const double ur = (double)U[pr], ui = (double)U[pi], vr = (double)V[pr], vi = (double)V[pi];
      double wbr = 0, wbi = 0;
      if (!lzero) {
        const int ks = k / N, k1 = k % N;
        double sr = 0.0, si = 0.0;
        for (int k2 = 0; k2 < N; ++k2) {
          const double dd = g.D[k1 * N + k2];
          sr = radd(sr, rmul(dd, rr[ks * N + k2]));
          si = radd(si, rmul(dd, ri[ks * N + k2]));
        }
        const double fac = g.hfac[ks];
        wbr = rsub((double)W[pr], rmul(dt, rmul(sr, fac)));
        wbi = rsub((double)W[pi], rmul(dt, rmul(si, fac)));
      }
      U[pr] = (T)rsub(ur, rsub(rmul(0.0, phr), rmul(dtx, phi)));
      U[pi] = (T)rsub(ui, radd(rmul(0.0, phi), rmul(dtx, phr)));
      V[pr] = (T)rsub(vr, rsub(rmul(0.0, phr), rmul(dty, phi)));
      V[pi] = (T)rsub(vi, radd(rmul(0.0, phi), rmul(dty, phr)));
      W[pr] = (T)wbr;
      W[pi] = (T)wbi;
    }
  }
}

// ===========================================================================
// Block-inverse solve, one CTA per task (row parallel).
//
// A = blockdiag(A_0..A_{ns-1}) + interface couplings (first row of block ks
// couples to the last row of ks-1 through c_ks, last row of ks to the first
// row of ks+1 through d_ks).  With y = blockdiag^-1 b the interface unknowns
// solve M z = r, r_e = <c_{e+1}, y_e> (e < ns-1), <d_t, y_{t+1}> (e = ns-1+t),
// and x = y - A_ks^-1 e_0 z_{ks-1} - A_ks^-1 e_{N-1} z_{ns-1+ks}.
// Because <c, A^-1 b> = <A^-T c, b>, the left vectors lvec = A^-T c, A^-T d
// are precomputed per system, so r comes straight from b and x from one sweep
// in which every inverse entry is read once (coalesced) and used for all R
// right-hand sides.  Each thread owns whole rows.
// ===========================================================================
constexpr int kSolveThreads = 128;

// dst = (accum ? dst : 0) + A^-1 src for R right-hand sides of length n.
// rz, zz: R*m doubles of shared scratch.  Ends synchronised.
template <int R>
__device__ void bi_apply_cta(const Geo& g, const double* __restrict__ ainv, const int* bmap,
                             const double* __restrict__ lvec, const double* __restrict__ minv, const double* src,
                             double* dst, double* rz, double* zz, bool accum) {
  const int N = g.N, ns = g.ns, n = g.nz, m = 2 * (ns - 1);
  const int tid = threadIdx.x;
  if (m > 0) {
    for (int q = tid; q < m * R; q += kSolveThreads) {
      const int r = q / m, e = q - r * m;
      const int blk = e < ns - 1 ? e : e - (ns - 1) + 1;
      const double* lv = lvec + (size_t)e * N;
      const double* sv = src + (size_t)r * n + blk * N;
      double acc = 0.0;
#pragma unroll 4
      for (int k = 0; k < N; ++k) acc += lv[k] * sv[k];
      rz[q] = acc;
    }
    __syncthreads();
    for (int q = tid; q < m * R; q += kSolveThreads) {
      const int r = q / m, e = q - r * m;
      const double* mr = minv + (size_t)e * m;
      const double* rr = rz + r * m;
      double z = 0.0;
#pragma unroll 4
      for (int c = 0; c < m; ++c) z += mr[c] * rr[c];
      zz[q] = z;
    }
    __syncthreads();
  }
  for (int row = tid; row < n; row += kSolveThreads) {
    const int ks = row / N, kk = row - ks * N;
    const double* ai = ainv + (size_t)bmap[ks] * N * N + kk;
    const double* sv = src + ks * N;
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0;
#pragma unroll 8
    for (int c = 0; c < N; ++c) {
      const double a = __ldg(ai + (size_t)c * N);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] += a * sv[(size_t)r * n + c];
    }
    const double p = ks >= 1 ? __ldg(ai) : 0.0;
    const double q = ks <= ns - 2 ? __ldg(ai + (size_t)(N - 1) * N) : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double x = acc[r];
      if (ks >= 1) x -= p * zz[r * m + ks - 1];
      if (ks <= ns - 2) x -= q * zz[r * m + ns - 1 + ks];
      double* d = dst + (size_t)r * n + row;
      *d = accum ? *d + x : x;
    }
  }
  __syncthreads();
}

// b -= A x for R right-hand sides (matrix free, FP64).  D2t/Dt: transposed
// differentiation matrices (Dt[k*N + k1] = D[k1][k]).
template <int R>
__device__ void sub_A_cta(const Geo& g, const double* __restrict__ D2t, const double* __restrict__ zh, double eps,
                          const double* __restrict__ pen, const double* x, double* b) {
  const int N = g.N, ns = g.ns, n = g.nz;
  for (int row = threadIdx.x; row < n; row += kSolveThreads) {
    const int ks = row / N, k1 = row - ks * N, km = ks * N;
    const double h2 = 2.0 / zh[ks];
    double s2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s2[r] = 0.0;
#pragma unroll 8
    for (int k = 0; k < N; ++k) {
      const double d = __ldg(D2t + k * N + k1);
#pragma unroll
      for (int r = 0; r < R; ++r) s2[r] += d * x[(size_t)r * n + km + k];
    }
    const double ee = eps * (h2 * h2);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double* xr = x + (size_t)r * n;
      double v = xr[row] - ee * s2[r];
      if (k1 == 0) {
        const double pa = pen[ks], pb = pen[ns + ks], t1 = pen[4 * ns + ks];
        double s0 = 0;
        for (int k = 0; k < N; ++k) s0 += g.D[k] * xr[km + k];
        v += t1 * pa * xr[km] - t1 * pb * eps * h2 * s0;
        if (ks > 0) {
          const double hl = 2.0 / zh[ks - 1];
          double sl = 0;
          for (int k = 0; k < N; ++k) sl += g.D[(N - 1) * N + k] * xr[km - N + k];
          v += -0.5 * t1 * pa * xr[km] + 0.5 * t1 * pb * eps * h2 * s0 - 0.5 * t1 * pa * xr[km - 1] +
               0.5 * t1 * pb * eps * hl * sl;
        }
      }
      if (k1 == N - 1) {
        const double pg = pen[2 * ns + ks], pd = pen[3 * ns + ks], t2 = pen[5 * ns + ks];
        double s1 = 0;
        for (int k = 0; k < N; ++k) s1 += g.D[(N - 1) * N + k] * xr[km + k];
        v += t2 * pg * xr[km + N - 1] + t2 * pd * eps * h2 * s1;
        if (ks < ns - 1) {
          const double hr = 2.0 / zh[ks + 1];
          double sr = 0;
          for (int k = 0; k < N; ++k) sr += g.D[k] * xr[km + N + k];
          v += -0.5 * t2 * pg * xr[km + N - 1] - 0.5 * t2 * pd * eps * h2 * s1 - 0.5 * t2 * pg * xr[km + N] -
               0.5 * t2 * pd * eps * hr * sr;
        }
      }
      b[(size_t)r * n + row] -= v;
    }
  }
  __syncthreads();
}

// dst[r][row] = sum_j L[kk][j] src[r][ks*N + j]: the Legendre filter of every
// subdomain (filtering.f:1225-1243 with the precombined matrix; Lt = L^T).
template <int R>
__device__ void legen_filter_cta(const Geo& g, const double* __restrict__ Lt, const double* src, double* dst) {
  const int N = g.N, n = g.nz;
  for (int row = threadIdx.x; row < n; row += kSolveThreads) {
    const int ks = row / N, kk = row - ks * N;
    const double* sv = src + ks * N;
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0;
#pragma unroll 8
    for (int j = 0; j < N; ++j) {
      const double l = __ldg(Lt + j * N + kk);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] += l * sv[(size_t)r * n + j];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) dst[(size_t)r * n + row] = acc[r];
  }
  __syncthreads();
}

// Solve of one task: <= R/per columns sharing system tk.sys, per = 4 right-hand
// sides per column for role 0 (u, v re/im), 2 otherwise; unused ones are zero.
// role 0: u/v (F0, F1), 1: w (F0), 2: rho (F0), 3: pressure from u*,v*,w*
// (F0, F1, F2) followed by the projection (calcuvwt.f:87-229, 826-901).
// refine: one FP64 residual sweep x += A^-1 (b - A x).
template <typename T, int R>
__global__ void __launch_bounds__(kSolveThreads) k_solve_cta(
    Geo g, BlockInv bi, SolveTabs tb, const Task* __restrict__ tasks, T* F0, T* F1, T* F2, const T* S0, const T* S1,
    int cols, double rdiv, int role, int cpen, int meanu, int refine, const double* __restrict__ Dt,
    const double* __restrict__ D2t, const double* __restrict__ Lt, const double* __restrict__ zh,
    const double* __restrict__ wnl, const double* __restrict__ wvr, int kstart) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int cj[R], cii[R];
  const Task tk = tasks[blockIdx.x];
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1);
  const int tid = threadIdx.x;
  double* b = sm;
  double* x = b + (size_t)R * n;
  double* rz = x + (size_t)R * n;
  double* zz = rz + (size_t)R * (m > 0 ? m : 1);
  // role 3: u*, v*, w* of the task's columns, [field][r][k], read from global
  // memory once for both the divergence and the projection
  T* fv = (T*)(zz + (size_t)R * (m > 0 ? m : 1));
  const int per = role == 0 ? 4 : 2;
  const int ncols = R / per;  // column slots per task
  const int s = tk.sys;
  const int ncolt = tk.count;
  const double dt = g.dt;
  if (tid < ncols) {
    const int c = tid < ncolt ? tb.col_order[tk.first + tid] : -1;
    cj[tid] = c < 0 ? -1 : c / g.nxhp;
    cii[tid] = c < 0 ? -1 : c % g.nxhp;
  }
  __syncthreads();
  // offset of row k of column slot ci in the sources (cols: scratch fields of
  // whole columns, [column][k] complex; the pressure also writes there)
  auto at = [&](int ci, int k) -> size_t {
    return cols ? ((size_t)(cj[ci] * g.nxhp + cii[ci]) * n + k) * 2 : fidx<T>(g, 2 * cii[ci], cj[ci], k);
  };
  if (role == 3) {
    // one 8-byte (re, im) load per field and column, all in flight at once
    typedef typename Pair<T>::t P2;
    for (int k = tid; k < n; k += kSolveThreads) {
#pragma unroll
      for (int ci = 0; ci < R / 2; ++ci) {
        P2 u2 = {0, 0}, v2 = {0, 0}, w2 = {0, 0};
        if (cj[ci] >= 0) {
          const size_t p = at(ci, k);
          u2 = *(const P2*)(F0 + p);
          v2 = *(const P2*)(F1 + p);
          w2 = *(const P2*)(F2 + p);
        }
        fv[(size_t)(2 * ci) * n + k] = u2.x;
        fv[(size_t)(2 * ci + 1) * n + k] = u2.y;
        fv[(size_t)(R + 2 * ci) * n + k] = v2.x;
        fv[(size_t)(R + 2 * ci + 1) * n + k] = v2.y;
        fv[(size_t)(2 * R + 2 * ci) * n + k] = w2.x;
        fv[(size_t)(2 * R + 2 * ci + 1) * n + k] = w2.y;
      }
    }
    __syncthreads();
  }
  if (s < 0 && role != 3) {  // w of the (0,0) mode is zero
    for (int ci = 0; ci < ncolt; ++ci)
      for (int k = tid; k < n; k += kSolveThreads) {
        F0[fidx<T>(g, 2 * cii[ci], cj[ci], k)] = 0;
        F0[fidx<T>(g, 2 * cii[ci] + 1, cj[ci], k)] = 0;
      }
    return;
  }
  const double* res = x;
  if (s < 0) {  // pressure of the (0,0) mode: phi = 0
    for (int q = tid; q < R * n; q += kSolveThreads) x[q] = 0.0;
    __syncthreads();
  } else {
    const SysDesc sd = bi.sys[s];
    const double eps = sd.eps;
    if (role == 3) {
      for (int k = tid; k < n; k += kSolveThreads) {  // w* columns into x (scratch)
#pragma unroll
        for (int r = 0; r < R; ++r) x[(size_t)r * n + k] = (double)fv[(size_t)(2 * R + r) * n + k];
      }
      __syncthreads();
      for (int k = tid; k < n; k += kSolveThreads) {
        const int ks = k / N, k1 = k - ks * N;
        double dw[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dw[r] = 0.0;
        for (int k2 = 0; k2 < N; ++k2) {
          const double dd = __ldg(Dt + k2 * N + k1);
#pragma unroll
          for (int r = 0; r < R; ++r) dw[r] += dd * x[(size_t)r * n + ks * N + k2];
        }
        const double fac = g.hfac[ks];
#pragma unroll
        for (int ci = 0; ci < R / 2; ++ci) {
          double vr = 0.0, vi = 0.0;
          if (cj[ci] >= 0) {
            const int j = cj[ci], ii = cii[ci];
            const double ur = (double)fv[(size_t)(2 * ci) * n + k], ui = (double)fv[(size_t)(2 * ci + 1) * n + k];
            const double wr = (double)fv[(size_t)(R + 2 * ci) * n + k];
            const double wi = (double)fv[(size_t)(R + 2 * ci + 1) * n + k];
            const double xw = g.xw[ii], yw = g.yw[j];
            const double dr = -(xw * ui) - (yw * wi) + dw[2 * ci] * fac;
            const double di = (xw * ur) + (yw * wr) + dw[2 * ci + 1] * fac;
            vr = -((dr / dt) * eps);
            vi = -((di / dt) * eps);
            if (k == 0) {
              const size_t p1 = (size_t)g.nxpp * j + 2 * ii;
              vr -= (sd.tau1_bot * (wnl[p1] + wvr[p1])) * eps;
              vi -= (sd.tau1_bot * (wnl[p1 + 1] + wvr[p1 + 1])) * eps;
            }
            if (k == n - 1) {
              const size_t p2 = (size_t)g.nxpp * (j + g.ny) + 2 * ii;
              vr += (sd.tau2_top * (wnl[p2] + wvr[p2])) * eps;
              vi += (sd.tau2_top * (wnl[p2 + 1] + wvr[p2 + 1])) * eps;
            }
          }
          b[(size_t)(2 * ci) * n + k] = vr;
          b[(size_t)(2 * ci + 1) * n + k] = vi;
        }
      }
    } else {
      for (int k = tid; k < n; k += kSolveThreads) {
        double v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int ci = r / per, rr = r - ci * per;
          const T* F = (role == 0 && rr >= 2) ? S1 : S0;
          v[r] = cj[ci] >= 0 ? (double)F[at(ci, k) + (rr & 1)] : 0.0;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) b[(size_t)r * n + k] = -(-(v[r] / rdiv) * eps);
      }
    }
    __syncthreads();
    const double* ainv = (const double*)bi.ainv + (size_t)s * bi.nb * N * N;
    const double* lv = bi.lvec + (size_t)s * (m > 0 ? m : 1) * N;
    const double* mi = bi.minv + (size_t)s * (m > 0 ? m * m : 1);
    bi_apply_cta<R>(g, ainv, bi.bmap, lv, mi, b, x, rz, zz, false);
    if (refine) {
      sub_A_cta<R>(g, D2t, zh, eps, bi.pen + (size_t)s * 6 * ns, x, b);
      bi_apply_cta<R>(g, ainv, bi.bmap, lv, mi, b, x, rz, zz, true);
    }
    if (cpen) {
      legen_filter_cta<R>(g, Lt, x, b);
      res = b;
    }
  }
  // write back
  if (role == 3) {
    for (int k = tid; k < n; k += kSolveThreads) {
      const int ks = k / N, k1 = k - ks * N;
      double dz[R];
#pragma unroll
      for (int r = 0; r < R; ++r) dz[r] = 0.0;
      for (int k2 = 0; k2 < N; ++k2) {
        const double dd = __ldg(Dt + k2 * N + k1);
#pragma unroll
        for (int r = 0; r < R; ++r) dz[r] += dd * res[(size_t)r * n + ks * N + k2];
      }
      const double fac = g.hfac[ks];
#pragma unroll
      for (int ci = 0; ci < R / 2; ++ci) {
        if (cj[ci] < 0) continue;
        const int j = cj[ci], ii = cii[ci];
        const size_t pr = at(ci, k), pi = pr + 1;
        if (k < kstart) {
          F0[pr] = 0;
          F0[pi] = 0;
          F1[pr] = 0;
          F1[pi] = 0;
          F2[pr] = 0;
          F2[pi] = 0;
          continue;
        }
        const double phr = res[(size_t)(2 * ci) * n + k], phi = res[(size_t)(2 * ci + 1) * n + k];
        double wbr = 0, wbi = 0;
        if (!(ii == 0 && j == 0)) {
          wbr = (double)fv[(size_t)(2 * R + 2 * ci) * n + k] - dt * (dz[2 * ci] * fac);
          wbi = (double)fv[(size_t)(2 * R + 2 * ci + 1) * n + k] - dt * (dz[2 * ci + 1] * fac);
        }
        const double dtx = dt * g.xw[ii], dty = dt * g.yw[j];
        const double ur = (double)fv[(size_t)(2 * ci) * n + k], ui = (double)fv[(size_t)(2 * ci + 1) * n + k];
        const double vr = (double)fv[(size_t)(R + 2 * ci) * n + k], vi = (double)fv[(size_t)(R + 2 * ci + 1) * n + k];
        F0[pr] = (T)(ur + dtx * phi);
        F0[pi] = (T)(ui - dtx * phr);
        F1[pr] = (T)(vr + dty * phi);
        F1[pi] = (T)(vi - dty * phr);
        F2[pr] = (T)wbr;
        F2[pi] = (T)wbi;
      }
    }
  } else {
    for (int k = tid; k < n; k += kSolveThreads) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int ci = r / per, rr = r - ci * per;
        if (cj[ci] < 0) continue;
        T* F = (role == 0 && rr >= 2) ? F1 : F0;
        double v = res[(size_t)r * n + k];
        if (role == 0 && rr < 2 && meanu && cii[ci] == 0 && cj[ci] == 0) v = tb.meang[k] * v;
        F[fidx<T>(g, 2 * cii[ci] + (rr & 1), cj[ci], k)] = (T)v;
      }
    }
  }
}

// ===========================================================================
// System-grouped solve.  One CTA per group of columns that share one system:
// up to 4 u/v columns (16 right-hand sides) or 8 columns of w, rho or the
// pressure (16 right-hand sides).  The system's distinct inverse blocks, its
// left vectors and its interface matrix come into shared memory once per CTA
// by bulk asynchronous copies (cp.async.bulk, completion counted on an
// mbarrier) while the CTA gathers its columns, so every product reads both
// operands from shared memory.  Thread t owns row t for all 16 right-hand
// sides: one shared load of an inverse entry serves 16 multiply-adds, and the
// right-hand sides are stored [row][16], so the 16 values of one row come as
// eight 16-byte broadcasts.  The arithmetic (order of every sum, the RHS and
// projection formulas) is the one of k_solve_cta, so both give the same bits.
// Used for n <= 512 rows, filter folded into the inverses (or no filter),
// no residual sweep and a system present; k_solve_cta takes the rest.
// ===========================================================================
constexpr int kSysR = 16;
// row stride of the right-hand sides in shared memory: 16 values + 2 of padding,
// so that the 16-byte stores of consecutive rows fall on different banks
constexpr int kSysRS = kSysR + 2;
constexpr int kSysMaxRows = 512;

struct SysSmem {  // offsets (doubles) of the shared-memory regions of k_solve_sys
  size_t a, l, m, b, rz, zz, d, total;
};
__host__ __device__ inline SysSmem sys_smem(int n, int N, int ns, int nb, bool dmat) {
  SysSmem o;
  const size_t m = 2 * (size_t)(ns - 1), m1 = m > 0 ? m : 1;
  o.a = 0;
  o.l = ((size_t)nb * N * N + 3) & ~(size_t)1;  // room for a copy that starts one double early
  o.m = o.l + m * N;
  o.b = o.m + m * m;
  o.rz = o.b + (size_t)n * kSysRS;
  o.zz = o.rz + kSysR * m1;
  o.d = o.zz + kSysR * m1;
  o.total = o.d + (dmat ? (((size_t)N * N + 1) & ~(size_t)1) : 0);
  return o;
}

// 8-byte shared load.  The 16 right-hand-side values of a row are the same
// for every lane of a warp that works in one block (a broadcast): as 8-byte
// loads each costs one shared-memory wavefront, as 16-byte loads four.
__device__ __forceinline__ double lds64(const double* p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(smem_u32(p)));
  return v;
}

// acc[r] = sum_c col[c*N] * b[(base + c)*RS + r]: one row of a block product;
// the loads go out in groups of BL
template <int BL = 8>
__device__ __forceinline__ void row_product16(const double* col, const double* bb, int N, double* acc) {
#pragma unroll
  for (int r = 0; r < kSysR; ++r) acc[r] = 0.0;
#pragma unroll 2
  for (int c = 0; c < N; ++c) {
    const double a = col[(size_t)c * N];
    const double* br = bb + (size_t)c * kSysRS;
#pragma unroll
    for (int h = 0; h < kSysR; h += BL) {
      double v[BL];
#pragma unroll
      for (int r = 0; r < BL; ++r) v[r] = lds64(br + h + r);
#pragma unroll
      for (int r = 0; r < BL; ++r) acc[h + r] += a * v[r];
    }
  }
}

// role 0: u/v (4 RHS per column), 1: w, 2: rho, 3: pressure + projection.
template <typename T, int ROLE>
__global__ void __maxnreg__(72) k_solve_sys(
    Geo g, BlockInv bi, const Task* __restrict__ tasks, const int* __restrict__ col_order, T* __restrict__ F0,
    T* __restrict__ F1, T* __restrict__ F2, double rdiv, int meanu, const double* __restrict__ meang,
    const double* __restrict__ Dt, const double* __restrict__ wnl, const double* __restrict__ wvr, int kstart,
    int* __restrict__ err) {
  typedef typename Pair<T>::t P2;
  constexpr int R = kSysR;
  constexpr int PER = ROLE == 0 ? 4 : 2;  // right-hand sides per column
  constexpr int NC = R / PER;             // column slots
  constexpr int RS = kSysRS;  // right-hand-side row stride
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int cj[NC], cii[NC];
  const Task tk = tasks[blockIdx.x];
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1), nb = bi.nb;
  const int tid = threadIdx.x;
  const int s = tk.sys;
  const SysSmem L = sys_smem(n, N, ns, nb, ROLE == 3);
  double* sA = sm + L.a;
  double* sL = sm + L.l;
  double* sM = sm + L.m;
  double* sb = sm + L.b;
  double* srz = sm + L.rz;
  double* szz = sm + L.zz;
  double* sD = sm + L.d;
  // the system's tables: one bulk copy each, all counted on one mbarrier
  const uintptr_t ga = (uintptr_t)((const double*)bi.ainv + (size_t)s * nb * N * N);
  const int offA = (int)((ga & 15u) >> 3);  // the copy starts one double early when ga is not 16-byte aligned
  const uint32_t bytesA = (uint32_t)((((size_t)nb * N * N + offA) * 8 + 15) & ~(size_t)15);
  const uint32_t bytesL = (uint32_t)((size_t)m * N * 8), bytesM = (uint32_t)((size_t)m * m * 8);
  if (tid == 0) mbar_init(&bar, 1);
  if (tid < NC) {
    const int c = tid < tk.count ? col_order[tk.first + tid] : -1;
    cj[tid] = c < 0 ? -1 : c / g.nxhp;
    cii[tid] = c < 0 ? -1 : c % g.nxhp;
  }
  __syncthreads();
  if (tid == 0) {
    mbar_expect_tx(&bar, bytesA + bytesL + bytesM);
    bulk_g2s(sA, (const void*)(ga - (uintptr_t)offA * 8), bytesA, &bar);
    if (m > 0) {
      bulk_g2s(sL, bi.lvec + (size_t)s * m * N, bytesL, &bar);
      bulk_g2s(sM, bi.minv + (size_t)s * m * m, bytesM, &bar);
    }
  }
  if (ROLE == 3)
    for (int q = tid; q < N * N; q += blockDim.x) sD[q] = Dt[q];
  const double eps = bi.sys[s].eps;
  const double dt = g.dt;
  const int k = tid;
  const bool live = k < n;
  const int ks = live ? k / N : 0, kk = k - ks * N;
  // gather this row of every column: [row][16]
  if (live) {
    double v[R];
#pragma unroll
    for (int ci = 0; ci < NC; ++ci) {
      P2 a = {0, 0}, b = {0, 0};
      if (cj[ci] >= 0) {
        const size_t p = fidx<T>(g, 2 * cii[ci], cj[ci], k);
        if (ROLE == 3) {
          a = *(const P2*)(F2 + p);
        } else {
          a = *(const P2*)(F0 + p);
          if (ROLE == 0) b = *(const P2*)(F1 + p);
        }
      }
      v[PER * ci] = (double)a.x;
      v[PER * ci + 1] = (double)a.y;
      if (ROLE == 0) {
        v[PER * ci + 2] = (double)b.x;
        v[PER * ci + 3] = (double)b.y;
      }
    }
    if (ROLE != 3) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = -(-(v[r] / rdiv) * eps);
    }
    double2* d2 = (double2*)(sb + (size_t)k * RS);
#pragma unroll
    for (int q = 0; q < R / 2; ++q) d2[q] = make_double2(v[2 * q], v[2 * q + 1]);
  }
  const bool ok = mbar_wait(&bar, 0, 2000000000ull);
  if (__syncthreads_or(!ok)) {  // the tables never arrived: report, let the copies finish, leave
    if (tid == 0) err[1] = 1;
    mbar_wait(&bar, 0, 2000000000ull);
    return;
  }
  double acc[R];
  if (ROLE == 3) {
    // divergence of u*: i kx u* + i ky v* + (2/h) D w*; RHS = -(div/dt) eps
    // plus the Neumann data at the walls (calcuvwt.f:87-229)
    if (live) {
      row_product16<ROLE == 3 ? 4 : 8>(sD + kk, sb + (size_t)ks * N * RS, N, acc);
      const double fac = g.hfac[ks];
      const SysDesc sd = bi.sys[s];
#pragma unroll
      for (int ci = 0; ci < NC; ++ci) {
        double vr = 0.0, vi = 0.0;
        if (cj[ci] >= 0) {
          const int j = cj[ci], ii = cii[ci];
          const size_t pr = fidx<T>(g, 2 * ii, j, k);
          const P2 u2 = *(const P2*)(F0 + pr), w2 = *(const P2*)(F1 + pr);
          const double ur = (double)u2.x, ui = (double)u2.y;
          const double wr = (double)w2.x, wi = (double)w2.y;
          const double xw = g.xw[ii], yw = g.yw[j];
          const double dr = -(xw * ui) - (yw * wi) + acc[2 * ci] * fac;
          const double di = (xw * ur) + (yw * wr) + acc[2 * ci + 1] * fac;
          vr = -((dr / dt) * eps);
          vi = -((di / dt) * eps);
          if (k == 0) {
            const size_t p1 = (size_t)g.nxpp * j + 2 * ii;
            vr -= (sd.tau1_bot * (wnl[p1] + wvr[p1])) * eps;
            vi -= (sd.tau1_bot * (wnl[p1 + 1] + wvr[p1 + 1])) * eps;
          }
          if (k == n - 1) {
            const size_t p2 = (size_t)g.nxpp * (j + g.ny) + 2 * ii;
            vr += (sd.tau2_top * (wnl[p2] + wvr[p2])) * eps;
            vi += (sd.tau2_top * (wnl[p2 + 1] + wvr[p2 + 1])) * eps;
          }
        }
        acc[2 * ci] = vr;  // column ci's divergence is no longer needed: the RHS takes its place
        acc[2 * ci + 1] = vi;
      }
    }
    __syncthreads();  // every row of w* has been read
    if (live) {
      double2* d2 = (double2*)(sb + (size_t)k * RS);
#pragma unroll
      for (int q = 0; q < R / 2; ++q) d2[q] = make_double2(acc[2 * q], acc[2 * q + 1]);
    }
    __syncthreads();
  }
  // interface system: r_e = <lvec_e, b_blk(e)>, z = M^-1 r; stored [e][r] and
  // computed with the right-hand side index fastest across lanes
  if (m > 0) {
    for (int q = tid; q < m * R; q += blockDim.x) {
      const int e = q / R, r = q - e * R;
      const int blk = e < ns - 1 ? e : e - (ns - 1) + 1;
      const double* lv = sL + (size_t)e * N;
      const double* sv = sb + (size_t)blk * N * RS + r;
      double a = 0.0;
      for (int c = 0; c < N; ++c) a += lv[c] * sv[(size_t)c * RS];
      srz[q] = a;
    }
    __syncthreads();
    for (int q = tid; q < m * R; q += blockDim.x) {
      const int e = q / R, r = q - e * R;
      const double* mr = sM + (size_t)e * m;
      double z = 0.0;
      for (int c = 0; c < m; ++c) z += mr[c] * srz[(size_t)c * R + r];
      szz[q] = z;
    }
    __syncthreads();
  }
  // x = A_ks^-1 b_ks - A_ks^-1 e_0 z_{ks-1} - A_ks^-1 e_{N-1} z_{ns-1+ks}
  double* x = acc;  // the solution replaces the product in place
  if (live) {
    const double* col = sA + offA + (size_t)bi.bmap[ks] * N * N + kk;
    row_product16<ROLE == 3 ? 4 : 8>(col, sb + (size_t)ks * N * RS, N, acc);
    const double p = ks >= 1 ? col[0] : 0.0;
    const double q = ks <= ns - 2 ? col[(size_t)(N - 1) * N] : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double xv = acc[r];
      if (ks >= 1) xv -= p * szz[(size_t)(ks - 1) * R + r];
      if (ks <= ns - 2) xv -= q * szz[(size_t)(ns - 1 + ks) * R + r];
      x[r] = xv;
    }
  }
  if (ROLE != 3) {
    if (ROLE == 0 && meanu && live) {
#pragma unroll
      for (int ci = 0; ci < NC; ++ci)
        if (cii[ci] == 0 && cj[ci] == 0) {
          x[PER * ci] = meang[k] * x[PER * ci];
          x[PER * ci + 1] = meang[k] * x[PER * ci + 1];
        }
    }
    if (!live) return;
#pragma unroll
    for (int ci = 0; ci < NC; ++ci) {
      if (cj[ci] < 0) continue;
      const size_t p = fidx<T>(g, 2 * cii[ci], cj[ci], k);
      const double a0 = x[PER * ci], a1 = x[PER * ci + 1];
      P2 o;
      o.x = (T)a0;
      o.y = (T)a1;
      *(P2*)(F0 + p) = o;
      if (ROLE == 0) {
        P2 o2;
        o2.x = (T)x[PER * ci + 2];
        o2.y = (T)x[PER * ci + 3];
        *(P2*)(F1 + p) = o2;
      }
    }
    return;
  }
  // pressure: phi into shared memory, (2/h) D phi, projection (calcuvwt.f:826-901)
  __syncthreads();  // every row of the RHS has been read
  if (live) {
    double2* d2 = (double2*)(sb + (size_t)k * RS);
#pragma unroll
    for (int q = 0; q < R / 2; ++q) d2[q] = make_double2(x[2 * q], x[2 * q + 1]);
  }
  __syncthreads();
  if (!live) return;
  row_product16<ROLE == 3 ? 4 : 8>(sD + kk, sb + (size_t)ks * N * RS, N, acc);
  const double fac = g.hfac[ks];
#pragma unroll
  for (int ci = 0; ci < NC; ++ci) {
    if (cj[ci] < 0) continue;
    const int j = cj[ci], ii = cii[ci];
    const size_t pr = fidx<T>(g, 2 * ii, j, k);
    P2 zu, zv, zw;
    if (k < kstart) {
      zu.x = zu.y = (T)0;
      *(P2*)(F0 + pr) = zu;
      *(P2*)(F1 + pr) = zu;
      *(P2*)(F2 + pr) = zu;
      continue;
    }
    const double phr = sb[(size_t)k * RS + 2 * ci], phi = sb[(size_t)k * RS + 2 * ci + 1];
    const P2 w2 = *(const P2*)(F2 + pr);
    double wbr = 0, wbi = 0;
    if (!(ii == 0 && j == 0)) {
      wbr = (double)w2.x - dt * (acc[2 * ci] * fac);
      wbi = (double)w2.y - dt * (acc[2 * ci + 1] * fac);
    }
    const double dtx = dt * g.xw[ii], dty = dt * g.yw[j];
    const P2 u2 = *(const P2*)(F0 + pr), v2 = *(const P2*)(F1 + pr);
    const double ur = (double)u2.x, ui = (double)u2.y, vr = (double)v2.x, vi = (double)v2.y;
    zu.x = (T)(ur + dtx * phi);
    zu.y = (T)(ui - dtx * phr);
    zv.x = (T)(vr + dty * phi);
    zv.y = (T)(vi - dty * phr);
    zw.x = (T)wbr;
    zw.y = (T)wbi;
    *(P2*)(F0 + pr) = zu;
    *(P2*)(F1 + pr) = zv;
    *(P2*)(F2 + pr) = zw;
  }
}

// ===========================================================================
// System-grouped solve with two rows per thread (u/v, w and rho).  The
// grouped solve above spends most of its time in the shared-memory pipe: each
// multiply-add of its block product takes one broadcast load of a
// right-hand-side value.  Here thread (ks, q) owns rows q and q + H of
// subdomain ks (H = ceil(N/2)), both of one inverse block, so every broadcast
// feeds two multiply-adds and the loads per multiply-add fall from 18/16 to
// 20/32.  The tables, the gather, the interface system and the order of every
// sum are those of k_solve_sys, so both give the same bits.
// ===========================================================================
constexpr int kSys2MaxThreads = 256;

// acc0/acc1[r] = sum_c col[c N (+ H)] * b[c RS + r] for two rows of one block
__device__ __forceinline__ void row_product16x2(const double* col, int H, bool has1, const double* bb, int N,
                                                double* acc0, double* acc1) {
#pragma unroll
  for (int r = 0; r < kSysR; ++r) acc0[r] = acc1[r] = 0.0;
#pragma unroll 1
  for (int c = 0; c < N; ++c) {
    const double a0 = col[(size_t)c * N];
    const double a1 = has1 ? col[(size_t)c * N + H] : 0.0;
    const double* br = bb + (size_t)c * kSysRS;
#pragma unroll
    for (int h = 0; h < kSysR; h += 8) {
      double v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = lds64(br + h + r);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        acc0[h + r] += a0 * v[r];
        acc1[h + r] += a1 * v[r];
      }
    }
  }
}

template <typename T, int ROLE>
__global__ void __launch_bounds__(kSys2MaxThreads, 2) k_solve_sys2(
    Geo g, BlockInv bi, const Task* __restrict__ tasks, const int* __restrict__ col_order, T* __restrict__ F0,
    T* __restrict__ F1, double rdiv, int meanu, const double* __restrict__ meang, int* __restrict__ err) {
  static_assert(ROLE >= 0 && ROLE <= 2, "u/v, w and rho only");
  typedef typename Pair<T>::t P2;
  constexpr int R = kSysR;
  constexpr int PER = ROLE == 0 ? 4 : 2;  // right-hand sides per column
  constexpr int NC = R / PER;             // column slots
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int cj[NC], cii[NC];
  const Task tk = tasks[blockIdx.x];
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1), nb = bi.nb;
  const int H = (N + 1) >> 1;
  const int tid = threadIdx.x;
  const int s = tk.sys;
  const SysSmem L = sys_smem(n, N, ns, nb, false);
  double* sA = sm + L.a;
  double* sL = sm + L.l;
  double* sM = sm + L.m;
  double* sb = sm + L.b;
  double* srz = sm + L.rz;
  double* szz = sm + L.zz;
  const uintptr_t ga = (uintptr_t)((const double*)bi.ainv + (size_t)s * nb * N * N);
  const int offA = (int)((ga & 15u) >> 3);
  const uint32_t bytesA = (uint32_t)((((size_t)nb * N * N + offA) * 8 + 15) & ~(size_t)15);
  const uint32_t bytesL = (uint32_t)((size_t)m * N * 8), bytesM = (uint32_t)((size_t)m * m * 8);
  if (tid == 0) mbar_init(&bar, 1);
  if (tid < NC) {
    const int c = tid < tk.count ? col_order[tk.first + tid] : -1;
    cj[tid] = c < 0 ? -1 : c / g.nxhp;
    cii[tid] = c < 0 ? -1 : c % g.nxhp;
  }
  __syncthreads();
  if (tid == 0) {
    mbar_expect_tx(&bar, bytesA + bytesL + bytesM);
    bulk_g2s(sA, (const void*)(ga - (uintptr_t)offA * 8), bytesA, &bar);
    if (m > 0) {
      bulk_g2s(sL, bi.lvec + (size_t)s * m * N, bytesL, &bar);
      bulk_g2s(sM, bi.minv + (size_t)s * m * m, bytesM, &bar);
    }
  }
  const double eps = bi.sys[s].eps;
  const int ks = tid / H, q0 = tid - ks * H;
  const bool live = ks < ns;
  const bool has1 = live && q0 + H < N;
  const int k0 = ks * N + q0, k1 = k0 + H;
  // gather rows k0 and k1 of every column: [row][16]
#pragma unroll 1
  for (int hr = 0; hr < 2; ++hr) {
    if (!(hr == 0 ? live : has1)) continue;
    const int k = hr == 0 ? k0 : k1;
    double v[R];
#pragma unroll
    for (int ci = 0; ci < NC; ++ci) {
      P2 a = {0, 0}, b = {0, 0};
      if (cj[ci] >= 0) {
        const size_t p = fidx<T>(g, 2 * cii[ci], cj[ci], k);
        a = *(const P2*)(F0 + p);
        if (ROLE == 0) b = *(const P2*)(F1 + p);
      }
      v[PER * ci] = (double)a.x;
      v[PER * ci + 1] = (double)a.y;
      if (ROLE == 0) {
        v[PER * ci + 2] = (double)b.x;
        v[PER * ci + 3] = (double)b.y;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = -(-(v[r] / rdiv) * eps);
    double2* d2 = (double2*)(sb + (size_t)k * kSysRS);
#pragma unroll
    for (int q = 0; q < R / 2; ++q) d2[q] = make_double2(v[2 * q], v[2 * q + 1]);
  }
  const bool ok = mbar_wait(&bar, 0, 2000000000ull);
  if (__syncthreads_or(!ok)) {  // the tables never arrived: report, let the copies finish, leave
    if (tid == 0) err[1] = 1;
    mbar_wait(&bar, 0, 2000000000ull);
    return;
  }
  // interface system (the loops and sums of k_solve_sys)
  if (m > 0) {
    for (int q = tid; q < m * R; q += blockDim.x) {
      const int e = q / R, r = q - e * R;
      const int blk = e < ns - 1 ? e : e - (ns - 1) + 1;
      const double* lv = sL + (size_t)e * N;
      const double* sv = sb + (size_t)blk * N * kSysRS + r;
      double a = 0.0;
      for (int c = 0; c < N; ++c) a += lv[c] * sv[(size_t)c * kSysRS];
      srz[q] = a;
    }
    __syncthreads();
    for (int q = tid; q < m * R; q += blockDim.x) {
      const int e = q / R, r = q - e * R;
      const double* mr = sM + (size_t)e * m;
      double z = 0.0;
      for (int c = 0; c < m; ++c) z += mr[c] * srz[(size_t)c * R + r];
      szz[q] = z;
    }
    __syncthreads();
  }
  if (!live) return;
  // x = A_ks^-1 b_ks - A_ks^-1 e_0 z_{ks-1} - A_ks^-1 e_{N-1} z_{ns-1+ks}, two rows
  const double* col = sA + offA + (size_t)bi.bmap[ks] * N * N + q0;
  double acc0[R], acc1[R];
  row_product16x2(col, H, has1, sb + (size_t)ks * N * kSysRS, N, acc0, acc1);
#pragma unroll 1
  for (int hr = 0; hr < 2; ++hr) {
    if (hr == 1 && !has1) break;
    const int k = hr == 0 ? k0 : k1;
    const double* cr = col + (hr == 0 ? 0 : H);
    const double p = ks >= 1 ? cr[0] : 0.0;
    const double qv = ks <= ns - 2 ? cr[(size_t)(N - 1) * N] : 0.0;
    double x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double xv = hr == 0 ? acc0[r] : acc1[r];
      if (ks >= 1) xv -= p * szz[(size_t)(ks - 1) * R + r];
      if (ks <= ns - 2) xv -= qv * szz[(size_t)(ns - 1 + ks) * R + r];
      x[r] = xv;
    }
    if (ROLE == 0 && meanu) {
#pragma unroll
      for (int ci = 0; ci < NC; ++ci)
        if (cii[ci] == 0 && cj[ci] == 0) {
          x[PER * ci] = meang[k] * x[PER * ci];
          x[PER * ci + 1] = meang[k] * x[PER * ci + 1];
        }
    }
#pragma unroll
    for (int ci = 0; ci < NC; ++ci) {
      if (cj[ci] < 0) continue;
      const size_t p2 = fidx<T>(g, 2 * cii[ci], cj[ci], k);
      P2 o;
      o.x = (T)x[PER * ci];
      o.y = (T)x[PER * ci + 1];
      *(P2*)(F0 + p2) = o;
      if (ROLE == 0) {
        P2 o2;
        o2.x = (T)x[PER * ci + 2];
        o2.y = (T)x[PER * ci + 3];
        *(P2*)(F1 + p2) = o2;
      }
    }
  }
}

// ===========================================================================
// System-grouped solve on the FP64 tensor cores (mma.sync m8n8k4, the FP64
// matrix instruction of sm_100a; tcgen05 has no FP64 kind).  A task's columns
// as in k_solve_sys; one warp owns one subdomain.  The products are formed
// transposed, X^T = B^T Op^T: the right-hand sides are the 8 rows of the A
// operand, the operator rows the 8 columns of the B operand, 4 operator
// columns per instruction in ascending order.  The instruction adds its four
// products one after the other, each with one rounding, so every sum is the
// FMA chain of k_solve_cta and k_solve_sys and all variants give the same bits.
// Every warp gathers the columns of its own subdomain (cp.async, in storage
// precision), so the CTA only meets for the tables and around the interface
// system: r_e = <lvec_e, b> (a sixth tile next to the block product's, from the
// same operand loads), z = M^-1 r, x = A^-1 b - A^-1 e_0 z' - A^-1 e_{N-1} z''
// (one more k step on the accumulators).  The pressure keeps the right-hand
// side and phi in accumulator registers between its three products (D w*, A^-1,
// D phi); four shuffles per k step turn them into the next A operand.
// What bounds it: the shared-memory pipe (an operator fragment is two wavefronts
// per tile product) and the gather and scatter of single complex values, then the
// matrix pipe (36.9 TFLOP/s).  B200, 512^2 x (12 x 33) mixed, against the
// FP64-pipe kernels (a broadcast load per multiply-add): pressure 7.97 -> 4.17 ms,
// u/v 3.04 -> 2.49, w 2.01 -> 1.32; 256^2 x (8 x 25) FP64: pressure 1.04 -> 0.47 ms.
// ===========================================================================
// Staged right-hand sides: [tile][row][8] values of T; of FP64 rows the halves
// swap places on every other pair of rows, so that an A fragment (4 rows x 8)
// has no bank conflicts (FP32 fragments are 32 consecutive words as they are).
template <typename T>
__device__ __forceinline__ int tc_pos(int r, int g) {
  return r * 8 + (sizeof(T) == 8 ? g ^ (((r >> 1) & 1) << 2) : g);
}
struct TcSmem {  // byte offsets
  size_t a, l, m, rz, zz, d, raw, total;
};
// tiles: staged tiles of 8 right-hand sides (2; the pressure 3: u*, v*, w*)
template <typename T>
__host__ __device__ inline TcSmem tc_smem(int n, int N, int ns, int nb, bool press) {
  TcSmem o;
  const size_t m = 2 * (size_t)(ns - 1), ap = tc_ap(N), D = sizeof(double), R = press ? 8 : 16;
  o.a = 0;
  o.l = o.a + (size_t)nb * tc_nc(N) * ap * D;
  o.m = o.l + m * N * D;
  o.rz = o.m + m * m * D;
  o.zz = o.rz + m * R * D;
  o.d = o.zz + m * R * D;
  o.raw = o.d + (press ? (size_t)tc_nc(N) * ap * D : 0);
  o.total = o.raw + (press ? 3 : 2) * (size_t)n * 8 * sizeof(T) + 16 * D;  // (room for a fragment past the last column)
  return o;
}
__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}
__device__ __forceinline__ void cp_async_8(double* smem, const double* gmem) {
  cp_async_c<float2>((float2*)smem, (const float2*)gmem);
}
// Markstein's division by a constant: y = RN(1 / d).  q within 2 ulp, one
// correction makes it faithful, the next correctly rounded (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000", 1990).
__device__ __forceinline__ double div_by(double v, double d, double y) {
  double q = __dmul_rn(v, y);
  q = __fma_rn(__fma_rn(-q, d, v), y, q);
  return __fma_rn(__fma_rn(-q, d, v), y, q);
}
// acc[i][nt][h] = sum_c op[c AP + 8 nt + 2 t + h] b_i(c) for right-hand side g of NI
// tiles: a(i, kt) gives b at row 4 kt + t (0 past N).  Rows past N read the padding of
// the column; their sums are not used.  LEFT: also lacc[i]: <l, b> for the left
// vector l of lane column g (null: 0).
template <int NT, int NI, bool LEFT, typename A>
__device__ __forceinline__ void tc_product(const double* op, int ap, int N, int g, int t, A&& a, double (&acc)[NI][NT][2],
                                           const double* l, double (&lacc)[NI][2]) {
#pragma unroll
  for (int i = 0; i < NI; ++i) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[i][nt][0] = acc[i][nt][1] = 0.0;
    lacc[i][0] = lacc[i][1] = 0.0;
  }
  const double* o = op + t * ap + g;
#pragma unroll
  for (int kt = 0; kt < 2 * NT; ++kt, o += 4 * ap)
    if (4 * kt < N) {  // the same for the whole warp
      double b[NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) b[i] = a(i, kt);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const double ov = o[8 * nt];
#pragma unroll
        for (int i = 0; i < NI; ++i) dmma884(acc[i][nt][0], acc[i][nt][1], b[i], ov);
      }
      if (LEFT) {
        const double lv = l ? l[4 * kt + t] : 0.0;
#pragma unroll
        for (int i = 0; i < NI; ++i) dmma884(lacc[i][0], lacc[i][1], b[i], lv);
      }
    }
}
// acc -= A^-1 e_0 z0 + A^-1 e_{N-1} z1 (z0, z1 of right-hand side g; 0 without that neighbour)
template <int NT>
__device__ __forceinline__ void tc_rank2(const double* op, int ap, int N, int g, int t, double z0, double z1,
                                         double (&acc)[NT][2]) {
  const double* o = op + (t == 1 ? (N - 1) * ap : 0) + g;
  const double b = t == 0 ? -z0 : t == 1 ? -z1 : 0.0;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) dmma884(acc[nt][0], acc[nt][1], b, o[8 * nt]);
}
// Accumulators v[nt][h] (row 8 nt + 2 t + h of lane (g, t)) as the A operand of the next
// product: row 4 kt + t
template <int NT, typename V>
__device__ __forceinline__ double tc_next(const V (&v)[NT][2], int kt, int g, int t) {
  const int src = 4 * g + 2 * (kt & 1) + (t >> 1);
  const V a = __shfl_sync(0xffffffffu, v[kt >> 1][0], src), b = __shfl_sync(0xffffffffu, v[kt >> 1][1], src);
  return (double)((t & 1) ? b : a);
}
// Lanes of an even and an odd right-hand side (re, im of one column) swap values
// so that each holds one complex value: row 8 nt + 2 t of the even lane, the next row of
// the odd one.
template <typename T>
__device__ __forceinline__ typename Pair<T>::t tc_pair(T v0, T v1, int g) {
  const bool odd = g & 1;
  const T r = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 4);
  typename Pair<T>::t o;
  o.x = odd ? r : v0;
  o.y = odd ? v1 : r;
  return o;
}
// z = M^-1 r for R right-hand sides, [e][r] in shared memory; ends synchronised
template <int R>
__device__ __forceinline__ void tc_interface(const double* sM, const double* srz, double* szz, int m, int nr) {
  __syncthreads();
  for (int q = threadIdx.x; q < m * R; q += blockDim.x) {
    const int e = q / R, r = q - e * R;
    if (r >= nr) continue;
    const double* mr = sM + (size_t)e * m;
    double z = 0.0;
#pragma unroll 4
    for (int c = 0; c < m; ++c) z = __fma_rn(mr[c], srz[(size_t)c * R + r], z);
    szz[q] = z;
  }
  __syncthreads();
}
// nb column-major N x N operators into AP-strided columns, each block followed by zero
// columns up to a multiple of 4; a warp takes every nw-th column
__device__ __forceinline__ void tc_columns(double* dst, const double* src, int nb, int N) {
  const int AP = tc_ap(N), NC = tc_nc(N), lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int b = 0; b < nb; ++b, dst += NC * AP, src += N * N) {
    const double* s = src + w * N + lane;
    double* d = dst + w * AP + lane;
    for (int c = w; c < NC; c += nw, s += nw * N, d += nw * AP) {
      if (c >= N) {
        if (lane < AP) *d = 0.0;
        if (lane + 32 < AP) d[32] = 0.0;
      } else {
        if (lane < N) cp_async_8(d, s);
        if (lane + 32 < N) cp_async_8(d + 32, s + 32);
      }
    }
  }
}
// the system's inverse blocks, left vectors and interface matrix
__device__ __forceinline__ void tc_tables(const double* ag, const double* lg, const double* mg, int nb, int N, int m,
                                          double* sA, double* sL, double* sM) {
  tc_columns(sA, ag, nb, N);
  for (int q = threadIdx.x; q < m * N; q += blockDim.x) cp_async_8(sL + q, lg + q);
  for (int q = threadIdx.x; q < m * m; q += blockDim.x) cp_async_8(sM + q, mg + q);
}

// A warp's gather of NS column slots (lane i < NS holds slot i's column, -1: none)
// from scratch fields of whole columns, [column][k] complex: consecutive lanes
// read consecutive rows of one column.
template <typename T, int NS, typename S, typename D>
__device__ __forceinline__ void tc_gather_cols(int c, int N, int lane, S&& src, D&& dst) {
  typedef typename Pair<T>::t P2;
  int slot = lane / N, r = lane - slot * N;
  for (int b = 0; b < NS * N; b += 32) {
    const int cs = __shfl_sync(0xffffffffu, c, min(slot, NS - 1));
    if (slot < NS) {
      P2* d = dst(slot, r);
      if (cs >= 0)
        cp_async_c<P2>(d, src(slot, r, cs));
      else
        *d = P2{0, 0};
    }
    r += 32;
    while (r >= N) {
      r -= N;
      ++slot;
    }
  }
}

// The u/v, w and rho solves do not depend on one another: one launch takes up
// to three of them as jobs.
template <typename T>
struct TcJob {
  const double *ainv, *lvec, *minv;
  const SysDesc* sys;
  const Task* tasks;
  int first;     // first CTA of the job
  int per;       // right-hand sides per column: 4 (u/v) or 2
  int zero00;    // the (0,0) column has no system and becomes 0 (w)
  int meanu;     // damp the (0,0) column of F0
  double rdiv, irdiv;
  T *F0, *F1;           // results
  const T *S0, *S1;     // right-hand sides: the same fields, or with cols scratch fields of whole columns
};
template <typename T>
struct TcJobs {
  TcJob<T> j[3];
  int n, nb, cols;
  int bmap[IW_MAX_SUBD];
};
template <typename T, int NT>
__global__ void __maxnreg__(NT <= 2 ? 56 : NT == 3 ? 64 : 80) k_solve_tc(Geo g, const __grid_constant__ TcJobs<T> jobs,
                                                  const int* __restrict__ col_order,
                                                  const double* __restrict__ meang) {
  typedef typename Pair<T>::t P2;
  constexpr int R = 16;
  extern __shared__ __align__(16) unsigned char smraw[];
  int ji = 0;
  while (ji + 1 < jobs.n && (int)blockIdx.x >= jobs.j[ji + 1].first) ++ji;
  const TcJob<T>& J = jobs.j[ji];
  const Task tk = J.tasks[(int)blockIdx.x - J.first];
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1), nb = jobs.nb, s = tk.sys;
  const int tid = threadIdx.x, lane = tid & 31, ks = tid >> 5, lg = lane >> 2, lt = lane & 3;
  const int AP = tc_ap(N);
  const bool uv = J.per == 4;
  const TcSmem L = tc_smem<T>(n, N, ns, nb, false);
  double* sA = (double*)(smraw + L.a);
  double* sL = (double*)(smraw + L.l);
  double* sM = (double*)(smraw + L.m);
  double* srz = (double*)(smraw + L.rz);
  double* szz = (double*)(smraw + L.zz);
  T* raw = (T*)(smraw + L.raw) + (size_t)ks * N * 8;  // this warp's rows of tile 0
  const size_t ts = (size_t)n * 8;                    // tile stride
  const int count = tk.count, nr = count * J.per, nmt = nr > 8 ? 2 : 1;
  {
    // complex slot sl of the 8 (2 tiles of 4): column sl (w, rho) or u, v of column sl / 2
    const int sl = lane & 7, ci = uv ? sl >> 1 : sl;
    const int c = ci < count ? col_order[tk.first + ci] : -1;
    if (jobs.cols) {
      tc_gather_cols<T, 8>(c, N, lane, [&](int slot, int r, int cs) -> const P2* {
        return (const P2*)(((uv && (slot & 1)) ? J.S1 : J.S0) + ((size_t)cs * n + ks * N + r) * 2);
      }, [&](int slot, int r) { return (P2*)(raw + (slot >> 2) * ts + tc_pos<T>(r, 2 * (slot & 3))); });
    } else {
      const int cj = c / g.nxhp;
      const T* src = ((uv && (sl & 1)) ? J.S1 : J.S0) + (c < 0 ? 0 : fidx<T>(g, 2 * (c - cj * g.nxhp), cj, ks * N));
      T* dst = raw + (sl >> 2) * ts;
      const int p = 2 * (sl & 3);
      for (int r = lane >> 3; r < N; r += 4) {
        P2* d = (P2*)(dst + tc_pos<T>(r, p));
        if (c >= 0)
          cp_async_c<P2>(d, (const P2*)(src + (size_t)r * g.plane));
        else
          *d = P2{0, 0};
      }
    }
  }
  tc_tables(J.ainv + (size_t)s * nb * N * N, J.lvec + (size_t)s * m * N, J.minv + (size_t)s * m * m, nb, N, m, sA, sL,
                sM);
  if (J.zero00 && (int)blockIdx.x == J.first)  // (0,0) column: element 0 of every plane
    for (int k = tid; k < n; k += blockDim.x) *(P2*)(J.F0 + (size_t)k * g.plane) = P2{0, 0};
  const double eps = J.sys[s].eps, rdiv = J.rdiv, irdiv = J.irdiv;
  cp_async_wait_all();
  __syncthreads();
  const bool lo = ks >= 1, hi = ks <= ns - 2;  // neighbours below and above
  // left vectors: c_{ks+1} on this block (lane column 0), d_{ks-1} (lane column 1)
  const double* l = lg == 0 ? (hi ? sL + (size_t)ks * N : nullptr) : lg == 1 && lo ? sL + (size_t)(ns - 2 + ks) * N : nullptr;
  const double* op = sA + (size_t)jobs.bmap[ks] * tc_nc(N) * AP;
  // right-hand side at row 4 kt + t: its place in the tile differs from that of row t by a constant of kt
  const T* rl[2] = {raw + tc_pos<T>(lt, lg), raw + ts + tc_pos<T>(lt, lg)};
  auto rhs = [&](int i, int kt) -> double {
    double v = 0.0;
    if ((NT > 2 && kt < 2 * NT - 2) || 4 * kt + lt < N) v = __dmul_rn(div_by((double)rl[i][32 * kt], rdiv, irdiv), eps);
    return v;
  };
  auto body = [&](auto ni) {
    constexpr int NI = decltype(ni)::value;
    double acc[NI][NT][2], lacc[NI][2];
    tc_product<NT, NI, true>(op, AP, N, lg, lt, rhs, acc, l, lacc);
    if (m > 0) {
      if (lt == 0) {
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          if (hi) srz[(size_t)ks * R + 8 * i + lg] = lacc[i][0];
          if (lo) srz[(size_t)(ns - 2 + ks) * R + 8 * i + lg] = lacc[i][1];
        }
      }
      tc_interface<R>(sM, srz, szz, m, 8 * NI);
#pragma unroll
      for (int i = 0; i < NI; ++i)
        tc_rank2<NT>(op, AP, N, lg, lt, lo ? szz[(size_t)(ks - 1) * R + 8 * i + lg] : 0.0,
                     hi ? szz[(size_t)(ns - 1 + ks) * R + 8 * i + lg] : 0.0, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int slot = 4 * i + (lg >> 1), ci = uv ? slot >> 1 : slot;
      const int c = ci < count ? col_order[tk.first + ci] : -1;
      const int jj = c / g.nxhp;
      T* dst = ((uv && (slot & 1)) ? J.F1 : J.F0) + (c < 0 ? 0 : fidx<T>(g, 2 * (c - jj * g.nxhp), jj, ks * N));
      const bool mean = J.meanu && c == 0 && !(slot & 1);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int r = 8 * nt + 2 * lt, ro = r + (lg & 1);
        double v0 = acc[i][nt][0], v1 = acc[i][nt][1];
        if (mean) {
          v0 = __dmul_rn(meang[ks * N + min(r, N - 1)], v0);
          v1 = __dmul_rn(meang[ks * N + min(r + 1, N - 1)], v1);
        }
        const P2 o = tc_pair<T>((T)v0, (T)v1, lg);
        if (c >= 0 && ro < N) *(P2*)(dst + (size_t)ro * g.plane) = o;
      }
    }
  };
  if (nmt == 2)
    body(std::integral_constant<int, 2>());
  else
    body(std::integral_constant<int, 1>());
}

// Pressure and projection (calcuvwt.f:87-229, 826-901), 4 columns (8 right-hand
// sides) per CTA; blockIdx.y takes the task's other columns.
template <typename T, int NT>
__global__ void __maxnreg__(NT <= 4 ? 64 : 80) k_press_tc(Geo g, const __grid_constant__ BlockInv bi,
                                                  const Task* __restrict__ tasks, const int* __restrict__ col_order,
                                                  T* __restrict__ U, T* __restrict__ V, T* __restrict__ W,
                                                  const double* __restrict__ Dt, const double* __restrict__ wnl,
                                                  const double* __restrict__ wvr, int kstart, int cols) {
  typedef typename Pair<T>::t P2;
  constexpr int R = 8;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Task tk = tasks[blockIdx.x];
  const int count = min(tk.count - 4 * (int)blockIdx.y, 4);
  if (count <= 0) return;
  const int* order = col_order + tk.first + 4 * blockIdx.y;
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1), nb = bi.nb, s = tk.sys;
  const int tid = threadIdx.x, lane = tid & 31, ks = tid >> 5, lg = lane >> 2, lt = lane & 3;
  const int AP = tc_ap(N);
  const TcSmem L = tc_smem<T>(n, N, ns, nb, true);
  double* sA = (double*)(smraw + L.a);
  double* sL = (double*)(smraw + L.l);
  double* sM = (double*)(smraw + L.m);
  double* srz = (double*)(smraw + L.rz);
  double* szz = (double*)(smraw + L.zz);
  double* sD = (double*)(smraw + L.d);
  T* raw = (T*)(smraw + L.raw) + (size_t)ks * N * 8;
  const size_t ts = (size_t)n * 8;
  {
    const int ci = lane & 3;
    const int c = ci < count ? order[ci] : -1;
    const int cj = c / g.nxhp;
    const size_t cb = c < 0 ? 0 : fidx<T>(g, 2 * (c - cj * g.nxhp), cj, ks * N);
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const T* src = f == 0 ? U : f == 1 ? V : W;
      if (cols) {
        tc_gather_cols<T, 4>(c, N, lane, [&](int, int r, int cs) -> const P2* {
          return (const P2*)(src + ((size_t)cs * n + ks * N + r) * 2);
        }, [&](int slot, int r) { return (P2*)(raw + f * ts + tc_pos<T>(r, 2 * slot)); });
      } else {
        for (int r = lane >> 2; r < N; r += 8) {
          P2* d = (P2*)(raw + f * ts + tc_pos<T>(r, 2 * ci));
          if (c >= 0)
            cp_async_c<P2>(d, (const P2*)(src + cb + (size_t)r * g.plane));
          else
            *d = P2{0, 0};
        }
      }
    }
  }
  tc_columns(sD, Dt, 1, N);
  tc_tables((const double*)bi.ainv + (size_t)s * nb * N * N, bi.lvec + (size_t)s * m * N, bi.minv + (size_t)s * m * m, nb,
                N, m, sA, sL, sM);
  const double eps = bi.sys[s].eps, dt = g.dt, fac = g.hfac[ks];
  const int c = (lg >> 1) < count ? order[lg >> 1] : -1;
  const bool cok = c >= 0;
  const int cj = cok ? c / g.nxhp : 0, cii = cok ? c - cj * g.nxhp : 0;
  const double xw = g.xw[cii], yw = g.yw[cj];
  cp_async_wait_all();
  __syncthreads();
  const bool lo = ks >= 1, hi = ks <= ns - 2, im = lg & 1;
  const double* l = lg == 0 ? (hi ? sL + (size_t)ks * N : nullptr) : lg == 1 && lo ? sL + (size_t)(ns - 2 + ks) * N : nullptr;
  const double* op = sA + (size_t)bi.bmap[ks] * tc_nc(N) * AP;
  const T *ru = raw, *rv = raw + ts, *rw = raw + 2 * ts;
  double acc[1][NT][2], bv[NT][2], lacc[1][2];
  const T* wl = rw + tc_pos<T>(lt, lg);
  tc_product<NT, 1, false>(sD, AP, N, lg, lt, [&](int, int kt) {
    double v = 0.0;
    if ((NT > 2 && kt < 2 * NT - 2) || 4 * kt + lt < N) v = (double)wl[32 * kt];
    return v;
  }, acc, nullptr, lacc);
  // b = -((i kx u* + i ky v* + (2/h) D w*) / dt) eps and the Neumann data at the walls
  const double idt = __drcp_rn(dt);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * nt + 2 * lt + h, k = ks * N + r;
      double v = 0.0;
      if (r < N) {
        const double up = (double)ru[tc_pos<T>(r, lg ^ 1)], vp = (double)rv[tc_pos<T>(r, lg ^ 1)];
        const double b = __fma_rn(xw, up, __dmul_rn(yw, vp));
        const double div = __fma_rn(acc[0][nt][h], fac, im ? b : -b);
        v = -__dmul_rn(div_by(div, dt, idt), eps);
        if (cok && k == 0) {
          const size_t p1 = (size_t)g.nxpp * cj + 2 * cii + im;
          v = __fma_rn(-__dmul_rn(bi.sys[s].tau1_bot, __dadd_rn(wnl[p1], wvr[p1])), eps, v);
        }
        if (cok && k == n - 1) {
          const size_t p2 = (size_t)g.nxpp * (cj + g.ny) + 2 * cii + im;
          v = __fma_rn(__dmul_rn(bi.sys[s].tau2_top, __dadd_rn(wnl[p2], wvr[p2])), eps, v);
        }
      }
      bv[nt][h] = v;
    }
  tc_product<NT, 1, true>(op, AP, N, lg, lt, [&](int, int kt) { return tc_next<NT>(bv, kt, lg, lt); }, acc, l, lacc);
  if (m > 0) {
    if (lt == 0) {
      if (hi) srz[(size_t)ks * R + lg] = lacc[0][0];
      if (lo) srz[(size_t)(ns - 2 + ks) * R + lg] = lacc[0][1];
    }
    tc_interface<R>(sM, srz, szz, m, R);
    tc_rank2<NT>(op, AP, N, lg, lt, lo ? szz[(size_t)(ks - 1) * R + lg] : 0.0,
                 hi ? szz[(size_t)(ns - 1 + ks) * R + lg] : 0.0, acc[0]);
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) bv[nt][h] = 8 * nt + 2 * lt + h < N ? acc[0][nt][h] : 0.0;
  tc_product<NT, 1, false>(sD, AP, N, lg, lt, [&](int, int kt) { return tc_next<NT>(bv, kt, lg, lt); }, acc, nullptr, lacc);
  const double dtx = __dmul_rn(dt, xw), dty = __dmul_rn(dt, yw);
  const size_t cb = cols ? ((size_t)max(c, 0) * n + ks * N) * 2 : fidx<T>(g, 2 * cii, cj, ks * N);
  const size_t rs = cols ? 2 : g.plane;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    T u[2], v[2], w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * nt + 2 * lt + h, p = tc_pos<T>(min(r, N - 1), lg);
      const double pp = __shfl_xor_sync(0xffffffffu, bv[nt][h], 4);  // the other part of phi
      u[h] = (T)__fma_rn(im ? -dtx : dtx, pp, (double)ru[p]);
      v[h] = (T)__fma_rn(im ? -dty : dty, pp, (double)rv[p]);
      w[h] = (T)__fma_rn(-dt, __dmul_rn(acc[0][nt][h], fac), (double)rw[p]);
      if (ks * N + r < kstart) u[h] = v[h] = w[h] = (T)0;
    }
    const P2 zu = tc_pair<T>(u[0], u[1], lg), zv = tc_pair<T>(v[0], v[1], lg), zw = tc_pair<T>(w[0], w[1], lg);
    const int ro = 8 * nt + 2 * lt + (lg & 1);
    if (cok && ro < N) {
      const size_t p = cb + (size_t)ro * rs;
      *(P2*)(U + p) = zu;
      *(P2*)(V + p) = zv;
      *(P2*)(W + p) = zw;
    }
  }
}

// Isolated solves (iw_helm_solve_batched, mode 0) with the products of k_solve_tc and one
// FP64 residual sweep, x += A^-1 (b - A x): the penalty rows of A are large, and the sweep
// brings the residual of the block-inverse form to that of the pivoted band LU.
// Right-hand sides and solutions are whole columns, [column][k] complex; 4 columns (8
// right-hand sides) per CTA, blockIdx.y takes the task's other columns.  x, A x and the
// residual stay in accumulator registers; the CTA exchanges four numbers per block and
// right-hand side (the boundary values and derivatives) for the coupling rows.
// 33024 columns of 8 x 25 points: 8.8 ms with the band LU (a warp per column, bound by the
// latency of its serial sweep).
struct HelmTc {
  const double *ainv, *lvec, *minv, *pen, *D, *D2t, *zh;
  const SysDesc* sys;
  const Task* tasks;
  const int* order;
  const double* rhs;
  double* sol;
  int nb;
  int bmap[IW_MAX_SUBD];
};
struct HelmSmem {  // byte offsets
  size_t a, l, m, rz, zz, d2, dr, ex, raw, total;
};
__host__ __device__ inline HelmSmem helm_smem(int n, int N, int ns, int nb) {
  HelmSmem o;
  const size_t m = 2 * (size_t)(ns - 1), ap = tc_ap(N), D = sizeof(double);
  o.a = 0;
  o.l = o.a + (size_t)nb * tc_nc(N) * ap * D;
  o.m = o.l + m * N * D;
  o.rz = o.m + m * m * D;
  o.zz = o.rz + m * 8 * D;
  o.d2 = o.zz + m * 8 * D;
  o.dr = o.d2 + (size_t)tc_nc(N) * ap * D;
  o.ex = o.dr + 2 * (size_t)tc_nc(N) * D;
  o.raw = o.ex + (size_t)ns * 4 * 8 * D;
  o.total = o.raw + (size_t)n * 8 * D + 16 * D;
  return o;
}
template <int NT>
__global__ void __maxnreg__(NT <= 3 ? 64 : 80) k_helm_tc(Geo g, const __grid_constant__ HelmTc H) {
  constexpr int R = 8;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Task tk = H.tasks[blockIdx.x];
  const int count = min(tk.count - 4 * (int)blockIdx.y, 4);
  if (count <= 0) return;
  const int* order = H.order + tk.first + 4 * blockIdx.y;
  const int n = g.nz, N = g.N, ns = g.ns, m = 2 * (ns - 1), s = tk.sys;
  const int tid = threadIdx.x, lane = tid & 31, ks = tid >> 5, lg = lane >> 2, lt = lane & 3;
  const int AP = tc_ap(N);
  const HelmSmem L = helm_smem(n, N, ns, H.nb);
  double* sA = (double*)(smraw + L.a);
  double* sL = (double*)(smraw + L.l);
  double* sM = (double*)(smraw + L.m);
  double* srz = (double*)(smraw + L.rz);
  double* szz = (double*)(smraw + L.zz);
  double* sD2 = (double*)(smraw + L.d2);
  double* sDr = (double*)(smraw + L.dr);  // rows 0 and N - 1 of D
  double* ex = (double*)(smraw + L.ex);   // [block][x_0, x_{N-1}, (D x)_0, (D x)_{N-1}][R]
  double* raw = (double*)(smraw + L.raw) + (size_t)ks * N * 8;
  {
    const int ci = lane & 3;
    const int c = ci < count ? order[ci] : -1;
    tc_gather_cols<double, 4>(c, N, lane, [&](int, int r, int cs) {
      return (const double2*)(H.rhs + ((size_t)cs * n + ks * N + r) * 2);
    }, [&](int slot, int r) { return (double2*)(raw + tc_pos<double>(r, 2 * slot)); });
  }
  tc_columns(sD2, H.D2t, 1, N);
  tc_tables(H.ainv + (size_t)s * H.nb * N * N, H.lvec + (size_t)s * m * N, H.minv + (size_t)s * m * m, H.nb, N, m, sA, sL, sM);
  for (int q = tid; q < 2 * tc_nc(N); q += blockDim.x) {
    const int c = q % tc_nc(N), row = q / tc_nc(N);
    sDr[q] = c < N ? H.D[(row ? N - 1 : 0) * N + c] : 0.0;
  }
  const double eps = H.sys[s].eps;
  cp_async_wait_all();
  __syncthreads();
  const bool lo = ks >= 1, hi = ks <= ns - 2;
  const double* l = lg == 0 ? (hi ? sL + (size_t)ks * N : nullptr) : lg == 1 && lo ? sL + (size_t)(ns - 2 + ks) * N : nullptr;
  const double* op = sA + (size_t)H.bmap[ks] * tc_nc(N) * AP;
  double acc[1][NT][2], lacc[1][2], xv[NT][2], rv[NT][2];
  auto solve = [&](auto&& rhs) {  // acc = A^-1 rhs
    tc_product<NT, 1, true>(op, AP, N, lg, lt, rhs, acc, l, lacc);
    if (m > 0) {
      if (lt == 0) {
        if (hi) srz[(size_t)ks * R + lg] = lacc[0][0];
        if (lo) srz[(size_t)(ns - 2 + ks) * R + lg] = lacc[0][1];
      }
      tc_interface<R>(sM, srz, szz, m, R);
      tc_rank2<NT>(op, AP, N, lg, lt, lo ? szz[(size_t)(ks - 1) * R + lg] : 0.0,
                   hi ? szz[(size_t)(ns - 1 + ks) * R + lg] : 0.0, acc[0]);
    }
  };
  const double* bl = raw + tc_pos<double>(lt, lg);
  solve([&](int, int kt) {
    double v = 0.0;
    if ((NT > 2 && kt < 2 * NT - 2) || 4 * kt + lt < N) v = bl[32 * kt];
    return v;
  });
  double* e = ex + (size_t)ks * 4 * R;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * nt + 2 * lt + h;
      xv[nt][h] = r < N ? acc[0][nt][h] : 0.0;
      if (r == 0) e[lg] = xv[nt][h];
      if (r == N - 1) e[R + lg] = xv[nt][h];
    }
  // D2 x and the derivatives at both ends of the block
  const double* dl = lg == 0 ? sDr : lg == 1 ? sDr + tc_nc(N) : nullptr;
  tc_product<NT, 1, true>(sD2, AP, N, lg, lt, [&](int, int kt) { return tc_next<NT>(xv, kt, lg, lt); }, acc, dl, lacc);
  if (lt == 0) {
    e[2 * R + lg] = lacc[0][0];
    e[3 * R + lg] = lacc[0][1];
  }
  __syncthreads();
  const double* pen = H.pen + (size_t)s * 6 * ns;
  const double h2 = 2.0 / H.zh[ks], ee = eps * (h2 * h2);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 8 * nt + 2 * lt + h;
      rv[nt][h] = 0.0;
      if (r < N) {
        double v = xv[nt][h] - ee * acc[0][nt][h];
        if (r == 0) {
          const double pa = pen[ks], pb = pen[ns + ks], t1 = pen[4 * ns + ks], s0 = e[2 * R + lg];
          v += t1 * pa * xv[nt][h] - t1 * pb * eps * h2 * s0;
          if (lo) {
            const double* el = e - 4 * R;
            v += -0.5 * t1 * pa * xv[nt][h] + 0.5 * t1 * pb * eps * h2 * s0 - 0.5 * t1 * pa * el[R + lg] +
                 0.5 * t1 * pb * eps * (2.0 / H.zh[ks - 1]) * el[3 * R + lg];
          }
        }
        if (r == N - 1) {
          const double pg = pen[2 * ns + ks], pd = pen[3 * ns + ks], t2 = pen[5 * ns + ks], s1 = e[3 * R + lg];
          v += t2 * pg * xv[nt][h] + t2 * pd * eps * h2 * s1;
          if (hi) {
            const double* eh = e + 4 * R;
            v += -0.5 * t2 * pg * xv[nt][h] - 0.5 * t2 * pd * eps * h2 * s1 - 0.5 * t2 * pg * eh[lg] -
                 0.5 * t2 * pd * eps * (2.0 / H.zh[ks + 1]) * eh[2 * R + lg];
          }
        }
        rv[nt][h] = raw[tc_pos<double>(r, lg)] - v;
      }
    }
  solve([&](int, int kt) { return tc_next<NT>(rv, kt, lg, lt); });
  const int c = (lg >> 1) < count ? order[lg >> 1] : -1;
  double* dst = H.sol + ((size_t)max(c, 0) * n + ks * N) * 2;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const double2 o = tc_pair<double>(xv[nt][0] + acc[0][nt][0], xv[nt][1] + acc[0][nt][1], lg);
    const int ro = 8 * nt + 2 * lt + (lg & 1);
    if (c >= 0 && ro < N) *(double2*)(dst + 2 * (size_t)ro) = o;
  }
}

// ===========================================================================
// z-column stages on the FP64 tensor cores (N <= 40), for either storage type.
// A warp owns 8 consecutive points of the flattened (x, y) plane of one field and
// subdomain, i.e. one row tile of the products X^T = F^T Op^T of k_solve_tc: lane
// (g, t) holds point g, the operand rows 4 kt + t and the result rows 8 nt + 2 t + h.
// D and L - I sit in shared memory once per persistent CTA; warps work on their own,
// without CTA-wide barriers, and walk the tiles in the order of memory, so that the
// SMs stay on the same few hundred pages (z-planes are a megabyte and more apart).  The
// products run in FP64 whatever the storage type, with one rounding of each result to
// it (FP64 fields: the FMA chain, i.e. the bits, of the tiled kernels).
// ===========================================================================
__device__ __forceinline__ void z_ops(double* op, const double* __restrict__ rowmajor, int N, int ap, bool minus1) {
  for (int q = threadIdx.x; q < tc_nc(N) * ap; q += blockDim.x) {
    const int c = q / ap, r = q - c * ap;
    op[q] = r < N && c < N ? rowmajor[r * N + c] - (minus1 && r == c ? 1.0 : 0.0) : 0.0;
  }
}
// A warp's walk over the tiles: first point t0 of the plane and (subdomain, field) row
struct ZWalk {
  unsigned t0, row, step, plane8;
  __device__ __forceinline__ ZWalk(unsigned plane) {
    plane8 = (plane + 7) & ~7u;
    step = ((gridDim.x * blockDim.x) >> 5) * 8;
    t0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 8;
    row = t0 / plane8;
    t0 -= row * plane8;
  }
  __device__ __forceinline__ void next() {
    t0 += step;
    while (t0 >= plane8) {
      t0 -= plane8;
      ++row;
    }
  }
};
// K_A: projection, w mean = 0, z derivative (proj < 0: the derivative alone, nothing
// is written to O).  The N x 8 operand goes from global memory straight to
// registers.
template <typename T, int NT>
__global__ void __launch_bounds__(512, 2) k_stageA_t(Geo g, const T* __restrict__ F0, const T* __restrict__ F1_,
                                                     const T* __restrict__ F2_, const T* __restrict__ F3_,
                                                     T* __restrict__ O0, T* __restrict__ O1, T* __restrict__ O2,
                                                     T* __restrict__ O3, T* __restrict__ Z0, T* __restrict__ Z1,
                                                     T* __restrict__ Z2, T* __restrict__ Z3, int proj,
                                                     int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* sD = (double*)smraw;
  const int N = g.N, AP = tc_ap(N), lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
  z_ops(sD, g.D, N, AP, false);
  __syncthreads();
  const unsigned pl = (unsigned)g.plane, nxpp = (unsigned)g.nxpp, rows = 4 * g.ns;
  const size_t pl4 = (size_t)4 * pl, pl8 = (size_t)8 * pl;
  const unsigned nx = (unsigned)g.nx;
  for (ZWalk w(pl); w.row < rows; w.next()) {
    const int q = w.row & 3, ks = w.row >> 2;
    const unsigned tt = w.t0 + lg, j = tt / nxpp, i = tt - j * nxpp;
    const size_t k0 = (size_t)(ks * N) * pl;
    const T* F = (q == 0 ? F0 : q == 1 ? F1_ : q == 2 ? F2_ : F3_) + k0;
    T* O = (q == 0 ? O0 : q == 1 ? O1 : q == 2 ? O2 : O3) + k0;
    T* Z = q == 0 ? Z0 : q == 1 ? Z1 : q == 2 ? Z2 : Z3;
    const double fac = g.hfac[ks];
    // the projection changes the kx = 0 and Nyquist columns
    const bool special = (proj > 0 && (i < 2 || i >= nx)) || (proj >= 0 && q == 2 && tt < 2);
    auto tile = [&](auto plain_) {
      constexpr bool PLAIN = decltype(plain_)::value;  // a whole tile of points the projection leaves alone
      const bool act = PLAIN || tt < pl;
      auto in = [&](int r, int last) { return ((NT > 2 && last < 8 * (NT - 1)) || r < N) && act; };  // rows <= last < N need no test
      T x[2 * NT];
      const T* f = F + tt + (size_t)lt * pl;
#pragma unroll
      for (int kt = 0; kt < 2 * NT; ++kt, f += pl4) {
        x[kt] = (T)0;
        if (in(4 * kt + lt, 4 * kt + 3)) x[kt] = *f;
      }
      // non-finite values are looked for after the projection, which drops the imaginary part of
      // the x-Nyquist column (the derivative alone: in the raw values)
      if (!PLAIN && special && proj > 0) {
#pragma unroll
        for (int kt = 0; kt < 2 * NT; ++kt)
          if (act && 4 * kt + lt < N) x[kt] = proj_val<T>(g, F, i, j, 4 * kt + lt);
      }
      bool bad = false;
#pragma unroll
      for (int kt = 0; kt < 2 * NT; ++kt) bad |= !isfinite(x[kt]);
      if (!PLAIN && proj >= 0 && q == 2 && tt < 2) {  // the mean of w
#pragma unroll
        for (int kt = 0; kt < 2 * NT; ++kt) x[kt] = (T)0;
      }
      if (bad) err[0] = 1;  // the state of the last step holds a NaN or Inf
      if (proj >= 0) {
        T* o = O + tt + (size_t)lt * pl;
#pragma unroll
        for (int kt = 0; kt < 2 * NT; ++kt, o += pl4)
          if (in(4 * kt + lt, 4 * kt + 3)) *o = x[kt];
      }
      if (Z == nullptr) return;
      double acc[1][NT][2], none[1][2];
      tc_product<NT, 1, false>(sD, AP, N, lg, lt, [&](int, int kt) { return (double)x[kt]; }, acc, nullptr, none);
      T* z = Z + k0 + tt + (size_t)(2 * lt) * pl;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt, z += pl8)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (in(8 * nt + 2 * lt + h, 8 * nt + 7)) z[h * (size_t)pl] = (T)__dmul_rn(acc[0][nt][h], fac);
    };
    if (__any_sync(0xffffffffu, special || tt >= pl))
      tile(std::false_type());
    else
      tile(std::true_type());
  }
}

// K_E.  Each warp stages its 7 x N rows of 8 points by cp.async; the next tile's copies
// go out as soon as the inputs are consumed, before the filter product and the
// stores.  cols: the filtered u* goes to a scratch field as whole columns, [column][k] complex,
// where the solves read it without strided accesses (a.F then is that scratch).
constexpr int kZArr = 7;  // Z, B, S_n, S_{n-1}, F1, F_n, F_{n-1}
// Staged place of row r, in rows [place][array][8 points]: rows of one parity take
// consecutive places, so the rows 2 t of a read in the layout of the results fall in
// different banks (of FP64 rows the halves also swap on every other pair of places).
__host__ __device__ __forceinline__ int ze_place(int r) { return (r & ~7) | ((r & 1) << 2) | ((r >> 1) & 3); }
template <typename T>
__device__ __forceinline__ int ze_pos(int r, int arr, int u) {
  const int sl = ze_place(r);
  return (sl * kZArr + arr) * 8 + (sizeof(T) == 8 ? u ^ (((sl >> 1) & 1) << 2) : u);
}
template <typename T>
__host__ __device__ inline size_t ze_buf(int N) {  // bytes of one warp's tiles
  int top = 0;
  for (int r = N & ~7; r < N; ++r) top = ze_place(r) > top ? ze_place(r) : top;
  return (size_t)((N & 7) ? top + 1 : N) * kZArr * 8 * sizeof(T);
}
template <typename T, int NT>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 640 : 512) k_stageE_t(Geo g, const __grid_constant__ EArgs<T> a, Coefs c,
                                                                        int cols, int v16) {
  typedef typename Pair<T>::t P2;
  constexpr int EC = 16 / (int)sizeof(T), CH = 8 / EC;  // points per 16-byte copy, copies per row
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = g.N, AP = tc_ap(N), lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
  double* sD = (double*)smraw;
  double* sL = sD + tc_nc(N) * AP;
  T* buf = (T*)((unsigned char*)(sL + tc_nc(N) * AP + 8) + (size_t)(threadIdx.x >> 5) * ze_buf<T>(N));
  z_ops(sD, g.D, N, AP, false);
  z_ops(sL, g.Lfil, N, AP, true);
  __syncthreads();
  const unsigned pl = (unsigned)g.plane, nxpp = (unsigned)g.nxpp, rows = 4 * g.ns;
  const size_t pl8 = (size_t)8 * pl;
  auto stage = [&](const ZWalk& w) {
    const int q = w.row & 3;
    const size_t o0 = (size_t)((int)(w.row >> 2) * N) * pl + w.t0;
#pragma unroll
    for (int arr = 0; arr < kZArr; ++arr) {
      const T* src = (arr == 0   ? a.Z[q]
                      : arr == 1 ? a.B[q]
                      : arr == 2 ? a.Snold[q]
                      : arr == 3 ? a.Snm_w[q]
                      : arr == 4 ? a.F1[q]
                      : arr == 5 ? a.Fn[q]
                                 : a.Fnm_w[q]) + o0;
      if (sizeof(T) == 8 || v16) {
        const int e = (lane % CH) * EC, rl = lane / CH;
        if (w.t0 + e < pl) {
          const T* s = src + e + (size_t)rl * pl;
          T* d = buf + ze_pos<T>(rl, arr, e);  // rows 8 apart: places 8 apart
#pragma unroll
          for (int m = 0; m < NT * CH / 4; ++m, s += (32 / CH) * (size_t)pl)
            if (m * (32 / CH) + rl < N) cp_async_c<double2>((double2*)(d + m * (32 / CH) * kZArr * 8), (const double2*)s);
          if ((NT * CH) % 4 != 0) {
            const int m = NT * CH / 4;
            if (m * (32 / CH) + rl < N) cp_async_c<double2>((double2*)(d + m * (32 / CH) * kZArr * 8), (const double2*)s);
          }
        }
      } else {  // rows of odd planes start 8 bytes into a unit
        const int e = (lane & 3) * 2;
        if (w.t0 + e < pl) {
          const T* s = src + e + (size_t)(lane >> 2) * pl;
          for (int r = lane >> 2; r < N; r += 8, s += pl8)
            cp_async_c<float2>((float2*)(buf + ze_pos<T>(r, arr, e)), (const float2*)s);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const T f1 = (T)c.fac1, f2 = (T)c.fac2, f3 = (T)c.fac3;
  const T* eb = buf + ze_pos<T>(2 * lt, 1, lg);  // B at row 2 t
  const T* zl = buf + (4 * (lt & 1) + (lt >> 1)) * kZArr * 8;
  const T* const zb[2] = {zl + lg, zl + (sizeof(T) == 8 ? lg ^ 4 : lg)};  // Z at rows 4 kt + t, kt even, odd
  ZWalk w(pl);
  if (w.row < rows) stage(w);
  while (w.row < rows) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    const int q = w.row & 3, ks = w.row >> 2;
    const unsigned tt = w.t0 + lg;
    const bool act = tt < pl;
    const unsigned j = tt / nxpp, i = tt - j * nxpp;
    const bool special = act && (i < 2 || i >= (unsigned)g.nx);  // columns that the projection changes
    const bool wq = q == 2 && (ks == 0 || ks == g.ns - 1);       // this subdomain holds a wall row of w
    const size_t o0 = (size_t)(ks * N) * pl + tt, o2 = o0 + (size_t)(2 * lt) * pl;
    double acc[1][NT][2], none[1][2];
    T fs[NT][2];
    tc_product<NT, 1, false>(sD, AP, N, lg, lt, [&](int, int kt) {
      T z = (T)0;  // rows past N are not staged
      if ((NT > 2 && kt < 2 * NT - 2) || 4 * kt + lt < N) z = zb[kt & 1][(8 * (kt >> 1) + 2 * (kt & 1)) * kZArr * 8];
      return (double)z;
    }, acc, nullptr, none);
    const double fac = g.hfac[ks];
    auto points = [&](auto plain_) {
      constexpr bool PLAIN = decltype(plain_)::value;  // a whole tile without wall rows and special columns
      T *sw = a.Snm_w[q] + o2, *fw = a.Fnm_w[q] + o2;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt, sw += pl8, fw += pl8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 8 * nt + 2 * lt + h;
          fs[nt][h] = (T)0;
          if ((NT > 2 && nt < NT - 1) || r < N) {  // (needs no test but in the last tile)
            const T* e = eb + (8 * nt + 4 * h) * kZArr * 8;
            const T sn = e[8], snm = e[16];
            T F2 = e[24];
            if (!PLAIN && special) {
              if (i < 2) {
                const T vb = a.F1[q][fidx<T>(g, i, (g.ny - (int)j) % g.ny, ks * N + r)];
                F2 = i == 0 ? (T)0.5 * (F2 + vb) : (T)0.5 * (F2 - vb);
              } else {
                F2 = i == (unsigned)g.nx ? F2 * (T)g.scaley : (T)0;
              }
            }
            const T S = (T)__fma_rn(acc[0][nt][h], fac, (double)e[0]);
            const T se = fma_t(f3, snm, fma_t(f2, sn, mul_t(f1, S)));
            fs[nt][h] = bdf_combine_rn<T>(c, se, F2, e[32], e[40]);
            if (!PLAIN && wq && act && ((ks == 0 && r == 0) || (ks == g.ns - 1 && r == N - 1)))
              a.wnl[tt + (ks == 0 && r == 0 ? 0 : g.plane)] = stageE_wall<T>(f1, f2, f3, S, sn, snm);
            if (PLAIN || act) {
              sw[h * (size_t)pl] = S;
              fw[h * (size_t)pl] = F2;
            }
          }
        }
    };
    if (__any_sync(0xffffffffu, special || !act) || wq)
      points(std::false_type());
    else
      points(std::true_type());
    __syncwarp();
    w.next();
    if (w.row < rows) stage(w);
    if (a.filter)  // (L - I) F* in FP64
      tc_product<NT, 1, false>(sL, AP, N, lg, lt, [&](int, int kt) { return tc_next<NT>(fs, kt, lg, lt); }, acc, nullptr, none);
    const double cfm1 = act && a.filter ? g.cfour[j * (unsigned)g.nxhp + (i >> 1)] - 1.0 : 0.0;
    T* dst = cols ? a.F[q] + (size_t)(tt >> 1) * (2 * g.nz) + 2 * (ks * N + 2 * lt + (lg & 1)) : a.F[q] + o2;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      T o[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        o[h] = a.filter ? (T)stageE_filtered((double)fs[nt][h], acc[0][nt][h], cfm1) : fs[nt][h];
      const bool whole = NT > 2 && nt < NT - 1;
      if (cols) {
        const P2 p = tc_pair<T>(o[0], o[1], lg);
        if (act && (whole || 8 * nt + 2 * lt + (lg & 1) < N)) *(P2*)(dst + 16 * nt) = p;
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (act && (whole || 8 * nt + 2 * lt + h < N)) dst[h * (size_t)pl] = o[h];
        dst += pl8;
      }
    }
  }
}

// ===========================================================================
// Interface averaging (penalty.f:714-775).
// ===========================================================================
// apply the round-trip projection P in place to all planes except the
// interface planes (km, k of every interface), which go through real
// transforms instead.  Thread per (j, k, field) for the kx=0 pair and the
// Nyquist column.
template <typename T>
__global__ void k_project_planes(Geo g, T* F0, T* F1, T* F2, T* F3, int skip_iface) {
  // grid: x over y rows, y over z levels, z over the 4 fields (32-bit indices)
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.ny) return;
  const int k = blockIdx.y, q = blockIdx.z;
  if (skip_iface) {
    int kl = k % g.N;
    if ((kl == 0 && k > 0) || (kl == g.N - 1 && k < g.nz - 1)) return;
  }
  T* F = q == 0 ? F0 : q == 1 ? F1 : q == 2 ? F2 : F3;
  int jp = (g.ny - j) % g.ny;
  // Nyquist: independent per j
  size_t pn = fidx<T>(g, g.nx, j, k);
  F[pn] = F[pn] * (T)g.scaley;
  F[pn + 1] = 0;
  if (j <= jp) {
    size_t pa = fidx<T>(g, 0, j, k), pb = fidx<T>(g, 0, jp, k);
    T ar = F[pa], ai = F[pa + 1], br = F[pb], bi = F[pb + 1];
    T nr = (T)0.5 * (ar + br), ni = (T)0.5 * (ai - bi);
    F[pa] = nr;
    F[pa + 1] = ni;
    if (jp != j) {
      F[pb] = nr;
      F[pb + 1] = -ni;
    }
  }
}

// gather the 4 planes around each interface into a compact buffer:
// G[(q*(ns-1)+f)*4 + m] plane = F_q level (f+1)*N - 2 + m; back: add the
// averaging change held in G to the two interface planes.
// Grid: x over the points of a plane, y over the 16 (ns - 1) planes (no
// 64-bit division per element).
template <typename T>
__global__ void k_iface_gather(Geo g, const T* F0, const T* F1, const T* F2, const T* F3, T* G, int back) {
  const size_t per = g.plane;
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= per) return;
  const int pl = blockIdx.y;
  int m = pl % 4;
  int f = (pl / 4) % (g.ns - 1);
  int q = pl / (4 * (g.ns - 1));
  int k = (f + 1) * g.N - 2 + m;
  const T* F = q == 0 ? F0 : q == 1 ? F1 : q == 2 ? F2 : F3;
  if (!back) {
    G[(size_t)pl * per + e] = F[(size_t)k * per + e];
  } else if (m == 1 || m == 2) {
    ((T*)F)[(size_t)k * per + e] += G[(size_t)pl * per + e];  // spectral change made by the averaging
  }
}

// per (row j, interface plane group): x-inverse of 4 rows, average, x-forward
// of the change of the 2 interface rows.
template <typename T>
__global__ void k_iface_rows(Geo g, T* G, FftPlan pl, const typename cplx_t<T>::type* __restrict__ Wm,
                             const typename cplx_t<T>::type* __restrict__ Wn, int* counts) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int M = g.nx / 2, nx = g.nx;
  C* A = (C*)smraw;
  C* B = A + 4 * M;
  const int j = blockIdx.x;
  const int grp = blockIdx.y;  // q*(ns-1)+f
  const int q = grp / (g.ns - 1);
  const size_t per = g.plane;
  for (int m = 0; m < 4; ++m)
    xinv_prep<C, T>(G + (size_t)(grp * 4 + m) * per + (size_t)j * g.nxpp, A + m * M, M, Wn, 0, (T)0, threadIdx.x,
                    blockDim.x);
  __syncthreads();
  C* ph = fft_run<C>(A, B, pl, 4, Wm, true, threadIdx.x, blockDim.x);
  T* P = (T*)ph;
  int cnt = 0;
  // The interface rows become the change made by the averaging (0 where it
  // does not trigger): the spectral planes are then P(F) + transform of the
  // change, so points left alone never take the round trip's rounding.
  for (int i = threadIdx.x; i < nx; i += blockDim.x) {
    T fsp = P[2 * nx + i], fsm = P[1 * nx + i];
    T favg2 = fsp + fsm;
    T c0 = fabs(fsp - fsm) / fabs(favg2);
    T d1 = 0, d2 = 0;
    if (c0 > (T)0.005) {
      T ff = P[0 * nx + i] * (T)0.5 + P[1 * nx + i] * (T)0 + P[2 * nx + i] * (T)0 + P[3 * nx + i] * (T)0.5;
      d1 = ff - fsm;
      d2 = ff - fsp;
      ++cnt;
    }
    P[1 * nx + i] = d1;
    P[2 * nx + i] = d2;
  }
  if (cnt) atomicAdd(counts + q, cnt);
  __syncthreads();
  C* other = (ph == A) ? B : A;
  C* sp = fft_run<C>(ph + M, other + M, pl, 2, Wm, false, threadIdx.x, blockDim.x);
  const T invN = (T)1 / (T)nx;
  for (int t = threadIdx.x; t < 2 * (M + 1); t += blockDim.x) {
    int m = t / (M + 1), kk = t % (M + 1);
    C v = xfwd_post<C>(sp + m * M, kk, M, Wn, invN);
    T* p = G + (size_t)(grp * 4 + 1 + m) * per + (size_t)j * g.nxpp + 2 * kk;
    p[0] = v.x;
    p[1] = v.y;
  }
}

// ===========================================================================
// generic whole-field helpers for the Fortran-style entry points
// ===========================================================================
template <typename T>
__global__ void k_xfft_field(Geo g, T* F, int nk, int inv, FftPlan pl, const typename cplx_t<T>::type* __restrict__ Wm,
                             const typename cplx_t<T>::type* __restrict__ Wn) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int M = g.nx / 2, nx = g.nx;
  C* A = (C*)smraw;
  C* B = A + M;
  const int row = blockIdx.x;  // j + ny*k
  T* rp = F + (size_t)row * g.nxpp;
  if (inv) {
    xinv_prep<C, T>(rp, A, M, Wn, 0, (T)0, threadIdx.x, blockDim.x);
    __syncthreads();
    C* r = fft_run<C>(A, B, pl, 1, Wm, true, threadIdx.x, blockDim.x);
    T* P = (T*)r;
    for (int i = threadIdx.x; i < g.nxpp; i += blockDim.x) rp[i] = i < nx ? P[i] : (T)0;
  } else {
    for (int i = threadIdx.x; i < M; i += blockDim.x) A[i] = cmk<C>(rp[2 * i], rp[2 * i + 1]);
    __syncthreads();
    C* r = fft_run<C>(A, B, pl, 1, Wm, false, threadIdx.x, blockDim.x);
    const T invN = (T)1 / (T)nx;
    for (int t = threadIdx.x; t < M + 1; t += blockDim.x) {
      C v = xfwd_post<C>(r, t, M, Wn, invN);
      // write after everyone has read r: r is a different buffer than rp
      rp[2 * t] = v.x;
      rp[2 * t + 1] = v.y;
    }
  }
}

template <typename T>
__global__ void k_mulikx(Geo g, T* F) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long)(g.ntot / 2)) return;
  size_t p = 2 * (size_t)gid;
  int ii = (int)((p % g.nxpp) / 2);
  T kx = (T)g.xw[ii];
  T a = F[p], b = F[p + 1];
  F[p] = -(kx * b);
  F[p + 1] = kx * a;
}

template <typename T>
__global__ void k_dz_field(Geo g, const T* __restrict__ a, T* __restrict__ b) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long)g.ntot) return;
  size_t e = gid % g.plane;
  int k = gid / g.plane;
  int ks = k / g.N, k1 = k % g.N;
  double s = 0.0;
  for (int k2 = 0; k2 < g.N; ++k2) s += g.D[k1 * g.N + k2] * (double)a[(size_t)(ks * g.N + k2) * g.plane + e];
  b[gid] = (T)(s * g.hfac[ks]);
}

// filter_3dlegenfourier on a spectral field, in place
template <typename T>
__global__ void k_filter_field(Geo g, T* F, int ifourier, int ilegen) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long total = (long)g.nxpp * g.ny * g.ns;
  if (gid >= total) return;
  int i = gid % g.nxpp;
  long r = gid / g.nxpp;
  int j = r % g.ny;
  int ks = r / g.ny;
  const int N = g.N;
  double v[kMaxN];
  double cf = ifourier ? g.cfour[(size_t)j * g.nxhp + (i >> 1)] : 1.0;
  for (int k = 0; k < N; ++k) v[k] = (double)F[fidx<T>(g, i, j, ks * N + k)] * cf;
  for (int k1 = 0; k1 < N; ++k1) {
    double s = 0;
    if (ilegen)
      for (int k2 = 0; k2 < N; ++k2) s += g.Lfil[k1 * N + k2] * v[k2];
    else
      s = v[k1];
    F[fidx<T>(g, i, j, ks * N + k1)] = (T)s;
  }
}

// Statistics of physical fields straight from their (kx, y) rows: a warp transforms a
// row of one list entry back in its own two buffers in shared memory (the next row's
// copy is in flight meanwhile) and adds the values up in registers; no physical
// field is written.  Entries: a field (KE sum over levels k >= 1, and maxcalc's extrema,
// CFL maximum (x, y: |f| dt/dx; z: |w| dt/dz with the reference's merged-interface
// spacing, dzinv; extrema start from 0, or 1 for rho, whose background 1 + rhograd z is
// added) and, for w, the sum of squares and count below zlim, various.f:665-987), or a derivative (sum of squares over k >= 1).  grid.y: the entry; a
// fixed grid and order, so repeated calls give the same bits.
// part[(entry gridDim.x + block) 6 + {sum, min, max, cfl, sum w^2, count}].
// 256^2 x (8 x 25) mixed, iw_diag: 4.8 ms with a transform, a derivative and a reduction
// kernel per field and derivative (16 transforms written and read back).
constexpr int kStatThreads = 128, kStatSlots = 6, kStatMax = 13;
template <typename T>
struct StatRows {
  const T* src[kStatMax];
  int q[kStatMax];   // field 0..3 whose statistics are wanted, -1: a derivative
  int kx[kStatMax];  // multiply by i kx first
  double cflh[2], rg, zlim;
  const double* dzinv;
};
template <typename T, int DPT, bool POW2, int MC = 0>
__global__ void __launch_bounds__(kStatThreads) k_xrow_stats(Geo g, const __grid_constant__ StatRows<T> a, FftPlan pl,
                                                            const typename cplx_t<T>::type* __restrict__ Wm,
                                                            const typename cplx_t<T>::type* __restrict__ Wn,
                                                            double* __restrict__ part) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double sh[kStatThreads / 32][kStatSlots];
  const int M = MC > 0 ? MC : g.nx / 2, RS = xstride(M);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = kStatThreads / 32;
  const int ent = blockIdx.y, q = a.q[ent], lines = g.ny * g.nz, step = gridDim.x * nw;
  const bool mulkx = a.kx[ent] != 0;
  const T kxs = (T)g.xw[1];
  C* buf = (C*)smraw + (size_t)wid * 2 * RS;
  const C* src = (const C*)a.src[ent];
  auto fetch = [&](int line, C* d) {
    if (line < lines)
      for (int kk = lane; kk <= M; kk += 32) cp_async_c<C>(d + fpad(kk), src + (size_t)line * (M + 1) + kk);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double sum = 0.0, mn = q == 3 ? 1.0 : 0.0, mx = 0.0, cf = 0.0, s2 = 0.0, cnt = 0.0;
  int line = blockIdx.x * nw + wid;
  fetch(line, buf);
  for (int p = 0; line < lines; line += step, p ^= 1) {
    C* row = buf + p * RS;
    fetch(line + step, buf + (p ^ 1) * RS);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncwarp();
    for (int kk = lane; kk <= M / 2; kk += 32) xprep_pair<C, T>(row, kk, M, Wn, mulkx, kxs);
    __syncwarp();
    if constexpr (MC > 0)
      fft_warp_ct<C, MC>(row, RS, 1, Wm, true, lane);
    else
      fft_warp<C, DPT, POW2>(row, RS, 1, pl, Wm, true, lane);
    const int k = line / g.ny;
    const double dzi = q == 2 ? a.dzinv[k] : 0.0, bg = q == 3 ? 1.0 + a.rg * g.zg[k] : 0.0;
    const bool low = q == 2 && g.zg[k] < a.zlim;
    double ls = 0.0;
    for (int i = lane; i < M; i += 32) {
      const C v = row[fpad(i)];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double x = (double)(h ? v.y : v.x);
        ls += x * x;
        if (q >= 0) {
          if (q < 2) cf = fmax(cf, fabs(x) * a.cflh[q]);
          if (q == 2) cf = fmax(cf, fabs(x) * g.dt * dzi);
          if (q == 3) x += bg;
          mn = fmin(mn, x);
          mx = fmax(mx, x);
        }
      }
    }
    if (low) s2 += ls;
    if (k >= 1) sum += ls;
    if (low && lane == 0) cnt += (double)g.nx;
    __syncwarp();
  }
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    cf = fmax(cf, __shfl_xor_sync(0xffffffffu, cf, o));
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) {
    const double v[kStatSlots] = {sum, mn, mx, cf, s2, cnt};
    for (int e = 0; e < kStatSlots; ++e) sh[wid][e] = v[e];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nw; ++w) {
      sum += sh[w][0];
      mn = fmin(mn, sh[w][1]);
      mx = fmax(mx, sh[w][2]);
      cf = fmax(cf, sh[w][3]);
      s2 += sh[w][4];
      cnt += sh[w][5];
    }
    double* o = part + ((size_t)ent * gridDim.x + blockIdx.x) * kStatSlots;
    o[0] = sum;
    o[1] = mn;
    o[2] = mx;
    o[3] = cf;
    o[4] = s2;
    o[5] = cnt;
  }
}

template <typename T>
__global__ void k_nonfinite(const T* __restrict__ a0, const T* __restrict__ a1, const T* __restrict__ a2,
                            const T* __restrict__ a3, size_t n, int* flag) {
  const T* a = blockIdx.y == 0 ? a0 : blockIdx.y == 1 ? a1 : blockIdx.y == 2 ? a2 : a3;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    if (!isfinite((double)a[t])) {
      atomicExch(flag, 1);
      return;
    }
}

template <typename T, typename U>
__global__ void k_convert(const T* __restrict__ a, U* __restrict__ b, size_t n) {
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    b[t] = (U)a[t];
}

#include "iw_host.inl"
