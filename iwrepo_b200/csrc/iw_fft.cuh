// Shared-memory FFT building blocks for sm_100a.
//
// Complex FFTs of length M (M = 2^a 3^b 5^c) are done as Stockham autosort
// passes (radix 8, 6, 5, 4, 3, 2, in-register DFTs) on data held in shared memory; a thread block
// works on a batch of independent transforms at once, one butterfly per
// thread per pass.  Real transforms of length N = 2M use the half-length
// complex transform plus the usual even/odd split.  Twiddles come from tables
// built on the host in long double.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace iw {

template <typename T>
struct cplx_t;
template <>
struct cplx_t<double> {
  typedef double2 type;
};
template <>
struct cplx_t<float> {
  typedef float2 type;
};

template <typename C>
__device__ __forceinline__ C cmk(decltype(C().x) a, decltype(C().x) b) {
  C c;
  c.x = a;
  c.y = b;
  return c;
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) {
  return cmk<C>(a.x + b.x, a.y + b.y);
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b) {
  return cmk<C>(a.x - b.x, a.y - b.y);
}
// two FP32 additions in one instruction (each rounded as ever)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  float2 d;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
// a b + c, written out so that a product's rounding does not depend on what the compiler does around it
__device__ __forceinline__ float cfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double cfma(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  return cmk<C>(cfma(a.x, b.x, -(a.y * b.y)), cfma(a.x, b.y, a.y * b.x));
}
template <typename C>
__device__ __forceinline__ C cconj(C a) {
  return cmk<C>(a.x, -a.y);
}
// multiply by -i (forward) or +i (inverse)
template <typename C>
__device__ __forceinline__ C cmul_mi(C a, bool inv) {
  return inv ? cmk<C>(-a.y, a.x) : cmk<C>(a.y, -a.x);
}

// Asynchronous global -> shared copy of one complex value (8 or 16 bytes,
// naturally aligned), so that a CTA can put all of its loads in flight before
// waiting once.
template <typename C>
__device__ __forceinline__ void cp_async_c(C* smem, const C* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if (sizeof(C) == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Plan of one complex length; radices in pass order.
struct FftPlan {
  int M;
  int npass;
  int rad[12];
  int ns[12];       // accumulated size before the pass
  int nbsh[12];     // log2(M/R) if a power of two, else -1
  int nssh[12];     // log2(ns) if a power of two, else -1
  float inb[12];    // 1 / (M/R), 1 / ns: (int)((q + 0.5f) * inv) is q / n for the small q here
  float ins[12];
};

// v * w with w = c - i s (forward) or c + i s (inverse)
template <typename C>
__device__ __forceinline__ C crot(C v, decltype(C().x) c, decltype(C().x) s, bool inv) {
  const decltype(C().x) t = inv ? s : -s;
  return cmk<C>(cfma(v.x, c, -(v.y * t)), cfma(v.x, t, v.y * c));
}

// In-register DFT of v[0..R-1] (natural order in and out) for R = 2, 3, 4, 5, 6, 8,
// 10, 16.
// R = 8 is split 2x4 (n = a + 2b, k = c + 4d); h = cos(pi/4).
template <typename C>
__device__ __forceinline__ void dft4(C& a0, C& a1, C& a2, C& a3, bool inv) {
  C t0 = cadd(a0, a2), t1 = csub(a0, a2);
  C t2 = cadd(a1, a3), t3 = cmul_mi(csub(a1, a3), inv);
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cadd(t1, t3);
  a3 = csub(t1, t3);
}

// R = 3: o1, o2 = v0 - t/2 -+ i (sqrt(3)/2) (v1 - v2), t = v1 + v2
template <typename C>
__device__ __forceinline__ void dft3(C& a0, C& a1, C& a2, bool inv) {
  typedef decltype(C().x) T;
  const T h = (T)0.86602540378443864676;  // sin(2 pi / 3)
  const C t = cadd(a1, a2), d = csub(a1, a2);
  const C m = cmk<C>(a0.x - (T)0.5 * t.x, a0.y - (T)0.5 * t.y);
  const C s = cmul_mi(cmk<C>(h * d.x, h * d.y), inv);
  a0 = cadd(a0, t);
  a1 = cadd(m, s);
  a2 = csub(m, s);
}
template <typename C>
__device__ __forceinline__ void dft5(C& a0, C& a1, C& a2, C& a3, C& a4, bool inv) {
  typedef decltype(C().x) T;
  // cosines and sines of 2 pi / 5 and 4 pi / 5
  const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
  const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
  const C t1 = cadd(a1, a4), t2 = cadd(a2, a3), d1 = csub(a1, a4), d2 = csub(a2, a3);
  const C m1 = cmk<C>(a0.x + c1 * t1.x + c2 * t2.x, a0.y + c1 * t1.y + c2 * t2.y);
  const C m2 = cmk<C>(a0.x + c2 * t1.x + c1 * t2.x, a0.y + c2 * t1.y + c1 * t2.y);
  const C n1 = cmul_mi(cmk<C>(cfma(s1, d1.x, s2 * d2.x), cfma(s1, d1.y, s2 * d2.y)), inv);
  const C n2 = cmul_mi(cmk<C>(cfma(s2, d1.x, -(s1 * d2.x)), cfma(s2, d1.y, -(s1 * d2.y))), inv);
  a0 = cadd(a0, cadd(t1, t2));
  a1 = cadd(m1, n1);
  a4 = csub(m1, n1);
  a2 = cadd(m2, n2);
  a3 = csub(m2, n2);
}
template <typename C, int R>
__device__ __forceinline__ void dft_reg(C* v, bool inv) {
  typedef decltype(C().x) T;
  const T h = (T)0.70710678118654752440;   // cos(pi/4)
  if (R == 2) {
    C t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  } else if (R == 3) {
    dft3(v[0], v[1], v[2], inv);
  } else if (R == 4) {
    dft4(v[0], v[1], v[2], v[3], inv);
  } else if (R == 5) {
    dft5(v[0], v[1], v[2], v[3], v[4], inv);
  } else if (R == 6) {
    // even and odd halves of three, joined with the sixth roots 1, (1 -+ i sqrt(3))/2, (-1 -+ i sqrt(3))/2
    const T g = (T)0.86602540378443864676;
    dft3(v[0], v[2], v[4], inv);
    dft3(v[1], v[3], v[5], inv);
    const C o1 = crot(v[3], (T)0.5, g, inv), o2 = crot(v[5], (T)-0.5, g, inv);
    const C e0 = v[0], e1 = v[2], e2 = v[4], o0 = v[1];
    v[0] = cadd(e0, o0);
    v[1] = cadd(e1, o1);
    v[2] = cadd(e2, o2);
    v[3] = csub(e0, o0);
    v[4] = csub(e1, o1);
    v[5] = csub(e2, o2);
  } else if (R == 8) {
    // a in {0,1}: DFT4 over v[a + 2b]
    dft4(v[0], v[2], v[4], v[6], inv);
    dft4(v[1], v[3], v[5], v[7], inv);
    // twiddle w8^c on the a = 1 half (c = 1..3 sit at v[3], v[5], v[7])
    v[3] = crot(v[3], h, h, inv);
    v[5] = cmul_mi(v[5], inv);
    v[7] = crot(v[7], -h, h, inv);
    C o[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      o[c] = cadd(v[2 * c], v[2 * c + 1]);
      o[c + 4] = csub(v[2 * c], v[2 * c + 1]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = o[i];
  } else if (R == 10) {
    // even and odd halves of five, joined with the tenth roots
    const T c1 = (T)0.80901699437494742410, s1 = (T)0.58778525229247312917;
    const T c2 = (T)0.30901699437494742410, s2 = (T)0.95105651629515357212;
    dft5(v[0], v[2], v[4], v[6], v[8], inv);
    dft5(v[1], v[3], v[5], v[7], v[9], inv);
    C o[5] = {v[1], crot(v[3], c1, s1, inv), crot(v[5], c2, s2, inv), crot(v[7], -c2, s2, inv),
              crot(v[9], -c1, s1, inv)};
    C e[5] = {v[0], v[2], v[4], v[6], v[8]};
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      v[c] = cadd(e[c], o[c]);
      v[c + 5] = csub(e[c], o[c]);
    }
  } else if (R == 16) {
    // a in 0..3: DFT4 over v[a + 4 b], twiddles w16^(a c), DFT4 over a
    const T c1 = (T)0.92387953251128675613, s1 = (T)0.38268343236508977173;  // pi / 8
#pragma unroll
    for (int a = 0; a < 4; ++a) dft4(v[a], v[a + 4], v[a + 8], v[a + 12], inv);
    v[5] = crot(v[5], c1, s1, inv);
    v[6] = crot(v[6], h, h, inv);
    v[7] = crot(v[7], s1, c1, inv);
    v[9] = crot(v[9], h, h, inv);
    v[10] = cmul_mi(v[10], inv);
    v[11] = crot(v[11], -h, h, inv);
    v[13] = crot(v[13], s1, c1, inv);
    v[14] = crot(v[14], -h, h, inv);
    v[15] = crot(v[15], -c1, -s1, inv);
    C o[16];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      dft4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3], inv);
#pragma unroll
      for (int d = 0; d < 4; ++d) o[c + 4 * d] = v[4 * c + d];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = o[i];
  }
}

// One Stockham pass of radix R over `nbatch` transforms stored contiguously
// (stride M) in src, written to dst.  W[e] = exp(-2 pi i e / M).
template <typename C, int R>
__device__ __forceinline__ void fft_pass_r(const C* __restrict__ src, C* __restrict__ dst, int M, int Ns, int nbatch,
                                           const C* __restrict__ W, bool inv, int tid, int nthr, int nbsh, int nssh) {
  const int nb = M / R;
  const int total = nb * nbatch;
  const int step = M / (Ns * R);
  for (int w = tid; w < total; w += nthr) {
    const int b = nbsh >= 0 ? (w >> nbsh) : (w / nb);
    const int j = w - b * nb;
    const C* s = src + (size_t)b * M;
    C* d = dst + (size_t)b * M;
    C v[R];
    const int jq = nssh >= 0 ? (j >> nssh) : (j / Ns);
    const int jm = j - jq * Ns;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = s[j + r * nb];
    if (Ns > 1) {
      const int e = jm * step;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        C tw = W[r * e];  // r*jm*step < R*Ns*step = M
        if (inv) tw.y = -tw.y;
        v[r] = cmul(v[r], tw);
      }
    }
    dft_reg<C, R>(v, inv);
    const int base = jq * Ns * R + jm;
#pragma unroll
    for (int r = 0; r < R; ++r) d[base + r * Ns] = v[r];
  }
}

// Full transform; returns the buffer (a or b) that holds the result.
// Caller must __syncthreads() before (inputs ready); this ends synced.
template <typename C>
__device__ C* fft_run(C* a, C* b, const FftPlan& pl, int nbatch, const C* W, bool inv, int tid, int nthr) {
  C* src = a;
  C* dst = b;
  for (int p = 0; p < pl.npass; ++p) {
    const int R = pl.rad[p], Ns = pl.ns[p], bs = pl.nbsh[p], ss = pl.nssh[p];
    switch (R) {
      case 8: fft_pass_r<C, 8>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
      case 4: fft_pass_r<C, 4>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
      case 2: fft_pass_r<C, 2>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
      case 3: fft_pass_r<C, 3>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
      case 6: fft_pass_r<C, 6>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
      default: fft_pass_r<C, 5>(src, dst, pl.M, Ns, nbatch, W, inv, tid, nthr, bs, ss); break;
    }
    __syncthreads();
    C* t = src;
    src = dst;
    dst = t;
  }
  return src;
}


// ---------------------------------------------------------------------------
// Warp-synchronous in-place transforms.  One warp owns a transform of length M, or
// several short ones at once, held in shared memory with one pad slot after every 16 values (index
// fpad(i)), which keeps the strided Stockham stores free of bank conflicts.
// Every pass loads all of its butterflies into registers, then stores them:
// no second buffer and no CTA-wide barrier.  DPT >= M/32 values per lane.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }
// Place of value i under layout L: 0 is fpad; 2 pads by two, so that values 64 apart lie half the
// banks apart; 1 also exchanges neighbours in the second half of each 16, so that two values 8 apart
// differ in parity (with an even column stride: neither those nor adjacent rows of 8 columns collide).
template <int L>
__host__ __device__ __forceinline__ int flay(int i) {
  return L == 0 ? fpad(i) : (L == 1 ? i ^ ((i >> 3) & 1) : i) + 2 * (i >> 4);
}
// slots needed for L padded values
__host__ __device__ __forceinline__ int fpadlen(int L) { return L > 0 ? fpad(L - 1) + 1 : 0; }

// One pass over G rows, RS values apart: as many whole rows at a time as the warp's lanes hold
// (M / R <= 32), or one row at a time in IT butterflies per lane (M / R <= 32 IT).  A lane keeps its
// butterflies' indexes and twiddles over the rows; of a single row (ONE, G = 1) the twiddles are read where
// they are used, which leaves their registers to the values.
template <typename C, int R, int IT, int L, bool ONE>
__device__ __forceinline__ void fft_pass_w(C* base, int RS, int G, int M, int Ns, float inb, float ins, int nssh,
                                           const C* __restrict__ W, bool inv, int lane) {
  const int nb = M / R, step = M / (Ns * R);
  const int rpi = !ONE && nb < 32 ? (int)(32.5f * inb) : 1;  // rows at a time
  const int g = !ONE && nb < 32 ? (int)(((float)lane + 0.5f) * inb) : 0, j0 = lane - g * nb;
  const bool act = ONE ? j0 < nb : g < rpi;
  // (values of idle lanes are set, or the compiler carries the registers of every radix through the
  // loop over the passes)
  C tw[ONE ? 1 : IT][R];
  int jq[IT], jm[IT];
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    const int j = j0 + 32 * q;
    jq[q] = nssh >= 0 ? j >> nssh : (int)(((float)j + 0.5f) * ins);
    jm[q] = j - jq[q] * Ns;
    if (ONE) continue;
#pragma unroll
    for (int r = 0; r < R; ++r) tw[q][r] = cmk<C>(1, 0);
    if (Ns > 1 && (q == 0 || j < nb)) {
      const int e = jm[q] * step;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        tw[q][r] = W[r * e];
        if (inv) tw[q][r].y = -tw[q][r].y;
      }
    }
  }
#pragma unroll 1
  for (int r0 = 0; r0 < (ONE ? 1 : G); r0 += rpi) {
    C* row = base + (r0 + g) * RS;
    const bool on = act && (ONE || r0 + g < G);
    C v[IT][R];
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (!ONE) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[q][r] = cmk<C>(0, 0);
      }
      if (on && (q == 0 || j0 + 32 * q < nb)) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[q][r] = row[flay<L>(j0 + 32 * q + r * nb)];
        if (Ns > 1) {
#pragma unroll
          for (int r = 1; r < R; ++r) {
            if (ONE) {
              tw[0][r] = W[r * jm[q] * step];
              if (inv) tw[0][r].y = -tw[0][r].y;
            }
            v[q][r] = cmul(v[q][r], tw[ONE ? 0 : q][r]);
          }
        }
        dft_reg<C, R>(v[q], inv);
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < IT; ++q)
      if (on && (q == 0 || j0 + 32 * q < nb)) {
        const int b0 = jq[q] * Ns * R + jm[q];
#pragma unroll
        for (int r = 0; r < R; ++r) row[flay<L>(b0 + r * Ns)] = v[q][r];
      }
  }
  __syncwarp();
}

// rows of length M that one warp transforms at a time with DPT values per lane
__host__ __device__ constexpr int fft_rows_of(int M, int DPT) { return 32 * DPT / M > 1 ? 32 * DPT / M : 1; }

// In-place transform of G padded rows of M <= 32 DPT values by one warp (all lanes call
// it).  POW2: the length is a power of two, so only radix 8, 4, 2 passes are
// compiled (every compiled radix raises the register count of the kernel).  ONE: G is 1.
template <typename C, int DPT, bool POW2, int L = 0, bool ONE = false>
__device__ __forceinline__ void fft_warp(C* base, int RS, int G, const FftPlan& pl, const C* __restrict__ W, bool inv,
                                         int lane) {
  for (int p = 0; p < pl.npass; ++p) {
    const int Ns = pl.ns[p];
    const float ib = pl.inb[p], is = pl.ins[p];
    const int ss = ONE && POW2 ? pl.nssh[p] : -1;  // (a shift costs fewer instructions than two conversions)
    switch (pl.rad[p]) {
      case 8: fft_pass_w<C, 8, (DPT + 7) / 8, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane); break;
      case 4: fft_pass_w<C, 4, (DPT + 3) / 4, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane); break;
      case 2: fft_pass_w<C, 2, (DPT + 1) / 2, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane); break;
      default:
        if (!POW2) {
          if (pl.rad[p] == 3)
            fft_pass_w<C, 3, (DPT + 2) / 3, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane);
          else if (pl.rad[p] == 6)
            fft_pass_w<C, 6, (DPT + 5) / 6, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane);
          else
            fft_pass_w<C, 5, (DPT + 4) / 5, L, ONE>(base, RS, G, pl.M, Ns, ib, is, ss, W, inv, lane);
        }
        break;
    }
  }
}

// minimum resident CTAs of 256 threads for a warp-transform kernel (the mixed-radix
// kernels hold every radix and get more registers)
template <typename T, int DPT, bool POW2 = true>
struct FftOcc {
  static constexpr int v = sizeof(T) == 4 ? (DPT <= 8 ? (POW2 ? 4 : 3) : DPT <= 16 ? 2 : 1) : DPT <= 8 ? 2 : 1;
};


// ---------------------------------------------------------------------------
// Compile-time plans for power-of-two lengths M (same passes as make_plan:
// ceil(log2 M / 3) passes of radix <= 8, bits spread evenly).  Strides,
// twiddle steps and lane guards become constants.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ct_log2(int v) { return v <= 1 ? 0 : 1 + ct_log2(v / 2); }
template <int M>
struct CtPlan {
  static constexpr int a = ct_log2(M);
  static constexpr int np = (a + 2) / 3;
  __host__ __device__ static constexpr int bits(int q) { return a / np + (q < a % np ? 1 : 0); }
};

// values per lane of the compile-time transforms: short rows share the warp
template <int M>
struct CtRows {
  static constexpr int DPT = M <= 256 ? 8 : M / 32;
  static constexpr int G = fft_rows_of(M, DPT);
};
template <typename C, int M, int R, int NS, int L>
__device__ __forceinline__ void fft_pass_ct(C* base, int RS, int G, const C* __restrict__ W, bool inv, int lane) {
  constexpr int nb = M / R;
  constexpr int step = M / (NS * R);
  constexpr int NB = (CtRows<M>::G * nb + 31) / 32;
  const int items = CtRows<M>::G > 1 ? G * nb : nb;
  C v[NB][R];
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const int it = lane + 32 * q;
#pragma unroll
    for (int r = 0; r < R; ++r) v[q][r] = cmk<C>(0, 0);
    if ((CtRows<M>::G == 1 && nb % 32 == 0) || it < items) {
      const int g = CtRows<M>::G > 1 ? it / nb : 0, j = CtRows<M>::G > 1 ? it % nb : it;
      const C* row = base + g * RS;
      const int jm = j & (NS - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) v[q][r] = row[flay<L>(j + r * nb)];
      if (NS > 1) {
        const int e = jm * step;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          C tw = W[r * e];
          if (inv) tw.y = -tw.y;
          v[q][r] = cmul(v[q][r], tw);
        }
      }
      dft_reg<C, R>(v[q], inv);
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const int it = lane + 32 * q;
    if ((CtRows<M>::G == 1 && nb % 32 == 0) || it < items) {
      const int g = CtRows<M>::G > 1 ? it / nb : 0, j = CtRows<M>::G > 1 ? it % nb : it;
      C* row = base + g * RS;
      const int jq = j / NS, jm = j & (NS - 1);
      const int b0 = jq * NS * R + jm;
#pragma unroll
      for (int r = 0; r < R; ++r) row[flay<L>(b0 + r * NS)] = v[q][r];
    }
  }
  __syncwarp();
}

// Passes P .. PEND-1 (the first or last pass may run elsewhere) of G <= CtRows<M>::G rows.
template <typename C, int M, int P, int PEND, int NS, int L = 0>
__device__ __forceinline__ void fft_passes_ct(C* base, int RS, int G, const C* __restrict__ W, bool inv, int lane) {
  if constexpr (P < PEND) {
    constexpr int R = 1 << CtPlan<M>::bits(P);
    fft_pass_ct<C, M, R, NS, L>(base, RS, G, W, inv, lane);
    fft_passes_ct<C, M, P + 1, PEND, NS * R, L>(base, RS, G, W, inv, lane);
  }
}

// In-place transform of G <= CtRows<M>::G padded rows of power-of-two length M by one warp.
template <typename C, int M, int L = 0>
__device__ __forceinline__ void fft_warp_ct(C* base, int RS, int G, const C* __restrict__ W, bool inv, int lane) {
  fft_passes_ct<C, M, 0, CtPlan<M>::np, 1, L>(base, RS, G, W, inv, lane);
}

}  // namespace iw
