// dft_pair.cuh -- register DFT codelets over two transforms at once.
//
// A c2 holds one complex element of each of two independent transforms, real
// parts together and imaginary parts together, so every operation of the DFT
// is the same on both and runs as one packed FP32 instruction (sm_100's
// add/sub/mul/fma.f32x2; each half rounds as the scalar instruction does).
// Against one transform per thread that halves the instructions issued per
// element, arithmetic and shared-memory accesses (16 bytes instead of 8)
// alike; the passes that use it are issue- and latency-bound.
//
// pdft<N, DIR>(v): as dft<N, DIR> (dft_codelets.cuh), on c2.
#pragma once
#include "dft_codelets.cuh"

namespace clarity {

struct c2 {
  float2 re, im;
};

__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }

__device__ __forceinline__ c2 padd(c2 a, c2 b) { return c2{padd(a.re, b.re), padd(a.im, b.im)}; }
__device__ __forceinline__ c2 psub(c2 a, c2 b) { return c2{psub(a.re, b.re), psub(a.im, b.im)}; }
// a + DIR*i*b
template <int DIR>
__device__ __forceinline__ c2 padd_diri(c2 a, c2 b) {
  if constexpr (DIR < 0)
    return c2{padd(a.re, b.im), psub(a.im, b.re)};
  else
    return c2{psub(a.re, b.im), padd(a.im, b.re)};
}
__device__ __forceinline__ float2 pneg(float2 a) { return pmul(a, both(-1.f)); }
// a * w, a * conj(w) with one w for both transforms, w as (re, re, im, im): a
// table stored so needs no moves to form the pairs
__device__ __forceinline__ c2 pcmul(c2 a, float4 w) {
  const float2 c = make_float2(w.x, w.y), s = make_float2(w.z, w.w);
  return c2{pfma(pneg(a.im), s, pmul(a.re, c)), pfma(a.re, s, pmul(a.im, c))};
}
__device__ __forceinline__ c2 pcmulc(c2 a, float4 w) {
  const float2 c = make_float2(w.x, w.y), s = make_float2(w.z, w.w);
  return c2{pfma(a.im, s, pmul(a.re, c)), pfma(pneg(a.re), s, pmul(a.im, c))};
}
__device__ __forceinline__ float4 twin(float2 w) { return make_float4(w.x, w.x, w.y, w.y); }
__device__ __forceinline__ c2 pcmul(c2 a, float2 w) { return pcmul(a, twin(w)); }
__device__ __forceinline__ c2 pcmulc(c2 a, float2 w) { return pcmulc(a, twin(w)); }

// v * exp(DIR * 2 pi i K / N), K and N compile time.
template <int K, int N, int DIR>
__device__ __forceinline__ c2 ptwc(c2 v) {
  constexpr int k = ((K % N) + N) % N;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (2 * k == N) {
    return c2{pmul(v.re, both(-1.f)), pmul(v.im, both(-1.f))};
  } else if constexpr (4 * k == N || 4 * k == 3 * N) {
    constexpr bool plus = (4 * k == N) == (DIR > 0);  // times +i or -i
    if constexpr (plus) return c2{pmul(v.im, both(-1.f)), v.re};
    else return c2{v.im, pmul(v.re, both(-1.f))};
  } else {
    constexpr cs_pair r = root_cs(k, N);
    constexpr float c = (float)r.c;
    constexpr float s = (float)(r.s * DIR);
    return c2{pfma(v.im, both(-s), pmul(v.re, both(c))), pfma(v.re, both(s), pmul(v.im, both(c)))};
  }
}

template <int N, int DIR>
struct PDFT;

template <int DIR>
struct PDFT<1, DIR> {
  __device__ __forceinline__ static void run(c2*) {}
};
template <int DIR>
struct PDFT<2, DIR> {
  __device__ __forceinline__ static void run(c2* v) {
    const c2 a = v[0], b = v[1];
    v[0] = padd(a, b);
    v[1] = psub(a, b);
  }
};
template <int DIR>
struct PDFT<3, DIR> {
  __device__ __forceinline__ static void run(c2* v) {
    constexpr float sn = (float)(DIR * 0.86602540378443864676);
    const c2 a0 = v[0], s = padd(v[1], v[2]), d = psub(v[1], v[2]);
    const c2 t{pfma(s.re, both(-0.5f), a0.re), pfma(s.im, both(-0.5f), a0.im)};
    v[0] = padd(a0, s);
    v[1] = c2{pfma(d.im, both(-sn), t.re), pfma(d.re, both(sn), t.im)};
    v[2] = c2{pfma(d.im, both(sn), t.re), pfma(d.re, both(-sn), t.im)};
  }
};
template <int DIR>
struct PDFT<4, DIR> {
  __device__ __forceinline__ static void run(c2* v) {
    const c2 s02 = padd(v[0], v[2]), d02 = psub(v[0], v[2]);
    const c2 s13 = padd(v[1], v[3]), d13 = psub(v[1], v[3]);
    v[0] = padd(s02, s13);
    v[1] = padd_diri<DIR>(d02, d13);
    v[2] = psub(s02, s13);
    v[3] = padd_diri<-DIR>(d02, d13);
  }
};

// Odd prime N >= 5: the symmetric direct form of DFTPrime.
template <int N, int DIR>
struct PDFTPrime {
  __device__ __forceinline__ static void run(c2* v) {
    constexpr int H = (N - 1) / 2;
    c2 a[H + 1], b[H + 1];
    const c2 x0 = v[0];
    c2 X0 = x0;
    static_for<H>([&](auto ti) {
      constexpr int t = decltype(ti)::value + 1;
      a[t] = padd(v[t], v[N - t]);
      b[t] = psub(v[t], v[N - t]);
      X0 = padd(X0, a[t]);
    });
    v[0] = X0;
    static_for<H>([&](auto ki) {
      constexpr int k = decltype(ki)::value + 1;
      c2 C = x0, S;
      static_for<H>([&](auto ti) {
        constexpr int t = decltype(ti)::value + 1;
        constexpr cs_pair r = root_cs((long)t * k, N);
        constexpr float c = (float)r.c;
        constexpr float s = (float)r.s;
        C = c2{pfma(a[t].re, both(c), C.re), pfma(a[t].im, both(c), C.im)};
        if constexpr (t == 1)
          S = c2{pmul(b[t].re, both(s)), pmul(b[t].im, both(s))};
        else
          S = c2{pfma(b[t].re, both(s), S.re), pfma(b[t].im, both(s), S.im)};
      });
      v[k] = padd_diri<DIR>(C, S);
      v[N - k] = padd_diri<-DIR>(C, S);
    });
  }
};

// Composite N = A * B: A-point DFTs with stride B, twiddles, B-point DFTs.
template <int N, int DIR>
struct PDFTSplit {
  static constexpr int A = first_split(N);
  static constexpr int B = N / A;
  __device__ __forceinline__ static void run(c2* v) {
    c2 u[N];
    static_for<B>([&](auto ii) {
      constexpr int i = decltype(ii)::value;
      c2 t[A];
      static_for<A>([&](auto ai) {
        constexpr int a = decltype(ai)::value;
        t[a] = v[i + B * a];
      });
      PDFT<A, DIR>::run(t);
      static_for<A>([&](auto ki) {
        constexpr int k = decltype(ki)::value;
        u[i + B * k] = ptwc<i * k, N, DIR>(t[k]);
      });
    });
    static_for<A>([&](auto ki) {
      constexpr int k = decltype(ki)::value;
      c2 s[B];
      static_for<B>([&](auto ii) {
        constexpr int i = decltype(ii)::value;
        s[i] = u[B * k + i];
      });
      PDFT<B, DIR>::run(s);
      static_for<B>([&](auto ji) {
        constexpr int j = decltype(ji)::value;
        v[k + A * j] = s[j];
      });
    });
  }
};

template <int N, int DIR>
struct PDFT {
  __device__ __forceinline__ static void run(c2* v) {
    if constexpr (is_prime(N)) PDFTPrime<N, DIR>::run(v);
    else PDFTSplit<N, DIR>::run(v);
  }
};

#ifdef CLARITY_HOST_EMULATION
// out of line: the sanitised host build of one codelet serves every pass
template <int N, int DIR>
__attribute__((noinline)) void pdft(c2* v) {
  PDFT<N, DIR>::run(v);
}
#else
template <int N, int DIR>
__device__ __forceinline__ void pdft(c2* v) {
  PDFT<N, DIR>::run(v);
}
#endif

}  // namespace clarity
