// s2d_pairs.cuh -- the fused RK3 stage for dealiased states, two lines per thread.
//
// A state whose cells outside the 2/3 band are zero (every seeded or stepped state) needs
// only the rows |ky| < N/3 and, in them, the columns |kx| < N/3.  Both stage kernels work on
// PAIRS of lines held as packed FP32x2 values (one complex number of each line side by side),
// so every butterfly, twiddle product and shared-memory access serves two lines:
//
//   k_pair_rows  rows ky and -ky of one pair per group of T = N/V threads.  A thread owns the
//                four cells (+-kx, +-ky) of each of its columns: they share |k|^2, 1/|k|^2,
//                the integrating factor (conjugated for -kx), the forcing envelope, and two
//                of the four Hermitian unpacks and forcing phases.  Its state cells are
//                loaded before the x-transform of Z and wait in registers.
//   k_pair_cols  columns x and x+1.  v is real, so its x-transformed spectrum obeys
//                PB(-ky, x) = conj PB(ky, x): only the rows ky >= 0 are stored, and the two
//                columns' v come out of ONE complex y-transform of V(x) + i V(x+1).
//
// Transforms per stage and row pair: 2 forward and 3 inverse lines (2 and 4 with both rows of
// PB); per column pair 3 inverse and 2 forward lines (4 and 2).  PB holds the Hermitian part
// of v_hat, whose inverse transform is the real part the stage reads, so a state that is not
// exactly Hermitian steps as before.
//
// States with cells outside the band, set by a caller, take the kernels of s2d_kernels.cuh.
#pragma once
#include "s2d_kernels.cuh"

namespace s2d {

// ------------------------------------------------------------------ two complex numbers
struct C2 {
  float2 re, im;
};
__device__ __forceinline__ float2 splat2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, splat2(-1.f), a); }
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ C2 csub(C2 a, C2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
template <int SIGN> __device__ __forceinline__ C2 cmul_si(C2 a) {
  return SIGN > 0 ? C2{neg2(a.im), a.re} : C2{a.im, neg2(a.re)};
}
// a * (c + i s) for one complex factor
__device__ __forceinline__ C2 cmul_cs(C2 a, float2 c, float2 s) {
  return {__ffma2_rn(a.re, c, neg2(__fmul2_rn(a.im, s))), __ffma2_rn(a.re, s, __fmul2_rn(a.im, c))};
}
__device__ __forceinline__ C2 cmul_w(C2 a, float2 w) { return cmul_cs(a, splat2(w.x), splat2(w.y)); }
template <int SIGN, int R> __device__ __forceinline__ C2 twmul_c(C2 a, int e) {
  const int k = ((e % R) + R) % R * (64 / R);
  if (k == 0) return a;
  if (k == 16) return cmul_si<SIGN>(a);
  if (k == 32) return {neg2(a.re), neg2(a.im)};
  if (k == 48) return cmul_si<-SIGN>(a);
  const float c = (float)cos64(k), s = (float)(SIGN * sin64(k));
  return cmul_cs(a, splat2(c), splat2(s));
}

// In-register DFT over either element type (natural order in and out); the same four-step
// split as Dft.
template <int R, int SIGN, class E> struct DftE {
  static constexpr int P = (R % 4 == 0 && R / 4 >= 2) ? 4 : 2;
  static constexpr int Q = R / P;
  __device__ __forceinline__ static void run(E* v) {
    E y[Q][P];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
      E t[P];
#pragma unroll
      for (int n1 = 0; n1 < P; ++n1) t[n1] = v[Q * n1 + n2];
      DftE<P, SIGN, E>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) y[n2][k1] = twmul_c<SIGN, R>(t[k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      E t[Q];
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) t[n2] = y[n2][k1];
      DftE<Q, SIGN, E>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) v[k1 + P * k2] = t[k2];
    }
  }
};
template <int SIGN, class E> struct DftE<2, SIGN, E> {
  __device__ __forceinline__ static void run(E* v) {
    const E a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};
template <int SIGN, class E> struct DftE<4, SIGN, E> {
  __device__ __forceinline__ static void run(E* v) {
    const E s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const E s13 = cadd(v[1], v[3]), d13 = cmul_si<SIGN>(csub(v[1], v[3]));
    v[0] = cadd(s02, s13);
    v[1] = cadd(d02, d13);
    v[2] = csub(s02, s13);
    v[3] = csub(d02, d13);
  }
};

// ------------------------------------------------------------------ pass-ordered twiddles
// Entry [r-1][jm] of pass p (p >= 1) is W_N^{jm r N/(NS R)} = c - i s as (c, c, s, s): lanes
// of a warp read consecutive entries (the plain table's stride would touch a line per lane),
// and both components arrive as packed operands.
template <int N, int V> struct PassTw {
  using PL = LinePlan<N, V>;
  __host__ __device__ static constexpr int offset(int p) {
    int o = 0;
    for (int q = 1; q < p; ++q) o += (PL::radix(q) - 1) * PL::ns(q);
    return o;
  }
  static constexpr int SIZE = offset(PL::P);
};
template <int N, int V> __global__ void k_pass_twiddles(float4* out, const float2* __restrict__ tw) {
  using PL = LinePlan<N, V>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int o = 0;
  for (int p = 1; p < PL::P; ++p) {
    const int ns = PL::ns(p), r = PL::radix(p), len = (r - 1) * ns;
    if (i >= o && i < o + len) {
      const int q = (i - o) / ns + 1, jm = (i - o) % ns;
      const float2 w = tw[jm * q * (N / (ns * r))];   // (cos, -sin)
      out[i] = make_float4(w.x, w.x, -w.y, -w.y);
    }
    o += len;
  }
}

// ------------------------------------------------------------------ launch shapes
// V values per thread and line; GP column pairs per column CTA; BTHREADS threads per row CTA
// (a multiple of T = N/V: whole row pairs); resident CTAs the register budget must allow.
template <int N_, int V_, int GP_, int BTHREADS_, int AMINB_, int BMINB_> struct PairTune {
  static constexpr int N = N_, V = V_, T = N / V;
  using PL = LinePlan<N, V>;
  static constexpr int KMAX = N / 3;          // largest in-band wavenumber: |k| < N/3, N a power of two
  static constexpr int BAND = KMAX + 1;       // in-band k = 0..KMAX: row pairs, and columns of a thread quad
  __host__ __device__ static constexpr int pad(int i) { return i + i / V; }
  static constexpr int PADDED = N + T;
  // columns
  static constexpr int GP = GP_, A_THREADS = GP * T, A_GRID = N / 2 / GP, A_MINB = AMINB_;
  static constexpr size_t A_SMEM = (size_t)PADDED * GP * (sizeof(float4) + sizeof(float2));
  // rows
  static constexpr int B_THREADS = BTHREADS_, PPB = B_THREADS / T, B_MINB = BMINB_;
  static constexpr int B_GRID = (BAND + PPB - 1) / PPB;
  static constexpr size_t B_SMEM = (size_t)PADDED * PPB * (sizeof(float4) + sizeof(float2));
  static_assert(B_THREADS % T == 0 && (N / 2) % GP == 0, "whole lines");
};
template <int N> struct PairShapeOf;
template <> struct PairShapeOf<32> { using type = PairTune<32, 8, 8, 32, 16, 16>; };
template <> struct PairShapeOf<64> { using type = PairTune<64, 8, 4, 32, 16, 16>; };
template <> struct PairShapeOf<128> { using type = PairTune<128, 8, 2, 32, 16, 16>; };
template <> struct PairShapeOf<256> { using type = PairTune<256, 8, 2, 32, 8, 16>; };
template <> struct PairShapeOf<512> { using type = PairTune<512, 8, 2, 64, 4, 8>; };
template <> struct PairShapeOf<1024> { using type = PairTune<1024, 8, 2, 128, 2, 4>; };
template <> struct PairShapeOf<2048> { using type = PairTune<2048, 8, 2, 256, 1, 2>; };
template <> struct PairShapeOf<4096> { using type = PairTune<4096, 8, 1, 512, 1, 1>; };
template <int N> using PairShape = typename PairShapeOf<N>::type;
template <class TU> __device__ __forceinline__ bool pair_inband(int i) { return i <= TU::KMAX || i >= TU::N - TU::KMAX; }
// whether register slot m (indices T m .. T m + T - 1) holds no in-band index
template <class TU> __host__ __device__ constexpr bool slot_empty(int m) {
  return TU::T * m > TU::KMAX && TU::T * m + TU::T - 1 < TU::N - TU::KMAX;
}

// barrier over the T threads that share a line (they are T consecutive threads)
template <int T, int NTHREADS> struct GroupSync {
  __device__ __forceinline__ void operator()() const {
    if constexpr (T <= 32) __syncwarp();
    else if constexpr (T == NTHREADS) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / T), "n"(T) : "memory");
  }
};

// One packed pair of lines and, with HASV, one more single line, transformed in lockstep.
// Element i of the pair is at l4[pad(i) * ST], of the single line at l2[pad(i) * ST].
template <class TU, int SIGN, bool HASV, int ST, class Sync>
__device__ __forceinline__ void pair_fft(C2 (&x)[TU::V], float2 (&y)[TU::V], float4* l4, float2* l2, int t,
                                         const float4* __restrict__ tw, const Sync& sync) {
  using PL = typename TU::PL;
  constexpr int N = TU::N, V = TU::V, T = TU::T;
  sfor<PL::P>([&](auto pc) {
    constexpr int p = decltype(pc)::value;
    constexpr int R = PL::radix(p), B = V / R, NS = PL::ns(p);
    C2 v[V];
    float2 w[V];
    if constexpr (p == 0) {
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[b * R + r] = x[b + B * r];
          if constexpr (HASV) w[b * R + r] = y[b + B * r];
        }
    } else {
      float4 f[V];
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 1; r < R; ++r)
          f[b * R + r] = __ldg(tw + PassTw<N, V>::offset(p) + (r - 1) * NS + ((t + T * b) & (NS - 1)));
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = TU::pad(t + T * b + r * (N / R)) * ST;
          const float4 q = l4[i];
          v[b * R + r] = {make_float2(q.x, q.y), make_float2(q.z, q.w)};
          if constexpr (HASV) w[b * R + r] = l2[i];
        }
      sync();
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const float4 q = f[b * R + r];
          const float2 c = make_float2(q.x, q.y), s = make_float2(q.z, q.w);
          v[b * R + r] = cmul_cs(v[b * R + r], c, SIGN > 0 ? s : neg2(s));
          if constexpr (HASV) w[b * R + r] = cmul(w[b * R + r], make_float2(q.x, SIGN > 0 ? q.z : -q.z));
        }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      DftE<R, SIGN, C2>::run(&v[b * R]);
      if constexpr (HASV) DftE<R, SIGN, float2>::run(&w[b * R]);
    }
    if constexpr (p < PL::P - 1) {
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const int j = t + T * b;
        const int base = (j / NS) * NS * R + (j & (NS - 1));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = TU::pad(base + r * NS) * ST;
          const C2 q = v[b * R + r];
          l4[i] = make_float4(q.re.x, q.re.y, q.im.x, q.im.y);
          if constexpr (HASV) l2[i] = w[b * R + r];
        }
      }
      sync();
    } else {
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          x[b + B * r] = v[b * R + r];
          if constexpr (HASV) y[b + B * r] = w[b * R + r];
        }
    }
  });
}

// ------------------------------------------------------------------ columns
// MODE as phys_cols_tile.  One column pair per group; groups interleave over lanes (two
// pairs are one 32-byte sector per row).  Returns this thread's max |u|+|v| (MODE != 1).
template <int MODE, class TU>
__device__ __forceinline__ float pair_cols_tile(const PhysArgs& a, int tile, float4* smem) {
  constexpr int N = TU::N, V = TU::V, T = TU::T, GP = TU::GP;
  const int g = threadIdx.x % GP, t = threadIdx.x / GP;
  const int x0 = 2 * (tile * GP + g);
  float4* const l4 = smem + g;
  float2* const l2 = reinterpret_cast<float2*>(smem + TU::PADDED * GP) + g;
  struct Sync {
    __device__ __forceinline__ void operator()() const {
      if constexpr (TU::A_THREADS <= 32) __syncwarp();
      else __syncthreads();
    }
  };
  C2 x[V];
  float2 y[V];
#pragma unroll
  for (int m = 0; m < V; ++m) {
    x[m] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    y[m] = make_float2(0.f, 0.f);
    const int row = t + T * m;
    if (!slot_empty<TU>(m) && pair_inband<TU>(row)) {
      const float4 p = __ldcs(reinterpret_cast<const float4*>(a.pa + (size_t)row * N + x0));
      const bool up = row < N / 2;
      const float4 q = __ldg(reinterpret_cast<const float4*>(a.pb + (size_t)(up ? row : N - row) * N + x0));
      x[m] = {make_float2(p.x, p.z), make_float2(p.y, p.w)};
      // V(x) + i V(x+1), conjugated spectra for -ky; row 0 is real
      if (row == 0) y[m] = make_float2(q.x, q.z);
      else y[m] = up ? make_float2(q.x - q.w, q.y + q.z) : make_float2(q.x + q.w, q.z - q.y);
    }
  }
  pair_fft<TU, +1, true, GP>(x, y, l4, l2, t, a.ptw, Sync{});
  // re = omega, im = u at (x, x+1); y = v at (x, x+1)
  float speed = 0.f;
  if constexpr (MODE != 1) {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const float2 u = x[m].im, v = y[m];
      *reinterpret_cast<float4*>(a.vel + (size_t)(t + T * m) * N + x0) = make_float4(u.x, v.x, u.y, v.y);
      speed = fmaxf(speed, fmaxf(fabsf(u.x) + fabsf(v.x), fabsf(u.y) + fabsf(v.y)));
    }
  }
  if constexpr (MODE != 0) {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const float2 om = x[m].re;
      x[m] = {__fmul2_rn(x[m].im, om), __fmul2_rn(y[m], om)};
    }
    pair_fft<TU, -1, false, GP>(x, y, l4, l2, t, a.ptw, Sync{});
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int row = t + T * m;
      if (!slot_empty<TU>(m) && pair_inband<TU>(row))
        *reinterpret_cast<float4*>(a.z + (size_t)row * N + x0) =
            make_float4(x[m].re.x, x[m].im.x, x[m].re.y, x[m].im.y);
    }
  }
  return speed;
}

template <int MODE, class TU>
__global__ void __launch_bounds__(TU::A_THREADS, TU::A_MINB) k_pair_cols(PhysArgs a) {
  extern __shared__ __align__(16) float4 smem4[];
  phys_latch(a);
  const float speed = pair_cols_tile<MODE, TU>(a, blockIdx.x, smem4);
  if constexpr (MODE != 1) cols_speed_finalize<TU::A_THREADS>(a, speed);
}

// ------------------------------------------------------------------ rows
// the state cells of one quad: (row a, col c), (a, -c), (b, c), (b, -c)
struct Quad {
  float2 v[4];
};
__device__ __forceinline__ Quad load_quad(const float2* s, size_t ra, size_t rb, int c, int mc) {
  return {{s[ra + c], s[ra + mc], s[rb + c], s[rb + mc]}};
}
__device__ __forceinline__ C2 pair_of(float2 a, float2 b) { return {make_float2(a.x, b.x), make_float2(a.y, b.y)}; }
// w + e w, w + conj(e) w
__device__ __forceinline__ C2 grow(C2 w, float2 e) { return cadd(w, cmul_w(w, e)); }

// out of the stage update rk_update<S> for the two cells of a column, all factors finite
template <int S> __device__ __forceinline__ C2 rk_pair(float2 e, float2 full, float2 mhalf, C2 w0, C2 adv) {
  if constexpr (S == 0) {
    return grow(adv, full);
  } else if constexpr (S == 1) {
    const C2 p = grow(w0, e), q = grow(adv, mhalf);
    return {__ffma2_rn(p.re, splat2(0.75f), __fmul2_rn(q.re, splat2(0.25f))),
            __ffma2_rn(p.im, splat2(0.75f), __fmul2_rn(q.im, splat2(0.25f)))};
  } else {
    const C2 p = grow(w0, full), q = grow(adv, e);   // q + (p - q)/3, see rk_update
    const C2 d = csub(p, q);
    return {__ffma2_rn(d.re, splat2(1.f / 3.f), q.re), __ffma2_rn(d.im, splat2(1.f / 3.f), q.im)};
  }
}

// one group's row pair; MODE as spec_rows_tile
template <int MODE, bool PTR, class TU>
__device__ __forceinline__ void pair_rows_tile(const SpecArgs& a, int tile, float4* smem) {
  constexpr int N = TU::N, V = TU::V, T = TU::T, BAND = TU::BAND, KMAX = TU::KMAX;
  constexpr int Q = (BAND + T - 1) / T;
  const int t = threadIdx.x % T, g = threadIdx.x / T;
  const int p = min(tile * TU::PPB + g, KMAX);   // the last CTA's spare groups repeat pair KMAX
  const size_t ra = (size_t)p * N, rb = (size_t)((N - p) & (N - 1)) * N;
  float4* const l4 = smem + g * TU::PADDED;
  float2* const l2 = reinterpret_cast<float2*>(smem + TU::PPB * TU::PADDED) + g * TU::PADDED;
  const GroupSync<T, TU::B_THREADS> sync;
  C2 x[V];
  float2 y[V];
  // every global load of the stage goes out here: Z first, then the quads' state cells
  if constexpr (MODE >= 0) {
#pragma unroll
    for (int m = 0; m < V; ++m) x[m] = pair_of(__ldcs(a.z + ra + t + T * m), __ldcs(a.z + rb + t + T * m));
  }
  Quad wq[Q], w0q[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = t + T * q, mc = (N - c) & (N - 1);
    if (c < BAND) {
      wq[q] = load_quad(a.wcur, ra, rb, c, mc);
      if constexpr (MODE >= 1) w0q[q] = load_quad(a.w0, ra, rb, c, mc);
    }
  }
  const DevParams& P = *a.params;
  const float dt = MODE >= 0 ? __ldg(a.dt) : 0.f;
  if constexpr (MODE >= 0) {
    pair_fft<TU, -1, false, 1>(x, y, l4, l2, t, a.ptw, sync);
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      if (!slot_empty<TU>(m) && pair_inband<TU>(c))
        l4[TU::pad(c)] = make_float4(x[m].re.x, x[m].re.y, x[m].im.x, x[m].im.y);
    }
    sync();
  }
  const float ky = (float)p;
  constexpr float inv_n2 = 1.0f / ((float)N * (float)N);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = t + T * q, mc = (N - c) & (N - 1);
    if (c < BAND) {
      const float kx = (float)c;
      const float k2 = kx * kx + ky * ky;
      C2 w = pair_of(wq[q].v[0], wq[q].v[2]), wm = pair_of(wq[q].v[1], wq[q].v[3]);   // columns c, -c
      if constexpr (MODE >= 0) {
        const float4 zc = l4[TU::pad(c)], zm = l4[TU::pad(mc)];   // (re a, re b, im a, im b)
        // right-hand sides at k = (kx, ky) and (-kx, ky); the other two cells hold the conjugates
        auto minus_nhat = [&](float kxs, float2 zk, float2 zp) {   // zp = Z(-k)
          const float2 q1 = make_float2(0.5f * (zk.x + zp.x), 0.5f * (zk.y - zp.y));
          const float2 q2 = make_float2(0.5f * (zk.y + zp.y), -0.5f * (zk.x - zp.x));
          return make_float2(kxs * q1.y + ky * q2.y, -(kxs * q1.x) - ky * q2.x);
        };
        float2 r1 = minus_nhat(kx, make_float2(zc.x, zc.z), make_float2(zm.y, zm.w));
        float2 r2 = minus_nhat(-kx, make_float2(zm.x, zm.z), make_float2(zc.y, zc.w));
        if (a.stochastic && k2 > 0.f) {
          const float2 fb = forcing_k2_bounds(P);
          if (k2 >= fb.x && k2 <= fb.y) {
            // the term of -k is the conjugate of that of k
            const float2 f1 = stochastic_term(P, N, p, c, kx, ky, k2, dt);
            const float2 f2 = stochastic_term(P, N, p, mc, -kx, ky, k2, dt);
            r1 = cadd(r1, f1);
            r2 = cadd(r2, f2);
          }
        }
        C2 r = {make_float2(r1.x, r2.x), make_float2(r1.y, -r2.y)};
        C2 rm = {make_float2(r2.x, r1.x), make_float2(r2.y, -r1.y)};
        if constexpr (PTR) {
          const Quad f = load_quad(a.fptr, ra, rb, c, mc);
          r = cadd(r, pair_of(f.v[0], f.v[2]));
          rm = cadd(rm, pair_of(f.v[1], f.v[3]));
        }
        const float2 e = half_factor_m1(P, kx, fmaxf(k2, 1.f), dt);
        const float2 e1 = make_float2(1.f + e.x, e.y);
        const float nrm = e1.x * e1.x + e1.y * e1.y;
        C2 w0 = w, w0m = wm;
        if constexpr (MODE >= 1) {
          w0 = pair_of(w0q[q].v[0], w0q[q].v[2]);
          w0m = pair_of(w0q[q].v[1], w0q[q].v[3]);
        }
        if (nrm > 1e-30f && nrm < 1e30f) {
          const float2 full = cmul(e, make_float2(2.f + e.x, e.y));
          float2 mhalf = make_float2(0.f, 0.f);
          if constexpr (MODE == 1) {
            const float rden = __frcp_rn(nrm);
            const float2 qq = cmul(e, cconj(e1));
            mhalf = make_float2(-qq.x * rden, -qq.y * rden);
          }
          const float2 d2 = splat2(dt);
          const C2 adv = {__ffma2_rn(r.re, d2, w.re), __ffma2_rn(r.im, d2, w.im)};
          const C2 advm = {__ffma2_rn(rm.re, d2, wm.re), __ffma2_rn(rm.im, d2, wm.im)};
          w = rk_pair<MODE>(e, full, mhalf, w0, adv);
          wm = rk_pair<MODE>(cconj(e), cconj(full), cconj(mhalf), w0m, advm);
        } else {
          // a factor that overflows or vanishes: cell by cell, zero modes stay zero
          auto one = [&](float2 ee, float2 v0, float2 vc, float2 rr) {
            const bool quiet = vc.x == 0.f && vc.y == 0.f && v0.x == 0.f && v0.y == 0.f && rr.x == 0.f && rr.y == 0.f;
            return quiet ? make_float2(0.f, 0.f) : rk_update<MODE>(ee, v0, vc, rr, dt);
          };
          auto two = [&](float2 ee, C2 v0, C2 vc, C2 rr) {
            return pair_of(one(ee, make_float2(v0.re.x, v0.im.x), make_float2(vc.re.x, vc.im.x), make_float2(rr.re.x, rr.im.x)),
                           one(ee, make_float2(v0.re.y, v0.im.y), make_float2(vc.re.y, vc.im.y), make_float2(rr.re.y, rr.im.y)));
          };
          w = two(e, w0, w, r);
          wm = two(cconj(e), w0m, wm, rm);
        }
        if (k2 == 0.f) w = wm = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        a.wout[ra + c] = make_float2(w.re.x, w.im.x);
        a.wout[ra + mc] = make_float2(wm.re.x, wm.im.x);
        a.wout[rb + c] = make_float2(w.re.y, w.im.y);
        a.wout[rb + mc] = make_float2(wm.re.y, wm.im.y);
      }
      // next-stage packs scaled by 1/N^2: w + i u_hat = w (1 -+ ky/k2) on rows +-ky, and the
      // Hermitian part of v_hat = -i kx w/k2 on row ky
      const float inv = k2 > 0.f ? __frcp_rn(k2) : 0.f;
      const float2 fa = make_float2((1.f - ky * inv) * inv_n2, (1.f + ky * inv) * inv_n2);
      const float fb = 0.5f * (kx * inv * inv_n2);
      const C2 pc = {__fmul2_rn(w.re, fa), __fmul2_rn(w.im, fa)}, pm = {__fmul2_rn(wm.re, fa), __fmul2_rn(wm.im, fa)};
      const float2 vc = make_float2((w.im.x - wm.im.y) * fb, -(w.re.x + wm.re.y) * fb);
      const float2 vm = make_float2(-(wm.im.x - w.im.y) * fb, (wm.re.x + w.re.y) * fb);
      l4[TU::pad(c)] = make_float4(pc.re.x, pc.re.y, pc.im.x, pc.im.y);
      l4[TU::pad(mc)] = make_float4(pm.re.x, pm.re.y, pm.im.x, pm.im.y);
      l2[TU::pad(c)] = vc;
      l2[TU::pad(mc)] = vm;
    }
  }
  sync();
#pragma unroll
  for (int m = 0; m < V; ++m) {
    const int c = t + T * m;
    x[m] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    y[m] = make_float2(0.f, 0.f);
    if (!slot_empty<TU>(m) && pair_inband<TU>(c)) {
      const float4 q = l4[TU::pad(c)];
      x[m] = {make_float2(q.x, q.y), make_float2(q.z, q.w)};
      y[m] = l2[TU::pad(c)];
    }
  }
  sync();
  pair_fft<TU, +1, true, 1>(x, y, l4, l2, t, a.ptw, sync);
#pragma unroll
  for (int m = 0; m < V; ++m) {
    const int c = t + T * m;
    a.pa[ra + c] = make_float2(x[m].re.x, x[m].im.x);
    a.pa[rb + c] = make_float2(x[m].re.y, x[m].im.y);
    a.pb[ra + c] = y[m];
    if (a.full_pb && p > 0) a.pb[rb + c] = cconj(y[m]);
  }
}

template <int MODE, bool PTR, class TU>
__global__ void __launch_bounds__(TU::B_THREADS, TU::B_MINB) k_pair_rows(SpecArgs a) {
  extern __shared__ __align__(16) float4 smem4[];
  pair_rows_tile<MODE, PTR, TU>(a, blockIdx.x, smem4);
}

// the row flags of packs written by k_pair_rows: in-band rows
static __global__ void k_band_flags(int* row_nz, int n) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) row_nz[r] = (r <= n / 3 || r >= n - n / 3) ? 1 : 0;
}
// packs written by k_pair_rows made whole: rows outside the band zero, PB(-ky) = conj PB(ky)
static __global__ void k_expand_packs(float2* pa, float2* pb, int n, int half_pb) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n * n) return;
  const int r = (int)(i / n), c = (int)(i & (n - 1));
  if (r > n / 3 && r < n - n / 3) pa[i] = pb[i] = make_float2(0.f, 0.f);
  else if (half_pb && r > n / 2) pb[i] = cconj(pb[(size_t)(n - r) * n + c]);
}

// whether a (prefix of a) complex n x n spectrum is zero outside the dealias band
inline bool band_limited(const float* w, size_t count, int n) {
  auto any = [&](size_t lo, size_t hi) {
    bool some = false;
    for (size_t i = lo, e = hi < count ? hi : count; i < e; ++i) some |= w[i] != 0.f;
    return some;
  };
  for (int r = 0; r < n; ++r) {
    const size_t row = (size_t)2 * n * r;
    const bool in = r <= n / 3 || r >= n - n / 3;
    if (any(row + (in ? 2 * (size_t)(n / 3 + 1) : 0), row + (in ? 2 * (size_t)(n - n / 3) : 2 * (size_t)n))) return false;
  }
  return true;
}

}  // namespace s2d
