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
//                of the four Hermitian unpacks and forcing phases.  Its cells are a rolled
//                loop with the state one column ahead, the first column's ahead of the
//                x-transform and of the launch dependency.
//   k_pair_cols  columns x and x+1.  v is real, so its x-transformed spectrum obeys
//                PB(-ky, x) = conj PB(ky, x): only the rows ky >= 0 are stored, and the two
//                columns' v come out of ONE complex y-transform of V(x) + i V(x+1).
//
// Transforms per stage and row pair: 2 forward and 3 inverse lines (2 and 4 with both rows of
// PB); per column pair 3 inverse and 2 forward lines (4 and 2).  PB holds the Hermitian part
// of v_hat, whose inverse transform is the real part the stage reads, so a state that is not
// exactly Hermitian steps as before.
//
// Bound (1024^2, cold launches under a profiler): latency.  Columns 11.9 us, 8.5 MB read, issue
// slots 32 % busy, 8 warps per SM (one CTA of 256 threads on each of 128 SMs: its registers are
// its lines); rows 14.1 us, 13.4 MB read, 34 %, 9 warps, waiting at the barriers of the
// transforms and for Z and the state.  The kernels of s2d_kernels.cuh take 13.9 and 23.3 us there, with
// 4.5 and 8.3 M warp instructions against 2.5 and 3.4 M.  An RK3 step, graph-replayed with
// forcing, against those kernels (us): 64^2 17 / 55.8, 256^2 20.6 / 56, 512^2 28.4 / 63,
// 1024^2 52 / 98, 2048^2 186 / 418, 4096^2 730 / 2023.
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
// Entry [r-1][jm] of pass p (p >= 1) is W_N^{jm r N/(NS R)} = c - i s as (c, s): lanes of a warp
// read consecutive entries (the plain table's stride would touch a line per lane).  As packed
// operands (c, c, s, s) the table costs twice the loads: 2048^2 step 198 against 186 us, 4096^2
// 798 / 760, 256 x 256^2 ensemble 593 / 581.
template <int N, int V> struct PassTw {
  using PL = LinePlan<N, V>;
  __host__ __device__ static constexpr int offset(int p) {
    int o = 0;
    for (int q = 1; q < p; ++q) o += (PL::radix(q) - 1) * PL::ns(q);
    return o;
  }
  static constexpr int SIZE = offset(PL::P);
};
template <int N, int V> __global__ void k_pass_twiddles(float2* out, const float2* __restrict__ tw) {
  using PL = LinePlan<N, V>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int o = 0;
  for (int p = 1; p < PL::P; ++p) {
    const int ns = PL::ns(p), r = PL::radix(p), len = (r - 1) * ns;
    if (i >= o && i < o + len) {
      const int q = (i - o) / ns + 1, jm = (i - o) % ns;
      const float2 w = tw[jm * q * (N / (ns * r))];   // (cos, -sin)
      out[i] = make_float2(w.x, -w.y);
    }
    o += len;
  }
}

// ------------------------------------------------------------------ launch shapes
// Column kernels run GP column pairs of T = N/V threads per CTA, row kernels THREADS / T whole
// row pairs; MINB is the number of resident CTAs the register budget must allow.  BP_: the
// packs between the two are stored in blocks of four columns, [x/4][ky][4], so that a column
// CTA reads contiguous lines (and a row CTA writes 32-byte sectors).
template <int N_, int V_, bool BP_ = false> struct PairLine {
  static constexpr int N = N_, V = V_, T = N / V;
  static constexpr bool BP = BP_;
  using PL = LinePlan<N, V>;
  static constexpr int KMAX = N / 3;          // largest in-band wavenumber: |k| < N/3, N a power of two
  static constexpr int BAND = KMAX + 1;       // in-band k = 0..KMAX: row pairs, and columns of a thread quad
  __host__ __device__ static constexpr int pad(int i) { return i + i / V; }
  static constexpr int PADDED = N + T;
};
template <int N_, int V_, int GP_, int MINB_, bool BP_ = false> struct PairCols : PairLine<N_, V_, BP_> {
  using L = PairLine<N_, V_, BP_>;
  static constexpr int GP = GP_, THREADS = GP * L::T, GRID = N_ / 2 / GP, MINB = MINB_;
  static constexpr size_t SMEM = (size_t)L::PADDED * GP * (sizeof(float4) + sizeof(float2));
  static_assert((N_ / 2) % GP == 0 && (!BP_ || GP == 2), "whole lines, one block of four columns");
};
template <int N_, int V_, int THREADS_, int MINB_, bool BP_ = false, bool SPLIT_ = false>
struct PairRows : PairLine<N_, V_, BP_> {
  using L = PairLine<N_, V_, BP_>;
  // SPLIT_: a CTA is one row pair with 2 T threads; the second half does the single line's
  // transform and half of the cells
  static constexpr bool SPLIT = SPLIT_;
  static constexpr int TP = SPLIT ? 2 * L::T : L::T;   // threads of a row pair
  static constexpr int THREADS = THREADS_, PPB = THREADS / TP, GRID = (L::BAND + PPB - 1) / PPB, MINB = MINB_;
  static constexpr size_t SMEM = (size_t)L::PADDED * PPB * (sizeof(float4) + sizeof(float2));
  static_assert(SPLIT ? THREADS == TP && L::T >= 32 : THREADS % L::T == 0, "whole lines");
};
// The shapes in use, each the fastest of those timed in turn on a B200 (us per launch, graph
// replayed without forcing, columns / rows of stage 1; "split": SPLIT_):
//   64     V=4  1.7 / 2.9
//   256    V=4, 4 columns a CTA, split 2.6 / 2.7     rows not split 3.2, V=8 split 3.7
//   512    V=8, split 3.4 / 4.5                      rows not split 4.9, V=4 split 5.3
//   1024   columns V=16, 8 columns a CTA 7.2 (4 columns 8.1, V=8 9.3); rows V=16, split, 3 CTAs/SM
//          8.7 (V=8 9.5, V=8 split 9.2; 2 or 4 CTAs/SM 13.1, 9.8)
//   2048   V=16 33 / 28 (rows split 28, 4 CTAs/SM 32)    V=8 43 / 33
//   4096   V=16 in blocks 109 / 129, in rows 189 / 125   V=8 183 / 173
// Small grids want more threads per line (the chain of a thread's cells sets the time), large
// ones fewer, longer passes (shared-memory traffic does).  Splitting a row pair shortens the
// chain by a third of the cells and the single line, and pays while SMs have room.  Blocked packs
// pay where a column's rows lie 32 KB apart (4096); at 2048 the row kernel loses what the
// column kernel gains.
template <int N> struct PairShape;
template <> struct PairShape<32> { using C = PairCols<32, 4, 4, 16>; using R = PairRows<32, 4, 32, 16>; };
template <> struct PairShape<64> { using C = PairCols<64, 4, 2, 16>; using R = PairRows<64, 4, 32, 16>; };
template <> struct PairShape<128> { using C = PairCols<128, 4, 1, 16>; using R = PairRows<128, 4, 64, 8, false, true>; };
template <> struct PairShape<256> { using C = PairCols<256, 4, 2, 4>; using R = PairRows<256, 4, 128, 4, false, true>; };
template <> struct PairShape<512> { using C = PairCols<512, 8, 2, 4>; using R = PairRows<512, 8, 128, 4, false, true>; };
template <> struct PairShape<1024> { using C = PairCols<1024, 16, 4, 1>; using R = PairRows<1024, 16, 128, 3, false, true>; };
template <> struct PairShape<2048> { using C = PairCols<2048, 16, 4, 1>; using R = PairRows<2048, 16, 128, 3>; };
template <> struct PairShape<4096> { using C = PairCols<4096, 16, 2, 1, true>; using R = PairRows<4096, 16, 256, 2, true>; };
template <int N> struct PairStepShape { using S = void; };
template <> struct PairStepShape<32>;
template <> struct PairStepShape<64>;
template <> struct PairStepShape<128>;
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

// A packed pair of lines (HASX) and/or one single line (HASY), transformed in lockstep.
// Element i of the pair is at l4[pad(i) * ST], of the single line at l2[pad(i) * ST].
template <class TU, int SIGN, bool HASX, bool HASY, int ST, class Sync>
__device__ __forceinline__ void lines_fft(C2 (&x)[TU::V], float2 (&y)[TU::V], float4* l4, float2* l2, int t,
                                          const float2* __restrict__ tw, const Sync& sync) {
  using PL = typename TU::PL;
  constexpr int N = TU::N, V = TU::V, T = TU::T;
  sfor<PL::P>([&](auto pc) {
    constexpr int p = decltype(pc)::value;
    constexpr int R = PL::radix(p), B = V / R, NS = PL::ns(p);
    [[maybe_unused]] C2 v[V];
    [[maybe_unused]] float2 w[V];
    if constexpr (p == 0) {
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (HASX) v[b * R + r] = x[b + B * r];
          if constexpr (HASY) w[b * R + r] = y[b + B * r];
        }
    } else {
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = TU::pad(t + T * b + r * (N / R)) * ST;
          if constexpr (HASX) {
            const float4 q = l4[i];
            v[b * R + r] = {make_float2(q.x, q.y), make_float2(q.z, q.w)};
          }
          if constexpr (HASY) w[b * R + r] = l2[i];
        }
      sync();
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const float2 q = __ldg(tw + PassTw<N, V>::offset(p) + (r - 1) * NS + ((t + T * b) & (NS - 1)));
          const float2 c = splat2(q.x), s = splat2(q.y);
          if constexpr (HASX) v[b * R + r] = cmul_cs(v[b * R + r], c, SIGN > 0 ? s : neg2(s));
          if constexpr (HASY) w[b * R + r] = cmul(w[b * R + r], make_float2(q.x, SIGN > 0 ? q.y : -q.y));
        }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      if constexpr (HASX) DftE<R, SIGN, C2>::run(&v[b * R]);
      if constexpr (HASY) DftE<R, SIGN, float2>::run(&w[b * R]);
    }
    if constexpr (p < PL::P - 1) {
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const int j = t + T * b;
        const int base = (j / NS) * NS * R + (j & (NS - 1));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = TU::pad(base + r * NS) * ST;
          if constexpr (HASX) {
            const C2 q = v[b * R + r];
            l4[i] = make_float4(q.re.x, q.re.y, q.im.x, q.im.y);
          }
          if constexpr (HASY) l2[i] = w[b * R + r];
        }
      }
      sync();
    } else {
#pragma unroll
      for (int b = 0; b < B; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (HASX) x[b + B * r] = v[b * R + r];
          if constexpr (HASY) y[b + B * r] = w[b * R + r];
        }
    }
  });
}

// ------------------------------------------------------------------ columns
// `mode` as phys_cols_tile's MODE, at run time: the stages of a step then share one kernel's
// code, which stays in the instruction caches from launch to launch.  `base` is the grid's first
// cell in the arrays of `a` (kernel arguments: pointers in registers cost spills) and ptw
// its twiddles.  One column pair per group; groups interleave over lanes (two pairs are one 32-byte sector per row).  Returns
// this thread's max |u|+|v| (mode != 1).
template <class TU>
__device__ __forceinline__ float pair_cols_tile(const PhysArgs& a, size_t base, const float2* ptw, int mode, int tile,
                                                float4* smem) {
  constexpr int N = TU::N, V = TU::V, T = TU::T, GP = TU::GP;
  const int g = threadIdx.x % GP, t = threadIdx.x / GP;
  const int x0 = 2 * (tile * GP + g);
  float4* const l4 = smem + g;
  float2* const l2 = reinterpret_cast<float2*>(smem + TU::PADDED * GP) + g;
  struct Sync {
    __device__ __forceinline__ void operator()() const {
      if constexpr (TU::THREADS <= 32) __syncwarp();
      else __syncthreads();
    }
  };
  C2 x[V];
  float2 y[V];
  auto at = [&](int r) { return base + (TU::BP ? ((size_t)(x0 >> 2) * N + r) * 4 + (x0 & 3) : (size_t)r * N + x0); };
  auto load_x = [&] {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int row = t + T * m;
      x[m] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      if (!slot_empty<TU>(m) && pair_inband<TU>(row)) {
        const float4 p = __ldcs(reinterpret_cast<const float4*>(a.pa + at(row)));
        x[m] = {make_float2(p.x, p.z), make_float2(p.y, p.w)};
      }
    }
  };
  auto load_y = [&] {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int row = t + T * m;
      y[m] = make_float2(0.f, 0.f);
      if (!slot_empty<TU>(m) && pair_inband<TU>(row)) {
        const bool up = row < N / 2;
        const float4 q = *reinterpret_cast<const float4*>(a.pb + at(up ? row : N - row));
        // V(x) + i V(x+1), conjugated spectra for -ky; row 0 is real
        if (row == 0) y[m] = make_float2(q.x, q.z);
        else y[m] = up ? make_float2(q.x - q.w, q.y + q.z) : make_float2(q.x + q.w, q.z - q.y);
      }
    }
  };
  load_x();
  load_y();
  lines_fft<TU, +1, true, true, GP>(x, y, l4, l2, t, ptw, Sync{});
  // re = omega, im = u at (x, x+1); y = v at (x, x+1)
  float speed = 0.f;
  if (mode != 1) {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const float2 u = x[m].im, v = y[m];
      *reinterpret_cast<float4*>(a.vel + (size_t)(t + T * m) * N + x0) = make_float4(u.x, v.x, u.y, v.y);
      speed = fmaxf(speed, fmaxf(fabsf(u.x) + fabsf(v.x), fabsf(u.y) + fabsf(v.y)));
    }
  }
  if (mode != 0) {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const float2 om = x[m].re;
      x[m] = {__fmul2_rn(x[m].im, om), __fmul2_rn(y[m], om)};
    }
    lines_fft<TU, -1, true, false, GP>(x, y, l4, l2, t, ptw, Sync{});
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int row = t + T * m;
      if (!slot_empty<TU>(m) && pair_inband<TU>(row))
        *reinterpret_cast<float4*>(a.z + base + (size_t)row * N + x0) =
            make_float4(x[m].re.x, x[m].im.x, x[m].re.y, x[m].im.y);
    }
  }
  return speed;
}

// bytes (a multiple of 16, from a 16-byte boundary) from global memory towards L2
__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// CTA maximum of |u|+|v| into *top (bits of a non-negative float order as integers); the row
// kernel behind it forms the next dt from the total (pair_cfl)
template <int NTHREADS> __device__ __forceinline__ void cols_speed_max(unsigned* top, float speed) {
  unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(speed));
  if constexpr (NTHREADS > 32) {
    __shared__ unsigned red[NTHREADS / 32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) m = __reduce_max_sync(0xffffffffu, threadIdx.x < NTHREADS / 32 ? red[threadIdx.x] : 0u);
  }
  if (threadIdx.x == 0) atomicMax(top, m);
}

// Bound by latency: up to 1024^2 one wave (see the head of this file); beyond, one CTA of 512
// threads on an SM at 128 registers, whose loads, transforms and stores have nothing beside them
// (cold, stage 1: 2048^2 L1 wavefronts 40 %, issue slots 34 %, HBM 10 %; 4096^2 56, 40 and 19 %).
// The stage is a run-time argument, as in the row kernel: three copies of the code fetched anew by
// each launch cost more than the tests.  1024^2 7.2 us a launch (k_phys_cols 14), 2048^2 33,
// 4096^2 109.
template <class TU>
__global__ void __launch_bounds__(TU::THREADS, TU::MINB) k_pair_cols(PhysArgs a, int mode) {
  extern __shared__ __align__(16) float4 smem4[];
  pdl_wait();
  phys_latch(a);
  if constexpr (TU::BP) {
    // blocked packs of a column CTA are three contiguous pieces: the CTA that follows on an SM
    // (148 SMs) finds its own on their way from HBM (4096^2: 121 -> 109 us; the row kernel's
    // rows gained nothing, 126 -> 130 us)
    const int next = blockIdx.x + 148 * TU::MINB;
    if (threadIdx.x == 0 && next < TU::GRID) {
      constexpr int W = 2 * TU::GP;   // columns
      const size_t b = (size_t)next * TU::N * W;
      l2_prefetch(a.pa + b, TU::BAND * W * sizeof(float2));
      l2_prefetch(a.pa + b + (size_t)(TU::N - TU::KMAX) * W, TU::KMAX * W * sizeof(float2));
      l2_prefetch(a.pb + b, TU::BAND * W * sizeof(float2));
    }
  }
  const float speed = pair_cols_tile<TU>(a, 0, a.ptw, mode, blockIdx.x, smem4);
  if (mode == 2) cols_speed_max<TU::THREADS>(a.ticket + 1, speed);
  else if (mode == 0) cols_speed_finalize<TU::THREADS>(a, speed);
}

// ------------------------------------------------------------------ rows
__device__ __forceinline__ C2 pair_of(float2 a, float2 b) { return {make_float2(a.x, b.x), make_float2(a.y, b.y)}; }
// w + e w
__device__ __forceinline__ C2 grow(C2 w, float2 e) { return cadd(w, cmul_w(w, e)); }

// Out-of-line parts of a cell quad: rare, and each would otherwise be copied into the kernel
// with its trigonometric argument reductions (the row kernel waited on instruction fetches).
// E(dt/2) - 1 where a series of half_factor_m1 does not reach
static __device__ __noinline__ float2 half_factor_far(float x, float half_th) {
  const float d = expm1_series(x);
  float sh, ch;
  sincos_series(half_th, &sh, &ch);
  const float g = -2.f * sh * sh, sn = 2.f * sh * ch;
  return make_float2(d + g + d * g, (1.f + d) * sn);
}
// the forcing of k = (kx, ky) and (-kx, ky); -k takes the conjugates
static __device__ __noinline__ float4 stochastic_pair(const DevParams* P, int n, int p, int c, float dt) {
  const float kx = (float)c, ky = (float)p, k2 = kx * kx + ky * ky;
  const float2 f1 = stochastic_term(*P, n, p, c, kx, ky, k2, dt);
  const float2 f2 = stochastic_term(*P, n, p, (n - c) & (n - 1), -kx, ky, k2, dt);
  return make_float4(f1.x, f1.y, f2.x, f2.y);
}
// the stage update cell by cell where a factor overflows or vanishes: zero modes stay zero
static __device__ __noinline__ float2 rk_cell(int stage, float2 e, float2 w0, float2 wc, float2 rhs, float dt) {
  const bool quiet = wc.x == 0.f && wc.y == 0.f && w0.x == 0.f && w0.y == 0.f && rhs.x == 0.f && rhs.y == 0.f;
  if (quiet) return make_float2(0.f, 0.f);
  return stage == 0 ? rk_update<0>(e, w0, wc, rhs, dt)
         : stage == 1 ? rk_update<1>(e, w0, wc, rhs, dt) : rk_update<2>(e, w0, wc, rhs, dt);
}

// One group's row pair.  `stage` is the RK stage at run time (one kernel for the step, see
// pair_cols_tile), -1 packs wcur only; the grid's parameters, step and twiddles come beside
// the arrays of `a`, its first cell is `base`.
template <class TU, bool WAIT = false>
__device__ __forceinline__ void pair_rows_tile(const SpecArgs& a, size_t base, const DevParams* P, float dt, bool forced,
                                               const float2* ptw, int stage, int tile, float4* smem) {
  constexpr int N = TU::N, V = TU::V, T = TU::T, BAND = TU::BAND, KMAX = TU::KMAX;
  const int t = threadIdx.x % T, g = threadIdx.x / TU::TP;
  // cells from column t0 on; with SPLIT the threads of the single line come second
  const int t0 = threadIdx.x % TU::TP;
  const bool has_x = !TU::SPLIT || t0 < T, has_y = !TU::SPLIT || t0 >= T;
  const int p = min(tile * TU::PPB + g, KMAX);   // the last CTA's spare groups repeat pair KMAX
  const size_t ra = base + (size_t)p * N, rb = base + (size_t)((N - p) & (N - 1)) * N;
  float4* const l4 = smem + g * TU::PADDED;
  float2* const l2 = reinterpret_cast<float2*>(smem + TU::PPB * TU::PADDED) + g * TU::PADDED;
  const GroupSync<T, TU::THREADS> sync;          // the threads of a line
  const GroupSync<TU::TP, TU::THREADS> psync;    // ... of the pair
  C2 x[V];
  float2 y[V];
  const bool two = stage >= 1;   // w0 is not wcur
  // state cells (row, column) = (a, c), (a, -c), (b, c), (b, -c) of the next column, the first
  // loaded ahead of the x-transform
  float2 nw[4], nw0[4];
  auto fetch = [&](int c) {
    if (c < BAND) {
      const int mc = (N - c) & (N - 1);
      nw[0] = a.wcur[ra + c], nw[1] = a.wcur[ra + mc], nw[2] = a.wcur[rb + c], nw[3] = a.wcur[rb + mc];
      if (two) nw0[0] = a.w0[ra + c], nw0[1] = a.w0[ra + mc], nw0[2] = a.w0[rb + c], nw0[3] = a.w0[rb + mc];
    }
  };
  fetch(t0);
  const float beta = P->beta, mu = P->mu, nu = P->nu_h;
  const int hyper = P->hyper_p;
  const float2 fb = forced ? forcing_k2_bounds(*P) : make_float2(1.f, 0.f);   // empty without forcing
  // Z-hat, then the packs, lie in natural order without padding: every access of theirs is a
  // run of consecutive slots, upwards or (-kx) downwards, at any alignment
  const float ky = (float)p;
  // all of the above is two or more launches old; Z is the launch before
  if constexpr (WAIT) pdl_wait();
  if (stage >= 0 && has_x) {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      x[m] = pair_of(__ldcs(a.z + ra + c), __ldcs(a.z + rb + c));
    }
    lines_fft<TU, -1, true, false, 1>(x, y, l4, l2, t, ptw, sync);
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      if (!slot_empty<TU>(m) && pair_inband<TU>(c))
        l4[c] = make_float4(x[m].re.x, x[m].re.y, x[m].im.x, x[m].im.y);
    }
  }
  psync();
  constexpr float inv_n2 = 1.0f / ((float)N * (float)N);
#pragma unroll 1
  for (int c = t0; c < BAND; c += TU::TP) {
    const int mc = (N - c) & (N - 1);
    const float kx = (float)c;
    const float k2 = kx * kx + ky * ky;
    float2 wq[4], w0q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      wq[k] = nw[k];
      w0q[k] = nw0[k];
    }
    fetch(c + TU::TP);
    C2 w = pair_of(wq[0], wq[2]), wm = pair_of(wq[1], wq[3]);   // columns c, -c
    if (stage >= 0) {
      const float4 zc = l4[c], zm = l4[mc];   // (re a, re b, im a, im b)
      // right-hand sides at k = (kx, ky) and (-kx, ky); the other two cells hold the conjugates
      auto minus_nhat = [&](float kxs, float2 zk, float2 zp) {   // zp = Z(-k)
        const float2 q1 = make_float2(0.5f * (zk.x + zp.x), 0.5f * (zk.y - zp.y));
        const float2 q2 = make_float2(0.5f * (zk.y + zp.y), -0.5f * (zk.x - zp.x));
        return make_float2(kxs * q1.y + ky * q2.y, -(kxs * q1.x) - ky * q2.x);
      };
      float2 r1 = minus_nhat(kx, make_float2(zc.x, zc.z), make_float2(zm.y, zm.w));
      float2 r2 = minus_nhat(-kx, make_float2(zm.x, zm.z), make_float2(zc.y, zc.w));
      if (k2 > 0.f && k2 >= fb.x && k2 <= fb.y) {
        const float4 f = stochastic_pair(P, N, p, c, dt);
        r1 = cadd(r1, make_float2(f.x, f.y));
        r2 = cadd(r2, make_float2(f.z, f.w));
      }
      C2 r = {make_float2(r1.x, r2.x), make_float2(r1.y, -r2.y)};
      C2 rm = {make_float2(r2.x, r1.x), make_float2(r2.y, -r1.y)};
      if (a.fptr) {
        r = cadd(r, pair_of(__ldg(a.fptr + ra + c), __ldg(a.fptr + rb + c)));
        rm = cadd(rm, pair_of(__ldg(a.fptr + ra + mc), __ldg(a.fptr + rb + mc)));
      }
      C2 w0 = w, w0m = wm;
      if (two) {
        w0 = pair_of(w0q[0], w0q[2]);
        w0m = pair_of(w0q[1], w0q[3]);
      }
      // E(dt/2) - 1 (half_factor_m1)
      const float ex = (-mu - nu * powi(k2, hyper)) * (0.5f * dt);
      const float hth = beta == 0.f ? 0.f : 0.5f * (beta * __fdividef(kx, fmaxf(k2, 1.f)) * (0.5f * dt));
      float2 e;
      if (fabsf(ex) < 0.25f && fabsf(hth) <= 0.78539816f) {
        const float m1 = expm1_series(ex);
        float sh, ch;
        sincos_series(hth, &sh, &ch);
        const float gg = -2.f * sh * sh, sn = 2.f * sh * ch;
        e = make_float2(m1 + gg + m1 * gg, (1.f + m1) * sn);
      } else {
        e = half_factor_far(ex, hth);
      }
      const float2 e1 = make_float2(1.f + e.x, e.y);
      const float nrm = e1.x * e1.x + e1.y * e1.y;
      if (nrm > 1e-30f && nrm < 1e30f) {
        // wout = B + cA (A - B), A = E(a dt) w0, B = E(b dt)(wcur + dt rhs): rk_update<stage>
        const float2 full = cmul(e, make_float2(2.f + e.x, e.y));
        float2 fA = full, fB = e;
        float cA = 1.f / 3.f;
        if (stage == 0) {
          fB = full;
          cA = 0.f;
        } else if (stage == 1) {
          const float rden = __frcp_rn(nrm);
          const float2 qq = cmul(e, cconj(e1));
          fA = e;
          fB = make_float2(-qq.x * rden, -qq.y * rden);
          cA = 0.75f;
        }
        const float2 d2 = splat2(dt), c2 = splat2(cA);
        auto blend = [&](C2 v0, C2 vc, C2 rr, float2 ea, float2 eb) {
          const C2 A = grow(v0, ea), B = grow({__ffma2_rn(rr.re, d2, vc.re), __ffma2_rn(rr.im, d2, vc.im)}, eb);
          const C2 dd = csub(A, B);
          return C2{__ffma2_rn(dd.re, c2, B.re), __ffma2_rn(dd.im, c2, B.im)};
        };
        w = blend(w0, w, r, fA, fB);
        wm = blend(w0m, wm, rm, cconj(fA), cconj(fB));
      } else {
        auto cell2 = [&](float2 ee, C2 v0, C2 vc, C2 rr) {
          return pair_of(rk_cell(stage, ee, make_float2(v0.re.x, v0.im.x), make_float2(vc.re.x, vc.im.x), make_float2(rr.re.x, rr.im.x), dt),
                         rk_cell(stage, ee, make_float2(v0.re.y, v0.im.y), make_float2(vc.re.y, vc.im.y), make_float2(rr.re.y, rr.im.y), dt));
        };
        w = cell2(e, w0, w, r);
        wm = cell2(cconj(e), w0m, wm, rm);
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
    const float hb = 0.5f * (kx * inv * inv_n2);
    const C2 pc = {__fmul2_rn(w.re, fa), __fmul2_rn(w.im, fa)}, pm = {__fmul2_rn(wm.re, fa), __fmul2_rn(wm.im, fa)};
    const float2 vc = make_float2((w.im.x - wm.im.y) * hb, -(w.re.x + wm.re.y) * hb);
    const float2 vm = make_float2(-(wm.im.x - w.im.y) * hb, (wm.re.x + w.re.y) * hb);
    l4[c] = make_float4(pc.re.x, pc.re.y, pc.im.x, pc.im.y);
    l4[mc] = make_float4(pm.re.x, pm.re.y, pm.im.x, pm.im.y);
    l2[c] = vc;
    l2[mc] = vm;
  }
  psync();
  // in-band elements of a line, zeros elsewhere
  auto load_x = [&] {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      x[m] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      if (!slot_empty<TU>(m) && pair_inband<TU>(c)) {
        const float4 q = l4[c];
        x[m] = {make_float2(q.x, q.y), make_float2(q.z, q.w)};
      }
    }
  };
  auto load_y = [&] {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      y[m] = !slot_empty<TU>(m) && pair_inband<TU>(c) ? l2[c] : make_float2(0.f, 0.f);
    }
  };
  const size_t bs = TU::BP && !a.full_pb ? (size_t)4 * N : 4, rs = TU::BP && !a.full_pb ? 4 : N;
  auto pat = [&](int r, int c) { return base + (size_t)r * rs + (size_t)(c >> 2) * bs + (c & 3); };
  auto store_y = [&] {
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t + T * m;
      a.pb[pat(p, c)] = y[m];
      if (a.full_pb && p > 0) a.pb[rb + c] = cconj(y[m]);
    }
  };
  if constexpr (TU::SPLIT) {
    if (has_y) {
      load_y();
      sync();
      lines_fft<TU, +1, false, true, 1>(x, y, l4, l2, t, ptw, sync);
      store_y();
      return;
    }
    load_x();
    sync();
    lines_fft<TU, +1, true, false, 1>(x, y, l4, l2, t, ptw, sync);
  } else {
    load_x();
    load_y();
    sync();
    lines_fft<TU, +1, true, true, 1>(x, y, l4, l2, t, ptw, sync);
    store_y();
  }
#pragma unroll
  for (int m = 0; m < V; ++m) {
    const int c = t + T * m;
    a.pa[pat(p, c)] = make_float2(x[m].re.x, x[m].im.x);
    a.pa[pat((N - p) & (N - 1), c)] = make_float2(x[m].re.y, x[m].im.y);
  }
}

// the next dt from the maximum k_pair_cols left, by one thread of the last stage's row kernel
// (its CTAs do not wait for it; as the column kernel's own last-CTA reduction it took 1.7 us)
__device__ __forceinline__ void pair_cfl(const SpecArgs& a) {
  const float m = __uint_as_float(*a.top);
  a.dt_out[0] = cfl_dt(*a.params, m);
  a.dt_out[1] = m;
  *a.top = 0u;
}

// Bound by latency: the barriers of two transforms and a chain of cells per thread (1024^2
// 8.7 us a launch where k_spec_rows takes 23; 2048^2 28, 4096^2 129).  The cell loop is rolled,
// with its rare parts out of line, since unrolled it waited on instruction fetches (64^2 5.2 us
// against 3.7; at 1024^2 3.8 such stalls per issue, now 0.6).
template <class TU>
__global__ void __launch_bounds__(TU::THREADS, TU::MINB) k_pair_rows(SpecArgs a, int stage) {
  extern __shared__ __align__(16) float4 smem4[];
  pair_rows_tile<TU, true>(a, 0, a.params, stage >= 0 ? __ldg(a.dt) : 0.f, a.stochastic != 0, a.ptw, stage, blockIdx.x,
                           smem4);
  if (stage == 2 && a.top && blockIdx.x == 0 && threadIdx.x == 0) pair_cfl(a);
}

// ------------------------------------------------------------------ a whole step in one launch
// Up to 128^2 a stage kernel is launch and latency (3.4 us each at 64^2 for 0.3 us of work), so
// one thread-block cluster runs the six passes: the packs and Z go through L2 as between
// launches, and the cluster barrier orders them.  64^2 20.6 -> 17 us a step, 128^2 22.7 -> 20
// (and one host launch of 3 us instead of six); at 256^2 sixteen CTAs have too much to do: 43
// against 25.
template <class C_, class R_, int CTAS_> struct PairStep {
  using C = C_;
  using R = R_;
  static constexpr int CTAS = CTAS_, THREADS = C::THREADS;
  static constexpr size_t SMEM = C::SMEM > R::SMEM ? C::SMEM : R::SMEM;
  static_assert(C::THREADS == R::THREADS && C::GRID % CTAS == 0, "one block shape");
};
template <> struct PairStepShape<32> { using S = PairStep<PairCols<32, 4, 16, 1>, PairRows<32, 4, 128, 1>, 1>; };
template <> struct PairStepShape<64> { using S = PairStep<PairCols<64, 4, 4, 1>, PairRows<64, 4, 64, 1>, 8>; };
template <> struct PairStepShape<128> { using S = PairStep<PairCols<128, 4, 4, 1>, PairRows<128, 4, 128, 1>, 16>; };
template <int CTAS> __device__ __forceinline__ void cluster_barrier() {
  if constexpr (CTAS == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
template <class S>
__global__ void __launch_bounds__(S::THREADS, 1) k_pair_step(PhysArgs pa, SpecArgs sa, float2* s0, float2* s1, float2* s2) {
  using C = typename S::C;
  using R = typename S::R;
  extern __shared__ __align__(16) float4 smem4[];
  pdl_wait();
  phys_latch(pa);
  const float dt = __ldg(sa.dt);
  float speed = 0.f;
#pragma unroll 1
  for (int stage = 0; stage < 3; ++stage) {
    for (int tile = blockIdx.x; tile < C::GRID; tile += S::CTAS) {
      speed = fmaxf(speed, pair_cols_tile<C>(pa, 0, pa.ptw, stage == 2 ? 2 : 1, tile, smem4));
      __syncthreads();
    }
    if (stage == 2) cols_speed_max<S::THREADS>(sa.top, speed);
    cluster_barrier<S::CTAS>();
    // the state ring of stage `stage` (k_pair_rows' arguments, launch by launch)
    sa.w0 = s0;
    sa.wcur = stage == 0 ? s0 : stage == 1 ? s1 : s2;
    sa.wout = stage == 1 ? s2 : s1;
    for (int tile = blockIdx.x; tile < R::GRID; tile += S::CTAS) {
      pair_rows_tile<R>(sa, 0, sa.params, dt, sa.stochastic != 0, sa.ptw, stage, tile, smem4);
      __syncthreads();
    }
    if (stage == 2 && blockIdx.x == 0 && threadIdx.x == 0) pair_cfl(sa);
    if (stage < 2) cluster_barrier<S::CTAS>();
  }
}

// the row flags of packs written by k_pair_rows: in-band rows
static __global__ void k_band_flags(int* row_nz, int n) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) row_nz[r] = (r <= n / 3 || r >= n - n / 3) ? 1 : 0;
}
// packs written by k_pair_rows made whole: rows outside the band zero, PB(-ky) = conj PB(ky);
// a blocked pack ([x/4][ky][4]) is first copied to tmp and comes out in rows
static __global__ void k_expand_packs(float2* pa, float2* pb, int n, int half_pb) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n * n) return;
  const int r = (int)(i / n), c = (int)(i & (n - 1));
  if (r > n / 3 && r < n - n / 3) pa[i] = pb[i] = make_float2(0.f, 0.f);
  else if (half_pb && r > n / 2) pb[i] = cconj(pb[(size_t)(n - r) * n + c]);
}
static __global__ void k_unblock_pack(float2* out, const float2* __restrict__ tmp, int n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n * n) return;
  const int r = (int)(i / n), c = (int)(i & (n - 1));
  out[i] = tmp[((size_t)(c >> 2) * n + r) * 4 + (c & 3)];
}

}  // namespace s2d
