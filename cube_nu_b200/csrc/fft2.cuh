// Size-specialised FFT passes for the batched Poisson solve.
//
// A length N = R1*R2 transform runs as two register passes over shared memory
// (four-step): with n = R2*n1 + n2 and k = k1 + R1*k2,
//   step 1 (thread n2): R1-point DFT over n1, times w_N^(n2*k1), written in place;
//   step 2 (thread k1): R2-point DFT over n2, written to k1 + R1*k2.
// The R-point DFTs are unrolled in registers, composed recursively from radix 2/3/4
// with inner twiddles that are compile-time constants; the twiddles between the steps come
// from a shared table tw[j] = e^{-2 pi i j/N} (built on the host in double precision).  With N a template
// parameter every index is strength-reduced; no runtime integer division remains in
// the butterflies.
//
// Passes:
//   k_fx_r2c   : rows of reals, two rows packed as one complex sequence, unpacked into
//                two half spectra (r2c)
//   k_fcol3    : columns (y or z) of the half spectrum, forward / inverse; sequences stay in
//                registers
//   k_fz_loop  : z pass, forward -> Green multiply -> inverse, for N <= 144
//   k_fz_stream: the same for larger N
//   k_fx_c2r   : two half-spectrum rows packed as one Hermitian-extended sequence,
//                inverse, real and imaginary parts are the two real rows (c2r)
//   k_fxy3_r2c : for N <= 144 the x and y forward passes of one plane in one block
//   k_fyx3_c2r : its inverse (y then x)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fft.cuh"

namespace cube {
namespace f2 {

// 4-byte asynchronous global -> shared copies (sm_80+ cp.async), used to prefetch the
// Green table while the column data are in flight.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

template <int DIR>
__device__ __forceinline__ float2 twid(const float2* tw, int j) {
  float2 w = tw[j];
  if (DIR > 0) w.y = -w.y;
  return w;
}

template <int R>
struct Split {
  static constexpr int A = (R % 4 == 0 && R != 4) ? 4 : (R % 3 == 0 && R != 3) ? 3 : (R % 2 == 0 && R != 2) ? 2 : R;
  static constexpr int B = R / A;
};

// cos and sin of 2 pi j / n at compile time (Taylor series in double, |angle| <= pi).
constexpr double ct_pi = 3.14159265358979323846;
__host__ __device__ constexpr double ct_series(double x, double term, int k) {  // sum of (-1)^i x^(2i+k) / (2i+k)!
  double s = 0.0;
  for (int i = 0; i < 24; ++i) {
    s += term;
    term *= -x * x / ((2 * i + k + 1) * (2 * i + k + 2));
  }
  return s;
}
__host__ __device__ constexpr double ct_angle(int j, int n) { return 2.0 * ct_pi * (2 * j > n ? j - n : j) / n; }
__host__ __device__ constexpr double ct_cos(int j, int n) { return ct_series(ct_angle(j, n), 1.0, 0); }
__host__ __device__ constexpr double ct_sin(int j, int n) { return ct_series(ct_angle(j, n), ct_angle(j, n), 1); }

template <int I>
struct Int {
  static constexpr int v = I;
};
template <int I, int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(Int<I>{});
    static_for<I + 1, N>(f);
  }
}

// u times e^{DIR 2 pi i J / R}, the constant an immediate operand; nothing but a swap for
// multiples of a quarter turn.
template <int R, int J, int DIR>
__device__ __forceinline__ float2 ct_twiddle(float2 u) {
  if constexpr (J == 0) return u;
  else if constexpr (2 * J == R) return make_float2(-u.x, -u.y);
  else if constexpr (4 * J == R || 4 * J == 3 * R) {
    constexpr bool plus = (4 * J == R) == (DIR > 0);  // times +i or -i
    return plus ? make_float2(-u.y, u.x) : make_float2(u.y, -u.x);
  } else {
    constexpr float c = (float)ct_cos(J, R), s = (float)(DIR * ct_sin(J, R));
    return make_float2(u.x * c - u.y * s, u.x * s + u.y * c);
  }
}

// R-point DFT in registers (sign DIR).  Sums and differences are packed, two components to
// an instruction, and the inner twiddles are constants: a 12-point transform takes 78
// floating-point instructions and no reads of the twiddle table, 128 and 6 without either
// (512 boxes of 144^3: 4.13 + 3.32 + 4.01 ms for the three passes, 3.86 + 3.10 + 3.86 with).
template <int R, int N, int DIR>
struct DFT {
  static constexpr int A = Split<R>::A, B = Split<R>::B;
  static_assert(N % R == 0, "DFT size must divide the table size");
  __device__ __forceinline__ static void run(float2* v) {
    float2 tmp[R];
    static_for<0, B>([&](auto i2) {
      constexpr int n2 = decltype(i2)::v;
      float2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[B * n1 + n2];
      DFT<A, N, DIR>::run(u);
      static_for<0, A>([&](auto i1) {
        constexpr int k1 = decltype(i1)::v;
        tmp[k1 * B + n2] = ct_twiddle<R, (n2 * k1) % R, DIR>(u[k1]);
      });
    });
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      float2 w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) w[n2] = tmp[k1 * B + n2];
      DFT<B, N, DIR>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = w[k2];
    }
  }
};

template <int N, int DIR>
struct DFT<1, N, DIR> {
  __device__ __forceinline__ static void run(float2*) {}
};

template <int N, int DIR>
struct DFT<2, N, DIR> {
  __device__ __forceinline__ static void run(float2* v) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <int N, int DIR>
struct DFT<3, N, DIR> {
  __device__ __forceinline__ static void run(float2* v) {
    const float s3 = 0.8660254037844386f * (float)DIR;
    const float2 t1 = cadd(v[1], v[2]);
    const float2 d = csub(v[1], v[2]);
    const float2 m0 = fma2(make_float2(-0.5f, -0.5f), t1, v[0]);
    v[0] = cadd(v[0], t1);
    v[1] = make_float2(fmaf(-d.y, s3, m0.x), fmaf(d.x, s3, m0.y));
    v[2] = make_float2(fmaf(d.y, s3, m0.x), fmaf(-d.x, s3, m0.y));
  }
};

template <int N, int DIR>
struct DFT<4, N, DIR> {
  __device__ __forceinline__ static void run(float2* v) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 b0 = cadd(v[1], v[3]), b1 = csub(v[1], v[3]);
    const float2 jb1 = (DIR < 0) ? make_float2(b1.y, -b1.x) : make_float2(-b1.y, b1.x);
    v[0] = cadd(a0, b0);
    v[2] = csub(a0, b0);
    v[1] = cadd(a1, jb1);
    v[3] = csub(a1, jb1);
  }
};

template <int R1, int R2>
struct TPS {
  static constexpr int T = R1 > R2 ? R1 : R2;  // threads per sequence
};

// Slot of (k1, n2) in the exchange between the two steps, skewed so that neither the writes
// (fixed k1) nor the reads (fixed n2) meet on a bank.
template <int R1, int R2>
__device__ __forceinline__ int skew(int k1, int n2) {
  int j = n2 + k1;  // < R1 + R2
  if (R1 <= R2) j = (j >= R2) ? j - R2 : j;
  else j = j % R2;
  return k1 * R2 + j;
}

// Mesh layouts (both in place, potential written over the input):
//  row-pitched (five-pass sizes): row pitch RP bytes = max(N*rb, (N/2+1)*8) up to 16, so a real
//    row and its half-spectrum row share bytes (FFTW's in-place r2c layout); plane = N rows;
//  plane-compact (fused sizes): real rows of N, half-spectrum rows of N/2+1 up to even and phi
//    rows of N packed from the start of each plane; plane pitch the larger of the two.
// Kernels take the row pitch (pr real elements, pc complex, pf floats) and the plane pitch
// in the same units (plr, plc, plf).

// ---------------------------------------------------------------------------------
// X pass, r2c.  Block: S = 256/T packed sequences (2S real rows), T threads side by side each.
// A thread loads its R1 points of both rows straight from memory, and the exchange between
// the steps is skewed; staging the rows in shared memory first, with an exchange that read
// it at a stride of R2, cost 0.98 and 1.12 ms in 20 transforms of a 256^3 mesh each way, 0.52
// and 0.49 now.  In place: a sequence's rows are loaded before the first barrier.
// ---------------------------------------------------------------------------------
constexpr int FX_T = 256;
template <int N, int R1, int R2>
struct FxShape {
  static constexpr int T = TPS<R1, R2>::T, S = FX_T / T, MINB = T <= 18 ? 3 : 2;
  static constexpr size_t SMEM = (size_t)(N + S * N) * 8;
};

template <int N, int R1, int R2, typename IN>
__global__ void __launch_bounds__(FX_T, FxShape<N, R1, R2>::MINB) k_fx_r2c(const IN* r, float2* c, int64_t nrows,
                                                                         const float2* __restrict__ gtw, float scale,
                                                                         int pr, int pc) {
  using FX = FxShape<N, R1, R2>;
  constexpr int T = FX::T, NH = N / 2 + 1;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  for (int i = threadIdx.x; i < N; i += FX_T) tw[i] = gtw[i];
  const int s = threadIdx.x / T, t = threadIdx.x % T;
  const int64_t row = ((int64_t)blockIdx.x * FX::S + s) * 2;
  const bool act = s < FX::S && row < nrows, two = row + 1 < nrows;
  float2* Zr = sm + N + (s < FX::S ? s : 0) * N;
  float2 v[R1];
  if (act && t < R2) {
    const IN* a = r + row * pr + t;
    const IN* b = a + (two ? pr : 0);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      float fa, fb;
      if (sizeof(IN) == 8) {
        fa = (float)((double)(long long)a[R2 * n1] * 9.094947017729282e-13);  // 2^-40
        fb = (float)((double)(long long)b[R2 * n1] * 9.094947017729282e-13);
      } else {
        fa = (float)a[R2 * n1];
        fb = (float)b[R2 * n1];
      }
      v[n1] = make_float2(__fmul_rn(fa, scale), __fmul_rn(two ? fb : 0.f, scale));
    }
  }
  __syncthreads();  // the table
  if (act && t < R2) {
    DFT<R1, N, -1>::run(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) Zr[skew<R1, R2>(k1, t)] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
  }
  __syncthreads();
  float2 w[R2];
  if (act && t < R1) {
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) w[n2] = Zr[skew<R1, R2>(t, n2)];
    DFT<R2, N, -1>::run(w);
  }
  __syncthreads();
  if (act && t < R1) {
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) Zr[t + R1 * k2] = w[k2];
  }
  __syncthreads();
  if (act) {
    float2* c0 = c + row * pc;
    for (int k = t; k < NH; k += T) {
      const float2 z = Zr[k], zc = Zr[k == 0 ? 0 : N - k];
      c0[k] = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
      if (two) c0[pc + k] = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
    }
  }
}

// ---------------------------------------------------------------------------------
// Column pass with the sequences kept in registers.  Thread (t, col), blockDim = W*T,
// col fastest (coalesced rows of the half spectrum).  Forward (N = R1*R2, n = R2*n1+n2):
// thread t = n2 loads x[R2*n1 + t] straight from global memory, R1-point DFT, twiddle,
// one shared-memory exchange, then thread t = k1 runs the R2-point DFT and holds
// X[t + R1*k2].  The inverse uses the swapped factorisation (n = R1*n1 + n2), whose
// first step needs in thread t exactly the X[t + R1*k2] it already holds, so
// forward -> Green multiply -> inverse (k_fz_loop, k_fz_stream) costs two exchanges in all.
//   MODE 0: forward, 1: inverse.
// Shared memory: tw[N], exchange slots [N][W] float2.
// ---------------------------------------------------------------------------------
// Column-block width: the whole half row when it fits one block, else an even split.
constexpr int fcol_width(int N, int T) {
  const int NH = N / 2 + 1, maxt = N == 144 ? 448 : 512;
  for (int nb = 1;; ++nb) {
    const int W = (NH + nb - 1) / nb;
    if (W * T <= maxt && W * N * 8 <= 100 * 1024) return W;
  }
}
// Launch bounds of the column pass: the block's own threads, two blocks per SM up to N = 288
// (64 or 72 registers; one block, as the bound of 512 threads left it, kept half of the SM's
// warps idle: the two y passes of eight 288^3 meshes took 1.06 ms).
template <int N, int T>
struct FcolBounds {
  static constexpr int MAXT = (fcol_width(N, T) * T + 31) / 32 * 32, MINB = (N <= 288) ? 2 : 1;
};

template <int N, int R1, int R2, int AXIS, int MODE>
__global__ void __launch_bounds__(FcolBounds<N, TPS<R1, R2>::T>::MAXT, FcolBounds<N, TPS<R1, R2>::T>::MINB) k_fcol3(float2* __restrict__ c,
                                                  const float2* __restrict__ gtw, int W, int pc, int64_t plc) {
  constexpr int NH = N / 2 + 1;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* A = sm + N;  // exchange slots, [N][W]
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = gtw[i];
  const int64_t line = blockIdx.x;
  const int64_t b = line / N;
  const int o = (int)(line - b * N);
  const int kx0 = blockIdx.y * W;
  const int col = threadIdx.x % W, t = threadIdx.x / W;
  const bool live = kx0 + col < NH;
  const int64_t es = (AXIS == 1) ? pc : plc;
  float2* base = c + b * (int64_t)N * plc + (AXIS == 1 ? (int64_t)o * plc : (int64_t)o * pc) + kx0 + col;
  float2* Ac = A + col;
  __syncthreads();
  if (MODE != 1) {
    // ---- forward: n = R2*n1 + n2 ----
    if (t < R2) {
      float2 v[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = live ? base[(int64_t)(R2 * n1 + t) * es] : make_float2(0.f, 0.f);
      DFT<R1, N, -1>::run(v);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) Ac[(k1 * R2 + t) * W] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
    }
    __syncthreads();
    float2 w[R2];
    if (t < R1) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) w[n2] = Ac[(t * R2 + n2) * W];
      DFT<R2, N, -1>::run(w);
    }
    if (t < R1 && live) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) base[(int64_t)(t + R1 * k2) * es] = w[k2];
    }
  } else {
    // ---- inverse only, n = R1*n1 + n2: thread t = n2 < R1 loads x[R1*n1 + t] ----
    if (t < R1) {
      float2 w[R2];
#pragma unroll
      for (int n1 = 0; n1 < R2; ++n1) w[n1] = live ? base[(int64_t)(R1 * n1 + t) * es] : make_float2(0.f, 0.f);
      DFT<R2, N, +1>::run(w);
#pragma unroll
      for (int k1 = 0; k1 < R2; ++k1) Ac[(k1 * R1 + t) * W] = (k1 == 0) ? w[0] : cmul(w[k1], twid<+1>(tw, t * k1));
    }
    __syncthreads();
    if (t < R2) {
      float2 u[R1];
#pragma unroll
      for (int n2 = 0; n2 < R1; ++n2) u[n2] = Ac[(t * R1 + n2) * W];
      DFT<R1, N, +1>::run(u);
      if (live) {
#pragma unroll
        for (int k2 = 0; k2 < R1; ++k2) base[(int64_t)(t + R2 * k2) * es] = u[k2];
      }
    }
  }
}

// Row pitch of the half spectrum in the plane-compact layout; real rows have N values.
__host__ __device__ constexpr int plane_pc(int N) { return (N / 2 + 2) / 2 * 2; }

// ---------------------------------------------------------------------------------
// z pass with Green multiply for the plane sizes (N <= 144): forward z DFT, Green multiply,
// inverse, with a block kept on one line y and one group of columns while it walks the boxes, so the
// group's Green values are read once, and the next box's columns are copied into the other
// of two shared-memory stages (16-byte copies) while the current one is transformed.  A
// stage doubles as the exchange: the first step writes the slots it read.  Four barriers a
// box.  One line per block, loaded when the block starts, two blocks per SM, left
// the loads exposed: 4.63 ms for 512 boxes of 144^3, 3.1 ms now (1.9 at the copy bandwidth).
// Column groups start at even columns, for the 16-byte copies; the row pitch is even.
// Only planes [lo, hi) are written: the potential is read in the physical cells and three
// cells around them, and the rest of the padding is not needed (k_fyx3_c2r).
// ---------------------------------------------------------------------------------
template <int N, int R1, int R2>
struct ZLoop {
  static constexpr int T = TPS<R1, R2>::T, NH = N / 2 + 1;
  static constexpr int NCG = (NH * T + 447) / 448;
  static constexpr int STEP = NCG == 1 ? NH : (NH + NCG - 1) / NCG / 2 * 2;  // columns between groups
  static constexpr int LAST = NH - STEP * (NCG - 1), COLS = LAST > STEP ? LAST : STEP;
  static constexpr int WC = (COLS + 1) / 2 * 2;  // columns copied
  static_assert(STEP * (NCG - 1) + WC <= (NH + 1) / 2 * 2, "copies stay in the row");
  static constexpr int THREADS = (COLS * T + 31) / 32 * 32;
  static constexpr int MINB = N == 96 ? 3 : N >= 96 ? 2 : N >= 64 ? 4 : N >= 48 ? 6 : 8;
  static constexpr size_t SMEM = (size_t)N * 8 + (size_t)2 * N * WC * 8 + (size_t)N * COLS * 4;
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

template <int N, int R1, int R2>
__global__ void __launch_bounds__(ZLoop<N, R1, R2>::THREADS, ZLoop<N, R1, R2>::MINB)
    k_fz_loop(float2* __restrict__ c, const float* __restrict__ green, const float2* __restrict__ gtw, int64_t plc,
              int64_t nbox, int nsplit, int lo, int hi) {
  using Z = ZLoop<N, R1, R2>;
  constexpr int NH = Z::NH, WC = Z::WC, COLS = Z::COLS;
  extern __shared__ __align__(16) float2 sm[];
  float2* const stg = sm;                                             // [2][N][WC]
  float2* const tw = sm + 2 * N * WC;                                 // [N]
  float* const gr = reinterpret_cast<float*>(tw + N);                 // [N][COLS]
  const int line = blockIdx.x / nsplit, y = line / Z::NCG, g = line - y * Z::NCG, kx0 = g * Z::STEP;
  const int ncol = g == Z::NCG - 1 ? Z::LAST : Z::STEP;
  const int col = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const bool live = col < ncol;
  for (int i = threadIdx.x; i < N; i += Z::THREADS) tw[i] = gtw[i];
  for (int i = threadIdx.x; i < N * COLS; i += Z::THREADS) {
    const int z = i / COLS, q = i - z * COLS;
    gr[i] = q < ncol ? green[((int64_t)z * N + y) * NH + kx0 + q] : 0.f;
  }
  auto base = [&](int64_t b) { return c + b * (int64_t)N * plc + y * plane_pc(N) + kx0; };
  auto issue = [&](int64_t b, int st) {
    const float2* src = base(b);
    float2* dst = stg + st * N * WC;
    for (int i = threadIdx.x; i < N * (WC / 2); i += Z::THREADS) {
      const int z = i / (WC / 2), q = 2 * (i - z * (WC / 2));
      cp_async16(dst + z * WC + q, src + (int64_t)z * plc + q);
    }
  };
  int64_t b = blockIdx.x - (int64_t)line * nsplit;
  if (b < nbox) issue(b, 0);
  cp_async_commit();
  for (int st = 0; b < nbox; b += nsplit, st ^= 1) {
    cp_async_wait_all();
    __syncthreads();  // the box's columns are in; the other stage is free
    if (b + nsplit < nbox) issue(b + nsplit, st ^ 1);
    cp_async_commit();
    float2* const A = stg + st * N * WC + col;
    if (t < R2) {  // forward, n = R2*n1 + n2, thread t = n2
      float2 v[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = A[(R2 * n1 + t) * WC];
      DFT<R1, N, -1>::run(v);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) A[(k1 * R2 + t) * WC] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
    }
    __syncthreads();
    float2 w[R2];
    if (t < R1) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) w[n2] = A[(t * R2 + n2) * WC];
      DFT<R2, N, -1>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {  // Green at kz = t + R1*k2
        const float gv = gr[(t + R1 * k2) * COLS + col];
        w[k2] = make_float2(w[k2].x * gv, w[k2].y * gv);
      }
      // inverse, n = R1*n1 + n2 with n2 = t, n1 = k2
      DFT<R2, N, +1>::run(w);
#pragma unroll
      for (int k1 = 1; k1 < R2; ++k1) w[k1] = cmul(w[k1], twid<+1>(tw, t * k1));
    }
    __syncthreads();
    if (t < R1) {
#pragma unroll
      for (int k1 = 0; k1 < R2; ++k1) A[(k1 * R1 + t) * WC] = w[k1];
    }
    __syncthreads();
    if (t < R2) {
      float2 u[R1];
#pragma unroll
      for (int n2 = 0; n2 < R1; ++n2) u[n2] = A[(t * R1 + n2) * WC];
      DFT<R1, N, +1>::run(u);
      if (live) {
        float2* out = base(b) + col;
#pragma unroll
        for (int k2 = 0; k2 < R1; ++k2) {
          const int z = t + R2 * k2;
          if (z >= lo && z < hi) out[(int64_t)z * plc] = u[k2];
        }
      }
    }
  }
}

// Blocks per line of k_fz_loop: enough to fill the chip once, and else about 24 boxes a block,
// which hides a block's start (its Green values, the first copy) and still deals the boxes
// out evenly (512 boxes of 144^3: 3.28 ms with one block a line, 3.14 so; 64 boxes: 0.74 ms
// with a box a block, 0.43 so).
inline int fz_loop_split(int lines, int resident, int64_t nbox) {
  const int64_t s = std::max<int64_t>(std::min<int64_t>(nbox, resident / lines), nbox / 24);
  return (int)std::max<int64_t>(1, s);
}

// ---------------------------------------------------------------------------------
// Persistent z pass with Green multiply for N > 144 (forward z DFT,
// Green multiply, inverse), one item = W columns of one line (box b, row y), looped over
// by a grid of a few blocks per SM.  The column data and Green values of the next item
// are copied into the other of two shared-memory stages with cp.async while the current
// one is transformed, so the loads stay in flight; the current stage doubles as the
// exchange slots.  Items: it = (b*N + y)*ncg + column group.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

__host__ __device__ constexpr int fzs_maxt(int N) { return N <= 192 ? 320 : 512; }

template <int N, int R1, int R2>
__global__ void __launch_bounds__(fzs_maxt(N), (N <= 192 ? 2 : 1)) k_fz_stream(float2* __restrict__ c, const float* __restrict__ green,
                                                            const float2* __restrict__ gtw, int W, int ncg, int pc,
                                                            int64_t plc, int64_t nitems) {
  constexpr int T = TPS<R1, R2>::T, NH = N / 2 + 1;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* stg = sm + N;                                          // [2][N][W] float2
  float* gst = reinterpret_cast<float*>(stg + (size_t)2 * N * W);  // [2][N][W] float
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = gtw[i];
  const int col = threadIdx.x % W, t = threadIdx.x / W;
  const bool thr = t < T;
  auto issue = [&](int64_t it, int st) {  // copy item `it` into stage `st`; always commits a group
    if (it < nitems && thr) {
      const int64_t line = it / ncg;
      const int kx = (int)(it - line * ncg) * W + col;
      if (kx < NH) {
        const int64_t b = line / N;
        const int y = (int)(line - b * N);
        const float2* base = c + b * (int64_t)N * plc + (int64_t)y * pc + kx;
        const float* gb = green + (int64_t)y * NH + kx;
        float2* ds = stg + (size_t)st * N * W + col;
        float* dg = gst + (size_t)st * N * W + col;
#pragma unroll 4
        for (int z = t; z < N; z += T) {
          cp_async8(ds + (size_t)z * W, base + (int64_t)z * plc);
          cp_async4(dg + (size_t)z * W, gb + (int64_t)z * N * NH);
        }
      }
    }
    cp_async_commit();
  };
  int64_t it = blockIdx.x;
  issue(it, 0);
  for (int s = 0; it < nitems; it += gridDim.x, s ^= 1) {
    issue(it + gridDim.x, s ^ 1);
    cp_async_wait_one();  // this thread's copies of item `it` have landed
    __syncthreads();      // and everyone's
    const int64_t line = it / ncg;
    const int kx = (int)(it - line * ncg) * W + col;
    const bool live = thr && kx < NH;
    const int64_t b = line / N;
    const int y = (int)(line - b * N);
    float2* out = c + b * (int64_t)N * plc + (int64_t)y * pc + kx;
    float2* Ac = stg + (size_t)s * N * W + col;
    const float* Gc = gst + (size_t)s * N * W + col;
    // forward, n = R2*n1 + n2: thread t = n2
    float2 v[R1];
    if (thr && t < R2) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = live ? Ac[(R2 * n1 + t) * W] : make_float2(0.f, 0.f);
      DFT<R1, N, -1>::run(v);
    }
    __syncthreads();  // the stage's data are in registers; its slots become the exchange
    if (thr && t < R2) {
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) Ac[(k1 * R2 + t) * W] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
    }
    __syncthreads();
    float2 w[R2];
    if (thr && t < R1) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) w[n2] = Ac[(t * R2 + n2) * W];
      DFT<R2, N, -1>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {  // Green at kz = t + R1*k2
        const float gv = Gc[(t + R1 * k2) * W];
        w[k2] = make_float2(w[k2].x * gv, w[k2].y * gv);
      }
      // inverse, n = R1*n1 + n2 with n2 = t, n1 = k2
      DFT<R2, N, +1>::run(w);
#pragma unroll
      for (int k1 = 1; k1 < R2; ++k1) w[k1] = cmul(w[k1], twid<+1>(tw, t * k1));
    }
    __syncthreads();
    if (thr && t < R1) {
#pragma unroll
      for (int k1 = 0; k1 < R2; ++k1) Ac[(k1 * R1 + t) * W] = w[k1];
    }
    __syncthreads();
    if (thr && t < R2) {
      float2 u[R1];
#pragma unroll
      for (int n2 = 0; n2 < R1; ++n2) u[n2] = Ac[(t * R1 + n2) * W];
      DFT<R1, N, +1>::run(u);
      if (live) {
#pragma unroll
        for (int k2 = 0; k2 < R1; ++k2) out[(int64_t)(t + R2 * k2) * plc] = u[k2];
      }
    }
    __syncthreads();  // this stage is free for the copy issued next iteration
  }
  cp_async_wait_all();
}

// Width and count of the column groups of k_fz_stream: two blocks per SM within
// ~100 KB of shared memory each, at most fzs_maxt(N) threads.
__host__ inline void fz_stream_shape(int N, int T, int& W, int& ncg) {
  const int NH = N / 2 + 1;
  int wmax = (int)((100 * 1024 - 8 * N) / (2 * 12 * N));
  wmax = std::min(wmax, fzs_maxt(N) / T);
  ncg = (NH + wmax - 1) / wmax;
  W = (NH + ncg - 1) / ncg;
}
__host__ inline size_t fz_stream_smem(int N, int W) { return (size_t)N * 8 + (size_t)2 * N * W * 12; }

// ---------------------------------------------------------------------------------
// X' pass, c2r, times `inv`: the mirror image of k_fx_r2c.  In place (complex rows pc -> real
// rows pf).
// ---------------------------------------------------------------------------------
template <int N, int R1, int R2>
__global__ void __launch_bounds__(FX_T, FxShape<N, R1, R2>::MINB) k_fx_c2r(const float2* c, float* r, int64_t nrows,
                                                                         const float2* __restrict__ gtw, float inv, int pc,
                                                                         int pf) {
  using FX = FxShape<N, R1, R2>;
  constexpr int T = FX::T, NH = N / 2 + 1;
  extern __shared__ float2 sm[];
  float2* tw = sm;
  for (int i = threadIdx.x; i < N; i += FX_T) tw[i] = gtw[i];
  const int s = threadIdx.x / T, t = threadIdx.x % T;
  const int64_t row = ((int64_t)blockIdx.x * FX::S + s) * 2;
  const bool act = s < FX::S && row < nrows, two = row + 1 < nrows;
  float2* Zr = sm + N + (s < FX::S ? s : 0) * N;
  float2 v[R1];
  if (act && t < R2) {
    const float2* c0 = c + row * pc;
    const float2* c1 = c0 + (two ? pc : 0);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {  // the Hermitian extension of both rows, packed
      const int x = R2 * n1 + t, k = x < NH ? x : N - x;
      float2 a0 = c0[k], a1 = c1[k];
      if (!two) a1 = make_float2(0.f, 0.f);
      if (k == 0 || 2 * k == N) {
        a0.y = 0.f;
        a1.y = 0.f;
      }
      if (x >= NH) {
        a0.y = -a0.y;
        a1.y = -a1.y;
      }
      v[n1] = make_float2(a0.x - a1.y, a0.y + a1.x);
    }
  }
  __syncthreads();  // the table, and every row is read
  if (act && t < R2) {
    DFT<R1, N, +1>::run(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) Zr[skew<R1, R2>(k1, t)] = (k1 == 0) ? v[0] : cmul(v[k1], twid<+1>(tw, t * k1));
  }
  __syncthreads();
  if (act && t < R1) {
    float2 w[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) w[n2] = Zr[skew<R1, R2>(t, n2)];
    DFT<R2, N, +1>::run(w);
    float* r0 = r + row * pf + t;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      r0[R1 * k2] = __fmul_rn(w[k2].x, inv);
      if (two) r0[pf + R1 * k2] = __fmul_rn(w[k2].y, inv);
    }
  }
}

// ---------------------------------------------------------------------------------
// Plane kernels with register-resident sequences (N <= 144, T = max(R1,R2) <= 16).
// Rows run warp-synchronously: each warp holds 32/L sequences (T of L lanes each), loads
// them straight from global memory and exchanges through a skewed
// slot layout (slot(k1, n2) = k1*R2 + (n2 + k1) mod R2) that is free of bank conflicts
// in both directions.  Columns run as in k_fcol3, W columns by T threads per round.
// The r2c unpack and the c2r Hermitian pack happen on the fly inside the other phase,
// and column results go straight to global memory.
// ---------------------------------------------------------------------------------
// Launch shape of the plane kernels for one N.  A sequence takes T = max(R1, R2) threads; a
// round of the column phase runs W columns, the fewest equal rounds that fit 448 threads, and
// the block has just the threads of one round.  The row phase gives a sequence L = 4, 8 or 16
// lanes, the smallest that hold T, so a warp runs 32/L of them.  Blocks per SM: about 900
// threads for N >= 96, whose 12- and 16-point DFTs want 72 registers, and up to 1300 for the
// smaller ones, which are bound by latency (N = 48, 4096 boxes, both passes: 5.2 ms with 448
// threads and 16 lanes a sequence, two blocks per SM).
template <int N, int R1, int R2>
struct PlaneShape {
  static constexpr int T = TPS<R1, R2>::T, NH = N / 2 + 1;
  static constexpr int L = T <= 4 ? 4 : T <= 8 ? 8 : 16;
  static constexpr int ROUNDS = (NH * T + 447) / 448, W = (NH + ROUNDS - 1) / ROUNDS;
  static constexpr int THREADS = (W * T + 31) / 32 * 32;
  static constexpr int MINB = N == 96 ? 3 : N >= 96 ? 2 : N >= 64 ? 4 : N >= 48 ? 6 : 8;
};

template <int N>
struct Plane3Sm {
  static constexpr int NH = N / 2 + 1;
  // forward: packed rows Z[N/2][N] + scratch for the self-conjugate columns 0, N/2
  static constexpr size_t FWD = (size_t)(N + (N / 2) * N + 2 * N) * 8;
  // inverse: half spectrum H[N][NH]
  static constexpr size_t INV = (size_t)(N + N * NH) * 8;
};

template <int N, int R1, int R2, typename IN>
__global__ void __launch_bounds__(PlaneShape<N, R1, R2>::THREADS, PlaneShape<N, R1, R2>::MINB) k_fxy3_r2c(const IN* __restrict__ r, float2* __restrict__ c,
                                                               const float2* __restrict__ gtw, float scale, int64_t plr,
                                                               int64_t plc) {
  constexpr int T = TPS<R1, R2>::T, NH = N / 2 + 1, NP = N / 2, PC = plane_pc(N);
  static_assert(T <= 16, "two sequences per warp");
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* Z = sm + N;  // packed rows, pitch N; then 2N exchange slots for columns 0 and N/2
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = gtw[i];
  const int64_t plane = blockIdx.x;
  const IN* rp = r + plane * plr;
  float2* cp = c + plane * plc;
  __syncthreads();
  {  // ---- rows: packed pairs (2p, 2p+1) as re/im ----
    constexpr int L = PlaneShape<N, R1, R2>::L;
    const int lane = threadIdx.x & 31, t = lane % L;
    const int g = (threadIdx.x >> 5) * (32 / L) + lane / L;
    constexpr int ngr = PlaneShape<N, R1, R2>::THREADS / L;
    for (int p0 = 0; p0 < NP; p0 += ngr) {
      const int p = p0 + g;
      const bool act = p < NP;
      float2* Zr = Z + (size_t)(act ? p : 0) * N;
      if (act && t < R2) {
        float2 v[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) {
          const int x = R2 * n1 + t;
          const IN a = rp[(2 * p) * N + x], b = rp[(2 * p + 1) * N + x];
          float fa, fb;
          if (sizeof(IN) == 8) {
            fa = (float)((double)(long long)a * 9.094947017729282e-13);
            fb = (float)((double)(long long)b * 9.094947017729282e-13);
          } else {
            fa = (float)a;
            fb = (float)b;
          }
          v[n1] = make_float2(__fmul_rn(fa, scale), __fmul_rn(fb, scale));
        }
        DFT<R1, N, -1>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) Zr[skew<R1, R2>(k1, t)] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
      }
      __syncwarp();
      float2 w[R2];
      if (act && t < R1) {
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) w[n2] = Zr[skew<R1, R2>(t, n2)];
        DFT<R2, N, -1>::run(w);
      }
      __syncwarp();
      if (act && t < R1) {
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) Zr[t + R1 * k2] = w[k2];
      }
      __syncwarp();
    }
  }
  __syncthreads();
  {  // ---- columns kx of the half spectrum, unpacked on the fly ----
    constexpr int W = PlaneShape<N, R1, R2>::W;
    const int col = threadIdx.x % W, t = threadIdx.x / W;
    for (int kx0 = 0; kx0 < NH; kx0 += W) {
      const int kx = kx0 + col;
      const bool act = t < T && kx < NH && col < W;
      const int kc = (N - kx) % N;
      // exchange slot s of column kx (columns kx and N-kx of Z are read only by column
      // kx): slot s < NP at lo + s*st, else at hi + s*st; the self-conjugate columns 0
      // and N/2 use the contiguous scratch S.
      const bool selfc = (kx == 0) || (2 * kx == N);
      const int st = selfc ? 1 : N;
      // offsets from Z (S follows Z): slot s at Z[lo + s*st] for s < NP, else Z[hi + s*st]
      const int lo = selfc ? NP * N + (kx ? N : 0) : kx;
      const int hi = selfc ? lo : kc - NP * N;
      float2 v[R1];
      if (act && t < R2) {
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) {
          const int y = R2 * n1 + t;
          const float2* zr = Z + (size_t)(y >> 1) * N;
          const float2 z = zr[kx], zc = zr[kc];
          v[n1] = (y & 1) ? make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x))
                          : make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
        }
        DFT<R1, N, -1>::run(v);
      }
      __syncthreads();  // all unpack reads of this round are done
      if (act && t < R2) {
        // s = k1*R2 + t < NP exactly when k1 < R1/2 (R1 even) -- resolved per unrolled k1
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
          const int sl = k1 * R2 + t;
          const int b = (k1 * R2 + R2 - 1 < NP) ? lo : ((k1 * R2 >= NP) ? hi : (sl < NP ? lo : hi));
          Z[b + sl * st] = (k1 == 0) ? v[0] : cmul(v[k1], twid<-1>(tw, t * k1));
        }
      }
      __syncthreads();
      if (act && t < R1) {
        float2 w[R2];
        const int s0 = t * R2;
        const bool whole = (s0 + R2 - 1 < NP) || (s0 >= NP);  // R1 even: always
        const int b = (s0 < NP) ? lo : hi;
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
          const int sl = s0 + n2;
          w[n2] = Z[(whole ? b : (sl < NP ? lo : hi)) + sl * st];
        }
        DFT<R2, N, -1>::run(w);
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) cp[(t + R1 * k2) * PC + kx] = w[k2];
      }
    }
  }
}

// Planes and rows [lo, hi) of each box (the part of the potential that is read; the whole box
// with 0, N): at N = 48 that leaves out two fifths of the pass.
template <int N, int R1, int R2>
__global__ void __launch_bounds__(PlaneShape<N, R1, R2>::THREADS, PlaneShape<N, R1, R2>::MINB) k_fyx3_c2r(const float2* __restrict__ c, float* __restrict__ r,
                                                               const float2* __restrict__ gtw, float inv, int64_t plc,
                                                               int64_t plf, int lo, int hi) {
  constexpr int T = TPS<R1, R2>::T, NH = N / 2 + 1, PC = plane_pc(N);
  static_assert(T <= 16, "two sequences per warp");
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* H = sm + N;  // half spectrum after the inverse y transforms, [N][NH]
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = gtw[i];
  const int64_t box = blockIdx.x / (unsigned)(hi - lo), plane = box * N + lo + (int)(blockIdx.x - box * (hi - lo));
  const float2* cp = c + plane * plc;
  float* rp = r + plane * plf;
  __syncthreads();
  {  // ---- inverse y transforms of the columns kx, n = R2*n1 + n2 ----
    constexpr int W = PlaneShape<N, R1, R2>::W;
    const int col = threadIdx.x % W, t = threadIdx.x / W;
    for (int kx0 = 0; kx0 < NH; kx0 += W) {
      const int kx = kx0 + col;
      const bool act = t < T && kx < NH && col < W;
      float2* Hc = H + kx;  // column kx: N slots, read and written only by column kx
      if (act && t < R2) {
        float2 v[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) v[n1] = cp[(R2 * n1 + t) * PC + kx];
        DFT<R1, N, +1>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) Hc[(k1 * R2 + t) * NH] = (k1 == 0) ? v[0] : cmul(v[k1], twid<+1>(tw, t * k1));
      }
      __syncthreads();
      float2 w[R2];
      if (act && t < R1) {
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) w[n2] = Hc[(t * R2 + n2) * NH];
        DFT<R2, N, +1>::run(w);
      }
      __syncthreads();  // every read of the column's slots is done
      if (act && t < R1) {
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) Hc[(t + R1 * k2) * NH] = w[k2];
      }
    }
  }
  __syncthreads();
  {  // ---- rows: pack (2p, 2p+1) over the Hermitian extension, inverse x transform ----
    constexpr int L = PlaneShape<N, R1, R2>::L;
    const int lane = threadIdx.x & 31, t = lane % L;
    const int g = (threadIdx.x >> 5) * (32 / L) + lane / L;
    constexpr int ngr = PlaneShape<N, R1, R2>::THREADS / L;
    const int p1 = (hi + 1) / 2;
    for (int p0 = lo / 2; p0 < p1; p0 += ngr) {
      const int p = p0 + g;
      const bool act = p < p1;
      float2* H0 = H + (size_t)(act ? 2 * p : 0) * NH;  // rows 2p, 2p+1: 2*NH >= N contiguous slots
      const float2* H1 = H0 + NH;
      float2 v[R1];
      if (act && t < R2) {
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) {
          const int x = R2 * n1 + t;
          const int k = (x < NH) ? x : N - x;
          float2 a0 = H0[k], a1 = H1[k];
          if (k == 0 || 2 * k == N) {
            a0.y = 0.f;
            a1.y = 0.f;
          }
          if (x >= NH) {
            a0.y = -a0.y;
            a1.y = -a1.y;
          }
          v[n1] = make_float2(a0.x - a1.y, a0.y + a1.x);
        }
        DFT<R1, N, +1>::run(v);
      }
      __syncwarp();  // the pack reads of rows 2p, 2p+1 are done
      if (act && t < R2) {
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) H0[skew<R1, R2>(k1, t)] = (k1 == 0) ? v[0] : cmul(v[k1], twid<+1>(tw, t * k1));
      }
      __syncwarp();
      if (act && t < R1) {
        float2 w[R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) w[n2] = H0[skew<R1, R2>(t, n2)];
        DFT<R2, N, +1>::run(w);
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
          const int x = t + R1 * k2;
          rp[(2 * p) * N + x] = __fmul_rn(w[k2].x, inv);
          rp[(2 * p + 1) * N + x] = __fmul_rn(w[k2].y, inv);
        }
      }
      __syncwarp();
    }
  }
}

}  // namespace f2
}  // namespace cube
