// Differentiable particle-mesh step and its hand-written adjoint (the PyTorch binding
// cube_nu_b200/adjoint.py wraps these behind torch.autograd.Function).  Included by
// cube_gpu.cu after kernels.cuh.
//
// The forward is one PM level on a periodic n^3 mesh in fine-cell units, with the
// reference's PM pieces: TSC mass assignment with the cell-centred convention of
// particle_mesh.f90:56-62 (cells floor(x)-1 .. floor(x)+1, l = x - floor(x)), the Green
// table of Green/Green.f90 applied between a forward and an inverse FFT, the 4-point
// gradient of the potential (particle_mesh.f90:224-247) and TSC interpolation of the
// force, in the KDK order of main.f90 (drift, then kick with dv = F * a_mid * dt/(6 pi)).
// Positions are real (not ZIPX codes), so the step is differentiable.
//
// Adjoints, for a cotangent u_i of the particle forces F_i = sum_c W(x_i - c) Fm(c),
// Fm = grad_h phi, phi = Gconv(rho), rho(c) = m sum_j W(x_j - c):
//   d(u.F)/dx_k = sum_c dW(x_k - c) (u_k . Fm(c))            (interpolation weights)
//               + m sum_c dW(x_k - c) psi(c)                 (mass assignment weights)
//   psi = Gconv(grad_h^T lamF),  lamF(c) = sum_i W(x_i - c) u_i
// Gconv is symmetric (a real Green table), grad_h^T = -grad_h (antisymmetric stencil).
#pragma once
#include "kernels.cuh"

namespace cube {

// 1-D TSC weights and their derivatives at x (fine units): cells fl-1, fl, fl+1.
__device__ __forceinline__ int dpm_w(float x, float w[3], float dw[3]) {
  const float fl = floorf(x);
  const float l = x - fl;
  const float a = 1.f - l;
  w[0] = 0.5f * a * a;
  w[2] = 0.5f * l * l;
  w[1] = 1.f - w[0] - w[2];
  dw[0] = -a;
  dw[2] = l;
  dw[1] = a - l;
  return (int)fl;
}

// The mesh cells floor(x)-1 .. floor(x)+1 of a position, wrapped (one division).
__device__ __forceinline__ void dpm_cells(int fl, int n, int c[3]) {
  const int f = wrapi(fl, n);
  c[0] = wrap1(f - 1, n);
  c[1] = f;
  c[2] = wrap1(f + 1, n);
}

// rho += m * W, into a mesh with row pitch pr and plane pitch pl (floats).  Bound by the L2
// reductions.  PAIR (dpm_pairs): the three cells of a row are two 8-byte reductions of aligned
// cells, the fourth value zero, instead of three of 4 bytes: 18 a particle for 27 (0.100 ms for
// 2^21 particles on 256^3 cells, 0.132 one by one).  A row that wraps has its cells one by one.
template <bool PAIR>
__global__ void k_dpm_deposit(int n, int64_t np, const float* __restrict__ x, float m, float* __restrict__ rho, int pr,
                              int64_t pl) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  float w[3][3], dw[3];
  int f[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) dpm_cells(dpm_w(x[3 * i + d], w[d], dw), n, f[d]);
  const bool wraps = f[0][2] != f[0][0] + 2, odd = f[0][0] & 1;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int64_t z = (int64_t)f[2][c] * pl;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int64_t y = (int64_t)f[1][b] * pr;
      float v[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) v[a] = m * w[0][a] * w[1][b] * w[2][c];
      if (PAIR && !wraps) {  // n even: the pairs end at cell n - 1 at most
        float2* const p = reinterpret_cast<float2*>(&rho[z + y + (f[0][0] & ~1)]);
        atomicAdd(p, odd ? make_float2(0.f, v[0]) : make_float2(v[0], v[1]));
        atomicAdd(p + 1, odd ? make_float2(v[1], v[2]) : make_float2(v[2], 0.f));
      } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) atomicAdd(&rho[z + y + f[0][a]], v[a]);
      }
    }
  }
}

// Cells 2k and 2k+1 of every row are one aligned 8-byte word.
inline bool dpm_pairs(int n, const float* rho, int pr, int64_t pl) {
  return n % 2 == 0 && pr % 2 == 0 && pl % 2 == 0 && (reinterpret_cast<uintptr_t>(rho) & 7) == 0;
}

// F_i = sum_c W Fm(c) (Fm: float4 per cell, dense, x fastest); then the KDK kick
// v += K F and, with D != 0, the next drift is not applied here.
__global__ void k_dpm_kick(int n, int64_t np, const float* __restrict__ x, const float4* __restrict__ fm, float K,
                           float* __restrict__ v) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  float w[3][3], dw[3];
  int f[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) dpm_cells(dpm_w(x[3 * i + d], w[d], dw), n, f[d]);
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int64_t z = (int64_t)f[2][c] * n * n;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int64_t y = (int64_t)f[1][b] * n;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float4 F = __ldg(&fm[z + y + f[0][a]]);
        const float ww = w[0][a] * w[1][b] * w[2][c];
        s0 += ww * F.x;
        s1 += ww * F.y;
        s2 += ww * F.z;
      }
    }
  }
  v[3 * i] += K * s0;
  v[3 * i + 1] += K * s1;
  v[3 * i + 2] += K * s2;
}

// x += D v, wrapped into [0, n).
__global__ void k_dpm_drift(int n, int64_t np3, float* __restrict__ x, const float* __restrict__ v, float D) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np3) return;
  float y = x[i] + D * v[i];
  const float fn = (float)n;
  y -= fn * floorf(y / fn);
  if (y >= fn) y -= fn;  // rounding of y / fn just below an integer
  x[i] = y;
}

// lamF(c) += sum_i W(x_i - c) u_i (float4 mesh, dense, x fastest; .w unused).  One 16-byte
// vector reduction per cell: three 4-byte ones took 0.74 ms for 128^3 particles.
__global__ void k_dpm_deposit_vec(int n, int64_t np, const float* __restrict__ x, const float* __restrict__ u,
                                  float4* __restrict__ lam) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  float w[3][3], dw[3];
  int f[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) dpm_cells(dpm_w(x[3 * i + d], w[d], dw), n, f[d]);
  const float u0 = u[3 * i], u1 = u[3 * i + 1], u2 = u[3 * i + 2];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int64_t z = (int64_t)f[2][c] * n * n;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int64_t y = (int64_t)f[1][b] * n;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float ww = w[0][a] * w[1][b] * w[2][c];
        atomicAdd(&lam[z + y + f[0][a]], make_float4(ww * u0, ww * u1, ww * u2, 0.f));
      }
    }
  }
}

// s(c) = (grad_h^T lamF)(c) = sum_d sum_o w_o lamF_d(c - o e_d), o in {-2,-1,1,2}, the
// transpose of the 4-point gradient; written into a mesh with row pitch pr, plane pl.
// Grid of force_grid.
__global__ void __launch_bounds__(FORCE_T) k_dpm_grad_t(int n, const float4* __restrict__ lam, float* __restrict__ s,
                                                        int pr, int64_t pl) {
  const int x = blockIdx.x * FORCE_T + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= n) return;
  const float w[4] = {(CUBE_W_ALPHA - 1.f) / 4.f, -CUBE_W_ALPHA / 2.f, CUBE_W_ALPHA / 2.f, (1.f - CUBE_W_ALPHA) / 4.f};
  const int o[4] = {-2, -1, 1, 2};
  auto L = [&](int a, int b, int c) { return reinterpret_cast<const float*>(lam + ((int64_t)c * n + b) * n + a); };
  float t = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    t += w[k] * __ldg(L(wrap1(x - o[k], n), y, z));
    t += w[k] * __ldg(L(x, wrap1(y - o[k], n), z) + 1);
    t += w[k] * __ldg(L(x, y, wrap1(z - o[k], n)) + 2);
  }
  s[(int64_t)z * pl + (int64_t)y * pr + x] = t;
}

// gx_k += sum_c dW(x_k - c) (u_k . Fm(c) + m psi(c)) over the 27 TSC cells; u or psi may be
// null (density adjoint: u = null, psi = lam with m the mass).
__global__ void k_dpm_grad_gather(int n, int64_t np, const float* __restrict__ x, const float* __restrict__ u,
                                  const float4* __restrict__ fm, const float* __restrict__ psi, int pr, int64_t pl,
                                  float m, float* __restrict__ gx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  float w[3][3], dw[3][3];
  int f[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) dpm_cells(dpm_w(x[3 * i + d], w[d], dw[d]), n, f[d]);
  const float u0 = u ? u[3 * i] : 0.f, u1 = u ? u[3 * i + 1] : 0.f, u2 = u ? u[3 * i + 2] : 0.f;
  float g0 = 0.f, g1 = 0.f, g2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int zz = f[2][c];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int yy = f[1][b];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int xx = f[0][a];
        float val = 0.f;
        if (u) {
          const float4 F = __ldg(&fm[((int64_t)zz * n + yy) * n + xx]);
          val = u0 * F.x + u1 * F.y + u2 * F.z;
        }
        if (psi) val += m * __ldg(&psi[(int64_t)zz * pl + (int64_t)yy * pr + xx]);
        g0 += dw[0][a] * w[1][b] * w[2][c] * val;
        g1 += w[0][a] * dw[1][b] * w[2][c] * val;
        g2 += w[0][a] * w[1][b] * dw[2][c] * val;
      }
    }
  }
  gx[3 * i] += g0;
  gx[3 * i + 1] += g1;
  gx[3 * i + 2] += g2;
}

}  // namespace cube
