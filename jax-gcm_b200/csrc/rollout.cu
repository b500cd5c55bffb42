// rollout.cu -- the vector updates of a column rollout and of its adjoint (rollout.py):
//   spd_rollout_step     x_{n+1} = x_n + dt f_n, the four evolved planes;
//   spd_rollout_reverse  xbar_n = xbar_{n+1} + g, the cotangent dt xbar_n of the step before, and
//                        the sums of the fixed fields' and the parameters' gradients.
// One launch each, one field per blockIdx.y, 128-bit accesses where every plane allows them.  On
// the grids a rollout runs on these are bound by latency: three multi-tensor launches of 8-10 us
// each did the reverse update of a T42 step with 8 levels, and one the forward update; a launch here
// takes 2 us (a 12-step T42 rollout with its gradient 1,790 -> 1,380 us).  The step is a fused
// multiply-add, the rounding of a multi-tensor add with a factor.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "speedy_b200.h"

namespace {

constexpr int kThreads = 256;

struct StepArgs {
  const float *x[4], *f[4];
  float* out[4];
  int64_t n;
  float dt;
};

struct ReverseArgs {
  const float *xbar[4], *g[4];
  float *out[4], *ct[4];
  const float *g_phi, *g_psa, *g_par;
  float *phi, *psa, *par;
  int64_t n, columns;
  float dt;
};

__device__ __forceinline__ float step1(float x, float f, float dt) { return fmaf(dt, f, x); }
__device__ __forceinline__ float4 step1(float4 x, float4 f, float dt) {
  return make_float4(step1(x.x, f.x, dt), step1(x.y, f.y, dt), step1(x.z, f.z, dt),
                     step1(x.w, f.w, dt));
}
__device__ __forceinline__ float add1(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float4 add1(float4 a, float4 b) {
  return make_float4(add1(a.x, b.x), add1(a.y, b.y), add1(a.z, b.z), add1(a.w, b.w));
}
__device__ __forceinline__ float mul1(float a, float s) { return __fmul_rn(a, s); }
__device__ __forceinline__ float4 mul1(float4 a, float s) {
  return make_float4(mul1(a.x, s), mul1(a.y, s), mul1(a.z, s), mul1(a.w, s));
}

// n: elements of V per plane.
template <class V>
__global__ void __launch_bounds__(kThreads) step_planes(const __grid_constant__ StepArgs A,
                                                        int64_t n) {
  const int j = blockIdx.y;
  const V* x = reinterpret_cast<const V*>(A.x[j]);
  const V* f = reinterpret_cast<const V*>(A.f[j]);
  V* out = reinterpret_cast<V*>(A.out[j]);
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kThreads)
    out[i] = step1(x[i], f[i], A.dt);
}

template <class V>
__global__ void __launch_bounds__(kThreads) reverse_planes(const __grid_constant__ ReverseArgs A,
                                                           int64_t n) {
  const int j = blockIdx.y;
  const int64_t first = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  if (j < 4) {
    const V* xb = reinterpret_cast<const V*>(A.xbar[j]);
    const V* g = reinterpret_cast<const V*>(A.g[j]);
    V* out = reinterpret_cast<V*>(A.out[j]);
    V* ct = reinterpret_cast<V*>(A.ct[j]);
    for (int64_t i = first; i < n; i += stride) {
      const V s = add1(xb[i], g[i]);
      out[i] = s;
      ct[i] = mul1(s, A.dt);
    }
  } else if (j == 4) {
    const V* g = reinterpret_cast<const V*>(A.g_phi);
    V* phi = reinterpret_cast<V*>(A.phi);
    for (int64_t i = first; i < n; i += stride) phi[i] = add1(phi[i], g[i]);
  } else {
    for (int64_t i = first; i < A.columns; i += stride) A.psa[i] = add1(A.psa[i], A.g_psa[i]);
    if (first < SPD_NUM_DIFF_PARAMS) A.par[first] = add1(A.par[first], A.g_par[first]);
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Blocks per plane: enough for one element per thread, at most 1,024 (grid-stride beyond).
unsigned blocks(int64_t n) {
  return (unsigned)std::min<int64_t>((n + kThreads - 1) / kThreads, 1024);
}

int shape(int32_t kx, int64_t columns, int64_t* n) {
  if (kx < 1 || kx > SPD_MAX_KX) return SPD_ERR_KX;
  if (columns <= 0 || columns > (1 << 30)) return SPD_ERR_SHAPE;
  *n = kx * columns;
  return SPD_OK;
}

}  // namespace

namespace spd {
int preload_rollout() {
  cudaFuncAttributes a;
  bool ok = cudaFuncGetAttributes(&a, step_planes<float>) == cudaSuccess;
  ok &= cudaFuncGetAttributes(&a, step_planes<float4>) == cudaSuccess;
  ok &= cudaFuncGetAttributes(&a, reverse_planes<float>) == cudaSuccess;
  ok &= cudaFuncGetAttributes(&a, reverse_planes<float4>) == cudaSuccess;
  return ok ? SPD_OK : SPD_ERR_CUDA;
}
}  // namespace spd

extern "C" {

int spd_rollout_step(int32_t kx, int64_t columns, float dt, const spd_cotangents_t* x,
                     const spd_cotangents_t* f, const spd_planes_t* out, void* stream) {
  if (!x || !f || !out) return SPD_ERR_NULL;
  StepArgs A = {{x->u_wind, x->v_wind, x->temperature, x->specific_humidity},
                {f->u_wind, f->v_wind, f->temperature, f->specific_humidity},
                {out->u_wind, out->v_wind, out->temperature, out->specific_humidity},
                0, dt};
  const int rc = shape(kx, columns, &A.n);
  if (rc != SPD_OK) return rc;
  bool vec = A.n % 4 == 0;
  for (int j = 0; j < 4; ++j) {
    if (!A.x[j] || !A.f[j] || !A.out[j]) return SPD_ERR_NULL;
    vec = vec && aligned16(A.x[j]) && aligned16(A.f[j]) && aligned16(A.out[j]);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (vec)
    step_planes<float4><<<dim3(blocks(A.n / 4), 4), kThreads, 0, st>>>(A, A.n / 4);
  else
    step_planes<float><<<dim3(blocks(A.n), 4), kThreads, 0, st>>>(A, A.n);
  return cudaGetLastError() == cudaSuccess ? SPD_OK : SPD_ERR_CUDA;
}

int spd_rollout_reverse(int32_t kx, int64_t columns, float dt, const spd_cotangents_t* xbar,
                        const spd_grads_t* g, const spd_planes_t* out, const spd_planes_t* ct,
                        float* phi_sum, float* psa_sum, float* params_sum, void* stream) {
  if (!xbar || !g || !out || !ct || !g->geopotential || !g->normalized_surface_pressure ||
      !g->params || !phi_sum || !psa_sum || !params_sum)
    return SPD_ERR_NULL;
  ReverseArgs A = {{xbar->u_wind, xbar->v_wind, xbar->temperature, xbar->specific_humidity},
                   {g->u_wind, g->v_wind, g->temperature, g->specific_humidity},
                   {out->u_wind, out->v_wind, out->temperature, out->specific_humidity},
                   {ct->u_wind, ct->v_wind, ct->temperature, ct->specific_humidity},
                   g->geopotential, g->normalized_surface_pressure, g->params,
                   phi_sum, psa_sum, params_sum, 0, columns, dt};
  const int rc = shape(kx, columns, &A.n);
  if (rc != SPD_OK) return rc;
  bool vec = A.n % 4 == 0 && aligned16(A.g_phi) && aligned16(A.phi);
  for (int j = 0; j < 4; ++j) {
    if (!A.xbar[j] || !A.g[j] || !A.out[j] || !A.ct[j]) return SPD_ERR_NULL;
    vec = vec && aligned16(A.xbar[j]) && aligned16(A.g[j]) && aligned16(A.out[j]) &&
          aligned16(A.ct[j]);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (vec)
    reverse_planes<float4><<<dim3(blocks(A.n / 4), 6), kThreads, 0, st>>>(A, A.n / 4);
  else
    reverse_planes<float><<<dim3(blocks(A.n), 6), kThreads, 0, st>>>(A, A.n);
  return cudaGetLastError() == cudaSuccess ? SPD_OK : SPD_ERR_CUDA;
}

}  // extern "C"
