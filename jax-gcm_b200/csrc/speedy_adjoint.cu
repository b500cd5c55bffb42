// speedy_adjoint.cu -- the adjoint of the forward: one instance (spd_vjp) or a ragged ensemble
// of them (spd_ensemble_vjp), both through the same three launches (the first clears what the
// others add to).
//
// Launch 2 is the forward's cloud-top pre-pass over the tile list of speedy_ensemble.cuh (each
// member's level set S and per-latitude solar table: neither carries a derivative).  Launch 3
// runs one thread per column, one block per tile: the reverse pass of speedy_vjp_smem.cuh
// recomputes the column's forward and walks its terms backwards, writing the state gradients;
// the 12 parameter gradients are summed per thread, then per warp, then per block, and added to the
// tile's member with one coalesced atomic.  A single instance is one member given by value to the same
// kernels.
//
// Measured (the whole call, against the fully unrolled reverse pass with its arrays in registers
// and local memory that this replaces): T425 with 16 levels 3,195 -> 890 us, T170 with 16
// levels and verify 578 -> 204 us, T85 with 16 levels 131 -> 51 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include <string.h>

#include <algorithm>
#include <mutex>

#include "speedy_vjp.h"

// the column's first half divides like the rest of the adjoint (speedy_vjp.h, fdiv)
#define SPD_DIV(a, b) (spdvjp::fdiv((a), (b)))
#define SPD_DIV_FULL(a, b) (spdvjp::fdiv_full((a), (b)))
#include "speedy_ensemble.cuh"
#include "speedy_vjp_smem.cuh"

namespace spd {

int check_instance(const spd_desc_t* d, const spd_inputs_t* in, const spd_outputs_t* out);
Consts make_consts(const spd_desc_t* d, const spd_vgrid_t* vg, const spd_params_t* p);

// Adds the block's sums of pacc to params, one coalesced atomic per tile.  Sixteen lanes' worth of
// sums (12 used) are folded by halves: a lane keeps the half of the values its bit selects and adds
// the other lane's, 16 shuffles where a butterfly per value takes 60.  The first warp adds the warps'
// sums in their order, so that those of an instance of one tile are the same on every call (an atomic
// per warp gave other bits in two of five calls beside another stream's work).  The warps that wait
// here hold nothing up: their block's resources are free only when its last warp is done.  (With
// no barrier, the last warp to come adding the sums, by an atomic count and fences, T85 with 16
// levels took 52.2 against 50.8 us.)  Every thread must call it; the block's barrier before its
// next tile keeps the tiles apart.
__device__ __forceinline__ void block_add_params(const float* pacc, float* params,
                                                 float (*sums)[SPD_NUM_DIFF_PARAMS]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = j < SPD_NUM_DIFF_PARAMS ? pacc[j] : 0.0f;
#pragma unroll
  for (int n = 8; n >= 1; n /= 2) {
    const bool hi = (lane & (2 * n)) != 0;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const float keep = hi ? v[j + n] : v[j], give = hi ? v[j] : v[j + n];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  const int j = lane >> 1;
  if ((lane & 1) == 0 && j < SPD_NUM_DIFF_PARAMS) sums[warp][j] = v[0];
  __syncthreads();
  if (threadIdx.x < SPD_NUM_DIFF_PARAMS) {
    float sum = sums[0][lane];
#pragma unroll
    for (int w = 1; w < kNT / 32; ++w) sum += sums[w][lane];
    atomicAdd(params + lane, sum);
  }
}

// Start of a call: every member's level set and parameter gradients at zero.  One block.
__global__ void __launch_bounds__(kBlock) vjp_begin(const __grid_constant__ VjpSource T) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int nm = T.members ? T.nmembers : 1;
  for (int i = threadIdx.x; i < nm * (SPD_NUM_DIFF_PARAMS + 1); i += blockDim.x) {
    const int j = i % (SPD_NUM_DIFF_PARAMS + 1);
    const VjpMemberDev* m = T.members ? T.members + i / (SPD_NUM_DIFF_PARAMS + 1) : nullptr;
    if (j == SPD_NUM_DIFF_PARAMS)
      *(m ? m->S : T.single.S) = 0u;
    else
      (m ? m->gr.params : T.single.gr.params)[j] = 0.0f;
  }
}

// Pre-pass: each member's level set and solar table.  It may start beside vjp_begin, and waits
// for it before it adds to a level set.
template <int KX>
__device__ __forceinline__ uint32_t prepass_bit(const Consts& K, const spd_inputs_t& in, int c,
                                                int C, ZonalRow* table, int il) {
  if (c < il) table[c] = zonal_row(K.tyear, __ldg(in.sia + c), __ldg(in.coa + c));
  return c < C ? prepass_column<KX>(K, in, c, C) : 0u;
}
__global__ void __launch_bounds__(kBlock)
    ensemble_vjp_prepass(const __grid_constant__ ClassArgs A,
                         const __grid_constant__ VjpSource T, int ntiles) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile tl = T.members ? T.tiles[t] : Tile{0, t * kNT};
    const VjpMemberDev& m = T.members ? T.members[tl.member] : T.single;
    const Consts& K = A.cls[m.cls].K;
    const int c = tl.col0 + threadIdx.x;
    uint32_t bit;
    switch (m.kx) {  // uniform per block
      case 16: bit = prepass_bit<16>(K, m.in, c, m.C, m.table, m.il); break;
      case 8: bit = prepass_bit<8>(K, m.in, c, m.C, m.table, m.il); break;
      default: bit = prepass_bit<7>(K, m.in, c, m.C, m.table, m.il); break;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    or_level_set_warp(bit, m.S);
  }
}

// The adjoint launch: one thread per column (speedy_vjp_smem.cuh), one block per tile with its
// level arrays in `sm` and no barrier but around its member's record and its parameter sums.  The threads past a member's
// last column run that column again and store nothing, so that every warp is whole (the
// convection's reverse votes).  The times below are of the form that each choice was made on; all
// of them have come down since (above).  Blocks of one
// warp, which make room as soon as their columns are done, are no faster: a block's four warps
// start together and share what they fetch of the code (T425 with 16 levels, 32 / 64 / 128 / 384
// threads: 1,029 / 972 / 942 / 1,001 us; with 8 levels 563 / 537 / 500 / 515 us).  Barriers at the
// stage boundaries cost 0.5 %.
// Three register budgets, which give the same bits, so that a member's gradients do not depend on
// the batch that carried it:
//  - 168 (twelve warps per SM), what the arena of 16 levels leaves room for (73,728 bytes and the
//    1,024 reserved per block, three blocks);
//  - 128 (sixteen) where the batch has at most 8 levels, whose arenas do not bind (T425 with 8
//    levels 458 against 500 us; the spills of 128 registers cost 16 levels 993 against 942 us, and
//    96 registers with twenty warps 442 us at T425 but 110 against 96 us at T170);
//  - 255 (eight), which spills next to nothing, where two warps per scheduler hold the whole batch
//    (T85 with 16 levels, 1,024 warps: 60 against 66 us; T170, 4,096 warps: 209 against 194 us).
// kVerify: whether any class fuses verify; without it the launch carries neither the limited levels
// nor the humidity tendencies they are found from (T425 with 16 levels 887 against 934
// us, T85 49.5 against 53.2).
template <int kWarpsPerSm, bool kVerify>
__global__ void __launch_bounds__(kNT, kWarpsPerSm / (kNT / 32))
    ensemble_adjoint(const __grid_constant__ ClassArgs A, const __grid_constant__ VjpSource T,
                     int ntiles) {
  extern __shared__ float sm[];
  __shared__ VjpMemberDev m;
  __shared__ float sums[kNT / 32][SPD_NUM_DIFF_PARAMS];
  constexpr int kWords = sizeof(VjpMemberDev) / sizeof(uint64_t);
  static_assert(kWords <= kNT && sizeof(VjpMemberDev) % sizeof(uint64_t) == 0,
                "one copy per thread");
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const Tile tl = T.members ? T.tiles[t] : Tile{0, t * kNT};
    __syncthreads();  // the last tile's columns are done with its record
    if (threadIdx.x < kWords) {
      const uint64_t* from =
          reinterpret_cast<const uint64_t*>(T.members ? T.members + tl.member : &T.single);
      reinterpret_cast<uint64_t*>(&m)[threadIdx.x] = from[threadIdx.x];
    }
    __syncthreads();
    const int C = m.C, at = tl.col0 + (int)threadIdx.x;
    const bool valid = at < C;
    const int c = valid ? at : C - 1;
    float pacc[SPD_NUM_DIFF_PARAMS];
#pragma unroll
    for (int j = 0; j < SPD_NUM_DIFF_PARAMS; ++j) pacc[j] = 0.0f;
    const ConstsD& CD = A.cls[m.cls];
    switch (m.kx) {  // uniform per block
      case 16: column_vjp_smem<16, kVerify>(CD, sm, m, c, C, valid, pacc); break;
      case 8: column_vjp_smem<8, kVerify>(CD, sm, m, c, C, valid, pacc); break;
      default: column_vjp_smem<7, kVerify>(CD, sm, m, c, C, valid, pacc); break;
    }
#pragma unroll
    for (int j = 0; j < SPD_NUM_DIFF_PARAMS; ++j) pacc[j] = valid ? pacc[j] : 0.0f;
    block_add_params(pacc, load_field(m.gr.params), sums);
  }
}

// The adjoint launch's forms: by warps per SM, without and with verify.
enum { kWarps8, kWarps12, kWarps16 };
static void (*const kAdjoint[])(const ClassArgs, const VjpSource, int) = {
    ensemble_adjoint<8, false>,  ensemble_adjoint<8, true>,  ensemble_adjoint<12, false>,
    ensemble_adjoint<12, true>, ensemble_adjoint<16, false>, ensemble_adjoint<16, true>};

// Allows the adjoint launch its arena on the current device, once per device (the attribute is a
// per-device setting of the kernel); gives the device's SM count.
static int allow_arena(int* sms = nullptr) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static int count[kMaxDevices] = {};  // SMs, once set up
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SPD_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (!count[dev]) {
    const int bytes = (int)vjp_arena_bytes(SPD_MAX_KX);
    int n = 0;
    for (auto* kernel : kAdjoint)
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
          cudaSuccess)
        return SPD_ERR_CUDA;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return SPD_ERR_CUDA;
    count[dev] = n;
  }
  if (sms) *sms = count[dev];
  return SPD_OK;
}

// The column's divisions and reciprocal as this file compiles them (spd_selftest_division).
__global__ void __launch_bounds__(kBlock)
    selftest_division(int n, const float* a, const float* b, float* out) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  const size_t m = n;
  out[i] = spdvjp::fdiv(a[i], b[i]);
  out[m + i] = spdvjp::frcp(b[i]);
  out[2 * m + i] = spdvjp::fdiv_full(a[i], b[i]);
}

struct OneMember {
  int ix, il;
};

inline PlanLayout single_layout(const spd_desc_t* d) {
  const OneMember m{d->ix, d->il};
  return plan_layout(&m, 1, sizeof(VjpMemberDev));
}

int preload_adjoint() {
  cudaFuncAttributes a;
  bool ok = true;
  ok &= cudaFuncGetAttributes(&a, vjp_begin) == cudaSuccess;
  ok &= cudaFuncGetAttributes(&a, ensemble_vjp_prepass) == cudaSuccess;
  for (auto* kernel : kAdjoint)
    ok &= cudaFuncGetAttributes(&a, kernel) == cudaSuccess;
  return ok && allow_arena() == SPD_OK ? SPD_OK : SPD_ERR_CUDA;
}

// The three launches; each but the first may start while the one before it runs.
static int launch_ensemble_vjp(const ClassArgs& A, int kx_layout, bool verify,
                               const VjpSource& T, int ntiles, int grid_blocks,
                               cudaStream_t st) {
  // Default: one block per tile.  The blocks are short (one tile's columns each), so the SMs
  // turn over often and a higher-priority stream's kernels (a forward batch) get them within
  // one block's time; a persistent grid would hold every SM until the whole batch is done.
  const int grid = grid_blocks > 0 ? std::min(grid_blocks, ntiles) : ntiles;
  const int grid_pre = std::min(ntiles, 65535);
  int sms = 0;
  if (allow_arena(&sms) != SPD_OK) return SPD_ERR_CUDA;
  vjp_begin<<<1, kBlock, 0, st>>>(T);
  int rc = launch_dependent(ensemble_vjp_prepass, grid_pre, kBlock, 0, st, A, T, ntiles);
  if (rc != SPD_OK) return rc;
  const int warps = grid * (kNT / 32) <= 8 * sms ? kWarps8 : kx_layout > 8 ? kWarps12 : kWarps16;
  rc = launch_dependent(kAdjoint[2 * warps + verify], grid, kNT, vjp_arena_bytes(kx_layout), st, A,
                        T, ntiles);
  if (rc != SPD_OK) return rc;
  return cudaGetLastError() == cudaSuccess ? SPD_OK : SPD_ERR_CUDA;
}

// The fields spd_vjp reads and writes, validated like spd_fwd's.
static int check_vjp_member(const spd_desc_t* desc, const spd_inputs_t* in,
                            const spd_cotangents_t* ct, const spd_grads_t* grads) {
  if (!desc || !in || !ct || !grads) return SPD_ERR_NULL;
  spd_outputs_t dummy = {};
  float* probe = grads->temperature;
  dummy.u_wind = dummy.v_wind = dummy.temperature = dummy.specific_humidity = probe;
  dummy.precnv = dummy.precls = probe;
  int rc = check_instance(desc, in, &dummy);
  if (rc != SPD_OK) return rc;
  const void* req[] = {ct->u_wind, ct->v_wind, ct->temperature, ct->specific_humidity,
                       grads->u_wind, grads->v_wind, grads->specific_humidity,
                       grads->geopotential, grads->normalized_surface_pressure, grads->params};
  for (const void* p : req)
    if (!p) return SPD_ERR_NULL;
  return SPD_OK;
}

}  // namespace spd

extern "C" {

size_t spd_vjp_scratch_bytes(const spd_desc_t* desc) {
  if (!desc || desc->ix <= 0 || desc->il <= 0) return 0;
  return spd::single_layout(desc).total;
}

int spd_vjp(const spd_desc_t* desc, const spd_vgrid_t* vgrid, const spd_params_t* params,
            const spd_inputs_t* in, const spd_cotangents_t* ct, const spd_grads_t* grads,
            void* scratch, size_t scratch_bytes, void* stream) {
  using namespace spd;
  if (!desc || !vgrid || !params || !in || !ct || !grads) return SPD_ERR_NULL;
  const int rc = check_vjp_member(desc, in, ct, grads);
  if (rc != SPD_OK) return rc;
  const PlanLayout L = single_layout(desc);
  if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 255u) || scratch_bytes < L.total)
    return SPD_ERR_SCRATCH;
  if (desc->kx != 7 && desc->kx != 8 && desc->kx != 16) return SPD_ERR_KX;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* base = static_cast<char*>(scratch);
  ClassArgs A;
  A.cls[0].K = make_consts(desc, vgrid, params);
  A.cls[0].D = derive_constants(desc, vgrid, params);
  VjpSource T{};
  T.single.in = *in;
  T.single.ct = *ct;
  T.single.gr = *grads;
  T.single.C = desc->ix * desc->il;
  T.single.il = desc->il;
  T.single.kx = desc->kx;
  T.single.cls = 0;
  T.single.S = reinterpret_cast<uint32_t*>(base + L.levelset);
  T.single.table = reinterpret_cast<ZonalRow*>(base + L.tables);
  T.nmembers = 1;
  return launch_ensemble_vjp(A, desc->kx, (desc->flags & SPD_FUSE_VERIFY) != 0, T, L.ntiles, 0,
                             st);
}

size_t spd_ensemble_vjp_plan_bytes(const spd_vjp_member_t* members, int nmembers) {
  if (!members || nmembers <= 0) return 0;
  return spd::plan_layout(members, nmembers, sizeof(spd::VjpMemberDev)).total;
}

int spd_ensemble_vjp_plan(const spd_class_t* classes, int nclasses,
                          const spd_vjp_member_t* members, int nmembers, void* plan_host,
                          void* plan_device, size_t plan_bytes, spd_plan_info_t* info) {
  using namespace spd;
  if (!classes || !members || !plan_host || !plan_device || !info) return SPD_ERR_NULL;
  if (nclasses <= 0 || nclasses > SPD_MAX_CLASSES || nmembers <= 0) return SPD_ERR_SHAPE;
  if (reinterpret_cast<uintptr_t>(plan_device) & 255u) return SPD_ERR_SCRATCH;
  const PlanLayout L = plan_layout(members, nmembers, sizeof(VjpMemberDev));
  if (plan_bytes < L.total) return SPD_ERR_SCRATCH;
  for (int i = 0; i < nmembers; ++i) {
    const spd_vjp_member_t& m = members[i];
    if (m.cls < 0 || m.cls >= nclasses) return SPD_ERR_SHAPE;
    spd_desc_t d = classes[m.cls].desc;
    d.ix = m.ix;
    d.il = m.il;
    const int rc = check_vjp_member(&d, &m.in, &m.ct, &m.grads);
    if (rc != SPD_OK) return rc;
  }
  char* h = static_cast<char*>(plan_host);
  memset(h, 0, L.total);
  VjpMemberDev* md = reinterpret_cast<VjpMemberDev*>(h + L.members);
  for (int i = 0; i < nmembers; ++i) {
    const spd_vjp_member_t& m = members[i];
    md[i].in = m.in;
    md[i].ct = m.ct;
    md[i].gr = m.grads;
    md[i].C = m.ix * m.il;
    md[i].il = m.il;
    md[i].kx = classes[m.cls].desc.kx;
    md[i].cls = m.cls;
  }
  const int t = plan_tiles(md, nmembers, L, static_cast<char*>(plan_device),
                           reinterpret_cast<Tile*>(h + L.tiles));
  info->nmembers = nmembers;
  info->ntiles = t;
  info->levelset_offset = L.levelset;
  info->levelset_bytes = align256((size_t)nmembers * sizeof(uint32_t));
  info->plan_bytes = L.total;
  return SPD_OK;
}

int spd_ensemble_vjp(const spd_class_t* classes, int nclasses, void* plan_device,
                     const spd_plan_info_t* info, int grid_blocks, void* stream) {
  using namespace spd;
  if (!classes || !plan_device || !info) return SPD_ERR_NULL;
  if (nclasses <= 0 || nclasses > SPD_MAX_CLASSES || info->ntiles <= 0) return SPD_ERR_SHAPE;
  ClassArgs A;
  int kx_layout = 0;
  bool verify = false;
  for (int i = 0; i < nclasses; ++i) {
    if (classes[i].desc.flags & SPD_FUSE_VERIFY) verify = true;
    A.cls[i].K = make_consts(&classes[i].desc, &classes[i].vgrid, &classes[i].params);
    A.cls[i].D = derive_constants(&classes[i].desc, &classes[i].vgrid, &classes[i].params);
    kx_layout = std::max(kx_layout, classes[i].desc.kx);
  }
  char* base = static_cast<char*>(plan_device);
  VjpSource T{};
  T.members = reinterpret_cast<const VjpMemberDev*>(base + 256);
  T.tiles = reinterpret_cast<const Tile*>(
      base + 256 + align256((size_t)info->nmembers * sizeof(VjpMemberDev)));
  T.nmembers = info->nmembers;
  return launch_ensemble_vjp(A, kx_layout, verify, T, info->ntiles, grid_blocks,
                             static_cast<cudaStream_t>(stream));
}

int spd_selftest_division(int n, const float* a, const float* b, float* out, void* stream) {
  using namespace spd;
  if (!a || !b || !out) return SPD_ERR_NULL;
  if (n <= 0 || n > (1 << 28)) return SPD_ERR_SHAPE;
  selftest_division<<<(n + kBlock - 1) / kBlock, kBlock, 0, static_cast<cudaStream_t>(stream)>>>(
      n, a, b, out);
  return cudaGetLastError() == cudaSuccess ? SPD_OK : SPD_ERR_CUDA;
}

}  // extern "C"
