// speedy_ensemble.cuh -- what the batched forward and the batched adjoint share: the tile
// list over ragged members, the per-class constants passed by value, the plan's layout and the
// programmatic dependent launch.
#pragma once

#include <algorithm>
#include <vector>

#include "speedy_kernels.cuh"

namespace spd {

// Level-set state of a member in the forward: S points at its accumulator T of the true level
// set; P (S[2 ls_stride]) is the level set its call uses, the one its last call formed.
// (S[ls_stride] is unused.)
enum { LS_T = 0, LS_P = 2 };

struct MemberDev {
  spd_inputs_t in;
  spd_outputs_t out;
  int C, il, kx, cls;
  uint32_t* S;
  int ls_stride, reserved;
};

struct ClassArgs {
  ConstsD cls[SPD_MAX_CLASSES];
};

struct Tile {
  int member, col0;
};

// Where a forward launch takes its tiles from: a plan's member table and tile list, or (when
// `members` is null) the one member given by value, whose tile t covers columns
// t*kNT .. t*kNT + kNT - 1.  Passed by value to the kernels.
struct TileSource {
  const MemberDev* members;
  const Tile* tiles;
  MemberDev single;
  int nmembers;
  uint32_t* redone;   // cumulative count of members redone
};

// The member of tile t, copied: the kernels read its field pointers from the copy, which no
// store to an output field can alias (a reference into the plan would make the compiler reload
// the pointers after every store).
__device__ __forceinline__ MemberDev tile_member(const TileSource& T, int t, int& col0) {
  if (T.members == nullptr) {
    col0 = t * kNT;
    return T.single;
  }
  const Tile tl = T.tiles[t];
  col0 = tl.col0;
  return T.members[tl.member];
}

// Prefetches into L2 the `nrows` rows of a full tile (row(r): the first float of row r, 128
// consecutive floats), one prefetch per 128-byte line, spread over the block's threads.
template <class RowFn>
__device__ __forceinline__ void prefetch_tile_rows(int nrows, RowFn row) {
  static_assert(kNT == 128, "a tile row is four 128-byte lines");
  for (int i = threadIdx.x; i < nrows * 4; i += kNT) {
    const float* p = row(i >> 2) + (i & 3) * 32;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  }
}

// The forward (speedy_ensemble.cu) over the ntiles tiles.  speculate: the fused launch uses each
// member's predicted level set P and a fixup launch redoes the members whose prediction missed;
// otherwise a level-set launch forms every T before the fused launch reads it.  grid_blocks:
// > 0 = the fused launch's persistent grid; 0 or SPD_GRID_PER_TILE = one block per tile (the
// 61-member ensemble took 143 us so, 161 us as a persistent grid of SMs x resident blocks, whose
// blocks own unequal strides of 8- and 16-level tiles).  verify: whether any class fuses verify.
// kx_layout is the largest level count among the tiles (it sizes the fused launch's shared-memory
// arena).
int launch_forward(const ClassArgs& A, const TileSource& T, int ntiles, int kx_layout,
                   int grid_blocks, bool speculate, bool verify, cudaStream_t st,
                   cudaEvent_t marker);

// Launches kernel<<<grid, threads, smem, st>>>(args...) as a programmatic dependent launch: its
// blocks may start as the previous launch's blocks retire (they wait on the device,
// griddepcontrol.wait, before reading what that launch writes).
template <class... KArgs, class... Args>
inline int launch_dependent(void (*kernel)(KArgs...), int grid, int threads, size_t smem,
                            cudaStream_t st,
                            Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) return SPD_ERR_CUDA;
  return SPD_OK;
}

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Device plan layout: header, member records, tile list, level-set region, solar tables.  The
// level-set region: 16 unused bytes, then nw words each of every member's T, an unused word and P
// (nw = member count rounded up to 4), then 16 bytes whose first word counts the members the
// forward redid (its prediction missed).
struct PlanLayout {
  size_t members, tiles, levelset, tables, total;
  int ntiles, nw;
};

inline size_t levelset_region_bytes(int nw) { return 16 + 12 * (size_t)nw + 16; }

// HM: host member description with ix and il.
template <class HM>
inline PlanLayout plan_layout(const HM* members, int n, size_t record_bytes) {
  PlanLayout L;
  int ntiles = 0;
  size_t tab = 0;
  for (int i = 0; i < n; ++i) {
    const int C = members[i].ix * members[i].il;
    ntiles += (C + kNT - 1) / kNT;
    tab += align256((size_t)members[i].il * sizeof(ZonalRow));
  }
  L.ntiles = ntiles;
  L.members = 256;
  L.tiles = L.members + align256((size_t)n * record_bytes);
  L.nw = (n + 3) & ~3;
  L.levelset = L.tiles + align256((size_t)ntiles * sizeof(Tile));
  L.tables = L.levelset + align256(levelset_region_bytes(L.nw));
  L.total = L.tables + tab;
  return L;
}

// The members' T words (device address) in a plan at dbase.
inline uint32_t* levelset_T(const PlanLayout& L, char* dbase) {
  return reinterpret_cast<uint32_t*>(dbase + L.levelset + 16);
}

// The tile list: tiles of 16-level members first, then fewer levels (heavier work first).
// Returns the tile count.  DM: device member record with C and kx.
template <class DM>
inline int plan_tile_list(const DM* md, int n, Tile* tl) {
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return md[a].kx > md[b].kx; });
  int t = 0;
  for (int i : order)
    for (int c0 = 0; c0 < md[i].C; c0 += kNT) tl[t++] = Tile{i, c0};
  return t;
}

// Fills each record's level-set and table pointers (device addresses) and the tile list:
// tiles of 16-level members first, then fewer levels (heavier work first).  Returns the tile
// count.  DM: device member record with C, il, kx, S and table.
template <class DM>
inline int plan_tiles(DM* md, int n, const PlanLayout& L, char* dbase, Tile* tl) {
  size_t tab = L.tables;
  for (int i = 0; i < n; ++i) {
    md[i].S = levelset_T(L, dbase) + i;
    md[i].table = reinterpret_cast<ZonalRow*>(dbase + tab);
    tab += align256((size_t)md[i].il * sizeof(ZonalRow));
  }
  return plan_tile_list(md, n, tl);
}

}  // namespace spd
