// Instantiates the fused stage kernel for one (dtype, scheme) pair; compiled
// once per pair with -DSWC_T=<float|double> -DSWC_SCHEME=<0..3>
// -DSWC_SUFFIX=<name> so the 32 kernel variants build in parallel.
#include "swc_launch.h"

#ifndef SWC_T
#error "SWC_T must be defined"
#endif

#define SWC_CAT2(a, b) a##b
#define SWC_CAT(a, b) SWC_CAT2(a, b)

namespace swc {
namespace {

// `a` with the z segment filled in where the caller left it to the library.
StageArgs with_zseg(const StageArgs& a, int ty, int tx, int per_sm) {
  StageArgs b = a;
  if (b.zseg <= 0)
    b.zseg = auto_zseg((long long)((a.ny + ty - 1) / ty) *
                           ((a.nx + tx - 1) / tx), a.nz, per_sm);
  b.zseg = b.zseg < a.nz ? b.zseg : a.nz;
  return b;
}
dim3 stage_grid(const StageArgs& a, int ty, int tx) {
  return dim3((a.ny + ty - 1) / ty, (a.nx + tx - 1) / tx,
              (a.nz + a.zseg - 1) / a.zseg);
}

template <typename T, int RM, bool V, bool PE>
int launch_plain(const StageArgs& a, cudaStream_t st) {
  constexpr int TY = 16, TX = 16;
  using Lay = Layout<T, SWC_SCHEME, V, TY, TX>;
  auto kern = stage_kernel<T, SWC_SCHEME, RM, V, TY, TX, PE>;
  // Set once per process (before any graph capture: the first launch of a
  // variant is always eager).
  static int attr_set = 0;
  cudaError_t e;
  if (!attr_set) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)Lay::SMEM);
    if (e != cudaSuccess) return SWC_ERR_LAUNCH;
    attr_set = 1;
  }
  const StageArgs b =
      with_zseg(a, TY, TX, stage_min_blocks<T, SWC_SCHEME, V>());
  kern<<<stage_grid(b, TY, TX), TY * TX, Lay::SMEM, st>>>(b);
  note_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SWC_OK : SWC_ERR_LAUNCH;
}

template <typename T, int RM, bool V>
int launch_rm(const StageArgs& a, cudaStream_t st) {
  return a.has_pe ? launch_plain<T, RM, V, true>(a, st)
                  : launch_plain<T, RM, V, false>(a, st);
}

// Batched launch of `nblocks` CTAs over the members of `b`. Tiles: 1 = 16x16
// (y x x), 2 = 8x32 for members with ny <= 8.
template <typename T, int RM, bool V, int TY, int TX, bool PE>
int launch_batch_tile(const StageBatch& b, int nblocks, cudaStream_t st) {
  using Lay = Layout<T, SWC_SCHEME, V, TY, TX>;
  auto kern = stage_batch_kernel<T, SWC_SCHEME, RM, V, TY, TX, PE>;
  static int attr_set = 0;
  cudaError_t e;
  if (!attr_set) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)Lay::SMEM);
    if (e != cudaSuccess) return SWC_ERR_LAUNCH;
    attr_set = 1;
  }
  kern<<<nblocks, TY * TX, Lay::SMEM, st>>>(b);
  note_launch();
  e = cudaGetLastError();
  return e == cudaSuccess ? SWC_OK : SWC_ERR_LAUNCH;
}

template <typename T, int RM, bool V>
int launch_batch_rm(const StageBatch& b, int nblocks, int tile, int pe,
                    cudaStream_t st) {
  if (tile == 2)
    return pe ? launch_batch_tile<T, RM, V, 8, 32, true>(b, nblocks, st)
              : launch_batch_tile<T, RM, V, 8, 32, false>(b, nblocks, st);
  return pe ? launch_batch_tile<T, RM, V, 16, 16, true>(b, nblocks, st)
            : launch_batch_tile<T, RM, V, 16, 16, false>(b, nblocks, st);
}

// Extended stage (scalars, helper states, face/flux overrides); the tile is
// ext_tile's.
template <typename T, int RM, bool V, int NS, bool HELP, bool EXT>
int launch_ext_v(const StageArgs& a, const SwcStageExt& e, cudaStream_t st) {
  constexpr ExtTile kT = ext_tile<T, SWC_SCHEME, V, NS, HELP, EXT>();
  constexpr int TY = kT.ty, TX = kT.tx;
  using Lay = Layout<T, SWC_SCHEME, V, TY, TX, NS, HELP>;
  auto kern = stage_kernel_ext<T, SWC_SCHEME, RM, V, TY, TX, kT.ctas, NS, HELP,
                               EXT>;
  static int attr_set = 0;
  cudaError_t err;
  if (!attr_set) {
    err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)Lay::SMEM);
    if (err != cudaSuccess) return SWC_ERR_LAUNCH;
    attr_set = 1;
  }
  const StageArgs b = with_zseg(a, TY, TX, kT.ctas);
  kern<<<stage_grid(b, TY, TX), TY * TX, Lay::SMEM, st>>>(b, e);
  note_launch();
  err = cudaGetLastError();
  return err == cudaSuccess ? SWC_OK : SWC_ERR_LAUNCH;
}

template <typename T, int RM, bool V, bool EXT>
int launch_ext_rm(const StageArgs& a, const SwcStageExt& e, int ns, bool help,
                  cudaStream_t st) {
  switch (ns * 2 + (help ? 1 : 0)) {
    case 0: return launch_ext_v<T, RM, V, 0, false, EXT>(a, e, st);
    case 1: return launch_ext_v<T, RM, V, 0, true, EXT>(a, e, st);
    case 2: return launch_ext_v<T, RM, V, 1, false, EXT>(a, e, st);
    case 3: return launch_ext_v<T, RM, V, 1, true, EXT>(a, e, st);
    case 4: return launch_ext_v<T, RM, V, 2, false, EXT>(a, e, st);
    case 5: return launch_ext_v<T, RM, V, 2, true, EXT>(a, e, st);
    case 6: return launch_ext_v<T, RM, V, 3, false, EXT>(a, e, st);
    default: return launch_ext_v<T, RM, V, 3, true, EXT>(a, e, st);
  }
}
template <typename T, int RM, bool V>
int launch_ext_rm(const StageArgs& a, const SwcStageExt& e, int ns, bool help,
                  bool overrides, cudaStream_t st) {
  return overrides ? launch_ext_rm<T, RM, V, true>(a, e, ns, help, st)
                   : launch_ext_rm<T, RM, V, false>(a, e, ns, help, st);
}

}  // namespace

int SWC_CAT(launch_stage_, SWC_SUFFIX)(const StageArgs& a, int riemann,
                                       int visc, cudaStream_t st) {
  using T = SWC_T;
  if (riemann == SWC_HLL)
    return visc ? launch_rm<T, 0, true>(a, st) : launch_rm<T, 0, false>(a, st);
  return visc ? launch_rm<T, 1, true>(a, st) : launch_rm<T, 1, false>(a, st);
}

int SWC_CAT(launch_stage_batch_, SWC_SUFFIX)(const StageBatch& b, int nblocks,
                                             int riemann, int visc, int tile,
                                             int pe, cudaStream_t st) {
  using T = SWC_T;
  if (riemann == SWC_HLL)
    return visc ? launch_batch_rm<T, 0, true>(b, nblocks, tile, pe, st)
                : launch_batch_rm<T, 0, false>(b, nblocks, tile, pe, st);
  return visc ? launch_batch_rm<T, 1, true>(b, nblocks, tile, pe, st)
              : launch_batch_rm<T, 1, false>(b, nblocks, tile, pe, st);
}

int SWC_CAT(launch_stage_ext_, SWC_SUFFIX)(const StageArgs& a,
                                           const SwcStageExt& e, int riemann,
                                           int visc, int ns, int help,
                                           int overrides, cudaStream_t st) {
  using T = SWC_T;
  const bool hp = help != 0, ov = overrides != 0;
  if (riemann == SWC_HLL)
    return visc ? launch_ext_rm<T, 0, true>(a, e, ns, hp, ov, st)
                : launch_ext_rm<T, 0, false>(a, e, ns, hp, ov, st);
  return visc ? launch_ext_rm<T, 1, true>(a, e, ns, hp, ov, st)
              : launch_ext_rm<T, 1, false>(a, e, ns, hp, ov, st);
}

size_t SWC_CAT(stage_batch_smem_, SWC_SUFFIX)(int visc, int tile) {
  using T = SWC_T;
  if (tile == 2)
    return visc ? Layout<T, SWC_SCHEME, true, 8, 32>::SMEM
                : Layout<T, SWC_SCHEME, false, 8, 32>::SMEM;
  return visc ? Layout<T, SWC_SCHEME, true, 16, 16>::SMEM
              : Layout<T, SWC_SCHEME, false, 16, 16>::SMEM;
}

}  // namespace swc
