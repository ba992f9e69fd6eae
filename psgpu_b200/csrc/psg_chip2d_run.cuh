// psg_chip2d_run.cuh -- launch side of the on-chip 2D integrator
// (psg_chip2d.cuh): which kernels are built, what each needs, and the launch of
// one grid size's instances as one cluster each.  Instantiated in
// psg_chip2d_f64.cu and psg_chip2d_f32.cu; other files see the declarations.
#pragma once
#include "psg_chip2d.cuh"
#include "psgpu_internal.h"

namespace psg {

// A kernel ready to launch: cluster size, threads, shared memory, whether the
// state arrays live in shared memory, and the clusters the device holds at once
// (`alone`: with an SM to every block; filled in where it is asked for).
struct ChipPlan {
  const void* fn = nullptr;
  int cs = 0, threads = 0, state = 0, resident = 0, alone = 0;
  size_t smem = 0;
};

constexpr int kChipThreads(int elem, int kind) { return elem == 4 && kind == CHIP_STEP ? 512 : 256; }

template <typename T, int N, int CS, int KIND, int PK>
__global__ void __launch_bounds__(kChipThreads(sizeof(T), KIND))
    chip2d(const ChipInst<T>* __restrict__ insts, const cpx<T>* __restrict__ tw, int state) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int rank = 0;
  if (CS > 1) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const ChipInst<T> I = insts[blockIdx.x / CS];
  Chip2D<T, N, CS, KIND, PK> c;
  c.run(I, tw, smem_raw, rank, state != 0);
}

// The cluster sizes built for a grid size, smallest first.  Small grids gain
// nothing from a second block; the largest need eight or sixteen blocks' shared
// memory for their lines.
template <typename T>
struct ChipSizes {
  static constexpr bool D = sizeof(T) == 8;
  static constexpr bool built(int n, int cs, int kind) {
    return n <= 32   ? cs == 1
           : n == 64 ? cs == 1 || cs == 4 || cs == 8
           : n == 128 ? (D ? (cs == 4 && kind != CHIP_TANGENT) || cs == 8 || cs == 16
                           : (cs == 1 && kind == CHIP_STEP) || cs == 2 || cs == 4 || cs == 8)
                      : (D ? cs == 16 && kind != CHIP_TANGENT : cs == 8 || cs == 16);
  }
};

// clusters of `cs` blocks of `threads` threads and `smem` bytes that the device holds
// at once; 0 where there is no room for one
inline int chip_resident(const void* fn, int cs, int threads, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}
// the same with an SM to every block (whose shared memory leaves no room beside it).
// A cluster lies in one GPC: on a B200 of 148 SMs 74 clusters of 2, 33 of 4, 15 of 8, 7 of 16.
inline int chip_alone(const ChipPlan& p) {
  int dev = 0, big = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&big, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  return 2 * p.smem > (size_t)big ? p.resident : chip_resident(p.fn, p.cs, p.threads, big);
}

// the kernel of (n, cs, kind, pk) at about `threads` threads a block; false when
// it is not built or does not fit the device
template <typename T>
bool chip2d_plan(int n, int cs, int kind, int pk, int threads, ChipPlan* out);
// one cluster per instance, m instances of one grid size
template <typename T>
cudaError_t chip2d_launch(const ChipPlan& p, const ChipInst<T>* d_insts, int m, const cpx<T>* tw,
                          cudaStream_t st);

#ifdef PSG_CHIP2D_INSTANTIATE
template <typename T, int N, int CS, int KIND, int PK>
bool chip2d_plan_one(int threads, ChipPlan* out) {
  if constexpr (!ChipSizes<T>::built(N, CS, KIND) || (PK != 0 && (sizeof(T) != 4 || KIND != CHIP_STEP))) {
    return false;
  } else {
    using S = ChipShape<T, N, CS, KIND>;
    int dev = 0, big = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&big, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
      return false;
    ChipPlan p;
    p.fn = (const void*)chip2d<T, N, CS, KIND, PK>;
    p.cs = CS;
    // no more threads than the widest phase has lines for, whole warps
    const int most = (S::lines() * S::G + 31) / 32 * 32;
    int nt = threads < kChipThreads(sizeof(T), KIND) ? threads : kChipThreads(sizeof(T), KIND);
    if (nt > most) nt = most;
    for (; nt >= 64; nt = nt / 64 * 32) {  // halve until the exchange space fits
      for (int state = 1; state >= 0; --state)
        if (S::smem(nt, state) <= (size_t)big) {
          p.threads = nt;
          p.state = state;
          p.smem = S::smem(nt, state);
          nt = 0;
          break;
        }
      if (!nt) break;
    }
    if (!p.threads) return false;
    if (cudaFuncSetAttribute(p.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, big) != cudaSuccess ||
        (CS > 8 && cudaFuncSetAttribute(p.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
      cudaGetLastError();
      return false;
    }
    p.resident = chip_resident(p.fn, CS, p.threads, p.smem);
    if (p.resident < 1) return false;
    *out = p;
    return true;
  }
}

template <typename T, int N, int KIND, int PK>
bool chip2d_plan_n(int cs, int threads, ChipPlan* out) {
  switch (cs) {
    case 1: return chip2d_plan_one<T, N, 1, KIND, PK>(threads, out);
    case 2: return chip2d_plan_one<T, N, 2, KIND, PK>(threads, out);
    case 4: return chip2d_plan_one<T, N, 4, KIND, PK>(threads, out);
    case 8: return chip2d_plan_one<T, N, 8, KIND, PK>(threads, out);
    case 16: return chip2d_plan_one<T, N, 16, KIND, PK>(threads, out);
  }
  return false;
}

template <typename T, int N>
bool chip2d_plan_k(int cs, int kind, int pk, int threads, ChipPlan* out) {
  if (kind == CHIP_BASE) return chip2d_plan_n<T, N, CHIP_BASE, 0>(cs, threads, out);
  if (kind == CHIP_TANGENT) return chip2d_plan_n<T, N, CHIP_TANGENT, 0>(cs, threads, out);
  return pk ? chip2d_plan_n<T, N, CHIP_STEP, 1>(cs, threads, out) : chip2d_plan_n<T, N, CHIP_STEP, 0>(cs, threads, out);
}

template <typename T>
bool chip2d_plan(int n, int cs, int kind, int pk, int threads, ChipPlan* out) {
  switch (n) {
    case 16: return chip2d_plan_k<T, 16>(cs, kind, pk, threads, out);
    case 32: return chip2d_plan_k<T, 32>(cs, kind, pk, threads, out);
    case 64: return chip2d_plan_k<T, 64>(cs, kind, pk, threads, out);
    case 128: return chip2d_plan_k<T, 128>(cs, kind, pk, threads, out);
    case 256: return chip2d_plan_k<T, 256>(cs, kind, pk, threads, out);
  }
  return false;
}

template <typename T>
cudaError_t chip2d_launch(const ChipPlan& p, const ChipInst<T>* d_insts, int m, const cpx<T>* tw,
                          cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(p.cs * m);
  cfg.blockDim = dim3(p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int state = p.state;
  void* args[] = {(void*)&d_insts, (void*)&tw, (void*)&state};
  return cudaLaunchKernelExC(&cfg, p.fn, args);
}

#define PSG_CHIP2D_TEMPLATES(T)                                             \
  template bool chip2d_plan<T>(int, int, int, int, int, ChipPlan*);         \
  template cudaError_t chip2d_launch<T>(const ChipPlan&, const ChipInst<T>*, int, const cpx<T>*, cudaStream_t);
#endif

extern template bool chip2d_plan<double>(int, int, int, int, int, ChipPlan*);
extern template bool chip2d_plan<float>(int, int, int, int, int, ChipPlan*);
extern template cudaError_t chip2d_launch<double>(const ChipPlan&, const ChipInst<double>*, int,
                                                  const cpx<double>*, cudaStream_t);
extern template cudaError_t chip2d_launch<float>(const ChipPlan&, const ChipInst<float>*, int,
                                                 const cpx<float>*, cudaStream_t);

}  // namespace psg
