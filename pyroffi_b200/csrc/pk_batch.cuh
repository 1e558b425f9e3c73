// Internal interface of the batched (work-queue) IK launchers: the two
// seed-group bodies (pk_lm.cu) and the warp-per-seed body (pk_lm_wide.cu)
// each run one persistent kernel over the items of their robot classes.
#pragma once

#include "pk_obstacles.cuh"
#include "pyroffi_b200.h"

namespace pk {

constexpr int PK_MAX_CLASSES = 8;

// body selector of a class (pk_ik_class.body)
constexpr int kBodySeedGroup = 0;    // TPS lanes per seed, registers (n_act <= 8, one EE)
constexpr int kBodyWarp = 1;         // one warp per seed, shared-memory state (n_act <= 32)
constexpr int kBodySeedGroup16 = 2;  // one lane per seed, registers (n_act <= 16, n_ee <= 2)

struct BatchCall {
  const pk_ik_class* cls;  // host array, n_classes entries
  int n_classes;
  WorldArgs w;
  pk_lm_options opt;
  const int4* items;       // device [n_items] (class, problem, first seed, seed count)
  int n_items;
  int* queue;              // device [2] item counters (cleared by the launcher)
  int blocks;              // persistent grid per kernel; 0 = one full wave
};

// The batch's persistent kernels, one per body, are independent of one another
// but share a stream.  From the second on they are launched with programmatic
// stream serialization: every block of a kernel lets the next one start as soon
// as it runs (batch_trigger), so the next kernel's blocks move in where the
// last items of the one before leave SMs idle, and a kernel that follows
// another ends only after it has (batch_join, at the end of every block), so
// what follows on the stream waits for all of them.  lm_warp_kernel has no
// batch_join: it is always the first (launch_seed_group_batch comes after it).
// Nothing waits on a kernel that is not wholly resident or done: a dependent's
// blocks start only after every block of the kernel before has.  512 problems
// of the mixed workload, 6 iterations: 7038 -> 5691 us, the same bits (the
// three kernels ran one after another, each with SMs idle for 12 to 39% of its
// time behind its last items).
__device__ __forceinline__ void batch_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void batch_join() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches kern<<<grid, threads, smem, st>>>(arg), `follows` another kernel of
// the same batch on the stream.
template <class Kernel, class Arg>
static inline cudaError_t batch_launch(Kernel kern, dim3 grid, int threads, size_t smem, cudaStream_t st, bool follows,
                                       const Arg& arg) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = follows ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, arg);
}

// The launch's class table is indexed at run time; reading it with constant
// indices (one case per class) keeps it in parameter space instead of a
// local-memory copy.
template <typename T, typename Table>
__device__ __forceinline__ void pick_class(const Table& tab, int c, T& dst) {
  switch (c) {
    case 0: dst = tab[0]; break;
    case 1: dst = tab[1]; break;
    case 2: dst = tab[2]; break;
    case 3: dst = tab[3]; break;
    case 4: dst = tab[4]; break;
    case 5: dst = tab[5]; break;
    case 6: dst = tab[6]; break;
    default: dst = tab[7]; break;
  }
}
static_assert(PK_MAX_CLASSES == 8, "pick_class covers 8 classes");

// Each launches its persistent kernel when some class uses its body and
// adds the number of kernels launched to *launched.
int launch_seed_group_batch(const BatchCall& b, cudaStream_t st, int* launched);
int launch_warp_batch(const BatchCall& b, cudaStream_t st, int* launched);

// Warp-per-seed LM over a plain (problems x seed blocks) grid, the route of
// pk_ls_ik_ex for robots beyond the seed-group kernel's buckets.
int launch_warp_grid(const pk_ik_class& c, const WorldArgs& w, const pk_lm_options& opt, cudaStream_t st);

}  // namespace pk
