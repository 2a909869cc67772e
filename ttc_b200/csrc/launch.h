// Launch dispatch shared by the plain and batched entry points.
#pragma once
#include <cuda_runtime.h>
#include "plan.h"

namespace ttcb {

// Launches one plan. va/vb are the access widths actually used (the plan's widths, or 1 when a
// pointer is not 16-byte aligned). variant: 0 = beta==0, 1 = beta==0 with streaming stores,
// 2 = beta != 0.
using LaunchFn = cudaError_t (*)(const ttcb_plan* p, const void* A, void* B, const void* alpha, const void* beta,
                                 cudaStream_t stream, int blocks);

struct KernelRef {
  LaunchFn fn = nullptr;
  const void* func = nullptr;  // the __global__ function (for occupancy queries and attributes)
};

// One definition per A/B type pair lives in kernels_<pair>.cu.
KernelRef pick_kernel(ttcb_dtype ta, ttcb_dtype tb, int kernel, int va, int vb, int variant);

// The counter words (claim, finished CTAs) of a launch of a plan's staged kernel with claimed tiles on
// `stream`. Two launches that run at the same time must not share them, so each stream (by its id, which
// the CUDA runtime never gives out twice) has a pair of its own, whose launches follow each other. Null,
// and the launch takes the round-robin order, when the plan has no counters, when kClaimSlots other
// streams have taken them, and under capture: a graph may be replayed beside any launch, and more than
// once at a time.
constexpr int kClaimSlots = 64;
unsigned int* plan_claim_slot(const ttcb_plan* p, cudaStream_t stream);

// Whether a launch of the staged kernel lets its successor in the stream begin beside it (abi.cu: the reason).
bool launch_overlaps_next(const ttcb_plan* p, const void* func, int blocks, cudaStream_t stream);

// Dynamic shared memory ceiling of every plan (the planner never exceeds it).
constexpr int kMaxDynamicSmem = 200 * 1024;
// True when a launch with this much dynamic shared memory needs the opt-in above 48 KB.
bool needs_large_smem(int dynamic_smem);
// Raises func's dynamic shared memory limit to kMaxDynamicSmem on the current device, once; it
// never lowers it. Every entry point that launches a kernel goes through this (defined in abi.cu).
void allow_large_smem(const void* func);

using BatchLaunchFn = cudaError_t (*)(const void* segs, unsigned int nseg, unsigned int* counter, const void* alpha,
                                      const void* beta, int blocks, int smem, cudaStream_t stream);
struct BatchKernelRef {
  BatchLaunchFn fn = nullptr;
  const void* func = nullptr;
};
BatchKernelRef pick_batch_kernel(ttcb_dtype ta, ttcb_dtype tb, int variant);

}  // namespace ttcb
