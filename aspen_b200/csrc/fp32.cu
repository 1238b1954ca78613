// The scheduler kernel of the fp32 mode, in a translation unit of its own: functions that are not inlined share one register
// limit per unit, and beside the tensor-core kernel (384 threads) that limit, 168, makes the fp32 blocks spill.
#include "internal.h"
#include "scheduler.cuh"
#include "fp32.h"

cudaError_t fp32_prepare(size_t smem_bytes) {
    return cudaFuncSetAttribute(sched::scheduler_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
}

void fp32_launch(unsigned ctas, size_t smem_bytes, cudaStream_t stream, const NasmDev *nasms, CtrlDev *ctrl, unsigned long long *queue, StatusHost *status,
                 unsigned long long *prof) {
    sched::scheduler_kernel<false><<<ctas, sched::threads<false>(), smem_bytes, stream>>>(nasms, ctrl, queue, status, prof);
}
