// Launch of the fp32 mode's scheduler kernel (fp32.cu).
#pragma once
#include <cuda_runtime.h>
#include "device_types.h"

cudaError_t fp32_prepare(size_t smem_bytes);
void fp32_launch(unsigned ctas, size_t smem_bytes, cudaStream_t stream, const NasmDev *nasms, CtrlDev *ctrl, unsigned long long *queue, StatusHost *status,
                 unsigned long long *prof);
