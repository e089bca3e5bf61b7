/*
 * smem_limit.h - the dynamic shared memory a kernel may be launched with.
 *
 * The limit (48 KB less the kernel's static part unless set) belongs to the
 * kernel, not to a launch.  Were it set to each launch's own size, a call could
 * lower it between another thread's setting and launch, and that launch would
 * be refused.  So a kernel's limit is always set to one value, the most that any
 * of its launches takes, and concurrent calls write the same.
 */
#ifndef BAMF_SMEM_LIMIT_H
#define BAMF_SMEM_LIMIT_H

#include <cstddef>

#include <cuda_runtime.h>

/* what a CTA can have (227 KB), less 1 KB for a kernel's static variables */
constexpr size_t DYNAMIC_SMEM_MOST = 226 * 1024;

template <typename Kern>
inline cudaError_t allow_smem(Kern kern, size_t most = DYNAMIC_SMEM_MOST)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

#endif
