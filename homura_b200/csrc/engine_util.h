// Shared by the engine's translation units.
#pragma once

#define HM_CUDA(call)                                      \
    do {                                                   \
        cudaError_t _e = (call);                           \
        if (_e != cudaSuccess) return cuda_fail(_e, #call); \
    } while (0)

#include <cuda_runtime.h>
#include <stddef.h>

namespace hm {
// Host memory to host memory, by several threads where it is large (engine_step.cu).
void copy_out(void* dst, const void* src, size_t bytes);
// Before the synchronisation that such a copy waits for: takes the page faults of the destination (its contents stay as they are) while the stream works.
void touch_out(void* dst, size_t bytes, cudaStream_t stream);
// kernel classes of profile_decode; the classes behind PC_COUNT exist in listed designs only
enum ProfClass { PC_EMBED = 0, PC_QKV, PC_ATTN, PC_O, PC_GATE_UP, PC_DOWN, PC_LM_HEAD, PC_SAMPLE, PC_COUNT, PC_LATENT = PC_COUNT, PC_KUP, PC_VUP, PC_KV_WRITE, PC_ROUTE, PC_NORM, PC_QUP, PC_RECUR, PC_COUNT_LISTED };
}  // namespace hm
