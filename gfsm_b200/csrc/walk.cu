// walk.cu -- memory and launches of the walk (walk_kernel.cuh).
#include <cuda_runtime.h>

#include "walk_kernel.cuh"

namespace gfsm {

uint64_t walk_queue_bytes(uint32_t core, int sms) {
    return (uint64_t)sms * kCtas * kWarps * queue_chunks(core) * 16;
}

// (the second list's place holds a whole walk's states)
static_assert((uint64_t)kWalkListed * 3 * sizeof(Chunk) >= 256ull * kCtas * kWarps * sizeof(WalkState), "states");

uint64_t walk_list_bytes(uint32_t core) { return 2ull * kWalkListed * (2 + tuple_chunks(core)) * 16; }

cudaError_t launch_walk(const WalkArgs &args, bool lab, bool limited, Chunk *lists, int p, uint32_t kept, int sms,
                        cudaStream_t st) {
    const WalkArgs a = walk_pass(args, limited, lists, p, kept, sms);
    const uint32_t smem = walk_smem(a.core);
    if (p && !limited) {
        cudaMemsetAsync(a.out, 0, sizeof(WalkResult::List), st);
        cudaMemsetAsync(&a.result->kept, 0, sizeof(uint32_t), st);
        k_split<<<(a.state_warps + kWarps - 1) / kWarps, kWalkThreads, 0, st>>>(a);
    }
    walk_kernel(a, lab, limited ? kLimited : p ? kLater : kWhole)<<<a.ctas, kWalkThreads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace gfsm
