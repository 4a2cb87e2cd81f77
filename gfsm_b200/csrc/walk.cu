// walk.cu -- memory and launches of the walk (walk_kernel.cuh).
#include <cuda_runtime.h>

#include "walk_kernel.cuh"

namespace gfsm {

uint64_t walk_queue_bytes(uint32_t core, int sms) {
    return (uint64_t)sms * kCtas * kWarps * queue_chunks(core) * 16;
}

uint64_t walk_list_bytes(uint32_t core) { return 2ull * kWalkListed * (2 + tuple_chunks(core)) * 16; }

cudaError_t launch_walk(const WalkArgs &args, bool lab, bool limited, Chunk *lists, int sms, cudaStream_t st) {
    WalkArgs a = args;
    const uint32_t smem = walk_smem(a.core);
    a.warp_chunks = queue_chunks(a.core);
    const WalkShape shape = walk_shape(a.units, a.roots, limited, sms);
    a.chunk = shape.chunk;
    Chunk *const list[2] = {lists, lists + (size_t)kWalkListed * (2 + tuple_chunks(a.core))};
    for (int p = 0; p < (limited ? kWalkPasses : 1); ++p) {
        a.pass = (uint32_t)p;
        a.max_rounds = limited ? kWalkRounds[p] : 0;
        a.list_in = p ? list[(p - 1) & 1] : nullptr;
        a.list_out = limited && p + 1 < kWalkPasses ? list[p & 1] : nullptr;
        a.last = p + 1 == (limited ? kWalkPasses : 1);
        const uint32_t ctas = p ? (uint32_t)sms * kCtas : shape.ctas;
        if (a.rows && lab) k_walk<true, false, true><<<ctas, kWalkThreads, smem, st>>>(a);
        else if (a.rows) k_walk<false, false, true><<<ctas, kWalkThreads, smem, st>>>(a);
        else if (lab && limited) k_walk<true, true, false><<<ctas, kWalkThreads, smem, st>>>(a);
        else if (lab) k_walk<true, false, false><<<ctas, kWalkThreads, smem, st>>>(a);
        else if (limited) k_walk<false, true, false><<<ctas, kWalkThreads, smem, st>>>(a);
        else k_walk<false, false, false><<<ctas, kWalkThreads, smem, st>>>(a);
    }
    return cudaGetLastError();
}

}  // namespace gfsm
