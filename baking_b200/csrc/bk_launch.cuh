// Programmatic dependent launch between the kernels of a substep and of its reverse: each is launched
// with programmatic stream serialisation (launch_chained), so the launch of the next kernel and the
// placement of its blocks overlap the tail of the one before it. Every such kernel first waits until
// the kernel before it in the stream has completed and its memory is visible (which makes the chain
// transitive), then lets the next kernel launch; its blocks only take SM slots left free by blocks
// already running. A kernel without a programmatic predecessor returns from the wait at once.
// Before the wait a kernel may only compute addresses and ask L2 for lines (prefetch_l2: a hint, whatever
// the kernel before it is still writing): the particle kernels do, so that their first loads find L2
// warm (elastic body of 41k particles 920 -> 872 us a 40-substep pass, 9k sphere 2106 -> 2049).
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <utility>

#include "baking_b200.h"
#include "bk_common.h"

namespace bk {

__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Blocks of a pass over the node box, whose size only the device knows: up to four per SM. A compact body
// is best served by one per 128 particles (9k sphere, 69 blocks: 46.9 us a substep, 49.6 with three per SM,
// 51.2 with four; 41k cube, 324 blocks: 22.3, with three per SM 24.3: the next kernel's blocks find emptier
// SMs), but a box may hold far more nodes than particles, up to the whole grid. So small bodies take three
// per SM where the grid has that many tiles of 256 nodes: two clumps of 324 particles across a 128^3 grid
// take 101 us a substep (two per SM: 112, four: 99; a block per 128 particles: 2000).
inline unsigned node_box_blocks(int64_t n, int resolution, int sms) {
    const int64_t grid = ((int64_t)resolution * resolution * resolution + 255) / 256;
    const int64_t few = std::max<int64_t>(std::min<int64_t>(grid, (int64_t)sms * 3), (n + 127) / 128);
    return (unsigned)std::min<int64_t>((int64_t)sms * 4, few);
}

// The status of a launch_chained call, as check_launch reports a launch's.
inline int check_chained(cudaError_t e, const char* name) {
    if (e == cudaSuccess) return check_launch(name);
    cudaGetLastError();
    char msg[256];
    snprintf(msg, sizeof msg, "%s: %s", name, cudaGetErrorString(e));
    return fail(BK_ERR_LAUNCH, msg);
}

template <class... KArgs, class... Args>
cudaError_t launch_chained(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                           Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace bk
