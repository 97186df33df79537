// The launch of room_steps, for the unit that compiles it in each field type.
#pragma once

#include "launch.h"

namespace pm {

// One cluster of room_steps: its launch, and the largest one that holds a room.
template <typename Real>
static cudaError_t room_steps_config(cudaLaunchConfig_t& c, cudaLaunchAttribute& at, int blocks, size_t smem, cudaStream_t s) {
    if (cudaError_t e = allow_smem(room_steps<Real>, (int)smem); e != cudaSuccess) return e;
    if (blocks > 8)
        if (cudaError_t e = cudaFuncSetAttribute(room_steps<Real>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            e != cudaSuccess)
            return e;
    c = cudaLaunchConfig_t{};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(kRoomThreads + 32);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaSuccess;
}
template <typename Real>
cudaError_t launch_room_steps(const RoomStepsArgs<Real>& a, int blocks, cudaStream_t s) {
    cudaLaunchConfig_t c;
    cudaLaunchAttribute at;
    if (cudaError_t e = room_steps_config<Real>(c, at, blocks, room_steps_smem<Real>(a.nx, a.rows), s); e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&c, room_steps<Real>, a);
}
template <typename Real>
int room_steps_cluster(int nx, int ny, int* rows) {
    for (int blocks = kRoomMaxCluster; blocks >= 1; blocks /= 2) {
        if (blocks > ny) continue;
        *rows = (ny + blocks - 1) / blocks;
        const size_t smem = room_steps_smem<Real>(nx, *rows);
        if (smem > 200 * 1024) break;  // a smaller cluster's blocks hold more rows
        cudaLaunchConfig_t c;
        cudaLaunchAttribute at;
        int fit = 0;
        if (room_steps_config<Real>(c, at, blocks, smem, nullptr) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&fit, room_steps<Real>, &c) == cudaSuccess && fit > 0)
            return blocks;
        cudaGetLastError();  // a cluster the device does not take is not an error of the stream
    }
    return 0;
}

}  // namespace pm
