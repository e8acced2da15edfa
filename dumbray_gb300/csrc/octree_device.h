// octree_device.h - a built octree in device memory: what scene creation makes its records from.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "octree_build.h"

namespace drb {

// Arrays as in FlatOctree; owned.
struct DeviceTree {
    float *xyz = nullptr;            // [n][3][3]
    float *lo = nullptr, *hi = nullptr;
    int32_t *child = nullptr;
    long long *leaf_first = nullptr;
    int32_t *leaf_count = nullptr;
    int32_t *refs = nullptr;
    DeviceTree() = default;
    DeviceTree(const DeviceTree &) = delete;
    DeviceTree &operator=(const DeviceTree &) = delete;
    ~DeviceTree() {
        for (void *p : {(void *)xyz, (void *)lo, (void *)hi, (void *)child, (void *)leaf_first, (void *)leaf_count, (void *)refs}) cudaFree(p);
    }
};

// build_octree_gpu that leaves the tree on the device as well (keep may be null).
bool build_octree_gpu(const float *xyz, int64_t n, const BuildOptions &opt, FlatOctree &out, DeviceTree *keep, std::string &err);

}  // namespace drb
