// How the attention kernels share out the items beyond whole waves of one per SM: each to a cluster whose
// CTAs take a part of the item's steps (kv tiles forward, query blocks backward) and join their results.
#pragma once

#include "host_util.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

namespace fu {

inline cudaLaunchAttribute cluster_attr(int csize)
{
    cudaLaunchAttribute attr = {};
    attr.id                  = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x    = static_cast<unsigned>(csize);
    attr.val.clusterDim.y    = 1;
    attr.val.clusterDim.z    = 1;
    return attr;
}

// How many clusters of `csize` CTAs of a kernel the device holds at once (a cluster stays inside a GPC);
// 0 when it cannot be asked. Asked once per device and size; also raises the kernel's shared-memory limit.
class ClusterCapacity {
public:
    template <typename Kernel>
    int of(Kernel kernel, int csize, int dev, int threads, int smem_bytes)
    {
        if (dev < 0 || dev >= 64) {
            return 0;
        }
        const std::lock_guard<std::mutex> guard(lock_);
        if (cached_[dev][csize] == 0) {
            cudaLaunchConfig_t  cfg  = {};
            cudaLaunchAttribute attr = cluster_attr(csize);
            cfg.gridDim              = dim3(static_cast<unsigned>(csize), 1, 1);
            cfg.blockDim             = dim3(static_cast<unsigned>(threads), 1, 1);
            cfg.dynamicSmemBytes     = static_cast<size_t>(smem_bytes);
            cfg.attrs                = &attr;
            cfg.numAttrs             = 1;
            int n                    = 0;
            if (raise_smem_limit(kernel, smem_bytes) != FU_OK || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                (void)cudaGetLastError();
                n = -1;
            }
            cached_[dev][csize] = n;
        }
        return std::max(0, cached_[dev][csize]);
    }

private:
    std::mutex lock_;
    int        cached_[64][9] = {};
};

struct ClusterPlan {
    int    whole, csize;  // items of the plain kernel; cluster size of the rest (1: no split)
    double cost;          // in steps
};
// Measured, in steps: what an item costs beyond its own steps (launch, first loads, write-out), what the
// exchange of a cluster adds, and what a second launch does.
struct ClusterCosts {
    double item, exchange, launch;
};

template <typename Capacity>
ClusterPlan plan_clusters(int items, int steps, int sms, const ClusterCosts& cost, Capacity capacity)
{
    const int   whole = items / sms * sms, rest = items - whole;
    ClusterPlan best{items, 1, static_cast<double>((items + sms - 1) / sms) * (steps + cost.item)};
    if (rest == 0) {
        return best;
    }
    for (const int csize : {2, 3, 4, 5, 6, 8}) {
        const int share = (steps + csize - 1) / csize;
        if (csize > steps || (steps + share - 1) / share != csize) {
            continue;  // a CTA would have nothing to do
        }
        const int cap = capacity(csize);
        if (cap < 1) {
            continue;
        }
        const double c = static_cast<double>(whole / sms) * (steps + cost.item)
                         + static_cast<double>((rest + cap - 1) / cap) * (share + cost.item + cost.exchange) + (whole > 0 ? cost.launch : 0.0);
        if (c < best.cost) {
            best = {whole, csize, c};
        }
    }
    return best;
}

}  // namespace fu
