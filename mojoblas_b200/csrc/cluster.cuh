// Thread-block clusters: a CTA's place in its cluster, the cluster barrier, reads of another
// CTA's shared memory, and the launch attributes.
#pragma once

#include "mbg_internal.cuh"

namespace mbg {
namespace clu {

constexpr int MAX_CTAS = 8;  // CTAs per cluster that any device takes

__device__ __forceinline__ uint32_t rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Every thread of every CTA of the cluster.  The aligned forms want a converged warp, which a loop
// with different trips per lane, or a lane's early `continue`, does not promise.
__device__ __forceinline__ void sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address in CTA `r`'s shared memory of what sits at `addr` in this one's.
__device__ __forceinline__ uint32_t peer(uint32_t addr, uint32_t r) {
    uint32_t v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(addr), "r"(r));
    return v;
}
__device__ __forceinline__ float4 load4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}
__device__ __forceinline__ double2 load2(uint32_t addr) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}

// SMs that clusters of S CTAs, one per SM, can fill at once on a B200 (what
// cudaOccupancyMaxActiveClusters reports, times S: the SMs come in groups of 16 to 20).
inline int usable_sms(int S) {
    constexpr int sms[MAX_CTAS + 1] = {0, 148, 148, 135, 132, 130, 132, 105, 120};
    return sms[S];
}

// A launch of `ctas` CTAs in clusters of S; pdl: as launch_pdl.
struct Launch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2]{};
    Launch(unsigned ctas, int S, int threads, size_t smem, cudaStream_t s, bool pdl = false) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(S);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(unsigned(threads));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 2 : 1;
    }
    Launch(const Launch&) = delete;
};

}  // namespace clu
}  // namespace mbg
