// Thread-block clusters: access to the other CTAs' shared memory and the
// barrier the cluster kernels (hard-stretch solve, differentiable rollout)
// step by.
#pragma once

#include <cooperative_groups.h>

#include "xpbd_math.cuh"

namespace xg {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Loads and stores by row address (16-byte rows, so the low four bits are
// free): kOwnBit marks the own CTA's memory, which is read as plain shared
// memory (the cluster window's path is slower even for it).  kOne: a cluster
// of one CTA.
constexpr unsigned kOwnBit = 8u;
template <bool kOne>
__device__ __forceinline__ float4 ld_cluster(unsigned addr) {
    float4 x;
    if (kOne || (addr & kOwnBit))
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(addr & ~kOwnBit) : "memory");
    else
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(addr) : "memory");
    return x;
}
template <bool kOne>
__device__ __forceinline__ void st_cluster(unsigned addr, float4 x) {
    if (kOne || (addr & kOwnBit))
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr & ~kOwnBit), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
    else
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
}

// Where vertex l (counted from the cloth's first) lives: CTA l / chunk, float4
// slot l % chunk of an array at `base` of its shared memory.  The quotient is
// taken by the multiplier ceil(2^32 / chunk), exact for l < 2^16 with chunk a
// multiple of 32.
template <bool kOne>
struct ClusterMap {
    unsigned base;
    int chunk;
    unsigned mult, rank;
    __device__ __forceinline__ ClusterMap(unsigned b, int c, int r)
        : base(b), chunk(c), mult(0xffffffffu / (unsigned)c + 1u), rank((unsigned)r) {}
    __device__ __forceinline__ unsigned addr(int l) const {
        if (kOne) return (base + ((unsigned)l << 4)) | kOwnBit;
        const unsigned r = __umulhi((unsigned)l, mult), a = base + (((unsigned)l - r * chunk) << 4);
        return r == rank ? (a | kOwnBit) : map_rank(a, r);
    }
};

// Barrier of a cluster: one thread per CTA arrives at every CTA's counter
// after its own CTA's barrier; every thread then waits on its own counter
// (initialised for `ctas` arrivals).  The waits are bounded: when one runs
// out the thread waits no more (`lost`), so the kernel ends, and end() tells
// every thread of the cluster, which then writes no result but reports it.
struct ClusterBarrier {
    unsigned counter, parity;
    int ctas;
    bool lost;
    // Every CTA's counter is set before the first arrival: call once, by all
    // threads, before a cluster-wide synchronisation.
    static __device__ __forceinline__ void init(unsigned long long* counter, int arrivals) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(counter)), "r"(arrivals) : "memory");
    }
    static __device__ __forceinline__ void init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        if (ctas > 1 && (int)threadIdx.x < ctas)
            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_rank(counter, threadIdx.x)) : "memory");
    }
    __device__ __forceinline__ void finish() {
        if (ctas == 1) return;
        wait(counter, parity);
        parity ^= 1u;
    }
    __device__ __forceinline__ void sync() {
        arrive();
        finish();
    }
    __device__ __forceinline__ void wait(unsigned bar, unsigned phase) {
        unsigned done = lost ? 1u : 0u;
        for (int tries = 0; !done; ++tries) {
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 100000;\nselp.u32 %0, 1, 0, p;\n}"
                : "=r"(done)
                : "r"(bar), "r"(phase)
                : "memory");
            if (!done && tries > 20000) lost = true, done = 1u;
        }
    }
    // sync that also tells every CTA whether `mark` (of the own CTA, written
    // before) holds `epoch` in some CTA; `any` is the cluster's answer, in one
    // of two places by turns: the next answer may be written while a slower
    // CTA still reads this one.  The CTA's threads agree on it, also where a
    // wait gave up: what they do next has block barriers.
    __device__ __forceinline__ bool sync_any(const volatile int* mark, volatile int* any, int epoch) {
        if (ctas == 1) return __syncthreads_or(*mark == epoch);
        __syncthreads();
        if ((int)threadIdx.x < ctas && *mark == epoch)
            asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(map_rank(smem_addr((const void*)any), threadIdx.x)), "r"(epoch) : "memory");
        sync();
        return __syncthreads_or(*any == epoch);
    }
    // The last barrier of a kernel: afterwards no CTA addresses another's
    // shared memory.  The hardware's, which waits for every thread of the
    // cluster (all come here, since every wait before is bounded).  Returns
    // whether a wait of some thread of the cluster gave up; `mark` is a word
    // of each CTA, zero since before the first arrival.
    __device__ __forceinline__ bool end(volatile int* mark) {
        if (lost)
            for (int r = 0; r < ctas; ++r)
                asm volatile("st.shared::cluster.s32 [%0], 1;" ::"r"(map_rank(smem_addr((const void*)mark), r)) : "memory");
        __syncwarp();
        if (ctas > 1)
            cooperative_groups::this_cluster().sync();
        else
            __syncthreads();
        return *mark != 0;
    }
};

// Clusters of c CTAs of `threads` threads with `smem` bytes of dynamic shared
// memory that fit this GPU at once (0: the shape cannot run).  `limit` is the
// most that any launch of the kernel asks for: one value for every call.
template <class K>
int cluster_fit(K kernel, int c, int threads, size_t smem, size_t limit) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c, 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return fit;
}

template <class... A, class... B>
cudaError_t cluster_launch(void (*kernel)(A...), int clusters, int c, int threads, size_t smem, cudaStream_t s, B&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * c), 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<A>(args)...);
}

}  // namespace xg
