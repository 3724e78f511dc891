// cta_team.cuh -- the CTAs of a cluster that share one piece of work and add
// (XOR) their shares through distributed shared memory.
#pragma once
#include <cooperative_groups.h>

#include <cstdint>

namespace mtgp {

// CS = 1: a CTA on its own.
template <int CS>
struct Team {
    int rank = 0;
    __device__ Team() {
        if constexpr (CS > 1) rank = (int)cooperative_groups::this_cluster().block_rank();
    }
    // A barrier of all CTAs.
    __device__ void sync() const {
        if constexpr (CS > 1) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
    // The sum of a word over the CTAs' copies.
    template <typename W>
    __device__ W sum(W *p) const {
        if constexpr (CS == 1) {
            return *p;
        } else {
            W v = 0;
#pragma unroll
            for (int r = 0; r < CS; r++) v ^= *cooperative_groups::this_cluster().map_shared_rank(p, r);
            return v;
        }
    }
};

// CTAs per team for n teams at once: as many as leave one per SM, with a
// quarter of the SMs to spare, as a cluster needs its SMs close together (16
// teams of eight no longer run side by side).
inline int teamSize(int n, int sms) {
    const int room = sms - sms / 4;
    return 8 * n <= room ? 8 : 4 * n <= room ? 4 : 2 * n <= room ? 2 : 1;
}

// Launch `kern` on n teams of `cs` CTAs.
template <class K, class... Args>
cudaError_t launchTeams(K kern, int n, int cs, int threads, size_t smem, cudaStream_t s,
                        Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(n * cs));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)cs;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = cs > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// SMs of the current device.
inline int smCount() {
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace mtgp
