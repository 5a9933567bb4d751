// Instantiations of the tcgen05 implicit-GEMM kernel for a 128-byte K tile (swizzle 128B).
#include "tc_kernel.cuh"

namespace chxq {
namespace tc {

int launch_tc_bk128(int bn, int epi, int split, const CUtensorMap& tmA, const CUtensorMap& tmB, const TcParams& p, int grid, cudaStream_t s) {
    return launch_bk<128>(bn, epi, split, tmA, tmB, p, grid, s);
}

namespace {
template <int SPLIT>
int query_split_slots() {
    using Cfg = TcConfig<64, 128>;
    auto* kernel = tc_igemm_kernel<64, 128, kEpiKInt32, SPLIT>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SPLIT, 1, 1);
    cfg.blockDim = dim3(608, 1, 1);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = SPLIT; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;  // then nothing is split
    }
    return n;
}
}  // namespace

// Clusters of `split` CTAs of the one-tile kernel that the current device keeps resident at once.  (Every instantiation has one CTA per SM.)
int split_slots(int split) {
    static std::atomic<int> known[2][64] = {};  // per device, slots + 1; every writer stores the same value
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const int which = split == 4 ? 1 : 0;
    int v = dev >= 0 && dev < 64 ? known[which][dev].load(std::memory_order_acquire) : 0;
    if (v == 0) {
        v = 1 + (split == 4 ? query_split_slots<4>() : query_split_slots<2>());
        if (dev >= 0 && dev < 64) known[which][dev].store(v, std::memory_order_release);
    }
    return v - 1;
}

}  // namespace tc
}  // namespace chxq
