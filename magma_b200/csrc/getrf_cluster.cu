// getrf_cluster.cu -- kernel and host dispatch of the FP64 LU of one matrix per
// thread-block cluster (device code and design in cluster_lu.cuh).
#include "internal.h"
#include "cluster_lu.cuh"
#include "batched_kernels.h"
#include "lu_sizes.h"
#include "vbatched.h"
#include <algorithm>

namespace mb200 {

template <int NB, int NT, int CS>
__global__ void __launch_bounds__(NT, (NT <= 128 ? 4 : 2))
getrf_cluster_kernel(WorkList wl, LuSizes sz, double** dA_array, int** ipiv_array, int* info_array) {
    extern __shared__ __align__(16) unsigned char getrf_cluster_smem[];
    auto& sh = *reinterpret_cast<ClusterLuShared<NB, NT, CS>*>(getrf_cluster_smem);
    const int rank = CS == 1 ? 0 : (int)cooperative_groups::this_cluster().block_rank();
    // A block's first pivot candidate goes to its peers before anything of the panel makes the
    // cluster meet, and a peer's shared memory may be stored to only once that peer runs. The
    // barrier that ends each matrix does the same for the matrices after it, and for the exit.
    if constexpr (CS > 1) cluster_sync<CS>();
    for (int w = blockIdx.x / CS; w < wl.size(); w += gridDim.x / CS) {
        const int id = wl.at(w);
        const int m = sz.get_m(id), n = sz.get_n(id), lda = sz.get_lda(id);
        int info = 0;
        if (m > 0 && n > 0)   // a null pivot array selects LU without pivoting (getrf_nopiv)
            cluster_getrf<NB, NT, CS>(dA_array[id], m, n, lda, ipiv_array ? ipiv_array[id] : nullptr, info, rank, sh);
        if (threadIdx.x == 0 && rank == 0) info_array[id] = info;
    }
}

template <int NB, int NT, int CS>
static void launch_getrf_cluster(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, double** A,
                                 int** ipiv, int* info, cudaStream_t s) {
    auto k = getrf_cluster_kernel<NB, NT, CS>;
    const int smem = (int)sizeof(ClusterLuShared<NB, NT, CS>);
    ensure_dynamic_smem((const void*)k, smem);
    int clusters = bound;
    if (persistent) clusters = std::min(bound, std::max(1, resident_blocks((const void*)k, NT, smem) / CS));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)clusters * CS);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CS > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k, wl, sz, A, ipiv, info);
}

magma_int_t getrf_cluster(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, int max_m, double** A,
                          int** ipiv, int* info, cudaStream_t s) {
    // One thread per row: blocks of 256 threads (128 for the smallest orders, whose four blocks an
    // SM overlap their panel steps), as many blocks as the rows need. Blocks of 128 threads in
    // clusters twice as large lose: their panel steps cross the cluster (orders 256 and 512,
    // 1,024 matrices' worth of work: 5.2 against 3.1 ms, 11.7 against 7.1 ms).
    if (max_m <= 128) launch_getrf_cluster<32, 128, 1>(wl, bound, persistent, sz, A, ipiv, info, s);
    else if (max_m <= 256) launch_getrf_cluster<32, 256, 1>(wl, bound, persistent, sz, A, ipiv, info, s);
    else if (max_m <= 512) launch_getrf_cluster<32, 256, 2>(wl, bound, persistent, sz, A, ipiv, info, s);
    else launch_getrf_cluster<32, 256, 4>(wl, bound, persistent, sz, A, ipiv, info, s);
    return launch_status();
}

}  // namespace mb200
