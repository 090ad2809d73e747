// getrf_blocked.cu -- kernels and host dispatch of the blocked batched LU
// (one matrix per thread block, up to 1024 rows): FP32, and in FP64 the factors of tall matrices
// (getrf_tall) and many solves of one right-hand side. Other FP64 calls run getrf_cluster.cu and
// getrs_tc.cu.
#include "internal.h"
#include "blocked_lu.cuh"
#include "getrs_blocked.cuh"
#include "batched_kernels.h"
#include "lu_sizes.h"
#include "vbatched.h"
#include <type_traits>

namespace mb200 {

// Resident blocks per SM the register allocation is sized for.
template <typename T, int NT>
constexpr int blocked_min_blocks() {
    return NT <= 128 ? 4 : NT == 256 ? (sizeof(T) == 8 ? 2 : 3) : 1;
}

template <typename T, int NB, int NT, int CW, int CB>
__global__ void __launch_bounds__(NT, (blocked_min_blocks<T, NT>()))
getrf_blocked_kernel(WorkList wl, LuSizes sz, T** dA_array, int** ipiv_array, int* info_array) {
    extern __shared__ __align__(16) unsigned char getrf_smem[];
    BlockedLuShared<T, NB, NT, CW>& sh = *reinterpret_cast<BlockedLuShared<T, NB, NT, CW>*>(getrf_smem);
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w);
        const int m = sz.get_m(id), n = sz.get_n(id), lda = sz.get_lda(id);
        int info = 0;
        if (m > 0 && n > 0)   // a null pivot array selects LU without pivoting (getrf_nopiv)
            blocked_getrf<T, NB, NT, CW, CB>(dA_array[id], m, n, lda, ipiv_array ? ipiv_array[id] : nullptr,
                                                  info, sh);
        if (threadIdx.x == 0) info_array[id] = info;
        __syncthreads();
    }
}

template <typename T, int NT, int R>
__global__ void __launch_bounds__(NT)
getrs_blocked_kernel(WorkList wl, LuSizes sz, bool trans, T** dA_array, int** ipiv_array, T** dB_array) {
    __shared__ BlockedRsShared<T, NT, R> sh;
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w);
        const int n = sz.get_n(id), lda = sz.get_lda(id), ldb = sz.get_ldb(id), nrhs = sz.get_nrhs(id);
        if (n > 0 && nrhs > 0)
            blocked_getrs<T, NT, R>(trans, dA_array[id], n, lda, ipiv_array ? ipiv_array[id] : nullptr,
                                    dB_array[id], nrhs, ldb, sh);
        __syncthreads();
    }
}

bool blocked_lu_supported(int max_m) { return max_m <= 1024; }

template <typename K>
static int blocked_grid(K kernel, int threads, int bound, bool persistent, size_t smem = 0) {
    if (!persistent) return std::max(1, bound);
    return std::max(1, std::min(bound, resident_blocks((const void*)kernel, threads, smem)));
}

template <typename T, int NB, int NT, int CW, int CB>
static void launch_getrf_blocked(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, T** A, int** ipiv,
                                 int* info, cudaStream_t s) {
    auto k = getrf_blocked_kernel<T, NB, NT, CW, CB>;
    const int smem = (int)sizeof(BlockedLuShared<T, NB, NT, CW>);
    ensure_dynamic_smem((const void*)k, smem);
    k<<<blocked_grid(k, NT, bound, persistent, smem), NT, smem, s>>>(wl, sz, A, ipiv, info);
}

// FP64 matrices of more rows than one block of the cluster kernel holds, but few columns: nearly all
// of their time is panel steps, which cross the cluster there and cost one block's barrier here.
// Measured, this kernel against the cluster (us):
//   257..512 rows (two blocks a matrix): 2,000 x (300 x 32) 341 against 634, (512 x 128) 2,898
//   against 3,390, (512 x 192) 5,705 against 6,050; 16 x (300 x 96) 124 against 135, (300 x 128)
//   182 against 182, (300 x 192) 334 against 284;
//   513..1024 rows (four blocks): 2,000 x (1024 x 8) 191 against 432, (1024 x 96) 4,293 against
//   5,620, 300 x (1024 x 128) 1,418 against 1,361; 16 x (600 x 16) 26 against 30, (1024 x 32) 60
//   against 48.
// The lines lie where the two meet. They move with the matrices per SM: up to half a matrix an SM, a
// cluster's blocks have SMs to themselves; from there on they share them, and what counts is the work
// of all. 2,000 x (600 x 128) 5,074 against 6,982, (800 x 160) 9,063 against 9,812; 100 x (600 x 128)
// 366 against 473.
static bool getrf_tall(int max_m, int max_n, int bound) {
    if (max_m <= 256) return false;
    const float per_sm = (float)bound / device_sm_count();
    if (max_m <= 512) return max_n <= (per_sm > 4 ? 192 : per_sm > 0.5f ? 160 : 96);
    if (per_sm > 0.5f && per_sm <= 1) return max_n <= 128;   // one wave of blocks, two of clusters
    return max_n <= (per_sm > 6 ? 160 : per_sm > 2 ? 128 : per_sm > 1 ? 96 : 16);
}

template <typename T>
magma_int_t getrf_blocked(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, int max_m, int max_n,
                          T** A, int** ipiv, int* info, cudaStream_t s) {
    if constexpr (std::is_same<T, double>::value) {
        if (getrf_tall(max_m, max_n, bound)) {
            if (max_m <= 512) launch_getrf_blocked<T, 32, 512, 128, 8>(wl, bound, persistent, sz, A, ipiv, info, s);
            else launch_getrf_blocked<T, 16, 1024, 128, 2>(wl, bound, persistent, sz, A, ipiv, info, s);
            return launch_status();
        }
        return getrf_cluster(wl, bound, persistent, sz, max_m, A, ipiv, info, s);
    } else {
        if (max_m <= 128) launch_getrf_blocked<T, 32, 128, 128, 16>(wl, bound, persistent, sz, A, ipiv, info, s);
        else if (max_m <= 256) launch_getrf_blocked<T, 32, 256, 128, 8>(wl, bound, persistent, sz, A, ipiv, info, s);
        else if (max_m <= 512) launch_getrf_blocked<T, 32, 512, 128, 8>(wl, bound, persistent, sz, A, ipiv, info, s);
        else launch_getrf_blocked<T, 16, 1024, 128, 4>(wl, bound, persistent, sz, A, ipiv, info, s);
        return launch_status();
    }
}

template <typename T, int NT>
static void launch_getrs_blocked(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool trans,
                                 int max_nrhs, T** A, int** ipiv, T** B, cudaStream_t s) {
    if (max_nrhs <= 1) {
        auto k = getrs_blocked_kernel<T, NT, 1>;
        k<<<blocked_grid(k, NT, bound, persistent), NT, 0, s>>>(wl, sz, trans, A, ipiv, B);
    } else {
        auto k = getrs_blocked_kernel<T, NT, 4>;
        k<<<blocked_grid(k, NT, bound, persistent), NT, 0, s>>>(wl, sz, trans, A, ipiv, B);
    }
}

template <typename T>
magma_int_t getrs_blocked(const WorkList& wl, int bound, bool persistent, bool trans, const LuSizes& sz, int max_n,
                          int max_nrhs, T** A, int** ipiv, T** B, cudaStream_t s) {
    if constexpr (std::is_same<T, double>::value) {
        // One right-hand side fills one of the sweeps' eight columns. That costs nothing while every
        // matrix has its block at once, which is up to five an SM; more matrices of one right-hand
        // side are through sooner with a thread per row (n = 65 and 128, this form against the
        // sweeps: 740 matrices 78 against 50 us and 118 against 81; 900, 77 against 80 and 124
        // against 146; 2,000, 81 against 129 and 148 against 211; above 128 rows the sweeps win,
        // 2,000 x 140^2 326 against 287).
        if (max_nrhs <= 1 && max_n <= 128 && bound > 5 * device_sm_count()) {
            auto k = getrs_blocked_kernel<T, 128, 1>;
            k<<<blocked_grid(k, 128, bound, persistent), 128, 0, s>>>(wl, sz, trans, A, ipiv, B);
            return launch_status();
        }
        return getrs_tc(wl, bound, persistent, trans, sz, max_n, max_nrhs, A, ipiv, B, s);
    } else {
        if (max_n <= 128) launch_getrs_blocked<T, 128>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
        else if (max_n <= 256) launch_getrs_blocked<T, 256>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
        else if (max_n <= 512) launch_getrs_blocked<T, 512>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
        else launch_getrs_blocked<T, 1024>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
        return launch_status();
    }
}

template magma_int_t getrf_blocked<double>(const WorkList&, int, bool, const LuSizes&, int, int, double**, int**, int*,
                                           cudaStream_t);
template magma_int_t getrf_blocked<float>(const WorkList&, int, bool, const LuSizes&, int, int, float**, int**, int*,
                                          cudaStream_t);
template magma_int_t getrs_blocked<double>(const WorkList&, int, bool, bool, const LuSizes&, int, int, double**, int**,
                                           double**, cudaStream_t);
template magma_int_t getrs_blocked<float>(const WorkList&, int, bool, bool, const LuSizes&, int, int, float**, int**,
                                          float**, cudaStream_t);

}  // namespace mb200
