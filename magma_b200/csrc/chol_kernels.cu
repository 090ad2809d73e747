// chol_kernels.cu -- batched Cholesky kernels (fixed and variable size) and
// their host launchers. Device code in chol.cuh.
#include "internal.h"
#include "chol.cuh"
#include "chol_team.cuh"
#include "lu_sizes.h"
#include "vbatched.h"
#include "chol_launch.h"

namespace mb200 {

template <int NW> struct CholShape { static constexpr int MPB = (NW == 1) ? 4 : 1; };

// ---- register-resident potrf (+ optional fused potrs), thread = row ----
template <typename T, int NC, int NW, int R, bool SOLVE>
__global__ void __launch_bounds__(32 * NW * CholShape<NW>::MPB)
chol_small_kernel(WorkList wl, LuSizes sz, bool upper, T** dA_array, T** dB_array, int* info_array) {
    constexpr int MPB = CholShape<NW>::MPB;
    __shared__ CholShared<T, NC> shm[MPB];
    const int local = (NW == 1) ? (threadIdx.x >> 5) : 0;
    const int tid = (NW == 1) ? (threadIdx.x & 31) : threadIdx.x;
    for (int w = blockIdx.x * MPB + local; w < wl.size(); w += gridDim.x * MPB) {
        chol_small_instance<T, NC, NW, R, SOLVE>(wl.at(w), sz, upper, dA_array, dB_array, info_array, tid,
                                                 shm[local]);
        mat_sync<NW>();
    }
}

// ---- register-resident potrs only ----
template <typename T, int NC, int NW, int R>
__global__ void __launch_bounds__(32 * NW * CholShape<NW>::MPB)
potrs_small_kernel(WorkList wl, LuSizes sz, bool upper, T** dA_array, T** dB_array) {
    constexpr int MPB = CholShape<NW>::MPB;
    __shared__ CholShared<T, NC> shm[MPB];
    const int local = (NW == 1) ? (threadIdx.x >> 5) : 0;
    const int tid = (NW == 1) ? (threadIdx.x & 31) : threadIdx.x;
    for (int w = blockIdx.x * MPB + local; w < wl.size(); w += gridDim.x * MPB) {
        potrs_small_instance<T, NC, NW, R>(wl.at(w), sz, upper, dA_array, dB_array, tid, shm[local]);
        mat_sync<NW>();
    }
}

// ---- blocked FP64 potrf (orders above 512), one matrix per block ----
template <int NB, int NT>
__global__ void __launch_bounds__(NT, 1)
potrf_blocked_kernel(WorkList wl, LuSizes sz, bool upper, double** dA_array, int* info_array) {
    extern __shared__ __align__(16) unsigned char potrf_smem[];
    BlockedCholShared<NB, NT>& sh = *reinterpret_cast<BlockedCholShared<NB, NT>*>(potrf_smem);
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w);
        const int n = sz.get_n(id), lda = sz.get_lda(id);
        int info = 0;
        if (n > 0) info = blocked_potrf(dA_array[id], n, lda, upper, sh);
        if (threadIdx.x == 0 && info_array) info_array[id] = info;
        __syncthreads();
    }
}

// ---- potrf (n <= S) and FP64 potrs (n <= ROWS) by a block of S threads ----
// FP32: 768 threads an SM at 80 registers (228 bytes of spills), 1,024 at 64 for S = 512. Up to S =
// 256 neither 512 threads (128 registers, 28 bytes) nor 1,024 (64, 304 bytes) change the mixed call by
// more than 8% either way (1,000 orders 65..128, 1 RHS 361 us, 339 and 343; 10,000 of them 2,521,
// 2,520 and 2,502). At S = 512, two blocks an SM against one: 1,000 orders 257..512, 1 RHS 4,937 us
// and 5,000; 1,000 orders 4..512, 1 RHS, where other orders run beside them, 1,633 and 1,324.
template <typename T, int S>
__global__ void __launch_bounds__(S, (sizeof(T) == 4 ? (S == 512 ? 2 : 768 / S) : S <= 128 ? 4 : S == 256 ? 2 : 1))
potrf_team_kernel(WorkList wl, LuSizes sz, bool upper, T** dA_array, int* info_array) {
    const BlockTeam team;
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w), n = sz.get_n(id);
        int info = 0;
        if (n > 0) info = chol_team_potrf(dA_array[id], n, sz.get_lda(id), upper, 0u, S, team);
        if (threadIdx.x == 0 && info_array) info_array[id] = info;
        __syncthreads();
    }
}

template <int S, int ROWS>
__global__ void __launch_bounds__(S, (S == 64 ? 5 : S == 128 ? 4 : 2))
potrs_team_kernel(WorkList wl, LuSizes sz, bool upper, double** dA_array, double** dB_array) {
    const BlockTeam team;
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w), n = sz.get_n(id);
        if (n > 0)
            chol_team_potrs(dA_array[id], n, sz.get_lda(id), upper, dB_array[id], sz.get_nrhs(id), sz.get_ldb(id),
                            0u, S, ROWS, blockIdx.y, gridDim.y, team);
    }
}

// ---------------------------------------------------------------------------
// Launchers. Each bucket launcher covers instances with n in (lo, hi].
template <typename K>
static int grid_for(K kernel, int threads, int items_upper_bound, bool bounded, size_t smem = 0) {
    if (!bounded) return max(1, items_upper_bound);
    const int res = resident_blocks((const void*)kernel, threads, smem);
    return max(1, min(items_upper_bound, res));
}

template <typename T, int NC, int NW>
static void launch_chol_small(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper,
                              T** A, T** B, int* info, bool solve, int max_nrhs, cudaStream_t s) {
    constexpr int MPB = CholShape<NW>::MPB;
    const int threads = 32 * NW * MPB;
    const int items = ceildiv(bound, MPB);
    auto launch = [&](auto k) {
        k<<<grid_for(k, threads, items, persistent), threads, 0, s>>>(wl, sz, upper, A, B, info);
    };
    if constexpr (std::is_same<T, float>::value) {   // the mixed solve's factor
        launch(chol_small_kernel<T, NC, NW, 1, false>);
    } else {
        if (!solve) launch(chol_small_kernel<T, NC, NW, 1, false>);
        else if (max_nrhs <= 1) launch(chol_small_kernel<T, NC, NW, 1, true>);
        else if (max_nrhs <= 4) launch(chol_small_kernel<T, NC, NW, 4, true>);
        else launch(chol_small_kernel<T, NC, NW, 8, true>);
    }
}

template <typename T, int NC, int NW>
static void launch_potrs_small(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper,
                               T** A, T** B, int max_nrhs, cudaStream_t s) {
    constexpr int MPB = CholShape<NW>::MPB;
    const int threads = 32 * NW * MPB;
    const int items = ceildiv(bound, MPB);
    if (max_nrhs <= 1) {
        auto k = potrs_small_kernel<T, NC, NW, 1>;
        k<<<grid_for(k, threads, items, persistent), threads, 0, s>>>(wl, sz, upper, A, B);
    } else if (max_nrhs <= 4) {
        auto k = potrs_small_kernel<T, NC, NW, 4>;
        k<<<grid_for(k, threads, items, persistent), threads, 0, s>>>(wl, sz, upper, A, B);
    } else {
        auto k = potrs_small_kernel<T, NC, NW, 8>;
        k<<<grid_for(k, threads, items, persistent), threads, 0, s>>>(wl, sz, upper, A, B);
    }
}

template <typename T, int S>
static void launch_potrf_team(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper, T** A,
                              int* info, cudaStream_t s) {
    auto k = potrf_team_kernel<T, S>;
    const int smem = (int)(sizeof(T) == 8 ? chol_team_smem(S) : sizeof(T) * (32 * S + 32 * 33 + 32) + 16);
    ensure_dynamic_smem((const void*)k, smem);
    k<<<grid_for(k, S, bound, persistent, smem), S, smem, s>>>(wl, sz, upper, A, info);
}

static void launch_potrf_blocked(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper,
                                 double** A, int* info, cudaStream_t s) {
    constexpr int NB = 16, NT = 1024;
    auto k = potrf_blocked_kernel<NB, NT>;
    const int smem = (int)sizeof(BlockedCholShared<NB, NT>);
    ensure_dynamic_smem((const void*)k, smem);
    k<<<grid_for(k, NT, bound, persistent, smem), NT, smem, s>>>(wl, sz, upper, A, info);
}

// FP64 potrs of orders up to ROWS; threads as the LU solves (getrs_tc.cu).
template <int ROWS>
static void launch_potrs_team(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper,
                              double** A, double** B, int max_nrhs, cudaStream_t s) {
    constexpr int S = ROWS < 256 ? ROWS / 2 : ROWS == 256 ? 128 : 256;
    auto k = potrs_team_kernel<S, ROWS>;
    const int smem = (int)(sizeof(double) * kTriRhs * ROWS + sizeof(TriStage));
    ensure_dynamic_smem((const void*)k, smem);
    const int gy = min(4, ceildiv(max(1, max_nrhs), kTriRhs));   // as the LU solves
    k<<<dim3(grid_for(k, S, bound, persistent, smem), gy), S, smem, s>>>(wl, sz, upper, A, B);
}

// Size buckets shared by the Cholesky launchers (upper edges, inclusive).
const int kCholEdges[kCholBuckets] = {8, 16, 32, 64, 128, 256, 512, 1024};

// FP32 is the mixed solve's factor: orders up to 512, no solve.
template <>
void chol_bucket<float>(int b, const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper, float** A,
                        float** B, int* info, bool, bool, int, cudaStream_t s) {
    switch (b) {
        case 0: launch_chol_small<float, 8, 1>(wl, bound, persistent, sz, upper, A, B, info, false, 0, s); break;
        case 1: launch_chol_small<float, 16, 1>(wl, bound, persistent, sz, upper, A, B, info, false, 0, s); break;
        case 2: launch_chol_small<float, 32, 1>(wl, bound, persistent, sz, upper, A, B, info, false, 0, s); break;
        case 3: launch_chol_small<float, 64, 2>(wl, bound, persistent, sz, upper, A, B, info, false, 0, s); break;
        case 4: launch_potrf_team<float, 128>(wl, bound, persistent, sz, upper, A, info, s); break;
        case 5: launch_potrf_team<float, 256>(wl, bound, persistent, sz, upper, A, info, s); break;
        default: launch_potrf_team<float, 512>(wl, bound, persistent, sz, upper, A, info, s); break;
    }
}

template <>
void chol_bucket<double>(int b, const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool upper,
                         double** A, double** B, int* info, bool factor, bool solve, int max_nrhs, cudaStream_t s) {
    using T = double;
    if (factor) {
        switch (b) {
            case 0: launch_chol_small<T, 8, 1>(wl, bound, persistent, sz, upper, A, B, info, solve, max_nrhs, s); break;
            case 1: launch_chol_small<T, 16, 1>(wl, bound, persistent, sz, upper, A, B, info, solve, max_nrhs, s); break;
            case 2: launch_chol_small<T, 32, 1>(wl, bound, persistent, sz, upper, A, B, info, solve, max_nrhs, s); break;
            case 3: launch_chol_small<T, 64, 2>(wl, bound, persistent, sz, upper, A, B, info, solve, max_nrhs, s); break;
            case 4: launch_potrf_team<T, 128>(wl, bound, persistent, sz, upper, A, info, s); break;
            case 5: launch_potrf_team<T, 256>(wl, bound, persistent, sz, upper, A, info, s); break;
            case 6: launch_potrf_team<T, 512>(wl, bound, persistent, sz, upper, A, info, s); break;
            default: launch_potrf_blocked(wl, bound, persistent, sz, upper, A, info, s); break;
        }
        if (!solve || b <= 3) return;   // small buckets fuse the solve into the factor kernel
    }
    switch (b) {
        case 0: launch_potrs_small<T, 8, 1>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 1: launch_potrs_small<T, 16, 1>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 2: launch_potrs_small<T, 32, 1>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 3: launch_potrs_small<T, 64, 2>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 4: launch_potrs_team<128>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 5: launch_potrs_team<256>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        case 6: launch_potrs_team<512>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
        default: launch_potrs_team<1024>(wl, bound, persistent, sz, upper, A, B, max_nrhs, s); break;
    }
}

int chol_bucket_of(int n) {
    for (int b = 0; b < kCholBuckets; ++b)
        if (n <= kCholEdges[b]) return b;
    return -1;
}

}  // namespace mb200
