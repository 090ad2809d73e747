// getrs_tc.cu -- FP64 solves with LU factors of orders above 64 on the tensor cores: kernel and
// host dispatch (the sweeps and their design in tri_solve.cuh). One block per matrix and group
// of eight right-hand sides: the groups of one matrix run side by side.
#include "internal.h"
#include "tri_solve.cuh"
#include "batched_kernels.h"
#include "lu_sizes.h"
#include "vbatched.h"
#include <algorithm>

namespace mb200 {

// Dynamic shared memory: X (NMAX x 8), the two staged blocks, the pivots.
template <int NMAX>
constexpr size_t getrs_tc_smem() {
    return sizeof(double) * NMAX * kTriRhs + sizeof(TriStage) + sizeof(int) * NMAX;
}

// Registers for five blocks of 64 threads an SM (168 a thread, 136 bytes of spills) rather than for
// four (253, none): 2,000 x 128^2, 8 RHS 210 against 255 us; n = 65, 128 against 150.
template <int NMAX, int NT>
__global__ void __launch_bounds__(NT, (NT == 64 ? 5 : NT == 128 ? 4 : 2))
getrs_tc_kernel(WorkList wl, LuSizes sz, bool trans, double** dA_array, int** ipiv_array, double** dB_array) {
    constexpr int NW = NT / 32, RPT = NMAX / NT;
    extern __shared__ __align__(16) unsigned char getrs_tc_raw[];
    double* X = reinterpret_cast<double*>(getrs_tc_raw);
    TriStage& dg = *reinterpret_cast<TriStage*>(X + NMAX * kTriRhs);
    int* piv = reinterpret_cast<int*>(&dg + 1);
    const BlockTeam team;
    const int tid = threadIdx.x;
    for (int w = blockIdx.x; w < wl.size(); w += gridDim.x) {
        const int id = wl.at(w);
        const int n = sz.get_n(id), lda = sz.get_lda(id), ldb = sz.get_ldb(id), nrhs = sz.get_nrhs(id);
        if (n <= 0 || (int)blockIdx.y * kTriRhs >= nrhs) continue;
        const double* A = dA_array[id];
        double* B = dB_array[id];
        const int* ipiv = ipiv_array ? ipiv_array[id] : nullptr;   // no pivots: identity
        // idx[j]: where row tid + j NT of B sits after DLASWP (NoTrans: forward; trans: inverse order)
        int idx[RPT];
#pragma unroll
        for (int j = 0; j < RPT; ++j) idx[j] = tid + j * NT;
        if (ipiv) {
            for (int k = tid; k < n; k += NT) piv[k] = ipiv[k] - 1;
            __syncthreads();
            for (int kk = 0; kk < n; ++kk) {
                const int k = trans ? n - 1 - kk : kk;
                const int p = piv[k];
#pragma unroll
                for (int j = 0; j < RPT; ++j) idx[j] = idx[j] == k ? p : idx[j] == p ? k : idx[j];
            }
        }
        const int npad = (n + 31) / 32 * 32;
        for (int c0 = blockIdx.y * kTriRhs; c0 < nrhs; c0 += gridDim.y * kTriRhs) {
#pragma unroll
            for (int j = 0; j < RPT; ++j) {
                const int t = tid + j * NT;
                if (t < npad) {
                    const int row = trans || t >= n ? t : idx[j];
#pragma unroll
                    for (int r = 0; r < kTriRhs; ++r)
                        X[tri_x(row, r)] = (t < n && c0 + r < nrhs) ? B[t + (size_t)(c0 + r) * ldb] : 0.0;
                }
            }
            __syncthreads();
            if (!trans) {
                tri_sweep<TriDiag::Unit, false>(A, 1, lda, n, X, dg, NW, team);
                tri_sweep<TriDiag::Divide, true>(A, 1, lda, n, X, dg, NW, team);
            } else {   // U^T (lower), then L^T (upper)
                tri_sweep<TriDiag::Divide, false>(A, lda, 1, n, X, dg, NW, team);
                tri_sweep<TriDiag::Unit, true>(A, lda, 1, n, X, dg, NW, team);
            }
#pragma unroll
            for (int j = 0; j < RPT; ++j) {
                const int t = tid + j * NT;
                if (t < n) {
#pragma unroll
                    for (int r = 0; r < kTriRhs; ++r)
                        if (c0 + r < nrhs) {
                            if (trans) B[idx[j] + (size_t)(c0 + r) * ldb] = X[tri_x(t, r)];
                            else       B[t + (size_t)(c0 + r) * ldb] = X[tri_x(t, r)];
                        }
                }
            }
            __syncthreads();
        }
    }
}

template <int NMAX, int NT>
static void launch_getrs_tc(const WorkList& wl, int bound, bool persistent, const LuSizes& sz, bool trans,
                            int max_nrhs, double** A, int** ipiv, double** B, cudaStream_t s) {
    auto k = getrs_tc_kernel<NMAX, NT>;
    const size_t smem = getrs_tc_smem<NMAX>();
    ensure_dynamic_smem((const void*)k, (int)smem);
    int gx = bound;
    if (persistent) gx = std::min(bound, resident_blocks((const void*)k, NT, smem));
    // At most four groups side by side: a matrix's pivots are replayed by each of its blocks. That
    // pays with as many matrices as SMs (148 x 1024^2, 128 RHS 5,260 us, with sixteen groups 5,535);
    // few matrices with many right-hand sides would gain from more (16 x 1024^2, 40 and 128 RHS 933
    // and 1,770 us, with sixteen 476 and 582), and two groups lose there (1,403 and 3,659).
    const int gy = std::min(4, ceildiv(std::max(1, max_nrhs), kTriRhs));
    k<<<dim3(std::max(1, gx), gy), NT, smem, s>>>(wl, sz, trans, A, ipiv, B);
}

magma_int_t getrs_tc(const WorkList& wl, int bound, bool persistent, bool trans, const LuSizes& sz, int max_n,
                     int max_nrhs, double** A, int** ipiv, double** B, cudaStream_t s) {
    if (max_n <= 128) launch_getrs_tc<128, 64>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
    else if (max_n <= 256) launch_getrs_tc<256, 128>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
    else if (max_n <= 512) launch_getrs_tc<512, 256>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
    else launch_getrs_tc<1024, 256>(wl, bound, persistent, sz, trans, max_nrhs, A, ipiv, B, s);
    return launch_status();
}

}  // namespace mb200
