// chol_team.cuh -- blocked Cholesky (potrf; FP64 or FP32) and FP64 solve (potrs) of one matrix by a team of
// warps (a thread block, or a range of warps of the one-launch kernel), n <= the team's threads.
//
//   for each panel of 32 columns (k0 = 0, 32, ...):
//     1. warp 0 has factored the 32x32 diagonal block (lane = row, in registers) and left L11^T
//        and the reciprocals of its diagonal in shared memory;
//     2. every row below solves its 32 entries against L11 on its own, in registers (thread =
//        row, no barrier between steps), and publishes them;
//     3. the trailing triangle is updated on the FP64 tensor cores from the published rows, a
//        warp taking 16 rows x 64 columns with its rows' multipliers in registers and the next
//        16 columns of C in flight -- while warp 0 updates the next diagonal block and factors it.
// A panel has two team barriers, and the chain of 32 square roots and divisions runs beside the
// update. (With every row stepping through the panel together, each step was a team barrier.)
//
// What bounds it (clock stamps, cycles a panel): up to n = 256 the chain of the diagonal block in
// warp 0 (about 15,000 alone, 17,000 to 25,000 with the SM full; the rows' phase 4,000 to 6,000
// beside it); at n = 512 that chain and the update (30,000 to 37,000 each). Measured against
// every row stepping through the panel and a row-per-thread solve (one launch for all orders,
// 8 RHS): 2,000 x 128^2 posv 885 -> 590 us, 740 x 256^2 1,418 -> 827, 444 x 512^2 4,099 -> 2,250;
// 50,000 orders 4..512 13.6 -> 8.6 ms.
//
// FP32 (the mixed solve's factor) runs the same code with FP32 arithmetic, its updates as fma's on
// the CUDA cores: a warp takes 16 rows x 64 columns there too, 4 x 8 a lane.
//
// Per element the operations are those of chol_panel_steps: l(i,k) = a(i,k) * (1 / sqrt(d_k)),
// a(i,j) = fma(-l(i,k), l(j,k), a(i,j)) for ascending k, so factors, solutions and info are
// bit-identical to the oracle.
#pragma once

#include "chol.cuh"
#include "tri_solve.cuh"

namespace mb200 {

// Bytes of shared memory a team of S threads needs: P (32 x S) and the diagonal block for the
// factorisation; X (S x 8) and the staged blocks for the solve (p[1] unused at 64 threads).
constexpr size_t chol_team_smem(int S) {
    const size_t f = sizeof(double) * (32 * (size_t)S + 32 * 33 + 32) + 16;
    const size_t s = sizeof(double) * kTriRhs * (size_t)S + sizeof(TriStage) - (S <= 64 ? sizeof(double) * 1024 : 0);
    return f > s ? f : s;
}

// Column c of P's row i sits at P[c * S + (i ^ chol_swz(c))] (see tri_e).
__device__ __forceinline__ int chol_swz(int c) { return ((c & 3) << 2) | ((c >> 2) & 3); }

// Row i's place in column c of P: swizzled for the FP64 fragments, plain for FP32's vectors.
template <typename T>
__device__ __forceinline__ int chol_pos(int i, int c) { return sizeof(T) == 8 ? i ^ chol_swz(c) : i; }

// Warp 0: factors the nbp x nbp diagonal block whose row `lane` is in `a` (zero past nbp), writes
// it to A (at element (i, j) = A + i si + j sj), L11^T to Lt (row k at Lt + 32 k) and
// 1 / L11(k,k) to rc. Returns the failing step or -1. The steps run in chunks of eight (one code,
// the registers move down): within a chunk only its own columns are updated, the multipliers
// travelling by shuffle, and the columns after it take the eight updates at the chunk's end, so a
// step's chain is the square root, the reciprocal, two products and a shuffle. No step branches:
// a row's entries right of its diagonal hold values that nothing reads, and from a failing pivot on
// the multipliers are zero.
template <typename T>
__device__ __forceinline__ int chol_team_diag(T (&a)[32], T* __restrict__ A, size_t si, size_t sj, int nbp, T* Lt,
                                              T* rc, int lane) {
    using V2 = typename Vec2<T>::type;
    int stop = 32;   // first step whose pivot is not positive (the zero padding's, past nbp, too)
#pragma unroll 1
    for (int c0 = 0; c0 < nbp; c0 += 8) {
        T l[8];
        T d = __shfl_sync(kFullMask, a[0], c0);
        static_for<0, 8>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            const int g = c0 + k;
            if (!(d > T(0))) stop = min(stop, g);   // not positive definite, or NaN: A(g,g) keeps d
            const bool ok = g < stop;
            const T s = sqrt_rn(ok ? d : T(1));
            const T r = T(1) / s;
            l[k] = ok ? a[k] * r : T(0);
            // the next pivot needs its own row's multiplier alone
            if constexpr (k < 7) d = __shfl_sync(kFullMask, fma_rn(-l[k], l[k], a[k + 1]), g + 1);
            if (ok) a[k] = lane == g ? s : l[k];
            if (lane == 0) rc[g] = r;
#pragma unroll
            for (int j = k + 1; j < 8; ++j) a[j] = fma_rn(-l[k], __shfl_sync(kFullMask, l[k], c0 + j), a[j]);
        });
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            Lt[32 * (c0 + k) + lane] = l[k];
            if (lane < nbp && c0 + k <= lane) A[lane * si + (c0 + k) * sj] = a[k];
        }
        __syncwarp();
#pragma unroll
        for (int jg = 8; jg < 32; jg += 8) {
            if (jg < 32 - c0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const V2* u2 = reinterpret_cast<const V2*>(Lt + 32 * (c0 + k) + c0 + jg);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const V2 u = u2[j / 2];
                        a[jg + j] = fma_rn(-l[k], u.x, a[jg + j]);
                        a[jg + j + 1] = fma_rn(-l[k], u.y, a[jg + j + 1]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j + 8 < 32; ++j) a[j] = a[j + 8];
    }
    return stop < nbp ? stop : -1;
}

// Dynamic shared memory of the kernel, from byte `off` on (functions that are not inlined take
// offsets: a pointer argument would lose its address space).
template <typename T>
__device__ __forceinline__ T* chol_smem(unsigned off) {
    extern __shared__ __align__(16) unsigned char chol_team_raw[];
    return reinterpret_cast<T*>(chol_team_raw + off);
}

// Warp 0's part of a panel: the diagonal block at k0, first brought up to date with the previous
// panel's rows (k0 > 0), is factored; *failed (behind rc) gets the failing step or -1. `off`: the
// team's shared memory (P, then Lt, rc, failed). Not inlined: its registers are its own and its
// code is in the instruction cache once.
template <typename T>
__device__ __noinline__ void chol_team_lead(T* A, size_t si, size_t sj, int n, int k0, unsigned off,
                                                   int S) {
    T* P = chol_smem<T>(off);
    T* Lt = P + 32 * (size_t)S;
    T* rc = Lt + 32 * 33;
    const int lane = threadIdx.x & 31, q = lane & 3, r8 = lane >> 2;
    const int nbp = min(32, n - k0);
    T* Ak = A + k0 * si + k0 * sj;
    T a[32];
    if constexpr (std::is_same<T, double>::value) {
        if (k0 > 0) {
            // 8x8 tiles of the lower triangle; a lane's A and B fragments are the same entries
            double c[4][4][2];
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int t = 0; t <= g; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = 8 * g + r8, j = 8 * t + 2 * q + h;
                        c[g][t][h] = (i < nbp && j <= i) ? Ak[i * si + j * sj] : 0.0;
                    }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                double f[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) f[g] = P[(4 * s + q) * S + ((k0 + 8 * g + r8) ^ chol_swz(4 * s + q))];
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int t = 0; t <= g; ++t) chol_dmma(c[g][t][0], c[g][t][1], -f[g], f[t]);
            }
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int t = 0; t <= g; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) Lt[33 * (8 * g + r8) + 8 * t + 2 * q + h] = c[g][t][h];
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = (lane < nbp && j <= lane) ? Lt[33 * lane + j] : 0.0;
            __syncwarp();
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = (lane < nbp && j <= lane) ? Ak[lane * si + j * sj] : 0.0;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) a[j] = (lane < nbp && j <= lane) ? Ak[lane * si + j * sj] : T(0);
        if (k0 > 0) {
#pragma unroll 2
            for (int c = 0; c < 32; ++c) {   // lane = row; the block's own columns are broadcast
                const T* Pc = P + c * S + k0;
                const T l = Pc[lane];
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(Pc + j);
                    a[j] = fma_rn(-l, u.x, a[j]);
                    a[j + 1] = fma_rn(-l, u.y, a[j + 1]);
                    a[j + 2] = fma_rn(-l, u.z, a[j + 2]);
                    a[j + 3] = fma_rn(-l, u.w, a[j + 3]);
                }
            }
        }
    }
    const int f = chol_team_diag(a, Ak, si, sj, nbp, Lt, rc, lane);
    if (lane == 0) *reinterpret_cast<int*>(rc + 32) = f;
    __syncwarp();
}

// FP32 trailing update of 16 rows from i0 on, columns jb .. je: lane = 4 rows x 8 columns.
__device__ __forceinline__ void chol_team_update(float* __restrict__ A, int n, size_t si, size_t sj, int i0, int jb,
                                                 int je, const float* P, int S, int lane) {
    const int i = i0 + 4 * (lane & 3), j = jb + 8 * (lane >> 2);
    if (j >= je) return;
    float acc[4][8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            acc[r][c] = (i + r < n && j + c <= i + r) ? A[(i + r) * si + (j + c) * sj] : 0.0f;
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        const float4 l = *reinterpret_cast<const float4*>(P + k * S + i);
        const float4 u = *reinterpret_cast<const float4*>(P + k * S + j);
        const float4 v = *reinterpret_cast<const float4*>(P + k * S + j + 4);
        const float lr[4] = {l.x, l.y, l.z, l.w}, uc[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[r][c] = fma_rn(-lr[r], uc[c], acc[r][c]);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (i + r < n && j + c <= i + r) A[(i + r) * si + (j + c) * sj] = acc[r][c];
}

// potrf of one n x n matrix (n <= S) by the team's S threads; `off`: its shared memory. Returns
// info; the caller synchronises the team before it reuses the shared memory.
template <typename T, typename Team>
__device__ int chol_team_potrf(T* __restrict__ A, int n, int lda, bool upper, unsigned off, int S,
                               const Team& team) {
    using V2 = typename Vec2<T>::type;
    T* P = chol_smem<T>(off);
    T* Lt = P + 32 * (size_t)S;   // the updated diagonal block (row i at 33 i), then L11^T
    T* rc = Lt + 32 * 33;
    int* failed = reinterpret_cast<int*>(rc + 32);
    const int tid = team.tid(), lane = tid & 31, warp = tid >> 5, NW = S >> 5;
    const int q = lane & 3, r8 = lane >> 2;
    // element (i, j) of the stored triangle (lower: A(i, j); upper: A(j, i))
    const size_t si = upper ? (size_t)lda : 1, sj = upper ? 1 : (size_t)lda;
    if (warp == 0) chol_team_lead(A, si, sj, n, 0, off, S);
    for (int k0 = 0;; k0 += 32) {
        team.sync();
        const int m0 = k0 + 32, fail = *failed, steps = fail >= 0 ? fail : 32;
        // ---- rows below the diagonal block ----
        if (tid >= m0 && tid < n) {
            T a[32];
            T* row = A + tid * si + k0 * sj;
#pragma unroll
            for (int c = 0; c < 32; ++c) a[c] = row[c * sj];
            static_for<0, 32>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                if (k < steps) {
                    const T l = a[k] * rc[k];
                    a[k] = l;
                    const V2* u2 = reinterpret_cast<const V2*>(Lt + 32 * k);
#pragma unroll
                    for (int j = (k + 1) & ~1; j < 32; j += 2) {
                        const V2 u = u2[j / 2];
                        if (j > k) a[j] = fma_rn(-l, u.x, a[j]);
                        a[j + 1] = fma_rn(-l, u.y, a[j + 1]);
                    }
                }
            });
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                row[c * sj] = a[c];
                P[c * S + chol_pos<T>(tid, c)] = a[c];
            }
        }
        if (fail >= 0) return k0 + fail + 1;
        if (m0 >= n) return 0;
        team.sync();
        // ---- trailing triangle ----
        if (warp == 0) {
            chol_team_lead(A, si, sj, n, m0, off, S);
        } else {
            const int i1 = m0 + 32;   // first row past the next diagonal block
            int turn = warp - 1;   // jobs go to the warps in turn
            for (int i0 = i1; i0 < n; i0 += 16) {
                for (int jb = m0; jb < i0 + 16; jb += 64) {
                    if (turn-- > 0) continue;
                    turn = NW - 2;
                    if constexpr (!std::is_same<T, double>::value) {
                        chol_team_update(A, n, si, sj, i0, jb, min(jb + 64, i0 + 16), P, S, lane);
                        continue;
                    } else {
                        const int ra = i0 + r8, rb = ra + 8, je = min(jb + 64, i0 + 16);
                        double cn[2][2][2];   // [tile][row group][column]
                        auto load_c = [&](int jt) {
#pragma unroll
                            for (int t = 0; t < 2; ++t)
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const int j = jt + 8 * t + 2 * q + h;
                                    cn[t][0][h] = (ra < n && j <= ra) ? A[ra * si + j * sj] : 0.0;
                                    cn[t][1][h] = (rb < n && j <= rb) ? A[rb * si + j * sj] : 0.0;
                                }
                        };
                        load_c(jb);
                        double fa[8], fb[8];
#pragma unroll
                        for (int s = 0; s < 8; ++s) {
                            const int c = 4 * s + q;
                            fa[s] = -P[c * S + (ra ^ chol_swz(c))];
                            fb[s] = -P[c * S + (rb ^ chol_swz(c))];
                        }
#pragma unroll 1
                        for (int jt = jb; jt < je; jt += 16) {
                            double cc[2][2][2];
#pragma unroll
                            for (int t = 0; t < 2; ++t)
#pragma unroll
                                for (int g = 0; g < 2; ++g) { cc[t][g][0] = cn[t][g][0]; cc[t][g][1] = cn[t][g][1]; }
                            if (jt + 16 < je) load_c(jt + 16);
#pragma unroll
                            for (int s = 0; s < 8; ++s) {
                                const int c = 4 * s + q;
                                const double b0 = P[c * S + ((jt + r8) ^ chol_swz(c))];
                                const double b1 = P[c * S + ((jt + 8 + r8) ^ chol_swz(c))];
                                chol_dmma(cc[0][0][0], cc[0][0][1], fa[s], b0);
                                chol_dmma(cc[0][1][0], cc[0][1][1], fb[s], b0);
                                chol_dmma(cc[1][0][0], cc[1][0][1], fa[s], b1);
                                chol_dmma(cc[1][1][0], cc[1][1][1], fb[s], b1);
                            }
#pragma unroll
                            for (int t = 0; t < 2; ++t)
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const int j = jt + 8 * t + 2 * q + h;
                                    if (ra < n && j <= ra) A[ra * si + j * sj] = cc[t][0][h];
                                    if (rb < n && j <= rb) A[rb * si + j * sj] = cc[t][1][h];
                                }
                        }
                    }
                }
            }
        }
    }
}

// potrs of one n x n matrix by the team's S threads, groups first, first + stride, .. of eight
// right-hand sides: L y = b, then L^T x = y. `rows` >= n: the rows X has room for.
template <typename Team>
__device__ void chol_team_potrs(const double* A, int n, int lda, bool upper, double* __restrict__ B, int nrhs, int ldb,
                                unsigned off, int S, int rows, int first, int stride, const Team& team) {
    double* X = chol_smem<double>(off);
    TriStage& st = *reinterpret_cast<TriStage*>(X + (size_t)rows * kTriRhs);
    const int NW = S >> 5, npad = (n + 31) / 32 * 32;
    const size_t si = upper ? (size_t)lda : 1, sj = upper ? 1 : (size_t)lda;
    for (int c0 = first * kTriRhs; c0 < nrhs; c0 += stride * kTriRhs) {
        for (int t = team.tid(); t < npad; t += S) {
#pragma unroll
            for (int r = 0; r < kTriRhs; ++r)
                X[tri_x(t, r)] = (t < n && c0 + r < nrhs) ? B[t + (size_t)(c0 + r) * ldb] : 0.0;
        }
        team.sync();
        tri_sweep<TriDiag::Reciprocal, false>(A, si, sj, n, X, st, NW, team);
        tri_sweep<TriDiag::Reciprocal, true>(A, sj, si, n, X, st, NW, team);
        for (int t = team.tid(); t < n; t += S) {
#pragma unroll
            for (int r = 0; r < kTriRhs; ++r)
                if (c0 + r < nrhs) B[t + (size_t)(c0 + r) * ldb] = X[tri_x(t, r)];
        }
        team.sync();
    }
}

}  // namespace mb200
