// tri_solve.cuh -- FP64 triangular sweeps T X = B of one matrix by a team of warps, eight
// right-hand sides at a time on the tensor cores (mma.sync m8n8k4 .f64: 8 rows x 8 right-hand
// sides x 4 columns of T).
//
// X (n x 8) lives in shared memory and T is read once, in 32-row blocks. While block J's
// solution is applied to the rows still open, one warp runs ahead: it updates the 32 rows of
// the next block first and solves them, so the only barrier of a block is the one after which
// its successor is known. The other warps copy the entries it needs next to shared memory
// asynchronously, one block ahead. The 32x32 diagonal block is solved in four 8-row pieces held in
// the MMA's accumulator layout (lane l: row l/4, right-hand sides 2(l%4), +1): a step broadcasts
// the solved row by shuffles, and a finished piece updates the pieces after it by MMAs.
// Pieces past n take no steps (2,000 x 65^2, 1 RHS: potrs 93 -> 84 us, getrs 145 -> 129).
//
// Every entry receives its updates as single fma's in the order of reference BLAS dtrsm (k
// ascending for a lower T, descending for an upper one): an m8n8k4 MMA applies its four
// products in ascending k index, each rounded, and a descending sweep numbers the four columns
// of a step backwards. Solutions are bit-identical to a row-per-thread sweep.
//
// What bounds it: the chain of a block's 32 steps in the leading warp (clock stamps: 60 cycles a
// step with a unit diagonal, 280 with a division, 2,400 to 3,000 a block around them), at few
// blocks an SM. Measured against a row-per-thread sweep of four right-hand sides at a time, all
// of a matrix's groups in one block: 4,000 x 128^2, 4 RHS 539 -> 392 us; 2,048 x 256^2
// 1,043 -> 518; 592 x 512^2 1,151 -> 492; 148 x 1024^2, 16 RHS 4,199 -> 718; 16 x 1024^2
// 3,963 -> 493.
#pragma once

#include "fast_div.cuh"
#include "small_lu.cuh"

namespace mb200 {

// How a solved row leaves the diagonal: as it is, times the rounded reciprocal (the oracle's
// dpotrs), or divided (dtrsm).
enum class TriDiag { Unit, Reciprocal, Divide };

constexpr int kTriRhs = 8;   // right-hand sides of a sweep

// Entry (row, col) of X; the swizzle spreads a B fragment's 4 rows x 4 columns over all banks.
__device__ __forceinline__ int tri_x(int row, int col) { return row * kTriRhs + (col ^ ((row & 2) << 1)); }

// The staged blocks of two successive steps: the u-th block in sweep order has its diagonal block
// in d[u & 1] and the block that couples it to its predecessor in p[(u + 1) & 1], entry (i, k) at
// tri_e(i, k). A matrix of two blocks never touches p[1].
// The elements keep T's own type (FP32 factors are widened when they are used).
template <typename E>
struct TriStageOf {
    E d[2][1024];
    E p[2][1024];
};
using TriStage = TriStageOf<double>;
// Swizzled so that A fragments, rows and columns of a block are read and written over all banks.
__device__ __forceinline__ int tri_e(int i, int k) { return i * 32 + (k ^ (((i & 3) << 2) | ((i >> 2) & 3))); }

// One element to shared memory, asynchronously; zero when !valid (nothing is read).
template <typename E>
__device__ __forceinline__ void tri_copy(E* dst, const E* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"((int)sizeof(E)), "r"(valid ? (int)sizeof(E) : 0)
                 : "memory");
}

__device__ __forceinline__ void tri_dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// One sweep of a team of NW >= 2 warps (team.sync() is its barrier). T(i, k) = A[i * rs + k * cs];
// lower and ascending, or upper and descending (DESC). X holds ceil(n / 32) * 32 rows. On entry
// every warp must see X; on return every warp does.
template <TriDiag MODE, bool DESC, typename E, typename Team>
__device__ __forceinline__ void tri_sweep(const E* A, size_t rs, size_t cs, int n, double* X, TriStageOf<E>& buf,
                                          int NW, const Team& team) {
    const int tid = team.tid(), lane = tid & 31, warp = tid >> 5;
    const int q = lane & 3, r8 = lane >> 2;
    const int nblk = (n + 31) / 32;
    auto block_of = [&](int s) { return DESC ? nblk - 1 - s : s; };
    // column 4s' + .. of a 32-column block behind MMA k index q of k-step s
    auto kof = [&](int s) { return DESC ? 31 - 4 * s - q : 4 * s + q; };

    // Warps first, first + count, .. : a share of the copies for the u-th block in sweep order.
    auto stage = [&](int u, int share, int shares) {
        E *bd = buf.d[u & 1], *bp = buf.p[(u + 1) & 1];
        const int j0 = block_of(u) * 32, p0 = u > 0 ? block_of(u - 1) * 32 : 0;
        for (int e = share; e < 32; e += shares) {
            const int i = rs == 1 ? lane : e, k = rs == 1 ? e : lane;   // lanes along the contiguous direction
            const bool vi = j0 + i < n;
            const bool vd = vi && j0 + k < n, vp = vi && p0 + k < n;
            const E* row = A + (j0 + i) * rs;
            tri_copy(&bd[tri_e(i, k)], vd ? row + (j0 + k) * cs : A, vd);
            if (u > 0) tri_copy(&bp[tri_e(i, k)], vp ? row + (p0 + k) * cs : A, vp);
        }
    };
    // Warp 0: applies the predecessor's solution to the rows of the u-th block and solves them.
    auto lead = [&](int u) {
        const E *bd = buf.d[u & 1], *bp = buf.p[(u + 1) & 1];
        const int j0 = block_of(u) * 32;
        if (u > 0) {
            const int p0 = block_of(u - 1) * 32;
            double c[4][2];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const double2 v = *reinterpret_cast<const double2*>(&X[tri_x(j0 + 8 * t + r8, 2 * q)]);
                c[t][0] = v.x;
                c[t][1] = v.y;
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const double b = -X[tri_x(p0 + kof(s), r8)];
#pragma unroll
                for (int t = 0; t < 4; ++t) tri_dmma(c[t][0], c[t][1], (double)bp[tri_e(8 * t + r8, kof(s))], b);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
                *reinterpret_cast<double2*>(&X[tri_x(j0 + 8 * t + r8, 2 * q)]) = make_double2(c[t][0], c[t][1]);
        }
        // the pieces in a loop: unrolled over all 32 steps the code outgrows the instruction cache
#pragma unroll 1
        for (int tt = 0; tt < 4; ++tt) {
            const int t = DESC ? 3 - tt : tt, i = 8 * t + r8;
            double2* xi = reinterpret_cast<double2*>(&X[tri_x(j0 + i, 2 * q)]);
            if (j0 + 8 * t >= n) {   // a piece past n: no steps, its rows stay zero
                *xi = make_double2(0.0, 0.0);
                __syncwarp();
                continue;
            }
            double2 c = *xi;
            double l[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) l[k] = (double)bd[tri_e(i, 8 * t + k)];
            Divisor v;
            bool slow = false;   // a diagonal entry of the piece that div_fast cannot take
            if constexpr (MODE != TriDiag::Unit) {
                v = make_divisor(j0 + i < n ? (double)bd[tri_e(i, i)] : 1.0);
                if (MODE == TriDiag::Divide) slow = __any_sync(kFullMask, !div_fast_den(v.d));
            }
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                const int k = DESC ? 7 - kk : kk;
                double2 x = c;
                if constexpr (MODE == TriDiag::Reciprocal) {
                    x.x *= v.hi;
                    x.y *= v.hi;
                } else if constexpr (MODE == TriDiag::Divide) {
                    // row k's lanes decide; the other lanes' quotients are not used
                    const bool bad = r8 == k && !(div_fast_num(c.x) && div_fast_num(c.y));
                    x = make_double2(div_fast(c.x, v), div_fast(c.y, v));
                    if (slow || __any_sync(kFullMask, bad)) x = make_double2(div_slow(c.x, v.d), div_slow(c.y, v.d));
                }
                const double y0 = __shfl_sync(kFullMask, x.x, 4 * k + q);
                const double y1 = __shfl_sync(kFullMask, x.y, 4 * k + q);
                if (MODE != TriDiag::Unit && r8 == k) c = x;
                if (DESC ? r8 < k : r8 > k) {
                    c.x = fma_rn(-y0, l[k], c.x);
                    c.y = fma_rn(-y1, l[k], c.y);
                }
            }
            *xi = j0 + i < n ? c : make_double2(0.0, 0.0);   // rows past n stay zero
            __syncwarp();
            // the pieces still open
            double b[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) b[h] = -X[tri_x(j0 + 8 * t + (DESC ? 7 - 4 * h - q : 4 * h + q), r8)];
#pragma unroll 1
            for (int w = tt + 1; w < 4 && (DESC || j0 + 8 * w < n); ++w) {
                const int iw = 8 * (DESC ? 3 - w : w) + r8;
                double2* xw = reinterpret_cast<double2*>(&X[tri_x(j0 + iw, 2 * q)]);
                double2 cw = *xw;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    tri_dmma(cw.x, cw.y, (double)bd[tri_e(iw, 8 * t + (DESC ? 7 - 4 * h - q : 4 * h + q))], b[h]);
                *xw = cw;
            }
            __syncwarp();
        }
    };

    stage(0, warp, NW);
    if (nblk > 1) stage(1, warp, NW);
    asm volatile("cp.async.wait_all;" ::: "memory");
    team.sync();
    if (warp == 0) lead(0);
    team.sync();
    for (int s = 0; s + 1 < nblk; ++s) {
        const int jn = block_of(s + 1), b0 = block_of(s) * 32;
        if (warp == 0) {
            lead(s + 1);
        } else {
            if (s + 2 < nblk) stage(s + 2, warp - 1, NW - 1);
            // the rows past block jn, 16 at a time, the next 16 rows' entries in flight
            const int lo = DESC ? 0 : (jn + 1) * 32, hi = DESC ? jn * 32 : n;
            const int pairs = (hi - lo + 15) / 16;
            if (warp - 1 < pairs) {
                double b[8];
                E a0[8], a1[8];
#pragma unroll
                for (int s8 = 0; s8 < 8; ++s8) b[s8] = -X[tri_x(b0 + kof(s8), r8)];
                auto load = [&](int p) {
                    const int i0 = lo + 16 * p + r8, i1 = i0 + 8;
#pragma unroll
                    for (int s8 = 0; s8 < 8; ++s8) {
                        const int k = b0 + kof(s8);
                        a0[s8] = (i0 < hi && k < n) ? A[i0 * rs + k * cs] : E(0);
                        a1[s8] = (i1 < hi && k < n) ? A[i1 * rs + k * cs] : E(0);
                    }
                };
                load(warp - 1);
                for (int p = warp - 1; p < pairs; p += NW - 1) {
                    const int i0 = lo + 16 * p + r8, i1 = i0 + 8;
                    double u0[8], u1[8];
#pragma unroll
                    for (int s8 = 0; s8 < 8; ++s8) { u0[s8] = (double)a0[s8]; u1[s8] = (double)a1[s8]; }
                    if (p + NW - 1 < pairs) load(p + NW - 1);
                    double2 c0 = *reinterpret_cast<const double2*>(&X[tri_x(i0, 2 * q)]);
                    double2 c1 = *reinterpret_cast<const double2*>(&X[tri_x(i1, 2 * q)]);
#pragma unroll
                    for (int s8 = 0; s8 < 8; ++s8) {
                        tri_dmma(c0.x, c0.y, u0[s8], b[s8]);
                        tri_dmma(c1.x, c1.y, u1[s8], b[s8]);
                    }
                    if (i0 < hi) *reinterpret_cast<double2*>(&X[tri_x(i0, 2 * q)]) = c0;
                    if (i1 < hi) *reinterpret_cast<double2*>(&X[tri_x(i1, 2 * q)]) = c1;
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        team.sync();
    }
}

}  // namespace mb200
