// cluster_lu.cuh -- blocked right-looking FP64 LU (getrf) of one matrix per thread-block
// cluster: CS blocks of NT threads factor a matrix of up to CS * NT rows.
//
// One block per matrix leaves a large order on one SM: its 1024 threads hold 64 registers
// each, every panel step crosses two 1024-thread barriers, and the trailing update has one
// SM's FP64 rate. Here the cluster shares the matrix:
//
//   for each panel of NB columns (k0 = 0, NB, ...):
//     1. thread t of the cluster (t = rank * NT + tid) holds row t of the panel in registers.
//        A step finds each block's best pivot candidate (warp reductions, one block barrier);
//        the candidate's thread writes its key, its row and the reciprocal of its pivot into
//        every block's shared memory, and after ONE cluster barrier all threads pick the same
//        winner among the CS candidates and apply the rank-1 update.
//     2. the panel is stored at the rows' new positions; the interchanges (which row each of
//        the NB pivot positions takes, where the rows they displace go) reach every block.
//     3. every block takes a slab of the other columns. Left of the panel it applies the
//        interchanges. Right of it, it gathers the pivot rows into shared memory, moves the
//        displaced rows, solves U12 = L11^-1 A12 (a thread per column) and updates its columns
//        of A22 -= L21 U12 on the FP64 tensor cores: a warp takes 16 rows x 64 columns, the
//        rows' multipliers as A fragments in registers, U12 as B fragments from shared memory,
//        the next 16 columns of C in flight while the current ones are multiplied.
//   After each panel the matrix is again in LAPACK's row order. Between panels the blocks of a
//   cluster meet at a cluster barrier; the matrix travels through L2 (all loads bypass L1).
//
// What bounds it (clock stamps, cycles a matrix): n = 256 at two blocks an SM, panel steps 37%
// (about 1,300 cycles a step: two barriers, the reductions, one division), update 28%, gather
// 15%; n = 1024 on four SMs, update 49% (2.6 times its FP64 rate's time), panel 30% (2,000 to
// 2,200 cycles a step, a cluster barrier among them). Measured against one block a matrix:
// 2,048 x 256^2 4.50 -> 3.07 ms, 4,000 x 128^2 1.42 -> 1.10 ms, 592 x 512^2 8.85 -> 7.14 ms,
// 148 x 1024^2 24.5 -> 14.4 ms, 16 x 1024^2 19.3 -> 3.29 ms.
//
// Every element receives its updates as single fma's in increasing step order, exactly like
// the unblocked dgetf2, so factors, pivots and info are bit-identical to the oracle
// restatement (an m8n8k4 FP64 MMA applies its four products in ascending k, each rounded).
#pragma once

#include <cooperative_groups.h>
#include "small_lu.cuh"

namespace mb200 {

// A block's pivot candidate as it travels to the other blocks, in 16-byte pieces.
template <int NB>
struct alignas(16) PivotCandidate {
    double   row[NB];
    double   rcp;      // 1 / pivot; 1 for a zero pivot (the column is left as it is)
    int      kind;     // 0: zero pivot, 1: scale by rcp, 2: divide (below the smallest normal number)
    int      p;        // row position
    unsigned hi, lo;   // key
    int      pad[2];
    static constexpr int kPieces = NB / 2 + 2;
};

template <int NB, int NT, int CS>
struct ClusterLuShared {
    static constexpr int NW = NT / 32;
    PivotCandidate<NB> cand[2][CS];      // the blocks' candidates, double-buffered by step parity
    unsigned red_hi[2][NW], red_lo[2][NW];
    int      red_p[2][NW], red_s[2][NW];
    int      src[NB];                    // row that moves to position k0 + s
    int      dst[NB];                    // position the row at k0 + s moves to, -1 if it is a pivot row
    double   L11[NB][NB + 1];
    double   U[NB][NT];                  // pivot rows' columns of the slab, then U12 (swizzled columns)
};

// One FP64 tensor-core step D = A B + D on an 8x8 tile (A 8x4 row-major, B 4x8
// column-major; lane l holds A(l/4, l%4), B(l%4, l/4), D(l/4, 2(l%4) .. +1)). Each
// element of D receives fma(a(i,0), b(0,j), d) then k = 1, 2, 3 in ascending order,
// rounded after every step (measured on B200 against the fma chain: 1.28 M of 1.28 M
// elements equal) -- the same operations as four single fma's in k order, which keeps the
// blocked update bit-identical to the unblocked elimination.
__device__ __forceinline__ void dmma_884(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// Column c of U's row r sits at c ^ u_swz(r): a warp reading rows 4s..4s+3 x 4 columns (a B
// fragment), one row across columns (the solve) or one column across rows (the gather) then
// touches all sixteen 8-byte banks.
__device__ __forceinline__ int u_swz(int r) { return ((r & 3) << 2) | ((r >> 2) & 3); }

template <int CS>
__device__ __forceinline__ void cluster_sync() {
    if constexpr (CS == 1) __syncthreads();
    else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
}

// Shared-memory address of `local` in block `rank` of the cluster, and stores through it.
__device__ __forceinline__ unsigned peer_addr(const void* local, int rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ void peer_store(unsigned a, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void peer_store(unsigned a, int x) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}

// U12 = L11^-1 A12 for column c of the slab chunk,
// in groups of H rows held in registers (each entry: fma(L11(r, rr), -U(rr, c), x), rr ascending).
template <int NB, int NT, int CS>
__device__ __forceinline__ void cluster_trsm_column(ClusterLuShared<NB, NT, CS>& sh, int c) {
    constexpr int H = 8;
#pragma unroll 1
    for (int q0 = 0; q0 < NB; q0 += H) {
        double x[H];
#pragma unroll
        for (int r = 0; r < H; ++r) x[r] = sh.U[q0 + r][c ^ u_swz(q0 + r)];
#pragma unroll 4
        for (int rr = 0; rr < q0; ++rr) {
            const double u = sh.U[rr][c ^ u_swz(rr)];
#pragma unroll
            for (int r = 0; r < H; ++r) x[r] = fma_rn(sh.L11[q0 + r][rr], -u, x[r]);
        }
        static_for<0, H>([&](auto rrc) {
            constexpr int rr = decltype(rrc)::value;
#pragma unroll
            for (int r = rr + 1; r < H; ++r) x[r] = fma_rn(sh.L11[q0 + r][q0 + rr], -x[rr], x[r]);
        });
#pragma unroll
        for (int r = 0; r < H; ++r) sh.U[q0 + r][c ^ u_swz(q0 + r)] = x[r];
    }
}

// Applies the panel's interchanges to columns [j, j + w) of A, lane = pivot position, a warp
// per column (eight loads in flight a lane). The pivot rows go to U (gather) or to their new
// positions. Within a column every read precedes every write.
template <int NB, int NT, int CS, bool GATHER>
__device__ __forceinline__ void cluster_laswp(double* __restrict__ A, int lda, int k0, int nbp, int j, int w,
                                              ClusterLuShared<NB, NT, CS>& sh) {
    static_assert(NB == 32, "a lane per pivot position");
    constexpr int NW = NT / 32, G = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool on = lane < nbp;
    const int src = on ? sh.src[lane] : 0, dst = on ? sh.dst[lane] : -1;
    const bool moves = on && src != k0 + lane;
    for (int c0 = warp; c0 < w; c0 += NW * G) {
        double u[G], d[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int c = c0 + g * NW;
            const double* col = A + (size_t)(j + c) * lda;
            u[g] = (c < w && (GATHER ? on : moves)) ? __ldcg(col + src) : 0.0;
            d[g] = (c < w && dst >= 0) ? __ldcg(col + k0 + lane) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int c = c0 + g * NW;
            double* col = A + (size_t)(j + c) * lda;
            if (c < w) {
                if constexpr (GATHER) sh.U[lane][c ^ u_swz(lane)] = u[g];
                else if (moves) col[k0 + lane] = u[g];
                if (dst >= 0) col[dst] = d[g];
            }
        }
    }
}

// A22 -= L21 U12 for the slab chunk's cw columns from j on: rows i0.. m of all groups of 16
// rows x 64 columns, a warp each.
template <int NB, int NT, int CS>
__device__ __forceinline__ void cluster_update(double* __restrict__ A, int m, int lda, int k0, int j, int cw,
                                               const ClusterLuShared<NB, NT, CS>& sh) {
    constexpr int NW = NT / 32, KS = NB / 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane & 3, r8 = lane >> 2;
    const int i0 = k0 + NB;
    const int groups = (m - i0 + 15) / 16, parts = (cw + 63) / 64;
    if (m <= i0) return;
    for (int task = warp; task < groups * parts; task += NW) {
        const int rg = task / parts, jb = (task - rg * parts) * 64, je = min(cw, jb + 64);
        const int ra = i0 + 16 * rg + r8, rb = ra + 8;
        const bool va = ra < m, vb = rb < m;
        double cn[2][2][2];   // [tile][row group][column]
        auto load_c = [&](int jt) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = jt + 8 * t + 2 * q + h;
                    const double* col = A + (size_t)(j + c) * lda;
                    cn[t][0][h] = (va && c < je) ? __ldcg(col + ra) : 0.0;
                    cn[t][1][h] = (vb && c < je) ? __ldcg(col + rb) : 0.0;
                }
        };
        load_c(jb);
        // the rows' multipliers, negated: (-l) u + c is the fma of the CUDA-core update
        double fa[KS], fb[KS];
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const double* col = A + (size_t)(k0 + 4 * s + q) * lda;
            fa[s] = va ? -__ldcg(col + ra) : 0.0;
            fb[s] = vb ? -__ldcg(col + rb) : 0.0;
        }
#pragma unroll 1
        for (int jt = jb; jt < je; jt += 16) {
            double cc[2][2][2];
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int g = 0; g < 2; ++g) { cc[t][g][0] = cn[t][g][0]; cc[t][g][1] = cn[t][g][1]; }
            if (jt + 16 < je) load_c(jt + 16);
            // columns past the chunk read U entries whose products are never stored
            const int c0 = (jt + r8) ^ (q << 2), c1 = (jt + 8 + r8) ^ (q << 2);
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                const double b0 = sh.U[4 * s + q][c0 ^ (s & 3)];
                const double b1 = sh.U[4 * s + q][c1 ^ (s & 3)];
                dmma_884(cc[0][0][0], cc[0][0][1], fa[s], b0);
                dmma_884(cc[0][1][0], cc[0][1][1], fb[s], b0);
                dmma_884(cc[1][0][0], cc[1][0][1], fa[s], b1);
                dmma_884(cc[1][1][0], cc[1][1][1], fb[s], b1);
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = jt + 8 * t + 2 * q + h;
                    double* col = A + (size_t)(j + c) * lda;
                    if (va && c < je) col[ra] = cc[t][0][h];
                    if (vb && c < je) col[rb] = cc[t][1][h];
                }
        }
    }
}

// The lane holding the warp's best pivot candidate: warp_argmax without the second and third
// reduction when one lane alone has the largest high key word (nearly always).
__device__ __forceinline__ int warp_argmax_lane(const PivotKey& key, int p) {
    const unsigned mhi = __reduce_max_sync(kFullMask, key.hi);
    unsigned who = __ballot_sync(kFullMask, key.hi == mhi);
    if (who & (who - 1)) {
        const unsigned mlo = __reduce_max_sync(kFullMask, key.hi == mhi ? key.lo : 0u);
        const bool top = key.hi == mhi && key.lo == mlo;
        const int pmin = __reduce_min_sync(kFullMask, top ? p : INT_MAX);
        who = __ballot_sync(kFullMask, top && p == pmin);
    }
    return __ffs(who) - 1;
}

// How a pivot scales its column: 0 a zero pivot (not at all), 1 by its reciprocal, 2 by division
// (below the smallest normal number, or NaN: dgetf2's other branch). From the bits: a comparison
// in FP64 costs a step's chain as much as two multiplications.
__device__ __forceinline__ int pivot_kind(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return (h | (unsigned)__double2loint(x)) == 0 ? 0 : h - 0x00100000u <= 0x7ff00000u - 0x00100000u ? 1 : 2;
}

// Factors panel columns k0 .. k0+nbp-1 of the rows held in `a` (thread t = row t of the
// cluster): the steps of lu_panel_steps with the pivot chosen across the cluster. The code of
// CK steps serves every chunk of CK columns: a finished chunk's columns go to U (column c of
// thread tid at U[c][tid]) and the registers move down by CK, which quarters the code and
// frees the registers that kept a finished row (the same time a step as all NB unrolled).
template <int NB, int NT, int CS>
__device__ __forceinline__ void cluster_panel(double (&a)[NB], int m, int nbp, int k0, int t, int rank, int& pos,
                                              int& my_ipiv, int& info, ClusterLuShared<NB, NT, CS>& sh, bool nopiv) {
    constexpr int NW = NT / 32, CK = 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
    for (int c0 = 0; c0 < nbp; c0 += CK) {
        const int left = NB - c0;   // columns still in registers
        static_for<0, CK>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if (c0 + k >= nbp) return;
            constexpr int buf = k & 1;
            const int g = k0 + c0 + k;
            int p = g;
            PivotKey key{0u, 0u};
            bool best;   // this thread's row is its block's candidate
            if (nopiv) {
                best = t == g;
            } else {
                const bool cand = pos >= g && t < m;
                key = pivot_key(a[k], cand);
                p = cand ? pos : INT_MAX;
                if (warp_argmax_lane(key, p) == lane) {
                    sh.red_hi[buf][warp] = key.hi; sh.red_lo[buf][warp] = key.lo;
                    sh.red_p[buf][warp] = p; sh.red_s[buf][warp] = tid;
                }
                __syncthreads();
                const bool v = lane < NW;
                const PivotKey wk{v ? sh.red_hi[buf][lane] : 0u, v ? sh.red_lo[buf][lane] : 0u};
                const int w = warp_argmax_lane(wk, v ? sh.red_p[buf][lane] : INT_MAX);
                best = tid == sh.red_s[buf][w];
                p = sh.red_p[buf][w];
            }
            // The candidate's thread publishes its row and the reciprocal of its pivot (formed once
            // here instead of by every row after the barrier).
            PivotCandidate<NB>& mine = sh.cand[buf][rank];
            if (best) {
                constexpr int jw = k & ~1;
                const double d = a[k];
                double2* row2 = reinterpret_cast<double2*>(mine.row);
#pragma unroll
                for (int j = jw; j < NB; j += 2) row2[j / 2] = make_double2(a[j], a[j + 1]);
                const int kd = pivot_kind(d);
                mine.kind = kd;
                mine.rcp = 1.0 / (kd ? d : 1.0);
                if constexpr (CS > 1) {
                    mine.hi = key.hi;
                    mine.lo = key.lo;
                    mine.p = p;
                }
            }
            if constexpr (CS > 1) {
                // its warp copies it to the other blocks, a 16-byte piece a lane
                if (__any_sync(kFullMask, best)) {
                    __syncwarp();
                    if (lane < PivotCandidate<NB>::kPieces) {
                        const double2 v = reinterpret_cast<const double2*>(&mine)[lane];
#pragma unroll
                        for (int c = 1; c < CS; ++c) peer_store(peer_addr(reinterpret_cast<const double2*>(&mine) + lane, (rank + c) % CS), v);
                    }
                }
            }
            cluster_sync<CS>();
            int b = 0;
            if constexpr (CS > 1) {
                if (nopiv) {
                    b = g / NT;
                } else {
                    PivotKey bk{sh.cand[buf][0].hi, sh.cand[buf][0].lo};
                    p = sh.cand[buf][0].p;
#pragma unroll
                    for (int c = 1; c < CS; ++c) {
                        const PivotKey k2{sh.cand[buf][c].hi, sh.cand[buf][c].lo};
                        const int p2 = sh.cand[buf][c].p;
                        if (key_beats(k2, p2, bk, p)) { bk = k2; p = p2; b = c; }
                    }
                }
            }
            const PivotCandidate<NB>& top = sh.cand[buf][b];
            const int kind = top.kind;
            if (t == g) my_ipiv = p + 1;
            if (kind) {
                if (pos == g) pos = p;
                if (best && b == rank) pos = g;
            } else if (info == 0) {
                info = g + 1;
            }
            if (pos > g && t < m) {
                if (kind == 2) a[k] = a[k] / top.row[k];
                else           a[k] = a[k] * top.rcp;
                const double l = a[k];
                const double2* row2 = reinterpret_cast<const double2*>(top.row);
#pragma unroll
                for (int j = (k + 1) & ~1; j < CK; j += 2) {
                    const double2 u = row2[j / 2];
                    if (j > k) a[j] = fma_rn(l, -u.x, a[j]);
                    a[j + 1] = fma_rn(l, -u.y, a[j + 1]);
                }
#pragma unroll
                for (int jg = CK; jg < NB; jg += CK) {
                    if (jg < left) {
#pragma unroll
                        for (int j = jg; j < jg + CK; j += 2) {
                            const double2 u = row2[j / 2];
                            a[j] = fma_rn(l, -u.x, a[j]);
                            a[j + 1] = fma_rn(l, -u.y, a[j + 1]);
                        }
                    }
                }
            }
        });
#pragma unroll
        for (int j = 0; j < CK; ++j) sh.U[c0 + j][tid] = a[j];
#pragma unroll
        for (int j = 0; j + CK < NB; ++j) a[j] = a[j + CK];
    }
}

template <int NB, int NT, int CS>
__device__ void cluster_getrf(double* __restrict__ A, int m, int n, int lda, int* __restrict__ ipiv, int& info,
                              int rank, ClusterLuShared<NB, NT, CS>& sh) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = rank * NT + tid;
    const int kmax = min(m, n);
    info = 0;
    for (int k0 = 0; k0 < kmax; k0 += NB) {
        const int nbp = min(NB, kmax - k0);
        const bool live = t >= k0 && t < m;
        // ---- 1. panel ----
        double a[NB];
#pragma unroll
        for (int c = 0; c < NB; ++c) a[c] = (live && c < nbp) ? __ldcg(A + t + (size_t)(k0 + c) * lda) : 0.0;
        int pos = t < m ? t : INT_MAX / 2;
        int my_ipiv = 0;
        cluster_panel<NB, NT, CS>(a, m, nbp, k0, t, rank, pos, my_ipiv, info, sh, ipiv == nullptr);
        if (ipiv && t >= k0 && t < k0 + nbp) ipiv[t] = my_ipiv;
        // ---- 2. panel to its new rows; interchanges to every block ----
        const bool pivot_row = live && pos < k0 + nbp;
        if (live) {
#pragma unroll 8
            for (int c = 0; c < nbp; ++c) A[pos + (size_t)(k0 + c) * lda] = sh.U[c][tid];
        }
        if constexpr (CS == 1) {
            if (pivot_row) sh.src[pos - k0] = t;
            if (live && t < k0 + nbp) sh.dst[t - k0] = pivot_row ? -1 : pos;
        } else {
#pragma unroll 1
            for (int c = 0; c < CS; ++c) {
                if (pivot_row) peer_store(peer_addr(&sh.src[pos - k0], c), t);
                if (live && t < k0 + nbp) peer_store(peer_addr(&sh.dst[t - k0], c), pivot_row ? -1 : pos);
            }
        }
        cluster_sync<CS>();
        // ---- 3. the block's columns ----
        const int right = n - k0 - nbp;
        if (right > 0)
            for (int e = tid; e < NB * nbp; e += NT) {
                const int r = e % NB, c = e / NB;
                sh.L11[r][c] = r < nbp ? __ldcg(A + k0 + r + (size_t)(k0 + c) * lda) : 0.0;
            }
        const int lw = (k0 + CS - 1) / CS, lb = min(k0, rank * lw);
        cluster_laswp<NB, NT, CS, false>(A, lda, k0, nbp, lb, min(lw, k0 - lb), sh);
        const int rw = ((right + CS - 1) / CS + 7) / 8 * 8;
        const int rb = min(right, rank * rw), re = min(right, rb + rw);
        for (int jc = rb; jc < re; jc += NT) {
            const int j = k0 + nbp + jc, cw = min(NT, re - jc);
            cluster_laswp<NB, NT, CS, true>(A, lda, k0, nbp, j, cw, sh);
            __syncthreads();
            if (tid < cw) cluster_trsm_column(sh, tid);
            __syncthreads();
            for (int c = warp; c < cw; c += NW)
                if (lane < nbp) A[k0 + lane + (size_t)(j + c) * lda] = sh.U[lane][c ^ u_swz(lane)];
            cluster_update<NB, NT, CS>(A, m, lda, k0, j, cw, sh);
            __syncthreads();   // U free for the next chunk
        }
        cluster_sync<CS>();    // the next panel's columns are complete
    }
}

}  // namespace mb200
