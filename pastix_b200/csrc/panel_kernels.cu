// Panel factorization of the wide cblks of one level, in one launch (LU in the row-block
// form only, where the level's widest diagonal block fits in shared memory).
//
// PaStiX factors a cblk's diagonal block with its blocked kernel and then solves
// the whole panel below it (cpucblk_zpotrfsp1d_panel, kernels/core_zpotrfsp.c:284-295:
// core_zpotrfsp, kernels/core_zpotrfsp.c:66-100, then cpucblk_ztrsmsp;
// cpucblk_zsytrfsp1d_panel, kernels/core_zsytrfsp.c:424-446: core_zsytrfsp,
// kernels/core_zsytrfsp.c:63-103, then the solve against D L^T).  Here the same
// factorization runs right-looking over 64-column steps j, with the panel's rows
// cut into row blocks b of 64 rows: blocks 0 .. ns-1 are the rows of the diagonal
// block (block j holds the diagonal tile of step j), the others the rows below it.
//
// Items (j, b) with b >= j:
//   b == j  factor the diagonal tile of step j in registers;
//   b >  j  solve the step's columns of row block b against that tile by
//           substitution (x_c = (a_c - sum_{l<c} x_l L_cl) / L_cc; LDL^T: unit L,
//           then division by D), then update the row block's columns right of the
//           step: A[b, c] -= L[b, j] (D_j) L[c, j]^T for every column block c > j
//           (c <= b among the diagonal block's rows; the lower triangle of tile (b, b)).
//
// Dependencies are counters in global memory, per row block: solved[b] = j + 1 once
// its columns of step j are final (for b == j: the factored tile), updated[b] = j + 1
// once its update of step j is done.  CTAs take items from an atomic ticket in a
// fixed order -- step by step, and within a step by row block (the critical tiles
// j and j + 1 of every cblk first) -- and every item depends only on items earlier
// in that order.  A CTA only ever waits for items that running CTAs have already
// taken, so the launch completes whatever the number of resident CTAs.  Every wait
// is bounded: on expiry the CTA sets bit 3 of err and an abort word that ends the
// other CTAs' waits, and returns.
//
// The solves of the tiles next to the critical path overlap with the rest of the
// step's rows and with the following steps (look-ahead without extra launches);
// the launch replaces three to four launches per 64-column step.
#include <algorithm>

#include "b200_internal.h"
#include "kernels.h"
#include "tile_ops.cuh"

namespace b200 {

namespace {

constexpr int PB = 64;   // tile edge
constexpr int XP = 68;   // pitch of the row block's columns (column-major, 16-byte aligned columns)
constexpr int PT = 256;  // threads per CTA
constexpr long long PANEL_WAIT_CYCLES = 1000000000LL;  // about 0.5 s at the maximum SM clock
constexpr int PANEL_SMEM_ELEMS = PB * PB + PB * XP + PB * PB + 3 * PB;

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Releases what the CTA wrote before its last barrier.
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait (one thread) until *flag >= target; returns the value seen, below target
// on expiry or abort.
__device__ int panel_wait(const int *flag, int target, const int *abort_word) {
    const long long t0 = clock64();
    for (int it = 0;; it++) {
        const int v = ld_acquire(flag);
        if (v >= target) return v;
        if ((it & 15) == 15) {
            if (ld_acquire(abort_word)) return v;
            if (clock64() - t0 > PANEL_WAIT_CYCLES) return v;
        }
        __nanosleep(32);
    }
}

template <typename T>
__device__ __forceinline__ void load4(const T *p, T v[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        const double2 q0 = *reinterpret_cast<const double2 *>(p), q1 = *reinterpret_cast<const double2 *>(p + 2);
        v[0] = q0.x; v[1] = q0.y; v[2] = q1.x; v[3] = q1.y;
    }
}

// bytes of a B-byte copy (the rest of it zeros) into shared memory
template <int B>
__device__ __forceinline__ void cp_async(void *dst, const void *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(B), "r"(bytes) : "memory");
}

template <typename T>
__device__ __forceinline__ void store4(T *p, T a, T b, T c, T d) {
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
    } else {
        *reinterpret_cast<double2 *>(p) = make_double2(a, b);
        *reinterpret_cast<double2 *>(p + 2) = make_double2(c, d);
    }
}

// Factorization of the wd x wd diagonal tile held in the registers of the CTA's 16 x 16
// threads: thread (tx, ty) has rows 4 tx .. 4 tx + 3 and columns 4 ty .. 4 ty + 3, acc[i][q]
// (identity past wd).  Step p: the half-warp of block column p takes the 4 x 4 diagonal
// block by shuffles, factors it in every lane and solves its own 4 columns with it (four
// dependent pivots), puts them in the strip, and after one barrier the threads right of
// it subtract their product.  The strip is double buffered, so the half-warp of the next
// step goes on as soon as its own columns are up to date.  What bounds a tile is this
// chain (16 steps of four pivots, a barrier and a strip read), not its multiply-adds;
// solving the strips in every thread that reads them, with no hand-off to wait for, took
// 825 cycles a step in FP32 and 2200 in FP64.  Static pivoting replaces a
// pivot below thr in magnitude by +-thr.  LDL^T keeps D on the diagonal and unit L below;
// LU keeps unit L below and U on and above the diagonal (its row strip is solved with the
// unit block by the threads that read it).
//
// An entry gathers the products of the 16-column blocks before its own from zero (its value
// waits in a slot of the strip's) and takes their sum in one subtraction when its own block's
// turn comes: 64 products subtracted one by one from the entry itself rounded 1.2 to 1.4 times
// worse than 32-column tiles (backward error of dense LU and LDL^T; twice in
// the factor of an indefinite 44 x 40 x 39 system).
// strip: 2 x STRIP elements, then 16 for each of 144 threads.
template <typename T, int FACTO>
__device__ void factor_tile_regs(T (&acc)[4][4], int wd, T *strip, double thr, int *s_piv, int *s_err) {
    constexpr int STRIP = 8 * PB;  // 4 solved columns, then LU's 4 raw rows; LDL^T's 4 pivots
    constexpr bool LU = FACTO == FACTO_GETRF;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    int piv = 0, neg = 0;
    constexpr int SLOTS = 144;
    const int turn = min(tx, ty) & ~3;  // the step at which the entry's own 16-column block begins
    const bool late = turn > 0 && 4 * turn < wd;
    T *slot = strip + 2 * STRIP + (tx - 4) + 12 * (ty - 4);  // this thread's, every SLOTS elements
    if (late) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                slot[SLOTS * (4 * i + q)] = acc[i][q];
                acc[i][q] = 0;
            }
    }
#pragma unroll 1
    for (int p = 0; 4 * p < wd; p++) {
        T *cb = strip + (p & 1) * STRIP, *rb = cb + 4 * PB;
        if (p == turn && late) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] += slot[SLOTS * (4 * i + q)];
        }
        if (ty == p) {
            const unsigned half = 0xffffu << (16 * (p & 1));
            T g[4][4], P[4][4], d[4], iv[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (LU || i >= k) g[i][k] = __shfl_sync(half, acc[i][k], p, 16);
                    P[i][k] = acc[i][k];
                }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                T a = g[c][c];
                const bool rep = fabs(a) < (T)thr;
                if (rep) a = (FACTO == FACTO_POTRF) ? (T)thr : ((a < (T)0) ? (T)(-thr) : (T)thr);
                if (4 * p + c < wd) piv += rep;
                if (FACTO == FACTO_POTRF) {
                    if (a < (T)0) {
                        if (4 * p + c < wd) neg = 1;
                        a = -a;
                    }
                    iv[c] = rsqrt(a);
                    d[c] = a * iv[c];
                } else {
                    iv[c] = (T)1 / a;
                    d[c] = a;
                }
                g[c][c] = d[c];
#pragma unroll
                for (int i = c + 1; i < 4; i++) g[i][c] *= iv[c];
#pragma unroll
                for (int j = c + 1; j < 4; j++)
#pragma unroll
                    for (int i = (LU ? c + 1 : j); i < 4; i++) {
                        if (LU) g[i][j] -= g[i][c] * g[c][j];
                        else if (FACTO == FACTO_SYTRF) g[i][j] -= (g[i][c] * d[c]) * g[j][c];
                        else g[i][j] -= g[i][c] * g[j][c];
                    }
                // this thread's rows: column c, and its terms in the columns after it
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    P[i][c] *= iv[c];
#pragma unroll
                    for (int j = c + 1; j < 4; j++) {
                        if (LU) P[i][j] -= P[i][c] * g[c][j];
                        else if (FACTO == FACTO_SYTRF) P[i][j] -= (P[i][c] * d[c]) * g[j][c];
                        else P[i][j] -= P[i][c] * g[j][c];
                    }
                }
            }
            if (LU && tx == p) {
                // the unit block, for the row strip's readers
#pragma unroll
                for (int k = 0; k < 4; k++) store4(cb + k * PB + 4 * p, g[0][k], g[1][k], g[2][k], g[3][k]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) store4(cb + k * PB + 4 * tx, P[0][k], P[1][k], P[2][k], P[3][k]);
            }
            if (FACTO == FACTO_SYTRF && tx == p) store4(rb, d[0], d[1], d[2], d[3]);
            if (tx == p) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (LU || i >= k) acc[i][k] = g[i][k];
            } else if (tx > p) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[i][k] = P[i][k];
            }
        }
        if (LU && tx == p && ty > p) {
#pragma unroll
            for (int i = 0; i < 4; i++) store4(rb + i * PB + 4 * ty, acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        if (ty <= p) continue;
        if (LU ? tx < p : tx < ty) continue;
        T P[4][4], Q[4][4];  // [row][k], [column][k]
#pragma unroll
        for (int k = 0; k < 4; k++) {
            T v[4];
            load4(cb + k * PB + 4 * tx, v);
#pragma unroll
            for (int i = 0; i < 4; i++) P[i][k] = v[i];
            load4((LU ? rb : cb) + k * PB + 4 * ty, v);
#pragma unroll
            for (int i = 0; i < 4; i++) Q[i][k] = v[i];
        }
        if (LU) {
            // Q = L_pp^{-1} (rows of A), the unit block's entries from the strip
            T l[4][4];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                T v[4];
                load4(cb + k * PB + 4 * p, v);
#pragma unroll
                for (int i = k + 1; i < 4; i++) l[i][k] = v[i];
            }
#pragma unroll
            for (int k = 0; k < 3; k++)
#pragma unroll
                for (int i = k + 1; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) Q[j][i] -= Q[j][k] * l[i][k];
            if (tx == p) {
#pragma unroll
                for (int k = 0; k < 4; k++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[k][j] = Q[j][k];
                continue;
            }
        }
        T d[4] = {(T)1, (T)1, (T)1, (T)1};
        if (FACTO == FACTO_SYTRF) load4(rb, d);
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const T m = (FACTO == FACTO_SYTRF) ? P[i][k] * d[k] : P[i][k];
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] -= m * Q[j][k];
            }
    }
    if (tx == 15) {  // one thread of every block column counted its pivots
        if (piv) atomicAdd(s_piv, piv);
        if (neg) *s_err = 1;
    }
}

// Rows of a tile loaded for factor_tile_regs: a(i, j) for i, j < wd (the lower triangle,
// LU both), identity past wd and zero above the diagonal.
template <typename T, int FACTO, typename Load>
__device__ __forceinline__ void load_tile_regs(T (&acc)[4][4], int wd, Load a) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = 4 * tx + i, c = 4 * ty + q;
            const bool in = r < wd && c < wd && (FACTO == FACTO_GETRF || r >= c);
            acc[i][q] = in ? a(r, c) : (r == c ? (T)1 : (T)0);
        }
}

// Solve of the R rows of xs (64 columns, pitch XP) against the lower triangular tile lt
// (lt[c + l * 64], l < c; identity past the step's width), x_c = (a_c - sum_{l<c} x_l t_cl)
// * rdiag[c], LDL^T then times dinv[c] = 1 / D_c, in 16-column blocks: one thread per row
// substitutes the block's columns in registers, then the threads of the columns right of it
// (thread (tx, ty): rows 4 tx + 64 h .., columns 4 ty ..) add its products to their sums,
// which are subtracted when the columns' own block comes.  A block's substitution keeps one
// warp per SM sub-partition busy (R = 128), its chain of 16 columns no longer than its
// multiply-adds; 4-column blocks of the threads (tx, ty), with 16 hand-offs, took 29.2 ms at
// 80^3 27-point split BF16 (28.2 now) and 20.4 ms for the 64^3 LU (19.9).  All PT threads; xs final after the closing barrier.
template <typename T, int FACTO, int R, int XP>
__device__ void trsm_tile(T *xs, const T *lt, const T *rdiag, const T *dinv) {
    constexpr int G = R / 64, CB = 16;  // groups of 64 rows; columns of a block
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    T *own = xs + 4 * tx + 4 * ty * XP;
    T acc[G][4][4] = {};  // [group][row][column]
#pragma unroll 1
    for (int c0 = 0; c0 < PB; c0 += CB) {
        if (c0 > 0) {
            if (4 * ty / CB == c0 / CB) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int h = 0; h < G; h++) {
                        T v[4];
                        load4(own + 64 * h + q * XP, v);
                        store4(own + 64 * h + q * XP, v[0] - acc[h][0][q], v[1] - acc[h][1][q], v[2] - acc[h][2][q],
                               v[3] - acc[h][3][q]);
                    }
            }
            __syncthreads();
        }
        if (tid < R) {
            T *row = xs + tid + c0 * XP;
            T x[CB];
#pragma unroll
            for (int c = 0; c < CB; c++) x[c] = row[c * XP];
#pragma unroll
            for (int l = 0; l < CB; l++) {
                x[l] *= rdiag[c0 + l];
#pragma unroll
                for (int c = l / 4 * 4; c < CB; c += 4) {
                    T t[4];
                    load4(lt + c0 + c + (c0 + l) * PB, t);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (c + q > l) x[c + q] -= x[l] * t[q];
                }
            }
#pragma unroll
            for (int c = 0; c < CB; c++) row[c * XP] = x[c];
        }
        __syncthreads();
        if (4 * ty / CB > c0 / CB) {
#pragma unroll 4
            for (int l = c0; l < c0 + CB; l++) {
                T t[4];
                load4(lt + 4 * ty + l * PB, t);
#pragma unroll
                for (int h = 0; h < G; h++) {
                    T v[4];
                    load4(xs + 4 * tx + 64 * h + l * XP, v);
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[h][i][q] += v[i] * t[q];
                }
            }
        }
    }
    if (FACTO == FACTO_SYTRF) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const T m = dinv[4 * ty + q];
#pragma unroll
            for (int h = 0; h < G; h++) {
                T v[4];
                load4(own + 64 * h + q * XP, v);
                store4(own + 64 * h + q * XP, v[0] * m, v[1] * m, v[2] * m, v[3] * m);
            }
        }
        __syncthreads();
    }
}

template <typename T>
__device__ __forceinline__ void load_vec(const T *p, T *v) {  // 16 bytes
    if constexpr (sizeof(T) == 4) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        const double2 q = *reinterpret_cast<const double2 *>(p);
        v[0] = q.x; v[1] = q.y;
    }
}
template <typename T>
__device__ __forceinline__ void store_vec(T *p, const T *v) {
    if constexpr (sizeof(T) == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
}

// acc = X B over 64 K values: X[r, l] = xs[l * R + r],
// B[l, c] = bs[l * 64 + c].  Thread (tx, ty): columns 4 ty .. 4 ty + 3, rows in groups of
// 16 bytes, group h at rows EPV (tx + 16 h) .. (a warp's reads of a group are 256
// contiguous bytes; 8 contiguous rows per thread met every bank twice).  The operands of
// the next l are read before the products of this one: two warps per SM sub-partition
// cannot hide a shared-memory read behind 16 or 32 multiply-adds otherwise (a 64 x 64 x 64
// FP32 product took 6.2 K cycles, three times its multiply-adds).
template <typename T, int R>
struct RowTile {
    static constexpr int MR = R / 16, EPV = 16 / (int)sizeof(T), G = MR / EPV;
    static __device__ __forceinline__ int row(int i) { return EPV * ((threadIdx.x & 15) + 16 * (i / EPV)) + i % EPV; }
    static __device__ __forceinline__ void mul(T (&acc)[MR][4], const T *xs, const T *bs) {
        const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
        const T *xp = xs + EPV * tx, *bp = bs + 4 * ty;
#pragma unroll
        for (int i = 0; i < MR; i++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][q] = 0;
        T av[2][MR], bv[2][4];
        auto fetch = [&](int l, int s) {
#pragma unroll
            for (int h = 0; h < G; h++) load_vec(xp + l * R + 16 * EPV * h, av[s] + EPV * h);
            load4(bp + l * PB, bv[s]);
        };
        fetch(0, 0);
#pragma unroll 1
        for (int l0 = 0; l0 < PB; l0 += 8) {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (u < 7 || l0 + 8 < PB) fetch(l0 + u + 1, (u + 1) & 1);
#pragma unroll
                for (int i = 0; i < MR; i++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[i][q] += av[u & 1][i] * bv[u & 1][q];
            }
        }
    }
};

template <typename T, int FACTO>
__global__ void __launch_bounds__(PT, sizeof(T) == 4 ? 2 : 1) panel_kernel(DevSym s, const PanelCblk *__restrict__ pcb,
                                                   const PanelItem *__restrict__ items, int nitems, int *ticket,
                                                   int *solved, int *updated, int *abort_word, T *L,
                                                   const double *__restrict__ thr_ptr, unsigned long long *npiv,
                                                   int *err) {
    extern __shared__ __align__(16) unsigned char pn_smem[];
    T *lt = reinterpret_cast<T *>(pn_smem);  // diagonal tile of the step
    T *xs = lt + PB * PB;                    // the row block's columns of the step (pitch XP)
    T *bs = xs + PB * XP;                    // update operand L[c, j] (D_j): bs[l * PB + row]
    T *rdiag = bs + PB * PB, *dinv = rdiag + PB, *dd = dinv + PB;
    __shared__ int s_item, s_ok, s_piv, s_err;
    const int tid = threadIdx.x;
    bool aborted = false;
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(ticket, 1);
            s_ok = 1;
            s_piv = 0;
            s_err = 0;
        }
        __syncthreads();
        const int t = s_item;
        if (t >= nitems) break;
        const PanelItem it = items[t];
        const PanelCblk pc = pcb[it.p];
        const int k = pc.k, j = it.j, b = it.b;
        const int W = s.ncols[k], S = s.stride[k], ld = s.ld[k];
        const double thr = cblk_threshold(s, thr_ptr, k);
        T *P = L + s.off[k];
        const int c0 = PB * j, wd = min(PB, W - c0);
        int *sol = solved + pc.flag0, *upd = updated + pc.flag0;
        if (tid == 0) {
            // the row block's update of the previous step, and the factored tile of this step
            if (j > 0 && panel_wait(upd + b, j, abort_word) < j) s_ok = 0;
            if (s_ok && b != j && panel_wait(sol + j, j + 1, abort_word) < j + 1) s_ok = 0;
        }
        __syncthreads();
        if (!s_ok) {
            aborted = true;
            break;
        }
        if (b == j) {
            // ---------------------------------------------- diagonal tile
            T *A = P + c0 + (size_t)c0 * ld;
            T acc[4][4];
            load_tile_regs<T, FACTO>(acc, wd, [&](int r, int c) { return __ldcg(A + r + (size_t)c * ld); });
            factor_tile_regs<T, FACTO>(acc, wd, lt, thr, &s_piv, &s_err);
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * (tid & 15) + i, c = 4 * (tid >> 4) + q;
                    if (r < wd && c < wd && r >= c) A[r + (size_t)c * ld] = acc[i][q];
                }
            __syncthreads();
            if (tid == 0) {
                if (s_piv) atomicAdd(cblk_pivot_counter(s, npiv, k), (unsigned long long)s_piv);
                if (s_err) atomicOr(err, 1);
                __threadfence();
                st_release(sol + b, j + 1);
                st_release(upd + b, j + 1);
            }
            __syncthreads();
            continue;
        }
        // -------------------------------------------------- solve of the row block
        const bool drows = b < pc.ns;
        const int r0 = drows ? PB * b : W + PB * (b - pc.ns);
        const int nr = min(PB, (drows ? W : S) - r0);
        const T *Dg = P + c0 + (size_t)c0 * ld;
        T *X = P + r0 + (size_t)c0 * ld;
        stage_n<PB * PB / PT, T>(
            [&](int u) {
                const int idx = tid + PT * u, c = idx & 63, l = idx >> 6;
                T v = 0;
                if (c < wd && l < wd) v = (c > l) ? __ldcg(Dg + c + (size_t)l * ld) : (c == l ? (T)1 : (T)0);
                else if (c == l) v = 1;
                return v;
            },
            [&](int u, T v) {
                const int idx = tid + PT * u;
                lt[idx] = v;
            });
        stage_n<PB * PB / PT, T>(
            [&](int u) {
                const int idx = tid + PT * u, r = idx & 63, c = idx >> 6;
                return (r < nr && c < wd) ? __ldcg(X + r + (size_t)c * ld) : (T)0;
            },
            [&](int u, T v) {
                const int idx = tid + PT * u;
                xs[(idx & 63) + (idx >> 6) * XP] = v;
            });
        if (tid < PB) {
            const T dgv = tid < wd ? __ldcg(Dg + (size_t)tid * (ld + 1)) : (T)1;
            rdiag[tid] = (FACTO == FACTO_POTRF) ? (T)1 / dgv : (T)1;
            dinv[tid] = (FACTO == FACTO_SYTRF) ? (T)1 / dgv : (T)1;
            dd[tid] = (FACTO == FACTO_SYTRF) ? dgv : (T)1;
        }
        __syncthreads();
        trsm_tile<T, FACTO, PB, XP>(xs, lt, rdiag, dinv);
        for (int idx = tid; idx < PB * wd; idx += PT) {
            const int r = idx & 63, c = idx >> 6;
            if (r < nr) X[r + (size_t)c * ld] = xs[r + c * XP];
        }
        __syncthreads();
        if (tid == 0 && drows) {
            __threadfence();
            st_release(sol + b, j + 1);
        }
        // -------------------------------------------------- update right of the step
        const int cmax = drows ? b : pc.ns - 1;
        const int tx = tid & 15, ty = tid >> 4;
        for (int c = j + 1; c <= cmax; c++) {
            if (tid == 0 && c != b && panel_wait(sol + c, j + 1, abort_word) < j + 1) s_ok = 0;
            __syncthreads();
            if (!s_ok) break;
            const int wc = min(PB, W - PB * c);
            const T *B = P + PB * c + (size_t)c0 * ld;
            stage_n<PB * PB / PT, T>(
                [&](int u) {
                    const int idx = tid + PT * u, rr = idx & 63, l = idx >> 6;
                    return (rr < wc && l < wd) ? __ldcg(B + rr + (size_t)l * ld) : (T)0;
                },
                [&](int u, T v) {
                    const int idx = tid + PT * u;
                    bs[idx] = (FACTO == FACTO_SYTRF) ? v * dd[idx >> 6] : v;
                });
            __syncthreads();
            T acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] = 0;
            for (int l = 0; l < wd; l++) {
                T av[4], bv[4];
                load4(xs + l * XP + 4 * tx, av);
                load4(bs + l * PB + 4 * ty, bv);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[i][q] += av[i] * bv[q];
            }
            T *C = P + r0 + (size_t)(PB * c) * ld;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int cc = 4 * ty + q;
                if (cc < wc) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int r = 4 * tx + i;
                        if (r < nr && (c != b || r >= cc)) {
                            T *p = C + r + (size_t)cc * ld;
                            *p = __ldcg(p) - acc[i][q];
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (!s_ok) {
            aborted = true;
            break;
        }
        if (tid == 0) {
            __threadfence();
            st_release(upd + b, j + 1);
        }
        __syncthreads();
    }
    if (aborted && tid == 0) {
        atomicOr(err, 8);
        st_release(abort_word, 1);
    }
}

// Row-block form (when a row block x the level's widest cblk fits in shared
// memory): one item per row block b, which keeps its rows resident in shared
// memory for all the steps -- solve of step j's columns, update of its columns
// right of the step, for every j before the row block's own diagonal tile (all ns
// steps for the rows below the diagonal block) -- and, for b < ns, finally
// factors its diagonal tile (b, b).  Each solved step of the diagonal block's
// rows is written back and announced at once (solved[b] = j + 1; b + 1 after the
// factorization), the only cross-item reads being the factored tiles L[j, j] and the
// diagonal block's solved tiles L[c, j].  Cholesky solves by substitution like the others:
// products with the tiles' inverses (no chain; 80^3 27-point split BF16 27.2 ms, 28.2 with
// it) lose digits with the tile's condition number: dense matrices of condition 1e13, 60 + 40
// columns, had a backward error of 6.9e-16, now 1.7e-16.  Row blocks: 64 rows in
// the diagonal block, R rows (64 or 128) below it.  Items: the diagonal blocks' row
// blocks of every cblk first (b ascending), then the rows below.
//
// LU (core_zgetrfsp / core_ztrsmsp, kernels/core_zgetrfsp.c:64-170, without row
// exchanges) is the same dataflow over two panels, L and V = U^T: a row block of side 0
// holds rows of L and is updated by L[b, c] -= L[b, j] V[c, j]^T, one of side 1 holds rows
// of V and is updated by V[b, c] -= V[b, j] L[c, j]^T; side 0 solves against V[j, j]
// (the stored U^T) and owns the diagonal tiles, side 1 against the unit L[j, j].
// solved counts side 0, solved_v side 1, whose item of a row block comes first.  The
// one-CTA diagonal blocks and row-by-row solves this replaces took 56 of the 66 ms of a
// 64^3 convection-diffusion LU in FP32; the panel launches take 7.0 ms.
struct RowsCtx {
    int *sol, *sol_v;     // counters of the cblk's row blocks
    const int *abort_word;
    int *known;           // shared: the counters' last values seen, [2][16]
    int *s_ok, *s_piv, *s_err;
    double thr;
};

// Wait until counter c of the given side has reached target, all threads; counters
// already seen that far cost one shared-memory read.
__device__ __forceinline__ bool rows_need(const RowsCtx &x, int side, int c, int target) {
    if (x.known[16 * side + c] < target) {  // the same value in every thread
        __syncthreads();
        if (threadIdx.x == 0) {
            const int v = panel_wait((side ? x.sol_v : x.sol) + c, target, x.abort_word);
            if (v < target) *x.s_ok = 0;
            x.known[16 * side + c] = v;
        }
        __syncthreads();
    }
    return *x.s_ok;
}

template <typename T, int FACTO, int R>
__device__ void rows_item(const DevSym &s, const PanelCblk &pc, int b, int side, T *L, T *U, T *lt, T *rdiag, T *dinv,
                          T *dd, T *xs, const RowsCtx &x) {
    constexpr bool LU = FACTO == FACTO_GETRF;
    const int tid = threadIdx.x;
    const int k = pc.k, W = s.ncols[k], S = s.stride[k], ld = s.ld[k];
    T *P = (LU && side ? U : L) + s.off[k];        // this side's panel
    T *Q = LU ? (side ? L : U) + s.off[k] : P;     // the panel its updates multiply with
    int *sol = side ? x.sol_v : x.sol;
    const int qside = LU ? 1 - side : 0;           // counters of Q
    const bool drows = b < pc.ns;
    const int r0 = drows ? PB * b : W + R * (b - pc.ns);
    const int nr = min(R, (drows ? W : S) - r0);
    // columns held (lower part for the diagonal block; V: left of its diagonal tile)
    const int ncol = drows ? (side ? PB * b : min(W, PB * (b + 1))) : W;
    const int nstep = drows ? b : pc.ns;                 // steps solved in this row block
    // the row block: rows past nr and (below the diagonal block) the last step's columns past
    // W as zeros; the whole of it in flight at once
    const int nzero = drows ? ncol : PB * pc.ns;
    constexpr int EPV = 16 / (int)sizeof(T);
    if (r0 % EPV == 0) {
        // 16-byte copies (every panel column starts on a 16-byte boundary)
        constexpr int RV = R / EPV;
        for (int idx = tid; idx < RV * nzero; idx += PT) {
            const int r = (idx % RV) * EPV, c = idx / RV;
            const int bytes = c < ncol && r < nr ? min(EPV, nr - r) * (int)sizeof(T) : 0;
            cp_async<16>(xs + r + c * R, bytes ? P + r0 + r + (size_t)c * ld : P, bytes);
        }
    } else {
        for (int idx = tid; idx < R * nzero; idx += PT) {
            const int r = idx % R, c = idx / R;
            const bool in = c < ncol && r < nr;
            cp_async<sizeof(T)>(xs + r + c * R, in ? P + r0 + r + (size_t)c * ld : P, in ? (int)sizeof(T) : 0);
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    if (LU && drows) {
        // the diagonal block is the sum of L's and the transposed U's (core_zgeadd): 8 rows x
        // 4 columns of it per warp access
        const int cfirst = side ? 0 : PB * b, nc = ncol - cfirst;
        __syncthreads();
        for (int t = tid >> 5; t < (PB / 8) * ((nc + 3) / 4); t += PT / 32) {
            const int r = 8 * (t % (PB / 8)) + (tid & 7), c = cfirst + 4 * (t / (PB / 8)) + ((tid & 31) >> 3);
            if (r < nr && c < ncol) xs[r + c * R] += __ldcg(Q + c + (size_t)(r0 + r) * ld);
        }
    }
    __syncthreads();
    const int tx = tid & 15, ty = tid >> 4;
    T pf[PB * PB / PT];  // tile read ahead: the next update operand, or the next step's diagonal tile
    // the tile the rows are solved against: lower triangle and diagonal, identity past W
    auto load_diag = [&](int j) {
        const int c0 = PB * j, wd = min(PB, W - c0);
        const T *Dg = Q + c0 + (size_t)c0 * ld;
#pragma unroll
        for (int u = 0; u < PB * PB / PT; u++) {
            const int idx = tid + PT * u, c = idx & 63, l = idx >> 6;
            pf[u] = (c < wd && l <= c) ? __ldcg(Dg + c + (size_t)l * ld) : (c == l ? (T)1 : (T)0);
        }
    };
    auto load_b = [&](int j, int c) {
        const int wd = min(PB, W - PB * j), wc = min(PB, W - PB * c);
        const T *B = Q + PB * c + (size_t)(PB * j) * ld;
#pragma unroll
        for (int u = 0; u < PB * PB / PT; u++) {
            const int idx = tid + PT * u, rr = idx & 63, l = idx >> 6;
            pf[u] = (rr < wc && l < wd) ? __ldcg(B + rr + (size_t)l * ld) : (T)0;
        }
    };
    bool have = false;  // pf holds the tile read next
    for (int j = 0; j < nstep; j++) {
        const int c0 = PB * j, wd = min(PB, W - c0);
        if (!have) {
            if (!rows_need(x, 0, j, j + 1)) return;
            load_diag(j);
        }
        have = false;
        // ---------------------------------------------- solve of step j's columns
#pragma unroll
        for (int u = 0; u < PB * PB / PT; u++) {
            const int idx = tid + PT * u, c = idx & 63;
            lt[idx] = pf[u];
            if (c == idx >> 6) {  // the diagonal, which the products do not read
                rdiag[c] = FACTO == FACTO_POTRF || (LU && side == 0) ? (T)1 / pf[u] : (T)1;
                if (FACTO == FACTO_SYTRF) {
                    dinv[c] = (T)1 / pf[u];
                    dd[c] = pf[u];
                }
            }
        }
        __syncthreads();
        trsm_tile<T, FACTO, R, R>(xs + c0 * R, lt, rdiag, dinv);
#pragma unroll 8
        for (int u = 0; u < R * PB / PT; u++) {
            const int r = (tid + PT * u) % R, c = (tid + PT * u) / R;
            if (r < nr && c < wd) P[r0 + r + (size_t)(c0 + c) * ld] = xs[r + (c0 + c) * R];
        }
        if (drows) {
            __syncthreads();
            if (tid == 0) {
                st_release(sol + b, j + 1);
            }
            if (LU)  // the other panel's diagonal block keeps the transposed factor (core_zgetmo)
                for (int t = tid >> 5; t < (PB / 8) * ((wd + 3) / 4); t += PT / 32) {
                    const int r = 8 * (t % (PB / 8)) + (tid & 7), c = c0 + 4 * (t / (PB / 8)) + ((tid & 31) >> 3);
                    if (r < nr && c < c0 + wd) Q[c + (size_t)(r0 + r) * ld] = xs[r + c * R];
                }
        }
        // ---------------------------------------------- update of the columns right of the step
        const int cmax = drows ? (side ? b - 1 : b) : pc.ns - 1;
        for (int c = j + 1; c <= cmax; c++) {
            const bool own = !LU && drows && c == b;  // this row block's solved columns, in shared memory
            if (!own && !have) {
                if (!rows_need(x, qside, c, j + 1)) return;
                load_b(j, c);
            }
            have = false;
            const int wc = min(PB, W - PB * c);
            T *bs = lt;  // bs[l * PB + row]
#pragma unroll
            for (int u = 0; u < PB * PB / PT; u++) {
                const int idx = tid + PT * u, rr = idx & 63, l = idx >> 6;
                const T v = own ? ((rr < wc && l < wd) ? xs[rr + (c0 + l) * R] : (T)0) : pf[u];
                bs[idx] = (FACTO == FACTO_SYTRF) ? v * dd[l] : v;
            }
            __syncthreads();
            // read ahead what comes next, when it is known to be there
            if (c < cmax) {
                if (!(!LU && drows && c + 1 == b) && x.known[16 * qside + c + 1] >= j + 1) {
                    load_b(j, c + 1);
                    have = true;
                }
            } else if (j + 1 < nstep && x.known[j + 1] >= j + 2) {
                load_diag(j + 1);
                have = true;
            }
            using RT = RowTile<T, R>;
            T acc[RT::MR][4];
            RT::mul(acc, xs + c0 * R, bs);  // a step with columns right of it is a full one
            T *xc = xs + (PB * c) * R;
            if (own) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int i = 0; i < RT::MR; i++) {
                        const int r = RT::row(i), cc = 4 * ty + q;
                        if (cc < wc && r >= cc) xc[r + cc * R] -= acc[i][q];
                    }
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int h = 0; h < RT::G; h++) {
                        if (4 * ty + q >= wc) continue;
                        T *p = xc + RT::EPV * (tx + 16 * h) + (4 * ty + q) * R;
                        T v[RT::EPV];
                        load_vec(p, v);
#pragma unroll
                        for (int i = 0; i < RT::EPV; i++) v[i] -= acc[RT::EPV * h + i][q];
                        store_vec(p, v);
                    }
            }
            __syncthreads();
        }
    }
    if (drows && side == 0) {
        // ---------------------------------------------- the row block's diagonal tile
        const int c0 = PB * b, wd = min(PB, W - c0);
        T *xt = xs + c0 * R;
        T acc[4][4];
        load_tile_regs<T, FACTO>(acc, wd, [&](int r, int c) { return xt[r + c * R]; });
        __syncthreads();
        factor_tile_regs<T, FACTO>(acc, wd, xt, x.thr, x.s_piv, x.s_err);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (LU || tx >= ty) store4(xt + 4 * tx + (4 * ty + q) * R, acc[0][q], acc[1][q], acc[2][q], acc[3][q]);
        __syncthreads();
        for (int idx = tid; idx < PB * PB; idx += PT) {
            const int i = idx & 63, jj = idx >> 6;
            if (i < wd && jj < wd && (LU || i >= jj)) P[c0 + i + (size_t)(c0 + jj) * ld] = xt[i + jj * R];
        }
        if (LU)
            for (int t = tid >> 5; t < (PB / 8) * ((wd + 3) / 4); t += PT / 32) {
                const int i = 8 * (t % (PB / 8)) + (tid & 7), jj = 4 * (t / (PB / 8)) + ((tid & 31) >> 3);
                if (i < wd && jj < wd) Q[c0 + jj + (size_t)(c0 + i) * ld] = xt[i + jj * R];
            }
        __syncthreads();
        if (tid == 0) {
            st_release(sol + b, b + 1);
        }
    }
}

template <typename T, int FACTO, int RB>
__global__ void __launch_bounds__(PT, 1)
    panel_rows_kernel(DevSym s, const PanelCblk *__restrict__ pcb, const PanelItem *__restrict__ items, int nitems,
                      int *ticket, int *solved, int *solved_v, int *abort_word, T *L, T *U,
                      const double *__restrict__ thr_ptr, unsigned long long *npiv, int *err) {
    extern __shared__ __align__(16) unsigned char pn_smem[];
    T *lt = reinterpret_cast<T *>(pn_smem);  // the solve's tile; the update's operand
    T *rdiag = lt + PB * PB, *dinv = rdiag + PB, *dd = dinv + PB;
    T *xs = dd + PB;                         // the row block, column-major (pitch = its rows)
    __shared__ int s_item, s_ok, s_piv, s_err;
    __shared__ int s_known[32];
    const int tid = threadIdx.x;
    bool aborted = false;
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(ticket, 1);
            s_ok = 1;
            s_piv = 0;
            s_err = 0;
        }
        if (tid < 32) s_known[tid] = 0;
        __syncthreads();
        const int t = s_item;
        if (t >= nitems) break;
        const PanelItem it = items[t];
        const PanelCblk pc = pcb[it.p];
        const RowsCtx x{solved + pc.flag0, solved_v + pc.flag0, abort_word, s_known, &s_ok, &s_piv, &s_err,
                        cblk_threshold(s, thr_ptr, pc.k)};
        if (it.b < pc.ns) rows_item<T, FACTO, PB>(s, pc, it.b, it.j, L, U, lt, rdiag, dinv, dd, xs, x);
        else rows_item<T, FACTO, RB>(s, pc, it.b, it.j, L, U, lt, rdiag, dinv, dd, xs, x);
        __syncthreads();
        if (!s_ok) {
            aborted = true;
            break;
        }
        if (tid == 0) {
            if (s_piv) atomicAdd(cblk_pivot_counter(s, npiv, pc.k), (unsigned long long)s_piv);
            if (s_err) atomicOr(err, 1);
        }
        __syncthreads();
    }
    if (aborted && tid == 0) {
        atomicOr(err, 8);
        st_release(abort_word, 1);
    }
}

int g_panel_ctas = 0;  // resident CTAs of the panel kernel on the device (all SMs)
int g_sms = 0, g_smem_optin = 0;
constexpr int PANEL_STATIC_SMEM = 256;  // room for the kernels' static shared variables

constexpr size_t rows_smem_elems(int nsmax, int rb) { return (size_t)PB * PB + 3 * PB + (size_t)rb * PB * nsmax; }

template <typename T, int FACTO>
int panel_occupancy() {
    const size_t smem = PANEL_SMEM_ELEMS * sizeof(T);
    if (cudaFuncSetAttribute(panel_kernel<T, FACTO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return 0;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_kernel<T, FACTO>, PT, smem) != cudaSuccess) return 0;
    return occ;
}

}  // namespace

int configure_panel_kernels() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&g_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return -1;
    g_sms = sms;
    const int dyn = g_smem_optin - PANEL_STATIC_SMEM;
    const void *rows[] = {
        (const void *)panel_rows_kernel<double, FACTO_POTRF, PB>, (const void *)panel_rows_kernel<double, FACTO_SYTRF, PB>,
        (const void *)panel_rows_kernel<double, FACTO_GETRF, PB>, (const void *)panel_rows_kernel<float, FACTO_POTRF, PB>,
        (const void *)panel_rows_kernel<float, FACTO_SYTRF, PB>, (const void *)panel_rows_kernel<float, FACTO_GETRF, PB>,
        (const void *)panel_rows_kernel<float, FACTO_POTRF, 2 * PB>,
        (const void *)panel_rows_kernel<float, FACTO_SYTRF, 2 * PB>,
        (const void *)panel_rows_kernel<float, FACTO_GETRF, 2 * PB>};
    for (const void *f : rows)
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn)) return -1;
    int occ = panel_occupancy<double, FACTO_POTRF>();
    occ = std::min(occ, panel_occupancy<double, FACTO_SYTRF>());
    occ = std::min(occ, panel_occupancy<float, FACTO_POTRF>());
    occ = std::min(occ, panel_occupancy<float, FACTO_SYTRF>());
    if (occ <= 0) return -1;
    g_panel_ctas = occ * sms;
    return 0;
}

template <typename T>
void launch_panel(int facto, const DevSym &s, const PanelCblk *pcb, const PanelItem *items, int nitems, int *ticket,
                  int *solved, int *updated, int *abort_word, T *L, const double *thr, unsigned long long *npiv,
                  int *err, cudaStream_t st) {
    if (nitems <= 0) return;
    const int grid = std::min(nitems, g_panel_ctas);
    const size_t smem = PANEL_SMEM_ELEMS * sizeof(T);
    if (facto == FACTO_POTRF)
        panel_kernel<T, FACTO_POTRF><<<grid, PT, smem, st>>>(s, pcb, items, nitems, ticket, solved, updated,
                                                            abort_word, L, thr, npiv, err);
    else
        panel_kernel<T, FACTO_SYTRF><<<grid, PT, smem, st>>>(s, pcb, items, nitems, ticket, solved, updated,
                                                            abort_word, L, thr, npiv, err);
}

int panel_rows_block(int nsmax, size_t esz) {
    const size_t lim = (size_t)g_smem_optin - PANEL_STATIC_SMEM;
    if (esz == 4 && rows_smem_elems(nsmax, 2 * PB) * esz <= lim) return 2 * PB;
    return rows_smem_elems(nsmax, PB) * esz <= lim ? PB : 0;
}

template <typename T, int FACTO, int RB>
static void launch_rows(const DevSym &s, const PanelCblk *pcb, const PanelItem *items, int nitems, int nsmax,
                        int *ticket, int *solved, int *solved_v, int *abort_word, T *L, T *U,
                        const double *thr, unsigned long long *npiv, int *err, cudaStream_t st) {
    const size_t smem = rows_smem_elems(nsmax, RB) * sizeof(T);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, panel_rows_kernel<T, FACTO, RB>, PT, smem);
    const int grid = std::min(nitems, std::max(occ, 1) * g_sms);
    panel_rows_kernel<T, FACTO, RB><<<grid, PT, smem, st>>>(s, pcb, items, nitems, ticket, solved, solved_v, abort_word,
                                                           L, U, thr, npiv, err);
}

template <typename T>
void launch_panel_rows(int facto, const DevSym &s, const PanelCblk *pcb, const PanelItem *items, int nitems,
                       int nsmax, int rb, int *ticket, int *solved, int *solved_v, int *abort_word, T *L, T *U,
                       const double *thr, unsigned long long *npiv, int *err, cudaStream_t st) {
    if (nitems <= 0) return;
    auto run = [&](auto f, auto r) {
        launch_rows<T, decltype(f)::value, decltype(r)::value>(s, pcb, items, nitems, nsmax, ticket, solved, solved_v,
                                                               abort_word, L, U, thr, npiv, err, st);
    };
    auto by_facto = [&](auto r) {
        if (facto == FACTO_POTRF) run(std::integral_constant<int, FACTO_POTRF>{}, r);
        else if (facto == FACTO_SYTRF) run(std::integral_constant<int, FACTO_SYTRF>{}, r);
        else run(std::integral_constant<int, FACTO_GETRF>{}, r);
    };
    if constexpr (sizeof(T) == 4) {
        if (rb == 2 * PB) {
            by_facto(std::integral_constant<int, 2 * PB>{});
            return;
        }
    }
    by_facto(std::integral_constant<int, PB>{});
}

template void launch_panel_rows<double>(int, const DevSym &, const PanelCblk *, const PanelItem *, int, int, int, int *,
                                        int *, int *, int *, double *, double *,
                                        const double *, unsigned long long *, int *, cudaStream_t);
template void launch_panel_rows<float>(int, const DevSym &, const PanelCblk *, const PanelItem *, int, int, int, int *,
                                       int *, int *, int *, float *, float *,
                                       const double *, unsigned long long *, int *, cudaStream_t);

template void launch_panel<double>(int, const DevSym &, const PanelCblk *, const PanelItem *, int, int *, int *, int *,
                                   int *, double *, const double *, unsigned long long *, int *, cudaStream_t);
template void launch_panel<float>(int, const DevSym &, const PanelCblk *, const PanelItem *, int, int *, int *, int *,
                                  int *, float *, const double *, unsigned long long *, int *, cudaStream_t);

}  // namespace b200
