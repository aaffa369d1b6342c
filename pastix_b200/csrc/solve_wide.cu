// Triangular sweeps of many right-hand sides at once.
//
// The vectors are held row-major (row i of the permuted block at x + i * ldr, its
// right-hand sides contiguous), so that a panel row's gather, its atomic accumulation
// and a cblk's rows are whole cache lines, and a tile of outputs runs its product over
// all the K values of the cblk (or over a segment of the panel's rows) before it goes
// out: one atomic per output instead of one per 64 K values.  The products are those of
// the narrow sweeps (solve_blok_zgemm and the diagonal products, kernels/solve_ztrsmsp.c:
// 275-280): forward  aux_k = W_k x_k, x[rows below] -= P_k aux_k; backward
// aux_k -= P_k^T x[rows below], x_k = W_k^T aux_k, W_k the inverse of the diagonal block.
#include <algorithm>
#include <type_traits>

#include "b200_internal.h"
#include "kernels.h"

namespace b200 {

namespace {

constexpr int WT = 64;  // outputs of a tile
constexpr int WK = 32;  // K values of a pipeline stage
enum { W_OFF_FWD = 0, W_OFF_BWD = 1, W_DIAG_FWD = 2, W_DIAG_BWD = 3 };

__device__ __forceinline__ unsigned smem_a(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
template <int B>
__device__ __forceinline__ void cp_async_n(void *dst, const void *src, int bytes) {
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_a(dst)), "l"(src), "r"(bytes));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(smem_a(dst)), "l"(src), "n"(B), "r"(bytes));
}
__device__ __forceinline__ void cp_commit_g() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait_g() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma_k16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
        "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
          "d"(b[1]), "d"(b[2]), "d"(b[3]));
}
__device__ __forceinline__ void mma_tf32_k8(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo: hi is x rounded to TF32's 11 bits (half an ulp added, the rest masked), so lo
// has either sign and the bit of it that the tensor core drops is not one-sided.
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}

template <typename T, int MODE, int NT>
struct WideSmem {
    static constexpr bool ROW = MODE == W_OFF_FWD || MODE == W_DIAG_FWD;
    static constexpr int EPV = 16 / (int)sizeof(T);
    static constexpr int RW = NT * 8;  // right-hand sides of a tile
    static constexpr int THREADS = 128;
    static constexpr int STAGES = sizeof(T) == 8 ? 2 : 3;  // 64 columns: 72 KB (3 CTAs per SM) and 55 KB (4)
    // pitches of conflict-free operand reads: ms[kk][output] (ROW) or ms[output][kk]
    static constexpr int PM = ROW ? WT + 8 : WK + 4;
    static constexpr int XP = RW + (sizeof(T) == 8 ? 4 : 8);
    static constexpr int MS = ROW ? WK * PM : WT * PM;
    static constexpr int STAGE = MS + WK * XP;
    static constexpr int OP = RW + 1;  // pitch of the output staging
    static constexpr int ELEMS = STAGES * STAGE > WT * OP ? STAGES * STAGE : WT * OP;
    static constexpr int BYTES = ELEMS * (int)sizeof(T);
};

// Products of one stage, sums in registers; out(): put the sums into os[output][column].
//
// FP64: DMMA m16n8k16, warp = 16 outputs x all columns (ntn groups of 8 in use).
template <typename T, int MODE, int NT>
struct WideTile {
    using SM = WideSmem<T, MODE, NT>;
    double acc[NT][4] = {};
    __device__ __forceinline__ void mul(const double *ms, const double *xs, int nout, int ntn) {
        const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3, o0w = (threadIdx.x >> 5) * 16;
        if (o0w >= nout) return;
#pragma unroll
        for (int kk = 0; kk < WK; kk += 16) {
            double a[8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int kq = kk + 4 * j + tg;
                a[2 * j] = SM::ROW ? ms[kq * SM::PM + o0w + g] : ms[(o0w + g) * SM::PM + kq];
                a[2 * j + 1] = SM::ROW ? ms[kq * SM::PM + o0w + g + 8] : ms[(o0w + g + 8) * SM::PM + kq];
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                if (nt < ntn) {
                    double b[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) b[j] = xs[(kk + 4 * j + tg) * SM::XP + nt * 8 + g];
                    dmma_k16(acc[nt], a, b);
                }
            }
        }
    }
    __device__ __forceinline__ void out(double *os) {
        const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3, o0w = (threadIdx.x >> 5) * 16;
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                os[(o0w + g + (e >> 1) * 8) * SM::OP + nt * 8 + 2 * tg + (e & 1)] = acc[nt][e];
    }
};

// FP32: 3xTF32 on mma.sync m16n8k8 (x = hi + lo, both in TF32), warp = 16 outputs x all
// columns.  The tensor core rounds its sums towards zero, which adds up over products of one
// sign: every 8 products start from zero, the small correction products first, and join the
// tile's sum in FP32.  The solutions' error against the 64-bit solve with the same FP32
// factor (b > 0, 40 x 41 x 39): 5.1e-7, the column-major tiles' 5.0e-6; a truncated hi, and
// sums over 32 products with the correction products in them, had 9.3e-6, and took 4.5 %
// less time (100^3, 64 right-hand sides, solve and CG: 53.3 ms, 55.8 now).  Plain
// multiply-adds (8 x 4 and 8 x 8 sums per thread) are bound by their shared-memory reads and
// were slower.
template <int MODE, int NT>
struct WideTile<float, MODE, NT> {
    using SM = WideSmem<float, MODE, NT>;
    float sum[NT][4] = {};
    __device__ __forceinline__ void mul(const float *ms, const float *xs, int nout, int ntn) {
        const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3, o0w = (threadIdx.x >> 5) * 16;
        if (o0w >= nout) return;
#pragma unroll
        for (int kk = 0; kk < WK; kk += 8) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int kq = kk + tg + 4 * (j >> 1), o = o0w + g + 8 * (j & 1);
                split_tf32(SM::ROW ? ms[kq * SM::PM + o] : ms[o * SM::PM + kq], ah[j], al[j]);
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                if (nt < ntn) {
                    uint32_t bh[2], bl[2];
                    split_tf32(xs[(kk + tg) * SM::XP + nt * 8 + g], bh[0], bl[0]);
                    split_tf32(xs[(kk + tg + 4) * SM::XP + nt * 8 + g], bh[1], bl[1]);
                    float t[4] = {};
                    mma_tf32_k8(t, al, bh);
                    mma_tf32_k8(t, ah, bl);
                    mma_tf32_k8(t, ah, bh);
#pragma unroll
                    for (int e = 0; e < 4; e++) sum[nt][e] += t[e];
                }
            }
        }
    }
    __device__ __forceinline__ void out(float *os) {
        const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3, o0w = (threadIdx.x >> 5) * 16;
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                os[(o0w + g + (e >> 1) * 8) * SM::OP + nt * 8 + 2 * tg + (e & 1)] = sum[nt][e];
    }
};

// One stage of a factor tile: K values [kc, kc + 32) up to k1, outputs [o0, o1) (at most
// 64), zeros outside; vec: every line of M starts on a 16-byte boundary.
template <typename T, typename SM>
__device__ __forceinline__ void stage_factor(T *ms, const T *Mk, int ldm, int kc, int k1, int o0, int o1, bool vec) {
    constexpr bool ROW = SM::ROW;
    constexpr int LINES = ROW ? WK : WT, LEN = ROW ? WT : WK, EPV = SM::EPV, CPL = LEN / EPV;
    // lines (ROW: K values, else outputs) of contiguous entries
    const int tid = threadIdx.x, line0 = ROW ? kc : o0, nline = ROW ? k1 : o1, e0 = ROW ? o0 : kc, e1 = ROW ? o1 : k1;
    if (vec) {
#pragma unroll
        for (int u = 0; u < LINES * CPL / SM::THREADS; u++) {
            const int idx = tid + SM::THREADS * u, l = idx / CPL, i = (idx % CPL) * EPV;
            int bytes = 0;
            if (line0 + l < nline && e0 + i < e1) bytes = min(EPV, e1 - e0 - i) * (int)sizeof(T);
            cp_async_n<16>(ms + l * SM::PM + i, bytes ? Mk + e0 + i + (size_t)(line0 + l) * ldm : Mk, bytes);
        }
    } else {
#pragma unroll 4
        for (int u = 0; u < LINES * LEN / SM::THREADS; u++) {
            const int idx = tid + SM::THREADS * u, l = idx / LEN, i = idx % LEN;
            const bool ok = line0 + l < nline && e0 + i < e1;
            cp_async_n<sizeof(T)>(ms + l * SM::PM + i, ok ? Mk + e0 + i + (size_t)(line0 + l) * ldm : Mk,
                                  ok ? (int)sizeof(T) : 0);
        }
    }
}

// One tile: 64 outputs of task {k, o0, k0, k1} x the right-hand sides
// [q0, q0 + 8 NT), q0 = 8 NT blockIdx.y (rows of the vectors start on 16-byte boundaries):
//   OFF_FWD  x[row o] -= sum_{k0 <= c < k1} P[o, c] aux[c]     (o panel rows; atomic)
//   OFF_BWD  aux[o]   -= sum_{k0 <= r < k1} P[r, o] x[row r]   (o columns; atomic)
//   DIAG_FWD aux[o]    = sum_c W[o, c] x[c]      DIAG_BWD x[o] = sum_r W[r, o] aux[r]
// Panel rows start at a multiple of 4 at or below the first off-diagonal row n (16-byte
// copies); rows below n are dropped (forward) or meet zeros (backward).  A
// cp.async pipeline over chunks of 32 K values.
template <typename T, int MODE, int NT>
__global__ void __launch_bounds__(WideSmem<T, MODE, NT>::THREADS) wide_mm_kernel(DevSym s, const WideTask *__restrict__ tasks,
                                                      const T *__restrict__ M, const int64_t *__restrict__ woff,
                                                      const T *in, T *out, int ldr, int nrhs) {
    using SM = WideSmem<T, MODE, NT>;
    constexpr bool OFF = MODE == W_OFF_FWD || MODE == W_OFF_BWD;
    constexpr int XP = SM::XP, EPV = SM::EPV;
    extern __shared__ __align__(16) unsigned char wd_smem[];
    T *sm = reinterpret_cast<T *>(wd_smem);
    const WideTask t = tasks[blockIdx.x];
    const int k = t.k, n = s.ncols[k], f0 = s.fcol[k];
    const int q0 = blockIdx.y * SM::RW, R = min(SM::RW, nrhs - q0), ntn = (R + 7) >> 3;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldm = OFF ? s.ld[k] : n;
    const int nout = min(WT, (MODE == W_OFF_FWD ? s.stride[k] : n) - t.o0);
    const T *Mk = M + (OFF ? s.off[k] : woff[k]);
    const int *prow = OFF ? s.prow + s.rbase[k] : nullptr;
    const bool vec = OFF || n % EPV == 0;  // 16-byte copies of the factor

    auto load = [&](int st, int kc) {
        T *ms = sm + st * SM::STAGE, *xs = ms + SM::MS;
        stage_factor<T, SM>(ms, Mk, ldm, kc, t.k1, t.o0, t.o0 + nout, vec);
        // right-hand sides of the chunk's K values
        auto xrow = [&](int kk) { return in + (size_t)(MODE == W_OFF_BWD ? __ldg(prow + kk) : f0 + kk) * ldr + q0; };
        auto used = [&](int kk) { return kk < t.k1 && (MODE != W_OFF_BWD || kk >= n); };
        constexpr int CPL = SM::RW / EPV;
#pragma unroll
        for (int u = 0; u < (WK * CPL + SM::THREADS - 1) / SM::THREADS; u++) {
            const int idx = tid + SM::THREADS * u, l = idx / CPL, j = (idx % CPL) * EPV;
            const bool ok = used(kc + l) && j < R;
            cp_async_n<16>(xs + l * XP + j, ok ? xrow(kc + l) + j : in, ok ? 16 : 0);
        }
    };

    WideTile<T, MODE, NT> tile;
    const int nk = (t.k1 - t.k0 + WK - 1) / WK;
#pragma unroll
    for (int st = 0; st < SM::STAGES - 1; st++) {
        if (st < nk) load(st, t.k0 + st * WK);
        cp_commit_g();
    }
#pragma unroll 1
    for (int i = 0; i < nk; i++) {
        cp_wait_g<SM::STAGES - 2>();
        __syncthreads();
        if (i + SM::STAGES - 1 < nk) load((i + SM::STAGES - 1) % SM::STAGES, t.k0 + (i + SM::STAGES - 1) * WK);
        cp_commit_g();
        const T *ms = sm + (i % SM::STAGES) * SM::STAGE;
        tile.mul(ms, ms + SM::MS, nout, ntn);
    }
    cp_wait_g<0>();
    __syncthreads();
    // outputs through shared memory, so that a warp adds (stores) whole rows
    tile.out(sm);
    __syncthreads();
    constexpr int CG = SM::RW < 32 ? SM::RW : 32, RG = 32 / CG;  // columns of a row, rows at a time
#pragma unroll 4
    for (int i = warp * RG + lane / CG; i < nout; i += SM::THREADS / 32 * RG) {
        const int o = t.o0 + i;
        if (MODE == W_OFF_FWD && o < n) continue;
        T *row = out + (size_t)(MODE == W_OFF_FWD ? __ldg(prow + o) : f0 + o) * ldr + q0;
#pragma unroll
        for (int j0 = 0; j0 < SM::RW; j0 += CG) {
            const int j = j0 + lane % CG;
            if (j >= R) continue;
            const T v = sm[i * SM::OP + j];
            if (OFF) atomicAdd(row + j, -v);
            else row[j] = v;
        }
    }
}

// Cblks of at most WIDE_LEAF columns: both products of one sweep by one warp for 32
// right-hand sides, lane = right-hand side, the cblk's rows of the vectors in registers.
// 32 rows of the panel at a time are staged with a row per line and read as broadcasts.
constexpr int WL_WARPS = 4;

template <typename T>
__device__ __forceinline__ void stage_rows(T (*ps)[WIDE_LEAF], const T *m, int ldm, int n, int nr, int lane) {
    T v[WIDE_LEAF];
#pragma unroll
    for (int c = 0; c < WIDE_LEAF; c++) v[c] = (c < n && lane < nr) ? m[lane + (size_t)c * ldm] : (T)0;
#pragma unroll
    for (int c = 0; c < WIDE_LEAF; c++) ps[lane][c] = v[c];
}

template <typename T>
__global__ void __launch_bounds__(32 * WL_WARPS) wide_leaf_kernel(DevSym s, const int *__restrict__ cblks, int ncblk,
                                                                  const T *__restrict__ P, const T *__restrict__ W,
                                                                  const int64_t *__restrict__ woff, T *x, T *aux,
                                                                  int ldr, int nrhs, int backward) {
    __shared__ __align__(16) T smem[WL_WARPS][32][WIDE_LEAF];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T(*ps)[WIDE_LEAF] = smem[w];
    const int ci = blockIdx.x * WL_WARPS + w;
    if (ci >= ncblk) return;
    const int k = cblks[ci];
    const int n = s.ncols[k], ld = s.ld[k], stride = s.stride[k], f0 = s.fcol[k];
    const T *Pk = P + s.off[k], *Wk = W + woff[k];
    const int *prow = s.prow + s.rbase[k];
    const int q = blockIdx.y * 32 + lane;
    const bool in = q < nrhs;
    T v[WIDE_LEAF];  // forward: aux_k; backward: aux_k - P_k^T x
    const T *src = (backward ? aux : x) + (size_t)f0 * ldr + q;
#pragma unroll
    for (int c = 0; c < WIDE_LEAF; c++) v[c] = (c < n && in) ? src[(size_t)c * ldr] : (T)0;
    stage_rows<T>(ps, Wk, n, n, n, lane);  // W_k[r][c]
    __syncwarp();
    if (!backward) {
#pragma unroll
        for (int r = WIDE_LEAF - 1; r >= 0; r--) {
            T a = 0;
#pragma unroll
            for (int c = 0; c <= r; c++) a += ps[r][c] * v[c];
            v[r] = a;
            if (r < n && in) aux[(size_t)(f0 + r) * ldr + q] = a;
        }
    }
    for (int b = n; b < stride; b += 32) {
        const int nr = min(32, stride - b), myg = lane < nr ? prow[b + lane] : 0;
        __syncwarp();
        stage_rows<T>(ps, Pk + b, ld, n, nr, lane);
        __syncwarp();
        for (int r0 = 0; r0 < nr; r0 += 4) {
            T *row[4];
            T a[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                row[i] = x + (size_t)__shfl_sync(0xffffffffu, myg, r0 + i) * ldr + q;
                a[i] = (backward && in && r0 + i < nr) ? *row[i] : (T)0;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (backward) {
#pragma unroll
                    for (int c = 0; c < WIDE_LEAF; c++) v[c] -= ps[r0 + i][c] * a[i];
                } else {
#pragma unroll
                    for (int c = 0; c < WIDE_LEAF; c++) a[i] += ps[r0 + i][c] * v[c];
                    if (in && r0 + i < nr) atomicAdd(row[i], -a[i]);
                }
            }
        }
    }
    if (backward) {
        __syncwarp();
        stage_rows<T>(ps, Wk, n, n, n, lane);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < WIDE_LEAF; c++) {
            T a = 0;
#pragma unroll
            for (int r = c; r < WIDE_LEAF; r++) a += ps[r][c] * v[r];
            if (c < n && in) x[(size_t)(f0 + c) * ldr + q] = a;
        }
    }
}

// The narrow top of the tree as one launch per sweep: the tiles above as items of 64
// outputs x 64 K values taken in order from a ticket, each waiting for the counters of its
// inputs (solve_flow_kernel's, FI_DIAG and FI_OFF items; the cblks have more than WIDE_LEAF
// columns).  An item's factor tile is on its way before it waits; its vectors, which other
// items of the launch write, are read through L2.  One tile covers all the right-hand sides
// (8 NT at most).  Outputs accumulate: the rows of aux
// (forward) and x (backward) of the launch's cblks are zero before it.
constexpr long long WFLOW_WAIT_CYCLES = 1000000000LL;  // about 0.5 s at the maximum SM clock

__device__ __forceinline__ int wflow_ld(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ bool wflow_wait(const int *c, int target, const int *abort_word) {
    const long long t0 = clock64();
    for (int it = 0;; it++) {
        if (wflow_ld(c) >= target) return true;
        if ((it & 15) == 15) {
            if (wflow_ld(abort_word)) return false;
            if (clock64() - t0 > WFLOW_WAIT_CYCLES) return false;
        }
        __nanosleep(32);
    }
}

template <typename T, int BWD, int NT>
struct WideFlowSmem {
    using SM = WideSmem<T, BWD ? W_OFF_BWD : W_OFF_FWD, NT>;
    static constexpr int XS = 2 * WK * SM::XP, OS = WT * SM::OP;
    static constexpr int BYTES = (2 * SM::MS + (XS > OS ? XS : OS)) * (int)sizeof(T);
};

template <typename T, int BWD, int NT>
__global__ void __launch_bounds__(WideSmem<T, BWD ? W_OFF_BWD : W_OFF_FWD, NT>::THREADS) wide_flow_kernel(DevSym s, WideFlow fw, int nitems,
                                                        const FlowItem *__restrict__ items, const T *P, const T *W,
                                                        const int64_t *__restrict__ woff, T *x, T *aux, int ldr,
                                                        int nrhs, int *ticket, int *cnt_a, int *cnt_b, int *abort_word,
                                                        int *err) {
    constexpr int MODE = BWD ? W_OFF_BWD : W_OFF_FWD;
    using SM = WideSmem<T, MODE, NT>;
    constexpr int XP = SM::XP, EPV = SM::EPV;
    extern __shared__ __align__(16) unsigned char wf_smem[];
    T *ms = reinterpret_cast<T *>(wf_smem), *xs = ms + 2 * SM::MS, *os = xs;
    __shared__ int s_item, s_ok;
    const int *need = BWD ? fw.need_b : fw.need_f, *nprev = BWD ? fw.nprev_b : fw.nprev_f;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntn = (nrhs + 7) >> 3;
    bool aborted = false;
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(ticket, 1);
            s_ok = 1;
        }
        __syncthreads();
        const int ti = s_item;
        if (ti >= nitems) break;
        const FlowItem it = items[ti];
        const int k = it.k, n = s.ncols[k], f0 = s.fcol[k];
        const bool diag = it.type == FI_DIAG;
        const int *prow = s.prow + s.rbase[k];
        // outputs [o0, o1), K values [k0, k1): diagonal items {output r0, K chunk n} of W or its
        // transpose; off-diagonal ones {panel rows from r0, columns from n}
        const int rows1 = min(it.r0 + WT, s.stride[k]), cols1 = min(it.n + WT, n);
        const int o0 = diag || !BWD ? it.r0 : it.n, k0 = diag || !BWD ? it.n : it.r0;
        const int o1 = diag ? min(o0 + WT, n) : BWD ? cols1 : rows1, k1 = diag || !BWD ? min(k0 + WT, n) : rows1;
        const T *Mk = diag ? W + woff[k] : P + s.off[k];
        const int ldm = diag ? n : s.ld[k];
        const bool vec = !diag || n % EPV == 0;
        stage_factor<T, SM>(ms, Mk, ldm, k0, k1, o0, o1, vec);
        if (k0 + WK < k1) stage_factor<T, SM>(ms + SM::MS, Mk, ldm, k0 + WK, k1, o0, o1, vec);
        if (tid == 0) {
            if (diag) {
                if (!wflow_wait(BWD ? cnt_b + k : cnt_a + k, BWD ? nprev[k] : need[k], abort_word)) s_ok = 0;
            } else if (!BWD) {
                if (!wflow_wait(cnt_b + k, nprev[k], abort_word)) s_ok = 0;
            } else {
                for (int i = 0; i < it.nf && s_ok; i++) {
                    const int f = fw.flist[it.f0 + i];
                    if (!wflow_wait(cnt_a + f, need[f], abort_word)) s_ok = 0;
                }
            }
        }
        __syncthreads();
        if (!s_ok) {
            aborted = true;
            break;
        }
        const bool rows_in = BWD && !diag;    // inputs are panel rows (from the first below the block)
        const bool rows_out = !BWD && !diag;  // outputs are
        const T *in = diag == (BWD != 0) ? aux : x;
        T *out = diag == (BWD != 0) ? x : aux;
        auto xrow = [&](int kk) { return in + (size_t)(rows_in ? __ldg(prow + kk) : f0 + kk) * ldr; };
        auto used = [&](int kk) { return kk < k1 && (!rows_in || kk >= n); };
        constexpr int CPL = SM::RW / EPV;
#pragma unroll
        for (int u = 0; u < 2 * WK * CPL / SM::THREADS; u++) {
            const int idx = tid + SM::THREADS * u, l = idx / CPL, j = (idx % CPL) * EPV;
            const bool ok = used(k0 + l) && j < nrhs;
            cp_async_n<16>(xs + l * XP + j, ok ? xrow(k0 + l) + j : in, ok ? 16 : 0);
        }
        cp_commit_g();
        cp_wait_g<0>();
        __syncthreads();
        WideTile<T, MODE, NT> tile;
        tile.mul(ms, xs, o1 - o0, ntn);
        if (k0 + WK < k1) tile.mul(ms + SM::MS, xs + WK * XP, o1 - o0, ntn);
        __syncthreads();
        tile.out(os);
        __syncthreads();
        constexpr int CG = SM::RW < 32 ? SM::RW : 32, RG = 32 / CG;
#pragma unroll 4
        for (int i = warp * RG + lane / CG; i < o1 - o0; i += SM::THREADS / 32 * RG) {
            const int o = o0 + i;
            if (rows_out && o < n) continue;
            T *row = out + (size_t)(rows_out ? __ldg(prow + o) : f0 + o) * ldr;
#pragma unroll
            for (int j0 = 0; j0 < SM::RW; j0 += CG) {
                const int j = j0 + lane % CG;
                if (j < nrhs) atomicAdd(row + j, diag ? os[i * SM::OP + j] : -os[i * SM::OP + j]);
            }
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            if (diag) {
                atomicAdd(BWD ? cnt_a + k : cnt_b + k, 1);
            } else if (BWD) {
                atomicAdd(cnt_b + k, 1);
            } else {
                for (int i = 0; i < it.nf; i++) atomicAdd(cnt_a + fw.flist[it.f0 + i], 1);
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (aborted && tid == 0) {
        atomicOr(err, 16);
        atomicExch(abort_word, 1);
    }
}

// the rows of the listed cblks to zero
template <typename T>
__global__ void wide_zero_kernel(DevSym s, const int *__restrict__ cblks, T *x, int ldr, int nrhs) {
    const int k = cblks[blockIdx.x];
    T *xk = x + (size_t)s.fcol[k] * ldr;
    for (int64_t i = threadIdx.x; i < (int64_t)s.ncols[k] * nrhs; i += blockDim.x) xk[i / nrhs * ldr + i % nrhs] = (T)0;
}

template <typename T, int BWD, int NT>
int flow_ctas() {
    int dev = 0, sms = 0, occ = 0;
    constexpr int smem = WideFlowSmem<T, BWD, NT>::BYTES;
    if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) ||
        cudaFuncSetAttribute(wide_flow_kernel<T, BWD, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, wide_flow_kernel<T, BWD, NT>, WideFlowSmem<T, BWD, NT>::SM::THREADS,
                                                      smem))
        return 0;
    return occ * sms;
}
int g_flow_ctas[2][2][4];  // [FP64, FP32][direction][16, 32, 48, 64 columns]

template <typename T, int BWD, int NT>
void run_flow(const DevSym &s, const WideFlow &fw, const T *P, const T *W, const int64_t *woff, T *x, T *aux, int ldr,
              int nrhs, int *ticket, int *cnt_a, int *cnt_b, int *abort_word, int *err, cudaStream_t st) {
    const int n = BWD ? fw.nb : fw.nf;
    const int grid = std::min(n, g_flow_ctas[sizeof(T) == 4][BWD][NT / 2 - 1]);
    wide_flow_kernel<T, BWD, NT><<<grid, WideFlowSmem<T, BWD, NT>::SM::THREADS, WideFlowSmem<T, BWD, NT>::BYTES, st>>>(
        s, fw, n, BWD ? fw.b : fw.f, P, W, woff, x, aux, ldr, nrhs, ticket, cnt_a, cnt_b, abort_word, err);
}

// dst[i * ldr + j] = (D) src[i + j * lds] (to = 1), or back (to = 0), 32 x 32 tiles
template <typename S, typename D, int TO_ROWS>
__global__ void __launch_bounds__(256) wide_transpose_kernel(int n, int nrhs, const S *__restrict__ src, int64_t lds,
                                                             D *__restrict__ dst, int64_t ldd) {
    __shared__ D t[32][33];
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32, a = threadIdx.x & 31, b = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < 32; u += 8) {
        const int i = TO_ROWS ? i0 + a : i0 + b + u, j = TO_ROWS ? j0 + b + u : j0 + a;
        if (i < n && j < nrhs)
            t[b + u][a] = (D)(TO_ROWS ? src[i + (size_t)j * lds] : src[(size_t)i * lds + j]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 32; u += 8) {
        const int i = TO_ROWS ? i0 + b + u : i0 + a, j = TO_ROWS ? j0 + a : j0 + b + u;
        if (i < n && j < nrhs) {
            if (TO_ROWS) dst[(size_t)i * ldd + j] = t[a][b + u];
            else dst[i + (size_t)j * ldd] = t[a][b + u];
        }
    }
}

// x[i * ldr + j] /= D_i (LDL^T), the D of every cblk's diagonal
template <typename T>
__global__ void wide_scale_kernel(DevSym s, const int *__restrict__ cblks, const T *__restrict__ L, T *x, int ldr,
                                  int nrhs) {
    const int k = cblks[blockIdx.x];
    const int n = s.ncols[k];
    const T *D = L + s.off[k];
    for (int idx = threadIdx.x; idx < n * nrhs; idx += blockDim.x) {
        const int i = idx / nrhs, j = idx % nrhs;
        x[(size_t)(s.fcol[k] + i) * ldr + j] /= D[(size_t)i * (s.ld[k] + 1)];
    }
}

template <typename T, int MODE, int NT>
void run_mm(const DevSym &s, const WideTask *tasks, int ntasks, const T *M, const int64_t *woff, const T *in, T *out,
            int ldr, int nrhs, cudaStream_t st) {
    const dim3 grid(ntasks, (nrhs + NT * 8 - 1) / (NT * 8));
    wide_mm_kernel<T, MODE, NT><<<grid, WideSmem<T, MODE, NT>::THREADS, WideSmem<T, MODE, NT>::BYTES, st>>>(s, tasks, M, woff, in, out, ldr, nrhs);
}

template <typename T, int MODE>
void run_mode(const DevSym &s, const WideTask *tasks, int ntasks, const T *M, const int64_t *woff, const T *in, T *out,
              int ldr, int nrhs, cudaStream_t st) {
    if (nrhs <= 16) run_mm<T, MODE, 2>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
    else if (nrhs <= 32) run_mm<T, MODE, 4>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
    else if (nrhs <= 48) run_mm<T, MODE, 6>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
    else run_mm<T, MODE, 8>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
}

template <typename T, int MODE, int NT>
int conf() {
    return (int)cudaFuncSetAttribute(wide_mm_kernel<T, MODE, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     WideSmem<T, MODE, NT>::BYTES);
}
template <typename T, int NT>
int conf_modes() {
    return conf<T, W_OFF_FWD, NT>() | conf<T, W_OFF_BWD, NT>() | conf<T, W_DIAG_FWD, NT>() | conf<T, W_DIAG_BWD, NT>();
}

}  // namespace

int configure_wide_kernels() {
    int rc = conf_modes<double, 2>() | conf_modes<double, 4>() | conf_modes<double, 6>() | conf_modes<double, 8>() |
             conf_modes<float, 2>() | conf_modes<float, 4>() | conf_modes<float, 6>() | conf_modes<float, 8>();
    auto flow = [&](int f, auto nt, int i) {
        constexpr int NT = decltype(nt)::value;
        g_flow_ctas[f][0][i] = f ? flow_ctas<float, 0, NT>() : flow_ctas<double, 0, NT>();
        g_flow_ctas[f][1][i] = f ? flow_ctas<float, 1, NT>() : flow_ctas<double, 1, NT>();
        if (g_flow_ctas[f][0][i] <= 0 || g_flow_ctas[f][1][i] <= 0) rc = 1;
    };
    for (int f = 0; f < 2; f++) {
        flow(f, std::integral_constant<int, 2>{}, 0);
        flow(f, std::integral_constant<int, 4>{}, 1);
        flow(f, std::integral_constant<int, 6>{}, 2);
        flow(f, std::integral_constant<int, 8>{}, 3);
    }
    return rc ? -1 : 0;
}

template <typename T>
void launch_wide_flow(const DevSym &s, const WideFlow &fw, const T *P, const T *W, const int64_t *woff, T *x, T *aux,
                      int ldr, int nrhs, int backward, int *ticket, int *cnt_a, int *cnt_b, int *abort_word, int *err,
                      cudaStream_t st) {
    auto run = [&](auto nt) {
        constexpr int NT = decltype(nt)::value;
        if (backward)
            run_flow<T, 1, NT>(s, fw, P, W, woff, x, aux, ldr, nrhs, ticket, cnt_a, cnt_b, abort_word, err, st);
        else
            run_flow<T, 0, NT>(s, fw, P, W, woff, x, aux, ldr, nrhs, ticket, cnt_a, cnt_b, abort_word, err, st);
    };
    if (nrhs <= 16) run(std::integral_constant<int, 2>{});
    else if (nrhs <= 32) run(std::integral_constant<int, 4>{});
    else if (nrhs <= 48) run(std::integral_constant<int, 6>{});
    else run(std::integral_constant<int, 8>{});
}

template <typename T>
void launch_wide_zero(const DevSym &s, const int *cblks, int ncblk, T *x, int ldr, int nrhs, cudaStream_t st) {
    if (ncblk > 0) wide_zero_kernel<T><<<ncblk, 256, 0, st>>>(s, cblks, x, ldr, nrhs);
}

template <typename T>
void launch_wide_off(const DevSym &s, const WideTask *tasks, int ntasks, const T *P, const T *in, T *out, int ldr,
                     int nrhs, int backward, cudaStream_t st) {
    if (ntasks <= 0) return;
    if (backward) run_mode<T, W_OFF_BWD>(s, tasks, ntasks, P, nullptr, in, out, ldr, nrhs, st);
    else run_mode<T, W_OFF_FWD>(s, tasks, ntasks, P, nullptr, in, out, ldr, nrhs, st);
}

template <typename T>
void launch_wide_diag(const DevSym &s, const WideTask *tasks, int ntasks, const T *W, const int64_t *woff, const T *in,
                      T *out, int ldr, int nrhs, int backward, cudaStream_t st) {
    if (ntasks <= 0) return;
    if (backward) run_mode<T, W_DIAG_BWD>(s, tasks, ntasks, W, woff, in, out, ldr, nrhs, st);
    else run_mode<T, W_DIAG_FWD>(s, tasks, ntasks, W, woff, in, out, ldr, nrhs, st);
}

template <typename T>
void launch_wide_leaf(const DevSym &s, const int *cblks, int ncblk, const T *P, const T *W, const int64_t *woff, T *x,
                      T *aux, int ldr, int nrhs, int backward, cudaStream_t st) {
    if (ncblk <= 0) return;
    const dim3 grid((ncblk + WL_WARPS - 1) / WL_WARPS, (nrhs + 31) / 32);
    wide_leaf_kernel<T><<<grid, 32 * WL_WARPS, 0, st>>>(s, cblks, ncblk, P, W, woff, x, aux, ldr, nrhs, backward);
}

template <typename S, typename D>
void launch_wide_transpose(int n, int nrhs, const S *src, int64_t lds, D *dst, int64_t ldd, int to_rows,
                           cudaStream_t st) {
    const dim3 grid((n + 31) / 32, (nrhs + 31) / 32);
    if (to_rows) wide_transpose_kernel<S, D, 1><<<grid, 256, 0, st>>>(n, nrhs, src, lds, dst, ldd);
    else wide_transpose_kernel<S, D, 0><<<grid, 256, 0, st>>>(n, nrhs, src, lds, dst, ldd);
}

template <typename T>
void launch_wide_scale(const DevSym &s, const int *cblks, int ncblk, const T *L, T *x, int ldr, int nrhs,
                       cudaStream_t st) {
    if (ncblk > 0) wide_scale_kernel<T><<<ncblk, 128, 0, st>>>(s, cblks, L, x, ldr, nrhs);
}

#define WIDE_INST(T)                                                                                                 \
    template void launch_wide_off<T>(const DevSym &, const WideTask *, int, const T *, const T *, T *, int, int, int, \
                                     cudaStream_t);                                                                  \
    template void launch_wide_diag<T>(const DevSym &, const WideTask *, int, const T *, const int64_t *, const T *,  \
                                      T *, int, int, int, cudaStream_t);                                             \
    template void launch_wide_leaf<T>(const DevSym &, const int *, int, const T *, const T *, const int64_t *, T *,  \
                                      T *, int, int, int, cudaStream_t);                                             \
    template void launch_wide_transpose<double, T>(int, int, const double *, int64_t, T *, int64_t, int, cudaStream_t); \
    template void launch_wide_flow<T>(const DevSym &, const WideFlow &, const T *, const T *, const int64_t *, T *,  \
                                      T *, int, int, int, int *, int *, int *, int *, int *, cudaStream_t);          \
    template void launch_wide_zero<T>(const DevSym &, const int *, int, T *, int, int, cudaStream_t);                \
    template void launch_wide_scale<T>(const DevSym &, const int *, int, const T *, T *, int, int, cudaStream_t);
WIDE_INST(double)
WIDE_INST(float)
template void launch_wide_transpose<float, double>(int, int, const float *, int64_t, double *, int64_t, int,
                                                   cudaStream_t);
#undef WIDE_INST

}  // namespace b200
