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

#include "b200_internal.h"
#include "kernels.h"

namespace b200 {

namespace {

constexpr int WT = 64;  // outputs of a tile
constexpr int WK = 32;  // K values of a pipeline stage
constexpr int WSTAGES = 3;
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
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
    hi = __float_as_uint(x) & 0xFFFFE000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}

// acc += A B over one stage: A(o, kk) = ms[kk * PM + o] (ROW) or ms[o * PM + kk],
// B(kk, j) = xs[kk * XP + j]; NT groups of 8 columns, ntn of them used.  FP64: DMMA.
template <int PM, int XP, bool ROW, int NT>
__device__ __forceinline__ void stage_mma(double (&acc)[NT][4], double (&)[NT][4], const double *ms, const double *xs,
                                          int o0w, int ntn) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int kk = 0; kk < WK; kk += 16) {
        double a[8];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int kq = kk + 4 * j + tg;
            a[2 * j] = ROW ? ms[kq * PM + o0w + g] : ms[(o0w + g) * PM + kq];
            a[2 * j + 1] = ROW ? ms[kq * PM + o0w + g + 8] : ms[(o0w + g + 8) * PM + kq];
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            if (nt < ntn) {
                double b[4];
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = xs[(kk + 4 * j + tg) * XP + nt * 8 + g];
                dmma_k16(acc[nt], a, b);
            }
        }
    }
}

// FP32: 3xTF32 (x = hi + lo; hi*hi in acc, the two correction products in cor).
template <int PM, int XP, bool ROW, int NT>
__device__ __forceinline__ void stage_mma(float (&acc)[NT][4], float (&cor)[NT][4], const float *ms, const float *xs,
                                          int o0w, int ntn) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int kk = 0; kk < WK; kk += 8) {
        uint32_t ah[4], al[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int kq = kk + tg + 4 * (j >> 1), o = o0w + g + 8 * (j & 1);
            split_tf32(ROW ? ms[kq * PM + o] : ms[o * PM + kq], ah[j], al[j]);
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            if (nt < ntn) {
                uint32_t bh[2], bl[2];
                split_tf32(xs[(kk + tg) * XP + nt * 8 + g], bh[0], bl[0]);
                split_tf32(xs[(kk + tg + 4) * XP + nt * 8 + g], bh[1], bl[1]);
                mma_tf32_k8(acc[nt], ah, bh);
                mma_tf32_k8(cor[nt], ah, bl);
                mma_tf32_k8(cor[nt], al, bh);
            }
        }
    }
}

template <typename T, int MODE, int NT>
struct WideSmem {
    static constexpr bool ROW = MODE == W_OFF_FWD || MODE == W_DIAG_FWD;
    static constexpr int EPV = 16 / (int)sizeof(T);
    // pitches: conflict-free fragment reads, and room for the rows copied before the
    // tile's first one to reach a 16-byte boundary
    static constexpr int PM = ROW ? WT + 8 : WK + 4;
    static constexpr int XP = NT * 8 + (sizeof(T) == 8 ? 4 : 8);
    static constexpr int MS = ROW ? WK * PM : WT * PM;
    static constexpr int XS = WK * XP;
    static constexpr int STAGE = MS + XS;
    static constexpr int OP = NT * 8 + 1;  // pitch of the output staging
    static constexpr int ELEMS = WSTAGES * STAGE > WT * OP ? WSTAGES * STAGE : WT * OP;
    static constexpr int BYTES = ELEMS * (int)sizeof(T);
};

// One tile: 64 outputs of task {k, o0, k0, k1} x the right-hand sides
// [q0, q0 + 8 NT), q0 = 8 NT blockIdx.y:
//   OFF_FWD  x[row o] -= sum_{k0 <= c < k1} P[o, c] aux[c]     (o panel rows; atomic)
//   OFF_BWD  aux[o]   -= sum_{k0 <= r < k1} P[r, o] x[row r]   (o columns; atomic)
//   DIAG_FWD aux[o]    = sum_c W[o, c] x[c]      DIAG_BWD x[o] = sum_r W[r, o] aux[r]
// 4 warps of 16 outputs; 3-stage cp.async pipeline over chunks of 32 K values.
template <typename T, int MODE, int NT>
__global__ void __launch_bounds__(128) wide_mm_kernel(DevSym s, const WideTask *__restrict__ tasks,
                                                      const T *__restrict__ M, const int64_t *__restrict__ woff,
                                                      const T *in, T *out, int ldr, int nrhs) {
    using SM = WideSmem<T, MODE, NT>;
    constexpr bool ROW = SM::ROW, OFF = MODE == W_OFF_FWD || MODE == W_OFF_BWD;
    constexpr int PM = SM::PM, XP = SM::XP, EPV = SM::EPV;
    extern __shared__ __align__(16) unsigned char wd_smem[];
    T *sm = reinterpret_cast<T *>(wd_smem);
    const WideTask t = tasks[blockIdx.x];
    const int k = t.k, n = s.ncols[k], f0 = s.fcol[k];
    const int q0 = blockIdx.y * NT * 8, R = min(NT * 8, nrhs - q0), ntn = (R + 7) >> 3;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldm = OFF ? s.ld[k] : n;
    const int nout = min(WT, (MODE == W_OFF_FWD ? s.stride[k] : n) - t.o0);
    const T *Mk = M + (OFF ? s.off[k] : woff[k]);
    const int *prow = OFF ? s.prow + s.rbase[k] : nullptr;
    const bool vec = OFF || n % EPV == 0;  // 16-byte copies of the factor
    const bool vecx = ldr % EPV == 0;      // and of the vectors
    // the tile's first contiguous index (ROW: outputs, else the chunk's K) rounded down
    const int shift_o = ROW && vec ? t.o0 % EPV : 0;

    auto load = [&](int st, int kc) {
        T *ms = sm + st * SM::STAGE, *xs = ms + SM::MS;
        // factor chunk: lines (ROW: K values, else outputs) of contiguous entries
        const int line0 = ROW ? kc : t.o0, nline = ROW ? t.k1 : t.o0 + nout;
        const int e0 = ROW ? t.o0 : kc, e1 = ROW ? t.o0 + nout : t.k1;
        constexpr int LINES = ROW ? WK : WT, LEN = ROW ? WT : WK;
        if (vec) {
            constexpr int CPL = LEN / EPV + 1;
            const int a0 = e0 - e0 % EPV;
            for (int idx = tid; idx < LINES * CPL; idx += 128) {
                const int l = idx / CPL, i = idx % CPL, e = a0 + i * EPV;
                int bytes = 0;
                if (line0 + l < nline && e < e1) bytes = min(EPV, e1 - e) * (int)sizeof(T);
                cp_async_n<16>(ms + l * PM + i * EPV, bytes ? Mk + e + (size_t)(line0 + l) * ldm : Mk, bytes);
            }
        } else {
            for (int idx = tid; idx < LINES * LEN; idx += 128) {
                const int l = idx / LEN, i = idx % LEN;
                const bool ok = line0 + l < nline && e0 + i < e1;
                cp_async_n<sizeof(T)>(ms + l * PM + i, ok ? Mk + e0 + i + (size_t)(line0 + l) * ldm : Mk,
                                      ok ? (int)sizeof(T) : 0);
            }
        }
        // right-hand sides of the chunk's K values
        auto xrow = [&](int kk) { return in + (size_t)(MODE == W_OFF_BWD ? __ldg(prow + kk) : f0 + kk) * ldr + q0; };
        if (vecx) {
            constexpr int CPL = NT * 8 / EPV;
            for (int idx = tid; idx < WK * CPL; idx += 128) {
                const int l = idx / CPL, j = (idx % CPL) * EPV;
                const bool ok = kc + l < t.k1 && j < R;
                cp_async_n<16>(xs + l * XP + j, ok ? xrow(kc + l) + j : in, ok ? 16 : 0);
            }
        } else {
            for (int idx = tid; idx < WK * NT * 8; idx += 128) {
                const int l = idx / (NT * 8), j = idx % (NT * 8);
                const bool ok = kc + l < t.k1 && j < R;
                cp_async_n<sizeof(T)>(xs + l * XP + j, ok ? xrow(kc + l) + j : in, ok ? (int)sizeof(T) : 0);
            }
        }
    };

    T acc[NT][4], cor[NT][4];
#pragma unroll
    for (int a = 0; a < NT; a++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[a][e] = cor[a][e] = (T)0;
    const int o0w = warp * 16;
    const int nk = (t.k1 - t.k0 + WK - 1) / WK;
#pragma unroll
    for (int st = 0; st < WSTAGES - 1; st++) {
        if (st < nk) load(st, t.k0 + st * WK);
        cp_commit_g();
    }
    for (int i = 0; i < nk; i++) {
        cp_wait_g<WSTAGES - 2>();
        __syncthreads();
        if (i + WSTAGES - 1 < nk) load((i + WSTAGES - 1) % WSTAGES, t.k0 + (i + WSTAGES - 1) * WK);
        cp_commit_g();
        if (o0w < nout) {
            const T *ms = sm + (i % WSTAGES) * SM::STAGE;
            // the staged entries start shift after the 16-byte boundary before them
            const int shift = ROW ? shift_o : (vec ? (t.k0 + i * WK) % EPV : 0);
            stage_mma<PM, XP, ROW, NT>(acc, cor, ms + shift, ms + SM::MS, o0w, ntn);
        }
    }
    cp_wait_g<0>();
    __syncthreads();
    // outputs through shared memory, so that a warp adds (stores) whole rows
    T *os = sm + o0w * SM::OP;
    {
        const int g = lane >> 2, tg = lane & 3;
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                os[(g + (e >> 1) * 8) * SM::OP + nt * 8 + 2 * tg + (e & 1)] =
                    sizeof(T) == 4 ? acc[nt][e] + cor[nt][e] : acc[nt][e];
    }
    __syncwarp();
    constexpr int CG = NT * 8 < 32 ? NT * 8 : 32, RG = 32 / CG;  // columns of a row, rows at a time
    for (int i = lane / CG; i < 16 && o0w + i < nout; i += RG) {
        const int o = t.o0 + o0w + i;
        T *row = out + (size_t)(MODE == W_OFF_FWD ? __ldg(prow + o) : f0 + o) * ldr + q0;
        for (int j = lane % CG; j < R; j += CG) {
            const T v = os[i * SM::OP + j];
            if (OFF) atomicAdd(row + j, -v);
            else row[j] = v;
        }
    }
}

// Cblks of at most 32 columns: both products of one sweep by one warp for 32
// right-hand sides, lane = right-hand side.  The factor's entries are staged 32 panel
// rows at a time and read as broadcasts.
template <typename T>
struct WideLeaf {
    T ys[32][32];       // the cblk's rows of x / aux
    T ps[32][32];       // ps[c][r]: W_k, then 32 panel rows
    T xr[32][32];       // backward: x of the 32 panel rows
};

template <typename T>
__global__ void __launch_bounds__(64) wide_leaf_kernel(DevSym s, const int *__restrict__ cblks, int ncblk,
                                                       const T *__restrict__ P, const T *__restrict__ W,
                                                       const int64_t *__restrict__ woff, T *x, T *aux, int ldr,
                                                       int nrhs, int backward) {
    extern __shared__ __align__(16) unsigned char wl_smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WideLeaf<T> &S = reinterpret_cast<WideLeaf<T> *>(wl_smem)[w];
    const int ci = blockIdx.x * 2 + w;
    if (ci >= ncblk) return;
    const int k = cblks[ci];
    const int n = s.ncols[k], ld = s.ld[k], stride = s.stride[k], f0 = s.fcol[k];
    const T *Pk = P + s.off[k], *Wk = W + woff[k];
    const int *prow = s.prow + s.rbase[k];
    const int q = blockIdx.y * 32 + lane;
    const bool in = q < nrhs;
    for (int c = 0; c < n; c++) S.ps[c][lane] = (lane < n && lane >= c) ? Wk[lane + (size_t)c * n] : (T)0;
    const T *src = backward ? aux : x;
    for (int c = 0; c < n; c++) S.ys[c][lane] = in ? src[(size_t)(f0 + c) * ldr + q] : (T)0;
    __syncwarp();
    if (!backward) {
        // aux_k = W_k x_k, from the last rows up (rows above still read x)
        for (int r0 = (n - 1) & ~3; r0 >= 0; r0 -= 4) {
            T a[4] = {};
            const int cend = min(n, r0 + 4);
            for (int c = 0; c < cend; c++) {
                const T v = S.ys[c][lane];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] += S.ps[c][r0 + i] * v;
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (r0 + i < n) {
                    S.ys[r0 + i][lane] = a[i];
                    if (in) aux[(size_t)(f0 + r0 + i) * ldr + q] = a[i];
                }
        }
        for (int b = n; b < stride; b += 32) {
            __syncwarp();
            for (int c = 0; c < n; c++) S.ps[c][lane] = b + lane < stride ? Pk[b + lane + (size_t)c * ld] : (T)0;
            const int myg = b + lane < stride ? prow[b + lane] : 0;
            __syncwarp();
            for (int r0 = 0; r0 < 32 && b + r0 < stride; r0 += 8) {
                T a[8] = {};
                for (int c = 0; c < n; c++) {
                    const T v = S.ys[c][lane];
#pragma unroll
                    for (int i = 0; i < 8; i++) a[i] += S.ps[c][r0 + i] * v;
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int g = __shfl_sync(0xffffffffu, myg, r0 + i);
                    if (in && b + r0 + i < stride) atomicAdd(x + (size_t)g * ldr + q, -a[i]);
                }
            }
        }
    } else {
        // t = aux_k - P_k^T x[rows below], 8 columns at a time; x_k = W_k^T t
        for (int b = n; b < stride; b += 32) {
            const int nr = min(32, stride - b);
            const int myg = lane < nr ? prow[b + lane] : 0;
            for (int r = 0; r < nr; r++) {
                const int g = __shfl_sync(0xffffffffu, myg, r);
                S.xr[r][lane] = in ? x[(size_t)g * ldr + q] : (T)0;
            }
            for (int c0 = 0; c0 < n; c0 += 8) {
                T a[8];
#pragma unroll
                for (int i = 0; i < 8; i++) a[i] = 0;
                // the panel's entries of the 8 columns, one per lane and column, by shuffle
                T p[8];
#pragma unroll
                for (int i = 0; i < 8; i++)
                    p[i] = (c0 + i < n && lane < nr) ? Pk[b + lane + (size_t)(c0 + i) * ld] : (T)0;
                for (int r = 0; r < nr; r++) {
                    const T v = S.xr[r][lane];
#pragma unroll
                    for (int i = 0; i < 8; i++) a[i] += __shfl_sync(0xffffffffu, p[i], r) * v;
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (c0 + i < n) S.ys[c0 + i][lane] -= a[i];
            }
        }
        for (int c = 0; c < n; c++) {
            T a = 0;
            for (int r = c; r < n; r++) a += S.ps[c][r] * S.ys[r][lane];
            if (in) x[(size_t)(f0 + c) * ldr + q] = a;
        }
    }
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
    wide_mm_kernel<T, MODE, NT><<<grid, 128, WideSmem<T, MODE, NT>::BYTES, st>>>(s, tasks, M, woff, in, out, ldr, nrhs);
}

template <typename T, int MODE>
void run_mode(const DevSym &s, const WideTask *tasks, int ntasks, const T *M, const int64_t *woff, const T *in, T *out,
              int ldr, int nrhs, cudaStream_t st) {
    if (nrhs <= 16) run_mm<T, MODE, 2>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
    else if (nrhs <= 32) run_mm<T, MODE, 4>(s, tasks, ntasks, M, woff, in, out, ldr, nrhs, st);
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
    int rc = conf_modes<double, 2>() | conf_modes<double, 4>() | conf_modes<double, 8>() | conf_modes<float, 2>() |
             conf_modes<float, 4>() | conf_modes<float, 8>();
    rc |= (int)cudaFuncSetAttribute(wide_leaf_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    2 * (int)sizeof(WideLeaf<double>));
    rc |= (int)cudaFuncSetAttribute(wide_leaf_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    2 * (int)sizeof(WideLeaf<float>));
    return rc ? -1 : 0;
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
    const dim3 grid((ncblk + 1) / 2, (nrhs + 31) / 32);
    wide_leaf_kernel<T><<<grid, 64, 2 * sizeof(WideLeaf<T>), st>>>(s, cblks, ncblk, P, W, woff, x, aux, ldr, nrhs,
                                                                   backward);
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
    template void launch_wide_scale<T>(const DevSym &, const int *, int, const T *, T *, int, int, cudaStream_t);
WIDE_INST(double)
WIDE_INST(float)
template void launch_wide_transpose<float, double>(int, int, const float *, int64_t, double *, int64_t, int,
                                                   cudaStream_t);
#undef WIDE_INST

}  // namespace b200
