// LCG matrix / RHS generation, bit-exact with the reference generator.
//
// Reference: panel_matgen_dev -> fill_panel_dev / fill_panel_diag_dev
// (matgen.hpp:8-117) and panel_colvgen (matgen.hpp:419-436).
//
// One kernel, each element made once.  d_i = sum_{j != i} |a_ij| in FP64 has to
// follow the reduction order of fill_panel_diag_dev (512 strided partials per
// row, tree 512 -> 4, then ((s0+s1)+s2)+s3) to be bit-identical to the
// reference's GPU path, so thread t of a 512-thread CTA makes the columns t, t +
// 512, ... of ROWS consecutive rows: it stores the elements (ROWS * 4
// contiguous bytes per column) and keeps the rows' t-th partials, and the CTA
// reduces them, writes A(i,i) = float(d_i) over the generator's value, and
// fills its rows of the right-hand side (stream column n).
// What bounds it is the store of the matrix (n = 61440: 15.1 GB) and, when
// only d is asked for, the FP64 and conversion pipes.  Separate passes for
// the elements and for d generated everything twice (n = 61440: 7.1 ms).
// ROWS = 16 amortises the jump-ahead of a thread's first state and writes 64
// bytes per column; up to kSmallN, where that would leave SMs without a CTA,
// ROWS = 4.
#include <algorithm>

#include "mxp_internal.cuh"

namespace mxp {

namespace {

constexpr int kGenThreads = 512;   // MATGEM_THREADS of matgen.hpp:7, pinned by the reduction order
constexpr int kSmallN = 148 * 16 * 2;
constexpr int kRedRows = 4;        // rows reduced together in shared memory

template <typename T>
struct GenArgs {
    int n, diag_rule;
    uint64_t s00;
    Aff jn, j512;      // jumps of one column and of 512 columns
    T *A;              // may be null, like d, rowsum and rhs
    int64_t lda;
    double *d, *rowsum, *rhs;
};

template <typename T, int ROWS>
__device__ __forceinline__ void gen_rows(const GenArgs<T> &g, int64_t row0) {
    static_assert(ROWS % kRedRows == 0, "whole reduction groups");
    __shared__ double sh[kRedRows][kGenThreads];
    const int t = threadIdx.x, n = g.n;
    const int rows = (int)imin64(ROWS, n - row0);
    const Aff inc1 = lcg_inc1();
    double acc[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) acc[q] = 0.0;
    const bool elements = g.A || g.d || g.rowsum;
    if (t < n && elements) {
        // element (row0, t): INC1^(row0 + n*t) = J_n^t o INC1^row0
        uint64_t s[ROWS];
        s[0] = aff_apply(aff_pow(g.jn, (uint64_t)t), aff_apply(aff_pow(inc1, (uint64_t)row0), g.s00));
#pragma unroll
        for (int q = 1; q < ROWS; ++q) s[q] = aff_apply(inc1, s[q - 1]);
        constexpr int V = 16 / sizeof(T);
        const bool vec = rows == ROWS && ((reinterpret_cast<uintptr_t>(g.A) | (uintptr_t)(g.lda * sizeof(T))) & 15) == 0;
        for (int64_t j = t; j < n; j += kGenThreads) {
            const int dq = (int)(j - row0);  // row of the diagonal element, when in 0 .. ROWS - 1
            T v[ROWS];
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const double x = lcg_to_double(s[q]);
                v[q] = static_cast<T>(x);  // float: round to nearest (RandStat::operator float)
                acc[q] += q == dq ? 0.0 : fabs(x);
                s[q] = aff_apply(g.j512, s[q]);
            }
            if (!g.A) continue;
            T *col = g.A + j * g.lda + row0;
            if (vec) {
#pragma unroll
                for (int q = 0; q < ROWS; q += V) {
                    if constexpr (sizeof(T) == 4)
                        *reinterpret_cast<float4 *>(col + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
                    else
                        *reinterpret_cast<double2 *>(col + q) = make_double2(v[q], v[q + 1]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < ROWS; ++q)
                    if (q < rows) col[q] = v[q];
            }
        }
    }
    if (g.rhs && t < rows) {
        const uint64_t s = aff_apply(aff_pow(inc1, (uint64_t)(row0 + t) + (uint64_t)n * (uint64_t)n), g.s00);
        g.rhs[row0 + t] = lcg_to_double(s);
    }
    if (!elements) return;
#pragma unroll
    for (int q0 = 0; q0 < ROWS; q0 += kRedRows) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kRedRows; ++q) sh[q][t] = acc[q0 + q];
        __syncthreads();
#pragma unroll
        for (int w = 256; w >= 4; w >>= 1) {
            for (int e = t; e < kRedRows * w; e += kGenThreads) sh[e / w][e % w] += sh[e / w][e % w + w];
            __syncthreads();
        }
        if (t < kRedRows && q0 + t < rows) {
            const int64_t row = row0 + q0 + t;
            const double s = ((sh[t][0] + sh[t][1]) + sh[t][2]) + sh[t][3];
            const double dv = g.diag_rule == MXP_DIAG_055_PLUS1 ? __dadd_rn(__dmul_rn(0.55, s), 1.0) : s;
            if (g.rowsum) g.rowsum[row] = s;
            if (g.d) g.d[row] = dv;
            if (g.A) g.A[row * g.lda + row] = static_cast<T>(dv);  // after the barriers: over the generator's value
        }
    }
}

template <typename T, int ROWS>
__global__ void __launch_bounds__(kGenThreads) gen_kernel(GenArgs<T> g) {
    gen_rows<T, ROWS>(g, (int64_t)blockIdx.x * ROWS);
}

// Many systems in one launch: blockIdx.y walks the systems, blockIdx.x a system's
// row bands (those past its order leave).
template <int ROWS>
__global__ void __launch_bounds__(kGenThreads)
gen_batch_kernel(const GenSys *sys, int count, float *A, double *d, double *rhs) {
    for (int i = blockIdx.y; i < count; i += gridDim.y) {
        const GenSys S = sys[i];
        const int64_t row0 = (int64_t)blockIdx.x * ROWS;
        if (row0 >= S.n) continue;
        GenArgs<float> g;
        g.n = S.n;
        g.diag_rule = MXP_DIAG_ROWSUM;
        g.s00 = lcg_stat00(S.seed);
        g.jn = aff_pow(lcg_inc1(), (uint64_t)S.n);
        g.j512 = aff_pow(g.jn, kGenThreads);
        g.A = A + S.a_off;
        g.lda = S.n;
        g.d = d + S.v_off;
        g.rowsum = nullptr;
        g.rhs = rhs + S.v_off;
        gen_rows<float, ROWS>(g, row0);
        __syncthreads();
    }
}

template <typename T>
mxp_status launch_gen(int n, uint64_t seed, int diag_rule, T *A, int64_t lda, double *d, double *rowsum,
                      double *rhs, cudaStream_t st) {
    if (!A && !d && !rowsum && !rhs) return MXP_OK;
    GenArgs<T> g;
    g.n = n;
    g.diag_rule = diag_rule;
    g.s00 = lcg_stat00(seed);
    g.jn = aff_pow(lcg_inc1(), (uint64_t)n);
    g.j512 = aff_pow(g.jn, kGenThreads);
    g.A = A;
    g.lda = lda;
    g.d = d;
    g.rowsum = rowsum;
    g.rhs = rhs;
    if (n <= kSmallN) gen_kernel<T, 4><<<(unsigned)cdiv(n, 4), kGenThreads, 0, st>>>(g);
    else gen_kernel<T, 16><<<(unsigned)cdiv(n, 16), kGenThreads, 0, st>>>(g);
    MXP_LAUNCHED();
    return MXP_OK;
}

}  // namespace

mxp_status launch_matgen(int n, uint64_t seed, int diag_rule, float *A, int64_t lda, double *d,
                         double *rowsum, double *rhs, cudaStream_t st) {
    if (n <= 0) return fail(MXP_INVALID_ARG, "mxp_matgen: n must be positive");
    if (A && lda < n) return fail(MXP_INVALID_ARG, "mxp_matgen: lda < n");
    if (diag_rule != MXP_DIAG_ROWSUM && diag_rule != MXP_DIAG_055_PLUS1)
        return fail(MXP_INVALID_ARG, "mxp_matgen: unknown diag_rule");
    return launch_gen<float>(n, seed, diag_rule, A, lda, d, rowsum, rhs, st);
}

mxp_status launch_matgen_batch(int count, const GenSys *sys, int nmax, float *A, double *d, double *rhs,
                               cudaStream_t st) {
    if (count <= 0) return MXP_OK;
    const dim3 grid((unsigned)cdiv(nmax, 16), (unsigned)std::min(count, 65535));
    gen_batch_kernel<16><<<grid, kGenThreads, 0, st>>>(sys, count, A, d, rhs);
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_matgen_f64(int n, uint64_t seed, int diag_rule, double *A, int64_t lda,
                             cudaStream_t st) {
    if (n <= 0 || !A) return fail(MXP_INVALID_ARG, "mxp_matgen_f64: bad arguments");
    if (lda < n) return fail(MXP_INVALID_ARG, "mxp_matgen_f64: lda < n");
    if (diag_rule != MXP_DIAG_ROWSUM && diag_rule != MXP_DIAG_055_PLUS1)
        return fail(MXP_INVALID_ARG, "mxp_matgen_f64: unknown diag_rule");
    return launch_gen<double>(n, seed, diag_rule, A, lda, nullptr, nullptr, nullptr, st);
}

}  // namespace mxp
