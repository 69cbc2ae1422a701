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
// What bounds it is the store of the matrix (n = 61440: 15.1 GB) and the FP64 and
// conversion pipes.  Separate passes for the elements and for d generated
// everything twice.  A thread's ROWS elements of a column are contiguous, but a
// warp's are 32 columns apart, so a warp exchanges its 32 columns x ROWS rows
// through shared memory and stores whole sectors, several columns per
// instruction (16-byte stores to 32 different columns each: n = 61440 7.2 ms).
// ROWS = 8: whole 32-byte sectors, a CTA per SM from n ~ 1200 on, and 64
// registers, so that two CTAs share an SM (16 rows spill there).
#include <algorithm>

#include "mxp_internal.cuh"

namespace mxp {

namespace {

constexpr int kGenThreads = 512;   // MATGEM_THREADS of matgen.hpp:7, pinned by the reduction order
constexpr int kGenRows = 8;
constexpr int kRedRows = 4;        // rows reduced together in shared memory

constexpr int kJumps = 31;         // powers J_n^(2^i) of the column jump

template <typename T>
struct GenArgs {
    int n, diag_rule;
    uint64_t s00;
    Aff jn;            // jump of one column
    T *A;              // may be null, like d, rowsum and rhs
    int64_t lda;
    double *d, *rowsum, *rhs;
};

// Dynamic shared memory: a tile per warp, 32 columns of ROWS values (pitch ROWS +
// 16 bytes: 16-byte accesses without conflicts), and the reduction after them.
template <typename T, int ROWS>
constexpr size_t gen_smem() {
    const size_t tiles = (size_t)kGenThreads * (ROWS * sizeof(T) + 16), red = sizeof(double) * kRedRows * kGenThreads;
    return tiles > red ? tiles : red;
}

template <typename T, int ROWS>
__device__ __forceinline__ void gen_rows(const GenArgs<T> &g, int64_t row0) {
    static_assert(kGenThreads == 512, "jp[9] is the step of a thread");
    static_assert(ROWS % kRedRows == 0, "whole reduction groups");
    extern __shared__ __align__(16) unsigned char gen_mem[];
    double(*sh)[kGenThreads] = reinterpret_cast<double(*)[kGenThreads]>(gen_mem);
    constexpr int V = 16 / sizeof(T), P = ROWS + V;  // values per 16 bytes, tile pitch
    const int t = threadIdx.x, lane = t & 31, n = g.n;
    T *tile = reinterpret_cast<T *>(gen_mem) + (size_t)(t - lane) * P;
    const int rows = (int)imin64(ROWS, n - row0);
    const Aff inc1 = lcg_inc1();
    double acc[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) acc[q] = 0.0;
    const bool elements = g.A || g.d || g.rowsum;
    // element (row0, c): J_n^c o INC1^row0 of the seed's state, from powers of the
    // two jumps made once per CTA (all of them commute): a jump-ahead per thread by
    // squaring took as long as a small system's elements
    __shared__ Aff jp[kJumps];
    __shared__ uint64_t base_sh;
    if (t == 0) {
        Aff f = g.jn;
        for (int i = 0; i < kJumps && ((n >> i) || i < 10); ++i) {
            jp[i] = f;
            f = aff_mul(f, f);
        }
    } else if (t == 32) {
        base_sh = aff_apply(aff_pow(inc1, (uint64_t)row0), g.s00);
    }
    __syncthreads();
    auto element = [&](uint64_t s, unsigned c) {  // state of (row, c) from that of (row, 0)
        for (int i = 0; c; ++i, c >>= 1)
            if (c & 1u) s = aff_apply(jp[i], s);
        return s;
    };
    if (elements && t - lane < n) {
        const Aff j512 = jp[9];
        uint64_t s0 = element(base_sh, (unsigned)t);
        const bool vec = rows == ROWS && ((reinterpret_cast<uintptr_t>(g.A) | (uintptr_t)(g.lda * sizeof(T))) & 15) == 0;
        for (int64_t jb = t - lane; jb < n; jb += kGenThreads) {  // the warp's 32 columns
            const int64_t j = jb + lane;
            const int dq = (int)(j - row0);  // row of the diagonal element, when in 0 .. ROWS - 1
            uint64_t s = s0;
#pragma unroll
            for (int q0 = 0; q0 < ROWS; q0 += V) {
                T v[V];
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const double x = lcg_to_double(s);
                    v[e] = static_cast<T>(x);  // float: round to nearest (RandStat::operator float)
                    // (columns past n add nothing)
                    acc[q0 + e] += q0 + e == dq || j >= n ? 0.0 : fabs(x);
                    s = aff_apply(inc1, s);
                }
                if (g.A) {
                    if constexpr (sizeof(T) == 4)
                        *reinterpret_cast<float4 *>(tile + lane * P + q0) = make_float4(v[0], v[1], v[2], v[3]);
                    else
                        *reinterpret_cast<double2 *>(tile + lane * P + q0) = make_double2(v[0], v[1]);
                }
            }
            s0 = aff_apply(j512, s0);
            if (!g.A) continue;
            __syncwarp();
            constexpr int L = ROWS / V;  // lanes per column
            if (vec) {
                const int r = (lane % L) * V;
#pragma unroll
                for (int c = lane / L; c < 32; c += 32 / L)
                    if (jb + c < n)
                        *reinterpret_cast<float4 *>(g.A + (jb + c) * g.lda + row0 + r) =
                            *reinterpret_cast<const float4 *>(tile + c * P + r);
            } else {
                const int r = lane % ROWS;
                for (int c = lane / ROWS; c < 32; c += 32 / ROWS)
                    if (jb + c < n && r < rows) g.A[(jb + c) * g.lda + row0 + r] = tile[c * P + r];
            }
            __syncwarp();
        }
    }
    if (g.rhs && t < rows) {
        uint64_t s = element(base_sh, (unsigned)n);
        for (int q = 0; q < t; ++q) s = aff_apply(inc1, s);
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
__global__ void __launch_bounds__(kGenThreads, ROWS > kGenRows ? 1 : 2) gen_kernel(GenArgs<T> g) {
    gen_rows<T, ROWS>(g, (int64_t)blockIdx.x * ROWS);
}

// Many systems in one launch: blockIdx.y walks the systems, blockIdx.x a system's
// row bands (those past its order leave).
template <int ROWS>
__global__ void __launch_bounds__(kGenThreads, 2)
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
        g.A = A + S.a_off;
        g.lda = S.n;
        g.d = d + S.v_off;
        g.rowsum = nullptr;
        g.rhs = rhs + S.v_off;
        gen_rows<float, ROWS>(g, row0);
        __syncthreads();
    }
}

// The right-hand side by itself (stream column n), a thread per row: in the kernel
// above its eight rows per CTA cost a CTA's jump powers each (n = 20000: 17 us, here
// 3).
__global__ void __launch_bounds__(256) rhs_kernel(int n, uint64_t s00, double *rhs) {
    const int64_t row = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (row < n) rhs[row] = lcg_to_double(aff_apply(aff_pow(lcg_inc1(), (uint64_t)row + (uint64_t)n * (uint64_t)n), s00));
}

template <typename T, int ROWS>
mxp_status launch_gen_rows(const GenArgs<T> &g, cudaStream_t st) {
    constexpr size_t smem = gen_smem<T, ROWS>();
    if (smem > 48 * 1024 - 1024)
        MXP_CUDA(cudaFuncSetAttribute(gen_kernel<T, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    gen_kernel<T, ROWS><<<(unsigned)cdiv(g.n, ROWS), kGenThreads, smem, st>>>(g);
    MXP_LAUNCHED();
    return MXP_OK;
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
    g.A = A;
    g.lda = lda;
    g.d = d;
    g.rowsum = rowsum;
    g.rhs = rhs;
    if (!A && !d && !rowsum) {
        rhs_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, g.s00, rhs);
        MXP_LAUNCHED();
        return MXP_OK;
    }
    // FP64 columns that do not all start on a sector (an odd pitch): a CTA's 64 bytes
    // of a column then touch three sectors, two of them shared with the neighbours'.
    // Twice the rows (one CTA per SM) make that five for 128: n = 8191 178 us (8
    // rows 296), n = 8192 with a pitch of 8193 168 (271).
    if (sizeof(T) == 8 && A && ((reinterpret_cast<uintptr_t>(A) | (uintptr_t)(lda * sizeof(T))) & 31))
        return launch_gen_rows<T, 2 * kGenRows>(g, st);
    return launch_gen_rows<T, kGenRows>(g, st);
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
    const dim3 grid((unsigned)cdiv(nmax, kGenRows), (unsigned)std::min(count, 65535));
    constexpr size_t smem = gen_smem<float, kGenRows>();
    gen_batch_kernel<kGenRows><<<grid, kGenThreads, smem, st>>>(sys, count, A, d, rhs);
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
