// The plain FP32 panel solves of the granular interface and of the LU with the
// tensor-core TRSM switched off: B <- B U^{-1} (GPUBLAS_STRSM R,U,N,NonUnit,
// panel_trf.hpp:188-207) and B <- L^{-1} B (L,L,N,Unit, panel_trf.hpp:225-246).
//
// The rows of B (columns, for L) are independent, so a CTA keeps a slice of
// them in shared memory through the whole triangle (up to kPanN wide; wider
// ones go panel by panel with an SGEMM between): per 64 columns a blocked
// substitution (dense_tile.cuh), then the slice's remaining columns minus
// their product with what was solved, the triangle's tiles streaming through
// L2 behind it, two buffers deep.  B is read and written once and the launch
// count does not grow with the triangle; a substitution launch and a rank-64
// SGEMM launch per 64 columns passed over B again each time (5003 x 500, both
// sides: 585 us).  What bounds it is shared-memory operand bandwidth (4 x 8
// outputs per thread: ~2/3 of the FMA rate).  The slice is as wide as
// spreads the rows over all SMs in whole waves, at most 64.
// Each 64-column block's products are summed by themselves and subtracted once.
#include <algorithm>

#include "dense_tile.cuh"
#include "mxp_internal.cuh"

namespace mxp {

namespace {

using namespace dt;

constexpr int kPanN = 512;   // widest triangle of one launch
constexpr int kSlice = 64;   // most rows (columns) of B per CTA
constexpr int kChunk = 96;   // columns (rows) of the triangle per streamed tile

__device__ __forceinline__ void cp_async4(void *dst, const void *src, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}

// dst[c * pitch + r] = src(r, c) for r < nr4 and c < nc4, zero past nr and nc; nr4 a multiple of 4.
__device__ __forceinline__ void request_rect(float *dst, int pitch, const float *src, int64_t ld, int nr, int nc,
                                             int nr4, int nc4) {
    if (aligned16(src) && (ld & 3) == 0) {
        const int g = nr4 >> 2;
        for (int idx = threadIdx.x; idx < g * nc4; idx += kCT) {
            const int c = idx / g, r = (idx % g) * 4;
            const int by = c < nc ? grp_bytes(r, nr) : 0;
            cp_async16(dst + c * pitch + r, by ? src + (int64_t)c * ld + r : src, by);
        }
    } else {
        for (int idx = threadIdx.x; idx < nr4 * nc4; idx += kCT) {
            const int c = idx / nr4, r = idx % nr4;
            const bool in = c < nc && r < nr;
            cp_async4(dst + c * pitch + r, in ? src + (int64_t)c * ld + r : src, in ? 4 : 0);
        }
    }
}

__device__ __forceinline__ void store_rect(const float *x, int pitch, float *dst, int64_t ld, int nr, int nc) {
    if (aligned16(dst) && (ld & 3) == 0 && (nr & 3) == 0) {
        const int g = nr >> 2;
        for (int idx = threadIdx.x; idx < g * nc; idx += kCT) {
            const int c = idx / g, r = (idx % g) * 4;
            *reinterpret_cast<float4 *>(dst + (int64_t)c * ld + r) = *reinterpret_cast<const float4 *>(x + c * pitch + r);
        }
    } else {
        for (int idx = threadIdx.x; idx < nr * nc; idx += kCT) {
            const int c = idx / nr, r = idx % nr;
            dst[(int64_t)c * ld + r] = x[c * pitch + r];
        }
    }
}

// The diagonal block of the triangle at 64 j (identity past its order nb).
__device__ __forceinline__ void fix_diag(Block64 T, int nb) {
    if (threadIdx.x >= nb && threadIdx.x < kNB) T[threadIdx.x][threadIdx.x] = 1.0f;
}

// C[c][r] -= sum_k A[k][r] B[c][k], k < 64: RT x CT outputs per thread, rows rg * RT ..
// (of nr) and columns cg * CT .. (of nc); A, B and C with their pitches.
template <int RT, int CT>
__device__ __forceinline__ void rank64(const float *A, int pa, const float *B, int pb, float *C, int pc, int nr,
                                       int nc) {
    const int tr = nr / RT, tc = nc / CT;
    for (int id = threadIdx.x; id < tr * tc; id += kCT) {
        const int r = (id % tr) * RT, c = (id / tr) * CT;
        float x[CT][RT];  // the sum by itself, subtracted once: C is larger than its terms
#pragma unroll
        for (int j = 0; j < CT; ++j)
#pragma unroll
            for (int i = 0; i < RT; ++i) x[j][i] = 0.0f;
#pragma unroll 2
        for (int k4 = 0; k4 < kNB / 4; ++k4) {
            float4 bq[CT];
#pragma unroll
            for (int j = 0; j < CT; ++j) bq[j] = *reinterpret_cast<const float4 *>(B + (c + j) * pb + 4 * k4);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                float av[RT];
#pragma unroll
                for (int i = 0; i < RT; i += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(A + (4 * k4 + s) * pa + r + i);
                    av[i] = a.x;
                    av[i + 1] = a.y;
                    av[i + 2] = a.z;
                    av[i + 3] = a.w;
                }
#pragma unroll
                for (int j = 0; j < CT; ++j) {
                    const float bv = s == 0 ? bq[j].x : s == 1 ? bq[j].y : s == 2 ? bq[j].z : bq[j].w;
#pragma unroll
                    for (int i = 0; i < RT; ++i) x[j][i] = fmaf(bv, av[i], x[j][i]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < CT; ++j)
#pragma unroll
            for (int i = 0; i < RT; i += 4) {
                float4 *p = reinterpret_cast<float4 *>(C + (c + j) * pc + r + i);
                const float4 v = *p;
                *p = make_float4(v.x - x[j][i], v.y - x[j][i + 1], v.z - x[j][i + 2], v.w - x[j][i + 3]);
            }
    }
}

struct __align__(16) SmemRight {
    float t[2][kNB][kNB + 4];          // diagonal blocks, t[.][col][row]
    float u[2][kChunk][kNB + 4];       // tiles right of them, u[.][col][row]
    float x[kPanN][kSlice + 4];        // the slice, x[col][row]
    float dinv[kNB];
};

// Rows [slice * blockIdx.x, ...) of B (m x n): B <- B U^{-1}, n <= kPanN.
__global__ void __launch_bounds__(kCT, 1)
panel_right_kernel(int m, int n, int slice, const float *__restrict__ U, int64_t ldu, float *B, int64_t ldb) {
    extern __shared__ __align__(16) unsigned char panel_smem[];
    SmemRight &s = *reinterpret_cast<SmemRight *>(panel_smem);
    const int64_t o = (int64_t)blockIdx.x * slice;
    const int w = (int)imin64(slice, m - o), nblk = (n + kNB - 1) / kNB;
    float *Bo = B + o;
    auto diag = [&](int j) {
        const int nb = min(kNB, n - j * kNB);
        request_rect(&s.t[j & 1][0][0], kNB + 4, U + (int64_t)j * kNB * (ldu + 1), ldu, nb, nb, kNB, kNB);
    };
    auto tile = [&](int j, int c0, int buf) {
        request_rect(&s.u[buf][0][0], kNB + 4, U + (int64_t)j * kNB + (int64_t)c0 * ldu, ldu, kNB, n - c0, kNB, kChunk);
    };
    diag(0);
    request_rect(&s.x[0][0], kSlice + 4, Bo, ldb, w, n, slice, nblk * kNB);
    cp_async_commit();
    for (int j = 0; j < nblk; ++j) {
        const int nb = min(kNB, n - j * kNB), c1 = (j + 1) * kNB;
        cp_async_wait<0>();
        __syncthreads();
        fix_diag(s.t[j & 1], nb);
        if (c1 < n) {  // the next diagonal block and the first tile, under the substitution
            diag(j + 1);
            tile(j, c1, 0);
        }
        cp_async_commit();
        __syncthreads();
        if (threadIdx.x < kNB) s.dinv[threadIdx.x] = 1.0f / s.t[j & 1][threadIdx.x][threadIdx.x];
        __syncthreads();
        block_solve_upper(s.t[j & 1], s.dinv, &s.x[j * kNB], slice);
        for (int c0 = c1, buf = 0; c0 < n; c0 += kChunk, buf ^= 1) {
            if (c0 + kChunk < n) tile(j, c0 + kChunk, buf ^ 1);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            // whole blocks of x: its columns past n are zero and stay so
            rank64<4, 8>(&s.x[j * kNB][0], kSlice + 4, &s.u[buf][0][0], kNB + 4, &s.x[c0][0], kSlice + 4, slice,
                         min(kChunk, nblk * kNB - c0));
            __syncthreads();
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    store_rect(&s.x[0][0], kSlice + 4, Bo, ldb, w, n);
}

struct __align__(16) SmemLeft {
    float t[2][kNB][kNB + 4];
    float l[2][kNB][kChunk + 4];       // tiles below the diagonal blocks, l[.][col][row]
    float x[kSlice][kPanN + 4];        // the slice, x[col][row]
};

// Columns [slice * blockIdx.x, ...) of B (m x n): B <- L^{-1} B, m <= kPanN.
__global__ void __launch_bounds__(kCT, 1)
panel_left_kernel(int m, int n, int slice, const float *__restrict__ L, int64_t ldl, float *B, int64_t ldb) {
    extern __shared__ __align__(16) unsigned char panel_smem[];
    SmemLeft &s = *reinterpret_cast<SmemLeft *>(panel_smem);
    const int64_t o = (int64_t)blockIdx.x * slice;
    const int w = (int)imin64(slice, n - o), nblk = (m + kNB - 1) / kNB;
    float *Bo = B + o * ldb;
    auto diag = [&](int j) {
        const int nb = min(kNB, m - j * kNB);
        request_rect(&s.t[j & 1][0][0], kNB + 4, L + (int64_t)j * kNB * (ldl + 1), ldl, nb, nb, kNB, kNB);
    };
    auto tile = [&](int j, int r0, int buf) {
        request_rect(&s.l[buf][0][0], kChunk + 4, L + r0 + (int64_t)j * kNB * ldl, ldl, m - r0, kNB, kChunk, kNB);
    };
    diag(0);
    request_rect(&s.x[0][0], kPanN + 4, Bo, ldb, m, w, nblk * kNB, slice);
    cp_async_commit();
    for (int j = 0; j < nblk; ++j) {
        const int r1 = (j + 1) * kNB;
        cp_async_wait<0>();
        __syncthreads();
        if (r1 < m) {
            diag(j + 1);
            tile(j, r1, 0);
        }
        cp_async_commit();
        block_solve_lower(s.t[j & 1], reinterpret_cast<float(*)[kPanN + 4]>(&s.x[0][j * kNB]), slice);
        for (int r0 = r1, buf = 0; r0 < m; r0 += kChunk, buf ^= 1) {
            if (r0 + kChunk < m) tile(j, r0 + kChunk, buf ^ 1);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            rank64<8, 4>(&s.l[buf][0][0], kChunk + 4, &s.x[0][j * kNB], kPanN + 4, &s.x[0][r0], kPanN + 4,
                         min(kChunk, nblk * kNB - r0), slice);
            __syncthreads();
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    store_rect(&s.x[0][0], kPanN + 4, Bo, ldb, m, w);
}

// Rows (columns) of B per CTA: whole waves over the SMs, a multiple of 4.
int panel_slice(int64_t m) {
    const int64_t sms = num_sms(), waves = cdiv(m, sms * kSlice);
    return (int)std::min<int64_t>(kSlice, cdiv(cdiv(m, sms * waves), 4) * 4);
}

// Narrow triangles against many rows.  The CTAs of the panel kernels hold a slice
// of whole panels, one to an SM, so from the second wave on (9472 rows) nothing
// hides a slice's loads, and a narrow triangle gives them little else to do.
// A thread per row (64 columns at a time, an SGEMM between) is then the better
// way, up to a width that grows with the waves; us, thread per row / slices:
// 32 wide 9500 rows 6.8 / 9.4, 60000 12.9 / 32.1; 64 wide 9500 11.6 / 9.8, 20000
// 12.5 / 13.9, 60000 22.7 / 35.0; 80 wide 20000 38.7 / 30.4; 96 wide 20000 39.2 /
// 30.5, 30000 41.7 / 45.2, 60000 76.5 / 79.9; 112 wide 40000 68.7 / 53.3, 60000
// 82.4 / 80.9.
bool rows_by_thread(int64_t m, int n) {
    const int64_t waves = cdiv(m, (int64_t)num_sms() * kSlice);
    return waves > 1 && n <= (waves == 2 ? 48 : waves == 3 ? 64 : 96);
}

// The same for the columns of the left solve, a warp per column: only for triangles of
// at most 16 (8 high 9500 columns 5.9 / 8.2 us, 60000 13.7 / 26.7; 16 high 9500 7.9 /
// 8.0, 60000 22.1 / 26.8; 32 high 9500 12.2 / 8.2), and for as few columns as
// each get a warp soon (16 high, 16 columns 2.8 / 3.8; 200 columns 7.3 / 4.1).
bool cols_by_warp(int m, int64_t n) { return m <= 16 && (n <= 32 || n > (int64_t)num_sms() * kSlice); }

}  // namespace

mxp_status launch_trsm_runn(int m, int n, const float *U, int64_t ldu, float *B, int64_t ldb,
                            cudaStream_t st) {
    if (m <= 0 || n <= 0) return MXP_OK;
    if (ldu < n || ldb < m) return fail(MXP_INVALID_ARG, "trsm_right_upper: bad leading dimension");
    MXP_CUDA(cudaFuncSetAttribute(panel_right_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemRight)));
    const int slice = panel_slice(m);
    const bool narrow = rows_by_thread(m, n);
    const int step = narrow ? kNB : kPanN;
    for (int j = 0; j < n; j += step) {
        const int w = std::min(step, n - j), rem = n - j - w;
        const float *Uj = U + (int64_t)j * (ldu + 1);
        float *Bj = B + (int64_t)j * ldb;
        mxp_status s = MXP_OK;
        if (narrow) {
            s = launch_trsm_runn_small(m, w, Uj, ldu, Bj, ldb, st);
        } else {
            panel_right_kernel<<<(unsigned)cdiv(m, slice), kCT, sizeof(SmemRight), st>>>(m, w, slice, Uj, ldu, Bj, ldb);
            MXP_LAUNCHED();
        }
        if (s != MXP_OK) return s;
        if (rem <= 0) break;
        s = launch_sgemm_sub(m, rem, w, Bj, ldb, U + j + (int64_t)(j + w) * ldu, ldu, Bj + (int64_t)w * ldb, ldb, st);
        if (s != MXP_OK) return s;
    }
    return MXP_OK;
}

mxp_status launch_trsm_llnu(int m, int n, const float *L, int64_t ldl, float *B, int64_t ldb,
                            cudaStream_t st) {
    if (m <= 0 || n <= 0) return MXP_OK;
    if (ldl < m || ldb < m) return fail(MXP_INVALID_ARG, "trsm_left_lower_unit: bad leading dimension");
    if (cols_by_warp(m, n)) return launch_trsm_llnu_small(m, n, L, ldl, B, ldb, st);
    MXP_CUDA(cudaFuncSetAttribute(panel_left_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemLeft)));
    const int slice = panel_slice(n);
    for (int j = 0; j < m; j += kPanN) {
        const int w = std::min(kPanN, m - j), rem = m - j - w;
        panel_left_kernel<<<(unsigned)cdiv(n, slice), kCT, sizeof(SmemLeft), st>>>(w, n, slice, L + (int64_t)j * (ldl + 1),
                                                                                   ldl, B + j, ldb);
        MXP_LAUNCHED();
        if (rem <= 0) break;
        mxp_status s = launch_sgemm_sub(rem, n, w, L + (j + w) + (int64_t)j * ldl, ldl, B + j, ldb, B + j + w, ldb, st);
        if (s != MXP_OK) return s;
    }
    return MXP_OK;
}

}  // namespace mxp
