// FP64 kernels of the iterative refinement.
//
//  * otf_gemv: y = beta*y + alpha*A*x with a_ij regenerated from the LCG in
//    FP64 (otf_gemv_h / otf_gemv_d / otf_gemv_diag_d, panel_gemv.hpp:13-117).
//    The reference launches one <<<b,256>>> kernel per b x b block pair and
//    synchronises after each; here one launch covers the matrix: each thread
//    owns two rows (two independent LCG chains) over a column range and
//    steps the state with J_n = INC1^n per column.  Each state enters as
//    its two exact 32-bit halves (no 64-bit converter, no rounding of the
//    integer), and the 2^-64 scale of RandStat::operator double is folded
//    into x.
//    Column splits write partial sums to the workspace and a second kernel
//    reduces them in a fixed order, so the result is deterministic.
//  * lu_solve: x <- U^{-1} L^{-1} x with the FP32 factors (trsvL_h /
//    trsvU_h, panel_trsv.hpp:308-597).  One persistent launch per triangle:
//    row blocks of 64 are claimed in order through an atomic ticket; a row
//    block streams its part of the factor against the already-solved blocks
//    (waiting, bounded, for their values), then solves its 64 x
//    64 diagonal triangle in FP64 and publishes.  Claim order guarantees every
//    awaited block is owned by a CTA that is already running.
//  * lu_solve_inv: the same solve in nb steps of bandwidth-bound products
//    with the stored inverses of the b x b diagonal blocks (used after
//    mxp_panel_lu, which keeps them); no chain of 64-row links.
//  * infnorm / vector ops (panel_norm.hpp:11-58, panel.hpp:525-623).
#include <algorithm>

#include "mxp_internal.cuh"

namespace mxp {

namespace {

// ---------------------------------------------------------------------------
// on-the-fly GEMV
// ---------------------------------------------------------------------------
constexpr int kGemvThreads = 128;
constexpr int kGemvRowsPerThread = 2;
constexpr int kGemvRows = kGemvThreads * kGemvRowsPerThread;  // 256 rows per CTA
constexpr int kGemvXChunk = 1024;
constexpr double kLcgScale = 0x1.fffffffffffffP-65;

// Per element the state s = hi * 2^32 + lo (hi signed, lo unsigned) enters
// as two exact doubles with a sum each: hi by the 32-bit integer converter (its
// sum times 2^32 at the end), and 2^52 + lo by placing lo in the mantissa of
// a biased constant, whose bias 2^52 is not removed per element: the CTA sums
// 2^52 * xs over its columns once and subtracts it from every row at the
// end (the bias terms are 2^-12 |x| each against |a_ij x| ~ |x|/4, so the
// extra rounding stays far below the FP64 rounding of the sum itself).  What
// bounds it is instructions per element (a loop of this element alone: 8.5
// elements per clock and SM; 7.8 with hi, too, built by a biased constant
// and a subtraction).  The
// diagonal column is accumulated like the others and its LCG value taken
// out afterwards (no compare per element), then d_i x_i is added.
__global__ void __launch_bounds__(kGemvThreads)
otf_gemv_kernel(int n, uint64_t s00, Aff jn, const double *__restrict__ d,
                const double *__restrict__ x, int64_t cols_per_split, double alpha, double beta,
                double *__restrict__ y, double *__restrict__ partials) {
    __shared__ double xs[kGemvXChunk];
    __shared__ double bias_red[kGemvThreads];
    const int64_t r0 = (int64_t)blockIdx.x * kGemvRows + threadIdx.x;
    const int64_t r1 = r0 + kGemvThreads;
    const int64_t j_begin = (int64_t)blockIdx.y * cols_per_split;
    const int64_t j_end = imin64(n, j_begin + cols_per_split);
    constexpr double kLoBias = 0x1p52;

    const Aff inc1 = lcg_inc1();
    // states of (r0, j_begin) and (r1, j_begin)
    uint64_t s0 = aff_apply(aff_pow(inc1, (uint64_t)r0 + (uint64_t)n * (uint64_t)j_begin), s00);
    uint64_t s1 = aff_apply(aff_pow(inc1, (uint64_t)kGemvThreads), s0);
    double acc0 = 0.0, acc1 = 0.0, hi0 = 0.0, hi1 = 0.0, bias = 0.0;
    for (int64_t jc = j_begin; jc < j_end; jc += kGemvXChunk) {
        const int len = (int)imin64(kGemvXChunk, j_end - jc);
        __syncthreads();
        for (int q = threadIdx.x; q < len; q += kGemvThreads) {
            const double v = x[jc + q] * kLcgScale;
            xs[q] = v;
            bias = __fma_rn(kLoBias, v, bias);
        }
        __syncthreads();
#pragma unroll 4
        for (int q = 0; q < len; ++q) {
            const double xq = xs[q];
            hi0 = __fma_rn((double)(int)(s0 >> 32), xq, hi0);
            hi1 = __fma_rn((double)(int)(s1 >> 32), xq, hi1);
            acc0 = __fma_rn(__hiloint2double(0x43300000, (int)(uint32_t)s0), xq, acc0);
            acc1 = __fma_rn(__hiloint2double(0x43300000, (int)(uint32_t)s1), xq, acc1);
            s0 = aff_apply(jn, s0);
            s1 = aff_apply(jn, s1);
        }
    }
    // the CTA's bias sum, in a fixed order
    bias_red[threadIdx.x] = bias;
    __syncthreads();
    for (int w = kGemvThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) bias_red[threadIdx.x] += bias_red[threadIdx.x + w];
        __syncthreads();
    }
    bias = bias_red[0];
    acc0 = __fma_rn(hi0, 0x1p32, acc0 - bias);
    acc1 = __fma_rn(hi1, 0x1p32, acc1 - bias);
    // diagonal entries come from d (otf_gemv_diag_d, panel_gemv.hpp:26): the
    // LCG value accumulated at (r, r) is taken out, d_r x_r added
    if (r0 < n && r0 >= j_begin && r0 < j_end) {
        const uint64_t sd = aff_apply(aff_pow(inc1, (uint64_t)r0 + (uint64_t)n * (uint64_t)r0), s00);
        acc0 = __fma_rn(-i64_to_double_rn(sd), x[r0] * kLcgScale, acc0) + d[r0] * x[r0];
    }
    if (r1 < n && r1 >= j_begin && r1 < j_end) {
        const uint64_t sd = aff_apply(aff_pow(inc1, (uint64_t)r1 + (uint64_t)n * (uint64_t)r1), s00);
        acc1 = __fma_rn(-i64_to_double_rn(sd), x[r1] * kLcgScale, acc1) + d[r1] * x[r1];
    }
    if (partials) {
        double *p = partials + (int64_t)blockIdx.y * n;
        if (r0 < n) p[r0] = acc0;
        if (r1 < n) p[r1] = acc1;
    } else {
        if (r0 < n) y[r0] = (beta == 0.0 ? 0.0 : beta * y[r0]) + alpha * acc0;
        if (r1 < n) y[r1] = (beta == 0.0 ? 0.0 : beta * y[r1]) + alpha * acc1;
    }
}

__global__ void gemv_reduce_kernel(int n, int splits, const double *__restrict__ partials,
                                   double alpha, double beta, double *__restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double t = 0.0;
    for (int s = 0; s < splits; ++s) t += partials[(int64_t)s * n + i];
    y[i] = (beta == 0.0 ? 0.0 : beta * y[i]) + alpha * t;
}

// The refinement's residual from the split partial sums, r = b - A x, with
// max |x| and max |r| for the stopping test (norms[0], norms[1]; zero at
// launch): as a copy, two norms and their clears each a launch or memset of its
// own, a refinement step of a small system spent ~25 us on them.
__global__ void residual_reduce_kernel(int n, int splits, const double *__restrict__ partials,
                                       const double *__restrict__ b, const double *__restrict__ x,
                                       double *__restrict__ r, unsigned long long *norms) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double mx = 0.0, mr = 0.0;
    if (i < n) {
        double t = 0.0;
        for (int s = 0; s < splits; ++s) t += partials[(int64_t)s * n + i];
        const double v = b[i] - t;
        r[i] = v;
        mx = max_nan(mx, fabs(x[i]));
        mr = max_nan(mr, fabs(v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = max_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mr = max_nan(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    }
    if ((threadIdx.x & 31) == 0) {  // (as infnorm_kernel: values without a sign order like their bits)
        atomicMax(norms, (unsigned long long)__double_as_longlong(mx));
        atomicMax(norms + 1, (unsigned long long)__double_as_longlong(mr));
    }
}

// ---------------------------------------------------------------------------
// sync-free block triangular solves
// ---------------------------------------------------------------------------
constexpr int kRB = 64;
constexpr int kTrsvThreads = 256;

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Block forward (LOWER: unit L) or backward (upper: U) substitution, one
// 64-row block per CTA, CTAs taking row blocks in solve order from a ticket.
//
// The blocks form a chain (block b needs x of every earlier block), so the
// time per link is what bounds the solve.  Everything that does not depend
// on the predecessor is done before waiting for it:
//   * Minv = inverse of the diagonal block (FP64, from the FP32 factor) and
//     P = Minv * A_adj, A_adj the off-diagonal block next in the chain;
//   * the products of all other off-diagonal blocks with their (already
//     solved) x, streamed with four column blocks of loads in flight;
//   * w = Minv (r_b - those products).
// When the predecessor publishes its x, the block finishes with one 64 x 64
// FP64 matrix-vector product, x_b = w - P x_adj, and publishes its own x.
// A value is published by its own 8-byte store to `mail`, which starts out as
// kNoMail everywhere: the value itself says that it is there, so a link
// takes neither a fence, a flag nor a second load (with a flag released after
// the values and polled before they are read a link took 3.7 us, of which
// ~1.4 us were those).  Sums run in four interleaved parts: a chain of
// dependent FP64 operations per column cost as much as the exchange.
// This is the block substitution of the reference's trsvL_h / trsvU_h
// (panel_trsv.hpp:308-597: FP64 solve of each upcast diagonal block, FP32 x
// FP64 products for the rest) with the diagonal solve applied as a product
// with its inverse.
constexpr unsigned long long kNoMail = ~0ull;  // a NaN no operation returns (published values are kept off it)

__device__ __forceinline__ unsigned long long ld_mail(const double *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_mail(double *p, double x) {
    unsigned long long v = (unsigned long long)__double_as_longlong(x);
    if (v == kNoMail) v = 0x7ff8000000000000ull;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The value at p, waited for (bounded): between polls the thread sleeps 100 ns for
// each of the `far` links the chain is away.  ok: cleared when the wait gave up.
__device__ __forceinline__ double take_mail(const double *p, int far, bool &ok) {
    unsigned long long v = ld_mail(p);
    if (v == kNoMail && ok) {
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t it = 1; (v = ld_mail(p)) == kNoMail; ++it) {
            if (far > 0) __nanosleep(100 * far);
            if ((it & 63u) == 0u && globaltimer_ns() - t0 > kWaitTimeoutNs) {
                ok = false;
                break;
            }
        }
    }
    return v == kNoMail ? 0.0 : __longlong_as_double((long long)v);
}

constexpr int kXChunk = 8;  // column blocks whose x is staged in shared memory at a time
constexpr int kMP = kRB + 4;    // pitch of Minv and P: four rows x four lanes on 16 banks
constexpr size_t kTrsvSmem = 2 * sizeof(double) * kRB * kMP + sizeof(float) * kRB * (kRB + 1) +
                             sizeof(double) * kRB + sizeof(double) * 4 * kRB +
                             sizeof(double) * 2 * kXChunk * kRB + 16;

template <bool LOWER>
__global__ void __launch_bounds__(kTrsvThreads)
trsv_kernel(int n, const float *__restrict__ LU, int64_t lda, double *x, double *mail, int *ticket,
            DevStatus *dst, int withhold) {
    extern __shared__ __align__(16) unsigned char trsv_smem[];
    double(*minv)[kMP] = reinterpret_cast<double(*)[kMP]>(trsv_smem);
    double(*pm)[kMP] = minv + kRB;
    float(*blk)[kRB + 1] = reinterpret_cast<float(*)[kRB + 1]>(pm + kRB);   // blk[col][row]
    double *zs = reinterpret_cast<double *>(blk + kRB);
    double(*part)[kRB] = reinterpret_cast<double(*)[kRB]>(zs + kRB);
    double(*xs)[kXChunk * kRB] = reinterpret_cast<double(*)[kXChunk * kRB]>(part + 4);  // 2 buffers
    int *s_ticket = reinterpret_cast<int *>(xs + 2);

    const int nrb = (n + kRB - 1) / kRB;
    const int tid = threadIdx.x;
    if (tid == 0) *s_ticket = atomicAdd(ticket, 1);
    __syncthreads();
    const int rb = LOWER ? *s_ticket : nrb - 1 - *s_ticket;
    const int64_t row0 = (int64_t)rb * kRB;
    const int nrows = (int)imin64(kRB, n - row0);
    const int ncb = LOWER ? rb : nrb - 1 - rb;  // off-diagonal column blocks
    const bool has_adj = ncb > 0;
    const int adj = LOWER ? rb - 1 : rb + 1;    // chain predecessor
    const double rhs = tid < nrows ? x[row0 + tid] : 0.0;

    // ---- Minv: inverse of the diagonal block (padded with the identity) ----
    for (int idx = tid; idx < kRB * kRB; idx += kTrsvThreads) {
        const int rr = idx % kRB, cc = idx / kRB;
        float v = (rr < nrows && cc < nrows) ? LU[(row0 + cc) * lda + row0 + rr] : 0.0f;
        if (rr == cc && (rr >= nrows || LOWER)) v = 1.0f;
        blk[cc][rr] = v;
    }
    __syncthreads();
    const int pi = tid >> 2, ph = tid & 3;
    {   // column pi of the inverse, T y = e_pi: four lanes share each sum over k
        const int j = pi;
        auto dot = [&](int i, int k0, int k1) {  // sum of T(i, k) y_k, k0 <= k < k1
            double s0 = 0.0, s1 = 0.0;
            int k = k0 + ph;
            for (; k + 4 < k1; k += 8) {
                s0 = __fma_rn((double)blk[k][i], minv[k][j], s0);
                s1 = __fma_rn((double)blk[k + 4][i], minv[k + 4][j], s1);
            }
            if (k < k1) s0 = __fma_rn((double)blk[k][i], minv[k][j], s0);
            s0 += s1;
            s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
            s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
            return s0;
        };
#pragma unroll 1
        for (int q = 0; q < kRB; ++q) {
            const int i = LOWER ? q : kRB - 1 - q;
            const double s = LOWER ? dot(i, j, i) : dot(i, i + 1, j + 1);
            if (ph == 0) {
                const double e = i == j ? 1.0 : 0.0;
                if (LOWER) minv[i][j] = i < j ? 0.0 : e - s;
                else minv[i][j] = i > j ? 0.0 : (e - s) / (double)blk[i][i];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // ---- P = Minv * A_adj ----
    // (row pi of a 64-vector, quarter ph of its columns)
    if (has_adj) {
        const int64_t c0 = (int64_t)adj * kRB;
        const int ncols = (int)imin64(kRB, n - c0);
        for (int idx = tid; idx < kRB * kRB; idx += kTrsvThreads) {
            const int rr = idx % kRB, cc = idx / kRB;
            blk[cc][rr] = (rr < nrows && cc < ncols) ? LU[(c0 + cc) * lda + row0 + rr] : 0.0f;
        }
        __syncthreads();
#pragma unroll 1
        for (int c = ph * 16; c < ph * 16 + 16; c += 4) {  // four columns: independent sums
            double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
            for (int k = 0; k < kRB; ++k) {
                const double m = minv[pi][k];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = __fma_rn(m, (double)blk[c + e][k], v[e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) pm[pi][c + e] = v[e];
        }
    }

    // ---- products with every other off-diagonal block ----
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0, acc3 = 0.0;
    bool timed_out = false;
    const int r = tid % kRB, cph = tid / kRB;  // 4 column phases of 16
    const int64_t grow = row0 + r;
    const bool row_ok = r < nrows;
    const int nstream = has_adj ? ncb - 1 : 0;
    auto load_l = [&](int q, float *d) {
        if (q >= nstream) return;
        const int cb = LOWER ? q : nrb - 1 - q;
        const int64_t c0 = (int64_t)cb * kRB + cph * 16;
        const int clen = (int)imin64(16, n - c0);
        const float *col = LU + c0 * lda + grow;
#pragma unroll
        for (int cc = 0; cc < 16; ++cc) d[cc] = (row_ok && cc < clen) ? col[cc * lda] : 0.0f;
    };
    // The x of the streamed column blocks is staged in shared memory kXChunk
    // blocks at a time (one coalesced load per thread and one barrier per
    // chunk, double-buffered) instead of one L2 round trip per column block:
    // the stream, not the chain, bounds the late blocks of a large solve.
    auto consume = [&](int buf, int qq, const float *lv) {
        const double *xv = xs[buf] + qq * kRB + cph * 16;
#pragma unroll
        for (int cc = 0; cc < 16; cc += 4) {
            acc0 = __fma_rn((double)lv[cc], xv[cc], acc0);
            acc1 = __fma_rn((double)lv[cc + 1], xv[cc + 1], acc1);
            acc2 = __fma_rn((double)lv[cc + 2], xv[cc + 2], acc2);
            acc3 = __fma_rn((double)lv[cc + 3], xv[cc + 3], acc3);
        }
    };
    // factor values do not depend on other blocks: keep four column blocks of
    // loads in flight (a register ring, unrolled so its indices stay static)
    float b0[16], b1[16], b2[16], b3[16];
    load_l(0, b0);
    load_l(1, b1);
    load_l(2, b2);
    load_l(3, b3);
    int buf = 0;
    for (int q0 = 0; q0 < nstream; q0 += kXChunk, buf ^= 1) {
        const int qn = min(kXChunk, nstream - q0);
        bool ok = true;
        for (int e = tid; e < qn * kRB; e += kTrsvThreads) {
            const int qq = e / kRB, cc = e % kRB;
            const int cb = LOWER ? q0 + qq : nrb - 1 - (q0 + qq);
            const int64_t col = (int64_t)cb * kRB + cc;
            const int far = min(32, (LOWER ? rb - cb : cb - rb) - 3);
            xs[buf][e] = (col < n) ? take_mail(mail + col, far, ok) : 0.0;
        }
        timed_out = !ok;
        // a wait that gave up anywhere in the CTA ends the stream everywhere
        timed_out = __syncthreads_or(timed_out) != 0;
        if (timed_out) break;
#pragma unroll
        for (int qq = 0; qq < kXChunk; qq += 4) {
            if (qq + 0 < qn) { consume(buf, qq + 0, b0); load_l(q0 + qq + 4, b0); }
            if (qq + 1 < qn) { consume(buf, qq + 1, b1); load_l(q0 + qq + 5, b1); }
            if (qq + 2 < qn) { consume(buf, qq + 2, b2); load_l(q0 + qq + 6, b2); }
            if (qq + 3 < qn) { consume(buf, qq + 3, b3); load_l(q0 + qq + 7, b3); }
        }
    }
    part[cph][r] = (acc0 + acc1) + (acc2 + acc3);
    __syncthreads();
    if (tid < kRB) {
        const double s = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
        zs[tid] = rhs - s;
    }
    __syncthreads();
    // ---- w = Minv z (row pi; lane ph of its four takes columns 4 c + ph) ----
    auto row_product = [&](const double (*m)[kMP], const double *v) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
            s0 = __fma_rn(m[pi][4 * c + ph], v[c], s0);
            s1 = __fma_rn(m[pi][4 * c + 4 + ph], v[c + 1], s1);
            s2 = __fma_rn(m[pi][4 * c + 8 + ph], v[c + 2], s2);
            s3 = __fma_rn(m[pi][4 * c + 12 + ph], v[c + 3], s3);
        }
        double s = (s0 + s1) + (s2 + s3);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        return s;
    };
    double xa[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) xa[c] = zs[4 * c + ph];
    double w = row_product(minv, xa);
    // ---- the chain link: x_b = w - P x_adj ----
    if (has_adj && !timed_out) {  // (the same in every thread)
        const int64_t c0 = (int64_t)adj * kRB;
        bool ok = true;
        // all sixteen together, again until none is missing (one by one each
        // would cost a round trip of its own)
        const double *mp = mail + c0 + ph;
        const int have = (int)imin64(kRB, n - c0) - ph;  // columns 4 c < have exist
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t it = 1;; ++it) {
            unsigned long long raw[16];
            bool missing = false;
#pragma unroll
            for (int c = 0; c < 16; ++c) raw[c] = 4 * c < have ? ld_mail(mp + 4 * c) : 0ull;
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                missing |= raw[c] == kNoMail;
                xa[c] = __longlong_as_double((long long)raw[c]);
            }
            if (!missing) break;
            if ((it & 63u) == 0u && globaltimer_ns() - t0 > kWaitTimeoutNs) {
                ok = false;
                break;
            }
        }
        w -= row_product(pm, xa);
        timed_out = !ok;
    }
    // published even after a timeout, so successors never stall; `withhold` (a
    // test of the bounded waits) leaves one block unpublished
    if (ph == 0 && pi < nrows) {
        if (rb != withhold) st_mail(mail + row0 + pi, w);
        x[row0 + pi] = w;
    }
    if (timed_out) report(dst, MXP_TIMEOUT, 10 + (LOWER ? 0 : 1), rb);
}

// ---------------------------------------------------------------------------
// block triangular solves with the stored inverses of the diagonal blocks
// ---------------------------------------------------------------------------
// The LU keeps inv(L_kk) and inv(U_kk) of every b x b diagonal block (the
// TRSM-by-inverse computes them anyway).  A triangle is then solved in nb
// steps of bandwidth-bound products instead of a chain of 64-row links:
//   lower, k = 0 .. nb-1:  x_k <- L_kk^{-1} x_k;  x_i -= L(i, k) x_k (rows below)
//   upper, k = nb-1 .. 0:  x_k <- U_kk^{-1} x_k;  x_i -= U(i, k) x_k (rows above)
// Block substitution as trsvL_h / trsvU_h (panel_trsv.hpp:308-597).  The
// diagonal-block solve is a product with the stored inverse X followed by
// one step of refinement against the factor block T, all in FP64:
//   t1 = X v,  s = v - T t1,  t = t1 + X s,
// so the result carries the square of the inverse's relative error (the
// inverse's tensor-core levels are near FP32, not FP32).  The unit diagonal
// of inv(L) and the diagonal 1/u_ii of inv(U) are applied exactly.  Every
// row is summed by one CTA in a fixed order: results are deterministic.
// The diagonal-block products are load-latency bound (a 13 MB triangle at
// b = 2560): small row tiles give many CTAs, each staging only the part of v
// its rows use; the trailing products stream the factor at HBM bandwidth.
//
// All steps of both triangles run in one cooperative launch, separated by grid
// barriers: a launch per product (four per step on the chain, two streams)
// spent ~23 us per step at b = 256 on launch gaps.  Per step:
//   1: t1 = X x_k   2: s = x_k - T t1   3: t2 = t1 + X s
//   4: x_i -= M(i,k) t2 for the rows of the next block (x_k = t2 with it)
// and the update of all rows beyond the next block, which only step k+2
// needs, is done in the barriers' shadow: a CTA that has arrived at barrier
// 4, 1 and 2 works off a third of its share before it waits, so for a large
// factor the chain hides behind that stream (HBM-bound) and for a small one
// the barriers are all there is.  Every row is summed by one CTA in a fixed
// order and receives its updates in step order.
constexpr int kIvThreads = 512;
constexpr int kIvWarps = kIvThreads / 32;
constexpr int kIvRowsUpd = 32;   // rows per tile of the trailing products (a column: one 128-byte line)
constexpr int kIvRowsDiag = 8;   // rows per tile on the chain (many CTAs, whole 32-byte sectors)
constexpr int kIvDepth = 4;      // 16-byte loads in flight per thread, two CTAs per SM

// bulk vector, the warps' row sums
size_t trsv_inv_smem(int b) { return ((size_t)b + kIvWarps * kIvRowsUpd) * sizeof(double); }

struct InvSolve {
    int n, b;
    const float *LU;
    int64_t lda;
    const float *X[2];   // inv(U_00), inv(L_00)
    int64_t xstride;
    double *x, *t;       // t: 4 b doubles
    unsigned int *count; // grid-barrier arrivals (zero at launch)
    int *abort;
    DevStatus *dst;
};

// Grid barrier in two halves.  The waiter gives up after kWaitTimeoutNs, or
// when another CTA did.
__device__ __forceinline__ void iv_arrive(const InvSolve &a) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.count) : "memory");
}
__device__ __forceinline__ bool iv_wait(const InvSolve &a, unsigned &epoch, int where) {
    __shared__ int ok_sh;
    epoch += gridDim.x;
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned long long t0 = globaltimer_ns();
        for (unsigned it = 1; (unsigned)ld_acquire(reinterpret_cast<const int *>(a.count)) < epoch; ++it) {
            if (it & 63u) continue;
            if (ld_acquire(a.abort)) {
                ok = 0;
                break;
            }
            if (globaltimer_ns() - t0 > kWaitTimeoutNs) {
                ok = 0;
                atomicExch(a.abort, 1);
                report(a.dst, MXP_TIMEOUT, where, blockIdx.x);
                break;
            }
        }
        ok_sh = ok;
    }
    __syncthreads();
    return ok_sh != 0;
}

// One tile: ROWS rows (ROWS/4 quads of four rows, one float4 per column) x
// kIvThreads / (ROWS/4) column groups (ROWS >= 8: a warp reads whole 32-byte
// sectors).  M: column-major FP32, ldm % 4 == 0, 16-byte
// aligned.  vs: cols doubles; VG: in global memory (written by other CTAs), else
// shared.  ready() is called when the first loads of M are under way and
// returns when vs may be read (the chain waits for its barrier there).  With
// sum_i over the mode's entries of row i:
//   MODE 0: out[i] = base[i] - sum_j M(i,j) v_j                 (all columns)
//   MODE 1: out[i] = [base[i] +] v_i + sum_{j<i} M(i,j) v_j      (unit lower inverse)
//   MODE 2: out[i] = [base[i] +] v_i / T(i,i) + sum_{j>i} M(i,j) v_j  (upper inverse)
//   MODE 3: out[i] = base[i] - v_i - sum_{j<i} M(i,j) v_j        (v - T v, T unit lower)
//   MODE 4: out[i] = base[i] - sum_{j>=i} M(i,j) v_j             (v - T v, T upper)
// T(i,i) is read from tdiag (ld ldt).  base and out are data other CTAs write.
template <int MODE, int ROWS, bool VG, typename Ready>
__device__ __forceinline__ void iv_tile(double (*red)[kIvRowsUpd], int cols, const float *__restrict__ M,
                                        int64_t ldm, int r0, const double *vs,
                                        Ready ready, const float *__restrict__ tdiag, int64_t ldt, const double *base,
                                        double *out) {
    constexpr int QUADS = ROWS / 4;
    constexpr int GROUPS = kIvThreads / QUADS;
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr bool kLow = MODE == 1 || MODE == 3;   // strictly lower entries
    constexpr bool kUpS = MODE == 2;                // strictly upper
    constexpr bool kUpD = MODE == 4;                // upper with the diagonal
    const int q = tid % QUADS, g = tid / QUADS;
    const int ri = r0 + 4 * q;  // first of this thread's four rows
    // column range the tile's rows need
    int jb = 0, je = cols;
    if (kLow) je = min(cols, r0 + ROWS - 1);
    if (kUpS) jb = r0 + 1;
    if (kUpD) jb = r0;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    const float *mp = M + ri;
    float4 m[kIvDepth];
    auto load = [&](int j) {
#pragma unroll
        for (int u = 0; u < kIvDepth; ++u)
            m[u] = j + GROUPS * u < je ? __ldcs(reinterpret_cast<const float4 *>(mp + (int64_t)(j + GROUPS * u) * ldm))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    int j = jb + g;
    load(j);
    ready();
    auto value = [&](int q) { return VG ? __ldcg(vs + q) : vs[q]; };
    for (; j < je; j += kIvDepth * GROUPS) {
        float4 c[kIvDepth];
        double v[VG ? kIvDepth : 1];
#pragma unroll
        for (int u = 0; u < kIvDepth; ++u) {
            c[u] = m[u];
            if constexpr (VG) v[u] = j + GROUPS * u < je ? value(j + GROUPS * u) : 0.0;
        }
        const int jn = j + kIvDepth * GROUPS;
        if (!VG && jn < je) load(jn);
#pragma unroll
        for (int u = 0; u < kIvDepth; ++u) {
            const int jj = j + GROUPS * u;
            if (jj >= je) break;
            double vj;
            if constexpr (VG) vj = v[u];
            else vj = vs[jj];
            if (MODE == 0) {
                a0 = __fma_rn((double)c[u].x, vj, a0);
                a1 = __fma_rn((double)c[u].y, vj, a1);
                a2 = __fma_rn((double)c[u].z, vj, a2);
                a3 = __fma_rn((double)c[u].w, vj, a3);
            } else {
                const bool k0 = kLow ? jj < ri : (kUpS ? jj > ri : jj >= ri);
                const bool k1 = kLow ? jj < ri + 1 : (kUpS ? jj > ri + 1 : jj >= ri + 1);
                const bool k2 = kLow ? jj < ri + 2 : (kUpS ? jj > ri + 2 : jj >= ri + 2);
                const bool k3 = kLow ? jj < ri + 3 : (kUpS ? jj > ri + 3 : jj >= ri + 3);
                a0 = __fma_rn(k0 ? (double)c[u].x : 0.0, vj, a0);
                a1 = __fma_rn(k1 ? (double)c[u].y : 0.0, vj, a1);
                a2 = __fma_rn(k2 ? (double)c[u].z : 0.0, vj, a2);
                a3 = __fma_rn(k3 ? (double)c[u].w : 0.0, vj, a3);
            }
        }
        if (VG && jn < je) load(jn);  // (the values of v take the registers a second batch would)
    }
    // sum over the column groups: the warp's by shuffles, the warps' in order
#pragma unroll
    for (int o = QUADS; o < 32; o <<= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        a3 += __shfl_xor_sync(0xffffffffu, a3, o);
    }
    __syncthreads();  // the previous tile's sums have been read
    if (lane < QUADS) {
        double *rd = &red[tid >> 5][4 * lane];
        rd[0] = a0;
        rd[1] = a1;
        rd[2] = a2;
        rd[3] = a3;
    }
    __syncthreads();
    if (tid < ROWS) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < kIvWarps; ++c) s += red[c][tid];
        const int i = r0 + tid;
        double y;
        if (MODE == 0) y = __ldcg(base + i) - s;
        else if (MODE == 1) y = value(i) + s;
        else if (MODE == 2) y = value(i) / (double)tdiag[(int64_t)i * (ldt + 1)] + s;
        else if (MODE == 3) y = __ldcg(base + i) - value(i) - s;
        else y = __ldcg(base + i) - s;
        if ((MODE == 1 || MODE == 2) && base) y += __ldcg(base + i);
        out[i] = y;
    }
}

// A product with a triangle of the diagonal block: out = ... over b rows.  wait():
// the barrier the product's vectors are complete after, called once, with the
// first tile's loads of M under way.
template <int MODE, typename Wait>
__device__ __forceinline__ void iv_chain(double (*red)[kIvRowsUpd], int b, const float *M, int64_t ldm,
                                         const double *v, const float *tdiag, int64_t ldt, const double *base,
                                         double *out, Wait wait) {
    int t = blockIdx.x;
    if (t * kIvRowsDiag >= b) {
        wait();
        return;
    }
    iv_tile<MODE, kIvRowsDiag, true>(red, b, M, ldm, t * kIvRowsDiag, v, wait, tdiag, ldt, base, out);
    for (t += gridDim.x; t * kIvRowsDiag < b; t += gridDim.x)
        iv_tile<MODE, kIvRowsDiag, true>(red, b, M, ldm, t * kIvRowsDiag, v, [] {}, tdiag, ldt, base, out);
}

// Both halves of a step's barriers are apart: a CTA arrives, works off a share of
// the bulk update, requests its part of the next product's matrix and then
// waits.  ok: cleared when a wait gave up (the CTA then leaves at the step's end).
template <bool LOWER>
__device__ bool iv_triangle(const InvSolve &a, double *vb, double (*red)[kIvRowsUpd], unsigned &epoch) {
    const int n = a.n, b = a.b, nb = n / b;
    double *t1 = a.t, *sv = a.t + b;
    const double *none = nullptr;
    bool ok = true;
    // rows beyond the next block, updated with the last step's t2 (in vb)
    const float *bulk_m = nullptr;
    double *bulk_x = nullptr;
    int bulk_next = 0, bulk_tiles = 0;
    auto bulk = [&](int parts) {  // 1/parts of what this CTA still has to do
        const int left = bulk_next < bulk_tiles ? (bulk_tiles - bulk_next + (int)gridDim.x - 1) / (int)gridDim.x : 0;
        for (int i = (left + parts - 1) / parts; i > 0; --i, bulk_next += gridDim.x)
            iv_tile<0, kIvRowsUpd, false>(red, b, bulk_m, a.lda, bulk_next * kIvRowsUpd, vb, [] {}, nullptr, 0, bulk_x,
                                          bulk_x);
    };
    auto wait = [&](int where) { ok = iv_wait(a, epoch, where) && ok; };
    for (int s = 0; s < nb; ++s) {
        const int k = LOWER ? s : nb - 1 - s;
        const int64_t kk = (int64_t)k * b;
        const float *X = a.X[LOWER ? 1 : 0] + k * a.xstride, *T = a.LU + kk + kk * a.lda;
        double *xk = a.x + kk, *t2 = a.t + (2 + (s & 1)) * (int64_t)b;
        // (the first step's x is complete at launch, or after the last triangle's final barrier)
        iv_chain<LOWER ? 1 : 2>(red, b, X, b, xk, T, a.lda, none, t1, [&] {
            if (s > 0) wait(53);
        });
        iv_arrive(a);
        bulk(2);
        iv_chain<LOWER ? 3 : 4>(red, b, T, a.lda, t1, T, a.lda, xk, sv, [&] { wait(50); });
        iv_arrive(a);
        bulk(1);
        iv_chain<LOWER ? 1 : 2>(red, b, X, b, sv, T, a.lda, t1, t2, [&] { wait(51); });
        iv_arrive(a);
        // the next block's rows, on the chain; t2 goes to vb for this step's updates, and is x_k
        auto take = [&] {
            wait(52);
            for (int j = threadIdx.x; j < b; j += kIvThreads) {
                const double v = __ldcg(t2 + j);
                vb[j] = v;
                if (blockIdx.x == 0) xk[j] = v;
            }
            __syncthreads();
        };
        int t = blockIdx.x;
        const bool next = s + 1 < nb;
        const int64_t nx = next ? (LOWER ? kk + b : kk - b) : 0;
        const float *Mn = a.LU + nx + kk * a.lda;
        if (next && t * kIvRowsDiag < b) {
            iv_tile<0, kIvRowsDiag, false>(red, b, Mn, a.lda, t * kIvRowsDiag, vb, take, nullptr, 0, a.x + nx, a.x + nx);
            for (t += gridDim.x; t * kIvRowsDiag < b; t += gridDim.x)
                iv_tile<0, kIvRowsDiag, false>(red, b, Mn, a.lda, t * kIvRowsDiag, vb, [] {}, nullptr, 0, a.x + nx,
                                               a.x + nx);
        } else {
            take();
        }
        const int64_t r0 = LOWER ? kk + 2 * (int64_t)b : 0;
        const int64_t rows = LOWER ? n - r0 : kk - b;
        bulk_m = a.LU + r0 + kk * a.lda;
        bulk_x = a.x + r0;
        bulk_tiles = rows > 0 ? (int)(rows / kIvRowsUpd) : 0;
        // the CTAs that had no tile on the chain take theirs first
        bulk_next = (int)gridDim.x - 1 - (int)blockIdx.x;
        if (!ok) return false;
        iv_arrive(a);
        bulk(3);
    }
    wait(53);
    return ok;
}

__global__ void __launch_bounds__(kIvThreads, 2) trsv_inv_kernel(InvSolve a) {
    extern __shared__ __align__(16) unsigned char iv_smem[];
    double *vb = reinterpret_cast<double *>(iv_smem);
    double(*red)[kIvRowsUpd] = reinterpret_cast<double(*)[kIvRowsUpd]>(vb + a.b);
    unsigned epoch = 0;
    if (!iv_triangle<true>(a, vb, red, epoch)) return;
    iv_triangle<false>(a, vb, red, epoch);
}

// ---------------------------------------------------------------------------
// norms and vector ops
// ---------------------------------------------------------------------------
__global__ void infnorm_kernel(int n, const double *__restrict__ x, unsigned long long *out) {
    double m = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        m = max_nan(m, fabs(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = max_nan(m, red[w]);
        // values without a sign order like their bit patterns, NaN above infinity
        atomicMax(out, (unsigned long long)__double_as_longlong(m));
    }
}

__global__ void norma_kernel(int n, const double *__restrict__ d, const double *__restrict__ rs,
                             unsigned long long *out) {
    double m = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        m = max_nan(m, rs ? rs[i] + d[i] : 2.0 * d[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = max_nan(m, red[w]);
        atomicMax(out, (unsigned long long)__double_as_longlong(m));
    }
}

__global__ void ir_init_kernel(int n, const double *__restrict__ rhs, const double *__restrict__ d,
                               double *__restrict__ x) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = rhs[i] / d[i];
}

__global__ void copy_kernel(int n, const double *__restrict__ s, double *__restrict__ t) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) t[i] = s[i];
}

__global__ void axpy_kernel(int n, double alpha, const double *__restrict__ x, double *__restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += alpha * x[i];
}

}  // namespace

// How a product of order n is split: row blocks x column splits of `cols` columns.
static void gemv_grid(int n, int max_splits, int *row_blocks, int *splits, int64_t *cols) {
    *row_blocks = (int)cdiv(n, kGemvRows);
    // 12 CTAs (48 warps) per SM where the column splits allow: an element is a
    // chain of an LCG step and three FP64 operations, hidden only by other warps
    // (n = 30011: 468 us with 4 CTAs per SM, 457 with 12)
    const int target = 12 * num_sms();
    int s = std::min((target + *row_blocks - 1) / *row_blocks, max_splits);
    *cols = cdiv(cdiv(n, s), 64) * 64;
    *splits = std::max(1, (int)cdiv(n, *cols));
}

mxp_status launch_otf_gemv(int n, uint64_t seed, const double *d, double alpha, const double *x,
                           double beta, double *y, double *partials, int max_splits,
                           cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    int row_blocks, splits;
    int64_t cols;
    gemv_grid(n, partials ? max_splits : 1, &row_blocks, &splits, &cols);
    const uint64_t s00 = lcg_stat00(seed);
    const Aff jn = aff_pow(lcg_inc1(), (uint64_t)n);
    dim3 grid((unsigned)row_blocks, (unsigned)splits);
    otf_gemv_kernel<<<grid, kGemvThreads, 0, st>>>(n, s00, jn, d, x, cols, alpha, beta, y,
                                                   splits > 1 ? partials : nullptr);
    MXP_LAUNCHED();
    if (splits > 1) {
        gemv_reduce_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, splits, partials, alpha, beta, y);
        MXP_LAUNCHED();
    }
    return MXP_OK;
}

mxp_status launch_residual(int n, uint64_t seed, const double *d, const double *b, const double *x, double *r,
                           double *norms, double *partials, int max_splits, cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    int row_blocks, splits;
    int64_t cols;
    gemv_grid(n, max_splits, &row_blocks, &splits, &cols);
    const uint64_t s00 = lcg_stat00(seed);
    const Aff jn = aff_pow(lcg_inc1(), (uint64_t)n);
    MXP_CUDA(cudaMemsetAsync(norms, 0, 2 * sizeof(double), st));
    dim3 grid((unsigned)row_blocks, (unsigned)splits);
    otf_gemv_kernel<<<grid, kGemvThreads, 0, st>>>(n, s00, jn, d, x, cols, 1.0, 0.0, nullptr, partials);
    MXP_LAUNCHED();
    residual_reduce_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, splits, partials, b, x, r,
                                                                   reinterpret_cast<unsigned long long *>(norms));
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_lu_solve(int n, const float *LU, int64_t lda, double *x, double *mail, int *tickets,
                           DevStatus *dst, cudaStream_t st, int withhold) {
    if (n <= 0) return MXP_OK;
    if (lda < n) return fail(MXP_INVALID_ARG, "lu_solve: lda < n");
    const int nrb = (int)cdiv(n, kRB);
    MXP_CUDA(cudaMemsetAsync(tickets, 0, 2 * sizeof(int), st));
    MXP_CUDA(cudaMemsetAsync(mail, 0xff, 2 * (size_t)n * sizeof(double), st));
    MXP_CUDA(cudaFuncSetAttribute(trsv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsvSmem));
    MXP_CUDA(cudaFuncSetAttribute(trsv_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsvSmem));
    trsv_kernel<true><<<nrb, kTrsvThreads, kTrsvSmem, st>>>(n, LU, lda, x, mail, tickets, dst, withhold);
    MXP_LAUNCHED();
    trsv_kernel<false><<<nrb, kTrsvThreads, kTrsvSmem, st>>>(n, LU, lda, x, mail + n, tickets + 1, dst, -1);
    MXP_LAUNCHED();
    return MXP_OK;
}

bool lu_solve_inv_supported(int n, int b, const float *LU, int64_t lda) {
    return n > 0 && b > 0 && n % b == 0 && b % kIvRowsUpd == 0 && lda % 4 == 0 &&
           (reinterpret_cast<uintptr_t>(LU) & 15u) == 0 && trsv_inv_smem(b) <= 200 * 1024;
}

mxp_status launch_lu_solve_inv(int n, int b, const float *LU, int64_t lda, const float *XU,
                               const float *XL, int64_t xstride, double *x, double *t, unsigned int *sync_words,
                               DevStatus *dst, cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    if (!lu_solve_inv_supported(n, b, LU, lda) || xstride % 4 != 0 ||
        ((reinterpret_cast<uintptr_t>(XU) | reinterpret_cast<uintptr_t>(XL)) & 15u))
        return fail(MXP_INVALID_ARG, "lu_solve_inv: shape or alignment not supported");
    InvSolve a{n, b, LU, lda, {XU, XL}, xstride, x, t, sync_words, reinterpret_cast<int *>(sync_words + 1), dst};
    void *args[] = {&a};
    const size_t smem = trsv_inv_smem(b);
    MXP_CUDA(cudaFuncSetAttribute(trsv_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    MXP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trsv_inv_kernel, kIvThreads, smem));
    if (per_sm < 1) return fail(MXP_UNSUPPORTED, "lu_solve_inv: kernel cannot be made resident");
    // as many CTAs as a step has tiles (fewer make the barriers cheaper), all co-resident
    const int64_t tiles = std::max<int64_t>(b / kIvRowsDiag, n / kIvRowsUpd);
    const int grid = (int)imin64(tiles, (int64_t)num_sms() * std::min(per_sm, 2));
    MXP_CUDA(cudaMemsetAsync(sync_words, 0, 2 * sizeof(unsigned int), st));
    MXP_CUDA(cudaLaunchCooperativeKernel((const void *)trsv_inv_kernel, dim3(grid), dim3(kIvThreads), args, smem, st));
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_infnorm(int n, const double *x, double *out, cudaStream_t st) {
    MXP_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
    if (n <= 0) return MXP_OK;
    const int blocks = (int)imin64(cdiv(n, 256), 2 * num_sms());
    infnorm_kernel<<<blocks, 256, 0, st>>>(n, x, reinterpret_cast<unsigned long long *>(out));
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_norma(int n, const double *d, const double *rowsum, double *out, cudaStream_t st) {
    MXP_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
    if (n <= 0) return MXP_OK;
    const int blocks = (int)imin64(cdiv(n, 256), 2 * num_sms());
    norma_kernel<<<blocks, 256, 0, st>>>(n, d, rowsum, reinterpret_cast<unsigned long long *>(out));
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_ir_init(int n, const double *rhs, const double *d, double *x, cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    ir_init_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, rhs, d, x);
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_copy(int n, const double *src, double *dst, cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    copy_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, src, dst);
    MXP_LAUNCHED();
    return MXP_OK;
}

mxp_status launch_axpy(int n, double alpha, const double *x, double *y, cudaStream_t st) {
    if (n <= 0) return MXP_OK;
    axpy_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(n, alpha, x, y);
    MXP_LAUNCHED();
    return MXP_OK;
}

}  // namespace mxp
