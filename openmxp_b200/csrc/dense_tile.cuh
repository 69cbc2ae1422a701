// SIMT FP32 building blocks shared by the cooperative diagonal-block
// factorisation (diag_coop.cu) and the batched solver (batched.cu): a
// 128 x 128 GEMM tile, the 64 x 64 no-pivot LU and the two 64-wide strip
// solves.  Every function is called by all kCT threads of the CTA (they
// contain __syncthreads) and reads its inputs through L2 (ld.global.cg), so it
// may follow writes made by other CTAs behind a grid barrier.
#pragma once

#include "mxp_internal.cuh"

namespace mxp {
namespace dt {
namespace {  // internal linkage: each translation unit keeps its own copy

constexpr int kCT = 256;  // threads per CTA
constexpr int kNB = 64;   // inner block of the LU
constexpr int GBM = 128, GBN = 128, GBK = 16;

struct SmemGemm {
    float As[GBK][GBM];
    float Bs[GBK][GBN + 4];
};
struct __align__(16) PanelRows {  // getrf64: four pivot rows at a time, for every lane
    float r[3][4][4][16];         // [warp][four-pivot step][row][column]
};
struct __align__(16) SmemTri {
    float t[kNB][kNB + 4];   // t[col][row] of a 64 x 64 block (16-byte rows)
    float us[kNB][kNB];      // us[k][c] = U(k, k + 1 + c): row k of U right of the diagonal, zero past the block
    float ls[kNB][kNB];      // ls[k][c] = L(k + 1 + c, k): column k of L below the diagonal, zero past the block
    float dinv[kNB];
    PanelRows rows;          // getrf64: pivot rows in exchange
};
union __align__(16) Smem {
    SmemGemm g;
    SmemTri t;
};

// A 64 x 64 block (rows r < nb, columns c < nb; zero elsewhere) from global
// memory through L2 into registers: 16 values per thread, element q at
// column (threadIdx.x + 256 q) / 64, row (threadIdx.x + 256 q) % 64.  All 16
// loads are issued before any is used, so the block costs one L2 round trip.
static_assert(kCT * 16 == kNB * kNB, "64 x 64 block = 16 values per thread");
template <int N>
__device__ __forceinline__ void load_block64(float (&v)[N], const float *D, int64_t ld, int nr, int nc) {
    static_assert(N >= 16, "16 values per thread");
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int idx = threadIdx.x + kCT * q;
        const int r = idx % kNB, c = idx / kNB;
        v[q] = (r < nr && c < nc) ? __ldcg(D + (int64_t)c * ld + r) : 0.0f;
    }
}

// One pivot of a right-looking elimination on a row held in registers that
// moves left by one column per pivot: x[c] = x[c + 1] - s[c] * v for c < W - 1,
// x[W - 1] = 0.  With x[0] the pivot column and s the pivot row (or column)
// right of the diagonal, this is x_j -= s_j v for j > k in the same operation
// (one fmaf) as the unrotated loop, but every pivot runs the same code, so the
// pivot loop stays rolled: fully unrolled 64-pivot eliminations are thousands
// of straight-line instructions, and their instruction fetch, not the FMA
// pipe, set their speed (~8-10 cycles per instruction in a per-step trace).
// W (the live width, 64 - 16 p in phase p of a 64-wide elimination) skips the
// columns the rotation has already emptied.  s is 16-byte aligned.
template <int W>
__device__ __forceinline__ void rot_axpy(float (&x)[kNB], const float *s, float v) {
#pragma unroll
    for (int c4 = 0; c4 < W / 4; ++c4) {
        const float4 u = *reinterpret_cast<const float4 *>(s + 4 * c4);
        x[4 * c4 + 0] = fmaf(-u.x, v, x[4 * c4 + 1]);
        x[4 * c4 + 1] = fmaf(-u.y, v, x[4 * c4 + 2]);
        x[4 * c4 + 2] = fmaf(-u.z, v, x[4 * c4 + 3]);
        x[4 * c4 + 3] = (4 * c4 + 4 < W) ? fmaf(-u.w, v, x[4 * c4 + 4]) : 0.0f;
    }
}


// ---- 128 x 128 SIMT GEMM tile ------------------------------------------------
// C[m0:m0+128, n0:n0+128] (clipped to m x n) = alpha * sum_{k in [kb, ke)} A(:,k) B(k,:)
// (+ C when accumulate).  8 x 8 outputs per thread.
// skip > 0 leaves the tile's top-left skip x skip corner untouched (another CTA
// owns it).
__device__ void gemm_tile(Smem &sm, int m, int n, int kb, int ke, float alpha,
                          const float *__restrict__ A, int64_t lda, const float *__restrict__ B,
                          int64_t ldb, bool accumulate, float *C, int64_t ldc, int m0, int n0,
                          int skip = 0) {
    const int t = threadIdx.x;
    const int tx = t % 16, ty = t / 16;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;

    float ra[8], rb[8];
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int idx = t + kCT * q;
            const int kk = idx / GBM, r = idx % GBM;
            const int gr = m0 + r, gk = k0 + kk;
            ra[q] = (gr < m && gk < ke) ? __ldcg(A + (int64_t)gk * lda + gr) : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int idx = t + kCT * q;
            const int cc = idx / GBK, kk = idx % GBK;
            const int gc = n0 + cc, gk = k0 + kk;
            rb[q] = (gc < n && gk < ke) ? __ldcg(B + (int64_t)gc * ldb + gk) : 0.0f;
        }
    };
    if (kb < ke) load(kb);
    for (int k0 = kb; k0 < ke; k0 += GBK) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int idx = t + kCT * q;
            sm.g.As[idx / GBM][idx % GBM] = ra[q];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int idx = t + kCT * q;
            sm.g.Bs[idx % GBK][idx / GBK] = rb[q];
        }
        __syncthreads();
        if (k0 + GBK < ke) load(k0 + GBK);
#pragma unroll
        for (int kk = 0; kk < GBK; ++kk) {
            const float4 a0 = *reinterpret_cast<const float4 *>(&sm.g.As[kk][tx * 4]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&sm.g.As[kk][64 + tx * 4]);
            const float4 b0 = *reinterpret_cast<const float4 *>(&sm.g.Bs[kk][ty * 4]);
            const float4 b1 = *reinterpret_cast<const float4 *>(&sm.g.Bs[kk][64 + ty * 4]);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
    // C is read in full before any store: interleaved loads and stores through a
    // pointer the compiler cannot disambiguate would serialise 64 L2 round trips
    if (accumulate) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int gc = n0 + (j < 4 ? ty * 4 + j : 64 + ty * 4 + (j - 4));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int gr = m0 + (i < 4 ? tx * 4 + i : 64 + tx * 4 + (i - 4));
                acc[i][j] *= alpha;
                if (gr < m && gc < n) acc[i][j] += __ldcg(C + (int64_t)gc * ldc + gr);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][j] *= alpha;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int gc = n0 + (j < 4 ? ty * 4 + j : 64 + ty * 4 + (j - 4));
        if (gc >= n) continue;
        float *cc = C + (int64_t)gc * ldc;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int gr = m0 + (i < 4 ? tx * 4 + i : 64 + tx * 4 + (i - 4));
            if (gr < m && !(gr - m0 < skip && gc - n0 < skip)) cc[gr] = acc[i][j];
        }
    }
    __syncthreads();  // shared tiles are reused by the caller's next item
}

// ---- 128 x 128 SIMT GEMM tile staged by cp.async -----------------------------
// The same tile as gemm_tile with the same per-element operation order (each
// output is one fmaf chain over k ascending from 0, then times alpha, then
// plus C), so the two give identical bits; only the data movement differs.
// gemm_tile moves 16-deep slices through registers with two CTA barriers
// each and reads C by scattered scalar loads after the products, which puts
// four L2 round trips and 64 uncoalesced requests per thread on every
// 128 x 128 x 64 tile.  Here 16-byte cp.async copies (L2 only, .cg: the data
// may come from other CTAs behind a grid barrier) bring a whole 64-deep
// slice of both operands and, for an accumulating tile, the C tile into
// shared memory at once, the next slice streams into the second buffer
// while the current one is multiplied, and C is written back by float4
// stores.  Needs 16-byte aligned bases, leading dimensions that are
// multiples of 4 floats and kb % 4 == 0 (gemm_tile_v_ok); ragged edges are
// zero-filled through cp.async's source size.
struct __align__(16) SmemGVBuf {
    float As[kNB][GBM];      // As[k][row]
    float Bs[GBN][kNB + 4];  // Bs[col][k]
};
struct __align__(16) SmemGV {
    SmemGVBuf buf[2];  // two 64-deep operand slices; a C tile Cs[col][row] (pitch 132) in buf[1]
};
static_assert(sizeof(SmemGVBuf) == sizeof(float) * GBN * (GBM + 4), "the C tile fills one operand buffer");

__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }
__device__ __forceinline__ bool gemm_tile_v_ok(const float *A, int64_t lda, const float *B, int64_t ldb,
                                               const float *C, int64_t ldc, int kb) {
    return aligned16(A) && aligned16(B) && aligned16(C) && ((lda | ldb | ldc) & 3) == 0 && (kb & 3) == 0;
}

// bytes of a 4-float group starting at index i of an extent e (0 .. 16)
__device__ __forceinline__ int grp_bytes(int i, int e) { return 4 * max(0, min(4, e - i)); }

// one 64-deep slice [k0, k0 + 64) ∩ [k0, ke) of A(m0:m0+128, :) and B(:, n0:n0+128)
__device__ __forceinline__ void gv_load_slice(SmemGVBuf &b, int m, int n, int k0, int ke, const float *A,
                                              int64_t lda, const float *B, int64_t ldb, int m0, int n0) {
    const int t = threadIdx.x;
#pragma unroll
    for (int q = 0; q < 8; ++q) {  // A: 64 k x 32 row groups
        const int idx = t + kCT * q;
        const int kk = idx >> 5, r = (idx & 31) * 4;
        const int gk = k0 + kk, gr = m0 + r;
        const int by = gk < ke ? grp_bytes(gr, m) : 0;
        cp_async16(&b.As[kk][r], by ? A + (int64_t)gk * lda + gr : A, by);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {  // B: 128 columns x 16 k groups
        const int idx = t + kCT * q;
        const int c = idx >> 4, kk = (idx & 15) * 4;
        const int gc = n0 + c, gk = k0 + kk;
        const int by = gc < n ? grp_bytes(gk, ke) : 0;
        cp_async16(&b.Bs[c][kk], by ? B + (int64_t)gc * ldb + gk : B, by);
    }
}

// MI = 4 (NJ = 4): the tile's live rows (columns) are its first 64 only, the
// caller guarantees m - m0 <= 64 (n - n0 <= 64), and the padding half is
// neither multiplied nor stored (the live elements' operations unchanged).
template <int MI = 8, int NJ = 8>
__device__ void gemm_tile_v(SmemGV &sv, int m, int n, int kb, int ke, float alpha, const float *__restrict__ A,
                            int64_t lda, const float *__restrict__ B, int64_t ldb, bool accumulate, float *C,
                            int64_t ldc, int m0, int n0, int skip = 0) {
    static_assert((MI == 4 || MI == 8) && (NJ == 4 || NJ == 8), "full or half tile sides");
    const int t = threadIdx.x;
    const int tx = t % 16, ty = t / 16;
    float(*Cs)[GBM + 4] = reinterpret_cast<float(*)[GBM + 4]>(&sv.buf[1]);
    const int nch = ke > kb ? (ke - kb + kNB - 1) / kNB : 0;
    const bool c_early = accumulate && nch <= 1;  // C shares buf[1] with the second slice
    __syncthreads();  // the caller's previous use of this memory is over
    if (nch > 0) gv_load_slice(sv.buf[0], m, n, kb, ke, A, lda, B, ldb, m0, n0);
    cp_async_commit();
    auto load_c = [&]() {
#pragma unroll
        for (int q = 0; q < 16; ++q) {  // 128 columns x 32 row groups
            const int idx = t + kCT * q;
            const int c = idx >> 5, r = (idx & 31) * 4;
            const int gc = n0 + c, gr = m0 + r;
            const int by = gc < n ? grp_bytes(gr, m) : 0;
            cp_async16(&Cs[c][r], by ? C + (int64_t)gc * ldc + gr : C, by);
        }
        cp_async_commit();
    };
    if (c_early) load_c();

    float acc[MI][NJ];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j] = 0.0f;

    for (int ch = 0; ch < nch; ++ch) {
        const int k0 = kb + ch * kNB;
        if (ch + 1 < nch) {
            gv_load_slice(sv.buf[(ch + 1) & 1], m, n, k0 + kNB, ke, A, lda, B, ldb, m0, n0);
            cp_async_commit();
            cp_async_wait<1>();  // slice ch has landed, ch + 1 may be in flight
        } else if (c_early) {
            cp_async_wait<1>();  // slice ch has landed, C may be in flight
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const SmemGVBuf &b = sv.buf[ch & 1];
        const int nk4 = (min(kNB, ke - k0) + 3) / 4;
#pragma unroll 1
        for (int k4 = 0; k4 < nk4; ++k4) {
            float4 bq[NJ];
#pragma unroll
            for (int j = 0; j < NJ; ++j)
                bq[j] = *reinterpret_cast<const float4 *>(&b.Bs[j < 4 ? ty * 4 + j : 64 + ty * 4 + (j - 4)][4 * k4]);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                float av[MI];
                {
                    const float4 a0 = *reinterpret_cast<const float4 *>(&b.As[4 * k4 + s][tx * 4]);
                    av[0] = a0.x;
                    av[1] = a0.y;
                    av[2] = a0.z;
                    av[3] = a0.w;
                }
                if constexpr (MI == 8) {
                    const float4 a1 = *reinterpret_cast<const float4 *>(&b.As[4 * k4 + s][64 + tx * 4]);
                    av[MI - 4] = a1.x;
                    av[MI - 3] = a1.y;
                    av[MI - 2] = a1.z;
                    av[MI - 1] = a1.w;
                }
                float bv[NJ];
#pragma unroll
                for (int j = 0; j < NJ; ++j) bv[j] = s == 0 ? bq[j].x : s == 1 ? bq[j].y : s == 2 ? bq[j].z : bq[j].w;
#pragma unroll
                for (int i = 0; i < MI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
            }
        }
        __syncthreads();  // buf[ch & 1] is refilled two slices on (or holds C)
    }
    if (accumulate) {
        if (!c_early) load_c();
        cp_async_wait<0>();
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int cl = j < 4 ? ty * 4 + j : 64 + ty * 4 + (j - 4);
        const int gc = n0 + cl;
        if (gc >= n) continue;
#pragma unroll
        for (int h = 0; h < MI / 4; ++h) {
            const int rl = h * 64 + tx * 4, gr = m0 + rl;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = acc[4 * h + e][j] * alpha;
            if (accumulate) {
                const float4 c4 = *reinterpret_cast<const float4 *>(&Cs[cl][rl]);
                v[0] += c4.x;
                v[1] += c4.y;
                v[2] += c4.z;
                v[3] += c4.w;
            }
            // element (rl + e, cl) of the tile is left alone when rl + e < skip and cl < skip
            float *dst = C + (int64_t)gc * ldc + gr;
            if (gr + 3 < m && (cl >= skip || rl >= skip)) {
                *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                continue;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (gr + e < m && !(cl < skip && rl + e < skip)) dst[e] = v[e];
        }
    }
    __syncthreads();  // shared memory is reused by the caller's next item
}

// ---- 64 x 64 SIMT GEMM tiles staged by cp.async ------------------------------
// The same sums as gemm_tile / gemm_tile_v (one fmaf chain over ascending k,
// times alpha, plus C), in tiles a quarter the size: the trailing updates of a
// diagonal block (rank 64, at most a few dozen 128 x 128 tiles for most
// steps) and the doubling levels of its inverses then spread over all CTAs
// instead of leaving most idle behind ~7 us tiles.  Operand slices (64 deep)
// and the C tile arrive by 16-byte cp.async, double-buffered across slices and
// across the CTA's tiles, so a tile's loads run under the previous one's
// products (4 x 4 outputs per thread, ~75 % of the FMA rate).  Alignment as
// gemm_tile_v_ok.
struct __align__(16) SmemT64Buf {
    float As[kNB][kNB];      // As[k][row]
    float Bs[kNB][kNB + 4];  // Bs[col][k]
    float Cs[kNB][kNB + 4];  // Cs[col][row]
};
struct __align__(16) SmemT64 {
    SmemT64Buf buf[2];
};

// One tile: C[m0:m0+64, n0:n0+64] (clipped to m x n) over k in [kb, ke).
struct Tile64 {
    const float *A, *B;
    float *C;
    int64_t lda, ldb, ldc;
    int m, n, m0, n0, kb, ke;
    float alpha;
};

__device__ __forceinline__ void t64_load_slice(SmemT64Buf &b, const Tile64 &w, int k0, bool with_c) {
    const int t = threadIdx.x;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int idx = t + kCT * q, i = idx >> 4, g = (idx & 15) * 4;
        {  // A: k = i, rows g..g+3
            const int gk = k0 + i, gr = w.m0 + g;
            const int by = gk < w.ke ? grp_bytes(gr, w.m) : 0;
            cp_async16(&b.As[i][g], by ? w.A + (int64_t)gk * w.lda + gr : w.A, by);
        }
        {  // B: column i, k = g..g+3
            const int gc = w.n0 + i, gk = k0 + g;
            const int by = gc < w.n ? grp_bytes(gk, w.ke) : 0;
            cp_async16(&b.Bs[i][g], by ? w.B + (int64_t)gc * w.ldb + gk : w.B, by);
        }
        if (with_c) {  // C: column i, rows g..g+3
            const int gc = w.n0 + i, gr = w.m0 + g;
            const int by = gc < w.n ? grp_bytes(gr, w.m) : 0;
            cp_async16(&b.Cs[i][g], by ? w.C + (int64_t)gc * w.ldc + gr : w.C, by);
        }
    }
}

// Tiles get(first), get(first + stride), ... < count.  get(i, w) fills w; every
// tile has at least one k.  ACC: C += ..., else C = ...
template <bool ACC, typename Get>
__device__ __forceinline__ void run_tiles64(SmemT64 &sm, int first, int stride, int count, Get get) {
    if (first >= count) return;
    const int t = threadIdx.x, tx = t % 16, ty = t / 16;
    Tile64 w, nw;
    get(first, w);
    nw = w;
    int it = first, k0 = w.kb, buf = 0;
    __syncthreads();  // the caller's previous use of this memory is over
    t64_load_slice(sm.buf[0], w, k0, ACC && k0 + kNB >= w.ke);
    cp_async_commit();
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    while (true) {
        const bool last = k0 + kNB >= w.ke;  // last slice of the tile
        int nk = k0 + kNB;
        bool more = true;
        if (last) {
            more = it + stride < count;
            if (more) {
                get(it + stride, nw);
                nk = nw.kb;
            }
        }
        if (more) {
            t64_load_slice(sm.buf[buf ^ 1], nw, nk, ACC && nk + kNB >= nw.ke);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const SmemT64Buf &b = sm.buf[buf];
        const int nk4 = (min(kNB, w.ke - k0) + 3) / 4;
#pragma unroll 4
        for (int k4 = 0; k4 < nk4; ++k4) {
            float4 bq[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) bq[j] = *reinterpret_cast<const float4 *>(&b.Bs[ty * 4 + j][4 * k4]);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float4 a4 = *reinterpret_cast<const float4 *>(&b.As[4 * k4 + s][tx * 4]);
                const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float bv = s == 0 ? bq[j].x : s == 1 ? bq[j].y : s == 2 ? bq[j].z : bq[j].w;
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][j] = fmaf(av[i], bv, acc[i][j]);
                }
            }
        }
        if (last) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int gc = w.n0 + ty * 4 + j, gr = w.m0 + tx * 4;
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = acc[i][j] * w.alpha;
                if (ACC) {
                    const float4 c4 = *reinterpret_cast<const float4 *>(&b.Cs[ty * 4 + j][tx * 4]);
                    v[0] += c4.x;
                    v[1] += c4.y;
                    v[2] += c4.z;
                    v[3] += c4.w;
                }
                if (gc < w.n) {
                    float *dst = w.C + (int64_t)gc * w.ldc + gr;
                    if (gr + 3 < w.m) {
                        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (gr + i < w.m) dst[i] = v[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i][j] = 0.0f;
            }
            it += stride;
        }
        __syncthreads();  // this buffer is refilled next
        if (!more) break;
        if (last) w = nw;
        k0 = nk;
        buf ^= 1;
    }
}

// ---- 64-wide triangular pieces, blocked by 16 columns --------------------------
// A block lives in shared memory as X[col][row] (pitch kNB + 4, or another that is 4 mod 32: 16-byte rows,
// conflict-free 16-byte accesses down a column of threads).  A shared-memory
// load returns at most 128 bytes per clock to the register file, broadcast or
// not, so a thread-per-row elimination that reads one 16-byte group per four
// FMAs is bound by those loads (a 64 x 64 strip solve: ~9.8 k cycles).  Here only
// 16 columns at a time are eliminated that way; the rest of the work is
// sub_gemm16, whose 4 x 4 outputs per thread use every loaded value four
// times.  Every element still receives one fmaf per pivot in ascending order.
typedef float (*Block64)[kNB + 4];

// C[c][r] -= sum_{k = k0 .. k0+15} A[k][r] * B[c][k] for r in [r0, r0 + nr), c in
// [c0, c0 + nc); nr and nc multiples of 4, a 4 x 4 tile per thread tid = 0, 1, ...
template <typename BA, typename BB, typename BC>
__device__ __forceinline__ void sub_gemm16(BA A, BB B, BC C, int k0, int r0, int nr, int c0, int nc, int tid) {
    const int tr = nr >> 2, tc = nc >> 2;
    const int rg = tid % tr, cg = tid / tr;
    if (tid < 0 || cg >= tc) return;
    const int r = r0 + 4 * rg, c = c0 + 4 * cg;
    float x[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float4 v = *reinterpret_cast<const float4 *>(&C[c + j][r]);
        x[j][0] = v.x;
        x[j][1] = v.y;
        x[j][2] = v.z;
        x[j][3] = v.w;
    }
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
        float4 bq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bq[j] = *reinterpret_cast<const float4 *>(&B[c + j][k0 + 4 * k4]);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const float4 a = *reinterpret_cast<const float4 *>(&A[k0 + 4 * k4 + s][r]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float bv = s == 0 ? bq[j].x : s == 1 ? bq[j].y : s == 2 ? bq[j].z : bq[j].w;
                x[j][0] = fmaf(-bv, a.x, x[j][0]);
                x[j][1] = fmaf(-bv, a.y, x[j][1]);
                x[j][2] = fmaf(-bv, a.z, x[j][2]);
                x[j][3] = fmaf(-bv, a.w, x[j][3]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(&C[c + j][r]) = make_float4(x[j][0], x[j][1], x[j][2], x[j][3]);
}

// The same in 2 x 2 tiles for 16 columns: a few dozen 4 x 4 tiles would leave most warps
// idle and run at one warp's issue rate.
__device__ __forceinline__ void sub_gemm16_narrow(Block64 A, Block64 B, Block64 C, int k0, int r0, int nr, int c0) {
    const int tr = nr >> 1;
    const int rg = threadIdx.x % tr, cg = threadIdx.x / tr;
    if (cg >= 8) return;
    const int r = r0 + 2 * rg, c = c0 + 2 * cg;
    float2 x0 = *reinterpret_cast<const float2 *>(&C[c][r]), x1 = *reinterpret_cast<const float2 *>(&C[c + 1][r]);
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
        const float4 b0 = *reinterpret_cast<const float4 *>(&B[c][k0 + 4 * k4]);
        const float4 b1 = *reinterpret_cast<const float4 *>(&B[c + 1][k0 + 4 * k4]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 a = *reinterpret_cast<const float2 *>(&A[k0 + 4 * k4 + e][r]);
            const float v0 = e == 0 ? b0.x : e == 1 ? b0.y : e == 2 ? b0.z : b0.w;
            const float v1 = e == 0 ? b1.x : e == 1 ? b1.y : e == 2 ? b1.z : b1.w;
            x0.x = fmaf(-v0, a.x, x0.x);
            x0.y = fmaf(-v0, a.y, x0.y);
            x1.x = fmaf(-v1, a.x, x1.x);
            x1.y = fmaf(-v1, a.y, x1.y);
        }
    }
    *reinterpret_cast<float2 *>(&C[c][r]) = x0;
    *reinterpret_cast<float2 *>(&C[c + 1][r]) = x1;
}

// Rows k0 .. k0+15 of column X[c]: x_r -= l(r, k) x_k for r > k, L the unit lower
// part of T's diagonal block at k0.
__device__ __forceinline__ void sub_solve_lower(Block64 T, float *col, int k0) {
    float u[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 v = *reinterpret_cast<const float4 *>(col + k0 + 4 * q);
        u[4 * q + 0] = v.x;
        u[4 * q + 1] = v.y;
        u[4 * q + 2] = v.z;
        u[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < 15; ++k) {
        const float uk = u[k];
#pragma unroll
        for (int r4 = (k + 1) / 4; r4 < 4; ++r4) {
            const float4 l = *reinterpret_cast<const float4 *>(&T[k0 + k][k0 + 4 * r4]);
            if (4 * r4 + 0 > k) u[4 * r4 + 0] = fmaf(-l.x, uk, u[4 * r4 + 0]);
            if (4 * r4 + 1 > k) u[4 * r4 + 1] = fmaf(-l.y, uk, u[4 * r4 + 1]);
            if (4 * r4 + 2 > k) u[4 * r4 + 2] = fmaf(-l.z, uk, u[4 * r4 + 2]);
            if (4 * r4 + 3 > k) u[4 * r4 + 3] = fmaf(-l.w, uk, u[4 * r4 + 3]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4 *>(col + k0 + 4 * q) = make_float4(u[4 * q], u[4 * q + 1], u[4 * q + 2], u[4 * q + 3]);
}

// Columns k0 .. k0+15 of row r of X: x_c = (x_c - sum_{k<c} x_k u(k, c)) / u(c, c), U the
// upper part of T's diagonal block at k0, dinv its reciprocal diagonal.
template <typename BX>
__device__ __forceinline__ void sub_solve_upper(Block64 T, const float *dinv, BX X, int r, int k0) {
    float x[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) x[c] = X[k0 + c][r];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
#pragma unroll
        for (int k4 = 0; 4 * k4 < c; ++k4) {
            const float4 u = *reinterpret_cast<const float4 *>(&T[k0 + c][k0 + 4 * k4]);
            x[c] = fmaf(-u.x, x[4 * k4], x[c]);
            if (4 * k4 + 1 < c) x[c] = fmaf(-u.y, x[4 * k4 + 1], x[c]);
            if (4 * k4 + 2 < c) x[c] = fmaf(-u.z, x[4 * k4 + 2], x[c]);
            if (4 * k4 + 3 < c) x[c] = fmaf(-u.w, x[4 * k4 + 3], x[c]);
        }
        x[c] *= dinv[k0 + c];
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) X[k0 + c][r] = x[c];
}

// X (nr rows x 64, nr <= 64 and a multiple of 4, in shared memory) <- X U^{-1}, and X (64 x nc
// columns, likewise) <- L^{-1} X, with the triangles of T.  All threads of the CTA.
template <typename BX>
__device__ __forceinline__ void block_solve_upper(Block64 T, const float *dinv, BX X, int nr) {
#pragma unroll 1
    for (int k0 = 0; k0 < kNB; k0 += 16) {
        if (threadIdx.x < nr) sub_solve_upper(T, dinv, X, threadIdx.x, k0);
        __syncthreads();
        if (k0 + 16 < kNB) {
            sub_gemm16(X, T, X, k0, 0, nr, k0 + 16, kNB - 16 - k0, threadIdx.x);
            __syncthreads();
        }
    }
}
template <typename BX>
__device__ __forceinline__ void block_solve_lower(Block64 T, BX X, int nc) {
#pragma unroll 1
    for (int k0 = 0; k0 < kNB; k0 += 16) {
        if (threadIdx.x < nc) sub_solve_lower(T, &X[threadIdx.x][0], k0);
        __syncthreads();
        if (k0 + 16 < kNB) {
            sub_gemm16(T, X, X, k0, k0 + 16, kNB - 16 - k0, 0, nc, threadIdx.x);
            __syncthreads();
        }
    }
}

// A block D (nr x nc <= 64 x 64; zero, or the identity when `unit`, elsewhere)
// from global memory into T[col][row], through L2: 16-byte cp.async when the
// addresses allow (not waited for here), else through registers.
__device__ __forceinline__ void request_block(Block64 T, const float *D, int64_t ld, int nr, int nc, bool unit) {
    if (aligned16(D) && (ld & 3) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int idx = threadIdx.x + kCT * q;
            const int c = idx >> 4, r = (idx & 15) * 4;
            float *dst = &T[c][r];
            if (c < nc && r + 4 <= nr) {
                cp_async16(dst, D + (int64_t)c * ld + r, 16);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    dst[e] = c < nc && r + e < nr ? __ldcg(D + (int64_t)c * ld + r + e) : (unit && c == r + e) ? 1.0f : 0.0f;
            }
        }
    } else {
        float v[16];
        load_block64(v, D, ld, nr, nc);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int idx = threadIdx.x + kCT * q;
            const int c = idx / kNB, r = idx % kNB;
            T[c][r] = c < nc && r < nr ? v[q] : (unit && c == r) ? 1.0f : 0.0f;
        }
    }
}

// ... and back (rows < nr, columns < nc).
__device__ __forceinline__ void store_block(Block64 T, float *D, int64_t ld, int nr, int nc) {
    if (aligned16(D) && (ld & 3) == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int idx = threadIdx.x + kCT * q;
            const int c = idx >> 4, r = (idx & 15) * 4;
            if (c >= nc) continue;
            if (r + 4 <= nr) {
                *reinterpret_cast<float4 *>(D + (int64_t)c * ld + r) = *reinterpret_cast<const float4 *>(&T[c][r]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (r + e < nr) D[(int64_t)c * ld + r + e] = T[c][r + e];
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int idx = threadIdx.x + kCT * q;
            const int c = idx / kNB, r = idx % kNB;
            if (c < nc && r < nr) D[(int64_t)c * ld + r] = T[c][r];
        }
    }
}

// ---- 64 x 64 no-pivot LU of D (nb <= 64) -------------------------------------
// sgetrf_nopiv_naive order (sgetrf_nopiv.cpp:27-61): scale by the reciprocal
// pivot, then the rank-1 update; every element receives its fmaf updates one
// by one in ascending pivot order, whatever the blocking, so the factors are
// those of the unblocked loop bit for bit.
//
// What bounds it is the chain of 64 pivots.  In blocks of 16 columns (the block
// in shared memory, T = t[col][row]):
//  * panel: warp w holds the 16 rows of the diagonal block in lanes 0..15 and
//    16 of the rows below in lanes 16..31, 16 columns each in registers: the
//    L panel is solved along with the diagonal block, which every warp
//    factors for itself (no exchange between warps).  Four pivots at a
//    time: the four pivot rows go through shared memory to every lane, and
//    each lane eliminates the 4 x 4 block and the rest of those rows for
//    itself, so the chain meets one exchange per four pivots (a shuffle per
//    pivot and column took ~340 cycles per pivot);
//  * then the 16 rows of U by sub_solve_lower and the next panel's columns by
//    sub_gemm16_narrow; the columns beyond it wait for the warps that the next
//    panel leaves idle.
// Rows and columns past nb are those of the identity.
// The 16 pivots of one panel on this warp's 32 rows (a: this lane's row).  kSafe:
// reciprocals of pivots outside the fast form's range (subnormal, or 2^126 and
// above).  Returns -1 or the first zero / non-finite pivot; extreme: set when
// the fast form met a pivot outside its range (the caller runs it again).
template <bool kSafe>
__device__ __forceinline__ int getrf64_panel(float (&a)[16], float (*rows)[4][16], bool &extreme) {
    const int ln = threadIdx.x & 31;
    int bad = -1;
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
        const int kk = 4 * k4;
        float(*p)[16] = rows[k4];
        if (ln >= kk && ln < kk + 4) {
#pragma unroll
            for (int q = k4; q < 4; ++q)
                *reinterpret_cast<float4 *>(&p[ln - kk][4 * q]) = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
        }
        __syncwarp();
        float r[4][16];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = k4; q < 4; ++q) {
                const float4 v = *reinterpret_cast<const float4 *>(&p[i][4 * q]);
                r[i][4 * q + 0] = v.x;
                r[i][4 * q + 1] = v.y;
                r[i][4 * q + 2] = v.z;
                r[i][4 * q + 3] = v.w;
            }
        float rp[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float pv = r[i][kk + i];
            rp[i] = kSafe ? rcp_rn_f32(pv) : rcp_rn_f32_fast(pv);
            if (!kSafe) extreme |= !rcp_fast_range(pv);
            const unsigned au = __float_as_uint(pv) & 0x7fffffffu;
            if (bad < 0 && au - 1u >= 0x7f7fffffu) bad = kk + i;
#pragma unroll
            for (int j = i + 1; j < 4; ++j) {
                const float l = r[j][kk + i] * rp[i];
#pragma unroll
                for (int c = kk + i + 1; c < 16; ++c) r[j][c] = fmaf(-r[i][c], l, r[j][c]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool act = ln > kk + i;
            const float l = a[kk + i] * rp[i];
            a[kk + i] = act ? l : a[kk + i];
#pragma unroll
            for (int c = kk + i + 1; c < 16; ++c) {
                const float v = fmaf(-r[i][c], l, a[c]);
                a[c] = act ? v : a[c];
            }
        }
    }
    return bad;
}

// in_smem: the block to factor is already in sm.t.t[col][row] (look_ahead), not
// read from D; either way the factors are written to D.
__device__ __noinline__ void getrf64(Smem &sm, int nb, float *D, int64_t lda, DevStatus *dst, int pivot_base,
                                     bool in_smem = false) {
    Block64 T = sm.t.t;  // T[c][r]: the block, written out at the end
    const int warp = threadIdx.x >> 5, ln = threadIdx.x & 31;
    if (!in_smem) {
        request_block(T, D, lda, nb, nb, true);
        cp_async_commit();
        cp_async_wait<0>();
    } else if (threadIdx.x >= nb && threadIdx.x < kNB) {
        T[threadIdx.x][threadIdx.x] = 1.0f;
    }
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0; k0 < kNB; k0 += 16) {
        const bool on = warp == 0 || 16 * warp + 16 < kNB - k0;
        // lanes 16..31: 16 rows below the diagonal block (the last panel has
        // none: those lanes follow the diagonal block's own rows)
        const bool below = k0 + 16 < kNB;
        const int row = k0 + (ln < 16 ? ln : below ? ln + 16 * warp : ln - 16);
        float a[16];
        int bad = -1;
        if (on) {
            bool extreme = false;
#pragma unroll
            for (int c = 0; c < 16; ++c) a[c] = T[k0 + c][row];
            bad = getrf64_panel<false>(a, sm.t.rows.r[warp], extreme);
            if (extreme) {  // the same in every warp: T still holds the panel
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 16; ++c) a[c] = T[k0 + c][row];
                bad = getrf64_panel<true>(a, sm.t.rows.r[warp], extreme);
            }
        } else if (k0 > 0 && below) {
            // the columns beyond this panel get the last panel's update from the
            // warps that have no part in this one
            sub_gemm16(T, T, T, k0 - 16, k0, kNB - k0, k0 + 16, kNB - 16 - k0, (int)threadIdx.x - 96);
        }
        __syncthreads();  // every warp has read the panel
        if (on && (ln >= 16 ? below : warp == 0)) {
#pragma unroll
            for (int c = 0; c < 16; ++c) T[k0 + c][row] = a[c];
        }
        if (warp == 0 && ln == 0 && bad >= 0 && k0 + bad < nb) report(dst, MXP_ZERO_PIVOT, pivot_base + k0 + bad + 1, 0);
        __syncthreads();
        if (!below) break;
        const int R = kNB - 16 - k0;
        if (threadIdx.x < R) sub_solve_lower(T, &T[k0 + 16 + threadIdx.x][0], k0);
        __syncthreads();
        sub_gemm16_narrow(T, T, T, k0, k0 + 16, R, k0 + 16);  // the next panel's columns
        __syncthreads();
    }
    store_block(T, D, lda, nb, nb);
    __syncthreads();
}

// Shared memory of the strip solves and of the look-ahead: the diagonal block (at
// the place of Smem's t, where getrf64 expects it) and two more blocks.
struct __align__(16) SmemStrip {
    float t[kNB][kNB + 4], x[kNB][kNB + 4], y[kNB][kNB + 4];
    float dinv[kNB];
};

// Look-ahead: T (in shared memory, for getrf64(..., in_smem = true)) = C - L U,
// the next diagonal block (nb x nb) with the strips' first 64 rows and columns.
// 8 x 4 outputs per thread.
__device__ __noinline__ void look_ahead(SmemStrip &s, int nb, const float *L, const float *U, const float *C,
                                        int64_t ld) {
    request_block(s.x, L, ld, nb, kNB, false);
    request_block(s.y, U, ld, kNB, nb, false);
    request_block(s.t, C, ld, nb, nb, false);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // two halves of k, 128 threads each, then one sum: eight warps hide the
    // operand loads that bound it
    const int id = threadIdx.x & 127, kh = threadIdx.x >> 7;
    const int r = 4 * (id % 8), c = 4 * (id / 8);
    float acc[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[j][i] = 0.0f;
#pragma unroll 4
    for (int k4 = kh * (kNB / 8); k4 < (kh + 1) * (kNB / 8); ++k4) {
        float4 bq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bq[j] = *reinterpret_cast<const float4 *>(&s.y[c + j][4 * k4]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float4 a0 = *reinterpret_cast<const float4 *>(&s.x[4 * k4 + e][r]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&s.x[4 * k4 + e][32 + r]);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float bv = e == 0 ? bq[j].x : e == 1 ? bq[j].y : e == 2 ? bq[j].z : bq[j].w;
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[j][i] = fmaf(av[i], bv, acc[j][i]);
            }
        }
    }
    __syncthreads();  // the operands are read: each half's sums of the other's rows go to x
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(&s.x[c + j][32 * (1 - kh) + r]) =
            make_float4(kh ? acc[j][0] : acc[j][4], kh ? acc[j][1] : acc[j][5], kh ? acc[j][2] : acc[j][6],
                        kh ? acc[j][3] : acc[j][7]);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float4 *t = reinterpret_cast<float4 *>(&s.t[c + j][32 * kh + r]);
        const float4 o = *reinterpret_cast<const float4 *>(&s.x[c + j][32 * kh + r]), v = *t;
        const float m0 = kh ? acc[j][4] : acc[j][0], m1 = kh ? acc[j][5] : acc[j][1];
        const float m2 = kh ? acc[j][6] : acc[j][2], m3 = kh ? acc[j][7] : acc[j][3];
        *t = make_float4(v.x - (m0 + o.x), v.y - (m1 + o.y), v.z - (m2 + o.z), v.w - (m3 + o.w));
    }
    __syncthreads();
}

// Strip items of kStripW rows (L strip, X U = B) or columns (U strip, L X = B):
// items 0 .. lit-1 are the L strip's, the rest the U strip's.  rem: rows of the
// L strip (columns of the U strip); ld of both.
constexpr int kStripW = 32;
__device__ __noinline__ void strip_items(SmemStrip &s, int first, int stride, int lit, int rem, const float *D,
                                         float *Ls, float *Us, int64_t ld) {
    for (int it = first; it < 2 * lit; it += stride) {
        const bool left = it < lit;
        const int o = (left ? it : it - lit) * kStripW, w = min(kStripW, rem - o);
        float *B = left ? Ls + o : Us + (int64_t)o * ld;
        if (it == first) request_block(s.t, D, ld, kNB, kNB, false);
        request_block(s.x, B, ld, left ? w : kNB, left ? kNB : w, false);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        if (left) {
            if (threadIdx.x < kNB) s.dinv[threadIdx.x] = 1.0f / s.t[threadIdx.x][threadIdx.x];
            __syncthreads();
            block_solve_upper(s.t, s.dinv, s.x, kStripW);
        } else {
            block_solve_lower(s.t, s.x, kStripW);
        }
        store_block(s.x, B, ld, left ? w : kNB, left ? kNB : w);
        __syncthreads();
    }
}

// D (nb x nb, factored) into shared memory: t[col][row], the skewed rows of U
// and columns of L the rotated strip solves read (us, ls), and the reciprocal
// diagonal.
__device__ void load_tri(Smem &sm, int nb, const float *D, int64_t lda) {
    float v[16];
    load_block64(v, D, lda, nb, nb);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int idx = threadIdx.x + kCT * q;
        sm.t.t[idx / kNB][idx % kNB] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int idx = threadIdx.x + kCT * q;
        const int k = idx / kNB, c = idx % kNB, j = k + 1 + c;
        sm.t.us[k][c] = j < nb ? sm.t.t[j][k] : 0.0f;
        sm.t.ls[k][c] = j < nb ? sm.t.t[k][j] : 0.0f;
    }
    if (threadIdx.x < nb) sm.t.dinv[threadIdx.x] = 1.0f / sm.t.t[threadIdx.x][threadIdx.x];
    __syncthreads();
}

// L strip rows [r0, r0 + rows) of B (m x nb), rows <= kCT: X = B U^{-1}, U =
// upper part of the diagonal block (load_tri).  Right-looking, thread per row
// (x_k final, then x_c -= u_kc x_k for c > k): per element the same
// operations in the same order as the dot-product form; the row rotates
// (rot_axpy) so the pivot loop stays rolled, and x_k is stored as soon as it
// is final.
template <int W>
__device__ __forceinline__ void trsm_rows_phase(Smem &sm, float (&x)[kNB], int k0, int k1, float *B, int64_t ldb,
                                                int i) {
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const float xk = x[0] * sm.t.dinv[k];
        B[(int64_t)k * ldb + i] = xk;
        rot_axpy<W>(x, &sm.t.us[k][0], xk);
    }
}

// The row of B this thread solves (zero when it has none), and the solve of a
// row loaded that way: split so a caller can issue the loads before load_tri.
__device__ __forceinline__ void trsm_rows_load(float (&x)[kNB], int m, int nb, const float *B, int64_t ldb, int r0,
                                               int rows) {
    const int i = r0 + threadIdx.x;
    const bool act = threadIdx.x < rows && i < m;
#pragma unroll
    for (int c = 0; c < kNB; ++c) x[c] = (act && c < nb) ? __ldcg(B + (int64_t)c * ldb + i) : 0.0f;
}
__device__ __forceinline__ void trsm_rows_solve(Smem &sm, float (&x)[kNB], int m, int nb, float *B, int64_t ldb,
                                                int r0, int rows) {
    const int i = r0 + threadIdx.x;
    if (threadIdx.x >= rows || i >= m) return;
    trsm_rows_phase<64>(sm, x, 0, min(nb, 16), B, ldb, i);
    trsm_rows_phase<48>(sm, x, 16, min(nb, 32), B, ldb, i);
    trsm_rows_phase<32>(sm, x, 32, min(nb, 48), B, ldb, i);
    trsm_rows_phase<16>(sm, x, 48, nb, B, ldb, i);
}

__device__ void trsm_rows(Smem &sm, int m, int nb, float *B, int64_t ldb, int r0, int rows = kCT) {
    float x[kNB];
    trsm_rows_load(x, m, nb, B, ldb, r0, rows);
    trsm_rows_solve(sm, x, m, nb, B, ldb, r0, rows);
}

// One column of X = L^{-1} B (L unit lower, load_tri) in registers: x_r -=
// l_rk x_k for r > k, rotated; x_k goes to out[k] as soon as it is final.
template <int W>
__device__ __forceinline__ void trsm_col_phase(Smem &sm, float (&x)[kNB], int k0, int k1, float *out) {
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const float xk = x[0];
        out[k] = xk;
        rot_axpy<W>(x, &sm.t.ls[k][0], xk);
    }
}

__device__ __forceinline__ void trsm_col(Smem &sm, float (&x)[kNB], int nb, float *out) {
    trsm_col_phase<64>(sm, x, 0, min(nb, 16), out);
    trsm_col_phase<48>(sm, x, 16, min(nb, 32), out);
    trsm_col_phase<32>(sm, x, 32, min(nb, 48), out);
    trsm_col_phase<16>(sm, x, 48, nb, out);
}

// Inverse of the 64 x 64 diagonal block `blk` of an upper non-unit (upper = true)
// or unit-lower triangle: the strip solves with the identity as right-hand
// side (a fully unrolled substitution spent ~30 us per block fetching
// instructions).
__device__ __noinline__ void inv_diag_block(SmemStrip &s, int n, const float *T, int64_t ldt, float *X, int64_t ldx,
                                            int blk, bool upper) {
    const int r0 = blk * kNB;
    const int nb = min(kNB, n - r0);
    request_block(s.t, T + r0 + (int64_t)r0 * ldt, ldt, nb, nb, true);
    request_block(s.x, nullptr, 0, 0, 0, true);  // the identity
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (upper) {
        if (threadIdx.x < kNB) s.dinv[threadIdx.x] = 1.0f / s.t[threadIdx.x][threadIdx.x];
        __syncthreads();
        block_solve_upper(s.t, s.dinv, s.x, kNB);
    } else {
        block_solve_lower(s.t, s.x, kNB);
    }
    store_block(s.x, X + r0 + (int64_t)r0 * ldx, ldx, nb, nb);
    __syncthreads();
}

// One batched GEMM of an inverse level.  tri: which operand is triangular, so
// its zero half is skipped along K: 1 A upper, 2 A lower, 3 B upper, 4 B lower.
struct Job {
    int m, n, K, batch, tri;
    float alpha;
    const float *A;
    int64_t lda, sA;
    const float *B;
    int64_t ldb, sB;
    float *C;
    int64_t ldc, sC;
};

// All tiles of the jobs, 64 x 64 (run_tiles64) when every job's operands allow
// 16-byte copies, else 128 x 128 (gemm_tile).  st: memory for run_tiles64.
__device__ void run_jobs(Smem &sm, const Job *jobs, int njobs, int cta, int ncta, SmemT64 &st) {
    bool vec = true;
    for (int q = 0; q < njobs; ++q) {
        const Job &J = jobs[q];
        vec = vec && gemm_tile_v_ok(J.A, J.lda, J.B, J.ldb, J.C, J.ldc, 0) && ((J.sA | J.sB | J.sC) & 3) == 0;
    }
    const int TS = vec ? kNB : GBM;
    int tiles[4] = {0, 0, 0, 0}, total = 0;
    for (int q = 0; q < njobs; ++q) {
        tiles[q] = ((jobs[q].m + TS - 1) / TS) * ((jobs[q].n + TS - 1) / TS) * jobs[q].batch;
        total += tiles[q];
    }
    auto get = [&](int it, Tile64 &w) {
        int q = 0, r = it;
        while (r >= tiles[q]) r -= tiles[q++];
        const Job &J = jobs[q];
        const int tm = (J.m + TS - 1) / TS, tn = (J.n + TS - 1) / TS;
        const int z = r / (tm * tn);
        const int rt = r % (tm * tn);
        w.m0 = (rt % tm) * TS;
        w.n0 = (rt / tm) * TS;
        w.kb = 0;
        w.ke = J.K;
        if (J.tri == 1) w.kb = w.m0;
        if (J.tri == 2) w.ke = min(J.K, w.m0 + TS);
        if (J.tri == 3) w.ke = min(J.K, w.n0 + TS);
        if (J.tri == 4) w.kb = w.n0;
        w.m = J.m;
        w.n = J.n;
        w.A = J.A + J.sA * z;
        w.B = J.B + J.sB * z;
        w.C = J.C + J.sC * z;
        w.lda = J.lda;
        w.ldb = J.ldb;
        w.ldc = J.ldc;
        w.alpha = J.alpha;
    };
    if (vec) {
        run_tiles64<false>(st, cta, ncta, total, get);
        return;
    }
    for (int it = cta; it < total; it += ncta) {
        Tile64 w;
        get(it, w);
        gemm_tile(sm, w.m, w.n, w.kb, w.ke, w.alpha, w.A, w.lda, w.B, w.ldb, false, w.C, w.ldc, w.m0, w.n0);
    }
}

// inv(U) -> XU and inv(L) -> XL (unit lower) of the factored n x n block A, by
// recursive doubling: 64 x 64 diagonal blocks first, then for adjacent
// S-blocks the off-diagonal block of the inverse is -inv(A) B inv(C), two GEMM
// phases per level with both triangles in the same phases and the zero half of
// every triangular operand skipped along K.  Work items are spread over
// (cta, ncta); sync(where) separates the phases (a grid barrier across CTAs or
// __syncthreads in a single CTA) and returns false to stop.  tmpU / tmpL hold
// n*n/2 + 64 n floats each.  s_stop > 0: stop before the level that joins
// blocks of size s_stop (the caller finishes those levels elsewhere).
template <typename Sync>
__device__ bool tri_inverses(Smem &sm, int n, const float *A, int64_t lda, float *XU, float *XL, int64_t ldx,
                             float *tmpU, float *tmpL, int cta, int G, Sync sync, int s_stop, SmemT64 &st, SmemStrip &ss) {
    const int nsteps = (n + kNB - 1) / kNB;
    // invert the diagonal 64 x 64 blocks and zero the opposite block-triangle
    const int nblk = nsteps;
    for (int it = cta; it < 2 * nblk; it += G)
        inv_diag_block(ss, n, A, lda, it < nblk ? XU : XL, ldx, it % nblk, it < nblk);
    {   // zero the opposite block-triangles: a column per warp, rows by lanes
        // (a flat index split by 64-bit division cost ~30 us per 2560 block)
        constexpr int W = kCT / 32;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        for (int c = cta * W + warp; c < n; c += G * W) {
            const int cb = c / kNB;
            float *xu = XU + (int64_t)c * ldx, *xl = XL + (int64_t)c * ldx;
            for (int r = lane; r < n; r += 32) {
                const int rb = r / kNB;
                if (rb > cb) xu[r] = 0.0f;
                if (rb < cb) xl[r] = 0.0f;
            }
        }
    }
    if (!sync(23)) return false;

    const float *U = A, *L = A;
    const int64_t ldu = lda, ldl = lda;
    for (int S = kNB; S < n && (s_stop <= 0 || S < s_stop); S *= 2) {
        const int np = n / (2 * S);
        const int rem = n - np * 2 * S;
        const int c = rem - S;  // ragged last pair (when > 0)
        const int64_t r0 = (int64_t)np * 2 * S;
        const int64_t stepX = 2 * (int64_t)S * (1 + ldx), stepA = 2 * (int64_t)S * (1 + lda);
        const int64_t SS = (int64_t)S * S;
        Job jb[4];
        int nj = 0;
        // phase a:  T_U = U12 inv(U22);  T_L = L21 inv(L11)
        if (np > 0) {
            jb[nj++] = Job{S, S, S, np, 3, 1.0f, U + (int64_t)S * ldu, ldu, stepA, XU + S + (int64_t)S * ldx,
                           ldx, stepX, tmpU, S, SS};
            jb[nj++] = Job{S, S, S, np, 4, 1.0f, L + S, ldl, stepA, XL, ldx, stepX, tmpL, S, SS};
        }
        if (c > 0) {
            jb[nj++] = Job{S, c, c, 1, 3, 1.0f, U + r0 + (r0 + S) * ldu, ldu, 0,
                           XU + (r0 + S) + (r0 + S) * ldx, ldx, 0, tmpU + np * SS, S, 0};
            jb[nj++] = Job{c, S, S, 1, 4, 1.0f, L + (r0 + S) + r0 * ldl, ldl, 0, XL + r0 + r0 * ldx, ldx, 0,
                           tmpL + np * SS, c, 0};
        }
        run_jobs(sm, jb, nj, cta, G, st);
        if (!sync(24)) return false;
        // phase b:  X12 = -inv(U11) T_U;  X21 = -inv(L22) T_L
        nj = 0;
        if (np > 0) {
            jb[nj++] = Job{S, S, S, np, 1, -1.0f, XU, ldx, stepX, tmpU, S, SS, XU + (int64_t)S * ldx, ldx, stepX};
            jb[nj++] = Job{S, S, S, np, 2, -1.0f, XL + S + (int64_t)S * ldx, ldx, stepX, tmpL, S, SS, XL + S,
                           ldx, stepX};
        }
        if (c > 0) {
            jb[nj++] = Job{S, c, S, 1, 1, -1.0f, XU + r0 + r0 * ldx, ldx, 0, tmpU + np * SS, S, 0,
                           XU + r0 + (r0 + S) * ldx, ldx, 0};
            jb[nj++] = Job{c, S, c, 1, 2, -1.0f, XL + (r0 + S) + (r0 + S) * ldx, ldx, 0, tmpL + np * SS, c, 0,
                           XL + (r0 + S) + r0 * ldx, ldx, 0};
        }
        run_jobs(sm, jb, nj, cta, G, st);
        if (!sync(25)) return false;
    }
    return true;
}

}  // namespace
}  // namespace dt
}  // namespace mxp
