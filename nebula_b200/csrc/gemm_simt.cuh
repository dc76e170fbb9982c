// CUDA-core fp32 contraction: GEMM, implicit-GEMM convolution (NB_MATH_FP32, and operands the tensor-core kernel
// cannot take) and the operator library's _gemm_.
//
// D[M,N] = A[M,K] * B[N,K]^T with A an implicit im2col view (row = output pixel, column = (kh,kw,c)) gathered through
// arbitrary element strides and B any strided matrix.  Exact fp32 products, fp32 FMA accumulation.  Replaces the same
// reference code as the tensor-core kernel (models/layers/convolutional_layer.cu:47-70, connected_layer.cu:21-38)
// and common/gemm.cu:38-153.
//
// Bound by: the FMA pipes (128 lanes x 2 flop per cycle and SM) for large products, the weight stream for few rows.
//   * Both operands lie in shared memory with K contiguous (rows of 16 floats, stride 20: eight rows of a 128-bit
//     read fall into 32 different banks), so the copies are cp.async straight from global memory in the operands'
//     own order (16 bytes each where alignment allows, else 4) and nothing is transposed by the threads.
//   * Copies advance their addresses from block to block and from tap to tap; a tap begins with a comparison per row (64-bit
//     products per copy and block were four tenths of all instructions, many of them on the FMA pipe).
//   * A thread owns RM x RN outputs and multiplies with packed fma.rn.f32x2 along K: a 128-bit read delivers two
//     packed pairs, the accumulator pair holds the even and the odd columns' sums.  At 8 x 8 outputs a k-quad is 16
//     reads for 128 packed FMAs; the read port is idle three quarters of the time.
//   * A long contraction with few output tiles is cut into S = 2..8 ranges of K, one CTA each, joined as a cluster:
//     the partial tiles stay in shared memory, every CTA adds a slice of the tile over the cluster's shared memory in
//     rank order and writes it.  No workspace, no second launch, no atomics.  In layers S depends on N, K and the pixels of
//     ONE image, never on the batch, so a batch and its slices add in the same order; in _gemm_ it depends on M as well.
// Measured against the 64 x 64 tile with scalar loads and two barriers per 16 columns (and a 16 x 16 tile for _gemm_)
// before it: AlexNet b4 in fp32 2938 -> 454 us (its connected layers by gemm_rows_kernel), 256 x 1024 x 1024 _gemm_ + bias + relu
// 183 -> 27 us.
//
// This header: the kernel and what launches must know of it.  gemm_simt_kernels.cu compiles it once per pair of copy modes (a
// module each: the first kernel of all 36 in one took 15 ms to load), gemm_simt.cu chooses and launches.
#pragma once
#include <cooperative_groups.h>

#include "device_math.cuh"
#include "nb_internal.h"

namespace nb {

namespace cg = cooperative_groups;

constexpr int BK = 16;          // K columns per stage
constexpr int LDK = 20;         // row stride in shared memory

// how an operand's tile is copied: 16 bytes along K; one float at a time, lanes along K; one float, lanes along the rows
enum CopyMode { VEC_K = 0, ONE_K = 1, ONE_ROW = 2 };

struct SimtParams {
    const float *a, *b;
    ConvGeom g;                 // A: row = (image, oh, ow); a plain matrix is one image of height 1
    long b_tap, b_row, b_col;   // element strides of B
    int M, N, Kc, ksize_w;
    int c_blocks, k_blocks, kb_per_split;       // 16-column blocks per tap and in all; blocks per cluster rank
    int n_tiles;
    const float *scale, *shift, *addend;
    long ld_addend;
    int act, round_out, addend_post;
    int blas;                   // y = alpha * acc + beta * y instead of the layer epilogue
    float alpha, beta;
    float *y;
    long ldy;
};

__device__ __forceinline__ void ffma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
// src_bytes 0: nothing is read and the destination becomes zero
__device__ __forceinline__ void cp_async16(uint32_t dst, const float *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// Which (row, column) of a ROWS x 16 tile copy i of this thread moves.
template <int ROWS, int THREADS, int MODE>
struct TileMap {
    static constexpr int PER_ROW = MODE == VEC_K ? BK / 4 : BK;
    static constexpr int TOTAL = ROWS * PER_ROW;
    static constexpr int COPIES = (TOTAL + THREADS - 1) / THREADS;
    static constexpr int ROW_SLOTS = MODE == ONE_ROW ? 1 : COPIES;      // different rows a thread touches
    // copy i lies this many floats behind copy 0 in shared memory
    static constexpr int STEP = MODE == ONE_ROW ? THREADS / ROWS : THREADS / PER_ROW * LDK;
    __device__ static bool active(int tid, int i) { return TOTAL % THREADS == 0 || tid + i * THREADS < TOTAL; }
    __device__ static int row(int tid, int i) {
        if (MODE == ONE_ROW) return tid % ROWS;         // THREADS is a multiple of ROWS
        return (tid + i * THREADS) / PER_ROW;
    }
    __device__ static int col(int tid, int i) {
        if (MODE == ONE_ROW) return (tid + i * THREADS) / ROWS;
        return (tid % PER_ROW) * (MODE == VEC_K ? 4 : 1);
    }
};

template <int BM, int BN, int RM, int RN, int STAGES>
struct Tile {
    static constexpr int TX = BN / RN, TY = BM / RM, THREADS = TX * TY;
    static constexpr int STAGE_FLOATS = (BM + BN) * LDK;
    static constexpr int RED_LD = BN + 8;       // four rows of eight lanes fall into 32 different banks
    static constexpr int SMEM_FLOATS = STAGES * STAGE_FLOATS > BM * RED_LD ? STAGES * STAGE_FLOATS : BM * RED_LD;
};

__device__ __forceinline__ void store_out(const SimtParams &p, long m, int n, float x) {
    if (p.blas) {
        float *c = p.y + m * p.ldy + n;
        *c = p.alpha * x + (p.beta == 0.0f ? 0.0f : p.beta * *c);
        return;
    }
    if (p.scale) x *= p.scale[n];
    if (p.shift) x += p.shift[n];
    if (p.addend && !p.addend_post) x += p.addend[m * p.ld_addend + n];
    x = apply_activation_fast(x, p.act);
    if (p.addend && p.addend_post) x += p.addend[m * p.ld_addend + n];
    p.y[m * p.ldy + n] = p.round_out ? round_tf32(x) : x;
}

template <int BM, int BN, int RM, int RN, int STAGES, int AMODE, int BMODE>
__global__ void __launch_bounds__((BM / RM) * (BN / RN)) gemm_fp32_simt_kernel(const SimtParams p) {
    using T = Tile<BM, BN, RM, RN, STAGES>;
    using MA = TileMap<BM, T::THREADS, AMODE>;
    using MB = TileMap<BN, T::THREADS, BMODE>;
    extern __shared__ __align__(16) float smem[];
    grid_dependents_start();
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    // a warp's lanes form 4 rows x 8 columns of threads
    const int tx = (warp % (T::TX / 8)) * 8 + (lane & 7), ty = (warp / (T::TX / 8)) * 4 + (lane >> 3);
    const long m0 = (long)(blockIdx.x / p.n_tiles) * BM;
    const int n0 = (int)(blockIdx.x % p.n_tiles) * BN;
    const int kb0 = blockIdx.z * p.kb_per_split, kb1 = min(kb0 + p.kb_per_split, p.k_blocks);

    // the K block the next copies fetch
    int c0 = 0, kh = 0, kw = 0;
    long b_tap = 0;
    if (kb0) {
        const int tap = kb0 / p.c_blocks;
        c0 = (kb0 - tap * p.c_blocks) * BK;
        kh = tap / p.ksize_w; kw = tap - kh * p.ksize_w;
        b_tap = (long)tap * p.b_tap;
    }
    // Where the copies read: an address only advances, by the same distance for all rows, from block to block and from tap to tap
    // (outside of the operand it is not used).  B's rows lie a constant distance apart, and so do the columns of a ONE_ROW thread:
    // one address for all of its copies.  With whole quads on both sides a tap begins from the rows' first addresses instead, which
    // is what the compiler makes shorter blocks of there and longer ones elsewhere (12 x 436 -> 12 15.2 us, advancing 16.4; but
    // a product of 2 x 464 x 312, B by columns, 11.5 and 9.9 advancing).
    constexpr bool FROM_FIRST = AMODE == VEC_K && BMODE == VEC_K;
    [[maybe_unused]] const float *a_first[MA::ROW_SLOTS];
    const float *a_src[MA::ROW_SLOTS], *b_src = p.b + b_tap + (long)(n0 + MB::row(tid, 0)) * p.b_row + (long)(c0 + MB::col(tid, 0)) * p.b_col;
    int a_h[MA::ROW_SLOTS], a_w[MA::ROW_SLOTS];         // the pixels' origins
#pragma unroll
    for (int i = 0; i < MA::ROW_SLOTS; i++) {
        const long m = m0 + MA::row(tid, i);
        a_h[i] = a_w[i] = -(1 << 30);                   // (no row: outside at every tap)
        a_src[i] = p.a;
        if (MA::active(tid, i) && m < p.M) {
            const int per = p.g.OH * p.g.OW;            // a row index fits 31 bits
            const int n = (int)m / per, rem = (int)m - n * per, oh = rem / p.g.OW;
            a_h[i] = oh * p.g.stride - p.g.pad;
            a_w[i] = (rem - oh * p.g.OW) * p.g.stride - (p.g.pad_w >= 0 ? p.g.pad_w : p.g.pad);
            a_src[i] += (long)n * p.g.sn + (long)a_h[i] * p.g.sh + (long)a_w[i] * p.g.sw + (long)MA::col(tid, i) * p.g.sc;
        }
        if constexpr (FROM_FIRST) a_first[i] = a_src[i];
        else a_src[i] += (long)kh * p.g.sh + (long)kw * p.g.sw + (long)c0 * p.g.sc;
    }
    unsigned a_in = 0, b_in = 0;            // row slots that lie inside
    auto begin_tap = [&]() {
        [[maybe_unused]] const long tap = (long)kh * p.g.sh + (long)kw * p.g.sw + (long)c0 * p.g.sc;
        a_in = 0;
#pragma unroll
        for (int s = 0; s < MA::ROW_SLOTS; s++) {
            const bool in = (unsigned)(a_h[s] + kh) < (unsigned)p.g.H && (unsigned)(a_w[s] + kw) < (unsigned)p.g.W;
            if constexpr (FROM_FIRST) a_src[s] = in ? a_first[s] + tap : p.a;
            a_in |= (in ? 1u : 0u) << s;
        }
    };
#pragma unroll
    for (int s = 0; s < MB::ROW_SLOTS; s++) b_in |= (MB::active(tid, s) && n0 + MB::row(tid, s) < p.N ? 1u : 0u) << s;
    begin_tap();
    grid_dependency_wait();
    const long a_step = AMODE == ONE_ROW ? BK * p.g.sc : BK, b_step = BMODE == ONE_ROW ? BK * p.b_col : BK;
    const long a_next = AMODE == ONE_ROW ? T::THREADS / BM * p.g.sc : 0;        // from one copy of a slot to the next
    const long b_next = BMODE == ONE_ROW ? T::THREADS / BN * p.b_col : T::THREADS / MB::PER_ROW * p.b_row;
    // from behind a tap's last block to the next tap's first, in the same row of the filter, and what a new row adds
    const long a_tap = p.g.sw - p.c_blocks * a_step, a_row = p.g.sh - p.ksize_w * p.g.sw, b_tap_step = p.b_tap - p.c_blocks * b_step;
    const bool whole = p.Kc % BK == 0;      // no block has columns past the last
    const uint32_t smem32 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t a_dst = smem32 + (uint32_t)(MA::row(tid, 0) * LDK + MA::col(tid, 0)) * 4;
    const uint32_t b_dst = smem32 + (uint32_t)((BM + MB::row(tid, 0)) * LDK + MB::col(tid, 0)) * 4;
    auto fetch = [&](int slot) {
        const uint32_t at = (uint32_t)(slot * T::STAGE_FLOATS * 4);
        const float *src = a_src[0];
#pragma unroll
        for (int i = 0; i < MA::COPIES; i++) {
            if (!MA::active(tid, i)) continue;
            const int s = AMODE == ONE_ROW ? 0 : i;
            const bool in = (a_in >> s & 1) && (whole || c0 + MA::col(tid, i) < p.Kc);
            if (AMODE != ONE_ROW) src = a_src[s];
            if (AMODE == VEC_K) cp_async16(a_dst + at + i * MA::STEP * 4, in ? src : p.a, in);
            else cp_async4(a_dst + at + i * MA::STEP * 4, in ? src : p.a, in);
            if (AMODE == ONE_ROW) src += a_next;
        }
#pragma unroll
        for (int s = 0; s < MA::ROW_SLOTS; s++) a_src[s] += a_step;
        src = b_src;
#pragma unroll
        for (int i = 0; i < MB::COPIES; i++) {
            if (!MB::active(tid, i)) continue;
            const bool in = (b_in >> (BMODE == ONE_ROW ? 0 : i) & 1) && (whole || c0 + MB::col(tid, i) < p.Kc);
            if (BMODE == VEC_K) cp_async16(b_dst + at + i * MB::STEP * 4, in ? src : p.b, in);
            else cp_async4(b_dst + at + i * MB::STEP * 4, in ? src : p.b, in);
            src += b_next;
        }
        b_src += b_step;
        c0 += BK;
        if (c0 >= p.Kc) {
            c0 = 0;
            long next = a_tap;
            if (++kw == p.ksize_w) { kw = 0; kh++; next += a_row; }
            if constexpr (!FROM_FIRST) {
#pragma unroll
                for (int s = 0; s < MA::ROW_SLOTS; s++) a_src[s] += next;
            }
            b_src += b_tap_step;
            begin_tap();
        }
    };

    unsigned long long acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) acc[i][j] = 0ull;

    const int blocks = kb1 - kb0;
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (s < blocks) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int slot = 0;
    for (int kb = 0; kb < blocks; kb++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                // this block has arrived, and the slot fetched into next is no longer read
        if (kb + STAGES - 1 < blocks) fetch(slot == 0 ? STAGES - 1 : slot - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *as = smem + slot * T::STAGE_FLOATS, *bs = as + BM * LDK;
#pragma unroll
        for (int q = 0; q < BK / 4; q++) {
            ulonglong2 a[RM];
#pragma unroll
            for (int i = 0; i < RM; i++) a[i] = *reinterpret_cast<const ulonglong2 *>(as + (ty + T::TY * i) * LDK + 4 * q);
#pragma unroll
            for (int j = 0; j < RN; j++) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(bs + (tx + T::TX * j) * LDK + 4 * q);
#pragma unroll
                for (int i = 0; i < RM; i++) {
                    ffma2(acc[i][j], a[i].x, b.x);
                    ffma2(acc[i][j], a[i].y, b.y);
                }
            }
        }
        if (++slot == STAGES) slot = 0;
    }

    auto sum = [](unsigned long long v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); };
    const int S = gridDim.z;
    if (S == 1) {
#pragma unroll
        for (int i = 0; i < RM; i++) {
            const long m = m0 + ty + T::TY * i;
#pragma unroll
            for (int j = 0; j < RN; j++) {
                const int n = n0 + tx + T::TX * j;
                if (m < p.M && n < p.N) store_out(p, m, n, sum(acc[i][j]));
            }
        }
        return;
    }
    // the cluster's partial tiles: each CTA adds and writes its share of the rows
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) smem[(ty + T::TY * i) * T::RED_LD + tx + T::TX * j] = sum(acc[i][j]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int rank = blockIdx.z, share = BM * BN / S;       // S is a power of two up to 8
    for (int e = rank * share + tid; e < (rank + 1) * share; e += T::THREADS) {
        const int r = e / BN, c = e % BN;
        const long m = m0 + r;
        const int n = n0 + c;
        if (m >= p.M || n >= p.N) continue;
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
            v[q] = q < S ? cluster.map_shared_rank(smem, q)[r * T::RED_LD + c] : 0.0f;
        float x = v[0];
#pragma unroll
        for (int q = 1; q < 8; q++)
            if (q < S) x += v[q];
        store_out(p, m, n, x);
    }
    cluster.sync();                     // no CTA may exit while another still reads its partial tile
}

typedef void (*SimtKernel)(const SimtParams);
struct SimtVariant { SimtKernel kernel; int bm, bn, threads, smem; };
// 8 x 8 (two CTAs per SM: one of 128 x 128 with a barrier for all of the SM's warps took twice as long on AlexNet's third and
// fourth layers, 82 -> 44 us and 115 -> 60), 8 x 4 and 4 x 4 outputs per thread; the last for few rows
constexpr int SIMT_VARIANTS = 4;

template <int AMODE, int BMODE, int BM, int BN, int RM, int RN, int STAGES>
SimtVariant simt_variant() {
    using T = Tile<BM, BN, RM, RN, STAGES>;
    return {gemm_fp32_simt_kernel<BM, BN, RM, RN, STAGES, AMODE, BMODE>, BM, BN, T::THREADS, (int)(T::SMEM_FLOATS * sizeof(float))};
}
// the four tile shapes for a pair of copy modes (defined where that pair is compiled)
template <int AMODE, int BMODE>
const SimtVariant *simt_variants();

}  // namespace nb
