// Choice and launch of the CUDA-core contraction (gemm_simt.cuh), and the operator library's _gemm_.
#include "gemm_simt.cuh"

namespace nb {

template <> const SimtVariant *simt_variants<VEC_K, VEC_K>();
template <> const SimtVariant *simt_variants<VEC_K, ONE_K>();
template <> const SimtVariant *simt_variants<VEC_K, ONE_ROW>();
template <> const SimtVariant *simt_variants<ONE_K, VEC_K>();
template <> const SimtVariant *simt_variants<ONE_K, ONE_K>();
template <> const SimtVariant *simt_variants<ONE_K, ONE_ROW>();
template <> const SimtVariant *simt_variants<ONE_ROW, VEC_K>();
template <> const SimtVariant *simt_variants<ONE_ROW, ONE_K>();
template <> const SimtVariant *simt_variants<ONE_ROW, ONE_ROW>();

namespace {

const SimtVariant *variants(int amode, int bmode) {
    static const SimtVariant *(*const table[3][3])() = {
        {simt_variants<VEC_K, VEC_K>, simt_variants<VEC_K, ONE_K>, simt_variants<VEC_K, ONE_ROW>},
        {simt_variants<ONE_K, VEC_K>, simt_variants<ONE_K, ONE_K>, simt_variants<ONE_K, ONE_ROW>},
        {simt_variants<ONE_ROW, VEC_K>, simt_variants<ONE_ROW, ONE_K>, simt_variants<ONE_ROW, ONE_ROW>}};
    return table[amode][bmode]();
}

// A product of at most eight rows: the weights stream once from HBM, and a tile of 16 rows would spend its FMAs on rows that are not
// there (AlexNet's connected layers at 4 images, 9216 -> 4096 and 4096 -> 4096: 79 and 38 us in 16 x 128 tiles, 38 and 19 here, 0.9
// of the copy rate being 26 and 11).  A thread owns an output column of all MR rows; 64 columns of weights at a time come through a
// ring of shared memory by 16-byte cp.async (rows of 64 floats, stride 68: a 128-bit read of eight rows falls into 32 banks), the
// rows of A beside them, read as broadcasts.  Ranges of K, packed FMAs along K and their order are the tiles' above, so that a
// row alone and in a batch that runs there gives the same bits.
constexpr int ROWS_BN = 64, ROWS_BK = 64, ROWS_LD = ROWS_BK + 4, ROWS_STAGES = 5;
constexpr int rows_smem(int MR) { return ROWS_STAGES * (ROWS_BN * ROWS_LD + MR * ROWS_BK) * 4; }

template <int MR>
__global__ void __launch_bounds__(ROWS_BN) gemm_rows_kernel(const SimtParams p) {
    constexpr int STAGE = ROWS_BN * ROWS_LD + MR * ROWS_BK;     // floats
    extern __shared__ __align__(16) float smem[];
    grid_begin();
    const int tid = threadIdx.x, n0 = blockIdx.x * ROWS_BN;
    const int k0 = blockIdx.z * p.kb_per_split * BK, k1 = min(k0 + p.kb_per_split * BK, p.Kc);
    const int blocks = max(0, (k1 - k0 + ROWS_BK - 1) / ROWS_BK);
    const uint32_t smem32 = (uint32_t)__cvta_generic_to_shared(smem);
    const int quad = tid & 15, row = tid >> 4;                  // of the first copy: 16 lanes copy a row, 4 rows at a time
    const float *src = p.b + (long)(n0 + row) * p.b_row + k0 + 4 * quad;
    auto fetch = [&](int block, int slot) {
        const uint32_t at = smem32 + (uint32_t)(slot * STAGE * 4);
        const bool in_k = k0 + block * ROWS_BK + 4 * quad < k1;
#pragma unroll
        for (int i = 0; i < ROWS_BN / 4; i++) {
            const bool in = in_k && n0 + row + 4 * i < p.N;
            cp_async16(at + (uint32_t)((row + 4 * i) * ROWS_LD + 4 * quad) * 4, in ? src + (long)block * ROWS_BK + (long)(4 * i) * p.b_row : p.b, in);
        }
#pragma unroll
        for (int i = 0; i < (MR * 16 + ROWS_BN - 1) / ROWS_BN; i++) {
            const int m = row + 4 * i;
            if (m >= MR) break;
            const bool in = in_k && m < p.M;
            cp_async16(at + (uint32_t)(ROWS_BN * ROWS_LD + m * ROWS_BK + 4 * quad) * 4, in ? p.a + (long)m * p.g.sw + k0 + block * ROWS_BK + 4 * quad : p.a, in);
        }
    };
    unsigned long long acc[MR];
#pragma unroll
    for (int m = 0; m < MR; m++) acc[m] = 0ull;
#pragma unroll
    for (int s = 0; s < ROWS_STAGES - 1; s++) {
        if (s < blocks) fetch(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int slot = 0;
    for (int block = 0; block < blocks; block++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_STAGES - 2) : "memory");
        __syncthreads();                // this block has arrived, and the slot fetched into next is no longer read
        if (block + ROWS_STAGES - 1 < blocks) fetch(block + ROWS_STAGES - 1, slot == 0 ? ROWS_STAGES - 1 : slot - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *bs = smem + slot * STAGE + tid * ROWS_LD, *as = smem + slot * STAGE + ROWS_BN * ROWS_LD;
#pragma unroll
        for (int q = 0; q < ROWS_BK / 4; q++) {
            const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(bs + 4 * q);
#pragma unroll
            for (int m = 0; m < MR; m++) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(as + m * ROWS_BK + 4 * q);
                ffma2(acc[m], a.x, b.x);
                ffma2(acc[m], a.y, b.y);
            }
        }
        if (++slot == ROWS_STAGES) slot = 0;
    }
    auto sum = [](unsigned long long v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); };
    const int S = gridDim.z, n = n0 + tid;
    if (S == 1) {
#pragma unroll
        for (int m = 0; m < MR; m++)
            if (m < p.M && n < p.N) store_out(p, m, n, sum(acc[m]));
        return;
    }
    // the cluster's partial sums: each CTA adds and writes its share
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MR; m++) smem[m * ROWS_BN + tid] = sum(acc[m]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = blockIdx.z * ROWS_BN + tid; e < MR * ROWS_BN; e += S * ROWS_BN) {
        const int m = e / ROWS_BN, c = n0 + e % ROWS_BN;
        if (m >= p.M || c >= p.N) continue;
        float x = cluster.map_shared_rank(smem, 0)[e];
        for (int q = 1; q < S; q++) x += cluster.map_shared_rank(smem, q)[e];
        store_out(p, m, c, x);
    }
    cluster.sync();                     // no CTA may exit while another still reads its partial sums
}

// _gemm_ with few columns of K and few tiles, where a product is a handful of dependent steps whatever its tiles: 16 x 16
// outputs per CTA, one per thread, operands loaded straight into both tiles.  Nothing is set up per copy and thread, which is
// what the kernel above spends such a call on (64 x 64 x 64: 4.3 us here, 6.6 there; 200 x 48 x 16: 2.0 and 3.7).  It adds in
// the same order (even and odd columns apart): the two give the same bits, and half the chain of one sum.
__global__ void __launch_bounds__(256) gemm_small_kernel(int ta, int tb, int M, int N, int K, float alpha, const float *A, int lda,
                                                         const float *B, int ldb, float beta, float *C, int ldc) {
    __shared__ float As[16][17], Bs[16][17];
    grid_dependents_start();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int row = blockIdx.y * 16 + ty, col = blockIdx.x * 16 + tx;
    float even = 0.0f, odd = 0.0f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        const int ka = k0 + tx, kb = k0 + ty;
        As[ty][tx] = (row < M && ka < K) ? (ta ? A[(size_t)ka * lda + row] : A[(size_t)row * lda + ka]) : 0.0f;
        Bs[ty][tx] = (col < N && kb < K) ? (tb ? B[(size_t)col * ldb + kb] : B[(size_t)kb * ldb + col]) : 0.0f;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
            even = fmaf(As[ty][k], Bs[k][tx], even);
            odd = fmaf(As[ty][k + 1], Bs[k + 1][tx], odd);
        }
        __syncthreads();
    }
    if (row < M && col < N) {
        float *c = C + (size_t)row * ldc + col;
        *c = alpha * (even + odd) + (beta == 0.0f ? 0.0f : beta * *c);
    }
}

// Fitted to 1101 products of 1 to 2048 rows, 16 to 4096 columns, K of 16 to 1024, timed without host time: what this kernel
// loses on more tiles than the SMs take at once against what it gains per call, more the fewer 16-byte copies the other can make.
bool small_gemm(bool ta, bool tb, int M, int N, int K) {
    const double tiles = (double)((M + 15) / 16) * ((N + 15) / 16);
    if (K <= 32) return tiles <= 2500;
    const bool quads = !ta && tb;               // both operands K-contiguous
    if (K > (quads ? 128 : 256)) return false;
    const double gain_us = quads ? 1.2 : (ta ? 2.2 + 0.008 * K : (K <= 128 ? 2.4 : 0.9));
    return (tiles - 230) * 1.2e-4 * K <= gain_us;
}

// Cycles of an SM that runs `on_sm` CTAs of tile shape i over K columns each: the share of the FMA rate that the shape reaches
// (fewer outputs per operand read, longer runs between barriers), and its start and stores.  The 64 x 128 tile alone on an SM
// lacks a second CTA to run behind its barriers, the more the shorter its copies.  Fitted to AlexNet's layers at 4 and 16 images and
// to products of 64 to 2048 rows and K of 60 to 4000; that tile's rate alone with whole quads to 880 layers and products timed with every
// shape (968 x 89 x 2352 takes 27 us in 64 x 64 tiles, 41 in the 64 x 128 that a rate of 0.47 chose; 2873 x 348 x 96 14 and 25), and its
// rate where A's rows come value by value, for which it lacks the registers (2508 x 74 -> 1344 48 and 68 us).  With ten blocks of K or
// fewer its start and its 64 stores per thread are most of it (5x5, 3 -> 384 at 9 images of 51 x 51, tanh, 195 us, 123 in 32 x 64; 3x3, 8 ->
// 352 at 10 of 58 x 58 59 and 43).
double tile_cost(int i, const SimtVariant &v, long on_sm, int K, bool quads, bool single_a, bool split) {
    static const double rate[] = {0.50, 0.41, 0.36, 0.33}, fixed[] = {4000, 1300, 200, 400};
    double r = i == 0 && single_a ? 0.44 : rate[i];
    if (i == 0 && on_sm == 1) r = quads ? 0.38 : 0.30;
    return on_sm * ((double)v.bm * v.bn * K / 128 / r + (i == 0 && !split && K <= 160 ? 12000 : fixed[i]));
}

// Ranges of K: none shorter than `least` columns, and only as many as it takes to occupy the SMs `times` over with 64 x 64 tiles of
// one image (one row of a connected layer, all rows of _gemm_).  _gemm_: 256 x 1024 x 1024 two ranges 29 us, eight 23.  A layer's
// S counts one image alone, so its batches fill the SMs anyway (64 -> 64 3x3 at 56 x 56, 16 images: whole 123 us, two ranges 137).
int split_of(const nb_handle_s *h, long unit_rows, int N, int k_blocks, int least, int times) {
    const long tiles = ((unit_rows + 63) / 64) * ((N + 63) / 64);
    int S = 1;
    while (S < 8 && tiles * S < (long)times * h->sm_count && k_blocks / (2 * S) >= least / BK) S *= 2;
    return S;
}

// The tile shape with the cheapest last wave, and its kernel for these copy modes, loaded and with its shared-memory limit set.
// None is loaded with the handle (all of them took 19 ms of a process's first one, while a handle uses a few at most): a plan
// asks for its own when it reserves its scratch (gemm_simt_load); a kernel first met by a launch, captured ones included, is
// loaded there.
constexpr int ROWS_MAX = 8;
const SimtVariant ROWS_VARIANTS[4] = {{gemm_rows_kernel<1>, 1, ROWS_BN, ROWS_BN, rows_smem(1)}, {gemm_rows_kernel<2>, 2, ROWS_BN, ROWS_BN, rows_smem(2)},
                                      {gemm_rows_kernel<4>, 4, ROWS_BN, ROWS_BN, rows_smem(4)}, {gemm_rows_kernel<8>, 8, ROWS_BN, ROWS_BN, rows_smem(8)}};

const SimtVariant &ready_variant(nb_handle_s *h, long M, int N, int K, bool plain, int S, int amode, int bmode) {
    const bool rows = plain && M <= ROWS_MAX && amode == VEC_K && bmode == VEC_K;
    const SimtVariant *all = rows ? ROWS_VARIANTS : variants(amode, bmode);
    int best = rows ? (M > 4 ? 3 : (M > 2 ? 2 : (int)M - 1)) : 0;
    double best_cost = 0;
    for (int i = 0; i < SIMT_VARIANTS && !rows; i++) {
        const SimtVariant &v = all[i];
        const long ctas = ((M + v.bm - 1L) / v.bm) * ((N + v.bn - 1L) / v.bn) * S;
        const long on_sm = (ctas + h->sm_count - 1) / h->sm_count;
        const double cost = tile_cost(i, v, on_sm, K / S, amode == VEC_K && bmode == VEC_K, amode == ONE_K, S > 1);
        if (i == 0 || cost < best_cost) { best_cost = cost; best = i; }
    }
    const SimtVariant &v = all[best];
    const unsigned long long bit = 1ull << (rows ? 9 * SIMT_VARIANTS + best : 9 * best + 3 * amode + bmode);
    if (!(h->simt_ready & bit)) {
        cudaFuncAttributes fa;          // (loads the code)
        if (v.smem > 48 * 1024) NB_CHECK_CUDA(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
        else NB_CHECK_CUDA(cudaFuncGetAttributes(&fa, v.kernel));
        h->simt_ready |= bit;
    }
    return v;
}

// A is a matrix: one image of height 1, a 1x1 filter.
bool plain_rows(const SimtParams &p) {
    return p.g.H == 1 && p.g.ksize == 1 && p.ksize_w == 1 && p.g.stride == 1 && p.g.pad == 0 && p.g.pad_w <= 0 && p.g.OW == p.M;
}

void launch(nb_handle_s *h, SimtParams &p, int amode, int bmode, int S) {
    const SimtVariant &v = ready_variant(h, p.M, p.N, p.k_blocks * BK, plain_rows(p), S, amode, bmode);
    p.n_tiles = (p.N + v.bn - 1) / v.bn;
    p.kb_per_split = (p.k_blocks + S - 1) / S;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((p.M + v.bm - 1L) / v.bm) * p.n_tiles), 1, (unsigned)S);
    cfg.blockDim = dim3((unsigned)v.threads);
    cfg.dynamicSmemBytes = (size_t)v.smem;
    cfg.stream = h->stream;
    // Not launched ahead of the kernel in front: several of these CTAs fit an SM, and those that became resident early
    // would crowd the SMs which that kernel leaves free (AlexNet b4 fp32: 650 us in order, 764 us ahead).
    // A few CTAs with little to do crowd nobody: 32 x 30 x 62 at the end of the deep belief network 10.5 -> 6.7 us, four layers of
    // 300 at 16 rows 61 -> 56.  With much to do they spend it on the SMs they crowded (24 CTAs of 15 552 columns of K each: 491 us in
    // order, about 680 ahead), and behind a layer of many rows, which is long itself, the line is lower (659 x 312 -> 10 and the three
    // layers in front 75.6 us ahead, 70.9 in order).
    const bool ahead = (long)cfg.gridDim.x * S <= h->sm_count / 4 && p.kb_per_split * BK <= (p.M <= 128 ? 512 : 256);
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = ahead ? 1 : 0;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = (unsigned)S;
    cfg.attrs = at;
    cfg.numAttrs = S > 1 ? 2 : 1;
    ProfileScope prof(h, 1, 2.0 * (double)p.M * p.N * p.Kc * p.g.ksize * p.ksize_w);
    (void)cudaLaunchKernelEx(&cfg, v.kernel, p);
    check_launch("gemm_fp32_simt_kernel");
    count_launch(h);
    prof.finish();
}

inline bool vec_ok(const float *p, long s0, long s1, long s2) {
    return (((uintptr_t)p) & 15) == 0 && s0 % 4 == 0 && s1 % 4 == 0 && s2 % 4 == 0;
}

}  // namespace

static void simt_params(const nb_handle_s *h, const GemmArgs &a, SimtParams *out, int *amode, int *bmode, int *S) {
    SimtParams &p = *out;
    p.a = a.a; p.b = a.b;
    if (a.a_is_conv) {
        p.g = a.g;
    } else {
        p.g = ConvGeom();
        p.g.batch = 1; p.g.C = a.Kc; p.g.H = 1; p.g.W = a.M; p.g.OH = 1; p.g.OW = a.M;
        p.g.sc = 1; p.g.sw = a.lda; p.g.sh = 0; p.g.sn = 0;
    }
    p.ksize_w = p.g.ksize_w > 0 ? p.g.ksize_w : p.g.ksize;
    p.b_tap = (long)a.N * a.ldb; p.b_row = a.ldb; p.b_col = 1;
    p.M = a.M; p.N = a.N; p.Kc = a.Kc;
    p.c_blocks = (a.Kc + BK - 1) / BK;
    p.k_blocks = p.c_blocks * p.g.ksize * p.ksize_w;
    p.scale = a.scale; p.shift = a.shift; p.addend = a.addend; p.ld_addend = a.ld_addend;
    p.act = a.act; p.round_out = a.round_out_tf32 ? 1 : 0; p.addend_post = a.addend_after_act ? 1 : 0;
    p.y = a.y; p.ldy = a.ldy;
    // 16-byte copies need whole quads of columns on 16-byte boundaries; a tensor whose pixels are contiguous per
    // channel (NCHW) is read with lanes along the pixels
    *amode = p.g.sc == 1 ? (a.Kc % 4 == 0 && vec_ok(p.a, p.g.sn, p.g.sh, p.g.sw) ? VEC_K : ONE_K) : ONE_ROW;
    *bmode = a.Kc % 4 == 0 && vec_ok(p.b, a.ldb, p.b_tap, 0) ? VEC_K : ONE_K;
    *S = split_of(h, a.a_is_conv ? (long)p.g.OH * p.g.OW : 1, a.N, p.k_blocks, 256, 1);
}

void gemm_simt_load(nb_handle_s *h, const GemmArgs &a) {
    SimtParams p{};
    int amode, bmode, S;
    simt_params(h, a, &p, &amode, &bmode, &S);
    ready_variant(h, p.M, p.N, p.k_blocks * BK, plain_rows(p), S, amode, bmode);
}

void gemm_simt(nb_handle_s *h, const GemmArgs &a) {
    if (a.addend && a.res_stride > 0) throw Error(NB_ERR_UNSUPPORTED, "the CUDA-core path takes no fused residual");
    SimtParams p{};
    int amode, bmode, S;
    simt_params(h, a, &p, &amode, &bmode, &S);
    launch(h, p, amode, bmode, S);
}

// _gemm_ (common/gemm.h:21-25) with the CPU path's meaning of every argument (row-major, leading dimensions honoured, all
// four transpose cases), unlike the reference's CUDA stand-in (common/gemm.cu:38-153) which ignores lda/ldb/ldc.
void launch_sgemm(nb_handle_s *h, bool ta, bool tb, int M, int N, int K, float alpha, const float *A, int lda,
                  const float *B, int ldb, float beta, float *C, int ldc) {
    // (the operator has refused more rows since its first kernel, whose grid they did not fit; the limit is part of it by now)
    if ((M + 15) / 16 > 65535) throw Error(NB_ERR_UNSUPPORTED, "gemm: M too large for this operator");
    if (small_gemm(ta, tb, M, N, K)) {
        gemm_small_kernel<<<dim3((N + 15) / 16, (M + 15) / 16), 256, 0, h->stream>>>(ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
        check_launch("gemm_small_kernel");
        count_launch(h);
        return;
    }
    SimtParams p{};
    p.a = A; p.b = B;
    p.g = ConvGeom();
    p.g.batch = 1; p.g.C = K; p.g.H = 1; p.g.W = M; p.g.OH = 1; p.g.OW = M;
    p.g.sc = ta ? lda : 1; p.g.sw = ta ? 1 : lda; p.g.sh = 0; p.g.sn = 0;
    p.ksize_w = 1;
    p.b_tap = 0; p.b_row = tb ? ldb : 1; p.b_col = tb ? 1 : ldb;
    p.M = M; p.N = N; p.Kc = K;
    p.c_blocks = p.k_blocks = (K + BK - 1) / BK;
    p.act = NB_ACT_LINEAR;
    p.blas = 1; p.alpha = alpha; p.beta = beta;
    p.y = C; p.ldy = ldc;
    const int amode = ta ? ONE_ROW : (K % 4 == 0 && vec_ok(A, lda, 0, 0) ? VEC_K : ONE_K);
    const int bmode = !tb ? ONE_ROW : (K % 4 == 0 && vec_ok(B, ldb, 0, 0) ? VEC_K : ONE_K);
    launch(h, p, amode, bmode, split_of(h, M, N, p.k_blocks, 128, 2));
}

void gemm(nb_handle_s *h, const GemmArgs &a) {
    if (h->math_mode != NB_MATH_FP32 && gemm_tc_supported(h, a)) {
        gemm_tc(h, a, h->math_mode == NB_MATH_TF32X3);
    } else {
        gemm_simt(h, a);
    }
}

}  // namespace nb
