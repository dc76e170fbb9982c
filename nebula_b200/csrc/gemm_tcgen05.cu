// Tensor-core GEMM / implicit-GEMM convolution for sm_100a.
//
//   D[M,N] = A[M,K] * B[N,K]^T   (both operands K-major, fp32 storage, TF32 math,
//                                 fp32 accumulation in tensor memory)
//
// Replaces the reference's per-image im2col + SGEMM pair
// (models/layers/convolutional_layer.cu:47-70, common/utils.cu:34-74) and its
// fully-connected SGEMM (models/layers/connected_layer.cu:21-38) with ONE
// persistent kernel over the whole batch:
//   * rows of A are output pixels (image, oh, ow); the im2col matrix is never
//     materialised -- for every filter tap (kh,kw) and 32-channel slice a TMA
//     box load fetches the shifted NHWC window, out-of-bounds coordinates give
//     the zero padding;
//   * columns of D are filters; B is the weight tensor re-laid out once as
//     [tap][filter][channel];
//   * tcgen05.mma (kind::tf32, M=128, N=BLOCK_N, K=8) accumulates into TMEM,
//     double-buffered so the epilogue of tile i overlaps the main loop of i+1;
//   * the epilogue applies folded batch-norm scale/shift + bias, an optional
//     addend (residual / LSTM input projection), the activation, and optional
//     TF32 rounding for the next contraction, and stores NHWC rows directly.
// A plain row-major matrix is the special case "image of height 1, 1x1 filter".
//
// Warp roles (320 threads; 448 with the extra operand warps):
//   warp 0      TMA producer (one elected lane)
//   warp 1      TMEM allocation + MMA issue (one elected lane)
//   warps 2-9   epilogue, two groups of four (TMEM -> registers -> shared-memory slab -> TMA store)
//   warps 10-13 three-pass mode: split each A tile into hi/lo TF32 terms in tensor memory; gather mode: build the
//               A tile in shared memory from a strided tensor (3-channel input layers)
//
// Every wait is bounded: a wait that runs out sets the CTA's abort flag and the
// device status word, all roles drain, TMEM is freed and the kernel returns.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>

#include "tc_common.cuh"

namespace nb {

using namespace tc;

namespace {

constexpr int RESIDUAL_OFFSET = 128 * 1024;     // of the shortcut's slab buffers (64 KB at most, in front of the staging buffers)
constexpr int GATHER_MAX_K = 384;      // largest k*k*C (rounded up to 32) the gather table in the kernel parameters holds

struct TcParams {
    CUtensorMap tm_a;
    CUtensorMap tm_b;
    CUtensorMap tm_b_lo;
    CUtensorMap tm_y;
    CUtensorMap tm_yp;          // 2x2/2 max-pooled output (pool mode)
    // tiling of the M dimension into (bw x bh x bn) boxes of output pixels
    int bw, bh, bn;
    int tiles_w, tiles_h, tiles_n;
    int OW, OH, NB;
    int ksize_w, stride, pad_w, pad_h;      // filter columns (the tap index is kh*ksize_w + kw) and paddings
    int c_blocks;               // 32-channel slices per tap
    int num_k_blocks;           // ksize*ksize*c_blocks
    int m_tiles, n_tiles;
    // tile order: consecutive tiles share the A tile (n fastest) or, when the weights are what streams from HBM
    // (connected layers wider than L2), the B tile (m fastest), so that the second reader finds it in L2
    int m_fastest;
    int tx_bytes_a;             // bytes one A box load delivers
    // split-K: a tile is (m_tile, n_tile, split); split s runs K blocks [s*kb_per_split, (s+1)*kb_per_split).  In a cluster
    // the splits of a tile are its CTAs, which finish it together; otherwise split s is stored into slab s of y (batch
    // coordinate n + s*NB): y then holds k_splits partial tensors
    int k_splits, kb_per_split;
    // The tensor core's fp32 accumulator rounds toward zero at every K=8 step (a bias that grows with K).
    // After every kb_per_part K blocks the partial sums are promoted to registers (round-to-nearest adds)
    // and the TMEM accumulator restarts; parts = number of such partial sums per tile (1: no promotion).
    int kb_per_part, parts;
    // Ring stages of `cbs` K blocks (1 or 2).  One TMA request costs its issuing thread a few hundred cycles whatever
    // its size, and a narrow tile's K block is only 180-350 cycles of MMAs, so tiles of up to 128 columns whose 32-column
    // slices pair up fetch two slices per request: the A map then has the slice index as a fifth dimension (tm_a is 5-D,
    // tm_b 4-D), a stage is [A0 | A1 | B0 | B1], `stages` of them fit the ring.  A slice of the A box is a_slice_bytes (a
    // whole number of 1024-byte swizzle repeats); the MMA reads 128 rows from its start, so A takes a_region bytes, and what
    // it reads past a box of fewer rows only feeds accumulator rows that are never stored.
    int cbs, stages, a_slice_bytes, a_region;
    // Filter-column stages (col3 = 1): 3x3 stride-1 convolutions with few input channels are bound by the L2 -> shared
    // memory traffic of re-loading the activation tile once per tap.  Here a stage is one filter COLUMN kw of one channel
    // slice: ONE activation box of bh + 2 image rows (a_box_bytes) and the three weight tiles kh = 0..2.  Tap (kh, kw)
    // reads the box from image row kh on: a start address kh * bw * 128 bytes further, which for bw = 16 stays on the
    // 1024-byte repeat of the swizzle pattern.  Three activation loads per slice instead of nine.
    int col3, a_box_bytes, stage_bytes;
    // col3 only: a tile of `halves` (1 or 2) vertically adjacent 16 x 8 boxes.  Both read the same activation box
    // (bh * halves + 2 image rows, the second half 8 image rows further down) and the same three weight tiles, which
    // halves the weight traffic per pixel; each half has its own accumulator columns.
    int halves;
    // Byte offset (from the ring's start) of a second staging buffer per epilogue group, or 0.  A bulk store takes over
    // a thousand cycles to read its 16 KB out of shared memory; where the ring leaves room, a group alternates between
    // two buffers and lets one store read while the next slab is staged.
    int slab2_offset;
    EpiParams e;                // fused epilogue
    int b_static;               // B is a plan's weights: its first tiles may be fetched before the kernels in front are done
    int *status;
};

// The gather variants' parameters: the offset table is three quarters of them, and the other variants' launches do not
// carry it.
struct TcGatherParams : TcParams {
    // gather mode: warps 10-13 build the A tile in shared memory from a strided activation tensor
    // (channel counts TMA cannot address, e.g. the 3-channel input layer); rows are output pixels
    const float *gx;
    long gsn, gsh, gsw;         // element strides of the gathered tensor
    int gks, gpad, gK;          // filter size, padding, k*k*C: column kk = (kh, kw, c), c fastest
    int gH, gW, gOH, gOW, gstride, gM, ground;
    // per column: {element offset of (c, kh-pad, kw-pad) from the pixel's origin, (kh-pad) & 0xffff | (kw-pad) << 16}
    int2 gtab[GATHER_MAX_K];
};
template <bool GATHER> struct ParamsOf { typedef TcParams type; };
template <> struct ParamsOf<true> { typedef TcGatherParams type; };

// in = false: nothing is read and the destination becomes zero
__device__ __forceinline__ void cp_async16(uint32_t dst, const float *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// The digits (split, n_tile, tw, th, tn) of a CTA's current tile.  Decoding a tile index costs seven integer
// divisions (over a thousand cycles of dependent instructions on a role's critical path), so the index is decoded
// once and then advanced by the digits of the grid stride, with carries.
struct TileIter {
    int split, n_tile, tw, th, tn;      // current tile
    int ds, dn, dw, dh, dt;             // the grid stride

    __device__ __forceinline__ static void decode(const TcParams &p, int tile, int &s, int &n, int &w, int &h, int &t) {
        s = tile % p.k_splits;
        const int mn = tile / p.k_splits;
        const int m_tile = p.m_fastest ? mn % p.m_tiles : mn / p.n_tiles;
        n = p.m_fastest ? mn / p.m_tiles : mn % p.n_tiles;
        w = m_tile % p.tiles_w;
        h = (m_tile / p.tiles_w) % p.tiles_h;
        t = m_tile / (p.tiles_w * p.tiles_h);
    }
    __device__ __forceinline__ TileIter(const TcParams &p, int first, int step) {
        decode(p, first, split, n_tile, tw, th, tn);
        decode(p, step, ds, dn, dw, dh, dt);
    }
    // digit + stride digit + carry < 2 * radix: one conditional subtraction per digit
    __device__ __forceinline__ static int add(int &digit, int inc, int radix) {
        digit += inc;
        const int carry = digit >= radix ? 1 : 0;
        if (carry) digit -= radix;
        return carry;
    }
    __device__ __forceinline__ void next(const TcParams &p) {
        int c = add(split, ds, p.k_splits);
        if (p.m_fastest) {
            c = add(tw, dw + c, p.tiles_w);
            c = add(th, dh + c, p.tiles_h);
            c = add(tn, dt + c, p.tiles_n);
            n_tile += dn + c;
        } else {
            c = add(n_tile, dn + c, p.n_tiles);
            c = add(tw, dw + c, p.tiles_w);
            c = add(th, dh + c, p.tiles_h);
            tn += dt + c;
        }
    }
};

// 3xTF32 multiplies every K block three times, and with both operands in shared memory the port is the bound: at N = 128
// twelve MMAs read 96 KB, the splitter reads 16 KB and writes 32, TMA writes 48: 1536 cycles of port per 768 of MMAs (1450
// measured).  So the splitter writes the two terms of A to tensor memory instead (TS): the MMAs then read only B from
// shared memory, 48 + 16 + 48 KB.  Tensor memory holds two accumulators, the cross terms of one tile (two at N = 64) and
// A_BUFS pairs of A terms, 64 columns each.
template <int BLOCK_N, bool THREE, bool GATHER>
struct Cfg {
    static constexpr bool TS = THREE && !GATHER;
    static constexpr int A_BUFS = BLOCK_N == 64 ? 4 : 2, X_BUFS = TS && BLOCK_N != 64 ? 1 : 2;
    static constexpr int A_COL = (2 + X_BUFS) * BLOCK_N;
    static constexpr int B_STAGE_BYTES = BLOCK_N * BLOCK_K * 4;
    static constexpr int STAGE_BYTES = TS ? A_STAGE_BYTES + 2 * B_STAGE_BYTES : (A_STAGE_BYTES + B_STAGE_BYTES) * (THREE ? 2 : 1);
    static constexpr int B_LO_OFFSET = TS ? B_STAGE_BYTES : B_STAGE_BYTES + A_STAGE_BYTES;      // from B's high-order terms
    static constexpr int STAGES = (196 * 1024) / STAGE_BYTES < 8 ? (196 * 1024) / STAGE_BYTES : 8;
    static constexpr int TMEM_COLS = 2 * BLOCK_N;
    static constexpr int OUT_STAGE_BYTES = BLOCK_M * 32 * 4;     // one 128 x 32 output slab
    static constexpr int LAYOUT_BYTES = STAGES * STAGE_BYTES + 2 * OUT_STAGE_BYTES + 256 /*barriers*/;
    // all of the 227 KB a CTA may have: what the layout leaves over holds the epilogue's scale/shift values
    static constexpr int SMEM_BYTES = 227 * 1024;
    static_assert(LAYOUT_BYTES + (THREE ? 0 : 2 * BLOCK_N * 4) <= SMEM_BYTES, "ring, staging buffers, barriers and scale/shift values must fit");
};

// All threads of the cluster; what each wrote to its shared memory before is visible to the others behind it.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t smem_addr, int rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_addr), "r"(rank) : "memory");
    return v;
}

// The epilogue warps of a CTA of a tile whose K is cut over a cluster.  Every CTA leaves its partial sums in its shared memory
// (the ring is free: its MMAs are done); behind the cluster's barrier each takes an equal share of the tile's rows, adds the
// partial sums over the cluster's shared memory in the order of K, and finishes them: folded batch-norm and bias, shortcut,
// activation, rounding, 2x2/2 max-pool, rows as NHWC or NCHW.  Bound by latency: with partial tensors in HBM and a kernel behind it
// that adds them a small layer took about 3 us more, and a tile's activations had one SM: a ResNet-50 image 466 -> 424 us, the RNN
// (tanh layers of 512 x 256 x 256) 113 -> 102, VGG-16 b1 in 3xTF32 567 -> 535.
template <int BLOCK_N, bool THREE, bool PROMOTE>
__device__ __forceinline__ void cluster_epilogue(const TcParams &p, uint8_t *smem, uint32_t tmem_base, uint64_t *acc_full, uint64_t *acc_empty,
                                                 bool cross_cols, volatile int *abort_flag) {
    using C = Cfg<BLOCK_N, THREE, false>;
    constexpr int CH = BLOCK_N / 64, N4 = BLOCK_N / 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = (warp - 2) >> 2, bar_id = 1 + grp, q = warp & 3, r = q * 32 + lane;
    const int t = threadIdx.x - 64;                         // 0..255
    const TileIter ti(p, blockIdx.x, gridDim.x);
    const int S = p.k_splits, rank = ti.split, n0 = ti.n_tile * BLOCK_N;
    const int box_rows = p.bw * p.bh * p.bn;
    float4 *part = reinterpret_cast<float4 *>(smem);        // [rows][BLOCK_N]: 16-byte chunk c of row r at c ^ (r % 8)

    // this CTA's share: rows, or pooled pixels; a thread has the same four columns in all of its items
    const int units = p.e.pool ? box_rows / 4 : box_rows, per = (units + S - 1) / S;
    const int u0 = rank * per, u_end = min(units, u0 + per);
    // (NCHW output: lanes along the pixels, else along the columns)
    const int c4 = p.e.plane ? t / (256 / N4) : t % N4, first_u = u0 + (p.e.plane ? t % (256 / N4) : t / N4), col = n0 + 4 * c4;
    const bool col_ok = col < p.e.N;                        // (convolutions: whole quads)
    float4 sc = make_float4(1.f, 1.f, 1.f, 1.f), sh = make_float4(0.f, 0.f, 0.f, 0.f);
    if (col_ok && p.e.scale) sc = __ldg(reinterpret_cast<const float4 *>(p.e.scale + col));
    if (col_ok && p.e.shift) sh = __ldg(reinterpret_cast<const float4 *>(p.e.shift + col));
    // row of the box -> output pixel
    struct Pixel { int n, oh, ow; bool ok; long row; };
    auto pixel = [&](int row) {
        Pixel x;
        x.ow = ti.tw * p.bw + row % p.bw; x.oh = ti.th * p.bh + row / p.bw % p.bh; x.n = ti.tn * p.bn + row / (p.bw * p.bh);
        x.ok = x.ow < p.OW && x.oh < p.OH && x.n < p.NB;
        x.row = ((long)x.n * p.OH + x.oh) * p.OW + x.ow;
        return x;
    };
    auto residual = [&](const Pixel &x) {
        const float *a = col < p.e.addend_cols ? addend_row(p.e, x.ok, x.row, x.n, x.oh, x.ow) : nullptr;
        return a ? *reinterpret_cast<const float4 *>(a + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    grid_dependency_wait();
    // (the first item's shortcut is fetched while the MMAs run)
    float4 first_res = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.e.addend && col_ok && first_u < u_end) first_res = residual(pixel(first_u));

    bool ok = true;
    auto keep = [&](const uint32_t (&v)[32], int chunk) {
        if (r >= box_rows) return;
#pragma unroll
        for (int j = 0; j < 8; j++)
            part[r * N4 + ((chunk * 8 + j) ^ (r & 7))] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                                    __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
    };
    const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16);
    if (!PROMOTE || p.parts == 1) {
        ok = epilogue_all(mbar_wait(&acc_full[0], 0, abort_flag, p.status), bar_id);
        if (ok) {
            tc_fence_after();
#pragma unroll 1
            for (int chunk = grp; chunk < BLOCK_N / 32; chunk += 2) {
                uint32_t v[32];
                tmem_ld_32x32(lanes + (uint32_t)(chunk * 32), v);
                tmem_ld_wait();
                keep(v, chunk);
            }
            tc_fence_before();
        }
    } else if constexpr (PROMOTE) {
        uint32_t sum[CH][32];
        const int tile_kb = min(p.kb_per_split, p.num_k_blocks - rank * p.kb_per_split);
        const int parts = (tile_kb + p.kb_per_part - 1) / p.kb_per_part;
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int i = 0; i < parts; i++) {
            if (!(ok = epilogue_all(mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.status), bar_id))) break;
            tc_fence_after();
#pragma unroll
            for (int ci = 0; ci < CH; ci++) {
                uint32_t v[32];
                tmem_ld_32x32(lanes + (uint32_t)(acc * BLOCK_N + (grp + 2 * ci) * 32), v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j++) sum[ci][j] = i == 0 ? v[j] : __float_as_uint(__uint_as_float(sum[ci][j]) + __uint_as_float(v[j]));
                if (cross_cols && i == parts - 1) {         // the cross terms: complete with the last MMAs
                    tmem_ld_32x32(lanes + (uint32_t)(2 * BLOCK_N + (grp + 2 * ci) * 32), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) sum[ci][j] = __float_as_uint(__uint_as_float(sum[ci][j]) + __uint_as_float(v[j]));
                }
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[acc]);
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        if (ok) {
#pragma unroll
            for (int ci = 0; ci < CH; ci++) keep(sum[ci], grp + 2 * ci);
        }
    }
    __syncwarp();
    cluster_barrier();

    const uint32_t part32 = smem_u32(part);
    auto value = [&](int row, const Pixel &x, bool first) {
        const uint32_t at = part32 + (uint32_t)(row * N4 + (c4 ^ (row & 7))) * 16;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < S; s0 += 8) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (s0 + i < S) v[i] = ld_cluster(at, s0 + i);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (s0 + i >= S) continue;
                if (s0 + i == 0) a = v[0];
                else { a.x += v[i].x; a.y += v[i].y; a.z += v[i].z; a.w += v[i].w; }
            }
        }
        if (p.e.scale) {
            a.x = fmaf(a.x, sc.x, sh.x); a.y = fmaf(a.y, sc.y, sh.y); a.z = fmaf(a.z, sc.z, sh.z); a.w = fmaf(a.w, sc.w, sh.w);
        } else {
            a.x += sh.x; a.y += sh.y; a.z += sh.z; a.w += sh.w;
        }
        if (p.e.addend) {
            const float4 b = first ? first_res : residual(x);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        a = apply_activation4_fast(a, p.e.act);
        if (p.e.round_out) { a.x = round_tf32(a.x); a.y = round_tf32(a.y); a.z = round_tf32(a.z); a.w = round_tf32(a.w); }
        return a;
    };
    for (int u = first_u; u < u_end && col_ok; u += 256 / N4) {
        float *dst;
        float4 a;
        if (!p.e.pool) {
            const Pixel x = pixel(u);
            if (!x.ok) continue;
            a = value(u, x, u == first_u);
            if (p.e.plane) {
                dst = p.e.y + ((long)x.n * p.e.N + col) * p.e.plane + (x.row - (long)x.n * p.e.plane);
                dst[0] = a.x; dst[p.e.plane] = a.y; dst[2L * p.e.plane] = a.z; dst[3L * p.e.plane] = a.w;
                continue;
            }
            dst = p.e.y + x.row * p.e.ldy + col;
        } else {
            const int hw = p.bw >> 1, hh = p.bh >> 1;
            const int r00 = ((u / (hw * hh)) * p.bh + 2 * (u / hw % hh)) * p.bw + 2 * (u % hw);
            const Pixel x = pixel(r00);         // (extents and boxes are even: a window lies inside or outside)
            if (!x.ok) continue;
            a = make_float4(-1e8f, -1e8f, -1e8f, -1e8f);        // the reference's identity
#pragma unroll 1
            for (int k = 0; k < 4; k++) {
                const float4 b = value(r00 + (k >> 1) * p.bw + (k & 1), x, false);
                a.x = b.x > a.x ? b.x : a.x; a.y = b.y > a.y ? b.y : a.y; a.z = b.z > a.z ? b.z : a.z; a.w = b.w > a.w ? b.w : a.w;
            }
            dst = p.e.y + (((long)x.n * (p.OH >> 1) + (x.oh >> 1)) * (p.OW >> 1) + (x.ow >> 1)) * p.e.ldy + col;
        }
        if (p.e.tma_store) *reinterpret_cast<float4 *>(dst) = a;        // (16-byte aligned rows)
        else {
            dst[0] = a.x;
            if (col + 1 < p.e.N) dst[1] = a.y;
            if (col + 2 < p.e.N) dst[2] = a.z;
            if (col + 3 < p.e.N) dst[3] = a.w;
        }
    }
}

// ------------------------------------------------------------------- kernel
// GATHER: warps 10-13 build the A tile (compiled apart so that the common variants, which launch ten warps, are not
// held to the register budget of fourteen).
// CLUSTER: a tile's K is cut over the k_splits CTAs of a cluster, one tile per cluster (cluster_epilogue).
// LEAN: only what epilogue_lean does.
// RESIDUAL: a folded shortcut besides, its slabs through shared memory by cp.async in coalesced rows, a tile ahead of their use: read
// by the lanes that add them, each its own row, they kept 32 KB per SM in flight, and a slab took an epilogue group 3300 to
// 4800 cycles where one without a shortcut takes 1500.  ResNet-50 b64 2234 -> 2042 us (expansions of 14 x 14 planes 41 -> 31 us, 28 x 28
// 67 -> 48, 56 x 56 112 -> 89); one K block per stage, for with two the 128 KB of ring hold two stages (2300 us).
template <int BLOCK_N, bool THREE, bool PROMOTE, bool GATHER, bool CLUSTER, bool LEAN, bool RESIDUAL>
__global__ void __launch_bounds__((THREE || GATHER) ? 448 : 320, 1)
gemm_tf32_tcgen05_kernel(const __grid_constant__ typename ParamsOf<GATHER>::type p) {
    using C = Cfg<BLOCK_N, THREE, GATHER>;
    constexpr int STAGES = C::STAGES;                   // barrier slots; the ring uses the first p.stages of them
    // The swizzle pattern repeats every 1024 bytes.  The compiler makes faster code of the variants where it does not see that the ring
    // begins at such an address (7x7, 88 -> 40 at 9 images of 78 x 78 124 and 115 us, VGG-16 b8 in 3xTF32 1546 and 1525, ResNet-50 b64 2017
    // and 2004, the deep belief network 128.3 and 126.2; but 1x1, 3 -> 257 at 25 of 68 x 73 72 and 75), and of the plain 64-wide one where it
    // does not see either that it is shared memory (1x1, 128 -> 24 at 50 of 62 x 62 75 and 72).
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw;
    if constexpr (BLOCK_N == 64 && !THREE && !PROMOTE && !GATHER && !CLUSTER && !LEAN) {
        asm volatile("" : "+l"(smem));
    } else {
        uint32_t offset = 0;
        asm volatile("" : "+r"(offset));
        smem += offset;
    }
    // per stage: [A | B], 3xTF32 [A | B | B_lo] (gathered: [A | B | A_lo | B_lo]), or [A0 | A1 | B0 | B1] with two K blocks per stage
    const int cbs = THREE ? 1 : p.cbs;
    const int stages = p.stages;
    const int a_region = (THREE || cbs == 1) ? A_STAGE_BYTES : p.a_region, a_slice = (THREE || cbs == 1) ? A_STAGE_BYTES : p.a_slice_bytes;
    const int stage_bytes = p.stage_bytes;
    const int halves = (THREE || PROMOTE || BLOCK_N > 128) ? 1 : p.halves;
    const int acc_cols = halves * BLOCK_N;              // TMEM columns of one accumulator set
    // 3xTF32 with several partial sums per tile: the two small cross terms (a_lo*b_hi + a_hi*b_lo) accumulate in a set of
    // columns of their own for the whole tile (their magnitude is 2^-11 of the product's, so what the tensor core's
    // truncating accumulation loses on them is nothing), one set per tile parity behind the two product accumulators.
    // Only the hi*hi chain is then promoted, and a K block adds 4 MMAs to it instead of 12: a third of the promotions
    // for the same chain length.
    const bool cross_cols = THREE && p.parts > 1;
    const uint32_t tmem_cols = C::TS ? 512u : (uint32_t)(C::TMEM_COLS * (THREE ? 2 : halves));
    uint8_t *out_stage = smem + STAGES * C::STAGE_BYTES;      // 2 x [128 rows][32 floats], 128B-swizzled
    uint64_t *bars = (uint64_t *)(out_stage + 2 * C::OUT_STAGE_BYTES);
    uint64_t *full = bars;                    // TMA -> (splitter or MMA)
    uint64_t *empty = bars + STAGES;          // MMA -> TMA
    uint64_t *split = bars + 2 * STAGES;      // splitter -> MMA (three-pass only)
    uint64_t *acc_full = bars + 3 * STAGES;   // MMA -> epilogue   [2]
    uint64_t *acc_empty = acc_full + 2;       // epilogue -> MMA   [2]
    uint64_t *x_empty = acc_empty + 2;        // epilogue -> MMA: the cross terms have been read (where there is one set)
    uint32_t *tmem_slot = (uint32_t *)(x_empty + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    // per epilogue group: scale [BLOCK_N / 2] then shift [BLOCK_N / 2] of the columns of its slabs
    float *aff_base = (float *)((uint8_t *)bars + 256);
    const bool aff_smem = LEAN || (!THREE && !PROMOTE && p.e.shift != nullptr && p.e.lstm_H == 0);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int total_tiles = p.m_tiles * p.n_tiles * p.k_splits;

    if (!GATHER) grid_dependents_start();       // (the gather variants run in stream order on both sides: gemm_tc)
    if (threadIdx.x == 0) {
        if (!GATHER) prefetch_tensor_map(&p.tm_a);
        prefetch_tensor_map(&p.tm_b);
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], GATHER ? 129 : 1);
            mbar_init(&empty[s], 1);
            mbar_init(&split[s], 128);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 256);
        }
        mbar_init(x_empty, 256);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // A pixel box of fewer than 128 rows leaves the tail rows of every A stage unwritten by TMA, and the MMA reads
    // all 128: those rows only feed accumulator rows that are never stored, but they are given a defined value
    // (zero) once, here; no copy touches them afterwards.
    {
        const int box_rows = (GATHER || p.col3) ? BLOCK_M : p.bw * p.bh * p.bn;
        if (box_rows < BLOCK_M) {
            const int tail16 = (BLOCK_M - box_rows) * 8;          // 16-byte chunks per stage tail
            for (int i = threadIdx.x; i < stages * tail16; i += blockDim.x) {
                const int s = i / tail16, c = i - s * tail16;
                reinterpret_cast<float4 *>(smem + s * stage_bytes + cbs * box_rows * 128)[c] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------ TMA producer
        // One elected lane runs the loop and issues every copy.  (Measured: running the loop and the waits in all 32 lanes
        // with only the copies elected -- uniform control flow -- changes nothing for narrow tiles and costs 256-wide
        // tiles 2 %.)
        const bool leader = elect_one();
        if (leader) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        TileIter ti(p, blockIdx.x, gridDim.x);
        const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), ring0 = smem_u32(smem);
        uint32_t sa = ring0;            // the current stage
        const uint32_t tx_bytes = (!THREE && p.col3)
            ? (uint32_t)(p.a_box_bytes + 3 * C::B_STAGE_BYTES)
            : (uint32_t)(((GATHER ? 0 : p.tx_bytes_a) + C::B_STAGE_BYTES * (THREE ? 2 : 1)) * cbs);
        // The first tile's weights fill the ring while the kernels in front still run; only the activations wait for them.
        int primed = 0;
        if (p.b_static) {
            const int kb0 = ti.split * p.kb_per_split, kb_end = min(kb0 + p.kb_per_split, p.num_k_blocks);
            const bool cols = !THREE && p.col3;
            const int loads = cols ? p.ksize_w * p.c_blocks : (kb_end - kb0 + cbs - 1) / cbs;
            primed = min(stages, loads);
            for (int i = 0; i < primed; i++) {
                uint8_t *sa = smem + i * stage_bytes;
                mbar_expect_tx(&full[i], tx_bytes);
                if (cols) {
                    const int cb3 = i / p.ksize_w;
                    tma_load_4d(sa + p.a_box_bytes, &p.tm_b, &full[i], cb3 * BLOCK_K, ti.n_tile * BLOCK_N, i - cb3 * p.ksize_w, 0);
                    continue;
                }
                const int kb = kb0 + i * cbs, tap = kb / p.c_blocks, cb = kb - tap * p.c_blocks;
                uint8_t *sb = sa + a_region;
                if (cbs == 2) {
                    tma_load_4d(sb, &p.tm_b, &full[i], 0, ti.n_tile * BLOCK_N, cb, tap);
                } else {
                    tma_load_3d(sb, &p.tm_b, &full[i], cb * BLOCK_K, ti.n_tile * BLOCK_N, tap);
                    if (THREE)
                        tma_load_3d(sb + C::B_LO_OFFSET, &p.tm_b_lo, &full[i], cb * BLOCK_K, ti.n_tile * BLOCK_N, tap);
                }
            }
        }
        grid_dependency_wait();
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ti.next(p)) {
            const int split = ti.split, n_tile = ti.n_tile, tw = ti.tw, th = ti.th, tn = ti.tn;
            const int w0 = tw * p.bw * p.stride - p.pad_w;
            const int h0 = th * p.bh * halves * p.stride - p.pad_h;
            const int n0 = tn * p.bn;
            const int kb0 = split * p.kb_per_split;
            const int kb_end = min(kb0 + p.kb_per_split, p.num_k_blocks);      // the last split may be shorter
            if (!THREE && p.col3) {
                // two requests per stage: the activation box and the three weight tiles of this filter column
                // (tm_b is 4-D here, {C, N, kw, kh}: a box of one kw and all three kh)
                for (int cb3 = 0; cb3 < p.c_blocks && ok; cb3++) {       // kw fastest, then the channel slice
                    for (int kw3 = 0; kw3 < p.ksize_w; kw3++) {
                        if (!(ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, p.status))) break;
                        const uint32_t bar = full0 + 8 * stage;
                        const bool b_there = primed > 0;
                        if (b_there) primed--;
                        else mbar_expect_tx(bar, tx_bytes);
                        tma_load_4d(sa, &p.tm_a, bar, cb3 * BLOCK_K, w0 + kw3, h0, n0);
                        if (!b_there)
                            tma_load_4d(sa + p.a_box_bytes, &p.tm_b, bar, cb3 * BLOCK_K, n_tile * BLOCK_N, kw3, 0);
                        sa += stage_bytes;
                        if (++stage == stages) { stage = 0; phase ^= 1; sa = ring0; }
                    }
                }
                continue;
            }
            int tap = 0, cb = 0, kh = 0, kw = 0;
            if (kb0) {
                tap = kb0 / p.c_blocks; cb = kb0 - tap * p.c_blocks;
                kh = tap / p.ksize_w; kw = tap - kh * p.ksize_w;
            }
            for (int kb = kb0; kb < kb_end; kb += cbs) {
                if (!(ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, p.status))) break;
                const uint32_t bar = full0 + 8 * stage, sb = sa + a_region;
                const bool b_there = primed > 0;
                if (b_there) primed--;
                else mbar_expect_tx(bar, tx_bytes);
                if (cbs == 2) {
                    tma_load_5d(sa, &p.tm_a, bar, 0, w0 + kw, h0 + kh, n0, cb);
                    if (!b_there) tma_load_4d(sb, &p.tm_b, bar, 0, n_tile * BLOCK_N, cb, tap);
                } else {
                    if (!GATHER) tma_load_4d(sa, &p.tm_a, bar, cb * BLOCK_K, w0 + kw, h0 + kh, n0);
                    if (!b_there) {
                        tma_load_3d(sb, &p.tm_b, bar, cb * BLOCK_K, n_tile * BLOCK_N, tap);
                        if (THREE)
                            tma_load_3d(sb + C::B_LO_OFFSET, &p.tm_b_lo, bar, cb * BLOCK_K,
                                        n_tile * BLOCK_N, tap);
                    }
                }
                if ((cb += cbs) == p.c_blocks) {
                    cb = 0; tap++;
                    if (++kw == p.ksize_w) { kw = 0; kh++; }
                }
                sa += stage_bytes;
                if (++stage == stages) { stage = 0; phase ^= 1; sa = ring0; }
            }
        }
        // Tail: the MMA warp's last release of every stage (an mbarrier arrive that the tensor core performs
        // when those MMAs retire) must have landed in this CTA's shared memory before the CTA may exit.
        for (int i = 0; i < stages && ok; i++) {
            ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status);
            if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        }
        __syncwarp();
        if (CLUSTER) cluster_barrier();
    } else if (warp == 1) {
        // -------------------------------------------------------- MMA issuer
        // One elected lane.  Its time per MMA is the tensor core's: about 65 cycles for a 128 x 64 x 8 TF32 MMA, 75 for
        // 128 x 128 x 8 and 138 for 128 x 256 x 8 (the issue blocks while the queue is full), so 64-filter tiles run the
        // tensor core at about half rate whatever the pipeline around it does.
        const bool leader = elect_one();
        if (leader) {
        constexpr uint32_t idesc = make_idesc(BLOCK_M, BLOCK_N);
        int stage = 0;
        uint32_t phase = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        int tile_parity = 0;
        bool ok = true;
        // this lane's instructions between two MMAs are on the critical path of narrow tiles: addresses advance by increments
        const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), ring0 = smem_desc_lo(smem_u32(smem));
        const uint32_t ring_step = (uint32_t)stage_bytes >> 4;
        uint32_t ring = ring0;          // the current stage's descriptor word
        int a_buf = 0;                  // tensor-memory buffer of the next K block's A terms
        uint32_t x_phase = 0;
        grid_dependency_wait();         // the bounded waits below must not count the kernels in front
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            if (!(ok = mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.status))) break;
            tc_fence_after();
            uint32_t d_tmem = tmem_base + (uint32_t)(acc * acc_cols);
            int kb_in_part = 0;
            if (!THREE && p.col3) {
                for (int it = 0; it < p.ksize_w * p.c_blocks; it++) {
                    if (!(ok = mbar_wait(full0 + 8 * stage, phase, abort_flag, p.status))) break;
                    tc_fence_after();
                    const uint32_t b_base = ring + ((uint32_t)p.a_box_bytes >> 4);
#pragma unroll
                    for (int kh3 = 0; kh3 < 3; kh3++) {
                        const uint32_t b_lo = b_base + kh3 * (C::B_STAGE_BYTES >> 4);
                        for (int hf = 0; hf < halves; hf++) {       // image row kh3 (+ 8 for the second half) of the 16 pixels wide box
                            const uint32_t a_lo = ring + (hf * 8 + kh3) * (16 * 128 >> 4);
#pragma unroll
                            for (int k = 0; k < BLOCK_K / UMMA_K; k++)
                                umma_tf32(d_tmem + (uint32_t)(hf * BLOCK_N), smem_desc(a_lo + 2 * k), smem_desc(b_lo + 2 * k),
                                          idesc, (it | kh3 | k) != 0);
                        }
                    }
                    umma_commit(empty0 + 8 * stage);
                    ring += ring_step;
                    if (++stage == stages) { stage = 0; phase ^= 1; ring = ring0; }
                }
                if (ok && leader) umma_commit(&acc_full[acc]);
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                continue;
            }
            const int ksplit = p.k_splits > 1 ? tile % p.k_splits : 0;
            const int tile_kb = min(p.kb_per_split, p.num_k_blocks - ksplit * p.kb_per_split);
            const uint32_t x_tmem = tmem_base + (uint32_t)(2 * BLOCK_N + (C::X_BUFS == 2 ? tile_parity : 0) * BLOCK_N);    // cross terms of this tile
            tile_parity ^= 1;
            if (C::X_BUFS == 1 && cross_cols) {
                if (!(ok = mbar_wait(x_empty, x_phase ^ 1, abort_flag, p.status))) break;
                x_phase ^= 1;
                tc_fence_after();
            }
            for (int kb = 0; kb < tile_kb; kb += cbs, kb_in_part += cbs) {
                if (kb_in_part == p.kb_per_part) {
                    // hand this partial sum to the epilogue warps and restart in the other accumulator
                    if (leader) umma_commit(&acc_full[acc]);
                    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                    if (!(ok = mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.status))) break;
                    tc_fence_after();
                    d_tmem = tmem_base + (uint32_t)(acc * acc_cols);
                    kb_in_part = 0;
                }
                const uint32_t ready = (THREE && !GATHER) ? full0 + 8 * (2 * STAGES + stage) : full0 + 8 * stage;
                if (!(ok = mbar_wait(ready, phase, abort_flag, p.status))) break;
                tc_fence_after();
                uint32_t a_lo = ring, b_lo = ring + ((uint32_t)a_region >> 4);
#pragma unroll 1
                for (int c = 0; c < cbs; c++, a_lo += (uint32_t)a_slice >> 4, b_lo += C::B_STAGE_BYTES >> 4) {
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; k++) {        // +32 bytes per K step = +2 in the descriptor
                        const uint64_t da = smem_desc(a_lo + 2 * k), db = smem_desc(b_lo + 2 * k);
                        if constexpr (C::TS) {
                            const uint64_t db_lo = smem_desc(b_lo + (C::B_LO_OFFSET >> 4) + 2 * k);
                            const uint32_t ta = tmem_base + (uint32_t)(C::A_COL + a_buf * 64 + k * UMMA_K), ta_lo = ta + 32;
                            const uint32_t xd = cross_cols ? x_tmem : d_tmem;
                            umma_tf32_ts(xd, ta_lo, db, idesc, ((cross_cols ? kb : kb_in_part) | k) != 0);
                            umma_tf32_ts(xd, ta, db_lo, idesc, 1);
                            umma_tf32_ts(d_tmem, ta, db, idesc, cross_cols ? (kb_in_part | k) != 0 : 1);
                        } else if (THREE) {
                            const uint64_t da_lo = smem_desc(b_lo + (C::B_STAGE_BYTES >> 4) + 2 * k);
                            const uint64_t db_lo = smem_desc(b_lo + (C::B_LO_OFFSET >> 4) + 2 * k);
                            if (cross_cols) {
                                umma_tf32(x_tmem, da_lo, db, idesc, (kb | k) != 0);
                                umma_tf32(x_tmem, da, db_lo, idesc, 1);
                                umma_tf32(d_tmem, da, db, idesc, (kb_in_part | k) != 0);
                            } else {
                                umma_tf32(d_tmem, da_lo, db, idesc, (kb_in_part | k) != 0);
                                umma_tf32(d_tmem, da, db_lo, idesc, 1);
                                umma_tf32(d_tmem, da, db, idesc, 1);
                            }
                        } else {
                            umma_tf32(d_tmem, da, db, idesc, (kb_in_part | c | k) != 0);
                        }
                    }
                }
                umma_commit(empty0 + 8 * stage);     // frees the stage (and A's buffer) once these MMAs have read it
                if (C::TS && ++a_buf == C::A_BUFS) a_buf = 0;
                ring += ring_step;
                if (++stage == stages) { stage = 0; phase ^= 1; ring = ring0; }
            }
            if (ok && leader) umma_commit(&acc_full[acc]);
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        }
        __syncwarp();
        if (CLUSTER) cluster_barrier();
    } else if (CLUSTER && warp < 10) {
        if constexpr (CLUSTER)
            cluster_epilogue<BLOCK_N, THREE, PROMOTE>(p, smem, tmem_base, acc_full, acc_empty, cross_cols, abort_flag);
    } else if (warp < 10) {
        // ---------------------------------------------------------- epilogue
        // Two groups of four warps; group g owns the 32-column slabs of parity g, its own staging
        // buffer, named barrier and TMA-store thread, so two slabs are in flight per tile and every
        // scheduler has two epilogue warps to alternate between.
        const int ew = warp - 2;                // 0..7
        const int grp = ew >> 2;
        const int bar_id = 1 + grp;
        const int q = warp & 3;                 // TMEM lane quarter this warp may read
        const int r = q * 32 + lane;            // row inside the tile
        const int t = (ew & 3) * 32 + lane;     // index inside the group
        const int rw = r % p.bw, rh = (r / p.bw) % p.bh, rn = r / (p.bw * p.bh);
        const bool store_thread = t == 0;
        constexpr int CH = BLOCK_N >= 64 ? BLOCK_N / 64 : 1;    // 32-column slabs per group
        float4 *slab0 = reinterpret_cast<float4 *>(out_stage + grp * C::OUT_STAGE_BYTES);
        float4 *slab1 = p.slab2_offset ? reinterpret_cast<float4 *>(smem + p.slab2_offset + grp * C::OUT_STAGE_BYTES) : slab0;
        const int stores_in_flight = p.slab2_offset ? 1 : 0;
        float4 *slab = slab0;
        int aff_tile = -1;
        int epi_tile_parity = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        TileIter ti(p, blockIdx.x, gridDim.x);
        // RESIDUAL: slab buffers of 32 rows per warp (one per slab of a tile) behind the shorter ring, and the tile the next copies are for
        [[maybe_unused]] TileIter ahead = ti;
        [[maybe_unused]] int ahead_tile = blockIdx.x;
        [[maybe_unused]] const uint32_t res_buf = smem_u32(smem) + RESIDUAL_OFFSET + (uint32_t)ew * (CH * 4096);
        [[maybe_unused]] auto fetch_residual = [&](int ci) {        // slab ci of tile `ahead`
            if (ahead_tile >= total_tiles) return;
            const int w = ahead.tw * p.bw + rw, h = ahead.th * p.bh + rh, n = ahead.tn * p.bn + rn;
            const int ih = h * p.e.res_stride, iw = w * p.e.res_stride;
            const bool in = rn < p.bn && w < p.OW && h < p.OH && n < p.NB && h < p.e.res_h && w < p.e.res_w && ih < p.e.res_h && iw < p.e.res_w;
            const int pixel = in ? (n * p.e.res_h + ih) * p.e.res_w + iw : -1;      // this lane's row
            const int col = ahead.n_tile * BLOCK_N + (grp + 2 * ci) * 32 + 4 * (lane & 7);
#pragma unroll
            for (int i = 0; i < 8; i++) {               // eight lanes a row, four rows at a time
                const int row = 4 * i + (lane >> 3), px = __shfl_sync(0xffffffffu, pixel, row);
                const bool ok = px >= 0 && col < p.e.addend_cols;
                cp_async16(res_buf + (uint32_t)(ci * 4096 + row * 128 + ((lane & 7) ^ (row & 7)) * 16),
                           ok ? p.e.addend + (long)px * p.e.ld_addend + col : p.e.addend, ok);
            }
        };
        grid_dependency_wait();                 // (addends, cell states; the outputs may still be read)
        if constexpr (RESIDUAL) {
#pragma unroll
            for (int ci = 0; ci < CH; ci++) fetch_residual(ci);
            ahead.next(p); ahead_tile += gridDim.x;
        }
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ti.next(p)) {
            const int split = ti.split, n_tile = ti.n_tile, tw = ti.tw, th = ti.th, tn = ti.tn;
            const int ow = tw * p.bw + rw, oh = th * p.bh * halves + rh, n = tn * p.bn + rn;
            const bool row_ok = (rn < p.bn) && ow < p.OW && oh < p.OH && n < p.NB;
            const long row = ((long)n * p.OH + oh) * p.OW + ow;
            const EpiRow erow{r, row, row_ok, RESIDUAL ? nullptr : addend_row(p.e, row_ok, row, n, oh, ow)};
            const EpiBox ebox{p.bw, p.bh, p.bn, tw * p.bw, th * p.bh * halves, tn * p.bn + split * p.NB};
            if (aff_smem && n_tile != aff_tile) {
                // this group's scale/shift values for the tile column (its slabs are chunks grp, grp + 2, ...)
                float *ga = aff_base + grp * BLOCK_N;
                epilogue_bar_sync(bar_id);          // the previous column's values are no longer read
                if (t < BLOCK_N / 2) {
                    const int col = n_tile * BLOCK_N + (grp + 2 * (t >> 5)) * 32 + (t & 31);
                    const bool in = col < ((p.e.N + 31) & ~31);     // the vectors are padded to a multiple of 32
                    ga[t] = (in && p.e.scale) ? p.e.scale[col] : 1.0f;
                    ga[BLOCK_N / 2 + t] = in ? p.e.shift[col] : 0.0f;
                }
                epilogue_bar_sync(bar_id);
                aff_tile = n_tile;
            }
            if (erow.arow) {
                // The addend (a residual tensor, the LSTM's input-side projection) comes from DRAM and each slab's
                // 128 bytes of it are needed only once the accumulators are in registers: start this group's lines
                // towards L2 now, while the tile's MMAs still run.
#pragma unroll 1
                for (int chunk = grp; chunk < BLOCK_N / 32; chunk += 2) {
                    const int col0 = n_tile * BLOCK_N + chunk * 32;
                    if (col0 >= p.e.addend_cols) break;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(erow.arow + col0));
                }
            }
            if (!PROMOTE || p.parts == 1) {
                if (!(ok = epilogue_all(mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.status), bar_id))) break;
                tc_fence_after();
                uint32_t v[32];
                bool loaded = false;            // v holds a tcgen05.ld issued while the previous slab was being stored
                if constexpr (RESIDUAL) {
                    asm volatile("cp.async.wait_all;" ::: "memory");        // this tile's slabs, under way since the tile before
                    __syncwarp();
                }
#pragma unroll 1
                for (int hf = 0; hf < halves; hf++) {
                    // the second half of a two-box tile: the same raster p.bh image rows further down
                    EpiRow hrow = erow;
                    EpiBox hbox = ebox;
                    if (hf) {
                        const int oh2 = oh + p.bh;
                        hrow.row_ok = (rn < p.bn) && ow < p.OW && oh2 < p.OH && n < p.NB;
                        hrow.grow = ((long)n * p.OH + oh2) * p.OW + ow;
                        hrow.arow = addend_row(p.e, hrow.row_ok, hrow.grow, n, oh2, ow);
                        hbox.oh0 += p.bh;
                    }
#pragma unroll 1
                    for (int chunk = grp; chunk < BLOCK_N / 32; chunk += 2) {
                        const int col0 = n_tile * BLOCK_N + chunk * 32;
                        if (col0 >= p.e.N) {              // uniform across the group
                            if constexpr (RESIDUAL) { fetch_residual(chunk >> 1); continue; }
                            break;
                        }
                        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * acc_cols + hf * BLOCK_N + chunk * 32);
                        if (!loaded) tmem_ld_32x32(taddr, v);
                        tmem_ld_wait();
                        loaded = false;
                        // this group's next slab of the tile: the next pair of columns, else the first of the other half
                        uint32_t next = 0;
                        if (PROMOTE) {}         // (those variants have no registers to spare for it)
                        else if (chunk + 2 < BLOCK_N / 32 && col0 + 64 < p.e.N) next = taddr + 64;
                        else if (hf + 1 < halves) next = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * acc_cols + (hf + 1) * BLOCK_N + grp * 32);
                        const float *aff = aff_smem ? aff_base + grp * BLOCK_N + (chunk >> 1) * 32 : nullptr;
                        auto staged = [&] { if (next) { tmem_ld_32x32(next, v); loaded = true; } };
                        if constexpr (RESIDUAL) {
                            epilogue_lean(p.e, &p.tm_y, v, col0, hrow, hbox, slab, bar_id, store_thread, stores_in_flight, staged, aff, BLOCK_N / 2,
                                          [&](uint32_t (&x)[32]) {
                                if (col0 < p.e.addend_cols) {
#pragma unroll
                                    for (int j = 0; j < 8; j++) {
                                        float4 a;
                                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
                                                     : "r"(res_buf + (uint32_t)((chunk >> 1) * 4096 + lane * 128 + (j ^ (lane & 7)) * 16)));
                                        x[4 * j] = __float_as_uint(__uint_as_float(x[4 * j]) + a.x);
                                        x[4 * j + 1] = __float_as_uint(__uint_as_float(x[4 * j + 1]) + a.y);
                                        x[4 * j + 2] = __float_as_uint(__uint_as_float(x[4 * j + 2]) + a.z);
                                        x[4 * j + 3] = __float_as_uint(__uint_as_float(x[4 * j + 3]) + a.w);
                                    }
                                }
                                __syncwarp();               // the buffer has been read
                                fetch_residual(chunk >> 1);
                            });
                        } else if constexpr (LEAN)
                            epilogue_lean(p.e, &p.tm_y, v, col0, hrow, hbox, slab, bar_id, store_thread, stores_in_flight, staged, aff, BLOCK_N / 2,
                                          [&](uint32_t (&x)[32]) { if (hrow.arow) add_quads(p.e, x, hrow.arow, col0); });
                        else
                            epilogue_chunk<THREE>(p.e, &p.tm_y, &p.tm_yp, v, col0, hrow, hbox, slab, bar_id, store_thread, t, stores_in_flight, staged,
                                                  aff, BLOCK_N / 2);
                        slab = slab == slab0 ? slab1 : slab0;
                    }
                }
                if constexpr (RESIDUAL) { ahead.next(p); ahead_tile += gridDim.x; }
                tc_fence_before();
                mbar_arrive(&acc_empty[acc]);
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
            } else if constexpr (PROMOTE) {
                // promoted accumulation: this group's slabs of every partial sum are added in registers
                uint32_t sum[CH][32];
                const int tile_kb = min(p.kb_per_split, p.num_k_blocks - split * p.kb_per_split);
                const int parts = (tile_kb + p.kb_per_part - 1) / p.kb_per_part;
                const uint32_t x_cols = (uint32_t)(2 * BLOCK_N + (C::X_BUFS == 2 ? epi_tile_parity : 0) * BLOCK_N);
                epi_tile_parity ^= 1;
                for (int part = 0; part < parts && ok; part++) {
                    if (!(ok = epilogue_all(mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.status), bar_id))) break;
                    tc_fence_after();
#pragma unroll
                    for (int ci = 0; ci < CH; ci++) {
                        const int chunk = grp + 2 * ci;
                        if (chunk * 32 < BLOCK_N && n_tile * BLOCK_N + chunk * 32 < p.e.N) {
                            uint32_t v[32];
                            tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BLOCK_N + chunk * 32), v);
                            tmem_ld_wait();
                            if (part == 0) {
#pragma unroll
                                for (int j = 0; j < 32; j++) sum[ci][j] = v[j];
                            } else {
#pragma unroll
                                for (int j = 0; j < 32; j++)
                                    sum[ci][j] = __float_as_uint(__uint_as_float(sum[ci][j]) + __uint_as_float(v[j]));
                            }
                            if (cross_cols && part == parts - 1) {      // the tile's cross terms: complete with its last MMAs
                                tmem_ld_32x32(tmem_base + ((uint32_t)(q * 32) << 16) + x_cols + (uint32_t)(chunk * 32), v);
                                tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 32; j++)
                                    sum[ci][j] = __float_as_uint(__uint_as_float(sum[ci][j]) + __uint_as_float(v[j]));
                            }
                        }
                    }
                    tc_fence_before();
                    mbar_arrive(&acc_empty[acc]);
                    if (C::X_BUFS == 1 && cross_cols && part == parts - 1) mbar_arrive(x_empty);
                    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
                }
                if (!ok) break;
#pragma unroll
                for (int ci = 0; ci < CH; ci++) {
                    const int chunk = grp + 2 * ci;
                    const int col0 = n_tile * BLOCK_N + chunk * 32;
                    if (chunk * 32 < BLOCK_N && col0 < p.e.N)
                        epilogue_chunk<THREE>(p.e, &p.tm_y, &p.tm_yp, sum[ci], col0, erow, ebox, slab0, bar_id, store_thread, t, 0, [] {});
                }
            }
        }
        if (store_thread) tma_store_wait_all();     // staged tiles must have left shared memory
        if constexpr (RESIDUAL) asm volatile("cp.async.wait_all;" ::: "memory");
    } else if constexpr (GATHER) {
        // ------------------------------------------------- in-kernel patch gather
        // One thread per tile row (output pixel): 32 columns (kh,kw,c) of this K block are read
        // through the cache (neighbouring threads read neighbouring pixels) and written as one
        // 128-byte swizzled row, TF32-rounded (or split into hi/lo for the three-pass kernel).
        grid_dependency_wait();
        const int t = threadIdx.x - 320;
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            const int m_tile = tile / p.k_splits / p.n_tiles;
            const long m = (long)m_tile * BLOCK_M + t;
            const bool valid = m < p.gM;
            int ih0 = 0, iw0 = 0;
            const float *base = p.gx;
            if (valid) {
                const int per = p.gOH * p.gOW;
                const int n = (int)(m / per), rem = (int)(m - (long)n * per);
                const int oh = rem / p.gOW, ow = rem - oh * p.gOW;
                ih0 = oh * p.gstride; iw0 = ow * p.gstride;
                base = p.gx + (long)n * p.gsn + (long)ih0 * p.gsh + (long)iw0 * p.gsw;
            }
            // does every tap of this pixel fall inside the image?  (true for all but border pixels)
            const int ihf = ih0 - p.gpad, iwf = iw0 - p.gpad;
            const bool interior = valid && ihf >= 0 && iwf >= 0 && ihf + p.gks <= p.gH && iwf + p.gks <= p.gW;
            for (int kb = 0; kb < p.kb_per_split; kb++) {        // gather mode never splits K
                if (!(ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status))) break;
                float4 *a_row = reinterpret_cast<float4 *>(smem + stage * C::STAGE_BYTES + t * 128);
                float4 *a_lo_row = reinterpret_cast<float4 *>(smem + stage * C::STAGE_BYTES + A_STAGE_BYTES + C::B_STAGE_BYTES + t * 128);
                const int2 *tab = p.gtab + kb * BLOCK_K;        // kernel-parameter (constant bank) table
                float x[32];
                if (interior) {
#pragma unroll
                    for (int i = 0; i < 32; i++)                // 32 independent loads in flight
                        x[i] = (kb * BLOCK_K + i < p.gK) ? __ldg(base + tab[i].x) : 0.0f;
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const int ih = ih0 + (int)(short)(tab[i].y & 0xffff), iw = iw0 + (tab[i].y >> 16);
                        const bool inb = valid && kb * BLOCK_K + i < p.gK && ih >= 0 && ih < p.gH && iw >= 0 && iw < p.gW;
                        x[i] = inb ? __ldg(base + tab[i].x) : 0.0f;
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    float v[4], lo[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (THREE) {
                            v[e] = round_tf32(x[4 * j + e]);
                            lo[e] = round_tf32(x[4 * j + e] - v[e]);
                        } else {
                            v[e] = p.ground ? round_tf32(x[4 * j + e]) : x[4 * j + e];
                        }
                    }
                    a_row[j ^ (t & 7)] = make_float4(v[0], v[1], v[2], v[3]);
                    if (THREE) a_lo_row[j ^ (t & 7)] = make_float4(lo[0], lo[1], lo[2], lo[3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive(&full[stage]);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if constexpr (THREE) {
        // ---------------------------------------------- hi/lo operand splitter
        // hi = RN_tf32(x) in integer arithmetic (cvt.rna runs at a quarter of that rate and was the pace of this kernel:
        // VGG-16 b8 1951 us with two of them per value, 1871 with one, 1756 with none); lo = x - hi, exact.  With ulp the
        // spacing of x, lo is a whole number of ulp up to 2^12, so its 11 leading bits lose the last bit of some odd numbers
        // above 2^11: one ulp(x), whether the tensor core's truncation drops it or a rounding moves that tie, and lo's
        // sign does not depend on x, so there is no bias.  A NaN whose payload overflows the addition survives in lo.
        // A thread owns a row: it reads the row's eight 16-byte chunks at their swizzled places (eight rows of a read fall into
        // different banks) and writes the two terms as 32 columns each of its tensor-memory lane.
        const int q = warp & 3, r = q * 32 + lane;      // TMEM lane quarter this warp may write
        grid_dependency_wait();
        int stage = 0, buf = 0;
        uint32_t phase = 0;
        int back = stages - C::A_BUFS;          // stage and phase of the K block A_BUFS before this one
        uint32_t back_phase = 1;
        long seen = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            const int tile_kb = min(p.kb_per_split, p.num_k_blocks - (tile % p.k_splits) * p.kb_per_split);
            for (int kb = 0; kb < tile_kb; kb++, seen++) {
                if (!(ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, p.status)))) break;
                const float4 *a = reinterpret_cast<const float4 *>(smem + stage * C::STAGE_BYTES + r * 128);
                uint32_t hi[32], lo[32];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 x = a[j ^ (r & 7)];
                    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        hi[4 * j + e] = (__float_as_uint(v[e]) + 0x1000u) & 0xFFFFE000u;
                        lo[4 * j + e] = __float_as_uint(v[e] - __uint_as_float(hi[4 * j + e]));
                    }
                }
                // the buffer is free when the MMAs of the K block that used it last have retired (they also freed its stage)
                if (seen >= C::A_BUFS && !(ok = __all_sync(0xffffffffu, mbar_wait(&empty[back], back_phase, abort_flag, p.status)))) break;
                tc_fence_after();
                const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(C::A_COL + buf * 64);
                tmem_st_32x32(ta, hi);
                tmem_st_32x32(ta + 32, lo);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&split[stage]);
                if (++stage == stages) { stage = 0; phase ^= 1; }
                if (++back == stages) { back = 0; back_phase ^= 1; }
                if (++buf == C::A_BUFS) buf = 0;
            }
        }
        __syncwarp();
        if (CLUSTER) cluster_barrier();
    }

    // ------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // give copies and MMAs still in flight time to land before TMEM is released
        for (int i = 0; i < 64; i++) __nanosleep(2000);
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    if (CLUSTER) {          // no CTA leaves while a peer reads its partial sums
        __syncwarp();
        cluster_barrier();
    }
}

// ---------------------------------------------------------------- host side
struct Box { int bw, bh, bn; };

// Chooses the (bw x bh x bn) pixel box (<= 128 rows) that wastes the fewest MMA rows.  Among equally full boxes the
// one that spans the fewest images wins (its rows are the longest contiguous runs in memory), then the widest.
// bn_divides: the images of a box must not run past the batch (split-K slabs follow each other in y)
// image_bytes: size of one image of the A tensor -- a box that runs past the batch makes the load unit read that many
// bytes per missing image behind the tensor, so such boxes are only taken while that stays small
Box choose_box(int OW, int OH, int NB, int stride, bool even, bool bn_divides, double image_bytes) {
    Box best{1, 1, 1};
    double best_eff = -1;
    const int max_dim = 256 / std::max(1, stride);     // TMA box extent limit (elements traversed)
    for (int bw = 1; bw <= std::min({OW, 128, max_dim}); bw++) {
        const int rem = 128 / bw;
        for (int bh = 1; bh <= std::min({OH, rem, max_dim}); bh++) {
            int bn = std::min({NB, 128 / (bw * bh), 256});
            if (bn < 1) continue;
            while ((bn_divides || (double)(((NB + bn - 1) / bn) * bn - NB) * image_bytes > 4e6) && NB % bn) bn--;
            if (even && ((bw | bh) & 1)) continue;      // 2x2 pooling windows must not straddle tiles
            auto eff1 = [](int ext, int b) { return (double)ext / ((double)((ext + b - 1) / b) * b); };
            double eff = eff1(OW, bw) * eff1(OH, bh) * eff1(NB, bn) * (double)(bw * bh * bn) / 128.0;
            eff += 1e-6 * bw + 1e-4 / bn;
            if (eff > best_eff) { best_eff = eff; best = Box{bw, bh, bn}; }
        }
    }
    return best;
}

// A box of whole 8-row groups that covers the plane with no more tiles, where there is one: its K slices can then be
// fetched in pairs.  Rows of the box past the plane are zero-filled loads and clipped stores.  The limits are choose_box's: a
// TMA box traverses at most 256 elements per dimension, and what it reads behind the tensor stays under 4 MB.
Box whole_groups(Box box, int OW, int OH, int stride, bool even, double row_bytes) {
    if ((box.bw * box.bh * box.bn) % 8 == 0) return box;
    const int max_dim = 256 / std::max(1, stride);
    if (OH == 1) {                      // a plain matrix: its rows lie along w
        const int bw = (box.bw + 7) / 8 * 8;
        return bw <= max_dim && bw * box.bn <= BLOCK_M && (OW + bw - 1) / bw <= (OW + box.bw - 1) / box.bw ? Box{bw, 1, box.bn} : box;
    }
    const int tiles = (OH + box.bh - 1) / box.bh;
    for (int d = 1; d < 8; d++)
        for (int bh : {box.bh + d, box.bh - d}) {
            if (bh < 1 || bh > max_dim || (even && (bh & 1)) || (box.bw * bh * box.bn) % 8 || box.bw * bh * box.bn > BLOCK_M) continue;
            const int t = (OH + bh - 1) / bh;
            if (t <= tiles && (double)(t * bh - OH) * stride * row_bytes <= 4e6) return Box{box.bw, bh, box.bn};
        }
    return box;
}

// filter-column stages: 3x3 / stride 1, at most 128 input channels and filters (the layers that are bound by
// re-loading activations from L2), a fixed 16 x 8 pixel box; not worth it when the box wastes much of the plane
// (the row-window layout of a layer with <= 4 input channels has the filter columns folded into its "channels":
// three filter rows, one column, no padding in w)
bool column_stages(const ConvGeom &g, int kc, int N) {
    const int ksize_w = g.ksize_w > 0 ? g.ksize_w : g.ksize;
    return g.ksize == 3 && g.stride == 1 && g.pad <= 1 &&
           ((ksize_w == 3 && (g.pad_w < 0 || g.pad_w == g.pad)) || (ksize_w == 1 && g.pad_w == 0)) &&
           kc <= 128 && N <= 128 && g.OW >= 16 && g.OH >= 8 &&
           ((double)g.OW / ((g.OW + 15) / 16 * 16)) * ((double)g.OH / ((g.OH + 7) / 8 * 8)) >= 0.8;
}

void encode(nb_handle_s *h, CUtensorMap *tm, const void *base, int rank, const cuuint64_t *dims,
            const cuuint64_t *strides_bytes, const cuuint32_t *box, const cuuint32_t *elem_strides) {
    encode_tensor_map(h, tm, base, rank, dims, strides_bytes, box, elem_strides);
}

struct Variant { const void *kernel; int smem; };      // takes a TcParams, or a TcGatherParams

template <int BLOCK_N, bool THREE, bool PROMOTE, bool GATHER, bool CLUSTER = false, bool LEAN = false, bool RESIDUAL = false>
Variant variant() { return {(const void *)gemm_tf32_tcgen05_kernel<BLOCK_N, THREE, PROMOTE, GATHER, CLUSTER, LEAN, RESIDUAL>, Cfg<BLOCK_N, THREE, GATHER>::SMEM_BYTES}; }

// index: [gather][three][promote][block_n: 0 = 64, 1 = 128, 2 = 256]; absent combinations are null
const Variant VARIANTS[2][2][2][3] = {
    {{{variant<64, false, false, false>(), variant<128, false, false, false>(), variant<256, false, false, false>()},
      {variant<64, false, true, false>(), variant<128, false, true, false>(), {nullptr, 0}}},
     {{{nullptr, 0}, {nullptr, 0}, {nullptr, 0}},
      {variant<64, true, true, false>(), variant<128, true, true, false>(), {nullptr, 0}}}},
    {{{variant<64, false, false, true>(), variant<128, false, false, true>(), {nullptr, 0}},
      {{nullptr, 0}, {nullptr, 0}, {nullptr, 0}}},
     {{{nullptr, 0}, {nullptr, 0}, {nullptr, 0}},
      {variant<64, true, true, true>(), variant<128, true, true, true>(), {nullptr, 0}}}},
};

// index: [three][promote][block_n]: K cut over clusters (in TF32 no wider tile was ever the better one)
const Variant CLUSTER_VARIANTS[2][2][3] = {
    {{variant<64, false, false, false, true>(), {nullptr, 0}, {nullptr, 0}}, {variant<64, false, true, false, true>(), {nullptr, 0}, {nullptr, 0}}},
    {{{nullptr, 0}, {nullptr, 0}, {nullptr, 0}},
     {variant<64, true, true, false, true>(), variant<128, true, true, false, true>(), {nullptr, 0}}},
};

// index: [block_n]: a folded shortcut through shared memory
const Variant RESIDUAL_VARIANTS[2] = {variant<64, false, false, false, false, true, true>(), variant<128, false, false, false, false, true, true>()};
// index: [block_n]: the plain epilogue by itself
const Variant LEAN_VARIANTS[3] = {variant<64, false, false, false, false, true>(), variant<128, false, false, false, false, true>(),
                                  variant<256, false, false, false, false, true>()};

// One worked-out launch: kernel parameters (tile geometry, tensor maps), kernel variant, grid.
struct TcLaunch : LaunchRecord {
    TcGatherParams p;       // the other variants take the TcParams it starts with
    Variant v;
    bool gather = false;
    int grid = 1, threads = 320, cluster = 1;
    double flops = 0;
    std::string desc;       // names the launch in error messages
};

inline bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

void gemm_tc_prepare_device() {
    for (auto &t : VARIANTS[0])
        for (auto &pr : t)
            for (auto &v : pr)
                if (v.kernel) NB_CHECK_CUDA(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
}

void gemm_tc_load(const nb_handle_s *h, unsigned groups) {
    groups &= ~h->tc_loaded;
    auto load = [](const Variant &v) {
        if (v.kernel) NB_CHECK_CUDA(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
    };
    if (groups & TC_GATHER)
        for (auto &t : VARIANTS[1])
            for (auto &pr : t)
                for (auto &v : pr) load(v);
    if (groups & TC_LEAN)
        for (auto &v : LEAN_VARIANTS) load(v);
    if (groups & TC_RESIDUAL)
        for (auto &v : RESIDUAL_VARIANTS) load(v);
    h->tc_loaded |= groups;
}

// Clusters of `size` CTAs, one per SM, that run at once.  The cluster kernels are loaded by the first layer that they are a
// candidate for, and the device is asked about the sizes that a layer could take, so a handle that has none pays for none.
static int clusters_at_once(const nb_handle_s *h, int size) {
    if (!h->tc_clusters_ready) {
        for (auto &t : CLUSTER_VARIANTS)
            for (auto &pr : t)
                for (auto &v : pr) {
                    if (!v.kernel) continue;
                    NB_CHECK_CUDA(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
                    NB_CHECK_CUDA(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
                }
        std::fill(std::begin(h->tc_clusters), std::end(h->tc_clusters), -1);
        h->tc_clusters_ready = true;
    }
    int &n = h->tc_clusters[size];
    if (n >= 0) return n;
    const Variant &v = CLUSTER_VARIANTS[0][0][0];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = (size_t)v.smem;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)size; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, v.kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    return n;
}

void encode_tensor_map(nb_handle_s *h, CUtensorMap *tm, const void *base, int rank, const cuuint64_t *dims,
                       const cuuint64_t *strides_bytes, const cuuint32_t *box, const cuuint32_t *elem_strides) {
    CUresult r = h->encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void *>(base), dims,
                                 strides_bytes, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(NB_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
}

std::string gemm_args_key(const GemmArgs &a, char tag, int extra) {
    std::string k;
    k.reserve(320);
    k.push_back(tag);
    key_add(k, extra);
    key_add(k, a.a); key_add(k, a.a_is_conv); key_add(k, a.lda);
    const ConvGeom &g = a.g;
    key_add(k, g.batch); key_add(k, g.C); key_add(k, g.H); key_add(k, g.W); key_add(k, g.OH); key_add(k, g.OW);
    key_add(k, g.ksize); key_add(k, g.stride); key_add(k, g.pad); key_add(k, g.ksize_w); key_add(k, g.pad_w);
    key_add(k, g.sn); key_add(k, g.sc); key_add(k, g.sh); key_add(k, g.sw);
    key_add(k, a.a_gather); key_add(k, a.b); key_add(k, a.b_lo); key_add(k, a.ldb);
    key_add(k, a.M); key_add(k, a.N); key_add(k, a.Kc);
    key_add(k, a.scale); key_add(k, a.shift); key_add(k, a.addend); key_add(k, a.ld_addend); key_add(k, a.addend_after_act);
    key_add(k, a.res_stride); key_add(k, a.res_c); key_add(k, a.res_h); key_add(k, a.res_w);
    key_add(k, a.act); key_add(k, a.round_out_tf32); key_add(k, a.y); key_add(k, a.ldy); key_add(k, a.y_nchw); key_add(k, a.y_pool);
    key_add(k, a.lstm_H); key_add(k, a.lstm_c_prev); key_add(k, a.lstm_c); key_add(k, a.lstm_h); key_add(k, a.lstm_h_round);
    key_add(k, a.b_static);
    key_add(k, a.split_k); key_add(k, a.split_cluster); key_add(k, a.block_n_hint); key_add(k, a.k_part); key_add(k, a.algo_flops);
    return k;
}

bool gemm_tc_supported(const nb_handle_s *h, const GemmArgs &a) {
    if (!h->encode_tiled || h->cc_major != 10) return false;
    if (a.a_gather) return (a.Kc % 32) == 0 && a.Kc <= GATHER_MAX_K && (a.ldb % 4) == 0 && aligned16(a.b);
    if (a.Kc < 32 || (a.Kc % 4) != 0 || (a.ldb % 4) != 0 || !aligned16(a.b) || !aligned16(a.a)) return false;
    if (a.a_is_conv) {
        const ConvGeom &g = a.g;
        // NHWC only: channel stride 1 and every other stride a multiple of 4 elements
        if (g.sc != 1 || (g.sw % 4) || (g.sh % 4) || (g.sn % 4)) return false;
        if (g.stride > 8) return false;
    } else {
        if ((a.lda % 4) != 0) return false;
    }
    return true;
}

int tc_blocks_per_split(int c_blocks, int blocks, int S, int block_n) {
    const int per = (blocks + S - 1) / S;
    // whole pairs of K slices per split where that leaves none empty (256-wide tiles do not fetch pairs)
    return per + (S > 1 && c_blocks % 2 == 0 && (per & 1) && block_n <= 128 && (long)(S - 1) * (per + 1) < blocks ? 1 : 0);
}

namespace {

// Works out one launch: tiling, kernel variant, tensor maps; checks that every operand's extent lies inside the
// device allocation its pointer belongs to.
std::unique_ptr<TcLaunch> build_launch(nb_handle_s *h, const GemmArgs &a, bool three_pass) {
    if (!gemm_tc_supported(h, a)) throw Error(NB_ERR_UNSUPPORTED, "operands do not satisfy the TMA layout rules");
    if (a.y_pool && a.a_gather) throw Error(NB_ERR_UNSUPPORTED, "fused pooling is not available with the gathered A operand");
    if (three_pass && !a.b_lo) throw Error(NB_ERR_INVALID_ARG, "three-pass GEMM needs the low-order weight split");
    std::unique_ptr<TcLaunch> L(new TcLaunch());
    TcGatherParams &p = L->p;
    std::memset((void *)&p, 0, sizeof p);

    ConvGeom g;
    const bool gather = a.a_gather;
    if (a.a_is_conv && !gather) {
        g = a.g;
    } else {
        // plain matrix = one image of height 1 and width M with Kc channels, 1x1 filter
        g.batch = 1; g.C = a.Kc; g.H = 1; g.W = a.M; g.OH = 1; g.OW = a.M;
        g.ksize = 1; g.stride = 1; g.pad = 0;
        g.sc = 1; g.sw = a.lda; g.sh = (long)a.lda * a.M; g.sn = (long)a.lda * a.M;
    }
    // Split-K: the K blocks (taps x channel slices) are divided among the `split_k` CTAs of a cluster, or among tiles that each
    // write their own slab of y ([split][batch][OH][OW][N]); the caller then adds the slabs and applies the epilogue.
    const int S = (!gather && a.split_k > 1) ? a.split_k : 1;
    const bool cluster = S > 1 && a.split_cluster;
    const int kc = a.Kc;
    const int ksize_w = g.ksize_w > 0 ? g.ksize_w : g.ksize;
    const int taps = g.ksize * ksize_w;
    const bool pool = a.y_pool != nullptr;
    Box box = choose_box(g.OW, g.OH, g.batch, g.stride, pool, S > 1 && !cluster, (double)g.sn * 4.0);
    const bool col3 = a.a_is_conv && !gather && !three_pass && S == 1 && column_stages(g, kc, a.N);
    const bool pairs = !col3 && !gather && !three_pass && kc % (2 * BLOCK_K) == 0;      // K slices may be fetched in pairs
    if (col3) box = Box{16, 8, 1};
    // two boxes per tile when the plane is tall enough for 16-row tiles not to waste much of it
    const int halves = (col3 && g.OH >= 16 && ((double)g.OW / ((g.OW + 15) / 16 * 16)) * ((double)g.OH / ((g.OH + 15) / 16 * 16)) >= 0.8)
                           ? 2 : 1;
    p.bw = box.bw; p.bh = box.bh; p.bn = box.bn;
    p.tiles_w = (g.OW + box.bw - 1) / box.bw;
    p.tiles_h = (g.OH + box.bh * halves - 1) / (box.bh * halves);
    p.tiles_n = (g.batch + box.bn - 1) / box.bn;
    p.OW = g.OW; p.OH = g.OH; p.NB = g.batch;
    p.ksize_w = ksize_w; p.stride = g.stride; p.pad_h = g.pad; p.pad_w = g.pad_w >= 0 ? g.pad_w : g.pad;
    p.c_blocks = (kc + BLOCK_K - 1) / BLOCK_K;
    p.num_k_blocks = taps * p.c_blocks;
    p.kb_per_split = tc_blocks_per_split(p.c_blocks, p.num_k_blocks, S, a.block_n_hint);
    if (S > 1 && (long)(S - 1) * p.kb_per_split >= p.num_k_blocks)
        throw Error(NB_ERR_INVALID_ARG, "split-K needs non-empty splits of ceil(K blocks / splits) blocks");
    if (S > 1 && !cluster && (a.y_pool || a.addend || a.scale || a.shift || a.act != NB_ACT_LINEAR))
        throw Error(NB_ERR_INVALID_ARG, "split-K into slabs needs a plain epilogue");
    if (cluster && (S > TC_MAX_CLUSTER || (a.a_is_conv && (a.N % 4) != 0) || a.lstm_H ||
                    (a.addend && (!a.a_is_conv || a.res_stride == 0 || (a.res_c % 4) != 0 || (a.ld_addend % 4) != 0 || !aligned16(a.addend)))))
        throw Error(NB_ERR_INVALID_ARG, "split-K over a cluster needs a convolution's columns, and a shortcut's, in quads");
    p.k_splits = S;
    p.m_tiles = p.tiles_w * p.tiles_h * p.tiles_n;
    p.e.N = a.N;
    p.tx_bytes_a = BLOCK_K * 4 * box.bw * box.bh * box.bn;
    p.e.scale = a.scale; p.e.shift = a.shift; p.e.addend = a.addend; p.e.ld_addend = a.ld_addend;
    p.e.act = a.act; p.e.round_out = a.round_out_tf32 ? 1 : 0;
    p.e.addend_vec = a.addend && aligned16(a.addend) && (a.ld_addend % 4) == 0;
    p.e.addend_cols = a.addend ? (a.res_stride > 0 ? a.res_c : a.N) : 0;
    p.e.res_stride = a.addend ? a.res_stride : 0; p.e.res_h = a.res_h; p.e.res_w = a.res_w;
    p.e.addend_post = (a.addend && a.addend_after_act) ? 1 : 0;
    if (a.lstm_H > 0 && a.act != NB_ACT_LINEAR && !p.e.addend_post)
        throw Error(NB_ERR_INVALID_ARG, "LSTM epilogue: a non-linear gate activation needs the addend added after it");
    p.e.y = a.y; p.e.ldy = a.ldy;
    p.e.tma_store = a.y && aligned16(a.y) && (a.ldy % 4) == 0 && !a.y_nchw;
    if (a.y_nchw) {
        if (!a.a_is_conv || gather || (S > 1 && !cluster) || pool || a.lstm_H > 0)
            throw Error(NB_ERR_INVALID_ARG, "NCHW output needs a whole convolution whose rows are pixels");
        p.e.plane = g.OH * g.OW;
    }
    if (S > 1 && !cluster && !p.e.tma_store) throw Error(NB_ERR_INVALID_ARG, "split-K needs a 16-byte aligned output with ldy % 4 == 0");
    p.e.pool = pool ? 1 : 0;
    if (pool) {
        if (!a.a_is_conv || (g.OW & 1) || (g.OH & 1) || (a.N % 4) || !aligned16(a.y_pool) || a.addend)
            throw Error(NB_ERR_UNSUPPORTED, "fused 2x2 pooling needs even output extents and a 16-byte aligned NHWC tensor");
        p.e.tma_store = cluster;            // (there: whether rows are quads on 16-byte boundaries)
        if (cluster) { p.e.y = a.y_pool; p.e.ldy = a.N; }
    } else if (a.lstm_H > 0) {
        if (a.a_is_conv || S > 1 || a.N != 4 * a.lstm_H || !a.lstm_c || !a.lstm_h)
            throw Error(NB_ERR_INVALID_ARG, "LSTM epilogue needs a plain [M,4H] product and c/h outputs");
        p.e.tma_store = 0;
        p.e.lstm_H = a.lstm_H; p.e.lstm_c_prev = a.lstm_c_prev; p.e.lstm_c = a.lstm_c; p.e.lstm_h = a.lstm_h;
        p.e.lstm_h_round = a.lstm_h_round;
        p.e.lstm_f32 = three_pass ? 0 : 1;
        p.e.lstm_vec = (a.lstm_H % 8) == 0 && aligned16(a.lstm_c) && aligned16(a.lstm_h) &&
                       (!a.lstm_c_prev || aligned16(a.lstm_c_prev)) && (!a.lstm_h_round || aligned16(a.lstm_h_round));
    } else if (!a.y) {
        throw Error(NB_ERR_INVALID_ARG, "GEMM without an output tensor");
    }
    p.status = h->d_status;
    p.b_static = a.b_static && !gather ? 1 : 0;

    // tile width in filters: widest tile that still gives every SM work
    // Promoted accumulation: always for 3xTF32 (its point is fp32-level agreement); in TF32 mode only for
    // very long contractions, where the accumulator's round-toward-zero bias (~K * 7.5e-9) nears TF32's own error.
    const bool promote = three_pass || (long)p.kb_per_split * BLOCK_K >= 8192 ||  // per split when K is split
                         (a.k_part > 0 && a.k_part < p.kb_per_split);
    int block_n = 256;
    if (three_pass || gather || promote) block_n = 128;
    if (a.block_n_hint) block_n = std::min(block_n, a.block_n_hint);
    if (!a.block_n_hint) {
        // Cost of a K block of a 128 x bn tile: its MMAs (128 / 64 / 48 cycles per K = 8 step at bn = 256 / 128 / 64) or
        // the operand bytes it needs at the ~71 B/cycle/SM that L2 delivers to 148 SMs loading at once, whichever is
        // larger; times the number of waves of tiles.  Wider tiles move fewer bytes per FLOP, so a single wave of
        // 256-wide tiles on two thirds of the SMs beats two waves of 128-wide ones (conv5_x at 32 images per GPU).
        const int widest = block_n;
        long best_cost = 0;
        for (int bn = widest; bn >= 64; bn /= 2) {
            if (bn > 64 && a.N <= bn / 2) continue;         // more than half of the tile would be padding
            const long tiles = (long)p.m_tiles * ((a.N + bn - 1) / bn) * S;
            const long waves = (tiles + h->sm_count - 1) / h->sm_count;
            const long mma = bn == 256 ? 512 : (bn == 128 ? 256 : 192);
            const long supply = (long)(BLOCK_M + bn) * BLOCK_K * 4 / 71;
            const long cost = waves * std::max(mma, supply);
            if (best_cost == 0 || cost < best_cost) { best_cost = cost; block_n = bn; }
        }
    }
    // a shortcut's slabs through shared memory: 1x1 layers of several tiles per SM.  (A single tile per SM has nothing to fetch ahead of,
    // and its short ring takes one K block per stage: ResNet-50 b1 412 us without, 423 with.  That ring costs more the longer K is: 640 ->
    // 1024 at 64 images of 14 x 14 62.3 us through shared memory and 59.5 from memory, 1024 -> 1024 89 and 76; 512 -> 1024 53 both.)
    const bool residual = a.addend && a.res_stride > 0 && !a.addend_after_act && !cluster && !promote && !gather && !col3 && p.e.addend_vec &&
                          p.e.addend_cols % 4 == 0 && !a.block_n_hint && taps == 1 && p.e.tma_store && a.shift &&
                          cheap_activation(a.act) && kc <= 512 && (long)p.m_tiles * ((a.N + 127) / 128) > h->sm_count;
    if (residual) block_n = std::min(block_n, 128);
    p.n_tiles = (a.N + block_n - 1) / block_n;
    p.m_fastest = (!a.a_is_conv && !gather && (size_t)a.N * a.Kc * 4 > ((size_t)48 << 20)) ? 1 : 0;
    // accumulation chains of at most 512 K elements (TF32) / 12 MMAs (3xTF32) in the tensor core: every accumulating MMA
    // truncates the running sum (a shrink of about 6e-8 per step that adds up layer after layer).  A 3xTF32 K block is
    // 12 MMAs, of which only the 4 hi*hi ones go into the promoted chain (the cross terms have columns of their own)
    // (a slice of two or three blocks is cut once more: in a single part its cross terms would go into the chain, 24 to 36 MMAs)
    p.kb_per_part = !promote ? p.kb_per_split : (three_pass ? (S > 1 && p.kb_per_split <= 3 ? (p.kb_per_split + 1) / 2 : 3) : (a.k_part > 0 ? a.k_part : 16));
    p.parts = (p.kb_per_split + p.kb_per_part - 1) / p.kb_per_part;

    // two K blocks per ring stage: tiles of up to 128 columns whose K slices pair up, a box of whole 8-row groups (the
    // second slice must start on a swizzle-pattern boundary), whole pairs per split.  A box of fewer than 128 rows only
    // where a tile steps through a short K alone (64 wide, one wave, up to 16 blocks: a ResNet-50 image 504 -> 487 us); with
    // longer K the shallower ring costs more (AlexNet b16 282 -> 291 us, ResNet-50 b64 2318 -> 2348 us)
    p.col3 = (col3 && !promote && block_n <= 128) ? 1 : 0;
    p.halves = p.col3 ? halves : 1;
    if (halves == 2 && !p.col3) throw Error(NB_ERR_UNSUPPORTED, "two-box tiles need the filter-column mode");
    const bool alone = block_n == 64 && a.a_is_conv && (long)p.m_tiles * p.n_tiles * S <= h->sm_count && p.kb_per_split <= 16;
    if (pairs && alone) {
        box = whole_groups(box, g.OW, g.OH, g.stride, pool, (double)g.sh * 4.0);
        p.bw = box.bw; p.bh = box.bh; p.bn = box.bn;
        p.tiles_w = (g.OW + box.bw - 1) / box.bw;
        p.tiles_h = (g.OH + box.bh - 1) / box.bh;
        p.m_tiles = p.tiles_w * p.tiles_h * p.tiles_n;
        p.tx_bytes_a = BLOCK_K * 4 * box.bw * box.bh * box.bn;
    }
    const int box_rows = box.bw * box.bh * box.bn;
    p.cbs = (pairs && !promote && !residual && (S == 1 || p.kb_per_split % 2 == 0) && block_n <= 128 &&
             (box_rows == BLOCK_M ? a.a_is_conv : alone && box_rows % 8 == 0)) ? 2 : 1;
    p.a_slice_bytes = box_rows * 128;
    p.a_region = A_STAGE_BYTES + (p.cbs - 1) * p.a_slice_bytes;
    {
        const int b_stage = block_n * BLOCK_K * 4;
        const int stage1 = three_pass && !gather ? A_STAGE_BYTES + 2 * b_stage : (A_STAGE_BYTES + b_stage) * (three_pass ? 2 : 1);
        const int ring = std::min(8, (196 * 1024) / stage1) * stage1;       // bytes the variant's ring holds
        p.a_box_bytes = BLOCK_K * 4 * box.bw * (box.bh * halves + 2);
        p.stage_bytes = p.col3 ? p.a_box_bytes + 3 * b_stage : (p.cbs == 2 ? p.a_region + 2 * b_stage : stage1);
        p.stages = std::min(8, (residual ? RESIDUAL_OFFSET : ring) / p.stage_bytes);
        // a second staging buffer per epilogue group in what the ring leaves unused; a one-column filter (row windows:
        // one stage per tile, bound by its epilogue) gives up its third stage for it
        if (p.col3 && ksize_w == 1 && p.stages > 2) p.stages = 2;
        const int ring_cap = residual ? 0 : std::min(8, (196 * 1024) / stage1) * stage1;
        const int used = p.stages * p.stage_bytes;
        p.slab2_offset = (!three_pass && !promote && !gather && ring_cap - used >= 2 * BLOCK_M * 32 * 4) ? used : 0;
    }
    if (gather) {
        p.gx = a.a;
        p.gsn = a.g.sn; p.gsh = a.g.sh; p.gsw = a.g.sw;
        p.gks = a.g.ksize; p.gpad = a.g.pad; p.gK = a.g.C * a.g.ksize * a.g.ksize;
        for (int kk = 0; kk < a.Kc; kk++) {
            int off = 0, dh = 30000, dw = 0;        // padding columns: a row offset that is never inside an image
            if (kk < p.gK) {
                const int tap = kk / a.g.C, c = kk - tap * a.g.C;
                dh = tap / a.g.ksize - a.g.pad; dw = tap % a.g.ksize - a.g.pad;
                off = (int)(c * a.g.sc + dh * a.g.sh + dw * a.g.sw);
            }
            p.gtab[kk] = make_int2(off, (dh & 0xffff) | (dw << 16));
        }
        p.gH = a.g.H; p.gW = a.g.W; p.gOH = a.g.OH; p.gOW = a.g.OW; p.gstride = a.g.stride; p.gM = a.M;
        p.ground = three_pass ? 0 : 1;
    }

    // ---- every operand must lie inside the allocation its pointer belongs to.  For the operands TMA loads, that
    // includes what the boxes at out-of-bounds coordinates cover: such elements arrive as zeros, but the load unit
    // still reads the addresses they map to (rows above the first image, past the last one, past the last filter).
    const long long F4 = 4;
    const long long n32 = ((long long)a.N + 31) / 32 * 32;
    const long long cmax = (long long)p.c_blocks * BLOCK_K - 1;
    if (gather) {
        const long long last = (long long)(a.g.batch - 1) * a.g.sn + (long long)(a.g.H - 1) * a.g.sh +
                               (long long)(a.g.W - 1) * a.g.sw + (long long)(a.g.C - 1) * a.g.sc;
        check_extent(h, a.a, 0, (last + 1) * F4, "gathered input tensor");
    } else {
        const long long wmin = -(long long)p.pad_w, hmin = -(long long)p.pad_h;
        const long long wmax = (long long)(p.tiles_w - 1) * box.bw * g.stride + wmin + (ksize_w - 1) + (long long)box.bw * g.stride - 1;
        const long long bh_tile = (long long)box.bh * halves;
        const long long hmax = (long long)(p.tiles_h - 1) * bh_tile * g.stride + hmin + (g.ksize - 1) + bh_tile * g.stride - 1;
        const long long nmax = (long long)p.tiles_n * box.bn - 1;
        const long long lo = std::min(wmin, 0LL) * g.sw + std::min(hmin, 0LL) * g.sh;
        const long long hi = wmax * g.sw + hmax * g.sh + nmax * g.sn + cmax + 1;
        check_extent(h, a.a, lo * F4, hi * F4, "A operand (with the out-of-bounds elements its boxes cover)");
    }
    {
        const long long rows = (long long)(taps - 1) * a.N + (long long)p.n_tiles * block_n;
        const long long b_floats = (rows - 1) * a.ldb + cmax + 1;
        check_extent(h, a.b, 0, b_floats * F4, "B operand (with the rows past the last filter its boxes cover)");
        if (three_pass) check_extent(h, a.b_lo, 0, b_floats * F4, "low-order B operand");
    }
    if (a.scale) check_extent(h, a.scale, 0, n32 * F4, "epilogue scale vector (padded to 32 columns)");
    if (a.shift) check_extent(h, a.shift, 0, n32 * F4, "epilogue shift vector (padded to 32 columns)");
    if (a.addend) {
        const long long fl = a.res_stride > 0
            ? ((long long)g.batch * a.res_h * a.res_w - 1) * a.ld_addend + a.res_c
            : ((long long)a.M - 1) * a.ld_addend + a.N;
        check_extent(h, a.addend, 0, fl * F4, "addend");
    }
    if (a.y && !pool && !a.lstm_H)
        check_extent(h, a.y, 0, (((long long)(cluster ? 1 : S) * a.M - 1) * a.ldy + a.N) * F4, "output");
    if (pool) check_extent(h, a.y_pool, 0, (long long)g.batch * (g.OH / 2) * (g.OW / 2) * a.N * F4, "pooled output");
    if (a.lstm_H > 0) {
        const long long fl = (long long)a.M * a.lstm_H * F4;
        if (a.lstm_c_prev) check_extent(h, a.lstm_c_prev, 0, fl, "previous cell state");
        check_extent(h, a.lstm_c, 0, fl, "cell state");
        check_extent(h, a.lstm_h, 0, fl, "hidden state");
        if (a.lstm_h_round) check_extent(h, a.lstm_h_round, 0, fl, "rounded hidden state");
    }

    if (p.cbs == 2) {   // A: dims {32, W, H, N, C/32}; B: dims {32, N, C/32, taps}: the channel slice is a dimension of its own
        cuuint64_t dims[5] = {(cuuint64_t)BLOCK_K, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.batch, (cuuint64_t)p.c_blocks};
        cuuint64_t strides[4] = {(cuuint64_t)g.sw * 4, (cuuint64_t)g.sh * 4, (cuuint64_t)g.sn * 4, (cuuint64_t)BLOCK_K * 4};
        cuuint32_t bx[5] = {(cuuint32_t)BLOCK_K, (cuuint32_t)(box.bw * g.stride), (cuuint32_t)(box.bh * g.stride),
                            (cuuint32_t)box.bn, 2};
        cuuint32_t es[5] = {1, (cuuint32_t)g.stride, (cuuint32_t)g.stride, 1, 1};
        encode(h, &p.tm_a, a.a, 5, dims, strides, bx, es);
        cuuint64_t bdims[4] = {(cuuint64_t)BLOCK_K, (cuuint64_t)a.N, (cuuint64_t)p.c_blocks, (cuuint64_t)taps};
        cuuint64_t bstrides[3] = {(cuuint64_t)a.ldb * 4, (cuuint64_t)BLOCK_K * 4, (cuuint64_t)a.ldb * 4 * (cuuint64_t)a.N};
        cuuint32_t bbx[4] = {(cuuint32_t)BLOCK_K, (cuuint32_t)block_n, 2, 1};
        cuuint32_t bes[4] = {1, 1, 1, 1};
        encode(h, &p.tm_b, a.b, 4, bdims, bstrides, bbx, bes);
    }
    if (!gather && p.cbs == 1) {   // A: dims {C, W, H, N}
        cuuint64_t dims[4] = {(cuuint64_t)kc, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.batch};
        cuuint64_t strides[3] = {(cuuint64_t)g.sw * 4, (cuuint64_t)g.sh * 4, (cuuint64_t)g.sn * 4};
        cuuint32_t bx[4] = {(cuuint32_t)BLOCK_K, (cuuint32_t)(box.bw * g.stride),
                            (cuuint32_t)(p.col3 ? box.bh * halves + 2 : box.bh * g.stride), (cuuint32_t)box.bn};
        cuuint32_t es[4] = {1, (cuuint32_t)g.stride, (cuuint32_t)g.stride, 1};
        encode(h, &p.tm_a, a.a, 4, dims, strides, bx, es);
    }
    if (p.col3) {       // B: dims {Kc, N, kw, kh}; a box is one filter column: kw fixed, kh = 0..2
        cuuint64_t dims[4] = {(cuuint64_t)kc, (cuuint64_t)a.N, (cuuint64_t)ksize_w, 3};
        cuuint64_t strides[3] = {(cuuint64_t)a.ldb * 4, (cuuint64_t)a.ldb * 4 * (cuuint64_t)a.N,
                                 (cuuint64_t)a.ldb * 4 * (cuuint64_t)a.N * (cuuint64_t)ksize_w};
        cuuint32_t bx[4] = {(cuuint32_t)BLOCK_K, (cuuint32_t)block_n, 1, 3};
        cuuint32_t es[4] = {1, 1, 1, 1};
        encode(h, &p.tm_b, a.b, 4, dims, strides, bx, es);
    } else if (p.cbs == 1) {   // B: dims {Kc, N, taps}
        cuuint64_t dims[3] = {(cuuint64_t)kc, (cuuint64_t)a.N, (cuuint64_t)taps};
        cuuint64_t strides[2] = {(cuuint64_t)a.ldb * 4, (cuuint64_t)a.ldb * 4 * (cuuint64_t)a.N};
        cuuint32_t bx[3] = {(cuuint32_t)BLOCK_K, (cuuint32_t)block_n, 1};
        cuuint32_t es[3] = {1, 1, 1};
        encode(h, &p.tm_b, a.b, 3, dims, strides, bx, es);
        if (three_pass) encode(h, &p.tm_b_lo, a.b_lo, 3, dims, strides, bx, es);
    }

    if (p.e.tma_store && !cluster) {   // Y: dims {N, OW, OH, NB}; the same pixel box as A, 32 columns wide
        cuuint64_t dims[4] = {(cuuint64_t)a.N, (cuuint64_t)g.OW, (cuuint64_t)g.OH, (cuuint64_t)g.batch * (cuuint64_t)S};
        cuuint64_t strides[3] = {(cuuint64_t)a.ldy * 4, (cuuint64_t)a.ldy * 4 * (cuuint64_t)g.OW,
                                 (cuuint64_t)a.ldy * 4 * (cuuint64_t)g.OW * (cuuint64_t)g.OH};
        cuuint32_t bx[4] = {32, (cuuint32_t)box.bw, (cuuint32_t)box.bh, (cuuint32_t)box.bn};
        cuuint32_t es[4] = {1, 1, 1, 1};
        encode(h, &p.tm_y, a.y, 4, dims, strides, bx, es);
    }

    if (pool && !cluster) {          // pooled Y: dims {N, OW/2, OH/2, NB}
        cuuint64_t dims[4] = {(cuuint64_t)a.N, (cuuint64_t)(g.OW / 2), (cuuint64_t)(g.OH / 2), (cuuint64_t)g.batch};
        cuuint64_t strides[3] = {(cuuint64_t)a.N * 4, (cuuint64_t)a.N * 4 * (cuuint64_t)(g.OW / 2),
                                 (cuuint64_t)a.N * 4 * (cuuint64_t)(g.OW / 2) * (cuuint64_t)(g.OH / 2)};
        cuuint32_t bx[4] = {32, (cuuint32_t)(box.bw / 2), (cuuint32_t)(box.bh / 2), (cuuint32_t)box.bn};
        cuuint32_t es[4] = {1, 1, 1, 1};
        encode(h, &p.tm_yp, a.y_pool, 4, dims, strides, bx, es);
    }

    const int width = block_n == 256 ? 2 : (block_n == 128 ? 1 : 0);
    const bool lean = !three_pass && !promote && !gather && !cluster && p.e.tma_store && p.e.shift &&
                      cheap_activation(a.act) &&
                      (!a.addend || (p.e.addend_vec && p.e.addend_cols % 4 == 0 && !p.e.addend_post));
    L->v = residual ? RESIDUAL_VARIANTS[width] : lean ? LEAN_VARIANTS[width] : cluster ? CLUSTER_VARIANTS[three_pass ? 1 : 0][promote ? 1 : 0][width] : VARIANTS[gather ? 1 : 0][three_pass ? 1 : 0][promote ? 1 : 0][width];
    gemm_tc_load(h, residual ? TC_RESIDUAL : lean ? TC_LEAN : gather ? TC_GATHER : 0);
    L->cluster = cluster ? S : 1;
    if (!L->v.kernel) throw Error(NB_ERR_UNSUPPORTED, "no tensor-core kernel variant for this tile width");
    const int tiles = p.m_tiles * p.n_tiles * p.k_splits;
    L->grid = cluster ? tiles : std::max(1, std::min(tiles, h->sm_count));
    L->threads = (three_pass || gather) ? 448 : 320;
    L->gather = gather;
    L->flops = a.algo_flops > 0 ? a.algo_flops : 2.0 * (double)a.M * a.N * a.Kc * taps;
    L->desc = " [M=" + std::to_string(a.M) + " N=" + std::to_string(a.N) + " K=" + std::to_string(a.Kc) + " taps=" +
              std::to_string(taps) + " stride=" + std::to_string(g.stride) + " out=" + std::to_string(g.OW) + "x" +
              std::to_string(g.OH) + "x" + std::to_string(g.batch) + " box=" + std::to_string(box.bw) + "x" +
              std::to_string(box.bh) + "x" + std::to_string(box.bn) + " block_n=" + std::to_string(block_n) +
              " splits=" + std::to_string(S) + (cluster ? "c" : "") + (p.col3 ? (p.halves == 2 ? " col3x2" : " col3") : "") + (p.cbs == 2 ? " cbs2" : "") + (gather ? " gather" : "") +
              (three_pass ? " 3xtf32" : "") +
              (pool ? " pool" : "") + (a.addend ? " addend" : "") + (a.lstm_H ? " lstm" : "") + "]";
    return L;
}

}  // namespace

// A convolution of one or a few small images has fewer tiles than SMs, and its tiles run their whole K alone: at about 0.15 us
// per 32-column block (two TMA requests of one thread) the 3x3 layers of a single ResNet-50 image (8 tiles, 72 and 144
// blocks) took 29 and 47 us.  Into slabs (a caller's NHWC tensor, and where tc_slab_cost is below the clusters' cost) such layers are
// cut until they occupy the SMs, four blocks per slice at least; the slices are added by splitk_reduce4_kernel (2-3 us), so layers of
// fewer than 32 blocks stay whole.  Tiles are counted over the
// whole batch, so an image alone and the same image in a batch that leaves the layer whole, or cuts it into fewer slices, add
// in different orders and may differ in the last bits.
int conv_tc_split(const nb_handle_s *h, const ConvGeom &g, int Kc, int N) {
    const int c_blocks = (Kc + BLOCK_K - 1) / BLOCK_K, blocks = g.ksize * (g.ksize_w > 0 ? g.ksize_w : g.ksize) * c_blocks;
    if (blocks < 32 || (N % 4) != 0) return 1;
    const Box box = choose_box(g.OW, g.OH, g.batch, g.stride, false, true, (double)g.C * g.H * g.W * 4.0);
    const long tiles = (long)((g.OW + box.bw - 1) / box.bw) * ((g.OH + box.bh - 1) / box.bh) * ((g.batch + box.bn - 1) / box.bn) *
                       ((N + 63) / 64);
    if (2 * tiles > h->sm_count) return 1;
    const int S = (int)std::min<long>({h->sm_count / tiles, blocks / 4, 16});
    int per = (blocks + S - 1) / S;
    if (c_blocks % 2 == 0) per += per & 1;      // whole pairs of slices: two-block ring stages stay possible
    return (blocks + per - 1) / per;
}

// The time of a contraction whose tiles are cut over clusters of S CTAs, all clusters resident at once, in units of a 64-wide
// TF32 K block (0.225 us); S = 1: whole, in waves.  Negative: it does not run that way.  Of a cluster each CTA adds S partial
// sums of 1/S of its tile, so the exchange costs most for the smallest and the largest, and a large cluster waits for that many
// SMs of one part of the device.  3x3 layers of one image (28 x 28 x 128, 14 x 14 x 256, 7 x 7 x 512), us: whole 13.1 / 21.0 /
// 37.7, S = 2: 11.1 / 15.0 / 22.4, 4: 7.6 / 9.8 / 13.6, 6: 7.6 / 7.9 / 11.1, 9: 7.9 / 7.9 / 9.3; the weight of S is a ResNet-50 image's
// (0.5: 435 us, 1: 427, 1.5: 424, 2: 425).  128-wide tiles were never better in TF32.  A 3xTF32 block takes half as long again, a
// 128-wide one a third more, and its exchange four times as long (3xTF32, 19 x 19 x 100 at 20 images: whole 25 us, two halves of K
// 30; 14 x 14 x 512 at 8: 64 and 50).
double tc_cluster_cost(const nb_handle_s *h, long m_tiles, int N, int blocks, int S, int bn, bool three_pass, int act) {
    const long tiles = m_tiles * ((N + bn - 1) / bn);
    const double block = (three_pass ? 1.5 : 1.0) * (bn == 64 ? 1.0 : 1.33);
    const double heavy = cheap_activation(act) ? 0.0 : 24.0 * bn / 64;     // the double formulas
    if (S == 1) return (double)((tiles + h->sm_count - 1) / h->sm_count) * (blocks * block + heavy);
    const int per = (blocks + S - 1) / S;
    if ((long)(S - 1) * per >= blocks || tiles * S > h->sm_count || tiles > clusters_at_once(h, S)) return -1;
    return per * block + heavy / S + 1.5 * S + 26.0 * (bn / 64) * (bn / 64) / (S * S);
}

// The time of the same cut into S slabs, by tiles in waves, and of the kernel that adds M rows of them (another 30 units behind the
// product, 8 bytes per partial sum at 5 TB/s).  Clusters give one layer 16 times as many SMs as it has tiles at most, slabs all of
// them: 10 x 42568 -> 28, a cluster of 16 31.6 us, 32 slabs 27.3; 55060 -> 80 35.2 and 23.5; 3xTF32, 7x7, 176 -> 32 at 5 images of 34 x 34,
// two CTAs 72 and three slabs 52.  But 6068 -> 12 at 3 rows 9.6 and 11.2, 10132 -> 392 at 105 rows 18.7 and 22.4.
double tc_slab_cost(const nb_handle_s *h, long m_tiles, long M, int N, int blocks, int S, int bn, bool three_pass) {
    const double block = (three_pass ? 1.5 : 1.0) * (m_tiles == 1 ? (bn == 64 ? 1.0 : (bn == 128 ? 1.1 : 1.3)) : (bn == 64 ? 1.0 : 1.33));
    const long tiles = m_tiles * ((N + bn - 1) / bn) * S;
    return (double)((tiles + h->sm_count - 1) / h->sm_count) * ((blocks + S - 1) / S) * block + 38.0 + 7.1e-6 * S * M * N;
}

// The tile width and cluster size of a convolution.  In TF32 only where its 64-wide tiles leave half of the SMs idle, as above.
// Of `slabs` (conv_tc_split) instead where those take less time, with a layout pass behind them if the output is NCHW: TcSplit{slabs, 0}.
TcSplit conv_tc_cluster(const nb_handle_s *h, const ConvGeom &g, int Kc, int N, int act, bool three_pass, bool pool, int slabs, bool nchw) {
    TcSplit best{1, 0};
    const int c_blocks = (Kc + BLOCK_K - 1) / BLOCK_K, blocks = g.ksize * (g.ksize_w > 0 ? g.ksize_w : g.ksize) * c_blocks;
    if ((N % 4) != 0) return best;
    const Box box = choose_box(g.OW, g.OH, g.batch, g.stride, pool, false, (double)g.C * g.H * g.W * 4.0);
    const long m_tiles = (long)((g.OW + box.bw - 1) / box.bw) * ((g.OH + box.bh - 1) / box.bh) * ((g.batch + box.bn - 1) / box.bn);
    if (!three_pass && 2 * m_tiles * ((N + 63) / 64) > h->sm_count) return best;
    // (filter-column stages fetch a block in less: 56 x 56 x 64 whole 7.8 us, in clusters 8 to 9.6)
    double best_cost = tc_cluster_cost(h, m_tiles, N, blocks, 1, 64, three_pass, act) * (!three_pass && column_stages(g, Kc, N) ? 0.6 : 1.0);
    if (three_pass && N > 64) best_cost = std::min(best_cost, tc_cluster_cost(h, m_tiles, N, blocks, 1, 128, true, act));
    for (int bn = 64; bn <= (three_pass && N > 64 ? 128 : 64); bn *= 2)
        for (int S = 2; S <= TC_MAX_CLUSTER; S++) {
            const double cost = tc_cluster_cost(h, m_tiles, N, blocks, S, bn, three_pass, act);
            if (cost >= 0 && cost < best_cost) { best_cost = cost; best = TcSplit{S, bn}; }
        }
    const long rows = (long)g.batch * g.OH * g.OW;
    if (best.S > 1 && slabs > 1 && tc_slab_cost(h, m_tiles, rows, N, blocks, slabs, 64, three_pass) + (nchw ? 12.0 + 7.1e-6 * rows * N : 0.0) < best_cost)
        return TcSplit{slabs, 0};
    return best;
}

// A lane of the epilogue owns a pixel, so in NCHW a warp's stores of a column are as contiguous as its box's pixels.  Boxes
// of many images and few pixels of each (13 x 13 at 128 images: one pixel of 128 images) scatter them: 512 -> 2048 1x1 there
// 558 us against 175 with a layout pass behind.  Of 360 layers measured, runs of 7 pixels and more and whole planes are the
// faster for it in all but five (7 x 7 at 32 images, 256 -> 1024: 12.7 against 18.3 us), single pixels never; in between while
// L2 holds the partial sectors until their neighbours arrive (runs of 2: 10 MB, of 4: 40 MB of output).
bool conv_tc_writes_nchw(const GemmArgs &a, bool three_pass) {
    const ConvGeom &g = a.g;
    if (!three_pass && column_stages(g, a.Kc, a.N)) return true;
    const Box b = choose_box(g.OW, g.OH, g.batch, g.stride, false, false, (double)g.sn * 4.0);
    const int run = b.bw == g.OW ? b.bw * b.bh : b.bw;
    return run >= 7 || (b.bw == g.OW && b.bh == g.OH) || (run >= 2 && 4.0 * a.M * a.N <= 2.5e6 * run * run);
}

void gemm_tc(nb_handle_s *h, const GemmArgs &a, bool three_pass) {
    std::string key = gemm_args_key(a, 'G', three_pass ? 1 : 0);
    auto it = h->launch_cache.find(key);
    if (it == h->launch_cache.end()) {
        if (h->launch_cache.size() > 4096) h->launch_cache.clear();
        it = h->launch_cache.emplace(std::move(key), build_launch(h, a, three_pass)).first;
    }
    const TcLaunch &L = static_cast<const TcLaunch &>(*it->second);
    ProfileScope prof(h, 0, L.flops);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.grid);
    cfg.blockDim = dim3((unsigned)L.threads);
    cfg.dynamicSmemBytes = (size_t)L.v.smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)L.cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    // The gather variants are not launched ahead.  Launched ahead, every second of two queued calls (30 channels, 3x3, 8
    // images of 33 x 33: 9 K blocks, 69 CTAs) left about ten CTAs whose accumulators never completed, so that the wait for them
    // ran out and the output kept the call's before; alone the same call is right.  They are the only launches with more than
    // 4096 bytes of parameters (TcGatherParams: 4160), the one thing that sets them apart; the cause is not proven.
    cfg.numAttrs = L.gather ? 0 : (L.cluster > 1 ? 2 : 1);
    void *args[1] = {const_cast<TcGatherParams *>(&L.p)};
    (void)cudaLaunchKernelExC(&cfg, L.v.kernel, args);
    try {
        check_launch("gemm_tf32_tcgen05_kernel");
    } catch (const Error &err) {
        throw Error(err.code, std::string(err.what()) + L.desc);    // an asynchronous fault is otherwise hard to place
    }
    count_launch(h);
    if (h->trace_host && !h->trace_names.empty()) h->trace_names.back() += L.desc;
    prof.finish();
}

}  // namespace nb
