// The recurrence of one TF32 LSTM layer as one cooperative kernel (lstm_layer.cc:262-311 per step), for the widths and batches whose
// clusters of four CTAs do not fit the device or tensor memory (lstm_persistent.cu, the faster way where it runs): 1088 to 1184 units,
// 1056 above 64 rows, and two steps of many rows.
//
// Bound by the latency of a step.  Every CTA owns 32 gate columns (8 hidden units x i,f,g,o), keeps its 32 x H slice of the recurrent
// weights in shared memory for the whole sequence (148 KB at H = 1184, loaded once by TMA) and the cell state of its units in registers.
// Per step it streams h_{t-1} (rounded to TF32, [B x H]) from L2 into a ring of 128-byte-swizzled K blocks by TMA, multiplies
// (tcgen05.mma kind::tf32, M = batch rows, N = 32, accumulators in TMEM), adds the input-side pre-activations, runs the cell update
// and writes c_t, h_t and the rounded h_t.  A grid-wide barrier (one atomic counter, bounded spin) separates the steps: step t + 1 of
// every CTA reads what all CTAs wrote in step t.  Against a launch per step, us a step of 64: H = 1088, 20 / 64 / 128 rows 15.7 / 16.7 /
// 19.3 -> 12.0 / 10.1 / 13.9; H = 1184 16.5 / 17.5 / 20.0 -> 12.6 / 13.2 / 14.6; H = 1056, 65 / 128 rows 16.5 / 18.7 -> 12.8 / 13.7.
//
// h_{t-1} was written by other SMs' ordinary stores earlier in this same kernel and is read here by TMA, i.e. through the async
// proxy: the writers release (a release-add on the barrier counter), the thread that issues the copies acquires the counter itself
// and then issues fence.proxy.async before its first copy of the step.  That one thread issues all copies in the order of their use,
// so a slot's barrier is never more than one phase behind.  The results are bit-identical to a launch per step: the slices of K that
// the width adds (lstm_in_slices) have accumulators of their own, added in their order.
#include <cstring>

#include "tc_common.cuh"

namespace nb {

using namespace tc;

namespace {

constexpr int LW_N = 32;                    // gate columns per CTA
constexpr int LW_STAGES = 4;                // most ring stages (barrier slots)
constexpr int LW_THREADS = 192;             // warps 0-3: epilogue; warp 4: MMA issue; warp 5: grid barrier and TMA
constexpr int LW_W_TILE = LW_N * 128;       // one K block of the weight slice: 32 rows x 128 bytes
constexpr int LW_PARTS = 4;                 // most slices of K with accumulators of their own
constexpr int LW_TMEM = LW_PARTS * LW_N;

struct LstmWParams {
    CUtensorMap tm_w;           // recurrent weights [4H rows][H], box {32, 32}
    CUtensorMap tm_h;           // rounded hidden states as {32, T*B rows, H/32}, box {32, B, cbs}
    int cbs;                    // K blocks per ring stage and TMA request (2 when B % 8 == 0 and H % 64 == 0)
    int stages, stage_bytes;    // ring geometry: a stage holds cbs slices of B rows and the 128-row window of the last
    const float *pre;           // [T][B][4H] input-side pre-activations (biases included), columns [unit][i,f,g,o]
    float *hr_w;                // [T][B][H] rounded hidden states: step t writes [t]; step t + 1 reads it through tm_h
    float *cell, *out;          // [T][B][H]
    int T, B, H;
    int kb_per_part, parts;     // K blocks per slice, and slices
    int t_first;                // first step this kernel runs (the steps before it are in cell/out/hr already)
    unsigned int *sync;         // grid barrier counter, zero at launch
    int *status;
};

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned int *p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__global__ void __launch_bounds__(LW_THREADS, 1) lstm_wide_kernel(const __grid_constant__ LstmWParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int KB = p.H / BLOCK_K;                           // K blocks per step
    uint8_t *w_smem = smem;                                  // [KB][32 rows][128 B], swizzled by TMA
    uint8_t *a_ring = smem + (size_t)KB * LW_W_TILE;         // [LW_STAGES][128 rows][128 B]
    const int stages = p.stages, stage_bytes = p.stage_bytes, cbs = p.cbs;
    uint64_t *bars = (uint64_t *)(a_ring + stages * stage_bytes);
    uint64_t *full = bars;                  // loaders -> MMA   [LW_STAGES]
    uint64_t *empty = bars + LW_STAGES;     // MMA -> loaders   [LW_STAGES]
    uint64_t *w_full = bars + 2 * LW_STAGES;
    uint64_t *acc_full = w_full + 1;
    uint32_t *tmem_slot = (uint32_t *)(acc_full + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < LW_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(w_full, 1);
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)LW_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // rows of the A tiles that no batch row fills: the MMA reads all 128, give them a defined value once
    for (int i = threadIdx.x; i < stages * stage_bytes / 16; i += blockDim.x)
        reinterpret_cast<float4 *>(a_ring)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int n0 = blockIdx.x * LW_N;                       // first gate column of this CTA
    const unsigned int ctas = gridDim.x;
    bool ok = true;

    if (warp == 4) {
        // ------------------------------------------------ weights (once), then the MMAs of every step
        if (elect_one()) {
            mbar_expect_tx(w_full, (uint32_t)(KB * LW_W_TILE));
            for (int kb = 0; kb < KB; kb++) tma_load_3d(w_smem + kb * LW_W_TILE, &p.tm_w, w_full, kb * BLOCK_K, n0, 0);
            ok = mbar_wait(w_full, 0, abort_flag, p.status);
            const uint32_t idesc = p.B <= 64 ? make_idesc(64, LW_N) : make_idesc(BLOCK_M, LW_N);     // 64-row MMAs for small batches
            int stage = 0;
            uint32_t phase = 0;
            for (int t = p.t_first; t < p.T && ok; t++) {
                uint32_t d = tmem_base;
                int in_part = 0;
                for (int kb = 0; kb < KB; kb += cbs) {
                    if (!(ok = mbar_wait(&full[stage], phase, abort_flag, p.status))) break;
                    tc_fence_after();
                    for (int c = 0; c < cbs; c++) {
                        const uint32_t a_lo = smem_desc_lo(smem_u32(a_ring + stage * stage_bytes + c * p.B * 128));
                        const uint32_t b_lo = smem_desc_lo(smem_u32(w_smem + (kb + c) * LW_W_TILE));
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; k++)
                            umma_tf32(d, smem_desc(a_lo + 2 * k), smem_desc(b_lo + 2 * k), idesc, (in_part | k) != 0);
                        if (++in_part == p.kb_per_part) { in_part = 0; d += LW_N; }
                    }
                    umma_commit(&empty[stage]);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit(acc_full);
            }
            // the last releases of the ring must have landed before the CTA may exit
            for (int i = 0; i < stages && ok; i++) {
                ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status);
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ------------------------------------------------ h_{t-1} of every step, one K block per ring stage
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            const uint32_t tx = (uint32_t)(p.B * BLOCK_K * 4 * cbs);
            for (int t = p.t_first; t < p.T && ok; t++) {
                if (t > p.t_first) {
                    // grid barrier: all CTAs have arrived with h_{t-1}.  Their stores (generic proxy) are ordered before this
                    // acquire; the fence orders the copies below (async proxy) behind it
                    const unsigned int target = ctas * (unsigned int)(t - p.t_first);
                    const long long t0 = clock64();
                    while (ld_acquire_u32(p.sync) < target) {
                        if (*abort_flag || clock64() - t0 > WAIT_LIMIT_CYCLES) {
                            *abort_flag = 1;
                            atomicExch(p.status, (int)DEV_TIMEOUT);
                            ok = false;
                            break;
                        }
                    }
                    if (!ok) break;
                    asm volatile("fence.proxy.async;" ::: "memory");
                }
                for (int kb = 0; kb < KB; kb += cbs) {
                    if (!(ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status))) break;
                    mbar_expect_tx(&full[stage], tx);
                    tma_load_3d(a_ring + stage * stage_bytes, &p.tm_h, &full[stage], 0, (t - 1) * p.B, kb);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------ epilogue of every step, then the grid barrier
        const int tid = threadIdx.x;                        // 0..127
        // the batch row whose accumulators this thread's TMEM lane holds: lane = row for a 128-row MMA; a 64-row MMA
        // puts 16 rows into the first 16 lanes of each 32-lane quarter
        const int lane = tid & 31;
        const int brow = p.B <= 64 ? (lane < 16 ? 16 * warp + lane : 1 << 20) : tid;
        const bool row_ok = brow < p.B;
        const int unit0 = n0 >> 2;                          // first hidden unit of this CTA (8 of them)
        float c[8];
#pragma unroll
        for (int u = 0; u < 8; u++) c[u] = 0.0f;
        if (row_ok && p.t_first > 0) {
            const float *cp = p.cell + ((size_t)(p.t_first - 1) * p.B + brow) * p.H + unit0;
            const float4 lo = *reinterpret_cast<const float4 *>(cp), hi = *reinterpret_cast<const float4 *>(cp + 4);
            c[0] = lo.x; c[1] = lo.y; c[2] = lo.z; c[3] = lo.w; c[4] = hi.x; c[5] = hi.y; c[6] = hi.z; c[7] = hi.w;
        }
        uint32_t acc_phase = 0;
        for (int t = p.t_first; t < p.T && ok; t++) {
            // gates of this CTA's 8 units for row `tid`; threads only leave the loop together, at the votes, so that
            // none is left alone at a barrier
            // the input-side pre-activations of this step come from DRAM: fetched while the MMAs run
            const size_t row = (size_t)t * p.B + brow;
            float4 z4[8];
            if (row_ok) {
                const float4 *zin = reinterpret_cast<const float4 *>(p.pre + row * 4 * p.H + n0);
#pragma unroll
                for (int u = 0; u < 8; u++) z4[u] = __ldg(zin + u);
            }
            ok = epilogue_all(mbar_wait(acc_full, acc_phase, abort_flag, p.status), 1);
            if (!ok) break;
            acc_phase ^= 1;
            tc_fence_after();
            uint32_t v[32];
            tmem_ld_32x32(tmem_base + ((uint32_t)(warp * 32) << 16), v);
            tmem_ld_wait();
            for (int part = 1; part < p.parts; part++) {
                uint32_t more[32];
                tmem_ld_32x32(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(part * LW_N), more);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(more[j]));
            }
            tc_fence_before();
            float hn[8];
            const size_t o = row * p.H + unit0;
            if (row_ok) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const float zi = __uint_as_float(v[4 * u]) + z4[u].x, zf = __uint_as_float(v[4 * u + 1]) + z4[u].y;
                    const float zg = __uint_as_float(v[4 * u + 2]) + z4[u].z, zo = __uint_as_float(v[4 * u + 3]) + z4[u].w;
                    const float2 ch = lstm_cell_unit_f32_inline(zi, zf, zg, zo, c[u]);
                    c[u] = ch.x; hn[u] = ch.y;
                }
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    *reinterpret_cast<float4 *>(p.hr_w + o + 4 * q) = make_float4(round_tf32(hn[4 * q]), round_tf32(hn[4 * q + 1]),
                                                                                   round_tf32(hn[4 * q + 2]), round_tf32(hn[4 * q + 3]));
                }
            }
            // ---- grid barrier, this CTA's arrival: its rounded h_t is written (the barrier orders the group's stores before
            // the release).  What the next step does not read leaves behind it, so that the release does not wait for it
            if (t + 1 < p.T) {
                epilogue_bar_sync(1);
                if (tid == 0) red_release_add(p.sync, 1u);
            }
            if (row_ok) {
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    *reinterpret_cast<float4 *>(p.cell + o + 4 * q) = make_float4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
                    *reinterpret_cast<float4 *>(p.out + o + 4 * q) = make_float4(hn[4 * q], hn[4 * q + 1], hn[4 * q + 2], hn[4 * q + 3]);
                }
            }
        }
        if (!ok) *abort_flag = 1;
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; i++) __nanosleep(2000);     // let copies and MMAs in flight land before TMEM goes
        __syncthreads();
    }
    if (warp == 4) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)LW_TMEM) : "memory");
    }
}

struct LstmWLaunch : LaunchRecord {
    LstmWParams p;
    int grid, smem;
    double flops;
};

}  // namespace

// Whether the recurrence of an LSTM layer can run as this kernel: TF32 mode on the tensor-core path, gate layers without an
// activation of their own, H a multiple of 32 whose weight slice and two ring stages fit in shared memory, one CTA per 32 gate
// columns with all of them resident at once, a batch of at most 128 rows.  Two steps have one product, for which the set-up pays with
// many rows and weights only (us, here and per step: 20 rows, H = 256 21.0 / 20.0, 768 24.9 / 24.0, 1184 29.3 / 28.9; 64 rows, H = 64
// 27.3 / 26.2, 256 19.6 / 21.1, 768 23.3 / 25.9, 1024 25.2 / 28.9; 128 rows, H = 256 20.6 / 22.7, 1024 29.3 / 31.1; 48 rows, H = 768
// 24.7 / 27.1, 1024 26.5 / 29.4, 1184 30.7 / 29.9).
bool lstm_wide_supported(const nb_handle_s *h, int T, int B, int H) {
    if (!h->encode_tiled || h->cc_major != 10 || !h->cooperative_launch) return false;
    if (T < 2 || B < 1 || B > 128 || (H % 32) != 0) return false;      // (a box of B rows: any B up to 128)
    if (T == 2 && (B < 40 || H < 256 || (B < 64 && (H < 768 || H > 1056)))) return false;
    const int ctas = 4 * H / LW_N;
    const size_t smem = (size_t)(H / BLOCK_K) * LW_W_TILE + 2 * (A_STAGE_BYTES + (size_t)B * 128) + 1024 + 256;   // two stages at least
    if (ctas > h->sm_count || smem > 227 * 1024) return false;
    if (!h->lstm_wide_ready) {      // (loads the kernel)
        NB_CHECK_CUDA(cudaFuncSetAttribute(lstm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        h->lstm_wide_ready = true;
    }
    return true;
}

// Steps t_first .. T-1 of the recurrence (t_first >= 1: c, h and the rounded h of step t_first - 1 are in place), K added in
// slices of kb_per_part blocks; cell and out on 16-byte boundaries.
void lstm_wide(nb_handle_s *h, const float *w_hi, const float *pre, float *cell, float *out, float *hr, int T, int B,
               int H, int kb_per_part, int t_first) {
    std::string key;
    key.push_back('W');
    key_add(key, w_hi); key_add(key, pre); key_add(key, cell); key_add(key, out); key_add(key, hr);
    key_add(key, T); key_add(key, B); key_add(key, H); key_add(key, kb_per_part); key_add(key, t_first);
    auto it = h->launch_cache.find(key);
    if (it == h->launch_cache.end()) {
        std::unique_ptr<LstmWLaunch> L(new LstmWLaunch());
        std::memset(&L->p, 0, sizeof L->p);
        const long long F4 = 4;
        check_extent(h, w_hi, 0, (long long)4 * H * H * F4, "recurrent weights");
        check_extent(h, pre, 0, (long long)T * B * 4 * H * F4, "input-side pre-activations");
        check_extent(h, cell, 0, (long long)T * B * H * F4, "cell states");
        check_extent(h, out, 0, (long long)T * B * H * F4, "hidden states");
        check_extent(h, hr, 0, (long long)T * B * H * F4, "rounded hidden states");
        cuuint64_t dims[3] = {(cuuint64_t)H, (cuuint64_t)(4 * H), 1};
        cuuint64_t strides[2] = {(cuuint64_t)H * 4, (cuuint64_t)H * 4 * (cuuint64_t)(4 * H)};
        cuuint32_t bx[3] = {(cuuint32_t)BLOCK_K, (cuuint32_t)LW_N, 1};
        cuuint32_t es[3] = {1, 1, 1};
        encode_tensor_map(h, &L->p.tm_w, w_hi, 3, dims, strides, bx, es);
        // two K blocks per request when the second slice starts on the swizzle pattern's 1024-byte repeat
        const int cbs = ((B % 8) == 0 && (H % (2 * BLOCK_K)) == 0) ? 2 : 1;
        const int stage_bytes = (cbs - 1) * B * 128 + A_STAGE_BYTES;
        const int w_bytes = (H / BLOCK_K) * LW_W_TILE;
        const int stages = std::min(LW_STAGES, (227 * 1024 - 1024 - 256 - w_bytes) / stage_bytes);
        cuuint64_t hdims[3] = {(cuuint64_t)BLOCK_K, (cuuint64_t)T * (cuuint64_t)B, (cuuint64_t)(H / BLOCK_K)};
        cuuint64_t hstrides[2] = {(cuuint64_t)H * 4, (cuuint64_t)BLOCK_K * 4};
        cuuint32_t hbx[3] = {(cuuint32_t)BLOCK_K, (cuuint32_t)B, (cuuint32_t)cbs};
        cuuint32_t hes[3] = {1, 1, 1};
        encode_tensor_map(h, &L->p.tm_h, hr, 3, hdims, hstrides, hbx, hes);
        L->p.cbs = cbs; L->p.stages = stages; L->p.stage_bytes = stage_bytes;
        L->p.pre = pre; L->p.hr_w = hr; L->p.cell = cell; L->p.out = out;
        L->p.T = T; L->p.B = B; L->p.H = H; L->p.t_first = t_first;
        L->p.kb_per_part = kb_per_part; L->p.parts = (H / BLOCK_K + kb_per_part - 1) / kb_per_part;
        if (L->p.parts > LW_PARTS) throw Error(NB_ERR_INVALID_ARG, "lstm_wide: more slices of K than accumulators");
        L->p.sync = h->d_grid_sync + lstm_persistent_counters(); L->p.status = h->d_status;
        L->grid = 4 * H / LW_N;
        L->smem = w_bytes + stages * stage_bytes + 1024 + 256;
        L->flops = 2.0 * (double)(T - t_first) * B * 4.0 * H * H;
        if (h->launch_cache.size() > 4096) h->launch_cache.clear();
        it = h->launch_cache.emplace(std::move(key), std::move(L)).first;
    }
    const LstmWLaunch &L = static_cast<const LstmWLaunch &>(*it->second);
    NB_CHECK_CUDA(cudaMemsetAsync(L.p.sync, 0, sizeof(unsigned int), h->stream));
    ProfileScope prof(h, 0, L.flops);
    void *args[1] = {const_cast<LstmWParams *>(&L.p)};
    NB_CHECK_CUDA(cudaLaunchCooperativeKernel((const void *)lstm_wide_kernel, dim3(L.grid), dim3(LW_THREADS), args, (size_t)L.smem,
                                              h->stream));
    check_launch("lstm_wide_kernel");
    count_launch(h);
    prof.finish();
}

}  // namespace nb
