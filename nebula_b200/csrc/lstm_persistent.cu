// The recurrence of one LSTM layer as ONE cooperative kernel over all time steps (lstm_layer.cc:250-311 per step), TF32 mode.
//
// Bound by the latency of a step: a launch per step costs 12 to 20 us on this part for a 64 x 4096 x 1024 product that needs 1.
// Clusters of four CTAs own 32 hidden units (128 gate columns) each, and each CTA of a cluster a quarter of K:
//   * its 128 x K/4 slice of the recurrent weights stays in tensor memory for the whole sequence, as the A operand of the MMAs
//     (M = gate columns, N = batch rows, K = 8): an MMA then reads nothing from shared memory but h, and its time falls with the
//     batch;
//   * per step it loads only its quarter of h_{t-1} (rounded to TF32) from L2 by TMA: 64 KB at B = 64, H = 1024;
//   * its partial sums leave for the four CTAs over distributed shared memory (st.async onto the receiver's mbarrier): TMEM lanes
//     32 q .. 32 q + 31 hold the eight units that CTA q finishes.  The receiver adds them in the
//     order of K, adds the input-side pre-activations, runs the cell update and writes c_t, h_t and the rounded h_t.
// Steps are chained through one arrival counter per K block of h (the warps of four CTAs write it): a lane per block polls its counter
// (bounded) and issues that block's copy, so a CTA waits only for the units it reads.
// Against one CTA per 32 columns with all of K in shared memory (M = batch rows, N = 32: 128 MMAs of 40 cycles, 256 KB of h per
// CTA and step, one grid-wide counter): T128 B64 H1024 9.3 -> 5.4 us a step,
// and two such layers with their projection 2963 -> 1950 us.
//
// A step is a chain of latencies (publishing 1300 cycles, polling 1000, a copy 700, MMAs 400, the exchange 700, a cell 1100; the
// rest is waiting for the slowest of its peers), not of volume: with an eighth of h copied it takes 0.2 us less.  So the batch
// runs as four groups of rows, each a chain of its own with its own warps, barriers and counters (one group 2082 us, two 1985,
// four 1949), and every warp publishes by itself.
//
// Why a step's buffers need no release by their reader.  A CTA starts the MMAs of step t + 2 after every unit of its quarter of
// h_{t+1} is published; each of those took the partial sums of step t + 1 of all four CTAs of its cluster, one of which read
// the units of h_t that this CTA published after it had read its accumulators and its received sums of step t.  So two
// accumulators, two receive buffers and two barriers per kind, by the parity of the step, are enough.
// That says nothing about the slots of the ring that h arrives in, which are released by the MMAs that read them: a block's counter
// belongs to another cluster, and may show h_t before this CTA has multiplied its blocks of h_{t-1}.
//
// h_{t-1} was written by other SMs' ordinary stores earlier in this same kernel and is read here by TMA, i.e. through the async
// proxy: the writers release (a release-add on the block's counter), the lane that issues the copy acquires the counter itself
// and then issues fence.proxy.async.  The results are bit-identical to the launch-per-step path: it sums the same quarters of K
// and adds them in the same order (lstm_k_part), step 0 and the cell use the same formulas.
#include <cstring>

#include "tc_common.cuh"

namespace nb {

using namespace tc;

namespace {

constexpr int LP_SLICES = 4;                // CTAs of a cluster = slices of K
constexpr int LP_UNITS = 32;                // hidden units of a cluster = columns of a K block of h
constexpr int LP_CELL_WARPS = 16;           // warps 0-15: accumulators and cells of all groups of rows
constexpr int LP_GROUPS = 4;                // groups of batch rows; each has a warp for its MMAs and one for its h_{t-1} too
constexpr int LP_THREADS = 32 * (LP_CELL_WARPS + 2 * LP_GROUPS);
constexpr int LP_MAX_STAGES = 16;           // of a group
constexpr int LP_SMEM = 227 * 1024;
constexpr int LP_TMEM = 512;
constexpr int LP_COUNTER_STRIDE = 32;       // words: a counter per 128-byte line
constexpr int LP_MAX_BLOCKS = 48;           // K blocks that have a counter
constexpr int LP_BARS = 2 * LP_MAX_STAGES + 4;      // barriers of a group

struct LstmPParams {
    CUtensorMap tm_h;           // rounded hidden states [T][B][H], box {32, Rg, 1}: rows past B arrive as zeros
    const float *w;             // recurrent weights [4H][H], rows [unit][i,f,g,o], TF32-rounded
    const float *pre;           // [T][B][4H] input-side pre-activations (biases included), columns [unit][i,f,g,o]
    float *hr;                  // [T][B][H] rounded hidden states: step t writes [t]; step t + 1 reads it through tm_h
    float *cell, *out;          // [T][B][H]
    int T, B, H;
    int chunk_rows;             // batch rows of a set of clusters
    int Rg;                     // rows of a group, the MMA's N (a multiple of 16)
    int kb_per_slice;           // K blocks per CTA (the last ones may have fewer, or none)
    int slices;                 // CTAs of a cluster that have K blocks
    int stages;                 // ring slots of a group, Rg x 32 floats each
    unsigned int *sync;         // a counter per group and K block, then the exit counter; all zero between launches
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
// ITEMS: cells that a thread finishes (16 warps of 8 units x 4 rows), 1 up to 64 rows, else 2.
template <int ITEMS>
__global__ void __launch_bounds__(LP_THREADS, 1) lstm_persistent_kernel(const __grid_constant__ LstmPParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the group of rows this warp works for: its place among the cell warps, the MMA warps, the TMA warps
    constexpr int CW = LP_CELL_WARPS / LP_GROUPS;
    const int grp = warp < LP_CELL_WARPS ? warp / CW : (warp - LP_CELL_WARPS) % LP_GROUPS;
    const int stage_bytes = p.Rg * 128, stages = p.stages;
    const int KB = (p.H + BLOCK_K - 1) / BLOCK_K;
    const int rank = blockIdx.x % LP_SLICES, cluster = blockIdx.x / LP_SLICES % KB, chunk = blockIdx.x / LP_SLICES / KB;
    const int row0 = chunk * p.chunk_rows + grp * p.Rg;     // the group's first row
    const int rows = max(0, min(p.Rg, min((chunk + 1) * p.chunk_rows, p.B) - row0)), row_end = row0 + rows;
    unsigned int *counters = p.sync + (size_t)(chunk * LP_GROUPS + grp) * KB * LP_COUNTER_STRIDE;     // of this group's rows
    const int quads = (rows + 3) / 4;                        // groups of four batch rows
    const int recv_floats = p.Rg * 32;                       // one CTA's partial sums of a group for this CTA's 32 gate columns
    uint8_t *ring = smem + grp * stages * stage_bytes;       // [stages][Rg rows][128 B], 128-byte swizzle
    float *recv = (float *)(smem + LP_GROUPS * stages * stage_bytes) + grp * 2 * LP_SLICES * recv_floats;   // [parity][source][quad][gate * 8 + unit][4 rows]
    uint64_t *bars = (uint64_t *)(smem + LP_GROUPS * (stages * stage_bytes + 2 * LP_SLICES * recv_floats * 4));
    uint64_t *full = bars + grp * LP_BARS;                   // TMA -> MMA
    uint64_t *empty = full + LP_MAX_STAGES;                  // MMA -> TMA
    uint64_t *acc_full = empty + LP_MAX_STAGES;              // MMA -> accumulator readers, by parity
    uint64_t *recv_full = acc_full + 2;                      // partial sums of all slices have arrived, by parity
    uint32_t *tmem_slot = (uint32_t *)(bars + LP_GROUPS * LP_BARS);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int kb0 = rank * p.kb_per_slice, nkb = max(0, min(p.kb_per_slice, KB - kb0));
    const int cell_warps = min(CW, p.Rg / 4);               // of a group, with rows to send or to finish
    const uint32_t recv_bytes = (uint32_t)(p.slices * quads * 32 * 16);
    if (warp < LP_CELL_WARPS && warp % CW == 0 && lane == 0) {
        for (int s = 0; s < LP_MAX_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&recv_full[a], 1);
        }
        if (warp == 0) *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(&recv_full[0], recv_bytes);          // a phase is armed one round ahead of its data
        mbar_expect_tx(&recv_full[1], recv_bytes);
    }
    if (warp == LP_CELL_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)LP_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t w_col = tmem_base + (uint32_t)(2 * LP_GROUPS * p.Rg), acc_col = tmem_base + (uint32_t)(2 * grp * p.Rg);

    if (warp < LP_CELL_WARPS) {
        // this CTA's slice of the weights: TMEM lane 32 q + 8 g + u holds gate g of unit 8 q + u of the cluster
        const int unit = cluster * LP_UNITS + 8 * (warp & 3) + (lane & 7);
        const float *src = p.w + ((long)4 * unit + (lane >> 3)) * p.H;
        for (int i = warp >> 2; i < nkb; i += LP_CELL_WARPS / 4) {
            const int k0 = (kb0 + i) * BLOCK_K;
            uint32_t v[32];
#pragma unroll
            for (int j = 0; j < 32; j += 4) {               // (H is a multiple of 4: quads lie inside the row or outside)
                const float4 x = unit < p.H && k0 + j < p.H ? __ldg(reinterpret_cast<const float4 *>(src + k0 + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[j] = __float_as_uint(x.x); v[j + 1] = __float_as_uint(x.y); v[j + 2] = __float_as_uint(x.z); v[j + 3] = __float_as_uint(x.w);
            }
            tmem_st_32x32(w_col + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(i * BLOCK_K), v);
        }
        tmem_st_wait();
        tc_fence_before();
    }
    __syncthreads();
    // every CTA of the cluster has its barriers ready before a peer's stores arrive
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc_fence_after();
    bool ok = true;

    if (rows == 0) {
        // (fewer rows than groups)
    } else if (warp >= LP_CELL_WARPS && warp < LP_CELL_WARPS + LP_GROUPS) {
        // ------------------------------------------------ the MMAs of every step
        if (elect_one()) {
            const uint32_t idesc = make_idesc(BLOCK_M, p.Rg);
            int stage = 0;
            uint32_t phase = 0;
            for (int t = 1; t < p.T && nkb > 0 && ok; t++) {
                const uint32_t d = acc_col + (uint32_t)((t & 1) * p.Rg);
                for (int i = 0; i < nkb; i++) {
                    if (!(ok = mbar_wait(&full[stage], phase, abort_flag, p.status))) break;
                    tc_fence_after();
                    const uint32_t b_lo = smem_desc_lo(smem_u32(ring + stage * stage_bytes));
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; k++)
                        umma_tf32_ts(d, w_col + (uint32_t)(i * BLOCK_K + k * UMMA_K), smem_desc(b_lo + 2 * k), idesc, (i | k) != 0);
                    umma_commit(&empty[stage]);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit(&acc_full[t & 1]);
            }
            // the last releases of the ring must have landed before the CTA may exit
            for (int i = 0; i < stages && ok; i++) {
                ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status);
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp >= LP_CELL_WARPS) {
        // ------------------------------------------------ h_{t-1} of every step: lane i fetches K block i of this slice
        int slot = lane % stages;
        uint32_t phase = (uint32_t)(lane / stages) & 1;
        const unsigned int *counter = counters + (size_t)(kb0 + lane) * LP_COUNTER_STRIDE;
        const uint32_t tx = (uint32_t)stage_bytes;
        // A slot's uses are issued in their order.  The use before this lane's belongs to an earlier step, all of whose copies are under
        // way, or to lane - stages (slices of more blocks than slots).  Once it is under way, the slot's barrier is in the phase that
        // ends with its release or in the next; tested earlier, it can be one phase further back, whose predecessor has the parity
        // waited for, and the copy would land on a tile that the MMAs have yet to read.
        const unsigned before = lane < stages ? 0 : 1u << (lane - stages);
        for (int t = 1; t < p.T && ok; t++) {
            bool done = lane >= nkb;
            const unsigned int target = (unsigned int)(LP_SLICES * cell_warps) * (unsigned int)t;
            const long long t0 = clock64();
            while (ok && !__all_sync(0xffffffffu, done)) {
                // lanes whose copy of this step is under way (asked only where two copies of a step share a slot: 20 ns a step)
                const unsigned issued = nkb > stages ? __ballot_sync(0xffffffffu, done) : 0xffffffffu;
                bool give_up = false;
                if (!done) {
                    if (ld_acquire_u32(counter) >= target && (issued & before) == before && mbar_try_wait(&empty[slot], phase ^ 1)) {
                        // the units' stores (generic proxy) are ordered before the acquire; the copy (async proxy) behind this fence
                        asm volatile("fence.proxy.async;" ::: "memory");
                        mbar_expect_tx(&full[slot], tx);
                        tma_load_3d(ring + slot * stage_bytes, &p.tm_h, &full[slot], (kb0 + lane) * BLOCK_K, row0, t - 1);
                        done = true;
                    } else if (*abort_flag || clock64() - t0 > WAIT_LIMIT_CYCLES) {
                        if (!*abort_flag) atomicExch(p.status, (int)DEV_TIMEOUT);
                        *abort_flag = 1;
                        give_up = true;
                    }
                }
                ok = !__any_sync(0xffffffffu, give_up);
            }
            slot += nkb;
            while (slot >= stages) { slot -= stages; phase ^= 1; }
        }
    } else if (warp % CW < cell_warps) {
        // ------------------------------------------------ accumulators to the cluster, cells, and the step's results
        // Every warp by itself: it waits for the MMAs, sends 16 batch rows of 32 gate columns to the CTA that finishes those
        // (TMEM lanes 32 q .. belong to warps of index q modulo 4), waits for what it was sent, finishes 8 units x 4 rows and
        // publishes them.  A cell is a chain of some 600 cycles whatever its neighbours do, so it takes the warps, a cell per
        // thread: four cells per thread of four warps took 2700 cycles of a step's 12 300, and their sends 1200.
        const int q = warp & 3, gw = warp % CW;
        const int u = lane & 7, unit = cluster * LP_UNITS + 8 * rank + u;   // the unit this thread finishes, and its row of a quad
        const bool unit_ok = unit < p.H;
        float c[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) c[i] = 0.0f;
        const uint32_t peer_recv = map_to_rank(smem_u32(recv), (uint32_t)q);
        const uint32_t peer_bar = map_to_rank(smem_u32(recv_full), (uint32_t)q);
        for (int t = 0; t < p.T && ok; t++) {
            const int par = t & 1;
            const uint32_t phase = (uint32_t)((t - 1) >> 1) & 1;            // of both barriers of this parity (t = 1, 2: the first)
            // the input-side pre-activations of this step come from DRAM: fetched while the MMAs run
            float4 z[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const int b = row0 + 4 * (gw + CW * i) + (lane >> 3);
                z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (unit_ok && b < row_end) z[i] = __ldg(reinterpret_cast<const float4 *>(p.pre + ((size_t)t * p.B + b) * 4 * p.H) + unit);
            }
            if (t > 0 && nkb > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[par], phase, abort_flag, p.status));
                if (!ok) break;
                tc_fence_after();
                const uint32_t dst = peer_recv + (uint32_t)(((par * LP_SLICES + rank) * recv_floats + lane * 4) * 4), bar = peer_bar + 8 * par;
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const int j0 = 4 * ((gw >> 2) + CW / 4 * i);            // the first of this warp's quads
                    if (j0 >= quads) break;
                    uint32_t v[16];
                    tmem_ld_32x16(acc_col + ((uint32_t)(q * 32) << 16) + (uint32_t)(par * p.Rg + 4 * j0), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (j0 + j < quads) st_async_v4(dst + (uint32_t)(j0 + j) * 512, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], bar);
                }
                tc_fence_before();
            }
            if (t > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait_cluster(smem_u32(&recv_full[par]), phase, abort_flag, p.status));
                if (!ok) break;
                if (gw == 0 && lane == 0) mbar_expect_tx(&recv_full[par], recv_bytes);      // step t + 2
            }
            float hn[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const int quad = gw + CW * i;
                const size_t b = row0 + 4 * quad + (lane >> 3);
                if (!unit_ok || b >= (size_t)row_end) continue;
                float2 ch;
                if (t == 0) {                   // nothing to multiply: h_{-1} = 0
                    ch = lstm_cell_unit(z[i].x, z[i].y, z[i].z, z[i].w, 0.0f);
                } else {
                    const float *src = recv + par * LP_SLICES * recv_floats + quad * 128 + u * 4 + (lane >> 3);
                    float g[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) g[k] = src[32 * k];
                    for (int s = 1; s < p.slices; s++) {        // the slices of K in order
                        src += recv_floats;
#pragma unroll
                        for (int k = 0; k < 4; k++) g[k] += src[32 * k];
                    }
                    ch = lstm_cell_unit_f32_inline(g[0] + z[i].x, g[1] + z[i].y, g[2] + z[i].z, g[3] + z[i].w, c[i]);
                }
                c[i] = ch.x; hn[i] = ch.y;
                p.hr[((size_t)t * p.B + b) * p.H + unit] = round_tf32(ch.y);
            }
            // ---- this warp's part of the block is published (and its accumulators and sums are read).  What the next step does
            // not read leaves behind it, so that the release does not wait for it
            if (t + 1 < p.T) {
                __syncwarp();
                if (lane == 0) red_release_add(counters + (size_t)cluster * LP_COUNTER_STRIDE, 1u);
            }
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const int b = row0 + 4 * (gw + CW * i) + (lane >> 3);
                if (!unit_ok || b >= row_end) continue;
                const size_t o = ((size_t)t * p.B + b) * p.H + unit;
                p.cell[o] = c[i];
                p.out[o] = hn[i];
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
    if (warp == LP_CELL_WARPS) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)LP_TMEM) : "memory");
    }
    // no CTA leaves while a peer may still store into it
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // the last CTA of the grid to get here leaves the counters as it found them (nobody polls any more)
    if (warp == 0) {
        const int exits = (int)gridDim.x / LP_SLICES * LP_GROUPS;
        bool last = false;
        if (lane == 0) {
            __threadfence();
            last = atomicAdd(p.sync + (size_t)exits * LP_COUNTER_STRIDE, 1u) == gridDim.x - 1;
        }
        if (__any_sync(0xffffffffu, last))
            for (int i = lane; i <= exits; i += 32) p.sync[(size_t)i * LP_COUNTER_STRIDE] = 0;
    }
}

struct LstmPLaunch : LaunchRecord {
    LstmPParams p;
    int grid, smem;
    double flops;
};

const void *kernel_of(int B) { return B <= 64 ? (const void *)lstm_persistent_kernel<1> : (const void *)lstm_persistent_kernel<2>; }

int rows_of(int B) { return (B + 16 * LP_GROUPS - 1) / (16 * LP_GROUPS) * 16; }       // of a group
int smem_of(int B, int stages) {
    return LP_GROUPS * (stages + 2 * LP_SLICES) * rows_of(B) * 128 + 1024 + 8 * LP_GROUPS * LP_BARS + 16;
}
int stages_of(int B) {
    int s = LP_MAX_STAGES;
    while (s > 1 && smem_of(B, s) > LP_SMEM) s--;
    return s;
}

}  // namespace

// Limits set, and clusters counted, when the first layer asks.
static int clusters_at_once(const nb_handle_s *h) {
    if (h->lstm_clusters >= 0) return h->lstm_clusters;
    for (int B : {64, 128}) NB_CHECK_CUDA(cudaFuncSetAttribute(kernel_of(B), cudaFuncAttributeMaxDynamicSharedMemorySize, LP_SMEM));
    // clusters of four that run at once, with a CTA per SM (the kernel takes all of tensor memory)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(LP_SLICES);
    cfg.blockDim = dim3(LP_THREADS);
    cfg.dynamicSmemBytes = LP_SMEM;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = LP_SLICES; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel_of(128), &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    return h->lstm_clusters = n;
}

int lstm_persistent_counters() { return (LP_GROUPS * LP_MAX_BLOCKS + 1) * LP_COUNTER_STRIDE; }

// K blocks of one slice of a recurrent product.
int lstm_k_part(int H) {
    const int KB = (H + BLOCK_K - 1) / BLOCK_K;
    return (KB + LP_SLICES - 1) / LP_SLICES;
}

namespace {

// A batch runs as equal chunks of at most 128 rows, each on a set of clusters of its own.
int chunks_of(int B) { return (B + 127) / 128; }
int chunk_rows_of(int B) { return (B + chunks_of(B) - 1) / chunks_of(B); }

}  // namespace

// Whether the recurrence of an LSTM layer can run as the persistent kernel: TF32 mode on the tensor-core path, gate layers
// without an activation of their own, whole quads of units, weights and accumulators that fit tensor memory, all clusters
// resident at once (up to 128 rows at H = 1024, 256 at 512, 1024 at 128).  A second launch for more rows gains little or loses:
// H = 1024, 8 steps: B = 129 / 256 / 512: 306 / 352 / 669 us in two or four launches, 309 / 344 / 472 launched step by step.
// Two steps have one product, and the kernel's set-up costs more than its launch (T2 B64 H416, two layers: 66 and 54 us).
bool lstm_persistent_supported(const nb_handle_s *h, int T, int B, int H) {
    if (!h->encode_tiled || h->cc_major != 10 || !h->cooperative_launch) return false;
    if (T < 3 || B < 1 || H < 32 || (H % 4) != 0 || (B > 128 && (H % 32) != 0)) return false;
    const long KB = (H + BLOCK_K - 1) / BLOCK_K;
    if (lstm_k_part(H) > 32 || KB * chunks_of(B) > std::min(clusters_at_once(h), LP_MAX_BLOCKS)) return false;
    return 2 * LP_GROUPS * rows_of(chunk_rows_of(B)) + lstm_k_part(H) * BLOCK_K <= LP_TMEM;
}

// The order of additions is the width's: the batches and sequences that a launch per step takes add the slices that this kernel would
// add, so that a batch and its slices give the same bits.  Against K whole, H = 1024, a step takes 19.4 -> 19.5 us at 256 rows, 25.9 ->
// 27.2 at 512; H = 416 at 1000 rows 20.5 -> 21.9.
bool lstm_in_slices(const nb_handle_s *h, int H) { return lstm_persistent_supported(h, 3, 1, H); }

// All steps of the recurrence: writes cell, out and hr.
void lstm_persistent(nb_handle_s *h, const float *w_hi, const float *pre, float *cell, float *out, float *hr, int T, int B, int H) {
    std::string key;
    key.push_back('P');
    key_add(key, w_hi); key_add(key, pre); key_add(key, cell); key_add(key, out); key_add(key, hr);
    key_add(key, T); key_add(key, B); key_add(key, H);
    auto it = h->launch_cache.find(key);
    if (it == h->launch_cache.end()) {
        std::unique_ptr<LstmPLaunch> L(new LstmPLaunch());
        std::memset(&L->p, 0, sizeof L->p);
        const long long F4 = 4;
        const int KB = (H + BLOCK_K - 1) / BLOCK_K, rows = chunk_rows_of(B), Rg = rows_of(rows);
        check_extent(h, w_hi, 0, (long long)4 * H * H * F4, "recurrent weights");
        check_extent(h, pre, 0, (long long)T * B * 4 * H * F4, "input-side pre-activations");
        check_extent(h, cell, 0, (long long)T * B * H * F4, "cell states");
        check_extent(h, out, 0, (long long)T * B * H * F4, "hidden states");
        // (columns past H and rows past B arrive as zeros, but are read)
        const long long last = (long long)(chunks_of(B) - 1) * rows + LP_GROUPS * Rg;
        check_extent(h, hr, 0, (((long long)(T - 1) * B + last) * H + KB * BLOCK_K - H) * F4, "rounded hidden states");
        cuuint64_t dims[3] = {(cuuint64_t)H, (cuuint64_t)B, (cuuint64_t)T};
        cuuint64_t strides[2] = {(cuuint64_t)H * 4, (cuuint64_t)H * 4 * (cuuint64_t)B};
        cuuint32_t bx[3] = {(cuuint32_t)BLOCK_K, (cuuint32_t)Rg, 1};
        cuuint32_t es[3] = {1, 1, 1};
        encode_tensor_map(h, &L->p.tm_h, hr, 3, dims, strides, bx, es);
        L->p.w = w_hi; L->p.pre = pre; L->p.hr = hr; L->p.cell = cell; L->p.out = out;
        L->p.T = T; L->p.B = B; L->p.H = H; L->p.chunk_rows = rows; L->p.Rg = Rg;
        L->p.kb_per_slice = lstm_k_part(H);
        L->p.slices = (KB + L->p.kb_per_slice - 1) / L->p.kb_per_slice;
        L->p.stages = stages_of(rows);
        L->p.sync = h->d_grid_sync; L->p.status = h->d_status;
        L->grid = KB * LP_SLICES * chunks_of(B);
        L->smem = smem_of(rows, L->p.stages);
        L->flops = 2.0 * (double)(T - 1) * B * 4.0 * H * H;
        if (h->launch_cache.size() > 4096) h->launch_cache.clear();
        it = h->launch_cache.emplace(std::move(key), std::move(L)).first;
    }
    const LstmPLaunch &L = static_cast<const LstmPLaunch &>(*it->second);
    ProfileScope prof(h, 0, L.flops);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.grid);
    cfg.blockDim = dim3(LP_THREADS);
    cfg.dynamicSmemBytes = (size_t)L.smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = LP_SLICES; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    void *args[1] = {const_cast<LstmPParams *>(&L.p)};
    NB_CHECK_CUDA(cudaLaunchKernelExC(&cfg, kernel_of(chunk_rows_of(B)), args));
    check_launch("lstm_persistent_kernel");
    count_launch(h);
    prof.finish();
}

}  // namespace nb
