// The recurrence of one LSTM or RNN layer as ONE kernel over all time steps, in exact fp32 on the CUDA cores
// (lstm_layer.cc:250-311, rnn_layer.cc:91-141): layers whose recurrent weights fit the shared memory of one cluster.
//
// Bound by latency: a step of such a layer is a few hundred nanoseconds of arithmetic, and a launch per step cost
// 15-30 us of pipeline fill, single-lane issue and activation chains (one SM's worth of them).  A cluster of CS CTAs
// keeps the whole recurrent matrix in its shared memory for all steps (CTA r: the rows of U hidden units, fp32),
// and each cluster runs RB rows of the batch by itself: batch rows never meet, so there is no grid barrier and no
// co-residency requirement beyond the cluster's own.  Per step every warp multiplies 16 weight rows by a slice of K
// for the RB states (both from shared memory, packed FMAs along K), four K lanes are added by shuffles, the warps' partial
// sums through shared memory; one thread per (unit, batch row) then adds the input-side values fetched a step ahead,
// runs the cell update and stores the new state into the shared memory of all CS CTAs; a cluster barrier ends the step.
// The step's results leave for HBM between the barrier's arrive and its wait: an arrive releases what was stored in front
// of it, so there it would wait for HBM on every step (T35 B20 H300: 4.1 us a step in front, 2.8 us behind).
// CS depends on the layer only, so batches that run here add in the same order as their slices; how large a batch runs
// here at all, and not a launch per step, depends on the batch too (recurrent_cluster_pays).
#include <cooperative_groups.h>

#include "tc_common.cuh"

namespace nb {

namespace {

namespace cg = cooperative_groups;
using namespace tc;

constexpr int RC_THREADS = 512, RC_WARPS = RC_THREADS / 32;
constexpr int RC_ITEMS = 2;             // (unit, batch row) pairs a thread may own

// Row stride in shared memory: whole quads, 4 floats off a multiple of 32, so that a 128-bit read of eight rows falls
// into 32 different banks.
__host__ __device__ inline int padded_stride(int H) { return (H - 4 + 31) / 32 * 32 + 4; }

struct Shape {
    int CS, RB;             // cluster size, batch rows per cluster
    int U, RP;              // units per CTA; pairs of weight rows (a multiple of 8)
    int rg, kg;             // warps along the rows and along K
    int Hs;
    int warps;              // > 0: recurrent_warp_kernel, with so many warps; its CTAs that have units, its columns per lane
    int active, kj;
    size_t smem;
};

struct RecParams {
    RecurrentArgs a;
    Shape s;
    int *status;
};

__device__ __forceinline__ void ffma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

template <int RB, int G>            // G: gates, 4 (LSTM) or 1 (RNN)
__global__ void __launch_bounds__(RC_THREADS, 1) recurrent_cluster_kernel(const RecParams p) {
    extern __shared__ __align__(16) float smem[];
    const RecurrentArgs &a = p.a;
    const int H = a.H, Hs = p.s.Hs, rows2 = 2 * p.s.RP;
    float *w_s = smem;                              // [2 RP][Hs]
    float *h_s = w_s + rows2 * Hs;                  // [2][RB][Hs]: the state read by this step and written by it
    float *part = h_s + 2 * RB * Hs;                // [kg][RB][2 RP]
    cg::cluster_group cluster = cg::this_cluster();
    const int CS = p.s.CS, rank = CS > 1 ? (int)cluster.block_rank() : 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = (int)(blockIdx.x / CS) * RB;
    const int unit0 = rank * p.s.U, nu = max(0, min(p.s.U, H - unit0));

    grid_dependents_start();
    // recurrent weights (constant: not waited for), zero where the layer has none
    for (int r = warp; r < rows2; r += RC_WARPS) {
        const float *src = a.w + ((long)G * unit0 + r) * H;
        for (int k = lane; k < Hs; k += 32) w_s[r * Hs + k] = (r < G * nu && k < H) ? __ldg(src + k) : 0.0f;
    }
    for (int i = tid; i < 2 * RB * Hs; i += RC_THREADS) h_s[i] = 0.0f;
    grid_dependency_wait();
    if (G == 1) {                                   // step 0 of an RNN multiplies the input gate's output
        __syncthreads();
        for (int i = tid; i < RB * H; i += RC_THREADS) {
            const int b = i / H, k = i - b * H;
            if (b0 + b < a.B) h_s[b * Hs + k] = a.pre[(long)(b0 + b) * H + k];
        }
    }

    // the (unit, batch row) pairs this thread finishes
    int item_u[RC_ITEMS], item_b[RC_ITEMS];
    float c[RC_ITEMS], z[RC_ITEMS][G], scale[RC_ITEMS], shift[RC_ITEMS][G];
    auto fetch_pre = [&](int t, int i, float (&v)[G]) {
        const float *src = a.pre + ((long)t * a.B + b0 + item_b[i]) * G * H + (long)G * (unit0 + item_u[i]);
        if constexpr (G == 4) {
            const float4 q = *reinterpret_cast<const float4 *>(src);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
            v[0] = *src;
        }
    };
#pragma unroll
    for (int i = 0; i < RC_ITEMS; i++) {
        const int e = tid + i * RC_THREADS;
        item_b[i] = nu ? e / nu : RB;
        item_u[i] = nu ? e - item_b[i] * nu : 0;
        if (item_b[i] >= RB || b0 + item_b[i] >= a.B) item_b[i] = -1;
        c[i] = 0.0f; scale[i] = 1.0f;
#pragma unroll
        for (int g = 0; g < G; g++) { z[i][g] = 0.0f; shift[i][g] = 0.0f; }
        if (item_b[i] >= 0) {
            fetch_pre(0, i, z[i]);
            if (a.scale) scale[i] = a.scale[unit0 + item_u[i]];
#pragma unroll
            for (int g = 0; g < G; g++)
                if (a.shift) shift[i][g] = a.shift[(long)G * (unit0 + item_u[i]) + g];
        }
    }
    if (CS > 1) cluster.sync();
    else __syncthreads();

    const int rp = (warp % p.s.rg) * 8 + (lane & 7), kg = warp / p.s.rg;
    const bool multiplies = kg < p.s.kg;
    const int KS = 4 * p.s.kg, ks = 4 * kg + (lane >> 3), H4 = (H + 3) / 4;
    const float *wa = w_s + rp * Hs, *wb = w_s + (rp + p.s.RP) * Hs;
    for (int t = 0; t < a.T; t++) {
        const float *h_cur = h_s + (t & 1) * RB * Hs;
        const int next_off = ((t + 1) & 1) * RB * Hs;
        if (multiplies) {
            unsigned long long acc[2][RB];
#pragma unroll
            for (int b = 0; b < RB; b++) acc[0][b] = acc[1][b] = 0ull;
            for (int k4 = ks; k4 < H4; k4 += KS) {
                const ulonglong2 v0 = *reinterpret_cast<const ulonglong2 *>(wa + 4 * k4);
                const ulonglong2 v1 = *reinterpret_cast<const ulonglong2 *>(wb + 4 * k4);
#pragma unroll
                for (int b = 0; b < RB; b++) {
                    const ulonglong2 hv = *reinterpret_cast<const ulonglong2 *>(h_cur + b * Hs + 4 * k4);
                    ffma2(acc[0][b], v0.x, hv.x); ffma2(acc[0][b], v0.y, hv.y);
                    ffma2(acc[1][b], v1.x, hv.x); ffma2(acc[1][b], v1.y, hv.y);
                }
            }
            // The 2 RB sums of eight rows' pairs lie in four lanes: two exchanges halve the values and the lanes' shares (each
            // lane ends with RB / 2 of them)
            constexpr int N = 2 * RB;
            float v[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                const unsigned long long s = acc[i / RB][i % RB];
                v[i] = __uint_as_float((unsigned)s) + __uint_as_float((unsigned)(s >> 32));
            }
            const bool hi = lane & 16, odd = lane & 8;
#pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const float mine = hi ? v[i + N / 2] : v[i], theirs = hi ? v[i] : v[i + N / 2];
                v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, 16);
            }
            if constexpr (N == 2) {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
                if (!odd) part[kg * rows2 + rp + (hi ? p.s.RP : 0)] = v[0];
            } else {
#pragma unroll
                for (int i = 0; i < N / 4; i++) {
                    const float mine = odd ? v[i + N / 4] : v[i], theirs = odd ? v[i] : v[i + N / 4];
                    v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, 8);
                }
#pragma unroll
                for (int i = 0; i < N / 4; i++)         // row half `hi`, batch row (odd ? RB / 2 : 0) + i
                    part[(kg * RB + (odd ? N / 4 : 0) + i) * rows2 + rp + (hi ? p.s.RP : 0)] = v[i];
            }
        }
        __syncthreads();
        const bool more = t + 1 < a.T;
        float y[RC_ITEMS];
#pragma unroll
        for (int i = 0; i < RC_ITEMS; i++) {
            if (item_b[i] < 0) continue;
            const int u = item_u[i], b = item_b[i];
            float v[G], state;
#pragma unroll
            for (int g = 0; g < G; g++) v[g] = 0.0f;
#pragma unroll 4
            for (int q = 0; q < p.s.kg; q++) {
                const float *src = part + (q * RB + b) * rows2 + G * u;
                if constexpr (G == 4) {
                    const float4 w = *reinterpret_cast<const float4 *>(src);
                    v[0] += w.x; v[1] += w.y; v[2] += w.z; v[3] += w.w;
                } else {
                    v[0] += *src;
                }
            }
            if constexpr (G == 4) {
#pragma unroll
                for (int g = 0; g < 4; g++)         // linear gate layers: their shifts are in `pre` already
                    v[g] = z[i][g] + (a.act == NB_ACT_LINEAR ? v[g] : apply_activation_call(v[g] + shift[i][g], a.act));
                const float2 ch = a.cell_f32 ? lstm_cell_unit_f32_inline(v[0], v[1], v[2], v[3], c[i])
                                             : lstm_cell_unit(v[0], v[1], v[2], v[3], c[i]);
                c[i] = ch.x; state = y[i] = ch.y;
            } else {
                const float hv = apply_activation_fast(a.scale ? fmaf(v[0], scale[i], shift[i][0]) : v[0] + shift[i][0], a.act);
                state = z[i][0] + hv;
                y[i] = t == 0 ? hv : state;         // what the output gate reads: h_0, then the states
            }
            if (more) {
                float *dst = h_s + next_off + b * Hs + unit0 + u;
                for (int q = 0; q < CS; q++) *(CS > 1 ? cluster.map_shared_rank(dst, q) : dst) = state;
            }
        }
        if (more && CS > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
#pragma unroll
        for (int i = 0; i < RC_ITEMS; i++) {
            if (item_b[i] < 0) continue;
            const long o = ((long)t * a.B + b0 + item_b[i]) * H + unit0 + item_u[i];
            if constexpr (G == 4) {
                a.cell[o] = c[i];
                a.out[o] = y[i];
                if (a.out_round) a.out_round[o] = round_tf32(y[i]);
            } else {
                a.out[o] = a.round_out ? round_tf32(y[i]) : y[i];
            }
            if (more) fetch_pre(t + 1, i, z[i]);
        }
        if (more) {         // (the last step sends nothing: no CTA leaves before its peers' stores)
            if (CS > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            else __syncthreads();
        }
    }
}

// ---- the same recurrence with the weights in registers, for layers of up to 384 units
// A warp owns four weight rows (the gates of a unit, or four units of an RNN) and a lane the columns lane, lane + 32, ... of them,
// in registers for the whole sequence: a step reads only the states from shared memory, once per warp for all four rows.  The
// 4 RB sums are reduced over the lanes by halving exchanges; each lane then finishes one gate (or RNN unit) of one batch row, so
// the gates' activations run side by side.  New states go straight to the CTAs of the cluster that have units, by st.async onto
// the receiver's mbarrier, which expects a whole step's states: no CTA-wide and no cluster-wide barrier in a step.  Two buffers and
// two barriers, by the parity of the step, are enough: a warp sends states of step t after it has received all of step t - 1, and so
// after every warp of the cluster has read the states of step t - 2.  The order of additions depends on the width only.
// Bound by the chain of a step and by its warps' instructions (about 360 a warp at 300 units and 4 rows, 160 of them FMAs).  Against
// weights in shared memory, per step: LSTM 300 units, 20 rows 2.71 -> 1.82 us, 100 units 1.44 -> 0.89, RNN 256 units, 32 rows 1.51 ->
// 1.28; the networks LSTM T35 B20 H300 254 -> 194 us, RNN T16 B32 H256 102 -> 91 us.
constexpr int RW_COLS = 12;             // most columns per lane
constexpr int RW_ROWS = 4;              // weight rows of a warp
constexpr int rw_max_warps(int RB) { return RB == 8 ? 19 : 24; }

template <int RB, int G>
__global__ void __launch_bounds__(32 * rw_max_warps(RB), 1) recurrent_warp_kernel(const RecParams p) {
    constexpr int VW = RB < 4 ? RB : 4, HALVES = RB / VW;           // batch rows of a vector of states
    constexpr int N = RW_ROWS * RB, D = 32 / N;                     // sums of a warp, lanes that end with the same one
    constexpr int SENDS = G == 4 ? 1 : (RB == 8 ? 4 : 2);           // vectors a lane sends: (4 units) x halves x 16 CTAs / 32
    extern __shared__ __align__(16) float smem[];
    const RecurrentArgs &a = p.a;
    const int H = a.H, K = 32 * p.s.kj;
    float *h_s = smem;                              // [2][HALVES][K][VW]
    uint64_t *bars = (uint64_t *)(h_s + 2 * K * RB);
    volatile int *abort_flag = (volatile int *)(bars + 2);
    const int CS = p.s.CS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)(blockIdx.x % CS), b0 = (int)(blockIdx.x / CS) * RB;
    const int unit0 = rank * p.s.U, nu = max(0, min(p.s.U, H - unit0));
    const int first = G == 4 ? warp : RW_ROWS * warp;               // this warp's first unit
    const bool active = first < nu;
    const uint32_t step_bytes = (uint32_t)(H * RB * 4);

    grid_dependents_start();
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(&bars[0], step_bytes);       // a phase is armed one round ahead of its data
        mbar_expect_tx(&bars[1], step_bytes);
    }
    for (int i = tid; i < 2 * K * RB; i += blockDim.x) h_s[i] = 0.0f;
    // recurrent weights (constant: not waited for), zero past the layer's
    float w[RW_ROWS][RW_COLS];
#pragma unroll
    for (int r = 0; r < RW_ROWS; r++) {
        const bool row_ok = active && (G == 4 || first + r < nu);
        const float *src = a.w + ((long)G * (unit0 + first) + r) * H;
#pragma unroll
        for (int j = 0; j < RW_COLS; j++) w[r][j] = row_ok && lane + 32 * j < H ? __ldg(src + lane + 32 * j) : 0.0f;
    }
    // the sum this lane ends with: weight row `row`, batch row `b`
    const int row = lane / D / RB, b = lane / D % RB;
    const int my_unit = unit0 + first + (G == 4 ? 0 : row);
    const bool mine = active && (G == 4 || first + row < nu) && b0 + b < a.B, writes = mine && lane % D == 0;
    const float scale = G == 1 && a.scale && mine ? a.scale[my_unit] : 1.0f;
    const float shift = a.shift && mine ? a.shift[G == 4 ? 4 * my_unit + row : my_unit] : 0.0f;
    // the vectors of states this lane sends: where to, and the lane that holds the first of them
    uint32_t to[SENDS], to_bar[SENDS];
    int from[SENDS];
#pragma unroll
    for (int i = 0; i < SENDS; i++) {
        const int e = lane + 32 * i, dest = e % p.s.active, rest = e / p.s.active, half = rest % HALVES, r = rest / HALVES;
        const bool in = active && r < (G == 4 ? 1 : RW_ROWS) && (G == 4 || first + r < nu);
        from[i] = in ? (r * RB + half * VW) * D : -1;
        const int k = unit0 + first + r;
        to[i] = in ? map_to_rank(smem_u32(h_s + (half * K + k) * VW), (uint32_t)dest) : 0;
        to_bar[i] = in ? map_to_rank(smem_u32(bars), (uint32_t)dest) : 0;
    }
    grid_dependency_wait();
    __syncthreads();
    if (G == 1) {                                   // step 0 of an RNN multiplies the input gate's output
        for (int i = tid; i < RB * H; i += blockDim.x) {
            const int bb = i / H, k = i - bb * H;
            if (b0 + bb < a.B) h_s[(bb / VW * K + k) * VW + bb % VW] = a.pre[(long)(b0 + bb) * H + k];
        }
    }
    auto fetch_pre = [&](int t) {
        const long at = (long)t * a.B + b0 + b;
        return mine ? a.pre[G == 4 ? (at * H + my_unit) * 4 + row : at * H + my_unit] : 0.0f;
    };
    float z = fetch_pre(0), c = 0.0f;
    // every CTA of the cluster has its barriers ready before a peer's stores arrive
    __syncwarp();
    if (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();

    bool ok = true;
    for (int t = 0; t < a.T && active; t++) {
        const int par = t & 1;
        const float *h_cur = h_s + par * K * RB;
        if (t > 0) {
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(smem_u32(&bars[par]), (uint32_t)((t - 1) >> 1) & 1, abort_flag, p.status));
            if (!ok) break;
            if (tid == 0) mbar_expect_tx(&bars[par], step_bytes);       // step t + 2
        }
        float v[N];
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = 0.0f;
        if (G == 1 || t > 0) {                      // (an LSTM starts from zero states)
#pragma unroll
            for (int j = 0; j < RW_COLS; j++) {
                if (j >= p.s.kj) break;
                float hv[RB];
#pragma unroll
                for (int q = 0; q < HALVES; q++) {
                    const float *src = h_cur + (q * K + lane + 32 * j) * VW;
                    if constexpr (VW == 4) {
                        const float4 x = *reinterpret_cast<const float4 *>(src);
                        hv[4 * q] = x.x; hv[4 * q + 1] = x.y; hv[4 * q + 2] = x.z; hv[4 * q + 3] = x.w;
                    } else if constexpr (VW == 2) {
                        const float2 x = *reinterpret_cast<const float2 *>(src);
                        hv[0] = x.x; hv[1] = x.y;
                    } else {
                        hv[0] = *src;
                    }
                }
#pragma unroll
                for (int r = 0; r < RW_ROWS; r++)
#pragma unroll
                    for (int i = 0; i < RB; i++) v[r * RB + i] = fmaf(w[r][j], hv[i], v[r * RB + i]);
            }
            // exchanges that halve the sums a lane keeps, then plain ones among the lanes that are left with the same sum
            int n = N;
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) {
                if (n > 1) {
                    n >>= 1;
                    const bool hi = lane & m;
#pragma unroll
                    for (int i = 0; i < N / 2; i++) {
                        if (i >= n) break;
                        const float keep = hi ? v[i + n] : v[i], give = hi ? v[i] : v[i + n];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
                    }
                } else {
                    v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
                }
            }
        }
        float state, y;
        if constexpr (G == 4) {
            // linear gate layers: their shifts are in `pre` already
            const float x = z + (a.act == NB_ACT_LINEAR ? v[0] : apply_activation_call(v[0] + shift, a.act));
            float gate;
            if (a.cell_f32) gate = row == 2 ? tanhf(x) : 1.0f / (1.0f + expf(-x));
            else gate = row == 2 ? tanh_double(x) : logistic_double(x);
            const float ig = __shfl_sync(0xffffffffu, gate, b * D), fg = __shfl_sync(0xffffffffu, gate, (RB + b) * D);
            const float gg = __shfl_sync(0xffffffffu, gate, (2 * RB + b) * D), og = __shfl_sync(0xffffffffu, gate, (3 * RB + b) * D);
            c = __fadd_rn(__fmul_rn(c, fg), __fmul_rn(ig, gg));         // separate roundings, as on the CPU path
            state = y = __fmul_rn(a.cell_f32 ? tanhf(c) : tanh_double(c), og);
        } else {
            const float hv = apply_activation_fast(a.scale ? fmaf(v[0], scale, shift) : v[0] + shift, a.act);
            state = z + hv;
            y = t == 0 ? hv : state;                // what the output gate reads: h_0, then the states
        }
        const bool more = t + 1 < a.T;
        if (more) {
            const uint32_t off = (uint32_t)((1 - par) * K * RB * 4), bar_off = (uint32_t)(8 * (1 - par));
#pragma unroll
            for (int i = 0; i < SENDS; i++) {
                uint32_t q[VW];
#pragma unroll
                for (int e = 0; e < VW; e++) q[e] = __float_as_uint(__shfl_sync(0xffffffffu, state, max(from[i], 0) + e * D));
                if (from[i] < 0) continue;
                if constexpr (VW == 4) st_async_v4(to[i] + off, q[0], q[1], q[2], q[3], to_bar[i] + bar_off);
                else if constexpr (VW == 2) st_async_v2(to[i] + off, q[0], q[1], to_bar[i] + bar_off);
                else st_async(to[i] + off, q[0], to_bar[i] + bar_off);
            }
        }
        if (writes) {
            const long o = ((long)t * a.B + b0 + b) * H + my_unit;
            if constexpr (G == 4) {                 // the lanes of the gates share the stores
                if (row == 0) a.cell[o] = c;
                else if (row == 1) a.out[o] = y;
                else if (row == 2 && a.out_round) a.out_round[o] = round_tf32(y);
            } else {
                a.out[o] = a.round_out ? round_tf32(y) : y;
            }
        }
        if (more) z = fetch_pre(t + 1);
    }
    if (!ok) *abort_flag = 1;
    __syncthreads();
    __syncwarp();
    if (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

typedef void (*RecKernel)(const RecParams);
const RecKernel WARP_KERNELS[2][4] = {
    {recurrent_warp_kernel<1, 1>, recurrent_warp_kernel<2, 1>, recurrent_warp_kernel<4, 1>, recurrent_warp_kernel<8, 1>},
    {recurrent_warp_kernel<1, 4>, recurrent_warp_kernel<2, 4>, recurrent_warp_kernel<4, 4>, recurrent_warp_kernel<8, 4>}};
const RecKernel KERNELS[2][4] = {       // [LSTM][rows per cluster: 1, 2, 4, 8]
    {recurrent_cluster_kernel<1, 1>, recurrent_cluster_kernel<2, 1>, recurrent_cluster_kernel<4, 1>, recurrent_cluster_kernel<8, 1>},
    {recurrent_cluster_kernel<1, 4>, recurrent_cluster_kernel<2, 4>, recurrent_cluster_kernel<4, 4>, recurrent_cluster_kernel<8, 4>}};
constexpr int MAX_SMEM = 227 * 1024;

bool shape_of(int gates, int H, int CS, int RB, bool registers, Shape *s) {
    s->CS = CS; s->RB = RB;
    s->U = (H + CS - 1) / CS;
    s->warps = 0;
    if (registers) {
        s->warps = gates == 4 ? s->U : (s->U + RW_ROWS - 1) / RW_ROWS;
        s->active = (H + s->U - 1) / s->U;
        s->kj = (H + 31) / 32;
        s->smem = sizeof(float) * 2 * 32 * s->kj * RB + 32;
        return s->warps <= rw_max_warps(RB);
    }
    s->RP = ((gates * s->U + 1) / 2 + 7) / 8 * 8;
    s->rg = s->RP / 8;
    if (s->rg > RC_WARPS || RB * s->U > RC_ITEMS * RC_THREADS) return false;
    s->kg = RC_WARPS / s->rg;
    s->Hs = padded_stride(H);
    s->smem = sizeof(float) * ((size_t)2 * s->RP * s->Hs + (size_t)2 * RB * s->Hs + (size_t)s->kg * 2 * s->RP * RB);
    return s->smem <= MAX_SMEM;
}

// Clock cycles of a step, fitted to measurements of RNN and LSTM layers of 40 to 600 units: every warp row-group reads its
// 16 weight rows (8 wavefronts per K quad and eight rows) and multiplies RB states with them; the rest of a step is the
// chain of reductions, cell and exchange (RNN H256, clusters of 8: 1.0 / 1.1 / 1.4 / 1.9 us at RB = 1 / 2 / 4 / 8; H40 in a
// single CTA: 0.7 us).
double step_cost(int gates, const Shape &s, int H) {
    // weights in registers: a warp takes some 2 cycles of its SM per column and batch row, and 25 for the rest of its step
    // (LSTM 300 units in 16 CTAs, 4 rows: 1.82 us; 100 in 16 / 8: 0.89 / 1.04; RNN 256 in 4, 1 / 2 / 4 rows: 1.28 / 1.43 / 1.75)
    if (s.warps) return (gates == 4 ? 1500.0 : 1700.0 + 200.0 * s.RB) - (s.CS > 1 ? 0.0 : 300.0) + s.warps * (2.0 * s.RB * s.kj + 25.0);
    return (double)s.rg * H / 16 * (8 + 2.5 * s.RB) + (s.CS > 1 ? 1600.0 : 1150.0) + 130.0 * s.RB;
}

// Rows per cluster from the batch, and the cluster size too where the order of additions does not depend on it; else that comes
// from the layer alone (at a batch of 32).
int waves_of(const nb_handle_s *h, const Shape &s, int B) {
    const int at_once = s.CS == 1 ? h->sm_count : h->clusters_at_once[s.CS];
    return ((B + s.RB - 1) / s.RB + at_once - 1) / at_once;
}

bool choose(const nb_handle_s *h, int gates, int H, int B, bool registers, Shape *best) {
    auto pick = [&](int batch, int cs_lo, int cs_hi) {
        double best_cost = -1;
        for (int CS = cs_lo; CS <= cs_hi; CS *= 2) {
            const int at_once = CS == 1 ? h->sm_count : h->clusters_at_once[CS];
            if (at_once < 1) continue;
            for (int RB = 1; RB <= 8; RB *= 2) {
                Shape s;
                if (!shape_of(gates, H, CS, RB, registers, &s)) continue;
                const double cost = waves_of(h, s, batch) * step_cost(gates, s, H);
                if (best_cost < 0 || cost < best_cost) { best_cost = cost; *best = s; }
            }
        }
        return best_cost >= 0;
    };
    if (registers) return pick(B, 1, 16);
    return pick(32, 1, 16) && pick(B, best->CS, best->CS);
}

// Do the weights lie in registers?  Where that takes less time over all waves: its CTAs hold 24 warps of four rows at most (19 with
// eight batch rows), so that wide layers need large clusters, few of which run at once (LSTM, 16 steps, two layers: 256 rows of 200
// units 490 us in registers, 266 in shared memory).  On the CUDA cores, up to 256 rows, the layer decides:
// at 32 and at 256 rows.
bool in_registers(const nb_handle_s *h, const RecurrentArgs &a) {
    auto less = [&](int B) {
        Shape reg, mem;
        if (!choose(h, a.gates, a.H, B, true, &reg)) return false;
        if (!choose(h, a.gates, a.H, B, false, &mem)) return true;
        return waves_of(h, reg, B) * step_cost(a.gates, reg, a.H) <= 1.25 * waves_of(h, mem, B) * step_cost(a.gates, mem, a.H);
    };
    return a.H <= 32 * RW_COLS && (a.by_layer ? less(32) && less(256) : less(a.B));
}

}  // namespace

// Once per handle, when a plan first asks whether its layer runs here (a millisecond for the first handle of a process that
// has such a plan, 0.03 ms for the others).
static void prepare_device(nb_handle_s *h) {
    if (h->recurrent_ready) return;
    for (auto &set : {KERNELS, WARP_KERNELS})
        for (int kind = 0; kind < 2; kind++)
            for (RecKernel k : set[kind]) {
                NB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
                NB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            }
    // how many clusters of each size run at once (they do not span the groups of SMs the part is made of, and 16 CTAs
    // are beyond the portable size)
    for (int CS = 2; CS <= 16; CS *= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)CS);
        cfg.blockDim = dim3(RC_THREADS);
        cfg.dynamicSmemBytes = MAX_SMEM;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)CS; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, KERNELS[1][0], &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
        h->clusters_at_once[CS] = n;
    }
    h->recurrent_ready = true;
}

// Fits, and beats a launch per step.  A cluster runs at most 8 rows, so large batches go through it in waves, each of which
// loads the weights again; a launch per step takes its batch at once.  Fitted in microseconds to LSTM and RNN layers of 33 to
// 864 units, batches of 1 to 2048, 4 and 36 steps; the better of the two is missed by 26 % at most, seldom by 10 %:
//   cluster   waves * (2 + 0.03 per KB of shared memory + T * step_cost * 1.4, 1.2 more for gate layers with an activation)
//   per step  T * step, without the first product where the state is zero, and two launches more for the RNN.  A TF32 step
//             takes 12.5 (LSTM), 17 (LSTM with an activation) or 15 us (RNN), a 3xTF32 one 17.5, 24 or 20, on the CUDA cores
//             16 + 0.02 H + 45 per GFLOP (LSTM), 14 + 0.005 H + 50 per GFLOP (RNN).
// (all with the weights in shared memory: which layers run here, and so in exact products, is left as it was before those that fit
// registers took a third less time)
// T = 36, TF32: LSTM H = 300 at B = 128 / 256: 12.4 / 20.7 us a step in the cluster, 16.0 / 16.0 launched; RNN H = 800 at
// B = 32 / 128: 8.7 / 29.2 and 17.0 / 19.9.
static bool pays(const nb_handle_s *h, int gates, int H, int B, int T, bool linear, GemmPath step_path) {
    Shape s;
    if (!choose(h, gates, H, B, false, &s)) return false;
    const int waves = waves_of(h, s, B);
    const bool lstm = gates == 4, activated = lstm && !linear;
    const double in_cluster = waves * (2.0 + 0.03 * (double)s.smem / 1024 + T * (1.4 * step_cost(gates, s, H) / 1900 + (activated ? 1.2 : 0.0)));
    double step;
    if (step_path == PATH_SIMT) {
        const double gflop = 2e-9 * B * gates * H * H;
        step = lstm ? 16 + 0.02 * H + 45 * gflop : 14 + 0.005 * H + 50 * gflop;
    } else {
        const bool three = step_path == PATH_TC3;
        step = activated ? (three ? 24 : 17) : (lstm ? (three ? 17.5 : 12.5) : (three ? 20 : 15));
    }
    return in_cluster <= (activated ? T * step : (lstm ? 2 + (T - 1) * step : (T + 2) * step));
}

// On the CUDA cores, whose results do not depend on the batch otherwise, the layer and its steps decide up to 256 rows.
bool recurrent_cluster_pays(nb_handle_s *h, int gates, int H, int B, int T, bool linear, GemmPath step_path) {
    Shape s;
    if (h->cc_major != 10 || !shape_of(gates, H, 16, 1, false, &s)) return false;      // (the largest cluster holds the most)
    prepare_device(h);
    if (step_path != PATH_SIMT) return pays(h, gates, H, B, T, linear, step_path);
    return pays(h, gates, H, 32, T, linear, step_path) && (B <= 256 || pays(h, gates, H, B, T, linear, step_path));
}

void recurrent_cluster(nb_handle_s *h, const RecurrentArgs &a) {
    RecParams p;
    p.a = a;
    p.status = h->d_status;
    if (!choose(h, a.gates, a.H, a.B, in_registers(h, a), &p.s)) throw Error(NB_ERR_UNSUPPORTED, "recurrent weights do not fit a cluster");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((a.B + p.s.RB - 1) / p.s.RB) * p.s.CS));
    cfg.blockDim = dim3((unsigned)(p.s.warps ? 32 * p.s.warps : RC_THREADS));
    cfg.dynamicSmemBytes = std::max(p.s.smem, (size_t)116 * 1024);      // one CTA per SM
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)p.s.CS; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    const RecKernel k = (p.s.warps ? WARP_KERNELS : KERNELS)[a.gates == 4][p.s.RB == 1 ? 0 : (p.s.RB == 2 ? 1 : (p.s.RB == 4 ? 2 : 3))];
    ProfileScope prof(h, 1, 2.0 * (double)a.T * a.B * a.gates * a.H * a.H);
    (void)cudaLaunchKernelEx(&cfg, k, p);
    check_launch("recurrent_cluster_kernel");
    count_launch(h);
    prof.finish();
}

}  // namespace nb
