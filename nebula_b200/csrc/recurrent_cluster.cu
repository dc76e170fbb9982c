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
// CS depends on the layer only, so a batch and its slices add in the same order.
#include <cooperative_groups.h>

#include "device_math.cuh"
#include "nb_internal.h"

namespace nb {

namespace {

namespace cg = cooperative_groups;

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
    size_t smem;
};

struct RecParams {
    RecurrentArgs a;
    Shape s;
};

__device__ __forceinline__ void ffma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

template <int RB>
__global__ void __launch_bounds__(RC_THREADS, 1) recurrent_cluster_kernel(const RecParams p) {
    extern __shared__ __align__(16) float smem[];
    const RecurrentArgs &a = p.a;
    const int H = a.H, G = a.gates, Hs = p.s.Hs, rows2 = 2 * p.s.RP;
    float *w_s = smem;                              // [2 RP][Hs]
    float *h_s = w_s + rows2 * Hs;                  // [2][RB][Hs]: the state read by this step and written by it
    float *part = h_s + 2 * RB * Hs;                // [kg][2 RP][RB]
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
    if (!a.lstm) {                                  // step 0 of an RNN multiplies the input gate's output
        __syncthreads();
        for (int i = tid; i < RB * H; i += RC_THREADS) {
            const int b = i / H, k = i - b * H;
            if (b0 + b < a.B) h_s[b * Hs + k] = a.pre[(long)(b0 + b) * H + k];
        }
    }

    // the (unit, batch row) pairs this thread finishes
    int item_u[RC_ITEMS], item_b[RC_ITEMS];
    float c[RC_ITEMS], z[RC_ITEMS][4], scale[RC_ITEMS], shift[RC_ITEMS][4];
    auto fetch_pre = [&](int t, int i, float (&v)[4]) {
        const float *src = a.pre + ((long)t * a.B + b0 + item_b[i]) * G * H + (long)G * (unit0 + item_u[i]);
        if (G == 4) {
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
        for (int g = 0; g < 4; g++) { z[i][g] = 0.0f; shift[i][g] = 0.0f; }
        if (item_b[i] >= 0) {
            fetch_pre(0, i, z[i]);
            if (a.scale) scale[i] = a.scale[unit0 + item_u[i]];
#pragma unroll
            for (int g = 0; g < 4; g++)
                if (a.shift && g < G) shift[i][g] = a.shift[(long)G * (unit0 + item_u[i]) + g];
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
        float zn[RC_ITEMS][4];
#pragma unroll
        for (int i = 0; i < RC_ITEMS; i++) {
#pragma unroll
            for (int g = 0; g < 4; g++) zn[i][g] = 0.0f;
            if (item_b[i] >= 0 && t + 1 < a.T) fetch_pre(t + 1, i, zn[i]);
        }
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
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int b = 0; b < RB; b++) {
                    float v = __uint_as_float((unsigned)acc[j][b]) + __uint_as_float((unsigned)(acc[j][b] >> 32));
                    v += __shfl_xor_sync(0xffffffffu, v, 8);
                    v += __shfl_xor_sync(0xffffffffu, v, 16);
                    if (lane < 8) part[(kg * rows2 + rp + j * p.s.RP) * RB + b] = v;
                }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < RC_ITEMS; i++) {
            if (item_b[i] < 0) continue;
            const int u = item_u[i], b = item_b[i];
            float v[4];
            for (int g = 0; g < G; g++) {
                float s = 0.0f;
                for (int q = 0; q < p.s.kg; q++) s += part[(q * rows2 + G * u + g) * RB + b];
                v[g] = s;
            }
            const long o = ((long)t * a.B + b0 + b) * H + unit0 + u;
            float state;
            if (a.lstm) {
                float zg[4];
#pragma unroll
                for (int g = 0; g < 4; g++)         // linear gate layers: their shifts are in `pre` already
                    zg[g] = a.act == NB_ACT_LINEAR ? z[i][g] + v[g] : z[i][g] + apply_activation_call(v[g] + shift[i][g], a.act);
                const float2 ch = a.cell_f32 ? lstm_cell_unit_f32(zg[0], zg[1], zg[2], zg[3], c[i])
                                             : lstm_cell_unit(zg[0], zg[1], zg[2], zg[3], c[i]);
                c[i] = ch.x; state = ch.y;
                a.cell[o] = c[i];
                a.out[o] = state;
                if (a.out_round) a.out_round[o] = round_tf32(state);
            } else {
                const float x = a.scale ? fmaf(v[0], scale[i], shift[i][0]) : v[0] + shift[i][0];
                const float hv = apply_activation_fast(x, a.act);
                state = z[i][0] + hv;
                const float y = t == 0 ? hv : state;        // what the output gate reads: h_0, then the states
                a.out[o] = a.round_out ? round_tf32(y) : y;
            }
            if (t + 1 < a.T) {
                float *dst = h_s + next_off + b * Hs + unit0 + u;
                for (int q = 0; q < CS; q++) *(CS > 1 ? cluster.map_shared_rank(dst, q) : dst) = state;
            }
#pragma unroll
            for (int g = 0; g < 4; g++) z[i][g] = zn[i][g];
        }
        if (t + 1 < a.T) {
            if (CS > 1) cluster.sync();             // (the last step sends nothing: no CTA leaves before its peers' stores)
            else __syncthreads();
        }
    }
}

typedef void (*RecKernel)(const RecParams);
const RecKernel KERNELS[4] = {recurrent_cluster_kernel<1>, recurrent_cluster_kernel<2>, recurrent_cluster_kernel<4>,
                              recurrent_cluster_kernel<8>};
constexpr int MAX_SMEM = 227 * 1024;

bool shape_of(int gates, int H, int CS, int RB, Shape *s) {
    s->CS = CS; s->RB = RB;
    s->U = (H + CS - 1) / CS;
    s->RP = ((gates * s->U + 1) / 2 + 7) / 8 * 8;
    s->rg = s->RP / 8;
    if (s->rg > RC_WARPS || RB * s->U > RC_ITEMS * RC_THREADS) return false;
    s->kg = RC_WARPS / s->rg;
    s->Hs = padded_stride(H);
    s->smem = sizeof(float) * ((size_t)2 * s->RP * s->Hs + (size_t)2 * RB * s->Hs + (size_t)s->kg * 2 * s->RP * RB);
    return s->smem <= MAX_SMEM;
}

// Clock cycles of a step: every warp row-group reads its 16 weight rows and RB states (8 + RB wavefronts per K quad and
// eight rows), plus the fixed chain of a step (measured: about 1000 cycles with a cluster barrier, 500 without).
double step_cost(const Shape &s, int H) { return (double)s.rg * H / 16 * (8 + s.RB) + (s.CS > 1 ? 1000.0 : 500.0); }

// Clusters that run at once: 148 SMs in groups of 16 to 18 that a cluster cannot span.
int clusters_at_once(const nb_handle_s *h, int CS) { return CS == 16 ? h->clusters_of_16 : (h->sm_count / 18) * (18 / CS); }

// Cluster size from the layer alone (at a batch of 32); rows per cluster from the batch.
bool choose(const nb_handle_s *h, int gates, int H, int B, Shape *best) {
    auto pick = [&](int batch, int cs_lo, int cs_hi) {
        double best_cost = -1;
        for (int CS = cs_lo; CS <= cs_hi; CS *= 2) {
            const int at_once = clusters_at_once(h, CS);
            if (at_once < 1) continue;
            for (int RB = 1; RB <= 8; RB *= 2) {
                Shape s;
                if (!shape_of(gates, H, CS, RB, &s)) continue;
                const int waves = ((batch + RB - 1) / RB + at_once - 1) / at_once;
                const double cost = waves * step_cost(s, H);
                if (best_cost < 0 || cost < best_cost) { best_cost = cost; *best = s; }
            }
        }
        return best_cost >= 0;
    };
    return pick(32, 1, 16) && pick(B, best->CS, best->CS);
}

}  // namespace

void recurrent_cluster_prepare_device(nb_handle_s *h) {
    for (RecKernel k : KERNELS) {
        NB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
        NB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    // clusters of 16 are beyond the portable size: ask how many of them the device holds
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(RC_THREADS);
    cfg.dynamicSmemBytes = MAX_SMEM;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, KERNELS[0], &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    h->clusters_of_16 = n;
}

bool recurrent_cluster_supported(const nb_handle_s *h, int gates, int H, int B) {
    Shape s;
    return h->cc_major == 10 && choose(h, gates, H, B, &s);
}

void recurrent_cluster(nb_handle_s *h, const RecurrentArgs &a) {
    RecParams p;
    p.a = a;
    if (!choose(h, a.gates, a.H, a.B, &p.s)) throw Error(NB_ERR_UNSUPPORTED, "recurrent weights do not fit a cluster");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((a.B + p.s.RB - 1) / p.s.RB) * p.s.CS));
    cfg.blockDim = dim3(RC_THREADS);
    cfg.dynamicSmemBytes = std::max(p.s.smem, (size_t)116 * 1024);      // one CTA per SM
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)p.s.CS; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    const RecKernel k = KERNELS[p.s.RB == 1 ? 0 : (p.s.RB == 2 ? 1 : (p.s.RB == 4 ? 2 : 3))];
    ProfileScope prof(h, 1, 2.0 * (double)a.T * a.B * a.gates * a.H * a.H);
    (void)cudaLaunchKernelEx(&cfg, k, p);
    check_launch("recurrent_cluster_kernel");
    count_launch(h);
    prof.finish();
}

}  // namespace nb
