// Per-layer plans: weight upload/re-layout and the forward bodies that a Nebula
// layer's _forward_() would call.
#include "plans.h"

#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>

namespace nb {

void upload(nb_handle_s *h, DeviceBuffer &dst, const float *src, size_t n, int mem, size_t guard) {
    dst.alloc(n, guard);
    if (!n) return;
    NB_REQUIRE(src != nullptr, "null source pointer");
    NB_CHECK_CUDA(cudaMemcpyAsync(dst.p, src, n * sizeof(float),
                                  mem == NB_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, h->stream));
    if (mem == NB_MEM_HOST) NB_CHECK_CUDA(cudaStreamSynchronize(h->stream));   // the host buffer may go away
}
void upload_vec(nb_handle_s *h, DeviceBuffer &dst, const std::vector<float> &v, size_t guard) {
    upload(h, dst, v.data(), v.size(), NB_MEM_HOST, guard);
}
// Per-column epilogue vectors are read 32 columns at a time: pad them to a multiple of 32.
void upload_padded(nb_handle_s *h, DeviceBuffer &dst, std::vector<float> v, float fill) {
    v.resize((v.size() + 31) / 32 * 32, fill);
    upload_vec(h, dst, v);
}
std::vector<float> to_host(nb_handle_s *h, const float *src, size_t n, int mem) {
    std::vector<float> v(n);
    if (!n) return v;
    NB_REQUIRE(src != nullptr, "null source pointer");
    if (mem == NB_MEM_DEVICE) {
        NB_CHECK_CUDA(cudaMemcpyAsync(v.data(), src, n * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        NB_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    } else {
        std::memcpy(v.data(), src, n * sizeof(float));
    }
    return v;
}

void fold_bn(int n, const float *bias, const float *gamma, const float *mean, const float *var, bool has_bn,
             std::vector<float> &scale, std::vector<float> &shift) {
    scale.clear();
    shift.resize(n);
    if (!has_bn) {
        for (int i = 0; i < n; i++) shift[i] = bias[i];
        return;
    }
    scale.resize(n);
    for (int i = 0; i < n; i++) {
        const double s = (double)gamma[i] / (std::sqrt((double)var[i]) + 0.00001);
        scale[i] = (float)s;
        shift[i] = (float)((double)bias[i] - (double)mean[i] * s);
    }
}

// -------------------------------------------------------------------- conv
ConvPlan::ConvPlan(nb_handle_s *hh, const nb_conv2d_desc_t &desc) : nb_plan_s(NB_PLAN_CONV, hh), d(desc) {
    NB_REQUIRE(d.batch > 0 && d.channels > 0 && d.height > 0 && d.width > 0, "conv: non-positive input extent");
    NB_REQUIRE(d.filters > 0 && d.size > 0 && d.stride > 0 && d.padding >= 0, "conv: bad filter geometry");
    NB_REQUIRE(d.height + 2 * d.padding >= d.size && d.width + 2 * d.padding >= d.size, "conv: filter larger than padded input");
    NB_REQUIRE(d.activation > NB_ACT_UNDEFINED && d.activation < NB_ACT_COUNT, "conv: undefined activation");
    NB_REQUIRE(d.layout == NB_LAYOUT_NCHW || d.layout == NB_LAYOUT_NHWC, "conv: bad layout");
    // convolutional_layer.cc:150-151
    OH = (d.height + 2 * d.padding - d.size) / d.stride + 1;
    OW = (d.width + 2 * d.padding - d.size) / d.stride + 1;
    Cp = (d.channels + 3) / 4 * 4;
    const int K = d.channels * d.size * d.size;
    Kpad = (K + 31) / 32 * 32;
    pack_ok = (Cp != d.channels || d.channels < 32) && Kpad <= 384;    // the gather table lives in the kernel parameters
    // row windows: 4 floats per pixel, a filter row of k taps is 4k floats, rounded up to whole 32-float K blocks
    rw_inner = (4 * d.size + 31) / 32 * 32;
    rw_wp = std::max((OW - 1) * d.stride + rw_inner / 4, d.width + 2 * d.padding);
    // NEBULA_B200_ROW_WINDOWS=0 (read when the plan is created) sends these layers through the in-kernel gather instead
    const char *rw_env = std::getenv("NEBULA_B200_ROW_WINDOWS");
    tc_split = conv_tc_split(h, conv_args(nullptr, true).g, d.channels, d.filters);
    rowwin_ok = !(rw_env && *rw_env == '0') && d.channels <= 4 && rw_inner <= 256 && d.stride <= 8 && h->encode_tiled &&
                h->cc_major == 10;
}

void ConvPlan::set_weights(const float *weight, const float *bias, const float *g, const float *m, const float *v,
                           int mem) {
    NB_REQUIRE(weight && bias, "conv: null weight or bias");
    NB_REQUIRE(!d.batch_normalize || (g && m && v), "conv: batch_normalize=1 needs scale, mean and variance");
    const size_t wn = (size_t)d.filters * d.channels * d.size * d.size;
    DeviceBuffer raw;
    upload(h, raw, weight, wn, mem);
    w.exact.alloc((size_t)d.size * d.size * d.filters * Cp, weight_guard(Cp));
    w.split_ready = false;
    launch_weight_relayout(h, raw.p, w.exact.p, d.filters, d.channels, d.size, Cp);
    const bool tensor_cores = h->encode_tiled && h->cc_major == 10;
    if (tensor_cores) w.ensure_split(h);
    if (rowwin_ok) {
        wr.exact.alloc((size_t)d.size * d.filters * rw_inner, weight_guard(rw_inner));
        wr.split_ready = false;
        launch_weight_rowwin(h, raw.p, wr.exact.p, d.filters, d.channels, d.size, rw_inner);
        wr.ensure_split(h);
    }
    if (pack_ok) {
        wp.exact.alloc((size_t)d.filters * Kpad, weight_guard(Kpad));
        wp.split_ready = false;
        launch_weight_pack(h, raw.p, wp.exact.p, d.filters, d.channels, d.size, Kpad);
        if (tensor_cores) wp.ensure_split(h);
    }
    NB_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    std::vector<float> hb = to_host(h, bias, d.filters, mem), hg, hm, hv, sc, sh;
    if (d.batch_normalize) {
        hg = to_host(h, g, d.filters, mem);
        hm = to_host(h, m, d.filters, mem);
        hv = to_host(h, v, d.filters, mem);
    }
    fold_bn(d.filters, hb.data(), hg.data(), hm.data(), hv.data(), d.batch_normalize != 0, sc, sh);
    has_scale = !sc.empty();
    if (has_scale) upload_padded(h, scale, sc, 1.0f);
    upload_padded(h, shift, sh, 0.0f);
    ready = true;
}

GemmPath ConvPlan::path(const ForwardOpts &) const {
    if (h->math_mode == NB_MATH_FP32) return PATH_SIMT;
    const bool tc_ok = h->encode_tiled && h->cc_major == 10 && Cp == d.channels && d.channels >= 32 && d.stride <= 8;
    if (!tc_ok) return PATH_SIMT;
    return h->math_mode == NB_MATH_TF32X3 ? PATH_TC3 : PATH_TC;
}

bool ConvPlan::can_fuse_pool() const {
    const GemmPath pth = path(ForwardOpts());
    return (pth == PATH_TC || pth == PATH_TC3) && !(OH & 1) && !(OW & 1) && (d.filters % 4) == 0 && OH >= 2 && OW >= 2;
}

bool ConvPlan::can_fuse_shortcut(int conn_c, int conn_h, int conn_w) const {
    const GemmPath pth = path(ForwardOpts());
    // sample == 1 (the connection is not smaller than this layer's output), linear conv, aligned channel rows
    return (pth == PATH_TC || pth == PATH_TC3) && d.activation == NB_ACT_LINEAR && conn_w >= OW && conn_h >= OH &&
           (conn_c % 4) == 0 && (d.filters % 4) == 0;
}

// K over clusters, whose CTAs run the whole epilogue.  A call on a caller's NHWC tensor, which takes a pass in front, keeps the
// product and the addition of its slices as two kernels: its launch count is relied on (tests/test_gpu_split.py), at 2 to 3 us a call.
TcSplit ConvPlan::splits(const ForwardOpts &o, bool *clusters) const {
    const GemmPath pth = path(o);
    *clusters = !(o.x_nhwc && (o.x_foreign || (pth == PATH_TC && !o.x_rounded)));
    if (pth == PATH_SIMT || o.addend) return TcSplit{1, 0};
    if (o.residual && ((o.res_c % 4) != 0 || ((uintptr_t)o.residual & 15))) return TcSplit{1, 0};     // (read in quads there)
    if (!*clusters) return TcSplit{tc_split, 0};
    TcSplit &t = tc_cluster[pth == PATH_TC3][o.pool_out != nullptr][!o.y_nhwc];
    if (t.S == 0)
        t = conv_tc_cluster(h, conv_args(nullptr, true).g, d.channels, d.filters, d.activation, pth == PATH_TC3, o.pool_out != nullptr, tc_split, !o.y_nhwc);
    *clusters = t.S == 1 || t.block_n > 0;
    return t;
}

// The TMA-fed tensor-core routes write NCHW themselves where their pixel boxes suit it; the others (CUDA cores, in-kernel
// gather, K slices) go through a layout pass.
bool ConvPlan::writes_nchw(const ForwardOpts &o) {
    if (o.y_nhwc || h->math_mode == NB_MATH_FP32) return false;
    const bool simt = path(o) == PATH_SIMT, three = h->math_mode == NB_MATH_TF32X3;
    bool clusters;
    if (simt) {
        if (!rowwin_ok) return false;
    } else if (splits(o, &clusters).S > 1) {
        return clusters;                // (they have small outputs)
    }
    if (nchw_direct[three] < 0)
        nchw_direct[three] = conv_tc_writes_nchw(simt ? rowwin_args(nullptr, nullptr, false) : conv_args(nullptr, true), three);
    return nchw_direct[three] > 0;
}

// The product of this layer: x as it lies, and as row windows (without the zero columns that fill up a tensor-core K block).
GemmArgs ConvPlan::conv_args(const float *x, bool nhwc) const {
    GemmArgs a;
    a.a = x; a.a_is_conv = true;
    ConvGeom &g = a.g;
    g.batch = d.batch; g.C = d.channels; g.H = d.height; g.W = d.width; g.OH = OH; g.OW = OW;
    g.ksize = d.size; g.stride = d.stride; g.pad = d.padding;
    if (nhwc) {
        g.sc = 1; g.sw = d.channels; g.sh = (long)d.width * d.channels; g.sn = (long)d.height * d.width * d.channels;
    } else {
        g.sw = 1; g.sh = d.width; g.sc = (long)d.height * d.width; g.sn = (long)d.channels * d.height * d.width;
    }
    a.ldb = Cp; a.M = d.batch * OH * OW; a.N = d.filters; a.Kc = d.channels;
    return a;
}
GemmArgs ConvPlan::rowwin_args(const float *xw, const float *weights, bool cuda_cores) const {
    GemmArgs a;
    a.a = xw; a.b = weights; a.a_is_conv = true;
    ConvGeom &g = a.g;
    g.batch = d.batch; g.C = rw_inner; g.H = d.height; g.W = rw_wp - rw_inner / 4 + 1; g.OH = OH; g.OW = OW;
    g.ksize = d.size; g.ksize_w = 1; g.stride = d.stride; g.pad = d.padding; g.pad_w = 0;
    g.sc = 1; g.sw = 4; g.sh = (long)rw_wp * 4; g.sn = (long)d.height * rw_wp * 4;
    a.ldb = rw_inner; a.M = d.batch * OH * OW; a.N = d.filters; a.Kc = cuda_cores ? 4 * d.size : rw_inner;
    return a;
}

// Which of the three routes forward() takes, and the scratch each needs.
size_t ConvPlan::reserve(const ForwardOpts &o) {
    const GemmPath pth = path(o);
    const size_t xin = (size_t)d.batch * d.channels * d.height * d.width;
    const size_t yout = (size_t)d.batch * d.filters * OH * OW;
    const bool tc_mode = h->math_mode != NB_MATH_FP32;
    if (!o.y_nhwc) y_scratch.reserve(yout);         // (also where this route writes NCHW itself: a later math mode may not)
    if (pth == PATH_SIMT && rowwin_ok) {
        x_rowwin.reserve((size_t)d.batch * d.height * rw_wp * 4);
        if (!tc_mode) gemm_simt_load(h, rowwin_args(nullptr, nullptr, true));
        else if (h->math_mode == NB_MATH_TF32 && cheap_activation(d.activation)) gemm_tc_load(h, TC_LEAN);
    } else if (pth == PATH_SIMT && pack_ok && tc_mode && h->encode_tiled) {
        gemm_tc_load(h, TC_GATHER);     // the kernel gathers x in place
    } else if (pth == PATH_SIMT) {
        gemm_simt_load(h, conv_args(nullptr, o.x_nhwc));
    } else {
        const bool need_round = (pth == PATH_TC) && !o.x_rounded;
        if (!o.x_nhwc || need_round || o.x_foreign) x_scratch.reserve(xin);
        if (pth == PATH_TC && cheap_activation(o.residual ? o.res_act : d.activation)) gemm_tc_load(h, o.residual ? TC_LEAN | TC_RESIDUAL : TC_LEAN);
        bool clusters;
        const int S = splits(o, &clusters).S;
        if (S > 1 && !clusters) split_ws.reserve((size_t)S * yout);
    }
    return workspace_bytes();
}

void ConvPlan::forward(const float *x, float *y, const ForwardOpts &o) {
    if (!ready) throw Error(NB_ERR_NO_WEIGHTS, "conv: forward before set_weights");
    NB_REQUIRE(x && (y || o.pool_out), "conv: null tensor pointer");
    const GemmPath pth = path(o);
    const size_t xin = (size_t)d.batch * d.channels * d.height * d.width;
    reserve(o);

    if (pth == PATH_SIMT && rowwin_ok) {
        // 1-4 input channels: one K slice per filter row (fetched by TMA on the tensor-core routes; on the CUDA cores a
        // slice of 4*size aligned floats per row instead of `size` taps of 1-4 scattered ones)
        const bool three = h->math_mode == NB_MATH_TF32X3, cuda_cores = h->math_mode == NB_MATH_FP32;
        float *xw = x_rowwin.p;
        if (o.x_rowwin) xw = const_cast<float *>(x);       // the caller already holds the input in this layout
        else launch_rowwin_input(h, x, xw, d.batch, d.channels, d.height, d.width, rw_wp, d.padding, o.x_nhwc,
                                 h->math_mode == NB_MATH_TF32);
        GemmArgs ra = rowwin_args(xw, cuda_cores ? wr.exact.p : wr.hi.p, cuda_cores);
        ra.scale = has_scale ? scale.p : nullptr; ra.shift = shift.p; ra.act = d.activation;
        ra.round_out_tf32 = o.round_out; ra.addend = o.addend; ra.ld_addend = d.filters;
        float *yo = y;
        ra.y_nchw = writes_nchw(o);
        if (!o.y_nhwc) {
            NB_REQUIRE(o.addend == nullptr, "conv: addend needs NHWC output");
            if (!ra.y_nchw) yo = y_scratch.p;
        }
        ra.y = yo; ra.ldy = d.filters;
        ra.algo_flops = 2.0 * (double)ra.M * d.filters * d.channels * d.size * d.size;
        ra.b_lo = wr.lo.p; ra.b_static = true;
        if (cuda_cores) {
            gemm_simt(h, ra);
            if (!o.y_nhwc) launch_layout(h, yo, y, d.batch, d.filters, OH, OW, false, false);
            return;
        }
        if (gemm_tc_supported(h, ra)) {
            gemm_tc(h, ra, three);
            if (yo != y) launch_layout(h, yo, y, d.batch, d.filters, OH, OW, false, false);
            return;
        }
    }
    if (pth == PATH_SIMT && pack_ok && h->math_mode != NB_MATH_FP32 && h->encode_tiled) {
        // tensor-core route for small channel counts: the kernel gathers the patches itself
        const bool three = h->math_mode == NB_MATH_TF32X3;
        GemmArgs pa = conv_args(x, o.x_nhwc);
        pa.a_gather = true;
        pa.ldb = Kpad; pa.Kc = Kpad;
        pa.scale = has_scale ? scale.p : nullptr; pa.shift = shift.p; pa.act = d.activation;
        pa.round_out_tf32 = o.round_out; pa.addend = o.addend; pa.ld_addend = d.filters;
        float *yo = y;
        if (!o.y_nhwc) {
            NB_REQUIRE(o.addend == nullptr, "conv: addend needs NHWC output");
            yo = y_scratch.p;
        }
        pa.y = yo; pa.ldy = d.filters;
        pa.algo_flops = 2.0 * (double)pa.M * d.filters * d.channels * d.size * d.size;
        const bool split_now = !wp.split_ready;
        wp.ensure_split(h);
        pa.b = wp.hi.p; pa.b_lo = wp.lo.p; pa.b_static = !split_now;
        gemm_tc(h, pa, three);
        if (!o.y_nhwc) launch_layout(h, yo, y, d.batch, d.filters, OH, OW, false, false);
        return;
    }

    const float *xa = x;
    bool nhwc = o.x_nhwc;
    if (pth != PATH_SIMT) {
        const bool need_round = (pth == PATH_TC) && !o.x_rounded;
        if (!nhwc) {
            launch_layout(h, x, x_scratch.p, d.batch, d.channels, d.height, d.width, true, need_round);
            xa = x_scratch.p;
            nhwc = true;
        } else if (need_round) {
            launch_round_tf32(h, x, x_scratch.p, xin);
            xa = x_scratch.p;
        } else if (o.x_foreign) {
            NB_CHECK_CUDA(cudaMemcpyAsync(x_scratch.p, x, xin * sizeof(float), cudaMemcpyDeviceToDevice, h->stream));
            xa = x_scratch.p;
        }
    }
    GemmArgs a = conv_args(xa, nhwc);
    a.scale = has_scale ? scale.p : nullptr;
    a.shift = shift.p;
    a.act = d.activation;
    a.round_out_tf32 = o.round_out;
    a.addend = o.addend;
    a.ld_addend = d.filters;
    float *yo = y;
    a.y_nchw = writes_nchw(o);
    if (!o.y_nhwc) {
        NB_REQUIRE(o.addend == nullptr, "conv: addend needs NHWC output");
        if (!a.y_nchw) yo = y_scratch.p;
    }
    a.y = yo;
    a.ldy = d.filters;
    if (o.residual) {
        NB_REQUIRE(o.y_nhwc && pth != PATH_SIMT && !o.addend && !o.pool_out, "conv: fused shortcut needs the tensor-core path and NHWC output");
        a.addend = o.residual;
        a.ld_addend = o.res_c;
        a.res_stride = std::max(1, o.res_w / OW);       // common/utils.cc:31
        a.res_c = std::min(o.res_c, d.filters);
        a.res_h = o.res_h; a.res_w = o.res_w;
        a.act = o.res_act;
    }
    if (o.pool_out) {
        NB_REQUIRE(o.y_nhwc && pth != PATH_SIMT, "conv: fused pooling needs the tensor-core path and NHWC output");
        a.y = nullptr;
        a.y_pool = o.pool_out;
    }
    if (pth == PATH_SIMT) {
        a.b = w.exact.p;
        gemm_simt(h, a);
    } else {
        a.b_static = w.split_ready;
        w.ensure_split(h);
        a.b = w.hi.p;
        a.b_lo = w.lo.p;
        bool clusters;
        const TcSplit split = splits(o, &clusters);
        int S = split.S;
        if (!clusters && o.residual && ((uintptr_t)y & 15)) S = 1;       // (the reduction writes a folded shortcut's sums in quads)
        if (S > 1 && clusters) {
            a.split_k = S; a.split_cluster = true; a.block_n_hint = split.block_n;
            gemm_tc(h, a, pth == PATH_TC3);
        } else if (S > 1) {
            GemmArgs sa = a;
            sa.split_k = S;
            sa.scale = sa.shift = sa.addend = nullptr; sa.res_stride = 0; sa.act = NB_ACT_LINEAR; sa.round_out_tf32 = false;
            sa.y = split_ws.p; sa.y_pool = nullptr;
            sa.algo_flops = 2.0 * (double)a.M * d.filters * d.channels * d.size * d.size;
            gemm_tc(h, sa, pth == PATH_TC3);
            SplitReduce r{};
            r.ws = split_ws.p; r.S = S; r.M = a.M; r.N = d.filters; r.scale = a.scale; r.shift = a.shift; r.act = a.act;
            r.round = o.round_out; r.y = o.pool_out ? o.pool_out : yo; r.OH = OH; r.OW = OW; r.pool = o.pool_out != nullptr;
            if (o.residual) {
                r.res = a.addend; r.res_ld = a.ld_addend; r.res_stride = a.res_stride;
                r.res_c = a.res_c; r.res_h = a.res_h; r.res_w = a.res_w;
            }
            launch_splitk_reduce(h, r);
        } else {
            gemm_tc(h, a, pth == PATH_TC3);
        }
    }
    if (!o.y_nhwc && yo != y) launch_layout(h, yo, y, d.batch, d.filters, OH, OW, false, false);
}

// ---------------------------------------------------------------------- fc
FcPlan::FcPlan(nb_handle_s *hh, const nb_fc_desc_t &desc) : nb_plan_s(NB_PLAN_FC, hh), d(desc) {
    NB_REQUIRE(d.batch > 0 && d.inputs > 0 && d.outputs > 0, "connected: non-positive extent");
    NB_REQUIRE(d.activation > NB_ACT_UNDEFINED && d.activation < NB_ACT_COUNT, "connected: undefined activation");
}

void FcPlan::set_weights(const float *weight, const float *bias, const float *g, const float *m, const float *v,
                         int mem) {
    NB_REQUIRE(weight && bias, "connected: null weight or bias");
    NB_REQUIRE(!d.batch_normalize || (g && m && v), "connected: batch_normalize=1 needs scale, mean and variance");
    const size_t wn = (size_t)d.outputs * d.inputs;
    w.split_ready = false;
    if (perm_c > 0 && perm_h * perm_w > 1) {
        NB_REQUIRE((size_t)perm_c * perm_h * perm_w == (size_t)d.inputs, "connected: permutation does not match inputs");
        DeviceBuffer raw;
        upload(h, raw, weight, wn, mem);
        w.exact.alloc(wn, weight_guard(d.inputs));
        launch_fc_permute(h, raw.p, w.exact.p, d.outputs, perm_c, perm_h, perm_w);
        NB_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    } else {
        upload(h, w.exact, weight, wn, mem, weight_guard(d.inputs));
    }
    if (h->encode_tiled && h->cc_major == 10 && (d.inputs % 4) == 0 && d.inputs >= 32) w.ensure_split(h);
    std::vector<float> hb = to_host(h, bias, d.outputs, mem), hg, hm, hv, sc, sh;
    if (d.batch_normalize) {
        hg = to_host(h, g, d.outputs, mem);
        hm = to_host(h, m, d.outputs, mem);
        hv = to_host(h, v, d.outputs, mem);
    }
    fold_bn(d.outputs, hb.data(), hg.data(), hm.data(), hv.data(), d.batch_normalize != 0, sc, sh);
    has_scale = !sc.empty();
    if (has_scale) upload_padded(h, scale, sc, 1.0f);
    upload_padded(h, shift, sh, 0.0f);
    ready = true;
}

GemmPath FcPlan::path() const {
    if (h->math_mode == NB_MATH_FP32) return PATH_SIMT;
    const bool tc_ok = h->encode_tiled && h->cc_major == 10 && (d.inputs % 4) == 0 && d.inputs >= 32;
    if (!tc_ok) return PATH_SIMT;
    return h->math_mode == NB_MATH_TF32X3 ? PATH_TC3 : PATH_TC;
}

// Few rows and a long contraction (weight streaming): split K so that every SM pulls weights.  Wide tiles keep the most weight
// bytes in flight per SM; the split count then fills the SMs, and of the tile widths the one that leaves the fewest SMs idle in
// the last wave wins.  In TF32 from 2048 columns on all of that depends on K, N and the SM count only: a batch and its slices
// add in the same order.  The rest depends on the rows as well, so that slices of a batch may differ from it in the last bits:
// 3xTF32, whose slices cost more to add than they gain once the 128 x 128 tiles of the batch fill a quarter of the SMs, half of
// them from 8192 columns on (2048 -> 1000 at 512 / 2048 rows: 33 / 90 us split, 36 / 48 us whole; 9216 -> 4096 at 256 / 512:
// 142 / 234 and 159 / 200); and shorter contractions, split only for a single row of tiles that leaves three quarters of the SMs
// idle (DBN at 32 images, 2000 -> 1000: 16 tiles of 63 K blocks took 36 us).
void FcPlan::split_choice(GemmPath pth, bool has_addend, int rows, int *S_out, int *block_n_out) const {
    int S = 1, block_n = 0;
    const int kblocks = (d.inputs + 31) / 32;
    const long tiles128 = (rows + 127L) / 128 * ((d.outputs + 127) / 128);
    if (pth == PATH_SIMT || has_addend || (d.outputs % 4) != 0) {
    } else if (pth == PATH_TC3 && d.inputs >= 2048 && 4 * tiles128 > h->sm_count * (d.inputs >= 8192 ? 2L : 1L)) {
    } else if (d.inputs >= 2048) {
        double best = 0.0;
        for (int bn = pth == PATH_TC3 ? 128 : 256; bn >= 64; bn /= 2) {
            const int nt = (d.outputs + bn - 1) / bn;
            int s = std::max(1, std::min({32, h->sm_count / nt, kblocks / 8}));
            const int per = (kblocks + s - 1) / s;
            s = (kblocks + per - 1) / per;
            const long tiles = (long)nt * s;
            const double fill = (double)tiles / (double)(((tiles + h->sm_count - 1) / h->sm_count) * h->sm_count);
            if (fill > best + 0.05) { best = fill; S = s; block_n = bn; }
        }
        if (S == 1) block_n = 0;
    } else if (rows <= 128 && kblocks >= 16) {
        const int nt = (d.outputs + 63) / 64;
        if (4 * nt <= h->sm_count) {
            S = std::min({8, h->sm_count / nt, kblocks / 4});
            const int per = (kblocks + S - 1) / S;
            S = (kblocks + per - 1) / per;
            block_n = 64;
        }
    }
    *S_out = S; *block_n_out = block_n;
}

// The same over clusters, which run the whole epilogue.  Clusters do not fill the SMs (132 CTAs of fours, 120 of eights, 112 of
// sixteens of 148), so weights that take long to stream go to slabs on all of them, and so do few columns of long K (tc_slab_cost);
// the others take the size with the shortest run, as convolutions do (conv_tc_cluster).  Any number of outputs: the rows of a
// ragged one are stored value by value (32 x 500 -> 30, logistic: 17.4 us whole, 6.2 here).
// In TF32 below 512 and from 2048 inputs on, the layer and the device alone decide in which slices a layer of clusters adds (below 512,
// where many rows are as usual as few, the size that suits one, two and four rows of tiles); of more tiles than are resident at once the
// same slices are slabs, or partial sums of whole tiles (442 x 5916 -> 408: as clusters one behind the other 54.3 us, as slabs 25;
// 1362 x 7408 -> 120 59 and 31).  Between them, and in 3xTF32, the rows count.
// (3xTF32 on a caller's tensor keeps the product and the addition of its slices as two kernels: its launch count is relied on,
// tests/test_gpu_ranges.py)
FcPlan::Split FcPlan::splits(GemmPath pth, const ForwardOpts &o, int rows) const {
    Split slabs{1, 0, 0, false};
    split_choice(pth, o.addend != nullptr, rows, &slabs.S, &slabs.block_n);
    const bool three = pth == PATH_TC3;
    if (pth == PATH_SIMT || o.addend || (three && (o.x_foreign || (slabs.S == 1 && d.inputs >= 2048)))) return slabs;
    if ((size_t)d.inputs * d.outputs > ((size_t)6 << 20)) return slabs;
    const int kblocks = (d.inputs + 31) / 32, N = d.outputs;
    const bool by_layer = !three && (d.inputs < 512 || d.inputs >= 2048);
    const long row_tiles = (rows + 127L) / 128, m_tiles = by_layer ? 1 : row_tiles;
    if (2 * m_tiles * ((N + 63) / 64) > h->sm_count) return slabs;
    auto cluster_cost = [&](long m, int S) { return tc_cluster_cost(h, m, N, kblocks, S, 64, three, d.activation); };
    auto cost_of = [&](int S) {
        double cost = cluster_cost(m_tiles, S);
        if (!by_layer || d.inputs >= 2048 || cost < 0) return cost;
        cost *= 2;
        for (int m = 2; m <= 4; m += 2) {
            const double whole = cluster_cost(m, 1), cut = S > 1 ? cluster_cost(m, S) : whole;
            cost += cut >= 0 ? std::min(cut, whole) : whole;
        }
        return cost;
    };
    Split best{1, 0, 0, false};
    double best_cost = cost_of(1);
    for (int S = 2; S <= TC_MAX_CLUSTER; S++) {
        const double cost = cost_of(S);
        if (cost >= 0 && cost < best_cost) { best_cost = cost; best = Split{S, 64, 0, true}; }
    }
    if (best.S == 1) return slabs;
    if (slabs.S > 1 && tc_slab_cost(h, m_tiles, by_layer ? 64 : rows, N, kblocks, slabs.S, slabs.block_n, three) < cluster_cost(m_tiles, best.S)) return slabs;
    if (!by_layer || row_tiles == 1) return best;

    const int per = tc_blocks_per_split(kblocks, kblocks, best.S, 64);
    best_cost = cluster_cost(row_tiles, best.S);
    Split run = best;
    for (int w = 64; w <= (N > 64 ? 128 : 64); w *= 2) {
        // (slices of 256 K blocks and more are partial sums themselves)
        const double whole = tc_cluster_cost(h, row_tiles, N, kblocks, 1, w, false, d.activation);
        if (per < 256 && (best_cost < 0 || whole < best_cost)) { best_cost = whole; run = Split{1, w, per, false}; }
        const double cut = tc_slab_cost(h, row_tiles, rows, N, kblocks, best.S, w, false);
        if ((N % 4) == 0 && (best_cost < 0 || cut < best_cost)) { best_cost = cut; run = Split{best.S, w, 0, false}; }
    }
    return run;
}

size_t FcPlan::reserve(const ForwardOpts &o, int rows) {
    const int M = rows > 0 ? rows : d.batch;
    const GemmPath pth = path();
    if ((pth == PATH_TC && !o.x_rounded) || (pth == PATH_TC3 && o.x_foreign)) x_scratch.reserve((size_t)M * d.inputs);
    if (pth == PATH_SIMT) {
        GemmArgs a;
        a.lda = a.ldb = a.Kc = d.inputs; a.M = M; a.N = d.outputs;
        gemm_simt_load(h, a);
    }
    if (pth == PATH_TC && cheap_activation(d.activation)) gemm_tc_load(h, TC_LEAN);
    const Split split = splits(pth, o, M);
    if (split.S > 1 && !split.cluster) split_ws.reserve((size_t)split.S * M * d.outputs);
    return workspace_bytes();
}

void FcPlan::forward(const float *x, float *y, const ForwardOpts &o, int rows) {
    if (!ready) throw Error(NB_ERR_NO_WEIGHTS, "connected: forward before set_weights");
    NB_REQUIRE(x && y, "connected: null tensor pointer");
    const int M = rows > 0 ? rows : d.batch;
    GemmPath pth = path();
    reserve(o, rows);
    if (pth != PATH_SIMT && (((uintptr_t)x) & 15)) pth = PATH_SIMT;
    GemmArgs a;
    const float *xa = x;
    if (pth == PATH_TC && !o.x_rounded) {
        launch_round_tf32(h, x, x_scratch.p, (size_t)M * d.inputs);
        xa = x_scratch.p;
    } else if (pth == PATH_TC3 && o.x_foreign) {
        NB_CHECK_CUDA(cudaMemcpyAsync(x_scratch.p, x, (size_t)M * d.inputs * sizeof(float), cudaMemcpyDeviceToDevice, h->stream));
        xa = x_scratch.p;
    }
    a.a = xa; a.lda = d.inputs;
    a.ldb = d.inputs;
    a.M = M; a.N = d.outputs; a.Kc = d.inputs;
    a.scale = has_scale ? scale.p : nullptr;
    a.shift = shift.p;
    a.act = d.activation;
    a.round_out_tf32 = o.round_out;
    a.addend = o.addend; a.ld_addend = d.outputs; a.addend_after_act = o.addend != nullptr && o.addend_post;
    a.y = y; a.ldy = d.outputs;
    if (pth == PATH_SIMT) {
        a.b = w.exact.p;
        gemm_simt(h, a);
        return;
    }
    a.b_static = w.split_ready;
    w.ensure_split(h);
    a.b = w.hi.p; a.b_lo = w.lo.p;
    const Split split = splits(pth, o, M);
    const int S = split.S;
    a.k_part = split.k_part; a.block_n_hint = split.block_n;
    if (S > 1 && split.cluster) {
        a.split_k = S; a.split_cluster = true;
        gemm_tc(h, a, pth == PATH_TC3);
    } else if (S > 1) {
        GemmArgs sa = a;
        sa.split_k = S;
        sa.scale = nullptr; sa.shift = nullptr; sa.act = NB_ACT_LINEAR; sa.round_out_tf32 = false;
        sa.y = split_ws.p; sa.ldy = d.outputs;
        sa.algo_flops = 2.0 * (double)M * d.outputs * d.inputs;
        gemm_tc(h, sa, pth == PATH_TC3);
        SplitReduce r{};
        r.ws = split_ws.p; r.S = S; r.M = M; r.N = d.outputs; r.scale = a.scale; r.shift = a.shift; r.act = d.activation;
        r.round = o.round_out; r.y = y;
        launch_splitk_reduce(h, r);
    } else {
        gemm_tc(h, a, pth == PATH_TC3);
    }
}

// -------------------------------------------------------------------- lstm
LstmPlan::LstmPlan(nb_handle_s *hh, const nb_lstm_desc_t &desc) : nb_plan_s(NB_PLAN_LSTM, hh), d(desc) {
    NB_REQUIRE(d.time_steps > 0 && d.batch > 0 && d.inputs > 0 && d.hidden > 0, "lstm: non-positive extent");
    NB_REQUIRE(d.activation > NB_ACT_UNDEFINED && d.activation < NB_ACT_COUNT, "lstm: undefined activation");
}

size_t LstmPlan::weight_count() const {
    size_t n = 0;
    for (int gidx = 0; gidx < 8; gidx++) {
        const size_t gin = gidx < 4 ? d.hidden : d.inputs;
        n += (size_t)d.hidden + (size_t)d.hidden * gin + (d.batch_normalize ? 3 * (size_t)d.hidden : 0);
    }
    return n;
}

void LstmPlan::set_weights(const float *stream, size_t count, int mem) {
    if (count != weight_count())
        throw Error(NB_ERR_WEIGHTS, "lstm: weight stream has " + std::to_string(count) + " floats, layer needs " +
                                        std::to_string(weight_count()));
    std::vector<float> hs = to_host(h, stream, count, mem);
    const int H = d.hidden, in = d.inputs;
    struct Blob { const float *bias, *w, *g, *m, *v; };
    Blob blob[8];
    size_t pos = 0;
    for (int gidx = 0; gidx < 8; gidx++) {     // file order iW,fW,oW,cW,iU,fU,oU,cU (lstm_layer.cc:194-206)
        const size_t gin = gidx < 4 ? H : in;
        blob[gidx].bias = hs.data() + pos; pos += H;
        blob[gidx].w = hs.data() + pos; pos += (size_t)H * gin;
        blob[gidx].g = blob[gidx].m = blob[gidx].v = nullptr;
        if (d.batch_normalize) {
            blob[gidx].g = hs.data() + pos; pos += H;
            blob[gidx].m = hs.data() + pos; pos += H;
            blob[gidx].v = hs.data() + pos; pos += H;
        }
    }
    // gate rows in the order i, f, g(cell), o; file indices of those gates:
    const int file_of_gate[4] = {0, 1, 3, 2};
    const bool linear = d.activation == NB_ACT_LINEAR;
    std::vector<float> u((size_t)4 * H * in), wr((size_t)4 * H * H), sh_u((size_t)4 * H, 0.0f), sh_w((size_t)4 * H, 0.0f);
    for (int gate = 0; gate < 4; gate++) {
        for (int side = 0; side < 2; side++) {      // 0: W (recurrent), 1: U (input)
            const Blob &b = blob[file_of_gate[gate] + (side ? 4 : 0)];
            const size_t gin = side ? in : H;
            std::vector<float> sc, s1;
            fold_bn(H, b.bias, b.g, b.m, b.v, d.batch_normalize != 0, sc, s1);
            // output row of hidden unit r, gate `gate`: 4*r + gate (a thread of the GEMM epilogue then holds all
            // four gates of a unit in neighbouring columns); a batch-norm scale is folded into the weight row
            float *dst = side ? u.data() : wr.data();
            for (int r = 0; r < H; r++) {
                const float s = sc.empty() ? 1.0f : sc[r];
                const size_t row = (size_t)4 * r + gate;
                for (size_t c = 0; c < gin; c++) dst[row * gin + c] = b.w[(size_t)r * gin + c] * s;
                // linear gate layers: both sides' shifts are one vector, applied once by the input-side GEMM
                ((side || linear) ? sh_u : sh_w)[row] += s1[r];
            }
        }
    }
    upload_vec(h, wu.exact, u, weight_guard(in));
    upload_vec(h, ww.exact, wr, weight_guard(H));
    wu.split_ready = ww.split_ready = false;
    if (h->encode_tiled && h->cc_major == 10) {
        if ((in % 4) == 0 && in >= 32) wu.ensure_split(h);
        if ((H % 4) == 0 && H >= 32) ww.ensure_split(h);
    }
    upload_padded(h, shift, sh_u, 0.0f);
    upload_padded(h, shift_w, sh_w, 0.0f);
    NB_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    ready = true;
}

// The modes that promise fp32 agreement, widths off 32 and gate layers with an activation run all steps in one kernel of exact
// fp32 products where that is the faster way.  Linear layers of widths that are multiples of 32 take TF32 products at every batch,
// whatever the cluster would cost (lstm_persistent.cu, a launch per step beyond its batches, which adds in the same order); a single
// step of linear gate layers has no product.  NEBULA_B200_LSTM_PERSISTENT=0: a launch per step in every case.
bool LstmPlan::one_kernel() const {
    const char *env = std::getenv("NEBULA_B200_LSTM_PERSISTENT");
    if (env && *env == '0') return false;
    const int H = d.hidden;
    const bool linear = d.activation == NB_ACT_LINEAR, three = h->math_mode == NB_MATH_TF32X3;
    const bool tc_w = h->math_mode != NB_MATH_FP32 && h->encode_tiled && h->cc_major == 10 && (H % 4) == 0 && H >= 32;
    if ((tc_w && !three && linear && (H % 32) == 0) || (d.time_steps == 1 && linear)) return false;
    return recurrent_cluster_pays(h, 4, H, d.batch, d.time_steps, linear, !tc_w ? PATH_SIMT : (three ? PATH_TC3 : PATH_TC));
}

size_t LstmPlan::reserve(bool own_cell, bool x_rounded, bool have_out_round, bool x_foreign) {
    const int T = d.time_steps, B = d.batch, H = d.hidden, in = d.inputs;
    const size_t rows = (size_t)T * B;
    const bool tcm = h->math_mode != NB_MATH_FP32 && h->encode_tiled && h->cc_major == 10;
    const bool tc_u = tcm && (in % 4) == 0 && in >= 32;
    const bool tc_w = tcm && (H % 4) == 0 && H >= 32;
    const bool three = h->math_mode == NB_MATH_TF32X3;
    if (tc_u && !three && d.activation == NB_ACT_LINEAR) gemm_tc_load(h, TC_LEAN);
    if (tc_w && !three && d.activation == NB_ACT_LINEAR) {      // (loads the kernels)
        (void)lstm_in_slices(h, H);
        if (!lstm_persistent_supported(h, T, B, H)) (void)lstm_wide_supported(h, T, B, H);
    }
    pre.reserve(rows * 4 * H);
    if (!tc_w) z.reserve((size_t)B * 4 * H);
    GemmArgs a;
    a.N = 4 * H;
    if (!tc_u) {
        a.lda = a.ldb = a.Kc = in; a.M = (int)rows;
        gemm_simt_load(h, a);
    }
    if (!one_kernel() && !tc_w) {
        a.lda = a.ldb = a.Kc = H; a.M = B;
        gemm_simt_load(h, a);
    }
    if (own_cell) cell_own.reserve(rows * H);
    if (!have_out_round && tc_w && !three) h_round.reserve(rows * H);
    if (tc_u && ((!three && !x_rounded) || (three && x_foreign))) x_round.reserve(rows * in);
    if (d.activation != NB_ACT_LINEAR && h_zero.reserve((size_t)B * H))
        NB_CHECK_CUDA(cudaMemsetAsync(h_zero.p, 0, (size_t)B * H * sizeof(float), h->stream));
    return workspace_bytes();
}

void LstmPlan::forward(const float *x, float *out, float *cell, bool x_rounded, float *out_round, bool x_foreign) {
    if (!ready) throw Error(NB_ERR_NO_WEIGHTS, "lstm: forward before set_weights");
    NB_REQUIRE(x && out, "lstm: null tensor pointer");
    const int T = d.time_steps, B = d.batch, H = d.hidden, in = d.inputs;
    const size_t rows = (size_t)T * B;
    const bool tcm = h->math_mode != NB_MATH_FP32 && h->encode_tiled && h->cc_major == 10;
    const bool tc_u = tcm && (in % 4) == 0 && in >= 32 && !(((uintptr_t)x) & 15);
    const bool tc_w = tcm && (H % 4) == 0 && H >= 32;
    const bool three = h->math_mode == NB_MATH_TF32X3;
    const bool linear = d.activation == NB_ACT_LINEAR;
    reserve(cell == nullptr, x_rounded, out_round != nullptr, x_foreign);
    if (!cell) cell = cell_own.p;
    float *hr = out_round;
    if (!hr && tc_w && !three) hr = h_round.p;
    // 1. input-side gate layers of every time step in one GEMM: pre = act(X * U^T + bU) (linear: + bW as well)
    {
        const float *xa = x;
        if (tc_u && !three && !x_rounded) {
            launch_round_tf32(h, x, x_round.p, rows * in);
            xa = x_round.p;
        } else if (tc_u && three && x_foreign) {
            NB_CHECK_CUDA(cudaMemcpyAsync(x_round.p, x, rows * in * sizeof(float), cudaMemcpyDeviceToDevice, h->stream));
            xa = x_round.p;
        }
        GemmArgs a;
        a.a = xa; a.lda = in; a.ldb = in; a.M = (int)rows; a.N = 4 * H; a.Kc = in;
        a.shift = shift.p; a.act = d.activation; a.y = pre.p; a.ldy = 4 * H;
        if (tc_u) {
            a.b_static = wu.split_ready;
            wu.ensure_split(h);
            a.b = wu.hi.p; a.b_lo = wu.lo.p;
            gemm_tc(h, a, three);
        } else {
            a.b = wu.exact.p;
            gemm_simt(h, a);
        }
    }
    // 2. the recurrence: z_t = pre_t + act(h_{t-1} * W^T + bW), then the cell update.  With linear gate layers
    //    step 0 has nothing to multiply (h_{-1} = 0 and bW is already in pre); otherwise act(bW) is not zero and
    //    step 0 runs the recurrent layer on a zero state like every other step.
    // All steps in one kernel where the layer has one: exact fp32 on a cluster, or, with linear gate layers on the TF32
    // tensor-core path, one cooperative kernel that keeps the recurrent weights in tensor memory (lstm_persistent.cu).
    if (one_kernel()) {
        RecurrentArgs r{};
        r.w = ww.exact.p; r.pre = pre.p; r.shift = linear ? nullptr : shift_w.p;
        r.cell = cell; r.out = out; r.out_round = hr;
        r.T = T; r.B = B; r.H = H; r.gates = 4; r.act = d.activation;
        r.cell_f32 = tc_w && !three;
        r.by_layer = !tc_w && B <= 256;
        recurrent_cluster(h, r);
        return;
    }
    const char *lp_env = std::getenv("NEBULA_B200_LSTM_PERSISTENT");
    const bool tf32_steps = tc_w && !three && linear && hr && !(lp_env && *lp_env == '0');
    if (tf32_steps && lstm_persistent_supported(h, T, B, H)) {
        ww.ensure_split(h);
        lstm_persistent(h, ww.hi.p, pre.p, cell, out, hr, T, B, H);
        return;
    }
    // (it stores quads)
    if (tf32_steps && !(((uintptr_t)out | (uintptr_t)cell) & 15) && lstm_wide_supported(h, T, B, H)) {
        launch_lstm_cell(h, pre.p, nullptr, cell, out, hr, B, H);
        ww.ensure_split(h);
        lstm_wide(h, ww.hi.p, pre.p, cell, out, hr, T, B, H, lstm_in_slices(h, H) ? lstm_k_part(H) : H / 32, 1);
        return;
    }
    for (int t = 0; t < T; t++) {
        const float *zt = pre.p + (size_t)t * B * 4 * H;
        float *ct = cell + (size_t)t * B * H, *ht = out + (size_t)t * B * H, *hrt = hr ? hr + (size_t)t * B * H : nullptr;
        const float *c_prev = t ? cell + (size_t)(t - 1) * B * H : nullptr;
        if (t > 0 || !linear) {
            GemmArgs a;
            const float *hprev = t == 0 ? h_zero.p
                                        : ((tc_w && !three) ? hr + (size_t)(t - 1) * B * H : out + (size_t)(t - 1) * B * H);
            a.a = hprev; a.lda = H; a.ldb = H; a.M = B; a.N = 4 * H; a.Kc = H;
            a.addend = zt; a.ld_addend = 4 * H; a.act = d.activation;
            if (!linear) { a.shift = shift_w.p; a.addend_after_act = true; }
            if (tc_w) {
                // the cell update runs in the GEMM epilogue: one launch per time step
                a.b_static = ww.split_ready;
                ww.ensure_split(h);
                a.b = ww.hi.p; a.b_lo = ww.lo.p;
                if (linear && !three && lstm_in_slices(h, H)) a.k_part = lstm_k_part(H);      // as the one-kernel recurrence adds
                a.lstm_H = H; a.lstm_c_prev = c_prev; a.lstm_c = ct; a.lstm_h = ht; a.lstm_h_round = hrt;
                gemm_tc(h, a, three);
                continue;
            }
            a.y = z.p; a.ldy = 4 * H;
            a.b = ww.exact.p;
            gemm_simt(h, a);
            zt = z.p;
        }
        launch_lstm_cell(h, zt, c_prev, ct, ht, hrt, B, H);
    }
}

// --------------------------------------------------------------------- rnn
RnnPlan::RnnPlan(nb_handle_s *hh, const nb_rnn_desc_t &desc) : nb_plan_s(NB_PLAN_RNN, hh), d(desc) {
    NB_REQUIRE(d.time_steps > 0 && d.batch > 0 && d.inputs > 0 && d.hidden > 0, "rnn: non-positive extent");
    NB_REQUIRE(d.activation > NB_ACT_UNDEFINED && d.activation < NB_ACT_COUNT, "rnn: undefined activation");
    // the three gates are connected layers built from the same section (rnn_layer.cc:47-54)
    nb_fc_desc_t g{};
    g.batch = d.batch; g.outputs = d.hidden; g.batch_normalize = d.batch_normalize; g.activation = d.activation;
    g.inputs = d.inputs;
    in_gate.reset(new FcPlan(h, g));
    g.inputs = d.hidden;
    hid_gate.reset(new FcPlan(h, g));
    out_gate.reset(new FcPlan(h, g));
}

size_t RnnPlan::weight_count() const {
    const size_t H = d.hidden, bn = d.batch_normalize ? 3 * H : 0;
    return (H + H * d.inputs + bn) + 2 * (H + H * H + bn);
}

void RnnPlan::set_weights(const float *stream, size_t count, int mem) {
    if (count != weight_count())
        throw Error(NB_ERR_WEIGHTS, "rnn: weight stream has " + std::to_string(count) + " floats, layer needs " +
                                        std::to_string(weight_count()));
    // blobs in the order input gate, hidden gate, output gate (rnn_layer.cc:69-73), each a connected-layer blob
    const size_t H = d.hidden;
    size_t pos = 0;
    FcPlan *gates[3] = {in_gate.get(), hid_gate.get(), out_gate.get()};
    for (FcPlan *g : gates) {
        const float *p = stream + pos;
        const size_t wn = H * g->d.inputs;
        g->set_weights(p + H, p, d.batch_normalize ? p + H + wn : nullptr, d.batch_normalize ? p + 2 * H + wn : nullptr,
                       d.batch_normalize ? p + 3 * H + wn : nullptr, mem);
        pos += H + wn + (d.batch_normalize ? 3 * H : 0);
    }
    ready = true;
}

bool RnnPlan::one_kernel() const {
    return recurrent_cluster_pays(h, 1, d.hidden, d.batch, d.time_steps, true, hid_gate->path());
}

size_t RnnPlan::reserve(bool x_rounded, bool x_foreign) {
    const size_t T = d.time_steps, B = d.batch, H = d.hidden;
    a_all.reserve(T * B * H);
    state.reserve(T * B * H);
    const bool tf32 = h->math_mode == NB_MATH_TF32;
    ForwardOpts o;
    o.x_rounded = x_rounded; o.x_foreign = x_foreign;
    in_gate->reserve(o, (int)(T * B));
    o.x_rounded = tf32; o.x_foreign = false;
    if (one_kernel()) {
        out_gate->reserve(o, (int)(T * B));
    } else {                                            // a launch per step; the output gate runs step 0 by itself
        h0.reserve(B * H);
        out_gate->reserve(o, (int)B);
        if (T > 1) out_gate->reserve(o, (int)((T - 1) * B));
        o.x_rounded = false;
        hid_gate->reserve(o, (int)B);                   // step 0 reads the (unrounded) input-gate output
    }
    return workspace_bytes();
}

void RnnPlan::forward(const float *x, float *out, bool x_rounded, bool round_out, bool x_foreign) {
    if (!ready) throw Error(NB_ERR_NO_WEIGHTS, "rnn: forward before set_weights");
    NB_REQUIRE(x && out, "rnn: null tensor pointer");
    const int T = d.time_steps, B = d.batch;
    const size_t BH = (size_t)B * d.hidden;
    const bool tf32 = h->math_mode == NB_MATH_TF32;     // stored states are then TF32 values, ready to be operands
    reserve(x_rounded, x_foreign);
    ForwardOpts o;
    // a_t for every step at once: the input gate does not depend on the state
    o.x_rounded = x_rounded; o.x_foreign = x_foreign;
    in_gate->forward(x, a_all.p, o, T * B);
    // all steps in one kernel where that is the faster way: its state buffer holds what the output gate reads, h_0 in the
    // place of s_0
    if (one_kernel()) {
        RecurrentArgs r{};
        r.w = hid_gate->w.exact.p; r.pre = a_all.p;
        r.scale = hid_gate->has_scale ? hid_gate->scale.p : nullptr; r.shift = hid_gate->shift.p;
        r.out = state.p;
        r.T = T; r.B = B; r.H = d.hidden; r.gates = 1; r.act = d.activation;
        const bool out_tc = out_gate->path() == PATH_TC;
        r.round_out = out_tc;
        r.by_layer = hid_gate->path() == PATH_SIMT && B <= 256;
        recurrent_cluster(h, r);
        ForwardOpts q;
        q.x_rounded = out_tc; q.round_out = round_out;
        out_gate->forward(state.p, out, q, T * B);
        return;
    }
    // step 0: the hidden gate reads the input gate's output, the output gate reads the hidden gate's
    o = ForwardOpts();
    o.round_out = tf32;
    hid_gate->forward(a_all.p, h0.p, o, B);
    o.addend = a_all.p; o.addend_post = true;
    hid_gate->forward(a_all.p, state.p, o, B);          // s_0 = a_0 + h_0 (same product, then the sum)
    // steps 1..T-1: h_t = hid(s_{t-1}), s_t = a_t + h_t
    for (int t = 1; t < T; t++) {
        ForwardOpts s;
        s.x_rounded = tf32; s.round_out = tf32;
        s.addend = a_all.p + t * BH; s.addend_post = true;
        hid_gate->forward(state.p + (t - 1) * BH, state.p + t * BH, s, B);
    }
    // outputs: step 0 from h_0, the others from their states in one product
    ForwardOpts q;
    q.x_rounded = tf32; q.round_out = round_out;
    out_gate->forward(h0.p, out, q, B);
    if (T > 1) out_gate->forward(state.p + BH, out + BH, q, (T - 1) * B);
}

}  // namespace nb
