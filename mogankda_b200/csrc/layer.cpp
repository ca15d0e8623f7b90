// Launches of one layer call: gate + cumsum (+ beta) -> L2 statistics and WY preparation -> state pass and output, and the backward
// pass.  Every intermediate is a torch allocation on the current stream.
#include "layer.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAStream.h>

#include <limits>

namespace mkda_host {

int dtype_code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return MKDA_F32;
        case at::kBFloat16: return MKDA_BF16;
        case at::kHalf: return MKDA_F16;
        default: break;
    }
    TORCH_CHECK_TYPE(false, "unsupported dtype ", t.scalar_type(), "; expected float32, bfloat16 or float16");
    return -1;
}

Tensor aligned(const Tensor& t, uintptr_t to) {
    if (!t.defined()) return t;
    Tensor c = t.is_contiguous() ? t : t.contiguous();
    return reinterpret_cast<uintptr_t>(c.data_ptr()) % to ? c.clone() : c;
}

Tensor new_cuda(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
    return Tensor(at::detail::empty_cuda(sizes, dt, dev, std::nullopt));
}

namespace {

Tensor aligned_f32(const Tensor& t) {
    if (!t.defined()) return t;
    return aligned(t.scalar_type() == at::kFloat ? t : t.to(at::kFloat));
}
float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
void check_rc(int rc, const char* what) {
    if (rc != MKDA_OK) throw LibraryError(std::string(what) + " failed (" + std::to_string(rc) + "): " + mkda_last_error());
}

// (row stride, column stride) in elements if `t` [..., 128] can be addressed as rows x 128 with one stride per axis (contiguous
// tensors, and broadcast views such as the gradient autograd produces for o.sum()); false otherwise
bool rows_strides(const Tensor& t, int64_t& row, int64_t& col) {
    int64_t span = -1;
    row = -1;
    for (int64_t d = t.dim() - 2; d >= 0; --d) {          // collapse the leading dims from the inside out
        if (t.size(d) == 1) continue;
        const int64_t sd = t.stride(d);
        if (row < 0) row = sd;
        else if (sd != span) return false;
        span = sd * t.size(d);
    }
    if (row < 0) row = 0;
    col = t.stride(-1);
    const int64_t most = std::numeric_limits<int>::max();
    return !(col == 1 && row % 8) && row <= most && col <= most && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// Few (chunk, q/k head) groups: handing a CTA a whole group of v-heads leaves others idle, and the extra tiles the finishing kernel then
// has to add stay in L2.  Worth it only while the grid is a couple of waves.
bool spread_v_heads(const Call& c) {
    const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount, G = c.HV / c.HK;
    const int64_t groups = (int64_t)c.NC * c.HK;
    return groups <= 2 * sms && (groups * G + sms - 1) / sms < G * ((groups + sms - 1) / sms);
}

// The gate in intra_fwd where that has at most one item per SM: a kernel and its cold start less (77 tokens x 16 heads 28.5 -> 26.1 us, 5.1 + 13.2 us of
// kernels -> 15.9).  With more items its work is not free, neither in intra_fwd's own warps nor in warps beside them, an item ahead: 3.5 items per SM 54 us against
// 40 + 8, 24 items 258 against 189 + 38.
bool gate_in_intra(const Call& c) { return (int64_t)c.NC * c.HV <= at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }

// Output in the kernel of the state chain, or in one of its own?  A separate one has all SMs where a few chains, or the last steps of a few long ones among many
// short, leave some idle; with at most half as many chains as SMs two CTAs share a chain of it besides.  In units of 1000 SM cycles a step of the chain without the
// output takes 4.2 shared and 5.5 not, with it what `step` says; the separate output takes 8.5 with a norm and 8.8 without per chunk and SM, and 7 to launch (8.4 with a 32-bit gate).  What takes the
// steps is the longest chain, or the even share of all.  Fitted to 656 equal and unequal batches of 60 to 700 chains x 1 to 48 steps and, each with and without backward
// pass, norm and 16-bit types, 266 of 4 to 400 chains.  Of the latter at most 3 in 266 are on the wrong side by 2 % or more, by up to 7 %.
// Times in us with norm and backward pass, fused and separate, x 16 heads: documents of 3000, 2000, 1500, 1000 and 692 tokens 421 and 374, one of 2048 and 12
// of 512 345 and 338, five of 1536 279 and 291; x 8 heads one of 1024 and 30 of 64 137 and 110.
// The rows of a 32-bit gate have no place in the shared memory of the fused kernel, whose epilogue fetches them from where they are, 16 at a time: 20 k cycles for
// a step of 10.  Forward only, x 16 heads, one document of 48 chunks and 30 of one 674 and 285 us, six of 48 chunks with a backward pass 1021 and 621.
bool output_in_chain(const Call& c, bool need_bwd, bool gate_32_bits) {
    static const double step[3][2][2] = {{{7.8, 7.3}, {11.4, 9.8}}, {{12.6, 19.2}, {12.6, 21.0}}, {{4.9, 5.5}, {7.9, 7.2}}};      // 16-bit gate, 32-bit, no norm; backward pass; not shared
    const double sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount, share = (double)c.NC * c.HV / sms;
    const bool shared = 2.0 * c.NS * c.HV <= sms;
    const double steps = shared ? c.chain : std::max((double)c.chain, share), fused = step[c.has_ep ? gate_32_bits : 2][need_bwd][!shared];
    // forward only the separate kernels allocate states and Vd, 96 KB per chunk and head, that the fused one never writes: 3 % has to be gained for more than 64 MB of
    // them (for any number: two documents of 256 tokens x 16 heads 38.2 us instead of 36.8)
    const bool costly = !need_bwd && c.tiles(MKDA_STATE_TILE_BYTES + MKDA_CHUNK_TILE_BYTES) > 64 << 20;
    return steps * fused <= (costly ? 1.03 : 1.0) * (steps * (shared ? 4.2 : 5.5) + share * (c.has_ep ? 8.5 : 8.8) + (gate_32_bits ? 8.4 : 7.0));
}

// Segments longest first, unless all of them run at once.  In the order of the documents a long one that starts late is waited for at the end:
// 22 documents of 1 to 19 chunks x 32 heads 156 -> 146 us, 86 of up to 76 chunks 1813 -> 1720 (forward) and 1270 -> 1221 (backward).
const int* segment_order(const Call& c) {
    return (int64_t)c.NS * c.HV > at::cuda::getCurrentDeviceProperties()->multiProcessorCount ? c.seg_order : nullptr;
}

}  // namespace

void run_step(const Call& c, const Inputs& in, Tensor& out, Tensor& ht) {
    const Tensor alog = aligned_f32(in.A_log), bias = aligned_f32(in.dt_bias), w = aligned(in.ep_w);
    MkdaStepFwd p{};
    p.short_only = out.defined();
    if (!out.defined()) {
        out = c.rows_out(c.HV, c.has_ep ? at::kFloat : in.q.scalar_type());
        if (c.want_ht) ht = c.states(c.N);
    }
    p.L = c.layout(); p.N = c.N; p.seq_chunk_off = c.seq_off; p.longest = c.longest;
    p.q = in.q.data_ptr(); p.k = in.k.data_ptr(); p.v = in.v.data_ptr(); p.qkv_dtype = c.qkv_dtype;
    p.x = in.x.data_ptr(); p.x_dtype = dtype_code(in.x); p.scalar_gate = c.scalar_gate; p.A_log = fptr(alog); p.dt_bias = fptr(bias);
    p.mode = c.mode; p.lower_bound = c.lower_bound; p.beta = in.beta.data_ptr(); p.beta_dtype = dtype_code(in.beta); p.beta_sigmoid = c.beta_sigmoid;
    p.beta_scale = c.beta_scale; p.l2 = c.l2; p.scale = c.scale; p.h0 = fptr(in.h0); p.ht = fptr(ht); p.state_v_first = c.vf; p.has_norm = c.has_ep;
    if (c.has_ep) {
        if (w.defined()) { p.norm_w = w.data_ptr(); p.norm_w_dtype = dtype_code(w); }
        p.gate = in.ep_gate.data_ptr(); p.gate_dtype = dtype_code(in.ep_gate); p.act = c.act; p.eps = c.eps;
    }
    p.out = out.data_ptr(); p.out_dtype = dtype_code(out);
    check_rc(mkda_step_fwd(&p, c10::cuda::getCurrentCUDAStream()), "mkda_step_fwd");
}

std::pair<Tensor, Tensor> run_forward(const Call& c, const Inputs& in, bool need_bwd, Saved& s) {
    cudaStream_t st = c10::cuda::getCurrentCUDAStream();
    const int64_t row = (int64_t)c.TT * c.HV * 128 * 4, seg_states = (int64_t)c.NS * c.HV * 65536;
    const Tensor alog = aligned_f32(in.A_log), bias = aligned_f32(in.dt_bias);
    Arena tmp;
    Arena& keep = s.arena;
    float *u = nullptr, *hs = nullptr, *s_in = nullptr;
    int* warm_start = nullptr;
    if (c.l2 && need_bwd) {
        keep.want(&s.q_rstd, (int64_t)c.TT * c.HK * 4);
        keep.want(&s.k_rstd, (int64_t)c.TT * c.HK * 4);
    }
    const bool one_kernel = gate_in_intra(c);
    if (need_bwd || !one_kernel) {
        keep.want(&s.g_c, c.scalar_gate ? row / 128 : row);
        keep.want(&s.beta_e, (int64_t)c.TT * c.HV * 4);
    }
    if (need_bwd) keep.want(&s.A, c.tiles(MKDA_QUARTER_TILE_BYTES));
    keep.want(&s.Aqk, c.tiles(MKDA_QUARTER_TILE_BYTES));
    keep.want(&s.nw, c.tiles(MKDA_CHUNK_TILE_BYTES));
    keep.want(&s.kbar, c.tiles(MKDA_CHUNK_TILE_BYTES));
    keep.want(&s.qs, c.tiles(MKDA_CHUNK_TILE_BYTES));
    keep.want(&s.gl, c.tiles(512));
    const bool fused = output_in_chain(c, need_bwd, c.has_ep && in.ep_gate.scalar_type() == at::kFloat);
    if (need_bwd || !fused) {
        keep.want(&s.h, c.tiles(MKDA_STATE_TILE_BYTES));
        keep.want(&s.Vd, c.tiles(MKDA_CHUNK_TILE_BYTES));
    }
    if (c.has_ep && need_bwd) keep.want(&s.o_raw, row);
    tmp.want(&u, c.tiles(MKDA_CHUNK_TILE_BYTES));
    if (c.segmented) {
        keep.want(&s.ms, seg_states);
        tmp.want(&hs, seg_states);
        tmp.want(&s_in, seg_states);
        if (c.warm) {
            keep.want(&s.warm_end, (int64_t)c.NS * c.HV * 4);
            tmp.want(&warm_start, (int64_t)c.NS * c.HV * 4);
        }
    }
    keep.allocate(c.dev);
    tmp.allocate(c.dev);
    const MkdaLayout L = c.layout();
    const int* order = segment_order(c);

    {
        MkdaGateFwd g{};
        g.L = L; g.x = in.x.data_ptr(); g.x_dtype = dtype_code(in.x); g.scalar_gate = c.scalar_gate;
        g.A_log = fptr(alog); g.dt_bias = fptr(bias); g.mode = c.mode; g.lower_bound = c.lower_bound;
        g.beta_raw = in.beta.data_ptr(); g.beta_dtype = dtype_code(in.beta); g.beta_sigmoid = c.beta_sigmoid;
        g.beta_scale = c.beta_scale; g.beta_out = s.beta_e; g.g_c = s.g_c;
        MkdaIntraFwd p{};
        p.L = L; p.q = in.q.data_ptr(); p.k = in.k.data_ptr(); p.v = in.v.data_ptr(); p.qkv_dtype = c.qkv_dtype;
        p.g_c = s.g_c; p.beta = s.beta_e; p.scalar_gate = c.scalar_gate; p.scale = c.scale;
        p.l2 = c.l2; p.l2_eps = 1e-6f; p.q_rstd_out = s.q_rstd; p.k_rstd_out = s.k_rstd;
        p.A = s.A; p.Aqk = s.Aqk; p.nw = s.nw; p.u = u; p.kbar = s.kbar; p.qs = s.qs; p.gl = s.gl;
        if (one_kernel) {
            check_rc(mkda_gate_intra_fwd(&g, &p, st), "mkda_gate_intra_fwd");
        } else {
            check_rc(mkda_gate_cumsum_fwd(&g, st), "mkda_gate_cumsum_fwd");
            check_rc(need_bwd ? mkda_intra_fwd(&p, st) : mkda_intra_fwd_forward_only(&p, st), "mkda_intra_fwd");
        }
    }
    Tensor ht;
    if (c.want_ht) ht = c.states(c.N);
    Tensor out = c.rows_out(c.HV, c.has_ep ? at::kFloat : in.q.scalar_type());
    const Tensor w = aligned(in.ep_w);
    MkdaChainFwd p{};
    MkdaRecurFwd& r = p.r;
    r.L = L; r.nw = s.nw; r.u = u; r.kbar = s.kbar; r.gl = s.gl; r.state_v_first = c.vf;
    if (c.segmented) {
        // pre-pass from zero: per-segment (state, transition); the prefix combine then gives the state entering every segment
        if (c.warm) {
            MkdaWarmup w{};
            w.L = L; w.gl = s.gl; w.threshold_log2 = c.warm_log2; w.warm_start = warm_start; w.warm_end = s.warm_end;
            check_rc(mkda_warmup_chunks(&w, st), "mkda_warmup_chunks");
        }
        MkdaRecurFwd pre = r;
        pre.state_v_first = 0; pre.ht = hs; pre.want_transition = 1; pre.mt = s.ms; pre.warm_start = warm_start;
        check_rc(mkda_recur_fwd_ordered(&pre, order, st), "mkda_recur_fwd");
        MkdaCombine m{};
        m.NG = c.N; m.HV = c.HV; m.grp_seg_off = c.grp_off; m.hs = hs; m.ms = s.ms; m.carry = fptr(in.h0); m.s_in = s_in;
        m.carry_v_first = c.vf;
        check_rc(mkda_state_combine(&m, st), "mkda_state_combine");
        r.h0 = s_in; r.h0_k_first = 1; r.seg_ht = c.seg_last;
    } else {
        r.h0 = fptr(in.h0);
    }
    r.h = s.h; r.Vd = s.Vd; r.ht = fptr(ht);
    MkdaOutFwd& o = p.o;
    o.L = L; o.qs = s.qs; o.Aqk = s.Aqk; o.has_norm = c.has_ep;
    if (c.has_ep) {
        if (w.defined()) { o.norm_w = w.data_ptr(); o.norm_w_dtype = dtype_code(w); }
        o.gate = in.ep_gate.data_ptr(); o.gate_dtype = dtype_code(in.ep_gate); o.act = c.act; o.eps = c.eps;
    }
    o.o_raw = s.o_raw; o.out = out.data_ptr(); o.out_dtype = dtype_code(out);
    if (fused) {
        check_rc(mkda_chain_fwd_ordered(&p, order, st), "mkda_chain_fwd");
    } else {
        o.h = s.h; o.Vd = s.Vd;
        check_rc(mkda_recur_fwd_ordered(&r, order, st), "mkda_recur_fwd");
        check_rc(mkda_out_fwd(&o, st), "mkda_out_fwd");
    }
    return {out, ht};
}

Grads run_backward(const Call& c, const Inputs& in, Saved& s, Tensor dy, Tensor dht, bool need_alog, bool need_bias, bool need_h0) {
    cudaStream_t st = c10::cuda::getCurrentCUDAStream();
    const MkdaLayout L = c.layout();
    const int* order = segment_order(c);
    Grads g;
    if (!dy.defined()) dy = at::zeros({c.B, c.T, c.HV, 128}, in.q.options().dtype(c.has_ep ? at::kFloat : in.q.scalar_type()));
    if (dht.defined()) dht = aligned(aligned_f32(dht), 32);
    need_h0 = need_h0 && in.h0.defined();

    Arena tmp;
    float *dO = nullptr, *dh = nullptr, *dVd = nullptr, *dq_v = nullptr, *dk_v = nullptr, *dgp = nullptr, *part_w = nullptr, *part_b = nullptr,
          *part_a = nullptr, *dloc = nullptr, *g_in = nullptr;
    const int64_t tile = MKDA_CHUNK_TILE_BYTES, seg_states = (int64_t)c.NS * c.HV * 65536;
    const int w_rows = std::min(c.NC * c.HV, MKDA_EPILOGUE_MAX_PART_ROWS);
    const int g_rows = std::min(c.NC, 256), g_width = c.scalar_gate ? c.HV : c.HV * 128;
    // bf16 gradients of an output without a norm are operands as they stand; only chunks that are not full need tiles
    const bool rows = !c.has_ep && c.qkv_dtype == MKDA_BF16 && dy.scalar_type() == at::kBFloat16, ragged = !c.covers_all || (int64_t)c.NC * 64 != c.TT;
    if (!rows || ragged) tmp.want(&dO, c.tiles(tile));
    tmp.want(&dh, c.tiles(MKDA_STATE_TILE_BYTES));
    tmp.want(&dVd, c.tiles(tile));
    const bool spread = spread_v_heads(c);
    const bool finished = !c.l2 && c.HV == c.HK;          // dq and dk leave the chunk kernel as they are
    if (!finished) {
        tmp.want(&dq_v, (int64_t)c.NC * (spread ? c.HV : c.HK) * tile);
        tmp.want(&dk_v, (int64_t)c.NC * (spread ? c.HV : c.HK) * tile);
    }
    tmp.want(&dgp, c.tiles(c.scalar_gate ? 256 : tile));
    if (c.has_ep && in.ep_w.defined()) tmp.want(&part_w, (int64_t)w_rows * 512);
    if (c.mode != MKDA_GATE_PRECOMPUTED) {
        if (need_bias) tmp.want(&part_b, (int64_t)g_rows * g_width * 4);
        if (need_alog) tmp.want(&part_a, (int64_t)g_rows * c.HV * 4);
    }
    if (c.segmented) { tmp.want(&dloc, seg_states); tmp.want(&g_in, seg_states); }
    tmp.allocate(c.dev);

    MkdaBwdDh d{};
    d.L = L;
    if (c.has_ep) {      // dO leaves the epilogue backward in the tile form the tensor-core kernels fetch
        int64_t rs, cs;
        if (!rows_strides(dy, rs, cs)) { dy = aligned(dy); rs = 128; cs = 1; }
        const Tensor w = aligned(in.ep_w);
        g.ep_gate = c.like_out(in.ep_gate);
        MkdaEpilogueBwdTiles p{};
        p.L = L; p.dy = dy.data_ptr(); p.dy_dtype = dtype_code(dy); p.dy_row_stride = (int)rs; p.dy_col_stride = (int)cs; p.o_raw = s.o_raw;
        if (w.defined()) { p.norm_w = w.data_ptr(); p.norm_w_dtype = dtype_code(w); }
        p.gate = in.ep_gate.data_ptr(); p.gate_dtype = dtype_code(in.ep_gate); p.act = c.act; p.eps = c.eps;
        p.dO_t = dO; p.dgate = g.ep_gate.data_ptr(); p.dgate_dtype = dtype_code(g.ep_gate); p.part_rows = w_rows; p.part_w = part_w;
        check_rc(mkda_epilogue_bwd_tiles(&p, st), "mkda_epilogue_bwd_tiles");
        d.dO_in_t = dO;
    } else {
        dy = aligned(dy);
        d.d_o = dy.data_ptr(); d.do_dtype = dtype_code(dy); d.dO_t = dO;
    }
    d.kbar = s.kbar; d.qs = s.qs; d.gl = s.gl; d.Aqk = s.Aqk; d.nw = s.nw;
    if (need_h0) g.h0 = c.states(c.N);
    MkdaBwdDh full = d;
    if (c.segmented) {
        // pre-pass from zero: only the gradient entering each segment is wanted, nothing per chunk is stored
        d.dh0 = dloc; d.warm_end = s.warm_end;
        check_rc(rows ? mkda_bwd_dh_rows(&d, order, st) : mkda_bwd_dh_ordered(&d, order, st), "mkda_bwd_dh");
        MkdaCombine m{};
        m.NG = c.N; m.HV = c.HV; m.grp_seg_off = c.grp_off; m.hs = dloc; m.ms = s.ms; m.carry = fptr(dht); m.reverse = 1; m.s_in = g_in;
        m.s_out = fptr(g.h0); m.carry_v_first = c.vf; m.out_v_first = c.vf;
        check_rc(mkda_state_combine(&m, st), "mkda_state_combine");
        full.dht = g_in;
    } else {
        full.dht = fptr(dht); full.state_v_first = c.vf; full.dh0 = fptr(g.h0);
    }
    full.dh = dh; full.dVd_t = dVd;
    if (c.segmented) full.dO_in_t = dO;                    // already in tile form
    check_rc(rows ? mkda_bwd_dh_rows(&full, order, st) : mkda_bwd_dh_ordered(&full, order, st), "mkda_bwd_dh");
    g.v = c.rows_out(c.HV, in.v.scalar_type());
    g.beta = c.like_out(in.beta);
    g.q = c.rows_out(c.HK, in.q.scalar_type());
    g.k = c.rows_out(c.HK, in.k.scalar_type());
    {
        MkdaBwdChunk p{};
        p.L = L; p.q = in.q.data_ptr(); p.k = in.k.data_ptr(); p.v = in.v.data_ptr(); p.qkv_dtype = c.qkv_dtype;
        p.q_rstd = s.q_rstd; p.k_rstd = s.k_rstd; p.g_c = s.g_c; p.beta = s.beta_e; p.scalar_gate = c.scalar_gate; p.A = s.A; p.h = s.h;
        p.dh = dh; p.Vd = s.Vd; p.dO_t = dO; p.dVd_t = dVd; p.scale = c.scale; p.beta_raw = in.beta.data_ptr(); p.beta_dtype = dtype_code(in.beta);
        p.beta_sigmoid = c.beta_sigmoid; p.beta_scale = c.beta_scale; p.dq_v = dq_v; p.dk_v = dk_v; p.dgp = dgp; p.dbeta = g.beta.data_ptr();
        p.dbeta_dtype = dtype_code(g.beta); p.dv = g.v.data_ptr(); p.per_v_head = spread;
        check_rc(mkda_bwd_chunk_rows(&p, rows ? dy.data_ptr() : nullptr, finished ? g.q.data_ptr() : nullptr, finished ? g.k.data_ptr() : nullptr, st), "mkda_bwd_chunk");
    }
    g.x = c.like_out(in.x);
    {
        const Tensor alog = aligned_f32(in.A_log), bias = aligned_f32(in.dt_bias);
        MkdaGateBwd p{};
        p.L = L; p.x = in.x.data_ptr(); p.x_dtype = dtype_code(in.x); p.scalar_gate = c.scalar_gate; p.A_log = fptr(alog);
        p.dt_bias = fptr(bias); p.mode = c.mode; p.lower_bound = c.lower_bound; p.dgp = dgp; p.dx = g.x.data_ptr(); p.dx_dtype = dtype_code(g.x);
        p.part_rows = std::max(g_rows, 1); p.part_bias = part_b; p.part_alog = part_a;
        check_rc(mkda_gate_bwd(&p, st), "mkda_gate_bwd");
    }
    if (part_w || part_b || part_a) {                      // the parameter gradients' second stage, in one launch (no chunk: sums of no rows)
        MkdaReduceMulti p{};
        if (part_w) { g.ep_w = new_cuda({128}, at::kFloat, c.dev); p.job[0] = {part_w, w_rows, 128, 1, fptr(g.ep_w)}; }
        if (part_b) { g.dt_bias = new_cuda(in.dt_bias.sizes(), at::kFloat, c.dev); p.job[1] = {part_b, g_rows, g_width, 1, fptr(g.dt_bias)}; }
        if (part_a) { g.A_log = new_cuda(in.A_log.sizes(), at::kFloat, c.dev); p.job[2] = {part_a, g_rows, c.HV, 1, fptr(g.A_log)}; }
        check_rc(mkda_reduce_multi(&p, st), "mkda_reduce_multi");
        auto cast = [](Tensor& t, const Tensor& like) { if (t.defined() && t.scalar_type() != like.scalar_type()) t = t.to(like.scalar_type()); };
        cast(g.ep_w, in.ep_w); cast(g.dt_bias, in.dt_bias); cast(g.A_log, in.A_log);
    }
    if (!finished) {
        MkdaQkGrad p{};
        p.L = L; p.dq_v = dq_v; p.dk_v = dk_v; p.q = in.q.data_ptr(); p.k = in.k.data_ptr(); p.x_dtype = c.qkv_dtype;
        p.q_rstd = s.q_rstd; p.k_rstd = s.k_rstd; p.dq = g.q.data_ptr(); p.dk = g.k.data_ptr(); p.per_v_head = spread;
        check_rc(mkda_qk_grad_finish(&p, st), "mkda_qk_grad_finish");
    }
    return g;
}

}  // namespace mkda_host
