// Host path of one layer call over the C ABI of libmkda: geometry, buffers and the launches of the forward and the backward pass.
// layer.cpp launches, binding.cpp is the autograd node and the Python entry points; neither holds device code.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/mkda.h"

namespace mkda_host {

using at::Tensor;

struct LibraryError : std::runtime_error { using std::runtime_error::runtime_error; };      // an entry point of libmkda returned an error
int dtype_code(const Tensor& t);           // MKDA_F32 / MKDA_BF16 / MKDA_F16; TypeError otherwise
// The kernels read and write their tensors with 16-byte vector accesses and bulk copies: operands are made contiguous and, where a
// contiguous view starts at an odd storage offset, copied.
Tensor aligned(const Tensor& t, uintptr_t to = 16);
Tensor new_cuda(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev);

// The intermediates of one pass, requested together.  Up to ARENA_SINGLE bytes they share one allocation (a call on a short sequence
// is bound by the host: one request instead of ten); above that each gets its own, so that the caching allocator can reuse the
// blocks one by one.
constexpr int64_t ARENA_SINGLE = 64 << 20;
struct Arena {
    struct Req { void** dst; int64_t bytes, offset; size_t block; };
    std::vector<Req> reqs;
    std::vector<Tensor> keep;
    template <typename T>
    void want(T** dst, int64_t bytes) { reqs.push_back({reinterpret_cast<void**>(dst), (std::max<int64_t>(bytes, 1) + 255) / 256 * 256, 0, 0}); }
    void allocate(const at::Device& dev) {
        int64_t total = 0;
        for (const auto& r : reqs) total += r.bytes;
        const bool single = total <= ARENA_SINGLE;
        if (single && total) keep.push_back(new_cuda({total}, at::kByte, dev));
        int64_t at = 0;
        for (auto& r : reqs) {
            if (!single) keep.push_back(new_cuda({r.bytes}, at::kByte, dev));
            r.block = keep.size() - 1;
            r.offset = single ? at : 0;
            at += r.bytes;
        }
        point();
    }
    void point() {                         // the pointers into the blocks of `keep`, which may have been elsewhere in between
        for (const auto& r : reqs) *r.dst = static_cast<char*>(keep[r.block].data_ptr()) + r.offset;
    }
};

// Options and geometry of a call.
struct Call {
    int B, T, HK, HV, N, NC, NS, TT, longest, chain, few;          // few: sequences of 1 to MKDA_STEP_MAX_TOKENS tokens
    bool segmented, covers_all, scalar_gate, l2, vf, want_ht, beta_sigmoid, has_ep, warm;
    int mode, act, qkv_dtype;
    float scale, lower_bound, beta_scale, eps, warm_log2;
    Tensor tables;                         // index.py: eight int32 tables, each padded to a multiple of four entries
    const int *chunk_start, *chunk_len, *seg_off, *grp_off, *seq_off, *seg_last, *seg_order;
    at::Device dev = at::Device(at::kCUDA);

    MkdaLayout layout() const { return MkdaLayout{TT, NC, NS, HK, HV, chunk_start, chunk_len, seg_off}; }
    void set_tables(const Tensor& t) {
        tables = t;
        const int* p = static_cast<const int*>(t.data_ptr());
        auto next = [&](int n) { const int* r = p; p += (n + 3) / 4 * 4; return r; };
        chunk_start = next(NC); chunk_len = next(NC); seg_off = next(NS + 1); grp_off = next(N + 1); seq_off = next(N + 1);
        next(NS);
        seg_last = next(NS);
        seg_order = next(NS);
    }
    int64_t tiles(int64_t bytes) const { return (int64_t)NC * HV * bytes; }
    Tensor rows_out(int64_t heads, at::ScalarType dt) const {      // [B,T,heads,128]; tokens outside every sequence are zero
        Tensor t = new_cuda({B, T, heads, 128}, dt, dev);
        if (!covers_all) t.zero_();
        return t;
    }
    Tensor like_out(const Tensor& x) const { return covers_all ? at::empty_like(x) : at::zeros_like(x); }
    Tensor states(int64_t n) const { return new_cuda({n, HV, 128, 128}, at::kFloat, dev); }
};

// What the forward pass leaves for the backward pass (pointers into `arena`).
struct Saved {
    Arena arena;
    float *q_rstd = nullptr, *k_rstd = nullptr, *g_c = nullptr, *beta_e = nullptr, *A = nullptr, *Aqk = nullptr, *nw = nullptr,
          *kbar = nullptr, *qs = nullptr, *gl = nullptr, *h = nullptr, *Vd = nullptr, *o_raw = nullptr, *ms = nullptr;
    int* warm_end = nullptr;
};

struct Inputs { Tensor q, k, v, x, beta, A_log, dt_bias, h0, ep_w, ep_gate; };
struct Grads { Tensor q, k, v, x, beta, A_log, dt_bias, h0, ep_w, ep_gate; };

// Every sequence token by token (undefined `out`: allocated here), or only those of a few tokens over the results of run_forward.
void run_step(const Call& c, const Inputs& in, Tensor& out, Tensor& ht);
std::pair<Tensor, Tensor> run_forward(const Call& c, const Inputs& in, bool need_bwd, Saved& s);
Grads run_backward(const Call& c, const Inputs& in, Saved& s, Tensor dy, Tensor dht, bool need_alog, bool need_bias, bool need_h0);

}  // namespace mkda_host
