// Serial state recurrences on the Blackwell tensor cores.
//
// One CTA per (v-head, segment) carries the whole 128 x 128 state, TRANSPOSED: accumulator lane = v, columns = K index.  The fp32 state
// lives in the registers of 512 compute threads (thread = one lane x 32 columns); with few chains recur_fwd and bwd_dh take two CTAs of 64 rows
// and 256 working compute threads each (split_chains).  Each step the state is split into packed bf16 hi / lo pairs in
// tensor memory, where the products take it as their left operand, and the products' result comes back from an fp32 accumulator:
//   forward   D^T = u^T + S^T nw^T = Vd^T        S^T <- S^T diag(gl) + Vd^T kbar
//   reverse   D^T = dO^T Aqk + dS^T kbar^T = dVd^T      dS^T <- dS^T diag(gl) + dO^T (scale q 2^g) + dVd^T nw
// The right operands are ready-made tiles (nw^T, kbar, u^T, dO, Aqk, scale q 2^g), fetched by bulk copy ahead of their step.
//
// What bounds it: with many chains HBM (192 / 240 KB per step and SM); with few the chain of a step, state -> operand -> product -> operand ->
// product.  Hence: both left operands in tensor memory (no shared-memory tile to build, to fence and to fetch from: 24 + 12 products of
// ~32 + 64 cycles instead of 49 + 64.5); one warp that issues products and one that issues copies, joined with the compute warps by
// mbarriers, so that nothing but the chain itself is waited for; everything else of a step (saved tiles, which leave as 32-byte pieces
// straight from registers; the next chunk's u^T; the products that do not depend on the state) is done while products run.
// 512 threads used to build both operands in shared memory behind CTA-wide barriers: 7.2 - 9.7 k cycles per step.
#include "host.h"
#include "intra.cuh"

#include <string.h>
#include <type_traits>

namespace mkda {

namespace rc {
constexpr int COMPUTE = 512, THREADS = 576, WARP_MMA = 16, WARP_LOAD = 17, WARP_STORE = 18, WARP_GATE = 19;
constexpr int KB = 1024;
constexpr int SH = 128, SL = 192, VH = 448, VL = 480;      // tensor-memory columns of the left operands (hi, lo)
constexpr int X = 0, D0 = 256, D1 = 320, O = 384;          // fp32 accumulators: state increment, D (two for the forward kernel), output

using umma::signal_tmem;
using umma::store_pair;
using umma::wait_mma;

// 32 bytes of fp32 in one load, `src` 32-byte aligned
__device__ __forceinline__ void ld32b(const void* src, float* v) {
    uint32_t w[8];
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(src));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
}
// The state <-> caller-visible memory: thread (row, cg) holds columns [32 cg, 32 cg + 32) of row `row` (v).
__device__ __forceinline__ void load_state(const float* __restrict__ src, bool v_first, int row, int cg, float (&s)[32]) {
    if (v_first) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ld32b(src + (size_t)row * DK + cg * 32 + i * 8, s + 8 * i);
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = src[(size_t)(cg * 32 + j) * DV + row];
    }
}
__device__ __forceinline__ void store_state(float* __restrict__ dst, bool v_first, int row, int cg, const float (&s)[32]) {
    if (v_first) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(s[8 * i + e]);
            st32b(dst + (size_t)row * DK + cg * 32 + i * 8, w);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[(size_t)(cg * 32 + j) * DV + row] = s[j];
    }
}
// s <- s gl + X for this thread's 32 columns, 16 at a time; gl points at the factors of its columns
__device__ __forceinline__ void advance_state(uint32_t taddr, const float* gl, float (&s)[32]) {
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        float x[16];
        umma::tmem_ld16(taddr + 16 * hf, x);
#pragma unroll
        for (int j4 = 0; j4 < 16; j4 += 4) {
            const float4 f = *reinterpret_cast<const float4*>(gl + 16 * hf + j4);
            const int j = 16 * hf + j4;
            unpack2(fma2(pack2(s[j], s[j + 1]), pack2(f.x, f.y), pack2(x[j4], x[j4 + 1])), s[j], s[j + 1]);
            unpack2(fma2(pack2(s[j + 2], s[j + 3]), pack2(f.z, f.w), pack2(x[j4 + 2], x[j4 + 3])), s[j + 2], s[j + 3]);
        }
    }
}
// the state as the left operand of the next products
__device__ __forceinline__ void state_operand(uint32_t tmem, int warp, int cg, const float (&s)[32], uint32_t (&h)[16], uint32_t (&l)[16],
                                              uint64_t* used = nullptr, uint32_t parity = 0) {        // `used`: completes once the old one has been read
#pragma unroll
    for (int i = 0; i < 16; ++i) umma::split2(s[2 * i], s[2 * i + 1], h[i], l[i]);
    if (used) wait_mma(used, parity);
    umma::tmem_st16(umma::tmem_addr(tmem, warp, SH + cg * 16), h);
    umma::tmem_st16(umma::tmem_addr(tmem, warp, SL + cg * 16), l);
    umma::tmem_wait_st();
}
__device__ __forceinline__ void save_state_tile(uint8_t* tile, int row, int cg, const uint32_t (&h)[16], const uint32_t (&l)[16]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        store_pair(tile, 128, row, 4 * cg + 2 * i, h + 8 * i);
        store_pair(tile + 32768, 128, row, 4 * cg + 2 * i, l + 8 * i);
    }
}
// one half (hi or lo) of this thread's part of the state tile in shared memory
__device__ __forceinline__ void stage_state(uint8_t* tile, int row, int cg, const uint32_t (&w)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(tile + umma::tile_chunk_offset(128, row, 4 * cg + i)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
}
// Vd^T (dVd^T) from its accumulator: left operand, and optionally the saved chunk tile
__device__ __forceinline__ void v_operand(uint32_t tmem, int d_col, int warp, int cg, uint32_t (&h)[8], uint32_t (&l)[8]) {
    float d[16];
    umma::tmem_ld16(umma::tmem_addr(tmem, warp, d_col + cg * 16), d);
#pragma unroll
    for (int i = 0; i < 8; ++i) umma::split2(d[2 * i], d[2 * i + 1], h[i], l[i]);
    umma::tmem_st8(umma::tmem_addr(tmem, warp, VH + cg * 8), h);
    umma::tmem_st8(umma::tmem_addr(tmem, warp, VL + cg * 8), l);
    umma::tmem_wait_st();
}
}  // namespace rc

// ---------------------------------------------------------------------------------------------------------
// forward.  OUT >= 0: the output O^T = S^T qs^T + Vd^T Aqk^T (qs = scale q 2^g) and its epilogue are computed in the same step.  Both left
// operands are in tensor memory anyway, the products fill the gaps in which the tensor pipe waits for the chain, and four more warps turn
// the accumulator into output rows: states and Vd need not travel through HBM to a kernel of their own (and are not written at all when
// no backward pass follows): 416 -> 320 KB per chunk and head with a backward pass, 400 -> 192 KB without.  OUT = type of the norm's gate,
// or of the output rows when there is no norm.
// The epilogue passes 16 rows at a time through shared memory ([row][value], conflict-free both ways): thread v reads its 16 values of the
// accumulator, then a warp takes four whole rows.  Gate rows come and output rows leave by tiled copies, and the state leaves through a
// 32 KB stage (hi half, then lo half): with plain loads and stores the load / store queue was what everything waited for (25 k cycles per
// chunk with thread-per-value accesses, 12 - 22 k with 512-byte rows).
// ---------------------------------------------------------------------------------------------------------
struct RecurShared {
    uint64_t fullN[2], fullK[2], fullU[2], fullQ, fullA;   // landed: nw^T and decay factors | kbar | u^T | scale q 2^g | Aqk
    uint64_t opS, opV, mmS, mmO, oFree;                    // state operand | Vd operand written; output products done; O accumulator read
    uint64_t uFree[2], mm1[2], mm2[2];                     // u^T used; the chain's products done.  Of even and odd steps: where their tiles have two
                                                           // buffers, the next step's could complete before the copying thread waits for this one's
    uint64_t fullG, gFree, ready[2], freed[2];             // gate rows landed | used; state halves staged | read by their copy
    uint32_t tmem;
    __align__(16) float gl[4][DK];                         // four deep: a step's factors are used at the start of the next one
    __align__(16) float w[DV];                             // weight of the norm
};
template <bool OUT>
struct RecurLayout {                                       // the plain recurrence double-buffers every tile
    static constexpr int D = OUT ? 1 : 2, T = 32 * rc::KB;
    static constexpr int N = 0, K = N + D * T, U = K + D * T, Q = U + D * T, A = Q + T, S = A + T / 2, G = S + T, STAGE = G + T / 2,
                         TILES = OUT ? STAGE + 32 * rc::KB : Q, SMEM = TILES + (int)sizeof(RecurShared),
                         THREADS = OUT ? 768 : 576, REGS = OUT ? 80 : 96;
    static_assert(SMEM <= 232448, "shared memory of one CTA");
};
struct ChainMaps { CUtensorMap gate, raw, out; };          // rows of a head: boxes of 64 (gate) and 16 rows

template <int DT, bool NORM>
__device__ __forceinline__ void recur_epilogue(const MkdaOutFwd& o, const ChainMaps& maps, RecurShared& sh, uint8_t* base, int h, int c_beg, int n) {
    using namespace rc;
    using L = RecurLayout<true>;
    const int HV = o.L.HV, tid = threadIdx.x & 127, w = tid >> 5, lane = tid & 31;
    const int r = tid >> 3, c = tid & 7;                   // row of a group, 16-byte piece: this thread's values are 4 (c + 8 i) + 0..3
    const uint32_t acc = umma::tmem_addr(sh.tmem, w, O);
    const bool silu = o.act == MKDA_ACT_SILU, raw = o.o_raw != nullptr;
    constexpr int ODT = NORM ? MKDA_F32 : DT;
    if (NORM) sh.w[tid] = o.norm_w ? ld1(o.norm_w, o.norm_w_dtype, tid) : 1.f;
    uint32_t buf = 0;
    for (int k = 0; k < n; ++k) {
        const int start = o.L.chunk_start[c_beg + k], len = o.L.chunk_len[c_beg + k];
        if (NORM && DT != MKDA_F32) umma::mbar_wait(&sh.fullG, k & 1);
        wait_mma(&sh.mmO, k & 1);
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
            if (16 * g >= len) break;
            float* st = reinterpret_cast<float*>(base + L::STAGE + (buf & 1) * 8192);
            uint8_t* so = base + L::STAGE + 16384 + (buf & 1) * 8192;
            {
                float x[16];
                umma::tmem_ld16(acc + 16 * g, x);
#pragma unroll
                for (int j = 0; j < 16; ++j) st[j * 128 + tid] = x[j];
            }
            if (16 * g + 16 >= len) signal_tmem(&sh.oFree, lane);
            asm volatile("bar.sync 2, 128;" ::: "memory");
            const int row = 16 * g + r;
            const bool whole = 16 * g + 16 <= len, valid = row < len;
            const size_t at = ((size_t)(start + (valid ? row : len - 1)) * HV + h) * 128 + 4 * c;
            float4 x[4];
            float f = 1.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(st + r * 128 + 4 * (c + 8 * i));
            if (!whole && raw && valid) {
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(o.o_raw + at + 32 * i) = x[i];
            }
            if (NORM) {
                float ss = norm_piece(x[0]);
#pragma unroll
                for (int i = 1; i < 4; ++i) ss = __fadd_rn(ss, norm_piece(x[i]));
                f = norm_rs(norm_butterfly(ss), o.eps);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (NORM) {
                    const float4 z = DT == MKDA_F32 ? ld4(o.gate, DT, at + 32 * i) : ld4(base + L::G, DT, row * 128 + 4 * (c + 8 * i));
                    x[i] = norm_gate(x[i], *reinterpret_cast<const float4*>(sh.w + 4 * (c + 8 * i)), z, f, silu);
                }
                if (whole) st4(so, ODT, r * 128 + 4 * (c + 8 * i), x[i]);
                else if (valid) st4(o.out, ODT, at + 32 * i, x[i]);
            }
            umma::fence_async_smem();
            if (tid == 0) umma::bulk_store_wait_read();    // the previous group's rows have left: the other buffers are free behind the barrier
            asm volatile("bar.sync 2, 128;" ::: "memory");
            if (whole && tid == 0) {
                if (raw) umma::tma_store_rows(&maps.raw, h * 128, start + 16 * g, st);
                umma::tma_store_rows(&maps.out, h * 128, start + 16 * g, so);
                umma::bulk_store_commit();
            }
            ++buf;
        }
        __syncwarp();
        if (lane == 0) umma::arrive(&sh.gFree);
    }
    if (tid == 0) umma::bulk_store_wait_read();
}

template <int OUT, bool NORM, bool SPLIT>
__device__ __forceinline__ void recur_body(const MkdaRecurFwd& p, const int* seg_order, const MkdaOutFwd& o, const ChainMaps& maps) {
    using namespace rc;
    using L = RecurLayout<(OUT >= 0)>;
    static_assert(!SPLIT || OUT < 0, "chain_fwd takes whole rows");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw;                              // no static shared memory: the dynamic block starts on a 1024-byte boundary
    RecurShared& sh = *reinterpret_cast<RecurShared*>(base + L::TILES);
    const bool trans = (SPLIT ? blockIdx.x >> 1 : blockIdx.x) == 1;
    const int v0 = SPLIT ? 64 * (blockIdx.x & 1) : 0;      // first of this CTA's rows of the transposed state, which are lanes 0, 1, ...
    const int h = blockIdx.y, HV = p.L.HV;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (umma::smem_u32(base) & 1023) {                     // ... and nothing runs if that ever fails to hold
        follow_stream();
        if (tid == 0) atomicExch(&umma::g_timeout_flag, 1u);
        return;
    }
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (tid == 0) {
        for (uint64_t* b : {&sh.fullN[0], &sh.fullN[1], &sh.fullK[0], &sh.fullK[1], &sh.fullU[0], &sh.fullU[1], &sh.fullQ, &sh.fullA, &sh.mm1[0], &sh.mm1[1],
                            &sh.mm2[0], &sh.mm2[1], &sh.mmS, &sh.mmO, &sh.fullG, &sh.freed[0], &sh.freed[1]})
            umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opS, &sh.opV, &sh.uFree[0], &sh.uFree[1], &sh.ready[0], &sh.ready[1]}) umma::mbar_init(b, SPLIT ? COMPUTE / 64 : COMPUTE / 32);
        umma::mbar_init(&sh.oFree, 4);
        umma::mbar_init(&sh.gFree, 4);
        umma::fence_barrier_init();
    }
    follow_stream();
    const int seg = seg_order ? seg_order[blockIdx.z] : blockIdx.z;

    // Warm-up truncation (a pass from zero only): where the decay accumulated from chunk warm_start to the segment's end
    // hides everything before it, the pass starts there; the transition is then zero and its CTA visits no chunk.
    int c_beg = p.L.seg_chunk_off[seg];
    const int c_end = p.L.seg_chunk_off[seg + 1];
    bool cut = false;
    if (p.warm_start) {
        const int w = p.warm_start[seg * HV + h];
        if (w > c_beg) { cut = true; c_beg = trans ? c_end : w; }
    }
    umma::fence_before_sync();
    __syncthreads();                                       // the table entries have travelled while barriers and tensor memory were set up
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;
    const int n = c_end - c_beg;
    const bool save_h = OUT >= 0 && p.h;
    // Where the chain itself is what takes the time (no norm: a short epilogue), the output's products stand behind the chain's, and without
    // states to save their place is a second buffer for nw^T, which each step starts with.  In the gap in front of X the products held X up
    // whenever their tile or their accumulator was late: 5.4 -> 4.7 k cycles per step (scalar gate, 64 chains of 32 steps: 107 -> 95 us; of 256
    // steps with states saved: 1073 -> 971).  With the norm the epilogue or HBM is the bound, and the other order is faster by 5 %.
    // (At compile time, and the table entries read in front of the first barrier: two steps x 16 chains with the norm 12.0 -> 11.7 us.)
    constexpr bool late = OUT >= 0 && !NORM;
    const int dn = L::D > 1 || (late && !save_h) ? 2 : 1;
    auto buf_n = [&](int k) { return base + (L::D > 1 ? L::N + (k & 1) * L::T : (k & 1) && dn == 2 ? L::S : L::N); };
    auto n_bar = [&](int k) { return &sh.fullN[dn == 2 ? k & 1 : 0]; };
    auto n_par = [&](int k) { return (uint32_t)(dn == 2 ? k >> 1 : k) & 1; };
    auto step_par = [](int k) { return (uint32_t)(k >> 1) & 1; };      // of the barriers of even and odd steps
    auto buf_k = [&](int k) { return base + L::K + (k % L::D) * L::T; };
    auto buf_u = [&](int k) { return base + L::U + (k % L::D) * L::T; };

    if (warp >= 16) {
        if (OUT >= 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == WARP_LOAD) {
            if (umma::elect_one()) {
                auto tile = [&](uint8_t* dst, const float* t, int k, uint32_t bytes, uint64_t* bar) {
                    umma::bulk_load(dst, reinterpret_cast<const uint8_t*>(t) + ((size_t)(c_beg + k) * HV + h) * bytes, bytes, bar);
                };
                auto one = [&](uint8_t* dst, const float* t, int k, uint64_t* bar) {
                    umma::mbar_expect_tx(bar, umma::CHUNK_TILE_BYTES);
                    tile(dst, t, k, umma::CHUNK_TILE_BYTES, bar);
                };
                auto load_n = [&](int k) {
                    if (k >= n) return;
                    uint64_t* bar = n_bar(k);
                    umma::mbar_expect_tx(bar, umma::CHUNK_TILE_BYTES + DK * 4);
                    tile(buf_n(k), p.nw, k, umma::CHUNK_TILE_BYTES, bar);
                    umma::bulk_load(sh.gl[k & 3], p.gl + ((size_t)(c_beg + k) * HV + h) * DK, DK * 4, bar);
                };
                auto load_k = [&](int k) { if (k < n) one(buf_k(k), p.kbar, k, &sh.fullK[k % L::D]); };
                auto load_u = [&](int k) {
                    if (k >= n || trans) return;
                    if (!SPLIT) return one(buf_u(k), p.u, k, &sh.fullU[k % L::D]);
                    const uint8_t* src = reinterpret_cast<const uint8_t*>(p.u) + ((size_t)(c_beg + k) * HV + h) * umma::CHUNK_TILE_BYTES + 128 * v0;
                    umma::mbar_expect_tx(&sh.fullU[k % L::D], umma::CHUNK_TILE_BYTES / 2);
                    umma::bulk_load(buf_u(k), src, 8192, &sh.fullU[k % L::D]);
                    umma::bulk_load(buf_u(k) + 16384, src + 16384, 8192, &sh.fullU[k % L::D]);
                };
                auto load_q = [&](int k) { if (OUT >= 0 && k < n) one(base + L::Q, o.qs, k, &sh.fullQ); };
                auto load_a = [&](int k) {
                    if (OUT < 0 || k >= n) return;
                    umma::mbar_expect_tx(&sh.fullA, umma::QUARTER_TILE_BYTES);
                    tile(base + L::A, o.Aqk, k, umma::QUARTER_TILE_BYTES, &sh.fullA);
                };
                load_u(0); load_n(0); load_k(0); load_q(0); load_a(0);
                if (dn > 1) load_n(1);
                if (L::D > 1) { load_u(1); load_k(1); }
                if (n > 0) { umma::mbar_wait(&sh.uFree[0], 0); load_u(L::D); }
                for (int k = 0; k < n; ++k) {              // each buffer is refilled as soon as its product is done
                    auto u_free = [&]() { umma::mbar_wait(&sh.uFree[(k + 1) & 1], step_par(k + 1)); };
                    umma::mbar_wait(&sh.mm1[k & 1], step_par(k));
                    load_n(k + dn);
                    if (L::D > 1 && k + 1 < n) { u_free(); load_u(k + 1 + L::D); }
                    umma::mbar_wait(&sh.mm2[k & 1], step_par(k));
                    load_k(k + L::D);
                    if (OUT >= 0) {
                        if (late && k + 1 < n) { u_free(); load_u(k + 2); }
                        umma::mbar_wait(&sh.mmS, k & 1);
                        load_q(k + 1);
                        umma::mbar_wait(&sh.mmO, k & 1);
                        load_a(k + 1);
                        if (!late && k + 1 < n) { u_free(); load_u(k + 2); }
                    }
                }
            }
            __syncwarp();
        } else if (warp == WARP_MMA) {
            if (umma::elect_one()) {
                for (int k = 0; k < n; ++k) {
                    umma::mbar_wait(n_bar(k), n_par(k));
                    wait_mma(&sh.opS, k & 1);
                    umma::gemm_ta(tmem + ((k & 1) ? D1 : D0), tmem + SH, tmem + SL, umma::opnd_mn(buf_n(k), buf_n(k) + 16384, 128), 64, 128, trans ? 0u : 1u);
                    umma::commit(&sh.mm1[k & 1]);
                    auto output = [&]() {
                        umma::mbar_wait(&sh.fullQ, k & 1);
                        if (k) wait_mma(&sh.oFree, (k - 1) & 1);
                        umma::gemm_ta(tmem + O, tmem + SH, tmem + SL, umma::opnd_k(base + L::Q, base + L::Q + 16384, 64), 64, 128, 0u);
                        umma::commit(&sh.mmS);
                    };
                    if (OUT >= 0 && !late) output();
                    umma::mbar_wait(&sh.fullK[k % L::D], (k / L::D) & 1);
                    wait_mma(&sh.opV, k & 1);
                    umma::gemm_ta(tmem + X, tmem + VH, tmem + VL, umma::opnd_mn(buf_k(k), buf_k(k) + 16384, 64), 128, 64, 0u);
                    umma::commit(&sh.mm2[k & 1]);
                    if (OUT >= 0) {
                        if (late) output();
                        umma::mbar_wait(&sh.fullA, k & 1);
                        umma::gemm_ta(tmem + O, tmem + VH, tmem + VL, umma::opnd_k(base + L::A, base + L::A + 8192, 64), 64, 64, 1u);
                        umma::commit(&sh.mmO);
                    }
                }
            }
            __syncwarp();
        } else if (OUT >= 0 && warp >= 20) {
            recur_epilogue<OUT < 0 ? 0 : OUT, NORM>(o, maps, sh, base, h, c_beg, n);
        } else if (OUT > 0 && NORM && warp == WARP_GATE) {
            if (umma::elect_one()) {
                for (int k = 0; k < n; ++k) {              // rows past the chunk's end belong to the next sequence (or read as zeros) and are never used
                    const int start = o.L.chunk_start[c_beg + k];
                    if (k) {
                        umma::tma_prefetch_rows(&maps.gate, h * 128, start);
                        umma::mbar_wait(&sh.gFree, (k - 1) & 1);
                    }
                    umma::mbar_expect_tx(&sh.fullG, 16384);
                    umma::tma_load_rows(base + L::G, &maps.gate, h * 128, start, &sh.fullG);
                }
            }
            __syncwarp();
        } else if (OUT >= 0 && warp == WARP_STORE) {
            if (save_h && umma::elect_one()) {
                for (int k = 0; k < n; ++k) {
                    uint8_t* dst = reinterpret_cast<uint8_t*>(p.h) + ((size_t)(c_beg + k) * HV + h) * umma::STATE_TILE_BYTES;
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        umma::mbar_wait(&sh.ready[hf], k & 1);
                        umma::bulk_store(dst + hf * 32768, base + L::S, 32768);
                        umma::bulk_store_wait_read();
                        umma::arrive(&sh.freed[hf]);
                    }
                }
            }
            __syncwarp();
        }
    } else if (!SPLIT || (warp & 3) < 2) {
        if (OUT >= 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        const int cg = warp >> 2, row = (warp & 3) * 32 + lane, vrow = v0 + row;
        const bool vf = p.state_v_first != 0;
        float s[32];
        const int h0row = p.seg_h0 ? p.seg_h0[seg] : seg;
        if (!trans && !cut && p.h0 && h0row >= 0) {
            load_state(p.h0 + ((size_t)h0row * HV + h) * DK * DV, vf && !p.h0_k_first, vrow, cg, s);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) s[j] = trans && !cut && cg * 32 + j == vrow ? 1.f : 0.f;
        }
        // u^T of step k into the accumulator that its first product adds to
        auto preload_u = [&](int k) {
            umma::mbar_wait(n_bar(k), n_par(k));                       // this thread reads the decay factors that come with nw^T
            if (!trans) {
                umma::mbar_wait(&sh.fullU[k % L::D], (k / L::D) & 1);
                const uint8_t* u = buf_u(k);
                float a[8];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    umma::load_tile8(u, u + 16384, 128, row, 2 * cg + i, a);
                    uint32_t w[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(a[e]);
                    umma::tmem_st8(umma::tmem_addr(tmem, warp, ((k & 1) ? D1 : D0) + cg * 16 + 8 * i), w);
                }
                umma::tmem_wait_st();
            }
            signal_tmem(&sh.uFree[k & 1], lane);
        };
        if (n > 0) preload_u(0);
        for (int k = 0; k < n; ++k) {
            const size_t it = (size_t)(c_beg + k) * HV + h;
            if (k) {
                wait_mma(&sh.mm2[(k - 1) & 1], step_par(k - 1));
                advance_state(umma::tmem_addr(tmem, warp, X + cg * 32), &sh.gl[(k - 1) & 3][cg * 32], s);
            }
            uint32_t hi[16], lo[16];
            state_operand(tmem, warp, cg, s, hi, lo, late && k ? &sh.mmS : nullptr, (k - 1) & 1);
            signal_tmem(&sh.opS, lane);
            if (save_h) {
                if (k) umma::mbar_wait(&sh.freed[1], (k - 1) & 1);
                stage_state(base + L::S, row, cg, hi);
                umma::signal(&sh.ready[0], lane);
            } else if (OUT < 0 && p.h && !trans) {
                save_state_tile(reinterpret_cast<uint8_t*>(p.h) + it * umma::STATE_TILE_BYTES, vrow, cg, hi, lo);
            }
            wait_mma(&sh.mm1[k & 1], step_par(k));
            {
                uint32_t vh[8], vl[8];
                v_operand(tmem, (k & 1) ? D1 : D0, warp, cg, vh, vl);
                signal_tmem(&sh.opV, lane);
                if (p.Vd && !trans) {
                    uint8_t* tile = reinterpret_cast<uint8_t*>(p.Vd) + it * umma::CHUNK_TILE_BYTES;
                    store_pair(tile, 128, vrow, 2 * cg, vh);
                    store_pair(tile + 16384, 128, vrow, 2 * cg, vl);
                }
            }
            if (save_h) {
                umma::mbar_wait(&sh.freed[0], k & 1);
                stage_state(base + L::S, row, cg, lo);
                umma::signal(&sh.ready[1], lane);
            }
            if (k + 1 < n) preload_u(k + 1);
        }
        if (n > 0) {
            wait_mma(&sh.mm2[(n - 1) & 1], step_par(n - 1));
            advance_state(umma::tmem_addr(tmem, warp, X + cg * 32), &sh.gl[(n - 1) & 3][cg * 32], s);
        }
        // transition: M[K out][K in] with this thread holding row `row` = K in; state: [K][V] or [V][K]
        if (trans) {
            if (p.mt) store_state(p.mt + ((size_t)seg * HV + h) * DK * DK, false, vrow, cg, s);
        } else if (p.ht) {
            const int r = p.seg_ht ? p.seg_ht[seg] : seg;
            if (r >= 0) store_state(p.ht + ((size_t)r * HV + h) * DK * DV, vf, vrow, cg, s);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

template <bool SPLIT>
__global__ void __launch_bounds__(RecurLayout<false>::THREADS, 1) recur_fwd_tc_kernel(const MkdaRecurFwd p, const int* seg_order) {
    recur_body<-1, false, SPLIT>(p, seg_order, MkdaOutFwd{}, ChainMaps{});
}
template <int OUT, bool NORM>
__global__ void __launch_bounds__(RecurLayout<true>::THREADS, 1) chain_fwd_tc_kernel(const MkdaChainFwd p, const int* seg_order, const __grid_constant__ ChainMaps maps) {
    recur_body<OUT, NORM, false>(p.r, seg_order, p.o, maps);
}
// Rows of the transposed state (v) never meet: S^T nw, Vd^T kbar and their reverses contract over K and over tokens.  So with at most half as many
// chains as SMs a chain is shared between two CTAs of 64 rows each, with the same bits.  Per step and SM a forward CTA moves 128 KB then
// instead of 192 (nw and kbar whole, u, h and Vd by halves) in 4.0 instead of 5.5 k cycles, a reverse one 176 instead of 240 KB (nw, kbar, qs, Aqk whole,
// dO, dh and dVd by halves) in 4.6 instead of 6.9 k: 33 to 39 B per cycle all four.  recur_fwd 45 steps x 48 chains 131 -> 99 us, 16 x 32 48.5 -> 37.5, 4 x 4
// 15.2 -> 11.9; bwd_dh 150 -> 113, 56 -> 43, 15.7 -> 12.2, 256 x 64 894 -> 702.  (chain_fwd, with its single buffers kept, gained nothing: 256 x 64
// 996 us, 32 x 64 95; what its step waits for has not been shown.)
static bool split_chains(long long chains) { return 2 * chains <= sm_count(); }

// ---------------------------------------------------------------------------------------------------------
// The pre-pass of a cut call: state from zero and transition of a segment in ONE CTA, when there are more of them than SMs.  A chain of its own
// waits most of its 3.9 k cycles per step for its own operands, products and barriers (the tensor pipe is busy for 1.5 k, HBM at 3.6 TB/s);
// two side by side fill each other's gaps and share the nw^T and kbar tiles.  Eight warps per chain (thread = one lane x 64 columns).  Tensor
// memory has room for both because operands lie where the accumulators were read: 16 columns of an accumulator become the 8 + 8 columns of hi
// and lo halves of the same 16 terms, by the thread that read them.  Every sum is formed in the order of the single chain: the same bits.
// 32 k tokens x 32 heads (512 pairs of 32 steps) 450 -> 339 us, 64 k 980 -> 655.  With fewer chains than SMs both run at once anyway, 2.1 us per
// step instead of 2.7.
// ---------------------------------------------------------------------------------------------------------
namespace pr {
constexpr int THREADS = 640, WARP_MMA = 16, WARP_LOAD = 17, LAUNCH_REGS = 96, T = 32 * rc::KB;
constexpr int N = 0, K = 2 * T, U = 4 * T, TILES = 6 * T;
struct Shared {
    // One barrier per buffer (k & 1): its next phase needs the copy that the wait for this one releases, however late the copying thread comes.
    uint64_t fullN[2], fullK[2], fullU[2], uFree[2];
    uint64_t opS[2], opV[2], mm1[2][2], mm2[2][2];          // per chain: state operand | Vd operand written; products done
    uint32_t tmem;
    __align__(16) float gl[4][DK];
};
constexpr int SMEM = TILES + (int)sizeof(Shared);
static_assert(SMEM <= 232448, "shared memory of one CTA");
// accumulator columns: S and the state increment of chain c; D and V (two for the state, whose D starts as u^T)
__device__ __forceinline__ int sx(int c) { return 128 * c; }
__device__ __forceinline__ int dv(int c, int k) { return c ? 384 : 256 + 64 * (k & 1); }

// D (+)= A B^T with A as pairs of 8-column hi and lo groups
__device__ __forceinline__ void gemm_pairs(uint32_t tmem_d, uint32_t a, const umma::Opnd& b, int N_, int KT, uint32_t accumulate) {
    const uint32_t idesc = umma::idesc_bf16(128, N_, 0, b.mn);
    const uint64_t bh = umma::opnd_base_desc(b, b.hi), bl = umma::opnd_base_desc(b, b.lo);
#pragma unroll
    for (int ks = 0; ks < KT / 16; ++ks) {
        const uint32_t bo = umma::opnd_step16(b, ks), ah = a + 16 * ks, al = ah + 8;
        umma::mma_bf16_ta(tmem_d, al, bh + bo, idesc, accumulate);
        umma::mma_bf16_ta(tmem_d, ah, bl + bo, idesc, 1u);
        umma::mma_bf16_ta(tmem_d, ah, bh + bo, idesc, 1u);
        accumulate = 1u;
    }
}
// 16 values -> their hi and lo groups in the 16 columns at `taddr`
__device__ __forceinline__ void store_pairs(uint32_t taddr, const float* v) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) umma::split2(v[2 * i], v[2 * i + 1], h[i], l[i]);
    umma::tmem_st8(taddr, h);
    umma::tmem_st8(taddr + 8, l);
}
}  // namespace pr

__global__ void __launch_bounds__(pr::THREADS, 1) recur_fwd_pair_tc_kernel(const MkdaRecurFwd p, const int* seg_order) {
    using namespace pr;
    using umma::signal_tmem;
    using umma::wait_mma;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw;                              // no static shared memory: the dynamic block starts on a 1024-byte boundary
    Shared& sh = *reinterpret_cast<Shared*>(base + TILES);
    const int h = blockIdx.y, HV = p.L.HV;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (umma::smem_u32(base) & 1023) {                     // ... and nothing runs if that ever fails to hold
        follow_stream();
        if (tid == 0) atomicExch(&umma::g_timeout_flag, 1u);
        return;
    }
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            for (uint64_t* b : {&sh.fullN[i], &sh.fullK[i], &sh.fullU[i], &sh.mm1[0][i], &sh.mm1[1][i], &sh.mm2[0][i], &sh.mm2[1][i]}) umma::mbar_init(b, 1);
            for (uint64_t* b : {&sh.opS[i], &sh.opV[i], &sh.uFree[i]}) umma::mbar_init(b, 8);
        }
        umma::fence_barrier_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;
    follow_stream();
    const int seg = seg_order ? seg_order[blockIdx.z] : blockIdx.z;
    const int c_beg = p.L.seg_chunk_off[seg], n = p.L.seg_chunk_off[seg + 1] - c_beg;
    if (warp >= 16) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == WARP_LOAD) {
            if (umma::elect_one()) {
                auto tile = [&](int off, const float* t, int k, uint64_t* bar) {
                    umma::bulk_load(base + off + (k & 1) * T, reinterpret_cast<const uint8_t*>(t) + ((size_t)(c_beg + k) * HV + h) * umma::CHUNK_TILE_BYTES,
                                    umma::CHUNK_TILE_BYTES, bar);
                };
                auto load_n = [&](int k) {
                    if (k >= n) return;
                    umma::mbar_expect_tx(&sh.fullN[k & 1], umma::CHUNK_TILE_BYTES + DK * 4);
                    tile(N, p.nw, k, &sh.fullN[k & 1]);
                    umma::bulk_load(sh.gl[k & 3], p.gl + ((size_t)(c_beg + k) * HV + h) * DK, DK * 4, &sh.fullN[k & 1]);
                };
                auto load = [&](int off, const float* t, int k, uint64_t* bars) {
                    if (k >= n) return;
                    umma::mbar_expect_tx(&bars[k & 1], umma::CHUNK_TILE_BYTES);
                    tile(off, t, k, &bars[k & 1]);
                };
                for (int k = 0; k < 2; ++k) { load(U, p.u, k, sh.fullU); load_n(k); load(K, p.kbar, k, sh.fullK); }
                for (int k = 0; k < n; ++k) {              // each buffer is refilled as soon as both chains are done with it
                    umma::mbar_wait(&sh.uFree[k & 1], (k >> 1) & 1);
                    load(U, p.u, k + 2, sh.fullU);
                    umma::mbar_wait(&sh.mm1[1][k & 1], (k >> 1) & 1);
                    load_n(k + 2);
                    umma::mbar_wait(&sh.mm2[1][k & 1], (k >> 1) & 1);
                    load(K, p.kbar, k + 2, sh.fullK);
                }
            }
            __syncwarp();
        } else if (warp == WARP_MMA) {
            if (umma::elect_one()) {
                for (int k = 0; k < n; ++k) {
                    uint8_t *bn = base + N + (k & 1) * T, *bk = base + K + (k & 1) * T;
                    umma::mbar_wait(&sh.fullN[k & 1], (k >> 1) & 1);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        wait_mma(&sh.opS[c], k & 1);
                        gemm_pairs(tmem + dv(c, k), tmem + sx(c), umma::opnd_mn(bn, bn + 16384, 128), 64, 128, c ? 0u : 1u);
                        umma::commit(&sh.mm1[c][k & 1]);
                    }
                    umma::mbar_wait(&sh.fullK[k & 1], (k >> 1) & 1);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        wait_mma(&sh.opV[c], k & 1);
                        gemm_pairs(tmem + sx(c), tmem + dv(c, k), umma::opnd_mn(bk, bk + 16384, 64), 128, 64, 0u);
                        umma::commit(&sh.mm2[c][k & 1]);
                    }
                }
            }
            __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        const int c = warp >> 3, half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane, col = 64 * half;
        float s[64];                                       // columns col .. col + 63 of lane `row`
#pragma unroll
        for (int j = 0; j < 64; ++j) s[j] = c && col + j == row ? 1.f : 0.f;
        auto advance = [&](int k, int b) {                 // s <- s gl + increment of step k, 16 columns
            float x[16];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, sx(c) + col + 16 * b), x);
            const float* gl = &sh.gl[k & 3][col + 16 * b];
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const float4 f = *reinterpret_cast<const float4*>(gl + j);
                float* t = s + 16 * b + j;
                unpack2(fma2(pack2(t[0], t[1]), pack2(f.x, f.y), pack2(x[j], x[j + 1])), t[0], t[1]);
                unpack2(fma2(pack2(t[2], t[3]), pack2(f.z, f.w), pack2(x[j + 2], x[j + 3])), t[2], t[3]);
            }
        };
        auto preload_u = [&](int k) {                      // u^T of step k into the accumulator that its first product adds to
            umma::mbar_wait(&sh.fullU[k & 1], (k >> 1) & 1);
            const uint8_t* u = base + U + (k & 1) * T;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float a[8];
                umma::load_tile8(u, u + 16384, 128, row, 4 * half + i, a);
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(a[e]);
                umma::tmem_st8(umma::tmem_addr(tmem, warp, dv(0, k) + 32 * half + 8 * i), w);
            }
            umma::tmem_wait_st();
            signal_tmem(&sh.uFree[k & 1], lane);
        };
        if (c == 0 && n > 0) preload_u(0);
        for (int k = 0; k < n; ++k) {
            umma::mbar_wait(&sh.fullN[k & 1], (k >> 1) & 1);           // this thread reads the decay factors that come with nw^T
            if (k) wait_mma(&sh.mm2[c][(k - 1) & 1], ((k - 1) >> 1) & 1);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (k) advance(k - 1, b);
                store_pairs(umma::tmem_addr(tmem, warp, sx(c) + col + 16 * b), s + 16 * b);
            }
            umma::tmem_wait_st();
            signal_tmem(&sh.opS[c], lane);
            wait_mma(&sh.mm1[c][k & 1], (k >> 1) & 1);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                float d[16];
                const uint32_t at = umma::tmem_addr(tmem, warp, dv(c, k) + 32 * half + 16 * b);
                umma::tmem_ld16(at, d);
                store_pairs(at, d);
            }
            umma::tmem_wait_st();
            signal_tmem(&sh.opV[c], lane);
            if (c == 0 && k + 1 < n) preload_u(k + 1);
        }
        if (n > 0) {
            wait_mma(&sh.mm2[c][(n - 1) & 1], ((n - 1) >> 1) & 1);
#pragma unroll
            for (int b = 0; b < 4; ++b) advance(n - 1, b);
        }
        // transition: M[K out][K in] with this thread holding row `row` = K in; state: [K][V] or [V][K]
        float* dst = nullptr;
        if (c) {
            dst = p.mt + ((size_t)seg * HV + h) * DK * DK;
        } else if (p.ht) {
            const int r = p.seg_ht ? p.seg_ht[seg] : seg;
            if (r >= 0) dst = p.ht + ((size_t)r * HV + h) * DK * DV;
        }
        if (dst) {
            const bool vf = !c && p.state_v_first;
#pragma unroll
            for (int j = 0; j < 64; ++j) dst[vf ? (size_t)row * DK + col + j : (size_t)(col + j) * DV + row] = s[j];
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

int launch_recur_fwd_tc(const MkdaRecurFwd* p, const int* seg_order, cudaStream_t stream) {
    if (p->want_transition && !p->h && !p->Vd && !p->h0 && !p->warm_start && 2ll * p->L.HV * p->L.NS > sm_count()) {
        auto pair = recur_fwd_pair_tc_kernel;
        if (int e = ensure_smem((const void*)pair, pr::SMEM, "recur_fwd")) return e;
        static const int regs = kernel_registers((const void*)pair);
        if (regs < pr::LAUNCH_REGS) return set_error(MKDA_ERR_LAUNCH, "recur_fwd: built with fewer registers than its warps redistribute");
        launch(pair, dim3(1, p->L.HV, p->L.NS), pr::THREADS, pr::SMEM, stream, *p, seg_order);
        return check_launch("recur_fwd");
    }
    using L = RecurLayout<false>;
    const int per_segment = p->want_transition ? 2 : 1;
    const bool split = split_chains((long long)per_segment * p->L.HV * p->L.NS);
    auto kern = split ? recur_fwd_tc_kernel<true> : recur_fwd_tc_kernel<false>;
    if (int e = ensure_smem((const void*)kern, L::SMEM, "recur_fwd")) return e;
    launch(kern, dim3(split ? 2 * per_segment : per_segment, p->L.HV, p->L.NS), L::THREADS, L::SMEM, stream, *p, seg_order);
    return check_launch("recur_fwd");
}

template <int OUT, bool NORM>
static int launch_chain_fwd_tc_n(const MkdaChainFwd* p, const int* seg_order, cudaStream_t stream) {
    using L = RecurLayout<true>;
    auto kern = chain_fwd_tc_kernel<OUT, NORM>;
    if (int e = ensure_smem((const void*)kern, L::SMEM, "chain_fwd")) return e;
    static const int regs = kernel_registers((const void*)kern);
    if (regs < L::REGS) return set_error(MKDA_ERR_LAUNCH, "chain_fwd: built with fewer registers than its warps redistribute");
    ChainMaps maps;
    memset(&maps, 0, sizeof(maps));
    const unsigned long long rows = (unsigned long long)p->o.L.TT, cols = (unsigned long long)p->o.L.HV * 128;
    int e = 0;
    if (NORM && OUT != MKDA_F32) e = make_rows_map(&maps.gate, p->o.gate, 2, rows, cols, "chain_fwd");
    if (!e && p->o.o_raw) e = make_rows_map(&maps.raw, p->o.o_raw, 4, rows, cols, "chain_fwd", 16);
    if (!e) e = make_rows_map(&maps.out, p->o.out, p->o.out_dtype == MKDA_F32 ? 4 : 2, rows, cols, "chain_fwd", 16);
    if (e) return e;
    launch(kern, dim3(1, p->r.L.HV, p->r.L.NS), L::THREADS, L::SMEM, stream, *p, seg_order, maps);
    return check_launch("chain_fwd");
}
template <int OUT>
static int launch_chain_fwd_tc_t(const MkdaChainFwd* p, const int* seg_order, cudaStream_t stream) {
    return p->o.has_norm ? launch_chain_fwd_tc_n<OUT, true>(p, seg_order, stream) : launch_chain_fwd_tc_n<OUT, false>(p, seg_order, stream);
}
int launch_chain_fwd_tc(const MkdaChainFwd* p, const int* seg_order, cudaStream_t stream) {
    switch (p->o.has_norm ? p->o.gate_dtype : p->o.out_dtype) {
        case MKDA_F32: return launch_chain_fwd_tc_t<MKDA_F32>(p, seg_order, stream);
        case MKDA_BF16: return launch_chain_fwd_tc_t<MKDA_BF16>(p, seg_order, stream);
        case MKDA_F16: return launch_chain_fwd_tc_t<MKDA_F16>(p, seg_order, stream);
    }
    return set_error(MKDA_ERR_ARG, "chain_fwd: unsupported dtype");
}

// ---------------------------------------------------------------------------------------------------------
// reverse: dS is the gradient of the state leaving the current chunk, walking backwards.  Per step the products are issued in the order
//   D = dO^T Aqk (ahead of the step) | D += dS^T kbar^T | X = dO^T (scale q 2^g) | X += dVd^T nw
// so that the two that do not depend on the chain run where the tensor pipe would wait for an operand.
// ---------------------------------------------------------------------------------------------------------
struct DhShared {
    uint64_t fullA[2], fullK, fullN;                       // dO, Aqk, scale q 2^g and decay factors | kbar | nw^T landed
    uint64_t opS, opV, mm1, mm2;
    uint32_t tmem;
    __align__(16) float gl[4][DK];
};
constexpr int DH_SET = 80 * rc::KB;                        // dO 32, scale q 2^g 32, Aqk 16
constexpr int DH_K = 2 * DH_SET, DH_N = DH_K + 32 * rc::KB, DH_TILES = DH_N + 32 * rc::KB;
constexpr int DH_SMEM = DH_TILES + (int)sizeof(DhShared);
static_assert(DH_SMEM <= 232448, "shared memory of one CTA");

// R = CUtensorMap: dO as bf16 rows, which are an operand as they stand, exact and without a low half.  A full chunk's are fetched from where they are (boxes of
// 64 columns in the layout of an operand tile); only chunks with rows past their end, which have to be zeros, come as tiles.  A third less products with dO, half
// of its bytes, and no pass that writes tiles: one document of 64 k tokens x 32 heads 238 us of that pass and 1930 -> 1800 us (both chains), 4 x 16 k tokens x
// 16 heads with a scalar gate 120 us and 707 -> 683.
struct NoRows {};
template <bool SPLIT, class R>
__global__ void __launch_bounds__(rc::THREADS, 1) bwd_dh_tc_kernel(const MkdaBwdDh p, const int* seg_order, const __grid_constant__ R rows) {
    using namespace rc;
    constexpr bool ROWS = std::is_same<R, CUtensorMap>::value;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw;                              // no static shared memory: the dynamic block starts on a 1024-byte boundary
    DhShared& sh = *reinterpret_cast<DhShared*>(base + DH_TILES);
    const int h = blockIdx.y, HV = p.L.HV, v0 = SPLIT ? 64 * blockIdx.x : 0;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (umma::smem_u32(base) & 1023) {                     // ... and nothing runs if that ever fails to hold
        follow_stream();
        if (tid == 0) atomicExch(&umma::g_timeout_flag, 1u);
        return;
    }
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (tid == 0) {
        for (uint64_t* b : {&sh.fullA[0], &sh.fullA[1], &sh.fullK, &sh.fullN, &sh.mm1, &sh.mm2}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opS, &sh.opV}) umma::mbar_init(b, SPLIT ? COMPUTE / 64 : COMPUTE / 32);
        umma::fence_barrier_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;
    follow_stream();
    const int seg = seg_order ? seg_order[blockIdx.z] : blockIdx.z;

    // Warm-up truncation (a pass from zero only): the reverse chain starts below chunk warm_end where the decay accumulated
    // over the segment's first chunks hides every later contribution from the segment's entrance.
    const int c_beg = p.L.seg_chunk_off[seg];
    int c_end = p.L.seg_chunk_off[seg + 1];
    bool cut = false;
    if (p.warm_end) {
        const int w = p.warm_end[seg * HV + h];
        if (w < c_end) { cut = true; c_end = w; }
    }
    const int n = c_end - c_beg;
    auto item = [&](int k) { return (size_t)(c_end - 1 - k) * HV + h; };

    if (warp == WARP_LOAD) {
        if (umma::elect_one()) {
            auto load = [&](int off, const float* t, size_t it, uint32_t bytes, uint64_t* bar) {
                umma::bulk_load(base + off, reinterpret_cast<const uint8_t*>(t) + it * bytes, bytes, bar);
            };
            int start = 0, len = 0;                        // of the next set's chunk, read a step ahead
            auto look = [&](int k) {
                if (!ROWS || k >= n) return;
                start = p.L.chunk_start[c_end - 1 - k]; len = p.L.chunk_len[c_end - 1 - k];
            };
            auto set_a = [&](int k) {
                uint64_t* bar = &sh.fullA[k & 1];
                umma::mbar_expect_tx(bar, (ROWS ? (SPLIT ? 5 : 6) : (SPLIT ? 6 : 8)) * umma::CHUNK_TILE_BYTES / 4 + umma::QUARTER_TILE_BYTES + DK * 4);
                if constexpr (ROWS) {
                    uint8_t* dst = base + (k & 1) * DH_SET;
                    if (len == CH || !p.dO_in_t) {
                        umma::tma_load_rows(dst, &rows, h * 128 + v0, start, bar);
                        if (!SPLIT) umma::tma_load_rows(dst + 8192, &rows, h * 128 + 64, start, bar);
                    } else {
                        umma::bulk_load(dst, reinterpret_cast<const uint8_t*>(p.dO_in_t) + item(k) * umma::CHUNK_TILE_BYTES + 128 * v0, SPLIT ? 8192 : 16384, bar);
                    }
                    look(k + 1);
                } else if (SPLIT) {                               // one 64-column block of the hi and of the lo tile; the products read the other block unloaded:
                    const uint8_t* src = reinterpret_cast<const uint8_t*>(p.dO_in_t) + item(k) * umma::CHUNK_TILE_BYTES + 128 * v0;
                    umma::bulk_load(base + (k & 1) * DH_SET, src, 8192, bar);              // accumulator lanes that nobody looks at
                    umma::bulk_load(base + (k & 1) * DH_SET + 16384, src + 16384, 8192, bar);
                } else {
                    load((k & 1) * DH_SET, p.dO_in_t, item(k), umma::CHUNK_TILE_BYTES, bar);
                }
                load((k & 1) * DH_SET + 65536, p.Aqk, item(k), umma::QUARTER_TILE_BYTES, bar);
                load((k & 1) * DH_SET + 32768, p.qs, item(k), umma::CHUNK_TILE_BYTES, bar);
                umma::bulk_load(sh.gl[k & 3], p.gl + item(k) * DK, DK * 4, bar);
            };
            auto one = [&](int off, const float* t, int k, uint64_t* bar) {
                umma::mbar_expect_tx(bar, umma::CHUNK_TILE_BYTES);
                load(off, t, item(k), umma::CHUNK_TILE_BYTES, bar);
            };
            look(0);
            if (n > 0) { set_a(0); one(DH_K, p.kbar, 0, &sh.fullK); one(DH_N, p.nw, 0, &sh.fullN); }
            if (n > 1) set_a(1);
            for (int k = 0; k + 1 < n; ++k) {              // each buffer is refilled as soon as its product is done
                umma::mbar_wait(&sh.mm1, k & 1);
                one(DH_K, p.kbar, k + 1, &sh.fullK);
                umma::mbar_wait(&sh.mm2, k & 1);
                one(DH_N, p.nw, k + 1, &sh.fullN);
                if (k + 2 < n) set_a(k + 2);
            }
        }
        __syncwarp();
    } else if (warp == WARP_MMA) {
        if (umma::elect_one()) {
            auto dO_mn = [&](int k) { uint8_t* t = base + (k & 1) * DH_SET; return umma::opnd_mn(t, ROWS ? nullptr : t + 16384, 64); };
            auto ahead = [&](int k) {
                uint8_t* t = base + (k & 1) * DH_SET + 65536;
                umma::mbar_wait(&sh.fullA[k & 1], (k >> 1) & 1);
                umma::gemm<true>(tmem + D0, dO_mn(k), umma::opnd_mn(t, t + 8192, 64), 128, 64, 64, 0u);
            };
            if (n > 0) ahead(0);
            for (int k = 0; k < n; ++k) {
                umma::mbar_wait(&sh.fullK, k & 1);
                wait_mma(&sh.opS, k & 1);
                umma::gemm_ta(tmem + D0, tmem + SH, tmem + SL, umma::opnd_k(base + DH_K, base + DH_K + 16384, 64), 64, 128, 1u);
                umma::commit(&sh.mm1);
                uint8_t* qs = base + (k & 1) * DH_SET + 32768;
                umma::gemm<true>(tmem + X, dO_mn(k), umma::opnd_mn(qs, qs + 16384, 64), 128, 128, 64, 0u);
                umma::mbar_wait(&sh.fullN, k & 1);
                wait_mma(&sh.opV, k & 1);
                umma::gemm_ta(tmem + X, tmem + VH, tmem + VL, umma::opnd_k(base + DH_N, base + DH_N + 16384, 128), 128, 64, 1u);
                umma::commit(&sh.mm2);
                if (k + 1 < n) ahead(k + 1);
            }
        }
        __syncwarp();
    } else if (!SPLIT || (warp & 3) < 2) {
        const int cg = warp >> 2, row = v0 + (warp & 3) * 32 + lane;
        const bool vf = p.state_v_first != 0;
        float s[32];
        const int drow = p.seg_dht ? p.seg_dht[seg] : seg;
        if (p.dht && drow >= 0 && !cut) {
            load_state(p.dht + ((size_t)drow * HV + h) * DK * DV, vf, row, cg, s);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) s[j] = 0.f;
        }
        auto advance = [&](int k) {                        // the state step k leaves behind
            wait_mma(&sh.mm2, k & 1);
            advance_state(umma::tmem_addr(tmem, warp, X + cg * 32), &sh.gl[k & 3][cg * 32], s);
        };
        for (int k = 0; k < n; ++k) {
            if (k) advance(k - 1);
            {
                uint32_t hi[16], lo[16];
                state_operand(tmem, warp, cg, s, hi, lo);
                signal_tmem(&sh.opS, lane);
                if (p.dh) save_state_tile(reinterpret_cast<uint8_t*>(p.dh) + item(k) * umma::STATE_TILE_BYTES, row, cg, hi, lo);
            }
            umma::mbar_wait(&sh.fullA[k & 1], (k >> 1) & 1);           // its decay factors are read by this thread
            wait_mma(&sh.mm1, k & 1);
            {
                uint32_t hi[8], lo[8];
                v_operand(tmem, D0, warp, cg, hi, lo);
                signal_tmem(&sh.opV, lane);
                // dVd^T leaves as a chunk tile (token columns past the end are exact zeros: Aqk has no such column and kbar no such row)
                if (p.dVd_t) {
                    uint8_t* tile = reinterpret_cast<uint8_t*>(p.dVd_t) + item(k) * umma::CHUNK_TILE_BYTES;
                    store_pair(tile, 128, row, 2 * cg, hi);
                    store_pair(tile + 16384, 128, row, 2 * cg, lo);
                }
            }
        }
        if (n > 0) advance(n - 1);
        if (p.dh0) store_state(p.dh0 + ((size_t)seg * HV + h) * DK * DV, vf, row, cg, s);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

template <class R>
static int launch_bwd_dh_tc_r(const MkdaBwdDh* p, const int* seg_order, const R& rows, cudaStream_t stream) {
    const bool split = split_chains((long long)p->L.HV * p->L.NS);
    auto kern = split ? bwd_dh_tc_kernel<true, R> : bwd_dh_tc_kernel<false, R>;
    if (int e = ensure_smem((const void*)kern, DH_SMEM, "bwd_dh")) return e;
    launch(kern, dim3(split ? 2 : 1, p->L.HV, p->L.NS), rc::THREADS, DH_SMEM, stream, *p, seg_order, rows);
    return check_launch("bwd_dh");
}
int launch_bwd_dh_tc(const MkdaBwdDh* p, const int* seg_order, bool rows, cudaStream_t stream) {
    if (!rows) return launch_bwd_dh_tc_r(p, seg_order, NoRows{}, stream);
    CUtensorMap map;
    if (int e = make_rows_map(&map, p->d_o, 2, (unsigned long long)p->L.TT, (unsigned long long)p->L.HV * 128, "bwd_dh", CH, 64)) return e;
    return launch_bwd_dh_tc_r(p, seg_order, map, stream);
}

int tc_recur_status(unsigned int* out) {
    return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1;
}
int tc_recur_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

}  // namespace mkda
