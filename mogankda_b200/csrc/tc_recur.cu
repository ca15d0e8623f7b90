// Serial state recurrences on the Blackwell tensor cores.
//
// One CTA per (v-head, segment) carries the whole 128 x 128 state, TRANSPOSED: accumulator lane = v, columns = K index.  The fp32 state
// lives in the registers of 512 compute threads (thread = one lane x 32 columns); each step it is split into packed bf16 hi / lo pairs in
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
#include "common.cuh"
#include "host.h"
#include "umma.cuh"

namespace mkda {

namespace rc {
constexpr int COMPUTE = 512, THREADS = 576, WARP_MMA = 16, WARP_LOAD = 17;
constexpr int KB = 1024;
constexpr int SH = 128, SL = 192, VH = 448, VL = 480;      // tensor-memory columns of the left operands (hi, lo)
constexpr int X = 0, D0 = 256, D1 = 320;                   // fp32 accumulators: state increment, D (two for the forward kernel)

using umma::signal_tmem;
using umma::wait_mma;

// 32 bytes to global memory in one piece
__device__ __forceinline__ void st32b(void* dst, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
__device__ __forceinline__ void ld32b(const void* src, float* v) {
    uint32_t w[8];
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(src));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
}
// Two neighbouring 16-byte chunks k8, k8 + 1 (k8 even) of row r of an operand tile: they fill one aligned 32-byte piece, in an order that
// the swizzle takes from the row's parity.
__device__ __forceinline__ void store_pair(uint8_t* tile, int R, int r, int k8, const uint32_t* w) {
    uint32_t o[8];
    const bool odd = r & 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) { o[i] = odd ? w[4 + i] : w[i]; o[4 + i] = odd ? w[i] : w[4 + i]; }
    st32b(tile + (umma::tile_chunk_offset(R, r, k8) & ~16u), o);
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
            s[j] = fmaf(s[j], f.x, x[j4]); s[j + 1] = fmaf(s[j + 1], f.y, x[j4 + 1]);
            s[j + 2] = fmaf(s[j + 2], f.z, x[j4 + 2]); s[j + 3] = fmaf(s[j + 3], f.w, x[j4 + 3]);
        }
    }
}
// the state as the left operand of the next products
__device__ __forceinline__ void state_operand(uint32_t tmem, int warp, int cg, const float (&s)[32], uint32_t (&h)[16], uint32_t (&l)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) umma::split2(s[2 * i], s[2 * i + 1], h[i], l[i]);
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
// forward
// ---------------------------------------------------------------------------------------------------------
struct RecurShared {
    uint64_t full[2];                                      // nw^T, kbar, u^T tiles and decay factors of a step landed
    uint64_t opS, opV, mm1, mm2;                           // state operand | Vd operand written; first | second product done
    uint32_t tmem;
    __align__(16) float gl[4][DK];                         // four deep: a step's factors are used at the start of the next one
};
constexpr int RECUR_BUF = 96 * rc::KB;                     // nw 32, kbar 32, u 32
constexpr int RECUR_SMEM = 2 * RECUR_BUF + (int)sizeof(RecurShared) + 1024;

__global__ void __launch_bounds__(rc::THREADS, 1) recur_fwd_tc_kernel(const MkdaRecurFwd p) {
    using namespace rc;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    RecurShared& sh = *reinterpret_cast<RecurShared*>(base + 2 * RECUR_BUF);
    const bool trans = blockIdx.x == 1;
    const int h = blockIdx.y, seg = blockIdx.z, HV = p.L.HV;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (tid == 0) {
        for (uint64_t* b : {&sh.full[0], &sh.full[1], &sh.mm1, &sh.mm2}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opS, &sh.opV}) umma::mbar_init(b, COMPUTE / 32);
        umma::fence_barrier_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;

    // Warm-up truncation (a pass from zero only): where the decay accumulated from chunk warm_start to the segment's end
    // hides everything before it, the pass starts there; the transition is then zero and its CTA visits no chunk.
    int c_beg = p.L.seg_chunk_off[seg];
    const int c_end = p.L.seg_chunk_off[seg + 1];
    bool cut = false;
    if (p.warm_start) {
        const int w = p.warm_start[seg * HV + h];
        if (w > c_beg) { cut = true; c_beg = trans ? c_end : w; }
    }
    const int n = c_end - c_beg;

    if (warp == WARP_LOAD) {
        if (umma::elect_one()) {
            for (int k = 0; k < n; ++k) {
                if (k >= 2) umma::mbar_wait(&sh.mm2, k & 1);          // step k - 2 is done with its buffer
                const size_t it = (size_t)(c_beg + k) * HV + h;
                uint8_t* buf = base + (k & 1) * RECUR_BUF;
                uint64_t* bar = &sh.full[k & 1];
                umma::mbar_expect_tx(bar, (trans ? 2 : 3) * umma::CHUNK_TILE_BYTES + DK * 4);
                umma::bulk_load(buf, reinterpret_cast<const uint8_t*>(p.nw) + it * umma::CHUNK_TILE_BYTES, umma::CHUNK_TILE_BYTES, bar);
                umma::bulk_load(buf + 32768, reinterpret_cast<const uint8_t*>(p.kbar) + it * umma::CHUNK_TILE_BYTES, umma::CHUNK_TILE_BYTES, bar);
                umma::bulk_load(sh.gl[k & 3], p.gl + it * DK, DK * 4, bar);
                if (!trans) umma::bulk_load(buf + 65536, reinterpret_cast<const uint8_t*>(p.u) + it * umma::CHUNK_TILE_BYTES, umma::CHUNK_TILE_BYTES, bar);
            }
        }
        __syncwarp();
    } else if (warp == WARP_MMA) {
        if (umma::elect_one()) {
            for (int k = 0; k < n; ++k) {
                const uint8_t* buf = base + (k & 1) * RECUR_BUF;
                umma::mbar_wait(&sh.full[k & 1], (k >> 1) & 1);
                wait_mma(&sh.opS, k & 1);
                umma::gemm_ta(tmem + ((k & 1) ? D1 : D0), tmem + SH, tmem + SL, umma::opnd_mn(buf, buf + 16384, 128), 64, 128, trans ? 0u : 1u);
                umma::commit(&sh.mm1);
                wait_mma(&sh.opV, k & 1);
                umma::gemm_ta(tmem + X, tmem + VH, tmem + VL, umma::opnd_mn(buf + 32768, buf + 49152, 64), 128, 64, 0u);
                umma::commit(&sh.mm2);
            }
        }
        __syncwarp();
    } else {
        const int cg = warp >> 2, row = (warp & 3) * 32 + lane;
        const bool vf = p.state_v_first != 0;
        float s[32];
        const int h0row = p.seg_h0 ? p.seg_h0[seg] : seg;
        if (!trans && !cut && p.h0 && h0row >= 0) {
            load_state(p.h0 + ((size_t)h0row * HV + h) * DK * DV, vf && !p.h0_k_first, row, cg, s);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) s[j] = trans && !cut && cg * 32 + j == row ? 1.f : 0.f;
        }
        // u^T of step k into the accumulator that its first product adds to
        auto preload_u = [&](int k) {
            umma::mbar_wait(&sh.full[k & 1], (k >> 1) & 1);
            if (trans) return;
            const uint8_t* u = base + (k & 1) * RECUR_BUF + 65536;
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
        };
        if (n > 0) preload_u(0);
        for (int k = 0; k < n; ++k) {
            const size_t it = (size_t)(c_beg + k) * HV + h;
            if (k) {
                wait_mma(&sh.mm2, (k - 1) & 1);
                advance_state(umma::tmem_addr(tmem, warp, X + cg * 32), &sh.gl[(k - 1) & 3][cg * 32], s);
            }
            {
                uint32_t hi[16], lo[16];
                state_operand(tmem, warp, cg, s, hi, lo);
                signal_tmem(&sh.opS, lane);
                if (p.h && !trans) save_state_tile(reinterpret_cast<uint8_t*>(p.h) + it * umma::STATE_TILE_BYTES, row, cg, hi, lo);
            }
            wait_mma(&sh.mm1, k & 1);
            {
                uint32_t hi[8], lo[8];
                v_operand(tmem, (k & 1) ? D1 : D0, warp, cg, hi, lo);
                signal_tmem(&sh.opV, lane);
                if (p.Vd && !trans) {
                    uint8_t* tile = reinterpret_cast<uint8_t*>(p.Vd) + it * umma::CHUNK_TILE_BYTES;
                    store_pair(tile, 128, row, 2 * cg, hi);
                    store_pair(tile + 16384, 128, row, 2 * cg, lo);
                }
            }
            if (k + 1 < n) preload_u(k + 1);
        }
        if (n > 0) {
            wait_mma(&sh.mm2, (n - 1) & 1);
            advance_state(umma::tmem_addr(tmem, warp, X + cg * 32), &sh.gl[(n - 1) & 3][cg * 32], s);
        }
        // transition: M[K out][K in] with this thread holding row `row` = K in; state: [K][V] or [V][K]
        if (trans) {
            if (p.mt) store_state(p.mt + ((size_t)seg * HV + h) * DK * DK, false, row, cg, s);
        } else if (p.ht) {
            const int r = p.seg_ht ? p.seg_ht[seg] : seg;
            if (r >= 0) store_state(p.ht + ((size_t)r * HV + h) * DK * DV, vf, row, cg, s);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

int launch_recur_fwd_tc(const MkdaRecurFwd* p, cudaStream_t stream) {
    auto kern = recur_fwd_tc_kernel;
    if (int e = ensure_smem((const void*)kern, RECUR_SMEM, "recur_fwd")) return e;
    kern<<<dim3(p->want_transition ? 2 : 1, p->L.HV, p->L.NS), rc::THREADS, RECUR_SMEM, stream>>>(*p);
    return check_launch("recur_fwd");
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

__global__ void __launch_bounds__(rc::THREADS, 1) bwd_dh_tc_kernel(const MkdaBwdDh p) {
    using namespace rc;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw;                              // no static shared memory: the dynamic block starts on a 1024-byte boundary
    DhShared& sh = *reinterpret_cast<DhShared*>(base + DH_TILES);
    const int h = blockIdx.y, seg = blockIdx.z, HV = p.L.HV;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (umma::smem_u32(base) & 1023) {                     // ... and nothing runs if that ever fails to hold
        if (tid == 0) atomicExch(&umma::g_timeout_flag, 1u);
        return;
    }
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (tid == 0) {
        for (uint64_t* b : {&sh.fullA[0], &sh.fullA[1], &sh.fullK, &sh.fullN, &sh.mm1, &sh.mm2}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opS, &sh.opV}) umma::mbar_init(b, COMPUTE / 32);
        umma::fence_barrier_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;

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
            auto set_a = [&](int k) {
                uint64_t* bar = &sh.fullA[k & 1];
                umma::mbar_expect_tx(bar, 2 * umma::CHUNK_TILE_BYTES + umma::QUARTER_TILE_BYTES + DK * 4);
                load((k & 1) * DH_SET, p.dO_in_t, item(k), umma::CHUNK_TILE_BYTES, bar);
                load((k & 1) * DH_SET + 65536, p.Aqk, item(k), umma::QUARTER_TILE_BYTES, bar);
                load((k & 1) * DH_SET + 32768, p.qs, item(k), umma::CHUNK_TILE_BYTES, bar);
                umma::bulk_load(sh.gl[k & 3], p.gl + item(k) * DK, DK * 4, bar);
            };
            auto one = [&](int off, const float* t, int k, uint64_t* bar) {
                umma::mbar_expect_tx(bar, umma::CHUNK_TILE_BYTES);
                load(off, t, item(k), umma::CHUNK_TILE_BYTES, bar);
            };
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
            auto dO_mn = [&](int k) { uint8_t* t = base + (k & 1) * DH_SET; return umma::opnd_mn(t, t + 16384, 64); };
            auto ahead = [&](int k) {
                uint8_t* t = base + (k & 1) * DH_SET + 65536;
                umma::mbar_wait(&sh.fullA[k & 1], (k >> 1) & 1);
                umma::gemm(tmem + D0, dO_mn(k), umma::opnd_mn(t, t + 8192, 64), 128, 64, 64, 0u);
            };
            if (n > 0) ahead(0);
            for (int k = 0; k < n; ++k) {
                umma::mbar_wait(&sh.fullK, k & 1);
                wait_mma(&sh.opS, k & 1);
                umma::gemm_ta(tmem + D0, tmem + SH, tmem + SL, umma::opnd_k(base + DH_K, base + DH_K + 16384, 64), 64, 128, 1u);
                umma::commit(&sh.mm1);
                uint8_t* qs = base + (k & 1) * DH_SET + 32768;
                umma::gemm(tmem + X, dO_mn(k), umma::opnd_mn(qs, qs + 16384, 64), 128, 128, 64, 0u);
                umma::mbar_wait(&sh.fullN, k & 1);
                wait_mma(&sh.opV, k & 1);
                umma::gemm_ta(tmem + X, tmem + VH, tmem + VL, umma::opnd_k(base + DH_N, base + DH_N + 16384, 128), 128, 64, 1u);
                umma::commit(&sh.mm2);
                if (k + 1 < n) ahead(k + 1);
            }
        }
        __syncwarp();
    } else {
        const int cg = warp >> 2, row = (warp & 3) * 32 + lane;
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

int launch_bwd_dh_tc(const MkdaBwdDh* p, cudaStream_t stream) {
    auto kern = bwd_dh_tc_kernel;
    if (int e = ensure_smem((const void*)kern, DH_SMEM, "bwd_dh")) return e;
    kern<<<dim3(1, p->L.HV, p->L.NS), rc::THREADS, DH_SMEM, stream>>>(*p);
    return check_launch("bwd_dh");
}

int tc_recur_status(unsigned int* out) {
    return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1;
}
int tc_recur_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

}  // namespace mkda
