// Intra-chunk forward kernel on the Blackwell tensor cores: WY preparation.  A persistent CTA per SM walks the (chunk, v-head) items.
//
//   Gamma_ij = sum_c k_ic k_jc 2^(g_ic - g_jc)  (i > j)        Aqk_ij = scale sum_c q_ic k_jc 2^(g_ic - g_jc)  (i >= j)
//   A  = (I + strictlower(diag(beta) Gamma))^-1
//   nw = -A diag(beta) (k 2^g)                                  u = A diag(beta) v
//
// Range / prefix invariance: the per-channel decay 2^(g_i - g_j) does not factor out of the contraction over channels,
// so each 16-row block I uses its first row a = 16 I as anchor: row operand k_i 2^(g_i - g_a) (<= 1), column operand
// k_j 2^(g_a - g_j) (<= |k| for j < a, <= 2^(15*5/ln2) |k| = 2^108 |k| inside the diagonal block).  An output element (i, j) therefore
// depends on rows i, j and a <= i only, never on later rows.  The rows are staged as they come, the L2 scales applied to what comes out, so |k|
// is whatever the caller's scale is: 2^48 goes from the column to the row operands (exact, and nothing in range changes by it), which leaves room
// for every row whose sum of squares is finite and keeps the low halves of small rows out of the subnormals.  Rows past the end of the sequence are staged as zeros
// (their g as the last valid row's), so they produce identity rows in A and are never stored.
//   row operand     Kr[i] = k_i 2^(48 + g_i - g_a(i)),  Qr[i] = q_i 2^(48 + g_i - g_a(i))      one tile for all 64 rows
//   column operand  Kc_I[j] = k_j 2^(g_aI - g_j - 48),  j < 16 (I + 1)                         one tile per row block
//
// What bounds it: the phases of an item depend on each other, and only one item's operands (144 KB) fit.  So the phases are split between two
// groups of warps that work on neighbouring items:
//   X, 16 warps, item n + 1: rows in -> operands -> (while [Gamma; Q K^T] is computed) L2 scales; nw, u of item n from their accumulators ->
//                            kbar, scale q 2^g and beta k 2^g tiles
//   Y, 8 warps, item n:      I + L and Aqk from the accumulators -> inverse (a chain of latencies that used to hold up 16 warps) -> A, beta v
// and four warps of one working thread each: products of X, products of Y, copies of X, copies of Y.  All are joined by mbarriers.
// beta goes to v and k 2^g and not into A, whose diagonal stays exact.  With A diag(beta) as the operand a bf16 v would be one as it stands and take a
// product less per k-step (6 to 12 % of the kernel), but a rounded beta on the diagonal is an error that all 128 values of a row have in common:
// dh0 1.03 times as far from fp64 (geometric mean of 90 bf16 layers; 1.4 at worst), fp32 gradients 1.08, final states 1.2.
// An item takes 16 k cycles, all of them X's (rows 3 k, operands 5 k, L2 statistics 1.5 k, nw and u 2.9 k, tiles 3 k), 11 k of them Y's; 12 k with a scalar gate, Y's.
// 6 k packed tokens x 32 heads 240 -> 190 us, 32 k tokens x 32 heads 1121 -> 860, scalar gate 4 x 2000 tokens x 16 heads 129 -> 99.
#include "gate.cuh"
#include "host.h"
#include "intra.cuh"

#include <string.h>
#include <type_traits>

namespace mkda {

namespace in {
// Eight warps of Y: the latency of its phases is what an item takes, also where X keeps shared memory busy.  Eight against four, per-channel gate, from 0.2 to
// 220 items per SM: 3 to 12 % faster throughout, bf16, fp16 and fp32 (bf16 6 k packed tokens x 32 heads 219 -> 190 us, 32 k tokens 1005 -> 860).
constexpr int X_WARPS = 16, Y_WARPS = 8, COPY_X = 1, THREADS = 32 * (X_WARPS + Y_WARPS + 4);
// registers of the launch (Y keeps them), of X and of the last four warps
constexpr int LAUNCH_REGS = 72, X_REGS = 80, ISSUE_REGS = 40;
static_assert(X_WARPS * X_REGS + Y_WARPS * LAUNCH_REGS + 4 * ISSUE_REGS <= (X_WARPS + Y_WARPS + 4) * LAUNCH_REGS, "registers of the launch");
constexpr float ROW_UP = 0x1p48f, COL_DOWN = 0x1p-48f;      // column operand: 108 + 64 - 48 < 127, row operand: 64 + 48 < 127 for |k| < 2^64
// the four column tiles stacked by rows into one 160-row tile (hi 40 KB, then lo)
__host__ __device__ constexpr int kc_row(int I) { return 8 * I * (I + 1); }
constexpr int KC_ROWS = 160, KC_BYTES = KC_ROWS * 128 * 2;  // one of hi / lo
constexpr int KQ = 2 * KC_BYTES;                            // [Kr; Qr] [128][128]: hi 32 KB, lo 32 KB
// Over both once their products are done: the hand-over tiles kbar, scale q 2^g and Aqk of the item over the column tiles (written last, half
// 0 in front of Aqk), the rows of the next one (dense [64][128] blocks) over [Kr; Qr].  fp32 rows do not fit: q waits until kbar has left.
constexpr int KB = 0, QS = 32768, AQ = 65536, RAW_G = KQ;
template <int DT, bool SCALAR>
struct Rows {
    static constexpr int BYTES = DT == MKDA_F32 ? 32768 : 16384, PITCH = BYTES / CH;
    static constexpr bool LATE_Q = DT == MKDA_F32 && !SCALAR;
    static constexpr int K = SCALAR ? KQ : KQ + 32768, Q = LATE_Q ? KB : K + BYTES;
    static_assert(LATE_Q || Q + BYTES <= KQ + 65536, "rows of the next item");
};
// Y's own: beta k 2^g [j][K index] (then nw^T), half of beta v [j][v] (16-bit: v before) and A [i][j] (then u^T over both), the triangular matrix
constexpr int BK = KQ + 65536, V_ = BK + 32768, A_ = V_ + 16384, T_ = A_, UT = V_, M_ = A_ + 16384;
constexpr int LD = 36, MB = 32 * LD;                        // I + L as three 32 x 32 blocks: (0, 0), (1, 0), (1, 1)
constexpr int TILES = M_ + 3 * MB * 4;
constexpr int D1 = 0, D1_COLS = 160, NW = 320, U = 384;      // accumulator columns (two of [Gamma; Q K^T]: Y is an item behind)

struct Shared {
    uint64_t ldin, fullV;                                   // rows | v landed
    uint64_t op1[2], mm1[2];                                // operands of channel half 0, 1 written; [Gamma; Q K^T] done, one per accumulator buffer:
                                                            // a scalar gate's can be done for the next item before Y comes to wait for this one's
    uint64_t rows, acc, hand, khFree;                       // row scales | Aqk | kbar, scale q 2^g, beta k 2^g written; the first two tiles and Aqk have left
    uint64_t opA, opV, mmV, mmN, mmU;                       // A and the high half of beta v | the low half written; high half used | nw^T, u^T done
    uint64_t nwReady, uReady, bkFree, abFree;               // nw^T, u^T staged | have left
    uint32_t tmem;
    __align__(16) float beta[2][CH];                        // Y is an item behind
    struct { int item, start, len, h, hk; } info[4];        // of the items, by the warp that requests their rows
    __align__(16) float rs[2][CH], part[2][CH];             // L2 scales of the k, q rows (first the sums of half their channels); of the other half
    // cumsum rows of the four block anchors, [4] = last valid row; first the lower then the upper four of every eight channels, so that the
    // threads of a row read them without bank conflicts.  2^(ga[I] - ga[I - 1]) of I = 2, 3
    __align__(16) float ga[5][DK], step[2][DK];
};
constexpr int SMEM = TILES + (int)sizeof(Shared);
static_assert(SMEM <= 232448, "shared memory of one CTA");

struct Maps { CUtensorMap k, q, g, v; };                    // g: the cumsum, or the raw gate of a kernel that forms it

// G = MkdaGateFwd: the gate is formed here too, for calls of at most one item per CTA (then a compile-time fact): X waits for its rows anyway, and 2.7 us of
// its time replace a kernel of 5.1 us (77 tokens x 16 heads).
struct NoGate {};
template <class G> constexpr bool GATED = std::is_same<G, MkdaGateFwd>::value;
constexpr int RAW_X = BK;                                   // raw gate of the item, fp32 or 16 bits: nothing else is there yet

__device__ __forceinline__ void sync_x() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void sync_y() { asm volatile("bar.sync 2, 256;" ::: "memory"); }
static_assert(X_WARPS == 16 && Y_WARPS == 8, "threads of the named barriers");

// The items of a CTA: gridDim.x apart, heads fastest (the threads that request copies walk them; the others read `info`).
struct Walk {
    int c, h, hk, start, len, dc, dh, HV, NC;
    float rG;
    const MkdaLayout& L;
    __device__ __forceinline__ Walk(const MkdaLayout& l) : L(l) {
        HV = l.HV; NC = l.NC;
        c = blockIdx.x / HV; h = blockIdx.x - c * HV; dc = gridDim.x / HV; dh = gridDim.x - dc * HV;
        rG = 1.f / (float)(HV / l.HK);
        table();
    }
    __device__ __forceinline__ void table() {
        hk = (int)(((float)h + 0.5f) * rG);
        const int i = min(c, NC - 1);
        start = L.chunk_start[i]; len = L.chunk_len[i];
    }
    __device__ __forceinline__ bool valid() const { return c < NC; }
    __device__ __forceinline__ int item() const { return c * HV + h; }
    __device__ __forceinline__ void next() {
        c += dc; h += dh;
        if (h >= HV) { h -= HV; ++c; }
        table();
    }
};
template <bool ONE>
__device__ __forceinline__ int item_count(const MkdaLayout& L) { return ONE ? 1 : (L.NC * L.HV - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x; }

// eight consecutive floats by the threads c = 0..7 of a row: the two 16-byte halves in an order that keeps the eight off each other's banks
__device__ __forceinline__ void lds8_swapped(const float* p, bool s, f32x2 (&v)[4]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p + (s ? 4 : 0)), b = *reinterpret_cast<const ulonglong2*>(p + (s ? 0 : 4));
    v[0] = s ? b.x : a.x; v[1] = s ? b.y : a.y; v[2] = s ? a.x : b.x; v[3] = s ? a.y : b.y;
}
template <int DT>
__device__ __forceinline__ void lds_raw8(const uint8_t* row, int k8, Raw8& r) {
    if (DT == MKDA_F32) {
        r.a = *reinterpret_cast<const uint4*>(row + k8 * 32);
        r.b = *reinterpret_cast<const uint4*>(row + k8 * 32 + 16);
    } else {
        r.a = *reinterpret_cast<const uint4*>(row + k8 * 16);
    }
}

// ---- the gate and its chunk-local inclusive cumsum (log2), summed in the same order as by the kernels that do nothing else (prologue.cu) ----
// One decay per token, by one warp: the raw values of rows 2 l and 2 l + 1 in, their cumsum out (the last valid one past the end).  Groups of eight rows,
// then the groups in order.
__device__ __forceinline__ void scalar_cumsum(const MkdaGateFwd& p, int h, int len, float& a, float& b, int lane) {
    const float E = p.A_log ? expf(p.A_log[h]) : 1.f, bias = p.dt_bias ? p.dt_bias[h] : 0.f;
    a = 2 * lane < len ? gate_value(p.mode, a + bias, E, p.lower_bound) : 0.f;
    const float v = 2 * lane + 1 < len ? gate_value(p.mode, b + bias, E, p.lower_bound) : 0.f;
    b = __fadd_rn(a, v);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
        const float t = __shfl_up_sync(0xffffffffu, b, 1);
        if ((lane & 3) == j) { a = __fadd_rn(t, a); b = __fadd_rn(a, v); }
    }
    float pre = 0.f;
#pragma unroll
    for (int w = 0; w < 7; ++w) {
        const float t = __shfl_sync(0xffffffffu, b, 4 * w + 3);
        if (w < (lane >> 2)) pre += t;
    }
    a = (pre + a) * RCP_LN2;
    b = (pre + b) * RCP_LN2;
}
// One decay per channel, by X: thread = 16 rows of a channel, four at a time: all of it is fetched cold, once, so short code is fast code.
// `raw` -> `rows`, both [64][128]; E and the bias were requested before the rows were waited for.
__device__ __forceinline__ void channel_cumsum(const MkdaGateFwd& p, const uint8_t* raw, float* rows, float (&tot)[5][DK], size_t first, int len, float E, float bias) {
    const int ch = threadIdx.x & 127, b = threadIdx.x >> 7;
    float run = 0.f, pre = 0.f;
#pragma unroll 1
    for (int r = 16 * b; r < 16 * b + 16; r += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float g = gate_value(p.mode, ld1(raw, p.x_dtype, (r + i) * 128 + ch) + bias, E, p.lower_bound);
            if (r + i < len) run = __fadd_rn(run, g);      // not contracted with the gate's last product
            rows[(r + i) * 128 + ch] = run;
        }
    }
    tot[b][ch] = run;
    sync_x();
    for (int w = 0; w < b; ++w) pre += tot[w][ch];
#pragma unroll 4
    for (int r = 16 * b; r < 16 * b + 16; ++r) {
        const float g = (pre + rows[r * 128 + ch]) * RCP_LN2;
        rows[r * 128 + ch] = g;
        if (p.g_c && r < len) p.g_c[first + (size_t)r * p.L.HV * 128] = g;
    }
    sync_x();
}
}  // namespace in

// ---- X ----------------------------------------------------------------------------------------------------------------------------------
// Thread: eight channels of the first half of row r = tid / 8 and eight of the second half of row r ^ 48: the products of channels 0..63 run
// while the operands of 64..127 are written, and as a row of block B enters 4 - B column tiles, each thread writes five.
// SCALAR: the gate is one decay per token (the same cumsum in all 128 channels).  It then commutes with the contraction
// over channels, Gamma_ij = (k_i . k_j) 2^(g_i - g_j), so the products are plain K K^T / Q K^T (one product over a stacked
// [K; Q] tile; bf16 rows have no low half) and the decay is applied to the accumulators, element by element and for i >= j only: nothing is
// anchored, no exponent is ever positive, and any g <= 0 is in range (the per-channel path needs g >= -5 per token).
template <int DT, bool SCALAR, class G>
__device__ __forceinline__ void intra_x(const MkdaIntraFwd& p, const G& gate, uint8_t* base, uint32_t tmem, in::Shared& sh) {
    using namespace in;
    using R = Rows<DT, SCALAR>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c8 = tid & 7;
    const bool odd = c8 & 4;
    auto row_of = [&](int hf) { return hf ? (tid >> 3) ^ 48 : tid >> 3; };
    uint8_t* sKQ = base + KQ;
    // nw^T [K index][tok] and u^T [v][tok] of an item leave as ready-made chunk tiles over their operands (the serial kernels fetch them with one
    // bulk copy; token columns past the end are exact zeros: rows of beta v and beta k are zero there)
    auto read_out = [&](int it) {
        auto stage = [&](int col, uint8_t* tile, float sign) {
            float a[16];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, col + 16 * (warp >> 2)), a);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                float o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = sign * a[8 * m + j];
                store_split8(tile, tile + 16384, 128, (warp & 3) * 32 + lane, 2 * (warp >> 2) + m, o);
            }
        };
        umma::wait_mma(&sh.mmN, it & 1);
        stage(NW, base + BK, -1.f);
        umma::signal(&sh.nwReady, lane);
        umma::wait_mma(&sh.mmU, it & 1);
        stage(U, base + UT, 1.f);
        umma::signal(&sh.uReady, lane);
    };
    const int count = item_count<GATED<G>>(p.L);
    for (int it = 0; it < count; ++it) {
        const uint32_t par = it & 1;
        float* beta = sh.beta[par];
        float* gs = &sh.ga[0][0] + par * CH;                // SCALAR: the cumsum of every row, two items (rows past the end: the last valid one)
        // ---- this item's rows into registers; park the anchor rows of g ----
        float E = 1.f, bias = 0.f, raw0 = 0.f, raw1 = 0.f;   // of a gate that is formed here, and beta or a scalar gate before it is
        if constexpr (GATED<G> && !SCALAR) {
            const int h = blockIdx.x % p.L.HV;
            if (gate.A_log) E = expf(gate.A_log[h]);
            if (gate.dt_bias) bias = gate.dt_bias[h * 128 + (tid & 127)];
        }
        umma::mbar_wait(&sh.ldin, par);
        const int len = sh.info[it & 3].len;
        if constexpr (GATED<G> && !SCALAR) {
            const size_t first = ((size_t)sh.info[0].start * p.L.HV + sh.info[0].h) * 128 + (tid & 127);
            channel_cumsum(gate, base + RAW_X, reinterpret_cast<float*>(base + RAW_G), sh.ga, first, len, E, bias);
        }
        Raw8 wk[2], wq[2];
        f32x2 vg[2][4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = row_of(hf), rr = r < len ? r : len - 1, k8 = c8 + 8 * hf;
            lds_raw8<DT>(base + R::K + rr * R::PITCH, k8, wk[hf]);
            lds_raw8<DT>(base + R::Q + rr * R::PITCH, k8, wq[hf]);
            if (r >= len) {                                 // rows past the end are zero
                wk[hf].a = wq[hf].a = make_uint4(0, 0, 0, 0);
                if (DT == MKDA_F32) wk[hf].b = wq[hf].b = make_uint4(0, 0, 0, 0);
            }
            if (!SCALAR) {
                const float* g = reinterpret_cast<const float*>(base + RAW_G) + k8 * 8;
                lds8_swapped(g + rr * 128, odd, vg[hf]);
                if (it && hf == 0) umma::mbar_wait(&sh.hand, par ^ 1);             // nobody reads the previous item's last row any more
                if ((r & 15) == 0) sts_halves(sh.ga[r >> 4], k8, vg[hf]);
                if (r == len - 1) sts_halves(sh.ga[4], k8, vg[hf]);
                if ((r & 15) == 0 && r >= 32) {
                    f32x2 prev[4];
                    lds8_swapped(g + (r - 16 < len ? r - 16 : len - 1) * 128, odd, prev);
#pragma unroll
                    for (int e = 0; e < 4; ++e) prev[e] = ex2f2_(sub2(vg[hf][e], prev[e]));
                    sts_halves(sh.step[(r >> 4) - 2], k8, prev);
                }
            }
        }
        {   // beta (and a scalar gate's cumsum), used once the products are done
            const size_t HV = p.L.HV;
            const int i = sh.info[it & 3].start + min(tid & (CH - 1), len - 1), h = sh.info[it & 3].h;
            if constexpr (GATED<G>) {
                if (tid < CH) {
                    raw0 = ld1(gate.beta_raw, gate.beta_dtype, i * HV + h);
                } else if (SCALAR && warp == 2) {           // two rows per lane
                    const size_t first = (size_t)sh.info[it & 3].start * HV + h;
                    raw0 = ld1(gate.x, gate.x_dtype, first + min(2 * lane, len - 1) * HV);
                    raw1 = ld1(gate.x, gate.x_dtype, first + min(2 * lane + 1, len - 1) * HV);
                }
            } else {
                if (tid < CH) cp_async4(&beta[tid], p.beta + i * HV + h);
                else if (SCALAR && tid < 2 * CH) cp_async4(gs + tid - CH, p.g_c + i * HV + h);
            }
        }
        umma::fence_before_sync();
        sync_x();
        umma::fence_after_sync();
        // ---- operands, half by half ----
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = row_of(hf), I0 = r >> 4, k8 = c8 + 8 * hf;
            if (SCALAR && DT == MKDA_BF16) {                // rows 0..63 = k, rows 64..127 = q, zero past the end
                *reinterpret_cast<uint4*>(sKQ + umma::tile_chunk_offset(128, r, k8)) = wk[hf].a;
                *reinterpret_cast<uint4*>(sKQ + umma::tile_chunk_offset(128, 64 + r, k8)) = wq[hf].a;
            } else if (SCALAR) {
                f32x2 x8[4];
                unpack8<DT>(wk[hf], x8);
                store_split8(sKQ, sKQ + 32768, 128, r, k8, x8);
                unpack8<DT>(wq[hf], x8);
                store_split8(sKQ, sKQ + 32768, 128, 64 + r, k8, x8);
            } else {
                f32x2 x8[4], d[4], e8[4], t8[4];
                lds_halves(sh.ga[I0], k8, d);
#pragma unroll
                for (int e = 0; e < 4; ++e) { d[e] = sub2(vg[hf][e], d[e]); e8[e] = mul2(ex2f2_(d[e]), both(ROW_UP)); }
                unpack8<DT>(wk[hf], x8);
#pragma unroll
                for (int e = 0; e < 4; ++e) t8[e] = mul2(x8[e], e8[e]);
                store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + (r & 15), k8, t8);
                unpack8<DT>(wq[hf], x8);
#pragma unroll
                for (int e = 0; e < 4; ++e) t8[e] = mul2(x8[e], e8[e]);
                store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + 16 + (r & 15), k8, t8);
                unpack8<DT>(wk[hf], x8);
#pragma unroll
                for (int e = 0; e < 4; ++e) { x8[e] = mul2(x8[e], both(COL_DOWN)); t8[e] = mul2(x8[e], ex2f2_(mul2(d[e], both(-1.f)))); }
                if (it && hf == 0) umma::mbar_wait(&sh.khFree, par ^ 1);           // the tiles under the column tiles have left
                store_split8(base, base + KC_BYTES, KC_ROWS, kc_row(I0) + r, k8, t8);
#pragma unroll
                for (int I = 1; I < 4; ++I) {
                    if (I <= I0) continue;                  // warp-uniform
                    if (I == I0 + 1) {
                        lds_halves(sh.ga[I], k8, d);
                        scale_ex2(t8, x8, d, vg[hf]);
                    } else {                                // a step of decay (<= 1) further down the anchors instead of one more exponential
                        lds_halves(sh.step[I - 2], k8, d);
#pragma unroll
                        for (int e = 0; e < 4; ++e) t8[e] = mul2(t8[e], d[e]);
                    }
                    store_split8(base, base + KC_BYTES, KC_ROWS, kc_row(I) + r, k8, t8);
                }
            }
            umma::signal(&sh.op1[hf], lane);
        }
        // ---- L2 scales, while the products run: they are applied to what comes out (Gamma and Q K^T are bilinear in the rows) and to the tiles
        // below.  Four sums (k, q of two half rows) over eight threads; lane bit 2 ends up choosing the half, bit 1 between k and q ----
        if (SCALAR && it) umma::mbar_wait(&sh.khFree, par ^ 1);     // Y has used the previous item's
        if (p.l2) {
            float t[2][2];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                f32x2 x8[4], a = 0;
                float a0, a1;
                unpack8<DT>(wk[hf], x8);
#pragma unroll
                for (int e = 0; e < 4; ++e) a = fma2(x8[e], x8[e], a);
                unpack2(a, a0, a1);
                t[hf][0] = a0 + a1;
                a = 0;
                unpack8<DT>(wq[hf], x8);
#pragma unroll
                for (int e = 0; e < 4; ++e) a = fma2(x8[e], x8[e], a);
                unpack2(a, a0, a1);
                t[hf][1] = a0 + a1;
            }
            float u[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) u[j] = (odd ? t[1][j] : t[0][j]) + __shfl_xor_sync(0xffffffffu, odd ? t[0][j] : t[1][j], 4);
            float s = (c8 & 2 ? u[1] : u[0]) + __shfl_xor_sync(0xffffffffu, c8 & 2 ? u[0] : u[1], 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (!(c8 & 1)) (odd ? sh.part : sh.rs)[(c8 >> 1) & 1][row_of(odd)] = s;
            sync_x();
            if (tid < 2 * CH) {
                const int i = tid & (CH - 1), x = tid >> 6;
                s = rsqrtf(sh.rs[x][i] + sh.part[x][i] + p.l2_eps);
                sh.rs[x][i] = s;
                const int HK = p.L.HK, hk = sh.info[it & 3].hk;
                if (p.k_rstd_out && sh.info[it & 3].h == hk * (p.L.HV / HK) && i < len)        // the backward pass reads them
                    (x ? p.q_rstd_out : p.k_rstd_out)[(size_t)(sh.info[it & 3].start + i) * HK + hk] = s;
            }
        } else if (tid < 2 * CH) {
            const int i = tid & (CH - 1), x = tid >> 6;
            sh.rs[x][i] = p.k_rstd ? (x ? p.q_rstd : p.k_rstd)[(size_t)(sh.info[it & 3].start + min(i, len - 1)) * p.L.HK + sh.info[it & 3].hk] : 1.f;
        }
        if constexpr (GATED<G>) {
            const size_t HV = p.L.HV, first = (size_t)sh.info[it & 3].start * HV + sh.info[it & 3].h;
            if (tid < CH) {
                const float b = gate.beta_sigmoid ? gate.beta_scale * sigmoidf_(raw0) : raw0;
                beta[tid] = tid < len ? b : 0.f;
                if (gate.beta_out && tid < len) gate.beta_out[first + tid * HV] = b;
            } else if (SCALAR && warp == 2) {
                scalar_cumsum(gate, sh.info[it & 3].h, len, raw0, raw1, lane);
                *reinterpret_cast<float2*>(gs + 2 * lane) = make_float2(raw0, raw1);
                if (gate.g_c && 2 * lane < len) gate.g_c[first + 2 * lane * HV] = raw0;
                if (gate.g_c && 2 * lane + 1 < len) gate.g_c[first + (2 * lane + 1) * HV] = raw1;
            }
        } else {
            cp_async_wait_all();
            if (tid < CH && tid >= len) beta[tid] = 0.f;
        }
        __syncwarp();
        if (lane == 0) umma::arrive(&sh.rows);
        if (it) read_out(it - 1);
        umma::wait_mma(&sh.mm1[par], (it >> 1) & 1);
        umma::mbar_wait(&sh.rows, par);
        // ---- over the dead operands: the state kernels' scaled operands, kbar = k 2^(gL - g) (gL = last valid row) and scale q 2^g; beta k 2^g for Y ----
        const float gLs = SCALAR ? gs[CH - 1] : 0.f;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = row_of(hf), k8 = c8 + 8 * hf;
            const float up = SCALAR ? ex2f_(gs[r]) : 1.f, fk = sh.rs[0][r], fq = sh.rs[1][r] * p.scale, fb = fk * beta[r];
            const f32x2 sk = both(SCALAR ? fk * ex2f_(gLs - gs[r]) : fk), sq = both(SCALAR ? fq * up : fq), sb = both(SCALAR ? fb * up : fb);
            f32x2 t8[4], e8[4], x8[4];
            unpack8<DT>(wk[hf], x8);
            if (SCALAR) {
#pragma unroll
                for (int e = 0; e < 4; ++e) t8[e] = mul2(x8[e], sk);
            } else {
                lds_halves(sh.ga[4], k8, e8);
                scale_ex2(t8, x8, e8, vg[hf]);
#pragma unroll
                for (int e = 0; e < 4; ++e) { t8[e] = mul2(t8[e], sk); e8[e] = ex2f2_(vg[hf][e]); }
            }
            store_split8(base + KB, base + KB + 16384, 64, r, k8, t8);
            unpack8<DT>(wq[hf], t8);
#pragma unroll
            for (int e = 0; e < 4; ++e) t8[e] = SCALAR ? mul2(t8[e], sq) : mul2(mul2(t8[e], sq), e8[e]);
            store_split8(base + QS, base + QS + 16384, 64, r, k8, t8);
            if (it && hf == 0) umma::mbar_wait(&sh.bkFree, par ^ 1);               // nw^T of the previous item has left
#pragma unroll
            for (int e = 0; e < 4; ++e) t8[e] = SCALAR ? mul2(x8[e], sb) : mul2(mul2(x8[e], sb), e8[e]);
            store_split8(base + BK, base + BK + 16384, 64, r, k8, t8);
        }
        const size_t item = sh.info[it & 3].item;
        if (SCALAR && tid < DK) p.gl[item * 128 + tid] = ex2f_(gLs);
        if (!SCALAR && warp == X_WARPS - 1 && lane < 16) {
            f32x2 gL[4];
            lds_halves(sh.ga[4], lane, gL);
#pragma unroll
            for (int e = 0; e < 4; ++e) gL[e] = ex2f2_(gL[e]);
            sts8(p.gl + item * 128 + lane * 8, gL);
        }
        umma::signal(&sh.hand, lane);
    }
    read_out(count - 1);
}

// ---- Y ----------------------------------------------------------------------------------------------------------------------------------
// Inverse of the unit lower-triangular matrix in place (fixed summation order) by recursive halving: the four 16 x 16 diagonal blocks by
// forward substitution, then the off-diagonal block of each 32 x 32 half and finally the 32 x 32 block below the diagonal, each as
// X = -B^-1 C A^-1  with A^-1 / B^-1 the inverses above / beside it.  Every entry depends on the rows up to its own only, and the order of the
// sums is fixed by the indices.  The merges are TF32 products with error compensation (three products, fp32 accumulation: ~2^-21 per product).
// T = 32 rows of scratch, free once `free` completes.
__device__ __forceinline__ void invert_unit_lower(float* M, float* T, uint64_t* free, int it) {
    using namespace in;
    const int y = (threadIdx.x >> 5) & (Y_WARPS - 1), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (y < 2) {
        float* D = M + y * 2 * MB;
        const int o = lane & 16, col = lane & 15;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float s[4] = {r == col ? 1.f : 0.f, 0.f, 0.f, 0.f};            // four partial sums: the chain from row to row is what takes the time
#pragma unroll
            for (int c = 0; c < r; c += 4) {
                const float4 m = *reinterpret_cast<const float4*>(D + (o + r) * LD + o + c);
                const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < r) s[e] = fmaf(-mv[e], x[c + e], s[e]);
            }
            x[r] = (s[0] + s[1]) + (s[2] + s[3]);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 16; ++r) D[(o + r) * LD + o + col] = x[r];
        __syncwarp();
        // (B^-1 C) A^-1: the first product stays in registers as the left operand of the second, whose terms are summed in the order in which an
        // accumulator's columns lie (2 t, 2 t + 1 of every eight in the place of t, t + 4)
        float acc[2][4], z[2][4];
        warp_mma_short<2, 16, LD, 1, LD, 1>(acc, D + 16 * LD + 16, D + 16 * LD);
        warp_mma_chained(z, acc, D, LD);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            *reinterpret_cast<float2*>(D + (16 + g) * LD + 8 * nt + 2 * t) = make_float2(-z[nt][0], -z[nt][1]);
            *reinterpret_cast<float2*>(D + (24 + g) * LD + 8 * nt + 2 * t) = make_float2(-z[nt][2], -z[nt][3]);
        }
    }
    if (it) umma::mbar_wait(free, (it & 1) ^ 1);
    sync_y();
    // 32 x 32 block (rows 32.., columns 0..31): a tile of 16 x 8 per warp
    const int m0 = 16 * (y >> 2), n0 = 8 * (y & 3);
    auto product = [&](const float* A, const float* B, float* D, float sign) {
        float acc[1][4];
        warp_mma_short<1, 32, LD, 1, LD, 1>(acc, A + m0 * LD, B + n0);
        *reinterpret_cast<float2*>(D + (m0 + g) * LD + n0 + 2 * t) = make_float2(sign * acc[0][0], sign * acc[0][1]);
        *reinterpret_cast<float2*>(D + (m0 + g + 8) * LD + n0 + 2 * t) = make_float2(sign * acc[0][2], sign * acc[0][3]);
        sync_y();
    };
    product(M + MB, M, T, 1.f);
    product(M + 2 * MB, T, M + MB, -1.f);
}

template <int DT, bool SCALAR, bool ONE>
__device__ __forceinline__ void intra_y(const MkdaIntraFwd& p, uint8_t* base, uint32_t tmem, in::Shared& sh) {
    using namespace in;
    constexpr int YT = 32 * Y_WARPS;
    const int tid = threadIdx.x & (YT - 1), warp = threadIdx.x >> 5, lane = tid & 31, q = warp & 3;
    const size_t HV = p.L.HV;
    float* M = reinterpret_cast<float*>(base + M_);
    const int count = item_count<ONE>(p.L);
    for (int it = 0; it < count; ++it) {
        const uint32_t par = it & 1;
        const float* beta = sh.beta[par];
        const float* gs = &sh.ga[0][0] + par * CH;
        // ---- I + L and Aqk from the accumulators ----
        // per channel: warp quadrant = row block (16 rows of Gamma, then 16 rows of Q K^T); scalar gate: 64 rows of K K^T, then of Q K^T
        umma::mbar_wait(&sh.rows, par);
        umma::wait_mma(&sh.mm1[par], (it >> 1) & 1);
        const int len = sh.info[it & 3].len;
        {
            const int i = SCALAR ? (q & 1) * 32 + lane : 16 * q + (lane & 15);
            const bool isq = SCALAR ? q >= 2 : lane >= 16;
            const float bi = isq ? p.scale * sh.rs[1][i] : beta[i] * sh.rs[0][i], gi = SCALAR ? gs[i] : 0.f;
#pragma unroll
            for (int cg = 2 * ((warp >> 2) & 1), last = cg + 2; cg < last; ++cg) {
                float v[16];
                if (SCALAR || cg <= q) {                     // warp-uniform
                    umma::tmem_ld16(umma::tmem_addr(tmem, warp, D1 + par * D1_COLS + (SCALAR ? 0 : kc_row(q)) + 16 * cg), v);
#pragma unroll
                    for (int j4 = 0; j4 < 16; j4 += 4) {
                        const float4 r4 = *reinterpret_cast<const float4*>(sh.rs[0] + 16 * cg + j4);
                        const float rj[4] = {r4.x, r4.y, r4.z, r4.w};
                        float E[4] = {1.f, 1.f, 1.f, 1.f};
                        if (SCALAR) {
                            const float4 g4 = *reinterpret_cast<const float4*>(gs + 16 * cg + j4);
                            const float gj[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) E[e] = ex2f_(fminf(gi - gj[e], 0.f));
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int j = 16 * cg + j4 + e;
                            const float x = SCALAR ? bi * v[j4 + e] * E[e] * rj[e] : bi * v[j4 + e] * rj[e];
                            v[j4 + e] = j < i ? x : j > i ? 0.f : isq ? x : 1.f;
                        }
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = 0.f;
                }
                if (isq) {                                   // Aqk leaves as a ready-made [row][column] operand tile (rows past the end: zeros)
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        float o[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) o[j] = v[8 * m + j];
                        store_split8(base + AQ, base + AQ + 8192, 64, i, 2 * cg + m, o);
                    }
                } else if (SCALAR ? q == 1 || cg < 2 : cg <= (q | 1)) {      // the blocks (0, 1) and (2, 3) above the diagonal are read as zeros
                    float* d = M + (i < 32 ? 0 : cg < 2 ? MB : 2 * MB) + (i & 31) * LD + 16 * (cg & 1);
#pragma unroll
                    for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(d + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
            }
        }
        umma::signal(&sh.acc, lane);
        sync_y();
        invert_unit_lower(M, reinterpret_cast<float*>(base + T_), &sh.abFree, it);         // there u^T of the previous item may still be leaving
        // A leaves as a ready-made [row][column] operand tile (rows past the end: identity rows) and is the operand of nw and u
        uint8_t* At = reinterpret_cast<uint8_t*>(p.A) + (size_t)sh.info[it & 3].item * umma::QUARTER_TILE_BYTES;
        const int k8 = tid & 7;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int r = 32 * m + (tid >> 3);
            float a8[8];
            if (m == 0 && k8 >= 4) {
#pragma unroll
                for (int e = 0; e < 8; ++e) a8[e] = 0.f;
            } else {
                f32x2 a[4];
                lds8_swapped(M + (m == 0 ? 0 : k8 < 4 ? MB : 2 * MB) + (r & 31) * LD + 8 * (k8 & 3), k8 & 2, a);
#pragma unroll
                for (int e = 0; e < 4; ++e) unpack2(a[e], a8[2 * e], a8[2 * e + 1]);
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (k8 * 8 + e > r) a8[e] = 0.f;
            }
            if (p.A) store_split8(At, At + 8192, 64, r, k8, a8);         // a forward-only call has no use for it
            store_split8(base + A_, base + A_ + 8192, 64, r, k8, a8);
        }
        // beta v in two halves, one after the other in the same place: u is formed in front of nw, as soon as the low half is there.  fp32 rows are read
        // from global memory, there is no place for them (6 k packed tokens x 32 heads all the same 344 -> 243 us by the split into two groups)
        constexpr int N = 4;
        uint32_t lo[N][4];
        if (DT != MKDA_F32) umma::mbar_wait(&sh.fullV, par);
        Raw8 raw[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int i = tid + YT * n, r = i >> 4;
            if (DT != MKDA_F32) raw[n].a = *reinterpret_cast<const uint4*>(base + V_ + umma::tile_chunk_offset(64, r, i & 15));
            else ldraw8<DT>(p.v, ((size_t)(sh.info[it & 3].start + min(r, len - 1)) * HV + sh.info[it & 3].h) * 128 + (i & 15) * 8, raw[n]);
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int i = tid + YT * n, r = i >> 4;
            float v8[8];
            unpack8<DT>(raw[n], v8);
            const float b = beta[r];
            uint32_t hi[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                umma::split2(b * v8[2 * e], b * v8[2 * e + 1], hi[e], lo[n][e]);
                if (r >= len) hi[e] = lo[n][e] = 0u;
            }
            *reinterpret_cast<uint4*>(base + V_ + umma::tile_chunk_offset(64, r, i & 15)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
        umma::signal(&sh.opA, lane);
        umma::wait_mma(&sh.mmV, par);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int i = tid + YT * n;
            *reinterpret_cast<uint4*>(base + V_ + umma::tile_chunk_offset(64, i >> 4, i & 15)) = make_uint4(lo[n][0], lo[n][1], lo[n][2], lo[n][3]);
        }
        umma::signal(&sh.opV, lane);
        sync_y();                                            // the matrix has been read
    }
}

// ---- the four warps of one thread each ---------------------------------------------------------------------------------------------------
// The base passes through an empty statement in front of each group of products: kept in registers over the loop, the operand descriptors of
// all of them would spill.
__device__ __forceinline__ uint8_t* fresh(uint8_t* smem) {
    asm volatile("" : "+l"(smem));
    return smem;
}
template <int DT, bool SCALAR, bool ONE>
__device__ __forceinline__ void intra_mm1(const MkdaIntraFwd& p, uint8_t* smem, uint32_t tmem, in::Shared& sh) {
    using namespace in;
    const int count = item_count<ONE>(p.L);
    for (int it = 0; it < count; ++it) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            umma::wait_mma(&sh.op1[hf], it & 1);
            uint8_t* base = fresh(smem);
            uint8_t* kq = base + KQ + hf * 16384;
            if (SCALAR) {      // D[m][j]: lanes 0..63 = K K^T rows, lanes 64..127 = Q K^T rows; columns j = K rows of the same tile
                const umma::Opnd o = umma::opnd_k(kq, DT == MKDA_BF16 ? nullptr : kq + 32768, 128);
                umma::gemm(tmem + D1 + (it & 1) * D1_COLS, o, o, 128, 64, 64, hf);
            } else {
                // ONE product over the stacked column tiles: D[32 I + t][kc_row(I') + j].  Only the blocks I' = I are meaningful (the
                // anchors of the two operands match there) and read back; the others are finite and ignored.  An MMA costs
                // (4 KB of A + 32 N bytes of B) / 128 B per cycle, so N = 160 once is far cheaper than N = 32 four times.
                uint8_t* kc = base + hf * KC_ROWS * 128;
                umma::gemm(tmem + D1 + (it & 1) * D1_COLS, umma::opnd_k(kq, kq + 32768, 128), umma::opnd_k(kc, kc + KC_BYTES, KC_ROWS), 128, KC_ROWS, 64, hf);
            }
        }
        umma::commit(&sh.mm1[it & 1]);
    }
}
template <bool ONE>
__device__ __forceinline__ void intra_mm3(const MkdaIntraFwd& p, uint8_t* smem, uint32_t tmem, in::Shared& sh) {
    using namespace in;
    const int count = item_count<ONE>(p.L);
    for (int it = 0; it < count; ++it) {
        const uint32_t par = it & 1;
        umma::wait_mma(&sh.hand, par);                      // beta k 2^g
        umma::wait_mma(&sh.opA, par);
        uint8_t* base = fresh(smem);
        const umma::Opnd a = umma::opnd_k(base + A_, base + A_ + 8192, 64), v = umma::opnd_mn(base + V_, nullptr, 64);
        auto product_nw = [&]() {
            umma::gemm(tmem + NW, umma::opnd_mn(base + BK, base + BK + 16384, 64), a, 128, 64, 64, 0u);
            umma::commit(&sh.mmN);
        };
        umma::gemm(tmem + U, v, a, 128, 64, 64, 0u);
        umma::commit(&sh.mmV);
        // Of the last item nw comes first, under Y's writing of the low half (77 tokens 13.8 -> 13.4 us).  In front of other items that would hold up
        // what waits for u: 14 items per SM 123 -> 129 us
        if (it + 1 == count) product_nw();
        umma::wait_mma(&sh.opV, par);
        umma::Opnd hi = a;
        hi.lo = 0;
        umma::gemm(tmem + U, v, hi, 128, 64, 64, 1u);
        umma::commit(&sh.mmU);
        if (it + 1 < count) product_nw();
    }
}
// rows past the chunk's end belong to the next sequence (or read as zeros) and are never used
template <int DT, bool SCALAR>
__device__ __forceinline__ void request_q(const in::Walk& w, const in::Maps& maps, uint8_t* base, in::Shared& sh) {
    umma::tma_load_rows(base + in::Rows<DT, SCALAR>::Q, &maps.q, w.hk * 128, w.start, &sh.ldin);
}
template <int DT, bool SCALAR, class G>
__device__ __forceinline__ void request_rows(const G& gate, const in::Walk& w, int it, const in::Maps& maps, uint8_t* base, in::Shared& sh) {
    using R = in::Rows<DT, SCALAR>;
    auto& i = sh.info[it & 3];
    i.item = w.item(); i.start = w.start; i.len = w.len; i.h = w.h; i.hk = w.hk;
    uint32_t g_bytes = SCALAR ? 0u : 32768u;
    if constexpr (in::GATED<G> && !SCALAR) g_bytes = gate.x_dtype == MKDA_F32 ? 32768u : 16384u;
    umma::mbar_expect_tx(&sh.ldin, 2 * R::BYTES + g_bytes);
    if (!SCALAR) umma::tma_load_rows(base + (in::GATED<G> ? in::RAW_X : in::RAW_G), &maps.g, w.h * 128, w.start, &sh.ldin);
    umma::tma_load_rows(base + R::K, &maps.k, w.hk * 128, w.start, &sh.ldin);
    if (!R::LATE_Q) request_q<DT, SCALAR>(w, maps, base, sh);
}
template <int DT, bool SCALAR, class G>
__device__ __forceinline__ void intra_copy_x(const MkdaIntraFwd& p, const G& gate, const in::Maps& maps, uint8_t* base, in::Shared& sh) {
    using namespace in;
    using R = Rows<DT, SCALAR>;
    Walk w(p.L);                                            // the first item's rows are on their way
    for (int it = 0; w.valid(); ++it) {
        const size_t item = w.item();
        if (GATED<G>) w.c = w.NC; else w.next();
        umma::mbar_wait(&sh.mm1[it & 1], (it >> 1) & 1);    // the operands are dead
        if (w.valid()) request_rows<DT, SCALAR>(gate, w, it + 1, maps, base, sh);
        umma::mbar_wait(&sh.acc, it & 1);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.Aqk) + item * umma::QUARTER_TILE_BYTES, base + AQ, umma::QUARTER_TILE_BYTES);
        umma::mbar_wait(&sh.hand, it & 1);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.kbar) + item * umma::CHUNK_TILE_BYTES, base + KB, umma::CHUNK_TILE_BYTES);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.qs) + item * umma::CHUNK_TILE_BYTES, base + QS, umma::CHUNK_TILE_BYTES);
        umma::bulk_store_wait_read();
        umma::arrive(&sh.khFree);
        if (R::LATE_Q && w.valid()) request_q<DT, SCALAR>(w, maps, base, sh);
    }
}
template <int DT, bool ONE>
__device__ __forceinline__ void intra_copy_y(const MkdaIntraFwd& p, const in::Maps& maps, uint8_t* base, in::Shared& sh) {
    using namespace in;
    auto load_v = [&](const Walk& w) {                      // two boxes of 64 channels: rows in the layout of an operand tile
        if (DT == MKDA_F32) return;
        umma::mbar_expect_tx(&sh.fullV, 16384);
        umma::tma_load_rows(base + V_, &maps.v, w.h * 128, w.start, &sh.fullV);
        umma::tma_load_rows(base + V_ + 8192, &maps.v, w.h * 128 + 64, w.start, &sh.fullV);
    };
    Walk w(p.L);
    load_v(w);
    for (uint32_t it = 0; w.valid(); ++it) {
        const size_t item = w.item();
        if (ONE) w.c = w.NC; else w.next();
        umma::mbar_wait(&sh.nwReady, it & 1);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.nw) + item * umma::CHUNK_TILE_BYTES, base + BK, umma::CHUNK_TILE_BYTES);
        umma::mbar_wait(&sh.uReady, it & 1);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.u) + item * umma::CHUNK_TILE_BYTES, base + UT, umma::CHUNK_TILE_BYTES);
        umma::bulk_store_wait_read_but<1>();
        umma::arrive(&sh.bkFree);
        umma::bulk_store_wait_read();
        umma::arrive(&sh.abFree);
        if (w.valid()) load_v(w);
    }
}

template <int DT, bool SCALAR, class G>
__global__ void __launch_bounds__(in::THREADS, 1) intra_fwd_tc_kernel(const MkdaIntraFwd p, const G gate, const __grid_constant__ in::Maps maps) {
    using namespace in;
    constexpr bool ONE = GATED<G>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw;                              // no static shared memory: the dynamic block starts on a 1024-byte boundary
    Shared& sh = *reinterpret_cast<Shared*>(base + TILES);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    if (umma::smem_u32(base) & 1023) {                     // ... and nothing runs if that ever fails to hold
        follow_stream();
        if (threadIdx.x == 0) atomicExch(&umma::g_timeout_flag, 1u);
        return;
    }
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 512);
    if (threadIdx.x == 0) {
        for (uint64_t* b : {&sh.fullV, &sh.mm1[0], &sh.mm1[1], &sh.khFree, &sh.mmV, &sh.mmN, &sh.mmU, &sh.bkFree, &sh.abFree}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.op1[0], &sh.op1[1], &sh.rows, &sh.hand, &sh.nwReady, &sh.uReady}) umma::mbar_init(b, X_WARPS);
        for (uint64_t* b : {&sh.opA, &sh.opV, &sh.acc}) umma::mbar_init(b, Y_WARPS);
        umma::fence_barrier_init();
    }
    // The first rows are requested while barriers and tensor memory are set up: with one item per CTA all the rest waits for them (77 tokens x 16 heads
    // 14.3 -> 13.8 us)
    if (warp == X_WARPS + Y_WARPS + COPY_X) {
        if (umma::elect_one()) {
            umma::mbar_init(&sh.ldin, 1);
            umma::fence_barrier_init();
            follow_stream();
            const Walk w(p.L);
            request_rows<DT, SCALAR>(gate, w, 0, maps, base, sh);
            if (Rows<DT, SCALAR>::LATE_Q) request_q<DT, SCALAR>(w, maps, base, sh);
        }
        __syncwarp();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;
    follow_stream();
    if (warp < X_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(X_REGS));
        intra_x<DT, SCALAR>(p, gate, base, tmem, sh);
    } else if (warp < X_WARPS + Y_WARPS) {
        intra_y<DT, SCALAR, ONE>(p, base, tmem, sh);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(ISSUE_REGS));
        if (umma::elect_one()) {
            switch (warp - X_WARPS - Y_WARPS) {
                case 0: intra_mm1<DT, SCALAR, ONE>(p, base, tmem, sh); break;
                case COPY_X: intra_copy_x<DT, SCALAR>(p, gate, maps, base, sh); break;
                case 2: intra_copy_y<DT, ONE>(p, maps, base, sh); break;
                default: intra_mm3<ONE>(p, base, tmem, sh);
            }
        }
        __syncwarp();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

int tc_intra_status(unsigned int* out) {
    return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1;
}
int tc_intra_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

template <int DT, bool SCALAR, class G>
static int launch_intra_fwd_tc_t(const MkdaIntraFwd* p, const G& gate, cudaStream_t stream) {
    auto kern = intra_fwd_tc_kernel<DT, SCALAR, G>;
    if (int e = ensure_smem((const void*)kern, in::SMEM, "intra_fwd")) return e;
    static const int regs = kernel_registers((const void*)kern);
    if (regs < in::LAUNCH_REGS) return set_error(MKDA_ERR_LAUNCH, "intra_fwd: built with fewer registers than its warps redistribute");
    in::Maps maps;
    memset(&maps, 0, sizeof(maps));
    const unsigned long long rows = (unsigned long long)p->L.TT, k_cols = (unsigned long long)p->L.HK * 128, v_cols = (unsigned long long)p->L.HV * 128;
    constexpr int ES = DT == MKDA_F32 ? 4 : 2;
    int e = make_rows_map(&maps.k, p->k, ES, rows, k_cols, "intra_fwd");
    if (!e) e = make_rows_map(&maps.q, p->q, ES, rows, k_cols, "intra_fwd");
    if constexpr (in::GATED<G>) {
        if (!e && !SCALAR) e = make_rows_map(&maps.g, gate.x, gate.x_dtype == MKDA_F32 ? 4 : 2, rows, v_cols, "intra_fwd");
    } else {
        if (!e && !SCALAR) e = make_rows_map(&maps.g, p->g_c, 4, rows, v_cols, "intra_fwd");
    }
    if (!e && DT != MKDA_F32) e = make_rows_map(&maps.v, p->v, 2, rows, v_cols, "intra_fwd", CH, 64);
    if (e) return e;
    const int items = p->L.NC * p->L.HV;
    launch(kern, items < sm_count() ? items : sm_count(), in::THREADS, in::SMEM, stream, *p, gate, maps);
    return check_launch("intra_fwd");
}
template <class G>
static int launch_intra_fwd_tc_g(const MkdaIntraFwd* p, const G& gate, cudaStream_t stream) {
    switch (p->qkv_dtype * 2 + (p->scalar_gate ? 1 : 0)) {
        case MKDA_F32 * 2: return launch_intra_fwd_tc_t<MKDA_F32, false>(p, gate, stream);
        case MKDA_BF16 * 2: return launch_intra_fwd_tc_t<MKDA_BF16, false>(p, gate, stream);
        case MKDA_F16 * 2: return launch_intra_fwd_tc_t<MKDA_F16, false>(p, gate, stream);
        case MKDA_F32 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_F32, true>(p, gate, stream);
        case MKDA_BF16 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_BF16, true>(p, gate, stream);
        case MKDA_F16 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_F16, true>(p, gate, stream);
    }
    return set_error(MKDA_ERR_ARG, "intra_fwd: unsupported dtype");
}
int launch_intra_fwd_tc(const MkdaIntraFwd* p, const MkdaGateFwd* gate, cudaStream_t stream) {
    return gate ? launch_intra_fwd_tc_g(p, *gate, stream) : launch_intra_fwd_tc_g(p, in::NoGate{}, stream);
}

}  // namespace mkda
