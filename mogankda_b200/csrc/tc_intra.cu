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
// What bounds it: the chain of phases of an item with one CTA per SM (18 k cycles; the item's own bytes take 8 k at 25 B per cycle).
// Packed 6 k prefill x 32 heads 288 -> 236 us (with the L2 statistics, formerly a kernel), 32 k tokens 1373 -> 1120 us.
#include "host.h"
#include "intra.cuh"

namespace mkda {

struct IntraShared {
    uint64_t ldin, op1, op2;                               // rows landed | operands of the first, second products written (16 warps)
    uint64_t mm1, mmN, mmU;                                // products done: [Gamma; Q K^T], nw^T, u^T
    uint32_t tmem;
    __align__(16) float beta[2][CH];                       // of this item and (arriving) the next
    float rk[CH], rq[CH];                                  // L2 scales of the rows
    __align__(16) float T[32][36];
};
constexpr int TLD = 36;
// 16 compute warps and one that issues the products (of a warpgroup of its own).  The tensor pipe accepts a product as slowly as it executes
// them: the compute warp that issued used to come 1.4 k cycles after the others (of 19.7 k per item).  Registers as in bwd_chunk:
// 16 x 32 x 112 + 4 x 32 x 32 = the 640 x 96 of the launch.
constexpr int INTRA_THREADS = 640, INTRA_WARP_MMA = 16, INTRA_LAUNCH_REGS = 96;
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

constexpr int MLD = 68;
constexpr float ROW_UP = 0x1p48f, COL_DOWN = 0x1p-48f;      // column operand: 108 + 64 - 48 < 127, row operand: 64 + 48 < 127 for |k| < 2^64
// the four column tiles stacked by rows into one 160-row tile (hi 40 KB, then lo)
__host__ __device__ constexpr int kc_row(int I) { return I == 0 ? 0 : I == 1 ? 16 : I == 2 ? 48 : 96; }
constexpr int KC_ALL_ROWS = 160;
constexpr int KC_ALL_BYTES = KC_ALL_ROWS * 128 * 2;        // one of hi / lo
constexpr int KQ_OFF = 81920;                              // [128][128] hi 32 KB, lo 32 KB
constexpr int OPND_BYTES = KQ_OFF + 65536;                 // 144 KB
constexpr int TA_OFF = 65536;                              // A, over the dead column tiles
// The 16-bit k, q and the g rows of the NEXT item arrive by tiled copy (one 64 x 128 box per tensor) while the current item's
// inverse and second products run: k and g rows in the upper 48 KB of the [Kr; Qr] tile, dead once the first products are
// done, q rows over the kbar tile as soon as that has left.  They are read back into registers before the next item's operands are staged over them.  (Loads
// into registers at that point are accepted only as fast as their data returns and occupied every thread for a fifth of
// the item; one small bulk copy per row is slower still.)
struct IntraMaps { CUtensorMap k, q, g; };
constexpr int RAW_K = 98304;                               // [64][128] 16-bit, 16 KB
constexpr int RAW_G = RAW_K + 16384;                       // [64][128] fp32, 32 KB
constexpr int RAW_Q = OPND_BYTES;                          // [64][128] 16-bit, 16 KB, over the kbar tile
constexpr int INTRA_TC_SMEM = OPND_BYTES + 32768 + 2 * CH * MLD * 4 + 1024;        // operands, kbar tile, scale q 2^g tile (later sM / sInv)
static_assert(RAW_G + 32768 <= OPND_BYTES, "k / g rows must fit in the dead part of the operand region");
static_assert(2 * CH * MLD * 4 >= 32768, "the scale q 2^g tile must fit below the end");
constexpr int STORER = 256;                                // the thread that issues every bulk store: its warp has no part in the inverse

// Inverse of the unit lower-triangular 64 x 64 matrix sM into sInv (fixed summation order) by recursive halving:
// the four 16 x 16 diagonal blocks by forward substitution, then the off-diagonal block of each 32 x 32 half and finally
// the 32 x 32 block below the diagonal, each as  X = -B^-1 (C A^-1)  with A^-1 / B^-1 the inverses above / beside it.
// Every entry depends on the rows up to its own only, and the order of the sums is fixed by the indices.  Blocks (0, 1) and (2, 3) have to
// be zero on entry; the blocks further above the diagonal are not touched.
// The merges are TF32 products with error compensation (three products, fp32 accumulation: ~2^-21 per product), one 16 x 8 tile per warp:
// fragments need a quarter of the shared-memory loads of fp32 register tiles, which bounded them (1.05 k cycles per 32 x 32 product).
__device__ __forceinline__ void invert_unit_lower(const float* __restrict__ sM, float* __restrict__ sInv, IntraShared& sh) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    if (warp < 2) {
        const int o = 32 * warp + (lane & 16), col = lane & 15;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float s[4] = {r == col ? 1.f : 0.f, 0.f, 0.f, 0.f};            // four partial sums: the chain from row to row is what takes the time
#pragma unroll
            for (int c = 0; c < r; c += 4) {
                const float4 m = *reinterpret_cast<const float4*>(sM + (o + r) * MLD + o + c);
                const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < r) s[e] = fmaf(-mv[e], x[c + e], s[e]);
            }
            x[r] = (s[0] + s[1]) + (s[2] + s[3]);
        }
#pragma unroll
        for (int r = 0; r < 16; ++r) sInv[(o + r) * MLD + o + col] = x[r];
        __syncwarp();
        // 16 x 16 block (1, 0) or (3, 2): both of its diagonal blocks are this warp's
        const int ro = 32 * warp + 16, co = 32 * warp;
        float* T = &sh.T[16 * warp][0];
        float acc[2][4];
        warp_mma_short<2, 16, MLD, 1, MLD, 1>(acc, sM + ro * MLD + co, sInv + co * MLD + co);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            *reinterpret_cast<float2*>(T + g * TLD + 8 * nt + 2 * t) = make_float2(acc[nt][0], acc[nt][1]);
            *reinterpret_cast<float2*>(T + (g + 8) * TLD + 8 * nt + 2 * t) = make_float2(acc[nt][2], acc[nt][3]);
        }
        __syncwarp();
        warp_mma_short<2, 16, MLD, 1, TLD, 1>(acc, sInv + ro * MLD + ro, T);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            *reinterpret_cast<float2*>(sInv + (ro + g) * MLD + co + 8 * nt + 2 * t) = make_float2(-acc[nt][0], -acc[nt][1]);
            *reinterpret_cast<float2*>(sInv + (ro + g + 8) * MLD + co + 8 * nt + 2 * t) = make_float2(-acc[nt][2], -acc[nt][3]);
        }
    }
    sync_compute();
    // 32 x 32 block (rows 32.., columns 0..31): eight warps, one 16 x 8 tile each.  (Leaving out the products with zero blocks needs the code
    // of several lengths and made the whole kernel 5 % slower: it is fetched anew for every item.)
    const int m0 = 16 * ((warp >> 2) & 1), n0 = 8 * (warp & 3);
    float acc[1][4];
    if (warp < 8) {
        warp_mma_short<1, 32, MLD, 1, MLD, 1>(acc, sM + (32 + m0) * MLD, sInv + n0);
        *reinterpret_cast<float2*>(&sh.T[m0 + g][n0 + 2 * t]) = make_float2(acc[0][0], acc[0][1]);
        *reinterpret_cast<float2*>(&sh.T[m0 + g + 8][n0 + 2 * t]) = make_float2(acc[0][2], acc[0][3]);
    }
    sync_compute();
    if (warp < 8) {
        warp_mma_short<1, 32, MLD, 1, TLD, 1>(acc, sInv + (32 + m0) * MLD + 32, &sh.T[0][n0]);
        *reinterpret_cast<float2*>(sInv + (32 + m0 + g) * MLD + n0 + 2 * t) = make_float2(-acc[0][0], -acc[0][1]);
        *reinterpret_cast<float2*>(sInv + (32 + m0 + g + 8) * MLD + n0 + 2 * t) = make_float2(-acc[0][2], -acc[0][3]);
    }
    sync_compute();
}

// The issuing thread.  The base passes through an empty statement in front of each group of products: kept in registers over the loop, the
// operand descriptors of all of them would spill.
template <bool SCALAR>
__device__ __forceinline__ void intra_issue(uint8_t* smem, uint32_t tmem, int total, IntraShared& sh) {
    uint8_t* base = smem;
    auto fresh = [&]() { base = smem; asm volatile("" : "+l"(base)); };
    uint32_t it = 0;
    for (int item = blockIdx.x; item < total; item += gridDim.x, ++it) {
        umma::wait_mma(&sh.op1, it & 1);
        fresh();
        uint8_t* sKQ = base + KQ_OFF;
        if (SCALAR) {      // D[m][j]: lanes 0..63 = K K^T rows, lanes 64..127 = Q K^T rows; columns j = K rows of the same tile
            umma::gemm(tmem, umma::opnd_k(sKQ, sKQ + 32768, 128), umma::opnd_k(sKQ, sKQ + 32768, 128), 128, 64, 128, 0u);
        } else {
            // ONE product over the stacked column tiles: D[32 I + t][kc_row(I') + j].  Only the blocks I' = I are meaningful (the
            // anchors of the two operands match there) and read back; the others are finite and ignored.  An MMA costs
            // (4 KB of A + 32 N bytes of B) / 128 B per cycle, so N = 160 once is far cheaper than N = 32 four times.
            umma::gemm(tmem, umma::opnd_k(sKQ, sKQ + 32768, 128), umma::opnd_k(base, base + KC_ALL_BYTES, KC_ALL_ROWS), 128, KC_ALL_ROWS, 128, 0u);
        }
        umma::commit(&sh.mm1);
        umma::wait_mma(&sh.op2, it & 1);
        fresh();
        const umma::Opnd bA = umma::opnd_k(base + TA_OFF, base + TA_OFF + 8192, 64);
        umma::gemm(tmem + 128, umma::opnd_mn(base, base + 16384, 64), bA, 128, 64, 64, 0u);
        umma::commit(&sh.mmN);
        umma::gemm(tmem + 192, umma::opnd_mn(base + 32768, base + 32768 + 16384, 64), bA, 128, 64, 64, 0u);
        umma::commit(&sh.mmU);
    }
}

// SCALAR: the gate is one decay per token (the same cumsum in all 128 channels).  It then commutes with the contraction
// over channels, Gamma_ij = (k_i . k_j) 2^(g_i - g_j), so the products are plain K K^T / Q K^T (one product over a stacked
// [K; Q] tile) and the decay is applied to the accumulators, element by element and for i >= j only: nothing is anchored,
// no exponent is ever positive, and any g <= 0 is in range (the per-channel path needs g >= -5 per token).
template <int DT, bool SCALAR, bool TMA>
__global__ void __launch_bounds__(INTRA_THREADS, 1) intra_fwd_tc_kernel(const MkdaIntraFwd p, const __grid_constant__ IntraMaps maps) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ IntraShared sh;
    // cumsum rows of the four block anchors, [4] = last valid row; first the lower then the upper four of every eight channels, so that the
    // 16 threads of a row read them without bank conflicts
    __shared__ __align__(16) float sGa[5][DK], sStep[2][DK];      // anchor rows; 2^(ga[I] - ga[I - 1]) of I = 2, 3
    __shared__ __align__(16) float sGsb[2][CH];                      // SCALAR: the cumsum of every row (rows past the end: the last valid one)
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sKQ = base + KQ_OFF;
    float* sM = reinterpret_cast<float*>(base + OPND_BYTES + 32768);
    float* sInv = sM + CH * MLD;
    uint8_t* sBk = base;                               // phase 3: beta k~ [j][K index], hi 16 KB + lo 16 KB
    uint8_t* sBv = base + 32768;                       // beta v [j][v]
    uint8_t* sTA = base + TA_OFF;                       // A [i][j], hi 8 KB + lo 8 KB
    uint8_t* sTQ = base + 81920;                       // Aqk [i][j], hi 8 KB + lo 8 KB (only copied out)
    uint8_t* sKB = base + OPND_BYTES;                  // kbar [tok][K index] hi + lo (32 KB), only copied out; later the q rows of the next item
    uint8_t* sQS = sKB + 32768;                        // scale q 2^g [tok][K index] hi + lo (32 KB), likewise; under sM and sInv

    const int HV = p.L.HV, HK = p.L.HK, total = p.L.NC * HV, stride = gridDim.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, cg = warp >> 2, row = q * 32 + lane;

    // Persistent: one CTA per SM walks the (chunk, v-head) items gridDim.x apart, heads fastest.  The k, q, g rows of the NEXT item are
    // requested as soon as the current item has no more use for their place, half way through the item, so that they travel while the
    // inverse and the second products run.  beta (and a scalar gate's cumsum) come by asynchronous copies into the other half of a double
    // buffer: a value that is loaded into a register under a condition is waited for where the paths join again (2 k cycles per item).
    constexpr bool BULK = TMA && DT != MKDA_F32;       // fp32 rows would not fit: they travel through registers
    f32x2 vk[2][4], vq[2][4], vg[2][4];
    Raw8 wk[2], wq[2];
    uint32_t nin = 0;                                  // phase counter of the input-row barrier
    struct Item { int c, h, hk, start, len; } cur, nxt;
    const int G = HV / HK, dc = stride / HV, dh = stride - dc * HV;
    const float rG = 1.f / (float)G;
    auto advance = [&](Item& i) { i.c += dc; i.h += dh; if (i.h >= HV) { i.h -= HV; ++i.c; } i.hk = (int)(((float)i.h + 0.5f) * rG); };
    auto table = [&](Item& i) { const int c = min(i.c, p.L.NC - 1); i.start = p.L.chunk_start[c]; i.len = p.L.chunk_len[c]; };
    auto load_inputs = [&](const Item& i, int buf) {
        if (tid < CH) cp_async4(&sh.beta[buf][tid], p.beta + (size_t)(i.start + min(tid, i.len - 1)) * HV + i.h);
        else if (SCALAR && tid < 2 * CH) cp_async4(&sGsb[buf][tid - CH], p.g_c + (size_t)(i.start + min(tid - CH, i.len - 1)) * HV + i.h);
        if (BULK && tid == 128) {                      // rows past the chunk's end belong to the next sequence (or read as zeros) and are never used
            umma::mbar_expect_tx(&sh.ldin, 16384u + 16384u + (SCALAR ? 0u : 32768u));
            umma::tma_load_rows(base + RAW_K, &maps.k, i.hk * 128, i.start, &sh.ldin);
            if (!SCALAR) umma::tma_load_rows(base + RAW_G, &maps.g, i.h * 128, i.start, &sh.ldin);
        }
        if (!BULK) {
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int r = (tid + n * 512) >> 4, k8 = tid & 15, rr = min(r, i.len - 1);
                const size_t tk = (size_t)(i.start + rr) * HK + i.hk;
                ldraw8<DT>(p.k, tk * 128 + k8 * 8, wk[n]);
                ldraw8<DT>(p.q, tk * 128 + k8 * 8, wq[n]);
                if (!SCALAR) lds8(p.g_c + ((size_t)(i.start + rr) * HV + i.h) * 128 + k8 * 8, vg[n]);
            }
        }
    };
    auto load_q = [&](const Item& i) { umma::tma_load_rows(base + RAW_Q, &maps.q, i.hk * 128, i.start, &sh.ldin); };
    if (warp == 0) umma::tmem_alloc(&sh.tmem, 256);
    if (tid == 0) { 
        for (uint64_t* b : {&sh.ldin, &sh.mm1, &sh.mmN, &sh.mmU}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.op1, &sh.op2}) umma::mbar_init(b, 16);
        umma::fence_barrier_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = sh.tmem;
    follow_stream();
    if (warp >= INTRA_WARP_MMA) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == INTRA_WARP_MMA && umma::elect_one()) intra_issue<SCALAR>(base, tmem, total, sh);
        __syncwarp();
    } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    cur.c = blockIdx.x / HV; cur.h = blockIdx.x - cur.c * HV; cur.hk = cur.h / G;
    table(cur);
    if ((int)blockIdx.x < total) {
        load_inputs(cur, 0);
        if (BULK && tid == STORER) load_q(cur);
    }
    nxt = cur;
    advance(nxt);

    for (int item = blockIdx.x, it = 0; item < total; item += stride, ++it) {
    const int c = cur.c, h = cur.h, hk = cur.hk, start = cur.start, len = cur.len;
    float* sBeta = sh.beta[it & 1];
    const float* sGs = sGsb[it & 1];
    table(nxt);                                        // the chunk table entries are read ahead of load_inputs: every address depends on them
    // ---- phase 0: this item's k, q, g rows into registers; park the anchor rows of g in shared memory ----
    cp_async_wait_all();
    if (tid < CH && tid >= len) sBeta[tid] = 0.f;
    if (BULK) {
        umma::mbar_wait(&sh.ldin, nin & 1); ++nin;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int i = tid + n * 512, r = i >> 4, k8 = i & 15, rr = r < len ? r : len - 1;
            wk[n].a = *reinterpret_cast<const uint4*>(base + RAW_K + rr * 256 + k8 * 16);
            wq[n].a = *reinterpret_cast<const uint4*>(base + RAW_Q + rr * 256 + k8 * 16);
            if (!SCALAR) lds8(reinterpret_cast<const float*>(base + RAW_G + rr * 512 + k8 * 32), vg[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int i = tid + n * 512, r = i >> 4, k8 = i & 15;
        if (!SCALAR && (r & 15) == 0) sts_halves(sGa[r >> 4], k8, vg[n]);
        if (!SCALAR && r == len - 1) sts_halves(sGa[4], k8, vg[n]);
        if (!SCALAR && (r & 15) == 0 && r >= 32) {
            const int rp = r - 16 < len ? r - 16 : len - 1;
            f32x2 prev[4];
            if (BULK) lds8(reinterpret_cast<const float*>(base + RAW_G + rp * 512 + k8 * 32), prev);
            else lds8(p.g_c + ((size_t)(start + rp) * HV + h) * 128 + k8 * 8, prev);
#pragma unroll
            for (int e = 0; e < 4; ++e) prev[e] = ex2f2_(sub2(vg[n][e], prev[e]));
            sts_halves(sStep[(r >> 4) - 2], k8, prev);
        }
        if (r >= len) {                                    // rows past the end are zero
            wk[n].a = wq[n].a = make_uint4(0, 0, 0, 0);
            if (DT == MKDA_F32) wk[n].b = wq[n].b = make_uint4(0, 0, 0, 0);
        }
        unpack8<DT>(wk[n], vk[n]);
        unpack8<DT>(wq[n], vq[n]);
    }
    if (tid == STORER) umma::bulk_store_wait_read();   // the previous item's tiles have left shared memory
    umma::fence_before_sync();
    sync_compute();
    umma::fence_after_sync();
    // ---- operands ---------------------------------------------------------------------------------------------------
    if (SCALAR) {          // one stacked tile: rows 0..63 = k, rows 64..127 = q (L2 statistics applied, zero past the end)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int i = tid + n * 512, r = i >> 4, k8 = i & 15;
            store_split8(sKQ, sKQ + 32768, 128, r, k8, vk[n]);
            store_split8(sKQ, sKQ + 32768, 128, 64 + r, k8, vq[n]);
        }
    } else {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int i = tid + n * 512, r = i >> 4, k8 = i & 15, I0 = r >> 4;
            f32x2 ga[4], t8[4], e8[4];
            lds_halves(sGa[I0], k8, ga);
#pragma unroll
            for (int e = 0; e < 4; ++e) { e8[e] = mul2(ex2f2_(sub2(vg[n][e], ga[e])), both(ROW_UP)); t8[e] = mul2(vk[n][e], e8[e]); }
            store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + (r & 15), k8, t8);
#pragma unroll
            for (int e = 0; e < 4; ++e) t8[e] = mul2(vq[n][e], e8[e]);
            store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + 16 + (r & 15), k8, t8);
            f32x2 kd[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) kd[e] = mul2(vk[n][e], both(COL_DOWN));
#pragma unroll
            for (int I = 0; I < 4; ++I) {
                if (I < I0) continue;
                if (I <= I0 + 1) {
                    if (I > I0) lds_halves(sGa[I], k8, ga);
                    scale_ex2(t8, kd, ga, vg[n]);
                } else {                                   // a step of decay (<= 1) further down the anchors: exponentials are what bounds this phase
                    lds_halves(sStep[I - 2], k8, ga);
#pragma unroll
                    for (int e = 0; e < 4; ++e) t8[e] = mul2(t8[e], ga[e]);
                }
                store_split8(base, base + KC_ALL_BYTES, KC_ALL_ROWS, kc_row(I) + r, k8, t8);      // the four column tiles stacked by rows
            }
        }
    }
    umma::signal(&sh.op1, lane);
    // The L2 scales are applied to what comes out (Gamma and Q K^T are bilinear in the rows) and to the tiles below: finding them takes no
    // time while the products run.  Four sums (k, q of two rows) over the 16 threads of a row; lane bits 3 and 2 end up spelling the sum.
    float fk[2] = {1.f, 1.f}, fq[2] = {1.f, 1.f};
    if (p.l2) {
        float t[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            f32x2 a = mul2(vk[n][0], vk[n][0]), b = mul2(vq[n][0], vq[n][0]);
#pragma unroll
            for (int e = 1; e < 4; ++e) { a = fma2(vk[n][e], vk[n][e], a); b = fma2(vq[n][e], vq[n][e], b); }
            float a0, a1, b0, b1;
            unpack2(a, a0, a1);
            unpack2(b, b0, b1);
            t[2 * n] = a0 + a1;
            t[2 * n + 1] = b0 + b1;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float recv = __shfl_xor_sync(0xffffffffu, (lane & 8) ? t[j] : t[j + 2], 8);
            t[j] = ((lane & 8) ? t[j + 2] : t[j]) + recv;
        }
        const float recv = __shfl_xor_sync(0xffffffffu, (lane & 4) ? t[0] : t[1], 4);
        float s = ((lane & 4) ? t[1] : t[0]) + recv;
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s = rsqrtf(s + p.l2_eps);
        const int rr = (tid >> 4) + 4 * (lane & 8);
        if ((lane & 3) == 0) {
            ((lane & 4) ? sh.rq : sh.rk)[rr] = s;
            if (p.k_rstd_out && h == hk * G && rr < len)                   // the backward pass reads them
                ((lane & 4) ? p.q_rstd_out : p.k_rstd_out)[(size_t)(start + rr) * HK + hk] = s;
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            fk[n] = __shfl_sync(0xffffffffu, s, (lane & 16) | (8 * n));
            fq[n] = __shfl_sync(0xffffffffu, s, (lane & 16) | (8 * n + 4));
        }
    } else {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int r = (tid + n * 512) >> 4;
            if (p.k_rstd) {
                const size_t tk = (size_t)(start + min(r, len - 1)) * HK + hk;
                fk[n] = p.k_rstd[tk];
                fq[n] = p.q_rstd[tk];
            }
            if ((lane & 15) == 0) { sh.rk[r] = fk[n]; sh.rq[r] = fq[n]; }
        }
    }
    // v for phase 3 is fetched while the products run
    Raw8 wv[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int i = tid + n * 512, r = i >> 4, k8 = i & 15, rr = r < len ? r : len - 1;
        ldraw8<DT>(p.v, ((size_t)(start + rr) * HV + h) * 128 + k8 * 8, wv[n]);
    }
    // ... and so are the hand-over tiles, built and sent off in the shadow of the products
    // The state kernels' scaled operands, as ready-made tiles: kbar = k 2^(gL - g) (gL = last valid row) and scale q 2^g,
    // plus gl = 2^gL.  Rows past the end are zero (their k / q were zeroed above).
    {
        f32x2 gLv[4];
        if (!SCALAR) lds_halves(sGa[4], tid & 15, gLv);
        const float gLs = SCALAR ? sGs[CH - 1] : 0.f;      // rows past the end carry the last valid one's
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int i = tid + n * 512, r = i >> 4, k8 = i & 15;
            f32x2 t8[4];
            const f32x2 sk = both(SCALAR ? fk[n] * ex2f_(gLs - sGs[r]) : fk[n]), sq = both(SCALAR ? fq[n] * p.scale * ex2f_(sGs[r]) : fq[n] * p.scale);
            if (SCALAR) {
#pragma unroll
                for (int e = 0; e < 4; ++e) t8[e] = mul2(vk[n][e], sk);
            } else {
                scale_ex2(t8, vk[n], gLv, vg[n]);
#pragma unroll
                for (int e = 0; e < 4; ++e) t8[e] = mul2(t8[e], sk);
            }
            store_split8(sKB, sKB + 16384, 64, r, k8, t8);
#pragma unroll
            for (int e = 0; e < 4; ++e) t8[e] = SCALAR ? mul2(vq[n][e], sq) : mul2(mul2(vq[n][e], sq), ex2f2_(vg[n][e]));
            store_split8(sQS, sQS + 16384, 64, r, k8, t8);
        }
        if (SCALAR && tid < DK) p.gl[((size_t)c * HV + h) * 128 + tid] = ex2f_(gLs);
        if (!SCALAR && tid < 16) {
            f32x2 e8[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) e8[e] = ex2f2_(gLv[e]);
            sts8(p.gl + ((size_t)c * HV + h) * 128 + tid * 8, e8);
        }
    }
    umma::fence_async_smem();
    sync_compute();
    if (tid == STORER) {                               // qs first: its place is needed first
        const size_t it = (size_t)c * HV + h;
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.qs) + it * umma::CHUNK_TILE_BYTES, sQS, umma::CHUNK_TILE_BYTES);
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.kbar) + it * umma::CHUNK_TILE_BYTES, sKB, umma::CHUNK_TILE_BYTES);
    }
    umma::wait_mma(&sh.mm1, it & 1);
    // phase-3 operands over the dead phase-1 tiles: beta k 2^g and beta v (rows past the end are zero)
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const int i = tid + n * 512, r = i >> 4, k8 = i & 15;
        const float b = sBeta[r];            // 0 for rows past the end
        const f32x2 b2 = both(b), fb = both(SCALAR ? b * fk[n] * ex2f_(sGs[r]) : b * fk[n]);
        f32x2 t8[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) t8[e] = SCALAR ? mul2(vk[n][e], fb) : mul2(mul2(vk[n][e], fb), ex2f2_(vg[n][e]));
        store_split8(sBk, sBk + 16384, 64, r, k8, t8);
        unpack8<DT>(wv[n], t8);
#pragma unroll
        for (int e = 0; e < 4; ++e) t8[e] = mul2(t8[e], b2);
        store_split8(sBv, sBv + 16384, 64, r, k8, t8);
    }
    if (tid == STORER) umma::bulk_store_wait_read_but<1>();        // the tile under sM / sInv has left shared memory
    sync_compute();
    if (item + stride < total) load_inputs(nxt, (it & 1) ^ 1);     // k, q, g, beta of the next item start travelling
    sInv[(32 * (tid >> 8) + ((tid >> 4) & 15)) * MLD + 32 * (tid >> 8) + 16 + (tid & 15)] = 0.f;       // blocks (0, 1) and (2, 3)
    auto store_row16 = [](float* dst, const float (&o)[16]) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
    };
    auto store_aqk = [&](int i, const float (&o)[16]) {        // Aqk leaves as a ready-made [row][column] operand tile (rows past the end: zeros)
        float lo[8], hi[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { lo[j] = o[j]; hi[j] = o[8 + j]; }
        store_split8(sTQ, sTQ + 8192, 64, i, 2 * cg, lo);
        store_split8(sTQ, sTQ + 8192, 64, i, 2 * cg + 1, hi);
    };
    if (SCALAR) {                             // lane = row (K rows, then Q rows), cg = 16 columns j: decay applied here, for i >= j only
        float v[16];
        umma::tmem_ld16(umma::tmem_addr(tmem, warp, 16 * cg), v);
        const int i = row & 63;
        const float gi = sGs[i], bi = q < 2 ? sBeta[i] * sh.rk[i] : p.scale * sh.rq[i];
        float o[16];
#pragma unroll
        for (int j4 = 0; j4 < 16; j4 += 4) {
            const float4 g4 = *reinterpret_cast<const float4*>(sGs + 16 * cg + j4), r4 = *reinterpret_cast<const float4*>(sh.rk + 16 * cg + j4);
            const float gj[4] = {g4.x, g4.y, g4.z, g4.w}, rj[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = 16 * cg + j4 + e;
                const float E = ex2f_(fminf(gi - gj[e], 0.f));
                const float w = bi * v[j4 + e] * E * rj[e];
                o[j4 + e] = j < i ? w : j > i ? 0.f : q < 2 ? 1.f : w;
            }
        }
        if (q < 2) store_row16(sM + i * MLD + 16 * cg, o);
        else store_aqk(i, o);
    } else {                                  // warp quadrant = row block I (lanes: 16 rows of Gamma, then 16 rows of Q K^T), cg = 16 columns j
        const int I = q, i = 16 * I + (lane & 15);
        const bool isq = lane >= 16;
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0.f;
        if (cg <= I) umma::tmem_ld16(umma::tmem_addr(tmem, warp, kc_row(I) + 16 * cg), v);      // warp-uniform condition
        const float bi = isq ? p.scale * sh.rq[i] : sBeta[i] * sh.rk[i];
        float o[16];
#pragma unroll
        for (int j4 = 0; j4 < 16; j4 += 4) {
            const float4 r4 = *reinterpret_cast<const float4*>(sh.rk + 16 * cg + j4);
            const float rj[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = 16 * cg + j4 + e;
                const float w = bi * v[j4 + e] * rj[e];
                o[j4 + e] = j < i ? w : j > i ? 0.f : isq ? w : 1.f;
            }
        }
        if (isq) store_aqk(i, o);
        else store_row16(sM + i * MLD + 16 * cg, o);
    }
    umma::fence_async_smem();
    sync_compute();
    if (tid == STORER) {
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.Aqk) + ((size_t)c * HV + h) * umma::QUARTER_TILE_BYTES, sTQ, umma::QUARTER_TILE_BYTES);
        if (BULK && item + stride < total) {
            umma::bulk_store_wait_read_but<1>();       // the kbar tile has left
            load_q(nxt);
        }
    }
    invert_unit_lower(sM, sInv, sh);
    {   // A as the B operand of phase 3; it also leaves as a ready-made [row][column] operand tile (rows past the end: identity rows)
        const int r = tid >> 3, k8 = tid & 7;
        float a8[8];
        lds8(sInv + r * MLD + k8 * 8, a8);
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (k8 * 8 + e > r) a8[e] = 0.f;
        store_split8(sTA, sTA + 8192, 64, r, k8, a8);
    }
    umma::signal(&sh.op2, lane);
    if (tid == STORER) {
        umma::mbar_wait(&sh.op2, it & 1);                  // all of A is there
        umma::bulk_store(reinterpret_cast<uint8_t*>(p.A) + ((size_t)c * HV + h) * umma::QUARTER_TILE_BYTES, sTA, umma::QUARTER_TILE_BYTES);
    }
    // nw^T is read out while the u^T products run
    umma::wait_mma(&sh.mmN, it & 1);
    {   // nw^T [K index][tok] leaves as a ready-made chunk tile (the serial kernels fetch it with one bulk copy; token
        // columns past the end are exact zeros: beta is 0 there)
        float a[16], n0[8], n1[8];
        umma::tmem_ld16(umma::tmem_addr(tmem, warp, 128 + 16 * cg), a);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (j < 8) n0[j] = -a[j]; else n1[j - 8] = -a[j];
        }
        store_split8(base, base + 16384, 128, row, 2 * cg, n0);          // beta k~ is dead
        store_split8(base, base + 16384, 128, row, 2 * cg + 1, n1);
    }
    umma::fence_async_smem();
    sync_compute();
    if (tid == STORER) umma::bulk_store(reinterpret_cast<uint8_t*>(p.nw) + ((size_t)c * HV + h) * umma::CHUNK_TILE_BYTES, base, umma::CHUNK_TILE_BYTES);
    {   // u^T [v][tok] leaves the same way (token columns past the end are exact zeros: A has identity rows there and
        // beta v zero rows), built next to the nw tile while that one is being copied
        float b[16], u0[8], u1[8];
        umma::wait_mma(&sh.mmU, it & 1);
        umma::tmem_ld16(umma::tmem_addr(tmem, warp, 192 + 16 * cg), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) { u0[j] = b[j]; u1[j] = b[8 + j]; }
        store_split8(base + 32768, base + 32768 + 16384, 128, row, 2 * cg, u0);
        store_split8(base + 32768, base + 32768 + 16384, 128, row, 2 * cg + 1, u1);
    }
    umma::fence_async_smem();
    sync_compute();
    if (tid == STORER) umma::bulk_store(reinterpret_cast<uint8_t*>(p.u) + ((size_t)c * HV + h) * umma::CHUNK_TILE_BYTES, base + 32768, umma::CHUNK_TILE_BYTES);
    cur = nxt;
    advance(nxt);
    }   // items
    if (tid == STORER) umma::bulk_store_wait_read();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

int tc_intra_status(unsigned int* out) {
    return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1;
}
int tc_intra_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

template <int DT, bool SCALAR, bool TMA>
static int launch_intra_fwd_tc_tt(const MkdaIntraFwd* p, const IntraMaps& maps, cudaStream_t stream) {
    auto kern = intra_fwd_tc_kernel<DT, SCALAR, TMA>;
    if (int e = ensure_smem((const void*)kern, INTRA_TC_SMEM, "intra_fwd")) return e;
    const int items = p->L.NC * p->L.HV;
    static const int regs = kernel_registers((const void*)kern);
    if (regs < INTRA_LAUNCH_REGS) return set_error(MKDA_ERR_LAUNCH, "intra_fwd: built with fewer registers than its warps redistribute");
    launch(kern, items < sm_count() ? items : sm_count(), INTRA_THREADS, INTRA_TC_SMEM, stream, *p, maps);
    return check_launch("intra_fwd");
}
template <int DT, bool SCALAR>
static int launch_intra_fwd_tc_t(const MkdaIntraFwd* p, cudaStream_t stream) {
    IntraMaps maps;
    memset(&maps, 0, sizeof(maps));
    // 16-bit rows travel by tiled copy when the tensors can be described (16-byte aligned); otherwise through registers
    if (DT != MKDA_F32 && make_rows_map(&maps.k, p->k, 2, (unsigned long long)p->L.TT, (unsigned long long)p->L.HK * 128, "intra_fwd") == MKDA_OK &&
        make_rows_map(&maps.q, p->q, 2, (unsigned long long)p->L.TT, (unsigned long long)p->L.HK * 128, "intra_fwd") == MKDA_OK &&
        (SCALAR || make_rows_map(&maps.g, p->g_c, 4, (unsigned long long)p->L.TT, (unsigned long long)p->L.HV * 128, "intra_fwd") == MKDA_OK))
        return launch_intra_fwd_tc_tt<DT, SCALAR, true>(p, maps, stream);
    return launch_intra_fwd_tc_tt<DT, SCALAR, false>(p, maps, stream);
}
int launch_intra_fwd_tc(const MkdaIntraFwd* p, cudaStream_t stream) {
    switch (p->qkv_dtype * 2 + (p->scalar_gate ? 1 : 0)) {
        case MKDA_F32 * 2: return launch_intra_fwd_tc_t<MKDA_F32, false>(p, stream);
        case MKDA_BF16 * 2: return launch_intra_fwd_tc_t<MKDA_BF16, false>(p, stream);
        case MKDA_F16 * 2: return launch_intra_fwd_tc_t<MKDA_F16, false>(p, stream);
        case MKDA_F32 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_F32, true>(p, stream);
        case MKDA_BF16 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_BF16, true>(p, stream);
        case MKDA_F16 * 2 + 1: return launch_intra_fwd_tc_t<MKDA_F16, true>(p, stream);
    }
    return set_error(MKDA_ERR_ARG, "intra_fwd: unsupported dtype");
}

}  // namespace mkda
