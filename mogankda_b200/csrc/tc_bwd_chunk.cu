// bwd_chunk: every gradient that is local to a (chunk, v-head) once the state gradients are known, in one kernel.
//
// With S the state entering the chunk, dS' the gradient of the state leaving it, k~ = k 2^g, A = (I + strictlower(diag(beta) Gamma))^-1
// and Vd = A diag(beta) (V - k~ S) as saved by the forward pass:
//   dW = A^T dVd          dV = diag(beta) dW          dAqk = lower(dO Vd^T)
//   dL = -strictlower(A^T dA A^T) with dA = (dVd X^T) diag(beta), X = V - k~ S.  Since A diag(beta) X = Vd this is
//   dL = -strictlower(dW Vd^T): one product of tiles that exist anyway, instead of rebuilding X and a chain of three products.
//   dbeta_i = (dW X^T)_ii + (dL Gamma^T)_ii = rowsum(dW * V) - rowsum(k~ * (dW S^T)) + rowsum(k * T).  (It also is (dW Vd^T)_ii / beta_i, the
//   diagonal of the product above, for nothing; but Vd carries the errors of the state chain where V is exact: over 50 cases that came to 1.16
//   times the error against fp64, up to 6.4e-6 instead of 3.7e-6.  So V is read, by the threads that have dW in fp32.)
// State part (up = 2^g, rest = 2^(g_L - g)):
//   dq_p = scale (dO S^T) up         dk_p = -beta (dW S^T) up + (Vd dS'^T) rest        dgl = rowsum_v(S * dS')
// Intra-chunk part, E_ij = 2^(g_i - g_j) per channel (i > j), Wq = scale strictlower(dAqk), dLs = strictlower(dL):
//   dq_row_i = sum_j Wq_ij k_j E_ij        T_i = sum_j dLs_ij k_j E_ij        dk_col_j = sum_i (Wq_ij q_i + beta_i dLs_ij k_i) E_ij
//   dq = dq_p + dq_row + scale dAqk_ii k   dk = dk_p + beta T + dk_col + scale dAqk_ii q
//   dg' = q dq_p + k dk_p (read part) - k (write part) + q dq_row + beta k T - k dk_col, last row += colsum(kbar dkbar) + gl dgl
// E_ij is factored through the anchor a of i's 16-row block exactly as in the forward kernel (tc_intra.cu).  Channels go on M.  Per row
// block I (anchor a = 16 I):
//   row terms   R_I^T[c][r]  = sum_j Kc_I[j][c] W[16 I + r][j]       W = Wq (-> dq_row) or dLs (-> T); N = 16 each
//   col terms   C_I^T[c][j]  = sum_{i in I} Qr[i][c] Wq[i][j] + beta_i Kr[i][c] dLs[i][j]      N = 16 (I + 1), K = 32 over [Qr; beta Kr]_I
//
// Roles: 16 compute warps, one warp that issues every tensor-core product, one that issues every bulk copy and one that fetches tables and per-row
// scalars, joined by mbarriers only, so that no compute warp waits for an issue slot of the tensor pipe (an N <= 64 product is accepted every ~50
// cycles) or for a copy.  Twenty warps start with 96 registers; the compute warps raise theirs to 112, the four others go down to 32 (16 x 32 x 112 +
// 4 x 32 x 32 = the launch's 61 440).
//
// Products in issue order (M = 128 throughout):
//   dW[tok x v]: two products of A^T (64 rows) with the halves of dVd^T; the second one's operand is moved one 64-group up, so that its result
//     lands in lanes 64..127 and all warps read dW at once (the other 64 lanes of each accumulator are undefined and unread)
//   [D1; Z][i x j] = [dO; dW] Vd^T and [Dq | Dk]^T[c x tok] = S [dO; dW]^T over one stacked row tile: dW is written below the dO rows
//   Db^T[c x tok] = dS' Vd^T, then the row and column terms.
// Channels are lanes: of the accumulators, and so of the threads that build the left operands of the row and column terms.  A thread has k, q and g of one
// channel and 16 tokens in registers from the first use to the last; its anchors are scalars, the column tiles go into tensor memory (over Dq and Dk),
// and of the intra-chunk part only [Qr; beta Kr] and the weights are in shared memory.  That leaves room there: S and Vd of the next item travel from the
// middle of this one on, where everything used to wait for its end (232 KB at 44 B per cycle while the epilogue wrote 96 KB, and nothing before).
// (Operands by token rows, as the forward kernel builds them: k, q and g requested twice, 2.5 k cycles each time, and 144 KB of operands in shared memory.)
// dW of the next item is computed under the epilogue: Dq and Dk leave their columns early, as the starting values of the row products.
// An item takes 23 k cycles (26 k by token rows).  Now: 1B shape 180 us, short documents 230, fp16 4 x 1000 tokens 61, 64 k packed tokens x 32 heads 2.84 to 3.26 ms, scalar
// gate 4 x 16 k tokens x 16 heads 1190 us; where a launch lasts a millisecond its clock is that of the power cap, and the same launch again and again takes 1157 to 1317.
// The 1B shape on the way here: 223 by token rows, 201 by channels, 193 with the hints of rows and the loads that leave L2 first, 180 with waits that look before they
// read the clock.
// Shared memory (KB): S [0,64) | stacked [dO; dW] [64,128): 8 KB pieces, dO even, dW odd -> weights [64,96), scratch in dW pieces | Vd^T [128,160) |
// dVd^T [160,192), A [192,208) -> dS' [160,224) -> [Qr; beta Kr].
// TMEM columns: R_I 32 I; [D1; Z] 128, later C_I 128 + {0, 16, 48, 96}; dW 320, later Dq 320 and Dk 384, later column tiles 288 + {0, 16, 48, 96}; Db 448.
#include "host.h"
#include "intra.cuh"

#include <type_traits>

namespace mkda {

namespace bc {
constexpr int COMPUTE = 512, THREADS = 640, WARP_MMA = 16, WARP_LOAD = 17, WARP_ROWS = 18, LAUNCH_REGS = 96;
constexpr int KB = 1024;
constexpr int S_ = 0, R_ = 64 * KB, V_ = 128 * KB, T_ = 160 * KB, W_ = T_, A_ = 192 * KB, TILES = 224 * KB;
constexpr int WD_ = R_, KQ_ = T_;                       // [Wq; dLs] 32 KB; [Qr; beta Kr] 64 KB
// 8 KB piece i of dO (hi block 0, hi block 1, lo block 0, lo block 1) and of the dW rows stacked below it
__host__ __device__ constexpr int o_piece(int i) { return R_ + 16 * KB * i; }
__host__ __device__ constexpr int w_piece(int i) { return R_ + 16 * KB * i + 8 * KB; }
constexpr int BD_HI = o_piece(2), BD_LO = o_piece(3);   // scalar gate only: beta dLs
constexpr int SCR_ = w_piece(2), DBP_ = w_piece(3);     // scratch; partial sums of rowsum(dW * V), [8][64]
// tensor-memory columns: accumulators, and the column tiles of the row blocks as left operands (hi, then lo; 16 (I + 1) tokens, two per column) over
// Dq and Dk, which have been read by then
__host__ __device__ constexpr int ccol(int I) { return I == 0 ? 128 : I == 1 ? 144 : I == 2 ? 176 : 224; }
__host__ __device__ constexpr int kcol(int I) { return 288 + 8 * I * (I + 1); }
constexpr int D1 = 128, DQ = 320, DKB = 384, DW = DQ, DB = 448;
constexpr int KT_HI = 288, KT_LO = 320, QT_HI = 352, QT_LO = 384;      // scalar gate: k^T and q^T, 64 tokens

// what the warps need to know of an item, by a warp of its own: two items
struct alignas(16) Rows {
    float beta[CH], rk[CH], rq[CH], gs[CH];              // gs: cumsum of a scalar gate (rows past the end: the last valid one; the others are 0 there)
    int item, group, start, len, h, hk, first;
};
struct Shared {
    uint64_t fullW, fullS, fullT, rows[2];              // copies landed: (dVd, A) | (S, dO, Vd) | dS'; Rows written
    uint64_t mmW, mmL, mmT, mmI[4];                     // products done: dW | [D1; Z], Dq, Dk | Db | row and column terms of block I and the later ones
    uint64_t opW, opI[4], free;                         // compute warps done: dW tile | intra-chunk operands per row block | S, dS' and Vd are dead
    uint32_t tmem;
    Rows row[2];
};
constexpr int SMEM = TILES + (int)sizeof(Shared);
static_assert(SMEM <= 232448, "shared memory of one CTA");
// scratch of the intra-chunk part and the epilogue, over dead dW rows
struct Scratch {
    float ga[5][DK];                                    // the anchor rows of g; [4] = the last valid row
    float col[4][DK], dgl[DK], diag[CH];
    float redg[4][CH], redb[4][CH], re[CH];
};
static_assert(sizeof(Scratch) <= 8 * KB, "scratch");

// dO as bf16 rows, as in bwd_dh: full chunks' are fetched from where they are, the others' as tiles, of either the high half only.  The low half below which the
// low half of dW is stacked is zeros: written once, or, where beta dLs passes through its place, again in each epilogue (two stores per thread; fetched from a
// block of zeros in L2 8 % slower).  The products still multiply it.  This kernel gains from rows with one decay per channel (4 x 16 k tokens x 16 heads, in turn: 1527 to 1729 us
// with tiles, 1431 to 1516 with rows) and not with a scalar gate (1157 to 1317, 1233 to 1373); the pass that writes tiles, 120 us, is gone in both.
struct NoRows {};
template <class R> constexpr bool ROWS = std::is_same<R, CUtensorMap>::value;

// dq and dk by token rows, [TT,HK,128] in the type of q and k, instead of fp32 tiles: with one v-head per q/k head and no L2 norm to go back through nothing is
// left to be done.  4 x 16 k tokens x 16 heads, scalar gate, in the whole call: this kernel 1190 us (1187 with tiles: half the bytes, but 256-byte pieces 4 KB apart), and
// 237 us of qk_grad_finish less.  (Two lanes that exchange values for 4-byte stores: 3 % slower.  Rows staged in shared memory have not been tried.)
struct Finished { void *dq, *dk; };

__device__ __forceinline__ void no_low_half(uint8_t* base) {
#pragma unroll
    for (int i = 2; i < 4; ++i) *reinterpret_cast<uint4*>(base + o_piece(i) + 16 * threadIdx.x) = make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
using umma::elect_one;
using umma::signal;
using umma::wait_mma;
}  // namespace bc

// fire-and-forget fp32 addition in global memory
__device__ __forceinline__ void red_add(float* addr, float v) {
    asm volatile("red.global.add.f32 [%0], %1;" :: "l"(addr), "f"(v) : "memory");
}

// The (chunk, v-head) items of a CTA: groups (chunk, q/k head) gridDim.x apart, heads fastest (CTAs that run together read neighbouring
// memory), and inside a group the G = HV / HK v-heads that share the q/k head one after the other.  Their dq and dk contributions are
// summed where they are written: the first v-head of a group stores its fp32 tile, the others add to it (red.global.add.f32 by the same
// thread to the same address, in the fixed order of the v-heads: deterministic).  The tile lives in L2 between the two passes.
// SPREAD (few items): a group is one v-head with tiles of its own, so that no CTA works through G of them alone.
// The walk goes on by additions: every warp takes it for every item, and an integer division is some 40 instructions.
template <bool SPREAD>
struct ItemWalk {
    int c, gr, j, G, H, HV, NC, dc, dg;                    // H groups per chunk; G v-heads per q/k head
    __device__ __forceinline__ ItemWalk(const MkdaLayout& L) {
        HV = L.HV; G = HV / L.HK; H = SPREAD ? HV : L.HK; NC = L.NC; j = 0;
        c = blockIdx.x / H; gr = blockIdx.x - c * H; dc = gridDim.x / H; dg = gridDim.x - dc * H;
    }
    __device__ __forceinline__ bool valid() const { return c < NC; }
    __device__ __forceinline__ int chunk() const { return c; }
    __device__ __forceinline__ int head() const { return SPREAD ? gr : gr * G + j; }
    __device__ __forceinline__ int hk() const { return SPREAD ? gr / G : gr; }
    __device__ __forceinline__ size_t group() const { return (size_t)c * H + gr; }
    __device__ __forceinline__ size_t item() const { return (size_t)c * HV + head(); }
    __device__ __forceinline__ void next() {
        if (SPREAD || ++j == G) {
            j = 0; c += dc; gr += dg;
            if (gr >= H) { gr -= H; ++c; }
        }
    }
};
template <bool SPREAD>
__device__ __forceinline__ int item_count(const MkdaLayout& L) {
    const int groups = L.NC * (SPREAD ? L.HV : L.HK);
    return (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * (SPREAD ? 1 : L.HV / L.HK);
}

// SCALAR (one decay per token): the intra-chunk part contracts the plain k / q rows with weights that already carry
// E_ij = 2^(g_i - g_j) (i > j, never a positive exponent):  [dq_row | T]^T = K^T [Wq E; dLs E]^T (N = 128),
// dk_col^T = Q^T (Wq E) + K^T (beta dLs E); no anchors, and any g <= 0 is in range.  TMEM: [dq_row | T] 0, dk_col 128.
template <bool SCALAR, bool SPREAD>
__device__ __forceinline__ void bwd_chunk_issue(const MkdaBwdChunk& p, uint8_t* smem, bc::Shared& sh) {
    using namespace bc;
    const uint32_t tmem = sh.tmem;
    uint8_t* base = smem;
    // The base passes through an empty statement in front of each group of products: kept in registers over the loop, the operand
    // descriptors of all of them spill (the warp has 32).
    auto fresh = [&]() { base = smem; asm volatile("" : "+l"(base)); };
    uint32_t n = 0;
    auto product_dW = [&](uint32_t par) {
        umma::mbar_wait(&sh.fullW, par);
        fresh();
        const umma::Opnd a_lo = umma::opnd_mn(base + A_, base + A_ + 8192, 64);
        umma::Opnd a_hi = a_lo;                          // rows 0..63 of the operand read the 8 KB in front of each half
        a_hi.hi -= 8192; a_hi.lo -= 8192;
        umma::gemm<true>(tmem + DW, a_lo, umma::opnd_k(base + W_, base + W_ + 16384, 128), 128, 64, 64, 0u);
        umma::gemm<true>(tmem + DW + 64, a_hi, umma::opnd_k(base + W_, base + W_ + 16384, 128, 64), 128, 64, 64, 0u);
        umma::commit(&sh.mmW);
    };
    ItemWalk<SPREAD> w(p.L);
    if (w.valid()) product_dW(0);
    for (; w.valid(); ++n) {
        const uint32_t par = n & 1;
        umma::mbar_wait(&sh.fullS, par);
        wait_mma(&sh.opW, par);                          // the dW rows stand below dO; the previous item's accumulators have been read
        fresh();
        const umma::Opnd v_mn = umma::opnd_mn(base + V_, base + V_ + 16384, 128), r_k = umma::opnd_k(base + R_, base + R_ + 32768, 128);
        umma::gemm<true>(tmem + D1, r_k, v_mn, 128, 64, 128, 0u);
        umma::gemm<true>(tmem + DQ, umma::opnd_mn(base + S_, base + S_ + 32768, 128), r_k, 128, 128, 128, 0u);
        umma::commit(&sh.mmL);
        umma::mbar_wait(&sh.fullT, par);
        umma::gemm<true>(tmem + DB, umma::opnd_mn(base + T_, base + T_ + 32768, 128), v_mn, 128, 64, 128, 0u);
        umma::commit(&sh.mmT);
        fresh();
        if (SCALAR) {
            uint8_t* sWD = base + WD_;
            wait_mma(&sh.opI[0], par);
            umma::gemm_ta(tmem + 0, tmem + KT_HI, tmem + KT_LO, umma::opnd_k(sWD, sWD + 16384, 128), 128, 64, 1u);
            umma::gemm_ta(tmem + 128, tmem + QT_HI, tmem + QT_LO, umma::opnd_mn(sWD, sWD + 16384, 128, 0), 64, 64, 0u);
            umma::gemm_ta(tmem + 128, tmem + KT_HI, tmem + KT_LO, umma::opnd_mn(base + BD_HI, base + BD_LO, 64, 0), 64, 64, 1u);
        } else {
#pragma unroll
            for (int I = 3; I >= 0; --I) {                 // the column tiles arrive block by block, the largest first
                wait_mma(&sh.opI[I], par);
                fresh();
                uint8_t* sWD = base + WD_;
                uint8_t* sKQ = base + KQ_ + (I >> 1) * 16384 + (I & 1) * 64;
                const int nj = 16 * (I + 1);
                // both row terms (dq_row | T) of the block in one N = 32 product, on top of the state terms
                umma::gemm_ta(tmem + 32 * I, tmem + kcol(I), tmem + kcol(I) + nj / 2, umma::opnd_k(sWD, sWD + 16384, 128, 32 * I), 32, nj, 1u);
                umma::gemm<true>(tmem + ccol(I), umma::opnd_k(sKQ, sKQ + 32768, 128), umma::opnd_mn(sWD, sWD + 16384, 128, 32 * I), 128, nj, 32, 0u);
                if (I) umma::commit(&sh.mmI[I]);
            }
        }
        umma::commit(&sh.mmI[0]);
        w.next();
        if (w.valid()) {                                 // under the epilogue of this item
            wait_mma(&sh.mmI[0], par);                   // its place was that of left operands
            product_dW(par ^ 1);
        }
    }
}

// Do the tiles of all items (272 KB each) take more than twice L2 (126 MB)?  What comes next is hinted into L2 then.
__device__ __forceinline__ bool from_hbm(const MkdaLayout& L) { return (size_t)L.NC * L.HV > (256u << 20) / (272u << 10); }

// Every tile is read here for the last time and may leave L2 at once, which keeps what comes next: the tiles that bwd_dh has written, and the gradients for
// the kernels behind (1B shape 201 -> 193 us, fp16 4 x 1000 tokens 66 -> 63, short documents 248 -> 242, 64k packed tokens no difference).
// S and Vd of the next item are requested once the state products and dgl of the current one are done, dO, dVd and A once the intra-chunk products
// are (with a scalar gate, whose products leave the place of dVd and A alone, these two go with S and Vd), dS' once dVd and A have been read.
template <bool SCALAR, bool SPREAD, class R>
__device__ __forceinline__ void bwd_chunk_load(const MkdaBwdChunk& p, const R& rows, uint8_t* base, bc::Shared& sh) {
    using namespace bc;
    auto src = [](const void* t, size_t it, uint32_t bytes, uint32_t off = 0) { return static_cast<const uint8_t*>(t) + it * bytes + off; };
    const bool hints = from_hbm(p.L);
    auto request_s = [&](size_t it) {
        umma::mbar_expect_tx(&sh.fullS, umma::STATE_TILE_BYTES + (ROWS<R> ? 3 : 4) * umma::CHUNK_TILE_BYTES / 2);
        umma::bulk_load_last(base + S_, src(p.h, it, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES, &sh.fullS);
        umma::bulk_load_last(base + V_, src(p.Vd, it, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES, &sh.fullS);
    };
    auto request_w = [&](size_t it) {
        umma::mbar_expect_tx(&sh.fullW, umma::CHUNK_TILE_BYTES + umma::QUARTER_TILE_BYTES);
        umma::bulk_load_last(base + W_, src(p.dVd_t, it, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES, &sh.fullW);
        umma::bulk_load_last(base + A_, src(p.A, it, umma::QUARTER_TILE_BYTES), umma::QUARTER_TILE_BYTES, &sh.fullW);
    };
    uint32_t n = 0;
    ItemWalk<SPREAD> w(p.L);
    int start = 0, len = 0;                                // of the next item's chunk, read an item ahead
    auto look = [&]() {
        if (!ROWS<R> || !w.valid()) return;
        start = p.L.chunk_start[w.chunk()]; len = p.L.chunk_len[w.chunk()];
    };
    look();
    for (; w.valid(); ++n) {
        const size_t it = w.item();
        const int x = w.head() * 128;
        if (n) {
            umma::mbar_wait(&sh.mmI[0], (n & 1) ^ 1);
        } else {
            request_w(it);
            request_s(it);
        }
        if (n && !SCALAR) request_w(it);
        if constexpr (ROWS<R>) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (len == CH || !p.dO_t) umma::tma_load_rows(base + o_piece(i), &rows, x + 64 * i, start, &sh.fullS);
                else umma::bulk_load_last(base + o_piece(i), src(p.dO_t, it, umma::CHUNK_TILE_BYTES, 8192 * i), 8192, &sh.fullS);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                umma::bulk_load_last(base + o_piece(i), src(p.dO_t, it, umma::CHUNK_TILE_BYTES, 8192 * i), 8192, &sh.fullS);
        }
        umma::mbar_wait(&sh.mmW, n & 1);                 // dVd and A have been read
        umma::mbar_expect_tx(&sh.fullT, umma::STATE_TILE_BYTES);
        umma::bulk_load_last(base + T_, src(p.dh, it, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES, &sh.fullT);
        w.next();
        if (!w.valid()) break;
        look();
        const size_t in = w.item();
        // Hints for what finds no room before the epilogue (3.47 -> 3.23 ms on 64k packed tokens x 32 heads, 1315 -> 1250 us on 4 x 16k x 16 heads with a
        // scalar gate, when all of the item's tiles waited for it).  Not where the tiles of all items come close to fitting into L2 as they are: 512
        // items lose 3 % by it.
        if (hints) {
            umma::mbar_wait(&sh.mmL, n & 1);
            umma::l2_prefetch(src(p.dVd_t, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES);
            umma::l2_prefetch(src(p.A, in, umma::QUARTER_TILE_BYTES), umma::QUARTER_TILE_BYTES);
            if constexpr (ROWS<R>) {
                if (len == CH || !p.dO_t) {
                    umma::tma_prefetch_rows(&rows, w.head() * 128, start);
                    umma::tma_prefetch_rows(&rows, w.head() * 128 + 64, start);
                } else {
                    umma::l2_prefetch(src(p.dO_t, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES / 2);
                }
            } else {
                umma::l2_prefetch(src(p.dO_t, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES);
            }
            umma::l2_prefetch(src(p.dh, in, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES);
        }
        umma::mbar_wait(&sh.free, n & 1);
        if (SCALAR) request_w(in);                       // no operand of the intra-chunk products in shared memory but the weights
        request_s(in);
    }
}

// Tables and per-row scalars of item n: requested in the middle of item n - 2, written in the middle of item n - 1 to the place of those of item n - 2, which
// everyone is done with by then.
template <int DT, bool SCALAR, bool SPREAD>
__device__ __forceinline__ void bwd_chunk_rows(const MkdaBwdChunk& p, bc::Shared& sh, int lane) {
    using namespace bc;
    constexpr uint32_t ROW = DT == MKDA_F32 ? 512 : 256;
    const bool hints = from_hbm(p.L);
    uint32_t n = 0;
    for (ItemWalk<SPREAD> w(p.L); w.valid(); w.next(), ++n) {
        const int start = p.L.chunk_start[w.chunk()], len = p.L.chunk_len[w.chunk()], h = w.head(), hk = w.hk();
        Rows& r = sh.row[n & 1];
        float b[2], k[2], q[2], g[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int i = lane + 32 * m, ii = i < len ? i : len - 1;
            const size_t tk = (size_t)(start + ii) * p.L.HK + hk, tv = (size_t)(start + ii) * p.L.HV + h;
            b[m] = p.beta[tv];
            k[m] = p.k_rstd ? p.k_rstd[tk] : 1.f;
            q[m] = p.q_rstd ? p.q_rstd[tk] : 1.f;
            g[m] = SCALAR ? p.g_c[tv] : 0.f;
        }
        if (n) umma::mbar_wait(&sh.free, (n & 1) ^ 1);                   // of item n - 1: everyone is done with item n - 2
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int i = lane + 32 * m;
            r.beta[i] = i < len ? b[m] : 0.f;
            r.rk[i] = i < len ? k[m] : 0.f;
            r.rq[i] = i < len ? q[m] : 0.f;
            if (SCALAR) r.gs[i] = g[m];
        }
        if (lane == 0) {
            r.item = (int)w.item(); r.group = (int)w.group(); r.start = start; r.len = len; r.h = h; r.hk = hk; r.first = w.j == 0;
        }
        __syncwarp();
        if (lane == 0) umma::arrive(&sh.rows[n & 1]);
        __syncwarp();
        if (hints) {                                       // the rows of v, g, k and q start on their way into L2
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int i = lane + 32 * m;
                if (i >= len) continue;
                const size_t tk = ((size_t)(start + i) * p.L.HK + hk), tv = ((size_t)(start + i) * p.L.HV + h);
                umma::l2_prefetch(static_cast<const uint8_t*>(p.v) + tv * ROW, ROW);
                if (!SCALAR) umma::l2_prefetch(p.g_c + tv * 128, 512);
                if (w.j == 0) {
                    umma::l2_prefetch(static_cast<const uint8_t*>(p.k) + tk * ROW, ROW);
                    umma::l2_prefetch(static_cast<const uint8_t*>(p.q) + tk * ROW, ROW);
                }
            }
        }
    }
}

// Compute warps.  Thread (q, lane, cg): accumulator lane `row` = 32 q + lane, columns or rows [16 cg, 16 cg + 16).
template <int DT, bool SCALAR, bool SPREAD, bool FINISH, bool ROWS>
__device__ __forceinline__ void bwd_chunk_compute(const MkdaBwdChunk& p, const bc::Finished& fin, uint8_t* base, bc::Shared& sh) {
    using namespace bc;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, cg = warp >> 2, row = q * 32 + lane;
    const int HV = p.L.HV, HK = p.L.HK;
    const uint32_t tmem = sh.tmem;
    Scratch& scr = *reinterpret_cast<Scratch*>(base + SCR_);
    const bool dv_sectors = (reinterpret_cast<uintptr_t>(p.dv) & 31) == 0;
    constexpr bool KEEP = DT != MKDA_F32;                  // 16-bit rows of k and q stay in registers, two tokens each; fp32 ones are read again by the epilogue

    const int count = item_count<SPREAD>(p.L);
    for (int n = 0; n < count; ++n) {
        const uint32_t par = n & 1;
        umma::mbar_wait(&sh.rows[par], (n >> 1) & 1);
        const Rows& it = sh.row[par];
        const int hk = it.hk, h = it.h, start = it.start, len = it.len;
        // ---- dW: rows of the stacked tile, dv = beta dW, rowsum(dW * V) ----
        float dbp;                                         // this thread's 16 of the row's terms
        const int t = row & 63, v0 = (q < 2 ? 0 : 64) + 16 * cg;          // token, first of 16 values
        Raw8 wv[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) ldraw8<DT>(p.v, ((size_t)(start + (t < len ? t : len - 1)) * HV + h) * 128 + v0 + 8 * m, wv[m]);
        sync_compute();
        wait_mma(&sh.mmW, par);
        {
            float dw[16];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, DW + v0), dw);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) umma::split2(dw[8 * m + 2 * e], dw[8 * m + 2 * e + 1], hi[e], lo[e]);
                const uint32_t off = umma::tile_chunk_offset(128, 64 + t, (v0 >> 3) + m);
                *reinterpret_cast<uint4*>(base + R_ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(base + R_ + 32768 + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            signal(&sh.opW, lane);
            if (t < len) {
                const float bt = it.beta[t];
                const size_t tv = ((size_t)(start + t) * HV + h) * 128 + v0;
                if (DT != MKDA_F32 && dv_sectors) {        // a lane's 16 values are one 32-byte sector (1B shape 215 -> 213 us, short documents 266 -> 262)
                    uint32_t o[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = pack16<DT>(bt * dw[2 * j], bt * dw[2 * j + 1]);
                    st32b(static_cast<uint16_t*>(p.dv) + tv, o);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; j += 8) {
                        float o8[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) o8[e] = bt * dw[j + e];
                        st8<DT>(p.dv, tv + j, o8);
                    }
                }
            }
            f32x2 sum = 0, v2[4];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                unpack8<DT>(wv[m], v2);
#pragma unroll
                for (int e = 0; e < 4; ++e) sum = fma2(pack2(dw[8 * m + 2 * e], dw[8 * m + 2 * e + 1]), v2[e], sum);
            }
            float odd;
            unpack2(sum, dbp, odd);
            dbp += odd;
        }
        // ---- k, q, g of channel `row`, tokens 16 cg .. 16 cg + 15 (past the end: the last one's), used once the state products are under way.
        // 16-bit k and q: a lane takes eight tokens of two channels, the lanes of a pair then exchange ----
        constexpr int NR = KEEP ? 8 : 16;
        uint32_t kr[NR], qr[NR];
        float gg[16];
        {   // one running offset per tensor: it stays where the chunk ends
            const int i0 = 16 * cg + (KEEP ? 8 * (lane & 1) : 0), first = i0 < len ? i0 : len - 1;
            const size_t tk = ((size_t)(start + first) * HK + hk) * 128 + row;
            const uint32_t *kp, *qp;
            if (KEEP) {
                kp = reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.k) + (tk & ~(size_t)1));
                qp = reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.q) + (tk & ~(size_t)1));
            } else {
                kp = static_cast<const uint32_t*>(p.k) + tk;
                qp = static_cast<const uint32_t*>(p.q) + tk;
            }
            uint32_t off = 0;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                kr[r] = kp[off];
                qr[r] = qp[off];
                if (i0 + r + 1 < len) off += HK * (KEEP ? 64 : 128);
            }
        }
        if (!SCALAR) {
            const int first = 16 * cg < len ? 16 * cg : len - 1;
            const float* gp = p.g_c + ((size_t)(start + first) * HV + h) * 128 + row;
            uint32_t off = 0;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                gg[r] = gp[off];
                if (16 * cg + r + 1 < len) off += HV * 128;
            }
        }
        // ---- dgl[c] = sum_v S[c][v] dS'[c][v] from the two tiles: warp = 8 channels, lanes = v ----
        float dgl;
        umma::mbar_wait(&sh.fullS, par);
        umma::mbar_wait(&sh.fullT, par);
        {
            f32x2 sum[4] = {0, 0, 0, 0};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                f32x2 s2[4], d2[4];
                umma::load_tile8(base + S_, base + S_ + 32768, 128, lane + 32 * m, warp, s2);
                umma::load_tile8(base + T_, base + T_ + 32768, 128, lane + 32 * m, warp, d2);
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] = fma2(s2[e], d2[e], sum[e]);
            }
            float acc[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) unpack2(sum[e], acc[2 * e], acc[2 * e + 1]);
            warp_colsum(acc, lane);
            dgl = acc[0];
        }
        if (KEEP) {
            const bool odd = lane & 1;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                uint32_t (&w)[NR] = x ? qr : kr;
                uint32_t a[4], b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {              // the even and the odd channel of tokens 2 j, 2 j + 1 of the lane's eight
                    const uint32_t lo = __byte_perm(w[2 * j], w[2 * j + 1], 0x5410), hi = __byte_perm(w[2 * j], w[2 * j + 1], 0x7632);
                    b[j] = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
                    a[j] = odd ? hi : lo;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) { w[j] = odd ? b[j] : a[j]; w[4 + j % (NR / 2)] = odd ? a[j] : b[j]; }
            }
        }
        wait_mma(&sh.mmL, par);
        if ((lane & 3) == 0) scr.dgl[warp * 8 + (lane >> 2)] = dgl;
        reinterpret_cast<float*>(base + DBP_)[((q >> 1) * 4 + cg) * CH + t] = dbp;
        if (!SCALAR) {
            scr.ga[cg][row] = gg[0];
            if (cg == 3) scr.ga[4][row] = gg[15];
        }
        // ---- the state terms of dq and of T become the starting values of the row products: scale ea Dq and -ea Dk of the block in its
        // 32 columns ----
        {
            const float ea = SCALAR ? 1.f : ex2f_(gg[0]);
            const f32x2 sa = both(p.scale * ea), na = both(-ea);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int c0 = 16 * cg + 8 * hf;
                f32x2 t[4], u[4];
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DQ + c0), umma::tmem_addr(tmem, warp, DKB + c0), t, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    f32x2 ft = sa, fu = na;
                    if (SCALAR) { const f32x2 up = ex2f2_(pack2(it.gs[c0 + 2 * e], it.gs[c0 + 2 * e + 1])); ft = mul2(sa, up); fu = mul2(na, up); }
                    t[e] = mul2(ft, t[e]); u[e] = mul2(fu, u[e]);
                }
                umma::tmem_st8(umma::tmem_addr(tmem, warp, SCALAR ? c0 : 32 * cg + 8 * hf), t);
                umma::tmem_st8(umma::tmem_addr(tmem, warp, SCALAR ? 64 + c0 : 32 * cg + 16 + 8 * hf), u);
            }
        }
        // ---- weights: lanes 0..63 hold D1 = dO Vd^T, lanes 64..127 Z = dW Vd^T = -dL
        {
            const int i = row & 63;
            float d[16];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, D1 + cg * 16), d);
            const float gi = SCALAR ? it.gs[i] : 0.f, f = q < 2 ? p.scale : -1.f, bt = SCALAR ? it.beta[i] : 0.f;
            // rows of the stacked weight tile: per channel 32 I + r = Wq, 32 I + 16 + r = dLs; scalar gate [Wq E; dLs E]
            const int wrow = SCALAR ? row : 32 * (i >> 4) + (i & 15) + (q < 2 ? 0 : 16);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float w8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int j = cg * 16 + hf * 8 + e;
                    const float E = SCALAR ? ex2f_(fminf(gi - it.gs[j], 0.f)) : 1.f;
                    w8[e] = j < i && i < len ? f * d[hf * 8 + e] * E : 0.f;
                    // the diagonal scale dAqk_ii (a predicated store: selecting d[i & 15] first makes the compiler index it in local
                    // memory, which every warp then waits for behind the next barrier)
                    if (j == i && q < 2) scr.diag[i] = i < len ? p.scale * d[hf * 8 + e] : 0.f;
                }
                store_split8(base + WD_, base + WD_ + 16384, 128, wrow, 2 * cg + hf, w8);
                if (SCALAR && q >= 2) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) w8[e] *= bt;
                    store_split8(base + BD_HI, base + BD_LO, 64, i, 2 * cg + hf, w8);
                }
            }
        }
        if (SCALAR && tid < CH) scr.re[tid] = ex2f_(it.gs[CH - 1] - it.gs[tid]);
        wait_mma(&sh.mmT, par);
        umma::fence_before_sync();
        sync_compute();                                    // everyone has read S, dS', [D1; Z], Dq and Dk; diag, scratch
        umma::fence_after_sync();
        signal(&sh.free, lane);
        // ---- left operands of the intra-chunk products, by channels ----
        auto rows2 = [&](const uint32_t (&w)[NR], int pr) {                // tokens 2 pr, 2 pr + 1 of the thread's 16
            if (!KEEP) return pack2(__uint_as_float(w[(2 * pr) % NR]), __uint_as_float(w[(2 * pr + 1) % NR]));
            if (DT == MKDA_BF16) return pack2(__uint_as_float(w[pr % NR] << 16), __uint_as_float(w[pr % NR] & 0xffff0000u));
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[pr % NR]));
            return pack2(f.x, f.y);
        };
        float a0 = 0.f, a1 = 0.f, fL = 1.f, f2 = 0.f, f3 = 0.f, egL;
        if (SCALAR) {
            egL = ex2f_(it.gs[CH - 1]);
            uint32_t kh[8], kl[8], qh[8], ql[8];
#pragma unroll
            for (int r4 = 0; r4 < 4; ++r4) {
                f32x2 rk4[2], rq4[2];
                lds4(it.rk + 16 * cg + 4 * r4, rk4); lds4(it.rq + 16 * cg + 4 * r4, rq4);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float a, b;
                    unpack2(mul2(rows2(kr, 2 * r4 + e), rk4[e]), a, b);
                    umma::split2(a, b, kh[2 * r4 + e], kl[2 * r4 + e]);
                    unpack2(mul2(rows2(qr, 2 * r4 + e), rq4[e]), a, b);
                    umma::split2(a, b, qh[2 * r4 + e], ql[2 * r4 + e]);
                }
            }
            umma::tmem_st8(umma::tmem_addr(tmem, warp, KT_HI + 8 * cg), kh);
            umma::tmem_st8(umma::tmem_addr(tmem, warp, KT_LO + 8 * cg), kl);
            umma::tmem_st8(umma::tmem_addr(tmem, warp, QT_HI + 8 * cg), qh);
            umma::tmem_st8(umma::tmem_addr(tmem, warp, QT_LO + 8 * cg), ql);
            umma::tmem_wait_st();
            signal(&sh.opI[0], lane);
        } else {
            // anchors of the thread's block, of the next one (or the end of the chunk), and the steps of decay further down: every decay that an element
            // needs is a power of its distance from one of the first two times a per-thread factor
            a0 = gg[0]; a1 = scr.ga[cg + 1][row];
            const float gL = scr.ga[4][row];
            fL = ex2f_(gL - a1); egL = ex2f_(gL);
            if (cg < 2) f2 = ex2f_(scr.ga[cg + 2][row] - a1);
            if (cg < 1) f3 = ex2f_(scr.ga[cg + 3][row] - a1);
            auto kv4 = [&](int r4, f32x2 (&v)[2]) {        // k of tokens 4 r4 .. 4 r4 + 3 of the thread's 16
                f32x2 rk4[2];
                lds4(it.rk + 16 * cg + 4 * r4, rk4);
                v[0] = mul2(rows2(kr, 2 * r4), rk4[0]); v[1] = mul2(rows2(kr, 2 * r4 + 1), rk4[1]);
            };
            if (cg < 3) {                                  // warp-uniform
                f32x2 kx[8];
#pragma unroll
                for (int r4 = 0; r4 < 4; ++r4) {
                    f32x2 kv[2];
                    kv4(r4, kv);
#pragma unroll
                    for (int e = 0; e < 2; ++e) kx[2 * r4 + e] = mul2(kv[e], ex2f2_(sub2(both(a1), pack2(gg[4 * r4 + 2 * e], gg[4 * r4 + 2 * e + 1]))));
                }
                auto column_tile = [&](int I, float f) {   // (k 2^(a1 - g)) f, 16 of the 16 (I + 1) tokens of block I's tile
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int pr = 0; pr < 8; ++pr) {
                        float a, b;
                        unpack2(mul2(kx[pr], both(f)), a, b);
                        umma::split2(a, b, hi[pr], lo[pr]);
                    }
                    umma::tmem_st8(umma::tmem_addr(tmem, warp, kcol(I) + 8 * cg), hi);
                    umma::tmem_st8(umma::tmem_addr(tmem, warp, kcol(I) + 8 * (I + 1) + 8 * cg), lo);
                    umma::tmem_wait_st();
                    signal(&sh.opI[I], lane);
                };
                if (cg < 1) column_tile(3, f3);
                if (cg < 2) column_tile(cg == 0 ? 2 : 3, f2);
                column_tile(cg + 1, 1.f);
            }
            // the block's own: k 2^(a0 - g), and [Qr; beta Kr] = [q; beta k] 2^(g - a0)
            {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int r4 = 0; r4 < 4; ++r4) {
                    f32x2 kv[2];
                    kv4(r4, kv);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float a, b;
                        unpack2(mul2(kv[e], ex2f2_(sub2(both(a0), pack2(gg[4 * r4 + 2 * e], gg[4 * r4 + 2 * e + 1])))), a, b);
                        umma::split2(a, b, hi[2 * r4 + e], lo[2 * r4 + e]);
                    }
                }
                umma::tmem_st8(umma::tmem_addr(tmem, warp, kcol(cg) + 8 * cg), hi);
                umma::tmem_st8(umma::tmem_addr(tmem, warp, kcol(cg) + 8 * (cg + 1) + 8 * cg), lo);
            }
            uint8_t* sKQ = base + KQ_;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                f32x2 e8[4], t8[4], kv[2][2];
                kv4(2 * hf, kv[0]); kv4(2 * hf + 1, kv[1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) e8[e] = ex2f2_(sub2(pack2(gg[8 * hf + 2 * e], gg[8 * hf + 2 * e + 1]), both(a0)));
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float* f = (x ? it.beta : it.rq) + 16 * cg + 8 * hf;
                    f32x2 s4[2][2];
                    lds4(f, s4[0]); lds4(f + 4, s4[1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) t8[e] = mul2(mul2(x ? kv[e >> 1][e & 1] : rows2(qr, 4 * hf + e), s4[e >> 1][e & 1]), e8[e]);
                    store_split8(sKQ, sKQ + 32768, 128, row, 4 * cg + 2 * x + hf, t8);
                }
            }
            umma::tmem_wait_st();
            signal(&sh.opI[cg], lane);
        }

        // ---- epilogue: channel `row`, rows 16 cg .. 16 cg + 15 ----
        // (the rows pass through empty statements: the compiler would keep their powers and unpacked values from above, 48 registers it does not have)
#pragma unroll
        for (int r = 0; r < NR; ++r) asm volatile("" : "+r"(kr[r]), "+r"(qr[r]));
        if (!SCALAR) {
#pragma unroll
            for (int r = 0; r < 16; ++r) asm volatile("" : "+f"(gg[r]));
        }
        // With e = 2^(g - ga[cg]) (the anchor of the row block), ea = 2^ga[cg], h1 = 2^(ga[cg + 1] - g) <= 1 (ga[4] = gL), every decay an element
        // needs is one of e, 1 / e and h1 times a per-thread factor:
        //   x = dq_row / e + scale ea Dq and y = T / e - ea Dk as accumulated     z = h1 (fL Db + sum_{I > cg} f_I C_I) + C_cg / e
        //   dq = e x + d k     dk = beta e y + z + d q     dg' = q e x + k (beta e y - z)     dbeta term = k e y      (d = scale dAqk_ii)
        float raw_beta = 0.f;
        if (tid < len && p.beta_sigmoid) raw_beta = ld1(p.beta_raw, p.beta_dtype, (size_t)(start + tid) * HV + h);
        const bool first_of_group = it.first;
        const size_t obk = it.group * (size_t)(CH * DK) + row;      // dq / dk: one tile per q/k head
        float* __restrict__ oq = FINISH ? nullptr : p.dq_v + obk;
        float* __restrict__ ok = FINISH ? nullptr : p.dk_v + obk;
        constexpr int FB = DT == MKDA_F32 ? 4 : 2;
        const size_t frow = (((size_t)start * HK + hk) * 128 + row) * FB;
        const uint32_t fpitch = HK * 128 * FB;
        char *fq = static_cast<char*>(fin.dq) + frow, *fk = static_cast<char*>(fin.dk) + frow;
        float* __restrict__ og = SCALAR ? p.dgp + (size_t)it.item * CH : p.dgp + it.item * (size_t)(CH * DK) + row;
        f32x2 cs2 = 0;
        float dg_last = 0.f;
        wait_mma(&sh.mmI[SCALAR ? 0 : cg], par);
        if (ROWS && SCALAR) no_low_half(base);             // for the next item's products, which follow this warp's next signal
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int c0 = 16 * cg + 8 * hf;
            f32x2 x[4], y[4], z[4];
            float kf[KEEP ? 1 : 8], qf[KEEP ? 1 : 8];
            if (!KEEP) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int i = c0 + r;
                    const size_t tk = ((size_t)(start + (i < len ? i : len - 1)) * HK + hk) * 128 + row;
                    kf[r % (KEEP ? 1 : 8)] = static_cast<const float*>(p.k)[tk];
                    qf[r % (KEEP ? 1 : 8)] = static_cast<const float*>(p.q)[tk];
                }
            }
            auto k2 = [&](int pr) { return KEEP ? rows2(kr, 4 * hf + pr) : pack2(kf[(2 * pr) % (KEEP ? 1 : 8)], kf[(2 * pr + 1) % (KEEP ? 1 : 8)]); };
            auto q2 = [&](int pr) { return KEEP ? rows2(qr, 4 * hf + pr) : pack2(qf[(2 * pr) % (KEEP ? 1 : 8)], qf[(2 * pr + 1) % (KEEP ? 1 : 8)]); };
            auto g2 = [&](int pr) { return pack2(gg[8 * hf + 2 * pr], gg[8 * hf + 2 * pr + 1]); };
            {   // z first: fewer accumulator columns in registers at a time
                f32x2 t[4], ci[4];
                if (SCALAR) {
                    umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DB + c0), umma::tmem_addr(tmem, warp, 128 + c0), t, z);
                } else {
                    umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DB + c0), umma::tmem_addr(tmem, warp, ccol(cg) + c0), t, ci);
#pragma unroll
                    for (int r = 0; r < 4; ++r) { t[r] = mul2(t[r], both(fL)); z[r] = t[r]; }
                    if (cg < 2) {                          // warp-uniform
                        f32x2 u[4], v[4];
                        umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, ccol(cg + 1) + c0), umma::tmem_addr(tmem, warp, ccol(cg + 2) + c0), u, v);
#pragma unroll
                        for (int r = 0; r < 4; ++r) z[r] = fma2(both(f2), v[r], add2(z[r], u[r]));
                    }
                    if (cg == 0 || cg == 2) {
                        f32x2 u[4];
                        umma::tmem_ld8(umma::tmem_addr(tmem, warp, ccol(3) + c0), u);
                        const float f = cg == 0 ? f3 : 1.f;
#pragma unroll
                        for (int r = 0; r < 4; ++r) z[r] = fma2(both(f), u[r], z[r]);
                    }
                }
#pragma unroll
                for (int r4 = 0; r4 < 2; ++r4) {
                    f32x2 rk4[2], re4[2];
                    lds4(it.rk + c0 + 4 * r4, rk4);
                    if (SCALAR) lds4(scr.re + c0 + 4 * r4, re4);
#pragma unroll
                    for (int r2 = 0; r2 < 2; ++r2) {
                        const int pr = 2 * r4 + r2;
                        const f32x2 kv = mul2(k2(pr), rk4[r2]);
                        if (SCALAR) {
                            const f32x2 w2 = mul2(re4[r2], t[pr]);
                            z[pr] = add2(w2, z[pr]);
                            cs2 = fma2(kv, w2, cs2);
                        } else {
                            const f32x2 ei = ex2f2_(sub2(both(a0), g2(pr))), h1 = ex2f2_(sub2(both(a1), g2(pr)));
                            z[pr] = fma2(h1, z[pr], mul2(ei, ci[pr]));
                            cs2 = fma2(mul2(kv, h1), t[pr], cs2);
                        }
                    }
                }
            }
            if (SCALAR) umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, c0), umma::tmem_addr(tmem, warp, 64 + c0), x, y);
            else umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, 32 * cg + 8 * hf), umma::tmem_addr(tmem, warp, 32 * cg + 16 + 8 * hf), x, y);
            // Rows past the end: it.rk, it.rq and it.beta are 0 there, the tiles' rows and the weights too; but 0 times what is not finite is not 0, and
            // these rows leave as zeros whatever the others hold.
            float bsv[8], dgs[8];
#pragma unroll
            for (int r4 = 0; r4 < 2; ++r4) {               // the rows' scalars four at a time: one broadcast read each instead of four
                f32x2 rk4[2], rq4[2], bt4[2], dn4[2];
                lds4(it.rk + c0 + 4 * r4, rk4); lds4(it.rq + c0 + 4 * r4, rq4); lds4(it.beta + c0 + 4 * r4, bt4); lds4(scr.diag + c0 + 4 * r4, dn4);
#pragma unroll
                for (int r2 = 0; r2 < 2; ++r2) {
                    const int pr = 2 * r4 + r2, i = c0 + 2 * pr;
                    const f32x2 kv = mul2(k2(pr), rk4[r2]), qv = mul2(q2(pr), rq4[r2]);
                    f32x2 ex = x[pr], ey = y[pr];
                    if (!SCALAR) {
                        const f32x2 e = ex2f2_(sub2(g2(pr), both(a0)));
                        ex = mul2(e, ex); ey = mul2(e, ey);
                    }
                    const f32x2 bey = mul2(bt4[r2], ey);
                    const f32x2 dg2 = fma2(qv, ex, mul2(kv, sub2(bey, z[pr]))), dq2 = fma2(dn4[r2], kv, ex), dk2 = fma2(dn4[r2], qv, add2(bey, z[pr]));
                    float dgv[2], dqv[2], dkv[2];
                    unpack2(mul2(kv, ey), bsv[2 * pr], bsv[2 * pr + 1]);
                    unpack2(dg2, dgv[0], dgv[1]); unpack2(dq2, dqv[0], dqv[1]); unpack2(dk2, dkv[0], dkv[1]);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const int io = i + o;
                        const float dq = io < len ? dqv[o] : 0.f, dk = io < len ? dkv[o] : 0.f, dg = io < len ? dgv[o] : 0.f;
                        if (FINISH) {
                            if (io < len) { st1(fq + (uint32_t)io * fpitch, DT, 0, dq); st1(fk + (uint32_t)io * fpitch, DT, 0, dk); }
                        } else if (first_of_group) { oq[io * DK] = dq; ok[io * DK] = dk; }
                        else { red_add(oq + io * DK, dq); red_add(ok + io * DK, dk); }
                        if (SCALAR) dgs[2 * pr + o] = dg;
                        else if (io == len - 1) dg_last = dg;
                        else og[io * DK] = dg;
                    }
                }
            }
            warp_colsum(bsv, lane);
            if ((lane & 3) == 0) scr.redb[q][c0 + (lane >> 2)] = bsv[0];
            if (SCALAR) {
                warp_colsum(dgs, lane);
                if ((lane & 3) == 0) scr.redg[q][c0 + (lane >> 2)] = dgs[0];
            }
        }
        float cs, cs_odd;
        unpack2(cs2, cs, cs_odd);
        cs += cs_odd;
        // gate term of the last valid row: column sum of the inter-chunk k gradient plus gl dgl
        if (SCALAR) {
            if (cg == 0) cs = fmaf(egL, scr.dgl[row], cs);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cs += __shfl_xor_sync(0xffffffffu, cs, o);
            if (lane == 0) scr.col[0][warp] = cs;
        } else {
            scr.col[cg][row] = cs;
        }
        sync_compute();
        if (!SCALAR && cg == (len - 1) >> 4)
            og[(len - 1) * DK] = dg_last + (((scr.col[0][row] + scr.col[1][row]) + (scr.col[2][row] + scr.col[3][row])) + egL * scr.dgl[row]);
        if (SCALAR && tid < CH) {
            float t = (scr.redg[0][tid] + scr.redg[1][tid]) + (scr.redg[2][tid] + scr.redg[3][tid]);
            if (tid == len - 1) {
                float e = 0.f;
#pragma unroll
                for (int k = 0; k < 16; ++k) e += scr.col[0][k];
                t += e;
            }
            og[tid] = t;
        }
        if (tid < len) {
            const float* part = reinterpret_cast<const float*>(base + DBP_) + tid;
            const float dwv = ((part[0] + part[CH]) + (part[2 * CH] + part[3 * CH])) + ((part[4 * CH] + part[5 * CH]) + (part[6 * CH] + part[7 * CH]));
            float db = dwv + ((scr.redb[0][tid] + scr.redb[1][tid]) + (scr.redb[2][tid] + scr.redb[3][tid]));
            if (p.beta_sigmoid) db *= it.beta[tid] * (1.f - sigmoidf_(raw_beta));          // beta = beta_scale sg: its derivative is beta (1 - sg)
            st1(p.dbeta, p.dbeta_dtype, (size_t)(start + tid) * HV + h, db);
        }
    }
}

template <int DT, bool SCALAR, bool SPREAD, bool FINISH, class R>
__global__ void __launch_bounds__(bc::THREADS, 1) bwd_chunk_tc_kernel(const MkdaBwdChunk p, const bc::Finished fin, const __grid_constant__ R rows) {
    using namespace bc;
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
        for (uint64_t* b : {&sh.fullW, &sh.fullS, &sh.fullT, &sh.rows[0], &sh.rows[1], &sh.mmW, &sh.mmL, &sh.mmT, &sh.mmI[0], &sh.mmI[1], &sh.mmI[2], &sh.mmI[3]}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opW, &sh.free}) umma::mbar_init(b, COMPUTE / 32);
        for (int I = 0; I < 4; ++I) umma::mbar_init(&sh.opI[I], SCALAR ? COMPUTE / 32 : 4 * (I + 1));
        umma::fence_barrier_init();
    }
    if (ROWS<R> && threadIdx.x < COMPUTE) no_low_half(base);
    publish();
    follow_stream();
    if (warp >= COMPUTE / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == WARP_MMA) {
            if (elect_one()) bwd_chunk_issue<SCALAR, SPREAD>(p, base, sh);
            __syncwarp();
        } else if (warp == WARP_LOAD) {
            if (elect_one()) bwd_chunk_load<SCALAR, SPREAD>(p, rows, base, sh);
            __syncwarp();
        } else if (warp == WARP_ROWS) {
            bwd_chunk_rows<DT, SCALAR, SPREAD>(p, sh, threadIdx.x & 31);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        bwd_chunk_compute<DT, SCALAR, SPREAD, FINISH, ROWS<R>>(p, fin, base, sh);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(sh.tmem, 512);
}

template <int DT, bool SCALAR, bool SPREAD, bool FINISH, class R>
static int launch_bwd_chunk_tc_t(const MkdaBwdChunk* p, const bc::Finished& fin, const R& rows, cudaStream_t stream) {
    auto kern = bwd_chunk_tc_kernel<DT, SCALAR, SPREAD, FINISH, R>;
    if (int e = ensure_smem((const void*)kern, bc::SMEM, "bwd_chunk")) return e;
    static const int regs = kernel_registers((const void*)kern);
    if (regs < bc::LAUNCH_REGS) return set_error(MKDA_ERR_LAUNCH, "bwd_chunk: built with fewer registers than its warps redistribute");
    const int groups = p->L.NC * (SPREAD ? p->L.HV : p->L.HK);              // a CTA takes whole (chunk, q/k head) groups
    launch(kern, groups < sm_count() ? groups : sm_count(), bc::THREADS, bc::SMEM, stream, *p, fin, rows);
    return check_launch("bwd_chunk");
}
template <int DT, bool SCALAR, class R>
static int launch_bwd_chunk_tc_r(const MkdaBwdChunk* p, const bc::Finished& fin, const R& rows, cudaStream_t stream) {
    if (fin.dq) return launch_bwd_chunk_tc_t<DT, SCALAR, true, true>(p, fin, rows, stream);
    return p->per_v_head ? launch_bwd_chunk_tc_t<DT, SCALAR, true, false>(p, fin, rows, stream) : launch_bwd_chunk_tc_t<DT, SCALAR, false, false>(p, fin, rows, stream);
}
template <int DT, bool SCALAR>
static int launch_bwd_chunk_tc_s(const MkdaBwdChunk* p, const bc::Finished& fin, const void* d_o, cudaStream_t stream) {
    if constexpr (DT == MKDA_BF16) {
        if (d_o) {
            CUtensorMap map;
            if (int e = make_rows_map(&map, d_o, 2, (unsigned long long)p->L.TT, (unsigned long long)p->L.HV * 128, "bwd_chunk", CH, 64)) return e;
            return launch_bwd_chunk_tc_r<DT, SCALAR>(p, fin, map, stream);
        }
    }
    return launch_bwd_chunk_tc_r<DT, SCALAR>(p, fin, bc::NoRows{}, stream);
}
int launch_bwd_chunk_tc(const MkdaBwdChunk* p, const void* d_o, void* dq, void* dk, cudaStream_t stream) {
    const bc::Finished fin{dq, dk};
    switch (p->qkv_dtype * 2 + (p->scalar_gate ? 1 : 0)) {
        case MKDA_F32 * 2: return launch_bwd_chunk_tc_s<MKDA_F32, false>(p, fin, d_o, stream);
        case MKDA_BF16 * 2: return launch_bwd_chunk_tc_s<MKDA_BF16, false>(p, fin, d_o, stream);
        case MKDA_F16 * 2: return launch_bwd_chunk_tc_s<MKDA_F16, false>(p, fin, d_o, stream);
        case MKDA_F32 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_F32, true>(p, fin, d_o, stream);
        case MKDA_BF16 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_BF16, true>(p, fin, d_o, stream);
        case MKDA_F16 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_F16, true>(p, fin, d_o, stream);
    }
    return set_error(MKDA_ERR_ARG, "bwd_chunk: unsupported dtype");
}

int tc_bwd_chunk_status(unsigned int* out) {
    return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1;
}
int tc_bwd_chunk_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

}  // namespace mkda
