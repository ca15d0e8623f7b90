// bwd_chunk: every gradient that is local to a (chunk, v-head) once the state gradients are known, in one kernel.
//
// With S the state entering the chunk, dS' the gradient of the state leaving it, k~ = k 2^g, A = (I + strictlower(diag(beta) Gamma))^-1
// and Vd = A diag(beta) (V - k~ S) as saved by the forward pass:
//   dW = A^T dVd          dV = diag(beta) dW          dAqk = lower(dO Vd^T)
//   dL = -strictlower(A^T dA A^T) with dA = (dVd X^T) diag(beta), X = V - k~ S.  Since A diag(beta) X = Vd this is
//   dL = -strictlower(dW Vd^T): one product of tiles that exist anyway, instead of rebuilding X and a chain of three products.
//   dbeta_i = (dW X^T)_ii + (dL Gamma^T)_ii = rowsum(dW * V) - rowsum(k~ * (dW S^T)) + rowsum(k * T).  (It also is (dW Vd^T)_ii / beta_i, the
//   diagonal of the product above, for nothing; but Vd carries the errors of the state chain where V is exact: over 50 cases that came to 1.16
//   times the error against fp64, up to 6.4e-6 instead of 3.7e-6.  So V is read (213 -> 228 us at the 1B shape, 3.15 -> 3.37 ms on 64k packed tokens),
//   and what the bf16 halves leave of dW, 2.4e-6 of the sum, is kept as a third part.)
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
// Roles: 16 compute warps, one warp that issues every tensor-core product and one that issues every bulk copy, joined by mbarriers only, so
// that no compute warp waits for an issue slot of the tensor pipe (an N <= 64 product is accepted every ~50 cycles) or for a copy.  Twenty
// warps start with 96 registers; the compute warps raise theirs to 112, the four others go down to 32 (16 x 32 x 112 + 4 x 32 x 32 = the
// launch's 61 440).
//
// Products in issue order (M = 128 throughout):
//   dW[tok x v]: two products of A^T (64 rows) with the halves of dVd^T; the second one's operand is moved one 64-group up, so that its result
//     lands in lanes 64..127 and all warps read dW at once (the other 64 lanes of each accumulator are undefined and unread)
//   [D1; Z][i x j] = [dO; dW] Vd^T and [Dq | Dk]^T[c x tok] = S [dO; dW]^T over one stacked row tile: dW is written below the dO rows
//   Db^T[c x tok] = dS' Vd^T, then the row and column terms.
// What bounds it: the tiles of an item are 272 KB, so no item can be fetched whole while another one is worked on, and an SM draws about
// 25 B per cycle from HBM.  S, dO, Vd, dVd and A of the next item travel under the epilogue, dS' under the dW phase; k, q and g are
// requested when that traffic is over and handed to the epilogue through shared memory (requested together with the tiles they wait
// behind 208 KB of copies: 6 k cycles at the top of every item and as much in the epilogue).  The products' operand reads, the copies and the
// compute warps' own accesses share the 128 B per cycle of shared memory: some 23 k cycles of the 25 k an item takes.
// dW of the next item is computed under the epilogue: Dq and Dk leave their columns early, as the starting values of the row products.
// 64k packed tokens x 32 heads: 3.80 -> 3.25 ms (3.37 with the reading of V) by that, by operand descriptors that no longer spill in the issuing warp, by row scalars
// read four at a time and by the L2 hint in the copy warp; 4 x 16k x 16 heads, scalar gate: 1355 -> 1250 us (1275).
// Shared memory (KB): S [0,64) -> [Qr; beta Kr] | stacked [dO; dW] [64,128): 8 KB pieces, dO even, dW odd -> Kc_0, Kc_1 in the dO pieces, raw k
// and q rows in the dW pieces | Vd^T [128,160) -> Kc_3 | dVd^T [160,192), A [192,208) -> dS' [160,224) -> [Wq; dLs] [160,192), Kc_2 [192,216),
// scratch [216,224).
// TMEM columns: [D1; Z] 128, later C_I 128 + {0, 16, 48, 96}; dW 320, later Dq 320 and Dk 384; R_I 32 I; Db 448.
#include "host.h"
#include "intra.cuh"

namespace mkda {

namespace bc {
constexpr int COMPUTE = 512, THREADS = 640, WARP_MMA = 16, WARP_LOAD = 17, LAUNCH_REGS = 96;
constexpr int KB = 1024;
constexpr int S_ = 0, R_ = 64 * KB, V_ = 128 * KB, T_ = 160 * KB, W_ = T_, A_ = 192 * KB, SCR_ = 216 * KB, TILES = 224 * KB;
constexpr int WD_ = T_, BD_ = V_;                       // [Wq; dLs] 32 KB; scalar gate only: beta dLs, 16 KB
// 8 KB piece i of dO (hi block 0, hi block 1, lo block 0, lo block 1) and of the dW rows stacked below it
__host__ __device__ constexpr int o_piece(int i) { return R_ + 16 * KB * i; }
__host__ __device__ constexpr int w_piece(int i) { return R_ + 16 * KB * i + 8 * KB; }
// column tiles of the row blocks, 16 (I + 1) rows
__host__ __device__ constexpr int kc_hi(int I) { return I == 0 ? o_piece(0) : I == 1 ? o_piece(1) : I == 2 ? 192 * KB : V_; }
__host__ __device__ constexpr int kc_lo(int I) { return I == 0 ? o_piece(0) + 4 * KB : I == 1 ? o_piece(2) : I == 2 ? 204 * KB : V_ + 16 * KB; }
constexpr int EARLY_GA = o_piece(3);
// over dead dO rows (pieces 0, 1): what the bf16 halves leave of dW, [64][128] bf16, 16-byte chunks swizzled with the row
__device__ __forceinline__ int rest_chunk(int t, int k8) { return o_piece(t >> 5) + (t & 31) * 256 + ((k8 ^ (t & 7)) << 4); }
// raw 16-bit k (pieces 0, 1) and q (2, 3) rows kept for the epilogue: 32 token rows of 256 bytes per piece
__device__ __forceinline__ int stash(int which, int tok) { return w_piece(2 * which + (tok >> 5)) + (tok & 31) * 256; }
__host__ __device__ constexpr int ccol(int I) { return I == 0 ? 128 : I == 1 ? 144 : I == 2 ? 176 : 224; }
// accumulator columns; dW of the next item takes the place of Dq and Dk; its rest waits in DWR (free until the column products)
constexpr int D1 = 128, DWR = 192, DQ = 320, DKB = 384, DW = DQ, DB = 448;

struct Shared {
    uint64_t fullW, fullS, fullT;                       // copies landed: (dVd, A) | (S, dO, Vd) | dS'
    uint64_t mmW, mmL, mmT, mmI[4];                     // products done: dW | [D1; Z], Dq, Dk | Db | row and column terms of block I and the later ones
    uint64_t opW, opI[4], accFree;                      // compute warps done: dW tile | intra-chunk operands per row block | scratch
    uint32_t tmem;
    alignas(16) float dgl[DK];
    float beta[CH], rk[CH], rq[CH], diag[CH], gs[CH], up[CH], dbw[CH];        // dbw: rowsum(dW * V)
};
constexpr int SMEM = TILES + (int)sizeof(Shared);
static_assert(SMEM <= 232448, "shared memory of one CTA");
// scratch of the intra-chunk part and the epilogue, inside the dS' tile (dead by then; the next item's arrives after accFree)
struct Scratch {
    float ga[5][DK];                                    // the anchor rows again, for the epilogue
    float col[4][DK];
    float redg[4][CH], redb[4][CH], re[CH];
};
static_assert(sizeof(Scratch) <= 8 * KB, "scratch");

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
            uint8_t* sKQ = base + S_;
            uint8_t* sWD = base + WD_;
            uint8_t* sBd = base + BD_;
            wait_mma(&sh.opI[0], par);
            umma::gemm<true>(tmem + 0, umma::opnd_mn(sKQ, sKQ + 32768, 128, 0), umma::opnd_k(sWD, sWD + 16384, 128), 128, 128, 64, 1u);
            umma::gemm<true>(tmem + 128, umma::opnd_mn(sKQ, sKQ + 32768, 128, 64), umma::opnd_mn(sWD, sWD + 16384, 128, 0), 128, 64, 64, 0u);
            umma::gemm<true>(tmem + 128, umma::opnd_mn(sKQ, sKQ + 32768, 128, 0), umma::opnd_mn(sBd, sBd + 8192, 64, 0), 128, 64, 64, 1u);
        } else {
#pragma unroll
            for (int I = 3; I >= 0; --I) {                 // the column tiles arrive block by block, the largest first
                wait_mma(&sh.opI[I], par);
                fresh();
                uint8_t* sKQ = base + S_;
                uint8_t* sWD = base + WD_;
                const int nj = 16 * (I + 1);
                // both row terms (dq_row | T) of the block in one N = 32 product, on top of the state terms
                umma::gemm<true>(tmem + 32 * I, umma::opnd_mn(base + kc_hi(I), base + kc_lo(I), nj), umma::opnd_k(sWD, sWD + 16384, 128, 32 * I), 128, 32, nj, 1u);
                umma::gemm<true>(tmem + ccol(I), umma::opnd_mn(sKQ, sKQ + 32768, 128, 32 * I), umma::opnd_mn(sWD, sWD + 16384, 128, 32 * I), 128, nj, 32, 0u);
                if (I) umma::commit(&sh.mmI[I]);
            }
        }
        umma::commit(&sh.mmI[0]);
        w.next();
        if (w.valid()) product_dW(par ^ 1);              // under the epilogue of this item; Dq and Dk were read before opI
    }
}

// S, dO, Vd, dVd and A of the next item are requested as soon as the intra-chunk products of the current one are done (the epilogue reads
// accumulators, the scratch and the raw rows only), dS' once dVd and A have been read and the scratch is free.
template <bool SPREAD>
__device__ __forceinline__ void bwd_chunk_load(const MkdaBwdChunk& p, uint8_t* base, bc::Shared& sh) {
    using namespace bc;
    auto src = [](const void* t, size_t it, uint32_t bytes, uint32_t off = 0) { return static_cast<const uint8_t*>(t) + it * bytes + off; };
    const bool from_hbm = (size_t)p.L.NC * p.L.HV > (256u << 20) / (272u << 10);          // twice L2 (126 MB)
    uint32_t n = 0;
    for (ItemWalk<SPREAD> w(p.L); w.valid(); ++n) {
        const size_t it = w.item();
        if (n) umma::mbar_wait(&sh.mmI[0], (n & 1) ^ 1);
        umma::mbar_expect_tx(&sh.fullW, umma::CHUNK_TILE_BYTES + umma::QUARTER_TILE_BYTES);
        umma::bulk_load(base + W_, src(p.dVd_t, it, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES, &sh.fullW);
        umma::bulk_load(base + A_, src(p.A, it, umma::QUARTER_TILE_BYTES), umma::QUARTER_TILE_BYTES, &sh.fullW);
        umma::mbar_expect_tx(&sh.fullS, umma::STATE_TILE_BYTES + 2 * umma::CHUNK_TILE_BYTES);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            umma::bulk_load(base + o_piece(i), src(p.dO_t, it, umma::CHUNK_TILE_BYTES, 8192 * i), 8192, &sh.fullS);
        umma::bulk_load(base + V_, src(p.Vd, it, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES, &sh.fullS);
        umma::bulk_load(base + S_, src(p.h, it, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES, &sh.fullS);
        umma::mbar_wait(&sh.mmW, n & 1);                 // dVd and A have been read
        umma::mbar_expect_tx(&sh.fullT, umma::STATE_TILE_BYTES);
        umma::bulk_load(base + T_, src(p.dh, it, umma::STATE_TILE_BYTES), SCR_ - T_, &sh.fullT);
        if (n) umma::mbar_wait(&sh.accFree, (n & 1) ^ 1);    // the last 8 KB are the scratch of the previous item's epilogue
        umma::bulk_load(base + SCR_, src(p.dh, it, umma::STATE_TILE_BYTES, SCR_ - T_), umma::STATE_TILE_BYTES - (SCR_ - T_), &sh.fullT);
        // Between here and the epilogue there is no room for another tile and nothing would be fetched: the next item's tiles start on their
        // way from HBM into L2 (3.47 -> 3.23 ms on 64k packed tokens x 32 heads, 1315 -> 1250 us on 4 x 16k x 16 heads with a scalar gate).
        // Not where the tiles of all items come close to fitting into L2 as they are: 512 items lose 3 % by it.
        w.next();
        if (from_hbm && w.valid()) {
            const size_t in = w.item();
            umma::mbar_wait(&sh.mmL, n & 1);
            umma::l2_prefetch(src(p.dVd_t, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES);
            umma::l2_prefetch(src(p.A, in, umma::QUARTER_TILE_BYTES), umma::QUARTER_TILE_BYTES);
            umma::l2_prefetch(src(p.dO_t, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES);
            umma::l2_prefetch(src(p.Vd, in, umma::CHUNK_TILE_BYTES), umma::CHUNK_TILE_BYTES);
            umma::l2_prefetch(src(p.h, in, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES);
            umma::l2_prefetch(src(p.dh, in, umma::STATE_TILE_BYTES), umma::STATE_TILE_BYTES);
        }
    }
}

// Compute warps.  Thread (q, lane, cg): accumulator lane `row` = 32 q + lane, columns or rows [16 cg, 16 cg + 16).
template <int DT, bool SCALAR, bool SPREAD>
__device__ __forceinline__ void bwd_chunk_compute(const MkdaBwdChunk& p, uint8_t* base, bc::Shared& sh) {
    using namespace bc;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, cg = warp >> 2, row = q * 32 + lane;
    const int HV = p.L.HV, HK = p.L.HK;
    const uint32_t tmem = sh.tmem;
    Scratch& scr = *reinterpret_cast<Scratch*>(base + SCR_);
    // cumsum rows of the four block anchors while the scratch is still dS', over dead dO rows; both copies stored as halves
    const int ga_col = ((row >> 3) << 2) + (row & 3) + ((row & 4) << 4);
    float (*early_ga)[DK] = reinterpret_cast<float (*)[DK]>(base + EARLY_GA);
    // the two token rows of a thread, of blocks 0 and 3 or 1 and 2: a row of block B enters 4 - B column tiles, so each thread writes five
    auto staged_row = [&](int m) { return m ? 32 + ((tid >> 4) ^ 16) : tid >> 4; };
    const bool dv_sectors = (reinterpret_cast<uintptr_t>(p.dv) & 31) == 0;
    constexpr bool STASH = DT != MKDA_F32;                 // fp32 rows do not fit: the epilogue reads them from global memory

    // chunk table entries and the per-row scalars (beta | L2 statistics | scalar gate) travel one item ahead: every address of an item
    // depends on the former, and a scalar stored where it is requested would be waited for there
    ItemWalk<SPREAD> w(p.L);
    int next_start = 0, next_len = 1;
    float ahead0 = 0.f, ahead1 = 0.f;
    auto row_scalars = [&](const ItemWalk<SPREAD>& it) {
        const int h = it.head(), hk = it.hk(), r = tid & (CH - 1), rr = r < next_len ? r : next_len - 1;
        const size_t tk = (size_t)(next_start + rr) * HK + hk, tv = (size_t)(next_start + rr) * HV + h;
        if (tid < CH) {
            ahead0 = r < next_len ? p.beta[tv] : 0.f;
        } else if (tid < 2 * CH) {
            ahead0 = r < next_len ? (p.k_rstd ? p.k_rstd[tk] : 1.f) : 0.f;
            ahead1 = r < next_len ? (p.q_rstd ? p.q_rstd[tk] : 1.f) : 0.f;
        } else if (SCALAR && tid < 3 * CH) {
            ahead0 = p.g_c[tv];                            // rows past the end: the last valid one
        }
    };
    if (w.valid()) {
        next_start = p.L.chunk_start[w.chunk()]; next_len = p.L.chunk_len[w.chunk()];
        row_scalars(w);
    }
    for (uint32_t n = 0; w.valid(); ++n) {
        const uint32_t par = n & 1;
        const int hk = w.hk(), h = w.head(), start = next_start, len = next_len;
        const size_t item = w.item();
        const bool first_of_group = w.j == 0;
        ItemWalk<SPREAD> nxt = w;
        nxt.next();
        {                                                  // loaded unconditionally, so in flight until used
            const int c = nxt.valid() ? nxt.chunk() : w.chunk();
            next_start = p.L.chunk_start[c]; next_len = p.L.chunk_len[c];
        }

        if (tid < CH) {
            sh.beta[tid] = ahead0;
        } else if (tid < 2 * CH) {
            sh.rk[tid - CH] = ahead0; sh.rq[tid - CH] = ahead1;
        } else if (SCALAR && tid < 3 * CH) {
            sh.gs[tid - 2 * CH] = ahead0;
            sh.up[tid - 2 * CH] = ex2f_(ahead0);
        }
        sync_compute();

        // ---- dW: rows of the stacked tile, dv = beta dW ----
        wait_mma(&sh.mmW, par);
        {
            const int t = row & 63, v0 = (q < 2 ? 0 : 64) + 16 * cg;      // token, first of 16 values
            float dw[16];
            uint32_t rest[8];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, DW + v0), dw);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) umma::split3(dw[8 * m + 2 * e], dw[8 * m + 2 * e + 1], hi[e], lo[e], rest[4 * m + e]);
                const uint32_t off = umma::tile_chunk_offset(128, 64 + t, (v0 >> 3) + m);
                *reinterpret_cast<uint4*>(base + R_ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(base + R_ + 32768 + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            umma::tmem_st8(umma::tmem_addr(tmem, warp, DWR + 8 * cg), rest);
            signal(&sh.opW, lane);
            if (t < len) {
                const float bt = sh.beta[t];
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
        }
        // ---- k, q, g, v rows, used once the state products are under way ----
        Raw8 wk[2], wq[2], wv[2];
        f32x2 vg[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int r = staged_row(m), k8 = tid & 15, rr = r < len ? r : len - 1;
            const size_t tk = ((size_t)(start + rr) * HK + hk) * 128 + k8 * 8;
            ldraw8<DT>(p.k, tk, wk[m]);
            ldraw8<DT>(p.q, tk, wq[m]);
            ldraw8<DT>(p.v, ((size_t)(start + rr) * HV + h) * 128 + k8 * 8, wv[m]);
            if (!SCALAR) lds8(p.g_c + ((size_t)(start + rr) * HV + h) * 128 + k8 * 8, vg[m]);
        }
        // ---- dgl[c] = sum_v S[c][v] dS'[c][v] from the two tiles: warp = 8 channels, lanes = v ----
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
            if ((lane & 3) == 0) sh.dgl[warp * 8 + (lane >> 2)] = acc[0];
        }
        wait_mma(&sh.mmL, par);
        {
            uint32_t r8[8];
            umma::tmem_wait_st();
            umma::tmem_ld8(umma::tmem_addr(tmem, warp, DWR + 8 * cg), r8);
            const int t = row & 63, k8 = (q < 2 ? 0 : 8) + 2 * cg;
            *reinterpret_cast<uint4*>(base + rest_chunk(t, k8)) = make_uint4(r8[0], r8[1], r8[2], r8[3]);
            *reinterpret_cast<uint4*>(base + rest_chunk(t, k8 + 1)) = make_uint4(r8[4], r8[5], r8[6], r8[7]);
        }
        // ---- rowsum(dW * V), as far as the halves of dW in the stacked tile go; the rest of dW over dead dO rows ----
        umma::mbar_wait(&sh.opW, par);                     // all of dW is there
        f32x2 dwv[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            f32x2 d2[4], v2[4];
            umma::load_tile8(base + R_, base + R_ + 32768, 128, 64 + staged_row(m), tid & 15, d2);
            unpack8<DT>(wv[m], v2);
            dwv[m] = mul2(d2[0], v2[0]);
#pragma unroll
            for (int e = 1; e < 4; ++e) dwv[m] = fma2(d2[e], v2[e], dwv[m]);
        }
        if (!SCALAR) {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int r = staged_row(m), k8 = tid & 15;
                if ((r & 15) == 0) sts_halves(early_ga[r >> 4], k8, vg[m]);
            }
        }
        sync_compute();                                    // every thread has read its part of S; anchor rows and the rest of dW visible
        {
            float t2[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                f32x2 d2[4], v2[4];
                Raw8 r;
                r.a = *reinterpret_cast<const uint4*>(base + rest_chunk(staged_row(m), tid & 15));
                unpack8<MKDA_BF16>(r, d2);
                unpack8<DT>(wv[m], v2);
#pragma unroll
                for (int e = 0; e < 4; ++e) dwv[m] = fma2(d2[e], v2[e], dwv[m]);
                float a0, a1;
                unpack2(dwv[m], a0, a1);
                t2[m] = a0 + a1;
            }
            // 16 threads per row; lane bit 3 ends up choosing between the thread's two rows
            const float recv = __shfl_xor_sync(0xffffffffu, (lane & 8) ? t2[0] : t2[1], 8);
            float t = ((lane & 8) ? t2[1] : t2[0]) + recv;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if ((lane & 7) == 0) sh.dbw[staged_row((lane >> 3) & 1)] = t;
        }
        // ---- [Qr; beta Kr] over S while Db is computed, then the weights and the column tiles ----
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int r = staged_row(m), k8 = tid & 15, I0 = r >> 4;
            const float rk = sh.rk[r], rq = sh.rq[r];
            f32x2 k8v[4], q8v[4];
            unpack8<DT>(wk[m], k8v);
            unpack8<DT>(wq[m], q8v);
            if (STASH) {
                *reinterpret_cast<uint4*>(base + stash(0, r) + k8 * 16) = wk[m].a;
                *reinterpret_cast<uint4*>(base + stash(1, r) + k8 * 16) = wq[m].a;
            }
            uint8_t* sKQ = base + S_;
            if (SCALAR) {
#pragma unroll
                for (int e = 0; e < 4; ++e) { k8v[e] = mul2(k8v[e], both(rk)); q8v[e] = mul2(q8v[e], both(rq)); }
                store_split8(sKQ, sKQ + 32768, 128, r, k8, k8v);
                store_split8(sKQ, sKQ + 32768, 128, 64 + r, k8, q8v);
            } else {
                const f32x2 kb = both(rk * sh.beta[r]), qb = both(rq);
                f32x2 ga[4];
                lds_halves(early_ga[I0], k8, ga);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const f32x2 f = ex2f2_(sub2(vg[m][e], ga[e]));
                    k8v[e] = mul2(mul2(k8v[e], kb), f);
                    q8v[e] = mul2(mul2(q8v[e], qb), f);
                }
                store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + (r & 15), k8, q8v);
                store_split8(sKQ, sKQ + 32768, 128, 32 * I0 + 16 + (r & 15), k8, k8v);
            }
        }
        // ---- the state terms of dq and of T become the starting values of the row products: scale ea Dq and -ea Dk of the block in its
        // 32 columns (over the old dW).  Dq and Dk are free from here on ----
        {
            const float ea = SCALAR ? 1.f : ex2f_(early_ga[cg][ga_col]);
            const f32x2 sa = both(p.scale * ea), na = both(-ea);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int c0 = 16 * cg + 8 * hf;
                f32x2 t[4], u[4];
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DQ + c0), umma::tmem_addr(tmem, warp, DKB + c0), t, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    f32x2 ft = sa, fu = na;
                    if (SCALAR) { const f32x2 up = pack2(sh.up[c0 + 2 * e], sh.up[c0 + 2 * e + 1]); ft = mul2(sa, up); fu = mul2(na, up); }
                    t[e] = mul2(ft, t[e]); u[e] = mul2(fu, u[e]);
                }
                umma::tmem_st8(umma::tmem_addr(tmem, warp, SCALAR ? c0 : 32 * cg + 8 * hf), t);
                umma::tmem_st8(umma::tmem_addr(tmem, warp, SCALAR ? 64 + c0 : 32 * cg + 16 + 8 * hf), u);
            }
            umma::tmem_wait_st();
        }
        wait_mma(&sh.mmT, par);
        // lanes 0..63 hold D1 = dO Vd^T, lanes 64..127 Z = dW Vd^T = -dL
        {
            const int i = row & 63;
            float d[16];
            umma::tmem_ld16(umma::tmem_addr(tmem, warp, D1 + cg * 16), d);
            const float gi = SCALAR ? sh.gs[i] : 0.f, f = q < 2 ? p.scale : -1.f, bt = SCALAR ? sh.beta[i] : 0.f;
            // rows of the stacked weight tile: per channel 32 I + r = Wq, 32 I + 16 + r = dLs; scalar gate [Wq E; dLs E]
            const int wrow = SCALAR ? row : 32 * (i >> 4) + (i & 15) + (q < 2 ? 0 : 16);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float w8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int j = cg * 16 + hf * 8 + e;
                    const float E = SCALAR ? ex2f_(fminf(gi - sh.gs[j], 0.f)) : 1.f;
                    w8[e] = j < i && i < len ? f * d[hf * 8 + e] * E : 0.f;
                    // the diagonal scale dAqk_ii (a predicated store: selecting d[i & 15] first makes the compiler index it in local
                    // memory, which every warp then waits for behind the next barrier)
                    if (j == i && q < 2) sh.diag[i] = i < len ? p.scale * d[hf * 8 + e] : 0.f;
                }
                store_split8(base + WD_, base + WD_ + 16384, 128, wrow, 2 * cg + hf, w8);
                if (SCALAR && q >= 2) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) w8[e] *= bt;
                    store_split8(base + BD_, base + BD_ + 8192, 64, i, 2 * cg + hf, w8);
                }
            }
        }
        if (SCALAR) {
            if (tid < CH) scr.re[tid] = ex2f_(sh.gs[CH - 1] - sh.gs[tid]);
        } else {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int r = staged_row(m), k8 = tid & 15;
                if ((r & 15) == 0) sts_halves(scr.ga[r >> 4], k8, vg[m]);
                if (r == CH - 1) sts_halves(scr.ga[4], k8, vg[m]);         // rows past the end carry the last valid row's
            }
        }
        sync_compute();                                    // diag, scratch
        if (!SCALAR) {
            f32x2 k8v[2][4];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float rk = sh.rk[staged_row(m)];
                unpack8<DT>(wk[m], k8v[m]);
#pragma unroll
                for (int e = 0; e < 4; ++e) k8v[m][e] = mul2(k8v[m][e], both(rk));
            }
            const int k8 = tid & 15;
            f32x2 ga[2][4];
            lds_halves(scr.ga[3], k8, ga[1]);
#pragma unroll
            for (int I = 3; I >= 0; --I) {
                if (I) lds_halves(scr.ga[I - 1], k8, ga[(I - 1) & 1]);      // one block ahead
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int r = staged_row(m);
                    if (r >= 16 * (I + 1)) continue;       // warp-uniform
                    f32x2 t8[4];
                    scale_ex2(t8, k8v[m], ga[I & 1], vg[m]);
                    store_split8(base + kc_hi(I), base + kc_lo(I), 16 * (I + 1), r, k8, t8);
                }
                signal(&sh.opI[I], lane);
            }
        }
        if (SCALAR) signal(&sh.opI[0], lane);

        // ---- epilogue: channel `row`, rows 16 cg .. 16 cg + 15; its inputs are fetched while the intra-chunk products run ----
        // With e = 2^(g - ga[cg]) (the anchor of the row block), ea = 2^ga[cg], h1 = 2^(ga[cg + 1] - g) <= 1 (ga[4] = gL), every decay an element
        // needs is one of e, 1 / e and h1 times a per-thread factor:
        //   x = dq_row / e + scale ea Dq and y = T / e - ea Dk as accumulated     z = h1 (fL Db + sum_{I > cg} f_I C_I) + C_cg / e
        //   dq = e x + d k     dk = beta e y + z + d q     dg' = q e x + k (beta e y - z)     dbeta term = k e y      (d = scale dAqk_ii)
        float kq[STASH ? 1 : 16], qq[STASH ? 1 : 16], gg[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int i = 16 * cg + r, ii = i < len ? i : len - 1;
            const size_t tk = ((size_t)(start + ii) * HK + hk) * 128 + row;
            if (!STASH) {
                kq[r] = ld1(p.k, DT, tk);
                qq[r] = ld1(p.q, DT, tk);
            }
            if (!SCALAR) gg[r] = p.g_c[((size_t)(start + ii) * HV + h) * 128 + row];
        }
        if (nxt.valid()) row_scalars(nxt);
        float raw_beta = 0.f;
        if (tid < len && p.beta_sigmoid) raw_beta = ld1(p.beta_raw, p.beta_dtype, (size_t)(start + tid) * HV + h);
        float a0 = 0.f, a1 = 0.f, fL = 1.f, f2 = 0.f, f3 = 0.f, egL;
        if (!SCALAR) {
            a0 = scr.ga[cg][ga_col]; a1 = scr.ga[cg + 1][ga_col];
            const float gL = scr.ga[4][ga_col];
            fL = ex2f_(gL - a1); egL = ex2f_(gL);
            if (cg < 2) f2 = ex2f_(scr.ga[cg + 2][ga_col] - a1);
            if (cg < 1) f3 = ex2f_(scr.ga[cg + 3][ga_col] - a1);
        } else {
            egL = ex2f_(sh.gs[CH - 1]);
        }
        const size_t obk = w.group() * (size_t)(CH * DK) + row;      // dq / dk: one tile per q/k head
        float* __restrict__ oq = p.dq_v + obk;
        float* __restrict__ ok = p.dk_v + obk;
        float* __restrict__ og = SCALAR ? p.dgp + item * CH : p.dgp + item * (size_t)(CH * DK) + row;
        f32x2 cs2 = 0;
        float dg_last = 0.f;
        wait_mma(&sh.mmI[SCALAR ? 0 : cg], par);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int c0 = 16 * cg + 8 * hf;
            f32x2 x[4], y[4], z[4], ci[4], t[4];
            if (SCALAR) {
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, c0), umma::tmem_addr(tmem, warp, 64 + c0), x, y);
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DB + c0), umma::tmem_addr(tmem, warp, 128 + c0), t, z);
            } else {
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, 32 * cg + 8 * hf), umma::tmem_addr(tmem, warp, 32 * cg + 16 + 8 * hf), x, y);
                umma::tmem_ld8x2(umma::tmem_addr(tmem, warp, DB + c0), umma::tmem_addr(tmem, warp, ccol(cg) + c0), t, ci);
#pragma unroll
                for (int r = 0; r < 4; ++r) { t[r] = mul2(t[r], both(fL)); z[r] = t[r]; }
                if (cg < 2) {                              // warp-uniform
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
            // Rows past the end: sh.rk and sh.rq are 0 there, every other factor is finite.
            float bsv[8], dgs[8];
#pragma unroll
            for (int r4 = 0; r4 < 2; ++r4) {               // the rows' scalars four at a time: one broadcast read each instead of four
                f32x2 rk4[2], rq4[2], bt4[2], dn4[2], re4[2];
                lds4(sh.rk + c0 + 4 * r4, rk4); lds4(sh.rq + c0 + 4 * r4, rq4); lds4(sh.beta + c0 + 4 * r4, bt4); lds4(sh.diag + c0 + 4 * r4, dn4);
                if (SCALAR) lds4(scr.re + c0 + 4 * r4, re4);
#pragma unroll
                for (int r2 = 0; r2 < 2; ++r2) {
                    const int pr = 2 * r4 + r2, i = c0 + 2 * pr, rr = 8 * hf + 2 * pr;
                    f32x2 kv, qv;
                    if (STASH) {
                        kv = pack2(ld1(base + stash(0, i), DT, row), ld1(base + stash(0, i + 1), DT, row));
                        qv = pack2(ld1(base + stash(1, i), DT, row), ld1(base + stash(1, i + 1), DT, row));
                    } else {
                        kv = pack2(kq[rr], kq[rr + 1]); qv = pack2(qq[rr], qq[rr + 1]);
                    }
                    kv = mul2(kv, rk4[r2]); qv = mul2(qv, rq4[r2]);
                    f32x2 ex, ey, zz;
                    if (SCALAR) {
                        ex = x[pr]; ey = y[pr];
                        const f32x2 w2 = mul2(re4[r2], t[pr]);
                        zz = add2(w2, z[pr]);
                        cs2 = fma2(kv, w2, cs2);
                    } else {
                        const f32x2 g = pack2(gg[rr], gg[rr + 1]);
                        const f32x2 e = ex2f2_(sub2(g, both(a0))), ei = ex2f2_(sub2(both(a0), g)), h1 = ex2f2_(sub2(both(a1), g));
                        ex = mul2(e, x[pr]); ey = mul2(e, y[pr]);
                        zz = fma2(h1, z[pr], mul2(ei, ci[pr]));
                        cs2 = fma2(mul2(kv, h1), t[pr], cs2);
                    }
                    const f32x2 bey = mul2(bt4[r2], ey);
                    const f32x2 dg2 = fma2(qv, ex, mul2(kv, sub2(bey, zz))), dq2 = fma2(dn4[r2], kv, ex), dk2 = fma2(dn4[r2], qv, add2(bey, zz));
                    float dgv[2], dqv[2], dkv[2];
                    unpack2(mul2(kv, ey), bsv[2 * pr], bsv[2 * pr + 1]);
                    unpack2(dg2, dgv[0], dgv[1]); unpack2(dq2, dqv[0], dqv[1]); unpack2(dk2, dkv[0], dkv[1]);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const int io = i + o;
                        const bool ok_row = io < len;
                        const float dg = ok_row ? dgv[o] : 0.f, dq_e = ok_row ? dqv[o] : 0.f, dk_e = ok_row ? dkv[o] : 0.f;
                        if (first_of_group) { oq[io * DK] = dq_e; ok[io * DK] = dk_e; }
                        else { red_add(oq + io * DK, dq_e); red_add(ok + io * DK, dk_e); }
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
            if (cg == 0) cs = fmaf(egL, sh.dgl[row], cs);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cs += __shfl_xor_sync(0xffffffffu, cs, o);
            if (lane == 0) scr.col[0][warp] = cs;
        } else {
            scr.col[cg][row] = cs;
        }
        sync_compute();
        if (!SCALAR && cg == (len - 1) >> 4)
            og[(len - 1) * DK] = dg_last + (((scr.col[0][row] + scr.col[1][row]) + (scr.col[2][row] + scr.col[3][row])) + egL * sh.dgl[row]);
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
            float db = sh.dbw[tid] + ((scr.redb[0][tid] + scr.redb[1][tid]) + (scr.redb[2][tid] + scr.redb[3][tid]));
            if (p.beta_sigmoid) db *= sh.beta[tid] * (1.f - sigmoidf_(raw_beta));          // beta = beta_scale sg: its derivative is beta (1 - sg)
            st1(p.dbeta, p.dbeta_dtype, (size_t)(start + tid) * HV + h, db);
        }
        signal(&sh.accFree, lane);
        w = nxt;
    }
}

template <int DT, bool SCALAR, bool SPREAD>
__global__ void __launch_bounds__(bc::THREADS, 1) bwd_chunk_tc_kernel(const MkdaBwdChunk p) {
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
        for (uint64_t* b : {&sh.fullW, &sh.fullS, &sh.fullT, &sh.mmW, &sh.mmL, &sh.mmT, &sh.mmI[0], &sh.mmI[1], &sh.mmI[2], &sh.mmI[3]}) umma::mbar_init(b, 1);
        for (uint64_t* b : {&sh.opW, &sh.opI[0], &sh.opI[1], &sh.opI[2], &sh.opI[3], &sh.accFree}) umma::mbar_init(b, COMPUTE / 32);
        umma::fence_barrier_init();
    }
    publish();
    follow_stream();
    if (warp >= COMPUTE / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == WARP_MMA) {
            if (elect_one()) bwd_chunk_issue<SCALAR, SPREAD>(p, base, sh);
            __syncwarp();
        } else if (warp == WARP_LOAD) {
            if (elect_one()) bwd_chunk_load<SPREAD>(p, base, sh);
            __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        bwd_chunk_compute<DT, SCALAR, SPREAD>(p, base, sh);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(sh.tmem, 512);
}

template <int DT, bool SCALAR, bool SPREAD>
static int launch_bwd_chunk_tc_t(const MkdaBwdChunk* p, cudaStream_t stream) {
    auto kern = bwd_chunk_tc_kernel<DT, SCALAR, SPREAD>;
    if (int e = ensure_smem((const void*)kern, bc::SMEM, "bwd_chunk")) return e;
    static const int regs = kernel_registers((const void*)kern);
    if (regs < bc::LAUNCH_REGS) return set_error(MKDA_ERR_LAUNCH, "bwd_chunk: built with fewer registers than its warps redistribute");
    const int groups = p->L.NC * (SPREAD ? p->L.HV : p->L.HK);              // a CTA takes whole (chunk, q/k head) groups
    launch(kern, groups < sm_count() ? groups : sm_count(), bc::THREADS, bc::SMEM, stream, *p);
    return check_launch("bwd_chunk");
}
template <int DT, bool SCALAR>
static int launch_bwd_chunk_tc_s(const MkdaBwdChunk* p, cudaStream_t stream) {
    return p->per_v_head ? launch_bwd_chunk_tc_t<DT, SCALAR, true>(p, stream) : launch_bwd_chunk_tc_t<DT, SCALAR, false>(p, stream);
}
int launch_bwd_chunk_tc(const MkdaBwdChunk* p, cudaStream_t stream) {
    switch (p->qkv_dtype * 2 + (p->scalar_gate ? 1 : 0)) {
        case MKDA_F32 * 2: return launch_bwd_chunk_tc_s<MKDA_F32, false>(p, stream);
        case MKDA_BF16 * 2: return launch_bwd_chunk_tc_s<MKDA_BF16, false>(p, stream);
        case MKDA_F16 * 2: return launch_bwd_chunk_tc_s<MKDA_F16, false>(p, stream);
        case MKDA_F32 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_F32, true>(p, stream);
        case MKDA_BF16 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_BF16, true>(p, stream);
        case MKDA_F16 * 2 + 1: return launch_bwd_chunk_tc_s<MKDA_F16, true>(p, stream);
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
