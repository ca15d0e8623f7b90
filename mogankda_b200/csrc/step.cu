// Forward pass over very short sequences (generation steps, speculative tokens): the recurrence itself, token by token, instead of the
// chunk algebra.
//   S <- diag(2^g) S        S <- S + k (beta (v - k^T S))        o = scale q^T S, then the optional gated RMSNorm
// The state is read and written once and everything in between, gate and L2 norm included, stays on chip.  [K,V] states: one CTA per (sequence, v-head) with the
// state in registers (thread = one v x 64 key channels).  [V,K] states: a kernel of its own (below).
// What bounds it: 128 KB of state traffic per (sequence, v-head).  The chunk path spends the same traffic several times over (operand tiles of 64 rows of
// which a few are real, and three or four launches).
// Up to how many tokens: a token costs time here, while a chunk takes the same for any number of rows.  Whole calls with cold caches, 32 heads, by steps / by chunks in us:
//                        [K,V] states: 1 token      8          16          [V,K] states: 1       8           16
//   one sequence                   14.3 / 31.7   18.5 / 31.7   28.7 / 31.7         12.3 / 33.8   16.4 / 33.8   20.4 / 33.8
//   8                              18.4 / 50.0   28.7 / 50.2   43.0 / 50.2         18.4 / 54.3   26.6 / 54.3   36.9 / 54.3
//   64                             79.9 / 269    137 / 269     223 / 273           67.6 / 302    123 / 306     197 / 310
#include "common.cuh"
#include "gate.cuh"
#include "host.h"
#include "intra.cuh"

namespace mkda {

constexpr int STEP_MAX = MKDA_STEP_MAX_TOKENS;
__device__ __forceinline__ float warp_sum_f(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// ---- [K,V] ----
struct StepShared {
    float k[STEP_MAX][DK], q[STEP_MAX][DK], d[STEP_MAX][DK], v[STEP_MAX][DV], o[STEP_MAX][DV], beta[STEP_MAX];
    float part[2][2][DV];
};

__global__ void __launch_bounds__(256, 2) step_fwd_kernel(const MkdaStepFwd p) {
    follow_stream();
    __shared__ __align__(16) StepShared sh;
    const int HV = p.L.HV, HK = p.L.HK, n = blockIdx.x / HV, h = blockIdx.x - n * HV, hk = h / (HV / HK);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int vi = tid & 127, half = tid >> 7;
    const int c = p.seq_chunk_off[n];
    const int chunks = p.seq_chunk_off[n + 1] - c;         // an empty sequence hands its state through
    const int start = chunks ? p.L.chunk_start[c] : 0, len = chunks ? p.L.chunk_len[c] : 0;
    if (p.short_only && (chunks != 1 || len > STEP_MAX)) return;

    // the state: 64 loads in flight per thread while the tokens are prepared
    float S[64];
    const size_t so = ((size_t)n * HV + h) * DK * DV;
    if (!p.h0) {
#pragma unroll
        for (int i = 0; i < 64; ++i) S[i] = 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) S[i] = p.h0[so + (size_t)(half * 64 + i) * DV + vi];
    }
    // tokens: warp w prepares w, w + 8, ...; lane = 4 channels
    const float E = p.A_log ? expf(p.A_log[h]) : 1.f;
    for (int t = warp; t < len; t += 8) {
        const size_t tk = ((size_t)(start + t) * HK + hk) * 128 + 4 * lane, th = (size_t)(start + t) * HV + h, tv = th * 128 + 4 * lane;
        const float4 k4 = ld4(p.k, p.qkv_dtype, tk), q4 = ld4(p.q, p.qkv_dtype, tk), v4 = ld4(p.v, p.qkv_dtype, tv);
        float rk = 1.f, rq = 1.f;
        if (p.l2) {
            rk = 1.f / sqrtf(warp_sum_f((k4.x * k4.x + k4.y * k4.y) + (k4.z * k4.z + k4.w * k4.w)) + 1e-6f);
            rq = 1.f / sqrtf(warp_sum_f((q4.x * q4.x + q4.y * q4.y) + (q4.z * q4.z + q4.w * q4.w)) + 1e-6f);
        }
        rq *= p.scale;
        float4 x, b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.scalar_gate) {
            const float s = ld1(p.x, p.x_dtype, th);
            x = make_float4(s, s, s, s);
            if (p.dt_bias) b.x = b.y = b.z = b.w = p.dt_bias[h];
        } else {
            x = ld4(p.x, p.x_dtype, tv);
            if (p.dt_bias) b = *reinterpret_cast<const float4*>(p.dt_bias + h * 128 + 4 * lane);
        }
        auto decay = [&](float s) { return ex2f_(gate_value(p.mode, s, E, p.lower_bound) * RCP_LN2); };
        *reinterpret_cast<float4*>(&sh.d[t][4 * lane]) = make_float4(decay(x.x + b.x), decay(x.y + b.y), decay(x.z + b.z), decay(x.w + b.w));
        *reinterpret_cast<float4*>(&sh.k[t][4 * lane]) = make_float4(k4.x * rk, k4.y * rk, k4.z * rk, k4.w * rk);
        *reinterpret_cast<float4*>(&sh.q[t][4 * lane]) = make_float4(q4.x * rq, q4.y * rq, q4.z * rq, q4.w * rq);
        *reinterpret_cast<float4*>(&sh.v[t][4 * lane]) = v4;
        if (lane == 0) {
            const float bt = ld1(p.beta, p.beta_dtype, th);
            sh.beta[t] = p.beta_sigmoid ? p.beta_scale * sigmoidf_(bt) : bt;
        }
    }
    __syncthreads();
    for (int t = 0; t < len; ++t) {
        const float *kt = &sh.k[t][half * 64], *qt = &sh.q[t][half * 64], *dt = &sh.d[t][half * 64];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(kt + i), d4 = *reinterpret_cast<const float4*>(dt + i);
            S[i] *= d4.x; S[i + 1] *= d4.y; S[i + 2] *= d4.z; S[i + 3] *= d4.w;
            a0 = fmaf(k4.x, S[i], a0); a1 = fmaf(k4.y, S[i + 1], a1); a2 = fmaf(k4.z, S[i + 2], a2); a3 = fmaf(k4.w, S[i + 3], a3);
        }
        sh.part[0][half][vi] = (a0 + a1) + (a2 + a3);
        __syncthreads();
        const float u = sh.beta[t] * (sh.v[t][vi] - (sh.part[0][0][vi] + sh.part[0][1][vi]));
        a0 = a1 = a2 = a3 = 0.f;
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(kt + i), q4 = *reinterpret_cast<const float4*>(qt + i);
            S[i] = fmaf(k4.x, u, S[i]); S[i + 1] = fmaf(k4.y, u, S[i + 1]); S[i + 2] = fmaf(k4.z, u, S[i + 2]); S[i + 3] = fmaf(k4.w, u, S[i + 3]);
            a0 = fmaf(q4.x, S[i], a0); a1 = fmaf(q4.y, S[i + 1], a1); a2 = fmaf(q4.z, S[i + 2], a2); a3 = fmaf(q4.w, S[i + 3], a3);
        }
        sh.part[1][half][vi] = (a0 + a1) + (a2 + a3);
        __syncthreads();
        if (half == 0) sh.o[t][vi] = sh.part[1][0][vi] + sh.part[1][1][vi];
    }
    if (p.ht) {
#pragma unroll
        for (int i = 0; i < 64; ++i) p.ht[so + (size_t)(half * 64 + i) * DV + vi] = S[i];
    }
    __syncthreads();
    // output rows: warp w takes tokens w, w + 8, ...; lane = 4 values
    float4 w4 = make_float4(1.f, 1.f, 1.f, 1.f);
    if (p.has_norm && p.norm_w) w4 = ld4(p.norm_w, p.norm_w_dtype, 4 * lane);
    for (int t = warp; t < len; t += 8) {
        float4 o = *reinterpret_cast<const float4*>(&sh.o[t][4 * lane]);
        const size_t off = ((size_t)(start + t) * HV + h) * 128 + 4 * lane;
        if (p.has_norm) {
            const float rs = 1.f / sqrtf(warp_sum_f((o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w)) * (1.f / 128.f) + p.eps);
            const float4 z = ld4(p.gate, p.gate_dtype, off);
            const float zz[4] = {z.x, z.y, z.z, z.w};
            float a[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float sg = sigmoidf_(zz[e]);
                a[e] = p.act == MKDA_ACT_SILU ? zz[e] * sg : sg;
            }
            o = make_float4(o.x * rs * w4.x * a[0], o.y * rs * w4.y * a[1], o.z * rs * w4.z * a[2], o.w * rs * w4.w * a[3]);
        }
        st4(p.out, p.out_dtype, off, o);
    }
}

// ---- [V,K] ----
// A row of the state is 512 bytes of one value: a warp has 8 values and all 128 key channels of them, a lane four of the channels, and sums over the channels are
// sums over a warp.  A persistent CTA per SM walks the (sequence, v-head) items: a warp of its own fetches the states of the next two into shared memory while this
// one's is updated in registers and the last one's is on its way out, and the tokens of the next item are requested before this one's are worked through.
// Launches one after another over states that are not in L2, x 32 heads, us: by the kernel above, which read and wrote such a state in 16-byte pieces 512 bytes
// apart, and by this one: one token of 1, 8, 64, 256 sequences 9.7 -> 6.3, 16.0 -> 12.6, 110 -> 61, 422 -> 223; 16 tokens 22.7 -> 15.0, 38.3 -> 30.5, 259 -> 188, 979 -> 727.
// Among longer sequences, which one warp passes over: 64 of one token and 64 of 200 116 -> 65, 8 and 248 34 -> 28, 24 and 1000 of 70 135 -> 126.
// ([K,V] states in this form: one token of 8 8.9 -> 11.3, 16 tokens of 64 218 -> 242; they stay where they are.)
namespace st {
constexpr int WARPS = 16, THREADS = 32 * (WARPS + 1), STATE = DK * DV;      // floats of a state
static_assert(STEP_MAX <= WARPS, "a warp prepares one token");
struct Shared {
    uint64_t known[2], full[2], empty[2];                  // what the item is | its state has landed | has been read
    struct { int item, start, len; } info[4];              // item < 0: no more
    int gave_up;                                           // a wait of a compute warp has
    __align__(16) float k[STEP_MAX][DK], q[STEP_MAX][DK], d[STEP_MAX][DK], v[STEP_MAX][DV], o[STEP_MAX][DV], beta[STEP_MAX];
};
constexpr int SMEM = 2 * STATE * 4 + (int)sizeof(Shared);
static_assert(SMEM <= 232448, "shared memory of one CTA");
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
// What the items are, and that there are no more, stands behind a wait: one that gives up ends the walk, for all lanes of its warp
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity)); }

// Four elements as they lie in memory, widened where they are used
__device__ __forceinline__ void ldraw4(const void* base, int dtype, size_t idx, uint4& r) {
    if (dtype == MKDA_F32) r = *reinterpret_cast<const uint4*>(static_cast<const float*>(base) + idx);
    else { const uint2 t = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + idx); r.x = t.x; r.y = t.y; }
}
__device__ __forceinline__ float4 widen4(const uint4& r, int dtype) {
    if (dtype == MKDA_F32) return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
    const uint2 t = make_uint2(r.x, r.y);
    return ld4(&t, dtype, 0);
}
}  // namespace st

// Items and their states, ahead of the compute warps.  Returns once no copy is on its way into shared memory
__device__ __forceinline__ void step_load(const MkdaStepFwd& p, float* states, st::Shared& sh, int lane) {
    using namespace st;
    const int HV = p.L.HV, items = p.N * HV;
    int j = 0;
    auto landed = [&](int i) { if (i >= 0) (void)umma::mbar_wait(&sh.full[i & 1], (i >> 1) & 1); };
    for (int it = blockIdx.x;; it += gridDim.x) {
        int start = 0, len = 0;
        if (it < items) {
            const int n = it / HV, c = p.seq_chunk_off[n], chunks = p.seq_chunk_off[n + 1] - c;        // an empty sequence hands its state through
            if (chunks) { start = p.L.chunk_start[c]; len = p.L.chunk_len[c]; }
            if (p.short_only && (chunks != 1 || len > STEP_MAX)) continue;
        }
        const int s = j & 1;
        if (j >= 2 && !wait_warp(&sh.empty[s], ((j - 2) >> 1) & 1)) break;
        if (lane == 0) {
            sh.info[j & 3] = {it < items ? it : -1, start, len};
            umma::arrive(&sh.known[s]);
        }
        if (it >= items) break;
        if (!p.h0) {
            if (lane == 0) umma::arrive(&sh.full[s]);
        } else {
            const float* src = p.h0 + (size_t)it * DK * DV;
            float* dst = states + s * STATE;
            if (lane == 0) umma::mbar_expect_tx(&sh.full[s], DK * DV * 4);
            __syncwarp();
            if (lane < 8) umma::bulk_load(dst + lane * 2048, src + lane * 2048, 8192, &sh.full[s]);
        }
        ++j;
    }
    landed(j - 2);
    landed(j - 1);
}

__global__ void __launch_bounds__(st::THREADS, 1) step_fwd_vk_kernel(const MkdaStepFwd p) {
    using namespace st;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    float* states = reinterpret_cast<float*>(smem_raw);
    Shared& sh = *reinterpret_cast<Shared*>(smem_raw + 2 * STATE * 4);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, HV = p.L.HV, HK = p.L.HK, G = HV / HK;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) { umma::mbar_init(&sh.known[i], 1); umma::mbar_init(&sh.full[i], 1); umma::mbar_init(&sh.empty[i], WARPS); }
        sh.gave_up = 0;
        umma::fence_barrier_init();
    }
    __syncthreads();
    follow_stream();
    if (warp == WARPS) return step_load(p, states, sh, lane);

    float4 w4 = make_float4(1.f, 1.f, 1.f, 1.f);
    if (p.has_norm && p.norm_w) w4 = ld4(p.norm_w, p.norm_w_dtype, 4 * lane);
    const int t = warp;                                    // the token that this warp prepares and writes
    uint4 rk, rq, rv, rx, rz;
    float rb = 0.f;
    int item = -1, start = 0, len = 0;
    volatile int* gave_up = &sh.gave_up;                   // written between two block-wide barriers, read behind the second: all compute warps leave together
    auto request = [&](int j) {                            // item j: its tokens
        item = -1;
        if (!wait_warp(&sh.known[j & 1], (j >> 1) & 1)) {
            *gave_up = 1;
            return;
        }
        item = sh.info[j & 3].item; start = sh.info[j & 3].start; len = sh.info[j & 3].len;
        if (item < 0 || t >= len) return;
        const int h = item % HV;
        const size_t tk = ((size_t)(start + t) * HK + h / G) * 128 + 4 * lane, th = (size_t)(start + t) * HV + h, tv = th * 128 + 4 * lane;
        ldraw4(p.k, p.qkv_dtype, tk, rk); ldraw4(p.q, p.qkv_dtype, tk, rq); ldraw4(p.v, p.qkv_dtype, tv, rv);
        if (!p.scalar_gate) ldraw4(p.x, p.x_dtype, tv, rx);
        else rx.x = __float_as_uint(ld1(p.x, p.x_dtype, th));
        if (p.has_norm) ldraw4(p.gate, p.gate_dtype, tv, rz);
        rb = ld1(p.beta, p.beta_dtype, th);
    };
    request(0);
    sync_compute();
    for (int j = 0, end = *gave_up; item >= 0 && !end; ++j) {
        const int h = item % HV, n_tok = len, first = start;
        const size_t so = (size_t)item * DK * DV;
        float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n_tok) {
            const float4 k4 = widen4(rk, p.qkv_dtype), q4 = widen4(rq, p.qkv_dtype), v4 = widen4(rv, p.qkv_dtype);
            float fk = 1.f, fq = 1.f;
            if (p.l2) {
                fk = 1.f / sqrtf(warp_sum_f((k4.x * k4.x + k4.y * k4.y) + (k4.z * k4.z + k4.w * k4.w)) + 1e-6f);
                fq = 1.f / sqrtf(warp_sum_f((q4.x * q4.x + q4.y * q4.y) + (q4.z * q4.z + q4.w * q4.w)) + 1e-6f);
            }
            fq *= p.scale;
            const float E = p.A_log ? expf(p.A_log[h]) : 1.f;
            float4 x, b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.scalar_gate) {
                const float g = __uint_as_float(rx.x);
                x = make_float4(g, g, g, g);
                if (p.dt_bias) b.x = b.y = b.z = b.w = p.dt_bias[h];
            } else {
                x = widen4(rx, p.x_dtype);
                if (p.dt_bias) b = *reinterpret_cast<const float4*>(p.dt_bias + h * 128 + 4 * lane);
            }
            auto decay = [&](float g) { return ex2f_(gate_value(p.mode, g, E, p.lower_bound) * RCP_LN2); };
            *reinterpret_cast<float4*>(&sh.d[t][4 * lane]) = make_float4(decay(x.x + b.x), decay(x.y + b.y), decay(x.z + b.z), decay(x.w + b.w));
            *reinterpret_cast<float4*>(&sh.k[t][4 * lane]) = make_float4(k4.x * fk, k4.y * fk, k4.z * fk, k4.w * fk);
            *reinterpret_cast<float4*>(&sh.q[t][4 * lane]) = make_float4(q4.x * fq, q4.y * fq, q4.z * fq, q4.w * fq);
            *reinterpret_cast<float4*>(&sh.v[t][4 * lane]) = v4;
            if (lane == 0) sh.beta[t] = p.beta_sigmoid ? p.beta_scale * sigmoidf_(rb) : rb;
            if (p.has_norm) z = widen4(rz, p.gate_dtype);
        }
        sync_compute();
        float S[4][8];                                     // channel 4 lane + i, value 8 warp + v
        const bool here = umma::mbar_wait(&sh.full[j & 1], (j >> 1) & 1);
        if (!here) *gave_up = 1;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const float4 a = p.h0 ? *reinterpret_cast<const float4*>(states + (j & 1) * STATE + (8 * warp + v) * DK + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            S[0][v] = a.x; S[1][v] = a.y; S[2][v] = a.z; S[3][v] = a.w;
        }
        __syncwarp();
        if (here && lane == 0) umma::arrive(&sh.empty[j & 1]);
        request(j + 1);
        for (int s = 0; s < n_tok; ++s) {
            const float4 d4 = *reinterpret_cast<const float4*>(sh.d[s] + 4 * lane), k4 = *reinterpret_cast<const float4*>(sh.k[s] + 4 * lane),
                         q4 = *reinterpret_cast<const float4*>(sh.q[s] + 4 * lane);
            const float d[4] = {d4.x, d4.y, d4.z, d4.w}, k[4] = {k4.x, k4.y, k4.z, k4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w};
            float a[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                a[v] = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) { S[i][v] *= d[i]; a[v] = fmaf(k[i], S[i][v], a[v]); }
            }
            warp_colsum(a, lane);                          // lanes 4 v .. 4 v + 3 have the sum of value v
            const int mine = 8 * warp + (lane >> 2);
            const float u = sh.beta[s] * (sh.v[s][mine] - a[0]);
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const float uv = __shfl_sync(0xffffffffu, u, 4 * v);
                a[v] = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) { S[i][v] = fmaf(k[i], uv, S[i][v]); a[v] = fmaf(q[i], S[i][v], a[v]); }
            }
            warp_colsum(a, lane);
            if ((lane & 3) == 0) sh.o[s][mine] = a[0];
        }
        if (p.ht) {
#pragma unroll
            for (int v = 0; v < 8; ++v)
                *reinterpret_cast<float4*>(p.ht + so + (size_t)(8 * warp + v) * DK + 4 * lane) = make_float4(S[0][v], S[1][v], S[2][v], S[3][v]);
        }
        sync_compute();
        end = *gave_up;
        if (t < n_tok) {                                   // output rows: lane = 4 values
            float4 o = *reinterpret_cast<const float4*>(&sh.o[t][4 * lane]);
            if (p.has_norm) {
                const float rs = 1.f / sqrtf(warp_sum_f((o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w)) * (1.f / 128.f) + p.eps);
                const float zz[4] = {z.x, z.y, z.z, z.w};
                float a[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float sg = sigmoidf_(zz[e]);
                    a[e] = p.act == MKDA_ACT_SILU ? zz[e] * sg : sg;
                }
                o = make_float4(o.x * rs * w4.x * a[0], o.y * rs * w4.y * a[1], o.z * rs * w4.z * a[2], o.w * rs * w4.w * a[3]);
            }
            st4(p.out, p.out_dtype, ((size_t)(first + t) * HV + h) * 128 + 4 * lane, o);
        }
    }
}

int step_status(unsigned int* out) { return cudaMemcpyFromSymbol(out, umma::g_timeout_flag, sizeof(unsigned int)) == cudaSuccess ? 0 : -1; }
int step_status_clear() {
    const unsigned int z = 0;
    return cudaMemcpyToSymbol(umma::g_timeout_flag, &z, sizeof(z)) == cudaSuccess ? 0 : -1;
}

}  // namespace mkda

using namespace mkda;

extern "C" int mkda_step_fwd(const MkdaStepFwd* p, void* stream) {
    if (!p || !p->q || !p->k || !p->v || !p->x || !p->beta || !p->out || !p->seq_chunk_off) return set_error(MKDA_ERR_ARG, "step_fwd: null argument");
    if (any_misaligned(p->q, p->k, p->v, p->out, p->gate, p->norm_w) || (!p->scalar_gate && any_misaligned(p->x, p->dt_bias)) ||
        (p->state_v_first && any_misaligned(p->h0, p->ht)))
        return set_error(MKDA_ERR_ARG, "step_fwd: tensors must be 16-byte aligned");
    if (p->L.HK <= 0 || p->L.HV % p->L.HK) return set_error(MKDA_ERR_ARG, "step_fwd: HV must be a multiple of HK");
    if (p->has_norm && !p->gate) return set_error(MKDA_ERR_ARG, "step_fwd: the gated norm needs a gate tensor");
    if (p->mode != MKDA_GATE_PRECOMPUTED && !(p->lower_bound < 0.f)) return set_error(MKDA_ERR_ARG, "step_fwd: lower_bound must be < 0");
    if (!p->short_only && p->longest > STEP_MAX) return set_error(MKDA_ERR_ARG, "step_fwd: a sequence is longer than MKDA_STEP_MAX_TOKENS");
    for (int dt : {p->qkv_dtype, p->x_dtype, p->beta_dtype, p->out_dtype})
        if (dt < MKDA_F32 || dt > MKDA_F16) return set_error(MKDA_ERR_ARG, "step_fwd: unsupported dtype");
    if (p->N == 0 || p->L.HV == 0) return MKDA_OK;
    const int items = p->N * p->L.HV;
    if (p->state_v_first) {
        if (int e = ensure_smem((const void*)step_fwd_vk_kernel, st::SMEM, "step_fwd")) return e;
        launch(step_fwd_vk_kernel, items < sm_count() ? items : sm_count(), st::THREADS, st::SMEM, (cudaStream_t)stream, *p);
    } else {
        launch(step_fwd_kernel, items, 256, 0, (cudaStream_t)stream, *p);
    }
    return check_launch("step_fwd");
}
