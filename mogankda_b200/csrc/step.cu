// Forward pass over very short sequences (generation steps, speculative tokens): the recurrence itself, token by token, instead of the
// chunk algebra.
//   S <- diag(2^g) S        S <- S + k (beta (v - k^T S))        o = scale q^T S, then the optional gated RMSNorm
// One CTA per (sequence, v-head) with the fp32 state in registers (thread = one v x 64 key channels): the state is read and written once and
// everything in between, gate and L2 norm included, stays on chip.
// What bounds it: 128 KB of state traffic per CTA.  The chunk path spends the same traffic several times over (operand tiles of 64 rows of
// which a few are real, and five launches): 63 us of kernels for one token of 8 sequences x 32 heads, against 9 us here (33.5 MB of states).
// Up to how many tokens: a token costs 1.6 us there, a chunk the same for any number of rows.  16 tokens, whole call with cold caches, here
// and by chunks: 43 / 52 us (8 sequences x 32 heads), 221 / 316 us (64 x 32), 29 / 30 us (1 x 32); one token 18 / 50, 80 / 306, 14 / 30.
#include "common.cuh"
#include "gate.cuh"
#include "host.h"

namespace mkda {

constexpr int STEP_MAX = MKDA_STEP_MAX_TOKENS;
struct StepShared {
    float k[STEP_MAX][DK], q[STEP_MAX][DK], d[STEP_MAX][DK], v[STEP_MAX][DV], o[STEP_MAX][DV], beta[STEP_MAX];
    float part[2][2][DV];
};

__device__ __forceinline__ float warp_sum_f(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

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
    } else if (p.state_v_first) {
        const float4* src = reinterpret_cast<const float4*>(p.h0 + so + (size_t)vi * DK + half * 64);
#pragma unroll
        for (int i = 0; i < 16; ++i) { const float4 a = src[i]; S[4 * i] = a.x; S[4 * i + 1] = a.y; S[4 * i + 2] = a.z; S[4 * i + 3] = a.w; }
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
        if (p.state_v_first) {
            float4* dst = reinterpret_cast<float4*>(p.ht + so + (size_t)vi * DK + half * 64);
#pragma unroll
            for (int i = 0; i < 16; ++i) dst[i] = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) p.ht[so + (size_t)(half * 64 + i) * DV + vi] = S[i];
        }
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
    launch(step_fwd_kernel, p->N * p->L.HV, 256, 0, (cudaStream_t)stream, *p);
    return check_launch("step_fwd");
}
