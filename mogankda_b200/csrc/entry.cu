// C-ABI entry points of the chunk kernels: argument checks, then the launcher of the tensor-core kernel.
#include "host.h"

using namespace mkda;

static int intra_fwd(const MkdaIntraFwd* given, bool forward_only, void* stream) {
    if (!given) return set_error(MKDA_ERR_ARG, "intra_fwd: null argument");
    MkdaIntraFwd call = *given;
    if (forward_only) call.A = nullptr;                    // whatever stands there
    const MkdaIntraFwd* p = &call;
    if (!p->q || !p->k || !p->v || !p->g_c || !p->beta || (!p->A && !forward_only) || !p->Aqk || !p->nw || !p->u || !p->kbar || !p->qs || !p->gl)
        return set_error(MKDA_ERR_ARG, "intra_fwd: null argument");
    if (any_misaligned(p->q, p->k, p->v, p->g_c, p->A, p->Aqk, p->nw, p->u, p->kbar, p->qs, p->gl))
        return set_error(MKDA_ERR_ARG, "intra_fwd: tensors must be 16-byte aligned");
    if (p->L.HK <= 0 || p->L.HV % p->L.HK) return set_error(MKDA_ERR_ARG, "intra_fwd: HV must be a multiple of HK");
    if (p->L.NC == 0) return MKDA_OK;
    return launch_intra_fwd_tc(p, nullptr, (cudaStream_t)stream);
}
extern "C" int mkda_intra_fwd(const MkdaIntraFwd* p, void* stream) { return intra_fwd(p, false, stream); }
extern "C" int mkda_intra_fwd_forward_only(const MkdaIntraFwd* p, void* stream) { return intra_fwd(p, true, stream); }

extern "C" int mkda_gate_intra_fwd(const MkdaGateFwd* g, const MkdaIntraFwd* p, void* stream) {
    if (!g || !p || !g->x || !g->beta_raw || !p->q || !p->k || !p->v || !p->Aqk || !p->nw || !p->u || !p->kbar || !p->qs || !p->gl)
        return set_error(MKDA_ERR_ARG, "gate_intra_fwd: null argument");
    if (any_misaligned(p->q, p->k, p->v, p->A, p->Aqk, p->nw, p->u, p->kbar, p->qs, p->gl) ||
        (!p->scalar_gate && any_misaligned(g->x, g->dt_bias, g->g_c)))
        return set_error(MKDA_ERR_ARG, "gate_intra_fwd: tensors must be 16-byte aligned");
    if (g->scalar_gate != p->scalar_gate) return set_error(MKDA_ERR_ARG, "gate_intra_fwd: one decay per token, or one per channel?");
    if (g->mode != MKDA_GATE_PRECOMPUTED && !(g->lower_bound < 0.f)) return set_error(MKDA_ERR_ARG, "gate_intra_fwd: lower_bound must be < 0");
    for (int dt : {g->x_dtype, g->beta_dtype})
        if (dt < MKDA_F32 || dt > MKDA_F16) return set_error(MKDA_ERR_ARG, "gate_intra_fwd: unsupported dtype");
    if (p->L.HK <= 0 || p->L.HV % p->L.HK) return set_error(MKDA_ERR_ARG, "gate_intra_fwd: HV must be a multiple of HK");
    if (p->L.NC == 0) return MKDA_OK;
    if ((long long)p->L.NC * p->L.HV > sm_count()) return set_error(MKDA_ERR_ARG, "gate_intra_fwd: more (chunk, v-head) pairs than SMs");
    MkdaGateFwd gate = *g;
    gate.L = p->L;
    return launch_intra_fwd_tc(p, &gate, (cudaStream_t)stream);
}

extern "C" int mkda_recur_fwd_ordered(const MkdaRecurFwd* p, const int* seg_order, void* stream) {
    if (!p || !p->nw || !p->u || !p->kbar || !p->gl) return set_error(MKDA_ERR_ARG, "recur_fwd: null argument");
    if (any_misaligned(p->nw, p->u, p->kbar, p->gl, p->h, p->Vd)) return set_error(MKDA_ERR_ARG, "recur_fwd: tensors must be 16-byte aligned");
    if (any_misaligned32(p->h, p->Vd) || (p->state_v_first && any_misaligned32(p->h0, p->ht)))
        return set_error(MKDA_ERR_ARG, "recur_fwd: saved tiles and [V,K] states must be 32-byte aligned");
    if (p->want_transition && !p->mt) return set_error(MKDA_ERR_ARG, "recur_fwd: want_transition needs mt");
    if (p->L.NS == 0) return MKDA_OK;
    return launch_recur_fwd_tc(p, seg_order, (cudaStream_t)stream);
}
extern "C" int mkda_recur_fwd(const MkdaRecurFwd* p, void* stream) { return mkda_recur_fwd_ordered(p, nullptr, stream); }

extern "C" int mkda_out_fwd(const MkdaOutFwd* p, void* stream) {
    if (!p || !p->qs || !p->Aqk || !p->Vd || !p->h || !p->out) return set_error(MKDA_ERR_ARG, "out_fwd: null argument");
    if (any_misaligned(p->qs, p->Aqk, p->Vd, p->h, p->out, p->o_raw, p->gate, p->norm_w)) return set_error(MKDA_ERR_ARG, "out_fwd: tensors must be 16-byte aligned");
    if (p->has_norm && !p->gate) return set_error(MKDA_ERR_ARG, "out_fwd: the gated norm needs a gate tensor");
    if (p->L.NC == 0) return MKDA_OK;
    return launch_out_fwd_tc(p, (cudaStream_t)stream);
}

extern "C" int mkda_chain_fwd_ordered(const MkdaChainFwd* p, const int* seg_order, void* stream) {
    if (!p || !p->r.nw || !p->r.u || !p->r.kbar || !p->r.gl || !p->o.qs || !p->o.Aqk || !p->o.out) return set_error(MKDA_ERR_ARG, "chain_fwd: null argument");
    if (any_misaligned(p->r.nw, p->r.u, p->r.kbar, p->r.gl, p->o.qs, p->o.Aqk, p->o.out, p->o.o_raw, p->o.gate, p->o.norm_w))
        return set_error(MKDA_ERR_ARG, "chain_fwd: tensors must be 16-byte aligned");
    if (any_misaligned32(p->r.h, p->r.Vd) || (p->r.state_v_first && any_misaligned32(p->r.h0, p->r.ht)))
        return set_error(MKDA_ERR_ARG, "chain_fwd: saved tiles and [V,K] states must be 32-byte aligned");
    if (p->r.want_transition || p->r.warm_start) return set_error(MKDA_ERR_ARG, "chain_fwd: no transition and no truncation in a main pass");
    if (p->o.has_norm && (!p->o.gate || p->o.out_dtype != MKDA_F32)) return set_error(MKDA_ERR_ARG, "chain_fwd: the gated norm needs a gate tensor and fp32 output");
    if (p->r.L.NS == 0) return MKDA_OK;
    return launch_chain_fwd_tc(p, seg_order, (cudaStream_t)stream);
}
extern "C" int mkda_chain_fwd(const MkdaChainFwd* p, void* stream) { return mkda_chain_fwd_ordered(p, nullptr, stream); }

static int check_bwd_dh(const MkdaBwdDh* p, bool source) {
    if (!p || !source || !p->kbar || !p->qs || !p->gl || !p->Aqk || !p->nw) return set_error(MKDA_ERR_ARG, "bwd_dh: null argument");
    if (any_misaligned(p->d_o, p->dO_in_t, p->kbar, p->qs, p->gl, p->Aqk, p->nw, p->dh, p->dVd_t, p->dO_t))
        return set_error(MKDA_ERR_ARG, "bwd_dh: tensors must be 16-byte aligned");
    if (any_misaligned32(p->dh, p->dVd_t) || (p->state_v_first && any_misaligned32(p->dht, p->dh0)))
        return set_error(MKDA_ERR_ARG, "bwd_dh: saved tiles and [V,K] states must be 32-byte aligned");
    return MKDA_OK;
}
extern "C" int mkda_bwd_dh_ordered(const MkdaBwdDh* p, const int* seg_order, void* stream) {
    if (int e = check_bwd_dh(p, p && (p->dO_in_t || (p->d_o && p->dO_t)))) return e;
    if (p->L.NS == 0) return MKDA_OK;
    if (p->dO_in_t) return launch_bwd_dh_tc(p, seg_order, false, (cudaStream_t)stream);
    if (int e = launch_rows_to_tiles(p->L, p->d_o, p->do_dtype, p->dO_t, (cudaStream_t)stream)) return e;
    MkdaBwdDh q = *p;
    q.dO_in_t = p->dO_t;
    return launch_bwd_dh_tc(&q, seg_order, false, (cudaStream_t)stream);
}
extern "C" int mkda_bwd_dh_rows(const MkdaBwdDh* p, const int* seg_order, void* stream) {
    if (int e = check_bwd_dh(p, p && p->d_o)) return e;
    if (p->do_dtype != MKDA_BF16) return set_error(MKDA_ERR_ARG, "bwd_dh_rows: unsupported dtype");
    if (p->L.NS == 0) return MKDA_OK;
    MkdaBwdDh q = *p;
    if (!q.dO_in_t && q.dO_t) {
        if (int e = launch_ragged_rows_to_tiles(q.L, q.d_o, q.dO_t, (cudaStream_t)stream)) return e;
        q.dO_in_t = q.dO_t;
    }
    return launch_bwd_dh_tc(&q, seg_order, true, (cudaStream_t)stream);
}
extern "C" int mkda_bwd_dh(const MkdaBwdDh* p, void* stream) { return mkda_bwd_dh_ordered(p, nullptr, stream); }

static int bwd_chunk(const MkdaBwdChunk* given, const void* d_o, bool finish, void* dq, void* dk, void* stream) {
    if (!given || (finish && (!dq || !dk))) return set_error(MKDA_ERR_ARG, "bwd_chunk: null argument");
    MkdaBwdChunk call = *given;
    if (finish) call.dq_v = call.dk_v = nullptr;           // whatever stands there
    const MkdaBwdChunk* p = &call;
    if (!p->q || !p->k || !p->v || !p->g_c || !p->beta || !p->A || !p->h || !p->dh || !p->Vd || (!p->dO_t && !d_o) || !p->dVd_t ||
        (!finish && (!p->dq_v || !p->dk_v)) || !p->dgp || !p->dbeta || !p->dv)
        return set_error(MKDA_ERR_ARG, "bwd_chunk: null argument");
    if (any_misaligned(p->q, p->k, p->v, p->g_c, p->A, p->h, p->dh, p->Vd, p->dO_t, p->dVd_t, p->dq_v, p->dk_v, p->dgp, p->dv, d_o, dq, dk))
        return set_error(MKDA_ERR_ARG, "bwd_chunk: tensors must be 16-byte aligned");
    if (p->beta_sigmoid && !p->beta_raw) return set_error(MKDA_ERR_ARG, "bwd_chunk: sigmoid beta needs the raw input");
    if (p->L.HK <= 0 || p->L.HV % p->L.HK) return set_error(MKDA_ERR_ARG, "bwd_chunk: HV must be a multiple of HK");
    if (finish && (p->L.HK != p->L.HV || p->q_rstd || p->k_rstd))
        return set_error(MKDA_ERR_ARG, "bwd_chunk_rows: finished dq and dk need one v-head per q/k head and rows that are not normalised");
    if (d_o && p->qkv_dtype != MKDA_BF16) return set_error(MKDA_ERR_ARG, "bwd_chunk_rows: rows of dO are taken in bf16 calls only");
    if (p->L.NC == 0) return MKDA_OK;
    return launch_bwd_chunk_tc(p, d_o, dq, dk, (cudaStream_t)stream);
}
extern "C" int mkda_bwd_chunk(const MkdaBwdChunk* p, void* stream) { return bwd_chunk(p, nullptr, false, nullptr, nullptr, stream); }
extern "C" int mkda_bwd_chunk_rows(const MkdaBwdChunk* p, const void* d_o, void* dq, void* dk, void* stream) {
    return bwd_chunk(p, d_o, dq || dk, dq, dk, stream);
}
