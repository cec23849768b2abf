// What the kernels that turn a row of logits into a token share: the row's parameters worked out, the penalties, the bounds
// that say which elements can still become candidates, the sort keys, and what a draw leaves behind.
#pragma once
#include "row_pipeline.h"

#include "device_expf.cuh"
#include "list_chain.cuh"
#include "ptx.cuh"

#include <cfloat>

namespace mk {

// top_p alone, first launch: the largest elements kept. The bound that keeps them is the edge of a histogram bin and lets
// about 1.4 times as many through; the one-warp finish takes 32. Rows that the flat rows' kernel does not take pay for a longer
// nucleus with a second stream of the row: they keep a few more, and the general finish has a look at what the one-warp finish
// could not settle; of the others that goes to the flat rows' kernel at once. (hist_k says which of the two a row is.)
constexpr uint32_t kNucleusGuess = 20, kNucleusGuessAlone = 24;

struct RowCfg {
    float temperature, inv_t, minp_eff, top_p;
    uint32_t top_k;
    uint32_t hist_k;    // the histogram bound keeps the hist_k largest elements
    float rep, presence, frequency;
    bool greedy, hist_mode, need_sum, use_topp, pen_active, optimistic;
    float delta_w;      // keep elements with l >= running max - delta_w
    bool force_none;    // inv_t is inf/NaN: no finite weight can exist
};

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)::"memory"); // (stays on its side of a barrier)
    return t;
}

// `flat`: whether the flat rows' kernel takes this row, should it be marked.
__device__ __forceinline__ RowCfg make_cfg(const mk_sampling_params& p, uint32_t n_vocab, int mode, uint32_t vp_k, int pass, bool flat)
{
    RowCfg c;
    c.temperature = p.temperature;
    c.greedy = p.temperature <= 0.0f;                       // sampler.hpp:26
    c.inv_t = __fdiv_rn(1.0f, p.temperature);               // sampler.cpp:29
    c.minp_eff = (1.0f < p.min_p) ? 1.0f : p.min_p;         // std::min(min_p, 1.0f), sampler.cpp:34
    c.top_p = p.top_p;
    c.top_k = p.top_k;
    c.rep = p.repetition_penalty;
    c.presence = p.presence_penalty;
    c.frequency = p.frequency_penalty;
    c.pen_active = !(c.rep == 1.0f && c.presence == 0.0f && c.frequency == 0.0f);
    c.use_topp = p.top_p < 1.0f;
    c.hist_mode = !c.greedy && p.top_k > 0 && p.top_k < n_vocab;
    // One more than top_k is kept, so that "more candidates than top_k" (which decides whether the reference
    // truncates, and with it the order of the list, sampler.cpp:39) can be told from the kept elements alone.
    c.hist_k = p.top_k + 1u;
    const bool minp_on = c.minp_eff > 0.0f;
    // The float total over "all candidates" is only needed when top_p is the only truncation.
    c.need_sum = !c.greedy && c.use_topp && !minp_on && !c.hist_mode;
    c.force_none = !c.greedy && (!(c.inv_t < __int_as_float(0x7f800000)) || !(c.inv_t == c.inv_t));
    // top_p alone: the first launch bets that the nucleus lies within the largest few elements and keeps
    // only those (the top_k histogram bound, with no top_k cut afterwards); a row whose nucleus does not close within
    // what was kept asks for a second launch, which keeps everything the mass bound allows.
    const uint32_t guess = flat ? kNucleusGuess : kNucleusGuessAlone;
    c.optimistic = c.need_sum && pass == 0 && mode != kModeVpLocal && guess < n_vocab;
    if (c.optimistic) {
        c.hist_mode = true;
        c.hist_k = guess;
    }
    if (mode == kModeVpLocal) {
        c.hist_mode = vp_k < n_vocab;
        c.top_k = vp_k;
        c.hist_k = vp_k;
        c.need_sum = true;
        c.use_topp = false;
        c.minp_eff = 0.0f;
    }
    // Distance below the row maximum, in units of (l - max) * inv_t, past which an element cannot be kept:
    //   q == 0 below about -103.98 (float underflow of expf);
    //   q < min_p below ln(min_p);
    //   with top_p alone, an element with q < (1 - top_p) / n_vocab is outside the nucleus, because all such
    //   elements together weigh less than (1 - top_p) * total (total >= 1: the maximum itself has q = 1).
    float d = 104.2f;
    if (mode != kModeVpLocal) {
        if (minp_on)
            d = fminf(d, -logf(c.minp_eff));
        if (c.need_sum) {
            float a = (1.0f - c.top_p) / (float)n_vocab;
            a = fminf(a, 1.0f);
            if (a > 0.0f)
                d = fminf(d, -logf(a));
        }
    }
    d = d * 1.001f + 1e-3f;
    c.delta_w = d * fmaxf(c.temperature, 0.0f);
    if (!(c.delta_w == c.delta_w))
        c.delta_w = __int_as_float(0x7f800000);
    return c;
}

// Threshold on the (edited) logit for the current running maximum; never -inf, so masked elements never pass.
__device__ __forceinline__ float keep_threshold(const RowCfg& c, float m_run)
{
    if (c.force_none || !(m_run < __int_as_float(0x7f800000)))
        return __int_as_float(0x7f800000); // no finite weight can exist (an infinite maximum makes l - max NaN or -inf)
    const float t = m_run - c.delta_w - fabsf(m_run) * 1e-6f;
    return fmaxf(t, -FLT_MAX);
}

// Penalties of one generated token with count n, exactly as sampler.cpp:24-27.
__device__ __forceinline__ float penalise(float l, uint32_t n, const RowCfg& c)
{
    if (c.rep != 1.0f)
        l = (l > 0.0f) ? __fdiv_rn(l, c.rep) : __fmul_rn(l, c.rep);
    const float step = __fadd_rn(c.presence, __fmul_rn(c.frequency, (float)n));
    return __fsub_rn(l, step);
}

__device__ __forceinline__ unsigned long long pack_by_weight(float q, uint32_t col)
{
    // ascending key order = (q descending, column ascending); q > 0 so its bit pattern is monotone
    return ((unsigned long long)(~__float_as_uint(q)) << 32) | col;
}
__device__ __forceinline__ unsigned long long pack_by_column(float q, uint32_t col)
{
    return ((unsigned long long)col << 32) | __float_as_uint(q);
}

// Where a row's results go (the output pointers of the launch), for the steps that live out of line.
struct RowOut {
    int32_t* token;
    float* prob;
    uint32_t* flags;
    uint32_t* n_cand;
    int32_t* accepted;
    float* total_out;
    int32_t* cand_ids;
    float* cand_q;
    uint32_t cand_cap;
    int32_t id_offset;
    unsigned long long* timing;
    int mode;
};

// What the draw leaves behind once its chains are known (sampler.cpp:64-73, 80-83, 100-106), for a list of n weights q in draw
// order (16-byte aligned; zeros, the gaps of a list laid out by column, never win; a rejected draft's weight is zeroed).
// col_of(i) names a weight's column; n_out is the number of candidates; in front of place `from`, a multiple of eight, there are
// only zeros. Whole CTA; the caller synchronises before.
template <int kThreads, class Col>
__device__ __forceinline__ void draw_long(ChainSmem<kThreads>& cs, float* q, uint32_t n, uint32_t n_out, uint32_t draft_idx,
                                          uint32_t row, uint32_t flags, float u_row, float u2_row, int32_t draft_row,
                                          const RowOut& o, Col&& col_of, uint32_t from = 0u)
{
    const uint32_t none = 0xffffffffu;
    const float total = chain<kThreads, false>(cs, q, n, 0.0f, from);
    const float q_draft = (draft_idx != none) ? q[draft_idx] : 0.0f;
    int32_t tok = -1, acc = 0;
    float prob = 0.0f, walk_total = total;
    if (o.mode == kModeDistOnly) {
        tok = -2; // nothing is drawn: the first candidate stands for the row below
    } else if (o.mode == kModeVerify) {
        acc = __fmul_rn(u_row, total) < q_draft;
        if (acc) {
            tok = draft_row;
            prob = __fdiv_rn(q_draft, total);
        } else {
            walk_total = __fsub_rn(total, q_draft);
        }
    }
    uint32_t hit = none, first = none, last = none;
    float r_hit = 0.0f, q_hit = 0.0f;
    if (tok == -1) {
        if (draft_idx != none && o.mode == kModeVerify) {
            __syncthreads(); // everyone has read the draft's weight
            if (threadIdx.x == 0)
                q[draft_idx] = 0.0f;
            __syncthreads();
        }
        chain<kThreads, true>(cs, q, n, __fmul_rn((o.mode == kModeVerify) ? u2_row : u_row, walk_total), from);
        hit = cs.hit;
        r_hit = cs.r_hit;
        q_hit = cs.q_hit;
    }
    // the first and the last candidate that could win: the edges of the CDF have no neighbour beyond them
    __syncthreads();
    if (threadIdx.x == 0) {
        cs.first = none;
        cs.last = 0u;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kThreads)
        if (q[i] > 0.0f) {
            atomicMin(&cs.first, i);
            break;
        }
    for (uint32_t i = threadIdx.x; i < n; i += kThreads)
        if (q[n - 1u - i] > 0.0f) {
            atomicMax(&cs.last, n - 1u - i);
            break;
        }
    __syncthreads();
    first = cs.first;
    last = cs.last;
    if (threadIdx.x != 0)
        return;
    if (tok == -2) {
        tok = (int32_t)col_of(first) + o.id_offset;
        prob = __fdiv_rn(q[first], total);
    } else if (tok == -1 && first == none) { // nothing but the rejected draft
        tok = draft_row;
        prob = 1.0f;
    } else if (tok == -1) {
        const float eps = 1e-6f * walk_total;
        if (hit != none) {
            if ((hit != first && r_hit < eps) || (hit < last && __fsub_rn(q_hit, r_hit) < eps))
                flags |= MK_FLAG_NEAR_CDF_BOUNDARY;
        } else { // rounding: the last candidate (sampler.cpp:72)
            hit = last;
            q_hit = q[last];
        }
        tok = (int32_t)col_of(hit) + o.id_offset;
        prob = __fdiv_rn(q_hit, walk_total);
    }
    if (o.token) o.token[row] = tok;
    if (o.prob) o.prob[row] = prob;
    if (o.flags) o.flags[row] = flags;
    if (o.n_cand) o.n_cand[row] = n_out;
    if (o.accepted) o.accepted[row] = acc;
    if (o.total_out) o.total_out[row] = total;
    if (o.timing) o.timing[(size_t)row * 64 + 3] = global_ns();
}

} // namespace mk
