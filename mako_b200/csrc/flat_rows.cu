// Flat rows of top_p alone: the rows whose nucleus the row pipeline's first launch could not settle with the few largest
// elements it keeps (src/gen/sampler.cpp:44-61 with neither min_p nor top_k). Hundreds to tens of thousands of tokens have
// to be ordered, summed and walked.
//
// One CTA of 1024 threads takes a marked row; the others return. What the first launch leaves is the row's maximum and its
// total weight (exact for what it kept, approximate for the rest), so the cut is known before the row is read again:
//   sample    an eighth of the columns counted by weight class (sixteenths of an octave) says below which weight the elements
//             sum up to a little less than the mass top_p leaves out; where the bound that cannot be too tight leaves no more
//             than a few thousand elements, that bound is the cut, and all of them get exact weights;
//   collect   one pass over the row keeps everything above that weight — the nucleus and a few per cent more — and sums
//             the approximate weights of the rest, one by one in double;
//   order     exact weights; the list is dealt into buckets of about six, of equal counts rather than equal widths, whose
//             members rank themselves, a lane each (a warp or the CTA sorts where equal weights crowd a bucket);
//   draw      double prefix sums for top_p, then the float total and the walk as scans (list_chain.cuh).
// A cut that proves too tight (a list that ends before the nucleus does) is replaced by the bound that cannot be, and the row
// is read once more. The generated and biased columns are edited apart: a bitmap takes them out of the row's stream, and their
// edited values join the list by themselves.
//
// Bound by the latency of one CTA's phases: the row itself (0.6 MB) takes about a quarter of the time of a row with a nucleus of
// some thousand tokens.
#include "row_common.cuh"

namespace mk {

namespace {

constexpr int kFlatThreads = 1024;
constexpr uint32_t kFlatWarps = kFlatThreads / 32;
constexpr uint32_t kClasses = 512;          // weight classes: sixteenths of an octave below the maximum's weight
constexpr uint32_t kSpecialCap = kFlatMaxEdits; // generated and biased columns of a row (history entries + bias entries)
constexpr uint32_t kFlatVocab = 163840;
constexpr uint32_t kFlatBmWords = kFlatVocab / 32 + 2;
constexpr uint32_t kMaxBuckets = 8192;
constexpr uint32_t kWarpSort = 4096;        // a bucket of more than 32 and up to this size is sorted by one warp
constexpr uint32_t kBigBuckets = 1024;
constexpr uint32_t kKeepWhole = 6144;       // elements above the loose bound that are not cut further (see the cut)

// Shared memory: the tables of the edits while the row is read, the list and its buckets afterwards.
constexpr uint32_t kOffBitmap = 0;
constexpr uint32_t kOffRanks = kOffBitmap + ((kFlatBmWords * 4u + 15u) & ~15u);
constexpr uint32_t kOffCount = kOffRanks + ((kFlatBmWords * 2u + 15u) & ~15u);
constexpr uint32_t kOffCol = kOffCount + kSpecialCap * 4u;
constexpr uint32_t kOffVal = kOffCol + kSpecialCap * 4u;
constexpr uint32_t kOffKeysEnd = 20480u * 8u;                  // the list, up to 20480 keys; a longer one stays in the scratch
constexpr uint32_t kListCap = kOffKeysEnd / 8u;
constexpr uint32_t kOffBuckets = kOffKeysEnd;                  // kMaxBuckets ends of buckets; then the weights in order
constexpr uint32_t kOffClass = kOffBuckets + kMaxBuckets * 4u; // kClasses (first bucket, buckets); sampling: the counts
constexpr uint32_t kOffBig = kOffClass + kClasses * 8u;        // buckets too large for one thread
constexpr uint32_t kFlatDyn = kOffBig + kBigBuckets * 4u;
static_assert(kOffVal + kSpecialCap * 4u <= kOffBuckets, "the edits' tables lie below the classes");

struct FlatSmem {
    ChainSmem<kFlatThreads> chain;
    unsigned long long exp2_table[32];
    double sum[2][kFlatWarps];
    uint32_t wsum[kFlatWarps];
    uint32_t rows[16], n_rows;
    uint32_t n_list, n_big, n_take, n_above;
    float cut;
    double run, prev;
};

__device__ __forceinline__ uint32_t block_exclusive(FlatSmem& s, uint32_t mine, uint32_t& total)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if ((int)lane >= o)
            inc += y;
    }
    if (lane == 31u)
        s.wsum[warp] = inc;
    __syncthreads();
    uint32_t w = s.wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if ((int)lane >= o)
            w += y;
    }
    total = __shfl_sync(0xffffffffu, w, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, w, (int)((warp + 31u) & 31u));
    __syncthreads(); // wsum may be written again
    return inc - mine + (warp ? before : 0u);
}

__device__ __forceinline__ double block_sum(FlatSmem& s, double v, int slot)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0)
        s.sum[slot][warp] = v;
    __syncthreads();
    double t = s.sum[slot][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, o);
    __syncthreads();
    return t;
}

// A float that is zero or normal, not negative, as a double: three integer instructions, where a conversion takes as long as the
// exponential before it. (Zero comes out as 2^-127, which is nothing beside a total of at least one.)
__device__ __forceinline__ double widen(float x)
{
    const uint32_t b = __float_as_uint(x);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// Four mask bits from column c on (c may be negative: columns in front of the row read as not allowed by the caller's test).
__device__ __forceinline__ uint32_t mask_nibble(const uint32_t* __restrict__ mrow, int32_t c, uint32_t V)
{
    uint32_t bits = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int32_t cj = c + j;
        if (cj >= 0 && (uint32_t)cj < V)
            bits |= ((__ldg(mrow + ((uint32_t)cj >> 5)) >> ((uint32_t)cj & 31u)) & 1u) << j;
    }
    return bits;
}

// Ascending sort of n keys by `n_thr` threads (this one is `thr`): bitonic merges whose first step mirrors, so that places
// past the end, which would hold the largest keys, are never touched.
template <class Sync>
__device__ __forceinline__ void sort_any(unsigned long long* keys, uint32_t n, uint32_t thr, uint32_t n_thr, Sync&& sync)
{
    uint32_t p2 = 2;
    while (p2 < n)
        p2 <<= 1;
    for (uint32_t k = 2; k <= p2; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t c = thr; c < (p2 >> 1); c += n_thr) {
                uint32_t i = ((c & ~(j - 1u)) << 1) | (c & (j - 1u)), l = i | j;
                if (j == (k >> 1))
                    l = i ^ (k - 1u); // the mirrored step
                if (l < n) {
                    const unsigned long long a = keys[i], b = keys[l];
                    if (a > b) {
                        keys[i] = b;
                        keys[l] = a;
                    }
                }
            }
            sync();
        }
    }
}

} // namespace

__global__ void __launch_bounds__(kFlatThreads, 1) flat_row_kernel(const RowKernelArgs a, uint32_t batch)
{
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ FlatSmem s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, full = 0xffffffffu;
    uint32_t* const bitmap = reinterpret_cast<uint32_t*>(dyn + kOffBitmap);
    uint16_t* const ranks = reinterpret_cast<uint16_t*>(dyn + kOffRanks);
    uint32_t* const count = reinterpret_cast<uint32_t*>(dyn + kOffCount);
    uint32_t* const scol = reinterpret_cast<uint32_t*>(dyn + kOffCol);
    float* const sval = reinterpret_cast<float*>(dyn + kOffVal);
    uint32_t* const cls = reinterpret_cast<uint32_t*>(dyn + kOffClass);
    uint2* const cls2 = reinterpret_cast<uint2*>(dyn + kOffClass);
    uint32_t* const ends = reinterpret_cast<uint32_t*>(dyn + kOffBuckets);
    uint32_t* const big = reinterpret_cast<uint32_t*>(dyn + kOffBig);
    const uint32_t V = a.n_vocab;

    if (tid < 32u)
        s.exp2_table[tid] = kExp2Tab[tid];
    uint32_t seen = 0; // marked rows of earlier chunks
    for (uint32_t chunk = 0; chunk < batch; chunk += (uint32_t)kFlatThreads) {
        // Which marked rows of this chunk are this CTA's. Every CTA counts the marks itself, whenever it comes to run, so they
        // stand until the next call's first launch.
        const uint32_t r_mine = chunk + tid;
        bool marked = false;
        if (r_mine < batch)
            marked = a.scratch[(size_t)r_mine * row_scratch_words(a.scratch_cap) + 4ull * a.scratch_cap] != 0u;
        uint32_t n_marked;
        const uint32_t at = seen + block_exclusive(s, marked ? 1u : 0u, n_marked);
        if (n_marked == 0u)
            continue;
        if (marked && at % gridDim.x == blockIdx.x)
            s.rows[at / gridDim.x - seen / gridDim.x] = r_mine; // see launch_flat_rows for the bound on a chunk's share
        // rows seen + k with (seen + k) % grid == this CTA: the first such k, then every grid-th
        const uint32_t first = (blockIdx.x + gridDim.x - seen % gridDim.x) % gridDim.x;
        const uint32_t slot0 = (seen + first) / gridDim.x - seen / gridDim.x;
        const uint32_t n_rows = first < n_marked ? (n_marked - first + gridDim.x - 1u) / gridDim.x : 0u;
        seen += n_marked;
        __syncthreads();
        for (uint32_t ri = 0; ri < n_rows; ++ri) {
            const uint32_t row = s.rows[slot0 + ri];
            // ---- the row -------------------------------------------------------------------------------------------
            const mk_sampling_params prm = a.params_dev ? a.params_dev[row] : a.params;
            const RowCfg cfg = make_cfg(prm, V, a.mode, a.vp_k, 1, true);
            uint32_t* const row_scratch = a.scratch + (size_t)row * row_scratch_words(a.scratch_cap);
            uint2* const list = reinterpret_cast<uint2*>(row_scratch);
            uint32_t* const state = row_scratch + 4ull * a.scratch_cap;
            const float m = __uint_as_float(state[1]);
            const double total0 = *reinterpret_cast<const double*>(state + 2);
            const float c2 = cfg.inv_t * 1.4426950408889634f;
            const float ninf = -__int_as_float(0x7f800000);
            const float* __restrict__ lrow = a.logits + (size_t)row * a.ld;
            const uint32_t shift = (uint32_t)((reinterpret_cast<uintptr_t>(lrow) >> 2) & 3u); // floats past a 16-byte boundary
            const float4* __restrict__ l4 = reinterpret_cast<const float4*>(lrow - shift);
            const uint32_t n4 = (V + shift + 3u) >> 2; // groups of four places; place p is column p - shift
            const uint32_t* __restrict__ mrow = a.mask ? a.mask + (size_t)row * a.mask_ld : nullptr;
            const mk_bias* __restrict__ brow = a.bias ? a.bias + (size_t)row * a.n_bias : nullptr;
            const uint32_t nb = a.bias ? a.n_bias : 0u;
            const uint32_t hlen_cap = (uint32_t)min((uint64_t)65535u, a.history_ld);
            const uint32_t hlen_dev = (a.history && a.history_len) ? (uint32_t)max(a.history_len[row], 0) : 0u;
            uint32_t flags = hlen_dev > hlen_cap ? MK_FLAG_HISTORY_FULL : 0u;
            const uint32_t hlen_all = a.history ? (a.history_len ? min(hlen_dev, hlen_cap) : a.n_history) : 0u;
            const uint32_t hlen = cfg.pen_active ? hlen_all : 0u;
            const int32_t* __restrict__ hrow = a.history ? a.history + (size_t)row * a.history_ld : nullptr;
            const float u_row = a.u ? __ldg(a.u + row) : 0.0f, u2_row = a.u2 ? __ldg(a.u2 + row) : 0.0f;
            const int32_t draft_row = a.draft ? __ldg(a.draft + row) : -1;
            if (!flat_row_takes(a, hlen, nb))
                continue; // the row pipeline's own second launch takes it
            const bool special = hlen > 0u || nb > 0u;
            // Four places of the row: fetched (nothing is, for a group that reaches past the row's ends), and edited; those that
            // are not the row's own, not allowed, or edited apart read as -inf.
            auto fetch4 = [&](uint32_t g) -> float4 {
                const uint32_t p = 4u * g;
                return (p >= shift && p + 4u <= V + shift) ? __ldg(l4 + g) : make_float4(ninf, ninf, ninf, ninf);
            };
            auto edit4 = [&](uint32_t g, const float4& v, float (&w)[4]) {
                const uint32_t p = 4u * g;
                w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
                if (g >= n4)
                    return;
                uint32_t off = special ? (bitmap[p >> 5] >> (p & 31u)) & 15u : 0u;
                if (mrow)
                    off |= ~(shift == 0u ? __ldg(mrow + (p >> 5)) >> (p & 31u) : mask_nibble(mrow, (int32_t)p - (int32_t)shift, V));
                if (p < shift || p + 4u > V + shift) {
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j)
                        if (p + j >= shift && p + j < V + shift)
                            w[j] = __ldg(lrow + (p + j - shift));
                }
                if (off & 15u) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if ((off >> j) & 1u)
                            w[j] = ninf;
                }
            };
            if (a.timing && tid == 0)
                a.timing[(size_t)row * 64 + 14] = global_ns();
            // ---- the edited columns --------------------------------------------------------------------------------
            uint32_t n_special = 0;
            if (special) {
                const uint32_t words = (V + shift + 31u) >> 5;
                for (uint32_t i = tid; i <= words; i += kFlatThreads)
                    bitmap[i] = 0u;
                for (uint32_t i = tid; i < kSpecialCap; i += kFlatThreads)
                    count[i] = 0u;
                constexpr uint32_t kMine = kSpecialCap / kFlatThreads;
                uint32_t place[kMine]; // of this thread's entries, or none
#pragma unroll
                for (uint32_t i = 0; i < kMine; ++i) {
                    const uint32_t j = tid + i * kFlatThreads;
                    place[i] = 0xffffffffu;
                    if (j < hlen + nb) {
                        const bool h = j < hlen;
                        const int32_t id = h ? __ldg(hrow + j) : brow[j - hlen].id;
                        const uint32_t c = (uint32_t)id - (uint32_t)a.id_offset; // an id below the first column wraps past V
                        if ((h || id >= 0) && c < V)
                            place[i] = c + shift;
                    }
                }
                __syncthreads();
#pragma unroll
                for (uint32_t i = 0; i < kMine; ++i)
                    if (place[i] != 0xffffffffu)
                        atomicOr(&bitmap[place[i] >> 5], 1u << (place[i] & 31u));
                __syncthreads();
                constexpr uint32_t kPer = (kFlatBmWords + kFlatThreads - 1u) / kFlatThreads;
                uint32_t pc[kPer], mine = 0;
#pragma unroll
                for (uint32_t i = 0; i < kPer; ++i) {
                    const uint32_t w = tid * kPer + i;
                    pc[i] = w < words ? (uint32_t)__popc(bitmap[w]) : 0u;
                    mine += pc[i];
                }
                uint32_t before = block_exclusive(s, mine, n_special);
#pragma unroll
                for (uint32_t i = 0; i < kPer; ++i) {
                    const uint32_t w = tid * kPer + i;
                    if (w < words)
                        ranks[w] = (uint16_t)before;
                    before += pc[i];
                }
                __syncthreads();
#pragma unroll
                for (uint32_t i = 0; i < kMine; ++i) {
                    const uint32_t j = tid + i * kFlatThreads, p = place[i];
                    if (p == 0xffffffffu)
                        continue;
                    const uint32_t r = ranks[p >> 5] + __popc(bitmap[p >> 5] & ((1u << (p & 31u)) - 1u));
                    scol[r] = p - shift;
                    if (j < hlen) {
                        atomicAdd(&count[r], 1u);
                    } else {
                        sval[r] = brow[j - hlen].value;
                        atomicOr(&count[r], 0x80000000u);
                    }
                }
                __syncthreads();
                for (uint32_t r = tid; r < n_special; r += kFlatThreads) {
                    const uint32_t c = scol[r], n = count[r];
                    float l = __ldg(lrow + c);
                    if (n & 0x80000000u)
                        l = __fadd_rn(l, sval[r]);
                    if (n & 0x7fffffffu)
                        l = penalise(l, n & 0x7fffffffu, cfg);
                    if (mrow && !((__ldg(mrow + (c >> 5)) >> (c & 31u)) & 1u))
                        l = ninf;
                    sval[r] = l;
                }
            }
            if (a.timing && tid == 0)
                a.timing[(size_t)row * 64 + 15] = global_ns();
            // ---- the cut ---------------------------------------------------------------------------------------------
            // Elements counted by weight class; a class's heaviest weight stands for all of its elements, so the mass below a
            // class is never taken for less than the sample says. An eighth of a long row is counted, in runs of 128 columns.
            for (uint32_t i = tid; i < kClasses; i += kFlatThreads)
                cls[i] = 0u;
            if (tid == 0)
                s.n_above = 0u;
            __syncthreads();
            const uint32_t every = n4 >= 24576u ? 8u : n4 >= 8192u ? 4u : 1u;
            const float loose = fmaxf(keep_threshold(cfg, m), -FLT_MAX);
            uint32_t above = 0; // the sample's elements above the loose bound
            auto enter = [&](float w, uint32_t n) {
                above += w >= loose ? n : 0u;
                const float x = (m - w) * (c2 * 16.0f);
                if (x < (float)kClasses) // false for NaN and for what is not there
                    atomicAdd(&cls[min((uint32_t)fmaxf(x, 0.0f), kClasses - 1u)], n);
            };
            for (uint32_t b0 = warp * 4u; b0 * 32u * every < n4; b0 += kFlatWarps * 4u) { // four loads in flight
                float w[4][4];
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k) {
                    const uint32_t b = b0 + k, g = b * 32u * every + (b % every) * 32u + lane;
                    edit4(g, fetch4(g), w[k]);
                }
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        enter(w[k][j], every);
            }
            for (uint32_t r = tid; r < n_special; r += kFlatThreads)
                enter(sval[r], 1u);
            above = __reduce_add_sync(full, above);
            if (lane == 0 && above)
                atomicAdd(&s.n_above, above);
            __syncthreads();
            if (warp == 0) { // lane l holds classes 16 l .. 16 l + 15; mass from the light end
                float sum = 0.0f, sq = 0.0f;
                for (uint32_t j = 16u; j-- > 0u;) {
                    const uint32_t b = lane * 16u + j;
                    const float w = ex2_approx(-(float)b * 0.0625f), mass = (float)cls[b] * w;
                    sum += mass;
                    sq += mass * w;
                }
                float lighter = sum, sq_lighter = sq;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float y = __shfl_down_sync(full, lighter, o), z = __shfl_down_sync(full, sq_lighter, o);
                    if ((int)lane + o < 32) {
                        lighter += y;
                        sq_lighter += z;
                    }
                }
                lighter -= sum; // the lanes behind this one
                sq_lighter -= sq;
                // The estimate's own scatter is its standard deviation, sqrt((every - 1) * sum of squares): four of them and
                // 3 % of the budget are kept in hand.
                const float budget = (float)((1.0 - (double)cfg.top_p) * total0) * 0.97f;
                uint32_t cut = kClasses; // the heaviest class that is left out, with all lighter ones
                for (uint32_t j = 16u; j-- > 0u;) {
                    const uint32_t b = lane * 16u + j;
                    const float w = ex2_approx(-(float)b * 0.0625f), mass = (float)cls[b] * w;
                    lighter += mass;
                    sq_lighter += mass * w;
                    if (lighter + 4.0f * sqrtf((float)(every - 1u) * fmaxf(sq_lighter, 0.0f)) <= budget)
                        cut = b;
                }
                cut = __reduce_min_sync(full, cut);
                if (lane == 0) {
                    // Place of the class's heavy edge as a logit, a rounding below. Lists of up to 4096 elements above the loose
                    // bound are kept whole, so that all of them count with their exact weights; the sample's own count of an eighth
                    // is off by 170 or so there, a clustered one by more.
                    const float t = m - ((float)cut * 0.0625f) / c2;
                    s.cut = cut < kClasses && s.n_above > kKeepWhole ? fmaxf(loose, t - fabsf(m) * 1e-6f - fabsf(t) * 1e-6f) : loose;
                }
            }
            __syncthreads();
            float thr = s.cut;
            if (a.timing && tid == 0)
                a.timing[(size_t)row * 64 + 16] = global_ns();
            // ---- collect, order, cut at top_p; once more with the loose bound if the list ends too early ---------------
            unsigned long long* keys = nullptr;
            uint32_t n = 0, n_take = 0;
            for (int attempt = 0; attempt < 2; ++attempt) {
                if (tid == 0) {
                    s.n_list = 0u;
                    s.n_big = 0u;
                }
                __syncthreads();
                double tail = 0.0;
                for (uint32_t g0 = warp * 128u; g0 < n4; g0 += kFlatThreads * 4u) {
                    float4 v[4];
                    float w[4][4];
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        v[k] = fetch4(g0 + k * 32u + lane);
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        edit4(g0 + k * 32u + lane, v[k], w[k]);
                    uint32_t keep = 0u; // one bit an element; nothing below branches on an element's own value
                    double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j) {
                            keep |= w[k][j] >= thr ? 1u << (4u * k + j) : 0u;
                            const float e = ex2_approx((w[k][j] - m) * c2); // (not w * c2 - m * c2: that rounds m * c2)
                            part[j] += widen(w[k][j] < thr ? e : 0.0f); // a NaN is neither
                        }
                    tail += (part[0] + part[1]) + (part[2] + part[3]);
                    const uint32_t mine = (uint32_t)__popc(keep);
                    if (__any_sync(full, mine != 0u)) {
                        uint32_t inc = mine;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t y = __shfl_up_sync(full, inc, o);
                            if ((int)lane >= o)
                                inc += y;
                        }
                        uint32_t slot = 0;
                        if (lane == 31u)
                            slot = atomicAdd(&s.n_list, inc);
                        uint2* at_list = list + (__shfl_sync(full, slot, 31) + inc - mine);
                        const uint32_t col = 4u * (g0 + lane) - shift;
#pragma unroll
                        for (uint32_t k = 0; k < 4u; ++k)
#pragma unroll
                            for (uint32_t j = 0; j < 4u; ++j)
                                if ((keep >> (4u * k + j)) & 1u)
                                    *at_list++ = make_uint2(__float_as_uint(w[k][j]), col + 128u * k + j);
                    }
                }
                for (uint32_t r = tid; r < n_special; r += kFlatThreads) {
                    const float w = sval[r];
                    if (w >= thr)
                        list[atomicAdd(&s.n_list, 1u)] = make_uint2(__float_as_uint(w), scol[r]);
                    else if (w < thr)
                        tail += (double)ex2_approx((w - m) * c2);
                }
                const double rest = block_sum(s, tail, 0);
                n = s.n_list;
                if (a.timing && tid == 0)
                    a.timing[(size_t)row * 64 + 17] = global_ns();
                // exact weights, in place of the logits; their sum; how many there are in each class of the float's own octaves
                for (uint32_t i = tid; i < kClasses; i += kFlatThreads)
                    cls2[i] = make_uint2(0u, 0u);
                __syncthreads();
                double exact = 0.0;
                for (uint32_t i0 = tid; i0 < n; i0 += 4u * kFlatThreads) {
                    uint32_t x[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        x[k] = i0 + k * kFlatThreads < n ? list[i0 + k * kFlatThreads].x : 0u;
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k) {
                        if (i0 + k * kFlatThreads >= n)
                            break;
                        const float q = expf_host_exact(__fmul_rn(__fsub_rn(__uint_as_float(x[k]), m), cfg.inv_t), s.exp2_table);
                        const bool in = q >= cfg.minp_eff && q > 0.0f;
                        exact += (double)q;
                        const uint32_t d = in ? 0x3f800000u - __float_as_uint(q) : 0xffffffffu; // 0 for the maximum
                        list[i0 + k * kFlatThreads].x = d;
                        if (in)
                            atomicAdd(&cls2[min(d >> 19, kClasses - 1u)].y, 1u);
                    }
                }
                const double sum = block_sum(s, exact, 1);
                const double total = sum + rest;
                // (an approximate weight: ex2.approx takes 2^-22, its argument's rounding 4e-8 an octave below the maximum: 2e-6 at most
                // where a weight still counts; the sum is double)
                const double band = 1e-5 * rest + 0x1p-36 * total, want = (double)cfg.top_p * total;
                if (a.timing && tid == 0)
                    a.timing[(size_t)row * 64 + 18] = global_ns();
                // buckets: each class gets as many as its count asks for
                uint32_t in_class = tid < kClasses ? cls2[tid].y : 0u, n_in, n_buckets;
                block_exclusive(s, in_class, n_in);
                const uint32_t per = max(6u, (n_in + 5999u) / 6000u);
                const uint32_t want_b = (in_class + per - 1u) / per;
                const uint32_t b0 = block_exclusive(s, want_b, n_buckets); // at most n / per + kClasses
                if (tid < kClasses)
                    cls2[tid] = make_uint2(b0, want_b);
                for (uint32_t i = tid; i < n_buckets; i += kFlatThreads)
                    ends[i] = 0u;
                __syncthreads();
                auto bucket = [&](uint32_t d) -> uint32_t {
                    const uint32_t c = min(d >> 19, kClasses - 1u);
                    const uint2 b = cls2[c];
                    if (c == kClasses - 1u) // everything lighter still: no finer order, one bucket
                        return b.x;
                    return b.x + (uint32_t)(((unsigned long long)(d & 0x7ffffu) * b.y) >> 19);
                };
                for (uint32_t i0 = tid; i0 < n; i0 += 4u * kFlatThreads) {
                    uint32_t d[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        d[k] = i0 + k * kFlatThreads < n ? list[i0 + k * kFlatThreads].x : 0xffffffffu;
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        if (d[k] != 0xffffffffu)
                            atomicAdd(&ends[bucket(d[k])], 1u);
                }
                __syncthreads();
                {
                    constexpr uint32_t kPer = kMaxBuckets / kFlatThreads;
                    uint32_t c[kPer], mine = 0, all;
#pragma unroll
                    for (uint32_t i = 0; i < kPer; ++i) {
                        const uint32_t b = tid * kPer + i;
                        c[i] = b < n_buckets ? ends[b] : 0u;
                        mine += c[i];
                    }
                    uint32_t before = block_exclusive(s, mine, all);
#pragma unroll
                    for (uint32_t i = 0; i < kPer; ++i) {
                        const uint32_t b = tid * kPer + i;
                        if (b < n_buckets)
                            ends[b] = before; // its start; the dealing below moves it to its end
                        before += c[i];
                    }
                }
                __syncthreads();
                // The list takes the place of the edits' tables, unless it is too long. Should the row have to be read once
                // more, the edited values are found behind the raw list in the scratch.
                const bool tables_go = n_in <= kListCap && (!special || n + n_special <= a.scratch_cap);
                keys = tables_go ? reinterpret_cast<unsigned long long*>(dyn)
                                 : reinterpret_cast<unsigned long long*>(row_scratch) + a.scratch_cap;
                uint2* const keep = list + n;
                if (tables_go && special) {
                    for (uint32_t r = tid; r < n_special; r += kFlatThreads)
                        keep[r] = make_uint2(__float_as_uint(sval[r]), scol[r]);
                    __syncthreads();
                }
                for (uint32_t i0 = tid; i0 < n; i0 += 4u * kFlatThreads) {
                    uint2 c[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        c[k] = i0 + k * kFlatThreads < n ? list[i0 + k * kFlatThreads] : make_uint2(0xffffffffu, 0u);
#pragma unroll
                    for (uint32_t k = 0; k < 4u; ++k)
                        if (c[k].x != 0xffffffffu)
                            keys[atomicAdd(&ends[bucket(c[k].x)], 1u)] =
                                ((unsigned long long)(c[k].x + ~0x3f800000u) << 32) | c[k].y; // pack_by_weight's key
                }
                __syncthreads();
                if (a.timing && tid == 0)
                    a.timing[(size_t)row * 64 + 19] = global_ns();
                for (uint32_t b = tid; b < n_buckets; b += kFlatThreads)
                    if (ends[b] - (b ? ends[b - 1u] : 0u) > 32u) {
                        const uint32_t at_big = atomicAdd(&s.n_big, 1u);
                        if (at_big < kBigBuckets)
                            big[at_big] = b;
                    }
                // Every warp takes the buckets that start in its share of the list, as many as 32 lanes hold at a time: a
                // lane counts the smaller keys of its bucket and puts its own there.
                {
                    const uint32_t share = (n_in + kFlatWarps - 1u) / kFlatWarps, p_end = min((warp + 1u) * share, n_in);
                    uint32_t p = min(warp * share, n_in);
                    bool whole = p == 0u; // whether p is the start of a bucket
                    while (p < p_end) {
                        const uint32_t i = p + lane;
                        unsigned long long key = 0ull;
                        uint32_t i0 = 0u, i1 = 0u;
                        if (i < n_in) {
                            key = keys[i];
                            const uint32_t b = bucket((uint32_t)(key >> 32) - ~0x3f800000u);
                            i0 = b ? ends[b - 1u] : 0u;
                            i1 = ends[b];
                        }
                        const uint32_t b0 = __shfl_sync(full, i0, 0), b1 = __shfl_sync(full, i1, 0);
                        if ((!whole && b0 != p) || b1 - b0 > 32u) { // another warp's, or a large one
                            p = b1;
                            whole = true;
                            continue;
                        }
                        const bool mine = i < n_in && i1 <= p + 32u && i0 < p_end;
                        uint32_t below = 0u;
                        if (mine)
                            for (uint32_t j = i0; j < i1; ++j)
                                below += keys[j] < key ? 1u : 0u;
                        __syncwarp();
                        if (mine)
                            keys[i0 + below] = key;
                        __syncwarp();
                        p = __reduce_max_sync(full, mine ? i1 : 0u);
                        whole = true;
                    }
                }
                __syncthreads();
                const uint32_t n_big = s.n_big;
                if (n_big > kBigBuckets) { // more than the list of them holds: one sort of everything
                    sort_any(keys, n_in, tid, (uint32_t)kFlatThreads, [] { __syncthreads(); });
                } else {
                    for (uint32_t i = 0; i < n_big; ++i) {
                        const uint32_t b = big[i], i0 = b ? ends[b - 1u] : 0u, len = ends[b] - i0;
                        if (len > kWarpSort)
                            sort_any(keys + i0, len, tid, (uint32_t)kFlatThreads, [] { __syncthreads(); });
                    }
                    for (uint32_t i = warp; i < n_big; i += kFlatWarps) {
                        const uint32_t b = big[i], i0 = b ? ends[b - 1u] : 0u, len = ends[b] - i0;
                        if (len <= kWarpSort)
                            sort_any(keys + i0, len, lane, 32u, [] { __syncwarp(); });
                    }
                    __syncthreads();
                }
                if (a.timing && tid == 0)
                    a.timing[(size_t)row * 64 + 20] = global_ns();
                // ---- top_p (sampler.cpp:44-61): the shortest prefix whose double sum is not below `want` --------------------
                auto q_key = [&](uint32_t i) -> float { return __uint_as_float(~(uint32_t)(keys[i] >> 32)); };
                const uint32_t run_len = ((n_in + kFlatThreads - 1u) / kFlatThreads) | 1u;
                const uint32_t r0 = min(tid * run_len, n_in), r1 = min(r0 + run_len, n_in);
                double mine = 0.0;
                for (uint32_t i = r0; i < r1; ++i)
                    mine += (double)q_key(i);
                double inc = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double y = __shfl_up_sync(full, inc, o);
                    if ((int)lane >= o)
                        inc += y;
                }
                if (lane == 31u)
                    s.sum[0][warp] = inc;
                if (tid == 0)
                    s.n_take = n_in + 1u;
                __syncthreads();
                double before = inc - mine;
                for (uint32_t w = 0; w < warp; ++w)
                    before += s.sum[0][w];
                uint32_t cand = n_in + 1u;
                double run = before, prev = before;
                if (r0 < r1 && before + mine >= want * (1.0 - 1e-12))
                    for (uint32_t i = r0; i < r1; ++i) {
                        prev = run;
                        run += (double)q_key(i);
                        if (!(run < want)) {
                            cand = i + 1u;
                            break;
                        }
                    }
                if (cand <= n_in)
                    atomicMin(&s.n_take, cand);
                __syncthreads();
                n_take = s.n_take;
                if (n_take <= n_in && cand == n_take) {
                    s.run = run;
                    s.prev = prev;
                }
                __syncthreads();
                if (n_take <= n_in) {
                    if (fabs(s.run - want) <= band || (n_take >= 2u && fabs(s.prev - want) <= band))
                        flags |= MK_FLAG_GUARD_BAND;
                    n = n_in;
                    break;
                }
                // the list ended before the nucleus did
                if (attempt == 1 || !(thr > loose)) {
                    flags |= MK_FLAG_GUARD_BAND;
                    n = n_in;
                    n_take = max(n_in, 1u);
                    break;
                }
                if (special && tables_go) {
                    for (uint32_t r = tid; r < n_special; r += kFlatThreads) {
                        sval[r] = __uint_as_float(keep[r].x);
                        scol[r] = keep[r].y;
                    }
                    const uint32_t words = (V + shift + 31u) >> 5;
                    for (uint32_t i = tid; i <= words; i += kFlatThreads)
                        bitmap[i] = 0u;
                    __syncthreads();
                    for (uint32_t r = tid; r < n_special; r += kFlatThreads) {
                        const uint32_t p = scol[r] + shift;
                        atomicOr(&bitmap[p >> 5], 1u << (p & 31u));
                    }
                }
                thr = loose;
                __syncthreads();
            }
            if (a.timing && tid == 0)
                a.timing[(size_t)row * 64 + 21] = global_ns();
            // ---- the draw --------------------------------------------------------------------------------------------
            uint32_t draft_idx = 0xffffffffu;
            if (a.mode == kModeVerify && draft_row >= 0) {
                if (tid == 0)
                    s.n_big = 0xffffffffu;
                __syncthreads();
                for (uint32_t i = tid; i < n_take; i += kFlatThreads)
                    if ((int32_t)(uint32_t)(keys[i] & 0xffffffffull) + a.id_offset == draft_row)
                        s.n_big = i;
                __syncthreads();
                draft_idx = s.n_big;
            }
            if (a.timing && tid == 0) {
                a.timing[(size_t)row * 64 + 9] = n;
                a.timing[(size_t)row * 64 + 10] = n_take;
            }
            // the weights alone, in order, for the chains
            const bool on_chip = reinterpret_cast<unsigned char*>(keys) == dyn;
            const uint32_t q_off = on_chip ? (n * 8u + 15u) & ~15u : 0u;
            float* const q = q_off + n_take * 4u <= kFlatDyn ? reinterpret_cast<float*>(dyn + q_off)
                                                             : reinterpret_cast<float*>(row_scratch); // the raw list is dead
            for (uint32_t i = tid; i < n_take; i += kFlatThreads)
                q[i] = __uint_as_float(~(uint32_t)(keys[i] >> 32));
            const uint32_t n_out = min(n_take, a.cand_cap);
            for (uint32_t i = tid; i < n_out; i += kFlatThreads) {
                if (a.cand_ids) a.cand_ids[(size_t)row * a.cand_cap + i] = (int32_t)(uint32_t)(keys[i] & 0xffffffffull) + a.id_offset;
                if (a.cand_q) a.cand_q[(size_t)row * a.cand_cap + i] = __uint_as_float(~(uint32_t)(keys[i] >> 32));
            }
            __syncthreads();
            const RowOut o = {a.token, a.prob, a.flags, a.n_cand, a.accepted, a.total_out, a.cand_ids, a.cand_q,
                              a.cand_cap, a.id_offset, a.timing, a.mode};
            draw_long<kFlatThreads>(s.chain, q, n_take, n_take, draft_idx, row, flags, u_row, u2_row, draft_row, o,
                                    [&](uint32_t i) -> uint32_t { return (uint32_t)(keys[i] & 0xffffffffull); });
            __syncthreads(); // (the mark stays: CTAs that start later count it too)
        }
    }
}

int flat_rows_take(const RowKernelArgs& a)
{
    if (a.n_vocab > kFlatVocab || a.spec_n_pos != 0u)
        return 0; // a column is a bit of the tables; a speculative round's rows have histories of their own kind
    const uint64_t hist = a.history ? (a.history_len ? a.history_ld : (uint64_t)a.n_history) : 0u;
    return hist + a.n_bias <= kSpecialCap ? 2 : 1;
}

cudaError_t launch_flat_rows(const RowKernelArgs& a, uint32_t batch, cudaStream_t stream)
{
    static bool configured[64] = {};
    static int sms[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(flat_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatDyn);
        if (e == cudaSuccess)
            e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess)
            return e;
        configured[dev] = true;
    }
    // One CTA per SM at most; of a chunk of 1024 rows a CTA gets at most ceil(1024 / 128) + 1 <= 16 (FlatSmem::rows), or, where
    // the grid is as large as the batch, one.
    const uint32_t grid = min(batch, (uint32_t)max(128, sms[dev]));
    flat_row_kernel<<<grid, kFlatThreads, kFlatDyn, stream>>>(a, batch);
    return cudaGetLastError();
}

} // namespace mk
