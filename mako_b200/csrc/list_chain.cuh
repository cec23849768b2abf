// The two sequential float chains of a draw — the total of the candidates' weights and the walk that subtracts them one
// by one from u * total (src/gen/sampler.cpp:64-73) — taken by a whole CTA, with the result of the left-to-right order
// to the bit.
//
// Why that is possible: while the running value stays within one binade [2^e, 2^(e+1)) it is a whole number k of units
// u = 2^(e-23), and rounding k*u + q to the nearest unit adds a whole number of units that depends on q alone — except
// for an exact tie, which goes to the even neighbour and so depends on the parity of k as well. A run of candidates is
// therefore a function of the parity it starts with: two increments. Such functions compose, so a scan over the lanes of
// a warp gives every lane the value its run starts with. The increments come from the float adder itself, by adding the run to
// the smallest even and the smallest odd value of the binade (the largest two for the walk). A run that leaves the
// binade, or in which the walk could end, is taken element by element; everything before it stands, and the next round
// starts behind it with the new unit. A value crosses at most a few dozen binades.
//
// Ties are rare: where no run of a round has one, the increments are plain numbers, and as long as their sum stays inside the binade
// (and, in a walk, above the largest weight) a round is one reduction. Such rounds are taken by the whole CTA, up to the first
// warp's share that is not like that; one warp takes the others (256 candidates). What bounds both is a round's latency, not
// the number of candidates. (128 masked rows of 3000 candidates: 61.9 us with a scan over the CTA's threads in every round, 60.3 so; lists
// of tens of thousands take the same either way.)
#pragma once
#include <cstdint>

namespace mk {

constexpr uint32_t kRun = 8;            // candidates a thread and round
constexpr uint32_t kUnitCap = 1u << 25; // increments are clamped here: past the binade's end whatever they are
constexpr uint32_t kHead = 64;          // the first candidates of a total, from its first place on
constexpr uint32_t kBeside = 32;        // candidates taken element by element where crossings are close together
constexpr uint32_t kCleanRounds = 4;    // rounds of one warp without a crossing before the CTA takes over
constexpr float kChainFloor = 0x1p-100f; // smaller running values are taken element by element: their unit would be a denormal

template <int kThreads>
struct ChainSmem {
    uint32_t sum[2][kThreads / 32], top[2][kThreads / 32]; // by round parity: a warp's units (bit 31: not a plain number), its largest weight
    float value;           // the running value and the place it stands at
    uint32_t pos;
    uint32_t hit;          // the walk's end
    float r_hit, q_hit;
    uint32_t first, last;  // for the caller: the list's ends that could win
};

// 2^e as a float, for -126 <= e <= 127.
__device__ __forceinline__ float exp2_int(int e)
{
    return __uint_as_float((uint32_t)(e + 127) << 23);
}

__device__ __forceinline__ void unit_compose(uint32_t& f0, uint32_t& f1, uint32_t a0, uint32_t a1)
{
    // (a then f): f is entered with the parity a leaves
    const uint32_t n0 = a0 + ((a0 & 1u) ? f1 : f0), n1 = a1 + ((a1 & 1u) ? f0 : f1);
    f0 = min(n0, kUnitCap);
    f1 = min(n1, kUnitCap);
}

__device__ __forceinline__ void warp_compose(uint32_t& f0, uint32_t& f1)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a0 = __shfl_up_sync(0xffffffffu, f0, o), a1 = __shfl_up_sync(0xffffffffu, f1, o);
        if ((int)(threadIdx.x & 31u) >= o)
            unit_compose(f0, f1, a0, a1);
    }
}

// The eight weights from place i on; zeros past the end, which change nothing and never win. i is a multiple of eight.
__device__ __forceinline__ void load_run(const float* q, uint32_t i, uint32_t n, float (&w)[kRun])
{
    if (i + kRun <= n) {
        const float4 x = *reinterpret_cast<const float4*>(q + i), y = *reinterpret_cast<const float4*>(q + i + 4);
        w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w, w[4] = y.x, w[5] = y.y, w[6] = y.z, w[7] = y.w;
    } else {
#pragma unroll
        for (uint32_t j = 0; j < kRun; ++j)
            w[j] = i + j < n ? q[i + j] : 0.0f;
    }
}

// The units of a binade, and what a run of candidates from i0 on adds to (kDown: takes from) a value in it.
template <bool kDown>
struct Binade {
    float unit, per_unit, base0, base1;
    uint32_t k; // the running value in units
    __device__ __forceinline__ explicit Binade(float value)
    {
        const int e = (int)(__float_as_uint(value) >> 23) - 127;
        unit = exp2_int(e - 23);
        per_unit = exp2_int(23 - e);
        base0 = kDown ? exp2_int(e) * 2.0f - 2.0f * unit : exp2_int(e);
        base1 = base0 + unit;
        k = (__float_as_uint(value) & 0x7fffffu) | 0x800000u;
    }
    __device__ __forceinline__ void run(const float* q, uint32_t i0, uint32_t n, uint32_t& u0, uint32_t& u1, float& top) const
    {
        float w[kRun];
        load_run(q, i0, n, w);
        float a0 = base0, a1 = base1;
        top = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < kRun; ++j) {
            a0 = kDown ? __fsub_rn(a0, w[j]) : __fadd_rn(a0, w[j]);
            a1 = kDown ? __fsub_rn(a1, w[j]) : __fadd_rn(a1, w[j]);
            if (kDown)
                top = fmaxf(top, w[j]);
        }
        u0 = min(__float2uint_rz((kDown ? base0 - a0 : a0 - base0) * per_unit), kUnitCap);
        u1 = min(__float2uint_rz((kDown ? base1 - a1 : a1 - base1) * per_unit), kUnitCap);
    }
    // the value in units after `before` units, and whether a run that takes it to `end` has to be looked at by element
    __device__ __forceinline__ uint32_t after(uint32_t from, uint32_t units) const
    {
        return kDown ? from - min(units, from) : from + units;
    }
    __device__ __forceinline__ bool bad(uint32_t end, float top) const
    {
        return kDown ? top > 0.0f && (end <= (1u << 23) || (float)end * unit < top) : end >= (1u << 24);
    }
};

// Eight steps of a chain, one after the other; true when the walk ends in them (`hit` of them are passed, v is what is left).
template <bool kDown>
__device__ __forceinline__ bool chain_steps(float& v, const float (&w)[kRun], uint32_t& hit)
{
    if (!kDown) {
#pragma unroll
        for (uint32_t j = 0; j < kRun; ++j)
            v = __fadd_rn(v, w[j]);
        return false;
    }
    uint32_t short_of = 0u;
    float r = v;
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j) {
        short_of |= (r < w[j]) ? 1u << j : 0u;
        r = __fsub_rn(r, w[j]);
    }
    if (!short_of) {
        v = r;
        return false;
    }
    hit = (uint32_t)__ffs((int)short_of) - 1u;
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j)
        if (j < hit)
            v = __fsub_rn(v, w[j]);
    return true;
}

// The chain over q[0 .. n) from `value` on (q 16-byte aligned, no weight negative; zeros change nothing and never win). It starts at
// `from`, a multiple of eight with nothing but zeros in front of it: while a total is zero there is no unit to count in, and a list
// laid out by column may have a hundred thousand of them (two rows of 151552 columns that allow the last 20000: 3.8 ms, 0.25 ms so). The
// total (kDown false): fl(...fl(fl(value + q0) + q1)...), returned. The walk (kDown true): the first i with r_i < q[i], r_0 =
// value, r_(i+1) = fl(r_i - q[i]), left with r_i and q[i] in cs.hit, cs.r_hit, cs.q_hit; cs.hit is 0xffffffff when nothing
// stops it. Whole CTA; the caller synchronises before; synchronised on return.
template <int kThreads, bool kDown>
__device__ __forceinline__ float chain(ChainSmem<kThreads>& cs, const float* q, uint32_t n, float value, uint32_t from = 0u)
{
    constexpr uint32_t kWarps = kThreads / 32, none = 0xffffffffu;
    const uint32_t full = 0xffffffffu, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t pos = from, round = 0;
    if (tid == 0)
        cs.hit = none;
    __syncthreads();
    while (pos < n) {
        if (warp == 0) { // every lane knows value and pos
            uint32_t clean = 0, hit = none;
            float r_hit = 0.0f;
            while (pos < n && clean < kCleanRounds && hit == none) {
                // Taken element by element: the start of a total, where the value doubles every few candidates; where a run
                // leaves the binade, with the runs behind it (it often leaves the next one soon); and small values.
                uint32_t stop = pos + kBeside;
                const bool small = !(value >= kChainFloor && value < __int_as_float(0x7f800000)); // a NaN too
                if (!small && (kDown || pos >= from + kHead)) {
                    const Binade<kDown> b(value);
                    uint32_t u0, u1;
                    float top;
                    b.run(q, pos + lane * kRun, n, u0, u1, top);
                    uint32_t e = 0u; // the units of the lanes before this one
                    if (__all_sync(full, u0 == u1)) {
                        const uint32_t end_all = b.after(b.k, __reduce_add_sync(full, u0));
                        const float top_all = kDown ? __uint_as_float(__reduce_max_sync(full, __float_as_uint(top))) : 0.0f;
                        if (!b.bad(end_all, top_all)) {
                            value = (float)end_all * b.unit;
                            pos += 32u * kRun;
                            ++clean;
                            continue;
                        }
                        e = u0;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t y = __shfl_up_sync(full, e, o);
                            if ((int)lane >= o)
                                e += y;
                        }
                        e -= u0;
                    } else {
                        uint32_t f0 = u0, f1 = u1;
                        warp_compose(f0, f1);
                        e = __shfl_up_sync(full, (b.k & 1u) ? f1 : f0, 1);
                        if (lane == 0u)
                            e = 0u;
                    }
                    const uint32_t start = b.after(b.k, e), end = b.after(start, (start & 1u) ? u1 : u0);
                    const uint32_t bad = __ballot_sync(full, b.bad(end, top));
                    if (!bad) {
                        value = (float)__shfl_sync(full, end, 31) * b.unit;
                        pos += 32u * kRun;
                        ++clean;
                        continue;
                    }
                    const uint32_t f = (uint32_t)__ffs((int)bad) - 1u;
                    value = (float)__shfl_sync(full, start, (int)f) * b.unit;
                    pos += f * kRun;
                    stop = pos + (f < 4u ? kBeside : kRun);
                    clean = 0;
                }
                for (; pos < min(stop, n) && hit == none; pos += kRun) {
                    float w[kRun];
                    load_run(q, pos, n, w);
                    uint32_t passed;
                    if (chain_steps<kDown>(value, w, passed)) {
                        hit = pos + passed;
                        r_hit = value;
                    }
                }
            }
            if (lane == 0u) {
                cs.value = value;
                cs.pos = hit != none ? n : pos;
                if (hit != none) {
                    cs.hit = hit;
                    cs.r_hit = r_hit;
                    cs.q_hit = q[hit];
                }
            }
        }
        __syncthreads();
        value = cs.value;
        pos = cs.pos;
        // Rounds of the whole CTA, a barrier each, for as long as no warp's runs cross a binade or hold a tie; warp 0 goes on
        // at the first that does.
        while (pos < n && value >= kChainFloor) {
            const Binade<kDown> b(value);
            uint32_t u0, u1;
            float top;
            b.run(q, pos + tid * kRun, n, u0, u1, top);
            const uint32_t slot = round & 1u;
            ++round;
            const bool plain = __all_sync(full, u0 == u1);
            const uint32_t own = min(__reduce_add_sync(full, u0), kUnitCap);
            const uint32_t largest = kDown ? __reduce_max_sync(full, __float_as_uint(top)) : 0u;
            if (lane == 0u) {
                cs.sum[slot][warp] = own | (plain ? 0u : 0x80000000u);
                cs.top[slot][warp] = largest;
            }
            __syncthreads();
            // lane w: warp w's units, and where they take the value
            const uint32_t entry = (lane < kWarps) ? cs.sum[slot][lane] : 0u, units = entry & 0x7fffffffu;
            const float top_w = (kDown && lane < kWarps) ? __uint_as_float(cs.top[slot][lane]) : 0.0f;
            uint32_t inc = units;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(full, inc, o);
                if ((int)lane >= o)
                    inc += y;
            }
            const uint32_t start = b.after(b.k, inc - units), end = b.after(b.k, inc);
            const uint32_t stops = __ballot_sync(full, (entry >> 31) || b.bad(end, top_w));
            if (stops) {
                const int f = __ffs((int)stops) - 1;
                value = (float)__shfl_sync(full, start, f) * b.unit;
                pos += (uint32_t)f * 32u * kRun;
                break;
            }
            value = (float)__shfl_sync(full, end, 31) * b.unit;
            pos += (uint32_t)kThreads * kRun;
        }
        __syncthreads(); // everyone has read the round's results before warp 0 writes there again
    }
    return value;
}

} // namespace mk
