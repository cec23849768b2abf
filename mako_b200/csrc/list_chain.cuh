// The two sequential float chains of a draw — the total of the candidates' weights and the walk that subtracts them one
// by one from u * total (src/gen/sampler.cpp:64-73) — taken by a whole CTA, with the result of the left-to-right order
// to the bit.
//
// Why that is possible: while the running value stays within one binade [2^e, 2^(e+1)) it is a whole number k of units
// u = 2^(e-23), and rounding k*u + q to the nearest unit adds a whole number of units that depends on q alone — except
// for an exact tie, which goes to the even neighbour and so depends on the parity of k as well. A run of candidates is
// therefore a function of the parity it starts with: two increments. Such functions compose, so a scan over the threads
// gives every thread the value its run starts with. The increments come from the float adder itself, by adding the run to
// the smallest even and the smallest odd value of the binade (the largest two for the walk). A run that leaves the
// binade, or in which the walk could end, is taken element by element by its thread; everything before it stands, and the
// next round starts behind it with the new unit. A value crosses at most a few dozen binades.
//
// Latency-bound: a round of kThreads * kRun candidates takes about 400 cycles (two barriers and two five-step scans), a chain
// of dependent additions four cycles and more a candidate.
#pragma once
#include <cstdint>

namespace mk {

constexpr int kRun = 8; // candidates a thread and round
constexpr uint32_t kUnitCap = 1u << 25; // increments are clamped here: past the binade's end whatever they are

template <int kThreads>
struct ChainSmem {
    uint32_t warp0[kThreads / 32], warp1[kThreads / 32]; // increments of whole warps, by starting parity
    uint32_t bad[2];       // first thread whose run leaves the binade (or may end the walk), by round parity
    float value;           // the running value after the round
    uint32_t hit;          // the walk's end
    float r_hit, q_hit;
};

__device__ __forceinline__ void unit_compose(uint32_t& f0, uint32_t& f1, uint32_t a0, uint32_t a1)
{
    // (a then f): f is entered with the parity a leaves
    const uint32_t n0 = a0 + ((a0 & 1u) ? f1 : f0), n1 = a1 + ((a1 & 1u) ? f0 : f1);
    f0 = min(n0, kUnitCap);
    f1 = min(n1, kUnitCap);
}

// Exclusive composition over all threads before this one, entered with parity `p`. One barrier.
template <int kThreads>
__device__ __forceinline__ uint32_t units_before(ChainSmem<kThreads>& cs, uint32_t i0, uint32_t i1, uint32_t p)
{
    constexpr uint32_t kWarps = kThreads / 32;
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t f0 = i0, f1 = i1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a0 = __shfl_up_sync(full, f0, o), a1 = __shfl_up_sync(full, f1, o);
        if ((int)lane >= o)
            unit_compose(f0, f1, a0, a1);
    }
    if (lane == 31u) {
        cs.warp0[warp] = f0;
        cs.warp1[warp] = f1;
    }
    uint32_t e0 = __shfl_up_sync(full, f0, 1), e1 = __shfl_up_sync(full, f1, 1);
    if (lane == 0u)
        e0 = e1 = 0u;
    __syncthreads();
    uint32_t w0 = (lane < kWarps) ? cs.warp0[lane] : 0u, w1 = (lane < kWarps) ? cs.warp1[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a0 = __shfl_up_sync(full, w0, o), a1 = __shfl_up_sync(full, w1, o);
        if ((int)lane >= o)
            unit_compose(w0, w1, a0, a1);
    }
    const uint32_t b0 = __shfl_sync(full, w0, (int)((warp + 31u) & 31u)), b1 = __shfl_sync(full, w1, (int)((warp + 31u) & 31u));
    const uint32_t before = (warp == 0u) ? 0u : (p ? b1 : b0);
    return min(before + (((p + before) & 1u) ? e1 : e0), 2u * kUnitCap);
}

// 2^e as a float, for -126 <= e <= 127.
__device__ __forceinline__ float exp2_int(int e)
{
    return __uint_as_float((uint32_t)(e + 127) << 23);
}

// Running values below this are taken element by element: the unit of a smaller one would be a denormal.
constexpr float kChainFloor = 0x1p-100f;

// fl(...fl(fl(q(0) + q(1)) + q(2))...), q(i) >= 0 (zeros change nothing). Whole CTA; every thread gets the total. The caller
// synchronises before (q readable by all) and need not after.
template <int kThreads, class Q>
__device__ __forceinline__ float chain_total(ChainSmem<kThreads>& cs, uint32_t n, Q&& q_of)
{
    const uint32_t tid = threadIdx.x;
    uint32_t pos = 0, round = 0;
    if (tid == 0) {
        cs.bad[0] = cs.bad[1] = (uint32_t)kThreads;
        cs.value = 0.0f;
    }
    float value = 0.0f;
    __syncthreads();
    while (pos < n) {
        if (!(value >= kChainFloor)) { // the first candidates, until the value is one whose units are normal floats
            if (tid == 0) {
                float v = value;
                uint32_t i = pos;
                const uint32_t stop = min(n, pos + 4096u);
                for (; i < stop && !(v >= kChainFloor); ++i)
                    v = __fadd_rn(v, q_of(i));
                cs.value = v;
                cs.hit = i;
            }
            __syncthreads();
            value = cs.value;
            pos = cs.hit;
            __syncthreads();
            continue;
        }
        const int e = (int)(__float_as_uint(value) >> 23) - 127;
        const float unit = exp2_int(e - 23), per_unit = exp2_int(23 - e), base0 = exp2_int(e), base1 = base0 + unit;
        const uint32_t k = (__float_as_uint(value) & 0x7fffffu) | 0x800000u;
        const uint32_t i0 = pos + tid * (uint32_t)kRun;
        float a0 = base0, a1 = base1;
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
            const float q = (i0 + (uint32_t)j < n) ? q_of(i0 + (uint32_t)j) : 0.0f;
            a0 = __fadd_rn(a0, q);
            a1 = __fadd_rn(a1, q);
        }
        const uint32_t u0 = min(__float2uint_rz((a0 - base0) * per_unit), kUnitCap);
        const uint32_t u1 = min(__float2uint_rz((a1 - base1) * per_unit), kUnitCap);
        const uint32_t start = k + units_before<kThreads>(cs, u0, u1, k & 1u);
        const uint32_t end = start + ((start & 1u) ? u1 : u0);
        const uint32_t slot = round & 1u;
        const bool bad = end >= (1u << 24);
        if (bad)
            atomicMin(&cs.bad[slot], tid);
        else if (tid == (uint32_t)kThreads - 1u)
            cs.value = (float)end * unit;
        if (tid == 0)
            cs.bad[slot ^ 1u] = (uint32_t)kThreads;
        __syncthreads();
        const uint32_t f = cs.bad[slot];
        if (f < (uint32_t)kThreads) { // this thread's run leaves the binade: element by element
            if (tid == f) {
                float v = (float)start * unit;
                for (int j = 0; j < kRun; ++j)
                    if (i0 + (uint32_t)j < n)
                        v = __fadd_rn(v, q_of(i0 + (uint32_t)j));
                cs.value = v;
            }
            __syncthreads();
        }
        value = cs.value;
        pos += (f < (uint32_t)kThreads ? f + 1u : (uint32_t)kThreads) * (uint32_t)kRun;
        ++round;
        // the next write of cs.value and cs.warp* lies behind a barrier of the next round or, for cs.value, behind its scan's
    }
    __syncthreads();
    return value;
}

// The walk: the first i with r_i < q(i), where r_0 = r and r_(i+1) = fl(r_i - q(i)); q(i) >= 0, zeros never win. Returns true
// and leaves i, r_i and q(i) in cs.hit, cs.r_hit, cs.q_hit; false when no candidate stops it. Whole CTA; synchronised on return.
template <int kThreads, class Q>
__device__ __forceinline__ bool chain_walk(ChainSmem<kThreads>& cs, uint32_t n, float r, Q&& q_of)
{
    const uint32_t tid = threadIdx.x;
    uint32_t pos = 0, round = 0;
    if (tid == 0) {
        cs.bad[0] = cs.bad[1] = (uint32_t)kThreads;
        cs.hit = 0xffffffffu;
    }
    __syncthreads();
    while (pos < n) {
        const bool small = !(r >= kChainFloor && r < __int_as_float(0x7f800000)); // also a NaN: no comparison holds
        const int e = small ? 0 : (int)(__float_as_uint(r) >> 23) - 127;
        const float unit = exp2_int(e - 23), per_unit = exp2_int(23 - e);
        const float base1 = exp2_int(e) * 2.0f - unit, base0 = base1 - unit;
        const uint32_t k = (__float_as_uint(r) & 0x7fffffu) | 0x800000u;
        const uint32_t i0 = pos + tid * (uint32_t)kRun;
        float a0 = base0, a1 = base1, top = 0.0f;
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
            const float q = (i0 + (uint32_t)j < n) ? q_of(i0 + (uint32_t)j) : 0.0f;
            a0 = __fsub_rn(a0, q);
            a1 = __fsub_rn(a1, q);
            top = fmaxf(top, q);
        }
        const uint32_t u0 = min(__float2uint_rz((base0 - a0) * per_unit), kUnitCap);
        const uint32_t u1 = min(__float2uint_rz((base1 - a1) * per_unit), kUnitCap);
        const uint32_t before = units_before<kThreads>(cs, u0, u1, k & 1u);
        const uint32_t start = k - min(before, k); // a value that has left the binade lies behind the first bad thread
        const uint32_t units = (start & 1u) ? u1 : u0;
        const uint32_t end = start - min(units, start);
        const uint32_t slot = round & 1u;
        // small values: every run with anything in it that could be larger is looked at element by element
        const bool bad = small ? (top > r) : (top > 0.0f && (end <= (1u << 23) || (float)end * unit < top));
        if (bad)
            atomicMin(&cs.bad[slot], tid);
        else if (tid == (uint32_t)kThreads - 1u)
            cs.value = (float)end * unit;
        if (tid == 0)
            cs.bad[slot ^ 1u] = (uint32_t)kThreads;
        __syncthreads();
        const uint32_t f = cs.bad[slot];
        if (small) {
            // Below the floor r only shrinks further, so the first candidate above it is at most where the walk ends; the few
            // steps up to there are taken one by one.
            if (tid == 0) {
                const uint32_t stop = min(n, pos + (f < (uint32_t)kThreads ? f + 1u : (uint32_t)kThreads) * (uint32_t)kRun);
                for (uint32_t i = pos; i < stop && cs.hit == 0xffffffffu; ++i) {
                    const float q = q_of(i);
                    if (r < q) {
                        cs.hit = i;
                        cs.r_hit = r;
                        cs.q_hit = q;
                    } else {
                        r = __fsub_rn(r, q);
                    }
                }
                cs.value = r;
            }
            __syncthreads();
        } else if (f < (uint32_t)kThreads) {
            if (tid == f) {
                float v = (float)start * unit;
                for (int j = 0; j < kRun && cs.hit == 0xffffffffu; ++j)
                    if (i0 + (uint32_t)j < n) {
                        const float q = q_of(i0 + (uint32_t)j);
                        if (v < q) {
                            cs.hit = i0 + (uint32_t)j;
                            cs.r_hit = v;
                            cs.q_hit = q;
                        } else {
                            v = __fsub_rn(v, q);
                        }
                    }
                cs.value = v;
            }
            __syncthreads();
        }
        if (cs.hit != 0xffffffffu)
            break;
        r = cs.value;
        pos += (f < (uint32_t)kThreads ? f + 1u : (uint32_t)kThreads) * (uint32_t)kRun;
        ++round;
    }
    __syncthreads();
    return cs.hit != 0xffffffffu;
}

} // namespace mk
