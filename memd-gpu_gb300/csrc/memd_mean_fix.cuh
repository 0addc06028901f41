// memd_mean_fix.cuh -- mean envelope of the FP64 form by impulse accumulation
// in wide fixed point (fixed number of sifts).
#pragma once

#include "memd_kernels.cuh"

namespace memd {

// The reference evaluates every envelope at every sample (REF:795-864): four
// FP64 operations per direction, envelope, channel and sample, on a pipe that
// issues two lanes per clock and SM (1.25 TFLOP/s, 1/63 of the FP32 rate).
// Here, as in the mixed form's mean (k_mean_cum), the mean is rebuilt from
// what happens at the knots: between an anchor sample and its neighbours the
// sum of all envelopes is one cubic, whose third-order coefficient jumps by
// d_j - d_{j-1} at every knot x_j.  FP64 operations are left at the knots
// (two) and at the anchors (ten) only; every sum is an integer sum.
//
// Fixed point: values are integers in units of 2^-sh, held as two words, v =
// hi 2^52 + lo with 0 <= lo < 2^52.  The unit is the span's own: 2^-sh =
// 2^(ex - 85) with 2^ex > max|x| over the channel's samples in the span, so a
// quiet stretch keeps its accuracy however loud the rest of the channel is (a
// third-order coefficient is rounded to the unit and then multiplied by up to
// (T/2)^3 = 2^15: with a unit of the whole channel, a stretch 2^-26 as loud as
// the channel's largest sample lost a few bits at T = 64).  Where a coefficient
// does not fit (knots or overshoot from outside the span, 2^12 and more times
// its samples), the unit is raised by exactly what the span's largest needs and
// the pairs are gone through once more for those channels.  Sums over at most
// 2048 (direction, envelope) pairs stay inside both words, and the exact sums
// make the result independent of the order, of the batch a record is in and of
// the direction passes (of several passes that need units raised differently,
// the sums are brought to the coarsest, within its rounding).
//
// Anchors: every T samples, T the power of two in [8, 64] with T <= 3 h (h:
// the record's mean knot spacing over all directions; 8 at the densest
// knots).  Rounding in a piece's coefficients grows with the distance from
// the anchor, at most T/2.  Error of the mean against a long double
// evaluation, relative to the signal (3 channels, 32 directions, EEG-shaped;
// direct FP64 evaluation 1.5e-16 in an IMF's first sift, 2.3e-17 .. 4.2e-17 in
// its last; the update's own rounding ~4e-17): T = 8 at h = 3.7 / 2.8: 3.8e-17
// / 6.2e-17; T = 16 at h = 7.0 / 5.2: 4.9e-17 / 7.5e-17; T = 32 at h = 13 / 10:
// 4.7e-17 / 7.4e-17; twice the span, 2x .. 4x the error.
// Measured (FP64 form, all sifts of a decomposition, against the direct
// evaluation of every envelope at every sample, 82% busy on the FP64 pipe): 32
// x 30,504, 64 directions, 80 sifts: 117.6 -> 21.2 ms of the mean (29.6 with T
// <= 2 h, integer conversions on the FP64 pipe, one CTA per 64 samples and the
// samples behind an anchor all by one warp); error of the IMFs against a
// separate FP64 evaluation 8.2e-16 -> 4.0e-16.  The unit per span (its samples
// read once more, the coefficients' exponents followed) costs 1.2% of the run:
// 43.5 -> 44.05 ms.
//
// A span with non-finite values, and one so small that its third-order
// coefficients would be subnormal, is evaluated directly, pair by pair in
// direction order, with k_eval_w's arithmetic.
struct FixSum {
    unsigned long long hi, lo;
};
constexpr unsigned long long kFixLo = (1ull << 52) - 1ull;
constexpr int kFixBits = 85;   // units per 2^ex: 2^85
constexpr int kFixMin = 128 << 20;  // smallest high word of a span's largest value (0: all zero)
constexpr int kFixInf = 0x7ff << 20;
constexpr int kFixUnitExp = 32;  // smallest exponent a unit is chosen for: 2^-1075, where no subnormal is too large
constexpr int kFixRows = 64;   // longest span
constexpr int kFixAnchors = 4; // anchors of a span: 32 / 8

// v 2^sh rounded to nearest; raises mx to |v|'s high word.  Integer
// instructions only: FP64 <-> integer conversions run on the FP64 pipe.
__device__ __forceinline__ FixSum to_fix(double v, int sh, int& mx)
{
    FixSum r;
    const long long b = __double_as_longlong(v);
    const int be = (int)((unsigned long long)b >> 52) & 0x7ff;
    long long m = (b & (long long)kFixLo) | (be ? (1ll << 52) : 0ll);
    if (b < 0) m = -m;
    const int s = max(be, 1) - 1075 + sh;  // value = m 2^s units
    if (s >= 0) {
        r.hi = (unsigned long long)(s < 52 ? m >> (52 - s) : m << min(s - 52, 63));
        r.lo = s < 52 ? ((unsigned long long)m << s) & kFixLo : 0ull;
    } else {
        const int q = min(-s, 62);
        const long long n = (m + (1ll << (q - 1))) >> q;
        r.hi = (unsigned long long)(n >> 52);
        r.lo = (unsigned long long)n & kFixLo;
    }
    mx = max(mx, __double2hiint(v) & 0x7fffffff);
    return r;
}
// how far the unit 2^-sh must be raised so that every value with a high word
// of at most mx stays below 2^lim units
__device__ __forceinline__ int fix_excess(int mx, int sh, int lim) { return (mx >> 20) - 1075 + sh - (lim - 53); }

// the 128-bit two's-complement integer n times 2^-sh, rounded to nearest even
__device__ __forceinline__ double from_fix(__int128 n, int sh)
{
    if (n == 0) return 0.0;
    const bool neg = n < 0;
    const unsigned __int128 a = neg ? -(unsigned __int128)n : (unsigned __int128)n;
    const unsigned long long ah = (unsigned long long)(a >> 64), al = (unsigned long long)a;
    const int lz = ah ? __clzll((long long)ah) : 64 + __clzll((long long)al);
    const unsigned __int128 t = a << lz;  // leading bit at 127
    unsigned long long top = (unsigned long long)(t >> 75);  // 53 bits
    const unsigned long long rest = (unsigned long long)(t >> 11);  // the 64 bits below, sticky from the last 11
    const bool sticky = ((unsigned long long)t & 0x7ffull) != 0ull;
    const unsigned long long half = 1ull << 63;
    if (rest > half || (rest == half && (sticky || (top & 1ull)))) ++top;  // 2^53: the exponent absorbs the carry
    const int be = 127 - lz - sh + 1023;
    double v;
    if (be >= 1 && be <= 2045) v = __longlong_as_double((long long)(((unsigned long long)be << 52) + (top - (1ull << 52))));
    else v = ldexp((double)top, 127 - lz - sh - 52);
    return neg ? -v : v;
}

// accumulator of several direction passes: the exact sum (below 2^115) in 116
// bits and, in the top 12, how far its unit is raised, or kFixDirect and the
// FP64 sum of a span that was evaluated directly
constexpr int kFixDirect = 0xfff;
__device__ __forceinline__ ulonglong2 fix_pack(__int128 v, int raise)
{
    return make_ulonglong2((unsigned long long)v,
                           ((unsigned long long)((unsigned __int128)v >> 64) & kFixLo) | ((unsigned long long)raise << 52));
}
__device__ __forceinline__ int fix_raise(ulonglong2 o) { return (int)(o.y >> 52); }
__device__ __forceinline__ __int128 fix_sum(ulonglong2 o)
{
    const long long hi = (long long)(o.y << 12) >> 12;
    return ((__int128)hi << 64) | (__int128)o.x;
}
// v in a unit raised by n >= 0 more, rounded to nearest
__device__ __forceinline__ __int128 fix_coarser(__int128 v, int n)
{
    if (n == 0) return v;
    return n > 120 ? (__int128)0 : (v + ((__int128)1 << (n - 1))) >> n;
}

// 2^ex > max|x|: ex from the high word of the largest sample
__device__ __forceinline__ int fix_shift(int mx) { return kFixBits - (max(mx >> 20, kFixUnitExp) - 1022); }

// 2 v (exact); by an integer addition to the exponent for a normal value
__device__ __forceinline__ double twice(double v)
{
    const int hi = __double2hiint(v);
    if ((unsigned)(hi & 0x7ff00000) - 0x00100000u < 0x7fd00000u) return __hiloint2double(hi + 0x00100000, __double2loint(v));
    return __dadd_rn(v, v);
}

// CTA: one 32-sample word x G channels, 8 warps; lane = (subgroup, channel); the
// (direction, envelope) pairs are dealt round-robin to the 8 * 32/G subgroups,
// which walk the word's pieces in order.  Where T = 64 the two CTAs of a
// cluster share a 64-sample span: each takes half the pairs, then, with the
// other's sums from distributed shared memory, half the rows.
// Bound by the FP64 pipe at dense knots, by load latency at sparse ones.
template <int G, bool MIR>
__global__ void __launch_bounds__(256, 3)
k_mean_fix(const double* __restrict__ X, double* __restrict__ Xout, ulonglong2* __restrict__ acc_buf,
           const uint32_t* __restrict__ bits, const int* __restrict__ wpref, const int* __restrict__ knots,
           const int* __restrict__ cnt, const double* __restrict__ rtab, const double2* __restrict__ rtab3,
           const double* __restrict__ sv, const double* __restrict__ yend, const unsigned long long* __restrict__ tot, Geom g, int k0, int Kc, int first_chunk, int last_chunk,
           RunState* st, Epochs ep, const int* __restrict__ mir)
{
    // MIR (mirror boundary, one record): the knot list is [left mirrored |
    // interior | right mirrored]

    constexpr int SUB = 32 / G;
    constexpr int NWS = 8 * SUB;
    constexpr int NE = 256;  // pairs described per round
    // sums, as four 32-bit words each (hi's low and high word, lo's low and high
    // word, NS apart): rows 0 .. kFixRows - 1 the jumps at row x - p0, then
    // [kFixAnchors][4] Taylor coefficients at the anchors; [..][G]
    constexpr int NS = (kFixRows + 4 * kFixAnchors) * G, AN = kFixRows * G;
    extern __shared__ __align__(16) unsigned sums[];
    auto add = [&](int i, unsigned long long hi, unsigned long long lo) {
        add_words(sums, sums + NS, i, hi);
        add_words(sums + 2 * NS, sums + 3 * NS, i, lo);
    };
    __shared__ int eJ[NE], eE[NE];  // first piece of the span (-1: the pair does not count); last piece of the record
    __shared__ int sQ, sT;
    __shared__ unsigned sBad;  // channels of the span to evaluate directly
    __shared__ int sMax[G], sRaise[G];  // high word of the channels' largest sample; how far their units are raised
    __shared__ unsigned long long sEt;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cc = lane % G, sub = lane / G;
    const int C = g.C;
    const int weven = (int)blockIdx.x & ~1;  // the cluster's first word (records start at even words)
    const int rec = ep.n > 0 ? ep.wep[weven] : 0;
    const int roff = ep.n > 0 ? ep.off[rec] : 0;
    const int rend = ep.n > 0 ? roff + ep.len[rec] : g.L;
    if (weven * 32 >= rend) return;  // gap between epochs; uniform over the cluster
    if (threadIdx.x == 0) {
        sQ = 0;
        sBad = 0u;
        sEt = 0ull;
    }
    if (threadIdx.x < G) sMax[threadIdx.x] = sRaise[threadIdx.x] = 0;
    __syncthreads();
    {
        // qualified directions, and the knots of all of them (spans of several
        // passes: counted beforehand, so that T does not depend on the passes)
        int q = 0;
        unsigned long long et = 0ull;
        for (int k = threadIdx.x; k < g.K; k += blockDim.x) {
            const int a = ep.n > 0 ? ep.cnt[(size_t)k * ep.n + rec] : cnt[k];
            const int b = ep.n > 0 ? ep.cnt[((size_t)g.K + k) * ep.n + rec] : cnt[g.K + k];
            q += (a > 3 && b > 3) ? 1 : 0;
            et += (unsigned long long)(a + b);
            if constexpr (MIR) {  // interior knots, as the count of several passes
                const int* mi = mir + (size_t)k * kMirWords;
                et -= (unsigned long long)(mi[kMirNl] + mi[kMirNr] + mi[kMirNl + 1] + mi[kMirNr + 1]);
            }
        }
        q = warp_sum(q);
        et = warp_sum(et);
        if (lane == 0) {
            if (q) atomicAdd(&sQ, q);
            if (et) atomicAdd(&sEt, et);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long et = tot ? tot[rec] : sEt;
        const unsigned long long lk = (unsigned long long)(rend - roff) * 2ull * (unsigned long long)g.K;
        int t = 8;  // T <= 3 h, h = lk / et
        while (t < kFixRows && (unsigned long long)(2 * t) * et <= 3ull * lk) t *= 2;
        sT = t;
    }
    __syncthreads();
    const int T = sT;
    const bool pair = T > 32;  // uniform over the cluster, and the returns below over the CTA
    const int half = (int)blockIdx.x & 1;
    const int w = pair ? weven : (int)blockIdx.x;
    const int p0 = w * 32;
    if (p0 >= rend) return;
    const int nl = min(pair ? 64 : 32, rend - p0);
    // this CTA's pairs
    const int e_lo = pair && half ? Kc : 0, e_hi = pair && !half ? Kc : 2 * Kc;
    const int nA = (nl + T - 1) / T;
    const int c = blockIdx.y * G + cc;
    const bool cok = c < C;
    const int cl = min(c, C - 1);  // loads of lanes past the last channel stay in bounds
    double xr[kFixRows * G / 256];  // the span's samples of this thread's channel (blockDim.x is a multiple of G)
#pragma unroll
    for (int k = 0; k < kFixRows * G / 256; ++k) {
        const int r = (int)threadIdx.x / G + k * (256 / G);
        xr[k] = r < nl ? X[(size_t)(p0 + r) * C + cl] : 0.0;
    }
    for (int j = 0; j < 4; ++j) {
        for (int i = threadIdx.x; i < nl * G; i += blockDim.x) sums[j * NS + i] = 0u;
        for (int i = threadIdx.x; i < nA * 4 * G; i += blockDim.x) sums[j * NS + AN + i] = 0u;
    }
    {
        int m = 0;
#pragma unroll
        for (int k = 0; k < kFixRows * G / 256; ++k) {
            const int h = (__double2hiint(xr[k]) & 0x7fffffff) | (__double2loint(xr[k]) ? 1 : 0);
            m = max(m, h < kFixInf ? h : 0);
        }
        if (m) atomicMax(&sMax[cc], m);
    }
    // the sum of the 2K envelopes stays below 2^115: A, B T/2, C (T/2)^2 and
    // d (T/2)^3 of each below 2^lim
    const int lim = 108 - (32 - __clz(2 * g.K - 1));
    const int lt = 30 - __clz(T);  // log2(T / 2)
    const int rlast = rend - 1;
    int raise = 0, sh = 0;                // how far the channel's unit is raised; 2^-sh, the unit
    bool again = false;
    unsigned obad = 0u;                   // the other half's sBad
    int mA = 0, mB = 0, mC = 0, mD = 0;   // high words of the largest of the anchors' coefficients and of d

    for (;;) {
    for (int base = e_lo; base < e_hi; base += NE) {
        __syncthreads();
        {
            // (1) per pair: the piece holding sample p0 and the record's last piece
            const int ei = base + (int)threadIdx.x;
            int j = -1, je = 0;
            if (ei < e_hi) {
                const int kk = ei >> 1, env = ei & 1, k = k0 + kk;
                const int Ex = cnt[k], En = cnt[g.K + k];
                if (Ex <= g.cap && En <= g.cap && dir_qualifies(g, ep, cnt, k, rec)) {
                    const size_t slot = (size_t)env * Kc + kk;
                    const int* wp = wpref + slot * (g.W + 1);
                    const int kb = ep.n > 0 ? wp[ep.w0[rec]] : 0;
                    je = (ep.n > 0 ? wp[ep.w0[rec + 1]] : (env ? En : Ex)) - 2;
                    int at = wp[w] + (int)(bits[slot * g.W + w] & 1u);  // knots at or before p0
                    if constexpr (MIR) {
                        int lp0, lp1, rp0, rp1;
                        mirror_positions(mir + (size_t)k * kMirWords, knots + slot * g.cap, env, je + 2, lp0, lp1, rp0,
                                         rp1);
                        at += mirror_before(p0 + 1, lp0, lp1, rp0, rp1);
                    }
                    j = min(max(at - 1, kb), je);
                }
            }
            if (threadIdx.x < NE) {
                eJ[threadIdx.x] = j;
                eE[threadIdx.x] = je;
            }
        }
        __syncthreads();
        sh = fix_shift(sMax[cc]) - raise;
        const int nround = min(NE, e_hi - base);
        for (int le = warp * SUB + sub; le < nround; le += NWS) {
            int j = eJ[le];
            if (j < 0) continue;
            const int je = eE[le];
            const int kk = (base + le) >> 1, env = (base + le) & 1;
            const size_t slot = (size_t)env * Kc + kk;
            const int* kn = knots + slot * g.cap;
            const double* sp = sv + slot * (size_t)g.cap * C + cl;
            const double* ye = yend + (slot * (ep.n > 0 ? ep.n : 1) + rec) * 2 * (size_t)C + cl;
            // (2) the pieces of the span in order: the jump of d at each interior
            //     knot past p0, the Taylor coefficients at each anchor
            int xj = kn[j], xn = kn[j + 1];
            double s0 = sp[(size_t)j * C], s1 = sp[(size_t)(j + 1) * C];
            FixSum qp{0ull, 0ull};
            int a = 0, na = p0 + min(T >> 1, nl - 1);
            bool jump = false;  // x_j is past p0 (the first piece's knot is not)
            for (;;) {
                const bool more = j < je && xn < p0 + nl;  // another piece begins in the span
                int x2 = 0;
                double s2 = 0.0;
                if (more) {
                    x2 = kn[j + 2];
                    s2 = sp[(size_t)(j + 2) * C];
                }
                const int h = xn - xj;
                const double2 r3 = rtab3[h];  // 1 / (3 h), h / 3
                const double d = __dmul_rn(__dsub_rn(s1, s0), r3.x);
                const FixSum qc = to_fix(d, sh, mD);
                if (jump && MEMD_CHECK(xj - p0 > 0 && xj - p0 < nl)) {
                    add((xj - p0) * G + cc, qc.hi - qp.hi, qc.lo - qp.lo);
                }
                qp = qc;
                while (a < nA && (na < xn || j == je)) {
                    // S(na + t) = A + B t + C t^2 + d t^3 on this piece
                    double y0, y1;
                    if constexpr (MIR) {
                        const int* mi = mir + (size_t)(k0 + kk) * kMirWords;
                        y0 = X[(size_t)mirror_source(mi, env, j, je + 2, xj) * C + cl];
                        y1 = X[(size_t)mirror_source(mi, env, j + 1, je + 2, xn) * C + cl];
                    } else {
                        y0 = (xj == roff) ? ye[0] : X[(size_t)xj * C + cl];
                        y1 = (xn == rlast) ? ye[C] : X[(size_t)xn * C + cl];
                    }
                    const double u = from_int<double>(na - xj), u3 = from_int<double>(3 * (na - xj));
                    const double b = __fma_rn(-r3.y, __fma_rn(2.0, s0, s1), __dmul_rn(__dsub_rn(y1, y0), rtab[h]));
                    const double e = __fma_rn(d, u, s0);
                    const double cB = __fma_rn(__fma_rn(d, u3, twice(s0)), u, b);
                    const int at = AN + a * 4 * G + cc;
                    const FixSum fA = to_fix(__fma_rn(__fma_rn(e, u, b), u, y0), sh, mA);
                    const FixSum fB = to_fix(cB, sh, mB);
                    const FixSum fC = to_fix(__fma_rn(d, u3, s0), sh, mC);
                    add(at, fA.hi, fA.lo);
                    add(at + G, fB.hi, fB.lo);
                    add(at + 2 * G, fC.hi, fC.lo);
                    add(at + 3 * G, qc.hi, qc.lo);
                    ++a;
                    na = p0 + a * T + min(T >> 1, nl - 1 - a * T);
                }
                if (!more) break;
                ++j;
                xj = xn;
                xn = x2;
                s0 = s1;
                s1 = s2;
                jump = true;
            }
        }
    }
    if (again) break;
    const int over = max(max(fix_excess(mA, sh, lim), fix_excess(mB, sh, lim - lt)),
                         max(fix_excess(mC, sh, lim - 2 * lt), fix_excess(mD, sh, lim - 3 * lt)));
    const int large = max(sMax[cc], mA);
    if (max(max(mA, mB), max(mC, mD)) >= kFixInf || (large > 0 && large < kFixMin)) atomicOr(&sBad, 1u << cc);
    else if (over > 0) atomicMax(&sRaise[cc], over);
    __syncthreads();
    raise = sRaise[cc];
    if (pair) {  // the same decisions in both halves
        namespace cg_ = cooperative_groups;
        const auto cl_ = cg_::this_cluster();
        cl_.sync();
        obad = *cl_.map_shared_rank(&sBad, 1 - half);
        raise = max(raise, cl_.map_shared_rank(sRaise, 1 - half)[cc]);
    }
    if (((sBad | obad) >> cc) & 1u) raise = 0;
    again = __syncthreads_or(raise > 0);
    if (!again) break;
    for (int j = 0; j < 4; ++j) {
        for (int i = threadIdx.x; i < nl * G; i += blockDim.x) sums[j * NS + i] = 0u;
        for (int i = threadIdx.x; i < nA * 4 * G; i += blockDim.x) sums[j * NS + AN + i] = 0u;
    }
    }  // once more
    if (again) __syncthreads();
    if (pair) {
        // the other half's sums: read them all, and only then change this CTA's
        namespace cg_ = cooperative_groups;
        const auto cl_ = cg_::this_cluster();
        if (again) cl_.sync();
        constexpr int NV = (kFixRows + 4) * G / 256 + 1;
        const unsigned* os = cl_.map_shared_rank(sums, 1 - half);
        const int nk = nl * G, nv = nk + 4 * G;  // rows, then the anchor (nA = 1)
        for (int word = 0; word < 4; word += 2) {
            unsigned long long v[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const int i = (int)threadIdx.x + 256 * j, at = (i < nk ? i : AN + i - nk) + word * NS;
                v[j] = i < nv ? ((unsigned long long)os[at + NS] << 32) | os[at] : 0ull;
            }
            cl_.sync();
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const int i = (int)threadIdx.x + 256 * j, at = (i < nk ? i : AN + i - nk) + word * NS;
                if (i < nv) {
                    v[j] += ((unsigned long long)sums[at + NS] << 32) | sums[at];
                    sums[at] = (unsigned)v[j];
                    sums[at + NS] = (unsigned)(v[j] >> 32);
                }
            }
        }
        __syncthreads();
    }
    const int Q = sQ;
    if (last_chunk && Q == 0 && blockIdx.y == 0 && threadIdx.x == 0) atomicOr(&st->flags, 1);
    if (!cok) return;
    const double qd = (double)Q, rq = Q > 0 ? __ddiv_rn(1.0, qd) : __longlong_as_double(0x7ff8000000000000ll);
    const bool bad = ((sBad | obad) >> cc) & 1u;
    // M's sum at row r is done: X -= M / 2 / Q, or on to the next pass; x: X there
    auto emit = [&](int r, __int128 v, double vd, double x) {
        const size_t off = (size_t)(p0 + r) * C + c;
        bool isd = bad;
        int up = raise, shv = sh;
        if (!first_chunk) {
            const ulonglong2 o = acc_buf[off];
            const int ro = fix_raise(o);
            if (ro == kFixDirect || isd) {
                const double od = ro == kFixDirect ? __longlong_as_double((long long)o.x)
                                                   : from_fix(fix_sum(o), sh + raise - ro);
                vd = __dadd_rn(od, isd ? vd : from_fix(v, sh));
                isd = true;
            } else {
                up = max(ro, raise);
                v = fix_coarser(v, up - raise) + fix_coarser(fix_sum(o), up - ro);
                shv = sh + raise - up;
            }
        }
        if (last_chunk) {
            // (sum / 2) / Q rounded as a division: quotient by the correctly
            // rounded reciprocal, one correction by the remainder (Markstein 1990;
            // the remainder is exact, the units of a sum that is not evaluated
            // directly being far above the subnormals)
            const double val = __dmul_rn(isd ? vd : from_fix(v, shv), 0.5);
            double m;
            if (isd) {
                m = __ddiv_rn(val, qd);
            } else {
                const double q0 = __dmul_rn(val, rq);
                m = __fma_rn(__fma_rn(-q0, qd, val), rq, q0);
                (void)MEMD_CHECK(m == __ddiv_rn(val, qd) || Q == 0);
            }
            Xout[off] = __dsub_rn(x, m);
        } else {
            acc_buf[off] = isd ? make_ulonglong2((unsigned long long)__double_as_longlong(vd), (unsigned long long)kFixDirect << 52)
                               : fix_pack(v, up);
        }
    };
    auto wide = [&](int i) -> __int128 {
        const unsigned long long hi = ((unsigned long long)sums[NS + i] << 32) | sums[i];
        const unsigned long long lo = ((unsigned long long)sums[3 * NS + i] << 32) | sums[2 * NS + i];
        return ((__int128)(long long)hi << 52) + (__int128)(long long)lo;
    };
    // (3) the samples on either side of an anchor, in blocks of at most RB rows
    //     (one block per subgroup): forwards from the anchor, or backwards, the
    //     cubic's coefficients carried from sample to sample (at first without
    //     output, up to the block) and d changed at every knot
    constexpr int RB = 4;
    const int nside = pair ? 1 : 2 * ((32 + T - 1) / T);   // sides this CTA covers
    const int per = max(1, NWS / nside);                   // blocks per side
    const int rows = (T / 2 + per - 1) / per;              // rows per block, at most RB
    for (int it = warp * SUB + sub; it < nside * per; it += NWS) {
        const int sd = it / per, blk = it - sd * per;
        const int a = pair ? 0 : sd >> 1, back = pair ? half : sd & 1;
        const int q0 = a * T;
        if (q0 >= nl) continue;
        const int q1 = min(nl, q0 + T);
        const int ra = q0 + min(T >> 1, nl - 1 - q0);
        const int lo = back ? max(q0, ra - (blk + 1) * rows) : ra + blk * rows;  // rows [lo, hi)
        const int hi = back ? ra - blk * rows : min(q1, lo + rows);
        if (lo >= hi) continue;
        double xs[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) xs[k] = last_chunk && lo + k < hi ? X[(size_t)(p0 + lo + k) * C + c] : 0.0;
        if (!bad) {
            const int at = AN + a * 4 * G + cc;
            __int128 vA = wide(at), vB = wide(at + G), vC = wide(at + 2 * G), vD = wide(at + 3 * G);
            auto forth = [&](int r) {  // from row r - 1 to row r
                vA += vB + vC + vD;
                vB += 2 * vC + 3 * vD;
                vC += 3 * vD;
                vD += wide(r * G + cc);
            };
            auto aback = [&](int r) {  // from row r to row r - 1
                vD -= wide(r * G + cc);
                vA += vC - vB - vD;
                vB += 3 * vD - 2 * vC;
                vC -= 3 * vD;
            };
            if (!back) {
                for (int r = ra + 1; r <= lo; ++r) forth(r);
#pragma unroll
                for (int k = 0; k < RB; ++k) {
                    if (lo + k >= hi) break;
                    if (k) forth(lo + k);
                    emit(lo + k, vA, 0.0, xs[k]);
                }
            } else {
                for (int r = ra; r > hi; --r) aback(r);
#pragma unroll
                for (int k = RB - 1; k >= 0; --k) {
                    if (lo + k >= hi) continue;
                    aback(lo + k + 1);
                    emit(lo + k, vA, 0.0, xs[k]);
                }
            }
        } else {
            for (int r = lo; r < hi; ++r) {
                const int n = p0 + r;
                double sum = 0.0;
                for (int kk = 0; kk < Kc; ++kk) {
                    const int k = k0 + kk;
                    if (cnt[k] > g.cap || cnt[g.K + k] > g.cap || !dir_qualifies(g, ep, cnt, k, rec)) continue;
                    double v[2];
                    for (int env = 0; env < 2; ++env) {
                        const size_t slot = (size_t)env * Kc + kk;
                        const int* wp = wpref + slot * (g.W + 1);
                        const int kb = ep.n > 0 ? wp[ep.w0[rec]] : 0;
                        const int wn = n >> 5;
                        const int before = wp[wn] + __popc(bits[slot * g.W + wn] & ((1u << (n & 31)) - 1u));
                        const int* kn = knots + slot * g.cap;
                        int i = max(before - 1, kb);
                        const int* mi = mir + (size_t)k * kMirWords;
                        const int E = cnt[env * g.K + k];
                        if constexpr (MIR) {
                            int lp0, lp1, rp0, rp1;
                            mirror_positions(mi, kn, env, E, lp0, lp1, rp0, rp1);
                            i = min(max(mirror_before(n, lp0, lp1, rp0, rp1) + before - 1, 0), E - 2);
                        }
                        const double* sp = sv + slot * (size_t)g.cap * C + c;
                        const double* ye = yend + (slot * (ep.n > 0 ? ep.n : 1) + rec) * 2 * (size_t)C + c;
                        const int xi = kn[i], xn = kn[i + 1];
                        const double y0 = MIR ? X[(size_t)mirror_source(mi, env, i, E, xi) * C + c]
                                                   : (xi == roff ? ye[0] : X[(size_t)xi * C + c]);
                        const double y1 = MIR ? X[(size_t)mirror_source(mi, env, i + 1, E, xn) * C + c]
                                                   : (xn == rlast ? ye[C] : X[(size_t)xn * C + c]);
                        const double s0 = sp[(size_t)i * C], s1 = sp[(size_t)(i + 1) * C];
                        const double t = (double)(n - xi);
                        const double h3 = __dmul_rn((double)(xn - xi), 1.0 / 3.0);
                        const double b = __fma_rn(-h3, __fma_rn(2.0, s0, s1), __dmul_rn(__dsub_rn(y1, y0), rtab[xn - xi]));
                        const double d = __dmul_rn(__dsub_rn(s1, s0), __dmul_rn(rtab[xn - xi], 1.0 / 3.0));
                        v[env] = __fma_rn(__fma_rn(__fma_rn(d, t, s0), t, b), t, y0);
                    }
                    sum = __dadd_rn(sum, __dadd_rn(v[0], v[1]));
                }
                emit(r, 0, sum, last_chunk ? X[(size_t)n * C + c] : 0.0);
            }
        }
    }
}

// Knots per record over all directions of a pass, added to tot[record] (runs
// of several direction passes, before the passes): one CTA per (slot, 4096
// words).
__global__ void __launch_bounds__(256)
k_count_knots(const uint32_t* __restrict__ bits, unsigned long long* __restrict__ tot, Geom g, Epochs ep)
{
    const uint32_t* b = bits + (size_t)blockIdx.y * g.W;
    const int w0 = blockIdx.x * 4096, w1 = min(g.W, w0 + 4096);
    unsigned long long n = 0ull;
    for (int w = w0 + (int)threadIdx.x; w < w1; w += blockDim.x) {
        const int p = __popc(b[w]);
        if (ep.n > 0) {
            if (p) atomicAdd(&tot[ep.wep[w]], (unsigned long long)p);
        } else {
            n += (unsigned long long)p;
        }
    }
    if (ep.n == 0) {
        n = warp_sum(n);
        if ((threadIdx.x & 31) == 0 && n) atomicAdd(&tot[0], n);
    }
}

inline size_t fix_smem_bytes(int G)
{
    return sizeof(unsigned long long) * 2 * (size_t)G * (kFixRows + 4 * kFixAnchors);
}

}  // namespace memd
