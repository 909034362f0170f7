// Device helpers shared by the level kernels: delays, cut searches, list
// readers, and the walk of one time segment.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <type_traits>
#include "gls_internal.h"

namespace gls {

__device__ __forceinline__ int check_delay(uint32_t pre, uint32_t cur)
{
    // CheckDelay, src/simulate.cpp:1178-1201
    if ((pre == kV0 && cur != kV0) || (cur == kV1 && pre != kV1)) return 1;
    if ((pre == kV1 && cur != kV1) || (cur == kV0 && pre != kV0)) return 2;
    if (pre == kVX && cur == kVZ) return 3;
    if (pre == kVZ && cur == kVX) return 4;
    return 0;
}

__device__ __forceinline__ uint32_t pick(uint32_t rise, uint32_t fall, int s)
{
    return s == 1 ? rise : s == 2 ? fall : s == 3 ? max(rise, fall) : min(rise, fall);
}

__device__ __forceinline__ uint32_t slot_val(uint32_t pack, int j) { return (pack >> (2 * j)) & 3u; }

// AddDelay, src/simulate.cpp:1012-1176, on delays pre-scaled by the time
// factor and truncated (truncation commutes with min/max on non-negative
// values, so selecting after truncation gives the same integer).
__device__ inline uint32_t select_delay(const ArcDev *__restrict__ arcs, int n_arcs, uint32_t chg, int so,
                                 uint32_t curp, uint32_t lastp, uint32_t defd)
{
    const int num_in = __popc(chg);
    if (num_in == 1) {
        int nrel = 0;
        ArcDev r0 = {0, 0, 0, 0};
        for (int a = 0; a < n_arcs; ++a) {
            ArcDev A = arcs[a];
            if (!((chg >> (A.info >> 2)) & 1u)) continue;
            if (nrel == 0) r0 = A;
            ++nrel;
        }
        if (nrel == 0) return defd;
        if (nrel == 1) return pick(r0.rise, r0.fall, so);
        const int j = r0.info >> 2;
        const int e = (check_delay(slot_val(lastp, j), slot_val(curp, j)) == 2) ? 1 : 0;
        for (int a = 0; a < n_arcs; ++a) {
            ArcDev A = arcs[a];
            if (!((chg >> (A.info >> 2)) & 1u)) continue;
            if ((int)(A.info & 3u) == e) return pick(A.rise, A.fall, so);
        }
        return defd;
    }
    uint32_t mn = kInf;
    bool any = false;
    for (int a = 0; a < n_arcs; ++a) {
        ArcDev A = arcs[a];
        const int j = A.info >> 2;
        if (!((chg >> j) & 1u)) continue;
        const int edge = A.info & 3u;
        if (edge != 2) {
            const int e = (check_delay(slot_val(lastp, j), slot_val(curp, j)) == 2) ? 1 : 0;
            if (e != edge) continue;
        }
        mn = min(mn, pick(A.rise, A.fall, so));
        any = true;
    }
    return any ? mn : defd;
}

static __device__ __noinline__ uint32_t select_delay_call(const ArcDev *__restrict__ arcs, int n_arcs, uint32_t chg, int so,
                                                          uint32_t curp, uint32_t lastp, uint32_t defd)
{
    return select_delay(arcs, n_arcs, chg, so, curp, lastp, defd);
}

// Delay of an active step of a regular gate output: the smallest delay the
// changed nets select for their own input edge and the output sense, or the
// default when none applies.  Equals AddDelay (src/simulate.cpp:1012-1176)
// whenever every input net has no arc, one both-edge arc, or one posedge and
// one negedge arc: then a single changed net selects exactly one arc (or
// none), and several changed nets take the minimum over their arcs.
template <int M>
__device__ __forceinline__ uint32_t regular_delay(const NetDelay *__restrict__ nd, uint32_t chg, uint32_t so1,
                                                  uint32_t curp, uint32_t lastp, uint32_t defd)
{
    uint32_t d = kInf;   // so1: the output sense minus one
    if (M > 1 && chg != 0u && (chg & (chg - 1u)) == 0u) {
        // one input net changed (most steps): one table entry, no loop
        const int j = __ffs(chg) - 1;
        const uint32_t neg = (kNegTab >> (slot_val(lastp, j) * 4 + slot_val(curp, j))) & 1u;
        d = __ldg(&nd[j].d[neg * 4 + so1]);
        return d == kInf ? defd : d;
    }
#pragma unroll
    for (int j = 0; j < M; ++j) {
        if ((chg >> j) & 1u) {
            const uint32_t neg = (kNegTab >> (slot_val(lastp, j) * 4 + slot_val(curp, j))) & 1u;
            d = min(d, __ldg(&nd[j].d[neg * 4 + so1]));
        }
    }
    return d == kInf ? defd : d;
}

__device__ __forceinline__ uint32_t lut_index(uint32_t curp, const DrvMeta &md)
{
    if (md.flags & kFlagIdent) return curp & ((1u << (2 * md.n_pins)) - 1u);
    uint32_t idx = 0;
    for (int p = 0; p < md.n_pins; ++p)
        idx |= slot_val(curp, (md.pin_slot >> (3 * p)) & 7u) << (2 * p);
    return idx;
}

// The windows a launch covers: one window passed by value (kernel
// parameter space, no indirection in the hot loops), or a device array.
template <bool kBatch> struct WinSet;
template <> struct WinSet<false> {
    static constexpr bool kIsBatch = false;
    WinDev w;
    __device__ __forceinline__ const WinDev &get(uint32_t) const { return w; }
    __device__ __forceinline__ uint32_t size() const { return 1; }
};
template <> struct WinSet<true> {
    static constexpr bool kIsBatch = true;
    const WinDev *wv;
    uint32_t n;
    __device__ __forceinline__ const WinDev &get(uint32_t k) const { return wv[k]; }
    __device__ __forceinline__ uint32_t size() const { return n; }
};

// First index of the change list x[0..n) with time >= key, searched from a
// guess: gallop away from the guess, then bisect.  Event lists of one gate
// share the clock, so a position scaled from another list is usually a few
// events off.  Compares whole words: time >= key <=> word >= key << 2.
template <class P>
__device__ __forceinline__ uint32_t search_from(P x, uint32_t n, uint32_t key, uint32_t g)
{
    using Wd = typename std::remove_cv<typename std::remove_reference<decltype(x[0])>::type>::type;
    if (n == 0) return 0;
    const Wd kw = (Wd)key << 2;
    if (g >= n) g = n - 1;
    int64_t lo, hi;
    if (x[g] < kw) {
        int64_t a = g, b;
        uint32_t step = 1;
        for (;;) {
            b = a + step;
            if (b >= (int64_t)n) { b = n; break; }
            if (x[b] >= kw) break;
            a = b;
            step <<= 1;
        }
        lo = a + 1; hi = b;
    } else {
        int64_t b = g, a;
        uint32_t step = 1;
        for (;;) {
            a = b - step;
            if (a < 0) { a = -1; break; }
            if (x[a] < kw) break;
            b = a;
            step <<= 1;
        }
        lo = a + 1; hi = b;
    }
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (x[mid] < kw) lo = mid + 1; else hi = mid;
    }
    return (uint32_t)lo;
}

// x * y / z for 32-bit operands, in 32-bit arithmetic when the product fits
__device__ __forceinline__ uint32_t mul_div(uint32_t x, uint32_t y, uint32_t z)
{
    if (__umulhi(x, y) == 0) return (x * y) / z;
    return (uint32_t)((uint64_t)x * y / z);
}

// output value for the input-net values `curp` (2 bits per net) from the
// slot truth table held in registers
template <int M>
__device__ __forceinline__ uint32_t slut_get(const uint4 &t, uint32_t curp)
{
    const uint32_t x = curp & ((1u << (2 * M)) - 1u);
    uint32_t wd = t.x;
    if (M == 3) wd = (x >> 4) == 0 ? t.x : ((x >> 4) == 1 ? t.y : ((x >> 4) == 2 ? t.z : t.w));
    return (wd >> (2 * (x & 15u))) & 3u;
}

// Time of the merged event of rank r (0-based) of two event lists X and Y
// (r < nx + ny), found by a merge-path search galloping from the guess g for
// the number of X events among the first r; on return ix / iy are the
// first events of X / Y at or after that time.  Equal times may sit in both
// lists (not within one), so a cut at the returned time keeps every time's
// events on one side.
template <class P>
__device__ __forceinline__ uint32_t rank_time2(P X, uint32_t nx, P Y, uint32_t ny, uint32_t r, uint32_t g,
                                               uint32_t &ix, uint32_t &iy)
{
    // short(i): the first r merged events hold more than i events of X
    // (true for small i, false from the answer on)
    auto short_x = [&](uint32_t i) { return i < nx && r - i > 0 && ev_time(Y[r - i - 1]) > ev_time(X[i]); };
    const uint32_t lo0 = r > ny ? r - ny : 0u, hi0 = min(r, nx);
    g = min(max(g, lo0), hi0);
    uint32_t lo, hi;   // the answer lies in [lo, hi]
    if (short_x(g)) {
        uint32_t a = g, step = 1;
        for (;;) {
            const uint32_t b = a + step;
            if (b >= hi0) { lo = a + 1; hi = hi0; break; }
            if (!short_x(b)) { lo = a + 1; hi = b; break; }
            a = b;
            step <<= 1;
        }
    } else {
        uint32_t b = g, step = 1;
        for (;;) {
            if (b - lo0 < step) { lo = lo0; hi = b; break; }
            const uint32_t a = b - step;
            if (short_x(a)) { lo = a + 1; hi = b; break; }
            b = a;
            step <<= 1;
        }
    }
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (short_x(mid)) lo = mid + 1; else hi = mid;
    }
    const uint32_t i = lo, j = r - lo;
    const uint32_t tx = i < nx ? ev_time(X[i]) : kInf, ty = j < ny ? ev_time(Y[j]) : kInf;
    const uint32_t T = min(tx, ty);
    ix = i - ((i > 0 && ev_time(X[i - 1]) == T) ? 1u : 0u);
    iy = j - ((j > 0 && ev_time(Y[j - 1]) == T) ? 1u : 0u);
    return T;
}

template <class P>
static __device__ __noinline__ uint32_t search_from_call(P x, uint32_t n, uint32_t key, uint32_t g)
{
    return search_from(x, n, key, g);
}
template <class P>
static __device__ __noinline__ uint32_t rank_time2_call(P X, uint32_t nx, P Y, uint32_t ny, uint32_t r, uint32_t g,
                                                        uint32_t &ix, uint32_t &iy)
{
    return rank_time2(X, nx, Y, ny, r, g, ix, iy);
}

// Cut sk of S (0 < sk < S) of a gate output's fan-in timeline: the time of
// the event of rank sk * (plen + slen) / S in the merge of its two longest
// input lists (piv, sec), so that those two (all of them for gates with two
// input nets) split into segments of equal size; with one input net the
// event of rank sk * plen / S of that list.  Returns that time; cut[j]
// receives list j's first event at or after it.  The cut time does not
// decrease with sk.  kCall: the searches are calls, not inlined (see k_gate).
template <int M, bool kCall = false, class Wd>
__device__ __forceinline__ uint32_t cut_at(const Wd *__restrict__ pool, const uint64_t (&off)[M],
                                       const uint32_t (&len)[M], int m, int piv, int sec, uint64_t poff, uint64_t soff,
                                       uint32_t plen, uint32_t slen, uint32_t sk, uint32_t S, uint32_t (&cut)[M])
{
    uint32_t ip, is = 0, T;
    if (sec >= 0) {
        const uint32_t r = mul_div(sk, plen + slen, S);
        const uint32_t g = mul_div(r, plen, plen + slen);
        T = kCall ? rank_time2_call(pool + poff, plen, pool + soff, slen, r, g, ip, is)
                  : rank_time2(pool + poff, plen, pool + soff, slen, r, g, ip, is);
    } else {
        ip = mul_div(sk, plen, S);
        T = ev_time(pool[poff + ip]);
    }
#pragma unroll
    for (int j = 0; j < M; ++j) {
        if (j < m) {
            if (j == piv) {
                cut[j] = ip;
            } else if (j == sec) {
                cut[j] = is;
            } else {
                const uint32_t g = mul_div(ip, len[j], plen);
                cut[j] = kCall ? search_from_call(pool + off[j], len[j], T, g) : search_from(pool + off[j], len[j], T, g);
            }
        }
    }
    return T;
}

// The time of cut sk alone (0 < sk < S), as cut_at computes it.
__device__ __forceinline__ uint32_t cut_time(const uint32_t *__restrict__ pool, int sec, uint64_t poff, uint64_t soff,
                                             uint32_t plen, uint32_t slen, uint32_t sk, uint32_t S)
{
    if (sec < 0) return ev_time(pool[poff + mul_div(sk, plen, S)]);
    uint32_t ip, is;
    const uint32_t r = mul_div(sk, plen + slen, S);
    return rank_time2(pool + poff, plen, pool + soff, slen, r, mul_div(r, plen, plen + slen), ip, is);
}

__device__ __forceinline__ int vclass(uint32_t v) { return v == kV0 ? 0 : (v == kV1 ? 1 : 2); }

// Window-relative clamped times in 32 bits.  Event times are at most
// kMaxTime, so max(t, t_begin) - t_begin never exceeds kMaxTime (or is 0
// when the window starts past every event): with the bounds capped at 2^31
// the clamp gives the same values as in 64 bits, and a relative time
// shifted left by 2 still fits 32 bits next to a 2-bit value class.
// With 64-bit words (times up to 2^32 - 2) the same runs in 64 bits: the
// bounds are capped at 2^32 and a relative time needs 33 bits.
template <class P> struct RelClampT;
template <> struct RelClampT<uint32_t> {
    uint32_t lo, hi;
    __device__ __forceinline__ RelClampT(unsigned long long b, unsigned long long e)
        : lo((uint32_t)min(b, 1ull << 31)), hi((uint32_t)min(e, 1ull << 31)) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t t) const { return min(max(t, lo), hi) - lo; }
};
template <> struct RelClampT<unsigned long long> {
    unsigned long long lo, hi;
    __device__ __forceinline__ RelClampT(unsigned long long b, unsigned long long e)
        : lo(min(b, 1ull << 32)), hi(min(e, 1ull << 32)) {}
    __device__ __forceinline__ unsigned long long operator()(uint32_t t) const
    {
        const unsigned long long x = t;
        return min(max(x, lo), hi) - lo;
    }
};
// the packed (relative time << 2 | value class) and the sums of a window's word type
template <class Wd> using SaifP = typename std::conditional<std::is_same<Wd, uint32_t>::value, uint32_t,
                                                            unsigned long long>::type;

// Reader of one change list a word at a time: the head and the event after
// it in registers, kInfW behind the list's end.  Moving on is branch-free, so
// that lanes whose lists move at different steps stay together.  (More
// events held ahead measured no faster: moving a register waits for the load
// that fills it.)
template <class Wd> struct ListReader;
template <>
struct ListReader<uint32_t> {
    uint32_t h, n;
    const uint32_t *q;   // the event after n
    uint32_t qe;         // low word of the list's end (a list is shorter than 2^30 events)

    static __device__ __forceinline__ uint32_t ld_if(const uint32_t *q, bool go)
    {
        uint32_t v;
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u32 %0, 0xFFFFFFFF;\n\t@p ld.global.u32 %0, [%1];\n\t}"
            : "=r"(v) : "l"(q), "r"((uint32_t)go));
        return v;
    }
    __device__ __forceinline__ void start(const uint32_t *x, uint32_t b, uint32_t len)
    {
        h = ld_if(x + b, b < len);
        n = ld_if(x + b + 1, b + 1 < len);
        q = x + min(b + 2, len);
        qe = (uint32_t)(uintptr_t)(x + len);
    }
    __device__ __forceinline__ void advance(bool go)
    {
        const bool more = go && (uint32_t)(uintptr_t)q != qe;
        h = go ? n : h;
        asm("{\n\t.reg .pred p, r;\n\tsetp.ne.u32 p, %2, 0;\n\tsetp.ne.u32 r, %3, 0;\n\t@p mov.u32 %0, 0xFFFFFFFF;\n\t"
            "@r ld.global.u32 %0, [%1];\n\t}"
            : "+r"(n) : "l"(q), "r"((uint32_t)go), "r"((uint32_t)more));
        q += more ? 1 : 0;
    }
};
template <>
struct ListReader<WideWord> {   // a list of up to 2^32 events: its end is a whole address
    WideWord h, n;
    const WideWord *q, *qe;

    static __device__ __forceinline__ WideWord ld_if(const WideWord *q, bool go)
    {
        WideWord v;
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u64 %0, -1;\n\t@p ld.global.u64 %0, [%1];\n\t}"
            : "=l"(v) : "l"(q), "r"((uint32_t)go));
        return v;
    }
    __device__ __forceinline__ void start(const WideWord *x, uint32_t b, uint32_t len)
    {
        h = ld_if(x + b, b < len);
        n = ld_if(x + b + 1, (uint64_t)b + 1 < len);
        q = x + min((uint64_t)b + 2, (uint64_t)len);
        qe = x + len;
    }
    __device__ __forceinline__ void advance(bool go)
    {
        const bool more = go && q != qe;
        h = go ? n : h;
        asm("{\n\t.reg .pred p, r;\n\tsetp.ne.u32 p, %2, 0;\n\tsetp.ne.u32 r, %3, 0;\n\t@p mov.u64 %0, -1;\n\t"
            "@r ld.global.u64 %0, [%1];\n\t}"
            : "+l"(n) : "l"(q), "r"((uint32_t)go), "r"((uint32_t)more));
        q += more ? 1 : 0;
    }
};

// The walk of one time segment of a gate output: from the
// segment's first event of every list (in rd, with the values before them in
// curp; before: some list has one) to its end time tnext (kInf: the lists' end),
// onto the stack ot.  tmax: no event of the segment is later.  Steps whose
// input values are all 0 or 1 before and after (nearly all of them: X and Z
// leave a net with its first real event) take the fast step; any other step,
// and every step of a gate output whose FastRec is not usable, takes the
// general one.
//
// What bounds it: instruction issue.  A lane walks its own segment, so a
// warp issues both the step and, on nearly every iteration, the output
// change of some lane.  The fast step therefore keeps everything in
// registers and is branch-free but for the rare pops: the truth table is one
// word shifted by the input state, the delays of all input nets are packed
// (rise, fall) pairs whose 16-bit minimum is one instruction, the end of the
// segment is a time (so no list needs an end position beyond its own end),
// the entry below the stack top is kept so that an inertial pop rarely reads
// the stack back, and the range check of output times is made once per
// segment (a delay is below 2^16).  What the fast step gave, in the kernels
// with a thread per segment of a level (k_sim, which walks by it without a
// step table, against sim_segment with inner branches and delay-table loads):
// the 3-input kernel of the 100,000-cell, 6-level large-configuration case 460
// -> 301 us and 350 -> 183 M warp instructions at 14 -> 25 active lanes, the
// 2-input one 320 -> 277 us and 205 -> 119 M.  With the step table, in k_gate,
// that case takes 4.2 warp instructions a fan-in event in all, at 28 lanes.
//
// kTab: `tab` is the shared address of the gate output's step table (see
// step_entry; aligned to its size).  clean: from the segment's start on, all
// input values are known and the lists hold nothing but alternating 0 and 1;
// then a step is one table read by the input state and the set of lists that
// move, a third fewer instructions than the fast step, which reads values,
// edges and delays for every list.
template <class Wd>
struct WalkOut {
    uint32_t cnt;    // entries on the stack
    Wd minw;         // word of the smallest candidate time (kInfW: no candidate)
    Wd top;          // the stack's top entry (cnt > 0)
    uint32_t xt;     // latest time an X or Z was pushed at (0: none but the first entry)
};

// Step table of a gate output with a usable FastRec: entry state << M | moves
// (a bit per input net) holds delay << 2 | value of the output change, kInf
// where the output stays.
template <int M>
__device__ __forceinline__ uint32_t step_entry(const uint4 &f0, const uint4 &f1, uint32_t e)
{
    const uint32_t dp[3] = {f0.x, f0.z, f1.x}, dn[3] = {f0.y, f0.w, f1.y};
    const uint32_t mv = e & ((1u << M) - 1u), from = e >> M, to = from ^ mv;
    auto out = [&](uint32_t x) { return (f1.z >> ((x & 1u) | (x & 2u) << 1 | (x & 4u) << 2)) & 1u; };
    const uint32_t F = out(to);
    if (mv == 0 || F == out(from)) return kInf;
    uint32_t d = kInf;
#pragma unroll
    for (int j = 0; j < M; ++j)
        if ((mv >> j) & 1u) {
            const uint32_t r = ((to >> j) & 1u) ? dp[j] : dn[j];
            d = min(d, F ? r & 0xFFFFu : r >> 16);
        }
    return d << 2 | (F ? kV1 : kV0);
}

// What a gate output's walks read from shared memory (tab: its address, a
// multiple of 256: rows of the step table are found by ORing).
struct GateTab {
    uint32_t step[64];   // the step table
    uint32_t slut[4];    // the truth table (LevelArgs::slut)
    uint32_t nd[24];     // its input nets' NetDelay entries (regular gate outputs)
};
__device__ __forceinline__ uint32_t lds32(uint32_t at)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}

// kSm: the general step reads the gate output's tables from shared memory too;
// kCall: delays of irregular arcs by a call.
template <int M, bool kTab, bool kSm, bool kCall, class Wd>
__device__ __forceinline__ WalkOut<Wd> walk_segment(const WinDev &w, const LevelArgs &a, uint32_t drv, uint32_t s,
                                                ListReader<Wd> (&rd)[M], uint32_t curp, bool before, uint32_t tnext,
                                                uint32_t tmax, Wd *ot, uint32_t tab = 0, bool clean = false)
{
    static_assert(!(kTab || kSm) || M <= 3, "the tables are for up to three input nets");
    constexpr bool kFast = M <= 3;
    constexpr Wd kEnd = EvW<Wd>::kInfW;
    constexpr uint32_t kSlut = offsetof(GateTab, slut), kNd = offsetof(GateTab, nd);
    const DrvMeta *__restrict__ mdp = a.meta + drv;
    // words at or above tend lie behind the segment
    const Wd tend = tnext != kInf ? (Wd)tnext << 2 : kEnd;
    uint4 f0 = {0, 0, 0, 0}, f1 = {0, 0, 0, 0};
    if (kFast) {
        f0 = __ldg(a.fast + 2ull * drv);
        f1 = __ldg(a.fast + 2ull * drv + 1);
    }
    const uint32_t dp[3] = {f0.x, f0.z, f1.x}, dn[3] = {f0.y, f0.w, f1.y};
    const uint32_t tt = f1.z;
    constexpr uint32_t kBits = 0x555u & ((1u << (2 * M)) - 1u);
    // a gate output without a usable FastRec, or times too close to the
    // largest one, take the general step throughout
    const uint32_t never = (kFast && f1.w != 0u && tmax <= EvW<Wd>::kMax - 0x10000u) ? 0u : kBits;
    // input values are 2 bits per net; 0x15 bits of `mixed` mark nets at X or Z
    uint32_t mixed = ((curp ^ (curp >> 1)) & kBits) | never;
    // Every step consumes an event and pushes at most one entry, so a
    // segment's stack ends within the gate output's scratch.
    uint32_t cnt = 0;
    // top of the stack and the entry below it (kEnd: not at hand).  With no
    // entry left the top reads as (0, X): below every later candidate, and
    // different from 0 and 1.
    Wd top = EvW<Wd>::word(0, kVX), below = kEnd;
    if (s == 0) { ot[0] = top; cnt = 1; }
    uint32_t fprev = kVX;
    auto out_of = [&](uint32_t x) -> uint32_t {   // the general step's truth table
        if constexpr (kSm) return (lds32(tab + kSlut + (M == 3 ? (x >> 4) * 4 : 0u)) >> (2 * (x & 15u))) & 3u;
        else if constexpr (kFast) return slut_get<M>(__ldg(a.slut + drv), x);
        else return __ldg(a.lut + mdp->lut_off + lut_index(x, *mdp));
    };
    if (before) fprev = out_of(curp);
    const bool regular = mdp->flags & kFlagRegular;
    Wd minw = kEnd;
    uint32_t xt = 0;
    for (;;) {
        Wd mk = rd[0].h | 3u;
#pragma unroll
        for (int j = 1; j < M; ++j) mk = min(mk, (Wd)(rd[j].h | 3u));
        if (mk >= tend || (kTab && clean)) break;
        const uint32_t lastp = curp;
        bool ch[M];
#pragma unroll
        for (int j = 0; j < M; ++j) {
            ch[j] = (rd[j].h | 3u) == mk;
            const uint32_t cj = (curp & ~(3u << (2 * j))) | (((uint32_t)rd[j].h << (2 * j)) & (3u << (2 * j)));
            curp = ch[j] ? cj : curp;
            rd[j].advance(ch[j]);
        }
        const uint32_t mixed0 = mixed;
        mixed = ((curp ^ (curp >> 1)) & kBits) | never;
        if (kFast && (mixed | mixed0) == 0u) {
            const uint32_t F = ((tt >> (curp & kBits)) & 1u) ? kV1 : kV0;
            const bool chg = F != fprev;
            fprev = F;
            const uint32_t fall = lastp & ~curp;
            uint32_t r[3] = {kInf, kInf, kInf};
#pragma unroll
            for (int j = 0; j < (M < 3 ? M : 3); ++j) r[j] = ch[j] ? ((fall & (1u << (2 * j))) ? dn[j] : dp[j]) : kInf;
            const uint32_t d2 = M == 1 ? r[0] : (M == 2 ? __vminu2(r[0], r[1]) : __vimin3_u16x2(r[0], r[1], r[2]));
            const uint32_t d = F ? (d2 & 0xFFFFu) : (d2 >> 16);
            const Wd lo = (mk ^ 3u) + (d << 2);
            minw = chg ? min(minw, lo) : minw;
            // inertial update, src/simulate.cpp:991-1009.  Both states of a
            // fast step are known, so it is not the first: lo > 0, and the
            // bottom (0, X) is never popped.
            if (chg && top >= lo) {
                do {
                    --cnt;
                    if (below != kEnd) top = below;
                    else top = cnt > 0 ? ot[cnt - 1] : EvW<Wd>::word(0, kVX);
                    below = kEnd;
                } while (top >= lo);
            }
            const bool push = chg && (((uint32_t)top ^ F) & 3u) != 0u;
            if (push) ot[cnt] = lo | F;
            below = push ? top : below;
            top = push ? lo | F : top;
            cnt += push ? 1u : 0u;
            continue;
        }
        // general step
        const uint32_t F = out_of(curp);
        if (F == fprev) continue;
        const uint32_t so1 = (kSense1Tab >> (2 * (fprev * 4 + F))) & 3u;
        fprev = F;
        uint32_t d;
        if (regular && kSm) {   // as regular_delay
            d = kInf;
#pragma unroll
            for (int j = 0; j < M; ++j) {
                const uint32_t neg = (kNegTab >> (slot_val(lastp, j) * 4 + slot_val(curp, j))) & 1u;
                if (ch[j]) d = min(d, lds32(tab + kNd + (j * 8 + neg * 4 + so1) * 4));
            }
            d = d == kInf ? a.def_delay : d;
        } else {
            uint32_t chg = 0;
#pragma unroll
            for (int j = 0; j < M; ++j) chg |= ch[j] ? 1u << j : 0u;
            d = regular ? regular_delay<M>(a.ndel + mdp->dt_off, chg, so1, curp, lastp, a.def_delay)
                : kCall ? select_delay_call(a.arcs + mdp->arc_off, mdp->n_arcs, chg, (int)so1 + 1, curp, lastp, a.def_delay)
                        : select_delay(a.arcs + mdp->arc_off, mdp->n_arcs, chg, (int)so1 + 1, curp, lastp, a.def_delay);
        }
        const uint64_t o64 = (uint64_t)ev_time(mk) + d;
        if (o64 > EvW<Wd>::kMax) { atomicOr(w.err, kErrTime); break; }
        const Wd lo = (Wd)o64 << 2;
        minw = min(minw, lo);
        int popped_v = -1;
        while (cnt > 0 && top >= lo) {
            if (s == 0 && cnt == 1) { popped_v = (int)ev_val(top); cnt = 0; break; }
            --cnt;
            top = cnt > 0 ? ot[cnt - 1] : EvW<Wd>::word(0, kVX);
            below = kEnd;
        }
        const int prevv = cnt > 0 ? (int)ev_val(top) : popped_v;
        if (prevv != (int)F) {
            below = kEnd;
            top = lo | F;
            ot[cnt++] = top;
            if (F == kVX || F == kVZ) xt = (uint32_t)(lo >> 2);
        } else if (cnt == 0) {
            atomicOr(w.err, kErrEmptied);
            break;
        }
    }
    if constexpr (kTab) {
        if (!clean) return {cnt, minw, top, xt};
        uint32_t so = tab;   // the table row of the input state
#pragma unroll
        for (int j = 0; j < M; ++j) so += ((curp >> (2 * j)) & 1u) << (2 + M + j);
        for (;;) {
            Wd mk = rd[0].h | 3u;
#pragma unroll
            for (int j = 1; j < M; ++j) mk = min(mk, (Wd)(rd[j].h | 3u));
            if (mk >= tend) break;
            uint32_t x = so;
#pragma unroll
            for (int j = 0; j < M; ++j) {
                const bool ch = (rd[j].h | 3u) == mk;
                x |= ch ? 4u << j : 0u;
                rd[j].advance(ch);
            }
            const uint32_t st = lds32(x);
            so ^= (x ^ so) << M;
            const bool chg = st != kInf;
            const Wd nw = mk - 3u + st;   // the candidate's event word
            minw = chg ? min(minw, nw) : minw;
            if (chg && (top | 3u) >= nw) {   // times only: the bottom lies below every candidate
                do {
                    --cnt;
                    if (below != kEnd) top = below;
                    else top = cnt > 0 ? ot[cnt - 1] : EvW<Wd>::word(0, kVX);
                    below = kEnd;
                } while ((top | 3u) >= nw);
            }
            const bool put = chg && (((uint32_t)top ^ (uint32_t)nw) & 3u) != 0u;
            if (put) ot[cnt] = nw;
            below = put ? top : below;
            top = put ? nw : top;
            cnt += put ? 1u : 0u;
        }
    }
    return {cnt, minw, top, xt};
}

}  // namespace gls
