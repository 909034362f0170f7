// k_gate: one level of gate outputs in one launch.
//
// A block takes one gate output at a time: it cuts its fan-in timeline into
// one time segment per thread, walks them, links the segments' stacks, places
// the list in the event pool, copies it there and takes its SAIF integral.
// Nothing but the finished list leaves the block, so a level needs no plan,
// no segment tables and no launches in between.
//
// What bounds it: on wide levels issue (59 % of the cycles, the integer pipe
// 60 %) by 32 warps an SM of 64 registers a thread, a quarter of whose time
// goes into waiting for the slowest warp of the block; on narrow levels the
// chain of dependent steps of one gate output (its record, its lists' places,
// the cut search, the walk: 646 gate outputs of 1,600 events, little more than
// a round of blocks, 25 us at 50 % issue).  Against plan, three classes of simulate, link
// and copy kernels with one thread per segment of a level-wide segment list
// (device ms): 2,000 cells over 1,000 cycles .95 -> .23; 37,501 cells, 3,333
// cycles 3.97 -> 1.43; 200,000 cells, 10,000 cycles 20.1 -> 12.7; 2 M cells,
// 5,000 cycles 95.8 -> 66.8.  The segment search is made once per segment
// instead of at both ends, the lanes of a warp walk the same gate output, and
// link and copy find the stacks in L1 and L2.
//
// The stack contract of a segment and why the split is exact: see the head of
// gls_kernels.cu.
#include <cuda_runtime.h>
#include <cstdint>
#include "gls_device.cuh"

namespace gls {

namespace {

// Threads per SM the kernels are compiled for, in blocks of any size up to
// that.  kSix: the class of four to six input nets, which walks by general
// steps in more registers (12 levels of 3,000 such gate outputs of 140,000
// events, in blocks of 256: 256 / 512 / 768 / 1,024 threads 113 / 71 / 59 / 63
// ms, the last with spills).  How many threads a block has: see gate_block in
// gls_capi.cpp.
template <bool kSix, class Wd> __host__ __device__ constexpr uint32_t gate_resident()
{
    return kSix ? (sizeof(Wd) == 4 ? 768u : 512u) : (sizeof(Wd) == 4 ? 1024u : 768u);
}

// Shared memory is L1 lost: each kernel has only what it uses, the step table
// (kTab) and the window's descriptor (kBatch), and behind the segments' words
// what meets between the warps there are (WarpParts).  With 512 bytes (432 now)
// before the segments' a 1,024-thread SM gets by with 16 KB (one step of the
// split more: 2 M cells 68.7 instead of 68.3 ms, 200,000 cells 13.1 instead of
// 12.9); one-warp blocks with 272 bytes instead of 1,280: 8 windows of 200,000
// cells 19.8 -> 19.5, 48 of 2,000 cells .89 -> .87.
template <bool kTab> struct TabSmem { GateTab tab; };   // the gate output's tables
template <> struct TabSmem<false> {};
template <class Wd> struct WarpParts {   // an entry per warp, at the end of the dynamic shared memory
    Wd *a;              // smallest candidate of its segments; at the end its part of T0
    Wd *b;              // kept entries; at the end its part of T1
    uint8_t *last;      // value of its last kept entry (4: none)
    __device__ __forceinline__ WarpParts(void *at, uint32_t nw)
        : a(static_cast<Wd *>(at)), b(a + nw), last(reinterpret_cast<uint8_t *>(b + nw)) {}
    static constexpr uint32_t kBytes = 2 * sizeof(Wd) + 1;   // per warp
};
template <bool kBatch> struct WindowSmem {
    WinDev win;                  // wave of windows: the descriptor of the block's current window
    uint32_t cw;                 // its number
};
template <> struct WindowSmem<false> {};
template <bool kBatch, bool kTab>
struct GateSmem : TabSmem<kTab>, WindowSmem<kBatch> {
    unsigned long long ctr[4];   // gate events, output events, segments, fan-in events of the window at hand
    unsigned long long scr, dst; // the gate output's stacks in the scratch, its list in the pool
    uint32_t q;                  // the block's gate output, kInf: none left
    uint32_t skip;               // its window has failed
    uint32_t ok;                 // the list has its place
    uint32_t xt;                 // latest X or Z of the list but its first entry
};

// kWarp: blocks of one warp
template <bool kWarp> __device__ __forceinline__ void sync_block()
{
    if (kWarp) __syncwarp();
    else __syncthreads();
}

// The thread's part of a gate output after the walk.
template <class Wd>
struct Walked {
    WalkOut<Wd> o;
    uint32_t region;         // its stack among the gate output's
    uint32_t S;              // segments of the gate output
    unsigned long long E;    // fan-in events of the gate output
};

// Cut and walk gate output i of the level.
template <int M, bool kTab, class Wd, class Smem>
__device__ __forceinline__ Walked<Wd> walk_gate(const WinDev &w, const LevelArgs &a, uint32_t i, Smem &sm,
                                            uint32_t *s_seg)
{
    constexpr bool kWarp = !kTab && M <= 3;
    const uint32_t tid = threadIdx.x, nthr = kWarp ? 32u : blockDim.x;
    const uint32_t drv = a.lo + i;
    const Wd *const pool = reinterpret_cast<const Wd *>(w.pool);
    const DrvMeta *__restrict__ mdp = a.meta + drv;
    constexpr bool kSm = kTab;
    uint4 f0 = {0, 0, 0, 0}, f1 = {0, 0, 0, 0};
    if (kTab) {
        f0 = __ldg(a.fast + 2ull * drv);
        f1 = __ldg(a.fast + 2ull * drv + 1);
    }
    const int m = mdp->m;
    uint64_t off[M], poff = 0, soff = 0;
    uint32_t len[M], plen = 0, slen = 0;
    unsigned long long E = 0;
    uint32_t lmin = kInf;
    uint32_t xmax = 0;   // the latest X, Z or repeated value of the input lists
    int piv = 0, sec = -1;   // the longest input list and the longest of the others
#pragma unroll
    for (int j = 0; j < M; ++j) {
        len[j] = 0; off[j] = 0;
        if (j < m) {
            const uint32_t net = mdp->net[j];
            off[j] = w.net_off[net];
            len[j] = w.net_len[net];
            E += len[j];
            lmin = min(lmin, len[j]);
            if (kTab && a.x_times) xmax = max(xmax, w.net_len[a.n_nets + net]);
            if (len[j] > plen) { sec = piv; slen = plen; plen = len[j]; piv = j; }
            else if (sec < 0 || len[j] > slen) { sec = j; slen = len[j]; }
        }
    }
    if (m < 2) sec = -1;
#pragma unroll
    for (int j = 0; j < M; ++j) {
        if (j == piv) poff = off[j];
        if (j == sec) soff = off[j];
    }
    // one segment per thread, none shorter than the smallest worth a search
    unsigned long long seg = a.seg_events ? max(a.seg_events, 8u) : kGateMinSeg;
    seg = max(seg, (E + nthr - 1) / nthr);
    const uint32_t S = (uint32_t)max(1ull, (E + seg - 1) / seg);
    const unsigned long long scr_need = (E + S + 3) & ~3ull;
    unsigned long long scr_at = 0;   // thread 0; used once the cuts are found
    if (tid == 0) scr_at = atomicAdd(&w.lvl[a.level].scr, scr_need);
    const bool usable = kTab && a.x_times && f1.w != 0u;   // the step table is
    uint32_t tabw = 0;   // a word of the tables, stored once the cuts are found
    const uint32_t tk = nthr - 1 - tid;
    if constexpr (kSm) {
        if (tk < 4) tabw = __ldg(reinterpret_cast<const uint32_t *>(a.slut + drv) + tk);
        else if (tk - 4 < 8 * (uint32_t)m && (mdp->flags & kFlagRegular)) tabw = __ldg(a.ndel[mdp->dt_off].d + (tk - 4));
    }
    // the segment's start; its end is the next thread's start.  With a step
    // table the first warp's segments, which walk without it, are cut to half
    // the others' length.
    const bool mine = tid < S;
    const bool half = usable && S > 64 && lmin > 1;
    const uint32_t sk = half && tid > 32 ? 2 * tid - 32 : tid, sn = half ? 2 * S - 32 : S;
    uint32_t cb[M], tcut = 0;
#pragma unroll
    for (int j = 0; j < M; ++j) cb[j] = 0;
    if (mine && tid > 0)
        tcut = cut_at<M, !kTab>(pool, off, len, m, piv, sec, poff, soff, plen, slen, sk, sn, cb);
    if (mine) s_seg[tid] = tcut;
    if constexpr (kTab) {
        if (usable)
            for (uint32_t e = tid; e < 1u << (2 * M); e += nthr) sm.tab.step[e] = step_entry<M>(f0, f1, e);
    }
    if constexpr (kSm) {
        if (tk < 28) (&sm.tab.slut[0])[tk] = tabw;   // slut, then nd
    }
    if (tid == 0) {
        sm.xt = 0;
        sm.scr = scr_at;
        sm.ok = scr_at + scr_need <= w.scr_cap;
        if (!sm.ok) atomicOr(w.err, kErrScratch);
    }
    sync_block<kWarp>();
    Wd *const scr = reinterpret_cast<Wd *>(w.scratch) + sm.scr;
    uint32_t region = tid;
    WalkOut<Wd> o = {0, EvW<Wd>::kInfW, 0, 0};
    if (mine && sm.ok) {
        uint32_t curp = 0x555u & ((1u << (2 * M)) - 1u), tmax = 0;
        bool before = false;
        ListReader<Wd> rd[M];
#pragma unroll
        for (int j = 0; j < M; ++j) {
            const Wd *x = pool + off[j];
            region += cb[j];
            if (cb[j] > 0) {
                curp = (curp & ~(3u << (2 * j))) | (ev_val(x[cb[j] - 1]) << (2 * j));
                before = true;
            }
            rd[j].start(x, cb[j], len[j]);
        }
        const uint32_t tnext = tid + 1 < S ? s_seg[tid + 1] : kInf;
        if (tnext != kInf) {
            tmax = tnext;
        } else {
#pragma unroll
            for (int j = 0; j < M; ++j)
                if (len[j]) tmax = max(tmax, ev_time(pool[off[j] + len[j] - 1]));
        }
        // the step table serves a warp whose segments all start in known
        // values, behind every X, Z and repeat: lanes of both kinds would
        // walk one kind after the other
        bool clean = false;
        if constexpr (kTab) {
            clean = usable && tmax <= EvW<Wd>::kMax - 0x10000u && tcut > xmax && ((curp ^ (curp >> 1)) & 0x15u) == 0u;
            clean = __all_sync(__activemask(), clean);
        }
        uint32_t tab = 0;
        if constexpr (kSm) tab = (uint32_t)__cvta_generic_to_shared(&sm.tab);
        o = walk_segment<M, kTab, kSm, !kTab>(w, a, drv, tid, rd, curp, before, tnext, tmax, scr + region, tab, clean);
        if (o.xt) atomicMax(&sm.xt, o.xt);
    }
    return {o, region, S, E};
}

// Link the walked segments' stacks, place the gate output's list and copy it.
// fetch: thread 0 sets sm.q and sm.skip to the block's next gate output; called
// where the wait for it overlaps others and every thread has read the present
// one.
template <bool kWarp, class Wd, class Smem, class Fetch>
__device__ __forceinline__ void finish_gate(const WinDev &w, const LevelArgs &a, uint32_t i, Smem &sm,
                                            uint32_t *s_seg, const Walked<Wd> &wk, Fetch fetch)
{
    const unsigned FULL = 0xffffffffu;
    const uint32_t tid = threadIdx.x, nthr = kWarp ? 32u : blockDim.x;
    const uint32_t lane = tid & 31u, wid = kWarp ? 0u : tid >> 5, nw = nthr >> 5;
    const DrvMeta *__restrict__ mdp = a.meta + a.lo + i;
    const WalkOut<Wd> &o = wk.o;
    const uint32_t region = wk.region, S = wk.S;
    const unsigned long long E = wk.E;
    const bool mine = tid < S;
    const WarpParts<Wd> wp(s_seg + nthr, nw);
    if (!sm.ok) {   // no room for its stacks; the same for the whole block
        sync_block<kWarp>();
        if (tid == 0) fetch();
        return;
    }
    Wd *const scr = reinterpret_cast<Wd *>(w.scratch) + sm.scr;
    const Wd *ot = scr + region;
    const Wd bottom = o.cnt ? ot[0] : Wd(0);   // on its way while the minima meet
    // later segments cut this one's stack at their smallest candidate
    Wd x = o.minw;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const Wd y = __shfl_down_sync(FULL, x, k);
        if (lane + k < 32) x = min(x, y);
    }
    Wd later = __shfl_down_sync(FULL, x, 1);
    if (lane == 31) later = EvW<Wd>::kInfW;
    if constexpr (!kWarp) {
        if (lane == 0) wp.a[wid] = x;
        __syncthreads();
        for (uint32_t k = wid + 1; k < nw; ++k) later = min(later, wp.a[k]);
    }
    uint32_t keep = o.cnt, firstv = 0, lastv = 0;
    if (keep && later != EvW<Wd>::kInfW)
        while (keep && ((keep == o.cnt ? o.top : ot[keep - 1]) | 3u) >= later) --keep;
    if (keep) {
        firstv = ev_val(bottom);
        lastv = ev_val(keep == o.cnt ? o.top : ot[keep - 1]);
    }
    // an entry at a segment's bottom that repeats the last kept value before it goes
    const unsigned bal = __ballot_sync(FULL, keep > 0);
    const unsigned prior = bal & ((1u << lane) - 1u);
    uint32_t vprev = __shfl_sync(FULL, lastv, prior ? 31 - __clz(prior) : 0);
    const uint32_t vtop = __shfl_sync(FULL, lastv, bal ? 31 - __clz(bal) : 0);
    if (!prior) vprev = kVX;
    if constexpr (!kWarp) {
        if (lane == 0) wp.last[wid] = bal ? vtop : 4u;
        __syncthreads();
        if (!prior)
            for (int k = (int)wid - 1; k >= 0; --k)
                if (wp.last[k] < 4u) { vprev = wp.last[k]; break; }
    }
    const uint32_t drop = (tid > 0 && keep > 0 && firstv == vprev) ? 1u : 0u;
    const uint32_t fin = keep - drop;
    uint32_t inc = fin;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, k);
        if (lane >= k) inc += y;
    }
    uint32_t pos = inc - fin, total = 0;
    if constexpr (kWarp) {
        total = __shfl_sync(FULL, inc, 31);
    } else {
        if (lane == 31) wp.b[wid] = inc;
        __syncthreads();
        for (uint32_t k = 0; k < nw; ++k) {
            const uint32_t n = (uint32_t)wp.b[k];
            if (k < wid) pos += n;
            total += n;
        }
    }
    // per warp, the segments that keep entries: where in the stacks the list's
    // entry 0 would be
    const unsigned some = __ballot_sync(FULL, fin > 0);
    uint32_t *const delta = s_seg + (tid & ~31u);
    __syncwarp();   // the cut times that were here have been read
    if (fin) delta[__popc(some & ((1u << lane) - 1u))] = region + drop - pos;
    if (tid == 0) {
        // the list's place: reserved up front for its bound or its predicted
        // length, or (exact placement, or a list longer than predicted) as long as it is
        unsigned long long need = (total + 3ull) & ~3ull;
        if (a.alloc_mode == kAllocBound) need = (E + 1 + 3) & ~3ull;
        else if (a.alloc_mode == kAllocLearned) {
            const unsigned long long res = min((E + 1 + 3) & ~3ull, ((unsigned long long)w.pred[i] + 3) & ~3ull);
            if (total > res) {
                atomicAdd(w.n_over, 1ull);
                atomicAdd(w.top, res);   // the slot it outgrew
            } else {
                need = res;
            }
        }
        const unsigned long long st = atomicAdd(w.top, need);
        fetch();
        sm.dst = st;
        sm.ok = st + need <= w.cap;
        if (!sm.ok) atomicOr(w.err, kErrPool);
        else {
            w.net_off[mdp->out_net] = st;
            w.net_len[mdp->out_net] = total;
            w.net_len[a.n_nets + mdp->out_net] = sm.xt;
        }
        sm.ctr[1] += total;
        sm.ctr[2] += S;
        sm.ctr[3] += E;
        if (mdp->flags & kFlagFirstOut) {   // first output of its instance: count fan-in per pin
            if (mdp->flags & kFlagIdent) sm.ctr[0] += E;
            else
                for (int p = 0; p < mdp->n_pins; ++p) sm.ctr[0] += w.net_len[mdp->net[(mdp->pin_slot >> (3 * p)) & 7u]];
        }
    }
    sync_block<kWarp>();
    if (!sm.ok) return;
    // Copy, with the SAIF integral: an entry at time t ends the hold of the
    // value before it and starts its own, so class c's time is the sum of t
    // over the entries after a value of class c minus the sum over those of
    // class c, plus t_end for the last value's class.  Times are
    // window-relative and below 2^30: the sums wrap in 32 bits and are read
    // back as signed.  A warp's segments make a contiguous part of the list:
    // it copies 32 entries at a time, and finds each one's segment by counting
    // the segments that start up to there.  The stacks come from L2, so U
    // times 32 entries are loaded before the first is stored.  Against eight
    // lanes a segment, four entries each at a time, device ms: 2 M cells 73.8
    // -> 69.6 (U = 1 / 2 / 4 / 6 / 8: 78.7 / 73.4 / 71.1 / 69.5 / 69.7),
    // 200,000 cells 13.7 -> 12.7 (15.1 / 13.8 / 13.1 / 12.8 / 12.7), waves of
    // 200,000 cells, whose warps hold some 300 entries, 23.3 -> 20.8 (- / 20.9
    // / 21.7 / - / -).
    constexpr uint32_t U = kWarp ? 2 : 8;
    using P = SaifP<Wd>;
    const RelClampT<P> rc(w.t_begin, w.t_end);
    P s0 = 0, s1 = 0;
    Wd *const dst = reinterpret_cast<Wd *>(w.pool) + sm.dst;
    const uint32_t end = __shfl_sync(FULL, pos + fin, 31);
    const uint32_t upto = 0xFFFFFFFFu >> (31 - lane);   // this lane and the ones below
    uint32_t first = 0u - 1u;                           // segments that start before the 32 entries, less one
    uint32_t before1 = __shfl_sync(FULL, vprev, 0);     // the value before them
    for (uint32_t c = __shfl_sync(FULL, pos, 0); c < end; c += 32 * U) {
        Wd wd[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t rel = pos - (c + 32 * u), e = c + 32 * u + lane;
            const unsigned starts = __reduce_or_sync(FULL, fin > 0 && rel < 32 ? 1u << rel : 0u);
            wd[u] = e < end ? scr[delta[first + __popc(starts & upto)] + e] : Wd(0);
            first += __popc(starts);
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t e = c + 32 * u + lane, v = ev_val(wd[u]);
            uint32_t before = __shfl_up_sync(FULL, v, 1);
            if (lane == 0) before = before1;
            before1 = __shfl_sync(FULL, v, 31);
            if (e < end) {
                dst[e] = wd[u];
                const P t = rc(ev_time(wd[u]));
                s0 += (before == kV0 ? t : P(0)) - (v == kV0 ? t : P(0));
                s1 += (before == kV1 ? t : P(0)) - (v == kV1 ? t : P(0));
            }
        }
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
        s0 += __shfl_xor_sync(FULL, s0, k);
        s1 += __shfl_xor_sync(FULL, s1, k);
    }
    uint32_t last = vtop;   // one warp: that of its last kept entry
    if constexpr (kWarp) {
        if (!bal) last = kVX;
    } else {
        if (lane == 0) { wp.a[wid] = s0; wp.b[wid] = s1; }
        __syncthreads();
    }
    if (tid == 0) {
        if constexpr (!kWarp) {
            last = kVX;
            s0 = s1 = 0;
            for (uint32_t k = 0; k < nw; ++k) {
                s0 += wp.a[k];
                s1 += wp.b[k];
                if (wp.last[k] < 4u) last = wp.last[k];
            }
        }
        using Sg = typename std::make_signed<P>::type;
        const unsigned long long D = w.t_end - w.t_begin;
        const unsigned long long t0 = (unsigned long long)(long long)(Sg)s0 + (last == kV0 ? D : 0ull);
        const unsigned long long t1 = (unsigned long long)(long long)(Sg)s1 + (last == kV1 ? D : 0ull);
        unsigned long long *sf = w.saif + 3ull * mdp->out_net;
        sf[0] = t0;
        sf[1] = t1;
        sf[2] = D - t0 - t1;
    }
}

}  // namespace

// kTab = false is the kernel of one-warp blocks (and of the class of four to
// six input nets).  Their 32 warps on an SM run all over it, and it is bound
// by instruction fetch (2.3 warps waiting for instructions per issue): it has
// one copy of finish_gate (three copies cost 28.6 instead of 26.7 ms on 8
// windows of 200,000 cells), the cut searches and irregular delays are calls
// (22.2 ms; on the 2 M cell design, whose blocks of four warps run the other
// kernel, calls cost 75.8 instead of 73.9), and what only meets between warps
// is left out (23.3 -> 20.8 ms).
//
// Gate outputs [d0, d1) of the level of every window of the launch (kSix: the
// class of four to six input nets, else the narrower ones; c1, c2: where the
// 2- and 3-input ones start).  Blocks take gate outputs from the back, the
// widest first, as they become free.
template <bool kBatch, bool kSix, bool kTab, class Wd>
__global__ void __launch_bounds__(kSix || kTab ? gate_resident<kSix, Wd>() : 32,
                                  kSix || kTab ? 1 : gate_resident<kSix, Wd>() / 32)
    k_gate(const WinSet<kBatch> ws, LevelArgs a, uint32_t d0, uint32_t d1, uint32_t c1, uint32_t c2)
{
    constexpr bool kWarp = !kSix && !kTab;
    __shared__ __align__(256) GateSmem<kBatch, kTab> sm;
    // per thread the time its segment starts at (then see finish_gate), then WarpParts
    extern __shared__ __align__(8) uint32_t s_seg[];
    const uint32_t nthr = kWarp ? 32u : blockDim.x;
    const uint32_t n = d1 - d0, total = n * ws.size();
    auto fetch = [&](uint32_t q) {   // thread 0
        sm.q = q < total ? q : kInf;
        if (q < total) sm.skip = *(volatile uint32_t *)ws.get(kBatch ? q / n : 0u).err != 0;
    };
    auto flush = [&]() {
        uint32_t win = 0;
        if constexpr (kBatch) win = sm.cw;
        const WinDev &w = ws.get(win);
        for (int k = 0; k < 4; ++k) {
            if (sm.ctr[k]) atomicAdd(&w.counters[k], sm.ctr[k]);
            sm.ctr[k] = 0;
        }
    };
    // launched while the previous level's last blocks run: nothing it wrote is
    // read before this; the next level's blocks may follow likewise
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        if constexpr (kBatch) sm.cw = kInf;
        for (int k = 0; k < 4; ++k) sm.ctr[k] = 0;
        fetch(blockIdx.x);   // the grid has at most one block per gate output
    }
    for (;;) {
        sync_block<kWarp>();
        const uint32_t q = sm.q;
        if (q == kInf) break;
        const bool skip = sm.skip != 0;
        const uint32_t win = kBatch ? q / n : 0u;
        if constexpr (kBatch) {
            // the window's descriptor in shared memory, out of the way of the walks
            const uint32_t cw = sm.cw;
            sync_block<kWarp>();
            if (win != cw) {
                if (threadIdx.x == 0) {
                    if (cw != kInf) flush();
                    sm.cw = win;
                }
                const uint32_t *src = reinterpret_cast<const uint32_t *>(&ws.get(win));
                uint32_t *d = reinterpret_cast<uint32_t *>(&sm.win);
                for (uint32_t k = threadIdx.x; k < sizeof(WinDev) / 4; k += nthr) d[k] = src[k];
                sync_block<kWarp>();
            }
        }
        auto next = [&]() { fetch(gridDim.x == total ? total : gridDim.x + atomicAdd(&ws.get(0).lvl[a.level].next[kSix ? 0 : 1], 1u)); };
        if (skip) {
            sync_block<kWarp>();   // sm.q is read
            if (threadIdx.x == 0) next();
            continue;
        }
        const uint32_t i = d1 - 1 - (kBatch ? q - win * n : q);
        auto go = [&](const WinDev &w) {
            Walked<Wd> wk;
            if constexpr (kSix) {
                wk = walk_gate<kMaxSlots, false, Wd>(w, a, i, sm, s_seg);
            } else {
                if (i >= c2) wk = walk_gate<3, kTab, Wd>(w, a, i, sm, s_seg);
                else if (i >= c1) wk = walk_gate<2, kTab, Wd>(w, a, i, sm, s_seg);
                else wk = walk_gate<1, kTab, Wd>(w, a, i, sm, s_seg);
            }
            finish_gate<kWarp, Wd>(w, a, i, sm, s_seg, wk, next);
        };
        if constexpr (kBatch) go(sm.win);
        else go(ws.get(0));
    }
    bool any = true;
    if constexpr (kBatch) any = sm.cw != kInf;
    if (threadIdx.x == 0 && any) flush();
}

void launch_gate(const WinDev *dw, const WinDev &h, uint32_t nwin, const LevelArgs &level, const uint32_t *cls,
                 GateThreads block, bool table, int sm_count, cudaStream_t st, uint32_t *launches)
{
    LevelArgs a = level;
    a.x_times = table ? 1u : 0u;
    auto go = [&](auto six, auto tab, uint32_t d0, uint32_t d1) {
        constexpr bool kSix = decltype(six)::value, kTab = decltype(tab)::value;
        if (d1 <= d0) return;
        const uint64_t total = (uint64_t)(d1 - d0) * nwin;
        const uint32_t resident = a.wide ? gate_resident<kSix, WideWord>() : gate_resident<kSix, uint32_t>();
        const uint32_t threads = kSix ? (block.six < resident ? block.six : resident) : block.narrow;
        const uint32_t parts = a.wide ? WarpParts<WideWord>::kBytes : WarpParts<uint32_t>::kBytes;
        const uint32_t smem = threads * 4 + (kSix || kTab ? threads / 32 * parts : 0);
        const uint64_t room = (uint64_t)sm_count * (resident / threads);
        const uint32_t grid = (uint32_t)(total < room ? total : room);
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(grid);
        lc.blockDim = dim3(threads);
        lc.dynamicSmemBytes = smem;
        lc.stream = st;
        lc.attrs = &at;
        lc.numAttrs = 1;
        if (a.wide)   // one window per launch
            cudaLaunchKernelEx(&lc, k_gate<false, kSix, kTab, WideWord>, WinSet<false>{h}, a, d0, d1, cls[1], cls[2]);
        else if (nwin == 1)
            cudaLaunchKernelEx(&lc, k_gate<false, kSix, kTab, uint32_t>, WinSet<false>{h}, a, d0, d1, cls[1], cls[2]);
        else
            cudaLaunchKernelEx(&lc, k_gate<true, kSix, kTab, uint32_t>, WinSet<true>{dw, nwin}, a, d0, d1, cls[1], cls[2]);
        ++*launches;
    };
    using T = std::integral_constant<bool, true>;
    using F = std::integral_constant<bool, false>;
    go(T(), F(), cls[3], cls[4]);
    // the step table is for warps none of whose segments starts at X: in a
    // block of one warp the first one does
    if (block.narrow > 32) go(F(), T(), 0u, cls[3]);
    else go(F(), F(), 0u, cls[3]);
}

}  // namespace gls
