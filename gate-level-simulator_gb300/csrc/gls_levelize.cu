// gls_levelize: Kahn levels of an instance graph on the GPU.
//
// The reference levelizes in `process` (GenerateAdjacencyList,
// SetInDegrees, TopologyOrder; src/process.cpp:90-176): level 0 holds the
// instances without predecessors, and every later level takes, in instance
// order, the instances whose predecessors are all placed.  An instance's
// level is therefore the length of the longest predecessor chain that ends
// at it.  Here threads look at their instances' predecessors until all have a
// level and then give one more than the largest of theirs; a stable radix
// sort by level packs the instances (the reference's level packing, 423-566).
//
// What bounds it: the chain of levels, one read through L2 each, then copies
// and calls.  A sweep that looked at every instance once and reported to the
// host after each, with the packing on the host, took 2.33 ms a call for
// 200,000 instances in 60 levels.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "gls.h"

namespace {

constexpr uint32_t kUnset = 0xFFFFFFFFu;
constexpr int kPolls = 256;             // looks at a thread's only instance per sweep
constexpr int kRounds = 32;             // looks at each of a thread's several
constexpr uint32_t kSortTile = 2048;    // instances per block of the sort, 256 threads
constexpr int kTileRounds = kSortTile / 256;

struct Status {
    unsigned long long placed;   // instances with a level
    uint32_t top;                // largest level given
    uint32_t bad;                // a predecessor out of range
};

// One sweep: an instance without a level takes one when all its
// predecessors have one.  A level word is written once, from kUnset to its
// final value, so a concurrent reader sees one or the other, and nothing waits
// for another thread without end.  A thread with one instance looks at it up
// to kPolls times, so a sweep places a run of levels.  A thread with several
// looks at each once a round, kRounds rounds a sweep: while it polled one, the
// predecessors of others' instances among its own would wait (in random file
// order 2 M instances of 400 levels took 178 ms with polls, of 60 levels 1 M
// 12.5; with a sweep of one look each 12.1 and 4.6, in rounds 5.5 and 1.4).
__global__ void k_level_sweep(uint32_t n, const uint64_t *__restrict__ ps, const uint32_t *__restrict__ pred,
                              uint32_t *lv, Status *st)
{
    uint32_t mine = 0, top = 0;
    volatile uint32_t *const v = lv;
    const uint32_t threads = gridDim.x * blockDim.x;
    const int polls = n > threads ? 1 : kPolls;
    uint64_t from = blockIdx.x * blockDim.x + threadIdx.x;   // the first instance not known to have a level
    for (int r = n > threads ? kRounds : 1; r > 0 && from < n; --r) {
        uint64_t left = n;
        for (uint64_t i = from; i < n; i += threads) {
            if (v[i] != kUnset) continue;
            uint64_t e = ps[i];
            const uint64_t end = ps[i + 1];
            uint32_t m = 0;
            bool out = false;
            for (int k = 0; e < end && k < polls; ++k) {
                const uint32_t p = pred[e];
                if (p >= n) { out = true; break; }
                const uint32_t l = v[p];
                if (l != kUnset) {
                    m = max(m, l + 1);
                    ++e;
                    --k;   // a predecessor passed is no look spent
                }
            }
            if (out) {
                st->bad = 1;
            } else if (e == end) {
                v[i] = m;
                ++mine;
                top = max(top, m);
            } else if (left == n) {
                left = i;
            }
        }
        from = left;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0 && mine) {
        atomicAdd(&st->placed, (unsigned long long)mine);
        atomicMax(&st->top, top);
    }
}

// ---- stable radix sort of the instances by level, 8 bits a pass

// instances of every digit in a tile
__global__ void __launch_bounds__(256) k_tile_count(uint32_t n, const uint32_t *__restrict__ key, const uint32_t *__restrict__ val,
                                                    int shift, uint32_t tiles, uint32_t *__restrict__ count)
{
    __shared__ uint32_t s[256];
    s[threadIdx.x] = 0;
    __syncthreads();
    for (int r = 0; r < kTileRounds; ++r) {
        const uint32_t k = blockIdx.x * kSortTile + r * 256 + threadIdx.x;
        if (k < n) atomicAdd(&s[(key[val ? val[k] : k] >> shift) & 255u], 1u);
    }
    __syncthreads();
    count[threadIdx.x * tiles + blockIdx.x] = s[threadIdx.x];
}

// exclusive scan of x[0..n), one block
__global__ void __launch_bounds__(1024) k_scan(uint32_t n, uint32_t *x)
{
    __shared__ uint32_t s[32];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t run = 0;
    for (uint32_t b = 0; b < n; b += 4096) {
        const uint32_t k = b + threadIdx.x * 4;
        uint32_t v[4], t = 0;
        for (int u = 0; u < 4; ++u) {
            v[u] = k + u < n ? x[k + u] : 0u;
            t += v[u];
        }
        uint32_t inc = t;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s[wid] = inc;
        __syncthreads();
        if (wid == 0) {
            uint32_t w = s[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            s[lane] = w;
        }
        __syncthreads();
        uint32_t at = run + (wid ? s[wid - 1] : 0u) + inc - t;
        run += s[31];
        for (int u = 0; u < 4; ++u) {
            if (k + u < n) x[k + u] = at;
            at += v[u];
        }
        __syncthreads();   // s is reused
    }
}

// a tile's instances to their places, in order: a warp takes an eighth of the
// tile, lanes of one digit rank themselves by a match
__global__ void __launch_bounds__(256) k_tile_scatter(uint32_t n, const uint32_t *__restrict__ key, const uint32_t *__restrict__ val,
                                                      int shift, uint32_t tiles, const uint32_t *__restrict__ base,
                                                      uint32_t *__restrict__ out)
{
    __shared__ uint32_t s[8][256];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    for (int w = 0; w < 8; ++w) s[w][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t first = blockIdx.x * kSortTile + wid * 256 + lane;
    uint32_t item[8], digit[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint32_t k = first + r * 32;
        item[r] = k < n ? (val ? val[k] : k) : kUnset;
        digit[r] = k < n ? (key[item[r]] >> shift) & 255u : 256u;
        const unsigned same = __match_any_sync(0xffffffffu, digit[r]);
        if (k < n && (same & ((1u << lane) - 1u)) == 0) s[wid][digit[r]] += __popc(same);
        __syncwarp();
    }
    __syncthreads();
    uint32_t run = base[threadIdx.x * tiles + blockIdx.x];
    for (int w = 0; w < 8; ++w) {
        const uint32_t c = s[w][threadIdx.x];
        s[w][threadIdx.x] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const unsigned same = __match_any_sync(0xffffffffu, digit[r]);
        const uint32_t before = __popc(same & ((1u << lane) - 1u));
        uint32_t at = 0;
        if (digit[r] < 256u) at = s[wid][digit[r]];
        __syncwarp();
        if (digit[r] < 256u) {
            out[at + before] = item[r];
            if (before == 0) s[wid][digit[r]] = at + __popc(same);
        }
        __syncwarp();
    }
}

// the first position of every level (each holds an instance)
__global__ void k_level_starts(uint32_t n, const uint32_t *__restrict__ lv, const uint32_t *__restrict__ order,
                               uint32_t nl, uint32_t *__restrict__ start)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t l = lv[order[k]];
        if (k == 0 || lv[order[k - 1]] != l) start[l] = k;
        if (k == n - 1) start[nl] = n;
    }
}

struct Buf {
    void *p = nullptr;
    ~Buf() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) { return cudaMalloc(&p, n ? n : 16); }
};

struct Stream {
    cudaStream_t st = nullptr;
    ~Stream() { if (st) cudaStreamDestroy(st); }
};

size_t up(size_t n) { return (n + 255) & ~(size_t)255; }

}  // namespace

extern "C" int gls_levelize(int device, uint32_t n_inst, const uint64_t *pred_start, const uint32_t *pred,
                            uint32_t *order, uint32_t *level_start, uint32_t *n_levels)
{
    if (!order || !level_start || !n_levels || (n_inst && !pred_start)) return GLS_EINVAL;
    *n_levels = 0;
    level_start[0] = 0;
    if (n_inst == 0) return GLS_OK;
    // a monotone start table keeps every read of the predecessor list in range
    if (pred_start[0] != 0) return GLS_EINVAL;
    for (uint32_t i = 0; i < n_inst; ++i)
        if (pred_start[i + 1] < pred_start[i]) return GLS_EINVAL;
    const uint64_t n_edges = pred_start[n_inst];
    if (n_edges && !pred) return GLS_EINVAL;
    if (cudaSetDevice(device) != cudaSuccess) return GLS_ECUDA;
    Stream s;
    Buf mem;   // one allocation: status, levels, two orders, tile counts, level starts, starts, predecessors
    if (cudaStreamCreateWithFlags(&s.st, cudaStreamNonBlocking) != cudaSuccess) return GLS_ECUDA;
    const uint32_t tiles = (n_inst + kSortTile - 1) / kSortTile;
    const size_t words = up((size_t)n_inst * 4), o_lv = 256, o_a = o_lv + words, o_b = o_a + words, o_cnt = o_b + words,
                 o_start = o_cnt + up((size_t)tiles * 1024), o_ps = o_start + up(((size_t)n_inst + 1) * 4),
                 o_pred = o_ps + up(((size_t)n_inst + 1) * 8);
    if (mem.alloc(o_pred + up(n_edges * 4))) return GLS_ENOMEM;
    char *const m = static_cast<char *>(mem.p);
    Status *const st = reinterpret_cast<Status *>(m);
    uint32_t *const lv = reinterpret_cast<uint32_t *>(m + o_lv), *const cnt = reinterpret_cast<uint32_t *>(m + o_cnt),
                   *const start = reinterpret_cast<uint32_t *>(m + o_start);
    uint64_t *const ps = reinterpret_cast<uint64_t *>(m + o_ps);
    uint32_t *const pr = reinterpret_cast<uint32_t *>(m + o_pred);
    if (cudaMemcpyAsync(ps, pred_start, ((size_t)n_inst + 1) * 8, cudaMemcpyHostToDevice, s.st) ||
        (n_edges && cudaMemcpyAsync(pr, pred, n_edges * 4, cudaMemcpyHostToDevice, s.st)) ||
        cudaMemsetAsync(lv, 0xFF, (size_t)n_inst * 4, s.st) || cudaMemsetAsync(st, 0, sizeof(Status), s.st))
        return GLS_ECUDA;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const uint32_t grid = std::max(1u, std::min((uint32_t)std::max(1, sms) * 8, (n_inst + 255) / 256));
    Status h{};
    for (unsigned long long before = 0;; before = h.placed) {
        k_level_sweep<<<grid, 256, 0, s.st>>>(n_inst, ps, pr, lv, st);
        if (cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, s.st) || cudaStreamSynchronize(s.st)) return GLS_ECUDA;
        if (h.bad) return GLS_EINVAL;              // a predecessor index out of range
        if (h.placed == n_inst) break;
        if (h.placed == before) return GLS_EINVAL; // nothing placed: the rest lies on or behind a loop
    }
    // level packing: the instances of every level in instance order
    const uint32_t nl = h.top + 1;
    const uint32_t *src = nullptr;   // the first pass takes the instances in order
    uint32_t *dst = reinterpret_cast<uint32_t *>(m + o_a), *other = reinterpret_cast<uint32_t *>(m + o_b);
    int shift = 0;
    do {
        k_tile_count<<<tiles, 256, 0, s.st>>>(n_inst, lv, src, shift, tiles, cnt);
        k_scan<<<1, 1024, 0, s.st>>>(tiles * 256, cnt);
        k_tile_scatter<<<tiles, 256, 0, s.st>>>(n_inst, lv, src, shift, tiles, cnt, dst);
        src = dst;
        std::swap(dst, other);
        shift += 8;
    } while (shift < 32 && (h.top >> shift));
    k_level_starts<<<grid, 256, 0, s.st>>>(n_inst, lv, src, nl, start);
    if (cudaGetLastError() || cudaMemcpyAsync(order, src, (size_t)n_inst * 4, cudaMemcpyDeviceToHost, s.st) ||
        cudaMemcpyAsync(level_start, start, ((size_t)nl + 1) * 4, cudaMemcpyDeviceToHost, s.st) ||
        cudaStreamSynchronize(s.st))
        return GLS_ECUDA;
    *n_levels = nl;
    return GLS_OK;
}
