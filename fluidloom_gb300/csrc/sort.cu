// sort.cu — LSD onesweep radix sort of uint64 keys with uint32 payloads.
//
// Replaces RadixSort::sortByKey (src/core/hashmap/RadixSort.cpp:55-104, a stub
// that launches nothing) and its kernels (kernels/hashmap/radix_sort.cl:14-122,
// whose atomic_inc scatter is unstable and whose digit is fixed at 8 bits,
// radix_sort.cl:5-6).  Design (onesweep, Adinets & Merrill 2022):
//  1. one upfront pass histograms every digit of every pass at once
//     (per-CTA shared histograms, then global atomics), and its last block
//     turns each pass histogram into exclusive bin offsets;
//  2. per pass, one kernel: each CTA takes the next tile (atomic ticket), ranks
//     its keys stably with warp __match_any_sync peer groups and per-warp
//     digit counters, publishes its per-digit counts, resolves its global
//     per-digit base by decoupled look-back over earlier tiles (one thread per
//     digit, bounded spin), stages the tile in shared memory in rank order and
//     writes it out with coalesced runs.
// Four shapes, chosen per context (fl_sort_set_config): 8- or 9-bit digits (9:
// 7 passes over 63-bit keys instead of 8) on tiles of 256 or 512 threads x 12
// keys, or x 4 for up to kSmallSort keys (512: half the tiles and twice the
// keys per digit run written, at 2 CTAs per SM; 256: 4 CTAs per SM with 8-bit
// digits, 3 with 9-bit, whose threads then take two digits each).
// Large sorts of many passes leave out low passes that the high ones decide (kPlannedSort).
// Stable: ties keep input order, so (key, payload) pairs match std::stable_sort.
#include "common.cuh"
#include "scan.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {

constexpr int kLargeItems = 12;            // keys per thread in a tile
constexpr int kSmallItems = 4;             // ... of a small sort
constexpr int kSmallWindow = 4;            // predecessors a small sort's look-back reads at once
constexpr int kMaxRadix = 512;
constexpr int kMaxPasses = 8;              // 64-bit keys, 8- or 9-bit digits

constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValMask = (1u << 30) - 1;

__host__ __device__ constexpr uint32_t digit_mask(int end_bit, int sh, int bits) {
    return end_bit - sh >= bits ? (1u << bits) - 1u : (1u << (end_bit - sh)) - 1u;
}

// A sort that may leave out passes keeps its state behind the histograms: the
// histogram's block count, the low passes left out, the runs to sort by their low digits.
struct SortPlan {
    unsigned done, defer, runs;
};
constexpr uint32_t kFewDigits = 32;
constexpr uint32_t kShortRun = 1024;       // keys of one high part that a warp sorts by counting

__host__ __device__ constexpr uint64_t range_mask(int begin_bit, int end_bit) {
    return end_bit - begin_bit >= 64 ? ~0ull : (1ull << (end_bit - begin_bit)) - 1;
}

// Every pass's histogram, then, in the block that finishes last (plan->done counts the
// blocks, starting at 0), each pass's bins scanned in place to exclusive offsets: a
// warp per pass, R / 32 consecutive bins a lane.  With kPlanned it also leaves
// out the low passes that meet at most kFewDigits different digits, and clears the
// table of k_sample.
template <int kBits, bool kPlanned>
__global__ void __launch_bounds__(256) k_histogram(const uint64_t* __restrict__ keys, size_t n, int begin_bit,
                                                   int end_bit, int passes, uint32_t* hist, SortPlan* plan,
                                                   uint64_t* table, size_t slots) {
    constexpr int R = 1 << kBits;
    __shared__ uint32_t h[kMaxPasses][R];
    __shared__ bool last;
    for (int i = threadIdx.x; i < kMaxPasses * R; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    size_t stride = (size_t)gridDim.x * blockDim.x;
    if (kPlanned)
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += stride) table[i] = ~0ull;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint64_t k = keys[i];
        for (int p = 0; p < passes; ++p) {
            int sh = begin_bit + kBits * p;
            atomicAdd(&h[p][(k >> sh) & digit_mask(end_bit, sh, kBits)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * R; i += blockDim.x) {
        uint32_t v = (&h[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&plan->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int lane = threadIdx.x & 31, p = threadIdx.x >> 5;  // 8 warps, at most 8 passes
    if (!kPlanned && p >= passes) return;
    if (p < passes) {
        uint32_t* g = hist + p * R + lane * (R / 32);
        uint32_t v[R / 32], sum = 0;
#pragma unroll
        for (int j = 0; j < R / 32; ++j) {
            v[j] = __ldcg(g + j);
            sum += v[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += t;
        }
        uint32_t run = incl - sum;
#pragma unroll
        for (int j = 0; j < R / 32; ++j) {
            g[j] = run;
            run += v[j];
        }
        if (kPlanned) {
            uint32_t used = 0;
#pragma unroll
            for (int j = 0; j < R / 32; ++j) used += v[j] ? 1u : 0u;
            used = __reduce_add_sync(0xFFFFFFFFu, used);
            if (lane == 0) h[p][0] = used;
        }
    }
    if (kPlanned) {
        __syncthreads();
        if (threadIdx.x == 0) {
            int d = 0;
            while (d < passes - 1 && h[d][0] <= kFewDigits) ++d;
            plan->defer = (unsigned)d;
        }
    }
}

__device__ __forceinline__ uint32_t ld_vol(const uint32_t* p) { return *(volatile const uint32_t*)p; }

// Before the passes: keys at random places meet in a table by what is above the digits left
// out.  Two with one high part and different low ones put the digit of their highest
// different bit, and those above, back among the passes.
template <int kBits>
__global__ void __launch_bounds__(256) k_sample(const uint64_t* __restrict__ keys, size_t n, int begin_bit, uint64_t mask,
                                                size_t samples, unsigned long long* table, int lg, SortPlan* plan) {
    const int defer = (int)ld_vol(&plan->defer);
    const size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (defer == 0 || w >= samples) return;
    uint64_t h = (w + 1) * 0x9e3779b97f4a7c15ull;
    h = (h ^ (h >> 32)) * 0x9e3779b97f4a7c15ull;
    h = (h ^ (h >> 29)) * 0x9e3779b97f4a7c15ull;
    const uint64_t k = (keys[__umul64hi(h, n)] >> begin_bit) & mask;
    const uint64_t high = k >> (kBits * defer);
    const uint64_t met = atomicExch(table + ((high * 0x9e3779b97f4a7c15ull) >> (64 - lg)), (unsigned long long)k);
    if (met != ~0ull && met != k && met >> (kBits * defer) == high)
        atomicMin(&plan->defer, (unsigned)((63 - __clzll((long long)(met ^ k))) / kBits));
}

// Dynamic shared memory of one onesweep tile: keys and values staged in rank
// order, per-warp digit counters, per-digit tile offsets and global bases,
// per-warp sums of the digit scan.
template <int kThreads, int kBits, int kItems>
__host__ __device__ constexpr size_t onesweep_smem() {
    return (size_t)kThreads * kItems * 12 +
           ((size_t)(kThreads / 32) * (1 << kBits) + 2 * (1 << kBits) + kThreads / 32) * 4;
}

// kPlanned: pass number `pass` of a sort that may leave passes out: nothing if this is one of them, else
// from the buffers where the passes run before it left the pairs.  Otherwise from the first into the second.
template <int kThreads, int kBits, int kItems, bool kPlanned>
__global__ void __launch_bounds__(kThreads, kThreads == 512 ? 2 : (kBits == 8 ? 4 : 3))
    k_onesweep(uint64_t* first_k, uint32_t* first_v, uint64_t* second_k, uint32_t* second_v, size_t n, int shift, uint32_t dmask,
               const uint32_t* bin_off, uint32_t* status, unsigned* ticket, uint32_t* dev_status,
               const SortPlan* plan, int pass) {
    constexpr int R = 1 << kBits;
    constexpr int kWarps = kThreads / 32;
    constexpr int kTile = kThreads * kItems;
    // digit scan: each of the first R / D threads takes D consecutive digits
    constexpr int D = R > kThreads ? R / kThreads : 1;
    static_assert(R % 32 == 0 && (R <= kThreads || R % kThreads == 0), "whole warps of digits");
    extern __shared__ __align__(16) unsigned char s_dyn[];
    uint64_t* s_keys = (uint64_t*)s_dyn;
    uint32_t* s_vals = (uint32_t*)(s_keys + kTile);
    uint32_t* s_warp_hist = s_vals + kTile;  // [kWarps][R]
    uint32_t* s_tile_excl = s_warp_hist + kWarps * R;
    uint32_t* s_glob = s_tile_excl + R;
    uint32_t* s_wsum = s_glob + R;
    __shared__ int s_tile;
    __shared__ int s_bad;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a tile before the wait helps the small sorts; in large ones (kPlanned: after it) 15,074,927 mesh keys
    // took 850 us with it before, 774 after
    if (!kPlanned) {
        if (threadIdx.x == 0) { s_tile = (int)atomicAdd(ticket, 1u); s_bad = 0; }
        for (int i = threadIdx.x; i < kWarps * R; i += kThreads) s_warp_hist[i] = 0;
    }
    // the passes are launched programmatically: this much of a pass overlaps the one before it,
    // whose output is read from here on
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    bool swapped = false;
    if (kPlanned) {
        // (every block waits above first: the pass after this one counts on the passes before)
        const int defer = (int)ld_vol(&plan->defer);
        if (pass < defer) return;
        swapped = (pass - defer) & 1;
    }
    // The pass before wrote the input while this kernel was already resident: ordinary loads, to which the
    // wait above makes it visible.  With __restrict__ a compiler may read buffers that a pass only reads
    // through the read-only cache, which is for data that nobody writes in the kernel's lifetime.  (__ldcg
    // for all of a tile before its ranking: 15,074,927 mesh keys and their sort 869 -> 940 us.)
    const uint64_t* kin = swapped ? second_k : first_k;
    const uint32_t* vin = swapped ? second_v : first_v;
    uint64_t* kout = swapped ? first_k : second_k;
    uint32_t* vout = swapped ? first_v : second_v;
    if (kPlanned) {
        if (threadIdx.x == 0) { s_tile = (int)atomicAdd(ticket, 1u); s_bad = 0; }
        for (int i = threadIdx.x; i < kWarps * R; i += kThreads) s_warp_hist[i] = 0;
    }
    __syncthreads();
    const int tile = s_tile;
    const size_t tbase = (size_t)tile * kTile;
    const size_t wbase = tbase + (size_t)warp * 32 * kItems;
    const unsigned lt = (1u << lane) - 1u;

    uint64_t k[kItems];
    uint32_t v[kItems];
    uint32_t rank[kItems];
    // stable in-warp ranking: iteration i handles keys wbase + i*32 + lane
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        size_t g = wbase + (size_t)i * 32 + lane;
        bool ok = g < n;
        k[i] = ok ? kin[g] : 0ull;
        v[i] = ok ? vin[g] : 0u;
        uint32_t d = ok ? (uint32_t)((k[i] >> shift) & dmask) : (uint32_t)R;
        unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
        // the group's first lane adds the group to the warp's digit counter and
        // hands the old count to its peers (one shared atomic, no warp barrier)
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0u;
        if (d < (uint32_t)R && lane == leader) base = atomicAdd(&s_warp_hist[warp * R + d], (uint32_t)__popc(peers));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
        rank[i] = base + __popc(peers & lt);
    }
    __syncthreads();
    // per-digit: tile count, cross-warp exclusive offsets (a thread per digit, or
    // R / kThreads digits per thread one after another)
    for (int d = threadIdx.x; d < R; d += kThreads) {
        uint32_t run = 0;
        for (int w = 0; w < kWarps; ++w) {
            uint32_t c = s_warp_hist[w * R + d];
            s_warp_hist[w * R + d] = run;
            run += c;
        }
        // publish aggregate, look back, publish inclusive
        uint32_t* st = status + (size_t)tile * R + d;
        uint32_t prefix = 0;
        // a status word carries its own value: no fence orders it after other data
        if (tile == 0) {
            *(volatile uint32_t*)st = kFlagInc | run;
        } else {
            *(volatile uint32_t*)st = kFlagAgg | run;
            int t = tile - 1;
            unsigned spins = 0;
            if constexpr (kItems == kSmallItems) {
                // kSmallWindow predecessors per round trip, the nearest first; tile 0 publishes
                // an inclusive word, so the walk ends there at the latest
                bool found = false;
                while (!found) {
                    uint32_t s[kSmallWindow];
#pragma unroll
                    for (int j = 0; j < kSmallWindow; ++j)
                        s[j] = t >= j ? ld_vol(status + (size_t)(t - j) * R + d) : 0u;
                    int used = 0;
                    bool ready = true;
#pragma unroll
                    for (int j = 0; j < kSmallWindow; ++j) {
                        ready = ready && !found && (s[j] & kFlagMask) != 0;
                        if (!ready) continue;
                        prefix += s[j] & kValMask;
                        found = (s[j] & kFlagMask) == kFlagInc;
                        ++used;
                    }
                    t -= used;
                    if (used == 0 && ++spins > FL_SPIN_LIMIT) {
                        atomicAdd(dev_status + FL_DEVSTAT_TIMEOUT, 1u);
                        s_bad = 1;
                        break;
                    }
                }
            } else {
                while (t >= 0) {
                    uint32_t s = ld_vol(status + (size_t)t * R + d);
                    if ((s & kFlagMask) == 0) {
                        if (++spins > FL_SPIN_LIMIT) {
                            atomicAdd(dev_status + FL_DEVSTAT_TIMEOUT, 1u);
                            s_bad = 1;
                            break;
                        }
                        continue;
                    }
                    prefix += s & kValMask;
                    if ((s & kFlagMask) == kFlagInc) break;
                    --t;
                }
            }
            *(volatile uint32_t*)st = kFlagInc | ((prefix + run) & kValMask);
        }
        s_glob[d] = bin_off[d] + prefix;
        // tile-local exclusive scan over digits of the tile counts
        s_tile_excl[d] = run;
    }
    __syncthreads();
    // block exclusive scan of s_tile_excl (R entries; thread t < R / D holds digits
    // tD .. tD + D - 1)
    {
        const int t0 = threadIdx.x * D;
        uint32_t c[D], sum = 0, incl = 0;
        if (t0 < R) {
#pragma unroll
            for (int j = 0; j < D; ++j) {
                c[j] = s_tile_excl[t0 + j];
                sum += c[j];
            }
            incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) s_wsum[warp] = incl;
        }
        __syncthreads();
        if (t0 < R) {
            uint32_t ex = incl - sum;
            for (int w = 0; w < warp; ++w) ex += s_wsum[w];
#pragma unroll
            for (int j = 0; j < D; ++j) {
                s_tile_excl[t0 + j] = ex;
                ex += c[j];
            }
        }
    }
    __syncthreads();
    // stage in rank order
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        size_t g = wbase + (size_t)i * 32 + lane;
        if (g < n) {
            uint32_t d = (uint32_t)((k[i] >> shift) & dmask);
            uint32_t pos = s_tile_excl[d] + s_warp_hist[warp * R + d] + rank[i];
            s_keys[pos] = k[i];
            s_vals[pos] = v[i];
        }
    }
    __syncthreads();
    if (s_bad) return;  // a timed-out look-back leaves this tile unwritten; the host reports the error
    size_t count = n - tbase < (size_t)kTile ? n - tbase : (size_t)kTile;
    for (int i = threadIdx.x; i < (int)count; i += kThreads) {
        uint64_t kk = s_keys[i];
        uint32_t d = (uint32_t)((kk >> shift) & dmask);
        size_t pos = (size_t)s_glob[d] + (size_t)(i - (int)s_tile_excl[d]);
        if (pos >= n) { atomicAdd(dev_status + FL_DEVSTAT_BOUNDS, 1u); continue; }
        kout[pos] = kk;
        vout[pos] = s_vals[i];
    }
}

// The pairs sorted by their high digits alone, where they are not in order (of the sorted bits: begin_bit up,
// as many as mask has): what is out of order shares its high part, so the first key of each run of one
// high part that is not in order goes into list (at most n / 2 of them).
template <int kBits>
__global__ void __launch_bounds__(256) k_order(const uint64_t* __restrict__ first_k, const uint64_t* __restrict__ second_k,
                                               size_t n, SortPlan* plan, int passes, int begin_bit, uint64_t mask,
                                               uint32_t* __restrict__ list) {
    const int defer = (int)plan->defer, low = kBits * defer;
    if (defer == 0) return;
    const uint64_t* __restrict__ keys = (passes - defer) & 1 ? second_k : first_k;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    auto key = [&](size_t i) { return (keys[i] >> begin_bit) & mask; };
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x + 1; i < n; i += stride) {
        uint64_t k = key(i - 1);
        if (key(i) >= k) continue;
        // back to the run's start, or to an earlier key out of order, whose thread lists the run
        size_t j = i - 1;
        bool first = true;
        while (first && j > 0) {
            const uint64_t before = key(j - 1);
            if (before >> low != k >> low) break;
            first = before <= k;
            k = before;
            --j;
        }
        if (first) list[atomicAdd(&plan->runs, 1u)] = (uint32_t)j;
    }
}

// The listed runs in order, a warp each, through the buffers that the last pass read.  In a short run a
// key's place is the number of the run's keys before it (equal ones in the order they have); a longer one
// takes stable passes over its low bits, eight at a time.
template <int kBits>
__global__ void __launch_bounds__(256) k_runs(uint64_t* first_k, uint32_t* first_v, uint64_t* second_k, uint32_t* second_v,
                                              size_t n, const SortPlan* plan, int passes, int begin_bit, uint64_t mask,
                                              const uint32_t* list) {
    __shared__ uint32_t s_count[8][256];
    const uint32_t runs = plan->runs;
    const int low = kBits * (int)plan->defer, lane = threadIdx.x & 31;
    const bool swapped = (passes - (int)plan->defer) & 1;
    uint64_t* const keys = swapped ? second_k : first_k;
    uint32_t* const vals = swapped ? second_v : first_v;
    uint64_t* const tk = swapped ? first_k : second_k;
    uint32_t* const tv = swapped ? first_v : second_v;
    auto bits = [&](uint64_t k) { return (k >> begin_bit) & mask; };
    uint32_t* c = s_count[threadIdx.x >> 5];
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < runs; r += warps) {
        const size_t start = list[r];
        const uint64_t high = bits(keys[start]) >> low;
        uint32_t len = 0;
        for (unsigned in = 0xFFFFFFFFu; in == 0xFFFFFFFFu;) {
            const size_t i = start + len + lane;
            in = __ballot_sync(0xFFFFFFFFu, i < n && bits(keys[i]) >> low == high);
            len += in == 0xFFFFFFFFu ? 32u : (uint32_t)__ffs(~in) - 1u;
        }
        bool moved = true;  // the run's order is in tk, tv
        if (len <= kShortRun) {
            for (uint32_t e = lane; e < len; e += 32u) {
                const uint64_t mine = bits(keys[start + e]);
                uint32_t at = 0;
                for (uint32_t j = 0; j < len; ++j) {
                    const uint64_t other = bits(keys[start + j]);
                    at += other < mine || (other == mine && j < e) ? 1u : 0u;
                }
                tk[start + at] = keys[start + e];
                tv[start + at] = vals[start + e];
            }
        } else {
            moved = false;
            for (int sh = 0; sh < low; sh += 8, moved = !moved) {
                const uint64_t* ak = (moved ? tk : keys) + start;
                const uint32_t* av = (moved ? tv : vals) + start;
                uint64_t* bk = (moved ? keys : tk) + start;
                uint32_t* bv = (moved ? vals : tv) + start;
                for (int i = lane; i < 256; i += 32) c[i] = 0u;
                __syncwarp();
                for (uint32_t e = lane; e < len; e += 32u) atomicAdd(&c[(bits(ak[e]) >> sh) & 255u], 1u);
                __syncwarp();
                uint32_t v[8], sum = 0;
                for (int j = 0; j < 8; ++j) sum += v[j] = c[lane * 8 + j];
                uint32_t run = sum;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, run, o);
                    if (lane >= o) run += t;
                }
                run -= sum;
                for (int j = 0; j < 8; ++j) {
                    c[lane * 8 + j] = run;
                    run += v[j];
                }
                __syncwarp();
                for (uint32_t e0 = 0; e0 < len; e0 += 32u) {
                    const bool in = e0 + lane < len;
                    const uint64_t k = in ? ak[e0 + lane] : 0ull;
                    const uint32_t d = in ? (uint32_t)(bits(k) >> sh) & 255u : 256u;
                    const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
                    const uint32_t base = in ? c[d] : 0u;
                    __syncwarp();
                    if (in && lane == __ffs(peers) - 1) c[d] = base + (uint32_t)__popc(peers);
                    __syncwarp();
                    if (in) {
                        const uint32_t at = base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
                        bk[at] = k;
                        bv[at] = av[e0 + lane];
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
        for (uint32_t e = lane; moved && e < len; e += 32u) {
            keys[start + e] = tk[start + e];
            vals[start + e] = tv[start + e];
        }
    }
}

// The sorted pairs back from the second buffers where an odd number of passes has run.
__global__ void __launch_bounds__(256) k_home(uint64_t* __restrict__ first_k, uint32_t* __restrict__ first_v,
                                              const uint64_t* __restrict__ second_k,
                                              const uint32_t* __restrict__ second_v, size_t n, const SortPlan* plan,
                                              int passes) {
    if (!((passes - (int)plan->defer) & 1)) return;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        first_k[i] = second_k[i];
        first_v[i] = second_v[i];
    }
}

// A pass of one tile is a chain of latencies (about 11,800 cycles at 12 keys per thread: 4,000 rank
// them, 1,800 stage them, 2,400 write them out), so while the tiles fit the GPU at once a sort takes
// as long as one tile, and fewer keys per thread make more and shorter tiles.  Their look-back is
// longer, so it reads kSmallWindow words per round trip, and each pass starts while the one before
// it ends.  Keys and sort: 40,961 30-bit keys 61 us with 12 keys per thread, 49 with 4, 37 with the
// passes overlapped too; 3,000 63-bit keys 85 -> 42, 240,000 117 -> 89, 1,000,000 180 -> 176, and
// 1,500,000, whose tiles no longer fit at once, 224 -> 225.
constexpr size_t kSmallSort = 1u << 20;

// Anchor keys of cells far above the key's depth: their low digits are set by the high ones (the
// walk down to a cell's first corner), so that sorting by the high digits sorts them.  A large sort
// of many passes looks: low passes that meet at most kFewDigits digits (every digit turns up in keys
// spread over them) are left out, unless a sample shows that the high digits don't decide them
// (k_sample), and the runs that are then not in order, too rare or too short for the sample, are sorted by
// themselves (k_order, k_runs).  Of kSampleShare sqrt(n) keys, s of n which lie in runs of one high part of
// r keys make about kSampleShare^2 r s / (2 n) pairs of one run, so those are a few per cent of the keys or
// less, and no longer than about sqrt(n) / 2.  All of it is decided on the device: the sort stays asynchronous.
// 63-bit keys of 30-bit cells: 15,074,927 in 1,213 us with every pass, 777 now; 4 M 403 and 265, 2.1 M 283 and
// 181.  Keys whose few low digits the high ones don't decide, 15,074,927: a tag of two bits beside keys that come
// up twice 1,187 and 1,161; eleven low parts at random 1,213 and 935 (2,141 and 1,819 where every pass ran again
// after the check).  Keys that fill their digits pay for the launches that find nothing to do, 15 us or so, which the
// rule keeps to sorts that are long beside it: 4 M take 440, 1.5 M without the plan 250.
constexpr size_t kSampleShare = 16;
constexpr size_t kPlannedSort = 2u << 20;
constexpr int kPlannedPasses = 6;

// Bytes of one pass's tile status words and ticket, for every shape: at most
// ceil(n / smallest tile) tiles of at most kMaxRadix digits (9-bit digits on the
// smallest tile reach both bounds at once).
size_t status_stride_min(size_t n) {
    const size_t tile = 256 * (n <= kSmallSort ? kSmallItems : kLargeItems);
    return fl_align256(((n + tile - 1) / tile) * kMaxRadix * 4 + 4) + 4096;
}

// All passes of one shape.  The scratch layout (fl_sort_scratch_bytes): the
// alternate key and value buffers, the pass histograms (kMaxPasses x
// kMaxRadix), a block count, then per pass its tile status words and ticket, at a stride that
// fits every shape's tiles (status_stride_min).
template <int kThreads, int kBits, int kItems>
int sort_passes(fl_ctx* ctx, uint64_t* keys, uint32_t* vals, size_t n, int begin_bit, int end_bit, void* scratch) {
    constexpr int R = 1 << kBits;
    constexpr int kTile = kThreads * kItems;
    const int passes = (end_bit - begin_bit + kBits - 1) / kBits;
    if (passes <= 0) return FL_OK;
    const size_t tiles = (n + kTile - 1) / kTile;
    char* p = (char*)scratch;
    uint64_t* kalt = (uint64_t*)p; p += fl_align256(n * 8);
    uint32_t* valt = (uint32_t*)p; p += fl_align256(n * 4);
    uint32_t* hist = (uint32_t*)p; p += fl_align256((size_t)kMaxPasses * kMaxRadix * 4);
    SortPlan* plan = (SortPlan*)p; p += 256;
    char* stat0 = p;
    const size_t stat_stride = fl_align256(tiles * R * 4 + 4);  // at most status_stride_min(n)
    // clear histograms, their block count and the per-pass status/tickets in one memset
    FL_TRY_CUDA(ctx, cudaMemsetAsync(hist, 0, fl_align256((size_t)kMaxPasses * kMaxRadix * 4) + 256 + passes * stat_stride,
                                     ctx->stream), "sort clear");
    constexpr size_t smem = onesweep_smem<kThreads, kBits, kItems>();
    constexpr bool kCanPlan = kItems == kLargeItems;
    const bool planned = kCanPlan && n >= kPlannedSort && passes >= kPlannedPasses;
    const auto kernel = planned ? k_onesweep<kThreads, kBits, kItems, kCanPlan> : k_onesweep<kThreads, kBits, kItems, false>;
    FL_TRY_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                "sort shared memory");
    unsigned hb = fl_blocks(n, 256, ctx->num_sms * 4);
    // the sample's table, at most a quarter full, in the alternate keys
    const size_t samples = std::max(kSampleShare * (size_t)std::sqrt((double)n), n / 256);
    int lg = 0;
    while ((1ull << lg) < 4 * samples) ++lg;
    const uint64_t mask = range_mask(begin_bit, end_bit);
    (planned ? k_histogram<kBits, true> : k_histogram<kBits, false>)<<<hb, 256, 0, ctx->stream>>>(
        keys, n, begin_bit, end_bit, passes, hist, plan, kalt, (size_t)1 << lg);
    FL_CHECK_LAUNCH(ctx, "k_histogram");
    if (planned) {
        k_sample<kBits><<<(unsigned)((samples + 255) / 256), 256, 0, ctx->stream>>>(keys, n, begin_bit, mask, samples,
                                                                                    (unsigned long long*)kalt, lg, plan);
        FL_CHECK_LAUNCH(ctx, "k_sample");
    }
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)tiles);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    uint64_t* ks[2] = {keys, kalt};
    uint32_t* vs[2] = {vals, valt};
    int cur = 0;  // of a planned sort the kernels work out the buffers
    for (int ps = 0; ps < passes; ++ps) {
        uint32_t* status = (uint32_t*)(stat0 + ps * stat_stride);
        unsigned* ticket = (unsigned*)(status + tiles * R);
        int sh = begin_bit + kBits * ps;
        const uint32_t* offs = hist + ps * R;
        cudaLaunchKernelEx(&cfg, kernel, ks[cur], vs[cur], ks[cur ^ 1], vs[cur ^ 1], n, sh, digit_mask(end_bit, sh, kBits),
                           offs, status, ticket, ctx->dev_status, (const SortPlan*)plan, ps);
        FL_CHECK_LAUNCH(ctx, "k_onesweep");
        if (!planned) cur ^= 1;
    }
    if (planned) {
        const unsigned grid = fl_blocks(n, 256, ctx->num_sms * 8);
        // over the status words, which the passes no longer need: passes * status_stride_min(n) >= 4 n bytes
        uint32_t* list = (uint32_t*)stat0;
        k_order<kBits><<<grid, 256, 0, ctx->stream>>>(keys, kalt, n, plan, passes, begin_bit, mask, list);
        FL_CHECK_LAUNCH(ctx, "k_order");
        k_runs<kBits><<<ctx->num_sms * 4, 256, 0, ctx->stream>>>(keys, vals, kalt, valt, n, plan, passes, begin_bit, mask,
                                                                 list);
        FL_CHECK_LAUNCH(ctx, "k_runs");
        k_home<<<grid, 256, 0, ctx->stream>>>(keys, vals, kalt, valt, n, plan, passes);
        FL_CHECK_LAUNCH(ctx, "k_home");
    }
    if (cur == 1) {
        FL_TRY_CUDA(ctx, cudaMemcpyAsync(keys, kalt, n * 8, cudaMemcpyDeviceToDevice, ctx->stream), "sort copy");
        FL_TRY_CUDA(ctx, cudaMemcpyAsync(vals, valt, n * 4, cudaMemcpyDeviceToDevice, ctx->stream), "sort copy");
    }
    return FL_OK;
}

}  // namespace

// passes: the 8-bit pass count of the key range (every shape needs at most as many).
size_t fl_sort_scratch_bytes(size_t n, int passes) {
    return fl_align256(n * 8) + fl_align256(n * 4) + fl_align256((size_t)kMaxPasses * kMaxRadix * 4) +
           (size_t)passes * status_stride_min(n) + 256;
}

int fl_sort_pairs_with(fl_ctx* ctx, uint64_t* keys, uint32_t* vals, size_t n, int begin_bit, int end_bit,
                       void* scratch) {
    if (n <= 1 || end_bit <= begin_bit) return FL_OK;
    const bool wide = ctx->sort_tile_threads == 512, nine = ctx->sort_digit_bits == 9;
    auto run = [&](auto items) {
        constexpr int I = decltype(items)::value;
        if (nine)
            return wide ? sort_passes<512, 9, I>(ctx, keys, vals, n, begin_bit, end_bit, scratch)
                        : sort_passes<256, 9, I>(ctx, keys, vals, n, begin_bit, end_bit, scratch);
        return wide ? sort_passes<512, 8, I>(ctx, keys, vals, n, begin_bit, end_bit, scratch)
                    : sort_passes<256, 8, I>(ctx, keys, vals, n, begin_bit, end_bit, scratch);
    };
    return n <= kSmallSort ? run(std::integral_constant<int, kSmallItems>()) : run(std::integral_constant<int, kLargeItems>());
}

extern "C" int fl_sort_set_config(fl_ctx* ctx, int digit_bits, int tile_threads) {
    if (!ctx) return FL_E_INVALID_ARG;
    const bool ok = (digit_bits == 8 || digit_bits == 9) && (tile_threads == 256 || tile_threads == 512);
    if (!ok)
        return fl_set_error(ctx, FL_E_INVALID_ARG,
                            "fl_sort_set_config: digit_bits 8 or 9, tile_threads 256 or 512");
    ctx->sort_digit_bits = digit_bits;
    ctx->sort_tile_threads = tile_threads;
    return FL_OK;
}

extern "C" int fl_sort_get_config(fl_ctx* ctx, int* digit_bits, int* tile_threads) {
    if (!ctx || !digit_bits || !tile_threads) return FL_E_INVALID_ARG;
    *digit_bits = ctx->sort_digit_bits;
    *tile_threads = ctx->sort_tile_threads;
    return FL_OK;
}

extern "C" int fl_sort_pairs_u64_u32(fl_ctx* ctx, uint64_t* keys, uint32_t* vals, size_t n, int begin_bit,
                                     int end_bit) {
    if (!ctx) return FL_E_INVALID_ARG;
    if (n <= 1) return FL_OK;
    if (!keys || !vals || begin_bit < 0 || end_bit > 64 || begin_bit >= end_bit)
        return fl_set_error(ctx, FL_E_INVALID_ARG, "fl_sort_pairs_u64_u32: bad pointer or bit range");
    if (n >= (1ull << 30)) return fl_set_error(ctx, FL_E_INVALID_ARG, "fl_sort_pairs_u64_u32: n >= 2^30");
    int passes = (end_bit - begin_bit + 7) / 8;
    int rc = fl_scratch_reserve(ctx, fl_sort_scratch_bytes(n, passes));
    if (rc) return rc;
    return fl_sort_pairs_with(ctx, keys, vals, n, begin_bit, end_bit, ctx->scratch);
}
