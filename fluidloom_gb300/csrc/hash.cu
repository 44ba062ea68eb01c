// hash.cu — GPU open-addressing hash table (key -> index), the sorted point
// locator and the neighbour table rebuilds.
//
// Replaces HashTableManager::rebuild/query (src/core/hashmap/HashTableManager.cpp:101-159,
// which launch nothing) with the kernels they name (kernels/hashmap/hash_build.cl:19-82,
// kernels/hashmap/hash_query.cl:22-98): EMPTY key = ~0, INVALID value = ~0,
// power-of-two capacity, linear probing, a repeated key keeps the value of
// the LAST input carrying it (the order sequential insertion gives; resolved
// with an atomicMax on the input index, in the API's tables only when a build
// meets repeated keys, so the result does not depend on thread timing).  The slot is the high bits of key * 0x9e3779b97f4a7c15
// (Fibonacci hashing); the reference masks the low bits, which for 12-state
// keys of coarse anchors fall on a handful of slots.
#include "common.cuh"
#include "hash.cuh"
#include "keys.cuh"
#include "scan.cuh"

#include <algorithm>
#include <cstring>

namespace {

constexpr int kProbeLimit = 256;

__global__ void k_hash_clear(uint64_t* __restrict__ tk, uint32_t* __restrict__ tv, uint64_t cap) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += stride) {
        if (tv) {
            tk[i] = FL_EMPTY_KEY;
            tv[i] = FL_INVALID_INDEX;
        } else {
            reinterpret_cast<ulonglong2*>(tk)[i] = make_ulonglong2(FL_EMPTY_KEY, 0ull);
        }
    }
}

// Insertion: the thread whose CAS claims an empty slot stores its value with a
// plain store; a thread that finds its key already there flags the build
// (FL_DEVSTAT_HASH_DUPS) and stores nothing.  Without repeated keys that is
// the table; with them the passes below give each repeated key the value
// of its last input.  kIndex: the values are the input indices, whose maximum (FL_INVALID_INDEX
// is -1 there) is the last input's at once.
template <bool kIndex>
__global__ void __launch_bounds__(256) k_hash_insert(uint64_t* __restrict__ tk, uint32_t* __restrict__ tv, int lg,
                                                     const uint64_t* __restrict__ keys,
                                                     const uint32_t* __restrict__ vals, size_t n,
                                                     uint32_t* dev_status) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const uint64_t mask = (1ull << lg) - 1;
    bool dup = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t k = keys[i];
        if (k == FL_EMPTY_KEY) continue;
        uint64_t s = fl_hash_slot(k, lg);
        int p = 0;
        for (; p < kProbeLimit; ++p) {
            const unsigned long long prev = atomicCAS((unsigned long long*)(tk + s), FL_EMPTY_KEY, k);
            if (kIndex) {
                if (prev == FL_EMPTY_KEY || prev == k) atomicMax((int*)(tv + s), (int)i);
            } else {
                if (prev == FL_EMPTY_KEY) tv[s] = vals ? vals[i] : (uint32_t)i;
                if (prev == k) dup = true;
            }
            if (prev == FL_EMPTY_KEY || prev == k) break;
            s = (s + 1) & mask;
        }
        if (p == kProbeLimit) atomicAdd(dev_status + FL_DEVSTAT_HASH_OVERFLOW, 1u);
    }
    if (dup) atomicOr(dev_status + FL_DEVSTAT_HASH_DUPS, 1u);
}

// A mesh's cells under their anchor keys (k_cell_keys') in the 16-byte-slot layout: the key worked out
// on the way in, the slot's key word by CAS, its value word by a 64-bit maximum of (cell + 1) << 32 |
// level << 27 | cell, so that of cells with one key the last is kept whatever the order of the threads.
// Keys and table in one pass (262,144 cells, ghosts filled from them: 80 us with k_cell_keys before, 74 now).
__global__ void __launch_bounds__(256) k_hash_insert_cells(uint64_t* __restrict__ tk, int lg, fl_mesh_dev m,
                                                           fl_domain_dev dom, uint32_t* dev_status) {
    __shared__ __align__(16) uint8_t t1[96];
    __shared__ __align__(16) uint16_t t3c[12 * 512];
    fl_keys_fill_tables_cat(t1, t3c);
    __syncthreads();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const uint64_t mask = (1ull << lg) - 1;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m.n; i += stride) {
        const int l = m.level[i], sh = dom.anchor_level - l;
        uint64_t k = fl_hilbert_encode_cat(t1, t3c, (uint32_t)m.x[i] << sh, (uint32_t)m.y[i] << sh,
                                           (uint32_t)m.z[i] << sh, dom.depth);
        if (m.case_id) k |= (uint64_t)m.case_id[i] << (3 * dom.depth);
        if (k == FL_EMPTY_KEY) continue;
        uint64_t s = fl_hash_slot(k, lg);
        int p = 0;
        for (; p < kProbeLimit; ++p) {
            const unsigned long long prev = atomicCAS((unsigned long long*)(tk + 2 * s), FL_EMPTY_KEY, k);
            if (prev == FL_EMPTY_KEY || prev == k) {
                atomicMax((unsigned long long*)(tk + 2 * s + 1),
                          ((unsigned long long)(i + 1) << 32) | ((uint32_t)l << kPackedIdxBits) | (uint32_t)i);
                break;
            }
            s = (s + 1) & mask;
        }
        if (p == kProbeLimit) atomicAdd(dev_status + FL_DEVSTAT_HASH_OVERFLOW, 1u);
    }
}

// Repeated keys only, launched when a build into separate arrays met some (three launches that
// returned at once in every other build took 11 us): every input takes the maximum of its slot's
// winner (input index + 1), then each claimed slot gets its winning value.
__global__ void k_hash_dup_winners(const uint64_t* __restrict__ tk, uint32_t* __restrict__ win, int lg,
                                   const uint64_t* __restrict__ keys, size_t n) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    const uint64_t mask = (1ull << lg) - 1;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t k = keys[i];
        if (k == FL_EMPTY_KEY) continue;
        uint64_t s = fl_hash_slot(k, lg);
        for (int p = 0; p < kProbeLimit; ++p) {
            const uint64_t cur = tk[s];
            if (cur == k) {
                atomicMax(win + s, (uint32_t)(i + 1));
                break;
            }
            if (cur == FL_EMPTY_KEY) break;  // not inserted (probe overflow, reported by the insertion)
            s = (s + 1) & mask;
        }
    }
}

__global__ void k_hash_dup_values(uint32_t* __restrict__ tv, const uint32_t* __restrict__ win,
                                  const uint32_t* __restrict__ vals, uint64_t cap) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += stride) {
        const uint32_t w = win[i];
        if (w) tv[i] = vals ? vals[w - 1] : w - 1;
    }
}

__global__ void k_hash_query(const uint64_t* __restrict__ tk, const uint32_t* __restrict__ tv, int lg,
                             const uint64_t* __restrict__ q, uint32_t* __restrict__ out, size_t n) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = fl_hash_lookup(tk, tv, lg, q[i]);
}

// range[0] = the deepest leaf level, range[1] = 255 - the shallowest (both start at 0); volume (when
// given) gets the leaves' volumes in cells of level `finest`, modulo 2^64.  16 levels a load, scalar
// loads before the first and after the last 16-byte boundary: a byte per thread took 55 us for 25 M
// leaves, these 13.
__global__ void __launch_bounds__(256) k_level_range(const uint8_t* __restrict__ level, size_t n,
                                                     uint32_t* __restrict__ range, int finest,
                                                     unsigned long long* __restrict__ volume) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    const size_t head = min(n, (size_t)((16 - ((uintptr_t)level & 15)) & 15)), nv = (n - head) / 16;
    const uint4* v = (const uint4*)(level + head);
    unsigned hi4 = 0u, lo4 = 0xFFFFFFFFu;
    unsigned long long sum = 0;
    auto size = [&](unsigned l) { return 1ull << ((3 * (finest - (int)l)) & 63); };  // (deeper levels are refused)
    for (size_t i = t; i < nv; i += stride) {
        const uint4 w = __ldg(v + i);
        hi4 = __vmaxu4(__vmaxu4(hi4, __vmaxu4(w.x, w.y)), __vmaxu4(w.z, w.w));
        lo4 = __vminu4(__vminu4(lo4, __vminu4(w.x, w.y)), __vminu4(w.z, w.w));
        if (volume) {
            const unsigned ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int k = 0; k < 16; ++k) sum += size((ws[k >> 2] >> (8 * (k & 3))) & 255u);
        }
    }
    unsigned hi = 0u, lo = 255u;
    for (int k = 0; k < 32; k += 8) {
        hi = max(hi, (hi4 >> k) & 255u);
        lo = min(lo, (lo4 >> k) & 255u);
    }
    const size_t rest = n - 16 * nv;  // scalar levels: the head, then the tail
    for (size_t i = t; i < rest; i += stride) {
        const unsigned l = level[i < head ? i : i + 16 * nv];
        hi = max(hi, l);
        lo = min(lo, l);
        sum += size(l);
    }
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    if (volume)
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31) == 0) {
        if (hi > 0) atomicMax(range, hi);
        if (lo < 255u) atomicMax(range + 1, 255u - lo);
        if (volume && sum) atomicAdd(volume, sum);
    }
}

// Run start of every leaf divided by 8^cut: the anchor shifted down by cut,
// encoded at depth - cut levels, the low 3(A - l - cut) bits cleared (the case
// id above bit 3 * (depth - cut)).
//
// order (when given) gets bit 0 when some run start is smaller than the one
// before it, bit 1 when some is the same (a leaf listed twice, or overlapping
// leaves).  A warp takes a range of consecutive leaves and keeps the last of
// 32 for the next 32, so only the start of its range is encoded twice (25 M
// leaves: 107 us and a pass of 41 over the keys, 135 now).
__global__ void __launch_bounds__(256) k_run_keys(fl_mesh_dev m, fl_domain_dev dom, int cut,
                                                  const uint32_t* __restrict__ deepest, uint64_t* __restrict__ keys,
                                                  uint32_t* __restrict__ order) {
    __shared__ __align__(16) uint8_t t1[96];
    __shared__ __align__(16) uint16_t t3c[12 * 512];
    fl_keys_fill_tables_cat(t1, t3c);
    __syncthreads();
    if (cut < 0) cut = max(dom.anchor_level - (int)*deepest, 0);  // not known on the host yet
    const int dc = dom.depth - cut;
    auto key_of = [&](size_t i) {
        const int sh = dom.anchor_level - m.level[i];
        uint64_t k = fl_hilbert_encode_cat(t1, t3c, ((uint32_t)m.x[i] << sh) >> cut, ((uint32_t)m.y[i] << sh) >> cut,
                                           ((uint32_t)m.z[i] << sh) >> cut, dc);
        k &= ~((1ull << (3 * (sh - cut))) - 1);
        if (m.case_id) k |= (uint64_t)m.case_id[i] << (3 * dc);
        return k;
    };
    const int lane = threadIdx.x & 31;
    const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5), pieces = (m.n + 31) / 32;
    const size_t per = (pieces + warps - 1) / warps * 32;
    const size_t first = ((size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per;
    if (first >= m.n) return;
    const size_t end = min(first + per, m.n);
    uint64_t last = order && first ? key_of(first - 1) : 0;
    unsigned bad = 0u;
    for (size_t i0 = first; i0 < end; i0 += 32) {
        const size_t i = i0 + lane;
        const uint64_t k = i < end ? key_of(i) : ~0ull;
        if (i < end) keys[i] = k;
        if (order) {
            uint64_t before = __shfl_up_sync(0xFFFFFFFFu, k, 1);
            if (lane == 0) before = last;
            bad |= k < before ? 1u : 0u;
            bad |= k == before && i > 0 && i < end ? 2u : 0u;
            last = __shfl_sync(0xFFFFFFFFu, k, 31);
        }
    }
    bad = __reduce_or_sync(0xFFFFFFFFu, bad);
    if (bad && lane == 0) atomicOr(order, bad);  // (bad is 0 where order is not given)
}

__global__ void k_iota(uint32_t* __restrict__ ids, size_t n) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) ids[i] = (uint32_t)i;
}

// dir[b] = first run whose bucket is >= b, b in [0, nb]: run i fills the
// buckets after its predecessor's up to its own.  A wide range (a gap in the
// keys, between cases say) is filled by the whole warp, so it costs 1/32 of
// its length; the buckets after the last run's (n: none starts there), up to
// a directory's worth when the keys span less than the directory (a uniform
// mesh), by the whole grid.
__global__ void k_locator_dir(const uint64_t* __restrict__ keys, size_t n, int log2nb, uint32_t* __restrict__ dir) {
    const uint64_t nb = 1ull << log2nb;
    const uint64_t k0 = keys[0], span = keys[n - 1] - k0;
    const int bits = span ? 64 - __clzll((long long)span) : 0;
    const int shift = bits > log2nb ? bits - log2nb : 0;
    const int lane = threadIdx.x & 31;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (uint64_t b = (span >> shift) + 1 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += stride)
        dir[b] = (uint32_t)n;
    for (size_t base = (size_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const size_t i = base + lane;
        uint64_t bl = 1, bh = 0;  // empty unless i < n
        if (i < n) {
            bh = (keys[i] - k0) >> shift;
            bl = i > 0 ? ((keys[i - 1] - k0) >> shift) + 1 : 0;
        }
        // short ranges (the common case: one or two buckets) by their own lane,
        // coalesced across the warp; long ones by the whole warp
        const bool wide = bl <= bh && bh - bl >= 4;
        if (!wide)
            for (uint64_t b = bl; b <= bh; ++b) dir[b] = (uint32_t)i;
        for (unsigned w = __ballot_sync(0xFFFFFFFFu, wide); w; w &= w - 1) {
            const int j = __ffs(w) - 1;
            const uint64_t lo = __shfl_sync(0xFFFFFFFFu, bl, j), hi = __shfl_sync(0xFFFFFFFFu, bh, j);
            for (uint64_t b = lo + lane; b <= hi; b += 32) dir[b] = (uint32_t)(base + j);
        }
    }
}

// Neighbour rows in two passes over 13 directions each.  Direction k and
// 25 - k are opposite, and a same-level neighbour relation is symmetric: when
// the first pass (k < 13) finds a leaf j of cell i's own level, i is j's
// neighbour in direction 25 - k on every sub-slot, so it writes that entry of
// j's row too and marks it (bit 12 - k of marks[j]); the second pass probes
// only the unmarked directions 13..25.  Blocks of kNbrThreads: kNbrCells / S cells
// x 13 directions x S sub-slots, a cell's probes in consecutive threads; three
// blocks per SM (32 registers a thread).
constexpr int kNbrCells = 48;        // cells per block at one sub-slot
constexpr int kNbrBlocksPerSM = 3;
constexpr int kNbrThreads = kNbrCells * 13;

template <int S, bool kFirst>
__global__ void __launch_bounds__(kNbrThreads, kNbrBlocksPerSM) k_neighbours_sorted(fl_mesh_dev m, fl_domain_dev dom,
                                                                        fl_locator L, uint32_t* __restrict__ nbr,
                                                                        uint32_t* __restrict__ marks) {
    constexpr int kCells = kNbrCells / S;
    __shared__ __align__(16) uint8_t t1[96];
    __shared__ __align__(16) uint16_t t3c[12 * 512];
    fl_keys_fill_tables_cat(t1, t3c);
    __syncthreads();
    const fl_probe P = fl_probe_make(t1, t3c, L, dom);
    const int cl = threadIdx.x / (13 * S);
    const int r = threadIdx.x - cl * (13 * S);
    const int k = r / S + (kFirst ? 0 : 13), s = r % S;
    const int kk = k < 13 ? k : k + 1;
    const int dv[3] = {kk % 3 - 1, (kk / 3) % 3 - 1, kk / 9 - 1};
    for (size_t base = (size_t)blockIdx.x * kCells; base < m.n; base += (size_t)gridDim.x * kCells) {
        const size_t i = base + cl;
        if (i >= m.n) continue;
        if (!kFirst && ((marks[i] >> (k - 13)) & 1u)) continue;
        const uint16_t cs = m.case_id ? m.case_id[i] : 0;
        const fl_domain_dev::Case& d = dom.c[m.case_id ? cs : 0];
        const int lvl = m.level[i];
        const int sh = dom.anchor_level - lvl;
        const int32_t anc[3] = {m.x[i] << sh, m.y[i] << sh, m.z[i] << sh};
        const int32_t size = 1 << sh;
        int32_t p[3];
        int bit = 0;
        bool in = true;
        for (int a = 0; a < 3; ++a) {
            if (dv[a] < 0) p[a] = anc[a] - 1;
            else if (dv[a] > 0) p[a] = anc[a] + size;
            else { p[a] = anc[a] + (((s >> bit) & 1) ? (size >> 1) : 0); ++bit; }
            in = in && fl_fold32(p[a], d.ext[a] << dom.anchor_level, d.periodic[a]);
        }
        const uint32_t res =
            in ? fl_probe_point(P, m.case_id != nullptr, cs, (uint32_t)p[0], (uint32_t)p[1], (uint32_t)p[2])
               : FL_INVALID_INDEX;
        nbr[i * (26 * S) + k * S + s] = res;
        if (kFirst && res != FL_INVALID_INDEX && m.level[res] == lvl) {
            nbr[(size_t)res * (26 * S) + (25 - k) * S + s] = (uint32_t)i;
            if (s == 0) atomicOr(marks + res, 1u << (12 - k));
        }
    }
}

// Octree of a single-case mesh for point location by coordinates: a dense grid of the cells of
// level g over the domain and, below it, nodes of eight entries (child x + 2 y + 4 z).  An entry is
// a leaf (its cell index), a node (kNodeBit | node) or kNoLeaf.  A point is found by one grid load
// and a load per level below g, where a Hilbert key is four dependent table steps before its search
// starts.
constexpr uint32_t kNodeBit = 0x80000000u, kNoLeaf = 0xFFFFFFFFu;

struct Octree {
    uint32_t* grid;
    uint32_t* node;
    int4* node_at;    // per node its cell (x, y, z) and level
    uint32_t* list;   // the leaves of level g and above, in any order, and at its end those in a gap
                      // (k_octree_gaps), in any order too; nullptr: all are of level g and above
    uint32_t* state;  // [0] not usable: overlapping or outside leaves, or too many nodes;
                      // [1] nodes, [2] leaves in list, [3] leaves with an entry below the grid, [4] leaves in a gap
    uint32_t node_cap, cleared;  // nodes there is room for, and those whose entries start as kNoLeaf
    int g, D;         // the grid's and the deepest level
    int32_t dim[3];   // cells of level 0 per axis
};

__device__ __forceinline__ bool is_node(uint32_t e) { return (int32_t)e < -1; }

__device__ __forceinline__ uint32_t* grid_cell(const Octree& T, int32_t x, int32_t y, int32_t z) {
    return T.grid + ((size_t)z * (size_t)(T.dim[1] << T.g) + (size_t)y) * (size_t)(T.dim[0] << T.g) + (size_t)x;
}

__device__ __forceinline__ uint32_t* node_entry(const Octree& T, uint32_t e, int32_t x, int32_t y, int32_t z, int sh) {
    return T.node + (size_t)(e & ~kNodeBit) * 8 + (((z >> sh) & 1) * 4 + ((y >> sh) & 1) * 2 + ((x >> sh) & 1));
}

__device__ __forceinline__ bool in_domain(const Octree& T, int32_t x, int32_t y, int32_t z, int l) {
    return x >= 0 && y >= 0 && z >= 0 && x < (T.dim[0] << l) && y < (T.dim[1] << l) && z < (T.dim[2] << l);
}

__device__ __forceinline__ void clear_node(const Octree& T, uint32_t id) {
    uint4* e = reinterpret_cast<uint4*>(T.node + (size_t)id * 8);
    e[0] = e[1] = make_uint4(kNoLeaf, kNoLeaf, kNoLeaf, kNoLeaf);
}

// Exclusive prefix of v over the block in thread order (256 threads), the block's total added to
// *counter: the block's share starts at the returned base.  One atomic per block: a same-address
// atomic per warp alone took 0.3 ms for 25 M leaves.
__device__ __forceinline__ uint32_t block_claim(uint32_t v, uint32_t* counter) {
    __shared__ uint32_t s_sum[8], s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();  // the last call's sums and base are read
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t t = s_sum[w];
            s_sum[w] = run;
            run += t;
        }
        s_base = run ? atomicAdd(counter, run) : 0u;
    }
    __syncthreads();
    return s_base + s_sum[warp] + incl - v;
}

// The nodes, not linked yet: the leaf at a node's lowest corner makes it, with every node of its
// chain that has the same corner (one maker per node in a mesh that fills its domain; of a mesh with
// gaps k_octree_gaps makes the others).  Four leaves a thread, their loads in flight together, 1,024
// consecutive leaves a block.
constexpr int kLeafBatch = 4;
__global__ void __launch_bounds__(256) k_octree_nodes(fl_mesh_dev m, Octree T) {
    bool out = false;
    for (size_t i0 = (size_t)blockIdx.x * 256 * kLeafBatch; i0 < m.n; i0 += (size_t)gridDim.x * 256 * kLeafBatch) {
        int l[kLeafBatch], make[kLeafBatch];
        int32_t x[kLeafBatch], y[kLeafBatch], z[kLeafBatch];
#pragma unroll
        for (int u = 0; u < kLeafBatch; ++u) {
            const size_t i = i0 + u * 256 + threadIdx.x;
            l[u] = i < m.n ? m.level[i] : 0;
            x[u] = i < m.n ? m.x[i] : 0;
            y[u] = i < m.n ? m.y[i] : 0;
            z[u] = i < m.n ? m.z[i] : 0;
        }
        uint32_t mine = 0;
#pragma unroll
        for (int u = 0; u < kLeafBatch; ++u) {
            const int32_t low = x[u] | y[u] | z[u];
            const int chain = low ? __ffs(low) - 1 : 31;  // levels up with the same lowest corner
            const bool in = in_domain(T, x[u], y[u], z[u], l[u]);
            out = out || !in;
            make[u] = l[u] > T.g && in ? min(chain, l[u] - T.g) : 0;
            mine += (uint32_t)make[u];
        }
        uint32_t id = block_claim(mine, T.state + 1);
#pragma unroll
        for (int u = 0; u < kLeafBatch; ++u)
            for (int k = 1; k <= make[u]; ++k, ++id) {
                if (id < T.node_cap) {
                    T.node_at[id] = make_int4(x[u] >> k, y[u] >> k, z[u] >> k, l[u] - k);
                    if (id >= T.cleared) clear_node(T, id);
                } else {
                    T.state[0] = 1u;
                }
            }
    }
    if (out) T.state[0] = 1u;
}

// The nodes of level a into their entries, those of the levels between g and a in place.  Where one of
// those is missing (a gap at its lowest corner) the node stays out, and so do all below it.
__global__ void __launch_bounds__(256) k_octree_link(Octree T, int a) {
    const uint32_t stop = *T.state;
    const uint32_t n = min(T.state[1], T.node_cap), stride = gridDim.x * blockDim.x;
    for (uint32_t id = blockIdx.x * blockDim.x + threadIdx.x; id < n; id += stride) {
        const int4 c = T.node_at[id];
        if (c.w != a || stop) continue;
        uint32_t* e = grid_cell(T, c.x >> (a - T.g), c.y >> (a - T.g), c.z >> (a - T.g));
        for (int sh = a - T.g - 1; e && sh >= 0; --sh) {
            const uint32_t v = *e;
            e = is_node(v) ? node_entry(T, v, c.x, c.y, c.z, sh) : nullptr;
        }
        if (e) *e = kNodeBit | id;
    }
}

// The leaves: into their entry below or of the grid, or, for a leaf above the grid's level, into every
// grid cell it covers (a warp per leaf); those of the grid's level and above also into the list,
// unless that is every leaf (list == nullptr), and those whose node is missing at the end of it.  A
// grid cell or an entry already taken means overlapping leaves; of two leaves of one cell below the grid one is lost, which the count of the
// entries shows (k_neighbours_nodes).  The walk is a chain of L2 latencies that occupancy hides: a
// leaf a thread at 2,048 threads an SM takes 370 us for 25 M leaves (two: 439).
__global__ void __launch_bounds__(256, 8) k_octree_leaves(fl_mesh_dev m, Octree T) {
    if (*T.state) return;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    bool bad = false;
    for (size_t base = (size_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < m.n; base += stride) {
        const size_t i = base + lane;
        int sh = -128;  // levels below the grid; -128: nothing to place
        bool gap = false;
        int32_t x = 0, y = 0, z = 0;
        if (i < m.n) {
            const int l = m.level[i];
            x = m.x[i];
            y = m.y[i];
            z = m.z[i];
            if (in_domain(T, x, y, z, l)) sh = l - T.g;
            else bad = true;
        }
        if (sh >= 0) {
            uint32_t* e = grid_cell(T, x >> sh, y >> sh, z >> sh);
            if (sh == 0) {
                bad = bad || atomicExch(e, (uint32_t)i) != kNoLeaf;
            } else {
                uint32_t v = __ldcg(e);
                for (int k = sh - 1; k >= 0 && is_node(v); --k) {
                    e = node_entry(T, v, x, y, z, k);
                    v = k ? __ldcg(e) : kNoLeaf - 2u;  // the leaf's own entry: below
                }
                const bool there = v == kNoLeaf - 2u && __ldcg(e) == kNoLeaf;
                gap = v == kNoLeaf;
                if (there) *e = (uint32_t)i;
                else if (!gap) bad = true;
            }
        }
        const bool up = sh <= 0 && sh != -128;
        if (T.list) {
            const unsigned all = __ballot_sync(0xFFFFFFFFu, up);
            if (all) {
                uint32_t first = 0;
                if (lane == 0) first = atomicAdd(T.state + 2, (uint32_t)__popc(all));
                first = __shfl_sync(0xFFFFFFFFu, first, 0);
                if (up) T.list[first + (uint32_t)__popc(all & ((1u << lane) - 1u))] = (uint32_t)i;
            }
            const unsigned gaps = __ballot_sync(0xFFFFFFFFu, gap);
            if (gaps) {
                uint32_t first = 0;
                if (lane == 0) first = atomicAdd(T.state + 4, (uint32_t)__popc(gaps));
                first = __shfl_sync(0xFFFFFFFFu, first, 0);
                if (gap) T.list[m.n - 1 - first - (uint32_t)__popc(gaps & ((1u << lane) - 1u))] = (uint32_t)i;
            }
        }
        for (unsigned w = __ballot_sync(0xFFFFFFFFu, up && sh < 0); w; w &= w - 1) {
            const int j = __ffs(w) - 1;
            const int s = -__shfl_sync(0xFFFFFFFFu, sh, j), mask = (1 << s) - 1;
            const int32_t x0 = __shfl_sync(0xFFFFFFFFu, x, j) << s, y0 = __shfl_sync(0xFFFFFFFFu, y, j) << s,
                          z0 = __shfl_sync(0xFFFFFFFFu, z, j) << s;
            for (int c = lane; c < 1 << (3 * s); c += 32)
                if (atomicExch(grid_cell(T, x0 + (c & mask), y0 + ((c >> s) & mask), z0 + (c >> (2 * s))),
                               (uint32_t)(base + j)) != kNoLeaf)
                    bad = true;
        }
    }
    if (bad) T.state[0] = 1u;
}

// The leaves whose nodes are missing, a thread each: a node on the way that is not there is made and put in
// place by whoever comes first (another's is left empty).  A mesh with a gap at one node's corner was left to the
// sorted locator, after the octree's work: 18.6 M leaves, 2 % of them left out, 5,840 us (5,330 the locator
// alone), 1,870 now.  Launched only where the leaves' volume shows gaps.
__global__ void __launch_bounds__(256) k_octree_gaps(fl_mesh_dev m, Octree T) {
    const uint32_t n = T.state[4], stride = gridDim.x * blockDim.x;
    if (*T.state) return;
    bool bad = false;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
        const uint32_t i = T.list[m.n - 1 - j];
        const int l = m.level[i];
        const int32_t x = m.x[i], y = m.y[i], z = m.z[i];
        uint32_t* e = grid_cell(T, x >> (l - T.g), y >> (l - T.g), z >> (l - T.g));
        int k = l - T.g - 1;
        for (; k >= 0; --k) {
            uint32_t v = __ldcg(e);
            if (v == kNoLeaf) {
                const uint32_t id = atomicAdd(T.state + 1, 1u);
                if (id >= T.node_cap) break;
                T.node_at[id] = make_int4(x >> (k + 1), y >> (k + 1), z >> (k + 1), l - k - 1);
                clear_node(T, id);
                __threadfence();
                v = atomicCAS(e, kNoLeaf, kNodeBit | id);
                if (v == kNoLeaf) v = kNodeBit | id;
            }
            if (!is_node(v)) break;  // a leaf: this one lies in it
            e = node_entry(T, v, x, y, z, k);
        }
        if (k >= 0 || atomicCAS(e, kNoLeaf, i) != kNoLeaf) bad = true;
    }
    if (bad) T.state[0] = 1u;
}

// Entry r = k S + s of a row: the probe point of direction k at sub-slot s.
struct RowProbe {
    int dv[3], half[3];
};
template <int S>
__device__ __forceinline__ RowProbe row_probe(int r) {
    RowProbe P;
    const int k = r / S, s = r % S, kk = k < 13 ? k : k + 1;
    P.dv[0] = kk % 3 - 1;
    P.dv[1] = (kk / 3) % 3 - 1;
    P.dv[2] = kk / 9 - 1;
    int bit = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) P.half[a] = P.dv[a] == 0 ? (s >> bit++) & 1 : 0;
    return P;
}

// Rows of the leaves below the grid, a warp per node.  Lanes 0-26 locate the node's cell and the 26
// of its size around it; every entry of its leaf children's rows is then the entry of one of these
// 27 -- a leaf for all of its children, or a child of that node by one load -- so a leaf's 26
// entries take 27 / 8 searches instead of 26, and neighbouring lanes write a row.  Latency bound (a
// node's chain: its cell, grid, nodes, entries), so the loads of kFlight rounds of entries are in
// flight together.  T.state[3] counts the leaves that have an entry.  25 M leaves: 869 us (1,324 us
// with one round in flight), 1.43 ms with the octree and the rows of the grid's level, against
// 4.51 ms for the sorted locator and its two passes of 13 searches a leaf.
template <int S>
__global__ void __launch_bounds__(256, 6) k_neighbours_nodes(fl_domain_dev dom, Octree T, uint32_t* __restrict__ nbr) {
    // per row entry of the eight children: the cell the probe point lies in (0-26), its child there,
    // for finer cells the bits of the point below the leaf's size (dv < 0: the last, else the first; a
    // half offset at dv = 0), the leaf's child place and the entry in its row
    constexpr int kEntries = 8 * 26 * S, kRounds = (kEntries + 31) / 32, kFlight = S == 1 ? kRounds : 9;
    __shared__ uint32_t s_plan[kRounds * 32];
    if (*T.state) return;  // no usable octree: the caller takes the sorted locator
    for (int e = threadIdx.x; e < kRounds * 32; e += blockDim.x) {
        const int c = e / (26 * S), r = e - c * (26 * S);
        const RowProbe P = row_probe<S>(r);
        int cell = 0, child = 0, first = 0, rest = 0, m3 = 1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int q = ((c >> a) & 1) + P.dv[a];
            cell += (q < 0 ? 0 : (q > 1 ? 2 : 1)) * m3;
            child |= (q & 1) << a;
            first |= (P.dv[a] < 0 ? 1 : P.half[a]) << a;
            rest |= (P.dv[a] < 0 ? 1 : 0) << a;
            m3 *= 3;
        }
        // past the last entry: lane 31 holds no child
        s_plan[e] = e < kEntries ? (uint32_t)(cell | child << 5 | first << 8 | rest << 11 | c << 14 | r << 19) : 31u << 14;
    }
    __syncthreads();
    const fl_domain_dev::Case d = dom.c[0];
    const int lane = threadIdx.x & 31;
    const int dv[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
    const uint32_t n = T.state[1], warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t* __restrict__ node = T.node;
    uint32_t leaves = 0;
    for (uint32_t id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; id < n; id += warps) {
        const int4 at = __ldg(T.node_at + id);
        const uint32_t own = lane < 8 ? __ldg(node + ((id << 3) | lane)) : kNoLeaf;
        const unsigned leaf8 = __ballot_sync(0xFFFFFFFFu, !is_node(own) && own != kNoLeaf);
        if (!leaf8) continue;
        leaves += (uint32_t)__popc(leaf8);
        uint32_t cell = kNoLeaf;
        if (lane < 27) {
            int32_t p[3] = {at.x + dv[0], at.y + dv[1], at.z + dv[2]};
            bool in = true;
#pragma unroll
            for (int a = 0; a < 3; ++a)
                if ((uint32_t)p[a] >= (uint32_t)(T.dim[a] << at.w)) in = in && fl_fold32(p[a], T.dim[a] << at.w, d.periodic[a]);
            if (in) {
                const int up = at.w - T.g;
                cell = __ldg(grid_cell(T, p[0] >> up, p[1] >> up, p[2] >> up));
                for (int sh = up - 1; sh >= 0 && is_node(cell); --sh)
                    cell = __ldg(node_entry(T, cell, p[0], p[1], p[2], sh));
            }
        }
#pragma unroll 1
        for (int t0 = 0; t0 < kRounds; t0 += kFlight) {
            uint32_t v[kFlight];
#pragma unroll
            for (int f = 0; f < kFlight; ++f) {  // every lane stays for the shuffles
                const uint32_t w = t0 + f < kRounds ? s_plan[(t0 + f) * 32 + lane] : 31u << 14;
                v[f] = __shfl_sync(0xFFFFFFFFu, cell, (int)(w & 31u));
                if (is_node(v[f])) v[f] = __ldg(node + ((v[f] << 3) | ((w >> 5) & 7u)));  // the node bit is shifted out
            }
#pragma unroll
            for (int f = 0; f < kFlight; ++f) {
                const uint32_t w = t0 + f < kRounds ? s_plan[(t0 + f) * 32 + lane] : 31u << 14;
                if (is_node(v[f])) {  // finer than the leaf
                    v[f] = __ldg(node + ((v[f] << 3) | ((w >> 8) & 7u)));
                    while (is_node(v[f])) v[f] = __ldg(node + ((v[f] << 3) | ((w >> 11) & 7u)));
                }
                const uint32_t i = __shfl_sync(0xFFFFFFFFu, own, (int)((w >> 14) & 31u));
                if (!is_node(i) && i != kNoLeaf) nbr[(size_t)i * (26 * S) + (w >> 19)] = v[f];
            }
        }
    }
    if (lane == 0 && leaves) atomicAdd(T.state + 3, leaves);
}

// Rows of the leaves of the grid's level and above, a thread per entry: the probe point located from
// the grid down.
constexpr int kRowCells = 24;  // leaves per block at one sub-slot
template <int S>
__global__ void __launch_bounds__(kRowCells * 26) k_neighbours_grid(fl_mesh_dev m, fl_domain_dev dom, Octree T,
                                                                    uint32_t* __restrict__ nbr) {
    if (*T.state) return;
    constexpr int kCells = kRowCells / S;
    const int cl = threadIdx.x / (26 * S);
    const int r = threadIdx.x - cl * (26 * S);
    const RowProbe P = row_probe<S>(r);
    const fl_domain_dev::Case d = dom.c[0];
    const uint32_t n = T.list ? T.state[2] : (uint32_t)m.n;
    for (uint32_t base = blockIdx.x * kCells; base < n; base += gridDim.x * kCells) {
        const uint32_t j = base + cl;
        if (j >= n) continue;
        const uint32_t i = T.list ? __ldg(T.list + j) : j;
        const int sh = T.D - m.level[i];
        const int32_t size = 1 << sh, mid = size >> 1;
        int32_t p[3] = {m.x[i] << sh, m.y[i] << sh, m.z[i] << sh};
        bool in = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            p[a] += P.dv[a] < 0 ? -1 : (P.dv[a] > 0 ? size : (P.half[a] ? mid : 0));
            if ((uint32_t)p[a] >= (uint32_t)(T.dim[a] << T.D)) in = in && fl_fold32(p[a], T.dim[a] << T.D, d.periodic[a]);
        }
        uint32_t e = kNoLeaf;
        if (in) {
            int b = T.D - T.g;
            e = __ldg(grid_cell(T, p[0] >> b, p[1] >> b, p[2] >> b));
            while (is_node(e)) {
                --b;
                e = __ldg(node_entry(T, e, p[0], p[1], p[2], b));
            }
        }
        nbr[(size_t)i * (26 * S) + r] = e;
    }
}

int locator_log2nb(size_t n) {
    int lg = 0;
    while ((1ull << lg) < n) ++lg;
    return lg > 11 ? lg + 1 : 10;  // about two buckets per run: most searches end in the directory
}

}  // namespace

size_t fl_locator_scratch_bytes(size_t n) {
    const size_t nb = (size_t)1 << locator_log2nb(n);
    return fl_align256(n * 8) + fl_align256(n * 4) + fl_align256((nb + 1) * 4) + 256 + fl_sort_scratch_bytes(n, 8);
}

int fl_locator_build(fl_ctx* ctx, const fl_mesh_dev& m, const fl_domain_dev& dom, void* scratch, fl_locator* L,
                     int level_bound, bool in_key_order, bool probed) {
    const size_t n = m.n;
    const int log2nb = locator_log2nb(n);
    char* p = (char*)scratch;
    uint64_t* keys = (uint64_t*)p; p += fl_align256(n * 8);
    uint32_t* ids = (uint32_t*)p; p += fl_align256(n * 4);
    uint32_t* dir = (uint32_t*)p; p += fl_align256((((size_t)1 << log2nb) + 1) * 4);
    uint32_t* flag = (uint32_t*)p; p += 256;
    *L = fl_locator{keys, nullptr, dir, m.level, n, log2nb, 0};
    if (n == 0) return FL_OK;
    FL_TRY_CUDA(ctx, cudaMemsetAsync(flag, 0, 12, ctx->stream), "locator");
    uint32_t hf[2] = {0, (uint32_t)std::max(level_bound, 0)};  // order (k_run_keys), deepest level
    if (level_bound < 0) {
        k_level_range<<<fl_blocks((n + 15) / 16, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(m.level, n, flag + 1, 0,
                                                                                                  nullptr);
        FL_CHECK_LAUNCH(ctx, "k_level_range");
    }
    const int bound_cut = level_bound < 0 ? -1 : std::max(dom.anchor_level - level_bound, 0);
    k_run_keys<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(m, dom, bound_cut, flag + 1, keys,
                                                                                 in_key_order ? nullptr : flag);
    FL_CHECK_LAUNCH(ctx, "k_run_keys");
    if (!in_key_order || level_bound < 0) {  // one wait for both
        const int rc = fl_read_back(ctx, hf, flag, level_bound < 0 ? 8 : 4, "locator");
        if (rc) return rc;
    }
    L->cut = std::max(dom.anchor_level - (int)hf[1], 0);
    // Stable: equal run starts keep mesh order, so the last of them is found.  A mesh in key order that
    // has some gets ids too, its own order: octets are not consecutive there, and want the search.
    if (hf[0]) {
        k_iota<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(ids, n);
        FL_CHECK_LAUNCH(ctx, "k_iota");
        if (hf[0] & 1u) {
            // the keys hold 3 (depth - cut) bits, plus 16 for case ids
            const int end_bit = std::min(64, 3 * (dom.depth - L->cut) + (m.case_id ? 16 : 0));
            int rc = fl_sort_pairs_with(ctx, keys, ids, n, 0, end_bit, p);
            if (rc) return rc;
        }
        L->ids = ids;
    }
    if (!probed && !L->ids) return FL_OK;  // octets in key order are found without a search
    k_locator_dir<<<fl_blocks(n + 1, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(keys, n, log2nb, dir);
    FL_CHECK_LAUNCH(ctx, "k_locator_dir");
    return FL_OK;
}

int fl_neighbours_sorted(fl_ctx* ctx, const fl_mesh_dev& m, const fl_domain_dev& dom, const fl_locator& L,
                         int subslots, uint32_t* nbr, uint32_t* marks) {
    if (m.n == 0) return FL_OK;
    FL_TRY_CUDA(ctx, cudaMemsetAsync(marks, 0, m.n * 4, ctx->stream), "neighbour marks");
    const size_t cells = (size_t)(kNbrCells / subslots);
    const unsigned grid =
        (unsigned)std::min<size_t>((m.n + cells - 1) / cells, (size_t)ctx->num_sms * kNbrBlocksPerSM);
    if (subslots == 4) {
        k_neighbours_sorted<4, true><<<grid, kNbrThreads, 0, ctx->stream>>>(m, dom, L, nbr, marks);
        FL_CHECK_LAUNCH(ctx, "k_neighbours_sorted");
        k_neighbours_sorted<4, false><<<grid, kNbrThreads, 0, ctx->stream>>>(m, dom, L, nbr, marks);
    } else {
        k_neighbours_sorted<1, true><<<grid, kNbrThreads, 0, ctx->stream>>>(m, dom, L, nbr, marks);
        FL_CHECK_LAUNCH(ctx, "k_neighbours_sorted");
        k_neighbours_sorted<1, false><<<grid, kNbrThreads, 0, ctx->stream>>>(m, dom, L, nbr, marks);
    }
    FL_CHECK_LAUNCH(ctx, "k_neighbours_sorted");
    return FL_OK;
}

// The octree's grid has at most two cells per leaf: its level g is the deepest that fits, at most
// kGridFill levels below the shallowest leaf (a leaf above the grid fills 8^(g - level) cells).
constexpr int kGridFill = 4;
constexpr int kMostNodeLevels = 8;  // below the grid: a pass over the nodes and a load per search each

static size_t octree_most_cells(size_t n) { return std::max<size_t>(2 * n, 64); }
// A mesh that fills its domain has at most n / 7 nodes below the grid; with gaps there are more to a leaf.
static size_t octree_most_nodes(size_t n) { return n / 4 + 8; }

size_t fl_neighbours_octree_scratch(size_t n) {
    return 256 + fl_align256(octree_most_cells(n) * 4) + fl_align256(octree_most_nodes(n) * 32) +
           fl_align256(octree_most_nodes(n) * 16) + fl_align256(n * 4);
}

int fl_neighbours_octree(fl_ctx* ctx, const fl_mesh_dev& m, const fl_domain_dev& dom, const int32_t* ext, int subslots,
                         void* scratch, uint32_t* nbr, bool* done, int* deepest) {
    *done = false;
    *deepest = -1;
    const size_t n = m.n, most = octree_most_cells(n);
    if (m.case_id || n >= kNodeBit) return FL_OK;  // so nodes * 8 stays below 2^32
    Octree T{};
    char* p = (char*)scratch;
    T.node_cap = (uint32_t)octree_most_nodes(n);
    T.cleared = (uint32_t)(n / 7 + 1);
    T.state = (uint32_t*)p; p += 256;
    T.grid = (uint32_t*)p; p += fl_align256(most * 4) + fl_align256((size_t)T.node_cap * 32);
    T.node_at = (int4*)p; p += fl_align256((size_t)T.node_cap * 16);
    T.list = (uint32_t*)p;
    struct { uint32_t deepest, above, volume[2]; } h;  // k_level_range's
    uint32_t* range = T.state + 8;
    FL_TRY_CUDA(ctx, cudaMemsetAsync(T.state, 0, 64, ctx->stream), "octree state");
    k_level_range<<<fl_blocks((n + 15) / 16, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
        m.level, n, range, dom.anchor_level, (unsigned long long*)(range + 2));
    FL_CHECK_LAUNCH(ctx, "k_level_range");
    int rc = fl_read_back(ctx, &h, range, sizeof(h), "level range");
    if (rc) return rc;
    *deepest = T.D = (int)h.deepest;
    const int lowest = 255 - (int)h.above;
    size_t cells = 1;
    uint64_t domain = 1ull << (3 * dom.anchor_level);  // its volume: at most 2^63, as ext << anchor_level is at most 2^21
    for (int a = 0; a < 3; ++a) {
        T.dim[a] = ext[a];
        cells = cells > most ? cells : cells * (size_t)ext[a];
        domain *= (uint64_t)ext[a];
    }
    if (T.D > dom.anchor_level || T.D > dom.max_level || cells > most) return FL_OK;
    // more than the domain holds: overlapping or outside leaves, found here before any work; less: gaps
    const uint64_t volume = (uint64_t)h.volume[1] << 32 | h.volume[0];
    if (volume > domain) return FL_OK;
    while (T.g < T.D && T.g < lowest + kGridFill && cells * 8 <= most) {
        ++T.g;
        cells *= 8;
    }
    if (T.D - T.g > kMostNodeLevels) return FL_OK;
    T.node = T.grid + fl_align256(cells * 4) / 4;  // behind the cells in use: one clear for both
    FL_TRY_CUDA(ctx, cudaMemsetAsync(T.grid, 0xFF, fl_align256(cells * 4) + (T.D > T.g ? (size_t)T.cleared * 32 : 0),
                                     ctx->stream), "octree entries");
    const unsigned nb = fl_blocks((n + kLeafBatch - 1) / kLeafBatch, 256, ctx->num_sms * 8);
    if (T.D > T.g) {
        k_octree_nodes<<<nb, 256, 0, ctx->stream>>>(m, T);
        FL_CHECK_LAUNCH(ctx, "k_octree_nodes");
        for (int a = T.g; a < T.D; ++a) {
            k_octree_link<<<fl_blocks(T.cleared, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(T, a);
            FL_CHECK_LAUNCH(ctx, "k_octree_link");
        }
    }
    if (T.D == T.g) T.list = nullptr;
    k_octree_leaves<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(m, T);
    FL_CHECK_LAUNCH(ctx, "k_octree_leaves");
    if (T.D > T.g && volume < domain) {
        k_octree_gaps<<<fl_blocks(n, 256, ctx->num_sms * 4), 256, 0, ctx->stream>>>(m, T);
        FL_CHECK_LAUNCH(ctx, "k_octree_gaps");
    }
    const size_t per_block = (size_t)(kRowCells / subslots);
    const unsigned rows = (unsigned)std::min<size_t>((n + per_block - 1) / per_block, (size_t)ctx->num_sms * 6);
    if (subslots == 4) k_neighbours_grid<4><<<rows, kRowCells * 26, 0, ctx->stream>>>(m, dom, T, nbr);
    else k_neighbours_grid<1><<<rows, kRowCells * 26, 0, ctx->stream>>>(m, dom, T, nbr);
    FL_CHECK_LAUNCH(ctx, "k_neighbours_grid");
    if (T.D > T.g) {
        const unsigned wb = fl_blocks((size_t)T.cleared * 32, 256, ctx->num_sms * 16);
        if (subslots == 4) k_neighbours_nodes<4><<<wb, 256, 0, ctx->stream>>>(dom, T, nbr);
        else k_neighbours_nodes<1><<<wb, 256, 0, ctx->stream>>>(dom, T, nbr);
        FL_CHECK_LAUNCH(ctx, "k_neighbours_nodes");
    }
    uint32_t st[4];
    rc = fl_read_enqueue(ctx, 0, T.state, sizeof(st), "octree state");
    if (rc) return rc;
    rc = fl_collect_device_status(ctx, "fl_neighbour_rebuild");  // waits for both reads
    if (rc) return rc;
    std::memcpy(st, ctx->host_read, sizeof(st));
    *done = !st[0] && (!T.list || (size_t)st[2] + st[3] == n);
    return FL_OK;
}

int fl_hash_lg(uint64_t cap) {
    int lg = 0;
    while ((1ull << lg) < cap) ++lg;
    return lg;
}

int fl_hash_build_cells(fl_ctx* ctx, uint64_t* tk, uint64_t cap, const fl_mesh_dev& m, const fl_domain_dev& dom) {
    if (m.n >= ((size_t)1 << kPackedIdxBits)) return fl_set_error(ctx, FL_E_CAPACITY, "a mesh of 2^27 or more cells");
    k_hash_clear<<<fl_blocks(cap, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(tk, nullptr, cap);
    FL_CHECK_LAUNCH(ctx, "k_hash_clear");
    if (m.n == 0) return FL_OK;
    k_hash_insert_cells<<<fl_blocks(m.n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(tk, fl_hash_lg(cap), m, dom,
                                                                                       ctx->dev_status);
    FL_CHECK_LAUNCH(ctx, "k_hash_insert_cells");
    return FL_OK;
}

uint64_t fl_table_capacity(size_t n) {
    uint64_t c = 1024;
    while (c < 2 * (uint64_t)n) c <<= 1;
    return c;
}

extern "C" {

uint64_t fl_hash_compute_capacity(size_t n) {
    // HashTableManager::computeCapacity (HashTableManager.cpp:47-57)
    double minc = (double)n / 0.6f;
    uint32_t lg = 0;
    while (n && (double)(1ull << lg) < minc) ++lg;
    if (lg < 20) lg = 20;
    if (lg > 30) lg = 30;
    return 1ull << lg;
}

int fl_hash_build(fl_ctx* ctx, uint64_t* table_keys, uint32_t* table_vals, uint64_t capacity, const uint64_t* keys,
                  const uint32_t* vals, size_t n) {
    if (!ctx) return FL_E_INVALID_ARG;
    if (!table_keys || !table_vals || capacity == 0 || (capacity & (capacity - 1)) || (n && !keys))
        return fl_set_error(ctx, FL_E_INVALID_ARG, "fl_hash_build: bad table or capacity not a power of two");
    if (n > capacity) return fl_set_error(ctx, FL_E_CAPACITY, "fl_hash_build: more keys than slots");
    const bool index = !vals && n < (1ull << 31);  // as int
    if (!index)
        FL_TRY_CUDA(ctx, cudaMemsetAsync(ctx->dev_status + FL_DEVSTAT_HASH_DUPS, 0, 4, ctx->stream), "hash flag");
    k_hash_clear<<<fl_blocks(capacity, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(table_keys, table_vals, capacity);
    FL_CHECK_LAUNCH(ctx, "k_hash_clear");
    if (n) {
        (index ? k_hash_insert<true> : k_hash_insert<false>)<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
            table_keys, table_vals, fl_hash_lg(capacity), keys, vals, n, ctx->dev_status);
        FL_CHECK_LAUNCH(ctx, "k_hash_insert");
    }
    int rc = fl_collect_device_status(ctx, "fl_hash_build");
    if (rc || index || !ctx->host_status[FL_DEVSTAT_HASH_DUPS]) return rc;
    // repeated keys: the winner of each slot in a second round
    rc = fl_scratch_reserve(ctx, capacity * 4);
    if (rc) return rc;
    uint32_t* win = (uint32_t*)ctx->scratch;
    FL_TRY_CUDA(ctx, cudaMemsetAsync(win, 0, capacity * 4, ctx->stream), "hash winners");
    k_hash_dup_winners<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(table_keys, win,
                                                                                    fl_hash_lg(capacity), keys, n);
    FL_CHECK_LAUNCH(ctx, "k_hash_dup_winners");
    k_hash_dup_values<<<fl_blocks(capacity, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(table_vals, win, vals, capacity);
    FL_CHECK_LAUNCH(ctx, "k_hash_dup_values");
    FL_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "fl_hash_build");  // neither pass has a status to report
    return FL_OK;
}

int fl_hash_query(fl_ctx* ctx, const uint64_t* table_keys, const uint32_t* table_vals, uint64_t capacity,
                  const uint64_t* queries, uint32_t* out, size_t n) {
    if (!ctx) return FL_E_INVALID_ARG;
    if (n == 0) return FL_OK;
    if (!table_keys || !table_vals || !queries || !out || capacity == 0 || (capacity & (capacity - 1)))
        return fl_set_error(ctx, FL_E_INVALID_ARG, "fl_hash_query: bad arguments");
    k_hash_query<<<fl_blocks(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(table_keys, table_vals,
                                                                             fl_hash_lg(capacity), queries, out, n);
    FL_CHECK_LAUNCH(ctx, "k_hash_query");
    return FL_OK;
}

}  // extern "C"
