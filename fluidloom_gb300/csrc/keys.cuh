// keys.cuh — device-side key codec pieces shared by the kernels that need keys.
// The 12-state table values are the reference's (src/core/hilbert/HilbertCodec.cpp:13-42);
// bit-exact keys require them.
#pragma once
#include "common.cuh"

constexpr uint8_t kHilbertEnc[12][8] = {
    {8, 17, 27, 18, 47, 38, 28, 37},   {16, 71, 1, 62, 51, 52, 2, 61},
    {0, 75, 95, 76, 9, 10, 86, 85},    {4, 77, 55, 78, 3, 66, 80, 65},
    {50, 49, 45, 46, 67, 88, 68, 7},   {6, 57, 39, 72, 5, 58, 84, 83},
    {12, 11, 29, 90, 79, 32, 30, 89},  {74, 91, 73, 40, 69, 92, 70, 15},
    {14, 13, 81, 82, 63, 36, 24, 35},  {20, 31, 19, 56, 53, 54, 42, 41},
    {26, 93, 43, 44, 25, 94, 64, 23},  {22, 87, 21, 60, 33, 48, 34, 59},
};
constexpr uint8_t kHilbertDec[12][8] = {
    {8, 17, 19, 26, 30, 39, 37, 44},   {16, 2, 6, 52, 53, 63, 59, 65},
    {0, 12, 13, 73, 75, 87, 86, 90},   {86, 71, 69, 4, 0, 73, 75, 50},
    {93, 49, 48, 68, 70, 42, 43, 7},   {75, 57, 61, 87, 86, 4, 0, 34},
    {37, 95, 91, 9, 8, 26, 30, 76},    {43, 74, 72, 89, 93, 68, 70, 15},
    {30, 82, 83, 39, 37, 9, 8, 60},    {59, 47, 46, 18, 16, 52, 53, 25},
    {70, 28, 24, 42, 43, 89, 93, 23},  {53, 36, 38, 63, 59, 18, 16, 81},
};

// The tables the key kernels keep in shared memory, worked out by the compiler: t1[s*8+q] (one
// level) and t3[s*512+w] where w holds three levels of input (MSB level first): interleaved, 3 bits
// a level (kCat false), or as concatenated coordinate bits x3 << 6 | y3 << 3 | z3 (kCat true), so an
// encoder reads each 9-bit step straight from the coordinates.
struct alignas(16) fl_key_tables {
    uint16_t t3[12 * 512];
    uint8_t t1[96];
};

constexpr fl_key_tables fl_make_key_tables(const uint8_t (&step)[12][8], bool cat) {
    fl_key_tables T{};
    for (int i = 0; i < 96; ++i) T.t1[i] = step[i >> 3][i & 7];
    for (int i = 0; i < 12 * 512; ++i) {
        unsigned s = (unsigned)i >> 9, out = 0;
        for (int k = 2; k >= 0; --k) {
            const unsigned q = cat ? ((((unsigned)i >> k) & 1u) << 2) | ((((unsigned)i >> (3 + k)) & 1u) << 1) |
                                         (((unsigned)i >> (6 + k)) & 1u)
                                   : ((unsigned)i >> (3 * k)) & 7u;
            const unsigned v = step[s][q];
            out = (out << 3) | (v & 7u);
            s = v >> 3;
        }
        T.t3[i] = (uint16_t)((s << 9) | out);
    }
    return T;
}

static __device__ const fl_key_tables g_enc_tables = fl_make_key_tables(kHilbertEnc, false);
static __device__ const fl_key_tables g_dec_tables = fl_make_key_tables(kHilbertDec, false);
static __device__ const fl_key_tables g_enc_tables_cat = fl_make_key_tables(kHilbertEnc, true);

// Fill a block's shared tables (every thread of the block, a __syncthreads before their use; t1 and
// t3 16-byte aligned): 774 16-byte copies from L2.  Working the three-level table out in each block
// instead, three dependent lookups an entry, put 2 us before every key kernel's first cell (67,000 leaves:
// k_run_keys 5.1 -> 2.9 us, k_cell_keys 5.2 -> 3.0, neighbour passes 18.6 + 13.7 -> 14.5 + 9.7).
static __device__ __forceinline__ void fl_keys_copy_tables(const fl_key_tables& g, uint8_t* t1, uint16_t* t3) {
    const uint4* src3 = reinterpret_cast<const uint4*>(g.t3);
    const uint4* src1 = reinterpret_cast<const uint4*>(g.t1);
    for (int i = threadIdx.x; i < 768; i += blockDim.x) reinterpret_cast<uint4*>(t3)[i] = __ldg(src3 + i);
    for (int i = threadIdx.x; i < 6; i += blockDim.x) reinterpret_cast<uint4*>(t1)[i] = __ldg(src1 + i);
}
static __device__ __forceinline__ void fl_keys_fill_tables(uint8_t* t1, uint16_t* t3, bool decode) {
    fl_keys_copy_tables(decode ? g_dec_tables : g_enc_tables, t1, t3);
}
static __device__ __forceinline__ void fl_keys_fill_tables_cat(uint8_t* t1, uint16_t* t3c) {
    fl_keys_copy_tables(g_enc_tables_cat, t1, t3c);
}

// hilbert::encode of the low `level` bits of x, y, z with the re-indexed table
// (same keys as fl_hilbert_encode_dev).
static __device__ __forceinline__ uint64_t fl_hilbert_encode_cat(const uint8_t* t1, const uint16_t* t3c, uint32_t x,
                                                                 uint32_t y, uint32_t z, int level) {
    uint64_t h = 0;
    unsigned s = 0;
    int i = level;
    for (int k = 0; k < level % 3; ++k) {  // leading single levels
        --i;
        unsigned q = (((z >> i) & 1u) << 2) | (((y >> i) & 1u) << 1) | ((x >> i) & 1u);
        unsigned v = t1[s * 8 + q];
        h = (h << 3) | (v & 7u);
        s = v >> 3;
    }
    while (i > 0) {
        i -= 3;
        unsigned c = (((x >> i) & 7u) << 6) | (((y >> i) & 7u) << 3) | ((z >> i) & 7u);
        unsigned v = t3c[s * 512 + c];
        h = (h << 9) | (v & 511u);
        s = v >> 9;
    }
    return h;
}

// Encoder state after the low `level` bits of x, y, z (most significant
// first): the digit of child (c & 1, c >> 1 & 1, c >> 2) of the cell (x, y, z)
// is then t1[state * 8 + c] & 7.
static __device__ __forceinline__ unsigned fl_hilbert_state_cat(const uint8_t* t1, const uint16_t* t3c, uint32_t x,
                                                                uint32_t y, uint32_t z, int level) {
    unsigned s = 0;
    int i = level;
    for (int k = 0; k < level % 3; ++k) {
        --i;
        s = t1[s * 8 + ((((z >> i) & 1u) << 2) | (((y >> i) & 1u) << 1) | ((x >> i) & 1u))] >> 3;
    }
    while (i > 0) {
        i -= 3;
        s = t3c[s * 512 + ((((x >> i) & 7u) << 6) | (((y >> i) & 7u) << 3) | ((z >> i) & 7u))] >> 9;
    }
    return s;
}

// Interleave up to 21 bits of three coordinates: bit i of x -> 3i, y -> 3i+1, z -> 3i+2.
static __device__ __forceinline__ uint64_t interleave3(uint32_t x, uint32_t y, uint32_t z) {
    auto sp = [](uint64_t v) {
        v &= 0x1FFFFFull;
        v = (v | (v << 32)) & 0x1F00000000FFFFull;
        v = (v | (v << 16)) & 0x1F0000FF0000FFull;
        v = (v | (v << 8)) & 0x100F00F00F00F00Full;
        v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
        v = (v | (v << 2)) & 0x1249249249249249ull;
        return v;
    };
    return sp(x) | (sp(y) << 1) | (sp(z) << 2);
}

static __device__ __forceinline__ uint32_t compact3(uint64_t v) {
    v &= 0x1249249249249249ull;
    v = (v ^ (v >> 2)) & 0x10C30C30C30C30C3ull;
    v = (v ^ (v >> 4)) & 0x100F00F00F00F00Full;
    v = (v ^ (v >> 8)) & 0x1F0000FF0000FFull;
    v = (v ^ (v >> 16)) & 0x1F00000000FFFFull;
    v = (v ^ (v >> 32)) & 0x1FFFFFull;
    return (uint32_t)v;
}

// hilbert::encode semantics (HilbertCodec.cpp:44-80) using the shared tables.
static __device__ __forceinline__ uint64_t fl_hilbert_encode_dev(const uint8_t* t1, const uint16_t* t3, uint32_t x, uint32_t y,
                                          uint32_t z, int level) {
    const uint32_t m = (1u << 21) - 1;
    uint64_t w = interleave3(x & m, y & m, z & m);  // 3-bit quadrant (z<<2|y<<1|x) per level
    uint64_t h = 0;
    unsigned s = 0;
    int i = level;
    int r = level % 3;
    for (int k = 0; k < r; ++k) {  // leading single levels
        --i;
        unsigned q = (unsigned)(w >> (3 * i)) & 7u;
        unsigned v = t1[s * 8 + q];
        h = (h << 3) | (v & 7u);
        s = v >> 3;
    }
    while (i > 0) {
        i -= 3;
        unsigned q = (unsigned)(w >> (3 * i)) & 511u;
        unsigned v = t3[s * 512 + q];
        h = (h << 9) | (v & 511u);
        s = v >> 9;
    }
    unsigned shift = (unsigned)(uint8_t)(64 - level * 3);
    if (shift < 64) { h <<= shift; h >>= shift; }
    return h;
}


int fl_launch_cell_keys(fl_ctx* ctx, const int32_t* x, const int32_t* y, const int32_t* z, const uint8_t* level,
                        const uint16_t* cs, int depth, int anchor_level, uint64_t* keys, size_t n);
