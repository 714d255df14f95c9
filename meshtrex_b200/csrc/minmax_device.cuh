// Device bodies of the leaf min/max pass (meshtrex: minMaxLeaf.comp.glsl:31-128),
// shared by the single-volume kernels (minmax.cu) and the batched kernel
// (batched.cu).
//
// A warp owns a 32 x 16-byte strip of voxel rows for one block row (by) and a
// run of block slabs (bz): per z slice it loads the B+1 rows of its strip with
// 16-byte vector loads, folds them with packed SIMD min/max, reduces each
// block's B+1 columns (the +1 halo column comes from the next lane by
// shuffle), and folds the slice into the running block of its z run.  The
// slice at z = (bz+1)*B is the halo of block bz and the first slice of bz+1,
// so it is loaded once.
#pragma once

#include <algorithm>

#include "mtx_internal.h"

namespace mtx {

// ---------------------------------------------------- packed 16-byte lanes
template <typename T> struct Lane16;

template <> struct Lane16<uint8_t> {
    static constexpr int V = 16;
    __device__ __forceinline__ static uint4 lo_id() { return make_uint4(~0u, ~0u, ~0u, ~0u); }
    __device__ __forceinline__ static uint4 hi_id() { return make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ static void fold(uint4 &mn, uint4 &mx, uint4 v) {
        mn.x = __vminu4(mn.x, v.x); mn.y = __vminu4(mn.y, v.y); mn.z = __vminu4(mn.z, v.z); mn.w = __vminu4(mn.w, v.w);
        mx.x = __vmaxu4(mx.x, v.x); mx.y = __vmaxu4(mx.y, v.y); mx.z = __vmaxu4(mx.z, v.z); mx.w = __vmaxu4(mx.w, v.w);
    }
    __device__ __forceinline__ static void merge(uint4 &mn, uint4 &mx, const uint4 &mn2, const uint4 &mx2) {
        mn.x = __vminu4(mn.x, mn2.x); mn.y = __vminu4(mn.y, mn2.y); mn.z = __vminu4(mn.z, mn2.z); mn.w = __vminu4(mn.w, mn2.w);
        mx.x = __vmaxu4(mx.x, mx2.x); mx.y = __vmaxu4(mx.y, mx2.y); mx.z = __vmaxu4(mx.z, mx2.z); mx.w = __vmaxu4(mx.w, mx2.w);
    }
    __device__ __forceinline__ static uint32_t elem(const uint4 &w, int i, bool is_max) {
        uint32_t word = (i >> 2) == 0 ? w.x : (i >> 2) == 1 ? w.y : (i >> 2) == 2 ? w.z : w.w;
        return (word >> (8 * (i & 3))) & 0xFFu;
    }
};

template <> struct Lane16<uint16_t> {
    static constexpr int V = 8;
    __device__ __forceinline__ static uint4 lo_id() { return make_uint4(~0u, ~0u, ~0u, ~0u); }
    __device__ __forceinline__ static uint4 hi_id() { return make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ static void fold(uint4 &mn, uint4 &mx, uint4 v) {
        mn.x = __vminu2(mn.x, v.x); mn.y = __vminu2(mn.y, v.y); mn.z = __vminu2(mn.z, v.z); mn.w = __vminu2(mn.w, v.w);
        mx.x = __vmaxu2(mx.x, v.x); mx.y = __vmaxu2(mx.y, v.y); mx.z = __vmaxu2(mx.z, v.z); mx.w = __vmaxu2(mx.w, v.w);
    }
    __device__ __forceinline__ static void merge(uint4 &mn, uint4 &mx, const uint4 &mn2, const uint4 &mx2) {
        mn.x = __vminu2(mn.x, mn2.x); mn.y = __vminu2(mn.y, mn2.y); mn.z = __vminu2(mn.z, mn2.z); mn.w = __vminu2(mn.w, mn2.w);
        mx.x = __vmaxu2(mx.x, mx2.x); mx.y = __vmaxu2(mx.y, mx2.y); mx.z = __vmaxu2(mx.z, mx2.z); mx.w = __vmaxu2(mx.w, mx2.w);
    }
    __device__ __forceinline__ static uint32_t elem(const uint4 &w, int i, bool is_max) {
        uint32_t word = (i >> 1) == 0 ? w.x : (i >> 1) == 1 ? w.y : (i >> 1) == 2 ? w.z : w.w;
        return (word >> (16 * (i & 1))) & 0xFFFFu;
    }
    __device__ __forceinline__ static void init(uint4 &mn, uint4 &mx, uint4 v) { mn = v; mx = v; }
    // two rows per instruction: three-input packed min/max
    __device__ __forceinline__ static void fold2(uint4 &mn, uint4 &mx, uint4 a, uint4 b) {
        mn.x = __vimin3_u16x2(mn.x, a.x, b.x); mn.y = __vimin3_u16x2(mn.y, a.y, b.y);
        mn.z = __vimin3_u16x2(mn.z, a.z, b.z); mn.w = __vimin3_u16x2(mn.w, a.w, b.w);
        mx.x = __vimax3_u16x2(mx.x, a.x, b.x); mx.y = __vimax3_u16x2(mx.y, a.y, b.y);
        mx.z = __vimax3_u16x2(mx.z, a.z, b.z); mx.w = __vimax3_u16x2(mx.w, a.w, b.w);
    }
};

template <> struct Lane16<float> {
    static constexpr int V = 4;
    // lanes hold order-preserving keys, one per float
    __device__ __forceinline__ static uint4 lo_id() { return make_uint4(~0u, ~0u, ~0u, ~0u); }
    __device__ __forceinline__ static uint4 hi_id() { return make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ static void fold(uint4 &mn, uint4 &mx, uint4 v) {
        uint32_t k0 = Vox<float>::key(__uint_as_float(v.x)), k1 = Vox<float>::key(__uint_as_float(v.y));
        uint32_t k2 = Vox<float>::key(__uint_as_float(v.z)), k3 = Vox<float>::key(__uint_as_float(v.w));
        mn.x = min(mn.x, k0); mn.y = min(mn.y, k1); mn.z = min(mn.z, k2); mn.w = min(mn.w, k3);
        mx.x = max(mx.x, k0); mx.y = max(mx.y, k1); mx.z = max(mx.z, k2); mx.w = max(mx.w, k3);
    }
    __device__ __forceinline__ static void merge(uint4 &mn, uint4 &mx, const uint4 &mn2, const uint4 &mx2) {
        mn.x = min(mn.x, mn2.x); mn.y = min(mn.y, mn2.y); mn.z = min(mn.z, mn2.z); mn.w = min(mn.w, mn2.w);
        mx.x = max(mx.x, mx2.x); mx.y = max(mx.y, mx2.y); mx.z = max(mx.z, mx2.z); mx.w = max(mx.w, mx2.w);
    }
    __device__ __forceinline__ static uint32_t elem(const uint4 &w, int i, bool is_max) {
        return i == 0 ? w.x : i == 1 ? w.y : i == 2 ? w.z : w.w;
    }
    __device__ __forceinline__ static uint4 keys(uint4 v) {
        return make_uint4(Vox<float>::key(__uint_as_float(v.x)), Vox<float>::key(__uint_as_float(v.y)),
                          Vox<float>::key(__uint_as_float(v.z)), Vox<float>::key(__uint_as_float(v.w)));
    }
    __device__ __forceinline__ static void init(uint4 &mn, uint4 &mx, uint4 v) { mn = mx = keys(v); }
    __device__ __forceinline__ static void fold2(uint4 &mn, uint4 &mx, uint4 a, uint4 b) {
        const uint4 ka = keys(a), kb = keys(b);
        mn.x = __vimin3_u32(mn.x, ka.x, kb.x); mn.y = __vimin3_u32(mn.y, ka.y, kb.y);
        mn.z = __vimin3_u32(mn.z, ka.z, kb.z); mn.w = __vimin3_u32(mn.w, ka.w, kb.w);
        mx.x = __vimax3_u32(mx.x, ka.x, kb.x); mx.y = __vimax3_u32(mx.y, ka.y, kb.y);
        mx.z = __vimax3_u32(mx.z, ka.z, kb.z); mx.w = __vimax3_u32(mx.w, ka.w, kb.w);
    }
};

// One warp's share of the leaf pass: warp w of the volume's
// nXS * GY * ceil(GZ / zchunk) warps.
template <typename T, int B, int ZU>
__device__ __forceinline__ void minmax_leaf_vec_warp(const T *__restrict__ vol, uint32_t X, uint32_t Y, uint32_t Z,
                                                     uint32_t GX, uint32_t GY, uint32_t GZ, uint32_t nXS,
                                                     uint32_t zchunk, uint64_t w, uint2 *__restrict__ leaf) {
    using L16 = Lane16<T>;
    constexpr int V = L16::V;
    constexpr int SEG = 32 * V;
    constexpr int NB = V >= B ? V / B : 1;      // blocks per lane
    constexpr int LPB = V >= B ? 1 : B / V;     // lanes per block
    constexpr int CNT = V >= B ? B : V;         // elements of one block in one lane
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t xs = (uint32_t)(w % nXS);
    const uint64_t rest = w / nXS;
    const uint32_t by = (uint32_t)(rest % GY);
    const uint32_t zc = (uint32_t)(rest / GY);
    const uint32_t bz0 = zc * zchunk;
    const uint32_t bz1 = min(GZ, bz0 + zchunk);
    if (bz0 >= GZ) return;

    const uint32_t x0 = xs * SEG + lane * V;
    const bool on = x0 < X;                       // X is a multiple of V
    const uint32_t xh = xs * SEG + SEG;           // halo column of the strip
    const bool halo_on = lane == 31 && xh < X;
    const uint32_t y0 = by * B;
    const uint32_t ny = min((uint32_t)B + 1u, Y - y0);
    const uint64_t plane = (uint64_t)X * Y;

    uint32_t amn[NB], amx[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) { amn[j] = ~0u; amx[j] = 0u; }

    const uint32_t zend = min(bz1 * B, Z - 1);
    uint32_t bz = bz0;
    for (uint32_t z0 = bz0 * B; z0 <= zend; z0 += ZU) {
        // issue every load of the ZU slices before any of them is folded
        uint4 v[ZU][B + 1];
        uint32_t hv[ZU][B + 1];
#pragma unroll
        for (int u = 0; u < ZU; ++u) {
            const T *row = vol + (uint64_t)(z0 + u) * plane + (uint64_t)y0 * X;
            const bool zon = z0 + u <= zend;
#pragma unroll
            for (int r = 0; r <= B; ++r) {
                v[u][r] = L16::lo_id();
                if (on && zon && (uint32_t)r < ny)
                    v[u][r] = __ldg(reinterpret_cast<const uint4 *>(row + (uint64_t)r * X + x0));
                hv[u][r] = 0;
                if (halo_on && zon && (uint32_t)r < ny) hv[u][r] = Vox<T>::key(__ldg(row + (uint64_t)r * X + xh));
            }
        }
#pragma unroll
        for (int u = 0; u < ZU; ++u) {
            const uint32_t z = z0 + u;
            if (z > zend) break;
            uint4 mn = L16::lo_id(), mx = L16::hi_id();
            uint32_t hmn = ~0u, hmx = 0u;
#pragma unroll
            for (int r = 0; r <= B; ++r) {
                if ((uint32_t)r < ny) {
                    if (on) L16::fold(mn, mx, v[u][r]);
                    if (halo_on) {
                        hmn = min(hmn, hv[u][r]);
                        hmx = max(hmx, hv[u][r]);
                    }
                }
            }
            // first column of the next lane is this lane's halo column
            uint32_t nmn = __shfl_down_sync(0xffffffffu, L16::elem(mn, 0, false), 1);
            uint32_t nmx = __shfl_down_sync(0xffffffffu, L16::elem(mx, 0, true), 1);
            if (lane == 31) { nmn = hmn; nmx = hmx; }

            uint32_t smn[NB], smx[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                uint32_t a = ~0u, b = 0u;
#pragma unroll
                for (int i = 0; i < CNT; ++i) {
                    a = min(a, L16::elem(mn, j * CNT + i, false));
                    b = max(b, L16::elem(mx, j * CNT + i, true));
                }
                const bool take_halo = V >= B ? true : ((lane % LPB) == LPB - 1);
                if (take_halo) {
                    if (V >= B && j + 1 < NB) {
                        a = min(a, L16::elem(mn, (j + 1) * B, false));
                        b = max(b, L16::elem(mx, (j + 1) * B, true));
                    } else {
                        a = min(a, nmn);
                        b = max(b, nmx);
                    }
                }
                smn[j] = a;
                smx[j] = b;
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) { amn[j] = min(amn[j], smn[j]); amx[j] = max(amx[j], smx[j]); }
            if (z == bz * B + B) {
                // halo slice of bz, first slice of bz + 1: write block bz
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    uint32_t a = amn[j], b = amx[j];
#pragma unroll
                    for (int o = 1; o < LPB; o <<= 1) {
                        a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
                        b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
                    }
                    if (on && (lane % LPB) == 0) {
                        const uint32_t bx = x0 / B + j;
                        if (MTX_BC(((uint64_t)bz * GY + by) * GX + bx, (uint64_t)GX * GY * GZ, kBcLeaf))
                            leaf[((uint64_t)bz * GY + by) * GX + bx] = make_uint2(a, b);
                    }
                    amn[j] = smn[j];
                    amx[j] = smx[j];
                }
                ++bz;
            }
        }
    }
    if (bz < bz1) {
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            uint32_t a = amn[j], b = amx[j];
#pragma unroll
            for (int o = 1; o < LPB; o <<= 1) {
                a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
                b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
            }
            if (on && (lane % LPB) == 0) {
                const uint32_t bx = x0 / B + j;
                if (MTX_BC(((uint64_t)bz * GY + by) * GX + bx, (uint64_t)GX * GY * GZ, kBcLeaf))
                    leaf[((uint64_t)bz * GY + by) * GX + bx] = make_uint2(a, b);
            }
        }
    }
}

// ------------------------------------------- any block edge, any alignment
// One aligned 32-bit word of a voxel row as operands of packed three-input
// min/max.  uint8 takes two: the even bytes alone, and the word as it is, in
// whose 16-bit halves the odd byte decides every comparison (the even byte
// below it only breaks ties), so that the winners' high bytes are the odd
// bytes' min and max.
template <typename T> struct RowWord;
template <> struct RowWord<uint8_t> {
    static constexpr int N = 2, VPW = 4;
    __device__ __forceinline__ static void split(uint32_t w, uint32_t v[2]) {
        v[0] = w & 0x00ff00ffu;
        v[1] = w;
    }
    __device__ __forceinline__ static uint32_t join(const uint32_t v[2]) {
        return (v[0] & 0x00ff00ffu) | (v[1] & 0xff00ff00u);
    }
    __device__ __forceinline__ static uint32_t lo(uint32_t a, uint32_t b) { return __vminu2(a, b); }
    __device__ __forceinline__ static uint32_t hi(uint32_t a, uint32_t b) { return __vmaxu2(a, b); }
    __device__ __forceinline__ static uint32_t lo3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u16x2(a, b, c); }
    __device__ __forceinline__ static uint32_t hi3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u16x2(a, b, c); }
    __device__ __forceinline__ static uint32_t column(const uint32_t *s, uint32_t c) {
        return reinterpret_cast<const uint8_t *>(s)[c];
    }
};
template <> struct RowWord<uint16_t> {
    static constexpr int N = 1, VPW = 2;
    __device__ __forceinline__ static void split(uint32_t w, uint32_t v[1]) { v[0] = w; }
    __device__ __forceinline__ static uint32_t join(const uint32_t v[1]) { return v[0]; }
    __device__ __forceinline__ static uint32_t lo(uint32_t a, uint32_t b) { return __vminu2(a, b); }
    __device__ __forceinline__ static uint32_t hi(uint32_t a, uint32_t b) { return __vmaxu2(a, b); }
    __device__ __forceinline__ static uint32_t lo3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u16x2(a, b, c); }
    __device__ __forceinline__ static uint32_t hi3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u16x2(a, b, c); }
    __device__ __forceinline__ static uint32_t column(const uint32_t *s, uint32_t c) {
        return reinterpret_cast<const uint16_t *>(s)[c];
    }
};
template <> struct RowWord<float> {
    static constexpr int N = 1, VPW = 1;
    __device__ __forceinline__ static void split(uint32_t w, uint32_t v[1]) {
        v[0] = Vox<float>::key(__uint_as_float(w));
    }
    __device__ __forceinline__ static uint32_t join(const uint32_t v[1]) { return v[0]; }
    __device__ __forceinline__ static uint32_t lo(uint32_t a, uint32_t b) { return min(a, b); }
    __device__ __forceinline__ static uint32_t hi(uint32_t a, uint32_t b) { return max(a, b); }
    __device__ __forceinline__ static uint32_t lo3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u32(a, b, c); }
    __device__ __forceinline__ static uint32_t hi3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u32(a, b, c); }
    __device__ __forceinline__ static uint32_t column(const uint32_t *s, uint32_t c) { return s[c]; }
};

// How a volume is cut into strips of whole blocks: nbs blocks a strip, nXS
// strips of almost equal width.  aligned: every row of every strip starts on a
// word, so no row has to be shifted.  wide: two words of a row a lane (strips
// of up to 64 float32, 128 uint16 or 256 uint8 columns), else one.
struct RowCut {
    uint32_t nbs, nXS, aligned, wide;
};
inline RowCut row_cut(const Problem &p, uint32_t esz) {
    RowCut c{};
    // uint8 rows of up to 160 voxels leave most of a 256-column strip's lanes idle.  256 x
    // 256 slices of such rows, us with one word a lane and two, at B = 3 / B = 8: X = 61
    // 7.1, 9.3 / 6.6, 8.1; 96 5.3, 6.6 / 4.3, 5.2; 128 8.4, 7.2 / 5.0, 5.3; 192 8.4, 7.2 /
    // 5.0, 5.4; 250 14.5, 15.9 / 11.4, 12.5; 1024 (and 1024 x 314) 152, 112 at B = 3
    c.wide = esz > 1 || p.X > 160;
    const uint32_t W = c.wide ? 2u : 1u, vpw = 4u / esz;
    // blocks are word-aligned columns apart when `step` of them are
    uint32_t step = 1;
    while ((step * p.B * esz) % 4) ++step;
    c.aligned = (uintptr_t)p.vol % 4 == 0 && ((uint64_t)p.X * esz) % 4 == 0 && (32 * W * vpw - 1) / p.B >= step;
    // a strip's columns: its blocks and the next block's first column
    uint32_t most = std::max(1u, ((c.aligned ? 32 * W : 32 * W - 1) * vpw - 1) / p.B);
    if (c.aligned) most = most / step * step;
    c.nXS = ceil_div(p.GX, most);
    c.nbs = ceil_div(p.GX, c.nXS);
    if (c.aligned) c.nbs = std::min(most, ceil_div(c.nbs, step) * step);
    c.nXS = ceil_div(p.GX, c.nbs);
    return c;
}

// Whether the byte offsets of a block's rows fit 32 bits and every row is a
// word or longer: then only the volume's first and last row have a word that
// reaches past the volume (is_edge below).  Other rows take minmax_leaf_one.
inline bool rows_ok(const Problem &p, uint32_t esz) {
    const uint64_t row = (uint64_t)p.X * esz;
    return row >= 4 && row * p.B < (1ull << 32);
}

// One warp's share of the leaf pass for any block edge and any row alignment:
// a strip of nbs whole blocks of one block row over a run of zchunk slabs.
// Lanes own columns (W words of consecutive voxels each): per z slice the
// B + 1 rows of the strip are loaded as aligned words, a slice ahead of their
// use; rows that do not start on a word (ALIGNED false) are shifted into
// place with the next lane's word.  Rows fold column by column, slices fold
// into the running slab, and only when a slab is complete -- once every B
// slices -- do the columns go to shared memory, where each lane takes the
// B + 1 columns of its blocks.  NR = B + 1 at compile time, 0: at run time,
// four rows in flight.  s: 64 * W words of the warp's own shared memory.
// nan_zero (float32): a NaN of positive sign takes the key of -0.0 instead of one
// above +inf, which would leave its block without an isovalue -- what volumes
// off the 16-byte passes have always had, while those passes keep the NaN's key.  Rows
// are 4 bytes or longer and the B + 1 rows of a strip span less than 4 GiB (rows_ok).
// Bound by instruction issue (about 2.5 a cycle and SM): every word costs an
// address, a load, for unaligned rows a shuffle and a shift, and half a
// min/max pair.  Against one thread a block, whose byte loads read every voxel
// of a block alone: 1024 x 1024 x 314 uint8 at B = 3, 477 -> 112 us (one word
// a lane instead of two: 152); 509 x 387 x 301 uint16 at B = 8, 74 -> 39;
// 250 x 198 x 171 float32 at B = 8, 75 -> 10.
template <typename T, int W, int NR, bool ALIGNED>
__device__ __forceinline__ void minmax_leaf_rows_warp(const T *__restrict__ vol, uint32_t X, uint32_t Y, uint32_t Z,
                                                      uint32_t B_, uint32_t GX, uint32_t GY, uint32_t GZ, uint32_t nXS,
                                                      uint32_t nbs, uint32_t zchunk, uint64_t w,
                                                      uint2 *__restrict__ leaf, uint32_t *s, bool nan_zero = true) {
    using RW = RowWord<T>;
    constexpr int N = RW::N;
    const uint32_t B = NR ? (uint32_t)(NR - 1) : B_, lane = threadIdx.x & 31;
    const uint32_t xs = (uint32_t)(w % nXS);
    const uint64_t rest = w / nXS;
    const uint32_t by = (uint32_t)(rest % GY);
    const uint64_t zc = rest / GY;
    if (zc * zchunk >= GZ) return;
    const uint32_t bz0 = (uint32_t)zc * zchunk, bz1 = min(GZ, bz0 + zchunk);
    const uint32_t xb0 = xs * nbs, x0 = xb0 * B, nb = min(nbs, GX - xb0);
    const uint32_t ncol = min(X - x0, nb * B + 1);  // columns the strip's blocks cover
    const uint32_t y0 = by * B, ny = min(B + 1, Y - y0);
    const uint64_t rowb = (uint64_t)X * sizeof(T), planeb = rowb * Y;
    const uintptr_t vbeg = reinterpret_cast<uintptr_t>(vol), vend = vbeg + planeb * Z;
    const uint32_t zend = min(bz1 * B, Z - 1);
    uint32_t *smn = s, *smx = s + 32 * W;

    uint32_t amn[W][N], amx[W][N];
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
        for (int n = 0; n < N; ++n) {
            amn[j][n] = ~0u;
            amx[j][n] = 0u;
        }
    uint32_t bz = bz0;
    // this lane's first word of the strip's first row, and its word's place in the strip
    uintptr_t slice = vbeg + (uint64_t)bz0 * B * planeb + (uint64_t)y0 * rowb + (uint64_t)x0 * sizeof(T) + 4u * lane;
    bool on[W];  // words that hold a column of the strip (or the bytes after one)
#pragma unroll
    for (int j = 0; j < W; ++j) on[j] = 4u * (32 * j + lane) < ncol * (uint32_t)sizeof(T) + (ALIGNED ? 0u : 3u);
    // byte offset of row r; a row past the block repeats its last one, which changes no min or max
    auto row_off = [&](uint32_t r) { return (uint32_t)rowb * min(r, ny - 1); };
    auto close = [&](uint32_t b) {  // the slab's columns -> its blocks
#pragma unroll
        for (int j = 0; j < W; ++j) {
            smn[32 * j + lane] = RW::join(amn[j]);
            smx[32 * j + lane] = RW::join(amx[j]);
        }
        __syncwarp();
        for (uint32_t i = lane; i < nb; i += 32) {
            const uint32_t c1 = min(i * B + B, ncol - 1);
            uint32_t lo = ~0u, hi = 0u;
            for (uint32_t c = i * B; c <= c1; ++c) {
                lo = min(lo, RW::column(smn, c));
                hi = max(hi, RW::column(smx, c));
            }
            if (MTX_BC(((uint64_t)b * GY + by) * GX + xb0 + i, (uint64_t)GX * GY * GZ, kBcLeaf))
                leaf[((uint64_t)b * GY + by) * GX + xb0 + i] = make_uint2(lo, hi);
        }
        __syncwarp();
    };
    auto load = [&](uintptr_t at, uint32_t r, uint32_t raw[W]) {
        const uintptr_t a = at + row_off(r);
        const uint32_t *src = reinterpret_cast<const uint32_t *>(ALIGNED ? a : a & ~(uintptr_t)3);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            [[maybe_unused]] const uintptr_t last = reinterpret_cast<uintptr_t>(src + 32 * j) + 3;
            raw[j] = on[j] && MTX_BC(last - vbeg, vend - vbeg, kBcVolume) ? __ldg(src + 32 * j) : 0u;
        }
    };
    // the same for a row with a word that may reach past the volume: its bytes one by one
    auto load_edge = [&](uintptr_t at, uint32_t r, uint32_t raw[W]) {
        const uintptr_t a = (at + row_off(r)) & ~(uintptr_t)3;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            raw[j] = 0;
            for (uint32_t k = 0; k < 4; ++k) {
                const uintptr_t q = a + 128 * j + k;
                if (q >= vbeg && q < vend) raw[j] |= (uint32_t)__ldg(reinterpret_cast<const uint8_t *>(q)) << (8 * k);
            }
        }
    };
    // a row's columns, this lane's starting sh bits into its word
    auto place = [&](uintptr_t at, uint32_t r, const uint32_t raw[W], uint32_t v[W][N]) {
        const uint32_t sh = ALIGNED ? 0u : 8u * (((uint32_t)at + row_off(r)) & 3u);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            uint32_t x = raw[j];
            if constexpr (!ALIGNED) {
                const uint32_t give = j + 1 < W && lane == 0 ? raw[j + 1 < W ? j + 1 : j] : raw[j];
                x = __funnelshift_r(x, __shfl_sync(0xffffffffu, give, (lane + 1) & 31), sh);
            }
            RW::split(x, v[j]);
            if constexpr (sizeof(T) == 4) v[j][0] = nan_zero && v[j][0] > 0xff800000u ? 0x7fffffffu : v[j][0];
        }
    };
    uint32_t tmn[W][N], tmx[W][N];  // the slice
    auto fold_pair = [&](bool start, const uint32_t v[W][N], const uint32_t u[W][N]) {
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                tmn[j][n] = start ? RW::lo(v[j][n], u[j][n]) : RW::lo3(tmn[j][n], v[j][n], u[j][n]);
                tmx[j][n] = start ? RW::hi(v[j][n], u[j][n]) : RW::hi3(tmx[j][n], v[j][n], u[j][n]);
            }
    };
    // only the volume's first and last row have a word that reaches past the volume
    auto is_edge = [&](uint32_t z) {
        return !ALIGNED && ((z == 0 && y0 == 0) || (z == Z - 1 && y0 + ny == Y));
    };
    constexpr int NA = NR ? NR : 1;
    uint32_t raw[NA][W];  // NR > 0: the slice's rows, loaded one slice ahead
    if constexpr (NR > 0) {
        if (!is_edge(bz0 * B)) {
#pragma unroll
            for (int r = 0; r < NR; ++r) load(slice, r, raw[r]);
        }
    }
    for (uint32_t z = bz0 * B; z <= zend; ++z, slice += planeb) {
        uint32_t v[W][N], u[W][N];
        const bool edge = is_edge(z);
        if (edge) {
            for (uint32_t r = 0; r < ny; ++r) {
                uint32_t w1[W];
                load_edge(slice, r, w1);
                place(slice, r, w1, v);
                if (r == 0) fold_pair(true, v, v);
                else fold_pair(false, v, v);
            }
        }
        if constexpr (NR > 0) {
            uint32_t cur[NA][W];
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int j = 0; j < W; ++j) cur[r][j] = raw[r][j];
            if (z < zend && !is_edge(z + 1)) {
#pragma unroll
                for (int r = 0; r < NR; ++r) load(slice + planeb, r, raw[r]);
            }
            if (!edge) {
                constexpr int R0 = (NR & 1) ? 1 : 2;
                place(slice, 0, cur[0], v);
                if (R0 == 2) {
                    place(slice, 1, cur[R0 - 1], u);
                    fold_pair(true, v, u);
                } else {
                    fold_pair(true, v, v);
                }
#pragma unroll
                for (int r = R0; r < NR; r += 2) {
                    place(slice, r, cur[r], v);
                    place(slice, r + 1, cur[r + 1], u);
                    fold_pair(false, v, u);
                }
            }
        } else if (!edge) {
            for (uint32_t r = 0; r < ny; r += 4) {
                uint32_t four[4][W];
#pragma unroll
                for (int k = 0; k < 4; ++k) load(slice, r + k, four[k]);
                place(slice, r, four[0], v);
                place(slice, r + 1, four[1], u);
                if (r == 0) fold_pair(true, v, u);
                else fold_pair(false, v, u);
                place(slice, r + 2, four[2], v);
                place(slice, r + 3, four[3], u);
                fold_pair(false, v, u);
            }
        }
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                amn[j][n] = RW::lo(amn[j][n], tmn[j][n]);
                amx[j][n] = RW::hi(amx[j][n], tmx[j][n]);
            }
        if (z == bz * B + B) {  // the halo slice of slab bz is the first slice of slab bz + 1
            close(bz);
            ++bz;
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int n = 0; n < N; ++n) {
                    amn[j][n] = tmn[j][n];
                    amx[j][n] = tmx[j][n];
                }
        }
    }
    if (bz < bz1) close(bz);
}

// One block by one thread: rows that rows_ok refuses.
template <typename T>
__device__ __forceinline__ void minmax_leaf_one(const T *__restrict__ vol, uint32_t X, uint32_t Y, uint32_t Z,
                                                uint32_t B, uint32_t GX, uint32_t GY, uint64_t b,
                                                uint2 *__restrict__ leaf) {
    uint32_t bx = (uint32_t)(b % GX), by = (uint32_t)((b / GX) % GY), bz = (uint32_t)(b / ((uint64_t)GX * GY));
    uint32_t x0 = bx * B, y0 = by * B, z0 = bz * B;
    uint32_t x1 = min(x0 + B, X - 1), y1 = min(y0 + B, Y - 1), z1 = min(z0 + B, Z - 1);
    uint32_t mn = ~0u, mx = 0u;
    for (uint32_t z = z0; z <= z1; ++z)
        for (uint32_t y = y0; y <= y1; ++y) {
            const T *row = vol + ((uint64_t)z * Y + y) * X;
            for (uint32_t x = x0; x <= x1; ++x) {
                uint32_t k = Vox<T>::key(__ldg(row + x));
                mn = min(mn, k);
                mx = max(mx, k);
            }
        }
    leaf[b] = make_uint2(mn, mx);
}

// ------------------------------------------------------------ octree
// Every octree level in one launch (minMaxOctreeReduce.comp.glsl:23-59 runs
// one dispatch per level).  A step of a CTA takes 32 x 8 x 8 texels of the
// launch's first level (the leaf level, or level 1 when the leaf pass wrote it):
// each thread reads the 2 x 2 x 2 texels of one texel of the next level, all
// eight loads in flight and those of its next step behind them, and the two
// levels after that follow by shuffles and one exchange through shared memory.
// A tile is one step, or 2 x 2 of them in y and z (`quad`), whose level-3
// texels make one level more.  The CTA that finishes last builds the rest and
// zeroes the counter (zero since the context's creation) for the next launch.
// Each texel is the min/max of its up-to-8 children; children past their
// level's extent are skipped (minMaxOctreeReduce.comp.glsl:37-47), which the
// identity {~0, 0} in their place does.
// Latency-bound: a step costs a round of loads and a barrier, so the CTAs of the
// launch stay and load ahead instead of one CTA a step with a counter each, and
// the serial levels of the last CTA begin one level higher.  For the 342 x 342 x
// 105 grid of a 1024 x 1024 x 314 volume at B = 3: 55 us with a CTA a step, 30 so
// (a CTA of 512 threads per 8^3 texels with a barrier pair a level: 203).
constexpr int kPyrMaxLevels = 32;
constexpr uint32_t kPyrThreads = 256, kPyrTileX = 32, kPyrTileYZ = 8;
struct PyrAll {
    uint2 *base[kPyrMaxLevels];
    uint32_t ext[kPyrMaxLevels][3];
    int levels;
    uint32_t quad;  // 1: tiles of 2 x 2 steps
    uint32_t tiles_x, tiles_y, ntiles;
    uint32_t ctas;  // CTAs of the launch that work on the octree, at most ntiles
    uint32_t *done;
};

__device__ __forceinline__ uint2 texel_join(uint2 a, uint2 b) { return make_uint2(min(a.x, b.x), max(a.y, b.y)); }
__device__ __forceinline__ uint2 texel_xor(uint2 a, int o) {
    return texel_join(a, make_uint2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o)));
}
__device__ __forceinline__ void texel_store(const PyrAll &L, int k, uint32_t x, uint32_t y, uint32_t z, uint2 v) {
    if (k < L.levels && x < L.ext[k][0] && y < L.ext[k][1] && z < L.ext[k][2] &&
        MTX_BC(((uint64_t)z * L.ext[k][1] + y) * L.ext[k][0] + x, (uint64_t)L.ext[k][0] * L.ext[k][1] * L.ext[k][2],
               kBcOctree))
        L.base[k][((uint64_t)z * L.ext[k][1] + y) * L.ext[k][0] + x] = v;
}

// The part of CTA `cta` of L.ctas, by all kPyrThreads threads of it.
__device__ __forceinline__ void pyramid_part(const PyrAll &L, uint32_t cta, uint2 (*s_part)[8][8], uint32_t *s_last) {
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t ox = t & 15, oy = (t >> 4) & 3, oz = t >> 6;  // 16 x 4 x 4 level-1 texels a step, a warp 16 x 2
    const uint32_t steps = L.quad ? 4u : 1u;
    uint32_t tx = 0, ty = 0, tz = 0;  // the step to load next, in steps
    auto place = [&](uint32_t tile, uint32_t s) {
        const uint32_t rest = tile / L.tiles_x;
        tx = tile - rest * L.tiles_x;
        tz = rest / L.tiles_y;
        ty = rest - tz * L.tiles_y;
        if (L.quad) {
            ty = 2 * ty + (s & 1);
            tz = 2 * tz + (s >> 1);
        }
    };
    uint2 v[8];
    auto load = [&]() {
        const uint32_t x = 2 * (tx * 16 + ox), y = 2 * (ty * 4 + oy), z = 2 * (tz * 4 + oz);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const uint32_t ux = x + (c & 1), uy = y + ((c >> 1) & 1), uz = z + (c >> 2);
            v[c] = make_uint2(~0u, 0u);
            if (ux < L.ext[0][0] && uy < L.ext[0][1] && uz < L.ext[0][2])
                v[c] = L.base[0][((uint64_t)uz * L.ext[0][1] + uy) * L.ext[0][0] + ux];
        }
    };
    place(cta, 0);
    load();
    uint32_t buf = 0;
    for (uint32_t tile = cta; tile < L.ntiles; tile += L.ctas) {
        uint2 quad = make_uint2(~0u, 0u);  // warp 0: the tile's level-3 texels so far
        for (uint32_t s = 0; s < steps; ++s) {
            const uint32_t sx = tx, sy = ty, sz = tz;
            uint2 r = v[0];
#pragma unroll
            for (int c = 1; c < 8; ++c) r = texel_join(r, v[c]);
            if (s + 1 < steps) {
                place(tile, s + 1);
                load();
            } else if (tile + L.ctas < L.ntiles) {
                place(tile + L.ctas, 0);
                load();
            }
            texel_store(L, 1, sx * 16 + ox, sy * 4 + oy, sz * 4 + oz, r);
            if (L.levels <= 2) continue;
            r = texel_xor(texel_xor(r, 1), 16);  // pairs in x and y
            if (lane < 16 && !(lane & 1)) s_part[buf][warp][lane >> 1] = r;
            __syncthreads();  // and warp 0 is done with the other buffer, two steps old
            if (warp == 0) {
                // level 2: 8 x 2 x 2 texels, lane = x | y << 3 | z << 4; warp 2 z + (y of level 1) / 2 holds a pair in y
                const uint32_t x = lane & 7, y = (lane >> 3) & 1, z = lane >> 4;
                r = texel_join(s_part[buf][4 * z + y][x], s_part[buf][4 * z + 2 + y][x]);
                texel_store(L, 2, sx * 8 + x, sy * 2 + y, sz * 2 + z, r);
                r = texel_xor(texel_xor(texel_xor(r, 1), 8), 16);
                if (!(lane & 25)) texel_store(L, 3, sx * 4 + (x >> 1), sy, sz, r);
                quad = texel_join(quad, r);
                if (L.quad && s == 3) {
                    quad = texel_xor(quad, 2);
                    if (!(lane & 27)) texel_store(L, 4, sx * 2 + (x >> 2), sy >> 1, sz >> 1, quad);
                }
            }
            buf ^= 1;
        }
    }
    const int top = L.quad ? 5 : 4;  // the levels below are written by the tiles
    if (L.levels <= top) return;
    if (warp == 0) {
        __threadfence();
        __syncwarp();
        if (lane == 0) *s_last = atomicAdd(L.done, 1u) == L.ctas - 1;
    }
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    for (int k = top; k < L.levels; ++k) {
        const uint32_t ex = L.ext[k][0], ey = L.ext[k][1];
        const uint32_t px = L.ext[k - 1][0], py = L.ext[k - 1][1], pz = L.ext[k - 1][2];
        const uint32_t cnt = ex * ey * L.ext[k][2];  // below 2^30 / 8^3
#pragma unroll 2
        for (uint32_t i = t; i < cnt; i += kPyrThreads) {
            const uint32_t q = i / ex, x = i - q * ex, z = q / ey, y = q - z * ey;
            uint2 r = make_uint2(~0u, 0u);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t ux = 2 * x + (c & 1), uy = 2 * y + ((c >> 1) & 1), uz = 2 * z + (c >> 2);
                if (ux < px && uy < py && uz < pz &&
                    MTX_BC((uz * py + uy) * px + ux, (uint64_t)px * py * pz, kBcOctree))
                    r = texel_join(r, __ldcg(&L.base[k - 1][(uz * py + uy) * px + ux]));
            }
            L.base[k][i] = r;
        }
        __threadfence();
        __syncthreads();
    }
    if (t == 0) *L.done = 0;
}

}  // namespace mtx
