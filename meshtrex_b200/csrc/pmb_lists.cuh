// Block bodies of the single-volume count and emit passes (extract.cu).
//
// A block's work is its listed cells, in canonical order: the mixed cells
// (case neither 0 nor 255) and, at the volume's high faces, voxels that own a
// cut edge but start no cell.  The count pass finds them by bit operations on
// the inside bits of the block's voxel rows, takes them 32 at a time, one a
// lane, and hands each to the emit pass as one word -- cell, case, cut owned
// edges and the triangles before it in its 32 -- so that the emit pass needs
// neither the voxel tile nor the inside bits.  For B > 8 the list would be
// longer than the inside bits: those are handed over, and the emit pass lists
// the cells again.
//
// Handing over lists costs 4 bytes a listed cell (75 of 512 at B = 8 on the
// fields measured) where the rows, prefixes and case bytes of every cell took
// 1920 bytes a block, and it leaves no lane idle behind the row with the most
// cells, as walks along the rows did.
#pragma once

#include <type_traits>

#include "pmb_device.cuh"

namespace mtx {

// Triangles of every case in case order: three edge numbers, 4 bits each; and
// of each case the first of its triangles | their number << 12.
constexpr uint32_t kTris = 820;
static __device__ uint16_t g_mc_tri[kTris];
static __device__ uint16_t g_mc_first[256];

[[maybe_unused]] static mtx_status load_list_tables(mtx_context *c) {
    static bool loaded[128] = {false};
    mtx_status r = load_case_tables(c);
    if (r != MTX_OK || (c->device >= 0 && c->device < 128 && loaded[c->device])) return r;
    uint16_t tri[kTris], first[256];
    uint32_t n = 0;
    for (uint32_t i = 0; i < 256; ++i) {
        const uint32_t k = (uint32_t)(MTX_MC_CASES[i] & 0xFu);
        if (n + k > kTris) return fail(c, MTX_ERR_INTERNAL, "case table has more triangles than expected");
        first[i] = (uint16_t)(n | (k << 12));
        for (uint32_t t = 0; t < k; ++t) tri[n++] = (uint16_t)((MTX_MC_CASES[i] >> (4 + 12 * t)) & 0xFFFu);
    }
    for (; n < kTris; ++n) tri[n] = 0;
    MTX_CUDA(c, cudaMemcpyToSymbol(g_mc_tri, tri, sizeof(tri)));
    MTX_CUDA(c, cudaMemcpyToSymbol(g_mc_first, first, sizeof(first)));
    if (c->device >= 0 && c->device < 128) loaded[c->device] = true;
    return MTX_OK;
}

// ------------------------------------------------------------------ plans
// List bits come in units, one a lane: 16 cells for B <= 8 (all of a block's in
// one round of 32 lanes), else 32.  A warp's list holds a round's cells and up
// to 31 not yet taken.
__host__ __device__ inline uint32_t list_unit(uint32_t B) { return B <= 8 ? 16u : 32u; }
__host__ __device__ inline uint32_t list_cap(uint32_t B) {
    return B <= 8 ? (B * B * B + 15) / 16 * 16 : 32u * 32u + 32u;
}

// State handed from count to emit, words a block: the list, padded to whole
// steps of 32 (B <= 8), or the inside bits of the (B+1)^2 rows.
__host__ __device__ inline uint32_t list_state_words(uint32_t B) {
    return B <= 8 ? (B * B * B + 31) / 32 * 32 : ((B + 1) * (B + 1) + 3) / 4 * 4;
}
__host__ __device__ inline uint32_t face_stride16(uint32_t B) { return (3 * B * B + 7) / 8 * 8; }  // 16-bit records
__host__ __device__ inline uint32_t list_words(uint32_t B) { return (B * B * B + 31) / 32; }

__host__ __device__ inline void plan_block(WPlan &p, uint32_t B) {
    p.B = B;
    p.B1 = B + 1;
    p.S1 = B + 1;
    p.BB = B * B;
    p.nb3 = 3 * B * B + 3 * B + 1;
    p.rB = (uint32_t)((0x100000000ull + B - 1) / B);
    p.rB1 = (uint32_t)((0x100000000ull + B) / (B + 1));
}

// A warp's shared memory in the count pass: TMA tile and barrier, inside rows,
// list bits, list, face records (which share the region of the plain loads'
// bitstream: that is dead once the rows are built).
__host__ __device__ inline WPlan make_count_plan(uint32_t B, uint32_t esz, bool tma) {
    WPlan p{};
    plan_block(p, B);
    uint32_t o = 0;
    p.off_tile = 0;
    if (tma) {
        p.PX = tile_pitch(B, esz, true);
        p.tile_bytes = p.PX * p.B1 * p.B1 * esz;
        o = align_up(p.tile_bytes, 16);
    }
    p.off_bar = o;
    o += 16;
    p.off_rows = o;
    o = align_up(o + 4 * p.B1 * p.B1, 16);
    p.off_mm = o;  // list bits
    o = align_up(o + 4 * list_words(B), 16);
    p.off_list = o;
    o = align_up(o + 2 * list_cap(B), 16);
    p.off_case = o;  // face records / bitstream
    const uint32_t bits = 4 * ((p.B1 * p.B1 * p.B1 + 31) / 32 + 1);
    o = align_up(o + std::max(2 * face_stride16(B), tma ? 0u : bits), 16);
    p.bytes = align_up(o, 128);
    return p;
}

// Shared memory of a count CTA before its warps' regions: the cases' triangle
// counts and (off) the tile's element offsets.
__host__ __device__ inline uint32_t count_fixed_bytes(uint32_t B, bool off) {
    return align_up(256 + (off ? 4 * (B + 1) * (B + 1) * (B + 1) : 0u), 128);
}

// In the emit pass: vertex table, job ring, first vertices of the block and
// its seven neighbours, and for B > 8 the inside rows, list bits and list.
__host__ __device__ inline WPlan make_emit_plan(uint32_t B) {
    WPlan p{};
    plan_block(p, B);
    uint32_t o = 0;
    p.off_jobs = o;
    o += 4 * kJobWin;
    p.off_nvid = o;
    o += 32;
    p.off_vtab = o;
    o = align_up(o + 2 * p.B1 * p.B1 * p.B1, 16);
    if (B > 8) {
        p.off_rows = o;
        o = align_up(o + 4 * p.B1 * p.B1, 16);
        p.off_mm = o;
        o = align_up(o + 4 * list_words(B), 16);
        p.off_list = o;
        o = align_up(o + 2 * list_cap(B), 16);
    }
    p.bytes = align_up(o, 16);
    return p;
}

// In the batched kernel, whose emit phase always takes inside rows over: both
// phases' regions, the count phase's face records and bitstream in the vertex
// table's place.
__host__ __device__ inline WPlan make_batch_plan(uint32_t B) {
    WPlan p{};
    plan_block(p, B);
    uint32_t o = 0;
    p.off_jobs = o;
    o += 4 * kJobWin;
    p.off_nvid = o;
    o += 32;
    p.off_vtab = p.off_case = o;
    const uint32_t T3 = p.B1 * p.B1 * p.B1;
    o = align_up(o + std::max(2 * T3, std::max(2 * face_stride16(B), 4 * ((T3 + 31) / 32 + 1))), 16);
    p.off_rows = o;
    o = align_up(o + 4 * p.B1 * p.B1, 16);
    p.off_mm = o;
    o = align_up(o + 4 * list_words(B), 16);
    p.off_list = o;
    o = align_up(o + 2 * list_cap(B), 16);
    p.bytes = o;
    return p;
}
// Words of inside rows a block hands over there.
__host__ __device__ inline uint32_t row_state_words(uint32_t B) { return ((B + 1) * (B + 1) + 3) / 4 * 4; }

// Shared memory of an emit CTA before its warps' regions: the triangles as
// vertex-table offsets, the cases' first triangles, the context-layer map.
__host__ __device__ inline uint32_t emit_fixed_bytes(uint32_t B) {
    return align_up(8 * kTris + 512 + 4 * (3 * B * B + 3 * B + 1), 128);
}

// ------------------------------------------------------- inside rows by loads
// Inside bits of the block's (B+1)^2 rows from plain loads (rows that are not
// 16-byte aligned): the warp takes 32 consecutive voxels of the (B+1)^3 tile at
// a time, their inside bits are one ballot, and row q is the B+1 bits from bit
// q (B+1) of that stream on.  off: element offsets of the tile's voxels
// (row_offsets), null where they do not fit 32 bits.
template <typename T>
__device__ __forceinline__ void load_rows(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g,
                                          const uint32_t *off) {
    constexpr uint32_t kBatch = 8;
    const T *vol = reinterpret_cast<const T *>(p.vol);
    uint32_t *words = reinterpret_cast<uint32_t *>(ws + pl.off_case);
    uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
    const uint32_t lane = threadIdx.x & 31, B1 = pl.B1, n = B1 * B1 * B1, nw = (n + 31) / 32;
    const bool inner = g.ox + pl.B < p.X && g.oy + pl.B < p.Y && g.oz + pl.B < p.Z;
    const T *base = vol + ((uint64_t)g.oz * p.Y + g.oy) * p.X + g.ox;
    const bool narrow = ((uint64_t)B1 * p.X * p.Y >> 32) == 0;  // the tile's offsets fit 32 bits
    for (uint32_t w0 = 0; w0 < nw; w0 += kBatch) {
        T v[kBatch];
        uint32_t in = 0;
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k) {
            const uint32_t i = (w0 + k) * 32 + lane;
            bool on = i < n;
            v[k] = T(0);
            if (inner && off) {
                if (on) v[k] = __ldg(base + off[i]);
            } else if (inner && narrow) {
                const uint32_t iq = fdiv(i, pl.rB1), z = fdiv(iq, pl.rB1);
                if (on) v[k] = __ldg(base + ((z * p.Y + iq - z * B1) * p.X + i - iq * B1));
            } else {
                const uint32_t iq = fdiv(i, pl.rB1);
                const uint32_t x = i - iq * B1, z = fdiv(iq, pl.rB1), y = iq - z * B1;
                on = on && g.ox + x < p.X && g.oy + y < p.Y && g.oz + z < p.Z;
                if (on) v[k] = __ldg(base + ((uint64_t)z * p.Y + y) * p.X + x);
            }
            in |= (on ? 1u : 0u) << k;
        }
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k) {
            const uint32_t bal = __ballot_sync(0xffffffffu, ((in >> k) & 1u) && Vox<T>::val(v[k]) <= p.iso);
            if (lane == 0 && w0 + k < nw) words[w0 + k] = bal;
        }
    }
    __syncwarp();
    const uint32_t mask = (1u << B1) - 1u;
    for (uint32_t q = lane; q < B1 * B1; q += 32) {
        const uint32_t bit = q * B1, w = bit >> 5;
        const uint32_t hi = w + 1 < nw ? words[w + 1] : 0u;
        if (MTX_BC(q, B1 * B1, kBcRows)) rows[q] = __funnelshift_r(words[w], hi, bit & 31u) & mask;
    }
    __syncwarp();
}

// Inside bits of the rows of a staged tile for a block edge known at compile
// time (build_rows otherwise).  Integer voxels: the sign of floor(iso) - value,
// shifted in voxel by voxel from the row's end; float voxels: the compare.
template <typename T, int BC>
__device__ __forceinline__ void tile_rows(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g) {
    constexpr uint32_t B1 = BC + 1;
    const T *tile = reinterpret_cast<const T *>(ws + pl.off_tile);
    uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
    const uint32_t xin = min(B1, p.X - g.ox);
    // integer voxels: value <= iso  <=>  value <= floor(iso) (never when iso < 0 or NaN)
    const bool never = Vox<T>::code != 2 && !(p.iso >= 0.0f);
    const int thr = never || Vox<T>::code == 2 ? 0 : (int)fminf(floorf(p.iso), sizeof(T) == 1 ? 255.0f : 65535.0f);
    const uint32_t xmask = never ? 0u : (1u << xin) - 1u;
    // rows of 8 and 16 voxels start on 8 (uint8) or 16 bytes
    constexpr bool kWide = BC == 8 || BC == 16;
    constexpr uint32_t NW = BC * sizeof(T) / 4;  // words of a row but its last voxel
    for (uint32_t q = threadIdx.x & 31; q < B1 * B1; q += 32) {
        const uint32_t z = q / B1, y = q - z * B1;
        const T *r = tile + q * pl.PX + g.xoff;
        uint32_t m = 0;
        if constexpr (kWide) {
            uint32_t w[NW];
#pragma unroll
            for (uint32_t i = 0; i < NW; i += (NW % 4 ? 2 : 4)) {
                if constexpr (NW % 4 == 0) {
                    const uint4 v = reinterpret_cast<const uint4 *>(r)[i / 4];
                    w[i] = v.x, w[i + 1] = v.y, w[i + 2] = v.z, w[i + 3] = v.w;
                } else {
                    const uint2 v = reinterpret_cast<const uint2 *>(r)[i / 2];
                    w[i] = v.x, w[i + 1] = v.y;
                }
            }
            const T last = r[BC];
#pragma unroll
            for (int x = BC; x >= 0; --x) {
                if constexpr (Vox<T>::code == 2) {
                    const float v = x == BC ? (float)last : __uint_as_float(w[x < BC ? x : 0]);
                    m = 2 * m + (v <= p.iso ? 1u : 0u);
                } else {
                    constexpr int PER = 4 / sizeof(T);
                    const int xi = x < BC ? x : 0;
                    const int v = x == BC ? (int)last
                                          : (int)((w[xi / PER] >> (8 * sizeof(T) * (xi % PER))) &
                                                  (sizeof(T) == 1 ? 0xffu : 0xffffu));
                    m = __funnelshift_l((uint32_t)(thr - v), m, 1);
                }
            }
        } else {
#pragma unroll
            for (int x = BC; x >= 0; --x) {
                if constexpr (Vox<T>::code == 2) m = 2 * m + (Vox<T>::val(r[x]) <= p.iso ? 1u : 0u);
                else m = __funnelshift_l((uint32_t)(thr - (int)r[x]), m, 1);
            }
        }
        if (Vox<T>::code != 2) m = ~m;
        rows[q] = g.oy + y < p.Y && g.oz + z < p.Z ? m & xmask : 0u;
    }
    __syncwarp();
}

// Element offsets of the (B+1)^3 tile's voxels from the block's first one,
// for one CTA.
__device__ __forceinline__ void row_offsets(const Problem &p, const WPlan &pl, uint32_t *off) {
    const uint32_t B1 = pl.B1, n = B1 * B1 * B1;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t iq = fdiv(i, pl.rB1);
        const uint32_t x = i - iq * B1, z = fdiv(iq, pl.rB1), y = iq - z * B1;
        off[i] = (z * p.Y + y) * p.X + x;
    }
}

// ---------------------------------------------------------------- the list
// Bits of the listed cells, cell q B + x at bit (q B + x) of the units.
template <int BC>
__device__ __forceinline__ void list_bits(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g) {
    const uint32_t lane = threadIdx.x & 31, B = pl.B, B1 = pl.B1;
    const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
    uint32_t *bits = reinterpret_cast<uint32_t *>(ws + pl.off_mm);
    const bool inner = g.ox + B < p.X && g.oy + B < p.Y && g.oz + B < p.Z;
    const uint32_t own = (1u << B) - 1u;
    if constexpr (BC != 8 && BC != 16) {
        for (uint32_t i = lane; i < list_words(B); i += 32) bits[i] = 0;
        __syncwarp();
    }
    for (uint32_t q = lane; q < pl.BB; q += 32) {
        const uint32_t z = fdiv(q, pl.rB), y = q - z * B, at = z * B1 + y;
        const uint32_t r00 = rows[at], r01 = rows[at + 1], r10 = rows[at + B1], r11 = rows[at + B1 + 1];
        const uint32_t all = r00 & r01 & r10 & r11, any = r00 | r01 | r10 | r11;
        uint32_t m = (any | (any >> 1)) & ~(all & (all >> 1)) & own;
        if (!inner) {  // cells need all eight corners in the volume, cut edges both ends
            const bool vy = g.oy + y + 1 < p.Y, vz = g.oz + z + 1 < p.Z;
            const uint32_t xe = p.X - g.ox - 1, vx = xe >= 32 ? 0xffffffffu : (1u << xe) - 1u;
            const uint32_t in = g.oy + y < p.Y && g.oz + z < p.Z ? (vx << 1) | 1u : 0u;  // voxels of the row
            uint32_t cut = (r00 ^ (r00 >> 1)) & vx;
            if (vy) cut |= r00 ^ r01;
            if (vz) cut |= r00 ^ r10;
            m = ((vy && vz ? m & vx : 0u) | (cut & in)) & own;
        }
        if constexpr (BC == 8) {
            reinterpret_cast<uint8_t *>(bits)[q] = (uint8_t)m;
        } else if constexpr (BC == 16) {
            reinterpret_cast<uint16_t *>(bits)[q] = (uint16_t)m;
        } else if (m) {
            const uint32_t b = q * B, w = b >> 5, s = b & 31u;
            atomicOr(&bits[w], m << s);
            if (s + B > 32) atomicOr(&bits[w + 1], m >> (32 - s));
        }
    }
    __syncwarp();
}

// Takes the listed cells in order, up to 32 at a time, from the warp's list.  A
// round turns 32 units of list bits into cells: a warp scan of the units' counts
// gives every lane its place, and each lane writes its own unit's cells.
struct ListWalk {
    uint32_t top = 0, done = 0;  // cells in the list, cells taken from it
    uint32_t next = 0;           // units not looked at
};
// The next n <= 32 cells are list[done + i]; advance done by n after use.  0 at the end.
template <bool BIG>
__device__ __forceinline__ uint32_t list_next(ListWalk &l, const WPlan &pl, unsigned char *ws) {
    const uint32_t lane = threadIdx.x & 31, unit = BIG ? 32u : 16u, nu = (pl.BB * pl.B + unit - 1) / unit;
    uint16_t *list = reinterpret_cast<uint16_t *>(ws + pl.off_list);
    while (l.top - l.done < 32 && l.next < nu) {
        if (BIG) {  // what is left moves to the front
            const uint32_t left = l.top - l.done;
            __syncwarp();
            const uint16_t v = lane < left ? list[l.done + lane] : (uint16_t)0;
            __syncwarp();
            if (lane < left) list[lane] = v;
            l.top = left;
            l.done = 0;
        }
        const uint32_t u = l.next + lane;
        uint32_t b = 0;
        if (u < nu) {
            if (BIG) b = reinterpret_cast<const uint32_t *>(ws + pl.off_mm)[u];
            else b = reinterpret_cast<const uint16_t *>(ws + pl.off_mm)[u];
        }
        uint32_t total;
        uint32_t at = l.top + warp_excl_scan(__popc(b), total);
        for (uint32_t c = u * unit; b; b &= b - 1u, ++at)
            if (MTX_BC(at, list_cap(pl.B), kBcList)) list[at] = (uint16_t)(c + __ffs(b) - 1);
        l.top += total;
        l.next += 32;
        __syncwarp();
    }
    return min(32u, l.top - l.done);
}

// list_next for the block edge BC, or at run time (0).
template <int BC>
__device__ __forceinline__ uint32_t list_take(ListWalk &l, const WPlan &pl, unsigned char *ws) {
    if constexpr (BC != 0) return list_next<(BC > 8)>(l, pl, ws);
    else return pl.B > 8 ? list_next<true>(l, pl, ws) : list_next<false>(l, pl, ws);
}

// A list word: cell (bits 0-11), case (12-19; 0 for a voxel that starts no
// cell), triangles before it in its step of 32 (20-27), cut owned edges (28-30).
__device__ __forceinline__ uint32_t listed_cell(const Problem &p, const WPlan &pl, const Geo &g, const uint32_t *rows,
                                                uint32_t cell, bool inner) {
    const uint32_t q = fdiv(cell, pl.rB), x = cell - q * pl.B, z = fdiv(q, pl.rB), y = q - z * pl.B;
    const uint32_t at = z * pl.B1 + y;
    const uint32_t a = rows[at] >> x, b = rows[at + 1] >> x, c = rows[at + pl.B1] >> x, d = rows[at + pl.B1 + 1] >> x;
    uint32_t cfg = (a & 3u) | ((b & 2u) << 1) | ((b & 1u) << 3) | ((c & 3u) << 4) | ((d & 2u) << 5) | ((d & 1u) << 7);
    uint32_t m = ((a ^ (a >> 1)) & 1u) | (((a ^ b) & 1u) << 1) | (((a ^ c) & 1u) << 2);
    if (!inner) {
        const uint32_t v = (g.ox + x + 1 < p.X ? 1u : 0u) | (g.oy + y + 1 < p.Y ? 2u : 0u) | (g.oz + z + 1 < p.Z ? 4u : 0u);
        m &= v;
        if (v != 7u) cfg = 0;
    }
    return cell | (cfg << 12) | (m << 28);
}

// Vertices of the step's cells before this lane's, and of all 32 (m: this lane's cut owned edges).
__device__ __forceinline__ uint32_t step_vertices(uint32_t m, uint32_t &total) {
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
    const uint32_t b0 = __ballot_sync(0xffffffffu, m & 1u), b1 = __ballot_sync(0xffffffffu, m & 2u),
                   b2 = __ballot_sync(0xffffffffu, m & 4u);
    total = __popc(b0) + __popc(b1) + __popc(b2);
    return __popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt);
}

// ------------------------------------------------------------- count body
// Block whose inside rows are built: list and counts, the face records -- for
// each voxel with x == 0 (index z B + y), y == 0 (BB + z B + x) or z == 0 (2BB +
// y B + x) that owns a vertex, its first vertex in the block (14 bits) and
// whether its x and y edges are cut (bits 14, 15) -- and the state: the list for
// B <= 8, else, or with ROWS, the inside rows.
template <int BC, bool ROWS = false>
__device__ __forceinline__ void count_block_list(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g,
                                                 const uint8_t *ntab, uint8_t *cases_out, mtx_meshlet_descriptor *dr,
                                                 uint16_t *faces, uint32_t *state) {
    const uint32_t lane = threadIdx.x & 31, B = pl.B, BB = pl.BB;
    const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
    const uint16_t *list = reinterpret_cast<const uint16_t *>(ws + pl.off_list);
    uint16_t *fr = reinterpret_cast<uint16_t *>(ws + pl.off_case);
    const bool inner = g.ox + B < p.X && g.oy + B < p.Y && g.oz + B < p.Z;
    for (uint32_t i = lane; i < face_stride16(B) / 8; i += 32) reinterpret_cast<uint4 *>(fr)[i] = make_uint4(0, 0, 0, 0);
    list_bits<BC>(p, pl, ws, g);
    if (cases_out)
        for (uint32_t c = lane; c < BB * B; c += 32) {
            const uint32_t q = fdiv(c, pl.rB), x = c - q * B, z = fdiv(q, pl.rB), y = q - z * B;
            cases_out[c] = cell_valid(p, g, x, y, z) ? (uint8_t)cell_case(rows, pl.B1, x, y, z) : (uint8_t)0;
        }
    if (ROWS || B > 8)
        for (uint32_t i = lane; i < pl.B1 * pl.B1; i += 32) state[i] = rows[i];
    ListWalk l;
    uint32_t nv = 0, nt = 0, steps = 0;
    while (const uint32_t n = list_take<BC>(l, pl, ws)) {
        uint32_t e = 0;
        if (lane < n) e = listed_cell(p, pl, g, rows, list[l.done + lane], inner);
        const uint32_t m = e >> 28, tris = lane < n ? ntab[(e >> 12) & 0xffu] : 0u;
        uint32_t vt, tt;
        const uint32_t rel = nv + step_vertices(m, vt);
        const uint32_t before = warp_excl_scan(tris, tt);
        if (!ROWS && B <= 8 && MTX_BC(steps + lane, list_state_words(B), kBcState)) state[steps + lane] = e | (before << 20);
        steps += 32;
        if (m) {
            const uint32_t cell = e & 0xfffu, q = fdiv(cell, pl.rB), x = cell - q * B, z = fdiv(q, pl.rB), y = q - z * B;
            const uint16_t rec = (uint16_t)(rel | ((m & 3u) << 14));
            if (x == 0 && MTX_BC(z * B + y, BB, kBcFaces)) fr[z * B + y] = rec;
            if (y == 0 && MTX_BC(z * B + x, BB, kBcFaces)) fr[BB + z * B + x] = rec;
            if (z == 0 && MTX_BC(y * B + x, BB, kBcFaces)) fr[2 * BB + y * B + x] = rec;
        }
        nv += vt;
        nt += tt;
        l.done += n;
    }
    __syncwarp();
    for (uint32_t i = lane; i < face_stride16(B) / 8; i += 32)
        reinterpret_cast<uint4 *>(faces)[i] = reinterpret_cast<const uint4 *>(fr)[i];
    if (lane == 0) *reinterpret_cast<uint2 *>(&dr->vertexCount) = make_uint2(nv, nt);
    __syncwarp();
}

// -------------------------------------------------------------- emit body
// Vertex table: for each voxel of the (B+1)^3 tile the first vertex it owns,
// relative to its block's (14 bits), and whether its x and y edges are cut
// (bits 14, 15) -- the face records' form, so that the context layer's entries
// are copies of them.  Which block a corner's voxel belongs to follows from the
// cell: the neighbour in +x / +y / +z exactly where the cell is the block's
// last along that axis and the edge's owner is the cell's far voxel.
constexpr uint32_t kRelMask = 0x3fffu, kCutMask = 0xc000u;

// The CTA's triangle table: three 16-bit corners a triangle, each the owner
// voxel's byte offset in the vertex table from the cell's low corner (bits
// 0-9), its steps along x, y and z (10-12) and the cut bits of the entry that
// count before the corner's axis (14, 15).
__device__ __forceinline__ void build_tris(const WPlan &pl, uint64_t *tri, uint16_t *first) {
    for (uint32_t i = threadIdx.x; i < kTris; i += blockDim.x) {
        const uint32_t e3 = __ldg(&g_mc_tri[i]);
        uint64_t w = 0;
        for (uint32_t k = 0; k < 3; ++k) {
            const uint32_t o = c_mc_owner[(e3 >> (4 * k)) & 0xfu], ax = o >> 3;
            const uint32_t off = (o & 1u) + ((o >> 1) & 1u) * pl.S1 + ((o >> 2) & 1u) * pl.S1 * pl.S1;
            w |= (uint64_t)((off << 1) | ((o & 7u) << 10) | (((1u << ax) - 1u) << 14)) << (16 * k);
        }
        tri[i] = w;
    }
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) first[i] = __ldg(&g_mc_first[i]);
}

// Map entry of context voxel j: the neighbour (bits 0-2), its face record
// (3-12) and the voxel's place in the vertex table (13-25).
__device__ __forceinline__ uint32_t ctx_entry(const WPlan &pl, uint32_t j) {
    const uint32_t B = pl.B, BB = pl.BB;
    uint32_t x, y, z;
    ctx_voxel(pl, j, x, y, z);
    const uint32_t dx = x == B, dy = y == B, dz = z == B;
    const uint32_t lx = dx ? 0 : x, ly = dy ? 0 : y, lz = dz ? 0 : z;
    const uint32_t e = dx ? lz * B + ly : (dy ? BB + lz * B + lx : 2 * BB + ly * B + lx);
    return (dx | (dy << 1) | (dz << 2)) | (e << 3) | (((z * pl.S1 + y) * pl.S1 + x) << 13);
}

// The context layer: face records of the neighbours (nb_rk: lane c holds
// neighbour c's rank or kNoVertex) into the vertex table, loads first.
// B = 8: two records a lane from each of the three faces and the 25 of the
// edges and the corner, four loads a lane in all.
struct Ctx8 {
    uint32_t face[3], edge;
};
__device__ __forceinline__ uint32_t ctx8_edge(uint32_t lane) {  // map entry (ctx_entry) of the lane's edge voxel
    const uint32_t k = lane & 7u;
    if (lane < 8) return 3u | ((8 * k) << 3) | (((k * 9 + 8) * 9 + 8) << 13);
    if (lane < 16) return 5u | (k << 3) | (((8 * 9 + k) * 9 + 8) << 13);
    if (lane < 24) return 6u | ((64 + k) << 3) | (((8 * 9 + 8) * 9 + k) << 13);
    return lane == 24 ? 7u | (728u << 13) : 0u;
}
// NC: the records come from an earlier launch (ld_in).
template <bool NC = true>
__device__ __forceinline__ Ctx8 ctx8_load(const uint16_t *faces, uint32_t nb_rk, uint32_t edge, uint64_t face_words) {
    const uint32_t lane = threadIdx.x & 31;
    Ctx8 c;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const uint32_t rk = __shfl_sync(0xffffffffu, nb_rk, 1 << f);
        const uint64_t at = (uint64_t)rk * 192 + 64 * f + 2 * lane;
        c.face[f] = 0;
        if (rk != kNoVertex && MTX_BC(at + 1, face_words, kBcFaces))
            c.face[f] = ld_in<NC>(reinterpret_cast<const uint32_t *>(faces + at));
    }
    const uint32_t rk = __shfl_sync(0xffffffffu, nb_rk, edge & 7u);
    const uint64_t at = (uint64_t)rk * 192 + ((edge >> 3) & 1023u);
    c.edge = 0;
    if (edge && rk != kNoVertex && MTX_BC(at, face_words, kBcFaces)) c.edge = ld_in<NC>(faces + at);
    return c;
}
__device__ __forceinline__ void ctx8_store(const Ctx8 &c, uint32_t edge, uint16_t *vtab) {
    const uint32_t lane = threadIdx.x & 31, u = lane >> 2, v = 2 * (lane & 3u);
    uint16_t *x = vtab + (u * 9 + v) * 9 + 8, *y = vtab + (u * 9 + 8) * 9 + v, *z = vtab + (8 * 9 + u) * 9 + v;
    x[0] = (uint16_t)c.face[0];
    x[9] = (uint16_t)(c.face[0] >> 16);
    y[0] = (uint16_t)c.face[1];
    y[1] = (uint16_t)(c.face[1] >> 16);
    z[0] = (uint16_t)c.face[2];
    z[1] = (uint16_t)(c.face[2] >> 16);
    if (edge && MTX_BC(edge >> 13, 9 * 9 * 9, kBcVoxTab)) vtab[edge >> 13] = (uint16_t)c.edge;
}

// Any B, through the map: up to 32 N context voxels from j0 on.
template <int N>
__device__ __forceinline__ void ctx_load(const WPlan &pl, const uint16_t *faces, uint32_t nb_rk, const uint32_t *cmap,
                                         uint32_t j0, uint32_t rec[N], uint64_t face_words) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t j = j0 + 32 * k + lane;
        rec[k] = 0;
        if (j0 + 32 * k >= pl.nb3) continue;  // uniform
        const uint32_t c = cmap[min(j, pl.nb3 - 1)];
        const uint32_t rk = __shfl_sync(0xffffffffu, nb_rk, c & 7u);
        const uint64_t at = (uint64_t)rk * face_stride16(pl.B) + ((c >> 3) & 1023u);
        if (j < pl.nb3 && rk != kNoVertex && MTX_BC((c >> 3) & 1023u, 3 * pl.BB, kBcContext) &&
            MTX_BC(at, face_words, kBcFaces))
            rec[k] = __ldg(faces + at);
    }
}
template <int N>
__device__ __forceinline__ void ctx_store(const WPlan &pl, uint16_t *vtab, const uint32_t *cmap, uint32_t j0,
                                          const uint32_t rec[N]) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t j = j0 + 32 * k + lane;
        if (j < pl.nb3 && MTX_BC(cmap[j] >> 13, pl.B1 * pl.B1 * pl.B1, kBcVoxTab)) vtab[cmap[j] >> 13] = (uint16_t)rec[k];
    }
}

// One step of the vertex phase: this lane's list word e (0: none) and its first
// vertex rel -> the voxel's table entry, and a job (cell | axis << 12) for each
// of its vertices, queued at the vertex's own number.  done: vertices written,
// or all before this step where none are (the jobs are not read then).
__device__ __forceinline__ void queue_vertices(const WPlan &pl, uint32_t e, uint32_t rel, uint16_t *vtab,
                                               uint32_t *jobs, [[maybe_unused]] uint32_t done) {
    const uint32_t m = e >> 28, cell = e & 0xfffu;
    if (!m) return;
    const uint32_t q = fdiv(cell, pl.rB), x = cell - q * pl.B, z = fdiv(q, pl.rB), y = q - z * pl.B;
    const uint32_t ti = (z * pl.S1 + y) * pl.S1 + x;
    if (MTX_BC(ti, pl.S1 * pl.S1 * pl.S1, kBcVoxTab)) vtab[ti] = (uint16_t)(rel | (m << 14));
    if (!MTX_BC(rel + __popc(m) - 1 - done, kJobWin, kBcJobs)) return;
    if (m & 1u) jobs[rel++ & (kJobWin - 1)] = cell;
    if (m & 2u) jobs[rel++ & (kJobWin - 1)] = cell | (1u << 12);
    if (m & 4u) jobs[rel & (kJobWin - 1)] = cell | (2u << 12);
}

// A voxel's value; AnyVoxel: of the volume's run-time type.
struct AnyVoxel {};
template <typename T>
__device__ __forceinline__ float voxel_value(const Problem &p, uint64_t i) {
    if constexpr (std::is_same<T, AnyVoxel>::value) {
        if (p.dtype == MTX_DTYPE_U8) return Vox<uint8_t>::val(__ldg(reinterpret_cast<const uint8_t *>(p.vol) + i));
        if (p.dtype == MTX_DTYPE_U16) return Vox<uint16_t>::val(__ldg(reinterpret_cast<const uint16_t *>(p.vol) + i));
        return __ldg(reinterpret_cast<const float *>(p.vol) + i);
    } else {
        return Vox<T>::val(__ldg(reinterpret_cast<const T *>(p.vol) + i));
    }
}

// Writes vertices [done, done + n) of the block's nv, n <= 32, one a lane; the
// first is vertex vbase of the mesh.
template <typename T, bool GENERIC>
__device__ __forceinline__ void put_vertices(const Problem &p, const WPlan &pl, const Geo &g, const uint32_t *jobs,
                                             uint32_t done, uint32_t n, [[maybe_unused]] uint32_t nv, bool inner,
                                             void *vertices, uint64_t vbase, uint32_t vfmt, uint32_t frame,
                                             uint32_t normals) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t job = jobs[(done + lane) & (kJobWin - 1)];
    const uint32_t cell = job & 0xfffu, a = job >> 12;
    const uint32_t q = fdiv(cell, pl.rB), x = cell - q * pl.B, z = fdiv(q, pl.rB), y = q - z * pl.B;
    const uint32_t gx = g.ox + x, gy = g.oy + y, gz = g.oz + z;
    // (a list the count pass did not finish must not lead past the volume)
    if (lane < n && MTX_BC(done + lane, nv, kBcVertex) &&
        (inner || (gx + (a == 0) < p.X && gy + (a == 1) < p.Y && gz + (a == 2) < p.Z))) {
        const uint64_t v = ((uint64_t)gz * p.Y + gy) * p.X + gx;
        const uint64_t step = a == 0 ? 1ull : a == 1 ? (uint64_t)p.X : (uint64_t)p.X * p.Y;
        const float t = edge_t(voxel_value<T>(p, v), voxel_value<T>(p, v + step), p.iso);
        float3 pos = make_float3((float)gx, (float)gy, (float)gz);
        if (a == 0) pos.x = __fadd_rn(pos.x, t);
        if (a == 1) pos.y = __fadd_rn(pos.y, t);
        if (a == 2) pos.z = __fadd_rn(pos.z, t);
        if (GENERIC && frame == MTX_FRAME_NDC) {
            pos.x = __fsub_rn(__fmul_rn(__fdiv_rn(pos.x, (float)p.X), 2.0f), 1.0f);
            pos.y = __fsub_rn(__fmul_rn(__fdiv_rn(pos.y, (float)p.Y), 2.0f), 1.0f);
            pos.z = __fsub_rn(__fmul_rn(__fdiv_rn(pos.z, (float)p.Z), 2.0f), 1.0f);
        }
        const uint64_t at = vbase + done + lane;
        if (!GENERIC || vfmt == MTX_VERTEX_XYZ) {  // each lane its own 12 bytes: L2 merges the warp's span
            float *o = reinterpret_cast<float *>(vertices) + 3 * at;
            o[0] = pos.x;
            o[1] = pos.y;
            o[2] = pos.z;
        } else {
            float3 nn = make_float3(0.0f, 0.0f, 0.0f);
            if (normals) {
                if constexpr (std::is_same<T, AnyVoxel>::value) nn = vertex_normal_any(p, gx, gy, gz, a, t);
                else nn = vertex_normal<T>(p, gx, gy, gz, a, t);
            }
            float4 *o = reinterpret_cast<float4 *>(vertices) + 2 * at;
            o[0] = make_float4(pos.x, pos.y, pos.z, 1.0f);
            o[1] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        }
    }
    __syncwarp();
}

// Queues the triangles of this lane's list word e, numbers [at, at + n) of the
// block, of which `done` are written; f: the entry of its case in `first`.
__device__ __forceinline__ void queue_triangles(const WPlan &pl, uint32_t e, uint32_t f, uint32_t at, uint32_t *jobs,
                                                [[maybe_unused]] uint32_t done) {
    const uint32_t cell = e & 0xfffu, n = f >> 12, q = fdiv(cell, pl.rB), x = cell - q * pl.B;
    const uint32_t z = fdiv(q, pl.rB), y = q - z * pl.B;
    const uint32_t end =
        (x + 1 == pl.B ? 1u << 26 : 0u) | (y + 1 == pl.B ? 1u << 27 : 0u) | (z + 1 == pl.B ? 1u << 28 : 0u);
    const uint32_t job = (((z * pl.S1 + y) * pl.S1 + x) << 1) | ((f & 0xfffu) << 16) | end;
#pragma unroll
    for (uint32_t t = 0; t < 5; ++t)  // at most five triangles a case
        if (t < n && MTX_BC(at + t - done, kJobWin, kBcJobs)) jobs[(at + t) & (kJobWin - 1)] = job + (t << 16);
}

// Writes triangles [done, done + n) of the block's nt, n <= 32, one a lane, each
// lane its own 12 bytes from dst on.  Job: the cell's byte offset in the vertex table
// (bits 0-15), the triangle (16-25), whether the cell is the block's last along
// x, y and z (26-28).  miss: bit c, neighbour c is not active.
__device__ __forceinline__ void put_triangles(const WPlan &pl, const unsigned char *vtab, const uint64_t *tri,
                                              const uint32_t *jobs, const uint32_t *nbase, uint32_t done, uint32_t n,
                                              [[maybe_unused]] uint32_t nt, uint32_t *dst, uint32_t miss, bool &bad) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane < n && MTX_BC(done + lane, nt, kBcIndex)) {
        const uint32_t job = jobs[(done + lane) & (kJobWin - 1)];
        const uint64_t w = MTX_BC((job >> 16) & 0x3ffu, kTris, kBcJobs) ? tri[(job >> 16) & 0x3ffu] : 0ull;
        const uint32_t ti = job & 0xffffu, c[3] = {(uint32_t)w, (uint32_t)w >> 16, (uint32_t)(w >> 32)};
        uint32_t id[3], from = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t e = MTX_BC(ti + (c[k] & 0x3ffu), 2 * pl.S1 * pl.S1 * pl.S1, kBcVoxTab)
                                   ? *reinterpret_cast<const uint16_t *>(vtab + ti + (c[k] & 0x3ffu))
                                   : 0u;
            const uint32_t b = (c[k] >> 10) & (job >> 26) & 7u;
            id[k] = nbase[b] + (e & kRelMask) + __popc(e & c[k] & kCutMask);
            from |= miss >> b;
        }
        bad |= from & 1u;
        uint32_t *o = dst + 3ull * (done + lane);
        o[0] = id[0];
        o[1] = id[1];
        o[2] = id[2];
    }
    __syncwarp();
}

}  // namespace mtx
