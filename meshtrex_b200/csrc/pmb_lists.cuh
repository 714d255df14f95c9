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

#include "pmb_device.cuh"

namespace mtx {

// Triangles of every case in case order: three edge numbers, 4 bits each; and
// of each case the first of its triangles | their number << 12.
constexpr uint32_t kTris = 820;
static __device__ uint16_t g_mc_tri[kTris];
static __device__ uint16_t g_mc_first[256];

static mtx_status load_list_tables(mtx_context *c) {
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
constexpr uint32_t kListRing = 64;  // listed cells not yet taken: fewer than 32, and a word's 32

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
    p.BB = B * B;
    p.nb3 = 3 * B * B + 3 * B + 1;
    p.rB = (uint32_t)((0x100000000ull + B - 1) / B);
    p.rB1 = (uint32_t)((0x100000000ull + B) / (B + 1));
    p.rBB = (uint32_t)((0x100000000ull + B * B - 1) / (B * B));
    p.R = 32 / B;
    p.nbuf = 1;
}

// A warp's shared memory in the count pass: TMA tile and barrier, inside rows,
// list bits, ring, face records (which share the region of the plain loads'
// bitstream: that is dead once the rows are built).
__host__ __device__ inline WPlan make_count_plan(uint32_t B, uint32_t esz, bool tma) {
    WPlan p{};
    plan_block(p, B);
    uint32_t o = 0;
    p.off_tile[0] = p.off_tile[1] = 0;
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
    p.off_list = o;  // ring
    o = align_up(o + 2 * kListRing, 16);
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
// its seven neighbours, and for B > 8 the inside rows, list bits and ring.
__host__ __device__ inline WPlan make_emit_plan(uint32_t B) {
    WPlan p{};
    plan_block(p, B);
    uint32_t o = 0;
    p.off_jobs = o;
    o += 4 * kJobWin;
    p.off_nvid = o;
    o += 32;
    p.off_vtab = o;
    o = align_up(o + (B <= 8 ? 2 : 4) * p.B1 * p.B1 * p.B1, 16);
    if (B > 8) {
        p.off_rows = o;
        o = align_up(o + 4 * p.B1 * p.B1, 16);
        p.off_mm = o;
        o = align_up(o + 4 * list_words(B), 16);
        p.off_list = o;
        o = align_up(o + 2 * kListRing, 16);
    }
    p.bytes = align_up(o, 16);
    return p;
}

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
template <typename T, int BC>
__device__ __forceinline__ void load_rows(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g,
                                          const uint32_t *off) {
    constexpr uint32_t kBatch = 8;
    const T *vol = reinterpret_cast<const T *>(p.vol);
    uint32_t *words = reinterpret_cast<uint32_t *>(ws + pl.off_case);
    uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
    const uint32_t lane = threadIdx.x & 31, B1 = pl.B1, n = B1 * B1 * B1, nw = (n + 31) / 32;
    const bool inner = g.ox + pl.B < p.X && g.oy + pl.B < p.Y && g.oz + pl.B < p.Z;
    const T *base = vol + ((uint64_t)g.oz * p.Y + g.oy) * p.X + g.ox;
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
// Bits of the listed cells, cell q B + x at bit (q B + x) of the word array.
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

// Takes the listed cells in order, up to 32 at a time.
struct ListWalk {
    uint32_t top = 0, done = 0;          // cells put into the ring, cells taken out of it
    uint32_t next = 0, group = 0, nz = 0;  // words not looked at, the 32 words held, those with cells left
    uint32_t word = 0;                   // this lane's word of the 32 held
};
// The next n <= 32 cells are ring[(done + i) & 63]; advance done by n after use.  0 at the end.
__device__ __forceinline__ uint32_t list_next(ListWalk &l, const WPlan &pl, unsigned char *ws) {
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u, nw = list_words(pl.B);
    const uint32_t *bits = reinterpret_cast<const uint32_t *>(ws + pl.off_mm);
    uint16_t *ring = reinterpret_cast<uint16_t *>(ws + pl.off_list);
    __syncwarp();
    while (l.top - l.done < 32) {
        if (!l.nz) {
            if (l.next >= nw) break;
            l.group = l.next;
            l.word = l.group + lane < nw ? bits[l.group + lane] : 0u;
            l.nz = __ballot_sync(0xffffffffu, l.word != 0);
            l.next += 32;
            continue;
        }
        const uint32_t k = __ffs(l.nz) - 1;
        l.nz &= l.nz - 1u;
        const uint32_t w = __shfl_sync(0xffffffffu, l.word, k);
        if ((w >> lane) & 1u) ring[(l.top + __popc(w & lt)) & (kListRing - 1)] = (uint16_t)((l.group + k) * 32 + lane);
        l.top += __popc(w);
    }
    __syncwarp();
    return min(32u, l.top - l.done);
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
// whether its x and y edges are cut (bits 14, 15) -- and the state.
template <int BC>
__device__ __forceinline__ void count_block_list(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g,
                                                 const uint8_t *ntab, uint8_t *cases_out, mtx_meshlet_descriptor *dr,
                                                 uint16_t *faces, uint32_t *state) {
    const uint32_t lane = threadIdx.x & 31, B = pl.B, BB = pl.BB;
    const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
    const uint16_t *ring = reinterpret_cast<const uint16_t *>(ws + pl.off_list);
    uint16_t *fr = reinterpret_cast<uint16_t *>(ws + pl.off_case);
    const bool inner = g.ox + B < p.X && g.oy + B < p.Y && g.oz + B < p.Z;
    for (uint32_t i = lane; i < face_stride16(B) / 8; i += 32) reinterpret_cast<uint4 *>(fr)[i] = make_uint4(0, 0, 0, 0);
    list_bits<BC>(p, pl, ws, g);
    if (cases_out)
        for (uint32_t c = lane; c < BB * B; c += 32) {
            const uint32_t q = fdiv(c, pl.rB), x = c - q * B, z = fdiv(q, pl.rB), y = q - z * B;
            cases_out[c] = cell_valid(p, g, x, y, z) ? (uint8_t)cell_case(rows, pl.B1, x, y, z) : (uint8_t)0;
        }
    if (B > 8)
        for (uint32_t i = lane; i < pl.B1 * pl.B1; i += 32) state[i] = rows[i];
    ListWalk l;
    uint32_t nv = 0, nt = 0;
    while (const uint32_t n = list_next(l, pl, ws)) {
        uint32_t e = 0;
        if (lane < n) e = listed_cell(p, pl, g, rows, ring[(l.done + lane) & (kListRing - 1)], inner);
        const uint32_t m = e >> 28, tris = lane < n ? ntab[(e >> 12) & 0xffu] : 0u;
        uint32_t vt, tt;
        const uint32_t rel = nv + step_vertices(m, vt);
        const uint32_t before = warp_excl_scan(tris, tt);
        if (B <= 8 && MTX_BC(l.done + lane, list_state_words(B), kBcState)) state[l.done + lane] = e | (before << 20);
        if (m) {
            const uint32_t cell = e & 0xfffu, q = fdiv(cell, pl.rB), x = cell - q * B, z = fdiv(q, pl.rB), y = q - z * B;
            const uint16_t rec = (uint16_t)(rel | ((m & 3u) << 14));
            if (x == 0) fr[z * B + y] = rec;
            if (y == 0) fr[BB + z * B + x] = rec;
            if (z == 0) fr[2 * BB + y * B + x] = rec;
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
// Entry of the vertex table, one a voxel of the (B+1)^3 tile: the voxel's
// first vertex relative to its block's, whether its x and y edges are cut, and
// the block (0 = this one, 1-7 the +x/+y/+z neighbour dx | dy << 1 | dz << 2).
// 16 bits for B <= 8 (11 + 2 + 3), else 32 (14 + 2 + 3).
template <bool BIG> struct VEntry;
template <> struct VEntry<false> {
    using E = uint16_t;
    static constexpr uint32_t kRel = 11, kShift = 1;  // log2 of the entry's bytes
};
template <> struct VEntry<true> {
    using E = uint32_t;
    static constexpr uint32_t kRel = 14, kShift = 2;
};

// The CTA's triangle table: three 16-bit corners a triangle, each the owner
// voxel's byte offset in the vertex table from the cell's low corner, and the
// two edge bits of the entry that count before the corner's axis.
template <bool BIG>
__device__ __forceinline__ void build_tris(const WPlan &pl, uint64_t *tri, uint16_t *first) {
    constexpr uint32_t kRel = VEntry<BIG>::kRel, kShift = VEntry<BIG>::kShift;
    for (uint32_t i = threadIdx.x; i < kTris; i += blockDim.x) {
        const uint32_t e3 = __ldg(&g_mc_tri[i]);
        uint64_t w = 0;
        for (uint32_t k = 0; k < 3; ++k) {
            const uint32_t o = c_mc_owner[(e3 >> (4 * k)) & 0xfu], ax = o >> 3;
            const uint32_t off = (o & 1u) + ((o >> 1) & 1u) * pl.B1 + ((o >> 2) & 1u) * pl.B1 * pl.B1;
            w |= (uint64_t)((off << kShift) | (((1u << ax) - 1u) << kRel)) << (16 * k);
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
    return (dx | (dy << 1) | (dz << 2)) | (e << 3) | (((z * pl.B1 + y) * pl.B1 + x) << 13);
}

// Face records of up to 32 N context voxels from j0 on, all loads issued; nb_rk: lane c
// holds neighbour c's rank or kNoVertex.
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
        if (j < pl.nb3 && rk != kNoVertex && MTX_BC(at, face_words, kBcFaces)) rec[k] = __ldg(faces + at);
    }
}

template <bool BIG, int N>
__device__ __forceinline__ void ctx_store(const WPlan &pl, typename VEntry<BIG>::E *vtab, const uint32_t *cmap,
                                          uint32_t j0, const uint32_t rec[N]) {
    constexpr uint32_t kRel = VEntry<BIG>::kRel;
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t j = j0 + 32 * k + lane;
        if (j < pl.nb3) {
            const uint32_t c = cmap[j];
            if (MTX_BC(c >> 13, pl.B1 * pl.B1 * pl.B1, kBcVoxTab))
                vtab[c >> 13] = (typename VEntry<BIG>::E)((rec[k] & ((1u << kRel) - 1u)) | ((rec[k] >> 14) << kRel) |
                                                          ((c & 7u) << (kRel + 2)));
        }
    }
}

// Writes vertex `at` on the +A edge of voxel (gx, gy, gz) whose value is fa and
// whose neighbour's is fb.
template <typename T, bool GENERIC, int A>
__device__ __forceinline__ void put_vertex(const Problem &p, uint32_t gx, uint32_t gy, uint32_t gz, float fa, float fb,
                                           void *vertices, uint64_t at, uint32_t vfmt, uint32_t frame,
                                           uint32_t normals) {
    const float t = edge_t(fa, fb, p.iso);
    float3 pos = make_float3((float)gx, (float)gy, (float)gz);
    if (A == 0) pos.x = __fadd_rn(pos.x, t);
    if (A == 1) pos.y = __fadd_rn(pos.y, t);
    if (A == 2) pos.z = __fadd_rn(pos.z, t);
    if (GENERIC && frame == MTX_FRAME_NDC) {
        pos.x = __fsub_rn(__fmul_rn(__fdiv_rn(pos.x, (float)p.X), 2.0f), 1.0f);
        pos.y = __fsub_rn(__fmul_rn(__fdiv_rn(pos.y, (float)p.Y), 2.0f), 1.0f);
        pos.z = __fsub_rn(__fmul_rn(__fdiv_rn(pos.z, (float)p.Z), 2.0f), 1.0f);
    }
    if (!GENERIC || vfmt == MTX_VERTEX_XYZ) {  // each lane its own 12 bytes: L2 merges the warp's span
        float *o = reinterpret_cast<float *>(vertices) + 3 * at;
        o[0] = pos.x;
        o[1] = pos.y;
        o[2] = pos.z;
    } else {
        float3 nn = make_float3(0.0f, 0.0f, 0.0f);
        if (normals) nn = vertex_normal<T>(p, gx, gy, gz, A, t);
        float4 *v = reinterpret_cast<float4 *>(vertices) + 2 * at;
        v[0] = make_float4(pos.x, pos.y, pos.z, 1.0f);
        v[1] = make_float4(nn.x, nn.y, nn.z, 0.0f);
    }
}

// One step of the vertex phase: this lane's list word e (0: none) and its
// first vertex rel -> the voxel's table entry and its vertices.
template <typename T, bool GENERIC, bool BIG>
__device__ __forceinline__ void emit_step_vertices(const Problem &p, const WPlan &pl, const Geo &g, uint32_t e,
                                                   uint32_t rel, typename VEntry<BIG>::E *vtab, void *vertices,
                                                   uint64_t vbase, uint32_t nv, uint32_t vfmt, uint32_t frame,
                                                   uint32_t normals) {
    const uint32_t m = e >> 28;
    if (!m) return;
    const uint32_t cell = e & 0xfffu, q = fdiv(cell, pl.rB), x = cell - q * pl.B, z = fdiv(q, pl.rB), y = q - z * pl.B;
    const uint32_t ti = (z * pl.B1 + y) * pl.B1 + x;
    if (MTX_BC(ti, pl.B1 * pl.B1 * pl.B1, kBcVoxTab))
        vtab[ti] = (typename VEntry<BIG>::E)(rel | ((m & 3u) << VEntry<BIG>::kRel));
    if (!vertices || rel + __popc(m) > nv) return;
    const uint32_t gx = g.ox + x, gy = g.oy + y, gz = g.oz + z;
    const T *v = reinterpret_cast<const T *>(p.vol) + ((uint64_t)gz * p.Y + gy) * p.X + gx;
    // the voxel and its cut neighbours, all loads in flight
    const T a = __ldg(v), bx = m & 1u ? __ldg(v + 1) : T(0), by = m & 2u ? __ldg(v + p.X) : T(0),
            bz = m & 4u ? __ldg(v + (uint64_t)p.X * p.Y) : T(0);
    const float fa = Vox<T>::val(a);
    uint64_t at = vbase + rel;
    if (m & 1u) put_vertex<T, GENERIC, 0>(p, gx, gy, gz, fa, Vox<T>::val(bx), vertices, at++, vfmt, frame, normals);
    if (m & 2u) put_vertex<T, GENERIC, 1>(p, gx, gy, gz, fa, Vox<T>::val(by), vertices, at++, vfmt, frame, normals);
    if (m & 4u) put_vertex<T, GENERIC, 2>(p, gx, gy, gz, fa, Vox<T>::val(bz), vertices, at, vfmt, frame, normals);
}

// Resolves triangle jobs [done, done + n), n <= 32, one a lane, each lane storing its own 12 bytes.
template <bool BIG>
__device__ __forceinline__ void put_triangles(const unsigned char *vtab, const uint64_t *tri, const uint32_t *jobs,
                                              const uint32_t *nbase, uint32_t done, uint32_t n, uint32_t *dst,
                                              uint32_t miss, bool &bad) {
    using V = VEntry<BIG>;
    using E = typename V::E;
    constexpr uint32_t kOff = (1u << V::kRel) - 1u, kCut = 3u << V::kRel;
    const uint32_t lane = threadIdx.x & 31;
    if (lane < n) {
        const uint32_t job = jobs[(done + lane) & (kJobWin - 1)];
        const uint64_t w = tri[job >> 16];
        const uint32_t ti = job & 0xffffu, c[3] = {(uint32_t)w, (uint32_t)w >> 16, (uint32_t)(w >> 32)};
        uint32_t id[3], from = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t e = *reinterpret_cast<const E *>(vtab + ti + (c[k] & kOff));
            const uint32_t b = (e >> (V::kRel + 2)) & 7u;
            id[k] = nbase[b] + (e & kOff) + __popc(e & c[k] & kCut);
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
