// Device building blocks of the PMB marching-cubes passes, shared by the
// single-volume kernels (extract.cu), the batched kernel (batched.cu) and the
// adjoint: per-warp shared-memory plans, tile staging, inside bitmasks, PMB
// edge ownership by bit operations, and the decoupled look-back used by the
// scans.
//
// Output order is canonical and equals the CPU oracle's: vertices by (block
// rank, owner voxel x-fastest in the block, axis x<y<z); triangles by (block
// rank, cell x-fastest in the block, triangle number in the case).
#pragma once

#include <algorithm>
#include <cstring>

#include "mtx_internal.h"

namespace mtx {

// Each translation unit has its own copy (no relocatable device code); load
// them with load_case_tables() before the first launch from that unit.
static __constant__ uint64_t c_mc_cases[256];
static __constant__ uint8_t c_mc_owner[12];

static mtx_status load_case_tables(mtx_context *c) {
    static bool loaded[128] = {false};
    if (c->device >= 0 && c->device < 128 && loaded[c->device]) return MTX_OK;
    MTX_CUDA(c, cudaMemcpyToSymbol(c_mc_cases, MTX_MC_CASES, sizeof(MTX_MC_CASES)));
    MTX_CUDA(c, cudaMemcpyToSymbol(c_mc_owner, MTX_MC_EDGE_OWNER, sizeof(MTX_MC_EDGE_OWNER)));
    if (c->device >= 0 && c->device < 128) loaded[c->device] = true;
    return MTX_OK;
}

constexpr uint32_t kNoVertex = 0xffffffffu;
constexpr uint32_t kJobWin = 256;                   // jobs (vertices or triangles) resolved per window
constexpr int kMaxWarps = 8;                        // warps per CTA of the extraction kernels

__host__ __device__ inline uint32_t align_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// ------------------------------------------------------- per-warp smem plan
struct WPlan {
    uint32_t B, B1, BB, PX, nb3;
    uint32_t S1;       // row of the vertex table: B + 1, or in a batch the largest block edge + 1
    uint32_t rB, rB1;  // ceil(2^32 / d) reciprocals: n / d == __umulhi(n, r) for the sizes used here
    uint32_t off_tile, off_bar, off_rows, off_vp, off_nvid, off_jobs;
    uint32_t off_case, off_mm;  // face records and bitstream, list bits
    uint32_t off_vtab, off_list;
    uint32_t bytes;       // per warp
    uint32_t tile_bytes;  // one tile (the TMA transaction size)
};

__host__ __device__ inline uint32_t tile_pitch(uint32_t B, uint32_t esz, bool tma) {
    if (!tma) return B + 1;
    const uint32_t A = 16 / esz;  // elements per 16 bytes
    uint32_t g = 1;
    for (uint32_t d = 1; d <= A; ++d)
        if (B % d == 0 && A % d == 0) g = d;
    const uint32_t xoff_max = (B % A == 0) ? 0 : A - g;
    return align_up(xoff_max + B + 1, A);
}

// n / d for the block-local sizes (n < 70000, 2 <= d < 300), exact.
__device__ __forceinline__ uint32_t fdiv(uint32_t n, uint32_t r) { return __umulhi(n, r); }

struct Geo {
    uint32_t ox, oy, oz;  // block origin (voxels)
    uint32_t bx, by, bz;
    uint32_t nx;          // voxels of the block inside the volume along x (<= B)
    uint32_t xoff;        // tile column of the block's first voxel
};

// Exact division of a block id by the grid's row and slice sizes through a
// 64-bit reciprocal and one high multiply (Lemire's method: m = floor((2^64 - 1)
// / d) + 1 gives floor(a / d) = high 64 bits of m * a for every 32-bit a; d = 1
// is taken apart), computed once per thread instead of two integer divisions
// per block.
struct GridDiv {
    uint64_t mx, mxy;
    uint32_t dx, dxy;
};
__host__ __device__ inline GridDiv grid_div(const Problem &p) {
    GridDiv d;
    d.dx = p.GX;
    d.dxy = p.GX * p.GY;
    d.mx = d.dx > 1 ? ~0ull / d.dx + 1 : 0;
    d.mxy = d.dxy > 1 ? ~0ull / d.dxy + 1 : 0;
    return d;
}
__device__ __forceinline__ uint32_t div_by(uint32_t a, uint64_t m, uint32_t d) {
    return d > 1 ? (uint32_t)__umul64hi(m, a) : a;
}

__device__ __forceinline__ Geo block_geo(uint32_t id, const Problem &p, bool tma, uint32_t esz, const GridDiv &dv) {
    Geo g;
    g.bz = div_by(id, dv.mxy, dv.dxy);
    const uint32_t rest = id - g.bz * dv.dxy;
    g.by = div_by(rest, dv.mx, dv.dx);
    g.bx = rest - g.by * dv.dx;
    g.ox = g.bx * p.B;
    g.oy = g.by * p.B;
    g.oz = g.bz * p.B;
    g.nx = min(p.B, p.X - g.ox);
    g.xoff = tma ? (g.ox % (16 / esz)) : 0u;
    return g;
}

// ----------------------------------------------------------- warp tiles
// Starts the TMA load of a block's (B+1)^3 tile (zero fill outside the volume):
// lane 0 issues one cp.async.bulk.tensor.
template <typename T>
__device__ __forceinline__ void tile_issue(const WPlan &pl, unsigned char *ws, const Geo &g, const CUtensorMap *map) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        uint64_t *bar = reinterpret_cast<uint64_t *>(ws + pl.off_bar);
        fence_proxy_async();  // earlier generic reads of the tile come first
        mbar_arrive_expect_tx(bar, pl.tile_bytes);
        tma_load_3d(ws + pl.off_tile, map, bar, (int)(g.ox - g.xoff), (int)g.oy, (int)g.oz);
    }
}

__device__ __forceinline__ bool tile_wait(const WPlan &pl, unsigned char *ws, const Geo &g, uint32_t &parity,
                                          DevStatus *st) {
    uint64_t *bar = reinterpret_cast<uint64_t *>(ws + pl.off_bar);
    const bool ok = mbar_wait_bounded(bar, parity);
    if (!__all_sync(0xffffffffu, ok)) {
        if ((threadIdx.x & 31) == 0) report(st, MTX_ERR_TIMEOUT, kSiteTmaWait, g.ox, g.oy);
        // give the copy in flight one more bounded wait before the warp leaves
        mbar_wait_bounded(bar, parity);
        return false;
    }
    parity ^= 1u;
    return true;
}

// Inside bitmask of every tile row: bit x <=> voxel at or below iso and inside
// the volume.  Integer voxels compare against floor(iso); rows that start on a
// 4-byte boundary are tested 2 (uint16) or 4 (uint8) voxels per instruction.
template <typename T>
__device__ __forceinline__ void build_rows(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g) {
    const T *tile = reinterpret_cast<const T *>(ws + pl.off_tile);
    uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
    const uint32_t xin = min(pl.B1, p.X - g.ox);
    const uint32_t xmask = (1u << xin) - 1u;  // xin <= 17
    // integer voxels: value <= iso  <=>  value <= floor(iso) (never when iso < 0 or NaN)
    const bool never = !(p.iso >= 0.0f);
    const uint32_t thr = never ? 0u : (uint32_t)fminf(floorf(p.iso), sizeof(T) == 1 ? 255.0f : 65535.0f);
    const bool simd = Vox<T>::code != 2 && ((pl.PX * sizeof(T)) % 4 == 0) && ((g.xoff * sizeof(T)) % 4 == 0);
    for (uint32_t q = threadIdx.x & 31; q < pl.B1 * pl.B1; q += 32) {
        const uint32_t z = fdiv(q, pl.rB1), y = q - z * pl.B1;
        uint32_t m = 0;
        if (g.oy + y < p.Y && g.oz + z < p.Z &&
            MTX_BC((z * pl.B1 + y) * pl.PX + g.xoff + xin, pl.PX * pl.B1 * pl.B1 + 1, kBcTile)) {
            const T *r = tile + (z * pl.B1 + y) * pl.PX + g.xoff;
            if (Vox<T>::code == 2) {
                for (uint32_t x = 0; x < xin; ++x) m |= (Vox<T>::val(r[x]) <= p.iso ? 1u : 0u) << x;
            } else if (never) {
                m = 0;
            } else if (simd && sizeof(T) == 2) {
                const uint32_t *w = reinterpret_cast<const uint32_t *>(r);
                const uint32_t t2 = thr | (thr << 16);
                for (uint32_t i = 0; 2 * i < xin; ++i) {
                    const uint32_t c = __vcmpleu2(w[i], t2) & 0x00010001u;
                    m |= ((c | (c >> 15)) & 3u) << (2 * i);
                }
                m &= xmask;
            } else if (simd && sizeof(T) == 1) {
                const uint32_t *w = reinterpret_cast<const uint32_t *>(r);
                const uint32_t t4 = thr * 0x01010101u;
                for (uint32_t i = 0; 4 * i < xin; ++i) {
                    const uint32_t c = __vcmpleu4(w[i], t4) & 0x01010101u;
                    m |= ((c * 0x01020408u) >> 24) << (4 * i);
                }
                m &= xmask;
            } else {
                for (uint32_t x = 0; x < xin; ++x) m |= ((uint32_t)r[x] <= thr ? 1u : 0u) << x;
            }
        }
        if (MTX_BC(q, pl.B1 * pl.B1, kBcRows)) rows[q] = m;
    }
    __syncwarp();
}

// Crossing masks of owned voxel row (y, z) (bit x of xc/yc/zc: the +x/+y/+z
// edge owned by voxel (x, y, z) is cut) from the inside bitmasks.
__device__ __forceinline__ void row_cross(const Problem &p, const WPlan &pl, const Geo &g, const uint32_t *rows,
                                          uint32_t y, uint32_t z, uint32_t &xc, uint32_t &yc, uint32_t &zc) {
    xc = yc = zc = 0;
    if (g.oy + y >= p.Y || g.oz + z >= p.Z) return;
    const uint32_t own = (1u << g.nx) - 1u;
    const uint32_t r0 = rows[z * pl.B1 + y];
    const uint32_t xe = p.X - g.ox - 1;  // +x edges exist for x < X - ox - 1
    const uint32_t xmask = xe >= 32 ? 0xffffffffu : ((1u << xe) - 1u);
    xc = (r0 ^ (r0 >> 1)) & own & xmask;
    if (g.oy + y + 1 < p.Y) yc = (r0 ^ rows[z * pl.B1 + y + 1]) & own;
    if (g.oz + z + 1 < p.Z) zc = (r0 ^ rows[(z + 1) * pl.B1 + y]) & own;
}

// Case index of the cell at (x, y, z) from the inside bitmasks (corner order
// of marching_cubes_pmb.mesh.glsl:84-93: r00 = row (y,z), r01 = (y+1,z),
// r10 = (y,z+1), r11 = (y+1,z+1)).
__device__ __forceinline__ uint32_t cell_case(const uint32_t *rows, uint32_t B1, uint32_t x, uint32_t y, uint32_t z) {
    const uint32_t r00 = rows[z * B1 + y] >> x, r01 = rows[z * B1 + y + 1] >> x;
    const uint32_t r10 = rows[(z + 1) * B1 + y] >> x, r11 = rows[(z + 1) * B1 + y + 1] >> x;
    return (r00 & 1u) | (r00 & 2u) | ((r01 & 2u) << 1) | ((r01 & 1u) << 3) | ((r10 & 1u) << 4) |
           ((r10 & 2u) << 4) | ((r11 & 2u) << 5) | ((r11 & 1u) << 7);
}

// Whether the cell at (x, y, z) of the block lies inside the volume.
__device__ __forceinline__ bool cell_valid(const Problem &p, const Geo &g, uint32_t x, uint32_t y, uint32_t z) {
    return g.ox + x + 1 < p.X && g.oy + y + 1 < p.Y && g.oz + z + 1 < p.Z;
}

__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t &total) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// ------------------------------------------------------------- numerics
// Edge parameter (marching_cubes_pmb.mesh.glsl:129-134): t = (iso - a)/(b - a)
// when |b - a| > 1e-5 else 0.5, clamped to [0, 1]; every operation rounds once.
__device__ __forceinline__ float edge_t(float fa, float fb, float iso) {
    const float den = __fsub_rn(fb, fa);
    float t = 0.5f;
    if (fabsf(den) > 1e-5f) t = __fdiv_rn(__fsub_rn(iso, fa), den);
    t = t < 0.0f ? 0.0f : t;
    t = t > 1.0f ? 1.0f : t;
    return t;
}

template <typename T>
__device__ __forceinline__ float gval(const Problem &p, uint32_t x, uint32_t y, uint32_t z) {
    const T *vol = reinterpret_cast<const T *>(p.vol);
    return Vox<T>::val(__ldg(vol + ((uint64_t)z * p.Y + y) * p.X + x));
}

__device__ __forceinline__ void normalize3(float &a, float &b, float &c) {
    float d = __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
    d = __fadd_rn(d, __fmul_rn(c, c));
    if (d == 0.0f) {
        a = b = c = 0.0f;
        return;
    }
    const float l = __fsqrt_rn(d);
    a = __fdiv_rn(a, l);
    b = __fdiv_rn(b, l);
    c = __fdiv_rn(c, l);
}

// Clamped central difference, normalised (calculate_normal, pmb.mesh.glsl:111-120).
template <typename T>
__device__ __forceinline__ void voxel_normal(const Problem &p, uint32_t x, uint32_t y, uint32_t z, float n[3]) {
    const uint32_t xl = x ? x - 1 : 0, xh = min(x + 1, p.X - 1);
    const uint32_t yl = y ? y - 1 : 0, yh = min(y + 1, p.Y - 1);
    const uint32_t zl = z ? z - 1 : 0, zh = min(z + 1, p.Z - 1);
    n[0] = __fsub_rn(gval<T>(p, xl, y, z), gval<T>(p, xh, y, z));
    n[1] = __fsub_rn(gval<T>(p, x, yl, z), gval<T>(p, x, yh, z));
    n[2] = __fsub_rn(gval<T>(p, x, y, zl), gval<T>(p, x, y, zh));
    normalize3(n[0], n[1], n[2]);
}

// Normal of the vertex at parameter t on the +axis edge of volume voxel
// (gx, gy, gz): normalize(mix(n1, n2, t)) (marching_cubes_pmb.mesh.glsl:126-137).
template <typename T>
__device__ __noinline__ float3 vertex_normal(const Problem &p, uint32_t gx, uint32_t gy, uint32_t gz, uint32_t a,
                                             float t) {
    float n1[3], n2[3];
    voxel_normal<T>(p, gx, gy, gz, n1);
    voxel_normal<T>(p, gx + (a == 0), gy + (a == 1), gz + (a == 2), n2);
    const float omt = __fsub_rn(1.0f, t);
    float3 n;
    n.x = __fadd_rn(__fmul_rn(n1[0], omt), __fmul_rn(n2[0], t));
    n.y = __fadd_rn(__fmul_rn(n1[1], omt), __fmul_rn(n2[1], t));
    n.z = __fadd_rn(__fmul_rn(n1[2], omt), __fmul_rn(n2[2], t));
    normalize3(n.x, n.y, n.z);
    return n;
}

// vertex_normal for a volume whose dtype is known only at run time (p.dtype).
static __device__ __noinline__ float3 vertex_normal_any(const Problem &p, uint32_t gx, uint32_t gy, uint32_t gz,
                                                        uint32_t a, float t) {
    if (p.dtype == MTX_DTYPE_U8) return vertex_normal<uint8_t>(p, gx, gy, gz, a, t);
    if (p.dtype == MTX_DTYPE_U16) return vertex_normal<uint16_t>(p, gx, gy, gz, a, t);
    return vertex_normal<float>(p, gx, gy, gz, a, t);
}

// -------------------------------------------------------------- emit pass
// Context voxel of compact index j: the (B+1)^2 voxels with x == B first, then
// those with y == B, then those with z == B.
__device__ __forceinline__ void ctx_voxel(const WPlan &pl, uint32_t j, uint32_t &x, uint32_t &y, uint32_t &z) {
    const uint32_t B = pl.B, B1 = pl.B1;
    if (j < B1 * B1) {
        x = B;
        z = fdiv(j, pl.rB1);
        y = j - z * B1;
    } else if (j < B1 * B1 + B * B1) {
        const uint32_t i = j - B1 * B1;
        y = B;
        z = fdiv(i, pl.rB);
        x = i - z * B;
    } else {
        const uint32_t i = j - B1 * B1 - B * B1;
        z = B;
        y = fdiv(i, pl.rB);
        x = i - y * B;
    }
}

// -------------------------------------------------------------- scan pass
constexpr uint64_t kCnt31 = 0x7fffffffull;

// Warp-cooperative decoupled look-back over per-tile status words
// ([63:62] flag 1 aggregate / 2 inclusive / 3 aborted, [61:31] triangles,
// [30:0] vertices).  Publishes this tile's aggregate, then its inclusive
// prefix; returns the exclusive prefix, false if aborted.  Totals that do
// not fit 31 bits (or 3 x triangles that do not fit 32) abort with
// MTX_ERR_CAPACITY.
// Sums the (vertices, triangles) of the tile words before tile r, back to and
// including the first inclusive one, in windows of 32 read by the warp;
// false if a predecessor aborted or the wait timed out.
__device__ __forceinline__ bool lookback_sum31(const uint64_t *status, uint32_t r, uint64_t &ev, uint64_t &et,
                                               DevStatus *st, uint32_t spin_limit = kSpinLimit) {
    const uint32_t lane = threadIdx.x & 31;
    ev = et = 0;
    int64_t j = (int64_t)r - 1;
    uint32_t spins = 0;
    while (true) {
        const int64_t k = j - (int64_t)lane;
        const uint64_t w = k >= 0 ? ld_volatile(&status[k]) : (2ull << 62);
        const uint32_t flag = (uint32_t)(w >> 62);
        if (__any_sync(0xffffffffu, flag == 3u)) return false;
        const uint32_t inc = __ballot_sync(0xffffffffu, flag == 2u);
        const uint32_t emp = __ballot_sync(0xffffffffu, flag == 0u);
        const uint32_t first = inc ? (uint32_t)(__ffs(inc) - 1) : 32u;
        const uint32_t window = first >= 31 ? 0xffffffffu : ((2u << first) - 1u);
        if (emp & window) {
            if (++spins >= spin_limit) {
                if (lane == 0) report(st, MTX_ERR_TIMEOUT, kSiteCountLookback, r, (uint32_t)j);
                return false;
            }
            backoff(spins);
            continue;
        }
        uint64_t a = lane <= first ? (w & kCnt31) : 0ull;
        uint64_t b = lane <= first ? ((w >> 31) & kCnt31) : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        ev += a;
        et += b;
        if (first < 32) return true;
        j -= 32;
    }
}

__device__ __forceinline__ bool lookback_counts(uint64_t *status, uint32_t r, uint32_t bnv, uint32_t bnt,
                                                uint64_t &ev, uint64_t &et, DevStatus *st,
                                                uint32_t spin_limit = kSpinLimit) {
    const uint32_t lane = threadIdx.x & 31;
    ev = et = 0;
    bool abort = false;
    if (r > 0) {
        if (lane == 0) st_volatile(&status[r], (1ull << 62) | ((uint64_t)bnt << 31) | bnv);
        abort = !lookback_sum31(status, r, ev, et, st, spin_limit);
    }
    const uint64_t iv = ev + bnv, it = et + bnt;
    if (!abort && (iv > kCnt31 || it > kCnt31 || 3ull * it > 0xffffffffull)) {
        if (lane == 0) report(st, MTX_ERR_CAPACITY, kSiteCountOverflow, (uint32_t)(iv >> 32), (uint32_t)it);
        abort = true;
    }
    if (lane == 0) st_volatile(&status[r], abort ? (3ull << 62) : ((2ull << 62) | (it << 31) | iv));
    return !abort;
}

// ----------------------------------------------------------- block bodies
// Data written earlier in the same launch must not be read through the
// read-only (non-coherent) cache; NC selects that path for data produced by
// an earlier launch, and L2-only loads are used otherwise.
template <bool NC, typename U>
__device__ __forceinline__ U ld_in(const U *p) {
    if constexpr (NC) return __ldg(p);
    else return __ldcg(p);
}

// Lane c in 1..7 returns the rank of neighbour block c = (dx, dy, dz) bits of
// block `id`, or kNoVertex when it is outside the grid or inactive.
template <bool NC = true>
__device__ __forceinline__ uint32_t neighbour_rank(const Problem &p, const Geo &g, uint32_t id,
                                                   const uint32_t *rank_map) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t rk = kNoVertex;
    if (lane >= 1 && lane < 8) {
        const uint32_t dx = lane & 1u, dy = (lane >> 1) & 1u, dz = lane >> 2;
        if (g.bx + dx < p.GX && g.by + dy < p.GY && g.bz + dz < p.GZ &&
            MTX_BC((uint64_t)id + dx + dy * p.GX + (uint64_t)dz * p.GX * p.GY, p.nblocks, kBcRank))
            rk = ld_in<NC>(rank_map + id + dx + dy * p.GX + dz * p.GX * p.GY);
    }
    return rk;
}

// Exclusive scan of the per-block vertex and triangle counts in rank order,
// one tile of up to kScanTile descriptors per CTA of kScanThreads: the tile
// resolves its offset with a decoupled look-back over the tiles before it,
// then fills vertexOffset and indexOffset; the last tile writes the totals.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
static_assert(kScanTile == 1024, "scan_tiles");

__device__ __forceinline__ void scan_tile(mtx_meshlet_descriptor *desc, uint32_t count, uint32_t t, uint64_t *status,
                                          uint32_t *totals, DevStatus *st, uint64_t *s_tmp, uint32_t *s_ok,
                                          uint64_t *s_pre, uint32_t spin_limit = kSpinLimit) {
    const uint32_t ntiles = (count + kScanTile - 1) / kScanTile;
    const uint32_t base = t * kScanTile + threadIdx.x * kScanItems;
    uint32_t nv[kScanItems], nt[kScanItems], sv = 0, stt = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        nv[i] = nt[i] = 0;
        if (base + i < count) {
            const uint2 c = *reinterpret_cast<const uint2 *>(&desc[base + i].vertexCount);
            nv[i] = c.x;
            nt[i] = c.y;
        }
        sv += nv[i];
        stt += nt[i];
    }
    uint64_t tot;
    const uint64_t pre = cta_exclusive_scan64<kScanThreads>(((uint64_t)stt << 32) | sv, s_tmp, &tot);
    if (threadIdx.x < 32) {
        uint64_t ev, et;
        const bool ok = lookback_counts(status, t, (uint32_t)tot, (uint32_t)(tot >> 32), ev, et, st, spin_limit);
        if (threadIdx.x == 0) {
            *s_ok = ok;
            s_pre[0] = ev;
            s_pre[1] = et;
            if (ok && t == ntiles - 1) {
                totals[0] = (uint32_t)(ev + (uint32_t)tot);
                totals[1] = 3u * (uint32_t)(et + (uint32_t)(tot >> 32));
                totals[2] = count;
                totals[3] = count;
            }
        }
    }
    __syncthreads();
    if (!*s_ok) return;
    uint32_t v = (uint32_t)s_pre[0] + (uint32_t)pre, tr = (uint32_t)s_pre[1] + (uint32_t)(pre >> 32);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < count) {
            *reinterpret_cast<uint2 *>(&desc[base + i].vertexOffset) = make_uint2(v, 3u * tr);
            v += nv[i];
            tr += nt[i];
        }
    }
}

}  // namespace mtx
