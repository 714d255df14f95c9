// Adjoint of the PMB extraction with the topology held fixed: dL/dvertex ->
// dL/dfield (dense) and dL/diso.  meshtrex has no backward pass; the forward
// this differentiates is the vertex placement of marching_cubes_pmb.mesh.glsl:
// 122-141, p = u + t * e_axis with t = (iso - f(u)) / (f(u + e_axis) - f(u)).
//
// One warp per active block builds the inside bits of the block's rows from the
// volume, lists the voxels that own a cut edge in canonical order (so vertex
// ids follow the forward's) and, 32 voxels a step, one a lane, recomputes t's
// inputs for their edges:
//   dL/df(u)  = g (iso - f(v)) / d^2,  dL/df(v) = g (f(u) - iso) / d^2,
//   dL/diso   = g / d,                 d = f(v) - f(u), v = u + e_axis.
// ATOMIC mode adds the field terms into dL/dfield with FP32 atomics.
// DETERMINISTIC mode accumulates them into a private (B+1)^3 tile in shared
// memory in four additions a step (the edges' first voxels, then their second
// ones along x, y and z), in each of which every tile voxel has at most one
// writer.  The tile's inner
// voxels belong to this block alone and go straight to dL/dfield; the others
// are kept as the block's partial, and a gather pass gives each of them one
// designated block that sums the partials of the blocks that own an edge at it
// -- its own block and those before it in x, y and z -- in that order.  dL/diso
// is summed per block -- each lane over its rows, axis by axis, so that the sum does
// not depend on how the list fell into steps -- and then over blocks in rank order
// in both modes.
// Staging each tile as float and walking its rows took 49 us (ATOMIC) for the
// 7,700 active blocks of a 512^3 volume, after 88 us of zeroing, and 34 us, with
// 36 us for a gather over whole tiles, for the 1,250 of 250 x 198 x 171
// (DETERMINISTIC); this takes 31, and 14 with 9.  Blocks with more terms than the
// shared memory holds list their voxels again for each axis: a noisy 300 x 400 x
// 512 float32 ball at B = 8, 232 vertices a block, takes 81 us, 132 with its gather
// (126 and 271 by tiles and rows; 142 and 223 with terms kept for at most 256 voxels
// a block and rows walked again by lane).
#include "pmb_lists.cuh"

namespace mtx {

constexpr uint32_t kAdjWarps = 4;
constexpr uint32_t kIsoThreads = 1024;

struct AdjArgs {
    Problem p;
    const uint32_t *ids;
    const uint32_t *rank_map;
    const mtx_meshlet_descriptor *desc;
    uint32_t n;           // active blocks
    uint32_t vcount;      // vertices of the forward mesh
    const float *g;       // dL/dvertex, gstride floats per vertex
    uint32_t gstride;
    float gscale[3];      // d(position)/dt per axis: 1 (voxel frame) or 2 / extent (NDC)
    float *dfield;
    float *partial;       // DETERMINISTIC: T3 floats per active block
    float *iso_part;      // dL/diso of each active block
    uint32_t T3;          // (B+1)^3
    DevStatus *st;
};

// dL/diso terms, one a vertex, that a warp's shared memory holds: all that a block
// of edge 6 or less can have, half of the most one of edge 8 can, and more than a
// surface through it has.
__host__ __device__ inline uint32_t iso_terms(uint32_t B) { return std::min(3 * B * B * B, B <= 8 ? 768u : 2304u); }

// A warp's shared memory: inside rows, list bits, list, the plain loads'
// bitstream, dL/diso terms, and for DETERMINISTIC the accumulation tile
// (off_tile).
__host__ __device__ inline WPlan make_adjoint_plan(uint32_t B, bool det) {
    WPlan p{};
    plan_block(p, B);
    const uint32_t T3 = p.B1 * p.B1 * p.B1;
    uint32_t o = 0;
    p.off_rows = o;
    o = align_up(o + 4 * p.B1 * p.B1, 16);
    p.off_mm = o;
    o = align_up(o + 4 * list_words(B), 16);
    p.off_list = o;
    o = align_up(o + 2 * list_cap(B), 16);
    p.off_case = o;
    o = align_up(o + 4 * ((T3 + 31) / 32 + 1), 16);
    p.off_vp = o;  // dL/diso terms, axis by axis
    o = align_up(o + 4 * iso_terms(B), 16);
    p.off_tile = o;
    if (det) o = align_up(o + 4 * T3, 16);
    p.bytes = o;
    return p;
}

// List bits of the voxels that own a cut edge.  Lane l takes rows [l R, l R + R),
// R = ceil(B^2 / 32): of the block's cut edges along an axis its own are
// [at, at + own).
struct CutRows {
    uint32_t at[2], own[2];  // of x | y << 16, z
    uint32_t nx, ny, nz;     // the block's
};
template <int BC>
__device__ __forceinline__ CutRows cut_bits(const Problem &p, const WPlan &pl, unsigned char *ws, const Geo &g) {
    const uint32_t lane = threadIdx.x & 31, B = pl.B, R = (pl.BB + 31) / 32;
    const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
    uint32_t *bits = reinterpret_cast<uint32_t *>(ws + pl.off_mm);
    for (uint32_t i = lane; i < list_words(B); i += 32) bits[i] = 0;
    __syncwarp();
    CutRows c{};
    for (uint32_t q = lane * R; q < min(pl.BB, lane * R + R); ++q) {
        const uint32_t z = fdiv(q, pl.rB), y = q - z * B;
        uint32_t xc, yc, zc;
        row_cross(p, pl, g, rows, y, z, xc, yc, zc);
        c.own[0] += __popc(xc) | (__popc(yc) << 16);
        c.own[1] += __popc(zc);
        const uint32_t m = xc | yc | zc;
        if constexpr (BC == 8) {
            reinterpret_cast<uint8_t *>(bits)[q] = (uint8_t)m;
        } else if (m) {
            const uint32_t b = q * B, w = b >> 5, s = b & 31u;
            atomicOr(&bits[w], m << s);
            if (s + B > 32) atomicOr(&bits[w + 1], m >> (32 - s));
        }
    }
    __syncwarp();
    uint32_t xy;  // at most 4096 an axis
    c.at[0] = warp_excl_scan(c.own[0], xy);
    c.nx = xy & 0xffffu;
    c.ny = xy >> 16;
    c.at[1] = warp_excl_scan(c.own[1], c.nz);
    return c;
}

// Of the step's cut edges along each axis, those of the voxels before this lane's
// and all of them (m: this lane's cut owned edges).
__device__ __forceinline__ void step_edges(uint32_t m, uint32_t before[3], uint32_t all[3]) {
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t b = __ballot_sync(0xffffffffu, (m >> k) & 1u);
        before[k] = __popc(b & lt);
        all[k] = __popc(b);
    }
}

// One vertex's dL/diso term (the gradient along its edge over the edge's value
// difference); 0 where t = 0.5.
__device__ __forceinline__ float iso_term(float gv, float scale, float den) {
    return fabsf(den) > 1e-5f ? __fdiv_rn(__fmul_rn(gv, scale), den) : 0.0f;
}

// CTAs an SM that the register count has to allow, where the compiler's own choice
// takes more registers than pay (0: its choice).  Block edge 5, ATOMIC: 122
// registers 337 us, 64 registers 263 (300 x 400 x 512 uint16, 35 vertices a
// block); at B = 2, 4 and 8 a bound of the same register count is 2 to 5% slower than
// none.
constexpr int adjoint_min_ctas(bool det, int BC) { return BC == 5 ? (det ? 7 : 8) : BC == 3 && !det ? 8 : 0; }

template <typename T, bool DET, int BC>
__global__ void __launch_bounds__(kAdjWarps * 32, adjoint_min_ctas(DET, BC))
    adjoint_block_kernel(const __grid_constant__ AdjArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    Problem p = a.p;
    p.B = BC;  // known at compile time: the plan and every division by the edge fold to constants
    const WPlan pl = make_adjoint_plan(p.B, DET);
    const GridDiv dv = grid_div(p);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    unsigned char *ws = smem + warp * pl.bytes;
    float *acc = reinterpret_cast<float *>(ws + pl.off_tile);
    const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
    const uint16_t *list = reinterpret_cast<const uint16_t *>(ws + pl.off_list);
    float *term = reinterpret_cast<float *>(ws + pl.off_vp);
    const uint32_t B = pl.B, B1 = pl.B1, T3 = B1 * B1 * B1;
    const float iso = p.iso;
    for (uint32_t r = blockIdx.x * W + warp; r < a.n; r += gridDim.x * W) {
        const Geo g = block_geo(__ldg(a.ids + r), p, false, 4, dv);
        const uint4 dq = __ldg(reinterpret_cast<const uint4 *>(a.desc + r));
        const uint32_t vbase = dq.x, nv = dq.z;
        const bool inner = g.ox + B < p.X && g.oy + B < p.Y && g.oz + B < p.Z;
        load_rows<T>(p, pl, ws, g, nullptr);
        const CutRows cr = cut_bits<BC>(p, pl, ws, g);
        const bool ok = cr.nx + cr.ny + cr.nz == nv && (uint64_t)vbase + nv <= a.vcount;
        if (!ok && lane == 0) report(a.st, MTX_ERR_INTERNAL, kSiteAdjoint, r, cr.nx + cr.ny + cr.nz);
        if (DET) {
            for (uint32_t i = lane; i < T3; i += 32) acc[i] = 0.0f;
            __syncwarp();
        }
        const bool keep = nv <= iso_terms(B);  // else the terms are computed again below
        ListWalk l;
        // the next vertex, and each axis's next term (x | y << 16, z)
        uint32_t run = vbase, to[2] = {cr.nx << 16, cr.nx + cr.ny};
        while (const uint32_t n = ok ? list_take<BC>(l, pl, ws) : 0u) {
            uint32_t m = 0, cell = 0;
            if (lane < n) {
                cell = list[l.done + lane];
                m = listed_cell(p, pl, g, rows, cell, inner) >> 28;
            }
            uint32_t before[3], all[3];
            step_edges(m, before, all);
            const uint32_t first = run + before[0] + before[1] + before[2];
            const uint32_t q = fdiv(cell, pl.rB), x = cell - q * B, z = fdiv(q, pl.rB), y = q - z * B;
            const uint64_t v0 = ((uint64_t)(g.oz + z) * p.Y + (g.oy + y)) * p.X + (g.ox + x);
            const uint64_t gstep[3] = {1ull, (uint64_t)p.X, (uint64_t)p.X * p.Y};
            const T *v = reinterpret_cast<const T *>(p.vol) + v0;
            // the voxel, its cut neighbours and their vertices' gradients, all loads in flight
            T raw[4] = {T(0), T(0), T(0), T(0)};
            float gv[3] = {0.0f, 0.0f, 0.0f};
            if (m) raw[3] = __ldg(v);
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k)
                if ((m >> k) & 1u) {
                    raw[k] = __ldg(v + gstep[k]);
                    gv[k] = __ldg(a.g + (uint64_t)(first + __popc(m & ((1u << k) - 1u))) * a.gstride + k);
                }
            const float fa = Vox<T>::val(raw[3]);
            float own = 0.0f, far[3];
            bool on[3];
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {
                const float fb = Vox<T>::val(raw[k]), den = __fsub_rn(fb, fa);
                on[k] = ((m >> k) & 1u) && fabsf(den) > 1e-5f;  // else t = 0.5: no gradient
                far[k] = 0.0f;
                const float s = (m >> k) & 1u ? iso_term(gv[k], a.gscale[k], den) : 0.0f;
                const uint32_t at = (k == 0 ? to[0] & 0xffffu : k == 1 ? to[0] >> 16 : to[1]) + before[k];
                if (keep && ((m >> k) & 1u) && MTX_BC(at, iso_terms(B), kBcTerms)) term[at] = s;
                if (on[k] && MTX_BC(v0 + gstep[k], (uint64_t)p.X * p.Y * p.Z, kBcField)) {
                    const float ta = __fdiv_rn(__fmul_rn(s, __fsub_rn(iso, fb)), den);
                    far[k] = __fdiv_rn(__fmul_rn(s, __fsub_rn(fa, iso)), den);
                    if (DET) {
                        own = __fadd_rn(own, ta);
                    } else {
                        atomicAdd(a.dfield + v0, ta);
                        atomicAdd(a.dfield + v0 + gstep[k], far[k]);
                    }
                }
            }
            if (DET) {
                // one writer a tile voxel in each of the four additions
                const uint32_t i = (z * B1 + y) * B1 + x;
                if (m && MTX_BC(i, T3, kBcTile)) acc[i] = __fadd_rn(acc[i], own);
                __syncwarp();
#pragma unroll
                for (uint32_t k = 0; k < 3; ++k) {
                    const uint32_t j = i + (k == 0 ? 1u : k == 1 ? B1 : B1 * B1);
                    if (on[k] && MTX_BC(j, T3, kBcTile)) acc[j] = __fadd_rn(acc[j], far[k]);
                    __syncwarp();
                }
            }
            run += all[0] + all[1] + all[2];
            to[0] += all[0] | (all[1] << 16);
            to[1] += all[2];
            l.done += n;
        }
        // dL/diso: each lane its rows' terms, axis by axis in canonical order, then the lanes' sums
        float diso = 0.0f;
        __syncwarp();
        if (ok && keep) {
            // (y's terms begin where x's end, z's where y's do)
            const float *tx = term + (cr.at[0] & 0xffffu), *ty = term + (to[0] & 0xffffu) + (cr.at[0] >> 16),
                        *tz = term + (to[0] >> 16) + cr.at[1];
            for (uint32_t i = 0; i < (cr.own[0] & 0xffffu); ++i) diso = __fadd_rn(diso, tx[i]);
            for (uint32_t i = 0; i < (cr.own[0] >> 16); ++i) diso = __fadd_rn(diso, ty[i]);
            for (uint32_t i = 0; i < cr.own[1]; ++i) diso = __fadd_rn(diso, tz[i]);
        } else if (ok) {
            // the list once more for each axis, its terms summed whenever they fill the room for them
            for (uint32_t k = 0; k < 3; ++k) {
                l = ListWalk{};
                run = vbase;
                uint32_t t0 = 0, held = 0;  // of the axis's terms, [t0, t0 + held) are held
                const uint64_t step = k == 0 ? 1ull : k == 1 ? (uint64_t)p.X : (uint64_t)p.X * p.Y;
                const uint32_t at = k == 0 ? cr.at[0] & 0xffffu : k == 1 ? cr.at[0] >> 16 : cr.at[1];
                const uint32_t own = k == 0 ? cr.own[0] & 0xffffu : k == 1 ? cr.own[0] >> 16 : cr.own[1];
                uint32_t n;
                do {
                    n = list_take<BC>(l, pl, ws);
                    if (!n || held + 32 > iso_terms(B)) {
                        __syncwarp();
                        const uint32_t i1 = min(at + own, t0 + held);
                        for (uint32_t i = max(at, t0); i < i1; ++i) diso = __fadd_rn(diso, term[i - t0]);
                        __syncwarp();
                        t0 += held;
                        held = 0;
                    }
                    uint32_t m = 0, cell = 0;
                    if (lane < n) {
                        cell = list[l.done + lane];
                        m = listed_cell(p, pl, g, rows, cell, inner) >> 28;
                    }
                    uint32_t before[3], all[3];
                    step_edges(m, before, all);
                    if (((m >> k) & 1u) && MTX_BC(held + before[k], iso_terms(B), kBcTerms)) {
                        const uint32_t q = fdiv(cell, pl.rB), x = cell - q * B, z = fdiv(q, pl.rB), y = q - z * B;
                        const T *v = reinterpret_cast<const T *>(p.vol) +
                                     ((uint64_t)(g.oz + z) * p.Y + (g.oy + y)) * p.X + (g.ox + x);
                        const float den = __fsub_rn(Vox<T>::val(__ldg(v + step)), Vox<T>::val(__ldg(v)));
                        const uint32_t vid = run + before[0] + before[1] + before[2] + __popc(m & ((1u << k) - 1u));
                        term[held + before[k]] = iso_term(__ldg(a.g + (uint64_t)vid * a.gstride + k), a.gscale[k], den);
                    }
                    run += all[0] + all[1] + all[2];
                    held += all[k];
                    l.done += n;
                } while (n);
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) diso = __fadd_rn(diso, __shfl_xor_sync(0xffffffffu, diso, o));
        if (lane == 0) a.iso_part[r] = diso;
        if (DET) {
            __syncwarp();
            float *dst = a.partial + (uint64_t)r * T3;
            for (uint32_t i = lane; i < T3; i += 32) {
                const uint32_t iq = fdiv(i, pl.rB1), lx = i - iq * B1, lz = fdiv(iq, pl.rB1), ly = iq - lz * B1;
                const float t = acc[i];
                if (lx % B == 0 || ly % B == 0 || lz % B == 0)  // shared with a neighbour: the gather pass's
                    dst[i] = t;
                else if (t != 0.0f &&  // (voxels outside the volume have none)
                         MTX_BC(g.ox + lx, p.X, kBcField) && MTX_BC(g.oy + ly, p.Y, kBcField) &&
                         MTX_BC(g.oz + lz, p.Z, kBcField))
                    a.dfield[((uint64_t)(g.oz + lz) * p.Y + (g.oy + ly)) * p.X + (g.ox + lx)] = t;
            }
        }
        __syncwarp();
    }
}

// DETERMINISTIC: the voxels on the faces of the active blocks' tiles.  A voxel w
// of block c gets terms from edges that c owns and, where it lies on c's low x,
// y or z face, from the edge that the block before c on that axis owns; the
// first active one of c, c - x, c - y, c - z writes the sum, taken in that order.
__global__ void __launch_bounds__(kAdjWarps * 32) adjoint_gather_kernel(const __grid_constant__ AdjArgs a) {
    const Problem &p = a.p;
    const GridDiv dv = grid_div(p);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const uint32_t B = p.B, B1 = B + 1, BB = B * B;
    const uint32_t rB = (uint32_t)((0x100000000ull + B - 1) / B);
    const uint32_t st[3] = {1u, B1, B1 * B1};  // tile steps
    for (uint32_t r = blockIdx.x * W + warp; r < a.n; r += gridDim.x * W) {
        const Geo g = block_geo(__ldg(a.ids + r), p, false, 4, dv);
        // ranks, one a lane: lanes 0-2 the blocks before this one along x, y, z; 3-5 those after it; 6 + 2 k, 7 + 2 k
        // the blocks before the one after it along axis k, on the other two axes in order
        uint32_t rk = kNoVertex;
        if (lane < 12) {
            int b[3] = {(int)g.bx, (int)g.by, (int)g.bz};
            if (lane < 3) {
                --b[lane];
            } else if (lane < 6) {
                ++b[lane - 3];
            } else {
                const uint32_t k = (lane - 6) >> 1, o = (lane & 1u) ? (k == 2 ? 1u : 2u) : (k == 0 ? 1u : 0u);
                ++b[k];
                --b[o];
            }
            if (b[0] >= 0 && b[1] >= 0 && b[2] >= 0 && b[0] < (int)p.GX && b[1] < (int)p.GY && b[2] < (int)p.GZ)
                rk = __ldg(a.rank_map + ((uint64_t)b[2] * p.GY + b[1]) * p.GX + b[0]);
        }
        uint32_t nb[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) nb[k] = __shfl_sync(0xffffffffu, rk, k);
        auto put = [&](uint32_t lx, uint32_t ly, uint32_t lz, float t) {
            const uint32_t wx = g.ox + lx, wy = g.oy + ly, wz = g.oz + lz;
            if (t != 0.0f && wx < p.X && wy < p.Y && wz < p.Z)
                a.dfield[((uint64_t)wz * p.Y + wy) * p.X + wx] = t;
        };
        auto from = [&](uint32_t rank, uint32_t i) {
            return MTX_BC(rank, a.n, kBcPartial) && MTX_BC(i, a.T3, kBcPartial)
                       ? __ldcg(a.partial + (uint64_t)rank * a.T3 + i)
                       : 0.0f;
        };
        // this block's voxels on its low faces: z == 0 (B^2), then y == 0 (B (B-1)), then x == 0 ((B-1)^2)
        const uint32_t nlow = BB + B * (B - 1) + (B - 1) * (B - 1);
        for (uint32_t j = lane; j < nlow; j += 32) {
            uint32_t lx, ly, lz;
            if (j < BB) {
                ly = fdiv(j, rB);
                lx = j - ly * B;
                lz = 0;
            } else if (j < BB + B * (B - 1)) {
                const uint32_t i = j - BB;
                lz = 1 + fdiv(i, rB);
                lx = i - (lz - 1) * B;
                ly = 0;
            } else {
                const uint32_t i = j - BB - B * (B - 1);
                lz = 1 + i / (B - 1);
                ly = 1 + i % (B - 1);
                lx = 0;
            }
            const uint32_t i = (lz * B1 + ly) * B1 + lx;
            float t = from(r, i);
            if (!lx && nb[0] != kNoVertex) t = __fadd_rn(t, from(nb[0], i + B * st[0]));
            if (!ly && nb[1] != kNoVertex) t = __fadd_rn(t, from(nb[1], i + B * st[1]));
            if (!lz && nb[2] != kNoVertex) t = __fadd_rn(t, from(nb[2], i + B * st[2]));
            put(lx, ly, lz, t);
        }
        // voxels of the block after this one along axis k, where that one is not active
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) {
            if (nb[3 + k] != kNoVertex) continue;
            const uint32_t u = k == 0 ? 1u : 0u, v = k == 2 ? 1u : 2u;  // the other axes, in order
            const uint32_t ru = nb[6 + 2 * k], rv = nb[7 + 2 * k];
            for (uint32_t j = lane; j < BB; j += 32) {
                const uint32_t lv = fdiv(j, rB), lu = j - lv * B;
                const uint32_t i = B * st[k] + lu * st[u] + lv * st[v];
                const bool tu = !lu && ru != kNoVertex, tv = !lv && rv != kNoVertex;
                // a block before that one on an axis before k writes the voxel
                if ((tu && u < k) || (tv && v < k)) continue;
                float t = from(r, i);
                const uint32_t c = lu * st[u] + lv * st[v];  // the voxel in its own block's tile
                if (tu) t = __fadd_rn(t, from(ru, c + B * st[u]));
                if (tv) t = __fadd_rn(t, from(rv, c + B * st[v]));
                put(k == 0 ? B : lu, k == 1 ? B : (k == 0 ? lu : lv), k == 2 ? B : lv, t);
            }
        }
    }
}

// dL/diso: the per-block sums added in rank order (double accumulation, one CTA).
__global__ void __launch_bounds__(kIsoThreads) adjoint_iso_kernel(const float *__restrict__ part, uint32_t n,
                                                                  float *out) {
    __shared__ double s[kIsoThreads];
    double acc = 0.0;
    const uint32_t per = (n + kIsoThreads - 1) / kIsoThreads;
    const uint32_t b0 = threadIdx.x * per, b1 = min(n, b0 + per);
    for (uint32_t i = b0; i < b1; ++i) acc += (double)part[i];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (uint32_t h = kIsoThreads / 2; h; h >>= 1) {
        if (threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = (float)s[0];
}

// Every block edge at compile time: against one kernel for run-time edges the block
// pass of a 300 x 400 x 512 float32 gyroid takes, us, ATOMIC / DETERMINISTIC, at B = 3
// 455, 517 where that takes 589, 898; at B = 6 211, 271 (238, 440); at B = 16 288, 1087
// (310, 1708).
template <typename T, bool DET>
static auto adjoint_fn(uint32_t B) {
    switch (B) {
    case 2: return adjoint_block_kernel<T, DET, 2>;
    case 3: return adjoint_block_kernel<T, DET, 3>;
    case 4: return adjoint_block_kernel<T, DET, 4>;
    case 5: return adjoint_block_kernel<T, DET, 5>;
    case 6: return adjoint_block_kernel<T, DET, 6>;
    case 7: return adjoint_block_kernel<T, DET, 7>;
    case 8: return adjoint_block_kernel<T, DET, 8>;
    case 9: return adjoint_block_kernel<T, DET, 9>;
    case 10: return adjoint_block_kernel<T, DET, 10>;
    case 11: return adjoint_block_kernel<T, DET, 11>;
    case 12: return adjoint_block_kernel<T, DET, 12>;
    case 13: return adjoint_block_kernel<T, DET, 13>;
    case 14: return adjoint_block_kernel<T, DET, 14>;
    case 15: return adjoint_block_kernel<T, DET, 15>;
    default: return adjoint_block_kernel<T, DET, 16>;  // MTX_MAX_BLOCK_EDGE (check_pc)
    }
}
template <typename T>
static auto adjoint_fn(bool det, uint32_t B) {
    return det ? adjoint_fn<T, true>(B) : adjoint_fn<T, false>(B);
}

MTX_BC_READER(bc_take_adjoint)

}  // namespace mtx

using namespace mtx;

extern "C" mtx_status mtx_extract_backward(mtx_context_t c, const mtx_volume *vol, const mtx_push_constants *pc,
                                           const mtx_filtering_output *filt, const mtx_meshlet_descriptor *meshlets,
                                           uint32_t vertexCount, const float *dl_dvertex, uint32_t vertexStride,
                                           uint32_t frame, float *dl_dfield, float *dl_diso, uint32_t mode) {
    if (!c) return MTX_ERR_INVALID_ARG;
    DeviceGuard dg(c->device);
    join_extract(c);
    if (!vol || !pc || !filt || !dl_dfield || !dl_diso) return fail(c, MTX_ERR_INVALID_ARG, "null argument");
    if (mode > MTX_ADJOINT_DETERMINISTIC || frame > MTX_FRAME_NDC || vertexStride < 3)
        return fail(c, MTX_ERR_INVALID_ARG, "bad adjoint mode, frame or vertex stride");
    mtx_status rs = check_volume(c, vol);
    if (rs != MTX_OK) return rs;
    if ((rs = check_pc(c, vol, pc)) != MTX_OK) return rs;
    const Problem p = make_problem(vol, pc->blockDim[0], pc->isovalue);
    const uint32_t n = filt->activeBlockCount;
    if (filt->totalBlocks != p.nblocks || n > p.nblocks)
        return fail(c, MTX_ERR_INVALID_ARG, "filtering output does not match the volume and block edge");
    if (n && (!meshlets || !filt->compactedBlockIdBuffer.ptr || !filt->blockRankBuffer.ptr ||
              (vertexCount && !dl_dvertex)))
        return fail(c, MTX_ERR_INVALID_ARG, "forward outputs are missing");
    cudaStream_t s = c->stream;
    mtx_profiler *prof = c->prof;
    prof_begin(prof, "Mesh_Extraction_Backward", s);
    MTX_CUDA(c, cudaMemsetAsync(dl_dfield, 0, nvox(vol->dims) * sizeof(float), s));
    if (n == 0) {
        MTX_CUDA(c, cudaMemsetAsync(dl_diso, 0, sizeof(float), s));
        prof_end(prof, s);
        return MTX_OK;
    }
    const bool det = mode == MTX_ADJOINT_DETERMINISTIC;
    const uint32_t B = p.B, T3 = (B + 1) * (B + 1) * (B + 1);
    if ((rs = scratch_reserve(c, c->adj_iso, sizeof(float) * (size_t)n)) != MTX_OK) return rs;
    if (det && (rs = scratch_reserve(c, c->adj_partial, sizeof(float) * (size_t)n * T3)) != MTX_OK) return rs;

    AdjArgs a{};
    a.p = p;
    a.ids = (const uint32_t *)filt->compactedBlockIdBuffer.ptr;
    a.rank_map = (const uint32_t *)filt->blockRankBuffer.ptr;
    a.desc = meshlets;
    a.n = n;
    a.vcount = vertexCount;
    a.g = dl_dvertex;
    a.gstride = vertexStride;
    for (int k = 0; k < 3; ++k) a.gscale[k] = frame == MTX_FRAME_NDC ? 2.0f / (float)vol->dims[k] : 1.0f;
    a.dfield = dl_dfield;
    a.partial = det ? (float *)c->adj_partial.ptr : nullptr;
    a.iso_part = (float *)c->adj_iso.ptr;
    a.T3 = T3;
    a.st = &c->ctrl->status;
    const WPlan pl = make_adjoint_plan(B, det);
    const uint32_t smem = kAdjWarps * pl.bytes;
    auto kern = p.dtype == MTX_DTYPE_U8    ? adjoint_fn<uint8_t>(det, B)
                : p.dtype == MTX_DTYPE_U16 ? adjoint_fn<uint16_t>(det, B)
                                           : adjoint_fn<float>(det, B);
    int occ = 0;
    if ((rs = ctas_per_sm(c, reinterpret_cast<const void *>(kern), kAdjWarps * 32, smem, &occ)) != MTX_OK) return rs;
    if (occ < 1) return fail(c, MTX_ERR_UNSUPPORTED, "adjoint warp layout does not fit shared memory");
    const uint32_t grid = std::min<uint32_t>((n + kAdjWarps - 1) / kAdjWarps, (uint32_t)(occ * c->sm_count));
    kern<<<grid, kAdjWarps * 32, smem, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint launch");
    if (det) {
        const uint32_t gg = std::min<uint32_t>((n + kAdjWarps - 1) / kAdjWarps, (uint32_t)(16 * c->sm_count));
        adjoint_gather_kernel<<<gg, kAdjWarps * 32, 0, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(c, e, "adjoint gather launch");
    }
    adjoint_iso_kernel<<<1, kIsoThreads, 0, s>>>(a.iso_part, n, dl_diso);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(c, e, "adjoint isovalue launch");
    prof_end(prof, s);
    return MTX_OK;
}
