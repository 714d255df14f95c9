// Stage 3: PMB marching cubes over the active blocks of one volume
// (meshtrex: marching_cubes_pmb.task.glsl:101-216 and
// marching_cubes_pmb.mesh.glsl:185-393, drawn by extractionManager.cpp:638-640).
//
// One warp owns one active block at a time (block bodies: pmb_lists.cuh); a CTA
// runs several such warps that share only the tables.  The count pass stages
// the (B+1)^3 voxel tile of its block in shared memory by TMA, or, when the
// volume's rows are not 16-byte aligned, takes the inside bits straight from
// plain loads; the next block's tile is issued as soon as the current block's
// inside bits are built.
//
//  count pass  per-block vertex/triangle counts, low-face records and the list
//              of the block's cells (B > 8: its inside bits) for the emit pass
//  scan pass   decoupled look-back scan of the counts -> meshlet descriptors, totals
//  emit pass   vertices (each exactly once) and triangles, indices resolved
//              through the block's vertex table and the neighbours' face records
#include "pmb_lists.cuh"

namespace mtx {

// ------------------------------------------------------------- count pass
// Warps a CTA at most: for B > 8 the shared memory of a warp (15 KB in the emit
// pass, 13 to 30 in the count pass) and not the registers bounds the warps of an
// SM, and one CTA with all of them wastes least of it.  640 x 512 x 448 uint16 at
// B = 16 (2869 active blocks), CTAs of 4 and 8 warps: count 37 us, emit 112; one
// CTA of 11 and 14: 30.5 and 85.
constexpr int kBigWarps = 16;
constexpr int cta_warps_max(int BC) { return BC == 0 || BC > 8 ? kBigWarps : kMaxWarps; }

// A warp's first block.  For B > 8 a volume has few blocks, each long: they go
// round the CTAs; else neighbours in a CTA share voxels and records in L1.
__device__ __forceinline__ uint32_t first_block(uint32_t B, uint32_t warp, uint32_t W) {
    return B > 8 ? warp * gridDim.x + blockIdx.x : blockIdx.x * W + warp;
}

// BC: the block edge at compile time (0: p.B at run time): the warp's
// shared-memory plan and every division by the edge fold to constants.
// Bound by instruction issue (2.6 a cycle and SM, 880 a block at B = 8).  Row
// walks over the crossing rows with case bytes and prefixes kept for every cell
// took 108 us for the 80,600 active blocks of the 1024^3 uint16 ball at B = 8;
// the list takes 93; 1024 x 1024 x 314 uint8 at B = 3 179 -> 123; 384 x 320 x
// 256 float32 at B = 4 58 -> 41; 640 x 512 x 448 uint16 at B = 16 53 -> 30.5.
template <typename T, bool TMA, int BC>
__global__ void __launch_bounds__(cta_warps_max(BC) * 32, BC == 0 ? 2 : BC > 8 ? 1 : 4)
    pmb_count_kernel(Problem p_, const __grid_constant__ CUtensorMap map, const uint32_t *__restrict__ ids,
                     const uint32_t *__restrict__ count_ptr, mtx_meshlet_descriptor *__restrict__ desc,
                     uint64_t desc_cap, uint16_t *__restrict__ faces, uint32_t *__restrict__ state,
                     uint32_t *totals, uint8_t *__restrict__ cell_cases, uint64_t block_cap, DevStatus *st,
                     uint64_t *scan_status, uint32_t scan_tiles, uint32_t *scan_ticket, bool use_off) {
    extern __shared__ __align__(128) unsigned char smem[];
    scan_reset(scan_status, scan_tiles, scan_ticket, totals);
    Problem p = p_;
    if (BC) p.B = BC;
    const WPlan pl = make_count_plan(p.B, sizeof(T), TMA);
    const GridDiv dv = grid_div(p);
    uint8_t *ntab = smem;
    uint32_t *off = reinterpret_cast<uint32_t *>(smem + 256);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    unsigned char *ws = smem + count_fixed_bytes(p.B, !TMA && use_off) + warp * pl.bytes;
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) ntab[i] = (uint8_t)(c_mc_cases[i] & 0xFu);
    if (!TMA && use_off) row_offsets(p, pl, off);
    if (lane == 0 && TMA) {
        mbar_init(reinterpret_cast<uint64_t *>(ws + pl.off_bar), 1);
        fence_mbar_init();
    }
    __syncthreads();
    const uint32_t count = *count_ptr;
    if (count > block_cap || count > desc_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            report(st, MTX_ERR_CAPACITY, kSiteEmitCapacity, count, 3);
            totals[3] = count;
        }
        return;
    }
    const uint32_t B3 = pl.BB * pl.B, slot = list_state_words(p.B), fslot = face_stride16(p.B);
    uint32_t parity = 0;

    uint32_t r = first_block(p.B, warp, W);
    const uint32_t nw = gridDim.x * W;
    Geo g{};
    if (r < count) {
        g = block_geo(__ldg(ids + r), p, TMA, sizeof(T), dv);
        if constexpr (TMA) tile_issue<T>(pl, ws, g, &map);
    }
    while (r < count) {
        const uint32_t rn = r + nw;
        Geo gn{};
        const bool have_next = rn < count;
        if (have_next) gn = block_geo(__ldg(ids + rn), p, TMA, sizeof(T), dv);
        if constexpr (TMA) {
            if (!tile_wait(pl, ws, g, parity, st)) break;
            if constexpr (BC != 0) tile_rows<T, BC>(p, pl, ws, g);
            else build_rows<T>(p, pl, ws, g);
            if (have_next) tile_issue<T>(pl, ws, gn, &map);  // the tile is dead once the rows are built
        } else {
            load_rows<T>(p, pl, ws, g, use_off ? off : nullptr);
        }
        count_block_list<BC>(p, pl, ws, g, ntab, cell_cases ? cell_cases + (uint64_t)r * B3 : nullptr, desc + r,
                             faces + (uint64_t)r * fslot, state + (uint64_t)r * slot);
        if (!have_next) break;
        r = rn;
        g = gn;
    }
}

// -------------------------------------------------------------- scan pass
// capacity: descriptors that desc and the tile words hold.  With more active
// blocks than that the count pass has reported the error and set the totals,
// and there is nothing to scan.
__global__ void __launch_bounds__(kScanThreads)
    pmb_scan_kernel(mtx_meshlet_descriptor *__restrict__ desc, const uint32_t *__restrict__ count_ptr,
                    uint64_t capacity, uint64_t *tile_status, uint32_t *ticket, uint32_t *totals, DevStatus *st,
                    uint32_t spin_limit, uint32_t skip, uint32_t *emit_ticket, uint32_t *emit_done) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *emit_ticket = *emit_done = 0;  // for the emit pass that follows
    __shared__ uint32_t s_tile, s_ok;
    __shared__ uint64_t s_tmp[kScanThreads / 32 + 1];
    __shared__ uint64_t s_pre[2];
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u) + skip;
    __syncthreads();
    const uint32_t t = s_tile;
    const uint32_t count = *count_ptr;
    if (count > capacity || t >= (count + kScanTile - 1) / kScanTile) return;
    scan_tile(desc, count, t, tile_status, totals, st, s_tmp, &s_ok, s_pre, spin_limit);
}

// A warp's blocks in the emit pass: three quarters of the list by a fixed stride,
// the rest by ticket, drawn one block ahead.  Warps' blocks differ in work, and
// with about ten blocks a warp (80,000 active blocks of a 1024^3 volume) fixed
// shares alone leave most warps waiting for the unluckiest; tickets alone are
// bound by the counter, which serves fewer than one draw a nanosecond (emit of
// the 1024^3 uint16 ball at block 8: 183 us by stride, 161 by tickets, 158 so;
// the count pass, at half the work a block, gets slower, 94 -> 134 us, and keeps
// the stride).  A half, 5/8, 3/4, 7/8 and all by stride, us: 512^3 float32 gyroid at B
// = 8 293, 293, 293, 317, 342; 1024 x 1024 x 314 uint8 at B = 3 741, 733, 726, 729, 788;
// a noisy 1024^3 uint16 ball of 209,000 dense blocks 974, 1043, 1099, 1187, 1246; with two
// or three blocks a warp (201 x 243 x 257 gyroid at B = 8) 50.8, 51.1, 50.8, 51.9, 45.3.
struct BlockShare {
    uint32_t fixed, stride;  // blocks given out by stride, warps of the grid
    uint32_t *ticket;
    __device__ __forceinline__ BlockShare(uint32_t count, uint32_t warps, uint32_t *t) : stride(warps), ticket(t) {
        const uint32_t rounds = count / warps;
        fixed = rounds ? max(rounds * 3 / 4, 1u) * warps : ~0u;  // the first round is by stride, always
    }
    // The block after block r of this warp (lane 0's value is the block for tickets: take it by shuffle).
    __device__ __forceinline__ uint32_t after(uint32_t r) const {
        if (fixed == ~0u || (uint64_t)r + stride < fixed) return min((uint64_t)r + stride, (uint64_t)~0u);
        uint32_t t = 0;
        if ((threadIdx.x & 31) == 0) t = fixed + atomicAdd(ticket, 1u);
        return t;
    }
};

// -------------------------------------------------------------- emit pass
// Bound by instruction issue (2.5 a cycle and SM, 1380 a block at B = 8) and the
// latency of each block's dependent loads (rank -> descriptor and face records;
// list -> voxels), under which four CTAs of eight warps an SM run; five, at 48
// registers, take the L1 that serves the second reading of the list and are
// slower.  Against the tile, the rows and the row walks of the former pass:
// 1024^3 uint16 ball at B = 8, 231 -> 157 us; 512^3 float32 gyroid at B = 8,
// 225 -> 135; 640 x 512 x 448 uint16 at B = 16, one CTA of four warps an SM
// before, 411 -> 85; 1024 x 1024 x 314 uint8 at B = 3, 251 -> 152.
template <typename T, bool GENERIC, int BC, bool BIG>
__global__ void __launch_bounds__((BIG ? kBigWarps : kMaxWarps) * 32, GENERIC || BIG ? 1 : 4)
    pmb_emit_kernel(Problem p_, const uint32_t *__restrict__ ids, const uint32_t *__restrict__ rank_map,
                    const uint32_t *__restrict__ count_ptr, const mtx_meshlet_descriptor *__restrict__ desc,
                    const uint16_t *__restrict__ faces, const uint32_t *__restrict__ state,
                    uint32_t *__restrict__ indices, uint64_t tcap, uint64_t block_cap, void *__restrict__ vertices,
                    uint64_t vcap, uint32_t vfmt, uint32_t frame, uint32_t normals, DevStatus *st, uint32_t *done,
                    uint32_t *status_out, uint32_t *ticket) {
    // context voxels a lane loads at once: all of them for B <= 8
    constexpr int N = BIG ? 8 : BC == 3 || BC == 4 ? 2 : 7;
    extern __shared__ __align__(128) unsigned char smem[];
    Problem p = p_;
    if (BC) p.B = BC;
    const WPlan pl = make_emit_plan(p.B);
    const GridDiv dv = grid_div(p);
    uint64_t *tri = reinterpret_cast<uint64_t *>(smem);
    uint16_t *first = reinterpret_cast<uint16_t *>(smem + 8 * kTris);
    uint32_t *cmap = reinterpret_cast<uint32_t *>(smem + 8 * kTris + 512);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    unsigned char *ws = smem + emit_fixed_bytes(p.B) + warp * pl.bytes;
    build_tris(pl, tri, first);
    for (uint32_t j = threadIdx.x; j < pl.nb3; j += blockDim.x) cmap[j] = ctx_entry(pl, j);
    __syncthreads();
    uint32_t count = *count_ptr;
    if (count > block_cap) count = 0;  // reported by the count pass
    const uint32_t slot = list_state_words(p.B), B3 = pl.BB * pl.B;
    const uint64_t face_words = block_cap * face_stride16(p.B);
    uint32_t *jobs = reinterpret_cast<uint32_t *>(ws + pl.off_jobs);
    uint32_t *nbase = reinterpret_cast<uint32_t *>(ws + pl.off_nvid);
    unsigned char *vtab_b = ws + pl.off_vtab;
    uint16_t *vtab = reinterpret_cast<uint16_t *>(vtab_b);
    const uint32_t edge8 = BC == 8 ? ctx8_edge(lane) : 0u;

    const BlockShare share(count, gridDim.x * W, ticket);
    uint32_t r = first_block(p.B, warp, W), drawn = share.after(r), nb_rk = kNoVertex;
    Geo g{};
    mtx_meshlet_descriptor d{};
    if (r < count) {
        const uint32_t id = __ldg(ids + r);
        d = desc[r];
        g = block_geo(id, p, false, sizeof(T), dv);
        nb_rk = neighbour_rank(p, g, id, rank_map);
    }
    while (r < count) {
        const uint32_t nb_vb =
            (nb_rk != kNoVertex && MTX_BC(nb_rk, count, kBcDesc)) ? __ldg(&desc[nb_rk].vertexOffset) : kNoVertex;
        const uint32_t miss = __ballot_sync(0xffffffffu, nb_rk == kNoVertex) & 0xfeu;
        uint32_t rec[N];
        Ctx8 c8;
        if (BC == 8) c8 = ctx8_load(faces, nb_rk, edge8, face_words);
        else if (!BIG) ctx_load<N>(pl, faces, nb_rk, cmap, 0, rec, face_words);
        // the next block's place, descriptor and neighbour ranks
        const uint32_t rn = __shfl_sync(0xffffffffu, drawn, 0);
        drawn = share.after(rn);
        uint32_t nb_rk_n = kNoVertex;
        Geo gn{};
        mtx_meshlet_descriptor dn{};
        if (rn < count) {
            const uint32_t idn = __ldg(ids + rn);
            dn = desc[rn];
            gn = block_geo(idn, p, false, sizeof(T), dv);
            nb_rk_n = neighbour_rank(p, gn, idn, rank_map);
        }
        const uint32_t tbase = d.indexOffset / 3u, nv = d.vertexCount, nt = d.primitiveCount;
        const bool fits = (uint64_t)tbase + nt <= tcap && !(vertices && (uint64_t)d.vertexOffset + nv > vcap);
        if (!fits && lane == 0) report(st, MTX_ERR_CAPACITY, kSiteEmitCapacity, r, 2);
        if (fits && (nt || (vertices && nv))) {
            const uint32_t *own = state + (uint64_t)r * slot;
            const bool inner = g.ox + pl.B < p.X && g.oy + pl.B < p.Y && g.oz + pl.B < p.Z;
            if (BIG) {
                uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
                for (uint32_t i = lane; i < pl.B1 * pl.B1; i += 32) rows[i] = __ldg(own + i);
                __syncwarp();
                list_bits<BC>(p, pl, ws, g);
            }
            if (lane < 8) nbase[lane] = lane ? nb_vb : d.vertexOffset;

            // vertices, and this block's entries of the vertex table
            const uint32_t *rows = reinterpret_cast<const uint32_t *>(ws + pl.off_rows);
            const uint16_t *list = reinterpret_cast<const uint16_t *>(ws + pl.off_list);
            ListWalk l;
            uint32_t vrun = 0, out = 0, ahead = BIG ? 0u : __ldg(own + lane);
            for (uint32_t s0 = 0; vrun < nv && (BIG || s0 < slot); s0 += 32) {
                uint32_t e = ahead;
                if (BIG) {
                    const uint32_t n = list_next<true>(l, pl, ws);
                    if (!n) break;
                    e = lane < n ? listed_cell(p, pl, g, rows, list[l.done + lane], inner) : 0u;
                    l.done += n;
                } else if (s0 + 32 < slot) {
                    ahead = __ldg(own + s0 + 32 + lane);  // past the list's end: not used
                }
                if (!BIG && (e & 0xfffu) >= B3) e = 0;  // a list the count pass did not finish (reported there)
                uint32_t vt;
                const uint32_t rel = vrun + step_vertices(e >> 28, vt);
                queue_vertices(pl, e, rel, vtab, jobs, vertices ? out : vrun);
                vrun += vt;
                __syncwarp();
                if (vertices) {
                    const uint32_t avail = min(vrun, nv);  // never past the block's vertices
                    while (avail - out >= (vrun >= nv ? 1u : 32u)) {
                        const uint32_t k = min(32u, avail - out);
                        put_vertices<T, GENERIC>(p, pl, g, jobs, out, k, nv, inner, vertices, d.vertexOffset, vfmt,
                                                 frame, normals);
                        out += k;
                    }
                }
            }
            // the context layer's entries
            if (BC == 8) {
                ctx8_store(c8, edge8, vtab);
            } else if (!BIG) {
                ctx_store<N>(pl, vtab, cmap, 0, rec);
            } else {
                for (uint32_t j0 = 0; j0 < pl.nb3; j0 += 32 * N) {
                    ctx_load<N>(pl, faces, nb_rk, cmap, j0, rec, face_words);
                    ctx_store<N>(pl, vtab, cmap, j0, rec);
                }
            }
            __syncwarp();

            // triangles: each cell queues its jobs, resolved 32 at a time
            bool bad = false;
            uint32_t top = 0;
            out = 0;
            l = ListWalk{};
            ahead = BIG ? 0u : __ldg(own + lane);
            for (uint32_t s0 = 0; top < nt && (BIG || s0 < slot); s0 += 32) {
                uint32_t e = ahead;
                if (BIG) {
                    const uint32_t n = list_next<true>(l, pl, ws);
                    if (!n) break;
                    e = lane < n ? listed_cell(p, pl, g, rows, list[l.done + lane], inner) : 0u;
                    l.done += n;
                } else if (s0 + 32 < slot) {
                    ahead = __ldg(own + s0 + 32 + lane);
                }
                if (!BIG && (e & 0xfffu) >= B3) e = 0;
                const uint32_t f = first[(e >> 12) & 0xffu], n = f >> 12;
                uint32_t before, total;
                if (BIG) {
                    before = warp_excl_scan(n, total);
                } else {
                    before = (e >> 20) & 0xffu;
                    total = __shfl_sync(0xffffffffu, before + n, 31);
                }
                queue_triangles(pl, e, f, top + before, jobs, out);
                top += total;
                __syncwarp();
                const uint32_t avail = min(top, nt);  // never past the block's triangles
                const bool last = top >= nt;
                while (avail - out >= (last ? 1u : 32u)) {
                    const uint32_t k = min(32u, avail - out);
                    put_triangles(pl, vtab_b, tri, jobs, nbase, out, k, nt, indices + 3ull * tbase, miss, bad);
                    out += k;
                }
            }
            if (vrun != nv || top != nt) bad = true;
            if (bad) report(st, MTX_ERR_INTERNAL, kSiteEmitNeighbour, r, 3);
            __syncwarp();
        }
        r = rn;
        g = gn;
        d = dn;
        nb_rk = nb_rk_n;
    }
    // the CTA that ends last hands out the error code the call's kernels left
    // (a copy after the kernel cost 1.5 us and its gap)
    if (status_out) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(done, 1u) == gridDim.x - 1) {
                __threadfence();
                *status_out = ld_volatile(&st->code);
            }
        }
    }
}

// ------------------------------------------------------------------ host

bool tma_ok(const Problem &p) {
    const uint32_t esz = dtype_size(p.dtype);
    return ((uintptr_t)p.vol % 16 == 0) && (((uint64_t)p.X * esz) % 16 == 0);
}

static bool use_tma(const Problem &p, uint32_t staging) {
    if (staging == MTX_STAGING_LDG) return false;
    return tma_ok(p);
}

template <typename K>
static mtx_status grid_for(mtx_context *c, K kernel, int threads, uint32_t smem, uint32_t host_count, int warps,
                           unsigned &grid) {
    int per_sm = 0;
    const mtx_status r = ctas_per_sm(c, reinterpret_cast<const void *>(kernel), threads, smem, &per_sm);
    if (r != MTX_OK) return r;
    if (per_sm < 1) return fail(c, MTX_ERR_UNSUPPORTED, "extraction kernel does not fit on an SM");
    if (c->tuning.extractCtasPerSm) per_sm = std::min(per_sm, (int)c->tuning.extractCtasPerSm);
    uint64_t g = (uint64_t)per_sm * c->sm_count;
    if (host_count) g = std::min<uint64_t>(g, (host_count + warps - 1) / warps);
    grid = (unsigned)std::max<uint64_t>(g, 1);
    return MTX_OK;
}

// Warps a CTA: threads/32 of the options (up to kMaxWarps), else the context's
// tuning, else the pass's own choice -- eight, for B > 8 as many as fit -- and no
// more than the shared memory holds.  The tuning's largest count is for B > 8 the
// own choice too, so that mtx_autotune, which tries 2, 4 and 8, reaches it (CTAs of
// 8 and of 11 to 14 warps at B = 16: count 37 and 30.5 us, emit 112 and 85, the
// volume of kBigWarps).  A cap on the CTAs of an SM counts CTAs of four warps:
// it is set for the room that they leave to another stream's kernels.
static uint32_t cta_warps(const mtx_context *c, const ExtractArgs &a, uint32_t B, uint32_t fixed, uint32_t per_warp) {
    const bool capped = c->tuning.extractCtasPerSm != 0;
    const uint32_t own = capped ? 4 : B > 8 ? kBigWarps : kMaxWarps, tuned = c->tuning.extractWarps;
    const uint32_t asked = a.threads ? std::max(a.threads / 32, 1u) : B > 8 && tuned == kMaxWarps && !capped ? 0u : tuned;
    const uint32_t W = asked ? std::min<uint32_t>(asked, kMaxWarps) : own;
    const uint32_t room = c->max_smem_optin > (int)fixed ? (uint32_t)c->max_smem_optin - fixed : 0u;
    return std::min<uint32_t>(W, std::max<uint32_t>(1, room / per_warp));
}

template <typename T, bool TMA>
static auto count_fn(uint32_t B) {
    switch (B) {
    case 3: return pmb_count_kernel<T, TMA, 3>;
    case 4: return pmb_count_kernel<T, TMA, 4>;
    case 8: return pmb_count_kernel<T, TMA, 8>;
    case 16: return pmb_count_kernel<T, TMA, 16>;
    default: return pmb_count_kernel<T, TMA, 0>;
    }
}

template <typename T>
static mtx_status run_count(mtx_context *c, const Problem &p, const ExtractArgs &a, cudaStream_t s) {
    const uint32_t staging = a.staging ? a.staging : c->tuning.staging;
    const bool tma = use_tma(p, staging);
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (tma) {
        const mtx_status rs = make_volume_tensor_map(c, p, tile_pitch(p.B, sizeof(T), true), &map);
        if (rs != MTX_OK) return rs;
    }
    // the tile's element offsets in shared memory, where they fit 32 bits and B <= 8 keeps them small
    const bool use_off = !tma && p.B <= 8 && (uint64_t)(p.B + 1) * p.X * p.Y < (1ull << 32);
    const WPlan pl = make_count_plan(p.B, sizeof(T), tma);
    // eight warps a CTA: the case counts are loaded half as often as with four and blocks
    // next to each other share voxels in L1 (256^3 uint8 at B = 8 10.8 -> 9.7 us, 1024 x 1024 x 314
    // at B = 3 127 -> 123, 1024^3 uint16 at B = 8 94.6 -> 93.1)
    const uint32_t fixed = count_fixed_bytes(p.B, use_off), W = cta_warps(c, a, p.B, fixed, pl.bytes);
    const uint32_t smem = fixed + W * pl.bytes;
    auto k = tma ? count_fn<T, true>(p.B) : count_fn<T, false>(p.B);
    unsigned grid;
    mtx_status r = grid_for(c, k, W * 32, smem, a.host_count, p.B > 8 ? 1 : W, grid);
    if (r != MTX_OK) return r;
    k<<<grid, W * 32, smem, s>>>(p, map, a.ids, a.count, a.desc, a.desc_capacity, a.faces, a.state, a.totals,
                                 a.cell_cases, a.block_capacity, &c->ctrl->status, (uint64_t *)c->count_status.ptr,
                                 scan_tiles(std::min(a.block_capacity, a.desc_capacity)), &c->ctrl->count_ticket,
                                 use_off);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "count launch");
    return MTX_OK;
}

template <typename T, bool GENERIC>
static auto emit_fn(uint32_t B) {
    switch (B) {
    case 3: return pmb_emit_kernel<T, GENERIC, 3, false>;
    case 4: return pmb_emit_kernel<T, GENERIC, 4, false>;
    case 8: return pmb_emit_kernel<T, GENERIC, 8, false>;
    case 16: return pmb_emit_kernel<T, GENERIC, 16, true>;
    default: return B <= 8 ? pmb_emit_kernel<T, GENERIC, 0, false> : pmb_emit_kernel<T, GENERIC, 0, true>;
    }
}

template <typename T>
static mtx_status run_emit(mtx_context *c, const Problem &p, const ExtractArgs &a, cudaStream_t s) {
    const WPlan pl = make_emit_plan(p.B);
    const uint32_t fixed = emit_fixed_bytes(p.B), W = cta_warps(c, a, p.B, fixed, pl.bytes);
    const uint32_t smem = fixed + W * pl.bytes;
    const bool generic = a.vertices && (a.vertex_format != MTX_VERTEX_XYZ || a.frame != MTX_FRAME_VOXEL);
    auto k = generic ? emit_fn<T, true>(p.B) : emit_fn<T, false>(p.B);
    unsigned grid;
    mtx_status r = grid_for(c, k, W * 32, smem, a.host_count, p.B > 8 ? 1 : W, grid);
    if (r != MTX_OK) return r;
    k<<<grid, W * 32, smem, s>>>(p, a.ids, a.rank_map, a.count, a.desc, a.faces, a.state, a.indices, a.tri_capacity,
                                 a.block_capacity, a.vertices, a.vertex_capacity, a.vertex_format, a.frame, a.normals,
                                 &c->ctrl->status, &c->ctrl->emit_done, a.status_out, &c->ctrl->emit_ticket);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "emit launch");
    return MTX_OK;
}

template <bool EMIT>
static mtx_status launch_stage(mtx_context *c, const Problem &p, const ExtractArgs &a, cudaStream_t s) {
    if (p.B < 2 || p.B > MTX_MAX_BLOCK_EDGE) return fail(c, MTX_ERR_UNSUPPORTED, "block edge must be in [2, 16]");
    mtx_status rs = load_list_tables(c);
    if (rs != MTX_OK) return rs;
    switch (p.dtype) {
    case MTX_DTYPE_U8: return EMIT ? run_emit<uint8_t>(c, p, a, s) : run_count<uint8_t>(c, p, a, s);
    case MTX_DTYPE_U16: return EMIT ? run_emit<uint16_t>(c, p, a, s) : run_count<uint16_t>(c, p, a, s);
    default: return EMIT ? run_emit<float>(c, p, a, s) : run_count<float>(c, p, a, s);
    }
}

size_t block_state_bytes(uint32_t B) { return 4 * (size_t)list_state_words(B); }
size_t face_record_bytes(uint32_t B) { return 2 * (size_t)face_stride16(B); }

// The scan over up to `capacity` descriptors, behind a kernel that ran scan_reset for it.
static mtx_status run_scan(mtx_context *c, mtx_meshlet_descriptor *desc, const uint32_t *count, uint64_t capacity,
                           uint32_t *totals, uint32_t skip, cudaStream_t s) {
    pmb_scan_kernel<<<scan_tiles(capacity), kScanThreads, 0, s>>>(
        desc, count, capacity, (uint64_t *)c->count_status.ptr, &c->ctrl->count_ticket, totals, &c->ctrl->status,
        c->wait_polls ? c->wait_polls : kSpinLimit, skip, &c->ctrl->emit_ticket, &c->ctrl->emit_done);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "scan launch");
    return MTX_OK;
}

// Counts, faces and the scan: after this the descriptors and totals are final.
mtx_status launch_count(mtx_context *c, const Problem &p, const ExtractArgs &a, cudaStream_t s) {
    const uint64_t cap = std::min<uint64_t>(a.block_capacity, a.desc_capacity);
    mtx_status r = scratch_reserve(c, c->count_status, sizeof(uint64_t) * (size_t)scan_tiles(cap));
    if (r != MTX_OK) return r;
    if ((r = launch_stage<false>(c, p, a, s)) != MTX_OK) return r;
    return run_scan(c, a.desc, a.count, cap, a.totals, (c->withhold >> 1) & 1u, s);
}

// The descriptor scan on its own: vertexOffset / indexOffset of count
// descriptors from their vertexCount / primitiveCount (totals as launch_count).
// The kernel that fills the counts runs scan_reset with the words of desc_scan_words.
mtx_status desc_scan_words(mtx_context *c, uint64_t capacity, uint64_t **words, uint32_t *tiles, uint32_t **ticket) {
    mtx_status r = scratch_reserve(c, c->count_status, sizeof(uint64_t) * (size_t)scan_tiles(capacity));
    if (r != MTX_OK) return r;
    *words = (uint64_t *)c->count_status.ptr;
    *tiles = scan_tiles(capacity);
    *ticket = &c->ctrl->count_ticket;
    return MTX_OK;
}

mtx_status launch_desc_scan(mtx_context *c, mtx_meshlet_descriptor *desc, const uint32_t *count, uint64_t capacity,
                            uint32_t *totals, cudaStream_t s) {
    return run_scan(c, desc, count, capacity, totals, 0, s);
}

// Vertices (when a.vertices is set) and triangles.
mtx_status launch_emit(mtx_context *c, const Problem &p, const ExtractArgs &a, cudaStream_t s) {
    return launch_stage<true>(c, p, a, s);
}

MTX_BC_READER(bc_take_extract)

}  // namespace mtx
