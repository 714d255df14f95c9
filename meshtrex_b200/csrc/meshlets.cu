// Meshlet split: a post-pass over the canonical mesh that cuts each block's
// triangles into meshlets of at most maxVertices vertices and maxPrimitives
// triangles, each with its own copy of the vertices it uses -- the contract of
// meshtrex's renderer (render.task.glsl:55-250 accepts a triangle only if its
// three vertices lie in its meshlet's [vertexOffset, vertexOffset +
// vertexCount); the limits 64 / 126 are those of pmb.task.glsl:24-25).
//
// Rule (deterministic, the oracle's orc_meshlets): a block's triangles are
// taken in canonical order; a triangle joins the current meshlet unless its
// new vertices would take it past maxVertices or the meshlet already has
// maxPrimitives triangles, in which case a new meshlet starts with it.
// Meshlets never span blocks, and a meshlet's vertices are listed in the
// order its triangles first use them.
//
// One warp per block, 32 triangles at a time, one a lane.  The warp keeps the
// current meshlet's vertices in a hash table in shared memory: the three
// corners of every lane's triangle enter their ids, each slot keeping the
// lowest position that entered it, so a corner is new to the meshlet exactly
// when its own position won.  Ballots of the new corners number them and tell
// how many of the triangles still fit; the first that does not closes the
// meshlet, and the table starts again from it.  A count pass sizes every
// block's meshlets, the descriptor scan places them, and the emit pass writes
// descriptors, meshlet vertex ids and indices.
// Bound by the latency of the shared-memory atomics, three inserts a step: one
// triangle at a time (a ballot against the vertex list a corner) took 163 us to
// count and 191 to emit the 6.3 thousand blocks of a 509 x 387 x 301 volume at
// B = 8; this takes 12 and 15.
#include <algorithm>

#include "mtx_internal.h"

namespace mtx {

constexpr uint32_t kMeshletWarps = 4;
constexpr uint32_t kMaxMeshletVertices = 64;
constexpr uint32_t kSlots = 256;  // at most 64 vertices and the 96 corners of a step
constexpr uint32_t kNoId = 0xffffffffu;

template <bool EMIT>
__global__ void __launch_bounds__(kMeshletWarps * 32)
    meshlet_kernel(const mtx_meshlet_descriptor *__restrict__ blocks, const uint32_t *__restrict__ count_ptr,
                   const uint32_t *__restrict__ indices, uint32_t maxV, uint32_t maxP,
                   mtx_meshlet_descriptor *__restrict__ per_block, mtx_meshlet_descriptor *__restrict__ meshlets,
                   uint32_t *__restrict__ mverts, uint32_t *__restrict__ midx, uint64_t *scan_words,
                   uint32_t scan_ntiles, uint32_t *scan_ticket, uint32_t *totals) {
    if (!EMIT) scan_reset(scan_words, scan_ntiles, scan_ticket, totals);
    __shared__ __align__(16) uint32_t s_key[kMeshletWarps][kSlots], s_pos[kMeshletWarps][kSlots];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t *key = s_key[warp], *pos = s_pos[warp];
    auto clear = [&]() {
        __syncwarp();
        for (uint32_t i = lane; i < kSlots / 4; i += 32) {
            reinterpret_cast<uint4 *>(key)[i] = make_uint4(kNoId, kNoId, kNoId, kNoId);
            reinterpret_cast<uint4 *>(pos)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        }
        __syncwarp();
    };
    const uint32_t n = *count_ptr;
    for (uint32_t r = blockIdx.x * kMeshletWarps + warp; r < n; r += gridDim.x * kMeshletWarps) {
        const mtx_meshlet_descriptor b = blocks[r];
        const uint32_t t0 = b.indexOffset / 3u, t1 = t0 + b.primitiveCount;
        uint32_t mbase = 0, vbase = 0;  // EMIT: the block's first meshlet and first meshlet vertex
        if (EMIT) {
            mbase = per_block[r].indexOffset / 3u;
            vbase = per_block[r].vertexOffset;
        }
        uint32_t mcount = 0, vused = 0;  // meshlets closed, their vertices
        uint32_t cur_v = 0, cur_p = 0, first_t = t0;
        auto load = [&](uint32_t t, uint32_t id[3]) {
            for (uint32_t k = 0; k < 3; ++k) id[k] = t < t1 ? __ldg(indices + 3ull * t + k) : kNoId;
        };
        auto close = [&](uint32_t next_t) {
            if (EMIT && lane == 0)
                meshlets[mbase + mcount] = mtx_meshlet_descriptor{vbase + vused, 3u * first_t, cur_v, cur_p};
            vused += cur_v;
            ++mcount;
            cur_v = cur_p = 0;
            first_t = next_t;
        };
        clear();
        uint32_t t = t0, id[3], ahead[3];
        load(t + lane, id);
        while (t < t1) {
            load(t + 32 + lane, ahead);  // the step after this one, should all of this one fit
            const bool on = t + lane < t1;
            uint32_t slot[3];
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {
                if (!on) continue;
                uint32_t h = (id[k] * 2654435769u) >> 24;
                for (uint32_t probe = 0; probe < kSlots; ++probe) {  // 160 entries at most: a slot is found
                    const uint32_t was = atomicCAS(&key[h], kNoId, id[k]);
                    if (was == kNoId || was == id[k]) break;
                    h = (h + 1) & (kSlots - 1);
                }
                slot[k] = h;
                atomicMin(&pos[h], kMaxMeshletVertices + 3 * lane + k);
            }
            __syncwarp();
            bool fresh[3];
            uint32_t nb[3];
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {
                fresh[k] = on && pos[slot[k]] == kMaxMeshletVertices + 3 * lane + k;
                nb[k] = __ballot_sync(0xffffffffu, fresh[k]);
            }
            const uint32_t before = cur_v + __popc(nb[0] & lt) + __popc(nb[1] & lt) + __popc(nb[2] & lt);
            const uint32_t after = before + fresh[0] + fresh[1] + fresh[2];
            const uint32_t over = __ballot_sync(0xffffffffu, !on || after > maxV || cur_p + lane + 1 > maxP);
            const uint32_t take = over ? (uint32_t)(__ffs(over) - 1) : 32u;  // triangles that join the meshlet
            const uint32_t head = take == 32 ? 0xffffffffu : (1u << take) - 1u;
            // number the new vertices, then every corner reads its own
            if (EMIT || take == 32) {
                uint32_t at = before;
#pragma unroll
                for (uint32_t k = 0; k < 3; ++k)
                    if (fresh[k] && lane < take) {
                        pos[slot[k]] = at;
                        if (EMIT) mverts[vbase + vused + at] = id[k];
                        ++at;
                    }
                __syncwarp();
                if (EMIT && lane < take) {
#pragma unroll
                    for (uint32_t k = 0; k < 3; ++k) midx[3ull * (t + lane) + k] = vbase + vused + pos[slot[k]];
                }
            }
            cur_v += __popc(nb[0] & head) + __popc(nb[1] & head) + __popc(nb[2] & head);
            cur_p += take;
            t += take;
            if (take == 32) {
                for (uint32_t k = 0; k < 3; ++k) id[k] = ahead[k];
            } else if (t < t1) {  // triangle t does not fit: a new meshlet starts with it
                close(t);
                clear();
                load(t + lane, id);
            }
            __syncwarp();
        }
        if (cur_p > 0) close(t1);
        if (!EMIT && lane == 0) per_block[r] = mtx_meshlet_descriptor{0u, 0u, vused, mcount};
    }
}

// The same rule for meshlets of few triangles.  A warp has the corners of
// kFewTriangles triangles one a lane, and a step takes as many of them as join
// the current meshlet: equal vertices are found by a match across the lanes, so
// there is no table to fill and clear.  A meshlet that has room for more keeps its
// vertices one a lane, and the next step's corners are compared with each.
// The words ahead are in registers, as where a meshlet ends is known only at
// its end.
// Taken (few_triangles) for up to kFewTriangles triangles a meshlet or
// kFewVertices vertices; above, meshlets outgrow a step.  Count and emit of a
// 201 x 243 x 257 volume at B = 8, us, one triangle at a time / 32 a step / so:
// (maxVertices, maxPrimitives) = (3, 1) and (3, 126) 1314 / 1737 / 976, (4, 126)
// 1225 / 1129 / 671, (8, 126) 1152 / 446 / 302, (64, 10) 1124 / 196 / 169; 32 a
// step take 182 at (64, 11) and 272 at (12, 126).
constexpr uint32_t kFewTriangles = 10, kFewVertices = 8;
static bool few_triangles(uint32_t maxV, uint32_t maxP) { return maxP <= kFewTriangles || maxV <= kFewVertices; }

template <bool EMIT>
__global__ void __launch_bounds__(kMeshletWarps * 32)
    meshlet_few_kernel(const mtx_meshlet_descriptor *__restrict__ blocks, const uint32_t *__restrict__ count_ptr,
                       const uint32_t *__restrict__ indices, uint32_t maxV, uint32_t maxP,
                       mtx_meshlet_descriptor *__restrict__ per_block, mtx_meshlet_descriptor *__restrict__ meshlets,
                       uint32_t *__restrict__ mverts, uint32_t *__restrict__ midx, uint64_t *scan_words,
                       uint32_t scan_ntiles, uint32_t *scan_ticket, uint32_t *totals) {
    if (!EMIT) scan_reset(scan_words, scan_ntiles, scan_ticket, totals);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tri = lane / 3u;
    const uint32_t upto = lane < 3 * kFewTriangles ? (8u << (3 * tri)) - 1u : 0u;  // corners up to this one's triangle's last
    const uint32_t n = *count_ptr;
    for (uint32_t r = blockIdx.x * kMeshletWarps + warp; r < n; r += gridDim.x * kMeshletWarps) {
        const mtx_meshlet_descriptor b = blocks[r];
        const uint32_t t0 = b.indexOffset / 3u, nt = b.primitiveCount, words = 3 * nt;
        uint32_t mbase = 0, vbase = 0;  // EMIT: the block's first meshlet and first meshlet vertex
        if (EMIT) {
            mbase = per_block[r].indexOffset / 3u;
            vbase = per_block[r].vertexOffset;
        }
        const uint32_t *src = indices + 3ull * t0;
        auto load = [&](uint32_t w) { return w < words ? __ldg(src + w) : 0u; };
        uint32_t mcount = 0, vused = 0;                 // meshlets closed, their vertices
        uint32_t cur_v = 0, cur_p = 0, mine = 0;        // the current one's; lane v: its vertex v
        uint32_t base = 0, w0 = load(lane), w1 = load(32 + lane);  // the block's words from base on
        for (uint32_t t = 0; t < nt;) {
            if (3 * t - base >= 32) {  // a step moves by 30 words at most
                w0 = w1;
                base += 32;
                w1 = load(base + 32 + lane);
            }
            const uint32_t at = 3 * t - base + lane;
            const uint32_t a0 = __shfl_sync(0xffffffffu, w0, at & 31), a1 = __shfl_sync(0xffffffffu, w1, at & 31);
            const uint32_t id = at < 32 ? a0 : a1;
            const bool on = upto && cur_p + tri < maxP && t + tri < nt;
            uint32_t num = kNoId;  // the corner's vertex in the meshlet, where it has it already
            for (uint32_t v = 0; v < cur_v; ++v)
                if (__shfl_sync(0xffffffffu, mine, v) == id) num = v;
            const uint32_t live = __ballot_sync(0xffffffffu, on);
            const uint32_t first = __ffs(__match_any_sync(0xffffffffu, id) & live) - 1;  // the vertex's first corner
            const bool own = on && first == lane && num == kNoId;
            const uint32_t fresh = __ballot_sync(0xffffffffu, own);
            const uint32_t fit = __ballot_sync(0xffffffffu, on && cur_v + __popc(fresh & upto) <= maxV);
            const uint32_t corners = __ffs(~fit) - 1, take = corners / 3u;  // triangles that join the meshlet
            const uint32_t used = __popc(fresh & ((1u << corners) - 1u));
            if (EMIT && lane < corners) {
                if (num == kNoId) num = cur_v + __popc(fresh & ((1u << first) - 1u));
                midx[3ull * (t0 + t) + lane] = vbase + vused + num;
                if (own) mverts[vbase + vused + num] = id;
            }
            t += take;
            if (take == kFewTriangles && cur_p + take < maxP && t < nt) {  // room for more
                const uint32_t k = lane - cur_v;
                const uint32_t from = k < used ? __fns(fresh, 0, (int)k + 1) : 0u;
                const uint32_t got = __shfl_sync(0xffffffffu, id, from);
                if (k < used) mine = got;
                cur_v += used;
                cur_p += take;
                continue;
            }
            cur_v += used;
            cur_p += take;
            if (EMIT && lane == 0)
                meshlets[mbase + mcount] =
                    mtx_meshlet_descriptor{vbase + vused, 3u * (t0 + t - cur_p), cur_v, cur_p};
            vused += cur_v;
            ++mcount;
            cur_v = cur_p = 0;
        }
        if (!EMIT && lane == 0) per_block[r] = mtx_meshlet_descriptor{0u, 0u, vused, mcount};
    }
}

// vertexData[j] = vertices[mverts[j]], stride words of type V per record (16-byte
// words for the 32-byte records, else floats); 64-bit indices and divisions by a
// run-time stride, a float a thread, took 12.5 us where this takes 6.4 (the same volume).
template <typename V, uint32_t STRIDE>
__global__ void __launch_bounds__(256) gather_vertices_kernel(const V *__restrict__ vertices,
                                                              const uint32_t *__restrict__ mverts, uint64_t n,
                                                              uint32_t run_stride, V *__restrict__ out) {
    const uint32_t stride = STRIDE ? STRIDE : run_stride;
    const uint64_t total = n * stride, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
        const uint64_t j = i >> 32 ? i / stride : (uint32_t)i / stride, k = i - j * stride;
        out[i] = __ldg(vertices + (uint64_t)__ldg(mverts + j) * stride + k);
    }
}

}  // namespace mtx

using namespace mtx;

extern "C" mtx_status mtx_build_meshlets(mtx_context_t c, const mtx_extraction_output *ext, uint32_t maxVertices,
                                         uint32_t maxPrimitives, mtx_meshlet_output *out) {
    if (!c) return MTX_ERR_INVALID_ARG;
    DeviceGuard dg(c->device);
    join_extract(c);
    if (!ext || !out) return fail(c, MTX_ERR_INVALID_ARG, "null argument");
    memset(out, 0, sizeof(*out));
    if (maxVertices < 3 || maxVertices > kMaxMeshletVertices || maxPrimitives < 1 || maxPrimitives > 1024)
        return fail(c, MTX_ERR_INVALID_ARG, "meshlet limits: 3 <= maxVertices <= 64, 1 <= maxPrimitives <= 1024");
    const uint32_t nb = ext->meshletCount, T = ext->indexCount / 3u;
    const uint32_t stride = ext->vertexStride ? ext->vertexStride / 4u : 3u;
    out->vertexStride = 4u * stride;
    if (nb == 0 || T == 0) return MTX_OK;
    if (!ext->meshletDescriptorBuffer.ptr || !ext->indexBuffer.ptr || !ext->vertexBuffer.ptr ||
        !ext->meshletDescriptorCountBuffer.ptr)
        return fail(c, MTX_ERR_INVALID_ARG, "extraction output is incomplete");
    cudaStream_t s = c->stream;
    void *per_block = nullptr, *counters = nullptr;
    mtx_status r;
    if ((r = dev_alloc(c, &per_block, sizeof(mtx_meshlet_descriptor) * (size_t)nb)) != MTX_OK) return r;
    auto bail = [&](mtx_status st) {
        dev_free(c, per_block);
        dev_free(c, counters);
        mtx_meshlet_output_free(c, out);
        return st;
    };
    if ((r = dev_alloc(c, &counters, 16)) != MTX_OK) return bail(r);
    const auto *blocks = (const mtx_meshlet_descriptor *)ext->meshletDescriptorBuffer.ptr;
    const auto *count = (const uint32_t *)ext->meshletDescriptorCountBuffer.ptr;
    const auto *indices = (const uint32_t *)ext->indexBuffer.ptr;
    uint64_t *words;
    uint32_t ntiles, *ticket;
    if ((r = desc_scan_words(c, nb, &words, &ntiles, &ticket)) != MTX_OK) return bail(r);
    const uint32_t grid = std::min<uint32_t>((nb + kMeshletWarps - 1) / kMeshletWarps, 16u * c->sm_count);
    const bool few = few_triangles(maxVertices, maxPrimitives);
    (few ? meshlet_few_kernel<false> : meshlet_kernel<false>)<<<grid, kMeshletWarps * 32, 0, s>>>(
        blocks, count, indices, maxVertices, maxPrimitives, (mtx_meshlet_descriptor *)per_block, nullptr, nullptr,
        nullptr, words, ntiles, ticket, (uint32_t *)counters);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return bail(cuda_fail(c, e, "meshlet count launch"));
    if ((r = launch_desc_scan(c, (mtx_meshlet_descriptor *)per_block, count, nb, (uint32_t *)counters, s)) != MTX_OK)
        return bail(r);
    uint32_t *tot = c->pinned;
    if ((e = cudaMemcpyAsync(tot, counters, 16, cudaMemcpyDeviceToHost, s)) == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bail(cuda_fail(c, e, "meshlet totals"));
    const uint32_t MV = tot[0], M = tot[1] / 3u;
    void *p_desc, *p_mv, *p_idx, *p_vd;
    if ((r = dev_alloc(c, &p_desc, sizeof(mtx_meshlet_descriptor) * (size_t)M)) != MTX_OK) return bail(r);
    out->meshletDescriptorBuffer = {p_desc, sizeof(mtx_meshlet_descriptor) * (uint64_t)M};
    if ((r = dev_alloc(c, &p_mv, 4ull * MV)) != MTX_OK) return bail(r);
    out->meshletVertexBuffer = {p_mv, 4ull * MV};
    if ((r = dev_alloc(c, &p_idx, 12ull * T)) != MTX_OK) return bail(r);
    out->indexBuffer = {p_idx, 12ull * T};
    if ((r = dev_alloc(c, &p_vd, 4ull * stride * MV)) != MTX_OK) return bail(r);
    out->vertexBuffer = {p_vd, 4ull * stride * MV};
    (few ? meshlet_few_kernel<true> : meshlet_kernel<true>)<<<grid, kMeshletWarps * 32, 0, s>>>(
        blocks, count, indices, maxVertices, maxPrimitives, (mtx_meshlet_descriptor *)per_block,
        (mtx_meshlet_descriptor *)p_desc, (uint32_t *)p_mv, (uint32_t *)p_idx, nullptr, 0, nullptr, nullptr);
    if ((e = cudaGetLastError()) != cudaSuccess) return bail(cuda_fail(c, e, "meshlet emit launch"));
    const bool wide = stride == 8 && ((uintptr_t)ext->vertexBuffer.ptr | (uintptr_t)p_vd) % 16 == 0;
    const uint64_t work = (uint64_t)MV * (wide ? 2 : stride);
    const uint32_t ggrid = std::max(1u, (uint32_t)std::min<uint64_t>((work + 255) / 256, 32ull * c->sm_count));
    if (wide)
        gather_vertices_kernel<float4, 2><<<ggrid, 256, 0, s>>>((const float4 *)ext->vertexBuffer.ptr,
                                                                (const uint32_t *)p_mv, MV, 2, (float4 *)p_vd);
    else if (stride == 3)
        gather_vertices_kernel<float, 3><<<ggrid, 256, 0, s>>>((const float *)ext->vertexBuffer.ptr,
                                                               (const uint32_t *)p_mv, MV, 3, (float *)p_vd);
    else
        gather_vertices_kernel<float, 0><<<ggrid, 256, 0, s>>>((const float *)ext->vertexBuffer.ptr,
                                                               (const uint32_t *)p_mv, MV, stride, (float *)p_vd);
    if ((e = cudaGetLastError()) != cudaSuccess) return bail(cuda_fail(c, e, "meshlet gather launch"));
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return bail(cuda_fail(c, e, "meshlet build"));
    dev_free(c, {per_block, counters});
    out->meshletCount = M;
    out->vertexCount = MV;
    out->indexCount = 3u * T;
    return MTX_OK;
}

extern "C" mtx_status mtx_meshlet_output_free(mtx_context_t c, mtx_meshlet_output *out) {
    if (!c || !out) return MTX_ERR_INVALID_ARG;
    DeviceGuard dg(c->device);
    join_extract(c);
    dev_free(c, {out->meshletDescriptorBuffer.ptr, out->meshletVertexBuffer.ptr, out->vertexBuffer.ptr,
                 out->indexBuffer.ptr});
    const uint32_t stride = out->vertexStride;
    memset(out, 0, sizeof(*out));
    out->vertexStride = stride;
    return MTX_OK;
}
