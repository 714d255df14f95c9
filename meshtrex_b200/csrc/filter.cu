// Stage 2: active-block filtering with ordered stream compaction
// (meshtrex: occupiedBlockPrefixSum.comp.glsl:50-177, dispatched by
// activeBlockFilteringPass.cpp:87-153; CPU rule blockFilteringTestUtils.h:438-478).
//
// meshtrex scans within a workgroup and then takes one atomicAdd per
// workgroup, so the compacted list is ordered only inside a workgroup.  Here
// the CTAs take tiles of consecutive block ids by ticket (4096 a tile, 16
// per thread, so that a 1024^3 volume at block 8 is one tile a CTA; 1024 in
// the no-allocation entry point, whose scratch is sized for them), count their
// active blocks (two ballots a round of 64 blocks), and resolve their global offsets with a
// single-pass decoupled look-back over the tiles before them: the list comes out
// in ascending block order, which is the order the CPU rule produces.  The pass
// also writes the rank of every block (0xffffffff for inactive ones), which
// the extraction uses to find a neighbouring block's vertices.
#include <mutex>

#include "minmax_device.cuh"

namespace mtx {

constexpr int kFilterThreads = 256;
constexpr int kFilterItems = 16;       // blocks a thread: tiles of 4096
constexpr uint32_t kFilterCtas = 4;    // CTAs an SM
constexpr int kNoallocItems = 4;       // tiles of 1024 in mtx_filter_active_blocks_noalloc
constexpr int kFilterTile = kFilterThreads * kFilterItems;
constexpr int kNoallocTile = kFilterThreads * kNoallocItems;

// Look-back words and tickets of one launch.  EPOCH (the context's own
// scratch): a status word is flag << 62 | epoch << 32 | count and the ticket
// word epoch << 32 | ticket; the CTA that draws a launch's last ticket starts
// the next epoch, so that the words of earlier launches read as empty and
// nothing has to be zeroed between launches (three memsets of about 4 us
// each on the timeline before).  The words and the ticket are zeroed when the
// scratch grows, after an error and when the context's stream changes
// (rezero): launches of one context that overlapped would leave the ticket
// short of an epoch's end or past it, and every later one waiting for tiles
// that are never handed out; a ticket past the last is reported.  Otherwise (the
// no-allocation entry point, whose array holds 32-bit words): flag << 30 |
// count, zeroed before the launch.
// flag: 0 empty, 1 aggregate, 2 inclusive, 3 aborted.
constexpr uint32_t kFlagAgg = 1u, kFlagInc = 2u, kFlagAbort = 3u;
template <bool EPOCH> struct TileWord;
template <> struct TileWord<false> {
    using U = uint32_t;
    __device__ __forceinline__ static U make(uint32_t flag, uint32_t, uint32_t count) { return (flag << 30) | count; }
    __device__ __forceinline__ static uint32_t flag(U w, uint32_t) { return w >> 30; }
    __device__ __forceinline__ static uint32_t count(U w) { return w & 0x3fffffffu; }
    __device__ __forceinline__ static uint32_t draw(U *ticket, uint32_t, uint32_t &epoch) {
        epoch = 0;
        return atomicAdd(ticket, 1u);
    }
    __device__ __forceinline__ static bool torn(uint32_t, uint32_t) { return false; }
};
template <> struct TileWord<true> {
    using U = uint64_t;
    __device__ __forceinline__ static U make(uint32_t flag, uint32_t epoch, uint32_t count) {
        return ((U)flag << 62) | ((U)epoch << 32) | count;
    }
    __device__ __forceinline__ static uint32_t flag(U w, uint32_t epoch) {
        return ((uint32_t)(w >> 32) & 0x3fffffffu) == epoch ? (uint32_t)(w >> 62) : 0u;
    }
    __device__ __forceinline__ static uint32_t count(U w) { return (uint32_t)w; }
    __device__ __forceinline__ static uint32_t draw(U *ticket, uint32_t draws, uint32_t &epoch) {
        const U t = atomicAdd(reinterpret_cast<unsigned long long *>(ticket), 1ull);
        epoch = (uint32_t)(t >> 32);
        if ((uint32_t)t == draws - 1) st_volatile(ticket, (U)((epoch + 1) & 0x3fffffffu) << 32);
        return (uint32_t)t;
    }
    // A ticket past a launch's last: the word was not left at an epoch's start.
    __device__ __forceinline__ static bool torn(uint32_t t, uint32_t draws) { return t >= draws; }
};

// A tile is ITEMS / 2 rounds of 64 consecutive blocks a warp, lane l taking
// blocks 2 l and 2 l + 1 of each round: the loads and the rank stores are
// coalesced and the ranks follow from two ballots a round.  A CTA takes tiles
// until its ticket is past the last one: each of the `ctas` CTAs draws one
// ticket too many, so a launch draws ntiles - skip + ctas.  Before a tile is
// resolved, the next one's blocks are counted and published and the loads of
// the one after are on their way: a look-back finds the tiles before it
// published, instead of waiting for loads that are behind other tiles' waits.
// Nothing waits for a tile that no running CTA holds: a CTA publishes and
// resolves its tiles in the order of their tickets, and what a look-back needs
// of an earlier tile, its count, is published before that tile's CTA waits for
// anything later.
// skip: failure injection, the tickets start at tile `skip`.
// Bound by that chain of tiles: keys and ranks of 12.3 million blocks (1024 x
// 1024 x 314 at B = 3) take 25 us without it.  One tile a CTA, its look-back
// behind its own loads, 62 us; with the next tile's loads ahead, 54; with the
// next tile's count published ahead as well, 32 (windows of 128 tiles a round of
// reads: 37).  2.4 million blocks and fewer (4096 a CTA, four CTAs an SM), a tile or
// less a CTA: 1 to 2 us less.
template <int ITEMS, bool EPOCH>
__device__ __forceinline__ void filter_tiles(const uint2 *__restrict__ leaf, uint64_t nblocks, uint32_t ntiles,
                                             uint32_t ctas, uint32_t dtype, float iso, uint32_t *__restrict__ ids,
                                             uint32_t *__restrict__ rank_map, uint32_t *__restrict__ count_out,
                                             typename TileWord<EPOCH>::U *tile_status,
                                             typename TileWord<EPOCH>::U *ticket, DevStatus *st, uint32_t spin_limit,
                                             uint32_t skip) {
    using TW = TileWord<EPOCH>;
    constexpr int R = ITEMS / 2, W = kFilterThreads / 32;
    static_assert(ITEMS <= 32, "a tile's ballots, one a lane");
    __shared__ uint32_t s_draw[2], s_epoch, s_prefix, s_abort;
    __shared__ uint32_t s_sum[2][W];  // active blocks of each warp, of the present tile and the next
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint32_t draws = ntiles - skip + ctas;
    if (threadIdx.x == 0) {
        uint32_t epoch;
        const uint32_t first = TW::draw(ticket, draws, epoch);
        s_draw[0] = first + skip;
        s_epoch = epoch;
        const bool torn = TW::torn(first, draws);
        if (torn) report(st, MTX_ERR_INTERNAL, kSiteFilterTicket, first, draws);
        if (torn || skip >= ntiles) *count_out = 0;  // no CTA may take the last tile
    }
    __syncthreads();
    uint32_t t = s_draw[0], e;
    const uint32_t epoch = s_epoch;
    if (t >= ntiles) return;

    auto base_of = [&](uint32_t tile) {
        return (uint64_t)tile * (kFilterThreads * ITEMS) + (uint64_t)warp * (32 * ITEMS) + 2 * lane;
    };
    uint4 v[R];  // the blocks of the tile to count next
    auto load = [&](uint32_t tile) {
        const uint64_t base = base_of(tile);
#pragma unroll
        for (int k = 0; k < R; ++k) {  // {0, 0} is an inactive block
            const uint64_t i = base + 64 * k;
            v[k] = make_uint4(0, 0, 0, 0);
            if (i + 1 < nblocks) {
                v[k] = __ldg(reinterpret_cast<const uint4 *>(leaf + i));
            } else if (i < nblocks) {
                const uint2 one = __ldg(leaf + i);
                v[k].x = one.x;
                v[k].y = one.y;
            }
        }
    };
    // The ballots of v, lane 2 k the first and 2 k + 1 the second blocks' of round k; the warp's sum.
    auto count = [&](uint32_t *sum) {
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint32_t b0 = __ballot_sync(0xffffffffu, block_active(dtype, v[k].x, v[k].y, iso));
            const uint32_t b1 = __ballot_sync(0xffffffffu, block_active(dtype, v[k].z, v[k].w, iso));
            if (lane == 2 * k) bits = b0;
            if (lane == 2 * k + 1) bits = b1;
        }
        const uint32_t n = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(bits));
        if (lane == 0) sum[warp] = n;
        return bits;
    };
    auto publish = [&](uint32_t tile, const uint32_t *sum) {  // warp 0
        const uint32_t n = __reduce_add_sync(0xffffffffu, lane < W ? sum[lane] : 0u);
        if (lane == 0) st_volatile(&tile_status[tile], TW::make(tile ? kFlagAgg : kFlagInc, epoch, n));
    };

    load(t);
    if (threadIdx.x == 0) s_draw[1] = TW::draw(ticket, draws, e) + skip;
    uint32_t bits = count(s_sum[0]);
    __syncthreads();
    if (warp == 0) publish(t, s_sum[0]);
    uint32_t next = s_draw[1];
    if (next < ntiles) load(next);
    for (uint32_t buf = 0; t < ntiles; buf ^= 1) {
        uint32_t after = next, bits_next = 0;
        if (next < ntiles) {
            if (threadIdx.x == 0) s_draw[0] = TW::draw(ticket, draws, e) + skip;
            bits_next = count(s_sum[buf ^ 1]);
        }
        __syncthreads();
        if (next < ntiles) {
            after = s_draw[0];
            if (warp == 0) publish(next, s_sum[buf ^ 1]);
            if (after < ntiles) load(after);
        }
        uint32_t total = 0, excl = 0;
#pragma unroll
        for (uint32_t w = 0; w < W; ++w) {
            if (w == warp) excl = total;
            total += s_sum[buf][w];
        }
        if (warp == 0) {
            uint32_t prefix = 0;
            bool abort = false;
            if (t > 0) {
                int64_t j = (int64_t)t - 1;
                uint32_t spins = 0;
                while (true) {
                    const int64_t k = j - (int64_t)lane;
                    const typename TW::U w = k >= 0 ? ld_volatile(&tile_status[k]) : TW::make(kFlagInc, epoch, 0);
                    const uint32_t flag = TW::flag(w, epoch);
                    abort = __any_sync(0xffffffffu, flag == kFlagAbort);
                    if (abort) break;
                    const uint32_t inc = __ballot_sync(0xffffffffu, flag == kFlagInc);
                    const uint32_t emp = __ballot_sync(0xffffffffu, flag == 0u);
                    const uint32_t first = inc ? (uint32_t)(__ffs(inc) - 1) : 32u;
                    const uint32_t window = first >= 31 ? 0xffffffffu : ((2u << first) - 1u);
                    if (emp & window) {
                        if (++spins >= spin_limit) {
                            if (lane == 0) report(st, MTX_ERR_TIMEOUT, kSiteFilterLookback, t, (uint32_t)j);
                            abort = true;
                            break;
                        }
                        backoff(spins);
                        continue;
                    }
                    prefix += lane <= first ? TW::count(w) : 0u;
                    if (first < 32) break;
                    j -= 32;
                }
                prefix = __reduce_add_sync(0xffffffffu, prefix);
                if (lane == 0)
                    st_volatile(&tile_status[t],
                                abort ? TW::make(kFlagAbort, epoch, 0) : TW::make(kFlagInc, epoch, prefix + total));
            }
            if (lane == 0) {
                s_prefix = prefix;
                s_abort = abort ? 1u : 0u;
                if (t == ntiles - 1) *count_out = abort ? 0u : prefix + total;
            }
        }
        __syncthreads();
        if (!s_abort) {
            uint32_t r = s_prefix + excl;
            const uint64_t base = base_of(t);
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const uint64_t i = base + 64 * k;
                const uint32_t b0 = __shfl_sync(0xffffffffu, bits, 2 * k), b1 = __shfl_sync(0xffffffffu, bits, 2 * k + 1);
                const bool f0 = (b0 >> lane) & 1u, f1 = (b1 >> lane) & 1u;
                const uint32_t r0 = r + __popc(b0 & lt) + __popc(b1 & lt), r1 = r0 + f0;
                if (f0 && MTX_BC(r0, nblocks, kBcRank)) ids[r0] = (uint32_t)i;
                if (f1 && MTX_BC(r1, nblocks, kBcRank)) ids[r1] = (uint32_t)i + 1;
                // rank of every block of the tile: its rank if active, else kNoRank
                const uint2 rk = make_uint2(f0 ? r0 : 0xffffffffu, f1 ? r1 : 0xffffffffu);
                if (i + 1 < nblocks) *reinterpret_cast<uint2 *>(rank_map + i) = rk;
                else if (i < nblocks) rank_map[i] = rk.x;
                r += __popc(b0) + __popc(b1);
            }
        }
        t = next;
        next = after;
        bits = bits_next;
    }
}

template <int ITEMS, bool EPOCH>
__global__ void __launch_bounds__(kFilterThreads, 4)
    filter_compact_kernel(const uint2 *__restrict__ leaf, uint64_t nblocks, uint32_t ntiles, uint32_t dtype,
                          float iso, uint32_t *__restrict__ ids, uint32_t *__restrict__ rank_map,
                          uint32_t *__restrict__ count_out, typename TileWord<EPOCH>::U *tile_status,
                          typename TileWord<EPOCH>::U *ticket, DevStatus *st, uint32_t spin_limit, uint32_t skip) {
    filter_tiles<ITEMS, EPOCH>(leaf, nblocks, ntiles, gridDim.x, dtype, iso, ids, rank_map, count_out, tile_status,
                               ticket, st, spin_limit, skip);
}

// The compaction and the octree in one launch (the asynchronous whole-path
// call): both read the leaf level, neither waits for the other, and the
// octree's few CTAs run under the compaction's look-back chain.  As two
// launches they took 6.4 + 6.4 us for a 256^3 volume at B = 8, and a gap.
__global__ void __launch_bounds__(kFilterThreads, 4)
    filter_octree_kernel(const uint2 *__restrict__ leaf, uint64_t nblocks, uint32_t ntiles, uint32_t dtype, float iso,
                         uint32_t *__restrict__ ids, uint32_t *__restrict__ rank_map, uint32_t *__restrict__ count_out,
                         uint64_t *tile_status, uint64_t *ticket, DevStatus *st, uint32_t spin_limit, uint32_t skip,
                         uint32_t ctas, const __grid_constant__ PyrAll L) {
    static_assert(kPyrThreads == kFilterThreads, "one CTA size for both");
    __shared__ uint2 s_part[2][8][8];
    __shared__ uint32_t s_last;
    if (blockIdx.x < ctas)
        filter_tiles<kFilterItems, true>(leaf, nblocks, ntiles, ctas, dtype, iso, ids, rank_map, count_out,
                                         tile_status, ticket, st, spin_limit, skip);
    else
        pyramid_part(L, blockIdx.x - ctas, s_part, &s_last);
}

MTX_BC_READER(bc_take_filter)

mtx_status launch_filter(mtx_context *c, const Problem &p, const uint2 *leaf, uint32_t *ids, uint32_t *rank_map,
                         uint32_t *count, cudaStream_t s, const PyrAll *octree) {
    if (p.nblocks >= (1ull << 30)) return fail(c, MTX_ERR_UNSUPPORTED, "more than 2^30 blocks");
    const uint32_t ntiles = (uint32_t)((p.nblocks + kFilterTile - 1) / kFilterTile);
    const void *before = c->filter_status.ptr;
    const size_t size = c->filter_status.size;
    mtx_status rs = scratch_reserve(c, c->filter_status, sizeof(uint64_t) * (size_t)ntiles);
    if (c->filter_status.ptr != before || c->filter_status.size != size)
        c->rezero |= mtx_context::kNewWords;  // no epoch's
    if (rs != MTX_OK || (rs = rezero(c, s)) != MTX_OK) return rs;
    uint64_t *words = (uint64_t *)c->filter_status.ptr;
    const uint32_t ctas = std::min(ntiles, kFilterCtas * (uint32_t)c->sm_count);
    const uint32_t polls = c->wait_polls ? c->wait_polls : kSpinLimit, skip = c->withhold & 1u;
    if (octree && octree->ntiles)
        filter_octree_kernel<<<ctas + octree->ctas, kFilterThreads, 0, s>>>(
            leaf, p.nblocks, ntiles, p.dtype, p.iso, ids, rank_map, count, words, &c->ctrl->filter_ticket,
            &c->ctrl->status, polls, skip, ctas, *octree);
    else
        filter_compact_kernel<kFilterItems, true><<<ctas, kFilterThreads, 0, s>>>(
            leaf, p.nblocks, ntiles, p.dtype, p.iso, ids, rank_map, count, words, &c->ctrl->filter_ticket,
            &c->ctrl->status, polls, skip);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "filter launch");
    return MTX_OK;
}

}  // namespace mtx

// ------------------------------------------------- compaction without allocation
// Some callers cannot allocate device memory while they run: an application
// with its own fixed device-memory budget, or code that runs where
// cudaMalloc is not allowed.  For them, mtx_filter_active_blocks_noalloc
// runs the same compaction kernel with its scratch (one look-back word per
// 1024-block tile and a ticket counter) in the statically sized array below
// instead of a context's arena.  The array lives in every GPU that loads the
// library until the process exits; it bounds the problem to
// kNoallocMaxTiles * 1024 blocks.  Calls that overlap on the GPU (two
// streams, two host threads) share the array and race: serialise them.
namespace mtx {
constexpr uint32_t kNoallocMaxTiles = 65536;                // up to 65536 * 1024 = 67,108,864 blocks
constexpr uint32_t kNoallocTicket = kNoallocMaxTiles;       // word index of the tile ticket
constexpr uint32_t kNoallocWords = kNoallocMaxTiles + 64;   // 256 KiB + 256 bytes
}  // namespace mtx

// Words [0, ntiles) hold the look-back status of each tile, then the ticket
// counter.
static __device__ __align__(256) uint32_t g_noalloc_scratch[mtx::kNoallocWords];

namespace {
// Device address of g_noalloc_scratch in the calling thread's current CUDA
// context.  Host code must not use the symbol itself as a pointer: on the
// host it names a stand-in object, not device memory.  The address belongs
// to the context that loaded the module, so it is cached per context id
// (cuCtxGetId, unique for the life of the process): after cudaDeviceReset,
// or under another context on the same device, the next call looks it up
// again instead of using a stale address.
typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long *);
struct NoallocSlot {
    unsigned long long ctx_id;
    uint32_t *ptr;
};
constexpr int kNoallocSlots = 64;
NoallocSlot g_noalloc_slots[kNoallocSlots] = {};
int g_noalloc_next = 0;
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
std::mutex g_noalloc_mu;

cudaError_t noalloc_scratch(int device, uint32_t **out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_ctx_get_current || !g_ctx_get_id) {
        void *f0 = nullptr, *f1 = nullptr;
        cudaDriverEntryPointQueryResult q0, q1;
        cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault, &q0);
        if (e != cudaSuccess) return e;
        e = cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault, &q1);
        if (e != cudaSuccess) return e;
        if (q0 != cudaDriverEntryPointSuccess || q1 != cudaDriverEntryPointSuccess || !f0 || !f1)
            return cudaErrorNotSupported;
        g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f0);
        g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f1);
    }
    CUcontext cu = nullptr;
    if (g_ctx_get_current(&cu) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
    if (!cu) {  // no context yet on this thread: bind the device's primary context, as a launch would
        const cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return e;
        if (g_ctx_get_current(&cu) != CUDA_SUCCESS || !cu) return cudaErrorDeviceUninitialized;
    }
    unsigned long long id = 0;
    if (g_ctx_get_id(cu, &id) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
    for (const NoallocSlot &s : g_noalloc_slots)
        if (s.ptr && s.ctx_id == id) {
            *out = s.ptr;
            return cudaSuccess;
        }
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_slots[g_noalloc_next] = {id, static_cast<uint32_t *>(p)};
    g_noalloc_next = (g_noalloc_next + 1) % kNoallocSlots;
    *out = static_cast<uint32_t *>(p);
    return cudaSuccess;
}
}  // namespace

extern "C" mtx_status mtx_filter_active_blocks_noalloc(const uint32_t *leaf_minmax, uint64_t total_blocks,
                                                       uint32_t dtype, float isovalue, uint32_t *compacted_ids,
                                                       uint32_t *block_rank, uint32_t *active_count,
                                                       uint32_t *device_status, void *stream) {
    using namespace mtx;
    if (!leaf_minmax || !compacted_ids || !block_rank || !active_count || !device_status ||
        dtype > MTX_DTYPE_F32 || total_blocks == 0)
        return MTX_ERR_INVALID_ARG;
    // the kernel reads the keys and writes the ranks as 16-byte words
    if ((reinterpret_cast<uintptr_t>(leaf_minmax) | reinterpret_cast<uintptr_t>(block_rank)) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(compacted_ids) % 4 != 0 || reinterpret_cast<uintptr_t>(active_count) % 4 != 0 ||
        reinterpret_cast<uintptr_t>(device_status) % 4 != 0)
        return MTX_ERR_INVALID_ARG;
    if (total_blocks > (uint64_t)kNoallocMaxTiles * kNoallocTile) return MTX_ERR_CAPACITY;
    const uint32_t ntiles = (uint32_t)((total_blocks + kNoallocTile - 1) / kNoallocTile);
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return MTX_ERR_NO_DEVICE;
    }
    uint32_t *sc = nullptr;
    if (noalloc_scratch(device, &sc) != cudaSuccess) {
        cudaGetLastError();
        return MTX_ERR_CUDA;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DevStatus *st = reinterpret_cast<DevStatus *>(device_status);
    // the array keeps the previous call's contents: clear what must start at zero
    if (cudaMemsetAsync(sc, 0, sizeof(uint32_t) * (size_t)ntiles, s) != cudaSuccess ||
        cudaMemsetAsync(sc + kNoallocTicket, 0, sizeof(uint32_t), s) != cudaSuccess ||
        cudaMemsetAsync(active_count, 0, sizeof(uint32_t), s) != cudaSuccess ||
        cudaMemsetAsync(device_status, 0, sizeof(DevStatus), s) != cudaSuccess) {
        cudaGetLastError();
        return MTX_ERR_CUDA;
    }
    filter_compact_kernel<kNoallocItems, false><<<std::min(ntiles, kFilterCtas * (uint32_t)sms), kFilterThreads, 0, s>>>(
        reinterpret_cast<const uint2 *>(leaf_minmax), total_blocks, ntiles, dtype, isovalue, compacted_ids, block_rank,
        active_count, sc, sc + kNoallocTicket, st, kSpinLimit, 0u);
    if (cudaGetLastError() != cudaSuccess) return MTX_ERR_CUDA;
    return MTX_OK;
}
