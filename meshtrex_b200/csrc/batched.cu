// Batched extraction: every (volume, isovalue) job of a batch in two
// launches.  The leaf min/max of all volumes runs as one kernel (a volume's
// min/max serves all of its isovalues); one persistent kernel then takes all
// jobs through filtering with ordered compaction, per-block counts, the
// offset scan and emission.  meshtrex extracts one volume at one isovalue per
// call (src/meshtrex.cpp:107-141); each job here gives exactly what that
// sequence gives for its volume, block edge and isovalue.
//
// The persistent kernel hands out work by ticket and a CTA only ever waits
// for work that was handed out before its own (to CTAs that are running), so
// it needs neither a co-residency guarantee nor a grid barrier:
//
//  filter   1024-block tiles of every job in job order, under one decoupled
//           look-back: pooled rank = (job, block id) order.  Each job's rank
//           map holds pooled ranks.
//  count    one active block per warp item, as in the single-volume count pass
//  scan     1024-descriptor tiles under a segmented look-back: a job's
//           offsets restart at its first block
//  bases    one CTA: each job's first vertex and index in the pooled buffers,
//           capacity checks
//  emit     one active block per warp item; indices count from the job's
//           first vertex
//
// Data written by an earlier phase of the same launch is read with L2-only
// loads (never the read-only cache), after a fenced hand-over counter.
#include <algorithm>
#include <vector>

#include "minmax_device.cuh"
#include "pmb_lists.cuh"

namespace mtx {

constexpr uint32_t kBThreads = 256;
constexpr uint32_t kBItems = 4;
constexpr uint32_t kBTile = kBThreads * kBItems;
constexpr uint32_t kBWarps = kBThreads / 32;
// triangle table, the cases' first triangles and triangle counts
constexpr uint32_t kBFixedBytes = (8 * kTris + 512 + 256 + 127) / 128 * 128;
constexpr uint32_t kBChunk = 2;                 // active blocks per warp ticket
constexpr uint32_t kPhaseSpinLimit = 1u << 26;  // about 17 s of polling at the longest back-off

struct BVol {
    Problem p;      // isovalue unset
    WPlan pl;       // this volume's block edge, offsets of the batch's shared warp layout
    GridDiv dv;     // reciprocals of the grid's row and slice sizes (block_geo)
    uint32_t nXS, nbs, zchunk;  // min/max: strips, blocks a strip (RowCut), slabs a warp
    uint32_t wide, aligned;     // RowCut
    bool nan_zero;              // minmax_leaf_rows_warp
    uint64_t leaf_off;  // first leaf entry of the volume in the pooled leaf array
    uint64_t mm_begin;  // first min/max warp of the volume
};

struct BJob {
    uint32_t vol;
    float iso;
    uint32_t tile_begin, ntiles;  // filter tiles of the job
    uint64_t rank_off;            // first word of the job's rank map
};

// Zeroed before every run.
struct BCtrl {
    uint32_t filter_ticket, filter_done, total_active, count_ticket;
    uint32_t count_done, scan_ticket, scan_done, bases_ticket;
    uint32_t bases_ready, emit_ok, emit_ticket, pad;
    uint64_t total_vertices, total_triangles;
    DevStatus status;
};

struct BatchArgs {
    const BVol *vols;
    const BJob *jobs;
    const uint32_t *tile_job;
    const uint2 *leaf;
    uint32_t njobs, n_ftiles;
    uint32_t ws_bytes, face_stride, state_stride;
    uint32_t block_warps;  // warps of a CTA that take count/emit work (the layout fits that many)
    uint32_t *rank_pool;
    uint32_t *ids, *job_of;
    uint64_t block_cap;
    mtx_meshlet_descriptor *desc;
    uint16_t *faces;
    uint32_t *state;  // inside rows of each active block (count -> emit)
    uint32_t *filter_status;
    uint64_t *scan_status;
    mtx_batch_job_result *res;
    uint32_t *job_end;
    void *vertices;
    uint64_t vcap;
    uint32_t *indices;
    uint64_t tcap;
    uint32_t vfmt, frame, normals, vsz;
    BCtrl *ctrl;
};

// ------------------------------------------------------------ min/max
// Every volume's leaf min/max in one launch; warp w belongs to the last
// volume whose mm_begin <= w.  The rows pass for every type: its strips are
// 64 to 256 columns wide where those of the 16-byte pass span 128 to 512, so
// narrow volumes keep their lanes busy (16 mixed volumes of edges 64 to 256 at
// B = 8: 106 -> 46 us, 96 registers instead of 216).
__global__ void __launch_bounds__(128) batch_minmax_kernel(const BVol *__restrict__ vols, uint32_t nvol,
                                                           uint64_t nwarps, uint2 *__restrict__ leaf) {
    __shared__ uint32_t s_col[4][128];
    const uint64_t w = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= nwarps) return;  // uniform per warp
    uint32_t lo = 0, hi = nvol - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (vols[mid].mm_begin <= w) lo = mid;
        else hi = mid - 1;
    }
    const BVol &v = vols[lo];
    const Problem &p = v.p;
    const uint64_t lw = w - v.mm_begin;
    uint2 *out = leaf + v.leaf_off;
    if (!v.nXS) {  // rows_ok: one block a thread
        const uint64_t b = lw * 32 + (threadIdx.x & 31);
        if (b >= p.nblocks) return;
        switch (p.dtype) {
        case MTX_DTYPE_U8: minmax_leaf_one<uint8_t>((const uint8_t *)p.vol, p.X, p.Y, p.Z, p.B, p.GX, p.GY, b, out); break;
        case MTX_DTYPE_U16: minmax_leaf_one<uint16_t>((const uint16_t *)p.vol, p.X, p.Y, p.Z, p.B, p.GX, p.GY, b, out); break;
        default: minmax_leaf_one<float>((const float *)p.vol, p.X, p.Y, p.Z, p.B, p.GX, p.GY, b, out); break;
        }
        return;
    }
#define MTX_MM(T, W, NR, AL)                                                                                          \
    minmax_leaf_rows_warp<T, W, NR, AL>((const T *)p.vol, p.X, p.Y, p.Z, p.B, p.GX, p.GY, p.GZ, v.nXS, v.nbs, v.zchunk, \
                                        lw, out, s_col[threadIdx.x >> 5], v.nan_zero)
    // type, words of a row a lane, block edge 8 at compile time, aligned rows
    switch (p.dtype * 8 + (p.B == 8) * 4 + v.wide * 2 + v.aligned) {
    case MTX_DTYPE_U8 * 8 + 0: MTX_MM(uint8_t, 1, 0, false); break;
    case MTX_DTYPE_U8 * 8 + 1: MTX_MM(uint8_t, 1, 0, true); break;
    case MTX_DTYPE_U8 * 8 + 2: MTX_MM(uint8_t, 2, 0, false); break;
    case MTX_DTYPE_U8 * 8 + 3: MTX_MM(uint8_t, 2, 0, true); break;
    case MTX_DTYPE_U8 * 8 + 4: MTX_MM(uint8_t, 1, 9, false); break;
    case MTX_DTYPE_U8 * 8 + 5: MTX_MM(uint8_t, 1, 9, true); break;
    case MTX_DTYPE_U8 * 8 + 6: MTX_MM(uint8_t, 2, 9, false); break;
    case MTX_DTYPE_U8 * 8 + 7: MTX_MM(uint8_t, 2, 9, true); break;
    case MTX_DTYPE_U16 * 8 + 2: MTX_MM(uint16_t, 2, 0, false); break;
    case MTX_DTYPE_U16 * 8 + 3: MTX_MM(uint16_t, 2, 0, true); break;
    case MTX_DTYPE_U16 * 8 + 6: MTX_MM(uint16_t, 2, 9, false); break;
    case MTX_DTYPE_U16 * 8 + 7: MTX_MM(uint16_t, 2, 9, true); break;
    case MTX_DTYPE_F32 * 8 + 2:
    case MTX_DTYPE_F32 * 8 + 3: MTX_MM(float, 2, 0, true); break;
    default: MTX_MM(float, 2, 9, true); break;
    }
#undef MTX_MM
}

// ------------------------------------------------------------ hand-over
// CTA-wide bounded wait until *word >= target.  Thread 0 polls, then fences
// so that what the producers wrote before their counter update is visible.
__device__ __forceinline__ bool cta_wait_geq(const uint32_t *word, uint32_t target, DevStatus *st, uint32_t phase,
                                             uint32_t *s_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t ok = 1, spins = 0;
        while (ld_volatile(word) < target) {
            if (++spins >= kPhaseSpinLimit) {
                report(st, MTX_ERR_TIMEOUT, kSiteBatched, phase, target);
                ok = 0;
                break;
            }
            backoff(spins);
        }
        __threadfence();
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
}

// Every thread fences its writes, then one thread bumps the counter.
__device__ __forceinline__ void cta_signal(uint32_t *word, uint32_t v) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(word, v);
}

__device__ __forceinline__ uint32_t warp_ticket(uint32_t *word, uint32_t n) {
    uint32_t t = 0;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(word, n);
    return __shfl_sync(0xffffffffu, t, 0);
}

// ------------------------------------------------------------ filter
// Tile words: [31:30] flag (1 aggregate, 2 inclusive, 3 aborted), [29:0] count.
__device__ __forceinline__ bool lookback_sum30(const uint32_t *status, uint32_t t, uint32_t &prefix,
                                               DevStatus *st) {
    const uint32_t lane = threadIdx.x & 31;
    prefix = 0;
    int64_t j = (int64_t)t - 1;
    uint32_t spins = 0;
    while (true) {
        const int64_t k = j - (int64_t)lane;
        const uint32_t w = k >= 0 ? ld_volatile(&status[k]) : (2u << 30);
        const uint32_t flag = w >> 30;
        if (__any_sync(0xffffffffu, flag == 3u)) return false;
        const uint32_t inc = __ballot_sync(0xffffffffu, flag == 2u);
        const uint32_t emp = __ballot_sync(0xffffffffu, flag == 0u);
        const uint32_t first = inc ? (uint32_t)(__ffs(inc) - 1) : 32u;
        const uint32_t window = first >= 31 ? 0xffffffffu : ((2u << first) - 1u);
        if (emp & window) {
            if (++spins >= kSpinLimit) {
                if (lane == 0) report(st, MTX_ERR_TIMEOUT, kSiteFilterLookback, t, (uint32_t)j);
                return false;
            }
            backoff(spins);
            continue;
        }
        uint32_t v = lane <= first ? (w & 0x3fffffffu) : 0u;
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        prefix += v;
        if (first < 32) return true;
        j -= 32;
    }
}

__device__ __forceinline__ void batch_filter_tile(const BatchArgs &a, uint32_t t, uint32_t *s_tmp, uint32_t *s_u) {
    const uint32_t tid = threadIdx.x;
    const uint32_t j = a.tile_job[t];
    const BJob job = a.jobs[j];
    const BVol &v = a.vols[job.vol];
    const uint64_t nb = v.p.nblocks;
    const uint32_t dtype = v.p.dtype;
    const uint64_t base = (uint64_t)(t - job.tile_begin) * kBTile + (uint64_t)tid * kBItems;
    const uint2 *leaf = a.leaf + v.leaf_off;
    uint32_t f[kBItems];
    if (base + kBItems <= nb) {
        const uint4 *q = reinterpret_cast<const uint4 *>(leaf + base);
        const uint4 x = __ldcg(q), y = __ldcg(q + 1);
        f[0] = block_active(dtype, x.x, x.y, job.iso);
        f[1] = block_active(dtype, x.z, x.w, job.iso);
        f[2] = block_active(dtype, y.x, y.y, job.iso);
        f[3] = block_active(dtype, y.z, y.w, job.iso);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kBItems; ++i) {
            f[i] = 0;
            if (base + i < nb) {
                const uint2 w = leaf[base + i];
                f[i] = block_active(dtype, w.x, w.y, job.iso);
            }
        }
    }
    uint32_t total;
    const uint32_t excl = cta_exclusive_scan<kBThreads>(f[0] + f[1] + f[2] + f[3], s_tmp, &total);
    if (tid < 32) {
        uint32_t prefix = 0;
        bool ok = true;
        if (t == 0) {
            if (tid == 0) st_volatile(&a.filter_status[0], (2u << 30) | total);
        } else {
            if (tid == 0) st_volatile(&a.filter_status[t], (1u << 30) | total);
            ok = lookback_sum30(a.filter_status, t, prefix, &a.ctrl->status);
            if (ok && prefix + total >= (1u << 30)) {
                if (tid == 0) report(&a.ctrl->status, MTX_ERR_CAPACITY, kSiteBatched, 1, prefix);
                ok = false;
            }
            if (tid == 0) st_volatile(&a.filter_status[t], ok ? ((2u << 30) | (prefix + total)) : (3u << 30));
        }
        if (tid == 0) {
            s_u[0] = prefix;
            s_u[1] = ok;
        }
    }
    __syncthreads();
    if (!s_u[1]) return;
    const uint32_t prefix = s_u[0];
    uint32_t r = prefix + excl;
    uint32_t rk[kBItems];
#pragma unroll
    for (uint32_t i = 0; i < kBItems; ++i) {
        rk[i] = kNoVertex;
        if (f[i]) {
            if (r < a.block_cap) {
                a.ids[r] = (uint32_t)(base + i);
                a.job_of[r] = j;
            }
            rk[i] = r++;
        }
    }
    uint32_t *rank_map = a.rank_pool + job.rank_off;
    if (base + kBItems <= nb) {
        *reinterpret_cast<uint4 *>(rank_map + base) = make_uint4(rk[0], rk[1], rk[2], rk[3]);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kBItems; ++i)
            if (base + i < nb) rank_map[base + i] = rk[i];
    }
    if (tid == 0) {
        if (t == job.tile_begin) a.res[j].meshletOffset = prefix;
        if (t == job.tile_begin + job.ntiles - 1) a.job_end[j] = prefix + total;
        if (t == a.n_ftiles - 1) a.ctrl->total_active = prefix + total;
    }
}

// ------------------------------------------------------------ segmented scan
// Tile words as in the single-volume scan ([63:62] flag, [61:31] triangles,
// [30:0] vertices).  A tile holding a job's first block publishes its
// inclusive word (the sum after its last job start) at once; it looks back
// only if its first block continues the job of the tile before.
__device__ __forceinline__ bool lookback_seg(uint64_t *status, uint32_t t, bool has_head, uint64_t tail,
                                             bool need_carry, uint64_t &cv, uint64_t &ct, DevStatus *st) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tv = (uint32_t)tail, tt = tail >> 32;
    cv = ct = 0;
    bool ok = true;
    if (has_head) {
        ok = tv <= kCnt31 && tt <= kCnt31 && 3ull * tt <= 0xffffffffull;
        if (lane == 0) st_volatile(&status[t], ok ? ((2ull << 62) | (tt << 31) | tv) : (3ull << 62));
        if (!ok && lane == 0) report(st, MTX_ERR_CAPACITY, kSiteCountOverflow, (uint32_t)tv, (uint32_t)tt);
    } else if (lane == 0) {
        st_volatile(&status[t], (1ull << 62) | (tt << 31) | tv);
    }
    if (need_carry && ok) ok = lookback_sum31(status, t, cv, ct, st);
    if (!has_head) {
        const uint64_t iv = cv + tv, it = ct + tt;
        if (ok && (iv > kCnt31 || it > kCnt31 || 3ull * it > 0xffffffffull)) {
            if (lane == 0) report(st, MTX_ERR_CAPACITY, kSiteCountOverflow, (uint32_t)(iv >> 32), (uint32_t)it);
            ok = false;
        }
        if (lane == 0) st_volatile(&status[t], ok ? ((2ull << 62) | (it << 31) | iv) : (3ull << 62));
    }
    return ok;
}

// x (later) absorbs y (earlier) unless x already holds a job start.
__device__ __forceinline__ void seg_add(uint64_t &x, uint32_t &fx, uint64_t y, uint32_t fy) {
    if (!fx) x += y;
    fx |= fy;
}

__device__ __forceinline__ void batch_scan_tile(const BatchArgs &a, uint32_t t, uint32_t n, uint64_t *s_v,
                                                uint32_t *s_f, uint64_t *s_carry, uint32_t *s_u) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t base = t * kBTile + tid * kBItems;
    uint64_t val[kBItems];
    uint32_t jb[kBItems], head = 0;
    uint32_t prev = base > 0 && base - 1 < n ? __ldcg(a.job_of + base - 1) : kNoVertex;
#pragma unroll
    for (uint32_t i = 0; i < kBItems; ++i) {
        const uint32_t r = base + i;
        val[i] = 0;
        jb[i] = kNoVertex;
        if (r < n) {
            const uint2 c = __ldcg(reinterpret_cast<const uint2 *>(&a.desc[r].vertexCount));
            val[i] = ((uint64_t)c.y << 32) | c.x;
            jb[i] = __ldcg(a.job_of + r);
            if (r == 0 || jb[i] != prev) head |= 1u << i;
            prev = jb[i];
        }
    }
    // thread aggregate: the sum after the thread's last job start
    uint64_t x = 0;
#pragma unroll
    for (uint32_t i = 0; i < kBItems; ++i) x = ((head >> i) & 1u) ? val[i] : x + val[i];
    uint32_t fx = head != 0;
    // inclusive segmented scan of the warp, then of the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        const uint32_t fy = __shfl_up_sync(0xffffffffu, fx, o);
        if (lane >= (uint32_t)o) seg_add(x, fx, y, fy);
    }
    if (lane == 31) {
        s_v[warp] = x;
        s_f[warp] = fx;
    }
    __syncthreads();
    if (warp == 0) {
        uint64_t w = lane < kBWarps ? s_v[lane] : 0ull;
        uint32_t fw = lane < kBWarps ? s_f[lane] : 0u;
#pragma unroll
        for (int o = 1; o < (int)kBWarps; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, w, o);
            const uint32_t fy = __shfl_up_sync(0xffffffffu, fw, o);
            if (lane >= (uint32_t)o) seg_add(w, fw, y, fy);
        }
        if (lane < kBWarps) {
            s_v[lane] = w;
            s_f[lane] = fw;
        }
    }
    __syncthreads();
    // exclusive value of the thread within the tile
    uint64_t ex = __shfl_up_sync(0xffffffffu, x, 1);
    uint32_t fex = __shfl_up_sync(0xffffffffu, fx, 1);
    if (lane == 0) {
        ex = 0;
        fex = 0;
    }
    if (warp > 0) seg_add(ex, fex, s_v[warp - 1], s_f[warp - 1]);  // (warps before) then (lanes before)
    if (warp == 0) {
        const uint64_t tail = s_v[kBWarps - 1];
        const bool has_head = s_f[kBWarps - 1] != 0;
        const bool need_carry = __shfl_sync(0xffffffffu, head & 1u, 0) == 0u;
        uint64_t cv, ct;
        const bool ok = lookback_seg(a.scan_status, t, has_head, tail, need_carry, cv, ct, &a.ctrl->status);
        if (lane == 0) {
            s_carry[0] = (ct << 32) | cv;
            s_u[0] = ok;
        }
    }
    __syncthreads();
    if (!s_u[0]) return;
    uint64_t cur = fex ? ex : ex + s_carry[0];
#pragma unroll
    for (uint32_t i = 0; i < kBItems; ++i) {
        const uint32_t r = base + i;
        if (r >= n) break;
        if ((head >> i) & 1u) cur = 0;
        *reinterpret_cast<uint2 *>(&a.desc[r].vertexOffset) =
            make_uint2((uint32_t)cur, 3u * (uint32_t)(cur >> 32));
        cur += val[i];
        const uint32_t next = i + 1 < kBItems ? jb[i + 1] : (r + 1 < n ? __ldcg(a.job_of + r + 1) : kNoVertex);
        if (r + 1 == n || next != jb[i]) {  // the job's last block: its totals
            a.res[jb[i]].vertexCount = (uint32_t)cur;
            a.res[jb[i]].indexCount = 3u * (uint32_t)(cur >> 32);
        }
    }
}

// ------------------------------------------------------------ bases
__device__ __forceinline__ void batch_bases(const BatchArgs &a, uint32_t n, uint32_t total_active,
                                            uint64_t *s_tmp) {
    const uint32_t tid = threadIdx.x;
    uint64_t vb = 0, ib = 0;
    for (uint32_t j0 = 0; j0 < a.njobs; j0 += kBThreads) {
        const uint32_t j = j0 + tid;
        uint32_t vc = 0, ic = 0;
        if (j < a.njobs) {
            vc = __ldcg(&a.res[j].vertexCount);
            ic = __ldcg(&a.res[j].indexCount);
        }
        uint64_t tv, ti;
        const uint64_t ev = cta_exclusive_scan64<kBThreads>(vc, s_tmp, &tv);
        const uint64_t ei = cta_exclusive_scan64<kBThreads>(ic, s_tmp, &ti);
        if (j < a.njobs) {
            a.res[j].vertexOffset = vb + ev;
            a.res[j].indexOffset = ib + ei;
            a.res[j].meshletCount = __ldcg(a.job_end + j) - __ldcg(&a.res[j].meshletOffset);
        }
        vb += tv;
        ib += ti;
    }
    if (tid == 0) {
        BCtrl *c = a.ctrl;
        c->total_vertices = vb;
        c->total_triangles = ib / 3;
        const bool fits = n == total_active && vb <= a.vcap && ib / 3 <= a.tcap;
        if (!fits) report(&c->status, MTX_ERR_CAPACITY, kSiteBatched, 5, total_active);
        c->emit_ok = fits && !failed(&c->status);
        __threadfence();
        st_volatile(&c->bases_ready, 1u);
    }
}

// ------------------------------------------------------------ per block
// The list bodies of the single-volume passes (pmb_lists.cuh).  A block hands
// its inside rows over, not its list: batches of many volumes and isovalues tend
// to have dense blocks, and the emit phase lists the cells again in less time
// than the longer lists take through memory.  Only the inside rows are built
// per voxel type; vertices switch on it at their two loads, so that the kernel's
// code stays small.  Bound by instruction issue (2.2 a cycle and SM, 4600 a block
// of 122 vertices and 238 triangles) and the latency of L2-only loads: 46 jobs on
// 16 mixed volumes (39,800 blocks), 280 us of which 20 compaction, 100 counts,
// 12 offsets; float tiles staged in both phases, with a vertex table of 5 bytes a
// voxel, took 313.  Loading the next block's job and place under the current one
// was slower (315: registers).
template <int BC>
__device__ __forceinline__ void batch_count_block(const BatchArgs &a, const Problem &p, const WPlan &pl,
                                                  const GridDiv &dv, unsigned char *ws, const uint8_t *ntab,
                                                  uint32_t id, uint32_t r) {
    const Geo g = block_geo(id, p, false, 4, dv);
    if (p.dtype == MTX_DTYPE_U8) load_rows<uint8_t>(p, pl, ws, g, nullptr);
    else if (p.dtype == MTX_DTYPE_U16) load_rows<uint16_t>(p, pl, ws, g, nullptr);
    else load_rows<float>(p, pl, ws, g, nullptr);
    count_block_list<BC, true>(p, pl, ws, g, ntab, nullptr, a.desc + r, a.faces + (uint64_t)r * a.face_stride,
                               a.state + (uint64_t)r * a.state_stride);
}

template <bool GENERIC, int BC>
__device__ __forceinline__ void batch_emit_block(const BatchArgs &a, const Problem &p, const WPlan &pl,
                                                 const GridDiv &dv, unsigned char *ws, const uint64_t *tri,
                                                 const uint16_t *first, uint32_t edge8, uint32_t id, uint32_t r,
                                                 uint64_t rank_off, const mtx_batch_job_result &jr) {
    const uint32_t lane = threadIdx.x & 31;
    const Geo g = block_geo(id, p, false, 4, dv);
    const uint4 d = __ldcg(reinterpret_cast<const uint4 *>(a.desc + r));
    const uint32_t nb_rk = neighbour_rank<false>(p, g, id, a.rank_pool + rank_off);
    const uint32_t nb_vb = nb_rk != kNoVertex ? __ldcg(&a.desc[nb_rk].vertexOffset) : kNoVertex;
    const uint32_t miss = __ballot_sync(0xffffffffu, nb_rk == kNoVertex) & 0xfeu;
    const uint64_t face_words = a.block_cap * a.face_stride;
    Ctx8 c8;
    if (BC == 8) c8 = ctx8_load<false>(a.faces, nb_rk, edge8, face_words);
    uint32_t *rows = reinterpret_cast<uint32_t *>(ws + pl.off_rows);
    const uint32_t *own = a.state + (uint64_t)r * a.state_stride;
    for (uint32_t i = lane; i < pl.B1 * pl.B1; i += 32) rows[i] = __ldcg(own + i);
    __syncwarp();
    const uint32_t tbase = d.y / 3u, nv = d.z, nt = d.w;
    void *verts = a.vertices ? (void *)((char *)a.vertices + jr.vertexOffset * a.vsz) : nullptr;
    if ((uint64_t)tbase + nt > jr.indexCount / 3u || (verts && (uint64_t)d.x + nv > jr.vertexCount)) {
        if (lane == 0) report(&a.ctrl->status, MTX_ERR_CAPACITY, kSiteEmitCapacity, r, 2);
        return;
    }
    if (!(nt || (verts && nv))) return;
    const bool inner = g.ox + pl.B < p.X && g.oy + pl.B < p.Y && g.oz + pl.B < p.Z;
    list_bits<BC>(p, pl, ws, g);
    uint32_t *jobs = reinterpret_cast<uint32_t *>(ws + pl.off_jobs);
    uint32_t *nbase = reinterpret_cast<uint32_t *>(ws + pl.off_nvid);
    uint16_t *vtab = reinterpret_cast<uint16_t *>(ws + pl.off_vtab);
    const uint16_t *list = reinterpret_cast<const uint16_t *>(ws + pl.off_list);
    if (lane < 8) nbase[lane] = lane ? nb_vb : d.x;

    // vertices, and this block's entries of the vertex table
    ListWalk l;
    uint32_t vrun = 0, out = 0;
    while (vrun < nv) {
        const uint32_t n = list_take<BC>(l, pl, ws);
        if (!n) break;
        const uint32_t e = lane < n ? listed_cell(p, pl, g, rows, list[l.done + lane], inner) : 0u;
        l.done += n;
        uint32_t vt;
        const uint32_t rel = vrun + step_vertices(e >> 28, vt);
        queue_vertices(pl, e, rel, vtab, jobs, verts ? out : vrun);
        vrun += vt;
        __syncwarp();
        if (verts) {
            const uint32_t avail = min(vrun, nv);
            while (avail - out >= (vrun >= nv ? 1u : 32u)) {
                const uint32_t k = min(32u, avail - out);
                put_vertices<AnyVoxel, GENERIC>(p, pl, g, jobs, out, k, nv, inner, verts, d.x, a.vfmt, a.frame,
                                                a.normals);
                out += k;
            }
        }
    }
    // the context layer's entries
    if (BC == 8) {
        ctx8_store(c8, edge8, vtab);
    } else {
        for (uint32_t j0 = 0; j0 < pl.nb3; j0 += 32) {
            const uint32_t j = j0 + lane, c = ctx_entry(pl, min(j, pl.nb3 - 1));
            const uint32_t rk = __shfl_sync(0xffffffffu, nb_rk, c & 7u);
            const uint64_t at = (uint64_t)rk * a.face_stride + ((c >> 3) & 1023u);
            if (j < pl.nb3 && MTX_BC(c >> 13, pl.S1 * pl.S1 * pl.S1, kBcVoxTab))
                vtab[c >> 13] = rk != kNoVertex && MTX_BC(at, face_words, kBcFaces) ? __ldcg(a.faces + at) : (uint16_t)0;
        }
    }
    __syncwarp();

    // triangles
    bool bad = vrun != nv;
    uint32_t top = 0;
    out = 0;
    if (BC == 8) l.done = 0;  // the list is still there
    else l = ListWalk{};
    while (top < nt) {
        const uint32_t n = list_take<BC>(l, pl, ws);
        if (!n) break;
        const uint32_t e = lane < n ? listed_cell(p, pl, g, rows, list[l.done + lane], inner) : 0u;
        l.done += n;
        const uint32_t f = first[(e >> 12) & 0xffu];
        uint32_t total;
        const uint32_t before = warp_excl_scan(f >> 12, total);
        queue_triangles(pl, e, f, top + before, jobs, out);
        top += total;
        __syncwarp();
        const uint32_t avail = min(top, nt);
        const uint32_t least = top >= nt ? 1u : 32u;
        while (avail - out >= least) {
            const uint32_t k = min(32u, avail - out);
            put_triangles(pl, ws + pl.off_vtab, tri, jobs, nbase, out, k, nt, a.indices + jr.indexOffset + 3ull * tbase,
                          miss, bad);
            out += k;
        }
    }
    bad |= top != nt;
    if (bad) report(&a.ctrl->status, MTX_ERR_INTERNAL, kSiteEmitNeighbour, r, 3);
    __syncwarp();
}

// ------------------------------------------------------------ the kernel
// BC: every volume's block edge at compile time (0: each volume's own, at run
// time).  When all volumes of a batch have edge 8 the plan and every division
// by the edge fold to constants, and the kernel's code gets smaller.  Its
// register use is held to four CTAs per SM.
template <bool GENERIC, int BC>
__global__ void __launch_bounds__(kBThreads, BC ? 4 : 2) batch_extract_kernel(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t s_u[4];
    __shared__ uint32_t s_tmp[kBWarps + 1];
    __shared__ uint64_t s_tmp64[kBWarps + 1];
    __shared__ uint32_t s_f[kBWarps];
    __shared__ uint64_t s_carry[1];
    uint64_t *tri = reinterpret_cast<uint64_t *>(smem);
    uint16_t *first = reinterpret_cast<uint16_t *>(smem + 8 * kTris);
    uint8_t *ntab = smem + 8 * kTris + 512;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char *ws = smem + kBFixedBytes + min(warp, a.block_warps - 1) * a.ws_bytes;
    for (uint32_t i = tid; i < 256; i += kBThreads) ntab[i] = (uint8_t)(c_mc_cases[i] & 0xFu);
    build_tris(BC ? make_batch_plan(BC) : a.vols[0].pl, tri, first);  // one table row for all volumes (S1)
    const uint32_t edge8 = BC == 8 ? ctx8_edge(lane) : 0u;
    __syncthreads();
    BCtrl *ctrl = a.ctrl;
    DevStatus *st = &ctrl->status;

    // filter + ordered compaction
    for (;;) {
        if (tid == 0) s_u[2] = atomicAdd(&ctrl->filter_ticket, 1u);
        __syncthreads();
        const uint32_t t = s_u[2];
        __syncthreads();
        if (t >= a.n_ftiles) break;
        batch_filter_tile(a, t, s_tmp, s_u);
        cta_signal(&ctrl->filter_done, 1u);
    }
    if (!cta_wait_geq(&ctrl->filter_done, a.n_ftiles, st, 1, &s_u[3])) return;
    const uint32_t total_active = __ldcg(&ctrl->total_active);
    const uint32_t n = total_active <= a.block_cap ? total_active : 0u;

    // per-block counts
    uint32_t done = 0;
    for (;;) {
        if (warp >= a.block_warps) break;
        const uint32_t c0 = warp_ticket(&ctrl->count_ticket, kBChunk);
        if (c0 >= n) break;
        const uint32_t c1 = min(c0 + kBChunk, n);
        for (uint32_t r = c0; r < c1; ++r) {
            const uint32_t j = __ldcg(a.job_of + r), id = __ldcg(a.ids + r);
            const BJob &job = a.jobs[j];
            const BVol &v = a.vols[job.vol];
            Problem p = v.p;
            p.iso = job.iso;
            if (BC) p.B = BC;
            const WPlan pl = BC ? make_batch_plan(BC) : v.pl;
            batch_count_block<BC>(a, p, pl, v.dv, ws, ntab, id, r);
            ++done;
        }
    }
    __threadfence();
    __syncwarp();
    if (lane == 0 && done) atomicAdd(&ctrl->count_done, done);
    if (!cta_wait_geq(&ctrl->count_done, n, st, 2, &s_u[3])) return;

    // segmented offset scan
    const uint32_t nst = (n + kBTile - 1) / kBTile;
    for (;;) {
        if (tid == 0) s_u[2] = atomicAdd(&ctrl->scan_ticket, 1u);
        __syncthreads();
        const uint32_t t = s_u[2];
        __syncthreads();
        if (t >= nst) break;
        batch_scan_tile(a, t, n, s_tmp64, s_f, s_carry, s_u);
        cta_signal(&ctrl->scan_done, 1u);
    }

    // job bases: the CTA with the first ticket
    if (tid == 0) s_u[2] = atomicAdd(&ctrl->bases_ticket, 1u);
    __syncthreads();
    if (s_u[2] == 0) {
        if (cta_wait_geq(&ctrl->scan_done, nst, st, 3, &s_u[3])) batch_bases(a, n, total_active, s_tmp64);
    }
    if (!cta_wait_geq(&ctrl->bases_ready, 1u, st, 4, &s_u[3])) return;
    if (!__ldcg(&ctrl->emit_ok)) return;

    // vertices and triangles
    for (;;) {
        if (warp >= a.block_warps) break;
        const uint32_t c0 = warp_ticket(&ctrl->emit_ticket, kBChunk);
        if (c0 >= n) break;
        const uint32_t c1 = min(c0 + kBChunk, n);
        for (uint32_t r = c0; r < c1; ++r) {
            const uint32_t j = __ldcg(a.job_of + r), id = __ldcg(a.ids + r);
            const BJob &job = a.jobs[j];
            const BVol &v = a.vols[job.vol];
            Problem p = v.p;
            p.iso = job.iso;
            if (BC) p.B = BC;
            const WPlan pl = BC ? make_batch_plan(BC) : v.pl;
            mtx_batch_job_result jr;
            jr.vertexOffset = __ldcg(&a.res[j].vertexOffset);
            jr.indexOffset = __ldcg(&a.res[j].indexOffset);
            jr.vertexCount = __ldcg(&a.res[j].vertexCount);
            jr.indexCount = __ldcg(&a.res[j].indexCount);
            batch_emit_block<GENERIC, BC>(a, p, pl, v.dv, ws, tri, first, edge8, id, r, job.rank_off, jr);
        }
    }
}

MTX_BC_READER(bc_take_batched)

}  // namespace mtx

// ------------------------------------------------------------------ host
using namespace mtx;

struct mtx_batch {
    mtx_context *ctx = nullptr;
    uint32_t nvol = 0, njobs = 0, n_ftiles = 0;
    uint64_t mm_warps = 0;
    uint32_t grid = 0, smem = 0, vsz = 12;
    uint64_t block_cap = 0, vcap = 0, tcap = 0;
    int variant = 0;  // edge at run time (0-1), edge 8 at compile time (2-3); + 1: GENERIC
    std::vector<void *> allocs;
    BVol *vols = nullptr;
    uint2 *leaf = nullptr;
    void *ctrl_region = nullptr;
    size_t ctrl_bytes = 0;
    BatchArgs args{};
    bool use_graph = false;
    cudaStream_t capture_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {

using KernelFn = void (*)(BatchArgs);
KernelFn batch_kernel(int variant) {
    switch (variant) {
    case 0: return batch_extract_kernel<false, 0>;
    case 1: return batch_extract_kernel<true, 0>;
    case 2: return batch_extract_kernel<false, 8>;
    default: return batch_extract_kernel<true, 8>;
    }
}

// Block edge B in the warp layout of the batch's largest.
WPlan plan_in_layout(uint32_t B, const WPlan &L) {
    WPlan p = L;
    plan_block(p, B);
    p.S1 = L.S1;
    return p;
}

uint64_t align4(uint64_t x) { return (x + 3) & ~3ull; }
size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

mtx_status batch_alloc(mtx_batch *b, void **p, size_t bytes) {
    mtx_status s = dev_alloc(b->ctx, p, std::max<size_t>(bytes, 16));
    if (s == MTX_OK) b->allocs.push_back(*p);
    return s;
}

void batch_release(mtx_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->capture_stream) cudaStreamDestroy(b->capture_stream);
    for (void *p : b->allocs) dev_free(b->ctx, p);
    delete b;
}

mtx_status batch_enqueue(mtx_batch *b, cudaStream_t s) {
    mtx_context *c = b->ctx;
    MTX_CUDA(c, cudaMemsetAsync(b->ctrl_region, 0, b->ctrl_bytes, s));
    if (b->mm_warps) {
        const uint64_t blocks = (b->mm_warps + 3) / 4;
        batch_minmax_kernel<<<(unsigned)blocks, 128, 0, s>>>(b->vols, b->nvol, b->mm_warps, b->leaf);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(c, e, "batch min/max launch");
    }
    batch_kernel(b->variant)<<<b->grid, kBThreads, b->smem, s>>>(b->args);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "batch extract launch");
    return MTX_OK;
}

}  // namespace

extern "C" {

mtx_status mtx_batch_create(mtx_context_t c, const mtx_batch_desc *d, mtx_batch_t *out) {
    if (!c || !d || !out) return MTX_ERR_INVALID_ARG;
    *out = nullptr;
    DeviceGuard dg(c->device);
    join_extract(c);
    if (d->volumeCount == 0 || d->jobCount == 0 || !d->volumes || !d->blockEdges || !d->jobs)
        return fail(c, MTX_ERR_INVALID_ARG, "batch: empty volume or job list");
    if (d->vertexFormat > MTX_VERTEX_DATA || d->frame > MTX_FRAME_NDC)
        return fail(c, MTX_ERR_INVALID_ARG, "batch: bad vertex format or frame");
    mtx_status rs = load_list_tables(c);
    if (rs != MTX_OK) return rs;

    mtx_batch *b = new mtx_batch();
    b->ctx = c;
    b->nvol = d->volumeCount;
    b->njobs = d->jobCount;
    b->vsz = d->vertexFormat == MTX_VERTEX_DATA ? 32u : 12u;

    // volume table, warp layout, min/max warps
    uint32_t Bmax = 2;
    for (uint32_t v = 0; v < b->nvol; ++v) {
        rs = check_volume(c, &d->volumes[v]);
        if (rs != MTX_OK) { batch_release(b); return rs; }
        const uint32_t B = d->blockEdges[v];
        if (B < 2 || B > 16) { batch_release(b); return fail(c, MTX_ERR_INVALID_ARG, "batch: block edge outside 2..16"); }
        Bmax = std::max(Bmax, B);
    }
    const WPlan L = make_batch_plan(Bmax);
    std::vector<BVol> vols(b->nvol);
    // min/max warps: four waves of them, shared out by the volumes' sizes
    uint64_t leaf_total = 0, want = (uint64_t)c->sm_count * 48 * 4;
    double voxels = 0;
    for (uint32_t v = 0; v < b->nvol; ++v) voxels += (double)nvox(d->volumes[v].dims);
    for (uint32_t v = 0; v < b->nvol; ++v) {
        const mtx_volume &mv = d->volumes[v];
        const uint32_t B = d->blockEdges[v], esz = dtype_size(mv.dtype);
        BVol &bv = vols[v];
        memset(&bv, 0, sizeof(bv));
        Problem &p = bv.p;
        p.vol = mv.data.ptr;
        p.X = mv.dims[0];
        p.Y = mv.dims[1];
        p.Z = mv.dims[2];
        p.dtype = mv.dtype;
        p.B = B;
        p.GX = ceil_div(p.X, B);
        p.GY = ceil_div(p.Y, B);
        p.GZ = ceil_div(p.Z, B);
        p.nblocks = (uint64_t)p.GX * p.GY * p.GZ;
        bv.pl = plan_in_layout(B, L);
        bv.dv = grid_div(p);
        bv.leaf_off = leaf_total;
        leaf_total += align4(p.nblocks);
        bv.mm_begin = b->mm_warps;
        if (!rows_ok(p, esz)) {
            b->mm_warps += (p.nblocks + 31) / 32;
            continue;
        }
        const RowCut cut = row_cut(p, esz);
        bv.wide = cut.wide;
        bv.aligned = cut.aligned;
        bv.nan_zero = (uintptr_t)p.vol % 16 != 0 || ((uint64_t)p.X * esz) % 16 != 0 || (B != 4 && B != 8 && B != 16);
        bv.nXS = cut.nXS;
        bv.nbs = cut.nbs;
        const uint64_t cols = (uint64_t)bv.nXS * p.GY;
        const uint64_t share = std::max<uint64_t>(1, (uint64_t)((double)want * (double)nvox(mv.dims) / voxels));
        const uint32_t nzc = (uint32_t)std::min<uint64_t>(p.GZ, std::max<uint64_t>(1, (share + cols - 1) / cols));
        bv.zchunk = ceil_div(p.GZ, nzc);
        b->mm_warps += cols * ceil_div(p.GZ, bv.zchunk);
    }

    // job table and filter tiles
    std::vector<BJob> jobs(b->njobs);
    std::vector<uint32_t> tile_job;
    uint64_t rank_total = 0, blocks_total = 0;
    for (uint32_t j = 0; j < b->njobs; ++j) {
        const mtx_batch_job &bj = d->jobs[j];
        if (bj.volume >= b->nvol) { batch_release(b); return fail(c, MTX_ERR_INVALID_ARG, "batch: job names no volume"); }
        const uint64_t nb = vols[bj.volume].p.nblocks;
        jobs[j].vol = bj.volume;
        jobs[j].iso = bj.isovalue;
        jobs[j].tile_begin = (uint32_t)tile_job.size();
        jobs[j].ntiles = (uint32_t)((nb + kBTile - 1) / kBTile);
        jobs[j].rank_off = rank_total;
        rank_total += align4(nb);
        blocks_total += nb;
        tile_job.insert(tile_job.end(), jobs[j].ntiles, j);
    }
    if (blocks_total >= (1ull << 30)) { batch_release(b); return fail(c, MTX_ERR_UNSUPPORTED, "batch: 2^30 blocks or more"); }
    b->n_ftiles = (uint32_t)tile_job.size();
    b->block_cap = d->maxActiveBlocks ? std::min<uint64_t>(d->maxActiveBlocks, blocks_total) : blocks_total;
    b->vcap = d->vertexCapacity ? d->vertexCapacity : b->block_cap * 4ull * Bmax * Bmax;
    b->tcap = d->triangleCapacity ? d->triangleCapacity : b->block_cap * 8ull * Bmax * Bmax;
    const uint32_t face_stride = face_stride16(Bmax), state_stride = row_state_words(Bmax);
    const uint64_t n_stiles = (b->block_cap + kBTile - 1) / kBTile;

    // device memory
    void *p_vols, *p_jobs, *p_tiles, *p_leaf, *p_rank, *p_ids, *p_jobof, *p_desc, *p_faces, *p_state, *p_verts, *p_idx;
    b->ctrl_bytes = align256(sizeof(BCtrl));
    const size_t off_fst = b->ctrl_bytes;
    const size_t off_sst = align256(off_fst + 4ull * b->n_ftiles);
    const size_t off_res = align256(off_sst + 8ull * n_stiles);
    const size_t off_end = align256(off_res + sizeof(mtx_batch_job_result) * b->njobs);
    b->ctrl_bytes = align256(off_end + 4ull * b->njobs);
    if ((rs = batch_alloc(b, &p_vols, sizeof(BVol) * b->nvol)) != MTX_OK ||
        (rs = batch_alloc(b, &p_jobs, sizeof(BJob) * b->njobs)) != MTX_OK ||
        (rs = batch_alloc(b, &p_tiles, 4ull * b->n_ftiles)) != MTX_OK ||
        (rs = batch_alloc(b, &p_leaf, 8ull * leaf_total)) != MTX_OK ||
        (rs = batch_alloc(b, &p_rank, 4ull * rank_total)) != MTX_OK ||
        (rs = batch_alloc(b, &p_ids, 4ull * b->block_cap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_jobof, 4ull * b->block_cap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_desc, sizeof(mtx_meshlet_descriptor) * b->block_cap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_faces, 2ull * face_stride * b->block_cap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_state, 4ull * state_stride * b->block_cap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_verts, (size_t)b->vsz * b->vcap)) != MTX_OK ||
        (rs = batch_alloc(b, &p_idx, 12ull * b->tcap)) != MTX_OK ||
        (rs = batch_alloc(b, &b->ctrl_region, b->ctrl_bytes)) != MTX_OK) {
        batch_release(b);
        return rs;
    }
    b->vols = (BVol *)p_vols;
    b->leaf = (uint2 *)p_leaf;
    cudaError_t e = cudaMemcpy(p_vols, vols.data(), sizeof(BVol) * b->nvol, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p_jobs, jobs.data(), sizeof(BJob) * b->njobs, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p_tiles, tile_job.data(), 4ull * b->n_ftiles, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        batch_release(b);
        return cuda_fail(c, e, "batch tables");
    }

    BatchArgs &a = b->args;
    char *cr = (char *)b->ctrl_region;
    a.vols = (const BVol *)p_vols;
    a.jobs = (const BJob *)p_jobs;
    a.tile_job = (const uint32_t *)p_tiles;
    a.leaf = (const uint2 *)p_leaf;
    a.njobs = b->njobs;
    a.n_ftiles = b->n_ftiles;
    a.ws_bytes = L.bytes;
    a.face_stride = face_stride;
    a.state_stride = state_stride;
    a.rank_pool = (uint32_t *)p_rank;
    a.ids = (uint32_t *)p_ids;
    a.job_of = (uint32_t *)p_jobof;
    a.block_cap = b->block_cap;
    a.desc = (mtx_meshlet_descriptor *)p_desc;
    a.faces = (uint16_t *)p_faces;
    a.state = (uint32_t *)p_state;
    a.filter_status = (uint32_t *)(cr + off_fst);
    a.scan_status = (uint64_t *)(cr + off_sst);
    a.res = (mtx_batch_job_result *)(cr + off_res);
    a.job_end = (uint32_t *)(cr + off_end);
    a.vertices = p_verts;
    a.vcap = b->vcap;
    a.indices = (uint32_t *)p_idx;
    a.tcap = b->tcap;
    a.vfmt = d->vertexFormat;
    a.frame = d->frame;
    a.normals = d->vertexFormat == MTX_VERTEX_DATA ? d->normals : 0u;
    a.vsz = b->vsz;
    a.ctrl = (BCtrl *)b->ctrl_region;

    // persistent grid: every CTA that fits at once
    const bool generic = d->vertexFormat != MTX_VERTEX_XYZ || d->frame != MTX_FRAME_VOXEL;
    bool all8 = true;
    for (uint32_t v = 0; v < b->nvol; ++v) all8 = all8 && d->blockEdges[v] == 8;
    b->variant = (all8 ? 2 : 0) + (generic ? 1 : 0);
    // as many block warps per CTA as the shared memory holds (8 unless the
    // largest block edge is near 16)
    const int static_smem = 1024;
    const int room = (c->max_smem_optin > 0 ? c->max_smem_optin : 227 * 1024) - (int)kBFixedBytes - static_smem;
    a.block_warps = (uint32_t)std::min<int>(kBWarps, std::max(0, room / (int)L.bytes));
    if (d->blockWarps > kBWarps) {
        batch_release(b);
        return fail(c, MTX_ERR_INVALID_ARG, "batch: blockWarps outside 0..8");
    }
    if (d->blockWarps) a.block_warps = std::min<uint32_t>(a.block_warps, d->blockWarps);
    if (a.block_warps == 0) {
        batch_release(b);
        return fail(c, MTX_ERR_UNSUPPORTED, "batch: warp layout does not fit shared memory");
    }
    b->smem = kBFixedBytes + a.block_warps * L.bytes;
    KernelFn fn = batch_kernel(b->variant);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b->smem);
    // all of the unified L1 as shared memory: more resident warps hide the
    // block bodies' shared-memory latencies
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    int occ = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBThreads, b->smem);
    if (e != cudaSuccess) {
        batch_release(b);
        return cuda_fail(c, e, "batch kernel occupancy");
    }
    if (occ < 1) {
        batch_release(b);
        return fail(c, MTX_ERR_UNSUPPORTED, "batch: warp layout does not fit shared memory");
    }
    b->grid = (uint32_t)occ * (uint32_t)c->sm_count;
    b->use_graph = d->useGraph != 0;
    *out = b;
    return MTX_OK;
}

mtx_status mtx_batch_run(mtx_batch_t b) {
    if (!b) return MTX_ERR_INVALID_ARG;
    mtx_context *c = b->ctx;
    DeviceGuard dg(c->device);
    join_extract(c);
    if (!b->use_graph) return batch_enqueue(b, c->stream);
    if (!b->exec) {
        if (!b->capture_stream) MTX_CUDA(c, cudaStreamCreateWithFlags(&b->capture_stream, cudaStreamNonBlocking));
        MTX_CUDA(c, cudaStreamBeginCapture(b->capture_stream, cudaStreamCaptureModeThreadLocal));
        mtx_status rs = batch_enqueue(b, b->capture_stream);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(b->capture_stream, &g);
        if (rs != MTX_OK) {
            if (g) cudaGraphDestroy(g);
            return rs;
        }
        if (e != cudaSuccess) return cuda_fail(c, e, "batch graph capture");
        b->graph = g;
        MTX_CUDA(c, cudaGraphInstantiate(&b->exec, b->graph, 0));
    }
    MTX_CUDA(c, cudaGraphLaunch(b->exec, c->stream));
    return MTX_OK;
}

mtx_status mtx_batch_get_outputs(mtx_batch_t b, mtx_batch_outputs *o) {
    if (!b || !o) return MTX_ERR_INVALID_ARG;
    memset(o, 0, sizeof(*o));
    o->vertexBuffer = {b->args.vertices, (uint64_t)b->vsz * b->vcap};
    o->indexBuffer = {b->args.indices, 12ull * b->tcap};
    o->meshletDescriptorBuffer = {b->args.desc, sizeof(mtx_meshlet_descriptor) * b->block_cap};
    o->jobResultBuffer = {b->args.res, sizeof(mtx_batch_job_result) * b->njobs};
    o->vertexStride = b->vsz;
    return MTX_OK;
}

mtx_status mtx_batch_read_results(mtx_batch_t b, mtx_batch_job_result *results, mtx_batch_totals *totals) {
    if (!b) return MTX_ERR_INVALID_ARG;
    mtx_context *c = b->ctx;
    DeviceGuard dg(c->device);
    join_extract(c);
    MTX_CUDA(c, cudaStreamSynchronize(c->stream));
    if (results)
        MTX_CUDA(c, cudaMemcpy(results, b->args.res, sizeof(mtx_batch_job_result) * b->njobs, cudaMemcpyDeviceToHost));
    BCtrl h;
    MTX_CUDA(c, cudaMemcpy(&h, b->ctrl_region, sizeof(BCtrl), cudaMemcpyDeviceToHost));
    if (totals) {
        totals->status = (int32_t)h.status.code;
        totals->activeBlocks = h.total_active;
        totals->vertexCount = h.total_vertices;
        totals->triangleCount = h.total_triangles;
    }
    if (h.status.code != 0)
        return fail(c, (mtx_status)h.status.code,
                    "batch run: device error at site " + std::to_string(h.status.where) + " (" +
                        std::to_string(h.status.info0) + ", " + std::to_string(h.status.info1) + ")");
    return MTX_OK;
}

mtx_status mtx_batch_destroy(mtx_batch_t b) {
    if (!b) return MTX_ERR_INVALID_ARG;
    DeviceGuard dg(b->ctx->device);
    join_extract(b->ctx);
    batch_release(b);
    return MTX_OK;
}

}  // extern "C"
