// What launches of one context that overlapped leave behind: the compaction's
// ticket off the start of an epoch, the octree's and the emit pass's counters
// off zero.  The program writes such values into a context's control words
// between calls, with nothing in flight, and expects that the next call
// reports an error instead of a stale count, that the call after it is right
// again, and that a change of the context's stream makes the next call right.
// Prints "ok".  Waits are bounded by mtx_debug_set_waits.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "mtx_internal.h"

#define CHECK(x)                                                      \
    do {                                                              \
        if (!(x)) {                                                   \
            std::fprintf(stderr, "line %d: %s\n", __LINE__, #x);      \
            std::exit(1);                                             \
        }                                                             \
    } while (0)

int main() {
    const uint32_t dims[3] = {160, 160, 160};  // 40^3 blocks of edge 4: 16 compaction tiles, 2 octree CTAs and more
    std::vector<uint8_t> vox(160u * 160 * 160);
    uint32_t seed = 7;
    for (size_t i = 0; i < vox.size(); ++i) {
        const int x = (int)(i % 160) - 80, y = (int)(i / 160 % 160) - 80, z = (int)(i / 25600) - 80;
        seed = seed * 1664525u + 1013904223u;
        vox[i] = (uint8_t)((x * x + y * y + z * z < 3600 ? 170 : 80) + (seed >> 28));
    }
    cudaStream_t s1, s2;
    CHECK(cudaStreamCreate(&s1) == cudaSuccess && cudaStreamCreate(&s2) == cudaSuccess);
    mtx_context_t c;
    CHECK(mtx_context_create(0, s1, &c) == MTX_OK);
    mtx_volume v;
    CHECK(mtx_volume_upload(c, vox.data(), dims, MTX_DTYPE_U8, &v) == MTX_OK);
    mtx_push_constants pc;
    CHECK(mtx_push_constants_init(dims, 4, 128.0f, &pc) == MTX_OK);
    uint64_t blocks = 64000;

    // one filter call; its status and, where that is MTX_OK, its count
    mtx_minmax_output mm;
    CHECK(mtx_compute_min_max_mip(c, &v, &pc, nullptr, &mm) == MTX_OK);
    auto filter = [&](uint32_t *n) {
        mtx_filtering_output f;
        CHECK(mtx_filter_active_blocks(c, &mm, &pc, nullptr, &f) == MTX_OK);
        const mtx_status r = mtx_read_active_block_count(c, &f);
        *n = f.activeBlockCount;
        CHECK(mtx_filtering_free(c, &f) == MTX_OK);
        return r;
    };
    auto tear = [&](uint32_t ticket) {
        CHECK(cudaDeviceSynchronize() == cudaSuccess);
        uint64_t w;
        CHECK(cudaMemcpy(&w, &c->ctrl->filter_ticket, 8, cudaMemcpyDeviceToHost) == cudaSuccess);
        w = (w & ~0xffffffffull) | ticket;
        CHECK(cudaMemcpy(&c->ctrl->filter_ticket, &w, 8, cudaMemcpyHostToDevice) == cudaSuccess);
    };
    uint32_t n = 0, want = 0;
    CHECK(filter(&want) == MTX_OK && want > 1000 && want < blocks);
    for (uint32_t ticket : {1u, 5u, 15u, 100000u}) {
        CHECK(mtx_debug_set_waits(c, 4096, 0) == MTX_OK);
        tear(ticket);
        const mtx_status r = filter(&n);
        CHECK(r == MTX_ERR_TIMEOUT || r == MTX_ERR_INTERNAL);
        CHECK(mtx_debug_set_waits(c, 0, 0) == MTX_OK);
        CHECK(filter(&n) == MTX_OK && n == want);
        CHECK(filter(&n) == MTX_OK && n == want);
    }
    // a change of stream
    for (uint32_t ticket : {5u, 100000u}) {
        tear(ticket);
        const uint32_t done = 1;
        CHECK(cudaMemcpy(&c->ctrl->pyr_done, &done, 4, cudaMemcpyHostToDevice) == cudaSuccess);
        CHECK(mtx_context_set_stream(c, ticket == 5u ? s2 : s1) == MTX_OK);
        mtx_minmax_output again;
        CHECK(mtx_compute_min_max_mip(c, &v, &pc, nullptr, &again) == MTX_OK);
        CHECK(filter(&n) == MTX_OK && n == want);
        std::vector<uint32_t> a(mm.minMaxImage.size / 4), b(a.size());
        CHECK(again.minMaxImage.size == mm.minMaxImage.size);
        CHECK(cudaMemcpy(a.data(), mm.minMaxImage.ptr, 4 * a.size(), cudaMemcpyDeviceToHost) == cudaSuccess);
        CHECK(cudaMemcpy(b.data(), again.minMaxImage.ptr, 4 * b.size(), cudaMemcpyDeviceToHost) == cudaSuccess);
        CHECK(a == b);
        CHECK(mtx_minmax_free(c, &again) == MTX_OK);
    }
    // the whole-path call hands out its error word whatever the emit pass's counter holds
    mtx_mesh_buffers m{};
    uint32_t *counters;
    CHECK(cudaMalloc(&counters, 32) == cudaSuccess);
    m.counters = counters;
    m.maxActiveBlocks = want;
    for (uint32_t done : {0u, 3u, 1u << 20}) {
        CHECK(cudaDeviceSynchronize() == cudaSuccess);
        CHECK(cudaMemset(counters, 0xff, 32) == cudaSuccess);
        CHECK(cudaMemcpy(&c->ctrl->emit_done, &done, 4, cudaMemcpyHostToDevice) == cudaSuccess);
        CHECK(mtx_extract_plain_async(c, &v, &pc, nullptr, &m) == MTX_OK);
        CHECK(mtx_synchronize(c) == MTX_ERR_CAPACITY);  // no vertex and triangle buffers
        uint32_t got[5];
        CHECK(cudaMemcpy(got, counters, 20, cudaMemcpyDeviceToHost) == cudaSuccess);
        CHECK(got[3] == want && got[4] == MTX_ERR_CAPACITY);
    }
    // a tile withheld where there is only one: the count is zero, not what the buffer held
    const uint32_t small[3] = {40, 40, 40};
    mtx_volume w;
    CHECK(mtx_volume_upload(c, vox.data(), small, MTX_DTYPE_U8, &w) == MTX_OK);
    CHECK(mtx_push_constants_init(small, 4, 128.0f, &pc) == MTX_OK);
    mtx_minmax_free(c, &mm);
    CHECK(mtx_compute_min_max_mip(c, &w, &pc, nullptr, &mm) == MTX_OK);
    CHECK(mtx_debug_set_waits(c, 4096, 1) == MTX_OK);
    CHECK(filter(&n) == MTX_OK && n == 0);
    CHECK(mtx_debug_set_waits(c, 0, 0) == MTX_OK);
    mtx_minmax_free(c, &mm);
    mtx_volume_free(c, &w);
    mtx_volume_free(c, &v);
    cudaFree(counters);
    CHECK(mtx_context_destroy(c) == MTX_OK);
    std::puts("ok");
    return 0;
}
