// Copies from device memory to pageable host arrays.
//
// Such a copy runs at the pace of one host thread that also takes the page
// faults of a fresh array (about 4 GB/s measured); the link does ten times
// that.  Two remedies by size:
//   * from 4 MiB, a few threads touch the arrays' pages first, while the GPU is
//     still at work on the results;
//   * from 32 MiB, the stream also copies chunk by chunk into a small pinned
//     ring of the context and the threads move the chunks on (96 MB of fields:
//     23 -> 9 ms).  The ring is made on first use, which takes about 5 ms:
//     smaller copies would not earn it back.
// Host memory that is pinned already goes straight to cudaMemcpyAsync.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <new>
#include <thread>
#include <vector>

#include "../../include/ouc.h"
#include "ctx.h"

namespace ouc {

struct HostRing {
    static constexpr size_t kChunk = 1 << 20;
    static constexpr int kSlots = 8;
    char* mem = nullptr;
    cudaEvent_t ev[kSlots] = {};
};

namespace host {

namespace {

constexpr size_t kTouch = 4 << 20;    // totals from which the pages are touched by a team
constexpr size_t kRing = 32 << 20;    // totals from which the copies go through the pinned ring
constexpr int kThreadsMax = 6;

HostRing* ring_of(ouc_ctx* ctx) {
    if (ctx->io) return ctx->io;
    HostRing* r = new (std::nothrow) HostRing();
    if (!r) return nullptr;
    bool ok = cudaMallocHost(&r->mem, HostRing::kChunk * HostRing::kSlots) == cudaSuccess;
    for (auto& e : r->ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ctx->io = r;
    if (!ok) {
        cudaGetLastError();
        free_ring(ctx);
    }
    return ctx->io;
}

bool pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

int copy_direct(ouc_ctx* ctx, const std::vector<HostCopy>& c, bool to_host, cudaStream_t st) {
    for (const auto& x : c) {
        const cudaError_t e = cudaMemcpyAsync(to_host ? x.host : x.dev, to_host ? x.dev : x.host, x.bytes,
                                              to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "host copy");
    }
    return OUC_OK;
}

int team_size() {
    const int hw = (int)std::thread::hardware_concurrency();
    return hw > 2 * kThreadsMax ? kThreadsMax : hw > 3 ? hw / 2 : 1;
}

}  // namespace

void free_ring(ouc_ctx* ctx) {
    if (!ctx->io) return;
    for (auto& e : ctx->io->ev)
        if (e) cudaEventDestroy(e);
    cudaFreeHost(ctx->io->mem);
    delete ctx->io;
    ctx->io = nullptr;
}

// Pinned arrays have their pages; only the others are touched.
bool touch_pages(std::vector<HostCopy> arrays) {
    arrays.erase(std::remove_if(arrays.begin(), arrays.end(),
                                [](const HostCopy& x) { return !x.host || x.bytes == 0 || pinned(x.host); }),
                 arrays.end());
    constexpr size_t kPage = 4096, kBlock = 256 * kPage;
    size_t total = 0;
    for (const auto& x : arrays) total += x.bytes;
    if (total < kTouch) return false;
    std::vector<HostCopy> blocks;
    for (const auto& x : arrays)
        for (size_t o = 0; o < x.bytes; o += kBlock)
            blocks.push_back({static_cast<char*>(x.host) + o, nullptr, x.bytes - o < kBlock ? x.bytes - o : kBlock});
    std::atomic<size_t> next{0};
    auto worker = [&]() {
        for (size_t k; (k = next.fetch_add(1)) < blocks.size();)
            for (size_t o = 0; o < blocks[k].bytes; o += kPage) {   // each byte written back as it is
                volatile char* q = static_cast<char*>(blocks[k].host) + o;
                *q = *q;
            }
    };
    run_team(team_size(), worker, [] {});   // without threads the copy takes the faults itself
    return true;
}

int copy_host(ouc_ctx* ctx, const std::vector<HostCopy>& copies, bool to_host, cudaStream_t st, bool touched) {
    if (!st) st = ctx->stream;
    if (!to_host) return copy_direct(ctx, copies, false, st);
    size_t total = 0;
    bool direct = false;
    for (const auto& x : copies) {
        total += x.bytes;
        direct = direct || pinned(x.host);
    }
    if (direct || total < kTouch) return copy_direct(ctx, copies, true, st);
    if (!touched) touch_pages(copies);
    HostRing* ring = total >= kRing && !overlapping(copies) ? ring_of(ctx) : nullptr;
    if (!ring) return copy_direct(ctx, copies, true, st);
    const cudaError_t ready = cudaStreamSynchronize(st);   // one thread waits for the work ahead, not the whole team
    if (ready != cudaSuccess) return cuda_fail(ctx, ready, "host copy");
    const int e = ring_copy(
        copies, ring->mem, HostRing::kChunk, HostRing::kSlots, team_size(),
        [&](int s, void* dev, size_t bytes) -> int {
            const cudaError_t q = cudaMemcpyAsync(ring->mem + (size_t)s * HostRing::kChunk, dev, bytes, cudaMemcpyDeviceToHost, st);
            return q != cudaSuccess ? q : cudaEventRecord(ring->ev[s], st);
        },
        [&](int s) -> int {
            cudaSetDevice(ctx->device);   // of the calling thread
            return cudaEventSynchronize(ring->ev[s]);
        });
    if (e < 0) return copy_direct(ctx, copies, true, st);   // no threads to be had
    return e ? cuda_fail(ctx, (cudaError_t)e, "host copy") : OUC_OK;
}

int records_in(ouc_ctx* ctx, const std::vector<Record>& recs, bool host, cudaStream_t st) {
    if (!st) st = ctx->stream;
    const bool xt = ctx->cfg.gather_layout == OUC_GATHER_XT;
    std::vector<HostCopy> batch;
    size_t first = 0, used = 0;   // records recs[first ..] are in the batch, `used` floats of the staging buffer
    auto flush = [&](size_t end) -> int {
        if (int rc = copy_host(ctx, batch, false, st)) return rc;
        size_t o = 0;
        for (size_t k = first; xt && k < end; ++k) {   // [X][nt] -> [nt][X]
            launch_transpose(ctx->staging + o, recs[k].dst_tx, recs[k].X, ctx->nt, st);
            ctx->timing.kernel_launches += 1;
            o += (size_t)ctx->nt * recs[k].X;
        }
        batch.clear();
        first = end;
        used = 0;
        return OUC_OK;
    };
    for (size_t k = 0; k < recs.size(); ++k) {
        const Record& r = recs[k];
        const size_t n = (size_t)ctx->nt * r.X;
        if (!host) {
            if (xt) {
                launch_transpose(r.src, r.dst_tx, r.X, ctx->nt, st);
                ctx->timing.kernel_launches += 1;
            } else {
                const cudaError_t e = cudaMemcpyAsync(r.dst_tx, r.src, n * 4, cudaMemcpyDeviceToDevice, st);
                if (e != cudaSuccess) return cuda_fail(ctx, e, "record copy");
            }
            continue;
        }
        if (xt && used + n > ctx->staging_n)
            if (int rc = flush(k)) return rc;
        batch.push_back({const_cast<float*>(r.src), xt ? ctx->staging + used : r.dst_tx, n * 4});
        used += n;
    }
    if (host)
        if (int rc = flush(recs.size())) return rc;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? OUC_OK : cuda_fail(ctx, e, "record transposes");
}

int records_fence(ouc_ctx* ctx) {
    cudaError_t e = cudaEventRecord(ctx->evb[1], ctx->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream2, ctx->evb[1], 0);
    return e == cudaSuccess ? OUC_OK : cuda_fail(ctx, e, "record copy");
}

int records_beside(ouc_ctx* ctx, const std::vector<Record>& recs, bool host) {
    if (recs.empty()) return OUC_OK;
    int rc = records_in(ctx, recs, host, ctx->stream2);
    cudaError_t e = cudaEventRecord(ctx->evb[0], ctx->stream2);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, ctx->evb[0], 0);
    return rc ? rc : e == cudaSuccess ? OUC_OK : cuda_fail(ctx, e, "record copy");
}

}  // namespace host
}  // namespace ouc
