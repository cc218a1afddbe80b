// Pinned staging ring and host copy threads (interface in fm_staging.h).
#include "fm_staging.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>

#include "fm_internal.h"

namespace fm {

// A few threads that split large host copies with the calling thread.
class CopyPool {
public:
    explicit CopyPool(int workers)
    {
        // as many as the system grants: the caller takes part in every round, alone if need be
        try {
            for (int i = 0; i < workers; ++i) threads_.emplace_back([this] { loop(); });
        } catch (const std::system_error&) {
        } catch (const std::bad_alloc&) {
        }
    }
    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> lk(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& t : threads_) t.join();
    }
    int size() const { return (int)threads_.size() + 1; }

    // Runs fn(0 .. tasks-1) on the workers and the caller; returns when every task is done
    // and no worker is still inside this call's task loop.
    void run(int tasks, const std::function<void(int)>& fn)
    {
        {
            std::lock_guard<std::mutex> lk(m_);
            fn_ = &fn;
            tasks_ = tasks;
            next_.store(0);
            done_ = 0;
            ++gen_;
        }
        cv_.notify_all();
        const int mine = work();
        std::unique_lock<std::mutex> lk(m_);
        done_ += mine;
        done_cv_.wait(lk, [&] { return done_ == tasks_ && active_ == 0; });
        fn_ = nullptr;
    }

private:
    // Takes tasks of the current round until none is left; returns how many it ran.
    int work()
    {
        int finished = 0;
        for (;;) {
            const int i = next_.fetch_add(1);
            if (i >= tasks_) break;
            (*fn_)(i);
            ++finished;
        }
        return finished;
    }
    void loop()
    {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(m_);
                cv_.wait(lk, [&] { return stop_ || (gen_ != seen && fn_); });
                if (stop_) return;
                seen = gen_;
                ++active_;   // the round cannot end (nor the next begin) while this is set
            }
            const int finished = work();
            std::lock_guard<std::mutex> lk(m_);
            done_ += finished;
            --active_;
            if (done_ == tasks_ && active_ == 0) done_cv_.notify_all();
        }
    }
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable cv_, done_cv_;
    const std::function<void(int)>* fn_ = nullptr;
    std::atomic<int> next_{0};
    int tasks_ = 0, done_ = 0, active_ = 0;
    uint64_t gen_ = 0;
    bool stop_ = false;
};

cudaError_t staging_ensure(fm_ctx* ctx)
{
    if (ctx->stage) return cudaSuccess;
    std::vector<cudaEvent_t> evs;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < kStageChunks && e == cudaSuccess; ++k) {
        cudaEvent_t ev = nullptr;
        e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e == cudaSuccess) evs.push_back(ev);
    }
    void* p = nullptr;
    if (e == cudaSuccess) e = cudaHostAlloc(&p, kStageChunk * kStageChunks, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        for (cudaEvent_t ev : evs) cudaEventDestroy(ev);
        return e;
    }
    ctx->stage = static_cast<char*>(p);
    ctx->stage_events = evs;
    if (!ctx->copy_pool) {
        const unsigned hw = std::thread::hardware_concurrency();
        const int workers = (int)std::min<unsigned>(hw > 1 ? hw - 1 : 0, 7);
        ctx->copy_pool = new (std::nothrow) CopyPool(workers);
    }
    return cudaSuccess;
}

void staging_release(fm_ctx* ctx)
{
    for (cudaEvent_t e : ctx->stage_events) {
        cudaEventSynchronize(e);
        cudaEventDestroy(e);
    }
    ctx->stage_events.clear();
    if (ctx->stage) cudaFreeHost(ctx->stage);
    ctx->stage = nullptr;
    delete ctx->copy_pool;
    ctx->copy_pool = nullptr;
}

void host_parallel(fm_ctx* ctx, int tasks, const std::function<void(int)>& fn)
{
    if (tasks <= 0) return;
    if (!ctx->copy_pool || ctx->copy_pool->size() == 1 || tasks == 1) {
        for (int i = 0; i < tasks; ++i) fn(i);
        return;
    }
    ctx->copy_pool->run(tasks, fn);
}

void copy_segments(fm_ctx* ctx, const std::vector<Segment>& segs)
{
    size_t total = 0;
    for (const Segment& g : segs) total += g.bytes;
    constexpr size_t kSlice = size_t(256) << 10;
    CopyPool* pool = ctx->copy_pool;
    const int tasks = pool ? (int)std::min<size_t>((total + kSlice - 1) / kSlice, (size_t)pool->size()) : 1;
    if (tasks <= 1) {
        for (const Segment& g : segs) std::memcpy(g.dst, g.src, g.bytes);
        return;
    }
    const size_t per = (total + tasks - 1) / tasks;
    pool->run(tasks, [&](int i) {
        // bytes [a, b) of the concatenated segments
        const size_t a = per * (size_t)i, b = std::min(total, a + per);
        size_t pos = 0;
        for (const Segment& g : segs) {
            const size_t lo = std::max(a, pos), hi = std::min(b, pos + g.bytes);
            if (lo < hi)
                std::memcpy(static_cast<char*>(g.dst) + (lo - pos), static_cast<const char*>(g.src) + (lo - pos), hi - lo);
            pos += g.bytes;
            if (pos >= b) break;
        }
    });
}

void Stager::flush()
{
    if (!host.empty()) {
        copy_segments(ctx, host);
        host.clear();
    }
    for (const Segment& g : device)
        if (err == cudaSuccess) err = cudaMemcpyAsync(g.dst, g.src, g.bytes, cudaMemcpyHostToDevice, s);
    device.clear();
}

// Closes the current chunk (its copies are issued) and waits until the next chunk's
// previous copies have finished with it.
void Stager::next_chunk()
{
    flush();
    if (chunk >= 0 && err == cudaSuccess) err = cudaEventRecord(ctx->stage_events[chunk], s);
    chunk = (chunk + 1) % kStageChunks;
    if (err == cudaSuccess) err = cudaEventSynchronize(ctx->stage_events[chunk]);
    used = 0;
}

void Stager::put(void* dst_dev, const void* src_host, size_t bytes, size_t pad_before)
{
    char* dst = static_cast<char*>(dst_dev);
    const char* src = static_cast<const char*>(src_host);
    if (pad_before && !device.empty() && used < kStageChunk) {
        Segment& last = device.back();
        char* end = static_cast<char*>(last.dst) + last.bytes;
        const size_t gap = (size_t)(dst - end);
        if (dst >= end && gap <= pad_before && static_cast<const char*>(last.src) + last.bytes ==
                                                   ctx->stage + (size_t)chunk * kStageChunk + used &&
            used + gap < kStageChunk) {
            used += gap;
            last.bytes += gap;
        }
    }
    while (bytes > 0 && err == cudaSuccess) {
        if (used == kStageChunk) next_chunk();
        if (err != cudaSuccess) return;
        const size_t k = std::min(bytes, kStageChunk - used);
        char* h = ctx->stage + (size_t)chunk * kStageChunk + used;
        host.push_back(Segment{h, src, k});
        Segment* last = device.empty() ? nullptr : &device.back();
        if (last && static_cast<char*>(last->dst) + last->bytes == dst &&
            static_cast<const char*>(last->src) + last->bytes == h)
            last->bytes += k;
        else
            device.push_back(Segment{dst, h, k});
        used += k;
        dst += k;
        src += k;
        bytes -= k;
    }
}

void Stager::close()
{
    flush();
    if (chunk >= 0 && err == cudaSuccess) err = cudaEventRecord(ctx->stage_events[chunk], s);
    used = kStageChunk;
}

namespace {

// dst[i] += src[i], split over the copy threads.
void add_doubles(fm_ctx* ctx, double* dst, const double* src, size_t n)
{
    constexpr size_t kSlice = size_t(1) << 15;
    const int tasks = (int)((n + kSlice - 1) / kSlice);
    host_parallel(ctx, tasks, [&](int i) {
        const size_t end = std::min(n, ((size_t)i + 1) * kSlice);
        for (size_t q = (size_t)i * kSlice; q < end; ++q) dst[q] += src[q];
    });
}

}  // namespace

namespace {

// Memory that only the host sees goes through the ring.  Page-locked memory the copy engine
// reaches by itself, and memory of a device the host must not touch: both are left to
// cudaMemcpyAsync.
bool is_pageable(const void* p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
}

// Whether some copies go through the ring: those that can, when they are kRingBytes in all and
// there is page-locked memory for the ring (plain copies need none).  Splits them from the rest.
template <class Copy, class Can>
bool split_copies(fm_ctx* ctx, const std::vector<Copy>& copies, std::vector<Copy>& ring, std::vector<Copy>& rest, Can&& can)
{
    size_t total = 0;
    for (const Copy& c : copies) total += c.bytes;
    if (total < kRingBytes) return false;
    total = 0;
    for (const Copy& c : copies) {
        const bool r = can(c);
        (r ? ring : rest).push_back(c);
        if (r) total += c.bytes;
    }
    if (total < kRingBytes) return false;
    if (staging_ensure(ctx) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

}  // namespace

cudaError_t copy_in(fm_ctx* ctx, cudaStream_t s, const std::vector<InCopy>& copies)
{
    std::vector<InCopy> ring, rest;
    const bool staged = split_copies(ctx, copies, ring, rest, [](const InCopy& c) { return is_pageable(c.src_host); });
    for (const InCopy& c : staged ? rest : copies) {
        const cudaError_t e = cudaMemcpyAsync(c.dst_dev, c.src_host, c.bytes, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
    }
    if (!staged) return cudaSuccess;
    Stager stager(ctx, s);
    for (const InCopy& c : ring) stager.put(c.dst_dev, c.src_host, c.bytes);
    stager.close();
    return stager.err;
}

cudaError_t copy_results(fm_ctx* ctx, cudaStream_t s, const std::vector<OutCopy>& copies)
{
    // sums are added by the host wherever they lie
    std::vector<OutCopy> ring, rest;
    const bool staged = split_copies(ctx, copies, ring, rest, [](const OutCopy& c) { return c.add || is_pageable(c.dst_host); });
    const std::vector<OutCopy>& plain = staged ? rest : copies;
    size_t added = 0;
    for (const OutCopy& c : plain)
        if (c.add) added += c.bytes / sizeof(double);
    std::vector<double> sums(added);
    size_t at = 0;
    for (const OutCopy& c : plain) {
        void* dst = c.dst_host;
        if (c.add) {
            dst = sums.data() + at;
            at += c.bytes / sizeof(double);
        }
        const cudaError_t e = cudaMemcpyAsync(dst, c.src_dev, c.bytes, cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) return e;
    }
    if (staged) return copy_out(ctx, s, ring);
    if (added == 0) return cudaSuccess;
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    at = 0;
    for (const OutCopy& c : plain) {
        if (!c.add) continue;
        double* dst = static_cast<double*>(c.dst_host);
        for (size_t q = 0; q < c.bytes / sizeof(double); ++q) dst[q] += sums[at + q];
        at += c.bytes / sizeof(double);
    }
    return cudaSuccess;
}

cudaError_t copy_out(fm_ctx* ctx, cudaStream_t s, const std::vector<OutCopy>& copies)
{
    cudaError_t e = staging_ensure(ctx);
    if (e != cudaSuccess) return e;
    // chunks of the ring, each a list of (host destination, offset in chunk, bytes)
    struct Part {
        char* dst;
        size_t off, bytes;
        bool add;
    };
    std::vector<std::vector<Part>> pending(kStageChunks);
    int slot = 0;
    size_t used = 0;
    auto drain = [&](int k) -> cudaError_t {
        cudaError_t r = cudaEventSynchronize(ctx->stage_events[k]);
        if (r != cudaSuccess) return r;
        const char* base = ctx->stage + (size_t)k * kStageChunk;
        std::vector<Segment> segs;
        for (const Part& p : pending[k])
            if (!p.add) segs.push_back(Segment{p.dst, base + p.off, p.bytes});
        copy_segments(ctx, segs);
        for (const Part& p : pending[k])
            if (p.add) add_doubles(ctx, reinterpret_cast<double*>(p.dst), reinterpret_cast<const double*>(base + p.off), p.bytes / sizeof(double));
        pending[k].clear();
        return cudaSuccess;
    };
    // closes the filling chunk and moves to the next, draining it first if it holds data
    auto advance = [&]() -> cudaError_t {
        cudaError_t r = cudaEventRecord(ctx->stage_events[slot], s);
        if (r != cudaSuccess) return r;
        slot = (slot + 1) % kStageChunks;
        used = 0;
        if (!pending[slot].empty()) return drain(slot);
        return cudaEventSynchronize(ctx->stage_events[slot]);   // an earlier host -> device use
    };
    if (e == cudaSuccess) e = cudaEventSynchronize(ctx->stage_events[0]);
    for (const OutCopy& c : copies) {
        char* dst = static_cast<char*>(c.dst_host);
        const char* src = static_cast<const char*>(c.src_dev);
        size_t bytes = c.bytes;
        used = std::min((used + 15) & ~size_t(15), kStageChunk);   // doubles are read in place
        while (bytes > 0 && e == cudaSuccess) {
            if (used == kStageChunk) {
                e = advance();
                if (e != cudaSuccess) break;
            }
            const size_t k = std::min(bytes, kStageChunk - used);
            e = cudaMemcpyAsync(ctx->stage + (size_t)slot * kStageChunk + used, src, k, cudaMemcpyDeviceToHost, s);
            pending[slot].push_back(Part{dst, used, k, c.add});
            used += k;
            dst += k;
            src += k;
            bytes -= k;
        }
    }
    if (e == cudaSuccess && used > 0) e = advance();
    for (int k = 0; k < kStageChunks && e == cudaSuccess; ++k) {
        const int j = (slot + k) % kStageChunks;
        if (!pending[j].empty()) e = drain(j);
    }
    return e;
}

}  // namespace fm
