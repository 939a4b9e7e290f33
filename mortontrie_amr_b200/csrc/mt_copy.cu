// Device results into the caller's host memory.
//
// The caller's arrays are ordinary (pageable) memory, often freshly allocated:
// a plain device-to-host copy into them runs at 3-8 GB/s, one thread copying
// out of the driver's staging buffer and taking every page fault.  Here the
// copy engine fills a ring of page-locked chunks and a few host threads empty
// it, so that the transfer, the faults and the copies overlap.
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>

#include "mt_internal.hpp"

namespace mt {

namespace {

struct Job;

}  // namespace

// page-locked ring and copying threads of one context, made at its first large
// copy, given back with it
struct HostStage {
    static constexpr size_t kChunk = 1u << 19;
    static constexpr int kSlots = 16;  // 8 MiB, page-locked in about 2 ms
    char *buf = nullptr;
    cudaEvent_t ev[kSlots] = {};
    std::mutex busy;  // one copy at a time; another thread's takes the plain path
    std::vector<std::thread> threads;
    std::mutex m;
    std::condition_variable cv;
    Job *job = nullptr;     // what the threads work on
    uint64_t turn = 0;      // counts jobs
    int working = 0;        // threads that have not finished the current one
    bool stop = false;
};

namespace {

// Arrays of this size are fresh mappings (the C library maps every allocation
// of 32 MiB and more, and reuses the pages of smaller ones): every page of the
// copy is a fault.  262 MB of a 4-level sphere's fields, 16 cores: 67 ms by
// plain copies, 52 with 2 threads, 46 with 4, 36 with 8.  Smaller arrays have
// their pages already, and a caller's own threads that still spin keep the
// copying threads from their cores: 34 MB of fields 5.9-7.5 ms plain, 7-27 ms
// by threads.
constexpr size_t kStagedFrom = 32u << 20;

// chunk c of the copy: filled by the stream, emptied by one thread
struct Job {
    HostStage *st;
    char *dst;
    size_t bytes;
    int64_t chunks;
    std::mutex m;
    std::condition_variable cv;
    int64_t filled = 0;               // chunks whose transfer is enqueued
    int64_t next = 0;                 // next chunk a thread takes
    int64_t emptied[HostStage::kSlots] = {};  // how often each slot has been emptied
    cudaError_t err = cudaSuccess;

    void work()
    {
        for (;;) {
            int64_t c;
            {
                std::unique_lock<std::mutex> lk(m);
                cv.wait(lk, [&] { return err != cudaSuccess || next < filled || next >= chunks; });
                if (err != cudaSuccess || next >= chunks) return;
                c = next++;
                if (next >= chunks) cv.notify_all();
            }
            const int s = (int)(c % HostStage::kSlots);
            const cudaError_t e = cudaEventSynchronize(st->ev[s]);
            const size_t at = (size_t)c * HostStage::kChunk;
            if (e == cudaSuccess)
                std::memcpy(dst + at, st->buf + s * HostStage::kChunk, std::min(HostStage::kChunk, bytes - at));
            std::lock_guard<std::mutex> lk(m);
            if (e != cudaSuccess && err == cudaSuccess) err = e;
            ++emptied[s];
            cv.notify_all();
        }
    }
};

void stage_thread(HostStage *st, int device)
{
    cudaSetDevice(device);
    uint64_t seen = 0;
    for (;;) {
        Job *job;
        {
            std::unique_lock<std::mutex> lk(st->m);
            st->cv.wait(lk, [&] { return st->stop || st->turn != seen; });
            if (st->stop) return;
            seen = st->turn;
            job = st->job;
        }
        job->work();
        std::lock_guard<std::mutex> lk(st->m);
        if (--st->working == 0) st->cv.notify_all();
    }
}

bool stage_init(HostStage &st, int device, int nthreads)
{
    if (!st.buf) {
        if (cudaMallocHost(&st.buf, HostStage::kChunk * HostStage::kSlots) != cudaSuccess) {
            cudaGetLastError();
            st.buf = nullptr;
            return false;
        }
        for (cudaEvent_t &e : st.ev)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
        try {
            for (int t = 0; t < nthreads; ++t) st.threads.emplace_back(stage_thread, &st, device);
        } catch (...) {
            // the threads there are do the work
        }
    }
    return !st.threads.empty();
}

void stage_free(HostStage &st)
{
    {
        std::lock_guard<std::mutex> lk(st.m);
        st.stop = true;
    }
    st.cv.notify_all();
    for (std::thread &t : st.threads) t.join();
    st.threads.clear();
    for (cudaEvent_t &e : st.ev) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    if (st.buf) cudaFreeHost(st.buf);
    st.buf = nullptr;
}

cudaError_t staged(Ctx &ctx, HostStage &st, char *dst, const char *src, size_t bytes)
{
    Job job;
    job.st = &st;
    job.dst = dst;
    job.bytes = bytes;
    job.chunks = (int64_t)((bytes + HostStage::kChunk - 1) / HostStage::kChunk);
    {
        std::lock_guard<std::mutex> lk(st.m);
        st.job = &job;
        ++st.turn;
        st.working = (int)st.threads.size();
    }
    st.cv.notify_all();
    for (int64_t c = 0; c < job.chunks; ++c) {
        const int s = (int)(c % HostStage::kSlots);
        {
            std::unique_lock<std::mutex> lk(job.m);
            job.cv.wait(lk, [&] { return job.err != cudaSuccess || job.emptied[s] == c / HostStage::kSlots; });
            if (job.err != cudaSuccess) break;
        }
        const size_t at = (size_t)c * HostStage::kChunk;
        cudaError_t e = cudaMemcpyAsync(st.buf + s * HostStage::kChunk, src + at, std::min(HostStage::kChunk, bytes - at),
                                        cudaMemcpyDeviceToHost, ctx.stream);
        if (e == cudaSuccess) e = cudaEventRecord(st.ev[s], ctx.stream);
        std::lock_guard<std::mutex> lk(job.m);
        if (e != cudaSuccess) {
            if (job.err == cudaSuccess) job.err = e;
        } else {
            job.filled = c + 1;
        }
        job.cv.notify_all();
        if (e != cudaSuccess) break;
    }
    {
        std::unique_lock<std::mutex> lk(st.m);
        st.cv.wait(lk, [&] { return st.working == 0; });
    }
    // the transfers into the ring are over before it is used again
    const cudaError_t e = cudaStreamSynchronize(ctx.stream);
    return job.err != cudaSuccess ? job.err : e;
}

}  // namespace

// `bytes` of device memory, after the stream's work, into host memory; the
// copy has landed once the stream is synchronised (one wait for a call's
// several copies: two cost a small cube's page-locked read-back 10 us)
int copy_out(Ctx &ctx, void *host, const void *dev, size_t bytes)
{
    if (!bytes) return MT_OK;
    auto pageable = [&] {
        cudaPointerAttributes attr{};
        if (cudaPointerGetAttributes(&attr, host) == cudaSuccess) return attr.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();
        return true;
    };
    const int nthreads = (int)std::min<unsigned>(8, std::thread::hardware_concurrency() / 2);
    if (bytes >= kStagedFrom && nthreads >= 2 && pageable()) {
        HostStage *st = nullptr;
        {
            std::lock_guard<std::mutex> lk(ctx.stage_mutex);
            if (!ctx.stage) ctx.stage = new (std::nothrow) HostStage;
            st = ctx.stage;
        }
        if (st && st->busy.try_lock()) {
            std::lock_guard<std::mutex> lk(st->busy, std::adopt_lock);
            if (stage_init(*st, ctx.device, nthreads)) {
                MT_CUDA(ctx, staged(ctx, *st, (char *)host, (const char *)dev, bytes));
                return MT_OK;
            }
        }
    }
    MT_CUDA(ctx, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx.stream));
    return MT_OK;
}

void copy_free(Ctx &ctx)
{
    if (!ctx.stage) return;
    stage_free(*ctx.stage);
    delete ctx.stage;
    ctx.stage = nullptr;
}

}  // namespace mt
