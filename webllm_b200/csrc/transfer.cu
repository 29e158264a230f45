// Host <-> device copies of pageable memory, for everything that a caller hands over or takes back (uploads, registrations,
// logits, dense weights).
//
// A cudaMemcpy of pageable memory goes through the driver's own staging buffer and one thread: 20 GB/s, where the link does 55 and
// one core's copy 18. Copies of 2 MB and more (to the device 8 MB: 2.2 MB up took 157 us either way) pass through a ring of pinned slots instead: while the calling thread keeps the
// transfers going, three helper threads (six measured no better) copy the pieces between the slots and the caller's memory.
// 512 KB pieces: smaller ones lose to the gap between two transfers, larger ones to the first and the last piece. Measured on 16
// cores: 17.4 MB to the host 850 -> 490 us, 64 MB either way 2.8 -> 1.8 ms.
//
// The ring (8 MB) and the helpers belong to the process, are made on first use, serve one copy at a time (a second thread that
// finds them busy copies the plain way) and are given back when the last context goes (a process that ends before that takes them with it).
#include <string.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>

#include "common.cuh"

namespace wb {
namespace {

constexpr size_t kPiece = 512 << 10, kHelpersFrom = 2 << 20, kHelpersUpFrom = 8 << 20;
constexpr int kSlots = 16, kHelpersMax = 3, kSpins = 20000;  // spins: about a millisecond

struct Job {
    char *host;
    size_t bytes;
    int pieces;
    bool to_host;
    std::atomic<int> next{0}, open{0};  // next piece to copy; pieces below `open` may be copied (arrived, or their slot is free)
    std::atomic<unsigned char> *done;   // per piece: copied
};

class Ring {
public:
    std::mutex use;  // held for the length of one copy
    char *pinned = nullptr;
    cudaEvent_t event[kSlots] = {};
    int device = -1;

    bool prepare(int dev)  // false: there is no such memory to be had now; the copy goes the plain way
    {
        if (pinned && device == dev) return true;
        release();
        cudaError_t err = cudaHostAlloc((void **)&pinned, kSlots * kPiece, cudaHostAllocPortable);
        if (err != cudaSuccess) pinned = nullptr;
        for (cudaEvent_t &e : event)
            if (err == cudaSuccess && (err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming)) != cudaSuccess) e = nullptr;
        if (err != cudaSuccess) {
            cudaGetLastError();
            release();
            return false;
        }
        device = dev;
        return true;
    }
    void release()
    {
        for (cudaEvent_t &e : event) {
            if (e) cudaEventSynchronize(e), cudaEventDestroy(e);
            e = nullptr;
        }
        if (pinned) cudaFreeHost(pinned);
        pinned = nullptr, device = -1;
    }
    // helper threads
    int start(Job *j)
    {
        if (!helpers) {
            const int n = std::min<int>(kHelpersMax, (int)std::thread::hardware_concurrency() / 2 - 1);
            try {
                for (int i = 0; i < n; i++) threads[i] = std::thread([this] { work(); }), helpers++;
            } catch (const std::system_error &) {  // no more threads for this process: those that there are do
            }
        }
        if (!helpers) return 0;
        {
            std::lock_guard<std::mutex> lk(m);  // (a helper between its last look and its sleep sees the new job)
            job.store(j, std::memory_order_release);
        }
        if (asleep.load(std::memory_order_acquire)) cv.notify_all();
        return helpers;
    }
    void finish(Job *j)
    {
        job.store(nullptr, std::memory_order_seq_cst);
        while (entered.load(std::memory_order_seq_cst)) pause();  // nobody is left that could still look at *j
    }
    void stop()
    {
        {
            std::lock_guard<std::mutex> lk(m);
            quit.store(true);
        }
        cv.notify_all();
        for (int i = 0; i < helpers; i++) threads[i].join();
        helpers = 0, quit.store(false);
    }
    static void pause() { __builtin_ia32_pause(); }
    static void copy_piece(Job *j, char *pinned, int i)
    {
        char *slot = pinned + (size_t)(i % kSlots) * kPiece, *host = j->host + (size_t)i * kPiece;
        const size_t n = std::min(kPiece, j->bytes - (size_t)i * kPiece);
        if (j->to_host) memcpy(host, slot, n);
        else memcpy(slot, host, n);
        j->done[i].store(1, std::memory_order_release);
    }

private:
    std::mutex m;
    std::condition_variable cv;
    std::thread threads[kHelpersMax];
    int helpers = 0;
    std::atomic<Job *> job{nullptr};
    std::atomic<int> entered{0}, asleep{0};
    std::atomic<bool> quit{false};

    void work()
    {
        int idle = 0;
        while (!quit.load(std::memory_order_relaxed)) {
            entered.fetch_add(1, std::memory_order_seq_cst);
            Job *j = job.load(std::memory_order_seq_cst);
            if (j)
                for (int i; (i = j->next.fetch_add(1, std::memory_order_relaxed)) < j->pieces; idle = 0) {
                    while (j->open.load(std::memory_order_acquire) <= i) pause();
                    copy_piece(j, pinned, i);
                }
            entered.fetch_sub(1, std::memory_order_seq_cst);
            // a wake-up takes as long as several pieces: helpers stay awake for a moment (copies come in groups), then sleep
            if (++idle < kSpins) {
                pause();
                continue;
            }
            std::unique_lock<std::mutex> lk(m);
            asleep.fetch_add(1);
            cv.wait(lk, [&] { return quit.load() || job.load() != nullptr; });
            asleep.fetch_sub(1);
            idle = 0;
        }
    }
};

Ring &g_ring = *new Ring;  // never destroyed: a process may end with a context open, and a running std::thread must not be destroyed
std::mutex g_users_lock;
int g_users = 0;

// The calling thread alone talks to CUDA: it starts the transfers and tells the helpers which
// pieces they may copy. Whatever fails, every piece is opened before it leaves, so that no helper waits for good.
int run_job(wb_context *ctx, Job *j, char *dev)
{
    int issued = 0, settled = 0;  // transfers started / known to be complete
    cudaError_t err = cudaSuccess;
    auto transfer = [&](int i) {
        char *slot = g_ring.pinned + (size_t)(i % kSlots) * kPiece, *d = dev + (size_t)i * kPiece;
        const size_t n = std::min(kPiece, j->bytes - (size_t)i * kPiece);
        cudaError_t e = cudaMemcpyAsync(j->to_host ? slot : d, j->to_host ? d : slot, n, j->to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(g_ring.event[i % kSlots], ctx->stream);
        if (err == cudaSuccess) err = e;
        issued++;
    };
    auto copied = [&](int i) { return j->done[i].load(std::memory_order_acquire) != 0; };
    if (j->to_host) {
        while (settled < j->pieces && err == cudaSuccess) {
            while (issued < j->pieces && (issued < kSlots || copied(issued - kSlots)) && err == cudaSuccess) transfer(issued);
            if (issued == settled) continue;  // every slot still waits for its helper
            const cudaError_t e = cudaEventSynchronize(g_ring.event[settled % kSlots]);
            if (err == cudaSuccess) err = e;
            j->open.store(++settled, std::memory_order_release);
        }
    } else {
        j->open.store(std::min(kSlots, j->pieces), std::memory_order_release);
        while (issued < j->pieces && err == cudaSuccess) {
            if (copied(issued)) {
                transfer(issued);
            } else if (settled < issued && cudaEventQuery(g_ring.event[settled % kSlots]) == cudaSuccess) {
                settled++;
                j->open.store(std::min(settled + kSlots, j->pieces), std::memory_order_release);
            } else {
                Ring::pause();
            }
        }
    }
    j->open.store(j->pieces, std::memory_order_release);
    for (int i = 0; i < j->pieces; i++)
        while (!copied(i)) Ring::pause();
    if (err != cudaSuccess) cudaStreamSynchronize(ctx->stream);  // the next copy finds no transfer under way in its slots
    WB_CUDA(err);
    return WB_OK;
}

int copy(wb_context *ctx, void *host, void *dev, size_t bytes, bool to_host)
{
    std::unique_lock<std::mutex> lk(g_ring.use, std::defer_lock);
    cudaPointerAttributes at;
    if (bytes >= (to_host ? kHelpersFrom : kHelpersUpFrom) && (cudaPointerGetAttributes(&at, host) != cudaSuccess || at.type == cudaMemoryTypeUnregistered) && lk.try_lock() &&
        g_ring.prepare(ctx->device)) {
        Job j;
        j.host = (char *)host, j.bytes = bytes, j.pieces = (int)((bytes + kPiece - 1) / kPiece), j.to_host = to_host;
        const std::unique_ptr<std::atomic<unsigned char>[]> done(new (std::nothrow) std::atomic<unsigned char>[(size_t)j.pieces]());
        j.done = done.get();
        if (j.done && g_ring.start(&j) > 0) {
            const int rc = run_job(ctx, &j, (char *)dev);
            g_ring.finish(&j);
            if (rc == WB_OK && !to_host) WB_CUDA(cudaStreamSynchronize(ctx->stream));  // the slots are free for the next copy
            return rc;
        }
    }
    WB_CUDA(cudaMemcpyAsync(to_host ? host : dev, to_host ? dev : host, bytes, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, ctx->stream));
    return WB_OK;
}

}  // namespace

int copy_to_host(wb_context *ctx, void *host, const void *dev, size_t bytes) { return copy(ctx, host, const_cast<void *>(dev), bytes, true); }
int copy_to_device(wb_context *ctx, void *dev, const void *host, size_t bytes) { return copy(ctx, const_cast<void *>(host), dev, bytes, false); }

void transfer_retain()
{
    std::lock_guard<std::mutex> lk(g_users_lock);
    g_users++;
}
void transfer_release()
{
    std::lock_guard<std::mutex> lk(g_users_lock);
    if (--g_users > 0) return;
    std::lock_guard<std::mutex> use(g_ring.use);
    g_ring.stop();
    g_ring.release();
}

}  // namespace wb
