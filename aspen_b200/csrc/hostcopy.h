// Results into pageable host memory.
//
// The results this library hands out are malloc'ed (the caller frees them).  The driver stages a copy into such memory through
// one thread, which also faults in the fresh pages: 6 GB/s, a 12.6 MB result took longer than most networks run.  Here
// a few threads copy (and fault) the pieces that the DMA engine has moved into a pinned ring.
// B200 host, 16 cores: 12.6 MB into a fresh buffer 1.97 -> 0.57 ms, 6.3 MB 0.91 -> 0.31.  Uploads stay with the driver: it
// reads resident pages at 13 - 20 GB/s, and the same team filling the ring was no faster.
// The threads, the ring (8 MB) and the small buffer belong to one engine and end with it; an engine's calls come from one host
// thread.  Pinned memory is allocated by `prepare`, which the engine calls only while no kernel of it is resident: a copy beside
// a resident kernel uses what there is, and the driver's staging otherwise.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

class HostCopy {
public:
    static constexpr size_t PIECE = 512u << 10, SLOTS = 16;
    static constexpr size_t MIN_BYTES = 1u << 20;      // below, waking the threads costs more than they save
    static constexpr size_t SMALL = 256u << 10;        // up to here one pinned buffer and a memcpy (the driver's staging takes 10 us more)

    HostCopy() {}
    HostCopy(const HostCopy &) = delete;
    ~HostCopy() {
        {
            std::lock_guard<std::mutex> l(m_);
            quit_ = true;
        }
        cv_.notify_all();
        for (std::thread &t : team_) t.join();
        for (cudaEvent_t e : ev_) if (e) cudaEventDestroy(e);
        if (ring_) cudaFreeHost(ring_);
        if (small_) cudaFreeHost(small_);
    }
    // Makes what copies of up to `bytes` use.  Nothing is lost if it fails: those copies then go through the driver.
    void prepare(size_t bytes) {
        if (!small_ && cudaHostAlloc(&small_, SMALL, cudaHostAllocDefault) != cudaSuccess) { small_ = nullptr; cudaGetLastError(); }
        if (bytes >= MIN_BYTES) start();
    }
    // Returns once the copy is complete.
    cudaError_t down(void *host, const void *dev, size_t bytes, cudaStream_t st);

private:
    // The ring counts as there once everything that goes with it is; otherwise what was made is given back, the copy goes through
    // the driver, and the next large one tries again.
    bool start() {
        if (ring_) return true;
        void *ring = nullptr;
        size_t made = 0;
        bool ok = cudaHostAlloc(&ring, PIECE * SLOTS, cudaHostAllocDefault) == cudaSuccess;
        while (ok && made < SLOTS && (ok = cudaEventCreateWithFlags(&ev_[made], cudaEventDisableTiming) == cudaSuccess)) made++;
        if (ok) {
            const unsigned n = std::min(8u, std::max(2u, std::thread::hardware_concurrency() / 2u));
            try {
                for (unsigned i = 0; i < n; i++) team_.emplace_back([this] { loop(); });
            } catch (const std::exception &) {     // no more threads: those that there are do the work
            }
            if (!team_.empty()) { ring_ = ring; return true; }
        }
        for (size_t i = 0; i < made; i++) { cudaEventDestroy(ev_[i]); ev_[i] = nullptr; }
        if (ring) cudaFreeHost(ring);
        cudaGetLastError();
        return false;
    }
    void loop() {
        for (unsigned seen = 0;;) {
            {
                std::unique_lock<std::mutex> l(m_);
                cv_.wait(l, [&] { return quit_ || job_ != seen; });
                if (quit_) return;
                seen = job_;
            }
            work();
            busy_.fetch_sub(1, std::memory_order_release);
        }
    }
    char *slot(size_t s) { return (char *)ring_ + s * PIECE; }
    bool done(size_t i) { return done_[i].load(std::memory_order_acquire) != 0; }
    void work() {
        for (size_t i; (i = next_.fetch_add(1)) < pieces_;) {
            while (i >= landed_.load(std::memory_order_acquire)) std::this_thread::yield();
            memcpy(host_ + i * PIECE, slot(i % SLOTS), std::min(PIECE, bytes_ - i * PIECE));
            done_[i].store(1, std::memory_order_release);
        }
    }

    void *ring_ = nullptr, *small_ = nullptr;
    cudaEvent_t ev_[SLOTS] = {};
    std::vector<std::thread> team_;
    std::mutex m_;
    std::condition_variable cv_;
    bool quit_ = false;
    unsigned job_ = 0;
    // the transfer in work
    char *host_ = nullptr;
    size_t bytes_ = 0, pieces_ = 0;
    std::atomic<size_t> next_{0}, landed_{0};       // pieces taken by the team / landed in the ring
    std::atomic<unsigned> busy_{0};
    std::vector<std::atomic<unsigned char>> done_;
};

inline cudaError_t HostCopy::down(void *host, const void *dev, size_t bytes, cudaStream_t st) {
    cudaPointerAttributes attr;
    const bool pinned = cudaPointerGetAttributes(&attr, host) == cudaSuccess && attr.type != cudaMemoryTypeUnregistered;
    if (bytes <= SMALL && !pinned && small_) {
        cudaError_t e = cudaMemcpyAsync(small_, dev, bytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) memcpy(host, small_, bytes);
        return e;
    }
    if (bytes < MIN_BYTES || pinned || !ring_) {
        const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
        return e != cudaSuccess ? e : cudaStreamSynchronize(st);
    }
    host_ = (char *)host; bytes_ = bytes;
    pieces_ = (bytes + PIECE - 1) / PIECE;
    if (done_.size() < pieces_) done_ = std::vector<std::atomic<unsigned char>>(pieces_);
    for (size_t i = 0; i < pieces_; i++) done_[i].store(0, std::memory_order_relaxed);
    next_.store(0);
    landed_.store(0);
    busy_.store((unsigned)team_.size());
    {
        std::lock_guard<std::mutex> l(m_);
        job_++;
    }
    cv_.notify_all();
    // This thread alone talks to the driver (its calls share a lock).  Pieces go through the ring in order.
    cudaError_t err = cudaSuccess;
    auto chk = [&](cudaError_t e) { if (e != cudaSuccess && err == cudaSuccess) err = e; };
    for (size_t issued = 0, landed = 0; landed < pieces_;) {
        if (issued < pieces_ && (issued < SLOTS || done(issued - SLOTS))) {
            const size_t s = issued % SLOTS, off = issued * PIECE;
            chk(cudaMemcpyAsync(slot(s), (const char *)dev + off, std::min(PIECE, bytes - off), cudaMemcpyDeviceToHost, st));
            chk(cudaEventRecord(ev_[s], st));
            issued++;
        } else if (landed < issued) {
            const cudaError_t q = cudaEventQuery(ev_[landed % SLOTS]);
            if (q == cudaErrorNotReady) continue;
            chk(q);
            landed_.store(++landed, std::memory_order_release);
        } else std::this_thread::yield();
    }
    while (busy_.load(std::memory_order_acquire)) std::this_thread::yield();
    return err;
}
