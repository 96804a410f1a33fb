// Copies between pageable host arrays and the device for the host-memory entry
// points.  A pageable cudaMemcpyAsync is staged by the driver through one
// thread at about 10 GB/s, which took nine tenths of a host-memory acoustic
// loop's time; here a few threads each stage 256 KB pieces through their own
// two pinned buffers, so the copies into (or out of) them run side by side and
// overlap the transfers.  95x95x50 loop of seven substeps, 32 MB both ways:
// 3.4 -> 2.2 ms (pieces of 64 and 128 KB 3.7 and 2.7).  Pinning the buffers
// takes one to several milliseconds, so a context sets a copier up only when it
// has copied kSetUpAfter bytes the ordinary way, which took as long, and the
// contexts of a device share one while any of them lives.
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>
#include <pthread.h>

namespace nimbus_host
{

class HostCopier
{
public:
    static constexpr size_t kPiece = 256 * 1024;
    static constexpr size_t kSmallest = 1024 * 1024;  // 0.66 MB copies gained nothing
    static constexpr size_t kSetUpAfter = 64 * 1024 * 1024;
    static constexpr unsigned kLanes = 4;  // threads, the caller among them

    explicit HostCopier(int device) : device_(device)
    {
        const unsigned cores = std::thread::hardware_concurrency();
        const unsigned lanes = std::min(kLanes, cores);
        if (lanes < 2) return;
        lanes_.resize(lanes);
        bool made = cudaMallocHost(reinterpret_cast<void**>(&block_), 2 * lanes * kPiece) == cudaSuccess;
        char* next = block_;
        for (Lane& l : lanes_)
            for (int b = 0; b < 2 && made; ++b, next += kPiece)
            {
                l.buf[b] = next;
                made = cudaEventCreateWithFlags(&l.done[b], cudaEventDisableTiming) == cudaSuccess;
            }
        if (!made)
        {
            (void)cudaGetLastError();
            return;
        }
        try
        {
            for (unsigned t = 1; t < lanes; ++t) threads_.emplace_back([this, t] { serve(t); });
            ready_ = true;
        }
        catch (...)  // no thread to be had: the caller copies the ordinary way
        {
        }
    }

    ~HostCopier()
    {
        {
            std::lock_guard<std::mutex> g(mutex_);
            stop_ = true;
            generation_.fetch_add(1, std::memory_order_release);
        }
        wake_.notify_all();
        for (std::thread& t : threads_) t.join();
        for (Lane& l : lanes_)
            for (int b = 0; b < 2; ++b)
                if (l.done[b])
                {
                    if (l.used[b]) cudaEventSynchronize(l.done[b]);
                    cudaEventDestroy(l.done[b]);
                }
        if (block_) cudaFreeHost(block_);
    }

    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;

    bool ready() const { return ready_; }

    // The device's copier; where no context holds one, a new one or null (not
    // asked for, or its set-up failed: then a later call may try again).
    static std::shared_ptr<HostCopier> of_device(int device, bool make)
    {
        static std::mutex mutex;
        static std::vector<std::weak_ptr<HostCopier>> all;
        std::lock_guard<std::mutex> g(mutex);
        if (all.size() <= static_cast<size_t>(device)) all.resize(static_cast<size_t>(device) + 1);
        std::weak_ptr<HostCopier>& slot = all[static_cast<size_t>(device)];
        std::shared_ptr<HostCopier> c = slot.lock();
        if (!c && make)
        {
            c = std::make_shared<HostCopier>(device);
            if (!c->ready()) return nullptr;
            slot = c;
        }
        return c;
    }

    // Stream-ordered copy to (up) or from the device.  Up: the host array has
    // been read when this returns; down: it has been written.  False, with
    // nothing done, while another context's copy is under way.
    bool copy(bool up, void* device, void* host, size_t bytes, cudaStream_t st, cudaError_t* result)
    {
        std::unique_lock<std::mutex> one(one_, std::try_to_lock);
        if (!one) return false;
        {
            std::lock_guard<std::mutex> g(mutex_);
            up_ = up;
            dev_ = static_cast<char*>(device);
            host_ = static_cast<char*>(host);
            bytes_ = bytes;
            stream_ = st;
            next_.store(0, std::memory_order_relaxed);
            error_.store(cudaSuccess, std::memory_order_relaxed);
            running_.store(static_cast<int>(threads_.size()), std::memory_order_relaxed);
            generation_.fetch_add(1, std::memory_order_release);
        }
        wake_.notify_all();
        work(lanes_[0]);
        while (running_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
        *result = static_cast<cudaError_t>(error_.load(std::memory_order_relaxed));
        return true;
    }

private:
    struct Lane
    {
        char* buf[2] = {nullptr, nullptr};
        cudaEvent_t done[2] = {nullptr, nullptr};
        bool used[2] = {false, false};
        int turn = 0;
    };

    void serve(unsigned lane)
    {
        pthread_setname_np(pthread_self(), "nimbus-copy");
        cudaSetDevice(device_);
        // These threads capture nothing: whether a copy may run beside another
        // thread's capture is for the calling thread's mode to say.
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        unsigned long long seen = 0;
        for (;;)
        {
            // The fields of one call follow each other closely: look for the
            // next copy for a moment before sleeping.
            for (int spin = 0; spin < 2000 && generation_.load(std::memory_order_acquire) == seen; ++spin)
                std::this_thread::yield();
            {
                std::unique_lock<std::mutex> g(mutex_);
                wake_.wait(g, [&] { return generation_.load(std::memory_order_relaxed) != seen; });
                seen = generation_.load(std::memory_order_relaxed);
                if (stop_) return;
            }
            work(lanes_[lane]);
            running_.fetch_sub(1, std::memory_order_release);
        }
    }

    bool check(cudaError_t e)
    {
        if (e == cudaSuccess) return true;
        int none = cudaSuccess;
        error_.compare_exchange_strong(none, e);
        return false;
    }

    // Waits until the transfer that last used buffer b is over.
    bool wait(Lane& l, int b)
    {
        if (!l.used[b]) return true;
        l.used[b] = false;
        return check(cudaEventSynchronize(l.done[b]));
    }

    void work(Lane& l)
    {
        size_t held = 0, held_len = 0;  // the piece in flight to the host and its buffer
        int held_buf = -1;
        bool ok = true;
        for (;;)
        {
            const size_t off = next_.fetch_add(1, std::memory_order_relaxed) * kPiece;
            if (off >= bytes_ || !ok) break;
            const size_t len = std::min(kPiece, bytes_ - off);
            const int b = l.turn;
            l.turn ^= 1;
            ok = wait(l, b);
            if (!ok) break;
            if (up_) std::memcpy(l.buf[b], host_ + off, len);
            ok = check(up_ ? cudaMemcpyAsync(dev_ + off, l.buf[b], len, cudaMemcpyHostToDevice, stream_)
                           : cudaMemcpyAsync(l.buf[b], dev_ + off, len, cudaMemcpyDeviceToHost, stream_)) &&
                 check(cudaEventRecord(l.done[b], stream_));
            l.used[b] = ok;
            if (up_ || !ok) continue;
            if (held_buf >= 0 && (ok = wait(l, held_buf))) std::memcpy(host_ + held, l.buf[held_buf], held_len);
            held = off;
            held_len = len;
            held_buf = b;
        }
        if (ok && held_buf >= 0 && wait(l, held_buf)) std::memcpy(host_ + held, l.buf[held_buf], held_len);
    }

    int device_;
    char* block_ = nullptr;  // the lanes' buffers
    bool ready_ = false;
    std::vector<Lane> lanes_;
    std::vector<std::thread> threads_;
    std::mutex one_, mutex_;
    std::condition_variable wake_;
    std::atomic<unsigned long long> generation_{0};
    bool stop_ = false;
    // The copy under way.
    bool up_ = true;
    char *dev_ = nullptr, *host_ = nullptr;
    size_t bytes_ = 0;
    cudaStream_t stream_ = nullptr;
    std::atomic<size_t> next_{0};
    std::atomic<int> running_{0}, error_{cudaSuccess};
};

}  // namespace nimbus_host
