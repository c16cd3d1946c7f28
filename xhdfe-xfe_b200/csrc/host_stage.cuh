// Copies between pageable host arrays and the device through pinned slots,
// filled and emptied by worker threads.
//
// A cudaMemcpyAsync of pageable memory is staged by the driver with one core:
// 152 MB in took 12 ms and 128 MB out 22 ms of a 50 ms call on 2M rows, 8 columns
// (three dims), and the calling thread is busy meanwhile.  With workers on half of
// 16 cores (kStageWorkers at most) the call takes 12.7 ms (50.8 before; its first,
// with the pinned slots to get, 47 for 81); the PCIe transfers alone need 5.  Here the arrays
// are cut into pieces of kStagePiece; a worker copies a piece into its own
// pinned slot and submits the slot's transfer, or submits a transfer into its
// slot and copies it out (taking the page faults of the result there).  No piece
// goes out before every piece in has been read, so results may lie over inputs.

#pragma once

#include <atomic>
#include <condition_variable>
#include <deque>
#include <mutex>
#include <thread>

#include "context.cuh"

namespace b200fe_host {

constexpr size_t kStagePiece = size_t(1) << 20;
constexpr int kStageSlots = 2;          // pinned slots per worker
constexpr int kStageWorkers = 12;       // at most
// Calls with fewer bytes of columns copy directly, the threads would cost more: 3
// columns, 7 MB 3.9 ms staged and 3.1 directly, 14 MB 4.4 and 4.7, 46 MB 7.2 and 12.7.
constexpr size_t kStageMinBytes = size_t(8) << 20;

// Memory that only a staged copy can move (neither pinned nor registered).
inline bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

class HostStager {
  public:
    ~HostStager() { finish(); }

    // Workers for copies on streams in / out; false (nothing started) when the
    // pinned slots or the threads cannot be had.
    bool start(b200fe_context* ctx, cudaStream_t in, cudaStream_t out, int groups) {
        device_ = ctx->device;
        in_ = in;
        out_ = out;
        left_.assign(groups, 0);
        event_.assign(groups, nullptr);
        submitted_.assign(groups, 0);
        const unsigned hw = std::thread::hardware_concurrency();
        const int workers = std::max(1, std::min(kStageWorkers, static_cast<int>(hw / 2)));
        if (!ctx->stage_pinned) {
            if (cudaHostAlloc(&ctx->stage_pinned, kStageWorkers * kStageSlots * kStagePiece, cudaHostAllocDefault) !=
                cudaSuccess) {
                cudaGetLastError();
                ctx->stage_pinned = nullptr;
                return false;
            }
        }
        char* base = static_cast<char*>(ctx->stage_pinned);
        try {
            for (int w = 0; w < workers; ++w)
                threads_.emplace_back([this, base, w] { work(base + w * kStageSlots * kStagePiece); });
        } catch (...) {
            if (threads_.empty()) return false;
        }
        return true;
    }
    // host -> device; ev is recorded on the in stream once group's last piece is submitted
    void add_in(void* dev, const void* host, size_t bytes, int group) {
        std::lock_guard<std::mutex> lk(mu_);
        for (size_t o = 0; o < bytes; o += kStagePiece) {
            queue_in_.push_back({static_cast<char*>(dev) + o, const_cast<char*>(static_cast<const char*>(host)) + o,
                                 std::min(kStagePiece, bytes - o), group});
            ++left_[group];
            ++unread_;
        }
    }
    // all of group's pieces are queued
    void close_group(int group, cudaEvent_t ev) {
        std::lock_guard<std::mutex> lk(mu_);
        event_[group] = ev;
        if (left_[group] == 0) submit_group(group);
        cv_.notify_all();
    }
    // waits until group's event is recorded; false after an error
    bool wait_in(int group) {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return submitted_[group] != 0 || error_ != cudaSuccess; });
        return error_ == cudaSuccess;
    }
    // device -> host, ordered behind what the out stream waits for by now
    void add_out(const void* dev, void* host, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu_);
        for (size_t o = 0; o < bytes; o += kStagePiece)
            queue_out_.push_back({const_cast<char*>(static_cast<const char*>(dev)) + o, static_cast<char*>(host) + o,
                                  std::min(kStagePiece, bytes - o), -1});
        cv_.notify_all();
    }
    // the queued copies done (or given up after an error), threads gone
    cudaError_t finish() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            closing_ = true;
            cv_.notify_all();
        }
        for (auto& t : threads_) t.join();
        threads_.clear();
        return error_;
    }

  private:
    struct Piece {
        char *dev, *host;
        size_t bytes;
        int group;  // -1: device -> host
    };
    void submit_group(int g) {  // mu_ held
        if (event_[g] && !submitted_[g]) {
            const cudaError_t e = cudaEventRecord(event_[g], in_);
            if (e != cudaSuccess) error_ = e;
            submitted_[g] = 1;
            cv_.notify_all();
        }
    }
    void work(char* slots) {
        cudaError_t e = cudaSetDevice(device_);
        cudaEvent_t ev[kStageSlots] = {nullptr};
        bool busy[kStageSlots] = {false};
        for (int i = 0; i < kStageSlots && e == cudaSuccess; ++i)
            e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
        for (int k = 0;; k = (k + 1) % kStageSlots) {
            Piece p;
            {
                std::unique_lock<std::mutex> lk(mu_);
                if (e != cudaSuccess && error_ == cudaSuccess) {
                    error_ = e;
                    cv_.notify_all();
                }
                cv_.wait(lk, [&] {
                    return error_ != cudaSuccess || !queue_in_.empty() ||
                           (unread_ == 0 && (closing_ || !queue_out_.empty()));
                });
                if (error_ != cudaSuccess) break;
                std::deque<Piece>& q = queue_in_.empty() ? queue_out_ : queue_in_;
                if (q.empty()) break;  // closing
                p = q.front();
                q.pop_front();
            }
            char* slot = slots + k * kStagePiece;
            if (busy[k]) e = cudaEventSynchronize(ev[k]);
            busy[k] = false;
            if (e == cudaSuccess && p.group >= 0) {
                std::memcpy(slot, p.host, p.bytes);
                e = cudaMemcpyAsync(p.dev, slot, p.bytes, cudaMemcpyHostToDevice, in_);
                if (e == cudaSuccess) e = cudaEventRecord(ev[k], in_);
                busy[k] = e == cudaSuccess;
                std::lock_guard<std::mutex> lk(mu_);
                if (--unread_ == 0) cv_.notify_all();
                if (e == cudaSuccess && --left_[p.group] == 0) submit_group(p.group);
            } else if (e == cudaSuccess) {
                e = cudaMemcpyAsync(slot, p.dev, p.bytes, cudaMemcpyDeviceToHost, out_);
                if (e == cudaSuccess) e = cudaEventRecord(ev[k], out_);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[k]);
                if (e == cudaSuccess) std::memcpy(p.host, slot, p.bytes);
            }
        }
        for (int i = 0; i < kStageSlots; ++i) {
            if (busy[i]) cudaEventSynchronize(ev[i]);  // the slot is the context's again
            if (ev[i]) cudaEventDestroy(ev[i]);
        }
    }
    int device_ = 0;
    cudaStream_t in_ = nullptr, out_ = nullptr;
    std::mutex mu_;
    std::condition_variable cv_;
    std::deque<Piece> queue_in_, queue_out_;
    int64_t unread_ = 0;  // pieces in not yet copied out of host memory
    std::vector<int64_t> left_;
    std::vector<cudaEvent_t> event_;
    std::vector<char> submitted_;
    std::vector<std::thread> threads_;
    cudaError_t error_ = cudaSuccess;
    bool closing_ = false;
};

}  // namespace b200fe_host
