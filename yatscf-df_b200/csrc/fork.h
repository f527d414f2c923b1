// Independent launches side by side: a Fork runs them on LANES streams between
// an event on the caller's stream and events that it waits for. Streams and
// events come from a per-device pool of at most KEEP sets (a set belongs to one
// Fork at a time, so threads do not share one), so nothing is created per call.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace tscf {

class Fork {
    static constexpr int LANES = 8, KEEP = 4;
    struct Set {
        cudaStream_t st[LANES] = {};
        cudaEvent_t begin = nullptr, done[LANES] = {};
        bool ok = true;
        Set()
        {
            ok = cudaEventCreateWithFlags(&begin, cudaEventDisableTiming) == cudaSuccess;
            for (int k = 0; k < LANES; k++)
                ok = ok && cudaStreamCreateWithFlags(&st[k], cudaStreamNonBlocking) == cudaSuccess &&
                     cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming) == cudaSuccess;
        }
        ~Set()
        {
            for (int k = 0; k < LANES; k++) {
                if (st[k]) cudaStreamDestroy(st[k]);
                if (done[k]) cudaEventDestroy(done[k]);
            }
            if (begin) cudaEventDestroy(begin);
        }
    };
    static std::mutex &lock();
    static std::vector<Set *> &pool(int dev);
    int dev_ = 0, n_ = 0;
    cudaStream_t s_;
    Set *set_ = nullptr;

public:
    // side = false: every launch stays on s
    Fork(cudaStream_t s, bool side) : s_(s)
    {
        if (!side) return;
        cudaGetDevice(&dev_);
        {
            std::lock_guard<std::mutex> g(lock());
            auto &v = pool(dev_);
            if (!v.empty()) {
                set_ = v.back();
                v.pop_back();
            }
        }
        if (!set_) set_ = new Set;
        if (!set_->ok || cudaEventRecord(set_->begin, s) != cudaSuccess) {
            cudaGetLastError();
            delete set_;
            set_ = nullptr;
        }
    }
    Fork(const Fork &) = delete;
    Fork &operator=(const Fork &) = delete;
    cudaStream_t next()
    {
        if (!set_) return s_;
        const int k = n_++ % LANES;
        if (n_ <= LANES) cudaStreamWaitEvent(set_->st[k], set_->begin, 0);
        return set_->st[k];
    }
    ~Fork()
    {
        if (!set_) return;
        for (int k = 0; k < LANES && k < n_; k++) {
            cudaEventRecord(set_->done[k], set_->st[k]);
            cudaStreamWaitEvent(s_, set_->done[k], 0);
        }
        std::lock_guard<std::mutex> g(lock());
        auto &v = pool(dev_);
        if ((int) v.size() < KEEP) v.push_back(set_);
        else delete set_;
    }
};

}  // namespace tscf
