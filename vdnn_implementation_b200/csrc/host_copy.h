// Copies between device memory and pageable host memory through pinned staging buffers and several host threads.
#ifndef VDNN_B200_HOST_COPY_H_
#define VDNN_B200_HOST_COPY_H_

#include <stddef.h>

#include <cuda_runtime.h>

#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace vdnn {

// A plain cudaMemcpy to pageable memory runs one staging loop on one host thread, and that thread also takes every page
// fault of a freshly allocated destination: 4.8 GB/s measured for the parameters of VGG16 (553 MB), a tenth of what the
// link carries.  Here each worker thread owns two pinned buffers and a stream and takes the next chunk of the tensor that
// nobody has taken yet: the copy engine fills one of its buffers while the thread moves the other to its destination.
// Chunks begin on 2 MB boundaries of the HOST address, so no two threads fault in the same huge page.
// The buffers (workers x 2 x 2 MB) and the threads, which sleep between copies, are made at the first large copy, kept for the
// object's life and released with it.  Where pinned memory, streams or threads run out, the workers that could be had do the
// copy, and cudaMemcpy does it where there is none; the next copy asks for the missing ones again.  Host threads may call at once, as they may cudaMemcpy: the buffers serve one copy at a
// time, the others wait for it.
class HostCopy {
public:
    HostCopy() : workers_(), made_(0), round_(0), wanted_(0), busy_(0), stop_(false) {}
    ~HostCopy();
    // The caller has synchronised whatever produces the source.  Returns a cudaError_t.
    cudaError_t to_host(void* dst_h, const void* src, size_t bytes, int device) { return run(dst_h, const_cast<void*>(src), bytes, device, true); }
    cudaError_t to_device(void* dst, const void* src_h, size_t bytes, int device) { return run(const_cast<void*>(src_h), dst, bytes, device, false); }

private:
    struct Worker { cudaStream_t stream; cudaEvent_t done[2]; char* pinned[2]; };
    static constexpr size_t kMaxWorkers = 8;
    static cudaError_t make(Worker* w);
    static void release(Worker* w);
    HostCopy(const HostCopy&);
    HostCopy& operator=(const HostCopy&);
    cudaError_t run(void* host, void* dev, size_t bytes, int device, bool to_host);
    size_t make_workers(size_t want);                   // returns how many of them there are
    void serve(size_t index);
    std::mutex turn_;                   // held for a copy that uses the members below
    Worker workers_[kMaxWorkers];
    size_t made_;
    // threads_[i] takes part in round n for worker i + 1 when job_ wants it to (i + 1 < wanted_)
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable wake_, done_;
    std::function<void(const Worker&)> job_;
    unsigned long long round_;
    size_t wanted_, busy_;
    bool stop_;
};

}  // namespace vdnn

#endif
