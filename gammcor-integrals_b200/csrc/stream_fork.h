// stream_fork.h -- auxiliary streams forked from a main stream and joined back.
#pragma once
#include <cuda_runtime_api.h>

namespace gci {

// Work launched on aux[0..n) between begin() and join() follows what the main stream held at
// begin(), and precedes what it gets after join().  Buffers are freed in the order of the main
// stream, so a scope that is left by an exception joins too: declare the fork after the buffers
// that its launches use.  Threads that share the events may interleave: a wait then takes the
// other thread's later record on the same stream.
class StreamFork {
public:
    StreamFork(cudaStream_t main, const cudaStream_t* aux, int n, cudaEvent_t fork, const cudaEvent_t* join)
        : main_(main), aux_(aux), n_(n), fork_(fork), join_(join) {}
    StreamFork(const StreamFork&) = delete;
    StreamFork& operator=(const StreamFork&) = delete;
    ~StreamFork() { (void)join(); }

    cudaError_t begin()
    {
        cudaError_t e = cudaEventRecord(fork_, main_);
        for (int q = 0; q < n_ && e == cudaSuccess; ++q) e = cudaStreamWaitEvent(aux_[q], fork_, 0);
        open_ = e == cudaSuccess;
        return e;
    }

    // All streams in any case; a stream that cannot be joined by its event is waited for here.
    // The first error.
    cudaError_t join()
    {
        if (!open_) return cudaSuccess;
        open_ = false;
        cudaError_t first = cudaSuccess;
        for (int q = 0; q < n_; ++q) {
            cudaError_t e = cudaEventRecord(join_[q], aux_[q]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, join_[q], 0);
            if (e != cudaSuccess) (void)cudaStreamSynchronize(aux_[q]);
            if (first == cudaSuccess) first = e;
        }
        return first;
    }

private:
    cudaStream_t main_;
    const cudaStream_t* aux_;
    int n_;
    cudaEvent_t fork_;
    const cudaEvent_t* join_;
    bool open_ = false;
};

} // namespace gci
