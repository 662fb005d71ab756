// A second stream for kernels of one call that do not depend on one another and are too small to fill the chip alone.
//
// fork() makes the side stream wait for what the caller's stream has been given so far; join() makes the caller's stream wait for the
// side stream.  One side stream and two events per host thread and device, made on first use and kept until the thread ends, so that
// threads never share one; calls of one thread on several streams order themselves behind one another on it.  A stream that is being
// captured gets none (nothing may be created there), and where creation fails the caller goes on with its own stream.
#pragma once
#include <cuda_runtime.h>

namespace llattn {

class SideStream {
  public:
    // null: use the caller's stream
    static inline SideStream* get(cudaStream_t caller);
    cudaStream_t stream() const { return s; }
    cudaError_t fork(cudaStream_t caller) {
        const cudaError_t e = cudaEventRecord(forked, caller);
        return e != cudaSuccess ? e : cudaStreamWaitEvent(s, forked, 0);
    }
    cudaError_t join(cudaStream_t caller) {
        const cudaError_t e = cudaEventRecord(done, s);
        return e != cudaSuccess ? e : cudaStreamWaitEvent(caller, done, 0);
    }

  private:
    static constexpr int MAX_DEVICES = 16;
    struct PerThread;
    void create() {
        state = 2;
        if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return;
        if (cudaEventCreateWithFlags(&forked, cudaEventDisableTiming) != cudaSuccess || cudaEventCreateWithFlags(&done, cudaEventDisableTiming) != cudaSuccess) return;
        state = 1;
    }
    void destroy() {
        // the runtime may be gone already when the process ends: errors do not matter here
        if (state != 1) return;
        cudaEventDestroy(forked);
        cudaEventDestroy(done);
        cudaStreamDestroy(s);
    }
    cudaStream_t s = nullptr;
    cudaEvent_t forked = nullptr, done = nullptr;
    int state = 0;      // 0 not made yet, 1 ready, 2 not available
};

struct SideStream::PerThread {
    SideStream of[MAX_DEVICES];
    ~PerThread() {
        for (SideStream& s : of) s.destroy();
    }
};

inline SideStream* SideStream::get(cudaStream_t caller) {
    static thread_local PerThread all;
    int dev = -1;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(caller, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) return nullptr;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return nullptr;
    SideStream& s = all.of[dev];
    if (s.state == 0) s.create();
    return s.state == 1 ? &s : nullptr;
}

}  // namespace llattn
