// The library's word for waits that gave up (wait_report.h has the idea): 4 bytes of pinned, portable host memory, made on the first
// launch that needs it and kept for the process.
#pragma once
#include <mutex>

#include "common.cuh"
#include "wait_report.h"

// One per library, also where both are loaded into a process (a function's static is one object for all that name it alike).
#ifndef B200_LIB
#define B200_LIB attn
#endif
namespace b200wait {
inline namespace B200_LIB {

inline B200WaitReport& report() {
    static B200WaitReport r;
    return r;
}

// B200_OK and the word's address for a launch's parameters; B200_EWAIT once after waits of earlier launches gave up.
inline int launch_word(uint32_t** out) {
    B200WaitReport& r = report();
    volatile uint32_t* w = r.word.load(std::memory_order_acquire);
    if (!w) {
        static std::mutex mu;
        std::lock_guard<std::mutex> lock(mu);
        w = r.word.load(std::memory_order_acquire);
        if (!w) {
            // allocating is allowed while a stream is being captured only in the relaxed mode
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            B200_CUDA_CHECK((b200_ctx*)nullptr, cudaThreadExchangeStreamCaptureMode(&mode));
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, sizeof(uint32_t), cudaHostAllocPortable | cudaHostAllocMapped);
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) {
                b200_tls_cuda_error() = cudaGetErrorString(e);
                return B200_ECUDA;
            }
            w = static_cast<volatile uint32_t*>(p);
            *w = 0;
            r.word.store(w, std::memory_order_release);
        }
    }
    *out = const_cast<uint32_t*>(w);
    return r.news() ? B200_EWAIT : B200_OK;
}

// Waits that gave up since the process began; launches stay silent about those that have been counted here.
inline uint32_t timeouts() {
    B200WaitReport& r = report();
    r.news();
    return r.told.load(std::memory_order_acquire);
}

}  // inline namespace
}  // namespace b200wait
