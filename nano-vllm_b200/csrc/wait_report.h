// How a kernel's bounded wait that gave up reaches the host.
//
// A kernel whose wait runs out leaves its results undefined, so the host has to hear of it.  It counts into one word of host memory that
// the device sees (no copy, no synchronisation: the host reads it wherever it likes).  Launches of such kernels look at the word first and
// refuse once after it has moved; a program that replays graphs, which launch nothing from here, asks for the count where it waits anyway.
// Plain C++: the allocation is the caller's (wait_report.cuh).
#pragma once
#include <atomic>
#include <cstdint>

struct B200WaitReport {
    std::atomic<volatile uint32_t*> word{nullptr};
    std::atomic<uint32_t> told{0};                 // the count that the host has heard of

    uint32_t count() const {
        const volatile uint32_t* w = word.load(std::memory_order_acquire);
        return w ? *w : 0;
    }
    // True once after waits have given up.
    bool news() {
        const uint32_t now = count();
        return told.exchange(now, std::memory_order_acq_rel) != now;
    }
};
