// host_stage.h -- the host side of a trace over pageable buffers: rays are copied into pinned staging
// slots and hits out of them, in units of 4096 rays, by the calling thread and a few helpers, while the
// device copies and traces other slots.
//
// A copy between the device and pageable memory goes through the driver's own staging on one core and
// holds up its caller, so that copies in, traces and copies out followed one another: 307,039 rays took
// 524 us in, 45 us traced, 162 us out of a call of 1.3 ms. Helpers fill the slots as fast as the link
// empties them (42 GB/s).
// The same call takes 0.74 ms (1.02 ms without helpers, 0.73 ms with 7), 4 M rays 6.8 ms instead of 32,
// 100 rays 54 us instead of 141.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <thread>

#include "../../include/liar_gpu.h"

namespace liar_gpu {

constexpr size_t kStageUnit = 4096;                  // rays copied at once: 128 KB in
constexpr size_t kStageUnits = 8;                    // units of a chunk (a slot)
constexpr size_t kStageChunk = kStageUnit * kStageUnits;
constexpr size_t kStageSlots = 4;                    // 4 MB of rays, 1 MB of hits
constexpr int kStageHelpers = 4;
// Pinning the slots takes about 3 ms once, which staging gives back after some 2^20 rays, a call counting
// for 2^14 more (its own waits): a context stages its host calls once it has been asked for that many.
constexpr size_t kStageAfter = (size_t)1 << 20, kStageCall = (size_t)1 << 14;

struct HostStage {
    const liar_ray* rays;  // caller's rays
    liar_hit* hits;        // caller's hits, or NULL: prim and t
    int32_t* prim;
    float* t;
    size_t n;
    liar_ray* pin_rays;  // kStageSlots chunks each
    liar_hit* pin_hits;

    std::atomic<size_t> in_next{0}, in_limit{0}, out_next{0}, out_limit{0};  // units claimed / allowed
    std::atomic<size_t> in_done[kStageSlots] = {}, out_done[kStageSlots] = {};  // units copied, per slot
    std::atomic<bool> stop{false};
    std::thread helpers[kStageHelpers];
    int n_helpers = 0;

    size_t units() const { return (n + kStageUnit - 1) / kStageUnit; }
    size_t chunks() const { return (n + kStageChunk - 1) / kStageChunk; }
    // units copied in (or out) of chunk k's slot once chunk k has been: earlier chunks of the slot are full
    size_t slot_count(size_t k) const {
        const size_t left = units() - k * kStageUnits;
        return (k / kStageSlots) * kStageUnits + (left < kStageUnits ? left : kStageUnits);
    }
    // chunks whose units may be copied now
    void allow_in(size_t chunks_allowed) { raise(in_limit, chunks_allowed); }
    void allow_out(size_t chunks_allowed) { raise(out_limit, chunks_allowed); }
    bool filled(size_t k) const { return in_done[k % kStageSlots].load(std::memory_order_acquire) >= slot_count(k); }
    bool emptied(size_t k) const { return out_done[k % kStageSlots].load(std::memory_order_acquire) >= slot_count(k); }

    // copies one unit, hits first (they free a slot); false: none may be copied now
    bool step() {
        size_t u;
        if (claim(out_next, out_limit, &u)) {
            copy_out(u);
            out_done[u / kStageUnits % kStageSlots].fetch_add(1, std::memory_order_release);
            return true;
        }
        if (claim(in_next, in_limit, &u)) {
            std::memcpy(pin_rays + place(u), rays + u * kStageUnit, count(u) * sizeof(liar_ray));
            in_done[u / kStageUnits % kStageSlots].fetch_add(1, std::memory_order_release);
            return true;
        }
        return false;
    }
    // one helper for every 8 units, below the number of cores
    void start() {
        size_t want = units() / 8;
        const size_t cores = std::thread::hardware_concurrency();
        if (want >= cores) want = cores ? cores - 1 : 0;
        if (want > (size_t)kStageHelpers) want = kStageHelpers;
        try {
            while (n_helpers < (int)want) {
                helpers[n_helpers] = std::thread([this] {
                    while (!stop.load(std::memory_order_acquire))
                        if (!step()) std::this_thread::yield();
                });
                ++n_helpers;
            }
        } catch (...) {  // no more threads: those that run, and the caller, do it
        }
    }
    ~HostStage() {
        stop.store(true, std::memory_order_release);
        for (int i = 0; i < n_helpers; ++i) helpers[i].join();
    }

private:
    size_t count(size_t u) const { return n - u * kStageUnit < kStageUnit ? n - u * kStageUnit : kStageUnit; }
    static size_t place(size_t u) {
        return (u / kStageUnits % kStageSlots) * kStageChunk + (u % kStageUnits) * kStageUnit;
    }
    void raise(std::atomic<size_t>& limit, size_t chunks_allowed) {
        const size_t u = chunks_allowed * kStageUnits, all = units();
        limit.store(u < all ? u : all, std::memory_order_release);
    }
    static bool claim(std::atomic<size_t>& next, std::atomic<size_t>& limit, size_t* u) {
        size_t v = next.load(std::memory_order_relaxed);
        while (v < limit.load(std::memory_order_acquire))
            if (next.compare_exchange_weak(v, v + 1, std::memory_order_relaxed)) {
                *u = v;
                return true;
            }
        return false;
    }
    void copy_out(size_t u) {
        const liar_hit* src = pin_hits + place(u);
        const size_t base = u * kStageUnit, m = count(u);
        if (hits) {
            std::memcpy(hits + base, src, m * sizeof(liar_hit));
            return;
        }
        int32_t* p = prim + base;
        float* d = t + base;
        for (size_t i = 0; i < m; ++i) {
            p[i] = src[i].prim;
            d[i] = src[i].t;
        }
    }
};

}  // namespace liar_gpu
