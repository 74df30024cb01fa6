// Host-side rules of libcrt that need neither CUDA nor a GPU, apart so that a
// plain C++ program can check them (what kernels use too is CRT_HOST_DEVICE).
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>
#include <mutex>

#ifdef __CUDACC__
#define CRT_HOST_DEVICE __host__ __device__
#else
#define CRT_HOST_DEVICE
#endif

namespace crt {

// Something derived from a tree by the first context that needs it and read by
// every later one.  A tree may be traced from several contexts at once (a host
// thread and a stream each): the derivation is enqueued once, on the stream of the
// context that came first, and every other context's stream waits for it before
// that context reads the result.  A reader never sees a result whose derivation is
// not yet enqueued, and never runs before it.
class Derived {
public:
    // who: the calling context.  derive() enqueues the derivation and a mark after
    // it on that context's stream; wait() makes that stream wait for the mark.
    // Returns what they return: 0, or an error, after which a failed derivation is
    // left to the next caller.
    template <class Derive, class Wait>
    auto use(uint64_t who, Derive derive, Wait wait) -> decltype(derive()) {
        std::lock_guard<std::mutex> hold(mutex_);
        if (ready_) return by_ == who ? decltype(derive()){} : wait();
        const auto status = derive();
        if (status == decltype(derive()){}) {
            ready_ = true;
            by_ = who;
        }
        return status;
    }
    // The source has changed.  Like the change itself, not beside other uses.
    void reset() {
        std::lock_guard<std::mutex> hold(mutex_);
        ready_ = false;
    }
    bool ready() const {
        std::lock_guard<std::mutex> hold(mutex_);
        return ready_;
    }

private:
    mutable std::mutex mutex_;
    bool ready_ = false;
    uint64_t by_ = 0;  // whose stream the derivation is on
};

// A device allocation that only grows, by Memory::alloc(size) (null: refused) and
// Memory::free(p).  Growing drops the contents; a refused one leaves it empty.
template <class Memory>
struct GrowingBuffer {
    void* p = nullptr;
    size_t cap = 0;
    // For what a call can do without: refusing it is no error.
    bool try_reserve(size_t bytes) {
        if (bytes <= cap) return true;
        release();
        const size_t want = wanted(bytes);
        p = Memory::alloc(want);
        cap = p ? want : 0;
        return p != nullptr;
    }
    void release() {
        if (p) Memory::free(p);
        p = nullptr;
        cap = 0;
    }
    static constexpr size_t wanted(size_t bytes) { return bytes + bytes / 8 + 256; }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

// Four page-locked words that a context's kernels raise errors in, so that its
// calls neither clear nor copy a device word.  begin() before a call enqueues its
// kernels, end() once it has; sync() waits for the context's stream and returns 0 or
// an error.  A call that returns between the two leaves kernels behind that may
// still raise something: the next begin() waits for them, so that no call reports
// another's error.
class HostErrorWords {
public:
    template <class Sync>
    auto begin(Sync sync) -> decltype(sync()) {
        if (open_) {
            const auto status = sync();
            if (status != decltype(sync()){}) return status;
        }
        clear();
        open_ = true;
        return {};
    }
    template <class Sync>
    auto end(Sync sync, uint32_t out[4]) -> decltype(sync()) {
        const auto status = sync();
        if (status != decltype(sync()){}) return status;
        for (int k = 0; k < 4; ++k) out[k] = words[k];
        open_ = false;
        return {};
    }
    volatile uint32_t* words = nullptr;

private:
    void clear() {
        for (int k = 0; k < 4; ++k) words[k] = 0u;
    }
    bool open_ = false;
};

// Blocks of a launch whose blocks wait for one another: as many as a device of sms
// SMs holds at once, per_sm of them an SM (at most per_sm_max); 0: it cannot run.
constexpr int resident_blocks(bool cooperative, int per_sm, int per_sm_max, int sms) {
    return !cooperative || per_sm <= 0 || sms <= 0 ? 0 : (per_sm < per_sm_max ? per_sm : per_sm_max) * sms;
}

// The build's default launches, each with its blocks on the current device.
struct PlocGrids {
    int wide = 0, wave = 0, places = 0;  // cooperative launches
    int cluster = 0;                     // blocks of the thread-block cluster
    constexpr bool supported() const { return wide > 0 && wave > 0 && places > 0 && cluster > 0; }
};

// Whether a build whose launch failed may start over on the launch-per-iteration
// path.  That path reads the first clusters, records and look-back words, so only
// while no kernel that changes them has been enqueued.
constexpr bool may_start_over(bool not_supported, bool enqueued) { return not_supported && !enqueued; }

// What the walk over the compressed nodes takes (crt_walk4.cuh), as far as the host
// can tell before a launch; each of these refuses every ray of a scene or an image,
// which then goes to the binary nodes at once instead of by way of the left-over
// list.  A scene's range (its largest coordinate or extent) is abs_eps * 2^20.
// Nodes are quantised for ranges of 2^-40 .. 2^50:
CRT_HOST_DEVICE constexpr bool walk4_scene(float abs_eps) {
    return abs_eps >= 8.673617379884035e-19f && abs_eps <= 1073741824.f;
}
// Camera rays: origins within 8 ranges, ranges within 2^20 of the unit directions
// (whose largest component is at least 0.57).
inline bool walk4_camera(const float eye[3], float abs_eps) {
    const float range = abs_eps * 1048576.f;
    return std::fabs(eye[0]) <= 8.f * range && std::fabs(eye[1]) <= 8.f * range && std::fabs(eye[2]) <= 8.f * range &&
           range <= 1048576.f && range * 1048576.f >= 0.5f;
}

// Tiles of `size` items that n items make, for every n that fits.
CRT_HOST_DEVICE constexpr uint32_t tiles_of(uint32_t n, uint32_t size) { return n / size + (n % size != 0u ? 1u : 0u); }

// Persistent warps take items from a 32-bit counter, which ends up past their number
// by at most 32 a resident warp (152 SMs of 64 warps): above this bound it could come
// round to 0 and hand them out again.
constexpr uint32_t kMostPoolItems = 0xFFF00000u;

// When the rays traced over a tree of n triangles pay for deriving its compressed
// nodes, which takes 0.035 ns a triangle and 30 us: until then they are walked on the
// binary nodes.  Rays count from the tree's last change on, so a tree that is traced
// again and again pays once.
//
// Large traces: 64 triangles a closest-hit ray, 16 an any-hit one.  First trace after
// a change, us, with the derivation / on the binary nodes (sphere rays and camera rays
// over uniform and clustered triangles):
//   closest   4.19 M triangles,  65,536 rays   470-530 / 590-680
//             8.39 M            131,072        640-760 / 850-910
//            16.8 M              65,536       1,150-1,320 / 870-1,190 (waits)
//            16.8 M             262,144       1,240-1,640 / 1,020-2,030
//   any       4.19 M             65,536        380-430 / 360-460 (waits)
//             4.19 M            262,144        460-530 / 460-640
//            16.8 M           1,048,576       1,100-2,260 / 810-3,320
// An any-hit ray ends early and gains a quarter; camera rays gain less than others.
struct Walk4Demand {
    static constexpr uint64_t closest(uint64_t rays) { return 64 * rays; }
    static constexpr uint64_t any(uint64_t rays) { return 16 * rays; }
    // Pixels, 4 triangles each (primary rays, or those and shadow rays).  First image
    // after a change, 230,400 to 2.07 M pixels over 1.0 to 8.4 M triangles of three kinds
    // of scene: from 0.26 pixels a triangle on faster with the derivation in every one
    // (1080p over 5.2 M triangles of a sphere 1,097 / 1,171 us, over 8.0 M clustered ones
    // 1,367 / 1,408, over 1.0 M uniform ones 1,007 / 1,047).
    static constexpr uint64_t pixels(uint64_t n) { return 4 * n; }
};
constexpr bool walk4_pays(uint64_t demand, uint32_t n) { return demand >= n; }

}  // namespace crt
