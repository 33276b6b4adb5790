// Something that a process does once per device, such as allowing a kernel its shared memory: attributes of a kernel belong to
// the device that is current when they are set, so a flag for the process would leave the second device without.
#pragma once
#include <atomic>
#include <stdint.h>

namespace qnn {

struct OncePerDevice {
    std::atomic<uint64_t> done{0};                               // a bit per device; beyond 64 devices it is done every time
    // what `act` returns if it is 0 once; until then it is tried again.  Two threads may both act.
    template <typename Act>
    int run(int device, Act act) {
        const bool counted = device >= 0 && device < 64;
        if (counted && (done.load(std::memory_order_acquire) >> device & 1)) return 0;
        const int rc = act();
        if (rc == 0 && counted) done.fetch_or(1ull << device, std::memory_order_release);
        return rc;
    }
};

// What a launcher asks about a device (how many of its blocks fit at once): the last answer, with what it was asked for.
struct KnownPerDevice {
    std::atomic<uint64_t> last[64] = {};                         // 0: nothing yet; else key + 1 above the answer
    template <typename Ask>
    int get(int device, uint32_t key, Ask ask) {
        if (device < 0 || device >= 64) return ask();
        const uint64_t have = last[device].load(std::memory_order_relaxed), mine = ((uint64_t)key + 1) << 32;
        if (have >> 32 == mine >> 32) return (int)(uint32_t)have;
        const int answer = ask();
        last[device].store(mine | (uint32_t)answer, std::memory_order_relaxed);
        return answer;
    }
};

}  // namespace qnn
