// A staged copy whose stream still runs earlier work leaves the ring to the
// copies of other streams (orrery_b200/csrc/host_copy.cpp) against the host-only
// CUDA stand-in: an operation on the first stream ends only after the second
// stream's copy has returned (or after a limit, which fails the test).
// Prints "ok" and exits 0 on success.
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "common.h"
#include "host_copy.h"

namespace {

int behind_a_busy_stream(bool upload, std::size_t count) {
    std::mutex m;
    std::condition_variable cv;
    bool done = false, in_time = false;
    fake::Stream busy, idle;
    busy.push([&] {
        std::unique_lock<std::mutex> g(m);
        in_time = cv.wait_for(g, std::chrono::seconds(20), [&] { return done; });
    });
    std::vector<float> a(count, 0.5f), b(count, 0.25f);
    std::vector<double> a_host(count, -7.0), b_host(count, -7.0);
    std::vector<float> up(count, 1.5f);
    std::thread waiting([&] {
        if (upload) {
            const orr::HostSpan span{up.data(), a.data(), count * sizeof(float)};
            orr::copy_to_device(&span, 1, &busy, 0);
        } else {
            const orr::HostSpan span{a_host.data(), a.data(), count * sizeof(float), true, 1.0};
            orr::copy_to_host(&span, 1, &busy, 0);
        }
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(200));   // the first copy waits for its stream
    const orr::HostSpan span{b_host.data(), b.data(), count * sizeof(float), true, 0.0};
    orr::copy_to_host(&span, 1, &idle, 0);
    {
        std::lock_guard<std::mutex> g(m);
        done = true;
    }
    cv.notify_all();
    waiting.join();
    if (!in_time) {
        std::printf("the second copy waited for the first one's stream (upload %d, %zu values)\n", upload, count);
        return 1;
    }
    for (std::size_t k = 0; k < count; ++k) {
        if (b_host[k] != 0.25 || (upload ? a[k] != 1.5f : a_host[k] != 1.5)) {
            std::printf("value %zu differs (upload %d)\n", k, upload);
            return 1;
        }
    }
    return 0;
}

} // namespace

int main() {
    const std::size_t small = 1000, large = std::size_t(5) << 20;   // one thread, and several chunks of 4 MiB
    if (behind_a_busy_stream(false, small) != 0 || behind_a_busy_stream(false, large) != 0 ||
        behind_a_busy_stream(true, large) != 0) {
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
