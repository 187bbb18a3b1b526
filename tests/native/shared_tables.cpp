// Test-only: akvisqol_b200/csrc/shared_tables.h. Prints one line a property:
// a key is formed while another one is; threads that ask for one key form it
// once and share it; a table without owners is formed again.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "../../akvisqol_b200/csrc/shared_tables.h"

int main() {
    using namespace vqb;
    SharedTables<int, int> shared;
    std::mutex mu;
    std::condition_variable cv;
    bool inside = false, other = false, met = false;
    std::thread slow([&] {
        shared.get(1, [&] {
            std::unique_lock<std::mutex> lock(mu);
            inside = true;
            cv.notify_all();
            met = cv.wait_for(lock, std::chrono::seconds(10), [&] { return other; });
            return std::make_shared<const int>(1);
        });
    });
    {
        std::unique_lock<std::mutex> lock(mu);
        cv.wait(lock, [&] { return inside; });
    }
    shared.get(2, [&] {
        std::lock_guard<std::mutex> lock(mu);
        other = true;
        cv.notify_all();
        return std::make_shared<const int>(2);
    });
    slow.join();
    std::puts(met ? "side by side" : "one after the other");

    std::atomic<int> made{0};
    std::vector<std::shared_ptr<const int>> got(8);
    std::vector<std::thread> pool;
    for (size_t t = 0; t < got.size(); ++t)
        pool.emplace_back([&, t] { got[t] = shared.get(3, [&] { return std::make_shared<const int>(++made); }); });
    for (auto &t : pool) t.join();
    bool same = true;
    for (auto &g : got) same = same && g == got[0];
    std::printf("formed %d, %s\n", made.load(), same ? "shared" : "not shared");
    got.clear();
    shared.get(3, [&] { return std::make_shared<const int>(++made); });
    std::printf("formed %d\n", made.load());
}
