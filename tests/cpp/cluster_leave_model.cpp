// Runs the cluster's end protocol (cluster_leave.hpp) with a thread per block.
// Every block works through `levels` levels, each of which starts with a
// barrier within the traversal (as the levels that read all parts do) and then
// uses every other block's memory; block `quitter` gives up in the wait at the
// end of level `at`, whose count the others have already got, so they go on to
// the next level.  Prints how many uses met a block that was gone, how many
// blocks did not report the give-up, and how many were still there at the end.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "cluster_leave.hpp"

struct Cluster {
    std::mutex mu;
    std::condition_variable cv;
    int there, arrived = 0, phase = 0;
    std::vector<std::atomic<int>> flag, alive;
    std::atomic<int> strayed{0};
    explicit Cluster(int n) : there(n), flag(n), alive(n) {
        for (auto& f : flag) f = 0;
        for (auto& a : alive) a = 1;
    }
    void turn() {  // with mu held: a full barrier moves on
        if (arrived < there || there == 0) return;
        arrived = 0;
        ++phase;
        cv.notify_all();
    }
    void sync() {
        std::unique_lock<std::mutex> l(mu);
        const int p = phase;
        ++arrived;
        turn();
        cv.wait(l, [&] { return phase != p; });
    }
    void exit(int b) {
        std::unique_lock<std::mutex> l(mu);
        alive[b] = 0;
        --there;
        turn();
    }
};

struct Block {
    Cluster& c;
    int b, n;
    void sync() { c.sync(); }
    void raise() {
        for (auto& f : c.flag) f = 1;
    }
    bool raised() { return c.flag[b] != 0; }
    void settle() {}
    void use() {
        for (int o = 0; o < n; ++o) {
            std::this_thread::sleep_for(std::chrono::microseconds(300));  // a use lasts a while
            if (!c.alive[o]) ++c.strayed;
        }
    }
};

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    const int n = std::atoi(argv[1]), levels = std::atoi(argv[2]), quitter = std::atoi(argv[3]), at = std::atoi(argv[4]);
    const bool notices = std::atoi(argv[5]) != 0;  // the others stand in a wait and see the flag there
    Cluster c(n);
    std::vector<std::thread> t;
    std::vector<int> reported(n, 0);
    for (int b = 0; b < n; ++b)
        t.emplace_back([&, b] {
            Block me{c, b, n};
            bool gaveUp = false;
            for (int level = 0; level < levels; ++level) {
                if (!gb::clusterMeet(me)) break;
                me.use();
                if (level == at && b == quitter) {
                    gaveUp = true;
                    break;
                }
                if (notices && level == at && b != 0) {  // its own count does not come either
                    while (!me.raised()) std::this_thread::yield();
                    gaveUp = true;
                    break;
                }
            }
            reported[b] = gb::clusterLeave(me, gaveUp);
            c.exit(b);
        });
    for (auto& x : t) x.join();
    int silent = 0;
    for (int r : reported) silent += r == 0;
    std::printf("%d %d %d\n", c.strayed.load(), quitter >= 0 ? silent : n - silent, c.there);
    return 0;
}
