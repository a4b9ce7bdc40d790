// The lock of a context (vq_b200/csrc/call_lock.hpp): other threads wait, the holder's own thread is told instead of waiting for
// itself, and the lock is free again afterwards.
#include <cstdio>
#include <thread>
#include <vector>

#include "../../vq_b200/csrc/call_lock.hpp"

int main()
{
    vqb::CallLock lock, other;
    int bad = 0, inside = 0;
    {
        vqb::CallLock::Hold a(lock);
        bad += !a;
        vqb::CallLock::Hold again(lock), b(other);
        bad += bool(again) || !b;
        {
            vqb::CallLock::Hold third(lock);
            bad += bool(third);
        }
        bad += bool(vqb::CallLock::Hold(lock)); // still held: the refused ones released nothing
    }
    bad += !vqb::CallLock::Hold(lock);
    std::vector<std::thread> threads;
    long total = 0;
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([&] {
            for (int i = 0; i < 20000; ++i) {
                vqb::CallLock::Hold h(lock);
                bad += !h || ++inside != 1;
                ++total;
                --inside;
            }
        });
    for (auto &t : threads) t.join();
    bad += total != 80000;
    std::printf(bad ? "call lock: %d failures\n" : "call lock ok\n", bad);
    return bad != 0;
}
