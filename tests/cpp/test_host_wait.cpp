// A wait of the host ends: with what it waited for, with the waited-for thing's own error, or with a message that names it.
#include <cstdio>
#include <cstring>
#include <stdexcept>

#include "../../vq_b200/csrc/host_wait.hpp"

int main()
{
    int bad = 0, polls = 0;
    bool named = false;
    auto what = [&] { return named = true, std::string("3 bytes"); };
    vqb::wait_until([&] { return ++polls == 10000; }, what, 30.0);
    bad += polls != 10000 || named;
    vqb::wait_until([] { return true; }, what, 0.0);
    bad += named;
    try {
        vqb::wait_until([] { return false; }, what, 0.05);
        ++bad;
    } catch (const vqb::Error &e) {
        bad += e.code != 100 || !std::strstr(e.what(), "waiting for 3 bytes");
    }
    try {
        vqb::wait_until([]() -> bool { throw std::runtime_error("the poll's own"); }, what, 30.0);
        ++bad;
    } catch (const std::runtime_error &e) {
        bad += std::strcmp(e.what(), "the poll's own") != 0;
    }
    std::printf(bad ? "host wait: %d failures\n" : "host wait ok\n", bad);
    return bad != 0;
}
