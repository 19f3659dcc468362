// The scanners' poll limit (ilgpu_b200/csrc/poll_limit.cuh) against a clock that the polls and the
// pauses move on: how long a scanner waits for a first count, and for a later one.  No GPU involved.
#include <cstdio>

#include "poll_limit.cuh"

static int g_checks = 0, g_failures = 0;
#define CHECK(cond)                                                             \
    do {                                                                        \
        ++g_checks;                                                             \
        if (!(cond)) { ++g_failures; std::printf("FAILED %s:%d: %s\n", __FILE__, __LINE__, #cond); } \
    } while (0)

constexpr double kPoll = 0.7e-6;  // seconds: one trip to L2

struct Outcome {
    bool came;
    double seconds;
    unsigned long long polls;
};

// Polls until `arrival` seconds have passed (or the limit says stop).
static Outcome poll_until(b200alg::ScannerPolls &limit, bool begun, double arrival) {
    Outcome o{false, 0.0, 0};
    while (true) {
        ++o.polls;
        o.seconds += kPoll;
        if (o.seconds >= arrival) {
            limit.progress();
            o.came = true;
            return o;
        }
        if (!limit.again(begun, [&](unsigned int ns) { o.seconds += ns * 1e-9; })) return o;
    }
}

int main() {
    // A kernel of another stream holds every other SM for half a minute before the first count can come.
    b200alg::ScannerPolls limit;
    Outcome o = poll_until(limit, false, 30.0);
    CHECK(o.came);
    // Nothing pauses while the wait is as short as it is in a call that has the GPU to itself.
    o = poll_until(limit, false, 0.01);
    CHECK(o.came && o.seconds < 0.01 + 2 * kPoll);
    // Every wait ends: after a number of polls, whether something has come before or not.
    for (int begun = 0; begun < 2; ++begun) {
        b200alg::ScannerPolls fresh;
        o = poll_until(fresh, begun != 0, 1e9);
        CHECK(!o.came && o.polls == b200alg::kMaxSpin + 1ull);
        CHECK(begun ? o.seconds < 10.0 : (o.seconds > 60.0 && o.seconds < 120.0));
    }
    // What has come makes the limit whole again.
    b200alg::ScannerPolls again;
    for (int k = 0; k < 3; ++k) {
        o = poll_until(again, true, 2.5);
        CHECK(o.came);
    }
    std::printf("poll limit on the host: %d checks, %d failures\n", g_checks, g_failures);
    return g_failures ? 1 : 0;
}
