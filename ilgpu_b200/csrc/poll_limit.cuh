// How long a kernel polls for a word before it gives up, as one rule that the device code and a
// host-side test share.
//
// A wait for a block that runs needs a limit of a few seconds at most.  The scanners of the digit pass
// and of unique (the first blocks of their kernel to start) wait for something else at first: the
// counts of blocks that may not have started, while a kernel of another stream holds the SMs.  How
// long that one takes is not theirs to judge, so until their first count has come they may poll as
// often, but past kEagerPolls with a pause in between: minutes instead of seconds.  From the first
// count on there is a block that runs to the end and takes every tile that nobody else takes.
#pragma once

#if defined(__CUDACC__)
#define B200ALG_HD __host__ __device__
#else
#define B200ALG_HD
#endif

namespace b200alg {

// Upper bound on polls without anything new.  Each poll is an L2 round trip of ~1 us under load, so this
// is seconds, far beyond any healthy run between blocks that run.
constexpr unsigned int kMaxSpin = 1u << 22;
constexpr unsigned int kEagerPolls = 1u << 16;      // some 50 ms; then
constexpr unsigned int kPauseNanoseconds = 20000u;  // this long between two polls: kMaxSpin of them take 1.4 minutes

class ScannerPolls {
public:
    // After a poll that brought nothing; `begun`: something has come before.  False: give up.
    template <typename Pause> B200ALG_HD bool again(bool begun, Pause pause) {
        if (++polls_ > kMaxSpin) return false;
        if (!begun && polls_ > kEagerPolls) pause(kPauseNanoseconds);
        return true;
    }
    B200ALG_HD void progress() { polls_ = 0u; }

private:
    unsigned int polls_ = 0u;
};

}  // namespace b200alg
