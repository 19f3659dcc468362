// The order check and the repair of the radix sort's tiles (ilgpu_b200/csrc/slot_order.cuh) on the host:
// slots as ranks leave them when the lanes of a warp are served in any order, threads for the threads of
// a block, against a stable sort.  No GPU involved.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include "slot_order.cuh"

static int g_checks = 0, g_failures = 0;
#define CHECK(cond)                                                             \
    do {                                                                        \
        ++g_checks;                                                             \
        if (!(cond)) { ++g_failures; std::printf("FAILED %s:%d: %s\n", __FILE__, __LINE__, #cond); } \
    } while (0)

// meet(p): whether p is true for any of the threads, as __syncthreads_or.
class Block {
public:
    explicit Block(int threads) : threads_(threads) {}
    bool meet(bool p) {
        std::unique_lock<std::mutex> g(mu_);
        const unsigned int mine = phase_;
        any_[mine & 1] |= p;
        if (++arrived_ == threads_) {
            arrived_ = 0;
            any_[~mine & 1] = false;
            ++phase_;
            all_here_.notify_all();
        } else {
            all_here_.wait(g, [&] { return phase_ != mine; });
        }
        ++meetings_;
        return any_[mine & 1];
    }
    int meetings() const { return meetings_ / threads_; }

private:
    const int threads_;
    int arrived_ = 0, meetings_ = 0;
    unsigned int phase_ = 0;
    bool any_[2] = {false, false};
    std::mutex mu_;
    std::condition_variable all_here_;
};

template <typename K> struct Flip {  // a descending sort's transform
    K operator()(K raw) const { return (K)~raw; }
};
template <typename K> struct Same {
    K operator()(K raw) const { return raw; }
};

template <typename K, bool VALUES, typename XF>
static bool any_out_of_order(const std::vector<K> &slots, const std::vector<unsigned short> &place, XF xf, int shift) {
    bool bad = false;
    for (size_t p = 0; p + 1 < slots.size(); ++p) bad |= b200alg::out_of_order<K, VALUES>(slots[p], slots[p + 1], place[p], place[p + 1], xf, shift);
    return bad;
}

template <typename K, bool VALUES, typename XF>
static void run(int tile, int threads, int shift, int few, bool in_lane_order, unsigned int seed) {
    std::mt19937_64 rng(seed);
    const XF xf;
    // the tile's keys in the order that the earlier passes have left
    std::vector<K> keys(tile);
    for (K &k : keys) k = few ? (K)((rng() % few) * (K)0x0101010101010101ull) : (K)rng();
    const K below = shift ? (K)((K)~(K)0 >> (8 * (int)sizeof(K) - shift)) : (K)0;
    std::stable_sort(keys.begin(), keys.end(), [&](K a, K b) { return (K)(xf(a) & below) < (K)(xf(b) & below); });
    auto digit = [&](K k) { return (unsigned int)(xf(k) >> shift) & 0xFFu; };
    std::vector<unsigned short> want(tile);
    for (int i = 0; i < tile; ++i) want[i] = (unsigned short)i;
    std::stable_sort(want.begin(), want.end(), [&](unsigned short a, unsigned short b) { return digit(keys[a]) < digit(keys[b]); });
    // slots by rank, where the 32 keys of one atomic of a warp may have been served in any order
    std::vector<int> served(tile);
    for (int i = 0; i < tile; ++i) served[i] = i;
    if (!in_lane_order)
        for (int i = 0; i < tile; i += 32) std::shuffle(served.begin() + i, served.begin() + std::min(i + 32, tile), rng);
    std::vector<int> start(257, 0);
    for (const K k : keys) ++start[digit(k) + 1];
    for (int d = 0; d < 256; ++d) start[d + 1] += start[d];
    std::vector<K> slots(tile);
    std::vector<unsigned short> place(tile);
    for (const int i : served) {
        const int slot = start[digit(keys[i])]++;
        slots[slot] = keys[i];
        place[slot] = (unsigned short)i;
    }
    // keys alone: whichever of two keys comes first that differ only above this digit, a later pass sees to it
    const K sorted_bits = (K)((K)~(K)0 >> (8 * (int)sizeof(K) - 8 - shift));
    auto right_at = [&](int p) {
        if (VALUES) return slots[p] == keys[want[p]] && place[p] == want[p];
        return (K)(xf(slots[p]) & sorted_bits) == (K)(xf(keys[want[p]]) & sorted_bits);
    };
    auto all_right = [&] {
        for (int p = 0; p < tile; ++p)
            if (!right_at(p)) return false;
        return true;
    };
    const bool right = all_right();
    CHECK((any_out_of_order<K, VALUES>(slots, place, xf, shift)) == !right);
    CHECK(right || !in_lane_order);

    Block block(threads);
    std::vector<std::thread> team;
    for (int t = 0; t < threads; ++t)
        team.emplace_back([&, t] {
            b200alg::put_in_order<K, VALUES>(slots.data(), place.data(), tile, t, threads, xf, shift, [&](bool moved) { return block.meet(moved); });
        });
    for (std::thread &t : team) t.join();
    CHECK(all_right());
    std::vector<K> have(slots), had(keys);  // and nothing got lost
    std::sort(have.begin(), have.end());
    std::sort(had.begin(), had.end());
    CHECK(have == had);
    CHECK(block.meetings() <= 2 * (32 + 1));  // nothing is further off than a warp's 32 keys
}

int main() {
    unsigned int seed = 1;
    for (const int tile : {1, 2, 33, 256, 1000}) {
        for (const int threads : {1, 4}) {
            for (const int few : {0, 1, 3}) {
                for (const bool in_lane_order : {false, true}) {
                    run<uint8_t, false, Same<uint8_t>>(tile, threads, 0, few, in_lane_order, seed++);
                    run<uint32_t, false, Same<uint32_t>>(tile, threads, 0, few, in_lane_order, seed++);
                    run<uint32_t, false, Flip<uint32_t>>(tile, threads, 24, few, in_lane_order, seed++);
                    run<uint64_t, false, Flip<uint64_t>>(tile, threads, 40, few, in_lane_order, seed++);
                    run<uint16_t, true, Same<uint16_t>>(tile, threads, 8, few, in_lane_order, seed++);
                    run<uint32_t, true, Flip<uint32_t>>(tile, threads, 16, few, in_lane_order, seed++);
                    run<uint64_t, true, Same<uint64_t>>(tile, threads, 56, few, in_lane_order, seed++);
                }
            }
        }
    }
    std::printf("slot order on the host: %d checks, %d failures\n", g_checks, g_failures);
    return g_failures ? 1 : 0;
}
