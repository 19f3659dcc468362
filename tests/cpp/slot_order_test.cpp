// The order check and the repair of the radix sort's tiles, and of the words of the sort in one block
// (ilgpu_b200/csrc/slot_order.cuh) on the host: slots as ranks leave them when the lanes of a warp are served in
// any order, threads for the threads of a block, against a stable sort.  No GPU involved.
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

static int g_checks = 0, g_failures = 0, g_repaired = 0;  // g_repaired: blocks whose words had come out of order
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

// One pass of ranks over words of which each 32 neighbours were served in any order.
template <typename Digit>
static std::vector<unsigned int> ranked(const std::vector<unsigned int> &words, Digit digit, bool in_lane_order, std::mt19937_64 &rng) {
    const int all = (int)words.size();
    std::vector<int> served(all);
    for (int i = 0; i < all; ++i) served[i] = i;
    if (!in_lane_order)
        for (int i = 0; i < all; i += 32) std::shuffle(served.begin() + i, served.begin() + std::min(i + 32, all), rng);
    std::vector<int> start(1025, 0);
    for (const unsigned int w : words) ++start[digit(w) + 1];
    for (int d = 0; d < 1024; ++d) start[d + 1] += start[d];
    std::vector<unsigned int> next(all);
    for (const int i : served) next[start[digit(words[i])]++] = words[i];
    return next;
}

template <typename K, bool PLACE>
static void repair(std::vector<unsigned int> &words, const K *keys, K low, int count, int threads) {
    Block block(threads);
    std::vector<std::thread> team;
    for (int t = 0; t < threads; ++t)
        team.emplace_back([&, t] {
            b200alg::put_words_in_order<K, PLACE>(words.data(), keys, low, count, (int)words.size(), t, threads, [&](bool moved) { return block.meet(moved); });
        });
    for (std::thread &t : team) t.join();
}

// As the kernel looks: strays first, then neighbours.
template <typename K, bool PLACE>
static bool any_wrong(const std::vector<unsigned int> &words, const std::vector<K> &keys, K low, int count) {
    for (int p = count; p < (int)words.size(); ++p)
        if (b200alg::is_stray<PLACE>(words[p], count)) return true;
    auto key_at = [&](int p) { return b200alg::word_key<K, PLACE>(words[p], keys.data(), low); };
    for (int p = 0; p + 1 < count; ++p)
        if (b200alg::words_out_of_order<K, PLACE>(key_at(p), words[p], key_at(p + 1), words[p + 1])) return true;
    return false;
}

// The last element and a place past it have changed places: what is left in front is in order.
static void run_stray() {
    const std::vector<uint64_t> keys = {1, 2, ~0ull, ~0ull, ~0ull};
    std::vector<unsigned int> words = {0, 1, 2, 4, 3};
    CHECK((any_wrong<uint64_t, true>(words, keys, 1, 4)));
    repair<uint64_t, true>(words, keys.data(), 1, 4, 2);
    CHECK((words == std::vector<unsigned int>{0, 1, 2, 3, 4}));
    words = {0, 5, ~0u, 9};
    CHECK((any_wrong<uint32_t, false>(words, {}, 7, 3)));
    repair<uint32_t, false>(words, nullptr, 7, 3, 2);
    CHECK((words == std::vector<unsigned int>{0, 5, 9, ~0u}));
}

// `all` places of a block of which `count` hold an element; distinct: that many different keys (0: random ones).
// width: of the digits of a pass, at most.  (With 2 and 4 different keys the largest shares its digit with the places
// past the last element.)  Every pass serves lanes in any order, or only the last one does.
template <typename K, bool PLACE>
static void run_words(int count, int all, int threads, int distinct, int width, bool in_lane_order, bool last_only, unsigned int seed) {
    std::mt19937_64 rng(seed);
    std::vector<K> keys(count);
    for (K &k : keys) k = distinct ? (K)(~(K)0 - (K)(rng() % distinct)) : (K)rng();  // (the largest key among them)
    K low = (K)~(K)0, high = 0;
    for (const K k : keys) {
        low = std::min(low, k);
        high = std::max(high, k);
    }
    keys.resize(all, (K)~(K)0);  // what lies past the last element: it looks as if it were in order
    std::vector<int> want(count);
    for (int i = 0; i < count; ++i) want[i] = i;
    std::stable_sort(want.begin(), want.end(), [&](int a, int b) { return keys[a] < keys[b]; });

    std::vector<unsigned int> words(all);
    for (int i = 0; i < all; ++i) words[i] = PLACE ? (unsigned int)i : i < count ? (unsigned int)(K)(keys[i] - low) : ~0u;
    int bits = 0;
    while (bits < 8 * (int)sizeof(K) && (K)(high - low) >> bits) ++bits;
    if (bits) width = (bits + (bits + width - 1) / width - 1) / ((bits + width - 1) / width);  // the passes share the bits evenly
    const unsigned int mask = (1u << width) - 1u;
    for (int shift = 0; shift < bits; shift += width) {
        auto digit = [&](unsigned int w) {
            if (!PLACE) return w >> shift & mask;
            const int at = (int)b200alg::place_of(w);
            return at < count ? (unsigned int)((K)(keys[at] - low) >> shift) & mask : mask;
        };
        words = ranked(words, digit, in_lane_order || (last_only && shift + width < bits), rng);
    }
    auto right = [&] {
        for (int p = 0; p < count; ++p) {
            if (PLACE && (int)b200alg::place_of(words[p]) != want[p]) return false;
            if (!PLACE && words[p] != (unsigned int)(K)(keys[want[p]] - low)) return false;
        }
        return true;
    };
    auto found_wrong = [&] { return any_wrong<K, PLACE>(words, keys, low, count); };
    const bool was_right = right();
    CHECK(found_wrong() == !was_right);
    CHECK(was_right || !in_lane_order);
    g_repaired += !was_right;
    repair<K, PLACE>(words, keys.data(), low, count, threads);
    CHECK(right());
    CHECK(!found_wrong());
}

// The words of the partition into buckets: bucket above place, those past the last element in a bucket of their own.
static void run_buckets(int count, int all, int threads, int buckets, bool in_lane_order, unsigned int seed) {
    std::mt19937_64 rng(seed);
    std::vector<unsigned int> words(all);
    for (int i = 0; i < all; ++i) words[i] = (i < count ? (unsigned int)(rng() % buckets) : 511u) << b200alg::kPlaceBits | (unsigned int)i;
    std::vector<unsigned int> want(words);
    std::sort(want.begin(), want.end());
    words = ranked(words, [](unsigned int w) { return w >> b200alg::kPlaceBits; }, in_lane_order, rng);
    bool found = false, right = true;
    for (int p = 0; p < count; ++p) {
        CHECK(words[p] >> b200alg::kPlaceBits == want[p] >> b200alg::kPlaceBits);  // in the right bucket in any case
        found |= p + 1 < count && words[p + 1] < words[p];
        right &= words[p] == want[p];
    }
    CHECK(found == !right);
    CHECK(right || !in_lane_order);
    g_repaired += !right;
    repair<unsigned int, false>(words, nullptr, 0u, count, threads);
    CHECK(std::equal(want.begin(), want.begin() + count, words.begin()));
}

int main() {
    unsigned int seed = 1;
    run_stray();
    for (const int threads : {1, 4}) {
        for (const bool in_lane_order : {false, true}) {
            for (const int count : {1, 31, 100, 500, 512}) {
                for (const int distinct : {0, 1, 2, 4, 200}) {
                    for (const bool last_only : {false, true}) {
                        const int all = count <= 31 ? 64 : 512;
                        run_words<uint64_t, true>(count, all, threads, distinct, 9, in_lane_order, last_only, seed++);
                        run_words<uint32_t, true>(count, all, threads, distinct, 7, in_lane_order, last_only, seed++);
                        run_words<uint8_t, true>(count, all, threads, distinct, 8, in_lane_order, last_only, seed++);
                        run_words<uint32_t, false>(count, all, threads, distinct, 8, in_lane_order, last_only, seed++);
                        run_words<uint16_t, false>(count, all, threads, distinct, 9, in_lane_order, last_only, seed++);
                    }
                }
                run_buckets(count, count <= 31 ? 64 : 512, threads, 1 + count / 8, in_lane_order, seed++);
            }
        }
    }
    CHECK(g_repaired > 200);
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
