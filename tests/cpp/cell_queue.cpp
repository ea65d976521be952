// The construct's cell queue (tfx_cell_queue.cuh) on 32 host threads, one per lane: every kept cell has to come back
// once, and no entry may be touched by two lanes, one of them writing, without a sync() between.  A ballot is a
// meeting point that orders nothing.  Prints the number of cells lost or doubled and the number of unordered pairs.
#include <barrier>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "tfx_cell_queue.cuh"

static std::barrier<> meeting(32);
static thread_local int laneOf;
static unsigned votes;
static std::mutex lock;
static int epoch = 0;

struct HostWarp {
    static unsigned ballot(bool p) {
        meeting.arrive_and_wait();
        if (laneOf == 0) votes = 0;
        meeting.arrive_and_wait();
        { std::lock_guard<std::mutex> g(lock); votes |= (unsigned)p << laneOf; }
        meeting.arrive_and_wait();
        return votes;
    }
    static void sync() {
        meeting.arrive_and_wait();
        if (laneOf == 0) ++epoch;
        meeting.arrive_and_wait();
    }
    static int count(unsigned m) { return __builtin_popcount(m); }
};

struct Slot {
    uint2 v{};
    int writer = -1, written = -1, read[32];
    Slot() { for (int& r : read) r = -1; }
};
static Slot slots[64];
static long unordered = 0;

struct Ref {
    Slot& s;
    operator uint2() const {
        std::lock_guard<std::mutex> g(lock);
        if (s.written == epoch && s.writer != laneOf) ++unordered;
        s.read[laneOf] = epoch;
        return s.v;
    }
    void operator=(uint2 v) const {
        std::lock_guard<std::mutex> g(lock);
        if (s.written == epoch && s.writer != laneOf) ++unordered;
        for (int l = 0; l < 32; ++l)
            if (l != laneOf && s.read[l] == epoch) ++unordered;
        s.v = v; s.writer = laneOf; s.written = epoch;
    }
};
struct Entries {
    Ref operator[](int i) const { return Ref{slots[i]}; }
};

int main(int argc, char** argv) {
    const int jobs = 40;
    long wrong = 0;
    std::vector<int> seen, kept;
    std::vector<std::thread> lanes;
    for (int l = 0; l < 32; ++l)
        lanes.emplace_back([&, l] {
            laneOf = l;
            for (int job = 0; job < jobs; ++job) {
                const int vol = 1 + (job * 97) % 700, density = 5 + (job * 29) % 96;   // percent
                if (l == 0) { seen.assign(vol, 0); kept.assign(vol, 0); }
                HostWarp::sync();
                tfx::CellQueue<HostWarp, Entries> q{Entries{}, l};
                auto evaluate = [&](uint2 e) {
                    std::lock_guard<std::mutex> g(lock);
                    if ((int)e.x < vol && e.y == 7 * e.x) ++seen[e.x]; else ++wrong;
                };
                for (int c = l; c - l < vol; c += 32) {
                    const bool keep = c < vol && (int)((c * 2654435761u + job * 40503u) >> 16) % 100 < density;
                    if (keep) { std::lock_guard<std::mutex> g(lock); kept[c] = 1; }
                    q.add(keep, make_uint2(c, 7 * c));
                    if (q.full()) evaluate(q.take());
                }
                uint2 e;
                if (q.last(e)) evaluate(e);
                HostWarp::sync();
                if (l == 0)
                    for (int c = 0; c < vol; ++c) wrong += seen[c] != kept[c];
                HostWarp::sync();
            }
        });
    for (auto& t : lanes) t.join();
    std::printf("%ld %ld\n", wrong, unordered);
    return 0;
}
