// Walks every interleaving of the bias ring of the D = 96 / 128 forward (csrc/evo_bias_ring.cuh): one
// warp that issues loads in order, loads that land in any order, two streams that wait, read and hand
// back.  Prints "ok" or the first thing that went wrong, for the kernel's ring and for one whose "full"
// barriers go by slot.
#include <array>
#include <cstdio>
#include <set>
#include <string>
#include <vector>

#include "evo_bias_ring.cuh"

using evo::WideBiasRing;
constexpr int SLOTS = WideBiasRing::SLOTS, ROUND = WideBiasRing::PER_ROUND, ROUNDS = 4, LOADS = ROUND * ROUNDS;

struct Where { int bar; unsigned parity; };

struct ByPlace {            // what the kernel does
    static Where full(int load, const WideBiasRing&) {
        const int i = load % ROUND;
        return {WideBiasRing::full_bar(i >> 1, i & 1), WideBiasRing::full_parity(load / ROUND)};
    }
};
struct BySlot {
    static Where full(int, const WideBiasRing& r) { return {r.slot, r.use & 1u}; }
};

struct State {
    int issued = 0;                              // loads issued
    std::array<int, SLOTS> content{}, released{};        // load that a slot holds (-1: garbage); completed phases of "empty"
    std::array<int, ROUND> done{};               // completed phases of the "full" barriers
    std::array<int, ROUND> armed{};              // loads armed and not landed
    std::array<bool, LOADS> flying{};
    std::array<int, 2> pos{};                    // half tiles a stream has finished, times two, plus one while it reads
    std::string key() const {
        std::string k;
        auto put = [&](int v) { k.push_back(static_cast<char>(v + 1)); };
        put(issued);
        for (int v : content) put(v);
        for (int v : released) put(v);
        for (int v : done) put(v);
        for (int v : armed) put(v);
        for (bool v : flying) put(v);
        for (int v : pos) put(v);
        return k;
    }
};
// mbarrier.try_wait.parity: passes once the phase in progress has the other parity
static bool passes(int completed, unsigned parity) { return (static_cast<unsigned>(completed) & 1u) != parity; }

template <class Rule>
static std::string explore() {
    State first;
    first.content.fill(-1);
    std::set<std::string> seen;
    std::vector<State> todo{first};
    while (!todo.empty()) {
        const State s = todo.back();
        todo.pop_back();
        if (!seen.insert(s.key()).second) continue;
        bool moved = false;
        auto push = [&](const State& t) { moved = true; todo.push_back(t); };
        if (s.issued < LOADS) {
            WideBiasRing r = WideBiasRing::at(0);
            for (int i = 0; i < s.issued; ++i) r.advance(1);
            if (r.use == 0 || passes(s.released[r.slot], r.empty_parity())) {
                State t = s;
                const Where w = Rule::full(s.issued, r);
                if (++t.armed[w.bar] > 1) return "a barrier is armed twice";
                t.flying[t.issued++] = true;
                push(t);
            }
        }
        for (int l = 0; l < LOADS; ++l)
            if (s.flying[l]) {
                State t = s;
                const WideBiasRing r = WideBiasRing::at(l);
                const Where w = Rule::full(l, r);
                t.flying[l] = false;
                t.content[r.slot] = l;
                --t.armed[w.bar];
                ++t.done[w.bar];
                push(t);
            }
        for (int st = 0; st < 2; ++st) {
            const int half_tiles = s.pos[st] / 2, n = half_tiles / 2, half = half_tiles & 1;
            if (n == ROUNDS) continue;
            WideBiasRing r = WideBiasRing::at(2 * st);
            for (int i = 0; i < half_tiles; ++i) r.advance((i & 1) ? 3 : 1);
            const int load = ROUND * n + 2 * st + half;
            if (s.pos[st] & 1) {                 // reading: the slot must not have changed
                if (s.content[r.slot] != load) return "a half tile is overwritten while it is read";
                State t = s;
                ++t.pos[st];
                ++t.released[r.slot];
                push(t);
            } else {
                const Where w = Rule::full(load, r);
                if (!passes(s.done[w.bar], w.parity)) continue;
                if (s.content[r.slot] != load) return "a stream reads a half tile that has not landed";
                State t = s;
                ++t.pos[st];
                push(t);
            }
        }
        if (!moved && (s.pos[0] < 4 * ROUNDS || s.pos[1] < 4 * ROUNDS)) return "everybody waits";
    }
    return "ok";
}

int main() {
    std::printf("kernel: %s\nby slot: %s\n", explore<ByPlace>().c_str(), explore<BySlot>().c_str());
    return 0;
}
