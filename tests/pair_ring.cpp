// The weight ring of the CTA-pair ternary product, run on the CPU: a producer, three unpack groups that go through it by PairWeightWalk, and the matrix
// unit that takes their items in order, as coroutines that a random schedule moves on one wait at a time.  Loads land in any order; a barrier answers by
// the parity of its phase and by nothing else, as the hardware's do.  Arguments: KB tiles stages seeds form; form 1 leaves out the loads that hold no item
// of a group.  Prints "stale N stuck M" over all seeds.
#include <stdio.h>
#include <stdlib.h>
#include <ucontext.h>
#include <functional>
#include <random>
#include <vector>
#include "gemm_tc_pair_walk.h"

using namespace wf;
constexpr int NU = 3;

struct Bar {
    int count = 1, pending = 1, phase = 0;
    void init(int c) { count = pending = c; phase = 0; }
    void arrive(int n = 1) { if ((pending -= n) == 0) { pending = count; ++phase; } }
    bool passed(int parity) const { return (phase & 1) != parity; }
};

struct Task { ucontext_t ctx; std::vector<char> stack; std::function<void()> body; std::function<bool()> ready; bool done = false; };
static ucontext_t home;
static Task* now;
static void enter() { now->body(); now->done = true; swapcontext(&now->ctx, &home); }
static void until(std::function<bool()> ready) {
    now->ready = ready;
    swapcontext(&now->ctx, &home);
}

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    const int KB = atoi(argv[1]), tiles = atoi(argv[2]), TS = atoi(argv[3]), seeds = atoi(argv[4]), form = atoi(argv[5]);
    const int per = (KB + TP_WKB - 1) / TP_WKB, loads = per * tiles, items = KB * tiles;
    long stale = 0, stuck = 0;
    for (int seed = 0; seed < seeds; ++seed) {
        std::mt19937 rng(seed);
        Bar full[TP_WS], empty[TP_WS], a_full[16], a_empty[16];
        int content[TP_WS];
        for (int s = 0; s < TP_WS; ++s) { full[s].init(1); empty[s].init(TP_WKB); content[s] = -1; }
        for (int s = 0; s < TS; ++s) { a_full[s].init(1); a_empty[s].init(1); }
        std::vector<int> flying;
        std::vector<Task> tasks(NU + 2);
        tasks[0].body = [&] {
            for (int c = 0; c < loads; ++c) {
                const int s = c % TP_WS;
                if (c >= TP_WS) until([&, c, s] { return empty[s].passed(((c / TP_WS) & 1) ^ 1); });
                content[s] = -1;
                flying.push_back(c);
                until([] { return true; });
            }
        };
        tasks[1].body = [&] {
            for (int it = 0; it < items; ++it) {
                until([&, it] { return a_full[it % TS].passed((it / TS) & 1); });
                until([] { return true; });
                a_empty[it % TS].arrive();
            }
        };
        for (int g = 0; g < NU; ++g)
            tasks[2 + g].body = [&, g] {
                PairWeightWalk<true> ragged(g, NU, KB);
                PairWeightWalk<false> even(g, NU, KB);
                int kb = g, first = 0, load = 0;
                auto wait = [&](int l) { until([&, l] { return full[l % TP_WS].passed((l / TP_WS) & 1); }); return true; };
                auto back = [&](int l) { empty[l % TP_WS].arrive(); };
                while (kb >= KB) { kb -= KB; first += per; }
                auto fetch = [&] {
                    int back_n = 0;
                    if (form) {
                        load = first + kb / TP_WKB;
                        wait(load);
                        back_n = kb == KB - 1 ? 1 + TP_WKB * per - KB : 1;
                        kb += NU;
                        while (kb >= KB) { kb -= KB; first += per; }
                    } else {
                        if (pair_ragged(KB, NU)) ragged.next(wait, back), load = ragged.load, back_n = ragged.count;
                        else even.next(wait, back), load = even.load, back_n = even.count;
                    }
                    stale += content[load % TP_WS] != load;
                    return back_n;
                };
                int n = 0;
                if (g < items) n = fetch();
                for (int it = g; it < items; it += NU) {
                    empty[load % TP_WS].arrive(n);
                    if (it + NU < items) n = fetch();
                    if (it >= TS) until([&, it] { return a_empty[it % TS].passed((it / TS - 1) & 1); });
                    until([] { return true; });
                    a_full[it % TS].arrive();
                }
            };
        for (auto& t : tasks) {
            t.stack.resize(1 << 16);
            getcontext(&t.ctx);
            t.ctx.uc_stack.ss_sp = t.stack.data(); t.ctx.uc_stack.ss_size = t.stack.size(); t.ctx.uc_link = &home;
            t.ready = [] { return true; };
            makecontext(&t.ctx, enter, 0);
        }
        // how eagerly each task and the landing of loads move differs from seed to seed
        std::vector<int> weight(NU + 3);
        for (auto& w : weight) w = 1 << (rng() % 6);
        const int order = rng() % 3;                   // in order, the last one first, any
        for (;;) {
            std::vector<int> can;
            bool left = false;
            for (int i = 0; i < NU + 2; ++i) {
                if (tasks[i].done) continue;
                left = true;
                if (tasks[i].ready()) can.insert(can.end(), weight[i], i);
            }
            if (!flying.empty()) can.insert(can.end(), weight[NU + 2], NU + 2);
            if (!left) break;
            if (can.empty()) { ++stuck; break; }
            const int i = can[rng() % can.size()];
            if (i == NU + 2) {
                const size_t k = order == 0 ? 0 : order == 1 ? flying.size() - 1 : rng() % flying.size();
                const int l = flying[k];
                flying.erase(flying.begin() + k);
                content[l % TP_WS] = l;
                full[l % TP_WS].arrive();
            } else {
                now = &tasks[i];
                swapcontext(&home, &now->ctx);
            }
        }
    }
    printf("stale %ld stuck %ld\n", stale, stuck);
    return 0;
}
