// The order in which an unpack group of gemm_tc_pair.cu goes through the ring of weight loads.  Plain C++: the CPU test drives the same code.
#pragma once

#ifdef __CUDACC__
#define WF_WALK_FN __host__ __device__ __forceinline__
#else
#define WF_WALK_FN inline
#endif

namespace wf {

constexpr int TP_WKB = 4;                           // k-blocks per weight load
constexpr int TP_WS = 3;                            // weight loads in the ring

// A tile has KB items (k-blocks) in ceil(KB / TP_WKB) loads, numbered over all tiles; group g of `groups` takes the items g, g + groups, ...  A tile's last
// load may hold fewer items than there are groups (RAGGED).  Every group waits for every load all the same and has a part in handing it back: a barrier's parity
// tells two neighbouring phases apart and no more, so a group that left a load out could take the load before it in that slot for the one that it is after.  A
// load is handed back by TP_WKB arrivals of each of a group's warps: one for an item, one by a group without an item there, and the last item's stands for what
// is missing.  (One arrival of every group as it leaves a load came to the same and made an item's path longer: 14336 x 4096, 48 tokens 11.8 -> 12.5 us; so did the
// look for loads to pass by where there can be none, 12.2.)
inline bool pair_ragged(int KB, int groups) { return groups > KB - (KB - 1) / TP_WKB * TP_WKB; }

template <bool RAGGED>
struct PairWeightWalk {
    int KB, loads, groups, tail;
    int kb, first;                                  // the next item's k-block in its tile, and that tile's first load
    int load = -1, part = 0, count = 0;             // the item in hand: its load, its place in it, its arrivals

    WF_WALK_FN PairWeightWalk(int group, int groups_, int KB_) : KB(KB_), loads((KB_ + TP_WKB - 1) / TP_WKB), groups(groups_), kb(group), first(0) {
        tail = 1 + TP_WKB * loads - KB;
        if (RAGGED) tail -= groups - (KB - (loads - 1) * TP_WKB);                  // groups without an item of a tile's last load
        wrap();
    }

    // on to the next item, the one in hand being handed back: back(l) is this group's arrival for a load l without an item of its own, wait(l) returns once load l
    // has landed (false: it gave up)
    template <typename Wait, typename Back>
    WF_WALK_FN bool next(Wait wait, Back back) {
        const int to = first + kb / TP_WKB;
        if (RAGGED) {
            for (int l = load + 1; l < to; ++l) {
                if (!wait(l)) return false;
                back(l);
            }
        }
        if (!wait(to)) return false;
        load = to;
        part = kb % TP_WKB;
        count = kb == KB - 1 ? tail : 1;
        kb += groups;
        wrap();
        return true;
    }

   private:
    WF_WALK_FN void wrap() {
        while (kb >= KB) { kb -= KB; first += loads; }
    }
};

}  // namespace wf
