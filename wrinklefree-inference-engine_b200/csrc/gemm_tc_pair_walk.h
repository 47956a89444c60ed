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
// load may hold fewer items than there are groups.  Every group waits for every load all the same and hands every load back, once, when it is
// through with it: a barrier's parity tells two neighbouring phases apart and no more, so a group that left a load out could take the load before it in
// that slot for the one that it is after.
struct PairWeightWalk {
    int KB, loads, groups;
    int kb, first;                                  // the next item's k-block in its tile, and that tile's first load
    int load = -1, part = 0;                        // the item in hand: its load, its place in it

    WF_WALK_FN PairWeightWalk(int group, int groups_, int KB_) : KB(KB_), loads((KB_ + TP_WKB - 1) / TP_WKB), groups(groups_), kb(group), first(0) { wrap(); }

    // on to the next item: back(l) hands load l back, wait(l) returns once it has landed (false: it gave up)
    template <typename Wait, typename Back>
    WF_WALK_FN bool next(Wait wait, Back back) {
        const int to = first + kb / TP_WKB;
        while (load < to) {
            if (load >= 0) back(load);
            if (!wait(load + 1)) return false;
            ++load;
        }
        part = kb % TP_WKB;
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
