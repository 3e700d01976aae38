// loop_order.h -- the order in which the items of a time-loop kernel are taken,
// wait for one another and hand planes on.  Plain C++, so that the rules can be
// checked on the host.
#pragma once

#ifdef __CUDACC__
#define FWI_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FWI_HOST_DEVICE inline
#endif

namespace fwi {

// An item: one step of one column of one shot.
struct Item {
    int shot, t, col;
};

// Ticket order: shots in groups of `group` whose steps interleave, then step,
// shot of the group, column.
FWI_HOST_DEVICE Item item_of(long long ticket, int nshot, int group, int nsteps, int ncol)
{
    const long long per_group = (long long)nsteps * ncol * group;
    const int first = (int)(ticket / per_group) * group;
    const long long r = ticket % per_group;
    const int per_step = (nshot - first < group ? nshot - first : group) * ncol;
    Item it;
    it.t = (int)(r / per_step);
    const int q = (int)(r - (long long)it.t * per_step);
    it.shot = first + q / ncol;
    it.col = q % ncol;
    return it;
}

// The columns whose progress an item waits for: lane 0 its own, lanes 1..4 the
// neighbours along z and x that exist; the other lanes wait for nothing (-1).
FWI_HOST_DEVICE int dependency_column(int lane, int col, int ntz, int ncol)
{
    const int zt = col % ntz;
    switch (lane) {
    case 0: return col;
    case 1: return zt > 0 ? col - 1 : -1;
    case 2: return zt < ntz - 1 ? col + 1 : -1;
    case 3: return col >= ntz ? col - ntz : -1;
    case 4: return col + ntz < ncol ? col + ntz : -1;
    default: return -1;
    }
}

// An item takes in the planes p = 4 .. nyy-1 one after another and stores plane
// p - 4 once it has p.  The planes below this number have to be stored by the
// step before when it takes in plane p; 0: none, since the outer four planes are
// never written.
FWI_HOST_DEVICE int planes_awaited(int p, int nyy) { return p < nyy - 4 ? p + 1 : 0; }

// Receiver samples of a step are read from memory, where step t+2 overwrites
// the level that step t stores.  It may store plane q once step t+1 has stored
// plane q + 4, for which step t+1 took in plane q + 8 of step t, so once step t
// has published more than q + 8 planes; and any plane once step t has published
// all.  Hence step t publishes at most kSampleLead planes beyond those it has
// sampled, and samples everything before it publishes the last ones.
constexpr int kSampleLead = 8;

// The planes below this number are published next: `published` are, `stored`
// are in memory.  lead 0: the work on a plane precedes its publication.
FWI_HOST_DEVICE int next_publication(int published, int stored, int lead)
{
    return lead > 0 && stored > published + lead ? published + lead : stored;
}

// Whether the work on the planes below `next` precedes their publication; `last`
// is the number published when the item is complete.
FWI_HOST_DEVICE bool work_first(int next, int last, int lead) { return lead == 0 || next == last; }

}  // namespace fwi
