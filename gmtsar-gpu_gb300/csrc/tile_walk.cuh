// The walk of one CTA of the persistent column stage over its tiles: chunks of
// K tiles from a counter all CTAs share, or one range.  Plain host and device
// code, so that a test can run it on the CPU.
#pragma once

#ifdef __CUDACC__
#define XCG_WALK_FN __host__ __device__ __forceinline__
#else
#define XCG_WALK_FN inline
#endif

namespace xcg {

struct TileWalk {
    int t, end;                 // the current tile, the end of its chunk
    int ntiles, K;
    // the chunk of K tiles from `first` on
    XCG_WALK_FN void enter(int first) {
        t = first;
        end = first + K < ntiles ? first + K : ntiles;
    }
    // the current tile is its chunk's last: what follows is the next chunk's first
    XCG_WALK_FN bool last() const { return t + 1 == end; }
    // the tile after the current one, -1: none.  grab: the counter's value for
    // the next chunk, taken where last() (no counter: ntiles)
    XCG_WALK_FN int next(int grab) const {
        if (!last()) return t + 1;
        return grab < ntiles ? grab : -1;
    }
    // on to tile tn = next(grab).  The chunk ends where last() says, not where
    // tn is not t + 1: the counter may hand a CTA the chunk right after its own,
    // whose tiles are then done once each like any other's.
    XCG_WALK_FN void go(int tn) {
        if (last()) enter(tn);
        else t = tn;
    }
};

}  // namespace xcg
